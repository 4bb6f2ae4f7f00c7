// walk.cuh — walking the periodic lattice by coordinates and reading FP64
// link fields at arbitrary sites (gauge links are periodic in every
// direction, Lattice.cpp:213-235).
#pragma once

#include "su3.cuh"

namespace sfh {

// coordinate and extent of a runtime direction, without indexing an array
__device__ __forceinline__ int coord_of(const Coord& c, int mu)
{
    return mu == 0 ? c.x[0] : (mu == 1 ? c.x[1] : (mu == 2 ? c.x[2] : c.x[3]));
}

__device__ __forceinline__ int extent_of(const Geom& g, int mu)
{
    return mu == 0 ? g.L[0] : (mu == 1 ? g.L[1] : (mu == 2 ? g.L[2] : g.L[3]));
}

// lexicographic offset of x + k mu, |k| <= 2 <= L (periodic)
__device__ __forceinline__ int step_offset(const Geom& g, const Coord& c, int mu, int k)
{
    const int L = extent_of(g, mu), x = coord_of(c, mu);
    int y = x + k;
    if (y < 0) y += L;
    if (y >= L) y -= L;
    return (y - x) * lex_stride(g, mu);
}

struct Walker {
    int x[4];
};

__device__ __forceinline__ void walk(const Geom& g, Walker& w, int mu, int dir)
{
    int v = w.x[mu] + dir;
    if (v < 0) v += g.L[mu];
    if (v >= g.L[mu]) v -= g.L[mu];
    w.x[mu] = v;
}

__device__ __forceinline__ int lex_of(const Geom& g, const Walker& w)
{
    return ((w.x[0] * g.L[1] + w.x[1]) * g.L[2] + w.x[2]) * g.L[3] + w.x[3];
}

__device__ __forceinline__ M3 link_at(const void* U, const Geom& g, const Walker& w, int mu)
{
    int par = (w.x[0] + w.x[1] + w.x[2] + w.x[3]) & 1;
    int i = lex_of(g, w) >> 1;
    const double2* b = (const double2*)U + ((size_t)(par * 4 + mu) * 9) * g.Vh + i;
    M3 m;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        double2 v = __ldg(b + (size_t)k * g.Vh);
        m.e[k] = {v.x, v.y};
    }
    return m;
}

}  // namespace sfh
