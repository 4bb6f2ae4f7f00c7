// gauge.cu — link-field kernels of the HMC: Symanzik gauge force, fermion
// force, momentum kick, link update U <- exp(i eps P) U, and the FP64
// reductions Tr P^2, gauge action, plaquette and Re<phi, X>.
//
// Fields are FP64 in the even-odd SoA layout of sfh_core.cuh, links indexed by
// (parity p, direction mu, checkerboard site i).  Gauge links are periodic in
// every direction (Lattice.cpp:213-235); the staple paths are those of
// compute_staple_sum_at_link (Lattice.cpp:249-313) and
// compute_rectangle_staple_sum_at_link (Lattice.cpp:315-499).
//
// Staples: the paths of one link through one direction +-nu share their
// pieces, so that the plaquette staple and the three rectangles of that side
// take 11 products of 3x3 matrices (staple_side) instead of the 18 of walking
// each path on its own; a block of six warps gives each of the six sides of 32
// links to one warp (the directions are then uniform in a warp, a thread holds
// four matrices instead of six, and the sides' links meet in the L1), and adds
// the sides through shared memory.  The products are FMA chains (su3.cuh).
// Measured on the B200, one thread and whole walks per link -> this: gauge
// force 363 -> 228 us at 16^4, 2196 -> 1160 us at 24^4 (1399 with the directions
// of a site far apart in the grid, 1242 with the links loaded as read-only
// data); staples 2470 -> 1300 us; a heatbath sweep 3.57 -> 0.60 ms at 16^4, 18.1 ->
// 3.3 ms at 24^4.  It runs at 15 TFLOP/s (198 a product), 0.38 of the FP64 pipe,
// latency bound on 12 warps per SM (168 registers): a third of the stalls are link loads, a
// fifth each FMA latency and instruction fetch.  A row of the staples per thread (80 registers, 24
// warps, every link read by three threads) was bound by the L1: 2696 us.
#include "sfh_internal.h"
#include "walk.cuh"

namespace sfh {

namespace {

constexpr int kThreads = 128;

// The links around a site x on one side, +nu or -nu, of direction mu:
// M(m, k) = U_mu(x + m mu + k side) and D(m, k), the step from x + m mu +
// k side further along the side: U_nu there, or U_nu^dag of the site below.
// One code for both sides (a D's elements are read transposed and their
// imaginary parts' signs flipped), at the same speed as a copy for each.
struct Side {
    const double2 *Um, *Un;   // the links of mu and of nu at x's parity ...
    const double2 *Vm, *Vn;   // ... and at the other one
    int Vh, lex;
    int m[4];                 // offsets of x + (k - 1) mu
    int sm[3], sd[2];         // of x + k side, and of where its D starts
    int rs, cs;               // a D's row and column strides
    unsigned conj;            // its imaginary parts' sign flip
    bool up;
};

__device__ __forceinline__ Side make_side(const void* U, const Geom& g, const Coord& c, int p, int mu, int nu, bool up)
{
    Side s;
    auto field = [&](int par, int a) { return (const double2*)U + ((size_t)(par * 4 + a) * 9) * g.Vh; };
    s.Um = field(p, mu);
    s.Vm = field(1 - p, mu);
    s.Un = field(up ? p : 1 - p, nu);
    s.Vn = field(up ? 1 - p : p, nu);
    s.Vh = g.Vh;
    s.lex = c.lex;
    s.up = up;
#pragma unroll
    for (int k = 0; k < 4; ++k) s.m[k] = step_offset(g, c, mu, k - 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) s.sm[k] = step_offset(g, c, nu, up ? k : -k);
    s.sd[0] = up ? s.sm[0] : s.sm[1];
    s.sd[1] = up ? s.sm[1] : s.sm[2];
    s.rs = up ? 3 * g.Vh : g.Vh;
    s.cs = up ? g.Vh : 3 * g.Vh;
    s.conj = up ? 0u : 0x80000000u;
    return s;
}

template <int M, int K>
__device__ __forceinline__ M3 side_m(const Side& s)
{
    const double2* b = (((M + K) & 1) ? s.Vm : s.Um) + ((s.lex + s.m[M + 1] + s.sm[K]) >> 1);
    M3 o;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const double2 v = b[(size_t)k * s.Vh];
        o.e[k] = {v.x, v.y};
    }
    return o;
}

template <int M, int K>
__device__ __forceinline__ M3 side_d(const Side& s)
{
    const double2* b = (((M + K) & 1) ? s.Vn : s.Un) + ((s.lex + s.m[M + 1] + s.sd[K]) >> 1);
    M3 o;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double2 v = b[i * s.rs + j * s.cs];
            o.e[3 * i + j] = {v.x, __hiloint2double(__double2hiint(v.y) ^ (int)s.conj, __double2loint(v.y))};
        }
    return o;
}

// The staples of U_mu(x) on one side, as walks from x to x + mu:
//   T  = D0 M1 D2^dag                      D0 = D(0,0), M1 = M(0,1), D2 = D(1,0)
//   R1 = D0 [D M D^dag](one step out) D2^dag
//   R2 = [M^dag D M](x - mu) M1 D2^dag      (starts backwards)
//   R3 = D0 M1 [M D^dag M^dag](x + mu)      (overshoots)
// SPLIT: S = T, R = R1 + R2 + R3; else S = c1 T + c2 (R1 + R2 + R3).
template <bool SPLIT>
__device__ __forceinline__ void staple_side(const Side& s, double c1, double c2, M3& S, M3& R)
{
    M3 A, B, t;
    t = m3_mul(side_d<0, 1>(s), side_m<0, 2>(s));
    A = m3_mul_adj(t, side_d<1, 1>(s));
    B = m3_mul(side_d<0, 0>(s), A);                       // R1 without its last step
    t = m3_adj_mul(side_m<-1, 0>(s), side_d<-1, 0>(s));
    A = m3_mul(t, side_m<-1, 1>(s));
    {
        const M3 M1 = side_m<0, 1>(s);
        m3_mul_to<true>(B, A, M1);                        // + R2's
        A = m3_mul(side_d<0, 0>(s), M1);
    }
    if constexpr (SPLIT) {
        const M3 D2 = side_d<1, 0>(s);
        S = m3_mul_adj(A, D2);
        R = m3_mul_adj(B, D2);
    } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) B.e[k] = {fma(c2, B.e[k].re, c1 * A.e[k].re), fma(c2, B.e[k].im, c1 * A.e[k].im)};
        S = m3_mul_adj(B, side_d<1, 0>(s));
    }
    t = m3_mul_adj(side_m<1, 1>(s), side_d<2, 0>(s));
    B = m3_mul_adj(t, side_m<1, 0>(s));
    if constexpr (SPLIT) {
        m3_mul_to<true>(R, A, B);
    } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) A.e[k] = {c2 * A.e[k].re, c2 * A.e[k].im};
        m3_mul_to<true>(S, A, B);
    }
}

// the links of x's plane mu, nu for the loops that start there
struct PlaneSite {
    const double2* U;
    int Vh, lex, p;
    int m[3], n[3];  // offsets of x + k mu and of x + k nu
};

__device__ __forceinline__ PlaneSite plane_site(const void* U, const Geom& g, const Coord& c, int p, int mu, int nu)
{
    PlaneSite s;
    s.U = (const double2*)U;
    s.Vh = g.Vh;
    s.lex = c.lex;
    s.p = p;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s.m[k] = step_offset(g, c, mu, k);
        s.n[k] = step_offset(g, c, nu, k);
    }
    return s;
}

// U_a(x + dm mu + dn nu)
__device__ __forceinline__ M3 plane_link(const PlaneSite& s, int a, int dm, int dn)
{
    const int i = (s.lex + s.m[dm] + s.n[dn]) >> 1, par = (s.p + dm + dn) & 1;
    const double2* b = s.U + ((size_t)(par * 4 + a) * 9) * s.Vh + i;
    M3 m;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const double2 v = b[(size_t)k * s.Vh];
        m.e[k] = {v.x, v.y};
    }
    return m;
}

// Blocks of the staple kernels: six warps, one side of 32 links each.  The
// parities and directions of a range of sites are adjacent in the grid, so that
// their links meet in the L2 (a field of 24^4 is larger).
constexpr int kSides = 6, kSideThreads = 32 * kSides;

// the sides' staples of the block's 32 links: 18 doubles each
struct SideSum {
    double e[kSides][18][32];
};

// the staples of this thread's link on its warp's side (staple_side)
template <bool SPLIT = false>
__device__ __forceinline__ void side_staples(const void* U, const Geom& g, const Coord& c, int p, int mu, double c1,
                                             double c2, M3& S, M3& R)
{
    const int side = threadIdx.x >> 5, k = side >> 1;
    staple_side<SPLIT>(make_side(U, g, c, p, mu, k + (k >= mu ? 1 : 0), !(side & 1)), c1, c2, S, R);
}

// adds the six sides (into e[0]); ends with the block synchronised
__device__ __forceinline__ void sum_sides(SideSum& sum, const M3& S)
{
    const int side = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        sum.e[side][2 * k][lane] = S.e[k].re;
        sum.e[side][2 * k + 1][lane] = S.e[k].im;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int k = 3 * side + e;
        double x = sum.e[0][k][lane];
#pragma unroll
        for (int w = 1; w < kSides; ++w) x += sum.e[w][k][lane];
        sum.e[0][k][lane] = x;
    }
    __syncthreads();
}

__device__ __forceinline__ M3 side_sum(const SideSum& sum)
{
    const int lane = threadIdx.x & 31;
    M3 S;
#pragma unroll
    for (int k = 0; k < 9; ++k) S.e[k] = {sum.e[0][2 * k][lane], sum.e[0][2 * k + 1][lane]};
    return S;
}

// F = -i f (Q - Q^dag), trace removed
__device__ __forceinline__ M3 antiherm_force(const M3& Q, double f)
{
    M3 F;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            Cx<double> d = csub(Q.e[i * 3 + j], cconj(Q.e[j * 3 + i]));
            F.e[i * 3 + j] = {f * d.im, -f * d.re};  // -i f d
        }
    m3_traceless(F);
    return F;
}

__device__ __forceinline__ Vec3<double> spinor_at(const void* f, int par, int i, int Vh)
{
    const double2* b = (const double2*)f + (size_t)par * 3 * Vh + i;
    Vec3<double> v;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double2 t = __ldg(b + (size_t)c * Vh);
        v.c[c] = {t.x, t.y};
    }
    return v;
}

// Fermions.cpp:443-515: c = eta bc / 4, A_f = (U Y(x+mu)) X(x)^dag,
// A_b = Y(x) X(x+mu)^dag U^dag, F = -i c [(A_f - A_f^dag) + (A_b - A_b^dag)]
__device__ __forceinline__ M3 fermion_force_link(const void* U, const void* X, const void* Y, const Geom& g,
                                                 const Coord& x, int p, int mu)
{
    const int i = x.lex >> 1, j = (x.lex + step_offset(g, x, mu, 1)) >> 1;
    const double c = 0.25 * eta_sign(x, mu) * ((mu == 3 && x.x[3] == g.L[3] - 1) ? -1.0 : 1.0);
    M3 Ux = ld_link(U, p, mu, i, g.Vh);
    Vec3<double> Xx = spinor_at(X, p, i, g.Vh), Xu = spinor_at(X, 1 - p, j, g.Vh);
    Vec3<double> Yx = spinor_at(Y, p, i, g.Vh), Yu = spinor_at(Y, 1 - p, j, g.Vh);
    Vec3<double> uy = mul_mv(Ux, Yu);
    M3 Af, T;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            Af.e[i * 3 + j] = cmul(uy.c[i], cconj(Xx.c[j]));
            T.e[i * 3 + j] = cmul(Yx.c[i], cconj(Xu.c[j]));
        }
    M3 Ab = m3_mul_adj(T, Ux);
    M3 S;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            S.e[i * 3 + j] = cadd(csub(Af.e[i * 3 + j], cconj(Af.e[j * 3 + i])),
                                  csub(Ab.e[i * 3 + j], cconj(Ab.e[j * 3 + i])));
    M3 F;
#pragma unroll
    for (int k = 0; k < 9; ++k) F.e[k] = {c * S.e[k].im, -c * S.e[k].re};  // -i c S
    m3_traceless(F);
    return F;
}

// F, to out or onto the momenta (P -= kick F)
__device__ __forceinline__ void force_out(const Geom& g, int p, int mu, int i, const M3& F, void* out, void* mom,
                                          double kick)
{
    if (mom) {
        M3 P = ld_link(mom, p, mu, i, g.Vh);
        m3_axpy(P, -kick, F);
        st_link(mom, p, mu, i, g.Vh, P);
    } else {
        st_link(out, p, mu, i, g.Vh, F);
    }
}

// the fermion force, one thread per link (add: onto the force in out)
__global__ void __launch_bounds__(kThreads) fermion_force_kernel(Geom g, const void* U, const void* X, const void* Y,
                                                                 int add, void* out, void* mom, double kick)
{
    int i = (blockIdx.x >> 3) * blockDim.x + threadIdx.x;
    int p = (blockIdx.x >> 2) & 1, mu = blockIdx.x & 3;
    if (i >= g.Vh) return;
    M3 F = fermion_force_link(U, X, Y, g, eo_coords(g, p, i), p, mu);
    if (add) m3_acc(F, ld_link(out, p, mu, i, g.Vh));
    force_out(g, p, mu, i, F, out, mom, kick);
}

// The gauge force F_g = -i (beta/12) (U V - (U V)^dag), V = c11 A1 + c12 A2
// (Fermions.cpp:372-384).
__global__ void __launch_bounds__(kSideThreads, 2) gauge_force_kernel(Geom g, const void* U, double beta, double c11,
                                                                      double c12, void* out, void* mom, double kick)
{
    __shared__ SideSum sum;
    const int i = (blockIdx.x >> 3) * 32 + (threadIdx.x & 31), p = (blockIdx.x >> 2) & 1, mu = blockIdx.x & 3;
    M3 S;
    side_staples(U, g, eo_coords(g, p, min(i, g.Vh - 1)), p, mu, c11, c12, S, S);
    sum_sides(sum, S);
    if (threadIdx.x >= 32 || i >= g.Vh) return;
    const M3 F = antiherm_force(m3_mul_adj(ld_link(U, p, mu, i, g.Vh), side_sum(sum)), beta / 12.0);
    force_out(g, p, mu, i, F, out, mom, kick);
}

// A1 (plaquette staples) and A2 (rectangle staples), walked from x + mu back to x
__global__ void __launch_bounds__(kSideThreads, 2) staple_kernel(Geom g, const void* U, void* A1out, void* A2out)
{
    __shared__ SideSum sum;
    const int i = (blockIdx.x >> 3) * 32 + (threadIdx.x & 31), p = (blockIdx.x >> 2) & 1, mu = blockIdx.x & 3;
    M3 S[2];
    side_staples<true>(U, g, eo_coords(g, p, min(i, g.Vh - 1)), p, mu, 1.0, 1.0, S[0], S[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        sum_sides(sum, S[k]);
        if (threadIdx.x < 32 && i < g.Vh) st_link(k == 0 ? A1out : A2out, p, mu, i, g.Vh, m3_adj(side_sum(sum)));
        __syncthreads();
    }
}

// Fermions.cpp:699-723, 984-994: U <- exp(i eps P) U.  check: the production
// path of the reference rejects P_pre with |P-P^dag| > 1e-10 or |tr P| > 1e-10.
__global__ void link_update_kernel(Geom g, void* U, const void* P, double eps, int check, int* err)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int p = blockIdx.y >> 2, mu = blockIdx.y & 3;
    if (i >= g.Vh) return;
    M3 Q = ld_link(P, p, mu, i, g.Vh);
#pragma unroll
    for (int k = 0; k < 9; ++k) Q.e[k] = cscale(Q.e[k], eps);
    if (check) {
        double n2 = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                Cx<double> d = csub(Q.e[a * 3 + b], cconj(Q.e[b * 3 + a]));
                n2 += d.re * d.re + d.im * d.im;
            }
        Cx<double> t = m3_tr(Q);
        if (sqrt(n2) > 1e-10 || sqrt(t.re * t.re + t.im * t.im) > 1e-10) {
            atomicOr(err, DEV_ERR_NOT_HERMITIAN);
            return;
        }
    }
    M3 E;
    if (!expiq(Q, E)) {
        atomicOr(err, DEV_ERR_DOMAIN);
        return;
    }
    M3 Uo = ld_link(U, p, mu, i, g.Vh);
    st_link(U, p, mu, i, g.Vh, m3_mul(E, Uo));
}

// ---------------------------------------------------------------------------
// deterministic FP64 reductions: fixed grid, per-block partials, one final
// block summing the partials in order
// ---------------------------------------------------------------------------
constexpr int kRedBlocks = 1184;  // eight per SM; launch_reduce's partial array holds 2048
constexpr int kRedThreads = 128;

__device__ __forceinline__ double block_reduce(double v, double* sm)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
        r = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    }
    __syncthreads();
    return r;
}

// The plane loops of site x, directions mu < nu: Re Tr of the plaquette and
// (RECT) of the two rectangles that start there, each loop of the lattice
// once.  The staple sums of the reference count a plaquette at each of its
// four links and a rectangle at each of its six, so that
// sum_links Re Tr(U A1) = 4 sum P and sum_links Re Tr(U A2) = 6 sum R; counting
// loops takes 8 products per site and plane instead of 37 per link and plane.
template <bool RECT>
__device__ __forceinline__ void plane_loops(const PlaneSite& s, int mu, int nu, double& plaq, double& rect)
{
    const M3 Un = plane_link(s, nu, 0, 0), Um = plane_link(s, mu, 0, 0);
    const M3 mn = m3_mul(Um, plane_link(s, nu, 1, 0));   // x -> x + mu -> x + mu + nu
    const M3 nm = m3_mul(Un, plane_link(s, mu, 0, 1));   // x -> x + nu -> x + mu + nu
    plaq = m3_retr_adj(mn, nm);
    rect = 0.0;
    if constexpr (RECT) {
        // 2 x 1: U_mu(x) U_mu(x + mu) U_nu(x + 2 mu) against nm U_mu(x + mu + nu)
        M3 a = m3_mul(Um, m3_mul(plane_link(s, mu, 1, 0), plane_link(s, nu, 2, 0)));
        rect = m3_retr_adj(a, m3_mul(nm, plane_link(s, mu, 1, 1)));
        // 1 x 2: mn U_nu(x + mu + nu) against U_nu(x) U_nu(x + nu) U_mu(x + 2 nu)
        a = m3_mul(Un, m3_mul(plane_link(s, nu, 0, 1), plane_link(s, mu, 0, 2)));
        rect += m3_retr_adj(m3_mul(mn, plane_link(s, nu, 1, 1)), a);
    }
}

// RED_TRP2: Re Tr P^2 of every link (Fermions.cpp:662-678); RED_ACTION:
// -(beta/3) (c11 P + c12 R) (Lattice.cpp:759-781) and RED_PLAQ: 4 P / 3
// (Lattice.cpp:784-804) of every site and plane; RED_DOT: Re<a, b> over spinors.
template <int KIND>
__global__ void __launch_bounds__(kRedThreads) reduce_kernel(Geom g, const void* A, const void* B, double beta,
                                                             double c11, double c12, double* partial)
{
    __shared__ double sm[32];
    double acc = 0.0;
    const long first = blockIdx.x * (long)blockDim.x + threadIdx.x, step = (long)gridDim.x * blockDim.x;
    if constexpr (KIND == RED_DOT) {
        const double* a = (const double*)A;
        const double* b = (const double*)B;
        const long n = 6L * g.V;
        for (long k = first; k < n; k += step) acc += a[k] * b[k];
    } else if constexpr (KIND == RED_TRP2) {
        const long nlinks = 4L * g.V;
        for (long l = first; l < nlinks; l += step) {
            const int pm = (int)(l / g.Vh), i = (int)(l - (long)pm * g.Vh);
            const M3 P = ld_link(A, pm >> 2, pm & 3, i, g.Vh);
            acc += m3_retr(P, P);
        }
    } else {
        // block-sized chunks of (parity, plane, site), the parities and planes of
        // a range of sites in turn, so that they meet in the L2
        const long chunks = (g.Vh + kRedThreads - 1) / kRedThreads;
        for (long u = blockIdx.x; u < 12 * chunks; u += gridDim.x) {
            const int pp = (int)(u % 12), i = (int)(u / 12) * kRedThreads + (int)threadIdx.x;
            if (i >= g.Vh) continue;
            const int p = pp >= 6 ? 1 : 0, plane = pp - 6 * p;  // (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
            const int mu = plane < 3 ? 0 : (plane < 5 ? 1 : 2), nu = plane < 3 ? plane + 1 : (plane < 5 ? plane - 1 : 3);
            const PlaneSite s = plane_site(A, g, eo_coords(g, p, i), p, mu, nu);
            double P, R;
            plane_loops<KIND == RED_ACTION>(s, mu, nu, P, R);
            acc += KIND == RED_PLAQ ? (4.0 / 3.0) * P : -(beta / 3.0) * (c11 * P + c12 * R);
        }
    }
    double r = block_reduce(acc, sm);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

__global__ void reduce_final(const double* partial, int n, double* out)
{
    __shared__ double sm[32];
    double acc = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) acc += partial[k];
    double r = block_reduce(acc, sm);
    if (threadIdx.x == 0) *out = r;
}

}  // namespace

// what: bit 0 gauge force, bit 1 fermion force; out = F, or P -= kick F (mom)
cudaError_t launch_force(const Geom& g, const void* U, const void* X, const void* Y, double beta, double c11,
                         double c12, int what, void* out, void* mom, double kick, cudaStream_t s)
{
    if (what & 1)
        gauge_force_kernel<<<8 * ((g.Vh + 31) / 32), kSideThreads, 0, s>>>(g, U, beta, c11, c12, out, mom, kick);
    if (what & 2)
        fermion_force_kernel<<<8 * ((g.Vh + kThreads - 1) / kThreads), kThreads, 0, s>>>(
            g, U, X, Y, (what & 1) && !mom, out, mom, kick);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Heatbath (single_link_heatbath, Lattice.cpp:722-757, with the SU(2)
// sampler of SU3_Sampling.cpp:17-199).  Per link: A = c11 A1 + c12 A2; for
// the subgroups R (0,1), S (0,2), T (1,2): W = the SU(2) projection of that
// block of U A, a = sqrt(det W); a <= 1e-14: a uniform SU(2) element, else X
// drawn with (a, 2 beta / 3) and R = X (W / a)^dag; U <- R U.  One launch
// updates one direction and one colour (x_mu mod 2) * 4 + (sum_{nu != mu} x_nu
// mod 4): links whose staples do not contain each other.  Uniforms: Philox-
// 4x32-10 keyed by the seed, counter (link, draw, sweep, 0x48420000 + subgroup).
// ---------------------------------------------------------------------------
struct HbRng {
    uint2 key;
    unsigned link, sweep, tag, draw;
    double buf[2];
    int have;
    __device__ double u()  // uniform in [0, 1)
    {
        if (have == 0) {
            uint4 r = Philox::gen(make_uint4(link, draw++, sweep, tag), key);
            unsigned long long a = (((unsigned long long)r.x << 21) ^ (unsigned long long)(r.y >> 11)) & ((1ull << 53) - 1);
            unsigned long long b = (((unsigned long long)r.z << 21) ^ (unsigned long long)(r.w >> 11)) & ((1ull << 53) - 1);
            buf[0] = (double)a * (1.0 / 9007199254740992.0);
            buf[1] = (double)b * (1.0 / 9007199254740992.0);
            have = 2;
        }
        return buf[2 - have--];
    }
};

// generate_x0 (SU3_Sampling.cpp:17-31)
__device__ double hb_x0(HbRng& r, double a, double beta)
{
    for (;;) {
        double r1 = 1.0 - r.u(), r2 = 1.0 - r.u(), r3 = 1.0 - r.u();
        double c = cospi(2.0 * r2);
        double l2 = -1.0 / (2.0 * a * beta) * (log(r1) + c * c * log(r3));
        double x = 1.0 - l2;
        double rr = r.u();
        if (rr * rr <= x && x >= -1.0 && x <= 1.0) return 1.0 - 2.0 * l2;
    }
}

template <int N>
__device__ void hb_unit(HbRng& r, double (&v)[N])
{
    for (;;) {
        double len2 = 0.0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            v[k] = 2.0 * r.u() - 1.0;
            len2 += v[k] * v[k];
        }
        double len = sqrt(len2);
        if (len <= 1.0 && len > 0.0) {
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] /= len;
            return;
        }
    }
}

// q0 I + i (q1 sx + q2 sy + q3 sz), row-major 2x2
__device__ __forceinline__ void quat_su2(const double (&q)[4], Cx<double> (&m)[4])
{
    m[0] = {q[0], q[3]};
    m[1] = {q[2], q[1]};
    m[2] = {-q[2], q[1]};
    m[3] = {q[0], -q[3]};
}

// element (a, b) of U S^dag
__device__ __forceinline__ Cx<double> hb_block(const M3& U, const M3& S, int a, int b)
{
    Cx<double> s;
    cfma_bc<true>(s, U.e[a * 3], S.e[b * 3]);
    cfma_bc<false>(s, U.e[a * 3 + 1], S.e[b * 3 + 1]);
    cfma_bc<false>(s, U.e[a * 3 + 2], S.e[b * 3 + 2]);
    return s;
}

// What the samplers of a block's 32 links draw, as far as it does not depend on
// the links: for each subgroup, of the first kHbTries attempts at x0 the
// logarithms' sum and the acceptance variate, and the unit vector that
// follows if that attempt is the accepted one (an attempt takes two Philox
// draws, and every subgroup starts anew).
constexpr int kHbTries = 4;
struct HbDraws {
    double l[3][kHbTries][32], r[3][kHbTries][32], v[3][kHbTries][3][32];
};

// the six warps take two attempts of one subgroup each
__device__ __forceinline__ void hb_draw(HbDraws& d, HbRng r)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = warp >> 1;
    r.tag = 0x48420000u + (unsigned)sub;
#pragma unroll 1
    for (int t = 2 * (warp & 1); t < 2 * (warp & 1) + 2; ++t) {
        r.draw = 2 * t;
        r.have = 0;
        const double r1 = 1.0 - r.u(), r2 = 1.0 - r.u(), r3 = 1.0 - r.u();
        const double c = cospi(2.0 * r2);
        d.l[sub][t][lane] = log(r1) + c * c * log(r3);
        d.r[sub][t][lane] = r.u();
        double v[3];
        hb_unit<3>(r, v);
#pragma unroll
        for (int k = 0; k < 3; ++k) d.v[sub][t][k][lane] = v[k];
    }
}

// one subgroup (rows I, J) of the link U with staple sum A = S^dag; r at its
// first draw
template <int i, int j>
__device__ __forceinline__ void hb_subgroup(const HbDraws& d, int sub, HbRng& r, M3& U, const M3& S, double beta)
{
    const int lane = threadIdx.x & 31;
    const Cx<double> b0 = hb_block(U, S, i, i), b1 = hb_block(U, S, i, j), b2 = hb_block(U, S, j, i),
                     b3 = hb_block(U, S, j, j);
    const double w0 = 0.5 * (b0.re + b3.re), w1 = 0.5 * (b1.im + b2.im);
    const double w2 = 0.5 * (b1.re - b2.re), w3 = 0.5 * (b0.im - b3.im);
    const double a = sqrt(w0 * w0 + w1 * w1 + w2 * w2 + w3 * w3);
    Cx<double> R[4];
    if (a <= 1e-14) {
        double q[4];
        hb_unit<4>(r, q);
        quat_su2(q, R);
    } else {
        const double b = 2.0 * beta / 3.0;
        double x0 = 0.0, v[3];
        int t = 0;
#pragma unroll 1
        for (; t < kHbTries; ++t) {
            const double l2 = -1.0 / (2.0 * a * b) * d.l[sub][t][lane];
            const double x = 1.0 - l2, rr = d.r[sub][t][lane];
            x0 = 1.0 - 2.0 * l2;
            if (rr * rr <= x && x >= -1.0 && x <= 1.0) break;
        }
        if (t < kHbTries) {
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = d.v[sub][t][k][lane];
        } else {
            r.draw = 2 * kHbTries;
            x0 = hb_x0(r, a, b);
            hb_unit<3>(r, v);
        }
        const double nx = sqrt(1.0 - x0 * x0);
        const double qx[4] = {x0, nx * v[0], nx * v[1], nx * v[2]};
        const double qw[4] = {w0 / a, -w1 / a, -w2 / a, -w3 / a};
        Cx<double> X[4], Wd[4];
        quat_su2(qx, X);
        quat_su2(qw, Wd);
        R[0] = cadd(cmul(X[0], Wd[0]), cmul(X[1], Wd[2]));
        R[1] = cadd(cmul(X[0], Wd[1]), cmul(X[1], Wd[3]));
        R[2] = cadd(cmul(X[2], Wd[0]), cmul(X[3], Wd[2]));
        R[3] = cadd(cmul(X[2], Wd[1]), cmul(X[3], Wd[3]));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // rows i and j of R U
        const Cx<double> ui = U.e[i * 3 + k], uj = U.e[j * 3 + k];
        cfma<true>(U.e[i * 3 + k], R[0], ui);
        cfma<false>(U.e[i * 3 + k], R[1], uj);
        cfma<true>(U.e[j * 3 + k], R[2], ui);
        cfma<false>(U.e[j * 3 + k], R[3], uj);
    }
}

// site k of the V / 8 sites of one colour of direction mu, in an order that
// keeps t fastest: the colour fixes x_mu mod 2 and one other coordinate (t, or
// z for mu = t) mod 4 given the rest
__device__ __forceinline__ Coord hb_site(const Geom& g, int mu, int colour, int k)
{
    const int d = mu == 3 ? 2 : 3;  // the coordinate that the sum fixes mod 4
    int x[4], rest = k, sum = 0;
#pragma unroll
    for (int nu = 3; nu >= 0; --nu) {
        const int n = nu == mu ? g.L[nu] / 2 : (nu == d ? g.L[nu] / 4 : g.L[nu]);
        x[nu] = rest % n;
        rest /= n;
        if (nu == mu) x[nu] = 2 * x[nu] + (colour >> 2);
        else if (nu != d) sum += x[nu];
    }
    const int r = ((colour & 3) - sum) & 3;
    if (mu == 3) x[2] = 4 * x[2] + r;
    else x[3] = 4 * x[3] + r;
    Coord c;
#pragma unroll
    for (int nu = 0; nu < 4; ++nu) c.x[nu] = x[nu];
    c.lex = ((x[0] * g.L[1] + x[1]) * g.L[2] + x[2]) * g.L[3] + x[3];
    return c;
}

// Only the colour's links have threads (one link in eight of a thread per site
// left every warp an eighth full): six warps share the staples of 32 of them (a
// launch at 16^4 has 8192 links, 55 per SM, and their staples are a chain of 66
// products), then one warp updates them: 112 -> 28 us a launch at 16^4.  What the
// samplers draw needs no link, so all six warps draw it first, while the
// launch before is still at work: 28 -> 27 us, with the programmatic dependency
// and plain loads of the links 19; at 4^4 21 -> 10.
__global__ void __launch_bounds__(kSideThreads, 2) heatbath_kernel(Geom g, void* U, int mu, int colour, double beta,
                                                                   double c11, double c12, unsigned long long seed,
                                                                   int sweep)
{
    __shared__ SideSum sum;
    __shared__ HbDraws draws;
    const int k = blockIdx.x * 32 + (threadIdx.x & 31), n = g.V / 8;
    const Coord c = hb_site(g, mu, colour, min(k, n - 1));
    const int p = (c.x[0] + c.x[1] + c.x[2] + c.x[3]) & 1, i = c.lex >> 1;
    HbRng r;
    r.key = make_uint2((unsigned)seed, (unsigned)(seed >> 32));
    r.link = (unsigned)(c.lex * 4 + mu);
    r.sweep = (unsigned)sweep;
    hb_draw(draws, r);
    pdl_begin();  // the draws need no link; plain loads from here, as the links were being written
    M3 S;
    side_staples(U, g, c, p, mu, c11, c12, S, S);
    sum_sides(sum, S);
    if (threadIdx.x >= 32 || k >= n) return;
    S = side_sum(sum);
    M3 u = ld_link(U, p, mu, i, g.Vh);
    auto restart = [&](int sub) {
        r.tag = 0x48420000u + (unsigned)sub;
        r.draw = 0;
        r.have = 0;
    };
    restart(0);
    hb_subgroup<0, 1>(draws, 0, r, u, S, beta);
    restart(1);
    hb_subgroup<0, 2>(draws, 1, r, u, S, beta);
    restart(2);
    hb_subgroup<1, 2>(draws, 2, r, u, S, beta);
    st_link(U, p, mu, i, g.Vh, u);
}

cudaError_t launch_heatbath(const Geom& g, void* U, double beta, double c11, double c12, unsigned long long seed,
                            int sweep0, int nsweeps, cudaStream_t s)
{
    // a launch's draws overlap the launch before it (pdl_begin)
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((g.V / 8 + 31) / 32);
    cfg.blockDim = dim3(kSideThreads);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    for (int sw = sweep0; sw < sweep0 + nsweeps; ++sw)
        for (int mu = 0; mu < 4; ++mu)
            for (int col = 0; col < 8; ++col) {
                const cudaError_t e =
                    cudaLaunchKernelEx(&cfg, heatbath_kernel, g, U, mu, col, beta, c11, c12, seed, sw);
                if (e != cudaSuccess) return e;
            }
    return cudaGetLastError();
}

// Y += a X over a link field (FP64 18-real)
__global__ void link_axpy_kernel(Geom g, double2* Y, double a, const double2* X, long n)
{
    long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double2 x = X[k], y = Y[k];
    Y[k] = make_double2(fma(a, x.x, y.x), fma(a, x.y, y.y));
}

cudaError_t launch_link_axpy(const Geom& g, void* Y, double a, const void* X, cudaStream_t s)
{
    long n = (long)g.V * 4 * 9;
    link_axpy_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, (double2*)Y, a, (const double2*)X, n);
    return cudaGetLastError();
}

cudaError_t launch_staples(const Geom& g, const void* U, void* A1, void* A2, cudaStream_t s)
{
    staple_kernel<<<8 * ((g.Vh + 31) / 32), kSideThreads, 0, s>>>(g, U, A1, A2);
    return cudaGetLastError();
}

cudaError_t launch_link_update(const Geom& g, void* U, const void* P, double eps, int check, int* err,
                               cudaStream_t s)
{
    link_update_kernel<<<dim3((g.Vh + 127) / 128, 8), 128, 0, s>>>(g, U, P, eps, check, err);
    return cudaGetLastError();
}

// partial must hold kRedBlocks doubles; the result lands in *out (device)
cudaError_t launch_reduce(const Geom& g, int kind, const void* A, const void* B, double beta, double c11,
                          double c12, double* partial, double* out, cudaStream_t s)
{
    const auto k = kind == RED_TRP2     ? reduce_kernel<RED_TRP2>
                   : kind == RED_ACTION ? reduce_kernel<RED_ACTION>
                   : kind == RED_PLAQ   ? reduce_kernel<RED_PLAQ>
                                        : reduce_kernel<RED_DOT>;
    k<<<kRedBlocks, kRedThreads, 0, s>>>(g, A, B, beta, c11, c12, partial);
    reduce_final<<<1, 1024, 0, s>>>(partial, kRedBlocks, out);
    return cudaGetLastError();
}

}  // namespace sfh
