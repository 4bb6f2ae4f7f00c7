// cg_site.cuh — per-site pieces of the CG shared by the per-phase kernels
// (cg.cu) and the dataflow kernel (cg_flow.cu): neighbour indices and hop
// signs, the FP64 hops of a reliable update, a site's dot product.
#pragma once

#include "cg_common.cuh"

namespace sfh {
namespace {

// neighbour checkerboard indices and hop signs of one output site, computed
// once and shared by every lane of the block
struct Nbr {
    int up[4], dn[4];
    unsigned eta;  // bit mu: eta_mu(x) = -1
    bool wu, wd;   // the forward / backward time hop wraps (anti-periodic sign)
};

__device__ __forceinline__ Nbr neighbours(const Geom& g, const Coord& c)
{
    Nbr n;
    n.eta = 0;
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        n.up[mu] = lex_up(g, c, mu) >> 1;
        n.dn[mu] = lex_dn(g, c, mu) >> 1;
        if (eta_sign(c, mu) < 0) n.eta |= 1u << mu;
    }
    n.wu = c.x[3] == g.L[3] - 1;
    n.wd = c.x[3] == 0;
    return n;
}

// FP64 hop of x_hi + x_lo for a lane in a reliable update: thi = K x
template <int XP, bool COH = false>
__device__ __forceinline__ void ru_hop1(const CgArgs& a, const CgSys& S, const Coord& c, int q, int i, int rid)
{
    const int nq = 1 - q, Vh = S.g.Vh;
    const void* xhi = rhs_ptr(a, rid, F_XHI);
    const void* xlo = rhs_ptr(a, rid, F_XLO);
    Vec3<double> acc;
    vzero(acc);
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
        const bool eta_neg = eta_sign(c, mu) < 0;
        const int lu = lex_up(S.g, c, mu) >> 1, ld = lex_dn(S.g, c, mu) >> 1;
        const bool wu = (mu == 3) && (c.x[3] == S.g.L[3] - 1);
        const bool wd = (mu == 3) && (c.x[3] == 0);
        {
            Mat3<double> U = GaugeFmt<GP_F64_18>::load(S.U64, q, mu, i, Vh);
            Vec3<double> x = vaxpy(SpinorFmt<SP_F64>::template load<COH>(xhi, nq, lu, Vh), 1.0,
                                   vcvt<double>(SpinorFmt<XP>::template load<COH>(xlo, nq, lu, Vh)));
            vacc(acc, mul_mv(U, x), eta_neg != wu);
        }
        {
            Mat3<double> U = GaugeFmt<GP_F64_18>::load(S.U64, nq, mu, ld, Vh);
            Vec3<double> x = vaxpy(SpinorFmt<SP_F64>::template load<COH>(xhi, nq, ld, Vh), 1.0,
                                   vcvt<double>(SpinorFmt<XP>::template load<COH>(xlo, nq, ld, Vh)));
            vacc(acc, mul_adj_mv(U, x), !(eta_neg != wd));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) acc.c[k] = {0.5 * acc.c[k].re, 0.5 * acc.c[k].im};
    SpinorFmt<SP_F64>::store(rhs_ptr(a, rid, F_THI), q, i, Vh, acc);
}

// the rest of a reliable update at the lane's own site, acc = 2 K thi there:
// x_hi += x_lo, x_lo = 0, r = b - M x_hi, the search direction moved to the
// true residual; returns the |r|^2 contribution (FP64)
template <int SP, int XP>
__device__ __forceinline__ double ru_residual(const CgRhs* a, int Vh, int q, int i, int rid, double m2,
                                              const Vec3<double>& acc)
{
    typedef typename SpinorFmt<SP>::R RS;
    void* xhi = rhs_ptr(a, rid, F_XHI);
    void* xlo = rhs_ptr(a, rid, F_XLO);
    Vec3<double> xn = vaxpy(SpinorFmt<SP_F64>::load_cg(xhi, q, i, Vh), 1.0,
                            vcvt<double>(SpinorFmt<XP>::load_cg(xlo, q, i, Vh)));
    SpinorFmt<SP_F64>::store(xhi, q, i, Vh, xn);
    Vec3<typename SpinorFmt<XP>::R> z;
    vzero(z);
    SpinorFmt<XP>::store(xlo, q, i, Vh, z);
    Vec3<double> b = SpinorFmt<SP_F64>::load(rhs_ptr(a, rid, F_B), q, i, Vh);
    Vec3<double> res;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        res.c[k].re = b.c[k].re - (m2 * xn.c[k].re - 0.5 * acc.c[k].re);
        res.c[k].im = b.c[k].im - (m2 * xn.c[k].im - 0.5 * acc.c[k].im);
    }
    // The search direction of the previous update, p = r_iter + beta p_old,
    // was built from the iterated residual; give it the true one instead,
    // p = r_true + beta p_old, by adding the correction r_true - r_iter.
    // Without it the low-precision lanes of ill-conditioned systems lose
    // their Krylov progress at every update (FP16 storage, eps = 1 links,
    // m = 0.02 on 16^4: 7648 iterations against FP64's 1564; 1750 with it).
    void* rp = rhs_ptr(a, rid, F_R);
    void* pp = rhs_ptr(a, rid, F_P);
    const Vec3<RS> r_iter = SpinorFmt<SP>::load_cg(rp, q, i, Vh);
    Vec3<RS> p = SpinorFmt<SP>::load_cg(pp, q, i, Vh);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p.c[k].re += (RS)res.c[k].re - r_iter.c[k].re;
        p.c[k].im += (RS)res.c[k].im - r_iter.c[k].im;
    }
    SpinorFmt<SP>::store(pp, q, i, Vh, p);
    SpinorFmt<SP>::store(rp, q, i, Vh, vcvt<RS>(res));
    return vdot_re(res, res);
}

// reliable update at the lane's own site: x_hi += x_lo, x_lo = 0,
// r = b - M x_hi; returns the |r|^2 contribution (FP64)
template <int SP, int XP, bool COH = false>
__device__ __forceinline__ double ru_hop2(const CgRhs* a, const CgSys& S, const Coord& c, int q, int i, int rid,
                                          double m2)
{
    const int nq = 1 - q, Vh = S.g.Vh;
    const void* thi = rhs_ptr(a, rid, F_THI);
    Vec3<double> acc;
    vzero(acc);
#pragma unroll 1
    for (int mu = 0; mu < 4; ++mu) {
        const bool eta_neg = eta_sign(c, mu) < 0;
        const int lu = lex_up(S.g, c, mu) >> 1, ld = lex_dn(S.g, c, mu) >> 1;
        const bool wu = (mu == 3) && (c.x[3] == S.g.L[3] - 1);
        const bool wd = (mu == 3) && (c.x[3] == 0);
        Mat3<double> U = GaugeFmt<GP_F64_18>::load(S.U64, q, mu, i, Vh);
        vacc(acc, mul_mv(U, SpinorFmt<SP_F64>::template load<COH>(thi, nq, lu, Vh)), eta_neg != wu);
        Mat3<double> Ud = GaugeFmt<GP_F64_18>::load(S.U64, nq, mu, ld, Vh);
        vacc(acc, mul_adj_mv(Ud, SpinorFmt<SP_F64>::template load<COH>(thi, nq, ld, Vh)), !(eta_neg != wd));
    }
    return ru_residual<SP, XP>(a, Vh, q, i, rid, m2, acc);
}

// one site's Re <a, b>: in FP32 for FP32 vectors (exactly the same value in
// every schedule, added to the FP64 partials), in FP64 for FP64 vectors
template <typename R>
__device__ __forceinline__ double site_dot(const Vec3<R>& a, const Vec3<R>& b)
{
    if constexpr (sizeof(R) == 4) {
        float s = a.c[0].re * b.c[0].re;
        s = fmaf(a.c[0].im, b.c[0].im, s);
#pragma unroll
        for (int k = 1; k < 3; ++k) {
            s = fmaf(a.c[k].re, b.c[k].re, s);
            s = fmaf(a.c[k].im, b.c[k].im, s);
        }
        return (double)s;
    } else {
        return vdot_re(a, b);
    }
}

}  // namespace
}  // namespace sfh
