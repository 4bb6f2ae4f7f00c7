// cg_flow.cu — the CG of small systems as one dataflow kernel.
//
// On a small lattice an iteration of the per-phase kernels (cg.cu) costs its
// three launches and their chains of dependent loads, 15 to 25 us up to 16^4,
// for 1 to 3 us of arithmetic.  Here one cooperative launch runs the whole
// solve.  Each block owns a range of checkerboard sites of both parities of one
// system for the whole solve: its search direction, residual, t = K p and v
// stay in shared memory, its links in registers or the L1, and its lanes'
// scalars are advanced by every block of the team for itself, from the same
// sums in the same order.
//
// Blocks exchange two vectors per iteration (p and t) and the four CG sums.
// There is no grid barrier on that path: a published vector is a few 16-byte
// words, each holding 12 bytes of data and the tag of the iteration that wrote
// it, written and read as single 128-bit accesses, and a reader takes a word
// once its tag is the one it waits for.  So a hand-over costs one store and one
// load through L2, where flag and barrier schemes add a fence and a second
// round trip.  Neighbours that the block owns itself are read from its shared
// memory.
//
// A word may be overwritten only when every reader has taken it: p and t of
// iteration k are read before their readers' blocks publish the sums of
// iteration k, and are overwritten after the writer has taken all those sums;
// the sums have one buffer per iteration parity for the same reason.
//
// The per-site arithmetic is that of the per-phase kernels, operand for
// operand (FP64: flow_hop), and the sums of the mixed precisions are FP64 sums
// of FP32 site products, so that their solutions equal the per-phase kernels'
// unless a sum's last bit turns the FP32 rounding of alpha or beta.  An FP64
// reliable update runs on the global arrays between two fenced team barriers.
// Every wait is bounded; one that gives up sets the error word, the others
// follow, and the solve runs again in the per-phase kernels.
//
// Measured, us per iteration, per-phase kernels -> this one: FP64 4^4 15 -> 6,
// 8^3 16 20 -> 8.5, 12^4 21 -> 12.7, 16^4 26 -> 21.5, 16^3 32 58 -> 53; FP32
// 12^3 24 22 -> 14, 16^3 32 38 -> 28, 16^3 48 48 -> 39; FP16 16^4 23 -> 15.5,
// 16^3 64 54 -> 50; FP16 8^4 with 8 RHS 29 -> 15.  What is left is latency: of
// the 8.5 us at 8^3 16, each hop takes 1.5 (0.6 of it the hand-over), the sums
// 3.5 (two hand-overs and the wait for the slowest of 128 blocks), the lanes'
// scalars 0.5 and the update 0.6.
#include <algorithm>
#include <vector>

#include "cg_flow.cuh"
#include "cg_site.cuh"

namespace sfh {

namespace {

// ---------------------------------------------------------------------------
// published words: 128-bit (64-bit) accesses at GPU scope, so that a word's
// data and its tag are always seen together
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 ld_word(const uint4* p)
{
    unsigned long long a, b;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
    return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}

__device__ __forceinline__ void st_word(uint4* p, uint4 w)
{
    const unsigned long long a = (unsigned long long)w.y << 32 | w.x, b = (unsigned long long)w.w << 32 | w.z;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(a), "l"(b)
                 : "memory");
}

__device__ __forceinline__ uint2 ld_word(const uint2* p)
{
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return make_uint2((unsigned)a, (unsigned)(a >> 32));
}

__device__ __forceinline__ void st_word(uint2* p, uint2 w)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((unsigned long long)w.y << 32 | w.x) : "memory");
}

// the block's waits
struct FlowCtx {
    int polls;          // bound on each
    int* err;
    volatile int dead;  // one gave up: none waits again
};

// whether a wait that has polled so often goes on
__device__ __forceinline__ bool wait_on(FlowCtx* c, int& polls)
{
    if (c->dead) return false;
    ++polls;
    if (polls > c->polls || ((polls & 1023) == 0 && __ldcg(c->err) != 0)) {
        atomicOr(c->err, 1);
        c->dead = 1;
        return false;
    }
    return true;
}

// One site's vector as stored by its owner (Val), as published (Word), and
// its place in an array of N sites: component arrays of N (FP64, FP32), or
// one word per site (the 16-bit formats with their scale).
template <int SP> struct FlowVec {  // FP64, FP32: six numbers in words of 12 bytes
    typedef typename SpinorFmt<SP>::R R;
    typedef typename C2<R>::T E;
    typedef Vec3<R> Val;
    static constexpr int NW = sizeof(R) == 8 ? 4 : 2;
    static constexpr int pub_bytes = 16 * NW;
    static constexpr int own_bytes = 6 * sizeof(R);
    struct Word {
        uint4 w[NW];
    };
    __device__ static __forceinline__ Vec3<R> vec(const Val& v) { return v; }
    __device__ static __forceinline__ Val pack(const Vec3<R>& v) { return v; }
    struct O {  // component arrays of N (in shared memory, or one parity of a global array)
        E* e;
        int N;
        __device__ __forceinline__ Val ld(int at) const
        {
            Val v;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const E x = e[c * N + at];
                v.c[c] = {x.x, x.y};
            }
            return v;
        }
        __device__ __forceinline__ void st(int at, const Val& v) const
        {
#pragma unroll
            for (int c = 0; c < 3; ++c) e[c * N + at] = E{v.c[c].re, v.c[c].im};
        }
    };
    __device__ static __forceinline__ O array(void* b, int N) { return {reinterpret_cast<E*>(b), N}; }
    __device__ static __forceinline__ void bits(const Val& v, unsigned (&u)[3 * NW])
    {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if constexpr (sizeof(R) == 8) {
                u[4 * c] = (unsigned)__double2loint(v.c[c].re);
                u[4 * c + 1] = (unsigned)__double2hiint(v.c[c].re);
                u[4 * c + 2] = (unsigned)__double2loint(v.c[c].im);
                u[4 * c + 3] = (unsigned)__double2hiint(v.c[c].im);
            } else {
                u[2 * c] = __float_as_uint(v.c[c].re);
                u[2 * c + 1] = __float_as_uint(v.c[c].im);
            }
        }
    }
    __device__ static __forceinline__ void publish(char* b, int N, int at, const Val& v, unsigned tag)
    {
        unsigned u[3 * NW];
        bits(v, u);
#pragma unroll
        for (int k = 0; k < NW; ++k)
            st_word(reinterpret_cast<uint4*>(b) + (size_t)k * N + at,
                    make_uint4(u[3 * k], u[3 * k + 1], u[3 * k + 2], tag));
    }
    // publish by the SPL threads of a site: thread h writes words h, h + SPL, ...
    template <int SPL>
    __device__ static __forceinline__ void publish_part(char* b, int N, int at, const Val& v, unsigned tag, int h)
    {
        unsigned u[3 * NW];
        bits(v, u);
#pragma unroll
        for (int k0 = 0; k0 < NW; k0 += SPL) {
            uint4 w = make_uint4(u[3 * k0], u[3 * k0 + 1], u[3 * k0 + 2], tag);
#pragma unroll
            for (int m = 1; m < SPL; ++m)
                if (k0 + m < NW && h == m) w = make_uint4(u[3 * (k0 + m)], u[3 * (k0 + m) + 1], u[3 * (k0 + m) + 2], tag);
            if (k0 + h < NW) st_word(reinterpret_cast<uint4*>(b) + (size_t)(k0 + h) * N + at, w);
        }
    }
    __device__ static __forceinline__ Word take(const char* b, int N, int at)
    {
        Word w;
#pragma unroll
        for (int k = 0; k < NW; ++k) w.w[k] = ld_word(reinterpret_cast<const uint4*>(b) + (size_t)k * N + at);
        return w;
    }
    __device__ static __forceinline__ bool ready(const Word& w, unsigned tag)
    {
        bool ok = true;
#pragma unroll
        for (int k = 0; k < NW; ++k) ok &= w.w[k].w == tag;
        return ok;
    }
    __device__ static __forceinline__ Val value(const Word& w)
    {
        unsigned u[3 * NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            u[3 * k] = w.w[k].x;
            u[3 * k + 1] = w.w[k].y;
            u[3 * k + 2] = w.w[k].z;
        }
        Val v;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if constexpr (sizeof(R) == 8)
                v.c[c] = {__hiloint2double((int)u[4 * c + 1], (int)u[4 * c]),
                          __hiloint2double((int)u[4 * c + 3], (int)u[4 * c + 2])};
            else
                v.c[c] = {__uint_as_float(u[2 * c]), __uint_as_float(u[2 * c + 1])};
        }
        return v;
    }
};

template <int SP> struct FlowVec16 {  // three 16-bit pairs and an FP32 scale: {pairs, tag}, {scale, tag}
    typedef float R;
    typedef uint4 Val;
    static constexpr int pub_bytes = 24;
    static constexpr int own_bytes = 16;
    struct Word {
        uint4 a;
        uint2 b;
    };
    __device__ static __forceinline__ Vec3<R> vec(const Val& v) { return SpinorFmt<SP>::unpack(v); }
    __device__ static __forceinline__ Val pack(const Vec3<R>& v) { return SpinorFmt<SP>::pack(v); }
    struct O {
        uint4* e;
        __device__ __forceinline__ Val ld(int at) const { return e[at]; }
        __device__ __forceinline__ void st(int at, const Val& v) const { e[at] = v; }
    };
    __device__ static __forceinline__ O array(void* b, int) { return {reinterpret_cast<uint4*>(b)}; }
    __device__ static __forceinline__ void publish(char* b, int N, int at, const Val& v, unsigned tag)
    {
        st_word(reinterpret_cast<uint4*>(b) + at, make_uint4(v.x, v.y, v.z, tag));
        st_word(reinterpret_cast<uint2*>(b + (size_t)16 * N) + at, make_uint2(v.w, tag));
    }
    template <int SPL>
    __device__ static __forceinline__ void publish_part(char* b, int N, int at, const Val& v, unsigned tag, int k)
    {
        if (k == 0) st_word(reinterpret_cast<uint4*>(b) + at, make_uint4(v.x, v.y, v.z, tag));
        else if (k == 1) st_word(reinterpret_cast<uint2*>(b + (size_t)16 * N) + at, make_uint2(v.w, tag));
    }
    __device__ static __forceinline__ Word take(const char* b, int N, int at)
    {
        Word w;
        w.a = ld_word(reinterpret_cast<const uint4*>(b) + at);
        w.b = ld_word(reinterpret_cast<const uint2*>(b + (size_t)16 * N) + at);
        return w;
    }
    __device__ static __forceinline__ bool ready(const Word& w, unsigned tag) { return w.a.w == tag && w.b.y == tag; }
    __device__ static __forceinline__ Val value(const Word& w) { return make_uint4(w.a.x, w.a.y, w.a.z, w.b.x); }
};
template <> struct FlowVec<SP_F16> : FlowVec16<SP_F16> {};
template <> struct FlowVec<SP_BF16> : FlowVec16<SP_BF16> {};

// SPL threads of a warp share a site's hop, 4 / SPL consecutive directions
// each: lane = (32 / SPL) h + (site mod 32 / SPL).  A whole hop is a chain of
// some 700 instructions, and a small lattice leaves a scheduler one or two
// warps to hide their latency; shared, it is shorter, and more of the
// neighbours' words are requested at once.

// One direction's neighbours of a site: the place of the neighbour's vector
// (of the block's own vectors, q n + s, with kNbrOwn; else of the published
// ones, q Vh + i) and the sign bits of the hop.
struct NbrPair {
    int up, dn;
};
constexpr int kNbrIdx = (1 << 28) - 1;      // places are below V <= 2^28
constexpr int kNbrEta = 1 << 28;            // in up: eta_mu(x) = -1
constexpr int kNbrWrap = 1 << 29;           // the time hop wraps (anti-periodic sign)
constexpr int kNbrOwn = (int)(1u << 31);

// i0, n: the block's range; tn: its stride between the parities
__device__ __forceinline__ NbrPair nbr_pair(const Geom& g, int q, int i, int mu, int i0, int n, int tn)
{
    const Coord c = eo_coords(g, q, i);
    auto place = [&](int j) {
        const int s = j - i0;
        return (unsigned)s < (unsigned)n ? ((1 - q) * tn + s) | kNbrOwn : (1 - q) * g.Vh + j;
    };
    NbrPair p = {place(lex_up(g, c, mu) >> 1), place(lex_dn(g, c, mu) >> 1)};
    if (eta_sign(c, mu) < 0) p.up |= kNbrEta;
    if (mu == 3 && c.x[3] == g.L[3] - 1) p.up |= kNbrWrap;
    if (mu == 3 && c.x[3] == 0) p.dn |= kNbrWrap;
    return p;
}

// A link ready for the products: FP16 unpacked to nine half2, else a matrix.
template <int GP, int SP> struct FlowLink {
    Mat3<typename GaugeFmt<GP>::R> u;
    __device__ __forceinline__ void load(const void* Ulo, int p, int mu, int i, int Vh)
    {
        u = GaugeFmt<GP>::load(Ulo, p, mu, i, Vh);
    }
};
template <> struct FlowLink<GP_F16_12, SP_F16> {
    __half2 u[9];
    __device__ __forceinline__ void load(const void* Ulo, int p, int mu, int i, int Vh)
    {
        hlink_load<false>(nullptr, kTile, Ulo, 0, p, mu, i, Vh, u);
    }
};

// what a hop reads
template <int SP> struct FlowIn {
    const char* pub;             // the published words of its input
    typename FlowVec<SP>::O own; // the block's own vectors of it
    int N2;                      // places of pub
    unsigned tag;
};

// acc = K in at the site of this thread's group (all its threads get it).
// The arithmetic is that of the per-phase kernels' hop (hop_lanes in cg.cu)
// operand for operand where one thread does it all, and for FP16 and FP32-12
// also where several do: each direction's product is formed by its thread
// and accumulated in the directions' order.  In the other formats that hop
// is one chain of FMAs over the directions; shared, each thread's chain
// starts from zero and they are added.
// nbr(k), lup(k, L), ldn(k, L): neighbours and links of the thread's k-th direction
template <int GP, int SP, int SPL, typename Nb, typename Lu, typename Ld>
__device__ __forceinline__ Vec3<typename GaugeFmt<GP>::R> flow_hop(FlowCtx* x, const FlowIn<SP>& in, Nb nbr, Lu lup,
                                                                   Ld ldn)
{
    typedef typename GaugeFmt<GP>::R R;
    typedef FlowVec<SP> F;
    constexpr int ND = 4 / SPL;                             // directions of this thread
    constexpr int G = SP == SP_F64 ? 1 : (ND < 2 ? ND : 2);  // and of a group of requests
    constexpr bool half = GP == GP_F16_12 && SP == SP_F16;
    constexpr bool direct = !half && (GaugeFmt<GP>::K == 9 || SpinorFmt<SP>::scaled);
    constexpr int W = 32 / SPL;
    const int site = threadIdx.x & (W - 1);
    Vec3<R> acc;
    Vec3<R> w[direct || half ? 1 : ND];                  // FP32-12: each direction's sum of both hops
    __half2 yu[half ? ND : 1][3], yd[half ? ND : 1][3];  // FP16: each hop's product and factor
    float fu[half ? ND : 1], fd[half ? ND : 1];
    R sg[ND];
    vzero(acc);
    if constexpr (direct) vzero(w[0]);
#pragma unroll
    for (int g = 0; g < ND; g += G) {
        NbrPair nb[G];
        typename F::Word wu[G], wd[G];
#pragma unroll
        for (int d = 0; d < G; ++d) {
            nb[d] = nbr(g + d);
            if (!(nb[d].up & kNbrOwn)) wu[d] = F::take(in.pub, in.N2, nb[d].up & kNbrIdx);
            if (!(nb[d].dn & kNbrOwn)) wd[d] = F::take(in.pub, in.N2, nb[d].dn & kNbrIdx);
        }
        auto fetch = [&](int code, typename F::Word& word) -> typename F::Val {
            if (code & kNbrOwn) return in.own.ld(code & kNbrIdx);
            int polls = 0;
            while (!F::ready(word, in.tag) && wait_on(x, polls)) word = F::take(in.pub, in.N2, code & kNbrIdx);
            return F::value(word);
        };
#pragma unroll
        for (int d = 0; d < G; ++d) {
            const int k = g + d;
            const R f = (nb[d].up & kNbrEta) ? R(-0.5) : R(0.5);
            const bool nu = nb[d].up & kNbrWrap, nd = nb[d].dn & kNbrWrap;
            sg[k] = f;
            if constexpr (half) {
                FlowLink<GP, SP> U;
                lup(k, U);
                const uint4 vu = fetch(nb[d].up, wu[d]);
                half_products<false>(U.u, vu, yu[k]);
                fu[k] = (nu ? -f : f) * __uint_as_float(vu.w);
                ldn(k, U);
                const uint4 vd = fetch(nb[d].dn, wd[d]);
                half_products<true>(U.u, vd, yd[k]);
                fd[k] = (nd ? f : -f) * __uint_as_float(vd.w);
                if constexpr (SPL == 1) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) acc_f32x2(acc.c[c], f32x2_bcast(fu[k]), __half22float2(yu[k][c]));
#pragma unroll
                    for (int c = 0; c < 3; ++c) acc_f32x2(acc.c[c], f32x2_bcast(fd[k]), __half22float2(yd[k][c]));
                }
            } else {
                {
                    FlowLink<GP, SP> U;
                    lup(k, U);
                    const typename F::Val v = fetch(nb[d].up, wu[d]);
                    if constexpr (SpinorFmt<SP>::scaled) mv_add<false>(w[0], U.u, hop_input_word<SP, R>(v, nu, f));
                    else if constexpr (direct) mv_add<false>(w[0], U.u, vneg_if(v, nu, f));
                    else mv_add<true>(w[k], U.u, vneg_if(v, nu));
                }
                {
                    FlowLink<GP, SP> U;
                    ldn(k, U);
                    const typename F::Val v = fetch(nb[d].dn, wd[d]);
                    if constexpr (SpinorFmt<SP>::scaled) mdv_sub(w[0], U.u, hop_input_word<SP, R>(v, nd, f));
                    else if constexpr (direct) mdv_sub(w[0], U.u, vneg_if(v, nd, f));
                    else mdv_sub(w[k], U.u, vneg_if(v, nd));
                }
                if constexpr (!direct && SPL == 1) vfma(acc, f, w[k]);
            }
        }
    }
    if constexpr (SPL == 1) {
        if constexpr (direct) acc = w[0];
    } else {
        __syncwarp();
#pragma unroll
        for (int m = 0; m < SPL; ++m) {
            const int src = W * m + site;
            if constexpr (direct) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    acc.c[c].re += __shfl_sync(0xffffffffu, w[0].c[c].re, src);
                    acc.c[c].im += __shfl_sync(0xffffffffu, w[0].c[c].im, src);
                }
            } else {
#pragma unroll
                for (int k = 0; k < ND; ++k) {
                    if constexpr (half) {
                        const unsigned long long f0 = f32x2_bcast(__shfl_sync(0xffffffffu, fu[k], src));
                        const unsigned long long f1 = f32x2_bcast(__shfl_sync(0xffffffffu, fd[k], src));
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            acc_f32x2(acc.c[c], f0, __half22float2(__shfl_sync(0xffffffffu, yu[k][c], src)));
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            acc_f32x2(acc.c[c], f1, __half22float2(__shfl_sync(0xffffffffu, yd[k][c], src)));
                    } else {
                        const R sm = __shfl_sync(0xffffffffu, sg[k], src);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            acc.c[c].re = fma(sm, __shfl_sync(0xffffffffu, w[k].c[c].re, src), acc.c[c].re);
                            acc.c[c].im = fma(sm, __shfl_sync(0xffffffffu, w[k].c[c].im, src), acc.c[c].im);
                        }
                    }
                }
            }
        }
    }
    return acc;
}

// 2 K in at the group's site in FP64, the two hops of a reliable update
// (ru_hop1, ru_hop2 of cg_site.cuh); a thread's products are added in the
// directions' order.  in(j): the vector of site j of the other parity.  Not
// inlined: it is rare, and would weigh on the iteration's registers.
template <int SPL, typename In>
__device__ __noinline__ Vec3<double> flow_ru_hop(const CgSys* S, int h, int q, int i, In in)
{
    constexpr int ND = 4 / SPL, W = 32 / SPL;
    const int Vh = S->g.Vh;
    const Coord c = eo_coords(S->g, q, i);
    Vec3<double> acc;
    vzero(acc);
#pragma unroll 1
    for (int k = 0; k < ND; ++k) {
        const int mu = h * ND + k, ju = lex_up(S->g, c, mu) >> 1, jd = lex_dn(S->g, c, mu) >> 1;
        const bool eta = eta_sign(c, mu) < 0;
        Vec3<double> u = mul_mv(GaugeFmt<GP_F64_18>::load(S->U64, q, mu, i, Vh), in(ju));
        Vec3<double> d = mul_adj_mv(GaugeFmt<GP_F64_18>::load(S->U64, 1 - q, mu, jd, Vh), in(jd));
        u = vneg_if(u, eta != (mu == 3 && c.x[3] == S->g.L[3] - 1));
        d = vneg_if(d, eta == (mu == 3 && c.x[3] == 0));
        if constexpr (ND == 1) {
            __syncwarp();
#pragma unroll
            for (int m = 0; m < SPL; ++m) {
                const int src = W * m + (threadIdx.x & (W - 1));
#pragma unroll
                for (int z = 0; z < 3; ++z) {
                    acc.c[z].re += __shfl_sync(0xffffffffu, u.c[z].re, src);
                    acc.c[z].im += __shfl_sync(0xffffffffu, u.c[z].im, src);
                }
#pragma unroll
                for (int z = 0; z < 3; ++z) {
                    acc.c[z].re += __shfl_sync(0xffffffffu, d.c[z].re, src);
                    acc.c[z].im += __shfl_sync(0xffffffffu, d.c[z].im, src);
                }
            }
        } else {
            vacc(acc, u, false);
            vacc(acc, d, false);
        }
    }
    if constexpr (ND > 1 && SPL > 1) {
        const Vec3<double> part = acc;
        __syncwarp();
        vzero(acc);
#pragma unroll
        for (int m = 0; m < SPL; ++m)
#pragma unroll
            for (int z = 0; z < 3; ++z) {
                acc.c[z].re += __shfl_sync(0xffffffffu, part.c[z].re, W * m + (threadIdx.x & (W - 1)));
                acc.c[z].im += __shfl_sync(0xffffffffu, part.c[z].im, W * m + (threadIdx.x & (W - 1)));
            }
    }
    return acc;
}

// one lane's scalars, advanced by every block of its team alike
struct FlowLane {
    double m2, bb, target, rr_old, rmax, rr_next, alpha, beta;
    int mode;    // LM_* of this iteration
    int next;    // of the next one
    int upd;     // this iteration's update still runs
    int was_ru;  // this iteration was a reliable update
    int iters, nru, status;
};

template <typename R>
__device__ __forceinline__ Vec3<R> sel(bool c, const Vec3<R>& a, const Vec3<R>& b)
{
    Vec3<R> o;
#pragma unroll
    for (int k = 0; k < 3; ++k) o.c[k] = {c ? a.c[k].re : b.c[k].re, c ? a.c[k].im : b.c[k].im};
    return o;
}

__device__ __forceinline__ bool flow_live(int mode) { return mode == LM_ACTIVE || mode == LM_RESTART; }

// the lane's step from its four sums: finish_lane of cg.cu on a copy of the
// lane's scalars
__device__ __forceinline__ void flow_finish(const CgArgs& a, FlowLane* L, const double* s)
{
    const int mode = L->mode;
    L->upd = 0;
    L->was_ru = 0;
    if (flow_live(mode)) {
        const double rr = s[3], pAp = s[0];
        const double alpha = rr / pAp;  // Fermions.cpp:573-586
        const double rr_next = rr - 2.0 * alpha * s[1] + alpha * alpha * s[2];
        const double beta = rr_next / rr;  // Fermions.cpp:594-601
        if (!isfinite(pAp) || fabs(pAp) < 1e-30 || !isfinite(alpha) || !isfinite(beta)) {
            L->next = LM_FAILED;
            L->status = SFH_ERR_BREAKDOWN;
            return;
        }
        L->alpha = alpha;
        L->beta = beta;
        L->rr_next = rr_next;
        L->iters += 1;
        L->upd = 1;
        L->next = LM_ACTIVE;
        if (!a.mixed) {
            if (rr_next < L->target) {  // Fermions.cpp:569
                L->next = LM_DONE;
            } else if (L->iters >= a.maxit) {  // Fermions.cpp:609-614
                L->next = LM_DONE;
                L->status = SFH_ERR_NOCONV;
            }
        } else {
            const double r = sqrt(fmax(rr_next, 0.0));
            if (rr_next < L->target || r < a.delta * L->rmax || L->iters >= a.maxit || rr_next > 4.0 * L->rr_old)
                L->next = LM_RU;
            else
                L->rmax = fmax(L->rmax, r);
        }
    } else if (mode == LM_RU) {  // s[3] = |b - M x|^2 in FP64
        const double rt = s[3], r_iter = L->rr_next;
        L->was_ru = 1;
        L->nru += 1;
        L->rr_next = rt;
        if (rt < L->target) {
            L->next = LM_DONE;
        } else if (!isfinite(rt)) {
            L->next = LM_FAILED;
            L->status = SFH_ERR_BREAKDOWN;
        } else if (L->iters >= a.maxit) {
            L->next = LM_DONE;
            L->status = SFH_ERR_NOCONV;
        } else {
            const bool restart = a.restart || rt > 0.5 * L->rr_old || rt > 1.5 * r_iter;
            L->rr_old = rt;
            L->rmax = sqrt(rt);
            L->next = restart ? LM_RESTART : LM_ACTIVE;
        }
    }
}

// every block of the team has arrived, and its writes are visible (fenced)
__device__ __forceinline__ void team_barrier(const FlowArgs& f, const FlowTeam& T, unsigned count, FlowCtx* c)
{
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(f.flags + blockIdx.x), "r"(count) : "memory");
#pragma unroll 1
    for (int b = threadIdx.x; b < T.nblk; b += blockDim.x) {
        unsigned v;
        int polls = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f.flags + T.blk0 + b) : "memory");
            if ((int)(v - count) >= 0 || !wait_on(c, polls)) break;
        }
    }
    __syncthreads();
}

// The CG sums of a team: up to kFlowEach blocks, each adds all the blocks' sums
// itself; above, the sums are shared out over the blocks, which publish each
// total in one copy per kFlowEach blocks.  Many readers of a word delay its
// writer: 64 blocks reading all of each other's sums took 11000 cycles, with
// shared-out sums 5500.
constexpr int kFlowEach = 8;

// the largest block: 255 registers a thread in FP64, 128 otherwise
template <int SP> struct FlowMax {
    static constexpr int threads = SP == SP_F64 ? 256 : 512;
};

// Four threads a site: every thread has one piece of a hop (ONE; flow_plan), whose
// neighbours and links it keeps in registers for the whole solve.
template <int GP, int SP, int SPL>
__global__ void __launch_bounds__(FlowMax<SP>::threads, 1) cg_flow(CgArgs a, FlowArgs f)
{
    constexpr bool ONE = SPL == 4;
    typedef typename GaugeFmt<GP>::R R;
    typedef typename SpinorFmt<SP>::R RS;
    typedef FlowVec<SP> F;
    constexpr int XP = XFmt<SP>::v;
    typedef FlowVec<XP> FX;
    typedef typename SpinorFmt<XP>::R RX;
    extern __shared__ __align__(16) char s_own[];
    __shared__ CgSys S;
    __shared__ FlowLane s_lane[kFlowMaxLanes];
    __shared__ double s_red[FlowMax<SP>::threads / 32][kFlowMaxLanes / 2 * kSums];
    __shared__ double s_tot[kFlowMaxLanes * kSums];
    __shared__ int s_live, s_ru;
    __shared__ FlowCtx s_ctx;
    __shared__ char* s_pub[kFlowMaxLanes / 2];
    __shared__ char* s_x[kFlowMaxLanes / 2];

    const FlowTeam T = f.teams[f.blk_team[blockIdx.x]];
    if (threadIdx.x == 0) {
        S = a.sys[T.sys];
        s_ctx.polls = f.polls;
        s_ctx.err = f.err;
        s_ctx.dead = 0;
        s_live = 1;
        s_ru = 0;
    }
    __syncthreads();
    const int Vh = S.g.Vh, nrhs = S.nrhs, both = S.both, nl = nrhs * (both ? 1 : 2), nm = nl * kSums;
    const int blk = (int)blockIdx.x - T.blk0;
    const int i0 = blk * T.n, n = min(T.n, Vh - i0), n2 = 2 * T.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = blockDim.x >> 1, nw = blockDim.x >> 5;
    const int q = (int)threadIdx.x >= half ? 1 : 0;  // this thread's parity
    const int s0 = (int)threadIdx.x - q * half;      // its own sites: s0, s0 + half, ...
    constexpr int W = 32 / SPL, ND = 4 / SPL;        // sites of a warp in a hop
    const int h = lane / W;                          // its share of a hop's directions
    // the hops' work, W sites of one RHS at a time: chunk c is RHS c / cpr;
    // the parity's warps take the chunks in turn
    const int cpr = (T.n + W - 1) / W, nchunk = nrhs * cpr, hw = nw >> 1, chunk0 = warp - q * hw;

    // the block's p, t, v and r of every RHS, in places j 2n + q n + s; the
    // neighbours of its sites
    const int N = nrhs * n2;
    constexpr int vb = F::own_bytes;
    const typename F::O op = F::array(s_own, N), ot = F::array(s_own + (size_t)vb * N, N),
                        ov = F::array(s_own + (size_t)2 * vb * N, N), orr = F::array(s_own + (size_t)3 * vb * N, N);
    NbrPair* s_nbr = reinterpret_cast<NbrPair*>(s_own + (size_t)4 * vb * N);  // [4][2 n]
    const int qn = q * T.n;
    auto lane_id = [&](int j, int par) { return both ? j : 2 * j + par; };
    auto global = [&](int field, int j) {  // this parity's part of a solver array, from the block's first site
        return F::array((char*)rhs_ptr(a, S.rhs0 + j, field) + (size_t)q * vb * Vh + (vb == 16 ? 16 : vb / 3) * (size_t)i0,
                        Vh);
    };
    auto xarr = [&](int j) {
        return FX::array(s_x[j] + (size_t)q * FX::own_bytes * Vh + (size_t)(FX::own_bytes / 3) * i0, Vh);
    };
    // a block that owns the whole system reads its own vectors only
    const bool pub = T.nblk > 1;

    if constexpr (!ONE)
#pragma unroll 1
        for (int m = 0; m < 4; ++m)
#pragma unroll 1
            for (int s = s0; s < n; s += half) s_nbr[m * n2 + qn + s] = nbr_pair(S.g, q, i0 + s, m, i0, n, T.n);
    if ((int)threadIdx.x < nl) {
        const CgLane* g = a.lanes + S.lane0 + threadIdx.x;
        FlowLane L;
        L.m2 = g->m2;
        L.bb = g->bb;
        L.target = g->target;
        L.rr_old = g->rr_old;
        L.rmax = g->rmax;
        L.rr_next = g->rr_next;
        L.alpha = L.beta = 0.0;
        L.mode = L.next = g->mode[0];
        L.upd = L.was_ru = 0;
        L.iters = L.nru = 0;
        L.status = SFH_OK;
        s_lane[threadIdx.x] = L;
    }
    if ((int)threadIdx.x < nrhs) {
        s_pub[threadIdx.x] = f.pub[S.rhs0 + threadIdx.x];
        s_x[threadIdx.x] = (char*)rhs_ptr(a, S.rhs0 + threadIdx.x, F_XLO);
    }
    __syncthreads();
    // the state after cg_init: r = p = b, x = 0
#pragma unroll 1
    for (int j = 0; j < nrhs; ++j)
#pragma unroll 1
        for (int s = s0; s < n; s += half) {
            const typename F::Val p = global(F_P, j).ld(s);
            op.st(j * n2 + qn + s, p);
            orr.st(j * n2 + qn + s, p);
            if (pub) F::publish(s_pub[j], 2 * Vh, q * Vh + i0 + s, p, 1u);
        }
    // ONE: this thread's site, neighbours and links
    const int j1 = chunk0 / cpr, g1 = (chunk0 - j1 * cpr) * W + lane % W;
    NbrPair nb1[ONE ? ND : 1];
    FlowLink<GP, SP> lu1[ONE ? ND : 1], ld1[ONE ? ND : 1];
    if constexpr (ONE) {
        const int i = i0 + min(g1, n - 1);
        const Coord c = eo_coords(S.g, q, i);
#pragma unroll
        for (int k = 0; k < ND; ++k) {
            const int mu = h * ND + k;
            nb1[k] = nbr_pair(S.g, q, i, mu, i0, n, T.n);
            lu1[k].load(S.Ulo, q, mu, i, Vh);
            ld1[k].load(S.Ulo, 1 - q, mu, lex_dn(S.g, c, mu) >> 1, Vh);
        }
    }
    __syncthreads();

    // K of the published vector t at site s of RHS j (all threads of the group)
    auto hop = [&](int t, int j, int s, unsigned tag) -> Vec3<R> {
        FlowIn<SP> in;
        in.pub = s_pub[j] + (size_t)t * F::pub_bytes * 2 * Vh;
        in.own = t == 0 ? op : ot;
        in.own.e += j * n2;
        in.N2 = 2 * Vh;
        in.tag = tag;
        if constexpr (ONE) {
            return flow_hop<GP, SP, SPL>(
                &s_ctx, in, [&](int k) { return nb1[k]; }, [&](int k, FlowLink<GP, SP>& L) { L = lu1[k]; },
                [&](int k, FlowLink<GP, SP>& L) { L = ld1[k]; });
        } else {
            const int i = i0 + s;
            const NbrPair* nbr = s_nbr + h * ND * n2 + qn + s;
            return flow_hop<GP, SP, SPL>(
                &s_ctx, in, [&](int k) { return nbr[k * n2]; },
                [&](int k, FlowLink<GP, SP>& L) { L.load(S.Ulo, q, h * ND + k, i, Vh); },
                [&](int k, FlowLink<GP, SP>& L) {
                    // the backward neighbour's checkerboard index, from its place
                    const int d = nbr[k * n2].dn, at = d & kNbrIdx;
                    const int jd = (d & kNbrOwn) ? at - (1 - q) * T.n + i0 : at - (1 - q) * Vh;
                    L.load(S.Ulo, 1 - q, h * ND + k, jd, Vh);
                });
        }
    };

    unsigned bars = 0;
    for (int k = 0; k < a.maxloop && s_live; ++k) {
        const unsigned tag = (unsigned)k + 1u;
        const bool ru = s_ru != 0;  // uniform over the team
        if (ru) {
            // the lanes due for a reliable update put their p and r into the
            // global arrays that ru_residual works on
#pragma unroll 1
            for (int j = 0; j < nrhs; ++j) {
                if (s_lane[lane_id(j, q)].mode != LM_RU) continue;
#pragma unroll 1
                for (int s = s0; s < n; s += half) {
                    global(F_P, j).st(s, op.ld(j * n2 + qn + s));
                    global(F_R, j).st(s, orr.ld(j * n2 + qn + s));
                }
            }
            team_barrier(f, T, ++bars, &s_ctx);
        }
        // t = K p on this thread's parity, for the lanes of the other one
#pragma unroll 1
        for (int c = chunk0; c < nchunk; c += hw) {
            const int j = ONE ? j1 : (nrhs == 1 ? 0 : c / cpr), g = ONE ? g1 : (c - j * cpr) * W + lane % W;
            const int s = min(g, n - 1), i = i0 + s;
            const int mode = s_lane[lane_id(j, 1 - q)].mode;
            if (flow_live(mode)) {
                const Vec3<R> acc = hop(0, j, s, tag);
                if (g < n) {
                    const typename F::Val t = F::pack(vcvt<RS>(acc));
                    if (pub) {
                        char* w = s_pub[j] + (size_t)F::pub_bytes * 2 * Vh;
                        if constexpr (SPL == 1) F::publish(w, 2 * Vh, q * Vh + i, t, tag);
                        else F::template publish_part<SPL>(w, 2 * Vh, q * Vh + i, t, tag, h);
                    }
                    if (h == SPL - 1) ot.st(j * n2 + qn + s, t);
                }
            } else if (SP != SP_F64 && mode == LM_RU) {
                const void *xhi = rhs_ptr(a, S.rhs0 + j, F_XHI), *xlo = s_x[j];
                Vec3<double> acc = flow_ru_hop<SPL>(&S, h, q, i, [=](int jn) {
                    return vaxpy(SpinorFmt<SP_F64>::load_cg(xhi, 1 - q, jn, Vh), 1.0,
                                 vcvt<double>(SpinorFmt<XP>::load_cg(xlo, 1 - q, jn, Vh)));
                });
#pragma unroll
                for (int z = 0; z < 3; ++z) acc.c[z] = {0.5 * acc.c[z].re, 0.5 * acc.c[z].im};
                if (g < n && h == 0) SpinorFmt<SP_F64>::store(rhs_ptr(a, S.rhs0 + j, F_THI), q, i, Vh, acc);
            }
        }
        if (ru) team_barrier(f, T, ++bars, &s_ctx);
        else __syncthreads();
        // v = m^2 p - K t on the lanes' own parity; thread h of a site adds
        // the site's terms of sums h, h + SPL, ...
        if (lane < nrhs * kSums) s_red[warp][lane] = 0.0;
        __syncwarp();
        {
            double sum[ND] = {};
            int jsum = -1;  // the RHS that sum holds
            auto flush = [&]() {
                if (jsum < 0) return;
#pragma unroll
                for (int m = 0; m < ND; ++m) {
#pragma unroll
                    for (int o = W / 2; o > 0; o >>= 1) sum[m] += __shfl_xor_sync(0xffffffffu, sum[m], o);
                    if (lane % W == 0) s_red[warp][jsum * kSums + m * SPL + h] = sum[m];
                    sum[m] = 0.0;
                }
            };
#pragma unroll 1
            for (int c = chunk0; c < nchunk; c += hw) {
                const int j = ONE ? j1 : (nrhs == 1 ? 0 : c / cpr), g = ONE ? g1 : (c - j * cpr) * W + lane % W;
                const int s = min(g, n - 1), at = j * n2 + qn + s;
                if (!ONE && j != jsum) flush();
                jsum = j;
                const FlowLane& L = s_lane[lane_id(j, q)];
                if (flow_live(L.mode)) {
                    const R m2 = (R)L.m2;
                    const Vec3<R> acc = hop(1, j, s, tag);
                    const Vec3<RS> r = F::vec(orr.ld(at)), p = F::vec(op.ld(at));
                    const Vec3<R> pr = vcvt<R>(p);
                    Vec3<R> w;
#pragma unroll
                    for (int z = 0; z < 3; ++z) {
                        w.c[z].re = fma(m2, pr.c[z].re, -acc.c[z].re);
                        w.c[z].im = fma(m2, pr.c[z].im, -acc.c[z].im);
                    }
                    const typename F::Val vw = F::pack(vcvt<RS>(w));
                    const Vec3<RS> vn = F::vec(vw);
                    if (g < n) {
                        if (h == SPL - 1) ov.st(at, vw);
#pragma unroll
                        for (int m = 0; m < ND; ++m) {
                            const int f4 = m * SPL + h;  // <p,v>, <r,v>, |v|^2, |r|^2
                            sum[m] += site_dot(sel(f4 == 0, p, sel(f4 == 2, vn, r)), sel(f4 == 3, r, vn));
                        }
                    }
                } else if (SP != SP_F64 && L.mode == LM_RU) {
                    const void* thi = rhs_ptr(a, S.rhs0 + j, F_THI);
                    const Vec3<double> acc = flow_ru_hop<SPL>(
                        &S, h, q, i0 + s, [=](int jn) { return SpinorFmt<SP_F64>::load_cg(thi, 1 - q, jn, Vh); });
                    if (g < n && h == SPL - 1)
                        sum[ND - 1] += ru_residual<SP, XP>(a.rhs, Vh, q, i0 + s, S.rhs0 + j, L.m2, acc);
                }
            }
            flush();
        }
        __syncthreads();
        // the block's sums, then the team's, added in the blocks' order: by
        // every block for itself in a small team; in a large one the sums are
        // shared out over the blocks, which publish the totals
        const int copies = (T.nblk + kFlowEach - 1) / kFlowEach;
        uint4* words = f.sums + T.words0 + (size_t)(k & 1) * (T.nblk + copies) * nm;
        uint4* totals = words + (size_t)T.nblk * nm;
        const bool each = copies == 1;
#pragma unroll 1
        for (int m = threadIdx.x; m < nm; m += blockDim.x) {
            const int l = m / kSums, j = both ? l : l >> 1, c = j * kSums + m % kSums;
            const int w0 = both ? 0 : (l & 1) * hw, w1 = both ? nw : w0 + hw;
            double x = 0.0;
#pragma unroll 4
            for (int w = w0; w < w1; ++w) x += s_red[w][c];
            if (pub)
                st_word(words + (size_t)m * T.nblk + blk, make_uint4((unsigned)__double2loint(x),
                                                                     (unsigned)__double2hiint(x), 0u, tag));
            else
                s_tot[m] = x;
        }
        if (pub) {
#pragma unroll 1
            for (int m = warp; m < nm; m += nw) {
                if (!each && m * T.nblk / nm != blk) continue;
                const uint4* from = words + (size_t)m * T.nblk;
                double x = 0.0;
#pragma unroll 1
                for (int b0 = 0; b0 < T.nblk; b0 += 160) {  // five words in flight per lane
                    uint4 w[5];
#pragma unroll
                    for (int u = 0; u < 5; ++u)
                        if (b0 + 32 * u + lane < T.nblk) w[u] = ld_word(from + b0 + 32 * u + lane);
#pragma unroll
                    for (int u = 0; u < 5; ++u) {
                        const int b = b0 + 32 * u + lane;
                        if (b >= T.nblk) continue;
                        int polls = 0;
                        while (w[u].w != tag && wait_on(&s_ctx, polls)) w[u] = ld_word(from + b);
                        x += __hiloint2double((int)w[u].y, (int)w[u].x);
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (each) {
                    if (lane == 0) s_tot[m] = x;
                } else {
                    for (int r = lane; r < copies; r += 32)
                        st_word(totals + r * nm + m,
                                make_uint4((unsigned)__double2loint(x), (unsigned)__double2hiint(x), 0u, tag));
                }
            }
            if (!each) {
#pragma unroll 1
                for (int m = threadIdx.x; m < nm; m += blockDim.x) {
                    const uint4* from = totals + (size_t)(blk / kFlowEach) * nm + m;
                    uint4 w = ld_word(from);
                    int polls = 0;
                    while (w.w != tag && wait_on(&s_ctx, polls)) w = ld_word(from);
                    s_tot[m] = __hiloint2double((int)w.y, (int)w.x);
                }
            }
        }
        __syncthreads();
        if (warp == 0) {
            int next = LM_DONE;
            if (lane < nl) {
                flow_finish(a, s_lane + lane, s_tot + lane * kSums);
                next = s_lane[lane].next;
            }
            const unsigned live = __ballot_sync(0xffffffffu, flow_live(next) || next == LM_RU);
            const unsigned due = __ballot_sync(0xffffffffu, next == LM_RU);
            if (lane == 0) {
                s_live = live != 0;
                s_ru = due != 0;
            }
        }
        __syncthreads();
        // x += alpha p, r -= alpha v, p = r + beta p on the block's own sites
#pragma unroll 1
        for (int u = s0; u < nrhs * n; u += half) {
            const int j = nrhs == 1 ? 0 : u / n, s = u - j * n, at = j * n2 + qn + s;
            const FlowLane& L = s_lane[lane_id(j, q)];
            if (L.upd) {
                const typename FX::O xo = xarr(j);
                const Vec3<RX> x = xo.ld(s);
                const Vec3<RS> p = F::vec(op.ld(at)), r = F::vec(orr.ld(at)), v = F::vec(ov.ld(at));
                const typename F::Val rn = F::pack(vaxpy(r, (RS)(-L.alpha), v));
                const typename F::Val pn = F::pack(vaxpy(F::vec(rn), (RS)L.beta, p));
                if (pub && flow_live(L.next)) F::publish(s_pub[j], 2 * Vh, q * Vh + i0 + s, pn, tag + 1u);
                orr.st(at, rn);
                op.st(at, pn);
                xo.st(s, vaxpy(x, (RX)L.alpha, vcvt<RX>(p)));
            } else if (L.was_ru && flow_live(L.next)) {
                // the updated residual and direction (p = r on a restart)
                const typename F::Val r = global(F_R, j).ld(s);
                const typename F::Val p = L.next == LM_RESTART ? r : global(F_P, j).ld(s);
                if (pub) F::publish(s_pub[j], 2 * Vh, q * Vh + i0 + s, p, tag + 1u);
                op.st(at, p);
                orr.st(at, r);
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < nl) s_lane[threadIdx.x].mode = s_lane[threadIdx.x].next;
        if (threadIdx.x == 0 && s_ctx.dead) s_live = 0;
        __syncthreads();
    }
    if (blk == 0 && (int)threadIdx.x < nl) {  // the lanes' final state
        CgLane* g = a.lanes + S.lane0 + threadIdx.x;
        const FlowLane& L = s_lane[threadIdx.x];
        g->mode[0] = g->mode[1] = L.mode;
        g->status = L.status;
        g->iters = L.iters;
        g->nru = L.nru;
        g->rr_next = L.rr_next;
        g->rr_old = L.rr_old;
        g->rmax = L.rmax;
        g->alpha = L.alpha;
        g->beta = L.beta;
    }
}

}  // namespace

static int vec_format(int prec)
{
    return prec == SFH_PREC_F64 ? SP_F64 : (prec == SFH_PREC_F16 ? SP_F16 : (prec == SFH_PREC_BF16 ? SP_BF16 : SP_F32));
}

static size_t pub_bytes(int prec)
{
    const int sp = vec_format(prec);
    return sp == SP_F64 ? FlowVec<SP_F64>::pub_bytes
                        : (sp == SP_F32 ? FlowVec<SP_F32>::pub_bytes : FlowVec<SP_F16>::pub_bytes);
}

// bytes of shared memory of a block of n sites per parity: p, t, v and r of
// every RHS, and the neighbours
static size_t block_bytes(int prec, int n, int nrhs)
{
    const int sp = vec_format(prec);
    return (size_t)2 * n * (nrhs * 4 * (sp == SP_F64 ? 48 : (sp == SP_F32 ? 24 : 16)) + 4 * sizeof(NbrPair));
}

// 208 of the 227 KB that a block may have: up to 6 go to its other arrays, and
// what the SM has left caches the links.  With one RHS FP32 meets this line at
// 832 sites, where the per-phase kernels catch up (20^3 30, 811 sites, 10.7 ms;
// 20^3 32, 865 sites, by these 11.7), and FP64 at 474 (16^3 32, 443 sites, 10.7
// ms either way); the 16-bit formats and several RHS in FP64 meet others first.
constexpr size_t kFlowMaxSmem = 208 * 1024;
// Checkerboard sites per parity and block: at least 32, so that a warp's
// words are whole lines (4^4 in one block 7.3 us, in four 5.9); site-lanes at
// most 1024, where the per-phase kernels catch up (FP16 at 886: 50 us against
// 54; FP64 at 443: 53 against 58).
constexpr int kFlowMinSites = 32;
constexpr int kFlowMaxSiteLanes = 1024;

// The GPU's SMs (one block each) are shared out so that the largest number of
// site-lanes of a block is as small as it gets.
bool flow_plan(const std::vector<CgSys>& sys, int prec, int num_sms, FlowPlan* plan)
{
    *plan = FlowPlan();
    if (sys.empty() || (int)sys.size() > num_sms) return false;
    for (const CgSys& S : sys)
        if (S.nrhs < 1 || S.nrhs > kFlowMaxLanes / 2) return false;
    auto share = [](const CgSys& S, int work) {  // sites per parity and block
        return std::min(S.g.Vh, std::max(kFlowMinSites / S.nrhs, work / S.nrhs));
    };
    auto blocks = [&](int work) {
        long n = 0;
        for (const CgSys& S : sys) n += (S.g.Vh + share(S, work) - 1) / share(S, work);
        return n;
    };
    if (blocks(kFlowMaxSiteLanes) > num_sms) return false;
    int lo = 1, hi = kFlowMaxSiteLanes;  // the smallest work per block that fits
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (blocks(mid) <= num_sms) hi = mid;
        else lo = mid + 1;
    }
    for (int k = 0; k < (int)sys.size(); ++k) {
        const CgSys& S = sys[k];
        FlowTeam t;
        t.sys = k;
        t.blk0 = (int)plan->blk_team.size();
        t.nblk = (S.g.Vh + share(S, lo) - 1) / share(S, lo);
        t.n = (S.g.Vh + t.nblk - 1) / t.nblk;  // even shares
        t.nblk = (S.g.Vh + t.n - 1) / t.n;     // none empty
        t.words0 = (int)plan->words;
        plan->words += (size_t)2 * (t.nblk + (t.nblk + kFlowEach - 1) / kFlowEach) * S.nrhs * (S.both ? 1 : 2) * kSums;
        plan->blk_team.insert(plan->blk_team.end(), t.nblk, k);
        for (int j = 0; j < S.nrhs; ++j) {
            plan->pub_at.push_back(plan->pub_bytes);
            plan->pub_bytes += (pub_bytes(prec) * 4 * S.g.Vh + 15) / 16 * 16;
        }
        plan->dyn = std::max(plan->dyn, block_bytes(prec, t.n, S.nrhs));
        plan->teams.push_back(t);
    }
    // as many threads per site as keep a hop to one round
    const int most = prec == SFH_PREC_F64 ? FlowMax<SP_F64>::threads : FlowMax<SP_F32>::threads;
    plan->split = 1;
    auto warps = [&](int split) {  // of one parity, for a hop in one round
        int n = 0;
        for (const FlowTeam& t : plan->teams) n = std::max(n, sys[t.sys].nrhs * ((split * t.n + 31) / 32));
        return n;
    };
    if (prec == SFH_PREC_F64 || prec == SFH_PREC_F32 || prec == SFH_PREC_F16)
        while (plan->split < 4 && 64 * warps(2 * plan->split) <= most) plan->split *= 2;
    const int all = warps(plan->split);
    plan->rounds = (64 * all + most - 1) / most;
    plan->threads = 64 * ((all + plan->rounds - 1) / plan->rounds);
    if (plan->dyn > kFlowMaxSmem) return false;
    // FP64 serves the RHS of a block one after the other, round by round, where
    // the per-phase kernels take a link for two: from five rounds on, with more
    // than four RHS from four on, these are the faster ones (12^4 with 6 RHS
    // 6.9 ms against 5.8, with 5 5.8 against 5.4; 16^4 with 2 6.0 against 6.1)
    int rhs = 1;
    for (const CgSys& S : sys) rhs = std::max(rhs, S.nrhs);
    return prec != SFH_PREC_F64 || plan->rounds <= (rhs > 4 ? 3 : 4);
}

// By the rounds of a hop, which serve the RHS of a block one after the other
// where the per-phase kernels share a link's load.  Best schedule / dataflow,
// five precisions: one RHS, three rounds 1.01 to 1.24, four 1.00; two to four
// RHS, two rounds 1.03 to 1.23, three 0.91 to 1.17; five to eight RHS, one round
// 1.08 to 1.38, two 0.86 to 1.07.
bool flow_beats_tuned(const std::vector<CgSys>& sys, const FlowPlan& plan)
{
    int most = 1;
    for (const CgSys& S : sys) most = std::max(most, S.nrhs);
    return plan.rounds <= (most == 1 ? 3 : (most <= 4 ? 2 : 1));
}

cudaError_t flow_launch(int prec, const CgArgs& a, const FlowArgs& f, const FlowPlan& plan, cudaStream_t stream)
{
    typedef void (*Kernel)(CgArgs, FlowArgs);
    // links in registers only where a thread has one direction (four threads a
    // site): 18 to 72 of its 128 or 255 (a hop of 8^3 16 in FP32 2700 cycles
    // against 4200)
    const int sl = plan.split / 2;
    static const Kernel f64[3] = {cg_flow<GP_F64_18, SP_F64, 1>, cg_flow<GP_F64_18, SP_F64, 2>,
                                  cg_flow<GP_F64_18, SP_F64, 4>};
    static const Kernel f32[3] = {cg_flow<GP_F32_12, SP_F32, 1>, cg_flow<GP_F32_12, SP_F32, 2>,
                                  cg_flow<GP_F32_12, SP_F32, 4>};
    static const Kernel f16[3] = {cg_flow<GP_F16_12, SP_F16, 1>, cg_flow<GP_F16_12, SP_F16, 2>,
                                  cg_flow<GP_F16_12, SP_F16, 4>};
    const Kernel k = prec == SFH_PREC_F64      ? f64[sl]
                     : prec == SFH_PREC_F32    ? f32[sl]
                     : prec == SFH_PREC_F16    ? f16[sl]
                     : prec == SFH_PREC_F32_18 ? cg_flow<GP_F32_18, SP_F32, 1>
                                               : cg_flow<GP_BF16_12, SP_BF16, 1>;
    // the same limit from every handle: it belongs to the kernel, and another
    // thread may be about to launch it with more than this plan takes
    cudaError_t e = cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlowMaxSmem);
    if (e != cudaSuccess) return e;
    CgArgs ca = a;
    FlowArgs fa = f;
    void* args[] = {&ca, &fa};
    return cudaLaunchCooperativeKernel((const void*)k, dim3((unsigned)plan.blk_team.size()), dim3(plan.threads), args,
                                       plan.dyn, stream);
}

}  // namespace sfh
