// Pieces shared by the uniform-cube step kernels: 16-byte row vectors, lane exchange, the occupancy
// floor per variant, and the BGK relaxation of V cells held in registers.
//
// The pull step (uniform.cu) and the in-place AA steps (uniform_aa.cu) relax with the same
// CellBgk code, so for the same collision inputs they produce the same bits.
#pragma once

#include <type_traits>
#include <utility>

#include "kernels.h"
#include "lattice.cuh"

namespace jp {

// ---- vector access helpers ---------------------------------------------------------------------

template <class RAW, int V>
struct Pack {
    static constexpr int bytes = int(sizeof(RAW)) * V;
    using word = typename std::conditional<bytes == 16, uint4,
                 typename std::conditional<bytes == 8, uint2,
                 typename std::conditional<bytes == 4, unsigned int, unsigned short>::type>::type>::type;
    union {
        word w;
        RAW v[V];
        unsigned int u32[(bytes + 3) / 4];
    };
};

// The steps' source array: a plain load.  Not the read-only path (__ldg): a step launched by launch_step is
// resident while its predecessor still writes that array, and only ordinary loads are ordered after step_wait
// (the two are as fast: N=512 FP32 1890 us by plain loads, 1888 by __ldg, FP16 1582 and 1591).
template <class RAW, int V>
__device__ __forceinline__ Pack<RAW, V> ld_step(const RAW* p) {
    Pack<RAW, V> r;
    r.w = *reinterpret_cast<const typename Pack<RAW, V>::word*>(p);
    return r;
}
// read-only for the kernel's lifetime
template <class RAW, int V>
__device__ __forceinline__ Pack<RAW, V> ld_pack(const RAW* p) {
    Pack<RAW, V> r;
    r.w = __ldg(reinterpret_cast<const typename Pack<RAW, V>::word*>(p));
    return r;
}
// coherent load at L2, for an array the same kernel writes (the in-place steps)
template <class RAW, int V>
__device__ __forceinline__ Pack<RAW, V> ld_pack_cg(const RAW* p) {
    Pack<RAW, V> r;
    r.w = __ldcg(reinterpret_cast<const typename Pack<RAW, V>::word*>(p));
    return r;
}
template <class RAW, int V>
__device__ __forceinline__ void st_pack(RAW* p, const Pack<RAW, V>& r) {
    __stcs(reinterpret_cast<typename Pack<RAW, V>::word*>(p), r.w);
}
template <class RAW, int V>
__device__ __forceinline__ void zero_pack(Pack<RAW, V>& r) {
#pragma unroll
    for (int i = 0; i < (Pack<RAW, V>::bytes + 3) / 4; ++i) r.u32[i] = 0u;
}

template <class RAW> __device__ __forceinline__ RAW ld_one(const RAW* p) { return __ldg(p); }
template <> __device__ __forceinline__ uint16_t ld_one<uint16_t>(const uint16_t* p) {
    return __ldg(reinterpret_cast<const unsigned short*>(p));
}

template <class RAW> __device__ __forceinline__ RAW shfl_up1(RAW v) { return __shfl_up_sync(0xffffffffu, v, 1); }
template <class RAW> __device__ __forceinline__ RAW shfl_dn1(RAW v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <> __device__ __forceinline__ uint16_t shfl_up1<uint16_t>(uint16_t v) {
    return (uint16_t)__shfl_up_sync(0xffffffffu, (unsigned)v, 1);
}
template <> __device__ __forceinline__ uint16_t shfl_dn1<uint16_t>(uint16_t v) {
    return (uint16_t)__shfl_down_sync(0xffffffffu, (unsigned)v, 1);
}
template <class T> __device__ __forceinline__ T shfl_from(T v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
template <> __device__ __forceinline__ uint16_t shfl_from<uint16_t>(uint16_t v, int lane) {
    return (uint16_t)__shfl_sync(0xffffffffu, (unsigned)v, lane);
}

// Programmatic dependent launch: a step launched with launch_step below may start while its predecessor in the
// stream drains.  Every thread waits for the predecessor's completion (and its writes) before it touches a
// state array (step_wait), and step_release lets the successor's CTAs take their places once every CTA of
// this grid has called it or ended.  Both are no-ops in a plain launch.  A CTA that does not call it lets them in at
// its end, which still hides their launch.
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void step_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Whether the CTAs of a lone cube's step release at once.  Successors that come early are dealt to the SMs with
// room, unevenly, so where the grid is about a wave they double up on some SMs; over several waves they fill the
// last one's gaps.  us per step, released at once / at the end: FP32 N=8 2.08 / 1.70, N=32 2.92 / 2.87, N=56 4.64 / 4.23,
// N=64 5.36 / 5.26, N=72 6.62 / 6.68, N=128 34.0 / 34.4, N=192 109.7 / 110.8;
// FP16 N=24 2.24 / 2.34, N=32 2.95 / 2.36, N=48 3.21 / 3.01, N=56 4.46 / 3.98, N=64 4.31 / 4.50, N=80 6.54 / 6.79;
// FP64 N=32 28.6 / 11.3 (a CTA keeps its SM's FP64 pipe busy).
// The two-step pass (N=8, 32, 128 and 192 above) goes by the same rule, for its figures alone: its CTAs fill an SM's
// registers each and its grid has at most one per SM, so a successor's CTA takes an SM that has none or whose
// CTA has ended; that is worth 1 % either way.
[[maybe_unused]] static bool release_early(bool shifted, bool fp64, int n) {
    const long long cells = (long long)n * n * n;
    if (fp64) return false;
    return shifted ? cells < 20000 || cells > 200000 : cells > 300000;
}
// launch with programmatic stream serialization
template <class K, class A>
static cudaError_t launch_step(K kern, unsigned grid, int threads, int smem, cudaStream_t st, const A& arg) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kern, arg);
}

// Occupancy floor per SM for a variant: the wide-vector variants need warps (to keep 19 vector
// loads per thread in flight, and for the issue-bound 16-bit collision) more than registers:
// FP32 V=4 and 16-bit V=4 to 128 registers, 16-bit V=8 to 168.
template <class ST, int V, int TPB>
constexpr int min_blocks() {
    return (sizeof(typename ST::raw) * V == 16 && sizeof(typename ST::raw) == 2) ? (384 / TPB > 0 ? 384 / TPB : 1)
         : (sizeof(typename ST::raw) * V >= 8 && sizeof(typename ST::raw) <= 4) ? (512 / TPB > 0 ? 512 / TPB : 1) : 1;
}

// ---- BGK relaxation of V cells ------------------------------------------------------------------
// f[v][q] holds the collision inputs of cell v in the collision type R: the shifts g = f - w_q when SA (FP32
// shifts on load), f itself for FP64.
//
// FP32: Blackwell issues two FP32 adds, multiplies or FMAs in one instruction (f32x2; __fadd2_rn,
// __fmul2_rn, __ffma2_rn, each lane rounded to nearest like its scalar op).  The FP32 steps hold V = 2,
// 4 or 8 cells per thread, so the relaxation runs on pairs of cells and issues half the FP32
// instructions; an odd V runs the same sequence on single floats.  FP64 runs it on single doubles.  Every
// operation is spelled out, so a cell's result does not depend on V, and the pull, two-step and in-place steps, which
// share this code, produce the same bits.  (The packed intrinsics keep each rounding, but the compiler may
// still merge a packed product into the sum that alone uses it; where it does, LaneBgk::pair says FMA.)  The
// sequence per cell, 117 operations and a reciprocal (the FP64 step is bound by its FP64 rate; FP32 merges one
// product):
//   S_q = g_q + g_opp, D_q = g_q - g_opp; s = g0 + the S, j = the signed sums of the D, in sum_order
//   rho = 1 + s (s itself in FP64), inv = 1 / rho (IEEE), e = s - 1.5 inv (jx jx + jy jy + jz jz) (two FMAs)
//   out0 = (1-om) g0 + om w0 e
//   a = (3 om w) (c_q . j), t = om w e + (1/(2 om w) inv) a a   [= om w rho (4.5 (c.u)^2 - 1.5 u.u) + om w s]
//   u = (1-om)/2 S + t, v = (1-om)/2 D + a; out_q = u + v, out_opp(q) = u - v.
// Measured against one product chain per population (147 operations; the 16-bit storages keep it, CellBgk16):
// error against 64 bits of N=64 FP32 after 200 steps 1.4-1.8e-7 -> 1.1-1.5e-7.
// order in which the pairs enter the sums: those with c_z = 0 first, as a sweep along z has them
__host__ __device__ constexpr int sum_order(int i) {
    constexpr int t[Q / 2] = {1, 3, 7, 9, 5, 11, 13, 15, 17};
    return t[i];
}
// the coefficients of a launch's cube: FP32's come with it (bgk_coefficients); FP64's need no such care
template <class R>
__device__ __forceinline__ BgkCoefOf<R> bgk_of(const UniSolve& d) {
    if constexpr (sizeof(R) == 4) {
        return d.bgk;
    } else {
        const double om = d.omega_d, a2 = om * (1.0 / 12.0);
        return {om, 0.5 * fma(-8.0, a2, om), a2, om * wgt<double>(0), om * wgt<double>(1), om * wgt<double>(7),
                d.half_inv_d * 18.0, d.half_inv_d * 36.0};
    }
}
// One lane set T (a float, a double, a pair of floats) of the sequence.  SA: the inputs are shifts.
template <class T, bool SA>
struct LaneBgk {
    using L = Lanes<T>;
    using R = typename L::real;
    R om;
    T s, jx, jy, jz;  // sum and momentum; finish() turns s into e
    T inv;            // 1 / rho
    T k, b, ax, ay, az;  // of the class at hand (faces, edges)

    BgkCoefOf<R> co;

    __device__ __forceinline__ LaneBgk(const BgkCoefOf<R>& c) : om(c.om), co(c) {}

    __device__ __forceinline__ void add_rest(T g0) { s = g0; }
    // the pair (q, q+1), in the order q = sum_order(0), sum_order(1), ...: ga, gb become S, D
    __device__ __forceinline__ void add(int q, T& ga, T& gb) {
        const T S = L::add(ga, gb), D = L::sub(ga, gb);
        s = L::add(s, S);
        if (cx(q) != 0) jx = q == 1 ? D : L::add(jx, D);
        if (cy(q) != 0) jy = q == 3 ? D : cy(q) > 0 ? L::add(jy, D) : L::sub(jy, D);
        if (cz(q) != 0) jz = q == 5 ? D : cz(q) > 0 ? L::add(jz, D) : L::sub(jz, D);
        ga = S;
        gb = D;
    }
    __device__ __forceinline__ void finish() {
        inv = L::rcp(SA ? L::add(L::bc(R(1)), s) : s);
        T t = L::mul(jx, jx);
        t = L::fma(jy, jy, t);
        t = L::fma(jz, jz, t);
        s = L::fma(L::mul(L::bc(R(-1.5)), inv), t, s);
    }
    __device__ __forceinline__ T rest(T g0) const {
        return L::fma(L::bc(R(1) - om), g0, L::mul(L::bc(co.b0), s));
    }
    // relaxed populations q and q+1 = opp(q) (q odd, ascending from 1) from S and D
    __device__ __forceinline__ void pair(int q, T S, T D, T& oa, T& ob) {
        if (q == 1 || q == 7) {
            const R w = q == 1 ? co.a1 : co.a2;
            b = L::mul(L::bc(q == 1 ? co.b1 : co.b2), s);
            k = L::mul(L::bc(q == 1 ? co.k1 : co.k2), inv);
            ax = L::mul(L::bc(w), jx);
            ay = L::mul(L::bc(w), jy);
            az = L::mul(L::bc(w), jz);
        }
        // om times the antisymmetric part: 3 om w c.j (c's first non-zero component is positive for odd q).  FP32: the
        // product by jx and the sum in one FMA for the edges along x, which the compiler makes of a packed
        // product and sum that have no other use for the product; written out, single floats take it too.
        T a = cx(q) != 0 ? ax : (cy(q) != 0 ? ay : az);
        if ((cx(q) != 0) + (cy(q) != 0) + (cz(q) != 0) == 2) {
            const bool plus = cz(q) != 0 ? cz(q) > 0 : cy(q) > 0;
            const T other = cz(q) != 0 ? az : ay;
            if (sizeof(R) == 4 && cx(q) != 0) a = L::fma(L::bc(co.a2), jx, plus ? other : L::neg(other));
            else a = plus ? L::add(a, other) : L::sub(a, other);
        }
        const T t = L::fma(L::mul(k, a), a, b);  // om times the symmetric part
        const T h = L::bc(R(0.5) * (R(1) - om));
        const T u = L::fma(h, S, t), v = L::fma(h, D, a);
        oa = L::add(u, v);
        ob = L::sub(u, v);
    }
};

template <class R, int V, bool SA>
struct CellBgk {
    static constexpr bool PAIR = sizeof(R) == 4 && V % 2 == 0;
    static constexpr int NP = PAIR ? V / 2 : V;  // lane sets
    using T = typename std::conditional<PAIR, float2, R>::type;
    LaneBgk<T, SA> c[NP];
    T orest[NP];
    T S[NP][Q / 2], D[NP][Q / 2];

    template <int... I>
    __device__ __forceinline__ CellBgk(const BgkCoefOf<R>& co, std::integer_sequence<int, I...>)
        : c{((void)I, LaneBgk<T, SA>(co))...} {}
    __device__ __forceinline__ CellBgk(const BgkCoefOf<R>& co) : CellBgk(co, std::make_integer_sequence<int, NP>{}) {}

    static __device__ __forceinline__ T get(const R (&f)[V][Q], int p, int q) {
        if constexpr (PAIR) return make_float2(f[2 * p][q], f[2 * p + 1][q]);
        else return f[p][q];
    }
    static __device__ __forceinline__ void put(R (&o)[V], int p, T v) {
        if constexpr (PAIR) {
            o[2 * p] = v.x;
            o[2 * p + 1] = v.y;
        } else {
            o[p] = v;
        }
    }

    __device__ __forceinline__ void moments(const R (&f)[V][Q]) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            c[p].add_rest(get(f, p, 0));
#pragma unroll
            for (int i = 0; i < Q / 2; ++i) {
                const int q = sum_order(i);
                S[p][q / 2] = get(f, p, q);
                D[p][q / 2] = get(f, p, q + 1);
                c[p].add(q, S[p][q / 2], D[p][q / 2]);
            }
            c[p].finish();
            orest[p] = c[p].rest(get(f, p, 0));
        }
    }

    // relaxed rest population of cell v (moments() computed it)
    __device__ __forceinline__ R rest(const R (&)[V][Q], int v) const {
        if constexpr (PAIR) return (v & 1) ? orest[v / 2].y : orest[v / 2].x;
        else return orest[v];
    }

    // relaxed populations q and q+1 = opp(q) (q odd, ascending from 1) of every cell
    __device__ __forceinline__ void pair(const R (&)[V][Q], int q, R (&oa)[V], R (&ob)[V]) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            T a, b;
            c[p].pair(q, S[p][q / 2], D[p][q / 2], a, b);
            put(oa, p, a);
            put(ob, p, b);
        }
    }
};

// ---- the relaxation of the 16-bit storages ------------------------------------------------------------
// A state rounded to 16 bits after every step keeps the last bit of its relaxation: another order of the
// same operations moves whole populations by 2^-11 (FP16) or 2^-8 (BF16) of their shift (2e-5 and 1e-4 of the
// state's norm after 15 steps), so these storages keep one product chain per population, on pairs of cells:
//   s = g0 + g1 + ... + g18, j = the signed sums in q order, rho = 1 + s, inv = 1/rho (IEEE), u = j inv
//   t = ux ux + uy uy + uz uz (two FMAs), base = -1.5 t, feq0 = w0 (s + rho base)
//   out0 = (1 - om) g0 + om feq0, and per odd q with a = c_q . u (two terms at most):
//   sym = fma(om w, s, om w rho (4.5 a a + base)), asym = 3 om w rho a, out_q = (1 - om) g_q + (sym + asym),
//   out_opp(q) = (1 - om) g_opp(q) + (sym - asym).
template <int V>
struct CellBgk16 {
    static constexpr bool PAIR = V % 2 == 0;
    static constexpr int NP = PAIR ? V / 2 : V;  // lanes
    using T = typename std::conditional<PAIR, float2, float>::type;
    using L = Lanes<T>;
    float om, omc;
    T s[NP], rho[NP], ux[NP], uy[NP], uz[NP], base[NP];
    T owr1[NP], owr2[NP], owr3a[NP], owr3b[NP];
    T orest[NP];

    __device__ __forceinline__ explicit CellBgk16(const BgkCoef& co) : om(co.om), omc(1.f - co.om) {}

    static __device__ __forceinline__ T get(const float (&f)[V][Q], int p, int q) {
        if constexpr (PAIR) return make_float2(f[2 * p][q], f[2 * p + 1][q]);
        else return f[p][q];
    }
    static __device__ __forceinline__ void put(float (&o)[V], int p, T v) {
        if constexpr (PAIR) {
            o[2 * p] = v.x;
            o[2 * p + 1] = v.y;
        } else {
            o[p] = v;
        }
    }
    // c_q . u for odd q (its first non-zero component is positive)
    __device__ __forceinline__ T cdot_odd(int q, int p) const {
        T a = cx(q) != 0 ? ux[p] : (cy(q) != 0 ? uy[p] : uz[p]);
        if (cx(q) != 0 && cy(q) != 0) a = cy(q) > 0 ? L::add(a, uy[p]) : L::sub(a, uy[p]);
        if ((cx(q) != 0 || cy(q) != 0) && cz(q) != 0) a = cz(q) > 0 ? L::add(a, uz[p]) : L::sub(a, uz[p]);
        return a;
    }

    __device__ __forceinline__ void moments(const float (&f)[V][Q]) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            T g[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) g[q] = get(f, p, q);
            T sm = g[0];
#pragma unroll
            for (int q = 1; q < Q; ++q) sm = L::add(sm, g[q]);
            // j in q order: a signed sum of the populations with that velocity component
            constexpr int kx[10] = {1, 2, 7, 8, 9, 10, 11, 12, 13, 14}, ky[10] = {3, 4, 7, 8, 9, 10, 15, 16, 17, 18},
                          kz[10] = {5, 6, 11, 12, 13, 14, 15, 16, 17, 18};
            T jx = g[1], jy = g[3], jz = g[5];
#pragma unroll
            for (int i = 1; i < 10; ++i) {
                jx = cx(kx[i]) > 0 ? L::add(jx, g[kx[i]]) : L::sub(jx, g[kx[i]]);
                jy = cy(ky[i]) > 0 ? L::add(jy, g[ky[i]]) : L::sub(jy, g[ky[i]]);
                jz = cz(kz[i]) > 0 ? L::add(jz, g[kz[i]]) : L::sub(jz, g[kz[i]]);
            }
            const T rh = L::add(L::bc(1.f), sm);
            const T inv = L::rcp(rh);
            s[p] = sm;
            rho[p] = rh;
            ux[p] = L::mul(jx, inv);
            uy[p] = L::mul(jy, inv);
            uz[p] = L::mul(jz, inv);
            T t = L::mul(ux[p], ux[p]);
            t = L::fma(uy[p], uy[p], t);
            t = L::fma(uz[p], uz[p], t);
            base[p] = L::mul(L::bc(-1.5f), t);
            // the folded per-class terms and the rest population
            const T feq0 = L::mul(L::bc(wf(0)), L::fma(rh, base[p], sm));
            orest[p] = L::fma(L::bc(omc), g[0], L::mul(L::bc(om), feq0));
            const T orho = L::mul(L::bc(om), rh);
            owr1[p] = L::mul(orho, L::bc(wf(1)));
            owr2[p] = L::mul(orho, L::bc(wf(7)));
            owr3a[p] = L::mul(L::bc(3.f), owr1[p]);
            owr3b[p] = L::mul(L::bc(3.f), owr2[p]);

        }
    }

    // relaxed rest population of cell v (moments() computed it)
    __device__ __forceinline__ float rest(const float (&)[V][Q], int v) const {
        if constexpr (PAIR) return (v & 1) ? orest[v / 2].y : orest[v / 2].x;
        else return orest[v];
    }

    // relaxed populations q and q+1 = opp(q) (q odd) of every cell
    __device__ __forceinline__ void pair(const float (&f)[V][Q], int q, float (&oa)[V], float (&ob)[V]) const {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const T a = cdot_odd(q, p);
            const T owr = q < 7 ? owr1[p] : owr2[p];
            const T t = L::mul(owr, L::fma(L::mul(L::bc(4.5f), a), a, base[p]));
            // + omega w s as one FMA (a product by a broadcast constant then an add is not compiled
            // alike in every kernel; an FMA is)
            const T osym = L::fma(L::bc(om * wf(q)), s[p], t);
            const T oasym = L::mul(q < 7 ? owr3a[p] : owr3b[p], a);
            put(oa, p, L::fma(L::bc(omc), get(f, p, q), L::add(osym, oasym)));
            put(ob, p, L::fma(L::bc(omc), get(f, p, q + 1), L::sub(osym, oasym)));
        }
    }
};

// Relaxed values of V cells into a row vector of storage words: 16-bit formats convert two cells per
// instruction; FP32 shifts back by w_q (SA without SH).
template <class ST, int V, bool SA>
__device__ __forceinline__ void put_row(Pack<typename ST::raw, V>& p, const typename ST::real (&o)[V], int q) {
    using R = typename ST::real;
    if constexpr (ST::shifted && V % 2 == 0) {
#pragma unroll
        for (int v = 0; v < V; v += 2) p.u32[v / 2] = ST::store2(o[v], o[v + 1]);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v) p.v[v] = ST::store((SA && !ST::shifted) ? o[v] + wgt<R>(q) : o[v]);
    }
}

}  // namespace jp
