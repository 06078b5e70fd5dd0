// Two lattice steps of uniform cubes in one pass over HBM (temporal blocking of the pull step).
//
// The single step (uniform.cu) reads and writes every population once and runs at the copy bandwidth
// of HBM, so its 152 B per update (FP32) are its time.  Here a CTA takes a tile of tx x ty cells of
// the x-y plane and marches it along z over a chunk of planes: for every plane it takes the first step
// on the tile and a one-cell halo around it (a thread per pair of x-adjacent cells, the populations
// pulled from global memory), keeps the relaxed populations in a ring of planes in shared memory, and
// takes the second step of the plane before, whose pulls come out of the ring.  HBM moves 152 B per two
// updates plus the chunks' two halo planes; the tile's halo (23 % of the first step's cells at 64 x 9) is
// recomputed and its loads hit L2, where the neighbouring tiles' CTAs have just read the same rows.  A
// population takes a plane's slot in the ring only while a second step still needs it: c_z = +1 for
// three planes, 0 for two, -1 for one; the populations with c_x = c_y = 0 never leave their thread.
// The next plane's loads are issued before the second step, whose arithmetic they fly across.
//
// Every cell goes through LaneBgk and the rounding of FP32 storage exactly as in the single step, in both of
// the two steps, so the two paths give the same bits.
//
// What bounds it (N=256, ncu): 2.56 GB of DRAM traffic per pass (the populations once each way) at 73 % of the
// copy rate; the rest is the alternation of its phases (loads, FP32 pipe, shared memory) at 12 warps per
// SM, 39 % issue.  Measured per step, single / two in one pass: N=512 2915 / 1866 us (46.0 / 71.9 GLUPS), N=256
// 364 / 254, N=128 48.0 / 34.0, N=96 17.5 / 16.4, N=32 3.4 / 2.9 (one launch less per two steps).  Shapes
// measured and left: 512 threads (128 registers: spills, and 155 KB of ring leave the loads in flight too
// little L1) 2315 us at N=512, 320 threads 2080, two CTAs of 256 or 192 threads (more halo) 2447 and 2262; a
// ring one plane longer, with one barrier per plane, 2333; planes staged by 16-byte cp.async in shared memory
// 2583; the second step's pulls read twice from the ring instead of held 1930; the two steps on two groups of
// warps with named barriers 2866 (each plane's chain of load, relax and hand-over is longer than its share of
// bandwidth).  16-bit storage stays with the single step: its relaxation keeps the per-cell sequence of
// operations (a regrouped one moves 16-bit results past their rounding), which is issue-bound, and the pass
// adds instructions (1462 to 1588 us in the forms tried with the regrouped one, against 1507 for that single step).
#include "kernels.h"
#include "lattice.cuh"
#include "uniform_common.cuh"

#include <algorithm>

namespace jp {

// Threads of a CTA (pairs of cells of a tile plane with its halo): 12 warps of 168 registers; the ring leaves
// 156 KB of L1 for a plane's loads in flight.
constexpr int kPairThreads = 384;
constexpr int kSlotBytes = kPairThreads * 8;      // one ring slot: a pair of floats per thread
constexpr int kRing0 = 0, kRingP = 2 * 8 * kSlotBytes, kRingM = kRingP + 3 * 4 * kSlotBytes;  // c_z = 0, +1, -1
constexpr int kPairSmem = kRingM + 4 * kSlotBytes;  // 32 slots, 96 KB

// index of population q within its class of c_z (+1, 0, -1), ascending q; 0, 5 and 6 (c_x = c_y = 0) stay
// in the thread's registers
__host__ __device__ constexpr int zrank(int q) {
    constexpr int t[Q] = {-1, 0, 1, 2, 3, -1, -1, 4, 5, 6, 7, 0, 0, 1, 1, 2, 2, 3, 3};
    return t[q];
}
__host__ __device__ constexpr bool own_column(int q) { return cx(q) == 0 && cy(q) == 0; }

struct PairSolve {
    const void* src;
    void* dst;
    int n, tx, ty, ntx, ntiles, zc;
    int begin;  // first item of the cube in the launch
    BgkCoef bgk;
};
template <int MAXB>
struct PairBatch {
    int count, items, release;
    PairSolve s[MAXB];
};

// the collision inputs of a pair's two cells from the words of population q, and the relaxed values as stored
__device__ __forceinline__ float2 pair_unpack(int q, unsigned w0, unsigned w1) {
    return __fadd2_rn(make_float2(__uint_as_float(w0), __uint_as_float(w1)), make_float2(-wf(q), -wf(q)));
}
__device__ __forceinline__ float2 pair_pack(int q, float2 o) { return __fadd2_rn(o, make_float2(wf(q), wf(q))); }

template <int MAXB>
__global__ void __launch_bounds__(kPairThreads, 1) k_stream_collide_pair(const __grid_constant__ PairBatch<MAXB> b) {
    constexpr int NT = kPairThreads, SB = kSlotBytes;
    extern __shared__ __align__(16) char ring[];
    const int t = threadIdx.x;
    if (MAXB == 1) {
        if (b.release) step_release();
        step_wait();
    }
    for (int it = blockIdx.x; it < b.items; it += gridDim.x) {
        int si = 0;
        if (MAXB > 1) {
#pragma unroll 1
            for (int i = 1; i < b.count; ++i) si = b.s[i].begin <= it ? i : si;
        }
        const PairSolve& d = b.s[si];
        const int n = d.n, P = d.tx / 2 + 2;
        const int row = t / P, col = t - row * P;
        const bool active = row < d.ty + 2;
        const bool inner = row >= 1 && row < d.ty + 1 && col >= 1 && col < P - 1;
        const float* src = static_cast<const float*>(d.src);
        float* __restrict__ dst = static_cast<float*>(d.dst);
        const size_t qs = (size_t)n * n * n;
        const unsigned n2 = (unsigned)n * n;
        auto wrap = [n](int a) {
            a %= n;
            return a < 0 ? a + n : a;
        };
        const int k = it - d.begin, zci = k / d.ntiles, tile = k - zci * d.ntiles;
        const int tyi = tile / d.ntx, txi = tile - tyi * d.ntx;
        const int ox = txi * d.tx + 2 * (col - 1), oy = tyi * d.ty + row - 1;
        const int zs = zci * d.zc, m = min(n, zs + d.zc) - zs;
        const int gx = wrap(ox), gy = wrap(oy);  // gx even (n is even), gx + 1 < n
        const bool valid = inner && ox < n && oy < n;
        const unsigned row0 = (unsigned)gy * n, rowm = (unsigned)(gy == 0 ? n - 1 : gy - 1) * n,
                       rowp = (unsigned)(gy + 1 == n ? 0 : gy + 1) * n;
        const unsigned xm = gx == 0 ? n - 1 : gx - 1, xp = gx + 2 == n ? 0 : gx + 2;
        unsigned a0[Q], a1[Q];
        auto load_plane = [&](int z) {
            const unsigned zo[3] = {(unsigned)(z == 0 ? n - 1 : z - 1) * n2, (unsigned)z * n2,
                                    (unsigned)(z + 1 == n ? 0 : z + 1) * n2};
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const float* p = src + q * qs + zo[1 - cz(q)];
                const unsigned ro = cy(q) > 0 ? rowm : cy(q) < 0 ? rowp : row0;
                auto one = [&](unsigned x) { return ld_step<float, 1>(p + (ro + x)).u32[0]; };
                if (cx(q) == 0) {
                    const Pack<float, 2> v = ld_step<float, 2>(p + (ro + gx));
                    a0[q] = v.u32[0];
                    a1[q] = v.u32[1];
                } else {
                    a0[q] = cx(q) > 0 ? one(xm) : one(gx + 1);
                    a1[q] = cx(q) > 0 ? one(gx) : one(xp);
                }
            }
        };
        __syncthreads();  // the last item's reads of the ring are done
        if (active) load_plane(zs == 0 ? n - 1 : zs - 1);
        // own column, as stored: 0 of plane r - 1, 5 of r - 2, 6 of r
        float2 h0{}, h0n{}, h5{}, h5n{}, h5nn{}, h6{};
        int s3 = 0;                         // r mod 3
        for (int r = 0; r <= m + 1; ++r) {  // first step of plane zs - 1 + r, second of zs + r - 2
            // slots: c_z = 0 written for r, read for r - 1; +1 for r and r - 2; -1 for r and r
            char* const wr0 = ring + kRing0 + (r & 1) * 8 * SB;
            char* const wr1 = ring + kRingP + s3 * 4 * SB;
            char* const wr2 = ring + kRingM;
            if (active) {
                float2 g[Q];
                LaneBgk<float2, true> c(d.bgk);
                g[0] = pair_unpack(0, a0[0], a1[0]);
                c.add_rest(g[0]);
#pragma unroll
                for (int i = 0; i < Q / 2; ++i) {
                    const int q = sum_order(i);
                    g[q] = pair_unpack(q, a0[q], a1[q]);
                    g[q + 1] = pair_unpack(q + 1, a0[q + 1], a1[q + 1]);
                    c.add(q, g[q], g[q + 1]);
                }
                c.finish();
                h0 = h0n;
                h5 = h5n;
                h5n = h5nn;
                auto put = [&](int q, float2 o) {
                    const float2 w = pair_pack(q, o);
                    if (own_column(q)) {
                        if (q == 0) h0n = w;
                        else if (q == 5) h5nn = w;
                        else h6 = w;
                        return;
                    }
                    char* slot = (cz(q) == 0 ? wr0 : cz(q) > 0 ? wr1 : wr2) + zrank(q) * SB;
                    // c_x != 0: the pairs' cells in two separate rows, which the shifted reads take without
                    // bank conflicts
                    if (cx(q) == 0) {
                        reinterpret_cast<float2*>(slot)[t] = w;
                    } else {
                        reinterpret_cast<float*>(slot)[t] = w.x;
                        reinterpret_cast<float*>(slot)[NT + t] = w.y;
                    }
                };
                put(0, c.rest(g[0]));
#pragma unroll
                for (int q = 1; q < Q; q += 2) {
                    float2 oa, ob;
                    c.pair(q, g[q], g[q + 1], oa, ob);
                    put(q, oa);
                    put(q + 1, ob);
                }
                if (r <= m) load_plane(zs + r == n ? 0 : zs + r);
            }
            __syncthreads();
            if (r >= 2 && valid) {
                const char* const rd0 = ring + kRing0 + ((r & 1) ^ 1) * 8 * SB;
                const char* const rd1 = ring + kRingP + (s3 == 2 ? 0 : s3 + 1) * 4 * SB;
                // the pulled pair of population q, from the first step's planes
                auto get = [&](int q) -> float2 {
                    if (own_column(q)) {
                        const float2 w = q == 0 ? h0 : q == 5 ? h5 : h6;
                        return pair_unpack(q, __float_as_uint(w.x), __float_as_uint(w.y));
                    }
                    const char* slot = (cz(q) == 0 ? rd0 : cz(q) > 0 ? rd1 : wr2) + zrank(q) * SB;
                    const unsigned* w = reinterpret_cast<const unsigned*>(slot);
                    const int i = t - cy(q) * P;
                    if (cx(q) == 0) return pair_unpack(q, w[2 * i], w[2 * i + 1]);
                    return cx(q) > 0 ? pair_unpack(q, w[NT + i - 1], w[i]) : pair_unpack(q, w[NT + i], w[i + 1]);
                };
                LaneBgk<float2, true> c(d.bgk);
                float2 g[Q];
                g[0] = get(0);
                c.add_rest(g[0]);
#pragma unroll
                for (int i = 0; i < Q / 2; ++i) {
                    const int q = sum_order(i);
                    g[q] = get(q);
                    g[q + 1] = get(q + 1);
                    c.add(q, g[q], g[q + 1]);
                }
                c.finish();
                const unsigned o0 = (unsigned)(zs + r - 2) * n2 + row0 + gx;
                auto store = [&](int q, float2 o) {
                    Pack<float, 2> pk;
                    const float2 w = pair_pack(q, o);
                    pk.v[0] = w.x;
                    pk.v[1] = w.y;
                    st_pack<float, 2>(dst + q * qs + o0, pk);
                };
                store(0, c.rest(g[0]));
#pragma unroll
                for (int q = 1; q < Q; q += 2) {
                    float2 oa, ob;
                    c.pair(q, g[q], g[q + 1], oa, ob);
                    store(q, oa);
                    store(q + 1, ob);
                }
            }
            __syncthreads();  // the second step has read what the next plane overwrites
            s3 = s3 == 2 ? 0 : s3 + 1;
        }
    }
}

// Time model of the plans, in microseconds.  A CTA walks its items' planes (chunk + 2 halo planes each).  A
// plane of a tile of 56 to 128 cells along x takes 2.4-2.6 us at N=128..512 whatever the tile's share of the
// threads, a third more for narrower tiles, whose rows are mostly halo; where both states fit L2 (up to 600,000
// cells) it takes 1.4-2.2 us with the share of threads at work.
constexpr double kL2Cells = 6e5;
static double plane_us(double cells, int tx, int ty) {
    if (cells <= kL2Cells) return 2.2 * (0.5 + 0.5 * (tx / 2 + 2) * (ty + 2) / kPairThreads);
    return tx < 48 ? 3.26 : 2.45;
}
// The single step: 21.7 ps per cell from HBM, 2.7 us and 11 ps per cell in L2 (measured N=16 2.8, N=32 3.1, N=48 4.0,
// N=64 5.5, N=80 8.2, N=128 48.0, N=192 154.6 us; the two-step pass 2.2, 3.0, 4.9, 7.0, 11.0, 34.6, 112.5).
static double single_us(double cells) { return cells <= kL2Cells ? 2.7 + cells * 11e-6 : cells * 21.7e-6; }
static bool pair_tile(int n, int tx, PairPlan& p) {
    const int P = tx / 2 + 2, tymax = std::min(n, kPairThreads / P - 2);
    if (tymax < 1) return false;
    const int nty = (n + tymax - 1) / tymax;
    p.tx = tx;
    p.ty = (n + nty - 1) / nty;
    p.tiles = (n + tx - 1) / tx * ((n + p.ty - 1) / p.ty);
    return true;
}
constexpr int kPairAlign = 8;  // x tiles start at 32-byte sectors
// pairs of cells at even x need an even n; cell indices are 32-bit
static bool pair_ok(int n, int sms) { return n >= 2 && n % 2 == 0 && n <= 1600 && sms > 0; }

// One cube: every tile width, and the chunks that fill 1 to 16 rounds of CTAs.  The two-step pass is used where
// the model puts it 5 % ahead.
PairPlan pair_plan(int n, int sms) {
    PairPlan best{};
    if (!pair_ok(n, sms)) return best;
    const double cells = double(n) * n * n;
    for (int tx = kPairAlign; tx <= 128 && tx < n + kPairAlign; tx += kPairAlign) {
        PairPlan p{};
        if (!pair_tile(n, tx, p)) break;
        const double plane = plane_us(cells, tx, p.ty);
        int last = 0;
        for (int rounds = 1; rounds <= 16; ++rounds) {  // the shortest chunk that fits each number of rounds
            const int nzc = std::min((long long)n, (long long)rounds * sms / p.tiles);
            if (nzc < 1 || nzc == last) continue;
            last = nzc;
            p.zc = (n + nzc - 1) / nzc;
            const long long items = (long long)p.tiles * ((n + p.zc - 1) / p.zc);
            p.us = double((items + sms - 1) / sms) * (p.zc + 2) * plane / 2;
            if (best.us == 0 || p.us < best.us) best = p;
        }
        if (best.us == 0) {  // more tiles than 16 rounds hold: whole columns
            p.zc = n;
            p.us = double((p.tiles + sms - 1) / sms) * (n + 2) * plane / 2;
            best = p;
        }
    }
    best.use = best.us < 0.95 * single_us(cells);
    return best;
}

// In a launch of many cubes a cube takes the tile with the fewest CTA planes ...
PairPlan pair_tile_plan(int n, int sms) {
    PairPlan best{};
    if (!pair_ok(n, sms)) return best;
    for (int tx = kPairAlign; tx <= 128 && tx < n + kPairAlign; tx += kPairAlign) {
        PairPlan p{};
        if (!pair_tile(n, tx, p)) break;
        p.us = p.tiles * plane_us(2 * kL2Cells, tx, p.ty);
        if (best.us == 0 || p.us < best.us) best = p;
    }
    return best;
}

// ... and all of them one chunk length: the one with the least mean load of a CTA plus its longest item.
bool pair_plan_batch(const int* n, int count, int sms, PairPlan* plans) {
    double cells = 0, best = 0;
    int best_zc = 0;
    for (int i = 0; i < count; ++i) {
        if (plans[i].tiles <= 0) return false;
        cells += double(n[i]) * n[i] * n[i];
    }
    for (int zc : {4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128, 1600}) {
        double sum = 0, longest = 0;
        for (int i = 0; i < count; ++i) {
            const int nzc = (n[i] + zc - 1) / zc, z = (n[i] + nzc - 1) / nzc;
            const double us = (z + 2) * plane_us(cells, plans[i].tx, plans[i].ty) / 2;
            sum += double(plans[i].tiles) * ((n[i] + z - 1) / z) * us;
            longest = std::max(longest, us);
        }
        const double us = std::max(sum / sms + 0.5 * longest, longest);
        if (best == 0 || us < best) {
            best = us;
            best_zc = zc;
        }
    }
    for (int i = 0; i < count; ++i) {
        const int nzc = (n[i] + best_zc - 1) / best_zc;
        plans[i].zc = (n[i] + nzc - 1) / nzc;
    }
    return best < 0.95 * single_us(cells);
}

template <int MAXB>
static cudaError_t launch_pair_t(const UniSolve* u, const PairPlan* plans, int count, int sms, cudaStream_t st) {
    auto kern = k_stream_collide_pair<MAXB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
    if (e != cudaSuccess) return e;
    PairBatch<MAXB> b;
    b.count = count;
    b.items = 0;
    b.release = count == 1 && release_early(false, false, u[0].n);
    for (int i = 0; i < count; ++i) {
        PairSolve& s = b.s[i];
        const PairPlan& p = plans[i];
        if (p.tx <= 0 || p.tx % 2 || p.ty <= 0 || p.zc <= 0 || (p.tx / 2 + 2) * (p.ty + 2) > kPairThreads ||
            !pair_ok(u[i].n, sms))
            return cudaErrorInvalidValue;
        s.src = u[i].src;
        s.dst = u[i].dst;
        s.n = u[i].n;
        s.bgk = u[i].bgk;
        s.tx = p.tx;
        s.ty = p.ty;
        s.zc = p.zc;
        s.ntx = (s.n + p.tx - 1) / p.tx;
        s.ntiles = s.ntx * ((s.n + p.ty - 1) / p.ty);
        s.begin = b.items;
        b.items += s.ntiles * ((s.n + p.zc - 1) / p.zc);
    }
    note_launch();
    if constexpr (MAXB == 1) return launch_step(kern, std::min(b.items, sms), kPairThreads, kPairSmem, st, b);
    kern<<<std::min(b.items, sms), kPairThreads, kPairSmem, st>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_stream_collide_pair(const UniSolve* solves, const PairPlan* plans, int count, int sms, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    if (count > kMaxBatch || sms <= 0) return cudaErrorInvalidValue;
    return count == 1 ? launch_pair_t<1>(solves, plans, count, sms, st) : launch_pair_t<kMaxBatch>(solves, plans, count, sms, st);
}

}  // namespace jp
