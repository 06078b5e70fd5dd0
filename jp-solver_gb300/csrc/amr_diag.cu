// Energy, enstrophy and mass of a three-level AMR state without its composite field.
//
// The reference (src/tgv3d_amr.cu:514-549) writes the state as a field on the finest grid, (4 N0)^3 records,
// and reduces that field with its six neighbours.  A coarse cell is 64 equal records there and a level-1 cell 8,
// so most of those cells have no gradient of their own: in the dynamic case (N0=96; 520 coarse and 172 level-1
// blocks refined) 3.4 M leaf cells stand for 56.6 M records.  Here the leaf cells' macroscopic values are computed
// once per cell (k_leaf_macro), and the reduction walks the leaf blocks and adds a cell's sub-cells in closed form:
//   a cell of edge f = 4, 2, 1 records has along each axis the half differences lo = (v - v_minus) / 2 in its
//   first layer of records, hi = (v_plus - v) / 2 in its last and zero between (f = 1: (v_plus - v_minus) / 2), so
//   sum over its f^3 records of (A - B)^2, A along one axis and B along another, is
//   f [ (Alo-Blo)^2 + (Alo-Bhi)^2 + (Ahi-Blo)^2 + (Ahi-Bhi)^2 + (f-2)(Alo^2 + Ahi^2 + Blo^2 + Bhi^2) ]
// as long as every face of the cell has one neighbour value.  A face whose neighbour block is finer has two by
// two values: the cell is then summed by octants of edge h = f / 2, each with one layer of records next to a
// neighbour along every axis (difference dA, dB) and h - 1 without a gradient:
//   h [ (dA-dB)^2 + (h-1)(dA^2 + dB^2) ].
// Terms and sums are in double-float as for the composite field (diag_terms.cuh), in a fixed order.  A warp
// takes a block, or a part of one where the grid has fewer blocks than the GPU has warps.
//
// What bounds it (ncu, that grid): k_leaf_macro reads the populations at 6.4 TB/s (46 us); k_leaf_diag (148 us) is bound
// by its instructions, 890 per leaf cell: 0.60 issued per cycle and scheduler, the largest stall their fetch (2.9
// of 9.7 warp cycles per instruction; faces, levels and octants are much code), DRAM at 5 %.
#include "amr_common.cuh"
#include "diag_terms.cuh"
#include "amr_kernels.h"
#include "kernels.h"
#include "uniform_common.cuh"

#include <algorithm>

namespace jp {
namespace amr {

namespace {

constexpr int kLeafThreads = 128;

struct Leaf {  // a unit of the walk: block b of a level
    int level, b;
};
__device__ __forceinline__ Leaf leaf_of(const AmrGrid& g, int unit) {
    if (unit < g.cnb0) return {0, unit};
    if (unit < g.cnb0 + g.nf1) return {1, unit - g.cnb0};
    return {2, unit - g.cnb0 - g.nf1};
}
__device__ __forceinline__ bool is_refined(const AmrGrid& g, Leaf l) {
    return l.level == 0 ? g.ref0[l.b] != 0 : l.level == 1 ? g.ref1[l.b] != 0 : false;
}

template <int MB, class ST>
__global__ void __launch_bounds__(kLeafThreads) k_leaf_macro(const AmrGrid g, const void* __restrict__ c0,
                                                             const void* __restrict__ f1, const void* __restrict__ f2,
                                                             float4* __restrict__ M) {
    using raw = typename ST::raw;
    constexpr int MB3 = MB * MB * MB;
    const Leaf l = leaf_of(g, blockIdx.x);
    if (is_refined(g, l)) return;
    const raw* p = static_cast<const raw*>(l.level == 0 ? c0 : l.level == 1 ? f1 : f2) + (size_t)l.b * Q * MB3;
    float4* out = M + (size_t)blockIdx.x * MB3;
    for (int c = 4 * threadIdx.x; c < MB3; c += 4 * kLeafThreads) {  // four cells: one vector per population
        Pack<raw, 4> v[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) v[q] = ld_pack<raw, 4>(p + q * MB3 + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float f[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) f[q] = PoolIO<ST>::f_of(v[q].v[k], q);
            float4 m;
            moments(f, m.x, m.y, m.z, m.w);
            out[c + k] = m;
        }
    }
}

// unit and cell of the leaf that holds record (x, y, z) of the finest grid (k_composite's lookup)
template <int MB>
__device__ __forceinline__ const float4* leaf_at(const AmrGrid& g, const float4* M, int x, int y, int z) {
    constexpr int MB3 = MB * MB * MB;
    auto cell = [](int a, int b, int c) { return ((c % MB) * MB + b % MB) * MB + a % MB; };
    const int lb = g.l1grid[((z / (2 * MB)) * g.l1gx + y / (2 * MB)) * g.l1gx + x / (2 * MB)];
    if (lb < 0) {
        const int i = x / 4, j = y / 4, k = z / 4;
        return M + (size_t)(((k / MB) * g.cgx + j / MB) * g.cgx + i / MB) * MB3 + cell(i, j, k);
    }
    if (!g.ref1[lb]) return M + (size_t)(g.cnb0 + lb) * MB3 + cell(x / 2, y / 2, z / 2);
    const int b = g.fof1[lb] + ((z / MB) % 2) * 4 + ((y / MB) % 2) * 2 + (x / MB) % 2;
    return M + (size_t)(g.cnb0 + g.nf1 + b) * MB3 + cell(x, y, z);
}

// sum over two layers and the f - 2 gradient-free ones between of (A - B)^2, without the factor f
__device__ __forceinline__ dterm::FF layer_squares(int f, dterm::FF alo, dterm::FF ahi, dterm::FF blo, dterm::FF bhi) {
    using namespace dterm;
    auto d2 = [](FF a, FF b) { return sq(add(a, {-b.hi, -b.lo})); };
    FF s = add_same_sign(add_same_sign(d2(alo, blo), d2(alo, bhi)), add_same_sign(d2(ahi, blo), d2(ahi, bhi)));
    if (f == 4) {
        FF t = add_same_sign(add_same_sign(sq(alo), sq(ahi)), add_same_sign(sq(blo), sq(bhi)));
        s = add_same_sign(s, {2.f * t.hi, 2.f * t.lo});
    }
    return s;
}

enum { FACE_SAME, FACE_COARSER, FACE_FINER };

template <int MB>
__global__ void __launch_bounds__(kLeafThreads) k_leaf_diag(const AmrGrid g, const float4* __restrict__ M, int units,
                                                            int parts, double* __restrict__ partials) {
    using namespace dterm;
    constexpr int MB3 = MB * MB * MB, MB2 = MB * MB;
    const int t = threadIdx.x, lane = t & 31, N2 = g.N2;
    const int nwarps = gridDim.x * (kLeafThreads / 32);
    Acc acc;
    for (int w = blockIdx.x * (kLeafThreads / 32) + (t >> 5); w < units * parts; w += nwarps) {
        const int unit = w / parts, first = (w - unit * parts) * 32 + lane, stride = parts * 32;
        const Leaf l = leaf_of(g, unit);
        if (is_refined(g, l)) continue;  // the whole warp
        const int f = 4 >> l.level;
        // the block's position on its level's grid of blocks
        const int G = g.cgx << l.level;
        int bx, by, bz;
        if (l.level == 0) {
            bx = l.b % G;
            by = l.b / G % G;
            bz = l.b / (G * G);
        } else {
            const int p = g.f1pos[l.level == 1 ? l.b : g.l2pl1[l.b]];
            bx = p % g.l1gx;
            by = p / g.l1gx % g.l1gx;
            bz = p / (g.l1gx * g.l1gx);
            if (l.level == 2) {
                const int o = g.l2oct[l.b];
                bx = 2 * bx + (o & 1);
                by = 2 * by + ((o >> 1) & 1);
                bz = 2 * bz + (o >> 2);
            }
        }
        // lanes 0..5: what is behind the faces -x +x -y +y -z +z, and its unit when FACE_SAME
        int kind_l = FACE_SAME, nb_l = 0;
        if (lane < 6) {
            const int s = (lane & 1) ? 1 : -1, axis = lane >> 1;
            auto step = [&](int b, int a) {
                b += a == axis ? s : 0;
                return b < 0 ? G - 1 : b == G ? 0 : b;
            };
            const int x = step(bx, 0), y = step(by, 1), z = step(bz, 2);
            if (l.level == 0) {
                nb_l = (z * G + y) * G + x;
                if (g.ref0[nb_l]) kind_l = FACE_FINER;
            } else if (l.level == 1) {
                const int lb = g.l1grid[(z * G + y) * G + x];
                kind_l = lb < 0 ? FACE_COARSER : g.ref1[lb] ? FACE_FINER : FACE_SAME;
                nb_l = g.cnb0 + lb;
            } else {
                const int lb = g.l1grid[((z >> 1) * g.l1gx + (y >> 1)) * g.l1gx + (x >> 1)];
                if (lb < 0 || !g.ref1[lb]) kind_l = FACE_COARSER;
                else nb_l = g.cnb0 + g.nf1 + g.fof1[lb] + (z & 1) * 4 + (y & 1) * 2 + (x & 1);
            }
        }
        int nb[6];
        unsigned same = 0, finer = 0;  // bit per face
#pragma unroll
        for (int e = 0; e < 6; ++e) {
            nb[e] = __shfl_sync(0xffffffffu, nb_l, e);
            const int k = __shfl_sync(0xffffffffu, kind_l, e);
            same |= unsigned(k == FACE_SAME) << e;
            finer |= unsigned(k == FACE_FINER) << e;
        }
        const float4* const own = M + (size_t)unit * MB3;
        const int ox = bx * MB * f, oy = by * MB * f, oz = bz * MB * f;  // the block's first record on the finest grid
        // the value across face `face` (axis, sign) of cell c, whose coordinate along the axis is a and index
        // step d, at the record (x, y, z) behind the face
        auto across = [&](int face, int c, int a, int d, int x, int y, int z) -> float4 {
            const int s = (face & 1) ? 1 : -1;
            if (unsigned(a + s) < unsigned(MB)) return __ldg(own + c + s * d);
            if ((same >> face) & 1) {
                const int u = face == 0 ? nb[0] : face == 1 ? nb[1] : face == 2 ? nb[2] : face == 3 ? nb[3]
                            : face == 4 ? nb[4] : nb[5];
                return __ldg(M + (size_t)u * MB3 + c - s * (MB - 1) * d);
            }
            auto in = [N2](int v) { return v < 0 ? v + N2 : v >= N2 ? v - N2 : v; };
            return __ldg(leaf_at<MB>(g, M, in(x), in(y), in(z)));
        };
        // faces of the cell (i, j, k) behind which the block is finer
        auto fine_faces = [&](int i, int j, int k) -> unsigned {
            return finer & (unsigned(i == 0) | unsigned(i == MB - 1) << 1 | unsigned(j == 0) << 2 | unsigned(j == MB - 1) << 3 |
                            unsigned(k == 0) << 4 | unsigned(k == MB - 1) << 5);
        };
        for (int c = first; c < MB3; c += stride) {
            const int i = c % MB, j = c / MB % MB, k = c / MB2;
            if (fine_faces(i, j, k)) continue;
            const int x = ox + i * f, y = oy + j * f, z = oz + k * f;
            const float4 me = __ldg(own + c);
            const float4 xm = across(0, c, i, 1, x - 1, y, z), xp = across(1, c, i, 1, x + f, y, z);
            const float4 ym = across(2, c, j, MB, x, y - 1, z), yp = across(3, c, j, MB, x, y + f, z);
            const float4 zm = across(4, c, k, MB2, x, y, z - 1), zp = across(5, c, k, MB2, x, y, z + f);
            FF e, ens;
            if (f == 1) {
                velocity_terms<false>(me.y, me.z, me.w, xp.z, xm.z, xp.w, xm.w, yp.y, ym.y, yp.w, ym.w, zp.y, zm.y, zp.z,
                                      zm.z, e, ens);
            } else {
                const float f3 = float(f * f * f);
                e = add_same_sign(add_same_sign(two_prod(me.y, me.y), two_prod(me.z, me.z)), two_prod(me.w, me.w));
                e = {e.hi * (0.5f * f3), e.lo * (0.5f * f3)};
                auto lo = [](float v, float m) { return half(two_sum(v, -m)); };
                FF s = layer_squares(f, lo(me.w, ym.w), lo(yp.w, me.w), lo(me.z, zm.z), lo(zp.z, me.z));
                s = add_same_sign(s, layer_squares(f, lo(me.y, zm.y), lo(zp.y, me.y), lo(me.w, xm.w), lo(xp.w, me.w)));
                s = add_same_sign(s, layer_squares(f, lo(me.z, xm.z), lo(xp.z, me.z), lo(me.y, ym.y), lo(yp.y, me.y)));
                ens = {s.hi * (0.5f * f), s.lo * (0.5f * f)};
            }
            acc.add_cell(e, ens, me.x * float(f * f * f));
        }
        // the cells on faces with finer neighbours, octant by octant; a cell on several such faces belongs to
        // the first of them
        const int h = f >> 1;
        for (int face = 0; face < 6; ++face) {
            if (!((finer >> face) & 1)) continue;
            const int axis = face >> 1, a = (face & 1) ? MB - 1 : 0;
            for (int v = first; v < 8 * MB2; v += stride) {
                const int oct = v & 7, p = v >> 3 & (MB - 1), q = (v >> 3) / MB;
                const int i = axis == 0 ? a : p, j = axis == 1 ? a : axis == 0 ? p : q, k = axis == 2 ? a : q;
                if (fine_faces(i, j, k) & ((1u << face) - 1)) continue;
                const int c = (k * MB + j) * MB + i;
                const bool hx = oct & 1, hy = oct & 2, hz = oct & 4;
                const int x = ox + i * f + (hx ? h : 0), y = oy + j * f + (hy ? h : 0), z = oz + k * f + (hz ? h : 0);
                const float4 me = __ldg(own + c);
                const float4 nx = across(hx ? 1 : 0, c, i, 1, hx ? x + h : x - 1, y, z);
                const float4 ny = across(hy ? 3 : 2, c, j, MB, x, hy ? y + h : y - 1, z);
                const float4 nz = across(hz ? 5 : 4, c, k, MB2, x, y, hz ? z + h : z - 1);
                // half differences along an axis: neighbour minus cell behind, cell minus neighbour before
                auto dif = [](bool high, float nbv, float mev) {
                    FF d = half(two_sum(nbv, -mev));
                    return high ? d : FF{-d.hi, -d.lo};
                };
                auto layer = [&](FF A, FF B) {
                    FF s = sq(add(A, {-B.hi, -B.lo}));
                    if (h == 2) s = add_same_sign(s, add_same_sign(sq(A), sq(B)));
                    return s;
                };
                FF s = layer(dif(hy, ny.w, me.w), dif(hz, nz.z, me.z));
                s = add_same_sign(s, layer(dif(hz, nz.y, me.y), dif(hx, nx.w, me.w)));
                s = add_same_sign(s, layer(dif(hx, nx.z, me.z), dif(hy, ny.y, me.y)));
                const float h3 = float(h * h * h);
                FF e = add_same_sign(add_same_sign(two_prod(me.y, me.y), two_prod(me.z, me.z)), two_prod(me.w, me.w));
                acc.add_cell({e.hi * (0.5f * h3), e.lo * (0.5f * h3)}, {s.hi * (0.5f * h), s.lo * (0.5f * h)}, me.x * h3);
            }
        }
    }
    acc.flush();
    double v[3] = {acc.de, acc.dens, acc.dmass};
    __shared__ double sh[3][kLeafThreads / 32];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if (lane == 0) sh[q][t >> 5] = v[q];
    }
    __syncthreads();
    if (t < 3) {
        double s = 0.0;
        for (int i = 0; i < kLeafThreads / 32; ++i) s += sh[t][i];
        partials[blockIdx.x * 3 + t] = s;
    }
}

template <int MB>
cudaError_t launch_mb(int storage, const AmrGrid& g, const void* c0, const void* f1, const void* f2, float4* M,
                      double* partials, double* out, cudaStream_t st) {
    const int units = g.cnb0 + g.nf1 + g.nf2;
    switch (storage) {
        case 0: k_leaf_macro<MB, StF32><<<units, kLeafThreads, 0, st>>>(g, c0, f1, f2, M); break;
        case 1: k_leaf_macro<MB, StF16><<<units, kLeafThreads, 0, st>>>(g, c0, f1, f2, M); break;
        case 2: k_leaf_macro<MB, StBF16><<<units, kLeafThreads, 0, st>>>(g, c0, f1, f2, M); break;
        default: return cudaErrorInvalidValue;
    }
    // parts of a block (of 32 cells at least) until every warp of the largest grid has two: N0=96 takes 221 us with
    // two, 251 with one, 229 with four, 234 with eight (the faces are looked up once per part)
    constexpr int kWarps = kLeafThreads / 32;
    int parts = 1;
    while (2 * parts * 32 <= MB * MB * MB && units * parts < 2 * kDiagBlocks * kWarps) parts *= 2;
    const int grid = std::min((units * parts + kWarps - 1) / kWarps, kDiagBlocks);
    k_leaf_diag<MB><<<grid, kLeafThreads, 0, st>>>(g, M, units, parts, partials);
    note_launch(2);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_diag_finish(partials, grid, 1.0 / (double(g.N2) * g.N2 * g.N2), out, st);
}

}  // namespace

cudaError_t launch_amr_diag(int storage, int mb, const AmrGrid& g, const void* c0, const void* f1, const void* f2,
                            void* macro, double* partials, double* out, cudaStream_t st) {
    float4* const M = static_cast<float4*>(macro);
    switch (mb) {
        case 4: return launch_mb<4>(storage, g, c0, f1, f2, M, partials, out, st);
        case 8: return launch_mb<8>(storage, g, c0, f1, f2, M, partials, out, st);
        case 16: return launch_mb<16>(storage, g, c0, f1, f2, M, partials, out, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace amr
}  // namespace jp
