// Internal launch interface between the C ABI (capi.cu) and the kernel translation units.
// Nothing here is exported from the shared library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

namespace jp {

// ---- uniform periodic cube, flat SoA layout [q][z][y][x] ----------------------------------------

// Coefficients of the relaxation (LaneBgk, uniform_common.cuh) for one omega: 3 om w and om w of the faces and
// edges, om w of the rest population, 1/(2 om w) of the faces and edges.
template <class R>
struct BgkCoefOf {
    R om, a1, a2, b0, b1, b2, k1, k2;
};
using BgkCoef = BgkCoefOf<float>;
// Rounded each for itself, the coefficients would gain or lose mass in every step: relaxing a cell changes its
// mass by (C0 - om) e + (2 K - 1.5 om) j.j / rho with C0 = b0 + 6 b1 + 12 b2 and K = k1 a1^2 + 4 k2 a2^2,
// which exact ones make zero.  Each is taken within one unit in the last place of its value so that this is smallest
// (N=64, Re=400, 2000 steps: mass drift 3.2e-7 with the nearest values, 8.1e-9 so, 2.1e-8 by a product chain per
// population).  The edges' a2 is the nearest, a1 what it leaves of the momentum's 2 a1 + 8 a2 = om (exact).
BgkCoef bgk_coefficients(float omega);

// One periodic cube of a batched stream-collide launch.
struct UniSolve {
    const void* src;         // populations at t   (19 * n^3 elements)
    void* dst;               // populations at t+1
    int n;                   // edge
    int nxs;                 // n / V: x segments per row
    BgkCoef bgk;             // of 1/tau (FP32 and shifted storages)
    double omega_d;          // 1/tau (FP64 storage)
    double half_inv_d;       // 1 / (2 omega_d)
    void set_omega(double w, const BgkCoef& c) {
        bgk = c;
        omega_d = w;
        half_inv_d = 0.5 / w;
    }
    long long blk_begin;     // first CUDA block of this cube in the launch
    long long nseg;          // n^3 / V threads
};
constexpr int kMaxBatch = 48;
template <int MAXB>
struct UniBatchOf {
    int count;
    int release;  // one cube: the CTAs let the successor's in at once (release_early)
    UniSolve s[MAXB];
};
using UniBatch = UniBatchOf<kMaxBatch>;

// Launch one stream-collide over `count` cubes of the same storage format (storage id of jp_storage).
// vec: cells per thread along x (0 = default), tpb: threads per block (0 = default).
// Returns the CUDA error of the launch.
cudaError_t launch_stream_collide(int storage, const UniSolve* solves, int count, int vec, int tpb,
                                  cudaStream_t st);

// In-place (AA) step over `count` cubes, each with src == dst: parity 0 (even step count) runs the
// local step, 1 the stream step (uniform_aa.cu).  vec must be the storage's default; the threads per
// block are the smallest of 128, 256, 512 that hold a whole x-row (tpb is not followed).
cudaError_t launch_stream_collide_inplace(int storage, const UniSolve* solves, int count, int parity, int vec,
                                          int tpb, cudaStream_t st);
// Threads per block the in-place steps use for cubes up to edge max_n (0: not supported).
int inplace_tpb(int storage, int vec, int tpb, int max_n);

// Two steps of `count` cubes in one pass (uniform_pair.cu): src -> dst holds the state two steps on, the
// same bits as two launch_stream_collide steps.  A plan gives a cube's tile (tx x ty cells, which a CTA
// marches along z over chunks of zc planes); us is the model's time per step, use whether that beats
// the single step.  FP32 storage, even n <= 1600.
struct PairPlan {
    int tx, ty, zc, tiles;
    double us;
    bool use;
};
PairPlan pair_plan(int n, int sms);
// a cube's tile in a launch of many cubes (zc not set), and the chunks of cubes of edges n[0..count) with the
// tiles plans[] in one launch: whether that beats single steps
PairPlan pair_tile_plan(int n, int sms);
bool pair_plan_batch(const int* n, int count, int sms, PairPlan* plans);
cudaError_t launch_stream_collide_pair(const UniSolve* solves, const PairPlan* plans, int count, int sms,
                                       cudaStream_t st);

// Largest supported vec for a storage; a valid vec divides n and keeps n^3/vec a multiple of 32.
int default_vec(int storage);
bool vec_supported(int storage, int vec);

// TGV initial state (src/tgv3d_uniform.cu:63-77) into flat storage; axis_tab: 3*n doubles of scratch.
// aa: in the in-place layout of step 0 (population q of cell x at [q][x + c_q]).
cudaError_t launch_init_tgv(int storage, void* f, int n, double u0, double kf, double* axis_tab, cudaStream_t st,
                            bool aa = false);

// Macroscopic field (rho, ux, uy, uz) per cell, linear (z*n+y)*n+x.  FP64 storage writes double4 (float4
// when as_float), every other storage float4 (k_macro, src/tgv3d_uniform.cu:80-90).  layout: 0 flat [q][x]; 1, 2 the
// in-place layouts after an even / odd step count (aa_layout()).
cudaError_t launch_macro(int storage, const void* f, void* field, int n, cudaStream_t st, int layout = 0,
                         bool as_float = false);

// Energy, enstrophy, mass of a macro field, reduced deterministically to out_dev[3] (device).
// partials_dev holds kDiagBlocks*3 doubles.  float_diff=true takes the velocity differences in
// float before widening (the uniform host loop, src/tgv3d_uniform.cu:103-105); false exactly
// (k_diag_reduce, src/tgv3d_amr.cu:542-546).  A float field is read in 16-byte cell records and must
// be 16-byte aligned (every solver's own field is).
constexpr int kDiagBlocks = 1216;   // 152 SMs x 8
constexpr int kDiagThreads = 256;
// block partials + launch_diag_pop's error word and count of finished CTAs (both zero between launches)
constexpr int kDiagPartials = kDiagBlocks * 3 + 1;
inline int* diag_err_word(double* partials) { return reinterpret_cast<int*>(partials + kDiagBlocks * 3); }
cudaError_t launch_diag_field(bool field_is_double, bool float_diff, const void* field, int n,
                              double* partials_dev, double* out_dev, cudaStream_t st);

// sum of `nparts` partial triples in a fixed order, scaled by inv_cells, into out_dev[3]
cudaError_t launch_diag_finish(const double* partials_dev, int nparts, double inv_cells, double* out_dev, cudaStream_t st);

// Energy, enstrophy, mass of a float-storage cube (storage 0 FP32, 1 FP16, 2 BF16) straight from its
// populations f in layout 0 / 1 / 2 (as launch_macro), with no macro field: the per-cell terms of
// launch_macro + launch_diag_field(float_diff=true), summed another way (double-float partials in a
// fixed order) to ~1e-13 of the result.
// Cubes it takes: even n (pairs of cells), n <= 1600 (32-bit cell indices).  partials_dev holds
// kDiagPartials doubles: the last is the kernel's error word and its count of finished CTAs (zero when
// allocated; the error word is set if a bounded wait between its warps gave up, and cleared by the launch's
// final sum, which copies it to *flag_out when flag_out is given and then writes NaN diagnostics).
// out_dev and flag_out may be pinned host memory.
cudaError_t launch_diag_pop(int storage, int layout, const void* f, int n, double* partials_dev, double* out_dev,
                            double* flag_out, cudaStream_t st);
inline bool diag_pop_ok(int storage, int n) { return storage >= 0 && storage <= 2 && n % 2 == 0 && n <= 1600; }

// Q-criterion, speed and (vel != nullptr) velocity of a macro field of edge n into device arrays.
cudaError_t launch_qspeed(bool field_is_double, bool float_diff, const void* field, int n, float* Q, float* speed,
                          float* vel, cudaStream_t st);

// Count of kernel launches issued by this library (for the bench's launch accounting).
void note_launch(int k = 1);
long long launch_count();
long long thread_launch_count();  // of the calling thread

}  // namespace jp
