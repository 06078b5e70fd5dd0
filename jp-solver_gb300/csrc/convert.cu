// Populations between a solver's storage and a host's element type and layout, converted on the device.
//
// The reference has no population I/O.  jp_get_populations / jp_set_populations hand out 32- or 64-bit
// values in the flat [q][z][y][x] or the blocked [block][q][cell] order; where the storage holds another
// type (shifted 16-bit) or order (flat, in-place layouts), these kernels convert between the state and a
// device scratch that one DMA moves, chunk by chunk.  A warp takes a unit: a row of the flat order, or a
// block's population; reads and writes are coalesced along x (8 cells at a time in blocks of edge 8).
// The conversion of N=96 FP16 to blocked FP32 (16.8 M values) takes ~0.03 ms beside its transfer (0.42 ms in
// all); on one host thread it took 0.2 s.
// Values are those of the host conversion: f = w_q + stored, stored = round(f - w_q) through float.
#include "kernels.h"
#include "lattice.cuh"
#include "solver.h"

#include <algorithm>

namespace jp {

namespace {

constexpr int kUnitsPerCta = 8;  // a warp each

// element of the state that holds population q of cell (x, y, z); aa as in launch_macro
__device__ __forceinline__ size_t state_slot(int aa, size_t cells, int n, int q, int x, int y, int z) {
    if (aa == 1) {
        x += cx(q);
        y += cy(q);
        z += cz(q);
        x = x < 0 ? x + n : x >= n ? x - n : x;
        y = y < 0 ? y + n : y >= n ? y - n : y;
        z = z < 0 ? z + n : z >= n ? z - n : z;
    } else if (aa == 2) {
        q = opp(q);
    }
    return (size_t)q * cells + ((size_t)z * n + y) * n + x;
}

template <class ST, class H>
__device__ __forceinline__ H to_host(typename ST::raw v, int q) {
    if constexpr (!ST::shifted) return H(ST::load(v));
    else if constexpr (sizeof(H) == 8) return double(wf(q)) + double(ST::load(v));
    else return __fadd_rn(wf(q), ST::load(v));
}
template <class ST, class H>
__device__ __forceinline__ typename ST::raw to_stored(H v, int q) {
    if constexpr (!ST::shifted) return typename ST::raw(v);
    else if constexpr (sizeof(H) == 8) return ST::store(float(v - double(wf(q))));
    else return ST::store(__fadd_rn(v, -wf(q)));
}

template <class ST, class H, bool EXPORT>
__global__ void __launch_bounds__(kUnitsPerCta * 32) k_convert(const PopMap m, typename ST::raw* __restrict__ state,
                                                               H* __restrict__ host, long long first, long long units) {
    const long long local = (long long)blockIdx.x * kUnitsPerCta + (threadIdx.x >> 5);
    if (local >= units) return;
    const long long u = first + local;
    const int lane = threadIdx.x & 31, n = m.n, mb = m.mb;
    H* const h = host + local * m.len;
    const size_t cells = (size_t)n * n * n;
    auto move = [&](int c, size_t o, int q) {
        if constexpr (EXPORT) h[c] = to_host<ST, H>(state[o], q);
        else state[o] = to_stored<ST, H>(h[c], q);
    };
    if (m.kind == PopMap::LINEAR) {  // the state is in the host's order already
        const int q = int(u % Q);
        for (int c = lane; c < m.len; c += 32) move(c, (size_t)u * m.len + c, q);
    } else if (m.kind == PopMap::FLAT) {
        const int y = int(u % n), z = int(u / n % n), q = int(u / ((long long)n * n));
        for (int x = lane; x < n; x += 32) move(x, state_slot(m.aa, cells, n, q, x, y, z), q);
    } else {
        const int g = n / mb, q = int(u % Q);
        const long long b = u / Q;
        const int x0 = int(b % g) * mb, y0 = int(b / g % g) * mb, z0 = int(b / ((long long)g * g)) * mb;
        for (int c = lane; c < m.len; c += 32)
            move(c, state_slot(m.aa, cells, n, q, x0 + c % mb, y0 + c / mb % mb, z0 + c / (mb * mb)), q);
    }
}

template <class ST, class H>
cudaError_t launch_t(const PopMap& m, void* state, void* host, long long first, long long units, bool to_host_order,
                     cudaStream_t st) {
    using raw = typename ST::raw;
    const long long blocks = (units + kUnitsPerCta - 1) / kUnitsPerCta;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    if (to_host_order)
        k_convert<ST, H, true><<<(unsigned)blocks, kUnitsPerCta * 32, 0, st>>>(m, (raw*)state, (H*)host, first, units);
    else
        k_convert<ST, H, false><<<(unsigned)blocks, kUnitsPerCta * 32, 0, st>>>(m, (raw*)state, (H*)host, first, units);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch(int storage, int dtype, const PopMap& m, void* state, void* host, long long first, long long units,
                   bool to_host_order, cudaStream_t st) {
    const bool d = dtype == JP_F64;
    switch (storage) {
        case JP_FP32: return d ? launch_t<StF32, double>(m, state, host, first, units, to_host_order, st)
                               : launch_t<StF32, float>(m, state, host, first, units, to_host_order, st);
        case JP_FP16: return d ? launch_t<StF16, double>(m, state, host, first, units, to_host_order, st)
                               : launch_t<StF16, float>(m, state, host, first, units, to_host_order, st);
        case JP_BF16: return d ? launch_t<StBF16, double>(m, state, host, first, units, to_host_order, st)
                               : launch_t<StBF16, float>(m, state, host, first, units, to_host_order, st);
        case JP_FP64: return d ? launch_t<StF64, double>(m, state, host, first, units, to_host_order, st)
                               : launch_t<StF64, float>(m, state, host, first, units, to_host_order, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

jp_status convert_populations(jp_solver* s, int storage, int dtype, const PopMap& m, void* state, void* scratch,
                              size_t scratch_bytes, void* host, bool to_host_order) {
    const size_t unit = (size_t)m.len * (dtype == JP_F64 ? 8 : 4);
    const long long chunk = (long long)(scratch_bytes / unit);
    if (chunk < 1) return fail(JP_ERR_NOMEM, "population scratch of %zu bytes", scratch_bytes);
    cudaError_t e = cudaSuccess;
    for (long long u = 0; u < m.units && e == cudaSuccess; u += chunk) {
        const long long k = std::min(chunk, m.units - u);
        char* const h = static_cast<char*>(host) + (size_t)u * unit;
        if (to_host_order) {
            e = launch(storage, dtype, m, state, scratch, u, k, true, s->stream);
            if (e == cudaSuccess) e = cudaMemcpyAsync(h, scratch, (size_t)k * unit, cudaMemcpyDeviceToHost, s->stream);
        } else {
            e = cudaMemcpyAsync(scratch, h, (size_t)k * unit, cudaMemcpyHostToDevice, s->stream);
            if (e == cudaSuccess) e = launch(storage, dtype, m, state, scratch, u, k, false, s->stream);
        }
    }
    const cudaError_t w = cudaStreamSynchronize(s->stream);  // also after a failure: the copies use the caller's memory
    if (e == cudaSuccess) e = w;
    if (e != cudaSuccess) return cuda_fail(e, "population conversion");
    return JP_OK;
}

}  // namespace jp
