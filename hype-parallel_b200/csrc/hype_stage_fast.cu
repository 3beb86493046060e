// hype_stage_fast.cu -- the FP64 performance form of the primitive-variable
// stage kernel (HYPE_PREC_FP64_FAST): stage_tile with FastSystem / ReconFast
// (hype_physics_fast.cuh).  This translation unit is built with FMA contraction
// (no --fmad=false): products and sums fuse where the compiler finds them, so
// its results differ from the reference's in the last bits; the tests hold
// them to a relative L-infinity difference of 1e-12 per RHS evaluation.
//
// Compiled once with HYPE_STAGE_SYS and HYPE_STAGE_ORDER for each system and order and once
// without, as hype_stage.cu.
#include <cuda.h>
#include <cuda_runtime.h>
#include "hype_stage_tile.cuh"

namespace hype {

struct FastEntry {
    const void *fn;
    const void *rhs;
    const void *axpy, *mix;   // of the whole grid, by mode
    int mix_mode;
    size_t smem;
    int threads;
};

template <int SYS, int N> FastEntry fast_entry_of(int cells);

#ifdef HYPE_STAGE_SYS
template <int SYS, int N, int CELLS>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_fast_kernel(const __grid_constant__ CUtensorMap tmap, const StageParams p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stage_tile<SYS, N, CELLS, false, false, true>(p, &tmap, blockIdx.x, p.run0 + (int)blockIdx.y, smem_raw);
}

template <int SYS, int N, int CELLS>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_fast_rhs_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ RhsParams p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stage_tile<SYS, N, CELLS, false, false, true, true>(p, &tmap, blockIdx.x, p.run0 + (int)blockIdx.y, smem_raw);
}

template <int SYS, int N, int CELLS, int MODE>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_fast_mode_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ ModeParams<MODE> p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stage_tile<SYS, N, CELLS, false, false, true>(p, &tmap, blockIdx.x, p.run0 + (int)blockIdx.y, smem_raw);
}

template <int SYS, int N, int CELLS>
static FastEntry fast_of()
{
    auto fn = [](auto *f) { return reinterpret_cast<const void *>(f); };
    FastEntry e{};
    e.fn = fn(stage_fast_kernel<SYS, N, CELLS>);
    e.rhs = fn(stage_fast_rhs_kernel<SYS, N, CELLS>);
    e.axpy = fn(stage_fast_mode_kernel<SYS, N, CELLS, OUT_AXPY>);
    if constexpr (N > 0) e.mix = fn(stage_fast_mode_kernel<SYS, N, CELLS, MIX_MODE<N>>);
    e.mix_mode = MIX_MODE<N>;
    e.smem = StageKernel<SYS, N, CELLS>::smem_bytes();
    e.threads = 2 * CELLS;
    return e;
}

template <int SYS, int N>
FastEntry fast_entry_of(int cells)
{
    return cells == 64 ? fast_of<SYS, N, 64>() : fast_of<SYS, N, 128>();
}
template FastEntry fast_entry_of<HYPE_STAGE_SYS, HYPE_STAGE_ORDER>(int cells);

}  // namespace hype
#else
template <int SYS>
static FastEntry fast_sys(int order, int cells)
{
    switch (order) {
    case 0: return fast_entry_of<SYS, 0>(cells);
    case 1: return fast_entry_of<SYS, 1>(cells);
    case 2: return fast_entry_of<SYS, 2>(cells);
    default: return fast_entry_of<SYS, 3>(cells);
    }
}

static FastEntry fast_entry(int sys, int order, int cells)
{
    switch (sys) {
    case SYS_EULER: return fast_sys<SYS_EULER>(order, cells);
    case SYS_KAPILA: return fast_sys<SYS_KAPILA>(order, cells);
    default: return fast_sys<SYS_BN>(order, cells);
    }
}

cudaError_t stage_fast_configure(int sys, int order, int cells)
{
    const FastEntry e = fast_entry(sys, order, cells);
    for (const void *f : {e.fn, e.rhs, e.axpy, e.mix}) {
        const cudaError_t r = f ? cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e.smem) : cudaSuccess;
        if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
}

int stage_fast_blocks_per_sm(int sys, int order, int cells)
{
    const FastEntry e = fast_entry(sys, order, cells);
    int nb = 0;
    if (cudaFuncSetAttribute(e.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e.smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, e.fn, e.threads, e.smem) != cudaSuccess) return 0;
    return nb;
}

cudaError_t launch_stage_fast(int sys, int order, int cells, const CUtensorMap &tmap, const StageParams &p, cudaStream_t s)
{
    const FastEntry e = fast_entry(sys, order, cells);
    CUtensorMap tm = tmap;
    StageParams pp = p;
    void *args[] = {&tm, &pp};
    const unsigned gy = (unsigned)(p.run_count > 0 ? p.run_count : p.runs);
    const bool whole = !p.out_aos && !p.row_off && !p.col_off && !p.push_lo && !p.push_hi;
    const void *f = whole && p.mode == OUT_AXPY ? e.axpy : whole && e.mix && p.mode == e.mix_mode ? e.mix : e.fn;
    return cudaLaunchKernel(f, dim3((unsigned)p.strips, gy, 1), dim3((unsigned)e.threads, 1, 1), args, e.smem, s);
}

cudaError_t launch_stage_fast_rhs(int sys, int order, int cells, const CUtensorMap &tmap, const StageParams &p, cudaStream_t s)
{
    const FastEntry e = fast_entry(sys, order, cells);
    CUtensorMap tm = tmap;
    RhsParams pp;
    static_cast<StageParams &>(pp) = p;
    void *args[] = {&tm, &pp};
    const unsigned gy = (unsigned)(p.run_count > 0 ? p.run_count : p.runs);
    return cudaLaunchKernel(e.rhs, dim3((unsigned)p.strips, gy, 1), dim3((unsigned)e.threads, 1, 1), args, e.smem, s);
}

// fast_rcp and IEEE division of the same arguments, for the accuracy test
__global__ void rcp_check_kernel(const double *x, double *fast, double *ieee, int n)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        fast[k] = fast_rcp(x[k]);
        ieee[k] = 1.0 / x[k];
    }
}

}  // namespace hype

// Test entry point (no counterpart in the reference): fast_rcp(x[k]) and the
// IEEE quotient 1.0 / x[k] on `device`, for host arrays of n values.
extern "C" HYPE_API int hype_test_fast_rcp(int device, const double *x, int n, double *fast, double *ieee)
{
    if (!x || !fast || !ieee || n <= 0) return HYPE_ERR_INVALID;
    int prev = 0;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return HYPE_ERR_NO_DEVICE;
    struct Restore { int d; ~Restore() { cudaSetDevice(d); } } restore{prev};
    double *d = nullptr;
    const size_t bytes = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 3 * bytes) != cudaSuccess) return HYPE_ERR_NOMEM;
    int rc = HYPE_OK;
    if (cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice) != cudaSuccess) rc = HYPE_ERR_CUDA;
    if (rc == HYPE_OK) {
        hype::rcp_check_kernel<<<(n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024, 256>>>(d, d + n, d + 2 * (size_t)n, n);
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) rc = HYPE_ERR_CUDA;
    }
    if (rc == HYPE_OK && (cudaMemcpy(fast, d + n, bytes, cudaMemcpyDeviceToHost) != cudaSuccess ||
                          cudaMemcpy(ieee, d + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost) != cudaSuccess))
        rc = HYPE_ERR_CUDA;
    cudaFree(d);
    return rc;
}
#endif
