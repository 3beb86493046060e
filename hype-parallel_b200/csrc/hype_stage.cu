// hype_stage.cu -- the primitive-variable stage kernels (RHSFunctionPrim,
// rhs_function_prim.c:12-626) in their grid form (one block per tile) and
// persistent form (blocks walk a work-list of tiles of many grids), and the
// host dispatch over (system, order, tile width).  The tile itself is
// stage_tile in hype_stage_tile.cuh.
//
// Compiled with HYPE_STAGE_SYS and HYPE_STAGE_ORDER for each system and order, once for the grid form and
// once, with HYPE_STAGE_BATCH, for the persistent one (the kernels, side by side in as many compiler
// processes), and once without (the dispatch).  An object is one module, which a process loads
// whole with its first kernel.
//
// Built with --fmad=false: arithmetic rounds exactly as the reference's C does.
#include <cuda.h>
#include <cuda_runtime.h>
#include <initializer_list>
#include <type_traits>
#include "hype_stage_tile.cuh"

namespace hype {

// the kernels of a system, order and tile width
struct StageEntry {
    const void *single;
    const void *rhs;
    const void *axpy, *mix;   // of the whole grid, by mode
    size_t smem;
    int threads;
    int aos_box;   // elements of one part of a cell-major row's box
    int mix_mode;
};
struct BatchEntry {
    const void *axpy, *mix, *rk;   // by mode; rk: N = 3's fifth stage, else null
    size_t smem;
    int threads;
    int mix_mode;
};

template <int SYS, int N> StageEntry stage_entry_of(int cells);
template <int SYS, int N> BatchEntry batch_entry_of(int cells);

#if defined(HYPE_STAGE_SYS) && !defined(HYPE_STAGE_BATCH)
template <int SYS, int N, int CELLS>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_kernel(const __grid_constant__ CUtensorMap tmap, const StageParams p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stage_tile<SYS, N, CELLS, false>(p, &tmap, blockIdx.x, p.run0 + (int)blockIdx.y, smem_raw);
}

template <int SYS, int N, int CELLS, int MODE>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_mode_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ ModeParams<MODE> p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stage_tile<SYS, N, CELLS, false>(p, &tmap, blockIdx.x, p.run0 + (int)blockIdx.y, smem_raw);
}

// The right-hand side from and to the caller's cell-major arrays (tmap: p.in, 2-D, rows of
// nx NV values)
template <int SYS, int N, int CELLS>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_rhs_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ RhsParams p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    stage_tile<SYS, N, CELLS, false, false, false, true>(p, &tmap, blockIdx.x, p.run0 + (int)blockIdx.y, smem_raw);
}

template <int SYS, int N, int CELLS>
static StageEntry entry_of()
{
    using K = StageKernel<SYS, N, CELLS>;
    auto fn = [](auto *f) { return reinterpret_cast<const void *>(f); };
    StageEntry e{};
    e.single = fn(stage_kernel<SYS, N, CELLS>);
    e.rhs = fn(stage_rhs_kernel<SYS, N, CELLS>);
    e.axpy = fn(stage_mode_kernel<SYS, N, CELLS, OUT_AXPY>);
    if constexpr (N > 0) e.mix = fn(stage_mode_kernel<SYS, N, CELLS, MIX_MODE<N>>);
    e.smem = K::smem_bytes();
    e.threads = 2 * CELLS;
    e.aos_box = K::AOS_BOX;
    e.mix_mode = MIX_MODE<N>;
    return e;
}

template <int SYS, int N>
StageEntry stage_entry_of(int cells)
{
    return cells == 64 ? entry_of<SYS, N, 64>() : entry_of<SYS, N, 128>();
}
template StageEntry stage_entry_of<HYPE_STAGE_SYS, HYPE_STAGE_ORDER>(int cells);
#elif defined(HYPE_STAGE_SYS)
// Persistent form: the block walks a list of (grid, tile) work items; every grid
// has its own parameters, tensor map and device scalars.
template <int SYS, int N, int CELLS, int MODE>
__global__ void __launch_bounds__(2 * CELLS, (StageKernel<SYS, N, CELLS>::MIN_BLOCKS))
stage_batch_kernel(const StageParams *__restrict__ inst, const CUtensorMap *__restrict__ tmaps,
                   const int2 *__restrict__ work, int *__restrict__ sched)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int item_s;
    // the item's parameters live in shared memory: re-read after every barrier
    // of the tile instead of pinning registers for the whole tile
    __shared__ BatchParamsOf<MODE> p_s;
    const int nwork = sched[0];
    const DevScalars *last = nullptr;
    for (;;) {
        const int w = work_take(sched, nwork, last, &item_s);
        if (w >= nwork) break;
        const int2 it = work[w];
        if (threadIdx.x == 0) {
            p_s.load(inst[it.x], item_refine(it.y));
            fence_tensormap_acquire(&tmaps[it.x]);
        }
        __syncthreads();
        const int tile = item_tile(it.y);
        stage_tile<SYS, N, CELLS, false>(p_s, &tmaps[it.x], tile % p_s.strips, tile / p_s.strips, smem_raw);
        last = p_s.sc;
    }
    work_finish(sched);
}

template <int SYS, int N, int CELLS>
static BatchEntry entry_of()
{
    using K = StageKernel<SYS, N, CELLS>;
    auto fn = [](auto *f) { return reinterpret_cast<const void *>(f); };
    BatchEntry e{};
    e.axpy = fn(stage_batch_kernel<SYS, N, CELLS, OUT_AXPY>);
    if constexpr (N > 0) e.mix = fn(stage_batch_kernel<SYS, N, CELLS, MIX_MODE<N>>);
    if constexpr (N == 3) e.rk = fn(stage_batch_kernel<SYS, N, CELLS, OUT_RK104_5>);
    e.smem = K::smem_bytes();
    e.threads = 2 * CELLS;
    e.mix_mode = MIX_MODE<N>;
    return e;
}

template <int SYS, int N>
BatchEntry batch_entry_of(int cells)
{
    return cells == 64 ? entry_of<SYS, N, 64>() : entry_of<SYS, N, 128>();
}
template BatchEntry batch_entry_of<HYPE_STAGE_SYS, HYPE_STAGE_ORDER>(int cells);
#else
// ---------------------------------------------------------------------------
// host dispatch over (system, order, tile width)
// ---------------------------------------------------------------------------
template <int SYS, class Of>
static auto entry_sys(int order, Of of)
{
    switch (order) {
    case 0: return of(std::integral_constant<int, SYS>{}, std::integral_constant<int, 0>{});
    case 1: return of(std::integral_constant<int, SYS>{}, std::integral_constant<int, 1>{});
    case 2: return of(std::integral_constant<int, SYS>{}, std::integral_constant<int, 2>{});
    default: return of(std::integral_constant<int, SYS>{}, std::integral_constant<int, 3>{});
    }
}
template <class Of>
static auto entry(int sys, int order, Of of)
{
    switch (sys) {
    case SYS_EULER: return entry_sys<SYS_EULER>(order, of);
    case SYS_KAPILA: return entry_sys<SYS_KAPILA>(order, of);
    default: return entry_sys<SYS_BN>(order, of);
    }
}
static StageEntry stage_entry(int sys, int order, int cells)
{
    return entry(sys, order, [cells](auto s, auto n) { return stage_entry_of<decltype(s)::value, decltype(n)::value>(cells); });
}
static BatchEntry batch_entry(int sys, int order, int cells)
{
    return entry(sys, order, [cells](auto s, auto n) { return batch_entry_of<decltype(s)::value, decltype(n)::value>(cells); });
}

size_t stage_smem_bytes(int sys, int order, int cells) { return stage_entry(sys, order, cells).smem; }
int stage_threads(int cells) { return 2 * cells; }

static cudaError_t allow_smem(std::initializer_list<const void *> kernels, size_t smem)
{
    for (const void *f : kernels) {
        const cudaError_t r = f ? cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
        if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
}

cudaError_t stage_configure(int sys, int order, int cells)
{
    const StageEntry e = stage_entry(sys, order, cells);
    return allow_smem({e.single, e.rhs, e.axpy, e.mix}, e.smem);
}

int stage_blocks_per_sm(int sys, int order, int cells)
{
    const StageEntry e = stage_entry(sys, order, cells);
    int nb = 0;
    if (allow_smem({e.single}, e.smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, e.single, e.threads, e.smem) != cudaSuccess) return 0;
    return nb;
}

int stage_batch_blocks_per_sm(int sys, int order, int cells)
{
    const BatchEntry e = batch_entry(sys, order, cells);
    int nb = 0;
    // the grid form's `single` gives the dt of an instance that joins
    if (allow_smem({stage_entry(sys, order, cells).single, e.axpy, e.mix, e.rk}, e.smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, e.axpy, e.threads, e.smem) != cudaSuccess) return 0;
    return nb;
}

cudaError_t launch_stage(int sys, int order, int cells, const CUtensorMap &tmap, const StageParams &p, cudaStream_t s)
{
    const StageEntry e = stage_entry(sys, order, cells);
    CUtensorMap tm = tmap;
    StageParams pp = p;
    void *args[] = {&tm, &pp};
    const unsigned gy = (unsigned)(p.run_count > 0 ? p.run_count : p.runs);
    const bool whole = !p.out_aos && !p.row_off && !p.col_off && !p.push_lo && !p.push_hi;
    const void *f = whole && p.mode == OUT_AXPY ? e.axpy : whole && e.mix && p.mode == e.mix_mode ? e.mix : e.single;
    return cudaLaunchKernel(f, dim3((unsigned)p.strips, gy, 1), dim3((unsigned)e.threads, 1, 1), args, e.smem, s);
}

int stage_aos_box(int sys, int order, int cells) { return stage_entry(sys, order, cells).aos_box; }

cudaError_t launch_stage_rhs(int sys, int order, int cells, const CUtensorMap &tmap, const StageParams &p, cudaStream_t s)
{
    const StageEntry e = stage_entry(sys, order, cells);
    CUtensorMap tm = tmap;
    RhsParams pp;
    static_cast<StageParams &>(pp) = p;
    void *args[] = {&tm, &pp};
    const unsigned gy = (unsigned)(p.run_count > 0 ? p.run_count : p.runs);
    return cudaLaunchKernel(e.rhs, dim3((unsigned)p.strips, gy, 1), dim3((unsigned)e.threads, 1, 1), args, e.smem, s);
}

cudaError_t launch_stage_batch(int sys, int order, int cells, int mode, const StageParams *inst, const CUtensorMap *tmaps,
                               const int2 *work, int *sched, int blocks, cudaStream_t s)
{
    const BatchEntry e = batch_entry(sys, order, cells);
    void *args[] = {&inst, &tmaps, &work, &sched};
    const void *f = mode == OUT_AXPY ? e.axpy : mode == OUT_RK104_5 ? e.rk : mode == e.mix_mode ? e.mix : nullptr;
    if (!f) return cudaErrorInvalidValue;
    return cudaLaunchKernel(f, dim3((unsigned)blocks, 1, 1), dim3((unsigned)e.threads, 1, 1), args, e.smem, s);
}

#endif

}  // namespace hype
