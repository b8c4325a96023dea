// Warp-per-column solvers of small scalar columns (the other kernels of the
// batched setup: spai_kernels.cu).
//
// The generic column solver is passed once or twice by a column of few unknowns,
// by 16 warps of an SM at different places: unrolled, its code does not stay in
// the instruction caches (adaptive 48^3 columns: 8.2 of 15.5 warps per issue
// waited for instructions, 2.8 ms; rolled 1.9 ms).
#define MSPAI_LOOP _Pragma("unroll 1")
#include "spai_kernels.h"
#include "spai_solve.cuh"

#include <algorithm>

namespace mspai {

template <class T>
__global__ void __launch_bounds__(kWarpKernelThreads)
    warp_solve_kernel(Problem pb, Caps cap, Output out, const int32_t* __restrict__ list,
                      int count, int32_t* __restrict__ counter, int slot_bytes)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ GroupScratch sc[kWarpKernelThreads / 32];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    WarpGroup g{&sc[w]};
    pb.bs = 1;  // scalar columns only: the block code and its local arrays go
    pb.qru = 0;
    SlotLayout<T> lay(cap, false);
    Slot<T> s = lay.at(smem + static_cast<size_t>(w) * slot_bytes, nullptr);
    while (true) {
        int t = 0;
        if (lane == 0)
            t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= count)
            break;
        solve_column<T>(g, pb, cap, s, out, list[t]);
    }
}

// A warp per column with the slot in global memory (scratch + slot_bytes per
// warp): the tiny bucket of adaptive setups, whose candidate bit vector over
// all problem columns does not fit a shared-memory slot.
template <class T>
__global__ void __launch_bounds__(kWarpKernelThreads)
    warp_solve_global_kernel(Problem pb, Caps cap, Output out, const int32_t* __restrict__ list,
                             int count, int32_t* __restrict__ counter, char* __restrict__ scratch,
                             size_t slot_bytes)
{
    __shared__ GroupScratch sc[kWarpKernelThreads / 32];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    WarpGroup g{&sc[w]};
    pb.bs = 1;  // scalar columns only: the block code and its local arrays go
    pb.qru = 0;
    SlotLayout<T> lay(cap, false);
    const size_t slot_id = static_cast<size_t>(blockIdx.x) * (kWarpKernelThreads / 32) + w;
    Slot<T> s = lay.at(scratch + slot_id * slot_bytes, nullptr);
    while (true) {
        int t = 0;
        if (lane == 0)
            t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= count)
            break;
        solve_column<T>(g, pb, cap, s, out, list[t]);
    }
}

// The same with the whole slot in shared memory, for adaptive scalar columns
// that end within kShareN unknowns and kShareE entries (FP64, no refinement);
// a column that outgrows it is appended to rest and starts again in the kernel
// above.  The arrays of the pattern update take W's place, which is dead by
// then; the candidates are collected in a hash set instead of a bit vector.
//   Bound: latency, 16 warps per SM (registers; the slots take 91 KB per CTA of
//   eight).  Convection-diffusion 48^3, 110,592 columns of one and then about
//   five unknowns: the setup took 5.9 ms in the kernel above as it was, 2.3 ms here
//   (3.2 ms with unrolled loops).
// The bounds hold three updates of five unknowns on a 7-point stencil; larger
// slots would leave fewer than 16 warps on an SM.
constexpr int kShareN = 16;
constexpr int kShareE = 112;      // 16 columns of a 7-point stencil
constexpr int kShareMw = 44;      // rows of the folded matrix
constexpr int kShareCand = 192;   // unique candidates
static_assert(kShareCand + 32 < kCandTable, "a probe meets a free place: the scan ends here");

struct ShareSlot {
    uint64_t keys[kShareE];
    double ev[kShareE], r[kShareE], x[kShareN], gv[kShareN];
    union {
        double W[kShareMw * (kShareN + 1)];
        struct {
            double rho[kShareCand];
            int32_t cand[256];  // next_pow2(kShareCand)
            int32_t ctmp[kShareCand + 1];
            int32_t ctab[kCandTable];
        } u;
    };
    int32_t J[kShareN + kShareMn], off[kShareN + 1], ejj[kShareE], pos[kShareE + 1], I[kShareE],
        rstart[kShareE + 1], tmp[kShareE + 1];
};

__global__ void __launch_bounds__(kWarpKernelThreads, 2)
    warp_adaptive_kernel(Problem pb, Output out, const int32_t* __restrict__ list, int count,
                         int32_t* __restrict__ counter, int32_t* __restrict__ rest,
                         int32_t* __restrict__ rest_count)
{
    // constants here: the solver's other branches go
    pb.bs = 1;
    pb.qru = 0;
    pb.refine = 0;
    __builtin_assume(pb.ns > 0);
    out.rstore = nullptr;
    Caps cap{};
    cap.emax = kShareE;
    cap.nmax = kShareN;
    cap.mwmax = kShareMw;
    cap.cmax = kShareCand;
    cap.nrhs = 1;
    extern __shared__ __align__(16) char smem[];
    __shared__ GroupScratch sc[kWarpKernelThreads / 32];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    WarpGroup g{&sc[w]};
    ShareSlot& a = reinterpret_cast<ShareSlot*>(smem)[w];
    Slot<double> s{};
    s.J = a.J;
    s.off = a.off;
    s.ejj = a.ejj;
    s.ev = a.ev;
    s.pos = a.pos;
    s.keys = a.keys;
    s.I = a.I;
    s.rstart = a.rstart;
    s.tmp = a.tmp;
    s.r = a.r;
    s.W = s.Wfast = a.W;
    s.wfast_elems = kShareMw * (kShareN + 1);
    s.x = a.x;
    s.gv = a.gv;
    s.cand = a.u.cand;
    s.ctmp = a.u.ctmp;
    s.rho = a.u.rho;
    s.ctab = a.u.ctab;
    while (true) {
        int t = 0;
        if (lane == 0)
            t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= count)
            break;
        const int col = list[t];
        solve_column<double>(g, pb, cap, s, out, col);
        if (lane == 0 && out.status[col] == 3) {
            for (int q = 0; q < 3; q++)
                out.work[3 * static_cast<size_t>(col) + q] = 0.0;
            rest[atomicAdd(rest_count, 1)] = col;
        }
    }
}

template <class T>
static cudaError_t launch_warp_t(const Problem& pb, const Caps& cap, const Output& out,
                                 const int32_t* list, int count, int32_t* counter, cudaStream_t st,
                                 int* grid_out)
{
    const int slot = static_cast<int>(SlotLayout<T>(cap, false).bytes);
    const size_t smem = static_cast<size_t>(slot) * (kWarpKernelThreads / 32);
    cudaError_t e = cudaFuncSetAttribute(warp_solve_kernel<T>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, warp_solve_kernel<T>,
                                                      kWarpKernelThreads, smem);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    int grid = per_sm * num_sms();
    const int need = (count + kWarpKernelThreads / 32 - 1) / (kWarpKernelThreads / 32);
    grid = std::max(1, std::min(grid, need));
    *grid_out = grid;
    warp_solve_kernel<T><<<grid, kWarpKernelThreads, smem, st>>>(pb, cap, out, list, count,
                                                                   counter, slot);
    return cudaGetLastError();
}

template <class T>
static int warp_global_grid(int count)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, warp_solve_global_kernel<T>,
                                                  kWarpKernelThreads, 0);
    const int need = (count + kWarpKernelThreads / 32 - 1) / (kWarpKernelThreads / 32);
    return std::max(1, std::min(std::max(per_sm, 1) * num_sms(), need));
}

size_t warp_global_scratch_bytes(const Caps& cap, int elem_bytes, int count)
{
    const int grid = elem_bytes == 4 ? warp_global_grid<float>(count) : warp_global_grid<double>(count);
    return warp_slot_bytes(cap, elem_bytes) * static_cast<size_t>(grid) * (kWarpKernelThreads / 32);
}

template <class T>
static cudaError_t launch_warp_global_t(const Problem& pb, const Caps& cap, const Output& out,
                                        const int32_t* list, int count, int32_t* counter,
                                        char* scratch, size_t scratch_bytes, cudaStream_t st,
                                        int* grid_out)
{
    const size_t slot = SlotLayout<T>(cap, false).bytes;
    int grid = warp_global_grid<T>(count);
    grid = std::max(1, std::min<int>(grid, static_cast<int>(
                                               scratch_bytes / (slot * (kWarpKernelThreads / 32)))));
    *grid_out = grid;
    warp_solve_global_kernel<T><<<grid, kWarpKernelThreads, 0, st>>>(pb, cap, out, list, count,
                                                                     counter, scratch, slot);
    return cudaGetLastError();
}

cudaError_t launch_warp_solve_global(int elem_bytes, const Problem& pb, const Caps& cap,
                                     const Output& out, const int32_t* list, int count,
                                     int32_t* counter, char* scratch, size_t scratch_bytes,
                                     cudaStream_t st, int* grid_out)
{
    if (elem_bytes == 4)
        return launch_warp_global_t<float>(pb, cap, out, list, count, counter, scratch,
                                           scratch_bytes, st, grid_out);
    return launch_warp_global_t<double>(pb, cap, out, list, count, counter, scratch,
                                        scratch_bytes, st, grid_out);
}

cudaError_t launch_warp_adaptive(const Problem& pb, const Output& out, const int32_t* list,
                                 int count, int32_t* counter, int32_t* rest,
                                 int32_t* rest_count, cudaStream_t st)
{
    const size_t smem = sizeof(ShareSlot) * (kWarpKernelThreads / 32);
    cudaError_t e = cudaFuncSetAttribute(warp_adaptive_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, warp_adaptive_kernel,
                                                      kWarpKernelThreads, smem);
    if (e != cudaSuccess)
        return e;
    const int need = (count + kWarpKernelThreads / 32 - 1) / (kWarpKernelThreads / 32);
    const int grid = std::max(1, std::min(std::max(per_sm, 1) * num_sms(), need));
    warp_adaptive_kernel<<<grid, kWarpKernelThreads, smem, st>>>(pb, out, list, count, counter,
                                                                 rest, rest_count);
    return cudaGetLastError();
}

cudaError_t launch_warp_solve(int elem_bytes, const Problem& pb, const Caps& cap,
                              const Output& out, const int32_t* list, int count, int32_t* counter,
                              cudaStream_t st, int* grid_out)
{
    if (elem_bytes == 4)
        return launch_warp_t<float>(pb, cap, out, list, count, counter, st, grid_out);
    return launch_warp_t<double>(pb, cap, out, list, count, counter, st, grid_out);
}

}  // namespace mspai
