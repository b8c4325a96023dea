// Launches of the solvers on the sparse normal equations (fixed_cg.cuh): a CTA per
// column from a work list with an atomic counter.  A column that does not fit
// the slot goes to the next launch's list (a larger slot); one that no slot would
// take, that has no certificate or does not converge goes to the dense
// factorizations at once.
#include "fixed_cg.cuh"

#include <algorithm>

namespace mspai {

// Solves column `col`; nothing of it is written unless it is taken (uniformly).
// AGAIN: a re-setup, which starts from M's previous values; a column that is too
// far from them is left to the launches without.  (Kernels of their own: at 64
// registers a thread the choice costs the other setups 2 % of their time, and a
// second start in the same kernel the re-setups 1.5 %.)
template <class T, int NW, int K, bool AGAIN>
__device__ Taken sparse_column(CgShared& sh, const Problem& pb, const Output& out, int col,
                               char* base, int cap, int widest)
{
    constexpr int NT = 32 * NW, LG = NT / 8;
    SharedEntries g;
    const Taken fit = gather_shared<NW>(sh, pb, col, base, cap, LG + NT * (K - 1), widest, g);
    if (fit != Taken::kYes)
        return fit;
    int at[K], parity = 0;
    const int nlong = column_slots<NW, K>(sh, g.n, at);
    if (!column_scales<NW, K>(g, at))
        return Taken::kNo;
    if constexpr (NW == 1) {
        return hub_solve<T, NW, K>(sh, parity, g, pb, out, col, base, at, nlong) ? Taken::kYes
                                                                                 : Taken::kNo;
    }
    else {
        const int steps = cg_solve<T, NW, K>(sh, parity, g, at, nlong, nullptr,
                                             AGAIN ? out.oval + g.p0 : nullptr);
        if (steps < 0)
            return AGAIN && steps == -2 ? Taken::kFar : Taken::kNo;
        write_column<NW, K>(sh, parity, g, out, col, at, steps * (4.0 * g.ns + 6.0 * g.n));
        if (AGAIN && threadIdx.x == 0)
            atomicAdd(out.reuse_count, 1);
        return Taken::kYes;
    }
}

namespace {

template <class T, int NW, int K, int MINB, bool AGAIN>
__global__ void __launch_bounds__(32 * NW, MINB)
    sparse_solve_kernel(Problem pb, Output out, const int32_t* __restrict__ list,
                        const int32_t* __restrict__ count_dev, int count_host,
                        int32_t* __restrict__ counter, WorkList larger, WorkList refused,
                        WorkList far, int slot_bytes, int widest)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ CgShared sh;
    const int count = count_dev ? *count_dev : count_host;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0)
            sh.next = atomicAdd(counter, 1);
        __syncthreads();
        const int t = sh.next;
        if (t >= count)
            break;
        const int col = list[t];
        const Taken taken =
            sparse_column<T, NW, K, AGAIN>(sh, pb, out, col, smem, slot_bytes, widest);
        if (taken != Taken::kYes && threadIdx.x == 0) {
            const WorkList& to =
                taken == Taken::kLarger ? larger : (taken == Taken::kFar ? far : refused);
            to.list[atomicAdd(to.count, 1)] = col;
        }
    }
}

template <class T, int NW, int K, int MINB, bool AGAIN>
cudaError_t launch_sparse_t(int slot_bytes, int widest, const Problem& pb, const Output& out,
                            const int32_t* list, const int32_t* count_dev, int count_host,
                            int32_t* counter, const WorkList& larger, const WorkList& refused,
                            const WorkList& far, cudaStream_t st)
{
    auto kern = sparse_solve_kernel<T, NW, K, MINB, AGAIN>;
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, slot_bytes);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * NW, slot_bytes);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    int grid = per_sm * num_sms();
    if (count_dev == nullptr)
        grid = std::min(grid, std::max(count_host, 1));
    kern<<<grid, 32 * NW, slot_bytes, st>>>(pb, out, list, count_dev, count_host, counter, larger,
                                            refused, far, slot_bytes, widest);
    return cudaGetLastError();
}

// The launch of a slot class; the narrow one at eight CTAs per SM in FP32, six in
// FP64.
template <class T, bool AGAIN>
auto sparse_launch(SparseLaunch kind)
{
    auto launch = launch_sparse_t<T, 4, 2, sizeof(T) == 4 ? 8 : 6, AGAIN>;
    if (kind == SparseLaunch::kMiddle)
        launch = launch_sparse_t<T, 4, 3, 5, AGAIN>;
    else if (kind == SparseLaunch::kWide)
        launch = launch_sparse_t<T, 4, 4, 2, AGAIN>;
    return launch;
}

}  // namespace

cudaError_t launch_sparse_solve(int elem_bytes, SparseLaunch kind, int slot_bytes, int widest,
                                const Problem& pb, const Output& out, const int32_t* list,
                                const int32_t* count_dev, int count_host, int32_t* counter,
                                const WorkList& larger, const WorkList& refused, const WorkList& far,
                                cudaStream_t st)
{
    if (kind == SparseLaunch::kTiny)
        return launch_sparse_t<double, 1, 2, 16, false>(slot_bytes, widest, pb, out, list,
                                                        count_dev, count_host, counter, larger,
                                                        refused, far, st);
    const auto launch = far.list
                            ? (elem_bytes == 4 ? sparse_launch<float, true>(kind)
                                               : sparse_launch<double, true>(kind))
                            : (elem_bytes == 4 ? sparse_launch<float, false>(kind)
                                               : sparse_launch<double, false>(kind));
    return launch(slot_bytes, widest, pb, out, list, count_dev, count_host, counter, larger,
                  refused, far, st);
}

}  // namespace mspai
