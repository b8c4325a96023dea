// Launches of the solvers on the sparse normal equations (fixed_cg.cuh): a CTA per
// column from a work list with an atomic counter.  A column that does not fit
// the slot goes to the next launch's list (a larger slot); one that no slot would
// take, that has no certificate or does not converge goes to the dense
// factorizations at once.
#include "fixed_cg.cuh"

#include <algorithm>

namespace mspai {

// Solves column `col`; nothing of it is written unless it is taken (uniformly).
template <class T, int NW, int K>
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
        // a re-setup starts from M's previous values
        const double* prev = out.reuse_steps > 0 ? out.oval + g.p0 : nullptr;
        const int steps = cg_solve<T, NW, K>(sh, parity, g, at, nlong, nullptr, prev);
        if (steps < 0)
            return Taken::kNo;
        write_column<NW, K>(sh, parity, g, out, col, at, steps * (4.0 * g.ns + 6.0 * g.n));
        if (prev && threadIdx.x == 0)
            atomicAdd(out.reuse_count, 1);
        return Taken::kYes;
    }
}

namespace {

template <class T, int NW, int K, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB)
    sparse_solve_kernel(Problem pb, Output out, const int32_t* __restrict__ list,
                        const int32_t* __restrict__ count_dev, int count_host,
                        int32_t* __restrict__ counter, WorkList larger, WorkList refused,
                        int slot_bytes, int widest)
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
        const Taken taken = sparse_column<T, NW, K>(sh, pb, out, col, smem, slot_bytes, widest);
        if (taken != Taken::kYes && threadIdx.x == 0) {
            const WorkList& to = taken == Taken::kLarger ? larger : refused;
            to.list[atomicAdd(to.count, 1)] = col;
        }
    }
}

template <class T, int NW, int K, int MINB>
cudaError_t launch_sparse_t(int slot_bytes, int widest, const Problem& pb, const Output& out,
                            const int32_t* list, const int32_t* count_dev, int count_host,
                            int32_t* counter, const WorkList& larger, const WorkList& refused,
                            cudaStream_t st)
{
    auto kern = sparse_solve_kernel<T, NW, K, MINB>;
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
                                            refused, slot_bytes, widest);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sparse_solve(int elem_bytes, SparseLaunch kind, int slot_bytes, int widest,
                                const Problem& pb, const Output& out, const int32_t* list,
                                const int32_t* count_dev, int count_host, int32_t* counter,
                                const WorkList& larger, const WorkList& refused, cudaStream_t st)
{
    const bool f = elem_bytes == 4;
    auto launch = launch_sparse_t<double, 1, 2, 16>;
    if (kind == SparseLaunch::kNarrow)
        launch = f ? launch_sparse_t<float, 4, 2, 8> : launch_sparse_t<double, 4, 2, 6>;
    else if (kind == SparseLaunch::kMiddle)
        launch = f ? launch_sparse_t<float, 4, 3, 5> : launch_sparse_t<double, 4, 3, 5>;
    else if (kind == SparseLaunch::kWide)
        launch = f ? launch_sparse_t<float, 4, 4, 2> : launch_sparse_t<double, 4, 4, 2>;
    return launch(slot_bytes, widest, pb, out, list, count_dev, count_host, counter, larger,
                  refused, st);
}

}  // namespace mspai
