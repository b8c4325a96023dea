// Launches of the solvers on the sparse normal equations (fixed_cg.cuh): a CTA per
// column from a work list with an atomic counter; a column that is not taken
// goes to the overflow list, which the next launch (a larger slot, then the
// dense factorizations) works through.
#include "fixed_cg.cuh"

#include <algorithm>

namespace mspai {

// Solves column `col`; false (uniformly) when neither solver takes it: nothing
// of the column is written then.
template <class T, int NW, int K>
__device__ bool sparse_column(CgShared& sh, const Problem& pb, const Output& out, int col,
                              char* base, int cap)
{
    constexpr int NT = 32 * NW, LG = NT / 8;
    SharedEntries g;
    if (!gather_shared<NW>(sh, pb, col, base, cap, LG + NT * (K - 1), g))
        return false;
    int at[K], parity = 0;
    const int nlong = column_slots<NW, K>(sh, g.n, at);
    if (!column_scales<NW, K>(g, at))
        return false;
    if constexpr (NW == 1) {
        return hub_solve<T, NW, K>(sh, parity, g, pb, out, col, base, at, nlong);
    }
    else {
        // a re-setup starts from M's previous values
        const double* prev = out.reuse_steps > 0 ? out.oval + g.p0 : nullptr;
        const int steps = cg_solve<T, NW, K>(sh, parity, g, at, nlong, nullptr, prev);
        if (steps < 0)
            return false;
        write_column<NW, K>(sh, parity, g, out, col, at, steps * (4.0 * g.ns + 6.0 * g.n));
        if (prev && threadIdx.x == 0)
            atomicAdd(out.reuse_count, 1);
        return true;
    }
}

namespace {

template <class T, int NW, int K, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB)
    sparse_solve_kernel(Problem pb, Output out, const int32_t* __restrict__ list,
                        const int32_t* __restrict__ count_dev, int count_host,
                        int32_t* __restrict__ counter, int32_t* __restrict__ ovf_list,
                        int32_t* __restrict__ ovf_count, int slot_bytes)
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
        const bool done = sparse_column<T, NW, K>(sh, pb, out, col, smem, slot_bytes);
        if (!done && threadIdx.x == 0)
            ovf_list[atomicAdd(ovf_count, 1)] = col;
    }
}

template <class T, int NW, int K, int MINB>
cudaError_t launch_sparse_t(int slot_bytes, const Problem& pb, const Output& out,
                            const int32_t* list, const int32_t* count_dev, int count_host,
                            int32_t* counter, int32_t* ovf_list, int32_t* ovf_count,
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
    kern<<<grid, 32 * NW, slot_bytes, st>>>(pb, out, list, count_dev, count_host, counter, ovf_list,
                                            ovf_count, slot_bytes);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sparse_solve(int elem_bytes, SparseLaunch kind, int slot_bytes,
                                const Problem& pb, const Output& out, const int32_t* list,
                                const int32_t* count_dev, int count_host, int32_t* counter,
                                int32_t* ovf_list, int32_t* ovf_count, cudaStream_t st)
{
    const bool f = elem_bytes == 4;
    auto launch = launch_sparse_t<double, 1, 2, 16>;
    if (kind == SparseLaunch::kNarrow)
        launch = f ? launch_sparse_t<float, 4, 2, 8> : launch_sparse_t<double, 4, 2, 6>;
    else if (kind == SparseLaunch::kMiddle)
        launch = f ? launch_sparse_t<float, 4, 3, 5> : launch_sparse_t<double, 4, 3, 5>;
    else if (kind == SparseLaunch::kWide)
        launch = f ? launch_sparse_t<float, 4, 4, 2> : launch_sparse_t<double, 4, 4, 2>;
    return launch(slot_bytes, pb, out, list, count_dev, count_host, counter, ovf_list, ovf_count,
                  st);
}

}  // namespace mspai
