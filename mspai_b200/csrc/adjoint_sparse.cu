// Adjoint of scalar columns on the sparse form of their least-squares problem
// (fixed_sparse.cuh), four warps per column.
//
// The general adjoint (adjoint.cu) sorts the entries of C(:, J_k) in a slot of
// global memory sized for the largest column and takes lambda_k from a
// triangular factor.  Here the shared rows are found and laid out in shared
// memory, the residual and C lambda are formed on them alone, and lambda_k =
// (C_k^T C_k)^-1 gbar_k comes from the certified Chebyshev iteration
// (fixed_cg.cuh), which needs no factor: FP32 steps restarted from the FP64
// residual gbar - C^T C lambda, to the rounding level, when the kept factors
// are FP32, FP64 steps otherwise.  A row with one entry v of column j has
// r = -v x_j and C lambda = v lambda_j, so its gradient needs no row at all:
//     dL/dv = 2 w v x_j^2 - 2 v x_j lambda_j.
// A column that does not fit the slot goes to the next launch (a larger one), one
// that is not certified to the general adjoint at once.
//   Bound: the passes over the entries of C and the FP64 atomics on dC.  12,000
//   ragged columns of 134 unknowns and 2,500 entries with a gbar: 17.9 ms in the
//   general adjoint, 2.4 ms here.
#include "fixed_cg.cuh"

#include <algorithm>

namespace mspai {

namespace {

template <class T, int NW, int K>
__device__ Taken adjoint_column(CgShared& sh, const Problem& pb, const AdjointIO& io, int col,
                                char* base, int cap, int widest)
{
    constexpr int NT = 32 * NW, LG = NT / 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = lane >> 3, l8 = lane & 7;
    SharedEntries g;
    const Taken fit = gather_shared<NW>(sh, pb, col, base, cap, LG + NT * (K - 1), widest, g);
    if (fit != Taken::kYes)
        return fit;
    const int n = g.n;
    // ---- the rest of the slot: M's values by position, the residual of the
    // shared rows, gbar by position, one bit per entry of C(:, J) (shared)
    double* xm = reinterpret_cast<double*>(base + ((g.free_lo + 15) & ~15));
    double* yr = xm + n;
    double* gb = yr + g.S;
    uint32_t* bits = reinterpret_cast<uint32_t*>(gb + (io.gbar ? n : 0));
    const int words = (g.E + 31) / 32;
    if (reinterpret_cast<char*>(bits + words) > base + g.free_hi)
        return Taken::kLarger;
    int at[K], parity = 0;
    const int nlong = column_slots<NW, K>(sh, n, at);
    if (!column_scales<NW, K>(g, at))
        return Taken::kNo;
    // ---- r = b - C m on the shared rows; ||r||^2, the target outside of I
    double part = 0.0, gx = 0.0;
#pragma unroll
    for (int t = 0; t < K; t++) {
        if (at[t] < n) {
            const int jj = g.ccol[at[t]];
            const double x = io.mval[g.p0 + jj];
            xm[at[t]] = x;
            g.xs[at[t]] = x;
            part += x * x * g.d0[jj];
            if (io.gbar) {
                const double q = io.gbar[g.p0 + jj];
                gb[at[t]] = q;
                gx += q * x;
            }
        }
    }
    for (int i = tid; i < words; i += NT)
        bits[i] = 0;
    shared_residual<NW, K>(sh, g, at, true);
    for (int i = tid; i < g.S; i += NT)
        yr[i] = g.y[i];
#pragma unroll 1
    for (int c = lane; c < g.nc; c += 32) {
        const uint32_t id = g.cand[-NW * c].x;
        if (id != kNone && (id & kFirst)) {
            const double v = g.y[id & ~kFirst];
            part += v * v;
        }
    }
    const int64_t tg0 = pb.bptr ? pb.bptr[col] : 0;
    const int ntg = pb.bptr ? static_cast<int>(pb.bptr[col + 1] - tg0) : 1;
    if (tid < ntg && g.tg_rid < 0)
        part += g.tg_val * g.tg_val;
    // ---- lambda in xs, -C lambda on the shared rows in y
    if (io.gbar) {
        __syncthreads();
        if (cg_solve<T, NW, K>(sh, parity, g, at, nlong, gb, nullptr) < 0)
            return Taken::kNo;
    }
    else {
        __syncthreads();
#pragma unroll
        for (int t = 0; t < K; t++)
            if (at[t] < n)
                g.xs[at[t]] = 0.0;
        for (int i = tid; i < g.S; i += NT)
            g.y[i] = 0.0;
    }
    // nothing of the column was written up to here
    // ---- entry numbers: g.tmp[i] = entries before C(:, J(i))
    if (warp == 0) {
        uint32_t run = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            uint32_t len = 0;
            if (i < n) {
                const int j = pb.pidx[g.p0 + i];
                len = static_cast<uint32_t>(pb.cptr[j + 1] - pb.cptr[j]);
            }
            uint32_t s = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(kNone, s, o);
                if (lane >= o)
                    s += u;
            }
            if (i < n)
                g.tmp[i] = run + s - len;
            run += __shfl_sync(kNone, s, 31);
        }
    }
    __syncthreads();
    // ---- shared entries
    const double w2 = 2.0 * io.wres;
#pragma unroll 1
    for (int c = lane; c < g.nc; c += 32) {
        const uint2 e = g.cand[-NW * c];
        if (e.x == kNone)
            continue;
        const uint32_t jj = e.y >> 16, li = e.y & 0xffffu;
        const uint32_t bit = g.tmp[jj] + li;
        atomicOr(&bits[bit >> 5], 1u << (bit & 31));
        const int p = g.cpos[jj], row = static_cast<int>(e.x & ~kFirst);
        // y is -C lambda
        const double gv = yr[row] * (g.xs[p] - w2 * xm[p]) + g.y[row] * xm[p];
        atomicAdd(&io.dC[g.cb[jj] + li], gv);
    }
    __syncthreads();
    // ---- entries alone in their row
    for (int c0 = 4 * warp; c0 < n; c0 += 4 * NW) {
        const int ci = c0 + grp;
        if (ci >= n)
            continue;
        const uint32_t first = g.tmp[ci];
        const int len = static_cast<int>((ci + 1 < n ? g.tmp[ci + 1] : g.E) - first);
        const int p = g.cpos[ci];
        const double x = xm[p], f = x * (w2 * x - 2.0 * g.xs[p]);
        for (int q = l8; q < len; q += 8) {
            const uint32_t bit = first + q;
            if (!((bits[bit >> 5] >> (bit & 31)) & 1u))
                atomicAdd(&io.dC[g.cb[ci] + q], f * __ldg(pb.cval + g.cb[ci] + q));
        }
    }
    if (io.dB && pb.bptr && tid < ntg)
        io.dB[tg0 + tid] =
            g.tg_rid >= 0 ? w2 * yr[g.tg_rid] - g.y[g.tg_rid] : w2 * g.tg_val;
    cta_sum2<NW>(sh, parity, part, gx);
    if (tid == 0)
        io.loss[col] = io.wres * part + gx;
    return Taken::kYes;
}

template <class T, int NW, int K, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB)
    adjoint_sparse_kernel(Problem pb, AdjointIO io, const int32_t* __restrict__ list,
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
        const Taken taken = adjoint_column<T, NW, K>(sh, pb, io, col, smem, slot_bytes, widest);
        if (taken != Taken::kYes && threadIdx.x == 0) {
            const WorkList& to = taken == Taken::kLarger ? larger : refused;
            to.list[atomicAdd(to.count, 1)] = col;
        }
    }
}

template <class T, int NW, int K, int MINB>
cudaError_t launch_t(int slot_bytes, int widest, const Problem& pb, const AdjointIO& io,
                     const int32_t* list, const int32_t* count_dev, int count_host,
                     int32_t* counter, const WorkList& larger, const WorkList& refused,
                     cudaStream_t st)
{
    auto kern = adjoint_sparse_kernel<T, NW, K, MINB>;
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
    const int grid = std::max(1, std::min(per_sm * num_sms(), count_host));
    kern<<<grid, 32 * NW, slot_bytes, st>>>(pb, io, list, count_dev, count_host, counter, larger,
                                            refused, slot_bytes, widest);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_adjoint_sparse(const Problem& pb, const AdjointIO& io, const int32_t* list,
                                  int count, int32_t* const rest[3], int32_t* counts,
                                  cudaStream_t st)
{
    // slots of six, four and two CTAs per SM
    constexpr int kNarrow = 34 * 1024, kMiddle = 52 * 1024, kWide = 108 * 1024;
    const bool f = io.rstore && io.r_elem == 4;
    auto a = f ? launch_t<float, 4, 2, 6> : launch_t<double, 4, 2, 6>;
    auto b = f ? launch_t<float, 4, 3, 4> : launch_t<double, 4, 3, 4>;
    auto c = f ? launch_t<float, 4, 4, 2> : launch_t<double, 4, 4, 2>;
    const WorkList refused{rest[0], counts}, r1{rest[1], counts + 1}, r2{rest[2], counts + 2};
    cudaError_t e = a(kNarrow, kWide, pb, io, list, nullptr, count, counts + 3, r1, refused, st);
    if (e == cudaSuccess)
        e = b(kMiddle, kWide, pb, io, r1.list, r1.count, count, counts + 4, r2, refused, st);
    if (e == cudaSuccess)
        e = c(kWide, kWide, pb, io, r2.list, r2.count, count, counts + 5, refused, refused, st);
    return e;
}

}  // namespace mspai
