// Fixed-pattern scalar columns of at most eight unknowns and 64 entries of
// C(:, J): eight lanes per column, four columns per warp, FP64.
//
// Stencil problems on their own pattern (five to seven unknowns, 13 to 25 rows)
// are far smaller than a warp: the general solver spends most of a warp's
// instructions on sorting 35 entries and on sums over 32 lanes of 15 rows.
// Here lane j of a column's group walks the entries of C(:, J(j)), which are
// sorted by row: the smallest head of the eight lanes is the next row of I
// (Get_I_Set, src/Spai_Sub.imp:65-122), and every lane writes its value in that
// row or zero, so the dense C(I, J) (Create_Submatrix_AHat, :221-282) comes out
// in shared memory in row order.  Lane l then takes rows l, l + 8, ... into
// registers and the group factors them by Householder reflections (dlarfg:
// beta = -sign(alpha) ||(alpha, x)||, tau = 0 for x = 0) with three-step sums.
// The residual is formed in FP64 from the matrix in shared memory.  A column whose
// solution is not finite (a zero on R's diagonal, an overflow) is left to the general
// warp solver: on dependent columns the two meet exact zeros in different places.
//   Bound: FP64 latency (a square root and a reciprocal per reflection) at 16
//   warps per SM (128 registers, 38 KB of shared memory a CTA of four warps; columns
//   of 33 to 64 rows: 8).  Anisotropic 1024^2 with two probing rows: 13.6 ms in the
//   general warp solver, 1.6 ms here.
#include "spai_kernels.h"
#include "spai_solve.cuh"

#include <algorithm>

namespace mspai {

namespace {

constexpr uint32_t kAll = 0xffffffffu;
constexpr int kRowLd = 9;       // row stride in shared memory (doubles)
constexpr int kSmallThreads = 128;

__device__ __forceinline__ double group_sum(double v)
{
    v += __shfl_xor_sync(kAll, v, 4);
    v += __shfl_xor_sync(kAll, v, 2);
    v += __shfl_xor_sync(kAll, v, 1);
    return v;
}

// R rows per lane: columns with at most 8 R rows; the others go to rest.
template <int R>
__global__ void __launch_bounds__(kSmallThreads)
    small_qr_kernel(Problem pb, Output out, const int32_t* __restrict__ list,
                    const int32_t* __restrict__ count_dev, int count_host,
                    int32_t* __restrict__ rest, int32_t* __restrict__ rest_count,
                    WorkList refused, int32_t* __restrict__ refused_any)
{
    constexpr int M = 8 * R;
    extern __shared__ __align__(16) char smem[];
    const int lane = threadIdx.x & 31, grp = lane >> 3, l8 = lane & 7;
    const int warp = threadIdx.x >> 5;
    double* mat = reinterpret_cast<double*>(smem) + (4 * warp + grp) * (M * kRowLd);
    int32_t* rowid = reinterpret_cast<int32_t*>(
                         smem + sizeof(double) * (kSmallThreads / 8) * M * kRowLd) +
                     (4 * warp + grp) * M;
    const int count = count_dev ? *count_dev : count_host;
    const int stride = gridDim.x * (kSmallThreads / 8);
    for (int t0 = (blockIdx.x * (kSmallThreads / 32) + warp) * 4; t0 < count; t0 += stride) {
        const int t = t0 + grp;
        const int col = t < count ? list[t] : -1;
        const int64_t p0 = col >= 0 ? pb.pptr[col] : 0;
        const int n = col >= 0 ? static_cast<int>(pb.pptr[col + 1] - p0) : 0;
        // ---- rows of C(:, J) in order
        int64_t e = 0, e1 = 0;
        if (l8 < n) {
            const int j = pb.pidx[p0 + l8];
            e = pb.cptr[j];
            e1 = pb.cptr[j + 1];
        }
        int entries = static_cast<int>(e1 - e);
        entries += __shfl_xor_sync(kAll, entries, 4);
        entries += __shfl_xor_sync(kAll, entries, 2);
        entries += __shfl_xor_sync(kAll, entries, 1);
        int row = e < e1 ? __ldg(pb.cidx + e) : 0x7fffffff;
        double val = e < e1 ? __ldg(pb.cval + e) : 0.0;
        // the entry after it, on its way while a row is worked on
        int next_row = e + 1 < e1 ? __ldg(pb.cidx + e + 1) : 0x7fffffff;
        double next_val = e + 1 < e1 ? __ldg(pb.cval + e + 1) : 0.0;
        int m = 0;
        while (true) {
            int low = min(row, __shfl_xor_sync(kAll, row, 4));
            low = min(low, __shfl_xor_sync(kAll, low, 2));
            low = min(low, __shfl_xor_sync(kAll, low, 1));
            const bool more = low != 0x7fffffff;
            if (!__any_sync(kAll, more))
                break;
            const bool mine = more && row == low;
            if (more && m < M) {
                mat[m * kRowLd + l8] = mine ? val : 0.0;
                if (l8 == 0)
                    rowid[m] = low;
            }
            m += more ? 1 : 0;
            if (mine) {
                e++;
                row = next_row;
                val = next_val;
                next_row = e + 1 < e1 ? __ldg(pb.cidx + e + 1) : 0x7fffffff;
                next_val = e + 1 < e1 ? __ldg(pb.cval + e + 1) : 0.0;
            }
        }
        const bool fits = m <= M;
        if (!fits && l8 == 0)
            rest[atomicAdd(rest_count, 1)] = col;
        const bool live = col >= 0 && fits;
        __syncwarp();
        // ---- this lane's rows and the target
        double a[R][8], b[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const bool has = live && l8 + 8 * r < m;
            b[r] = 0.0;
#pragma unroll
            for (int c = 0; c < 8; c++)
                a[r][c] = has ? mat[(l8 + 8 * r) * kRowLd + c] : 0.0;
        }
        if (live) {
            if (pb.bptr == nullptr) {
#pragma unroll
                for (int r = 0; r < R; r++)
                    if (l8 + 8 * r < m && rowid[l8 + 8 * r] == col)
                        b[r] = 1.0;
            }
            else {
                for (int64_t q = pb.bptr[col]; q < pb.bptr[col + 1]; q++) {
                    const int br = pb.bidx[q];
#pragma unroll
                    for (int r = 0; r < R; r++)
                        if (l8 + 8 * r < m && rowid[l8 + 8 * r] == br)
                            b[r] = pb.bval[q];
                }
            }
        }
        double rhs[R];
#pragma unroll
        for (int r = 0; r < R; r++)
            rhs[r] = b[r];
        const int nmax = __reduce_max_sync(kAll, n), mmax = __reduce_max_sync(kAll, min(m, M));
        // ---- Householder QR, the reflectors unscaled: v = scale x
        double rinv = 0.0;  // lane k: 1 / R(k, k)
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k >= nmax)
                break;
            double x2 = l8 > k ? a[0][k] * a[0][k] : 0.0;
#pragma unroll
            for (int r = 1; r < R; r++)
                if (8 * r < mmax)
                    x2 += a[r][k] * a[r][k];
            x2 = group_sum(x2);
            const double alpha = __shfl_sync(kAll, a[0][k], k, 8);
            double beta = alpha, tau = 0.0, scale = 0.0, ib;
            if (x2 != 0.0) {
                beta = -copysign(sqrt(alpha * alpha + x2), alpha);
                scale = 1.0 / (alpha - beta);
                ib = 1.0 / beta;
                tau = (beta - alpha) * ib;
            }
            else {
                ib = 1.0 / alpha;
            }
            if (k < n && l8 == k)
                rinv = ib;
            // v^T of the later columns and of the right-hand side
            double d[9];
#pragma unroll
            for (int c = 0; c < 9; c++) {
                d[c] = 0.0;
                if (c > k && (c == 8 || c < nmax)) {
                    d[c] = l8 > k ? a[0][k] * (c < 8 ? a[0][c % 8] : b[0]) : 0.0;
#pragma unroll
                    for (int r = 1; r < R; r++)
                        if (8 * r < mmax)
                            d[c] += a[r][k] * (c < 8 ? a[r][c % 8] : b[r]);
                    d[c] = scale * group_sum(d[c]);
                    d[c] = tau * (d[c] + __shfl_sync(kAll, c < 8 ? a[0][c % 8] : b[0], k, 8));
                }
            }
#pragma unroll
            for (int c = 0; c < 9; c++) {
                if (c > k && (c == 8 || c < nmax)) {
                    const double f0 = l8 > k ? d[c] * scale * a[0][k] : (l8 == k ? d[c] : 0.0);
                    if (c < 8)
                        a[0][c % 8] -= f0;
                    else
                        b[0] -= f0;
#pragma unroll
                    for (int r = 1; r < R; r++) {
                        if (8 * r < mmax) {
                            if (c < 8)
                                a[r][c % 8] -= d[c] * scale * a[r][k];
                            else
                                b[r] -= d[c] * scale * a[r][k];
                        }
                    }
                }
            }
        }
        // ---- back substitution; x is not finite when R has a zero on its diagonal
        double x = b[0];
        double xs[8];
#pragma unroll
        for (int k = 7; k >= 0; k--) {
            xs[k] = 0.0;
            if (k >= nmax)
                continue;
            if (l8 == k && k < n)
                x *= rinv;
            const double xk = __shfl_sync(kAll, x, k, 8);
            xs[k] = k < n ? xk : 0.0;
            if (l8 < k && k < n)
                x -= a[0][k] * xk;
        }
        // ---- FP64 residual from the matrix
        double r2 = 0.0;
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (live && l8 + 8 * r < m) {
                double v = rhs[r];
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (c < nmax)
                        v -= mat[(l8 + 8 * r) * kRowLd + c] * xs[c];
                r2 += v * v;
            }
        }
        r2 = group_sum(r2);
        const uint32_t odd = __ballot_sync(kAll, l8 < n && !isfinite(x));
        __syncwarp();
        const bool bad = ((odd >> (8 * grp)) & 0xffu) != 0 || !isfinite(r2);
        if (live && bad) {
            if (l8 == 0) {
                refused.list[atomicAdd(refused.count, 1)] = col;
                *refused_any = 1;
            }
        }
        else if (live) {
            if (l8 < n)
                out.oval[p0 + l8] = x;
            if (l8 == 0) {
                const double res = sqrt(r2);
                const double dn = n, dm = m;
                double* wk = out.work + 3 * static_cast<size_t>(col);
                const double w = 2.0 * dm * dn * dn - (2.0 / 3.0) * dn * dn * dn + 4.0 * dm * dn;
                wk[0] += w + 2.0 * entries;
                wk[1] += w + 2.0 * dm * dn;
                wk[2] += 12.0 * entries + 16.0 * dn + 8.0 * dm;
                out.olen[col] = n;
                out.res[col] = res;
                out.steps[col] = 1;
                out.status[col] = 0;
            }
        }
    }
}

template <int R>
cudaError_t launch_small_t(const Problem& pb, const Output& out, const int32_t* list,
                           const int32_t* count_dev, int count_host, int32_t* rest,
                           int32_t* rest_count, const WorkList& refused, int32_t* refused_any,
                           cudaStream_t st)
{
    auto kern = small_qr_kernel<R>;
    const int bytes = (kSmallThreads / 8) * 8 * R *
                      (kRowLd * static_cast<int>(sizeof(double)) + static_cast<int>(sizeof(int32_t)));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSmallThreads, bytes);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    const int per_cta = kSmallThreads / 8;
    const int grid = std::max(1, std::min(per_sm * num_sms(), (count_host + per_cta - 1) / per_cta));
    kern<<<grid, kSmallThreads, bytes, st>>>(pb, out, list, count_dev, count_host, rest,
                                             rest_count, refused, refused_any);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_small_qr(const Problem& pb, const Output& out, const int32_t* list, int count,
                            int32_t* rest, int32_t* rest_count, const WorkList& refused,
                            int32_t* refused_any, cudaStream_t st)
{
    cudaError_t e = launch_small_t<4>(pb, out, list, nullptr, count, rest, rest_count, refused,
                                      refused_any, st);
    if (e != cudaSuccess)
        return e;
    // the columns of 33 to 64 rows (at most 64 entries: none is left)
    return launch_small_t<8>(pb, out, rest, rest_count, count, rest, rest_count + 1, refused,
                             refused_any, st);
}

}  // namespace mspai
