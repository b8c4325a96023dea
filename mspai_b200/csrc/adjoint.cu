// Adjoint of the setup (no reference counterpart).
//
// For problem column k (a scalar column, or a block column of bs scalar
// columns sharing J_k) with C_k = C(I_k, J_k), the right-hand sides b_k,c =
// B(I_k, bs k + c), the solutions m_k,c of the setup (read from its result M)
// and r_k,c = b_k,c - C_k m_k,c, the loss
//     L = w ||C M - B||_F^2 + sum_k gbar_k^T m_k      (gbar: scalar columns)
// has, at the pattern the setup chose (fixed, or the final pattern of the
// updates: the pattern is a discrete choice and carries no gradient):
//     dL/dC_k  = sum_c -2w r_k,c m_k,c^T  +  r_k lambda_k^T - (C_k lambda_k) m_k^T
//     dL/db_k,c = 2w r_k,c  +  C_k lambda_k
//     lambda_k = (C_k^T C_k)^-1 gbar_k = R_k^-1 R_k^-T gbar_k
// (envelope theorem for the squared residual -- M is stationary, so no
// re-solve is needed for it -- and the least-squares sensitivity for gbar),
// plus dL/dB(i, .) = 2w B(i, .) for target entries outside I_k.  lambda_k comes
// from two triangular solves with the R the setup kept (keep_factors), refined
// in FP64 against C_k^T C_k from the sparse entries when R is FP32; without a
// kept R the folded Householder QR is recomputed here in FP64.  Q is never
// formed or stored.  Every column adds its part to the nonzeros of C(:, J_k)
// with FP64 atomics.
#include "mspai_b200.h"
#include "spai_kernels.h"
#include "spai_solve.cuh"

#include <algorithm>
#include <vector>

namespace mspai {

// FP64 q = C(I, J) v on I (the sorted entries' runs), in q[0 .. m).
template <class G>
__device__ void adj_apply_c(const G& g, const Slot<double>& s, int m, const double* v, double* q)
{
    for (int u = g.rank(); u < m; u += G::kSize) {
        double acc = 0.0;
        for (int i = s.rstart[u]; i < s.rstart[u + 1]; i++) {
            const int e = static_cast<int>(s.keys[i] & kEntryMask);
            acc += s.ev[e] * v[s.ejj[e]];
        }
        q[u] = acc;
    }
    g.sync();
}

// lambda (in gv) = (C^T C)^-1 gbar with the kept R (packed by columns, TR):
// two triangular solves, then FP64 refinement steps gv += R^-1 R^-T (gbar -
// C^T C gv) until the correction is below 2^-44 of lambda (R may be FP32, or
// of values before a re-setup).  q (m entries) and tmp (n) are scratch.
// Returns (group-uniformly) false when the corrections do not get there.
template <class TR, class G>
__device__ bool adj_lambda_kept(const G& g, const Slot<double>& s, const TR* R, int m, int n,
                                const double* gbar, double* gv, double* q, double* tmp)
{
    for (int jj = g.rank(); jj < n; jj += G::kSize)
        gv[jj] = gbar[jj];
    g.sync();
    const RView<TR> rv{R, 0};
    group_normal_correction_blocked<TR>(g, rv, n, gv);
    double d2_prev = 0.0;
    for (int it = 0; it < 24; it++) {
        adj_apply_c(g, s, m, gv, q);
        // tmp = gbar - C^T q, a warp per column over its entries
        for (int jj = g.warp(); jj < n; jj += G::kWarps) {
            double acc = 0.0;
            for (int e = s.off[jj] + g.lane(); e < s.off[jj + 1]; e += 32)
                acc += s.ev[e] * q[s.pos[e]];
            acc = warp_sum(acc);
            if (g.lane() == 0)
                tmp[jj] = gbar[jj] - acc;
        }
        g.sync();
        group_normal_correction_blocked<TR>(g, rv, n, tmp);
        double d2 = 0.0, x2 = 0.0;
        for (int jj = g.rank(); jj < n; jj += G::kSize) {
            const double v = gv[jj] + tmp[jj];
            gv[jj] = v;
            d2 += tmp[jj] * tmp[jj];
            x2 += v * v;
        }
        d2 = g.sum(d2);
        x2 = g.sum(x2);
        g.sync();
        if (d2 <= 0x1p-88 * x2)
            return true;
        if (it > 0 && !(d2 <= 0.25 * d2_prev))
            return false;
        d2_prev = d2;
    }
    return false;
}

template <class TR, class G>
__device__ void adjoint_column(const G& g, const Problem& pb, const Caps& cap, Slot<double> s,
                               const AdjointIO& io, int kb)
{
    const int lane = g.lane();
    const int bs = pb.bs;
    const int sc0 = bs * kb;                 // first scalar column of the problem
    const int64_t p0 = io.mptr[sc0];
    const int n = static_cast<int>(io.mptr[sc0 + 1] - p0);
    if (n > cap.nmax || bs > cap.nrhs)
        return;
    // J and the solutions from the setup's result (the bs scalar columns of a
    // block column share J)
    for (int t = g.rank(); t < n; t += G::kSize) {
        const int j = io.midx[p0 + t];
        s.J[t] = j;
        s.off[t] = static_cast<int>(pb.cptr[j + 1] - pb.cptr[j]);
        for (int c = 0; c < bs; c++)
            s.x[static_cast<size_t>(c) * n + t] = io.mval[io.mptr[sc0 + c] + t];
    }
    g.sync();
    const int E = group_exclusive_scan(g, s.off, n);
    if (g.rank() == 0)
        s.off[n] = E;
    if (E > cap.emax)
        return;
    g.sync();
    for (int jj = g.warp(); jj < n; jj += G::kWarps) {
        const int j = s.J[jj];
        const int64_t base = pb.cptr[j];
        const int o = s.off[jj];
        const int len = s.off[jj + 1] - o;
        for (int t = lane; t < len; t += 32) {
            const int e = o + t;
            s.ejj[e] = jj;
            s.ev[e] = pb.cval[base + t];
            s.keys[e] = (static_cast<uint64_t>(pb.cidx[base + t]) << kEntryBits) |
                        static_cast<uint64_t>(e);
        }
    }
    const int L = next_pow2(E > 0 ? E : 1);
    for (int i = E + g.rank(); i < L; i += G::kSize)
        s.keys[i] = ~uint64_t(0);
    g.sync();
    group_bitonic_sort(g, s.keys, L);
    for (int i = g.rank(); i < E; i += G::kSize)
        s.tmp[i] = (i == 0 || (s.keys[i] >> kEntryBits) != (s.keys[i - 1] >> kEntryBits)) ? 1 : 0;
    g.sync();
    const int m = group_exclusive_scan(g, s.tmp, E);
    for (int i = g.rank(); i < E; i += G::kSize) {
        const bool first = (i == 0 || (s.keys[i] >> kEntryBits) != (s.keys[i - 1] >> kEntryBits));
        const int u = first ? s.tmp[i] : s.tmp[i] - 1;
        s.pos[static_cast<int>(s.keys[i] & kEntryMask)] = u;
        if (first) {
            s.I[u] = static_cast<int>(s.keys[i] >> kEntryBits);
            s.rstart[u] = i;
        }
    }
    if (g.rank() == 0)
        s.rstart[m] = E;
    g.sync();
    // r_c = b_c - C m_c on I (s.r + c m), ||r||_F^2
    const double r2 =
        group_residual(g, pb, kb, s.keys, s.I, s.rstart, s.ejj, s.ev, s.x, s.r, m, n, bs);
    g.sync();
    // lambda = R^-1 R^-T gbar_k (scalar columns with a gbar)
    double gx = 0.0;
    double* q = s.rho;     // C lambda on I (cmax >= emax doubles)
    const bool lam = io.gbar != nullptr && bs == 1;
    if (lam) {
        const double* gb = io.gbar + io.mptr[kb];
        for (int jj = g.rank(); jj < n; jj += G::kSize)
            gx += gb[jj] * s.x[jj];
        if (!io.rstore || !adj_lambda_kept<TR>(g, s, static_cast<const TR*>(io.rstore) + io.roff[kb],
                                               m, n, gb, s.gv, q, s.rinv)) {
            // recompute R: the folded Householder QR of the forward, in FP64
            for (int u = g.rank(); u < m; u += G::kSize)
                s.tmp[u] = (s.rstart[u + 1] - s.rstart[u]) >= 2 ? 1 : 0;
            g.sync();
            const int S = group_exclusive_scan(g, s.tmp, m);
            const int mw = S + n;
            if (mw > cap.mwmax)
                return;
            double* W = s.W;
            const int ld = mw;
            for (int i = g.rank(); i < mw * n; i += G::kSize)
                W[i] = 0.0;
            g.sync();
            for (int i = g.rank(); i < E; i += G::kSize) {
                const int e = static_cast<int>(s.keys[i] & kEntryMask);
                const int u = s.pos[e];
                if (s.rstart[u + 1] - s.rstart[u] >= 2)
                    W[static_cast<size_t>(s.ejj[e]) * ld + s.tmp[u]] = s.ev[e];
            }
            for (int jj = g.warp(); jj < n; jj += G::kWarps) {
                double sig = 0.0;
                for (int e = s.off[jj] + lane; e < s.off[jj + 1]; e += 32) {
                    const int u = s.pos[e];
                    if (s.rstart[u + 1] - s.rstart[u] == 1)
                        sig += s.ev[e] * s.ev[e];
                }
                sig = warp_sum(sig);
                if (lane == 0)
                    W[static_cast<size_t>(jj) * ld + S + jj] = sqrt(sig);
            }
            g.sync();
            group_householder<double>(g, W, ld, mw, n, 0);
            for (int jj = g.rank(); jj < n; jj += G::kSize)
                s.gv[jj] = gb[jj];
            g.sync();
            group_normal_correction<double>(g, W, ld, n, s.gv);
        }
        adj_apply_c(g, s, m, s.gv, q);
    }
    gx = g.sum(gx);
    // dL/dC at the nonzeros of C(:, J_k)
    for (int jj = g.warp(); jj < n; jj += G::kWarps) {
        const int j = s.J[jj];
        const int64_t base = pb.cptr[j];
        const int o = s.off[jj];
        const int len = s.off[jj + 1] - o;
        const double lj = lam ? s.gv[jj] : 0.0;
        for (int t = lane; t < len; t += 32) {
            const int u = s.pos[o + t];
            double gval = 0.0;
            for (int c = 0; c < bs; c++)
                gval -= s.r[static_cast<size_t>(c) * m + u] * s.x[static_cast<size_t>(c) * n + jj];
            gval *= 2.0 * io.wres;
            if (lam)
                gval += s.r[u] * lj - q[u] * s.x[jj];
            atomicAdd(&io.dC[base + t], gval);
        }
    }
    // dL/dB at the target entries, and the loss of the target outside I_k
    double outside = 0.0;
    for (int c = 0; c < bs; c++) {
        const int col = sc0 + c;
        if (pb.bptr) {
            const int64_t b0 = pb.bptr[col], b1 = pb.bptr[col + 1];
            for (int64_t p = b0 + g.rank(); p < b1; p += G::kSize) {
                const int row = pb.bidx[p];
                const int u = lower_bound_i32(s.I, m, row);
                double gbv;
                if (u < m && s.I[u] == row) {
                    gbv = 2.0 * io.wres * s.r[static_cast<size_t>(c) * m + u] +
                          (lam ? q[u] : 0.0);
                }
                else {
                    gbv = 2.0 * io.wres * pb.bval[p];
                    outside += pb.bval[p] * pb.bval[p];
                }
                if (io.dB)
                    io.dB[p] = gbv;
            }
        }
        else if (g.rank() == 0) {
            const int u = lower_bound_i32(s.I, m, col);
            if (!(u < m && s.I[u] == col))
                outside += 1.0;  // e_col has its 1 outside I_k
        }
    }
    outside = g.sum(outside);
    if (g.rank() == 0)
        io.loss[kb] = io.wres * (r2 + outside) + gx;
    g.sync();
}

// E[k] = entries of C(:, J_k), nk[k] = |J_k| for problem column k, J_k the
// pattern of scalar column bs k of the result; eight lanes per column
__global__ void adjoint_plan_kernel(const int64_t* __restrict__ cptr,
                                    const int64_t* __restrict__ mptr,
                                    const int32_t* __restrict__ midx, int nprob, int bs,
                                    int32_t* __restrict__ E, int32_t* __restrict__ nk)
{
    const int lane = threadIdx.x & 7;
    const int groups = (gridDim.x * blockDim.x) >> 3;
    const int first = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    for (int64_t base = 0; base < nprob; base += groups) {  // every lane of a warp takes part
        const int64_t kb = base + first;
        int64_t a = 0, b = 0, e = 0;
        if (kb < nprob) {
            a = mptr[bs * kb];
            b = mptr[bs * kb + 1];
        }
        for (int64_t p = a + lane; p < b; p += 8) {
            const int j = midx[p];
            e += cptr[j + 1] - cptr[j];
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
            e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0 && kb < nprob) {
            E[kb] = static_cast<int32_t>(e > 0x7fffffff ? 0x7fffffff : e);
            nk[kb] = static_cast<int32_t>(b - a);
        }
    }
}

cudaError_t launch_adjoint_plan(const int64_t* cptr, const int64_t* mptr, const int32_t* midx,
                                int nprob, int bs, int32_t* E, int32_t* nk, cudaStream_t st)
{
    if (nprob <= 0)
        return cudaSuccess;
    const int blocks = std::max(1, std::min((nprob + 31) / 32, num_sms() * 8));
    adjoint_plan_kernel<<<blocks, 256, 0, st>>>(cptr, mptr, midx, nprob, bs, E, nk);
    return cudaGetLastError();
}

template <class TR, int NT>
__global__ void __launch_bounds__(NT)
    adjoint_cta_kernel(Problem pb, Caps cap, AdjointIO io, const int32_t* __restrict__ list,
                       int count, char* scratch, size_t slot_bytes, int32_t* counter)
{
    __shared__ GroupScratch sc;
    CtaGroup<NT> g{&sc};
    SlotLayout<double> lay(cap, false);
    Slot<double> s = lay.at(scratch + static_cast<size_t>(blockIdx.x) * slot_bytes, nullptr);
    while (true) {
        if (threadIdx.x == 0)
            sc.i[5] = atomicAdd(counter, 1);
        __syncthreads();
        const int t = sc.i[5];
        __syncthreads();
        if (t >= count)
            break;
        adjoint_column<TR>(g, pb, cap, s, io, list[t]);
    }
}

template <class TR>
__global__ void __launch_bounds__(kWarpKernelThreads)
    adjoint_warp_kernel(Problem pb, Caps cap, AdjointIO io, const int32_t* __restrict__ list,
                        int count, char* scratch, size_t slot_bytes, int32_t* counter)
{
    __shared__ GroupScratch sc[kWarpKernelThreads / 32];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    WarpGroup g{&sc[w]};
    SlotLayout<double> lay(cap, false);
    const size_t slot_id = static_cast<size_t>(blockIdx.x) * (kWarpKernelThreads / 32) + w;
    Slot<double> s = lay.at(scratch + slot_id * slot_bytes, nullptr);
    while (true) {
        int t = 0;
        if (lane == 0)
            t = atomicAdd(counter, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= count)
            break;
        adjoint_column<TR>(g, pb, cap, s, io, list[t]);
    }
}

template <class TR>
static void launch_adjoint_t(const Problem& pb, const Caps& cap, const AdjointIO& io,
                             const int32_t* list, int n, bool warp, char* scratch,
                             size_t scratch_bytes, int32_t* counter, cudaStream_t st)
{
    const size_t slot = SlotLayout<double>(cap, false).bytes;
    const int sms = num_sms();
    if (warp) {
        const int per_block = kWarpKernelThreads / 32;
        int grid = std::min<int>(sms * 8, (n + per_block - 1) / per_block);
        grid = std::max(1, std::min<int>(grid, static_cast<int>(scratch_bytes / (slot * per_block))));
        adjoint_warp_kernel<TR><<<grid, kWarpKernelThreads, 0, st>>>(pb, cap, io, list, n, scratch,
                                                                     slot, counter);
    }
    else {
        int grid = std::min(sms * 4, n);
        grid = std::max(1, std::min<int>(grid, static_cast<int>(scratch_bytes / slot)));
        adjoint_cta_kernel<TR, 128><<<grid, 128, 0, st>>>(pb, cap, io, list, n, scratch, slot,
                                                          counter);
    }
}

cudaError_t launch_adjoint(const Problem& pb, const Caps& cap, const AdjointIO& io,
                           const int32_t* list, int count, bool warp, char* scratch,
                           size_t scratch_bytes, int32_t* counter, cudaStream_t st)
{
    if (io.rstore && io.r_elem == 4)
        launch_adjoint_t<float>(pb, cap, io, list, count, warp, scratch, scratch_bytes, counter,
                                st);
    else
        launch_adjoint_t<double>(pb, cap, io, list, count, warp, scratch, scratch_bytes, counter,
                                 st);
    return cudaGetLastError();
}

// Scalar columns of at most eight unknowns without a gbar, eight lanes per
// column, four columns per warp.  Lane j walks the sorted entries of C(:, J(j));
// the smallest head of the eight lanes is the next row of I_k, its residual is
// the target's value there less the sum of the lanes' products, and the lanes
// with an entry in the row add -2 w r x_j to dC.  Nothing is stored or sorted.
// Bound: the FP64 atomics on dC and the latency of the reads of C (1,048,576
// columns of 35 entries: 6.8 ms in the warp kernel above, 0.54 ms here).
__global__ void __launch_bounds__(256)
    adjoint_small_kernel(Problem pb, AdjointIO io, const int32_t* __restrict__ list, int count)
{
    constexpr uint32_t all = 0xffffffffu;
    const int lane = threadIdx.x & 31, grp = lane >> 3, l8 = lane & 7;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int64_t t0 = 4 * static_cast<int64_t>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
         t0 < count; t0 += 4 * static_cast<int64_t>(warps)) {
        const int col = t0 + grp < count ? list[t0 + grp] : -1;
        int64_t e = 0, e1 = 0, q = 0, q1 = 0;
        double x = 0.0;
        if (col >= 0) {
            const int64_t p0 = io.mptr[col];
            const int n = static_cast<int>(io.mptr[col + 1] - p0);
            if (l8 < n) {
                const int j = io.midx[p0 + l8];
                x = io.mval[p0 + l8];
                e = pb.cptr[j];
                e1 = pb.cptr[j + 1];
            }
            if (pb.bptr) {
                q = pb.bptr[col];
                q1 = pb.bptr[col + 1];
            }
        }
        int row = e < e1 ? __ldg(pb.cidx + e) : 0x7fffffff;
        double val = e < e1 ? __ldg(pb.cval + e) : 0.0;
        int brow = q < q1 ? __ldg(pb.bidx + q) : 0x7fffffff;
        double loss = 0.0;
        bool seen = pb.bptr != nullptr || col < 0;  // identity target: e_col met in I_k
        // target entries in rows outside I_k, up to row `below`
        auto outside = [&](int below) {
            while (brow < below) {
                const double b = pb.bval[q];
                loss += b * b;
                if (io.dB && l8 == 0)
                    io.dB[q] = 2.0 * io.wres * b;
                q++;
                brow = q < q1 ? __ldg(pb.bidx + q) : 0x7fffffff;
            }
        };
        while (true) {
            int low = min(row, __shfl_xor_sync(all, row, 4));
            low = min(low, __shfl_xor_sync(all, low, 2));
            low = min(low, __shfl_xor_sync(all, low, 1));
            const bool more = low != 0x7fffffff;
            if (!__any_sync(all, more))
                break;
            const bool mine = more && row == low;
            double s = mine ? val * x : 0.0;
            s += __shfl_xor_sync(all, s, 4);
            s += __shfl_xor_sync(all, s, 2);
            s += __shfl_xor_sync(all, s, 1);
            if (!more)
                continue;
            double b = 0.0;
            outside(low);
            const bool hit = brow == low;
            if (hit)
                b = pb.bval[q];
            else if (pb.bptr == nullptr && low == col) {
                b = 1.0;
                seen = true;
            }
            const double r = b - s;
            loss += r * r;
            if (hit) {
                if (io.dB && l8 == 0)
                    io.dB[q] = 2.0 * io.wres * r;
                q++;
                brow = q < q1 ? __ldg(pb.bidx + q) : 0x7fffffff;
            }
            if (mine) {
                atomicAdd(&io.dC[e], -(r * x) * (2.0 * io.wres));
                e++;
                row = e < e1 ? __ldg(pb.cidx + e) : 0x7fffffff;
                val = e < e1 ? __ldg(pb.cval + e) : 0.0;
            }
        }
        outside(0x7fffffff);
        if (!seen)
            loss += 1.0;  // e_col has its 1 outside I_k
        if (l8 == 0 && col >= 0)
            io.loss[col] = io.wres * loss;
        __syncwarp();
    }
}

cudaError_t launch_adjoint_small(const Problem& pb, const AdjointIO& io, const int32_t* list,
                                 int count, cudaStream_t st)
{
    if (count <= 0)
        return cudaSuccess;
    const int blocks = std::max(1, std::min((count + 31) / 32, num_sms() * 8));
    adjoint_small_kernel<<<blocks, 256, 0, st>>>(pb, io, list, count);
    return cudaGetLastError();
}

// s + c += v, exactly up to the last bits of c (Neumaier).
__device__ __forceinline__ void add_compensated(double& s, double& c, double v)
{
    const double t = s + v;
    c += fabs(s) >= fabs(v) ? (s - t) + v : (v - t) + s;
    s = t;
}

// The columns' losses are often nearly equal and a plain sum of a million lets
// their rounding errors add up: every thread sums its share with compensation,
// and the pairs are combined in a fixed order.  (On the host this took 3 ms a
// call for 1,048,576 columns, the copy included.)
__global__ void __launch_bounds__(256)
    loss_parts_kernel(const double* __restrict__ v, int n, double* __restrict__ parts)
{
    __shared__ double ss[256], sc[256];
    double s = 0.0, c = 0.0;
    for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += 256 * static_cast<int64_t>(gridDim.x))
        add_compensated(s, c, v[i]);
    ss[threadIdx.x] = s;
    sc[threadIdx.x] = c;
    for (int o = 128; o > 0; o >>= 1) {
        __syncthreads();
        if (threadIdx.x < o) {
            double a = ss[threadIdx.x], b = sc[threadIdx.x];
            add_compensated(a, b, ss[threadIdx.x + o]);
            b += sc[threadIdx.x + o];
            ss[threadIdx.x] = a;
            sc[threadIdx.x] = b;
        }
    }
    if (threadIdx.x == 0) {
        parts[2 * blockIdx.x] = ss[0];
        parts[2 * blockIdx.x + 1] = sc[0];
    }
}

__global__ void loss_total_kernel(const double* __restrict__ parts, int n, double* __restrict__ total)
{
    __shared__ double ss[kLossParts], sc[kLossParts];
    for (int i = threadIdx.x; i < kLossParts; i += blockDim.x) {
        ss[i] = i < n ? parts[2 * i] : 0.0;
        sc[i] = i < n ? parts[2 * i + 1] : 0.0;
    }
    for (int o = kLossParts / 2; o > 0; o >>= 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < o; i += blockDim.x) {
            double a = ss[i], b = sc[i];
            add_compensated(a, b, ss[i + o]);
            b += sc[i + o];
            ss[i] = a;
            sc[i] = b;
        }
    }
    if (threadIdx.x == 0)
        *total = ss[0] + sc[0];
}

cudaError_t launch_loss_sum(const double* v, int n, double* tmp, double* total, cudaStream_t st)
{
    const int blocks = std::max(1, std::min((n + 1023) / 1024, kLossParts));
    loss_parts_kernel<<<blocks, 256, 0, st>>>(v, n, tmp);
    loss_total_kernel<<<1, 256, 0, st>>>(tmp, blocks, total);
    return cudaGetLastError();
}

size_t adjoint_scratch_bytes(const Caps& cap, int n, bool warp)
{
    const size_t slot = SlotLayout<double>(cap, false).bytes;
    const int sms = num_sms();
    const size_t slots = warp ? static_cast<size_t>(std::min(sms * 8, (n + 7) / 8)) * 8
                              : static_cast<size_t>(std::min(sms * 4, n));
    return slot * std::max<size_t>(slots, 1);
}

}  // namespace mspai
