// Block columns (bs > 1) at their start pattern: Cholesky of C^T C and FP64
// refinement, one CTA per block column, everything in shared memory.
//
// The general solver folds C(I, J) into a dense matrix in global memory and
// factors it by Householder reflections (the reference's
// Spai_Unrestrained_Block, src/Spai_Unrestrained_Block.imp:33-205).  A 27-point
// block column has 81 unknowns and 375 rows of 18 entries: the normal matrix
// from the sparse entries costs a fifth of the reflections' flops and fits in
// shared memory with the factor.
//
//  1. The rows of C(:, J) are numbered in the order of their first entry with a
//     hash table; the entries are listed by row as well (column after column, so
//     the order is fixed).
//  2. G = C^T C, four columns at a time: they are scattered into a dense array
//     over the rows, and four lanes per earlier column sum its products with all
//     four (one 16-byte load of the array per entry).
//  3. Blocked Cholesky and the FP64 refinement x += R^-1 R^-T C^T (b - C x) from
//     x = 0 of fixed_solve.cuh, for the bs right-hand sides, with its tests; FP64
//     mode, which has no refinement, keeps the result only when the first
//     correction is already below 2^-44 of the solution.
// A column that does not fit goes to the next launch (more shared memory); one that
// does not converge or (pattern updates) whose residual is above the tolerance would
// be refused there as well and goes to the general solver at once.  The row structure
// that the updates need is only built when a column is left.
//   Bound: latency of the blocked Cholesky and of the triangular solves at two
//   CTAs of 256 threads per SM (mixed), one (FP64).  8,000 block columns of a
//   20^3 27-point stencil with 3 x 3 blocks: 36.9 ms in the general solver, 12.7 ms
//   here with a walk over C's values per right-hand side, 6.8 ms with one for all;
//   64,000 of the block diagonal (3 unknowns, 246 entries, eight lanes each; CTAs of
//   64 threads took 2.7): 3.6 ms there, 1.7 ms here.
#include "fixed_solve.cuh"
#include "spai_kernels.h"

#include <algorithm>

namespace mspai {

namespace {

__device__ __forceinline__ void load4(const float* p, float (&v)[4])
{
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
}
__device__ __forceinline__ void load4(const double* p, double (&v)[4])
{
    const double2 a = reinterpret_cast<const double2*>(p)[0];
    const double2 b = reinterpret_cast<const double2*>(p)[1];
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}

// What becomes of a block column.
enum class Fit {
    kYes,     // solved
    kLarger,  // it does not fit the arena
    kNo       // left to the general solver
};

// Solves block column kb (uniformly); nothing is written unless it is taken.
template <class T, int NT>
__device__ Fit block_column(const CtaGroup<NT>& g, FixShared<T>& fs, const Problem& pb,
                             const Output& out, int kb, char* base, int cap)
{
    const int tid = threadIdx.x, lane = tid & 31;
    const int bs = pb.bs;
    const int64_t p0 = pb.pptr[kb];
    const int n = bs * static_cast<int>(pb.pptr[kb + 1] - p0);
    if (n < 1 || n > 255)
        return Fit::kNo;
    auto scol = [&](int jj) { return bs * pb.pidx[p0 + jj / bs] + jj % bs; };
    FixArena a{base, cap, 0, cap};
    int32_t* off = a.low<int32_t>(n + 1);
    uint32_t* cb = a.low<uint32_t>(n);
    double* x = a.low<double>(n * bs);
    T* gv = a.low<T>(n * bs);
    if (!a.ok())
        return Fit::kLarger;
    for (int jj = tid; jj < n; jj += NT) {
        const int j = scol(jj);
        cb[jj] = static_cast<uint32_t>(pb.cptr[j]);
        off[jj] = static_cast<int>(pb.cptr[j + 1] - pb.cptr[j]);
    }
    g.sync();
    const int E = group_exclusive_scan(g, off, n);
    if (tid == 0) {
        off[n] = E;
        fs.chol_fail = 0;
        fs.mcount = 0;
    }
    if (E < 1 || E > 0xffff)
        return Fit::kNo;
    uint16_t* R = a.low<uint16_t>(E);  // row number of entry e
    // ---- rows: a hash table of 1.25 times the rows that the arena can hold (what
    // every entry and every row takes below), or of 1.5 E slots.  A column with more
    // rows than that ends here: its insertion stops at the first row too many, so
    // that at most one more a thread is inserted and a probe meets a free slot.
    const int room = cap - a.lo - E * (5 + static_cast<int>(sizeof(T))) -
                     fix_rs(n, n) * static_cast<int>(sizeof(T));
    const int most_rows = min(E, room / (8 + 8 * bs + 4 * static_cast<int>(sizeof(T))));
    if (most_rows < 1)
        return Fit::kLarger;
    const int hs = next_pow2(max(
        64, most_rows < E ? min(E + E / 2, most_rows + most_rows / 4 + NT) : E + E / 2));
    const int hbits = 31 - __clz(hs);
    int32_t* key = a.high<int32_t>(hs);
    int32_t* first = a.high<int32_t>(hs);
    int32_t* flag = a.high<int32_t>(E);
    if (!a.ok() || hs > 0x10000)
        return Fit::kLarger;
    g.sync();
    for (int i = tid; i < hs; i += NT) {
        key[i] = -1;
        first[i] = 0x7fffffff;
    }
    g.sync();
    const volatile int* rows = &fs.mcount;
    for (int jj = tid / 8; jj < n; jj += NT / 8) {
        const int o = off[jj], len = off[jj + 1] - o;
        for (int q = tid & 7; q < len && *rows <= most_rows; q += 8) {
            const int row = __ldg(pb.cidx + cb[jj] + q);
            uint32_t s = (static_cast<uint32_t>(row) * 2654435761u) >> (32 - hbits);
            int old = atomicCAS(&key[s], -1, row);
            while (old != -1 && old != row) {
                s = (s + 1) & (hs - 1);
                old = atomicCAS(&key[s], -1, row);
            }
            if (old == -1)
                atomicAdd(&fs.mcount, 1);
            atomicMin(&first[s], o + q);
            R[o + q] = static_cast<uint16_t>(s);
        }
    }
    g.sync();
    if (fs.mcount > most_rows)
        return Fit::kLarger;
    for (int e = tid; e < E; e += NT)
        flag[e] = first[R[e]] == e ? 1 : 0;
    g.sync();
    const int m = group_exclusive_scan(g, flag, E);
    uint16_t* by = a.low<uint16_t>(E);     // entries by row ...
    uint8_t* bj = a.low<uint8_t>(E);       // ... and their columns
    int32_t* I = a.low<int32_t>(m);        // rows
    int32_t* rs = a.low<int32_t>(m + 1);   // starts of the rows' entries
    double* r = a.low<double>(m * bs);     // residual
    if (!a.ok())
        return Fit::kLarger;
    // (a first entry's slot is overwritten by its own thread only after every
    // flag is made: the scan's barriers lie in between)
    for (int e = tid; e < E; e += NT) {
        const int next = e + 1 < E ? flag[e + 1] : m;
        if (next > flag[e]) {
            I[flag[e]] = key[R[e]];
            first[R[e]] = flag[e];
        }
    }
    for (int i = tid; i <= m; i += NT)
        rs[i] = 0;
    g.sync();
    for (int e = tid; e < E; e += NT) {
        const int row = first[R[e]];
        R[e] = static_cast<uint16_t>(row);
        atomicAdd(&rs[row], 1);
    }
    g.sync();
    group_exclusive_scan(g, rs, m);
    if (tid == 0)
        rs[m] = E;
    int32_t* fill = flag;  // next place of each row
    g.sync();
    for (int i = tid; i < m; i += NT)
        fill[i] = rs[i];
    g.sync();
    for (int jj = 0; jj < n; jj++) {  // a column has a row at most once
        for (int e = off[jj] + tid; e < off[jj + 1]; e += NT) {
            const int q = fill[R[e]]++;
            by[q] = static_cast<uint16_t>(e);
            bj[q] = static_cast<uint8_t>(jj);
        }
        g.sync();
    }
    // ---- G = C^T C, upper triangle packed by rows (fix_rs)
    a.hi = cap;  // the table is dead
    const int r_el = fix_rs(n, n);
    const int nblk = (n + kFixPanel - 1) / kFixPanel;
    T* V = a.low<T>(E);
    T* G = a.low<T>(r_el);
    T* r11 = a.low<T>(kFixPanel * kFixPanel);
    // four columns over the rows; the Cholesky's tile, then the inverted
    // diagonal blocks take its place
    T* d = a.low<T>(max(4 * m, max(kFixPanel * n, kFixPanel * kFixPanel * nblk)));
    T* tile = d;
    if (!a.ok())
        return Fit::kLarger;
    for (int jj = tid / 8; jj < n; jj += NT / 8)
        for (int e = off[jj] + (tid & 7); e < off[jj + 1]; e += 8)
            V[e] = static_cast<T>(__ldg(pb.cval + cb[jj] + (e - off[jj])));
    // FP64 value of entry e of column jj: FP32 copies serve G alone
    auto value = [&](int e, int jj) -> double {
        if constexpr (sizeof(T) == 8)
            return V[e];
        else
            return __ldg(pb.cval + cb[jj] + (e - off[jj]));
    };
    for (int i = tid; i < r_el; i += NT)
        G[i] = T(0);
    for (int i = tid; i < 4 * m; i += NT)
        d[i] = T(0);
    g.sync();
    for (int j0 = 0; j0 < n; j0 += 4) {
        const int j1 = min(n, j0 + 4);
        for (int e = off[j0] + tid; e < off[j1]; e += NT) {
            int c = 0;
            while (c < 3 && j0 + c + 1 < j1 && e >= off[j0 + c + 1])
                c++;
            d[4 * R[e] + c] = V[e];
        }
        g.sync();
        // four lanes per column i (warp-uniform trips: shuffles)
        for (int i0 = 0; i0 < j1; i0 += NT / 4) {
            const int i = i0 + tid / 4, q = tid & 3;
            T acc[4] = {T(0), T(0), T(0), T(0)};
            if (i < j1) {
                for (int e = off[i] + q; e < off[i + 1]; e += 4) {
                    T w[4];
                    load4(d + 4 * R[e], w);
                    const T v = V[e];
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        acc[c] += v * w[c];
                }
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
                acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
            }
            const T mine = q == 0 ? acc[0] : (q == 1 ? acc[1] : (q == 2 ? acc[2] : acc[3]));
            if (i < j1 && j0 + q < j1 && i <= j0 + q)
                G[fix_rs(i, n) + (j0 + q - i)] = mine;
        }
        g.sync();
        for (int e = off[j0] + tid; e < off[j1]; e += NT) {
            T* p = d + 4 * R[e];
            p[0] = p[1] = p[2] = p[3] = T(0);
        }
        g.sync();
    }
    if (!fix_cholesky<T, NT>(g, fs, G, n, tile, r11))
        return Fit::kNo;
    T* D = tile;
    fix_invert_diag<T, NT>(G, n, D);
    for (int i = tid; i < n * bs; i += NT)
        x[i] = 0.0;
    g.sync();
    // ---- r = b - C x per right-hand side, its squared norm; with grad C^T r
    auto residual = [&](bool grad) -> double {
        double part = 0.0;
        // all right-hand sides of a row by one thread: its values are read once
        for (int u = tid; u < m; u += NT) {
            double v[kMaxBlockSize];
#pragma unroll
            for (int c = 0; c < kMaxBlockSize; c++)
                v[c] = c < bs ? target_value(pb, bs * kb + c, I[u]) : 0.0;
            const int q1 = rs[u + 1];
#pragma unroll 4
            for (int q = rs[u]; q < q1; q++) {
                const int jj = bj[q];
                const double a = value(by[q], jj);
#pragma unroll
                for (int c = 0; c < kMaxBlockSize; c++)
                    if (c < bs)
                        v[c] -= a * x[c * n + jj];
            }
#pragma unroll
            for (int c = 0; c < kMaxBlockSize; c++)
                if (c < bs) {
                    r[c * m + u] = v[c];
                    part += v[c] * v[c];
                }
        }
        const double r2 = g.sum(part);  // includes a barrier: r is complete
        if (grad) {
            // eight lanes per column (warp-uniform trips)
            for (int j0 = 0; j0 < n; j0 += NT / 8) {
                const int jj = j0 + tid / 8, q = tid & 7;
                double acc[kMaxBlockSize];
#pragma unroll
                for (int c = 0; c < kMaxBlockSize; c++)
                    acc[c] = 0.0;
                if (jj < n) {
                    const int e1 = off[jj + 1];
#pragma unroll 4
                    for (int e = off[jj] + q; e < e1; e += 8) {
                        const double a = value(e, jj);
                        const double* re = r + R[e];
#pragma unroll
                        for (int c = 0; c < kMaxBlockSize; c++)
                            if (c < bs)
                                acc[c] += a * re[c * m];
                    }
                }
#pragma unroll
                for (int c = 0; c < kMaxBlockSize; c++) {
                    if (c >= bs)
                        break;
                    acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 4);
                    acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 2);
                    acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 1);
                    if (jj < n && q == 0)
                        gv[c * n + jj] = static_cast<T>(acc[c]);
                }
            }
            g.sync();
        }
        return r2;
    };
    const int most = pb.refine > 0 ? pb.refine + 2 : 3;
    bool conv = false;
    double d2_prev = 0.0;
    int steps = 0;
    double r2 = residual(true);
    for (int it = 0; it < most; it++) {
        steps++;
        for (int c = 0; c < bs; c++) {
            fix_forward_inv<T, NT>(g, G, D, n, gv + c * n);
            fix_back_inv<T, NT>(g, G, D, n, gv + c * n);
        }
        double d2 = 0.0, x2 = 0.0;
        for (int i = tid; i < n * bs; i += NT) {
            const double dl = static_cast<double>(gv[i]), x1 = x[i] + dl;
            d2 += dl * dl;
            x2 += x1 * x1;
            x[i] = x1;
        }
        d2 = g.sum(d2);
        x2 = g.sum(x2);
        conv = d2 <= 0x1p-88 * x2;
        const bool last = conv || it + 1 == most || (it > 0 && !(d2 <= 0.25 * d2_prev)) ||
                          (it == 1 && pb.refine == 0);
        d2_prev = d2;
        r2 = residual(!last);
        if (last)
            break;
    }
    const double res = sqrt(r2);
    if (!conv || (pb.ns > 0 && !(res <= pb.ep * sqrt(static_cast<double>(bs)))))
        return Fit::kNo;
    // ---- the bs scalar columns of M
    for (int c = 0; c < bs; c++) {
        const int sc = bs * kb + c;
        const int64_t o0 = out.optr[sc];
        int bad = 0;
        for (int t = tid; t < n; t += NT) {
            const double v = x[c * n + t];
            if (!isfinite(v))
                bad = 1;
            out.oval[o0 + t] = v;
            if (out.write_idx)
                out.oidx[o0 + t] = scol(t);
        }
        bad = g.sum(bad);
        if (tid == 0) {
            out.olen[sc] = n;
            out.res[sc] = res;
            out.steps[sc] = 1;
            out.status[sc] = (bad || !isfinite(res)) ? 2 : 0;
        }
    }
    if (tid == 0) {
        const double dn = n, dm = m, dr = bs;
        double* wk = out.work + 3 * static_cast<size_t>(kb);
        wk[0] += dn * E + dn * dn * dn / 3.0 + steps * dr * (2.0 * dn * dn + 4.0 * E);
        wk[1] += 2.0 * dm * dn * dn - (2.0 / 3.0) * dn * dn * dn + 4.0 * dm * dn * dr +
                 2.0 * dm * dn * dr;
        wk[2] += 12.0 * E + 16.0 * dn + 8.0 * dm * dr;
    }
    (void)lane;
    return Fit::kYes;
}

// Block columns of at most eight unknowns, FP64: eight lanes per column, four
// columns per warp.  Lane j walks the sorted entries of C(:, J)'s column j and
// lane c those of the target's column c; the smallest head is the next row.  The
// first walk sums G = C^T C (lane j: its row) and C^T b, each further one forms
// the residual row by row and C^T (b - C x) for the refinement, so that nothing
// is stored.
__device__ __forceinline__ double sum8(double v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

__global__ void __launch_bounds__(128)
    block_small_kernel(Problem pb, Output out, const int32_t* __restrict__ list, int count,
                       WorkList larger, WorkList left)
{
    constexpr uint32_t all = 0xffffffffu;
    const int lane = threadIdx.x & 31, grp = lane >> 3, l8 = lane & 7;
    const int bs = pb.bs;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int most = pb.refine > 0 ? pb.refine + 2 : 3;
    for (int64_t t0 = 4 * static_cast<int64_t>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
         t0 < count; t0 += 4 * static_cast<int64_t>(warps)) {
        const int kb = t0 + grp < count ? list[t0 + grp] : -1;
        int n = 0, col = 0;
        bool wide = false;  // more than eight unknowns
        int64_t a0 = 0, a1 = 0, q0 = 0, q1 = 0;
        if (kb >= 0) {
            const int64_t p0 = pb.pptr[kb];
            n = bs * static_cast<int>(pb.pptr[kb + 1] - p0);
            wide = n > 8;
            if (n > 8 || n < 1) {
                n = 0;
            }
            else if (l8 < n) {
                col = bs * pb.pidx[p0 + l8 / bs] + l8 % bs;
                a0 = pb.cptr[col];
                a1 = pb.cptr[col + 1];
            }
            if (pb.bptr && l8 < bs) {
                q0 = pb.bptr[bs * kb + l8];
                q1 = pb.bptr[bs * kb + l8 + 1];
            }
        }
        bool live = n > 0;  // still a candidate
        bool done = !live;  // converged, or left to the other kernels
        const int nmax = __reduce_max_sync(all, n);
        double G[8], lk[8], lt[8], linv = 0.0;
        double x[8], gr[8];  // per right-hand side: this lane's unknown
#pragma unroll
        for (int i = 0; i < 8; i++)
            G[i] = lk[i] = lt[i] = x[i] = gr[i] = 0.0;
        double r2 = 0.0, d2_prev = 0.0;
        int m = 0, solves = 0;
        for (int it = 0;; it++) {
            // ---- one walk over the rows
            int64_t e = a0, q = q0;
            int row = e < a1 ? __ldg(pb.cidx + e) : 0x7fffffff;
            double val = e < a1 ? __ldg(pb.cval + e) : 0.0;
            int brow = pb.bptr ? (q < q1 ? __ldg(pb.bidx + q) : 0x7fffffff)
                               : (kb >= 0 && l8 < bs ? bs * kb + l8 : 0x7fffffff);
            double part = 0.0;
#pragma unroll
            for (int c = 0; c < 8; c++)
                gr[c] = 0.0;
            while (true) {
                int low = min(row, __shfl_xor_sync(all, row, 4));
                low = min(low, __shfl_xor_sync(all, low, 2));
                low = min(low, __shfl_xor_sync(all, low, 1));
                const bool more = low != 0x7fffffff;
                if (!__any_sync(all, more))
                    break;
                const bool mine = more && row == low;
                const double v = mine ? val : 0.0;
                if (pb.bptr)
                    while (more && brow < low) {
                        q++;
                        brow = q < q1 ? __ldg(pb.bidx + q) : 0x7fffffff;
                    }
                const double b = (more && brow == low) ? (pb.bptr ? __ldg(pb.bval + q) : 1.0) : 0.0;
                if (it == 0) {
                    m += more ? 1 : 0;
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (i < nmax)
                            G[i] += v * __shfl_sync(all, v, i, 8);
                }
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    if (c < bs) {
                        double r = __shfl_sync(all, b, c, 8);
                        if (it > 0)
                            r -= sum8(v * x[c]);
                        gr[c] += v * r;
                        part += r * r;
                    }
                }
                if (mine) {
                    e++;
                    row = e < a1 ? __ldg(pb.cidx + e) : 0x7fffffff;
                    val = e < a1 ? __ldg(pb.cval + e) : 0.0;
                }
            }
            r2 = part;
            if (it == 0) {
                // ---- Cholesky, a lane per row: lk its row of L, lt its column
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    if (k >= nmax)
                        break;
                    const double piv = __shfl_sync(all, G[k], k, 8);
                    const bool in = k < n;
                    // (an infinite pivot would give x = 0 and pass for converged)
                    const bool pos = piv > 0.0 && isfinite(piv);
                    if (in && !pos)
                        done = true, live = false;
                    const double inv = in && pos ? 1.0 / sqrt(piv) : 0.0;
                    if (l8 == k)
                        linv = inv;
                    const double l = l8 > k ? G[k] * inv : 0.0;
                    lk[k] = l;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (i > k && i < nmax) {
                            const double li = __shfl_sync(all, l, i, 8);
                            G[i] -= l * li;
                            if (l8 == k)
                                lt[i] = li;
                        }
                    }
                }
            }
            // this walk only gave the residual of the converged columns
            if (__all_sync(all, done))
                break;
            // ---- x += G^-1 gr
            double d2 = 0.0, x2 = 0.0;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                if (c >= bs)
                    break;
                double z = gr[c];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    if (k >= nmax)
                        break;
                    if (l8 == k)
                        z *= linv;
                    const double zk = __shfl_sync(all, z, k, 8);
                    if (l8 > k)
                        z -= lk[k] * zk;
                }
#pragma unroll
                for (int k = 7; k >= 0; k--) {
                    if (k >= nmax)
                        continue;
                    if (l8 == k)
                        z *= linv;
                    const double zk = __shfl_sync(all, z, k, 8);
                    if (l8 < k)
                        z -= lt[k] * zk;
                }
                if (!done && l8 < n) {
                    x[c] += z;
                    d2 += z * z;
                    x2 += x[c] * x[c];
                }
            }
            d2 = sum8(d2);
            x2 = sum8(x2);
            if (!done) {
                solves++;
                if (d2 <= 0x1p-88 * x2) {
                    done = true;
                }
                else if (it + 1 == most || (it > 0 && !(d2 <= 0.25 * d2_prev)) ||
                         (it == 1 && pb.refine == 0)) {
                    done = true;
                    live = false;
                }
                d2_prev = d2;
            }
        }
        const double res = sqrt(r2);
        if (pb.ns > 0 && !(res <= pb.ep * sqrt(static_cast<double>(bs))))
            live = false;
        int entries = static_cast<int>(a1 - a0);
        entries += __shfl_xor_sync(all, entries, 4);
        entries += __shfl_xor_sync(all, entries, 2);
        entries += __shfl_xor_sync(all, entries, 1);
        if (wide && l8 == 0)
            larger.list[atomicAdd(larger.count, 1)] = kb;
        else if (kb >= 0 && !live && l8 == 0)
            left.list[atomicAdd(left.count, 1)] = kb;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            if (c >= bs)
                break;
            const uint32_t odd = __ballot_sync(all, l8 < n && !isfinite(x[c]));
            if (!live)
                continue;
            const int sc = bs * kb + c;
            const int64_t o0 = out.optr[sc];
            if (l8 < n) {
                out.oval[o0 + l8] = x[c];
                if (out.write_idx)
                    out.oidx[o0 + l8] = col;
            }
            if (l8 == 0) {
                const bool bad = ((odd >> (8 * grp)) & 0xffu) != 0 || !isfinite(res);
                out.olen[sc] = n;
                out.res[sc] = res;
                out.steps[sc] = 1;
                out.status[sc] = bad ? 2 : 0;
            }
        }
        if (live && l8 == 0) {
            const double dn = n, dm = m, dr = bs, E = entries;
            double* wk = out.work + 3 * static_cast<size_t>(kb);
            wk[0] += dn * E + dn * dn * dn / 3.0 + solves * dr * (2.0 * dn * dn + 4.0 * E);
            wk[1] += 2.0 * dm * dn * dn - (2.0 / 3.0) * dn * dn * dn + 4.0 * dm * dn * dr +
                     2.0 * dm * dn * dr;
            wk[2] += 12.0 * E + 16.0 * dn + 8.0 * dm * dr;
        }
        __syncwarp();
    }
}

// kLast: no larger arena follows.
template <class T, int NT, int MINB, bool kLast>
__global__ void __launch_bounds__(NT, MINB)
    block_solve_kernel(Problem pb, Output out, const int32_t* __restrict__ list,
                       const int32_t* __restrict__ count_dev, int count_host,
                       int32_t* __restrict__ counter, WorkList larger, WorkList left,
                       int arena_bytes)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ FixShared<T> fs;
    CtaGroup<NT> g{&fs.sc};
    const int count = count_dev ? *count_dev : count_host;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0)
            fs.sc.i[5] = atomicAdd(counter, 1);
        __syncthreads();
        const int t = fs.sc.i[5];
        __syncthreads();
        if (t >= count)
            break;
        const int kb = list[t];
        const Fit fit = block_column<T, NT>(g, fs, pb, out, kb, smem, arena_bytes);
        if (fit != Fit::kYes && threadIdx.x == 0) {
            if (!kLast && fit == Fit::kLarger)
                larger.list[atomicAdd(larger.count, 1)] = kb;
            else
                left.list[atomicAdd(left.count, 1)] = kb;
        }
    }
}

template <class T, int NT, int MINB, bool kLast>
cudaError_t launch_block_t(int arena, const Problem& pb, const Output& out, const int32_t* list,
                           const int32_t* count_dev, int count, int32_t* counter,
                           const WorkList& larger, const WorkList& left, cudaStream_t st)
{
    auto kern = block_solve_kernel<T, NT, MINB, kLast>;
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, arena);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, arena);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    const int grid = std::max(1, std::min(per_sm * num_sms(), count));
    kern<<<grid, NT, arena, st>>>(pb, out, list, count_dev, count, counter, larger, left, arena);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_block_solve(int elem_bytes, const Problem& pb, const Output& out,
                               const int32_t* list, int count, int32_t* const rest[3],
                               int32_t* counts, cudaStream_t st)
{
    // at most eight unknowns: eight lanes; small columns in FP64 (no refinement
    // to speak of on a few unknowns), 64 threads and eight CTAs per SM (15 KB and
    // the static 10 KB of shared memory); then 256 threads and two CTAs per SM, in
    // FP64 one
    const WorkList wide{rest[0], counts}, large{rest[1], counts + 1}, left{rest[2], counts + 2};
    const int blocks = std::max(1, std::min((count + 15) / 16, num_sms() * 16));
    block_small_kernel<<<blocks, 128, 0, st>>>(pb, out, list, count, wide, left);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = launch_block_t<double, 64, 8, false>(15 * 1024, pb, out, wide.list, wide.count, count,
                                           counts + 3, large, left, st);
    if (e != cudaSuccess)
        return e;
    if (elem_bytes == 4)
        return launch_block_t<float, 256, 2, true>(107 * 1024, pb, out, large.list, large.count, count,
                                             counts + 4, left, left, st);
    return launch_block_t<double, 256, 1, true>(212 * 1024, pb, out, large.list, large.count, count,
                                          counts + 4, left, left, st);
}

}  // namespace mspai
