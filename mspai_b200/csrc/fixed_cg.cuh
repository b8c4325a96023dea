// Fixed-pattern columns on the sparse normal equations: two solvers over the
// shared entries of fixed_sparse.cuh.
//
// cg_solve (four warps per column): iteration, for columns whose scaled normal
// matrix is diagonally dominant.  With G = C_J^T C_J, D = diag(G) and
// B = D^-1/2 |G - D| D^-1/2, a positive w with B w <= rho w gives spectral
// radius(B) <= rho (Collatz-Wielandt), so the eigenvalues of D^-1/2 G D^-1/2
// lie in [1 - rho, 1 + rho].  Columns with rho <= 0.9 after three power steps
// (|C|^T |C| bounds |G|) have a condition number of at most 19; the Chebyshev
// iteration (Saad, "Iterative methods for sparse linear systems", 2nd ed.,
// algorithm 12.1) then needs no dot products, and its number of steps follows
// from rho (ragged workload: rho 0.45, 27 steps).  A product with G visits the
// shared entries only, about 270 for a column of 134 unknowns and 2,500
// entries, where the dense path forms and factors a 134 x 134 triangle.  It is
// restarted from the FP64 gradient C^T (b - C x) until that is at the rounding
// level; mixed mode iterates in FP32 between restarts, as its factor is FP32 in
// the dense path.
//   Bound: instruction issue (0.5 to 0.6 per scheduler and cycle) and the
//   latency of two barriers a step; slots of 25 KB (and 1.7 KB static) allow
//   eight CTAs per SM.  Ragged workload, 1,000,000 columns: 700 ms in the dense
//   path, 76 ms here, 34 of them for finding and laying out the shared entries.
//
// hub_solve (a warp per column, small columns): elimination.  G has an
// off-diagonal entry only where two columns share a row.  A set of columns of
// which no two share a row (the leaves: in every row the column with the fewest
// shared entries) is eliminated exactly, each with its scalar pivot; the Schur
// complement of the others (the hubs, at most 32) is factored by Cholesky in
// FP64.  Patterns of at most 32 columns are all hubs.  The factor preconditions
// the FP64 refinement x += G^-1 C^T (b - C x), which ends at the least-squares
// solution as the dense path's does (fixed_solve.cuh), with the same test of
// the correction; FP64 mode, whose dense path takes no refinement, keeps the
// result only when the first correction is already at that level.
//
// Columns that neither takes (too many columns or entries for the slot, a zero
// column, values that are not finite, no certificate, no convergence) go to the
// dense factorizations of fixed_solve.cuh.  Every sum has a fixed order or is
// made of integers, so repeated setups are bit-identical.
#pragma once

#include "fixed_sparse.cuh"

namespace mspai {

constexpr int kCgRestarts = 6;
constexpr int kRowRegs = 3;         // entries of a row and of a column in registers
constexpr int kColRegs = 4;
constexpr float kCgRho = 0.9f;      // bound of the certificate
constexpr int kHubs = 32;           // at most this many hubs
constexpr int kHubLd = kHubs + 1;   // row stride of the Schur complement
constexpr int kLeafHubs = 4;        // at most this many hubs at a leaf

// Sum of two values over the CTA (two buffers: one barrier).
template <int NW>
__device__ __forceinline__ void cta_sum2(CgShared& sh, int& parity, double& a, double& b)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(kNone, a, o);
        b += __shfl_xor_sync(kNone, b, o);
    }
    if (NW > 1) {
        if (lane == 0) {
            sh.red[parity][warp][0] = a;
            sh.red[parity][warp][1] = b;
        }
        __syncthreads();
        a = sh.red[parity][0][0];
        b = sh.red[parity][0][1];
#pragma unroll
        for (int w = 1; w < NW; w++) {
            a += sh.red[parity][w][0];
            b += sh.red[parity][w][1];
        }
        parity ^= 1;
    }
}

__device__ __forceinline__ double sum_of_8(double a)
{
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
        a += __shfl_xor_sync(kNone, a, o);
    return a;
}
__device__ __forceinline__ float sum_of_8(float a)
{
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
        a += __shfl_xor_sync(kNone, a, o);
    return a;
}

// Part of sum v z over the entries q0, q0 + dq, ... of row or column i.
template <class Z>
__device__ __forceinline__ double jag_sum(const uint32_t* jag, const double* val,
                                          const uint16_t* idx, const Z* z, int i, int q0, int dq,
                                          bool absolute)
{
    double a = 0.0;
#pragma unroll 1
    for (int q = q0; q <= kCgMaxLen; q += dq) {
        const uint32_t j = jag[q];
        if (i >= static_cast<int>(j & 0xffffu))
            break;
        const int e = static_cast<int>(j >> 16) + i;
        const double v = val[e];
        a += (absolute ? fabs(v) : v) * z[idx[e]];
    }
    return a;
}

// y = b - C_s x on the shared rows (target: with b, else -C_s x), x by position
// in xs; us is overwritten.
template <int NW, int K>
__device__ __forceinline__ void shared_residual(CgShared& sh, const SharedEntries& g,
                                                const int (&at)[K], bool target)
{
    constexpr int NT = 32 * NW;
#pragma unroll
    for (int t = 0; t < K; t++)
        if (at[t] < g.n)
            g.us[at[t]] = -g.xs[at[t]];
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < g.S; i += NT)
        g.y[i] = jag_sum(sh.rows, g.ev, g.ec, g.us, i, 0, 1, false);
    __syncthreads();
    if (target && g.tg_rid >= 0)
        g.y[g.tg_rid] += g.tg_val;
    __syncthreads();
}

// r = (scaled C)^T (b - C x) per slot, or the scaled rhs - C^T C x when a
// right-hand side (by position) is given; y: see shared_residual.
template <int NW, int K>
__device__ __forceinline__ void scaled_gradient(CgShared& sh, const SharedEntries& g,
                                                const int (&at)[K], int nlong,
                                                const double* scale, const double* rhs,
                                                double (&r)[K])
{
    const int tid = threadIdx.x, warp = tid >> 5, l8 = tid & 7;
    shared_residual<NW, K>(sh, g, at, rhs == nullptr);
    r[0] = 0.0;
    if (4 * warp < nlong)
        r[0] = sum_of_8(tid / 8 < nlong ? jag_sum(sh.cols, g.cv, g.cr, g.y, tid / 8, l8, 8, false)
                                        : 0.0);
#pragma unroll
    for (int t = 1; t < K; t++)
        r[t] = at[t] < g.n ? jag_sum(sh.cols, g.cv, g.cr, g.y, at[t], 0, 1, false) : 0.0;
#pragma unroll
    for (int t = 0; t < K; t++) {
        if (at[t] < g.n) {
            const double v = rhs ? r[t] + rhs[at[t]] : r[t];
            r[t] = (v - g.xs[at[t]] * g.d0[g.ccol[at[t]]]) * scale[at[t]];
        }
        else {
            r[t] = 0.0;
        }
    }
}

// Writes the column's results; y holds the residual of the shared rows.
template <int NW, int K>
__device__ __forceinline__ void write_column(CgShared& sh, int& parity, const SharedEntries& g,
                                             const Output& out, int col, const int (&at)[K],
                                             double solve_flops)
{
    const int tid = threadIdx.x, lane = tid & 31;
    // residual norm: shared rows in candidate order, single rows from d0
    double r2 = 0.0, nonfinite = 0.0;
#pragma unroll 1
    for (int c = lane; c < g.nc; c += 32) {
        const uint32_t id = g.cand[-NW * c].x;
        if (id != kNone && (id & kFirst)) {
            const double v = g.y[id & ~kFirst];
            r2 += v * v;
        }
    }
#pragma unroll
    for (int t = 0; t < K; t++) {
        if (at[t] < g.n) {
            const int jj = g.ccol[at[t]];
            const double x = g.xs[at[t]];
            r2 += x * x * g.d0[jj];
            if (!isfinite(x))
                nonfinite = 1.0;
            out.oval[g.p0 + jj] = x;
        }
    }
    cta_sum2<NW>(sh, parity, r2, nonfinite);
    if (tid == 0) {
        const double dn = g.n, dm = (g.E - g.nctot) + sh.distinct;
        double* wk = out.work + 3 * static_cast<size_t>(col);
        wk[0] += 4.0 * g.E + solve_flops;
        wk[1] += 2.0 * dm * dn * dn - (2.0 / 3.0) * dn * dn * dn + 4.0 * dm * dn + 2.0 * dm * dn;
        wk[2] += 12.0 * g.E + 16.0 * dn + 8.0 * dm;
        out.olen[col] = g.n;
        out.res[col] = sqrt(r2);
        out.steps[col] = 1;
        out.status[col] = (nonfinite == 0.0 && isfinite(r2)) ? 0 : 2;
    }
}

// Positions of this thread's columns: slot 0 the NT / 8 longest ones with more
// than four entries, one for each group of eight lanes (its first lane owns
// it), then one column a thread in each slot; n: none.  Returns the number of
// columns with eight lanes.
template <int NW, int K>
__device__ __forceinline__ int column_slots(const CgShared& sh, int n, int (&at)[K])
{
    constexpr int NT = 32 * NW, LG = NT / 8;
    const int tid = threadIdx.x;
    const int nlong =
        min(LG, max(static_cast<int>(sh.cols[4] & 0xffffu), n - NT * (K - 1)));
    at[0] = ((tid & 7) == 0 && tid / 8 < nlong) ? tid / 8 : n;
#pragma unroll
    for (int t = 1; t < K; t++)
        at[t] = min(n, nlong + NT * (t - 1) + tid);
    return nlong;
}

// 1 / ||c_j|| by position into scale (which is gd); false (uniformly) when a
// column is zero or not finite.  us is overwritten; ends with a barrier.
template <int NW, int K>
__device__ __forceinline__ bool column_scales(const SharedEntries& g, const int (&at)[K])
{
    double sd[K];
    bool bad = false;
#pragma unroll
    for (int t = 0; t < K; t++) {
        sd[t] = 0.0;
        if (at[t] < g.n) {
            const double q = g.gd[g.ccol[at[t]]];
            bad = bad || !(q > 0.0) || !(q < 1e300);
            sd[t] = 1.0 / sqrt(q);
        }
    }
    if (__syncthreads_or(bad))
        return false;
#pragma unroll
    for (int t = 0; t < K; t++)
        if (at[t] < g.n)
            g.gd[at[t]] = sd[t];
    __syncthreads();
    return true;
}

// Fixed-point numbers whose sums do not depend on the order: the entries of the
// scaled matrices are at most a few, and a sum that wraps around all the same
// gives a factor whose refinement does not converge.
template <class T>
struct Fixed;
template <>
struct Fixed<double> {
    typedef long long type;
    static __device__ __forceinline__ void add(long long* p, double v)
    {
        atomicAdd(reinterpret_cast<unsigned long long*>(p),
                  static_cast<unsigned long long>(__double2ll_rn(v * 0x1p58)));
    }
    static __device__ __forceinline__ double value(long long v) { return v * 0x1p-58; }
    static constexpr long long one = 1ll << 58;
};

template <class T, int NW, int K>
__device__ bool hub_solve(CgShared& sh, int& parity, const SharedEntries& g, const Problem& pb,
                          const Output& out, int col, char* base, const int (&at)[K], int nlong)
{
    typedef typename Fixed<T>::type Fix;
    constexpr int NT = 32 * NW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = g.n;
    Fix* schur = reinterpret_cast<Fix*>(base + ((g.free_lo + 15) & ~15));
    const int most_hubs = min(n, kHubs);
    Fix* hacc = schur + most_hubs * kHubLd;      // right-hand side of the hubs
    T* hx = reinterpret_cast<T*>(hacc + kHubs);  // their solution
    uint8_t* hub = reinterpret_cast<uint8_t*>(hx + kHubs);  // by position; 0xff: leaf
    if (reinterpret_cast<char*>(hub + n) > base + g.free_hi)
        return false;
    const double* scale = g.gd;
    for (int i = tid; i < n; i += NT)
        hub[i] = n <= kHubs ? 0 : 0xff;
    for (int i = tid; i < most_hubs * kHubLd + kHubs; i += NT)
        schur[i] = 0;
    __syncthreads();
    // ---- hubs: every column of a row but the last one in the order of
    // decreasing shared entries
    auto entry = [&](int i, int q) {
        const uint32_t j = q <= kCgMaxLen ? sh.rows[q] : 0u;
        return i < static_cast<int>(j & 0xffffu) ? static_cast<int>(j >> 16) + i : -1;
    };
    if (n > kHubs) {
#pragma unroll 1
        for (int i = tid; i < g.S; i += NT) {
            uint32_t last = 0;
            for (int q = 0, e; (e = entry(i, q)) >= 0; q++)
                last = max(last, static_cast<uint32_t>(g.ec[e]));
            for (int q = 0, e; (e = entry(i, q)) >= 0; q++)
                if (g.ec[e] != last)
                    hub[g.ec[e]] = 0;
        }
        __syncthreads();
    }
    if (warp == 0) {
        int nh = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const bool h = i0 + lane < n && hub[i0 + lane] == 0;
            const uint32_t b = __ballot_sync(kNone, h);
            if (h)
                hub[i0 + lane] = static_cast<uint8_t>(min(254, nh + __popc(b & ((1u << lane) - 1u))));
            nh += __popc(b);
        }
        if (lane < min(nh, kHubs))
            schur[lane * kHubLd + lane] = Fixed<T>::one;
        if (lane == 0) {
            sh.nrows = nh;
            sh.over = 0;
            sh.bound[0] = 0;
        }
    }
    __syncthreads();
    const int nh = sh.nrows;
    if (nh > kHubs)
        return false;
    // ---- Schur complement: products inside the hubs (lower triangle) ...
#pragma unroll 1
    for (int i = tid; i < g.S; i += NT) {
        for (int q = 1, e; (e = entry(i, q)) >= 0; q++) {
            const int p1 = g.ec[e], h1 = hub[p1];
            if (h1 == 0xff)
                continue;
            const T v1 = static_cast<T>(g.ev[e] * scale[p1]);
            for (int k = 0; k < q; k++) {
                const int f = entry(i, k), p2 = g.ec[f], h2 = hub[p2];
                if (h2 != 0xff)
                    Fixed<T>::add(&schur[max(h1, h2) * kHubLd + min(h1, h2)],
                                  v1 * static_cast<T>(g.ev[f] * scale[p2]));
            }
        }
    }
    // ... less those through the leaves.  A leaf's rows hold it and hubs only.
    uint32_t lh[K];             // its hubs, a byte each
    T lg[K][kLeafHubs];         // and the entries of the scaled matrix
    int ln[K];                  // how many; -1: not a leaf
#pragma unroll
    for (int t = 0; t < K; t++) {
        lh[t] = 0;
        ln[t] = -1;
#pragma unroll
        for (int q = 0; q < kLeafHubs; q++)
            lg[t][q] = T(0);
        if (at[t] >= n || hub[at[t]] != 0xff)
            continue;
        ln[t] = 0;
#pragma unroll 1
        for (int q = 0; q <= kCgMaxLen; q++) {
            const uint32_t j = sh.cols[q];
            if (at[t] >= static_cast<int>(j & 0xffffu))
                break;
            const int e = static_cast<int>(j >> 16) + at[t];
            const int row = g.cr[e];
            const T v = static_cast<T>(g.cv[e] * scale[at[t]]);
            for (int k = 0, f; (f = entry(row, k)) >= 0; k++) {
                const int p = g.ec[f];
                if (p == at[t])
                    continue;
                const uint32_t h = hub[p];
                const T gv = v * static_cast<T>(g.ev[f] * scale[p]);
                bool found = false;
#pragma unroll
                for (int s = 0; s < kLeafHubs; s++) {
                    if (s < ln[t] && ((lh[t] >> (8 * s)) & 0xffu) == h) {
                        lg[t][s] += gv;
                        found = true;
                    }
                }
                if (!found) {
                    if (ln[t] >= kLeafHubs) {
                        sh.over = 1;
                    }
                    else {
#pragma unroll
                        for (int s = 0; s < kLeafHubs; s++) {
                            if (s == ln[t]) {
                                lh[t] |= h << (8 * s);
                                lg[t][s] = gv;
                            }
                        }
                        ln[t]++;
                    }
                }
            }
        }
#pragma unroll
        for (int a = 0; a < kLeafHubs; a++) {
#pragma unroll
            for (int b = 0; b <= a; b++) {
                if (a < ln[t]) {
                    const int ha = (lh[t] >> (8 * a)) & 0xffu, hb = (lh[t] >> (8 * b)) & 0xffu;
                    Fixed<T>::add(&schur[max(ha, hb) * kHubLd + min(ha, hb)],
                                  -(lg[t][a] * lg[t][b]));
                }
            }
        }
    }
    __syncthreads();
    if (sh.over)
        return false;
    // ---- Cholesky of the hubs by warp 0, left-looking, a lane per row
    T* L = reinterpret_cast<T*>(schur);
    T inv = T(0);  // 1 / L(lane, lane)
    if (warp == 0) {
        for (int j = 0; j < nh; j++)
            if (lane < nh)
                L[lane * kHubLd + j] = Fixed<T>::value(schur[lane * kHubLd + j]);
        __syncwarp();
        // FP64 without refinement: beyond a condition of 2^13 the first correction
        // does not reach 2^-44 (1 is the largest pivot of the scaled matrix), so the
        // column is refused here and not after two corrections
        const T least = pb.refine > 0 ? T(0) : T(0x1p-13);
        bool bad = false;
#pragma unroll 1
        for (int j = 0; j < nh; j++) {
            T s = (lane >= j && lane < nh) ? L[lane * kHubLd + j] : T(0);
            if (lane >= j && lane < nh) {
#pragma unroll 4
                for (int k = 0; k < j; k++)
                    s -= L[lane * kHubLd + k] * L[j * kHubLd + k];
            }
            const T piv = __shfl_sync(kNone, s, j);
            bad = bad || !(piv > least);
            const T iv = T(1) / tsqrt<T>(bad ? T(1) : piv);
            if (lane == j)
                inv = iv;
            if (lane > j && lane < nh)
                L[lane * kHubLd + j] = s * iv;
            __syncwarp();
        }
        if (bad && lane == 0)
            sh.bound[0] = 1;
    }
#pragma unroll
    for (int t = 0; t < K; t++)
        if (at[t] < n)
            g.xs[at[t]] = 0.0;
    __syncthreads();
    if (sh.bound[0])
        return false;
    // ---- refinement from x = 0
    const int most = pb.refine > 0 ? pb.refine + 2 : 3;
    int steps = 0;
    bool conv = false;
    double d2_prev = 0.0;
#pragma unroll 1
    for (int it = 0; it < most; it++) {
        double r[K];
        scaled_gradient<NW, K>(sh, g, at, nlong, scale, nullptr, r);
        double gam = 0.0, unused = 0.0;
#pragma unroll
        for (int t = 0; t < K; t++)
            gam += r[t] * r[t];
        cta_sum2<NW>(sh, parity, gam, unused);
        if (!(gam < 1e300))
            return false;
        if (gam == 0.0) {  // x solves the normal equations as it is
            conv = true;
            break;
        }
        steps++;
        const double size = sqrt(gam), unit = 1.0 / size;
        T rt[K];
#pragma unroll
        for (int t = 0; t < K; t++) {
            rt[t] = static_cast<T>(r[t] * unit);
            if (at[t] < n) {
                if (ln[t] < 0) {
                    Fixed<T>::add(&hacc[hub[at[t]]], rt[t]);
                }
                else {
#pragma unroll
                    for (int s = 0; s < kLeafHubs; s++)
                        if (s < ln[t])
                            Fixed<T>::add(&hacc[(lh[t] >> (8 * s)) & 0xffu], -(lg[t][s] * rt[t]));
                }
            }
        }
        __syncthreads();
        if (warp == 0) {
            T b = Fixed<T>::value(hacc[lane]);
            hacc[lane] = 0;
            const T* mine = L + lane * kHubLd;
#pragma unroll 1
            for (int j = 0; j < nh; j++) {  // L z = b
                if (lane == j)
                    b *= inv;
                const T z = __shfl_sync(kNone, b, j);
                if (lane > j && lane < nh)
                    b -= mine[j] * z;
            }
#pragma unroll 1
            for (int j = nh - 1; j >= 0; j--) {  // L^T x = z
                if (lane == j)
                    b *= inv;
                const T z = __shfl_sync(kNone, b, j);
                if (lane < j)
                    b -= L[j * kHubLd + lane] * z;
            }
            hx[lane] = b;
        }
        __syncthreads();
        double d2 = 0.0, x2 = 0.0;
#pragma unroll
        for (int t = 0; t < K; t++) {
            if (at[t] < n) {
                T d;
                if (ln[t] < 0) {
                    d = hx[hub[at[t]]];
                }
                else {
                    d = rt[t];
#pragma unroll
                    for (int s = 0; s < kLeafHubs; s++)
                        if (s < ln[t])
                            d -= lg[t][s] * hx[(lh[t] >> (8 * s)) & 0xffu];
                }
                const double dx = static_cast<double>(d) * (size * scale[at[t]]);
                const double x = g.xs[at[t]] + dx;
                g.xs[at[t]] = x;
                d2 += dx * dx;
                x2 += x * x;
            }
        }
        cta_sum2<NW>(sh, parity, d2, x2);
        // converged: the correction is below 2^-44 of the solution; FP64 without
        // refinement has to reach that with its first correction
        conv = d2 <= 0x1p-88 * x2;
        if (conv || (it > 0 && !(d2 <= 0.25 * d2_prev)) || (it == 1 && pb.refine == 0))
            break;
        d2_prev = d2;
    }
    if (!conv)
        return false;
    shared_residual<NW, K>(sh, g, at, true);
    write_column<NW, K>(sh, parity, g, out, col, at,
                        nh * (nh * nh / 3.0) + steps * (4.0 * g.ns + 12.0 * n + 2.0 * nh * nh));
    return true;
}

// Solves min ||C x - b|| (rhs: C^T C x = rhs) into xs; returns the steps taken,
// -1 (uniformly) when the column is not certified or does not converge.  y
// holds b - C x (-C x) on the shared rows.  prev: a previous solution in the
// order of J to start from, or null; -2 when its gradient is not below 1/16 of
// that of x = 0 (the values have changed too much for a start from it).
template <class T, int NW, int K>
__device__ int cg_solve(CgShared& sh, int& parity, const SharedEntries& g, const int (&at)[K],
                        int nlong, const double* rhs, const double* prev)
{
    constexpr int NT = 32 * NW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l8 = lane & 7;
    const int n = g.n, S = g.S;
    const double *d0 = g.d0, *ev = g.ev, *cv = g.cv;
    const uint16_t *ccol = g.ccol, *ec = g.ec, *cr = g.cr;
    double *us = g.us, *xs = g.xs, *y = g.y;
    const double* scale = g.gd;
    // ---- the entries of this thread's rows and columns in registers, in T and
    // scaled to columns of norm one: the first two of two rows (numbers tid and
    // NT + tid) and of each column, four of a column with eight lanes; what lies
    // beyond is read from shared memory
    auto entry = [&](const uint32_t* jag, int i, int q) {
        const uint32_t j = q <= kCgMaxLen ? jag[q] : 0u;
        return i < static_cast<int>(j & 0xffffu) ? static_cast<int>(j >> 16) + i : -1;
    };
    constexpr int KC = K > 2 ? 2 : 1;  // column slots with entries in registers
    T rv[2][kRowRegs], cw[KC][kColRegs], lv[4];
    uint32_t ri[2][2], ci2[KC][2], li[2];  // two places in one word
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint32_t id[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < kRowRegs; q++) {
            const int e = entry(sh.rows, NT * k + tid, q);
            id[q] = e >= 0 ? ec[e] : 0u;
            rv[k][q] = e >= 0 ? static_cast<T>(ev[e] * scale[id[q]]) : T(0);
        }
        ri[k][0] = id[0] | (id[1] << 16);
        ri[k][1] = id[2] | (id[3] << 16);
    }
#pragma unroll
    for (int t = 1; t <= KC; t++) {
        uint32_t id[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < kColRegs; q++) {
            const int e = at[t] < n ? entry(sh.cols, at[t], q) : -1;
            id[q] = e >= 0 ? cr[e] : 0u;
            cw[t - 1][q] = e >= 0 ? static_cast<T>(cv[e] * scale[at[t]]) : T(0);
        }
        ci2[t - 1][0] = id[0] | (id[1] << 16);
        ci2[t - 1][1] = id[2] | (id[3] << 16);
    }
    const bool in_long = tid / 8 < nlong;
    const double sdl = in_long ? scale[tid / 8] : 0.0;
#pragma unroll
    for (int m = 0; m < 2; m++) {
        uint32_t id[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int e = in_long ? entry(sh.cols, tid / 8, l8 + 8 * (2 * m + q)) : -1;
            id[q] = e >= 0 ? cr[e] : 0u;
            lv[2 * m + q] = e >= 0 ? static_cast<T>(cv[e] * sdl) : T(0);
        }
        li[m] = id[0] | (id[1] << 16);
    }
    // w = (scaled C_s)^T (scaled C_s) d for d in zt; with absolute, of |C_s|.
    // Entries beyond the registers are scaled on the way.
    T* zt = reinterpret_cast<T*>(us);  // d, by position
    T* yt = reinterpret_cast<T*>(y);
    // rows and columns with entries beyond the registers
    const int rfar = static_cast<int>(sh.rows[kRowRegs] & 0xffffu);
    const int cfar = static_cast<int>(sh.cols[kColRegs] & 0xffffu);
    const int cols32 = static_cast<int>(sh.cols[32] & 0xffffu);
    // a row's sum does not depend on where its entries are read: its number, and
    // so the path it takes, may differ from call to call
    auto far_row = [&](int i, int q0, T a, bool absolute) {
#pragma unroll 1
        for (int q = q0; q <= kCgMaxLen; q++) {
            const uint32_t j = sh.rows[q];
            if (i >= static_cast<int>(j & 0xffffu))
                break;
            const int e = static_cast<int>(j >> 16) + i;
            const uint32_t c = ec[e];
            const T v = static_cast<T>(ev[e] * scale[c]);
            a = fma(absolute ? abs(v) : v, zt[c], a);
        }
        return a;
    };
    auto product = [&](T (&w)[K], bool absolute) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int i = NT * k + tid;
            if (NT * k + 32 * warp >= S)
                break;
            if (i < S) {
                T a = T(0);
#pragma unroll
                for (int q = 0; q < kRowRegs; q++) {
                    const T v = absolute ? abs(rv[k][q]) : rv[k][q];
                    a = fma(v, zt[(ri[k][q / 2] >> (16 * (q % 2))) & 0xffffu], a);
                }
                if (i < rfar)
                    a = far_row(i, kRowRegs, a, absolute);
                yt[i] = a;
            }
        }
#pragma unroll 1
        for (int i = 2 * NT + tid; i < S; i += NT)
            yt[i] = far_row(i, 0, T(0), absolute);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < K; t++)
            w[t] = T(0);
        if (4 * warp < nlong) {
            T a = T(0);
            if (in_long) {
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const T v0 = absolute ? abs(lv[2 * m]) : lv[2 * m];
                    const T v1 = absolute ? abs(lv[2 * m + 1]) : lv[2 * m + 1];
                    a += v0 * yt[li[m] & 0xffffu] + v1 * yt[li[m] >> 16];
                }
                if (tid / 8 < cols32)
                    a += static_cast<T>(sdl * jag_sum(sh.cols, cv, cr, yt, tid / 8, 32 + l8, 8,
                                                   absolute));
            }
            w[0] = sum_of_8(a);
        }
#pragma unroll
        for (int t = 1; t < K; t++) {
            if (nlong + NT * (t - 1) + 32 * warp >= n)
                break;  // no lane of this warp has a column here
            if (at[t] < n) {
                T a = T(0);
                if (t <= KC) {
#pragma unroll
                    for (int q = 0; q < kColRegs; q++) {
                        const T v = absolute ? abs(cw[(t - 1) % KC][q]) : cw[(t - 1) % KC][q];
                        a = fma(v, yt[(ci2[(t - 1) % KC][q / 2] >> (16 * (q % 2))) & 0xffffu], a);
                    }
                }
                if (t > KC || at[t] < cfar)
                    a += static_cast<T>(scale[at[t]] * jag_sum(sh.cols, cv, cr, yt, at[t],
                                                            t <= KC ? kColRegs : 0, 1, absolute));
                w[t] = a;
            }
        }
    };
    // ---- certificate: three power steps with |C_s|^T |C_s| without its
    // diagonal, the smallest of their bounds
    T dh[K];  // the single rows' part of the scaled diagonal
#pragma unroll
    for (int t = 0; t < K; t++)
        dh[t] = at[t] < n ? static_cast<T>(d0[ccol[at[t]]] * scale[at[t]] * scale[at[t]]) : T(0);
    float rho = 2.0f;
    {
        T w[K];
#pragma unroll
        for (int t = 0; t < K; t++)
            w[t] = T(1);
        if (tid < 3)
            sh.bound[tid] = 0;
#pragma unroll 1
        for (int it = 0; it < 3; it++) {
            __syncthreads();
#pragma unroll
            for (int t = 0; t < K; t++)
                if (at[t] < n)
                    zt[at[t]] = w[t];
            __syncthreads();
            T a[K];
            product(a, true);
            float worst = 0.0f;
#pragma unroll
            for (int t = 0; t < K; t++) {
                if (at[t] < n) {
                    // fmax: rounding may leave a tiny negative sum
                    const T u = max(T(0), a[t] - (T(1) - dh[t]) * w[t]);
                    const float q = static_cast<float>(u / w[t]);
                    worst = q >= 0.0f ? fmaxf(worst, q) : 2.0f;
                    w[t] = u + T(0.3) * w[t];
                }
            }
            const int wi = __reduce_max_sync(kNone, __float_as_int(worst));
            if (lane == 0)
                atomicMax(&sh.bound[it], wi);
            __syncthreads();
            rho = fminf(rho, __int_as_float(sh.bound[it]));
        }
        // 1e-4: more than the rounding of the bound itself
        rho += 1e-4f;
        if (!(rho <= kCgRho))
            return -1;
    }
    // ---- Chebyshev iteration on the scaled system, restarted from the FP64
    // residual: steps that reduce the error by 2^-18 (T = float) or 2^-28
    double r[K];
#pragma unroll
    for (int t = 0; t < K; t++)
        if (at[t] < n)
            xs[at[t]] = 0.0;
    constexpr float kBits = sizeof(T) == 4 ? 18.0f : 28.0f;
    const float rb = fmaxf(rho, 0.02f);
    // the error shrinks by sigma = rho / (1 + sqrt(1 - rho^2)) a step
    const int m_steps = static_cast<int>(
        ceilf((kBits + 1.0f) / -log2f(rb / (1.0f + sqrtf(1.0f - rb * rb)))));
    int steps = 0;
    double g0 = 0.0, gam_prev = 1e300;
    bool conv = false;
#pragma unroll 1
    for (int restart = prev ? -1 : 0; restart <= kCgRestarts; restart++) {
        scaled_gradient<NW, K>(sh, g, at, nlong, scale, rhs, r);
        double gam = 0.0, unused = 0.0;
#pragma unroll
        for (int t = 0; t < K; t++)
            gam += r[t] * r[t];
        cta_sum2<NW>(sh, parity, gam, unused);
        if (restart < 0) {
            // x = 0 gave the size of the right-hand side; now the previous solution
            g0 = gam;
#pragma unroll
            for (int t = 0; t < K; t++)
                if (at[t] < n)
                    xs[at[t]] = prev[ccol[at[t]]];
            continue;
        }
        if (restart == 0) {
            if (!prev)
                g0 = gam;
            else if (!(gam <= 0x1p-8 * g0))
                return -2;
        }
        // the gradient is 2^-52 of its first value (or zero), or below 2^-48 and
        // no longer shrinking: rounding level
        conv = gam <= 0x1p-104 * g0 ||
               (gam <= 0x1p-96 * g0 && (gam > 0x1p-20 * gam_prev || restart == kCgRestarts));
        gam_prev = gam;
        if (conv || !(gam < 1e300) || restart == kCgRestarts)
            break;
        const double size = sqrt(gam), unit = 1.0 / size;
        T d[K], rt[K], xt[K];
#pragma unroll
        for (int t = 0; t < K; t++) {
            rt[t] = d[t] = static_cast<T>(r[t] * unit);
            xt[t] = T(0);
        }
        const T s1 = T(1) / static_cast<T>(rb);
        T c = static_cast<T>(rb);
#pragma unroll 1
        for (int it = 0; it < m_steps; it++) {
#pragma unroll
            for (int t = 0; t < K; t++)
                if (at[t] < n)
                    zt[at[t]] = d[t];
            __syncthreads();
            T w[K];
            product(w, false);
            const T c1 = T(1) / (T(2) * s1 - c);
            const T e1 = c1 * c, e2 = T(2) * c1 * s1;
            c = c1;
#pragma unroll
            for (int t = 0; t < K; t++) {
                xt[t] += d[t];
                rt[t] -= w[t] + dh[t] * d[t];
                d[t] = e1 * d[t] + e2 * rt[t];
            }
        }
        steps += m_steps;
#pragma unroll
        for (int t = 0; t < K; t++)
            if (at[t] < n)
                xs[at[t]] += static_cast<double>(xt[t]) * (size * scale[at[t]]);
        __syncthreads();  // zt and yt are done before us and y are written
    }
    return conv ? steps : -1;
}

}  // namespace mspai

