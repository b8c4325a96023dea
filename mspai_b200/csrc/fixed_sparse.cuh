// The sparse form of a fixed-pattern column's least-squares problem, shared by
// the solvers of fixed_cg.cu: the rows of C(:, J) with two or more entries,
// found and laid out in shared memory by the NW warps of a CTA.
//
// C(:, J) of a column (the reference's I set and submatrix, src/Spai_Sub.imp:
// 65-122, 221-282) is very sparse: most of its rows have one entry.  Such a row
// only adds v^2 to the diagonal of the normal matrix C^T C, so only the other
// rows are kept.
//
//  1. A first pass over the rows of C(:, J) sets one bit per row in a hashed bit
//     map and, where the bit was set before, a bit in a second map; a second
//     pass keeps the entries whose row hits the second map (candidates) and sums
//     the squares of the others into d0.  Both passes are bound by the latency
//     of the reads of C: eight lanes a column, four columns a warp, the next
//     four on their way.
//  2. The candidates are grouped by row in a small exact hash table; one that is
//     alone after all goes to d0 as well.
//  3. The shared entries are stored twice, by row and by column, rows and
//     columns in the order of decreasing length with the q-th entries of all
//     rows side by side (jagged diagonals): a thread owns a row or a column,
//     every access to values and indices is conflict free and nothing is padded.
//
// The order of the entries of a row and of a column does not depend on the
// schedule; the numbers of the rows do.
#pragma once

#include "spai_kernels.h"
#include "spai_solve.cuh"

namespace mspai {

constexpr int kCgMaxTargets = 16;   // entries of B(:, k)
constexpr int kCgMaxLen = 127;      // shared entries of a row or a column
constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kFirst = 0x80000000u;  // candidate is the first entry of its row

__device__ __forceinline__ uint32_t cg_hash(uint32_t row, int bits)
{
    return (row * 2654435761u) >> (32 - bits);
}

// Exclusive sum over the lanes above this one.
__device__ __forceinline__ uint32_t cg_sum_above(uint32_t v, int lane)
{
    uint32_t s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_down_sync(kNone, s, o);
        if (lane + o < 32)
            s += t;
    }
    return s - v;
}

// Shared state of a column's CTA beside its slot.
struct CgShared {
    double red[2][4][2];            // dot products of the warps, two buffers
    uint32_t bins[kCgMaxLen + 1];   // histogram of lengths, then the next number of a length
    uint32_t rows[kCgMaxLen + 1];   // per q: first entry number q << 16 | rows longer than q
    uint32_t cols[kCgMaxLen + 1];   // the same of the columns
    int ncw[4];                     // candidates of each warp
    int bound[3];                   // the certificate's bounds, as float bits
    int entries, longest, distinct, shared_entries, nrows, over, next;
};

// From the histogram of lengths in bins: the first number of each length in
// decreasing order back into bins, and per q the first place of the q-th
// entries and how many there are; warp 0.  Returns (warp 0) the number of rows
// that are not empty.
__device__ __forceinline__ uint32_t cg_order(uint32_t* bins, uint32_t* jag, int lane)
{
    constexpr int B = (kCgMaxLen + 1) / 32;
    uint32_t b[B], sum = 0;
#pragma unroll
    for (int i = 0; i < B; i++) {
        b[i] = bins[B * lane + i];
        sum += b[i];
    }
    uint32_t above = cg_sum_above(sum, lane);  // rows of the lengths of later lanes
    uint32_t part = 0;
#pragma unroll
    for (int i = B - 1; i >= 0; i--) {
        const uint32_t t = b[i];
        b[i] = above;  // rows longer than B lane + i
        part += above;
        above += t;
    }
    uint32_t first = part;  // entries before those of this lane's lengths
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kNone, first, o);
        if (lane >= o)
            first += t;
    }
    first -= part;
#pragma unroll
    for (int i = 0; i < B; i++) {
        bins[B * lane + i] = b[i];
        jag[B * lane + i] = (first << 16) | b[i];
        first += b[i];
    }
    return __shfl_sync(kNone, b[0], 0);
}

// Entries of a row over the warps' byte counts.
__device__ __forceinline__ uint32_t cg_count(uint32_t packed)
{
    packed &= ~kFirst;
    return (packed & 0xffu) + ((packed >> 8) & 0xffu) + ((packed >> 16) & 0xffu) + (packed >> 24);
}

// A column's shared entries.
struct SharedEntries {
    int n;                // |J|
    int E;                // entries of C(:, J)
    int nc;               // this warp's candidates
    int nctot;            // all candidates
    int ns;               // shared entries
    int S;                // shared rows
    int free_lo, free_hi; // free bytes of the slot
    int64_t p0;
    double* d0;           // per column of J: squares of the entries alone in their row
    double* gd;           // squares of all entries
    double* us;           // n values
    double* xs;           // n values: the solution, by position
    uint32_t* cb;         // start of C(:, J(i))
    uint32_t* tmp;        // n words
    uint16_t* cpos;       // position of each column of J (decreasing shared entries)
    uint16_t* ccol;       // column of J at each position
    double* ev;           // shared entries by row: value and position of the column
    uint16_t* ec;
    double* cv;           // by column: value and row number
    uint16_t* cr;
    double* y;            // one value per shared row
    uint2* cand;          // candidate c of this warp at cand[-NW c]; x: its row, with
                          // kFirst in the row's first candidate, kNone: not shared
    int tg_rid;           // this thread's target entry: shared row (-1: none) and value
    double tg_val;
};

// What becomes of a column.
enum class Taken {
    kYes,
    kLarger,  // it does not fit this slot
    kFar,     // a re-setup's column, too far from its previous solution
    kNo       // it fits no slot, or the solver refuses it: the next slot would as well
};

constexpr int kWidestN = 400;  // columns of J in the largest slot

// Lays column `col` out in the slot (uniformly); at most nmax columns of J.
// widest: bytes of the largest slot that the launches use.
template <int NW>
__device__ Taken gather_shared(CgShared& sh, const Problem& pb, int col, char* base, int cap,
                               int nmax, int widest, SharedEntries& g)
{
    constexpr int NT = 32 * NW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const int64_t p0 = pb.pptr[col];
    const int n = static_cast<int>(pb.pptr[col + 1] - p0);
    if (n < 1 || n > kWidestN)
        return Taken::kNo;
    if (n > nmax)
        return Taken::kLarger;
    // ---- fixed part of the slot
    double* d0 = reinterpret_cast<double*>(base);
    double* gd = d0 + n;
    double* us = gd + n;
    double* xs = us + n;                                 // the solution, by position
    uint32_t* cb = reinterpret_cast<uint32_t*>(xs + n);  // start of C(:, J(i))
    uint32_t* clen = cb + n;                             // its length; later its shared entries
    uint16_t* cpos = reinterpret_cast<uint16_t*>(clen + n);
    uint16_t* ccol = cpos + n;
    const int ra = static_cast<int>((reinterpret_cast<char*>(ccol + n) - base + 15) & ~15);
    const int64_t tg0 = pb.bptr ? pb.bptr[col] : 0;
    const int ntg = pb.bptr ? static_cast<int>(pb.bptr[col + 1] - tg0) : 1;
    if (ntg > kCgMaxTargets)
        return Taken::kNo;
    if (ra >= cap)
        return ra >= widest ? Taken::kNo : Taken::kLarger;
    if (tid == 0) {
        sh.entries = sh.longest = sh.distinct = sh.shared_entries = sh.over = 0;
    }
    __syncthreads();
    {
        int e = 0, longest = 0;
#pragma unroll 1
        for (int i = tid; i < n; i += NT) {
            const int j = pb.pidx[p0 + i];
            const int64_t b0 = pb.cptr[j];
            const int l = static_cast<int>(pb.cptr[j + 1] - b0);
            cb[i] = static_cast<uint32_t>(b0);
            clen[i] = static_cast<uint32_t>(l);
            e += l;
            longest = max(longest, l);
        }
        e = __reduce_add_sync(kNone, e);
        longest = __reduce_max_sync(kNone, longest);
        if (lane == 0) {
            atomicAdd(&sh.entries, e);
            atomicMax(&sh.longest, longest);
        }
    }
    const bool is_tg = tid < ntg;
    int tg_row = -1;
    double tg_val = 0.0;
    if (is_tg) {
        tg_row = pb.bptr ? pb.bidx[tg0 + tid] : col;
        tg_val = pb.bptr ? pb.bval[tg0 + tid] : 1.0;
    }
    __syncthreads();
    const int E = sh.entries;
    if (sh.longest > 0xffff || E < 1 || E > (1 << 20))
        return Taken::kNo;
    // ---- the two bit maps: 8 to 16 bits per entry
    const int hb = max(10, 32 - __clz(8 * E - 1));
    const int mapw = 1 << (hb - 5);
    uint32_t* bm1 = reinterpret_cast<uint32_t*>(base + ra);
    uint32_t* bm2 = bm1 + mapw;
    const int room = cap - ra - 8 * mapw;  // candidates, from the slot's end down
    if (room < 16 * n)
        return widest - ra - 8 * mapw < 16 * n ? Taken::kNo : Taken::kLarger;
    // candidate c of warp w at cand[-(NW c + w)]
    uint2* cand = reinterpret_cast<uint2*>(base + cap) - 1 - warp;
#pragma unroll 1
    for (int i = tid; i < mapw / 2; i += NT)
        reinterpret_cast<uint4*>(bm1)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (is_tg) {
        const uint32_t h = cg_hash(static_cast<uint32_t>(tg_row), hb);
        atomicOr(&bm1[h >> 5], 1u << (h & 31));
        atomicOr(&bm2[h >> 5], 1u << (h & 31));
    }
    // ---- pass 1: four columns a warp at a time, eight lanes each, four rows a
    // lane in flight and the next four columns' rows on their way
    const int grp = lane >> 3, l8 = lane & 7;
    auto column_of = [&](int c0, int& len, uint32_t& at) {
        const int ci = c0 + grp;
        len = ci < n ? static_cast<int>(clen[ci]) : 0;
        at = ci < n ? cb[ci] : 0u;
    };
    auto load_rows = [&](int len, uint32_t at, int o, int (&r)[4]) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int e = o + 8 * q + l8;
            r[q] = e < len ? __ldg(pb.cidx + at + e) : -1;
        }
    };
    {
        auto mark = [&](const int (&r)[4], int left) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (8 * q < left && r[q] >= 0) {
                    const uint32_t h = cg_hash(static_cast<uint32_t>(r[q]), hb);
                    const uint32_t bit = 1u << (h & 31);
                    if (atomicOr(&bm1[h >> 5], bit) & bit)
                        atomicOr(&bm2[h >> 5], bit);
                }
            }
        };
        int len, rn[4];
        uint32_t at;
        column_of(4 * warp, len, at);
        load_rows(len, at, 0, rn);
        __syncthreads();  // the target rows' bits are set
        for (int c0 = 4 * warp; c0 < n; c0 += 4 * NW) {
            int r[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
                r[q] = rn[q];
            const int most = __reduce_max_sync(kNone, len);
            const int len0 = len;
            const uint32_t at0 = at;
            column_of(c0 + 4 * NW, len, at);
            load_rows(len, at, 0, rn);
            mark(r, most);
            for (int o = 32; o < most; o += 32) {
                load_rows(len0, at0, o, r);
                mark(r, most - o);
            }
        }
    }
    __syncthreads();
    // ---- pass 2: squares of the entries alone in their row, candidates
    int nc = 0;
    {
        auto load_values = [&](int len, uint32_t at, int o, double (&v)[4]) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int e = o + 8 * q + l8;
                v[q] = e < len ? __ldg(pb.cval + at + e) : 0.0;
            }
        };
        double s0, s1;
        auto split = [&](const int (&r)[4], const double (&v)[4], int ci, int o, int left) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (8 * q >= left)
                    break;
                bool f = false;
                if (r[q] >= 0) {
                    const uint32_t h = cg_hash(static_cast<uint32_t>(r[q]), hb);
                    f = (bm2[h >> 5] >> (h & 31)) & 1u;
                }
                if (f)
                    s1 += v[q] * v[q];
                else
                    s0 += v[q] * v[q];
                const uint32_t b = __ballot_sync(kNone, f);
                const int c = nc + __popc(b & lt);
                if (f && 8 * NW * (c + 1) <= room)
                    cand[-NW * c] = make_uint2(static_cast<uint32_t>(r[q]),
                                               (static_cast<uint32_t>(ci) << 16) |
                                                   static_cast<uint32_t>(o + 8 * q + l8));
                nc += __popc(b);
            }
        };
        int len, rn[4];
        uint32_t at;
        double vn[4];
        column_of(4 * warp, len, at);
        load_rows(len, at, 0, rn);
        load_values(len, at, 0, vn);
        for (int c0 = 4 * warp; c0 < n; c0 += 4 * NW) {
            int r[4];
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                r[q] = rn[q];
                v[q] = vn[q];
            }
            const int most = __reduce_max_sync(kNone, len);
            const int len0 = len;
            const uint32_t at0 = at;
            column_of(c0 + 4 * NW, len, at);
            load_rows(len, at, 0, rn);
            load_values(len, at, 0, vn);
            s0 = s1 = 0.0;
            const int ci = c0 + grp;
            split(r, v, ci, 0, most);
            for (int o = 32; o < most; o += 32) {
                load_rows(len0, at0, o, r);
                load_values(len0, at0, o, v);
                split(r, v, ci, o, most - o);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                s0 += __shfl_xor_sync(kNone, s0, o);
                s1 += __shfl_xor_sync(kNone, s1, o);
            }
            if (l8 == 0 && ci < n) {
                d0[ci] = s0;
                gd[ci] = s0 + s1;
            }
        }
        if (lane == 0)
            sh.ncw[warp] = nc;
    }
    __syncthreads();
    int ncmax = 0, nctot = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) {
        ncmax = max(ncmax, sh.ncw[w]);
        nctot += sh.ncw[w];
    }
    // ---- candidates grouped by row: exact hash table (keys, counts by warp)
    const int ht = max(64, next_pow2(nctot + nctot / 2));
    const int htb = 31 - __clz(ht);
    const int smax = nctot / 2 + kCgMaxTargets;  // bound of the shared rows
    const int top = (cap - 8 * NW * ncmax - 8 * smax) & ~7;
    uint32_t* key = reinterpret_cast<uint32_t*>(base + ra);
    uint32_t* cnt = key + ht;
    uint32_t* rcnt = reinterpret_cast<uint32_t*>(base + top);  // entries by warp of a row
    uint32_t* rfill = rcnt + smax;
    // the candidates beside the bit maps, then beside the table and the rows' counts
    const int need = ra + 8 * NW * ncmax + max(8 * mapw, 8 * ht + 8 * smax);
    if (8 * NW * ncmax > room || 8 * ht > top - ra)
        return need > widest ? Taken::kNo : Taken::kLarger;
#pragma unroll 1
    for (int i = tid; i < ht / 4; i += NT) {
        reinterpret_cast<uint4*>(key)[i] = make_uint4(kNone, kNone, kNone, kNone);
        reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
    }
#pragma unroll 1
    for (int i = tid; i < smax; i += NT)
        rfill[i] = 0;
#pragma unroll 1
    for (int i = tid; i < n; i += NT)
        clen[i] = 0;
    for (int i = tid; i <= kCgMaxLen; i += NT)
        sh.bins[i] = 0;
    __syncthreads();
    int distinct = 0;
#pragma unroll 1
    for (int i = 0; i < nc; i += 32) {
        const int c = i + lane;
        bool mine = false;
        if (c < nc) {
            const uint32_t row = cand[-NW * c].x;
            uint32_t s = cg_hash(row, htb);
            while (true) {
                const uint32_t old = atomicCAS(&key[s], kNone, row);
                mine = old == kNone;
                if (mine || old == row)
                    break;
                s = (s + 1) & (ht - 1);
            }
            atomicAdd(&cnt[s], 1u << (8 * warp));
            cand[-NW * c].x = s | (mine ? kFirst : 0u);
        }
        distinct += __popc(__ballot_sync(kNone, mine));
    }
    if (lane == 0)
        atomicAdd(&sh.distinct, distinct);
    __syncthreads();
    // the rows of the target stay, whatever their length
    uint32_t tg_slot = kNone;
    if (is_tg) {
        uint32_t s = cg_hash(static_cast<uint32_t>(tg_row), htb);
        while (key[s] != kNone && key[s] != static_cast<uint32_t>(tg_row))
            s = (s + 1) & (ht - 1);
        if (key[s] != kNone) {
            tg_slot = s;
            cnt[s] |= kFirst;
        }
    }
    __syncthreads();
    // rows by decreasing length: their numbers, none for single entries
#pragma unroll 1
    for (int c = lane; c < nc; c += 32) {
        const uint32_t x = cand[-NW * c].x;
        if (x & kFirst) {
            const uint32_t pk = cnt[x & ~kFirst], k = cg_count(pk);
            if (k > kCgMaxLen)
                sh.over = 1;
            else if (k >= 2 || (pk & kFirst))
                atomicAdd(&sh.bins[k], 1u);
        }
    }
    __syncthreads();
    if (sh.over)
        return Taken::kNo;
    if (warp == 0) {
        const uint32_t rows = cg_order(sh.bins, sh.rows, lane);
        if (lane == 0)
            sh.nrows = static_cast<int>(rows);
    }
    __syncthreads();
    const int S = sh.nrows;
#pragma unroll 1
    for (int c = lane; c < nc; c += 32) {
        const uint32_t x = cand[-NW * c].x;
        if (x & kFirst) {
            const uint32_t s = x & ~kFirst;
            const uint32_t pk = cnt[s], k = cg_count(pk);
            uint32_t rid = kNone;
            if (k >= 2 || (pk & kFirst)) {
                rid = atomicAdd(&sh.bins[k], 1u);
                rcnt[rid] = pk & ~kFirst;
            }
            key[s] = rid;
        }
    }
    __syncthreads();
    int tg_rid = -1;
    if (tg_slot != kNone)
        tg_rid = static_cast<int>(key[tg_slot]);
    {
        int ns = 0;
#pragma unroll 1
        for (int c = lane; c < nc; c += 32) {
            const uint2 x = cand[-NW * c];
            const uint32_t rid = key[x.x & ~kFirst];
            cand[-NW * c].x = rid;
            if (rid != kNone) {
                atomicAdd(&clen[x.y >> 16], 1u);
                ns++;
            }
        }
        ns = __reduce_add_sync(kNone, ns);
        if (lane == 0)
            atomicAdd(&sh.shared_entries, ns);
    }
    for (int i = tid; i <= kCgMaxLen; i += NT)
        sh.bins[i] = 0;
    if (tid == 0)
        sh.over = 0;
    __syncthreads();
    // columns by decreasing number of shared entries
#pragma unroll 1
    for (int i = tid; i < n; i += NT) {
        if (clen[i] > kCgMaxLen)
            sh.over = 1;
        else
            atomicAdd(&sh.bins[clen[i]], 1u);
    }
    __syncthreads();
    if (sh.over)
        return Taken::kNo;
    if (warp == 0) {
        cg_order(sh.bins, sh.cols, lane);
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const uint32_t b = i < n ? clen[i] : kNone;
            const uint32_t m = __match_any_sync(kNone, b);
            const int rank = __popc(m & lt);
            uint32_t pos = 0;
            if (i < n) {
                pos = sh.bins[b] + rank;
                cpos[i] = static_cast<uint16_t>(pos);
                ccol[pos] = static_cast<uint16_t>(i);
            }
            __syncwarp();
            if (i < n && rank == __popc(m) - 1)
                sh.bins[b] = pos + 1;
            __syncwarp();
        }
    }
    __syncthreads();
    // ---- the shared entries by row (ev, ec) and by column (cv, cr): entry q of
    // the rows longer than q side by side, in the rows' order
    const int ns = sh.shared_entries;
    double* ev = reinterpret_cast<double*>(base + ra);
    double* cv = ev + ns;
    double* y = cv + ns;
    uint16_t* ec = reinterpret_cast<uint16_t*>(y + S);
    uint16_t* cr = ec + ns;
    if (20 * ns + 8 * S > top - ra || ns > 0xffff)
        return 20 * ns + 8 * S > top - ra + widest - cap || ns > 0xffff ? Taken::kNo
                                                                        : Taken::kLarger;
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < n; i += NT)
        us[i] = 0.0;
    uint32_t* cfill = reinterpret_cast<uint32_t*>(us);
    __syncthreads();
#pragma unroll 1
    for (int i = 0; i < nc; i += 32) {
        const int c = i + lane;
        const bool have = c < nc;
        const uint2 x = have ? cand[-NW * c] : make_uint2(kNone, 0u);
        const bool real = have && x.x != kNone;
        const uint32_t jj = x.y >> 16;
        double v = 0.0;
        if (have)
            v = __ldg(pb.cval + cb[jj] + (x.y & 0xffffu));
        const uint32_t other = 0x40000000u | lane;
        const uint32_t m1 = __match_any_sync(kNone, real ? x.x : other);
        const uint32_t m2 = __match_any_sync(kNone, have ? (jj | (real ? 0x10000u : 0u)) : other);
        const int rank1 = __popc(m1 & lt), rank2 = __popc(m2 & lt);
        uint32_t q1 = 0, q2 = 0;
        const uint32_t pos = have ? cpos[jj] : 0u;
        if (real) {
            // the row's entries of the warps before this one, then this warp's
            const uint32_t before = rcnt[x.x] & ((1u << (8 * warp)) - 1u);
            q1 = cg_count(before) + ((rfill[x.x] >> (8 * warp)) & 0xffu) + rank1;
            q2 = cfill[pos] + rank2;
        }
        __syncwarp();
        if (real) {
            if (rank1 == __popc(m1) - 1)
                atomicAdd(&rfill[x.x], static_cast<uint32_t>(rank1 + 1) << (8 * warp));
            if (rank2 == __popc(m2) - 1)
                cfill[pos] = q2 + 1;
            const int er = static_cast<int>((sh.rows[q1] >> 16) + x.x);
            ev[er] = v;
            ec[er] = static_cast<uint16_t>(pos);
            if (q1 == 0)
                cand[-NW * c].x = x.x | kFirst;
            const int eq = static_cast<int>((sh.cols[q2] >> 16) + pos);
            cv[eq] = v;
            cr[eq] = static_cast<uint16_t>(x.x);
        }
        // single entries after all: their squares, one a column at a time
        const bool alone = have && !real;
        const int rounds = __reduce_max_sync(kNone, alone ? rank2 + 1 : 0);
        for (int r = 0; r < rounds; r++) {
            if (alone && rank2 == r)
                d0[jj] += v * v;
            __syncwarp();
        }
        // the next pass reads the counts that other lanes have written in this one
        __syncwarp();
    }
    __syncthreads();
    g.n = n;
    g.E = E;
    g.nc = nc;
    g.nctot = nctot;
    g.ns = ns;
    g.S = S;
    g.free_lo = static_cast<int>(reinterpret_cast<char*>(cr + ns) - base);
    g.free_hi = cap - 8 * NW * ncmax;
    g.p0 = p0;
    g.d0 = d0;
    g.gd = gd;
    g.us = us;
    g.xs = xs;
    g.cb = cb;
    g.tmp = clen;
    g.cpos = cpos;
    g.ccol = ccol;
    g.ev = ev;
    g.ec = ec;
    g.cv = cv;
    g.cr = cr;
    g.y = y;
    g.cand = cand;
    g.tg_rid = tg_rid;
    g.tg_val = tg_val;
    return Taken::kYes;
}

}  // namespace mspai
