// Kernels of the batched MSPAI setup and their launchers.
//
//   plan_kernel      per column: |J_k| and the number of entries of C(:, J_k)
//                    (the size that decides the bucket), warp per column
//   bucket_kernel    size-binned work lists (atomic append per bucket) and
//                    per-bucket maxima of the sizes
//   warp_solve       one warp per column (spai_warp.cu)
//   cta_solve        one CTA per column from a work queue (persistent grid);
//                    the folded least-squares matrix lives in shared memory
//                    (W_SMEM) or in a per-CTA global scratch slot
//   compact_kernel   gathers per-column results into M's CSC arrays
//
// The column loop of the reference (src/Spai.imp:160-167 with
// Load_Balance::Grab_M_Col, src/Load_Balance.imp:33-69) becomes these work
// queues: an atomic counter per bucket hands out columns.
#include "spai_kernels.h"
#include "spai_solve.cuh"

#include <algorithm>
#include <cstdio>

namespace mspai {

#ifdef MSPAI_PHASE_TIMERS
extern "C" int mspai_profile_phase_cycles(unsigned long long* out, int reset)
{
    cudaMemcpyFromSymbol(out, g_phase_cycles, sizeof(unsigned long long) * 16);
    if (reset) {
        unsigned long long z[16] = {};
        cudaMemcpyToSymbol(g_phase_cycles, z, sizeof(z));
    }
    return 0;
}
#endif

// ------------------------------------------------------------------ planning
// Eight lanes per column: a stencil's pattern has five to 27 entries, and a warp
// per column left most lanes idle (1,048,576 columns of five entries: 177 us,
// eight lanes 88 us).
__global__ void plan_kernel(const int64_t* __restrict__ cptr, const int64_t* __restrict__ pptr,
                            const int32_t* __restrict__ pidx, int nprob, int bs,
                            int32_t* __restrict__ E, int32_t* __restrict__ nk)
{
    const int lane = threadIdx.x & 7;
    const int groups = (gridDim.x * blockDim.x) >> 3;
    const int first = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    for (int64_t base = 0; base < nprob; base += groups) {  // every lane of a warp takes part
        const int64_t col = base + first;
        int64_t a = 0, b = 0, e = 0;
        if (col < nprob) {
            a = pptr[col];
            b = pptr[col + 1];
        }
        for (int64_t p = a + lane; p < b; p += 8) {
            const int j = pidx[p];
            e += cptr[bs * j + bs] - cptr[bs * j];
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
            e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0 && col < nprob) {
            E[col] = static_cast<int32_t>(e > 0x7fffffff ? 0x7fffffff : e);
            nk[col] = static_cast<int32_t>((b - a) * bs);
        }
    }
}

// bucket ids: 0 warp (tiny), 1 CTA + shared-memory W, 2 CTA + global W (with a
// small_list: columns of the small QR instead), 3 small columns of the sparse solver
// A block bins kBinTile columns at a time: the places inside the tile are counted
// in shared memory, and the tile takes its places in the lists with one atomic
// per bucket (one atomic per column serialised on three addresses: 1.37 ms for
// 1,048,576 columns, 18 us now).
constexpr int kBinThreads = 256;
constexpr int kBinTile = 4 * kBinThreads;

__global__ void __launch_bounds__(kBinThreads)
    bucket_kernel(const int32_t* __restrict__ E, const int32_t* __restrict__ nk, int n,
                  BucketRule rule, int32_t* __restrict__ counts, int32_t* __restrict__ maxE,
                  int32_t* __restrict__ maxN, int32_t* __restrict__ lists)
{
    __shared__ int32_t tile_count[4], tile_base[4];
    const int lane = threadIdx.x & 31;
    int32_t top_e[4] = {0, 0, 0, 0}, top_n[4] = {0, 0, 0, 0};
    for (int64_t c0 = static_cast<int64_t>(blockIdx.x) * kBinTile; c0 < n;
         c0 += static_cast<int64_t>(gridDim.x) * kBinTile) {
        if (threadIdx.x < 4)
            tile_count[threadIdx.x] = 0;
        __syncthreads();
        int bucket[4], place[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t col = c0 + u * kBinThreads + threadIdx.x;
            int b = -1;
            if (col < n && col >= rule.lo && col < rule.hi &&  // the requested column range
                !(rule.rep && rule.rep[col] != col)) {         // solved by its representative
                // sizes after at most ns pattern updates
                const int64_t nf = static_cast<int64_t>(nk[col]) + rule.grow_n;
                const int64_t ef = static_cast<int64_t>(E[col]) + rule.grow_e;
                if (rule.small_list > 0 && ef <= kSmallE && nf <= kSmallN)
                    b = 2;
                else if (rule.single_bucket >= 0)
                    b = rule.single_bucket;
                else if (rule.allow_warp && ef <= rule.warp_emax && nf <= rule.warp_nmax)
                    b = 0;
                else if (rule.tiny_list > 0 && ef <= rule.tiny_emax && nf <= rule.tiny_nmax)
                    b = 3;
                else {
                    const int64_t mw = ef / 2 + nf;
                    const int64_t wbytes = (mw * nf + mw) * rule.elem_bytes;
                    b = (wbytes <= rule.smem_w_bytes) ? 1 : 2;
                }
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    if (b == x) {
                        top_e[x] = max(top_e[x], static_cast<int32_t>(
                                                     ef > 0x7fffffff ? 0x7fffffff : ef));
                        top_n[x] = max(top_n[x], static_cast<int32_t>(nf));
                    }
                }
            }
            bucket[u] = b;
            place[u] = 0;
#pragma unroll
            for (int x = 0; x < 4; x++) {
                const uint32_t m = __ballot_sync(0xffffffffu, b == x);
                if (m == 0)
                    continue;
                int base = 0;
                if (lane == __ffs(m) - 1)
                    base = atomicAdd(&tile_count[x], __popc(m));
                base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
                if (b == x)
                    place[u] = base + __popc(m & ((1u << lane) - 1u));
            }
        }
        __syncthreads();
        if (threadIdx.x < 4 && tile_count[threadIdx.x] > 0)
            tile_base[threadIdx.x] = atomicAdd(&counts[threadIdx.x], tile_count[threadIdx.x]);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int b = bucket[u];
            if (b < 0)
                continue;
            const int to =
                b == 3 ? rule.tiny_list : (b == 2 && rule.small_list > 0 ? rule.small_list : b);
            lists[static_cast<int64_t>(to) * n + tile_base[b] + place[u]] =
                static_cast<int32_t>(c0 + u * kBinThreads + threadIdx.x);
        }
        __syncthreads();
    }
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const int e = __reduce_max_sync(0xffffffffu, top_e[x]);
        const int m = __reduce_max_sync(0xffffffffu, top_n[x]);
        if (lane == 0 && (e > 0 || m > 0)) {
            atomicMax(&maxE[x], e);
            atomicMax(&maxN[x], m);
        }
    }
}

// ------------------------------------------------------------------ solvers
// The solver is latency bound: throughput grows with the columns in flight
// per SM.  MINB CTAs of 128 threads per SM bound the registers per thread
// (128 for 4, 64 for 8); the shared-memory area per CTA is chosen with it.
template <class T, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    cta_solve_kernel(Problem pb, Caps cap, Output out, const int32_t* __restrict__ list, int count,
                     int32_t* __restrict__ counter, char* __restrict__ scratch, size_t slot_bytes,
                     int wfast_elems, int blocked)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ GroupScratch sc;
    __shared__ BlockedScratch<T> bsc;
    CtaGroup<NT> g{&sc};
    SlotLayout<T> lay(cap, false);
    Slot<T> s = lay.at(scratch + static_cast<size_t>(blockIdx.x) * slot_bytes, nullptr);
    s.Wfast = wfast_elems > 0 ? reinterpret_cast<T*>(smem) : nullptr;
    s.wfast_elems = wfast_elems;
    s.bsc = blocked ? &bsc : nullptr;
    while (true) {
        if (threadIdx.x == 0)
            sc.i[5] = atomicAdd(counter, 1);
        __syncthreads();
        const int t = sc.i[5];
        __syncthreads();
        if (t >= count)
            break;
        solve_column<T>(g, pb, cap, s, out, list[t]);
    }
}

// ------------------------------------------------------------------ assembly
__global__ void compact_kernel(const int64_t* __restrict__ cap_ptr, const int32_t* __restrict__ cidx,
                               const double* __restrict__ cval, const int64_t* __restrict__ out_ptr,
                               int32_t* __restrict__ oidx, double* __restrict__ oval, int n)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int col = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; col < n; col += warps) {
        const int64_t a = cap_ptr[col];
        const int64_t o = out_ptr[col];
        const int len = static_cast<int>(out_ptr[col + 1] - o);
        for (int t = lane; t < len; t += 32) {
            oidx[o + t] = cidx[a + t];
            oval[o + t] = cval[a + t];
        }
    }
}

// exclusive scan of int32 lengths into int64 pointers (3-phase, device-wide)
__global__ void scan_blocks_kernel(const int32_t* __restrict__ len, int n, int64_t* __restrict__ out,
                                   int64_t* __restrict__ block_sums)
{
    __shared__ int64_t sh[1024];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t v = (i < n) ? len[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < blockDim.x; o <<= 1) {
        int64_t t = (threadIdx.x >= o) ? sh[threadIdx.x - o] : 0;
        __syncthreads();
        sh[threadIdx.x] += t;
        __syncthreads();
    }
    if (i < n)
        out[i] = sh[threadIdx.x] - v;
    if (threadIdx.x == blockDim.x - 1)
        block_sums[blockIdx.x] = sh[threadIdx.x];
}

__global__ void scan_add_kernel(int64_t* __restrict__ out, int n, const int64_t* __restrict__ block_off)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] += block_off[blockIdx.x];
}

// Exclusive scan of the block sums by one CTA, 1024 at a time (one thread took
// 25 us for the 192 sums of 192,000 columns).
__global__ void __launch_bounds__(1024) scan_sums_kernel(int64_t* __restrict__ v, int nb)
{
    __shared__ int64_t part[32];
    __shared__ int64_t carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        const int64_t own = i < nb ? v[i] : 0;
        int64_t s = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o)
                s += t;
        }
        if (lane == 31)
            part[warp] = s;
        __syncthreads();
        if (warp == 0) {
            const int64_t p = part[lane];
            int64_t q = p;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(0xffffffffu, q, o);
                if (lane >= o)
                    q += t;
            }
            part[lane] = q - p;
        }
        __syncthreads();
        const int64_t before = carry + part[warp] + s - own;
        if (i < nb)
            v[i] = before;
        __syncthreads();
        if (threadIdx.x == 1023)
            carry = before + own;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        v[nb] = carry;
}

__global__ void finish_ptr_kernel(int64_t* __restrict__ ptr, int n, const int32_t* __restrict__ len)
{
    // ptr[n] = ptr[n-1] + len[n-1]
    if (blockIdx.x == 0 && threadIdx.x == 0)
        ptr[n] = (n > 0) ? ptr[n - 1] + len[n - 1] : 0;
}

// entries of a packed triangle of |P(:, k)|: n_k (n_k + 1) / 2
// Order-independent 64-bit digest of a CSC structure: the wrapping sum of a
// mix of (position, value) over the column pointers and the row indices, so
// that the result does not depend on the launch shape or the order of the
// atomic adds.
__device__ __forceinline__ unsigned long long struct_mix(unsigned long long v)
{
    // SplitMix64 finaliser
    v += 0x9e3779b97f4a7c15ull;
    v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ull;
    v = (v ^ (v >> 27)) * 0x94d049bb133111ebull;
    return v ^ (v >> 31);
}

__global__ void structure_hash_kernel(const int64_t* __restrict__ ptr,
                                      const int32_t* __restrict__ idx, int ncols, int64_t nnz,
                                      unsigned long long salt, unsigned long long* acc)
{
    unsigned long long part = 0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i <= ncols;
         i += stride)
        part += struct_mix(salt ^ (static_cast<unsigned long long>(i) << 1) ^
                           (static_cast<unsigned long long>(ptr[i]) * 0x100000001b3ull));
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nnz;
         i += stride)
        part += struct_mix(~salt ^ (static_cast<unsigned long long>(i) << 1) ^
                           (static_cast<unsigned long long>(static_cast<uint32_t>(idx[i])) << 33));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0)
        atomicAdd(acc, part);
}

cudaError_t launch_structure_hash(const int64_t* ptr, const int32_t* idx, int ncols, int64_t nnz,
                                  unsigned long long salt, unsigned long long* acc,
                                  cudaStream_t st)
{
    const int blocks = std::max(1, std::min<int>(num_sms() * 8,
                                                 static_cast<int>((nnz + ncols + 255) / 256)));
    structure_hash_kernel<<<blocks, 256, 0, st>>>(ptr, idx, ncols, nnz, salt, acc);
    return cudaGetLastError();
}

__global__ void tri_len_kernel(const int64_t* __restrict__ pptr, int n, int32_t* __restrict__ len)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int64_t nk = pptr[k + 1] - pptr[k];
        len[k] = static_cast<int32_t>(nk * (nk + 1) / 2);
    }
}

cudaError_t launch_tri_len(const int64_t* pptr, int n, int32_t* len, cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    int blocks = std::min((n + 255) / 256, num_sms() * 8);
    tri_len_kernel<<<blocks, 256, 0, st>>>(pptr, n, len);
    return cudaGetLastError();
}

// capacity of scalar column sc: bs * (|P(:, sc / bs)| + grow) entries
__global__ void capacity_len_kernel(const int64_t* __restrict__ pptr, int n, int bs, int grow,
                                    int32_t* __restrict__ len)
{
    for (int sc = blockIdx.x * blockDim.x + threadIdx.x; sc < n; sc += gridDim.x * blockDim.x) {
        const int kb = sc / bs;
        len[sc] = static_cast<int32_t>((pptr[kb + 1] - pptr[kb] + grow) * bs);
    }
}

__global__ void max_len_kernel(const int64_t* __restrict__ ptr, int n, int32_t* __restrict__ out)
{
    int m = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = max(m, static_cast<int>(ptr[i + 1] - ptr[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0)
        atomicMax(out, m);
}

// ------------------------------------------------------------------ input checks
// First error found in a CSC structure: err[0] = kind (1 pointers do not match
// nnz, 2 pointers decrease, 3 row out of range, 4 rows not sorted/unique,
// 5 empty column), err[1] = column, err[2] = row.  Pointers are checked
// before any entry of their column is read.
__global__ void validate_csc_kernel(const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                    int ncols, int nrows, int64_t nnz, int nonempty,
                                    int32_t* __restrict__ err)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    auto report = [&](int kind, int c, int r) {
        if (atomicCAS(err, 0, kind) == 0) {
            err[1] = c;
            err[2] = r;
        }
    };
    if (tid == 0 && (ptr[0] != 0 || ptr[ncols] != nnz))
        report(1, -1, 0);
    for (int c = tid; c < ncols; c += gridDim.x * blockDim.x) {
        const int64_t a = ptr[c], b = ptr[c + 1];
        if (a < 0 || b > nnz || b < a) {
            report(b < a ? 2 : 1, c, 0);
            continue;
        }
        if (nonempty && a == b)
            report(5, c, 0);
        int prev = -1;
        for (int64_t p = a; p < b; p++) {
            const int r = idx[p];
            if (r < 0 || r >= nrows) {
                report(3, c, r);
                break;
            }
            if (r <= prev) {
                report(4, c, r);
                break;
            }
            prev = r;
        }
    }
}

// ------------------------------------------------------------------ launchers
namespace {
int g_num_sms = 0;
}  // namespace

int num_sms()
{
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_num_sms <= 0)
            g_num_sms = 1;
    }
    return g_num_sms;
}

cudaError_t launch_validate_csc(const int64_t* ptr, const int32_t* idx, int ncols, int nrows,
                                int64_t nnz, bool nonempty, int32_t* err, cudaStream_t st)
{
    const int blocks = std::max(1, std::min((ncols + 255) / 256, num_sms() * 8));
    validate_csc_kernel<<<blocks, 256, 0, st>>>(ptr, idx, ncols, nrows, nnz, nonempty ? 1 : 0,
                                                err);
    return cudaGetLastError();
}

cudaError_t launch_plan(const int64_t* cptr, const int64_t* pptr, const int32_t* pidx, int nprob,
                        int bs, int32_t* E, int32_t* nk, cudaStream_t st)
{
    if (nprob <= 0)
        return cudaSuccess;
    const int threads = 256;
    int blocks = (nprob + 31) / 32;
    blocks = std::min(blocks, num_sms() * 8);
    plan_kernel<<<blocks, threads, 0, st>>>(cptr, pptr, pidx, nprob, bs, E, nk);
    return cudaGetLastError();
}

cudaError_t launch_bucket(const int32_t* E, const int32_t* nk, int n, const BucketRule& rule,
                          int32_t* counts, int32_t* maxE, int32_t* maxN, int32_t* lists,
                          cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    int blocks = std::min((n + kBinTile - 1) / kBinTile, num_sms() * 4);
    bucket_kernel<<<blocks, kBinThreads, 0, st>>>(E, nk, n, rule, counts, maxE, maxN, lists);
    return cudaGetLastError();
}

size_t warp_slot_bytes(const Caps& cap, int elem_bytes)
{
    if (elem_bytes == 4)
        return SlotLayout<float>(cap, false).bytes;
    return SlotLayout<double>(cap, false).bytes;
}

size_t cta_slot_bytes(const Caps& cap, int elem_bytes, bool w_smem)
{
    if (elem_bytes == 4)
        return SlotLayout<float>(cap, w_smem).bytes;
    return SlotLayout<double>(cap, w_smem).bytes;
}

size_t w_bytes(const Caps& cap, int elem_bytes)
{
    return static_cast<size_t>(cap.mwmax) * (cap.nmax + std::max(1, cap.nrhs)) * elem_bytes;
}

template <class T, int NT, int MINB>
static cudaError_t launch_cta_t(const Problem& pb, const Caps& cap, const Output& out,
                                const int32_t* list, int count, int32_t* counter, char* scratch,
                                size_t scratch_bytes, size_t smem, int blocked, cudaStream_t st,
                                int* grid_out)
{
    const size_t slot = SlotLayout<T>(cap, false).bytes;
    cudaError_t e = cudaFuncSetAttribute(cta_solve_kernel<T, NT, MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cta_solve_kernel<T, NT, MINB>, NT,
                                                      smem);
    if (e != cudaSuccess)
        return e;
    if (per_sm < 1)
        return cudaErrorInvalidConfiguration;
    int grid = std::min(per_sm, MINB) * num_sms();
    grid = std::max(1, std::min(grid, count));
    const size_t slots_fit = slot > 0 ? scratch_bytes / slot : 0;
    if (slots_fit < 1)
        return cudaErrorMemoryAllocation;
    grid = static_cast<int>(std::min<size_t>(grid, slots_fit));
    *grid_out = grid;
    const int wfast = static_cast<int>(smem / sizeof(T));
    cta_solve_kernel<T, NT, MINB><<<grid, NT, smem, st>>>(pb, cap, out, list, count, counter,
                                                          scratch, slot, wfast, blocked);
    return cudaGetLastError();
}

cudaError_t launch_cta_solve(int elem_bytes, size_t smem_w_bytes, bool blocked,
                             const Problem& pb, const Caps& cap, const Output& out,
                             const int32_t* list, int count, int32_t* counter, char* scratch,
                             size_t scratch_bytes, cudaStream_t st, int* grid_out)
{
    const int per_sm = cta_per_sm(elem_bytes, smem_w_bytes);
    if (elem_bytes == 4) {
        if (per_sm == 8)
            return launch_cta_t<float, 128, 8>(pb, cap, out, list, count, counter, scratch,
                                               scratch_bytes, smem_w_bytes, blocked ? 1 : 0, st,
                                               grid_out);
        if (per_sm == 6)
            return launch_cta_t<float, 128, 6>(pb, cap, out, list, count, counter, scratch,
                                               scratch_bytes, smem_w_bytes, blocked ? 1 : 0, st,
                                               grid_out);
        return launch_cta_t<float, 128, 4>(pb, cap, out, list, count, counter, scratch,
                                           scratch_bytes, smem_w_bytes, blocked ? 1 : 0, st,
                                           grid_out);
    }
    return launch_cta_t<double, 128, 4>(pb, cap, out, list, count, counter, scratch,
                                        scratch_bytes, smem_w_bytes, blocked ? 1 : 0, st,
                                        grid_out);
}

int cta_per_sm(int elem_bytes, size_t smem_w_bytes)
{
    if (elem_bytes != 4)
        return 4;
    if (smem_w_bytes <= 24 * 1024)
        return 8;
    if (smem_w_bytes <= 32 * 1024)
        return 6;
    return 4;
}

size_t cta_scratch_needed(int elem_bytes, const Caps& cap, int count, size_t smem_w_bytes)
{
    const size_t slot = cta_slot_bytes(cap, elem_bytes, false);
    const size_t slots =
        static_cast<size_t>(std::min(count, cta_per_sm(elem_bytes, smem_w_bytes) * num_sms()));
    return slot * std::max<size_t>(slots, 1);
}

cudaError_t launch_scan_lengths(const int32_t* len, int n, int64_t* ptr, int64_t* tmp,
                                cudaStream_t st)
{
    // ptr has n+1 entries; tmp has >= nb + 1 entries
    if (n <= 0) {
        return cudaMemsetAsync(ptr, 0, sizeof(int64_t), st);
    }
    const int bs = 1024;
    const int nb = (n + bs - 1) / bs;
    scan_blocks_kernel<<<nb, bs, 0, st>>>(len, n, ptr, tmp);
    scan_sums_kernel<<<1, 1024, 0, st>>>(tmp, nb);
    scan_add_kernel<<<nb, bs, 0, st>>>(ptr, n, tmp);
    finish_ptr_kernel<<<1, 1, 0, st>>>(ptr, n, len);
    return cudaGetLastError();
}

cudaError_t launch_capacity_len(const int64_t* pptr, int n, int bs, int grow, int32_t* len,
                                cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    int blocks = std::min((n + 255) / 256, num_sms() * 8);
    capacity_len_kernel<<<blocks, 256, 0, st>>>(pptr, n, bs, grow, len);
    return cudaGetLastError();
}

cudaError_t launch_compact(const int64_t* cap_ptr, const int32_t* cidx, const double* cval,
                           const int64_t* out_ptr, int32_t* oidx, double* oval, int n,
                           cudaStream_t st)
{
    if (n <= 0)
        return cudaSuccess;
    int blocks = std::min((n + 7) / 8, num_sms() * 16);
    compact_kernel<<<blocks, 256, 0, st>>>(cap_ptr, cidx, cval, out_ptr, oidx, oval, n);
    return cudaGetLastError();
}

cudaError_t launch_max_len(const int64_t* ptr, int n, int32_t* out, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(int32_t), st);
    if (e != cudaSuccess || n <= 0)
        return e;
    int blocks = std::min((n + 255) / 256, num_sms() * 8);
    max_len_kernel<<<blocks, 256, 0, st>>>(ptr, n, out);
    return cudaGetLastError();
}

}  // namespace mspai
