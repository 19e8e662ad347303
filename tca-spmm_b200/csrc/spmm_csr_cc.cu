// spmm_csr_cc.cu -- CSR x dense SpMM on CUDA cores.
//
// C[r, :] = alpha * sum_j val_j * B[col_j, :] + beta * C[r, :], FP32 accumulation.
// This restates the computation of kernel_our_spmm_balanced
// (src/our_spmm.cu:290-346) without its host-built warp schedule and without
// using mma.sync as a dot-product engine.
//
// Kernels:
//   * spmm_rows_kernel: straight from a CSR, blocks of consecutive rows whose
//     nonzeros are cut into equal runs -- the plan-free forward
//     (tca_spmm_csr), and planned forwards whose dense operands are not
//     16-byte aligned;
//   * planned (tca_spmm / tca_spmm_batched): warps stream through work items
//     of consecutive sorted rows of one or many plans (spmm_cc_stream_kernel,
//     below), or compute them as small mma.sync products (spmm_cc_mma_kernel,
//     an autotuner candidate for FP16).
//
// Malformed CSR never faults: row ranges are clamped to [0, nnz] and
// nonzeros whose column is outside [0, K) contribute nothing.
#include <algorithm>
#include <climits>
#include <memory>
#include <vector>
#include <cuda_fp8.h>
#include "tca_internal.cuh"
#include "plan.cuh"
#include "ptx.cuh"

namespace tca {
namespace {

__device__ __forceinline__ void load8(const __half *p, float *v)
{
    uint4 u = *reinterpret_cast<const uint4 *>(p);
    const __half2 *h = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float2 f = __half22float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ void load8(const float *p, float *v)
{
    float4 a = reinterpret_cast<const float4 *>(p)[0];
    float4 b = reinterpret_cast<const float4 *>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(__half *p, const float *v)
{
    uint4 u;
    __half2 *h = reinterpret_cast<__half2 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4 *>(p) = u;
}
__device__ __forceinline__ void store8(float *p, const float *v)
{
    reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

template <typename T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float to_f<float>(float x) { return x; }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }

__device__ __forceinline__ void clamp_range(int &start, int &end, int nnz)
{
    start = max(0, min(start, nnz));
    end = max(start, min(end, nnz));
}

constexpr int kMaxCcJobs = 32;

// ---------------------------------------------------------------------------
// Rows straight from a CSR: the caller's (plan-free) or a plan's re-ordered
// one when the dense operands do not allow 16-byte accesses.
//
// A row of a skewed matrix can hold every column (one group of lanes walking
// 1024 nonzeros took 120 us), so no row belongs to one group. Block b takes
// the rows whose key row_ptr[r] + w * r lies in the b-th of equal parts (found by a
// 32-way search: rows and nonzeros are both balanced, whatever the order of
// the rows) and cuts their nonzeros, laid end to end, into equal runs, one per
// group of LPR lanes. A group writes the rows that lie in its run; of a row
// that began before its run it leaves the partial sum in shared memory, and
// the group in which the row began adds those in run order (a fixed order) and
// writes it. What bounds it is the gather of B rows from L2, U of them in
// flight per lane.
// Malformed CSR: rows are clamped to [0, nnz] one by one and indices are
// checked, as everywhere in this file.
// ---------------------------------------------------------------------------
constexpr int kRowsThreads = 512;
// A row's weight beside a nonzero's in the cut: sorted rows lie with others of
// their length, so by nonzeros alone the last blocks hold hundreds of short
// rows, whose writes and offsets cost more than their nonzeros (2048 x 2048,
// Zipf rows of 5 %, N = 301: 113 us, 61 with weight 4, 49 with 8; 4096 x 1024
// at 20 %, N = 201: 113, 85, 79, and 78 with 16). In the caller's order long
// and short rows mix and the weight gives as often as it takes (1024 x 1024,
// N = 256: 33 -> 27 us; 1500 x 900, N = 301: 48 -> 56).
constexpr long long kSortedRowKey = 8;
// U nonzeros that lie in one row and whose columns are valid, as almost all do,
// need neither predicates nor zeros for absent loads (54 warp instructions per
// nonzero without this path; 4096 x 4096 at 95 %, N = 512: 118 -> 82 us; 4096 x 1024
// at 80 %, Zipf, N = 256: 73 -> 53 us, 8.1 TB/s of B rows from L2; 3001 x 1777, N =
// 203: 40 -> 29 us). Groups of fewer lanes meet too many row ends side by side
// in a warp, which then runs both paths (300 x 4096, N = 32: 23.4 us without, 27.8
// with), and so do groups of 16 lanes where rows are short on average, from about
// kFastMean on less than it gives (4096 x 1024 at 5 %, Zipf, 51 per row, N = 128:
// 24.4 without, 25.0 with; equal rows of 40, 16000 x 2000, N = 96: 25.2 without,
// 22.4 with, of 60 38.5 and 32.4; 4096 x 4096 at 90 %, N = 99: 76 and 58).
constexpr int kFastLpr = 16, kFastMean = 32;
constexpr int kRowsMax = kRowsThreads; // rows in shared memory at a time: a thread each
// Positions of those rows' nonzeros, laid end to end, are 32-bit numbers.
// Offsets that are not increasing can make rows overlap, so that 512 of them
// hold more than that: the rows taken at a time end where the next one would
// pass this many (two groups' lanes below the largest int, as positions are
// looked at that far ahead).
constexpr int kRowsNnz = 0x7fffffff - 64;

struct RowsJob {
    const int *row_ptr, *col;
    const int *perm; // row i of the CSR -> row of C; NULL: itself
    const __half *val, *B;
    void *C;
    int M, K, nnz, N, ldb, ldc;
    int base;     // row_ptr[0]: the rows may be a part of a CSR
    int n_blocks; // blocks per N-slice
    float alpha, beta;
    unsigned flags;
};
template <int CAP> struct RowsBatchT {
    int n_jobs;
    int block_start[CAP + 1];
    RowsJob job[CAP];
};

// W output columns per lane of a group of LPR lanes. VEC: 8 consecutive ones,
// B read in 16-byte accesses (16-byte aligned rows of at least N rounded up to
// 8 columns), C written so too with VC (N % 8 == 0, 16-byte aligned rows);
// else every LPR-th column.
template <typename OutT, int LPR, int W, bool VEC, bool VC, int CAP, bool FAST>
__global__ void __launch_bounds__(kRowsThreads, 2) spmm_rows_kernel(const __grid_constant__ RowsBatchT<CAP> batch)
{
    static_assert(!VEC || W == 8, "16-byte accesses cover 8 columns");
    constexpr int G = kRowsThreads / LPR;
    constexpr int U = VEC ? 4 : W >= 8 ? 2 : W >= 4 ? 4 : 8; // nonzeros in flight per lane
    __shared__ int s_start[kRowsMax], s_pre[kRowsMax + 1], s_warp[kRowsThreads / 32], s_range[2];
    __shared__ __align__(16) float s_part[G * LPR * W];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & (LPR - 1), g = (int)threadIdx.x / LPR;
    const unsigned gmask = LPR == 32 ? 0xffffffffu : (((1u << LPR) - 1u) << (lane & ~(LPR - 1)));
    int jb = 0;
    while (jb + 1 < batch.n_jobs && batch.block_start[jb + 1] <= (int)blockIdx.x) jb++;
    const RowsJob &a = batch.job[jb];
    const int local = (int)blockIdx.x - batch.block_start[jb];
    const int slice = local / a.n_blocks, b = local - slice * a.n_blocks;

    const long long row_key = a.perm ? kSortedRowKey : 1;
    // this block's rows: each half of the threads finds the first row whose
    // key is at least its bound, kRowsThreads / 2 probes at a time
    {
        constexpr int kProbes = kRowsThreads / 2;
        const int half = (int)threadIdx.x / kProbes, p = (int)threadIdx.x % kProbes, part = b + half;
        const long long bound = ((long long)a.nnz - a.base + row_key * a.M) * part / a.n_blocks + a.base;
        int lo = 0, len = part == 0 ? 0 : a.M; // the row is in [lo, lo + len]
        if (part == a.n_blocks) {
            lo = a.M;
            len = 0;
        }
        while (__syncthreads_or(len > 0)) { // both halves take the same number of rounds
            // (unsigned: with nearly 2^31 rows the last probes' offsets pass the largest int)
            const unsigned step = ((unsigned)len + kProbes - 1) / kProbes, probe = (unsigned)p * step;
            if (p == 0) s_range[half] = kProbes; // probe p is row lo + p * step
            __syncthreads();
            if (probe < (unsigned)len) {
                const int r = lo + (int)probe;
                if ((long long)min(max(__ldg(a.row_ptr + r), 0), a.nnz) + row_key * r >= bound) atomicMin(&s_range[half], p);
            }
            __syncthreads();
            const unsigned first = (unsigned)s_range[half];
            if (len > 0) { // the row lies after probe first - 1 and not after probe first
                const int hi = lo + (int)min((unsigned)len, first * step);
                if (first > 0) lo += (int)((min(first, ((unsigned)len + step - 1) / step) - 1) * step) + 1;
                len = hi - lo;
            }
        }
        if (p == 0) s_range[half] = lo;
    }
    __syncthreads();
    const int row_end = s_range[1];
    for (int row0 = s_range[0], n_rows = 0; row0 < row_end; row0 += n_rows) {
    n_rows = min(kRowsMax, row_end - row0);
    { // the rows' starts and the prefix sums of their lengths
        int len = 0;
        if ((int)threadIdx.x < n_rows) {
            int st = __ldg(a.row_ptr + row0 + threadIdx.x), en = __ldg(a.row_ptr + row0 + threadIdx.x + 1);
            clamp_range(st, en, a.nnz);
            len = en - st;
            s_start[threadIdx.x] = st;
        }
        auto add = [](int x, int y) -> int { return (int)min((unsigned)x + (unsigned)y, 0x7fffffffu); }; // saturating
        int sum = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum = add(sum, v);
        }
        if (lane == 31) s_warp[warp] = sum;
        __syncthreads();
        int carry = 0;
        for (int k = 0; k < warp; k++) carry = add(carry, s_warp[k]);
        sum = add(carry, sum);
        if ((int)threadIdx.x < n_rows) s_pre[threadIdx.x + 1] = sum;
        if (threadIdx.x == 0) s_pre[0] = 0;
        n_rows = max(1, __syncthreads_count((int)threadIdx.x < n_rows && sum <= kRowsNnz));
    }
    const int total = s_pre[n_rows];
    // a valid CSR's rows follow one another: position v is nonzero first + v
    const int first = s_start[0];
    const bool dense = __syncthreads_and((int)threadIdx.x >= n_rows ||
                                         (unsigned)s_start[threadIdx.x] == (unsigned)first + (unsigned)s_pre[threadIdx.x]);
    auto run_start = [&](int k) -> int { return (int)((long long)total * k / G); };
    // the row that holds position v of the block's nonzeros: the last one starting at or before v
    auto row_of = [&](int v) -> int {
        int lo = 0, hi = n_rows - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_pre[mid] <= v) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    };
    const int n0 = slice * (LPR * W) + (VEC ? sub * W : sub);
    auto col_ok = [&](int w) -> bool { return VEC ? n0 < a.N : n0 + w * LPR < a.N; };
    auto write = [&](int i, const float *acc) {
        const int r = row0 + i;
        OutT *cp = reinterpret_cast<OutT *>(a.C) + (size_t)(a.perm ? __ldg(a.perm + r) : r) * a.ldc + n0;
        if constexpr (VEC && !VC) {
#pragma unroll
            for (int w = 0; w < 8; w++) {
                if (n0 + w >= a.N)
                    continue;
                float o = a.alpha * acc[w];
                if (a.beta != 0.f) o = fmaf(a.beta, to_f<OutT>(cp[w]), o);
                cp[w] = from_f<OutT>(o);
            }
        } else if constexpr (VEC) {
            if (!col_ok(0))
                return;
            float o[8];
            if (a.beta != 0.f) {
                float old[8];
                load8(cp, old);
#pragma unroll
                for (int w = 0; w < 8; w++) o[w] = fmaf(a.alpha, acc[w], a.beta * old[w]);
            } else {
#pragma unroll
                for (int w = 0; w < 8; w++) o[w] = a.alpha * acc[w];
            }
            store8(cp, o);
        } else {
#pragma unroll
            for (int w = 0; w < W; w++) {
                if (!col_ok(w))
                    continue;
                float o = a.alpha * acc[w];
                if (a.beta != 0.f) o = fmaf(a.beta, to_f<OutT>(cp[w * LPR]), o);
                cp[w * LPR] = from_f<OutT>(o);
            }
        }
    };
    float *part = s_part + (g * LPR + sub) * W;
    auto leave = [&](const float *acc) {
#pragma unroll
        for (int w = 0; w < W; w++) part[w] = acc[w];
    };

    const int v0 = run_start(g), v1 = run_start(g + 1);
    float acc[W];
#pragma unroll
    for (int w = 0; w < W; w++) acc[w] = 0.f;
    int cr = 0, ce = 0;
    bool before = false, tail = false; // row cr began in an earlier run; goes on in a later one
    if (v0 < v1) {
        cr = row_of(v0);
        ce = s_pre[cr + 1];
        before = s_pre[cr] < v0;
        auto flush = [&](int v) { // row cr ends at v
            if (before) leave(acc);
            else write(cr, acc);
            before = false;
#pragma unroll
            for (int w = 0; w < W; w++) acc[w] = 0.f;
            do cr++; while (cr + 1 < n_rows && s_pre[cr + 1] <= v);
            ce = cr < n_rows ? s_pre[cr + 1] : 0x7fffffff;
        };
        const __half *Bn = a.B + n0;
        // lanes past N read the first columns instead; their sums go nowhere
        const char *Bs = reinterpret_cast<const char *>(a.B + (col_ok(0) ? n0 : 0));
        const unsigned ldb_bytes = 2u * (unsigned)a.ldb;
        // nonzero of this lane in the LPR from `base` on
        auto load_nz = [&](int base, int &c, unsigned short &x) {
            c = -1;
            x = 0;
            const int v = base + sub;
            if (v < v1) {
                int j = first + v;
                if (!dense) {
                    const int i = row_of(v);
                    j = s_start[i] + (v - s_pre[i]);
                }
                if (j >= 0 && j < a.nnz) {
                    c = __ldg(a.col + j);
                    x = __half_as_ushort(a.val[j]);
                    if (c < 0 || c >= a.K) { c = -1; x = 0; } // adds 0 * 0
                }
            }
        };
        int c, cn;
        unsigned short x, xn;
        load_nz(v0, cn, xn);
        for (int base = v0; base < v1; base += LPR) {
            c = cn;
            x = xn;
            load_nz(base + LPR, cn, xn);
            const int cnt = min(LPR, v1 - base);
            // no malformed columns: U nonzeros of one row take the short path
            const bool valid = FAST && !__any_sync(gmask, sub < cnt && c < 0);
            for (int t = 0; t < cnt; t += U) {
                if constexpr (FAST) {
                    if (valid && t + U <= cnt && base + t + U <= ce) {
                        uint4 bv[U];
                        unsigned short xf[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const unsigned cf = (unsigned)__shfl_sync(gmask, c, t + u, LPR);
                            xf[u] = (unsigned short)__shfl_sync(gmask, (int)x, t + u, LPR);
                            bv[u] = __ldg(reinterpret_cast<const uint4 *>(Bs + (unsigned long long)cf * ldb_bytes));
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const unsigned short *h = reinterpret_cast<const unsigned short *>(&bv[u]);
#pragma unroll
                            for (int w = 0; w < 8; w++) acc[w] = ptx::fma_f16_f32(xf[u], h[w], acc[w]);
                        }
                        continue;
                    }
                }
                int cu[U];
                unsigned short xu[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    cu[u] = __shfl_sync(gmask, c, (t + u) & (LPR - 1), LPR);
                    xu[u] = (unsigned short)__shfl_sync(gmask, (int)x, (t + u) & (LPR - 1), LPR);
                    if (t + u >= cnt) cu[u] = -1;
                }
                if constexpr (VEC) {
                    uint4 bv[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        bv[u] = make_uint4(0, 0, 0, 0);
                        if (cu[u] >= 0 && col_ok(0))
                            bv[u] = __ldg(reinterpret_cast<const uint4 *>(Bn + (size_t)cu[u] * a.ldb));
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (t + u < cnt) {
                            if (base + t + u >= ce) flush(base + t + u);
                            const unsigned short *h = reinterpret_cast<const unsigned short *>(&bv[u]);
#pragma unroll
                            for (int w = 0; w < 8; w++) acc[w] = ptx::fma_f16_f32(xu[u], h[w], acc[w]);
                        }
                    }
                } else {
                    unsigned short bv[U][W];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const __half *br = Bn + (size_t)max(cu[u], 0) * a.ldb;
#pragma unroll
                        for (int w = 0; w < W; w++)
                            bv[u][w] = cu[u] >= 0 && col_ok(w) ? __half_as_ushort(br[w * LPR]) : (unsigned short)0;
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (t + u < cnt) {
                            if (base + t + u >= ce) flush(base + t + u);
#pragma unroll
                            for (int w = 0; w < W; w++) acc[w] = ptx::fma_f16_f32(xu[u], bv[u][w], acc[w]);
                        }
                    }
                }
            }
        }
        // the run's last row
        if (ce <= v1) {
            if (before) leave(acc);
            else write(cr, acc);
        } else if (before) {
            leave(acc);
        } else {
            tail = true;
        }
    } else {
        leave(acc); // an empty run adds zero to a row that spans it
    }
    __syncthreads();
    if (tail) { // the row goes on in the next runs: add their parts in run order
        int k_end = g + 1;
        while (k_end < G && run_start(k_end) < ce) k_end++;
        const float *q = part;
#pragma unroll 4
        for (int k = g + 1; k < k_end; k++) {
            q += LPR * W;
#pragma unroll
            for (int w = 0; w < W; w++) acc[w] += q[w];
        }
        write(cr, acc);
    }
    if (!(a.flags & TCA_FLAG_KEEP_EMPTY_ROWS)) {
#pragma unroll
        for (int w = 0; w < W; w++) acc[w] = 0.f;
        for (int i = g; i < n_rows; i += G)
            if (s_pre[i] == s_pre[i + 1])
                write(i, acc);
    }
    __syncthreads(); // the next rows reuse shared memory
    }
    // beside a tensor-core launch: complete no earlier than it (as the stream kernel)
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Short rows on average (at most kShortMean nonzeros), plan-free, 16-byte
// accesses: a group of LPR lanes per row, so that a row costs four dependent
// loads and none of the balancing above (4096 x 1024 at 99 %, N = 128: 3.4 us
// against 8.3 us). The rows of more than kShortRow nonzeros wait until the
// block's other rows are done; then its groups are dealt to them in proportion
// to their lengths, at least one each, take equal runs of their row, and the
// row's first group adds the parts in run order. (All groups on one long row
// after the other pay barriers and a sum per row: 20000 x 110, Zipf rows of 12,
// N = 32, 58.7 us against 16.0; of 26, N = 256, 55.5 against 36.5; 16000 x 2000,
// one row of 90 among 50 of 1, N = 32, 22.7 against 7.2.) Block b takes rows b, b + gridDim.x, ..,
// so that neither sorted nor clustered long rows meet in one block. blockIdx.y:
// the slice of 8 LPR columns.
constexpr int kShortMean = 32, kShortRow = 64;

template <typename OutT, int LPR>
__global__ void __launch_bounds__(kRowsThreads, 2) spmm_rows_short_kernel(const RowsJob a)
{
    constexpr int G = kRowsThreads / LPR, U = 4;
    __shared__ __align__(16) float s_part[G * LPR * 8];
    __shared__ int s_row[G], s_beg[G], s_end[G], s_last[G], s_n; // the long rows; the group after each one's last
    const int lane = threadIdx.x & 31, sub = lane & (LPR - 1), g = (int)threadIdx.x / LPR;
    const unsigned gmask = LPR == 32 ? 0xffffffffu : (((1u << LPR) - 1u) << (lane & ~(LPR - 1)));
    const int n0 = (int)blockIdx.y * LPR * 8 + sub * 8;
    const bool active = n0 < a.N;
    const __half *Bn = a.B + n0;
    // lanes past N read the first columns instead; their sums go nowhere
    const char *Bs = reinterpret_cast<const char *>(a.B + (active ? n0 : 0));
    const unsigned ldb_bytes = 2u * (unsigned)a.ldb;
    if (threadIdx.x == 0)
        s_n = 0;
    __syncthreads();
    auto range = [&](int r, int &start, int &end) {
        start = __ldg(a.row_ptr + r);
        end = __ldg(a.row_ptr + r + 1);
        clamp_range(start, end, a.nnz);
    };
    // acc += the products of nonzeros [start, end), by this group
    auto run = [&](int start, int end, float *acc) {
        for (int base = start; base < end; base += LPR) {
            int c = -1;
            unsigned short x = 0;
            if (base + sub < end) {
                c = __ldg(a.col + base + sub);
                x = __half_as_ushort(a.val[base + sub]);
                if (c < 0 || c >= a.K) { c = -1; x = 0; }
            }
            const int cnt = min(LPR, end - base);
            const bool valid = LPR >= kFastLpr && !__any_sync(gmask, sub < cnt && c < 0); // no malformed columns
            for (int t = 0; t < cnt; t += U) {
                uint4 bv[U];
                if (valid && t + U <= cnt) {
                    unsigned short xf[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const unsigned cf = (unsigned)__shfl_sync(gmask, c, t + u, LPR);
                        xf[u] = (unsigned short)__shfl_sync(gmask, (int)x, t + u, LPR);
                        bv[u] = __ldg(reinterpret_cast<const uint4 *>(Bs + (unsigned long long)cf * ldb_bytes));
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const unsigned short *h = reinterpret_cast<const unsigned short *>(&bv[u]);
#pragma unroll
                        for (int w = 0; w < 8; w++) acc[w] = ptx::fma_f16_f32(xf[u], h[w], acc[w]);
                    }
                    continue;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int cu = __shfl_sync(gmask, c, (t + u) & (LPR - 1), LPR);
                    bv[u] = make_uint4(0, 0, 0, 0);
                    if (t + u < cnt && cu >= 0 && active)
                        bv[u] = __ldg(reinterpret_cast<const uint4 *>(Bn + (size_t)cu * a.ldb));
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    unsigned short xu = (unsigned short)__shfl_sync(gmask, (int)x, (t + u) & (LPR - 1), LPR);
                    if (t + u >= cnt) xu = 0;
                    const unsigned short *h = reinterpret_cast<const unsigned short *>(&bv[u]);
#pragma unroll
                    for (int w = 0; w < 8; w++) acc[w] = ptx::fma_f16_f32(xu, h[w], acc[w]);
                }
            }
        }
    };
    auto write = [&](int r, const float *acc) {
        if (!active)
            return;
        OutT *cp = reinterpret_cast<OutT *>(a.C) + (size_t)r * a.ldc + n0;
        float o[8];
        if (a.beta != 0.f) {
            float old[8];
            load8(cp, old);
#pragma unroll
            for (int w = 0; w < 8; w++) o[w] = fmaf(a.alpha, acc[w], a.beta * old[w]);
        } else {
#pragma unroll
            for (int w = 0; w < 8; w++) o[w] = a.alpha * acc[w];
        }
        store8(cp, o);
    };
    float acc[8];
    const int r = (int)(blockIdx.x + (unsigned)g * gridDim.x);
    if ((unsigned)r < (unsigned)a.M) { // uniform across the group; (the rounded-up row count can pass the largest int)
        int start, end;
        range(r, start, end);
        if (end - start > kShortRow) {
            if (sub == 0) {
                const int q = atomicAdd(&s_n, 1);
                s_row[q] = r;
                s_beg[q] = start;
                s_end[q] = end;
            }
        } else if (start < end || !(a.flags & TCA_FLAG_KEEP_EMPTY_ROWS)) {
#pragma unroll
            for (int w = 0; w < 8; w++) acc[w] = 0.f;
            run(start, end, acc);
            write(r, acc);
        }
    }
    __syncthreads();
    const int n_long = s_n;
    if (n_long == 0)
        return;
    int q = 0, first = 0, parts = G; // the row of this group, the row's first group, their number
    if (n_long > 1) {
        if (threadIdx.x < 32) { // a group for each long row, the others in proportion to the rows' lengths
            long long total = 0;
            for (int i = lane; i < n_long; i += 32) total += s_end[i] - s_beg[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
            int base = 0;
            for (int i0 = 0; i0 < n_long; i0 += 32) {
                const int i = i0 + lane;
                int sum = i < n_long ? 1 + (int)((long long)(G - n_long) * (s_end[i] - s_beg[i]) / total) : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += v;
                }
                if (i < n_long) s_last[i] = base + sum;
                base += __shfl_sync(0xffffffffu, sum, 31);
            }
        }
        __syncthreads();
        int hi = n_long; // the first row whose groups end after this one
        while (q < hi) {
            const int mid = (q + hi) >> 1;
            if (s_last[mid] <= g) q = mid + 1;
            else hi = mid;
        }
        first = q > 0 ? s_last[q - 1] : 0;
        parts = q < n_long ? s_last[q] - first : 0;
    }
#pragma unroll
    for (int w = 0; w < 8; w++) acc[w] = 0.f;
    if (parts > 0) {
        const int start = s_beg[q];
        const long long len = s_end[q] - start;
        run(start + (int)(len * (g - first) / parts), start + (int)(len * (g - first + 1) / parts), acc);
    }
    if (g > first) {
#pragma unroll
        for (int w = 0; w < 8; w++) s_part[(g * LPR + sub) * 8 + w] = acc[w];
    }
    __syncthreads();
    if (parts > 0 && g == first) {
        for (int k = g + 1; k < first + parts; k++)
#pragma unroll
            for (int w = 0; w < 8; w++) acc[w] += s_part[(k * LPR + sub) * 8 + w];
        write(s_row[q], acc);
    }
}

// Rows of plans, batched and streamed. Every job (one forward of one plan)
// contributes its work items: runs of consecutive sorted rows with about
// kItemNnz nonzeros in total. A group of L lanes takes one item and streams
// through its nonzeros -- which are contiguous in the plan's re-ordered CSR --
// with U = 8 independent 16-byte B loads in flight per lane, flushing a row's
// accumulators to C[perm[row]] whenever the stream crosses a row end. Short
// rows thus cost no dependent load chain per row, and a launch keeps
// thousands of items in flight.
struct CcJob {
    const int2 *items;
    const int *perm, *p_row_ptr, *p_col;
    const __half *p_val;
    const __half *B;
    void *C;
    // E4M3 forward: values, B (row stride ldq bytes) and their scales
    const uint8_t *p_val8, *Bq;
    const float *row_scale, *col_scale;
    int ldq;
    int n_items;
    int slices; // > 1: an item is taken once per 32 W columns of N, by as many warps
    int parts;  // > 1: its rows are cut among as many warps
    int M, K, N, ldb, ldc;
    float alpha, beta;
    unsigned flags;
};

// A launch's jobs; the stream kernel is also built for CAP = 1, whose
// parameter block launches faster for a single forward.
template <int CAP>
struct CcBatchT {
    int n_jobs;
    int item_start[CAP + 1]; // first item of each job in the flattened list
    CcJob job[CAP];
};
using CcBatch = CcBatchT<kMaxCcJobs>;

// ---------------------------------------------------------------------------
// Vectorised item stream: one warp per stream of items, persistent.
//
// Warp w takes items w, w + n_warps, ... of the flattened item list of all
// jobs. Each item's metadata is fetched by a three-deep software pipeline so
// that no dependent load chain is exposed between items: while item i is
// computed, the nonzeros (column, value) of item i+1, the row offsets and
// output rows of item i+2 and the descriptor of item i+3 are in flight.
// Lane k holds row offset k and output row k of its item and nonzero k of its
// first 32; every lane owns W consecutive output columns (W halves of B per
// load, 8 loads in flight per lane) and accumulates with mixed-precision FMA
// (FP16 x FP16 + FP32, one rounding -- the same value as converting both
// factors to FP32 and using fmaf).
// ---------------------------------------------------------------------------
template <int W> struct HalfVec;
template <> struct HalfVec<8> { using T = uint4; };
template <> struct HalfVec<4> { using T = uint2; };
template <> struct HalfVec<2> { using T = unsigned; };

using ptx::fma_f16_f32;

template <int W> __device__ __forceinline__ void load_out(const __half *p, float *v)
{
    using V = typename HalfVec<W>::T;
    const V u = *reinterpret_cast<const V *>(p);
    const __half *h = reinterpret_cast<const __half *>(&u);
#pragma unroll
    for (int i = 0; i < W; i++) v[i] = __half2float(h[i]);
}
template <int W> __device__ __forceinline__ void load_out(const float *p, float *v)
{
#pragma unroll
    for (int i = 0; i < W; i += 2) {
        const float2 f = reinterpret_cast<const float2 *>(p)[i / 2];
        v[i] = f.x;
        v[i + 1] = f.y;
    }
}
template <int W> __device__ __forceinline__ void store_out(__half *p, const float *v)
{
    using V = typename HalfVec<W>::T;
    V u;
    __half2 *h = reinterpret_cast<__half2 *>(&u);
#pragma unroll
    for (int i = 0; i < W / 2; i++) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<V *>(p) = u;
}
template <int W> __device__ __forceinline__ void store_out(float *p, const float *v)
{
    if constexpr (W >= 4) {
#pragma unroll
        for (int i = 0; i < W; i += 4)
            reinterpret_cast<float4 *>(p)[i / 4] = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    }
}

struct ItemDesc {
    int job, r0, nrows; // job | N-slice << 8
};

template <typename Batch>
__device__ __forceinline__ ItemDesc load_desc(const Batch &b, int item)
{
    ItemDesc d{0, 0, 0};
    if (item < b.item_start[b.n_jobs]) {
        int j = 0, hi = b.n_jobs - 1; // the last job whose first item is <= item
        while (j < hi) {
            const int mid = (j + hi + 1) >> 1;
            if (b.item_start[mid] <= item)
                j = mid;
            else
                hi = mid - 1;
        }
        const CcJob &a = b.job[j];
        const int slices = a.slices, parts = a.parts;
        int local = item - b.item_start[j];
        d.job = j;
        if (slices > 1) {
            d.job = j | local % slices << 8;
            local /= slices;
        }
        int part = 0;
        if (parts > 1) { // one part after the other: side by side the same part would fall to a warp every time
            part = local / a.n_items;
            local -= part * a.n_items;
        }
        const int2 it = __ldg(a.items + local);
        const int rows = it.y - it.x, first = parts > 1 ? rows * part / parts : 0;
        d.r0 = it.x + first;
        d.nrows = (parts > 1 ? rows * (part + 1) / parts : rows) - first; // no rows: nothing to do in this part
    }
    return d;
}

// B vectors of W elements: W halves, or W E4M3 bytes.
template <int W, bool F8> struct BVec { using T = typename HalfVec<W>::T; };
template <> struct BVec<8, true> { using T = uint2; };
template <> struct BVec<4, true> { using T = unsigned; };
template <> struct BVec<2, true> { using T = unsigned short; };

// One output row's W columns: t = acc (E4M3: x row scale sa x column scales
// sb), then alpha t + beta C.
template <typename OutT, int W, bool F8>
__device__ __forceinline__ void store_row(const CcJob &a, int orow, int n0, const float *acc, float sa,
                                          const float *sb)
{
    OutT *cp = reinterpret_cast<OutT *>(a.C) + (size_t)orow * a.ldc + n0;
    float t[W], o[W];
#pragma unroll
    for (int i = 0; i < W; i++) {
        if constexpr (F8)
            t[i] = acc[i] * (sa * sb[i]);
        else
            t[i] = acc[i];
    }
    if (a.beta != 0.f) {
        float old[W];
        load_out<W>(cp, old);
#pragma unroll
        for (int i = 0; i < W; i++) o[i] = fmaf(a.alpha, t[i], a.beta * old[i]);
    } else {
#pragma unroll
        for (int i = 0; i < W; i++) o[i] = a.alpha * t[i];
    }
    store_out<W>(cp, o);
}

// acc[i] = v * b[i] + acc[i] over one B vector (E4M3 pairs unpacked to FP16).
template <int W, bool F8, typename V>
__device__ __forceinline__ void fma_vec(float *acc, unsigned short v, const V &bv)
{
    if constexpr (F8) {
        const __nv_fp8x2_storage_t *q = reinterpret_cast<const __nv_fp8x2_storage_t *>(&bv);
#pragma unroll
        for (int i = 0; i < W / 2; i++) {
            const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(q[i], __NV_E4M3);
            acc[2 * i] = fma_f16_f32(v, h.x, acc[2 * i]);
            acc[2 * i + 1] = fma_f16_f32(v, h.y, acc[2 * i + 1]);
        }
    } else {
        const unsigned short *h = reinterpret_cast<const unsigned short *>(&bv);
#pragma unroll
        for (int i = 0; i < W; i++) acc[i] = fma_f16_f32(v, h[i], acc[i]);
    }
}

// F8: values and B are E4M3 (every E4M3 value is an FP16 value, so the
// products are formed exactly by the same mixed-precision FMA); the flush
// multiplies the FP32 sum by row scale x column scale, as the tensor-core
// epilogue does.
//
// Three blocks per SM (80 registers a thread). Beside the tensor-core
// kernel's block one of them is resident at a time (a warp's registers come
// from its SM sub-partition, and the tensor-core warps leave room for two
// more warps per sub-partition). U B loads are in flight per lane: 8, or 4
// at W = 8, which keeps the register budget without spills.
template <typename OutT, int W, bool F8, int CAP = kMaxCcJobs>
__global__ void __launch_bounds__(256, 3) spmm_cc_stream_kernel(const __grid_constant__ CcBatchT<CAP> b)
{
    using V = typename BVec<W, F8>::T;
    constexpr int U = W == 8 ? 4 : 8;
    // Launched as a programmatic dependent (beside the tensor-core kernel, or
    // behind another CUDA-core launch): let the next launch start as well.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int n_warps = (int)gridDim.x * 8;
    int item = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5);

    // row offsets (lane k <= nrows), output rows and E4M3 row scales (lane k < nrows) of an item
    auto load_rows = [&](const ItemDesc &d, int &rs, int &orow, float &sc) {
        rs = 0;
        orow = 0;
        sc = 0.f;
        if (lane <= d.nrows && d.nrows > 0) {
            const CcJob &a = b.job[d.job & 255];
            rs = __ldg(a.p_row_ptr + d.r0 + lane);
            if (lane < d.nrows) {
                orow = __ldg(a.perm + d.r0 + lane);
                if constexpr (F8)
                    sc = __ldg(a.row_scale + d.r0 + lane);
            }
        }
    };
    auto value = [&](const CcJob &a, int j) -> unsigned short {
        if constexpr (F8)
            return __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)a.p_val8[j], __NV_E4M3).x;
        else
            return __half_as_ushort(a.p_val[j]);
    };
    // the item's first 32 nonzeros, one per lane (values as FP16 bits)
    auto load_nz = [&](const ItemDesc &d, int rs, int &col, unsigned short &val) {
        const int j0 = __shfl_sync(full, rs, 0), j1 = __shfl_sync(full, rs, d.nrows & 31);
        col = 0;
        val = 0;
        if (d.nrows > 0 && j0 + lane < j1) {
            const CcJob &a = b.job[d.job & 255];
            col = __ldg(a.p_col + j0 + lane);
            val = value(a, j0 + lane);
        }
    };

    ItemDesc d0 = load_desc(b, item), d1 = load_desc(b, item + n_warps), d2 = load_desc(b, item + 2 * n_warps);
    int rs0, out0, rs1, out1, col0;
    float sc0, sc1;
    unsigned short val0;
    load_rows(d0, rs0, out0, sc0);
    load_rows(d1, rs1, out1, sc1);
    load_nz(d0, rs0, col0, val0);

    while (item < b.item_start[b.n_jobs]) {
        // ---- pipeline: nonzeros of i+1, rows of i+2, descriptor of i+3
        int col1;
        unsigned short val1;
        load_nz(d1, rs1, col1, val1);
        int rs2, out2;
        float sc2;
        load_rows(d2, rs2, out2, sc2);
        const ItemDesc d3 = load_desc(b, item + 3 * n_warps);

        // ---- item i
        const CcJob &a = b.job[d0.job & 255];
        const int nrows = d0.nrows;
        const int j0 = __shfl_sync(full, rs0, 0), j1 = __shfl_sync(full, rs0, nrows);
        const bool keep = (a.flags & TCA_FLAG_KEEP_EMPTY_ROWS) != 0;
        // Items whose rows hold one nonzero each (the short-row tails of skewed
        // matrices): C[row] = alpha v B[col] (+ beta C[row]) row by row, with U
        // rows' B vectors in flight and no row-boundary tracking.
        const int rs_next = __shfl_down_sync(full, rs0, 1);
        const bool singles = __all_sync(full, lane >= nrows || rs_next - rs0 == 1); // (also without rows)
        const int nb0 = (d0.job >> 8) * 32 * W, nb1 = a.slices > 1 ? min(a.N, nb0 + 32 * W) : a.N;
        for (int nb = nb0; singles && nb < nb1; nb += 32 * W) {
            const int n0 = nb + lane * W;
            const bool active = n0 < a.N;
            const uint8_t *Bn = F8 ? a.Bq + (active ? n0 : 0)
                                   : reinterpret_cast<const uint8_t *>(a.B + (active ? n0 : 0));
            const size_t brow = F8 ? (size_t)a.ldq : (size_t)a.ldb * 2; // bytes per B row
            float sb[F8 ? W : 1];
            if constexpr (F8) {
#pragma unroll
                for (int i = 0; i < W; i++) sb[i] = active ? __ldg(a.col_scale + n0 + i) : 0.f;
            }
            for (int t = 0; t < nrows; t += U) {
                V bv[U];
                unsigned short av[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int r = (t + u) & 31;
                    const int cu = __shfl_sync(full, col0, r);
                    av[u] = (unsigned short)__shfl_sync(full, (int)val0, r);
                    bv[u] = V{};
                    if (active && t + u < nrows)
                        bv[u] = __ldg(reinterpret_cast<const V *>(Bn + (size_t)cu * brow));
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int r = (t + u) & 31;
                    const int orow = __shfl_sync(full, out0, r);
                    float sa = 1.f;
                    if constexpr (F8)
                        sa = __shfl_sync(full, sc0, r);
                    if (active && t + u < nrows) {
                        float acc[W];
#pragma unroll
                        for (int i = 0; i < W; i++) acc[i] = 0.f;
                        fma_vec<W, F8>(acc, av[u], bv[u]);
                        store_row<OutT, W, F8>(a, orow, n0, acc, sa, sb);
                    }
                }
            }
        }
        for (int nb = nb0; !singles && nb < nb1; nb += 32 * W) {
            const int n0 = nb + lane * W;
            const bool active = n0 < a.N;
            const uint8_t *Bn = F8 ? a.Bq + (active ? n0 : 0)
                                   : reinterpret_cast<const uint8_t *>(a.B + (active ? n0 : 0));
            const size_t brow = F8 ? (size_t)a.ldq : (size_t)a.ldb * 2; // bytes per B row
            float sb[F8 ? W : 1];
            if constexpr (F8) {
#pragma unroll
                for (int i = 0; i < W; i++) sb[i] = active ? __ldg(a.col_scale + n0 + i) : 0.f;
            }
            float acc[W];
#pragma unroll
            for (int i = 0; i < W; i++) acc[i] = 0.f;
            int cr = 0;
            int ce = __shfl_sync(full, rs0, 1);
            auto flush = [&]() {
                const int rstart = __shfl_sync(full, rs0, cr);
                const int orow = __shfl_sync(full, out0, cr);
                float sa = 1.f;
                if constexpr (F8)
                    sa = __shfl_sync(full, sc0, cr);
                if (active && !(keep && rstart == ce))
                    store_row<OutT, W, F8>(a, orow, n0, acc, sa, sb);
#pragma unroll
                for (int i = 0; i < W; i++) acc[i] = 0.f;
                cr++;
                const int nxt = __shfl_sync(full, rs0, min(cr + 1, 31));
                ce = cr < nrows ? nxt : 0x7fffffff;
            };
            for (int base = j0; base < j1; base += 32) {
                int c = col0;
                unsigned short v = val0;
                if (base != j0) { // a row longer than 32 nonzeros: the rest is loaded here
                    c = 0;
                    v = 0;
                    if (base + lane < j1) {
                        c = __ldg(a.p_col + base + lane);
                        v = value(a, base + lane);
                    }
                }
                const int m = min(32, j1 - base);
                for (int t = 0; t < m; t += U) {
                    V bv[U];
                    unsigned short av[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int cu = __shfl_sync(full, c, t + u);
                        av[u] = (unsigned short)__shfl_sync(full, (int)v, t + u);
                        bv[u] = V{};
                        if (active && t + u < m)
                            bv[u] = __ldg(reinterpret_cast<const V *>(Bn + (size_t)cu * brow));
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (t + u < m) { // uniform across the warp
                            while (base + t + u >= ce) flush();
                            fma_vec<W, F8>(acc, av[u], bv[u]);
                        }
                    }
                }
            }
            while (cr < nrows) flush();
        }

        // ---- rotate the pipeline
        d0 = d1; rs0 = rs1; out0 = out1; sc0 = sc1; col0 = col1; val0 = val1;
        d1 = d2; rs1 = rs2; out1 = out2; sc1 = sc2;
        d2 = d3;
        item += n_warps;
    }
    // Complete no earlier than the launch this one depends on (a no-op for an
    // ordinary launch): work after this kernel on the stream then also finds
    // the tensor-core kernel done, whatever the stream's ordering rules for
    // programmatic dependents. That kernel never waits on this one and all of
    // its blocks were resident before this grid started, so the wait ends.
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

bool vec_ok(const void *B, int ldb, int N, const void *C, int ldc, int c_dtype)
{
    const size_t c_elem = (c_dtype == TCA_DTYPE_F16) ? 2 : 4;
    return (N % 8 == 0) && (ldb % 8 == 0) && aligned16(B) && aligned16(C) && ((ldc * c_elem) % 16 == 0);
}

} // namespace

namespace {

// Lanes and blocks of a job of the rows kernel. A group covers N in one slice
// up to 256 columns: narrower groups spend more instructions per byte gathered
// (measured, 4096 x 4096 at 95 %, N = 512: 8 lanes a row 193 us, 32 lanes
// 118 us). Blocks: about 64 nonzeros and rows per group, so that a
// block's fixed cost (search, prefix sums, first dependent loads) is small
// beside them, in whole waves of two blocks per SM, while a group keeps 8.
struct RowsShape { int lpr, w; };
RowsShape rows_shape(int N, bool vec)
{
    if (vec)
        return {N <= 32 ? 4 : N <= 64 ? 8 : N <= 128 ? 16 : 32, 8};
    return {32, N <= 32 ? 1 : N <= 64 ? 2 : N <= 128 ? 4 : 8};
}
int rows_blocks(const RowsJob &a, const RowsShape &sh, int slices) // per N-slice
{
    const long long groups = kRowsThreads / sh.lpr, keys = (long long)a.nnz - a.base + a.M;
    const long long wave = 2 * kSMs; // resident blocks
    // whole waves over all slices (3001 x 1777 at 92 %, N = 203: 419 blocks, 1.4 waves, 41.6 us; 296 34.5 us, before the short path)
    const long long waves = std::max(1LL, (keys * slices / (groups * 64) + wave / 2) / wave);
    const long long n = std::min(std::max(1LL, waves * wave / slices), (keys + groups * 8 - 1) / (groups * 8));
    return (int)std::max<long long>(1, std::min<long long>({n, a.M, INT_MAX / slices}));
}

// The kernel with the short path (kFastLpr) or without.
template <typename OutT, int LPR, int W, bool VEC, bool VC, int CAP> auto rows_kernel(const RowsBatchT<CAP> &b)
{
    if constexpr (!VEC || LPR < kFastLpr) {
        return &spmm_rows_kernel<OutT, LPR, W, VEC, VC, CAP, false>;
    } else if constexpr (LPR == 32) {
        return &spmm_rows_kernel<OutT, LPR, W, VEC, VC, CAP, true>;
    } else {
        for (int i = 0; i < b.n_jobs; i++)
            if ((long long)b.job[i].nnz - b.job[i].base <= (long long)kFastMean * b.job[i].M)
                return &spmm_rows_kernel<OutT, LPR, W, VEC, VC, CAP, false>;
        return &spmm_rows_kernel<OutT, LPR, W, VEC, VC, CAP, true>;
    }
}

// beside: a programmatic dependent of the tensor-core launch before it (as
// launch_stream_cap).
template <typename OutT, int LPR, int W, bool VEC>
int launch_rows(const RowsBatchT<kMaxCcJobs> &b, cudaStream_t s, bool beside)
{
    const int grid = b.block_start[b.n_jobs];
    if (b.n_jobs == 0 || grid == 0)
        return TCA_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kRowsThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = beside ? 1 : 0;
    if (b.n_jobs == 1) {
        RowsBatchT<1> one;
        one.n_jobs = 1;
        one.block_start[0] = 0;
        one.block_start[1] = grid;
        one.job[0] = b.job[0];
        TCA_CUDA_TRY(cudaLaunchKernelEx(&cfg, rows_kernel<OutT, LPR, W, VEC, VEC, 1>(one), one));
    } else {
        TCA_CUDA_TRY(cudaLaunchKernelEx(&cfg, rows_kernel<OutT, LPR, W, VEC, VEC, kMaxCcJobs>(b), b));
    }
    return TCA_OK;
}

template <typename OutT>
int launch_rows_shape(const RowsBatchT<kMaxCcJobs> &b, const RowsShape &sh, bool vec, cudaStream_t s, bool beside = false)
{
    if (vec) {
        switch (sh.lpr) {
        case 4: return launch_rows<OutT, 4, 8, true>(b, s, beside);
        case 8: return launch_rows<OutT, 8, 8, true>(b, s, beside);
        case 16: return launch_rows<OutT, 16, 8, true>(b, s, beside);
        default: return launch_rows<OutT, 32, 8, true>(b, s, beside);
        }
    }
    switch (sh.w) {
    case 1: return launch_rows<OutT, 32, 1, false>(b, s, beside);
    case 2: return launch_rows<OutT, 32, 2, false>(b, s, beside);
    case 4: return launch_rows<OutT, 32, 4, false>(b, s, beside);
    default: return launch_rows<OutT, 32, 8, false>(b, s, beside);
    }
}

void rows_add(RowsBatchT<kMaxCcJobs> &b, RowsJob &a, const RowsShape &sh)
{
    const int slices = (a.N + sh.lpr * sh.w - 1) / (sh.lpr * sh.w);
    a.n_blocks = rows_blocks(a, sh, slices);
    b.job[b.n_jobs] = a;
    b.block_start[b.n_jobs + 1] = b.block_start[b.n_jobs] + a.n_blocks * slices;
    b.n_jobs++;
}

} // namespace

namespace {

// Copies rows of N halves to rows of ldp (a multiple of 8, at least N), zeros
// after them: a warp per 256 columns of a row, every access coalesced.
__global__ void __launch_bounds__(256) k_pad_rows(const __half *__restrict__ src, int rows, int N, int ld,
                                                  __half *__restrict__ dst, int ldp)
{
    const int slices = (ldp + 255) / 256, lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= (long long)rows * slices)
        return;
    const long long r = w / slices;
    const int n0 = (int)(w - r * slices) * 256 + lane;
    unsigned short v[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
        v[u] = n0 + u * 32 < N ? __ldg(reinterpret_cast<const unsigned short *>(src) + r * ld + n0 + u * 32) : (unsigned short)0;
#pragma unroll
    for (int u = 0; u < 8; u++)
        if (n0 + u * 32 < ldp)
            reinterpret_cast<unsigned short *>(dst)[r * ldp + n0 + u * 32] = v[u];
}

// C = alpha * S + beta * C from FP32 sums S (rows of lds), FP16 C of any
// alignment; rows without nonzeros are skipped with KEEP_EMPTY_ROWS. A warp
// per 256 columns of a sorted row. A tile product multiplies a row's zeros by
// the chunk's other rows of B as well, so an infinity or NaN in B reaches the
// sums of rows that hold no nonzero of its column: a sum that is not finite is
// formed anew from the row's nonzeros and the padded B (rows of lds).
__global__ void __launch_bounds__(256)
k_unpad_rows(const float *__restrict__ sums, int lds, const int *__restrict__ perm, const int *__restrict__ p_row_ptr,
             const int *__restrict__ p_col, const __half *__restrict__ p_val, const __half *__restrict__ B, int M,
             int N, __half *__restrict__ C, int ldc, float alpha, float beta, unsigned flags)
{
    const int slices = (N + 255) / 256, lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= (long long)M * slices)
        return;
    const int i = (int)(w / slices), n0 = (int)(w - (long long)i * slices) * 256 + lane;
    if ((flags & TCA_FLAG_KEEP_EMPTY_ROWS) && __ldg(p_row_ptr + i + 1) == __ldg(p_row_ptr + i))
        return;
    const size_t r = (size_t)__ldg(perm + i);
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = n0 + u * 32 < N ? __ldg(sums + r * lds + n0 + u * 32) : 0.f;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (n0 + u * 32 >= N)
            break;
        __half *c = C + r * ldc + n0 + u * 32;
        if (!isfinite(v[u])) {
            v[u] = 0.f;
            for (int j = __ldg(p_row_ptr + i); j < __ldg(p_row_ptr + i + 1); j++)
                v[u] = fmaf(__half2float(p_val[j]), __half2float(B[(size_t)p_col[j] * lds + n0 + u * 32]), v[u]);
        }
        float o = alpha * v[u];
        if (beta != 0.f) o = fmaf(beta, __half2float(*c), o);
        *c = __float2half_rn(o);
    }
}

template <typename OutT> int launch_rows_short(const RowsJob &a, int lpr, int slices, cudaStream_t s)
{
    const int groups = kRowsThreads / lpr;
    const dim3 grid(((unsigned)a.M + groups - 1) / groups, (unsigned)slices);
    switch (lpr) {
    case 4: spmm_rows_short_kernel<OutT, 4><<<grid, kRowsThreads, 0, s>>>(a); break;
    case 8: spmm_rows_short_kernel<OutT, 8><<<grid, kRowsThreads, 0, s>>>(a); break;
    case 16: spmm_rows_short_kernel<OutT, 16><<<grid, kRowsThreads, 0, s>>>(a); break;
    default: spmm_rows_short_kernel<OutT, 32><<<grid, kRowsThreads, 0, s>>>(a); break;
    }
    TCA_CUDA_TRY(cudaGetLastError());
    return TCA_OK;
}

template <typename OutT, int LPR> int launch_rows_padded(const RowsBatchT<1> &b, cudaStream_t s)
{
    rows_kernel<OutT, LPR, 8, true, false, 1>(b)<<<b.block_start[1], kRowsThreads, 0, s>>>(b);
    TCA_CUDA_TRY(cudaGetLastError());
    return TCA_OK;
}

// The rows kernel over a padded (aligned) copy of B, C as it is.
template <typename OutT> int rows_over_padded(RowsJob a, cudaStream_t s)
{
    const RowsShape sh = rows_shape(a.N, true);
    RowsBatchT<kMaxCcJobs> all;
    all.n_jobs = 0;
    all.block_start[0] = 0;
    rows_add(all, a, sh);
    RowsBatchT<1> b;
    b.n_jobs = 1;
    b.block_start[0] = 0;
    b.block_start[1] = all.block_start[1];
    b.job[0] = all.job[0];
    switch (sh.lpr) {
    case 4: return launch_rows_padded<OutT, 4>(b, s);
    case 8: return launch_rows_padded<OutT, 8>(b, s);
    case 16: return launch_rows_padded<OutT, 16>(b, s);
    default: return launch_rows_padded<OutT, 32>(b, s);
    }
}

// Stream-ordered scratch of one call on a stream that is not being captured.
// Allocating is refused while another thread captures (in the global mode), and
// the attempt would break that capture: this thread's mode is relaxed meanwhile.
struct Scratch {
    void *p = nullptr;
    cudaStream_t s;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    explicit Scratch(cudaStream_t st) : s(st) { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Scratch()
    {
        dev_free(p, s);
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
};

} // namespace

// A forward whose B or C does not allow 16-byte accesses (an odd N, unaligned
// rows) through an aligned copy of B, when that pays: two-byte accesses gather
// B at about half the rate of 16-byte ones (3001 x 1777 at 92 %, N = 203: 48
// us; 2 us for the copy and 26 us after it). The rows kernel takes the copy,
// FP32 FMAs as without it. For a plan whose caller asked for tensor cores (path
// 2) its tensor-core windows run there: that needs an aligned C too, so the sums
// go to an FP32 buffer and from there to an FP16 C (4096 x 4096 at 90 %, N =
// 1001: 45 us, 324 on CUDA cores). Not unasked: tensor-core sums lie 4 to 100
// times as far from those in 64 bits (1058 x 3570 at 74 %, positive operands:
// 7.6e-6 against 6.6e-8), of which the rounding to FP16 leaves little (12 drawn
// problems: 1.000001 to 1.001 times the error of the result) but not nothing.
// The rule: nnz * N >= 2^25 (below, the two-byte kernel takes less than ~25
// us and the copy and its launch eat the gain), copies of at most kPadMax
// bytes, and not under stream capture, where this call allocates nothing.
// *done = false: the caller runs the two-byte kernel.
constexpr size_t kPadMax = 64u << 20;

int spmm_padded(const SpmmJob *sj, const int *row_ptr, const int *col, const __half *val, int M, int K, int nnz,
                const __half *B, int ldb, int N, void *C, int ldc, int c_dtype, float alpha, float beta, unsigned flags,
                cudaStream_t s, bool *done)
{
    *done = false;
    const int ldp = (N + 63) & ~63;
    const size_t b_bytes = sizeof(__half) * (size_t)K * ldp, c_bytes = sizeof(float) * (size_t)M * ldp;
    if ((long long)nnz * N < (1LL << 25) || b_bytes > kPadMax || c_bytes > kPadMax)
        return TCA_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
        cudaGetLastError();
        return TCA_OK;
    }
    if (cap != cudaStreamCaptureStatusNone)
        return TCA_OK;
    const bool tc = sj && sj->p->opts.path == 2 && sj->p->n_tc > 0 && c_dtype == TCA_DTYPE_F16;
    Scratch ws(s);
    if (dev_malloc(&ws.p, b_bytes + (tc ? c_bytes : 0), s) != TCA_OK) {
        cudaGetLastError();
        clear_error();
        return TCA_OK;
    }
    *done = true;
    __half *Bp = static_cast<__half *>(ws.p);
    const long long warps = (long long)K * ((ldp + 255) / 256);
    k_pad_rows<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(B, K, N, ldb, Bp, ldp);
    TCA_CUDA_TRY(cudaGetLastError());
    if (!tc) {
        RowsJob a{row_ptr, col, sj ? sj->p->perm : nullptr, val, Bp, C, M, K, nnz, N, ldp, ldc, 0, 0, alpha, beta, flags};
        return c_dtype == TCA_DTYPE_F16 ? rows_over_padded<__half>(a, s) : rows_over_padded<float>(a, s);
    }
    float *sums = reinterpret_cast<float *>(static_cast<char *>(ws.p) + b_bytes); // b_bytes: a multiple of 128
    SpmmJob job = *sj;
    job.B = Bp;
    job.ldb = ldp;
    job.N = ldp;
    job.C = sums;
    job.ldc = ldp;
    job.tc = true;
    job.n_tile = pick_tc_tile(sj->p, ldp, false);
    TCA_TRY(run_jobs_with_events(&job, 1, TCA_DTYPE_F32, 1.f, 0.f, 0u, s, nullptr));
    const long long out_warps = (long long)M * ((N + 255) / 256);
    k_unpad_rows<<<(unsigned)((out_warps * 32 + 255) / 256), 256, 0, s>>>(
        sums, ldp, sj->p->perm, row_ptr, col, val, Bp, M, N, static_cast<__half *>(C), ldc, alpha, beta, flags);
    TCA_CUDA_TRY(cudaGetLastError());
    return TCA_OK;
}

int launch_spmm_csr_cc(const int *row_ptr, const int *col_idx, const __half *vals, int M, int K, int nnz,
                       const __half *B, int ldb, int N, void *C, int ldc, int c_dtype,
                       float alpha, float beta, unsigned flags, cudaStream_t stream)
{
    const bool vec = vec_ok(B, ldb, N, C, ldc, c_dtype);
    if (!vec) {
        bool done = false;
        TCA_TRY(spmm_padded(nullptr, row_ptr, col_idx, vals, M, K, nnz, B, ldb, N, C, ldc, c_dtype, alpha, beta, flags,
                            stream, &done));
        if (done)
            return TCA_OK;
    }
    const RowsShape sh = rows_shape(N, vec);
    RowsBatchT<kMaxCcJobs> b;
    b.n_jobs = 0;
    b.block_start[0] = 0;
    RowsJob a{row_ptr, col_idx, nullptr, vals, B, C, M, K, nnz, N, ldb, ldc, 0, 0, alpha, beta, flags};
    const int slices = (N + sh.lpr * 8 - 1) / (sh.lpr * 8);
    if (vec && nnz <= (long long)kShortMean * M && slices <= 65535)
        return c_dtype == TCA_DTYPE_F16 ? launch_rows_short<__half>(a, sh.lpr, slices, stream)
                                        : launch_rows_short<float>(a, sh.lpr, slices, stream);
    rows_add(b, a, sh);
    return c_dtype == TCA_DTYPE_F16 ? launch_rows_shape<__half>(b, sh, vec, stream)
                                    : launch_rows_shape<float>(b, sh, vec, stream);
}

bool dense_operands_vec_ok(const void *B, int ldb, int N, const void *C, int ldc, int c_dtype)
{
    return vec_ok(B, ldb, N, C, ldc, c_dtype);
}

namespace {

// ---------------------------------------------------------------------------
// Tensor-core item kernel (mma.sync, FP16): the CUDA-core windows' work items
// as tiny dense products. An item of R <= 31 rows and Z <= 32 nonzeros is
// C_item[R x N] = A_item[R x Z] * B_item[Z x N], where A_item holds each
// nonzero in its own column (row of the nonzero, position in the item) and
// B_item is the item's gathered B rows. Per 64-column slice of N, the warp
// stages B_item in shared memory (32 rows x 128 bytes, 16-byte chunks XOR-
// swizzled by row), reads it with ldmatrix.trans as m16n8k16 B fragments and
// issues 8 mma.sync per 16 rows and 16 nonzeros; A fragments come from the
// nonzeros in lane registers by shuffle. The accumulators go through shared
// memory so that every output row is stored as 128 contiguous bytes. A row
// longer than 32 nonzeros (an item of its own) is walked 32 nonzeros at a
// time into the same accumulators. Per output element this issues about a
// third of the instructions of the shuffle-and-FMA stream kernel; the
// products are exact in FP32 and sums accumulate in FP32.
// ---------------------------------------------------------------------------
constexpr int kMmaWarps = 8;
constexpr int kCcMma = 16; // cc_cols value that selects this kernel
constexpr int kMmaSliceCols = 64;
constexpr int kMmaAccStride = 72; // floats per staged accumulator row (2-way bank conflicts at most)
constexpr int kMmaWarpSmem = 16 * kMmaAccStride * 4; // >= 32 x 128 bytes of B staging

__device__ __forceinline__ void mma_16816(float *d, const uint32_t *a, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t *r)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

template <typename OutT>
__global__ void __launch_bounds__(kMmaWarps * 32, 2) spmm_cc_mma_kernel(const __grid_constant__ CcBatch b)
{
    __shared__ __align__(16) uint8_t s_all[kMmaWarps * kMmaWarpSmem];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint8_t *ws = s_all + wid * kMmaWarpSmem;
    const uint32_t ws_addr = (uint32_t)__cvta_generic_to_shared(ws);
    float *acc_s = reinterpret_cast<float *>(ws);
    const int n_warps = (int)gridDim.x * kMmaWarps;
    int item = (int)blockIdx.x * kMmaWarps + wid;
    const int g = lane >> 2, c4 = lane & 3;

    auto load_rows = [&](const ItemDesc &d, int &rs, int &orow) {
        rs = 0;
        orow = 0;
        if (lane <= d.nrows && d.nrows > 0) {
            const CcJob &a = b.job[d.job & 255];
            rs = __ldg(a.p_row_ptr + d.r0 + lane);
            if (lane < d.nrows)
                orow = __ldg(a.perm + d.r0 + lane);
        }
    };
    auto load_nz = [&](const ItemDesc &d, int rs, int &col, unsigned short &val) {
        const int j0 = __shfl_sync(full, rs, 0), j1 = __shfl_sync(full, rs, d.nrows & 31);
        col = 0;
        val = 0;
        if (d.nrows > 0 && j0 + lane < j1) {
            const CcJob &a = b.job[d.job & 255];
            col = __ldg(a.p_col + j0 + lane);
            val = __half_as_ushort(a.p_val[j0 + lane]);
        }
    };

    ItemDesc d0 = load_desc(b, item), d1 = load_desc(b, item + n_warps), d2 = load_desc(b, item + 2 * n_warps);
    int rs0, out0, rs1, out1, col0;
    unsigned short val0;
    load_rows(d0, rs0, out0);
    load_rows(d1, rs1, out1);
    load_nz(d0, rs0, col0, val0);

    while (d0.nrows > 0) {
        int col1;
        unsigned short val1;
        load_nz(d1, rs1, col1, val1);
        int rs2, out2;
        load_rows(d2, rs2, out2);
        const ItemDesc d3 = load_desc(b, item + 3 * n_warps);

        const CcJob &a = b.job[d0.job & 255];
        const int R = d0.nrows;
        const int j0 = __shfl_sync(full, rs0, 0), j1 = __shfl_sync(full, rs0, R);
        const int Z = j1 - j0;
        const int G = R > 16 ? 2 : 1; // 16-row groups
        const bool keep = (a.flags & TCA_FLAG_KEEP_EMPTY_ROWS) != 0;
        // local row of this lane's nonzero (rows of an item are consecutive)
        int rz = 0;
        for (int r = 1; r < R; r++) rz += (lane >= __shfl_sync(full, rs0, r) - j0) ? 1 : 0;

        for (int n0 = 0; n0 < a.N; n0 += kMmaSliceCols) {
            float acc[2][8][4];
#pragma unroll
            for (int gg = 0; gg < 2; gg++)
#pragma unroll
                for (int t = 0; t < 8; t++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[gg][t][q] = 0.f;
            for (int kb = 0; kb < Z; kb += 32) {
                int col = col0, zr = rz;
                unsigned short val = val0;
                if (kb > 0) { // a row longer than 32 nonzeros: its next 32
                    col = 0;
                    val = 0;
                    zr = 0;
                    if (kb + lane < Z) {
                        col = __ldg(a.p_col + j0 + kb + lane);
                        val = __half_as_ushort(a.p_val[j0 + kb + lane]);
                    }
                }
                const int zc = min(32, Z - kb);
                // stage B rows z = 4 i + lane / 8, 16-byte chunk lane % 8 of the slice
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int z = 4 * i + (lane >> 3), q = lane & 7;
                    const int cz = __shfl_sync(full, col, z);
                    uint4 v = make_uint4(0, 0, 0, 0);
                    if (z < zc && n0 + 8 * q < a.N)
                        v = __ldg(reinterpret_cast<const uint4 *>(a.B + (size_t)cz * a.ldb + n0 + 8 * q));
                    *reinterpret_cast<uint4 *>(ws + z * 128 + ((q ^ (z & 7)) << 4)) = v;
                }
                __syncwarp();
#pragma unroll
                for (int ks = 0; ks < 2; ks++) {
                    if (16 * ks >= zc)
                        break; // uniform
                    // A fragments: k = 16 ks + 2 c4 + {0, 1} (+ 8); rows 16 gg + g (+ 8)
                    uint32_t af[2][4];
                    int kk[4] = {16 * ks + 2 * c4, 16 * ks + 2 * c4 + 1, 16 * ks + 2 * c4 + 8, 16 * ks + 2 * c4 + 9};
                    int rk[4];
                    unsigned short vk[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        rk[u] = __shfl_sync(full, zr, kk[u]);
                        vk[u] = (unsigned short)__shfl_sync(full, (int)val, kk[u]);
                        if (kk[u] >= zc) rk[u] = -1;
                    }
#pragma unroll
                    for (int gg = 0; gg < 2; gg++) {
                        const int r_lo = 16 * gg + g, r_hi = r_lo + 8;
                        auto pk = [&](int u0, int u1, int row) -> uint32_t {
                            const uint32_t lo = rk[u0] == row ? vk[u0] : 0u;
                            const uint32_t hi = rk[u1] == row ? vk[u1] : 0u;
                            return lo | (hi << 16);
                        };
                        af[gg][0] = pk(0, 1, r_lo);
                        af[gg][1] = pk(0, 1, r_hi);
                        af[gg][2] = pk(2, 3, r_lo);
                        af[gg][3] = pk(2, 3, r_hi);
                    }
#pragma unroll
                    for (int p = 0; p < 4; p++) {
                        const int mi = lane >> 3;
                        const int krow = 16 * ks + (lane & 7) + (mi & 1) * 8;
                        const int nch = 2 * p + (mi >> 1);
                        uint32_t bf[4];
                        ldmatrix_x4_trans(ws_addr + krow * 128 + ((nch ^ (krow & 7)) << 4), bf);
                        mma_16816(acc[0][2 * p], af[0], bf[0], bf[1]);
                        mma_16816(acc[0][2 * p + 1], af[0], bf[2], bf[3]);
                        if (G == 2) {
                            mma_16816(acc[1][2 * p], af[1], bf[0], bf[1]);
                            mma_16816(acc[1][2 * p + 1], af[1], bf[2], bf[3]);
                        }
                    }
                }
            }
            // ---- epilogue of the slice, per 16-row group, through shared memory
#pragma unroll
            for (int gg = 0; gg < 2; gg++) {
                if (gg >= G)
                    break;
                __syncwarp();
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    *reinterpret_cast<float2 *>(acc_s + g * kMmaAccStride + 8 * t + 2 * c4) =
                        make_float2(acc[gg][t][0], acc[gg][t][1]);
                    *reinterpret_cast<float2 *>(acc_s + (g + 8) * kMmaAccStride + 8 * t + 2 * c4) =
                        make_float2(acc[gg][t][2], acc[gg][t][3]);
                }
                __syncwarp();
                const int rows = min(16, R - 16 * gg);
                for (int i = 0; 4 * i < rows; i++) {
                    const int rl = 4 * i + (lane >> 3); // row within the group
                    const int r = 16 * gg + rl;          // row within the item
                    const int orow = __shfl_sync(full, out0, r & 31);
                    const int rstart = __shfl_sync(full, rs0, r & 31), rend = __shfl_sync(full, rs0, (r + 1) & 31);
                    const int n = n0 + (lane & 7) * 8;
                    if (rl < rows && n < a.N && !(keep && rstart == rend)) {
                        const float4 v0 = *reinterpret_cast<const float4 *>(acc_s + rl * kMmaAccStride + (lane & 7) * 8);
                        const float4 v1 =
                            *reinterpret_cast<const float4 *>(acc_s + rl * kMmaAccStride + (lane & 7) * 8 + 4);
                        const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
                        OutT *cp = reinterpret_cast<OutT *>(a.C) + (size_t)orow * a.ldc + n;
                        float o[8];
                        if (a.beta != 0.f) {
                            float old[8];
                            load_out<8>(cp, old);
#pragma unroll
                            for (int q = 0; q < 8; q++) o[q] = fmaf(a.alpha, v[q], a.beta * old[q]);
                        } else {
#pragma unroll
                            for (int q = 0; q < 8; q++) o[q] = a.alpha * v[q];
                        }
                        store_out<8>(cp, o);
                    }
                }
            }
        }

        d0 = d1; rs0 = rs1; out0 = out1; col0 = col1; val0 = val1;
        d1 = d2; rs1 = rs2; out1 = out2;
        d2 = d3;
        item += n_warps;
    }
}

// Persistent grid of the stream kernel: enough warps for every item, at most
// the resident blocks of all SMs.
// beside_regs > 0: the launch directly follows a tensor-core launch whose
// one block per SM holds that many registers. It is issued as a programmatic
// dependent of that launch (which triggers at entry), so its blocks start as
// soon as the tensor-core blocks are resident, and its grid is cut to the
// blocks that the SM's registers as a whole leave beside them (two per SM:
// the first starts at once, the second when the first ends -- measured
// faster than both a wider first block and claiming items from a counter
// with more blocks). The kernel reads nothing the tensor-core kernel writes,
// so it never waits on it.
template <typename OutT, int W, bool F8, int CAP>
int launch_stream_cap(const CcBatchT<CAP> &b, int beside_regs, cudaStream_t s)
{
    const int total = b.item_start[b.n_jobs];
    if (b.n_jobs == 0 || total == 0)
        return TCA_OK;
    static int per_sm = 0, regs = 0;
    if (per_sm == 0) {
        int n = 0;
        TCA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, spmm_cc_stream_kernel<OutT, W, F8, CAP>, 256, 0));
        TCA_TRY(block_regs((const void *)spmm_cc_stream_kernel<OutT, W, F8, CAP>, 256, &regs));
        per_sm = n > 0 ? n : 1;
    }
    const int fit = beside_regs > 0 ? std::max(1, std::min(per_sm, (kSmRegs - beside_regs) / regs)) : per_sm;
    const int grid = std::min((total + 7) / 8, kSMs * fit);
    if (beside_regs > 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        TCA_CUDA_TRY(cudaLaunchKernelEx(&cfg, spmm_cc_stream_kernel<OutT, W, F8, CAP>, b));
        return TCA_OK;
    }
    spmm_cc_stream_kernel<OutT, W, F8, CAP><<<grid, 256, 0, s>>>(b);
    TCA_CUDA_TRY(cudaGetLastError());
    return TCA_OK;
}

template <typename OutT, int W, bool F8>
int launch_stream_group(const CcBatch &b, int beside_regs, cudaStream_t s)
{
    if (b.n_jobs == 1) {
        CcBatchT<1> one;
        one.n_jobs = 1;
        one.item_start[0] = b.item_start[0];
        one.item_start[1] = b.item_start[1];
        one.job[0] = b.job[0];
        return launch_stream_cap<OutT, W, F8, 1>(one, beside_regs, s);
    }
    return launch_stream_cap<OutT, W, F8, kMaxCcJobs>(b, beside_regs, s);
}

template <typename OutT>
int launch_mma_group(const CcBatch &b, cudaStream_t s)
{
    const int total = b.item_start[b.n_jobs];
    if (b.n_jobs == 0 || total == 0)
        return TCA_OK;
    static int per_sm = 0;
    if (per_sm == 0) {
        int n = 0;
        TCA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, spmm_cc_mma_kernel<OutT>, kMmaWarps * 32, 0));
        per_sm = n > 0 ? n : 1;
    }
    const int grid = std::min((total + kMmaWarps - 1) / kMmaWarps, kSMs * per_sm);
    spmm_cc_mma_kernel<OutT><<<grid, kMmaWarps * 32, 0, s>>>(b);
    TCA_CUDA_TRY(cudaGetLastError());
    return TCA_OK;
}

// Columns per lane of the stream kernel: 8 for N > 128, 4 for N > 64, else 2.
inline int pick_w(int N) { return N > 128 ? 8 : N > 64 ? 4 : 2; }

template <typename OutT, bool F8>
int launch_stream_w(const CcBatch &b, int w, int beside_regs, cudaStream_t s)
{
    switch (w) {
    case 2: return launch_stream_group<OutT, 2, F8>(b, beside_regs, s);
    case 4: return launch_stream_group<OutT, 4, F8>(b, beside_regs, s);
    default: return launch_stream_group<OutT, 8, F8>(b, beside_regs, s);
    }
}

template <typename OutT>
int launch_cc_typed(const CcBatch &b, int w, bool f8, int beside_regs, cudaStream_t s)
{
    if (w == kCcMma) return launch_mma_group<OutT>(b, s);
    return f8 ? launch_stream_w<OutT, true>(b, w, beside_regs, s) : launch_stream_w<OutT, false>(b, w, beside_regs, s);
}

} // namespace

// Fewer items than this leave warps of the stream kernel without one (16 warps per SM).
constexpr int kFewItems = 16 * kSMs;

int launch_cc_jobs(const SpmmJob *jobs, int n_jobs, int c_dtype, float alpha, float beta, unsigned flags,
                   cudaStream_t s, LaunchList *defer, int beside_regs)
{
    long long all_items = 0; // of all jobs: what fills the warps
    for (int i = 0; i < n_jobs; i++)
        if (jobs[i].N > 0) all_items += jobs[i].tc ? jobs[i].p->n_cc_items : jobs[i].p->n_all_items;
    if (all_items == 0)
        return TCA_OK;
    const bool few = all_items < kFewItems;
    // The rows kernel takes the jobs whose operands do not allow 16-byte
    // accesses (every window of the plan: the tensor-core kernel needs them
    // too), and those whose few rows are long: a row of more than kItemNnz
    // nonzeros is one warp's item in the stream kernel, a serial chain, which
    // only many other items hide (the ragged last window of 401 x 2286 at 93 %,
    // N = 624, 17 rows of 164: 66 us; 14 us here).
    auto long_rows = [&](const SpmmJob &sj) {
        const tca_plan *p = sj.p;
        return !sj.f8 && sj.cc_w == 0 && vec_ok(sj.B, sj.ldb, sj.N, sj.C, sj.ldc, c_dtype) &&
               few && (sj.tc ? p->cc_row0 >= 0 && p->cc_max_row > kItemNnz : p->max_row > kItemNnz);
    };
    for (int kind : {1, 2, 4, 8, -4, -8, -16, -32}) { // columns per lane, or minus the lanes per row (16-byte accesses)
        const int w = kind;
        RowsBatchT<kMaxCcJobs> b;
        b.n_jobs = 0;
        b.block_start[0] = 0;
        auto flush = [&]() -> int {
            if (b.n_jobs == 0)
                return TCA_OK;
            auto run = [c_dtype, w, beside_regs](const RowsBatchT<kMaxCcJobs> &bb, cudaStream_t st) {
                const RowsShape sh = w > 0 ? RowsShape{32, w} : RowsShape{-w, 8};
                return c_dtype == TCA_DTYPE_F16 ? launch_rows_shape<__half>(bb, sh, w < 0, st, beside_regs > 0)
                                                : launch_rows_shape<float>(bb, sh, w < 0, st, beside_regs > 0);
            };
            int status = TCA_OK;
            if (defer) {
                auto held = std::make_shared<RowsBatchT<kMaxCcJobs>>(b);
                defer->push_back([held, run](cudaStream_t st) { return run(*held, st); });
            } else {
                status = run(b, s);
            }
            b.n_jobs = 0;
            return status;
        };
        for (int i = 0; i < n_jobs; i++) {
            const SpmmJob &sj = jobs[i];
            const tca_plan *p = sj.p;
            if (sj.f8 || sj.N <= 0 || p->M == 0)
                continue;
            const bool vec = vec_ok(sj.B, sj.ldb, sj.N, sj.C, sj.ldc, c_dtype);
            if (vec && !long_rows(sj))
                continue;
            const RowsShape sh = rows_shape(sj.N, vec);
            if ((vec ? -sh.lpr : sh.w) != w)
                continue;
            RowsJob a{p->p_row_ptr, p->p_col, p->perm, p->p_val, sj.B, sj.C, p->M, p->K, p->nnz, sj.N, sj.ldb, sj.ldc,
                      0, 0, alpha, beta, flags};
            if (vec && sj.tc) { // the rows of the CUDA-core windows
                a.row_ptr += p->cc_row0;
                a.perm += p->cc_row0;
                a.M = p->cc_row_end - p->cc_row0;
                a.nnz = p->cc_end;
                a.base = p->cc_base;
            }
            rows_add(b, a, sh);
            if (b.n_jobs == kMaxCcJobs)
                TCA_TRY(flush());
        }
        TCA_TRY(flush());
    }
    // groups: (columns per lane, E4M3) -- stream kernel with 2/4/8 columns and
    // the FP16 tensor-core item kernel (kCcMma)
    const int kinds[7][2] = {{2, 0}, {4, 0}, {8, 0}, {kCcMma, 0}, {2, 1}, {4, 1}, {8, 1}};
    for (const auto &kd : kinds) {
        CcBatch b;
        b.n_jobs = 0;
        b.item_start[0] = 0;
        auto flush = [&]() -> int {
            if (b.n_jobs == 0)
                return TCA_OK;
            const int w = kd[0];
            const bool f8 = kd[1] != 0;
            auto run = [c_dtype, w, f8, beside_regs](const CcBatch &bb, cudaStream_t st) {
                return (c_dtype == TCA_DTYPE_F16) ? launch_cc_typed<__half>(bb, w, f8, beside_regs, st)
                                                  : launch_cc_typed<float>(bb, w, f8, beside_regs, st);
            };
            int status = TCA_OK;
            if (defer) {
                auto held = std::make_shared<CcBatch>(b);
                defer->push_back([held, run](cudaStream_t st) { return run(*held, st); });
            } else {
                status = run(b, s);
            }
            b.n_jobs = 0;
            return status;
        };
        for (int i = 0; i < n_jobs; i++) {
            const SpmmJob &sj = jobs[i];
            const tca_plan *p = sj.p;
            const int n_items = sj.tc ? p->n_cc_items : p->n_all_items;
            if (n_items == 0 || sj.N <= 0)
                continue;
            // E4M3 jobs always qualify (B is the library's own aligned copy; C was checked)
            if (!sj.f8 && (!vec_ok(sj.B, sj.ldb, sj.N, sj.C, sj.ldc, c_dtype) || long_rows(sj)))
                continue;
            int w = (sj.cc_w == 2 || sj.cc_w == 4 || sj.cc_w == 8) ? sj.cc_w : pick_w(sj.N);
            if (sj.cc_w == kCcMma && !sj.f8)
                w = kCcMma;
            if (w != kd[0] || (sj.f8 ? 1 : 0) != kd[1])
                continue;
            CcJob &a = b.job[b.n_jobs];
            a.items = sj.tc ? p->cc_items : p->all_items;
            a.perm = p->perm;
            a.p_row_ptr = p->p_row_ptr;
            a.p_col = p->p_col;
            a.p_val = p->p_val;
            a.B = sj.B;
            a.C = sj.C;
            a.p_val8 = p->p_val_f8;
            a.Bq = sj.Bq;
            a.row_scale = p->row_scale;
            a.col_scale = sj.col_scale;
            a.ldq = sj.ldq;
            a.n_items = n_items;
            // few items: the slices of N go to different warps (with many, the
            // repeated loads of an item's rows and nonzeros cost more)
            a.slices = w != kCcMma && few ? (sj.N + 32 * w - 1) / (32 * w) : 1;
            // fewer still: their rows too (an item of 31 rows is a chain of 8
            // rounds of loads: 4096 x 1024 at 80 %, N = 256, 290 items, 11.6 -> 5.1 us)
            // With a few rounds of items the last, partial round counts: halves
            // (32 problems, 5,056 items on 2,368 warps: the step 48.2 -> 46.6
            // us; thirds 48.5: the loads ahead no longer cover an item). They
            // pay where an item is long: its rows several times over N (5,000
            // items of 8 rows of 4, N = 512 30.4 -> 28.7 us, N = 1024 57.4 -> 52.3;
            // of 2 rows of 16, N = 1024 45.6 -> 41.9), or in one pass many rows and
            // few rounds (31 rows of 1, N = 256, 5,000 items 20.1 -> 19.3, 8,500
            // even; 3 rows of 10 14.4 -> 15.2), but not at fewer columns a lane (8 rows of 4,
            // N = 32, 2,600 items 8.3 -> 9.0), nor with a row an item (of 50,
            // N = 256: 19.7 -> 27.5, as halves side by side).
            const long long rows = sj.tc ? std::min((long long)p->M, (long long)p->n_cc * kWindowRows) : p->M;
            const bool halves = sj.N > 32 * w ? rows >= 2LL * n_items && all_items < 4LL * kFewItems
                                              : w == 8 && rows >= 8LL * n_items && 2 * all_items < 5LL * kFewItems;
            a.parts = w == kCcMma ? 1
                      : few       ? (int)std::max(1LL, std::min(4LL, kFewItems / (all_items * a.slices)))
                      : halves    ? 2
                                  : 1;
            a.M = p->M;
            a.K = p->K;
            a.N = sj.N;
            a.ldb = sj.ldb;
            a.ldc = sj.ldc;
            a.alpha = alpha;
            a.beta = beta;
            a.flags = flags;
            b.item_start[b.n_jobs + 1] = b.item_start[b.n_jobs] + a.n_items * a.slices * a.parts;
            b.n_jobs++;
            if (b.n_jobs == kMaxCcJobs)
                TCA_TRY(flush());
        }
        TCA_TRY(flush());
    }
    return TCA_OK;
}

} // namespace tca
