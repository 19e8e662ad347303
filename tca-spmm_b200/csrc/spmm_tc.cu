// spmm_tc.cu -- tensor-core (tcgen05, sm_100a) forward over the dense-enough
// windows of one or many plans.
//
// The reference (src/our_spmm.cu:25-156) uses mma.sync m16n8k8 as a batched
// dot-product engine on one row's nonzeros, of which only the diagonal 8x8
// blocks are useful (:70-72, :123-124), and re-gathers a 64-column slice of B
// per nonzero. Here a 128-row window of sorted rows becomes a sequence of
// dense 128 x 64 A tiles over the window's condensed (distinct) columns; each
// tile multiplies the 64 matching rows of B on the 5th-generation tensor
// cores: D[128 x NT] (FP32, tensor memory) += A[128 x 64] * B[64 x NT].
//
// Work items are (job, window, NT-wide slice of N); persistent CTAs (one per
// SM) stream the chunks of their items through a ring of kStages (A tile,
// B tile) stages, with decoupled roles:
//   * two loader warps: one brings the 64 B rows of a chunk whose columns are
//     64 consecutive rows of B, one TMA box for the whole slice; the other the
//     chunk's pre-rendered, pre-swizzled dense A tile (chunks with >= 512
//     nonzeros: one 16 KB cp.async.bulk) or its packed entries and condensed
//     columns (cp.async.bulk into a staging slot, four chunks ahead);
//   * scatter warps, once those landed and the stage is free, issue a condensed
//     chunk's tile::gather4 (4 rows x 128 bytes each into a 128-byte swizzled
//     N-major tile; padding columns and n >= N are out of the tensor and arrive
//     as zeros) and zero a sparse chunk's A tile and scatter its entries into
//     the swizzled K-major layout;
//   * one MMA lane issues 4 tcgen05.mma (K = 16 each) per chunk into the FP32
//     accumulator in tensor memory and releases the stage with tcgen05.commit;
//   * finally 4 warps read the accumulator (TMEM lane = row) and store
//     alpha * D + beta * C to C[perm[row]] (FP16 or FP32).
//
// What bounds it: a chunk of 128 x 256 x 64 takes the tensor core 512 cycles
// (0.27 us at 1.9 GHz), and loading its 48 KB takes a ring without MMAs 0.38
// us when the images come from HBM (148 CTAs). The loaders decide whether that
// rate is reached: the issue of one TMA instruction takes ~0.1 us, so the
// chunk's two are issued by two warps, by one elected lane each that walks
// ready-made records. %clock traces, 4096 x 4096 at 90 %, N = 1024 (128 CTAs,
// 64 chunks each): one loader warp behind `lane == 0` 0.36 us per chunk,
// elected lane 0.30, two loaders 0.27; the call went from 46.0 to 34.8 us with
// the coalesced stores of store_rows (3.5 -> 2.4 us of a tile's epilogue), the
// 32-problem sweep step from 60.6 to 55.2 us, the 24-layer batch from 100.9 to
// 80.6 us.
// Every mbarrier wait is bounded (about one second of %globaltimer); on
// expiry the CTA records kStatusTimeout in the job's status word and runs to
// completion without hanging. No load uses cluster multicast.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <climits>
#include <functional>
#include <memory>
#include <mutex>
#include <vector>
#include "tca_internal.cuh"
#include "plan.cuh"
#include "ptx.cuh"

namespace tca {
namespace {

constexpr int kBLoaderWarp = 0;  // TMA issue of the B rows
constexpr int kALoaderWarp = 1;  // TMA issue of the A images and entries
constexpr int kMmaWarp = 2;      // TMEM allocation, tcgen05.mma issue
constexpr int kScatterWarp0 = 3; // warps 3-6: scatter of sparse entries, gathers of condensed columns
constexpr int kScatterWarps = 4;
constexpr int kEpiWarp0 = 7;     // warps 7-10: epilogue
constexpr int kEpiThreads = 128;
constexpr int kThreads = 352;
constexpr int kAhead = 4;        // chunks by which the entries of a sparse chunk precede its stage
constexpr int kRecords = 64;     // chunk records of A kept: two batches of 32
constexpr int kRecordsB = 32;    // of B: one
constexpr int kMaxCtaItems = 32;      // work items per persistent CTA
constexpr int kEpiBar = 3;           // named barrier of the epilogue warps
constexpr int kStagingBytes = ((kImageMinNnz + 3) * 4 + 15) & ~15; // entries of a sparse chunk, 16-byte rounded
constexpr int kMaxJobs = 32;                                  // jobs per launch (kernel parameter space)

struct TcJob {
    CUtensorMap tmap_b;    // B as a 2-D tensor {N, K}, box {64, 1}, 128-byte swizzle (gather4 source)
    CUtensorMap tmap_tile; // 64 contiguous rows of B: the same tensor, box {64, 64}, or (tile3d) {64, K, N / 64}, box {64, 64, NT / 64}
    const int4 *win_info; // per tensor-core window: window, first chunk, chunk count
    const int2 *pairs;    // pair kernel: tensor-core window pairs (second -1: alone)
    const int *tile_ptr, *win_cols, *img_idx, *perm, *p_row_ptr;
    const uint32_t *entries;
    const uint8_t *images;   // dense tile images (16 KB FP16 or 8 KB E4M3 each)
    const float *row_scale;  // E4M3: per sorted row
    const float *col_scale;  // E4M3: per column of N
    const __half *B;
    void *C;
    int *status;
    int M, N, ldb, ldc, ntiles;
    int nt;                  // width of its N-slices, at most the kernel's
    int tile3d;              // tmap_tile covers the whole NT-wide slice in one box
    int gathers;             // some chunk's columns are not 64 consecutive ones
    float alpha, beta;
    unsigned flags;
};

// A launch's jobs. The kernel is also built for CAP = 1: a single forward's
// parameter block is then ~0.4 KB instead of ~12 KB (measured: the launch
// took 5-15 us of host time with the full block); and for CAP = kOrdered,
// whose block also carries the order of the items (9 KB more, 1 us of a
// launch that does not need it).
constexpr int kOrdered = kMaxJobs + 1;
template <int CAP>
struct TcBatchT {
    static constexpr int kJobs = CAP == kOrdered ? kMaxJobs : CAP;
    int n_jobs;
    int item_start[kJobs + 1];
    TcJob job[kJobs];
    // Item k of CTA b: b + k * gridDim.x; kOrdered: order[k * gridDim.x + b]
    // (kNoItem: no more), which the host dealt so that the CTAs end together
    // (schedule_items).
    uint16_t order[CAP == kOrdered ? kMaxCtaItems * kSMs : 1];
};
using TcBatch = TcBatchT<kMaxJobs>;
using TcOrdered = TcBatchT<kOrdered>;
constexpr uint16_t kNoItem = 0xffffu;

using namespace ptx;

// kind::f16 instruction descriptor: D FP32, A/B FP16, A K-major, B N-major, M = 128.
__host__ __device__ constexpr uint32_t idesc_f16(int n)
{
    return (1u << 4) | (0u << 7) | (0u << 10) | (0u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accum)
                 : "memory");
}
__device__ __forceinline__ void umma_f8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accum)
                 : "memory");
}
__device__ __forceinline__ void store8_out(__half *p, const float *v, float alpha, float beta)
{
    uint4 u;
    __half2 *h = reinterpret_cast<__half2 *>(&u);
    if (beta != 0.f) {
        uint4 o = *reinterpret_cast<const uint4 *>(p);
        const __half2 *oh = reinterpret_cast<const __half2 *>(&o);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __half22float2(oh[i]);
            h[i] = __floats2half2_rn(fmaf(alpha, v[2 * i], beta * f.x), fmaf(alpha, v[2 * i + 1], beta * f.y));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(alpha * v[2 * i], alpha * v[2 * i + 1]);
    }
    *reinterpret_cast<uint4 *>(p) = u;
}
__device__ __forceinline__ void store8_out(float *p, const float *v, float alpha, float beta)
{
    float o[8];
    if (beta != 0.f) {
        float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
        const float old[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = fmaf(alpha, v[i], beta * old[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = alpha * v[i];
    }
    reinterpret_cast<float4 *>(p)[0] = make_float4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(o[4], o[5], o[6], o[7]);
}

// Shared memory (1024-byte aligned base): kStages x (A tile | B tile),
// kSlots entry staging buffers, the chunk records of both loaders, the CTA's item table,
// mbarriers and the TMEM slot.
// F8: E4M3 operands -- an 8 KB A tile (64-byte swizzled K-major) and 64 x NT
// byte B tiles, so the ring holds more stages.
template <int NT, bool F8> struct TcCfg {
    static constexpr int kElem = F8 ? 1 : 2;
    static constexpr int kATileBytes = kWindowRows * kChunkCols * kElem;
    static constexpr int kBoxCols = 128 / kElem; // N columns per 128-byte swizzle atom / TMA box
    static constexpr int kStages = F8 ? (NT == 256 ? 8 : 11) : (NT == 256 ? 4 : NT == 128 ? 6 : 8);
    static constexpr int kBTileBytes = kChunkCols * NT * kElem;
    static constexpr int kStage = kATileBytes + kBTileBytes;
    static constexpr int kStagingOff = kStages * kStage;
    // entry staging slots: kStages + kAhead, rounded up to a multiple of the scatter warps (see the scatter role)
    static constexpr int kSlots = (kStages + kAhead + kScatterWarps - 1) / kScatterWarps * kScatterWarps;
    static constexpr int kColsOff = kStagingOff + kSlots * kStagingBytes; // int4 [kSlots][16]: condensed columns
    static constexpr int kRecOff = kColsOff + kSlots * kChunkCols * 4;    // TcRecordA [kRecords], TcRecordB [kRecordsB]
    static constexpr int kItemOff = kRecOff + kRecords * 32 + kRecordsB * 16;            // int4 [kMaxCtaItems]
    static constexpr int kPendOff = kItemOff + kMaxCtaItems * 16;         // int4 [kSlots]: stage, entries, item (-1: no gather)
    static constexpr int kCumOff = kPendOff + kSlots * 16;                // int [kMaxCtaItems + 4]: first chunk of each item
    static constexpr int kScaleOff = kCumOff + (kMaxCtaItems + 4) * 4;    // E4M3: float [2][NT] column scales
    static constexpr int kBarOff = kScaleOff + (F8 ? 2 * NT * 4 : 0);
    // full, empty [kStages]; staged [kSlots]; accum_full, accum_empty [2]; drain; TMEM slot
    static constexpr int kSmem = kBarOff + (2 * kStages + kSlots + 5) * 8 + 8;
    // of the SM's 228 KB, 1 KB per resident block is reserved: this block and two of the CUDA-core kernel
    // (300 bytes more for E4M3 at N = 256 left room for one: 32-problem step 52.5 -> 63.1 us)
    static_assert(kSmem + 3 * 1024 <= 228 * 1024, "room for the CUDA-core blocks beside this one");
    static_assert(kSmem <= 227 * 1024, "shared memory budget");
    static_assert(kStage % 1024 == 0 && kATileBytes % 1024 == 0, "swizzled tiles need 1024-byte alignment");
    static_assert(kStagingOff % 16 == 0 && kStagingBytes % 16 == 0 && kPendOff % 16 == 0, "16-byte alignment");
    static_assert(kRecOff % 16 == 0 && kItemOff % 16 == 0 && kBarOff % 8 == 0, "aligned regions");
};

// Work item (job, tensor-core window, N slice) -> table entry {window,
// first chunk, chunk count, job << 16 | N-slice index}.
template <typename Batch>
__device__ __forceinline__ int4 decode_item(const Batch &batch, int item)
{
    int j = 0, hi = batch.n_jobs - 1; // the last job whose first item is <= item
    while (j < hi) {
        const int mid = (j + hi + 1) >> 1;
        if (batch.item_start[mid] <= item) j = mid;
        else hi = mid - 1;
    }
    const TcJob &a = batch.job[j];
    prefetch_tensormap(&a.tmap_tile);
    const int local = item - batch.item_start[j];
    const int4 wi = __ldg(a.win_info + local / a.ntiles);
    return make_int4(wi.x, wi.y, wi.z, (j << 16) | (local % a.ntiles));
}

// A chunk as the two loaders issue it, in shared memory.
struct __align__(16) TcRecordA {
    const void *src;  // dense image or (16-byte aligned) first entry
    const int *cols;  // condensed chunk: its columns, else NULL
    int bytes;        // of src: kATileBytes for an image, fewer for entries
    int ent;          // entries: count << 2 | entries before the first one
    int item;
};
constexpr int kSlabBits = 26;
constexpr uint32_t kSlabMask = (1u << kSlabBits) - 1u;
struct __align__(16) TcRecordB {
    const CUtensorMap *map;
    int col0;   // first of 64 consecutive columns; -1: condensed ones, whose rows a scatter warp gathers
    uint32_t x; // 128-byte slab of n0 | slabs of the slice << kSlabBits | top bit: one 3-D box
};

// 16-byte unit u of an output row: alpha x 8 accumulators as FP16, or 4 as FP32.
template <typename OutT> __device__ __forceinline__ uint4 pack_unit(const float *v, float alpha)
{
    uint4 u;
    if constexpr (sizeof(OutT) == 2) {
        __half2 *h = reinterpret_cast<__half2 *>(&u);
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(alpha * v[2 * i], alpha * v[2 * i + 1]);
    } else {
        u = make_uint4(__float_as_uint(alpha * v[0]), __float_as_uint(alpha * v[1]), __float_as_uint(alpha * v[2]),
                       __float_as_uint(alpha * v[3]));
    }
    return u;
}

// The warp's 32 accumulator rows (lane = row, its row of C in out_row, -1:
// none) times alpha, NT columns from n0 on, for beta = 0. Tensor memory gives
// a lane its own row, but 32 lanes storing 16 bytes to 32 rows touch 32 lines
// per instruction (measured: 3.5 us for a 128 x 256 FP16 tile). So groups of
// four lanes transpose four 16-byte units among themselves by shuffles, and an
// instruction stores 64 consecutive bytes of each of 8 rows.
template <int NT, typename OutT, bool F8>
__device__ __forceinline__ void store_rows(uint32_t acc, OutT *C, int ldc, int out_row, int n0, int N, float alpha,
                                           float sa, const float *sb, int lane)
{
    constexpr int kUnit = 16 / (int)sizeof(OutT); // columns per unit
    const int i = lane & 3;
    int rows[4]; // rows of C that this lane stores to: those of its group
#pragma unroll
    for (int u = 0; u < 4; u++) rows[u] = __shfl_sync(0xffffffffu, out_row, (lane & ~3) + u);
    for (int cb = 0; cb < NT / 32; cb++) {
        if (n0 + cb * 32 >= N)
            break; // uniform across the warp
        uint32_t r[32];
        tmem_ld32(acc + (uint32_t)(cb * 32), r);
        float *f = reinterpret_cast<float *>(r);
        if constexpr (F8) { // dequantise: row scale x column scale
#pragma unroll
            for (int q = 0; q < 32; q++) f[q] *= sa * sb[cb * 32 + q];
        }
#pragma unroll
        for (int h = 0; h < 32 / (4 * kUnit); h++) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = pack_unit<OutT>(f + (h * 4 + u) * kUnit, alpha);
            // 4 x 4 transpose: afterwards v[u] is unit i of the group's row u
#pragma unroll
            for (int m = 1; m < 4; m <<= 1) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (u & m)
                        continue;
                    const bool hi = (lane & m) != 0;
                    uint4 x = hi ? v[u] : v[u | m];
                    x.x = __shfl_xor_sync(0xffffffffu, x.x, m);
                    x.y = __shfl_xor_sync(0xffffffffu, x.y, m);
                    x.z = __shfl_xor_sync(0xffffffffu, x.z, m);
                    x.w = __shfl_xor_sync(0xffffffffu, x.w, m);
                    if (hi) v[u] = x;
                    else v[u | m] = x;
                }
            }
            const int n = n0 + cb * 32 + (h * 4 + i) * kUnit;
            if (n < N) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (rows[u] >= 0)
                        *reinterpret_cast<uint4 *>(C + (size_t)rows[u] * ldc + n) = v[u];
            }
        }
    }
}

// Persistent CTAs, one per SM: CTA b processes its work items (TcBatchT; at
// most kMaxCtaItems), as one continuous stream of total_chunks chunks
// through the stage ring; every role runs over exactly those chunks. Roles
// (kThreads threads):
//   warps 0 and 1 (loaders of B and of A): a TMA instruction takes its issuer
//     about 0.1 us (a %clock trace), so each chunk's two go out from two
//     warps. The chunk records -- tensor map and coordinates; image or entry
//     range -- are made 32 at a time, one per lane, from loads issued 32
//     chunks ahead, and kept in shared memory, so that one elected lane can
//     walk the chunks alone: acquire the stage ("empty"), set its part of the
//     "full" transaction count and issue. Both do the first two for every
//     chunk, whoever issues its copies: "full" then needs them once per pass
//     over the ring, and "empty" holds them back, so neither is ever more than
//     one phase from a barrier it waits on or arrives at (a parity tells no
//     more apart; a loader that skipped chunks would run ahead, or fall
//     behind, by whole passes). B: ONE 3-D box of 64 rows x NT
//     columns for a direct chunk (64-column slabs as the third dimension; 2-D
//     boxes of one slab each when N is not whole slabs), nothing for a
//     condensed one, whose gathers a scatter warp issues. A: the dense image
//     (cp.async.bulk); and the release of a sparse or condensed chunk to the
//     scatter warps ("staged"), whose entries and columns were sent for kAhead
//     chunks before (cp.async.bulk into a staging slot, completing on its
//     "staged").
//     Jobs of narrower N-slices than the kernel's run in the same launch
//     (smaller boxes, narrower MMAs).
//   warp 2, one lane (MMA): per chunk wait "full"; on an item's first chunk
//     wait until its TMEM accumulator buffer (item parity) is drained
//     ("accum_empty"); 4 x tcgen05.mma (2 for E4M3); commit "empty"; on the
//     item's last chunk commit "accum_full".
//   warps 3-6 (scatter): the q-th sparse or condensed chunk belongs to warp
//     q % 4, which, once its entries and columns are in and the stage is free
//     ("staged"), issues the tile::gather4 of a condensed chunk's B rows and,
//     for a sparse chunk, zeroes the A tile, writes the entries into the
//     swizzled layout and arrives on "full" -- while the B rows are still on
//     their way. Direct image chunks pass them by. A warp issues a gather every
//     32 ns, 64 of them per chunk at N = 256, so one loader warp would pace the
//     ring (2000 x 16384 at 99.6 %, sparse chunks, N = 256: 102 us against 42;
//     15246 x 12743 with a few full columns, 4 in 10 chunks images, N = 128: 74
//     us against 28; 12799 x 19423, half of them, N = 256: 65 against 22);
//     the loader of B counts the bytes in, before or after they land ("full"
//     cannot complete without its arrival). A warp per chunk and not all four
//     per chunk: the steps of a chunk are a chain of ~0.6 us, and four chunks
//     then run through it at once.
//     Chunk q uses slot q % kSlots; it is filled when chunk g is issued, at most
//     kAhead chunks before its own, so chunk q - kSlots lies at least kStages
//     chunks before g and is consumed; kSlots is a multiple of 4, so a slot
//     always belongs to one warp and no wait is more than one phase behind its
//     barrier.
//   warps 7-10 (epilogue): per item wait "accum_full", tcgen05.ld the rows
//     (warp w reads TMEM lanes 32 (w % 4) ..), alpha/beta, store to C[perm],
//     arrive "accum_empty" -- overlapping the next item's main loop.
// 64 registers a thread: two blocks of the CUDA-core kernel then fit beside
// this one on an SM.
template <int NT, typename OutT, bool F8, int CAP = kMaxJobs>
__global__ void __maxnreg__(64) spmm_tc_kernel(const __grid_constant__ TcBatchT<CAP> batch)
{
    using Cfg = TcCfg<NT, F8>;
    constexpr int S = Cfg::kStages;
    constexpr int kATileBytes = Cfg::kATileBytes;
    extern __shared__ __align__(1024) uint8_t smem[];
    int4 *pend = reinterpret_cast<int4 *>(smem + Cfg::kPendOff);
    TcRecordA *rec_a = reinterpret_cast<TcRecordA *>(smem + Cfg::kRecOff);
    TcRecordB *rec_b = reinterpret_cast<TcRecordB *>(rec_a + kRecords);
    int4 *items = reinterpret_cast<int4 *>(smem + Cfg::kItemOff);
    int *cum = reinterpret_cast<int *>(smem + Cfg::kCumOff);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + Cfg::kBarOff);
    uint64_t *empty = full + S;
    uint64_t *staged = empty + S;               // [kSlots]
    uint64_t *acc_full = staged + Cfg::kSlots; // [2]
    uint64_t *acc_empty = acc_full + 2;         // [2]
    uint64_t *drain = acc_empty + 2;            // the MMA lane's last commit: every MMA it issued has completed
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);

    // A CUDA-core launch that follows on the stream as a programmatic
    // dependent may start as soon as every block of this grid is resident: it
    // reads nothing this kernel writes (the two paths own disjoint rows of C).
    // E4M3: both read what the quantization before them writes, so the trigger
    // comes after this grid's own wait for it, below.
    if constexpr (!F8)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int total = batch.item_start[batch.n_jobs];
    // this CTA's items (kOrdered: counted by the loaders, below)
    int n_items = blockIdx.x < total ? min(kMaxCtaItems, (total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) : 0;
    // a job's N-slice width: a single forward runs in the kernel of its own width
    auto width = [](const TcJob &a) { return CAP == 1 ? NT : a.nt; };
    if (smem_u32(smem) & 1023u) { // the swizzled tiles and TMA destinations need a 1024-byte aligned base
        if (threadIdx.x == 0 && total > 0)
            atomicOr(batch.job[0].status, kStatusLayout);
        return;
    }
    // chunk g of the stream: its item (found from `k` on) and its place in the plan
    auto locate = [&](int g, int &k) -> int {
        while (k + 1 < n_items && cum[k + 1] <= g) k++;
        const int4 it = items[k];
        // windows of one problem start their chunk walks at different
        // chunks, so that they do not read the same rows of B at once
        int i = g - cum[k] + it.x % it.z;
        if (i >= it.z) i -= it.z;
        return it.y + i;
    };
    // a loader's chunk metadata from the plan, one chunk per lane: the columns
    // of its ends, its image, and for A its entry range
    int k = 0, c = 0, m0 = 0, m1 = 0, img = -1, c0 = 0, c1 = 0;
    auto fetch = [&](int g, int k0) {
        k = k0;
        if (g < cum[n_items]) {
            c = locate(g, k);
            const TcJob &a = batch.job[items[k].w >> 16];
            c0 = __ldg(a.win_cols + (size_t)c * kChunkCols);
            c1 = __ldg(a.win_cols + (size_t)c * kChunkCols + kChunkCols - 1);
            img = __ldg(a.img_idx + c);
            if (warp == kALoaderWarp) {
                m0 = __ldg(a.tile_ptr + c);
                m1 = __ldg(a.tile_ptr + c + 1);
            }
        }
    };
    if (warp == kBLoaderWarp || warp == kALoaderWarp) {
        // The item table and the first chunk of each item (a warp scan of the
        // chunk counts), by both loaders alike -- the same values to the same
        // places --, so that each can go on to its first records' loads, on
        // their way during the rest of the set-up (a chain of cold misses:
        // parameters, window list, chunk lists, then the data).
        int z = 0;
        int item = (int)blockIdx.x + lane * (int)gridDim.x;
        if constexpr (CAP == kOrdered) {
            item = batch.order[lane * (int)gridDim.x + (int)blockIdx.x];
            n_items = __popc(__ballot_sync(0xffffffffu, item != kNoItem));
            if (lane == 0)
                cum[kMaxCtaItems + 1] = n_items;
        }
        if (lane < n_items) {
            const int4 it = decode_item(batch, item);
            items[lane] = it;
            z = it.z;
        }
        int sum = z;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        cum[lane + 1] = sum;
        if (lane == 0) cum[0] = 0;
        __syncwarp();
        fetch(lane, 0);
    } else if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * NT)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else if (warp == kScatterWarp0 && lane == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 2); // both loaders' parts (of a sparse chunk: the loader of B's and a scatter warp's)
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < Cfg::kSlots; s++) mbar_init(&staged[s], 1);
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kEpiThreads);
        }
        mbar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if constexpr (CAP == kOrdered)
        n_items = cum[kMaxCtaItems + 1];
    if constexpr (F8) {
        asm volatile("griddepcontrol.wait;" ::: "memory"); // B is quantized
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    bool ok = true;
    const int total_chunks = cum[n_items]; // of this CTA's items: every role runs over exactly these

    if (warp == kBLoaderWarp) {
        // ---------------- loader of B ----------------
        // records of chunks g0 .. g0 + 31 (fetched), and the loads of the next 32
        auto make_records = [&](int g0) {
            if (g0 + lane < total_chunks) {
                const int4 it = items[k];
                const TcJob &a = batch.job[it.w >> 16];
                TcRecordB r;
                const int n0 = (it.w & 0xffff) * width(a);
                r.map = &a.tmap_tile;
                r.col0 = c0 >= 0 && c1 == c0 + kChunkCols - 1 ? c0 : -1;
                r.x = (uint32_t)(n0 / Cfg::kBoxCols) | (uint32_t)(width(a) / Cfg::kBoxCols) << kSlabBits |
                      (a.tile3d ? 0x80000000u : 0u);
                rec_b[(g0 + lane) % kRecordsB] = r;
            }
            fetch(g0 + 32 + lane, __shfl_sync(0xffffffffu, k, 31));
            __syncwarp();
        };
        auto boxes = [](const TcRecordB &r) { return CAP == 1 ? NT / Cfg::kBoxCols : (int)(r.x >> kSlabBits & 7u); }; // 128-byte-wide ones of its slice
        // a direct chunk's B rows into stage s
        auto issue_boxes = [&](const TcRecordB &r, int s) {
            const uint32_t b_s = smem_u32(smem + s * Cfg::kStage) + kATileBytes;
            const int slab = (int)(r.x & kSlabMask);
            if (r.x >> 31) {
                tma_tile3d(b_s, r.map, 0, r.col0, slab, &full[s]);
            } else {
                for (int bx = 0; bx < boxes(r); bx++)
                    tma_tile2d(b_s + bx * (kChunkCols * 128), r.map, (slab + bx) * Cfg::kBoxCols, r.col0, &full[s]);
            }
        };
        int s = 0;
        uint32_t phase = 1; // of "empty": the first pass over the ring finds every stage free
        for (int g = 0; g < total_chunks;) {
            make_records(g);
            const int ge = min(total_chunks, g + 32);
            int s1 = s;
            uint32_t phase1 = phase;
            if (elect_one()) {
                TcRecordB r = rec_b[g % kRecordsB];
                for (int h = g; h < ge; h++) {
                    const TcRecordB nxt = rec_b[(h + 1) % kRecordsB];
                    if (!mbar_wait(&empty[s1], phase1)) { ok = false; break; }
                    mbar_arrive_expect_tx(&full[s1], (uint32_t)boxes(r) * (kChunkCols * 128));
                    if (r.col0 >= 0)
                        issue_boxes(r, s1);
                    if (++s1 == S) { s1 = 0; phase1 ^= 1; }
                    r = nxt;
                }
            }
            if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
            // the ring's place after this run of chunks, which the elected lane walked alone
            phase ^= (uint32_t)((s + ge - g) / S) & 1u;
            s = (s + ge - g) % S;
            g = ge;
        }
    } else if (warp == kALoaderWarp) {
        // ---------------- loader of A ----------------
        auto make_records = [&](int g0) {
            if (g0 + lane < total_chunks) {
                const TcJob &a = batch.job[items[k].w >> 16];
                TcRecordA r;
                r.src = img >= 0 ? (const void *)(a.images + (size_t)img * kATileBytes)
                                 : (const void *)(a.entries + (m0 & ~3));
                r.bytes = img >= 0 ? kATileBytes : m1 > m0 ? ((m1 - (m0 & ~3)) * 4 + 15) & ~15 : 0;
                r.ent = ((m1 - m0) << 2) | (m0 & 3);
                r.cols = c0 >= 0 && c1 == c0 + kChunkCols - 1 ? nullptr : a.win_cols + (size_t)c * kChunkCols;
                r.item = k;
                rec_a[(g0 + lane) % kRecords] = r;
            }
            fetch(g0 + 32 + lane, __shfl_sync(0xffffffffu, k, 31));
            __syncwarp();
        };
        // send for the entries (a sparse chunk) and the columns (a condensed one) of chunk h
        int pslot = 0, slot = 0, s = 0;
        uint32_t phase = 1;
        auto prefetch = [&](int h) {
            if (h < total_chunks) {
                const TcRecordA r = rec_a[h % kRecords];
                const bool image = r.bytes == kATileBytes;
                if (!image && r.bytes) {
                    mbar_expect_tx(&staged[pslot], (uint32_t)r.bytes);
                    bulk_copy_g2s(smem_u32(smem + Cfg::kStagingOff + pslot * kStagingBytes), r.src, (uint32_t)r.bytes,
                                  &staged[pslot]);
                }
                if (r.cols) {
                    mbar_expect_tx(&staged[pslot], kChunkCols * 4);
                    bulk_copy_g2s(smem_u32(smem + Cfg::kColsOff + pslot * kChunkCols * 4), r.cols, kChunkCols * 4,
                                  &staged[pslot]);
                }
                if ((!image || r.cols) && ++pslot == Cfg::kSlots) pslot = 0;
            }
        };
        make_records(0);
        // one lane walks the chunks; every lane joins it to make the next records
        const bool leader = elect_one();
        if (leader)
            for (int h = 0; h < kAhead; h++) prefetch(h);
        for (int g = 0; g < total_chunks;) {
            if (g > 0)
                make_records(g + kAhead); // g + kAhead is a multiple of 32 here
            const int ge = min(total_chunks, (g + kAhead) / 32 * 32 + 32 - kAhead);
            if (leader) {
                TcRecordA r = rec_a[g % kRecords];
                for (int h = g; h < ge; h++) {
                    const TcRecordA nxt = rec_a[(h + 1) % kRecords];
                    if (!mbar_wait(&empty[s], phase)) { ok = false; break; }
                    const bool image = r.bytes == kATileBytes;
                    if (image) {
                        mbar_arrive_expect_tx(&full[s], kATileBytes);
                        bulk_copy_g2s(smem_u32(smem + s * Cfg::kStage), r.src, kATileBytes, &full[s]);
                    }
                    if (!image || r.cols) {
                        pend[slot] = make_int4(s, r.ent, r.cols ? r.item : -1, image ? 1 : 0);
                        mbar_arrive(&staged[slot]); // of a sparse chunk the scatter warp arrives on "full"
                        if (++slot == Cfg::kSlots) slot = 0;
                    }
                    prefetch(h + kAhead);
                    if (++s == S) { s = 0; phase ^= 1; }
                    r = nxt;
                }
            }
            if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
            g = ge;
        }
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
                        // test hook: the CTA's last accumulator is never announced, so the
            // epilogue's bounded wait for it runs out (TCA_FLAG_TEST_WITHHOLD_ACCUM)
            const bool withhold = (batch.job[0].flags & TCA_FLAG_TEST_WITHHOLD_ACCUM) != 0;
            int s = 0;
            uint32_t phase = 0;
            for (int k = 0; k < n_items && ok; k++) {
                const int b = k & 1;
                const uint32_t d = tmem + (uint32_t)(b * NT);
                // E4M3 has format code 0 in kind::f8f6f4 as FP16 in kind::f16
                const uint32_t idesc = idesc_f16(width(batch.job[items[k].w >> 16]));
                if (k >= 2 && !mbar_wait(&acc_empty[b], ((k >> 1) - 1) & 1)) { ok = false; break; }
                uint32_t accum = 0;
                for (int i = items[k].z; i > 0; i--) {
                    if (!mbar_wait(&full[s], phase)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_s = smem_u32(smem + s * Cfg::kStage), b_s = a_s + kATileBytes;
                    if constexpr (F8) {
                        // 2 x K = 32: A rows of 64 bytes (64-byte swizzle, 8-row groups 512 bytes apart),
                        // B k-rows of 128 bytes (128-byte swizzle, atoms along N 8 KB apart)
#pragma unroll
                        for (int kk = 0; kk < kChunkCols / 32; kk++) {
                            const uint64_t ad = smem_desc(a_s + kk * 32, 16, 512, 4);
                            const uint64_t bd = smem_desc(b_s + kk * 4096, kChunkCols * 128, 1024);
                            umma_f8(d, ad, bd, idesc, kk == 0 ? accum : 1u);
                        }
                    } else {
#pragma unroll
                        for (int kk = 0; kk < kChunkCols / 16; kk++) {
                            const uint64_t ad = smem_desc(a_s + kk * 32, 16, 1024);
                            const uint64_t bd = smem_desc(b_s + kk * 2048, kChunkCols * 128, 1024);
                            umma_f16(d, ad, bd, idesc, kk == 0 ? accum : 1u);
                        }
                    }
                    accum = 1;
                    umma_commit(&empty[s]);
                    if (++s == S) { s = 0; phase ^= 1; }
                }
                if (ok && !(withhold && k == n_items - 1))
                    umma_commit(&acc_full[b]);
            }
            // every MMA issued has completed before the tensor memory is
            // released, also when a role gave up early
            umma_commit(drain);
            if (!mbar_wait(drain, 0))
                ok = false;
        }
        __syncwarp();
    } else if (warp < kEpiWarp0) {
        // ---------------- scatter ----------------
        int n_mine = 0, k = 0; // sparse or condensed chunks of this CTA
        for (int g0 = 0; g0 < total_chunks; g0 += 32) {
            bool mine = false;
            if (g0 + lane < total_chunks) {
                const int c = locate(g0 + lane, k);
                const TcJob &a = batch.job[items[k].w >> 16];
                mine = __ldg(a.img_idx + c) < 0;
                if (a.gathers) {
                    const int first = __ldg(a.win_cols + (size_t)c * kChunkCols);
                    const int last = __ldg(a.win_cols + (size_t)c * kChunkCols + kChunkCols - 1);
                    mine = mine || first < 0 || last != first + kChunkCols - 1;
                }
            }
            n_mine += __popc(__ballot_sync(0xffffffffu, mine));
        }
        for (int q = warp - kScatterWarp0; q < n_mine; q += kScatterWarps) {
            const int slot = q % Cfg::kSlots;
            if (!mbar_wait(&staged[slot], (uint32_t)(q / Cfg::kSlots) & 1u)) { ok = false; break; }
            const int4 pd = pend[slot];
            uint8_t *At = smem + pd.x * Cfg::kStage;
            if (pd.z >= 0) { // its B rows: gather g = lane, lane + 32, .. reads the 4 columns of lane g % 16
                const int4 it = items[pd.z];
                const TcJob &a = batch.job[it.w >> 16];
                const int boxes = width(a) / Cfg::kBoxCols, n0 = (it.w & 0xffff) * width(a);
                const int4 y = reinterpret_cast<const int4 *>(smem + Cfg::kColsOff + slot * kChunkCols * 4)[lane & 15];
                const uint32_t b_s = smem_u32(At) + kATileBytes + (lane & 15) * 512;
                for (int g = lane; g < 16 * boxes; g += 32)
                    tma_gather4(b_s + (g >> 4) * (kChunkCols * 128), &a.tmap_b, n0 + (g >> 4) * Cfg::kBoxCols, y.x, y.y,
                                y.z, y.w, &full[pd.x]);
            }
            if (pd.w) // its A tile is an image
                continue;
#pragma unroll 8
            for (int o = 0; o < kATileBytes / (16 * 32); o++)
                reinterpret_cast<uint4 *>(At)[lane + o * 32] = make_uint4(0, 0, 0, 0);
            __syncwarp();
            const uint32_t *st = reinterpret_cast<const uint32_t *>(smem + Cfg::kStagingOff + slot * kStagingBytes);
            const int end = (pd.y >> 2) + (pd.y & 3);
            // eight loads before the first store: the compiler may not move a
            // shared load over a shared store, and one entry at a time is a
            // chain of ~100 cycles
            for (int e = (pd.y & 3) + lane; e < end; e += 8 * 32) {
                uint32_t v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = e + u * 32 < end ? st[e + u * 32] : 0xffffffffu; // row 1023: none
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    if (v[u] == 0xffffffffu)
                        continue;
                    if constexpr (F8)
                        At[swz64_offset(v[u] >> 22, (v[u] >> 16) & 63u)] = (uint8_t)(v[u] & 0xffu);
                    else
                        *reinterpret_cast<uint16_t *>(At + swz128_offset(v[u] >> 22, (v[u] >> 16) & 63u)) =
                            (uint16_t)(v[u] & 0xffffu);
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&full[pd.x]);
        }
    } else {
        // ---------------- epilogue ----------------
        const int quarter = warp & 3;
        for (int k = 0; k < n_items; k++) {
            const int4 it = items[k];
            const TcJob &a = batch.job[it.w >> 16];
            const int nt = width(a), n0 = (it.w & 0xffff) * nt, n_end = min(a.N, n0 + nt);
            const int i = it.x * kWindowRows + quarter * 32 + lane;
            int out_row = -1;
            if (i < a.M && !((a.flags & TCA_FLAG_KEEP_EMPTY_ROWS) && a.p_row_ptr[i + 1] == a.p_row_ptr[i]))
                out_row = a.perm[i];
            const int b = k & 1;
            if constexpr (F8) {
                // the item's column scales, once, into shared memory (buffer b
                // was last read for item k - 2, which every epilogue thread
                // finished before the barrier of item k - 1)
                float *sc = reinterpret_cast<float *>(smem + Cfg::kScaleOff) + b * NT;
                for (int c = quarter * 32 + lane; c < nt; c += kEpiThreads)
                    sc[c] = n0 + c < a.N ? __ldg(a.col_scale + n0 + c) : 0.f;
            }
            uint32_t got = 0;
            if (lane == 0)
                got = mbar_wait(&acc_full[b], (k >> 1) & 1) ? 1u : 0u;
            got = __shfl_sync(0xffffffffu, got, 0);
            // the four warps agree, so that none is left at a later barrier
            if (!named_bar_and(kEpiBar, kEpiThreads, got != 0)) { ok = false; break; }
            tc_fence_after();
            OutT *Crow = out_row >= 0 ? reinterpret_cast<OutT *>(a.C) + (size_t)out_row * a.ldc : nullptr;
            float sa = 1.f;
            if constexpr (F8)
                sa = (i < a.M) ? a.row_scale[i] : 0.f;
            const float *sb0 = reinterpret_cast<const float *>(smem + Cfg::kScaleOff) + b * NT;
            const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * NT);
            if (a.beta == 0.f)
                store_rows<NT, OutT, F8>(acc, reinterpret_cast<OutT *>(a.C), a.ldc, out_row, n0, n_end, a.alpha, sa, sb0,
                                         lane);
            for (int cb = 0; a.beta != 0.f && cb < NT / 16; cb++) {
                const int n = n0 + cb * 16;
                if (n >= n_end)
                    break; // uniform across the warp
                uint32_t r[16];
                tmem_ld16(acc + (uint32_t)(cb * 16), r);
                if constexpr (F8) { // dequantise: row scale x column scale (staged above; the barrier orders it)
                    float *f = reinterpret_cast<float *>(r);
                    const float *sb = sb0 + cb * 16;
#pragma unroll
                    for (int q = 0; q < 16; q++) f[q] *= sa * sb[q];
                }
                if (Crow) {
                    store8_out(Crow + n, reinterpret_cast<const float *>(r), a.alpha, a.beta);
                    if (n + 8 < n_end)
                        store8_out(Crow + n + 8, reinterpret_cast<const float *>(r) + 8, a.alpha, a.beta);
                }
            }
            tc_fence_before();
            mbar_arrive(&acc_empty[b]);
        }
    }

    tc_fence_before();
    if (__syncthreads_or(!ok)) {
        // A role gave up after a bounded wait: record it, then give bulk
        // copies that loaders issued and nobody consumed a bounded time
        // (1 ms; a copy lands within microseconds) to land before this
        // CTA's shared memory is released.
        if (threadIdx.x == 0) {
            if (n_items > 0)
                atomicOr(batch.job[items[0].w >> 16].status, kStatusTimeout);
            const uint64_t t0 = global_ns();
            while (global_ns() - t0 < 1000000ull) {
            }
        }
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * NT) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Window pairs on CTA pairs (tcgen05 cta_group::2).
//
// A chunk of the kernel above holds 48 KB (A tile 16 KB, B tile 64 x 256 x 2)
// and its ring fits 4 stages; the chunk time is the ring's round trip (loads
// land ~2 us after issue whatever their size, measured) over those 4 stages.
// Two windows whose chunks have the same columns (direct windows that touch
// every 64-column block of K) share every B tile, so a cluster of two CTAs on
// two SMs runs them as one M = 256 product: each CTA loads its own window's A
// tile and HALF of the B tile (128 of the 256 columns of N), the first CTA's
// single MMA lane multiplies both (tcgen05.mma.cta_group::2 reads the
// operands from both CTAs' shared memory) and each CTA's tensor memory holds
// its own window's 128 x 256 accumulator. A stage is then 32 KB (E4M3:
// 16 KB), so 6 (E4M3: 12) fit. A window without a partner runs with an empty
// one (zero A tile, no stores).
//   Opt-in (tca_plan_opts_t.pair_windows): correct, but measured slower on the
// 32-problem sweep step (FP16 63 us against 50 us for spmm_tc_kernel, E4M3 59
// against 37 us). Traces show each CTA's chunks completing one per ~0.9 us
// (FP16) / ~0.65 us (E4M3) whatever the stage count (4 to 12) and however the
// partner's completions are waited for -- half the per-SM throughput of the
// single-window kernel -- so the halved B bytes per SM buy nothing, and 192
// pair items on 74 CTA pairs balance worse than 352 items on 148 CTAs.
//   Per CTA the roles are those of spmm_tc_kernel. Synchronisation between
// the two: the second CTA's warp 5 forwards each stage's completion ("full",
// its loads landed and scattered) to the first CTA's "peer_full"; the MMA
// lane releases the stage in both CTAs and announces finished accumulators
// to both epilogues with multicast commits; each epilogue reports its drained
// accumulator to the first CTA's "acc_empty" (count 2). Every wait is bounded
// as above; waits on phases the partner completes poll with test_wait. At
// exit each CTA waits (bounded) until its partner has made its last access to
// this CTA's shared memory. No load uses multicast.
constexpr int kPairN = 256;
// roles of the pair kernel
namespace pair {
constexpr int kScatterThreads = 128; // warps 0-3: sparse-entry scatter
constexpr int kLoaderWarp = 4;       // TMA issue, chunks g = 0 (mod kLoaders)
constexpr int kMmaWarp = 5;          // TMEM allocation, tcgen05.mma issue
constexpr int kEpiWarp0 = 6;         // warps 6-9: epilogue
constexpr int kLoaderWarp1 = 10;     // warps 10..: TMA issue, chunks g = 1, 2, .. (mod kLoaders)
constexpr int kLoaders = 4;          // loader warps, each issuing every kLoaders-th chunk
constexpr int kThreads = 320 + (kLoaders - 1) * 32;
} // namespace pair

template <bool F8> struct Tc2Cfg {
    static constexpr int kElem = F8 ? 1 : 2;
    static constexpr int kATileBytes = kWindowRows * kChunkCols * kElem;
    static constexpr int kHalfCols = kPairN / 2;             // columns of N whose B rows this CTA loads
    static constexpr int kBoxCols = 128 / kElem;             // N columns per 128-byte swizzle atom / TMA box
    static constexpr int kBoxes = kHalfCols / kBoxCols;      // 2 (FP16) or 1 (E4M3)
    static constexpr int kBTileBytes = kChunkCols * kHalfCols * kElem;
    static constexpr int kStage = kATileBytes + kBTileBytes; // 32 KB / 16 KB
    static constexpr int kStages = F8 ? 12 : 6;
    static constexpr int kStagingOff = kStages * kStage;
    static constexpr int kPendOff = kStagingOff + kStages * kStagingBytes;
    static constexpr int kPend2Off = kPendOff + kStages * 16;
    static constexpr int kItemOff = kPend2Off + kStages * 16; // int4 [kMaxCtaItems][2]
    static constexpr int kScaleOff = kItemOff + kMaxCtaItems * 32;
    static constexpr int kBarOff = kScaleOff + (F8 ? 2 * kPairN * 4 : 0);
    // full, empty, staged, peer_full [kStages]; acc_full, acc_empty [2]; drain; bye; 4 flags, TMEM slot
    static constexpr int kSmem = kBarOff + (4 * kStages + 6) * 8 + 24;
    static_assert(kSmem <= 227 * 1024, "shared memory budget");
    static_assert(kStage % 1024 == 0 && kATileBytes % 1024 == 0, "swizzled tiles need 1024-byte alignment");
    static_assert(kPendOff % 16 == 0 && kItemOff % 16 == 0 && kBarOff % 16 == 0, "16-byte aligned regions");
    static_assert(kStages % 2 == 0 && pair::kLoaders <= kStages, "two scatter groups; loaders may not lap a stage");
};

// kind::f16 / kind::f8f6f4 instruction descriptor for M = 256 across the pair
// (FP32 D, A K-major, B N-major, N = 256); E4M3 uses format code 0 as FP16.
__host__ __device__ constexpr uint32_t idesc_pair()
{
    return (1u << 4) | (1u << 16) | ((uint32_t)(kPairN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}

__device__ __forceinline__ void umma_pair_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                              uint32_t accum)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accum)
                 : "memory");
}
__device__ __forceinline__ void umma_pair_f8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t accum)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accum)
                 : "memory");
}
// Arrive on the mbarrier at `bar`'s offset in both CTAs of the pair once every
// tcgen05.mma this thread issued has completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}

// Pair work item (job, pair, 256-wide N slice) -> this CTA's two table
// entries: {A chunk base (-1: empty partner), B chunk base, chunk count,
// job << 16 | slice} and {window of its rows (-1: none), rotation base, 0, 0}.
// Both CTAs walk the chunks of the first window's list, so that both load
// the same B rows for the same chunk.
__device__ __forceinline__ void decode_pair_item(const TcBatch &batch, int item, uint32_t rank, int4 *e0, int4 *e1)
{
    int j = 0;
    while (j + 1 < batch.n_jobs && batch.item_start[j + 1] <= item) j++;
    const TcJob &a = batch.job[j];
    const int local = item - batch.item_start[j];
    const int2 pr = a.pairs[local / a.ntiles];
    const int4 w0 = a.win_info[pr.x];
    const int mine = rank == 0 ? pr.x : pr.y;
    const int4 wm = mine >= 0 ? a.win_info[mine] : make_int4(-1, -1, 0, 0);
    *e0 = make_int4(wm.y, w0.y, w0.z, (j << 16) | (local % a.ntiles));
    *e1 = make_int4(wm.x, w0.x, 0, 0);
}

template <typename OutT, bool F8>
__global__ void __launch_bounds__(pair::kThreads, 1) spmm_tc_pair_kernel(const __grid_constant__ TcBatch batch)
{
    using Cfg = Tc2Cfg<F8>;
    constexpr int S = Cfg::kStages;
    constexpr int kATileBytes = Cfg::kATileBytes;
    constexpr int kGathers = 16 * Cfg::kBoxes; // gather4 instructions per condensed chunk
    extern __shared__ __align__(1024) uint8_t smem[];
    int4 *pend = reinterpret_cast<int4 *>(smem + Cfg::kPendOff);
    int4 *pend2 = reinterpret_cast<int4 *>(smem + Cfg::kPend2Off);
    int4 *items = reinterpret_cast<int4 *>(smem + Cfg::kItemOff); // [k][2]
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + Cfg::kBarOff);
    uint64_t *empty = full + S;
    uint64_t *staged = empty + S;
    uint64_t *peer_full = staged + S;    // first CTA: the partner's stage s is full
    uint64_t *acc_full = peer_full + S;  // [2]
    uint64_t *acc_empty = acc_full + 2;  // [2], first CTA: both epilogues drained it
    uint64_t *drain = acc_empty + 2;     // every MMA of the pair has completed
    uint64_t *bye = drain + 1;           // the partner is done with this CTA's shared memory
    volatile int *flag = reinterpret_cast<volatile int *>(bye + 1);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bye + 1) + 4;
    constexpr int kGroupThreads = pair::kScatterThreads / 2;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const uint32_t rank = cluster_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pair_id = (int)blockIdx.x >> 1, n_pairs_grid = (int)gridDim.x >> 1;
    const int total = batch.item_start[batch.n_jobs];
    const int n_items =
        pair_id < total ? min(kMaxCtaItems, (total - 1 - pair_id) / n_pairs_grid + 1) : 0;
    // both CTAs are resident before either touches the other's shared memory
    cluster_sync_all();
    if (smem_u32(smem) & 1023u) { // the same in both CTAs: both leave here, before any shared state
        if (threadIdx.x == 0 && n_items > 0)
            atomicOr(batch.job[0].status, kStatusLayout);
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], kGroupThreads);
            mbar_init(&empty[s], 1);
            mbar_init(&staged[s], 1);
            mbar_init(&peer_full[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2);
        }
        mbar_init(drain, 1);
        mbar_init(bye, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if ((int)threadIdx.x < n_items)
        decode_pair_item(batch, pair_id + (int)threadIdx.x * n_pairs_grid, rank, &items[2 * threadIdx.x],
                         &items[2 * threadIdx.x + 1]);
    if (warp == pair::kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * kPairN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster_sync_all(); // barriers initialised and tensor memory allocated in both CTAs
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    int total_chunks = 0;
    for (int k = 0; k < n_items; k++) total_chunks += items[2 * k].z;

    if (warp == pair::kLoaderWarp || warp >= pair::kLoaderWarp1) {
        // ---------------- loaders (as in spmm_tc_kernel; B: this CTA's half of N) ----------------
        const int ld = warp == pair::kLoaderWarp ? 0 : warp - pair::kLoaderWarp1 + 1;
        auto advance = [&](int &k, int &i) {
            while (k < n_items && i >= items[2 * k].z) { i -= items[2 * k].z; k++; }
        };
        struct Meta { int4 cols; int img, e0, e1; };
        auto fetch = [&](int k, int i, Meta &m) {
            m.cols = make_int4(-1, -1, -1, -1);
            m.img = -1;
            m.e0 = m.e1 = 0;
            if (k < n_items) {
                const int4 it = items[2 * k], it2 = items[2 * k + 1];
                const TcJob &a = batch.job[it.w >> 16];
                const int r = (i + it2.y % it.z) % it.z; // the same chunk order in both CTAs
                if (lane < 16)
                    m.cols = __ldg(reinterpret_cast<const int4 *>(a.win_cols + (size_t)(it.y + r) * kChunkCols) + lane);
                if (it.x >= 0) { // else an empty partner: a zero A tile
                    m.img = __ldg(a.img_idx + it.x + r);
                    m.e0 = __ldg(a.tile_ptr + it.x + r);
                    m.e1 = __ldg(a.tile_ptr + it.x + r + 1);
                }
            }
        };
        int k = 0, i = ld;
        advance(k, i);
        int g = ld;
        auto step = [&](Meta &cur, Meta &nxt) -> bool {
            if (g >= total_chunks || !ok)
                return false;
            int k2 = k, i2 = i + pair::kLoaders;
            advance(k2, i2);
            fetch(k2, i2, nxt);
            const int s = g % S;
            uint32_t got = 1;
            if (lane == 0 && g >= S)
                got = mbar_poll_cluster(&empty[s], ((g / S) - 1) & 1) ? 1u : 0u;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!got) { ok = false; return false; }
            const int4 it = items[2 * k];
            const TcJob &a = batch.job[it.w >> 16];
            const int n0 = (it.w & 0xffff) * kPairN + (int)rank * Cfg::kHalfCols;
            const uint32_t a_s = smem_u32(smem + s * Cfg::kStage), b_s = a_s + kATileBytes;
            if (lane == 0) {
                const int img = cur.img, e0 = cur.e0, e1 = cur.e1, e0a = e0 & ~3;
                pend[s] = make_int4(img, e0, e0a, e1);
                pend2[s] = make_int4((i == 0 ? 1 : 0) | (i == it.z - 1 ? 2 : 0), k & 1, k, 0);
                mbar_expect_tx(&full[s], Cfg::kBTileBytes + (img >= 0 ? kATileBytes : 0));
                if (img >= 0) {
                    bulk_copy_g2s(a_s, a.images + (size_t)img * kATileBytes, kATileBytes, &full[s]);
                    mbar_arrive(&staged[s]);
                } else if (e1 > e0) {
                    const uint32_t bytes = (uint32_t)(((e1 - e0a) * 4 + 15) & ~15);
                    mbar_arrive_expect_tx(&staged[s], bytes);
                    bulk_copy_g2s(smem_u32(smem + Cfg::kStagingOff + s * kStagingBytes), a.entries + e0a, bytes,
                                  &staged[s]);
                } else {
                    mbar_arrive(&staged[s]);
                }
            }
            __syncwarp();
            const int col0 = __shfl_sync(0xffffffffu, cur.cols.x, 0);
            const int col63 = __shfl_sync(0xffffffffu, cur.cols.w, 15);
            if (col0 >= 0 && col63 == col0 + kChunkCols - 1) {
                if (lane < Cfg::kBoxes)
                    tma_tile2d(b_s + lane * (kChunkCols * 128), &a.tmap_tile, n0 + lane * Cfg::kBoxCols, col0,
                               &full[s]);
            } else {
                const int src = lane & 15;
                const int y0 = __shfl_sync(0xffffffffu, cur.cols.x, src);
                const int y1 = __shfl_sync(0xffffffffu, cur.cols.y, src);
                const int y2 = __shfl_sync(0xffffffffu, cur.cols.z, src);
                const int y3 = __shfl_sync(0xffffffffu, cur.cols.w, src);
                for (int q = lane; q < kGathers; q += 32) {
                    const int box = q >> 4;
                    tma_gather4(b_s + box * (kChunkCols * 128) + src * 512, &a.tmap_b, n0 + box * Cfg::kBoxCols, y0,
                                y1, y2, y3, &full[s]);
                }
            }
            k = k2;
            i = i2;
            g += pair::kLoaders;
            return true;
        };
        Meta ma, mb;
        fetch(k, i, ma);
        while (step(ma, mb) && step(mb, ma)) {
        }
    } else if (warp < 4) {
        // ---------------- scatter (as in spmm_tc_kernel, two groups) ----------------
        const int grp = warp >> 1;
        const int sid = (int)threadIdx.x - grp * kGroupThreads;
        int it = 0;
        for (int g = grp; g < total_chunks; g += 2, it++) {
            const int s = g % S;
            volatile int *fl = flag + grp * 2 + (it & 1);
            if (sid == 0)
                *fl = mbar_wait(&staged[s], (g / S) & 1) ? 1 : 0;
            named_bar_sync(1 + grp, kGroupThreads);
            if (*fl == 0) { ok = false; break; }
            const int4 pd = pend[s];
            if (pd.x == -1) {
                uint8_t *At = smem + s * Cfg::kStage;
#pragma unroll
                for (int q = 0; q < kATileBytes / (16 * kGroupThreads); q++)
                    reinterpret_cast<uint4 *>(At)[sid + q * kGroupThreads] = make_uint4(0, 0, 0, 0);
                named_bar_sync(1 + grp, kGroupThreads);
                const uint32_t *st = reinterpret_cast<const uint32_t *>(smem + Cfg::kStagingOff + s * kStagingBytes);
                for (int e = pd.y + sid; e < pd.w; e += kGroupThreads) {
                    const uint32_t v = st[e - pd.z];
                    if constexpr (F8)
                        At[swz64_offset(v >> 22, (v >> 16) & 63u)] = (uint8_t)(v & 0xffu);
                    else
                        *reinterpret_cast<uint16_t *>(At + swz128_offset(v >> 22, (v >> 16) & 63u)) =
                            (uint16_t)(v & 0xffffu);
                }
                fence_proxy_async();
            }
            mbar_arrive(&full[s]);
        }
    } else if (warp == pair::kMmaWarp) {
        if (lane == 0) {
            if (rank == 0) {
                // ---------------- MMA issuer for the pair ----------------
                constexpr uint32_t idesc = idesc_pair();
                const bool withhold = (batch.job[0].flags & TCA_FLAG_TEST_WITHHOLD_ACCUM) != 0;
                for (int g = 0; g < total_chunks; g++) {
                    const int s = g % S;
                    if (!mbar_wait(&full[s], (g / S) & 1) || !mbar_poll_cluster(&peer_full[s], (g / S) & 1)) {
                        ok = false;
                        break;
                    }
                    const int4 f = pend2[s];
                    const int b = f.y, k = f.z;
                    if ((f.x & 1) && k >= 2 && !mbar_poll_cluster(&acc_empty[b], ((k >> 1) - 1) & 1)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_s = smem_u32(smem + s * Cfg::kStage), b_s = a_s + kATileBytes;
                    const uint32_t d = tmem + (uint32_t)(b * kPairN);
                    if constexpr (F8) {
#pragma unroll
                        for (int kk = 0; kk < kChunkCols / 32; kk++) {
                            const uint64_t ad = smem_desc(a_s + kk * 32, 16, 512, 4);
                            const uint64_t bd = smem_desc(b_s + kk * 4096, kChunkCols * 128, 1024);
                            umma_pair_f8(d, ad, bd, idesc, ((f.x & 1) && kk == 0) ? 0u : 1u);
                        }
                    } else {
#pragma unroll
                        for (int kk = 0; kk < kChunkCols / 16; kk++) {
                            const uint64_t ad = smem_desc(a_s + kk * 32, 16, 1024);
                            const uint64_t bd = smem_desc(b_s + kk * 2048, kChunkCols * 128, 1024);
                            umma_pair_f16(d, ad, bd, idesc, ((f.x & 1) && kk == 0) ? 0u : 1u);
                        }
                    }
                    umma_commit_pair(&empty[s]);
                    if ((f.x & 2) && !(withhold && k == n_items - 1))
                        umma_commit_pair(&acc_full[b]);
                }
                umma_commit_pair(drain);
            } else {
                // ---------------- relay: this CTA's stages to the first CTA ----------------
                for (int g = 0; g < total_chunks; g++) {
                    const int s = g % S;
                    if (!mbar_wait(&full[s], (g / S) & 1)) { ok = false; break; }
                    mbar_arrive_cluster(cluster_map(smem_u32(&peer_full[s]), 0u));
                }
            }
            // every MMA of the pair has completed (both CTAs' tensor memory and
            // shared memory are no longer read or written by it)
            if (!mbar_poll_cluster(drain, 0))
                ok = false;
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: this CTA's window, all 256 columns ----------------
        const int quarter = warp & 3;
        for (int k = 0; k < n_items; k++) {
            const int4 it = items[2 * k], it2 = items[2 * k + 1];
            const TcJob &a = batch.job[it.w >> 16];
            const int n0 = (it.w & 0xffff) * kPairN;
            const int i = it2.x * kWindowRows + quarter * 32 + lane;
            int out_row = -1;
            if (it2.x >= 0 && i < a.M && !((a.flags & TCA_FLAG_KEEP_EMPTY_ROWS) && a.p_row_ptr[i + 1] == a.p_row_ptr[i]))
                out_row = a.perm[i];
            const int b = k & 1;
            if constexpr (F8) {
                float *sc = reinterpret_cast<float *>(smem + Cfg::kScaleOff) + b * kPairN;
                for (int c = quarter * 32 + lane; c < kPairN; c += kEpiThreads)
                    sc[c] = n0 + c < a.N ? __ldg(a.col_scale + n0 + c) : 0.f;
            }
            uint32_t got = 0;
            if (lane == 0)
                got = mbar_poll_cluster(&acc_full[b], (k >> 1) & 1) ? 1u : 0u;
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!named_bar_and(kEpiBar, kEpiThreads, got != 0)) { ok = false; break; }
            tc_fence_after();
            OutT *Crow = out_row >= 0 ? reinterpret_cast<OutT *>(a.C) + (size_t)out_row * a.ldc : nullptr;
            float sa = 1.f;
            if constexpr (F8)
                sa = (it2.x >= 0 && i < a.M) ? a.row_scale[i] : 0.f;
            for (int cb = 0; it2.x >= 0 && cb < kPairN / 16; cb++) {
                const int n = n0 + cb * 16;
                if (n >= a.N)
                    break;
                uint32_t r[16];
                tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * kPairN + cb * 16), r);
                if constexpr (F8) {
                    float *f = reinterpret_cast<float *>(r);
                    const float *sb = reinterpret_cast<const float *>(smem + Cfg::kScaleOff) + b * kPairN + cb * 16;
#pragma unroll
                    for (int q = 0; q < 16; q++) f[q] *= sa * sb[q];
                }
                if (Crow) {
                    store8_out(Crow + n, reinterpret_cast<const float *>(r), a.alpha, a.beta);
                    if (n + 8 < a.N)
                        store8_out(Crow + n + 8, reinterpret_cast<const float *>(r) + 8, a.alpha, a.beta);
                }
            }
            tc_fence_before();
            named_bar_sync(kEpiBar, kEpiThreads); // the four warps are done with buffer b
            if (warp == pair::kEpiWarp0 && lane == 0) {
                if (rank == 0)
                    mbar_arrive(&acc_empty[b]);
                else
                    mbar_arrive_cluster(cluster_map(smem_u32(&acc_empty[b]), 0u));
            }
        }
    }

    tc_fence_before();
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
            if (n_items > 0)
                atomicOr(batch.job[items[0].w >> 16].status, kStatusTimeout);
            const uint64_t t0 = global_ns();
            while (global_ns() - t0 < 1000000ull) {
            }
        }
        __syncthreads();
    }
    // The partner makes no further access to this CTA's shared memory once
    // it has arrived here (its roles are done, the MMAs it issued completed);
    // the wait is bounded like every other.
    if (threadIdx.x == 0) {
        mbar_arrive_cluster(cluster_map(smem_u32(bye), rank ^ 1u));
        if (!mbar_poll_cluster(bye, 0) && n_items > 0)
            atomicOr(batch.job[items[0].w >> 16].status, kStatusTimeout);
    }
    __syncthreads();
    if (warp == pair::kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kPairN) : "memory");
    }
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

} // namespace

namespace {
int encode_tiled(CUtensorMap *map, CUtensorMapDataType dtype, int rank, const void *base, const cuuint64_t *dims,
                 const cuuint64_t *strides, const cuuint32_t *box, CUtensorMapSwizzle swizzle)
{
    auto enc = tensor_map_encoder();
    if (!enc)
        return set_error(TCA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint32_t estr[3] = {1, 1, 1};
    auto encode = [&] {
        return enc(map, dtype, (cuuint32_t)rank, const_cast<void *>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT) { // a host thread's first CUDA call: make the device's context current
        int dev = 0;
        TCA_CUDA_TRY(cudaGetDevice(&dev));
        TCA_CUDA_TRY(cudaSetDevice(dev));
        r = encode();
    }
    if (r != CUDA_SUCCESS)
        return set_error(TCA_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d): dims {%llu, %llu}, stride %llu, box {%u, %u}",
                         (int)r, (unsigned long long)dims[0], (unsigned long long)dims[1],
                         (unsigned long long)strides[0], box[0], box[1]);
    return TCA_OK;
}
} // namespace

int encode_tensor_map_2d(CUtensorMap *map, CUtensorMapDataType dtype, const void *base, uint64_t d0, uint64_t d1,
                         uint64_t row_stride_bytes, uint32_t b0, uint32_t b1, CUtensorMapSwizzle swizzle)
{
    const cuuint64_t dims[2] = {(cuuint64_t)d0, (cuuint64_t)(d1 > 0 ? d1 : 1)};
    const cuuint64_t strides[1] = {(cuuint64_t)row_stride_bytes};
    const cuuint32_t box[2] = {b0, b1};
    return encode_tiled(map, dtype, 2, base, dims, strides, box, swizzle);
}

int encode_tensor_map_slabs(CUtensorMap *map, CUtensorMapDataType dtype, int elem, const void *base, uint64_t slabs,
                            uint64_t d1, uint64_t row_stride_bytes, uint32_t b1, uint32_t bslabs)
{
    const cuuint64_t dims[3] = {(cuuint64_t)(128 / elem), (cuuint64_t)(d1 > 0 ? d1 : 1), (cuuint64_t)slabs};
    const cuuint64_t strides[2] = {(cuuint64_t)row_stride_bytes, 128};
    const cuuint32_t box[3] = {(cuuint32_t)(128 / elem), b1, bslabs};
    return encode_tiled(map, dtype, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

namespace {

// B (K x N, row-major, leading dimension ldb) as a TMA source: dims {N, K},
// row stride ldb * 2 bytes, box {64, rows}, 128-byte swizzle, zero fill.
int encode_b_map(const SpmmJob &sj, int K, int rows, CUtensorMap *map)
{
    return encode_tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, sj.B, (uint64_t)sj.N, (uint64_t)K,
                                (uint64_t)sj.ldb * 2, 64, (uint32_t)rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

// NT: the slice width of the single-window kernel; 0: the pair kernel.
int make_job(const SpmmJob &sj, float alpha, float beta, unsigned flags, int NT, TcJob *out)
{
    const tca_plan *p = sj.p;
    TcJob &j = *out;
    const int slab = sj.f8 ? 128 : 64; // columns of a 128-byte slab of B
    // One box per chunk when N is whole slabs (load-only ring of 148 CTAs,
    // 48 KB chunks: 0.38 us per chunk against 0.44 us with a 2-D box per slab);
    // else the tensor map must know where a row ends inside a slab.
    j.tile3d = NT > 0 && sj.N % slab == 0;
    j.gathers = p->has_gathers;
    if (NT == 0)
        NT = kPairN;
    if (sj.f8) {
        // E4M3 B (K x N bytes, row stride ldq): boxes of 128 columns
        if (p->has_gathers)
            TCA_TRY(encode_tensor_map_2d(&j.tmap_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, sj.Bq, (uint64_t)sj.N, (uint64_t)p->K,
                                         (uint64_t)sj.ldq, 128, 1, CU_TENSOR_MAP_SWIZZLE_128B));
        if (j.tile3d)
            TCA_TRY(encode_tensor_map_slabs(&j.tmap_tile, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, sj.Bq,
                                            (uint64_t)(sj.N / slab), (uint64_t)p->K, (uint64_t)sj.ldq, kChunkCols,
                                            (uint32_t)(NT / slab)));
        else
            TCA_TRY(encode_tensor_map_2d(&j.tmap_tile, CU_TENSOR_MAP_DATA_TYPE_UINT8, sj.Bq, (uint64_t)sj.N,
                                         (uint64_t)p->K, (uint64_t)sj.ldq, 128, kChunkCols,
                                         CU_TENSOR_MAP_SWIZZLE_128B));
        j.entries = p->tile_entries_f8;
        j.images = p->images_f8;
        j.row_scale = p->row_scale;
        j.col_scale = sj.col_scale;
    } else {
        if (p->has_gathers) // nothing else reads it
            TCA_TRY(encode_b_map(sj, p->K, 1, &j.tmap_b));
        if (j.tile3d)
            TCA_TRY(encode_tensor_map_slabs(&j.tmap_tile, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, sj.B,
                                            (uint64_t)(sj.N / slab), (uint64_t)p->K, (uint64_t)sj.ldb * 2, kChunkCols,
                                            (uint32_t)(NT / slab)));
        else
            TCA_TRY(encode_b_map(sj, p->K, kChunkCols, &j.tmap_tile));
        j.entries = p->tile_entries;
        j.images = reinterpret_cast<const uint8_t *>(p->images);
        j.row_scale = nullptr;
        j.col_scale = nullptr;
    }
    j.win_info = p->tc_win_info;
    j.pairs = p->tc_pairs;
    j.tile_ptr = p->tile_ptr;
    j.win_cols = p->win_cols;
    j.img_idx = p->img_idx;
    j.perm = p->perm;
    j.p_row_ptr = p->p_row_ptr;
    j.B = sj.B;
    j.C = sj.C;
    j.status = p->d_status;
    j.M = p->M;
    j.N = sj.N;
    j.ldb = sj.ldb;
    j.ldc = sj.ldc;
    j.nt = NT;
    j.ntiles = (sj.N + NT - 1) / NT;
    j.alpha = alpha;
    j.beta = beta;
    j.flags = flags;
    return TCA_OK;
}

template <int NT, typename OutT, bool F8, int CAP>
int launch_group_cap(const TcBatchT<CAP> &b, bool dependent, cudaStream_t s)
{
    const int smem = TcCfg<NT, F8>::kSmem;
    TCA_CUDA_TRY(cudaFuncSetAttribute(spmm_tc_kernel<NT, OutT, F8, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      smem));
    // The whole 228 KB carveout: with the smallest one that holds this block
    // (196 KB for the E4M3 rings) no room is left for the 1 KB that each
    // CUDA-core block reserves, and the launch that should run beside this
    // one waits for it to end (measured: E4M3 step, CUDA-core blocks starting
    // as the first tensor-core blocks exit).
    TCA_CUDA_TRY(cudaFuncSetAttribute(spmm_tc_kernel<NT, OutT, F8, CAP>,
                                      cudaFuncAttributePreferredSharedMemoryCarveout,
                                      (int)cudaSharedmemCarveoutMaxShared));
    const int total = b.item_start[b.n_jobs];
    const int grid = std::min(total, std::max(kSMs, (total + kMaxCtaItems - 1) / kMaxCtaItems));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = F8 && dependent ? 1 : 0;
    TCA_CUDA_TRY(cudaLaunchKernelEx(&cfg, spmm_tc_kernel<NT, OutT, F8, CAP>, b));
    return TCA_OK;
}

template <typename OutT, int CAP>
int launch_group_out(const TcBatchT<CAP> &b, int NT, bool f8, bool dependent, cudaStream_t s)
{
    if (f8)
        return NT == 128 ? launch_group_cap<128, OutT, true>(b, dependent, s)
                         : launch_group_cap<256, OutT, true>(b, dependent, s);
    switch (NT) {
    case 64: return launch_group_cap<64, OutT, false>(b, dependent, s);
    case 128: return launch_group_cap<128, OutT, false>(b, dependent, s);
    default: return launch_group_cap<256, OutT, false>(b, dependent, s);
    }
}

template <int CAP>
int launch_typed(const TcBatchT<CAP> &b, int NT, bool f8, int c_dtype, bool dependent, cudaStream_t s)
{
    return c_dtype == TCA_DTYPE_F16 ? launch_group_out<__half>(b, NT, f8, dependent, s)
                                    : launch_group_out<float>(b, NT, f8, dependent, s);
}

// Pair kernel: clusters of two CTAs (one per SM), persistent over the pair
// items, as many clusters as fit at once (or more when an item list would
// exceed kMaxCtaItems per cluster).
template <typename OutT, bool F8>
int launch_pair_group(const TcBatch &b, cudaStream_t s)
{
    const int smem = Tc2Cfg<F8>::kSmem;
    auto kernel = spmm_tc_pair_kernel<OutT, F8>;
    TCA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    TCA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      (int)cudaSharedmemCarveoutMaxShared));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(pair::kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    static int max_clusters = 0;
    if (max_clusters == 0) {
        cfg.gridDim = dim3(2 * (kSMs / 2));
        int n = 0;
        TCA_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
        if (n <= 0)
            return set_error(TCA_ERR_CUDA, "no CTA pair of the tensor-core pair kernel fits on this device");
        max_clusters = n;
    }
    const int total = b.item_start[b.n_jobs];
    const int clusters = std::min(total, std::max(max_clusters, (total + kMaxCtaItems - 1) / kMaxCtaItems));
    cfg.gridDim = dim3((unsigned)(2 * clusters));
    TCA_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, b));
    return TCA_OK;
}

int launch_pair_typed(const TcBatch &b, bool f8, int c_dtype, cudaStream_t s)
{
    if (b.n_jobs == 0 || b.item_start[b.n_jobs] == 0)
        return TCA_OK;
    if (c_dtype == TCA_DTYPE_F16)
        return f8 ? launch_pair_group<__half, true>(b, s) : launch_pair_group<__half, false>(b, s);
    return f8 ? launch_pair_group<float, true>(b, s) : launch_pair_group<float, false>(b, s);
}

int launch_group_typed(const TcBatch &b, int NT, bool f8, int c_dtype, bool dependent, cudaStream_t s)
{
    if (b.n_jobs == 0 || b.item_start[b.n_jobs] == 0)
        return TCA_OK;
    if (b.n_jobs == 1 && b.job[0].nt == NT) {
        TcBatchT<1> one;
        one.n_jobs = 1;
        one.item_start[0] = b.item_start[0];
        one.item_start[1] = b.item_start[1];
        one.job[0] = b.job[0];
        return launch_typed(one, NT, f8, c_dtype, dependent, s);
    }
    return launch_typed(b, NT, f8, c_dtype, dependent, s);
}

} // namespace

int pick_tc_tile(const tca_plan *p, int N, bool batched, bool f8)
{
    const int n_tc = p->n_tc;
    const int lo = f8 ? 128 : 64; // E4M3 B tiles are whole 128-byte swizzle atoms
    int NT = N <= 64 ? 64 : N <= 128 ? 128 : 256;
    NT = std::max(NT, lo);
    // a single forward halves the slice while that leaves fewer than about
    // three quarters of the SMs with an item (measured: A^T of 512 x 2048,
    // N = 4096, 4 windows: NT = 128, 128 items, 30.5 us; NT = 64, 40.4 us)
    if (!batched)
        while (NT > lo && (long long)n_tc * ((N + NT - 1) / NT) < (3 * kSMs) / 4)
            NT /= 2;
    return NT;
}

int tc_block_regs(bool f8, int *regs)
{
    static int worst[2] = {0, 0};
    if (worst[f8] == 0) {
        const void *f16_fns[] = {
            (const void *)spmm_tc_kernel<64, __half, false>, (const void *)spmm_tc_kernel<128, __half, false>,
            (const void *)spmm_tc_kernel<256, __half, false>, (const void *)spmm_tc_kernel<64, float, false>,
            (const void *)spmm_tc_kernel<128, float, false>, (const void *)spmm_tc_kernel<256, float, false>,
            (const void *)spmm_tc_kernel<64, __half, false, 1>, (const void *)spmm_tc_kernel<128, __half, false, 1>,
            (const void *)spmm_tc_kernel<256, __half, false, 1>, (const void *)spmm_tc_kernel<64, float, false, 1>,
            (const void *)spmm_tc_kernel<128, float, false, 1>, (const void *)spmm_tc_kernel<256, float, false, 1>};
        const void *f8_fns[] = {
            (const void *)spmm_tc_kernel<128, __half, true>, (const void *)spmm_tc_kernel<256, __half, true>,
            (const void *)spmm_tc_kernel<128, float, true>, (const void *)spmm_tc_kernel<256, float, true>,
            (const void *)spmm_tc_kernel<128, __half, true, 1>, (const void *)spmm_tc_kernel<256, __half, true, 1>,
            (const void *)spmm_tc_kernel<128, float, true, 1>, (const void *)spmm_tc_kernel<256, float, true, 1>};
        const void *pair_fns[2][2] = {
            {(const void *)spmm_tc_pair_kernel<__half, false>, (const void *)spmm_tc_pair_kernel<float, false>},
            {(const void *)spmm_tc_pair_kernel<__half, true>, (const void *)spmm_tc_pair_kernel<float, true>}};
        int w = 0;
        auto widest = [&w](const void *f, int threads) -> int {
            int r = 0;
            TCA_TRY(block_regs(f, threads, &r));
            w = std::max(w, r);
            return TCA_OK;
        };
        if (f8)
            for (const void *f : f8_fns) TCA_TRY(widest(f, kThreads));
        else
            for (const void *f : f16_fns) TCA_TRY(widest(f, kThreads));
        for (const void *f : pair_fns[f8]) TCA_TRY(widest(f, pair::kThreads));
        worst[f8] = w;
    }
    *regs = worst[f8];
    return TCA_OK;
}

namespace {

// Time of an item: its chunks by the width of its slice, and its epilogue
// (units of 25 ns: 0.40, 0.27 and 0.25 us a chunk, 2.5 us; %clock traces).
int item_cost(int chunks, int n_tile) { return chunks * (n_tile == 256 ? 16 : n_tile == 128 ? 11 : 10) + 100; }

// Deals a launch's items to its CTAs, the longest first, each to the CTA with
// the least so far, when there is more than one round of them and they differ
// by a quarter.
// Round-robin left 24 layers of mixed shapes with CTAs ending between 9 and 36
// us (43.0 us a replay, 39.3 dealt out); a launch of about equal items keeps it
// (false).
// The host pays for this in every call that is not a replay (sorted items and a
// heap of CTAs: 175 us for 3,072 items, six layers of 8192 rows, whose call took
// 364 us, 298 without and 240 this way): costs are counted in kCostSteps steps of the longest, so
// windows sort by counting, and the CTAs wait in a ring of queues, one per step
// of their time so far -- the least never decreases and no CTA is more than one
// longest item ahead of it.
constexpr int kCostSteps = 512;

bool may_schedule(const TcBatch &b)
{
    const int total = b.item_start[b.n_jobs];
    return b.n_jobs >= 2 && total > kSMs && total <= kSMs * kMaxCtaItems;
}

bool schedule_items(const TcBatch &b, const SpmmJob *const *jobs, uint16_t *order)
{
    auto cost = [&](int j, int t) {
        const std::vector<int> &first = jobs[j]->p->h_tile_first;
        return item_cost(first[t + 1] - first[t], b.job[j].nt);
    };
    int lo = INT_MAX, hi = 0, windows = 0;
    for (int j = 0; j < b.n_jobs; j++)
        for (int t = 0; t < jobs[j]->p->n_tc; t++, windows++) {
            lo = std::min(lo, cost(j, t));
            hi = std::max(hi, cost(j, t));
        }
    if (4LL * hi < 5LL * lo) // nearly equal: neighbours in time stay neighbours in a problem
        return false;
    auto steps = [&](int c) { return (int)(((long long)c * (kCostSteps - 1) + hi - 1) / hi); }; // 1 .. kCostSteps - 1
    // windows by cost, the longest first
    struct Window {
        int first_item, n_items, steps;
    };
    int place[kCostSteps + 1] = {};
    for (int j = 0; j < b.n_jobs; j++)
        for (int t = 0; t < jobs[j]->p->n_tc; t++) place[kCostSteps - steps(cost(j, t))]++;
    for (int k = 0, sum = 0; k <= kCostSteps; k++) {
        const int n = place[k];
        place[k] = sum;
        sum += n;
    }
    std::vector<Window> sorted((size_t)windows);
    for (int j = 0; j < b.n_jobs; j++)
        for (int t = 0; t < jobs[j]->p->n_tc; t++) {
            const int c = steps(cost(j, t));
            sorted[place[kCostSteps - c]++] = Window{b.item_start[j] + t * b.job[j].ntiles, b.job[j].ntiles, c};
        }
    std::fill(order, order + (size_t)kMaxCtaItems * kSMs, kNoItem);
    int count[kSMs] = {};
    int16_t head[kCostSteps], tail[kCostSteps], next[kSMs]; // queues of CTAs by time so far, modulo kCostSteps
    std::fill(head, head + kCostSteps, (int16_t)-1);
    auto enqueue = [&](int c, int at) {
        next[c] = -1;
        if (head[at] < 0) head[at] = (int16_t)c;
        else next[tail[at]] = (int16_t)c;
        tail[at] = (int16_t)c;
    };
    for (int c = 0; c < kSMs; c++) enqueue(c, 0);
    int now = 0;
    for (const Window &w : sorted)
        for (int n = 0; n < w.n_items; n++) { // at most kMaxCtaItems each: a full CTA leaves the queues
            while (head[now] < 0) now = (now + 1) % kCostSteps;
            const int c = head[now];
            head[now] = next[c];
            order[count[c] * kSMs + c] = (uint16_t)(w.first_item + n);
            if (++count[c] < kMaxCtaItems) enqueue(c, (now + w.steps) % kCostSteps);
        }
    return true;
}

} // namespace

// A window alone on a CTA pair keeps two SMs for one window's chunks, so the
// pair kernel takes a plan when at least two thirds of its tensor-core
// windows are paired.
bool pair_eligible(const tca_plan *p, int NT)
{
    return NT == kPairN && p->opts.pair_windows != 0 && p->tc_pairs != nullptr && 3 * p->n_full_pairs >= p->n_tc;
}

int launch_tc_jobs(const SpmmJob *jobs, int n_jobs, int c_dtype, float alpha, float beta, unsigned flags,
                   cudaStream_t s, LaunchList *defer, bool dependent)
{
    if (n_jobs == 1 && !pair_eligible(jobs[0].p, jobs[0].n_tile)) {
        // a single forward: no batch of job slots to fill and copy
        const SpmmJob &sj = jobs[0];
        if (!sj.tc || sj.p->n_tc == 0 || sj.N <= 0)
            return TCA_OK;
        TcBatchT<1> one;
        one.n_jobs = 1;
        TCA_TRY(make_job(sj, alpha, beta, flags, sj.n_tile, &one.job[0]));
        one.item_start[0] = 0;
        one.item_start[1] = sj.p->n_tc * one.job[0].ntiles;
        const int NT = sj.n_tile;
        const bool f8 = sj.f8;
        if (!defer)
            return launch_typed(one, NT, f8, c_dtype, dependent, s);
        defer->push_back([one, NT, f8, c_dtype, dependent](cudaStream_t st) {
            return launch_typed(one, NT, f8, c_dtype, dependent, st);
        });
        return TCA_OK;
    }
    auto emit = [&](const TcBatch &b, int NT, bool f8) -> int {
        if (b.n_jobs == 0 || b.item_start[b.n_jobs] == 0)
            return TCA_OK;
        auto run = [NT, f8, c_dtype, dependent](const TcBatch &bb, cudaStream_t st) {
            return NT == 0 ? launch_pair_typed(bb, f8, c_dtype, st)
                           : launch_group_typed(bb, NT, f8, c_dtype, dependent, st);
        };
        if (!defer)
            return run(b, s);
        auto held = std::make_shared<TcBatch>(b);
        defer->push_back([held, run](cudaStream_t st) { return run(*held, st); });
        return TCA_OK;
    };
    // All jobs of a precision in one launch, as wide as their widest N-slice:
    // launches run one after the other, each with its own set-up and its own
    // partly filled last round (24 layers with N of 64 to 1024: three launches
    // 73.9 us, one 43.5 us). Jobs with more chunks per item first: rounds of
    // equal items, the short ones last (schedule_items deals them out).
    auto cost = [](const SpmmJob &j) { // of one item, on average
        return item_cost(j.p->n_tc_chunks / std::max(1, j.p->n_tc), j.n_tile);
    };
    for (bool f8 : {false, true}) {
        for (bool pair : {false, true}) {
            std::vector<const SpmmJob *> sel;
            for (int i = 0; i < n_jobs; i++) {
                const SpmmJob &sj = jobs[i];
                if (sj.tc && sj.f8 == f8 && sj.p->n_tc > 0 && sj.N > 0 && pair_eligible(sj.p, sj.n_tile) == pair)
                    sel.push_back(&sj);
            }
            std::stable_sort(sel.begin(), sel.end(),
                             [&](const SpmmJob *x, const SpmmJob *y) { return cost(*x) > cost(*y); });
            for (size_t i0 = 0; i0 < sel.size(); i0 += kMaxJobs) {
                TcBatch b;
                b.n_jobs = 0;
                b.item_start[0] = 0;
                int NT = 0;
                for (size_t i = i0; i < std::min(sel.size(), i0 + kMaxJobs); i++) {
                    const SpmmJob &sj = *sel[i];
                    TCA_TRY(make_job(sj, alpha, beta, flags, pair ? 0 : sj.n_tile, &b.job[b.n_jobs]));
                    const int units = pair ? sj.p->n_pairs : sj.p->n_tc;
                    b.item_start[b.n_jobs + 1] = b.item_start[b.n_jobs] + units * b.job[b.n_jobs].ntiles;
                    b.n_jobs++;
                    if (!pair) NT = std::max(NT, sj.n_tile);
                }
                if (!pair && may_schedule(b)) {
                    std::shared_ptr<TcOrdered> held(new TcOrdered);
                    if (schedule_items(b, &sel[i0], held->order)) {
                        held->n_jobs = b.n_jobs;
                        std::copy(b.item_start, b.item_start + kMaxJobs + 1, held->item_start);
                        std::copy(b.job, b.job + b.n_jobs, held->job);
                        if (!defer)
                            TCA_TRY(launch_typed(*held, NT, f8, c_dtype, dependent, s));
                        else
                            defer->push_back([held, NT, f8, c_dtype, dependent](cudaStream_t st) {
                                return launch_typed(*held, NT, f8, c_dtype, dependent, st);
                            });
                        continue;
                    }
                }
                TCA_TRY(emit(b, NT, f8));
            }
        }
    }
    return TCA_OK;
}

} // namespace tca
