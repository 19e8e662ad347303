// sddmm_tc.cu -- the SDDMM adjoint dA = alpha * (dY B^T) on A's pattern, on
// the tensor cores (tcgen05, sm_100a), over the plan's tensor-core windows.
//
// The reference has no backward pass; the adjoint follows from its forward
// (src/our_spmm.cu:290-346, Y[r, :] = sum_j a_j B[c_j, :]):
//   dL/da_j = sum_n dY[r_j, n] * B[c_j, n].
// For a tensor-core window (128 sorted rows) and one of its 64-column chunks,
// the tile D[128 x 64] = dY[window rows, :] B[chunk columns, :]^T holds the
// values of every nonzero of the chunk: a GEMM tile with K = N (the width of
// dY and B), A = dY rows (K-major) and B = B rows (K-major), accumulated in
// FP32 in tensor memory. Only chunks that hold nonzeros are computed, and the
// epilogue writes only the nonzeros (the chunk's tile entries), in the
// caller's nonzero order.
//
// Work unit: (window, group of up to 8 of its chunks -- 8 x 64 accumulator
// columns fill tensor memory --, part of the n range). Per 64-wide step of n
// two loader warps bring the window's dY rows (16 KB; one 128-row box when the
// window's rows follow one another in dY, else tile::gather4 of the rows
// perm[...]) and a third the B rows, a half of the group (4 chunks, 32 KB) per
// stage: one 256-row box when the chunks are consecutive blocks of K, else a
// 64-row box per direct chunk and tile::gather4 per condensed one. The MMA
// lane multiplies the dY stage with each half (M = 128, N = up to 256). No
// load uses cluster multicast; rows and columns outside the tensors (a
// window's rows beyond M, padding columns, n >= N) arrive as zeros.
//
// What bounds it: the issue of the gathers. One warp issues a tile::gather4
// every 32 ns, so a window's 32 per step took longer than the step's MMAs
// (1024 cycles); two warps need 0.64 us per step, 0.79 us with the B boxes
// beside them (a load-only ring), and the eight 8 KB B loads per step are now
// two. 2048 x 512 at 90 %, N = 4096: 41 us -> 19 us (sums included). All warps
// take part in the epilogue (the entries are read four at a time).
//
// When the windows' groups are fewer than the SMs, the n range is cut into
// parts; each part leaves its values in a workspace slice (one float per
// tensor-core entry), and after the launch k_sddmm_sum adds the parts of
// every entry in part order -- a fixed order, so the result does not depend
// on which part finished when -- and writes dA. No CTA waits for another.
// Every mbarrier wait is bounded (about one second); on expiry the CTA records
// kStatusTimeout in the plan's status word and ends; the sums are not written
// while that bit is set.
#include <cuda.h>
#include <algorithm>
#include "tca_internal.cuh"
#include "plan.cuh"
#include "ptx.cuh"

namespace tca {
namespace {

using namespace ptx;

constexpr int kSdYWarps = 2;   // warps 0-1: dY rows
constexpr int kSdBWarp = 2;    // B rows
constexpr int kSdMmaWarp = 3;
constexpr int kSdThreads = 256; // warps 4-7 join for the epilogue only
constexpr int kSdMaxChunks = 8;  // chunks per unit: 8 x 64 FP32 accumulator columns = all of tensor memory
constexpr int kSdHalf = 4;       // chunks per B stage: the MMA's N = 256
constexpr int kSdYStages = 3;    // dY ring: 128 rows x 64 n, 16 KB each
constexpr int kSdBStages = 5;    // B ring: 256 rows x 64 n, 32 KB each
constexpr int kSdYBytes = kWindowRows * 64 * 2;
constexpr int kSdChunkBytes = kChunkCols * 64 * 2;
constexpr int kSdBBytes = kSdHalf * kSdChunkBytes;
constexpr int kSdStageRow = 68;  // floats per row of the epilogue's staging tiles (64 + 4: fewer bank conflicts)
constexpr int kSdStageChunks = 4; // chunks staged at once in the epilogue
constexpr int kSdYOff = 0;
constexpr int kSdBOff = kSdYOff + kSdYStages * kSdYBytes;
constexpr int kSdBarOff = kSdBOff + kSdBStages * kSdBBytes;
// y_full, y_empty [kSdYStages]; b_full, b_empty [kSdBStages]; acc_full; TMEM slot
constexpr int kSdSmem = kSdBarOff + (2 * kSdYStages + 2 * kSdBStages + 1) * 8 + 8;
static_assert(kSdBarOff >= kSdStageChunks * kWindowRows * kSdStageRow * 4, "the rings hold the epilogue's staging tiles");
static_assert(kSdYBytes % 1024 == 0 && kSdChunkBytes % 1024 == 0, "swizzled tiles need 1024-byte alignment");
static_assert(kSdSmem <= 227 * 1024, "shared memory budget");

struct SdJob {
    CUtensorMap tmap_y;    // dY as {N, M}, box {64, 1}, 128-byte swizzle (gather4 of window rows)
    CUtensorMap tmap_yrun; // the same, box {64, 128} (a window of consecutive rows)
    CUtensorMap tmap_b;    // B as {N, K}, box {64, 1} (gather4 of condensed columns)
    CUtensorMap tmap_tile; // B as {N, K}, box {64, 64} (64 consecutive rows: a direct chunk)
    CUtensorMap tmap_run;  // B as {N, K}, box {64, 256} (consecutive direct chunks)
    const int4 *win_info;  // per tensor-core window: window, first chunk, chunk count
    const int *win_cols, *tile_ptr, *perm, *src, *tile_src;
    const uint32_t *entries;
    void *out;             // nnz values in the caller's order (FP16 or FP32)
    float *partials;       // parts > 1: parts x part_stride floats
    int *status;
    int M, N, n_steps, parts, steps_per_part, out_f16;
    int n_win, groups_per_win, group_chunks; // tensor-core windows; chunk groups of the widest window; chunks per group
    long long part_stride; // floats per part: the tensor-core entries, rounded up to 4
    float alpha;
};

// kind::f16 instruction descriptor: D FP32, A/B FP16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t sd_idesc(int n)
{
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void sd_umma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(accum)
                 : "memory");
}

// Unit u -> (tensor-core window t, chunk group gi: chunks [n gi, n gi + n)
// of the window with n = group_chunks, part q of the n range); units are ordered window, group,
// part. A window with fewer groups than the widest leaves its extra units
// empty: false.
struct SdUnit {
    int t, g0, nch, q, group;
};

__device__ __forceinline__ bool sd_decode(const SdJob &a, int u, SdUnit &x)
{
    x.q = u % a.parts;
    x.group = u / a.parts;
    x.t = x.group / a.groups_per_win;
    x.g0 = (x.group - x.t * a.groups_per_win) * a.group_chunks;
    if (x.t >= a.n_win)
        return false;
    const int z = __ldg(&a.win_info[x.t].z);
    x.nch = min(a.group_chunks, z - x.g0);
    return x.nch > 0;
}

__global__ void __launch_bounds__(kSdThreads, 1) k_sddmm_tc(const __grid_constant__ SdJob a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *y_full = reinterpret_cast<uint64_t *>(smem + kSdBarOff);
    uint64_t *y_empty = y_full + kSdYStages;
    uint64_t *b_full = y_empty + kSdYStages;
    uint64_t *b_empty = b_full + kSdBStages;
    uint64_t *acc_full = b_empty + kSdBStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    // the sums of the parts (a programmatic dependent) may take their place on
    // the SMs; they wait for this grid to end before they read anything
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    SdUnit x;
    if (!sd_decode(a, blockIdx.x, x))
        return; // uniform: no unit for this CTA
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0)
            atomicOr(a.status, kStatusLayout);
        return;
    }
    const int4 wi = __ldg(a.win_info + x.t);
    const int c_first = wi.y + x.g0; // the group's first chunk (plan-wide index)
    const int ks0 = x.q * a.steps_per_part, ks1 = min(a.n_steps, ks0 + a.steps_per_part);
    const int steps = ks1 - ks0;
    const int halves = (x.nch + kSdHalf - 1) / kSdHalf;
    int tcols = 32;
    while (tcols < x.nch * 64) tcols <<= 1;
    // the part's n steps, each window starting at a different one, so that
    // the windows do not read the same columns of B at once
    const int rot = x.t % max(1, steps);
    auto step_n = [&](int st) { return (ks0 + (st + rot) % steps) * 64; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSdYStages; s++) {
            mbar_init(&y_full[s], kSdYWarps);
            mbar_init(&y_empty[s], 1);
        }
        for (int s = 0; s < kSdBStages; s++) {
            mbar_init(&b_full[s], 1);
            mbar_init(&b_empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init_fence();
    }
    if (warp == kSdMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tcols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp < kSdYWarps) {
        // ---------------- dY rows ----------------
        // the window's 128 rows (caller rows; -1 beyond M: zero rows), four per
        // lane; warp w gathers those of lanes 16 w .. 16 w + 15
        int rows[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int i = wi.x * kWindowRows + 4 * lane + r;
            rows[r] = i < a.M ? __ldg(a.perm + i) : -1;
        }
        const int row0 = __shfl_sync(0xffffffffu, rows[0], 0);
        const bool run = __all_sync(0xffffffffu, rows[0] == row0 + 4 * lane && rows[1] == rows[0] + 1 &&
                                                     rows[2] == rows[0] + 2 && rows[3] == rows[0] + 3);
        const int mine = warp * (32 / kSdYWarps);
        int s = 0;
        uint32_t phase = 1;
        for (int st = 0; st < steps; st++) {
            const int n0 = step_n(st);
            const uint32_t dst = smem_u32(smem + kSdYOff + s * kSdYBytes);
            if (elect_one()) {
                ok = mbar_wait(&y_empty[s], phase);
                if (ok) {
                    if (!run) {
                        mbar_arrive_expect_tx(&y_full[s], kSdYBytes / kSdYWarps);
                    } else if (warp == 0) {
                        mbar_arrive_expect_tx(&y_full[s], kSdYBytes);
                        tma_tile2d(dst, &a.tmap_yrun, n0, row0, &y_full[s]);
                    } else {
                        mbar_arrive(&y_full[s]);
                    }
                }
            }
            if (__any_sync(0xffffffffu, !ok)) { ok = false; break; } // also: the transaction count is set
            if (!run && lane >= mine && lane < mine + 32 / kSdYWarps)
                tma_gather4(dst + lane * 512, &a.tmap_y, n0, rows[0], rows[1], rows[2], rows[3], &y_full[s]);
            if (++s == kSdYStages) { s = 0; phase ^= 1; }
        }
    } else if (warp == kSdBWarp) {
        // ---------------- B rows ----------------
        // each chunk's 64 columns (lanes 0-15: four each); bit c of `direct`:
        // 64 consecutive ones, first in lane c of `col0`; bit h of `runs`:
        // the direct chunks of half h follow one another
        int4 cols[kSdMaxChunks];
        uint32_t direct = 0, runs = 0;
        int col0 = -1;
#pragma unroll
        for (int c = 0; c < kSdMaxChunks; c++) {
            cols[c] = make_int4(-1, -1, -1, -1);
            if (c < x.nch && lane < 16)
                cols[c] = __ldg(reinterpret_cast<const int4 *>(a.win_cols + (size_t)(c_first + c) * kChunkCols) + lane);
        }
#pragma unroll
        for (int c = 0; c < kSdMaxChunks; c++) {
            const int first = __shfl_sync(0xffffffffu, cols[c].x, 0), last = __shfl_sync(0xffffffffu, cols[c].w, 15);
            if (first >= 0 && last == first + kChunkCols - 1) direct |= 1u << c;
            if (lane == c) col0 = first;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            bool run = true;
            const int first = __shfl_sync(0xffffffffu, col0, h * kSdHalf);
            for (int c = h * kSdHalf; c < min(x.nch, (h + 1) * kSdHalf); c++)
                run = run && (direct >> c & 1u) &&
                      __shfl_sync(0xffffffffu, col0, c) == first + (c - h * kSdHalf) * kChunkCols;
            if (run) runs |= 1u << h;
        }
        int s = 0;
        uint32_t phase = 1;
        for (int st = 0; st < steps && ok; st++) {
            const int n0 = step_n(st);
            for (int h = 0; h < halves; h++) {
                const int c0 = h * kSdHalf, nc = min(kSdHalf, x.nch - c0);
                const uint32_t dst = smem_u32(smem + kSdBOff + s * kSdBBytes);
                const bool run = (runs >> h & 1u) != 0;
                const int first = __shfl_sync(0xffffffffu, col0, c0);
                if (elect_one()) {
                    ok = mbar_wait(&b_empty[s], phase);
                    if (ok) {
                        mbar_arrive_expect_tx(&b_full[s], run ? kSdBBytes : nc * kSdChunkBytes);
                        if (run)
                            tma_tile2d(dst, &a.tmap_run, n0, first, &b_full[s]);
                    }
                }
                if (__any_sync(0xffffffffu, !ok)) { ok = false; break; }
                if (!run) {
#pragma unroll
                    for (int c = 0; c < kSdMaxChunks; c++) {
                        if (c < c0 || c >= c0 + nc)
                            continue;
                        const uint32_t d = dst + (uint32_t)(c - c0) * kSdChunkBytes;
                        if (direct >> c & 1u) {
                            if (lane == 0)
                                tma_tile2d(d, &a.tmap_tile, n0, cols[c].x, &b_full[s]);
                        } else if (lane < 16) {
                            tma_gather4(d + lane * 512, &a.tmap_b, n0, cols[c].x, cols[c].y, cols[c].z, cols[c].w,
                                        &b_full[s]);
                        }
                    }
                }
                if (++s == kSdBStages) { s = 0; phase ^= 1; }
            }
        }
    } else if (warp == kSdMmaWarp) {
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
            int sy = 0, sb = 0;
            uint32_t py = 0, pb = 0;
            for (int st = 0; st < steps && ok; st++) {
                if (!mbar_wait(&y_full[sy], py)) { ok = false; break; }
                const uint32_t ys = smem_u32(smem + kSdYOff + sy * kSdYBytes);
                for (int h = 0; h < halves; h++) {
                    if (!mbar_wait(&b_full[sb], pb)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t bs = smem_u32(smem + kSdBOff + sb * kSdBBytes);
                    const uint32_t idesc = sd_idesc(min(kSdHalf, x.nch - h * kSdHalf) * kChunkCols);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        sd_umma(tmem + (uint32_t)(h * kSdHalf * kChunkCols), smem_desc(ys + kk * 32, 16, 1024),
                                smem_desc(bs + kk * 32, 16, 1024), idesc, (st > 0 || kk > 0) ? 1u : 0u);
                    umma_commit(&b_empty[sb]);
                    if (++sb == kSdBStages) { sb = 0; pb ^= 1; }
                }
                umma_commit(&y_empty[sy]);
                if (++sy == kSdYStages) { sy = 0; py ^= 1; }
            }
            umma_commit(acc_full); // every MMA issued, also when this lane gave up: tensor memory is released after it
        }
        __syncwarp();
    }
    // ---------------- epilogue: all warps ----------------
    {
        bool got = true;
        if (lane == 0)
            got = mbar_wait(acc_full, 0);
        if (__any_sync(0xffffffffu, !got)) ok = false;
    }
    tc_fence_before();
    if (__syncthreads_or(!ok)) {
        // a role gave up after a bounded wait: record it, then give bulk
        // copies in flight a bounded time (1 ms) to land before the CTA's
        // shared memory is released
        if (threadIdx.x == 0) {
            atomicOr(a.status, kStatusTimeout);
            const uint64_t t0 = global_ns();
            while (global_ns() - t0 < 1000000ull) {
            }
        }
    } else {
        tc_fence_after();
        // The MMAs are complete, so both rings are free: they hold the
        // staging tiles of up to kSdStageChunks chunks at a time (row-major,
        // kSdStageRow floats a row); then the entries of those chunks --
        // contiguous in the plan -- are read from them, four per thread and
        // access (the plan's entry arrays are padded to that).
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane; // TMEM lane = row of the window
        float *stage = reinterpret_cast<float *>(smem + kSdYOff);
        for (int g0 = 0; g0 < x.nch; g0 += kSdStageChunks) {
            const int ng = min(kSdStageChunks, x.nch - g0);
            for (int c = warp >> 2; c < ng; c += 2) {
#pragma unroll
                for (int cb = 0; cb < 2; cb++) {
                    uint32_t r[32];
                    tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((g0 + c) * 64 + cb * 32), r);
                    float4 *dst = reinterpret_cast<float4 *>(stage + (c * kWindowRows + row) * kSdStageRow + cb * 32);
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        dst[q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                             __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
                }
            }
            int bound[kSdStageChunks + 1];
#pragma unroll
            for (int c = 0; c <= kSdStageChunks; c++) bound[c] = __ldg(a.tile_ptr + c_first + g0 + min(c, ng));
            __syncthreads();
            const int e_begin = bound[0], e_end = bound[kSdStageChunks];
#pragma unroll 2
            for (int e0 = (e_begin & ~3) + 4 * (int)threadIdx.x; e0 < e_end; e0 += 4 * kSdThreads) {
                const uint4 v4 = __ldg(reinterpret_cast<const uint4 *>(a.entries + e0));
                const uint32_t v[4] = {v4.x, v4.y, v4.z, v4.w};
                float d[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    int c = 0;
#pragma unroll
                    for (int k = 1; k < kSdStageChunks; k++) c += e0 + u >= bound[k] ? 1 : 0;
                    const bool in = e0 + u >= e_begin && e0 + u < e_end;
                    d[u] = in ? stage[(c * kWindowRows + (v[u] >> 22)) * kSdStageRow + ((v[u] >> 16) & 63u)] : 0.f;
                }
                if (a.parts > 1) {
                    float *dst = a.partials + (size_t)x.q * a.part_stride + e0;
                    if (e0 >= e_begin && e0 + 4 <= e_end) {
                        *reinterpret_cast<float4 *>(dst) = make_float4(d[0], d[1], d[2], d[3]);
                    } else {
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if (e0 + u >= e_begin && e0 + u < e_end) dst[u] = d[u];
                    }
                } else {
                    int j[4];
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        j[u] = e0 + u >= e_begin && e0 + u < e_end ? __ldg(a.tile_src + e0 + u) : -1;
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (j[u] >= 0) j[u] = __ldg(a.src + j[u]);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (j[u] < 0)
                            continue;
                        if (a.out_f16)
                            reinterpret_cast<__half *>(a.out)[j[u]] = __float2half_rn(a.alpha * d[u]);
                        else
                            reinterpret_cast<float *>(a.out)[j[u]] = a.alpha * d[u];
                    }
                }
            }
            __syncthreads(); // the staging tiles are reused by the next group
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kSdMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
    }
}

// After a launch with parts: dA of every tensor-core entry e = alpha x (part
// 0 + part 1 + ...) in part order, written in the caller's nonzero order;
// nothing while the plan's status word says that a CTA gave up.
template <typename OutT>
__global__ void __launch_bounds__(256)
k_sddmm_sum(const float *__restrict__ partials, long long tc_nnz, long long stride, int parts,
            const int *__restrict__ tile_src, const int *__restrict__ src, const int *status, OutT *__restrict__ out,
            float alpha)
{
    asm volatile("griddepcontrol.wait;" ::: "memory"); // every part is written
    if (*(volatile const int *)status & kStatusTimeout)
        return;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < tc_nnz;
         e += (long long)gridDim.x * blockDim.x) {
        float x[8];
        float d = 0.f;
        for (int q0 = 0; q0 < parts; q0 += 8) {
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (q0 + u < parts)
                    x[u] = __ldcg(partials + (size_t)(q0 + u) * stride + e);
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (q0 + u < parts)
                    d = (q0 + u == 0) ? x[u] : d + x[u];
        }
        const int j = __ldg(src + __ldg(tile_src + e));
        if constexpr (sizeof(OutT) == 2)
            out[j] = __float2half_rn(alpha * d);
        else
            out[j] = alpha * d;
    }
}

} // namespace

// The SDDMM over the plan's tensor-core windows on the tensor cores (see the
// top of this file). dY (M x N, row stride ldy) and B (K x N, row stride ldb)
// need 16-byte aligned rows. Values of the nonzeros outside tensor-core
// windows are not written (the caller's CUDA-core pass covers them).
int sddmm_tc(const tca_plan *p, const __half *dY, int ldy, const __half *B, int ldb, int N, void *out, bool out_f16,
             float alpha, cudaStream_t s)
{
    if (p->n_tc == 0 || N == 0)
        return TCA_OK;
    // units: (window, group of up to kSdMaxChunks chunks, part of the n range)
    int max_z = 0;
    for (int t = 0; t < p->n_tc; t++) max_z = std::max(max_z, p->h_tile_first[t + 1] - p->h_tile_first[t]);
    const int n_steps = (N + 63) / 64;
    // Groups of 8 chunks while the parts of the n range fill the SMs; smaller
    // groups (dY is gathered once per group) when n has too few steps for that
    // (512 x 512 at 90 %, N = 64, 4 windows: 16.9 -> 6.1 us).
    int group_chunks = kSdMaxChunks, groups_per_win = 0, n_groups = 0, parts = 1;
    for (;; group_chunks /= 2) {
        groups_per_win = (max_z + group_chunks - 1) / group_chunks;
        n_groups = p->n_tc * groups_per_win;
        parts = std::max(1, std::min(n_steps, kSMs / n_groups));
        if (group_chunks == 1 || 2LL * n_groups * parts > kSMs)
            break;
    }
    const int steps_per_part = (n_steps + parts - 1) / parts;
    parts = (n_steps + steps_per_part - 1) / steps_per_part; // no empty part

    SdJob j{};
    TCA_TRY(encode_tensor_map_2d(&j.tmap_y, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, dY, (uint64_t)N, (uint64_t)p->M,
                                 (uint64_t)ldy * 2, 64, 1, CU_TENSOR_MAP_SWIZZLE_128B));
    TCA_TRY(encode_tensor_map_2d(&j.tmap_b, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, B, (uint64_t)N, (uint64_t)p->K,
                                 (uint64_t)ldb * 2, 64, 1, CU_TENSOR_MAP_SWIZZLE_128B));
    TCA_TRY(encode_tensor_map_2d(&j.tmap_tile, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, B, (uint64_t)N, (uint64_t)p->K,
                                 (uint64_t)ldb * 2, 64, kChunkCols, CU_TENSOR_MAP_SWIZZLE_128B));
    TCA_TRY(encode_tensor_map_2d(&j.tmap_yrun, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, dY, (uint64_t)N, (uint64_t)p->M,
                                 (uint64_t)ldy * 2, 64, kWindowRows, CU_TENSOR_MAP_SWIZZLE_128B));
    TCA_TRY(encode_tensor_map_2d(&j.tmap_run, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, B, (uint64_t)N, (uint64_t)p->K,
                                 (uint64_t)ldb * 2, 64, kSdHalf * kChunkCols, CU_TENSOR_MAP_SWIZZLE_128B));
    j.win_info = p->tc_win_info;
    j.win_cols = p->win_cols;
    j.tile_ptr = p->tile_ptr;
    j.perm = p->perm;
    j.src = p->src;
    j.tile_src = p->tile_src;
    j.entries = p->tile_entries;
    j.out = out;
    j.status = p->d_status;
    j.M = p->M;
    j.N = N;
    j.n_steps = n_steps;
    j.parts = parts;
    j.steps_per_part = steps_per_part;
    j.out_f16 = out_f16 ? 1 : 0;
    j.part_stride = (p->tc_nnz + 3) & ~3LL;
    j.alpha = alpha;
    j.n_win = p->n_tc;
    j.groups_per_win = groups_per_win;
    j.group_chunks = group_chunks;

    // with parts: the partial values, for this call only (stream-ordered;
    // under capture the graph's own memory)
    void *ws = nullptr;
    if (parts > 1) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        TCA_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
        const size_t bytes = sizeof(float) * (size_t)parts * (size_t)j.part_stride;
        if (cap == cudaStreamCaptureStatusActive)
            TCA_CUDA_TRY(cudaMallocAsync(&ws, bytes, s));
        else
            TCA_TRY(dev_malloc(&ws, bytes, s));
        j.partials = static_cast<float *>(ws);
    }
    cudaError_t e = cudaFuncSetAttribute(k_sddmm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kSdSmem);
    if (e == cudaSuccess) {
        k_sddmm_tc<<<n_groups * parts, kSdThreads, kSdSmem, s>>>(j);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && ws) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)std::min<long long>((p->tc_nnz + 255) / 256, 8LL * kSMs));
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const float *partials = j.partials;
        const int *tile_src = p->tile_src, *src = p->src, *status = p->d_status;
        const long long tc_nnz = p->tc_nnz, stride = j.part_stride;
        if (out_f16)
            e = cudaLaunchKernelEx(&cfg, k_sddmm_sum<__half>, partials, tc_nnz, stride, parts, tile_src, src, status,
                                   static_cast<__half *>(out), alpha);
        else
            e = cudaLaunchKernelEx(&cfg, k_sddmm_sum<float>, partials, tc_nnz, stride, parts, tile_src, src, status,
                                   static_cast<float *>(out), alpha);
    }
    if (ws)
        cudaFreeAsync(ws, s);
    if (e != cudaSuccess)
        return set_error(TCA_ERR_CUDA, "tensor-core SDDMM launch failed: %s", cudaGetErrorString(e));
    return TCA_OK;
}

} // namespace tca
