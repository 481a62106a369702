// spmm.cu -- blocked SpMM Y = A_blocks * X on the row-window block format.
//
// Replaces the reference's GCN SpMM kernels (gcn/SpMM/src/spmmKernel.cu:158-265
// fp16, :959-1075 tf32, :2066-2330 the "_acc" variants) behind
// SpMM_sr_bcrs.forward_{fp16,tf32}_gnn[_acc] (gcn/SpMM/src/benchmark.cpp:35-335).
//
// Design (sm_103a):
//  * One CTA per SM; a warp owns one work item = (part, chunk of FC features) at
//    a time and streams its condensed columns in chunks of 32: the gathered X
//    rows (FC features each) and the value blocks are copied global->shared with
//    16-byte cp.async ahead of the products and across item boundaries, so the
//    gather stream never drains (spmm_stream.cuh).
//  * The contraction is D[feature, row] += X^T[feature, col] * V[col, row]:
//    M = 16 features, N = 8 window rows, K = 16 columns, so the sparse block
//    is the dense B operand and the gathered rows are A.  ldmatrix.trans
//    turns the row-major gathered X tile into the A fragment; the value tile
//    feeds B through a plain ldmatrix.  fp32 accumulators stay in registers.
//    (The reference uses m16n8k8 with fp16 accumulation; this accumulates in
//    fp32.)
//  * TF32 runs m16n8k8 as a 3xTF32 split (hi*hi + hi*lo + lo*hi): fp32-level
//    accuracy.
//  * Output: a part of an unsplit window stores its whole W-row tile with
//    plain stores; parts of split windows add with red.global.add.f32.  A
//    small pre-pass, which the kernel behind it overlaps, zeroes a small Y whole
//    and of a larger one only the rows that no unsplit part writes (split
//    windows, windows without parts, trailing rows).
#include "att_common.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <mutex>
#include <string.h>
#include <type_traits>

namespace att {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;

struct PartInfo {
    int start, nreal, nsteps;
};

// A part must start and end on a block boundary of the layout the kernel
// reads (the value tile of a 16-column step is read whole); a part that does
// not is flagged and skipped instead of read past its end.
template <int WIDE>
__device__ __forceinline__ PartInfo part_check(int start, int e, int pend, int32_t *err) {
    PartInfo pi;
    pi.start = start;
    pi.nreal = e > pi.start ? e - pi.start : 0;
    if ((pi.start % WIDE) != 0 || (pend % WIDE) != 0 || pend < pi.start + pi.nreal) {
        if (err) atomicOr(err, 2);
        pi.nreal = 0;
    }
    pi.nsteps = (pi.nreal + 15) >> 4;
    return pi;
}
template <int WIDE>
__device__ __forceinline__ PartInfo part_info(const int32_t *__restrict__ rowptr, int64_t p,
                                              int32_t *err) {
    return part_check<WIDE>(__ldg(rowptr + 2 * p), __ldg(rowptr + 2 * p + 1), __ldg(rowptr + 2 * p + 2), err);
}

// XOR swizzle of the 16-byte chunk index within a shared row of `row_bytes`
template <int ROW_BYTES>
__device__ __forceinline__ int swz(int r) {
    if constexpr (ROW_BYTES >= 128) return r & 7;
    else return (r >> 1) & 3;  // 64-byte rows: two rows share a 128-byte bank window
}

}  // namespace
}  // namespace att

#include "spmm_stream.cuh"

namespace att {
namespace {

// ---------------------------------------------------------------------------
// 16-bit operand kernel (fp16 / bf16 values and features)
// ---------------------------------------------------------------------------
// The chunk stream of spmm_stream.cuh; the lane layout and the contraction are
// those described at the top of this file.
template <int W, int FC, int WIDE, int S>
struct Cfg16 : StreamCfg<FC * 2, 2, W, WIDE, S, (W == 16 ? (FC == 128 ? 12 : 16) : (FC == 32 ? 32 : 24))> {
    static constexpr int NT = W / 8;   // n8 tiles
    static constexpr int MT = FC / 16; // m16 tiles
};

// Products of 16 gathered rows (FC features; `xl`: the lane's ldmatrix.trans
// address of feature tile 0) with their values' fragments.
template <typename T, int NT, int FC>
__device__ __forceinline__ void half_mma(float (&acc)[FC / 16][NT][4], uint32_t xl, const uint32_t (&b)[NT][2]) {
#pragma unroll
    for (int j = 0; j < FC / 16; ++j) {
        uint32_t a[4];
        ldsm_x4_trans((xl ^ ((j & 3) << 5)) + (j >> 2) * 128, a[0], a[1], a[2], a[3]);
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_16816<T>(acc[j][t], a, b[t][0], b[t][1]);
    }
}

// S: chunk buffers per warp (two steps each)
template <typename T, int W, int FC, int WIDE, int S, typename IT, bool FULL>
__global__ void __launch_bounds__((Cfg16<W, FC, WIDE, S>::NW * 32), 1)
    k_spmm16(const __grid_constant__ StreamArgs A, float *__restrict__ Y, int64_t m_out, int64_t ldy) {
    using C = Cfg16<W, FC, WIDE, S>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int queue;
    const int lane = threadIdx.x & 31, warp = warp_uniform(threadIdx.x >> 5);
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    const int gid = lane >> 2, tig = lane & 3;
    // ldmatrix lanes: matrix q = lane / 8, row lane % 8
    const int q = lane >> 3, rr = lane & 7;
    const int xk = (q >> 1) * 8 + rr;
    const uint32_t xlane = sbase + xk * C::XROW + (((q & 1) ^ swz<C::XROW>(xk)) << 4);
    // 16-byte piece of the values: 8 columns (kb) of window row r
    auto vpiece = [](int kb, int r) { return WIDE == 8 ? (kb * W + r) * 16 : (kb >> 1) * W * 32 + r * 32 + (kb & 1) * 16; };
    // W 8: matrix q = columns 8 q ..; W 16: columns 8 (q & 1) .., rows 8 (q >> 1) .. of a half
    const uint32_t vlane = sbase + C::VAL + (W == 8 ? vpiece(q, rr) : vpiece(q & 1, (q >> 1) * 8 + rr));

    float acc[C::MT][C::NT][4];
#pragma unroll
    for (int j = 0; j < C::MT; ++j)
#pragma unroll
        for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;

    Stream<C, 2, FC, IT, FULL, true> st(A, lane, warp, sbase, &queue);
    while (st.more()) {
        const Chunk c = st.next();
        if (c.left > 0) {
            uint32_t b[2][C::NT][2];
            if constexpr (W == 8) {
                ldsm_x4(vlane + st.rbuf, b[0][0][0], b[0][0][1], b[1][0][0], b[1][0][1]);
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    ldsm_x4(vlane + st.rbuf + h * 32 * W, b[h][0][0], b[h][0][1], b[h][1][0], b[h][1][1]);
            }
            half_mma<T, C::NT, FC>(acc, xlane + st.rbuf, b[0]);
            if (c.left > 16) half_mma<T, C::NT, FC>(acc, xlane + st.rbuf + C::HALF, b[1]);
        }
        st.release();
        if (c.left > 32) continue;
        // ---- the part's last chunk: its W x FC tile ----
        const IT f0 = (IT)c.fc * FC + gid;
        const Target to = target(c.win, W, Y, m_out, ldy, A.tiles, A.F);
        if (to.add || A.wait) griddep_wait();  // the window's rows are zeroed by then
#pragma unroll
        for (int t = 0; t < C::NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t r = to.row0 + t * 8 + 2 * tig + h;
                float *dst = to.base + (r * to.ld + f0);
                if (r < to.limit) {
                    // Y is written once: a streaming store leaves L2 to the X rows
                    if (to.add) {
#pragma unroll
                        for (int j = 0; j < 2 * C::MT; ++j)
                            if (FULL || f0 + 8 * j < st.F) red_add_f32(dst + 8 * j, acc[j / 2][t][h + 2 * (j & 1)]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 2 * C::MT; ++j)
                            if (FULL || f0 + 8 * j < st.F) __stcs(dst + 8 * j, acc[j / 2][t][h + 2 * (j & 1)]);
                    }
                }
            }
#pragma unroll
        for (int j = 0; j < C::MT; ++j)
#pragma unroll
            for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;
    }
    cp_async_wait<0>();
    griddep_wait();  // this kernel ends after the one before it
}

constexpr uint32_t kMaxPolls = 1u << 24;  // bounded mbarrier waits

// ---------------------------------------------------------------------------
// 16-bit operand kernel with bulk row copies (8-row windows, 8-wide blocks,
// 64-feature chunks)
// ---------------------------------------------------------------------------
// Same contraction and epilogue as k_spmm16; the producer moves each gathered
// row's 128 bytes with one cp.async.bulk (lanes 0-15, one row each) instead of
// eight 16-byte cp.async spread over the warp, so the issue cost per gathered
// row drops.  Rows sit at a 144-byte pitch: the 16-byte pad keeps
// ldmatrix.trans conflict-free without a swizzle (a bulk copy cannot swizzle)
// and holds one 16-byte chunk of the step's value tile (chunk r = block r / 8,
// window row r % 8), so a stage stays 16 x 144 bytes.  Each stage completes on
// its own mbarrier (32 arrivals + the copied bytes); waits are bounded and a
// timeout sets error bit 4.  Padding rows (column -1) and value blocks past
// the part's real columns are zero-filled with shared stores instead of read.
constexpr int kBulkPitch = 144;

template <typename T, int S, typename IT>
__global__ void __launch_bounds__(kThreads) k_spmm16_bulk(
    const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
    const T *__restrict__ val, const int32_t *__restrict__ win,
    const int32_t *__restrict__ atomic, int64_t n_parts, const T *__restrict__ X, int64_t n_x_,
    int64_t F_, int64_t ldx_, float *__restrict__ Y, int64_t m_out_, int64_t ldy_, int n_chunks,
    int32_t *__restrict__ err) {
    constexpr int W = 8, WIDE = 8, FC = 64, MT = FC / 16;
    constexpr int STAGE = 16 * kBulkPitch;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[kWarps][S];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sbase = smem_u32(smem) + warp * (S * STAGE);
    const uint32_t bar0 = smem_u32(&bars[warp][0]);
    const IT n_x = (IT)n_x_, F = (IT)F_, ldx = (IT)ldx_, m_out = (IT)m_out_, ldy = (IT)ldy_;
    const IT n_items = (IT)(n_parts * n_chunks);
    const IT stride = (IT)gridDim.x * kWarps;
    const int gid = lane >> 2, tig = lane & 3;

    if (lane == 0)
        for (int s = 0; s < S; ++s) mbar_init(bar0 + 8 * s, 32);
    mbar_fence_init();
    __syncwarp();

    IT p_item = (IT)blockIdx.x * kWarps + warp;
    int p_step = 0, p_myc = -1;
    PartInfo p_pi = {0, 0, 0};
    int p_fc = 0;
    auto p_load = [&]() {
        while (p_item < n_items) {
            const IT part = p_item / n_chunks;
            p_fc = (int)(p_item - part * n_chunks);
            p_pi = part_info<WIDE>(rowptr, part, err);
            p_step = 0;
            if (p_pi.nsteps > 0) return;
            p_item += stride;
        }
    };
    auto issue = [&](int stage) {
        const uint32_t xs = sbase + stage * STAGE;
        const uint32_t bar = bar0 + 8 * stage;
        uint32_t bytes = 0;
        if (lane < 16) {
            const int r = lane;
            int cidx = p_myc;  // this lane's own column id (row r of the step)
            if ((uint64_t)(int64_t)(cidx + 1) > (uint64_t)n_x) {
                if (err) atomicOr(err, 1);
                cidx = -1;
            }
            const IT fbase = (IT)p_fc * FC;
            const uint32_t dst = xs + r * kBulkPitch;
            fence_proxy_async_smem();  // earlier generic reads of this stage before the async writes
            if (cidx >= 0) {
                const uint32_t nb = (uint32_t)(fbase + FC <= F ? FC * 2 : (F - fbase) * 2);
                bulk_g2s(dst, X + ((IT)cidx * ldx + fbase), nb, bar);
                bytes += nb;
            } else {
#pragma unroll
                for (int q = 0; q < FC * 2 / 16; ++q)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst + 16 * q), "r"(0)
                                 : "memory");
            }
            const int c0 = p_step * 16;
            const int blk = r >> 3;  // value chunk r: block r / 8, window row r % 8
            if (c0 + blk * WIDE < p_pi.nreal) {
                bulk_g2s(dst + 128, val + ((IT)(p_pi.start + c0) * W + r * 8), 16, bar);
                bytes += 16;
            } else {
                asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst + 128), "r"(0)
                             : "memory");
            }
        }
        if (bytes)
            mbar_arrive_expect_tx(bar, bytes);
        else
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
    };
    auto p_fetch = [&]() {
        p_myc = -1;
        if (p_item < n_items && p_step * 16 + (lane & 15) < p_pi.nreal)
            p_myc = __ldg(col + p_pi.start + p_step * 16 + (lane & 15));
    };
    auto p_advance = [&]() {
        if (++p_step >= p_pi.nsteps) {
            p_item += stride;
            p_load();
        }
        p_fetch();
    };

    p_load();
    p_fetch();
#pragma unroll
    for (int s = 0; s < S - 1; ++s)
        if (p_item < n_items) {
            issue(s);
            p_advance();
        }

    float acc[MT][4];
#pragma unroll
    for (int j = 0; j < MT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

    uint32_t phase = 0;  // bit s: parity of stage s's next completion
    int cstage = 0, pstage = S - 1;
    for (IT c_item = (IT)blockIdx.x * kWarps + warp; c_item < n_items; c_item += stride) {
        const IT part = c_item / n_chunks;
        const int fc = (int)(c_item - part * n_chunks);
        const PartInfo pi = part_info<WIDE>(rowptr, part, nullptr);
        for (int step = 0; step < pi.nsteps; ++step) {
            if (!mbar_wait_bounded(bar0 + 8 * cstage, (phase >> cstage) & 1u, kMaxPolls)) {
                if (err) atomicOr(err, 4);
            }
            phase ^= 1u << cstage;
            __syncwarp();
            const uint32_t xs = sbase + cstage * STAGE;
            uint32_t b0, b1;
            {
                // B: value tile rows = window rows; matrix kb = block kb
                const int kb = (lane >> 3) & 1, rr = lane & 7;
                ldsm_x2(xs + (kb * 8 + rr) * kBulkPitch + 128, b0, b1);
            }
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                const int q = lane >> 3, rr = lane & 7;
                const int k = (q >> 1) * 8 + rr;
                const int ch = 2 * j + (q & 1);
                uint32_t a[4];
                ldsm_x4_trans(xs + k * kBulkPitch + ch * 16, a[0], a[1], a[2], a[3]);
                mma_16816<T>(acc[j], a, b0, b1);
            }
            __syncwarp();
            if (p_item < n_items) {
                issue(pstage);
                p_advance();
            }
            cstage = cstage + 1 == S ? 0 : cstage + 1;
            pstage = pstage + 1 == S ? 0 : pstage + 1;
        }
        const int wrow = __ldg(win + part);
        const bool add = __ldg(atomic + part) != 0;
        const IT f0 = (IT)fc * FC;
        const bool full = f0 + FC <= F;
        const IT r0 = (IT)wrow * W + 2 * tig;
#pragma unroll
        for (int j = 0; j < MT; ++j) {
            const IT fa = f0 + 16 * j + gid;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const IT r = r0 + (h & 1);
                const IT f = fa + (h >> 1) * 8;
                if (r < m_out && (full || f < F)) {
                    float *dst = Y + (r * ldy + f);
                    if (add) red_add_f32(dst, acc[j][h]);
                    else *dst = acc[j][h];
                }
                acc[j][h] = 0.f;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// 16-bit operand kernel fed by TMA: tile::gather4 row gathers
// ---------------------------------------------------------------------------
// Same contraction and epilogue as k_spmm16; the producer is one bulk-tensor
// instruction per 4 gathered rows and 64 features instead of 16 cp.async per
// lane.  X is described by a 2-D tensor map (features x rows) with an
// 80 x 1 box and no swizzle: a gathered row occupies 160 bytes, so the 8 rows
// an ldmatrix reads fall on distinct 32-byte bank groups within a 4-row group
// (two groups share them: 2-way), and 4 rows (640 bytes) keep every TMA
// destination 128-byte aligned without padding.  Of the 80 features, the 64
// wanted plus 16 chosen outside [0, F) where possible (left of feature 0, or
// right of the last), which TMA zero-fills without reading memory.  Rows of
// padding columns are fetched from row n_x, outside the tensor, also
// zero-filled.  The step's value tile is one contiguous bulk copy.  Each
// stage completes on an mbarrier carrying the byte count; every wait is
// bounded, and a timeout raises bit 4 of err and ends the warp after draining
// its copies in flight.
constexpr int kBox = 80;            // features per TMA box
constexpr int kPitch = kBox * 2;    // bytes per gathered row in shared memory
constexpr int kGroup = 4 * kPitch;  // one gather4 destination (640 B, 128-aligned)

template <int W, int FC, int S>
struct CfgTma {
    static constexpr int FCH = FC / 64;            // 64-feature boxes per gathered row
    static constexpr int CHUNK = 4 * kGroup;       // 16 rows of one box
    static constexpr int XSTAGE = FCH * CHUNK;
    static constexpr int VSTAGE = 16 * W * 2;
    static constexpr int STAGE = (XSTAGE + VSTAGE + 127) / 128 * 128;
    static constexpr int WARP_SMEM = (S * STAGE + S * 8 + 127) / 128 * 128;
    static constexpr int SMEM = kWarps * WARP_SMEM + 128;  // + alignment slack
    static constexpr int MT = FC / 16;
    static constexpr int NT = W / 8;
};

// 16 of the 80 features of a box are extra: to the left of `fb` (box starts
// at fb - 16) unless the right side is past F (box starts at fb)
__device__ __forceinline__ bool box_left(int64_t fb, int64_t F) { return fb == 0 || fb + 64 < F; }

template <typename T, int W, int FC, int WIDE, int S>
__global__ void __launch_bounds__(kThreads) k_spmm16_tma(
    const __grid_constant__ CUtensorMap tmX, const int32_t *__restrict__ rowptr,
    const int32_t *__restrict__ col, const T *__restrict__ val, const int32_t *__restrict__ win,
    const int32_t *__restrict__ atomic, int64_t n_parts, int64_t n_x, int64_t F,
    float *__restrict__ Y, int64_t m_out, int64_t ldy, int n_chunks, int32_t *__restrict__ err) {
    using C = CfgTma<W, FC, S>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sbase = ((smem_u32(smem) + 127u) & ~127u) + warp * C::WARP_SMEM;
    const int64_t n_items = n_parts * n_chunks;
    const int64_t stride = (int64_t)gridDim.x * kWarps;
    const int gid = lane >> 2, tig = lane & 3;
    const int oob_row = (int)n_x;  // one past the last row: zero-filled by TMA
    auto xstage = [&](int stage) { return sbase + stage * C::STAGE; };
    auto vtile = [&](int stage) { return sbase + stage * C::STAGE + C::XSTAGE; };
    auto sbar = [&](int stage) { return sbase + S * C::STAGE + 8 * stage; };

    // value tiles start zeroed (a tile whose second block lies past its part
    // keeps finite data that only ever meets zero rows); barriers armed once
    for (int st = 0; st < S; ++st)
        for (int i = lane; i < C::VSTAGE / 4; i += 32)
            asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(vtile(st) + 4 * i), "r"(0) : "memory");
    if (lane == 0) {
        for (int st = 0; st < S; ++st) mbar_init(sbar(st), 1);
        mbar_fence_init();
    }
    fence_proxy_async_smem();
    __syncwarp();

    int64_t p_item = (int64_t)blockIdx.x * kWarps + warp;
    int p_step = 0, p_fc = 0, p_pend = 0, p_myc = -1;
    PartInfo p_pi = {0, 0, 0};
    auto p_load = [&]() {
        while (p_item < n_items) {
            int64_t part = p_item / n_chunks;
            p_fc = (int)(p_item - part * n_chunks);
            p_pi = part_info<WIDE>(rowptr, part, err);
            p_pend = __ldg(rowptr + 2 * part + 2);
            p_step = 0;
            if (p_pi.nsteps > 0) return;
            p_item += stride;
        }
    };
    auto issue = [&](int stage) {
        const uint32_t bar = sbar(stage);
        const int c0 = p_step * 16;
        const int vcols = min(16, p_pend - p_pi.start - c0);
        const uint32_t vbytes = (uint32_t)(vcols * W * 2);
        if (lane == 0) mbar_arrive_expect_tx(bar, C::FCH * 4 * 4 * kPitch + vbytes);
        int y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // ids of rows 4*lane+i (prefetched one step ahead)
            int cidx = __shfl_sync(0xffffffffu, p_myc, (4 * lane + i) & 15);
            if (cidx >= n_x || cidx < -1) {
                if (err && lane < 4) atomicOr(err, 1);
                cidx = -1;
            }
            y[i] = cidx >= 0 ? cidx : oob_row;
        }
        (void)c0;
        __syncwarp();
        if (lane < 4) {
#pragma unroll
            for (int ch = 0; ch < C::FCH; ++ch) {
                const int64_t fb = (int64_t)p_fc * FC + 64 * ch;
                const int x = (int)(box_left(fb, F) ? fb - 16 : fb);
                tma_gather4(xstage(stage) + ch * C::CHUNK + lane * kGroup, &tmX, x, y[0], y[1], y[2],
                            y[3], bar);
            }
        } else if (lane == 4) {
            bulk_g2s(vtile(stage), val + (int64_t)(p_pi.start + c0) * W, vbytes, bar);
        }
    };
    // column ids of the producer's position, fetched one step ahead so the
    // load latency overlaps the consumer's work instead of stalling issue()
    auto p_fetch = [&]() {
        p_myc = -1;
        if (p_item < n_items && p_step * 16 + (lane & 15) < p_pi.nreal)
            p_myc = __ldg(col + p_pi.start + p_step * 16 + (lane & 15));
    };
    auto p_advance = [&]() {
        if (++p_step >= p_pi.nsteps) {
            p_item += stride;
            p_load();
        }
        p_fetch();
    };

    p_load();
    p_fetch();
    int inflight = 0;
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (p_item < n_items) {
            issue(s);
            p_advance();
            ++inflight;
        }
    }

    float acc[C::MT][C::NT][4];
#pragma unroll
    for (int j = 0; j < C::MT; ++j)
#pragma unroll
        for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;

    uint32_t phase = 0;  // bit s: parity of stage s's next completion
    int cstage = 0, pstage = S - 1;
    for (int64_t c_item = (int64_t)blockIdx.x * kWarps + warp; c_item < n_items; c_item += stride) {
        const int64_t part = c_item / n_chunks;
        const int fc = (int)(c_item - part * n_chunks);
        const PartInfo pi = part_info<WIDE>(rowptr, part, nullptr);
        for (int step = 0; step < pi.nsteps; ++step) {
            const uint32_t bar = sbar(cstage);
            if (!mbar_wait_bounded(bar, (phase >> cstage) & 1u, kMaxPolls)) {
                // give up: record it, drain the copies still in flight, leave
                if (lane == 0 && err) atomicOr(err, 4);
                for (int k = 1; k < inflight; ++k) {
                    const int s2 = (cstage + k) % S;
                    mbar_wait_bounded(sbar(s2), (phase >> s2) & 1u, kMaxPolls);
                }
                return;
            }
            phase ^= 1u << cstage;
            --inflight;
            const uint32_t vs = vtile(cstage);
            uint32_t b[C::NT][2];
            {
                const int q = lane >> 3, rr = lane & 7;
                if constexpr (C::NT == 2) {
                    const int kb = q & 1, r = (q >> 1) * 8 + rr;
                    const int e = (kb * 8 / WIDE) * W * WIDE + r * WIDE + (kb * 8) % WIDE;
                    ldsm_x4(vs + e * 2, b[0][0], b[0][1], b[1][0], b[1][1]);
                } else {
                    const int kb = q & 1, r = rr;
                    const int e = (kb * 8 / WIDE) * W * WIDE + r * WIDE + (kb * 8) % WIDE;
                    ldsm_x2(vs + e * 2, b[0][0], b[0][1]);
                }
            }
#pragma unroll
            for (int j = 0; j < C::MT; ++j) {
                const int q = lane >> 3, rr = lane & 7;
                const int k = (q >> 1) * 8 + rr;
                const int bx = j >> 2;  // 64-feature box
                const int fo = (box_left((int64_t)fc * FC + 64 * bx, F) ? 16 : 0) + (j & 3) * 16 +
                               (q & 1) * 8;
                uint32_t a[4];
                ldsm_x4_trans(xstage(cstage) + bx * C::CHUNK + (k >> 2) * kGroup + (k & 3) * kPitch +
                                  fo * 2,
                              a[0], a[1], a[2], a[3]);
#pragma unroll
                for (int t = 0; t < C::NT; ++t) mma_16816<T>(acc[j][t], a, b[t][0], b[t][1]);
            }
            __syncwarp();
            if (p_item < n_items) {
                fence_proxy_async_smem();
                issue(pstage);
                p_advance();
                ++inflight;
            }
            cstage = cstage + 1 == S ? 0 : cstage + 1;
            pstage = pstage + 1 == S ? 0 : pstage + 1;
        }
        const int wrow = __ldg(win + part);
        const bool add = __ldg(atomic + part) != 0;
        const int64_t f0 = (int64_t)fc * FC;
#pragma unroll
        for (int t = 0; t < C::NT; ++t) {
            const int64_t r0 = (int64_t)wrow * W + t * 8 + 2 * tig;
#pragma unroll
            for (int j = 0; j < C::MT; ++j) {
                const int64_t fa = f0 + 16 * j + gid;
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int64_t r = r0 + (h & 1);
                    const int64_t f = fa + (h >> 1) * 8;
                    if (r >= 0 && r < m_out && f < F) {
                        float *dst = Y + r * ldy + f;
                        if (add) red_add_f32(dst, acc[j][t][h]);
                        else *dst = acc[j][t][h];
                    }
                    acc[j][t][h] = 0.f;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// fp32 operand kernel: 3xTF32 m16n8k8
// ---------------------------------------------------------------------------
// The chunk stream of spmm_stream.cuh.  Per 8-column k-step lane (gid, tig)
// reads rows 2 tig and 2 tig + 1 (the MMA's k = tig and tig + 4: both operands
// use this order) with 16-byte loads, conflict-free under the row swizzle;
// each brings four features of one row, the m = gid and gid + 8 elements of
// two feature tiles, so a tile's rows are features 4 gid + 2 v (+ 1) and a lane
// ends up with four adjacent features of its window rows: one float4 store.
// 169,343 nodes, mean degree 14, F = 100: 184 us a call, 9.4 TB/s into the SMs;
// with one 4-byte load per fragment element in a per-step ring it took 388.
template <int W, int FC, int WIDE, int S>
struct CfgTF32 : StreamCfg<FC * 4, 4, W, WIDE, S, (W == 16 ? 12 : 20)> {
    static constexpr int MT = FC / 16;
    static constexpr int NT = W / 8;
};

template <int W, int FC, int WIDE, int S, typename IT>
__global__ void __launch_bounds__((CfgTF32<W, FC, WIDE, S>::NW * 32), 1)
    k_spmm_tf32(const __grid_constant__ StreamArgs A, float *__restrict__ Y, int64_t m_out, int64_t ldy, int vec_out) {
    using C = CfgTF32<W, FC, WIDE, S>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int queue;
    const int lane = threadIdx.x & 31, warp = warp_uniform(threadIdx.x >> 5);
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    const unsigned char *sgen = smem + warp * C::WARP_SMEM;
    const int gid = lane >> 2, tig = lane & 3;
    const int x0off = 2 * tig * C::XROW + ((gid ^ (2 * tig)) << 4);
    const int x1off = (2 * tig + 1) * C::XROW + ((gid ^ (2 * tig + 1)) << 4);
    // values of columns 2 tig, 2 tig + 1 (of a k-step) and window row gid
    const int voff = C::VAL + 4 * ((2 * tig / WIDE * W + gid) * WIDE + 2 * tig % WIDE);

    float acc[C::MT][C::NT][4];
#pragma unroll
    for (int j = 0; j < C::MT; ++j)
#pragma unroll
        for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;

    Stream<C, 4, FC, IT, false> st(A, lane, warp, sbase, &queue);
    while (st.more()) {
        const Chunk c = st.next();
        const unsigned char *buf = sgen + st.rbuf;
#pragma unroll 1
        for (int ks = 0; 8 * ks < c.left && ks < 4; ++ks) {  // 8 columns
            const unsigned char *xs = buf + ks * 8 * C::XROW;
            uint32_t bh[C::NT][2], bl[C::NT][2];
#pragma unroll
            for (int t = 0; t < C::NT; ++t) {
                const float2 v = *reinterpret_cast<const float2 *>(buf + voff + ks * 32 * W + t * 32 * WIDE);
                split_tf32x3(v.x, bh[t][0], bl[t][0]);
                split_tf32x3(v.y, bh[t][1], bl[t][1]);
            }
#pragma unroll
            for (int u = 0; u < C::MT / 2; ++u) {
                const float4 r0 = *reinterpret_cast<const float4 *>(xs + x0off + 128 * u);
                const float4 r1 = *reinterpret_cast<const float4 *>(xs + x1off + 128 * u);
                const float x[2][4] = {{r0.x, r0.y, r1.x, r1.y}, {r0.z, r0.w, r1.z, r1.w}};
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    uint32_t ah[4], al[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) split_tf32x3(x[v][k], ah[k], al[k]);
#pragma unroll
                    for (int t = 0; t < C::NT; ++t) {
                        float(&d)[4] = acc[2 * u + v][t];
                        mma_1688_tf32(d, al[0], al[1], al[2], al[3], bh[t][0], bh[t][1]);
                        mma_1688_tf32(d, ah[0], ah[1], ah[2], ah[3], bl[t][0], bl[t][1]);
                        mma_1688_tf32(d, ah[0], ah[1], ah[2], ah[3], bh[t][0], bh[t][1]);
                    }
                }
            }
        }
        st.release();
        if (c.left > 32) continue;
        const IT f0 = (IT)c.fc * FC + 4 * gid;
        const bool add = (c.win & 3) == kAdd;
        if (add || A.wait) griddep_wait();  // the window's rows are zeroed by then
#pragma unroll
        for (int t = 0; t < C::NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t r = window_of(c.win) * W + t * 8 + 2 * tig + h;
                if (r >= m_out) continue;
                float *dst = Y + (r * ldy + f0);
#pragma unroll
                for (int u = 0; u < C::MT / 2; ++u)
                    if (f0 + 32 * u < st.F)  // F is a multiple of 4
                        put4(dst + 32 * u, add, vec_out, acc[2 * u][t][h], acc[2 * u][t][h + 2],
                             acc[2 * u + 1][t][h], acc[2 * u + 1][t][h + 2]);
            }
#pragma unroll
        for (int j = 0; j < C::MT; ++j)
#pragma unroll
            for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;
    }
    cp_async_wait<0>();
    griddep_wait();  // this kernel ends after the one before it
}

// ---------------------------------------------------------------------------
// FP8 E4M3 features with per-row fp32 scales (values fp16)
// ---------------------------------------------------------------------------
// The gathered rows are e4m3 (half the bytes of fp16), staged by 16-byte
// cp.async in a deep ring; the consumer dequantizes the step's 16 rows into
// one fp16 tile per warp -- cvt e4m3x2 -> f16x2 is exact, then one multiply by
// the row's scale (done here on X, where it cannot underflow to fp16
// subnormals as it could on the small block values) -- and runs the fp16
// ldmatrix.trans + mma.sync path with fp32 accumulation.
constexpr int kF8Stages = 3;

template <int W, int FC, int S = kF8Stages>
struct CfgF8 {
    static constexpr int XROW8 = FC;             // bytes per gathered e4m3 row
    static constexpr int XSTAGE = 16 * XROW8;
    static constexpr int VSTAGE = 16 * W * 2;
    static constexpr int SSTAGE = 64;            // 16 fp32 scales
    static constexpr int STAGE = XSTAGE + VSTAGE + SSTAGE;
    static constexpr int XROW16 = FC * 2;        // dequantized fp16 tile row
    static constexpr int TILE16 = 16 * XROW16;
    static constexpr int WARP_SMEM = S * STAGE + TILE16;
    static constexpr int SMEM = kWarps * WARP_SMEM;
    static constexpr int CPR = FC / 16;          // 16-byte e4m3 chunks per row
    static constexpr int MT = FC / 16;
    static constexpr int NT = W / 8;
    static constexpr int VCH = VSTAGE / 16;
};

__device__ __forceinline__ uint32_t e4m3x2_to_f16x2(uint16_t v) {
    uint32_t r;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;\n" : "=r"(r) : "h"(v));
    return r;
}

// IT: index type of items and element offsets (int32_t when they fit)
template <int W, int FC, int WIDE, typename IT>
__global__ void __launch_bounds__(kThreads) k_spmm_fp8(
    const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
    const __half *__restrict__ val, const int32_t *__restrict__ win,
    const int32_t *__restrict__ atomic, int64_t n_parts, const uint8_t *__restrict__ X,
    const float *__restrict__ xscale, int64_t n_x_, int64_t F_, int64_t ldx_, float *__restrict__ Y,
    int64_t m_out_, int64_t ldy_, int n_chunks, int32_t *__restrict__ err) {
    const IT n_x = (IT)n_x_, F = (IT)F_, ldx = (IT)ldx_, m_out = (IT)m_out_, ldy = (IT)ldy_;
    using C = CfgF8<W, FC>;
    constexpr int S = kF8Stages;
    static_assert(C::WARP_SMEM == S * C::STAGE + C::TILE16, "layout");
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    const unsigned char *sgen = smem + warp * C::WARP_SMEM;
    const uint32_t tile = sbase + S * C::STAGE;
    const IT n_items = (IT)(n_parts * n_chunks);
    const IT stride = (IT)gridDim.x * kWarps;
    const int gid = lane >> 2, tig = lane & 3;

    IT p_item = (IT)blockIdx.x * kWarps + warp;
    int p_step = 0, p_fc = 0, p_myc = -1;
    PartInfo p_pi = {0, 0, 0};
    auto p_load = [&]() {
        while (p_item < n_items) {
            const IT part = p_item / n_chunks;
            p_fc = (int)(p_item - part * n_chunks);
            p_pi = part_info<WIDE>(rowptr, part, err);
            p_step = 0;
            if (p_pi.nsteps > 0) return;
            p_item += stride;
        }
    };
    auto issue = [&](int stage) {
        const uint32_t xs = sbase + stage * C::STAGE;
        const uint32_t vs = xs + C::XSTAGE;
        const uint32_t ss = vs + C::VSTAGE;
        const int c0 = p_step * 16;
        int myc = p_myc;  // loaded one step ahead
        if ((uint64_t)(int64_t)(myc + 1) > (uint64_t)n_x) {  // valid: -1 .. n_x - 1
            if (err) atomicOr(err, 1);
            myc = -1;
        }
        const IT fbase = (IT)p_fc * FC;
        const bool full = fbase + FC <= F;
#pragma unroll
        for (int i = 0; i < 16 * C::CPR / 32; ++i) {
            const int idx = i * 32 + lane;
            const int r = idx / C::CPR, ch = idx % C::CPR;
            const int cidx = __shfl_sync(0xffffffffu, myc, r);
            const IT f = fbase + ch * 16;
            const bool ok = cidx >= 0 && (full || f < F);
            const IT off = ok ? (IT)cidx * ldx + f : (IT)0;
            cp_async16(xs + r * C::XROW8 + ch * 16, X + off, ok ? 16 : 0);
        }
#pragma unroll
        for (int q = lane; q < C::VCH; q += 32) {
            const int e = q * 8;
            const int blk = e / (W * WIDE);
            const bool ok = c0 + blk * WIDE < p_pi.nreal;
            const __half *src = val + ((IT)(p_pi.start + c0) * W + e);
            cp_async16(vs + q * 16, ok ? (const void *)src : (const void *)val, ok ? 16 : 0);
        }
        if (lane < 16) {
            const bool ok = myc >= 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(ss + 4 * lane),
                         "l"(ok ? xscale + myc : xscale), "r"(ok ? 4 : 0));
        }
    };
    // column ids of the producer's position, fetched one step ahead so the
    // load latency overlaps the consumer's work instead of stalling issue()
    auto p_fetch = [&]() {
        p_myc = -1;
        if (p_item < n_items && p_step * 16 + (lane & 15) < p_pi.nreal)
            p_myc = __ldg(col + p_pi.start + p_step * 16 + (lane & 15));
    };
    auto p_advance = [&]() {
        if (++p_step >= p_pi.nsteps) {
            p_item += stride;
            p_load();
        }
        p_fetch();
    };

    p_load();
    p_fetch();
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (p_item < n_items) {
            issue(s);
            p_advance();
        }
        cp_async_commit();
    }

    float acc[C::MT][C::NT][4];
#pragma unroll
    for (int j = 0; j < C::MT; ++j)
#pragma unroll
        for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;

    int cstage = 0, pstage = S - 1;
    for (IT c_item = (IT)blockIdx.x * kWarps + warp; c_item < n_items; c_item += stride) {
        const IT part = c_item / n_chunks;
        const int fc = (int)(c_item - part * n_chunks);
        const PartInfo pi = part_info<WIDE>(rowptr, part, nullptr);
        for (int step = 0; step < pi.nsteps; ++step) {
            cp_async_wait<S - 2>();
            __syncwarp();
            const unsigned char *x8 = sgen + cstage * C::STAGE;
            const float *sc = (const float *)(x8 + C::XSTAGE + C::VSTAGE);
            const uint32_t vs = sbase + cstage * C::STAGE + C::XSTAGE;
            // dequantize: 8 lanes per row, one 16-byte e4m3 chunk each
#pragma unroll
            for (int i = 0; i < 16 * C::CPR / 32; ++i) {
                const int idx = i * 32 + lane;
                const int r = idx / C::CPR, ch = idx % C::CPR;
                const uint4 raw = *reinterpret_cast<const uint4 *>(x8 + r * C::XROW8 + ch * 16);
                const __half2 s2 = __float2half2_rn(sc[r]);
                const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
                uint32_t h[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    uint32_t lo = e4m3x2_to_f16x2((uint16_t)(w[k] & 0xffffu));
                    uint32_t hi = e4m3x2_to_f16x2((uint16_t)(w[k] >> 16));
                    __half2 l2 = __hmul2(*reinterpret_cast<__half2 *>(&lo), s2);
                    __half2 h2 = __hmul2(*reinterpret_cast<__half2 *>(&hi), s2);
                    h[2 * k] = *reinterpret_cast<uint32_t *>(&l2);
                    h[2 * k + 1] = *reinterpret_cast<uint32_t *>(&h2);
                }
                // fp16 chunks 2ch, 2ch+1 of row r, XOR-swizzled as in k_spmm16
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int c16 = 2 * ch + u;
                    const uint32_t dst = tile + r * C::XROW16 + ((c16 ^ swz<C::XROW16>(r)) << 4);
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst),
                                 "r"(h[4 * u]), "r"(h[4 * u + 1]), "r"(h[4 * u + 2]),
                                 "r"(h[4 * u + 3])
                                 : "memory");
                }
            }
            __syncwarp();
            uint32_t b[C::NT][2];
            {
                const int q = lane >> 3, rr = lane & 7;
                if constexpr (C::NT == 2) {
                    const int kb = q & 1, r = (q >> 1) * 8 + rr;
                    const int e = (kb * 8 / WIDE) * W * WIDE + r * WIDE + (kb * 8) % WIDE;
                    ldsm_x4(vs + e * 2, b[0][0], b[0][1], b[1][0], b[1][1]);
                } else {
                    const int kb = q & 1, r = rr;
                    const int e = (kb * 8 / WIDE) * W * WIDE + r * WIDE + (kb * 8) % WIDE;
                    ldsm_x2(vs + e * 2, b[0][0], b[0][1]);
                }
            }
#pragma unroll
            for (int j = 0; j < C::MT; ++j) {
                const int q = lane >> 3, rr = lane & 7;
                const int k = (q >> 1) * 8 + rr;
                const int ch = 2 * j + (q & 1);
                uint32_t a[4];
                ldsm_x4_trans(tile + k * C::XROW16 + ((ch ^ swz<C::XROW16>(k)) << 4), a[0], a[1],
                              a[2], a[3]);
#pragma unroll
                for (int t = 0; t < C::NT; ++t) mma_16816<__half>(acc[j][t], a, b[t][0], b[t][1]);
            }
            __syncwarp();
            if (p_item < n_items) {
                issue(pstage);
                p_advance();
            }
            cp_async_commit();
            cstage = cstage + 1 == S ? 0 : cstage + 1;
            pstage = pstage + 1 == S ? 0 : pstage + 1;
        }
        const int wrow = __ldg(win + part);
        const bool add = __ldg(atomic + part) != 0;
        const IT f0 = (IT)fc * FC;
        const bool full = f0 + FC <= F;
#pragma unroll
        for (int t = 0; t < C::NT; ++t) {
            const IT r0 = (IT)wrow * W + t * 8 + 2 * tig;
#pragma unroll
            for (int j = 0; j < C::MT; ++j) {
                const IT fa = f0 + 16 * j + gid;
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const IT r = r0 + (h & 1);
                    const IT f = fa + (h >> 1) * 8;
                    if (r < m_out && (full || f < F)) {
                        float *dst = Y + (r * ldy + f);
                        if (add) red_add_f32(dst, acc[j][t][h]);
                        else *dst = acc[j][t][h];
                    }
                    acc[j][t][h] = 0.f;
                }
            }
        }
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// FP8 E4M3 features dequantized in registers (values fp16)
// ---------------------------------------------------------------------------
// Same staging ring as k_spmm_fp8, without the fp16 tile: ldmatrix.trans
// reads the e4m3 rows as 16-bit feature pairs, so each register holds
// features (f, f+1) of two gathered rows (c, c+1).  One byte permute regroups
// it into (f: c, c+1) | (f+1: c, c+1), and two cvt.e4m3x2 -> f16x2 give the A
// fragments of two MMA rows.  The per-row scales are folded into the B
// fragment (the step's block values, 16 gathered rows x 8 or 16 window rows):
// B' = fp16(V * s * 2^15), a few multiplies per step instead of one per A
// register, and the fp32 accumulators are multiplied by 2^-15 at the store
// (both factors are powers of two, so exact).  A step whose scaled values
// would leave fp16's normal range scales A by fp16(s) instead.  The MMA rows
// are a permutation of the features (row m < 8 is feature 2m of its
// 16-feature tile, row m + 8 is feature 2m + 1), which the epilogue undoes:
// each lane ends up owning two adjacent features of two window rows and
// stores them as float2.  This removes the shared-memory round trip of the
// fp16 tile (4 KB of shared traffic and four 16-byte stores per lane per
// step) and lets one work item cover 128 features.  2.45M nodes, F = 128:
// 1.30 ms on the chunk stream, 1.83 ms in a per-step ring (bound by issue).
constexpr float kF8Shift = 32768.f;
constexpr float kF8Unshift = 1.f / 32768.f;

constexpr unsigned kF16Min = 0x38800000u, kF16Max = 0x477fe000u;  // 2^-14 and 65504 as fp32 bits

template <int W, int FC, int WIDE>
struct CfgF8R : StreamCfg<FC, 2, W, WIDE, 2, (W == 16 ? 12 : (FC == 128 ? 20 : 24)), 128> {  // + the 32 row scales
    static constexpr int MT = FC / 16;           // 16-feature MMA tiles
    static constexpr int NT = W / 8;
};

__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, __half2 s) {
    __half2 r = __hmul2(*reinterpret_cast<__half2 *>(&a), s);
    return *reinterpret_cast<uint32_t *>(&r);
}

template <int W, int FC, int WIDE, typename IT, bool FULL>
__global__ void __launch_bounds__((CfgF8R<W, FC, WIDE>::NW * 32), 1)
    k_spmm_fp8r(const __grid_constant__ StreamArgs A, float *__restrict__ Y, int64_t m_out, int64_t ldy, int vec_out) {
    using C = CfgF8R<W, FC, WIDE>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int queue;
    const int lane = threadIdx.x & 31, warp = warp_uniform(threadIdx.x >> 5);
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    const unsigned char *sgen = smem + warp * C::WARP_SMEM;
    const int gid = lane >> 2, tig = lane & 3;
    // ldmatrix lane roles: matrix mi = lane / 8 holds gathered rows
    // (mi / 2) * 8 + lane % 8 and 16-feature piece (mi % 2) of a 32-feature pair
    const int q = lane >> 3, rr = lane & 7;
    const int lm_k = (q >> 1) * 8 + rr;
    const uint32_t xlane = sbase + lm_k * C::XROW + (((q & 1) ^ swz<C::XROW>(lm_k)) << 4);
    // value pieces as in k_spmm16
    auto vpiece = [](int kb, int r) { return WIDE == 8 ? (kb * W + r) * 16 : (kb >> 1) * W * 32 + r * 32 + (kb & 1) * 16; };
    const uint32_t vlane = sbase + C::VAL + vpiece(q & 1, (W == 16 ? (q >> 1) * 8 : 0) + rr);

    float acc[C::MT][C::NT][4];
#pragma unroll
    for (int j = 0; j < C::MT; ++j)
#pragma unroll
        for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;

    Stream<C, 1, FC, IT, FULL> st(A, lane, warp, sbase, &queue);
    while (st.more()) {
        const Chunk c = st.next();
        const float *scales = reinterpret_cast<const float *>(sgen + st.rbuf + C::EXT);
#pragma unroll 1  // unrolled it spills at this register bound
        for (int hf = 0; hf < 2 && 16 * hf < c.left; ++hf) {
            uint32_t b[C::NT][2];
            if constexpr (W == 16) ldsm_x4(vlane + st.rbuf + hf * 32 * W, b[0][0], b[0][1], b[1][0], b[1][1]);
            else ldsm_x2(vlane + st.rbuf + hf * 32 * W, b[0][0], b[0][1]);
            const uint32_t xl = xlane + st.rbuf + hf * C::HALF;
            // scale pairs of the gathered rows this lane's A fragments hold:
            // rows (2 tig, 2 tig + 1) and (8 + 2 tig, 9 + 2 tig)
            const float2 s_lo = *reinterpret_cast<const float2 *>(scales + 16 * hf + 2 * tig);
            const float2 s_hi = *reinterpret_cast<const float2 *>(scales + 16 * hf + 8 + 2 * tig);
            // The row scales go on the B fragment: b[t][0] holds the values of
            // gathered rows (2 tig, 2 tig + 1), b[t][1] of (8 + 2 tig, 9 + 2 tig),
            // exactly the rows of the lane's scale pairs.  V * s is multiplied
            // by kF8Shift (2^15) into fp16's normal range, so the accumulators
            // hold 2^15 * Y until the store; if any scaled value of the step
            // would be neither zero nor a normal fp16, the warp scales A
            // instead for that step (accumulators brought back to 1 * Y around
            // it, exact: powers of two).
            const float sk[4] = {s_lo.x * kF8Shift, s_lo.y * kF8Shift, s_hi.x * kF8Shift, s_hi.y * kF8Shift};
            uint32_t bs[C::NT][2];
            // magnitudes as integers order like the floats; 0 - 1 wraps, so a
            // zero never is the smallest (and a NaN is above any finite value)
            unsigned lo = ~0u, hi = 0;
#pragma unroll
            for (int t = 0; t < C::NT; ++t) {
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(&b[t][g]));
                    const float p0 = v.x * sk[2 * g], p1 = v.y * sk[2 * g + 1];
                    const unsigned m0 = __float_as_uint(p0) & 0x7fffffffu, m1 = __float_as_uint(p1) & 0x7fffffffu;
                    lo = min(lo, min(m0 - 1, m1 - 1));
                    hi = max(hi, max(m0, m1));
                    const __half2 hp = __floats2half2_rn(p0, p1);
                    bs[t][g] = *reinterpret_cast<const uint32_t *>(&hp);
                }
            }
            const bool bside = __all_sync(0xffffffffu, lo >= kF16Min - 1 && hi <= kF16Max);
            auto products = [&](auto scaled, __half2 h_lo, __half2 h_hi) {
                constexpr bool kScaleA = decltype(scaled)::value;
#pragma unroll
                for (int jp = 0; jp < C::MT / 2; ++jp) {
                    uint32_t R[4];  // (rows 0-7 | 8-15) x (tile 2jp | 2jp+1)
                    ldsm_x4_trans(xl ^ (jp << 5), R[0], R[1], R[2], R[3]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // bytes (f: c, f+1: c, f: c+1, f+1: c+1) -> (f: c, c+1 | f+1: c, c+1)
                        const uint32_t p0 = __byte_perm(R[h], 0, 0x3120);      // rows 2tig, 2tig+1
                        const uint32_t p1 = __byte_perm(R[h + 2], 0, 0x3120);  // rows 8+2tig, 9+2tig
                        uint32_t a[4];
                        a[0] = e4m3x2_to_f16x2((uint16_t)(p0 & 0xffffu));
                        a[1] = e4m3x2_to_f16x2((uint16_t)(p0 >> 16));
                        a[2] = e4m3x2_to_f16x2((uint16_t)(p1 & 0xffffu));
                        a[3] = e4m3x2_to_f16x2((uint16_t)(p1 >> 16));
                        if constexpr (kScaleA) {
                            a[0] = hmul2_u32(a[0], h_lo);
                            a[1] = hmul2_u32(a[1], h_lo);
                            a[2] = hmul2_u32(a[2], h_hi);
                            a[3] = hmul2_u32(a[3], h_hi);
                        }
#pragma unroll
                        for (int t = 0; t < C::NT; ++t)
                            mma_16816<__half>(acc[2 * jp + h][t], a, kScaleA ? b[t][0] : bs[t][0],
                                              kScaleA ? b[t][1] : bs[t][1]);
                    }
                }
            };
            if (bside) {
                products(std::false_type{}, __half2{}, __half2{});
            } else {
#pragma unroll
                for (int j = 0; j < C::MT; ++j)
#pragma unroll
                    for (int t = 0; t < C::NT; ++t)
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[j][t][k] *= kF8Unshift;
                products(std::true_type{}, __floats2half2_rn(s_lo.x, s_lo.y), __floats2half2_rn(s_hi.x, s_hi.y));
#pragma unroll
                for (int j = 0; j < C::MT; ++j)
#pragma unroll
                    for (int t = 0; t < C::NT; ++t)
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[j][t][k] *= kF8Shift;
            }
        }
        st.release();
        if (c.left > 32) continue;
        // epilogue: tile j, lane -> features f0 + 16 j + 2 gid (+1), window
        // rows t * 8 + 2 tig (+1); F is a multiple of 16, so both features of
        // a pair are inside F together
        const bool add = (c.win & 3) == kAdd;
        if (add || A.wait) griddep_wait();  // the window's rows are zeroed by then
        const IT f0 = (IT)c.fc * FC + 2 * gid;
#pragma unroll
        for (int t = 0; t < C::NT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t r = window_of(c.win) * W + t * 8 + 2 * tig + h;
                if (r >= m_out) continue;
                float *dst = Y + (r * ldy + f0);
#pragma unroll
                for (int j = 0; j < C::MT; ++j)
                    if (FULL || f0 + 16 * j < st.F)
                        put2(dst + 16 * j, add, vec_out, acc[j][t][h] * kF8Unshift, acc[j][t][h + 2] * kF8Unshift);
            }
#pragma unroll
        for (int j = 0; j < C::MT; ++j)
#pragma unroll
            for (int t = 0; t < C::NT; ++t) acc[j][t][0] = acc[j][t][1] = acc[j][t][2] = acc[j][t][3] = 0.f;
    }
    cp_async_wait<0>();
    griddep_wait();  // this kernel ends after the one before it
}

// ---------------------------------------------------------------------------
// Batched SpMM over many graphs in one launch (the serving loop's kernel)
// ---------------------------------------------------------------------------
// The job table lives in device memory: a header {n_jobs, total items, total
// empty windows, total multi-group windows, work counter} and, per job, the
// block format, its groups, X and Y of one graph plus exclusive prefixes of its
// work items (groups x feature chunks), empty windows and multi-group windows.
// Launch parameters are only the table pointers, so one launch captured in a
// CUDA graph can be replayed every scheduler tick after the table is
// rewritten.  A group (<= group_parts consecutive parts of one window, chosen
// when the groups are built) is one contiguous run of condensed columns, so it
// streams like one long part.  Warps take work items from a queue (the
// counter header[4]): the first item of each warp is fixed, the rest come
// from an atomic counter, which evens out items of very different lengths
// (one step to 16 x group_parts steps).  The per-warp cp.async pipeline runs
// across item and job boundaries as in k_spmm16; a small per-warp ring in
// shared memory hands the producer's item sequence to the consumer.

// find the job whose [begin, next begin) range of `which` (0 items, 1 empty
// windows, 2 multi-group windows) holds v
__device__ __forceinline__ int64_t find_prefix(const att_spmm_job *__restrict__ jobs, int64_t n_jobs,
                                               int64_t v, int which) {
    int64_t lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        const int64_t b = which == 0 ? jobs[mid].item_begin
                          : which == 1 ? jobs[mid].empty_begin : jobs[mid].red_begin;
        if (b <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// A job's element offsets (X rows, Y rows, partial slots) fit in 31 bits:
// the batched kernel computes them in 32-bit arithmetic and skips (error bit
// 8) a job that does not fit instead of addressing it.
__device__ __forceinline__ bool job_small(const att_spmm_job *j) {
    const int64_t lim = (int64_t)INT32_MAX - 4096;
    return j->n_x * j->ldx < lim && j->m_out * j->ldy < lim && j->n_slots * 8 * j->F < lim &&
           j->F < lim && j->ldx < lim && j->ldy < lim;
}

// The chunk stream of spmm_stream.cuh over the job table: the same cursors, with
// an item's pointers (X, values, ids of its job) beside its chunk, and two more
// stages ahead of the fetch cursor because an item is found through the table
// (job, group, part).  Items are drawn in increasing order, so a warp's job
// search goes forward from its last job.
using CfgBatch = StreamCfg<128, 2, 8, 8, 2, 20>;

struct BatchStream {
    using C = CfgBatch;
    static constexpr int FC = 64, W = 8;
    struct Work {
        int start, left;       // first condensed column, real columns left in the group
        int fc;                // feature chunk, -1: no more items
        int job, g, win;       // win -1: the job does not fit 32-bit offsets, nothing is stored
    };
    const att_spmm_job *const jobs;
    int64_t *const header;
    int32_t *const err;
    const int lane;
    const uint32_t sbase;
    const int n_items, n_jobs;
    uint32_t xdst, idsrc;
    int ch;
    // drawn -> group range in flight -> rowptr in flight -> entered
    int d_after;                                        // lane 0, in flight
    int job, job_begin, job_end;                        // of the last item found
    int r_job, r_g, r_fc, r_p0, r_p1;
    int e_job, e_g, e_fc, e_start, e_end, e_pend, e_win;
    Work f, p, pend;
    int fid;
    const int32_t *f_col;
    const char *p_X;
    const char *p_val;
    int p_row_bytes;
    unsigned n_x;
    bool started;
    bool p_whole, p_live;                               // p_live: the lane's piece lies inside F
    uint32_t wbuf, rbuf;

    __device__ __forceinline__ BatchStream(const att_spmm_job *jobs_, int64_t *header_, int32_t *err_, int lane_,
                                           int warp, uint32_t sbase_)
        : jobs(jobs_), header(header_), err(err_), lane(lane_), sbase(sbase_), n_items((int)header_[1]),
          n_jobs((int)header_[0]) {
        const int rg = lane / C::CPR;
        ch = lane % C::CPR;
        xdst = sbase + rg * C::RPL * C::XROW + ((ch ^ swz<C::XROW>(rg * C::RPL)) << 4);
        idsrc = sbase + C::IDS + rg * C::RPL * 4;
        job = -1;
        job_begin = job_end = 0;
        started = false;
        find((int)blockIdx.x * C::NW + warp);
        draw();
        rows();
        enter();
        wbuf = rbuf = 0;
        take();
        copy();
        pend = p;
        wbuf = C::BUF;
        __syncwarp();  // the copied chunk's ids have been read
        take();
    }
    __device__ __forceinline__ void draw() {
        if (lane == 0)
            d_after = (int)gridDim.x * C::NW + (int)atomicAdd(reinterpret_cast<unsigned int *>(header + 4), 1u);
    }
    // item's job, group and feature chunk; the group's parts in flight
    __device__ __forceinline__ void find(int item) {
        r_fc = -1;
        r_p0 = r_p1 = 0;
        if (item >= n_items || item < 0) return;
        while (item >= job_end) {
            ++job;
            job_begin = warp_uniform((int)jobs[job].item_begin);
            job_end = job + 1 < n_jobs ? warp_uniform((int)jobs[job + 1].item_begin) : n_items;
        }
        // counted in 64 bits: a width that does not fit is skipped further on
        const int nch = warp_uniform((int)((jobs[job].F + FC - 1) / FC));
        const int local = item - job_begin;
        r_job = job;
        r_g = nch == 1 ? local : local / nch;
        r_fc = local - r_g * nch;
        r_p0 = __ldg(jobs[job].group_part + r_g);
        r_p1 = __ldg(jobs[job].group_part + r_g + 1);
    }
    __device__ __forceinline__ void rows() {
        e_job = r_job;
        e_g = r_g;
        e_fc = r_fc;
        e_start = e_end = e_pend = 0;
        e_win = -1;
        if (e_fc >= 0) {
            const att_spmm_job *j = jobs + e_job;
            e_start = __ldg(j->rowptr + 2 * r_p0);
            e_end = __ldg(j->rowptr + 2 * r_p1 - 1);
            e_pend = __ldg(j->rowptr + 2 * r_p1);
            e_win = __ldg(j->window_of_part + r_p0);
        }
        const int nxt = warp_uniform(d_after);
        draw();
        find(nxt);
    }
    __device__ __forceinline__ void fetch_ids() { fid = lane < f.left ? __ldg(f_col + f.start + lane) : -1; }
    __device__ __forceinline__ void enter() {
        const PartInfo pi = part_check<8>(e_start, e_end, e_pend, err);
        f.start = warp_uniform(pi.start);
        f.left = warp_uniform(pi.nreal);
        f.fc = e_fc;
        f.job = e_job;
        f.g = e_g;
        f.win = warp_uniform(e_win);
        if (f.fc >= 0) {
            const att_spmm_job *j = jobs + f.job;
            f_col = j->col;
            if (!job_small(j)) {  // not addressed: nothing gathered, nothing stored
                if (err) atomicOr(err, 8);
                f.left = 0;
                f.win = -1;
            }
        }
        rows();
        fetch_ids();
    }
    __device__ __forceinline__ void take() {
        const bool same = p_is(f);
        p = f;
        if (p.fc < 0) return;
        const att_spmm_job *j = jobs + p.job;
        if (!same) {
            const int F = (int)j->F, fe = p.fc * FC + ch * 8;
            p_live = fe < F;
            p_X = reinterpret_cast<const char *>(j->X) + 2 * (int64_t)fe;
            p_val = reinterpret_cast<const char *>(j->val) + lane * 16;
            p_row_bytes = 2 * (int)j->ldx;
            n_x = (unsigned)j->n_x;
        }
        int c = fid;  // valid ids are -1 (padding) .. n_x - 1
        const bool none = (unsigned)c >= n_x;
        if (none && c != -1) {
            if (err) atomicOr(err, 1);
            c = -1;
        }
        p_whole = !__any_sync(0xffffffffu, none);
        asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(sbase + C::IDS + 4 * lane), "r"(c) : "memory");
        if (f.left > 32) {
            f.start += 32;
            f.left -= 32;
            fetch_ids();
        } else {
            enter();
        }
        __syncwarp();
    }
    // the chunk continues the copy cursor's item
    __device__ __forceinline__ bool p_is(const Work &w) {
        const bool same = started && w.job == p.job && w.g == p.g && w.fc == p.fc;
        started = true;
        return same;
    }
    template <bool WHOLE>
    __device__ __forceinline__ void copy_half(uint32_t dst, uint32_t ids) {
        auto at = [&](int k) { return (dst ^ (swz<C::XROW>(k) << 4)) + k * C::XROW; };
        int id[C::RPL];
        lds_ids<C::RPL>(id, ids);
#pragma unroll
        for (int k = 0; k < C::RPL; ++k) {
            const bool ok = WHOLE || id[k] >= 0;
            cp_async16(at(k), p_X + (ok ? (int64_t)id[k] * p_row_bytes : 0), ok ? 16 : 0);
        }
    }
    __device__ __forceinline__ void copy() {
        if (p.fc >= 0 && p.left > 0) {
            if (p_live) {  // pieces past F stay as they are (their products are never stored)
                if (p_whole) {
                    copy_half<true>(xdst + wbuf, idsrc);
                    copy_half<true>(xdst + wbuf + C::HALF, idsrc + 64);
                } else {
                    copy_half<false>(xdst + wbuf, idsrc);
                    if (p.left > 16) copy_half<false>(xdst + wbuf + C::HALF, idsrc + 64);
                }
            }
            const bool ok = lane / 8 * 8 < p.left;  // a block past the group's real columns is zeros
            cp_async16(sbase + C::VAL + wbuf + lane * 16, ok ? p_val + (int64_t)p.start * (W * 2) : p_val, ok ? 16 : 0);
        }
        cp_async_commit();
    }
    __device__ __forceinline__ bool more() const { return pend.fc >= 0; }
    __device__ __forceinline__ Work next() {
        const Work c = pend;
        copy();
        pend = p;
        __syncwarp();  // the copied chunk's ids have been read
        take();
        wbuf ^= C::BUF;
        cp_async_wait<1>();
        __syncwarp();
        return c;
    }
    __device__ __forceinline__ void release() {
        __syncwarp();
        rbuf ^= C::BUF;
    }
};

__global__ void __launch_bounds__(CfgBatch::NW * 32, 1)
    k_spmm16_batched(const att_spmm_job *__restrict__ jobs, int64_t *__restrict__ header, int32_t *__restrict__ err) {
    using C = CfgBatch;
    constexpr int FC = 64, MT = FC / 16;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = warp_uniform(threadIdx.x >> 5);
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    // items, and the draws past them (three a warp), must be 32-bit
    if (header[1] > (int64_t)INT32_MAX - 4 * (int64_t)gridDim.x * C::NW - 1) {
        if (err && threadIdx.x == 0 && blockIdx.x == 0) atomicOr(err, 8);
        return;
    }
    const int gid = lane >> 2, tig = lane & 3;
    const int q = lane >> 3, rr = lane & 7;
    const int xk = (q >> 1) * 8 + rr;
    const uint32_t xlane = sbase + xk * C::XROW + (((q & 1) ^ swz<C::XROW>(xk)) << 4);
    const uint32_t vlane = sbase + C::VAL + lane * 16;

    float acc[MT][1][4];
#pragma unroll
    for (int j = 0; j < MT; ++j) acc[j][0][0] = acc[j][0][1] = acc[j][0][2] = acc[j][0][3] = 0.f;

    BatchStream st(jobs, header, err, lane, warp, sbase);
    while (st.more()) {
        const BatchStream::Work c = st.next();
        if (c.left > 0) {
            uint32_t b[2][1][2];
            ldsm_x4(vlane + st.rbuf, b[0][0][0], b[0][0][1], b[1][0][0], b[1][0][1]);
            half_mma<__half, 1, FC>(acc, xlane + st.rbuf, b[0]);
            if (c.left > 16) half_mma<__half, 1, FC>(acc, xlane + st.rbuf + C::HALF, b[1]);
        }
        st.release();
        if (c.left > 32) continue;
        if (c.win >= 0) {
            const att_spmm_job *cj = jobs + c.job;
            const int slot = __ldg(cj->group_slot + c.g);
            const int F = (int)cj->F, m_out = (int)cj->m_out, f0 = c.fc * FC + gid;
            // whole window: rows of Y; else rows of partial slot `slot` ([8, F], ld F)
            float *const base = slot < 0 ? cj->Y + c.win * 8 * (int)cj->ldy : cj->partial + slot * 8 * F;
            const int ld = slot < 0 ? (int)cj->ldy : F;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int rl = 2 * tig + h;
                if (c.win * 8 + rl >= m_out) continue;
                float *dst = base + rl * ld + f0;
#pragma unroll
                for (int j = 0; j < 2 * MT; ++j)
                    if (f0 + 8 * j < F) dst[8 * j] = acc[j / 2][0][h + 2 * (j & 1)];
            }
        }
#pragma unroll
        for (int j = 0; j < MT; ++j) acc[j][0][0] = acc[j][0][1] = acc[j][0][2] = acc[j][0][3] = 0.f;
    }
    cp_async_wait<0>();
}

// First pass of the batched SpMM: resets the work counter and zeroes the
// rows of windows that own no part (listed per job in empty_win; one warp per
// window).
template <int W>
__global__ void k_zero_empty_batched(const att_spmm_job *__restrict__ jobs, int64_t *__restrict__ header) {
    if (blockIdx.x == 0 && threadIdx.x == 0) header[4] = 0;
    const int lane = threadIdx.x & 31;
    const int64_t n_jobs = header[0], n_e = header[2];
    const int64_t wstride = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t ge = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; ge < n_e; ge += wstride) {
        const att_spmm_job *j = jobs + find_prefix(jobs, n_jobs, ge, 1);
        const int64_t w = __ldg(j->empty_win + (ge - j->empty_begin));
        const int64_t r1 = (w + 1) * W < j->m_out ? (w + 1) * W : j->m_out;
        for (int64_t r = w * W; r < r1; ++r)
            for (int64_t f = lane; f < j->F; f += 32) j->Y[r * j->ldy + f] = 0.f;
    }
}

// Last pass: Y rows of a multi-group window = sum of its groups' partial slots
// in group order.  One CTA per window; a thread per (row, 4 features).  The
// window's slots are consecutive: [group_slot[first group], group_slot[first
// group of the next multi-group window]) (n_slots after the last).
template <int W>
__global__ void __launch_bounds__(256) k_reduce_groups_batched(const att_spmm_job *__restrict__ jobs,
                                                               const int64_t *__restrict__ header) {
    const int64_t n_jobs = header[0], n_r = header[3];
    for (int64_t gr = blockIdx.x; gr < n_r; gr += gridDim.x) {
        const att_spmm_job *j = jobs + find_prefix(jobs, n_jobs, gr, 2);
        if (!job_small(j)) continue;  // skipped by the main pass (error bit 8)
        const int64_t k = gr - j->red_begin;
        const int g0 = __ldg(j->red_first + k);
        const int64_t w = __ldg(j->window_of_part + __ldg(j->group_part + g0));
        const int s0 = __ldg(j->group_slot + g0);
        const int s1 = k + 1 < j->n_red ? __ldg(j->group_slot + __ldg(j->red_first + k + 1))
                                        : (int)j->n_slots;
        const int64_t F = j->F, F4 = F >> 2;
        const float4 *part = reinterpret_cast<const float4 *>(j->partial);
        for (int64_t u = threadIdx.x; u < W * F4; u += blockDim.x) {
            const int64_t rl = u / F4, f4 = u - rl * F4;
            const int64_t r = w * W + rl;
            if (r >= j->m_out) continue;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            int sl = s0;
#pragma unroll 4
            for (; sl < s1; ++sl) {
                const float4 v = __ldg(part + ((int64_t)sl * W + rl) * F4 + f4);
                s.x += v.x;
                s.y += v.y;
                s.z += v.z;
                s.w += v.w;
            }
            float *y = j->Y + r * j->ldy + f4 * 4;
            y[0] = s.x;
            y[1] = s.y;
            y[2] = s.z;
            y[3] = s.w;
        }
    }
}

// ---- groups of a block format -------------------------------------------------
// Per part p of window w (parts of a window are consecutive): rank = p - first
// part of w, np = parts of w.  p starts a group when rank % G == 0; a window
// with np > G is multi-group: each of its groups owns a partial slot and its
// first group opens a reduction entry.  The three flags are packed in 21-bit
// fields of one int64 and scanned together.  Empty windows (no part) below
// n_windows are listed by a second scan.
constexpr int kFieldBits = 21;
constexpr int64_t kFieldMask = (int64_t(1) << kFieldBits) - 1;

__device__ __forceinline__ int64_t lower_bound_win(const int32_t *__restrict__ win, int64_t P, int64_t w) {
    int64_t a = 0, b = P;
    while (a < b) {
        const int64_t m = (a + b) >> 1;
        if (__ldg(win + m) < w) a = m + 1; else b = m;
    }
    return a;
}

__device__ __forceinline__ void part_rank(const int32_t *__restrict__ win, int64_t P, int64_t p,
                                          int64_t &rank, int64_t &np) {
    const int32_t w = __ldg(win + p);
    int64_t a = 0, b = p;
    while (a < b) {
        const int64_t m = (a + b) >> 1;
        if (__ldg(win + m) < w) a = m + 1; else b = m;
    }
    int64_t c = p + 1, d = P;
    while (c < d) {
        const int64_t m = (c + d) >> 1;
        if (__ldg(win + m) <= w) c = m + 1; else d = m;
    }
    rank = p - a;
    np = c - a;
}

__global__ void k_group_flags(const int32_t *__restrict__ win, int64_t P, int G,
                              int64_t *__restrict__ flags) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    int64_t rank, np;
    part_rank(win, P, p, rank, np);
    const int64_t gs = rank % G == 0, multi = np > G;
    flags[p] = gs | ((gs & multi) << kFieldBits) | ((int64_t)(multi && rank == 0) << (2 * kFieldBits));
}

__global__ void k_group_scatter(const int32_t *__restrict__ win, int64_t P, int G,
                                const int64_t *__restrict__ scanned, int32_t *__restrict__ group_part,
                                int32_t *__restrict__ group_slot, int32_t *__restrict__ red_first,
                                int64_t *__restrict__ counts) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (P == 0) {
        if (p == 0) {
            group_part[0] = 0;
            red_first[0] = 0;
            counts[0] = counts[1] = counts[2] = 0;
        }
        return;
    }
    if (p >= P) return;
    int64_t rank, np;
    part_rank(win, P, p, rank, np);
    const bool gs = rank % G == 0, multi = np > G;
    const int64_t ex = scanned[p];
    const int64_t gi = ex & kFieldMask, si = (ex >> kFieldBits) & kFieldMask, ri = ex >> (2 * kFieldBits);
    if (gs) {
        group_part[gi] = (int32_t)p;
        group_slot[gi] = multi ? (int32_t)si : -1;
    }
    if (multi && rank == 0) red_first[ri] = (int32_t)gi;
    if (p == P - 1) {
        const int64_t ng = gi + gs, ns = si + (gs && multi), nr = ri + (multi && rank == 0);
        group_part[ng] = (int32_t)P;
        red_first[nr] = (int32_t)ng;
        counts[0] = ng;
        counts[1] = nr;
        counts[2] = ns;
    }
}

__global__ void k_empty_flags(const int32_t *__restrict__ win, int64_t P, int64_t n_windows,
                              int64_t *__restrict__ flags) {
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= n_windows) return;
    const int64_t a = lower_bound_win(win, P, w);
    flags[w] = !(a < P && __ldg(win + a) == w);
}

__global__ void k_empty_scatter(const int32_t *__restrict__ win, int64_t P, int64_t n_windows,
                                const int64_t *__restrict__ scanned, int32_t *__restrict__ empty_win,
                                int64_t *__restrict__ counts) {
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n_windows == 0) {
        if (w == 0) counts[3] = 0;
        return;
    }
    if (w >= n_windows) return;
    const int64_t a = lower_bound_win(win, P, w);
    const bool empty = !(a < P && __ldg(win + a) == w);
    if (empty) empty_win[scanned[w]] = (int32_t)w;
    if (w == n_windows - 1) counts[3] = scanned[w] + empty;
}

// Zeroes the rows of Y that no unsplit part stores (windows whose parts add
// with red.add, windows without parts, rows past the last window) for the SpMM
// kernel behind it.  Eight lanes per part, plus one group for the end: the
// first part of each window zeroes the windows between the previous part's
// window and its own, and its own window when that window is split; the extra
// group zeroes the windows after the last part's.  No searches: every group
// reads at most two window ids and one flag.  A gap of many windows (a graph
// with long runs of empty rows) is shared by the whole warp.  The SpMM kernel
// is launched as this one's programmatic dependent, so it gathers meanwhile
// and waits only before its first addition (or its end); with the two in
// sequence, this pass was 8 of 54 us on the 169,343-node graph and 27 us of
// 1,770 on the 2.45M-node one.
__global__ void k_zero_uncovered(const int32_t *__restrict__ win, const int32_t *__restrict__ atomic,
                                 int64_t n_parts, int W, float *__restrict__ Y, int64_t m_out,
                                 int64_t F, int64_t ldy, int vec) {
    griddep_launch();
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const int64_t n_w = (m_out + W - 1) / W;
    const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    int64_t g0 = 0, g1 = 0, own = -1;  // gap [g0, g1) and the own window to zero
    if (p < n_parts) {
        const int64_t w = __ldg(win + p);
        const int64_t prev = p > 0 ? (int64_t)__ldg(win + p - 1) : -1;
        if (prev != w) {
            g0 = prev + 1;
            g1 = w;
            if (__ldg(atomic + p) != 0) own = w;
        }
    } else if (p == n_parts) {
        g0 = n_parts > 0 ? (int64_t)__ldg(win + n_parts - 1) + 1 : 0;
        g1 = n_w;
    }
    g0 = g0 < 0 ? 0 : g0;
    g1 = g1 > n_w ? n_w : g1;
    if (own >= n_w) own = -1;
    // lane `i` of `n` zeroes its share of the rows of windows [w0, w1)
    auto zero = [&](int64_t w0, int64_t w1, int i, int n) {
        const int64_t r1 = w1 * W < m_out ? w1 * W : m_out;
        for (int64_t r = w0 * W; r < r1; ++r) {
            float *row = Y + r * ldy;
            if (vec)
                for (int64_t f = 4 * i; f < F; f += 4 * n)
                    *reinterpret_cast<float4 *>(row + f) = make_float4(0.f, 0.f, 0.f, 0.f);
            else
                for (int64_t f = i; f < F; f += n) row[f] = 0.f;
        }
    };
    if (own >= 0) zero(own, own + 1, sub, 8);
    const bool large = g1 - g0 > 32;
    if (g1 > g0 && !large) zero(g0, g1, sub, 8);
    unsigned m = __ballot_sync(0xffffffffu, large && sub == 0);
    while (m) {
        const int l = __ffs(m) - 1;
        m &= m - 1;
        zero(__shfl_sync(0xffffffffu, g0, l), __shfl_sync(0xffffffffu, g1, l), lane, 32);
    }
}

// Y up to this size is zeroed whole, whatever the order of the windows (and of a
// window's parts); the SpMM kernel then waits before its first store.
// k_zero_uncovered takes larger ones and needs ascending windows.  It is the
// cheaper of the two near the limit (65,536 nodes, degree 10, F = 128: 30 us a
// call against 36; 16,384 nodes, F = 64: 20.8 against 19.2), but small part lists
// in any order are calls that this function takes.
constexpr int64_t kZeroAllBytes = 32ll << 20;
inline bool zero_all(int64_t m_out, int64_t ldy) {
    return m_out <= kZeroAllBytes / (int64_t)sizeof(float) / ldy;
}

__global__ void k_zero_all(float *__restrict__ Y, int64_t m_out, int64_t F, int64_t ldy, int vec) {
    griddep_launch();
    const int64_t per = vec ? F >> 2 : F;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m_out * per) return;
    const int64_t r = t / per, f = t - r * per;
    if (vec) *reinterpret_cast<float4 *>(Y + r * ldy + 4 * f) = make_float4(0.f, 0.f, 0.f, 0.f);
    else Y[r * ldy + f] = 0.f;
}

// Adds the tiles of split windows to Y (rows that the zero pass cleared): for each
// run of three and more parts of one window, their tiles in part order with the
// rounding errors kept beside the sum (Knuth's two-sum), as exactly as in fp64.  A
// block looks at 256 parts and 64 float4s of their tiles.  Its four groups of 64
// threads share the short runs that open there, a run each; a long one is cut into
// four stretches (a hub has hundreds of parts, read eight at a time), whose sums
// meet in order.
// With red.add in the kernel itself the order in which parts end decides the last
// bits of a split window's rows, and a layer that rounds them to 16 bits shows it
// (its weight gradient varies by up to 6e-5 from run to run).  us a call without and with this: 169,343 nodes, F = 64 43,
// 54; 472,772 nodes of degree 35, F = 128 323, 369; 2.45M nodes, F = 128 1,549, 1,714.
// Bound by the latency of short chains: the tiles of the middle one are 122 MB, 46 us.
struct TileSum {
    float s[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
    __device__ __forceinline__ void add(const float (&x)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float t = s[i] + x[i], b = t - s[i];
            e[i] += (s[i] - (t - b)) + (x[i] - b);
            s[i] = t;
        }
    }
    // n tiles of `per` float4s, eight in flight
    __device__ __forceinline__ void add(const float4 *src, int64_t n, int per) {
        for (; n > 0; n -= 8, src += 8 * (int64_t)per) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < n) v[u] = __ldcs(src + u * (int64_t)per);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < n) add({v[u].x, v[u].y, v[u].z, v[u].w});
        }
    }
    // an infinite or NaN sum has no error term
    __device__ __forceinline__ float get(int i) const { return isfinite(s[i]) ? s[i] + e[i] : s[i]; }
};

constexpr int kLongRun = 8;

template <int W>
__global__ void __launch_bounds__(256, 4) k_merge_tiles(const int32_t *__restrict__ win, const int32_t *__restrict__ atomic,
                                                        int64_t n_parts, const float4 *__restrict__ tiles, int F,
                                                        float *__restrict__ Y, int64_t m_out, int64_t ldy, int vec) {
    __shared__ int s_win[256 + 32], s_short[256], s_long[256], s_n[2];
    __shared__ TileSum part[3][64];
    const int lane = threadIdx.x & 31, group = threadIdx.x >> 6, place = threadIdx.x & 63;
    const int64_t p0 = (int64_t)blockIdx.x * 256, p = p0 + threadIdx.x;
    const int w = p < n_parts ? __ldg(win + p) : -1;
    const int before = p > 0 && p < n_parts ? __ldg(win + p - 1) : -1;
    const bool split = p < n_parts && __ldg(atomic + p) != 0;
    s_win[threadIdx.x] = w;
    if (threadIdx.x < 32) s_win[256 + threadIdx.x] = p + 256 < n_parts ? __ldg(win + p + 256) : -1;
    if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
    __syncthreads();
    if (split && w != before) {  // runs of one and two were added by the SpMM kernel
        int n = 1;
        while (n <= kLongRun && s_win[threadIdx.x + n] == w) ++n;
        if (n > kLongRun) s_long[atomicAdd(&s_n[1], 1)] = threadIdx.x;
        else if (n > 2) s_short[atomicAdd(&s_n[0], 1)] = threadIdx.x | n << 16;
    }
    __syncthreads();
    griddep_wait();
    const int per = W / 4 * F;  // float4s of a tile
    const int o = blockIdx.y * 64 + place;
    const bool live = o < per;
    auto put = [&](const TileSum &t, int wq) {  // features 4 o .. 4 o + 3 of the tile
        const int r = 4 * o / F;
        const int64_t row = (int64_t)wq * W + r;
        // added, not stored: parts of one window need not stand together in a small list
        if (row >= 0 && row < m_out) put4(Y + row * ldy + (4 * o - r * F), true, vec, t.get(0), t.get(1), t.get(2), t.get(3));
    };
    for (int i = group; i < s_n[0]; i += 4) {
        const int l = s_short[i] & 0xffff, n = s_short[i] >> 16;
        if (!live) break;
        TileSum t;
        t.add(tiles + (p0 + l) * per + o, n, per);
        put(t, s_win[l]);
    }
    for (int i = 0; i < s_n[1]; ++i) {
        const int l = s_long[i], wq = s_win[l];
        int64_t n = kLongRun + 1;
        for (;;) {
            const int64_t k = p0 + l + n + lane;
            const unsigned other = ~__ballot_sync(0xffffffffu, k < n_parts && __ldg(win + k) == wq);
            n += other ? __ffs(other) - 1 : 32;
            if (other) break;
        }
        const int64_t k0 = n * group / 4, k1 = n * (group + 1) / 4;
        TileSum t;
        if (live) t.add(tiles + (p0 + l + k0) * per + o, k1 - k0, per);
        if (group > 0) part[group - 1][place] = t;
        __syncthreads();
        if (group == 0 && live) {
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const TileSum &u = part[g][place];
                t.add(u.s);
#pragma unroll
                for (int j = 0; j < 4; ++j) t.e[j] += u.e[j];
            }
            put(t, wq);
        }
        __syncthreads();
    }
}

template <typename K>
int occupancy_grid(K kernel, int smem, int64_t items) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem);
    if (per_sm < 1) per_sm = 1;
    int64_t want = (items + kWarps - 1) / kWarps;
    int64_t cap = (int64_t)sm_count() * per_sm;
    return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

// Launches a kernel that may start while the one before it on the stream (one
// that calls griddep_launch) still runs; it calls griddep_wait before it
// touches what that one writes.
template <typename... P, typename... Q>
int launch_dependent(void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t st, const char *what,
                     const Q &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    return launch_status(what);  // and clears the error: the next launch must not report it
}

// A kernel as a type, for the generic lambdas that launch one of several
template <auto K>
struct KernelOf {
    static constexpr auto value = K;
};

template <int W>
int merge_tiles(const int32_t *win, const int32_t *atomic, int64_t n_parts, const float *tiles, int64_t F, float *Y,
                int64_t m_out, int64_t ldy, cudaStream_t st) {
    const int vec = ldy % 4 == 0 && ((uintptr_t)Y & 15) == 0;
    const dim3 grid((unsigned)((n_parts + 255) / 256), (unsigned)((W / 4 * F + 63) / 64));
    return launch_dependent(k_merge_tiles<W>, grid, 256, 0, st, "k_merge_tiles", win, atomic, n_parts,
                            reinterpret_cast<const float4 *>(tiles), (int)F, Y, m_out, ldy, vec);
}

template <typename T, int W, int FC, int WIDE, int S>
int launch16(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
             const int32_t *atomic, int64_t n_parts, const void *X, int64_t n_x, int64_t F,
             int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int32_t *err, float *tiles, cudaStream_t st) {
    using C = Cfg16<W, FC, WIDE, S>;
    const int n_chunks = (int)((F + FC - 1) / FC);
    const int64_t items = n_parts * n_chunks;
    if (items == 0) return ATT_OK;
    // 32-bit items (plus one grid stride of overshoot) and row pitch of X;
    // offsets into X, Y and the values are 64-bit either way
    const int64_t lim = INT32_MAX - (1 << 22);
    const bool small = ldx * (int64_t)sizeof(T) < lim && F < lim && items < lim;
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int prep = dynamic_smem<kernel>(C::SMEM);
        if (prep != ATT_OK) return prep;
        const int grid = (int)(items < sm_count() ? items : sm_count());
        const StreamArgs A{rowptr, col, win, atomic, val, X, nullptr, n_parts, n_x, F, ldx, n_chunks, zero_all(m_out, ldy), tiles, err};
        const int s = launch_dependent(kernel, grid, C::NW * 32, C::SMEM, st, "k_spmm16", A, Y, m_out, ldy);
        return s != ATT_OK || !tiles ? s : merge_tiles<W>(win, atomic, n_parts, tiles, F, Y, m_out, ldy, st);
    };
    if (small && F % FC == 0) return run(KernelOf<k_spmm16<T, W, FC, WIDE, S, int32_t, true>>{});
    if (small) return run(KernelOf<k_spmm16<T, W, FC, WIDE, S, int32_t, false>>{});
    return run(KernelOf<k_spmm16<T, W, FC, WIDE, S, int64_t, false>>{});
}

template <typename T, int S>
int launch16_bulk(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
                  const int32_t *atomic, int64_t n_parts, const void *X, int64_t n_x, int64_t F,
                  int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int32_t *err,
                  cudaStream_t st) {
    constexpr int SMEM = kWarps * S * 16 * kBulkPitch;
    const int n_chunks = (int)((F + 63) / 64);
    const int64_t items = n_parts * n_chunks;
    if (items == 0) return ATT_OK;
    const int64_t lim = INT32_MAX - (1 << 22);
    const bool small = n_x * ldx < lim && m_out * ldy < lim && items < lim;
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int prep = dynamic_smem<kernel>(SMEM);
        if (prep != ATT_OK) return prep;
        const int grid = occupancy_grid(kernel, SMEM, items);
        kernel<<<grid, kThreads, SMEM, st>>>(rowptr, col, (const T *)val, win, atomic, n_parts,
                                             (const T *)X, n_x, F, ldx, Y, m_out, ldy, n_chunks, err);
        return launch_status("k_spmm16_bulk");
    };
    if (small) return run(KernelOf<k_spmm16_bulk<T, S, int32_t>>{});
    return run(KernelOf<k_spmm16_bulk<T, S, int64_t>>{});
}

template <int W, int FC, int WIDE, int S>
int launch_tf32(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
                const int32_t *atomic, int64_t n_parts, const void *X, int64_t n_x, int64_t F,
                int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int32_t *err, cudaStream_t st) {
    using C = CfgTF32<W, FC, WIDE, S>;
    const int n_chunks = (int)((F + FC - 1) / FC);
    const int64_t items = n_parts * n_chunks;
    if (items == 0) return ATT_OK;
    const int64_t lim = INT32_MAX - (1 << 22);  // as in launch16
    const bool small = ldx * 4 < lim && F < lim && items < lim;
    const int vec_out = ldy % 4 == 0 && ((uintptr_t)Y & 15) == 0;
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int prep = dynamic_smem<kernel>(C::SMEM);
        if (prep != ATT_OK) return prep;
        const int grid = (int)(items < sm_count() ? items : sm_count());
        const StreamArgs A{rowptr, col, win, atomic, val, X, nullptr, n_parts, n_x, F, ldx, n_chunks, zero_all(m_out, ldy), nullptr, err};
        return launch_dependent(kernel, grid, C::NW * 32, C::SMEM, st, "k_spmm_tf32", A, Y, m_out, ldy, vec_out);
    };
    if (small) return run(KernelOf<k_spmm_tf32<W, FC, WIDE, S, int32_t>>{});
    return run(KernelOf<k_spmm_tf32<W, FC, WIDE, S, int64_t>>{});
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

template <typename T, int W, int FC, int WIDE, int S>
int launch16_tma(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
                 const int32_t *atomic, int64_t n_parts, const void *X, int64_t n_x, int64_t F,
                 int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int32_t *err, cudaStream_t st) {
    using C = CfgTma<W, FC, S>;
    constexpr auto kernel = k_spmm16_tma<T, W, FC, WIDE, S>;
    const int prep = dynamic_smem<kernel>(C::SMEM);
    if (prep != ATT_OK) return prep;
    const int n_chunks = (int)((F + FC - 1) / FC);
    const int64_t items = n_parts * n_chunks;
    if (items == 0) return ATT_OK;
    CUtensorMap tm;
    const cuuint64_t gdim[2] = {(cuuint64_t)F, (cuuint64_t)n_x};
    const cuuint64_t gstride[1] = {(cuuint64_t)ldx * sizeof(T)};
    const cuuint32_t box[2] = {(cuuint32_t)kBox, 1};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = tensor_map_encoder()(
        &tm, sizeof(T) == 2 && std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                               : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
        2, const_cast<void *>(X), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    ATT_CHECK(r == CUDA_SUCCESS, ATT_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    const int grid = occupancy_grid(kernel, C::SMEM, items);
    kernel<<<grid, kThreads, C::SMEM, st>>>(tm, rowptr, col, (const T *)val, win, atomic, n_parts,
                                            n_x, F, Y, m_out, ldy, n_chunks, err);
    return launch_status("k_spmm16_tma");
}

constexpr int kTmaStages = 5;

// Launch-shape options of att_spmm.  Each has a process-wide default
// (att_set_option, atomic) and a per-thread override (att_set_thread_option,
// -1 = follow the default), so a caller -- or the autotuner -- can pick the
// shape of its own calls without changing the shape of calls made by other
// threads.
//  * spmm_gather: row-gather mechanism of the 16-bit kernel, 0 = cp.async
//    (default), 1 = TMA tile::gather4, 2 = cp.async.bulk per row.
//  * spmm_stages / spmm_fc: chunk buffers per warp of the 16-bit kernel (2, 3:
//    two; 4: three) and features per work item for F > 64 (a thread's 64 or 128 and
//    a process-wide 128 are taken as they are; the process-wide 64, the default,
//    leaves the choice to wide_items).  Three buffers gain nothing: 2.45M
//    nodes, F = 128, 64 features x 2 buffers 1,727 us, x 3 1,737; 128 x 2 1,555,
//    x 3 1,667.
//  * spmm_fp8: 1 = A fragments dequantized in registers (k_spmm_fp8r, 128
//    features per item when F > 64), 0 = through an fp16 shared tile
//    (k_spmm_fp8).
//  * spmm_tf32: fp32-feature (3xTF32) kernel shape 0..3 (dispatch_fc32).
enum SpmmOpt { kOptGather = 0, kOptStages, kOptFc, kOptFp8, kOptTf32, kNumOpts };
const char *const kOptNames[kNumOpts] = {"spmm_gather", "spmm_stages", "spmm_fc", "spmm_fp8",
                                         "spmm_tf32"};
std::atomic<int> g_opt[kNumOpts] = {{0}, {3}, {64}, {1}, {0}};
thread_local int t_opt[kNumOpts] = {-1, -1, -1, -1, -1};

inline int opt(SpmmOpt i) {
    const int v = t_opt[i];
    return v >= 0 ? v : g_opt[i].load(std::memory_order_relaxed);
}

int opt_index(const char *key) {
    for (int i = 0; i < kNumOpts; ++i)
        if (strcmp(key, kOptNames[i]) == 0) return i;
    return -1;
}

bool opt_valid(int i, int v) {
    switch (i) {
        case kOptGather: return v >= 0 && v <= 2;
        case kOptStages: return v == 2 || v == 3 || v == 4;
        case kOptFc: return v == 64 || v == 128;
        case kOptFp8: return v == 0 || v == 1;
        case kOptTf32: return v >= 0 && v <= 3;
    }
    return false;
}

template <int W, int FC, int WIDE>
int launch_fp8(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
               const int32_t *atomic, int64_t n_parts, const void *X, const float *xscale,
               int64_t n_x, int64_t F, int64_t ldx, float *Y, int64_t m_out, int64_t ldy,
               int32_t *err, cudaStream_t st) {
    using C = CfgF8<W, FC>;
    const int n_chunks = (int)((F + FC - 1) / FC);
    const int64_t items = n_parts * n_chunks;
    if (items == 0) return ATT_OK;
    const int64_t lim = INT32_MAX - (1 << 22);
    const bool small = n_x * ldx < lim && m_out * ldy < lim && items < lim;
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int prep = dynamic_smem<kernel>(C::SMEM);
        if (prep != ATT_OK) return prep;
        const int grid = occupancy_grid(kernel, C::SMEM, items);
        kernel<<<grid, kThreads, C::SMEM, st>>>(rowptr, col, (const __half *)val, win, atomic,
                                                n_parts, (const uint8_t *)X, xscale, n_x, F, ldx,
                                                Y, m_out, ldy, n_chunks, err);
        return launch_status("k_spmm_fp8");
    };
    if (small) return run(KernelOf<k_spmm_fp8<W, FC, WIDE, int32_t>>{});
    return run(KernelOf<k_spmm_fp8<W, FC, WIDE, int64_t>>{});
}

template <int W, int FC, int WIDE>
int launch_fp8r(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
                const int32_t *atomic, int64_t n_parts, const void *X, const float *xscale,
                int64_t n_x, int64_t F, int64_t ldx, float *Y, int64_t m_out, int64_t ldy,
                int32_t *err, cudaStream_t st) {
    using C = CfgF8R<W, FC, WIDE>;
    const int n_chunks = (int)((F + FC - 1) / FC);
    const int64_t items = n_parts * n_chunks;
    if (items == 0) return ATT_OK;
    const int64_t lim = INT32_MAX - (1 << 22);  // as in launch16
    const bool small = ldx < lim && F < lim && items < lim;
    const int vec_out = (ldy % 2 == 0 && ((uintptr_t)Y & 7) == 0) ? 1 : 0;
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int prep = dynamic_smem<kernel>(C::SMEM);
        if (prep != ATT_OK) return prep;
        const int grid = (int)(items < sm_count() ? items : sm_count());
        const StreamArgs A{rowptr, col, win, atomic, val, X, xscale, n_parts, n_x, F, ldx, n_chunks, zero_all(m_out, ldy), nullptr, err};
        return launch_dependent(kernel, grid, C::NW * 32, C::SMEM, st, "k_spmm_fp8r", A, Y, m_out, ldy, vec_out);
    };
    if (small && F % FC == 0) return run(KernelOf<k_spmm_fp8r<W, FC, WIDE, int32_t, true>>{});
    if (small) return run(KernelOf<k_spmm_fp8r<W, FC, WIDE, int32_t, false>>{});
    return run(KernelOf<k_spmm_fp8r<W, FC, WIDE, int64_t, false>>{});
}

// Features per work item of the 16-bit kernel where the caller has not chosen:
// 128 when that leaves no more than half a 64-feature item unused in the last
// item (an even number of 64-feature items) and there are at least 4096 parts
// (two items for each of the 152 x 12 warps that take them); else 64.  The 128-wide
// item reads a part's column list and values once for twice the features and
// gathers twice the bytes per id.  Same additions in the same order, so the
// results are the same.  us, 64 against 128 features per item, 8-row windows:
//   parts        F = 72        96          128         136         192         256
//   0.7K      12.2 12.3   12.1 12.3   11.6 11.4   12.9 14.8   12.2 14.2   13.1 13.1
//   2.1K      17.2 17.4   16.7 17.5   15.9 16.0   18.8 24.1   18.2 22.5   20.6 21.1
//   4.9K      34.9 30.3   30.8 28.8   28.8 27.2
//   8.1K      32.4 29.9   31.2 29.3   29.0 28.4
//   22K       85.4 72.3   78.8 67.7   71.9 66.8    112  148    103  121    130  119
//   2.45M nodes           2100 1490   1734 1549                           3884 3363
// and 16-row windows (300,000 nodes, degree 20) 309 246 at 96, 299 271 at 128.
constexpr int64_t kWideItemParts = 4096;
inline bool wide_items(int64_t F, int64_t n_parts) {
    if (t_opt[kOptFc] >= 0) return t_opt[kOptFc] == 128;
    if (g_opt[kOptFc].load(std::memory_order_relaxed) == 128) return true;
    return (F + 63) / 64 % 2 == 0 && n_parts >= kWideItemParts;
}
inline int item_features(int64_t F, int64_t n_parts) {
    return F <= 32 ? 32 : F <= 64 || !wide_items(F, n_parts) ? 64 : 128;
}

template <typename T, int W, int WIDE>
int dispatch_fc16(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
                  const int32_t *atomic, int64_t n_parts, const void *X, int64_t n_x, int64_t F,
                  int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int32_t *err, float *tiles,
                  cudaStream_t st) {
    // TMA row gathers for F >= 64 (the tensor map's 64-feature box fits); the
    // cp.async kernel for narrower features or an X without rows
    if (opt(kOptGather) == 1 && F >= 64 && n_x > 0 && n_x < INT32_MAX &&
        tensor_map_encoder() != nullptr) {
        if (F <= 64)
            return launch16_tma<T, W, 64, WIDE, kTmaStages>(rowptr, col, val, win, atomic, n_parts,
                                                            X, n_x, F, ldx, Y, m_out, ldy, err, st);
        return launch16_tma<T, W, 128, WIDE, kTmaStages>(rowptr, col, val, win, atomic, n_parts, X,
                                                         n_x, F, ldx, Y, m_out, ldy, err, st);
    }
    if (F <= 32)
        return launch16<T, W, 32, WIDE, 2>(rowptr, col, val, win, atomic, n_parts, X, n_x, F, ldx, Y,
                                        m_out, ldy, err, tiles, st);
    if constexpr (W == 8 && WIDE == 8) {
        if (opt(kOptGather) == 2 && (F <= 64 || opt(kOptFc) != 128))
            return launch16_bulk<T, 3>(rowptr, col, val, win, atomic, n_parts, X, n_x, F, ldx, Y,
                                       m_out, ldy, err, st);
    }
#define ATT_L16S(FCv, Sv)                                                                       \
    return launch16<T, W, FCv, WIDE, Sv>(rowptr, col, val, win, atomic, n_parts, X, n_x, F, ldx, \
                                         Y, m_out, ldy, err, tiles, st)
    if (item_features(F, n_parts) == 64) {
        if (opt(kOptStages) == 4) ATT_L16S(64, 3);
        ATT_L16S(64, 2);
    }
    if (opt(kOptStages) == 4) ATT_L16S(128, 3);
    ATT_L16S(128, 2);
#undef ATT_L16S
}

template <int W, int WIDE>
int dispatch_fc32(const int32_t *rowptr, const int32_t *col, const void *val, const int32_t *win,
                  const int32_t *atomic, int64_t n_parts, const void *X, int64_t n_x, int64_t F,
                  int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int32_t *err,
                  cudaStream_t st) {
#define ATT_LTF(FCv, Sv)                                                                        \
    return launch_tf32<W, FCv, WIDE, Sv>(rowptr, col, val, win, atomic, n_parts, X, n_x, F, ldx, \
                                         Y, m_out, ldy, err, st)
    // shapes (features per item x chunk buffers): 0, 3 = 64 x 2, 1 = 32 x 2,
    // 2 = 32 x 3 (F <= 32 always takes 32-feature items).  169,343 nodes, mean
    // degree 14, us for shapes 0, 1, 2: F 64 92, 103, 121; F 100 184, 195, 230;
    // F 128 171, 191, 226 (rows of 400 bytes do not start on 128-byte lines)
    if (F <= 32 || opt(kOptTf32) == 1 || opt(kOptTf32) == 2) {
        if (opt(kOptTf32) == 2) ATT_LTF(32, 3);
        ATT_LTF(32, 2);
    }
    ATT_LTF(64, 2);
#undef ATT_LTF
}

}  // namespace
}  // namespace att

using namespace att;

namespace att {
namespace {

// tiles: null, or att_spmm_scratch_bytes of scratch for the parts of split windows
int spmm(const int32_t *rowptr, const int32_t *col, const void *val, int val_dtype, const int32_t *window_of_part,
         const int32_t *atomic, int64_t n_parts, const void *X, int x_dtype, const float *x_scale, int64_t n_x_rows,
         int64_t F, int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int window, int wide, int32_t *err_flag,
         float *tiles, cudaStream_t st) {
    ATT_CHECK(n_parts >= 0 && m_out >= 0 && F >= 0 && n_x_rows >= 0, ATT_ERR_INVALID,
              "negative size");
    ATT_CHECK(window == 8 || window == 16, ATT_ERR_UNSUPPORTED, "window must be 8 or 16, got %d",
              window);
    ATT_CHECK(m_out == 0 || F == 0 || Y != nullptr, ATT_ERR_INVALID, "Y is null");
    ATT_CHECK(ldy >= F, ATT_ERR_INVALID, "ldy %lld < F %lld", (long long)ldy, (long long)F);
    ATT_CHECK(n_parts == 0 || (rowptr && col && val && window_of_part && atomic && X),
              ATT_ERR_INVALID, "null format or X pointer");
    if (m_out == 0 || F == 0) return ATT_OK;
    // the grid of k_merge_tiles: 64 float4s of a tile a block, at most 65,535 blocks in y
    if (F > 65535 * 64 / (window / 4)) tiles = nullptr;
    int s = ATT_OK;
    {
        const int64_t threads = (n_parts + 1) * 8;
        const int vec = F % 4 == 0 && ldy % 4 == 0 && ((uintptr_t)Y & 15) == 0;
        if (zero_all(m_out, ldy)) {
            const int64_t n = m_out * (vec ? F / 4 : F);
            k_zero_all<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(Y, m_out, F, ldy, vec);
            s = launch_status("k_zero_all");
        } else {
            k_zero_uncovered<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(
                window_of_part, atomic, n_parts, window, Y, m_out, F, ldy, vec);
            s = launch_status("k_zero_uncovered");
        }
        if (s != ATT_OK) return s;
    }
    if (n_parts == 0) return ATT_OK;
    const bool is16 = (val_dtype == ATT_F16 && x_dtype == ATT_F16) ||
                      (val_dtype == ATT_BF16 && x_dtype == ATT_BF16);
    if (is16) {
        ATT_CHECK(wide == 8 || wide == 16, ATT_ERR_UNSUPPORTED,
                  "16-bit values need wide 8 or 16, got %d", wide);
        ATT_CHECK(F % 8 == 0 && ldx % 8 == 0 && ((uintptr_t)X & 15) == 0 && ((uintptr_t)val & 15) == 0,
                  ATT_ERR_UNSUPPORTED,
                  "16-bit SpMM needs F and ldx multiples of 8 and 16-byte aligned X and values");
        ATT_CHECK(ldx >= F, ATT_ERR_INVALID, "ldx < F");
#define ATT_SPMM16(T, Wv, WIDEv)                                                             \
    return dispatch_fc16<T, Wv, WIDEv>(rowptr, col, val, window_of_part, atomic, n_parts, X, \
                                       n_x_rows, F, ldx, Y, m_out, ldy, err_flag, tiles, st)
        if (val_dtype == ATT_F16) {
            if (window == 8 && wide == 8) ATT_SPMM16(__half, 8, 8);
            if (window == 8 && wide == 16) ATT_SPMM16(__half, 8, 16);
            if (window == 16 && wide == 8) ATT_SPMM16(__half, 16, 8);
            ATT_SPMM16(__half, 16, 16);
        } else {
            if (window == 8 && wide == 8) ATT_SPMM16(__nv_bfloat16, 8, 8);
            if (window == 8 && wide == 16) ATT_SPMM16(__nv_bfloat16, 8, 16);
            if (window == 16 && wide == 8) ATT_SPMM16(__nv_bfloat16, 16, 8);
            ATT_SPMM16(__nv_bfloat16, 16, 16);
        }
#undef ATT_SPMM16
    }
    if (val_dtype == ATT_F32 && x_dtype == ATT_F32) {
        ATT_CHECK(wide == 4 || wide == 8, ATT_ERR_UNSUPPORTED, "fp32 values need wide 4 or 8, got %d",
                  wide);
        ATT_CHECK(F % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)X & 15) == 0 && ((uintptr_t)val & 15) == 0,
                  ATT_ERR_UNSUPPORTED,
                  "fp32 SpMM needs F and ldx multiples of 4 and 16-byte aligned X and values");
        ATT_CHECK(ldx >= F, ATT_ERR_INVALID, "ldx < F");
        if (window == 8 && wide == 4)
            return dispatch_fc32<8, 4>(rowptr, col, val, window_of_part, atomic, n_parts, X,
                                       n_x_rows, F, ldx, Y, m_out, ldy, err_flag, st);
        if (window == 8 && wide == 8)
            return dispatch_fc32<8, 8>(rowptr, col, val, window_of_part, atomic, n_parts, X,
                                       n_x_rows, F, ldx, Y, m_out, ldy, err_flag, st);
        if (window == 16 && wide == 4)
            return dispatch_fc32<16, 4>(rowptr, col, val, window_of_part, atomic, n_parts, X,
                                        n_x_rows, F, ldx, Y, m_out, ldy, err_flag, st);
        return dispatch_fc32<16, 8>(rowptr, col, val, window_of_part, atomic, n_parts, X, n_x_rows,
                                    F, ldx, Y, m_out, ldy, err_flag, st);
    }
    if (val_dtype == ATT_F16 && x_dtype == ATT_F8E4M3) {
        ATT_CHECK(x_scale != nullptr, ATT_ERR_INVALID, "fp8 features need per-row scales");
        ATT_CHECK(wide == 8 || wide == 16, ATT_ERR_UNSUPPORTED, "fp16 values need wide 8 or 16");
        ATT_CHECK(F % 16 == 0 && ldx % 16 == 0 && ((uintptr_t)X & 15) == 0 &&
                      ((uintptr_t)val & 15) == 0 && ldx >= F,
                  ATT_ERR_UNSUPPORTED,
                  "fp8 SpMM needs F and ldx multiples of 16 and 16-byte aligned X and values");
#define ATT_F8R(Wv, FCv, WIDEv)                                                                \
    return launch_fp8r<Wv, FCv, WIDEv>(rowptr, col, val, window_of_part, atomic, n_parts, X,   \
                                       x_scale, n_x_rows, F, ldx, Y, m_out, ldy, err_flag, st)
        if (opt(kOptFp8) == 1) {
            if (F > 64) {
                if (window == 8) { if (wide == 8) ATT_F8R(8, 128, 8); ATT_F8R(8, 128, 16); }
                if (wide == 8) ATT_F8R(16, 128, 8);
                ATT_F8R(16, 128, 16);
            }
            if (window == 8) { if (wide == 8) ATT_F8R(8, 64, 8); ATT_F8R(8, 64, 16); }
            if (wide == 8) ATT_F8R(16, 64, 8);
            ATT_F8R(16, 64, 16);
        }
#undef ATT_F8R
#define ATT_F8(Wv, FCv, WIDEv)                                                                \
    return launch_fp8<Wv, FCv, WIDEv>(rowptr, col, val, window_of_part, atomic, n_parts, X,   \
                                      x_scale, n_x_rows, F, ldx, Y, m_out, ldy, err_flag, st)
        // 64 features per work item: like the 16-bit kernel, throughput
        // follows resident warps per SM
        if (window == 8) { if (wide == 8) ATT_F8(8, 64, 8); ATT_F8(8, 64, 16); }
        if (wide == 8) ATT_F8(16, 64, 8);
        ATT_F8(16, 64, 16);
#undef ATT_F8
    }
    set_error("unsupported (val_dtype=%d, x_dtype=%d) combination", val_dtype, x_dtype);
    return ATT_ERR_UNSUPPORTED;
}

}  // namespace
}  // namespace att

extern "C" int att_spmm(const int32_t *rowptr, const int32_t *col, const void *val, int val_dtype,
                        const int32_t *window_of_part, const int32_t *atomic, int64_t n_parts,
                        const void *X, int x_dtype, const float *x_scale, int64_t n_x_rows,
                        int64_t F, int64_t ldx, float *Y, int64_t m_out, int64_t ldy, int window,
                        int wide, int32_t *err_flag, void *stream) {
    clear_error();
    return spmm(rowptr, col, val, val_dtype, window_of_part, atomic, n_parts, X, x_dtype, x_scale, n_x_rows, F, ldx, Y,
                m_out, ldy, window, wide, err_flag, nullptr, (cudaStream_t)stream);
}

extern "C" size_t att_spmm_scratch_bytes(int64_t n_parts, int window, int64_t F) {
    if (n_parts <= 0 || window <= 0 || F <= 0) return 0;
    return (size_t)n_parts * (size_t)window * (size_t)F * sizeof(float);
}

extern "C" int att_spmm_ordered(const int32_t *rowptr, const int32_t *col, const void *val, int val_dtype,
                                const int32_t *window_of_part, const int32_t *atomic, int64_t n_parts, const void *X,
                                int x_dtype, const float *x_scale, int64_t n_x_rows, int64_t F, int64_t ldx, float *Y,
                                int64_t m_out, int64_t ldy, int window, int wide, int32_t *err_flag, void *scratch,
                                size_t scratch_bytes, void *stream) {
    clear_error();
    const size_t need = att_spmm_scratch_bytes(n_parts, window, F);
    ATT_CHECK(need == 0 || (scratch && ((uintptr_t)scratch & 15) == 0 && scratch_bytes >= need), ATT_ERR_WORKSPACE,
              "scratch of %zu bytes, %zu needed (16-byte aligned)", scratch_bytes, need);
    return spmm(rowptr, col, val, val_dtype, window_of_part, atomic, n_parts, X, x_dtype, x_scale, n_x_rows, F, ldx, Y,
                m_out, ldy, window, wide, err_flag, need ? (float *)scratch : nullptr, (cudaStream_t)stream);
}

extern "C" int att_set_option(const char *key, int value) {
    clear_error();
    ATT_CHECK(key != nullptr, ATT_ERR_INVALID, "null option name");
    const int i = opt_index(key);
    ATT_CHECK(i >= 0, ATT_ERR_INVALID, "unknown option '%s'", key);
    ATT_CHECK(opt_valid(i, value), ATT_ERR_INVALID, "invalid value %d for option '%s'", value,
              key);
    g_opt[i].store(value, std::memory_order_relaxed);
    return ATT_OK;
}

extern "C" int att_set_thread_option(const char *key, int value) {
    clear_error();
    ATT_CHECK(key != nullptr, ATT_ERR_INVALID, "null option name");
    const int i = opt_index(key);
    ATT_CHECK(i >= 0, ATT_ERR_INVALID, "unknown option '%s'", key);
    ATT_CHECK(value == -1 || opt_valid(i, value), ATT_ERR_INVALID,
              "invalid value %d for option '%s'", value, key);
    t_opt[i] = value;
    return ATT_OK;
}

extern "C" int att_get_option(const char *key, int *value) {
    clear_error();
    ATT_CHECK(key != nullptr && value != nullptr, ATT_ERR_INVALID, "null argument");
    const int i = opt_index(key);
    ATT_CHECK(i >= 0, ATT_ERR_INVALID, "unknown option '%s'", key);
    *value = opt((SpmmOpt)i);
    return ATT_OK;
}

extern "C" int att_spmm_item_features(int64_t F, int64_t n_parts) { return item_features(F, n_parts); }

extern "C" size_t att_spmm_groups_scratch_bytes(int64_t n_parts, int64_t n_windows) {
    if (n_parts < 0) n_parts = 0;
    if (n_windows < 0) n_windows = 0;
    const int64_t m = n_parts > n_windows ? n_parts : n_windows;
    return align_up((size_t)n_parts * 8, 256) + align_up((size_t)n_windows * 8, 256) +
           scan64_tmp_bytes(m);
}

extern "C" int att_spmm_groups(const int32_t *window_of_part, int64_t n_parts, int64_t n_windows,
                               int group_parts, int32_t *group_part, int32_t *group_slot,
                               int32_t *red_first, int32_t *empty_win, int64_t *counts,
                               void *scratch, size_t scratch_bytes, void *stream) {
    clear_error();
    ATT_CHECK(n_parts >= 0 && n_parts < kFieldMask, ATT_ERR_UNSUPPORTED,
              "att_spmm_groups takes fewer than %lld parts", (long long)kFieldMask);
    ATT_CHECK(n_windows >= 0 && n_windows <= INT32_MAX, ATT_ERR_INVALID, "bad window count");
    ATT_CHECK(group_parts >= 1 && group_parts <= 1024, ATT_ERR_INVALID,
              "group_parts %d outside [1, 1024]", group_parts);
    ATT_CHECK(group_part && red_first && counts, ATT_ERR_INVALID, "null output");
    ATT_CHECK(n_parts == 0 || (window_of_part && group_slot), ATT_ERR_INVALID, "null input");
    ATT_CHECK(n_windows == 0 || empty_win, ATT_ERR_INVALID, "null empty-window output");
    ATT_CHECK(scratch && scratch_bytes >= att_spmm_groups_scratch_bytes(n_parts, n_windows),
              ATT_ERR_WORKSPACE, "scratch of %zu bytes, %zu needed", scratch_bytes,
              att_spmm_groups_scratch_bytes(n_parts, n_windows));
    cudaStream_t st = (cudaStream_t)stream;
    int64_t *pflags = (int64_t *)scratch;
    int64_t *wflags = (int64_t *)((char *)scratch + align_up((size_t)n_parts * 8, 256));
    int64_t *tmp = (int64_t *)((char *)wflags + align_up((size_t)n_windows * 8, 256));
    const unsigned pblocks = (unsigned)((n_parts + 255) / 256);
    const unsigned wblocks = (unsigned)((n_windows + 255) / 256);
    int s;
    if (n_parts > 0) {
        k_group_flags<<<pblocks, 256, 0, st>>>(window_of_part, n_parts, group_parts, pflags);
        if ((s = launch_status("k_group_flags")) != ATT_OK) return s;
        if ((s = scan64_exclusive(pflags, n_parts, tmp, st)) != ATT_OK) return s;
    }
    k_group_scatter<<<pblocks > 0 ? pblocks : 1, 256, 0, st>>>(window_of_part, n_parts, group_parts,
                                                               pflags, group_part, group_slot,
                                                               red_first, counts);
    if ((s = launch_status("k_group_scatter")) != ATT_OK) return s;
    if (n_windows > 0) {
        k_empty_flags<<<wblocks, 256, 0, st>>>(window_of_part, n_parts, n_windows, wflags);
        if ((s = launch_status("k_empty_flags")) != ATT_OK) return s;
        if ((s = scan64_exclusive(wflags, n_windows, tmp, st)) != ATT_OK) return s;
    }
    k_empty_scatter<<<wblocks > 0 ? wblocks : 1, 256, 0, st>>>(window_of_part, n_parts, n_windows,
                                                               wflags, empty_win, counts);
    return launch_status("k_empty_scatter");
}

extern "C" int att_host_device_pointer(const void *host, void **device) {
    clear_error();
    ATT_CHECK(host && device, ATT_ERR_INVALID, "null pointer");
    cudaPointerAttributes a;
    ATT_CUDA(cudaPointerGetAttributes(&a, host), "cudaPointerGetAttributes");
    ATT_CHECK(a.type == cudaMemoryTypeHost && a.devicePointer != nullptr, ATT_ERR_INVALID,
              "%p is not page-locked host memory mapped for the device", host);
    *device = a.devicePointer;
    return ATT_OK;
}

extern "C" size_t att_spmm_batched_grid(void) {
    if (dynamic_smem<k_spmm16_batched>(CfgBatch::SMEM) != ATT_OK) return 0;
    return (size_t)sm_count();
}

extern "C" int att_spmm_batched(const att_spmm_job *jobs, int64_t *header, int64_t grid,
                                int window, int wide, int32_t *err_flag, void *stream) {
    clear_error();
    ATT_CHECK(window == 8 && wide == 8, ATT_ERR_UNSUPPORTED,
              "the batched SpMM takes the (8-row, 8-wide) fp16 format");
    ATT_CHECK(jobs && header && grid > 0, ATT_ERR_INVALID, "null table or empty grid");
    const int prep = dynamic_smem<k_spmm16_batched>(CfgBatch::SMEM);
    if (prep != ATT_OK) return prep;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned side = (unsigned)(sm_count() * 8);
    k_zero_empty_batched<8><<<side, 256, 0, st>>>(jobs, header);
    int s = launch_status("k_zero_empty_batched");
    if (s != ATT_OK) return s;
    k_spmm16_batched<<<(unsigned)grid, CfgBatch::NW * 32, CfgBatch::SMEM, st>>>(jobs, header, err_flag);
    s = launch_status("k_spmm16_batched");
    if (s != ATT_OK) return s;
    k_reduce_groups_batched<8><<<(unsigned)(sm_count() * 4), 256, 0, st>>>(jobs, header);
    return launch_status("k_reduce_groups_batched");
}
