// spmm_stream.cuh -- the gather pipeline of the blocked SpMM kernels: a warp's
// stream of condensed-column chunks, copied global -> shared ahead of the
// products.  Included by spmm.cu.
//
// These kernels are bound by the latency of the gathers and by instruction
// issue (by DRAM traffic on graphs whose X is far larger than L2), so the
// stream works in chunks of 32 condensed columns with one set of waits, ids,
// value copies and branches per chunk, and three cursors that run one chunk
// apart across part boundaries:
//   fetch    the chunk whose column ids are in flight (one per lane), with the
//            next part's rowptr, window and split flag behind it
//   copy     the chunk whose rows are being copied: ids (-1 where there is
//            none) pass through shared memory, from which the lanes that copy
//            rows RPL g .. RPL g + RPL - 1 of a 16-row half read theirs with
//            one vector load
//   multiply the chunk whose copies have landed
// A half is 16 gathered rows with their 16-byte pieces XOR-swizzled by row
// (copies and fragment loads free of bank conflicts); rows and halves keep
// their source's alignment to 32 bytes (a padded pitch instead of the swizzle
// made the copies 1.5x slower) and halves start on multiples of 128 bytes (not
// of 256), so a swizzled address is one register and one XOR with a constant
// below 128.  The cursors
// hold warp-uniform values, so their branches need no convergence barriers.
//
// 500,000 nodes, mean degree 25, 64 fp16 features, L2-resident X (64 MB):
// 159 us, 11.8 TB/s into the SMs, at the 10.6-12.5 TB/s that random 128-byte
// reads of 64 MB reach; the ring with a cursor per 16-column step before it
// took 212 us (135 M instructions instead of 100 M, and every step waited for
// ids loaded one step ahead).  Loading the rows straight into MMA fragments
// (no shared memory) took 291 us: the fragments' lane order reads four rows
// per quarter warp, a four-way conflict in the L1 data array.
#pragma once

namespace att {
namespace {

// A value that is the same in every lane, handed to the compiler as such.
__device__ __forceinline__ int warp_uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

__device__ __forceinline__ void red_add_f32x4(float *p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}
__device__ __forceinline__ void red_add_f32x2(float *p, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(p), "f"(a), "f"(b) : "memory");
}

// Adjacent floats of an output row: stored (streaming: Y is written once, L2
// is left to the X rows) or, for a part of a split window, added.  `vec`: the
// row's floats are aligned for one vector access.
__device__ __forceinline__ void put4(float *dst, bool add, bool vec, float a, float b, float c, float d) {
    if (vec) {
        if (add) red_add_f32x4(dst, a, b, c, d);
        else __stcs(reinterpret_cast<float4 *>(dst), make_float4(a, b, c, d));
    } else if (add) {
        red_add_f32(dst, a);
        red_add_f32(dst + 1, b);
        red_add_f32(dst + 2, c);
        red_add_f32(dst + 3, d);
    } else {
        dst[0] = a;
        dst[1] = b;
        dst[2] = c;
        dst[3] = d;
    }
}
__device__ __forceinline__ void put2(float *dst, bool add, bool vec, float a, float b) {
    if (vec) {
        if (add) red_add_f32x2(dst, a, b);
        else __stcs(reinterpret_cast<float2 *>(dst), make_float2(a, b));
    } else if (add) {
        red_add_f32(dst, a);
        red_add_f32(dst + 1, b);
    } else {
        dst[0] = a;
        dst[1] = b;
    }
}

// What the last chunk of a part does with its tile: stores it in the rows of its
// window, adds it to them (split windows), or stores it in the part's own rows of
// the tiles, which are added in part order later.  A window of two parts needs no
// tiles: 0 + a + b is the same in either order.
enum : int { kStore = 0, kAdd = 1, kTile = 2 };
struct Target {
    float *base;
    int64_t row0, limit, ld;
    bool add;
};
// a Chunk's win holds its window (or part) as 30 unsigned bits: an id of 2^29 and
// more lies past the output, not before it
__device__ __forceinline__ int64_t window_of(int win) { return (uint32_t)win >> 2; }
__device__ __forceinline__ Target target(int win, int W, float *Y, int64_t m_out, int64_t ldy, float *tiles, int64_t F) {
    const int64_t row0 = window_of(win) * W;
    if ((win & 3) == kTile) return {tiles, row0, INT64_MAX, F, false};
    return {Y, row0, m_out, ldy, (win & 3) == kAdd};
}

// RPL column ids from shared memory
template <int RPL>
__device__ __forceinline__ void lds_ids(int (&id)[RPL], uint32_t p) {
    if constexpr (RPL == 2) {
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(id[0]), "=r"(id[1]) : "r"(p) : "memory");
    } else {
#pragma unroll
        for (int k = 0; k < RPL; k += 4)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                         : "=r"(id[k]), "=r"(id[k + 1]), "=r"(id[k + 2]), "=r"(id[k + 3])
                         : "r"(p + 4 * k)
                         : "memory");
    }
}

// Shared memory of a warp: S chunk buffers (two halves of 16 rows of XROW
// bytes, the chunk's 32 x W values of VSZ bytes, EXTRA bytes), then the
// current chunk's ids.
// One CTA per SM of NW warps (as many as shared memory holds, MAXW at most, which
// bounds the registers); its warps take the CTA's items from a counter in shared
// memory: parts differ in length up to 16 times, and with a fixed share per
// warp the last warps ran 15 % longer than the mean one.
template <int XROW_, int VSZ_, int W_, int WIDE_, int S_, int MAXW, int EXTRA_ = 0>
struct StreamCfg {
    static constexpr int XROW = XROW_, VSZ = VSZ_, W = W_, WIDE = WIDE_, S = S_, EXTRA = EXTRA_;
    static constexpr int HALF = 16 * XROW;
    static constexpr int VAL = 2 * HALF;
    static constexpr int EXT = VAL + 32 * W * VSZ;
    static constexpr int BUF = EXT + EXTRA;
    static constexpr int IDS = S * BUF;
    static constexpr int WARP_SMEM = IDS + 128;
    static constexpr int FIT = (227 * 1024 - 16) / WARP_SMEM;
    static constexpr int NW = (FIT < MAXW ? FIT : MAXW) / 4 * 4;  // as many on each of the four schedulers
    static constexpr int SMEM = NW * WARP_SMEM;
    static constexpr int CPR = XROW / 16;               // 16-byte pieces (copying lanes) per row
    static constexpr int RPL = CPR / 2;                 // rows per copying lane and half
    static constexpr int VP = 2 * W * VSZ / 32;         // 16-byte value pieces per lane and chunk
};

// One chunk of a work item (part, feature chunk)
struct Chunk {
    int start, left;  // first condensed column, real columns left in the part (0: an empty part)
    int fc;           // feature chunk, -1: no more items
    int win;          // window * 4 + kStore / kAdd, or part * 4 + kTile
};

struct StreamArgs {
    const int32_t *rowptr, *col, *win, *atomic;
    const void *val, *X;
    const float *xscale;  // EXTRA: per-row scales
    int64_t n_parts, n_x, F, ldx;
    int n_chunks;
    int wait;      // every row was zeroed: no store before that is done
    float *tiles;  // null, or [n_parts][W][F]: where parts of split windows are stored
    int32_t *err;
};

// IT: type of items and of X's row pitch in bytes -- int32_t when they fit
// (the common case), else int64_t.  ESZ: bytes per feature; FC: features per
// item; FULL: F is a multiple of FC; TILES: parts of split windows may go to tiles
// (only where the kernel asks for it: in the e4m3 kernel the choice cost 9 %).
template <typename C, int ESZ, int FC, typename IT, bool FULL, bool TILES = false>
struct Stream {
    static_assert(FC * ESZ == C::XROW, "rows");
    const StreamArgs &A;
    const int lane;
    const uint32_t sbase;
    int *const queue;              // the CTA's next item (in items of its own)
    const unsigned n_x;
    const IT n_parts, n_chunks, row_bytes, F;
    uint32_t xdst, idsrc;
    int ch;
    // fetch cursor
    IT i_part;                     // next item to enter
    int i_fc;
    int i_after;                   // lane 0: the CTA's item after that, in flight
    Chunk f;
    int fid;                       // the fetched chunk's ids, in flight
    int n_rp[3], n_win, n_atomic;  // of the next item, in flight until it is entered
    int n_near;                    // with tiles: lane k < 5 the window of part k - 2 of it
    // copy cursor
    Chunk p;
    int pid;                       // the lane's id of the chunk (EXTRA)
    bool p_whole;                  // no padding among its ids
    // chunks between the copy and the multiply cursor, oldest first
    Chunk pend[C::S - 1];
    uint32_t wbuf, rbuf;

    __device__ __forceinline__ Stream(const StreamArgs &A_, int lane_, int warp, uint32_t sbase_, int *queue_)
        : A(A_), lane(lane_), sbase(sbase_), queue(queue_), n_x(A_.n_x > INT32_MAX ? 1u << 31 : (unsigned)A_.n_x),
          n_parts((IT)A_.n_parts), n_chunks((IT)A_.n_chunks), row_bytes((IT)(A_.ldx * ESZ)), F((IT)A_.F) {
        const int rg = lane / C::CPR;
        ch = lane % C::CPR;
        xdst = sbase + rg * C::RPL * C::XROW + ((ch ^ swz<C::XROW>(rg * C::RPL)) << 4);
        idsrc = sbase + C::IDS + rg * C::RPL * 4;
        if (threadIdx.x == 0) *queue = C::NW;
        __syncthreads();
        set_item(warp);
        draw();
        fid = pid = -1;
        load_item();
        enter();
        wbuf = rbuf = 0;
#pragma unroll
        for (int s = 0; s < C::S - 1; ++s) {
            take();
            copy();
            pend[s] = p;
            wbuf += C::BUF;
            __syncwarp();  // the copied chunk's ids have been read
        }
        take();
    }
    __device__ __forceinline__ void set_item(int k) {  // the CTA's k-th item
        const IT item = (IT)k * (IT)gridDim.x + (IT)blockIdx.x;
        i_part = n_chunks == 1 ? item : item / n_chunks;
        i_fc = (int)(item - i_part * n_chunks);
    }
    __device__ __forceinline__ void draw() {
        if (lane == 0) i_after = atomicAdd(queue, 1);
    }
    __device__ __forceinline__ void load_item() {
        n_rp[0] = n_rp[1] = n_rp[2] = n_win = n_atomic = 0;
        if constexpr (TILES) n_near = -1;
        if (i_part < n_parts) {
#pragma unroll
            for (int k = 0; k < 3; ++k) n_rp[k] = __ldg(A.rowptr + 2 * (int64_t)i_part + k);
            n_win = __ldg(A.win + i_part);
            n_atomic = __ldg(A.atomic + i_part);
            if constexpr (TILES) {
                const int64_t near = (int64_t)i_part + lane - 2;
                if (A.tiles && lane < 5 && near >= 0 && near < A.n_parts) n_near = __ldg(A.win + near);
            }
        }
    }
    __device__ __forceinline__ void fetch_ids() { fid = lane < f.left ? __ldg(A.col + f.start + lane) : -1; }
    // f = the first chunk of the next item, which moves on
    __device__ __forceinline__ void enter() {
        const PartInfo pi = part_check<C::WIDE>(n_rp[0], n_rp[1], n_rp[2], A.err);
        f.start = warp_uniform(pi.start);
        f.left = warp_uniform(pi.nreal);
        f.win = (int)(4u * (uint32_t)n_win + (n_atomic != 0 ? kAdd : kStore));
        if (TILES && A.tiles) {  // three parts of one window in a row, this one among them
            const unsigned b = __ballot_sync(0xffffffffu, n_near == n_win);
            if (n_atomic != 0 && ((b & b >> 1 & b >> 2) & 7) != 0) f.win = (int)(4u * (uint32_t)i_part + kTile);
        }
        f.win = warp_uniform(f.win);
        f.fc = i_part < n_parts ? i_fc : -1;
        set_item(warp_uniform(i_after));
        draw();
        load_item();
        fetch_ids();
    }
    // the fetched chunk's ids go to shared memory and it becomes the copy
    // cursor's; the fetch cursor moves on
    __device__ __forceinline__ void take() {
        p = f;
        if (p.fc < 0) return;
        int c = fid;  // valid ids are -1 (padding) .. n_x - 1
        const bool none = (unsigned)c >= n_x;
        if (none && c != -1) {
            if (A.err) atomicOr(A.err, 1);
            c = -1;
        }
        p_whole = !__any_sync(0xffffffffu, none);
        if constexpr (C::EXTRA > 0) pid = c;
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
    __device__ __forceinline__ void copy_half(uint32_t dst, uint32_t ids, const char *Xl) {
        // row k's pieces are swizzled by k more than the first row's
        auto at = [&](int k) { return (dst ^ (swz<C::XROW>(k) << 4)) + k * C::XROW; };
        int id[C::RPL];
        lds_ids<C::RPL>(id, ids);
        if (p_whole) {
#pragma unroll
            for (int k = 0; k < C::RPL; ++k) cp_async16(at(k), Xl + (int64_t)id[k] * row_bytes, 16);
        } else {
#pragma unroll
            for (int k = 0; k < C::RPL; ++k) {
                const bool ok = id[k] >= 0;
                cp_async16(at(k), Xl + (ok ? (int64_t)id[k] * row_bytes : 0), ok ? 16 : 0);
            }
        }
    }
    // the copy cursor's chunk into buffer wbuf, as one cp.async group
    __device__ __forceinline__ void copy() {
        if (p.fc >= 0 && p.left > 0) {
            const IT fe = (IT)p.fc * FC + ch * (16 / ESZ);
            const char *Xl = reinterpret_cast<const char *>(A.X) + (int64_t)fe * ESZ;
            if (FULL || fe < F) {  // pieces past F stay as they are (their products are never stored)
                copy_half(xdst + wbuf, idsrc, Xl);
                if (p.left > 16) copy_half(xdst + wbuf + C::HALF, idsrc + 64, Xl);
            }
            const char *src = reinterpret_cast<const char *>(A.val) + ((int64_t)p.start * (C::W * C::VSZ) + lane * 16);
#pragma unroll
            for (int i = 0; i < C::VP; ++i) {
                // columns before the block that the lane's piece sits in; a
                // block past the part's real columns is zeros
                constexpr int PPB = C::W * C::WIDE * C::VSZ / 16;  // pieces per block
                const bool ok = (i * 32 + lane) / PPB * C::WIDE < p.left;
                cp_async16(sbase + C::VAL + wbuf + (i * 32 + lane) * 16, ok ? (const void *)(src + i * 512) : A.val,
                           ok ? 16 : 0);
            }
            if constexpr (C::EXTRA > 0) {
                const bool ok = pid >= 0;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sbase + C::EXT + wbuf + 4 * lane),
                             "l"(ok ? A.xscale + pid : A.xscale), "r"(ok ? 4 : 0));
            }
        }
        cp_async_commit();
    }
    __device__ __forceinline__ bool more() const { return pend[0].fc >= 0; }
    // Copies the next chunk and waits for the oldest one, whose buffer is at
    // rbuf; call release() once it has been read.
    __device__ __forceinline__ Chunk next() {
        const Chunk c = pend[0];
        copy();
#pragma unroll
        for (int s = 0; s < C::S - 2; ++s) pend[s] = pend[s + 1];
        pend[C::S - 2] = p;
        __syncwarp();  // the copied chunk's ids have been read
        take();
        wbuf = wbuf == (C::S - 1) * C::BUF ? 0 : wbuf + C::BUF;
        cp_async_wait<C::S - 1>();
        __syncwarp();
        return c;
    }
    __device__ __forceinline__ void release() {
        __syncwarp();
        rbuf = rbuf == (C::S - 1) * C::BUF ? 0 : rbuf + C::BUF;
    }
};

}  // namespace
}  // namespace att
