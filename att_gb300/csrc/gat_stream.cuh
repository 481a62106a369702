// gat_stream.cuh -- the gather pipeline of the fused GAT kernels: the chunk
// stream of the SpMM kernels (spmm_stream.cuh: 32 condensed columns at a time,
// three cursors a chunk apart, one CTA per SM whose warps draw their items from
// a counter) over work items (run of parts of one window, head), with the
// occupancy bits of the chunk's slots and a per-column scalar beside the rows.
// Included by gat_fused.cu.
//
// The kernels are bound by issue and latency (X' fits L2): the ring with a
// cursor per 16-column step that this replaces spent half of its instructions
// on the cursor and waited every step for ids loaded one step ahead.
#pragma once

namespace att {
namespace {

__device__ __forceinline__ int warp_uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

// XOR swizzle of 16-byte pieces by row, for rows of ROW_BYTES bytes
template <int ROW_BYTES>
__device__ __forceinline__ int swz_rb(int r) {
    if constexpr (ROW_BYTES >= 128) return r & 7;
    else return (r >> 1) & 3;
}

// A warp's shared memory: S chunk buffers (32 rows of XROW bytes, 32 bytes of
// occupancy bits in 128, 32 scalars if SCALAR), the copied chunk's ids, TAIL bytes
// of the kernel's own.
template <int XROW_, bool SCALAR_, int TAIL_, int S_, int MAXW>
struct GStreamCfg {
    static constexpr int XROW = XROW_;
    static constexpr bool SCALAR = SCALAR_;
    static constexpr int S = S_;
    static constexpr int HALF = 16 * XROW;
    static constexpr int MASK = 2 * HALF;
    static constexpr int SC = MASK + 128;
    static constexpr int BUF = SC + (SCALAR ? 128 : 0);
    static constexpr int IDS = S * BUF;
    static constexpr int TAIL = IDS + 128;
    static constexpr int WARP_SMEM = (TAIL + TAIL_ + 127) / 128 * 128;
    static constexpr int FIT = (227 * 1024 - 16) / WARP_SMEM;
    static constexpr int NW = (FIT < MAXW ? FIT : MAXW) / 4 * 4;  // as many on each of the four schedulers
    static constexpr int SMEM = NW * WARP_SMEM;
    static constexpr int CPR = XROW / 16;
    static constexpr int RPL = CPR / 2;  // rows per copying lane and half
    static_assert(CPR >= 4 && CPR <= 32, "row of 64 to 512 bytes");
};

struct GStreamArgs {
    const int32_t *rowptr, *col, *win;
    const uint32_t *mask;
    const int32_t *run_begin;  // [n_runs + 1] part ranges
    const int32_t *run_slot;   // [n_runs]
    int64_t n_runs, H, n_nodes, F;
    int wide;
    const void *X;             // gathered rows: id's of head h at X + id * ld + h * F
    int64_t ld;
    const float *sc;           // per-column scalars [H][n_nodes] (SCALAR)
    int32_t *err;
};

struct GChunk {
    int start, left;  // first condensed column, real columns left in the run
    int h;            // head, -1: no more items
    int win;          // window, -1: an empty run (nothing to write)
    int slot;         // run_slot, or kGoesOn: more of the run follows its last chunk
};
constexpr int kGoesOn = -2;

// IT: index type of items and element offsets (int32_t when every offset fits)
template <typename C, typename T, typename IT>
struct GatStream {
    const GStreamArgs &A;
    const int lane;
    const uint32_t sbase;
    int *const queue;
    const int n_items, H;
    const unsigned n_x;
    const IT ld;
    uint32_t xdst, idsrc;
    int ch;
    // items: drawn -> part range in flight -> rowptr in flight -> entered
    int d_after;                   // lane 0: drawn, in flight
    int r_item, r_p0, r_p1, r_slot;
    int e_item, e_p0, e_p1, e_slot, e_start, e_end, e_pend, e_win;
    GChunk f, p;
    GChunk pend[C::S - 1];         // between the copy and the multiply cursor, oldest first
    int fid, pid, f_pend, p_pend;  // ids of the fetched / copied chunk; padded columns left
    bool p_whole, e_near;
    uint32_t wbuf, rbuf;

    __device__ __forceinline__ GatStream(const GStreamArgs &A_, int lane_, int warp, uint32_t sbase_, int *queue_)
        : A(A_), lane(lane_), sbase(sbase_), queue(queue_), n_items((int)(A_.n_runs * A_.H)), H((int)A_.H),
          n_x(A_.n_nodes > INT32_MAX ? 1u << 31 : (unsigned)A_.n_nodes), ld((IT)A_.ld) {
        const int rg = lane / C::CPR;
        ch = lane % C::CPR;
        xdst = sbase + rg * C::RPL * C::XROW + ((ch ^ swz_rb<C::XROW>(rg * C::RPL)) << 4);
        idsrc = sbase + C::IDS + rg * C::RPL * 4;
        if (threadIdx.x == 0) *queue = C::NW;
        __syncthreads();
        range((int)blockIdx.x + warp * (int)gridDim.x);
        draw();
        rows();
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
    __device__ __forceinline__ void draw() {
        if (lane == 0) d_after = (int)blockIdx.x + atomicAdd(queue, 1) * (int)gridDim.x;
    }
    // item's part range
    __device__ __forceinline__ void range(int item) {
        r_item = item;
        r_p0 = r_p1 = 0;
        r_slot = -1;
        if (item < n_items) {
            const int run = H == 1 ? item : item / H;
            r_p0 = __ldg(A.run_begin + run);
            r_p1 = __ldg(A.run_begin + run + 1);
            r_slot = __ldg(A.run_slot + run);
        }
    }
    struct Part {
        int start, end, pend;
        bool good;  // starts and ends on a block boundary
    };
    __device__ __forceinline__ Part part(int k) const {
        const int s = __ldg(A.rowptr + 2 * (int64_t)k), e = __ldg(A.rowptr + 2 * (int64_t)k + 1),
                  q = __ldg(A.rowptr + 2 * (int64_t)k + 2);
        return {s, e, q, (s & (A.wide - 1)) == 0 && (q & (A.wide - 1)) == 0 && q >= e};
    }
    // its rowptr; the next drawn item's range
    __device__ __forceinline__ void rows() {
        e_item = r_item;
        e_p0 = r_p0;
        e_p1 = r_p1;
        e_slot = r_slot;
        e_start = e_end = e_pend = 0;
        e_win = -1;
        if (e_p1 > e_p0) {
            e_start = __ldg(A.rowptr + 2 * (int64_t)e_p0);
            e_end = __ldg(A.rowptr + 2 * (int64_t)e_p1 - 1);
            e_pend = __ldg(A.rowptr + 2 * (int64_t)e_p1);
            e_win = __ldg(A.win + e_p0);
            // every part of the run starts and ends on a block boundary
            for (int k = e_p0 + lane; k < e_p1; k += 32)
                if (!part(k).good) e_end = INT32_MIN;
        }
        e_near = false;
        const int nxt = warp_uniform(d_after);
        draw();
        range(nxt);
    }
    // ids and occupancy bits of the next run's first 1024 columns into L2 (they
    // stream from DRAM, whose latency is about a chunk's time)
    __device__ __forceinline__ void near() {
        e_near = true;
        if (e_start + 32 * lane < e_end)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(A.col + e_start + 32 * lane));
        if (lane < 8 && e_start + 128 * lane < e_end)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(reinterpret_cast<const char *>(A.mask) + e_start + 128 * lane));
    }
    __device__ __forceinline__ void fetch_ids() { fid = lane < f.left ? __ldg(A.col + f.start + lane) : -1; }
    __device__ __forceinline__ void enter() {
        f.start = warp_uniform(e_start);
        f.left = warp_uniform(e_end <= e_start ? 0 : e_end - e_start);
        f_pend = warp_uniform(e_pend - e_start);
        f.win = warp_uniform(e_win);
        f.slot = warp_uniform(e_slot);
        const int item = warp_uniform(e_item);
        f.h = item < n_items ? (H == 1 ? 0 : item - item / H * H) : -1;
        // a run with a misaligned part among its parts goes one good part at a time
        if (__any_sync(0xffffffffu, e_end == INT32_MIN)) good_part();
        if (f.slot != kGoesOn) rows();
        fetch_ids();
    }
    // The next good part of the run; the run's other ones, if any, by later calls.
    __device__ __forceinline__ void good_part() {
        if (A.err) atomicOr(A.err, 2);
        f.left = f_pend = 0;
        for (int k = e_p0; k < e_p1; ++k) {
            const Part t = part(k);
            if (!t.good || t.end <= t.start) continue;
            if (f.left > 0) {
                e_p0 = k;
                f.slot = kGoesOn;
                break;
            }
            f.start = warp_uniform(t.start);
            f.left = warp_uniform(t.end - t.start);
            f_pend = warp_uniform(t.pend - t.start);
        }
    }
    __device__ __forceinline__ void take() {
        p = f;
        p_pend = f_pend;
        if (p.h < 0) return;
        int c = fid;  // valid ids are -1 (padding) .. n_nodes - 1
        const bool none = (unsigned)c >= n_x;
        if (none && c != -1) {
            if (A.err) atomicOr(A.err, 1);
            c = -1;
        }
        p_whole = !__any_sync(0xffffffffu, none);
        pid = c;
        asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(sbase + C::IDS + 4 * lane), "r"(c) : "memory");
        if (f.left > 32) {
            f.start += 32;
            f.left -= 32;
            f_pend -= 32;
            fetch_ids();
            if (!e_near) near();
        } else {
            enter();
        }
        __syncwarp();
    }
    // `whole`: no padding among the chunk's ids; else an id of -1 copies zeros
    template <bool WHOLE>
    __device__ __forceinline__ void copy_half(uint32_t dst, uint32_t ids, IT base) {
        auto at = [&](int k) { return (dst ^ (swz_rb<C::XROW>(k) << 4)) + k * C::XROW; };
#pragma unroll
        for (int k0 = 0; k0 < C::RPL; k0 += 4) {
            int id[4] = {0, 0, 0, 0};
            if constexpr (C::RPL == 2)
                asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(id[0]), "=r"(id[1]) : "r"(ids) : "memory");
            else
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                             : "=r"(id[0]), "=r"(id[1]), "=r"(id[2]), "=r"(id[3])
                             : "r"(ids + 4 * k0)
                             : "memory");
#pragma unroll
            for (int k = 0; k < (C::RPL < 4 ? C::RPL : 4); ++k) {
                const bool ok = WHOLE || id[k] >= 0;
                const IT o = ok ? base + (IT)id[k] * ld : (IT)0;
                cp_async16(at(k0 + k), (const T *)A.X + o, ok ? 16 : 0);
            }
        }
    }
    // the copy cursor's chunk into buffer wbuf, as one cp.async group
    __device__ __forceinline__ void copy() {
        if (p.h >= 0 && p.left > 0) {
            const IT base = (IT)p.h * (IT)A.F + ch * (16 / (int)sizeof(T));
            if (p_whole) {
                copy_half<true>(xdst + wbuf, idsrc, base);
                copy_half<true>(xdst + wbuf + C::HALF, idsrc + 64, base);
            } else {
                copy_half<false>(xdst + wbuf, idsrc, base);
                if (p.left > 16) copy_half<false>(xdst + wbuf + C::HALF, idsrc + 64, base);
            }
            // a byte of occupancy bits per column, 4 columns a piece; zeros
            // past the run's padded end
            if (lane < 8) {
                const bool ok = 4 * lane < p_pend;
                const char *m = reinterpret_cast<const char *>(A.mask) + (int64_t)p.start + 4 * lane;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sbase + C::MASK + wbuf + 4 * lane),
                             "l"(ok ? m : reinterpret_cast<const char *>(A.mask)), "r"(ok ? 4 : 0));
            }
            if constexpr (C::SCALAR) {
                const bool ok = pid >= 0;
                const IT o = (IT)p.h * (IT)A.n_nodes + (ok ? pid : 0);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sbase + C::SC + wbuf + 4 * lane),
                             "l"(A.sc + o), "r"(ok ? 4 : 0));
            }
        }
        cp_async_commit();
    }
    __device__ __forceinline__ bool more() const { return pend[0].h >= 0; }
    // Copies the next chunk and waits for the oldest, whose buffer is at rbuf;
    // call release() once it has been read.
    __device__ __forceinline__ GChunk next() {
        const GChunk c = pend[0];
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
