// gat_fused.cu -- one-pass GAT attention layer on the row-window block format.
//
// Replaces the reference's chain of separate ops for a GAT layer
// (end2end_ori/gat_final/mgat_csr/mgat_conv.py:173-198: att/SDDMM ->
// LeakyReLU -> exp -> row sums -> SpMM -> divide, each a kernel with an
// nnz-sized intermediate) by one kernel that never materialises per-edge
// values.  Per 8-row window and 16 condensed columns at a time:
//
//   logits  mode 0 (dot):      S[c][r] = X'_c . X'_r  -- mma.sync m16n8k16, K = F
//           mode 1 (additive): S[c][r] = s0[r] + s1[c] -- GAT's a0/a1 scores
//   e = LeakyReLU(S) on occupied slots (per-slot bitmap), -inf elsewhere
//   online softmax: running row max m and sum l in fp32 registers, reduced
//     across the 8 lanes of a row with shuffles; the accumulator is rescaled
//     by exp(m_old - m_new) whenever the max grows
//   P = exp(e - m) -> fp16/bf16, transposed in registers (movmatrix) into the
//     B operand of acc[f][r] += X'^T[f][c] . P[c][r]  -- mma.sync m16n8k16
//
// X' rows are gathered once, 32 columns at a time (gat_stream.cuh), and feed both
// products.
// A work item is a chunk of up to `parts_per_chunk` consecutive parts of one
// window; a window covered by one chunk is finalised in place (out = acc/l,
// plus the row max and sum for the backward pass); a window spread over
// several chunks writes (m, l, acc) partials that k_gat_combine merges.
#include "att_common.cuh"

#include <type_traits>

namespace att {
namespace {

constexpr int kGWarps = 4;
constexpr int kGThreads = kGWarps * 32;
constexpr int kW = 8;  // window rows

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(y) : "r"(x));
    return y;
}

template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t v);
template <>
__device__ __forceinline__ float2 unpack2<__half>(uint32_t v) {
    return __half22float2(*reinterpret_cast<__half2 *>(&v));
}
template <>
__device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t v) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&v));
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}

__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src),
                 "r"(src_bytes));
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src),
                 "r"(src_bytes));
}

template <int F>
__device__ __forceinline__ int swz_row(int r) {
    if constexpr (F * 2 >= 128) return r & 7;
    else return (r >> 1) & 3;
}

}  // namespace
}  // namespace att

#include "gat_stream.cuh"

namespace att {
namespace {

struct GatArgs {
    GStreamArgs S;                // rows: X'; scalar: s1 (mode 1)
    const float *s0;              // [H][n_nodes] row scores (mode 1)
    float slope;
    float *out;                   // [n_nodes, H*F] rows of ldo
    int64_t ldo;
    float *row_max, *row_sum;     // [H][n_nodes] or null
    float *partial;               // [n_partial][H][kW][F + 2]
};

// Warps per SM: 16 leave 128 registers a thread; fp32 X' is bounded by shared
// memory (12 at 64 features).
template <typename T, int F, int MODE>
struct GCfg : GStreamCfg<F * (int)sizeof(T), MODE == 1, sizeof(T) == 4 ? 32 * kW * 4 : 0, 2,
                         F == 128 ? 12 : 16> {
    static constexpr bool F32 = sizeof(T) == 4;  // fp32 X': 3xTF32 products
    static constexpr int MT = F / 16;
};

// PSPLIT: aggregate with P as a hi + lo pair of 16-bit values (fp32-accurate
// output); the training path needs it so that dout . out matches the
// backward's recomputed probabilities.
// IT: index type of element offsets (int32_t when every offset fits)
template <typename T, int F, int MODE, bool PSPLIT, typename IT>
__global__ void __launch_bounds__((GCfg<T, F, MODE>::NW * 32), 1) k_gat_fused(const __grid_constant__ GatArgs A) {
    using C = GCfg<T, F, MODE>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int queue;
    const int lane = threadIdx.x & 31, warp = warp_uniform(threadIdx.x >> 5);
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    const unsigned char *sgen = smem + warp * C::WARP_SMEM;
    const int gid = lane >> 2, tig = lane & 3;
    const IT H = (IT)A.S.H, n_nodes = (IT)A.S.n_nodes, ldx = (IT)A.S.ld, ldo = (IT)A.ldo;
    const T *X = (const T *)A.S.X;
    const float NEG_INF = -INFINITY;
    // logits may exceed a row's reference by this much before it moves
    constexpr float kLazy = 8.f;
    float *ptile = (float *)(smem + warp * C::WARP_SMEM + C::TAIL);  // fp32 only: the half's P, re-read transposed
    (void)ptile;

    // this lane's four (column, row) slots of a half (columns gid, gid + 8,
    // rows 2 tig, 2 tig + 1): word and bit of its occupancy
    const int wide = A.S.wide;
    uint32_t maddr[4], mbit[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int c = gid + 8 * (u >> 1), r = 2 * tig + (u & 1);
        const int bit = (c & ~(wide - 1)) * kW + r * wide + (c & (wide - 1));
        maddr[u] = sbase + C::MASK + (bit >> 5) * 4;
        mbit[u] = 1u << (bit & 31);
    }
    // ldmatrix lanes (matrix q = lane / 8, row lane % 8): rows as MMA rows
    // (logits) and, transposed, as MMA columns (aggregation)
    const int q = lane >> 3, rr = lane & 7;
    const int lrow = (q & 1) * 8 + rr, arow = (q >> 1) * 8 + rr;
    const uint32_t llane = sbase + lrow * C::XROW + (((q >> 1) ^ swz_rb<C::XROW>(lrow)) << 4);
    const uint32_t alane = sbase + arow * C::XROW + (((q & 1) ^ swz_rb<C::XROW>(arow)) << 4);
    // piece 2 j (+ 0 or 1, in the lane's address) of a row under the swizzle
    auto piece = [](uint32_t at, int j) { return (at ^ ((j & 3) << 5)) + (j >> 2) * 128; };

    // query side of the window: B fragments (mode 0; fp32: split) or row scores
    uint32_t bq[C::MT][2];
    uint32_t bqh[C::F32 ? F / 8 : 1][2], bql[C::F32 ? F / 8 : 1][2];
    float s0r[2] = {0.f, 0.f};
    float m_run[2], mref[2], l_run[2];
    float acc[C::MT][4];
    bool first = true;
    // slope 0 is left out: there 0 * -inf is a NaN, which fmaxf would drop
    const bool convex = A.slope > 0.f && A.slope <= 1.f;

    GatStream<C, T, IT> st(A.S, lane, warp, sbase, &queue);
    while (st.more()) {
        const GChunk c = st.next();
        const IT h = c.h, wrow = (IT)c.win * kW;
        if (first && c.win >= 0) {
            if constexpr (MODE == 0 && !C::F32) {
#pragma unroll
                for (int kk = 0; kk < C::MT; ++kk)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const IT row = wrow + gid;
                        const int f = 16 * kk + 2 * tig + 8 * u;
                        bq[kk][u] = row < n_nodes ? *(const uint32_t *)(X + (row * ldx + h * F + f)) : 0u;
                    }
            } else if constexpr (MODE == 0) {
#pragma unroll
                for (int kk = 0; kk < F / 8; ++kk)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const IT row = wrow + gid;
                        const int f = 8 * kk + tig + 4 * u;
                        split_tf32x3(row < n_nodes ? (float)X[row * ldx + h * F + f] : 0.f, bqh[kk][u], bql[kk][u]);
                    }
            } else {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const IT row = wrow + 2 * tig + u;
                    s0r[u] = row < n_nodes ? A.s0[h * n_nodes + row] : 0.f;
                }
            }
            m_run[0] = m_run[1] = NEG_INF;
            mref[0] = mref[1] = l_run[0] = l_run[1] = 0.f;
#pragma unroll
            for (int j = 0; j < C::MT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
        }
        if (c.left > 0) {
            // Both halves at once: twice the independent work per warp hides
            // the latency of the products and of the softmax chain (232,965
            // nodes, 114 M edges, fp16: 1,762 us with 16 warps an SM; half
            // after half with 20 warps 2,108, in the ring before the chunk
            // stream 2,551).  A second
            // half past the run's end has no occupied slot (its rows are
            // whatever the buffer held: nothing of it is used).
            float sv[2][4];
            if constexpr (MODE == 0 && !C::F32) {
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) sv[hf][0] = sv[hf][1] = sv[hf][2] = sv[hf][3] = 0.f;
#pragma unroll
                for (int kk = 0; kk < C::MT; ++kk)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint32_t a[4];
                        ldsm_x4(piece(llane + st.rbuf + hf * C::HALF, kk), a[0], a[1], a[2], a[3]);
                        mma_16816<T>(sv[hf], a, bq[kk][0], bq[kk][1]);
                    }
            } else if constexpr (MODE == 0) {
                // 8 features per k-step; ldmatrix of 16-byte rows hands each
                // lane the fp32 element (row gid, feature tig) of every 8 x 4
                // matrix: the m16n8k8 A fragment.  3xTF32: lo.hi + hi.lo and
                // hi.hi in two chains, added at the end
                float sl[2][4];
#pragma unroll
                for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                    for (int u = 0; u < 4; ++u) sv[hf][u] = sl[hf][u] = 0.f;
#pragma unroll
                for (int kk = 0; kk < F / 8; ++kk)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint32_t a[4], ah[4], al[4];
                        ldsm_x4(piece(llane + st.rbuf + hf * C::HALF, kk), a[0], a[1], a[2], a[3]);
#pragma unroll
                        for (int u = 0; u < 4; ++u) split_tf32x3(__uint_as_float(a[u]), ah[u], al[u]);
                        mma_1688_tf32(sl[hf], al[0], al[1], al[2], al[3], bqh[kk][0], bqh[kk][1]);
                        mma_1688_tf32(sv[hf], ah[0], ah[1], ah[2], ah[3], bqh[kk][0], bqh[kk][1]);
                        mma_1688_tf32(sl[hf], ah[0], ah[1], ah[2], ah[3], bql[kk][0], bql[kk][1]);
                    }
#pragma unroll
                for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                    for (int u = 0; u < 4; ++u) sv[hf][u] += sl[hf][u];
            } else {
                const float *s1s = (const float *)(sgen + st.rbuf + C::SC);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const float c_lo = s1s[16 * hf + gid], c_hi = s1s[16 * hf + gid + 8];
                    sv[hf][0] = s0r[0] + c_lo;
                    sv[hf][1] = s0r[1] + c_lo;
                    sv[hf][2] = s0r[0] + c_hi;
                    sv[hf][3] = s0r[1] + c_hi;
                }
            }
            // LeakyReLU on occupied slots, -inf on empty ones
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint32_t w;
                    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(w) : "r"(maddr[u] + st.rbuf + 16 * hf) : "memory");
                    const float x = sv[hf][u], y = A.slope * x;
                    // the same value as x > 0 ? x : y where 0 < slope <= 1
                    const float z = convex ? fmaxf(x, y) : x > 0.f ? x : y;
                    sv[hf][u] = (w & mbit[u]) ? z : NEG_INF;
                }
            // online softmax, rows 2tig (u even) and 2tig+1 (u odd), with
            // lazy rescaling: a row's reference m_run moves (max over the
            // row's lanes, accumulators and partial sums rescaled) only on
            // its first occupied slot or when a logit exceeds it by more
            // than kLazy, so most chunks run no reduction at all; the
            // probabilities stay below e^kLazy, well inside the 16-bit P
            // range.  Each lane sums its own columns' probabilities
            // (l_run holds that partial until the end of the item).
            auto over = [&](const float(&x)[4]) {
                return (x[0] > m_run[0] + kLazy) | (x[2] > m_run[0] + kLazy) | (x[1] > m_run[1] + kLazy) |
                       (x[3] > m_run[1] + kLazy);
            };
            auto move = [&](const float(&x)[4]) {
                float mx[2] = {fmaxf(x[0], x[2]), fmaxf(x[1], x[3])};
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], o));
                    mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], o));
                }
                float alpha[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float mn = fmaxf(m_run[u], mx[u]);
                    alpha[u] = mn == NEG_INF ? 1.f : __expf(m_run[u] - mn);
                    // rounded here: contracted with the addition of the half
                    // behind it, a row's sum would depend on which half of a
                    // chunk moves its reference
                    l_run[u] = __fmul_rn(l_run[u], alpha[u]);
                    m_run[u] = mn;
                    mref[u] = mn == NEG_INF ? 0.f : mn;
                }
#pragma unroll
                for (int j = 0; j < C::MT; ++j) {
                    acc[j][0] *= alpha[0];
                    acc[j][1] *= alpha[1];
                    acc[j][2] *= alpha[0];
                    acc[j][3] *= alpha[1];
                }
            };
            // probabilities of a half, in its logits' place
            auto probs = [&](float(&x)[4]) {
#pragma unroll
                for (int u = 0; u < 4; ++u) x[u] = __expf(x[u] - mref[u & 1]);
                l_run[0] += x[0] + x[2];
                l_run[1] += x[1] + x[3];
            };
            auto aggregate = [&](const float(&p)[4], int hf) {
                if constexpr (!C::F32) {
                    // P^T into B fragments: (col gid, rows 2tig..) -> (row gid, cols 2tig..)
                    const uint32_t h01 = pack2<T>(p[0], p[1]), h23 = pack2<T>(p[2], p[3]);
                    const uint32_t b0 = movmatrix_trans(h01);
                    const uint32_t b1 = movmatrix_trans(h23);
                    uint32_t bl0 = 0, bl1 = 0;
                    if constexpr (PSPLIT) {
                        const float2 r01 = unpack2<T>(h01), r23 = unpack2<T>(h23);
                        bl0 = movmatrix_trans(pack2<T>(p[0] - r01.x, p[1] - r01.y));
                        bl1 = movmatrix_trans(pack2<T>(p[2] - r23.x, p[3] - r23.y));
                    }
#pragma unroll
                    for (int j = 0; j < C::MT; ++j) {
                        uint32_t a[4];
                        ldsm_x4_trans(piece(alane + st.rbuf + hf * C::HALF, j), a[0], a[1], a[2], a[3]);
                        mma_16816<T>(acc[j], a, b0, b1);
                        if constexpr (PSPLIT) mma_16816<T>(acc[j], a, bl0, bl1);
                    }
                } else {
                    // P through shared memory: written as (col, row), read back as the
                    // m16n8k8 B fragment of each 8-column k-step: row gid, columns
                    // 2 tig (k = tig) and 2 tig + 1 (k = tig + 4), the order in which
                    // 16-byte loads of the X' rows are free of bank conflicts
                    float *pt = ptile + hf * 16 * kW;
#pragma unroll
                    for (int u = 0; u < 4; ++u) pt[(gid + 8 * (u >> 1)) * kW + 2 * tig + (u & 1)] = p[u];
                    __syncwarp();
                    const unsigned char *xt = sgen + st.rbuf + hf * C::HALF;
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {
                        uint32_t ph[2], pl[2];
                        split_tf32x3(pt[(8 * ks + 2 * tig) * kW + gid], ph[0], pl[0]);
                        split_tf32x3(pt[(8 * ks + 2 * tig + 1) * kW + gid], ph[1], pl[1]);
                        const unsigned char *x0 = xt + (8 * ks + 2 * tig) * C::XROW + ((gid ^ (2 * tig)) << 4);
                        const unsigned char *x1 = xt + (8 * ks + 2 * tig + 1) * C::XROW + ((gid ^ (2 * tig + 1)) << 4);
#pragma unroll
                        for (int u = 0; u < C::MT / 2; ++u) {
                            // four features of both columns: tile 2 u + v holds
                            // features 32 u + 4 gid + 2 v (m = gid) and + 1 (m = gid + 8)
                            const float4 r0 = *reinterpret_cast<const float4 *>(x0 + 128 * u);
                            const float4 r1 = *reinterpret_cast<const float4 *>(x1 + 128 * u);
                            const float x[2][4] = {{r0.x, r0.y, r1.x, r1.y}, {r0.z, r0.w, r1.z, r1.w}};
#pragma unroll
                            for (int v = 0; v < 2; ++v) {
                                uint32_t ah[4], al[4];
#pragma unroll
                                for (int k = 0; k < 4; ++k) split_tf32x3(x[v][k], ah[k], al[k]);
                                float(&d)[4] = acc[2 * u + v];
                                mma_1688_tf32(d, al[0], al[1], al[2], al[3], ph[0], ph[1]);
                                mma_1688_tf32(d, ah[0], ah[1], ah[2], ah[3], pl[0], pl[1]);
                                mma_1688_tf32(d, ah[0], ah[1], ah[2], ah[3], ph[0], ph[1]);
                            }
                        }
                    }
                    __syncwarp();  // P has been read
                }
            };
            // The references move half by half, as if one followed the other:
            // where the second half moves them again, the first is aggregated
            // before (16-bit probabilities are rounded against their half's own
            // reference; the fp32 ones need no such care).
            bool apart = false;
            if (__any_sync(0xffffffffu, over(sv[0]) | over(sv[1]))) {
                if (__any_sync(0xffffffffu, over(sv[0]))) move(sv[0]);
                apart = __any_sync(0xffffffffu, over(sv[1]));
                if (C::F32 && apart) move(sv[1]);
            }
            probs(sv[0]);
            if (!C::F32 && apart) {
                aggregate(sv[0], 0);
                move(sv[1]);
                probs(sv[1]);
            } else {
                probs(sv[1]);
                aggregate(sv[0], 0);
            }
            if (c.left > 16) aggregate(sv[1], 1);
        }
        st.release();
        first = c.left <= 32 && c.slot != kGoesOn;
        if (!first || c.win < 0) continue;
        // row sums: the lanes' partial sums over their own columns
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], o);
            l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], o);
        }
        // ---- epilogue: acc[j][u] = row 2 tig + (u & 1), feature ----
        auto feature = [&](int j, int u) {
            return C::F32 ? 32 * (j >> 1) + 4 * gid + 2 * (j & 1) + (u >> 1) : 16 * j + gid + 8 * (u >> 1);
        };
        if (c.slot < 0) {
            float inv[2] = {l_run[0] > 0.f ? 1.f / l_run[0] : 0.f, l_run[1] > 0.f ? 1.f / l_run[1] : 0.f};
#pragma unroll
            for (int j = 0; j < C::MT; ++j)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const IT row = wrow + 2 * tig + (u & 1);
                    if (row < n_nodes) A.out[row * ldo + h * F + feature(j, u)] = acc[j][u] * inv[u & 1];
                }
            if (gid == 0) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const IT row = wrow + 2 * tig + u;
                    if (row < n_nodes) {
                        if (A.row_max) A.row_max[h * n_nodes + row] = m_run[u];
                        if (A.row_sum) A.row_sum[h * n_nodes + row] = l_run[u];
                    }
                }
            }
        } else {
            float *pp = A.partial + ((IT)c.slot * H + h) * kW * (F + 2);
#pragma unroll
            for (int j = 0; j < C::MT; ++j)
#pragma unroll
                for (int u = 0; u < 4; ++u) pp[(2 * tig + (u & 1)) * (F + 2) + feature(j, u)] = acc[j][u];
            if (gid == 0) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int r = 2 * tig + u;
                    pp[r * (F + 2) + F] = m_run[u];
                    pp[r * (F + 2) + F + 1] = l_run[u];
                }
            }
        }
    }
    cp_async_wait<0>();
}

// Merge the partials of windows spread over several chunks: one block per
// (window, head), one warp per window row; the window's chunks are
// [multi[2i], multi[2i+1]).  Lane c of a group of 32 chunks holds its weight
// exp(m_c - m), so the features are one weighted sum whose loads do not wait
// for one another.  Bound by the partials' bytes: on the
// 232,965-node graph (114 M edges) 159 us; a dependent load and exp per chunk
// and feature took 202.
template <int V>  // F / 32 features per lane
__global__ void __launch_bounds__(kW * 32) k_gat_combine(
    const int32_t *__restrict__ multi_chunk_begin, const int32_t *__restrict__ chunk_slot,
    const int32_t *__restrict__ chunk_begin, const int32_t *__restrict__ win, int64_t H, int64_t n_nodes,
    const float *__restrict__ partial, float *__restrict__ out, int64_t ldo, float *row_max, float *row_sum) {
    constexpr int F = 32 * V;
    const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int64_t mwin = blockIdx.x / H, h = blockIdx.x - mwin * H;
    const int cb = multi_chunk_begin[2 * mwin], ce = multi_chunk_begin[2 * mwin + 1];
    const int64_t row = (int64_t)win[chunk_begin[cb]] * kW + r;
    if (row >= n_nodes) return;
    const int64_t pitch = kW * (F + 2);
    auto part_row = [&](int c) { return ((int64_t)chunk_slot[c] * H + h) * pitch + r * (F + 2); };
    float m = -INFINITY;
    for (int c = cb + lane; c < ce; c += 32) m = fmaxf(m, partial[part_row(c) + F]);
    m = warp_max(m);
    const float mref = m == -INFINITY ? 0.f : m;
    float l = 0.f, a[V];
#pragma unroll
    for (int v = 0; v < V; ++v) a[v] = 0.f;
    for (int c0 = cb; c0 < ce; c0 += 32) {
        int64_t at = 0;
        float w = 0.f;
        if (c0 + lane < ce) {
            at = part_row(c0 + lane);
            w = __expf(partial[at + F] - mref);
            l += w * partial[at + F + 1];
        }
        const int n = ce - c0 < 32 ? ce - c0 : 32;
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const float wk = __shfl_sync(0xffffffffu, w, k);
            const float *pp = partial + __shfl_sync(0xffffffffu, at, k) + lane;
#pragma unroll
            for (int v = 0; v < V; ++v) a[v] += wk * pp[32 * v];
        }
    }
    l = warp_sum(l);
    const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
    for (int v = 0; v < V; ++v) out[row * ldo + h * F + lane + 32 * v] = a[v] * inv;
    if (lane == 0) {
        if (row_max) row_max[h * n_nodes + row] = m;
        if (row_sum) row_sum[h * n_nodes + row] = l;
    }
}

// rows of windows that own no part (and rows past the last window): zero
__global__ void k_gat_zero_rows(const int32_t *__restrict__ win, int64_t n_parts, int64_t n_nodes,
                                int64_t H, int64_t F, float *out, int64_t ldo, float *row_max,
                                float *row_sum) {
    const int lane = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t n_w = (n_nodes + kW - 1) / kW;
    if (w >= n_w) return;
    int64_t lo = 0, hi = n_parts;
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (win[mid] < w) lo = mid + 1; else hi = mid;
    }
    if (lo < n_parts && win[lo] == w) return;
    for (int64_t r = w * kW; r < (w + 1) * kW && r < n_nodes; ++r) {
        for (int64_t f = lane; f < H * F; f += 32) out[r * ldo + f] = 0.f;
        if (lane < H) {
            if (row_max) row_max[lane * n_nodes + r] = -INFINITY;
            if (row_sum) row_sum[lane * n_nodes + r] = 0.f;
        }
    }
}

// occupancy bitmap from the per-edge slot index
__global__ void k_slot_mask(const int32_t *__restrict__ edge_slot, int64_t nnz, uint32_t *mask) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    const int32_t s = edge_slot[e];
    if (s >= 0) atomicOr(mask + (s >> 5), 1u << (s & 31));
}

// A kernel as a type, for the generic lambdas that launch one of two
template <auto K>
struct GatKernel {
    static constexpr auto value = K;
};

template <typename T, int F, int MODE, bool PSPLIT>
int run_gat(const GatArgs &P, cudaStream_t st, int64_t n_partial) {
    using C = GCfg<T, F, MODE>;
    const GStreamArgs &S = P.S;
    const int64_t items = S.n_runs * S.H;
    if (items == 0) return ATT_OK;
    // 32-bit offsets when X', the output, the statistics and the partials all
    // stay below 2^31 elements
    const int64_t lim = INT32_MAX - (1 << 22);
    ATT_CHECK(items < lim, ATT_ERR_UNSUPPORTED, "too many work items");
    const bool small = S.n_nodes * S.ld < lim && S.n_nodes * P.ldo < lim && S.H * S.n_nodes < lim &&
                       n_partial * S.H * kW * (F + 2) < lim;
    const int grid = (int)(items < sm_count() ? items : sm_count());
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int s = dynamic_smem<kernel>(C::SMEM);
        if (s != ATT_OK) return s;
        kernel<<<grid, C::NW * 32, C::SMEM, st>>>(P);
        return launch_status("k_gat_fused");
    };
    if (small) return run(GatKernel<k_gat_fused<T, F, MODE, PSPLIT, int32_t>>{});
    return run(GatKernel<k_gat_fused<T, F, MODE, PSPLIT, int64_t>>{});
}

template <typename T, int MODE>
int dispatch_gat_f(const GatArgs &P, cudaStream_t st, int64_t np) {
    // statistics requested: training path (16-bit P as hi + lo); fp32 X'
    // always runs 3xTF32 products
    const bool split = P.row_sum != nullptr && sizeof(T) == 2;
    if constexpr (sizeof(T) == 4) {
        switch (P.S.F) {
            case 32: return run_gat<T, 32, MODE, false>(P, st, np);
            case 64: return run_gat<T, 64, MODE, false>(P, st, np);
            case 128: return run_gat<T, 128, MODE, false>(P, st, np);
            default:
                set_error("fused GAT supports F in {32, 64, 128}, got %lld", (long long)P.S.F);
                return ATT_ERR_UNSUPPORTED;
        }
    } else {
        switch (P.S.F) {
            case 32: return split ? run_gat<T, 32, MODE, true>(P, st, np) : run_gat<T, 32, MODE, false>(P, st, np);
            case 64: return split ? run_gat<T, 64, MODE, true>(P, st, np) : run_gat<T, 64, MODE, false>(P, st, np);
            case 128: return split ? run_gat<T, 128, MODE, true>(P, st, np) : run_gat<T, 128, MODE, false>(P, st, np);
            default:
                set_error("fused GAT supports F in {32, 64, 128}, got %lld", (long long)P.S.F);
                return ATT_ERR_UNSUPPORTED;
        }
    }
}

// ---------------------------------------------------------------------------
// Backward of the additive GAT layer, fused.  With the forward's row max m and
// sum l saved, and c_i = dout_i . out_i, every edge term is local:
//   p_ij  = exp(LeakyReLU(s0_i + s1_j) - m_i) / l_i
//   dp_ij = dout_i . X'_j
//   dz_ij = p_ij (dp_ij - c_i) LeakyReLU'(s0_i + s1_j)
//   dX'_j += p_ij dout_i      (the SpMM adjoint)
//   ds1_j += dz_ij,  ds0_i += dz_ij
// One pass over the block format of the TRANSPOSED graph: window rows are the
// j's, condensed columns the i's.  Per 16 columns: the dout rows of the i's
// are gathered (cp.async ring) and feed dp (mma, K = F) and the adjoint
// product (mma after a movmatrix transpose of p); ds1 is a register row sum,
// ds0 one atomic add per (window, column).  All outputs are accumulated with
// red.global.add into zeroed buffers.
struct GatBwdArgs {
    const int32_t *rowptr, *col, *win;
    const uint32_t *mask;
    int64_t n_parts;
    int wide;
    const void *Xp;    // X'[j][h*F + f]  (rows of the transposed windows)
    const void *dout;     // dout[i][h*F + f] (gathered)
    const void *dout_lo;  // dout - dout (rounded), same layout, or null
    int64_t n_nodes, H, F, ldx, ldd;
    const float *s0, *s1, *m, *l, *c;  // [H][n_nodes]
    float slope;
    float *dXp;  // [n_nodes][H*F] fp32, ld ldg
    int64_t ldg;
    float *ds0, *ds1;  // [H][n_nodes]
    int32_t *err;
};

// the backward's ring depth: 2 stages leave room for 6 CTAs per SM where 3
// stages allowed 4 (the kernel is latency-bound: warps matter more than depth)
constexpr int kBStages = 2;

template <typename T, int F, bool SPLIT>
struct BCfg {
    static constexpr int XROW = F * 2;
    static constexpr int TILE = 16 * XROW;
    static constexpr int XSTAGE = (SPLIT ? 2 : 1) * TILE;
    static constexpr int MSTAGE = 16;
    static constexpr int CSTAGE = 5 * 64;  // s0, m, l, c and the ids of the 16 columns
    static constexpr int STAGE = XSTAGE + MSTAGE + CSTAGE;
    static constexpr int WARP_SMEM = kBStages * STAGE;
    static constexpr int SMEM = kGWarps * WARP_SMEM;
    static constexpr int CPR = XROW / 16;
    static constexpr int PASSES = (16 * CPR + 31) / 32;
    static constexpr int MT = F / 16;
};

// IT: index type of items and element offsets (int32_t when every offset fits)
template <typename T, int F, bool SPLIT, typename IT>
__global__ void __launch_bounds__(kGThreads) k_gat_backward(GatBwdArgs A) {
    using C = BCfg<T, F, SPLIT>;
    const IT H = (IT)A.H, n_nodes = (IT)A.n_nodes, ldd = (IT)A.ldd, ldx = (IT)A.ldx,
             ldg = (IT)A.ldg;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sbase = smem_u32(smem) + warp * C::WARP_SMEM;
    const unsigned char *sgen = smem + warp * C::WARP_SMEM;
    const int gid = lane >> 2, tig = lane & 3;
    const IT n_items = (IT)(A.n_parts * A.H);
    const IT stride = (IT)gridDim.x * kGWarps;
    const T *Xq = (const T *)A.Xp;
    const T *D = (const T *)A.dout;
    const T *DL = (const T *)A.dout_lo;

    IT p_item = (IT)blockIdx.x * kGWarps + warp;
    IT p_h = 0;
    int p_start = 0, p_nreal = 0, p_pend = 0, p_step = 0, p_myc = -1;
    auto p_load = [&]() {
        while (p_item < n_items) {
            const IT part = p_item / H;
            p_h = p_item - part * H;
            p_start = A.rowptr[2 * part];
            const int e = A.rowptr[2 * part + 1];
            p_pend = A.rowptr[2 * part + 2];
            p_nreal = e > p_start ? e - p_start : 0;
            if ((p_start % A.wide) != 0 || (p_pend % A.wide) != 0 || p_pend < p_start + p_nreal) {
                if (A.err) atomicOr(A.err, 2);
                p_nreal = 0;
            }
            p_step = 0;
            if (p_nreal > 0) return;
            p_item += stride;
        }
    };
    auto issue = [&](int stage) {
        const uint32_t xs = sbase + stage * C::STAGE;
        const uint32_t ms = xs + C::XSTAGE;
        const uint32_t cs = ms + C::MSTAGE;
        const int c0 = p_step * 16;
        int myc = p_myc;  // fetched one step ahead
        if (myc >= n_nodes || myc < -1) {
            if (A.err) atomicOr(A.err, 1);
            myc = -1;
        }
#pragma unroll
        for (int i = 0; i < C::PASSES; ++i) {
            const int idx = i * 32 + lane;
            const int r = idx / C::CPR, ch = idx % C::CPR;
            const int cidx = __shfl_sync(0xffffffffu, myc, r & 15);
            if (idx < 16 * C::CPR) {
                const bool ok = cidx >= 0;
                const IT o = (IT)cidx * ldd + p_h * F + ch * 8;
                const uint32_t d = r * C::XROW + ((ch ^ swz_row<F>(r)) << 4);
                cp_async16(xs + d, ok ? D + o : D, ok ? 16 : 0);
                if constexpr (SPLIT) cp_async16(xs + C::TILE + d, ok ? DL + o : DL, ok ? 16 : 0);
            }
        }
        if (lane < 2) {
            const bool ok = c0 + 8 * lane < p_pend - p_start;
            const int64_t bit0 = (int64_t)(p_start + c0 + 8 * lane) * kW;  // bit index: 64-bit always
            cp_async8(ms + 8 * lane, ok ? (const void *)(A.mask + (bit0 >> 5)) : (const void *)A.mask,
                      ok ? 8 : 0);
        }
        if (lane < 16) {
            const bool ok = myc >= 0;
            const IT o = p_h * n_nodes + (ok ? myc : 0);
            const float *arrs[4] = {A.s0, A.m, A.l, A.c};
#pragma unroll
            for (int a = 0; a < 4; ++a)
                cp_async4(cs + a * 64 + 4 * lane, arrs[a] + o, ok ? 4 : 0);
            // the column ids themselves, for the ds0 scatter (-1: none)
            asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(cs + 4 * 64 + 4 * lane), "r"(myc)
                         : "memory");
        }
    };
    auto p_fetch = [&]() {
        p_myc = -1;
        if (p_item < n_items && p_step * 16 + (lane & 15) < p_nreal)
            p_myc = A.col[p_start + p_step * 16 + (lane & 15)];
    };
    auto p_advance = [&]() {
        if (++p_step * 16 >= p_nreal) {
            p_item += stride;
            p_load();
        }
        p_fetch();
    };

    p_load();
    p_fetch();
#pragma unroll
    for (int s = 0; s < kBStages - 1; ++s) {
        if (p_item < n_items) {
            issue(s);
            p_advance();
        }
        cp_async_commit();
    }

    const int wmask = A.wide - 1;  // wide is a power of two
    int mbit[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int c = gid + 8 * (u >> 1), r = 2 * tig + (u & 1);
        mbit[u] = (c & ~wmask) * kW + r * A.wide + (c & wmask);
    }
    int cstage = 0, pstage = kBStages - 1;
    for (IT c_item = (IT)blockIdx.x * kGWarps + warp; c_item < n_items; c_item += stride) {
        const IT part = c_item / H;
        const IT h = c_item - part * H;
        const int start = A.rowptr[2 * part];
        const int e = A.rowptr[2 * part + 1];
        const int pend = A.rowptr[2 * part + 2];
        int nreal = e > start ? e - start : 0;
        if ((start & wmask) != 0 || (pend & wmask) != 0 || pend < start + nreal) nreal = 0;
        const int nsteps = (nreal + 15) >> 4;
        if (nsteps == 0) continue;
        const IT wrow = (IT)A.win[part] * kW;
        uint32_t bq[C::MT][2];
#pragma unroll
        for (int kk = 0; kk < C::MT; ++kk)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const IT row = wrow + gid;
                const int f = 16 * kk + 2 * tig + 8 * u;
                bq[kk][u] = row < n_nodes ? *(const uint32_t *)(Xq + row * ldx + h * F + f) : 0u;
            }
        float s1r[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const IT row = wrow + 2 * tig + u;
            s1r[u] = row < n_nodes ? A.s1[h * n_nodes + row] : 0.f;
        }
        float ds1_acc[2] = {0.f, 0.f};
        float acc[C::MT][4];
#pragma unroll
        for (int j = 0; j < C::MT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

        for (int step = 0; step < nsteps; ++step) {
            cp_async_wait<kBStages - 2>();
            __syncwarp();
            const uint32_t xs = sbase + cstage * C::STAGE;
            const uint32_t *mw = (const uint32_t *)(sgen + cstage * C::STAGE + C::XSTAGE);
            const float *cv = (const float *)(sgen + cstage * C::STAGE + C::XSTAGE + C::MSTAGE);
            // dp[c][r] = dout_c . X'_r
            float dp[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kk = 0; kk < C::MT; ++kk) {
                const int q = lane >> 3, rr = lane & 7;
                const int mrow = (q & 1) * 8 + rr;
                const int ch = 2 * kk + (q >> 1);
                const uint32_t ad = mrow * C::XROW + ((ch ^ swz_row<F>(mrow)) << 4);
                uint32_t a[4];
                ldsm_x4(xs + ad, a[0], a[1], a[2], a[3]);
                mma_16816<T>(dp, a, bq[kk][0], bq[kk][1]);
                if constexpr (SPLIT) {
                    ldsm_x4(xs + C::TILE + ad, a[0], a[1], a[2], a[3]);
                    mma_16816<T>(dp, a, bq[kk][0], bq[kk][1]);
                }
            }
            const int c0 = step * 16;
            float p[4], dz[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = gid + 8 * (u >> 1);
                const bool occ = c0 + c < nreal && ((mw[mbit[u] >> 5] >> (mbit[u] & 31)) & 1u);
                const float s0c = cv[c], mc = cv[16 + c], lc = cv[32 + c], cc = cv[48 + c];
                const float z = s0c + s1r[u & 1];
                const float lr = z > 0.f ? z : A.slope * z;
                const float pv = occ && lc > 0.f ? __fdividef(__expf(lr - mc), lc) : 0.f;
                p[u] = pv;
                dz[u] = pv * (dp[u] - cc) * (z > 0.f ? 1.f : A.slope);
            }
            // ds1 (rows): each lane sums its own columns; the row's lanes are
            // reduced once per work item
            ds1_acc[0] += dz[0] + dz[2];
            ds1_acc[1] += dz[1] + dz[3];
            // ds0 (columns): sum over the 8 rows, one atomic per column
            float c_lo = dz[0] + dz[1], c_hi = dz[2] + dz[3];
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                c_lo += __shfl_xor_sync(0xffffffffu, c_lo, o);
                c_hi += __shfl_xor_sync(0xffffffffu, c_hi, o);
            }
            if (tig == 0) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int ci = ((const int *)(cv + 64))[gid + 8 * u];  // -1 past nreal
                    if (ci >= 0 && ci < n_nodes)
                        red_add_f32(A.ds0 + h * n_nodes + ci, u ? c_hi : c_lo);
                }
            }
            // dX'_r += sum_c p[c][r] dout_c
            const uint32_t b0 = movmatrix_trans(pack2<T>(p[0], p[1]));
            const uint32_t b1 = movmatrix_trans(pack2<T>(p[2], p[3]));
#pragma unroll
            for (int j = 0; j < C::MT; ++j) {
                const int q = lane >> 3, rr = lane & 7;
                const int k = (q >> 1) * 8 + rr;
                const int ch = 2 * j + (q & 1);
                const uint32_t ad = k * C::XROW + ((ch ^ swz_row<F>(k)) << 4);
                uint32_t a[4];
                ldsm_x4_trans(xs + ad, a[0], a[1], a[2], a[3]);
                mma_16816<T>(acc[j], a, b0, b1);
                if constexpr (SPLIT) {
                    ldsm_x4_trans(xs + C::TILE + ad, a[0], a[1], a[2], a[3]);
                    mma_16816<T>(acc[j], a, b0, b1);
                }
            }
            __syncwarp();
            if (p_item < n_items) {
                issue(pstage);
                p_advance();
            }
            cp_async_commit();
            cstage = cstage + 1 == kBStages ? 0 : cstage + 1;
            pstage = pstage + 1 == kBStages ? 0 : pstage + 1;
        }
#pragma unroll
        for (int j = 0; j < C::MT; ++j)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const IT row = wrow + 2 * tig + (u & 1);
                const int f = 16 * j + gid + 8 * (u >> 1);
                if (row < n_nodes) red_add_f32(A.dXp + row * ldg + h * F + f, acc[j][u]);
            }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            ds1_acc[0] += __shfl_xor_sync(0xffffffffu, ds1_acc[0], o);
            ds1_acc[1] += __shfl_xor_sync(0xffffffffu, ds1_acc[1], o);
        }
        if (gid == 0) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const IT row = wrow + 2 * tig + u;
                if (row < n_nodes) red_add_f32(A.ds1 + h * n_nodes + row, ds1_acc[u]);
            }
        }
    }
    cp_async_wait<0>();
}

template <typename T, int F, bool SPLIT>
int run_gat_bwd(const GatBwdArgs &P, cudaStream_t st) {
    using C = BCfg<T, F, SPLIT>;
    const int64_t items = P.n_parts * P.H;
    if (items == 0) return ATT_OK;
    auto run = [&](auto k) {
        constexpr auto kernel = decltype(k)::value;
        const int prep = dynamic_smem<kernel>(C::SMEM);
        if (prep != ATT_OK) return prep;
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kGThreads, C::SMEM);
        if (per_sm < 1) per_sm = 1;
        const int64_t want = (items + kGWarps - 1) / kGWarps;
        const int64_t cap = (int64_t)sm_count() * per_sm;
        kernel<<<(unsigned)(want < cap ? want : cap), kGThreads, C::SMEM, st>>>(P);
        return launch_status("k_gat_backward");
    };
    // 32-bit offsets when rows of X', dout and dXp, the per-head node arrays
    // and the item count (plus one grid stride) all stay below 2^31
    const int64_t lim = INT32_MAX - (1 << 22);
    int64_t ld = P.ldx > P.ldd ? P.ldx : P.ldd;
    ld = ld > P.ldg ? ld : P.ldg;
    const bool small = P.n_nodes * ld < lim && P.n_nodes * P.H < lim && items < lim;
    if (small) return run(GatKernel<k_gat_backward<T, F, SPLIT, int32_t>>{});
    return run(GatKernel<k_gat_backward<T, F, SPLIT, int64_t>>{});
}

template <typename T>
int dispatch_gat_bwd(const GatBwdArgs &P, cudaStream_t st) {
    const bool split = P.dout_lo != nullptr;
    switch (P.F) {
        case 32: return split ? run_gat_bwd<T, 32, true>(P, st) : run_gat_bwd<T, 32, false>(P, st);
        case 64: return split ? run_gat_bwd<T, 64, true>(P, st) : run_gat_bwd<T, 64, false>(P, st);
        case 128: return split ? run_gat_bwd<T, 128, true>(P, st) : run_gat_bwd<T, 128, false>(P, st);
        default:
            set_error("fused GAT backward supports F in {32, 64, 128}, got %lld", (long long)P.F);
            return ATT_ERR_UNSUPPORTED;
    }
}

}  // namespace
}  // namespace att

using namespace att;

extern "C" int att_slot_mask(const int32_t *edge_slot, int64_t nnz, uint32_t *mask,
                             int64_t n_words, void *stream) {
    clear_error();
    cudaStream_t st = (cudaStream_t)stream;
    if (n_words > 0) {
        ATT_CHECK(mask != nullptr, ATT_ERR_INVALID, "null mask");
        ATT_CUDA(cudaMemsetAsync(mask, 0, (size_t)n_words * 4, st), "memset mask");
    }
    if (nnz == 0) return ATT_OK;
    ATT_CHECK(edge_slot != nullptr, ATT_ERR_INVALID, "null edge_slot");
    k_slot_mask<<<(unsigned)((nnz + 255) / 256), 256, 0, st>>>(edge_slot, nnz, mask);
    return launch_status("k_slot_mask");
}

extern "C" int att_gat_forward(const int32_t *rowptr, const int32_t *col, const uint32_t *slot_mask,
                               const int32_t *window_of_part, int64_t n_parts,
                               const int32_t *chunk_begin, const int32_t *chunk_slot,
                               int64_t n_chunks, const int32_t *multi_chunk_begin,
                               int64_t n_multi, int window, int wide, const void *Xp, int x_dtype,
                               int64_t n_nodes, int64_t n_heads, int64_t F, int64_t ldx, int mode,
                               const float *s0, const float *s1, float slope, float *out,
                               int64_t ldo, float *row_max, float *row_sum, float *partial,
                               int32_t *err_flag, void *stream) {
    clear_error();
    ATT_CHECK(window == kW, ATT_ERR_UNSUPPORTED, "fused GAT needs 8-row windows");
    ATT_CHECK(wide == 4 || wide == 8 || wide == 16, ATT_ERR_UNSUPPORTED, "wide must be 4, 8 or 16");
    ATT_CHECK(mode == 0 || mode == 1, ATT_ERR_INVALID, "mode must be 0 (dot) or 1 (additive)");
    ATT_CHECK(x_dtype == ATT_F16 || x_dtype == ATT_BF16 || x_dtype == ATT_F32, ATT_ERR_UNSUPPORTED,
              "fused GAT takes fp16, bf16 or fp32 (3xTF32) features");
    ATT_CHECK(n_heads > 0 && n_heads <= 32 && F > 0, ATT_ERR_INVALID, "bad heads / features");
    ATT_CHECK(ldx % (x_dtype == ATT_F32 ? 4 : 8) == 0 && ((uintptr_t)Xp & 15) == 0 &&
                  ldx >= n_heads * F,
              ATT_ERR_UNSUPPORTED, "X' rows must be 16-byte aligned with ldx >= heads*F");
    ATT_CHECK(ldo >= n_heads * F, ATT_ERR_INVALID, "ldo < heads*F");
    ATT_CHECK(mode == 0 || (s0 && s1), ATT_ERR_INVALID, "additive mode needs node scores");
    cudaStream_t st = (cudaStream_t)stream;
    if (n_nodes == 0) return ATT_OK;
    {
        const int64_t threads = (n_nodes + kW - 1) / kW * 32;
        k_gat_zero_rows<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(
            window_of_part, n_parts, n_nodes, n_heads, F, out, ldo, row_max, row_sum);
        int s = launch_status("k_gat_zero_rows");
        if (s != ATT_OK) return s;
    }
    if (n_chunks == 0) return ATT_OK;
    ATT_CHECK(rowptr && col && slot_mask && window_of_part && chunk_begin && chunk_slot,
              ATT_ERR_INVALID, "null format pointer");
    ATT_CHECK(n_multi == 0 || (partial && multi_chunk_begin), ATT_ERR_INVALID,
              "split windows need the partial buffer");
    GatArgs P{GStreamArgs{rowptr, col, window_of_part, slot_mask, chunk_begin, chunk_slot, n_chunks, n_heads, n_nodes,
                          F, wide, Xp, ldx, s1, err_flag},
              s0, slope, out, ldo, row_max, row_sum, partial};
    int s;
    // partial slots are at most one per chunk
    const int64_t np = n_chunks;
    if (x_dtype == ATT_F16)
        s = mode == 0 ? dispatch_gat_f<__half, 0>(P, st, np) : dispatch_gat_f<__half, 1>(P, st, np);
    else if (x_dtype == ATT_F32)
        s = mode == 0 ? dispatch_gat_f<float, 0>(P, st, np) : dispatch_gat_f<float, 1>(P, st, np);
    else
        s = mode == 0 ? dispatch_gat_f<__nv_bfloat16, 0>(P, st, np)
                      : dispatch_gat_f<__nv_bfloat16, 1>(P, st, np);
    if (s != ATT_OK) return s;
    if (n_multi > 0) {
        auto combine = [&](auto kernel) {
            kernel<<<(unsigned)(n_multi * n_heads), kW * 32, 0, st>>>(multi_chunk_begin, chunk_slot, chunk_begin,
                                                                    window_of_part, n_heads, n_nodes, partial, out,
                                                                    ldo, row_max, row_sum);
        };
        if (F == 32) combine(k_gat_combine<1>);
        else if (F == 64) combine(k_gat_combine<2>);
        else combine(k_gat_combine<4>);
        s = launch_status("k_gat_combine");
    }
    return s;
}

extern "C" int att_gat_backward(const int32_t *rowptr_t, const int32_t *col_t,
                                const uint32_t *slot_mask_t, const int32_t *window_of_part_t,
                                int64_t n_parts_t, int window, int wide, const void *Xp,
                                const void *dout, const void *dout_lo, int x_dtype, int64_t n_nodes, int64_t n_heads,
                                int64_t F, int64_t ldx, int64_t ldd, const float *s0,
                                const float *s1, const float *row_max, const float *row_sum,
                                const float *c, float slope, float *dXp, int64_t ldg, float *ds0,
                                float *ds1, int32_t *err_flag, void *stream) {
    clear_error();
    ATT_CHECK(window == kW, ATT_ERR_UNSUPPORTED, "fused GAT backward needs 8-row windows");
    ATT_CHECK(wide == 4 || wide == 8 || wide == 16, ATT_ERR_UNSUPPORTED, "wide must be 4, 8 or 16");
    ATT_CHECK(x_dtype == ATT_F16 || x_dtype == ATT_BF16, ATT_ERR_UNSUPPORTED,
              "fused GAT backward takes fp16 or bf16 X' and dout");
    ATT_CHECK(n_heads > 0 && F > 0, ATT_ERR_INVALID, "bad heads / features");
    ATT_CHECK(ldx % 8 == 0 && ldd % 8 == 0 && ((uintptr_t)Xp & 15) == 0 &&
                  ((uintptr_t)dout & 15) == 0 && ((uintptr_t)dout_lo & 15) == 0,
              ATT_ERR_UNSUPPORTED, "X' and dout rows must be 16-byte aligned");
    ATT_CHECK(s0 && s1 && row_max && row_sum && c && dXp && ds0 && ds1, ATT_ERR_INVALID,
              "null pointer");
    if (n_parts_t == 0 || n_nodes == 0) return ATT_OK;
    ATT_CHECK(rowptr_t && col_t && slot_mask_t && window_of_part_t, ATT_ERR_INVALID,
              "null format pointer");
    GatBwdArgs P{rowptr_t, col_t, window_of_part_t, slot_mask_t, n_parts_t, wide, Xp, dout,
                 dout_lo, n_nodes, n_heads, F, ldx, ldd, s0, s1, row_max, row_sum, c, slope, dXp, ldg,
                 ds0, ds1, err_flag};
    cudaStream_t st = (cudaStream_t)stream;
    return x_dtype == ATT_F16 ? dispatch_gat_bwd<__half>(P, st) : dispatch_gat_bwd<__nv_bfloat16>(P, st);
}

// ---------------------------------------------------------------------------
// Elementwise ends of the fused GAT backward (one pass each over [N, H*F])
// ---------------------------------------------------------------------------
namespace att {
namespace {

template <typename T>
__device__ __forceinline__ T to_t(float v);
template <>
__device__ __forceinline__ __half to_t<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 to_t<__nv_bfloat16>(float v) {
    return __float2bfloat16_rn(v);
}
template <typename T>
__device__ __forceinline__ float from_t(T v);
template <>
__device__ __forceinline__ float from_t<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float from_t<__nv_bfloat16>(__nv_bfloat16 v) {
    return __bfloat162float(v);
}

// One warp per node row: c[h][n] = dout[n, h] . out[n, h] (fp32), and dout
// split into a 16-bit hi part and the 16-bit rounding of its remainder.
template <typename T>
__global__ void k_gat_grad_prepare(const float *__restrict__ dout, int64_t ldd,
                                   const float *__restrict__ out, int64_t ldo, int64_t n_nodes,
                                   int64_t H, int64_t F, T *__restrict__ hi, T *__restrict__ lo,
                                   int64_t ldh, float *__restrict__ c) {
    const int lane = threadIdx.x & 31;
    const int64_t n = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (n >= n_nodes) return;
    for (int64_t h = 0; h < H; ++h) {
        float s = 0.f;
        for (int64_t f = lane; f < F; f += 32) {
            const int64_t col = h * F + f;
            const float d = dout[n * ldd + col];
            s += d * out[n * ldo + col];
            const T dh = to_t<T>(d);
            hi[n * ldh + col] = dh;
            lo[n * ldh + col] = to_t<T>(d - from_t<T>(dh));
        }
        s = warp_sum(s);
        if (lane == 0) c[h * n_nodes + n] = s;
    }
}

// The same for F = 32 NF, with 16-byte loads and the same order of sums: 8
// lanes per (node, head), lane k holding features 4 k + i + 32 j, whose partial
// sums over j are those of lanes 4 k + i above; lanes k ^ 4, 2, 1 exchange them
// (steps 16, 8, 4 of the warp sum), the last two steps are its own.  Bound by the
// bytes of dout, out and the two 16-bit halves (520 MB at 169,343 nodes, 4 heads x 64):
// 127 -> 79 us.
template <typename T, int NF>
__global__ void __launch_bounds__(256) k_gat_grad_prepare_vec(
    const float *__restrict__ dout, int64_t ldd, const float *__restrict__ out, int64_t ldo, int64_t n_nodes,
    int64_t H, T *__restrict__ hi, T *__restrict__ lo, int64_t ldh, float *__restrict__ c) {
    constexpr int F = 32 * NF;
    const int k = threadIdx.x & 7;
    const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const bool ok = g < n_nodes * H;
    const int64_t n = ok ? g / H : 0, h = ok ? g - n * H : 0;
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    if (ok) {
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int64_t col = h * F + 32 * j + 4 * k;
            const float4 d = __ldcs(reinterpret_cast<const float4 *>(dout + n * ldd + col));
            const float4 o = __ldcs(reinterpret_cast<const float4 *>(out + n * ldo + col));
            const float dv[4] = {d.x, d.y, d.z, d.w}, ov[4] = {o.x, o.y, o.z, o.w};
            alignas(8) T hv[4], lv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                t[i] += dv[i] * ov[i];
                hv[i] = to_t<T>(dv[i]);
                lv[i] = to_t<T>(dv[i] - from_t<T>(hv[i]));
            }
            *reinterpret_cast<uint2 *>(hi + n * ldh + col) = *reinterpret_cast<const uint2 *>(hv);
            *reinterpret_cast<uint2 *>(lo + n * ldh + col) = *reinterpret_cast<const uint2 *>(lv);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] += __shfl_xor_sync(0xffffffffu, t[i], o);
    if (ok && k == 0) c[h * n_nodes + n] = (t[0] + t[2]) + (t[1] + t[3]);
}

// dX[n, hF+f] = cast(dXp[n, hF+f] + ds0[h][n] a0[h][f] + ds1[h][n] a1[h][f]);
// da0[h][f] += sum_n ds0[h][n] X'[n, hF+f], da1 likewise (fp32 atomics, one
// per column per thread).  A block covers 256 columns of several rows per
// sweep (256 / HF rows when HF <= 256).
template <typename T>
__global__ void __launch_bounds__(256) k_gat_grad_finish(
    const float *__restrict__ dXp, int64_t ldg, const float *__restrict__ ds0,
    const float *__restrict__ ds1, const float *__restrict__ a0, const float *__restrict__ a1,
    const T *__restrict__ Xp, int64_t ldx, int64_t n_nodes, int64_t H, int64_t F,
    T *__restrict__ dX, int64_t ldo, float *__restrict__ da0, float *__restrict__ da1) {
    const int64_t HF = H * F;
    const int t = threadIdx.x;
    const int64_t cols = HF < 256 ? HF : 256;
    const int64_t rows = 256 / cols;  // rows per sweep of the block
    const int64_t roff = t / cols;
    if (roff >= rows) return;
    for (int64_t cb = 0; cb < HF; cb += 256) {
        const int64_t col = cb + t % cols;
        if (col >= HF) continue;
        const int64_t h = col / F;
        const float w0 = a0[col], w1 = a1[col];
        float acc0 = 0.f, acc1 = 0.f;
        for (int64_t n = (int64_t)blockIdx.x * rows + roff; n < n_nodes; n += (int64_t)gridDim.x * rows) {
            const float g0 = ds0[h * n_nodes + n], g1 = ds1[h * n_nodes + n];
            const float x = from_t<T>(Xp[n * ldx + col]);
            dX[n * ldo + col] = to_t<T>(dXp[n * ldg + col] + g0 * w0 + g1 * w1);
            acc0 += g0 * x;
            acc1 += g1 * x;
        }
        atomicAdd(da0 + col, acc0);
        atomicAdd(da1 + col, acc1);
    }
}

}  // namespace
}  // namespace att

extern "C" int att_gat_grad_prepare(const float *dout, int64_t ldd, const float *out, int64_t ldo,
                                    int64_t n_nodes, int64_t n_heads, int64_t F, void *dout_hi,
                                    void *dout_lo, int dtype, int64_t ldh, float *c, void *stream) {
    using namespace att;
    clear_error();
    ATT_CHECK(dtype == ATT_F16 || dtype == ATT_BF16, ATT_ERR_UNSUPPORTED,
              "dout splits into fp16 or bf16");
    ATT_CHECK(n_nodes >= 0 && n_heads > 0 && F > 0, ATT_ERR_INVALID, "bad sizes");
    ATT_CHECK(ldd >= n_heads * F && ldo >= n_heads * F && ldh >= n_heads * F, ATT_ERR_INVALID,
              "row strides shorter than heads x F");
    if (n_nodes == 0) return ATT_OK;
    ATT_CHECK(dout && out && dout_hi && dout_lo && c, ATT_ERR_INVALID, "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    // whole rows of 32 features and 16-byte pieces; any other layout by the
    // scalar kernel
    const bool vec = (F == 32 || F == 64 || F == 128) && ldd % 4 == 0 && ldo % 4 == 0 && ldh % 4 == 0 &&
                     (((uintptr_t)dout | (uintptr_t)out) & 15) == 0 &&
                     (((uintptr_t)dout_hi | (uintptr_t)dout_lo) & 7) == 0;
    auto run = [&](auto *t) {
        using T = std::remove_pointer_t<decltype(t)>;
        if (vec) {
            const unsigned grid = (unsigned)((n_nodes * n_heads * 8 + 255) / 256);
            auto go = [&](auto kernel) {
                kernel<<<grid, 256, 0, st>>>(dout, ldd, out, ldo, n_nodes, n_heads, (T *)dout_hi, (T *)dout_lo, ldh, c);
            };
            if (F == 32) go(k_gat_grad_prepare_vec<T, 1>);
            else if (F == 64) go(k_gat_grad_prepare_vec<T, 2>);
            else go(k_gat_grad_prepare_vec<T, 4>);
        } else {
            k_gat_grad_prepare<T><<<(unsigned)((n_nodes * 32 + 255) / 256), 256, 0, st>>>(
                dout, ldd, out, ldo, n_nodes, n_heads, F, (T *)dout_hi, (T *)dout_lo, ldh, c);
        }
    };
    if (dtype == ATT_F16) run((__half *)nullptr);
    else run((__nv_bfloat16 *)nullptr);
    return launch_status("k_gat_grad_prepare");
}

extern "C" int att_gat_grad_finish(const float *dXp, int64_t ldg, const float *ds0, const float *ds1,
                                   const float *a0, const float *a1, const void *Xp, int dtype,
                                   int64_t ldx, int64_t n_nodes, int64_t n_heads, int64_t F, void *dX,
                                   int64_t ld_dx, float *da0, float *da1, void *stream) {
    using namespace att;
    clear_error();
    ATT_CHECK(dtype == ATT_F16 || dtype == ATT_BF16, ATT_ERR_UNSUPPORTED,
              "X' and dX are fp16 or bf16");
    ATT_CHECK(n_nodes >= 0 && n_heads > 0 && F > 0, ATT_ERR_INVALID, "bad sizes");
    ATT_CHECK(ldg >= n_heads * F && ldx >= n_heads * F && ld_dx >= n_heads * F, ATT_ERR_INVALID,
              "row strides shorter than heads x F");
    if (n_nodes == 0) return ATT_OK;
    ATT_CHECK(dXp && ds0 && ds1 && a0 && a1 && Xp && dX && da0 && da1, ATT_ERR_INVALID,
              "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t HF = n_heads * F;
    const int64_t rows = 256 / (HF < 256 ? HF : 256);
    int64_t want = (n_nodes + rows - 1) / rows;
    const int64_t cap = (int64_t)sm_count() * 8;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    if (dtype == ATT_F16)
        k_gat_grad_finish<__half><<<grid, 256, 0, st>>>(dXp, ldg, ds0, ds1, a0, a1,
                                                        (const __half *)Xp, ldx, n_nodes, n_heads,
                                                        F, (__half *)dX, ld_dx, da0, da1);
    else
        k_gat_grad_finish<__nv_bfloat16><<<grid, 256, 0, st>>>(
            dXp, ldg, ds0, ds1, a0, a1, (const __nv_bfloat16 *)Xp, ldx, n_nodes, n_heads, F,
            (__nv_bfloat16 *)dX, ld_dx, da0, da1);
    return launch_status("k_gat_grad_finish");
}
