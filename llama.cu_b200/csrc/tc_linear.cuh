// What the tcgen05 forms of the linear layer share: the vector epilogues and the operand maps.
#pragma once
#include "gemv.cuh"
#include "tc.cuh"

namespace lcu {

constexpr int TC_BK = 64;  // K elements per stage (128 bytes: one swizzle row)

// ---- Q8_0 weights as pairs of f16: scale * q = hi + lo, hi the rounded product, lo the rest.  Exact: the product is a whole multiple
// of 2^-24 with at most 19 bits, so both halves are f16 numbers (subnormal ones among them) wherever hi does not overflow (tc_q8_mend), and f16
// products summed in f32 lose no more than integer products scaled block by block.  Twice the MMAs of f16 weights.
constexpr int TQ_K = 256;  // K elements per unit of the form with weights on lanes: 16 bytes of scales a row

#ifdef __CUDACC__
__device__ __forceinline__ void tc_q8_split(const uint4 &q, __half2 s, uint32_t hi[8], uint32_t lo[8]) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t h[2];
        q8x4_to_h2(w[i], h[0], h[1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const __half2 v = *reinterpret_cast<__half2 *>(&h[k]), p = __hmul2(v, s), r = __hfma2(v, s, __hneg2(p));
            hi[2 * i + k] = *reinterpret_cast<const uint32_t *>(&p);
            lo[2 * i + k] = *reinterpret_cast<const uint32_t *>(&r);
        }
    }
}
// Sums that are not finite: the split has overflowed (a scale times 127 beyond the range of f16), or the activations are not finite
// themselves and an infinity has met a low half that is zero or of the other sign.  Then the products are taken block by block in
// f32; the whole warp works on one token, for four rows per lane (below 0: none):
//   a NaN among the activations     every product is NaN, as the sums are already;
//   infinities                      only they and blocks whose scale is not finite decide, so a lane walks those for its own rows;
//   finite activations              the lanes share the blocks of one row after the other.
// A round waits for its slowest token, so this may not cost much more than the products themselves.  28672 x 4096, against one thread
// per product: all of 500 tokens NaN 256 -> 0.24 ms (finite 0.23, mma.sync kernel 1.04), one of 64 tokens 2.3 -> 0.067 ms (finite
// 0.064), infinities in all of 500 tokens 256 -> 1.8 to 3 ms (of one overflow, only the next matrix sees infinities: norms turn them
// into NaN).
enum { TQ_UNKNOWN = 0, TQ_FINITE, TQ_INF, TQ_NAN };  // what a token's activations hold
template <int R>
struct TqRows {
    float v[R];
    int known;
};
template <int R>
__device__ __noinline__ TqRows<R> tc_q8_rows(const int8_t *q, const __half *s, const __half *x, int in, int4 rows, int known) {
    const int lane = threadIdx.x & 31, nb = in / 32, row[4] = {rows.x, rows.y, rows.z, rows.w};
    TqRows<R> o;
#pragma unroll
    for (int r = 0; r < R; ++r) o.v[r] = 0.f;
    o.known = known;
    auto load = [&](int k, uint4 v[8]) {  // this lane's eight of every 256 activations, 2048 at once (in % 256 == 0: lanes go round together)
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = k + 256 * j < in ? *reinterpret_cast<const uint4 *>(x + k + 256 * j) : make_uint4(0, 0, 0, 0);
    };
    if (known == TQ_UNKNOWN) {
        unsigned top = 0;  // the largest magnitudes, as bits
        bool nan = false;
        for (int k = lane * 8; k < in && !nan; k += 2048) {
            uint4 v[8];
            load(k, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) top = __vmaxu2(top, w[i] & 0x7fff7fffu);
            }
            nan = __any_sync(0xffffffffu, (top & 0xffffu) > 0x7c00u || (top >> 16) > 0x7c00u);
        }
        o.known = nan ? TQ_NAN : __any_sync(0xffffffffu, (top & 0xffffu) == 0x7c00u || (top >> 16) == 0x7c00u) ? TQ_INF : TQ_FINITE;
    }
    if (o.known == TQ_NAN) {
#pragma unroll
        for (int r = 0; r < R; ++r) o.v[r] = NAN;
        return o;
    }
    if (o.known == TQ_INF) {
        for (int k0 = 0; k0 < in; k0 += 2048) {
            uint4 v[8];
            load(k0 + lane * 8, v);
            unsigned long long inf = 0, neg = 0;  // which of this lane's 64, and their signs
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned h = w[i >> 1] >> (16 * (i & 1));
                    inf |= (unsigned long long)((h & 0x7fffu) == 0x7c00u) << (8 * j + i);
                    neg |= (unsigned long long)(h >> 15 & 1u) << (8 * j + i);
                }
            }
            for (unsigned lanes = __ballot_sync(0xffffffffu, inf != 0); lanes; lanes &= lanes - 1) {
                const int l = __ffs(lanes) - 1;
                const unsigned long long sign = __shfl_sync(0xffffffffu, neg, l);
                for (unsigned long long of = __shfl_sync(0xffffffffu, inf, l); of; of &= of - 1) {
                    const int i = __ffsll((long long)of) - 1, k = k0 + (i >> 3) * 256 + l * 8 + (i & 7);
                    const float xi = sign >> i & 1ull ? -INFINITY : INFINITY;
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (row[r] >= 0) o.v[r] = fmaf(__half2float(s[(size_t)row[r] * nb + k / 32]), (float)q[(size_t)row[r] * in + k] * xi, o.v[r]);
                    bool open = false;
#pragma unroll
                    for (int r = 0; r < R; ++r) open = open || (row[r] >= 0 && o.v[r] == o.v[r]);
                    if (!__any_sync(0xffffffffu, open)) return o;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (row[r] >= 0) {
                const uint4 *sr = reinterpret_cast<const uint4 *>(s + (size_t)row[r] * nb);  // eight scales each
                for (int c = 0; c < nb / 8; ++c) {
                    const uint4 v = sr[c];
                    const unsigned w[4] = {v.x, v.y, v.z, v.w};
                    bool odd = false;
#pragma unroll
                    for (int i = 0; i < 4; ++i) odd = odd || (w[i] & 0x7c00u) == 0x7c00u || (w[i] & 0x7c000000u) == 0x7c000000u;
                    for (int b = 8 * c; odd && b < 8 * c + 8; ++b) {
                        const float sc = __half2float(s[(size_t)row[r] * nb + b]);
                        if (fabsf(sc) < INFINITY) continue;
                        float d = 0.f;
                        for (int i = 32 * b; i < 32 * b + 32; ++i) d = fmaf((float)q[(size_t)row[r] * in + i], __half2float(x[i]), d);
                        o.v[r] = fmaf(sc, d, o.v[r]);
                    }
                }
            }
        return o;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        for (unsigned lanes = __ballot_sync(0xffffffffu, row[r] >= 0); lanes; lanes &= lanes - 1) {
            const int l = __ffs(lanes) - 1;
            const size_t at = (size_t)__shfl_sync(0xffffffffu, row[r], l);
            float sum = 0.f;
            for (int b = lane; b < nb; b += 32) {
                float d = 0.f;
                for (int i = 32 * b; i < 32 * b + 32; ++i) d = fmaf((float)q[at * in + i], __half2float(x[i]), d);
                sum = fmaf(__half2float(s[at * nb + b]), d, sum);
            }
#pragma unroll
            for (int k = 16; k; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
            if (lane == l) o.v[r] = sum;
        }
    return o;
}
// (apart from the kernels, whose registers the values leave only when this is called)
template <int CNT>
__device__ __noinline__ int tc_q8_slow(const int8_t *q, const __half *s, const __half *x, int stride_x, int in, int out, bool todo, int n, int row0, int lim0, int row1,
                                       int known, float *v) {
    const int lane = threadIdx.x & 31;
    constexpr int R = CNT == 64 ? 2 : 4;
    unsigned bad[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < CNT; ++i)
        if (!(fabsf(v[i]) < INFINITY) && (i < CNT / 2 ? row0 + i < lim0 : row1 + i - CNT / 2 < out)) bad[i / 32] |= 1u << (i & 31);
#pragma unroll 1
    for (unsigned lanes = __ballot_sync(0xffffffffu, todo); lanes;) {
        const int src = __ffs(lanes) - 1, tok = __shfl_sync(0xffffffffu, n, src);
        const unsigned same = CNT == 64 ? 1u << src : __ballot_sync(0xffffffffu, todo && n == tok);
        lanes &= ~same;
        int row[4] = {-1, -1, -1, -1};
#pragma unroll
        for (int r = 0; r < R; ++r) {  // item 32 r + lane: value i of the m-th of these lanes
            const int m = (32 * r + lane) / CNT, i = (32 * r + lane) % CNT, l = CNT == 64 ? src : m < __popc(same) ? (int)__fns(same, 0, m + 1) : -1, at = l < 0 ? 0 : l;
            const unsigned b0 = __shfl_sync(0xffffffffu, bad[0], at), b1 = __shfl_sync(0xffffffffu, bad[1], at);
            const int f0 = __shfl_sync(0xffffffffu, row0, at), f1 = __shfl_sync(0xffffffffu, row1, at);
            row[r] = l >= 0 && ((i < 32 ? b0 : b1) >> (i & 31) & 1u) ? (i < CNT / 2 ? f0 + i : f1 + i - CNT / 2) : -1;
        }
        const TqRows<R> p = tc_q8_rows<R>(q, s, x + (size_t)tok * stride_x, in, make_int4(row[0], row[1], row[2], row[3]),
                                    __shfl_sync(0xffffffffu, known, src));
        const bool here = same >> lane & 1u;
        if (here) known = p.known;
        if (p.known == TQ_NAN) continue;  // (so are the sums)
        const int first = CNT == 64 ? 0 : __popc(same & ((1u << lane) - 1u)) * CNT;
#pragma unroll
        for (int i = 0; i < CNT; ++i) {
            const int w = first + i;
            float t = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (CNT == 64 && r != i / 32) continue;
                const float got = __shfl_sync(0xffffffffu, p.v[r], w & 31);
                if (CNT == 64 || r == w >> 5) t = got;
            }
            if (here && (bad[i / 32] >> (i & 31) & 1u)) v[i] = t;
        }
    }
    return known;
}
template <int CNT>
__device__ __forceinline__ bool tc_q8_odd(const float *v) {  // whether one of them is not finite
    float z[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < CNT; ++i) z[i & 1] = fmaf(v[i], 0.f, z[i & 1]);  // 0, or NaN
    return z[0] + z[1] != 0.f;
}
// Replaces the sums of token n that are not finite (`mine`: the lane has a token).  v[i]: weight row row0 + i (below lim0), from CNT / 2
// on row1 + i - CNT / 2 (below a.out).  Lanes with the same token (no more than 128 / CNT of them; one of 64) have theirs done together.
// `known` stays with the token.  All lanes of the warp come here.
template <int CNT>
__device__ __forceinline__ void tc_q8_mend(const GemvArgs &a, bool mine, int n, int row0, int lim0, int row1, float *v, int *known) {
    const bool odd = mine && tc_q8_odd<CNT>(v);
    if (!__any_sync(0xffffffffu, odd)) return;
    const int was = mine ? *known : TQ_UNKNOWN;
    float w[CNT];
#pragma unroll
    for (int i = 0; i < CNT; ++i) w[i] = v[i];
    const int now = tc_q8_slow<CNT>(reinterpret_cast<const int8_t *>(a.w), reinterpret_cast<const __half *>(a.w_scales), reinterpret_cast<const __half *>(a.x), a.stride_x, a.in,
                            a.out, odd && was != TQ_NAN, n, row0, lim0, row1, was, w);
    if (mine && now != was) *known = now;
#pragma unroll
    for (int i = 0; i < CNT; ++i) v[i] = w[i];
}

// Vector form of the fused epilogues for one token and 8 consecutive outputs.  Everything a thread reads
// from global memory for its items (residual, rotation table, page number) is fetched by tc_prefetch
// before tc_finish stores anything: outputs may alias inputs (the residual is updated in place), so the
// compiler cannot hoist those loads itself, and a chain of dependent round trips per item is what made
// the scalar form slow.  Every access is 16 bytes.
//   STORE / RESIDUAL / ROPE_KV: v[0..7] = 8 consecutive rows;  SWIGLU: v = gate, u = up of 8 pairs
struct TcPre {
    uint4 res;
    float4 sn, cs;
    uint32_t p;
    int page;
};

template <class T>
__device__ __forceinline__ void tc_prefetch(const GemvArgs &a, int n, int first, TcPre &pre) {
    if (a.epilogue == EPI_RESIDUAL) {
        pre.res = *reinterpret_cast<const uint4 *>(reinterpret_cast<const T *>(a.res) + (size_t)n * a.stride_res + first);
    } else if (a.epilogue == EPI_ROPE_KV) {
        const int sect = first < a.qd ? 0 : (first < a.qd + a.kvd ? 1 : 2);
        const int rr = first - (sect == 0 ? 0 : (sect == 1 ? a.qd : a.qd + a.kvd));
        const int e = rr % a.dh;
        pre.p = a.pos[n];
        if (sect < 2) {
            const size_t ti = (size_t)pre.p * (a.dh >> 1) + (e >> 1);
            pre.sn = *reinterpret_cast<const float4 *>(a.sin_t + ti);
            pre.cs = *reinterpret_cast<const float4 *>(a.cos_t + ti);
        }
        if (sect > 0) pre.page = a.page_table[(size_t)a.tok_seq[n] * a.pt_stride + (pre.p >> a.geom.page_shift)];
    }
}

template <class T>
__device__ __forceinline__ void tc_finish(const GemvArgs &a, int n, int first, float v[8], const float u[8], const TcPre &pre) {
    T *dst = reinterpret_cast<T *>(a.y) + (size_t)n * a.stride_y + first;
    if (a.epilogue == EPI_SWIGLU) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = swiglu_act(round_act<T>(v[i]), round_act<T>(u[i]));
    } else if (a.epilogue == EPI_RESIDUAL) {
        const uint32_t rw[4] = {pre.res.x, pre.res.y, pre.res.z, pre.res.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 rf = Act<T>::to_f2(rw[i]);
            v[2 * i] += rf.x;
            v[2 * i + 1] += rf.y;
        }
    } else if (a.epilogue == EPI_ROPE_KV) {
        const int sect = first < a.qd ? 0 : (first < a.qd + a.kvd ? 1 : 2);
        const int rr = first - (sect == 0 ? 0 : (sect == 1 ? a.qd : a.qd + a.kvd));
        const int head = rr / a.dh, e = rr - head * a.dh;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = round_act<T>(v[i]);  // the projection is materialised before rope
        if (sect < 2) {
            const float sn[4] = {pre.sn.x, pre.sn.y, pre.sn.z, pre.sn.w}, cs[4] = {pre.cs.x, pre.cs.y, pre.cs.z, pre.cs.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float xa = v[2 * i], xb = v[2 * i + 1];
                v[2 * i] = xa * cs[i] - xb * sn[i];
                v[2 * i + 1] = xa * sn[i] + xb * cs[i];
            }
        }
        if (sect > 0) {
            const int slot = pre.p & (a.geom.page_tokens - 1);
            dst = reinterpret_cast<T *>(a.kv_pool) + a.geom.block_off(pre.page, a.layer, sect - 1, head) + (size_t)slot * a.dh + e;
        }
    }
    if (a.epilogue >= EPI_CAP)
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = cap_logit(v[i], a.cap);
    if (a.epilogue == EPI_STORE_F32 || a.epilogue == EPI_CAP_F32) {
        float4 *f = reinterpret_cast<float4 *>(reinterpret_cast<float *>(a.y) + (size_t)n * a.stride_y + first);
        f[0] = make_float4(v[0], v[1], v[2], v[3]);
        f[1] = make_float4(v[4], v[5], v[6], v[7]);
        return;
    }
    if (a.epilogue == EPI_XIELU) {
        const float sp = softplus_f(__ldg(a.act_pq)), sq = softplus_f(__ldg(a.act_pq + 1));
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = xielu_act(v[i], sp, sq);
    }
    if (a.epilogue == EPI_RELU2) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = relu2_act(v[i]);
    }
    if (a.epilogue == EPI_GLU) {
        const float sc = a.row_scale ? a.row_scale[n] : 1.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = glu_act(sc * v[2 * i], sc * v[2 * i + 1], a.glu);
        *reinterpret_cast<uint2 *>(reinterpret_cast<T *>(a.y) + (size_t)n * a.stride_y + first / 2) = make_uint2(Act<T>::pack(v[0], v[1]), Act<T>::pack(v[2], v[3]));
        return;
    }
    uint4 o;
    o.x = Act<T>::pack(v[0], v[1]); o.y = Act<T>::pack(v[2], v[3]); o.z = Act<T>::pack(v[4], v[5]); o.w = Act<T>::pack(v[6], v[7]);
    if (a.push.n && (a.epilogue == EPI_STORE || a.epilogue == EPI_RESIDUAL)) {
        // tensor parallelism: the partial goes to the owner's (scatter form) or every rank's all-reduce slot over peer memory
        if (a.push.scatter_cols) {
            *reinterpret_cast<uint4 *>(reinterpret_cast<T *>(a.push.slot[first / a.push.scatter_cols]) + (size_t)n * a.stride_y + first) = o;
            return;
        }
        for (int k = 0; k < a.push.n; ++k)
            *reinterpret_cast<uint4 *>(reinterpret_cast<T *>(a.push.slot[k]) + (size_t)n * a.stride_y + first) = o;
        return;
    }
    *reinterpret_cast<uint4 *>(dst) = o;
}
#endif  // __CUDACC__

// 2-D map of a row-major [rows, cols] matrix of 16-bit elements; box = 64 columns x box_rows rows, 128-byte swizzle
inline int tc_make_map(CUtensorMap *m, const void *base, int dt, uint64_t rows, uint64_t cols, uint64_t row_stride,
                       uint32_t box_rows) {
    TcEncodeFn fn = tc_encode_fn();
    if (!fn) {
        set_error("gemm_tc: cuTensorMapEncodeTiled is not available");
        return LCU_ERR_CUDA;
    }
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstr[1] = {row_stride * 2};
    cuuint32_t box[2] = {TC_BK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, dt == LCU_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                    const_cast<void *>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("gemm_tc: cuTensorMapEncodeTiled failed with %d (base %p, %llu x %llu, stride %llu)", (int)r, base,
                  (unsigned long long)rows, (unsigned long long)cols, (unsigned long long)row_stride);
        return LCU_ERR_CUDA;
    }
    return LCU_OK;
}

// Q8_0: the bytes in boxes of 128 columns x 64 rows (128-byte swizzle), the scales in boxes of 8 columns x 64 rows
inline int tc_make_q8_maps(CUtensorMap *mq, CUtensorMap *ms, const void *q, const void *scales, uint64_t rows, uint64_t cols) {
    TcEncodeFn fn = tc_encode_fn();
    LCU_REQUIRE(fn, "gemm_tc: cuTensorMapEncodeTiled is not available");
    const cuuint64_t qd[2] = {cols, rows}, qs[1] = {cols}, sd[2] = {cols / 32, rows}, ss[1] = {cols / 16};
    const cuuint32_t qb[2] = {128, 64}, sb[2] = {TQ_K / 32, 64}, es[2] = {1, 1};
    const CUresult r1 = fn(mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(q), qd, qs, qb, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    const CUresult r2 = fn(ms, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(scales), sd, ss, sb, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r1 != CUDA_SUCCESS || r2 != CUDA_SUCCESS) {
        set_error("gemm_tc: cuTensorMapEncodeTiled failed with %d, %d (Q8_0, %llu x %llu)", (int)r1, (int)r2, (unsigned long long)rows, (unsigned long long)cols);
        return LCU_ERR_CUDA;
    }
    return LCU_OK;
}

inline bool tc_vec(const GemvArgs &a) {  // whether the 16-byte epilogues apply
    const bool f32 = a.epilogue == EPI_STORE_F32 || a.epilogue == EPI_CAP_F32;
    bool ok = a.stride_y % (f32 ? 4 : 8) == 0 && ((uintptr_t)a.y % 16) == 0 && (a.epilogue == EPI_SWIGLU ? a.di % 8 == 0 : a.out % 8 == 0);
    if (a.epilogue == EPI_RESIDUAL) ok = ok && a.stride_res % 8 == 0 && ((uintptr_t)a.res % 16) == 0;
    if (a.epilogue == EPI_ROPE_KV)
        ok = ok && a.dh % 8 == 0 && a.qd % 8 == 0 && a.kvd % 8 == 0 && ((uintptr_t)a.kv_pool % 16) == 0 && ((uintptr_t)a.sin_t % 16) == 0 &&
             ((uintptr_t)a.cos_t % 16) == 0;
    return ok;
}

// 256 x up to 256 tiles on pairs of SMs for rounds of many tokens (gemm_pair.cu); the arguments are those of gemm_tc_launch.
bool gemm_pair_takes(const GemvArgs &a);
int gemm_pair_launch(const GemvArgs &a, int dt, cudaStream_t s, bool pdl, uint32_t *status, int pieces);  // pieces: of a sum
int gemm_pair_warm(int dt, bool q8);

}  // namespace lcu
