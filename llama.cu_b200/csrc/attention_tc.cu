// Attention of rounds that hold prompts on the 5th-generation tensor cores (paged cache, causal, grouped heads): the arithmetic
// contract of attention.cu (f32 scores and softmax, probabilities rounded to the activation type, row sums over the rounded values,
// one rounding of the output), but for the exponential: ex2.approx.ftz of scores in powers of two in place of expf, off by 2^-22 and
// zero for subnormal weights, neither of which the rounding of the weights to 16 bits lets through.
//
// A CTA owns a KV head and up to 256 query rows (token, head of the group): two tiles of 128 rows that share every K / V tile of
// 128 positions and take turns on the tensor pipe, one tile's products under the other's softmax:
//   scores   S_t[128 rows x 128 positions] = Q_t K^T     both operands in shared memory, as stored (K-major)
//   output   O_t[128 rows x dh]           += P_t V       P_t in tensor memory, over the columns of S_t; V as stored (MN-major)
// Bound by the exponentials: 16384 a tile at 16 per cycle are 1024 cycles, the products of a tile 512 (dh 64) or 1024 (dh 128).
//   - warp 0: TMA producer, page by page (boxes of 64 columns, 128-byte swizzle); K and V have rings of their own;
//   - warp 1: MMA issuer.  The products of a CTA execute in order, so S_t of the next tile may follow O_t in the columns of P_t, and
//     the commit behind S_t says that O_t is at rest as well;
//   - warps 2..5 and 6..9: softmax of tile 0 and 1, one row per thread: maxima and sums need no exchange.  Weights are relative to the
//     running maximum, as in attention.cu, so that they are rounded alike; O_t is rescaled in tensor memory where a row's moves.
//     (A reference that moves by factors of 2^8 only is no faster and rounds every weight in another place.)
// Measured, the kernel timed alone: 8000 tokens of the 1B shape (dh 64) 1488 -> 456 us, 997 tokens of the 8B shape (dh 128) 85 -> 29 us,
// against mma.sync on 64 rows per CTA; in a round, where its neighbours overlap, it gave 0.94 ms and 47 us a layer.
// Rows past the context are zeroed in the V tile (whatever a page holds there, its weight is zero).  Every wait is bounded: when one
// runs out the CTA records a status bit, waits for its own copies, frees its tensor memory and returns.
#include "attention.cuh"
#include "tc.cuh"

namespace lcu {

constexpr int AT_THREADS = 320;
constexpr int AT_BOX = 128 * 128;      // bytes of [128 rows x 64 columns]
constexpr int AT_MAX_STAGES = 4;

struct AtShared {
    unsigned long long k_full[AT_MAX_STAGES], k_empty[AT_MAX_STAGES], v_full[AT_MAX_STAGES], v_empty[AT_MAX_STAGES];
    unsigned long long q_full, s_full[2], p_ready[2], o_done[2], drain;
    uint32_t tmem_base;
    int abort_flag;
};

template <int DH> constexpr int at_stages() { return DH == 64 ? 4 : 2; }
template <int DH> constexpr size_t at_smem() { return 1024 + (size_t)(DH / 64) * AT_BOX * (2 + 2 * at_stages<DH>()) + sizeof(AtShared); }

__device__ __forceinline__ void at_tma_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
                 " @e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n}"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// A in tensor memory (K = 16: 8 columns), B in shared memory
__device__ __forceinline__ void at_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred e, p;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// MN-major operand, 128-byte swizzle: 64-element pieces AT_BOX bytes apart, groups of 8 rows (the K direction) 1024 bytes apart
__device__ __forceinline__ uint64_t at_desc_mn(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(AT_BOX >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void at_ld32(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
                 "%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
                   "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                   "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void at_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ float at_exp2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// pairs of f32 in one instruction, and the largest of three
__device__ __forceinline__ unsigned long long at_pair(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 at_unpair(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long at_fma2(unsigned long long x, unsigned long long y, unsigned long long z) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ unsigned long long at_add2(unsigned long long x, unsigned long long y) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ float at_max3(float x, float y, float z) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
    return r;
}

// groups: (first token in the round, tokens) of up to 256 / G consecutive tokens of one sequence
template <class T, int DH>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_tc_kernel(const AttnArgs a, const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
               const int2 *__restrict__ groups, int g_shift, uint32_t fmt) {
    constexpr int NB = DH / 64, TILE = NB * AT_BOX, ST = at_stages<DH>();
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (tc_smem(smem_raw) & 1023u)) & 1023u);
    unsigned char *Qs = smem, *Ks = Qs + 2 * TILE, *Vs = Ks + ST * TILE;
    AtShared *sh = reinterpret_cast<AtShared *>(Vs + ST * TILE);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    grid_dep_launch();
    const int hkv = blockIdx.x;
    const int2 grp = groups[gridDim.y - 1 - blockIdx.y];   // the last groups of a prompt have the longest contexts: they start first
    const int per = 128 >> g_shift;                        // tokens of a tile
    const bool two = grp.y > per;
    const int pos0 = (int)a.tok_pos[grp.x], ctx = pos0 + grp.y, seq = a.tok_seq[grp.x];
    const int n_tiles = (ctx + 127) >> 7;

    if (tid == 0) {
        for (int i = 0; i < ST; ++i) {
            tc_mbar_init(tc_smem(&sh->k_full[i]), 1);
            tc_mbar_init(tc_smem(&sh->k_empty[i]), 1);
            tc_mbar_init(tc_smem(&sh->v_full[i]), 1);
            tc_mbar_init(tc_smem(&sh->v_empty[i]), 1);
        }
        tc_mbar_init(tc_smem(&sh->q_full), 1);
        tc_mbar_init(tc_smem(&sh->drain), 1);
        for (int t = 0; t < 2; ++t) {
            tc_mbar_init(tc_smem(&sh->s_full[t]), 1);
            tc_mbar_init(tc_smem(&sh->p_ready[t]), 4);
            tc_mbar_init(tc_smem(&sh->o_done[t]), 1);
        }
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh->tmem_base, tmem_o = tmem + 256;  // S_t in columns 128 t .., O_t behind them
    auto give_up = [&]() {
        if (lane == 0) atomicOr(a.status, 4u);
        sh->abort_flag = 1;
    };
    int k_issued = 0, v_issued = 0;  // stages that warp 0 has requested

    if (warp == 0) {
        // ---------------- TMA producer
        const uint32_t q_bar = tc_smem(&sh->q_full), kf = tc_smem(&sh->k_full[0]), ke = tc_smem(&sh->k_empty[0]), vf = tc_smem(&sh->v_full[0]),
                       ve = tc_smem(&sh->v_empty[0]);
        const int pt = a.geom.page_tokens, ppt = 128 >> a.geom.page_shift;  // pages of a tile
        const int blocks = a.geom.n_layers * 2 * a.geom.nkvh, kb = a.layer * 2 * a.geom.nkvh + hkv, vb = kb + a.geom.nkvh;
        const int32_t *pages = a.page_table + (size_t)seq * a.pt_stride;
        auto page_of = [&](int tile) {  // lane i: page i of the tile
            const int p = tile * 128 + lane * pt;
            return lane < ppt && p < ctx ? pages[p >> a.geom.page_shift] : 0;
        };
        int id = page_of(0);
        grid_dep_wait();
        tc_warp_expect_tx(q_bar, (uint32_t)((two ? 2 : 1) * TILE));
        for (int t = 0; t < (two ? 2 : 1); ++t)
            for (int b = 0; b < NB; ++b)
                at_tma_3d(tc_smem(Qs) + (uint32_t)(t * TILE + b * AT_BOX), &map_q, 64 * b, hkv << g_shift, grp.x + t * per, q_bar);
        auto load = [&](uint32_t dst, uint32_t bar, int n, int block) {
            tc_warp_expect_tx(bar, (uint32_t)(n * pt * 128 * NB));
            for (int i = 0; i < n; ++i) {
                const int z = __shfl_sync(0xffffffffu, id, i) * blocks + block;
                for (int b = 0; b < NB; ++b) at_tma_3d(dst + (uint32_t)(b * AT_BOX + i * pt * 128), &map_kv, 64 * b, 0, z, bar);
            }
        };
        int slot = 0;
        uint32_t phase = 1;
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const int n = min(ppt, (ctx - j * 128 + pt - 1) >> a.geom.page_shift);
            ok = tc_warp_wait(ke + 8 * slot, phase, &sh->abort_flag);
            if (!ok) break;
            load(tc_smem(Ks) + (uint32_t)(slot * TILE), kf + 8 * slot, n, kb);
            ++k_issued;
            ok = tc_warp_wait(ve + 8 * slot, phase, &sh->abort_flag);
            if (!ok) break;
            load(tc_smem(Vs) + (uint32_t)(slot * TILE), vf + 8 * slot, n, vb);
            ++v_issued;
            if (j + 1 < n_tiles) id = page_of(j + 1);
            if (++slot == ST) { slot = 0; phase ^= 1u; }
        }
        if (!ok) give_up();
    } else if (warp == 1) {
        // ---------------- MMA issuer
        const uint32_t id_s = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t id_o = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 16) | ((uint32_t)(DH >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t q0 = tc_desc(tc_smem(Qs)), k0 = tc_desc(tc_smem(Ks)), v0 = at_desc_mn(tc_smem(Vs));
        const uint32_t kf = tc_smem(&sh->k_full[0]), ke = tc_smem(&sh->k_empty[0]), vf = tc_smem(&sh->v_full[0]), ve = tc_smem(&sh->v_empty[0]);
        const uint32_t sf = tc_smem(&sh->s_full[0]), pr = tc_smem(&sh->p_ready[0]), od = tc_smem(&sh->o_done[0]);
        const int nt = two ? 2 : 1;
        auto scores = [&](int t, int slot) {
#pragma unroll
            for (int b = 0; b < NB; ++b)
                tc_warp_mma4(tmem + 128 * t, q0 + (uint64_t)((t * TILE + b * AT_BOX) >> 4), k0 + (uint64_t)((slot * TILE + b * AT_BOX) >> 4), id_s, b > 0);
            tc_warp_commit(sf + 8 * t);
        };
        bool ok = tc_warp_wait(tc_smem(&sh->q_full), 0u, &sh->abort_flag) && tc_warp_wait(kf, 0u, &sh->abort_flag);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int t = 0; t < nt; ++t) scores(t, 0);
            tc_warp_commit(ke);
        }
        int slot = 0;
        uint32_t phase = 0;
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int next = slot + 1 == ST ? 0 : slot + 1;
            const uint32_t next_phase = slot + 1 == ST ? phase ^ 1u : phase;
            ok = tc_warp_wait(vf + 8 * slot, phase, &sh->abort_flag);
            if (ok && j + 1 < n_tiles) ok = tc_warp_wait(kf + 8 * next, next_phase, &sh->abort_flag);
            for (int t = 0; t < nt && ok; ++t) {
                ok = tc_warp_wait(pr + 8 * t, (uint32_t)j & 1u, &sh->abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int k = 0; k < 8; ++k)  // 16 positions: 8 columns of weights, 2 KB of the V tile
                    at_mma_ts(tmem_o + DH * t, tmem + 128 * t + 8 * k, v0 + (uint64_t)((slot * TILE + k * 2048) >> 4), id_o, j > 0 || k > 0);
                if (t == nt - 1) tc_warp_commit(ve + 8 * slot);
                if (j + 1 < n_tiles) {
                    scores(t, next);
                    if (t == nt - 1) tc_warp_commit(ke + 8 * next);
                } else {
                    tc_warp_commit(od + 8 * t);
                }
            }
            slot = next;
            phase = next_phase;
        }
        if (!ok) give_up();
    } else {
        // ---------------- softmax and output of one tile: a row per thread
        const int t = (warp - 2) >> 2, q = warp & 3, row = q * 32 + lane;  // a warp may only touch TMEM lanes [32 q, 32 q + 32)
        if (t == 0 || two) {
            const int tok = t * per + (row >> g_shift);        // of the group
            const int lim = pos0 + min(tok, grp.y - 1);        // last position of the row (rows past the group: of any token, not stored)
            const int lim_tile = pos0 + t * per;               // ... of the tile's first row
            const uint32_t ts = tmem + ((uint32_t)(q * 32) << 16) + 128 * t, to = tmem_o + ((uint32_t)(q * 32) << 16) + DH * t;
            const float scale2 = 1.4426950408889634f / sqrtf((float)DH);  // scores in powers of two
            float ref = -INFINITY, l = 0.f;
            bool ok = true;
            for (int j = 0; j < n_tiles; ++j) {
                const int p0 = j * 128;
                if (t == 0 && p0 + 128 > ctx) {  // V rows past the context
                    const int slot = j % ST;
                    ok = tc_mbar_wait(tc_smem(&sh->v_full[slot]), (uint32_t)(j / ST) & 1u, &sh->abort_flag);
                    uint4 *v = reinterpret_cast<uint4 *>(Vs + (size_t)slot * TILE);
                    for (int i = (ctx - p0) * 8 + (tid - 64); ok && i < 128 * 8; i += 128)
#pragma unroll
                        for (int b = 0; b < NB; ++b) v[b * (AT_BOX / 16) + i] = make_uint4(0, 0, 0, 0);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                ok = ok && tc_mbar_wait(tc_smem(&sh->s_full[t]), (uint32_t)j & 1u, &sh->abort_flag);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t s[128];
#pragma unroll
                for (int c = 0; c < 128; c += 32) at_ld32(ts + c, s + c);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (p0 + 127 > lim_tile) {
#pragma unroll
                    for (int c = 0; c < 128; ++c)
                        if (p0 + c > lim) s[c] = 0xff800000u;
                }
                float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 128; c += 8)
#pragma unroll
                    for (int i = 0; i < 4; ++i) m4[i] = at_max3(m4[i], __uint_as_float(s[c + i]), __uint_as_float(s[c + 4 + i]));
                const float m = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * scale2;
                if (__any_sync(0xffffffffu, m > ref)) {  // (true for the first tile: ref is -inf)
                    const float mn = fmaxf(ref, m), corr = ref == -INFINITY ? 0.f : at_exp2(ref - mn);
                    l *= corr;
                    ref = mn;
                    if (j > 0) {
#pragma unroll 1
                        for (int c = 0; c < DH; c += 16) {
                            uint32_t o[16];
                            tc_ld16(to + c, o);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                            at_st16(to + c, o);
                        }
                    }
                }
                const float sub = ref == -INFINITY ? 0.f : ref;  // a row whose scores are all -inf keeps zero weights
                const unsigned long long mul = at_pair(scale2, scale2), off = at_pair(-sub, -sub);
                unsigned long long l2[2] = {0ull, 0ull};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int c = 32 * h + 2 * i;
                        const float2 x = at_unpair(at_fma2(at_pair(__uint_as_float(s[c]), __uint_as_float(s[c + 1])), mul, off));
                        w[i] = Act<T>::pack(at_exp2(x.x), at_exp2(x.y));
                        const float2 f = Act<T>::to_f2(w[i]);
                        l2[i & 1] = at_add2(l2[i & 1], at_pair(f.x, f.y));
                    }
                    at_st16(ts + 16 * h, w);
                }
                const float2 la = at_unpair(at_add2(l2[0], l2[1]));
                l += la.x + la.y;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&sh->p_ready[t])) : "memory");
            }
            ok = ok && tc_mbar_wait(tc_smem(&sh->o_done[t]), 0u, &sh->abort_flag);
            if (__all_sync(0xffffffffu, ok)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const float inv = 1.f / l;
                T *dst = reinterpret_cast<T *>(a.o) + (size_t)(grp.x + tok) * a.stride_o + (size_t)((hkv << g_shift) + (row & ((1 << g_shift) - 1))) * DH;
#pragma unroll
                for (int c = 0; c < DH; c += 32) {
                    uint32_t o[32];
                    at_ld32(to + c, o);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (tok >= grp.y) continue;
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 u;
                        u.x = Act<T>::pack(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                        u.y = Act<T>::pack(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                        u.z = Act<T>::pack(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                        u.w = Act<T>::pack(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                        *reinterpret_cast<uint4 *>(dst + c + i) = u;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            } else {
                give_up();
            }
        }
    }
    __syncthreads();
    if (sh->abort_flag) {  // a wait has run out: what still writes to the CTA's memory ends first
        if (warp == 0) {
            tc_warp_drain(tc_smem(&sh->q_full), 0u);
            tc_warp_drain_ring(tc_smem(&sh->k_full[0]), k_issued, ST);
            tc_warp_drain_ring(tc_smem(&sh->v_full[0]), v_issued, ST);
        }
        if (warp == 1) {
            tc_warp_commit(tc_smem(&sh->drain));
            tc_warp_drain(tc_smem(&sh->drain), 0u);
        }
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ------------------------------------------------------------------ host side

static int at_map(CUtensorMap *m, int dt, const void *base, const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box) {
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = tc_encode_fn()(m, dt == LCU_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                                      const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    LCU_REQUIRE(r == CUDA_SUCCESS, "attention: cuTensorMapEncodeTiled failed with %d", (int)r);
    return LCU_OK;
}

template <class T, int DH>
static int at_launch(const AttnArgs &a, const void *groups, int n_groups, int dt, cudaStream_t s, bool dry) {
    if (dry) {
        LCU_CHECK_CUDA(cudaFuncSetAttribute(attn_tc_kernel<T, DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)at_smem<DH>()));
        return LCU_OK;
    }
    const int G = a.nh / a.nkvh, gs = G == 8 ? 3 : G == 4 ? 2 : G - 1;
    CUtensorMap mq, mkv;
    const cuuint64_t qd[3] = {(cuuint64_t)DH, (cuuint64_t)a.nh, (cuuint64_t)a.n_tok}, qs[2] = {(cuuint64_t)DH * 2, (cuuint64_t)a.stride_q * 2};
    const cuuint32_t qb[3] = {64, (cuuint32_t)G, (cuuint32_t)(128 / G)};
    int rc = at_map(&mq, dt, a.q, qd, qs, qb);
    if (rc) return rc;
    const cuuint64_t pt = (cuuint64_t)a.geom.page_tokens;
    const cuuint64_t kd[3] = {(cuuint64_t)DH, pt, (cuuint64_t)a.n_pages * a.geom.n_layers * 2 * a.geom.nkvh}, ks[2] = {(cuuint64_t)DH * 2, pt * DH * 2};
    const cuuint32_t kb[3] = {64, (cuuint32_t)pt, 1};
    rc = at_map(&mkv, dt, a.kv_pool, kd, ks, kb);
    if (rc) return rc;
    LCU_CHECK_CUDA(launch_kernel(attn_tc_kernel<T, DH>, dim3(a.nkvh, n_groups), dim3(AT_THREADS), at_smem<DH>(), s, false, a, mq, mkv,
                                 reinterpret_cast<const int2 *>(groups), gs, dt == LCU_BF16 ? 1u : 0u));
    return LCU_OK;
}

int attn_tc_group_tokens(int nh, int nkvh) { return 256 / (nh / nkvh); }

bool attn_tc_takes(const KvGeom &g, int n_pages, const void *pool) {
    // blocks of a page are one coordinate of the map (32 bits); the map's base is 16-byte aligned
    return tuning().attn_tc && tc_encode_fn() && (uintptr_t)pool % 16 == 0 && (unsigned long long)n_pages * g.n_layers * 2 * g.nkvh < (1ull << 31);
}

int attn_tc_launch(const AttnArgs &a, const void *groups_dev, int n_groups, int dt, cudaStream_t s, bool dry) {
    if (n_groups <= 0 && !dry) return LCU_OK;
    LCU_REQUIRE(dry || (a.kv_pool && groups_dev && a.status && n_groups <= 65535 && a.stride_q % 8 == 0 && a.stride_o % 8 == 0 &&
                        ((uintptr_t)a.q | (uintptr_t)a.o) % 16 == 0),
                "attention (tensor-core form): needs the paged cache, groups, a status word and aligned rows");
    if (dt == LCU_F16) return a.dh == 64 ? at_launch<__half, 64>(a, groups_dev, n_groups, dt, s, dry) : at_launch<__half, 128>(a, groups_dev, n_groups, dt, s, dry);
    return a.dh == 64 ? at_launch<__nv_bfloat16, 64>(a, groups_dev, n_groups, dt, s, dry)
                      : at_launch<__nv_bfloat16, 128>(a, groups_dev, n_groups, dt, s, dry);
}

}  // namespace lcu
