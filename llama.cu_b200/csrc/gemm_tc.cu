// Batched `Linear` on the 5th-generation tensor cores: tcgen05.mma with TMA-fed shared-memory
// operands and the accumulator in tensor memory (TMEM) — for 9..64 tokens per pass (batched decode
// rounds and prefill chunks), with Q8_0 weights from 3 tokens on.  Same operator as llama.cu/src/op/linear.rs:17-120 (the reference
// calls cuBLAS GemmEx with m = out, n = bucketed token count, k = in).
//
// The GEMM is computed "swapped": D[128 weight rows x N tokens] += W_tile[128 x 64] · X[N x 64]^T,
// so the weight dimension fills the 128-row MMA and the small token block is N (16, 32 or 64; Q8_0 also 48).
//   - warp 0 (as a whole; one elected lane issues): TMA producer — cp.async.bulk.tensor.2d loads of the weight tile (two
//     64-row boxes) and of the activation tile into a ring of stages, 128-byte swizzle,
//     completion on mbarriers.  Each weight byte is read once from HBM;
//   - warp 1 (likewise): MMA issuer — four tcgen05.mma (K = 16 each) per stage, accumulating into
//     TMEM; tcgen05.commit frees the stage and, after the last one, signals the epilogue;
//   - warps 2..5: epilogue — tcgen05.ld of the 128 x N f32 accumulator into registers, staging
//     through shared memory, then the same fused epilogues as the GEMV (gemv_epilogue: store,
//     residual, RoPE + KV append, SwiGLU).  The two rows of a pair sit in one tile (adjacent rows,
//     or 64 gate rows followed by their 64 up rows);
//   - matrices with few rows are split along K across CTAs (grid.y); partial sums go through
//     scratch memory and the last CTA of a row block to arrive adds them in split order.
// Every mbarrier wait is bounded by a wall-clock limit: on expiry the kernel records a status bit,
// skips the remaining work, waits for its own copies and MMAs, frees its TMEM and returns.
#include <cstdlib>
#include <map>
#include <mutex>

#include "gemv.cuh"
#include "tc.cuh"
#include "tc_linear.cuh"

namespace lcu {

constexpr int TC_THREADS = 192;
constexpr int TC_BM = 128;         // weight rows per CTA tile
constexpr int TC_A_BYTES = TC_BM * TC_BK * 2;

constexpr int TC_MAX_STAGES = 12;
constexpr int TC_LONG = 32;        // K blocks of an accumulator that show: 2048 products err by 2.4e-6, an 80th of f16's rounding

// Q8_0 weights: 8 more warps turn a unit's weights into f16 pairs in tensor memory, from where the MMA takes them as its A operand
// (lane = row); through shared memory they would cost it four times the bytes that HBM delivers.
constexpr int TQ_THREADS = TC_THREADS + 256;
constexpr int TQ_W_BYTES = TC_BM * TQ_K, TQ_S_BYTES = TC_BM * (TQ_K / 32) * 2;
constexpr int TQ_RING = 6, TQ_COL = 128;  // K blocks in tensor memory, the first one's column
template <bool Q8> constexpr int tc_unit_w_bytes() { return Q8 ? TQ_W_BYTES + TQ_S_BYTES : TC_A_BYTES; }
template <bool Q8> __host__ __device__ constexpr int tc_unit_bytes(int N) { return Q8 ? TQ_W_BYTES + TQ_S_BYTES + N * 2 * TQ_K : TC_A_BYTES + N * 128; }

__device__ __forceinline__ void tq_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred e, p;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
                 " @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tq_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

struct TcShared {
    unsigned long long full[TC_MAX_STAGES], empty[TC_MAX_STAGES], tmem_full[2], tmem_empty[2], a_full[TQ_RING], a_empty[TQ_RING], drain;
    uint32_t tmem_base;
    int abort_flag;
    int last;
    int known[64];  // Q8_0: what the tokens' activations hold (tc_q8_mend)
};

// Behind the CTA's last barrier: where a wait has run out, what still writes to its memory ends first.
__device__ __forceinline__ void tc_leave(TcShared *sh, int warp, int issued, int n_stages) {
    if (!sh->abort_flag) return;
    if (warp == 0) tc_warp_drain_ring(tc_smem(&sh->full[0]), issued, n_stages);
    if (warp == 1) {
        tc_warp_commit(tc_smem(&sh->drain));
        tc_warp_drain(tc_smem(&sh->drain), 0u);
    }
    __syncthreads();
}

// Q8_0: the items of a row block that the epilogue left out because their sums are not finite.  A warp has the items that it had there
// (the threads go round together); `part`: the segments' partial sums, where the row block is shared; pairs > 0: items of a row pair.
template <class T>
__device__ __noinline__ void tc_q8_redo(const GemvArgs *args, const float *stg, const float *part, int n_seg, int rb, int N, int pairs, int *known) {
    const GemvArgs &a = *args;
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    const int et = (int)threadIdx.x - 64, chunks = swiglu ? 8 : 16;
    auto sum = [&](int row, int n) {
        if (!part) return stg[row * (N + 1) + n];
        float s = 0.f;
        for (int i = 0; i < n_seg; ++i) s += __ldcg(part + ((size_t)i * N + n) * TC_BM + row);
        return s;
    };
    if (pairs) {
        for (int idx = et; idx < 64 * N; idx += 128) {
            const int j = idx / N, n = idx - j * N, p = rb * 64 + j;
            const bool mine = p < pairs && n < a.n_tok;
            float v[2] = {0.f, 0.f};
            if (mine) { v[0] = sum(swiglu ? j : 2 * j, n); v[1] = sum(swiglu ? 64 + j : 2 * j + 1, n); }
            const bool odd = tc_q8_odd<2>(v);
            tc_q8_mend<2>(a, odd, n, swiglu ? p : 2 * p, a.out, swiglu ? a.di + p : 2 * p + 1, v, known + n);
            if (odd) gemv_epilogue<T>(a, p, n, v[0], v[1]);
        }
        return;
    }
    for (int idx = et; idx < chunks * N; idx += 128) {
        const int c = idx % chunks, n = idx / chunks, first = rb * (8 * chunks) + 8 * c;
        const bool mine = n < a.n_tok && first + 8 <= (swiglu ? a.di : a.out);
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = mine && (i < 8 || swiglu) ? sum(i < 8 ? 8 * c + i : 64 + 8 * c + i - 8, n) : 0.f;
        const bool odd = tc_q8_odd<16>(v);
        if (swiglu) tc_q8_mend<16>(a, odd, n, first, a.di, a.di + first, v, known + n);
        else tc_q8_mend<8>(a, odd, n, first, a.out, first + 4, v, known + n);
        if (!odd) continue;
        TcPre pre;
        tc_prefetch<T>(a, n, first, pre);
        tc_finish<T>(a, n, first, v, v + 8, pre);
    }
}

// Persistent: grid = min(tiles, SMs); a tile is (row block of 128 rows = 64 pairs, K split); CTA c takes
// tiles c, c + grid, ...  The shared-memory ring keeps running across tiles and the accumulator is
// double-buffered in TMEM, so the epilogue of one tile overlaps the loads and MMAs of the next.
// block = 6 warps: TMA producer, MMA issuer, 4 epilogue warps; Q8_0: 8 warps more.
// Q8_0: a unit is 256 K elements of a row block with their scales, in four K blocks of 64.  The converting warps work in two groups
// that take the K blocks in turns (a row per thread) and hand them to the MMA through a ring of six in tensor memory, 64 columns
// each: one group's waits run under the other's arithmetic, which is about 180 cycles a K block against 370 that its bytes take.
// 8B shape, 16 sequences: 5.13 -> 3.87 ms per round against the mma.sync kernel (28672 x 4096 in 34 us, its bytes 20).
template <class T, bool Q8>
__global__ void __launch_bounds__(Q8 ? TQ_THREADS : TC_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ GemvArgs a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_x,
               int n_pairs, int N, int n_stages, int units_per_cta, int max_seg, int vec, uint32_t idesc, float *ws,
               unsigned *tickets, uint32_t *status) {
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment: the 128-byte swizzle pattern repeats every 8 rows = 1024 bytes
    unsigned char *smem = smem_raw + ((1024u - (tc_smem(smem_raw) & 1023u)) & 1023u);
    const int stage_bytes = tc_unit_bytes<Q8>(N);
    float *stg = reinterpret_cast<float *>(smem + (size_t)n_stages * stage_bytes);  // [128][N + 1]
    TcShared *sh = reinterpret_cast<TcShared *>(reinterpret_cast<unsigned char *>(stg) + (size_t)TC_BM * (N + 1) * 4);

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (a.pdl_trigger == 0) grid_dep_launch();
    const int nkb = a.in / (Q8 ? TQ_K : TC_BK);  // K blocks (Q8_0: units) of a whole row block
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    const int acc_cols = N < 32 ? 32 : (N == 48 ? 64 : N);  // TMEM columns of one accumulator
    const int tm_cols = Q8 ? 512 : 2 * acc_cols;            // two accumulators (Q8_0: and the weights)
    const int n_rb = (n_pairs + 63) / 64;
    // work units = (row block, K block) pairs in row-block-major order; this CTA owns a contiguous range and
    // walks it as segments that end at row-block boundaries (stream-K)
    const int total_units = n_rb * nkb;
    const int u_begin = min(total_units, (int)blockIdx.x * units_per_cta);
    const int u_end = min(total_units, u_begin + units_per_cta);

    if (tid == 0) {
        for (int i = 0; i < n_stages; ++i) {
            tc_mbar_init(tc_smem(&sh->full[i]), 1);
            tc_mbar_init(tc_smem(&sh->empty[i]), Q8 ? 9 : 1);  // Q8_0: the MMAs and the 8 converting warps
        }
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(tc_smem(&sh->tmem_full[i]), 1);
            tc_mbar_init(tc_smem(&sh->tmem_empty[i]), Q8 ? 4 : 1);
        }
        for (int i = 0; Q8 && i < TQ_RING; ++i) {
            tc_mbar_init(tc_smem(&sh->a_full[i]), 4);
            tc_mbar_init(tc_smem(&sh->a_empty[i]), 1);
        }
        tc_mbar_init(tc_smem(&sh->drain), 1);
        sh->abort_flag = 0;
        sh->last = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (Q8 && tid >= 64 && tid < 128) sh->known[tid - 64] = TQ_UNKNOWN;
    if (warp == 1) {  // TMEM allocation is a warp-wide operation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)), "r"(tm_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh->tmem_base;
    int issued = 0;  // stages that warp 0 has requested

    if (warp == 0) {
        // ---------------- TMA producer: units u_begin .. u_end - 1, unit = (row block, K block).  The whole warp runs the loop (one
        // elected lane issues) and places, phases and coordinates run along: the divisions of a lane that works them out for
        // every stage take longer than a stage's bytes (8B shape, f16, 32 sequences: 4.84 -> 4.28 ms per round; 33 tokens of the
        // 1B shape 1.71 -> 1.51 ms, together with the peers' pieces of the cluster form requested at once)
        const int n_units = u_end - u_begin;
        const uint32_t full0 = tc_smem(&sh->full[0]), empty0 = tc_smem(&sh->empty[0]), smem0 = tc_smem(smem);
        const int row_step = swiglu ? 64 : TC_BM, second = swiglu ? a.di : 64;
        auto weights = [&](int slot, int kb, int rb) {
            const uint32_t bar = full0 + 8 * slot, dst = smem0 + (uint32_t)(slot * stage_bytes);
            tc_warp_expect_tx(bar, (uint32_t)stage_bytes);
            if constexpr (Q8) {
#pragma unroll
                for (int i = 0; i < 4; ++i)  // [2 x 128 K][2 x 64 rows], then the scales [2 x 64 rows]
                    tc_warp_tma_2d(dst + i * (TQ_W_BYTES / 4), &map_w, kb * TQ_K + (i >> 1) * 128, (i & 1) * second + rb * row_step, bar);
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    tc_warp_tma_2d(dst + TQ_W_BYTES + i * (TQ_S_BYTES / 2), &map_s, kb * (TQ_K / 32), i * second + rb * row_step, bar);
            } else {
                tc_warp_tma_2d(dst, &map_w, kb * TC_BK, rb * row_step, bar);
                tc_warp_tma_2d(dst + TC_A_BYTES / 2, &map_w, kb * TC_BK, second + rb * row_step, bar);
            }
        };
        auto acts = [&](int slot, int kb) {
            const uint32_t dst = smem0 + (uint32_t)(slot * stage_bytes + tc_unit_w_bytes<Q8>());
            for (int i = 0; i < (Q8 ? 4 : 1); ++i) tc_warp_tma_2d(dst + (uint32_t)(i * N * 128), &map_x, (kb * (Q8 ? 4 : 1) + i) * TC_BK, 0, full0 + 8 * slot);
        };
        // The weights do not depend on the previous kernel: when this launch was allowed to start early
        // (programmatic dependent launch) the first ring of weight tiles is already streaming while the predecessor
        // finishes; the activation tiles of those stages follow once it has.
        const int first = n_units < n_stages ? n_units : n_stages;
        int rb = u_begin / nkb, kb = u_begin - rb * nkb, kb_x = kb;
        for (int j = 0; j < first; ++j) {
            weights(j, kb, rb);
            if (++kb == nkb) { kb = 0; ++rb; }
        }
        grid_dep_wait();
        for (int j = 0; j < first; ++j) {
            acts(j, kb_x);
            if (++kb_x == nkb) kb_x = 0;
        }
        issued = first;
        uint32_t phase = 0;
        for (int j = first, slot = 0; j < n_units; ++j) {  // (only a full ring leaves units over)
            if (!tc_warp_wait(empty0 + 8 * slot, phase, &sh->abort_flag)) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
                break;
            }
            weights(slot, kb, rb);
            acts(slot, kb);
            ++issued;
            if (++kb == nkb) { kb = 0; ++rb; }
            if (++slot == n_stages) { slot = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the whole warp, as above)
        const uint32_t full0 = tc_smem(&sh->full[0]), empty0 = tc_smem(&sh->empty[0]);
        const uint64_t desc0 = tc_desc(tc_smem(smem));
        int slot = 0, ti = 0, kb0 = u_begin % nkb;
        uint32_t phase = 0;
        [[maybe_unused]] int at = 0;  // Q8_0: the ring in tensor memory
        [[maybe_unused]] uint32_t at_phase = 0;
        bool stop = false;
        for (int u = u_begin; u < u_end; ++ti) {
            const int kb1 = Q8 ? kb0 + 1 : min(nkb, kb0 + (u_end - u));  // Q8_0: every unit has an accumulator of its own
            const int ab = ti & 1;
            // the epilogue must have drained this accumulator (two tiles ago)
            if (!tc_warp_wait(tc_smem(&sh->tmem_empty[ab]), ((uint32_t)(ti >> 1) & 1u) ^ 1u, &sh->abort_flag)) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d_tmem = tmem + (uint32_t)(ab * acc_cols);
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!tc_warp_wait(full0 + 8 * slot, phase, &sh->abort_flag)) {
                    if (lane == 0) atomicOr(status, 4u);
                    sh->abort_flag = 1;
                    stop = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t da = desc0 + (uint64_t)((slot * stage_bytes) >> 4);
                if constexpr (Q8) {
                    bool ok = true;
                    for (int b = 0; b < 4; ++b) {
                        ok = tc_warp_wait(tc_smem(&sh->a_full[0]) + 8 * at, at_phase, &sh->abort_flag);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint64_t db = da + (uint64_t)((tc_unit_w_bytes<Q8>() + b * N * 128) >> 4);
                        const uint32_t ta = tmem + TQ_COL + 64 * at;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            tq_mma(d_tmem, ta + 8 * k, db + 2 * k, idesc, kb > kb0 || b > 0 || k > 0);
                            tq_mma(d_tmem, ta + 32 + 8 * k, db + 2 * k, idesc, 1u);
                        }
                        tc_warp_commit(tc_smem(&sh->a_empty[0]) + 8 * at);
                        if (++at == TQ_RING) { at = 0; at_phase ^= 1u; }
                    }
                    if (!ok) {
                        if (lane == 0) atomicOr(status, 4u);
                        sh->abort_flag = 1;
                        stop = true;
                        break;
                    }
                } else {
                    tc_warp_mma4(d_tmem, da, da + (TC_A_BYTES >> 4), idesc, kb > kb0 ? 1u : 0u);
                }
                tc_warp_commit(empty0 + 8 * slot);  // the stage is free once these MMAs have read it
                if (++slot == n_stages) { slot = 0; phase ^= 1u; }
            }
            if (stop) break;                                 // (one that lacks K blocks is never handed over)
            tc_warp_commit(tc_smem(&sh->tmem_full[ab]));     // accumulator complete
            u += kb1 - kb0;
            kb0 = Q8 && kb1 < nkb ? kb1 : 0;
        }
    } else if (Q8 && warp >= TC_THREADS / 32) {
        // ---------------- Q8_0: a thread turns a row's 64 K elements (two quantisation blocks) into f16 pairs
        if constexpr (Q8) {
            const int q = warp & 3, grp = (warp - TC_THREADS / 32) >> 2, row = q * 32 + lane;  // a warp may only touch TMEM lanes [32 q, 32 q + 32)
            const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + TQ_COL;
            int slot = 0, at = grp;  // this group's places: grp, grp + 2, grp + 4
            uint32_t phase = 0, at_phase = 1;
            bool ok = true;
            for (int u = u_begin; u < u_end && ok; ++u) {
                ok = tc_warp_wait(tc_smem(&sh->full[0]) + 8 * slot, phase, &sh->abort_flag);
                if (!ok) break;
                const unsigned char *unit = smem + (size_t)slot * stage_bytes;
                const uint4 sc = *reinterpret_cast<const uint4 *>(unit + TQ_W_BYTES + row * 16);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t sw = i ? (grp ? sc.w : sc.z) : (grp ? sc.y : sc.x);
                    const unsigned char *line = unit + i * (TQ_W_BYTES / 2) + row * 128;  // 128-byte swizzle
                    uint4 raw[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) raw[c] = *reinterpret_cast<const uint4 *>(line + (((grp * 4 + c) ^ (row & 7)) << 4));
                    ok = tc_warp_wait(tc_smem(&sh->a_empty[0]) + 8 * at, at_phase, &sh->abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const __half2 pair = *reinterpret_cast<const __half2 *>(&sw);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t hi[16], lo[16];
                        const __half2 s2 = h ? __high2half2(pair) : __low2half2(pair);
                        tc_q8_split(raw[2 * h], s2, hi, lo);
                        tc_q8_split(raw[2 * h + 1], s2, hi + 8, lo + 8);
                        tq_st16(ta + 64 * at + 16 * h, hi);
                        tq_st16(ta + 64 * at + 32 + 16 * h, lo);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&sh->a_full[0]) + 8 * at) : "memory");
                        if (i == 1) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&sh->empty[0]) + 8 * slot) : "memory");
                    }
                    at += 2;
                    if (at >= TQ_RING) { at = grp; at_phase ^= 1u; }
                }
                if (++slot == n_stages) { slot = 0; phase ^= 1u; }
            }
            if (!ok) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
            }
        }
    } else if (warp >= 2) {
        // ---------------- epilogue warps: TMEM -> registers -> shared staging -> fused epilogue
        const int et = tid - 64;
        const int q = warp & 3;                      // a warp may only touch TMEM lanes [32q, 32q + 32)
        const int row = q * 32 + lane;
        int ti = 0;
        [[maybe_unused]] int tu = 0;  // Q8_0: units taken
        for (int u = u_begin; u < u_end; ++ti) {
            const int rb = u / nkb, kb0 = u - rb * nkb;
            const int kb1 = min(nkb, kb0 + (u_end - u));
            u += kb1 - kb0;
            const bool whole = kb0 == 0 && kb1 == nkb;  // this CTA holds the complete sum of the row block
            // otherwise: CTAs first_cta .. last_cta share the row block, in K order
            const int first_cta = (rb * nkb) / units_per_cta, last_cta = (rb * nkb + nkb - 1) / units_per_cta;
            const int n_seg = last_cta - first_cta + 1, seg = (int)blockIdx.x - first_cta;
            const int ab = ti & 1;
            bool ok;
            [[maybe_unused]] float sum[Q8 ? 64 : 1];
            if constexpr (Q8) {
                // the tensor pipe cuts a sum off where it would have to round it, which thousands of products in a row show: units are
                // added up here, rounded
#pragma unroll
                for (int i = 0; i < 64; ++i) sum[i] = 0.f;
                ok = true;
                for (int kb = kb0; kb < kb1 && ok; ++kb, ++tu) {
                    const int ub = tu & 1;
                    ok = __all_sync(0xffffffffu, tc_mbar_wait(tc_smem(&sh->tmem_full[ub]), (uint32_t)(tu >> 1) & 1u, &sh->abort_flag));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int c0 = 0; c0 < 64; c0 += 16)
                        if (c0 < N) {
                            uint32_t r[16];
                            tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ub * acc_cols + c0), r);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 16; ++i) sum[c0 + i] += __uint_as_float(r[i]);
                        }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&sh->tmem_empty[ub])) : "memory");
                }
            } else {
                ok = __all_sync(0xffffffffu, tc_mbar_wait(tc_smem(&sh->tmem_full[ab]), (uint32_t)(ti >> 1) & 1u, &sh->abort_flag));  // (the loads take the whole warp)
            }
            if (!ok) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if constexpr (Q8) {
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (i < N) stg[row * (N + 1) + i] = sum[i];
            } else if (ok) {
                for (int c0 = 0; c0 < N; c0 += 16) {
                    uint32_t r[16];
                    tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ab * acc_cols + c0), r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; ++i) stg[row * (N + 1) + c0 + i] = __uint_as_float(r[i]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            // the barrier also ANDs every thread's `ok`: the 128 epilogue threads leave the loop together or not at
            // all (a thread whose wait ran out must not strand the others at the next barrier)
            uint32_t all_ok;
            asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 2, 128, p;\n selp.u32 %0, 1, 0, q;\n}"
                         : "=r"(all_ok) : "r"((uint32_t)ok) : "memory");
            if (!Q8 && et == 0) {  // the accumulator may be overwritten from here on
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&sh->tmem_empty[ab])) : "memory");
            }
            if (!all_ok) break;
            const int items = 64 * N;
            [[maybe_unused]] bool odd = false;  // Q8_0: items left out, whose sums are not finite
            if (whole && vec) {
                // (token, 8 outputs) items; residual vectors are fetched first, then everything is stored
                const int chunks = swiglu ? 8 : 16;
                TcPre pre[8];
                int cnt = 0;
                for (int idx = et; idx < chunks * N; idx += 128, ++cnt) {
                    int c = idx % chunks, n = idx / chunks;
                    int first = swiglu ? rb * 64 + 8 * c : rb * TC_BM + 8 * c;
                    if (n < a.n_tok && first + 8 <= (swiglu ? a.di : a.out)) tc_prefetch<T>(a, n, first, pre[cnt]);
                }
                cnt = 0;
                for (int idx = et; idx < chunks * N; idx += 128, ++cnt) {
                    int c = idx % chunks, n = idx / chunks;
                    int first = swiglu ? rb * 64 + 8 * c : rb * TC_BM + 8 * c;
                    if (!(n < a.n_tok && first + 8 <= (swiglu ? a.di : a.out))) continue;
                    float v[16];  // 8 outputs (SwiGLU: their gates, then their ups)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        v[i] = stg[(8 * c + i) * (N + 1) + n];
                        v[8 + i] = swiglu ? stg[(64 + 8 * c + i) * (N + 1) + n] : 0.f;
                    }
                    if (Q8 && tc_q8_odd<16>(v)) { odd = true; continue; }
                    tc_finish<T>(a, n, first, v, v + 8, pre[cnt]);
                }
            } else if (whole) {
                for (int idx = et; idx < items; idx += 128) {
                    int j = idx / N, n = idx - j * N;
                    int p = rb * 64 + j;
                    if (p >= n_pairs || n >= a.n_tok) continue;
                    int ra = swiglu ? j : 2 * j, rb2 = swiglu ? 64 + j : 2 * j + 1;
                    float v[2] = {stg[ra * (N + 1) + n], stg[rb2 * (N + 1) + n]};
                    if (Q8 && tc_q8_odd<2>(v)) { odd = true; continue; }
                    gemv_epilogue<T>(a, p, n, v[0], v[1]);
                }
            } else {
                // the row block is shared (the host only cuts row blocks when the vector epilogue applies).  Partial
                // tiles go to scratch token-major, 128 floats per (row block, segment, token); the CTA that takes
                // the last ticket sums them in K order and finishes.
                for (int idx = et; idx < 16 * N; idx += 128) {
                    int c = idx & 15, n = idx >> 4;
                    if (n >= a.n_tok) continue;
                    float4 lo, hi;
                    lo.x = stg[(8 * c + 0) * (N + 1) + n]; lo.y = stg[(8 * c + 1) * (N + 1) + n];
                    lo.z = stg[(8 * c + 2) * (N + 1) + n]; lo.w = stg[(8 * c + 3) * (N + 1) + n];
                    hi.x = stg[(8 * c + 4) * (N + 1) + n]; hi.y = stg[(8 * c + 5) * (N + 1) + n];
                    hi.z = stg[(8 * c + 6) * (N + 1) + n]; hi.w = stg[(8 * c + 7) * (N + 1) + n];
                    float *dst = ws + (((size_t)rb * max_seg + seg) * N + n) * TC_BM + 8 * c;
                    __stcg(reinterpret_cast<float4 *>(dst), lo);
                    __stcg(reinterpret_cast<float4 *>(dst + 4), hi);
                }
                __threadfence();
                asm volatile("bar.sync 2, 128;" ::: "memory");
                if (et == 0) {
                    unsigned ticket = atomicAdd(&tickets[rb], 1u);
                    sh->last = ticket == (unsigned)n_seg - 1;
                    if (sh->last) tickets[rb] = 0;
                }
                asm volatile("bar.sync 2, 128;" ::: "memory");
                if (sh->last) {
                    __threadfence();
                    // Merge of the segments' partial sums.  A partial row lives in the L2 slice of whichever SM wrote
                    // it and one dependent round trip costs more than a microsecond here, so the loads of up to 6
                    // segments (Q8_0, whose threads have fewer registers: 3) for TWO rows of 8 floats are all issued before the
                    // first add, the adds then run in K order.
                    // Measured on a 6-segment merge of a 128 x 32 tile: 11 us with one segment after the other.
                    constexpr int MB = Q8 ? 3 : 6;
                    const size_t seg_stride = (size_t)N * TC_BM;
                    auto merge2 = [&](const float *r0, const float *r1, float o0[8], float o1[8]) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) o0[i] = o1[i] = 0.f;
                        for (int base = 0; base < n_seg; base += MB) {  // (more than 6 CTAs on one row block: small launches only)
                            float4 b0[2 * MB], b1[2 * MB];
#pragma unroll
                            for (int s2 = 0; s2 < MB; ++s2) {
                                if (base + s2 < n_seg) {
                                    const size_t off = (size_t)(base + s2) * seg_stride;
                                    b0[2 * s2] = __ldcg(reinterpret_cast<const float4 *>(r0 + off));
                                    b0[2 * s2 + 1] = __ldcg(reinterpret_cast<const float4 *>(r0 + off + 4));
                                    b1[2 * s2] = __ldcg(reinterpret_cast<const float4 *>(r1 + off));
                                    b1[2 * s2 + 1] = __ldcg(reinterpret_cast<const float4 *>(r1 + off + 4));
                                }
                            }
#pragma unroll
                            for (int s2 = 0; s2 < MB; ++s2) {
                                if (base + s2 < n_seg) {
                                    o0[0] += b0[2 * s2].x; o0[1] += b0[2 * s2].y; o0[2] += b0[2 * s2].z; o0[3] += b0[2 * s2].w;
                                    o0[4] += b0[2 * s2 + 1].x; o0[5] += b0[2 * s2 + 1].y; o0[6] += b0[2 * s2 + 1].z; o0[7] += b0[2 * s2 + 1].w;
                                    o1[0] += b1[2 * s2].x; o1[1] += b1[2 * s2].y; o1[2] += b1[2 * s2].z; o1[3] += b1[2 * s2].w;
                                    o1[4] += b1[2 * s2 + 1].x; o1[5] += b1[2 * s2 + 1].y; o1[6] += b1[2 * s2 + 1].z; o1[7] += b1[2 * s2 + 1].w;
                                }
                            }
                        }
                    };
                    const float *tile0 = ws + (size_t)rb * max_seg * seg_stride;
                    const float zero8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    if (swiglu) {
                        // one item (8 pairs of one token) per pass: its gate row and its up row
                        for (int idx = et; idx < 8 * N; idx += 128) {
                            const int c = idx & 7, n = idx >> 3;
                            const int first = rb * 64 + 8 * c;
                            if (!(n < a.n_tok && first + 8 <= a.di)) continue;
                            float v[16];  // gates, ups
                            const float *r = tile0 + (size_t)n * TC_BM + 8 * c;
                            merge2(r, r + 64, v, v + 8);
                            if (Q8 && tc_q8_odd<16>(v)) { odd = true; continue; }
                            TcPre pre;
                            tc_finish<T>(a, n, first, v, v + 8, pre);
                        }
                    } else {
                        // two items per pass: 8 consecutive rows of token n and of token n + 8 (idx and idx + 128)
                        for (int idx = et; idx < 16 * N; idx += 256) {
                            const int c = idx & 15, n0 = idx >> 4, n1 = n0 + 8;
                            const int first = rb * TC_BM + 8 * c;
                            const bool rows_ok = first + 8 <= a.out;
                            const bool v0 = rows_ok && n0 < a.n_tok, v1 = rows_ok && n1 < a.n_tok && idx + 128 < 16 * N;
                            if (!v0 && !v1) continue;
                            TcPre pre0, pre1;
                            if (v0) tc_prefetch<T>(a, n0, first, pre0);
                            if (v1) tc_prefetch<T>(a, n1, first, pre1);
                            float o0[8], o1[8];
                            const float *r0 = tile0 + (size_t)(v0 ? n0 : n1) * TC_BM + 8 * c;
                            const float *r1 = tile0 + (size_t)(v1 ? n1 : n0) * TC_BM + 8 * c;
                            merge2(r0, r1, o0, o1);
                            const bool odd0 = Q8 && v0 && tc_q8_odd<8>(o0), odd1 = Q8 && v1 && tc_q8_odd<8>(o1);
                            if (v0 && !odd0) tc_finish<T>(a, n0, first, o0, zero8, pre0);
                            if (v1 && !odd1) tc_finish<T>(a, n1, first, o1, zero8, pre1);
                            odd = odd || odd0 || odd1;
                        }
                    }
                }
            }
            if constexpr (Q8)
                if (__any_sync(0xffffffffu, odd))
                    tc_q8_redo<T>(&a, stg, whole ? nullptr : ws + (size_t)rb * max_seg * N * TC_BM, n_seg, rb, N, whole && !vec ? n_pairs : 0, sh->known);
            asm volatile("bar.sync 2, 128;" ::: "memory");  // staging buffer is reused by the next tile
        }
    }
    // ---------------- tail: everyone meets, then the allocating warp returns the TMEM columns
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    p2p_signal(a.push);  // no-op without tensor parallelism
    __syncthreads();
    tc_leave(sh, warp, issued, n_stages);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tm_cols) : "memory");
    }
}

// ------------------------------------------------------------------ cluster split-K form
// For matrices with fewer row blocks than SMs.  The KS CTAs that share a row block form a thread-block cluster
// (consecutive blockIdx.x): each accumulates its K range in TMEM, stages the partial tile token-major in its own
// shared memory, and after a cluster barrier every CTA sums ITS share of the (token, 8 rows) items over all peers'
// tiles through distributed shared memory (peers in K order, so the result does not depend on timing) and runs the
// fused epilogue for them.  No scratch in global memory, no fence / ticket / reload chain: the hand-over costs two
// cluster barriers and one round of DSMEM loads.  A second cluster barrier keeps every tile alive until all peers
// have read it.  All threads of all CTAs reach both barriers on every path (a timed-out wait only skips work).
constexpr int TCK_LD = TC_BM + 4;  // floats per token row of the staged tile (16-byte aligned, bank-skewed)

__device__ __forceinline__ uint32_t tc_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void tc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 tc_ld_dsmem4(uint32_t local_saddr, uint32_t cta) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local_saddr), "r"(cta));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
    return v;
}

// Token blocks of 128 and 256 (prefill): the MMA takes all N tokens at once (tcgen05 allows N up to 256 columns of
// TMEM per accumulator), so a weight tile is streamed once per 256 tokens instead of once per 64; the epilogue then
// walks the accumulator in passes of NS = 64 tokens through the same staging tile and the same two cluster barriers.
// Rounds of more than 256 tokens put their 256-token blocks on grid.y of ONE launch.
template <class T>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tck_kernel(const GemvArgs a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                int N, int n_stages, int KS, int accs, uint32_t idesc, uint32_t *status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (tc_smem(smem_raw) & 1023u)) & 1023u);
    const int stage_bytes = TC_A_BYTES + N * 128;
    const int NS = N > 64 ? 64 : N;  // tokens per epilogue pass
    float *stg = reinterpret_cast<float *>(smem + (size_t)n_stages * stage_bytes);  // [NS][TCK_LD]
    TcShared *sh = reinterpret_cast<TcShared *>(reinterpret_cast<unsigned char *>(stg) + (size_t)NS * TCK_LD * 4);

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (a.pdl_trigger == 0) grid_dep_launch();
    const int nkb = a.in / TC_BK;
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    const int ks = (int)tc_cluster_rank();
    const int rb = (int)blockIdx.x / KS;
    int tb = (int)blockIdx.y * N, n_end = a.n_tok, wrow = 0;  // first token of this CTA's block, end of the tokens, first weight row
    if (a.tiles) {  // grouped: the table is the predecessor's; every CTA of a cluster has the same tile
        grid_dep_wait();
        const int4 tile = a.tiles[blockIdx.y];
        if (tile.z == 0) return;
        tb = tile.y; n_end = tile.y + tile.z; wrow = tile.x * a.out;
    }
    const int kb0 = (int)((long)ks * nkb / KS), kb1 = (int)((long)(ks + 1) * nkb / KS);
    const int n_units = kb1 - kb0;
    const int acc_cols = N < 32 ? 32 : N, tm_cols = accs * acc_cols, half = accs > 1 ? (n_units + 1) / 2 : n_units;  // K blocks of the first accumulator

    if (tid == 0) {
        for (int i = 0; i < n_stages; ++i) {
            tc_mbar_init(tc_smem(&sh->full[i]), 1);
            tc_mbar_init(tc_smem(&sh->empty[i]), 1);
        }
        tc_mbar_init(tc_smem(&sh->tmem_full[0]), 1);
        tc_mbar_init(tc_smem(&sh->drain), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)), "r"(tm_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh->tmem_base;

    bool ok = true;  // epilogue warps: the accumulator is complete
    int issued = 0;  // stages that warp 0 has requested
    if (warp == 0) {
        // ---------------- TMA producer (weights of the first ring before the dependency wait, whole warp: as in gemm_tc_kernel)
        const uint32_t full0 = tc_smem(&sh->full[0]), empty0 = tc_smem(&sh->empty[0]), smem0 = tc_smem(smem);
        const int row_a = wrow + (swiglu ? rb * 64 : rb * TC_BM), row_b = swiglu ? wrow + a.di + rb * 64 : row_a + 64;
        auto weights = [&](int slot, int kx) {
            const uint32_t bar = full0 + 8 * slot, dst = smem0 + (uint32_t)(slot * stage_bytes);
            tc_warp_expect_tx(bar, (uint32_t)stage_bytes);
            tc_warp_tma_2d(dst, &map_w, kx, row_a, bar);
            tc_warp_tma_2d(dst + TC_A_BYTES / 2, &map_w, kx, row_b, bar);
        };
        auto acts = [&](int slot, int kx) {
            tc_warp_tma_2d(smem0 + (uint32_t)(slot * stage_bytes + TC_A_BYTES), &map_x, kx, tb, full0 + 8 * slot);
        };
        const int first = n_units < n_stages ? n_units : n_stages;
        for (int j = 0; j < first; ++j) weights(j, (kb0 + j) * TC_BK);
        grid_dep_wait();
        for (int j = 0; j < first; ++j) acts(j, (kb0 + j) * TC_BK);
        issued = first;
        uint32_t phase = 0;
        for (int kb = kb0 + first, slot = 0; kb < kb1; ++kb) {
            if (!tc_warp_wait(empty0 + 8 * slot, phase, &sh->abort_flag)) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
                break;
            }
            weights(slot, kb * TC_BK);
            acts(slot, kb * TC_BK);
            ++issued;
            if (++slot == n_stages) { slot = 0; phase ^= 1u; }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer
        const uint32_t full0 = tc_smem(&sh->full[0]), empty0 = tc_smem(&sh->empty[0]);
        const uint64_t desc0 = tc_desc(tc_smem(smem));
        uint32_t phase = 0;
        bool stop = false;
        for (int j = 0, slot = 0; j < n_units; ++j) {
            if (!tc_warp_wait(full0 + 8 * slot, phase, &sh->abort_flag)) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
                stop = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t da = desc0 + (uint64_t)((slot * stage_bytes) >> 4);
            tc_warp_mma4(j < half ? tmem : tmem + acc_cols, da, da + (TC_A_BYTES >> 4), idesc, j > 0 && j != half);
            tc_warp_commit(empty0 + 8 * slot);
            if (++slot == n_stages) { slot = 0; phase ^= 1u; }
        }
        if (!stop) tc_warp_commit(tc_smem(&sh->tmem_full[0]));  // (an accumulator that lacks K blocks is never handed over)
    } else if (warp >= 2) {
        ok = __all_sync(0xffffffffu, tc_mbar_wait(tc_smem(&sh->tmem_full[0]), 0u, &sh->abort_flag));  // (the loads take the whole warp)
        if (!ok) {
            if (lane == 0) atomicOr(status, 4u);
            sh->abort_flag = 1;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }

    // every thread of every CTA of the cluster walks the same number of passes and reaches both barriers of each
    for (int t0 = 0; t0 < N; t0 += NS) {
        if (warp >= 2) {
            // ---------------- accumulator columns [t0, t0 + NS) -> token-major staging tile
            const int q = warp & 3;
            const int row = q * 32 + lane;
            for (int c0 = 0; c0 < NS; c0 += 32) {
                uint32_t r[32];
                const bool more = c0 + 16 < NS;
                if (ok) {
                    const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(t0 + c0);
                    tc_ld16(at, r);
                    if (more) tc_ld16(at + 16, r + 16);
                    if (half < n_units) {
                        uint32_t r2[32];
                        tc_ld16(at + acc_cols, r2);
                        if (more) tc_ld16(at + acc_cols + 16, r2 + 16);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < 16 || more) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(r2[i]));
                    } else {
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    }
                }
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i < 16 || more) stg[(size_t)(c0 + i) * TCK_LD + row] = ok ? __uint_as_float(r[i]) : 0.f;
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        tc_cluster_sync();  // every CTA of the row block has staged its partial tile

        if (warp >= 2 && tb + t0 < n_end) {
            // ---------------- this CTA's share of the items: chunk c of 8 rows (8 pairs for SwiGLU) with c % KS == ks
            const int et = tid - 64;
            const int chunks = swiglu ? 8 : 16;
            const int mine = (chunks - ks + KS - 1) / KS;  // chunks ks, ks + KS, ...
            TcPre pre[8];
            int cnt = 0;
            for (int idx = et; idx < mine * NS; idx += 128, ++cnt) {
                const int c = ks + (idx % mine) * KS, n = tb + t0 + idx / mine;
                const int first = swiglu ? rb * 64 + 8 * c : rb * TC_BM + 8 * c;
                if (n < n_end && first + 8 <= (swiglu ? a.di : a.out)) tc_prefetch<T>(a, n, first, pre[cnt]);
            }
            cnt = 0;
            for (int idx = et; idx < mine * NS; idx += 128, ++cnt) {
                const int c = ks + (idx % mine) * KS, nl = idx / mine, n = tb + t0 + nl;
                const int first = swiglu ? rb * 64 + 8 * c : rb * TC_BM + 8 * c;
                if (!(n < n_end && first + 8 <= (swiglu ? a.di : a.out))) continue;
                float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, u[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                const uint32_t sv = tc_smem(stg + (size_t)nl * TCK_LD + 8 * c);
                // every peer's piece is requested before the first add (a round trip per peer otherwise); the sum runs in K order
                auto sum = [&](uint32_t at, float o[8]) {
                    float4 lo[8], hi[8];
#pragma unroll
                    for (int p = 0; p < 8; ++p)
                        if (p < KS) { lo[p] = tc_ld_dsmem4(at, (uint32_t)p); hi[p] = tc_ld_dsmem4(at + 16, (uint32_t)p); }
#pragma unroll
                    for (int p = 0; p < 8; ++p)
                        if (p < KS) {
                            o[0] += lo[p].x; o[1] += lo[p].y; o[2] += lo[p].z; o[3] += lo[p].w;
                            o[4] += hi[p].x; o[5] += hi[p].y; o[6] += hi[p].z; o[7] += hi[p].w;
                        }
                };
                sum(sv, v);
                if (swiglu) sum(sv + 64 * 4, u);
                tc_finish<T>(a, n, first, v, u, pre[cnt]);
            }
        }
        tc_cluster_sync();  // nobody overwrites or leaves while a peer may still read its tile
    }
    p2p_signal(a.push);  // no-op without tensor parallelism
    __syncthreads();
    tc_leave(sh, warp, issued, n_stages);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tm_cols) : "memory");
    }
}

// ------------------------------------------------------------------ host side

// status word for callers that have no context (the stand-alone operator)
static __device__ uint32_t g_tc_fallback_status;

static thread_local float *g_tc_ws = nullptr;
static thread_local size_t g_tc_ws_bytes = 0;
static thread_local unsigned *g_tc_tickets = nullptr;
static thread_local int g_tc_n_tickets = 0;
static thread_local uint32_t *g_tc_status = nullptr;

void gemm_tc_set_scratch(void *ws, size_t ws_bytes, unsigned *tickets, int n_tickets, uint32_t *status) {
    g_tc_ws = reinterpret_cast<float *>(ws);
    g_tc_ws_bytes = ws_bytes;
    g_tc_tickets = tickets;
    g_tc_n_tickets = n_tickets;
    g_tc_status = status;
}

bool gemm_tc_supported(int in, int w_q8) { return in >= TC_BK && in % (w_q8 ? TQ_K : TC_BK) == 0 && tc_encode_fn() != nullptr; }

template <bool Q8>
static size_t tc_smem_bytes(int N, int stages) {
    return 1024 + (size_t)stages * tc_unit_bytes<Q8>(N) + (size_t)TC_BM * (N + 1) * 4 + sizeof(TcShared) + 64;
}

// Clusters of ks CTAs of the cluster form that run at once on the current device (0: unknown, not possible).
template <class T>
static int tck_clusters(int ks, size_t smem) {
    static std::mutex mu;
    static std::map<std::pair<int, std::pair<int, size_t>>, int> cache;
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(dev, std::make_pair(ks, smem));
    const auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ks);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_tck_kernel<T>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    return cache[key] = n;
}

// Tokens of a launch: the MMA's N.  Q8_0 launches take 64 at most (the ring's units are large).
template <bool Q8>
static int tc_columns(const GemvArgs &a) {
    if (Q8) return a.n_tok <= 16 ? 16 : (a.n_tok <= 32 ? 32 : (a.n_tok <= 48 ? 48 : 64));
    return a.tiles ? a.tile_rows : a.n_tok <= 16 ? 16 : (a.n_tok <= 32 ? 32 : (a.n_tok <= 64 ? 64 : (a.n_tok <= 128 ? 128 : 256)));
}

template <class T, bool Q8>
static int tc_launch_t(const GemvArgs &a, int dt, cudaStream_t s, bool pdl, bool dry) {
    auto kernel = gemm_tc_kernel<T, Q8>;
    const int N = tc_columns<Q8>(a);
    int stages = 8;
    while (stages > 2 && tc_smem_bytes<Q8>(N, stages) > (size_t)227 * 1024) --stages;
    const size_t smem = tc_smem_bytes<Q8>(N, stages);
    static std::mutex mu;
    static std::map<int, uint32_t *> done;  // device -> fallback status word (also marks the attribute as set)
    int dev = 0;
    cudaGetDevice(&dev);
    uint32_t *status = g_tc_status;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = done.find(dev);
        if (it == done.end()) {
            LCU_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            if (!Q8) LCU_CHECK_CUDA(cudaFuncSetAttribute(gemm_tck_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            void *p = nullptr;
            LCU_CHECK_CUDA(cudaGetSymbolAddress(&p, g_tc_fallback_status));
            it = done.emplace(dev, reinterpret_cast<uint32_t *>(p)).first;
        }
        if (!status) status = it->second;
    }
    if (dry) return gemm_pair_warm(dt, Q8);
    // A sum is cut into no fewer pieces than CTAs would fill the GPU with (the tensor pipe's error grows with the products of one
    // accumulator), however few CTAs the launch divides K among: the rest are accumulators of one CTA.  The stand-alone operator,
    // which has no scratch, counts a block of 64 tokens.
    const int row_blocks = (a.out / 2 + 63) / 64, tok_blocks = g_tc_ws ? (a.n_tok + 255) / 256 : 1;
    int pieces = a.tiles ? 1 : sm_count() / (row_blocks * tok_blocks);
    pieces = pieces > 8 ? 8 : pieces < 1 ? 1 : pieces;
    while (pieces > 1 && a.in / TC_BK / pieces < 4) --pieces;
    if (a.in / TC_BK < TC_LONG) pieces = 1;
    if (gemm_pair_takes(a)) return gemm_pair_launch(a, dt, s, pdl, status, pieces);
    const int n_pairs = a.out / 2;
    const int sms = sm_count();
    const uint32_t fmt = dt == LCU_BF16 ? 1u : 0u;
    CUtensorMap mw, ms, mx;
    int rc;
    // 16-byte epilogue accesses need aligned, 8-divisible outputs
    bool vec_ok = a.stride_y % 8 == 0 && ((uintptr_t)a.y % 16) == 0 && (a.epilogue == EPI_SWIGLU ? a.di % 8 == 0 : a.out % 8 == 0);
    if (a.epilogue == EPI_RESIDUAL) vec_ok = vec_ok && a.stride_res % 8 == 0 && ((uintptr_t)a.res % 16) == 0;
    if (a.epilogue == EPI_ROPE_KV)
        vec_ok = vec_ok && a.dh % 8 == 0 && a.qd % 8 == 0 && a.kvd % 8 == 0 && ((uintptr_t)a.kv_pool % 16) == 0 &&
                 ((uintptr_t)a.sin_t % 16) == 0 && ((uintptr_t)a.cos_t % 16) == 0;
    const int vec = vec_ok ? 1 : 0;
    LCU_REQUIRE(vec || a.epilogue < EPI_STORE_F32, "gemm_tc: epilogue %d needs rows of a multiple of 8 outputs", a.epilogue);
    if ((N > 64 && !vec) || (Q8 && a.n_tok > 64)) {
        // the 16-byte epilogue does not apply to this shape, or Q8_0 weights: 64-token passes of the general form
        for (int t0 = 0; t0 < a.n_tok; t0 += 64) {
            GemvArgs b = a;
            b.n_tok = a.n_tok - t0 < 64 ? a.n_tok - t0 : 64;
            b.x = reinterpret_cast<const unsigned char *>(a.x) + (size_t)t0 * a.stride_x * 2;
            b.y = reinterpret_cast<unsigned char *>(a.y) + (size_t)t0 * a.stride_y * 2;  // 16-bit outputs only (f32 ones have the 16-byte epilogue)
            if (a.res) b.res = reinterpret_cast<const unsigned char *>(a.res) + (size_t)t0 * a.stride_res * 2;
            if (a.pos) { b.pos = a.pos + t0; b.tok_seq = a.tok_seq + t0; }
            int rc2 = tc_launch_t<T, Q8>(b, dt, s, pdl, dry);
            if (rc2) return rc2;
        }
        return LCU_OK;
    }
    // ---- weight rows on M (any output shape; row blocks of 128)
    if constexpr (Q8) {
        rc = tc_make_q8_maps(&mw, &ms, a.w, a.w_scales, (uint64_t)a.out, (uint64_t)a.in);
    } else {
        rc = tc_make_map(&mw, a.w, dt, (uint64_t)a.out * (a.tiles ? a.groups : 1), (uint64_t)a.in, (uint64_t)a.in, 64);
        ms = mw;
    }
    if (rc) return rc;
    // the activation map has exactly n_tok rows: the rest of the N-row box is out of bounds and zero-filled
    rc = tc_make_map(&mx, a.x, dt, (uint64_t)a.n_tok, (uint64_t)a.in, (uint64_t)a.stride_x, (uint32_t)N);
    if (rc) return rc;
    // ---- few row blocks: the CTAs of a row block form a cluster and merge through distributed shared memory
    if constexpr (!Q8) {
        // tuning 1: where it costs less than the stream-K split, 2: wherever it applies, 0: never
        const int cluster_mode = tuning().tc_cluster;
        const int n_rb_c = (n_pairs + 63) / 64, nkb_c = a.in / TC_BK;
        const int n_tb = a.tiles ? a.n_tiles : (a.n_tok + N - 1) / N;  // token blocks: more than one for rounds of more than 256 tokens, and tiles
        const int stage_bytes = TC_A_BYTES + N * 128;
        const int NS = N > 64 ? 64 : N;
        const size_t fixed = 1024 + (size_t)NS * TCK_LD * 4 + sizeof(TcShared) + 64;
        int st = (int)(((size_t)227 * 1024 - fixed) / stage_bytes);
        if (st > TC_MAX_STAGES) st = TC_MAX_STAGES;
        // CTAs per row block: a cluster lives in one GPC, so fewer of them fit than SMs / KS, and the ones left over start when the
        // first wave is done (16 clusters of 8: 15 fit, 20 us instead of 8).  Cost in us, from CTAs' own clocks on the 1B and 8B
        // shapes: start and merge of a wave 8, of a stream-K launch 13; a stage 0.25, but no less than the weights' bytes at 6 TB/s.
        // Per round with 33 tokens of the 1B shape 1.51 -> 1.07 ms, 32 sequences of the 8B shape 4.28 -> 4.01 ms.
        const int blocks = n_rb_c * n_tb;
        const double bytes = 2e-6 * (double)a.out * a.in * n_tb / 6.;
        auto cost = [&](double start, double stages) { return start + fmax(0.25 * stages, bytes); };
        int KS = 1;
        double best = 1e30;
        for (int ks = 1; ks <= 8 && (ks == 1 || nkb_c / ks >= 4); ++ks) {
            const int room = ks == 1 ? sms : blocks * ks <= sms ? tck_clusters<T>(ks, fixed + (size_t)st * stage_bytes) : 0;
            if (room <= 0) continue;
            const int waves = (blocks + room - 1) / room;
            const double c = cost(8. * waves, (double)waves * ((nkb_c + ks - 1) / ks));
            if (c < best) { best = c; KS = ks; }
        }
        if (a.tiles) KS = 1;
        // blocks of more than 64 tokens, and tiles, exist in this form only (clusters of one CTA where the matrix has row blocks to spare)
        const bool only = a.tiles || N > 64;
        const bool cluster_on = only || (cluster_mode == 2 && KS >= 2) || (cluster_mode == 1 && best <= cost(13., (double)((blocks * nkb_c + sms - 1) / sms)));
        if (vec && cluster_on) {
            const uint32_t idesc_c = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(n_rb_c * KS, n_tb);
            cfg.blockDim = dim3(TC_THREADS);
            cfg.dynamicSmemBytes = fixed + (size_t)st * stage_bytes;
            cfg.stream = s;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)KS;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = pdl ? 2 : 1;
            LCU_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_tck_kernel<T>, a, mw, mx, N, st, KS, KS < pieces && nkb_c / KS >= TC_LONG ? 2 : 1, idesc_c, status));
            g_linear_last_ctas = n_rb_c * KS * n_tb;
            return LCU_OK;
        }
    }
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
    // Work split (stream-K): the (row block, K block) units are dealt to the SMs in equal contiguous ranges, so
    // the launch is balanced whatever the row-block count; row blocks cut between CTAs are summed through scratch.
    // Without scratch, or when the vector epilogue does not apply, ranges are whole row blocks.
    const int n_rb = (n_pairs + 63) / 64, nkb = a.in / (Q8 ? TQ_K : TC_BK), total = n_rb * nkb;
    int units = (total + sms - 1) / sms;
    if (units < (Q8 ? 2 : 8)) units = Q8 ? 2 : 8;  // at least 8 K blocks (128 KB of weights, Q8_0: 68 KB) per CTA
    // a row block is shared by at most 6 CTAs: the merge loads 6 segments at once, beyond that it walks them one
    // round trip at a time (a [1280 x 8192] projection cut 15 ways took 41 us for 21 MB)
    if (units < (nkb + 4) / 5) units = (nkb + 4) / 5;
    int max_seg = (nkb + units - 1) / units + 1;
    const bool cut = vec && g_tc_ws && g_tc_tickets && n_rb <= g_tc_n_tickets &&
                     (size_t)n_rb * max_seg * N * TC_BM * 4 <= g_tc_ws_bytes;
    if (!cut || units % nkb == 0) {
        units = nkb * ((n_rb + sms - 1) / sms);
        max_seg = 1;
    }
    dim3 grid((total + units - 1) / units);
    LCU_CHECK_CUDA(launch_kernel(kernel, grid, dim3(Q8 ? TQ_THREADS : TC_THREADS), smem, s, pdl, a, mw, ms, mx, n_pairs, N, stages, units, max_seg, vec,
                                 idesc, g_tc_ws, g_tc_tickets, status));
    g_linear_last_ctas = (int)grid.x;
    return LCU_OK;
}

int gemm_tc_launch(const GemvArgs &a, int dt, cudaStream_t s, bool pdl, bool dry) {
    LCU_REQUIRE(a.n_tok >= 1 && a.n_tok <= GEMM_TC_MAX_TOKENS, "gemm_tc: n_tok = %d (1..%d)", a.n_tok, GEMM_TC_MAX_TOKENS);
    LCU_REQUIRE(dry || gemm_tc_supported(a.in, a.w_q8), "gemm_tc: in = %d unsupported", a.in);
    LCU_REQUIRE(a.out > 0 && a.out % 2 == 0, "gemm_tc: out = %d must be even", a.out);
    LCU_REQUIRE(a.prologue == PRO_NONE && !a.x_rows, "gemm_tc: takes prepared activations only");
    LCU_REQUIRE(a.stride_x % 8 == 0, "gemm_tc: x row stride %d must be a multiple of 8 elements", a.stride_x);
    LCU_REQUIRE(dry || (((uintptr_t)a.x | (uintptr_t)a.w) % 16) == 0, "gemm_tc: operands must be 16-byte aligned");
    LCU_REQUIRE(!a.tiles || (a.out % 8 == 0 && (a.tile_rows == 64 || a.tile_rows == 128 || a.tile_rows == 256) && a.n_tiles <= 65535),
                "gemm_tc: groups of %d rows in %d tiles of %d", a.out, a.n_tiles, a.tile_rows);
    if (a.epilogue == EPI_SWIGLU) LCU_REQUIRE(a.out == 2 * a.di, "gemm_tc: swiglu needs out == 2*di");
    if (a.w_q8) {
        LCU_REQUIRE(dt == LCU_F16 && !a.tiles && a.epilogue <= EPI_SWIGLU, "gemm_tc: Q8_0 weights need f16 activations and a LLaMA epilogue");
        LCU_REQUIRE(dry || ((uintptr_t)a.w_scales % 16) == 0, "gemm_tc: operands must be 16-byte aligned");
        return tc_launch_t<__half, true>(a, dt, s, pdl, dry);
    }
    if (dt == LCU_F16) return tc_launch_t<__half, false>(a, dt, s, pdl, dry);
    if (dt == LCU_BF16) return tc_launch_t<__nv_bfloat16, false>(a, dt, s, pdl, dry);
    set_error("gemm_tc: activation dtype %d unsupported", dt);
    return LCU_ERR_INVALID;
}

int gemm_tc_warm(int dt, bool q8) {
    GemvArgs a{};
    a.w_q8 = q8; a.in = 256; a.out = 256; a.n_tok = 16; a.stride_x = 256; a.epilogue = EPI_STORE;
    return gemm_tc_launch(a, dt, nullptr, false, true);
}

}  // namespace lcu
