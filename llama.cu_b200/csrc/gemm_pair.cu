// `Linear` for rounds of many tokens (llama.cu/src/op/linear.rs:17-120) on pairs of SMs: tcgen05.mma.cta_group::2.
//
// Bound by the tensor pipe from a few hundred tokens on.  A CTA that computes a 128 x 256 tile alone writes 48 KB of operands
// to its shared memory and reads as much for 512 cycles of MMA, which is more than shared memory carries; two CTAs that share
// a 256 x 256 tile hold half of the weights' rows each and feed both tensor cores from them: 32 KB.  Hence:
//   - D[256 tokens x NT weight rows]: CTA r of a pair owns tokens 128 r .. 128 r + 127 (lanes of its TMEM) and loads those
//     rows of x and half of the tile's weight rows.  Tokens on lanes: a thread holds consecutive outputs of one token, so
//     the 16-byte epilogues need no exchange through shared memory (gemm_tc.cu has weights on lanes);
//   - persistent: one pair per two SMs, accumulators double-buffered in TMEM (2 x 256 columns), so the epilogue of a tile runs
//     under the MMAs of the next; tiles in token-major order, so that neighbouring pairs read the same weights from L2;
//   - warp 0 of both CTAs: TMA producer; warp 1 of the even CTA: MMA issuer; warps 2..9: epilogue, two per TMEM quadrant.
// Measured (products alone, weights beyond L2): 28672 x 4096 with 997 tokens 356 -> 195 us (1.20 PFLOP/s), with 8000 tokens 2543 ->
// 1356 us (1.39 PFLOP/s; cuBLAS 1267 us), 4096 x 14336 with 997 tokens 115 -> 104 us, against one CTA per 128 x 256 tile.
// Barriers `full` and `tmem_empty` count in the even CTA; `empty` and `tmem_full` are signalled in both by tcgen05.commit.
// Every mbarrier wait is bounded as in gemm_tc.cu: on expiry a status bit is set and the remaining work is skipped; the pair leaves
// when its copies have landed and its MMAs have ended.
#include <map>
#include <mutex>

#include "gemv.cuh"
#include "tc.cuh"
#include "tc_linear.cuh"

namespace lcu {

constexpr int TP_THREADS = 320, TP_SPAN_THREADS = 576;
// The tensor pipe cuts a sum off where it would have to round it, so the error of a sum grows with the products of one accumulator
// (4096 in a row: 4.9e-6 of the result, 14336: 1.7e-5; f16 rounds by 2e-4).  Where smaller launches divide K among CTAs, so that
// their sums are shorter, this kernel cuts K into as many spans with an accumulator each, which are added up, rounded: two of tiles
// of 128 rows fit into tensor memory side by side; more of them, or of larger tiles, are taken one by one into registers, by twice
// the epilogue warps with 64 sums each (997 tokens of the 8B shape, all in spans of 1024: 14.8 -> 15.1 ms; with 128 sums in half
// of the warps 16.4).
enum { TP_PLAIN, TP_SPANS, TP_Q8 };
constexpr int TP_BM = 128;                       // tokens per CTA
constexpr int TP_A_BYTES = TP_BM * TC_BK * 2;
constexpr int TP_STAGES = 7;
// Q8_0 weights: tiles of 128 weight rows, 64 per CTA.  One more warp fetches their bytes and scales, 256 K elements at a time; eight
// more turn them into pairs of f16 (tc_linear.cuh) and write them to shared memory as two operands, which the tensor pipe multiplies
// one after the other.  Every 256 K elements have an accumulator of their own, and the epilogue warps add these up, rounded: the
// tensor pipe cuts sums off, which thousands of products in a row show.  128 rows and not 256 because a thread then holds 64 sums.
// Bound by shared memory: 88 KB per 64 K elements (x 16, bytes 8, pairs 16 written, x twice and pairs once read) are 690 cycles, the
// MMAs 512; measured 830.  28672 x 4096 with 500 tokens in 170 us (0.69 PFLOP/s, counting each product once), eight passes of the
// mma.sync kernel 1080 us; 500 tokens of the 8B shape 67.7 -> 16.5 ms.
constexpr int TPQ_STAGES = 5, TPQ_GROUPS = 3;
constexpr int TPQ_CONVERT = 320;                          // first converting thread
constexpr int TPQ_THREADS = TPQ_CONVERT + 256 + 32;
constexpr int TPQ_ROWS = 64;                              // weight rows of a CTA
constexpr int TPQ_Q_BYTES = TPQ_ROWS * TQ_K, TPQ_G_BYTES = TPQ_Q_BYTES + TPQ_ROWS * (TQ_K / 32) * 2;
template <int MODE> constexpr int tp_threads() { return MODE == TP_Q8 ? TPQ_THREADS : MODE == TP_SPANS ? TP_SPAN_THREADS : TP_THREADS; }
constexpr int TP_COLS = 256;                     // TMEM columns of one accumulator

struct TpShared {
    unsigned long long full[TP_STAGES], empty[TP_STAGES], tmem_full[2], tmem_empty[2], g_full[TPQ_GROUPS], g_empty[TPQ_GROUPS], drain;
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ uint32_t tp_in_leader(uint32_t saddr) {  // the same place in the shared memory of the pair's even CTA
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(saddr));
    return r;
}
// issued by one lane of a converged warp (tc.cuh)
__device__ __forceinline__ void tp_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
                 " @e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];\n}"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tp_mma4(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(LCU_TC_MMA4("2") ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tp_commit_both(uint32_t bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
                 " @e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ uint32_t tp_add(uint32_t x, uint32_t y) { return __float_as_uint(__uint_as_float(x) + __uint_as_float(y)); }
__device__ __forceinline__ void tp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// waits for arrivals of both CTAs, and for what their threads wrote before them
__device__ __forceinline__ bool tp_wait_both(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    auto attempt = [&]() {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        return __all_sync(0xffffffffu, ok != 0);
    };
    if (attempt()) return true;
    const unsigned long long t0 = tc_ns();
    for (unsigned it = 1;; ++it) {
        if (attempt()) return true;
        if ((it & 255u) == 0 && __any_sync(0xffffffffu, *abort_flag || tc_ns() - t0 > TC_WAIT_NS)) return false;
    }
}

// NT: weight rows of a tile (a multiple of 64; SwiGLU: NT / 2 gate rows, then their NT / 2 up rows)
template <class T, int MODE>
__global__ void __launch_bounds__(tp_threads<MODE>(), 1) __cluster_dims__(2, 1, 1)
gemm_pair_kernel(const GemvArgs a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s, const __grid_constant__ CUtensorMap map_x, int NT,
                 int n_mt, int n_tiles, int span, uint32_t idesc, uint32_t *status) {
    constexpr bool Q8 = MODE == TP_Q8;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (tc_smem(smem_raw) & 1023u)) & 1023u);
    const int half = NT / 2;
    constexpr int STAGES = Q8 ? TPQ_STAGES : TP_STAGES, COPIES = Q8 ? 2 : 1;
    const int SPAN = Q8 ? TQ_K / TC_BK : span;
    const int stage_bytes = TP_A_BYTES + COPIES * half * 128;
    unsigned char *raw = smem + (size_t)STAGES * (TP_A_BYTES + (Q8 ? 2 * TPQ_ROWS : TP_COLS / 2) * 128);  // Q8_0: bytes and scales
    TpShared *sh = reinterpret_cast<TpShared *>(raw + (Q8 ? TPQ_GROUPS * TPQ_G_BYTES : 0));

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (a.pdl_trigger == 0) grid_dep_launch();
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int nkb = a.in / TC_BK;
    const bool swiglu = a.epilogue == EPI_SWIGLU;
    const int step = swiglu ? half : NT;  // outputs of a tile

    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) {
            tc_mbar_init(tc_smem(&sh->full[i]), Q8 ? 5 : 1);  // Q8_0: and a lane of the two converting warps of both CTAs
            tc_mbar_init(tc_smem(&sh->empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(tc_smem(&sh->tmem_full[i]), 1);
            tc_mbar_init(tc_smem(&sh->tmem_empty[i]), MODE == TP_SPANS ? 32 : 16);  // a lane of every epilogue warp of both CTAs
        }
        for (int i = 0; Q8 && i < TPQ_GROUPS; ++i) {
            tc_mbar_init(tc_smem(&sh->g_full[i]), 1);
            tc_mbar_init(tc_smem(&sh->g_empty[i]), 8);
        }
        tc_mbar_init(tc_smem(&sh->drain), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)), "r"(2 * TP_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    tp_cluster_sync();  // the peer's barriers exist
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh->tmem_base;
    int issued = 0;  // stages (warp 0) and groups (the last warp of the Q8_0 form) that this warp has requested

    if (warp == 0) {
        // ---------------- TMA producer of this CTA's operands; their bytes count on the even CTA's barrier.  Places in the ring,
        // phases and coordinates run along: one warp issues everything, and four integer divisions per stage cost more than
        // the stage's MMAs
        const uint32_t full0 = tc_smem(&sh->full[0]), full0_leader = tp_in_leader(full0), smem0 = tc_smem(smem);
        const int w_off = rank == 0 ? 0 : (swiglu ? a.di : half);
        auto weights = [&](int slot, int kx, int nt) {
            if (rank == 0) tc_warp_expect_tx(full0 + 8 * slot, (uint32_t)(2 * (Q8 ? TP_A_BYTES : stage_bytes)));
            if (!Q8) tp_tma_2d(smem0 + (uint32_t)(slot * stage_bytes + TP_A_BYTES), &map_w, kx, nt * step + w_off, full0_leader + 8 * slot);
        };
        auto acts = [&](int slot, int kx, int mt) {
            tp_tma_2d(smem0 + (uint32_t)(slot * stage_bytes), &map_x, kx, (2 * mt + rank) * TP_BM, full0_leader + 8 * slot);
        };
        // the weights do not depend on the previous kernel: the first ring of them (of this CTA's first tile) is requested ahead
        // of the wait
        const int early = nkb < STAGES ? nkb : STAGES;
        int slot = 0;
        uint32_t phase = 1;
        bool primed = false, stop = false;
        for (int tile = pair; tile < n_tiles && !stop; tile += n_pairs) {
            const int nt = tile / n_mt, mt = tile - nt * n_mt;
            int kb = 0;
            if (!primed) {
                for (int j = 0; j < early; ++j) weights(j, j * TC_BK, nt);
                grid_dep_wait();
                for (int j = 0; j < early; ++j) acts(j, j * TC_BK, mt);
                kb = issued = early;
                slot = early == STAGES ? 0 : early;
                phase = early == STAGES ? 0 : 1;
                primed = true;
            }
            for (; kb < nkb; ++kb) {
                if (!tc_warp_wait(tc_smem(&sh->empty[0]) + 8 * slot, phase, &sh->abort_flag)) {
                    if (lane == 0) atomicOr(status, 4u);
                    sh->abort_flag = 1;
                    stop = true;
                    break;
                }
                weights(slot, kb * TC_BK, nt);
                acts(slot, kb * TC_BK, mt);
                ++issued;
                if (++slot == STAGES) { slot = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // ---------------- MMA issuer
            const uint32_t full0 = tc_smem(&sh->full[0]), empty0 = tc_smem(&sh->empty[0]);
            const uint64_t desc0 = tc_desc(tc_smem(smem));
            int ti = 0, slot = 0, kb = 0;  // accumulators taken: one per span
            bool stop = false;
            uint32_t phase = 0;
            const int n_acc = pair < n_tiles ? (n_tiles - pair + n_pairs - 1) / n_pairs * (MODE == TP_PLAIN ? 1 : (nkb + SPAN - 1) / SPAN) : 0;
            for (; ti < n_acc && !stop; ++ti) {
                const int ab = ti & 1;
                if (!tc_warp_wait(tc_smem(&sh->tmem_empty[ab]), ((uint32_t)(ti >> 1) & 1u) ^ 1u, &sh->abort_flag)) {
                    if (lane == 0) atomicOr(status, 4u);
                    sh->abort_flag = 1;
                    stop = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tmem = tmem + (uint32_t)(ab * TP_COLS);
                const int k0 = kb, k1 = Q8 ? kb + SPAN : MODE == TP_PLAIN ? nkb : min(nkb, kb + SPAN);
                const int k2 = MODE == TP_PLAIN && span < nkb ? span : 0;  // from here on in a second accumulator
                for (; kb < k1; ++kb) {
                    if (!(Q8 ? tp_wait_both(full0 + 8 * slot, phase, &sh->abort_flag) : tc_warp_wait(full0 + 8 * slot, phase, &sh->abort_flag))) {
                        if (lane == 0) atomicOr(status, 4u);
                        sh->abort_flag = 1;
                        stop = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = desc0 + (uint64_t)((slot * stage_bytes) >> 4), db = da + (TP_A_BYTES >> 4);
                    tp_mma4(MODE == TP_PLAIN && k2 && kb >= k2 ? d_tmem + NT : d_tmem, da, db, idesc, kb > k0 && (MODE != TP_PLAIN || kb != k2));
                    if (Q8) tp_mma4(d_tmem, da, db + (uint64_t)((half * 128) >> 4), idesc, 1u);
                    tp_commit_both(empty0 + 8 * slot);
                    if (++slot == STAGES) { slot = 0; phase ^= 1u; }
                }
                if (kb == nkb) kb = 0;
                if (!stop) tp_commit_both(tc_smem(&sh->tmem_full[ab]));  // (an accumulator that lacks K blocks is never handed over)
            }
        }
    } else if (Q8 && warp == TPQ_THREADS / 32 - 1) {
        // ---------------- Q8_0: TMA producer of the weights' bytes and scales (no kernel writes them: no dependency wait)
        int slot = 0;
        uint32_t phase = 1;
        bool stop = false;
        for (int tile = pair; tile < n_tiles && !stop; tile += n_pairs) {
            const int row = tile / n_mt * step + (rank == 0 ? 0 : (swiglu ? a.di : half));
            for (int kb = 0; kb < nkb; kb += 4) {
                if (!tc_warp_wait(tc_smem(&sh->g_empty[0]) + 8 * slot, phase, &sh->abort_flag)) {
                    if (lane == 0) atomicOr(status, 4u);
                    sh->abort_flag = 1;
                    stop = true;
                    break;
                }
                const uint32_t bar = tc_smem(&sh->g_full[0]) + 8 * slot, dst = tc_smem(raw) + (uint32_t)(slot * TPQ_G_BYTES);
                tc_warp_expect_tx(bar, (uint32_t)TPQ_G_BYTES);
                tc_warp_tma_2d(dst, &map_w, kb * TC_BK, row, bar);
                tc_warp_tma_2d(dst + TPQ_Q_BYTES / 2, &map_w, kb * TC_BK + 128, row, bar);
                tc_warp_tma_2d(dst + TPQ_Q_BYTES, &map_s, kb * 2, row, bar);
                ++issued;
                if (++slot == TPQ_GROUPS) { slot = 0; phase ^= 1u; }
            }
        }
    } else if (Q8 && warp >= TPQ_CONVERT / 32) {
        // ---------------- Q8_0: the converting warps work in pairs, one stage of a group each (a row per thread): the fence and the
        // hand-over of a stage take longer than its arithmetic, and so they run side by side
        if constexpr (Q8) {
            const int u = (warp - TPQ_CONVERT / 32) >> 1, row = (tid - TPQ_CONVERT) & (TPQ_ROWS - 1);
            const uint32_t empty0 = tc_smem(&sh->empty[0]), full0_leader = tp_in_leader(tc_smem(&sh->full[0]));
            int slot = u, gs = 0;
            uint32_t phase = 1, g_phase = 0;
            bool stop = false;
            for (int tile = pair; tile < n_tiles && !stop; tile += n_pairs)
                for (int kb = 0; kb < nkb; kb += 4) {
                    stop = !tc_warp_wait(tc_smem(&sh->g_full[0]) + 8 * gs, g_phase, &sh->abort_flag);
                    if (stop) break;
                    const unsigned char *group = raw + (size_t)gs * TPQ_G_BYTES;
                    const __half2 pair2 = *reinterpret_cast<const __half2 *>(group + TPQ_Q_BYTES + row * 16 + 4 * u);
                    uint4 q[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        q[c] = *reinterpret_cast<const uint4 *>(group + (u >> 1) * (TPQ_Q_BYTES / 2) + row * 128 + ((((u & 1) * 4 + c) ^ (row & 7)) << 4));
                    stop = !tc_warp_wait(empty0 + 8 * slot, phase, &sh->abort_flag);
                    if (stop) break;
                    unsigned char *line = smem + (size_t)slot * stage_bytes + TP_A_BYTES + row * 128;  // 128-byte swizzle
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t hi[8], lo[8];
                        tc_q8_split(q[c], c >> 1 ? __high2half2(pair2) : __low2half2(pair2), hi, lo);
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int at = ((c * 2 + k) ^ (row & 7)) << 4;
                            *reinterpret_cast<uint4 *>(line + at) = make_uint4(hi[4 * k], hi[4 * k + 1], hi[4 * k + 2], hi[4 * k + 3]);
                            *reinterpret_cast<uint4 *>(line + TPQ_ROWS * 128 + at) = make_uint4(lo[4 * k], lo[4 * k + 1], lo[4 * k + 2], lo[4 * k + 3]);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(full0_leader + 8 * slot) : "memory");
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&sh->g_empty[0]) + 8 * gs) : "memory");
                    }
                    slot += 4;
                    if (slot >= STAGES) { slot -= STAGES; phase ^= 1u; }
                    if (++gs == TPQ_GROUPS) { gs = 0; g_phase ^= 1u; }
                }
            if (stop) {
                if (lane == 0) atomicOr(status, 4u);
                sh->abort_flag = 1;
            }
        }
    } else if (MODE == TP_PLAIN && warp >= 2) {
        // ---------------- epilogue: a thread has one token; the two warps of a quadrant take half of the columns each
        if constexpr (MODE == TP_PLAIN) {
            const int q = warp & 3, h = (warp - 2) >> 2;
            int ti = 0;
            grid_dep_wait();  // residual rows and the round descriptor are earlier kernels'
            for (int tile = pair; tile < n_tiles; tile += n_pairs, ++ti) {
                const int mt = tile % n_mt, nt = tile / n_mt;
                const int ab = ti & 1;
                if (!__all_sync(0xffffffffu, tc_mbar_wait(tc_smem(&sh->tmem_full[ab]), (uint32_t)(ti >> 1) & 1u, &sh->abort_flag))) {  // (the loads take the whole warp)
                    if (lane == 0) atomicOr(status, 4u);
                    sh->abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int n = mt * 2 * TP_BM + rank * TP_BM + q * 32 + lane;
                const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ab * TP_COLS);
                if (swiglu) {
                    for (int c0 = h * (half / 2); c0 < (h + 1) * (half / 2); c0 += 16) {
                        uint32_t g[16], u[16];
                        tc_ld16(acc + (uint32_t)c0, g);
                        tc_ld16(acc + (uint32_t)(half + c0), u);
                        if (span < nkb) {
                            uint32_t g2[16], u2[16];
                            tc_ld16(acc + (uint32_t)(NT + c0), g2);
                            tc_ld16(acc + (uint32_t)(NT + half + c0), u2);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 16; ++i) { g[i] = tp_add(g[i], g2[i]); u[i] = tp_add(u[i], u2[i]); }
                        }
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        TcPre pre;
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int first = nt * step + c0 + 8 * k;
                            if (n >= a.n_tok || first + 8 > a.di) continue;
                            float v[8], w[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) { v[i] = __uint_as_float(g[8 * k + i]); w[i] = __uint_as_float(u[8 * k + i]); }
                            tc_finish<T>(a, n, first, v, w, pre);
                        }
                    }
                } else {
                    for (int c0 = h * half; c0 < (h + 1) * half; c0 += 32) {
                        const int first = nt * step + c0;
                        TcPre pre[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (n < a.n_tok && first + 8 * k + 8 <= a.out) tc_prefetch<T>(a, n, first + 8 * k, pre[k]);
                        uint32_t r[32];
                        tc_ld16(acc + (uint32_t)c0, r);
                        tc_ld16(acc + (uint32_t)(c0 + 16), r + 16);
                        if (span < nkb) {
                            uint32_t r2[32];
                            tc_ld16(acc + (uint32_t)(NT + c0), r2);
                            tc_ld16(acc + (uint32_t)(NT + c0 + 16), r2 + 16);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = tp_add(r[i], r2[i]);
                        }
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (n >= a.n_tok || first + 8 * k + 8 > a.out) continue;
                            float v[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[8 * k + i]);
                            tc_finish<T>(a, n, first + 8 * k, v, v, pre[k]);
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tp_in_leader(tc_smem(&sh->tmem_empty[ab]))) : "memory");
            }
        }
    } else if (warp >= 2) {
        // ---------------- epilogue of spans: a thread has one token; the four warps of a quadrant (Q8_0: two) share the columns and add
        // the spans up.
        // The first half of the sums and the second (SwiGLU: gates and their ups) are `len_a` and `len_b` columns from c_a and c_b on.
        constexpr int COLS = 64, WPQ = Q8 ? 2 : 4;  // most columns of a thread, warps of a quadrant
        const int cols = NT / WPQ;
        const int q = warp & 3, h = (warp - 2) >> 2;
        const int c_a = swiglu ? h * (cols / 2) : h * cols, c_b = swiglu ? half + c_a : c_a + COLS / 2;
        const int len_a = swiglu ? cols / 2 : min(cols, COLS / 2), len_b = cols - len_a;
        int ti = 0;
        [[maybe_unused]] int known = TQ_UNKNOWN, known_n = -1;
        bool ok = true;
        grid_dep_wait();  // residual rows and the round descriptor are earlier kernels'
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int nt = tile / n_mt, mt = tile - nt * n_mt;
            const int n = mt * 2 * TP_BM + rank * TP_BM + q * 32 + lane;
            float sum[COLS];
#pragma unroll
            for (int i = 0; i < COLS; ++i) sum[i] = 0.f;
            for (int kb = 0; kb < nkb && ok; kb += SPAN, ++ti) {
                const int ab = ti & 1;
                ok = __all_sync(0xffffffffu, tc_mbar_wait(tc_smem(&sh->tmem_full[ab]), (uint32_t)(ti >> 1) & 1u, &sh->abort_flag));  // (the loads take the whole warp)
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ab * TP_COLS);
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    const int at = c % (COLS / 2), len = c < COLS / 2 ? len_a : len_b;
                    if (!Q8 && at >= len) continue;
                    uint32_t r[16];
                    if (Q8 || at + 16 <= len) {
                        tc_ld16(acc + (uint32_t)((c < COLS / 2 ? c_a : c_b) + at), r);
                    } else {  // (24 columns)
                        tc_ld8(acc + (uint32_t)((c < COLS / 2 ? c_a : c_b) + at), r);
#pragma unroll
                        for (int i = 8; i < 16; ++i) r[i] = 0u;
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(r[i]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tp_in_leader(tc_smem(&sh->tmem_empty[ab]))) : "memory");
            }
            if (!ok) break;
            const int first = nt * step + c_a;
            if constexpr (Q8) {
                if (n != known_n) { known = TQ_UNKNOWN; known_n = n; }
                tc_q8_mend<COLS>(a, n < a.n_tok, n, first, swiglu ? a.di : a.out, swiglu ? a.di + first : first + COLS / 2, sum, &known);
            }
            if (n >= a.n_tok) continue;
            if (swiglu) {
#pragma unroll
                for (int c = 0; c < COLS / 2; c += 8) {
                    if (c >= len_a || first + c + 8 > a.di) continue;
                    TcPre pre;
                    tc_finish<T>(a, n, first + c, sum + c, sum + COLS / 2 + c, pre);
                }
            } else {  // (c_b follows the first half)
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    if (c >= cols) continue;
                    TcPre pre[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        if (first + c + 8 * k + 8 <= a.out) tc_prefetch<T>(a, n, first + c + 8 * k, pre[k]);
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        if (first + c + 8 * k + 8 <= a.out) tc_finish<T>(a, n, first + c + 8 * k, sum + c + 8 * k, sum + c + 8 * k, pre[k]);
                }
            }
        }
        if (!ok) {
            if (lane == 0) atomicOr(status, 4u);
            sh->abort_flag = 1;
        }
    }
    // ---------------- tail: both CTAs are done with each other's barriers and accumulators
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (sh->abort_flag) {
        // both CTAs' operands count on the even CTA's barriers, and its MMAs read both CTAs' memory: it waits for both
        if (rank == 0 && warp == 0) tc_warp_drain_ring(tc_smem(&sh->full[0]), issued, STAGES);
        if (rank == 0 && warp == 1) {
            tp_commit_both(tc_smem(&sh->drain));
            tc_warp_drain(tc_smem(&sh->drain), 0u);
        }
        if (Q8 && warp == TPQ_THREADS / 32 - 1) tc_warp_drain_ring(tc_smem(&sh->g_full[0]), issued, TPQ_GROUPS);
    }
    tp_cluster_sync();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TP_COLS) : "memory");
    }
}

// ------------------------------------------------------------------ host side

template <bool Q8>
static size_t tp_smem_bytes() { return 1024 + (size_t)(Q8 ? TPQ_STAGES * (TP_A_BYTES + 2 * TPQ_ROWS * 128) + TPQ_GROUPS * TPQ_G_BYTES : TP_STAGES * (TP_A_BYTES + TP_COLS / 2 * 128)) + sizeof(TpShared); }

// Weight rows of a tile: the time of a stage goes with the rows that both operands bring (0.29 us for 256 + 128, 0.43 us for
// 256 + 256), so the fewest rows that the busiest pair loads.
static int tp_tile(int n_mt, int rows, int pairs) {
    int NT = 256, best = 1 << 30;
    for (int nt = 256; nt >= 128; nt -= 64) {
        const int tiles = n_mt * ((rows + nt - 1) / nt);
        const int cost = (tiles + pairs - 1) / pairs * (2 * TP_BM + nt);
        if (cost < best) { best = cost; NT = nt; }
    }
    return NT;
}

bool gemm_pair_takes(const GemvArgs &a) {
    const int min = tuning().tc_pair_min;
    if (min <= 0 || a.n_tok < min || a.tiles || a.push.n || !tc_vec(a)) return false;
    if (min == 1 || a.w_q8) return true;  // (Q8_0 weights have passes of 64 tokens otherwise)
    const int rows = a.epilogue == EPI_SWIGLU ? 2 * a.di : a.out, n_mt = (a.n_tok + 2 * TP_BM - 1) / (2 * TP_BM), pairs = sm_count() / 2;
    const int NT = tp_tile(n_mt, rows, pairs);
    return 2 * n_mt * ((rows + NT - 1) / NT) > pairs;
}

template <class T, int MODE>
static int tp_launch(const GemvArgs &a, int dt, cudaStream_t s, bool pdl, uint32_t *status, bool dry, int pieces) {
    constexpr bool Q8 = MODE == TP_Q8;
    static std::mutex mu;
    static std::map<int, bool> done;
    int dev = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!done[dev]) {
            LCU_CHECK_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tp_smem_bytes<Q8>()));
            done[dev] = true;
        }
    }
    if (dry) return LCU_OK;
    const int pairs = sm_count() / 2;
    const int n_mt = (a.n_tok + 2 * TP_BM - 1) / (2 * TP_BM);
    const int outs = a.epilogue == EPI_SWIGLU ? a.di : a.out, per = a.epilogue == EPI_SWIGLU ? 2 : 1;
    const int NT = Q8 ? 2 * TPQ_ROWS : tp_tile(n_mt, outs * per, pairs);
    const int n_nt = (outs * per + NT - 1) / NT;
    CUtensorMap mw, ms, mx;
    int rc = Q8 ? tc_make_q8_maps(&mw, &ms, a.w, a.w_scales, (uint64_t)a.out, (uint64_t)a.in) : tc_make_map(&mw, a.w, dt, (uint64_t)a.out, (uint64_t)a.in, (uint64_t)a.in, (uint32_t)NT / 2);
    if (!rc) rc = tc_make_map(&mx, a.x, dt, (uint64_t)a.n_tok, (uint64_t)a.in, (uint64_t)a.stride_x, TP_BM);
    if (rc) return rc;
    const uint32_t fmt = dt == LCU_BF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(2 * TP_BM >> 4) << 24);
    const int tiles = n_mt * n_nt, nkb = a.in / TC_BK;
    const int grid = 2 * (tiles < pairs ? tiles : pairs);
    LCU_CHECK_CUDA(launch_kernel(gemm_pair_kernel<T, MODE>, dim3(grid), dim3(tp_threads<MODE>()), tp_smem_bytes<Q8>(), s, pdl, a, mw, Q8 ? ms : mw, mx, NT, n_mt, tiles,
                                 (nkb + pieces - 1) / pieces, idesc, status));
    g_linear_last_ctas = grid;
    return LCU_OK;
}

template <class T>
static int tp_16bit(const GemvArgs &a, int dt, cudaStream_t s, bool pdl, uint32_t *status, bool dry, int pieces) {
    const int rows = a.epilogue == EPI_SWIGLU ? 2 * a.di : a.out, n_mt = (a.n_tok + 2 * TP_BM - 1) / (2 * TP_BM);
    if (dry || pieces <= (tp_tile(n_mt, rows, sm_count() / 2) <= TP_COLS / 2 ? 2 : 1)) {
        const int rc = tp_launch<T, TP_PLAIN>(a, dt, s, pdl, status, dry, pieces);
        if (rc || !dry) return rc;
    }
    return tp_launch<T, TP_SPANS>(a, dt, s, pdl, status, dry, pieces);
}

int gemm_pair_launch(const GemvArgs &a, int dt, cudaStream_t s, bool pdl, uint32_t *status, int pieces) {
    if (a.w_q8) return tp_launch<__half, TP_Q8>(a, dt, s, pdl, status, false, 1);
    return dt == LCU_F16 ? tp_16bit<__half>(a, dt, s, pdl, status, false, pieces) : tp_16bit<__nv_bfloat16>(a, dt, s, pdl, status, false, pieces);
}

int gemm_pair_warm(int dt, bool q8) {
    GemvArgs a{};
    if (q8) return tp_launch<__half, TP_Q8>(a, dt, nullptr, false, nullptr, true, 1);
    return dt == LCU_F16 ? tp_16bit<__half>(a, dt, nullptr, false, nullptr, true, 1) : tp_16bit<__nv_bfloat16>(a, dt, nullptr, false, nullptr, true, 1);
}

}  // namespace lcu
