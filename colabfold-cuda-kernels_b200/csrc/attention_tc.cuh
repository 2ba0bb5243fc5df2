// Token attention on the 5th-generation tensor cores: TO = softmax(q·kᵀ/√48 + L_b)·v ⊙ g.
//
// Item = (head, block of 128 queries, sample). A CTA keeps two items in flight, one per track: a
// track is an independent pipeline with its own shared-memory rings, its own TMEM columns and its own
// group of four softmax warps (one thread per query row), so that the bubbles of one item (its
// prologue and epilogue, the waits inside a chunk) are filled by the other item's arithmetic on the
// same SM sub-partitions. Roles:
//   warps 0 and 10   TMA of track 0 and of track 1: the Q tile of an item (128 x 64
//                        columns of QKVG of which 48 are used); per chunk of 64 keys the K tile and the
//                        transposed V tile from VT into a 3-deep ring (a chunk's tiles are asked for one
//                        chunk ahead and stay until its P·V is done), and the 128 x 64 tile of pair
//                        logits into a 2-deep ring of its own, released with the P that came of it
//   warps 1 and 11   tcgen05.mma of track 0 and of track 1. One wait per chunk: once
//                        the group's P of chunk g is complete, O += P·V of chunk g (128 x 48, K = 64,
//                        P read from TMEM) and S = Q·Kᵀ of chunk g + 2 (128 x 64, K = 48) into the S
//                        buffer that chunk g has just left go out back to back, so S is always a chunk
//                        ahead of the softmax and nothing waits for two hand-overs in a row
//   8 softmax warps      track = warp group; thread = query row: S out of TMEM, + pair logits, online
//                        base-2 softmax, P (bf16) into the track's P columns of TMEM; finally
//                        O / l · gate -> TO. The gate rows come into a per-warp stage by asynchronous
//                        copies while the chunks run, the output rows replace them there and leave by
//                        one TMA store per warp; the completion counters of TO are raised for an item
//                        when that store has landed, under the next item's first chunk.
// O stays in TMEM for the whole item: P·V accumulates over the chunks. The exponentials of a row are
// taken against a reference value that follows the row's running maximum lazily: it moves only when
// a chunk's exponentials add up to more than 2^8 (a warp decides together, since TMEM accesses are
// warp-wide), and then the row's O and sum are rescaled in place and the chunk's exponentials taken again.
// Until then P may reach 2^8 instead of 1, which changes nothing in bf16 or f32 but the exponent.
// Math as the reference's token attention (src/diffusion/attention.cuh:145-249): logits in base 2,
// P rounded to bf16 before P·V, row sums from the unrounded P.
#pragma once

#include "attention.cuh"

namespace cck {

constexpr int kTcKeys = 64;                       // keys per chunk
constexpr int kTcTracks = 2;                      // items in flight per CTA
constexpr int kTcWarps = kWorkWarps / kTcTracks;  // softmax warps per item
constexpr int kTcRows = kTcWarps * 32;            // query rows per item = softmax threads per track
static_assert(kTcRows == kBM, "one softmax thread per row of a 128-row UMMA");
static_assert(kTcWarps == kAttnItemWarps, "the completion counters of TO count the warps of an item");
constexpr int kTcTmaWarp1 = kAuxWarp0, kTcMmaWarp1 = kAuxWarp0 + 1; // the second track's TMA and MMA threads
constexpr int kTcKvStages = 3, kTcBiasStages = 2; // (pair logits: one slot per chunk parity, as S and P)
// The exponentials' reference value trails the running maximum by up to 2^8: an exponential above that makes its
// chunk's sum exceed it too. (So do 64 exponentials of a little over 2^2: the rule sends a chunk round again earlier than
// one on the maximum itself would, and a repeated chunk takes its pass twice. ms per step against the form that
// looked for the maximum of every chunk: 2048 x 1 with flat logits 4.10 -> 3.24, pair logits with a deviation of 6
// 4.10 -> 3.61, one chunk of each row far above the others 4.10 -> 3.73, every chunk far above the one before 4.26 -> 4.14;
// 512 x 5 likewise 2.96 -> 2.41, 2.99 -> 2.62, 3.02 -> 2.71, 3.02 -> 2.71. The older figures are of a kernel without
// the other changes made since.)
constexpr float kTcLazySum = 256.f;
constexpr int kTcKBytes = kTcKeys * 128;          // 8 KB: 64 keys x 64 columns
constexpr int kTcVBytes = kHeadD * 128;           // 6 KB: 48 head dims x 64 keys
constexpr int kTcKvBytes = kTcKBytes + kTcVBytes; // 14 KB
constexpr int kTcBiasBytes = kTcRows * 128;       // 16 KB: 128 queries x 64 keys
constexpr int kTcQBytes = kTcRows * 128;          // 16 KB
// shared memory of a track: [Q][K|V ring][pair-logit ring][gate / output stage] = 102 KB
constexpr int kTcKvOff = kTcQBytes, kTcBiasOff = kTcKvOff + kTcKvStages * kTcKvBytes;
// Per softmax warp, a stage for its 32 rows of the gate and then of TO, dense rows of 96 bytes: the gate
// comes in by asynchronous copies with the lanes side by side in a row, the thread that owns a row
// replaces it by its row of the output, and one TMA store takes the 32 rows away. (Stores by the
// threads themselves held a warp for some 3000 cycles per item, however the lanes were laid out.)
constexpr int kTcOutPitch = kHeadD * 2, kTcOutPieces = kTcOutPitch / 16, kTcOutWarpBytes = 32 * kTcOutPitch;
constexpr int kTcOutOff = kTcBiasOff + kTcBiasStages * kTcBiasBytes;
constexpr int kTcTrackBytes = kTcOutOff + kTcWarps * kTcOutWarpBytes;
static_assert(kTcTracks * kTcTrackBytes <= kScratchBytes, "the attention buffers live in the scratch area");
static_assert(kTcTrackBytes % 1024 == 0 && kTcKvBytes % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
// TMEM columns of a track (the GEMM accumulators are idle in this phase): S0, S1 by chunk parity (64
// each), P0, P1 by chunk parity (32 each: 64 keys as bf16 pairs), O (48 of 64)
constexpr uint32_t kTcTrackCols = 256, kTcS = 0, kTcP = 128, kTcO = 192;
static_assert(kTcTracks * kTcTrackCols <= kTmemCols, "two tracks share the CTA's TMEM");

struct TcTrackBars {
    uint64_t q_full, q_empty;                             // TMA -> MMA; MMA (every Q·Kᵀ of the item done) -> TMA
    uint64_t kv_full[kTcKvStages], kv_empty[kTcKvStages]; // TMA -> MMA; MMA (P·V of the chunk done) -> TMA
    uint64_t s_full[2], p_full[2];                        // MMA (S) and TMA (pair logits) -> softmax; softmax (P stored, O rescaled, pair logits read) -> MMA, TMA
    uint64_t pv_done[2];                                  // MMA (P·V of the chunk done: O is current, for a rescale)
    uint64_t o_full;                                      // MMA (the item's last P·V done) -> softmax
};
// Pipeline positions are counted per track over the whole launch (every role of a track passes the
// same number of items and chunks in a phase), kept here between phases.
struct TcBars {
    TcTrackBars t[kTcTracks];
    uint32_t items[kTcTracks], chunks[kTcTracks];
};
static_assert(kTcBarsOff + sizeof(TcBars) <= kCtlBytes, "the attention barriers outgrew the control block");

__device__ __forceinline__ TcBars* tc_bars() {
    return reinterpret_cast<TcBars*>(smem_base() + kCtlOff + kTcBarsOff);
}
__device__ inline void attn_tc_init() {
    if (threadIdx.x == 0) {
        TcBars* b = tc_bars();
        for (int t = 0; t < kTcTracks; t++) {
            TcTrackBars& tb = b->t[t];
            mbar_init(&tb.q_full, 1), mbar_init(&tb.q_empty, 1);
            for (int i = 0; i < kTcKvStages; i++) {
                mbar_init(&tb.kv_full[i], 1), mbar_init(&tb.kv_empty[i], 1);
            }
            for (int i = 0; i < 2; i++) {
                mbar_init(&tb.s_full[i], 2), mbar_init(&tb.p_full[i], kTcRows), mbar_init(&tb.pv_done[i], 1);
            }
            mbar_init(&tb.o_full, 1);
            b->items[t] = 0, b->chunks[t] = 0;
        }
        fence_mbar_init();
    }
}

// two f32 plus the two bf16 of a word
__device__ __forceinline__ float2 add_bf2(uint32_t w, float2 x) {
    float2 y;
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.bf16 %0, lo, %3;\n\tadd.rn.f32.bf16 %1, hi, %4;\n\t}"
        : "=f"(y.x), "=f"(y.y)
        : "r"(w), "f"(x.x), "f"(x.y));
    return y;
}
// 16 f32 columns of this warp's 32 TMEM lanes, without the wait
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// 8 columns of this warp's 32 TMEM lanes from registers (lane l writes TMEM lane base + l)
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :
                 : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        :
        : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Item it -> (sample, head, block of queries). With barriers around the phase, consecutive items are
// the samples of one (head, block of queries): they share its pair logits. On completion counters
// the items of a sample come together, blocks of queries in order: a sample starts as soon as its
// rows of QKVG are complete, and the rows of TO that a tile of WO reads are complete early.
struct TcItem {
    int s, h, qb;
};
__device__ __forceinline__ TcItem tc_item(int it, int S, int qblocks, bool flow) {
    // (a division by a number known only at run time costs a chain of some hundred cycles, at the
    // start of every item: the multipliers are prepared once)
    const KP& p = kp();
    TcItem i;
    if (flow) {
        const uint32_t u = uint32_t(it) / kHeads, v = div_prepared(u, p.tc_div_qblocks);
        i.s = int(v), i.qb = int(u) - int(v) * qblocks, i.h = it % kHeads;
    } else {
        const uint32_t u = div_prepared(uint32_t(it), p.tc_div_s);
        i.s = it - int(u) * S, i.h = int(u % kHeads), i.qb = int(u / kHeads);
    }
    return i;
}
// The CTA's items of a phase are first, first + grid, ...; track t takes every second one from the
// t-th on. How many that is:
__device__ __forceinline__ int tc_track_items(int first, int items, int t) {
    const int mine = items > first ? int(div_prepared(uint32_t(items - first + int(gridDim.x) - 1), kp().div_grid)) : 0;
    return (mine - t + kTcTracks - 1) / kTcTracks;
}
__device__ __forceinline__ int tc_track_item(int first, int t, int j) {
    return first + (t + kTcTracks * j) * int(gridDim.x);
}
// one phase: all items of this CTA
__device__ CCK_PHASE_FN void token_attention_tc(const Launch& L, Deal& d, int b, unsigned int epoch) {
    const KP& p = kp();
    char* sm = smem_base();
    SmemCtl* ctl = smem_ctl();
    TcBars* bars = tc_bars();
    const int N = p.N, np = p.np, npb = p.npb, S = p.S;
    const int qblocks = cdiv(N, kTcRows), items = kHeads * qblocks * S, chunks = np / kTcKeys;
    const int warp = warp_id(), lane = lane_id(), first = d.first();
    d.advance(items);
    const uint32_t tmem = ctl->tmem_base;
    const bool flow = p.flow;
    const int alt = flow ? int(epoch & 1) : 0; // which of the two buffers holds this block's q, k, v and gates
    const bf16* const qkvg = alt ? p.buf.qkvg2 : p.buf.qkvg;

    if (warp == 0 || warp == kTcTmaWarp1) {
        // ---- TMA producer of one track (the whole warp passes here, one lane issues: ptx.cuh). Issue order:
        // the chunk's pair logits, then K and V of the chunk after it (their slots free up in that order),
        // then, after an item's last chunk, the next item's Q tile (free once every Q·Kᵀ of the item is done).
        const int t = uni(warp != 0);
        const int n = uni(tc_track_items(first, items, t)), nchunks = uni(chunks);
        if (n > 0) {
            const uint32_t el = elect_one();
            const uint64_t policy = l2_policy(S == 1); // the pair logits: one sample reads them once, several meet in L2
            TcTrackBars& B = bars->t[t];
            const uint32_t base = uni(smem_u32(sm + t * kTcTrackBytes)), bar0 = uni(smem_u32(&B));
            auto bar = [&](uint64_t& x) { return bar0 + uint32_t(reinterpret_cast<char*>(&x) - reinterpret_cast<char*>(&B)); };
            const CUtensorMap* mqk = &L.tmap[TM_T_QK + alt];
            const CUtensorMap* mvt = &L.tmap[TM_T_VT + alt];
            const CUtensorMap* mpl = &L.tmap[TM_T_PLG];
            const unsigned int qkvg_done = (epoch + 1) * (unsigned int)(gd_table()[GD_TOK_QKVG].nt * kWorkWarps); // (the counters count on through the launch)
            const uint32_t j0 = uni(bars->items[t]), g0 = uni(bars->chunks[t]);
            const int rows_n = uni(N);
            CCK_TRACE_BEGIN_IF(t, el);
            int ready = -1; // the sample whose rows of QKVG are known to be complete
            // the item whose tiles are being asked for, as map coordinates
            int is = 0, ih = 0, qrow = 0, brow = 0;
            auto set_item = [&](int j) {
                const TcItem ti = tc_item(tc_track_item(first, t, j), S, qblocks, flow);
                is = uni(ti.s), ih = uni(ti.h);
                qrow = is * rows_n + uni(ti.qb) * kTcRows, brow = uni((b * kHeads + ti.h) * npb + ti.qb * kTcRows);
                if (flow && is != ready) {
                    // every column tile of QKVG over the sample's rows (q, k, v and the gate), and over the
                    // next sample's rows that the last chunk of keys reaches into (masked, but read)
                    flow_wait_warp(flow_cnt(p, FC_QKVG), is * N / kBM, (min(is * N + np, S * N) - 1) / kBM, qkvg_done, &ctl->abort);
                    __syncwarp();
                    ready = is;
                }
            };
            auto load_q = [&](uint32_t jg) {
                mbar_wait(&B.q_empty, (jg & 1) ^ 1, &ctl->abort);
                mbar_expect_tx_el(el, bar(B.q_full), kTcQBytes);
                tma_load_2d_el(el, base, mqk, ih * kHeadD, qrow, bar(B.q_full));
                tma_load_2d_el(el, base + kTcQBytes / 2, mqk, ih * kHeadD, qrow + 64, bar(B.q_full));
            };
            uint32_t kst = g0 % kTcKvStages, kpar = (g0 / kTcKvStages) & 1; // the next K|V slot and its phase parity
            auto load_kv = [&](int c) {
                mbar_wait(&B.kv_empty[kst], kpar ^ 1, &ctl->abort);
                const uint32_t ks = base + kTcKvOff + kst * kTcKvBytes, kb = bar(B.kv_full[0]) + 8 * kst;
                mbar_expect_tx_el(el, kb, kTcKvBytes);
                tma_load_2d_el(el, ks, mqk, kTokC + ih * kHeadD, is * rows_n + c * kTcKeys, kb);
                tma_load_2d_el(el, ks + kTcKBytes, mvt, c * kTcKeys, (is * kHeads + ih) * kHeadD, kb);
                if (++kst == kTcKvStages) {
                    kst = 0, kpar ^= 1;
                }
            };
            auto load_bias = [&](int c, int row, uint32_t g) {
                // (the slot's last reader is through when P of the chunk two before is there)
                const uint32_t st = g & 1, bb = bar(B.s_full[0]) + 8 * st;
                mbar_wait(&B.p_full[st], ((g >> 1) & 1) ^ 1, &ctl->abort);
                mbar_expect_tx_el(el, bb, kTcBiasBytes);
                tma_load_2d_hint_el(el, base + kTcBiasOff + st * kTcBiasBytes, mpl, c * kTcKeys, row, bb, policy);
            };
            if (t == 1 && p.attn_skew > 0) { // a test's skew between the pipelines: results must not depend on it
                const long long t0 = clock64();
                while (clock64() - t0 < p.attn_skew + 37 * int(blockIdx.x % 64)) {
                }
                __syncwarp();
            }
            // (one loop over all chunks, so that each of the loads above is there once: this function's loops share an
            // instruction cache, and eight warps of softmax want most of it)
            const int total = n * nchunks;
            int j = 0, c = 0, bias_c = 0, bias_row = 0;
#pragma unroll 1
            for (int i = 0; i <= total; i++) {
                if (i > 0) {
                    load_bias(bias_c, bias_row, g0 + uint32_t(i - 1));
                    CCK_TRACE_EV(0x10 + t, i - 1);
                }
                if (i < total) {
                    if (c == 0) {
                        set_item(j);
                    }
                    load_kv(c);
                    CCK_TRACE_EV(0x12 + t, i);
                    if (c == 0) {
                        load_q(j0 + uint32_t(j));
                    }
                }
                bias_c = c, bias_row = brow;
                if (++c == nchunks) {
                    c = 0, j++;
                }
            }
            CCK_TRACE_END();
        }
    } else if (warp == 1 || warp == kTcMmaWarp1) {
        // ---- MMA issuer of one track (the whole warp, one lane issues). One wait per chunk: when the group's
        // P of chunk i is complete (and with it everybody has read S of chunk i), O (+)= P·V of chunk i and S
        // of chunk i + 2 go out back to back. Everything an MMA needs is prepared: descriptors differ by constants.
        const int t = uni(warp != 1);
        const int n = uni(tc_track_items(first, items, t)), nchunks = uni(chunks), total = n * nchunks;
        if (total > 0) {
            const uint32_t el = elect_one();
            TcTrackBars& B = bars->t[t];
            const uint32_t base = uni(smem_u32(sm + t * kTcTrackBytes)), bar0 = uni(smem_u32(&B));
            auto bar = [&](uint64_t& x) { return bar0 + uint32_t(reinterpret_cast<char*>(&x) - reinterpret_cast<char*>(&B)); };
            const uint32_t tt = uni(tmem) + t * kTcTrackCols;
            const uint32_t idesc_s = umma_idesc_bf16(kTcRows, kTcKeys), idesc_o = umma_idesc_bf16(kTcRows, kHeadD);
            const uint32_t j0 = uni(bars->items[t]), g0 = uni(bars->chunks[t]);
            const uint64_t dq = umma_desc_sw128(base), dk0 = umma_desc_sw128(base + kTcKvOff);
            constexpr uint64_t kStageStep = kTcKvBytes >> 4, kVStep = kTcKBytes >> 4; // in the descriptor's address units
            // the next S to issue: chunk number within the phase, its chunk within the item, its item, its K|V slot
            int qk_i = 0, qk_c = 0, qk_j = 0;
            uint32_t qk_g = g0, qk_st = g0 % kTcKvStages, qk_par = (g0 / kTcKvStages) & 1;
            // S of the next chunk = Q·Kᵀ. Its S buffer was read by the whole group (the caller has seen the
            // group's P of the chunk two before complete, or the phase has just begun).
            auto issue_qk = [&]() {
                if (qk_c == 0) {
                    mbar_wait(&B.q_full, (j0 + uint32_t(qk_j)) & 1, &ctl->abort);
                }
                mbar_wait(&B.kv_full[qk_st], qk_par, &ctl->abort);
                tc_fence_after();
                umma_bf16_k48_el(el, tt + kTcS + (qk_g & 1) * 64, dq, dk0 + qk_st * kStageStep, idesc_s);
                umma_commit_el(el, bar(B.s_full[0]) + 8 * (qk_g & 1));
                qk_i++, qk_g++;
                if (++qk_st == kTcKvStages) {
                    qk_st = 0, qk_par ^= 1;
                }
                if (++qk_c == nchunks) {
                    umma_commit_el(el, bar(B.q_empty)); // every Q·Kᵀ of the item is issued
                    qk_c = 0, qk_j++;
                }
            };
            // S stays two chunks ahead of the softmax. Within the current item the warp waits for what a
            // chunk needs (K lands well ahead); a chunk of the next item goes out ahead only if its Q and K
            // are there already (its sample's rows of QKVG may still be in the making), else when that item starts.
            auto pump = [&](int upto, int item) {
                while (qk_i < upto && qk_i < total) {
                    if (qk_j != item) {
                        const bool ready = mbar_test(&B.kv_full[qk_st], qk_par) && (qk_c != 0 || mbar_test(&B.q_full, (j0 + uint32_t(qk_j)) & 1));
                        if (!uni(int(ready))) {
                            break;
                        }
                    }
                    issue_qk();
                }
            };
            tc_fence_after();
            uint32_t st = g0 % kTcKvStages;
            int j = 0, c = 0;
            CCK_TRACE_BEGIN_IF(2 + t, el);
#pragma unroll 1
            for (int i = 0; i < total; i++) {
                pump(i + 2, j);
                const uint32_t g = g0 + uint32_t(i), bi = g & 1;
                mbar_wait(&B.p_full[bi], (g >> 1) & 1, &ctl->abort);
                tc_fence_after();
                CCK_TRACE_EV(0x20 + t, i);
                umma_bf16_ts_k64_el(el, tt + kTcO, tt + kTcP + bi * 32, dk0 + st * kStageStep + kVStep, idesc_o, c);
                umma_commit_el(el, bar(B.pv_done[0]) + 8 * bi);
                umma_commit_el(el, bar(B.kv_empty[0]) + 8 * st);
                CCK_TRACE_EV(0x22 + t, i);
                if (++st == kTcKvStages) {
                    st = 0;
                }
                if (++c == nchunks) {
                    umma_commit_el(el, bar(B.o_full)); // the item's O is complete
                    c = 0, j++;
                }
            }
            CCK_TRACE_END();
        }
    } else if (warp >= kWorkWarp0 && warp < kAuxWarp0) {
        // ---- softmax: this thread owns one query row of its track's items
        const int t = work_group(), q = work_quarter(), row_in = q * 32 + lane;
        TcTrackBars& B = bars->t[t];
        const char* base = sm + t * kTcTrackBytes;
        char* stage = sm + t * kTcTrackBytes + kTcOutOff + q * kTcOutWarpBytes;
        const uint32_t tt = tmem + t * kTcTrackCols + (uint32_t(q * 32) << 16);
        const float scale = kLog2e / sqrtf(float(kHeadD));
        const float2 scale2 = make_float2(scale, scale);
        const int n = tc_track_items(first, items, t);
        const uint32_t j0 = bars->items[t], g0 = bars->chunks[t];
        uint32_t g = g0;
        // This warp's rows of TO of the item before: one arrival at every block of 128 rows that the
        // item's queries touch, once the TMA store has completed.
        int pend_lo = -1, pend_hi = -1;
        auto publish = [&]() {
            if (lane == 0) {
                bulk_wait_done();
            }
            if (pend_lo >= 0) {
                flow_signal(flow_cnt(p, FC_TO), pend_lo / kBM, pend_hi / kBM);
                pend_lo = -1;
            }
        };
        CCK_TRACE_BEGIN_IF(4 + t, row_in == 0);
#pragma unroll 1
        for (int j = 0; j < n; j++) {
            CCK_TRACE_EV(0x44 + t, j);
            const TcItem ti = tc_item(tc_track_item(first, t, j), S, qblocks, flow);
            const int s = ti.s, h = ti.h, qb = ti.qb;
            const uint32_t jg = j0 + j;
            float m = 0.f, l = 0.f; // the reference value of the row's exponentials, the row sum against it
#pragma unroll 1
            for (int c = 0; c < chunks; c++, g++) {
                const uint32_t bi = g & 1, bpar = (g >> 1) & 1;
                CCK_TRACE_EV(0x30 + t, g - g0);
                mbar_wait(&B.s_full[bi], bpar, &ctl->abort); // the scores and the pair logits (one wait: one that passes costs 90 cycles)
                tc_fence_after();
                CCK_TRACE_EV(0x32 + t, g - g0);
                if (c == 0) {
                    // The warp's rows of the gate, on their way into its stage while the chunks run. (The
                    // TMA thread saw the sample's rows of QKVG complete before it asked for the item's Q
                    // tile, and S of that Q has been seen; the copies read L2, where the other CTAs' stores are.)
                    if (lane == 0) {
                        bulk_wait_read(); // the previous item's store has read the stage
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < kTcOutPieces; i++) {
                        const int pc = i * 32 + lane, r = pc / kTcOutPieces, o = pc % kTcOutPieces;
                        const size_t grow = size_t(s) * N + min(qb * kTcRows + q * 32 + r, N - 1);
                        cp_async16(stage + r * kTcOutPitch + o * 16, qkvg + grow * kQKVG + 3 * kTokC + h * kHeadD + o * 8, true);
                    }
                    cp_async_commit();
                }
                const char* brow = base + kTcBiasOff + bi * kTcBiasBytes + row_in * 128; // the row's 64 pair logits: 8 swizzled 16-byte pieces
                // One pass over the chunk: exponentials of the scores (base 2, pair logits added) against the
                // reference value m, P = 2^(score - m) as bf16 to TMEM (16 keys are 8 columns), and their sum. A
                // warp issues an instruction every two cycles or so, and eight warps of softmax are what
                // the SM has: the pass is as short as it can be. The pair logits are added as they are (a mixed
                // f32 + bf16 addition instead of unpacking), and only an item's first chunk looks for its
                // maximum: later ones take the reference of the chunks before on trust. Where a score has
                // outgrown it by more than 2^8, its exponential alone makes the sum exceed kTcLazySum; the pass is then repeated.
                // The chunk's P buffer held P of chunk g - 2. That chunk's P·V was issued before this chunk's
                // Q·Kᵀ, by the same warp, and the commit behind s_full covers everything issued before it:
                // having seen S, the buffer is free.
                // (rounded once, as the pass rounds score - m: where all logits are masked ones, -1.4e9 with a step of 128, a
                // product rounded by itself could go to the other neighbour and leave an exponential of 2^128)
                auto row_max = [&]() {
                    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll 1
                    for (int hf = 0; hf < 2; hf++) {
                        uint32_t sr[32];
                        tmem_ld32_issue(tt + kTcS + bi * 64 + 32 * hf, sr);
                        tmem_ld_wait(sr);
#pragma unroll
                        for (int jj = 0; jj < 4; jj++) {
                            const uint4 bw = *reinterpret_cast<const uint4*>(brow + (((4 * hf + jj) ^ (row_in & 7)) << 4));
                            const uint32_t w[4] = {bw.x, bw.y, bw.z, bw.w};
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const float2 x = __ffma2_rn(make_float2(__uint_as_float(sr[8 * jj + 2 * k]), __uint_as_float(sr[8 * jj + 2 * k + 1])), scale2,
                                                            make_float2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xFFFF0000u)));
                                mx[k & 1] = max3(mx[k & 1], x.x, x.y);
                            }
                        }
                    }
                    return fmaxf(mx[0], mx[1]);
                };
                if (c == 0) {
                    m = row_max();
                }
                float chunk_l;
                for (;;) {
                    const float2 neg_m = make_float2(-m, -m);
                    float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                    for (int hf = 0; hf < 2; hf++) {
                        uint32_t sr[32];
                        tmem_ld32_issue(tt + kTcS + bi * 64 + 32 * hf, sr);
                        tmem_ld_wait(sr);
#pragma unroll
                        for (int jj = 0; jj < 2; jj++) {
                            uint32_t pk[8];
#pragma unroll
                            for (int q4 = 0; q4 < 2; q4++) {
                                const uint4 bw = *reinterpret_cast<const uint4*>(brow + (((4 * hf + 2 * jj + q4) ^ (row_in & 7)) << 4));
                                const uint32_t w[4] = {bw.x, bw.y, bw.z, bw.w};
#pragma unroll
                                for (int k = 0; k < 4; k++) {
                                    const int i = 16 * jj + 8 * q4 + 2 * k;
                                    const float2 x = add_bf2(w[k], __ffma2_rn(make_float2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), scale2, neg_m));
                                    const float2 e = make_float2(ex2_fast(x.x), ex2_fast(x.y));
                                    sum2[k & 1] = __fadd2_rn(sum2[k & 1], e);
                                    pk[4 * q4 + k] = pack_bf2(e.x, e.y);
                                }
                            }
                            tmem_st8(tt + kTcP + bi * 32 + 16 * hf + 8 * jj, pk);
                        }
                    }
                    chunk_l = (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
                    if (c == 0 || !__any_sync(0xffffffffu, !(chunk_l <= kTcLazySum))) {
                        break;
                    }
                    // The reference value moves: the rows of this warp rescale what they have accumulated
                    // (every lane, by its own factor: TMEM accesses are warp-wide). O is current once the
                    // previous chunk's P·V is done, and the next P·V waits for this chunk's P.
                    const float mn = fmaxf(m, row_max());
                    if (!__any_sync(0xffffffffu, mn > m)) { // (a large sum of small exponentials)
                        break;
                    }
                    const float f = ex2_fast(m - mn);
                    m = mn, l *= f;
                    mbar_wait(&B.pv_done[bi ^ 1], ((g - 1) >> 1) & 1, &ctl->abort);
                    tc_fence_after();
#pragma unroll 1
                    for (int i = 0; i < kHeadD; i += 16) {
                        uint32_t r[16];
                        tmem_ld16_issue(tt + kTcO + i, r);
                        tmem_ld_wait(r);
#pragma unroll
                        for (int k = 0; k < 16; k++) {
                            r[k] = __float_as_uint(__uint_as_float(r[k]) * f);
                        }
                        tmem_st16(tt + kTcO + i, r);
                    }
                }
                l += chunk_l;
                CCK_TRACE_EV(0x34 + t, g - g0);
                // The tile of pair logits has been used, too: its slot may be refilled. The refill is a TMA write (async
                // proxy) over what this thread has read with ordinary loads: the proxy fence orders the two.
                fence_async_smem();
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&B.p_full[bi]);
                CCK_TRACE_EV(0x38 + t, g - g0);
                if (c == 0 && pend_lo >= 0) {
                    publish();
                }
            }
            cp_async_wait<0>();
            __syncwarp(); // the warp's rows of the gate are in its stage
            CCK_TRACE_EV(0x3a + t, j);
            mbar_wait(&B.o_full, jg & 1, &ctl->abort);
            tc_fence_after();
            CCK_TRACE_EV(0x3c + t, j);
            {
                // own row: O / l times the gate, in place of the gate, 16 columns at a time
                const float inv = 1.f / l;
                uint4* mine = reinterpret_cast<uint4*>(stage + lane * kTcOutPitch);
#pragma unroll
                for (int i = 0; i < kHeadD; i += 16) {
                    uint32_t o[16];
                    tmem_ld16_issue(tt + kTcO + i, o);
                    tmem_ld_wait(o);
#pragma unroll
                    for (int jj = 0; jj < 2; jj++) {
                        const uint4 gw = mine[i / 8 + jj];
                        const uint32_t w[4] = {gw.x, gw.y, gw.z, gw.w};
                        uint32_t out[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const float a0 = __uint_as_float(o[8 * jj + 2 * k]), a1 = __uint_as_float(o[8 * jj + 2 * k + 1]);
                            out[k] = pack_bf2(a0 * inv * bf_to_f32(w[k] & 0xFFFFu), a1 * inv * bf_to_f32(w[k] >> 16));
                        }
                        mine[i / 8 + jj] = make_uint4(out[0], out[1], out[2], out[3]);
                    }
                }
                CCK_TRACE_EV(0x40 + t, j);
                tc_fence_before(); // (the next item's first P·V, which overwrites O, follows the group's P of that chunk: after this read)
                // the warp's 32 rows to TO. A sample's last rows may be fewer (the rows after them are the
                // next sample's): those go out row by row.
                const int row0 = qb * kTcRows + q * 32, rows = min(N - row0, 32);
                if (rows == 32) {
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&L.tmap[TM_T_TO], h * kHeadD, s * N + row0, stage);
                        bulk_commit();
                    }
                } else if (lane < rows) {
                    uint4* dst = reinterpret_cast<uint4*>(p.buf.to + (size_t(s) * N + row0 + lane) * kTokC + h * kHeadD);
#pragma unroll
                    for (int jj = 0; jj < kTcOutPieces; jj++) {
                        dst[jj] = mine[jj];
                    }
                }
            }
            CCK_TRACE_EV(0x42 + t, j);
            if (flow) { // to be published once the store has landed: under the next item's first chunk, or after the last item
                pend_lo = s * N + qb * kTcRows, pend_hi = min(pend_lo + kTcRows, (s + 1) * N) - 1;
            }
            CCK_TRACE_EV(0x3e + t, j);
        }
        publish(); // (also: this warp's stores have landed before the phase ends)
        CCK_TRACE_END();
        if (q == 0 && lane == 0) { // one thread of the track
            bars->items[t] = j0 + uint32_t(n), bars->chunks[t] = g;
        }
    }
}

} // namespace cck
