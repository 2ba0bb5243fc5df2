// The dense GEMM engine: C = A·Wᵀ with bf16 operands and f32 accumulation on the 5th-generation
// tensor cores. Per CTA: one warp feeds a shared-memory ring with TMA tile loads, one warp issues
// tcgen05.mma into a double-buffered TMEM accumulator (2 x 256 columns), and eight warps drain finished
// accumulators with tcgen05.ld and apply the fused epilogue, so the epilogue of tile i overlaps the main
// loop of tile i+1. Tiles are 128 x bn (bn = 32..256) x 64.
// A main loop runs at the rate of its MMAs when both roles issue from warp-uniform code (ptx.cuh): measured
// inside the kernel, a k-block went from some 590 cycles at any width to 265 (bn = 128) and 525 (bn = 256).
//
// The epilogue kinds restate the reference's (src/diffusion/gemm.cuh:156-325) on a
// one-thread-per-row accumulator layout.
#pragma once


#include "params.cuh"
#include "ptx.cuh"

namespace cck {

constexpr int kBM = 128, kBK = 64, kMaxBN = 256;
constexpr int kStageA = kBM * kBK * 2; // 16 KB
constexpr int kPipeBytes = 192 << 10;
// The operand ring: a slot holds one k-block of A and of W. Its size follows the column tile, so that a
// narrow tile has more k-blocks in flight: the way of a k-block (request, L2, MMA, slot free again) takes
// some 2200 cycles whatever its width, and with four slots of any width a tile of 64 or 128 columns ran at
// that time / 4 = 590 cycles per k-block, where its MMAs take 245 or 290.
constexpr int kMaxSlots = 8;
__host__ __device__ constexpr int ring_slots(int bn) {
    return bn > 128 ? 4 : bn > 64 ? 6 : kMaxSlots;
}
__host__ __device__ constexpr int ring_slot_bytes(int bn) {
    return kStageA + bn * kBK * 2;
}
static_assert(ring_slots(256) * ring_slot_bytes(256) <= kPipeBytes && ring_slots(192) * ring_slot_bytes(192) <= kPipeBytes &&
                  ring_slots(128) * ring_slot_bytes(128) <= kPipeBytes && ring_slots(64) * ring_slot_bytes(64) <= kPipeBytes,
              "the ring outgrew its part of shared memory");
constexpr int kTmemCols = 512;
// Warp roles in the tensor-core phases: warp 0 holds the TMA thread, warp 1 the MMA thread, warps
// 2..9 are the workers that read TMEM (accumulator epilogues, attention softmax). A warp may only
// touch the TMEM lanes 32·(warp % 4).., so the eight workers form two groups of four, each group
// covering all 128 lanes; the groups split a tile's columns between them.
// Two more warps follow the workers: in the token attention, which runs two pipelines per CTA, they
// hold the second pipeline's TMA and MMA threads; in GEMM phases they have no role.
constexpr int kWorkWarp0 = 2, kWorkWarps = 8, kAuxWarp0 = kWorkWarp0 + kWorkWarps;
static_assert(kAuxWarp0 + 2 == kWarps, "TMA, MMA, eight workers (two per TMEM lane quarter), and the second pipeline's TMA and MMA");
constexpr int kAttnItemWarps = 4; // softmax warps that store the rows of one token-attention item (one group of workers)
__device__ __forceinline__ int work_quarter() {
    return warp_id() & 3;
}
__device__ __forceinline__ int work_group() {
    return (warp_id() - kWorkWarp0) >> 2;
}

// shared-memory control block
struct SmemCtl {
    uint64_t full[kMaxSlots], empty[kMaxSlots]; // TMA -> MMA, MMA -> TMA
    uint64_t tfull[2], tempty[2];           // MMA -> epilogue, epilogue -> MMA
    uint32_t tmem_base;
    volatile int abort;
    volatile int quit;                      // the launch has failed somewhere: leave the schedule
    unsigned long long t0;                  // end of the previous phase, ns (timing record, CTA 0)
    int ring_bn;                            // the column tile that the ring's slots are laid out for (TMA thread)
    const Launch* launch;                   // the kernel's parameter block
    unsigned int parts[4];                  // worker warps' parts of tiles counted so far, tile t in slot t % 4 (flow_signal_tile)
};

// CCK_TRACE=n builds another diagnostics variant: threads of CTA n - 1 write (cycle, event, value)
// records of what they pass, each role into its own 2048 slots (no atomics, one store per event), over
// the phases of a launch; mk_trace reads and clears them. Roles: 0, 1 the TMA threads; 2, 3 the MMA
// threads; 4, 5 the first worker thread of each group (token attention: per pipeline); 6 thread 0
// between the operations (operation begins, ends, grid barrier reached, passed).
// Events: 0x10.. TMA, 0x20.. MMA, 0x30.. softmax of the token attention (+1: second pipeline);
// 0x50.. TMA, 0x60.. MMA, 0x70.. epilogue of a GEMM; 0x80.. the schedule.
#ifndef CCK_TRACE
#define CCK_TRACE 0
#endif
#if CCK_TRACE
constexpr int kTraceRoles = 7, kTraceSlots = 2048;
__device__ unsigned long long g_trace[kTraceRoles][kTraceSlots];
__device__ unsigned int g_trace_n[kTraceRoles];
constexpr int kBarWaitSlots = 1024;
__device__ unsigned int g_barwait[kBarWaitSlots][160]; // [grid barrier][CTA]: cycles waited | phase kind << 24
#define CCK_TRACE_BEGIN_IF(role, cond) \
    const int tr_role_ = (role);       \
    unsigned int tr_n_ = (blockIdx.x == CCK_TRACE - 1 && (cond)) ? g_trace_n[tr_role_] : 0xffffffffu
#define CCK_TRACE_BEGIN(role) CCK_TRACE_BEGIN_IF(role, true)
#define CCK_TRACE_EV(code, val)                                                                                  \
    do {                                                                                                         \
        if (tr_n_ < kTraceSlots) {                                                                               \
            g_trace[tr_role_][tr_n_++] = (unsigned long long)(clock64()) << 16 | (unsigned long long)((code) << 8 | ((val) & 255)); \
        }                                                                                                        \
    } while (0)
#define CCK_TRACE_END()                                        \
    do {                                                       \
        if (tr_n_ != 0xffffffffu) g_trace_n[tr_role_] = tr_n_; \
    } while (0)
#define CCK_TRACE_ONE_IF(role, code, val, cond) \
    do {                                        \
        CCK_TRACE_BEGIN_IF(role, cond);         \
        CCK_TRACE_EV(code, val);                \
        CCK_TRACE_END();                        \
    } while (0)
#define CCK_TRACE_ONE(role, code, val) CCK_TRACE_ONE_IF(role, code, val, true)
#else
#define CCK_TRACE_BEGIN_IF(role, cond) do { } while (0)
#define CCK_TRACE_BEGIN(role) do { } while (0)
#define CCK_TRACE_EV(code, val) do { } while (0)
#define CCK_TRACE_END() do { } while (0)
#define CCK_TRACE_ONE_IF(role, code, val, cond) do { } while (0)
#define CCK_TRACE_ONE(role, code, val) do { } while (0)
#endif

static_assert(sizeof(SmemCtl) <= 256, "SmemCtl outgrew its part of the control block");
// Shared memory of the CTA: [pipeline stages | epilogue stages | control | schedule state | the
// parameter block | GEMM descriptors]. The first two are contiguous: phases without a GEMM use
// them as one scratch area.
constexpr int kEpiStageBytes = 32 * 16 * 4;                     // per worker warp: 32 rows x 16 floats
constexpr int kEpiOff = kPipeBytes;
constexpr int kScratchBytes = kPipeBytes + kWorkWarps * kEpiStageBytes;
constexpr int kCtlOff = kScratchBytes;                          // SmemCtl, the timing record, the attention barriers
constexpr int kTimingOff = 256, kTcBarsOff = 640;               // in the control block: per-kind [ns, phases] of the timing record; the attention barriers
static_assert(kTimingOff + 2 * kKinds * 8 <= kTcBarsOff, "the control block's parts overlap");
constexpr int kRunSlot = 24;                                    // bytes of per-thread schedule state (Run)
constexpr int kCtlBytes = 1280;
constexpr int kRunOff = kCtlOff + kCtlBytes;
constexpr int kKpOff = kRunOff + kRunSlot * kThreads;           // the CTA's copy of the parameter block
constexpr int kKpBytes = 1280;
constexpr int kGdOff = kKpOff + kKpBytes;                       // prepared GEMM descriptors
constexpr int kGdBytes = 4800;
constexpr int kProgOff = kGdOff + kGdBytes;                     // the phase program
constexpr int kProgBytes = 512;
static_assert(sizeof(Program) <= kProgBytes, "the phase program outgrew its shared-memory slot");
constexpr int kBiasOff = kProgOff + kProgBytes;                 // per worker warp: the bias of one 32-column unit
constexpr int kSmemBytes = kBiasOff + kWorkWarps * 128;
static_assert(sizeof(KP) <= kKpBytes, "KP outgrew its shared-memory slot");
constexpr int kSmemAlloc = kSmemBytes + 1024;                   // slack to align the base to 1024 bytes
static_assert(kSmemAlloc <= 232448, "more than the 227 KB a CTA may have");

__device__ __forceinline__ char* smem_base() {
    extern __shared__ char smem_raw[];
    const uint32_t a = smem_u32(smem_raw);
    return smem_raw + ((1024u - (a & 1023u)) & 1023u);
}
// the same, worked out anew where it is asked for: nothing of it is held in registers from an earlier place
__device__ __forceinline__ char* smem_base_anew() {
    extern __shared__ char smem_raw[];
    uint32_t a;
    asm volatile("mov.u32 %0, %1;" : "=r"(a) : "r"(smem_u32(smem_raw)));
    return static_cast<char*>(__cvta_shared_to_generic((a + 1023u) & ~1023u));
}
// The parameter block with the call's real extents filled in (the kernel parameter holds the
// bucket's): every CTA keeps a copy in shared memory
__device__ __forceinline__ const KP& kp() {
    return *reinterpret_cast<const KP*>(smem_base() + kKpOff);
}
__device__ __forceinline__ SmemCtl* smem_ctl() {
    return reinterpret_cast<SmemCtl*>(smem_base() + kCtlOff);
}
__device__ __forceinline__ long long wait_limit() {
    return kp().wait_cycles;
}
// Records the launch's first failure and tells the grid: the poison bit in the barrier word ends
// every CTA's wait at its next barrier (sampler.cuh: grid_barrier), after which the schedule is left.
__device__ __forceinline__ void fail_launch(unsigned int code, unsigned int where) {
    Control* c = kp().ctl;
    if (atomicCAS(&c->status, ST_OK, code) == ST_OK) {
        c->where = where;
    }
    atomicOr(&c->barrier, kBarrierPoison);
}

// n / d with a prepared multiplier (div_magic; 0: d = 1). A division by a number known only at run time is some 40
// instructions, and an operation's way in and out is run once per operation, from a cold instruction cache at 5 to 9
// cycles an instruction.
__host__ __device__ constexpr uint32_t div_magic(uint32_t d) {
    return d > 1 ? 0xFFFFFFFFu / d + 1u : 0u; // exact while n·d < 2^32
}
// the same for rows up to `most`; 0 where the product would not fit: divide
__host__ __device__ constexpr uint32_t div_magic_rows(uint32_t d, unsigned long long most) {
    return most * d < 0x100000000ull ? div_magic(d) : 0u;
}
__device__ __forceinline__ int div_rows(int r, int d, uint32_t magic) {
    return magic ? int(__umulhi(uint32_t(r), magic)) : r / d;
}
__device__ __forceinline__ int mod_rows(int r, int d, uint32_t magic) {
    return r - div_rows(r, d, magic) * d;
}
__device__ __forceinline__ uint32_t div_prepared(uint32_t n, uint32_t magic) {
    return magic ? __umulhi(n, magic) : n;
}

// per-thread pipeline positions, kept across phases for the whole launch
struct Pipe {
    uint32_t ring = 0; // phase parity of each slot of the operand ring, as this role passes them
    uint32_t tile = 0; // accumulator tiles issued (MMA thread) or drained (worker threads)
};

// Work dealing: item i of a phase goes to CTA (start + i) mod grid, and consecutive work lists of
// one phase continue the rotation (as the reference's Deal, src/diffusion/gemm.cuh:84-95)
struct Deal {
    int start = 0;
    __device__ __forceinline__ int first() const {
        const int f = int(blockIdx.x) - start;
        return f < 0 ? f + int(gridDim.x) : f;
    }
    __device__ __forceinline__ void advance(int items) {
        const uint32_t n = uint32_t(start + items);
        start = int(n - div_prepared(n, kp().div_grid) * gridDim.x);
    }
};

__host__ __device__ inline int cdiv(int a, int b) {
    return (a + b - 1) / b;
}

// ---- epilogues
// An accumulator tile leaves TMEM with one row per lane. Global memory wants the opposite:
// consecutive lanes on consecutive columns of one row. So each worker warp turns 32 rows x 16
// columns at a time through a private shared-memory stage (64-byte rows, 16-byte pieces XOR-swizzled:
// conflict-free both ways), after which lane l holds the four columns 4(l % 4).. of rows l / 4 + 8i,
// i < 4: every warp access covers eight full 64-byte row segments.
constexpr int kPiece = 16;
static_assert(kTokMods1 == 4 && kTokModSlots - kTokMods1 == 2 && kTokC % kMaxBN == 0, "EPI_MODS finds block and slot by shifts, once per tile");
__device__ __forceinline__ float* epi_stage() {
    return reinterpret_cast<float*>(smem_base() + kEpiOff + (warp_id() - kWorkWarp0) * kEpiStageBytes);
}
// row-per-lane values of 16 columns -> column-per-lane t[i] (row l / 4 + 8i)
__device__ __forceinline__ void epi_turn(float* st, const float* v, float4 (&t)[4]) {
    const int l = lane_id();
    float4* w = reinterpret_cast<float4*>(st + l * kPiece);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        w[i ^ ((l >> 1) & 3)] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    __syncwarp();
    const int r = l >> 2, c = l & 3;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = r + 8 * i;
        t[i] = *reinterpret_cast<const float4*>(st + row * kPiece + 4 * (c ^ ((row >> 1) & 3)));
    }
    __syncwarp();
}
__device__ __forceinline__ float4 unpack_bf4(uint2 u) {
    return make_float4(bf_to_f32(u.x & 0xFFFFu), bf_to_f32(u.x >> 16), bf_to_f32(u.y & 0xFFFFu), bf_to_f32(u.y >> 16));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// f32 outputs, one piece after the turn: rows r0 + 8i, columns c..c+3 (of the GEMM). The few of these with a bias fetch it here.
template <int E> __device__ __forceinline__ void epi_store(const GemmDesc& g, int r0, int c, const float4 (&t)[4]) {
    float* const o = static_cast<float*>(g.out) + c;
    const float4 b = E == EPI_F32 && g.bias && c < g.bias_cols ? *reinterpret_cast<const float4*>(g.bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = r0 + 8 * i;
        if (row >= g.m) {
            continue;
        }
        float4* p = reinterpret_cast<float4*>(o + size_t(row) * g.ldo);
        if constexpr (E == EPI_F32) {
            float4 x = add4(t[i], b);
            if (g.relu) {
                x = make_float4(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f), fmaxf(x.z, 0.f), fmaxf(x.w, 0.f));
            }
            *p = x;
        } else { // EPI_SCRES
            *p = add4(*p, t[i]);
        }
    }
}

// The pair logits of one unit: a tile's rows are 128 consecutive keys k of one query q (rbase
// encodes q·ktiles·128 + k0), the column is the table (block·16 + head); base-2 logits. Keys past the real tokens
// are masked, keys past the padded extent (a multiple of 64: a warp's 32 are in or out together) are not stored. The
// 32 tables x 32 keys leave the warp's stage as one block of the tables' planes, clipped at the last table; stored by the lanes themselves, 2 bytes to
// a lane and 32 addresses to a unit, a tile took 22,000 cycles (a run of one step, 2048 x 1: 7.33 -> 4.62 ms; 512 x 5: 2.63 -> 2.47).
__device__ __forceinline__ void pair_unit(const GemmDesc& g, const CUtensorMap* mo, float* st, int rbase, int c0, const float (&v)[32]) {
    const int q = rbase / (g.ktiles * kBM), k0 = rbase % (g.ktiles * kBM), l = lane_id(), k = k0 + l;
    if (q < g.nreal && k0 < g.npreal) {
        const TokenW& tw = kp().tw;
        const bool masked = k >= g.nreal || tw.tmask[k] == 0.f;
        const size_t pq = size_t(q) * g.ldn + (masked ? 0 : k);
        const float mean = tw.pcs[2 * pq], rstd = tw.pcs[2 * pq + 1];
        const float extra = kp().plx ? bf_to_f32(tw.plx[pq]) : 0.f;
        const bool table = c0 + l < kp().nb * kPairHeads; // (with an odd number of blocks the last unit has 16)
        const float ws = table ? tw.plws[c0 + l] : 0.f, wb = table ? tw.plb[c0 + l] : 0.f; // (lane l: of table c0 + l)
        if (l == 0) {
            bulk_wait_read(); // the previous store has read the stage
        }
        __syncwarp();
        bf16* out = reinterpret_cast<bf16*>(st) + l;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            const float wi = __shfl_sync(0xffffffffu, ws, i), bi = __shfl_sync(0xffffffffu, wb, i); // (by all lanes, masked or not)
            const float y = kLog2e * (masked ? -kMaskBias : rstd * (v[i] - mean * wi) + bi + extra);
            out[32 * i] = bf16(pack_bf2(y, 0.f) & 0xFFFFu);
        }
        fence_async_smem();
        __syncwarp();
        if (l == 0) {
            tma_store_3d(mo, k0, q, c0, st);
            bulk_commit();
        }
    }
}
// the v columns of QKVG, transposed: lanes are consecutive tokens, column hd of 32 tokens is one
// 64-byte run of VT
__device__ __forceinline__ void vt_unit(const GemmDesc& g, int rbase, int c0, const float (&v)[32]) {
    const int row = rbase + lane_id();
    if (row < g.m) {
        const int s = div_rows(row, g.period, g.div_period);
        bf16* o = g.vt + (size_t(s) * kTokC + (c0 - 2 * kTokC)) * g.np + (row - s * g.period);
#pragma unroll
        for (int i = 0; i < 32; i++) {
            o[size_t(i) * g.np] = bf16(pack_bf2(v[i], 0.f) & 0xFFFFu);
        }
    }
}

// A unit of bf16 output: the warp's 32 rows x 32 columns go row-per-lane (as they leave TMEM) into the
// warp's stage in the 64-byte-swizzled layout of the store map, and one lane issues the store. No turn, no per-row
// address arithmetic. In the last row tile, where what the store would write past the GEMM's rows is somebody else's, the lanes
// store their rows themselves. (A second epilogue for that, with the turn, was half of the code of these kinds: ms per
// step with it gone: 32 x 1 0.920 -> 0.903, 256 x 5 1.511 -> 1.489, 512 x 5 2.317 -> 2.287, 391 x 5 2.103 -> 2.048.)
__device__ __forceinline__ void store_unit(const CUtensorMap* mo, float* st, int x, int y, bool whole, bf16* own, const float (&v)[32]) {
    const int l = lane_id();
    uint4 w[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        w[c] = make_uint4(pack_bf2(v[8 * c], v[8 * c + 1]), pack_bf2(v[8 * c + 2], v[8 * c + 3]), pack_bf2(v[8 * c + 4], v[8 * c + 5]),
                          pack_bf2(v[8 * c + 6], v[8 * c + 7]));
    }
    if (!whole) {
        if (own) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                reinterpret_cast<uint4*>(own)[c] = w[c];
            }
        }
        return;
    }
    if (l == 0) {
        bulk_wait_read(); // the previous store has read the stage
    }
    __syncwarp();
    uint4* row = reinterpret_cast<uint4*>(reinterpret_cast<char*>(st) + 64 * l);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        row[c ^ ((l >> 1) & 3)] = w[c];
    }
    fence_async_smem();
    __syncwarp();
    if (l == 0) {
        tma_store_2d(mo, x, y, st);
        bulk_commit();
    }
}

// The epilogue of one 128 x bn accumulator held in TMEM columns [acc, acc + bn), by the eight
// worker warps: units of 32 output columns alternate between the two groups. Waits for the
// accumulator itself; of a bf16 output with a bias, the first unit's bias is under way by then.
template <int E> __device__ __forceinline__ void epilogue_tile(const GemmDesc& g, const CUtensorMap* mo, uint32_t acc, int row0, int col0,
                                                               uint64_t* tfull, uint32_t tpar, volatile int* abort) {
    const int q = work_quarter(), gp = work_group(), rbase = row0 + q * 32;
    const uint32_t taddr = acc + (uint32_t(q * 32) << 16);
    float* st = epi_stage();
    if constexpr (E == EPI_BF16 || E == EPI_GLU || E == EPI_MODS) {
        const int kIn = E == EPI_GLU ? g.glu_unit : 32; // accumulator columns per unit
        const int units = g.bn / kIn;
        // output column of unit u: a GLU unit of 64 (or 96) columns gives 32
        const int oc0 = E == EPI_GLU ? col0 / kIn * kGluHalf : col0;
        const bool whole = rbase + 32 <= g.m;
        // the unit's bias (one value per lane) waits in the warp's shared-memory slot, fetched a unit ahead
        float* bs = reinterpret_cast<float*>(smem_base() + kBiasOff) + (warp_id() - kWorkWarp0) * 32;
        const bool has_bias = E != EPI_GLU && g.bias != nullptr;
        float bnext = 0.f;
        if (has_bias && gp < units && oc0 + 32 * gp < g.bias_cols) {
            bnext = g.bias[oc0 + 32 * gp + lane_id()];
        }
        // MODS: a tile lies in one slot of one block (768 is a multiple of every width): column c is slot slot0 + (c / 768) % slots of block c / (slots·768)
        int x0 = oc0, y = rbase;
        bool msig = false;
        if constexpr (E == EPI_MODS) {
            const int s = oc0 / kTokC, blk = g.slots == 4 ? s >> 2 : s >> 1, slot = g.slot0 + (s & (g.slots - 1));
            msig = g.sig_slots >> slot & 1, x0 = oc0 - s * kTokC, y = (blk * kTokModSlots + slot) * g.period + rbase;
        }
        mbar_wait(tfull, tpar, abort);
        tc_fence_after();
#pragma unroll 1
        for (int u = gp; u < units; u += 2) {
            const int oc = oc0 + 32 * u, x = x0 + 32 * u;
            const bool biased = has_bias && oc < g.bias_cols; // (a unit has a bias or has none: bias_cols is a multiple of 32. Zeros added instead: 256 x 5 and 512 x 5 0.3 to 0.5 % more, small folds the same)
            if (biased) {
                __syncwarp();
                bs[lane_id()] = bnext;
                __syncwarp();
                if (u + 2 < units && oc + 64 < g.bias_cols) {
                    bnext = g.bias[oc + 64 + lane_id()];
                }
            }
            float v[32];
            if constexpr (E == EPI_GLU) {
                uint32_t ga[32], pr[32];
                tmem_ld32_issue(taddr + u * kIn, ga);
                tmem_ld32_issue(taddr + u * kIn + kGluHalf, pr);
                tmem_ld_wait(ga);
                tmem_ld_wait(pr);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float2 z = __fmul2_rn(silu_fast2(make_float2(__uint_as_float(ga[i]), __uint_as_float(ga[i + 1]))),
                                                make_float2(__uint_as_float(pr[i]), __uint_as_float(pr[i + 1])));
                    v[i] = z.x, v[i + 1] = z.y;
                }
                if (kIn > 2 * kGluHalf) { // [gate | proj | a_to_b]: the third part multiplies
                    float ab[32];
                    tmem_ld32(taddr + u * kIn + 2 * kGluHalf, ab);
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        v[i] *= ab[i];
                    }
                }
            } else {
                tmem_ld32(taddr + u * kIn, v);
            }
            if (biased) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 bb = reinterpret_cast<const float4*>(bs)[i];
                    v[4 * i] += bb.x, v[4 * i + 1] += bb.y, v[4 * i + 2] += bb.z, v[4 * i + 3] += bb.w;
                }
            }
            bool sig = msig;
            if constexpr (E == EPI_BF16) {
                sig = oc >= g.sig_from;
                if (g.vt && oc >= 2 * kTokC && oc < 3 * kTokC) {
                    vt_unit(g, rbase, oc, v);
                }
            }
            if (sig) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float2 z = sigmoid_fast2(make_float2(v[i], v[i + 1]));
                    v[i] = z.x, v[i + 1] = z.y;
                }
            }
            bf16* own = rbase + lane_id() < g.m ? static_cast<bf16*>(g.out) + size_t(y + lane_id()) * (E == EPI_MODS ? kTokC : g.ldo) + x : nullptr;
            store_unit(mo, st, x, y, whole, own, v);
        }
    } else {
        const int r0 = rbase + (lane_id() >> 2), cl = 4 * (lane_id() & 3), units = g.bn / 32;
        mbar_wait(tfull, tpar, abort);
        tc_fence_after();
#pragma unroll 1
        for (int u = gp; u < units; u += 2) {
            const int oc = col0 + 32 * u;
            if constexpr (E == EPI_PAIR) {
                float v[32];
                tmem_ld32(taddr + u * 32, v);
                pair_unit(g, mo, st, rbase, oc, v);
            } else {
#pragma unroll 1
                for (int k = 0; k < 32; k += kPiece) {
                    float v[16];
                    tmem_ld16(taddr + u * 32 + k, v);
                    float4 t[4];
                    epi_turn(st, v, t);
                    epi_store<E>(g, r0, oc + k + cl, t);
                }
            }
        }
    }
}

// The gated residual update out = src + gate ⊙ C · rowmask. Everything it reads besides the
// accumulator depends on addresses only, so it is fetched into registers while the main loop runs: the
// residual and the gates of 16 NP columns per warp (group 0 the tile's left half, group 1 its right one), 4
// rows x 4 columns of a piece of 16 columns per lane. f32 gates (the atom GEMMs) come a piece ahead instead:
// beside the residual they would not fit.
constexpr int kResidMaxBnBf = 128, kResidMaxBnF32 = 64;
template <bool GF32, int NP>
__device__ __forceinline__ void resid_tile(const GemmDesc& g, const void* gate, uint32_t acc, int row0, int col0, uint64_t* tfull, uint32_t tpar,
                                           volatile int* abort) {
    const int q = work_quarter(), c0 = work_group() * NP * kPiece;
    const int r0 = row0 + q * 32 + (lane_id() >> 2), cl = 4 * (lane_id() & 3);
    const uint32_t taddr = acc + (uint32_t(q * 32) << 16) + c0;
    const int m = g.m, ldo = g.ldo;
    float* const op = static_cast<float*>(g.out) + col0 + c0 + cl;
    float4 x[NP][4];
    float mask[4];
    uint2 gb[GF32 ? 1 : NP][4];
    float4 gf[2][4];
    const char* gp[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = min(r0 + 8 * i, m - 1), p = mod_rows(row, g.period, g.div_period);
        mask[i] = g.rowmask ? g.rowmask[p] : 1.f;
        gp[i] = static_cast<const char*>(gate) + (size_t(p) * g.ldg + col0 + c0 + cl) * (GF32 ? 4 : 2);
#pragma unroll
        for (int k = 0; k < NP; k++) {
            x[k][i] = __ldcg(reinterpret_cast<const float4*>(op + size_t(row) * ldo + kPiece * k));
            if constexpr (!GF32) {
                gb[k][i] = *reinterpret_cast<const uint2*>(gp[i] + 2 * kPiece * k);
            }
        }
        if constexpr (GF32) {
            gf[0][i] = *reinterpret_cast<const float4*>(gp[i]);
        }
    }
    mbar_wait(tfull, tpar, abort);
    tc_fence_after();
    float* st = epi_stage();
#pragma unroll
    for (int k = 0; k < NP; k++) {
        if constexpr (GF32) {
            if (k + 1 < NP) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    gf[(k + 1) & 1][i] = *reinterpret_cast<const float4*>(gp[i] + 4 * kPiece * (k + 1));
                }
            }
        }
        float h[16];
        tmem_ld16(taddr + kPiece * k, h);
        float4 t[4];
        epi_turn(st, h, t);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = r0 + 8 * i;
            if (row < m) {
                const float4 gt = GF32 ? gf[k & 1][i] : unpack_bf4(gb[GF32 ? 0 : k][i]);
                const float4 y = x[k][i], cc = t[i];
                *reinterpret_cast<float4*>(op + size_t(row) * ldo + kPiece * k) =
                    make_float4(y.x + gt.x * cc.x * mask[i], y.y + gt.y * cc.y * mask[i], y.z + gt.z * cc.z * mask[i], y.w + gt.w * cc.w * mask[i]);
            }
        }
    }
}

// tile t -> (row tile, column tile) without an integer division
__device__ __forceinline__ void tile_coords(const GemmDesc& g, int t, int& row0, int& col0) {
    // t = major · inner + minor: (column tile, row tile) with inner = mt, or with nfast (row tile,
    // column tile) with inner = nt: a row tile's column tiles are dealt together, its rows complete early
    const int inner = (g.fl & GF_NFAST) ? g.nt : g.mt;
    const int major = g.mt_magic ? int(__umulhi((unsigned int)t, g.mt_magic)) : t / inner, minor = t - major * inner;
    row0 = ((g.fl & GF_NFAST) ? major : minor) * kBM, col0 = ((g.fl & GF_NFAST) ? minor : major) * g.bn;
}
__host__ __device__ inline void gd_finish(GemmDesc& g) {
    g.nt = g.n / g.bn;
    g.mt = cdiv(g.m, kBM), g.tiles = g.mt * g.nt;
    const int inner = (g.fl & GF_NFAST) ? g.nt : g.mt;
    // exact while t · inner < 2^32; otherwise 0: divide
    g.mt_magic = (unsigned long long)(g.tiles) * inner < 0x100000000ull ? (unsigned int)((0x100000000ull + inner - 1) / inner) : 0u;
    if (inner == 1) {
        g.mt_magic = 0; // 2^32 does not fit
    }
    g.div_period = div_magic_rows(g.period, g.m);
}

// ---- prepared GEMM descriptors: built once per launch into shared memory, so that a phase starts
// with a few shared-memory loads instead of a few hundred dependent scalar instructions
__device__ __forceinline__ GemmDesc* gd_table() {
    return reinterpret_cast<GemmDesc*>(smem_base() + kGdOff);
}
constexpr int kMaxGd = kGdBytes / int(sizeof(GemmDesc));

// ---- completion counters between operations of one phase (FlowCnt)
__device__ __forceinline__ unsigned int* flow_cnt(const KP& p, int which) {
    return p.flow_cnt + (which < kFlowTok ? which * p.flow_n : kFlowTok * p.flow_n + (which - kFlowTok) * p.flow_na) * kFlowPitch;
}
// The calling warp's part of a unit is stored: its lanes' writes (and lane 0's TMA stores, which the
// caller has waited for) are published with one release add per counter in [c0, c1]. The proxy fence that a
// TMA read of ordinary stores needs is on the reader's side, behind its acquire (FlowWait::acquire, flow_wait,
// flow_wait_warp): one on the path from the write to the read is enough, and here it would be paid by every warp (0.1 to 0.3 %).
// No writer has one, so every wait that a TMA load may follow must keep its own, whatever it costs.
__device__ __forceinline__ void flow_signal(unsigned int* cnt, int c0, int c1) {
    __syncwarp();
    if (lane_id() == 0) {
        for (int c = c0; c <= c1; c++) {
            red_release_add(cnt + c * kFlowPitch, 1u);
        }
    }
}
// The same for a GEMM tile, by the eight worker warps together: each counts itself in shared memory (acquire and
// release at the CTA's scope), and the one that comes last publishes all eight parts with one release add. A release at
// the grid's scope waits for the stores in flight and takes some 1500 cycles; eight of them at once got in each
// other's way (ms per step 32 x 1 0.892 -> 0.889, 64 x 5 1.042 -> 1.017, 256 x 5 1.512 -> 1.482, 512 x 1 1.288 -> 1.259,
// 512 x 5 2.314 -> 2.279, 1024 x 5 0.3 %). The token attention and the row passes, whose warps finish further apart, lose by it.
// Tile t is counted in slot t % 4: a warp that is through with tile t + 3 has seen its accumulator, whose buffer tile
// t + 1 held, so that every warp had read that one and, before it, counted itself for tile t.
__device__ __forceinline__ void flow_signal_tile(unsigned int* cnt, unsigned int* parts) {
    __syncwarp();
    if (lane_id() == 0 && (atom_add_cta(parts, 1u) & (kWorkWarps - 1)) == kWorkWarps - 1) {
        red_release_add(cnt, (unsigned int)(kWorkWarps));
    }
}
static_assert((kWorkWarps & (kWorkWarps - 1)) == 0, "a tile's last part is told by the low bits of the count");
// One thread's wait for one counter, in single looks, so that it can do something else in between.
// Bounded as every wait here: when it gives up, or the launch has failed elsewhere, ready() says true and
// the abort flag is set.
struct FlowWait {
    const unsigned int* cnt;
    unsigned int target, looks;
    volatile int* abort;
    long long t0;
    __device__ __forceinline__ FlowWait(const unsigned int* c, unsigned int tgt, volatile int* ab) : cnt(c), target(tgt), looks(0), abort(ab) {
        t0 = clock64();
        if (*abort) { // a wait inside this CTA gave up earlier: tell the grid, which would otherwise wait for this CTA's units
            fail_launch(ST_PIPE_TIMEOUT, 0);
        }
    }
    __device__ __forceinline__ bool ready() {
        if (ld_acquire(cnt) >= target) { // (an acquire at every look, so that no fence, which takes as long as a look, follows the last)
            return true;
        }
        return *abort || (++looks % 32 == 0 && given_up()); // (the status word is another way to L2: not at every look)
    }
    // another CTA gave up (its units will not come), or this wait ran out: the launch drains
    __device__ __noinline__ bool given_up() {
        if (ld_relaxed(&kp().ctl->status) == ST_OK && clock64() - t0 <= wait_limit()) {
            return false;
        }
        fail_launch(ST_PIPE_TIMEOUT, 0);
        *abort = 1;
        return true;
    }
    // what the signalling warps wrote is visible to what follows: this thread's reads and TMA loads
    __device__ __forceinline__ void acquire() {
        fence_async_global();
    }
};
// One thread waits until the counters [c0, c1] have reached target, one after the other; what it then reads is what
// the signalling warps wrote.
__device__ __forceinline__ void flow_wait(const unsigned int* cnt, int c0, int c1, unsigned int target, volatile int* abort) {
    const long long t0 = clock64();
    unsigned int looks = 0;
    if (*abort) { // a wait inside this CTA gave up earlier: tell the grid, which would otherwise wait for this CTA's units
        fail_launch(ST_PIPE_TIMEOUT, 0);
    }
    for (int c = c0; c <= c1; c++) {
        while (ld_acquire(cnt + c * kFlowPitch) < target) {
            if (*abort) {
                return;
            }
            // another CTA gave up (its units will not come), or this wait ran out: the launch drains
            if (++looks % 32 == 0 && (ld_relaxed(&kp().ctl->status) != ST_OK || clock64() - t0 > wait_limit())) {
                fail_launch(ST_PIPE_TIMEOUT, 0);
                *abort = 1;
                return;
            }
        }
    }
    fence_async_global();
}
// The same by a whole warp, a lane to a counter: the counters of a sample of the token attention (5 at 512 tokens, 16 at
// 2048) then cost one trip to L2 when the last of them is complete, not one each (ms per step 512 x 1 1.349 -> 1.333, 512 x 5 2.358
// -> 2.344, 2048 x 1 3.257 -> 3.204). The atom rows, which wait for two or three, lose by it what they gain.
__device__ __forceinline__ void flow_wait_warp(const unsigned int* cnt, int c0, int c1, unsigned int target, volatile int* abort) {
    const long long t0 = clock64();
    unsigned int looks = 0;
    if (*abort) { // (as flow_wait)
        fail_launch(ST_PIPE_TIMEOUT, 0);
    }
#pragma unroll 1
    for (int c = c0; c <= c1; c += 32) {
        const unsigned int* mine = cnt + min(c + lane_id(), c1) * kFlowPitch;
        while (!__all_sync(0xffffffffu, ld_acquire(mine) >= target)) {
            if (__any_sync(0xffffffffu, *abort != 0)) {
                return;
            }
            if (++looks % 32 == 0 && __any_sync(0xffffffffu, ld_relaxed(&kp().ctl->status) != ST_OK || clock64() - t0 > wait_limit())) {
                fail_launch(ST_PIPE_TIMEOUT, 0);
                *abort = 1;
                return;
            }
        }
    }
    fence_async_global();
}
// Arrivals that complete row block rb of a GEMM's A (descriptor g, depc set) in one token block. TO:
// the attention items of every block of 128 queries (per sample of g.period rows) that the rows
// touch, 16 heads x 4 warps each. TC: the column tiles of W1 over these rows, 8 warps each. ACA: the same of the atoms. TX,
// TX0, AX, AXT: the rows of the block.
__device__ __noinline__ unsigned int flow_target_to(const GemmDesc& g, int rb) {
    const int lo = rb * kBM, hi = min(lo + kBM, g.m) - 1, qblocks = cdiv(g.period, kBM);
    const int ilo = lo / g.period * qblocks + lo % g.period / kBM, ihi = hi / g.period * qblocks + hi % g.period / kBM;
    return (unsigned int)(kHeads * kAttnItemWarps * (ihi - ilo + 1));
}
__device__ __forceinline__ unsigned int flow_target(const GemmDesc& g, int which, int rb) {
    if (g.dep_target) {
        return g.dep_target;
    }
    return which == FC_TO ? flow_target_to(g, rb) : (unsigned int)(min(kBM, g.m - rb * kBM));
}
// (part of the descriptor, once all of them are there)
__device__ inline void gd_finish_target(GemmDesc& g) {
    const int which = int(g.fl >> GF_DEP_SHIFT & GF_CNT_MASK) - 1;
    g.dep_target = which == FC_TC    ? (unsigned int)(gd_table()[GD_TOK_W1].nt * kWorkWarps)
                   : which == FC_ACA ? (unsigned int)(gd_table()[GD_ENC_W1].nt * kWorkWarps)
                   : which == FC_TO && g.period % kBM == 0 ? (unsigned int)(kHeads * kAttnItemWarps)
                                                           : 0u;
}

// the worker warps' loop over the tiles of one GEMM, block b of its stack; every finished tile is
// reported to the completion counter of its block of 128 rows, if the descriptor names one
template <int E> __device__ CCK_HOT_FN void worker_tiles(const GemmDesc& gd, const CUtensorMap* mo, int b, Pipe& pipe, int tb, int te, int ts,
                                                         unsigned int epoch) {
    uint32_t tile = pipe.tile;
    SmemCtl* ctl = smem_ctl();
    GemmDesc g = gd; // a private copy: stores through its pointers cannot alias it
    g.bias = g.bias ? g.bias + size_t(b) * g.bias_step : nullptr;
    if constexpr (E == EPI_BF16) {
        if ((gd.fl & GF_ALT) && (epoch & 1)) {
            g.out = kp().buf.qkvg2, g.vt = kp().buf.vt2;
        }
    }
    CCK_TRACE_BEGIN_IF(4, threadIdx.x == kWorkWarp0 * 32);
    CCK_TRACE_EV(0x70, E);
    for (int t = tb; t < te; t += ts, tile++) {
        int row0, col0;
        tile_coords(gd, t, row0, col0); // (from the shared-memory descriptor: nothing of it held across the epilogue)
        const uint32_t buf = tile & 1, tpar = (tile >> 1) & 1;
        const uint32_t acc = ctl->tmem_base + buf * kMaxBN;
        if constexpr (E == EPI_RESID) {
            // The epilogue fetches the residual rows ahead, under the main loop. On completion counters the
            // operation that wrote them last may still be running elsewhere: W2 of the block before for WO, which the
            // attention's adaLN rows have waited for; WO for W2, which the transition's have. (Not the rows of A that the
            // tile itself waits for: those come later, and eight warps would stand polling for them, each look emptying the
            // SM's L1. 61 x 5 1.079 -> 1.070 ms per step, 512 x 1 1.329 -> 1.319, 391 x 5 2.134 -> 2.124.)
            if (const int depc = gd.fl >> GF_DEP_SHIFT & GF_CNT_MASK) {
                if (lane_id() == 0) {
                    const int rows = depc == 1 + FC_TO ? FC_TX0 : depc == 1 + FC_TC ? FC_TX : FC_AXT, rb = row0 / kBM;
                    flow_wait(flow_cnt(kp(), rows), rb, rb, (epoch + 1) * (unsigned int)(min(kBM, gd.m - row0)), &ctl->abort);
                }
                __syncwarp();
            }
            const char* gate = static_cast<const char*>(gd.gate) + (long long)(b)*gd.gate_step;
            if (gd.gate_f32) {
                if (gd.bn == 64) {
                    resid_tile<true, 2>(gd, gate, acc, row0, col0, &ctl->tfull[buf], tpar, &ctl->abort);
                } else {
                    resid_tile<true, 1>(gd, gate, acc, row0, col0, &ctl->tfull[buf], tpar, &ctl->abort);
                }
            } else if (gd.bn == 128) {
                resid_tile<false, 4>(gd, gate, acc, row0, col0, &ctl->tfull[buf], tpar, &ctl->abort);
            } else if (gd.bn == 64) {
                resid_tile<false, 2>(gd, gate, acc, row0, col0, &ctl->tfull[buf], tpar, &ctl->abort);
            } else {
                resid_tile<false, 1>(gd, gate, acc, row0, col0, &ctl->tfull[buf], tpar, &ctl->abort);
            }
        } else {
            epilogue_tile<E>(g, mo, acc, row0, col0, &ctl->tfull[buf], tpar, &ctl->abort);
        }
        tc_fence_before();
        __syncwarp();
        CCK_TRACE_EV(0x72, t); // the accumulator is read
        if (lane_id() == 0) {
            mbar_arrive(&ctl->tempty[buf]);
        }
        if constexpr (E == EPI_BF16 || E == EPI_GLU || E == EPI_RESID) {
            if (const int sigc = gd.fl >> GF_SIG_SHIFT & GF_CNT_MASK) {
                if (E != EPI_RESID && lane_id() == 0) {
                    bulk_wait_done();
                }
                int r0, c0; // (recomputed: not held across the epilogue)
                tile_coords(gd, t, r0, c0);
                flow_signal_tile(flow_cnt(kp(), sigc - 1) + r0 / kBM * kFlowPitch, &ctl->parts[tile & 3]);
            }
        }
        CCK_TRACE_EV(0x74, t); // stored and reported
    }
    pipe.tile = tile;
    if constexpr (E == EPI_BF16 || E == EPI_GLU || E == EPI_MODS || E == EPI_PAIR) {
        if (lane_id() == 0) {
            bulk_wait_done(); // this warp's TMA stores have landed before the phase ends
        }
        __syncwarp();
    }
    CCK_TRACE_EV(0x76, 0);
    CCK_TRACE_END();
}

// ---- the TMA and MMA roles over the tiles of one GEMM
// Tiles tb, tb + ts, ... < te of descriptor gd with block b of its stack applied; one warp each (what a
// single lane must do is predicated, see ptx.cuh). Both roles take the ring's slots in order from slot 0 at
// the start of a GEMM; a slot's phase parity is a bit of pipe.ring, so the number of slots may change from
// one GEMM to the next.

// Where a tile's operands lie: row of A's map (pair GEMM: row tile (q, key tile) starts at row q·ldn + k0
// of PC) and row of W's map
struct TileRows {
    int a, b;
};
__device__ __forceinline__ TileRows tile_rows(const GemmDesc& gd, int b, int t) {
    int row0, col0;
    tile_coords(gd, t, row0, col0);
    TileRows r;
    r.a = uni(gd.ktiles ? row0 / (gd.ktiles * kBM) * gd.ldn + row0 % (gd.ktiles * kBM) : gd.a_row0 + row0);
    r.b = uni(gd.b_row0 + b * gd.b_step + col0);
    return r;
}
// A GEMM with another column tile lays the ring out anew: what the slots hold must have been consumed.
__device__ __forceinline__ void ring_layout(SmemCtl* ctl, uint32_t ring, int bn) {
    if (uni(ctl->ring_bn) != bn) {
        if (lane_id() < kMaxSlots) { // (a lane per slot: a wait that passes costs 90 cycles)
            mbar_wait(&ctl->empty[lane_id()], (ring >> lane_id() & 1) ^ 1, &ctl->abort);
        }
        __syncwarp();
        ctl->ring_bn = bn;
        __syncwarp();
    }
}
// A sampling step of the smallest fold reads 400 MB of weights, which push everything else out of the 126 MB of
// L2: inputs, intermediate rows and the kernel's own code (half a megabyte, most of it run once per step)
// then come from HBM. Where few row tiles share a weight tile, within microseconds, the weights are marked as
// the first to leave: 1.20 -> 1.11 ms per step at 32 x 1, 1.37 -> 1.34 at 61 x 5. With many row tiles that
// loses the weights between two of them (5.37 -> 5.51 ms at 1024 x 5; with 24 for the limit, 16 to 20 row tiles
// read 0.5 GB per step more from HBM than with 8: 512 x 5 2.440 -> 2.417, 391 x 5 2.230 -> 2.200). 2, 4, 8 and 12 are alike.
constexpr int kOnceRowTiles = 8;
__device__ __forceinline__ uint64_t weights_policy(const GemmDesc& gd) {
    return l2_policy(uni(gd.mt) <= kOnceRowTiles);
}
// The weights of the first k-blocks of this CTA's first tile, asked for ahead of everything the tile has to
// wait for (a grid barrier): they depend on nothing that the launch computes. Returns how many.
__device__ CCK_PHASE_FN int gemm_prefetch_w(const Launch& L, Pipe& pipe, const GemmDesc& gd, int b, int tb, int te) {
    if (tb >= te) {
        return 0;
    }
    SmemCtl* ctl = smem_ctl();
    const uint32_t el = elect_one(), ring = uni(pipe.ring);
    const uint64_t policy = weights_policy(gd);
    const int bn = uni(gd.bn);
    ring_layout(ctl, ring, bn);
    const CUtensorMap* mb = &L.tmap[uni(gd.map_b)];
    const uint32_t bytes = ring_slot_bytes(bn), w0 = uni(smem_u32(smem_base())) + kStageA, full = uni(smem_u32(&ctl->full[0]));
    const int n = uni(min(gd.k / kBK, ring_slots(bn))), kwrap = uni(gd.b_kwrap ? gd.b_kwrap : 1 << 30), row = tile_rows(gd, b, tb).b;
    for (int i = 0; i < n; i++) {
        mbar_wait(&ctl->empty[i], (ring >> i & 1) ^ 1, &ctl->abort);
        mbar_expect_tx_el(el, full + 8 * i, bytes);
        const int k = i * kBK;
        tma_load_2d_hint_el(el, w0 + i * bytes, mb, k >= kwrap ? k - kwrap : k, row, full + 8 * i, policy);
    }
    return n;
}
// The TMA role. `ahead`: run by the warp that saw a grid barrier open, right there, before the rest of the
// CTA has found its way to the operation; pipe.tile of this warp (otherwise unused) then says that the
// next call has nothing left to do. `have`: k-blocks of the first tile whose weights are already on their
// way (gemm_prefetch_w). While a tile waits for the rows of A that it reads, its weights are fetched into
// the slots that are free: when the rows are complete, only A's way is left.
__device__ CCK_PHASE_FN void gemm_produce(const Launch& L, Pipe& pipe, const GemmDesc& gd, int b, int tb, int te, int ts, bool ahead,
                                          int have, unsigned int epoch) {
    if (pipe.tile) { // produced ahead
        pipe.tile = 0;
        return;
    }
    if (tb < te) {
        SmemCtl* ctl = smem_ctl();
        const uint32_t el = elect_one();
        const uint64_t policy = weights_policy(gd);
        const CUtensorMap* ma = &L.tmap[uni(gd.map_a)];
        const CUtensorMap* mb = &L.tmap[uni(gd.map_b)];
        const int bn = uni(gd.bn), kblocks = uni(gd.k / kBK), slots = ring_slots(bn), depc = uni(gd.fl >> GF_DEP_SHIFT & GF_CNT_MASK);
        const int kwrap = uni(gd.b_kwrap ? gd.b_kwrap : 1 << 30);
        const uint32_t bytes = ring_slot_bytes(bn), sm = uni(smem_u32(smem_base())), full = uni(smem_u32(&ctl->full[0])),
                       empty = uni(smem_u32(&ctl->empty[0]));
        uint32_t ring = uni(pipe.ring);
        int s = 0;
        have = uni(have), tb = uni(tb), te = uni(te), ts = uni(ts);
        if (have == 0) {
            ring_layout(ctl, ring, bn);
        }
        CCK_TRACE_BEGIN_IF(0, el);
        CCK_TRACE_EV(0x50, gd.epi);
        for (int t = tb; t < te; t += ts, have = 0) {
            const TileRows r = tile_rows(gd, b, t);
            if (depc) { // until the rows of A that this tile reads are complete
                int row0, col0;
                tile_coords(gd, t, row0, col0);
                const int rb = row0 / kBM;
                FlowWait w(flow_cnt(kp(), depc - 1) + rb * kFlowPitch, (epoch + 1) * flow_target(gd, depc - 1, rb), &ctl->abort);
                const int most = min(kblocks, slots);
                int f = s + have < slots ? s + have : s + have - slots; // the slot of k-block `have`
                while (!uni(int(w.ready()))) {
                    if (have < most && uni(int(mbar_test_a(empty + 8 * f, (ring >> f & 1) ^ 1)))) {
                        mbar_expect_tx_el(el, full + 8 * f, bytes);
                        const int k = have * kBK;
                        tma_load_2d_hint_el(el, sm + f * bytes + kStageA, mb, k >= kwrap ? k - kwrap : k, r.b, full + 8 * f, policy);
                        have++;
                        f = f + 1 < slots ? f + 1 : 0;
                    }
                }
                w.acquire();
            }
            CCK_TRACE_EV(0x52, t); // what the tile reads is complete
            for (int kb = 0; kb < kblocks; kb++) {
                const uint32_t st = sm + s * bytes, bar = full + 8 * s;
                const int k = kb * kBK;
                if (kb >= have) {
                    mbar_wait(&ctl->empty[s], (ring >> s & 1) ^ 1, &ctl->abort);
                    mbar_expect_tx_el(el, bar, bytes);
                    tma_load_2d_hint_el(el, st + kStageA, mb, k >= kwrap ? k - kwrap : k, r.b, bar, policy);
                }
                tma_load_2d_el(el, st, ma, k, r.a, bar);
                ring ^= 1u << s;
                s = s + 1 < slots ? s + 1 : 0;
            }
            CCK_TRACE_EV(0x54, t); // every k-block is asked for
        }
        CCK_TRACE_END();
        pipe.ring = ring;
    }
    pipe.tile = ahead;
}
__device__ CCK_PHASE_FN void gemm_issue(Pipe& pipe, const GemmDesc& gd, int tb, int te, int ts) {
    if (tb >= te) {
        return;
    }
    SmemCtl* ctl = smem_ctl();
    const uint32_t el = elect_one();
    const int bn = uni(gd.bn), kblocks = uni(gd.k / kBK), slots = ring_slots(bn);
    const uint32_t idesc = umma_idesc_bf16(kBM, bn), tmem = uni(ctl->tmem_base), full = uni(smem_u32(&ctl->full[0])),
                   empty = uni(smem_u32(&ctl->empty[0])), tfull = uni(smem_u32(&ctl->tfull[0]));
    uint32_t ring = uni(pipe.ring), tile = uni(pipe.tile);
    tb = uni(tb), te = uni(te), ts = uni(ts);
    // the operands' descriptors differ from slot to slot by the slot's size (in units of 16 bytes)
    const uint64_t d0 = umma_desc_sw128(uni(smem_u32(smem_base()))), step = uint64_t(ring_slot_bytes(bn) >> 4);
    int s = 0;
    uint64_t da = d0;
    CCK_TRACE_BEGIN_IF(2, el);
    CCK_TRACE_EV(0x60, gd.epi);
    for (int t = tb; t < te; t += ts, tile++) {
        const uint32_t buf = tile & 1, tpar = (tile >> 1) & 1;
        mbar_wait(&ctl->tempty[buf], tpar ^ 1, &ctl->abort);
        CCK_TRACE_EV(0x62, t); // the accumulator buffer is free
        const uint32_t acc = tmem + buf * kMaxBN;
        bool landed = false;
        for (int kb = 0; kb < kblocks; kb++) {
            if (!landed) {
                mbar_wait(&ctl->full[s], ring >> s & 1, &ctl->abort);
            }
            tc_fence_after();
            if (kb == 0) {
                CCK_TRACE_EV(0x64, t); // the first operands have landed
            }
            const uint64_t d = da;
            const int cs = s;
            ring ^= 1u << s;
            if (++s < slots) {
                da += step;
            } else {
                s = 0, da = d0;
            }
            // (the next k-block's barrier is looked at under this one's MMAs: a wait that passes costs 88 cycles)
            landed = kb + 1 < kblocks && mbar_test_a(full + 8 * s, ring >> s & 1);
            umma_bf16_kblock_el(el, acc, d, d + (kStageA >> 4), idesc, kb);
            umma_commit_el(el, empty + 8 * cs);
        }
        umma_commit_el(el, tfull + 8 * buf);
        CCK_TRACE_EV(0x66, t); // the tile's last MMA is issued
    }
    CCK_TRACE_END();
    pipe.ring = ring, pipe.tile = tile;
}

// once per launch, by the whole CTA: barriers and the TMEM allocation
__device__ inline void gemm_init() {
    SmemCtl* ctl = smem_ctl();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxSlots; i++) {
            mbar_init(&ctl->full[i], 1);
            mbar_init(&ctl->empty[i], 1);
        }
        ctl->ring_bn = 0;
        ctl->parts[0] = ctl->parts[1] = ctl->parts[2] = ctl->parts[3] = 0;
        for (int i = 0; i < 2; i++) {
            mbar_init(&ctl->tfull[i], 1);
            mbar_init(&ctl->tempty[i], kWorkWarps);
        }
        ctl->abort = 0, ctl->quit = 0;
        ctl->t0 = 0;
        fence_mbar_init();
    }
    if (warp_id() == 0) {
        tmem_alloc(&ctl->tmem_base, kTmemCols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}
__device__ inline void gemm_fini() {
    tc_fence_before();
    __syncthreads();
    if (warp_id() == 0) {
        tmem_dealloc(smem_ctl()->tmem_base, kTmemCols);
    }
}

} // namespace cck
