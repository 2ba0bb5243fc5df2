// Thin inline-PTX layer for sm_100a: mbarriers, TMA tile loads, tcgen05 (TMEM allocation, UMMA,
// commit, TMEM loads), proxy fences and the acquire/release accesses of the grid barrier.
// Every wait in this file is bounded: it gives up after kWaitCycles and reports through a flag.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

// Phase functions (what one operation of the schedule runs): out of line, called from the
// interpreter with nothing live in registers but addresses.
#ifndef CCK_PHASE_FN
#define CCK_PHASE_FN __noinline__
#endif
// The register-hungry ones are inlined into the kernel itself instead: out of line they would have
// to save and restore the registers that the calling convention preserves, in every phase.
#ifndef CCK_HOT_FN
#define CCK_HOT_FN __forceinline__
#endif

namespace cck {

// ~1 s at 1.9 GHz: far above any phase of a fold, far below a watchdog
constexpr long long kWaitCycles = 1ll << 31;
// The limit of this launch: kWaitCycles unless a test has shortened it (defined once the CTA's copy
// of the parameter block is known: gemm.cuh)
__device__ __forceinline__ long long wait_limit();

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ int lane_id() {
    return threadIdx.x & 31;
}
__device__ __forceinline__ int warp_id() {
    return threadIdx.x >> 5;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// ---- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// has the phase with this parity completed? Never blocks.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// mbar_try_wait with a suspend-time hint (ns): the thread sleeps in hardware until the phase completes or
// the time is over, instead of coming back to spin. A waiting thread then leaves its SM
// sub-partition's issue slots to the warps that share it.
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
// ---- Instructions for a role that a whole warp runs. Every lane passes the same loop; what must happen once is
// predicated on one elected lane (`el`) inside the statement instead of sitting in a one-lane branch. The
// operands of tcgen05 and TMA instructions live in the uniform register file, which the compiler feeds
// directly only where control flow is warp-uniform: in a branch of one thread a k-block of four
// tcgen05.mma, a wait and a commit took 541 cycles to issue whatever its width, in this form 260 at 128 columns
// (the rate of the tensor pipe) and 500 at 256; a wait and two TMA loads 309 against 253.
// uni(): the value of lane 0, which the compiler then knows to be the same in all lanes
__device__ __forceinline__ int uni(int v) {
    return __shfl_sync(0xffffffffu, v, 0);
}
__device__ __forceinline__ uint32_t uni(uint32_t v) {
    return __shfl_sync(0xffffffffu, v, 0);
}
__device__ __forceinline__ bool mbar_test_a(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_expect_tx_el(uint32_t el, uint32_t bar, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
        "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar),
        "r"(bytes), "r"(el)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d_el(uint32_t el, uint32_t smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
        :
        : "r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(el)
        : "memory");
}
// the same with an L2 policy: what is read once and not soon again is the first to leave
__device__ __forceinline__ uint64_t l2_policy(bool once) {
    uint64_t first, normal;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(normal));
    return once ? first : normal;
}
__device__ __forceinline__ void tma_load_2d_hint_el(uint32_t el, uint32_t smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar, uint64_t policy) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %6;\n\t}"
        :
        : "r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(el), "l"(policy)
        : "memory");
}
// one k-block of 64: four MMAs of K = 16 (32 bytes along k inside the 128-byte swizzle row: +2 in the
// descriptors' address field); the first one accumulates if `acc` is not zero
__device__ __forceinline__ void umma_bf16_kblock_el(uint32_t el, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q, e;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "add.u64 a, %1, 2;\n\tadd.u64 b, %2, 2;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n\t"
        "add.u64 a, %1, 4;\n\tadd.u64 b, %2, 4;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n\t"
        "add.u64 a, %1, 6;\n\tadd.u64 b, %2, 6;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n\t}"
        :
        : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(el)
        : "memory");
}
// three MMAs of K = 16: a head of 48
__device__ __forceinline__ void umma_bf16_k48_el(uint32_t el, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p, q, e;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 e, %4, 0;\n\tsetp.eq.b32 q, 0, 0;\n\tsetp.ne.b32 p, 0, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "add.u64 a, %1, 2;\n\tadd.u64 b, %2, 2;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n\t"
        "add.u64 a, %1, 4;\n\tadd.u64 b, %2, 4;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n\t}"
        :
        : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(el)
        : "memory");
}
// four MMAs of K = 16 with A in tensor memory (16 bf16 of k are 8 columns)
__device__ __forceinline__ void umma_bf16_ts_k64_el(uint32_t el, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q, e;\n\t.reg .b64 b;\n\t.reg .b32 a;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "add.u32 a, %1, 8;\n\tadd.u64 b, %2, 2;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, q;\n\t"
        "add.u32 a, %1, 16;\n\tadd.u64 b, %2, 4;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, q;\n\t"
        "add.u32 a, %1, 24;\n\tadd.u64 b, %2, 6;\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, q;\n\t}"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc), "r"(el)
        : "memory");
}
// the mbarrier gets one arrival when every MMA issued so far by this lane has completed
__device__ __forceinline__ void umma_commit_el(uint32_t el, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
        "r"(el)
        : "memory");
}

// Waits for the phase with the given parity. Returns false if it gave up; *abort (shared memory)
// is then set so that every later wait of the CTA returns at once.
#ifndef CCK_WAIT_HINT_NS
#define CCK_WAIT_HINT_NS 4000
#endif
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
    if (mbar_try_wait(bar, parity)) {
        return true;
    }
    const long long t0 = clock64();
    while (!mbar_try_wait_hint(bar, parity, CCK_WAIT_HINT_NS)) {
        if (*abort) {
            return false;
        }
        if (clock64() - t0 > wait_limit()) {
            *abort = 1;
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// ---- proxies
// generic-proxy writes (st.shared / st.global) made visible to the async proxy (TMA, UMMA)
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// generic-proxy accesses of global memory ordered with those of the async proxy: what the grid barrier needs on either side, and
// what the reader of a completion counter needs behind its acquire
__device__ __forceinline__ void fence_async_global() {
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

// ---- TMA stores (the loads are with the roles' instructions above)
// one 2D tile from shared memory to global memory (rows and columns past the tensor's extent are
// clipped), as part of this thread's bulk async-group
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* smem_src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                 :
                 : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int x, int y, int z, const void* smem_src) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 :
                 : "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// every bulk store of this thread has read its shared-memory source / has completed
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_done() {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with the
// 128-byte swizzle (what a TMA box of 64 bf16 x rows writes): 8-row groups are 1024 bytes apart.
// Fields: start address >> 4 in bits [0,14), leading byte offset >> 4 in [16,30) (unused for
// swizzled K-major, set to 1), stride byte offset >> 4 in [32,46), version 1 in [46,48),
// layout type 2 (128-byte swizzle) in [61,64).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= uint64_t((saddr & 0x3FFFFu) >> 4);
    d |= uint64_t(1) << 16;
    d |= uint64_t(1024 >> 4) << 32;
    d |= uint64_t(1) << 46;
    d |= uint64_t(2) << 61;
    return d;
}
// Instruction descriptor, kind::f16: f32 accumulator (bits [4,6) = 1), bf16 A and B (bits [7,10)
// and [10,13) = 1), both K-major (bits 15, 16 = 0), N >> 3 in [17,23), M >> 4 in [24,29).
__device__ __forceinline__ uint32_t umma_idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}
// 32 lanes x 32 consecutive f32 columns: thread l of the warp gets lane (base lane + l)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) {
        v[i] = __uint_as_float(r[i]);
    }
}
// the same load without the wait: the registers are valid only after tmem_ld_wait on them
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// waits for every TMEM load of this thread; the registers pass through the statement so that no
// use of them can be scheduled before it
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) {
        v[i] = __uint_as_float(r[i]);
    }
}

// ---- grid barrier accesses
__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_relaxed_add(unsigned int* p, unsigned int v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int atom_add_cta(unsigned int* p, unsigned int v) { // shared memory
    unsigned int old;
    asm volatile("atom.acq_rel.cta.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(smem_u32(p)), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// a counter read that orders nothing by itself: several can be in flight, one fence follows them
__device__ __forceinline__ unsigned int ld_relaxed(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void fence_acq_rel_gpu() {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
}

// ---- small math: the fast forms of the gate functions and the base-2 exponent
__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two at a time: a packed instruction costs the pipe what two scalar ones do, but it is one to fetch and to issue. A GEMM's
// epilogue is run from instructions that are mostly fetched anew (past 32 KB of code 6.5 cycles an instruction, within it
// 1.5 to 4, measured with straight-line code): ms per step against the scalar forms 32 x 1 0.892 -> 0.889, 64 x 5 1.022 ->
// 1.017, 256 x 5 1.485 -> 1.482, 512 x 5 2.283 -> 2.279.
__device__ __forceinline__ float2 tanh2(float2 x) {
    return make_float2(tanh_approx(x.x), tanh_approx(x.y));
}
__device__ __forceinline__ float2 sigmoid_fast2(float2 x) {
    const float2 half = make_float2(0.5f, 0.5f);
    return __ffma2_rn(half, tanh2(__fmul2_rn(x, half)), half);
}
__device__ __forceinline__ float2 silu_fast2(float2 x) {
    const float2 h = __fmul2_rn(x, make_float2(0.5f, 0.5f));
    return __ffma2_rn(h, tanh2(h), h);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Keeps a packed value packed until this point of the program: the compiler may not move the
// unpacking above it (which would hold the unpacked copy in twice the registers for longer)
__device__ __forceinline__ void keep_packed(uint2& u) {
    asm volatile("" : "+r"(u.x), "+r"(u.y));
}

// bf16 as raw bits, round to nearest even
__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
    uint32_t u;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u) : "f"(hi), "f"(lo));
    return u;
}
__host__ __device__ __forceinline__ float bf_to_f32(uint32_t b) {
    union {
        uint32_t u;
        float f;
    } c;
    c.u = b << 16;
    return c.f;
}
__device__ __forceinline__ float round_bf(float x) {
    return bf_to_f32(pack_bf2(x, 0.f) & 0xFFFFu);
}

} // namespace cck
