// PTX wrappers and descriptor helpers shared by the tcgen05 / TMEM decode kernels: mbarriers with
// bounded waits, cp.async, named barriers, TMEM allocation / load / store, tcgen05.mma issue and
// commit, shared-memory matrix descriptors and instruction descriptors (kind::f8f6f4).
#pragma once

#include "mla_common.cuh"

namespace b200mla {
namespace sm100 {

constexpr long long WAIT_LIMIT_CYCLES = 2000000000LL;   // ~1 s: far beyond any legitimate wait of this kernel

// ----------------------------------------------------------------------------------------------
// PTX wrappers
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// may sleep up to `ns` nanoseconds
__device__ __forceinline__ bool mbar_try_for(uint64_t* bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(ns) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) { return mbar_try_for(bar, parity, 20000u); }
// Wait for completion number `n` (0-based) of the barrier; n = -1 passes at once.
// The wait is bounded: when it expires the thread raises the CTA's abort flag and carries on, and
// every later wait of the CTA returns at once.  Control flow never depends on the outcome, so all
// threads still meet at the same barriers; the results of such a launch are garbage and the
// kernel reports ST_TIMEOUT through the status word.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, int n, volatile int* abort_flag) {
    const uint32_t parity = (uint32_t)n & 1u;
    if (mbar_try(bar, parity)) return;
    const long long t0 = clock64();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try(bar, parity)) return;
        if ((it & 63u) == 0u) {
            if (*abort_flag) return;
            if (clock64() - t0 > WAIT_LIMIT_CYCLES) break;
        }
    }
    *abort_flag = 1;
}

// Copy-engine instructions by one elected lane of a converged warp, all operands warp-uniform.  (Issued by several divergent
// lanes they become a loop over the lanes, each turn moving every operand into uniform registers first: ~150 cycles.)
__device__ __forceinline__ void mbar_arrive_expect_tx_elect(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred P1;\n\t.reg .b32 e;\n\telect.sync e|P1, 0xffffffff;\n\t"
                 "@P1 mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
                 ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Tiled 2-D TMA loads of rows of 576 bytes: their four 128-byte columns to `lat` and PANEL bytes on from one to the next, the last 64 bytes
// to `rope`, by the two maps' boxes (PANEL and the columns x are multiples of 16 bytes).  Completion is counted in bytes on `bar`.  `policy`: see
// l2_evict_first_policy.  All five behind one election: with one each, and every operand brought into uniform registers each time, the boxes of a
// unit of 16 rows took 600 cycles.
// The box whose first row is y.
template <int PANEL>
__device__ __forceinline__ void tma_rows_box_elect(uint32_t lat, uint32_t rope, const void* lat_map, const void* rope_map, int y, uint64_t* bar, uint64_t policy) {
    static_assert(PANEL % 16 == 0, "TMA destinations");
    asm volatile(
        "{\n\t.reg .pred P1;\n\t.reg .b32 e, d1, d2, d3, x0, x1, x2, x3, x4;\n\telect.sync e|P1, 0xffffffff;\n\t"
        "mov.b32 x0, 0;\n\tmov.b32 x1, 128;\n\tmov.b32 x2, 256;\n\tmov.b32 x3, 384;\n\tmov.b32 x4, 512;\n\t"
        "add.u32 d1, %0, %7;\n\tadd.u32 d2, %0, 2*%7;\n\tadd.u32 d3, %0, 3*%7;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%2, {x0, %4}], [%5], %6;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [d1], [%2, {x1, %4}], [%5], %6;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [d2], [%2, {x2, %4}], [%5], %6;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [d3], [%2, {x3, %4}], [%5], %6;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%1], [%3, {x4, %4}], [%5], %6;\n\t}"
        ::"r"(lat), "r"(rope), "l"(lat_map), "l"(rope_map), "r"(y), "r"(smem_u32(bar)), "l"(policy), "n"(PANEL) : "memory");
}
// FOUR rows (y0..y3, any order, any distance), one below the other; the maps' boxes are one row high.  This GPU's memory only.
template <int PANEL>
__device__ __forceinline__ void tma_rows_gather4_elect(uint32_t lat, uint32_t rope, const void* lat_map, const void* rope_map, int y0, int y1, int y2, int y3,
                                                       uint64_t* bar, uint64_t policy) {
    static_assert(PANEL % 16 == 0, "TMA destinations");
    asm volatile(
        "{\n\t.reg .pred P1;\n\t.reg .b32 e, d1, d2, d3, x0, x1, x2, x3, x4;\n\telect.sync e|P1, 0xffffffff;\n\t"
        "mov.b32 x0, 0;\n\tmov.b32 x1, 128;\n\tmov.b32 x2, 256;\n\tmov.b32 x3, 384;\n\tmov.b32 x4, 512;\n\t"
        "add.u32 d1, %0, %10;\n\tadd.u32 d2, %0, 2*%10;\n\tadd.u32 d3, %0, 3*%10;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%2, {x0, %4, %5, %6, %7}], [%8], %9;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes.L2::cache_hint [d1], [%2, {x1, %4, %5, %6, %7}], [%8], %9;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes.L2::cache_hint [d2], [%2, {x2, %4, %5, %6, %7}], [%8], %9;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes.L2::cache_hint [d3], [%2, {x3, %4, %5, %6, %7}], [%8], %9;\n\t"
        "@P1 cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes.L2::cache_hint [%1], [%3, {x4, %4, %5, %6, %7}], [%8], %9;\n\t}"
        ::"r"(lat), "r"(rope), "l"(lat_map), "l"(rope_map), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(smem_u32(bar)), "l"(policy), "n"(PANEL) : "memory");
}
// Policy word for data that is read once (the cache rows): its lines are the first to leave L2, so the streaming
// megabytes do not push out what every launch needs again - the kernels' code, Q, the page table.
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint4& v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ void red_release(int* counter, int v) {
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(counter), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void or_release(int* word, int bits) {
    asm volatile("red.release.gpu.global.or.b32 [%0], %1;" ::"l"(word), "r"(bits) : "memory");
}
__device__ __forceinline__ int add_acq_rel(int* counter, int v) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(counter), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ int load_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// One thread looks at a counter (lower 16 bits) in global memory until it has reached `total`, for at most `cycles`.
__device__ __forceinline__ bool count_reached(const int* counter, int total, int cycles) {
    const long long t0 = clock64();
    do {
        if ((load_acquire(counter) & 0xffff) >= total) return true;
    } while (clock64() - t0 < cycles);
    return false;
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes));
}
// The barrier receives one arrival once all cp.async copies issued so far by this thread have landed.
__device__ __forceinline__ void cp_async_mbar_arrive_noinc(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void named_bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ bool named_bar_or(int id, int n, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 q, %3, 0;\n\t"
        "bar.red.or.pred p, %1, %2, q;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(r) : "r"(id), "r"(n), "r"((uint32_t)pred) : "memory");
    return r != 0;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Warp-wide forms: every lane of a converged warp executes them and one elected lane (the same one every time for a
// full mask) issues the instruction.  The surrounding loop then runs warp-uniformly, which keeps the descriptor
// arithmetic off the issuing thread's critical path: 34 MMAs of a decode tile issue in ~1370 cycles this way against
// ~1950 from a single thread inside an `if (lane == 0)` region (measured, M = 128, N = 16 / 32).
__device__ __forceinline__ void umma_f8_elect(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred P1, p;\n\t.reg .b32 r;\n\t"
        "elect.sync r|P1, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@P1 tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Four of them behind one election: D, A and B move by D_STEP columns, A_STEP and B_STEP bytes from one to the next; `first` for the first
// and `rest` for the others: whether D is accumulated into.  The steps are immediates, so that only the first descriptors have to be
// brought into uniform registers: 16 MMAs of M = 128, K = 32, N = 16 from one idle warp take 918 cycles one by one and 802 so, 39 each and
// some 190 from the last one to the commit's arrival (977 and 961 with N = 64, 48 each).
template <int D_STEP, int A_STEP, int B_STEP>
__device__ __forceinline__ void umma_f8_x4_elect(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t first, uint32_t rest) {
    static_assert(A_STEP % 16 == 0 && B_STEP % 16 == 0, "descriptors count in 16 bytes");
    asm volatile(
        "{\n\t.reg .pred P1, p, q;\n\t.reg .b32 r, d1, d2, d3;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
        "elect.sync r|P1, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "add.u32 d1, %0, %6;\n\tadd.u32 d2, %0, 2*%6;\n\tadd.u32 d3, %0, 3*%6;\n\t"
        "add.u64 a1, %1, %7;\n\tadd.u64 a2, %1, 2*%7;\n\tadd.u64 a3, %1, 3*%7;\n\t"
        "add.u64 b1, %2, %8;\n\tadd.u64 b2, %2, 2*%8;\n\tadd.u64 b3, %2, 3*%8;\n\t"
        "@P1 tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t"
        "@P1 tcgen05.mma.cta_group::1.kind::f8f6f4 [d1], a1, b1, %3, q;\n\t"
        "@P1 tcgen05.mma.cta_group::1.kind::f8f6f4 [d2], a2, b2, %3, q;\n\t"
        "@P1 tcgen05.mma.cta_group::1.kind::f8f6f4 [d3], a3, b3, %3, q;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(first), "r"(rest), "n"(D_STEP), "n"(A_STEP / 16), "n"(B_STEP / 16) : "memory");
}
__device__ __forceinline__ void umma_commit_elect(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred P1;\n\t.reg .b32 r;\n\t"
        "elect.sync r|P1, 0xffffffff;\n\t"
        "@P1 tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t addr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t addr, const float* v) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(addr) : "memory");
}

// Shared-memory matrix descriptor (tcgen05): start address, leading / stride byte offsets (all
// in 16-byte units), descriptor version 1, swizzle mode in the top bits.
constexpr uint64_t SWIZZLE_NONE = 0, SWIZZLE_128B = 2, SWIZZLE_64B = 4;
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint64_t swizzle) {
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3fffu) << 32) | (1ull << 46) | (swizzle << 61);
}
// Same layout, start address moved by `bytes` (the address field never carries: smem < 256 KB).
__device__ __forceinline__ uint64_t desc_advance(uint64_t desc, uint32_t bytes) { return desc + (uint64_t)(bytes >> 4); }
// Instruction descriptor, kind::f8f6f4: fp32 accumulate, e4m3 x e4m3.
__host__ __device__ constexpr uint32_t make_idesc(int m, int n, bool a_mn_major, bool b_mn_major) {
    return (1u << 4) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// packed fp32 pairs: one instruction, two IEEE fp32 operations
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpk2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// pack four floats into four e4m3 bytes (round to nearest even, saturating)
__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
    uint16_t lo, hi;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(lo) : "f"(a), "f"(b));
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(hi) : "f"(c), "f"(d));
    return (uint32_t)lo | ((uint32_t)hi << 16);
}
__device__ __forceinline__ float2 unpack_e4m3x2(uint16_t v) { return __half22float2(e4m3x2_to_half2(v)); }


}  // namespace sm100
}  // namespace b200mla
