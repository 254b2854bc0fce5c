// Shared device helpers for the sm_100a MoE kernels: bounded mbarrier waits, TMA loads
// (never with cluster multicast), tcgen05 MMA / TMEM access, descriptors.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace b200moe {

// Device error word values (written to status[0] of the workspace, first error wins).
enum : int {
    ERR_NONE = 0,
    ERR_WAIT_SMEM_EMPTY = 1,   // producer gave up waiting for a free shared-memory stage
    ERR_WAIT_SMEM_FULL = 2,    // MMA warp gave up waiting for TMA data
    ERR_WAIT_TMEM_EMPTY = 3,   // MMA warp gave up waiting for a free accumulator buffer
    ERR_WAIT_TMEM_FULL = 4,    // promotion warps gave up waiting for MMA results
    ERR_BAD_SCHEDULE = 5,      // unit decoded outside the expert tables
    ERR_WAIT_GROUP = 6,        // epilogue warps of one column group gave up waiting for each other (or for the work queue)
    // 7 = a rank gave up waiting for a peer's barrier flag (ep_p2p.cuh)
    ERR_WAIT_CHUNKS = 8,       // the finisher of a chunked unit gave up waiting for the other chunks' partial sums
};

constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;  // every device-side wait gives up after 2 s

// The (token, expert) pairs of a call, in token-major order, are cut into slices of SLICE_PAIRS pairs;
// the routing kernel histograms every slice separately so that the permutation can run one CTA per slice.
constexpr int SLICE_PAIRS = 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------- programmatic dependent launch
// A kernel launched with the programmatic-stream-serialization attribute may start while the
// kernel before it on the stream still runs; pdl_wait() blocks until that kernel has completed
// and its writes are visible (everything before it may only touch memory the previous kernel
// does not write); pdl_launch() lets the NEXT kernel on the stream begin its own prologue.
// Both are no-ops for a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One lane of a fully converged warp.  A warp whose lanes all run the same control flow and only pick the issuing lane
// here, at the instruction, keeps the operands of TMA and tcgen05 instructions in uniform registers; code that runs
// under `lane == 0` instead issues them several times slower (measured: a 128-K block's MMAs and commits 570 -> 260
// cycles of the issuing warp, its TMA loads 500 -> 250).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// One look at a barrier; never suspends the thread (try_wait may, for as long as the hardware likes).
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait whose answer is data, not control flow: `ok` becomes 0 when the wait gave up, and then every later wait with
// the same `ok` gives up after two tries.  For loops that cannot afford a vote and a branch per step (40 cycles of a
// promotion warp's ~450): the caller looks at `ok` once per piece of work, votes there and records the error.  It answers per
// lane, and lanes may leave it apart in time: a `__syncwarp` has to stand between it (or mbar_test) and anything that takes the
// whole warp.
__device__ __forceinline__ void mbar_wait_flag(uint32_t bar, uint32_t parity, uint32_t& ok) {
    const unsigned long long limit = ok ? WAIT_LIMIT_NS : 0ull;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u64 t0, t1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE;\n\t"
        "mov.u64 t0, %%globaltimer;\n\t"
        "AGAIN:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE;\n\t"
        "mov.u64 t1, %%globaltimer;\n\t"
        "sub.u64 t1, t1, t0;\n\t"
        "setp.lt.u64 q, t1, %3;\n\t"
        "@q bra AGAIN;\n\t"
        "mov.u32 %0, 0;\n\t"
        "DONE:\n\t}"
        : "+r"(ok) : "r"(bar), "r"(parity), "l"(limit) : "memory");
}
// Keeps the compiler from drawing conclusions about a flag at the place where the paths that set it meet.  Without it
// the code that follows a wait is duplicated for "the first try succeeded" and "a later one did", and again for every wait
// after that: the GEMM kernels grew to two and a half times their size, and their epilogues no longer stayed in the
// instruction cache (20-30 k cycles for the first one of a launch, from L2 under full load, instead of 4 k).
__device__ __forceinline__ bool merged(bool flag) {
    uint32_t f = flag;
    asm volatile("" : "+r"(f));
    return f != 0;
}
// Bounded wait.  Returns false (after recording `code` in *status, first error wins) when
// the phase did not complete within WAIT_LIMIT_NS; the caller then leaves its loop and
// falls through to the kernel's common teardown.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status, int code) {
    bool ok = mbar_try_wait(bar, parity);
    if (!ok) {
        const unsigned long long t0 = globaltimer_ns();
#pragma unroll 1
        for (uint32_t it = 1;; ++it) {
            ok = mbar_try_wait(bar, parity);
            if (ok || ((it & 0x3FFu) == 0 && globaltimer_ns() - t0 > WAIT_LIMIT_NS)) break;
        }
        if (!ok) atomicCAS(status, 0, code);
    }
    return merged(ok);
}

// The same by a converged warp, with a vote on the answer: the branch on it is then uniform for the compiler, and what the
// loop around it carries (stage, buffer, phase) stays in uniform registers, which TMA, tcgen05.mma and tcgen05.ld take
// their operands from.  (A 128-K block of four MMAs: 606 cycles of the issuing loop without, 513 with.)
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int* status, int code) {
    bool ok = __all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity));      // the usual case costs one try and one vote
    if (!ok) ok = __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, status, code));
    return merged(ok);
}
// Two barriers by a converged warp: both are tried before either answer is looked at (one round trip when both phases
// have completed), and the answers are voted on, so the control flow after it stays uniform for the compiler.
__device__ __forceinline__ bool mbar_wait_both(uint32_t bar_a, uint32_t parity_a, int code_a, uint32_t bar_b, uint32_t parity_b,
                                               int code_b, int* status) {
    const bool a = mbar_try_wait(bar_a, parity_a), b = mbar_try_wait(bar_b, parity_b);
    bool ok = __all_sync(0xFFFFFFFFu, a && b);
    if (!ok) {
        ok = mbar_wait(bar_a, parity_a, status, code_a);
        ok = mbar_wait(bar_b, parity_b, status, code_b) && ok;
        ok = __all_sync(0xFFFFFFFFu, ok);
    }
    return merged(ok);
}

// The wrappers below are one PTX instruction each; their bodies are fixed by the ISA (operand order, state spaces,
// qualifiers), so any sm_100a code base that wraps the same instructions reads alike.
// ---------------------------------------------------------------- TMA (non-multicast only)
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* m, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap* m, int x, int y,
                                                 uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%2, %3}], [%4], %5;"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(bar), "l"(policy) : "memory");
}
// Four arbitrary rows r0..r3 of a 2-D tensor (map encoded with one-row boxes), columns [x, x + box), land as four
// consecutive rows at dst (swizzled like a tiled load of the same rows).  A row index outside the tensor reads the
// fill value (zeros); x must be a multiple of 16 bytes like every TMA coordinate of the innermost dimension.
__device__ __forceinline__ void tma_gather4_2d(uint32_t dst, const CUtensorMap* m, int x, int r0, int r1, int r2, int r3,
                                               uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(bar) : "memory");
}
// A read of shared memory that a barrier hands back behind it: through the shared window, where loads and the arrival that
// follows them are performed in order.
__device__ __forceinline__ float4 ld_shared_f4(uint32_t src) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(src) : "memory");
    return v;
}
// Untiled bulk copy global -> shared; both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar) : "memory");
}
// Per-thread asynchronous 4-byte copy global -> shared, for values a thread needs several steps later
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// ... of 16 bytes, both addresses 16-byte aligned
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// ---------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, e4m3 x e4m3 -> f32, one K=32 step.
__device__ __forceinline__ void umma_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on an mbarrier when every tcgen05 op issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Shared-memory matrix descriptor: K-major tile of rows x 128 bytes, 128-byte swizzle,
// 8-row atoms 1024 bytes apart.  Fields: start address >> 4 at bit 0, leading byte offset
// (unused for swizzled K-major, set to 1) at bit 16, stride byte offset 1024 >> 4 at bit 32,
// descriptor version 1 at bit 46, layout type 2 (128-byte swizzle) at bit 61.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
    uint64_t d = (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// Instruction descriptor, kind::f8f6f4: D = f32 (1 at bit 4), A = B = e4m3 (0 at bits 7, 10),
// both K-major (0 at bits 15, 16), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t make_idesc_f8(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// 32 lanes x 32 bit, 16 consecutive columns: thread i of the warp gets lane (quarter*32 + i).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 256-bit global stores (sm_100): one full 32-byte sector per thread and instruction
__device__ __forceinline__ void st_global_v8(void* ptr, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e,
                                             uint32_t f, uint32_t g, uint32_t h) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(ptr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(e), "r"(f), "r"(g), "r"(h) : "memory");
}

// 256-bit global load of read-once data (sm_100), 32-byte aligned
__device__ __forceinline__ void ld_global_v8(const void* ptr, uint32_t* v) {
    asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(ptr) : "memory");
}

// e4m3 helpers
__device__ __forceinline__ uint16_t f32x2_to_e4m3x2(float lo, float hi) {
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return r;  // low byte = lo, high byte = hi
}
__device__ __forceinline__ float2 e4m3x2_to_f32x2(uint16_t v) {
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(v));
    __half2 h = *reinterpret_cast<__half2*>(&h2);
    return __half22float2(h);
}

}  // namespace b200moe
