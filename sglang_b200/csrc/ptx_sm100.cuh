// Inline-PTX wrappers for the Blackwell (sm_100a) features the GEMMs use: mbarriers, TMA tile
// loads and stores, tensor memory (TMEM) management, tcgen05.mma / commit / ld.  Every wait on an
// mbarrier is bounded: on expiry the caller records a status word and unwinds; nothing traps.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace sglb200 {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ---- programmatic dependent launch ----------------------------------------------------------
// A kernel launched with the programmatic-stream-serialization attribute may be scheduled while its predecessor in
// the stream is still running (once every CTA of the predecessor has called launch_dependents or exited);
// grid_dependency_wait() then blocks until the predecessor has completed and its writes are visible.  Both are
// no-ops in launches without the attribute.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Redistribution of the block's registers between warpgroups (four consecutive warps each, executed by all of them):
// the sum over the warpgroups must not exceed what the block was launched with.
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- mbarrier ------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Bounded waits.  Each probe (mbarrier.try_wait with a time hint) may suspend the thread for up to `kProbeHintNs`
// and resumes at once when the phase completes, so a waiting warp spends a couple of instructions per microsecond
// instead of competing for issue slots with the warps that have work.
constexpr uint32_t kProbeHintNs = 4000;
constexpr uint32_t kProbeLimit = 1u << 22;  // default number of probes after which a wait gives up (seconds)
constexpr uint32_t kProbesNone = 0xffffffffu;  // as a limit: give up without probing (exercises the give-up paths)
// Whether the phase has completed, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
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
// The same in two steps, so that the shared-memory round trip of the question (hundreds of clocks beside TMA writes and
// MMA operand reads) is not waited for where it is asked: `ask` leaves the outcome in a predicate register of the
// kernel, declared once with SGLB_MBAR_ASK_DECL, `answer` reads it.  The compiler knows nothing of that register, so
// `ask` returns a value that `answer` takes: that makes the answer depend on its question.  One question may be open at
// a time, and a kernel declares the register once (a second declaration in a scope does not assemble).  The outcome as
// an ordinary value cost 0.5 % of 4096 x 36864 x 7168 (1060.7 us against 1055.1): it is then waited for at the question.
#define SGLB_MBAR_ASK_DECL() asm volatile(".reg .pred sglb_asked;")
__device__ __forceinline__ uint32_t mbar_ask(uint32_t bar, uint32_t parity) {
  uint32_t asked;
  asm volatile("mbarrier.test_wait.parity.shared::cta.b64 sglb_asked, [%1], %2;\n\tmov.u32 %0, 0;"
               : "=r"(asked)
               : "r"(bar), "r"(parity)
               : "memory");
  return asked;
}
__device__ __forceinline__ bool mbar_answer(uint32_t asked) {
  uint32_t ok;
  asm volatile("selp.u32 %0, 1, %1, sglb_asked;" : "=r"(ok) : "r"(asked));
  return ok != 0;
}
// Up to `limit` probes in one asm block; true when the phase completed.
__device__ __forceinline__ bool mbar_probe(uint32_t bar, uint32_t parity, uint32_t limit) {
  if (limit == kProbesNone) return false;
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .u32 n;\n\t"
      "mov.u32 n, 0;\n"
      "QUIET_LOOP:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "@p bra QUIET_DONE;\n\t"
      "add.u32 n, n, 1;\n\t"
      "setp.lt.u32 p, n, %4;\n\t"
      "@p bra QUIET_LOOP;\n\t"
      "setp.ne.u32 p, 0, 0;\n"
      "QUIET_DONE:\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kProbeHintNs), "r"(limit)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_quiet(uint32_t bar, uint32_t parity) { return mbar_probe(bar, parity, kProbeLimit); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The same without ordering anything, for a hand-back of tensor memory only: there tcgen05.wait::ld and the fence before
// it order the reads, and a release would first wait for the thread's earlier accesses.  Shared memory that has been read
// goes back with a release (after a __syncwarp where one lane arrives for the warp).
__device__ __forceinline__ void mbar_arrive_relaxed_if(uint32_t bar, uint32_t pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "@p mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar),
      "r"(pred)
      : "memory");
}
// Arrive from the threads whose `pred` is set, without a branch around the instruction.
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, uint32_t pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar),
      "r"(pred)
      : "memory");
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// A load that stays where it is written: asked for early, its value is used much later.
__device__ __forceinline__ int ldg_here_s32(const int32_t* at) {
  int v;
  asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(at));
  return v;
}

__device__ __forceinline__ float ldg_here_f32(const float* at) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(at));
  return v;
}

__device__ __forceinline__ float4 lds_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// (a0, a1) += (r0, r1) * sc: one packed float32 FMA for two adjacent columns.
__device__ __forceinline__ void fma2(float& a0, float& a1, uint32_t r0, uint32_t r1, float sc) {
  asm("{\n\t.reg .b64 ra, rs, rc;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rs, {%4, %4};\n\t"
      "mov.b64 rc, {%0, %1};\n\t"
      "fma.rn.f32x2 rc, ra, rs, rc;\n\t"
      "mov.b64 {%0, %1}, rc;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "r"(r0), "r"(r1), "f"(sc));
}

// The same with a scale of its own per column.
__device__ __forceinline__ void fma2(float& a0, float& a1, uint32_t r0, uint32_t r1, float s0, float s1) {
  asm("{\n\t.reg .b64 ra, rs, rc;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rs, {%4, %5};\n\t"
      "mov.b64 rc, {%0, %1};\n\t"
      "fma.rn.f32x2 rc, ra, rs, rc;\n\t"
      "mov.b64 {%0, %1}, rc;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "r"(r0), "r"(r1), "f"(s0), "f"(s1));
}

// Two 32-bit words as one 64-bit register (shared-memory matrix descriptors are built from halves).
__device__ __forceinline__ uint64_t pack_f32x2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}

// ---- TMA tile loads (every CTA fetches its own tiles) ----------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// Four single rows r0..r3 of a 2-D tensor (its map's box is one row high), one below the other.
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int r0, int r1, int r2,
                                            int r3) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
      : "memory");
}

// ---- shared-memory accesses ---------------------------------------------------------------------
__device__ __forceinline__ void sts_64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ uint4 lds_128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float2 lds_f32x2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}

// ---- thread-block clusters (partial sums of a split K, exchanged through distributed shared memory) --------------
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// In two halves; every thread of the cluster takes part in each barrier.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// The address of `addr` (this CTA's shared memory) in the CTA of rank `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void sts_cluster_f32x4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ float2 lds_cluster_f32x2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}

// ---- TMA tile store (shared memory -> global, clipped to the tensor's extents) ---------------------
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Returns once every committed store of this thread has finished READING shared memory (the source may be
// overwritten; the global writes complete on their own).
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// Returns once every committed store of this thread has been performed (used before the kernel ends when the
// destination is another GPU's memory and a later kernel tells that GPU that the data is there).
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Orders this thread's ordinary shared-memory writes before later reads by the TMA engine.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void sts_128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// ---- tensor memory ---------------------------------------------------------------------------
// Whole-warp calls (.sync.aligned).  `slot` is a shared-memory word receiving the base address.
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc], e4m3 x e4m3 -> f32, issued by ONE thread.
__device__ __forceinline__ void mma_f8f6f4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The mbarrier receives one arrival when every tcgen05.mma issued so far by this thread has finished.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}


// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives lane (base_lane + i).
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// For the loads in front of it in straight-line code: with a branch between the loads and the wait a buffer of tensor memory
// was handed back, and written by the next MMA, before the last load had read it.
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 16 lanes x 8 N columns: per 8 columns a thread receives columns 2 (lane % 4), + 1 of lane (lane / 4) in r[0], r[1] and of
// lane (lane / 4 + 8) in r[2], r[3].
__device__ __forceinline__ void tmem_ld_16x256_x2(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_16x256_x4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_16x256_x8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x8.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                 "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr)
               : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld_16x256(uint32_t taddr, uint32_t* r) {
  if constexpr (N >= 8) {
    tmem_ld_16x256_x8(taddr, r);
    if constexpr (N > 8) tmem_ld_16x256<N - 8>(taddr + 64, r + 32);
  } else if constexpr (N >= 4) {
    tmem_ld_16x256_x4(taddr, r);
    if constexpr (N > 4) tmem_ld_16x256<N - 4>(taddr + 32, r + 16);
  } else {
    static_assert(N == 2, "even numbers of 8-column units");
    tmem_ld_16x256_x2(taddr, r);
  }
}

// Four 8 x 8 fragments of 16-bit values, one below the other (word k of a lane: row 8 k + lane / 4, columns 2 (lane % 4),
// + 1), transposed: the lane receives rows 8 (lane % 4) .. + 7 of column lane / 4.
__device__ __forceinline__ uint4 transpose_frags(const uint32_t (&m)[4], int lane) {
  uint32_t t[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)  // word k: column lane / 4, rows 8 k + 2 (lane % 4), + 1
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(t[k]) : "r"(m[k]));
  // the four lanes of a column exchange words: lane c keeps block c
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, (lane & 1) ? t[k] : t[k + 1], 1);
    if (lane & 1) t[k] = got; else t[k + 1] = got;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, (lane & 2) ? t[k] : t[k + 2], 2);
    if (lane & 2) t[k] = got; else t[k + 2] = got;
  }
  return make_uint4(t[0], t[1], t[2], t[3]);
}

// Instruction descriptor for kind::f8f6f4: e4m3 x e4m3 (formats 0/0), f32 accumulate (1 at bit 4),
// both operands K-major, N/8 at bit 17, M/16 at bit 24.
__host__ __device__ constexpr uint32_t make_idesc_e4m3_f32(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

}  // namespace ptx
}  // namespace sglb200
