// Device-side toolkit for sm_100a: mbarrier, TMA (each CTA loads its own tiles), TMEM and
// tcgen05 wrappers in inline PTX, plus the shared-memory swizzle used by the
// 128-byte-swizzled UMMA operand layouts.
//
// Every wait in this file is bounded: a wait that does not complete within
// PR_WAIT_BUDGET_NS sets the CTA's abort flag and returns false, the caller
// skips to its teardown (TMEM is released there) and the host reads a status
// word.  Nothing here traps, asserts or spins without a limit.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

namespace pr {

// compile-time loop: f(std::integral_constant<int, I>{}) for I in [I0, N)
template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}


#ifndef PR_WAIT_BUDGET_NS
#define PR_WAIT_BUDGET_NS 2000000000ull  // 2 s per wait, far above any kernel's run time
#endif

// status word values written by kernels (host maps them to error codes)
enum : int { ST_OK = 0, ST_TIMEOUT = 1, ST_BAD_ARG = 2 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// make generic-proxy shared-memory writes visible to the async proxy (TMA, tcgen05.mma)
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  `abort_flag` lives in shared memory and is shared by the CTA.  The slow
// path is kept out of line so that heavily unrolled callers stay small.
static __device__ __noinline__ bool mbar_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                   uint64_t budget_ns = PR_WAIT_BUDGET_NS) {
  const uint64_t t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (globaltimer_ns() - t0 > budget_ns) {
      *abort_flag = 1;
      return false;
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, abort_flag);
}
// The same wait with a caller-chosen budget (the self-test of the give-up path uses a few ms).
__device__ __forceinline__ bool mbar_wait_for(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                              uint64_t budget_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, abort_flag, budget_ns);
}

// The one thread of a converged warp that issues TMA copies and tcgen05.mma.  Not `lane == 0`: only elect.sync tells
// the compiler that a single thread runs the branch, so that descriptors go straight into uniform registers.
// Measured back to back at M = 128, N = 64, K = 16 with A in tensor memory: 32 clocks per product (the pipe's own
// rate) against 54 behind `lane == 0`, and more than that where the descriptors are computed in between.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.b32 %0, 1, 0, P;\n}" : "=r"(p));
  return p != 0;
}
// Index of the warp in its block, known to be the same in all of its threads.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

// ------------------------------------------------ programmatic dependent launch
// The inference kernels (decode.cu) are launched with programmatic stream serialisation allowed
// (host.cuh: launch()): their CTAs may become resident while the kernel before them in the stream
// is still draining, run their set-up (barrier initialisation, tensor-memory allocation, index
// arithmetic), and stop at pdl_wait() until that kernel has completed and its writes are visible.
// On a 25 us decode step this hides about 2 us.  (The training kernels are launched in plain stream
// order: measured with the same scheme they gained nothing at one head per GPU and lost 2 % at eight.)
// Rules such a kernel follows: EVERY thread executes pdl_wait() exactly once, before its first
// access to global memory and before any exit (a grid that completes without having waited would let
// its own dependents run ahead of the grid before it); pdl_launch_dependents() comes first, so
// the next grid may start as soon as all CTAs of this one are running.  Without the launch
// attribute both instructions do nothing.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// ------------------------------------------------------- taking over CTAs
// A persistent kernel keeps its grid: when a CTA has planned its tile, one thread asks for the index of a CTA of the
// same grid that has not been launched yet and the CTA does that one's work next (cluster launch control), so set-up,
// cold instruction fetches and the write-out of one tile overlap the next tile, and long and short tiles balance.
// Two responses in flight: `full` completes when a response has arrived (16 bytes), `empty` when every reading
// warp has taken it.
struct ClcRing {
  uint4 resp[2];
  uint64_t full[2], empty[2];
};
__device__ __forceinline__ void clc_init(ClcRing* c, uint32_t readers) {
  for (int i = 0; i < 2; ++i) {
    mbar_init(&c->full[i], 1);
    mbar_init(&c->empty[i], readers);
  }
}
// one thread asks for the tile after tile number `it`
__device__ __forceinline__ bool clc_ask(ClcRing* c, int it, volatile int* abort_flag) {
  const int s = it & 1;
  if (it >= 2 && !mbar_wait(&c->empty[s], ((it >> 1) - 1) & 1, abort_flag)) return false;
  mbar_expect_tx(&c->full[s], 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_u32(&c->resp[s])),
               "r"(smem_u32(&c->full[s]))
               : "memory");
  return true;
}
// Every reading warp (or its one issuing thread): the tile after tile number `it` into `x, y, z`; false when there is
// none.  `arrive`: this thread reports the warp's reading.
__device__ __forceinline__ bool clc_next(ClcRing* c, int it, dim3* next, bool arrive, bool warp_wide,
                                         volatile int* abort_flag) {
  const int s = it & 1;
  if (!mbar_wait(&c->full[s], (it >> 1) & 1, abort_flag)) return false;
  uint32_t got, x, y, z;
  asm volatile(
      "{\n .reg .b128 h;\n .reg .pred p;\n ld.shared.b128 h, [%4];\n"
      " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n selp.u32 %0, 1, 0, p;\n"
      " mov.u32 %1, 0;\n mov.u32 %2, 0;\n mov.u32 %3, 0;\n"
      " @p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, h;\n}"
      : "=r"(got), "=r"(x), "=r"(y), "=r"(z)
      : "r"(smem_u32(&c->resp[s]))
      : "memory");
  fence_async_smem();  // the read comes before the next response's write
  if (warp_wide) __syncwarp();
  if (arrive) mbar_arrive(&c->empty[s]);
  *next = dim3(x, y, z);
  return got != 0;
}

// --------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y,
                                            int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

// Untiled bulk copy global -> shared memory of this CTA: both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Tiled store shared -> global (bulk async group of the issuing thread).  Elements of the box that
// lie outside the tensor are not written.  x must be a multiple of 16 bytes; no coordinate negative.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// at most N of this thread's bulk groups still have to READ their shared-memory source
template <int N>
__device__ __forceinline__ void bulk_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
// at most N of this thread's bulk groups are still incomplete (their global writes not yet performed)
template <int N>
__device__ __forceinline__ void bulk_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// one full 32-byte sector per thread; `dst` 32-byte aligned
__device__ __forceinline__ void st_global_v8(void* dst, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// the same for a load of eight floats
__device__ __forceinline__ void ld_global_v8(const float* src, float (&v)[8]) {
  asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(src));
}

// -------------------------------------------------------------------- TMEM
// One full warp calls alloc / dealloc.  ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
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
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x N consecutive 32-bit columns; thread i of the warp gets lane (base lane + i).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
      "%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// ----------------------------------------------------------- UMMA descriptors
// 64-bit shared-memory matrix descriptor, 128-byte swizzle.
//   K-major  operand: rows (M or N index) of 128 bytes = 64 16-bit K elements,
//                     8-row groups `sbo` bytes apart; one MMA consumes 32 bytes of
//                     each row, so K-step k starts at base + 32*k bytes.
//   MN-major operand: rows (K index) of 128 bytes = 64 16-bit M/N elements,
//                     8-row groups `sbo` bytes apart, further 64-element blocks in
//                     M/N `lbo` bytes apart; K-step k starts at base + 16 rows.
// The tile base must be 1024-byte aligned so that the address-based XOR pattern
// (byte-address bits [4,7) ^= bits [7,10)) matches swz128() below.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}
// byte offset of 16-byte chunk `chunk` (0..7) of 128-byte row `row` in a swizzled tile
__device__ __forceinline__ uint32_t swz128(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

// 32-bit instruction descriptor for kind::f16 with fp32 accumulation.
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N, bool bf16, bool a_mn_major, bool b_mn_major) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; A is K-major in TMEM: lane = row, two 16-bit K
// elements per 32-bit column (8 columns per K=16 step).
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// mbarrier arrives once all MMAs issued so far by this thread have completed
// (implies tcgen05.fence::before_thread_sync).
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// the largest / smallest of a converged warp's values, in one instruction
__device__ __forceinline__ float warp_max(float x) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float warp_min(float x) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}

// 1 / l guarded against an exact zero only.  Row sums of real states are positive, but a
// caller may hand over any state, and the reference divides by negative sums too.
__device__ __forceinline__ float safe_recip(float l) {
  return 1.f / (fabsf(l) < 1e-37f ? copysignf(1e-37f, l) : l);
}

// ------------------------------------------------------------------ packing
template <typename T>
struct Pack2;
template <>
struct Pack2<__nv_bfloat16> {
  using V2 = __nv_bfloat162;
  static __device__ __forceinline__ uint32_t from_f32(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 to_f32(uint32_t u) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
  static constexpr bool is_bf16 = true;
};
template <>
struct Pack2<__half> {
  using V2 = __half2;
  static __device__ __forceinline__ uint32_t from_f32(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 to_f32(uint32_t u) {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
  static constexpr bool is_bf16 = false;
};
// Expansion of one stage of the block layout (see layout.cuh): the 64 entries of four
// consecutive first factors a0..a0+3 (a0 a multiple of 4) against the 16 second factors x2 of
// one block, as 32 packed products.  `r` is the thread's own gated row in the tile in shared memory
// (128 bytes, 128-byte swizzle); expand_second() fetches the block's second factors from it.
template <typename T>
__device__ __forceinline__ void expand_stage(const uint8_t* tile, int r, int a0, const uint32_t (&x2)[8],
                                             uint32_t (&out)[32]) {
  const uint2 h = *reinterpret_cast<const uint2*>(tile + swz128(r, a0 >> 3) + ((a0 & 7) << 1));
  const uint32_t xa[4] = {__byte_perm(h.x, h.x, 0x1010), __byte_perm(h.x, h.x, 0x3232),
                          __byte_perm(h.y, h.y, 0x1010), __byte_perm(h.y, h.y, 0x3232)};
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) out[8 * k + j] = Pack2<T>::mul(xa[k], x2[j]);
}
__device__ __forceinline__ void expand_second(const uint8_t* tile, int r, int Y, uint32_t (&x2)[8]) {
  const uint4 lo = *reinterpret_cast<const uint4*>(tile + swz128(r, 2 * Y));
  const uint4 hi = *reinterpret_cast<const uint4*>(tile + swz128(r, 2 * Y + 1));
  x2[0] = lo.x; x2[1] = lo.y; x2[2] = lo.z; x2[3] = lo.w;
  x2[4] = hi.x; x2[5] = hi.y; x2[6] = hi.z; x2[7] = hi.w;
}

}  // namespace pr
