// Host-side helpers shared by every entry point of the C ABI: error strings,
// CUDA error checks, the per-device status word that kernels write when a
// bounded wait runs out, and TMA tensor-map encoding through the driver entry
// point (no link-time dependency on libcuda).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../include/pr_b200.h"

namespace pr {

inline char* err_buf() {
  static thread_local char buf[512] = {0};
  return buf;
}
inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(err_buf(), 512, fmt, ap);
  va_end(ap);
  return code;
}

#define PR_CUDA(expr)                                                                          \
  do {                                                                                         \
    cudaError_t e__ = (expr);                                                                  \
    if (e__ != cudaSuccess)                                                                    \
      return ::pr::fail(PR_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), \
                        __FILE__, __LINE__);                                                   \
  } while (0)

#define PR_REQUIRE(cond, code, ...) \
  do {                              \
    if (!(cond)) return ::pr::fail(code, __VA_ARGS__); \
  } while (0)

// Per-device status word in mapped pinned host memory.  Kernels write a non-zero
// value only on failure, so the fast path costs nothing.
int status_word(int device, int** dev_ptr, volatile int** host_ptr);

// 2-D..4-D tiled tensor map with 128-byte swizzle (or none).  dims/strides are
// innermost first; strides[0] is implied (elem size) and strides[i] are bytes.
int make_tmap(CUtensorMap* out, const void* base, int elem_bytes, int rank, const uint64_t* dims,
              const uint64_t* strides_bytes, const uint32_t* box, bool swizzle128);

// A stack of `count` dense d x d 16-bit matrices as boxes of 64 x 64 (rows and columns past d read as zeros).
inline int gram_tmap(CUtensorMap* out, const void* base, int d, uint64_t count) {
  const uint64_t dims[3] = {(uint64_t)d, (uint64_t)d, count}, strides[3] = {0, (uint64_t)d * 2, (uint64_t)d * d * 2};
  const uint32_t box[3] = {64, 64, 1};
  return make_tmap(out, base, 2, 3, dims, strides, box, true);
}

// The kernels work on 64 features; narrower heads are widened with zeros by the TMA loads (boxes wider than the
// tensor) and only their own features are written back.
inline bool head_dim_ok(int d) { return d >= 16 && d <= 64 && d % 16 == 0; }

// Division by a number that is fixed for a launch: what a persistent CTA does to find its next tile's place would
// otherwise be a chain of integer divisions, about 150 clocks each, in front of every tile's first step (chunk_state
// 233 -> 201 us, chunk_dkv 414 -> 395, chunk_dq 202 -> 198 at b1 t65536 h8 with chunks of 1024).
// q = (mulhi(n, m) + n) >> s with s = ceil(log2 d), m = floor(2^32 (2^s - d) / d) + 1 is exact for 0 <= n < 2^31
// (T. Granlund, P. Montgomery, Division by invariant integers using multiplication, 1994).
struct Div {
  uint32_t d, m, s;
  Div() = default;
  explicit Div(int divisor) : d((uint32_t)divisor), s(0) {
    while ((1ull << s) < d) ++s;
    m = (uint32_t)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
  }
  __device__ __forceinline__ int of(int n) const { return (int)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s); }
  __device__ __forceinline__ void of(int n, int* q, int* r) const {
    *q = of(n);
    *r = n - *q * (int)d;
  }
};

// Chunks of a sequence of t tokens; the last one may be shorter.
inline int chunks_of(int t, int c) { return (t + c - 1) / c; }

// pr_chunk_out for sequences whose last chunk is shorter: tq queries and tk keys per batch element.
int chunk_out(int dtype, int b, int tq, int tk, int cq, int ck, int hq, int h, int d, const void* Q, const void* K,
              const void* V, const float* a, const void* Z, const void* zg_hi, const void* zg_lo, int state_from_chunk,
              int q_gate_last, int normalize, float scale, int deg, void* O, float* l_out, int device, void* stream);
// pr_dout_prep with dy optional.
int dout_prep(int dtype, long long rows, int d, const void* O, const void* dO, const float* l, void* dy, float* dl,
              int device, void* stream);
// pr_gate_prep / pr_chunk_state for the chunks [chunk0, chunk0 + n_run) only (pr_gate_prep: the copies; the gate sums are
// made for all); chunk_state for every head dim of head_dim_ok.
int gate_prep(int dtype, int b, int t, int h, int hx, int d, int c, const float* log_g, const void* x, float* a_out,
              float* A_out, void* xt, const float* row_scale, void* xts, int query_side, float mult, int write_a,
              int chunk0, int n_run, int device, void* stream);
int chunk_state(int dtype, int b, int t, int nh, int group, int d, int c, const void* xt, const void* xts, const void* v,
                void* out, float* gram, int key_weights, int chunk0, int n_run, int device, void* stream);

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
// what a thread's 32-byte stores want
inline bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

// Dynamic shared memory of a kernel: the attribute is raised once per kernel and device (and again only when a
// later launch needs more), not on every launch.  The record is kept per kernel function, not per call site: a
// second site that set a smaller size for the same kernel would lower the limit under the first one's launches.
// `carveout`: also ask for the largest shared-memory partition.
int smem_attr(const void* kernel, size_t bytes, int device, bool carveout);
#define PR_SMEM_ATTR(kernel, bytes, device, carveout)                                                    \
  do {                                                                                                   \
    int rc_ = ::pr::smem_attr(reinterpret_cast<const void*>(kernel), (bytes), (device), (carveout));     \
    if (rc_) return rc_;                                                                                 \
  } while (0)

// 0 when the environment variable PR_PDL=0 asks for plain stream order (read once).
bool pdl_enabled();

// Kernel launch with programmatic stream serialisation allowed (see pdl_wait() in sm100.cuh): the
// kernel may start while its predecessor in the stream drains and blocks at its own
// griddepcontrol.wait.  Stream capture records the edge as a programmatic dependency.
template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace pr
