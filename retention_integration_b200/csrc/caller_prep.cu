// What the reference's callers do between their projection GEMM and the operator, in one pass:
//
//   deploy/nanoGPT/model.py:66-84        qkvg = c_attn(x); split into q, k, v and the gate column;
//                                        log_g = logsigmoid(6.906768 + gate.float()); rotary on q and k
//                                        (interleaved pairs, :153-164); .contiguous() copies
//   deploy/models/powercoder/modeling_powercoder.py:152-159
//                                        the same with separate projections, logsigmoid without a bias
//                                        and the half-split rotary of :43-74
//
// Unfused that is six elementwise kernels and two copies over tensors the size of the
// activations.  Here one kernel reads the projection output once and writes Q [b,t,hq,d],
// K, V [b,t,h,d] (16 bit) and log_g [b,t,h] (fp32) in the layout the operator takes; a second one
// is its gradient.  HBM bound: every thread moves 16-byte vectors, a token's row of the input is
// read by consecutive threads, cos / sin come from a small fp32 table [t, d/2] that stays in L2.
//
// Arithmetic as deploy/nanoGPT/model.py:159-164: x * cos and rotate(x) * sin are rounded fp32
// products, their sum is rounded once more, then cast to the input's dtype (no fused multiply-add,
// so that the 16-bit results are the reference's bit for bit).

#include "host.cuh"
#include "sm100.cuh"

namespace pr {
namespace {

constexpr int kCpThreads = 256;
constexpr int kCpVectors = 4;  // 16-byte vectors per thread

// numerically safe log(sigmoid(x)) = min(x, 0) - log1p(exp(-|x|))
__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(__expf(-fabsf(x))); }

template <typename T>
__device__ __forceinline__ void unpack8(const uint4& v, float (&x)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 p = Pack2<T>::to_f32(w[k]);
    x[2 * k] = p.x;
    x[2 * k + 1] = p.y;
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  return make_uint4(Pack2<T>::from_f32(x[0], x[1]), Pack2<T>::from_f32(x[2], x[3]), Pack2<T>::from_f32(x[4], x[5]),
                    Pack2<T>::from_f32(x[6], x[7]));
}

// y = x cos + rot(x) sin with rot(x)[2i] = -x[2i+1], rot(x)[2i+1] = x[2i]; sign = -1 gives the
// transpose (the gradient).  Each product and the sum rounded separately.
__device__ __forceinline__ void rotate_pair(float x0, float x1, float c, float s, float sign, float* y0, float* y1) {
  *y0 = __fadd_rn(__fmul_rn(x0, c), __fmul_rn(-sign * x1, s));
  *y1 = __fadd_rn(__fmul_rn(x1, c), __fmul_rn(sign * x0, s));
}

struct CallerPrepParams {
  int t, h, hq, d;
  long long in_stride;    // elements between consecutive tokens of the projection output
  long long cs_bstride;   // floats between batch entries of cos / sin (0: one table for all)
  int half_split;         // 0: pairs (2i, 2i+1); 1: pairs (i, i + d/2)
  int gated;
  float gate_bias;
  size_t tokens;          // b * t
};

// A head row is cut into units: one 16-byte vector, or (half-split pairs) the two vectors that rotate into each other;
// the same cut for q, k and v heads.  A thread takes kCpVectors vectors of one token that sit at the same place of
// their heads, W units apart: one pair of table loads and one split of the index serve all of them, and all of a
// thread's loads are in flight together, which HBM needs (one vector per turn of a grid-stride loop, as this kernel had
// it, read the tables once per vector and took 82.7 us a pass at b1 t65536 h8 d64 against 77.4; two vectors per thread
// took 79.9, eight 77.7).  Consecutive threads take
// consecutive units, so a warp reads and writes 512 contiguous bytes per vector.  The index is split with 32-bit
// arithmetic whenever the problem allows (IDX = unsigned).
// GRAD: inputs are dQ, dK, dV, dlog_g and the saved projection output (for the gate's derivative);
// the output is the gradient with respect to the projection output.
template <typename T, bool GRAD, bool HALF, typename IDX>
__global__ void __launch_bounds__(kCpThreads, 4)
caller_prep_kernel(const CallerPrepParams p, const T* __restrict__ in, const float* __restrict__ cosT,
                   const float* __restrict__ sinT, T* __restrict__ Q, T* __restrict__ K, T* __restrict__ V,
                   float* __restrict__ log_g, T* __restrict__ grad_in) {
  constexpr int NV = HALF ? 2 : 1, R = kCpVectors / NV;  // vectors per unit, units per thread
  const int d = p.d, ur = d / 8 / NV;                    // units per head row
  const int heads = p.hq + 2 * p.h, n_rot = p.hq + p.h, hstep = (heads + R - 1) / R;
  const IDX W = (IDX)(hstep * ur);
  const float sign = GRAD ? -1.f : 1.f;
  const IDX idx = (IDX)blockIdx.x * kCpThreads + threadIdx.x;
  const IDX tok_i = idx / W;
  if (tok_i >= (IDX)p.tokens) return;
  const int u = (int)(idx - tok_i * W);
  const int head0 = u / ur, j = u - head0 * ur;
  const size_t tok = tok_i;
  const T* row_in = in + tok * p.in_stride;
  T* row_g = GRAD ? grad_in + tok * p.in_stride : nullptr;
  // the token's vector of Q, K or V
  auto dense = [&](int head) -> T* {
    T* base = head < p.hq ? Q + (tok * p.hq + head) * d
                          : (head < n_rot ? K + (tok * p.h + (head - p.hq)) * d : V + (tok * p.h + (head - n_rot)) * d);
    return base + j * 8;
  };

  uint4 v[R][NV];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int head = head0 + i * hstep;
    if (head < heads) {
      const T* src = GRAD ? dense(head) : row_in + (long long)head * d + j * 8;
#pragma unroll
      for (int k = 0; k < NV; ++k) v[i][k] = *reinterpret_cast<const uint4*>(src + k * (d / 2));
    }
  }
  // a gate rides with the first unit of its value head
  float gate[R], up[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int gh = head0 + i * hstep - n_rot;
    if (p.gated && j == 0 && gh >= 0 && gh < p.h) {
      gate[i] = float(row_in[(long long)heads * d + gh]) + p.gate_bias;
      if (GRAD) up[i] = log_g[tok * p.h + gh];
    }
  }
  // cosines and sines of this place: 4 pairs of a vector, or 8 of a unit of two
  constexpr int NP = 4 * NV;
  float c[NP], s[NP];
  if (head0 < n_rot) {
    const IDX batch = tok_i / (IDX)p.t;
    const size_t trow = (size_t)batch * p.cs_bstride + (size_t)(tok_i - batch * (IDX)p.t) * (d / 2) + j * NP;
#pragma unroll
    for (int k = 0; k < NP; k += 4) {
      *reinterpret_cast<float4*>(c + k) = *reinterpret_cast<const float4*>(cosT + trow + k);
      *reinterpret_cast<float4*>(s + k) = *reinterpret_cast<const float4*>(sinT + trow + k);
    }
  }

#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int head = head0 + i * hstep;
    if (head >= heads) break;
    if (head < n_rot) {
      float x[NV][8], y[NV][8];
#pragma unroll
      for (int k = 0; k < NV; ++k) unpack8<T>(v[i][k], x[k]);
      if constexpr (!HALF) {
#pragma unroll
        for (int e = 0; e < 4; ++e) rotate_pair(x[0][2 * e], x[0][2 * e + 1], c[e], s[e], sign, &y[0][2 * e], &y[0][2 * e + 1]);
      } else {
        // elements 8j..8j+7 pair with 8j + d/2 .. 8j + d/2 + 7
#pragma unroll
        for (int e = 0; e < 8; ++e) rotate_pair(x[0][e], x[NV - 1][e], c[e], s[e], sign, &y[0][e], &y[NV - 1][e]);
      }
#pragma unroll
      for (int k = 0; k < NV; ++k) v[i][k] = pack8<T>(y[k]);
    }
    T* dst = GRAD ? row_g + (long long)head * d + j * 8 : dense(head);
#pragma unroll
    for (int k = 0; k < NV; ++k) *reinterpret_cast<uint4*>(dst + k * (d / 2)) = v[i][k];
    const int gh = head - n_rot;
    if (p.gated && j == 0 && gh >= 0) {
      if (GRAD)
        row_g[(long long)heads * d + gh] = T(up[i] * (1.f / (1.f + __expf(gate[i]))));  // d/dx log sigmoid(x) = sigmoid(-x)
      else
        log_g[tok * p.h + gh] = log_sigmoid(gate[i]);
    }
  }
}

template <typename T>
int launch_caller_prep(bool grad, const CallerPrepParams& p, const void* in, const float* cosT, const float* sinT, void* Q,
                       void* K, void* V, float* log_g, void* grad_in, cudaStream_t s) {
  const int nv = p.half_split ? 2 : 1, r = kCpVectors / nv;
  const size_t per_tok = (size_t)((p.hq + 2 * p.h + r - 1) / r) * (p.d / 8 / nv);
  const size_t ctas = (p.tokens * per_tok + kCpThreads - 1) / kCpThreads;
  PR_REQUIRE(ctas < ((size_t)1 << 31), PR_ERR_BAD_ARG, "%zu CTAs exceed the grid limit", ctas);
  const unsigned grid = (unsigned)ctas;
  const bool small = ctas * kCpThreads < ((size_t)1 << 32);  // the index may not wrap
#define PR_LAUNCH_CP(G, H)                                                                                         \
  do {                                                                                                             \
    if (small)                                                                                                     \
      caller_prep_kernel<T, G, H, unsigned><<<grid, kCpThreads, 0, s>>>(                                           \
          p, static_cast<const T*>(in), cosT, sinT, static_cast<T*>(Q), static_cast<T*>(K), static_cast<T*>(V),    \
          log_g, static_cast<T*>(grad_in));                                                                        \
    else                                                                                                           \
      caller_prep_kernel<T, G, H, unsigned long long><<<grid, kCpThreads, 0, s>>>(                                 \
          p, static_cast<const T*>(in), cosT, sinT, static_cast<T*>(Q), static_cast<T*>(K), static_cast<T*>(V),    \
          log_g, static_cast<T*>(grad_in));                                                                        \
  } while (0)
  if (grad) {
    if (p.half_split) PR_LAUNCH_CP(true, true); else PR_LAUNCH_CP(true, false);
  } else {
    if (p.half_split) PR_LAUNCH_CP(false, true); else PR_LAUNCH_CP(false, false);
  }
#undef PR_LAUNCH_CP
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

int check_caller_prep(int dtype, int b, int t, int h, int hq, int d, long long in_stride, int gated, int half_split) {
  PR_REQUIRE(dtype == PR_BF16 || dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", dtype);
  PR_REQUIRE(b > 0 && t > 0 && h > 0 && hq > 0 && hq % h == 0, PR_ERR_BAD_ARG, "bad sizes b=%d t=%d h=%d hq=%d", b, t, h, hq);
  PR_REQUIRE(d % 8 == 0 && d >= 8 && (!half_split || d % 16 == 0), PR_ERR_BAD_ARG, "head dim %d", d);
  const long long need = (long long)(hq + 2 * h) * d + (gated ? h : 0);
  PR_REQUIRE(in_stride >= need && in_stride % 8 == 0, PR_ERR_BAD_ARG,
             "row stride %lld: at least %lld elements and a multiple of 8", in_stride, need);
  return PR_OK;
}

}  // namespace
}  // namespace pr

extern "C" int pr_caller_prep_fwd(int dtype, int b, int t, int h, int hq, int d, const void* qkvg, long long row_stride,
                                  const float* cos_table, const float* sin_table, long long table_bstride,
                                  int half_split, int gated, float gate_bias, void* Q, void* K, void* V, float* log_g,
                                  int device, void* stream) {
  using namespace pr;
  int rc = check_caller_prep(dtype, b, t, h, hq, d, row_stride, gated, half_split);
  if (rc) return rc;
  PR_REQUIRE(qkvg && cos_table && sin_table && Q && K && V && (!gated || log_g), PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE(aligned16(qkvg) && aligned16(cos_table) && aligned16(sin_table) && aligned16(Q) && aligned16(K) &&
                 aligned16(V) && table_bstride % 4 == 0,
             PR_ERR_BAD_ARG, "misaligned pointer");
  PR_CUDA(cudaSetDevice(device));
  CallerPrepParams p{t, h, hq, d, row_stride, table_bstride, half_split, gated, gate_bias, (size_t)b * t};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == PR_BF16
             ? launch_caller_prep<__nv_bfloat16>(false, p, qkvg, cos_table, sin_table, Q, K, V, log_g, nullptr, s)
             : launch_caller_prep<__half>(false, p, qkvg, cos_table, sin_table, Q, K, V, log_g, nullptr, s);
}

extern "C" int pr_caller_prep_bwd(int dtype, int b, int t, int h, int hq, int d, const void* qkvg, long long row_stride,
                                  const float* cos_table, const float* sin_table, long long table_bstride,
                                  int half_split, int gated, float gate_bias, const void* dQ, const void* dK,
                                  const void* dV, const float* dlog_g, void* dqkvg, int device, void* stream) {
  using namespace pr;
  int rc = check_caller_prep(dtype, b, t, h, hq, d, row_stride, gated, half_split);
  if (rc) return rc;
  PR_REQUIRE(qkvg && cos_table && sin_table && dQ && dK && dV && dqkvg && (!gated || dlog_g), PR_ERR_BAD_ARG,
             "null pointer");
  PR_REQUIRE(aligned16(qkvg) && aligned16(cos_table) && aligned16(sin_table) && aligned16(dQ) && aligned16(dK) &&
                 aligned16(dV) && aligned16(dqkvg) && table_bstride % 4 == 0,
             PR_ERR_BAD_ARG, "misaligned pointer");
  PR_CUDA(cudaSetDevice(device));
  CallerPrepParams p{t, h, hq, d, row_stride, table_bstride, half_split, gated, gate_bias, (size_t)b * t};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the kernel's Q, K, V, log_g arguments carry the incoming gradients in this direction
  void* q = const_cast<void*>(dQ);
  void* k = const_cast<void*>(dK);
  void* v = const_cast<void*>(dV);
  float* g = const_cast<float*>(dlog_g);
  return dtype == PR_BF16 ? launch_caller_prep<__nv_bfloat16>(true, p, qkvg, cos_table, sin_table, q, k, v, g, dqkvg, s)
                          : launch_caller_prep<__half>(true, p, qkvg, cos_table, sin_table, q, k, v, g, dqkvg, s);
}
