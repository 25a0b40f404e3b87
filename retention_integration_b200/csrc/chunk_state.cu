// Token-contracting expansion kernel:  out[D2, e] = w (.) sum_i phi(x_i) v_i^T  per
// (batch, chunk, head), and the d x d Gram matrix  gram = sum_i xs_i x_i^T.
//
// Forward use (the reference's update_state, retention/_update_state/reference.py:31-53):
//   x = discounted keys, v = values, key weights on -> chunk state S_m; the Gram matrix
//   of the discounted keys carries the same information as the reference's sum_of_keys
//   N_m (N[(a,b)] = w(a,b) * gram[a][b]).
// Backward use (gradient of the state read-out, retention/_query_state/triton.py:337-448):
//   x = gated queries, v = dO / l, weights off -> dZ_m; xs = x * dl -> gram = d(gram of Z).
//
// An item is two tiles of 128 expanded rows of one state, so every operand stage fetched from L2 feeds two products, or a
// state's Gram matrix.  The expansion is never written to shared or global memory: a thread owns the expanded rows
// (a, b) and (a + 8, b) - the same row of both tiles, which share their second factor - multiplies rows a, a + 8 and b
// of the transposed operand (TMA-loaded, 128-byte swizzled) with packed 16-bit multiplies and stores the products
// straight into tensor memory as the A operands of tcgen05.mma; the values come in by TMA as the MN-major B operand;
// fp32 accumulation in tensor memory.
//
// One persistent CTA per SM takes over item after item (ClcRing).  Four groups of four warps take the 64-token stages in
// turn, each with a slot of its own in tensor memory; one thread per tile issues the products; four more warps write an
// item out from the first pair of accumulators while the next one fills the second.  A CTA per item spent half of its
// life on set-up, first loads and write-out.
// Bound by the shared-memory pipe, about 560 clocks a stage (the operand reads, 8 wavefronts for 16 products; the tensor
// core's own reads; tensor-memory stores) against 256 of the tensor pipe, and by 1500 clocks at the change of items.
// 252 -> 201 us (a CTA per item -> now) at b1 t65536 h8 with chunks of 1024, 83 -> 56 at b4 t4096 h2 with four query heads
// summed, 406 -> 365 at b16 t2048 h32 in one chunk, 15.1 -> 14.1 at b1 t2048 h2.
//
// EXACT (a token cache compressed into an inference state, retention/power_retention_maker.py:374-388): the read-out
// writes the state in the exact layout, state * e^a_last + the cache's part in fp32, and sum_of_keys from the Gram
// matrix.  Pairs that the block layout holds twice are written from one of their rows, with weight 2.  A pass of its
// own that converted and added cost 75 us at b16 t2048 h32, half as much again as the bytes it moved needed.
#include "host.cuh"
#include "layout.cuh"
#include "sm100.cuh"

namespace pr {

namespace cs {
constexpr int HD = 64;          // head dim handled by this build of the kernel
constexpr int NT = 2;           // tiles of 128 expanded rows per item: every loaded stage feeds both
constexpr int NG = 4;           // groups of 4 warps that expand the stages in turn
constexpr int NS = 8;           // shared-memory pipeline stages
constexpr int TOK = 64;         // tokens per stage
constexpr int W_OUT = 4 * NG, W_TMA = W_OUT + 4, W_MMA = W_TMA + 1;  // four write-out warps, one issuing warp per tile
constexpr int THREADS = 32 * (W_MMA + NT);
constexpr int XT_BYTES = HD * TOK * 2;   // 8 KB
constexpr int W_BYTES = TOK * HD * 2;    // 8 KB
constexpr int R_BYTES = XT_BYTES + W_BYTES;
constexpr size_t SMEM = 1024 + NS * R_BYTES + XT_BYTES;  // + the rows past a Gram operand, which the products read for nothing
constexpr uint32_t TMEM_COLS = 512;
__device__ __forceinline__ constexpr uint32_t col_acc(int tb, int tile) { return (uint32_t)(tb * NT + tile) * 64u; }
__device__ __forceinline__ constexpr uint32_t col_a(int grp, int tile) { return 256u + (uint32_t)(grp * NT + tile) * 32u; }
}  // namespace cs

struct ChunkStateParams {
  int n_slots;      // items of two tiles of 128 expanded rows per state
  int n_states;     // states (batch, chunk, head); grid.x = n_slots * n_states + (Gram matrices wanted ? n_states : 0)
  Div by_slots, by_heads, by_run;  // by n_slots, nh, n_run
  int nh;           // kv heads of the output
  int group;        // operand heads summed into one output head (GQA ratio in backward)
  int c, cp;        // chunk length, padded to 64
  int n_chunks;     // chunks per batch element
  int chunk0, n_run;  // the chunks that are wanted: n_run from chunk0 on
  int t, d;         // tokens (the last chunk may be shorter), features (a multiple of 16)
  int key_weights;  // 1: weight 2 on pairs from different 16-blocks; 0: all weights 1
  void* out;        // [b, n, nh, D2, 64]
  float* gram;      // [b, n, nh, 64, 64] or null
  // EXACT: the state to add to (null: none) with its sum_of_keys, the log decay [b, nh] (null: none), and the new
  // sum_of_keys; `out` is the new state [b, nh, d(d+1)/2, d], `gram` is not written
  const void* state;
  const float* sok;
  const float* a_last;
  float* new_sok;
  int* status;
};

// What a CTA index stands for: two tiles of 128 expanded rows of one state, or its Gram matrix.  The tiles of a state
// follow one another and share its operands through L2; the Gram matrices come last: they are short, which evens out
// the end of the launch.
struct StateItem {
  int slot, chunk, head, batch, ch, kblocks, total;
  bool gram;
  __device__ __forceinline__ StateItem(const ChunkStateParams& p, unsigned cta) {
    const unsigned n = (unsigned)p.n_slots * (unsigned)p.n_states;
    gram = cta >= n;
    int which = (int)(cta - n), rest;
    slot = 0;
    if (!gram) p.by_slots.of((int)cta, &which, &slot);
    p.by_heads.of(which, &rest, &head);
    p.by_run.of(rest, &batch, &chunk);
    chunk += p.chunk0;
    ch = (batch * p.n_chunks + chunk) * p.nh + head;
    kblocks = (min(p.c, p.t - chunk * p.c) + cs::TOK - 1) / cs::TOK;
    total = kblocks * p.group;
  }
};

template <typename T, bool EXACT>
__global__ void __launch_bounds__(cs::THREADS, 1)
chunk_state_kernel(const ChunkStateParams p, const __grid_constant__ CUtensorMap tm_xt,
                   const __grid_constant__ CUtensorMap tm_xs, const __grid_constant__ CUtensorMap tm_w) {
  using namespace cs;
  extern __shared__ uint8_t smem_raw[];
  // full: a stage's operands have arrived.  a_full: a group has written the expansion of its stage.  done: the products
  // of a stage have completed, which frees both the stage (TMA) and the group's slot in tensor memory.  A Gram matrix has
  // no expansions: the groups report on a_full that they have seen their last phases of `done` before its products start,
  // and wait for gram_done, or they could fall two phases behind, or be two ahead, on the ring's barriers.
  // acc_full / acc_free: an item's accumulators are complete / read out.
  __shared__ uint64_t full[NS], done[NS], a_full[NG], gram_done, acc_full[2], acc_free[2];
  __shared__ ClcRing clc;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smR = smem_raw + (sbase - smem_u32(smem_raw));  // NS x (rows = features, 64 tokens; rows = tokens, 64 features)

  if (warp == W_TMA) {
    if (elect_one()) {
      tma_prefetch_desc(&tm_xt);
      tma_prefetch_desc(&tm_w);
      abort_flag = 0;
      for (int s = 0; s < NS; ++s) {
        mbar_init(&full[s], 1);
        mbar_init(&done[s], NT);
      }
      for (int g = 0; g < NG; ++g) mbar_init(&a_full[g], 4);
      mbar_init(&gram_done, NT);
      for (int b = 0; b < 2; ++b) {
        mbar_init(&acc_full[b], NT);
        mbar_init(&acc_free[b], 4);
      }
      clc_init(&clc, 4 * NG + 4 + 1 + NT);
      fence_mbar_init();
    }
    __syncwarp();
    named_bar_arrive(1, THREADS);  // the first loads need not wait for the tensor memory
  } else {
    if (warp == 0) {
      tmem_alloc(&tmem_base_s, TMEM_COLS);
      tmem_relinquish();
    }
    tc_fence_before();
    named_bar_sync(1, THREADS);
    tc_fence_after();
  }

  if (warp == W_TMA) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      bool ok = true;
      dim3 cta = blockIdx;
      int s = 0;
      uint32_t ph = 1;
      for (int it = 0; ok; ++it) {
        const StateItem w(p, cta.x);
        int kb = 0, xhead = w.head * p.group;
        int xrow = ((w.batch * p.n_chunks + w.chunk) * (p.nh * p.group) + xhead) * p.d;
        for (int i = 0; i < w.total && ok; ++i) {
          ok = mbar_wait(&done[s], ph, &abort_flag);
          if (!ok) break;
          uint8_t* dst = smR + s * R_BYTES;
          mbar_expect_tx(&full[s], p.d * (TOK * 2) + (w.gram ? p.d * (TOK * 2) : W_BYTES));
          tma_load_2d(dst, &tm_xt, &full[s], kb * TOK, xrow);
          if (w.gram)
            tma_load_2d(dst + XT_BYTES, &tm_xs, &full[s], kb * TOK, xrow);
          else
            tma_load_4d(dst + XT_BYTES, &tm_w, &full[s], 0, xhead, w.chunk * p.c + kb * TOK, w.batch);
          if (i == 0) ok = clc_ask(&clc, it, &abort_flag);
          if (++kb == w.kblocks) kb = 0, ++xhead, xrow += p.d;
          if (++s == NS) s = 0, ph ^= 1;
        }
        if (!ok || !clc_next(&clc, it, &cta, true, false, &abort_flag)) break;
      }
    }
  } else if (warp >= W_MMA) {
    // ------------------------------------------------------------- MMA issuers
    // One thread per tile: a stage's four products of a tile take the tensor pipe 128 clocks, about what one thread
    // needs for the wait, the issue and the commit.
    if (elect_one()) {
      const uint32_t tmem = tmem_base_s;
      const int tl = warp - W_MMA;
      const uint32_t ring = smem_u32(smR);
      const uint32_t idesc = umma_idesc(128, HD, Pack2<T>::is_bf16, false, true);
      const uint32_t idesc_g = umma_idesc(128, HD / 2, Pack2<T>::is_bf16, false, false);
      const uint64_t d_w0 = umma_desc_sw128(ring + XT_BYTES, 8192, 1024);
      // the Gram matrix: each thread half of its columns
      const uint64_t d_g0 = umma_desc_sw128(ring + XT_BYTES, 16, 1024),
                     d_x0 = umma_desc_sw128(ring + tl * (HD / 2 * 128), 16, 1024);
      bool ok = true;
      dim3 cta = blockIdx;
      int s = 0, grp = 0;
      uint32_t ph = 0, a_ph = 0;
      for (int it = 0; ok; ++it) {
        const StateItem w(p, cta.x);
        const int tb = it & 1;
        if (it >= 2) ok = mbar_wait(&acc_free[tb], ((it >> 1) - 1) & 1, &abort_flag);
        if (w.gram) {
          const uint32_t acc = tmem + col_acc(tb, 0) + tl * (HD / 2);
          for (int j = 0; j < NG && ok; ++j) {
            ok = mbar_wait(&a_full[grp], a_ph, &abort_flag);
            if (++grp == NG) grp = 0, a_ph ^= 1;
          }
          for (int i = 0; i < w.total && ok; ++i) {
            ok = mbar_wait(&full[s], ph, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t off = (uint32_t)s * (R_BYTES >> 4);
#pragma unroll
            for (int ks = 0; ks < TOK / 16; ++ks)
              umma_ss(acc, d_g0 + off + 2 * ks, d_x0 + off + 2 * ks, idesc_g, (i > 0 || ks > 0) ? 1u : 0u);
            umma_commit(&done[s]);
            if (++s == NS) s = 0, ph ^= 1;
          }
          if (ok) umma_commit(&gram_done);
        } else {
          const uint32_t acc = tmem + col_acc(tb, tl);
          for (int i = 0; i < w.total && ok; ++i) {
            // the warps that wrote the operand have seen the stage's arrival
            ok = mbar_wait(&a_full[grp], a_ph, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint64_t d_w = d_w0 + (uint32_t)s * (R_BYTES >> 4);
            const uint32_t ca = tmem + col_a(grp, tl);
#pragma unroll
            for (int ks = 0; ks < TOK / 16; ++ks)
              umma_ts(acc, ca + ks * 8, d_w + ks * (2048 >> 4), idesc, (i > 0 || ks > 0) ? 1u : 0u);
            umma_commit(&done[s]);
            if (++s == NS) s = 0, ph ^= 1;
            if (++grp == NG) grp = 0, a_ph ^= 1;
          }
        }
        if (ok) umma_commit(&acc_full[tb]);
        if (!ok || !clc_next(&clc, it, &cta, true, false, &abort_flag)) break;
      }
    }
  } else if (warp >= W_OUT) {
    // ------------------------------------------------------------------ write-out
    const uint32_t tmem = tmem_base_s;
    const int row_in_tile = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    dim3 cta = blockIdx;
    for (int it = 0; ok; ++it) {
      const StateItem w(p, cta.x);
      const int tb = it & 1;
      const float decay = !EXACT || p.state == nullptr ? 0.f : (p.a_last ? __expf(p.a_last[w.ch]) : 1.f);
      ok = mbar_wait(&acc_full[tb], (it >> 1) & 1, &abort_flag);
      if (!ok) break;
      tc_fence_after();
      int a, b;
      ref_decode(w.slot * (NT * 128) + row_in_tile, &a, &b);
#pragma unroll 1
      for (int part = 0; part < 2 * NT; ++part) {
        // 32 columns of the row in tile part / 2
        const int tl = part >> 1, c0 = 32 * (part & 1);
        uint32_t acc[32];
        tmem_ld32(tmem + lane_addr + col_acc(tb, tl) + c0, acc);
        tmem_wait_ld();
        if (part == 2 * NT - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free[tb]);
        }
        const int ar = a + 8 * tl;  // the two tiles share their second factors
        if (w.gram) {
          if (tl == 0 && row_in_tile < p.d) {
            if (EXACT) {
              // row a of the Gram matrix holds the pairs (a, b >= a), which lie side by side
              const size_t at = (size_t)w.ch * exact_dim(HD) + exact_row(HD, row_in_tile, row_in_tile) - row_in_tile;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (c0 + j >= row_in_tile)
                  p.new_sok[at + c0 + j] = (p.sok != nullptr ? p.sok[at + c0 + j] * decay : 0.f) +
                                           __uint_as_float(acc[j]) * (c0 + j == row_in_tile ? 1.f : 2.f);
            } else {
              float4* dst = reinterpret_cast<float4*>(p.gram + ((size_t)w.ch * p.d + row_in_tile) * p.d + c0);
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (c0 + 4 * j < p.d)
                  dst[j] = make_float4(__uint_as_float(acc[4 * j]), __uint_as_float(acc[4 * j + 1]),
                                       __uint_as_float(acc[4 * j + 2]), __uint_as_float(acc[4 * j + 3]));
            }
          }
        } else if (EXACT) {
          if (ar <= b) {
            const float wgt = ar == b ? 1.f : 2.f;
            const size_t at = ((size_t)w.ch * exact_dim(HD) + exact_row(HD, ar, b)) * HD + c0;
            T* dst = static_cast<T*>(p.out) + at;
            const T* old = static_cast<const T*>(p.state) + at;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              uint4 o[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
              if (p.state != nullptr) {
                o[0] = *reinterpret_cast<const uint4*>(old + 16 * j);
                o[1] = *reinterpret_cast<const uint4*>(old + 16 * j + 8);
              }
              const uint32_t ow[8] = {o[0].x, o[0].y, o[0].z, o[0].w, o[1].x, o[1].y, o[1].z, o[1].w};
              uint32_t v[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                // the reference rounds state * decay to the state's dtype before adding (:374-382)
                const float2 raw = Pack2<T>::to_f32(ow[k]);
                const float2 od = Pack2<T>::to_f32(Pack2<T>::from_f32(raw.x * decay, raw.y * decay));
                v[k] = Pack2<T>::from_f32(od.x + wgt * __uint_as_float(acc[16 * j + 2 * k]),
                                          od.y + wgt * __uint_as_float(acc[16 * j + 2 * k + 1]));
              }
              st_global_v8(dst + 16 * j, v);
            }
          }
        } else {
          const float wgt = p.key_weights ? ref_key_weight(ar, b) : 1.f;
          T* dst = static_cast<T*>(p.out) + ((size_t)w.ch * (p.n_slots * NT * 128) + (w.slot * NT + tl) * 128 + row_in_tile) * p.d + c0;
          // 32-byte stores: a full sector per thread and instruction
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (c0 + 16 * j >= p.d) break;
            uint32_t v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
              v[k] = Pack2<T>::from_f32(wgt * __uint_as_float(acc[16 * j + 2 * k]), wgt * __uint_as_float(acc[16 * j + 2 * k + 1]));
            st_global_v8(dst + 16 * j, v);
          }
        }
      }
      if (!clc_next(&clc, it, &cta, lane == 0, true, &abort_flag)) break;
    }
  } else {
    // ------------------------------------------------------------------ expansion
    const uint32_t tmem = tmem_base_s;
    const int grp = warp >> 2;
    const int row_in_tile = (warp & 3) * 32 + lane;
    const uint32_t ca = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col_a(grp, 0);
    bool ok = true;
    dim3 cta = blockIdx;
    int g0 = 0, u0 = 0;  // stages and expansions before the item; expansion u is group u % NG's
    int grams = 0;       // Gram matrices so far
    int last_g = -1;     // the stage of this group's latest expansion
    auto slot_free = [&]() {  // its products have completed
      if (last_g >= 0) ok = mbar_wait(&done[last_g % NS], (last_g / NS) & 1, &abort_flag);
      tc_fence_after();
    };
    auto report = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[grp]);
    };
    for (int it = 0; ok; ++it) {
      const StateItem w(p, cta.x);
      if (!w.gram) {
        // this thread's row of both tiles: first factors a0 and a0 + 8, common second factor b
        int a0, b;
        ref_decode(w.slot * (NT * 128) + row_in_tile, &a0, &b);
        // swz128(row, j) = (row * 128 + ((row & 7) << 4)) ^ (j << 4): one XOR per address
        const uint32_t a0_base = a0 * 128 + ((a0 & 7) << 4), a1_base = a0_base + 8 * 128,
                       b_base = b * 128 + ((b & 7) << 4);
        for (int i = (grp - u0) & (NG - 1); i < w.total; i += NG) {
          const int g = g0 + i, s = g % NS;
          ok = mbar_wait(&full[s], (g / NS) & 1, &abort_flag);
          if (!ok) break;
          const uint8_t* xs = smR + s * R_BYTES;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t r0[16], r1[16];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
              const uint32_t off = (uint32_t)((4 * hf + jj) << 4);
              const uint4 vb = *reinterpret_cast<const uint4*>(xs + (b_base ^ off));
              const uint4 va = *reinterpret_cast<const uint4*>(xs + (a0_base ^ off));
              const uint4 vc = *reinterpret_cast<const uint4*>(xs + (a1_base ^ off));
              r0[4 * jj + 0] = Pack2<T>::mul(va.x, vb.x);
              r0[4 * jj + 1] = Pack2<T>::mul(va.y, vb.y);
              r0[4 * jj + 2] = Pack2<T>::mul(va.z, vb.z);
              r0[4 * jj + 3] = Pack2<T>::mul(va.w, vb.w);
              r1[4 * jj + 0] = Pack2<T>::mul(vc.x, vb.x);
              r1[4 * jj + 1] = Pack2<T>::mul(vc.y, vb.y);
              r1[4 * jj + 2] = Pack2<T>::mul(vc.z, vb.z);
              r1[4 * jj + 3] = Pack2<T>::mul(vc.w, vb.w);
            }
            if (hf == 0) {
              slot_free();
              if (!ok) break;
            }
            tmem_st16(ca + 16 * hf, r0);
            tmem_st16(ca + 32 + 16 * hf, r1);
          }
          if (!ok) break;
          last_g = g;
          // The stage goes back to TMA once its products have completed, which is after these stores, and so after
          // every load of it has delivered its data.  (Released right after the loads were issued, a refill overtook
          // loads still queued: single rows of the state were built from the wrong 64 tokens.)  The proxy fence orders
          // this thread's generic-proxy reads before the async-proxy write.
          fence_async_smem();
          tmem_wait_st();
          tc_fence_before();
          report();
        }
        u0 += w.total;
      } else {
        slot_free();
        if (!ok) break;
        last_g = -1;
        report();
        ok = mbar_wait(&gram_done, grams & 1, &abort_flag);
        ++grams;
      }
      g0 += w.total;
      if (!ok || !clc_next(&clc, it, &cta, lane == 0, true, &abort_flag)) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_flag) *p.status = ST_TIMEOUT;
  if (warp == 0) tmem_dealloc(tmem_base_s, TMEM_COLS);
}

template <typename T, bool EXACT>
static int launch_chunk_state(const ChunkStateParams& p, const CUtensorMap& tm_xt, const CUtensorMap& tm_xs,
                              const CUtensorMap& tm_w, cudaStream_t stream) {
  using namespace cs;
  int device = 0;
  PR_CUDA(cudaGetDevice(&device));  // the entry point has made the caller's device current
  PR_SMEM_ATTR((chunk_state_kernel<T, EXACT>), SMEM, device, true);
  dim3 grid((unsigned)((p.n_slots + (EXACT || p.gram ? 1 : 0)) * p.n_states));
  chunk_state_kernel<T, EXACT><<<grid, THREADS, SMEM, stream>>>(p, tm_xt, tm_xs, tm_w);
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

// Fills the sizes and tensor maps and launches.
template <bool EXACT>
static int run_chunk_state(int dtype, int b, int t, int nh, int group, int d, int c, const void* xt, const void* xts,
                           const void* v, ChunkStateParams p, int chunk0, int n_run, int device, void* stream) {
  if (n_run <= 0) return PR_OK;
  p.n_slots = ref_dim(d) / (cs::NT * 128);  // exact: 2, 6, 12 or 20 tiles
  // the items' indices are 32-bit (StateItem): counted before anything is narrowed
  const long long most = ((1ll << 31) - 1) / (p.n_slots + (EXACT || p.gram ? 1 : 0));
  PR_REQUIRE((long long)b * n_run <= most && (long long)b * n_run * nh <= most, PR_ERR_BAD_ARG,
             "b=%d, %d chunks and %d heads exceed the grid limit of %lld states", b, n_run, nh, most);
  PR_CUDA(cudaSetDevice(device));
  p.chunk0 = chunk0;
  p.n_run = n_run;
  p.n_states = b * n_run * nh;
  p.by_slots = Div(p.n_slots);
  p.by_heads = Div(nh);
  p.by_run = Div(n_run);
  p.nh = nh;
  p.group = group;
  p.c = c;
  p.cp = (c + 63) / 64 * 64;
  p.n_chunks = chunks_of(t, c);
  p.t = t;
  p.d = d;
  int rc = status_word(device, &p.status, nullptr);
  if (rc) return rc;
  const int hx = nh * group;
  CUtensorMap tm_xt, tm_xs, tm_w;
  {
    uint64_t dims[2] = {(uint64_t)p.cp, (uint64_t)b * p.n_chunks * hx * d};
    uint64_t strides[2] = {0, (uint64_t)p.cp * 2};
    uint32_t box[2] = {64, (uint32_t)d};
    rc = make_tmap(&tm_xt, xt, 2, 2, dims, strides, box, true);
    if (rc) return rc;
    rc = make_tmap(&tm_xs, xts, 2, 2, dims, strides, box, true);
    if (rc) return rc;
  }
  {
    uint64_t dims[4] = {(uint64_t)d, (uint64_t)hx, (uint64_t)t, (uint64_t)b};
    uint64_t strides[4] = {0, (uint64_t)d * 2, (uint64_t)hx * d * 2, (uint64_t)t * hx * d * 2};
    uint32_t box[4] = {64, 1, 64, 1};
    rc = make_tmap(&tm_w, v, 2, 4, dims, strides, box, true);
    if (rc) return rc;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return dtype == PR_BF16 ? launch_chunk_state<__nv_bfloat16, EXACT>(p, tm_xt, tm_xs, tm_w, s)
                          : launch_chunk_state<__half, EXACT>(p, tm_xt, tm_xs, tm_w, s);
}

}  // namespace pr

int pr::chunk_state(int dtype, int b, int t, int nh, int group, int d, int c, const void* xt, const void* xts,
                    const void* v, void* out, float* gram, int key_weights, int chunk0, int n_run, int device,
                    void* stream) {
  PR_REQUIRE(head_dim_ok(d), PR_ERR_BAD_ARG, "head dim %d: a multiple of 16 up to 64", d);
  PR_REQUIRE(b > 0 && t > 0 && nh > 0 && group > 0 && c > 0, PR_ERR_BAD_ARG,
             "bad sizes b=%d t=%d heads=%d group=%d c=%d", b, t, nh, group, c);
  PR_REQUIRE(dtype == PR_BF16 || dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", dtype);
  PR_REQUIRE(xt && v && out && aligned16(xt) && aligned16(v) && aligned32(out), PR_ERR_BAD_ARG,
             "null or misaligned pointer (out: 32 bytes)");
  PR_REQUIRE(gram == nullptr || (xts != nullptr && aligned16(xts) && aligned16(gram)), PR_ERR_BAD_ARG,
             "gram requested without a scaled operand");
  ChunkStateParams p{};
  p.key_weights = key_weights;
  p.out = out;
  p.gram = gram;
  return run_chunk_state<false>(dtype, b, t, nh, group, d, c, xt, gram ? xts : xt, v, p, chunk0, n_run, device, stream);
}

extern "C" int pr_chunk_state(int dtype, int b, int t, int nh, int group, int d, int c, const void* xt, const void* xts,
                              const void* v, void* out, float* gram, int key_weights, int device, void* stream) {
  PR_REQUIRE(d == pr::cs::HD, PR_ERR_BAD_ARG, "head dim %d: this entry point handles d = 64", d);
  return pr::chunk_state(dtype, b, t, nh, group, d, c, xt, xts, v, out, gram, key_weights, 0,
                         pr::chunks_of(t, c > 0 ? c : 1), device, stream);
}

extern "C" int pr_compress_cache(int dtype, int b, int tk, int h, int d, const void* xt, const void* v, const void* state,
                                 const float* sum_of_keys, const float* a_last, void* new_state, float* new_sum_of_keys,
                                 int device, void* stream) {
  using namespace pr;
  PR_REQUIRE(d == cs::HD, PR_ERR_BAD_ARG, "head dim %d: inference states are built for d = 64", d);
  PR_REQUIRE(b > 0 && tk > 0 && h > 0, PR_ERR_BAD_ARG, "bad sizes b=%d tk=%d h=%d", b, tk, h);
  PR_REQUIRE(dtype == PR_BF16 || dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", dtype);
  PR_REQUIRE(xt && v && new_state && new_sum_of_keys, PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE((state == nullptr) == (sum_of_keys == nullptr), PR_ERR_BAD_ARG, "state and sum_of_keys come together");
  PR_REQUIRE(aligned16(xt) && aligned16(v) && aligned16(state) && aligned32(new_state),
             PR_ERR_BAD_ARG, "misaligned pointer (new_state: 32 bytes)");
  ChunkStateParams p{};
  p.out = new_state;
  p.state = state;
  p.sok = sum_of_keys;
  p.a_last = a_last;
  p.new_sok = new_sum_of_keys;
  return run_chunk_state<true>(dtype, b, tk, h, 1, d, tk, xt, xt, v, p, 0, 1, device, stream);
}
