// Backward of the intra-chunk attention with respect to keys and values, merged with the
// state-path gradients (the reference's attn_bwd_dkdv, retention/_attention/triton.py:390-493,
// and the dV part of retention/_update_state/reference.py:55-60).
//
// A tile is 128 key rows of one (batch, chunk, kv head).  For every tile of 64 queries at or after the key
// tile, of every query head of the group:
//     S^T = K_J Q_I^T,  dP^T = V_J dO_I^T                (tensor cores)
//     p / l = (s S)^2 e^{a_i-a_j} / l_i,  dS = 2 s^2 S e^{a_i-a_j} (dP + delta_i) / l_i,  delta_i = -<O_i, dO_i>
//     dV += (P / l)^T dO_I,   dK += dS^T Q_I             (A operands from tensor memory)
//     da_j -= sum_i p dp                                 (gate gradient, key side)
// then the state path of the values, dV += phi(k~_j)^T (w (.) dS_m) with k~ the discounted
// key (same expansion pipeline as the forward read-out).  The epilogue adds the state-path
// key gradient (fp32, from the expansion-gradient kernel) and writes dK, dV.
//
// Three groups of four warps own the key rows, one row per thread in each group, and take the steps in turn, each in
// its own tensor-memory buffer; one warp issues TMA loads, one tcgen05.mma; two warps make, step by step in turn and up to
// six ahead, what the rows need of a step's queries (Cols).  One persistent CTA per SM takes over tile after tile
// (ClcRing); the next tile's gates and the state-path gradients are fetched before the write-out.
// Bound by the latency of a step's serial chain - S and dP products, barrier, tensor-memory loads, arithmetic, stores,
// barrier, dV and dK products - of which the three buffers overlap three, and by the end of a tile, where rows lie 2 KB
// apart, a line per lane and instruction.  The columns' factors (loads, two divisions, a logarithm, exponentials) are a
// chain of 1000-1900 clocks: on the row warps it stood in front of a step's own 1000-1500, and the TMA warp alone cannot
// keep up with it (467 -> 483 us).
// 490 -> 373 us at b1 t65536 h8 with chunks of 1024 and states (one group per CTA -> now); the factors on warps of their own
// instead of the row warps: 467 -> 413, 80 -> 68 at b4 t2048 h8 in one chunk, 119 -> 102 at b4 t5000 h2x4.
#include "host.cuh"
#include "layout.cuh"
#include "sm100.cuh"

namespace pr {

namespace dkv {
constexpr int HD = 64;
constexpr int NG = 3;                    // row groups, each with its own buffer in tensor memory
constexpr int NR = 7;                    // shared-memory ring: stages of 16 KB (a query and a dO tile, or two state blocks)
constexpr int NF = 2;                    // warps that make the columns' factors, step by step in turn
constexpr int NC = 2 * NG;               // steps whose factors are held; a multiple of NF
constexpr int W_TMA = 4 * NG, W_MMA = W_TMA + 1, W_COL = W_MMA + 1;
constexpr int THREADS = 32 * (W_COL + NF);
constexpr int TILE_BYTES = 128 * 128;   // 128 key rows x 64 features
constexpr int TW = 64;                  // queries per step
constexpr int QD_BYTES = TW * 128;      // one query or dO tile
constexpr int Z_BYTES = 64 * 128;
constexpr int R_BYTES = 2 * QD_BYTES;   // one ring stage
constexpr size_t SMEM = 1024 + 4 * TILE_BYTES + NR * R_BYTES;
// What the row warps need of a step's 64 queries: e^{a_i - r} / l_i (r = gate sum at the step's first query), 1 / l_i, a_i
// and deg * delta_i; r, log of the largest l_i, largest a_i - r.
struct alignas(16) Cols {
  float fs[TW], il[TW], aq[TW], de[TW];
  float4 top;
};
constexpr uint32_t TMEM_COLS = 512;
// A buffer is 128 columns: S and dP, overwritten by P / l and dS (the first half of each); in the state phase 256
// expanded entries.
constexpr uint32_t COL_DV = 0, COL_DK = 64;
__device__ __forceinline__ constexpr uint32_t col_b(int grp) { return 128u + 128u * (uint32_t)grp; }
}  // namespace dkv

struct ChunkDkvParams {
  int hq, h, n_chunks, c, tiles_per_chunk;
  int ratio;               // query heads per kv head
  Div by_tiles, by_ratio;
  int t, d;               // tokens (the last chunk may be shorter), features (a multiple of 16)
  int nblk;               // stages of 64 expanded rows of a state
  int state_chunk_hi;     // chunks <= this have a state-path dV term
  float scale;
  const float* a;         // [b, t, h] or null
  const float* A;         // [b, n, h] or null
  const float* dl;        // [b, t, hq]
  const float* l;         // [b, t, hq] row sums saved by the forward
  const float* dk_state;  // [b, t, h, d] fp32 or null
  void* dK;
  void* dV;
  int aligned32;          // dK and dV start on 32-byte boundaries
  int state_aligned32;    // dk_state does
  float* da_k;            // [b, t, h]
  int* status;
};

struct DkvTile {
  int chunk, kvhead, batch, row0, tok_chunk;
  int c;        // tokens of the chunk
  int qt0;      // first query tile that can see this key tile
  int n_steps;  // (query tiles from qt0 on) x (query heads of the group)
  int nI;       // state items of 256 expanded entries
  bool empty;   // past the end of a shorter last chunk
  __device__ __forceinline__ DkvTile(const ChunkDkvParams& p, const dim3& cta) {
    const int x = (int)cta.x;
    int tile_j;
    p.by_tiles.of(x, &chunk, &tile_j);  // the longest tiles of a head first
    kvhead = (int)cta.y;
    batch = (int)cta.z;
    row0 = tile_j * 128;
    tok_chunk = chunk * p.c;
    c = min(p.c, p.t - tok_chunk);
    empty = row0 >= c;
    qt0 = row0 / dkv::TW;
    n_steps = empty ? 0 : ((c + dkv::TW - 1) / dkv::TW - qt0) * p.ratio;
    nI = (!empty && chunk <= p.state_chunk_hi) ? p.nblk / 4 : 0;
  }
};

// One 16-column piece of a step for one key row: P / l into `pk`, dS into `dk`, deg times the row sum of p * dp into
// acc.  SEP: the gate factor is c_j * fq[col] (c_j carries s^deg, fq 1 / l); otherwise s^deg e^{aq[col] - a_j} fq[col].
// de: deg * delta.  MASK: columns before `lo` (queries that precede this key) are dropped.
template <typename T, int DEG, bool SEP, bool MASK>
__device__ __forceinline__ void dkv_piece(const uint32_t (&sv)[16], const uint32_t (&pv)[16], const float* __restrict__ fq,
                                          const float* __restrict__ de, const float* __restrict__ aq, float c_j, float a_j,
                                          int lo, uint32_t (&pk)[8], uint32_t (&dk)[8], float2& acc) {
  // two columns per instruction: packed fp32 multiplies and FMAs
  const float4* f4 = reinterpret_cast<const float4*>(fq);
  const float4* d4 = reinterpret_cast<const float4*>(de);
  const float4* a4 = reinterpret_cast<const float4*>(aq);
  const float2 c2 = make_float2(c_j, c_j), deg2 = make_float2((float)DEG, (float)DEG);
#pragma unroll
  for (int j = 0; j < 16; j += 4) {
    const float4 f = f4[j >> 2], dq = d4[j >> 2];
    const float2 fv[2] = {make_float2(f.x, f.y), make_float2(f.z, f.w)};
    const float2 dv[2] = {make_float2(dq.x, dq.y), make_float2(dq.z, dq.w)};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int col = j + 2 * u;
      const float2 s = make_float2(__uint_as_float(sv[col]), __uint_as_float(sv[col + 1]));
      const float2 p = make_float2(__uint_as_float(pv[col]), __uint_as_float(pv[col + 1]));
      float2 g = __fmul2_rn(c2, fv[u]);
      if (!SEP) {
        const float4 a = a4[j >> 2];
        g.x *= __expf((u ? a.z : a.x) - a_j);
        g.y *= __expf((u ? a.w : a.y) - a_j);
      }
      if (MASK) {
        g.x = (col >= lo) ? g.x : 0.f;
        g.y = (col + 1 >= lo) ? g.y : 0.f;
      }
      const float2 sp = DEG == 4 ? __fmul2_rn(s, __fmul2_rn(s, s)) : s;  // S^(deg-1)
      const float2 sg = __fmul2_rn(sp, g);             // s^deg S^(deg-1) e^{a_i-a_j} / l_i
      const float2 dp = __ffma2_rn(p, deg2, dv[u]);    // deg (dP + delta)
      const float2 ds = __fmul2_rn(sg, dp);
      acc = __ffma2_rn(ds, s, acc);
      const float2 pw = __fmul2_rn(sg, s);
      pk[col >> 1] = Pack2<T>::from_f32(pw.x, pw.y);
      dk[col >> 1] = Pack2<T>::from_f32(ds.x, ds.y);
    }
  }
}

// A whole step: the loads of the next piece are in flight while one is computed.
template <typename T, int DEG, bool SEP, bool MASK>
__device__ __forceinline__ void dkv_step(uint32_t cb, const float* __restrict__ fq, const float* __restrict__ de,
                                         const float* __restrict__ aq, float c_j, float a_j, int lo, float& da) {
  uint32_t sv[2][16], pv[2][16], pk[8], dk[8];
  float2 acc = make_float2(0.f, 0.f);
  tmem_ld16(cb, sv[0]);
  tmem_ld16(cb + 64, pv[0]);
#pragma unroll
  for (int q = 0; q < dkv::TW / 16; ++q) {
    tmem_wait_ld();
    if (q + 1 < dkv::TW / 16) {
      tmem_ld16(cb + (q + 1) * 16, sv[(q + 1) & 1]);
      tmem_ld16(cb + 64 + (q + 1) * 16, pv[(q + 1) & 1]);
    }
    dkv_piece<T, DEG, SEP, MASK>(sv[q & 1], pv[q & 1], fq + q * 16, de + q * 16, aq + q * 16, c_j, a_j, lo - q * 16, pk, dk,
                                 acc);
    tmem_st8(cb + q * 8, pk);
    tmem_st8(cb + 64 + q * 8, dk);
  }
  da += acc.x + acc.y;
}

template <typename T, int DEG>
__global__ void __launch_bounds__(dkv::THREADS, 1)
chunk_dkv_kernel(const ChunkDkvParams p, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_q,
                 const __grid_constant__ CUtensorMap tm_dy, const __grid_constant__ CUtensorMap tm_ds) {
  using namespace dkv;
  extern __shared__ uint8_t smem_raw[];
  // kv_*: the key and value tiles, two pairs in flight.  r_*: the ring of operand tiles.  s_full: S and dP in a
  // group's buffer; op_full: the group has written its A operands.  c_full / c_free: a step's factors.  acc_full /
  // acc_free: accumulators complete / read out; rows: the row warps meet.
  __shared__ uint64_t kv_full[2], kv_free[2], r_full[NR], r_empty[NR], s_full[NG], op_full[NG], c_full[NC], c_free[NC],
      acc_full, acc_free, rows;
  __shared__ ClcRing clc;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ Cols sm_c[NC];
  __shared__ float sm_da[2][NG][128];

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (sbase - smem_u32(smem_raw));
  uint8_t* smKV = sm;                    // 2 x (key tile, value tile)
  // One ring serves both phases and all tiles: an attention step takes a stage (query tile, then dO tile), a state
  // item two (two 64-row state blocks each), so operands stream in while the steps before are still being computed.
  uint8_t* smR = smKV + 4 * TILE_BYTES;  // NR x R_BYTES

  if (warp == W_TMA) {
    if (elect_one()) {
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_dy);
      abort_flag = 0;
      for (int s = 0; s < 2; ++s) {
        mbar_init(&kv_full[s], 1);
        mbar_init(&kv_free[s], 4 * NG);
      }
      for (int s = 0; s < NR; ++s) {
        mbar_init(&r_full[s], 1);
        mbar_init(&r_empty[s], 1);
      }
      for (int s = 0; s < NG; ++s) {
        mbar_init(&s_full[s], 1);
        mbar_init(&op_full[s], 4);
      }
      for (int s = 0; s < NC; ++s) {
        mbar_init(&c_full[s], 1);
        mbar_init(&c_free[s], 4);
      }
      mbar_init(&acc_full, 1);
      mbar_init(&acc_free, 4 * NG);
      mbar_init(&rows, 4 * NG);
      clc_init(&clc, 4 * NG + 2 + NF);
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
  const int ratio = p.ratio;

  if (warp == W_TMA) {
    if (elect_one()) {
      bool ok = true;
      dim3 cta = blockIdx;
      int s = 0;           // ring stage and its phase
      uint32_t s_ph = 0;
      auto next_stage = [&]() -> uint8_t* {
        ok = ok && mbar_wait(&r_empty[s], s_ph ^ 1, &abort_flag);
        if (ok) mbar_expect_tx(&r_full[s], R_BYTES);
        return smR + s * R_BYTES;
      };
      auto advance = [&]() {
        if (++s == NR) s = 0, s_ph ^= 1;
      };
      for (int it = 0; ok; ++it) {
        const DkvTile w(p, cta);
        if (it >= 2) ok = mbar_wait(&kv_free[it & 1], ((it >> 1) - 1) & 1, &abort_flag);
        if (!ok) break;
        if (!w.empty) {
          uint8_t* kv = smKV + (it & 1) * 2 * TILE_BYTES;
          mbar_expect_tx(&kv_full[it & 1], 2 * TILE_BYTES);
          tma_load_4d(kv, &tm_k, &kv_full[it & 1], 0, w.kvhead, w.tok_chunk + w.row0, w.batch);
          tma_load_4d(kv + TILE_BYTES, &tm_v, &kv_full[it & 1], 0, w.kvhead, w.tok_chunk + w.row0, w.batch);
          int I = w.qt0, qh = w.kvhead * ratio;
          for (int st = 0; st < w.n_steps && ok; ++st) {
            uint8_t* dst = next_stage();
            if (!ok) break;
            tma_load_4d(dst, &tm_q, &r_full[s], 0, qh, w.tok_chunk + I * TW, w.batch);
            tma_load_4d(dst + QD_BYTES, &tm_dy, &r_full[s], 0, qh, w.tok_chunk + I * TW, w.batch);
            if (++qh == (w.kvhead + 1) * ratio) qh = w.kvhead * ratio, ++I;
            advance();
            if (st == 0) ok = clc_ask(&clc, it, &abort_flag);
          }
          const int blk0 = ((w.batch * p.n_chunks + w.chunk) * p.h + w.kvhead) * p.nblk;
          for (int k = 0; k < 2 * w.nI && ok; ++k) {
            uint8_t* dst = next_stage();
            if (!ok) break;
            tma_load_2d(dst, &tm_ds, &r_full[s], 0, (blk0 + 2 * k) * 64);
            tma_load_2d(dst + Z_BYTES, &tm_ds, &r_full[s], 0, (blk0 + 2 * k + 1) * 64);
            advance();
          }
        } else {
          mbar_arrive(&kv_full[it & 1]);  // nothing to load: the phase passes all the same
          ok = clc_ask(&clc, it, &abort_flag);
        }
        if (!ok || !clc_next(&clc, it, &cta, true, false, &abort_flag)) break;
      }
    }
  } else if (warp == W_MMA) {
    const uint32_t tmem = tmem_base_s;
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc(128, TW, Pack2<T>::is_bf16, false, false);
      const uint32_t idesc_o = umma_idesc(128, HD, Pack2<T>::is_bf16, false, true);
      // positions in the rotation: group and ring stage with the phases of op_full and r_full there, of the next
      // operand and of the next scores, which run NG operands ahead
      struct Pos {
        int g = 0, s = 0;
        uint32_t g_ph = 0, s_ph = 0;
        __device__ __forceinline__ void stage() {
          if (++s == NR) s = 0, s_ph ^= 1;
        }
        __device__ __forceinline__ void group() {
          if (++g == NG) g = 0, g_ph ^= 1;
        }
      } at, sc;
      // descriptors of stage 0; a stage on is R_BYTES >> 4 on in the address field
      const uint32_t ring = smem_u32(smR);
      const uint64_t d_qk = umma_desc_sw128(ring, 16, 1024), d_dk = umma_desc_sw128(ring + QD_BYTES, 16, 1024),
                     d_qm = umma_desc_sw128(ring, 8192, 1024), d_dm = umma_desc_sw128(ring + QD_BYTES, 8192, 1024);
      bool ok = true;
      dim3 cta = blockIdx;
      int tiles = 0;
      for (int it = 0; ok; ++it) {
        const DkvTile w(p, cta);
        if (!w.empty) {
          const uint32_t kv = smem_u32(smKV + (it & 1) * 2 * TILE_BYTES);
          const uint64_t d_k = umma_desc_sw128(kv, 16, 1024), d_v = umma_desc_sw128(kv + TILE_BYTES, 16, 1024);
          ok = mbar_wait(&kv_full[it & 1], (it >> 1) & 1, &abort_flag);
          auto issue_scores = [&]() -> bool {
            if (!mbar_wait(&r_full[sc.s], sc.s_ph, &abort_flag)) return false;
            tc_fence_after();
            const uint32_t off = (uint32_t)sc.s * (R_BYTES >> 4), cb = tmem + col_b(sc.g);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ss(cb, d_k + 2 * ks, d_qk + off + 2 * ks, idesc_s, ks > 0 ? 1u : 0u);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ss(cb + 64, d_v + 2 * ks, d_dk + off + 2 * ks, idesc_s, ks > 0 ? 1u : 0u);
            umma_commit(&s_full[sc.g]);
            sc.stage();
            sc.group();
            return true;
          };
          sc = at;
          for (int st = 0; st < min(w.n_steps, NG) && ok; ++st) ok = issue_scores();
          // the accumulators of the tile before have been read out
          if (ok && tiles > 0) ok = mbar_wait(&acc_free, (tiles - 1) & 1, &abort_flag);
          for (int st = 0; st < w.n_steps && ok; ++st) {
            ok = mbar_wait(&op_full[at.g], at.g_ph, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t off = (uint32_t)at.s * (R_BYTES >> 4), cb = tmem + col_b(at.g);
#pragma unroll
            for (int ks = 0; ks < TW / 16; ++ks)
              umma_ts(tmem + COL_DV, cb + ks * 8, d_dm + off + ks * (2048 >> 4), idesc_o, (st > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
            for (int ks = 0; ks < TW / 16; ++ks)
              umma_ts(tmem + COL_DK, cb + 64 + ks * 8, d_qm + off + ks * (2048 >> 4), idesc_o, (st > 0 || ks > 0) ? 1u : 0u);
            umma_commit(&r_empty[at.s]);
            at.stage();
            at.group();
            // the group's next scores, into the buffer that the products just issued read (products execute in order)
            if (st + NG < w.n_steps) ok = issue_scores();
          }
          for (int k = 0; k < w.nI && ok; ++k) {
            // 256 expanded entries against four state blocks (two ring stages)
            ok = mbar_wait(&op_full[at.g], at.g_ph, &abort_flag);
            for (int hf = 0; hf < 2 && ok; ++hf) {
              ok = mbar_wait(&r_full[at.s], at.s_ph, &abort_flag);
              if (!ok) break;
              tc_fence_after();
              const uint32_t off = (uint32_t)at.s * (R_BYTES >> 4), cb = tmem + col_b(at.g) + 64 * hf;
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                umma_ts(tmem + COL_DV, cb + ks * 8, d_qm + off + (ks >> 2) * (Z_BYTES >> 4) + (ks & 3) * (2048 >> 4), idesc_o, 1u);
              umma_commit(&r_empty[at.s]);
              at.stage();
            }
            at.group();
          }
          if (ok) umma_commit(&acc_full);
          ++tiles;
        }
        if (!ok || !clc_next(&clc, it, &cta, true, false, &abort_flag)) break;
      }
    }
  } else if (warp >= W_COL) {
    // ------------------------------------------------------- the columns' factors
    const bool gated = p.a != nullptr;
    bool ok = true;
    dim3 cta = blockIdx;
    int n0 = 0;  // steps before the tile
    for (int it = 0; ok; ++it) {
      const DkvTile w(p, cta);
      const size_t tok_base = (size_t)w.batch * p.t + w.tok_chunk;
      const float* a_chunk = gated ? p.a + tok_base * p.h + w.kvhead : nullptr;
      int st = (warp - W_COL - n0) & (NF - 1);
      int I, rem;  // the step's query tile, and its head within the group
      p.by_ratio.of(st, &I, &rem);
      I += w.qt0;
      // per-query values, two per lane, loaded one step ahead
      float av[2], dlv[2], lv[2], rs = 0.f;
      auto load_cols = [&]() {
        rs = gated ? a_chunk[(size_t)(I * TW) * p.h] : 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int qp = I * TW + lane + 32 * k;
          const bool v = qp < w.c;
          const size_t ix = (tok_base + qp) * p.hq + w.kvhead * ratio + rem;
          av[k] = !v ? -1e30f : gated ? a_chunk[(size_t)qp * p.h] : 0.f;
          dlv[k] = v ? p.dl[ix] : 0.f;
          lv[k] = v ? p.l[ix] : 0.f;  // 0: no such query
        }
      };
      if (st < w.n_steps) load_cols();
      for (; st < w.n_steps && ok; st += NF) {
        const int n = n0 + st, slot = n % NC;
        float log_l = 0.f;
        if (gated)
          log_l = __logf(__uint_as_float(
              __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(fabsf(lv[0]), fabsf(lv[1])), 1.f)))));
        const float top = warp_max(fmaxf(av[0], av[1]) - rs);
        float il[2], fs[2], de[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const bool v = I * TW + lane + 32 * k < w.c;
          il[k] = v ? safe_recip(lv[k]) : 0.f;
          fs[k] = v ? il[k] * __expf(av[k] - rs) : 0.f;
          de[k] = (float)DEG * dlv[k] * lv[k];
        }
        if (n >= NC) ok = __all_sync(0xffffffffu, mbar_wait(&c_free[slot], (n / NC - 1) & 1, &abort_flag));
        if (!ok) break;
        Cols& cl = sm_c[slot];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          cl.fs[lane + 32 * k] = fs[k];
          cl.il[lane + 32 * k] = il[k];
          cl.aq[lane + 32 * k] = av[k];
          cl.de[lane + 32 * k] = de[k];
        }
        if (lane == 0) cl.top = make_float4(rs, log_l, top, 0.f);
        __syncwarp();
        if (lane == 0) mbar_arrive(&c_full[slot]);
        for (rem += NF; rem >= ratio; rem -= ratio) ++I;
        if (st + NF < w.n_steps) load_cols();
      }
      n0 += w.n_steps;
      if (!ok || !clc_next(&clc, it, &cta, lane == 0, true, &abort_flag)) break;
    }
  } else {
    const uint32_t tmem = tmem_base_s;
    const int grp = warp >> 2, r = tid & 127;  // row group, key row inside the tile
    const int wrow = (warp & 3) * 32;
    const uint32_t lane_addr = (uint32_t)wrow << 16;
    const uint32_t cb = tmem + lane_addr + col_b(grp);
    const bool gated = p.a != nullptr;
    const float sdeg = DEG == 4 ? (p.scale * p.scale) * (p.scale * p.scale) : p.scale * p.scale;  // s^deg
    bool ok = true;
    dim3 cta = blockIdx;
    int tiles = 0;             // tiles with rows so far
    int grp0 = 0, g0 = 0, n0 = 0;  // group of the tile's first operand, ring stages and steps before the tile
    int last_g = -1;           // last ring stage that this group's latest operand was multiplied with
    uint32_t s_ph = 0, row_ph = 0;
    // the row warps meet; bounded like every wait
    auto meet = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(&rows);
      if (ok) ok = mbar_wait(&rows, row_ph, &abort_flag);
      row_ph ^= 1;
    };
    auto operand_written = [&](int g) {
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[grp]);
      last_g = g;
    };
    // gate sums of this thread's row and of the whole chunk, loaded before the write-out of the tile before
    float a_n = 0.f, A_n = 0.f;
    auto load_row = [&](const DkvTile& w) {
      a_n = A_n = 0.f;
      if (gated && w.row0 + r < w.c) {
        a_n = p.a[((size_t)w.batch * p.t + w.tok_chunk + w.row0 + r) * p.h + w.kvhead];
        if (w.nI > 0) A_n = p.A[(w.batch * p.n_chunks + w.chunk) * p.h + w.kvhead];
      }
    };
    load_row(DkvTile(p, cta));
    for (int it = 0; ok; ++it) {
      const DkvTile w(p, cta);
      bool more = false;
      if (!w.empty) {
        uint8_t* smK = smKV + (it & 1) * 2 * TILE_BYTES;
        const int row = w.row0 + r;  // key index inside the chunk
        const bool row_valid = row < w.c;
        const size_t tok_base = (size_t)w.batch * p.t + w.tok_chunk;
        const float a_j = a_n, A_c = A_n;
        float da = 0.f;  // deg times the row sum of p * dp
        const int first = (grp - grp0 + NG) % NG;  // this group's first operand in the tile
        int I, rem;
        p.by_ratio.of(first, &I, &rem);
        I += w.qt0;
        for (int st = first; st < w.n_steps && ok; st += NG) {
          const int qp0 = I * TW, n = n0 + st;
          const Cols& cl = sm_c[n % NC];
          ok = mbar_wait(&c_full[n % NC], (n / NC) & 1, &abort_flag);
          if (!ok) break;
          const float4 top = cl.top;
          const float rs = top.x;
          // The gate factor separates, e^{a_i - a_j} = e^{a_i - r} * e^{r - a_j}: one exponential per
          // key and per query instead of one per pair (both exponents <= 0 off the diagonal for gates
          // <= 0; a warp falls back to the per-pair form if one exceeds 80).  The query's factor also holds 1 / l_i, so
          // the key's exponent is tested together with the largest log l_i: near the diagonal, where the gates'
          // factors make up for each other, e^{a_i - r} / l_i would lose its bits below the smallest normal number
          // otherwise (15 % off in dK and dV with gates of -1.24 a token and row sums of 1e12).  It cannot grow too large:
          // l_i >= e^{a_i - r} (s q_i.k_r)^deg, the weight of the key at r.  Steps whose queries all
          // come after this warp's keys need no mask; a warp whose keys all come after the step's
          // queries writes zeros without reading the scores.
          const bool sep = !__any_sync(0xffffffffu, fmaxf(top.z, rs - a_j + top.y) > 80.f);
          const float c_j = sep ? sdeg * __expf(rs - a_j) : sdeg;
          ok = mbar_wait(&s_full[grp], s_ph, &abort_flag);
          s_ph ^= 1;
          if (!ok) break;
          tc_fence_after();
          const int wrow0 = w.row0 + wrow;
          if (qp0 + TW - 1 < wrow0 || wrow0 >= w.c) {
            uint32_t z[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = 0u;
            tmem_st16(cb, z);
            tmem_st16(cb + 16, z);
            tmem_st16(cb + 64, z);
            tmem_st16(cb + 80, z);
          } else {
            const bool mask = (wrow0 + 31 > qp0) || (wrow0 + 31 >= w.c);
            const int lo = row_valid ? row - qp0 : TW;  // first query column this key keeps
            if (!sep) dkv_step<T, DEG, false, true>(cb, cl.il, cl.de, cl.aq, c_j, a_j, lo, da);
            else if (mask) dkv_step<T, DEG, true, true>(cb, cl.fs, cl.de, cl.fs, c_j, a_j, lo, da);
            else dkv_step<T, DEG, true, false>(cb, cl.fs, cl.de, cl.fs, c_j, a_j, lo, da);
          }
          operand_written(g0 + st);
          if (lane == 0) mbar_arrive(&c_free[n % NC]);  // after the operand's __syncwarp
          for (rem += NG; rem >= ratio; rem -= ratio) ++I;
        }

        if (w.nI > 0) {
          meet();  // every score product of the tile has completed: the key tile may be rewritten
          // The discounted key takes the row's place in the key tile, where the expansion fetches its factors by a
          // runtime index; each group does every third 16-byte piece.
          if (ok) ok = mbar_wait(&kv_full[it & 1], (it >> 1) & 1, &abort_flag);
          float f = 1.f;
          if (gated) f = __expf(0.5f * (A_c - a_j));
          for (int j = grp; j < 8; j += NG) {
            uint4* slot = reinterpret_cast<uint4*>(smK + swz128(r, j));
            const uint4 v = *slot;
            uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 f2 = Pack2<T>::to_f32(x[k]);
              x[k] = Pack2<T>::from_f32(f2.x * f, f2.y * f);
            }
            *slot = make_uint4(x[0], x[1], x[2], x[3]);
          }
          meet();
          // items of 16 first factors x 16 second factors: block Y of second factors has Y + 1 of them
          int k = (grp - (grp0 + w.n_steps) % NG + NG) % NG;
          for (; k < w.nI; k += NG) {
            const int Y = (k > 0) + (k > 2) + (k > 5);
            const int a0 = 16 * (k - Y * (Y + 1) / 2);
            uint32_t x2[8], x[32];
            expand_second(smK, r, Y, x2);
            expand_stage<T>(smK, r, a0, x2, x);
            // the buffer is free once the products that read its last operand have completed
            if (ok && last_g >= 0) ok = mbar_wait(&r_empty[last_g % NR], (last_g / NR) & 1, &abort_flag);
            tc_fence_after();
            if (ok) tmem_st32(cb, x);
#pragma unroll
            for (int q = 1; q < 4; ++q) {
              expand_stage<T>(smK, r, a0 + 4 * q, x2, x);
              if (ok) tmem_st32(cb + 32 * q, x);
            }
            if (ok) operand_written(g0 + w.n_steps + 2 * k + 1);
          }
        }
        // the key and value tiles may be refilled (their last reads come before the async proxy's writes; the products
        // that read them have completed with the scores)
        fence_async_smem();
        sm_da[tiles & 1][first][r] = da;  // by step, not by group: a fixed order of the sum whatever the CTA did before
        // The groups share the write-out: 16 of the 64 columns of dV (units 0-3) or dK (units 4-7) at a time.  The
        // state-path gradients come in while the rows meet and the last products run, and the next tile's gates too.
        const size_t tok = tok_base + row;
        const float* st = p.dk_state ? p.dk_state + (tok * p.h + w.kvhead) * p.d : nullptr;
        constexpr int UNITS = (8 + NG - 1) / NG;
        float add[UNITS - 1][2][8];
#pragma unroll
        for (int i = 1; i < UNITS; ++i) {
          const int unit = grp + NG * i, c0 = 16 * (unit & 3);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int k = 0; k < 8; ++k) add[i - 1][j][k] = 0.f;
            if (st != nullptr && row_valid && unit >= 4 && unit < 8 && c0 < p.d) {
              if (p.state_aligned32) {
                ld_global_v8(st + c0 + 8 * j, add[i - 1][j]);
              } else {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const float4 v = reinterpret_cast<const float4*>(st + c0 + 8 * j)[k];
                  add[i - 1][j][4 * k] = v.x, add[i - 1][j][4 * k + 1] = v.y;
                  add[i - 1][j][4 * k + 2] = v.z, add[i - 1][j][4 * k + 3] = v.w;
                }
              }
            }
          }
        }
        meet();
        if (lane == 0) mbar_arrive(&kv_free[it & 1]);

        more = ok && clc_next(&clc, it, &cta, lane == 0, true, &abort_flag);
        if (more) load_row(DkvTile(p, cta));
        if (ok) ok = mbar_wait(&acc_full, tiles & 1, &abort_flag);
        tc_fence_after();
#pragma unroll
        for (int i = 0; i < UNITS; ++i) {
          const int unit = grp + NG * i, c0 = 16 * (unit & 3);
          if (!ok || unit >= 8) continue;
          uint32_t acc[16];
          tmem_ld16(tmem + lane_addr + 16 * unit, acc);
          tmem_wait_ld();
          if (row_valid && c0 < p.d) {
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float ad[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) ad[k] = i > 0 ? add[i > 0 ? i - 1 : 0][j >> 1][4 * (j & 1) + k] : 0.f;
              v[2 * j] = Pack2<T>::from_f32(__uint_as_float(acc[4 * j]) + ad[0], __uint_as_float(acc[4 * j + 1]) + ad[1]);
              v[2 * j + 1] =
                  Pack2<T>::from_f32(__uint_as_float(acc[4 * j + 2]) + ad[2], __uint_as_float(acc[4 * j + 3]) + ad[3]);
            }
            T* dst = static_cast<T*>(unit < 4 ? p.dV : p.dK) + (tok * p.h + w.kvhead) * p.d + c0;
            if (p.aligned32) {
              st_global_v8(dst, v);
            } else {
              reinterpret_cast<uint4*>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
              reinterpret_cast<uint4*>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_free);
        if (grp == 0 && row_valid) {
          const float sum = (sm_da[tiles & 1][0][r] + sm_da[tiles & 1][1][r]) + sm_da[tiles & 1][2][r];
          p.da_k[tok * p.h + w.kvhead] = (-1.f / DEG) * sum;
        }
        grp0 = (grp0 + w.n_steps + w.nI) % NG;
        g0 += w.n_steps + 2 * w.nI;
        n0 += w.n_steps;
        ++tiles;
      } else {
        // Not before the producer has come to this tile, and so has seen the last phase of this slot's kv_free: in a
        // run of empty tiles the row warps could pass it, and two phases on the parity that it waits for looks open.
        ok = mbar_wait(&kv_full[it & 1], (it >> 1) & 1, &abort_flag);
        __syncwarp();
        if (lane == 0) mbar_arrive(&kv_free[it & 1]);
        more = ok && clc_next(&clc, it, &cta, lane == 0, true, &abort_flag);
        if (more) load_row(DkvTile(p, cta));
      }
      if (!more) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && abort_flag) *p.status = ST_TIMEOUT;
  if (warp == 0) tmem_dealloc(tmem_base_s, TMEM_COLS);
}

}  // namespace pr

extern "C" int pr_chunk_dkv(int dtype, int b, int t, int hq, int h, int d, int c, const void* Q, const void* dO,
                            const void* K, const void* V, const void* wdS, const float* a, const float* A,
                            const float* dl, const float* l, const float* dk_state, int state_chunk_hi, float scale,
                            int deg, void* dK, void* dV, float* da_k, int device, void* stream) {
  using namespace pr;
  using namespace pr::dkv;
  PR_REQUIRE(deg == 2 || (deg == 4 && wdS == nullptr && dk_state == nullptr), PR_ERR_BAD_ARG,
             "deg=%d: states exist for deg 2; deg 4 runs state-free (attention only)", deg);
  PR_REQUIRE(head_dim_ok(d), PR_ERR_BAD_ARG, "head dim %d: a multiple of 16 up to 64", d);
  PR_REQUIRE(b > 0 && t > 0 && hq > 0 && h > 0 && hq % h == 0 && c > 0, PR_ERR_BAD_ARG,
             "bad sizes b=%d t=%d hq=%d h=%d c=%d", b, t, hq, h, c);
  PR_REQUIRE(dtype == PR_BF16 || dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", dtype);
  PR_REQUIRE(Q && dO && K && V && dl && l && dK && dV && da_k, PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE(aligned16(Q) && aligned16(dO) && aligned16(K) && aligned16(V) && aligned16(dK) && aligned16(dV) &&
                 aligned16(wdS) && aligned16(dk_state),
             PR_ERR_BAD_ARG, "misaligned pointer");
  PR_REQUIRE(!(wdS != nullptr && a != nullptr) || A != nullptr, PR_ERR_BAD_ARG,
             "gated state path needs the chunk gate totals A");
  PR_REQUIRE(h <= 65535 && b <= 65535, PR_ERR_BAD_ARG, "h and b must be <= 65535");
  PR_CUDA(cudaSetDevice(device));
  ChunkDkvParams p;
  p.hq = hq;
  p.h = h;
  p.n_chunks = chunks_of(t, c);
  p.t = t;
  p.d = d;
  p.nblk = ref_dim(d) / 64;
  p.c = c;
  p.tiles_per_chunk = (c + 127) / 128;
  p.ratio = hq / h;
  p.by_tiles = Div(p.tiles_per_chunk);
  p.by_ratio = Div(p.ratio);
  p.state_chunk_hi = wdS ? state_chunk_hi : -1;
  p.scale = scale;
  p.a = a;
  p.A = A;
  p.dl = dl;
  p.l = l;
  p.dk_state = dk_state;
  p.dK = dK;
  p.dV = dV;
  p.aligned32 = aligned32(dK) && aligned32(dV);
  p.state_aligned32 = aligned32(dk_state);
  p.da_k = da_k;
  int rc = status_word(device, &p.status, nullptr);
  if (rc) return rc;
  CUtensorMap tm_q, tm_dy, tm_k, tm_v, tm_ds;
  uint64_t dq_[4] = {(uint64_t)d, (uint64_t)hq, (uint64_t)t, (uint64_t)b};
  uint64_t sq[4] = {0, (uint64_t)d * 2, (uint64_t)hq * d * 2, (uint64_t)t * hq * d * 2};
  uint64_t dk[4] = {(uint64_t)d, (uint64_t)h, (uint64_t)t, (uint64_t)b};
  uint64_t sk[4] = {0, (uint64_t)d * 2, (uint64_t)h * d * 2, (uint64_t)t * h * d * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  uint32_t box_q[4] = {64, 1, (uint32_t)TW, 1};
  if ((rc = make_tmap(&tm_q, Q, 2, 4, dq_, sq, box_q, true))) return rc;
  if ((rc = make_tmap(&tm_dy, dO, 2, 4, dq_, sq, box_q, true))) return rc;
  if ((rc = make_tmap(&tm_k, K, 2, 4, dk, sk, box, true))) return rc;
  if ((rc = make_tmap(&tm_v, V, 2, 4, dk, sk, box, true))) return rc;
  if (wdS) {
    uint64_t dz[2] = {(uint64_t)d, (uint64_t)b * p.n_chunks * h * ref_dim(d)};
    uint64_t st[2] = {0, (uint64_t)d * 2};
    uint32_t bz[2] = {64, 64};
    if ((rc = make_tmap(&tm_ds, wdS, 2, 2, dz, st, bz, true))) return rc;
  } else {
    tm_ds = tm_q;
  }
  dim3 grid(p.tiles_per_chunk * p.n_chunks, h, b);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define PR_LAUNCH_DKV(TT, DG)                                                                                      \
  do {                                                                                                             \
    PR_SMEM_ATTR((chunk_dkv_kernel<TT, DG>), SMEM, device, true);                                                   \
    chunk_dkv_kernel<TT, DG><<<grid, THREADS, SMEM, s>>>(p, tm_k, tm_v, tm_q, tm_dy, tm_ds);                         \
  } while (0)
  if (dtype == PR_BF16) {
    if (deg == 4) PR_LAUNCH_DKV(__nv_bfloat16, 4); else PR_LAUNCH_DKV(__nv_bfloat16, 2);
  } else {
    if (deg == 4) PR_LAUNCH_DKV(__half, 4); else PR_LAUNCH_DKV(__half, 2);
  }
#undef PR_LAUNCH_DKV
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}
