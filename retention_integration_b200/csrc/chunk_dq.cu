// Backward of the intra-chunk attention with respect to the queries, merged with the
// state-path query gradient (the reference's attn_bwd_dq, retention/_attention/triton.py:496-603,
// for deg = 2 without the division by the score).
//
// A tile is 128 query rows of one (batch, chunk, query head).  For every tile of 64 keys up to the diagonal:
//     S  = Q K_J^T,  dP = dO V_J^T                      (tensor cores, fp32 in tensor memory)
//     p  = (s S)^2 e^{a_i-a_j},  dp = dP / l_i + dl_i,  e = p dp,  dS = 2 s^2 S e^{a_i-a_j} dp
//     dQ += dS K_J                                      (A = dS from tensor memory)
//     da_i += sum_j e_ij                                (gate gradient, query side)
// with dl = -<O, dO> / l from the backward prologue.  dO enters the tensor cores unscaled and
// 1/l_i is applied in fp32, so the cancellation between dP / l and dl (exact for a row with a
// single key) is not spoiled by a 16-bit rounding of dO / l.  The epilogue adds the
// state-path gradient (fp32, from the expansion-gradient kernel) and writes dQ.
//
// Three groups of four warps own the query rows, one row per thread in each group, and take the steps in turn, each in
// its own tensor-memory buffer; one warp issues TMA loads, one tcgen05.mma; two warps make, step by step in turn and up to
// six ahead, the gate factors of a step's keys (Cols).  One persistent CTA per SM takes over tile after tile (ClcRing);
// a tile's row values are fetched before the write-out of the tile before.  Bound by the latency of a step's chain
// (products, barrier, tensor-memory loads, arithmetic, stores, barrier, product).
// 232 -> 196 us at b1 t65536 h8 with chunks of 1024 (one group per CTA, two CTAs per SM -> now); the factors on warps of their
// own instead of every row warp: 217 -> 202, 56 -> 52 at b4 t2048 h8 in one chunk.
#include "host.cuh"
#include "sm100.cuh"

namespace pr {

namespace dq {
constexpr int HD = 64;
constexpr int NG = 3;                    // row groups, each with its own buffer in tensor memory
constexpr int NR = 6;                    // shared-memory ring: stages of a key and a value tile
constexpr int NF = 2;                    // warps that make the columns' factors, step by step in turn
constexpr int NC = 2 * NG;               // steps whose factors are held; a multiple of NF
constexpr int W_TMA = 4 * NG, W_MMA = W_TMA + 1, W_COL = W_MMA + 1;
constexpr int THREADS = 32 * (W_COL + NF);
constexpr int TILE_BYTES = 128 * 128;   // 128 query rows x 64 features
constexpr int TW = 64;                  // keys per step
constexpr int KV_BYTES = TW * 128;      // one key or value tile
constexpr int R_BYTES = 2 * KV_BYTES;
constexpr size_t SMEM = 1024 + 4 * TILE_BYTES + NR * R_BYTES;
// What the row warps need of a step's 64 keys: e^{r - a_j} (r = gate sum at the step's last key) and a_j; r, smallest a_j.
struct alignas(16) Cols {
  float fk[TW], ak[TW];
  float2 top;
};
constexpr uint32_t TMEM_COLS = 512;
// the accumulator, then a buffer of 128 columns per group: S, overwritten by dS (its first half), and dP
__device__ __forceinline__ constexpr uint32_t col_b(int grp) { return 128u + 128u * (uint32_t)grp; }
}  // namespace dq

struct ChunkDqParams {
  int hq, h, n_chunks, c, tiles_per_chunk;
  Div by_tiles, by_ratio;  // by tiles_per_chunk, by query heads per kv head
  int t, d;               // tokens (the last chunk may be shorter), features (a multiple of 16)
  float scale;
  const float* a;         // [b, t, h] or null
  const float* dl;        // [b, t, hq]
  const float* l;         // [b, t, hq] row sums saved by the forward
  const float* dq_state;  // [b, t, hq, d] fp32 or null
  void* dQ;               // [b, t, hq, d]
  int aligned32;          // dQ starts on a 32-byte boundary
  int state_aligned32;    // dq_state does
  float* da_q;            // [b, t, hq]
  int* status;
};

struct DqTile {
  int chunk, qhead, kvhead, batch, row0, tok_chunk;
  int c;        // tokens of the chunk
  int nJ;       // steps: key tiles up to the diagonal
  bool empty;   // past the end of a shorter last chunk
  __device__ __forceinline__ DqTile(const ChunkDqParams& p, const dim3& cta) {
    const int x = (int)cta.x;
    // the longest tiles of a head first
    int tile_i;
    p.by_tiles.of(x, &chunk, &tile_i);
    tile_i = p.tiles_per_chunk - 1 - tile_i;
    qhead = (int)cta.y;
    batch = (int)cta.z;
    kvhead = p.by_ratio.of(qhead);
    row0 = tile_i * 128;
    tok_chunk = chunk * p.c;
    c = min(p.c, p.t - tok_chunk);
    empty = row0 >= c;
    nJ = empty ? 0 : min(c - 1, row0 + 127) / dq::TW + 1;
  }
};

// One 16-column piece of a step for one row: dS = deg s^deg S^(deg-1) g dp into `pk`, row sum of dS * S into acc.
// SEP: the gate factor is c_i * fk[col] (c_i carries deg s^deg); otherwise c_i e^{a_i - ak[col]} per pair.
// MASK: columns beyond `lim` (the row's own position, relative to the step) are dropped.
template <typename T, int DEG, bool SEP, bool MASK>
__device__ __forceinline__ void dq_piece(const uint32_t (&sv)[16], const uint32_t (&pv)[16], const float* __restrict__ fk,
                                         float c_i, float a_i, float inv_l, float dl_i, int lim, uint32_t (&pk)[8],
                                         float2& acc) {
  // two columns per instruction: packed fp32 multiplies and FMAs
  const float4* f4 = reinterpret_cast<const float4*>(fk);
  const float2 c2 = make_float2(c_i, c_i), il2 = make_float2(inv_l, inv_l), dl2 = make_float2(dl_i, dl_i);
#pragma unroll
  for (int j = 0; j < 16; j += 4) {
    const float4 f = f4[j >> 2];
    const float2 fv[2] = {make_float2(f.x, f.y), make_float2(f.z, f.w)};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int col = j + 2 * u;
      const float2 s = make_float2(__uint_as_float(sv[col]), __uint_as_float(sv[col + 1]));
      const float2 p = make_float2(__uint_as_float(pv[col]), __uint_as_float(pv[col + 1]));
      const float2 dp = __ffma2_rn(p, il2, dl2);
      float2 g;
      if (SEP) {
        g = __fmul2_rn(c2, fv[u]);
      } else {
        g = make_float2(c_i * __expf(a_i - fv[u].x), c_i * __expf(a_i - fv[u].y));
      }
      if (MASK) {
        g.x = (col <= lim) ? g.x : 0.f;
        g.y = (col + 1 <= lim) ? g.y : 0.f;
      }
      const float2 sp = DEG == 4 ? __fmul2_rn(s, __fmul2_rn(s, s)) : s;  // S^(deg-1)
      const float2 ds = __fmul2_rn(__fmul2_rn(sp, g), dp);  // deg s^deg S^(deg-1) e^{a_i-a_j} dp
      acc = __ffma2_rn(ds, s, acc);
      pk[col >> 1] = Pack2<T>::from_f32(ds.x, ds.y);
    }
  }
}

// A whole step: the loads of the next piece are in flight while one is computed.
template <typename T, int DEG, bool SEP, bool MASK>
__device__ __forceinline__ void dq_step(uint32_t cb, const float* __restrict__ fk, float c_i, float a_i, float inv_l,
                                        float dl_i, int lim, float& da) {
  uint32_t sv[2][16], pv[2][16], pk[8];
  float2 acc = make_float2(0.f, 0.f);
  tmem_ld16(cb, sv[0]);
  tmem_ld16(cb + 64, pv[0]);
#pragma unroll
  for (int q = 0; q < dq::TW / 16; ++q) {
    tmem_wait_ld();
    if (q + 1 < dq::TW / 16) {
      tmem_ld16(cb + (q + 1) * 16, sv[(q + 1) & 1]);
      tmem_ld16(cb + 64 + (q + 1) * 16, pv[(q + 1) & 1]);
    }
    dq_piece<T, DEG, SEP, MASK>(sv[q & 1], pv[q & 1], fk + q * 16, c_i, a_i, inv_l, dl_i, lim - q * 16, pk, acc);
    tmem_st8(cb + q * 8, pk);
  }
  da += acc.x + acc.y;
}

template <typename T, int DEG>
__global__ void __launch_bounds__(dq::THREADS, 1)
chunk_dq_kernel(const ChunkDqParams p, const __grid_constant__ CUtensorMap tm_q,
                const __grid_constant__ CUtensorMap tm_dy, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v) {
  using namespace dq;
  extern __shared__ uint8_t smem_raw[];
  // q_*: the query and dO tiles, two pairs in flight.  r_*: the ring of key and value tiles.  s_full: S and dP in a
  // group's buffer; op_full: the group has written dS.  c_full / c_free: a step's factors.  acc_full / acc_free:
  // accumulator complete / read out; rows: the row warps meet.
  __shared__ uint64_t q_full[2], q_free[2], r_full[NR], r_empty[NR], s_full[NG], op_full[NG], c_full[NC], c_free[NC],
      acc_full, acc_free, rows;
  __shared__ ClcRing clc;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ Cols sm_c[NC];
  __shared__ float sm_da[2][NG][128];

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (sbase - smem_u32(smem_raw));
  uint8_t* smQD = sm;                    // 2 x (query tile, dO tile)
  uint8_t* smR = smQD + 4 * TILE_BYTES;  // NR x R_BYTES

  if (warp == W_TMA) {
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_dy);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      abort_flag = 0;
      for (int s = 0; s < 2; ++s) {
        mbar_init(&q_full[s], 1);
        mbar_init(&q_free[s], 1);
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

  if (warp == W_TMA) {
    if (elect_one()) {
      bool ok = true;
      dim3 cta = blockIdx;
      int s = 0;           // ring stage and its phase
      uint32_t s_ph = 0;
      for (int it = 0; ok; ++it) {
        const DqTile w(p, cta);
        if (it >= 2) ok = mbar_wait(&q_free[it & 1], ((it >> 1) - 1) & 1, &abort_flag);
        if (!ok) break;
        if (!w.empty) {
          uint8_t* qd = smQD + (it & 1) * 2 * TILE_BYTES;
          mbar_expect_tx(&q_full[it & 1], 2 * TILE_BYTES);
          tma_load_4d(qd, &tm_q, &q_full[it & 1], 0, w.qhead, w.tok_chunk + w.row0, w.batch);
          tma_load_4d(qd + TILE_BYTES, &tm_dy, &q_full[it & 1], 0, w.qhead, w.tok_chunk + w.row0, w.batch);
          for (int J = 0; J < w.nJ; ++J) {
            if (!(ok = mbar_wait(&r_empty[s], s_ph ^ 1, &abort_flag))) break;
            mbar_expect_tx(&r_full[s], R_BYTES);
            tma_load_4d(smR + s * R_BYTES, &tm_k, &r_full[s], 0, w.kvhead, w.tok_chunk + J * TW, w.batch);
            tma_load_4d(smR + s * R_BYTES + KV_BYTES, &tm_v, &r_full[s], 0, w.kvhead, w.tok_chunk + J * TW, w.batch);
            if (++s == NR) s = 0, s_ph ^= 1;
            if (J == 0 && !(ok = clc_ask(&clc, it, &abort_flag))) break;
          }
        } else {
          mbar_arrive(&q_full[it & 1]);  // nothing to load: the phase passes all the same
          ok = clc_ask(&clc, it, &abort_flag);
        }
        if (!ok || !clc_next(&clc, it, &cta, true, false, &abort_flag)) break;
      }
    }
  } else if (warp == W_MMA) {
    const uint32_t tmem = tmem_base_s;
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc(128, TW, Pack2<T>::is_bf16, false, false);
      const uint32_t idesc_q = umma_idesc(128, HD, Pack2<T>::is_bf16, false, true);
      // positions in the rotation: group and ring stage with the phases of op_full and r_full there, of the next
      // operand and of the next scores, which run NG operands ahead
      struct Pos {
        int g = 0, s = 0;
        uint32_t g_ph = 0, s_ph = 0;
        __device__ __forceinline__ void step() {
          if (++g == NG) g = 0, g_ph ^= 1;
          if (++s == NR) s = 0, s_ph ^= 1;
        }
      } at, sc;
      // descriptors of stage 0; a stage on is R_BYTES >> 4 on in the address field
      const uint32_t ring = smem_u32(smR);
      const uint64_t d_k = umma_desc_sw128(ring, 16, 1024), d_v = umma_desc_sw128(ring + KV_BYTES, 16, 1024),
                     d_km = umma_desc_sw128(ring, 8192, 1024);
      bool ok = true;
      dim3 cta = blockIdx;
      int tiles = 0;
      for (int it = 0; ok; ++it) {
        const DqTile w(p, cta);
        ok = mbar_wait(&q_full[it & 1], (it >> 1) & 1, &abort_flag);
        if (!w.empty) {
          const uint32_t qd = smem_u32(smQD + (it & 1) * 2 * TILE_BYTES);
          const uint64_t d_q = umma_desc_sw128(qd, 16, 1024), d_dy = umma_desc_sw128(qd + TILE_BYTES, 16, 1024);
          auto issue_scores = [&](bool last) -> bool {
            if (!mbar_wait(&r_full[sc.s], sc.s_ph, &abort_flag)) return false;
            tc_fence_after();
            const uint32_t off = (uint32_t)sc.s * (R_BYTES >> 4), cb = tmem + col_b(sc.g);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ss(cb, d_q + 2 * ks, d_k + off + 2 * ks, idesc_s, ks > 0 ? 1u : 0u);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ss(cb + 64, d_dy + 2 * ks, d_v + off + 2 * ks, idesc_s, ks > 0 ? 1u : 0u);
            umma_commit(&s_full[sc.g]);
            if (last) umma_commit(&q_free[it & 1]);  // the query and dO tiles have been read
            sc.step();
            return true;
          };
          sc = at;
          for (int J = 0; J < min(w.nJ, NG) && ok; ++J) ok = issue_scores(J == w.nJ - 1);
          // the accumulator of the tile before has been read out
          if (ok && tiles > 0) ok = mbar_wait(&acc_free, (tiles - 1) & 1, &abort_flag);
          for (int J = 0; J < w.nJ && ok; ++J) {
            ok = mbar_wait(&op_full[at.g], at.g_ph, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t off = (uint32_t)at.s * (R_BYTES >> 4), cb = tmem + col_b(at.g);
#pragma unroll
            for (int ks = 0; ks < TW / 16; ++ks)
              umma_ts(tmem, cb + ks * 8, d_km + off + ks * (2048 >> 4), idesc_q, (J > 0 || ks > 0) ? 1u : 0u);
            umma_commit(&r_empty[at.s]);
            at.step();
            // the group's next scores, into the buffer that the product just issued reads (products execute in order)
            if (J + NG < w.nJ) ok = issue_scores(J + NG == w.nJ - 1);
          }
          if (ok) umma_commit(&acc_full);
          ++tiles;
        } else {
          mbar_arrive(&q_free[it & 1]);
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
      const DqTile w(p, cta);
      const float* a_chunk = gated ? p.a + ((size_t)w.batch * p.t + w.tok_chunk) * p.h + w.kvhead : nullptr;
      int J = (warp - W_COL - n0) & (NF - 1);
      // gate sums, two keys per lane, loaded one step ahead
      float av0 = 0.f, av1 = 0.f, rs = 0.f;
      auto load_gates = [&]() {
        if (gated) {
          const int kp = J * TW + lane;
          rs = a_chunk[(size_t)min(J * TW + TW - 1, w.c - 1) * p.h];
          av0 = kp < w.c ? a_chunk[(size_t)kp * p.h] : 0.f;
          av1 = kp + 32 < w.c ? a_chunk[(size_t)(kp + 32) * p.h] : 0.f;
        }
      };
      if (J < w.nJ) load_gates();
      while (J < w.nJ && ok) {
        const int n = n0 + J, slot = n % NC;
        const float low = warp_min(fminf(av0, av1)), f0 = __expf(rs - av0), f1 = __expf(rs - av1);
        if (n >= NC) ok = __all_sync(0xffffffffu, mbar_wait(&c_free[slot], (n / NC - 1) & 1, &abort_flag));
        if (!ok) break;
        Cols& cl = sm_c[slot];
        cl.fk[lane] = f0;
        cl.fk[lane + 32] = f1;
        cl.ak[lane] = av0;
        cl.ak[lane + 32] = av1;
        if (lane == 0) cl.top = make_float2(rs, low);
        __syncwarp();
        if (lane == 0) mbar_arrive(&c_full[slot]);
        J += NF;
        if (J < w.nJ) load_gates();
      }
      n0 += w.nJ;
      if (!ok || !clc_next(&clc, it, &cta, lane == 0, true, &abort_flag)) break;
    }
  } else {
    const uint32_t tmem = tmem_base_s;
    const int grp = warp >> 2, r = tid & 127;  // row group, query row inside the tile
    const int wrow = (warp & 3) * 32;
    const uint32_t lane_addr = (uint32_t)wrow << 16;
    const uint32_t cb = tmem + lane_addr + col_b(grp);
    const bool gated = p.a != nullptr;
    const float sdeg = DEG == 4 ? 4.f * (p.scale * p.scale) * (p.scale * p.scale) : 2.f * p.scale * p.scale;  // deg s^deg
    bool ok = true;
    dim3 cta = blockIdx;
    int tiles = 0, own = 0, n0 = 0, grp0 = 0;  // tiles with rows, steps of this group and of all so far; group of the first
    uint32_t row_ph = 0;
    // this thread's row: gate sum, dl and row sum, loaded before the write-out of the tile before
    float a_n = 0.f, dl_n = 0.f, l_n = 0.f;
    auto load_row = [&](const DqTile& w) {
      a_n = dl_n = l_n = 0.f;
      if (w.row0 + r < w.c) {
        const size_t tok = (size_t)w.batch * p.t + w.tok_chunk + w.row0 + r;
        if (gated) a_n = p.a[tok * p.h + w.kvhead];
        dl_n = p.dl[tok * p.hq + w.qhead];
        l_n = p.l[tok * p.hq + w.qhead];
      }
    };
    load_row(DqTile(p, cta));
    for (int it = 0; ok; ++it) {
      const DqTile w(p, cta);
      bool more = false;
      if (!w.empty) {
        const int row = w.row0 + r;
        const bool row_valid = row < w.c;
        const size_t tok0 = (size_t)w.batch * p.t + w.tok_chunk;
        const size_t ix = (tok0 + row) * p.hq + w.qhead;
        const float a_i = a_n, dl_i = dl_n;
        const float inv_l = row_valid ? safe_recip(l_n) : 0.f;
        const int wrow0 = w.row0 + wrow;  // first row of this warp
        float da = 0.f;                   // deg times the row sum of p * dp
        const int first = (grp - grp0 + NG) % NG;  // this group's first step in the tile
        for (int J = first; J < w.nJ && ok; J += NG, ++own) {
          const int kp0 = J * TW;
          const int n = n0 + J;
          const Cols& cl = sm_c[n % NC];
          ok = mbar_wait(&c_full[n % NC], (n / NC) & 1, &abort_flag);
          if (!ok) break;
          const float2 top = cl.top;
          const float rs = top.x;
          // The gate factor separates, e^{a_i - a_j} = e^{a_i - r} * e^{r - a_j}: one exponential
          // per row and per key instead of one per pair.  Both exponents are <= 0 below the
          // diagonal for gates <= 0; if one exceeds 80 (growing gates) the warp takes the per-pair
          // form.  Steps wholly below the diagonal need no mask; a warp whose rows all precede the
          // step's keys writes zeros without reading the scores.
          const bool sep = !__any_sync(0xffffffffu, fmaxf(rs - top.y, a_i - rs) > 80.f);
          const float c_i = sep ? sdeg * __expf(a_i - rs) : sdeg;
          ok = mbar_wait(&s_full[grp], own & 1, &abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (kp0 > min(wrow0 + 31, w.c - 1)) {
            uint32_t z[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = 0u;
            tmem_st16(cb, z);
            tmem_st16(cb + 16, z);
          } else {
            const bool mask = (kp0 + TW - 1 > wrow0) || (kp0 + TW - 1 >= w.c);
            const int lim = min(row, w.c - 1) - kp0;  // last column this row keeps
            if (!sep) dq_step<T, DEG, false, true>(cb, cl.ak, c_i, a_i, inv_l, dl_i, lim, da);
            else if (mask) dq_step<T, DEG, true, true>(cb, cl.fk, c_i, a_i, inv_l, dl_i, lim, da);
            else dq_step<T, DEG, true, false>(cb, cl.fk, c_i, a_i, inv_l, dl_i, lim, da);
          }
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&op_full[grp]);
            mbar_arrive(&c_free[n % NC]);
          }
        }
        sm_da[tiles & 1][first][r] = da;  // by step, not by group: a fixed order of the sum whatever the CTA did before
        // the row warps meet; bounded like every wait
        __syncwarp();
        if (lane == 0) mbar_arrive(&rows);
        // the groups share the write-out, 16 of the 64 columns at a time; the state-path gradient comes in meanwhile
        const float* st = p.dq_state ? p.dq_state + ix * p.d : nullptr;
        float add[2][2][8];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int c0 = 16 * (grp + NG * q);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int k = 0; k < 8; ++k) add[q][j][k] = 0.f;
            if (st != nullptr && row_valid && c0 < p.d && c0 < HD) {
              if (p.state_aligned32) {
                ld_global_v8(st + c0 + 8 * j, add[q][j]);
              } else {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  const float4 v = reinterpret_cast<const float4*>(st + c0 + 8 * j)[k];
                  add[q][j][4 * k] = v.x, add[q][j][4 * k + 1] = v.y;
                  add[q][j][4 * k + 2] = v.z, add[q][j][4 * k + 3] = v.w;
                }
              }
            }
          }
        }
        more = ok && clc_next(&clc, it, &cta, lane == 0, true, &abort_flag);
        if (more) load_row(DqTile(p, cta));
        if (ok) ok = mbar_wait(&rows, row_ph, &abort_flag);
        row_ph ^= 1;
        if (ok) ok = mbar_wait(&acc_full, tiles & 1, &abort_flag);
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int c0 = 16 * (grp + NG * q);
          if (!ok || c0 >= HD) continue;
          uint32_t acc[16];
          tmem_ld16(tmem + lane_addr + c0, acc);
          tmem_wait_ld();
          if (row_valid && c0 < p.d) {
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float* ad = add[q][j >> 1] + 4 * (j & 1);
              v[2 * j] = Pack2<T>::from_f32(__uint_as_float(acc[4 * j]) + ad[0], __uint_as_float(acc[4 * j + 1]) + ad[1]);
              v[2 * j + 1] =
                  Pack2<T>::from_f32(__uint_as_float(acc[4 * j + 2]) + ad[2], __uint_as_float(acc[4 * j + 3]) + ad[3]);
            }
            T* dst = static_cast<T*>(p.dQ) + ix * p.d + c0;
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
        if (grp == NG - 1 && row_valid)
          p.da_q[ix] = (1.f / DEG) * ((sm_da[tiles & 1][0][r] + sm_da[tiles & 1][1][r]) + sm_da[tiles & 1][2][r]);
        grp0 = (grp0 + w.nJ) % NG;
        n0 += w.nJ;
        ++tiles;
      } else {
        more = clc_next(&clc, it, &cta, lane == 0, true, &abort_flag);
        if (more) load_row(DqTile(p, cta));
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

extern "C" int pr_chunk_dq(int dtype, int b, int t, int hq, int h, int d, int c, const void* Q, const void* dO,
                           const void* K, const void* V, const float* a, const float* dl, const float* l,
                           const float* dq_state, float scale, int deg, void* dQ, float* da_q, int device,
                           void* stream) {
  using namespace pr;
  using namespace pr::dq;
  PR_REQUIRE(deg == 2 || (deg == 4 && dq_state == nullptr), PR_ERR_BAD_ARG,
             "deg=%d: states exist for deg 2; deg 4 runs state-free (attention only)", deg);
  PR_REQUIRE(head_dim_ok(d), PR_ERR_BAD_ARG, "head dim %d: a multiple of 16 up to 64", d);
  PR_REQUIRE(b > 0 && t > 0 && hq > 0 && h > 0 && hq % h == 0 && c > 0, PR_ERR_BAD_ARG,
             "bad sizes b=%d t=%d hq=%d h=%d c=%d", b, t, hq, h, c);
  PR_REQUIRE(dtype == PR_BF16 || dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", dtype);
  PR_REQUIRE(Q && dO && K && V && dl && l && dQ && da_q, PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE(aligned16(Q) && aligned16(dO) && aligned16(K) && aligned16(V) && aligned16(dQ) && aligned16(dq_state),
             PR_ERR_BAD_ARG, "misaligned pointer");
  PR_REQUIRE(hq <= 65535 && b <= 65535, PR_ERR_BAD_ARG, "hq and b must be <= 65535");
  PR_CUDA(cudaSetDevice(device));
  ChunkDqParams p;
  p.hq = hq;
  p.h = h;
  p.n_chunks = chunks_of(t, c);
  p.t = t;
  p.d = d;
  p.c = c;
  p.tiles_per_chunk = (c + 127) / 128;
  p.by_tiles = Div(p.tiles_per_chunk);
  p.by_ratio = Div(hq / h);
  p.scale = scale;
  p.a = a;
  p.dl = dl;
  p.l = l;
  p.dq_state = dq_state;
  p.dQ = dQ;
  p.aligned32 = aligned32(dQ);
  p.state_aligned32 = aligned32(dq_state);
  p.da_q = da_q;
  int rc = status_word(device, &p.status, nullptr);
  if (rc) return rc;
  CUtensorMap tm_q, tm_dy, tm_k, tm_v;
  uint64_t dq_[4] = {(uint64_t)d, (uint64_t)hq, (uint64_t)t, (uint64_t)b};
  uint64_t sq[4] = {0, (uint64_t)d * 2, (uint64_t)hq * d * 2, (uint64_t)t * hq * d * 2};
  uint64_t dk[4] = {(uint64_t)d, (uint64_t)h, (uint64_t)t, (uint64_t)b};
  uint64_t sk[4] = {0, (uint64_t)d * 2, (uint64_t)h * d * 2, (uint64_t)t * h * d * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  if ((rc = make_tmap(&tm_q, Q, 2, 4, dq_, sq, box, true))) return rc;
  if ((rc = make_tmap(&tm_dy, dO, 2, 4, dq_, sq, box, true))) return rc;
  uint32_t box_kv[4] = {64, 1, (uint32_t)TW, 1};
  if ((rc = make_tmap(&tm_k, K, 2, 4, dk, sk, box_kv, true))) return rc;
  if ((rc = make_tmap(&tm_v, V, 2, 4, dk, sk, box_kv, true))) return rc;
  dim3 grid(p.tiles_per_chunk * p.n_chunks, hq, b);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define PR_LAUNCH_DQ(TT, DG)                                                                                      \
  do {                                                                                                           \
    PR_SMEM_ATTR((chunk_dq_kernel<TT, DG>), SMEM, device, true);                                                   \
    chunk_dq_kernel<TT, DG><<<grid, THREADS, SMEM, s>>>(p, tm_q, tm_dy, tm_k, tm_v);                         \
  } while (0)
  if (dtype == PR_BF16) {
    if (deg == 4) PR_LAUNCH_DQ(__nv_bfloat16, 4); else PR_LAUNCH_DQ(__nv_bfloat16, 2);
  } else {
    if (deg == 4) PR_LAUNCH_DQ(__half, 4); else PR_LAUNCH_DQ(__half, 2);
  }
#undef PR_LAUNCH_DQ
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}
