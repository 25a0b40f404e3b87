// Fused output kernel: intra-chunk causal power attention, state read-out, merge and
// normalisation in one pass (the reference's _attention followed by _query_state,
// retention/_attention/reference.py:10-69 and retention/_query_state/reference.py:36-96,
// with the gate glue of retention/power_retention_maker.py:180-190).
//
// One CTA owns 128 query rows of one (batch, chunk, query head).  For deg = 2
//     y_i = sum_{j<=i} (s q_i.k_j)^2 e^{a_i-a_j} v_j + phi(q~_i)^T Z_m
//     l_i = sum_{j<=i} (s q_i.k_j)^2 e^{a_i-a_j}     + q~_i^T Zg_m q~_i
//     O_i = y_i / l_i,           q~_i = s q_i e^{a_i/2}
// where Z_m is the state entering the chunk (pair-aligned triangle layout) and Zg_m the
// scanned Gram matrix of the discounted keys (equivalent to the reference's sum_of_keys).
// Because both terms share one fp32 accumulator in tensor memory, the reference's
// rowmax / sqrt(D) range management is not needed.
//
// Two groups of four warps own the query rows, one row per thread in each group, and take the steps in turn (scores ->
// weights P, expansion phi(q~)); there is no running maximum, so a row's partial sums are simply added at the end.  One
// more warp issues TMA loads and makes the gate factors of a step's keys for all rows (Cols); one issues tcgen05.mma.  Two
// persistent CTAs per SM take over tile after tile (ClcRing): the loads and the first scores of a tile overlap the
// write-out of the one before, and ring stages, buffers and groups go on rotating across tiles.  The issuing thread keeps
// running positions and prepared descriptors, since what it executes between two batches leaves the tensor pipe idle.
// Bound by the latency of a step's chain, about 2000 clocks for a 64-key step whose products take 320: two groups in two
// CTAs overlap four such chains per SM.
// 637 -> 392 us (one group and one tile per CTA -> now) at b16 t2048 h32 without states, 317 -> 257 at b1 t65536 h8 with
// chunks of 1024 and states.  The factors on the TMA warp against every row warp making its own: 477 -> 400 without states;
// with states 261 -> 266, and 257 once tiles are found without divisions; a few steps in front of a state are 0.25 us slower
// (b1 t4096 h4 c256 14.5 -> 14.75).  Slower: three groups per CTA; 256 rows per CTA at one CTA per SM; factors three
// stages behind the loads; all loads that have room before a tile's first gates are waited for (257 -> 277).
//   S = Q K_J^T        : A, B K-major in shared memory (TMA, 128-byte swizzle)
//   acc += P V_J       : A = P written to tensor memory by the row threads, B = V_J MN-major
//   acc += phi(q~) Z   : A = expansion written to tensor memory 64 rows at a time,
//                        B = 64-row blocks of Z by TMA
//   u = q~ Zg          : A = q~ in tensor memory, B = Zg (hi + lo halves)
#include "host.cuh"
#include "layout.cuh"
#include "sm100.cuh"

namespace pr {

namespace co {
constexpr int HD = 64;
constexpr int NG = 2;                  // row groups
constexpr int NB = 3;                  // buffers of 64 columns in tensor memory
constexpr int NR = 4;                  // ring stages of 16 KB (key and value tile, Gram operand, two state blocks)
constexpr int W_TMA = 4 * NG, W_MMA = W_TMA + 1;
constexpr int THREADS = 32 * (W_MMA + 1);
constexpr uint32_t TMEM_COLS = 256;    // two CTAs per SM
constexpr int TILE_BYTES = 128 * 128;  // 128 rows x 64 16-bit features
constexpr int TW = 64;                 // keys per attention step
constexpr int KV_BYTES = TW * 128;     // one key or value tile
constexpr int Z_BYTES = 64 * 128;      // 64 expanded rows x 64 features
constexpr int R_BYTES = 2 * KV_BYTES;  // one ring stage
// What the row warps need of a step's 64 keys, made by the TMA warp while the tiles are on their way: e^{r - a_j} (r = gate
// sum at the step's last key) and a_j; r, smallest a_j.
struct alignas(16) Cols {
  float fk[TW], ak[TW];
  float2 top;
};
constexpr size_t SMEM = 1024 + 2 * TILE_BYTES + NR * (R_BYTES + sizeof(Cols));
// Tensor memory: the accumulator, then the buffers.  A buffer holds scores, overwritten by their weights P; in the
// state read-out 128 expanded entries, and for a while u = q~ Zg.  Operand number u of a CTA goes to buffer u % NB and
// is written by group u % NG.
__device__ __forceinline__ constexpr uint32_t col_b(int b) { return 64u * (uint32_t)(1 + b); }
}  // namespace co

struct ChunkOutParams {
  int hq, h;            // query heads, kv heads
  int n_chunks;         // chunks per batch element
  int cq, ck;           // queries / keys per chunk (query i sits at key position i + ck - cq)
  int tq, tk;           // queries / keys per batch element: the last chunk may be shorter than the others
  int d;                // features (a multiple of 16; TMA fills the tiles' columns up to 64 with zeros)
  int nblk;             // stages of 64 expanded rows of a state: ref_dim(d) / 64
  int tiles_per_chunk;  // ceil(cq / 128)
  Div by_tiles, by_ratio;  // by tiles_per_chunk, by query heads per kv head
  int state_from_chunk; // chunks >= this read the state (n_chunks: never)
  int q_gate_last;      // 1: gate the state read-out with the gate at the last key (inference)
  int normalize;        // 1: O = y / l; 0: O = y (l is written either way when l_out != null)
  int has_attn;         // 0: no keys at all (state-only read-out)
  float scale;          // s
  const float* a;       // [b, n*ck, h] cumulative log gates inside each chunk, or null
  void* O;              // [b, n*cq, hq, 64]
  int o_aligned32;      // O starts on a 32-byte boundary
  float* l_out;         // [b, n*cq, hq] or null
  int* status;
};

// What a CTA index stands for: a tile of 128 query rows of one (batch, chunk, query head).
struct OutTile {
  int chunk, qhead, kvhead, batch, row0;
  int cq, ck, q_off;   // queries and keys of the chunk; key position of query 0
  int nJ;              // attention steps: rows see keys up to their position
  int nI;              // operands of the state read-out: q~ itself, then 128 expanded entries each
  bool empty;          // past the end of a shorter last chunk
  __device__ __forceinline__ OutTile(const ChunkOutParams& p, const dim3& cta) {
    const int x = (int)cta.x;
    // the longest tiles of a head first
    int tile_i;
    p.by_tiles.of(x, &chunk, &tile_i);
    tile_i = p.tiles_per_chunk - 1 - tile_i;
    qhead = (int)cta.y;
    batch = (int)cta.z;
    kvhead = p.by_ratio.of(qhead);
    cq = min(p.cq, p.tq - chunk * p.cq);
    ck = min(p.ck, p.tk - chunk * p.ck);
    q_off = ck - cq;
    row0 = tile_i * 128;
    empty = row0 >= cq;
    nJ = (p.has_attn && !empty) ? min(ck - 1, row0 + 127 + q_off) / co::TW + 1 : 0;
    nI = (chunk >= p.state_from_chunk && !empty) ? 1 + p.nblk / 2 : 0;
  }
};

// One 16-column piece of an attention step for one query row: p = s^2 S^2 g into `pk`, row sum into
// l_acc.  SEP: the gate factor is c_i * fk[col] (c_i carries s^2); otherwise s^2 e^{a_i - ak[col]} per
// pair.  MASK: columns beyond `lim` (the row's own key position, relative to the step) are dropped.
template <typename T, int DEG, bool SEP, bool MASK>
__device__ __forceinline__ void out_piece(const uint32_t (&sv)[16], const float* __restrict__ fk, float c_i, float a_i,
                                          int lim, uint32_t (&pk)[8], float2& acc) {
  // two columns per instruction: packed fp32 multiplies and adds
  const float4* f4 = reinterpret_cast<const float4*>(fk);
  const float2 c2 = make_float2(c_i, c_i);
#pragma unroll
  for (int j = 0; j < 16; j += 4) {
    const float4 f = f4[j >> 2];
    const float2 fv[2] = {make_float2(f.x, f.y), make_float2(f.z, f.w)};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int col = j + 2 * u;
      const float2 s = make_float2(__uint_as_float(sv[col]), __uint_as_float(sv[col + 1]));
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
      float2 sq = __fmul2_rn(s, s);
      if (DEG == 4) sq = __fmul2_rn(sq, sq);
      const float2 pv = __fmul2_rn(sq, g);
      acc = __fadd2_rn(acc, pv);
      pk[col >> 1] = Pack2<T>::from_f32(pv.x, pv.y);
    }
  }
}

// A whole step: the load of the next piece is in flight while one is computed.
template <typename T, int DEG, bool SEP, bool MASK>
__device__ __forceinline__ void out_step(uint32_t cs, const float* __restrict__ fk, float c_i, float a_i, int lim,
                                         float& l_acc) {
  uint32_t sv[2][16], pk[8];
  float2 acc = make_float2(0.f, 0.f);
  tmem_ld16(cs, sv[0]);
#pragma unroll
  for (int q = 0; q < co::TW / 16; ++q) {
    tmem_wait_ld();
    if (q + 1 < co::TW / 16) tmem_ld16(cs + (q + 1) * 16, sv[(q + 1) & 1]);
    out_piece<T, DEG, SEP, MASK>(sv[q & 1], fk + q * 16, c_i, a_i, lim - q * 16, pk, acc);
    tmem_st8(cs + q * 8, pk);
  }
  l_acc += acc.x + acc.y;
}

template <typename T, int DEG>
__global__ void __launch_bounds__(co::THREADS, 2)
chunk_out_kernel(const ChunkOutParams p, const __grid_constant__ CUtensorMap tm_q,
                 const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                 const __grid_constant__ CUtensorMap tm_z, const __grid_constant__ CUtensorMap tm_ghi,
                 const __grid_constant__ CUtensorMap tm_glo) {
  using namespace co;
  extern __shared__ uint8_t smem_raw[];
  // q_*: the query tiles, two in flight.  r_*: the ring of operand tiles; operand number u takes stage u % NR, and
  // r_empty says that the products that read both have completed; c_full: a step's factors.  s_full: scores in a buffer; op_full: a group has
  // written an A operand (weights, q~, expansion) into it.  u_full: the Gram product; acc_full / acc_free:
  // accumulator complete / read out; rows: the row warps meet.
  __shared__ uint64_t q_full[2], q_free[2], r_full[NR], r_empty[NR], c_full[NR], s_full[NB], op_full[NB];
  __shared__ uint64_t u_full, acc_full, acc_free, rows;
  __shared__ ClcRing clc;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ float sm_l[2][NG][128];            // row sums of the groups

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sm = smem_raw + (sbase - smem_u32(smem_raw));
  uint8_t* smQ0 = sm;                         // 2 x TILE_BYTES
  // One ring serves both phases: an attention step takes a stage (key tile, then value tile); the state read-out goes
  // on with the same stage counter, two 64-row state blocks per stage, and so does the next tile, so the operands of
  // what comes next stream in while the last steps are still being computed.
  uint8_t* smR = smQ0 + 2 * TILE_BYTES;       // NR x R_BYTES
  Cols* smC = reinterpret_cast<Cols*>(smR + NR * R_BYTES);  // NR

  if (warp == W_TMA) {
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      abort_flag = 0;
      for (int s = 0; s < 2; ++s) {
        mbar_init(&q_full[s], 1);
        mbar_init(&q_free[s], 4 * NG);
      }
      for (int s = 0; s < NR; ++s) {
        mbar_init(&r_full[s], 1);
        mbar_init(&c_full[s], 1);
        mbar_init(&r_empty[s], 1);
      }
      for (int s = 0; s < NB; ++s) {
        mbar_init(&s_full[s], 1);
        mbar_init(&op_full[s], 4);
      }
      mbar_init(&u_full, 1);
      mbar_init(&acc_full, 1);
      mbar_init(&acc_free, 4 * NG);
      mbar_init(&rows, 4 * NG);
      clc_init(&clc, 4 * NG + 2);
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
    // -------------------------------------- TMA producer, and the factors of the keys
    const bool lead = elect_one();
    const bool gated = p.a != nullptr;
    bool ok = true;
    dim3 cta = blockIdx;
    int g = 0;  // ring stages so far
    auto ask = [&](int it) { ok = __all_sync(0xffffffffu, ok && (!lead || clc_ask(&clc, it, &abort_flag))); };
    for (int it = 0; ok; ++it) {
      const OutTile w(p, cta);
      if (it >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&q_free[it & 1], ((it >> 1) - 1) & 1, &abort_flag));
      if (!ok) break;
      if (!w.empty) {
        if (lead) {
          mbar_expect_tx(&q_full[it & 1], TILE_BYTES);
          tma_load_4d(smQ0 + (it & 1) * TILE_BYTES, &tm_q, &q_full[it & 1], 0, w.qhead, w.chunk * p.cq + w.row0, w.batch);
        }
        const int ch = (w.batch * p.n_chunks + w.chunk) * p.h + w.kvhead;
        const float* a_chunk =
            gated ? p.a + ((size_t)w.batch * p.tk + (size_t)w.chunk * p.ck) * p.h + w.kvhead : nullptr;
        // gate sums of the next step, two keys per lane, loaded one step ahead
        float av0 = 0.f, av1 = 0.f, r_n = 0.f;
        auto load_gates = [&](int J) {
          if (gated) {
            const int kp = J * TW + lane;
            r_n = a_chunk[(size_t)min(J * TW + TW - 1, w.ck - 1) * p.h];
            av0 = kp < w.ck ? a_chunk[(size_t)kp * p.h] : 0.f;
            av1 = kp + 32 < w.ck ? a_chunk[(size_t)(kp + 32) * p.h] : 0.f;
          }
        };
        if (w.nJ > 0) load_gates(0);
        for (int i = 0; i < w.nJ + w.nI && ok; ++i, ++g) {
          if (i == 1) ask(it);  // after the loads that the tile starts with
          const int s = g % NR;
          ok = __all_sync(0xffffffffu, ok && mbar_wait(&r_empty[s], ((g / NR) & 1) ^ 1, &abort_flag));
          if (!ok) break;
          uint8_t* dst = smR + s * R_BYTES;
          const int k = i - w.nJ;
          // c_full passes with every stage, so that its phases are the ring's; where there are no factors, before the loads
          if (k >= 0 && lane == 0) mbar_arrive(&c_full[s]);
          __syncwarp();
          if (lead) {
            mbar_expect_tx(&r_full[s], R_BYTES);
            if (k < 0) {
              tma_load_4d(dst, &tm_k, &r_full[s], 0, w.kvhead, w.chunk * p.ck + i * TW, w.batch);
              tma_load_4d(dst + KV_BYTES, &tm_v, &r_full[s], 0, w.kvhead, w.chunk * p.ck + i * TW, w.batch);
            } else if (k == 0) {
              tma_load_3d(dst, &tm_ghi, &r_full[s], 0, 0, ch);
              tma_load_3d(dst + Z_BYTES, &tm_glo, &r_full[s], 0, 0, ch);
            } else {
              tma_load_2d(dst, &tm_z, &r_full[s], 0, (ch * p.nblk + 2 * (k - 1)) * 64);
              tma_load_2d(dst + Z_BYTES, &tm_z, &r_full[s], 0, (ch * p.nblk + 2 * (k - 1) + 1) * 64);
            }
          }
          if (k < 0) {
            Cols& cl = smC[s];
            cl.fk[lane] = __expf(r_n - av0);
            cl.fk[lane + 32] = __expf(r_n - av1);
            cl.ak[lane] = av0;
            cl.ak[lane + 32] = av1;
            const float low = warp_min(fminf(av0, av1));
            if (lane == 0) cl.top = make_float2(r_n, low);
            if (i + 1 < w.nJ) load_gates(i + 1);
            __syncwarp();
            if (lane == 0) mbar_arrive(&c_full[s]);
          }
        }
        if (w.nJ + w.nI == 1) ask(it);
      } else {
        if (lead) mbar_arrive(&q_full[it & 1]);  // nothing to load: the phase passes all the same
        ask(it);
      }
      if (!ok || !clc_next(&clc, it, &cta, lane == 0, true, &abort_flag)) break;
    }
  } else if (warp == W_MMA) {
    const uint32_t tmem = tmem_base_s;
    // -------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc(128, TW, Pack2<T>::is_bf16, false, false);
      const uint32_t idesc_v = umma_idesc(128, HD, Pack2<T>::is_bf16, false, true);
      const uint32_t idesc_g = umma_idesc(128, HD, Pack2<T>::is_bf16, false, false);
      bool ok = true;
      dim3 cta = blockIdx;
      // Positions in the rotation of buffers and ring stages, with the phases of op_full and r_full there: of the next
      // operand (b, s), and of the next scores, which run up to NB operands ahead.
      struct Pos {
        int b = 0, s = 0;
        uint32_t b_ph = 0, s_ph = 0;
        __device__ __forceinline__ void step() {
          if (++b == NB) b = 0, b_ph ^= 1;
          if (++s == NR) s = 0, s_ph ^= 1;
        }
      } at, sc;
      int tiles = 0;
      const uint32_t ring = smem_u32(smR);
      // descriptors of stage 0; a stage on is R_BYTES >> 4 on in the address field
      const uint64_t d_k = umma_desc_sw128(ring, 16, 1024), d_v = umma_desc_sw128(ring + KV_BYTES, 8192, 1024),
                     d_z = umma_desc_sw128(ring, 8192, 1024);
      for (int it = 0; ok; ++it) {
        const OutTile w(p, cta);
        if (!w.empty) {
          const uint64_t d_q = umma_desc_sw128(smem_u32(smQ0 + (it & 1) * TILE_BYTES), 16, 1024);
          ok = mbar_wait(&q_full[it & 1], (it >> 1) & 1, &abort_flag);
          auto issue_scores = [&]() -> bool {
            if (!mbar_wait(&r_full[sc.s], sc.s_ph, &abort_flag)) return false;
            tc_fence_after();
            const uint64_t d = d_k + (uint32_t)sc.s * (R_BYTES >> 4);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_ss(tmem + col_b(sc.b), d_q + 2 * ks, d + 2 * ks, idesc_s, ks > 0 ? 1u : 0u);
            umma_commit(&s_full[sc.b]);
            sc.step();
            return true;
          };
          sc = at;
          for (int J = 0; J < min(w.nJ, NB) && ok; ++J) ok = issue_scores();
          // the accumulator of the tile before has been read out
          if (ok && tiles > 0) ok = mbar_wait(&acc_free, (tiles - 1) & 1, &abort_flag);
          for (int J = 0; J < w.nJ && ok; ++J) {
            ok = mbar_wait(&op_full[at.b], at.b_ph, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint64_t d = d_v + (uint32_t)at.s * (R_BYTES >> 4);
#pragma unroll
            for (int ks = 0; ks < TW / 16; ++ks)
              umma_ts(tmem, tmem + col_b(at.b) + ks * 8, d + ks * (2048 >> 4), idesc_v, (J > 0 || ks > 0) ? 1u : 0u);
            umma_commit(&r_empty[at.s]);
            at.step();
            // the next scores, into the buffer that the product just issued reads (products execute in order)
            if (J + NB < w.nJ) ok = issue_scores();
          }
          for (int k = 0; k < w.nI && ok; ++k) {
            ok = mbar_wait(&op_full[at.b], at.b_ph, &abort_flag) && mbar_wait(&r_full[at.s], at.s_ph, &abort_flag);
            if (!ok) break;
            tc_fence_after();
            if (k == 0) {
              // u = q~ Zg (hi then lo), into the buffer of the operand after next
              const uint64_t d = d_k + (uint32_t)at.s * (R_BYTES >> 4);
              const int bu = at.b == 0 ? 2 : at.b - 1;
#pragma unroll
              for (int hl = 0; hl < 2; ++hl)
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                  umma_ts(tmem + col_b(bu), tmem + col_b(at.b) + ks * 8, d + hl * (Z_BYTES >> 4) + 2 * ks, idesc_g,
                          (hl > 0 || ks > 0) ? 1u : 0u);
              umma_commit(&u_full);
            } else {
              // 128 expanded entries against two state blocks
              const uint64_t d = d_z + (uint32_t)at.s * (R_BYTES >> 4);
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                umma_ts(tmem, tmem + col_b(at.b) + ks * 8, d + (ks >> 2) * (Z_BYTES >> 4) + (ks & 3) * (2048 >> 4), idesc_v,
                        (w.nJ > 0 || k > 1 || ks > 0) ? 1u : 0u);
            }
            umma_commit(&r_empty[at.s]);
            at.step();
          }
          if (ok) umma_commit(&acc_full);
          ++tiles;
        }
        if (!ok || !clc_next(&clc, it, &cta, true, false, &abort_flag)) break;
      }
    }
  } else {
    // --------------------------------------------------------- row-owning warps
    const uint32_t tmem = tmem_base_s;
    const int grp = warp >> 2, r = tid & 127;   // row group, row inside a tile
    const int wrow = (warp & 3) * 32;
    const uint32_t lane_addr = (uint32_t)wrow << 16;
    const float s2 = DEG == 4 ? (p.scale * p.scale) * (p.scale * p.scale) : p.scale * p.scale;  // s^deg
    const bool gated = p.a != nullptr;
    bool ok = true;
    dim3 cta = blockIdx;
    int u0 = 0, tiles = 0, grams = 0;  // operands before this tile, tiles with rows, Gram products so far
    uint32_t s_base = 0, row_ph = 0;   // phase of each buffer's s_full at the tile's start (one bit each), and of rows
    // the row warps meet; bounded like every wait
    auto meet = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(&rows);
      if (ok) ok = mbar_wait(&rows, row_ph, &abort_flag);
      row_ph ^= 1;
    };
    auto operand_written = [&](int u) {
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[u % NB]);
    };
    // buffer u % NB is free once the products that read its operand before u have completed
    auto buffer_free = [&](int u) {
      if (ok && u >= NB) ok = mbar_wait(&r_empty[(u - NB) % NR], ((u - NB) / NR) & 1, &abort_flag);
      tc_fence_after();
    };
    // gate sum of this thread's row, loaded before the write-out of the tile before
    float a_n = 0.f;
    auto load_row = [&](const OutTile& w) {
      a_n = (gated && w.row0 + r < w.cq)
                ? p.a[((size_t)w.batch * p.tk + (size_t)w.chunk * p.ck + w.row0 + r + w.q_off) * p.h + w.kvhead]
                : 0.f;
    };
    load_row(OutTile(p, cta));
    for (int it = 0; ok; ++it) {
      const OutTile w(p, cta);
      bool more = false;
      if (!w.empty) {
        uint8_t* smQ = smQ0 + (it & 1) * TILE_BYTES;
        const float* a_chunk =
            gated ? p.a + ((size_t)w.batch * p.tk + (size_t)w.chunk * p.ck) * p.h + w.kvhead : nullptr;
        const int row = w.row0 + r;             // query index inside the chunk
        const int qpos = row + w.q_off;         // its key position
        const float a_i = a_n;
        float l_acc = 0.f;
        const int first = (u0 + grp) & 1;       // this group's first operand in the tile
        static_assert(NG == 2, "the group of operand u is u & 1");

        for (int J = first; J < w.nJ && ok; J += NG) {
          const int u = u0 + J, b = u % NB;
          const int kp0 = J * TW;
          const Cols& cl = smC[u % NR];
          ok = mbar_wait(&c_full[u % NR], (u / NR) & 1, &abort_flag);
          if (!ok) break;
          const float2 top = cl.top;
          const float rs = top.x;
          // The gate factor separates, e^{a_i - a_j} = e^{a_i - r} * e^{r - a_j}: one exponential per
          // row and per key instead of one per pair (both exponents <= 0 below the diagonal for gates
          // <= 0; a warp falls back to the per-pair form if one exceeds 80).  Steps wholly below the
          // diagonal need no mask; a warp whose rows all precede the step's keys writes zeros
          // without reading the scores.
          const bool sep = !__any_sync(0xffffffffu, fmaxf(rs - top.y, a_i - rs) > 80.f);
          const float c_i = sep ? s2 * __expf(a_i - rs) : s2;
          ok = mbar_wait(&s_full[b], ((s_base >> b) + J / NB) & 1, &abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t cs = tmem + lane_addr + col_b(b);
          const int wq0 = w.row0 + wrow + w.q_off;  // key position of this warp's first query
          if (kp0 > min(wq0 + 31, w.ck - 1)) {
            uint32_t z[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = 0u;
            tmem_st16(cs, z);
            tmem_st16(cs + 16, z);
          } else {
            const bool mask = (kp0 + TW - 1 > wq0) || (kp0 + TW - 1 >= w.ck);
            const int lim = min(qpos, w.ck - 1) - kp0;  // last column this row keeps
            if (!sep) out_step<T, DEG, false, true>(cs, cl.ak, c_i, a_i, lim, l_acc);
            else if (mask) out_step<T, DEG, true, true>(cs, cl.fk, c_i, a_i, lim, l_acc);
            else out_step<T, DEG, true, false>(cs, cl.fk, c_i, a_i, lim, l_acc);
          }
          operand_written(u);
        }

        if (w.nI > 0) {
          meet();  // every score product of the tile has completed: the query tile may be rewritten
          // The gated, scaled row q~ takes the row's place in the query tile, where the expansion fetches its factors
          // by a runtime index; each group does every other 16-byte piece.
          if (ok) ok = mbar_wait(&q_full[it & 1], (it >> 1) & 1, &abort_flag);
          const float f =
              p.scale * (gated ? __expf(0.5f * (p.q_gate_last ? a_chunk[(size_t)(w.ck - 1) * p.h] : a_i)) : 1.f);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            uint4* slot = reinterpret_cast<uint4*>(smQ + swz128(r, 2 * jj + grp));
            const uint4 v = *slot;
            uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 f2 = Pack2<T>::to_f32(x[k]);
              x[k] = Pack2<T>::from_f32(f2.x * f, f2.y * f);
            }
            *slot = make_uint4(x[0], x[1], x[2], x[3]);
          }
          meet();  // q~ is in place
          const int ui = u0 + w.nJ;
          if ((ui & 1) == grp) {
            // operand 0: q~ itself (for u = q~ Zg); then u comes out of the buffer of operand 2, which is this group's
            // too: its dot product with q~ is the state's part of the row sum
            buffer_free(ui);
            {
              uint32_t q2[32];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const uint4 v = *reinterpret_cast<const uint4*>(smQ + swz128(r, j));
                q2[4 * j] = v.x;
                q2[4 * j + 1] = v.y;
                q2[4 * j + 2] = v.z;
                q2[4 * j + 3] = v.w;
              }
              if (ok) {
                tmem_st32(tmem + lane_addr + col_b(ui % NB), q2);
                operand_written(ui);
              }
            }
            if (ok) ok = mbar_wait(&u_full, grams & 1, &abort_flag);
            tc_fence_after();
            if (ok) {
              float ls0 = 0.f, ls1 = 0.f;
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                uint32_t u[32];
                tmem_ld32(tmem + lane_addr + col_b((ui + 2) % NB) + 32 * hf, u);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const uint4 v = *reinterpret_cast<const uint4*>(smQ + swz128(r, 4 * hf + j));
                  const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    const float2 qv = Pack2<T>::to_f32(x[k]);
                    ls0 = fmaf(__uint_as_float(u[8 * j + 2 * k]), qv.x, ls0);
                    ls1 = fmaf(__uint_as_float(u[8 * j + 2 * k + 1]), qv.y, ls1);
                  }
                }
              }
              l_acc += ls0 + ls1;
              tc_fence_before();
            }
          }
          ++grams;
          // operands 1 .. nblk/2: 128 expanded entries (64 packed products) each
          for (int k = (ui & 1) == grp ? 2 : 1; k < w.nI; k += NG) {
            // operands 1-2, 3-6, 7-12, 13-20 have their second factors in block Y = 0, 1, 2, 3
            const int Y = (k > 2) + (k > 6) + (k > 12);
            const int a0 = 8 * (k - 1 - Y * (Y + 1));
            const uint32_t ca = tmem + lane_addr + col_b((ui + k) % NB);
            uint32_t x2[8], x[32];
            expand_second(smQ, r, Y, x2);
            expand_stage<T>(smQ, r, a0, x2, x);
            buffer_free(ui + k);
            if (ok) tmem_st32(ca, x);
            expand_stage<T>(smQ, r, a0 + 4, x2, x);
            if (ok) {
              tmem_st32(ca + 32, x);
              operand_written(ui + k);
            }
          }
        }
        // The query tile may be refilled (its last reads come before the async proxy's writes).  After the meeting: a
        // group that has no step in the tile has waited for nothing of it before, and could give the slot back twice
        // while the other is still in a run of empty tiles.
        fence_async_smem();
        sm_l[tiles & 1][grp][r] = l_acc;
        meet();
        if (lane == 0) mbar_arrive(&q_free[it & 1]);
        more = ok && clc_next(&clc, it, &cta, lane == 0, true, &abort_flag);
        if (more) load_row(OutTile(p, cta));
        if (ok) ok = mbar_wait(&acc_full, tiles & 1, &abort_flag);
        tc_fence_after();
        // each group writes two pieces of 16 of the row's 64 columns, one 32-byte store each
        if (ok) {
          const float l = sm_l[tiles & 1][0][r] + sm_l[tiles & 1][1][r];
          const float inv = p.normalize ? safe_recip(l) : 1.f;
          const size_t tok = (size_t)w.batch * p.tq + (size_t)w.chunk * p.cq + row;
          uint32_t acc[2][16];
          tmem_ld16(tmem + lane_addr + 32 * grp, acc[0]);
          tmem_ld16(tmem + lane_addr + 32 * grp + 16, acc[1]);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_free);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int c0 = 32 * grp + 16 * q;
            if (row < w.cq && c0 < p.d) {
              uint32_t v[8];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                v[j] = Pack2<T>::from_f32(inv * __uint_as_float(acc[q][2 * j]), inv * __uint_as_float(acc[q][2 * j + 1]));
              T* dst = static_cast<T*>(p.O) + (tok * p.hq + w.qhead) * p.d + c0;
              if (p.o_aligned32) {
                st_global_v8(dst, v);
              } else {
                reinterpret_cast<uint4*>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
                reinterpret_cast<uint4*>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
              }
            }
          }
          if (p.l_out != nullptr && grp == 0 && row < w.cq) p.l_out[tok * p.hq + w.qhead] = l;
        }
        // the score products of the tile: buffer b had one for every step J with (u0 + J) % NB == b
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const int j0 = (b - u0 % NB + NB) % NB;
          if (j0 < w.nJ) s_base ^= (((w.nJ - 1 - j0) / NB + 1) & 1) << b;
        }
        u0 += w.nJ + w.nI;
        ++tiles;
      } else {
        // Not before the producer has come to this tile, and so has seen the last phase of this slot's q_free: in a
        // run of empty tiles the row warps could pass it, and two phases on the parity that it waits for looks open.
        ok = mbar_wait(&q_full[it & 1], (it >> 1) & 1, &abort_flag);
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_free[it & 1]);
        more = ok && clc_next(&clc, it, &cta, lane == 0, true, &abort_flag);
        if (more) load_row(OutTile(p, cta));
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

int pr::chunk_out(int dtype, int b, int tq, int tk, int cq, int ck, int hq, int h, int d, const void* Q, const void* K,
                  const void* V, const float* a, const void* Z, const void* zg_hi, const void* zg_lo,
                  int state_from_chunk, int q_gate_last, int normalize, float scale, int deg, void* O, float* l_out,
                  int device, void* stream) {
  using namespace pr::co;
  PR_REQUIRE(head_dim_ok(d), PR_ERR_BAD_ARG, "head dim %d: a multiple of 16 up to 64", d);
  const int n_chunks = cq > 0 ? (tq + cq - 1) / cq : 0;
  PR_REQUIRE(b > 0 && n_chunks > 0 && cq > 0 && ck >= cq && hq > 0 && h > 0 && hq % h == 0 &&
                 (n_chunks == 1 || (cq == ck && tq == tk)) && tk >= tq,
             PR_ERR_BAD_ARG, "bad sizes b=%d n=%d cq=%d ck=%d hq=%d h=%d", b, n_chunks, cq, ck, hq, h);
  PR_REQUIRE(dtype == PR_BF16 || dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", dtype);
  PR_REQUIRE(deg == 2 || (deg == 4 && Z == nullptr), PR_ERR_BAD_ARG,
             "deg=%d: states exist for deg 2; deg 4 runs state-free (attention only)", deg);
  const bool has_attn = (K != nullptr && V != nullptr);
  PR_REQUIRE(Q && O && aligned16(Q) && aligned16(O) && aligned16(K) && aligned16(V), PR_ERR_BAD_ARG,
             "null or misaligned pointer");
  PR_REQUIRE(has_attn || (Z != nullptr && state_from_chunk <= 0), PR_ERR_BAD_ARG,
             "a chunk with neither keys / values nor a state");
  const bool with_state = (Z != nullptr) && state_from_chunk < n_chunks;
  PR_REQUIRE(!with_state || (zg_hi && zg_lo && aligned16(Z) && aligned16(zg_hi) && aligned16(zg_lo)), PR_ERR_BAD_ARG,
             "state given without its Gram matrices");
  PR_REQUIRE(hq <= 65535 && b <= 65535, PR_ERR_BAD_ARG, "hq and b must be <= 65535");
  PR_CUDA(cudaSetDevice(device));
  ChunkOutParams p;
  p.hq = hq;
  p.h = h;
  p.n_chunks = n_chunks;
  p.cq = cq;
  p.ck = ck;
  p.tq = tq;
  p.tk = tk;
  p.d = d;
  p.nblk = ref_dim(d) / 64;
  p.tiles_per_chunk = (cq + 127) / 128;
  p.by_tiles = Div(p.tiles_per_chunk);
  p.by_ratio = Div(hq / h);
  p.state_from_chunk = with_state ? state_from_chunk : n_chunks;
  p.q_gate_last = q_gate_last;
  p.normalize = normalize;
  p.has_attn = has_attn ? 1 : 0;
  p.scale = scale;
  p.a = a;
  p.O = O;
  p.o_aligned32 = aligned32(O);
  p.l_out = l_out;
  int rc = status_word(device, &p.status, nullptr);
  if (rc) return rc;
  CUtensorMap tm_q, tm_k, tm_v, tm_z, tm_ghi, tm_glo;
  {
    uint64_t dq[4] = {(uint64_t)d, (uint64_t)hq, (uint64_t)tq, (uint64_t)b};
    uint64_t sq[4] = {0, (uint64_t)d * 2, (uint64_t)hq * d * 2, (uint64_t)tq * hq * d * 2};
    uint64_t dk[4] = {(uint64_t)d, (uint64_t)h, (uint64_t)tk, (uint64_t)b};
    uint64_t sk[4] = {0, (uint64_t)d * 2, (uint64_t)h * d * 2, (uint64_t)tk * h * d * 2};
    uint32_t box[4] = {64, 1, 128, 1};
    uint32_t box_kv[4] = {64, 1, (uint32_t)TW, 1};
    if ((rc = make_tmap(&tm_q, Q, 2, 4, dq, sq, box, true))) return rc;
    if (has_attn) {
      if ((rc = make_tmap(&tm_k, K, 2, 4, dk, sk, box_kv, true))) return rc;
      if ((rc = make_tmap(&tm_v, V, 2, 4, dk, sk, box_kv, true))) return rc;
    } else {
      tm_k = tm_q;
      tm_v = tm_q;
    }
  }
  if (with_state) {
    uint64_t dz[2] = {(uint64_t)d, (uint64_t)b * n_chunks * h * ref_dim(d)};
    uint64_t st[2] = {0, (uint64_t)d * 2};
    uint32_t box[2] = {64, 64};
    if ((rc = make_tmap(&tm_z, Z, 2, 2, dz, st, box, true))) return rc;
    if ((rc = gram_tmap(&tm_ghi, zg_hi, d, (uint64_t)b * n_chunks * h))) return rc;
    if ((rc = gram_tmap(&tm_glo, zg_lo, d, (uint64_t)b * n_chunks * h))) return rc;
  } else {
    tm_z = tm_q;
    tm_ghi = tm_q;
    tm_glo = tm_q;
  }
  dim3 grid(p.tiles_per_chunk * n_chunks, hq, b);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define PR_LAUNCH_OUT(TT, DG)                                                                                      \
  do {                                                                                                             \
    PR_SMEM_ATTR((chunk_out_kernel<TT, DG>), SMEM, device, true);                                                   \
    chunk_out_kernel<TT, DG><<<grid, THREADS, SMEM, s>>>(p, tm_q, tm_k, tm_v, tm_z, tm_ghi, tm_glo);                 \
  } while (0)
  if (dtype == PR_BF16) {
    if (deg == 4) PR_LAUNCH_OUT(__nv_bfloat16, 4); else PR_LAUNCH_OUT(__nv_bfloat16, 2);
  } else {
    if (deg == 4) PR_LAUNCH_OUT(__half, 4); else PR_LAUNCH_OUT(__half, 2);
  }
#undef PR_LAUNCH_OUT
  PR_CUDA(cudaGetLastError());
  return PR_OK;
}

extern "C" int pr_chunk_out(int dtype, int b, int n_chunks, int cq, int ck, int hq, int h, int d, const void* Q,
                            const void* K, const void* V, const float* a, const void* Z, const void* zg_hi,
                            const void* zg_lo, int state_from_chunk, int q_gate_last, int normalize, float scale,
                            int deg, void* O, float* l_out, int device, void* stream) {
  return pr::chunk_out(dtype, b, n_chunks * cq, n_chunks * ck, cq, ck, hq, h, d, Q, K, V, a, Z, zg_hi, zg_lo,
                       state_from_chunk, q_gate_last, normalize, scale, deg, O, l_out, device, stream);
}
