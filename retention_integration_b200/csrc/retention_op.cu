// Whole-operator entry points: the chunked forward and backward of power retention
// (retention/power_retention_maker.py:96-197 and what autograd executes for it) as ONE call
// each, and those of the state-free branch (:128-132), where one chunk holds the whole sequence.
// The launch sequences live here in native code, so a host in any language runs the operator
// through three symbols per branch (pr_workspace_bytes, pr_retention_fwd, pr_retention_bwd;
// pr_attention_workspace_bytes, pr_attention_fwd, pr_attention_bwd).
//
// Memory: the caller allocates everything.  `saved` is what the backward needs from the
// forward (gate sums, row sums, scanned states and Gram matrices); `scratch` is dead when the
// call returns its work to the stream and may be reused by the next call on the same stream.
#include <atomic>
#include <mutex>

#include "host.cuh"
#include "layout.cuh"

namespace pr {
namespace {

constexpr size_t kAlign = 256;
inline size_t up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }

struct Sizes {
  int n, cp, DR, esz;
  size_t a, A, l, Z, zh, zfull;             // saved
  size_t KT, gram;                          // forward scratch
  size_t dy, dl, QT, dZ, dZg, partS, partG, gh, dqs, gq, dks, wk, daq, dak;  // backward scratch
  int blocksS, blocksG;
};

int sizes_of(const pr_problem* p, Sizes* s) {
  PR_REQUIRE(p != nullptr, PR_ERR_BAD_ARG, "problem is null");
  PR_REQUIRE(p->d == 16 || p->d == 32 || p->d == 64, PR_ERR_BAD_ARG, "head dim %d: this build handles 16, 32 and 64", p->d);
  PR_REQUIRE(p->dtype == PR_BF16 || p->dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", p->dtype);
  PR_REQUIRE(p->b > 0 && p->t > 0 && p->h > 0 && p->hq > 0 && p->hq % p->h == 0 && p->c > 0,
             PR_ERR_BAD_ARG, "bad sizes b=%d t=%d h=%d hq=%d c=%d", p->b, p->t, p->h, p->hq, p->c);
  const size_t b = p->b, t = p->t, h = p->h, hq = p->hq, d = p->d;
  s->n = chunks_of(p->t, p->c);
  s->cp = (p->c + 63) / 64 * 64;
  s->DR = ref_dim(p->d);
  s->esz = 2;
  const size_t n = s->n, DR = s->DR, cp = s->cp;
  s->a = up(b * t * h * 4);
  s->A = up(b * n * h * 4);
  s->l = up(b * t * hq * 4);
  s->Z = up(b * n * h * DR * d * 2);
  s->zh = up(b * n * h * d * d * 2);
  s->zfull = up(b * n * h * d * d * 4);
  s->KT = up(b * n * h * d * cp * 2);
  s->gram = up(b * n * h * d * d * 4);
  s->dy = up(b * t * hq * d * 2);
  s->dl = up(b * t * hq * 4);
  s->QT = up(b * n * hq * d * cp * 2);
  s->dZ = s->Z;
  s->dZg = s->gram;
  s->blocksS = pr_discumsum_bwd_blocks((long long)DR * d);
  s->blocksG = pr_gram_scan_bwd_blocks(p->d);
  s->partS = up(b * h * s->blocksS * n * 4);
  s->partG = up(b * h * s->blocksG * n * 4);
  s->gh = s->zh;
  s->dqs = up(b * t * hq * d * 4);
  s->gq = up(b * t * hq * 4);
  s->dks = up(b * t * h * d * 4);
  s->wk = up(b * t * h * 4);
  s->daq = up(b * t * hq * 4);
  s->dak = up(b * t * h * 4);
  return PR_OK;
}

struct Carver {
  uint8_t* p;
  template <typename T>
  T* take(size_t bytes) {
    T* r = reinterpret_cast<T*>(p);
    p += bytes;
    return r;
  }
};

struct Saved {
  float *a, *A, *l, *zfull;
  void *Z, *zhi, *zlo;
};
Saved carve_saved(void* base, const Sizes& s) {
  Carver c{static_cast<uint8_t*>(base)};
  Saved v;
  v.a = c.take<float>(s.a);
  v.A = c.take<float>(s.A);
  v.l = c.take<float>(s.l);
  v.Z = c.take<void>(s.Z);
  v.zhi = c.take<void>(s.zh);
  v.zlo = c.take<void>(s.zh);
  v.zfull = c.take<float>(s.zfull);
  return v;
}

// The backward has two independent branches after dout_prep: the query side (expand_grad on the
// saved states, then chunk_dq) needs nothing from the reverse scan, which heads the key side
// (gate_prep, chunk_state, scan, expand_grad, chunk_dkv).  The query side is enqueued on a second
// stream, forked from and joined back into the caller's stream with events, so that its CTAs fill
// the partial last wave of each key-side launch (and vice versa).
//
// A device has kSideStreams such streams, created together by its first backward outside a capture and kept for the
// process.  Which one a backward uses depends on its caller's stream, so that callers on different streams seldom wait
// for one another; `mu` is held while a backward is being enqueued.  While a caller's stream is being captured, the
// second stream belongs to that capture until it ends (the fork and the join are recorded like any cross-stream
// dependency): a backward of another stream that comes to it meanwhile is enqueued on its caller's stream alone,
// because it could neither join that capture nor leave it undisturbed.
struct SideStream {
  std::mutex mu;
  cudaStream_t stream = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};
constexpr int kMaxDevices = 64;
constexpr int kSideStreams = 8;
struct DeviceSides {
  std::mutex mu;  // creation
  std::atomic<bool> ready{false};
  SideStream side[kSideStreams];
};
DeviceSides g_side[kMaxDevices];

bool overlap_enabled() {
  static const bool on = [] {
    const char* e = getenv("PR_BWD_OVERLAP");
    return !(e && e[0] == '0');
  }();
  return on;
}

// The capture that a stream takes part in; 0: none, ~0: one that has failed and not ended yet.
int capture_of(cudaStream_t stream, unsigned long long* id) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  *id = 0;
  PR_CUDA(cudaStreamGetCaptureInfo(stream, &status, id));
  if (status != cudaStreamCaptureStatusActive) *id = status == cudaStreamCaptureStatusNone ? 0 : ~0ull;
  return PR_OK;
}

// The device's streams, or none yet (*out = null) when the first backward is being captured.
int side_streams(int device, cudaStream_t caller, DeviceSides** out) {
  DeviceSides& d = g_side[device];
  *out = &d;
  if (d.ready.load(std::memory_order_acquire)) return PR_OK;
  std::lock_guard<std::mutex> lock(d.mu);
  if (d.ready.load(std::memory_order_relaxed)) return PR_OK;
  unsigned long long capture = 0;
  int rc = capture_of(caller, &capture);
  if (rc) return rc;
  if (capture) {
    *out = nullptr;
    return PR_OK;
  }
  for (SideStream& s : d.side) {
    if (!s.stream) PR_CUDA(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
    if (!s.fork) PR_CUDA(cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming));
    if (!s.join) PR_CUDA(cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming));
  }
  d.ready.store(true, std::memory_order_release);
  return PR_OK;
}

// The fork of one backward pass: begin(), launches on side(), side_done(), launches on the caller's stream, join().
class Fork {
 public:
  int begin(int device, void* stream) {
    PR_REQUIRE(device >= 0 && device < kMaxDevices, PR_ERR_BAD_ARG, "device ordinal %d out of range", device);
    main_ = static_cast<cudaStream_t>(stream);
    if (!overlap_enabled()) return PR_OK;
    PR_CUDA(cudaSetDevice(device));
    DeviceSides* d = nullptr;
    int rc = side_streams(device, main_, &d);
    if (rc || !d) return rc;
    // handles are pointers or small numbers: mixed so that both spread over the streams
    const uint64_t mix = reinterpret_cast<uintptr_t>(stream) * 0x9E3779B97F4A7C15ull;
    SideStream& s = d->side[mix >> 61];
    static_assert(kSideStreams == 8, "three bits of the mixed handle");
    std::unique_lock<std::mutex> lock(s.mu);
    unsigned long long theirs = 0, ours = 0;
    if ((rc = capture_of(s.stream, &theirs))) return rc;
    if (theirs) {
      if ((rc = capture_of(main_, &ours))) return rc;
      if (ours != theirs) return PR_OK;  // another caller's capture
    }
    PR_CUDA(cudaEventRecord(s.fork, main_));
    PR_CUDA(cudaStreamWaitEvent(s.stream, s.fork, 0));
    lock_ = std::move(lock);
    s_ = &s;
    return PR_OK;
  }
  void* side() const { return s_ ? s_->stream : main_; }
  // recorded even after an error, so that a capture of the caller's stream is left in a closable state
  void side_done() {
    if (s_) cudaEventRecord(s_->join, s_->stream);
  }
  int join(int rc) {
    if (!s_) return rc;
    cudaError_t e = cudaStreamWaitEvent(main_, s_->join, 0);
    lock_.unlock();
    return (!rc && e != cudaSuccess) ? fail(PR_ERR_CUDA, "joining the second stream failed: %s", cudaGetErrorString(e)) : rc;
  }

 private:
  SideStream* s_ = nullptr;
  cudaStream_t main_ = nullptr;
  std::unique_lock<std::mutex> lock_;
};

}  // namespace
}  // namespace pr

// The chunk size to run a request with.  The operator's result does not depend on the chunk size, its speed
// does: every chunk's state is written, scanned and read again (1.3 GB per pass at chunk 128 against 0.17 GB at
// 1024 for b1 t65536 h8), and above 1024 the intra-chunk attention grows.  Forward + backward of that shape in ms, as
// asked: chunk 128 4.46, 256 3.01, 512 2.38, 1024 2.24, 2048 2.46, 4096 2.97.  Below 1024: the largest multiple of the
// request up to 1024 that rounds the length up by at most 1/16 more than the request does; above: the largest divisor
// of the request in [256, 1024]; 0 (no chunking) on more than 2048 tokens: 1024 or 512 if that rounds the length up by
// at most 1/16, else 0.
// The rounding was work while sequences were padded to whole chunks.  They no longer are, and by work the rule errs
// where it still decides: t 2000 with chunk 128 takes two chunks of 1024 (105 us replayed from a graph, b1 h2) where
// one without states takes 68, t 1100 three of 384 (87 us, b1 h4; 49), and t 7200 unchunked stays one (334 us, b1 h4)
// where chunks of 1024 take 177.  Mirrors retention.py: effective_chunk, for hosts that do not go through the Python API.
extern "C" int pr_fast_chunk(long long t, int requested) {
  const int fast = 1024;
  if (t <= 0 || requested < 0) return requested;
  auto rounded_to = [t](long long c) { return (t + c - 1) / c * c; };
  if (requested == 0) {
    if (t <= 2 * fast) return 0;
    for (int ce : {fast, fast / 2})
      if (rounded_to(ce) <= t + t / 16) return ce;
    return 0;
  }
  if (requested > fast) {
    for (int ce = fast; ce >= 256; --ce)
      if (requested % ce == 0) return ce;
    return requested;
  }
  if (requested == fast) return requested;
  const long long asked = rounded_to(requested);
  for (int m = fast / requested; m > 1; --m) {
    const long long ce = (long long)m * requested;
    if (rounded_to(ce) <= asked + asked / 16) return (int)ce;
  }
  return requested;
}

extern "C" int pr_workspace_bytes(const pr_problem* prob, int what, size_t* out) {
  using namespace pr;
  PR_REQUIRE(out != nullptr, PR_ERR_BAD_ARG, "out is null");
  Sizes s;
  int rc = sizes_of(prob, &s);
  if (rc) return rc;
  switch (what) {
    case PR_WS_SAVED:
      *out = s.a + s.A + s.l + s.Z + 2 * s.zh + s.zfull;
      break;
    case PR_WS_FWD_SCRATCH:
      *out = s.KT + s.gram;
      break;
    case PR_WS_BWD_SCRATCH:
      *out = s.dy + s.dl + 2 * s.QT + s.dZ + s.dZg + s.partS + s.partG + 2 * s.gh + s.dqs + s.gq + s.dks + s.wk +
             s.daq + s.dak;
      break;
    default:
      return fail(PR_ERR_BAD_ARG, "workspace kind %d", what);
  }
  return PR_OK;
}

extern "C" int pr_retention_fwd(const pr_problem* prob, const void* Q, const void* K, const void* V,
                                const float* log_G, const float* carry_state, const float* carry_gram, void* O,
                                void* saved, void* scratch, float* final_state, float* final_gram, int device,
                                void* stream) {
  using namespace pr;
  Sizes s;
  int rc = sizes_of(prob, &s);
  if (rc) return rc;
  PR_REQUIRE(Q && K && V && O && saved && scratch, PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE(aligned32(saved) && aligned32(scratch), PR_ERR_BAD_ARG, "workspaces must be 32-byte aligned");
  PR_REQUIRE((carry_state == nullptr) == (carry_gram == nullptr), PR_ERR_BAD_ARG, "the two carries come together");
  PR_REQUIRE((final_state == nullptr) == (final_gram == nullptr), PR_ERR_BAD_ARG, "the two final carries come together");
  const pr_problem& p = *prob;
  const bool gated = log_G != nullptr;
  Saved sv = carve_saved(saved, s);
  Carver c{static_cast<uint8_t*>(scratch)};
  void* KT = c.take<void>(s.KT);
  float* gram = c.take<float>(s.gram);
  const long long E = (long long)s.DR * p.d;
  // Nothing reads the last chunk's state when no final state is asked for (the scan loads what lies there and drops
  // it): neither its keys' copy nor the state is made.  One chunk of five at b4 t5000 h2x4, where it and the first
  // chunk's dZ below took 529 -> 509 us off forward and backward; one of 64 at b1 t65536.
  const int used = final_state ? s.n : s.n - 1;
  // gate sums, discounted transposed keys
  if ((rc = gate_prep(p.dtype, p.b, p.t, p.h, p.h, p.d, p.c, log_G, K, gated ? sv.a : nullptr, sv.A, KT, nullptr,
                      nullptr, 0, 1.f, 1, 0, used, device, stream)))
    return rc;
  // chunk states and Gram matrices, then their scans (in place: Z[m] = state entering chunk m)
  if ((rc = chunk_state(p.dtype, p.b, p.t, p.h, 1, p.d, p.c, KT, KT, V, sv.Z, gram, 1, 0, used, device, stream)))
    return rc;
  if ((rc = pr_state_scan_fwd(p.dtype, p.b, s.n, p.h, p.d, E, sv.Z, sv.A, carry_state, final_state, gram, sv.zhi,
                              sv.zlo, sv.zfull, carry_gram, final_gram, device, stream)))
    return rc;
  // attention + state read-out + normalisation
  return chunk_out(p.dtype, p.b, p.t, p.t, p.c, p.c, p.hq, p.h, p.d, Q, K, V, gated ? sv.a : nullptr, sv.Z, sv.zhi,
                      sv.zlo, carry_state ? 0 : 1, 0, 1, p.scale, 2, O, sv.l, device, stream);
}

extern "C" int pr_retention_bwd(const pr_problem* prob, const void* Q, const void* K, const void* V,
                                const float* log_G, const void* O, const void* dO, int had_carry, void* saved,
                                void* scratch, void* dQ, void* dK, void* dV, float* dlog_G, int device, void* stream) {
  using namespace pr;
  Sizes s;
  int rc = sizes_of(prob, &s);
  if (rc) return rc;
  PR_REQUIRE(Q && K && V && O && dO && saved && scratch && dQ && dK && dV, PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE(aligned32(saved) && aligned32(scratch), PR_ERR_BAD_ARG, "workspaces must be 32-byte aligned");
  const pr_problem& p = *prob;
  const bool gated = log_G != nullptr;
  PR_REQUIRE(!gated || dlog_G != nullptr, PR_ERR_BAD_ARG, "gated problem without a dlog_G output");
  Saved sv = carve_saved(saved, s);
  Carver c{static_cast<uint8_t*>(scratch)};
  void* dy = c.take<void>(s.dy);
  float* dl = c.take<float>(s.dl);
  void* QT = c.take<void>(s.QT);
  void* QTs = c.take<void>(s.QT);
  void* dZ = c.take<void>(s.dZ);
  float* dZg = c.take<float>(s.dZg);
  float* partS = c.take<float>(s.partS);
  float* partG = c.take<float>(s.partG);
  void* ghi = c.take<void>(s.gh);
  void* glo = c.take<void>(s.gh);
  float* dqs = c.take<float>(s.dqs);
  float* gq = c.take<float>(s.gq);
  float* dks = c.take<float>(s.dks);
  float* wk = c.take<float>(s.wk);
  float* daq = c.take<float>(s.daq);
  float* dak = c.take<float>(s.dak);
  const long long E = (long long)s.DR * p.d;
  const float* a = gated ? sv.a : nullptr;
  const float* A = gated ? sv.A : nullptr;
  const int group = p.hq / p.h;
  // dy = dO / l, dl = -<O, dO> / l
  if ((rc = pr_dout_prep(p.dtype, (long long)p.b * p.t * p.hq, p.d, O, dO, sv.l, dy, dl, device, stream))) return rc;

  // ---- query side, on the second stream when there is one: gradient through the read-out's expansion
  // (saved states), then the attention backward merged with it
  Fork fork;
  if ((rc = fork.begin(device, stream))) return rc;
  void* qstream = fork.side();
  rc = pr_expand_grad(p.dtype, p.b, p.t, p.h, p.hq, p.d, p.c, dy, Q, sv.Z, sv.zhi, sv.zlo, a, A, dl, 1, p.scale, 2.f,
                      had_carry ? 0 : 1, s.n - 1, dqs, gq, device, qstream);
  if (!rc)
    rc = pr_chunk_dq(p.dtype, p.b, p.t, p.hq, p.h, p.d, p.c, Q, dO, K, V, a, dl, sv.l, dqs, p.scale, 2, dQ, daq, device,
                     qstream);
  fork.side_done();

  // ---- key side: gradient of the state read-out (dZ_m, dZg_m from the gated queries; the forward's
  // cumulative gates are read, not rescanned), reverse scans (in place: dZ becomes w (.) dS_m), gradient
  // through the chunk states' expansion, attention backward merged with it
  // (no gradient is asked of the state that enters the first chunk: its dZ is not made)
  if (!rc)
    rc = gate_prep(p.dtype, p.b, p.t, p.h, p.hq, p.d, p.c, log_G, Q, gated ? sv.a : nullptr, nullptr, QT, dl, QTs, 1,
                   p.scale, 0, 1, s.n - 1, device, stream);
  if (!rc)
    rc = chunk_state(p.dtype, p.b, p.t, p.h, group, p.d, p.c, QT, QTs, dy, dZ, dZg, 0, 1, s.n - 1, device, stream);
  if (!rc)
    rc = pr_state_scan_bwd(p.dtype, p.b, s.n, p.h, p.d, E, dZ, sv.Z, sv.A, nullptr, nullptr, partS, dZg, sv.zfull, ghi,
                           glo, nullptr, nullptr, partG, device, stream);
  if (!rc)
    rc = pr_expand_grad(p.dtype, p.b, p.t, p.h, p.h, p.d, p.c, V, K, dZ, ghi, glo, a, A, nullptr, 0, 1.f, 1.f, 0,
                        s.n - 2, dks, wk, device, stream);
  if (!rc)
    rc = pr_chunk_dkv(p.dtype, p.b, p.t, p.hq, p.h, p.d, p.c, Q, dO, K, V, dZ, a, A, dl, sv.l, dks, s.n - 2, p.scale, 2,
                      dK, dV, dak, device, stream);
  rc = fork.join(rc);
  if (rc) return rc;
  if (gated)
    return pr_gate_grad(p.b, p.t, p.h, p.hq, p.c, daq, gq, dak, wk, partS, s.blocksS, partG, s.blocksG, dlog_G, device,
                        stream);
  return PR_OK;
}

// ---- The state-free branch: one chunk holds the whole sequence, so there is no state to form, scan or read.
namespace pr {
namespace {

// Saved from forward to backward: gate sums, row sums.  Backward scratch: dl, da_q, da_k.
int attention_check(const pr_problem* p, int deg) {
  PR_REQUIRE(p != nullptr, PR_ERR_BAD_ARG, "problem is null");
  PR_REQUIRE(p->d == 16 || p->d == 32 || p->d == 64, PR_ERR_BAD_ARG, "head dim %d: this build handles 16, 32 and 64", p->d);
  PR_REQUIRE(p->dtype == PR_BF16 || p->dtype == PR_FP16, PR_ERR_BAD_ARG, "dtype %d", p->dtype);
  PR_REQUIRE(p->b > 0 && p->t > 0 && p->h > 0 && p->hq > 0 && p->hq % p->h == 0, PR_ERR_BAD_ARG,
             "bad sizes b=%d t=%d h=%d hq=%d", p->b, p->t, p->h, p->hq);
  PR_REQUIRE(deg == 2 || deg == 4, PR_ERR_BAD_ARG, "deg=%d: 2 or 4", deg);
  return PR_OK;
}

}  // namespace
}  // namespace pr

extern "C" int pr_attention_workspace_bytes(const pr_problem* prob, int what, size_t* out) {
  using namespace pr;
  PR_REQUIRE(out != nullptr, PR_ERR_BAD_ARG, "out is null");
  int rc = attention_check(prob, 2);
  if (rc) return rc;
  const size_t a = up((size_t)prob->b * prob->t * prob->h * 4), l = up((size_t)prob->b * prob->t * prob->hq * 4);
  PR_REQUIRE(what == PR_WS_SAVED || what == PR_WS_BWD_SCRATCH, PR_ERR_BAD_ARG, "workspace kind %d", what);
  *out = what == PR_WS_SAVED ? a + l : a + 2 * l;
  return PR_OK;
}

extern "C" int pr_attention_fwd(const pr_problem* prob, int deg, const void* Q, const void* K, const void* V,
                                const float* log_G, void* O, void* saved, int device, void* stream) {
  using namespace pr;
  int rc = attention_check(prob, deg);
  if (rc) return rc;
  PR_REQUIRE(Q && K && V && O && saved, PR_ERR_BAD_ARG, "null pointer");
  const pr_problem& p = *prob;
  Carver c{static_cast<uint8_t*>(saved)};
  float* a = c.take<float>(up((size_t)p.b * p.t * p.h * 4));
  float* l = c.take<float>(0);
  // one chunk longer than the chunk-local scan holds in shared memory takes the plain cumulative sum
  if (log_G != nullptr) {
    if (p.t > 16384)
      rc = pr_gate_cumsum(p.b, p.t, p.h, log_G, (long long)p.t * p.h, a, device, stream);
    else
      rc = pr_gate_prep(p.dtype, p.b, p.t, p.h, p.h, p.d, p.t, log_G, K, a, nullptr, nullptr, nullptr, nullptr, 0, 1.f,
                        1, device, stream);
    if (rc) return rc;
  }
  return chunk_out(p.dtype, p.b, p.t, p.t, p.t, p.t, p.hq, p.h, p.d, Q, K, V, log_G ? a : nullptr, nullptr, nullptr,
                   nullptr, 1, 0, 1, p.scale, deg, O, l, device, stream);
}

extern "C" int pr_attention_bwd(const pr_problem* prob, int deg, const void* Q, const void* K, const void* V,
                                const float* log_G, const void* O, const void* dO, void* saved, void* scratch, void* dQ,
                                void* dK, void* dV, float* dlog_G, int device, void* stream) {
  using namespace pr;
  int rc = attention_check(prob, deg);
  if (rc) return rc;
  PR_REQUIRE(Q && K && V && O && dO && saved && scratch && dQ && dK && dV, PR_ERR_BAD_ARG, "null pointer");
  PR_REQUIRE(log_G == nullptr || dlog_G != nullptr, PR_ERR_BAD_ARG, "gated problem without a dlog_G output");
  const pr_problem& p = *prob;
  const size_t asz = up((size_t)p.b * p.t * p.h * 4), lsz = up((size_t)p.b * p.t * p.hq * 4);
  Carver c{static_cast<uint8_t*>(saved)};
  const float* a = c.take<float>(asz);
  const float* l = c.take<float>(lsz);
  if (log_G == nullptr) a = nullptr;
  Carver w{static_cast<uint8_t*>(scratch)};
  float* dak = w.take<float>(asz);
  float* dl = w.take<float>(lsz);
  float* daq = w.take<float>(lsz);
  if ((rc = dout_prep(p.dtype, (long long)p.b * p.t * p.hq, p.d, O, dO, l, nullptr, dl, device, stream))) return rc;
  Fork fork;
  if ((rc = fork.begin(device, stream))) return rc;
  // Both kernels hold one CTA per SM while they have tiles.  With grouped queries chunk_dkv's tiles, one per key tile of a
  // kv head, are fewer and longer: in front they leave SMs to chunk_dq from the start, behind it they run alone at the
  // end.  Eager launches come out in that order anyway, a replayed graph keeps the one they were recorded in.  With as many
  // kv heads as query heads the grids are equal and either order is within 4 % of the other.  Replayed forward and
  // backward in us, chunk_dq / chunk_dkv first: b4 t2048 h2x4 239 / 154, b4 t2048 h2x12 639 / 351, b1 t2048 h2x12 472 / 288,
  // b8 t1024 h4x8 332 / 272; b1 t2048 h4 64 / 64, b4 t2048 h8 170 / 166, b4 t2000 h4 119 / 123, b1 t7200 h4 325 / 334.
  const bool keys_first = p.hq > p.h;
  auto query_side = [&] {
    return pr_chunk_dq(p.dtype, p.b, p.t, p.hq, p.h, p.d, p.t, Q, dO, K, V, a, dl, l, nullptr, p.scale, deg, dQ, daq, device,
                       fork.side());
  };
  if (!keys_first) rc = query_side();
  if (!rc)
    rc = pr_chunk_dkv(p.dtype, p.b, p.t, p.hq, p.h, p.d, p.t, Q, dO, K, V, nullptr, a, nullptr, dl, l, nullptr, -1,
                      p.scale, deg, dK, dV, dak, device, stream);
  if (keys_first && !rc) rc = query_side();
  fork.side_done();
  rc = fork.join(rc);
  if (rc || log_G == nullptr) return rc;
  return pr_gate_grad(p.b, p.t, p.h, p.hq, p.t, daq, nullptr, dak, nullptr, nullptr, 0, nullptr, 0, dlog_G, device,
                      stream);
}
