// C ABI (include/transducer_b200.h) and the reference-compatible C++-linkage entry
// points (include/transducer.h) on top of the kernel launchers.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <sstream>
#include <string>

#include "../../include/transducer.h"
#include "../../include/transducer_b200.h"
#include "../../include/transducer_cuda.h"
#include "api_internal.h"
#include "kernels.h"
#include "profile.h"

namespace tb200 {
namespace {

thread_local cudaStream_t g_stream = nullptr;
thread_local std::string g_error;

// Process-wide switches (tb200_set_option); atomics, because the stream and the error
// message are per thread but these are shared.
struct Options {
  std::atomic<int> lognorm_path{0};
  std::atomic<int> grads_path{0};
  std::atomic<int> grad_passes{2};
  std::atomic<int> fused_gather{1};
  std::atomic<int> maxplus_path{0};   // 0 auto, 1 dense, 2 pruned (error if unsupported)
};
Options g_opt;

int fail(int code, const std::string& msg) {
  g_error = msg;
  return code;
}

// Runs `body`, mapping exceptions to status codes.
template <typename F>
int guarded(F&& body) {
  try {
    body();
    return kOk;
  } catch (const CudaError& e) {
    return fail(kErrCuda, e.what());
  } catch (const std::invalid_argument& e) {
    return fail(kErrInvalidArgument, e.what());
  } catch (const std::exception& e) {
    return fail(kErrCuda, e.what());
  }
}

void check_dims(const Dims& d) {
  if (d.B < 0 || d.maxT < 0 || d.maxU < 0 || d.V <= 0)
    throw std::invalid_argument("negative batch/length or non-positive alphabet size");
  if (d.blank < 0 || d.blank >= d.V) throw std::invalid_argument("blank outside [0, alphabetSize)");
}

// Bump allocator over the caller's workspace; every block is 256-byte aligned.
struct Carver {
  char* base;
  size_t used = 0;
  explicit Carver(void* p) : base(static_cast<char*>(p)) {}
  template <typename T>
  T* take(size_t n) {
    used = (used + 255) & ~size_t(255);
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += n * sizeof(T);
    return p;
  }
  size_t total() const { return (used + 255) & ~size_t(255); }
};

int ld_w(const Dims& d) { return (int)round_up64(d.maxU > 0 ? d.maxU : 1, 32); }

struct LogNormWs {
  unsigned* ticket;  // alpha kernel's completion counters: of the batch, then of the utterances
  float* split;      // exp(P) hi/lo operand of the tensor-core path
  float* maxPScratch;
  LogNormWs(Carver& c, const Dims& d) {
    ticket = c.take<unsigned>(16 + (size_t)d.B);
    maxPScratch = c.take<float>((size_t)d.B * d.maxU);
    split = c.take<float>(lognorm_umma_workspace_floats(d));
  }
};

// What the forward call leaves for the backward call (opaque to the caller).
struct SavedState {
  float *rowRef, *maxP, *alphas, *ebl;
  float *LN = nullptr, *deltas = nullptr;                 // label axis <= 256
  float2* arcs = nullptr;
  float *LNs = nullptr, *ELs = nullptr;                   // longer ones
  SavedState(Carver& c, const Dims& d) {
    const size_t B = d.B;
    rowRef = c.take<float>(B * d.maxT);
    maxP = c.take<float>(B * d.maxU);
    ebl = c.take<float>(B * d.maxT);
    if (sweep_supported(d)) {
      const SweepGeom g = sweep_geom(d);
      alphas = c.take<float>(B * g.stride);
      arcs = c.take<float2>(B * g.stride);
      LN = c.take<float>(B * d.maxT * d.maxU);
      deltas = c.take<float>(B * std::max(g.nBlk, 2));   // (costs alone: an offset per half)
    } else {
      const SkewGeom g = skew_geom(d);
      alphas = c.take<float>(B * g.stride);
      LNs = c.take<float>(B * g.stride);
      ELs = c.take<float>(B * g.stride);
    }
  }
};

struct ForwardWs {
  float* EL;  // label emissions E[t,label_u] gathered by the log-normaliser pass
  float* LN;        // row-major log-normalisers before the re-layout (label axis > 256)
  ForwardWs(Carver& c, const Dims& d) {
    const size_t cells = (size_t)d.B * d.maxT * d.maxU;
    EL = c.take<float>(lognorm_umma_gathers(d) ? cells : 0);
    LN = c.take<float>(sweep_supported(d) ? 0 : cells);
  }
};

struct BackwardWs {
  float *expP, *W, *em, *emT, *nref, *ebl, *eBlank, *pBlank, *pLabel, *maxPScratch;
  SweepScratch sweep{};                 // label axis <= 256
  float* gradPartial = nullptr;
  float *Ws = nullptr, *EMs = nullptr;  // longer ones
  BackwardWs(Carver& c, const Dims& d) {
    const size_t B = d.B, T = d.maxT, U = d.maxU, V = d.V;
    expP = c.take<float>(B * U * V);  // SIMT path only
    if (sweep_supported(d)) {
      const SweepGeom g = sweep_geom(d);
      sweep.F = c.take<float2>(B * g.stride);
      sweep.g = c.take<float>(B * g.stride);
      sweep.ticket = c.take<unsigned>(B);
      sweep.gradTickets = c.take<unsigned>(kGradTickets);
      gradPartial = c.take<float>(grads_umma_partial_floats(d));
      sweep.partial = c.take<float>(sweep_partial_floats(d));
    } else {
      const SkewGeom g = skew_geom(d);
      Ws = c.take<float>(B * g.stride);
      EMs = c.take<float>(B * g.stride);
    }
    W = c.take<float>(B * T * ld_w(d));
    em = c.take<float>(B * T * U);            // SIMT path
    emT = c.take<float>(B * U * grads_umma_ld_t(d));  // tensor-core path
    nref = c.take<float>(B * grads_umma_ld_t(d));
    ebl = c.take<float>(B * grads_umma_ld_t(d));
    eBlank = c.take<float>(B * T);
    pBlank = c.take<float>(B * U);
    pLabel = c.take<float>(B * U);
    maxPScratch = c.take<float>(B * U);
  }
};

struct ViterbiWs {
  float *LN, *rowRef, *maxP, *best;
  uint32_t* decBits;
  float* nodes;   // skewed operands of the single-warp sweep (label axis <= 256)
  char* prune;    // candidate lists of the pruned max-plus (null where it does not apply)
  ViterbiWs(Carver& c, const Dims& d) {
    const size_t B = d.B, T = d.maxT, U = d.maxU;
    LN = c.take<float>(B * T * U);
    rowRef = c.take<float>(B * T);
    maxP = c.take<float>(B * U);
    best = c.take<float>(B * T * U);
    decBits = c.take<uint32_t>(std::max(viterbi_decbits_words(d), viterbi_warp_decbits_words(d)));
    nodes = c.take<float>(viterbi_warp_scratch_floats(d));
    prune = c.take<char>(maxplus_pruned_scratch_bytes(d));
  }
};

// Label-arc scores of every node, by the pruned evaluation where it applies.
void best_label_scores(const float* E, const float* P, float* best, const int* inLens,
                       const int* labLens, const Dims& d, void* pruneScratch) {
  const bool can = maxplus_pruned_supported(d) && pruneScratch != nullptr;
  if (g_opt.maxplus_path == 2 && !can)
    throw std::invalid_argument("pruned max-plus does not apply to these sizes");
  if (can && g_opt.maxplus_path != 1)
    launch_maxplus_pruned(E, P, best, inLens, labLens, d, pruneScratch, device_status_word(),
                          g_stream);
  else
    launch_maxplus(E, P, best, inLens, labLens, d, g_stream);
}

void need(size_t have, size_t want, const void* ws) {
  if (want > 0 && (ws == nullptr || have < want))
    throw std::invalid_argument("workspace too small: need " + std::to_string(want) +
                                " bytes, got " + std::to_string(have));
}

// Log-normalisers plus the row shifts.  With the SIMT kernels rowRef is the true row
// maximum of E.
// keepBits: where gradients follow, or may follow, the weights behind the sweeps are rounded to TF32, and other
// log-normalisers, however close, would flip some of those roundings (lattice_sweep.cu): the TF32 kernel at any size.
// Returns true if the pass also produced the label / blank emissions (EL, ebl) it was offered.
bool log_norms_impl(const void* E, const void* P, float* LN, float* rowRef, float* maxP,
                    const int* inLens, const int* labLens, const Dims& d, LogNormWs& ws,
                    bool fixup = true, const int* labels = nullptr, float* EL = nullptr,
                    float* ebl = nullptr, bool keepBits = true) {
  if (d.B <= 0 || d.maxT <= 0 || d.maxU <= 0) return false;
  const bool can = lognorm_umma_supported(E, P, d);
  const int path = g_opt.lognorm_path;
  const bool tensorCore = can && (path == 0 || path == 2 || path == 4);
  if ((path == 2 || path == 4) && !can)
    throw std::invalid_argument(
        "tensor-core log-normaliser needs alphabetSize % 4 == 0, alphabetSize >= 32, "
        "maxLabelLength <= 256 and 16-byte aligned emissions");
  if (d.dtype != kDtypeF32 && !tensorCore)
    throw std::invalid_argument(
        "bf16 emissions need the tensor-core log-normaliser: alphabetSize % 8 == 0, "
        "alphabetSize >= 32, 16-byte aligned emissions and predictions");
  if (tensorCore) {
    // the kernel needs somewhere to put the row shifts even if the caller does not want them
    float* mp = maxP ? maxP : ws.maxPScratch;
    if (!rowRef) throw std::invalid_argument("rowRef must not be null");
    // Emissions that stay in the L2 (126 MB) until the re-layout are gathered there: handing them out
    // costs this kernel 5..10 us (the labels are sorted, and a chunk's labels are served one after the
    // other), a gather from L2 1..3 us.  Forward time of the two kernels, handed out / gathered:
    // E of 6 MB 60 / 51 us, 65 MB 88 / 84, 256 MB 138 / 144, 640 MB 260 / 270.
    const size_t bytesE = (size_t)d.B * d.maxT * d.V * (d.dtype == kDtypeBf16 ? 2 : 4);
    const int handOut = g_opt.fused_gather;
    const bool gathers = labels && EL && ebl && lognorm_umma_gathers(d) &&
                         (handOut == 2 || (handOut == 1 && bytesE > (size_t)96 << 20));
    launch_lognorm_umma(E, P, LN, rowRef, mp, inLens, labLens, d, ws.split,
                        device_status_word(),
                        path == 4                                           ? PairFormat::f16
                        : path == 0 && !keepBits && lognorm_f16_pays(d) ? PairFormat::f16_if_close
                                                                            : PairFormat::tf32,
                        fixup, g_stream, gathers ? labels : nullptr,
                        gathers ? EL : nullptr, gathers ? ebl : nullptr);
    return gathers;
  }
  const float* Ef = static_cast<const float*>(E);
  const float* Pf = static_cast<const float*>(P);
  const bool exact = path == 1 || rowRef == nullptr || (path != 3 && !lognorm_factored_pays(d));
  launch_lognorm_simt(Ef, Pf, LN, rowRef, exact ? maxP : (maxP ? maxP : ws.maxPScratch), inLens,
                      labLens, d, exact, exact ? nullptr : device_status_word(), g_stream);
  if (!exact && fixup) launch_lognorm_fixup(E, P, LN, inLens, labLens, d, g_stream);
  return false;
}

}  // namespace

int api_fail(int code, const std::string& msg) { return fail(code, msg); }
cudaStream_t api_stream() { return g_stream; }

}  // namespace tb200

using namespace tb200;

extern "C" {

int tb200_version(void) { return 100; }

const char* tb200_last_error(void) { return g_error.c_str(); }

int tb200_set_stream(void* stream) {
  g_stream = static_cast<cudaStream_t>(stream);
  return kOk;
}
void* tb200_get_stream(void) { return g_stream; }

int tb200_set_option(const char* key, int value) {
  if (!key) return fail(kErrInvalidArgument, "null option key");
  if (!strcmp(key, "lognorm_path") && value >= 0 && value <= 4) g_opt.lognorm_path = value;
  else if (!strcmp(key, "grads_path") && value >= 0 && value <= 2) g_opt.grads_path = value;
  else if (!strcmp(key, "grad_passes") && value >= 1 && value <= 3) g_opt.grad_passes = value;
  else if (!strcmp(key, "fused_gather") && value >= 0 && value <= 2) g_opt.fused_gather = value;
  else if (!strcmp(key, "maxplus_path") && value >= 0 && value <= 2) g_opt.maxplus_path = value;
  else return fail(kErrInvalidArgument, std::string("unknown option or bad value: ") + key);
  return kOk;
}

int tb200_get_option(const char* key, int* value) {
  if (!key || !value) return fail(kErrInvalidArgument, "null argument");
  if (!strcmp(key, "lognorm_path")) *value = g_opt.lognorm_path;
  else if (!strcmp(key, "grads_path")) *value = g_opt.grads_path;
  else if (!strcmp(key, "grad_passes")) *value = g_opt.grad_passes;
  else if (!strcmp(key, "fused_gather")) *value = g_opt.fused_gather;
  else if (!strcmp(key, "maxplus_path")) *value = g_opt.maxplus_path;
  else return fail(kErrInvalidArgument, std::string("unknown option: ") + key);
  return kOk;
}

long long tb200_launch_count(void) { return launch_count(); }
int tb200_profile_enable(int on) {
  profile_enable(on != 0);
  return kOk;
}
int tb200_profile_reset(void) {
  profile_reset();
  return kOk;
}
size_t tb200_profile_report(char* buf, size_t bufBytes) {
  const std::string s = profile_report();
  if (buf && bufBytes > 0) {
    const size_t n = s.size() < bufBytes - 1 ? s.size() : bufBytes - 1;
    memcpy(buf, s.data(), n);
    buf[n] = 0;
  }
  return s.size();
}

int tb200_forward(const float* E, const float* P, float* costs, float* alphas,
                  const float* LN, const int* labels, const int* inLens,
                  const int* labLens, int B, int maxT, int maxU, int V, int blank) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank};
    check_dims(d);
    launch_alpha(E, P, costs, alphas, LN, labels, inLens, labLens, d, nullptr, nullptr,
                 g_stream);
  });
}

int tb200_backward(const float* E, const float* P, float* egrads, float* pgrads,
                   float* lngrads, const float* alphas, const float* LN,
                   const int* labels, const int* inLens, const int* labLens, int B,
                   int maxT, int maxU, int V, int blank) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank};
    check_dims(d);
    const size_t b = B, t = maxT, u = maxU, v = V;
    if (b * t * v) TB200_CUDA_CHECK(cudaMemsetAsync(egrads, 0, sizeof(float) * b * t * v, g_stream));
    if (b * u * v) TB200_CUDA_CHECK(cudaMemsetAsync(pgrads, 0, sizeof(float) * b * u * v, g_stream));
    if (b * t * u) TB200_CUDA_CHECK(cudaMemsetAsync(lngrads, 0, sizeof(float) * b * t * u, g_stream));
    launch_gamma_abi(E, P, egrads, pgrads, lngrads, alphas, LN, labels, inLens, labLens, d,
                     g_stream);
  });
}

int tb200_viterbi(const float* E, const float* P, const float* LN, int* labels,
                  const int* inLens, const int* labLens, int B, int maxT, int maxU, int V,
                  int blank) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank};
    check_dims(d);
    if (B == 0 || maxT == 0 || maxU == 0) return;
    const size_t cells = (size_t)B * maxT * maxU;
    const bool warp = viterbi_warp_supported(d);  // label axis <= 256: single-warp sweep
    const size_t decWords = warp ? viterbi_warp_decbits_words(d) : viterbi_decbits_words(d);
    // Temporaries from the stream-ordered allocator, as the reference takes them
    // (transducer_cuda.cu:364-369); released in stream order on every way out.
    struct Temporaries {
      float* best = nullptr;
      uint32_t* dec = nullptr;
      float* nodes = nullptr;
      void* prune = nullptr;
      cudaStream_t stream;
      ~Temporaries() {
        if (best) cudaFreeAsync(best, stream);
        if (dec) cudaFreeAsync(dec, stream);
        if (nodes) cudaFreeAsync(nodes, stream);
        if (prune) cudaFreeAsync(prune, stream);
      }
    } tmp;
    tmp.stream = g_stream;
    TB200_CUDA_CHECK(cudaMallocAsync((void**)&tmp.best, sizeof(float) * cells, g_stream));
    TB200_CUDA_CHECK(cudaMallocAsync((void**)&tmp.dec, sizeof(uint32_t) * decWords, g_stream));
    if (warp)
      TB200_CUDA_CHECK(cudaMallocAsync((void**)&tmp.nodes, sizeof(float) * viterbi_warp_scratch_floats(d),
                                       g_stream));
    if (maxplus_pruned_supported(d) && g_opt.maxplus_path != 1)
      TB200_CUDA_CHECK(cudaMallocAsync(&tmp.prune, maxplus_pruned_scratch_bytes(d), g_stream));
    best_label_scores(E, P, tmp.best, inLens, labLens, d, tmp.prune);
    if (warp)
      launch_viterbi_warp(E, P, const_cast<float*>(LN), /*fix=*/false, tmp.best, tmp.nodes, tmp.dec, labels,
                          inLens, labLens, d, g_stream);
    else
      launch_viterbi_lattice(E, P, LN, tmp.best, tmp.dec, labels, inLens, labLens, d, g_stream);
  });
}

size_t tb200_log_norms_workspace_bytes(int B, int maxT, int maxU, int V) {
  Dims d{B, maxT, maxU, V, 0};
  Carver c(nullptr);
  LogNormWs ws(c, d);
  return c.total();
}

int tb200_log_norms(const float* E, const float* P, float* LN, float* rowRef, float* maxP,
                    const int* inLens, const int* labLens, int B, int maxT, int maxU, int V,
                    void* workspace, size_t workspaceBytes) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, 0};
    check_dims(d);
    need(workspaceBytes, tb200_log_norms_workspace_bytes(B, maxT, maxU, V), workspace);
    Carver c(workspace);
    LogNormWs ws(c, d);
    log_norms_impl(E, P, LN, rowRef, maxP, inLens, labLens, d, ws);
  });
}

size_t tb200_loss_saved_bytes(int B, int maxT, int maxU, int V) {
  Dims d{B, maxT, maxU, V, 0};
  Carver c(nullptr);
  SavedState s(c, d);
  return c.total();
}

size_t tb200_loss_forward_workspace_bytes(int B, int maxT, int maxU, int V) {
  Dims d{B, maxT, maxU, V, 0};
  Carver c(nullptr);
  ForwardWs f(c, d);
  LogNormWs l(c, d);
  return c.total();
}

namespace {

// score: no backward call will read what is left in `saved`, which may then sit behind the workspace.
int loss_forward_any(const void* E, const void* P, const int* labels, const int* inLens,
                     const int* labLens, float* costs, float* lossSum, void* saved,
                     size_t savedBytes, int B, int maxT, int maxU, int V, int blank,
                     void* workspace, size_t workspaceBytes, int dtype, bool score = false) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank, dtype};
    check_dims(d);
    if (dtype != kDtypeF32 && maxU > 128)
      throw std::invalid_argument("bf16 emissions: the label axis must not exceed 128 positions");
    const size_t forwardBytes = tb200_loss_forward_workspace_bytes(B, maxT, maxU, V);
    need(workspaceBytes, score ? tb200_loss_score_workspace_bytes(B, maxT, maxU, V) : forwardBytes, workspace);
    if (score) saved = static_cast<char*>(workspace) + forwardBytes;
    else need(savedBytes, tb200_loss_saved_bytes(B, maxT, maxU, V), saved);
    Carver cs(saved);
    SavedState st(cs, d);
    Carver c(workspace);
    ForwardWs fw(c, d);
    LogNormWs ws(c, d);
    // The shape (and whether a backward call may follow) alone decides which sweeps run: the backward call
    // must pick the ones that match the saved state.
    const bool sweep = sweep_supported(d);
    float* LN = sweep ? st.LN : fw.LN;
    // (nodes the tensor-core log-normaliser could not represent are recomputed by the re-layout)
    const bool gathered = log_norms_impl(E, P, LN, st.rowRef, st.maxP, inLens, labLens, d, ws,
                                         /*fixup=*/false, labels, fw.EL, st.ebl,
                                         /*keepBits=*/!score);
    TB200_CUDA_CHECK(cudaMemsetAsync(ws.ticket, 0, sizeof(unsigned) * (16 + (size_t)B), g_stream));
    if (lossSum && B == 0) TB200_CUDA_CHECK(cudaMemsetAsync(lossSum, 0, sizeof(float), g_stream));
    unsigned* ticket = lossSum ? ws.ticket : nullptr;
    if (sweep) {
      launch_sweep_forward(E, P, LN, gathered ? fw.EL : nullptr, st.ebl, st.arcs,
                           st.alphas, st.deltas, costs, lossSum, ticket, ws.ticket + 16, labels, inLens,
                           labLens, sweep_geom(d), d, score, g_stream);
      return;
    }
    const SkewGeom g = skew_geom(d);
    const float* Ef = static_cast<const float*>(E);
    const float* Pf = static_cast<const float*>(P);
    launch_lattice_prep(Ef, Pf, LN, st.LNs, st.ELs, st.ebl, labels, inLens, labLens, g, d, g_stream);
    launch_alpha_skew(Pf, costs, st.alphas, st.LNs, st.ELs, st.ebl, g, labels, inLens, labLens, d,
                      lossSum, ticket, g_stream);
  });
}

}  // namespace

int tb200_loss_forward(const float* E, const float* P, const int* labels, const int* inLens,
                       const int* labLens, float* costs, float* lossSum, void* saved,
                       size_t savedBytes, int B, int maxT, int maxU, int V, int blank,
                       void* workspace, size_t workspaceBytes) {
  return loss_forward_any(E, P, labels, inLens, labLens, costs, lossSum, saved, savedBytes, B, maxT,
                          maxU, V, blank, workspace, workspaceBytes, kDtypeF32);
}

int tb200_loss_forward_bf16(const void* E, const void* P, const int* labels, const int* inLens,
                            const int* labLens, float* costs, float* lossSum, void* saved,
                            size_t savedBytes, int B, int maxT, int maxU, int V, int blank,
                            void* workspace, size_t workspaceBytes) {
  return loss_forward_any(E, P, labels, inLens, labLens, costs, lossSum, saved, savedBytes, B, maxT,
                          maxU, V, blank, workspace, workspaceBytes, kDtypeBf16);
}

size_t tb200_loss_score_workspace_bytes(int B, int maxT, int maxU, int V) {
  return tb200_loss_forward_workspace_bytes(B, maxT, maxU, V) + tb200_loss_saved_bytes(B, maxT, maxU, V);
}

int tb200_loss_score(const float* E, const float* P, const int* labels, const int* inLens,
                     const int* labLens, float* costs, float* lossSum, int B, int maxT, int maxU, int V,
                     int blank, void* workspace, size_t workspaceBytes) {
  return loss_forward_any(E, P, labels, inLens, labLens, costs, lossSum, nullptr, 0, B, maxT, maxU, V, blank,
                          workspace, workspaceBytes, kDtypeF32, /*score=*/true);
}

int tb200_loss_score_bf16(const void* E, const void* P, const int* labels, const int* inLens,
                          const int* labLens, float* costs, float* lossSum, int B, int maxT, int maxU, int V,
                          int blank, void* workspace, size_t workspaceBytes) {
  return loss_forward_any(E, P, labels, inLens, labLens, costs, lossSum, nullptr, 0, B, maxT, maxU, V, blank,
                          workspace, workspaceBytes, kDtypeBf16, /*score=*/true);
}

size_t tb200_loss_backward_workspace_bytes(int B, int maxT, int maxU, int V) {
  Dims d{B, maxT, maxU, V, 0};
  Carver c(nullptr);
  BackwardWs ws(c, d);
  return c.total();
}

namespace {

int loss_backward_any(const void* E, const void* P, const int* labels, const int* inLens,
                      const int* labLens, const void* saved, size_t savedBytes,
                      const float* deltas, void* egrads, void* pgrads, int B, int maxT,
                      int maxU, int V, int blank, void* workspace, size_t workspaceBytes,
                      int dtype) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank, dtype};
    check_dims(d);
    need(workspaceBytes, tb200_loss_backward_workspace_bytes(B, maxT, maxU, V), workspace);
    need(savedBytes, tb200_loss_saved_bytes(B, maxT, maxU, V), saved);
    if (B == 0) return;
    Carver cs(const_cast<void*>(saved));
    SavedState st(cs, d);
    Carver c(workspace);
    BackwardWs ws(c, d);
    const int ldW = ld_w(d);
    const int passes = g_opt.grad_passes;
    const bool can = grads_umma_supported(E, P, egrads, pgrads, d, passes);
    if (g_opt.grads_path == 2 && !can)
      throw std::invalid_argument(
          "tensor-core gradients need alphabetSize % 4 == 0, alphabetSize >= 32, "
          "maxLabelLength <= 256 and 16-byte aligned emissions and egrads");
    const bool tensorCore = can && g_opt.grads_path != 1;
    const bool oneLaunch = tensorCore && maxU <= 128;
    if (dtype != kDtypeF32 && !oneLaunch)
      throw std::invalid_argument(
          "bf16 gradients need the tensor-core gradient kernel: alphabetSize % 8 == 0, "
          "maxLabelLength <= 128, grad_passes = 2, 16-byte aligned buffers");
    if ((egrads == E || pgrads == P) && !oneLaunch)
      throw std::invalid_argument(
          "gradients in place (egrads == emissions / pgrads == predictions) need the "
          "tensor-core gradient kernel: alphabetSize % 4 == 0, maxLabelLength <= 128");
    const float* Ef = static_cast<const float*>(E);   // (fp32 from here on where used as such)
    const float* Pf = static_cast<const float*>(P);
    float* egf = static_cast<float*>(egrads);
    float* pgf = static_cast<float*>(pgrads);
    if (sweep_supported(d)) {
      launch_sweep_backward(ws.sweep, Pf, st.ebl, labels, st.arcs, st.alphas, st.deltas, st.LN, st.rowRef, st.maxP,
                            deltas, ws.W, tensorCore ? ws.emT : ws.em,
                            tensorCore ? ws.nref : nullptr, tensorCore ? ws.ebl : ws.eBlank,
                            ws.pBlank, ws.pLabel, inLens, labLens, sweep_geom(d), d, tensorCore,
                            g_stream);
    } else {
      const SkewGeom g = skew_geom(d);
      launch_gamma_skew(Pf, st.alphas, st.LNs, st.ELs, st.ebl, g, st.rowRef, st.maxP, labels,
                        inLens, labLens, ws.Ws, ws.EMs, ws.eBlank, ws.pBlank, ws.pLabel, d,
                        g_stream);
      launch_lattice_unskew(ws.Ws, ws.EMs, ws.W, ldW, ws.em, inLens, labLens, g, d, g_stream);
    }
    if (tensorCore) {   // (label axes of more than 160 positions: one launch per part of the axis)
      launch_grads_umma(E, P, st.maxP, ws.W, ws.emT, ws.nref, ws.ebl, ws.pBlank, ws.pLabel, labels,
                        deltas, egrads, pgrads, inLens, labLens, d, passes, ws.gradPartial,
                        ws.sweep.gradTickets, device_status_word(), g_stream);
      return;
    }
    launch_exp_rows(Pf, ws.expP, ws.maxPScratch, labLens, B, maxU, V, g_stream);
    launch_egrad_simt(Ef, st.rowRef, ws.W, ldW, ws.expP, ws.eBlank, ws.em, labels, deltas,
                      egf, inLens, labLens, d, g_stream);
    launch_pgrad_simt(Ef, st.rowRef, ws.W, ldW, ws.expP, ws.pBlank, ws.pLabel, labels, deltas,
                      pgf, inLens, labLens, d, g_stream);
  });
}

}  // namespace

int tb200_loss_backward(const float* E, const float* P, const int* labels, const int* inLens,
                        const int* labLens, const void* saved, size_t savedBytes,
                        const float* deltas, float* egrads, float* pgrads, int B, int maxT,
                        int maxU, int V, int blank, void* workspace, size_t workspaceBytes) {
  return loss_backward_any(E, P, labels, inLens, labLens, saved, savedBytes, deltas, egrads, pgrads,
                           B, maxT, maxU, V, blank, workspace, workspaceBytes, kDtypeF32);
}

int tb200_loss_backward_bf16(const void* E, const void* P, const int* labels, const int* inLens,
                             const int* labLens, const void* saved, size_t savedBytes,
                             const float* deltas, void* egrads, void* pgrads, int B, int maxT,
                             int maxU, int V, int blank, void* workspace, size_t workspaceBytes) {
  return loss_backward_any(E, P, labels, inLens, labLens, saved, savedBytes, deltas, egrads, pgrads,
                           B, maxT, maxU, V, blank, workspace, workspaceBytes, kDtypeBf16);
}

size_t tb200_label_arc_scores_workspace_bytes(int B, int maxT, int maxU, int V) {
  Dims d{B, maxT, maxU, V, 0};
  return (maxplus_pruned_scratch_bytes(d) + 255) & ~size_t(255);
}

int tb200_label_arc_scores(const float* E, const float* P, const int* inLens, const int* labLens,
                           float* best, int B, int maxT, int maxU, int V, int blank,
                           void* workspace, size_t workspaceBytes) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank};
    check_dims(d);
    need(workspaceBytes, tb200_label_arc_scores_workspace_bytes(B, maxT, maxU, V), workspace);
    if (B == 0 || maxT == 0 || maxU == 0) return;
    best_label_scores(E, P, best, inLens, labLens, d,
                      maxplus_pruned_supported(d) ? workspace : nullptr);
  });
}

size_t tb200_viterbi_decode_workspace_bytes(int B, int maxT, int maxU, int V) {
  Dims d{B, maxT, maxU, V, 0};
  Carver c(nullptr);
  ViterbiWs ws(c, d);
  LogNormWs lw(c, d);
  return c.total();
}

int tb200_viterbi_decode(const float* E, const float* P, const int* inLens,
                         const int* labLens, int* labels, int B, int maxT, int maxU, int V,
                         int blank, void* workspace, size_t workspaceBytes) {
  return guarded([&] {
    Dims d{B, maxT, maxU, V, blank};
    check_dims(d);
    need(workspaceBytes, tb200_viterbi_decode_workspace_bytes(B, maxT, maxU, V), workspace);
    if (B == 0 || maxT == 0 || maxU == 0) return;
    Carver c(workspace);
    ViterbiWs ws(c, d);
    LogNormWs lw(c, d);
    // (nodes the log-normaliser could not represent are recomputed by the re-layout)
    const bool warp = viterbi_warp_supported(d);
    log_norms_impl(E, P, ws.LN, ws.rowRef, ws.maxP, inLens, labLens, d, lw, /*fixup=*/!warp, nullptr, nullptr,
                   nullptr, /*keepBits=*/false);
    best_label_scores(E, P, ws.best, inLens, labLens, d, ws.prune);
    if (warp)
      launch_viterbi_warp(E, P, ws.LN, /*fix=*/true, ws.best, ws.nodes, ws.decBits, labels, inLens,
                          labLens, d, g_stream);
    else
      launch_viterbi_lattice(E, P, ws.LN, ws.best, ws.decBits, labels, inLens, labLens, d,
                             g_stream);
  });
}

}  // extern "C"

// ---- transducer.h-compatible C++ entry points --------------------------------

namespace {
void rethrow(int rc) {
  if (rc == kOk) return;
  if (rc == kErrInvalidArgument) throw std::invalid_argument(tb200_last_error());
  throw std::runtime_error(tb200_last_error());
}
void require_cuda(bool useCuda) {
  if (!useCuda) throw std::invalid_argument("Transducer not built with a CPU backend.");
}
}  // namespace

void forward(const float* emissions, const float* predictions, float* costs, float* alphas,
             const float* logNorms, const int* labels, const int* inputLengths,
             const int* labelLengths, int batchSize, int maxInputLength, int maxLabelLength,
             int alphabetSize, int blank, bool useCuda) {
  require_cuda(useCuda);
  rethrow(tb200_forward(emissions, predictions, costs, alphas, logNorms, labels, inputLengths,
                        labelLengths, batchSize, maxInputLength, maxLabelLength, alphabetSize,
                        blank));
}

void backward(const float* emissions, const float* predictions, float* egrads, float* pgrads,
              float* lngrads, const float* alphas, const float* logNorms, const int* labels,
              const int* inputLengths, const int* labelLengths, int batchSize,
              int maxInputLength, int maxLabelLength, int alphabetSize, int blank,
              bool useCuda) {
  require_cuda(useCuda);
  rethrow(tb200_backward(emissions, predictions, egrads, pgrads, lngrads, alphas, logNorms,
                         labels, inputLengths, labelLengths, batchSize, maxInputLength,
                         maxLabelLength, alphabetSize, blank));
}

void viterbi(const float* emissions, const float* predictions, const float* logNorms,
             int* labels, const int* inputLengths, const int* labelLengths, int batchSize,
             int maxInputLength, int maxLabelLength, int alphabetSize, int blank,
             bool useCuda) {
  require_cuda(useCuda);
  rethrow(tb200_viterbi(emissions, predictions, logNorms, labels, inputLengths, labelLengths,
                        batchSize, maxInputLength, maxLabelLength, alphabetSize, blank));
}

// ---- transducer_cuda.h-compatible namespace (transducer/transducer_cuda.h:7-59) ----------

namespace cuda {

void cudaCheck(cudaError_t err, const char* file, int line) {
  if (err != cudaSuccess) {
    std::ostringstream ess;
    ess << '[' << file << ':' << line << "] CUDA error: " << cudaGetErrorString(err);
    throw std::runtime_error(ess.str());
  }
}

void forward(const float* emissions, const float* predictions, float* costs, float* alphas,
             const float* logNorms, const int* labels, const int* inputLengths,
             const int* labelLengths, int batchSize, int maxInputLength, int maxLabelLength,
             int alphabetSize, int blank) {
  rethrow(tb200_forward(emissions, predictions, costs, alphas, logNorms, labels, inputLengths,
                        labelLengths, batchSize, maxInputLength, maxLabelLength, alphabetSize,
                        blank));
}

void backward(const float* emissions, const float* predictions, float* egrads, float* pgrads,
              float* lngrads, const float* alphas, const float* logNorms, const int* labels,
              const int* inputLengths, const int* labelLengths, int batchSize,
              int maxInputLength, int maxLabelLength, int alphabetSize, int blank) {
  rethrow(tb200_backward(emissions, predictions, egrads, pgrads, lngrads, alphas, logNorms,
                         labels, inputLengths, labelLengths, batchSize, maxInputLength,
                         maxLabelLength, alphabetSize, blank));
}

void viterbi(const float* emissions, const float* predictions, const float* logNorms, int* labels,
             const int* inputLengths, const int* labelLengths, int batchSize, int maxInputLength,
             int maxLabelLength, int alphabetSize, int blank) {
  rethrow(tb200_viterbi(emissions, predictions, logNorms, labels, inputLengths, labelLengths,
                        batchSize, maxInputLength, maxLabelLength, alphabetSize, blank));
}

}  // namespace cuda
