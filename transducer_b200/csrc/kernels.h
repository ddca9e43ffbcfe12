// Host-side launchers of the sm_100a kernels.  Every launcher enqueues work on
// `stream` and returns without synchronising; errors are thrown as tb200::CudaError.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace tb200 {

// Problem geometry shared by all launchers (names follow transducer/transducer.h):
// emissions [B,maxT,V], predictions [B,maxU,V] (maxU = longest label + 1),
// lattices [B,maxT,maxU], labels [B,maxU-1].
// dtype: storage type of emissions, predictions and their gradients (kDtypeF32 / kDtypeBf16);
// launchers that take them as `const void*` read it, all others are fp32 only.
struct Dims {
  int B, maxT, maxU, V, blank;
  int dtype = kDtypeF32;
};

constexpr int kMaxLatticeU = 8192;  // widest label axis the wavefront kernels take

// ---- lattice.cu ------------------------------------------------------------
// transducer.h `forward`: row-major lattices, emission terms gathered from E.
void launch_alpha(const float* E, const float* P, float* costs, float* alphas,
                  const float* LN, const int* labels, const int* inLens,
                  const int* labLens, Dims d, float* lossSum, unsigned* ticket,
                  cudaStream_t stream);

// transducer.h `backward`: the three outputs must already be zero-filled; lngrads
// receives the node occupancies and the sparse blank/label terms are subtracted in
// place from egrads/pgrads.
void launch_gamma_abi(const float* E, const float* P, float* egrads, float* pgrads,
                      float* lngrads, const float* alphas, const float* LN,
                      const int* labels, const int* inLens, const int* labLens,
                      Dims d, cudaStream_t stream);

// Skewed lattice storage used by the fused path: node (t,u) of utterance b lives at
// b*stride + (t+u)*ld + u, so one wavefront step reads and writes one contiguous row.
struct SkewGeom {
  int ld;       // floats per anti-diagonal row (maxU rounded up to 32)
  int nDiag;    // rows per utterance
  i64 stride;   // floats per utterance
};
SkewGeom skew_geom(Dims d);

// Label axes of more than 256 positions (shorter ones: lattice_sweep.cu).
// LN (row-major) -> LNs (skewed); ELs[t,u] = E[t,label_u] (skewed); ebl[b,t] = E[t,blank].  NaN
// entries of LN (nodes a factored log-normaliser marked) are recomputed here exactly.
void launch_lattice_prep(const float* E, const float* P, const float* LN, float* LNs, float* ELs,
                         float* ebl, const int* labels, const int* inLens, const int* labLens,
                         SkewGeom g, Dims d, cudaStream_t stream);

void launch_alpha_skew(const float* P, float* costs, float* alphasS, const float* LNs,
                       const float* ELs, const float* ebl, SkewGeom g, const int* labels,
                       const int* inLens, const int* labLens, Dims d, float* lossSum,
                       unsigned* ticket, cudaStream_t stream);

// Fused-path reverse sweep on skewed lattices.  Writes (skewed) Ws[t,u] = occupancy *
// exp(rowRef[t] + maxP[u] - LN[t,u]) and the label-arc occupancies EMs, plus the summed
// sparse terms eBlank [B,maxT], pBlank [B,maxU], pLabel [B,maxU].
void launch_gamma_skew(const float* P, const float* alphasS, const float* LNs,
                       const float* ELs, const float* ebl, SkewGeom g, const float* rowRef,
                       const float* maxP, const int* labels, const int* inLens,
                       const int* labLens, float* Ws, float* EMs, float* eBlank,
                       float* pBlank, float* pLabel, Dims d, cudaStream_t stream);

// Ws/EMs (skewed) -> W [B,maxT,ldW] (zero outside the valid lattice) and em [B,maxT,maxU].
void launch_lattice_unskew(const float* Ws, const float* EMs, float* W, int ldW, float* em,
                           const int* inLens, const int* labLens, SkewGeom g, Dims d,
                           cudaStream_t stream);

// Max-plus wavefront + bounded on-device backtrack + label argmax on the path.
// best [B,maxT,maxU] holds max_{v != blank}(E[t,v]+P[u,v]); decBits is scratch of
// viterbi_decbits_words(d) 32-bit words.
size_t viterbi_decbits_words(Dims d);
void launch_viterbi_lattice(const float* E, const float* P, const float* LN,
                            const float* best, uint32_t* decBits, int* labels,
                            const int* inLens, const int* labLens, Dims d,
                            cudaStream_t stream);

// ---- lognorm_simt.cu ---------------------------------------------------------
// fp32 log-normalisers of every valid (t,u) on the SIMT pipes; rowRef[b,t] = max_v E[b,t,v] and
// maxP[b,u] likewise (0 for padded rows), each unless null.  exact: one logsumexp per node; else the
// factored sum (rowRef and maxP must not be null), with nodes whose sum left the fp32 range as NaN
// for the caller to have recomputed (lattice re-layouts, launch_lognorm_fixup) and counted in
// status[1].
void launch_lognorm_simt(const float* E, const float* P, float* LN, float* rowRef, float* maxP,
                         const int* inLens, const int* labLens, Dims d, bool exact, int* status,
                         cudaStream_t stream);
// Is the factored sum the faster of the two for these sizes?
bool lognorm_factored_pays(Dims d);
// expP[b,u,v] = exp(P[b,u,v]-maxP[b,u]) for u <= labLens[b], 0 for padded rows;
// also writes maxP[b,u] (0 for padded rows).
void launch_exp_rows(const float* P, float* expP, float* maxP, const int* labLens,
                     int B, int maxU, int V, cudaStream_t stream);

// ---- lognorm_umma.cu ----------------------------------------------------------
// Tensor-core log-normalisers (one pass over E; E and P of d.dtype, bf16 only for label axes of
// at most 128 positions).  Usable when lognorm_umma_supported();
// splitWs holds lognorm_umma_workspace_floats(d) floats; status is the device status word
// (api_internal.h): [0] first device-side error code (0 = none), [1] nodes recomputed exactly.
// pairs: the TF32 kernel, or lognorm_f16.cu with the TF32 kernel for the tiles that it marks, or that
// unless a sample of the scores says that most tiles would be marked.  lognorm_f16_pays: is the last
// the fastest for these sizes?
enum class PairFormat { tf32, f16, f16_if_close };
bool lognorm_f16_pays(Dims d);
bool lognorm_umma_supported(const void* E, const void* P, Dims d);
size_t lognorm_umma_workspace_floats(Dims d);
// Nodes whose factored sum left the fp32 range come out of the kernel as NaN; with `fixup` a
// second kernel recomputes them exactly, without it the caller must (lattice_prep does).
// With labels, EL [B,maxU,maxT] (frames contiguous) and ebl [B,maxT] (all three non-null) and
// lognorm_umma_gathers(d), the kernel also writes EL[b,u,t] = E[b,t,labels[b,u]] (u < U_b - 1)
// and ebl[b,t] = E[b,t,blank] for the valid frames, from the chunks it streams anyway.
// launch_lognorm_fixup: the recomputation, by itself.
void launch_lognorm_fixup(const void* E, const void* P, float* LN, const int* inLens,
                          const int* labLens, Dims d, cudaStream_t stream);
bool lognorm_umma_gathers(Dims d);
void launch_lognorm_umma(const void* E, const void* P, float* LN, float* rowRef, float* maxP,
                         const int* inLens, const int* labLens, Dims d, float* splitWs,
                         int* status, PairFormat pairs, bool fixup, cudaStream_t stream,
                         const int* labels = nullptr, float* EL = nullptr, float* ebl = nullptr);

// ---- lognorm_f16.cu ------------------------------------------------------------
// The workspace of launch_lognorm_umma, shared by both kernels.
struct LogNormScratch {
  float* operand;      // exp(P): fp16 pairs, or (TF32 kernel) two fp32 arrays
  float* partial;      // partial sums of split tiles
  float* rowSums;
  float* sumP;         // [B,maxU]
  unsigned* tickets;   // zero
  int* marks;          // zero; kMarkTiles + B * tiles
  int nSM;             // SMs of the device
};
// LN of every tile whose sums can be trusted; the others are marked (ws.marks) for the TF32 kernel.  sample:
// none at all, if a sample of the nodes says that most tiles would be.
void launch_lognorm_f16(const void* E, const void* P, float* LN, float* rowRef, float* maxP,
                        const int* inLens, const int* labLens, Dims d, const LogNormScratch& ws,
                        int* status, bool sample, cudaStream_t stream, const int* labels, float* EL, float* ebl);

// ---- grads_umma.cu --------------------------------------------------------------
// Tensor-core gradients: one pass over E produces egrads and pgrads.  Usable when
// grads_umma_supported(); passes = 1..3 selects the operand precision (see grads_umma.cu).
int grads_umma_ld_w(Dims d);  // row length of W: maxU rounded up to 32
int grads_umma_ld_t(Dims d);  // row length of nref / ebl / emT: maxT rounded up to 4
bool grads_umma_supported(const void* E, const void* P, const void* egrads,
                          const void* pgrads, Dims d, int passes);
// E, P, egrads and pgrads are of d.dtype (bf16: passes = 2 only, label axes up to 128; fp32:
// label axes up to 256 positions, long ones as two launches over parts of the axis).
// partial: scratch of grads_umma_partial_floats(d) floats; tickets: kGradTickets zeros, left zero.
constexpr int kGradTickets = 148;   // one per SM
size_t grads_umma_partial_floats(Dims d);
void launch_grads_umma(const void* E, const void* P, const float* maxP, const float* W,
                       const float* emT, const float* nref, const float* ebl, const float* pBlank,
                       const float* pLabel, const int* labels, const float* deltas, void* egrads,
                       void* pgrads, const int* inLens, const int* labLens, Dims d, int passes,
                       float* partial, unsigned* tickets, int* status, cudaStream_t stream);

// ---- lattice_sweep.cu ------------------------------------------------------------
// Sweeps for label axes of at most 256 positions (file comment there).  Lattices are skewed:
// node (t,u) of utterance b at b*stride + (t+u)*ld + u (pairs: permuted within the row).
bool sweep_supported(Dims d);
struct SweepGeom {
  int npl;      // adjacent label positions per lane of a sweep
  int ld;       // positions per anti-diagonal row, 32 * npl
  int nDiag;    // rows per utterance
  int nBlk;     // blocks of 16 rows: entries of `deltas` per utterance
  i64 stride;   // ld * nDiag
};
SweepGeom sweep_geom(Dims d);
// Arc terms (NaN entries of LN [B,maxT,maxU] -- nodes the tensor-core log-normaliser marked --
// are recomputed in place first, exactly), alphas, costs [B] (+inf for an empty utterance) and, if
// lossSum is not null, their sum in index order.  ELrow [B,maxU,maxT] and ebl [B,maxT]: label and
// blank emissions as written by launch_lognorm_umma, or both null, and they are gathered from E.
// E and P are of d.dtype.  ticket (with lossSum) and halves [B]: zeros.  For the backward call: arcs and
// alphas [B,stride], deltas [B,nBlk] and, for axes of more than 128 positions, ebl (written here where
// it is not an input).  score: no backward call will follow; alphas and deltas are scratch then.
void launch_sweep_forward(const void* E, const void* P, float* LN, const float* ELrow,
                          float* ebl, float2* arcs, float* alphas, float* deltas, float* costs,
                          float* lossSum, unsigned* ticket, unsigned* halves, const int* labels,
                          const int* inLens, const int* labLens, SweepGeom g, Dims d, bool score,
                          cudaStream_t stream);
struct SweepScratch {   // of the backward call
  float2* F;         // [B,stride]
  float* g;          // [B,stride]
  unsigned* ticket;  // [B]
  unsigned* gradTickets;  // [kGradTickets], zeroed for launch_grads_umma
  float* partial;    // sweep_partial_floats(d)
};
size_t sweep_partial_floats(Dims d);
// Reverse sweep, then the occupancies in the layout the gradient kernels read:
//   tensorCore: W [B,maxT,ldW] rounded to TF32, emT [B,maxU,ldT], ebl [B,ldT] (sums over u of the
//               blank-arc occupancies), nref [B,ldT] = -rowRef*log2(e); W, emT and ebl are scaled
//               by deltas[b] (1 if deltas is null).  Operands of launch_grads_umma.
//   otherwise:  W [B,maxT,ldW] unrounded and unscaled, label-arc occupancies [B,maxT,maxU] (passed
//               as emT), eBlank [B,maxT] (passed as ebl); nref and deltas unused.  Operands of the
//               SIMT gradient kernels.
//   both:       pBlank / pLabel [B,maxU], sums over t of the two occupancies, unscaled.
void launch_sweep_backward(const SweepScratch& w, const float* P, const float* blankEmissions,
                           const int* labels, const float2* arcs, const float* alphas,
                           const float* alphaDeltas, const float* LN, const float* rowRef,
                           const float* maxP, const float* deltas, float* W, float* emT, float* nref,
                           float* ebl, float* pBlank, float* pLabel, const int* inLens,
                           const int* labLens, SweepGeom g, Dims d, bool tensorCore,
                           cudaStream_t stream);

// ---- lattice_warp.cu -------------------------------------------------------------
// Viterbi sweep in one warp per utterance (label axis <= 256): same results as
// launch_viterbi_lattice.  scratch: viterbi_warp_scratch_floats(d) floats (8-byte aligned), decBits:
// viterbi_warp_decbits_words(d) words.  fix: NaN entries of LN are recomputed in place first (else LN is
// only read).
bool viterbi_warp_supported(Dims d);
size_t viterbi_warp_scratch_floats(Dims d);
size_t viterbi_warp_decbits_words(Dims d);  // its decision bits are packed along t+u
void launch_viterbi_warp(const float* E, const float* P, float* LN, bool fix, const float* best,
                         float* scratch, uint32_t* decBits, int* labels, const int* inLens,
                         const int* labLens, Dims d, cudaStream_t stream);

// ---- maxplus.cu --------------------------------------------------------------
// best[b,t,u] = max over v != blank of E[b,t,v] + P[b,u,v] for t < T_b, u < U_b - 1.  With
// `guard`, the kernel does nothing unless *guard > guardCap (read on the device).
void launch_maxplus(const float* E, const float* P, float* best, const int* inLens,
                    const int* labLens, Dims d, cudaStream_t stream, const int* guard = nullptr,
                    int guardCap = 0);

// ---- maxplus_pruned.cu -------------------------------------------------------
// The same result, bit for bit, from candidate lists with an exact bound; nodes the bound does
// not settle are evaluated densely.  `scratch` holds maxplus_pruned_scratch_bytes(d) bytes.
bool maxplus_pruned_supported(Dims d);
size_t maxplus_pruned_scratch_bytes(Dims d);
void launch_maxplus_pruned(const float* E, const float* P, float* best, const int* inLens,
                           const int* labLens, Dims d, void* scratch, int* status,
                           cudaStream_t stream);

// ---- grads_simt.cu -----------------------------------------------------------
// egrads[b,t,v] = delta_b*(exp(E-rowRef)*sum_u W[t,u]*expP[u,v] - [v==blank]*eBlank[t]),
// minus the label-arc terms delta_b*em[t,u] at v = label_u; zero for t >= T_b.
void launch_egrad_simt(const float* E, const float* rowRef, const float* W, int ldW,
                       const float* expP, const float* eBlank, const float* em,
                       const int* labels, const float* deltas, float* egrads,
                       const int* inLens, const int* labLens, Dims d,
                       cudaStream_t stream);
// pgrads[b,u,v] = delta_b*(expP*sum_t W[t,u]*exp(E[t,v]-rowRef[t]) - [v==blank]*pBlank[u]
//                          - [v==label_u]*pLabel[u]), zero for u >= U_b.
void launch_pgrad_simt(const float* E, const float* rowRef, const float* W, int ldW,
                       const float* expP, const float* pBlank, const float* pLabel,
                       const int* labels, const float* deltas, float* pgrads,
                       const int* inLens, const int* labLens, Dims d,
                       cudaStream_t stream);

}  // namespace tb200
