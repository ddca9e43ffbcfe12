// Viterbi sweep for label axes of at most 256 positions: the recursion runs in ONE warp.
//
// Lane l of the warp owns adjacent label positions; all nodes of a diagonal d = t + u are
// independent, the one value per lane that crosses from the neighbouring lane arrives by a warp
// shuffle, and the operands of a node, a pair, come by cp.async through the ring of pair_ring.cuh.
// (Not from both ends, as the costs alone: the scores are added in the reference's order.)
#include <algorithm>

#include "kernels.h"
#include "pair_ring.cuh"
#include "profile.h"
#include "sm100.cuh"

namespace tb200 {
namespace {

using namespace sm100;
using namespace sweep;

// ---------------------------------------------------------------------------
// Viterbi: max-plus sweep in one warp, bit-packed decisions, backtrack, label argmax
// ---------------------------------------------------------------------------
// Per node the sweep needs LN[t,u], best[t,u] (the max-plus label score of maxplus.cu) and E[t,blank].  The
// first two are a pair of the skewed rows written by viterbi_prep_kernel; the blank emissions are in shared
// memory, and a lane reads one of them per diagonal: position r + 1 meets a frame one diagonal after
// position r.  The scores are formed in the reference's operation order, ((score + E[t,blank]) +
// P[u,blank]) - LN and (score + best) - LN, so every comparison, and with it the path, is bit-identical
// to transducer_cpu.cpp:145-222.  Nodes outside the lattice hold the pair (1e30, 0): whatever
// enters them leaves as about -1e30, which loses every comparison against a real score, as does the
// label arc of the last position, whose best is -1e30.  With that the sweep needs no case distinctions
// at all: the blank arc into frame 0 and the label arc into position 0 come from such nodes
// (or from the -inf fed to lane 0) and lose by themselves.
constexpr float kNoNode = -1.0e30f;

struct VitPrepParams {
  const float* E;
  const float* P;
  float* LN;               // [B,maxT,maxU]
  bool fix;                // recompute its marked (NaN) nodes, in place
  const float* best;
  float2* nodes;
  float* ebl;              // [B,maxT]
  const int* inLens;
  const int* labLens;
  int maxT, maxU, V, blank, npl, extra;
  i64 stride;
};

// One CTA per 32x32 (t,u) tile; the tiles beyond both ends of the time axis (`extra` of them on each side)
// write the pairs of nodes outside the lattice, so that the array needs no fill.  Bound by memory: 8
// bytes read and 8 written per node.  (Records of 16 bytes, a fill of the array and a pass over LN for
// marked nodes before it took 126 us at B = 64, T = 750..1500, U' = 76..151, this takes 48; the sweep
// on those records 232 us, on pairs 166.)
__global__ void __launch_bounds__(256) viterbi_prep_kernel(const VitPrepParams p) {
  __shared__ float tLn[32][kTileLd], tBs[32][kTileLd];
  const int b = blockIdx.z, t0 = ((int)blockIdx.y - p.extra) * 32, u0 = blockIdx.x * 32;
  const int T = min(p.inLens[b], p.maxT), U = min(p.labLens[b] + 1, p.maxU);
  if (T <= 0 || U <= 0) return;
  const int Uw = (U + p.npl - 1) / p.npl * p.npl, S = T + U - 1;
  if (u0 >= Uw || t0 + u0 + 62 < 0 || t0 + u0 >= S) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, u = u0 + lane;
  if (t0 + 31 >= 0 && t0 < T && u0 < U) {   // does the tile hold any node?
    const float* e = p.E + (i64)b * p.maxT * p.V;
    const float* pr = p.P + (i64)b * p.maxU * p.V;
    float* ln = p.LN + (i64)b * p.maxT * p.maxU;
    const float* bs = p.best + (i64)b * p.maxT * p.maxU;
    const int uc = min(u, U - 1), ub = min(u, max(U - 2, 0));
    float va[4], vb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const i64 at = (i64)min(t0 + w * 4 + k, T - 1) * p.maxU;
      va[k] = ln[at + uc];
      vb[k] = bs[at + ub];
    }
    if (u0 == 0 && threadIdx.x < 32 && t0 + lane < T)
      p.ebl[(i64)b * p.maxT + t0 + lane] = e[(i64)(t0 + lane) * p.V + p.blank];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int tt = w * 4 + k, t = t0 + tt;
      unsigned todo = __ballot_sync(0xffffffffu, p.fix && t < T && u < U && va[k] != va[k]);
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const float exact = warp_logsumexp(e + (i64)t * p.V, pr + (i64)(u0 + src) * p.V, p.V, lane);
        if (lane == src) ln[(i64)t * p.maxU + u] = va[k] = exact;
      }
      tLn[tt][lane] = va[k];
      tBs[tt][lane] = u < U - 1 ? vb[k] : kNoNode;   // the label arc of the last position does not exist
    }
  }
  __syncthreads();
  float2* nodes = p.nodes + (i64)b * p.stride + pair_slot(u, p.npl);
#pragma unroll
  for (int k = 0; k < 4; ++k) {   // diagonal i of the tile in the lanes up to i, i + 32 in the others
    const int tt = (w + 8 * k - lane) & 31, t = t0 + tt, d = t + u;
    if (d < 0 || d >= S || u >= Uw) continue;
    nodes[(i64)d * (32 * p.npl)] =
        t >= 0 && t < T && u < U ? make_float2(tLn[tt][lane], tBs[tt][lane]) : make_float2(-kNoNode, 0.0f);
  }
}

// Decision bits of the single-warp sweep are packed along the DIAGONAL d = t + u: word
// [(b*maxU + u)*wordsD + d/32] bit (d%32) is 1 when node (t,u) was entered by the label arc
// from (t,u-1).  All positions then flush their words at the same steps.
__host__ __device__ inline int viterbi_words_d(int maxT, int maxU) { return (maxT + maxU + 31) / 32; }

// NPL label positions per lane: u = NPL*lane + r.  One warp per utterance sweeps, then its
// first thread backtracks and writes, for every label position, the frame at which the label was
// emitted (frames [B,maxU], -1 where there is none); viterbi_labels_kernel resolves the labels.
// The decision bits live in shared memory behind the ring where they fit (decInSmem), in the
// decBits scratch otherwise: the backtrack is a chain of dependent reads of them.
template <int NPL>
__global__ void __launch_bounds__(32) viterbi_warp_kernel(
    const float* __restrict__ P, const float2* __restrict__ nodes, const float* __restrict__ ebl,
    i64 stride, int maxStage, uint32_t* __restrict__ decBits, int decInSmem,
    int* __restrict__ frames, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int maxT, int maxU, int V, int blank) {
  constexpr int ld = 32 * NPL, kRing = ring_blocks(NPL);
  extern __shared__ __align__(128) uint8_t smemV[];
  __shared__ int sFrame[256];  // frame at which label u-1 was emitted (U <= 256 here)
  const int b = blockIdx.x, i = threadIdx.x, lane = i;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  int* fr = frames + (i64)b * maxU;
  if (T <= 0 || U <= 0) {
    for (int u = i; u < maxU; u += 32) fr[u] = -1;
    return;
  }
  const float* p = P + (i64)b * maxU * V;
  const int wordsD = viterbi_words_d(maxT, maxU);
  // shared memory: ring, blank emissions (of utterances of up to maxStage frames), decision bits
  float* sEb = reinterpret_cast<float*>(smemV + kRing * kDiag * ld * 8);
  uint32_t* dec = decInSmem ? reinterpret_cast<uint32_t*>(sEb + maxStage)
                            : decBits + (i64)b * maxU * wordsD;
  for (int u = i; u < 256; u += 32) sFrame[u] = -1;
  const int S = T + U - 1, nBlocks = (S + kDiag - 1) / kDiag, u0 = NPL * lane;
  PairRing<NPL> ring(smemV, nodes + (i64)b * stride, lane, U, 0x7149f2cau /* 1e30 */, 0u);
  auto issue = [&](int k) { ring.issue(k % kRing, (i64)k * kDiag, k < nBlocks ? min(kDiag, S - k * kDiag) : 0); };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  const float* eb0 = ebl + (i64)b * maxT;
  const bool staged = T <= maxStage;
  if (staged) {
#pragma unroll 8
    for (int t = lane; t < T; t += 32) sEb[t] = eb0[t];
  }
  __syncwarp();
  const float* ebRow = staged ? sEb : eb0;
  auto eblAt = [&](int t) { return ebRow[min(max(t, 0), T - 1)]; };
  float pbl[NPL], eb[NPL], stay[NPL], stepOut[NPL];
  uint32_t bits[NPL];
#pragma unroll
  for (int r = 0; r < NPL; ++r) {
    pbl[r] = (u0 + r < U) ? p[(i64)(u0 + r) * V + blank] : 0.0f;
    eb[r] = eblAt(-(u0 + r));
    stay[r] = stepOut[r] = kNoNode;
    bits[r] = 0u;
  }
  if (lane == 0) stay[0] = 0.0f;  // score 0 enters the origin (as if by its blank arc)
  float up = neg_inf();
  for (int k = 0; k < nBlocks; ++k) {
    issue(k + kRing - 1);
    ring.wait();
    const int slot = k % kRing, nd = min(kDiag, S - k * kDiag);
    const int tNext = k * kDiag + 1 - u0;   // frame of position u0 on the diagonal after the block's first
    const uint32_t bit0 = 1u << (kDiag * (k & 1));
    auto diag = [&](int dd) {
      float ln[NPL], bs[NPL];
      ring.read(slot, dd, ln, bs);
      const float ebNext = eblAt(tNext + dd), first = lane ? up : neg_inf();
      // the last position first, whose step leaves by a shuffle; each position still needs the
      // previous diagonal's step of the one below it
#pragma unroll
      for (int r = NPL - 1; r >= 0; --r) {
        const float left = r ? stepOut[(r + NPL - 1) % NPL] : first;
        // the larger of the two arcs, the blank arc on ties (strict '>', as the reference)
        const bool takeStep = left > stay[r];
        const float sc = takeStep ? left : stay[r];
        if (takeStep) bits[r] |= bit0 << dd;
        stay[r] = ((sc + eb[r]) + pbl[r]) - ln[r];
        stepOut[r] = (sc + bs[r]) - ln[r];
        if (r == NPL - 1) up = __shfl_up_sync(0xffffffffu, stepOut[r], 1);
      }
#pragma unroll
      for (int r = NPL - 1; r > 0; --r) eb[r] = eb[r - 1];
      eb[0] = ebNext;
    };
    if (nd == kDiag) {
#pragma unroll
      for (int dd = 0; dd < kDiag; ++dd) diag(dd);
    } else {
#pragma unroll 1
      for (int dd = 0; dd < nd; ++dd) diag(dd);
    }
    if ((k & 1) || k == nBlocks - 1) {   // a word of 32 diagonals is complete
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        if (u0 + r < U) dec[(i64)(u0 + r) * wordsD + (k >> 1)] = bits[r];
        bits[r] = 0u;
      }
    }
  }
  ring.drain();
  __threadfence_block();
  __syncthreads();

  // Backtrack from (T-1,U-1) along row u in diagonal coordinates d = t + u.  Each iteration
  // consumes either one label or one 32-diagonal word of blanks, so it ends within
  // U + (T+U)/32 + 1 iterations; the explicit cap only guards against corrupted scratch.
  // (Node (0,u), u > 0, is always entered by its label arc, so the scan of a row never runs
  // into the bits of nodes before frame 0.)
  if (i == 0) {
    int t = T - 1, u = U - 1;
    int guard = U + wordsD + 2;
    while (u > 0 && t >= 0 && guard-- > 0) {
      const int d = t + u;
      const uint32_t keep = 0xffffffffu >> (31 - (d & 31));
      const uint32_t w = ((volatile uint32_t*)dec)[(i64)u * wordsD + (d >> 5)] & keep;
      if (w == 0u) { t = (d & ~31) - 1 - u; continue; }
      t = (d & ~31) + (31 - __clz(w)) - u;
      sFrame[u] = t;
      --u;
    }
  }
  __syncthreads();
  for (int u = i; u < maxU; u += 32) fr[u] = (u < U) ? sFrame[u] : -1;
}

// Label on each emitting arc of the path: lowest-index argmax over v != blank of
// E[t,v] + P[u-1,v] (strict '>' in index order, as the reference's getMax,
// transducer_cpu.cpp:156-169), one warp per label position, t = frames[b,u].
__global__ void __launch_bounds__(256) viterbi_labels_kernel(
    const float* __restrict__ E, const float* __restrict__ P, const int* __restrict__ frames,
    int* __restrict__ labelsOut, const int* __restrict__ labLens, int B, int maxT, int maxU,
    int V, int blank) {
  const int lane = threadIdx.x & 31;
  const int u = 1 + blockIdx.x * 8 + (threadIdx.x >> 5);
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
  if (u >= min(labLens[b] + 1, maxU)) continue;
  const int t = frames[(i64)b * maxU + u];
  if (t < 0) continue;
  const float* er = E + ((i64)b * maxT + t) * V;
  const float* pr = P + ((i64)b * maxU + u - 1) * V;
  const bool vec4 = (V & 3) == 0 && ((reinterpret_cast<uintptr_t>(er) | reinterpret_cast<uintptr_t>(pr)) & 15) == 0;
  float m = neg_inf();
  int arg = 0x7fffffff;
  if (vec4) {  // 16 loads in flight per lane; each lane still visits its entries in index order
    const float4* e4 = reinterpret_cast<const float4*>(er);
    const float4* p4 = reinterpret_cast<const float4*>(pr);
    const int n4 = V >> 2;
    for (int q0 = lane; q0 < n4; q0 += 128) {
      float4 a[4], c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int q = min(q0 + 32 * j, n4 - 1);
        a[j] = e4[q];
        c[j] = p4[q];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int q = q0 + 32 * j;
        if (q < n4) {
          const float x[4] = {a[j].x + c[j].x, a[j].y + c[j].y, a[j].z + c[j].z, a[j].w + c[j].w};
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int v = 4 * q + h;
            if (v != blank && x[h] > m) { m = x[h]; arg = v; }
          }
        }
      }
    }
  } else {
    for (int v = lane; v < V; v += 32) {
      if (v == blank) continue;
      const float x = er[v] + pr[v];
      if (x > m) { m = x; arg = v; }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const int a2 = __shfl_xor_sync(0xffffffffu, arg, o);
    if (m2 > m || (m2 == m && a2 < arg)) { m = m2; arg = a2; }
  }
  if (lane == 0) labelsOut[(i64)b * (maxU - 1) + u - 1] = (arg == 0x7fffffff) ? 0 : arg;
  }
}

}  // namespace

bool viterbi_warp_supported(Dims d) { return d.maxU >= 1 && d.maxU <= 256; }

size_t viterbi_warp_decbits_words(Dims d) {
  // decision bits, then the frames at which the labels are emitted [B,maxU]
  return viterbi_warp_supported(d)
             ? (size_t)d.B * (size_t)d.maxU * (size_t)(viterbi_words_d(d.maxT, d.maxU) + 1)
             : 0;
}

// Rows of pairs: positions per lane (up to 8) and length of an utterance.
static int viterbi_npl(Dims d) { return div_up(std::max(d.maxU, 1), 32); }
static i64 viterbi_stride(Dims d) { return (i64)32 * viterbi_npl(d) * (d.maxT + d.maxU); }

size_t viterbi_warp_scratch_floats(Dims d) {
  return viterbi_warp_supported(d) ? (size_t)d.B * (2 * (size_t)viterbi_stride(d) + (size_t)d.maxT) : 0;
}

void launch_viterbi_warp(const float* E, const float* P, float* LN, bool fix, const float* best,
                         float* scratch, uint32_t* decBits, int* labels, const int* inLens,
                         const int* labLens, Dims d, cudaStream_t stream) {
  if (d.B <= 0 || d.maxT <= 0 || d.maxU <= 0) return;
  const int npl = viterbi_npl(d), ld = 32 * npl;
  const i64 stride = viterbi_stride(d);
  float2* nodes = reinterpret_cast<float2*>(scratch);
  float* ebl = scratch + 2 * (size_t)d.B * stride;
  {
    VitPrepParams q{};
    q.E = E; q.P = P; q.LN = LN; q.fix = fix; q.best = best; q.nodes = nodes; q.ebl = ebl;
    q.inLens = inLens; q.labLens = labLens;
    q.maxT = d.maxT; q.maxU = d.maxU; q.V = d.V; q.blank = d.blank; q.npl = npl;
    q.extra = div_up(d.maxU, 32); q.stride = stride;
    dim3 grid(div_up(d.maxU, 32), div_up(d.maxT, 32) + 2 * q.extra, d.B);
    ScopedKernel sk("viterbi_prep", stream);
    viterbi_prep_kernel<<<grid, 256, 0, stream>>>(q);
    TB200_CHECK_LAUNCH();
  }
  // shared memory: the ring, the blank emissions and the decision bits where they fit
  constexpr int room = 216 * 1024;
  const int ringBytes = ring_blocks(npl) * kDiag * ld * 8;
  const int stage = std::min(d.maxT, (room - ringBytes) / 4);
  const i64 decBytes = (i64)d.maxU * viterbi_words_d(d.maxT, d.maxU) * 4;
  const int decInSmem = ringBytes + stage * 4 + decBytes <= room ? 1 : 0;
  const int smem = ringBytes + stage * 4 + (decInSmem ? (int)decBytes : 0);
  int* frames = reinterpret_cast<int*>(decBits) +
                (size_t)d.B * d.maxU * viterbi_words_d(d.maxT, d.maxU);
  {
  ScopedKernel sk("viterbi_warp", stream);
#define CALL(NPL)                                                                              \
  do {                                                                                         \
    allow_dyn_smem(viterbi_warp_kernel<NPL>, room);                                            \
    viterbi_warp_kernel<NPL><<<d.B, 32, smem, stream>>>(                                       \
        P, nodes, ebl, stride, stage, decBits, decInSmem, frames, inLens, labLens, d.maxT,     \
        d.maxU, d.V, d.blank);                                                                 \
  } while (0)
  switch (npl) {
    case 1: CALL(1); break;
    case 2: CALL(2); break;
    case 3: CALL(3); break;
    case 4: CALL(4); break;
    case 5: CALL(5); break;
    case 6: CALL(6); break;
    case 7: CALL(7); break;
    default: CALL(8); break;
  }
#undef CALL
  }
  TB200_CHECK_LAUNCH();
  if (d.maxU > 1) {
    ScopedKernel sk("viterbi_labels", stream);
    viterbi_labels_kernel<<<dim3(div_up(d.maxU - 1, 8), std::min(d.B, 65535)), 256, 0, stream>>>(
        E, P, frames, labels, labLens, d.B, d.maxT, d.maxU, d.V, d.blank);
    TB200_CHECK_LAUNCH();
  }
}

}  // namespace tb200
