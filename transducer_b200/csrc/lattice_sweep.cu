// Lattice sweeps for label axes of at most 256 positions: each recursion runs in ONE warp per
// utterance, and everything that does not depend on the recursion in kernels of its own that use
// the whole GPU.
//
//   sweep_prep       arc log-probabilities of every node (log2 units), skewed
//   alpha_sweep      alpha recursion                                          (forward call)
//   score_sweep      costs alone: alpha and beta recursions up to the middle  (score call)
//   gamma_factors    2^(alpha + arc - alpha') of every arc                    (backward call)
//   gamma_sweep      occupancy recursion: two products and a sum per node
//   occupancy        the operands of the gradient kernels
//
//   alpha   transducer/transducer_cpu.cpp:30-79   (transducer_cuda.cu:32-97)
//   reverse transducer/transducer_cpu.cpp:81-143  (transducer_cuda.cu:99-176)
//
// Axes of up to 128 positions run on rebased base-2 logarithms (alpha_sweep_kernel); longer ones
// (NPL >= 5, "natural" below) on natural logarithms at full magnitude, in the operation order of the
// block-wide kernels of lattice.cu (costs bit-identical to theirs: 18 shapes, T = 77..5000,
// U' = 129..256).
//
// Diagonal d = t + u of an utterance is one row of ld = 32 NPL numbers; lane l of a sweep owns the
// NPL adjacent positions u = NPL l + r.  All nodes of a diagonal are independent; the one value
// per lane that crosses from the neighbouring lane arrives by a warp shuffle.  A sweep is a chain
// of T + U - 1 dependent diagonals whatever the batch, so what counts is how few instructions a
// diagonal takes: operands are brought to shared memory by cp.async, each lane copying just the
// 8 NPL bytes a row that it reads itself (no barrier, no other warp), several blocks of 16
// diagonals ahead, and the loop holds nothing but the recursion and its store.
// Measured (T = 2000, U' = 101, device time, B = 8 / 32): alpha 132 us (147 with bulk copies issued and
// waited for by the sweeping warp); reverse sweep 12 / 27 us for the factors + 60 us for the recursion
// (152 us when helper warps of the same CTA prepared the factors and carried away the results).
// B = 64, T = 750..1500, U' = 151: alpha 195 us, factors 69 + recursion 76 us, operands 105 us, against
// 384, 512 and (lattices re-laid out twice) 168 us of the block-wide kernels, which take a barrier
// per diagonal.  B = 8, T = 4000, U' = 251: alpha 855 us, block-wide 954.
//
// COSTS ALONE.  Every path crosses each of the S = T + U - 1 diagonals once, so with alpha (all paths to a
// node) up to the middle diagonal M and beta (all paths from a node) down to it, the total is the sum
// over M of alpha beta.  The two halves are two warps that know nothing of each other, both chains are
// half as long, nothing but their ends is stored, and every label axis runs on rebased logarithms.  B = 64,
// T = 500..1000, U' = 101..201: 242 -> 64 us.
// With gradients to follow each recursion keeps to one warp from one end.  The weights W of the gradient
// products are rounded to TF32 behind the sweeps, and any other order of operations in front of that
// rounding flips some of them by one step, 2^-10 of a weight near one.  Where a blank is nearly certain
// its gradient is the small difference of two occupancies, and the flip shows: blank emissions raised by 4,
// entries differed by up to 3.3e-2 of the larger of themselves and the rms (4.74e-5 at B = 20, where
// 2^-10 / B is 4.88e-5), while the whole gradient differed by 3e-5 to 1e-4.  (Both sweeps took 113 us
// instead of 192 us so, at T = 2000, U' = 101.)
#include <algorithm>

#include "kernels.h"
#include "pair_ring.cuh"
#include "profile.h"
#include "sm100.cuh"

namespace tb200 {
namespace {

using namespace sm100;
using namespace sweep;

// The diagonal at which the halves of an utterance of S >= 1 diagonals meet: a whole number of blocks, so
// that the blocks of the first half are full.
__device__ __forceinline__ int middle(int S) { return (S / 2) & ~(kDiag - 1); }
constexpr float kLn2F = 0.6931471805599453f;
constexpr float kLog2e = 1.4426950408889634f;
// "No such arc": a large negative finite number (-5.97e29), the identity of the alpha recursion without -inf
// arithmetic, so that the sweeps need no validity logic.  An exponent below kNoPath means that every path
// has such an arc: the cost is +inf.
constexpr unsigned kNoArcBits = 0xF0F0F0F0u;
constexpr float kNoPath = -5.5e29f;

// A log-probability as an arc term: a word masked by -inf makes no arc (two of them into a node would make
// NaN of their difference); NaN stays NaN.
__device__ __forceinline__ float arc_term(float x) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(x), "f"(__uint_as_float(kNoArcBits)));
  return y;
}

// -inf becomes the lowest number; NaN stays NaN.
__device__ __forceinline__ float not_below_lowest(float x) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(x), "f"(-3.402823466e38f));
  return y;
}

__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A lane's numbers of a row (row points at its beginning).
template <int NPL>
__device__ __forceinline__ void store_row(float* row, int lane, const float (&a)[NPL]) {
  float* q = row + NPL * lane;
  if constexpr (NPL == 4) *reinterpret_cast<float4*>(q) = make_float4(a[0], a[1], a[2], a[3]);
  else if constexpr (NPL == 2) *reinterpret_cast<float2*>(q) = make_float2(a[0], a[1]);
  else {
#pragma unroll
    for (int r = 0; r < NPL; ++r) row[r * 32 + lane] = a[r];
  }
}
template <int NPL>
__device__ __forceinline__ void load_row(const float* row, int lane, float (&a)[NPL]) {
  const float* q = row + NPL * lane;
  if constexpr (NPL == 4) {
    const float4 f = *reinterpret_cast<const float4*>(q);
    a[0] = f.x; a[1] = f.y; a[2] = f.z; a[3] = f.w;
  } else if constexpr (NPL == 2) {
    const float2 f = *reinterpret_cast<const float2*>(q);
    a[0] = f.x; a[1] = f.y;
  } else {
#pragma unroll
    for (int r = 0; r < NPL; ++r) a[r] = row[r * 32 + lane];
  }
}

__device__ __forceinline__ void finish_cost(float* costs, int b, float cost, int B, float* lossSum,
                                            unsigned* ticket) {
  costs[b] = cost;
  if (lossSum == nullptr) return;
  __threadfence();
  const unsigned done = atomicAdd(ticket, 1u);
  if (done == (unsigned)(B - 1)) {  // last utterance: add the costs in index order
    __threadfence();
    float s = 0.0f;
    for (int k = 0; k < B; ++k) s += ((volatile float*)costs)[k];
    *lossSum = s;
    *ticket = 0u;
  }
}

// ---------------------------------------------------------------------------
// alpha
// ---------------------------------------------------------------------------
// The recursion runs in log2 units,
//   a(t,u) = log2( 2^(a(t-1,u) + blank arc) + 2^(a(t,u-1) + label arc) ),
// so that the two transcendental steps are the bare ex2 / lg2 instructions, and the alphas are
// stored in log2 units too: the reverse sweep must form a(t,u) + arc with the very same
// rounding as here, or the occupancies stop being a conserved flow.
//
// REBASED alphas.  After 2000 frames an alpha is of magnitude 1e4 and an fp32 ulp there is
// 1e-3: the reference carries its alphas at that magnitude (transducer_cpu.cpp:30-79) and its
// gradients are 2e-3..6e-3 of their maximum away from a float64 evaluation for it (measured).
// Here every block of 16 diagonals stores its alphas relative to an offset of its own: at the
// start of block k the whole carried state is lowered by delta_k = the floor of its largest
// entry (an integer, so that the running offset -- needed only for the final cost -- adds up
// exactly).  As delta_k is taken one block early, a stored number that matters lies at most 32
// arcs below its offset: a few hundred for N(0,1..2) scores (ulp 3e-5), 4600 for arcs of
// 100 nats; nothing else bounds it.  delta_k is written to `deltas` for the reverse sweep, which
// subtracts it at the same point of the same sum.  The loss and the gradients then sit ~1e-4 from
// the float64 result.
//
// The pace is set by the special-function unit: NPL ex2 and NPL lg2 per diagonal, 8 issue cycles
// each, in a chain.  (Cutting the label axis over two or four warps that run a block apart was
// measured and is slower: every node then waits for a shuffle.)
template <int NPL>
__global__ void __launch_bounds__(32) alpha_sweep_kernel(
    const float2* __restrict__ arcs, float* __restrict__ costs, float* __restrict__ alphas,
    float* __restrict__ deltas, i64 stride, int nDiag, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int B, int maxT, int maxU, float* lossSum, unsigned* ticket) {
  constexpr int ld = 32 * NPL;
  extern __shared__ __align__(128) uint8_t smemA[];
  const int b = blockIdx.x, lane = threadIdx.x;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (T <= 0 || U <= 0) {
    if (lane == 0) finish_cost(costs, b, pos_inf(), B, lossSum, ticket);
    return;
  }
  const int S = T + U - 1, nBlocks = (S + kDiag - 1) / kDiag, u0 = NPL * lane;
  constexpr int kRing = ring_blocks(NPL);
  PairRing<NPL> ring(smemA, arcs + (i64)b * stride, lane, U, kNoArcBits, kNoArcBits);
  auto issue = [&](int k) { ring.issue(k % kRing, (i64)k * kDiag, k < nBlocks ? min(kDiag, S - k * kDiag) : 0); };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  float* al = alphas + (i64)b * stride;
  float* dl = deltas + (i64)b * ((nDiag + kDiag - 1) / kDiag);
  const float kNone = __uint_as_float(kNoArcBits);
  float stayIn[NPL], stepOut[NPL];
#pragma unroll
  for (int r = 0; r < NPL; ++r) stayIn[r] = stepOut[r] = kNone;
  if (lane == 0) stayIn[0] = 0.0f;  // alpha(0,0) = 0
  float up = kNone;        // stepOut of the lane below's last position, one diagonal back
  float offset = 0.0f;     // sum of the deltas so far: an integer, exact in fp32
  float nextDelta = 0.0f;  // by how much the state is lowered at the start of the next block
  for (int k = 0; k < nBlocks; ++k) {
    issue(k + kRing - 1);
    if (k > 0) {
      // rebase (entries of nodes outside the lattice are ~ -6e29 and stay there)
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        stayIn[r] -= nextDelta;
        stepOut[r] -= nextDelta;
      }
      up -= nextDelta;
      offset += nextDelta;
      if (lane == 0) dl[k] = nextDelta;
    }
    // The delta applied at the start of the NEXT block is the floor of the largest entry of
    // the state now, at the start of this one: the warp-wide maximum then has a whole block to
    // arrive, off the dependent chain.  (By then the state has sunk by another 16 arcs.)
    {
      float m = kNone;
#pragma unroll
      for (int r = 0; r < NPL; ++r) m = fmaxf(m, fmaxf(stayIn[r], stepOut[r]));
      nextDelta = (float)__reduce_max_sync(0xffffffffu, __float2int_rd(fmaxf(m, -1.0e9f)));
    }
    ring.wait();
    const int slot = k % kRing, nd = min(kDiag, S - k * kDiag);
    float* out = al + (i64)k * kDiag * ld;
    auto diag = [&](int i) {
      float fx[NPL], fy[NPL], left[NPL], m[NPL], e[NPL], a[NPL];
      ring.read(slot, i, fx, fy);
      // The last position first: its result feeds the shuffle of the next diagonal; position 0
      // last: it waits for the shuffle of this one.  (A warp issues in order.)
      left[0] = lane ? up : kNone;
#pragma unroll
      for (int r = 1; r < NPL; ++r) left[r] = stepOut[r - 1];
#pragma unroll
      for (int r = NPL - 1; r >= 0; --r) {
        m[r] = fmaxf(left[r], stayIn[r]);
        e[r] = ex2_approx(-fabsf(left[r] - stayIn[r]));
      }
#pragma unroll
      for (int r = NPL - 1; r >= 0; --r) {
        a[r] = m[r] + lg2_approx(1.0f + e[r]);
        stayIn[r] = a[r] + fx[r];
        stepOut[r] = a[r] + fy[r];
        if (r == NPL - 1) up = __shfl_up_sync(0xffffffffu, stepOut[NPL - 1], 1);
      }
      if (ring.act) store_row<NPL>(out + i * ld, lane, a);
    };
    if (nd == kDiag) {
#pragma unroll
      for (int i = 0; i < kDiag; ++i) diag(i);
    } else {
#pragma unroll 1
      for (int i = 0; i < nd; ++i) diag(i);
    }
  }
  ring.drain();
  // the last diagonal holds only the terminal node (T-1, U-1); its blank arc ends the path
#pragma unroll
  for (int r = 0; r < NPL; ++r)
    if (u0 + r == U - 1)
      finish_cost(costs, b, stayIn[r] < kNoPath ? pos_inf() : -(stayIn[r] + offset) * kLn2F, B, lossSum, ticket);
}

// ---------------------------------------------------------------------------
// costs alone
// ---------------------------------------------------------------------------
// (rebased like alpha_sweep_kernel; the betas in blocks of 16 from the end)
__device__ __forceinline__ float lse2_log2(float a, float b) {
  return fmaxf(a, b) + lg2_approx(1.0f + ex2_approx(-fabsf(a - b)));
}

// floor of the largest of a lane's numbers over the warp, at least -1e9: the next delta
__device__ __forceinline__ float next_delta(float m) {
  return (float)__reduce_max_sync(0xffffffffu, __float2int_rd(fmaxf(m, -1.0e9f)));
}

// alpha of the middle diagonal M into `row`; returns its offset
template <int NPL>
__device__ __forceinline__ float alpha_half(uint8_t* smem, const float2* arcs, float* row, int lane, int U, int M) {
  constexpr int kRing = ring_blocks(NPL);
  const int nBlocks = M / kDiag;
  PairRing<NPL> ring(smem, arcs, lane, U, kNoArcBits, kNoArcBits);
  auto issue = [&](int k) { ring.issue(k % kRing, (i64)k * kDiag, k < nBlocks ? kDiag : 0); };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  const float kNone = __uint_as_float(kNoArcBits);
  float stayIn[NPL], stepOut[NPL];
#pragma unroll
  for (int r = 0; r < NPL; ++r) stayIn[r] = stepOut[r] = kNone;
  if (lane == 0) stayIn[0] = 0.0f;  // alpha(0,0) = 0
  float up = kNone;        // stepOut of the lane below's last position, one diagonal back
  float offset = 0.0f;     // sum of the deltas so far: an integer, exact in fp32
  float nextDelta = 0.0f;  // by how much the state is lowered at the start of the next block
  for (int k = 0; k <= nBlocks; ++k) {
    issue(k + kRing - 1);
    if (k > 0) {
      // rebase (entries of nodes outside the lattice are ~ -6e29 and stay there)
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        stayIn[r] -= nextDelta;
        stepOut[r] -= nextDelta;
      }
      up -= nextDelta;
      offset += nextDelta;
    }
    if (k == nBlocks) {   // the middle diagonal: nothing leaves it here
      float a[NPL];
#pragma unroll
      for (int r = 0; r < NPL; ++r) a[r] = lse2_log2(r ? stepOut[(r + NPL - 1) % NPL] : lane ? up : kNone, stayIn[r]);
      if (ring.act) store_row<NPL>(row, lane, a);
      break;
    }
    // The delta applied at the start of the NEXT block is the floor of the largest entry of
    // the state now, at the start of this one: the warp-wide maximum then has a whole block to
    // arrive, off the dependent chain.  (By then the state has sunk by another 16 arcs.)
    {
      float m = kNone;
#pragma unroll
      for (int r = 0; r < NPL; ++r) m = fmaxf(m, fmaxf(stayIn[r], stepOut[r]));
      nextDelta = next_delta(m);
    }
    ring.wait();
    const int slot = k % kRing;
#pragma unroll
    for (int i = 0; i < kDiag; ++i) {
      float fx[NPL], fy[NPL], left[NPL], m[NPL], e[NPL], a[NPL];
      ring.read(slot, i, fx, fy);
      // The last position first: its result feeds the shuffle of the next diagonal; position 0
      // last: it waits for the shuffle of this one.  (A warp issues in order.)
      left[0] = lane ? up : kNone;
#pragma unroll
      for (int r = 1; r < NPL; ++r) left[r] = stepOut[r - 1];
#pragma unroll
      for (int r = NPL - 1; r >= 0; --r) {
        m[r] = fmaxf(left[r], stayIn[r]);
        e[r] = ex2_approx(-fabsf(left[r] - stayIn[r]));
      }
#pragma unroll
      for (int r = NPL - 1; r >= 0; --r) {
        a[r] = m[r] + lg2_approx(1.0f + e[r]);
        stayIn[r] = a[r] + fx[r];
        stepOut[r] = a[r] + fy[r];
        if (r == NPL - 1) up = __shfl_up_sync(0xffffffffu, stepOut[NPL - 1], 1);
      }
    }
  }
  ring.drain();
  return offset;
}

// beta of the middle diagonal into `row`, from the end; returns its offset
template <int NPL>
__device__ __forceinline__ float beta_half(uint8_t* smem, const float2* arcs, float* row, int lane, int U, int S,
                                           int M) {
  constexpr int kRing = ring_blocks(NPL);
  const int nBlocks = (S - M + kDiag - 1) / kDiag, u0 = NPL * lane;
  PairRing<NPL> ring(smem, arcs, lane, U, kNoArcBits, kNoArcBits);
  // block k holds the rows [max(S - 16(k+1), M), S - 16k)
  auto issue = [&](int k) {
    const int lo = max(S - kDiag * (k + 1), M);
    ring.issue(k % kRing, lo, k < nBlocks ? S - kDiag * k - lo : 0);
  };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  const float kNone = __uint_as_float(kNoArcBits);
  float bt[NPL];   // of the diagonal above; at first of the node beyond the terminating blank
#pragma unroll
  for (int r = 0; r < NPL; ++r) bt[r] = u0 + r == U - 1 ? 0.0f : kNone;
  // (lane 31 gets its own back: harmless, the label arc of its last position never exists)
  float right = __shfl_down_sync(0xffffffffu, bt[0], 1);
  float offset = 0.0f, nextDelta = 0.0f;
  for (int k = 0; k < nBlocks; ++k) {
    issue(k + kRing - 1);
    if (k > 0) {
#pragma unroll
      for (int r = 0; r < NPL; ++r) bt[r] -= nextDelta;
      right -= nextDelta;
      offset += nextDelta;
    }
    {
      float m = kNone;
#pragma unroll
      for (int r = 0; r < NPL; ++r) m = fmaxf(m, bt[r]);
      nextDelta = next_delta(m);
    }
    ring.wait();
    const int slot = k % kRing, lo = max(S - kDiag * (k + 1), M), nd = S - kDiag * k - lo;
    auto diag = [&](int i) {
      float x[NPL], y[NPL], m[NPL], e[NPL];
      ring.read(slot, i, x, y);
      // position 0 first, whose result leaves by the shuffle; the last one waits for it
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        const float p = bt[r] + x[r], q = (r < NPL - 1 ? bt[(r + 1) % NPL] : right) + y[r];
        m[r] = fmaxf(p, q);
        e[r] = ex2_approx(-fabsf(p - q));
      }
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        bt[r] = m[r] + lg2_approx(1.0f + e[r]);
        if (r == 0) right = __shfl_down_sync(0xffffffffu, bt[0], 1);
      }
    };
    if (nd == kDiag) {
#pragma unroll
      for (int i = kDiag - 1; i >= 0; --i) diag(i);
    } else {
#pragma unroll 1
      for (int i = nd - 1; i >= 0; --i) diag(i);
    }
  }
  ring.drain();
  if (ring.act) store_row<NPL>(row, lane, bt);
  return offset;
}

// Of a lane's nodes of the middle diagonal: 2^(alpha + beta - m), m the largest exponent of the warp, into
// w; returns m, and the warp's sum of w in `total`.  No path at all (m < kNoPath): total = 0, w = 0.
template <int NPL>
__device__ __forceinline__ float meet(const float* al, const float* be, int lane, int U, float (&w)[NPL], float& total) {
  float m = -INFINITY;
#pragma unroll
  for (int r = 0; r < NPL; ++r) {
    const int u = NPL * lane + r, at = row_slot(min(u, U - 1), NPL);
    w[r] = u < U ? __ldcg(al + at) + __ldcg(be + at) : -INFINITY;
    m = fmaxf(m, w[r]);
  }
  m = warp_max(m);
  float s = 0.0f;
#pragma unroll
  for (int r = 0; r < NPL; ++r) {
    const bool nan = w[r] != w[r];
    w[r] = m >= kNoPath || nan ? exp2f(w[r] - m) : 0.0f;
    s += w[r];
  }
  total = warp_sum(s);
  return m;
}

// One warp per half of an utterance (blockIdx.y); the half that finishes last adds up the cost.
// ends [B, 2, 32 NPL] and offsets [B, 2]: scratch; halves [B]: zeros.
template <int NPL>
__global__ void __launch_bounds__(32) score_sweep_kernel(
    const float2* __restrict__ arcs, float* __restrict__ costs, float* ends, float* offsets, i64 stride,
    const int* __restrict__ inLens, const int* __restrict__ labLens, int B, int maxT, int maxU,
    float* lossSum, unsigned* ticket, unsigned* halves) {
  extern __shared__ __align__(128) uint8_t smemA[];
  const int b = blockIdx.x, lane = threadIdx.x;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (T <= 0 || U <= 0) {
    if (lane == 0 && blockIdx.y == 0) finish_cost(costs, b, pos_inf(), B, lossSum, ticket);
    return;
  }
  const int S = T + U - 1, M = middle(S);
  float* al = ends + (i64)b * 64 * NPL;
  float* be = al + 32 * NPL;
  const float offset = blockIdx.y == 0 ? alpha_half<NPL>(smemA, arcs + (i64)b * stride, al, lane, U, M)
                                       : beta_half<NPL>(smemA, arcs + (i64)b * stride, be, lane, U, S, M);
  if (lane == 0) offsets[2 * b + blockIdx.y] = offset;
  __threadfence();
  __syncwarp();
  unsigned before = 0;
  if (lane == 0) before = atomicAdd(&halves[b], 1u);
  if (__shfl_sync(0xffffffffu, before, 0) == 0u) return;
  __threadfence();
  float w[NPL], total;
  const float m = meet<NPL>(al, be, lane, U, w, total);
  if (lane == 0) {
    const double log2p = (double)__ldcg(offsets + 2 * b) + (double)__ldcg(offsets + 2 * b + 1) + (double)(m + log2f(total));
    finish_cost(costs, b, total == 0.0f ? pos_inf() : (float)(-log2p * 0.69314718055994530942), B, lossSum, ticket);
  }
}

// What the natural sweeps know of an utterance's positions besides the pair rows.
struct NaturalTerms {
  const float* P;        // [B,maxU,V]
  const float* ebl;      // [B,maxT] blank emissions
  const int* labels;
  int V, blank;
};

// log(exp(a)+exp(b)) with the reference's -inf handling and operation order; the correction term
// is evaluated with the hardware ex2/lg2 units (absolute error ~2e-7, far below one ulp of the
// alphas it is added to once they exceed a few units in magnitude).
// What counts is the number of instructions (895 instead of ~200 cycles per diagonal with branches for
// -inf).  One of them -inf: the correction is log(1 + 0) by itself.  Both: the minimum with 0 turns
// the NaN of their difference into a finite correction.  The .ftz forms have the same results: an
// exponential that would be subnormal adds nothing to 1.
__device__ __forceinline__ float lse2_fast(float a, float b) {
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));   // (NaN if one of them is)
  return m + lg2_approx(1.0f + ex2_approx(fminf(-fabsf(a - b), 0.0f) * kLog2e)) * kLn2F;
}

// Label axes of 129..256 positions: pair rows (LN, E[t,label_u]), (+inf, 0) where there is no node,
// so that whatever leaves such a node is -inf.  E[t,blank] of a lane's first position is read from
// shared memory (an utterance of more than maxStage frames: from global), the others' follow from it:
// position r + 1 meets a frame one diagonal after position r.
template <int NPL>
__global__ void __launch_bounds__(32) alpha_natural_kernel(
    const float2* __restrict__ rows, const NaturalTerms n, float* __restrict__ costs,
    float* __restrict__ alphas, i64 stride, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int B, int maxT, int maxU, int maxStage, float* lossSum,
    unsigned* ticket) {
  constexpr int ld = 32 * NPL, kRing = ring_blocks(NPL);
  extern __shared__ __align__(128) uint8_t smemA[];
  const int b = blockIdx.x, lane = threadIdx.x;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (T <= 0 || U <= 0) {
    if (lane == 0) finish_cost(costs, b, pos_inf(), B, lossSum, ticket);
    return;
  }
  const int S = T + U - 1, nBlocks = (S + kDiag - 1) / kDiag, u0 = NPL * lane;
  PairRing<NPL> ring(smemA, rows + (i64)b * stride, lane, U, 0x7f800000u, 0u);
  auto issue = [&](int k) { ring.issue(k % kRing, (i64)k * kDiag, k < nBlocks ? min(kDiag, S - k * kDiag) : 0); };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  const float* ebl = n.ebl + (i64)b * maxT;
  float* sEb = reinterpret_cast<float*>(smemA + kRing * kDiag * ld * 8);
  const bool staged = T <= maxStage;
  for (int t = lane; staged && t < T; t += 32) sEb[t] = ebl[t];
  __syncwarp();
  const float* ebRow = staged ? sEb : ebl;
  auto eblAt = [&](int t) { return ebRow[min(max(t, 0), T - 1)]; };
  float* al = alphas + (i64)b * stride;
  float pbl[NPL], plab[NPL], eb[NPL], stay[NPL], step[NPL];
#pragma unroll
  for (int r = 0; r < NPL; ++r) {
    const int u = u0 + r, uc = min(u, U - 1);
    const float* p = n.P + ((i64)b * maxU + uc) * n.V;
    pbl[r] = p[n.blank];
    plab[r] = u < U - 1 ? p[n.labels[(i64)b * (maxU - 1) + u]] : 0.0f;
    eb[r] = eblAt(-u);
    stay[r] = step[r] = neg_inf();
  }
  if (lane == 0) stay[0] = 0.0f;   // alpha(0,0) = 0
  float up = neg_inf();
  for (int k = 0; k < nBlocks; ++k) {
    issue(k + kRing - 1);
    ring.wait();
    const int slot = k % kRing, nd = min(kDiag, S - k * kDiag);
    float* out = al + (i64)k * kDiag * ld;
    const int tNext = k * kDiag + 1 - u0;   // frame of position u0 on the diagonal after the block's first
    auto diag = [&](int i) {
      float lnv[NPL], el[NPL], a[NPL];
      ring.read(slot, i, lnv, el);
      const float ebNext = eblAt(tNext + i), first = lane ? up : neg_inf();
      // the last position first, whose step leaves by a shuffle; each position still needs the
      // previous diagonal's step of the one below it
#pragma unroll
      for (int r = NPL - 1; r >= 0; --r) {
        a[r] = lse2_fast(r ? step[(r + NPL - 1) % NPL] : first, stay[r]);
        stay[r] = ((a[r] + eb[r]) + pbl[r]) - lnv[r];
        step[r] = ((a[r] + el[r]) + plab[r]) - lnv[r];
        if (r == NPL - 1) up = __shfl_up_sync(0xffffffffu, step[r], 1);
      }
#pragma unroll
      for (int r = NPL - 1; r > 0; --r) eb[r] = eb[r - 1];
      eb[0] = ebNext;
      if (ring.act) store_row<NPL>(out + i * ld, lane, a);
    };
    if (nd == kDiag) {
#pragma unroll
      for (int i = 0; i < kDiag; ++i) diag(i);
    } else {
#pragma unroll 1
      for (int i = 0; i < nd; ++i) diag(i);
    }
  }
  ring.drain();
#pragma unroll
  for (int r = 0; r < NPL; ++r)
    if (u0 + r == U - 1) finish_cost(costs, b, -stay[r], B, lossSum, ticket);
}

// ---------------------------------------------------------------------------
// reverse occupancy sweep
// ---------------------------------------------------------------------------
// With g(t,u) the occupancy of node (t,u) (the reference's dalphas, sign dropped):
//   stay(t,u) = g(t+1,u) * FB(t,u),  FB = 2^((alpha(t,u) + blank arc) - alpha(t+1,u))
//   step(t,u) = g(t,u+1) * FL(t,u),  FL = 2^((alpha(t,u) + label arc) - alpha(t,u+1))
//   (alphas and arcs in log2 units; the parenthesised sums are rounded exactly as in the alpha
//   kernel, so FB and FL of the arcs entering a node add up to 1 to within the error of ex2/lg2.
//   The stored alphas are relative to a per-block offset, see alpha_sweep_kernel: where the
//   successors' diagonal opens a new block, that block's delta is subtracted from the sum first,
//   exactly as the alpha kernel lowered its carried state.)
//   g(t,u) = stay + step,            g(T-1,U-1) = 1 (the terminating blank, booked as stay)
//
// gamma_factors_kernel: the pairs (FB, FL) of every node of the diagonals below S, zero where there
// is no arc (natural: from the pair rows of alpha_natural_kernel, by the accurate expf).  One warp
// per 4 diagonals.  Bound by memory: a pair and an alpha (12 bytes) read, 8 written per node.
constexpr int kFactorRows = 4, kFactorWarps = 8;
template <int NPL>
__global__ void __launch_bounds__(32 * kFactorWarps) gamma_factors_kernel(
    const float2* __restrict__ arcs, const float* __restrict__ alphas,
    const float* __restrict__ deltas, const NaturalTerms n, float2* __restrict__ F,
    unsigned* __restrict__ occTicket, i64 stride, int nDiag, const int* __restrict__ inLens, const int* __restrict__ labLens, int maxT,
    int maxU) {
  constexpr int ld = 32 * NPL, kPieces = NPL / 2;
  const int b = blockIdx.y, lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) occTicket[b] = 0u;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU), S = T + U - 1;
  const int d0 = (blockIdx.x * kFactorWarps + (threadIdx.x >> 5)) * kFactorRows, u0 = NPL * lane;
  if (T <= 0 || U <= 0 || d0 >= S || u0 >= U) return;
  const float* al = alphas + (i64)b * stride;
  const float* dl = deltas + (i64)b * ((nDiag + kDiag - 1) / kDiag);
  const int next = row_slot(min(u0 + NPL, ld - 1), NPL);   // (the last position has no label arc)
  float a[kFactorRows + 1][NPL], aN[kFactorRows + 1], x[kFactorRows][NPL], y[kFactorRows][NPL];
#pragma unroll
  for (int i = 0; i <= kFactorRows; ++i) {
    const i64 row = (i64)min(d0 + i, S - 1) * ld;
    load_row<NPL>(al + row, lane, a[i]);
    aN[i] = al[row + next];
    if constexpr (natural(NPL)) {   // (nodes that nothing leads to: no differences of infinities)
#pragma unroll
      for (int r = 0; r < NPL; ++r) a[i][r] = not_below_lowest(a[i][r]);
      aN[i] = not_below_lowest(aN[i]);
    }
    if (i < kFactorRows) {
      const float2* ar = arcs + (i64)b * stride + row;
#pragma unroll
      for (int q = 0; q < kPieces; ++q) {
        const float4 f = reinterpret_cast<const float4*>(ar)[q * 32 + lane];
        x[i][2 * q] = f.x;
        y[i][2 * q] = f.y;
        x[i][2 * q + 1] = f.z;
        y[i][2 * q + 1] = f.w;
      }
      if constexpr (NPL & 1) {
        const float2 f = ar[kPieces * 64 + lane];
        x[i][NPL - 1] = f.x;
        y[i][NPL - 1] = f.y;
      }
    }
  }
  float pbl[NPL], plab[NPL];
  if constexpr (natural(NPL)) {
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
      const int u = u0 + r;
      const float* p = n.P + ((i64)b * maxU + min(u, U - 1)) * n.V;
      pbl[r] = p[n.blank];
      plab[r] = u < U - 1 ? p[n.labels[(i64)b * (maxU - 1) + u]] : 0.0f;
    }
  }
#pragma unroll
  for (int i = 0; i < kFactorRows; ++i) {
    const int d = d0 + i;
    if (d >= S) break;
    // (rebased) the successors' diagonal opens a block: the carried sums were lowered by its delta
    const float dlt = (!natural(NPL) && (d + 1) % kDiag == 0 && d + 1 < S) ? dl[(d + 1) / kDiag] : 0.0f;
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
      const int u = u0 + r, t = d - u;
      const bool valid = u < U && t >= 0 && t < T;
      const float art = r < NPL - 1 ? a[i + 1][(r + 1) % NPL] : aN[i + 1];
      float fb, fl;
      if constexpr (natural(NPL)) {
        const float eb = n.ebl[(i64)b * maxT + min(max(t, 0), T - 1)], lnv = x[i][r], el = y[i][r];
        fb = expf((((a[i][r] + eb) + pbl[r]) - lnv) - a[i + 1][r]);
        fl = expf((((a[i][r] + el) + plab[r]) - lnv) - art);
      } else {
        fb = ex2_approx(((a[i][r] + x[i][r]) - dlt) - a[i + 1][r]);
        fl = ex2_approx(((a[i][r] + y[i][r]) - dlt) - art);
      }
      x[i][r] = (valid && t < T - 1) ? fb : 0.0f;
      if (t == T - 1 && u == U - 1) x[i][r] = 1.0f;   // terminating blank, fed by g(T,U-1) := 1
      y[i][r] = (valid && u < U - 1) ? fl : 0.0f;
    }
    float2* out = F + (i64)b * stride + (i64)d * ld;
#pragma unroll
    for (int q = 0; q < kPieces; ++q)
      reinterpret_cast<float4*>(out)[q * 32 + lane] = make_float4(x[i][2 * q], y[i][2 * q], x[i][2 * q + 1], y[i][2 * q + 1]);
    if constexpr (NPL & 1) out[kPieces * 64 + lane] = make_float2(x[i][NPL - 1], y[i][NPL - 1]);
  }
}

// The recursion on the prepared factors: g of the diagonals S (the node beyond the terminating
// blank) down to 0.
template <int NPL>
__global__ void __launch_bounds__(32) gamma_sweep_kernel(
    const float2* __restrict__ F, float* __restrict__ g, unsigned* __restrict__ gradTickets, i64 stride,
    const int* __restrict__ inLens, const int* __restrict__ labLens, int maxT, int maxU) {
  constexpr int ld = 32 * NPL;
  extern __shared__ __align__(128) uint8_t smemG[];
  const int b = blockIdx.x, lane = threadIdx.x;
  if (b == 0)   // the counters of the gradient kernel behind this one
    for (int i = lane; i < kGradTickets; i += 32) gradTickets[i] = 0u;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (T <= 0 || U <= 0) return;
  const int S = T + U - 1, nBlocks = (S + kDiag - 1) / kDiag, u0 = NPL * lane;
  constexpr int kRing = ring_blocks(NPL);
  PairRing<NPL> ring(smemG, F + (i64)b * stride, lane, U, 0u, 0u);
  // block k holds the rows [max(S - 16(k+1), 0), S - 16k)
  auto issue = [&](int k) {
    const int lo = max(S - kDiag * (k + 1), 0);
    ring.issue(k % kRing, lo, k < nBlocks ? S - kDiag * k - lo : 0);
  };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  float* out0 = g + (i64)b * stride;
  float s[NPL];
#pragma unroll
  for (int r = 0; r < NPL; ++r) s[r] = (u0 + r == U - 1) ? 1.0f : 0.0f;
  if (ring.act) store_row<NPL>(out0 + (i64)S * ld, lane, s);
  // (lane 31 gets its own s[0] back: harmless, the label arc of its last position never exists)
  float right = __shfl_down_sync(0xffffffffu, s[0], 1);
  for (int k = 0; k < nBlocks; ++k) {
    issue(k + kRing - 1);
    ring.wait();
    const int slot = k % kRing, lo = max(S - kDiag * (k + 1), 0), nd = S - kDiag * k - lo;
    float* out = out0 + (i64)lo * ld;
    auto diag = [&](int i) {
      float x[NPL], y[NPL], n[NPL];
      ring.read(slot, i, x, y);
      // position 0 first: its result is shuffled for the next diagonal; the last position, which
      // waits for the shuffle, at the end
      const float in = right;
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        const float nb = r < NPL - 1 ? s[(r + 1) % NPL] : in;
        n[r] = __fadd_rn(__fmul_rn(s[r], x[r]), __fmul_rn(nb, y[r]));
        if (r == 0) right = __shfl_down_sync(0xffffffffu, n[0], 1);
      }
#pragma unroll
      for (int r = 0; r < NPL; ++r) s[r] = n[r];
      if (ring.act) store_row<NPL>(out + i * ld, lane, s);
    };
    if (nd == kDiag) {
#pragma unroll
      for (int i = kDiag - 1; i >= 0; --i) diag(i);
    } else {
#pragma unroll 1
      for (int i = nd - 1; i >= 0; --i) diag(i);
    }
  }
  ring.drain();
}

// ---------------------------------------------------------------------------------
// arc terms
// ---------------------------------------------------------------------------------
struct PrepParams {
  const void* E;
  const void* P;
  float* LN;                 // [B,maxT,maxU]; marked nodes are recomputed in place
  const float* ELrow;        // [B,maxU,maxT] label emissions, or null
  float* ebl;                // [B,maxT] blank emissions: read with ELrow, else written for the natural sweeps
  float2* arcs;
  const int* labels;
  const int* inLens;
  const int* labLens;
  int maxT, maxU, V, blank, npl, ld, extra;
  bool nat;                  // for the natural sweeps
  i64 stride;
};

// One CTA per 32x32 (t,u) tile: the log-probabilities (log2 units) of the two arcs leaving every
// node, written along the diagonals,
//   (E[t,blank]   + P[u,blank]   - LN[t,u]) * log2(e)
//   (E[t,label_u] + P[u,label_u] - LN[t,u]) * log2(e),  u < U-1
// or, for the natural sweeps, (LN[t,u], E[t,label_u]).
// The tiles beyond both ends of the time axis (`extra` of them on each side) write the "no such
// arc" of nodes outside the lattice, so that the array needs no fill.  Log-normalisers marked by
// the tensor-core kernel (NaN) are recomputed exactly first.
// Bound by memory: reads 8 and writes 8 bytes per node.
template <typename TIn>
__global__ void __launch_bounds__(256) sweep_prep_kernel(const PrepParams p) {
  __shared__ float tLn[32][kTileLd], tEl[32][kTileLd], tEb[32];
  const int b = blockIdx.z, t0 = ((int)blockIdx.y - p.extra) * 32, u0 = blockIdx.x * 32;
  const int T = min(p.inLens[b], p.maxT), U = min(p.labLens[b] + 1, p.maxU);
  if (T <= 0 || U <= 0) return;
  const int Uw = (U + p.npl - 1) / p.npl * p.npl, S = T + U - 1;
  if (u0 >= Uw || t0 + u0 + 62 < 0 || t0 + u0 >= S) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int u = u0 + lane;
  float2* arcs = p.arcs + (i64)b * p.stride + pair_slot(u, p.npl);
  const bool live = t0 + 31 >= 0 && t0 < T && u0 < U;   // does the tile hold any node?
  float pbl = 0.0f, plab = 0.0f;
  if (live) {
    const TIn* e = static_cast<const TIn*>(p.E) + (i64)b * p.maxT * p.V;
    const TIn* pr0 = static_cast<const TIn*>(p.P) + (i64)b * p.maxU * p.V;
    float* ln = p.LN + (i64)b * p.maxT * p.maxU;
    const float* elr = p.ELrow ? p.ELrow + (i64)b * p.maxU * p.maxT : nullptr;
    const int* lab = p.labels + (i64)b * (p.maxU - 1);
    const int uc = min(u, U - 1);
    const int labc = (uc < U - 1) ? lab[uc] : p.blank;
    // all loads first (unconditional, clamped into the lattice)
    float va[4], vc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int tc = min(t0 + w * 4 + k, T - 1);
      va[k] = ln[(i64)tc * p.maxU + uc];
      vc[k] = elr ? elr[(i64)min(u0 + w * 4 + k, max(U - 2, 0)) * p.maxT + min(t0 + lane, T - 1)]
                  : to_f32(e[(i64)tc * p.V + labc]);
    }
    pbl = to_f32(pr0[(i64)uc * p.V + p.blank]);
    plab = to_f32(pr0[(i64)uc * p.V + labc]);
    if (threadIdx.x < 32) {
      const int tc = min(t0 + lane, T - 1);
      tEb[lane] = elr ? p.ebl[(i64)b * p.maxT + tc] : to_f32(e[(i64)tc * p.V + p.blank]);
      if (!elr && p.nat && u0 == 0) p.ebl[(i64)b * p.maxT + tc] = tEb[lane];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int tt = w * 4 + k, t = t0 + tt;
      float a = (t < T && u < U) ? va[k] : 0.0f;
      unsigned todo = __ballot_sync(0xffffffffu, a != a);
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const float exact = warp_logsumexp(e + (i64)t * p.V, pr0 + (i64)(u0 + src) * p.V, p.V, lane);
        if (lane == src) {
          a = exact;
          ln[(i64)t * p.maxU + u] = a;
        }
      }
      tLn[tt][lane] = a;
      if (elr) tEl[lane][tt] = vc[k];   // loaded with lane <-> frame, row <-> label position
      else tEl[tt][lane] = vc[k];
    }
  }
  __syncthreads();
  // (lane <-> position; step i takes diagonal i of the tile in the lanes up to i and diagonal
  // i + 32 in the others: every lane has a node and a warp touches two rows)
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int tt = (w + 8 * k - lane) & 31, t = t0 + tt, d = t + u;
    if (d < 0 || d >= S || u >= Uw) continue;
    float2 f = p.nat ? make_float2(pos_inf(), 0.0f)
                     : make_float2(__uint_as_float(kNoArcBits), __uint_as_float(kNoArcBits));
    if (t >= 0 && t < T && u < U) {
      const float lnv = tLn[tt][lane];
      f.x = p.nat ? lnv : ((tEb[tt] + pbl) - lnv) * kLog2e;
      if (u < U - 1) f.y = p.nat ? tEl[tt][lane] : ((tEl[tt][lane] + plab) - lnv) * kLog2e;
      if (!p.nat) f = make_float2(arc_term(f.x), arc_term(f.y));
    }
    arcs[(i64)d * p.ld] = f;
  }
}

// ---------------------------------------------------------------------------------
// operands of the gradient kernels
// ---------------------------------------------------------------------------------
struct OccParams {
  const float2* F;
  const float* g;
  const float *LN, *rowRef, *maxP, *deltas;
  float *W, *emT, *nref, *ebl, *pBlank, *pLabel;
  float* partial;                // [B, tiles, 2, maxU]
  unsigned* ticket;              // [B], zero on entry
  const int *inLens, *labLens;
  int maxT, maxU, ldW, ldT, npl;
  i64 stride;
};

// One CTA per 32 frames of one utterance, the 32x32 lattice tiles of the label axis side by side,
// kOccWarps warps each.  With delta_b the upstream gradient:
//   stay(t,u) = g(t+1,u) FB(t,u), step(t,u) = g(t,u+1) FL(t,u)
//   W [B,maxT,ldW] = delta_b * (stay + step) * exp(ref(t) + maxP(u) - LN(t,u)), rounded to TF32
//                   (round-to-nearest; the tensor core would otherwise truncate), zero outside
//                   the valid lattice.  (The exponent is clamped at 80: it only gets there where
//                   the factored log-normaliser had underflowed.)
//   emT [B,maxU,ldT] = delta_b * step with the frames contiguous, so a tile's slice for one label is
//                   one TMA row; zero outside
//   ebl [B,ldT] = delta_b * sum_u stay(t,u), added in a fixed order;  nref [B,ldT] = -rowRef*log2(e)
//                   (row lengths: multiples of 4 floats as TMA requires)
//   pBlank / pLabel [B,maxU] = sum_t stay / step: every CTA leaves its partial sums, the CTA of the
//                   utterance that finishes last adds them in tile order.
// With delta_b folded in here the gradient kernel never multiplies by it per element, and frames
// at or beyond T_b come out as exact zeros without a select.
// TC = false serves the SIMT gradient kernels: W unrounded and unscaled, step row-major
// [B,maxT,maxU] (through emT), the row sums with row length maxT (through ebl), no nref.
// Bound by memory: 16 bytes read and 8 written per node.
constexpr int kOccWarps = 4;              // warps per 32 label positions
constexpr int kOccRows = 32 / kOccWarps;  // frames (diagonals of the tile) per warp
// shared memory in floats: two tiles per 32 positions, row sums, column sums per warp, a flag
__host__ __device__ constexpr int occ_smem_floats(int blocks) {
  return blocks * (2 * 32 * kTileLd + 32 + 2 * 32 * kOccWarps) + 4;
}
template <bool TC, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS <= 640 ? 2 : 1) occupancy_kernel(const OccParams p) {
  using Tile = float[32][kTileLd];
  extern __shared__ __align__(16) float smemO[];
  const int blocks = p.ldW / 32, cols = p.ldW;   // blocks of 32 positions
  Tile* tS = reinterpret_cast<Tile*>(smemO);
  Tile* tE = tS + blocks;
  float* sRow = reinterpret_cast<float*>(tE + blocks);   // [blocks][32]
  float* sCol = sRow + cols;                             // [kOccWarps][2][cols]
  int* sLast = reinterpret_cast<int*>(sCol + 2 * kOccWarps * cols);
  const int b = blockIdx.y, t0 = blockIdx.x * 32;
  const int T = min(p.inLens[b], p.maxT), U = min(p.labLens[b] + 1, p.maxU);
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % kOccWarps, ub = threadIdx.x / (32 * kOccWarps);
  const int ld = 32 * p.npl;
  const float delta = (TC && p.deltas) ? p.deltas[b] : 1.0f;
  const bool some = T > 0 && U > 0 && t0 < T;
  float* part = p.partial + ((i64)b * gridDim.x + blockIdx.x) * 2 * p.maxU;
  const int u0 = ub * 32, u = u0 + lane;
  const bool live = some && u0 < U;
  float shift[kOccRows];   // exp(ref + maxP - LN) of the frames whose row of W this warp writes
  if (live) {
    const int uc = min(u, U - 1);
    const float mp = p.maxP[(i64)b * p.maxU + uc];
#pragma unroll
    for (int k = 0; k < kOccRows; ++k) {
      const i64 t = (i64)b * p.maxT + min(t0 + w * kOccRows + k, T - 1);
      shift[k] = (p.rowRef[t] + mp) - p.LN[t * p.maxU + uc];
    }
    const float2* F = p.F + (i64)b * p.stride + pair_slot(uc, p.npl);
    const float* g = p.g + (i64)b * p.stride;
    // Step i takes diagonal i of the tile in the lanes up to i and diagonal i + 32 in the others:
    // every lane has a node and a warp touches two rows.  Four steps at a time with all their
    // loads issued before the first use (unconditional, clamped into the lattice).
    const int slot1 = row_slot(uc, p.npl), slot2 = row_slot(min(u + 1, U - 1), p.npl);
#pragma unroll
    for (int q = 0; q < kOccRows; q += 4) {
      float2 f[4];
      float g1[4], g2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const i64 row = (i64)(min(t0 + ((w + kOccWarps * (q + j) - lane) & 31), T - 1) + uc) * ld;
        f[j] = F[row];
        g1[j] = g[row + ld + slot1];
        g2[j] = g[row + ld + slot2];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int tt = (w + kOccWarps * (q + j) - lane) & 31;
        const bool in = t0 + tt < T && u < U;
        // (arcs that do not exist have factor 0; what they would lead to may never have been
        // written, hence the selects)
        tS[ub][tt][lane] = in && f[j].x != 0.0f ? __fmul_rn(g1[j], f[j].x) : 0.0f;
        tE[ub][tt][lane] = in && f[j].y != 0.0f ? __fmul_rn(g2[j], f[j].y) : 0.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < kOccRows; ++k) shift[k] = expf(fminf(shift[k], 80.0f));
  }
  __syncthreads();
  // rows w kOccRows .. of the tile (frames for W, label positions for the transposed emT); beyond
  // T_b and U_b both occupancies are zero, and so is W
  const int k0 = w * kOccRows;
  const int frames = min(kOccRows, p.maxT - (t0 + k0)), positions = min(kOccRows, p.maxU - (u0 + k0));
  float colS = 0.0f, colE = 0.0f;   // sums over the warp's frames
  if (live) {
    float* Wp = p.W + ((i64)b * p.maxT + t0 + k0) * p.ldW + u;
#pragma unroll
    for (int k = 0; k < kOccRows; ++k) {
      const float st = tS[ub][k0 + k][lane], sp = tE[ub][k0 + k][lane];
      colS += st;
      colE += sp;
      float x = u < U && t0 + k0 + k < T ? __fadd_rn(st, sp) * shift[k] * delta : 0.0f;
      if (TC) x = tf32_round(x);
      if (k < frames) Wp[k * p.ldW] = x;
    }
    if (TC) {  // transposed: lane <-> frame, row <-> label position
      float* Ep = p.emT + ((i64)b * p.maxU + u0 + k0) * p.ldT + t0 + lane;
      if (t0 + lane < p.ldT) {
#pragma unroll
        for (int k = 0; k < kOccRows; ++k)
          if (k < positions) Ep[k * p.ldT] = tE[ub][lane][k0 + k] * delta;
      }
    } else if (u < p.maxU) {
      float* Ep = p.emT + ((i64)b * p.maxT + t0 + k0) * p.maxU + u;
#pragma unroll
      for (int k = 0; k < kOccRows; ++k)
        if (k < frames) Ep[k * p.maxU] = tE[ub][k0 + k][lane];
    }
    if (w == 0) {  // lane <-> frame: sum over the block's positions
      float v = 0.0f;
#pragma unroll 8
      for (int j = 0; j < 32; ++j) v += tS[ub][lane][j];
      sRow[u0 + lane] = v;
    }
  } else {
    for (int k = 0; k < frames; ++k) {
      p.W[((i64)b * p.maxT + t0 + k0 + k) * p.ldW + u] = 0.0f;
      if (!TC && u < p.maxU) p.emT[((i64)b * p.maxT + t0 + k0 + k) * p.maxU + u] = 0.0f;
    }
    if (TC && t0 + lane < p.ldT)
      for (int k = 0; k < positions; ++k) p.emT[((i64)b * p.maxU + u0 + k0 + k) * p.ldT + t0 + lane] = 0.0f;
    if (w == 0) sRow[u0 + lane] = 0.0f;
  }
  sCol[2 * w * cols + u] = colS;
  sCol[(2 * w + 1) * cols + u] = colE;
  __syncthreads();
  for (int i = threadIdx.x; some && i < 2 * cols; i += blockDim.x) {
    const int cw = i >= cols, cu = i - cw * cols;
    if (cu < p.maxU) {
      float s = sCol[i];
#pragma unroll
      for (int k = 1; k < kOccWarps; ++k) s += sCol[2 * k * cols + i];
      part[cw * p.maxU + cu] = s;
    }
  }
  if (threadIdx.x < 32) {
    const int t = t0 + lane;
    const bool ok = some && t < T;
    float rs = sRow[lane];
    for (int j = 1; j < blocks; ++j) rs += sRow[j * 32 + lane];
    if (TC) {
      if (t < p.ldT) {
        p.nref[(i64)b * p.ldT + t] = ok ? -p.rowRef[(i64)b * p.maxT + t] * kLog2e : 0.0f;
        p.ebl[(i64)b * p.ldT + t] = ok ? rs * delta : 0.0f;
      }
    } else if (t < p.maxT) {
      p.ebl[(i64)b * p.maxT + t] = ok ? rs : 0.0f;
    }
  }
  // the CTA of the utterance that finishes last adds the partial sums
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *sLast = atomicAdd(&p.ticket[b], 1u) == gridDim.x - 1 ? 1 : 0;
  }
  __syncthreads();
  if (!*sLast) return;
  __threadfence();
  const int tiles = (T > 0 && U > 0) ? (T + 31) / 32 : 0;
  float* acc = smemO;            // [4][2][cols] sums of the four quarters of the tiles
  const float* all = p.partial + (i64)b * gridDim.x * 2 * p.maxU;
  for (int i = threadIdx.x; i < 4 * 2 * p.maxU; i += blockDim.x) {
    const int q = i / (2 * p.maxU), c = i - q * 2 * p.maxU;
    const int z0 = tiles * q / 4, z1 = tiles * (q + 1) / 4;
    float s = 0.0f;
#pragma unroll 8
    for (int z = z0; z < z1; ++z) s += __ldcg(all + (i64)z * 2 * p.maxU + c);
    acc[q * 2 * cols + c] = s;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * p.maxU; c += blockDim.x) {
    const int cu2 = c < p.maxU ? c : c - p.maxU;
    const float s = cu2 < U ? ((acc[c] + acc[2 * cols + c]) + acc[4 * cols + c]) + acc[6 * cols + c] : 0.0f;
    (c < p.maxU ? p.pBlank : p.pLabel)[(i64)b * p.maxU + cu2] = s;
  }
}

}  // namespace

bool sweep_supported(Dims d) { return d.maxU >= 1 && d.maxU <= 256; }

SweepGeom sweep_geom(Dims d) {
  SweepGeom g;
  g.npl = d.maxU <= 32 ? 1 : d.maxU <= 64 ? 2 : d.maxU <= 128 ? 4 : div_up(d.maxU, 32);
  g.ld = 32 * g.npl;
  g.nDiag = d.maxT + d.maxU;   // one spare row: the node beyond the terminating blank
  g.nBlk = (g.nDiag + kDiag - 1) / kDiag;
  g.stride = (i64)g.ld * g.nDiag;
  return g;
}

size_t sweep_partial_floats(Dims d) {
  return (size_t)d.B * div_up((int)round_up64(d.maxT, 4), 32) * 2 * d.maxU;
}

#define TB200_BY_NPL(npl, CALL)              \
  do {                                       \
    if ((npl) == 1) { CALL(1); }             \
    else if ((npl) == 2) { CALL(2); }        \
    else { CALL(4); }                        \
  } while (0)
#define TB200_BY_NPL_NATURAL(npl, CALL)      \
  do {                                       \
    if ((npl) == 5) { CALL(5); }             \
    else if ((npl) == 6) { CALL(6); }        \
    else if ((npl) == 7) { CALL(7); }        \
    else { CALL(8); }                        \
  } while (0)
#define TB200_BY_NPL_ANY(npl, CALL)          \
  do {                                       \
    if ((npl) <= 4) { TB200_BY_NPL(npl, CALL); } \
    else { TB200_BY_NPL_NATURAL(npl, CALL); } \
  } while (0)

void launch_sweep_forward(const void* E, const void* P, float* LN, const float* ELrow,
                          float* ebl, float2* arcs, float* alphas, float* deltas, float* costs,
                          float* lossSum, unsigned* ticket, unsigned* halves, const int* labels,
                          const int* inLens, const int* labLens, SweepGeom g, Dims d, bool score,
                          cudaStream_t stream) {
  if (d.B <= 0) return;
  const bool nat = natural(g.npl) && !score;
  if (nat && d.dtype != kDtypeF32)
    throw std::invalid_argument("bf16 emissions: the label axis must not exceed 128 positions");
  if (d.maxT > 0) {
    PrepParams q{};
    q.E = E; q.P = P; q.LN = LN; q.ELrow = ELrow; q.ebl = ebl; q.arcs = arcs;
    q.labels = labels; q.inLens = inLens; q.labLens = labLens;
    q.maxT = d.maxT; q.maxU = d.maxU; q.V = d.V; q.blank = d.blank; q.npl = g.npl; q.ld = g.ld;
    q.extra = div_up(d.maxU, 32); q.nat = nat; q.stride = g.stride;
    const dim3 grid(div_up(d.maxU, 32), div_up(d.maxT, 32) + 2 * q.extra, d.B);
    ScopedKernel sk("sweep_prep", stream);
    if (d.dtype == kDtypeBf16) sweep_prep_kernel<bf16><<<grid, 256, 0, stream>>>(q);
    else sweep_prep_kernel<float><<<grid, 256, 0, stream>>>(q);
    TB200_CHECK_LAUNCH();
  }
  const int ringBytes = ring_blocks(g.npl) * kDiag * g.ld * 8;
  if (score) {
    ScopedKernel sk("score_sweep", stream);
#define CALL(NPL)                                                                                \
  allow_dyn_smem(score_sweep_kernel<NPL>, ringBytes);                                            \
  score_sweep_kernel<NPL><<<dim3(d.B, 2), 32, ringBytes, stream>>>(arcs, costs, alphas, deltas,  \
                                                                   g.stride, inLens, labLens, d.B, \
                                                                   d.maxT, d.maxU, lossSum, ticket, halves)
    TB200_BY_NPL_ANY(g.npl, CALL);
#undef CALL
    TB200_CHECK_LAUNCH();
    return;
  }
  ScopedKernel sk("alpha_sweep", stream);
  if (nat) {
    const NaturalTerms n{static_cast<const float*>(P), ebl, labels, d.V, d.blank};
    // blank emissions in shared memory: as many frames as two CTAs per SM leave room for
    constexpr int kCeiling = 112 * 1024;
    const int stage = std::min(d.maxT, (kCeiling - ringBytes) / 4), smem = ringBytes + stage * 4;
#define CALL(NPL)                                                                                \
  allow_dyn_smem(alpha_natural_kernel<NPL>, kCeiling);                                           \
  alpha_natural_kernel<NPL><<<d.B, 32, smem, stream>>>(arcs, n, costs, alphas, g.stride, inLens, \
                                                       labLens, d.B, d.maxT, d.maxU, stage,      \
                                                       lossSum, ticket)
    TB200_BY_NPL_NATURAL(g.npl, CALL);
#undef CALL
    TB200_CHECK_LAUNCH();
    return;
  }
  const int smem = ringBytes;
#define CALL(NPL)                                                                                \
  allow_dyn_smem(alpha_sweep_kernel<NPL>, smem);                                                 \
  alpha_sweep_kernel<NPL><<<d.B, 32, smem, stream>>>(arcs, costs, alphas, deltas, g.stride,      \
                                                     g.nDiag, inLens, labLens, d.B, d.maxT,      \
                                                     d.maxU, lossSum, ticket)
  TB200_BY_NPL(g.npl, CALL);
#undef CALL
  TB200_CHECK_LAUNCH();
}

void launch_sweep_backward(const SweepScratch& w, const float* P, const float* blankEmissions,
                           const int* labels, const float2* arcs, const float* alphas,
                           const float* alphaDeltas, const float* LN, const float* rowRef,
                           const float* maxP, const float* deltas, float* W, float* emT, float* nref,
                           float* ebl, float* pBlank, float* pLabel, const int* inLens,
                           const int* labLens, SweepGeom g, Dims d, bool tensorCore,
                           cudaStream_t stream) {
  if (d.B <= 0 || d.maxT <= 0) return;
  {
    ScopedKernel sk("gamma_factors", stream);
    const dim3 grid(div_up(g.nDiag, kFactorRows * kFactorWarps), d.B);
#define CALL(NPL)                                                                              \
  gamma_factors_kernel<NPL><<<grid, 32 * kFactorWarps, 0, stream>>>(                           \
      arcs, alphas, alphaDeltas, n, w.F, w.ticket, g.stride, g.nDiag, inLens, labLens, d.maxT, d.maxU)
    const NaturalTerms n{P, blankEmissions, labels, d.V, d.blank};
    TB200_BY_NPL_ANY(g.npl, CALL);
#undef CALL
    TB200_CHECK_LAUNCH();
  }
  {
    const int smem = ring_blocks(g.npl) * kDiag * g.ld * 8;
    ScopedKernel sk("gamma_sweep", stream);
#define CALL(NPL)                                                                              \
  allow_dyn_smem(gamma_sweep_kernel<NPL>, smem);                                               \
  gamma_sweep_kernel<NPL><<<d.B, 32, smem, stream>>>(w.F, w.g, w.gradTickets, g.stride, inLens,   \
                                                   labLens, d.maxT, d.maxU)
    TB200_BY_NPL_ANY(g.npl, CALL);
#undef CALL
    TB200_CHECK_LAUNCH();
  }
  OccParams o{};
  o.F = w.F; o.g = w.g; o.LN = LN; o.rowRef = rowRef; o.maxP = maxP;
  o.deltas = tensorCore ? deltas : nullptr; o.W = W; o.emT = emT; o.nref = nref; o.ebl = ebl;
  o.pBlank = pBlank; o.pLabel = pLabel; o.partial = w.partial; o.ticket = w.ticket;
  o.inLens = inLens; o.labLens = labLens; o.maxT = d.maxT; o.maxU = d.maxU;
  o.ldW = grads_umma_ld_w(d); o.ldT = grads_umma_ld_t(d); o.npl = g.npl; o.stride = g.stride;
  const dim3 grid(div_up(o.ldT, 32), d.B);
  ScopedKernel sk("occupancy", stream);
  const int threads = o.ldW * kOccWarps, smem = occ_smem_floats(o.ldW / 32) * (int)sizeof(float);
  auto go = [&](auto kernel, int maxThreads) {
    allow_dyn_smem(kernel, occ_smem_floats(maxThreads / (32 * kOccWarps)) * (int)sizeof(float));
    kernel<<<grid, threads, smem, stream>>>(o);
  };
  // (two CTAs per SM up to 160 positions: registers are limited to that)
  if (threads <= 512) tensorCore ? go(occupancy_kernel<true, 512>, 512) : go(occupancy_kernel<false, 512>, 512);
  else if (threads <= 640) tensorCore ? go(occupancy_kernel<true, 640>, 640) : go(occupancy_kernel<false, 640>, 640);
  else tensorCore ? go(occupancy_kernel<true, 1024>, 1024) : go(occupancy_kernel<false, 1024>, 1024);
  TB200_CHECK_LAUNCH();
}

}  // namespace tb200
