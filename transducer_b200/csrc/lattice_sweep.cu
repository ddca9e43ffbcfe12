// Lattice sweeps for label axes of at most 128 positions: each recursion runs in ONE warp per
// utterance, and everything that does not depend on the recursion in kernels of its own that use
// the whole GPU.
//
//   sweep_prep       arc log-probabilities of every node (log2 units), skewed
//   alpha_sweep      alpha recursion                                          (forward call)
//   gamma_factors    2^(alpha + arc - alpha') of every arc                    (backward call)
//   gamma_sweep      occupancy recursion: two products and a sum per node
//   occupancy        the operands of the gradient kernels
//
//   alpha   transducer/transducer_cpu.cpp:30-79   (transducer_cuda.cu:32-97)
//   reverse transducer/transducer_cpu.cpp:81-143  (transducer_cuda.cu:99-176)
//
// Diagonal d = t + u of an utterance is one row of ld = 32 NPL numbers; lane l of a sweep owns the
// NPL adjacent positions u = NPL l + r.  All nodes of a diagonal are independent; the one value
// per lane that crosses from the neighbouring lane arrives by a warp shuffle.  A sweep is a chain
// of T + U - 1 dependent diagonals whatever the batch, so what counts is how few instructions a
// diagonal takes: operands are brought to shared memory by cp.async, each lane copying just the
// 8 NPL bytes a row that it reads itself (no barrier, no other warp), several blocks of 16
// diagonals ahead, and the loop holds nothing but the recursion and its store.
#include <algorithm>

#include "kernels.h"
#include "profile.h"
#include "sm100.cuh"

namespace tb200 {
namespace {

using namespace sm100;

constexpr int kDiag = 16;   // diagonals per block
constexpr int kRing = 4;    // blocks in shared memory
constexpr float kLn2F = 0.6931471805599453f;
constexpr float kLog2e = 1.4426950408889634f;
// "No such arc": a large negative finite number, the identity of the alpha recursion without -inf
// arithmetic, so that the sweeps need no validity logic.
constexpr unsigned kNoArcBits = 0xF0F0F0F0u;

__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Place of position u within a row of pairs (arcs, factors): 16-byte pieces of two positions, the
// pieces of the 32 lanes side by side, so that a warp's 16-byte accesses are contiguous.
__host__ __device__ constexpr int pair_slot(int u, int npl) {
  return npl == 1 ? u : (((u % npl) >> 1) * 32 + u / npl) * 2 + (u % npl & 1);
}

// Copies blocks of pair rows into this lane's share of a shared-memory ring and reads them back.
// Lanes without positions of the utterance hold `fill` throughout.
template <int NPL>
struct PairRing {
  static constexpr int ld = 32 * NPL, kRowBytes = ld * 8;
  static constexpr int kPieces = NPL == 1 ? 1 : NPL / 2, kPiece = NPL == 1 ? 8 : 16;
  uint8_t* mine;
  const uint8_t* src;
  bool act;
  __device__ PairRing(uint8_t* ring, const float2* rows, int lane, int U, unsigned fill)
      : mine(ring + lane * kPiece), src(reinterpret_cast<const uint8_t*>(rows) + lane * kPiece), act(NPL * lane < U) {
    if (!act)
      for (int i = 0; i < kRing * kDiag; ++i)
#pragma unroll
        for (int q = 0; q < kPieces; ++q) {
          uint2* z = reinterpret_cast<uint2*>(mine + i * kRowBytes + q * 32 * kPiece);
          z[0] = make_uint2(fill, fill);
          if (kPiece == 16) z[1] = make_uint2(fill, fill);
        }
  }
  // rows [row, row + n) -> slot
  __device__ __forceinline__ void issue(int slot, i64 row, int n) {
    if (act) {
      const uint32_t dst = smem_u32(mine) + (uint32_t)slot * (kDiag * kRowBytes);
      const uint8_t* from = src + row * kRowBytes;
      auto one = [&](int i) {
#pragma unroll
        for (int q = 0; q < kPieces; ++q) {
          const uint32_t to = dst + i * kRowBytes + q * 32 * kPiece;
          const uint8_t* f = from + i * kRowBytes + q * 32 * kPiece;
          if (kPiece == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(f) : "memory");
          else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(f) : "memory");
        }
      };
      if (n == kDiag) {
#pragma unroll
        for (int i = 0; i < kDiag; ++i) one(i);
      } else {
#pragma unroll 1
        for (int i = 0; i < n; ++i) one(i);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // all but the newest kRing - 1 groups have landed
  __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory"); }
  __device__ __forceinline__ void drain() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
  __device__ __forceinline__ void read(int slot, int i, float (&x)[NPL], float (&y)[NPL]) const {
    const uint8_t* p = mine + (slot * kDiag + i) * kRowBytes;
    if constexpr (NPL == 1) {
      const float2 f = *reinterpret_cast<const float2*>(p);
      x[0] = f.x;
      y[0] = f.y;
    } else {
#pragma unroll
      for (int q = 0; q < kPieces; ++q) {
        const float4 f = *reinterpret_cast<const float4*>(p + q * 32 * kPiece);
        x[2 * q] = f.x;
        y[2 * q] = f.y;
        x[2 * q + 1] = f.z;
        y[2 * q + 1] = f.w;
      }
    }
  }
};

template <int NPL>
__device__ __forceinline__ void store_row(float* q, const float (&a)[NPL]) {
  if constexpr (NPL == 4) *reinterpret_cast<float4*>(q) = make_float4(a[0], a[1], a[2], a[3]);
  else if constexpr (NPL == 2) *reinterpret_cast<float2*>(q) = make_float2(a[0], a[1]);
  else q[0] = a[0];
}
template <int NPL>
__device__ __forceinline__ void load_row(const float* q, float (&a)[NPL]) {
  if constexpr (NPL == 4) {
    const float4 f = *reinterpret_cast<const float4*>(q);
    a[0] = f.x; a[1] = f.y; a[2] = f.z; a[3] = f.w;
  } else if constexpr (NPL == 2) {
    const float2 f = *reinterpret_cast<const float2*>(q);
    a[0] = f.x; a[1] = f.y;
  } else {
    a[0] = q[0];
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
// exactly), which keeps every stored number below ~500 in magnitude (ulp 3e-5).  delta_k is
// written to `deltas` for the reverse sweep, which subtracts it at the same point of the same
// sum.  The loss and the gradients then sit ~1e-4 from the float64 result.
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
  PairRing<NPL> ring(smemA, arcs + (i64)b * stride, lane, U, kNoArcBits);
  auto issue = [&](int k) { ring.issue(k % kRing, (i64)k * kDiag, k < nBlocks ? min(kDiag, S - k * kDiag) : 0); };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  float* al = alphas + (i64)b * stride + u0;
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
    // arrive, off the dependent chain.  (By then the state has sunk by another ~16 arcs; all
    // that matters is that the stored numbers stay small: below ~1000, ulp 6e-5.)
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
      if (ring.act) store_row<NPL>(out + i * ld, a);
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
    if (u0 + r == U - 1) finish_cost(costs, b, -(stayIn[r] + offset) * kLn2F, B, lossSum, ticket);
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
// is no arc.  One warp per 4 diagonals.  Bound by memory: 16 bytes read, 8 written per node.
constexpr int kFactorRows = 4, kFactorWarps = 8;
template <int NPL>
__global__ void __launch_bounds__(32 * kFactorWarps) gamma_factors_kernel(
    const float2* __restrict__ arcs, const float* __restrict__ alphas,
    const float* __restrict__ deltas, float2* __restrict__ F, unsigned* __restrict__ occTicket,
    i64 stride, int nDiag, const int* __restrict__ inLens, const int* __restrict__ labLens, int maxT,
    int maxU) {
  constexpr int ld = 32 * NPL, kPieces = NPL == 1 ? 1 : NPL / 2;
  const int b = blockIdx.y, lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) occTicket[b] = 0u;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU), S = T + U - 1;
  const int d0 = (blockIdx.x * kFactorWarps + (threadIdx.x >> 5)) * kFactorRows, u0 = NPL * lane;
  if (T <= 0 || U <= 0 || d0 >= S || u0 >= U) return;
  const float* al = alphas + (i64)b * stride;
  const float* dl = deltas + (i64)b * ((nDiag + kDiag - 1) / kDiag);
  const int uNext = min(u0 + NPL, ld - 1);   // (position 127 has no label arc)
  float a[kFactorRows + 1][NPL], aN[kFactorRows + 1];
  float4 f[kFactorRows][kPieces];
#pragma unroll
  for (int i = 0; i <= kFactorRows; ++i) {
    const i64 row = (i64)min(d0 + i, S - 1) * ld;
    load_row<NPL>(al + row + u0, a[i]);
    aN[i] = al[row + uNext];
    if (i < kFactorRows) {
      const float2* ar = arcs + (i64)b * stride + row;
#pragma unroll
      for (int q = 0; q < kPieces; ++q) {
        if constexpr (NPL == 1) {
          const float2 x = ar[lane];
          f[i][q] = make_float4(x.x, x.y, 0.0f, 0.0f);
        } else {
          f[i][q] = reinterpret_cast<const float4*>(ar)[q * 32 + lane];
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kFactorRows; ++i) {
    const int d = d0 + i;
    if (d >= S) break;
    // the successors' diagonal opens a block: the carried sums were lowered by its delta
    const float dlt = ((d + 1) % kDiag == 0 && d + 1 < S) ? dl[(d + 1) / kDiag] : 0.0f;
    float x[NPL], y[NPL];
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
      const int u = u0 + r, t = d - u;
      const bool valid = u < U && t >= 0 && t < T;
      const float4 q = f[i][r / 2];
      const float ax = r % 2 ? q.z : q.x, ay = r % 2 ? q.w : q.y;
      x[r] = (valid && t < T - 1) ? ex2_approx(((a[i][r] + ax) - dlt) - a[i + 1][r]) : 0.0f;
      if (t == T - 1 && u == U - 1) x[r] = 1.0f;   // terminating blank, fed by g(T,U-1) := 1
      const float art = r < NPL - 1 ? a[i + 1][(r + 1) % NPL] : aN[i + 1];
      y[r] = (valid && u < U - 1) ? ex2_approx(((a[i][r] + ay) - dlt) - art) : 0.0f;
    }
    float2* out = F + (i64)b * stride + (i64)d * ld;
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
      if constexpr (NPL == 1) out[lane] = make_float2(x[0], y[0]);
      else reinterpret_cast<float4*>(out)[q * 32 + lane] = make_float4(x[(2 * q) % NPL], y[(2 * q) % NPL], x[(2 * q + 1) % NPL], y[(2 * q + 1) % NPL]);
    }
  }
}

// The recursion on the prepared factors: g of the diagonals S (the node beyond the terminating
// blank) down to 0.
template <int NPL>
__global__ void __launch_bounds__(32) gamma_sweep_kernel(
    const float2* __restrict__ F, float* __restrict__ g, i64 stride, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int maxT, int maxU) {
  constexpr int ld = 32 * NPL;
  extern __shared__ __align__(128) uint8_t smemG[];
  const int b = blockIdx.x, lane = threadIdx.x;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (T <= 0 || U <= 0) return;
  const int S = T + U - 1, nBlocks = (S + kDiag - 1) / kDiag, u0 = NPL * lane;
  PairRing<NPL> ring(smemG, F + (i64)b * stride, lane, U, 0u);
  // block k holds the rows [max(S - 16(k+1), 0), S - 16k)
  auto issue = [&](int k) {
    const int lo = max(S - kDiag * (k + 1), 0);
    ring.issue(k % kRing, lo, k < nBlocks ? S - kDiag * k - lo : 0);
  };
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) issue(k);
  float* out0 = g + (i64)b * stride + u0;
  float s[NPL];
#pragma unroll
  for (int r = 0; r < NPL; ++r) s[r] = (u0 + r == U - 1) ? 1.0f : 0.0f;
  if (ring.act) store_row<NPL>(out0 + (i64)S * ld, s);
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
      if (ring.act) store_row<NPL>(out + i * ld, s);
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
  const float* ebl;          // [B,maxT] blank emissions (with ELrow)
  float2* arcs;
  const int* labels;
  const int* inLens;
  const int* labLens;
  int maxT, maxU, V, blank, npl, ld, extra;
  i64 stride;
};

// One CTA per 32x32 (t,u) tile: the log-probabilities (log2 units) of the two arcs leaving every
// node, written along the diagonals,
//   (E[t,blank]   + P[u,blank]   - LN[t,u]) * log2(e)
//   (E[t,label_u] + P[u,label_u] - LN[t,u]) * log2(e),  u < U-1
// The tiles beyond both ends of the time axis (`extra` of them on each side) write the "no such
// arc" of nodes outside the lattice, so that the array needs no fill.  Log-normalisers marked by
// the tensor-core kernel (NaN) are recomputed exactly first.
// Bound by memory: reads 8 and writes 8 bytes per node.
template <typename TIn>
__global__ void __launch_bounds__(256) sweep_prep_kernel(const PrepParams p) {
  __shared__ float tLn[32][33], tEl[32][33], tEb[32];
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
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int tt = w * 4 + k, t = t0 + tt;
      float a = (t < T && u < U) ? va[k] : 0.0f;
      unsigned todo = __ballot_sync(0xffffffffu, a != a);
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const TIn* er = e + (i64)t * p.V;
        const TIn* pr = pr0 + (i64)(u0 + src) * p.V;
        float m = neg_inf();
        for (int v = lane; v < p.V; v += 32) m = fmaxf(m, to_f32(er[v]) + to_f32(pr[v]));
        m = warp_max(m);
        float s = 0.0f;
        if (m != neg_inf() && m != pos_inf())
          for (int v = lane; v < p.V; v += 32) s += expf((to_f32(er[v]) + to_f32(pr[v])) - m);
        s = warp_sum(s);
        if (lane == src) {
          a = logf(s) + m;
          ln[(i64)t * p.maxU + u] = a;
        }
      }
      tLn[tt][lane] = a;
      if (elr) tEl[lane][tt] = vc[k];   // loaded with lane <-> frame, row <-> label position
      else tEl[tt][lane] = vc[k];
    }
  }
  __syncthreads();
  for (int ds = w; ds < 63; ds += 8) {
    const int tt = ds - lane, t = t0 + tt, d = t0 + u0 + ds;
    if (tt < 0 || tt > 31 || d < 0 || d >= S || u >= Uw) continue;
    float2 f = make_float2(__uint_as_float(kNoArcBits), __uint_as_float(kNoArcBits));
    if (t >= 0 && t < T && u < U) {
      const float lnv = tLn[tt][lane];
      f.x = ((tEb[tt] + pbl) - lnv) * kLog2e;
      if (u < U - 1) f.y = ((tEl[tt][lane] + plab) - lnv) * kLog2e;
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

// One CTA per 32 frames of one utterance, the (up to four) 32x32 lattice tiles of the label axis
// side by side.  With delta_b the upstream gradient:
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
constexpr int kOccThreads = 4 * 32 * kOccWarps;
constexpr int kOccRows = 32 / kOccWarps;  // frames (diagonals of the tile) per warp
template <bool TC>
__global__ void __launch_bounds__(kOccThreads, 2) occupancy_kernel(const OccParams p) {
  __shared__ float tS[4][32][33], tE[4][32][33];
  __shared__ float sRow[4][32], sCol[kOccWarps][2][128];
  __shared__ int sLast;
  const int b = blockIdx.y, t0 = blockIdx.x * 32;
  const int T = min(p.inLens[b], p.maxT), U = min(p.labLens[b] + 1, p.maxU);
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % kOccWarps, ub = threadIdx.x / (32 * kOccWarps);
  const int ld = 32 * p.npl;
  const float delta = (TC && p.deltas) ? p.deltas[b] : 1.0f;
  const bool some = T > 0 && U > 0 && t0 < T;
  float* part = p.partial + ((i64)b * gridDim.x + blockIdx.x) * 2 * p.maxU;
  const int u0 = ub * 32, u = u0 + lane;
  const bool inRange = u0 < p.ldW;
  const bool live = inRange && some && u0 < U;
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
    // Lane `lane` of local warp w holds the tile's diagonals ds = w + kOccWarps i with
    // 0 <= ds - lane < 32: exactly kOccRows of them, taken four at a time with all their loads
    // issued before the first use (unconditional, clamped into the lattice).
    const int first = w + (lane > w ? (lane - w + kOccWarps - 1) / kOccWarps * kOccWarps : 0) - lane;
    const int un = min(u + 1, U - 1);
#pragma unroll
    for (int q = 0; q < kOccRows; q += 4) {
      float2 f[4];
      float g1[4], g2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const i64 row = (i64)(min(t0 + first + kOccWarps * (q + j), T - 1) + uc) * ld;
        f[j] = F[row];
        g1[j] = g[row + ld + uc];
        g2[j] = g[row + ld + un];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int tt = first + kOccWarps * (q + j);
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
  float colS = 0.0f, colE = 0.0f;   // sums over the warp's frames
#pragma unroll
  for (int k = 0; k < kOccRows; ++k) {
    const int tt = w * kOccRows + k, t = t0 + tt;
    const float st = live ? tS[ub][tt][lane] : 0.0f, sp = live ? tE[ub][tt][lane] : 0.0f;
    colS += st;
    colE += sp;
    if (inRange) {
      if (t < p.maxT) {
        // (beyond T_b and U_b both occupancies are zero, and so is W)
        float x = 0.0f;
        if (live && t < T && u < U) x = __fadd_rn(st, sp) * shift[k] * delta;
        if (TC) x = tf32_round(x);
        p.W[((i64)b * p.maxT + t) * p.ldW + u] = x;
      }
      if (TC) {  // transposed: lane <-> frame, row <-> label position
        const int uu = u0 + tt, t2 = t0 + lane;
        if (uu < p.maxU && t2 < p.ldT) p.emT[((i64)b * p.maxU + uu) * p.ldT + t2] = live ? tE[ub][lane][tt] * delta : 0.0f;
      } else if (t < p.maxT && u < p.maxU) {
        p.emT[((i64)b * p.maxT + t) * p.maxU + u] = sp;
      }
    }
    float v = st;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sRow[ub][tt] = v;
  }
  sCol[w][0][u] = colS;
  sCol[w][1][u] = colE;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int t = t0 + lane;
    const bool ok = some && t < T;
    const float rs = ((sRow[0][lane] + sRow[1][lane]) + sRow[2][lane]) + sRow[3][lane];
    if (TC) {
      if (t < p.ldT) {
        p.nref[(i64)b * p.ldT + t] = ok ? -p.rowRef[(i64)b * p.maxT + t] * kLog2e : 0.0f;
        p.ebl[(i64)b * p.ldT + t] = ok ? rs * delta : 0.0f;
      }
    } else if (t < p.maxT) {
      p.ebl[(i64)b * p.maxT + t] = ok ? rs : 0.0f;
    }
  }
  const int cw = threadIdx.x >> 7, cu = threadIdx.x & 127;
  if (some && cw < 2 && cu < p.maxU) {
    float s = sCol[0][cw][cu];
#pragma unroll
    for (int k = 1; k < kOccWarps; ++k) s += sCol[k][cw][cu];
    part[cw * p.maxU + cu] = s;
  }
  // the CTA of the utterance that finishes last adds the partial sums
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    sLast = atomicAdd(&p.ticket[b], 1u) == gridDim.x - 1 ? 1 : 0;
  }
  __syncthreads();
  if (!sLast) return;
  __threadfence();
  const int tiles = (T > 0 && U > 0) ? (T + 31) / 32 : 0;
  float* acc = &tS[0][0][0];     // [4][2 * 128] sums of the four quarters of the tiles
  const float* all = p.partial + (i64)b * gridDim.x * 2 * p.maxU;
  for (int i = threadIdx.x; i < 4 * 2 * p.maxU; i += kOccThreads) {
    const int q = i / (2 * p.maxU), c = i - q * 2 * p.maxU;
    const int z0 = tiles * q / 4, z1 = tiles * (q + 1) / 4;
    float s = 0.0f;
#pragma unroll 8
    for (int z = z0; z < z1; ++z) s += __ldcg(all + (i64)z * 2 * p.maxU + c);
    acc[q * 256 + c] = s;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * p.maxU; c += kOccThreads) {
    const int cu2 = c < p.maxU ? c : c - p.maxU;
    const float s = cu2 < U ? ((acc[c] + acc[256 + c]) + acc[512 + c]) + acc[768 + c] : 0.0f;
    (c < p.maxU ? p.pBlank : p.pLabel)[(i64)b * p.maxU + cu2] = s;
  }
}

template <typename K>
void allow_dyn_smem(K kernel, int bytes) {
  TB200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

}  // namespace

bool sweep_supported(Dims d) { return d.maxU >= 1 && d.maxU <= 128; }

SweepGeom sweep_geom(Dims d) {
  SweepGeom g;
  g.npl = d.maxU <= 32 ? 1 : d.maxU <= 64 ? 2 : 4;
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

void launch_sweep_forward(const void* E, const void* P, float* LN, const float* ELrow,
                          const float* ebl, float2* arcs, float* alphas, float* deltas, float* costs,
                          float* lossSum, unsigned* ticket, const int* labels, const int* inLens,
                          const int* labLens, SweepGeom g, Dims d, cudaStream_t stream) {
  if (d.B <= 0) return;
  if (d.maxT > 0) {
    PrepParams q{};
    q.E = E; q.P = P; q.LN = LN; q.ELrow = ELrow; q.ebl = ebl; q.arcs = arcs;
    q.labels = labels; q.inLens = inLens; q.labLens = labLens;
    q.maxT = d.maxT; q.maxU = d.maxU; q.V = d.V; q.blank = d.blank; q.npl = g.npl; q.ld = g.ld;
    q.extra = div_up(d.maxU, 32); q.stride = g.stride;
    const dim3 grid(div_up(d.maxU, 32), div_up(d.maxT, 32) + 2 * q.extra, d.B);
    ScopedKernel sk("sweep_prep", stream);
    if (d.dtype == kDtypeBf16) sweep_prep_kernel<bf16><<<grid, 256, 0, stream>>>(q);
    else sweep_prep_kernel<float><<<grid, 256, 0, stream>>>(q);
    TB200_CHECK_LAUNCH();
  }
  const int smem = kRing * kDiag * g.ld * 8;
  ScopedKernel sk("alpha_sweep", stream);
#define CALL(NPL)                                                                                \
  allow_dyn_smem(alpha_sweep_kernel<NPL>, smem);                                                 \
  alpha_sweep_kernel<NPL><<<d.B, 32, smem, stream>>>(arcs, costs, alphas, deltas, g.stride,      \
                                                     g.nDiag, inLens, labLens, d.B, d.maxT,      \
                                                     d.maxU, lossSum, ticket)
  TB200_BY_NPL(g.npl, CALL);
#undef CALL
  TB200_CHECK_LAUNCH();
}

void launch_sweep_backward(const SweepScratch& w, const float2* arcs, const float* alphas,
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
      arcs, alphas, alphaDeltas, w.F, w.ticket, g.stride, g.nDiag, inLens, labLens, d.maxT, d.maxU)
    TB200_BY_NPL(g.npl, CALL);
#undef CALL
    TB200_CHECK_LAUNCH();
  }
  {
    const int smem = kRing * kDiag * g.ld * 8;
    ScopedKernel sk("gamma_sweep", stream);
#define CALL(NPL)                                                                              \
  allow_dyn_smem(gamma_sweep_kernel<NPL>, smem);                                               \
  gamma_sweep_kernel<NPL><<<d.B, 32, smem, stream>>>(w.F, w.g, g.stride, inLens, labLens, d.maxT, d.maxU)
    TB200_BY_NPL(g.npl, CALL);
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
  if (tensorCore) occupancy_kernel<true><<<grid, kOccThreads, 0, stream>>>(o);
  else occupancy_kernel<false><<<grid, kOccThreads, 0, stream>>>(o);
  TB200_CHECK_LAUNCH();
}

}  // namespace tb200
