// Log-normalisers as an exp-factored tensor-core contraction on fp16 pairs (tcgen05 / TMEM / TMA).
//
//   LN[b,t,u] = log( sum_v exp(E[b,t,v]-ref[b,t]) * exp(P[b,u,v]-maxP[b,u]) ) + ref[b,t] + maxP[b,u]
//
// (transducer/torch_binding.py:35-40: row maxima, exp, bmm, log) in one pass over E, as
// lognorm_umma.cu does with TF32 pairs.  There a product of two fp32 numbers is three kind::tf32
// MMAs; here every factor is hi + lo with both halves fp16 (round-to-nearest: 22 bits, and the dropped
// lo * lo is at most 2^-22 of the product too, of either sign) and the three products are kind::f16 MMAs, which take half the time for
// half the operand bytes.  Distance to float64 of the two, N(0,1..2) scores over 64..8000 words: rms
// 3e-7..5e-7 here, 1.5e-6 there (half as many truncating accumulation steps besides).  What fp16 lacks is
// range, so
//   * each frame's 64 words of a stage are scaled by a power of two of their own (their largest
//     becomes 2^14..2^15) and the accumulator holds one stage only: the drain warps undo the scale when
//     they add the stage's 128 x N products to the running fp32 sums, one FMA where an
//     addition was;
//   * exp(P - maxP) is scaled by 2^15;
//   * a factor further below its scale than 2^-40 is lost.  The error this leaves in a sum S(t,u) is at
//     most 2^-40 (sum_v exp(E) + max_v exp(E) * sum_v exp(P)), all of them relative to the same
//     references; both sums over v are formed on the way, and a tile with a node where that
//     exceeds 2^-20 S, or whose S leaves [1e-30, 1e30], is marked.  Marked tiles are recomputed by the
//     TF32 kernel behind this one (which returns at once when there are none).  N(0, 2) scores
//     over 10000 words stay clear of that, as do words 6 above the rest; a frame and a position
//     that each have one word 10 above all others, not the same one, do not.  Where a sample of the
//     nodes says so, the TF32 kernel has the whole call to itself (see spread_vote).
//
// Work item: 128 frames of one utterance (UMMA M=128) x up to 160 label positions (longer axes: two
// column ranges) x the whole vocabulary in stages of 64 words.  Roles inside a CTA (one per SM):
//   warps 0-11   operand transform, one group of four per stage of the ring.  Thread r of
//                a group owns frame r of the tile (= TMEM lane r): raw row from shared memory,
//                exponentials, scale, hi / lo packed in pairs into TENSOR MEMORY (A operand: 64 columns
//                a stage), 32 words at a time.  It also hands out E[t,label_u] and E[t,blank].
//   next 4 x ND  accumulator drain + epilogue, DCOLS accumulator columns each.
//   then         a TMA producer for E and one for exp(P) (an E stage is free once it is in registers, an
//                exp(P) stage only after its MMAs), two MMA issuers, one per accumulator, twelve MMAs a
//                stage.
// What bounds it (cycle stamps of every role, B = 32, T = 1750, U' = 101, V = 10000): the roles' own work per
// word, not the tensor pipe and not the copies.  With stages of 32 words and two transform groups a
// group was busy 2200 of every 2600 cycles it had for a stage; with three groups the drain warps, which need
// ~1400 cycles from one accumulator to the next whatever it holds, were.  Hence 64 words a
// stage: half as many drains, barriers and commits per word.  Measured, this kernel / the TF32 kernel, us:
// B = 32, T = 1500..2000, U' = 61..101, V = 10000 680 / 834 (bf16 emissions 626 / 785), B = 64, T = 750..1500,
// U' = 76..151, V = 4096 376 / 723, B = 64, T = 500..1000, U' = 101..201, V = 32000 2790 / 3620.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.h"
#include "lognorm_items.cuh"
#include "profile.h"
#include "sm100.cuh"

namespace tb200 {
namespace {

using namespace sm100;
using namespace lognorm;

constexpr int kStages = 3;           // of the ring; one transform group each
constexpr int kStageK = 64;          // words of a stage
constexpr int kScaleBits = 15;       // both operands' largest entries are brought to 2^15
constexpr int kScaleSlots = 8;       // stages whose scales are kept (the ring and five)
constexpr float kSpread = 9.5367431640625e-7f;   // 2^-20: a node's sum must reach this share of the bound's two
constexpr int kMinExp = -96, kMaxExp = 110;   // of a stage's largest exponential
// raw E of a stage: two boxes of 32 fp32 words or one of 64 bf16 words, rows of 128 bytes
__host__ __device__ constexpr int stage_raw_bytes(bool bf) { return kTileM * kStageK * (bf ? 2 : 4); }

// words 16 w .. 16 w + 15 of frame r's 64 words, as fp32; and one of them
template <bool BF>
__device__ __forceinline__ void stage_words16(const uint8_t* raw, int r, int w, float (&x)[16]) {
  if constexpr (BF) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint4 q = *reinterpret_cast<const uint4*>(raw + r * 128 + (((2 * w + j) ^ (r & 7)) << 4));
      const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        x[8 * j + 2 * k] = __uint_as_float(v[k] << 16);
        x[8 * j + 2 * k + 1] = __uint_as_float(v[k] & 0xffff0000u);
      }
    }
  } else {
    load_words16<false>(raw + (w >> 1) * raw_bytes(false) + r * 128, r, w & 1, x);
  }
}
template <bool BF>
__device__ __forceinline__ float stage_word(const uint8_t* raw, int r, int off) {
  if constexpr (BF) {
    const unsigned short h = *reinterpret_cast<const unsigned short*>(
        raw + r * 128 + (((off >> 3) ^ (r & 7)) << 4) + (off & 7) * 2);
    return __uint_as_float((uint32_t)h << 16);
  } else {
    return load_word<false>(raw + (off >> 5) * raw_bytes(false) + r * 128, r, off & 31);
  }
}

// Two fp32 numbers in a 64-bit register: each element rounded as by itself, one instruction for both.
__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
  float2 c;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(c.x), "=f"(c.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return c;
}

// hi + lo of two numbers, packed in pairs (first number in the low half)
__device__ __forceinline__ void split_f16(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 d = fma_pair(__half22float2(h), make_float2(-1.0f, -1.0f), make_float2(a, b));
  const __half2 l = __floats2half2_rn(d.x, d.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// ---------------------------------------------------------------------------------
// Would most tiles be marked?  A frame and a position of a sharp model each have one word far above their others, mostly
// not the same one, and then nearly every tile holds a node that fails, for a share of its nodes that is
// small at first: with one random word per frame and one per position raised by g over N(0,1), 4096 words, 0 of 8
// tiles at g = 9, some at 10, all at 11, for 0.1 % of the nodes.  Both kernels would run, so a few hundred nodes
// spread over the batch are looked at first, in fp32, against a bound eight times as high: 0.1 % of them fail it at
// g = 9, 2 % at 10, 9 % at 11.  One CTA a node, two rows read.  They are the first CTAs of the launch that brings P
// to pairs, whose others stop as soon as the votes are there (nobody reads the pairs then).
// ---------------------------------------------------------------------------------
template <typename TIn>
__device__ __noinline__ void spread_vote(
    const TIn* __restrict__ E, const TIn* __restrict__ P, const int* __restrict__ inLens,
    const int* __restrict__ labLens, unsigned i, int B, int maxT, int maxU, int V, int* __restrict__ marks) {
  __shared__ float red[32][5];
  const int warps = blockDim.x >> 5;
  const int b = (int)(i % (unsigned)B);
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (T <= 0 || U <= 0) return;
  // node i / B of the utterance: two sequences that fill [0, 1) evenly (multiples of the golden ratio, of sqrt 2)
  const unsigned k = i / (unsigned)B + 1u;
  const int t = (int)__umulhi((k + 7u * (unsigned)b) * 2654435769u, (unsigned)T);
  const int u = (int)__umulhi((k + 5u * (unsigned)b) * 1779033704u, (unsigned)U);
  const TIn* e = E + ((i64)b * maxT + t) * V;
  const TIn* p = P + ((i64)b * maxU + u) * V;
  // sums relative to the largest words so far (in units of log2; words masked below that count for nothing)
  float mE = -1e30f, mP = -1e30f, s = 0.0f, sE = 0.0f, sP = 0.0f;
  auto rescale = [&](float toE, float toP) {
    const float fE = ex2_approx(mE - toE), fP = ex2_approx(mP - toP);
    sE *= fE;
    sP *= fP;
    s *= fE * fP;
    mE = toE;
    mP = toP;
  };
#pragma unroll 4
  for (int v = 4 * threadIdx.x; v < V; v += 4 * blockDim.x) {   // (V % 4 == 0)
    const float4 x4 = ld4(e + v), y4 = ld4(p + v);
    const float x[4] = {x4.x, x4.y, x4.z, x4.w}, y[4] = {y4.x, y4.y, y4.z, y4.w};
    rescale(fmaxf(mE, fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])) * kLog2e),
            fmaxf(mP, fmaxf(fmaxf(y[0], y[1]), fmaxf(y[2], y[3])) * kLog2e));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = ex2_approx(fmaf(x[j], kLog2e, -mE)), c = ex2_approx(fmaf(y[j], kLog2e, -mP));
      sE += a;
      sP += c;
      s = fmaf(a, c, s);
    }
  }
  rescale(warp_max(mE), warp_max(mP));
  s = warp_sum(s);
  sE = warp_sum(sE);
  sP = warp_sum(sP);
  if ((threadIdx.x & 31) == 0) {
    float* mine = red[threadIdx.x >> 5];
    mine[0] = mE; mine[1] = mP; mine[2] = sE; mine[3] = sP; mine[4] = s;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const float* mine = red[min((int)threadIdx.x, warps - 1)];
  const bool one = (int)threadIdx.x < warps;
  mE = mine[0]; mP = mine[1]; sE = one ? mine[2] : 0.0f; sP = one ? mine[3] : 0.0f; s = one ? mine[4] : 0.0f;
  rescale(warp_max(mE), warp_max(mP));
  s = warp_sum(s);
  sE = warp_sum(sE);
  sP = warp_sum(sP);
  // (no votes from rows without a word and from NaN: their tiles are marked in any case)
  if (threadIdx.x == 0 && sE > 0.0f && sP > 0.0f && s < 8.0f * kSpread * (sE + sP)) atomicAdd(&marks[kMarkVotes], 1);
}

// ---------------------------------------------------------------------------------
// exp(P - maxP) * 2^15 as rows of [B][nPad][stage][hi 64 | lo 64] halves, zero beyond V; maxP and
// the rows' sums of exp(P - maxP).  Bound by memory: one read (the second comes from L2), one write.
// ---------------------------------------------------------------------------------
// The first `samples` CTAs vote (see spread_vote), in rows of the grid of their own: with one row for all CTAs, and
// a division in each, the launch took 3 % longer.
template <typename TIn>
__global__ void __launch_bounds__(1024) expp_f16_kernel(
    const TIn* __restrict__ E, const TIn* __restrict__ P, uint8_t* __restrict__ out, float* __restrict__ maxP,
    float* __restrict__ sumP, const int* __restrict__ inLens, const int* __restrict__ labLens, int samples, int B,
    int maxT, int maxU, int V, int nPad, int kPad, int* marks) {
  __shared__ float red[32], redS[32];
  const int voteRows = (samples + maxU - 1) / maxU;
  if ((int)blockIdx.y < voteRows) {
    const int i = blockIdx.y * maxU + blockIdx.x;
    if (i < samples) spread_vote(E, P, inLens, labLens, i, B, maxT, maxU, V, marks);
    return;
  }
  const int b = (int)blockIdx.y - voteRows, u = blockIdx.x;
  // (an old number from L1 will do: if not this CTA, a later one sees them)
  const int votes = samples > 0 ? marks[kMarkVotes] : 0;
  const int U = min(labLens[b] + 1, maxU);
  if (u >= U) {
    // (rows beyond the utterance's label axis only feed accumulator columns that nobody reads)
    if (u < maxU && threadIdx.x == 0) maxP[(i64)b * maxU + u] = 0.0f;
    return;
  }
  const TIn* p = P + ((i64)b * maxU + u) * V;
  uint8_t* row = out + ((i64)b * nPad + u) * kPad * 4;
  float m = neg_inf();
  if (votes < kVotes)
    for (int v = threadIdx.x; v < V / 4; v += blockDim.x) {
      const float4 x = ld4(p + 4 * v);
      m = fmaxf(fmaxf(m, fmaxf(x.x, x.y)), fmaxf(x.z, x.w));
    }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  if (__syncthreads_or(votes >= kVotes)) return;
  m = red[0];
  for (int k = 1; k < (int)blockDim.x / 32; ++k) m = fmaxf(m, red[k]);
  float s = 0.0f;
  for (int v = threadIdx.x; v < kPad / 4; v += blockDim.x) {
    float xs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (4 * v < V) {
      const float4 x = ld4(p + 4 * v);
      xs[0] = expf(x.x - m); xs[1] = expf(x.y - m); xs[2] = expf(x.z - m); xs[3] = expf(x.w - m);
      s += (xs[0] + xs[1]) + (xs[2] + xs[3]);
    }
    uint2 hi, lo;
    constexpr float kUp = (float)(1 << kScaleBits);
    split_f16(xs[0] * kUp, xs[1] * kUp, hi.x, lo.x);
    split_f16(xs[2] * kUp, xs[3] * kUp, hi.y, lo.y);
    uint8_t* at = row + (v >> 4) * 256 + (v & 15) * 8;   // 16 float4 of the input per stage
    *reinterpret_cast<uint2*>(at) = hi;
    *reinterpret_cast<uint2*>(at + 128) = lo;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) redS[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)blockDim.x / 32; ++k) s += redS[k];
    maxP[(i64)b * maxU + u] = m;
    sumP[(i64)b * maxU + u] = s;
  }
}

// ---------------------------------------------------------------------------------
// main kernel
// ---------------------------------------------------------------------------------
struct F16Params {
  float* LN;
  float* rowRef;
  const float* maxP;
  const float* sumP;
  const int* inLens;
  const int* labLens;
  int* status;
  int maxT, maxU, V, tmemCols;
  int nPad, halves;      // label positions per column range, ranges
  int B, tilesX, nSM;
  float* partial;        // [nSM][kTileM][nPad] partial sums of split tiles
  float* rowSums;        // [nSM][2][kTileM] their sums and maxima of exp(E)
  unsigned* tickets;     // [nSM] parts finished per split tile (zero on entry, zero again on exit)
  int* marks;            // (see kMarkAny)
  const int* labels;     // label / blank emissions handed out (null: not wanted), see hand_out
  float* EL;
  float* ebl;
  int blank;
};

template <int ND, int DCOLS, bool BF>
__global__ void __launch_bounds__((4 * kStages + 4 * ND + 4) * 32, 1) lognorm_f16_kernel(
    const __grid_constant__ CUtensorMap tmE, const __grid_constant__ CUtensorMap tmP,
    const F16Params p) {
  static_assert(DCOLS % 8 == 0, "columns move in eights");
  constexpr int kDrainWarp0 = 4 * kStages, kLoadE = kDrainWarp0 + 4 * ND, kLoadP = kLoadE + 1, kMmaWarp = kLoadP + 1;
  constexpr int kRaw = stage_raw_bytes(BF);
  const bool none = all_marked(p.marks);   // (looked at behind the lengths)
  const LnItem it = ln_item(p.inLens, p.labLens, p.maxT, p.maxU, p.V, p.B, p.tilesX, p.halves, p.nPad, p.nSM);
  if (it.b < 0 || none) return;
  const int b = it.b, T = it.T, U = it.U, t0 = it.t0, uOff = it.uOff;
  const int part = it.part, parts = it.parts, splitIdx = it.split;

  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) &
                                             ~uintptr_t(1023));
  const int pBytes = p.nPad * 256;
  uint8_t* smemP = smem + kStages * kRaw;
  __shared__ uint64_t barEFull[kStages], barEFree[kStages], barPFull[kStages], barDone[kStages];
  __shared__ uint64_t barReady[kStages][2];
  __shared__ uint64_t barAccFull[2], barAccEmpty[2], barRef, barEnd;
  __shared__ uint32_t tmemBase;
  __shared__ int abortFlag, sLast;
  __shared__ float sMaxP[160], sSumP[160];
  __shared__ float sRef[kTileM], sSumE[kStages][kTileM], sMaxE[kStages][kTileM];
  __shared__ signed char sExp[kScaleSlots][kTileM];   // stage c's scale exponents in slot c % kScaleSlots
  __shared__ int sKey[kMaxLabels];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this part's stages of the vocabulary [cBegin, cEnd); iteration i of the pipeline handles firstWord(i)
  const int nAll = (p.V + kStageK - 1) / kStageK;
  const int cBegin = (int)((i64)part * nAll / parts), cEnd = (int)((i64)(part + 1) * nAll / parts);
  const bool refFirst = part > 0;  // iteration 0 fetches the first words for the frames' shifts only
  const int n = cEnd - cBegin + (refFirst ? 1 : 0);
  auto firstWord = [&](int i) { return (refFirst ? (i == 0 ? 0 : cBegin + i - 1) : cBegin + i) * kStageK; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&barEFull[s], 1);
      mbar_init(&barEFree[s], 4);   // the stage's transform group
      mbar_init(&barPFull[s], 1);
      mbar_init(&barReady[s][0], 4);
      mbar_init(&barReady[s][1], 4);
      mbar_init(&barDone[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&barAccFull[a], 2);   // the MMAs, and the issuer for the scales it has seen arrive
      mbar_init(&barAccEmpty[a], 4 * ND);
    }
    mbar_init(&barRef, 4);
    mbar_init(&barEnd, 4 * kStages);
    abortFlag = 0;
    fence_mbar_init();
  }
  for (int u = threadIdx.x; u < p.nPad; u += blockDim.x) {
    sMaxP[u] = (uOff + u < U) ? p.maxP[(i64)b * p.maxU + uOff + u] : 0.0f;
    sSumP[u] = (uOff + u < U) ? p.sumP[(i64)b * p.maxU + uOff + u] : 0.0f;
  }
  const bool gather = p.EL != nullptr && uOff == 0;   // (one range hands out the emissions)
  const int nLab = gather ? min(U - 1, kMaxLabels) : 0;
  if (gather) {
    __shared__ int sLab[kMaxLabels];
    sort_labels(p.labels + (i64)b * (p.maxU - 1), nLab, sLab, sKey);
  }
  if (warp == kMmaWarp) {
    tmem_alloc(&tmemBase, (uint32_t)p.tmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tBase = tmemBase;                       // two accumulators of nPad columns
  const uint32_t tA = tBase + (uint32_t)(2 * p.nPad);    // operand stages: 64 columns, [hi 16 | lo 16] per 32 words
  volatile int* abortp = &abortFlag;

  if (warp == kLoadE || warp == kLoadP) {
    // ---------------- TMA producers ----------------
    const bool isE = warp == kLoadE;
    if (lane == 0) {
      uint64_t* full = isE ? barEFull : barPFull;
      uint64_t* free = isE ? barEFree : barDone;
      const CUtensorMap* tm = isE ? &tmE : &tmP;
      tma_prefetch_desc(tm);
      uint8_t* st = isE ? smem : smemP;
      const uint32_t bytes = isE ? kRaw : (uint32_t)pBytes;
      int issued = 0, s = 0;
      uint32_t ph = 1;  // phase of the PREVIOUS release of the stage
      for (int c = 0; c < n; ++c) {
        if (c >= kStages && !mbar_wait(&free[s], ph, abortp, p.status, kStatusTimeoutStageFree)) break;
        mbar_arrive_expect_tx(&full[s], bytes);
        const int w0 = firstWord(c);
        uint8_t* dst = st + (size_t)s * bytes;
        if (isE) {
          tma_load_3d(dst, tm, &full[s], w0, t0, b);
          if (!BF) tma_load_3d(dst + raw_bytes(false), tm, &full[s], w0 + kChunkK, t0, b);
        } else {
          tma_load_3d(dst, tm, &full[s], 2 * w0, uOff, b);
          tma_load_3d(dst + p.nPad * 128, tm, &full[s], 2 * w0 + kStageK, uOff, b);
        }
        issued = c + 1;
        if (++s == kStages) { s = 0; ph ^= 1u; }
      }
      if (*abortp) {
        // after an abort: give the copies still in flight a bounded time to land
        for (int c = max(0, issued - kStages); c < issued; ++c) {
          const unsigned long long t1 = global_timer_ns();
          while (!mbar_try_wait(&full[c % kStages], (c / kStages) & 1) &&
                 global_timer_ns() - t1 < 50000000ull) {
          }
        }
      }
    }
  } else if (warp >= kMmaWarp) {
    // ---------------- MMA issuers: issuer m takes the stages c with c % 2 == m, into accumulator m ----------------
    // (Stage c + 3 has the other issuer and the same ring slot as stage c.  Its issuer cannot mistake the
    // slot's earlier phases for its own: it waits for the drain of c + 1 first, which follows that of c.)
    const int m = warp - kMmaWarp;
    if (lane == 0) {
      const uint32_t idesc = idesc_f16(kTileM, p.nPad);
      const uint64_t descP = smem_desc_sw128(smem_u32(smemP), 16, 1024);
      const uint32_t dAcc = tBase + (uint32_t)(m * p.nPad), loRows = (uint32_t)(p.nPad * 128) >> 4;
      bool ok = true;
      int s = m;
      uint32_t ph = 0, aph = 1;   // phase of the ring slot; of the PREVIOUS drain of the accumulator
      for (int c = m; c < n; c += 2) {
        if (c >= 2) ok = mbar_wait(&barAccEmpty[m], aph, abortp, p.status, kStatusTimeoutStageFree);
        ok = ok && mbar_wait(&barPFull[s], ph, abortp, p.status, kStatusTimeoutTma);
        const uint64_t d0 = descP + (uint64_t)((uint32_t)(s * pBytes) >> 4);
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // 32 words each
          ok = ok && mbar_wait(&barReady[s][h], ph, abortp, p.status, kStatusTimeoutOperand);
          if (!ok) break;
          tc_fence_after();
          const uint32_t aHi = tA + (uint32_t)(s * 64 + h * 32), aLo = aHi + 16;
#pragma unroll
          for (int k = 0; k < 2; ++k) {   // 16 words a step: 8 columns of A, 32 bytes of a row of exp(P)
            const uint64_t dHi = d0 + h * 4 + k * 2, dLo = dHi + loRows;
            mma_f16_ts(dAcc, aHi + k * 8, dHi, idesc, (h | k) ? 1u : 0u);
            mma_f16_ts(dAcc, aLo + k * 8, dHi, idesc, 1u);
            mma_f16_ts(dAcc, aHi + k * 8, dLo, idesc, 1u);
          }
        }
        if (!ok) break;
        mma_commit(&barDone[s]);
        mma_commit(&barAccFull[m]);
        mbar_arrive(&barAccFull[m]);
        aph ^= 1u;
        s += 2;
        if (s >= kStages) { s -= kStages; ph ^= 1u; }
      }
    }
  } else if (warp < kDrainWarp0) {
    // ---------------- operand transform (thread = frame = TMEM lane) ----------------
    const int q = warp & 3, s = warp >> 2;      // lane quarter; my group's ring slot
    const int r = q * 32 + lane;                // frame within the tile, 0..127
    const uint32_t dst = tA + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * 64);
    const uint8_t* raw = smem + (size_t)s * kRaw;
    float shift = 0.0f, sumE = 0.0f, maxE = 0.0f;   // (shift: the frame's reference, an integer power of 2)
    bool ok = true;
    if (s > 0) {  // the frame's shift is found by group 0 in the first stage
      ok = mbar_wait(&barRef, 0, abortp, p.status, kStatusTimeoutOperand);
      ok = __all_sync(0xffffffffu, ok);
      shift = sRef[r];
    }
    int cur = 0;  // cursor into the sorted label list (see hand_out)
    int nextCol = (gather && nLab > 0) ? (sKey[0] >> 8) : 0x7fffffff;
    float* elCol = gather ? p.EL + (i64)b * p.maxU * p.maxT + t0 + r : nullptr;  // my frame
    float* eblAt = gather ? p.ebl + (i64)b * p.maxT + t0 + r : nullptr;
    uint32_t ph = 0;
    for (int c = s; c < n && ok; c += kStages, ph ^= 1u) {
      ok = mbar_wait(&barEFull[s], ph, abortp, p.status, kStatusTimeoutTma);
      ok = __all_sync(0xffffffffu, ok);  // keep the warp converged for the aligned TMEM ops
      if (!ok) break;
      const int w0 = firstWord(c);
      const bool refOnly = refFirst && c == 0;               // its terms belong to part 0
      const int left = refOnly ? 0 : p.V - w0;               // words of this stage that count
      // 16 words at a time; those beyond the vocabulary count for nothing
      auto words = [&](int w, float (&x)[16]) {
        stage_words16<BF>(raw, r, w, x);
        if (left < 16 * w + 16) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (16 * w + j >= left) x[j] = neg_inf();
        }
      };
      auto max16 = [](const float (&x)[16], float m) {
        float a = fmaxf(fmaxf(x[0], x[1]), x[2]), e = fmaxf(fmaxf(x[3], x[4]), x[5]);
        a = fmaxf(fmaxf(a, x[6]), x[7]);
        e = fmaxf(fmaxf(e, x[8]), x[9]);
        a = fmaxf(fmaxf(a, x[10]), x[11]);
        e = fmaxf(fmaxf(e, x[12]), x[13]);
        return fmaxf(fmaxf(fmaxf(a, e), fmaxf(x[14], x[15])), m);
      };
      if (c == 0) {
        // the frame's shift: maximum of the first 32 entries of the row (not of all of it, which
        // would cost a second pass over E)
        float x[16];
        stage_words16<BF>(raw, r, 0, x);
        float m = max16(x, neg_inf());
        stage_words16<BF>(raw, r, 1, x);
        m = max16(x, m);
        // a -inf/NaN prefix would poison every term; fall back to 0 and let the
        // range check route the row to the exact path if needed
        const float ref = (m > -3.0e38f && m < 3.0e38f) ? m : 0.0f;
        shift = rintf(ref * kLog2e);
        sRef[r] = shift;
        if (t0 + r < T && part == 0 && uOff == 0) p.rowRef[(i64)b * p.maxT + t0 + r] = ref;
      }
      if (gather && !refOnly)
        hand_out([&](int off) { return stage_word<BF>(raw, r, off); }, w0, kStageK, sKey, nLab, cur, nextCol,
                 elCol, p.maxT, p.blank, eblAt, t0 + r < T);
      // the stage's scale 2^(15 - R), R = the exponent of its largest exponential rounded up; it is
      // part of the exponentials' argument, which is rounded once (the shift is an integer)
      float x0[16], x1[16], top = neg_inf();
      words(2, x0);
      words(3, x1);
      top = max16(x1, max16(x0, top));
      words(0, x0);
      words(1, x1);
      top = fmaf(max16(x1, max16(x0, top)), kLog2e, -shift);
      const float R = ceilf(fminf(fmaxf(top, (float)kMinExp), (float)kMaxExp));
      const float pw = __int_as_float(((int)R + 127) << 23);
      maxE = fmaxf(maxE, pw);
      sExp[c % kScaleSlots][r] = (signed char)(int)R;
      const float2 mul = make_float2(kLog2e, kLog2e), add = make_float2((kScaleBits - R) - shift, (kScaleBits - R) - shift);
      float2 scaledSum = make_float2(0.0f, 0.0f);
      auto convert = [&](const float (&x)[16], uint32_t at) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 a = fma_pair(make_float2(x[2 * j], x[2 * j + 1]), mul, add);
          const float2 e = make_float2(ex2_approx(a.x), ex2_approx(a.y));
          scaledSum = add_pair(scaledSum, e);
          split_f16(e.x, e.y, hi[j], lo[j]);
        }
        tmem_st8(at, hi);
        tmem_st8(at + 16, lo);
      };
      // the slot's operand columns are free once the MMAs of stage c - 3 are done
      if (c >= kStages) {
        ok = mbar_wait(&barDone[s], ph ^ 1u, abortp, p.status, kStatusTimeoutMma);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
      }
      convert(x0, dst);
      words(2, x0);
      convert(x1, dst + 8);
      words(3, x1);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&barEFree[s]);   // (everything is in registers)
        mbar_arrive(&barReady[s][0]);
        if (c == 0) mbar_arrive(&barRef);
      }
      convert(x0, dst + 32);
      convert(x1, dst + 40);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&barReady[s][1]);
      sumE = fmaf(scaledSum.x + scaledSum.y, pw * (1.0f / (1 << kScaleBits)), sumE);
    }
    sSumE[s][r] = sumE;
    sMaxE[s][r] = maxE;
    __syncwarp();
    if (lane == 0) mbar_arrive(&barEnd);
  } else {
    // ---------------- accumulator drain + epilogue ----------------
    const int h = (warp - kDrainWarp0) >> 2;     // which column slice
    const int q = warp & 3;                      // TMEM lane quarter this warp may touch
    const int r = q * 32 + lane;
    const uint32_t laneAddr = (uint32_t)(q * 32) << 16;
    const int c0 = h * DCOLS, c1 = min(p.nPad, c0 + DCOLS);
    float sum[DCOLS];
#pragma unroll
    for (int j = 0; j < DCOLS; ++j) sum[j] = 0.0f;
    bool ok = true;
    for (int c = 0; c < n; ++c) {
      const int a = c & 1;
      ok = mbar_wait(&barAccFull[a], (c >> 1) & 1, abortp, p.status, kStatusTimeoutMma);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      // (exponents -126 .. 80: a normal number)
      const float down = __int_as_float(((int)sExp[c % kScaleSlots][r] - 2 * kScaleBits + 127) << 23);
      const uint32_t src = tBase + laneAddr + (uint32_t)(a * p.nPad + c0);
#pragma unroll
      for (int i = 0; i < DCOLS; i += 8) {   // (more columns in flight do not fit the registers)
        uint32_t v[8];
        if (c0 + i < c1) tmem_ld8(src + i, v);
        tmem_wait_ld();
        if (i + 8 >= DCOLS) {   // all read: the issuer may go on
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&barAccEmpty[a]);
        }
        if (c0 + i < c1) {
#pragma unroll
          for (int j = 0; j < 8; ++j) sum[i + j] = fmaf(__uint_as_float(v[j]), down, sum[i + j]);
        }
      }
    }
    if (ok) ok = mbar_wait(&barEnd, 0, abortp, p.status, kStatusTimeoutOperand);
    ok = __all_sync(0xffffffffu, ok);
    // A warp that gave up (ok == false; the cause is in the status word) turns its sums into
    // NaN: the tile is then marked instead of showing stale memory.
    const float bad = __int_as_float(0x7fc00000);
    if (!ok) {
#pragma unroll
      for (int j = 0; j < DCOLS; ++j) sum[j] = bad;
    }
    float sumE = 0.0f, maxE = 0.0f;
#pragma unroll
    for (int g = 0; g < kStages; ++g) {
      sumE += sSumE[g][r];
      maxE = fmaxf(maxE, sMaxE[g][r]);
    }
    bool writer = true;  // does this CTA write the tile's log-normalisers?
    if (parts > 1) {
      // split tile: park the partial sums; the part that finishes last adds all of them in
      // part order (so the result does not depend on which part that is) and goes on
      const int slot = splitIdx * parts + part;
      float* mine = p.partial + ((size_t)slot * kTileM + r) * p.nPad + c0;
#pragma unroll
      for (int j = 0; j < DCOLS; ++j)
        if (c0 + j < c1) mine[j] = sum[j];
      if (h == 0) {
        p.rowSums[(size_t)slot * 2 * kTileM + r] = sumE;
        p.rowSums[((size_t)slot * 2 + 1) * kTileM + r] = maxE;
      }
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(4 * ND * 32) : "memory");
      if (warp == kDrainWarp0 && lane == 0) {
        const unsigned done = atomicAdd(&p.tickets[splitIdx], 1u);
        sLast = (done == (unsigned)(parts - 1)) ? 1 : 0;
        if (sLast) p.tickets[splitIdx] = 0u;  // ready for the next launch
      }
      asm volatile("bar.sync 1, %0;" ::"n"(4 * ND * 32) : "memory");
      writer = sLast != 0;
      if (writer) {
        __threadfence();
#pragma unroll
        for (int j = 0; j < DCOLS; ++j) sum[j] = 0.0f;
        sumE = maxE = 0.0f;
        for (int z = 0; z < parts; ++z) {
          const int from = splitIdx * parts + z;
          const float* src = p.partial + ((size_t)from * kTileM + r) * p.nPad + c0;
#pragma unroll
          for (int j = 0; j < DCOLS; ++j)
            if (c0 + j < c1) sum[j] += __ldcg(src + j);
          sumE += __ldcg(p.rowSums + (size_t)from * 2 * kTileM + r);
          maxE = fmaxf(maxE, __ldcg(p.rowSums + ((size_t)from * 2 + 1) * kTileM + r));
        }
      }
    }
    if (writer) {
      const int t = t0 + r;
      const float ref = ok ? sRef[r] * 0.693147180559945309f : 0.0f;
      bool marked = false;
      if (t < T) {
        float* out = p.LN + ((i64)b * p.maxT + t) * p.maxU;
#pragma unroll
        for (int j = 0; j < DCOLS; ++j) {
          const int u = uOff + c0 + j;
          if (c0 + j < c1 && u < U) {
            const float acc = sum[j];
            out[u] = (logf(acc) + ref) + sMaxP[c0 + j];
            marked |= !(acc >= kSumLo && acc <= kSumHi &&
                        acc >= kSpread * fmaf(maxE, sSumP[c0 + j], sumE));
          }
        }
      }
      if (marked) {
        p.marks[kMarkTiles + b * p.tilesX + t0 / kTileM] = 1;
        p.marks[kMarkAny] = 1;
      }
    }
  }

  // ---------------- teardown (all roles, also after an abort) ----------------
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kMmaWarp) tmem_dealloc(tBase, (uint32_t)p.tmemCols);
}

int pow2_at_least(int x) {
  int p = 32;
  while (p < x) p <<= 1;
  return p;
}

// Label axis as the kernel sees it: up to 160 positions (two accumulators and three operand stages fill
// the tensor memory) in one column range, more in two equal ranges.
struct LabelAxis {
  int ranges, part;
  int rows() const { return ranges * part; }
};
LabelAxis label_axis(int maxU) {
  const int n = (int)round_up64(maxU > 0 ? maxU : 1, 16);
  if (n <= 160) return LabelAxis{1, n};
  return LabelAxis{2, (int)round_up64((n + 1) / 2, 16)};
}

}  // namespace

void launch_lognorm_f16(const void* E, const void* P, float* LN, float* rowRef, float* maxP,
                        const int* inLens, const int* labLens, Dims d, const LogNormScratch& ws,
                        int* status, bool sample, cudaStream_t stream, const int* labels, float* EL, float* ebl) {
  const LabelAxis axis = label_axis(d.maxU);
  const int rows = axis.rows(), kPad = (int)round_up64(d.V, kStageK);
  const bool bf = d.dtype == kDtypeBf16;
  uint8_t* operand = reinterpret_cast<uint8_t*>(ws.operand);
  {
    ScopedKernel sk("expp_f16", stream);
    int samples = !sample ? 0 : d.V <= 8192 ? 4 * ws.nSM : ws.nSM;   // (half of the first round's CTAs at most)
    if (d.B + div_up(samples, d.maxU) > 65535) samples = 0;
    auto go = [&](auto k, auto* e, auto* p) {
      k<<<dim3(d.maxU, d.B + div_up(samples, d.maxU)), expp_threads(d.V), 0, stream>>>(
          e, p, operand, maxP, ws.sumP, inLens, labLens, samples, d.B, d.maxT, d.maxU, d.V, rows, kPad, ws.marks);
    };
    if (bf) go(expp_f16_kernel<bf16>, static_cast<const bf16*>(E), static_cast<const bf16*>(P));
    else go(expp_f16_kernel<float>, static_cast<const float*>(E), static_cast<const float*>(P));
  }
  TB200_CHECK_LAUNCH();
  const CUtensorMap tmE =
      bf ? make_tmap_bf16_3d(E, (uint64_t)d.V, (uint64_t)d.maxT, (uint64_t)d.B, (uint64_t)d.V * 2,
                             (uint64_t)d.maxT * d.V * 2, kStageK, kTileM)
         : make_tmap_f32_3d(E, (uint64_t)d.V, (uint64_t)d.maxT, (uint64_t)d.B, (uint64_t)d.V * 4,
                            (uint64_t)d.maxT * d.V * 4, kTileM);
  // (16-bit elements that are only copied: the 64 halves hi or lo of a stage make a row of 128 bytes)
  const CUtensorMap tmP = make_tmap_bf16_3d(operand, (uint64_t)kPad * 2, (uint64_t)rows, (uint64_t)d.B,
                                            (uint64_t)kPad * 4, (uint64_t)rows * kPad * 4,
                                            kStageK, axis.part);
  F16Params p{};
  p.LN = LN; p.rowRef = rowRef; p.maxP = maxP; p.sumP = ws.sumP; p.inLens = inLens; p.labLens = labLens;
  p.status = status;
  p.maxT = d.maxT; p.maxU = d.maxU; p.V = d.V; p.nPad = axis.part; p.halves = axis.ranges;
  p.B = d.B;
  p.tilesX = div_up(d.maxT, kTileM);
  p.nSM = ws.nSM;
  p.partial = ws.partial; p.rowSums = ws.rowSums; p.tickets = ws.tickets; p.marks = ws.marks;
  p.blank = d.blank;
  if (labels != nullptr && EL != nullptr && ebl != nullptr) {
    p.labels = labels; p.EL = EL; p.ebl = ebl;
  }
  // Tensor memory: two accumulators, 64 columns a stage.
  constexpr int kCeiling = 217 * 1024;   // (the static shared memory takes up to 9 KB)
  p.tmemCols = pow2_at_least(2 * axis.part + kStages * 64);
  const int smem = std::max(kStages * (stage_raw_bytes(bf) + axis.part * 256) + 1024, 120 * 1024);   // one CTA per SM
  const dim3 grid((unsigned)(p.tilesX * p.halves * d.B + p.nSM));
  {
    ScopedKernel sk("lognorm_f16", stream);
    auto go = [&](auto k, int drains) {
      allow_dyn_smem(k, kCeiling);
      k<<<grid, (4 * kStages + 4 * drains + 4) * 32, smem, stream>>>(tmE, tmP, p);
    };
    // (three drain groups leave 72 registers a thread, four 64)
    if (axis.part > 120) bf ? go(lognorm_f16_kernel<4, 40, true>, 4) : go(lognorm_f16_kernel<4, 40, false>, 4);
    else bf ? go(lognorm_f16_kernel<3, 40, true>, 3) : go(lognorm_f16_kernel<3, 40, false>, 3);
  }
  TB200_CHECK_LAUNCH();
}

}  // namespace tb200
