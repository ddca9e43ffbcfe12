// fp32 log-normalisers on the SIMT pipes and the row statistics the factored kernels need.
//
// lognorm_exact: logsumexp_v(E[t,v]+P[u,v]) per lattice node with the maximum
// subtracted before exponentiation -- the brute-force definition the reference's
// tests use (transducer/test.h:51-80).  One warp per node, lanes stride over the
// vocabulary, warp-shuffle reductions.
//
// lognorm_factored: the sum as a product of factors, sum_v exp(E-maxE) exp(P-maxP), as the
// reference forms it with torch ops (transducer/torch_binding.py:35-40), for the shapes the
// TMA-fed tensor-core kernel cannot take (vocabulary not a multiple of 4 floats or below 32,
// unaligned base pointers): a multiply-add per node and word instead of an exponential.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "profile.h"

namespace tb200 {
namespace {

__device__ __forceinline__ float node_logsumexp(const float* __restrict__ er,
                                                const float* __restrict__ pr, int V,
                                                int lane) {
  float m = neg_inf();
  for (int v = lane; v < V; v += 32) m = fmaxf(m, er[v] + pr[v]);
  m = warp_max(m);
  float s = 0.0f;
  if (m != neg_inf() && m != pos_inf()) {
    for (int v = lane; v < V; v += 32) s += expf((er[v] + pr[v]) - m);
  }
  s = warp_sum(s);
  return logf(s) + m;
}

constexpr int kWarpsPerCta = 8;

// grid = (ceil(maxU / 8), maxT, B); warp w of CTA (x,t,b) owns node (t, x*8+w).
__global__ void __launch_bounds__(kWarpsPerCta * 32) lognorm_exact_kernel(
    const float* __restrict__ E, const float* __restrict__ P, float* __restrict__ LN,
    const int* __restrict__ inLens, const int* __restrict__ labLens, int maxT, int maxU,
    int V) {
  const int b = blockIdx.z, t = blockIdx.y;
  const int u = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (t >= T || u >= U) return;
  const int lane = threadIdx.x & 31;
  const float r = node_logsumexp(E + ((i64)b * maxT + t) * V, P + ((i64)b * maxU + u) * V,
                                 V, lane);
  if (lane == 0) LN[((i64)b * maxT + t) * maxU + u] = r;
}

// One CTA per 32 frames x 32 label positions.  The vocabulary goes by in steps of 64 words, shared
// out to four groups of 64 threads, 16 words each; thread (ty, tx) of a group owns 4 frames x 4
// positions, and the groups' sums are added at the end: an utterance has few nodes per thread, so
// the split is what fills the chip.  exp(E - rowMax) and exp(P - maxP) of a step are formed once
// per CTA and stored transposed (lanes = 8 words x 4 rows: the stores of a warp fall into 32
// different banks), while the next step's entries are already on their way into registers.
// Precision: the exponentials are exact to the hardware's ex2 whatever the row's maximum (below), sums
// have three levels (16 words, 16 steps, the rest), and the logarithm is taken and the references added
// in fp64, so that the result is no further from float64 than lognorm_exact's.  Measured, V = 29..8041,
// rms over the nodes relative to lognorm_exact's own (1e-7..1.5e-6, mostly the rounding of the
// result): N(0,1..5) scores 0.74..0.91, confident words 5..45 above the rest 0.61..0.92, such words
// cancelled by P 0.77..0.92, crossing 0.40..1.02, log-softmax rows 0.65..0.99.  (With ex2 of the
// rounded difference and logf: up to 8.5.)
// The references lie 2^46 below the rows' maxima: a factor is at most 2^47, a sum V 2^94, and what
// factors below 2^-126 lose, V 2^-126 2^47, is below 2^-26 of a sum of V 2^-53 or more, i.e. down
// to sums e^-94 (V = 1025) of the two maxima's product.
// A batch of few tiles would leave most of the chip idle through a long vocabulary: a cluster of up
// to 8 CTAs then shares a tile, each with its part of the steps, and the first adds the others'
// sums, read from their shared memory, in rank order.
// Nodes with a smaller sum, or one that is not finite, become NaN, as from the tensor-core kernel:
// the caller has them recomputed exactly.
// Per word and thread 16 FFMA, two 16-byte shared loads and one exponential with its load and store, about
// ten instructions more; bound by the shared-memory and special-function queue (44 % of the issue
// slots used, stalls: short scoreboard 1.9, queue full 1.5 per instruction), so that two products per
// instruction (fma.rn.f32x2) gained 1 % and were not kept.  (B=16 T=600 U'=81 V=1025: 130 us; 135 with
// rint, 158 with expf of the difference and the remainder of a 2Sum, 115 with the bare ex2 of it.)
constexpr float kFacShift = 46.0f;
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fac_ref(float rowMax) { return rintf(rowMax * 1.4426950408889634f) - kFacShift; }
constexpr int kFacM = 32, kFacK = 64, kFacLd = kFacM + 4;
__global__ void __launch_bounds__(256) lognorm_factored_kernel(
    const float* __restrict__ E, const float* __restrict__ P, const float* __restrict__ rowMax,
    const float* __restrict__ maxP, float* __restrict__ LN, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int* status, int maxT, int maxU, int V) {
  __shared__ __align__(16) float Es[2][kFacK][kFacLd];
  __shared__ __align__(16) float Ps[2][kFacK][kFacLd];
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();   // ranks along x
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const int b = blockIdx.z, t0 = blockIdx.y * kFacM, u0 = (blockIdx.x / ranks) * kFacM;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  if (t0 >= T || u0 >= U) return;   // (the same for the whole cluster)
  // this rank's words [vBegin, vEnd)
  const int steps = (V + kFacK - 1) / kFacK;
  const int vBegin = (int)((i64)rank * steps / ranks) * kFacK;
  const int vEnd = min((int)((i64)(rank + 1) * steps / ranks) * kFacK, V);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int grp = tid >> 6, ty = (tid & 63) >> 3, tx = tid & 7;
  // what this thread loads: words kk + 8 i of E row and P row 4 w + mm
  const int kk = lane & 7, row = 4 * w + (lane >> 3);
  const i64 tRow = (i64)b * maxT + min(t0 + row, T - 1), uRow = (i64)b * maxU + min(u0 + row, U - 1);
  const float *er = E + tRow * V + vBegin + kk, *pr = P + uRow * V + vBegin + kk;   // advanced step by step
  const float eRef = fac_ref(rowMax[tRow]), pRef = fac_ref(maxP[uRow]);
  float xe[2][8], xp[2][8];   // entries of the next two steps
  int left = vEnd - vBegin - kk;   // words from the next step's first one on
  auto load = [&](float (&ye)[8], float (&yp)[8]) {
    if (left + kk >= kFacK) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        ye[i] = er[i * 8];
        yp[i] = pr[i * 8];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        ye[i] = i * 8 < left ? er[i * 8] : neg_inf();   // (its exponential is the zero that is wanted)
        yp[i] = i * 8 < left ? pr[i * 8] : neg_inf();
      }
    }
    er += kFacK;
    pr += kFacK;
    left -= kFacK;
  };
  // exp(x) 2^-ref = 2^f 2^(n - ref), n = rint(x log2(e)) and |f| <= 1/2 by Cody and Waite's reduction with
  // log2(e) in two parts: the reference is an integer in the exponent, so that nothing is rounded
  // off a word however far below its row's maximum it lies.  (f is not finite where it is masked.)
  auto ex = [](float x, float ref) {
    constexpr float kLog2e = 1.4426950408889634f, kLog2eLo = 1.9259629911e-8f;
    constexpr float kRound = 12582912.0f;   // 1.5 2^23: adding it rounds to an integer
    const float n = (x * kLog2e + kRound) - kRound, f = fmaf(x, kLog2eLo, fmaf(x, kLog2e, -n)), k = n - ref;
    return k < -200.0f ? 0.0f : ex2_ftz(f) * ex2_ftz(k);
  };
  auto put = [&](int s, const float (&ye)[8], const float (&yp)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      Es[s][i * 8 + kk][row] = ex(ye[i], eRef);
      Ps[s][i * 8 + kk][row] = ex(yp[i], pRef);
    }
  };
  float total[4][4], sum[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = sum[i][j] = 0.0f;
  int step = 0;
  // words v0.. are in buffer q, those of the step after in xe[q ^ 1] / xp[q ^ 1]
  auto one = [&](auto qc, int v0) {
    constexpr int q = decltype(qc)::value;
    if (v0 + 2 * kFacK < vEnd) load(xe[q], xp[q]);
    float acc[4][4];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const float4 a4 = *reinterpret_cast<const float4*>(&Es[q][grp * 16 + k][ty * 4]);
      const float4 c4 = *reinterpret_cast<const float4*>(&Ps[q][grp * 16 + k][tx * 4]);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = k ? fmaf(a[i], c[j], acc[i][j]) : a[i] * c[j];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] += acc[i][j];
    if (++step == 16) {
      step = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          total[i][j] += sum[i][j];
          sum[i][j] = 0.0f;
        }
    }
    if (v0 + kFacK < vEnd) put(q ^ 1, xe[q ^ 1], xp[q ^ 1]);   // (last read before the previous barrier)
    __syncthreads();
  };
  load(xe[0], xp[0]);
  if (vBegin + kFacK < vEnd) load(xe[1], xp[1]);
  put(0, xe[0], xp[0]);
  __syncthreads();
  for (int v0 = vBegin; v0 < vEnd; v0 += 2 * kFacK) {
    one(std::integral_constant<int, 0>{}, v0);
    if (v0 + kFacK < vEnd) one(std::integral_constant<int, 1>{}, v0 + kFacK);
  }
  // the groups' sums, [grp][frame][position], over the operand buffers
  float* red = &Es[0][0][0];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      red[grp * 1024 + (ty * 4 + i) * 32 + tx * 4 + j] = total[i][j] + sum[i][j];
  __syncthreads();
  if (ranks > 1) {   // my sum of groups in place of the first group's, then everybody's at rank 0
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = q * 256 + tid;
      red[i] = (red[i] + red[1024 + i]) + (red[2048 + i] + red[3072 + i]);
    }
    cluster.sync();
  }
  const float smallest = (float)V * 0x1p-53f;
  int flagged = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = q * 256 + tid, t = t0 + (i >> 5), u = u0 + (i & 31);
    if (rank == 0 && t < T && u < U) {
      float x;
      if (ranks == 1) {
        x = (red[i] + red[1024 + i]) + (red[2048 + i] + red[3072 + i]);
      } else {
        x = red[i];
        for (int r = 1; r < ranks; ++r) x += cluster.map_shared_rank(red, r)[i];
      }
      const double ref = (double)fac_ref(rowMax[(i64)b * maxT + t]) + (double)fac_ref(maxP[(i64)b * maxU + u]);
      float ln = (float)(ref * 0.6931471805599453 + log((double)x));
      if (!(x >= smallest && x < pos_inf())) {
        ln = __int_as_float(0x7fc00000);
        ++flagged;
      }
      LN[((i64)b * maxT + t) * maxU + u] = ln;
    }
  }
  if (flagged) atomicAdd(&status[1], flagged);
  if (ranks > 1) cluster.sync();   // (no rank's shared memory goes before it was read)
}

// One warp per row: the maxima of the rows of E (rowMaxE, rows t < T_b) and of P (maxP, rows
// u <= label length) of every utterance; rows beyond get 0.
__global__ void __launch_bounds__(256) row_max_kernel(
    const float* __restrict__ E, float* __restrict__ rowMaxE, const float* __restrict__ P,
    float* __restrict__ maxP, const int* __restrict__ inLens, const int* __restrict__ labLens,
    int maxT, int maxU, int V) {
  const int b = blockIdx.y, lane = threadIdx.x & 31;
  const int ctasE = (maxT + 7) / 8;
  const bool isE = (int)blockIdx.x < ctasE;
  const int row = (isE ? blockIdx.x : blockIdx.x - ctasE) * 8 + (threadIdx.x >> 5);
  const int rows = isE ? maxT : maxU, n = min(isE ? inLens[b] : labLens[b] + 1, rows);
  float* out = isE ? rowMaxE : maxP;
  if (row >= rows || out == nullptr) return;
  float m = 0.0f;
  if (row < n) {
    const float* x = (isE ? E : P) + ((i64)b * rows + row) * V;
    m = neg_inf();
    for (int v = lane; v < V; v += 32) m = fmaxf(m, x[v]);
    m = warp_max(m);
  }
  if (lane == 0) out[(i64)b * rows + row] = m;
}

// One CTA per prediction row: maxP and expP = exp(P - maxP); zeros for padded rows.
__global__ void __launch_bounds__(256) exp_rows_kernel(
    const float* __restrict__ P, float* __restrict__ expP, float* __restrict__ maxP,
    const int* __restrict__ labLens, int maxU, int V) {
  __shared__ float red[8];
  const int b = blockIdx.y, u = blockIdx.x;
  const int U = min(labLens[b] + 1, maxU);
  const float* p = P + ((i64)b * maxU + u) * V;
  float* o = expP + ((i64)b * maxU + u) * V;
  if (u >= U) {
    for (int v = threadIdx.x; v < V; v += blockDim.x) o[v] = 0.0f;
    if (threadIdx.x == 0) maxP[(i64)b * maxU + u] = 0.0f;
    return;
  }
  float m = neg_inf();
  for (int v = threadIdx.x; v < V; v += blockDim.x) m = fmaxf(m, p[v]);
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
#pragma unroll
  for (int k = 1; k < 8; ++k) m = fmaxf(m, red[k]);
  for (int v = threadIdx.x; v < V; v += blockDim.x) o[v] = expf(p[v] - m);
  if (threadIdx.x == 0) maxP[(i64)b * maxU + u] = m;
}

// How lognorm_factored is cut: tiles, and the ranks that share one -- as many as keep the grid within
// two CTAs per SM (what is resident at once) and leave every rank two steps.  Measured (us, 1 rank /
// this rule): B=5 T=69 U'=5 V=8042 116 / 17; B=2 T=44 U'=7 V=23850 348 / 54; B=4 T=400 U'=101
// V=5001 131 / 131.
constexpr int kFacResident = 2 * 148;
struct FacGrid {
  i64 tiles;
  int steps, ranks;
};
FacGrid fac_grid(Dims d) {
  FacGrid g{(i64)div_up(d.maxU, kFacM) * div_up(d.maxT, kFacM) * d.B, div_up(d.V, kFacK), 1};
  while (g.ranks < 8 && g.tiles * g.ranks * 2 <= kFacResident && g.ranks * 4 <= g.steps) g.ranks *= 2;
  return g;
}

}  // namespace

// Estimates of both kernels' time in us: a warp of lognorm_exact passes over the vocabulary twice,
// with about 340 words' worth of fixed work; lognorm_factored computes whole tiles whatever the
// label axis, 1.8 us per step of 64 words with two CTAs on an SM and 1.2 with one.  The line lies at
// 4 to 9 label positions for many nodes and higher for few.  Measured (us for the call, exact /
// factored; row maxima and, for the latter, the pass over marked nodes included): B=64 T=1000 V=1301
// U'=2 220 / 347, 4 343 / 348, 6 472 / 348; B=8 T=400 V=1025 U'=2 19 / 33, 8 29 / 33, 12 42 / 34;
// B=8 T=400 V=8041 U'=4 136 / 150, 8 202 / 151; B=1 T=300 V=1025 U'=33 19 / 23, 65 27 / 23.
bool lognorm_factored_pays(Dims d) {
  const FacGrid g = fac_grid(d);
  const double ctas = (double)g.tiles * g.ranks, nodes = (double)d.B * d.maxT * d.maxU;
  const double exact = 4e-3 * d.V + 0.6e-6 * nodes * (d.V + 340.0);
  const double factored = 9.0 + (ctas <= kFacResident / 2 ? 1.2 : 1.8) * std::max(1.0, ctas / kFacResident) *
                                    div_up(g.steps, g.ranks);
  return factored < exact;
}

void launch_lognorm_simt(const float* E, const float* P, float* LN, float* rowRef, float* maxP,
                         const int* inLens, const int* labLens, Dims d, bool exact, int* status,
                         cudaStream_t stream) {
  if (d.B <= 0) return;
  if (d.maxT > 65535 || d.B > 65535)
    throw std::invalid_argument("exact log-normaliser: batch or frame count above 65535");
  if (rowRef || maxP) {
    ScopedKernel sk("row_max", stream);
    row_max_kernel<<<dim3(div_up(d.maxT, 8) + div_up(d.maxU, 8), d.B), 256, 0, stream>>>(
        E, rowRef, P, maxP, inLens, labLens, d.maxT, d.maxU, d.V);
    TB200_CHECK_LAUNCH();
  }
  if (exact) {
    ScopedKernel sk("lognorm_exact", stream);
    lognorm_exact_kernel<<<dim3(div_up(d.maxU, kWarpsPerCta), d.maxT, d.B), kWarpsPerCta * 32, 0, stream>>>(
        E, P, LN, inLens, labLens, d.maxT, d.maxU, d.V);
  } else {
    ScopedKernel sk("lognorm_factored", stream);
    const int ranks = fac_grid(d).ranks;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(div_up(d.maxU, kFacM) * ranks, div_up(d.maxT, kFacM), d.B);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ranks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    TB200_CUDA_CHECK(cudaLaunchKernelEx(&cfg, lognorm_factored_kernel, E, P, (const float*)rowRef,
                                        (const float*)maxP, LN, inLens, labLens, status, d.maxT, d.maxU, d.V));
  }
  TB200_CHECK_LAUNCH();
}

void launch_exp_rows(const float* P, float* expP, float* maxP, const int* labLens, int B,
                     int maxU, int V, cudaStream_t stream) {
  if (B <= 0 || maxU <= 0) return;
  dim3 grid(maxU, B);
  ScopedKernel sk("exp_rows", stream);
  exp_rows_kernel<<<grid, 256, 0, stream>>>(P, expP, maxP, labLens, maxU, V);
  TB200_CHECK_LAUNCH();
}

}  // namespace tb200
