// Dense part of the emission / prediction gradients on the SIMT pipes.
//
// The reference forms these with torch ops (transducer/torch_binding.py:85-89):
//   Wn = occupancy / expLN;  egrads += expE * bmm(Wn, expP);
//   pgrads += expP * bmm(Wn^T, expE);  both scaled by deltas[b].
// Here W[t,u] = occupancy * exp(rowRef[t] + maxP[u] - LN[t,u]) is the same weight
// (expLN = exp(LN - rowRef - maxP)), expE is recomputed from E on the fly (never
// stored), and every element of egrads/pgrads is written exactly once: no memset,
// no read-modify-write of the dense buffers except the label-arc scatter.
//
// These fp32 FMA kernels take any vocabulary size and alignment; the tensor-core
// kernels replace them for shapes TMA can address.
#include "kernels.h"
#include "profile.h"

namespace tb200 {
namespace {

// Tiles of 64x64 outputs, 256 threads with 4x4 each; the contraction runs in steps of 32 whose
// entries are loaded into registers one step ahead and shared memory alternates between two
// buffers: one barrier a step.  Bound by the latency of few CTAs (small shapes) or by shared-
// memory bandwidth (16 FFMA to two 16-byte loads).
constexpr int BM = 64, BN = 64, BK = 32;

__device__ __forceinline__ void tile_step(const float (*A)[BM + 4], const float (*B)[BN], int ty,
                                          int tx, float (&acc)[4][4]) {
#pragma unroll
  for (int k = 0; k < BK; ++k) {
    const float4 a = *reinterpret_cast<const float4*>(&A[k][ty * 4]);
    const float4 c = *reinterpret_cast<const float4*>(&B[k][tx * 4]);
    const float av[4] = {a.x, a.y, a.z, a.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) acc[m][n] = fmaf(av[m], cv[n], acc[m][n]);
  }
}

// egrads tile: rows t0..t0+63 of utterance b, columns v0..v0+63; label-arc terms included:
//   egrads[t, label_u] -= delta * em[t,u], in position order, so that repeated labels on a frame
// are combined deterministically.  (They were a kernel of their own in which one thread per frame
// walked the labels: 35 us at T = 600, U' = 81 against 3 us here.)
__global__ void __launch_bounds__(256) egrad_simt_kernel(
    const float* __restrict__ E, const float* __restrict__ rowRef,
    const float* __restrict__ W, int ldW, const float* __restrict__ expP,
    const float* __restrict__ eBlank, const float* __restrict__ em, const int* __restrict__ labels,
    const float* __restrict__ deltas, float* __restrict__ egrads, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int maxT, int maxU, int V, int blank) {
  __shared__ __align__(16) float Ws[2][BK][BM + 4];
  __shared__ __align__(16) float Ps[2][BK][BN];
  __shared__ short sU[256], sV[256];
  __shared__ int sCnt[8];
  const int b = blockIdx.z, t0 = blockIdx.y * BM, v0 = blockIdx.x * BN;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  float* out = egrads + (i64)b * maxT * V;

  if (t0 >= T || U <= 0) {  // padded frames: exact zeros, inputs not read
    for (int m = tid >> 6; m < BM; m += 4)
      if (t0 + m < maxT && v0 + (tid & 63) < V) out[(i64)(t0 + m) * V + v0 + (tid & 63)] = 0.0f;
    return;
  }
  // W tile, transposed into [u][t]: thread <-> frame tid >> 2, 8 positions (rows of W are whole
  // multiples of 32 floats, zero outside the lattice); expP tile: thread <-> word tid & 63
  const float* wr = W + ((i64)b * maxT + min(t0 + (tid >> 2), T - 1)) * ldW + (tid & 3) * 8;
  const int vc = min(v0 + (tid & 63), V - 1);
  const float* xp = expP + (i64)b * maxU * V + vc;
  const bool tIn = t0 + (tid >> 2) < T;
  float4 rw[2];
  float rp[8];
  auto load = [&](int u0) {
    rw[0] = *reinterpret_cast<const float4*>(wr + u0);
    rw[1] = *reinterpret_cast<const float4*>(wr + u0 + 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) rp[i] = xp[(i64)min(u0 + i * 4 + (tid >> 6), U - 1) * V];
  };
  auto put = [&](int s) {
    const float w[8] = {rw[0].x, rw[0].y, rw[0].z, rw[0].w, rw[1].x, rw[1].y, rw[1].z, rw[1].w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      Ws[s][(tid & 3) * 8 + i][tid >> 2] = tIn ? w[i] : 0.0f;
      Ps[s][i * 4 + (tid >> 6)][tid & 63] = rp[i];   // (positions beyond U meet a zero of W)
    }
  };
  float acc[4][4] = {};
  load(0);
  put(0);
  __syncthreads();
  int s = 0;
  for (int u0 = 0; u0 < U; u0 += BK, s ^= 1) {
    const bool more = u0 + BK < U;
    if (more) load(u0 + BK);
    tile_step(Ws[s], Ps[s], ty, tx, acc);
    if (more) put(s ^ 1);
    __syncthreads();
  }
  // The tile of sums goes through shared memory once, so that E is read and the gradient written
  // along the rows: thread <-> column c, frames r0 + 4 i.
  const float delta = deltas ? deltas[b] : 1.0f;
  const int c = tid & 63, r0 = tid >> 6, v = v0 + c;
  float* tile = &Ws[0][0][0];          // [64][65]
  static_assert(BM * (BN + 1) <= 2 * BK * (BM + 4), "the tile fits the W buffers");
  float val[16];
  {
    const float* e = E + (i64)b * maxT * V + vc;
    const float* ref = rowRef + (i64)b * maxT;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int t = min(t0 + r0 + 4 * i, T - 1);
      val[i] = e[(i64)t * V] - ref[t];
    }
  }
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) tile[(ty * 4 + m) * (BN + 1) + tx * 4 + n] = acc[m][n];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = r0 + 4 * i, t = t0 + r;
    float x = expf(val[i]) * tile[r * (BN + 1) + c];
    if (v == blank) x -= eBlank[(i64)b * maxT + min(t, T - 1)];
    val[i] = t < T ? x * delta : 0.0f;
  }
  // label arcs, 256 positions at a time: those whose label falls into the tile, in position
  // order, their occupancies staged 32 positions x 64 frames at a time
  const int lane = tid & 31, warp = tid >> 5;
  float (*sEm)[BM] = reinterpret_cast<float (*)[BM]>(&Ps[0][0][0]);
  for (int uB = 0; uB < U - 1; uB += 256) {
    const int u = uB + tid;
    const int col = u < U - 1 ? labels[(i64)b * (maxU - 1) + u] - v0 : -1;
    const bool hit = col >= 0 && col < BN;
    const unsigned mask = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) sCnt[warp] = __popc(mask);
    __syncthreads();
    int pos = __popc(mask & ((1u << lane) - 1)), n = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) pos += sCnt[w];
      n += sCnt[w];
    }
    if (hit) {
      sU[pos] = (short)u;
      sV[pos] = (short)col;
    }
    __syncthreads();
    for (int k0 = 0; k0 < n; k0 += BK) {
      const int nk = min(BK, n - k0);
      for (int i = tid; i < nk * BM; i += 256) {
        const int k = i % nk, m = i / nk;   // (neighbouring threads: neighbouring positions of a frame)
        sEm[k][m] = t0 + m < T ? em[((i64)b * maxT + t0 + m) * maxU + sU[k0 + k]] : 0.0f;
      }
      __syncthreads();
      for (int k = 0; k < nk; ++k)
        if (sV[k0 + k] == c) {
#pragma unroll
          for (int i = 0; i < 16; ++i) val[i] -= delta * sEm[k][r0 + 4 * i];
        }
      __syncthreads();
    }
  }
  if (v < V) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (t0 + r0 + 4 * i < maxT) out[(i64)(t0 + r0 + 4 * i) * V + v] = val[i];
  }
}

// pgrads tile: rows u0..u0+63 of utterance b, columns v0..v0+63; the contraction runs over frames.
__global__ void __launch_bounds__(256) pgrad_simt_kernel(
    const float* __restrict__ E, const float* __restrict__ rowRef,
    const float* __restrict__ W, int ldW, const float* __restrict__ expP,
    const float* __restrict__ pBlank, const float* __restrict__ pLabel,
    const int* __restrict__ labels, const float* __restrict__ deltas,
    float* __restrict__ pgrads, const int* __restrict__ inLens,
    const int* __restrict__ labLens, int maxT, int maxU, int V, int blank) {
  __shared__ __align__(16) float Ws[2][BK][BM + 4];
  __shared__ __align__(16) float Es[2][BK][BN];
  const int b = blockIdx.z, u0 = blockIdx.y * BM, v0 = blockIdx.x * BN;
  const int T = min(inLens[b], maxT), U = min(labLens[b] + 1, maxU);
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  float* out = pgrads + (i64)b * maxU * V;

  if (u0 >= U || T <= 0) {
    for (int m = tid >> 6; m < BM; m += 4)
      if (u0 + m < maxU && v0 + (tid & 63) < V) out[(i64)(u0 + m) * V + v0 + (tid & 63)] = 0.0f;
    return;
  }
  const int c = tid & 63, k0 = tid >> 6;   // this thread loads column c of rows k0 + 4 i
  const int uc = min(u0 + c, ldW - 1), vc = min(v0 + c, V - 1);
  const bool uIn = u0 + c < ldW;
  const float* w = W + (i64)b * maxT * ldW + uc;
  const float* e = E + (i64)b * maxT * V + vc;
  const float* ref = rowRef + (i64)b * maxT;
  float rw[8], re[8], rr[8];
  auto load = [&](int t0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = min(t0 + i * 4 + k0, T - 1);
      rw[i] = w[(i64)t * ldW];
      re[i] = e[(i64)t * V];
      rr[i] = ref[t];
    }
  };
  auto put = [&](int s, int t0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = i * 4 + k0;
      Ws[s][k][c] = (uIn && t0 + k < T) ? rw[i] : 0.0f;
      Es[s][k][c] = expf(re[i] - rr[i]);   // (frames beyond T meet a zero of W)
    }
  };
  float acc[4][4] = {};
  load(0);
  put(0, 0);
  __syncthreads();
  int s = 0;
  for (int t0 = 0; t0 < T; t0 += BK, s ^= 1) {
    const bool more = t0 + BK < T;
    if (more) load(t0 + BK);
    tile_step(Ws[s], Es[s], ty, tx, acc);
    if (more) put(s ^ 1, t0 + BK);
    __syncthreads();
  }
  const float delta = deltas ? deltas[b] : 1.0f;
  const float* xp = expP + (i64)b * maxU * V;
  const int* lab = labels + (i64)b * (maxU - 1);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int u = u0 + ty * 4 + m;
    if (u >= maxU) continue;
    const bool live = u < U;
    const int myLab = (live && u < U - 1) ? lab[u] : -1;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int v = v0 + tx * 4 + n;
      if (v >= V) continue;
      float val = 0.0f;
      if (live) {
        val = xp[(i64)u * V + v] * acc[m][n];
        if (v == blank) val -= pBlank[(i64)b * maxU + u];
        if (v == myLab) val -= pLabel[(i64)b * maxU + u];
        val *= delta;
      }
      out[(i64)u * V + v] = val;
    }
  }
}

}  // namespace

void launch_egrad_simt(const float* E, const float* rowRef, const float* W, int ldW,
                       const float* expP, const float* eBlank, const float* em,
                       const int* labels, const float* deltas, float* egrads,
                       const int* inLens, const int* labLens, Dims d,
                       cudaStream_t stream) {
  if (d.B <= 0 || d.maxT <= 0 || d.V <= 0) return;
  dim3 grid(div_up(d.V, BN), div_up(d.maxT, BM), d.B);
  ScopedKernel sk("egrad_simt", stream);
  egrad_simt_kernel<<<grid, 256, 0, stream>>>(E, rowRef, W, ldW, expP, eBlank, em, labels, deltas,
                                              egrads, inLens, labLens, d.maxT, d.maxU, d.V,
                                              d.blank);
  TB200_CHECK_LAUNCH();
}

void launch_pgrad_simt(const float* E, const float* rowRef, const float* W, int ldW,
                       const float* expP, const float* pBlank, const float* pLabel,
                       const int* labels, const float* deltas, float* pgrads,
                       const int* inLens, const int* labLens, Dims d,
                       cudaStream_t stream) {
  if (d.B <= 0 || d.maxU <= 0 || d.V <= 0) return;
  dim3 grid(div_up(d.V, BN), div_up(d.maxU, BM), d.B);
  ScopedKernel sk("pgrad_simt", stream);
  pgrad_simt_kernel<<<grid, 256, 0, stream>>>(E, rowRef, W, ldW, expP, pBlank, pLabel,
                                              labels, deltas, pgrads, inLens, labLens,
                                              d.maxT, d.maxU, d.V, d.blank);
  TB200_CHECK_LAUNCH();
}

}  // namespace tb200
