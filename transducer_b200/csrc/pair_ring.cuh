// Pieces shared by the single-warp sweeps (lattice_sweep.cu, lattice_warp.cu): rows of pairs, one row per
// anti-diagonal, and the ring through which a warp reads them.
#pragma once

#include "sm100.cuh"

namespace tb200 {
namespace sweep {

constexpr int kDiag = 16;   // diagonals per block
// blocks in shared memory (three of the wide ones leave room for two CTAs per SM)
__host__ __device__ constexpr int ring_blocks(int npl) { return npl <= 4 ? 4 : 3; }
__host__ __device__ constexpr bool natural(int npl) { return npl > 4; }   // (where gradients are to follow)

// Place of position u within a row of pairs (operands, factors): 16-byte pieces of two positions,
// the pieces of the 32 lanes side by side, so that a warp's 16-byte accesses are contiguous; the
// last position of an odd NPL makes a piece of its own.
__host__ __device__ constexpr int pair_slot(int u, int npl) {
  const int lane = u / npl, r = u % npl, q = r >> 1;
  return q < npl / 2 ? (q * 32 + lane) * 2 + (r & 1) : q * 64 + lane;
}
// Place of position u within a row of single numbers (alphas, g): as it comes where a lane's
// positions make one vector access, else one plane of 32 lanes per position of a lane.
__host__ __device__ constexpr int row_slot(int u, int npl) {
  return npl <= 4 ? u : (u % npl) * 32 + u / npl;
}

// Copies blocks of pair rows into this lane's share of a shared-memory ring and reads them back.
// Lanes without positions of the utterance hold `fill` throughout.
template <int NPL>
struct PairRing {
  static constexpr int ld = 32 * NPL, kRowBytes = ld * 8, kRing = ring_blocks(NPL);
  static constexpr int kPieces = NPL / 2, kOdd = kPieces * 512;   // byte offset of the odd position's plane
  uint8_t* ring;
  const uint8_t* src;
  int lane;
  bool act;
  __device__ PairRing(uint8_t* ring_, const float2* rows, int lane_, int U, unsigned fillX, unsigned fillY)
      : ring(ring_), src(reinterpret_cast<const uint8_t*>(rows)), lane(lane_), act(NPL * lane_ < U) {
    if (!act)
      for (int i = 0; i < kRing * kDiag; ++i) {
        uint8_t* row = ring + i * kRowBytes;
#pragma unroll
        for (int q = 0; q < kPieces; ++q)
          *reinterpret_cast<uint4*>(row + (q * 32 + lane) * 16) = make_uint4(fillX, fillY, fillX, fillY);
        if (NPL & 1) *reinterpret_cast<uint2*>(row + kOdd + lane * 8) = make_uint2(fillX, fillY);
      }
  }
  // rows [row, row + n) -> slot
  __device__ __forceinline__ void issue(int slot, i64 row, int n) {
    if (act) {
      const uint32_t dst = sm100::smem_u32(ring) + (uint32_t)slot * (kDiag * kRowBytes) + lane * 16;
      const uint8_t* from = src + row * kRowBytes + lane * 16;
      auto one = [&](int i) {
#pragma unroll
        for (int q = 0; q < kPieces; ++q)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * kRowBytes + q * 512),
                       "l"(from + i * kRowBytes + q * 512) : "memory");
        if (NPL & 1)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + i * kRowBytes + kOdd - lane * 8),
                       "l"(from + i * kRowBytes + kOdd - lane * 8) : "memory");
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
    const uint8_t* p = ring + (slot * kDiag + i) * kRowBytes;
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
      const float4 f = *reinterpret_cast<const float4*>(p + (q * 32 + lane) * 16);
      x[2 * q] = f.x;
      y[2 * q] = f.y;
      x[2 * q + 1] = f.z;
      y[2 * q + 1] = f.w;
    }
    if constexpr (NPL & 1) {
      const float2 f = *reinterpret_cast<const float2*>(p + kOdd + lane * 8);
      x[NPL - 1] = f.x;
      y[NPL - 1] = f.y;
    }
  }
};

// Row length of a 32x32 tile in shared memory that is written by rows and read along the
// anti-diagonals (or the other way): element (d - lane, lane) is at d * ld - (ld - 1) * lane, so ld
// has to be even for 32 different banks -- 33 would put a whole anti-diagonal into one -- and 34
// keeps columns at a two-way conflict.  (33 -> 34 and two rows per access: sweep_prep 62 -> 38 us at
// B = 32, T = 2000, U' = 101.)
constexpr int kTileLd = 34;

}  // namespace sweep
}  // namespace tb200
