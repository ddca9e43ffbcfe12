// What the two tensor-core log-normalisers (lognorm_f16.cu, lognorm_umma.cu) share: the division of a
// batch into work items, and the access to a raw chunk of emissions in shared memory.
#pragma once

#include "sm100.cuh"

namespace tb200 {
namespace lognorm {

// Threads of the CTA that brings a row of P to exp(P) pairs, in two passes over it.  The 2048 threads of an SM
// hold 8 rows with 256 of them, and the second pass finds the row in L2 only while 8 rows per SM leave
// room there: fewer and larger CTAs for long rows.  Short rows want many.  us with 256 / 512 / 1024, TF32
// pairs: B = 32, U' <= 101, V = 10000 77 / 67 / 91, V = 32000 273 / 256 / 216; fp16 pairs, B = 64, U' <= 151
// V = 4096 62 / 85 / 142, V = 8192 108 / 119 / 185, U' <= 201 V = 16384 363 / 278 / 337, V = 24000 562 / 458 /
// 487, V = 32000 745 / 667 / 602.
inline int expp_threads(int V) { return V <= 8192 ? 256 : V <= 28000 ? 512 : 1024; }

constexpr int kTileM = 128;    // frames per work item (UMMA M)
constexpr int kChunkK = 32;    // words per chunk of the vocabulary
constexpr int kMaxSMs = 256;   // slots for the partial sums of split tiles
constexpr int kMaxParts = 8;
constexpr int kMaxLabels = 256;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kSumLo = 1e-30f, kSumHi = 1e30f;   // sums outside are not trusted

// Marks of the fp16 kernel for the TF32 kernel behind it: any tile marked, votes of the sampled nodes, a word per
// tile.  Enough votes (kVotes, see spread_kernel) leave every tile to the TF32 kernel.
constexpr int kMarkAny = 0, kMarkVotes = 1, kMarkTiles = 2;
constexpr int kVotes = 2;
__device__ __forceinline__ bool all_marked(const int* marks) { return marks[kMarkVotes] >= kVotes; }
// raw E chunk of a stage: 128 frames x 32 words, rows of 128 bytes (fp32) or 64 bytes (bf16)
__host__ __device__ constexpr int raw_bytes(bool bf) { return kTileM * kChunkK * (bf ? 2 : 4); }

// 16 consecutive words of frame r's row of the raw chunk, starting at word 16 * half, as fp32
template <bool BF>
__device__ __forceinline__ void load_words16(const uint8_t* row, int r, int half, float (&x)[16]) {
  if constexpr (BF) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int jj = half * 2 + j;  // 16-byte piece (8 words) of the 64-byte row
      const uint4 q = *reinterpret_cast<const uint4*>(row + ((jj ^ ((r >> 1) & 3)) << 4));
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        x[8 * j + 2 * k] = __uint_as_float(w[k] << 16);
        x[8 * j + 2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int jj = half * 4 + j;  // 16-byte piece of the 128-byte row
      const float4 v4 = *reinterpret_cast<const float4*>(row + ((jj ^ (r & 7)) << 4));
      x[4 * j] = v4.x; x[4 * j + 1] = v4.y; x[4 * j + 2] = v4.z; x[4 * j + 3] = v4.w;
    }
  }
}

// word `off` (0..31) of frame r's row
template <bool BF>
__device__ __forceinline__ float load_word(const uint8_t* row, int r, int off) {
  if constexpr (BF) {
    const unsigned short h = *reinterpret_cast<const unsigned short*>(
        row + (((off >> 3) ^ ((r >> 1) & 3)) << 4) + (off & 7) * 2);
    return __uint_as_float((uint32_t)h << 16);
  } else {
    return *reinterpret_cast<const float*>(row + (((off >> 2) ^ (r & 7)) << 4) + (off & 3) * 4);
  }
}

// Work items.  A tile (128 frames of one utterance x the whole vocabulary) takes the same time
// whatever it holds, and one CTA fits an SM, so n live tiles on nSM SMs cost ceil(n / nSM)
// rounds: 454 tiles on 148 SMs pay for 592.  The tiles of the last, partly filled round are
// therefore split along the vocabulary into k = min(8, nSM / rem) parts (rem = n mod nSM):
// part 0 runs in the tile's own CTA, parts 1..k-1 in `worker` CTAs appended to the grid (the
// hardware dispatches CTAs in index order, so they start exactly when the last round does).
// Every part keeps the frame's shift of the whole tile (a part that does not begin at chunk 0
// first fetches chunk 0 for it and feeds zeros to the tensor core for that chunk), writes its
// partial sums to `partial`, and the part that finishes last adds the parts in index order.
// The grid is (tilesX * halves * B + nSM) x 1; lengths are on the device, so every CTA derives the
// schedule from them itself (B <= 1024; larger batches are not split).
struct LnItem {
  int b;               // utterance, or -1: nothing to do
  int T, U;            // its lengths
  int t0, uOff;        // first frame; first label position of the column range
  int part, parts, split;
};

// Called by all threads of the CTA (warp 0 scans the lengths).
__device__ __forceinline__ LnItem ln_item(const int* inLens, const int* labLens, int maxT, int maxU,
                                          int V, int B, int tilesX, int halves, int nPad, int nSM) {
  __shared__ int sItem[5];  // b, tile, part, parts, split-tile index
  if (threadIdx.x < 32) {
    const int lane0 = threadIdx.x;
    const int perUtt = tilesX * halves;   // grid slots per utterance
    const int nNatural = perUtt * B;
    const bool worker = (int)blockIdx.x >= nNatural;
    const int myB = worker ? -1 : (int)blockIdx.x / perUtt, myX = worker ? 0 : (int)blockIdx.x % perUtt;
    // live work items of an utterance: tiles x column ranges that hold positions (item ix is
    // range ix % ranges of tile ix / ranges, so the ranges of a tile run side by side and
    // share its chunks of E in L2)
    auto ranges = [&](int bb) {
      const int Ub = min(labLens[bb] + 1, maxU);
      return min(halves, (Ub + nPad - 1) / nPad);
    };
    auto liveTiles = [&](int bb) {
      if (bb >= B) return 0;
      const int Tb = min(inLens[bb], maxT), Ub = min(labLens[bb] + 1, maxU);
      return (Tb > 0 && Ub > 0) ? ((Tb + kTileM - 1) / kTileM) * ranges(bb) : 0;
    };
    int n = 0, before = 0;  // live tiles in all, and in the utterances before mine
    for (int b0 = 0; b0 < B; b0 += 32) {
      const int v = liveTiles(b0 + lane0);
      const int tot = __reduce_add_sync(0xffffffffu, v);
      const int pre = __reduce_add_sync(0xffffffffu, (b0 + lane0 < myB) ? v : 0);
      n += tot;
      before += pre;
    }
    const int full = (n / nSM) * nSM, rem = n - full;
    int k = (rem > 0 && B <= 1024) ? min(kMaxParts, nSM / rem) : 1;
    k = min(k, ((V + kChunkK - 1) / kChunkK) / 16);  // a part is worth >= 16 chunks
    if (k < 2) k = 1;
    int ib = -1, ix = 0, part = 0, parts = 1, split = 0, valid = 0;
    if (!worker) {
      if (myX < liveTiles(myB)) {
        valid = 1; ib = myB; ix = myX;
        const int r = before + myX;
        if (k > 1 && r >= full) { parts = k; split = r - full; }
      }
    } else if (k > 1) {
      const int w = (int)blockIdx.x - nNatural;
      if (w < rem * (k - 1)) {
        split = w / (k - 1);
        part = 1 + w % (k - 1);
        parts = k;
        // locate the tile of live rank full + split
        const int target = full + split;
        int run = 0;
        for (int b0 = 0; b0 < B && !valid; b0 += 32) {
          const int v = liveTiles(b0 + lane0);
          int incl = v;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane0 >= o) incl += up;
          }
          const int lo = run + incl - v, hi = run + incl;  // my utterance holds ranks [lo, hi)
          const unsigned hit = __ballot_sync(0xffffffffu, target >= lo && target < hi);
          if (hit) {
            const int src = __ffs(hit) - 1;
            ib = b0 + src;
            ix = target - __shfl_sync(0xffffffffu, lo, src);
            valid = 1;
          }
          run += __shfl_sync(0xffffffffu, incl, 31);
        }
      }
    }
    if (lane0 == 0) {
      sItem[0] = valid ? ib : -1; sItem[1] = ix; sItem[2] = part; sItem[3] = parts; sItem[4] = split;
    }
  }
  __syncthreads();
  LnItem it;
  it.b = sItem[0];
  it.part = sItem[2]; it.parts = sItem[3]; it.split = sItem[4];
  it.T = it.U = it.t0 = it.uOff = 0;
  if (it.b < 0) return it;
  it.T = min(inLens[it.b], maxT);
  it.U = min(labLens[it.b] + 1, maxU);
  const int nRanges = min(halves, (it.U + nPad - 1) / nPad);
  it.t0 = (sItem[1] / nRanges) * kTileM;
  it.uOff = (sItem[1] % nRanges) * nPad;
  return it;
}

// The labels of an utterance sorted by column (column << 8 | position, ascending; ties keep position
// order), for the transform threads that hand out E[t, label_u] from the chunks they hold.  All
// threads of the CTA; sLab and sKey hold kMaxLabels ints.
__device__ __forceinline__ void sort_labels(const int* lab, int nLab, int* sLab, int* sKey) {
  for (int i = threadIdx.x; i < nLab; i += blockDim.x) sLab[i] = lab[i];
  __syncthreads();
  for (int i = threadIdx.x; i < nLab; i += blockDim.x) {
    const int mine = sLab[i];
    int rank = 0;
    for (int j = 0; j < nLab; ++j) {
      const int o = sLab[j];
      rank += (o < mine || (o == mine && j < i)) ? 1 : 0;
    }
    sKey[rank] = (mine << 8) | i;
  }
}

// Hands out the entries of columns [col0, col0 + width) that the lattice sweeps need, word(off) being
// E[t, col0 + off] of the thread's frame: E[t,label_u] into el (frame's place in row 0; rows maxT apart)
// and E[t,blank] into ebl.  cur: cursor into the sorted labels; nextCol: column of the entry it points to,
// kept in a register so that columns without any cost one comparison.  (Uniform control flow: the list
// and the cursor are the same in all threads of the group; its 128 threads write 128 consecutive floats.)
template <typename F>
__device__ __forceinline__ void hand_out(F word, int col0, int width, const int* sKey, int nLab,
                                         int& cur, int& nextCol, float* el, int maxT, int blank,
                                         float* ebl, bool live) {
  if (nextCol < col0 + width) {
    int key = sKey[cur];
    while ((key >> 8) < col0 && ++cur < nLab) key = sKey[cur];   // the other groups' columns
    while (cur < nLab && (key >> 8) < col0 + width) {
      const float v = word((key >> 8) - col0);
      if (live) el[(i64)(key & 0xff) * maxT] = v;
      if (++cur < nLab) key = sKey[cur];
    }
    nextCol = cur < nLab ? (key >> 8) : 0x7fffffff;
  }
  if (blank >= col0 && blank < col0 + width) {
    const float v = word(blank - col0);
    if (live) *ebl = v;
  }
}

}  // namespace lognorm
}  // namespace tb200
