// Output phase of the backward GEMMs (integer and split-bf16 paths): one warp
// adds its 32 x 128 part of a tile of C = O^T R + R^T O to the gradient.
#pragma once

#include <cuda_runtime.h>

#include "ccm_internal.cuh"
#include "ccm_layout.cuh"
#include "ccm_ptx.cuh"

namespace ccm {

// Threads of a backward kernel: warpgroup 0 holds the TMA (warp 0) and MMA (warp 1)
// roles, warpgroups 1 and 2 the epilogue.  An epilogue thread holds 128 accumulator
// values; with the 168 registers that 384 threads leave each, it spills, so
// warpgroup 0 gives most of its share up: 128 x 40 + 256 x 232 = 384 x 168.
constexpr int kWgThreads = 384;
constexpr int kWgRegsLoad = 40, kWgRegsEpi = 232;

// Shared memory of one warp's transpose buffer: 32 rows x 16 columns of floats.
constexpr int kBwdOutWarpBytes = 32 * 16 * 4;

// A slot as one integer: (q L + l) << 11 | l for a real (state, column) slot,
// kSlotOnes for the ones slot, kSlotNone for padding.  q L + l indexes the rows of
// the coupling matrix (stride 32 L) and its columns alike; l (below 2048: the
// int-sized parameter vector ends at L = 1787) tells the self-edge blocks.
constexpr int kSlotNone = -1, kSlotOnes = -2;
template <class G>
__device__ __forceinline__ int pack_slot(int s, int L) {
  const int t = s / G::kSlots, r = s % G::kSlots;
  if (s == G::kOnes) return kSlotOnes;
  const int q = r / G::kCols, l = t * G::kCols + r % G::kCols;
  return r < G::kUsed && l < L ? (q * L + l) << 11 | l : kSlotNone;
}

// acc[i] of lane r is C[s1][s2] with s1 = rowbase + r, s2 = sQ + i.  Every element
// with s1 <= s2 (SYM; else every element) goes to
//   direct      g2 row (b,k) = s1, column (a,j) = s2
//   mirrored    g2 row (a,j) = s2, column (b,k) = s1   (SYM, s1 < s2)
// without the self-edge blocks (SYM), and the ones slot's row and column to g1d.
// g2 already holds the regulariser term and every entry receives exactly one
// atomic add, so the result does not depend on the order of the adds.
//
// Mirrored adds leave straight from the registers: the lanes of an instruction are
// 32 consecutive slots, i.e. runs of G::kCols consecutive k.  Direct adds go
// through a 16-column transpose (rotated, so that neither side meets a bank
// conflict): an instruction covers 2 rows x 16 columns, runs of consecutive j.
// Each slot is decoded once per tile, by one lane, and passed on by shuffles, and
// the adds are predicated, not branched around.  Decoding slots per element, in a
// loop over the columns of an 8-column buffer, made the split-bf16 backward 61 us at
// L = 90, N = 600 (now 54); the phase overlaps the next tile's MMAs but for a pair's
// last tile, which is what small alignments consist of.
template <class G, bool SYM>
__device__ __forceinline__ void bwd_output(const float (&acc)[128], float *Tb, float *g2, float *g1d,
                                           int L, int lane, int rowbase, int sQ) {
  constexpr unsigned kFull = 0xffffffffu;
  const int p1 = pack_slot<G>(rowbase + lane, L);
  int p2[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) p2[c] = pack_slot<G>(sQ + 32 * c + lane, L);
  char *const gb = reinterpret_cast<char *>(g2);
  const bool ones = rowbase <= G::kOnes;  // this warp's rows or its tile may hold the ones slot
  const uint32_t pitch = 4u * kQPad * L;  // bytes of a row of g2
  const int off = rowbase - sQ;
  if (SYM) {
    // columns i > lo of this lane's row lie above the diagonal
    const int lo = p1 >= 0 ? off + lane : 128;
    char *const base = gb + 4 * (p1 >> 11);
#pragma unroll
    for (int i = 0; i < 128; ++i) {
      const int p = __shfl_sync(kFull, p2[i >> 5], i & 31);
      red_add_if(reinterpret_cast<float *>(base + (uint64_t)(uint32_t)(p >> 11) * pitch), acc[i],
                 i > lo && p >= 0 && ((p ^ p1) & 2047) != 0);
    }
  }
  const int col = lane & 15, rlo = lane >> 4;
#pragma unroll
  for (int cb = 0; cb < 8; ++cb) {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 16; ++e) Tb[lane * 16 + ((e + (lane >> 1)) & 15)] = acc[cb * 16 + e];
    const int p = __shfl_sync(kFull, p2[cb >> 1], (cb & 1) * 16 + col);
    __syncwarp();
    // rows up to rmax of this lane's column lie on or above the diagonal
    const int rmax = SYM ? cb * 16 + col - off : 32;
    char *const base = gb + 4 * (p >> 11);
#pragma unroll
    for (int it = 0; it < 16; ++it) {
      const int row = 2 * it + rlo;
      const int pr = __shfl_sync(kFull, p1, row);
      const float v = Tb[row * 16 + ((col + it) & 15)];
      red_add_if(reinterpret_cast<float *>(base + (uint64_t)(uint32_t)(pr >> 11) * pitch), v,
                 row <= rmax && (p | pr) >= 0 && (!SYM || ((p ^ pr) & 2047) != 0));
      if (ones && row <= rmax) {
        if (pr == kSlotOnes && p >= 0 && (p >> 11) < (kQ - 1) * L) g1d[p >> 11] = v;
        else if (SYM && p == kSlotOnes && pr >= 0 && (pr >> 11) < (kQ - 1) * L) g1d[pr >> 11] = v;
      }
    }
  }
}

// The same for natural slots (s = q L + l, the ones slot at 21 L): rows and columns of
// a tile are contiguous runs of g2's rows and columns, aligned to 128 bytes.  acc[i] of
// lane r is C[s1][s2], s1 = row0 + r, s2 = col0 + i.
//   tiles above the diagonal (SYM)  each element directly and mirrored
//   tiles on it (SYM)               directly, both triangles (C is symmetric bit for
//                                   bit: the sums are integers)
//   !SYM                            directly
// Self-edge blocks (SYM) and the slots from 21 L on take part with zeros, so that no
// add needs a test of its element.  A mirrored add is 32 lanes on 128 contiguous bytes.
// Direct adds go through a 16-column transpose: four columns a lane, 64 contiguous
// bytes a row (16-byte chunk c of row r at chunk c ^ ((r >> 1) & 3): no bank conflict
// either way), as one 16-byte add where g2 is aligned.
// Bound: the rate at which an SM's adds leave for L2 (measured: 32-lane adds on runs
// of 9 floats 2.5, contiguous 4.0, 16-byte ones 5.5 floats a cycle), and below it the
// DRAM sectors of g2, which contiguous runs use whole.  The phase took 96-130 k cycles
// per tile on the 9-column slot groups of the forward (59 k alone on the chip) and
// takes 10-18 k here; with 325 instead of 351 tiles the backward went from 470 to
// 375 us at L = 300, N = 5000 and from 53 to 23 us at L = 50, N = 200.
template <bool SYM>
__device__ __forceinline__ void bwd_output_natural(float (&acc)[128], float *Tb,
                                                   const BwdArgs &args, float *g1, float *g2,
                                                   const float *x1, int lane, int row0, int col0,
                                                   bool diagonal) {
  const int L = args.L, nat = kQ * L;
  const int row = row0 + lane;
  const long long pitch = (long long)kQPad * L;
  auto single = [&](int v, float data) {  // g1 entry v (below 20 L) from its data term
    args.g1d[v] = data;
    g1[v] = data + 2.0f * args.fin.lambda_single * x1[v];
  };
  if (SYM) {
    // the ones slot's column: the single-field gradient
    if (col0 <= nat && nat < col0 + 128) {
      float v = 0.0f;
#pragma unroll
      for (int i = 0; i < 128; ++i) v = i == nat - col0 ? acc[i] : v;
      if (row < (kQ - 1) * L) single(row, v);
    }
    // columns of the same alignment column as this row
    int self = (row - col0) % L;
    if (self < 0) self += L;
#pragma unroll
    for (int i = 0; i < 128; ++i)
      if (i == self) {
        acc[i] = 0.0f;
        self += L;
      }
  } else if (row0 <= nat && nat < row0 + 32) {
    if (row == nat) {
#pragma unroll
      for (int i = 0; i < 128; ++i)
        if (col0 + i < (kQ - 1) * L) single(col0 + i, acc[i]);
    }
  }
  if (col0 + 128 > nat) {
#pragma unroll
    for (int i = 0; i < 128; ++i)
      if (col0 + i >= nat) acc[i] = 0.0f;
  }
  if (SYM && !diagonal) {
    // rows of a tile above the diagonal are real slots (only the last block is not full)
    float *p = g2 + col0 * pitch + row;
#pragma unroll
    for (int i = 0; i < 128; ++i, p += pitch) red_add_if(p, acc[i], col0 + i < nat);
  }
  float *const d = g2 + col0 + 4 * (lane & 3);
#pragma unroll
  for (int cb = 0; cb < 8; ++cb) {
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c)
      *reinterpret_cast<float4 *>(Tb + lane * 16 + ((c ^ (lane >> 1)) & 3) * 4) =
          make_float4(acc[cb * 16 + 4 * c], acc[cb * 16 + 4 * c + 1], acc[cb * 16 + 4 * c + 2],
                      acc[cb * 16 + 4 * c + 3]);
    __syncwarp();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int r = 8 * it + (lane >> 2);
      const float4 v = *reinterpret_cast<const float4 *>(Tb + r * 16 + (((lane & 3) ^ (r >> 1)) & 3) * 4);
      // (a 16-byte group that straddles 21 L adds zeros to a padding state)
      const bool in = row0 + r < nat && col0 + cb * 16 + 4 * (lane & 3) < nat;
      float *p = d + (row0 + r) * pitch + cb * 16;
      if (args.vec) {
        red_add4_if(p, v, in);
      } else {
        red_add_if(p, v.x, in);
        red_add_if(p + 1, v.y, in);
        red_add_if(p + 2, v.z, in);
        red_add_if(p + 3, v.w, in);
      }
    }
  }
}

// The record into the pinned copy of a host that waits for this evaluation: no copy
// behind the last kernel.  The host cleared the status; only an error is written, so that
// this never covers one that the same kernel records on its own.
__device__ __forceinline__ void finalize_host(const FinalizeArgs &args, double fx, double data) {
  args.host->fx = fx;
  args.host->f_data = data;
  args.host->reg = fx - data;
  const int status = *reinterpret_cast<const volatile int *>(&args.out->status);
  if (status) *reinterpret_cast<volatile int *>(&args.host->status) = status;
}

}  // namespace ccm
