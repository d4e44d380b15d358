// Integer tensor-core evaluation (CCM_PATH_TC_I8X3): the same two contractions as
// the split-bf16 path (ccm_tc.cu), with 8-bit operands and exact 32-bit integer
// accumulation on tcgen05 (kind::i8, cta_group::2).
//
// Fixed-point digits.  A value v with scale 2^e (|v| <= 2^e) is represented by the
// integer Q = clamp(rint(v * 2^(21 - e)), -2^21, 2^21 - 1) and stored as three
// bytes: d0 = Q >> 14 (signed, -128..127), d1 = (Q >> 7) & 127, d2 = Q & 127, so
// that Q = d0 * 2^14 + d1 * 2^7 + d2.  The one-hot operand is stored twice, as
// unsigned bytes 1 and 128, and the contractions accumulate
//   hi = sum O1 * d0,   lo = sum O128 * d1 + sum O1 * d2 = sum O * (Q & 0x3fff)
// in two s32 TMEM accumulators; sum O * Q = hi * 2^14 + lo exactly.  W takes one
// power-of-two scale per coupling column (a, j) (its column maximum rounded up),
// R = w (P - onehot), |R| < 1, takes the scale 1.  Quantisation error: at most
// 2^-22 of the column scale per element; modelled against FP64 it gives a 3x
// smaller gradient error than the hi+lo bf16 split, and the sums are exact.
// Per K element the tensor cores do three 8-bit products (at twice the bf16
// rate) where the split-bf16 path does two bf16 products: 3/4 of the cycles.
//
// One evaluation: on the dense path colmax (+ the fused CG step), prep (digits of W,
// g2 <- 2 l2 x, sum x^2), forward, backward, finalize (shared with ccm_tc.cu); on the
// sparse path four launches, scan (colmax, step, g2, sum x^2), digits, forward, backward
// (with the sums of f and g1).
#include <cfloat>
#include <cmath>
#include <type_traits>

#include <cuda_bf16.h>

#include "ccm_bwd_out.cuh"
#include "ccm_internal.cuh"
#include "ccm_layout.cuh"
#include "ccm_ptx.cuh"

namespace ccm {

constexpr int kI8FracBits = 21;

__device__ __forceinline__ uint8_t *i8_align1024(uint8_t *p) {
  const uint32_t s = smem_u32(p);
  return p + ((1024u - (s & 1023u)) & 1023u);
}

__device__ __forceinline__ void i8_record_error(int *status, int bit, int *abort_flag) {
  atomicOr(status, bit);
  *reinterpret_cast<volatile int *>(abort_flag) = 1;
}

__device__ __forceinline__ bool i8_aborted(const int *abort_flag) {
  return *reinterpret_cast<const volatile int *>(abort_flag) != 0;
}

// 2^s as a float, s in [-126, 127].
__device__ __forceinline__ float pow2f(int s) { return __int_as_float((s + 127) << 23); }
inline float pow2_host(int s) { return std::ldexp(1.0f, s); }

// Smallest e with 2^e >= m for the float m with bits `mbits` (m >= 0), limited to
// [-100, 127] so that 2^(21 - e) stays a normal float; 0 for m == 0.
__device__ __forceinline__ int col_exponent(uint32_t mbits) {
  if (mbits == 0) return 0;
  const int E = (int)(mbits >> 23) - 127;
  const int e = (mbits & 0x7FFFFFu) ? E + 1 : E;
  return max(e, -100);
}

// ---------------------------------------------------------------- colmax
// Column maxima of |W| over the 21 L rows (b, k), per coupling column c = a*L + j
// (a < 21), as float bits with atomicMax (|v| >= 0 orders like its bits).  Block
// (bx, by): 256 consecutive columns c of a 32 L row, rows [by*R, by*R + R).
// STEP = true also takes the CG trial step: v = fmaf(alpha, s, x) is written to
// xt for every element of x (the last row of blocks steps the single fields).
// cols = 21 L instead of 32 L leaves out the padding states (a solve that keeps
// them zero in x, s and xt).
template <bool STEP>
__global__ void __launch_bounds__(256) i8_colmax_kernel(const float *__restrict__ x,
                                                        const float *__restrict__ s,
                                                        const double *__restrict__ alpha,
                                                        float *__restrict__ xt,
                                                        uint32_t *__restrict__ colmax, int L,
                                                        long long nsp, int rows_per_block,
                                                        int cols) {
  griddep_wait();
  griddep_launch();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int w32 = kQPad * L;
  float a = 0.0f;
  if (STEP) {
    a = (float)alpha[0];
    if (blockIdx.y == gridDim.y - 1) {
      for (long long i = c; i < nsp; i += (long long)gridDim.x * blockDim.x)
        xt[i] = fmaf(a, s[i], x[i]);
      return;
    }
  }
  if (c >= cols) return;  // cols = 32 L, or 21 L when the padding states are skipped
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(r0 + rows_per_block, kQ * L);
  float m = 0.0f;
  for (int r = r0; r < r1; ++r) {
    // rows in the reverse of the order in which prep reads them, so that prep's first
    // rows are the ones read last here and are still in L2
    const int row = kQ * L - 1 - r;
    const long long i = nsp + (long long)row * w32 + c;
    float v = x[i];
    if (STEP) {
      v = fmaf(a, s[i], v);
      xt[i] = v;
    }
    m = fmaxf(m, fabsf(v));
  }
  if (c < kQ * L && m > 0.0f) atomicMax(colmax + c, __float_as_uint(m));
}

// Per slot s of the dense path: the encoding factor 2^(21 - e) of the digits
// of its coupling column (e the column's exponent, from the maxima above), 0 for
// padding slots; read by prep.
__global__ void i8_scales_kernel(const uint32_t *__restrict__ colmax, float *__restrict__ enc,
                                 int L, int S) {
  using G = Groups256;
  griddep_wait();
  griddep_launch();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  const int t = s / G::kSlots, r = s % G::kSlots;
  float f = 0.0f;
  if (r < G::kUsed) {
    const int a = r / G::kCols, j = t * G::kCols + r % G::kCols;
    if (j < L) f = pow2f(kI8FracBits - col_exponent(colmax[a * L + j]));
  }
  enc[s] = f;
}

// Operand storage of the sparse forward.  Every operand tile a stage needs is
// stored contiguously in global memory as the exact shared-memory image the
// MMA reads (swizzle included), so that one TMA box of 256-byte rows moves it;
// tiles with 16-, 32- or 64-byte rows cost one TMA request per row and leave the
// kernel bound by the L1/TMA request rate.  KB = KP / 128 K blocks.
//   A (compressed one-hot, 128 rows x 64 bytes, 64-byte swizzle): tile
//     (m128, kb) at ((m128 * KB + kb) * 128 + r) * 64; 16-byte chunk c of row r
//     stored at chunk c ^ ((r >> 1) & 3).
//   E (metadata, 128 rows x 16 bytes, no swizzle): tile (m128, kb) at
//     ((m128 * KB + kb) * 128 + r) * 16.
//   B (digits of W; per forward tile t and CTA half h, 128 K rows x 96 slots as
//     three atoms of 32 slots, 32-byte swizzle): atom i at
//     (((t * 2 + h) * KB + kb) * 3 + i) * 4096 + r * 32; chunk c of row r stored
//     at chunk c ^ ((r >> 2) & 1).
__host__ __device__ constexpr long long i8sp_a_offset(int n, int col, int KB) {
  // col: byte of the compressed row (0 .. KP/2)
  return (((long long)(n >> 7) * KB + (col >> 6)) * 128 + (n & 127)) * 64 +
         ((((col >> 4) & 3) ^ (((n & 127) >> 1) & 3)) << 4) + (col & 15);
}
__host__ __device__ constexpr long long i8sp_e_offset(int n, int byte, int KB) {
  return (((long long)(n >> 7) * KB + (byte >> 4)) * 128 + (n & 127)) * 16 + (byte & 15);
}
__host__ __device__ constexpr long long i8sp_b_offset(int kr, int s, int KB) {
  // kr: K row (l * 21 + q), s: slot of the 192-slot groups
  const int t = s / Groups192::kSlots, c = s % Groups192::kSlots;
  const int h = c / 96, i = (c % 96) >> 5, x = c & 31, r = kr & 127;
  return ((((long long)t * 2 + h) * KB + (kr >> 7)) * 3 + i) * 4096 + r * 32 +
         ((((x >> 4) ^ (r >> 2)) & 1) << 4) + (x & 15);
}

// ---------------------------------------------------------------- scan and digits
// The sparse path's first two kernels.
//
// i8sp_scan_kernel, one pass over x (row blocks of its 21 L coupling rows, four columns
// per thread, eight rows of loads in flight): column maxima of |W| into cmacc (float
// bits, atomicMax; zero between evaluations), sum x^2 partials (FP64 squares: float ones
// of four columns at a time are no faster), the regulariser gradient g2 <- g2_scale * x2
// (the backward adds C to it), and, STEP, the CG trial step v = fmaf(alpha, s, x) into xt
// (the last row of blocks steps the single fields), in a solve's trial after the update
// of s.  It also clears the result record.
// Rows go in K-row order k * 21 + b backwards, so that the digits kernel's first rows
// are the ones read last here and are still in L2.  HBM-bound.  Together with the
// digits kernel 110 us at L = 253, N = 7001 and 144 us at L = 300; the column-maximum,
// factor and row-per-block digit kernels before them took 226 us (scalar loads where
// 4 does not divide L) and 165 us.  (The backward writing g2_scale * x2 + C itself, or
// filling g2 while its MMAs run, saves this kernel 20 us at L = 300 and costs the
// backward 20-60: its loads and stores share the L2 port with the operand stream.)
template <bool STEP>
__global__ void __launch_bounds__(256) i8sp_scan_kernel(I8ScanArgs args) {
  griddep_wait();
  griddep_launch();
  const int L = args.L, nreal = kQ * L;
  const int c = (blockIdx.x * 256 + threadIdx.x) * 4;
  float alpha = 0.0f, beta = 0.0f;
  int mode = 0;  // of the direction update
  const float *x = args.x, *gp = nullptr;
  float *xt = args.xt, *g2 = args.g2, *const s = args.s;
  if (STEP) {
    alpha = (float)args.alpha[0];
    if (args.sw.parity) {
      const int q = *args.sw.parity;
      mode = *args.dir_mode;
      beta = (float)*args.beta;
      x = args.sw.at_x(q);
      xt = args.sw.at_x(1 - q);
      gp = args.sw.at_g(q);
      g2 = args.sw.at_g(1 - q) + args.nsp;
    }
  }
  auto direct = [&](float sv, float gv) { return mode == 1 ? -gv : fmaf(beta, sv, -gv); };
  if (STEP && blockIdx.y == gridDim.y - 1) {
    for (long long i = blockIdx.x * 256 + threadIdx.x; i < args.nsp; i += gridDim.x * 256LL) {
      float sv = s[i];
      if (mode) s[i] = sv = direct(sv, gp[i]);
      xt[i] = fmaf(alpha, sv, x[i]);
    }
    return;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < args.out_vecs)
    reinterpret_cast<uint4 *>(args.out)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
  float m[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  double acc = 0.0;
  if (c < args.cols) {
    // (cols = 21 L: the group that straddles 21 L reaches up to three padding states,
    // which are zero then)
    const float *x2 = x + args.nsp + c;
    auto load = [&](const float *p) {
      return args.vec ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
    };
    auto store = [&](float *p, float4 v) {
      if (args.vec) *reinterpret_cast<float4 *>(p) = v;
      else { p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w; }
    };
    const int r0 = blockIdx.y * args.rows_per_block;
    const int r1 = min(r0 + args.rows_per_block, nreal);
    constexpr int kU = STEP ? 4 : 8;
    for (int r = r0; r < r1; r += kU) {
      float4 v[kU], sv[STEP ? kU : 1];
      long long at[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int rr = nreal - 1 - min(r + u, r1 - 1);
        at[u] = ((long long)(rr % kQ) * L + rr / kQ) * kQPad * L;
        v[u] = load(x2 + at[u]);
        if (STEP) sv[u] = load(s + args.nsp + c + at[u]);
      }
      if (STEP && mode) {
        float4 gv[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) gv[u] = load(gp + args.nsp + c + at[u]);
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          sv[u] = make_float4(direct(sv[u].x, gv[u].x), direct(sv[u].y, gv[u].y),
                              direct(sv[u].z, gv[u].z), direct(sv[u].w, gv[u].w));
          if (r + u < r1) store(s + args.nsp + c + at[u], sv[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if (r + u >= r1) break;
        if (STEP) {
          v[u] = make_float4(fmaf(alpha, sv[u].x, v[u].x), fmaf(alpha, sv[u].y, v[u].y),
                             fmaf(alpha, sv[u].z, v[u].z), fmaf(alpha, sv[u].w, v[u].w));
          store(xt + args.nsp + c + at[u], v[u]);
        }
        acc += ((double)v[u].x * v[u].x + (double)v[u].y * v[u].y) +
               ((double)v[u].z * v[u].z + (double)v[u].w * v[u].w);
        m[0] = fmaxf(m[0], fabsf(v[u].x));
        m[1] = fmaxf(m[1], fabsf(v[u].y));
        m[2] = fmaxf(m[2], fabsf(v[u].z));
        m[3] = fmaxf(m[3], fabsf(v[u].w));
        const float k = args.g2_scale;
        store(g2 + at[u] + c, make_float4(k * v[u].x, k * v[u].y, k * v[u].z, k * v[u].w));
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c + e < nreal && m[e] > 0.0f) atomicMax(args.cmacc + c + e, __float_as_uint(m[e]));
  }
  __shared__ double red[8];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int w = 0; w < 8; ++w) sum += red[w];
    args.part_reg[blockIdx.y * gridDim.x + blockIdx.x] = sum;
  }
}

// i8sp_digits_kernel: the three digits of W in the forward's tiled storage
// (i8sp_b_offset).  A block takes `gpb` slot groups (9 gpb alignment columns with their
// 21 states) and a run of K rows, ROWS at a time: a thread's elements are the
// same columns of every row, so that their index arithmetic and encoding factors are
// computed once; consecutive threads read runs of 9 gpb floats.  The fixed-point
// integers go through shared memory in slot order (groups 200 words apart, rows an odd
// multiple of 4 words apart modulo 32: no bank conflict), and 16 consecutive threads
// write 256 contiguous bytes of a tile.  The first row of blocks also copies the column
// maxima to `colmax`, which the forward reads: cmacc is cleared by the backward.
// ROWS: eight, or four where eight make less than eight blocks per SM (L <= 89; L = 60
// 16.2 us for both kernels with four, 18.3 with eight; L = 300 144 with eight, 171 with four).
// Small blocks, two groups each: the barriers between a step's loads, conversion and
// stores stop 128 threads, not 384, and eight blocks fill an SM (scan and digits with
// eight groups and 384 threads a block: 50 us at L = 150, 159 at L = 300; so 43 and 144;
// one group and 64 threads 46 and 151).  Loads of the next step in flight during the
// stores, or registers capped for more blocks, spill and cost 5-9 us at L = 300.
constexpr int kDigThreads = 128, kDigRows = 8, kDigRowsFew = 4, kDigGroups = 2, kDigGroupWords = 200;
constexpr int dig_row_words(int gpb) { return (gpb * kDigGroupWords + 31) / 32 * 32 + 4; }
template <int ROWS>
__global__ void __launch_bounds__(kDigThreads) i8sp_digits_kernel(I8DigitsArgs args) {
  extern __shared__ __align__(16) int qs[];  // ROWS rows of dig_row_words(gpb)
  griddep_wait();
  griddep_launch();
  constexpr int kE = (kDigGroups * Groups192::kUsed + kDigThreads - 1) / kDigThreads;
  const int L = args.L, gpb = args.gpb, cols = gpb * Groups192::kCols;
  const int t0 = blockIdx.x * gpb, j0 = t0 * Groups192::kCols;
  const int row_words = dig_row_words(gpb);
  int off[kE], slot[kE];
  float enc[kE];
#pragma unroll
  for (int u = 0; u < kE; ++u) {
    const int e = threadIdx.x + u * kDigThreads;
    const int a = e / cols, jj = e % cols, j = j0 + jj;
    off[u] = -1;
    slot[u] = 0;
    enc[u] = 0.0f;
    if (a < kQ && j < L) {
      off[u] = a * L + j;
      slot[u] = jj / Groups192::kCols * kDigGroupWords + a * Groups192::kCols + jj % Groups192::kCols;
      const uint32_t m = args.cmacc[off[u]];
      enc[u] = pow2f(kI8FracBits - col_exponent(m));
      if (blockIdx.y == 0) args.colmax[off[u]] = m;
    }
  }
  // padding slots of the groups stay zero
  for (int i = threadIdx.x; i < ROWS * row_words; i += kDigThreads) qs[i] = 0;
  const int k_rows = kQ * L;
  const float *x2 = args.sw.parity ? args.sw.at_x(1 - *args.sw.parity) + args.nsp : args.x2;
  const int r1 = min((int)(blockIdx.y + 1) * args.rows_per_block, k_rows);
  for (int r0 = blockIdx.y * args.rows_per_block; r0 < r1; r0 += ROWS) {
    float v[ROWS][kE];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int kr = min(r0 + i, r1 - 1);
      const float *row = x2 + ((long long)(kr % kQ) * L + kr / kQ) * kQPad * L;
#pragma unroll
      for (int u = 0; u < kE; ++u) v[i][u] = off[u] >= 0 ? row[off[u]] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int u = 0; u < kE; ++u)
        if (off[u] >= 0) {
          const int q = __float2int_rn(v[i][u] * enc[u]);  // exact scaling
          qs[i * row_words + slot[u]] = min(max(q, -(1 << kI8FracBits)), (1 << kI8FracBits) - 1);
        }
    __syncthreads();
    // 16 slots of one row per thread: chunk (group, 32-slot atom), row, half
    const int chunks = gpb * 6 * 2 * ROWS;
    for (int u = threadIdx.x; u < chunks; u += kDigThreads) {
      const int hc = u & 1, i = (u >> 1) & (ROWS - 1), ga = u / (2 * ROWS);
      const int g = ga / 6, c = ga % 6 * 32 + hc * 16;
      if (r0 + i >= r1 || t0 + g >= args.T) continue;
      const int *from = qs + i * row_words + g * kDigGroupWords + c;
      uint32_t p0[4], p1[4], p2[4];
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4) {
        const int4 qv = *reinterpret_cast<const int4 *>(from + e4 * 4);
        // byte e of each word = digit of element e (as in the dense forward's R digits)
        auto pack = [](int b0, int b1, int b2, int b3) {
          return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
        };
        p0[e4] = pack(qv.x >> 14, qv.y >> 14, qv.z >> 14, qv.w >> 14);
        p1[e4] = pack(qv.x >> 7, qv.y >> 7, qv.z >> 7, qv.w >> 7) & 0x7F7F7F7Fu;
        p2[e4] = pack(qv.x, qv.y, qv.z, qv.w) & 0x7F7F7F7Fu;
      }
      const long long at = i8sp_b_offset(r0 + i, (t0 + g) * Groups192::kSlots + c, args.KB);
      *reinterpret_cast<uint4 *>(args.wdig[0] + at) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
      *reinterpret_cast<uint4 *>(args.wdig[1] + at) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
      *reinterpret_cast<uint4 *>(args.wdig[2] + at) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
    }
  }
}

// ---------------------------------------------------------------- prep
// The dense path's preparation.  One block per row (b, k) of W, as tc_prep: g2 <-
// g2_coef * lambda2 * x, the FP64 partial of sum x^2, and row s(b, k) of the three digit
// matrices of Wperm (16 slots per thread, one 16-byte store per digit matrix).  args.S
// is the row length.  The row is staged in shared memory in slot order, so that the
// digit pass reads 16 consecutive slots per thread (vector loads, no index arithmetic)
// with their per-slot factors.
__global__ void __launch_bounds__(256) i8_prep_kernel(const float *__restrict__ x2,
                                                      float *__restrict__ g2, I8PrepArgs args) {
  griddep_wait();
  griddep_launch();
  extern __shared__ __align__(16) float xrow[];  // S floats: the row in slot order
  const int L = args.L;
  using G = Groups256;
  const int row = blockIdx.x;
  const int b = row / L, k = row % L;
  const long long base = (long long)row * kQPad * L;
  const float two_l2 = args.g2_coef * args.lambda_pair;
  const int nreal = kQ * L;
  double acc = 0.0;
  if (args.vec) {
    const float4 *src = reinterpret_cast<const float4 *>(x2 + base);
    float4 *dst = reinterpret_cast<float4 *>(g2 + base);
    const int n4 = args.ncols / 4, nreal4 = nreal / 4;
    constexpr int kU = 4;
    for (int i0 = threadIdx.x; i0 < n4; i0 += kU * blockDim.x) {
      float4 v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int i = i0 + u * blockDim.x;
        v[u] = i < n4 ? __ldcs(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int i = i0 + u * blockDim.x;
        if (i < n4) {
          acc += ((double)v[u].x * v[u].x + (double)v[u].y * v[u].y) +
                 ((double)v[u].z * v[u].z + (double)v[u].w * v[u].w);
          if (i < nreal4) {
            // c = 4i = a L + j, j a multiple of 4: the four elements share a, and
            // j .. j+3 stay inside the row's column range
            const int c = 4 * i;
            const int a = (int)(((float)c + 0.5f) * args.inv_L);
            const int j = c - a * L;
            const float vv[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) xrow[G::slot_of(a, j + e)] = vv[e];
          }
          __stcs(dst + i, make_float4(two_l2 * v[u].x, two_l2 * v[u].y, two_l2 * v[u].z,
                                      two_l2 * v[u].w));
        }
      }
    }
  } else {
    for (int i = threadIdx.x; i < args.ncols; i += blockDim.x) {
      const float v = x2[base + i];
      acc += (double)v * v;
      if (i < nreal) xrow[G::slot_of(i / L, i % L)] = v;
      g2[base + i] = two_l2 * v;
    }
  }
  __syncthreads();
  const long long srow = (long long)G::slot_of(b, k) * args.S;
  for (int u = threadIdx.x; u < args.S / 16; u += blockDim.x) {
    uint32_t p0[4], p1[4], p2[4];
#pragma unroll
    for (int e4 = 0; e4 < 4; ++e4) {
      const float4 xv = reinterpret_cast<const float4 *>(xrow)[u * 4 + e4];
      const float4 fv = __ldg(reinterpret_cast<const float4 *>(args.enc) + u * 4 + e4);
      const float xs[4] = {xv.x, xv.y, xv.z, xv.w}, fs[4] = {fv.x, fv.y, fv.z, fv.w};
      int qv[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // padding slots have factor 0 and are never staged: their digits are 0
        const int q = fs[e] != 0.0f ? __float2int_rn(xs[e] * fs[e]) : 0;  // exact scaling
        qv[e] = min(max(q, -(1 << kI8FracBits)), (1 << kI8FracBits) - 1);
      }
      // byte e of each word = digit of element e (as in the forward's R digits)
      auto pack = [](int b0, int b1, int b2, int b3) {
        return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
      };
      p0[e4] = pack(qv[0] >> 14, qv[1] >> 14, qv[2] >> 14, qv[3] >> 14);
      p1[e4] = pack(qv[0] >> 7, qv[1] >> 7, qv[2] >> 7, qv[3] >> 7) & 0x7F7F7F7Fu;
      p2[e4] = pack(qv[0], qv[1], qv[2], qv[3]) & 0x7F7F7F7Fu;
    }
    const long long off = srow + (long long)u * 16;
    *reinterpret_cast<uint4 *>(args.wdig[0] + off) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
    *reinterpret_cast<uint4 *>(args.wdig[1] + off) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
    *reinterpret_cast<uint4 *>(args.wdig[2] + off) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
  }
  __shared__ double red[32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += red[w];
    args.part_reg[row] = sum;
  }
}

// Backward operands of the sparse path.  Slots in natural order, s = q L + l (the
// row and column index of the coupling matrix itself), the ones slot at 21 L, padded
// to SB = a multiple of 256; rows n of the alignment are the contraction index and
// lie contiguous (K-major).  The 128-slot x 32-row tile (sb = s / 128, kb = n / 32)
// that one pipeline stage of one CTA reads is stored as the shared-memory image the
// MMA reads, 32 bytes per slot with the 32-byte swizzle (16-byte half h of slot r
// stored at half h ^ ((r >> 2) & 1)); the matrices that a stage needs side by side
// follow one another, so that one TMA box of 256-byte rows moves them:
//   one-hot  x1 | x128      8 KB at (sb * KB + kb) * 8192,  KB = Npad / 32
//   digits   r0 | r1 | r2  12 KB at (sb * KB + kb) * 12288
// Natural slots make a tile's rows and columns contiguous runs of the gradient (see
// the output phase), K-major tiles let a warp of the forward's epilogue, whose lanes
// are 32 consecutive rows n, write one full 32-byte sector per slot and digit for
// any order of the slots.
constexpr int kNatTile = 128 * 32;
__host__ __device__ constexpr long long i8nat_offset(int n, int s, int KB, int mats) {
  return ((long long)(s >> 7) * KB + (n >> 5)) * (mats * kNatTile) + (s & 127) * 32 +
         ((n & 31) ^ ((s & 4) << 2));
}

// x1 | x128 one-hot of the backward: 1 / 128 where column l of row n holds state q,
// and in the ones slot of every real row.  One thread per (slot, 32 rows):
// consecutive threads read consecutive bytes of the alignment.
__global__ void __launch_bounds__(128) i8nat_onehot_kernel(const uint8_t *__restrict__ msa,
                                                           uint8_t *__restrict__ o, int L, int N,
                                                           int KB) {
  const int s = blockIdx.y * 128 + threadIdx.x, kb = blockIdx.x;
  const int q = s / L, l = s % L;
  uint32_t v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int n = kb * 32 + i;
    bool one = false;
    if (n < N) one = s == kQ * L || (s < kQ * L && msa[(long long)n * L + l] == q);
    v[i >> 2] |= (one ? 1u : 0u) << (8 * (i & 3));
  }
  uint4 *p = reinterpret_cast<uint4 *>(o + i8nat_offset(kb * 32, s, KB, 2) - ((s & 4) << 2));
  const int h = (s >> 2) & 1;
  p[h] = make_uint4(v[0], v[1], v[2], v[3]);
  p[h ^ 1] = make_uint4(v[4], v[5], v[6], v[7]);
  p += kNatTile / 16;
  p[h] = make_uint4(v[0] << 7, v[1] << 7, v[2] << 7, v[3] << 7);
  p[h ^ 1] = make_uint4(v[4] << 7, v[5] << 7, v[6] << 7, v[7] << 7);
}

// One-hot operands of the dense integer path: O1[n][s] = 1 and O128[n][s] = 128 where
// the state of column l(s) in row n is q(s), and in the ones slot of every real row;
// 0 elsewhere.
__global__ void i8_onehot_kernel(const uint8_t *__restrict__ msa, uint8_t *__restrict__ o1,
                                 uint8_t *__restrict__ o128, int L, int N, int S, int Npad) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)Npad * S) return;
  const int n = (int)(idx / S), s = (int)(idx % S);
  const int t = s / kGroupSlots, r = s % kGroupSlots;
  bool one = false;
  if (n < N) {
    if (s == kOnesSlot) {
      one = true;
    } else if (r < kGroupUsed) {
      const int q = r / kGroupCols, l = t * kGroupCols + r % kGroupCols;
      one = l < L && msa[(long long)n * L + l] == q;
    }
  }
  o1[idx] = one ? 1 : 0;
  o128[idx] = one ? 128 : 0;
}

}  // namespace ccm

namespace ccm {

// hi * 2^14 + lo rounded once to float, for |hi + (lo >> 14)| < 2^24 (the forward: at
// most 129 L; the backward: |hi| <= 2^23, lo >> 14 < 2^17): the low 14 bits of lo and
// the rest, carried into hi, are both exact floats, so the one rounding is the FMA's.
// The same float as a conversion of the 64-bit sum, which runs at a quarter of the rate.
__device__ __forceinline__ float i8_merge_exact(uint32_t hi, uint32_t lo) {
  const int h = (int)hi + ((int)lo >> 14);
  return fmaf(__int2float_rn(h), 16384.0f, __int2float_rn((int)(lo & 16383u)));
}

// ---------------------------------------------------------------- forward
// Pair tiles of 256 rows x 256 slots as in tc_forward.  Per tile the MMAs run in
// two phases: first the low digits into `lo` (O128 x d1 + O1 x d2), then the high
// digit into `hi` (O1 x d0).  The epilogue merges z = (hi * 2^14 + lo) * scale + V
// into float logits written back over `hi`, releases `lo` (the next tile's low
// phase may start), runs the softmax passes on `hi`, writes the digits of R and
// releases `hi`.  TMEM: hi = columns [0, 256), lo = [256, 512).
constexpr int kI8BM = 128, kI8PairM = 256, kI8BN = 256, kI8HalfN = 128, kI8FwdBK = 64;
constexpr int kI8Threads = 320;

struct I8FwdSmem {
  static constexpr int kStages = 6;
  static constexpr int kTile = kI8BM * kI8FwdBK;  // 8 KB: A 128 rows x 64 B, B 64 rows x 128 B
  static constexpr int kOffA1 = 0;
  static constexpr int kOffA128 = kTile;
  static constexpr int kOffB = 2 * kTile;          // lo phase: d1, d2
  // hi phase: two K blocks per stage: O1 (kb) at 0, O1 (kb+1) at kTile, d0 (kb) at
  // 2 kTile, d0 (kb+1) at 3 kTile, so that a stage feeds four MMAs in both phases
  static constexpr int kStage = 4 * kTile;
  static constexpr int kBarOff = kStages * kStage;
  static constexpr int kTabOff = kBarOff + 256;    // per tile: scale[256], V[256]
  static constexpr int kXOff = kTabOff + 2 * kGroupSlots * 4;
  static constexpr int kXBytes = 2 * kI8BM * 2 * kGroupCols * 4;  // (max, sum) per half
  static constexpr int kTotal = kXOff + kXBytes + 1024;
};

// Epilogue of one tile for one warp (TMEM lane quarter q, column half H: columns
// 128 H .. 128 H + 127 of the tile).  Three passes over TMEM, one exp per element:
//   merge: z = (hi * 2^14 + lo) * scale + V (exact integer sum, one rounding),
//          written over hi; per alignment column jj the maximum m of the own
//          states and the logit of the observed state; then `lo` is released;
//   B:     e = exp(z - m) written over z, s = sum e;
//          (m, s) exchanged with the partner warp (same rows, other half):
//          M = max(m, m'), S = s exp(m - M) + s' exp(m' - M) (same order in both
//          halves), lse = M + log S;
//   C:     P = e * exp(m - M) / S, R = w (P - onehot) as its three digits.
// hi * 2^14 + lo, rounded once to float.  A row of the one-hot operand holds L
// ones, so |hi| <= 128 L and 0 <= lo <= 16383 L: with L <= kI8NarrowMaxL the exact
// sum lies in [-2^31, 2^31) and the 32-bit conversion (NARROW) gives the float the
// 64-bit one gives.
constexpr int kI8NarrowMaxL = 1024;
template <bool NARROW>
__device__ __forceinline__ float i8_merge_digits(uint32_t hi, uint32_t lo) {
  if constexpr (NARROW) {
    return __int2float_rn((int)(hi * 16384u + lo));
  } else {
    return __ll2float_rn((long long)(int)hi * 16384 + (long long)(int)lo);
  }
}

template <int H, bool NARROW>
__device__ __forceinline__ void i8_fwd_epilogue_tile(const I8FwdArgs &args, uint32_t t_hi,
                                                     uint32_t t_lo, const float *tab_scale,
                                                     const float *tab_v, float *xbuf, int q,
                                                     int lane, int n, int t, long long part,
                                                     uint32_t lo_bar) {
  constexpr int kChunks = kGroupSlots / 64;  // 32-column chunks per half
  const int L = args.L;
  const int j0 = t * kGroupCols;
  const bool live = n < args.N;
  const float wn = live ? args.w[n] : 0.0f;
  const int row = q * 32 + lane;
  const int pair_bar = 2 + q;
  int xr[kGroupCols];
#pragma unroll
  for (int jj = 0; jj < kGroupCols; ++jj) {
    const int j = j0 + jj;
    xr[jj] = (live && j < L) ? (int)args.msa[(long long)n * L + j] : -1;
  }
  float mx[kGroupCols], tg[kGroupCols], se[kGroupCols];
#pragma unroll
  for (int jj = 0; jj < kGroupCols; ++jj) { mx[jj] = -FLT_MAX; tg[jj] = 0.0f; se[jj] = 0.0f; }
  // merge + maxima
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int cc = kChunks * H + c;
    uint32_t vh[32], vl[32];
    __syncwarp();
    tmem_ld32(t_hi + cc * 32, vh);
    tmem_ld32(t_lo + cc * 32, vl);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int col = cc * 32 + i;
      const float z = fmaf(i8_merge_digits<NARROW>(vh[i], vl[i]), tab_scale[col], tab_v[col]);
      vh[i] = __float_as_uint(z);
      if (col < kGroupUsed) {
        const int a = col / kGroupCols, jj = col % kGroupCols;
        mx[jj] = fmaxf(mx[jj], z);
        if (xr[jj] == a) tg[jj] = z;
      }
    }
    tmem_st32(t_hi + cc * 32, vh);
  }
  tmem_wait_st();
  tc_fence_before();
  __syncwarp();
  // the next tile's low phase may start
  if (lane == 0) mbar_arrive_remote(lo_bar);
  // B: e = exp(z - m), sum
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int cc = kChunks * H + c;
    uint32_t v[32];
    __syncwarp();
    tmem_ld32(t_hi + cc * 32, v);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int col = cc * 32 + i;
      if (col < kGroupUsed) {
        const int jj = col % kGroupCols;
        const float e = expf(__uint_as_float(v[i]) - mx[jj]);
        se[jj] += e;
        v[i] = __float_as_uint(e);
      }
    }
    tmem_st32(t_hi + cc * 32, v);
  }
  float *mine = xbuf + (H * kI8BM + row) * (2 * kGroupCols);
  const float *other = xbuf + ((1 - H) * kI8BM + row) * (2 * kGroupCols);
#pragma unroll
  for (int jj = 0; jj < kGroupCols; ++jj) {
    mine[jj] = mx[jj];
    mine[kGroupCols + jj] = se[jj];
  }
  named_bar_sync(pair_bar, 64);
  double floss = 0.0;
  // R * 2^21 = e * cw - [observed] * won, with cw = w exp(m - M) / S * 2^21
  float cw[kGroupCols];
  const float won = live ? wn * args.r_enc : 0.0f;
#pragma unroll
  for (int jj = 0; jj < kGroupCols; ++jj) {
    const float mo = other[jj], so = other[kGroupCols + jj];
    const float M = fmaxf(mx[jj], mo);
    const float fa = expf(mx[jj] - M), fo = expf(mo - M);
    const float S = H == 0 ? se[jj] * fa + so * fo : so * fo + se[jj] * fa;
    const float lse = M + logf(S);
    cw[jj] = xr[jj] >= 0 ? (fa / S) * won : 0.0f;
    if (xr[jj] >= 0 && (xr[jj] * kGroupCols + jj) / (kGroupSlots / 2) == H)
      floss += (double)(wn * (lse - tg[jj]));
  }
  tmem_wait_st();
  // C: R = w (P - onehot), three digits per element
  const long long rbase = (long long)n * args.S + (long long)t * kGroupSlots;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int cc = kChunks * H + c;
    uint32_t v[32];
    __syncwarp();
    tmem_ld32(t_hi + cc * 32, v);
    tmem_wait_ld();
    uint32_t w0[8], w1[8], w2[8];
#pragma unroll
    for (int e4 = 0; e4 < 8; ++e4) {
      int qv[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = e4 * 4 + e;
        const int col = cc * 32 + i;
        float t = 0.0f;
        if (col < kGroupUsed) {
          const int a = col / kGroupCols, jj = col % kGroupCols;
          t = fmaf(__uint_as_float(v[i]), cw[jj], xr[jj] == a ? -won : 0.0f);
        }
        // |R| 2^-eR <= 1: only the top of the range needs the clamp (P rounding to 1)
        qv[e] = min(__float2int_rn(t), (1 << kI8FracBits) - 1);
      }
      // byte e of each word = digit of element e: d0 = q >> 14, d1 = (q >> 7) & 127,
      // d2 = q & 127 (two byte permutes per pair, one per word)
      auto pack = [](int b0, int b1, int b2, int b3) {
        return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
      };
      w0[e4] = pack(qv[0] >> 14, qv[1] >> 14, qv[2] >> 14, qv[3] >> 14);
      w1[e4] = pack(qv[0] >> 7, qv[1] >> 7, qv[2] >> 7, qv[3] >> 7) & 0x7F7F7F7Fu;
      w2[e4] = pack(qv[0], qv[1], qv[2], qv[3]) & 0x7F7F7F7Fu;
    }
    const long long off = rbase + cc * 32;
    st_global_v8(args.r[0] + off, w0);
    st_global_v8(args.r[1] + off, w1);
    st_global_v8(args.r[2] + off, w2);
  }
  for (int o = 16; o > 0; o >>= 1) floss += __shfl_xor_sync(0xffffffffu, floss, o);
  if (lane == 0) args.part_f[part * 8 + H * 4 + q] = floss;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kI8Threads, 1)
    i8_forward_kernel(const __grid_constant__ I8FwdMaps maps, I8FwdArgs args) {
  using SM = I8FwdSmem;
  constexpr int kStages = SM::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = i8_align1024(smem_raw);
  // full[] and the *_empty barriers are used in the leader only; empty[] and
  // acc_full in both CTAs (the leader's commits reach both)
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + SM::kBarOff);
  uint64_t *empty = full + kStages;
  uint64_t *acc_full = empty + kStages;
  uint64_t *lo_empty = acc_full + 1;
  uint64_t *hi_empty = lo_empty + 1;
  uint64_t *drain = hi_empty + 1;
  // a barrier that no thread ever arrives on: the epilogue waits on it instead
  // of on acc_full when a test asks for a wait that runs out (acc_wait_cycles)
  uint64_t *never = drain + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(never + 1);
  int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
  float *tab_scale = reinterpret_cast<float *>(smem + SM::kTabOff);
  float *tab_v = tab_scale + kGroupSlots;
  float *xbuf = reinterpret_cast<float *>(smem + SM::kXOff);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int n_tiles = args.m_tiles * args.T;
  const int k_blocks = args.S / kI8FwdBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(lo_empty, 16);
    mbar_init(hi_empty, 16);
    mbar_init(drain, 1);
    mbar_init(never, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&maps.a1);
    prefetch_tmap(&maps.a128);
    for (int i = 0; i < 3; ++i) prefetch_tmap(&maps.b[i]);
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  // the prologue above overlaps the previous kernel's tail; its outputs from here
  griddep_launch();
  griddep_wait();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t t_hi = tmem_base, t_lo = tmem_base + kI8BN;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer (both CTAs), in the MMA's order
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok && !i8_aborted(abort_flag); tile += npairs) {
        const int m = tile % args.m_tiles, t = tile / args.m_tiles;
        const int row0 = m * kI8PairM + (int)rank * kI8BM;
        const int col0 = t * kI8BN + (int)rank * kI8HalfN;
        for (int phase = 0; phase < 2 && ok; ++phase) {  // 0: low digits, 1: high digit
          for (int kb = 0; kb < k_blocks; kb += (phase == 0 ? 1 : 2), ++it) {
            const int stage = it % kStages;
            const uint32_t round = it / kStages;
            if (!mbar_wait(&empty[stage], (round & 1) ^ 1)) {
              i8_record_error(args.status, kErrFwdTimeout, abort_flag);
              ok = false;
              break;
            }
            uint8_t *st = smem + stage * SM::kStage;
            const uint32_t fb = mapa_shared(smem_u32(&full[stage]), 0);
            const int kx = kb * kI8FwdBK;
            if (phase == 0) {
              if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * 4 * SM::kTile);
              tma_load_2d_pair(st + SM::kOffA1, &maps.a1, fb, kx, row0);
              tma_load_2d_pair(st + SM::kOffA128, &maps.a128, fb, kx, row0);
              tma_load_2d_pair(st + SM::kOffB, &maps.b[1], fb, col0, kx);
              tma_load_2d_pair(st + SM::kOffB + SM::kTile, &maps.b[2], fb, col0, kx);
            } else {
              if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * 4 * SM::kTile);
              tma_load_2d_pair(st, &maps.a1, fb, kx, row0);
              tma_load_2d_pair(st + SM::kTile, &maps.a1, fb, kx + kI8FwdBK, row0);
              tma_load_2d_pair(st + 2 * SM::kTile, &maps.b[0], fb, col0, kx);
              tma_load_2d_pair(st + 3 * SM::kTile, &maps.b[0], fb, col0, kx + kI8FwdBK);
            }
          }
        }
      }
      const uint32_t issued = it;
      for (uint32_t r = (issued > kStages ? issued - kStages : 0); r < issued; ++r) {
        const bool w = rank == 0 ? mbar_wait(&full[r % kStages], (r / kStages) & 1)
                                 : mbar_wait(&empty[r % kStages], (r / kStages) & 1);
        if (!w) {
          i8_record_error(args.status, kErrFwdTimeout, abort_flag);
          break;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ---------------- MMA issuer (leader): 256 x 256 x 32 pair MMAs, u8 x s8 -> s32
      constexpr uint32_t idesc = idesc_i8_s32(kI8PairM, kI8BN, 0, 1, 0, 1);
      uint32_t it = 0;
      int local = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok && !i8_aborted(abort_flag);
           tile += npairs, ++local) {
        const uint32_t wpar = (local & 1) ^ 1;
        for (int phase = 0; phase < 2 && ok; ++phase) {
          if (!mbar_wait(phase == 0 ? lo_empty : hi_empty, wpar)) {
            i8_record_error(args.status, kErrFwdTimeout, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
          for (int kb = 0; kb < k_blocks; kb += (phase == 0 ? 1 : 2), ++it) {
            const int stage = it % kStages;
            const uint32_t round = it / kStages;
            if (!mbar_wait(&full[stage], round & 1)) {
              i8_record_error(args.status, kErrFwdTimeout, abort_flag);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t s0 = smem_u32(smem + stage * SM::kStage);
#pragma unroll
            for (int k32 = 0; k32 < kI8FwdBK / 32; ++k32) {
              if (phase == 0) {
                const uint64_t a1 = sdesc_sw64(s0 + SM::kOffA1 + k32 * 32, 16, 512);
                const uint64_t a128 = sdesc_sw64(s0 + SM::kOffA128 + k32 * 32, 16, 512);
                const uint64_t bA = sdesc_sw128(s0 + SM::kOffB + k32 * 32 * 128, SM::kTile, 1024);
                const uint64_t bB =
                    sdesc_sw128(s0 + SM::kOffB + SM::kTile + k32 * 32 * 128, SM::kTile, 1024);
                umma_i8_pair(t_lo, a128, bA, idesc, (kb | k32) != 0);
                umma_i8_pair(t_lo, a1, bB, idesc, 1);
              } else {
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                  const uint64_t a1 = sdesc_sw64(s0 + sub * SM::kTile + k32 * 32, 16, 512);
                  const uint64_t b0 = sdesc_sw128(s0 + (2 + sub) * SM::kTile + k32 * 32 * 128,
                                                  SM::kTile, 1024);
                  umma_i8_pair(t_hi, a1, b0, idesc, (kb | sub | k32) != 0);
                }
              }
            }
            umma_commit_pair(&empty[stage], 0x3);
          }
        }
        if (ok) umma_commit_pair(acc_full, 0x3);
      }
      umma_commit_pair(drain, 0x1);
      if (!mbar_wait(drain, 0)) i8_record_error(args.status, kErrFwdTimeout, abort_flag);
    }
  } else {
    // ---------------- epilogue (both CTAs): 8 warps, lane quarter q, column half
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int ethr = threadIdx.x - 64;
    const int L = args.L;
    const uint32_t lo_bar = mapa_shared(smem_u32(lo_empty), 0);
    const uint32_t hi_bar = mapa_shared(smem_u32(hi_empty), 0);

    int local = 0;
    for (int tile = pair; tile < n_tiles; tile += npairs, ++local) {
      // all eight warps finished the previous tile (tables free) and saw no abort
      if (named_bar_or(1, 256, i8_aborted(abort_flag))) break;
      const int m = tile % args.m_tiles, t = tile / args.m_tiles;
      {
        // slot tables of this tile: merge scale 2^(e - 21) and the single field V
        const int r = ethr;
        float sc = 0.0f, vv = 0.0f;
        if (r < kGroupUsed) {
          const int a = r / kGroupCols, j = t * kGroupCols + r % kGroupCols;
          if (j < L) {
            sc = pow2f(col_exponent(args.colmax[a * L + j]) - kI8FracBits);
            if (a < kQ - 1) vv = args.x1[a * L + j];
          }
        }
        tab_scale[r] = sc;
        tab_v[r] = vv;
      }
      named_bar_sync(1, 256);
      const int n = m * kI8PairM + (int)rank * kI8BM + q * 32 + lane;
      // (with acc_wait_cycles set, a wait that runs out by design: see `never`)
      const bool ok = args.acc_wait_cycles > 0 ? mbar_wait(never, 0, args.acc_wait_cycles)
                                               : mbar_wait(acc_full, local & 1);
      if (__any_sync(0xffffffffu, !ok)) {
        if (lane == 0) i8_record_error(args.status, kErrFwdTimeout, abort_flag);
        continue;
      }
      tc_fence_after();
      const uint32_t lq = (uint32_t)(q * 32) << 16;
      const long long part = (long long)tile * 2 + rank;
      const bool narrow = L <= kI8NarrowMaxL;
#define CCM_TILE_ARGS \
  args, t_hi + lq, t_lo + lq, tab_scale, tab_v, xbuf, q, lane, n, t, part, lo_bar
      if (half == 0 && narrow) i8_fwd_epilogue_tile<0, true>(CCM_TILE_ARGS);
      else if (half == 0) i8_fwd_epilogue_tile<0, false>(CCM_TILE_ARGS);
      else if (narrow) i8_fwd_epilogue_tile<1, true>(CCM_TILE_ARGS);
      else i8_fwd_epilogue_tile<1, false>(CCM_TILE_ARGS);
#undef CCM_TILE_ARGS
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(hi_bar);
    }
  }

  tc_fence_before();
  cluster_sync();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ---------------------------------------------------------------- sparse forward
// CCM_PATH_TC_I8SP.  The one-hot operand with its K order changed to
// k' = l * 21 + q (alignment column major): any four consecutive k' span at most
// two alignment columns, and a row has exactly one 1 per column, so every group
// of four holds at most two ones -- the 2:4 structured sparsity that
// tcgen05.mma.sp runs at twice the dense rate.  A is stored compressed (the two
// kept values of each group) with 4 bits of metadata per group: the kept
// positions i0 < i1 in bits 0-1 and 2-3, group c of a row in nibble c of the
// row's metadata bytes (low nibble first).  A group with a single 1 keeps it
// with a zero partner, an empty group keeps (0, 1) with two zeros.
// One thread per metadata byte (two groups, eight logical K).
__global__ void i8sp_onehot_kernel(const uint8_t *__restrict__ msa, uint32_t *__restrict__ ac1,
                                   uint32_t *__restrict__ ac128, uint8_t *__restrict__ meta,
                                   int L, int N, int KP, int Npad) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nb = KP / 8;
  if (idx >= (long long)Npad * nb) return;
  const int n = (int)(idx / nb), byte = (int)(idx % nb);
  uint32_t vals = 0, m = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = 2 * byte + h;
    int pos[2] = {0, 0}, cnt = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int k = 4 * c + p;
      if (n < N && k < kQ * L && msa[(long long)n * L + k / kQ] == k % kQ) {
        if (cnt < 2) pos[cnt] = p;
        ++cnt;
      }
    }
    int i0 = 0, i1 = 1, v0 = 0, v1 = 0;
    if (cnt >= 2) {
      i0 = pos[0]; i1 = pos[1]; v0 = 1; v1 = 1;
    } else if (cnt == 1) {
      if (pos[0] < 3) { i0 = pos[0]; i1 = 3; v0 = 1; }
      else { i0 = 2; i1 = 3; v1 = 1; }
    }
    m |= (uint32_t)(i0 | (i1 << 2)) << (4 * h);
    vals |= (uint32_t)(v0 | (v1 << 8)) << (16 * h);
  }
  // compressed row n: KP / 2 bytes, four per metadata byte (one aligned word)
  const int KB = KP / 128;
  meta[i8sp_e_offset(n, byte, KB)] = (uint8_t)m;
  const long long ao = i8sp_a_offset(n, 4 * byte, KB) >> 2;
  ac1[ao] = vals;
  ac128[ao] = vals * 128;  // the same with values 128
}

// As i8_forward_kernel on 256 x 192 tiles (Groups192, nine alignment columns per
// tile), with sparse MMAs (K = 64 logical per instruction).  Per 128 logical K
// the CTA holds A compressed as 128 rows x 64 bytes (64-byte swizzle), the
// metadata as 128 rows x 16 bytes (no swizzle), copied into TMEM by tcgen05.cp
// ahead of the MMAs that read it (the copy and the MMAs issue from one thread and
// execute in order; two metadata slots alternate), and B -- the digits of W with
// rows in the K order k' -- MN-major, 96 columns per CTA as three 32-byte
// swizzled atoms of 128 K rows.  Each of these is one TMA box of the tiled
// storage above (no TMA swizzle: the images are stored swizzled).
// One pass per tile: a stage holds everything one block of 128 logical K needs
// for the three digit products (A x1, A x128, B d0..d2, E; 54 KB), so the one-hot
// operand and its metadata cross L2 once per tile, not once per digit phase.  Two
// bounds lie close together (L = 300, N = 5000, 303 us; timing copies): the operand stream
// alone, with two of the six MMAs, 254 us (all SMs together are at L2's throughput: an L2
// prefetch makes it slower), and the MMAs alone, with 38 of the 54 KB loaded, 264 us
// (sparse MMAs issue at 106 cycles each, 96 ideal, and wait for the issuing thread).  A
// expanded into TMEM by four more warps (36 KB per block) took 304 us.  The epilogue takes
// the sums out of both accumulators into registers and releases them at once, so the
// next tile's MMAs overlap the softmax and the R digits.
// TMEM: hi = [0, 192), lo = [256, 448), metadata slots at 456 and 460.
constexpr int kSpBN = Groups192::kSlots, kSpBK = 128;
constexpr int kSpHalf = kSpBN / 2;  // tile columns of an epilogue warp

struct I8SpSmem {
  static constexpr int kStages = 3;
  static constexpr int kA = kI8BM * kSpBK / 2;  // 8 KB
  static constexpr int kAtom = kSpBK * 32;      // 4 KB: 128 K rows x 32 columns
  static constexpr int kB = 3 * kAtom;          // 12 KB: 96 columns
  static constexpr int kE = kI8BM * kSpBK / 8;  // 2 KB
  // one K block of 128 logical K for all three digit products:
  // A x1 | A x128 | B d0 | B d1 | B d2 | E
  static constexpr int kOffA1 = 0, kOffA128 = kA, kOffB = 2 * kA, kOffE = 2 * kA + 3 * kB;
  static constexpr int kStage = kOffE + kE;
  static constexpr int kBarOff = kStages * kStage;
  static constexpr int kTabOff = kBarOff + 256;  // per tile: scale and V per column
  static constexpr int kXOff = kTabOff + 2 * kSpBN * 4;  // per half, column and row: (max, sum)
  static constexpr int kXBytes = 2 * Groups192::kCols * kI8BM * 8;
  static constexpr int kROff = kXOff + kXBytes;  // per epilogue warp: 3 digits x 32 slots x 32 rows
  static constexpr int kRWarp = 3 * 32 * 32;
  static constexpr int kTotal = kROff + 8 * kRWarp + 1024;
};

// Epilogue of one tile for one warp (TMEM lane quarter q, column half `half`: tile columns
// 96 half .. 96 half + 95):
//   drain  hi * 2^14 + lo of the half into registers (NARROW: as the exact 32-bit
//          integer, one instruction; else as the rounded float), the next 16 columns
//          in flight; then both accumulators are released, so that the next tile's
//          MMAs run during everything below;
//   A      z = sum * scale + V; per alignment column the maximum m of the own states
//          (from -FLT_MAX: fields of -inf may leave a half without one, whose share is
//          then 0) and the logit of the observed state;
//   B      e = exp(z - m), s = sum e; (m, s) exchanged with the partner warp (same
//          rows, other half): M = max(m, m'), S = s exp(m - M) + s' exp(m' - M) (same
//          order in both halves), lse = M + log S;
//   C      P = e * exp(m - M) / S, R = w (P - onehot) as its three digits, 32 slots x
//          32 rows at a time through shared memory, so that a lane moves 16 rows of one
//          slot with one store (byte stores straight to global memory, one sector each,
//          took 60 k cycles per tile, this takes 20 k).
// The whole half (96 values a thread) stays in registers: warpgroup 0 cedes its share
// (kWgRegsLoad / kWgRegsEpi).  The accumulators are held for about 2 k of the tile's
// 50 k cycles; a drain that also applied the scales and took the maxima held them 6 k.
// Both halves run the same instructions: element i of half 1 is tile column 96 + i,
// alignment column (i + 6) mod 9, so that with its columns taken in the order lj = i mod
// 9 its state is i / 9 + 10 (+ 1 from lj = 3 on); `xr` holds the observed states less
// these, and its last three elements (no state) have scale 0 and V = -inf.  This
// straight-line code is some 50 KB, and one copy per half did not fit the instruction
// cache.
template <bool NARROW>
__device__ __forceinline__ bool i8sp_epilogue_tile(const I8FwdArgs &args, uint32_t t_hi,
                                                   uint32_t t_lo, const float *tab_scale,
                                                   const float *tab_v, float2 *xbuf,
                                                   uint8_t *rstage, int half, int q, int lane,
                                                   int n, int t, long long part,
                                                   uint64_t *full_bar, uint32_t full_par,
                                                   long long budget, uint32_t empty_bar) {
  constexpr int kCols = Groups192::kCols;
  const int L = args.L;
  const int j0 = t * kCols;
  const bool live = n < args.N;
  const float wn = live ? args.w[n] : 0.0f;
  const int row = q * 32 + lane;
  int xr[kCols];  // by lj; -100: none
#pragma unroll
  for (int lj = 0; lj < kCols; ++lj) {
    const int j = j0 + (half ? (lj + 6) % kCols : lj);
    const int first = half ? 10 + (lj >= 3) : 0;
    xr[lj] = (live && j < L) ? (int)args.msa[(long long)n * L + j] - first : -100;
  }
  if (__any_sync(0xffffffffu, !mbar_wait(full_bar, full_par, budget))) {
    named_bar_sync(2 + q, 64);  // the partner may have got past its wait
    return false;
  }
  tc_fence_after();
  float z[kSpHalf];
  {
    const uint32_t c0 = half * kSpHalf;
    auto merge = [](uint32_t hi, uint32_t lo) {
      return NARROW ? __uint_as_float(hi * 16384u + lo) : i8_merge_exact(hi, lo);
    };
    uint32_t vh[2][16], vl[2][16];
    tmem_ld16(t_hi + c0, vh[0]);
    tmem_ld16(t_lo + c0, vl[0]);
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      tmem_wait_ld();
      if (c < 5) {
        tmem_ld16(t_hi + c0 + (c + 1) * 16, vh[(c + 1) & 1]);
        tmem_ld16(t_lo + c0 + (c + 1) * 16, vl[(c + 1) & 1]);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) z[c * 16 + i] = merge(vh[c & 1][i], vl[c & 1][i]);
    }
  }
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive_remote(empty_bar);
  // A
  float mx[kCols], tg[kCols], se[kCols];
#pragma unroll
  for (int lj = 0; lj < kCols; ++lj) { mx[lj] = -FLT_MAX; tg[lj] = 0.0f; se[lj] = 0.0f; }
#pragma unroll
  for (int i4 = 0; i4 < kSpHalf; i4 += 4) {
    const float4 sc = *reinterpret_cast<const float4 *>(tab_scale + half * kSpHalf + i4);
    const float4 vv = *reinterpret_cast<const float4 *>(tab_v + half * kSpHalf + i4);
    const float scs[4] = {sc.x, sc.y, sc.z, sc.w}, vvs[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i4 + e, lj = i % kCols;
      const float sum = NARROW ? __int2float_rn(__float_as_int(z[i])) : z[i];
      z[i] = fmaf(sum, scs[e], vvs[e]);
      mx[lj] = fmaxf(mx[lj], z[i]);
      if (xr[lj] == i / kCols) tg[lj] = z[i];
    }
  }
  // B
#pragma unroll
  for (int i = 0; i < kSpHalf; ++i) {
    const int lj = i % kCols;
    z[i] = expf(z[i] - mx[lj]);
    se[lj] += z[i];
  }
#pragma unroll
  for (int lj = 0; lj < kCols; ++lj) {
    const int jj = half ? (lj + 6) % kCols : lj;
    xbuf[(half * kCols + jj) * kI8BM + row] = make_float2(mx[lj], se[lj]);
  }
  named_bar_sync(2 + q, 64);
  double floss = 0.0;
  // R * 2^21 = e * cw - [observed] * won, with cw = w exp(m - M) / S * 2^21
  float cw[kCols];
  const float won = live ? wn * args.r_enc : 0.0f;
#pragma unroll
  for (int lj = 0; lj < kCols; ++lj) {
    const int jj = half ? (lj + 6) % kCols : lj;
    const float2 other = xbuf[((1 - half) * kCols + jj) * kI8BM + row];
    const float mo = other.x, so = other.y;
    const float M = fmaxf(mx[lj], mo);
    const float fa = expf(mx[lj] - M), fo = expf(mo - M);
    // (half 0's term is the fused one in both halves: the same float)
    const float S = half == 0 ? fmaf(se[lj], fa, __fmul_rn(so, fo)) : fmaf(so, fo, __fmul_rn(se[lj], fa));
    const float lse = M + logf(S);
    cw[lj] = xr[lj] > -100 ? (fa / S) * won : 0.0f;
    // the half that holds the observed state's column adds the loss term
    const int col = (xr[lj] + (half ? 10 + (lj >= 3) : 0)) * kCols + jj;
    if (xr[lj] > -100 && (col >= kSpHalf) == (half == 1)) floss += (double)(wn * (lse - tg[lj]));
  }
  // C
  uint8_t *const rrow = args.rnat + (long long)(n >> 5) * (3 * kNatTile);
  const long long sbytes = (long long)(args.Npad >> 5) * (3 * kNatTile);
#pragma unroll
  for (int c = 0; c < kSpHalf / 32; ++c) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int lj = (c * 32 + i) % kCols;
      const float r = fmaf(z[c * 32 + i], cw[lj], xr[lj] == (c * 32 + i) / kCols ? -won : 0.0f);
      // |R| 2^-eR <= 1: only the top of the range needs the clamp (P rounding to 1)
      const int d = min(__float2int_rn(r), (1 << kI8FracBits) - 1);
      rstage[i * 32 + lane] = (uint8_t)(d >> 14);
      rstage[1024 + i * 32 + lane] = (uint8_t)((d >> 7) & 127);
      rstage[2048 + i * 32 + lane] = (uint8_t)(d & 127);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = 16 * u + (lane >> 1), col = half * kSpHalf + c * 32 + i;
      const int a = col / kCols, j = j0 + col % kCols;
      if (col < Groups192::kUsed && j < L) {
        const uint32_t s = (uint32_t)(a * L + j);
        uint8_t *p = rrow + (long long)(s >> 7) * sbytes + (s & 127) * 32 + (((lane ^ (s >> 2)) & 1) << 4);
        const uint4 *from = reinterpret_cast<const uint4 *>(rstage + i * 32 + (lane & 1) * 16);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4 *>(p + k * kNatTile) = from[k * 64];
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) floss += __shfl_xor_sync(0xffffffffu, floss, o);
  if (lane == 0) args.part_f[part * 8 + half * 4 + q] = floss;
  return true;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWgThreads, 1)
    i8sp_forward_kernel(const __grid_constant__ I8SpMaps maps, I8FwdArgs args) {
  using SM = I8SpSmem;
  constexpr int kStages = SM::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = i8_align1024(smem_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + SM::kBarOff);
  uint64_t *empty = full + kStages;
  uint64_t *acc_full = empty + kStages;
  uint64_t *acc_empty = acc_full + 1;
  uint64_t *drain = acc_empty + 1;
  // a barrier that no thread ever arrives on: the epilogue waits on it instead
  // of on acc_full when a test asks for a wait that runs out (acc_wait_cycles)
  uint64_t *never = drain + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(never + 1);
  int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
  float *tab_scale = reinterpret_cast<float *>(smem + SM::kTabOff);
  float *tab_v = tab_scale + kSpBN;
  float2 *xbuf = reinterpret_cast<float2 *>(smem + SM::kXOff);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int n_tiles = args.m_tiles * args.T;
  const int k_blocks = args.KP / kSpBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 16);
    mbar_init(drain, 1);
    mbar_init(never, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&maps.a1);
    prefetch_tmap(&maps.a128);
    prefetch_tmap(&maps.e);
    for (int i = 0; i < 3; ++i) prefetch_tmap(&maps.b[i]);
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  // the prologue above overlaps the previous kernel's tail; its outputs from here
  griddep_launch();
  griddep_wait();
  const uint32_t tmem_base = *tmem_slot;
  // TMEM: hi [0, 192), lo [256, 448), metadata 456 / 460
  const uint32_t t_hi = tmem_base, t_lo = tmem_base + 256, t_e = tmem_base + 456;

  if (warp < 4) reg_dec<kWgRegsLoad>();
  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer (both CTAs), in the MMA's order
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok && !i8_aborted(abort_flag); tile += npairs) {
        const int m = tile % args.m_tiles, t = tile / args.m_tiles;
        // tile rows of the tiled operands (256-byte rows): A 32, E 8, B 48 per K block
        const int m128 = 2 * m + (int)rank, tb = 2 * t + (int)rank;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int stage = it % kStages;
          const uint32_t round = it / kStages;
          if (!mbar_wait(&empty[stage], (round & 1) ^ 1)) {
            i8_record_error(args.status, kErrFwdTimeout, abort_flag);
            ok = false;
            break;
          }
          uint8_t *st = smem + stage * SM::kStage;
          const uint32_t fb = mapa_shared(smem_u32(&full[stage]), 0);
          const int ya = (m128 * k_blocks + kb) * 32, yb = (tb * k_blocks + kb) * 48;
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * SM::kStage);
          tma_load_2d_pair(st + SM::kOffA1, &maps.a1, fb, 0, ya);
          tma_load_2d_pair(st + SM::kOffA128, &maps.a128, fb, 0, ya);
          for (int i = 0; i < 3; ++i)
            tma_load_2d_pair(st + SM::kOffB + i * SM::kB, &maps.b[i], fb, 0, yb);
          tma_load_2d_pair(st + SM::kOffE, &maps.e, fb, 0, (m128 * k_blocks + kb) * 8);
        }
      }
      const uint32_t issued = it;
      for (uint32_t r = (issued > kStages ? issued - kStages : 0); r < issued; ++r) {
        const bool w = rank == 0 ? mbar_wait(&full[r % kStages], (r / kStages) & 1)
                                 : mbar_wait(&empty[r % kStages], (r / kStages) & 1);
        if (!w) {
          i8_record_error(args.status, kErrFwdTimeout, abort_flag);
          break;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ---------------- MMA issuer (leader): 256 x 192 x 64 (logical) sparse pair MMAs.
      // The loop carries its stage, phase and descriptor words along: see umma_i8sp_block
      constexpr uint32_t idesc = idesc_i8_s32(kI8PairM, kSpBN, 0, 1, 0, 1) | kIdescSparse;
      constexpr uint32_t kStep = SM::kStage >> 4;
      const uint32_t s0 = smem_u32(smem);
      const uint32_t a0 = sdesc_low(s0 + SM::kOffA1, 16), b0 = sdesc_low(s0 + SM::kOffB, SM::kAtom);
      const uint32_t a_top = sdesc_high(512, 4), b_top = sdesc_high(256, 6);
      uint32_t stage = 0, phase = 0, te = t_e;
      int local = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok && !i8_aborted(abort_flag);
           tile += npairs, ++local) {
        // both accumulators free: the previous tile's epilogue has drained them
        if (!mbar_wait(acc_empty, (local & 1) ^ 1)) {
          i8_record_error(args.status, kErrFwdTimeout, abort_flag);
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(&full[stage], phase)) {
            i8_record_error(args.status, kErrFwdTimeout, abort_flag);
            ok = false;
            break;
          }
          tmem_cp_pair_128x128b(te, sdesc_noswz(s0 + stage * SM::kStage + SM::kOffE, 2048, 128));
          umma_i8sp_block<SM::kA / 16, 2, SM::kB / 16, 128>(t_hi, t_lo, a0 + stage * kStep, a_top,
                                                            b0 + stage * kStep, b_top, idesc, te, kb);
          umma_commit_pair(&empty[stage], 0x3);
          te ^= 4;
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit_pair(acc_full, 0x3);
      }
      umma_commit_pair(drain, 0x1);
      if (!mbar_wait(drain, 0)) i8_record_error(args.status, kErrFwdTimeout, abort_flag);
    }
  } else if (warp >= 4) {
    reg_inc<kWgRegsEpi>();
    // ---------------- epilogue (both CTAs): 8 warps, lane quarter q, column half
    const int q = warp & 3;
    const int half = (warp - 4) >> 2;
    const int ethr = threadIdx.x - 128;
    const int L = args.L;
    const float *x1 = args.sw.parity ? args.sw.at_x(1 - *args.sw.parity) : args.x1;
    uint8_t *const rstage = smem + SM::kROff + (warp - 4) * SM::kRWarp;
    const uint32_t empty_bar = mapa_shared(smem_u32(acc_empty), 0);

    int local = 0;
    for (int tile = pair; tile < n_tiles; tile += npairs, ++local) {
      if (named_bar_or(1, 256, i8_aborted(abort_flag))) break;
      const int m = tile % args.m_tiles, t = tile / args.m_tiles;
      if (ethr < kSpBN) {
        const int a = ethr / Groups192::kCols, j = t * Groups192::kCols + ethr % Groups192::kCols;
        float sc = 0.0f, vv = 0.0f;
        if (a >= kQ) {
          vv = -INFINITY;  // no state
        } else if (j < L) {
          sc = pow2f(col_exponent(args.colmax[a * L + j]) - kI8FracBits);
          if (a < kQ - 1) vv = x1[a * L + j];
        }
        tab_scale[ethr] = sc;
        tab_v[ethr] = vv;
      }
      named_bar_sync(1, 256);
      const int n = m * kI8PairM + (int)rank * kI8BM + q * 32 + lane;
      const uint32_t lq = (uint32_t)(q * 32) << 16;
      const long long part = (long long)tile * 2 + rank;
      // (with acc_wait_cycles set, a wait that runs out by design: see `never`)
      const bool test = args.acc_wait_cycles > 0;
#define CCM_TILE_ARGS                                                                             \
  args, t_hi + lq, t_lo + lq, tab_scale, tab_v, xbuf, rstage, half, q, lane, n, t, part,          \
      test ? never : acc_full, test ? 0u : (uint32_t)(local & 1),                                 \
      test ? args.acc_wait_cycles : kWaitBudgetCycles, empty_bar
      const bool ok = L <= kI8NarrowMaxL ? i8sp_epilogue_tile<true>(CCM_TILE_ARGS)
                                         : i8sp_epilogue_tile<false>(CCM_TILE_ARGS);
#undef CCM_TILE_ARGS
      if (!ok && lane == 0) i8_record_error(args.status, kErrFwdTimeout, abort_flag);
    }
  }

  tc_fence_before();
  cluster_sync();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace ccm

namespace ccm {

// ---------------------------------------------------------------- backward
// Pair tiles of 256 x 256 slots (P <= Q for the symmetric gradient) as in
// tc_backward.  Per K step of 32 rows, with the digits r0..r2 of R and the two
// one-hot operands O1, O128 (both sides MN-major, 8-bit):
//   hi += O1_P^T r0_Q + r0_P^T O1_Q
//   lo += O128_P^T r1_Q + O1_P^T r2_Q + r1_P^T O128_Q + r2_P^T O1_Q
// (SYM = false: the O^T R products only).  The sums are exact in s32 for up to
// 32768 rows; longer alignments are cut into K chunks of that length, each merged
// as (hi * 2^14 + lo) * 2^-21 (exact, one rounding) into FP32 registers.  The
// output phase (ccm_bwd_out.cuh) is one atomic add per g2 element.
constexpr int kI8BwdBK = 32;
constexpr int kI8BwdChunkKB = 1024;  // 32768 rows: |lo| <= 32768 * 2 * 16383 < 2^31

struct I8BwdSmem {
  static constexpr int kStages = 5;
  static constexpr int kTile = 128 * kI8BwdBK;  // 4 KB: 128 slots x 32 rows, 8-bit
  // P side: O1, O128, r0, r1, r2 (this CTA's 128 P slots); Q side: the same (its 128 Q slots)
  static constexpr int kStage = 10 * kTile;
  static constexpr int kBarOff = kStages * kStage;
  static constexpr int kTOff = kBarOff + 256;
  static constexpr int kTBytes = 8 * kBwdOutWarpBytes;
  static constexpr int kTotal = kTOff + kTBytes + 1024;
};

// sum V^2 of the single fields in FP64, in a fixed order, as each lane's part of it.
__device__ __forceinline__ double i8nat_squares(const float *x1, int ns, int lane) {
  double s = 0.0;
  for (int i0 = lane; i0 < ns; i0 += 16 * 32) {
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = i0 + 32 * u < ns ? x1[i0 + 32 * u] : 0.0f;
#pragma unroll
    for (int u = 0; u < 16; ++u) s += (double)v[u] * (double)v[u];
  }
  return s;
}

// An evaluation whose gradient replaces its point (d_g == d_x): the scan leaves x as it is
// (its g2 is 1 x), and this kernel, between the forward, the last to read x2 and all of V,
// and the backward, which writes g1, makes g2 of it and takes each lane's sum of V^2.
__global__ void __launch_bounds__(256) i8sp_in_place_kernel(float *g2, long long n, float g2_scale,
                                                            const float *x1, int ns,
                                                            double *squares) {
  griddep_wait();
  griddep_launch();
  if (blockIdx.x == 0 && threadIdx.x < 32) squares[threadIdx.x] = i8nat_squares(x1, ns, threadIdx.x);
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) g2[i] *= g2_scale;
}

// fx = sum(loss partials) + lambda1 sum V^2 + 0.5 lambda2 sum x2^2 in FP64, in a fixed
// order, and the padding of g1 (the backward's output phase writes g1 itself); one warp.
__device__ __forceinline__ void i8nat_finalize(const FinalizeArgs &args, const float *x1, float *g1,
                                               int lane) {
  auto sum = [&](const double *p, long long n) {
    double s = 0.0;
    for (long long i0 = lane; i0 < n; i0 += 8 * 32) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = i0 + 32 * u < n ? p[i0 + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    return s;
  };
  const int ns = (int)nsingle_of(args.L);
  double acc[3] = {sum(args.part_f, args.n_part_f), sum(args.part_reg, args.n_part_reg),
                   args.squares ? args.squares[lane] : i8nat_squares(x1, ns, lane)};
  for (long long i = ns + lane; i < args.nsp; i += 32) g1[i] = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  if (lane == 0) {
    const double F = acc[0];
    const double fx = F + (double)args.lambda_single * acc[2] + 0.5 * (double)args.lambda_pair * acc[1];
    args.out->fx = fx;
    args.out->f_data = F;
    args.out->reg = fx - F;
    if (args.host) finalize_host(args, fx, F);
  }
}

// (finalize_host may have written the record already)
__device__ __forceinline__ void i8_backward_error(const BwdArgs &args, int *abort_flag) {
  i8_record_error(args.status, kErrBwdTimeout, abort_flag);
  if (args.fin.host) *reinterpret_cast<volatile int *>(&args.fin.host->status) = kErrBwdTimeout;
}

// CUT: a last wave of tiles that fills at most half of the pairs is cut along K (the rows):
// every part is an entry of its own in the tile list, and the epilogue warp that finishes
// a tile's part last adds the parts' integer sums (exact, so that the gradient is that of
// the uncut tile bit for bit) and writes the output.
// NAT: natural slots, K-major operands in the storage of i8nat_offset (the sparse
// path); else Groups256 slots, row-major Npad x S operands (MN-major).  The MMAs run
// at the same rate either way.
// Bound on the sparse path: the MMAs, 768 cycles of a K block's six (their issue rate is
// the peak of kind::i8; at L = 1000 the power cap lowers the clock), then the last wave's
// fill (i8_cut_parts) and, below N = 2000, the output phase of a pair's last tile.
// L = 300, N = 5000 375 us, L = 253, N = 7001 374, L = 50, N = 200 23.
template <bool SYM, bool NAT, bool CUT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWgThreads, 1)
    i8_backward_kernel(const __grid_constant__ I8BwdMaps maps, BwdArgs args) {
  using SM = I8BwdSmem;
  constexpr int kStages = SM::kStages;
  constexpr int kBN = 256, kHalfN = 128, kPairM = 256, kBM = 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = i8_align1024(smem_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + SM::kBarOff);
  uint64_t *empty = full + kStages;
  uint64_t *acc_full = empty + kStages;
  uint64_t *acc_empty = acc_full + 1;
  uint64_t *drain = acc_empty + 1;
  // as in the forward: waited on instead of acc_full when a test asks for a wait that runs
  // out (acc_wait_cycles)
  uint64_t *never = drain + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(never + 1);
  int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int n_tiles = args.n_tiles;
  const int k_blocks = args.Npad / kI8BwdBK;
  // K blocks [first, end) of an entry of the tile list
  auto cut_of = [&](int tile) { return CUT ? args.cuts[tile] : 0; };
  auto k_first = [&](int cut) { return CUT ? k_blocks * (cut & 255) / (cut >> 8 & 255) : 0; };
  auto k_end = [&](int cut) { return CUT ? k_first(cut + 1) : k_blocks; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 16);
    mbar_init(drain, 1);
    mbar_init(never, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&maps.o1);
    prefetch_tmap(&maps.r[0]);
    if (!NAT) {
      prefetch_tmap(&maps.o128);
      prefetch_tmap(&maps.r[1]);
      prefetch_tmap(&maps.r[2]);
    }
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  // the prologue above overlaps the previous kernel's tail; its outputs from here
  griddep_launch();
  griddep_wait();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t t_hi = tmem_base, t_lo = tmem_base + kBN;

  if (warp < 4) reg_dec<kWgRegsLoad>();
  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok && !i8_aborted(abort_flag); tile += npairs) {
        const int2 pq = args.tiles[tile];
        const int xP = pq.x * kPairM + (int)rank * kBM;
        const int xQ = pq.y * kBN + (int)rank * kHalfN;
        const int cut = cut_of(tile), kb_end = k_end(cut);
        for (int kb = k_first(cut); kb < kb_end; ++kb, ++it) {
          const int stage = it % kStages;
          const uint32_t round = it / kStages;
          if (!mbar_wait(&empty[stage], (round & 1) ^ 1)) {
            i8_backward_error(args, abort_flag);
            ok = false;
            break;
          }
          uint8_t *st = smem + stage * SM::kStage;
          const uint32_t fb = mapa_shared(smem_u32(&full[stage]), 0);
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * (SYM ? 10 : 5) * SM::kTile);
          uint8_t *const stq = st + 5 * SM::kTile;
          if constexpr (NAT) {
            // rows of 256 bytes: 32 per one-hot tile pair, 48 per digit tile triple
            const int tp = (xP >> 7) * k_blocks + kb, tq = (xQ >> 7) * k_blocks + kb;
            tma_load_2d_pair(st, &maps.o1, fb, 0, tp * 32);
            if (SYM) tma_load_2d_pair(st + 2 * SM::kTile, &maps.r[0], fb, 0, tp * 48);
            if (SYM) tma_load_2d_pair(stq, &maps.o1, fb, 0, tq * 32);
            tma_load_2d_pair(stq + 2 * SM::kTile, &maps.r[0], fb, 0, tq * 48);
          } else {
            const int y = kb * kI8BwdBK;
            tma_load_2d_pair(st + 0 * SM::kTile, &maps.o1, fb, xP, y);
            tma_load_2d_pair(st + 1 * SM::kTile, &maps.o128, fb, xP, y);
            if (SYM) {
              for (int i = 0; i < 3; ++i)
                tma_load_2d_pair(st + (2 + i) * SM::kTile, &maps.r[i], fb, xP, y);
              tma_load_2d_pair(stq, &maps.o1, fb, xQ, y);
              tma_load_2d_pair(stq + SM::kTile, &maps.o128, fb, xQ, y);
            }
            for (int i = 0; i < 3; ++i)
              tma_load_2d_pair(stq + (2 + i) * SM::kTile, &maps.r[i], fb, xQ, y);
          }
        }
      }
      const uint32_t issued = it;
      for (uint32_t r = (issued > (uint32_t)kStages ? issued - kStages : 0); r < issued; ++r) {
        const bool w = rank == 0 ? mbar_wait(&full[r % kStages], (r / kStages) & 1)
                                 : mbar_wait(&empty[r % kStages], (r / kStages) & 1);
        if (!w) {
          i8_backward_error(args, abort_flag);
          break;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr int mn = NAT ? 0 : 1;
      constexpr uint32_t id_us = idesc_i8_s32(kPairM, kBN, 0, 1, mn, mn);  // A = one-hot, B = R
      constexpr uint32_t id_su = idesc_i8_s32(kPairM, kBN, 1, 0, mn, mn);  // A = R, B = one-hot
      uint32_t it = 0, chunk = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok && !i8_aborted(abort_flag); tile += npairs) {
        const int cut = cut_of(tile), kb_end = k_end(cut);
        for (int kb0 = k_first(cut); kb0 < kb_end && ok; kb0 += kI8BwdChunkKB, ++chunk) {
          if (!mbar_wait(acc_empty, (chunk & 1) ^ 1)) {
            i8_backward_error(args, abort_flag);
            ok = false;
            break;
          }
          tc_fence_after();
          const int kb1 = min(kb0 + kI8BwdChunkKB, kb_end);
          for (int kb = kb0; kb < kb1; ++kb, ++it) {
            const int stage = it % kStages;
            const uint32_t round = it / kStages;
            if (!mbar_wait(&full[stage], round & 1)) {
              i8_backward_error(args, abort_flag);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t s0 = smem_u32(smem + stage * SM::kStage);
            auto d = [&](int i) {
              return NAT ? sdesc_sw32(s0 + i * SM::kTile, 16, 256)
                         : sdesc_sw128(s0 + i * SM::kTile, SM::kTile, 1024);
            };
            const uint32_t first = kb == kb0 ? 0u : 1u;
            umma_i8_pair(t_hi, d(0), d(7), id_us, first);  // O1_P^T r0_Q
            umma_i8_pair(t_lo, d(1), d(8), id_us, first);  // O128_P^T r1_Q
            umma_i8_pair(t_lo, d(0), d(9), id_us, 1);      // O1_P^T r2_Q
            if (SYM) {
              umma_i8_pair(t_hi, d(2), d(5), id_su, 1);    // r0_P^T O1_Q
              umma_i8_pair(t_lo, d(3), d(6), id_su, 1);    // r1_P^T O128_Q
              umma_i8_pair(t_lo, d(4), d(5), id_su, 1);    // r2_P^T O1_Q
            }
            umma_commit_pair(&empty[stage], 0x3);
          }
          if (!ok) break;
          umma_commit_pair(acc_full, 0x3);
        }
      }
      umma_commit_pair(drain, 0x1);
      if (!mbar_wait(drain, 0)) i8_backward_error(args, abort_flag);
    }
  } else if (NAT && warp == 2) {
    // the sums of the loss and regulariser partials, while the MMAs run
    if (blockIdx.x == 0) {
      const int q = args.sw.parity ? 1 - *args.sw.parity : 0;
      i8nat_finalize(args.fin, args.sw.parity ? args.sw.at_x(q) : args.fin.x1,
                     args.sw.parity ? args.sw.at_g(q) : args.fin.g1, lane);
    }
  } else if (NAT && warp == 3) {
    // the column maxima's accumulator, for the next evaluation's scan
    if (blockIdx.x == 0)
      for (int i = lane; i < kQ * args.L; i += 32) args.cmacc[i] = 0u;
  } else if (warp >= 4) {
    reg_inc<kWgRegsEpi>();
    // Epilogue: each K chunk merged from the two integer accumulators (16 columns
    // per TMEM load, the next 16 in flight) into FP32 registers, then added to g.
    const int q = warp & 3;
    const int half = (warp - 4) >> 2;
    float *Tb = reinterpret_cast<float *>(smem + SM::kTOff + (warp - 4) * kBwdOutWarpBytes);
    const float r_dec = args.r_dec;
    const uint32_t empty_bar = mapa_shared(smem_u32(acc_empty), 0);
    const uint32_t col0 = half * kHalfN + ((uint32_t)(q * 32) << 16);
    // the point evaluated and its gradient
    const int buf = args.sw.parity ? 1 - *args.sw.parity : 0;
    const float *x1 = args.sw.parity ? args.sw.at_x(buf) : args.fin.x1;
    float *g1 = args.sw.parity ? args.sw.at_g(buf) : args.fin.g1;
    uint32_t chunk = 0;
    bool ok = true;
    // (as instances of their own, the waits of a test cost an evaluation 0.7 us at L = 50 and
    // 1.6 at L = 150: more kernels in the module; as an argument nothing)
    auto acc_ready = [&] {
      return args.acc_wait_cycles ? mbar_wait(never, 0, args.acc_wait_cycles) : mbar_wait(acc_full, chunk & 1);
    };
    for (int tile = pair; tile < n_tiles && ok; tile += npairs) {
      float accv[kHalfN];
      // one K chunk: wait for it, merge it into accv (or add it there), release it
      auto take = [&](auto first) {
        const bool w_ok = acc_ready();
        if (__any_sync(0xffffffffu, !w_ok)) {
          if (lane == 0) i8_backward_error(args, abort_flag);
          return false;
        }
        tc_fence_after();
        uint32_t vh[2][16], vl[2][16];
        __syncwarp();
        tmem_ld16(t_hi + col0, vh[0]);
        tmem_ld16(t_lo + col0, vl[0]);
#pragma unroll
        for (int c = 0; c < kHalfN / 16; ++c) {
          tmem_wait_ld();
          if (c + 1 < kHalfN / 16) {
            tmem_ld16(t_hi + col0 + (c + 1) * 16, vh[(c + 1) & 1]);
            tmem_ld16(t_lo + col0 + (c + 1) * 16, vl[(c + 1) & 1]);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            // exact scaling by 2^(eR - 21)
            const float v = i8_merge_exact(vh[c & 1][i], vl[c & 1][i]);
            if constexpr (decltype(first)::value) accv[c * 16 + i] = v * r_dec;
            else accv[c * 16 + i] = fmaf(v, r_dec, accv[c * 16 + i]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(empty_bar);
        ++chunk;
        return true;
      };
      // One part of a cut tile: its sums to cut_sums, unless the other parts are there
      // already; the warp that finishes last adds the parts' integers (exact, in any
      // order) and goes on to the output.  Nobody waits.  0: error, 1: not last, 2: last.
      auto take_part = [&](int cut) {
        const bool w_ok = acc_ready();
        if (__any_sync(0xffffffffu, !w_ok)) {
          if (lane == 0) i8_backward_error(args, abort_flag);
          return 0;
        }
        tc_fence_after();
        const int part = cut & 255, parts = cut >> 8 & 255;
        const int who = (cut >> 16) * kCutCounters + (int)rank * 8 + (warp - 4);
        // [cut tile, CTA, warp][part][16-column chunk, hi | lo, 4 columns][lane]
        uint4 *sums = reinterpret_cast<uint4 *>(args.cuts + cut_sums_offset(args.n_tiles)) +
                      (long long)who * parts * 64 * 32 + lane;
        unsigned *done = reinterpret_cast<unsigned *>(args.fin.out + 1) + who;
        auto seen = [&](bool count) {
          unsigned n = 0;
          if (lane == 0) n = count ? atomicAdd(done, 1u) : *reinterpret_cast<volatile unsigned *>(done);
          return __shfl_sync(0xffffffffu, n, 0);
        };
        bool last = seen(false) == (unsigned)parts - 1;
        if (!last) {
#pragma unroll 1
          for (int c = 0; c < kHalfN / 16; ++c) {
            uint32_t v[2][16];
            tmem_ld16(t_hi + col0 + c * 16, v[0]);
            tmem_ld16(t_lo + col0 + c * 16, v[1]);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i)
              __stcg(sums + (part * 64 + c * 8 + i) * 32,
                     make_uint4(v[i >> 2][(i & 3) * 4], v[i >> 2][(i & 3) * 4 + 1],
                                v[i >> 2][(i & 3) * 4 + 2], v[i >> 2][(i & 3) * 4 + 3]));
          }
          __threadfence();
          __syncwarp();
          last = seen(true) == (unsigned)parts - 1;
        }
        if (last) {
          __threadfence();
          __syncwarp();
#pragma unroll
          for (int c = 0; c < kHalfN / 16; ++c) {
            uint32_t v[2][16];
            tmem_ld16(t_hi + col0 + c * 16, v[0]);
            tmem_ld16(t_lo + col0 + c * 16, v[1]);
            tmem_wait_ld();
#pragma unroll 1
            for (int p = 0; p < parts; ++p) {
              if (p == part) continue;
              uint4 o[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = __ldcg(sums + (p * 64 + c * 8 + i) * 32);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                v[i >> 2][(i & 3) * 4] += o[i].x;
                v[i >> 2][(i & 3) * 4 + 1] += o[i].y;
                v[i >> 2][(i & 3) * 4 + 2] += o[i].z;
                v[i >> 2][(i & 3) * 4 + 3] += o[i].w;
              }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) accv[c * 16 + i] = i8_merge_exact(v[0][i], v[1][i]) * r_dec;
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(empty_bar);
        ++chunk;
        return last ? 2 : 1;
      };
      bool cut_tile = false;
      if constexpr (CUT) {
        const int cut = cut_of(tile);
        cut_tile = (cut >> 8 & 255) > 1;
        if (cut_tile) {
          const int got = take_part(cut);
          ok = got != 0;
          if (got == 1) continue;
        }
      }
      if (!cut_tile) {
        ok = take(std::true_type{});
        for (int kb0 = kI8BwdChunkKB; kb0 < k_blocks && ok; kb0 += kI8BwdChunkKB)
          ok = take(std::false_type{});
      }
      if (!ok) break;
      const int2 pq = args.tiles[tile];
      const int s1 = pq.x * kPairM + (int)rank * kBM + q * 32, s2 = pq.y * kBN + half * kHalfN;
      if constexpr (NAT)
        bwd_output_natural<SYM>(accv, Tb, args, g1, g1 + args.fin.nsp, x1, lane, s1, s2, pq.x == pq.y);
      else
        bwd_output<Groups256, SYM>(accv, Tb, args.g2, args.g1d, args.L, lane, s1, s2);
    }
  }

  tc_fence_before();
  cluster_sync();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace ccm

namespace ccm {

// ---------------------------------------------------------------- launchers
// Evaluation at d_x, or, with d_s, at d_xt = d_x + alpha d_s (the step is taken
// by the column-max pass, which writes d_xt), or, with trial (sparse path), a solve's
// trial on its own buffers.  Profile marks: [colmax + prep |
// forward | backward | finalize].
static cudaError_t i8_prepare_dense(ccm_context *c, const float *d_x, float *g2, const float *d_s,
                                    const double *d_alpha, float *d_xt) {
  const int L = c->L;
  const bool step = d_s != nullptr;
  const float *x2 = (step ? d_xt : d_x) + c->nsp;
  cudaError_t e;
  if ((e = zero_words(c->d_colmax, (long long)kQ * L, c->stream)) != cudaSuccess) return e;
  constexpr int kRows = 32;
  const int cols = (c->skip_padding ? kQ : kQPad) * L;
  const dim3 cgrid((cols + 255) / 256, (kQ * L + kRows - 1) / kRows + (step ? 1 : 0));
  if (step)
    e = launch_pdl(i8_colmax_kernel<true>, cgrid, dim3(256), 0, c->stream, d_x, d_s, d_alpha, d_xt,
                   c->d_colmax, L, c->nsp, kRows, cols);
  else
    e = launch_pdl(i8_colmax_kernel<false>, cgrid, dim3(256), 0, c->stream, d_x,
                   (const float *)nullptr, (const double *)nullptr, (float *)nullptr, c->d_colmax,
                   L, c->nsp, kRows, cols);
  if (e != cudaSuccess) return e;
  // per-slot factors after the column maxima, 16-byte aligned for the float4 loads
  float *enc = reinterpret_cast<float *>(c->d_colmax + ((kQ * L + 3) & ~3));
  e = launch_pdl(i8_scales_kernel, dim3((c->S + 255) / 256), dim3(256), 0, c->stream,
                 (const uint32_t *)c->d_colmax, enc, L, c->S);
  if (e != cudaSuccess) return e;
  I8PrepArgs pa{};
  for (int i = 0; i < 3; ++i) pa.wdig[i] = c->d_wdig[i];
  pa.enc = enc;
  pa.part_reg = c->d_part_reg;
  pa.L = L; pa.S = c->S; pa.lambda_pair = c->lambda_pair;
  pa.g2_coef = c->gradient == CCM_GRADIENT_PARTIAL ? 1.0f : 2.0f;
  pa.inv_L = 1.0f / (float)L;
  pa.ncols = cols;
  pa.vec = (L & 3) == 0 &&
           ((reinterpret_cast<uintptr_t>(x2) | reinterpret_cast<uintptr_t>(g2)) & 15) == 0;
  count_launch(c, 4);
  return launch_pdl(i8_prep_kernel, dim3(kQ * L), dim3(256), sizeof(float) * c->S, c->stream, x2, g2,
                    pa);
}

// Rows of a scan block and of a digits block: enough blocks to fill the chip a few
// times over, few enough that a block's set-up and its column maxima's atomics stay
// small beside its rows.
static int scan_rows(int L, int col_blocks) {
  const int want = 8 * 148 / col_blocks;  // row blocks
  const int rows = (kQ * L + want - 1) / want;
  return rows < 16 ? 16 : rows > 64 ? 64 : (rows + 7) / 8 * 8;
}

static float i8_g2_scale(const ccm_context *c) {
  return (c->gradient == CCM_GRADIENT_PARTIAL ? 1.0f : 2.0f) * c->lambda_pair;
}

static cudaError_t i8_prepare_sparse(ccm_context *c, const float *d_x, float *g2, const float *d_s,
                                     const double *d_alpha, float *d_xt, const CgTrialArgs *trial) {
  const int L = c->L;
  const bool step = d_s != nullptr || trial;
  const float *x2 = trial ? nullptr : (step ? d_xt : d_x) + c->nsp;
  I8ScanArgs sa{};
  sa.x = d_x; sa.s = const_cast<float *>(d_s); sa.alpha = d_alpha; sa.xt = d_xt;
  if (trial) {
    sa.s = trial->s; sa.alpha = trial->alpha;
    sa.sw = trial->sw; sa.beta = trial->beta; sa.dir_mode = trial->dir_mode;
  }
  sa.cmacc = c->d_cmacc; sa.part_reg = c->d_part_reg; sa.g2 = g2; sa.out = c->d_out;
  sa.nsp = c->nsp; sa.L = L;
  sa.out_vecs = (int)(sizeof(ccm_result) + 4 * kCutCounters * c->n_cut_tiles + 15) / 16;
  sa.cols = (c->skip_padding ? kQ : kQPad) * L;
  // (over x itself: see i8sp_in_place_kernel)
  sa.g2_scale = g2 && g2 == x2 ? 1.0f : i8_g2_scale(c);
  auto bits = [](const void *p) { return reinterpret_cast<uintptr_t>(p); };
  const CgSwap &w = sa.sw;
  sa.vec = ((bits(d_x) | bits(sa.s) | bits(d_xt) | bits(g2) | bits(w.x[0]) | bits(w.x[1]) |
             bits(w.g[0]) | bits(w.g[1])) & 15) == 0;
  const int cb = (sa.cols + 1023) / 1024;
  sa.rows_per_block = scan_rows(L, cb);
  const int rb = (kQ * L + sa.rows_per_block - 1) / sa.rows_per_block;
  c->n_part_reg = cb * rb;
  cudaError_t e = launch_pdl(step ? i8sp_scan_kernel<true> : i8sp_scan_kernel<false>,
                             dim3(cb, rb + (step ? 1 : 0)), dim3(256), 0, c->stream, sa);
  if (e != cudaSuccess) return e;

  I8DigitsArgs da{};
  for (int i = 0; i < 3; ++i) da.wdig[i] = c->d_wdig[i];
  da.x2 = x2; da.sw = sa.sw; da.nsp = c->nsp; da.cmacc = c->d_cmacc; da.colmax = c->d_colmax;
  da.L = L; da.T = c->T; da.KB = c->KP / 128;
  const int gb = (c->T + kDigGroups - 1) / kDigGroups;  // blocks along the groups, evenly filled
  da.gpb = (c->T + gb - 1) / gb;
  const int row_tiles = (kQ * L + kDigRows - 1) / kDigRows;
  const bool few = row_tiles * gb <= 8 * 148;
  const int rows = few ? kDigRowsFew : kDigRows;
  const int per = (row_tiles * gb + 16 * 148 - 1) / (16 * 148);  // two waves of blocks
  da.rows_per_block = rows * (per < 4 ? per : 4);
  count_launch(c, 2);
  return launch_pdl(few ? i8sp_digits_kernel<kDigRowsFew> : i8sp_digits_kernel<kDigRows>,
                    dim3(gb, (kQ * L + da.rows_per_block - 1) / da.rows_per_block),
                    dim3(kDigThreads), sizeof(int) * rows * dig_row_words(da.gpb), c->stream, da);
}

// A K block is 768 cycles of MMAs (not symmetric: 384), and cutting a tile in p saves
// (p - 1) / p of its last wave.  It costs what writing the sums and adding p - 1 of them
// takes (512 KB per part, L2 to two SMs), measured as 12 k + 6 k p cycles, and 8 k cycles in the
// next scan, whose L2 these sums occupy.  The measured sides, backward alone, uncut and
// cut: L = 300, 29 of 325 tiles left over, p = 2: N = 3000 246 and 239 us, N = 5000 391 and
// 375; L = 253, 9 of 231 tiles: N = 3000, p = 4 200 and 188, N = 7001, p = 5 417 and 374
// (N = 2000 149, and 159 in eight parts: left whole); L = 150, 17 of 91, p = 4: N = 3500 122
// and 108 (N = 2000 78 and 89: left whole); L = 200, N = 20000, 5 of 153, p = 8: 843 and
// 698.  More than half as many tiles as pairs are never cut: a part each is a pair each.
// Rows beyond one chunk are not cut: their sums leave the integers chunk by chunk.
int i8_cut_parts(int tiles, int pairs, int Npad, bool sym) {
  const int k_blocks = Npad / kI8BwdBK, rest = tiles % pairs;
  if (rest == 0 || rest > kMaxCutTiles || k_blocks > kI8BwdChunkKB) return 1;
  const int max_parts = pairs / rest < 8 ? pairs / rest : 8;
  int best = 1, best_gain = 0;
  for (int p = 2; p <= max_parts; ++p) {
    const int gain = k_blocks * (sym ? 768 : 384) * (p - 1) / p - 20000 - 6000 * p;
    if (gain > best_gain) best = p, best_gain = gain;
  }
  return best;
}

static auto backward_kernel(bool sym, bool sp, bool cut) {
  return sp && cut ? (sym ? i8_backward_kernel<true, true, true> : i8_backward_kernel<false, true, true>)
         : sp      ? (sym ? i8_backward_kernel<true, true, false> : i8_backward_kernel<false, true, false>)
         : sym     ? i8_backward_kernel<true, false, false>
                   : i8_backward_kernel<false, false, false>;
}

cudaError_t i8_evaluate(ccm_context *c, const float *d_x, float *d_g, const float *d_s,
                        const double *d_alpha, float *d_xt, const CgTrialArgs *trial) {
  const int L = c->L;
  const bool sp = c->path == CCM_PATH_TC_I8SP;
  const float *x1 = d_s != nullptr ? d_xt : d_x;
  const float *x2 = trial ? nullptr : x1 + c->nsp;
  float *g2 = trial ? nullptr : d_g + c->nsp;
  cudaError_t e;

  prof_mark(c);
  e = sp ? i8_prepare_sparse(c, d_x, g2, d_s, d_alpha, d_xt, trial)
         : i8_prepare_dense(c, d_x, g2, d_s, d_alpha, d_xt);
  if (e != cudaSuccess) return e;
  prof_mark(c);

  I8FwdArgs fa{};
  fa.msa = c->d_msa; fa.w = c->d_w; fa.x1 = x1; fa.colmax = c->d_colmax;
  for (int i = 0; i < 3; ++i) fa.r[i] = c->d_rdig[i];
  fa.rnat = c->d_rnat;
  if (trial) fa.sw = trial->sw;
  fa.part_f = c->d_part_f; fa.status = c->d_status;
  fa.L = L; fa.N = c->N; fa.S = c->S; fa.T = c->T; fa.Npad = c->Npad;
  fa.m_tiles = c->Npad / kI8PairM;
  fa.KP = c->KP;
  fa.r_enc = pow2_host(kI8FracBits - c->r_exp);
  fa.acc_wait_cycles = c->acc_wait_cycles;
  const int pair_tiles = fa.m_tiles * c->T;
  const int fpairs = pair_tiles < c->fwd_pairs ? pair_tiles : c->fwd_pairs;
  if (sp)
    e = launch_pdl(i8sp_forward_kernel, dim3(2 * fpairs), dim3(kWgThreads), I8SpSmem::kTotal,
                   c->stream, c->i8sp_maps, fa);
  else
    e = launch_pdl(i8_forward_kernel, dim3(2 * fpairs), dim3(kI8Threads), I8FwdSmem::kTotal,
                   c->stream, c->i8fwd_maps, fa);
  if (e != cudaSuccess) return e;
  prof_mark(c);

  BwdArgs ba{};
  ba.g2 = g2; ba.g1d = c->d_g1d; ba.tiles = c->d_bwd_tiles;
  ba.n_tiles = c->n_bwd_tiles; ba.status = c->d_status; ba.L = L; ba.S = c->S; ba.Npad = c->Npad;
  ba.r_dec = pow2_host(c->r_exp - kI8FracBits);
  ba.acc_wait_cycles = c->bwd_wait_cycles;
  const int bpairs = c->n_bwd_tiles < c->bwd_pairs ? c->n_bwd_tiles : c->bwd_pairs;
  const bool sym = c->gradient != CCM_GRADIENT_PARTIAL;
  if (sp) {
    // the sums and g1 are the backward's own (no finalize)
    ba.cmacc = c->d_cmacc;
    ba.cuts = c->d_cuts;
    ba.vec = (reinterpret_cast<uintptr_t>(g2) & 15) == 0;
    if (trial) {
      ba.sw = trial->sw;
      ba.vec = ((reinterpret_cast<uintptr_t>(ba.sw.g[0]) | reinterpret_cast<uintptr_t>(ba.sw.g[1])) & 15) == 0;
    }
    ba.fin = finalize_args(c, x1, d_g, 2LL * pair_tiles);
    ba.fin.n_part_reg = c->n_part_reg;
    if (g2 && g2 == x2) {
      const long long n = c->nvarp - c->nsp, blocks = (n + 255) / 256;
      ba.fin.squares = c->d_fin_part;
      e = launch_pdl(i8sp_in_place_kernel, dim3((unsigned)(blocks < 1184 ? blocks : 1184)), dim3(256),
                     0, c->stream, g2, n, i8_g2_scale(c), x1, nsingle_of(L), c->d_fin_part);
      if (e != cudaSuccess) return e;
      count_launch(c);
    }
  }
  const dim3 bgrid(2 * bpairs);
  const auto bwd = backward_kernel(sym, sp, c->d_cuts != nullptr);
  e = launch_pdl(bwd, bgrid, dim3(kWgThreads), I8BwdSmem::kTotal, c->stream, c->i8bwd_maps, ba);
  if (e != cudaSuccess) return e;
  prof_mark(c);

  if (!sp && (e = launch_tc_finalize(c, x1, d_g, 2LL * pair_tiles)) != cudaSuccess) return e;
  prof_mark(c);
  count_launch(c, sp ? 2 : 3);
  return cudaGetLastError();
}

cudaError_t i8_configure_kernels() {
  cudaError_t e;
  const int kMax = cudaFuncAttributeMaxDynamicSharedMemorySize;
  // the staged row is S floats: up to L = 2688 (the 227 KB per block, less the
  // kernel's static reduction buffer)
  if ((e = cudaFuncSetAttribute(i8_prep_kernel, (cudaFuncAttribute)kMax, 230000)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(i8sp_digits_kernel<kDigRows>, (cudaFuncAttribute)kMax,
                                (int)sizeof(int) * kDigRows * dig_row_words(kDigGroups))) != cudaSuccess ||
      (e = cudaFuncSetAttribute(i8sp_digits_kernel<kDigRowsFew>, (cudaFuncAttribute)kMax,
                                (int)sizeof(int) * kDigRowsFew * dig_row_words(kDigGroups))) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(i8_forward_kernel, (cudaFuncAttribute)kMax, I8FwdSmem::kTotal)) !=
          cudaSuccess ||
      (e = cudaFuncSetAttribute(i8sp_forward_kernel, (cudaFuncAttribute)kMax, I8SpSmem::kTotal)) !=
          cudaSuccess)
    return e;
  for (int i = 0; i < 8; ++i)
    if ((e = cudaFuncSetAttribute(backward_kernel(i & 1, i & 2, i & 4), (cudaFuncAttribute)kMax,
                                  I8BwdSmem::kTotal)) != cudaSuccess)
      return e;
  return cudaSuccess;
}

cudaError_t i8_forward_max_pairs(int *pairs) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(kI8Threads, 1, 1);
  cfg.dynamicSmemBytes = I8FwdSmem::kTotal;
  *pairs = 0;
  return cudaOccupancyMaxActiveClusters(pairs, i8_forward_kernel, &cfg);
}

cudaError_t i8sp_forward_max_pairs(int *pairs) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(kWgThreads, 1, 1);
  cfg.dynamicSmemBytes = I8SpSmem::kTotal;
  *pairs = 0;
  return cudaOccupancyMaxActiveClusters(pairs, i8sp_forward_kernel, &cfg);
}

cudaError_t i8_backward_max_pairs(int *pairs) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(kWgThreads, 1, 1);
  cfg.dynamicSmemBytes = I8BwdSmem::kTotal;
  *pairs = 0;
  return cudaOccupancyMaxActiveClusters(pairs, backward_kernel(true, false, false), &cfg);
}

// One-hot operands for a context of the integer paths (Npad x S bytes each), and
// for the sparse path the compressed forward operand with its metadata.
cudaError_t i8_build_onehot(ccm_context *c) {
  if (c->path != CCM_PATH_TC_I8SP) {
    const long long total = (long long)c->Npad * c->S;
    i8_onehot_kernel<<<(unsigned)((total + 255) / 256), 256, 0, c->stream>>>(
        c->d_msa, c->d_o1, c->d_o128, c->L, c->N, c->S, c->Npad);
    return cudaGetLastError();
  }
  i8nat_onehot_kernel<<<dim3(c->Npad / 32, c->SB / 128), 128, 0, c->stream>>>(
      c->d_msa, c->d_onat, c->L, c->N, c->Npad / 32);
  const long long bytes = (long long)c->Npad * (c->KP / 8);
  i8sp_onehot_kernel<<<(unsigned)((bytes + 255) / 256), 256, 0, c->stream>>>(
      c->d_msa, reinterpret_cast<uint32_t *>(c->d_ac1), reinterpret_cast<uint32_t *>(c->d_ac128),
      c->d_meta, c->L, c->N, c->KP, c->Npad);
  return cudaGetLastError();
}

// Matrix `mat` of the `mats` side by side of the backward's natural storage
// (i8nat_offset), as Npad x S bytes of the forward's 192-slot groups in 32-row x
// 128-slot tiles, tile (n / 32, s / 128) at 4096 ((s / 128) KB + n / 32), the 16-byte
// chunk c of a row n of 128 slots at chunk c ^ (n & 7): the order in which
// ccm_debug_copy hands these operands out.
void i8nat_to_groups(const ccm_context *c, const uint8_t *nat, int mats, int mat, uint8_t *dst) {
  const int KB = c->Npad / 32;
  for (int s = 0; s < c->S; ++s) {
    const int t = s / Groups192::kSlots, r = s % Groups192::kSlots;
    const int l = t * Groups192::kCols + r % Groups192::kCols;
    int ns = -1;
    if (s == Groups192::kOnes) ns = kQ * c->L;
    else if (r < Groups192::kUsed && l < c->L) ns = (r / Groups192::kCols) * c->L + l;
    for (int n = 0; n < c->Npad; ++n)
      dst[((long long)(s >> 7) * KB + (n >> 5)) * 4096 + (n & 31) * 128 +
          (((((s & 127) >> 4) ^ (n & 7)) & 7) << 4) + (s & 15)] =
          ns < 0 ? 0 : nat[i8nat_offset(n, ns, KB, mats) + (long long)mat * kNatTile];
  }
}

}  // namespace ccm
