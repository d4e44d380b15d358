// Identity-threshold sequence reweighting, bit-exact with the serial reference
// (src/reweighting.c:9-58).
//
// ids(i,j) = #{k : X_ik == X_jk} = L - diff(i,j).  The alignment is packed into bit
// planes, one 32-bit word per 32 columns and bit of the state, so that 32 columns of
// a pair take five three-input logic operations, a population count and an addition.
// A 64 x 64 tile of pairs is given up as soon as every pair of it differs in too many
// columns to reach the threshold: for unrelated rows that is a quarter of the way.
// count_i gets +1 for every j != i with ids > idthres and +2 for j == i (the
// reference's i <= j loop visits the diagonal once and increments w[i] twice).
// Counts are integers, so the order of the atomic additions does not matter.
#include <climits>
#include <cstdio>

#include <cuda_runtime.h>

#include "ccm_internal.cuh"

namespace ccm {

constexpr int kRwTile = 64;
constexpr int kRwChunk = 32;  // packed words per shared-memory chunk (byte variant below)
constexpr int kRwWords = 8;   // plane words (32 columns each) per shared-memory chunk
constexpr int kRwPitch = kRwWords + 2;  // words: 8-byte loads of 16 neighbouring rows meet no conflict

// Bit planes of the alignment: word w of plane p of row n at planes[(p N + n) words + w],
// words = a multiple of kRwWords, zero past L.  One warp packs 256 columns of a row.  All
// eight planes are written; *high becomes nonzero if a state uses bits 5..7 (a caller's
// states above 31; the alphabet needs five bits).
__global__ void __launch_bounds__(256) rw_planes_kernel(const uint8_t *__restrict__ msa,
                                                        uint32_t *__restrict__ planes,
                                                        int *__restrict__ high, int L, int N,
                                                        int words) {
  const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, chunks = words / kRwWords;
  const int n = (int)(warp / chunks), w0 = (int)(warp % chunks) * kRwWords;
  if (n >= N) return;
  uint32_t lo = 0, hi = 0, any = 0;  // this lane's word: plane lane / 8 (and + 4), word lane % 8
#pragma unroll
  for (int j = 0; j < kRwWords; ++j) {
    const int k = (w0 + j) * 32 + lane;
    const uint32_t x = k < L ? msa[(long long)n * L + k] : 0u;
    any |= x;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const uint32_t v = __ballot_sync(0xffffffffu, (x >> p) & 1);
      if (lane == (p & 3) * 8 + j) { if (p < 4) lo = v; else hi = v; }
    }
  }
  const long long at = ((long long)(lane >> 3) * N + n) * words + w0 + (lane & 7);
  planes[at] = lo;
  planes[at + 4LL * N * words] = hi;
  if (__any_sync(0xffffffffu, any > 31) && lane == 0) *high = 1;
}

// One 64 x 64 tile of row pairs per block (blockIdx.x: the tiles on and above the
// diagonal), 4 x 4 pairs per thread: rows ty + 16 u against rows tx + 16 v.  Bound by
// the integer pipe: six operations per 32 columns of a pair; byte compares (a compare, a
// population count and an addition per 4 columns) without the early end took 16 ms for
// L = 1000, N = 20000 with 30 % near-duplicate rows, this takes 2.
template <int PLANES>
__device__ __forceinline__ void rw_diff_chunk(const uint32_t *As, const uint32_t *Bs, int ty, int tx,
                                              int pairs, int (&diff)[4][4]) {
#pragma unroll 1
  for (int q = 0; q < pairs; ++q) {
    uint2 d[4][4];
#pragma unroll
    for (int p = 0; p < PLANES; ++p) {
      uint2 a[4], b[4];
      const uint32_t *ap = As + p * kRwTile * kRwPitch + 2 * q, *bp = Bs + p * kRwTile * kRwPitch + 2 * q;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a[u] = *reinterpret_cast<const uint2 *>(ap + (ty + 16 * u) * kRwPitch);
        b[u] = *reinterpret_cast<const uint2 *>(bp + (tx + 16 * u) * kRwPitch);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          if (p == 0) d[u][v] = make_uint2(0, 0);
          d[u][v].x |= a[u].x ^ b[v].x;
          d[u][v].y |= a[u].y ^ b[v].y;
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) diff[u][v] += __popc(d[u][v].x) + __popc(d[u][v].y);
  }
}

__global__ void __launch_bounds__(256, 3) rw_count_kernel(const uint32_t *__restrict__ planes,
                                                       const int *__restrict__ high, int N, int L,
                                                       int words, int idthres,
                                                       int *__restrict__ counts) {
  // tile IB <= JB from the linear index t = JB (JB + 1) / 2 + IB
  const long long t = blockIdx.x;
  int JB = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while ((long long)(JB + 1) * (JB + 2) / 2 <= t) ++JB;
  while ((long long)JB * (JB + 1) / 2 > t) --JB;
  const int IB = (int)(t - (long long)JB * (JB + 1) / 2);
  extern __shared__ __align__(16) uint32_t sm[];  // [A | B][plane][row][kRwPitch]
  __shared__ int ci[kRwTile], cj[kRwTile];
  const int np = *high ? 8 : 5;
  uint32_t *As = sm, *Bs = sm + np * kRwTile * kRwPitch;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int i0 = IB * kRwTile, j0 = JB * kRwTile;
  if (threadIdx.x < kRwTile) { ci[threadIdx.x] = 0; cj[threadIdx.x] = 0; }
  int diff[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) diff[u][v] = 0;
  // ids > idthres  <=>  diff < limit
  const int limit = L - idthres;
  const int used = (L + 31) / 32;
  bool open = true;  // some pair of this warp may still reach the threshold
  for (int w0 = 0; w0 < used; w0 += kRwWords) {
    if (!__syncthreads_or(open)) break;
    for (int e = threadIdx.x; e < 2 * np * kRwTile * (kRwWords / 4); e += 256) {
      const int c = e % (kRwWords / 4), r = e / (kRwWords / 4) % kRwTile;
      const int ps = e / (kRwWords / 4 * kRwTile), p = ps % np, side = ps / np;
      const int row = (side ? j0 : i0) + r;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (row < N)
        v = *reinterpret_cast<const uint4 *>(planes + ((long long)p * N + row) * words + w0 + 4 * c);
      uint2 *to = reinterpret_cast<uint2 *>(sm + (ps * kRwTile + r) * kRwPitch + 4 * c);
      to[0] = make_uint2(v.x, v.y);
      to[1] = make_uint2(v.z, v.w);
    }
    __syncthreads();
    if (open) {
      const int pairs = (min(used - w0, kRwWords) + 1) / 2;
      if (np == 5) rw_diff_chunk<5>(As, Bs, ty, tx, pairs, diff);
      else rw_diff_chunk<8>(As, Bs, ty, tx, pairs, diff);
      int least = diff[0][0];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) least = min(least, diff[u][v]);
      open = __any_sync(0xffffffffu, least < limit);
    }
  }
  __syncthreads();
  if (open) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int il = ty + 16 * u, jl = tx + 16 * v;
        const int i = i0 + il, j = j0 + jl;
        if (i >= N || j >= N || diff[u][v] >= limit) continue;
        if (IB == JB) {
          if (i < j) { atomicAdd(&ci[il], 1); atomicAdd(&ci[jl], 1); }
          else if (i == j) atomicAdd(&ci[il], 2);
        } else {
          atomicAdd(&ci[il], 1);
          atomicAdd(&cj[jl], 1);
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < kRwTile) {
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.x;
    if (i < N && ci[threadIdx.x]) atomicAdd(&counts[i], ci[threadIdx.x]);
    if (IB != JB && j < N && cj[threadIdx.x]) atomicAdd(&counts[j], cj[threadIdx.x]);
  }
}

// w_i = (float)(1. / ((float)count_i - 1)) as in src/reweighting.c:43-45
__global__ void rw_weights_kernel(const int *__restrict__ counts, float *__restrict__ w, int N) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const float cf = (float)counts[i];
  w[i] = (float)(1.0 / (double)(cf - 1.0f));
}

cudaError_t reweight_counts(int device, const uint8_t *d_msa, int L, int N, int idthres,
                            int *d_counts, cudaStream_t stream) {
  // identities are 0 .. L: a threshold beyond them is as good as one next to them (and
  // L - idthres stays an int; NaN and what an int does not hold come as INT_MIN)
  idthres = idthres < -1 ? -1 : idthres > L ? L : idthres;
  const long long nb = (N + (long long)kRwTile - 1) / kRwTile, tiles = nb * (nb + 1) / 2;
  if (tiles > INT_MAX) return cudaErrorInvalidConfiguration;  // 4,194,240 rows
  const int words = ((L + 31) / 32 + kRwWords - 1) / kRwWords * kRwWords;
  const size_t plane_bytes = sizeof(uint32_t) * 8 * (size_t)N * words;
  uint32_t *planes = nullptr;  // the planes, then the flag of states above 31
  cudaError_t e = pool_alloc(device, reinterpret_cast<void **>(&planes), plane_bytes + 16, stream);
  if (e != cudaSuccess) return e;
  int *high = reinterpret_cast<int *>(reinterpret_cast<char *>(planes) + plane_bytes);
  cudaMemsetAsync(high, 0, sizeof(int), stream);
  cudaMemsetAsync(d_counts, 0, sizeof(int) * N, stream);
  const long long warps = (long long)N * (words / kRwWords);
  rw_planes_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, stream>>>(d_msa, planes, high, L, N, words);
  constexpr int kSmem = 2 * 8 * kRwTile * kRwPitch * 4;  // 40 KB for eight planes
  rw_count_kernel<<<(unsigned)tiles, 256, kSmem, stream>>>(planes, high, N, L, words, idthres, d_counts);
  cudaFreeAsync(planes, stream);
  return cudaGetLastError();
}

cudaError_t reweight_weights(const int *d_counts, float *d_w, int N, cudaStream_t stream) {
  rw_weights_kernel<<<(N + 255) / 256, 256, 0, stream>>>(d_counts, d_w, N);
  return cudaGetLastError();
}

}  // namespace ccm

// ----------------------------------------------------------------------------
// Allocation-free variant of the sequence reweighting (ccm_calculate_weights_noalloc).
//
// Its only scratch, one identity count per sequence, lives in the file-scope
// device array below instead of memory obtained from cudaMalloc/cudaMallocAsync,
// and the count kernel packs the alignment bytes into words in shared memory
// instead of in a packed copy in global memory.  The array is part of the
// library image: every GPU that loads the library holds it until the process
// exits.  All calls share it and it keeps the counts of the last call, so each
// call clears the part it uses first; calls that overlap on the GPU (different
// streams, or different host threads on one device) race on it.
namespace ccm {

constexpr int kNoAllocMaxRows = 262144;  // 1 MiB of int counts
static __device__ __align__(256) int g_noalloc_counts[kNoAllocMaxRows];

__global__ void __launch_bounds__(256) rw_count_bytes_kernel(const uint8_t *__restrict__ msa,
                                                             int L, int N, int words, int npad,
                                                             int idthres, int *__restrict__ counts) {
  const int IB = blockIdx.y, JB = blockIdx.x;
  if (JB < IB) return;
  __shared__ uint32_t As[kRwTile][kRwChunk + 1];
  __shared__ uint32_t Bs[kRwTile][kRwChunk + 1];
  __shared__ int ci[kRwTile], cj[kRwTile];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int i0 = IB * kRwTile, j0 = JB * kRwTile;
  if (threadIdx.x < kRwTile) { ci[threadIdx.x] = 0; cj[threadIdx.x] = 0; }
  int ids[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) ids[u][v] = 0;

  for (int w0 = 0; w0 < words; w0 += kRwChunk) {
    __syncthreads();
    // bytes straight into the word rows (byte b of word wd = column 4 wd + b):
    // consecutive threads read consecutive bytes of one row, so each warp load
    // covers one 32-byte sector of the alignment
    constexpr int kRowBytes = 4 * kRwChunk;
    for (int e = threadIdx.x; e < kRwTile * kRowBytes; e += blockDim.x) {
      const int r = e / kRowBytes, bt = e % kRowBytes;
      const int k = w0 * 4 + bt;
      const int ia = i0 + r, jb = j0 + r;
      const bool in = k < L;
      reinterpret_cast<uint8_t *>(&As[r][0])[bt] =
          (in && ia < N) ? msa[(long long)ia * L + k] : (uint8_t)0;
      reinterpret_cast<uint8_t *>(&Bs[r][0])[bt] =
          (in && jb < N) ? msa[(long long)jb * L + k] : (uint8_t)0;
    }
    __syncthreads();
    const int wmax = (words - w0) < kRwChunk ? (words - w0) : kRwChunk;
    for (int wd = 0; wd < wmax; ++wd) {
      uint32_t a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = As[ty * 4 + u][wd];
#pragma unroll
      for (int v = 0; v < 4; ++v) b[v] = Bs[tx * 4 + v][wd];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) ids[u][v] += __popc(__vcmpeq4(a[u], b[v]));
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int il = ty * 4 + u, jl = tx * 4 + v;
      const int i = i0 + il, j = j0 + jl;
      if (i >= N || j >= N) continue;
      const int same = ids[u][v] / 8 - npad;
      if (same <= idthres) continue;
      if (IB == JB) {
        if (i < j) { atomicAdd(&ci[il], 1); atomicAdd(&ci[jl], 1); }
        else if (i == j) atomicAdd(&ci[il], 2);
      } else {
        atomicAdd(&ci[il], 1);
        atomicAdd(&cj[jl], 1);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < kRwTile) {
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.x;
    if (i < N && ci[threadIdx.x]) atomicAdd(&counts[i], ci[threadIdx.x]);
    if (IB != JB && j < N && cj[threadIdx.x]) atomicAdd(&counts[j], cj[threadIdx.x]);
  }
}

}  // namespace ccm

// See include/ccmpred_b200.h.  Every call looks up the device address of the
// count array with cudaGetSymbolAddress in the context that is current on the
// calling thread -- host code must not use the array's name as a device
// pointer, and an address found in one context (the device's primary context,
// say) is not valid in another context of the same device.  The lookup
// allocates nothing once the library's module is loaded in that context (the
// first call in a context loads it); then a call enqueues a memset and two
// kernels.
extern "C" CCM_API int ccm_calculate_weights_noalloc(const unsigned char *d_msa, int ncol,
                                                     int nrow, float threshold, float *d_w,
                                                     void *stream) {
  using namespace ccm;
  if (!d_msa || !d_w || ncol <= 0 || nrow <= 0) {
    return set_last_error(CCM_ERR_INVALID, "ccm_calculate_weights_noalloc: invalid arguments");
  }
  if (nrow > kNoAllocMaxRows) {
    return set_last_error(CCM_ERR_INVALID,
                          "ccm_calculate_weights_noalloc: nrow=%d exceeds the fixed scratch of %d "
                          "sequences",
                          nrow, kNoAllocMaxRows);
  }
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_counts);
  if (e != cudaSuccess || !p) {
    return set_last_error(CCM_ERR_CUDA,
                          "ccm_calculate_weights_noalloc: cudaGetSymbolAddress failed in the "
                          "current context (%s)",
                          cudaGetErrorString(e));
  }
  int *counts = static_cast<int *>(p);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float prod = threshold * (float)(uint64_t)ncol;  // src/reweighting.c:10
  const int idthres = (int)ceil((double)prod);
  const int words = (ncol + 3) / 4;
  const int npad = words * 4 - ncol;
  e = cudaMemsetAsync(counts, 0, sizeof(int) * (size_t)nrow, s);
  if (e == cudaSuccess) {
    const int nb = (nrow + kRwTile - 1) / kRwTile;
    rw_count_bytes_kernel<<<dim3(nb, nb), 256, 0, s>>>(d_msa, ncol, nrow, words, npad, idthres,
                                                        counts);
    rw_weights_kernel<<<(nrow + 255) / 256, 256, 0, s>>>(counts, d_w, nrow);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    return set_last_error(CCM_ERR_CUDA, "ccm_calculate_weights_noalloc: %s", cudaGetErrorString(e));
  }
  return CCM_OK;
}
