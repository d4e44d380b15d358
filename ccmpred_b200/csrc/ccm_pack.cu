// Parameters of the autograd wrapper to and from the padded layout, one pass each:
//   V (L, 20) and W (L, L, 21, 21), W[k, j, b, a], any strides
//   x[a L + j] = V[j, a];  x[nsp + ((b L + k) 32 + a) L + j] = W[k, j, b, a]
// W's states are innermost, x's columns: a block takes one k and a run of JT columns j
// with all 441 state pairs through shared memory (pitch JT + 1 words: no bank conflict),
// so that both sides are read and written in runs.  Bound by memory (W and x once each,
// 15 and 12 us at L = 150), which takes many loads in flight and little arithmetic per
// element: the threads keep their place in a row and step by strides, seven or sixteen
// loads at a time.  With an index divided out per element and one load in flight packing
// took 41 and unpacking 48 us at L = 150, here 23 and 17.
// (As torch operations -- permute, pad, concatenate and their backwards -- this was
// some twenty launches and three copies of x: 300 of an evaluation's 500 us at L = 150.)
#include <cuda_runtime.h>

#include "ccm_internal.cuh"
#include "ccm_layout.cuh"

namespace ccm {

struct PackStrides {
  long long v[2], w[4];
};

template <typename T> constexpr int kPackJ = sizeof(T) == 4 ? 16 : 8;
constexpr int kPackThreads = 256;

template <typename T, bool UNPACK>
__global__ void __launch_bounds__(kPackThreads) pack_kernel(T *V, T *W, T *x, const T *scale,
                                                            PackStrides st, int L) {
  constexpr int JT = kPackJ<T>, kQQ = kQ * kQ;
  __shared__ T tile[kQQ * (JT + 1)];
  const int jt = blockIdx.x, k = blockIdx.y, j0 = jt * JT;
  const long long nsp = nsingle_padded_of(L);
  const T s = UNPACK ? *scale : T(1);
  if (k == L) {  // the single fields, and x's padding after them
    for (long long i = jt * (long long)kPackThreads + threadIdx.x; i < nsp;
         i += (long long)gridDim.x * kPackThreads) {
      const bool real = i < nsingle_of(L);
      const long long at = real ? i % L * st.v[0] + i / L * st.v[1] : 0;
      if (!UNPACK) x[i] = real ? V[at] : T(0);
      else if (real && V) V[at] = s * x[i];
    }
    return;
  }
  if (UNPACK && !W) return;
  // x's side: thread (jj, gr) has column jj of the rows (b, k, a), a = gr, gr + kG, ...;
  // seven states b at a time
  constexpr int kG = kPackThreads / JT, kB = 7;
  const int jj = threadIdx.x % JT, gr = threadIdx.x / JT;
  T *const px = x + nsp + ((long long)k * kQPad + gr) * L + j0 + jj;
  const long long bstep = (long long)kQPad * L * L;
  auto rows = [&](auto move) {
    if (j0 + jj >= L) return;
#pragma unroll
    for (int h = 0; h < kQPad / kG; ++h) {
      const int a = gr + h * kG;
      if (UNPACK && a >= kQ) break;
      T *p = px + (long long)(h * kG) * L;
      int t = a * (JT + 1) + jj;
      for (int b = 0; b < kQ; b += kB, p += kB * bstep, t += kB * kQ * (JT + 1)) move(p, t, a < kQ);
    }
  };
  // W's side: thread has the state pairs threadIdx.x and threadIdx.x + 256 of every
  // column, eight columns at a time
  constexpr int kP = (kQQ + kPackThreads - 1) / kPackThreads, kC = 8;
  long long wp[kP];
#pragma unroll
  for (int u = 0; u < kP; ++u) {
    const int ba = threadIdx.x + u * kPackThreads;
    wp[u] = ba / kQ * st.w[2] + ba % kQ * st.w[3];
  }
  T *pw = W + k * st.w[0] + j0 * st.w[1];
  auto in = [&](int u, int c) { return threadIdx.x + u * kPackThreads < kQQ && j0 + c < L; };
  const int t0 = threadIdx.x * (JT + 1);
  constexpr int kTU = kPackThreads * (JT + 1);
  if (!UNPACK) {
    for (int c0 = 0; c0 < JT; c0 += kC) {
      T v[kP][kC];
#pragma unroll
      for (int u = 0; u < kP; ++u)
#pragma unroll
        for (int c = 0; c < kC; ++c)
          v[u][c] = in(u, c0 + c) ? pw[(c0 + c) * st.w[1] + wp[u]] : T(0);
#pragma unroll
      for (int u = 0; u < kP; ++u)
#pragma unroll
        for (int c = 0; c < kC; ++c)
          if (in(u, c0 + c)) tile[t0 + u * kTU + c0 + c] = v[u][c];
    }
    __syncthreads();
    rows([&](T *p, int t, bool real) {
#pragma unroll
      for (int b = 0; b < kB; ++b) p[b * bstep] = real ? tile[t + b * kQ * (JT + 1)] : T(0);
    });
  } else {
    rows([&](const T *p, int t, bool) {
      T v[kB];
#pragma unroll
      for (int b = 0; b < kB; ++b) v[b] = p[b * bstep];
#pragma unroll
      for (int b = 0; b < kB; ++b) tile[t + b * kQ * (JT + 1)] = v[b];
    });
    __syncthreads();
    for (int c0 = 0; c0 < JT; c0 += kC)
#pragma unroll
      for (int u = 0; u < kP; ++u)
#pragma unroll
        for (int c = 0; c < kC; ++c)
          if (in(u, c0 + c)) pw[(c0 + c) * st.w[1] + wp[u]] = s * tile[t0 + u * kTU + c0 + c];
  }
}

template <typename T, bool UNPACK>
static cudaError_t launch_pack(void *V, void *W, void *x, const void *scale, const PackStrides &st,
                               int L, cudaStream_t stream) {
  const dim3 grid((L + kPackJ<T> - 1) / kPackJ<T>, L + 1);
  pack_kernel<T, UNPACK><<<grid, kPackThreads, 0, stream>>>(
      static_cast<T *>(V), static_cast<T *>(W), static_cast<T *>(x), static_cast<const T *>(scale), st, L);
  return cudaGetLastError();
}

}  // namespace ccm

using namespace ccm;

extern "C" CCM_API int ccm_pack_parameters(const void *V, const long long *v_strides, const void *W,
                                           const long long *w_strides, int ncol, int elem_bytes,
                                           void *x, void *stream) {
  if (!V || !W || !x || !v_strides || !w_strides || ncol <= 0 || (elem_bytes != 4 && elem_bytes != 8))
    return set_last_error(CCM_ERR_INVALID, "ccm_pack_parameters: invalid arguments");
  PackStrides st;
  for (int i = 0; i < 2; ++i) st.v[i] = v_strides[i];
  for (int i = 0; i < 4; ++i) st.w[i] = w_strides[i];
  void *v = const_cast<void *>(V), *w = const_cast<void *>(W);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = elem_bytes == 4 ? launch_pack<float, false>(v, w, x, nullptr, st, ncol, s)
                                        : launch_pack<double, false>(v, w, x, nullptr, st, ncol, s);
  if (e != cudaSuccess)
    return set_last_error(CCM_ERR_CUDA, "ccm_pack_parameters: %s", cudaGetErrorString(e));
  return CCM_OK;
}

extern "C" CCM_API int ccm_unpack_gradient(const void *g, const void *scale, int ncol, int elem_bytes,
                                           void *dV, const long long *v_strides, void *dW,
                                           const long long *w_strides, void *stream) {
  if (!g || !scale || !v_strides || !w_strides || ncol <= 0 || (elem_bytes != 4 && elem_bytes != 8))
    return set_last_error(CCM_ERR_INVALID, "ccm_unpack_gradient: invalid arguments");
  PackStrides st;
  for (int i = 0; i < 2; ++i) st.v[i] = v_strides[i];
  for (int i = 0; i < 4; ++i) st.w[i] = w_strides[i];
  void *x = const_cast<void *>(g);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = elem_bytes == 4 ? launch_pack<float, true>(dV, dW, x, scale, st, ncol, s)
                                        : launch_pack<double, true>(dV, dW, x, scale, st, ncol, s);
  if (e != cudaSuccess)
    return set_last_error(CCM_ERR_CUDA, "ccm_unpack_gradient: %s", cudaGetErrorString(e));
  return CCM_OK;
}
