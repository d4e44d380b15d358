// Parameters of the autograd wrapper to and from the padded layout, one pass each:
//   V (L, 20) and W (L, L, 21, 21), W[k, j, b, a], any strides
//   x[a L + j] = V[j, a];  x[nsp + ((b L + k) 32 + a) L + j] = W[k, j, b, a]
// W's states are innermost, x's columns: a block takes one k and a run of JT columns j
// with all 441 state pairs through shared memory (pitch JT + 1 words: no bank conflict),
// so that both sides are read and written in runs.  Bound by memory: W and x once each.
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
  T *const w = W + k * st.w[0];
  // x's side: JT consecutive columns of a row (b, k, a)
  auto rows = [&](auto f) {
    const int states = UNPACK ? kQ : kQPad;
    for (int i = threadIdx.x; i < kQ * states * JT; i += kPackThreads) {
      const int jj = i % JT, a = i / JT % states, b = i / (JT * states);
      if (j0 + jj < L) f(x + nsp + (((long long)b * L + k) * kQPad + a) * L + j0 + jj, b, a, jj);
    }
  };
  // W's side: the state pairs of one column
  auto pairs = [&](auto f) {
    for (int i = threadIdx.x; i < kQQ * JT; i += kPackThreads) {
      const int ba = i % kQQ, jj = i / kQQ;
      if (j0 + jj < L)
        f(w + (j0 + jj) * st.w[1] + ba / kQ * st.w[2] + ba % kQ * st.w[3], ba * (JT + 1) + jj);
    }
  };
  if (!UNPACK) {
    pairs([&](const T *p, int t) { tile[t] = *p; });
    __syncthreads();
    rows([&](T *p, int b, int a, int jj) { *p = a < kQ ? tile[(b * kQ + a) * (JT + 1) + jj] : T(0); });
  } else {
    rows([&](const T *p, int b, int a, int jj) { tile[(b * kQ + a) * (JT + 1) + jj] = *p; });
    __syncthreads();
    pairs([&](T *p, int t) { *p = s * tile[t]; });
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
