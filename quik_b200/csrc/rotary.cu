// Rotary position embedding applied in place to the q and k projections of a decoder block: the step between
// the q/k/v layers and attention (the caller after the quantized layers; QUIK experiments/llama.py leaves it to
// transformers' LlamaAttention).  One pass over q and k: 16-byte loads of the two halves of a head, the
// angle tables read once per token, each product and sum rounded to the storage type like the elementwise torch
// expression  x * cos + rotate_half(x) * sin  rounds them (so results are bit-identical to it).
#include "common.cuh"

namespace quik {
namespace {

// A CTA takes whole tokens, its threads the 16-byte pieces of the token's heads, so that the one division left is of 32 bits.  (Heads
// and tokens by 64-bit division of a flat index, in a launch that waited for its predecessor to end: 14 us for q and k of
// [2048, 4096].)
template <typename T>
__global__ void rotary_kernel(T *q, T *k, const T *cos_t, const T *sin_t, int tokens, int q_heads, int k_heads, int head_dim) {
  const int half = head_dim / 2;
  const unsigned vec_per_head = (unsigned)half / 8, pieces = (unsigned)(q_heads + k_heads) * vec_per_head;
  pdl_wait();      // (launches after this one start when it is complete)
  for (int t = blockIdx.x; t < tokens; t += gridDim.x) {
    for (unsigned i = threadIdx.x; i < pieces; i += blockDim.x) {
      const int h = (int)(i / vec_per_head), v = (int)(i - (unsigned)h * vec_per_head);
      T *base = h < q_heads ? q + ((size_t)t * q_heads + h) * head_dim
                            : k + ((size_t)t * k_heads + (h - q_heads)) * head_dim;
      uint4 lo = *reinterpret_cast<const uint4 *>(base + v * 8);
      uint4 hi = *reinterpret_cast<const uint4 *>(base + half + v * 8);
      const uint4 cv = *reinterpret_cast<const uint4 *>(cos_t + (size_t)t * half + v * 8);
      const uint4 sv = *reinterpret_cast<const uint4 *>(sin_t + (size_t)t * half + v * 8);
      T *l = reinterpret_cast<T *>(&lo), *u = reinterpret_cast<T *>(&hi);
      const T *c = reinterpret_cast<const T *>(&cv), *s = reinterpret_cast<const T *>(&sv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = Traits<T>::to_float(l[j]), b = Traits<T>::to_float(u[j]);
        const float cc = Traits<T>::to_float(c[j]), ss = Traits<T>::to_float(s[j]);
        // every product of two 11-bit (8-bit) significands is exact in fp32: rounding it to T equals the
        // storage-type multiply; the sums likewise
        const float ac = Traits<T>::to_float(Traits<T>::from_float(__fmul_rn(a, cc)));
        const float nbs = Traits<T>::to_float(Traits<T>::from_float(__fmul_rn(-b, ss)));
        const float bc = Traits<T>::to_float(Traits<T>::from_float(__fmul_rn(b, cc)));
        const float as = Traits<T>::to_float(Traits<T>::from_float(__fmul_rn(a, ss)));
        l[j] = Traits<T>::from_float(__fadd_rn(ac, nbs));
        u[j] = Traits<T>::from_float(__fadd_rn(bc, as));
      }
      *reinterpret_cast<uint4 *>(base + v * 8) = lo;
      *reinterpret_cast<uint4 *>(base + half + v * 8) = hi;
    }
  }
}

}  // namespace

int launch_rotary(void *q, void *k, const void *cos_t, const void *sin_t, int dtype, int tokens, int q_heads,
                  int k_heads, int head_dim, cudaStream_t st) {
  if (tokens == 0 || q_heads + k_heads == 0) return QUIK_OK;
  const int cap = num_sms() * 8;
  LaunchCfg lc(dim3(tokens < cap ? tokens : cap), dim3(256), 0, st);
  auto launch = [&](auto zero) {
    using T = decltype(zero);
    return cudaLaunchKernelEx(&lc.cfg, rotary_kernel<T>, static_cast<T *>(q), static_cast<T *>(k), static_cast<const T *>(cos_t),
                              static_cast<const T *>(sin_t), tokens, q_heads, k_heads, head_dim);
  };
  if (dtype == QUIK_F16) QUIK_CUDA_TRY(launch(__half()));
  else QUIK_CUDA_TRY(launch(__nv_bfloat16()));
  return check_launch("rotary_kernel");
}

}  // namespace quik
