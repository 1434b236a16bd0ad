// Elementwise dequantize / unpack kernels (HBM-bound, 128-bit accesses).
#include "common.cuh"

namespace quik {
namespace {

// QUIK src/asymmetric/asymmetric.cu:119-173.  The arithmetic is kept in the reference's order
// with explicit round-to-nearest multiplies and adds so that the compiler cannot contract them
// into fused multiply-adds: out = T( x*(s_r*s_c) + (((z_r + shift*s_r) * wred_c) + y) ).
__device__ __forceinline__ float dequant_value(int acc, float srow, float zrow, float shift,
                                               float scol, float wred, float y) {
  const float sh = __fmul_rn(__fadd_rn(zrow, __fmul_rn(shift, srow)), wred);
  const float xe = __fmul_rn((float)acc, __fmul_rn(srow, scol));
  return __fadd_rn(xe, __fadd_rn(sh, y));
}

// Rows by 32-bit division wherever the matrix allows (a 64-bit one costs more than the eight values it is for).  It may be a dependent
// launch: what the kernel reads comes after its wait, by ordinary loads of pointers that are not declared constant.  Launches after
// it start when it is complete: its result may be a layer's outlier weights, which the ring streaming engine loads before its wait.
template <typename T, int VEC, typename Index>
__global__ void asym_dequantize_kernel(const int32_t *x, const T *meta, const T *scale_col, const T *wred, const T *y, T *__restrict__ out,
                                       Index total, int cols, float shift) {
  const unsigned cvec = (unsigned)cols / VEC;
  pdl_wait();
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (Index)gridDim.x * blockDim.x) {
    const int r = (int)(i / cvec), c0 = (int)(i % cvec) * VEC;
    const float srow = Traits<T>::to_float(meta[2 * (size_t)r]);
    const float zrow = Traits<T>::to_float(meta[2 * (size_t)r + 1]);
    const size_t off = (size_t)r * cols + c0;
    if (VEC == 8) {
      const int4 a0 = reinterpret_cast<const int4 *>(x + off)[0];
      const int4 a1 = reinterpret_cast<const int4 *>(x + off)[1];
      const uint4 yv = *reinterpret_cast<const uint4 *>(y + off);
      const uint4 sv = *reinterpret_cast<const uint4 *>(scale_col + c0);
      const uint4 wv = *reinterpret_cast<const uint4 *>(wred + c0);
      const int acc[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const T *ye = reinterpret_cast<const T *>(&yv);
      const T *se = reinterpret_cast<const T *>(&sv);
      const T *we = reinterpret_cast<const T *>(&wv);
      uint4 o;
      T *oe = reinterpret_cast<T *>(&o);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        oe[j] = Traits<T>::from_float(dequant_value(acc[j], srow, zrow, shift, Traits<T>::to_float(se[j]),
                                                    Traits<T>::to_float(we[j]), Traits<T>::to_float(ye[j])));
      *reinterpret_cast<uint4 *>(out + off) = o;
    } else {
      out[off] = Traits<T>::from_float(dequant_value(x[off], srow, zrow, shift,
                                                     Traits<T>::to_float(scale_col[c0]),
                                                     Traits<T>::to_float(wred[c0]),
                                                     Traits<T>::to_float(y[off])));
    }
  }
}

// QUIK src/symmetric/symmetric.cu:80-113: fp16 per-operation arithmetic.
template <typename X>
__device__ __forceinline__ __half to_half_rn(X v) { return __int2half_rn((int)v); }
template <> __device__ __forceinline__ __half to_half_rn<__half>(__half v) { return v; }

template <typename X>
__global__ void sym_dequantize_kernel(const X *__restrict__ x, const __half *__restrict__ srow,
                                      const __half *__restrict__ scol, const __half *__restrict__ y,
                                      __half *__restrict__ out, int rows, int cols) {
  const size_t total = (size_t)rows * cols;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / cols), c = (int)(i % cols);
    // _rn forms: never contracted into a fused multiply-add, so each operation rounds like the torch
    // expression the reference asserts against (test/python/test_cuaprseLt.py:44-47)
    out[i] = __hadd_rn(__hmul_rn(__hmul_rn(to_half_rn<X>(x[i]), srow[r]), scol[c]), y[i]);
  }
}

// Packed int4 -> int8, 16 bytes in / 32 bytes out per thread step (include/int4.h:78-98 order: low nibble first); one or two
// matrices per launch.
struct Unpack {
  const uint8_t *src;
  int8_t *dst;
  size_t nbytes;
};
__device__ __forceinline__ void unpack_matrix(const Unpack &m, size_t first, size_t step, int vec) {
  if (vec) {
    const size_t nvec = m.nbytes >> 4;
    for (size_t i = first; i < nvec; i += step) {
      const uint4 p = reinterpret_cast<const uint4 *>(m.src)[i];
      const uint32_t w[4] = {p.x, p.y, p.z, p.w};
      uint32_t o[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // sign-extend 8 nibbles: (n ^ 8) - 8 per byte lane
        const uint32_t lo = w[j] & 0x0F0F0F0Fu, hi = (w[j] >> 4) & 0x0F0F0F0Fu;
        const uint32_t slo = __vsub4(lo ^ 0x08080808u, 0x08080808u);
        const uint32_t shi = __vsub4(hi ^ 0x08080808u, 0x08080808u);
        // interleave bytes: lo0 hi0 lo1 hi1 | lo2 hi2 lo3 hi3
        o[2 * j] = __byte_perm(slo, shi, 0x5140);
        o[2 * j + 1] = __byte_perm(slo, shi, 0x7362);
      }
      uint4 *d = reinterpret_cast<uint4 *>(m.dst) + 2 * i;
      d[0] = make_uint4(o[0], o[1], o[2], o[3]);
      d[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
  } else {
    for (size_t i = first; i < m.nbytes; i += step) {
      const int b = m.src[i];
      m.dst[2 * i] = (int8_t)(((b & 0xF) ^ 8) - 8);
      m.dst[2 * i + 1] = (int8_t)((((b >> 4) & 0xF) ^ 8) - 8);
    }
  }
}
// The int4 product widens both operands before it starts: one launch for the two, which the product's own setup overlaps (two
// ordinary launches before).  RELEASE: the product may start early.  Not where the caller has a matrix widened: it may be a layer's
// weights, which the ring streaming engine loads before its wait.
template <bool RELEASE>
__global__ void unpack_int4_kernel(const Unpack a, const Unpack b, int vec) {
  if (RELEASE) pdl_launch_dependents();
  pdl_wait();
  const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  unpack_matrix(a, first, step, vec & 1);
  unpack_matrix(b, first, step, vec >> 1);
}

inline int ew_grid(size_t total, int threads) {
  size_t blocks = (total + threads - 1) / threads;
  size_t cap = (size_t)num_sms() * 16;
  return (int)(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

}  // namespace

int launch_asym_dequantize(const int32_t *x, const void *meta, const void *scale_col,
                           const void *w_reduced, const void *y, void *out, int dtype, int rows,
                           int cols, int bits, cudaStream_t st) {
  if (rows == 0 || cols == 0) return QUIK_OK;
  const float shift = bits == 4 ? 8.0f : 128.0f;
  const bool vec = (cols % 8 == 0) && aligned16(x) && aligned16(y) && aligned16(out) &&
                   aligned16(scale_col) && aligned16(w_reduced);
  const int threads = 256;
  const int grid = ew_grid((size_t)rows * (vec ? cols / 8 : cols), threads);
  const size_t total = (size_t)rows * (vec ? cols / 8 : cols);
  const bool small = total < ((size_t)1 << 31);
  LaunchCfg lc(dim3(grid), dim3(threads), 0, st);
  // A dependent launch for small matrices only.  Its blocks take the SMs as the product's blocks leave them and wait there, and from some size
  // on that costs more than the early start gives.  Product and this, us, dependent and ordinary launch: int32 result of 73 MB 68.6 / 56.8,
  // 144 MB 168 / 145, 187 MB 177 / 140; quantizer, int4 product and this over drawn sizes, speed of the ordinary launch against the
  // dependent one: below 4 MB 0.992, to 16 MB 0.993, to 40 MB 1.002, beyond 1.02.
  if ((size_t)rows * cols * 4 > ((size_t)16 << 20)) lc.cfg.numAttrs = 0;
#define QUIK_DQ_I(T, V, I)                                                                                                     \
  QUIK_CUDA_TRY(cudaLaunchKernelEx(&lc.cfg, asym_dequantize_kernel<T, V, I>, x, static_cast<const T *>(meta),                  \
                                   static_cast<const T *>(scale_col), static_cast<const T *>(w_reduced),                       \
                                   static_cast<const T *>(y), static_cast<T *>(out), (I)total, cols, shift))
#define QUIK_DQ(T, V)                              \
  do {                                             \
    if (small) QUIK_DQ_I(T, V, unsigned);          \
    else QUIK_DQ_I(T, V, unsigned long long);      \
  } while (0)
  if (dtype == QUIK_F16) { if (vec) QUIK_DQ(__half, 8); else QUIK_DQ(__half, 1); }
  else { if (vec) QUIK_DQ(__nv_bfloat16, 8); else QUIK_DQ(__nv_bfloat16, 1); }
#undef QUIK_DQ
#undef QUIK_DQ_I
  return check_launch("asym_dequantize_kernel");
}

int launch_sym_dequantize(const void *x, int x_bits, const void *scale_row, const void *scale_col,
                          const void *y, void *out, int rows, int cols, cudaStream_t st) {
  if (rows == 0 || cols == 0) return QUIK_OK;
  const int threads = 256, grid = ew_grid((size_t)rows * cols, threads);
  auto sr = static_cast<const __half *>(scale_row), sc = static_cast<const __half *>(scale_col),
       yy = static_cast<const __half *>(y);
  __half *o = static_cast<__half *>(out);
  if (x_bits == 8) sym_dequantize_kernel<int8_t><<<grid, threads, 0, st>>>(static_cast<const int8_t *>(x), sr, sc, yy, o, rows, cols);
  else if (x_bits == 16) sym_dequantize_kernel<__half><<<grid, threads, 0, st>>>(static_cast<const __half *>(x), sr, sc, yy, o, rows, cols);
  else sym_dequantize_kernel<int32_t><<<grid, threads, 0, st>>>(static_cast<const int32_t *>(x), sr, sc, yy, o, rows, cols);
  return check_launch("sym_dequantize_kernel");
}

template <bool RELEASE>
static int launch_unpack(const Unpack &ua, const Unpack &ub, cudaStream_t st) {
  if (ua.nbytes + ub.nbytes == 0) return QUIK_OK;
  auto vec = [](const Unpack &m) { return (m.nbytes % 16 == 0) && aligned16(m.src) && aligned16(m.dst); };
  const size_t steps_a = vec(ua) ? ua.nbytes / 16 : ua.nbytes, steps_b = vec(ub) ? ub.nbytes / 16 : ub.nbytes;
  const int threads = 256;
  LaunchCfg lc(dim3(ew_grid(steps_a > steps_b ? steps_a : steps_b, threads)), dim3(threads), 0, st);
  QUIK_CUDA_TRY(cudaLaunchKernelEx(&lc.cfg, unpack_int4_kernel<RELEASE>, ua, ub, (int)vec(ua) | (int)vec(ub) << 1));
  return check_launch("unpack_int4_kernel");
}

int launch_unpack_int4(const uint8_t *src, int8_t *dst, int rows, int cols, cudaStream_t st) {
  return launch_unpack<false>(Unpack{src, dst, (size_t)rows * (cols / 2)}, Unpack{nullptr, nullptr, 0}, st);
}

int launch_unpack_int4_operands(const uint8_t *a, int8_t *a8, int rows_a, const uint8_t *b, int8_t *b8, int rows_b, int cols, cudaStream_t st) {
  return launch_unpack<true>(Unpack{a, a8, (size_t)rows_a * (cols / 2)}, Unpack{b, b8, (size_t)rows_b * (cols / 2)}, st);
}

}  // namespace quik
