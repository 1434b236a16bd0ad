// Epilogue of the tiled tcgen05 GEMMs (gemm_tcgen05.cu, gemm_tcgen05_ts.cu): launch parameters and the work of
// the epilogue warps of a CTA -- rounding the outlier product and keeping it, the dequantize arithmetic of
// QUIK src/asymmetric/asymmetric.cu:134-146 and the stores of the finished tile.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "tcgen05_ptx.cuh"

namespace quik {

namespace {

constexpr int BLOCK_M = 128;
constexpr int STAGE_K_BYTES = 128;           // one 128B-swizzle row of K per stage
constexpr int EPI_BUF_BYTES = 32 * 32;       // output staging of one epilogue warp: 32 rows x 32 bytes
constexpr int SMEM_LIMIT = 227 * 1024;

struct GemmParams {
  int M, N;
  int block_n;                    // tile width: multiple of 16
  int split_n;                    // columns of a tile that each group of four epilogue warps takes (multiple of 32)
  int num_m_tiles, num_tiles;
  int int_kb, fp_kb;              // k-blocks per tile: integer (128 codes each) and outlier (64 elems)
  uint32_t idesc_int, idesc_fp;   // tcgen05 instruction descriptors
  int mode;                       // 0: int32 C, 1: dequantize
  int acc_shift;                  // the integer accumulator holds the product times 2^acc_shift (operands widened on chip)
  int a_slots;                    // operand slots in tensor memory (engine with the token operand in tensor memory)
  int l2_hint;                    // token-operand loads carry an L2 evict-last hint
  int32_t *C;
  void *out;
  long long ldo;                  // row pitch of `out` in elements (>= N)
  const void *row_scale;          // element (row * row_stride)
  const void *row_zero;           // may be NULL
  int row_stride;
  const void *scale_col, *w_reduced, *bias, *y;
  float shift_value;
  int vec_out;                    // 16-byte stores allowed (pitch and base aligned)
  int vec_y;
  unsigned long long *dbg;         // optional per-CTA cycle counters (16 per CTA), NULL = off
  unsigned int *status;            // device status word that a wait which ran out sets
};

template <typename T> __device__ __forceinline__ float ldf(const void *p, size_t i) {
  return Traits<T>::to_float(static_cast<const T *>(p)[i]);
}

// ---------------------------------------------------------------------------------------------
// Work of one CTA (or pair) = its tiles t_0, t_1, ...  Tensor memory holds two accumulator regions.  INT(t_j), the integer
// product (s32), lives in region j & 1; FP(t_j), the outlier product (f32), is issued in the middle of INT(t_j) into the other
// region, which the epilogue of t_{j-1} has left by then.  The epilogue warps round FP(t_j) + bias to T and keep it in
// registers (drain), which frees that region for INT(t_{j+1}), and combine it with the integer product when that is complete
// (finish).  So both hide behind integer products and only the last tile's finish has nothing to hide behind.
// (Before, FP(t_{j+1}) was issued in the middle of INT(t_j), its rounded value parked in the tile's place in `out` until
// INT(t_{j+1}) was complete and fetched back in the epilogue, and the first drain had nothing to hide behind.  Llama-2-7B at 2048
// tokens, before and now: drain 6.1 -> 3.6 and finish 9.2 -> 8.6 thousand cycles per 256 x 224 tile, the issuing warp waits for a
// free region 23.4 of 136 -> 12.7 of 121 thousand cycles in the qkv layer and 58 of 242 -> 23.7 of 206 in gate+up; 87.5 -> 81.4 us
// and 155.4 -> 140.3 us.)
// This walks the k-blocks in issue order; fn(j, fp, kb) returns false to stop.  `fp` is a compile-time flag (std::true_type /
// std::false_type): a narrow tile's block occupies the tensor pipe for less than 200 cycles, the issuing warp has none to spare
// for choosing between the two kinds of instruction.
template <bool HAS_FP, typename Fn>
__device__ __forceinline__ void for_each_block(int n_local, int int_kb, int fp_kb, Fn fn) {
  const int int_half = (int_kb + 1) / 2;
  for (int j = 0; j < n_local; ++j) {
#pragma unroll 1
    for (int part = 0; part < (HAS_FP ? 2 : 1); ++part) {
      const int end = HAS_FP && part == 0 ? int_half : int_kb;
      for (int kb = part == 0 ? 0 : int_half; kb < end; ++kb)
        if (!fn(j, std::false_type(), kb)) return;
      if (HAS_FP && part == 0)
        for (int kb = 0; kb < fp_kb; ++kb)
          if (!fn(j, std::true_type(), kb)) return;
    }
  }
}
// What the first k-block of a product has to wait for: barrier and parity, or nullptr.  acc_empty[j & 1] completes when
// finish(j) is done, fp_drained[j & 1] when drain(j) is.
template <bool HAS_FP>
__device__ __forceinline__ uint64_t *region_barrier(int j, bool fp, uint64_t *acc_empty, uint64_t *fp_drained, uint32_t &parity) {
  if (HAS_FP) {
    parity = (uint32_t)((j - 1) >> 1) & 1u;
    return j == 0 ? nullptr : (fp ? acc_empty : fp_drained) + ((j - 1) & 1);
  }
  parity = ((uint32_t)(j >> 1) & 1u) ^ 1u;
  return acc_empty + (j & 1);
}

// One epilogue warp.  Warp (sub, group) owns rows [32*sub, 32*sub+32) of the CTA's 128 rows of the tile and the
// columns [cb, cb + cn), COLS at most, of it (group g: the g-th split_n columns).  It walks them 16 at a time.
template <typename T, bool HAS_FP, int CTAS, int COLS>
struct EpilogueWarp {
  static constexpr int CHUNKS = COLS / 16;
  const GemmParams &p;
  uint32_t tmem_base;
  int region_stride;                 // tensor-memory columns between the two accumulator regions
  int unit, num_units, rank;         // this CTA's unit (CTA or pair), number of units, rank inside the pair
  int lane, sub;
  int cb, cn, cn32;
  float *s_scol, *s_wred, *s_bias;   // [COLS] each, private to this warp
  unsigned char *s_stage;            // 32 x 32 bytes, private to this warp
  uint64_t *acc_full, *acc_empty, *fp_full, *fp_drained;
  volatile int *abort_flag;
  bool ok = true;
  long long e_wait_fp = 0, e_wait_acc = 0, e_drain = 0, e_finish = 0;

  __device__ __forceinline__ EpilogueWarp(const GemmParams &p_, uint32_t tmem_base_, int region_stride_, int unit_,
                                          int num_units_, int rank_, int e, int sub_, int lane_, float *s_vec,
                                          unsigned char *s_out, uint64_t *acc_full_, uint64_t *acc_empty_,
                                          uint64_t *fp_full_, uint64_t *fp_drained_, volatile int *abort_flag_)
      : p(p_), tmem_base(tmem_base_), region_stride(region_stride_), unit(unit_), num_units(num_units_), rank(rank_),
        lane(lane_), sub(sub_), acc_full(acc_full_), acc_empty(acc_empty_), fp_full(fp_full_), fp_drained(fp_drained_),
        abort_flag(abort_flag_) {
    cb = min((e >> 2) * p.split_n, p.block_n);
    cn = min(p.split_n, p.block_n - cb);
    cn32 = (cn + 31) & ~31;
    s_scol = s_vec + e * 3 * COLS;
    s_wred = s_scol + COLS;
    s_bias = s_wred + COLS;
    s_stage = s_out + e * EPI_BUF_BYTES;
  }

  // this warp's part of tile j: first row, first column, valid columns from there on (<= 0: none)
  struct Part {
    int m0, n0, lim;
  };
  __device__ __forceinline__ Part part(int j) const {
    const int tile = unit + j * num_units;
    Part t;
    t.m0 = (tile % p.num_m_tiles) * (BLOCK_M * CTAS) + rank * BLOCK_M + sub * 32;
    t.n0 = (tile / p.num_m_tiles) * p.block_n + cb;
    t.lim = min(p.N - t.n0, cn);
    return t;
  }
  __device__ __forceinline__ uint32_t accumulators(int region) const {
    return tmem_base + ((uint32_t)(sub * 32) << 16) + region * region_stride + cb;
  }
  __device__ __forceinline__ bool wait(uint64_t *bars, int j, long long &waited) {
    const long long t0 = clock64();
    ok = mbar_wait_warp(smem_u32(bars + (j & 1)), (uint32_t)(j >> 1) & 1u, abort_flag, p.status);
    waited += clock64() - t0;
    tc_fence_after();
    return ok;
  }
  __device__ __forceinline__ void arrive(uint64_t *bars, int j) const {
    tc_fence_before();
    if (CTAS == 1) mbar_arrive(smem_u32(bars + (j & 1)));
    else mbar_arrive_leader(smem_u32(bars + (j & 1)));
  }

  // round and keep the outlier product of tile j
  __device__ __forceinline__ void drain(int j, uint32_t (&keep)[COLS / 2]) {
    const Part t = part(j);
    __syncwarp();
    for (int c = lane; c < cn32; c += 32)
      s_bias[c] = (c < t.lim && p.bias) ? ldf<T>(p.bias, t.n0 + c) : 0.f;
    __syncwarp();
    if (!wait(fp_full, j, e_wait_fp)) return;
    const long long t0 = clock64();
    const uint32_t taddr = accumulators((j + 1) & 1);
    uint32_t v[2][16];                       // the next 16 columns are on their way while these are worked on
    if (t.lim > 0) tmem_ld16(taddr, v[0]);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (16 * c >= t.lim) break;            // warp-uniform
      uint32_t (&f)[16] = v[c & 1];
      tmem_ld_wait(f);
      if (c + 1 < CHUNKS && 16 * (c + 1) < t.lim) tmem_ld16(taddr + 16 * (c + 1), v[(c + 1) & 1]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        keep[8 * c + i] = Traits<T>::pack2(__uint_as_float(f[2 * i]) + s_bias[16 * c + 2 * i],
                                           __uint_as_float(f[2 * i + 1]) + s_bias[16 * c + 2 * i + 1]);
    }
    arrive(fp_drained, j);
    e_drain += clock64() - t0;
  }

  // Two 16-byte pieces per lane (32 bytes of its row, ELEM-byte elements) -> memory at dst (row m0 of the warp), `bytes` of
  // them valid.  Transposed through shared memory so that one warp instruction stores 16 rows x 32 contiguous bytes (whole
  // sectors) instead of 32 rows x 16 bytes; rows without 16-byte alignment are stored element by element, still 32 contiguous
  // bytes of a row at a time (one row per lane was a sector per element: 741 tokens through int4 5152 x 3333 took 85.6 us,
  // now 22.6).
  template <int ELEM>
  __device__ __forceinline__ void store_row_pieces(uint4 p0, uint4 p1, unsigned char *dst, size_t pitch, int rows, int bytes) const {
    __syncwarp();                            // the buffer has been read out
    const int flip = (lane >> 2) & 1;        // swizzle: the eight lanes of a store phase touch every bank once
    *reinterpret_cast<uint4 *>(s_stage + lane * 32 + 16 * flip) = p0;
    *reinterpret_cast<uint4 *>(s_stage + lane * 32 + 16 * (flip ^ 1)) = p1;
    __syncwarp();
    if (p.vec_out) {
      const int pc = lane & 1;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int rr = 16 * k + (lane >> 1);
        const uint4 piece = *reinterpret_cast<const uint4 *>(s_stage + rr * 32 + 16 * (pc ^ ((rr >> 2) & 1)));
        if (16 * pc + 16 <= bytes && rr < rows) *reinterpret_cast<uint4 *>(dst + (size_t)rr * pitch + 16 * pc) = piece;
      }
    } else {
      constexpr int PER_ROW = 32 / ELEM, ROWS = 32 / PER_ROW;
      const int off = (lane % PER_ROW) * ELEM;
#pragma unroll 4
      for (int k = 0; k < 32 / ROWS; ++k) {
        const int rr = ROWS * k + lane / PER_ROW;
        const unsigned char *src = s_stage + rr * 32 + 16 * ((off >> 4) ^ ((rr >> 2) & 1)) + (off & 15);
        if (off < bytes && rr < rows) {
          if (ELEM == 2) *reinterpret_cast<uint16_t *>(dst + (size_t)rr * pitch + off) = *reinterpret_cast<const uint16_t *>(src);
          else *reinterpret_cast<uint32_t *>(dst + (size_t)rr * pitch + off) = *reinterpret_cast<const uint32_t *>(src);
        }
      }
    }
  }

  // the addend y of this lane's row, chunk c; all lanes take part
  __device__ __forceinline__ void load_y(const Part &t, int c, uint32_t *w) const {
    const T *src = static_cast<const T *>(p.y) + (size_t)t.m0 * p.N + t.n0 + 16 * c;
    const int rows = p.M - t.m0, valid = t.lim - 16 * c;
    if (p.vec_y && valid >= 16) {
      const uint4 *mine = reinterpret_cast<const uint4 *>(src + (size_t)max(0, min(lane, rows - 1)) * p.N);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (lane < rows) v = mine[jj];
        w[4 * jj] = v.x; w[4 * jj + 1] = v.y; w[4 * jj + 2] = v.z; w[4 * jj + 3] = v.w;
      }
    } else {
      // half a warp fetches the 16 columns of a row (32 contiguous bytes); the staging buffer turns them
      __syncwarp();
      const int cc = lane & 15;
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const int rr = 2 * k + (lane >> 4);
        T x = Traits<T>::from_float(0.f);
        if (cc < valid && rr < rows) x = src[(size_t)rr * p.N + cc];
        *reinterpret_cast<T *>(s_stage + rr * 32 + 16 * ((cc >> 3) ^ ((rr >> 2) & 1)) + 2 * (cc & 7)) = x;
      }
      __syncwarp();
      const int flip = (lane >> 2) & 1;
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const uint4 v = *reinterpret_cast<const uint4 *>(s_stage + lane * 32 + 16 * (flip ^ jj));
        w[4 * jj] = v.x; w[4 * jj + 1] = v.y; w[4 * jj + 2] = v.z; w[4 * jj + 3] = v.w;
      }
    }
  }

  // `keep`: the kept outlier product, or room for the addend y of a tile without one
  __device__ __forceinline__ void finish(int j, uint32_t (&keep)[COLS / 2]) {
    const Part t = part(j);
    const int row = t.m0 + lane;
    float srow = 0.f, zs = 0.f;
    // everything that comes from memory is fetched before waiting for the integer product
    if (p.mode == 1) {
      __syncwarp();                         // previous readers of the vectors are done
      for (int c = lane; c < cn32; c += 32) {
        const int col = t.n0 + c;
        const bool in = c < t.lim;
        s_scol[c] = in ? ldf<T>(p.scale_col, col) : 0.f;
        s_wred[c] = (in && p.w_reduced) ? ldf<T>(p.w_reduced, col) : 0.f;
        if (!HAS_FP) s_bias[c] = (in && p.bias) ? ldf<T>(p.bias, col) : 0.f;   // with outliers the drain added it
      }
      if (row < p.M) {
        srow = ldf<T>(p.row_scale, (size_t)row * p.row_stride);
        const float zrow = p.row_zero ? ldf<T>(p.row_zero, (size_t)row * p.row_stride) : 0.f;
        zs = fmaf(p.shift_value, srow, zrow);
      }
      __syncwarp();
      if (!HAS_FP && p.y != nullptr) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c)
          if (16 * c < t.lim) load_y(t, c, keep + 8 * c);
      }
    }
    if (!wait(acc_full, j, e_wait_acc)) return;
    const long long t1 = clock64();
    const int shift = p.acc_shift;
    const uint32_t taddr = accumulators(j & 1);
    const int rows = p.M - t.m0;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (16 * c >= t.lim) break;            // warp-uniform
      uint32_t v[16];
      __syncwarp();                          // tcgen05.ld is warp-collective: reconverge first
      tmem_ld16(taddr + 16 * c, v);
      tmem_ld_wait(v);
      const int valid = t.lim - 16 * c, col0 = t.n0 + 16 * c;
      if (p.mode == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = (uint32_t)((int)v[i] >> shift);
        int32_t *dst = p.C + (size_t)t.m0 * p.N + col0;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          store_row_pieces<4>(make_uint4(v[8 * h], v[8 * h + 1], v[8 * h + 2], v[8 * h + 3]),
                              make_uint4(v[8 * h + 4], v[8 * h + 5], v[8 * h + 6], v[8 * h + 7]),
                              reinterpret_cast<unsigned char *>(dst + 8 * h), (size_t)p.N * 4, rows, 4 * (valid - 8 * h));
        continue;
      }
      float o[16];
#pragma unroll
      for (int i4 = 0; i4 < 4; ++i4) {
        const float4 sc4 = reinterpret_cast<const float4 *>(s_scol + 16 * c)[i4];
        const float4 wr4 = reinterpret_cast<const float4 *>(s_wred + 16 * c)[i4];
        const float sc[4] = {sc4.x, sc4.y, sc4.z, sc4.w};
        const float wr[4] = {wr4.x, wr4.y, wr4.z, wr4.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = 4 * i4 + q;
          float a;
          if (HAS_FP) {
            a = Traits<T>::unpack(keep[8 * c + i / 2], i & 1);
          } else {
            a = s_bias[16 * c + i];
            if (p.y != nullptr) a += Traits<T>::unpack(keep[8 * c + i / 2], i & 1);
          }
          // out = acc * (s_row * s_col) + ((zero + shift * s_row) * w_red + addend), fused multiply-adds
          o[i] = fmaf((float)((int)v[i] >> shift), srow * sc[q], fmaf(zs, wr[q], a));
        }
      }
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = Traits<T>::pack2(o[2 * i], o[2 * i + 1]);
      T *dst = static_cast<T *>(p.out) + (size_t)t.m0 * p.ldo + col0;
      store_row_pieces<2>(make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]),
                          reinterpret_cast<unsigned char *>(dst), (size_t)p.ldo * 2, rows, 2 * valid);
    }
    arrive(acc_empty, j);
    e_finish += clock64() - t1;
  }

  // all tiles of this CTA
  __device__ __forceinline__ void run(int n_local) {
    uint32_t keep[COLS / 2];
    for (int j = 0; j < n_local && ok; ++j) {
      if (HAS_FP) drain(j, keep);
      if (ok) finish(j, keep);
    }
  }

  __device__ __forceinline__ void write_counters(int cta) const {
    unsigned long long *d = p.dbg + (size_t)cta * 16;
    d[4] = (unsigned long long)e_wait_fp;     // epilogue warp: waiting for an outlier product
    d[5] = (unsigned long long)e_wait_acc;    // ... waiting for an integer product
    d[6] = (unsigned long long)e_drain;       // ... rounding and keeping outlier products
    d[7] = (unsigned long long)e_finish;      // ... final epilogues
  }
};

// ---- host helpers shared by the launchers -----------------------------------------------------
struct TileGeometry {
  int ctas, block_n;
};
// fills the shape-independent fields of GemmParams from the epilogue description
inline void fill_epilogue_params(GemmParams &p, const Epilogue &ep, int M, int N) {
  p.M = M;
  p.N = N;
  p.mode = ep.mode;
  p.C = ep.C;
  p.out = ep.out;
  p.ldo = ep.ldo > 0 ? ep.ldo : N;
  if (ep.meta) {
    const size_t eb = 2;
    p.row_scale = ep.meta;
    p.row_zero = static_cast<const unsigned char *>(ep.meta) + eb;
    p.row_stride = 2;
  } else {
    p.row_scale = ep.scale_row;
    p.row_zero = ep.zero_row;
    p.row_stride = 1;
  }
  p.scale_col = ep.scale_col;
  p.w_reduced = ep.w_reduced;
  p.bias = ep.bias;
  p.y = ep.y;
  p.shift_value = ep.shift_value;
  if (ep.mode == 0) p.vec_out = (N % 4 == 0) && aligned16(ep.C);
  else p.vec_out = (N % 8 == 0) && (p.ldo % 8 == 0) && aligned16(ep.out);
  p.vec_y = ep.y && (N % 8 == 0) && aligned16(ep.y);
  p.dbg = get_debug_counters();
  p.status = device_status_word();
}
// columns of a tile per group of four epilogue warps
inline int split_columns(int block_n, int groups) { return (block_n / groups + 31) & ~31; }

}  // namespace
}  // namespace quik
