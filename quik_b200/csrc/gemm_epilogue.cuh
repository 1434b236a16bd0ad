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
constexpr int EPI_RING_PITCH = 80;           // output staging of one epilogue warp: 64 bytes of each of 32 rows, padded
constexpr int EPI_BUF_BYTES = 32 * EPI_RING_PITCH;
constexpr int SMEM_LIMIT = 227 * 1024;

struct GemmParams {
  int M, N;
  int block_n;                    // tile width: multiple of 16
  int split_n;                    // columns of a tile that each group of four epilogue warps takes (multiple of 32)
  int num_m_tiles, num_tiles;
  int int_kb, fp_kb;              // k-blocks per tile: integer (128 codes each) and outlier (64 elems)
  uint32_t idesc_int, idesc_fp;   // tcgen05 instruction descriptors
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
// KIND: 0 the int32 product as it is, 1 dequantize, 2 dequantize with an outlier product, 3 dequantize with an addend y.  SHIFT: the integer accumulator holds the
// product times 2^SHIFT (operands widened on chip).
// ROWS_ARE: of what alignment the result's rows are; ALIGNED: 16 bytes, and there is a map of the result for bulk stores.  (Known when
// the kernel is compiled, as is the tile's capacity, by which unaligned rows are stored: over 1132 drawn layers 1.3 % faster than all
// forms of the stores in one kernel; 741 tokens through 5152 x 3333 28.2 us, now 27.6.)
// (The addend has a kind of its own: its loads, eight times in the code, are fetched, or jumped over, by launches that have none.  As a
// branch of kind 1 they cost layers without outliers 180 tokens x 2496 -> 12544 16.9 us, now 15.2; 402 x 3584 -> 4864 18.1, now 16.7.)
enum RowAlignment { ANY, ALIGNED, UNALIGNED };
template <typename T, int KIND, int SHIFT, int CTAS, int COLS, int ROWS_ARE>
struct EpilogueWarp {
  static constexpr bool HAS_FP = KIND == 2, HAS_Y = KIND == 3;
  static constexpr int CHUNKS = COLS / 16;
  static constexpr int LANE_COLS = COLS / 32;         // columns whose vectors a lane fetches
  const GemmParams &p;
  const CUtensorMap *out_map;        // the result for bulk stores, or nullptr
  uint32_t tmem_base;
  int region_stride;                 // tensor-memory columns between the two accumulator regions
  int unit, num_units, rank;         // this CTA's unit (CTA or pair), number of units, rank inside the pair
  int lane, sub;
  int cb, cn;
  float *s_scol, *s_wred, *s_bias;   // [COLS] each, private to this warp
  unsigned char *s_stage;            // EPI_BUF_BYTES, private to this warp: 32 rows x 32 bytes, a box of 32 x 64, or 32 rings of 64
  uint64_t *acc_full, *acc_empty, *fp_full, *fp_drained;
  volatile int *abort_flag;
  float srow = 0.f, zs = 0.f;        // of this lane's row: scale, zero + shift * scale
  bool ok = true;
  unsigned e_wait_fp = 0, e_wait_acc = 0, e_drain = 0, e_finish = 0;      // cycles

  __device__ __forceinline__ EpilogueWarp(const GemmParams &p_, const CUtensorMap *out_map_, uint32_t tmem_base_, int region_stride_, int unit_,
                                          int num_units_, int rank_, int e, int sub_, int lane_, float *s_vec,
                                          unsigned char *s_out, uint64_t *acc_full_, uint64_t *acc_empty_,
                                          uint64_t *fp_full_, uint64_t *fp_drained_, volatile int *abort_flag_)
      : p(p_), out_map(out_map_), tmem_base(tmem_base_), region_stride(region_stride_), unit(unit_), num_units(num_units_), rank(rank_),
        lane(lane_), sub(sub_), acc_full(acc_full_), acc_empty(acc_empty_), fp_full(fp_full_), fp_drained(fp_drained_),
        abort_flag(abort_flag_) {
    cb = min((e >> 2) * p.split_n, p.block_n);
    cn = min(p.split_n, p.block_n - cb);
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
  __device__ __forceinline__ bool wait(uint64_t *bars, int j, unsigned &waited) {
    const unsigned t0 = (unsigned)clock();
    ok = mbar_wait_warp(smem_u32(bars + (j & 1)), (uint32_t)(j >> 1) & 1u, abort_flag, p.status);
    waited += (unsigned)clock() - t0;
    tc_fence_after();
    return ok;
  }
  __device__ __forceinline__ void arrive(uint64_t *bars, int j) const {
    tc_fence_before();
    __syncwarp();
    if (lane != 0) return;
    if (CTAS == 1) mbar_arrive(smem_u32(bars + (j & 1)));
    else mbar_arrive_leader(smem_u32(bars + (j & 1)));
  }

  // The column vectors and this lane's row factors of a tile on their way from memory.
  struct Fetched {
    uint16_t scol[LANE_COLS], wred[LANE_COLS], bias[LANE_COLS];
    uint16_t srow, zrow;
  };
  __device__ __forceinline__ void fetch(int j, Fetched &x) const {
    if (KIND == 0) return;
    const Part t = part(j);
    auto ld = [](const void *v, size_t i) { return static_cast<const uint16_t *>(v)[i]; };
#pragma unroll
    for (int i = 0; i < LANE_COLS; ++i) {
      const int c = lane + 32 * i;
      const bool in = c < t.lim;
      x.scol[i] = in ? ld(p.scale_col, t.n0 + c) : (uint16_t)0;
      x.wred[i] = in && p.w_reduced ? ld(p.w_reduced, t.n0 + c) : (uint16_t)0;
      x.bias[i] = in && p.bias ? ld(p.bias, t.n0 + c) : (uint16_t)0;
    }
    const int row = t.m0 + lane;
    x.srow = row < p.M ? ld(p.row_scale, (size_t)row * p.row_stride) : (uint16_t)0;
    x.zrow = row < p.M && p.row_zero ? ld(p.row_zero, (size_t)row * p.row_stride) : (uint16_t)0;
  }
  __device__ __forceinline__ static float value(uint16_t raw) { return Traits<T>::unpack(raw, 0); }
  // ... into place, all columns of the warp's part (zero beyond the matrix)
  __device__ __forceinline__ void place(const Fetched &x) {
    if (KIND == 0) return;
    __syncwarp();                            // previous readers of the vectors are done
#pragma unroll
    for (int i = 0; i < LANE_COLS; ++i) {
      const int c = lane + 32 * i;
      s_scol[c] = value(x.scol[i]);
      s_wred[c] = value(x.wred[i]);
      s_bias[c] = value(x.bias[i]);
    }
    srow = value(x.srow);
    zs = fmaf(p.shift_value, srow, value(x.zrow));
    __syncwarp();
  }

  // The kept words move on by two chunks, so that loops over the chunks need not be unrolled to name them.  Code is fetched from
  // L2, or from memory where weights have streamed through L2 since the last launch, and most launches have one or two tiles per
  // CTA: unrolled eight times, the epilogue's code took longer to arrive than to run (the four layers of Llama-2-7B at 333 tokens: 147.5
  // us, in loops 134.2).
  __device__ __forceinline__ static void rotate(uint32_t (&keep)[COLS / 2]) {
#pragma unroll
    for (int i = 0; i < COLS / 2 - 16; ++i) keep[i] = keep[i + 16];
  }

  // round and keep the outlier product of tile j
  __device__ __forceinline__ void drain(int j, uint32_t (&keep)[COLS / 2]) {
    const Part t = part(j);
    if (!wait(fp_full, j, e_wait_fp)) return;
    const unsigned t0 = (unsigned)clock();
    const uint32_t taddr = accumulators((j + 1) & 1);
    uint32_t v[2][16];                       // the next 16 columns are on their way while these are worked on
    if (t.lim > 0) tmem_ld16(taddr, v[0]);
#pragma unroll 1
    for (int c0 = 0; c0 < CHUNKS; c0 += 2) {
      rotate(keep);                          // the new words go to the end; after all rounds the first ones are at the start
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + h;
        if (16 * c >= t.lim) break;          // warp-uniform
        uint32_t (&f)[16] = v[h];
        tmem_ld_wait(f);
        if (16 * (c + 1) < t.lim) tmem_ld16(taddr + 16 * (c + 1), v[h ^ 1]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          keep[COLS / 2 - 16 + 8 * h + i] = Traits<T>::pack2(__uint_as_float(f[2 * i]) + s_bias[16 * c + 2 * i],
                                                             __uint_as_float(f[2 * i + 1]) + s_bias[16 * c + 2 * i + 1]);
      }
    }
    arrive(fp_drained, j);
    e_drain += (unsigned)clock() - t0;
  }

  // Where a part's rows go: first byte of row 0, row pitch, rows and bytes per row that exist.
  struct Rows {
    unsigned char *dst;
    size_t pitch;
    int rows, bytes;
    __device__ __forceinline__ unsigned char *row(int r) const { return dst + (size_t)r * pitch; }
  };

  // Piece c of a part: 32 bytes of this lane's row (two 16-byte halves) to memory, rows with 16-byte alignment.  Transposed
  // through shared memory so that one warp instruction stores 16 rows x 32 contiguous bytes (whole sectors) instead of 32 rows x
  // 16 bytes.
  __device__ __forceinline__ void store_aligned(const Rows &o, int c, uint4 p0, uint4 p1) const {
    reuse_stage();                           // the buffer has been read out
    const int flip = (lane >> 2) & 1;        // swizzle: the eight lanes of a store phase touch every bank once
    *reinterpret_cast<uint4 *>(s_stage + lane * 32 + 16 * flip) = p0;
    *reinterpret_cast<uint4 *>(s_stage + lane * 32 + 16 * (flip ^ 1)) = p1;
    __syncwarp();
    const int pc = lane & 1;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int rr = 16 * k + (lane >> 1);
      const uint4 piece = *reinterpret_cast<const uint4 *>(s_stage + rr * 32 + 16 * (pc ^ ((rr >> 2) & 1)));
      if (32 * c + 16 * pc + 16 <= o.bytes && rr < o.rows) *reinterpret_cast<uint4 *>(o.row(rr) + 32 * c + 16 * pc) = piece;
    }
  }

  // The same by bulk stores, two pieces at a time: 64 bytes of each of the warp's rows, in the layout of the 64-byte swizzle; one
  // lane issues the store of the box and nobody waits for it until the buffer is needed again.  (With store instructions, 16 rows x 32
  // bytes each, the products waited for the epilogue: 7B qkv at 2048 tokens, back to back, 80.5 -> 77.4 us; 541 instead of 591 cycles
  // per k-block with no stores at all.)
  __device__ __forceinline__ void store_bulk(const Part &t, const Rows &o, int c, int odd, uint4 p0, uint4 p1) const {
    if (!odd) reuse_stage();
    const int turn = (lane >> 1) & 3, u = 2 * odd;
    *reinterpret_cast<uint4 *>(s_stage + lane * 64 + 16 * (u ^ turn)) = p0;
    *reinterpret_cast<uint4 *>(s_stage + lane * 64 + 16 * ((u + 1) ^ turn)) = p1;
    if (odd) {
      fence_async_shared();
      __syncwarp();
      if (lane == 0 && o.rows > 0) tma_store_2d(out_map, smem_u32(s_stage), t.n0 + (KIND == 0 ? 8 : 16) * (c - 1), t.m0);
    }
  }
  // Comes before whatever writes the staging buffer anew: it has been read out, by the warp's lanes and by its bulk stores.
  __device__ __forceinline__ void reuse_stage() const {
    if (lane == 0) tma_store_wait_read();
    __syncwarp();
  }

  // The same for rows without 16-byte alignment (an odd N): every row starts somewhere inside a 32-byte sector.  Its bytes pass
  // through a ring of two sectors per row in shared memory at the place that they have in memory, modulo 64; when piece c is in,
  // sector c of the row is complete and leaves as two 16-byte stores, and only the first and the last sector of the part are
  // written in pieces.  (Element by element, 32 bytes of a row at a time, 3111 tokens through 1024 x 25036 took 194 us, now 133.)
  struct Sectors {
    int word;                // of the lane's own row: word of its sector that the part starts in,
    uint32_t turn;           // bits that the pieces are shifted by to words of memory,
    uint32_t carry;          // last word of the piece before
    unsigned char *to[2];    // of the two rows that the lane stores 16 bytes of: its place in sector 0,
    int off[2];              // and where that is in the row
  };
  template <int ELEM>
  __device__ __forceinline__ void start_sectors(const Rows &o, Sectors &x) const {
    const uint32_t at = (uint32_t)reinterpret_cast<uintptr_t>(o.row(lane)) & 31u;        // of the row's first byte, in its sector
    x.word = at >> 2;
    x.turn = ELEM == 2 ? 8 * (at & 2) : 0;
    x.carry = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      unsigned char *row = o.row(16 * k + (lane >> 1));
      x.off[k] = 16 * (lane & 1) - (int)(reinterpret_cast<uintptr_t>(row) & 31u);
      x.to[k] = row + x.off[k];
    }
  }
  template <int ELEM>
  __device__ __forceinline__ void store_sector(const Rows &o, Sectors &x, int c, int odd, bool last, uint4 p0, uint4 p1) const {
    const uint32_t w[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
    uint32_t *mine = reinterpret_cast<uint32_t *>(s_stage + lane * EPI_RING_PITCH) + x.word + 8 * odd;
    __syncwarp();                            // the sector that this piece runs into has been read out
#pragma unroll
    for (int k = 0; k < 8; ++k)
      mine[odd && k + x.word >= 8 ? k - 16 : k] = __funnelshift_l(k == 0 ? x.carry : w[k - 1], w[k], x.turn);
    x.carry = w[7];
    if (last && x.turn) mine[odd ? -8 : 8] = w[7] >> 16;
    __syncwarp();
    if (c > 0 && !last) {                    // inside every row of the part
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int rr = 16 * k + (lane >> 1);
        const uint4 v = *reinterpret_cast<const uint4 *>(s_stage + rr * EPI_RING_PITCH + 32 * odd + 16 * (lane & 1));
        if (rr < o.rows) *reinterpret_cast<uint4 *>(x.to[k] + 32 * c) = v;
      }
    } else {
#pragma unroll 1
      for (int e = c; e <= c + last; ++e) edge_sector<ELEM>(o, x, e);
    }
  }
  template <int ELEM>
  __device__ __forceinline__ void edge_sector(const Rows &o, const Sectors &x, int c) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int rr = 16 * k + (lane >> 1), off = x.off[k] + 32 * c;      // of the 16 bytes in the row
      const uint4 v = *reinterpret_cast<const uint4 *>(s_stage + rr * EPI_RING_PITCH + 32 * (c & 1) + 16 * (lane & 1));
      unsigned char *to = x.to[k] + 32 * c;
      const int first = -off, end = rr < o.rows ? o.bytes - off : 0;     // of the 16 bytes, those of the row
      if (first <= 0 && end >= 16) {
        *reinterpret_cast<uint4 *>(to) = v;
      } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int b = 0; b < 16; b += ELEM) {
          if (b < first || b >= end) continue;
          if (ELEM == 2) *reinterpret_cast<uint16_t *>(to + b) = (uint16_t)(w[b / 4] >> (8 * (b & 2)));
          else *reinterpret_cast<uint32_t *>(to + b) = w[b / 4];
        }
      }
    }
  }

  // The same element by element, still 32 contiguous bytes of a row at a time: for parts of up to 64 columns (COLS: tiles of up to
  // 128), of whose few sectors most are first or last ones.  (By sectors, and element by element: 136 tokens through 2368 x 4287, 64
  // columns to a tile, 16.7 us, now 14.9; 430 through 1280 x 2109 13.6, now 11.9.  In tiles of 160 the two are equal, beyond that whole
  // sectors gain.)
  template <int ELEM>
  __device__ __forceinline__ void store_elements(const Rows &o, int c, uint4 p0, uint4 p1) const {
    __syncwarp();                            // the buffer has been read out
    const int flip = (lane >> 2) & 1;
    *reinterpret_cast<uint4 *>(s_stage + lane * 32 + 16 * flip) = p0;
    *reinterpret_cast<uint4 *>(s_stage + lane * 32 + 16 * (flip ^ 1)) = p1;
    __syncwarp();
    constexpr int PER_ROW = 32 / ELEM, ROWS = 32 / PER_ROW;
    const int off = (lane % PER_ROW) * ELEM;
#pragma unroll 4
    for (int k = 0; k < 32 / ROWS; ++k) {
      const int rr = ROWS * k + lane / PER_ROW;
      const unsigned char *from = s_stage + rr * 32 + 16 * ((off >> 4) ^ ((rr >> 2) & 1)) + (off & 15);
      if (32 * c + off >= o.bytes || rr >= o.rows) continue;
      if (ELEM == 2) *reinterpret_cast<uint16_t *>(o.row(rr) + 32 * c + off) = *reinterpret_cast<const uint16_t *>(from);
      else *reinterpret_cast<uint32_t *>(o.row(rr) + 32 * c + off) = *reinterpret_cast<const uint32_t *>(from);
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
      // half a warp fetches the 16 columns of a row (32 contiguous bytes); the staging buffer turns them.  A bulk store of the
      // tile before may still be reading it.
      reuse_stage();
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
  // STORES: SECTORS and ELEMENTS for any rows, ROWS for rows of 16-byte alignment, BULK for those where there is a map of the result
  enum Stores { SECTORS, ELEMENTS, ROWS, BULK };
  template <int STORES>
  __device__ __forceinline__ void finish(int j, uint32_t (&keep)[COLS / 2], const Rows &o) {
    const Part t = part(j);
    const uint32_t taddr = accumulators(j & 1);
    Sectors x;
    if (STORES == SECTORS) start_sectors<KIND == 0 ? 4 : 2>(o, x);
    uint32_t acc[2][16];                     // the next 16 columns are on their way while these are worked on
    __syncwarp();                            // tcgen05.ld is warp-collective: reconverge first
    if (t.lim > 0) tmem_ld16(taddr, acc[0]);
#pragma unroll 1
    for (int c0 = 0; 16 * c0 < t.lim; c0 += 2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + h;
        if (16 * c >= t.lim) break;            // warp-uniform
        uint32_t (&v)[16] = acc[h];
        __syncwarp();
        tmem_ld_wait(v);
        if (16 * (c + 1) < t.lim) tmem_ld16(taddr + 16 * (c + 1), acc[h ^ 1]);
        auto piece = [&](int n, int odd, uint4 p0, uint4 p1) {      // odd: n & 1, known when this is compiled
          if (STORES == ROWS || (STORES == BULK && KIND != 0 && !odd && 32 * (n + 1) >= o.bytes)) store_aligned(o, n, p0, p1);
          else if (STORES == BULK) store_bulk(t, o, n, odd, p0, p1);
          else if (STORES == ELEMENTS) store_elements<KIND == 0 ? 4 : 2>(o, n, p0, p1);
          else store_sector<KIND == 0 ? 4 : 2>(o, x, n, odd, 32 * (n + 1) >= o.bytes, p0, p1);
        };
        if (KIND == 0) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = (uint32_t)((int)v[i] >> SHIFT);
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (STORES == BULK || 8 * (2 * c + e) < t.lim)      // (a box is stored when both its halves are in)
              piece(2 * c + e, e, make_uint4(v[8 * e], v[8 * e + 1], v[8 * e + 2], v[8 * e + 3]),
                    make_uint4(v[8 * e + 4], v[8 * e + 5], v[8 * e + 6], v[8 * e + 7]));
          continue;
        }
        uint32_t w[8];
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) {
          const float4 sc4 = reinterpret_cast<const float4 *>(s_scol + 16 * c)[i4];
          const float4 wr4 = reinterpret_cast<const float4 *>(s_wred + 16 * c)[i4];
          const float sc[4] = {sc4.x, sc4.y, sc4.z, sc4.w};
          const float wr[4] = {wr4.x, wr4.y, wr4.z, wr4.w};
          float f[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = 4 * i4 + q;
            float a;
            if (HAS_FP) {
              a = Traits<T>::unpack(keep[8 * h + i / 2], i & 1);
            } else {
              a = s_bias[16 * c + i];
              if (HAS_Y) a += Traits<T>::unpack(keep[8 * h + i / 2], i & 1);
            }
            // out = acc * (s_row * s_col) + ((zero + shift * s_row) * w_red + addend), fused multiply-adds
            f[q] = fmaf((float)((int)v[i] >> SHIFT), srow * sc[q], fmaf(zs, wr[q], a));
          }
          w[2 * i4] = Traits<T>::pack2(f[0], f[1]);
          w[2 * i4 + 1] = Traits<T>::pack2(f[2], f[3]);
        }
        piece(c, h, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
      }
      if (HAS_FP || HAS_Y) rotate(keep);
    }
  }

  // all tiles of this CTA
  __device__ __forceinline__ void run(int n_local) {
    if (ROWS_ARE == ALIGNED) {
      run_tiles<BULK>(n_local);
      if (lane == 0) tma_store_wait_all();
    } else if (ROWS_ARE == ANY && p.vec_out) {
      run_tiles<ROWS>(n_local);
    } else {
      run_tiles<COLS <= 64 ? ELEMENTS : SECTORS>(n_local);
    }
  }
  template <int STORES>
  __device__ __forceinline__ void run_tiles(int n_local) {
    uint32_t keep[COLS / 2];
    Fetched next;
    if (n_local > 0) fetch(0, next);
    for (int j = 0; j < n_local && ok; ++j) {
      place(next);
      if (HAS_FP) drain(j, keep);
      if (!ok) break;
      const Part t = part(j);
      if (HAS_Y) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c)
          if (16 * c < t.lim) load_y(t, c, keep + 8 * c);
      }
      // the next tile's vectors travel while this one is finished (fetched at its start they cost their latency with nothing to
      // hide it where the products are ready first)
      if (j + 1 < n_local) fetch(j + 1, next);
      if (!wait(acc_full, j, e_wait_acc)) break;
      const unsigned t1 = (unsigned)clock();
      Rows o;
      o.rows = p.M - t.m0;
      o.bytes = (KIND == 0 ? 4 : 2) * t.lim;
      if (KIND == 0) {
        o.dst = reinterpret_cast<unsigned char *>(p.C + (size_t)t.m0 * p.N + t.n0);
        o.pitch = (size_t)p.N * 4;
      } else {
        o.dst = reinterpret_cast<unsigned char *>(static_cast<T *>(p.out) + (size_t)t.m0 * p.ldo + t.n0);
        o.pitch = (size_t)p.ldo * 2;
      }
      finish<STORES>(j, keep, o);
      arrive(acc_empty, j);
      e_finish += (unsigned)clock() - t1;
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
// fills the shape-independent fields of GemmParams from the epilogue description
inline void fill_epilogue_params(GemmParams &p, const Epilogue &ep, int M, int N) {
  p.M = M;
  p.N = N;
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
