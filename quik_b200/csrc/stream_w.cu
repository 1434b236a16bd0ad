// Weight-streaming fused layer for few tokens (M <= 128) on the tcgen05 tensor cores.
//
// With few tokens the layer (QUIK experiments/qlinear.py:122-145) is bound by reading the weights
// once from HBM, so the kernel is built around the weight stream and keeps the weights in their storage
// format: packed int4 (two codes per byte, low nibble first, QUIK include/int4.h:78-98) or int8.
//
// The product is computed transposed, out^T[n, m] = sum_k W[n, k] * Xq[m, k]: 128 weight rows are the
// M = 128 operand of tcgen05.mma, the tokens (zero-padded to the next multiple of 16) its N operand, so one
// instruction consumes 128 x 32 weight codes.  Per CTA (one 128-row slab of W, one share of K):
//   warp 0      TMA producer: k-blocks of W (128 rows x 128 bytes, 128B swizzle) and of the token codes /
//               outlier values (ntok rows x 128 bytes) into a ring of shared-memory stages.
//   warps 2-9   int4 only: each thread takes 64 packed bytes of "its" weight row from shared memory, widens
//               the 128 nibbles to signed bytes that carry 16 x the code (shift, two masks and two byte
//               permutes per 8 codes, natural k order) and writes them with tcgen05.st into a ring of TMEM
//               slots: the widened weights never touch shared or global memory.
//   warp 1      walks the blocks as a whole warp, one elected lane issues tcgen05.mma (kind::i8 with A read from TMEM
//               (int4) or from the shared-memory stage (int8), B always from shared memory; kind::f16 for the outlier
//               columns) into an s32 and an f32 accumulator of ntok columns each in TMEM.
//   warps 2-9   epilogue: tcgen05.ld of the accumulators, split-K reduction, dequantize arithmetic of
//               QUIK src/asymmetric/asymmetric.cu:134-146, stores of out[m, n] (64 contiguous bytes per warp
//               and token).
// K is split over the CTAs of a thread-block cluster (1, 2, 4 or 8) when the layer has too few 128-row slabs
// to fill the GPU: every CTA leaves its exact int32 partial sums in its own shared memory (in the drained ring), and
// after a cluster barrier CTA r adds up the sums of all of them for its share of the tokens and finishes those.  (Adding
// into the leader's shared memory with red.shared::cluster cost 8 us more for 32 tokens split eight ways than for 16: 21.1 against 12.5 us for int8 11008 x 4096.)  The first CTA alone handles the outlier
// product, so the floating-point arithmetic has one fixed order.
// Every mbarrier wait is bounded; a wait that runs out sets the device status word, all roles leave their
// loops, the cluster barriers are still passed by every thread, TMEM is released and the kernel returns.
#include <cuda.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "tcgen05_ptx.cuh"

namespace quik {
namespace {

constexpr int SW_THREADS = 320;                    // TMA warp, MMA warp, 8 widen/epilogue warps
constexpr int SW_ROWS = 128;                       // weight rows per CTA (the MMA's M)
constexpr int SW_W_BYTES = SW_ROWS * 128;          // one k-block of W: 128 bytes per row
constexpr int SW_A_COLS = 64;                      // 256 int8 codes per row = 64 32-bit columns
constexpr int SW_MAX_STAGES = 10;
constexpr int SW_AUX_BYTES = 2048;                 // barriers, then the token scales
constexpr int SW_SMEM_SM = 227 * 1024;

// Sizes that depend on the number of tokens (the MMA's N, a multiple of 16): shared-memory ring and tensor-memory plan.
// Up to 64 tokens two CTAs may share an SM (256 tensor-memory columns and at most 113 KB each; the rule is in launch_stream_w),
// beyond that one CTA has it.
struct StreamPlan {
  int ctas_per_sm, tmem_cols, a_slots, d_int, d_fp;
  int x_bytes, stage_bytes, stages;
  size_t smem;
};
inline StreamPlan plan_stream(int bits, int ntok, int ctas_per_sm) {
  StreamPlan c{};
  c.ctas_per_sm = ctas_per_sm;
  c.tmem_cols = c.ctas_per_sm == 2 ? 256 : 512;
  const int d_cols = ntok <= 32 ? 32 : (ntok <= 64 ? 64 : 128);
  c.d_fp = c.tmem_cols - d_cols;                                         // f32 accumulator
  c.d_int = c.d_fp - (bits == 8 ? 2 : 1) * d_cols;                       // s32 accumulator; int8: two, d_cols apart
  c.a_slots = bits == 4 ? c.d_int / SW_A_COLS : 0;                       // ring of widened W k-blocks, from column 0 on
  if (c.a_slots > 4) c.a_slots = 4;
  c.x_bytes = ntok * 128;                                                // one 128-byte k-block of the token operand
  c.stage_bytes = SW_W_BYTES + (bits == 4 ? 2 : 1) * c.x_bytes;          // int4: 256 codes of W need two token blocks
  const int room = SW_SMEM_SM / c.ctas_per_sm - 1024 - 1024 - SW_AUX_BYTES;      // (1 KB of alignment, 1 KB that the system takes)
  c.stages = room / c.stage_bytes;
  if (c.stages > SW_MAX_STAGES) c.stages = SW_MAX_STAGES;
  c.smem = 1024 + (size_t)c.stages * c.stage_bytes + SW_AUX_BYTES;      // stages >= 3: room for two tiles of 4-byte sums
  // No CTA may wait for tensor memory that a CTA of a later launch of the same stream holds (launches overlap): shared
  // memory has to keep them apart.  256 columns: at most two CTAs fit an SM; 512 columns: nothing of the kind fits beside.
  const size_t least = c.tmem_cols == 256 ? SW_SMEM_SM / 3 : SW_SMEM_SM - SW_SMEM_SM / 3;
  if (c.smem <= least) c.smem = least + 1024;
  return c;
}

struct StreamParams {
  int M, N;
  int nk, nf;                     // k-blocks of the integer part (128 bytes of a W row each) and of the outliers
  int splits;                     // CTAs that share one slab (= cluster size)
  int ntok;                       // tokens rounded up to a multiple of 16: the MMA's N
  int stages, stage_bytes, x_bytes;
  int a_slots, d_int, d_fp, tmem_cols;
  uint32_t idesc_int, idesc_fp;
  const void *meta, *scale_col, *w_reduced, *bias;
  void *out;
  long long ldo;
  float shift_value;
  unsigned int *status;
  unsigned long long *dbg;        // optional cycle counters (16 per CTA), NULL = off
};

template <typename T, int BITS>
__global__ void __launch_bounds__(SW_THREADS, 2)
stream_w_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                const __grid_constant__ CUtensorMap tm_fw, const __grid_constant__ CUtensorMap tm_fx,
                const StreamParams p) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  const int STAGES = p.stages, STAGE_BYTES = p.stage_bytes, X_BYTES = p.x_bytes;
  unsigned char *aux = tiles + STAGES * STAGE_BYTES;
  int *sum_i = reinterpret_cast<int *>(tiles);                  // [token][row] partial sums in the drained ring, where K is split
  float *sum_f = reinterpret_cast<float *>(sum_i + p.ntok * SW_ROWS);   // ... of the outlier product (first CTA)
  uint64_t *full_bar = reinterpret_cast<uint64_t *>(aux);       // [STAGES] stage loaded
  uint64_t *empty_bar = full_bar + SW_MAX_STAGES;               // [STAGES] stage consumed
  uint64_t *a_full = empty_bar + SW_MAX_STAGES;                 // [a_slots] widened block written to TMEM
  uint64_t *a_empty = a_full + 4;                               // [a_slots] ... consumed by the MMAs
  uint64_t *acc_full = a_empty + 4;                             // all MMAs of this CTA complete
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  float *s_srow = reinterpret_cast<float *>(aux + 256);         // [128] token scale
  float *s_zs = s_srow + 128;                                   // [128] zero + shift * scale

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool worker = warp >= 2;                                  // widening + epilogue warps
  const int S = p.splits;
  const int rank = S > 1 ? (int)cluster_ctarank() : 0;
  const int n0 = ((int)blockIdx.x / S) * SW_ROWS;
  // Blocks of the slab in one sequence: outlier blocks first (so that they all fall to rank 0, which the
  // host guarantees by its choice of S), then the integer blocks; rank r takes an equal contiguous share.
  const int total = p.nk + p.nf;
  const int c0 = (int)(((long long)rank * total) / S), c1 = (int)(((long long)(rank + 1) * total) / S);
  const int nb = c1 - c0;
  const int n_fp = c0 < p.nf ? (c1 < p.nf ? c1 : p.nf) - c0 : 0;   // leading outlier blocks of this CTA
  const int n_int = nb - n_fp;
  const int kb_first = c0 + n_fp - p.nf;                           // first integer k-block

  // one block of the sequence, weight tile and token tile(s), into its stage
  auto load_block = [&](int i, int stage) {
    const uint32_t fb = smem_u32(full_bar + stage), sw = smem_u32(tiles + stage * STAGE_BYTES), sx = sw + SW_W_BYTES;
    if (i < n_fp) {
      mbar_expect_tx(fb, SW_W_BYTES + X_BYTES);
      tma_load_2d<1>(sw, &tm_fw, fb, (c0 + i) * 64, n0);
      tma_load_2d<1>(sx, &tm_fx, fb, (c0 + i) * 64, 0);
      return;
    }
    const int kb = kb_first + i - n_fp;
    mbar_expect_tx(fb, STAGE_BYTES);
    tma_load_2d<1>(sw, &tm_w, fb, kb * 128, n0);
    if (BITS == 4) {                                                   // 128 packed bytes of W = 256 codes
      tma_load_2d<1>(sx, &tm_x, fb, kb * 256, 0);
      tma_load_2d<1>(sx + X_BYTES, &tm_x, fb, kb * 256 + 128, 0);
    } else {
      tma_load_2d<1>(sx, &tm_x, fb, kb * 128, 0);
    }
  };

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(full_bar + s), 1);
      mbar_init(smem_u32(empty_bar + s), 1 + (BITS == 4 ? 8 : 1));   // MMA commit, and the 8 widening warps or the other issuer
    }
    for (int s = 0; s < p.a_slots; ++s) {
      mbar_init(smem_u32(a_full + s), 8);
      mbar_init(smem_u32(a_empty + s), 1);
    }
    mbar_init(smem_u32(acc_full), BITS == 8 ? 2 : 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    prefetch_tmap(&tm_w);
    prefetch_tmap(&tm_x);
    if (p.nf > 0) {
      prefetch_tmap(&tm_fw);
      prefetch_tmap(&tm_fx);
    }
  }
  if (warp == 1) {
    tmem_alloc<1>(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish<1>();
  }
  if (warp == 0) {
    // Ask L2 for the weight tiles of the first ring fill while the producer of the token codes may still run (more tiles
    // measured slower: their requests delay the first loads).  The loads themselves come after the wait: an earlier launch of
    // the stream may have written the weights.  Loading the first ring fill into shared memory here gave nothing: four
    // layers of Llama-2-7B at 20 / 64 / 128 tokens 70.9 / 75.3 / 97.5 us, with the prefetch 71.5 / 75.8 / 97.3 us, with
    // neither 74.3 / 78.2 / 97.7 us.
    __syncwarp();
    for (int i = lane; i < (nb < STAGES ? nb : STAGES); i += 32) {
      if (i < n_fp) tma_prefetch_2d(&tm_fw, (c0 + i) * 64, n0);
      else tma_prefetch_2d(&tm_w, (kb_first + i - n_fp) * 128, n0);
    }
  }
  __syncwarp();
  pdl_wait();      // first global access below
  if (worker) {
    const int te = threadIdx.x - 64;
    if (te < p.ntok) {
      float s = 0.f, z = 0.f;
      if (te < p.M) {
        s = Traits<T>::to_float(static_cast<const T *>(p.meta)[2 * te]);
        z = Traits<T>::to_float(static_cast<const T *>(p.meta)[2 * te + 1]);
      }
      s_srow[te] = s;
      s_zs[te] = fmaf(p.shift_value, s, z);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // epilogue vectors of this thread's weight row, fetched while the weights stream
  // (kept in storage format until the end: converting here would wait for the loads, which take microseconds
  // while the weight stream saturates HBM)
  T ep_scol = Traits<T>::from_float(0.f), ep_wred = ep_scol, ep_bias = ep_scol;
  if (worker) {
    const int n = n0 + (warp & 3) * 32 + lane;
    if (n < p.N) {
      ep_scol = static_cast<const T *>(p.scale_col)[n];
      ep_wred = static_cast<const T *>(p.w_reduced)[n];
      if (p.bias) ep_bias = static_cast<const T *>(p.bias)[n];
    }
  }

  if (warp == 0) {
    // ================= TMA producer =================
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < nb; ++i) {
      if (!mbar_wait_warp(smem_u32(empty_bar + stage), phase ^ 1, abort_flag, p.status)) break;
      if (elected) load_block(i, stage);
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    __syncwarp();
  } else if (warp == 1 || (BITS == 8 && warp == 2)) {
    // ================= MMA issuer =================
    // The loop's exits are warp votes, so its counters and the descriptors made from them are uniform over the warp and
    // the elected lane issues back to back.  (A loop inside a `lane == 0` branch issued one instruction every ~62 ns.)
    // Waiting for a stage and issuing its four products still takes one warp 600 cycles, more than an int8 block takes to arrive:
    // two warps (the second has nothing else to do until the epilogue) take the int8 blocks in turn, each into an
    // accumulator of its own (75 slabs of 10752 int8 columns, 33 / 64 tokens: 34.3 / 35.4 -> 31.2 / 31.9 us).
    const int me = warp - 1;
    const bool elected = elect_one();
    const uint64_t dw0 = make_smem_desc(smem_u32(tiles));
    const uint32_t d_int = tmem_base + p.d_int + me * ((p.d_fp - p.d_int) / 2);
    int stage = 0, slot = 0;
    uint32_t phase = 0, slot_phase = 0;
    long long w_full = 0, w_a = 0;
    const bool dbg = p.dbg != nullptr;
    const long long t_begin = clock64();
    for (int i = 0; i < nb; ++i) {
      const long long t0 = dbg ? clock64() : 0;
      if (!mbar_wait_warp(smem_u32(full_bar + stage), phase, abort_flag, p.status)) break;
      if (dbg) w_full += clock64() - t0;
      if (BITS == 8 && me != (i < n_fp ? 0 : (i - n_fp) & 1)) {
        // the other warp's block.  A stage is filled again only when both have seen it: a barrier's phase is one bit, so a warp
        // may neither miss a fill nor fall behind by two.
        if (elected) mbar_arrive(smem_u32(empty_bar + stage));
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        continue;
      }
      const uint64_t dw = dw0 + (uint32_t)(stage * (STAGE_BYTES >> 4));      // 16-byte units of the start-address field
      const uint64_t dx = dw + (SW_W_BYTES >> 4);
      if (i < n_fp) {
        tc_fence_after();
        if (elected)
#pragma unroll
          for (int k = 0; k < 4; ++k)    // 16 values (32 bytes) of K per instruction
            mma_f16<1>(tmem_base + p.d_fp, dw + 2 * k, dx + 2 * k, p.idesc_fp, (i > 0 || k > 0) ? 1u : 0u);
      } else if (BITS == 8) {
        tc_fence_after();
        if (elected)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_i8<1>(d_int, dw + 2 * k, dx + 2 * k, p.idesc_int, (i > n_fp + 1 || k > 0) ? 1u : 0u);
      } else {
        const long long t1 = dbg ? clock64() : 0;
        if (!mbar_wait_warp(smem_u32(a_full + slot), slot_phase, abort_flag, p.status)) break;
        if (dbg) w_a += clock64() - t1;
        tc_fence_after();
        if (elected) {
          const uint64_t dx1 = dx + (uint32_t)(X_BYTES >> 4);
          const uint32_t a = tmem_base + slot * SW_A_COLS;
#pragma unroll
          for (int k = 0; k < 8; ++k)      // 32 codes = 8 TMEM columns of A per instruction
            mma_i8_ts<1>(d_int, a + 8 * k, (k < 4 ? dx : dx1) + 2 * (k & 3), p.idesc_int,
                         (i > n_fp || k > 0) ? 1u : 0u);
          mma_commit<1>(smem_u32(a_empty + slot));
        }
        if (++slot == p.a_slots) { slot = 0; slot_phase ^= 1; }
      }
      if (elected) mma_commit<1>(smem_u32(empty_bar + stage));
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (elected) mma_commit<1>(smem_u32(acc_full));     // also after an aborted loop: the epilogue wait ends either way
    __syncwarp();
    if (dbg && me == 0 && lane == 0) {
      unsigned long long *d = p.dbg + (size_t)blockIdx.x * 16;
      d[0] = (unsigned long long)(clock64() - t_begin);   // MMA warp: issue loop
      d[1] = (unsigned long long)w_full;                  // ... waiting for a loaded stage
      d[2] = (unsigned long long)w_a;                     // ... waiting for widened weights
      d[3] = (unsigned long long)nb;
    }
  } else if (BITS == 4) {
    // ================= widening warps: packed W (shared memory) -> int8 W (TMEM) =================
    const int q = warp & 3;                   // TMEM lane quarter this warp may access
    const int h = (warp - 2) >> 2;            // which 64 bytes of the 128-byte packed row
    const int row = q * 32 + lane;
    int stage = 0, slot = 0;
    uint32_t phase = 0, slot_phase = 0;
    const bool dbg = p.dbg != nullptr;
    long long c_full = 0, c_slot = 0, c_st = 0;
    const long long c_begin = clock64();
    for (int i = 0; i < nb; ++i) {
      const long long t0 = dbg ? clock64() : 0;
      if (!mbar_wait_warp(smem_u32(full_bar + stage), phase, abort_flag, p.status)) break;
      if (dbg) c_full += clock64() - t0;
      if (i >= n_fp) {
        const unsigned char *wrow = tiles + stage * STAGE_BYTES + row * 128;
        uint4 pk[4];
#pragma unroll
        for (int c = 0; c < 4; ++c)      // 16-byte chunk c of the row sits at chunk position c ^ (row % 8)
          pk[c] = *reinterpret_cast<const uint4 *>(wrow + ((((4 * h + c) ^ (row & 7))) << 4));
        uint32_t v[32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          widen8(pk[c].x, v[8 * c + 0], v[8 * c + 1]);
          widen8(pk[c].y, v[8 * c + 2], v[8 * c + 3]);
          widen8(pk[c].z, v[8 * c + 4], v[8 * c + 5]);
          widen8(pk[c].w, v[8 * c + 6], v[8 * c + 7]);
        }
        const long long t1 = dbg ? clock64() : 0;
        if (!mbar_wait_warp(smem_u32(a_empty + slot), slot_phase ^ 1u, abort_flag, p.status)) break;
        const long long t2 = dbg ? clock64() : 0;
        c_slot += t2 - t1;
        tc_fence_after();
        tmem_st32(tmem_base + ((uint32_t)(q * 32) << 16) + slot * SW_A_COLS + h * 32, v);
        tmem_st_wait();
        if (dbg) c_st += clock64() - t2;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(a_full + slot));
        if (++slot == p.a_slots) { slot = 0; slot_phase ^= 1; }
      }
      if (lane == 0) mbar_arrive(smem_u32(empty_bar + stage));   // this warp no longer reads the stage
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (dbg && warp == 2 && lane == 0) {
      unsigned long long *d = p.dbg + (size_t)blockIdx.x * 16;
      d[4] = (unsigned long long)(clock64() - c_begin);   // widening warp: whole loop
      d[5] = (unsigned long long)c_full;                  // ... waiting for a loaded stage
      d[6] = (unsigned long long)c_slot;                  // ... waiting for a free TMEM slot
      d[7] = (unsigned long long)c_st;                    // ... tcgen05.st until complete
    }
  }

  // ================= epilogue (warps 2-9) =================
  // Thread (q, lane, h) finishes weight row 32 q + lane for the tokens [h * ntok / 2, (h + 1) * ntok / 2), eight at a time.
  bool have = false;
  const int q = warp & 3, h = (warp - 2) >> 2;
  const int chunks = p.ntok / 16;                    // 8-token chunks per thread
  const uint32_t lane_base = (uint32_t)(q * 32) << 16;
  auto load_int = [&](int tok0, uint32_t (&acc)[8]) {
    if (n_int > 0) {
      tmem_ld8(tmem_base + lane_base + p.d_int + tok0, acc);
      tmem_ld_wait(acc);
      if (BITS == 8 && n_int > 1) {
        uint32_t second[8];
        tmem_ld8(tmem_base + lane_base + (p.d_int + p.d_fp) / 2 + tok0, second);
        tmem_ld_wait(second);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += second[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0;
    }
  };
  __syncwarp();
  if (worker) {
    have = mbar_wait(smem_u32(acc_full), 0, abort_flag, p.status) && !*abort_flag;
    have = __all_sync(0xFFFFFFFFu, have);
    tc_fence_after();
  }
  const int row = q * 32 + lane, n = n0 + row;
  const float scol = Traits<T>::to_float(ep_scol), wred = Traits<T>::to_float(ep_wred), bias = Traits<T>::to_float(ep_bias);
  T *out = static_cast<T *>(p.out);
  auto finish = [&](int m, int acc, float fp) {
    if (BITS == 4) acc >>= 4;                        // the weights carried a factor 16; the quotient is exact
    const float add = fmaf(s_zs[m], wred, fp + bias);
    out[(size_t)m * p.ldo + n] = Traits<T>::from_float(fmaf((float)acc, s_srow[m] * scol, add));
  };
  if (S > 1) {
    if (worker && have) {                            // all MMAs are complete, so nothing reads or fills the ring any more
#pragma unroll 1
      for (int c = 0; c < chunks; ++c) {
        const int tok0 = h * (p.ntok / 2) + 8 * c;
        uint32_t acc[8];
        load_int(tok0, acc);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum_i[(tok0 + j) * SW_ROWS + row] = (int)acc[j];
        if (n_fp > 0) {
          tmem_ld8(tmem_base + lane_base + p.d_fp + tok0, acc);
          tmem_ld_wait(acc);
#pragma unroll
          for (int j = 0; j < 8; ++j) sum_f[(tok0 + j) * SW_ROWS + row] = __uint_as_float(acc[j]);
        }
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                  // the sums of all CTAs are in place
    if (worker && have && n < p.N) {
      // This CTA's share of the tokens, every second one from h on.  All loads of a batch are under way before the first is
      // used: one at a time they cost 0.2 us per token (80 tokens, 33 slabs of 1600 int4 columns: 14.2 -> 9.7 us).
      const int t0 = rank * p.ntok / S + h, last = min(p.M, (rank + 1) * p.ntok / S) - 1;
      const uint32_t own_i = smem_u32(sum_i), fp0 = map_to_rank(smem_u32(sum_f), 0);
      auto finish_share = [&](auto ctas) {
        constexpr int C = decltype(ctas)::value, U = 32 / C;
        for (int m0 = t0; m0 <= last; m0 += 2 * U) {
          int v[C][U], f[U];
#pragma unroll
          for (int s = 0; s < C; ++s) {
            const uint32_t theirs = map_to_rank(own_i, s);
#pragma unroll
            for (int u = 0; u < U; ++u) v[s][u] = ld_cluster_s32(theirs + (uint32_t)((min(m0 + 2 * u, last) * SW_ROWS + row) * 4));
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            f[u] = p.nf > 0 ? ld_cluster_s32(fp0 + (uint32_t)((min(m0 + 2 * u, last) * SW_ROWS + row) * 4)) : 0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (m0 + 2 * u > last) break;
            int acc = 0;
#pragma unroll
            for (int s = 0; s < C; ++s) acc += v[s][u];
            finish(m0 + 2 * u, acc, __int_as_float(f[u]));
          }
        }
      };
      if (S == 2) finish_share(std::integral_constant<int, 2>());
      else if (S == 4) finish_share(std::integral_constant<int, 4>());
      else finish_share(std::integral_constant<int, 8>());
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                  // no CTA leaves while another reads its sums
  } else if (worker && have) {
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      const int tok0 = h * (p.ntok / 2) + 8 * c;
      if (tok0 >= p.M) break;                        // warp-uniform
      uint32_t acc_i[8], acc_f[8];
      __syncwarp();                                  // tcgen05.ld is warp-collective: all lanes, also rows beyond N, converged
      load_int(tok0, acc_i);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc_f[j] = 0;
      if (n_fp > 0) {
        tmem_ld8(tmem_base + lane_base + p.d_fp + tok0, acc_f);
        tmem_ld_wait(acc_f);
      }
      if (n < p.N) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (tok0 + j < p.M) finish(tok0 + j, (int)acc_i[j], __uint_as_float(acc_f[j]));
      }
    }
  }

  // ---- teardown: every thread arrives here, also after an aborted wait
  if (*abort_flag) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);   // let bulk copies in flight land
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, p.tmem_cols);
  }
}

// Clusters of `size` CTAs (2, 4 or 8) that run at once on the current device.  Fewer than SMs x CTAs per SM / size: a cluster has
// to fit the SMs of one processing cluster of the GPU.  The occupancy call answers that for one CTA per SM (74, 33 and 15 on a
// GPU of 148 SMs; it does not know that two of these kernels fit an SM).  With two per SM a cluster takes half as many SMs:
// measured by the launch time's jump, 33 clusters of eight run at once and 69 to 71 of four (of 74: launches overlap and leave
// gaps).  Counting slots alone sent 72 to 74 slabs to a second wave: 19.8 us for 64 tokens of 4096 int4 columns, now 12.7.
int resident_clusters(int ctas_per_sm, int size) {
  if (ctas_per_sm == 2) {
    if (size == 2) return num_sms();
    const int r = resident_clusters(1, size / 2);
    return size == 4 ? r - r / 14 : r;
  }
  static std::atomic<int> cached[kMaxDevices][4];        // 0 = not asked yet, else the answer + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  std::atomic<int> &known = cached[dev][size == 2 ? 1 : (size == 4 ? 2 : 3)];
  int n = known.load() - 1;
  if (n >= 0) return n;
  auto kern = stream_w_kernel<__half, 8>;                // the others take the same room
  LaunchCfg lc(dim3(2 * size * num_sms()), dim3(SW_THREADS), 200 * 1024, nullptr, size);
  lc.cfg.numAttrs = 1;                                   // the cluster shape only
  n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM_SM) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &lc.cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known.store(n + 1);
  return n;
}

template <typename T, int BITS>
int launch_t(const CUtensorMap &tw, const CUtensorMap &tx, const CUtensorMap &tfw, const CUtensorMap &tfx,
             const StreamParams &p, int slabs, size_t smem, cudaStream_t st) {
  auto kern = stream_w_kernel<T, BITS>;
  static PerDeviceSmem state;
  {
    const int rc = ensure_smem(state, kern, SW_SMEM_SM);
    if (rc != QUIK_OK) return rc;
  }
  LaunchCfg lc(dim3(slabs * p.splits), dim3(SW_THREADS), smem, st, p.splits);
  QUIK_CUDA_TRY(cudaLaunchKernelEx(&lc.cfg, kern, tw, tx, tfw, tfx, p));
  return check_launch("stream_w_kernel");
}

// Rows [first, first + count) of the layer (first a multiple of SW_ROWS), in one launch.
int launch_rows(const void *q, const void *w, int bits, int M, int first, int count, int K_int, const Epilogue &ep, int per_sm, int splits,
                cudaStream_t st) {
  const int ntok = (M + 15) & ~15;                                                // the MMA's N
  StreamParams p{};
  p.M = M;
  p.N = count;
  const size_t at = (size_t)first;
  const int w_row_bytes = bits == 4 ? K_int / 2 : K_int;
  p.nk = (w_row_bytes + 127) / 128;
  p.nf = ep.fp_a != nullptr && ep.F > 0 ? (ep.F + 63) / 64 : 0;
  const int slabs = (count + SW_ROWS - 1) / SW_ROWS;
  p.splits = splits;
  const StreamPlan plan = plan_stream(bits, ntok, per_sm);
  p.ntok = ntok;
  p.stages = plan.stages;
  p.stage_bytes = plan.stage_bytes;
  p.x_bytes = plan.x_bytes;
  p.a_slots = plan.a_slots;
  p.d_int = plan.d_int;
  p.d_fp = plan.d_fp;
  p.tmem_cols = plan.tmem_cols;
  p.idesc_int = make_idesc(2, 1, SW_ROWS, ntok);
  p.idesc_fp = make_idesc(1, ep.dtype == QUIK_BF16 ? 1 : 0, SW_ROWS, ntok);
  p.meta = ep.meta;
  auto row = [&](const void *v, size_t bytes) { return v ? static_cast<const unsigned char *>(v) + at * bytes : nullptr; };
  p.scale_col = row(ep.scale_col, 2);
  p.w_reduced = row(ep.w_reduced, 2);
  p.bias = row(ep.bias, 2);
  p.out = static_cast<unsigned char *>(ep.out) + at * 2;
  p.ldo = ep.ldo;
  p.shift_value = ep.shift_value;
  p.dbg = get_debug_counters();
  p.status = device_status_word();
  if (p.status == nullptr) return QUIK_ERR_CUDA;

  CUtensorMap tw, tx, tfw, tfx;
  int rc;
  if ((rc = make_tmap(&tw, row(w, w_row_bytes), CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, count, w_row_bytes, SW_ROWS)) != QUIK_OK) return rc;
  if ((rc = make_tmap(&tx, q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K_int, ntok)) != QUIK_OK) return rc;
  if (p.nf > 0) {
    const CUtensorMapDataType fdt = ep.dtype == QUIK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    if ((rc = make_tmap(&tfw, row(ep.fp_b, 2 * (size_t)ep.F), fdt, 2, count, ep.F, SW_ROWS)) != QUIK_OK) return rc;
    if ((rc = make_tmap(&tfx, ep.fp_a, fdt, 2, M, ep.F, ntok)) != QUIK_OK) return rc;
  } else {
    tfw = tw;
    tfx = tx;
  }
  if (ep.dtype == QUIK_BF16)
    return bits == 4 ? launch_t<__nv_bfloat16, 4>(tw, tx, tfw, tfx, p, slabs, plan.smem, st)
                     : launch_t<__nv_bfloat16, 8>(tw, tx, tfw, tfx, p, slabs, plan.smem, st);
  return bits == 4 ? launch_t<__half, 4>(tw, tx, tfw, tfx, p, slabs, plan.smem, st)
                   : launch_t<__half, 8>(tw, tx, tfw, tfx, p, slabs, plan.smem, st);
}


}  // namespace

// q: [M, K_int] int8 codes (one per byte); w: [N, K_int/2] packed int4 (bits == 4) or [N, K_int] int8.
int launch_stream_w(const void *q, const void *w, int bits, int M, int N, int K_int, const Epilogue &ep,
                    cudaStream_t st) {
  if (M == 0 || N == 0) return QUIK_OK;
  if (M > QUIK_STREAM_M_MAX) return QUIK_ERR_UNSUPPORTED;
  if (K_int <= 0 || K_int % (bits == 4 ? 32 : 16) != 0) return QUIK_ERR_SHAPE;
  if (!aligned16(q) || !aligned16(w)) return QUIK_ERR_ALIGN;
  const bool has_fp = ep.fp_a != nullptr && ep.F > 0;
  if (has_fp && (ep.F % 8 != 0 || !aligned16(ep.fp_a) || !aligned16(ep.fp_b))) return QUIK_ERR_ALIGN;
  if (ep.meta == nullptr || ep.w_reduced == nullptr || ep.y != nullptr) return QUIK_ERR_UNSUPPORTED;

  const int ntok = (M + 15) & ~15, sms = num_sms();
  const int nf = has_fp ? (ep.F + 63) / 64 : 0, total = ((bits == 4 ? K_int / 2 : K_int) + 127) / 128 + nf;
  const int slabs = (N + SW_ROWS - 1) / SW_ROWS;
  // Split K over a cluster while all CTAs still run at once, every CTA keeps at least two k-blocks and the outlier
  // blocks all fall to the first CTA.
  auto choose_splits = [&](int ctas_per_sm, int of_slabs) {
    int s = 1;
    while (s < 8 && total / (s * 2) >= (nf > 2 ? nf : 2) && of_slabs <= resident_clusters(ctas_per_sm, s * 2)) s *= 2;
    return s;
  };
  int per_sm = 1, splits = choose_splits(1, slabs);
  if (ntok <= 64) {
    // Two CTAs per SM, each with half of the ring, or one?  More slabs than SMs: two (172 slabs of 4096 int4 columns, 48 tokens:
    // 19.3 against 27.6 us).  Otherwise two only where they allow a deeper split of a long K: each CTA starts and
    // finishes its own pipeline, so up to 20 blocks per CTA one is as good or better (96 slabs of 4096 int4 columns, 33 / 64
    // tokens: 14.2 / 14.7 against 15.2 / 16.2 us; 40 slabs 11.1 / 11.6 against 11.2 / 11.8), beyond that two keep the widening
    // warps busier (40 slabs of 11008 columns 16.8 / 18.1 against 18.3 / 18.8 us, 120 slabs 26.1 / 27.4 against 29.9 /
    // 30.2); int8 blocks need no widening and gain only while most CTAs still have an SM for themselves (40 and 96
    // slabs of 11008 columns, 33 tokens: 17.1 against 19.7 and 29.6 against 31.3 us, 120 slabs: 33.3 against 32.1).
    const int s2 = choose_splits(2, slabs);
    if (slabs > sms || (s2 > splits && total / splits > 20 && (bits == 4 || 5 * slabs * s2 <= 7 * sms))) {
      per_sm = 2;
      splits = s2;
    }
  }
  Epilogue e = ep;
  if (e.ldo <= 0) e.ldo = N;
  // More slabs than run at once: the ones beyond the last full wave may go to a launch of their own that splits K (its setup and
  // first prefetch overlap the end of the first launch, its loads come after).  It costs about 4 us and takes integer blocks out of the
  // chain.  With one CTA per SM a block of the last wave is 0.5 us (int8: 0.25), however many slabs are left: at least 8
  // (int8: 16) blocks have to go.  Two CTAs per SM share the weight stream: few slabs leave SMs with one CTA, whose blocks then
  // come faster, and many fill the SMs anyway, so only up to a quarter of a wave, and for about twice the blocks.  From three full
  // waves on CTAs do not end together any more, the last slabs start as SMs come free: twice the blocks again.
  // One launch against two, us: 80 tokens, slabs beyond 148, columns (blocks saved): int4 37, 2048 (4) 24.0 / 24.7; 60, 4096 (8)
  // 34.2 / 33.0; 18, 8192 (24) 51.5 / 42.3; 74, 16384 (32) 91.2 / 77.7; int8 37, 2048 (8) 25.5 / 25.6; 18, 4096 (24) 35.8 / 33.1.
  // 20 tokens, beyond 296: int4 36, 4096 (12) 34.9 / 36.1; 36, 8192 (24) 55.9 / 53.7; 74, 16384 (32) 98.5 / 90.5; 120, 8192 (16)
  // 57.3 / 60.2; int8 74, 4096 (16) 46.8 / 48.1; 36, 11008 (64) 99.0 / 89.0; 148, 11008 (43) 109 / 113.  (A line at 8 blocks for all, as
  // it was before, took 5 us too long in places.  Of 700 drawn layers with up to half a wave beyond full ones, not those that the
  // lines were drawn by, 308 now get two launches, one of them wrongly by more than 1 %: 1.6 %.)
  const int wave = sms * per_sm, beyond = slabs > wave ? slabs % wave : 0;
  if (beyond > 0 && (per_sm == 1 || 4 * beyond <= wave)) {
    const int s = choose_splits(per_sm, beyond), nk = total - nf;
    int least = per_sm == 1 ? (bits == 4 ? 8 : 16) : (bits == 4 ? 20 : 32);
    if (slabs >= 3 * wave) least *= 2;
    if (nk - (nk + s - 1) / s >= least) {
      const int first = (slabs - beyond) * SW_ROWS;
      const int rc = launch_rows(q, w, bits, M, 0, first, K_int, e, per_sm, 1, st);
      if (rc != QUIK_OK) return rc;
      return launch_rows(q, w, bits, M, first, N - first, K_int, e, per_sm, s, st);
    }
  }
  return launch_rows(q, w, bits, M, 0, N, K_int, e, per_sm, splits, st);
}

}  // namespace quik
