// int8 x int8 -> int32 GEMM on the Blackwell tensor cores (tcgen05.mma kind::i8) with TMA-fed
// shared-memory tiles, TMEM accumulators and a fused dequantize epilogue that can also add an
// fp16/bf16 "outlier" GEMM (tcgen05.mma kind::f16 into a second TMEM accumulator).
//
// Computes, per 128 x block_n output tile (QUIK experiments/qlinear.py:122-145 in one launch):
//   acc_i[m,n] = sum_k A[m,k] * B[n,k]            (int8 operands, exact int32)   matmul.cu:98-136
//   acc_f[m,n] = sum_j FA[m,j] * FB[n,j]          (fp16/bf16 operands, fp32)     qlinear.py:124
//   out = T( acc_i * (s_m * sc_n) + ((z_m + shift * s_m) * wred_n + (acc_f + bias_n + y[m,n])) )
//                                                                                asymmetric.cu:134-146
// or stores acc_i as int32 (mode 0).
//
// Structure (one persistent CTA per SM or one CTA pair per two SMs, 384 threads per CTA):
//   warp 0    TMA producer: cp.async.bulk.tensor.2d loads of the A / B k-blocks (128 bytes of K
//             per row, 128B swizzle) into a ring of shared-memory stages, completion on mbarriers.
//   warp 1    allocates TMEM; one elected lane issues tcgen05.mma (M=128 or 256, N=block_n, K=32
//             bytes) from shared-memory descriptors and commits each stage back to the producer.
//   warps 4-11 epilogue: tcgen05.ld the accumulators (32 lanes x 16 columns per warp and step),
//             apply the dequantize arithmetic in fp32 and store through shared memory (bulk stores where rows allow).
// Outlier k-blocks (64 fp16 values = 128 bytes per row) travel through the same ring as the integer
// k-blocks; TMEM holds two accumulator regions so the epilogue of tile i overlaps the MMAs of tile
// i+1 (schedule in gemm_epilogue.cuh).
// The tile width block_n is a launch parameter (any multiple of 16 up to the kernel's capacity CAP_N,
// which fixes the shared-memory and TMEM plan): the host picks it per problem so that the tiles fill
// whole waves of CTAs (choose_tile below).
// Every wait is bounded: when a limit is hit the kernel records it in a device status word,
// all roles leave their loops, TMEM is released and the kernel returns.
#include <cuda.h>

#include <atomic>
#include <mutex>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tcgen05_ptx.cuh"

namespace quik {

__device__ unsigned int g_device_status = 0;

namespace {

constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 128 + 32 * EPI_WARPS;     // TMA warp, MMA warp, two that only fill their warpgroup, epilogue warps
// Registers per thread once the roles part: the launch gives 168 to each of 384 threads; the first four warps hand most of theirs to
// the epilogue warps, which keep 64 words of the outlier product and work on two chunks of an accumulator at once.
constexpr int REGS_LAUNCH = 168, REGS_ISSUE = 72, REGS_EPILOGUE = 216;
static_assert(128 * REGS_ISSUE + 32 * EPI_WARPS * REGS_EPILOGUE <= NUM_THREADS * REGS_LAUNCH, "register split");
// Process-wide tuning knobs (quik_config_set): plain words, meant to be set once before the layers run; a
// launch reads each of them once.
std::atomic<int> g_tile_n{0};                                 // 0 = choose by shape, else a multiple of 16 in [32, 256]
std::atomic<int> g_cta_pair{0};                               // 0 = by shape, 1 = never, 2 = always
std::atomic<int> g_l2_hint{0};                                // 1 = token-operand loads carry an L2 evict-last hint
std::atomic<unsigned long long *> g_dbg{nullptr};             // diagnostic counters (device memory), off by default

// Shared-memory plan after the 1024-byte aligned ring of stages: 256 bytes of barriers etc. and the
// per-warp epilogue vectors (rounded to 1024 together), then the output staging of each epilogue
// warp.
constexpr int EPI_COLS(int cap_n) { return cap_n / (EPI_WARPS / 4); }       // most columns per epilogue warp
constexpr int AUX_BYTES(int cap_n) { return ((256 + EPI_WARPS * 3 * EPI_COLS(cap_n) * 4) + 1023) / 1024 * 1024; }
constexpr int stage_bytes(int cap_n, int ctas) { return (BLOCK_M + cap_n / ctas) * STAGE_K_BYTES; }
// Ring depth: as many stages as fit (at most 8).
constexpr int num_stages(int cap_n, int ctas) {
  const int n = (SMEM_LIMIT - 1024 - AUX_BYTES(cap_n) - EPI_WARPS * EPI_BUF_BYTES) / stage_bytes(cap_n, ctas);
  return n > 8 ? 8 : n;
}

// ---------------------------------------------------------------------------------------------
// The tiles of a CTA are blockIdx.x + j * gridDim.x; their two accumulator regions in TMEM (CAP_N columns apart) and the order
// of their products are described in gemm_epilogue.cuh.
//
// CTAS == 2: two CTAs on neighbouring SMs (a cluster of 2) work on one 256 x block_n tile.  Each
// loads its own 128 rows of A and only its half of the B rows, so a CTA moves a third less operand
// data per multiply-accumulate than alone.  The leader (cluster rank 0) issues the MMAs for the pair
// and owns the barriers that count loads and region releases; commits reach both CTAs.
// KIND, ROWS_ARE: what becomes of the integer product and how it is stored, see EpilogueWarp.
template <typename T, int CAP_N, int KIND, int CTAS, int ROWS_ARE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_fa, const __grid_constant__ CUtensorMap tmap_fb,
                    const __grid_constant__ CUtensorMap tmap_out, const GemmParams p) {
  constexpr bool HAS_FP = KIND == 2;
  constexpr int A_BYTES = BLOCK_M * STAGE_K_BYTES;
  constexpr int STAGE_BYTES = stage_bytes(CAP_N, CTAS);      // room for the widest tile; narrower ones use less of it
  constexpr int STAGES = num_stages(CAP_N, CTAS);
  constexpr int TMEM_ALLOC = 2 * CAP_N;                       // two accumulator regions, CAP_N columns apart
  constexpr int TILE_M = BLOCK_M * CTAS;
  const int bn = p.block_n;
  const int b_rows = bn / CTAS;                               // B rows this CTA loads per k-block
  const uint32_t stage_tx = (uint32_t)(A_BYTES + b_rows * STAGE_K_BYTES) * CTAS;   // bytes of the whole pair

  extern __shared__ unsigned char smem_dyn[];
  // 128B-swizzled tiles need 1024-byte alignment
  unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  unsigned char *aux = tiles + STAGES * STAGE_BYTES;
  uint64_t *full_bar = reinterpret_cast<uint64_t *>(aux);               // [STAGES]
  uint64_t *empty_bar = full_bar + STAGES;                             // [STAGES]
  uint64_t *acc_full = empty_bar + STAGES;                             // [2] integer product complete
  uint64_t *acc_empty = acc_full + 2;                                  // [2] region free again
  uint64_t *fp_full = acc_empty + 2;                                   // [2] outlier product complete
  uint64_t *fp_drained = fp_full + 2;                                  // [2] outlier product kept, region free
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fp_drained + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  // per-column epilogue vectors, one private copy per epilogue warp (no cross-warp barrier needed)
  float *s_vec = reinterpret_cast<float *>(aux + 256);                 // [EPI_WARPS][3][EPI_COLS], 16-byte aligned
  // output staging: [EPI_WARPS][EPI_BUF_BYTES], 1024-byte aligned
  unsigned char *s_out = tiles + STAGES * STAGE_BYTES + AUX_BYTES(CAP_N);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(full_bar + s), 1);
      mbar_init(smem_u32(empty_bar + s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(acc_full + s), 1);
      mbar_init(smem_u32(acc_empty + s), EPI_WARPS * CTAS);    // epilogue warps of the whole pair
      mbar_init(smem_u32(fp_full + s), 1);
      mbar_init(smem_u32(fp_drained + s), EPI_WARPS * CTAS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    if (ROWS_ARE == ALIGNED) prefetch_tmap(&tmap_out);
    if (HAS_FP) {
      prefetch_tmap(&tmap_fa);
      prefetch_tmap(&tmap_fb);
    }
  }
  if (warp == 1) {
    tmem_alloc<CTAS>(smem_u32(tmem_slot), TMEM_ALLOC);
    tmem_relinquish<CTAS>();
  }
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();          // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                                 // set-up done; everything below reads or writes global memory

  const int rank = CTAS == 2 ? (int)cluster_ctarank() : 0;
  const int unit = (int)blockIdx.x / CTAS, num_units = (int)gridDim.x / CTAS;    // a unit = CTA or CTA pair
  const int n_local = (p.num_tiles - unit + num_units - 1) / num_units;           // tiles of this unit

  if (warp >= 4) {
    // ================= epilogue (warps 4..11): gemm_epilogue.cuh =================
    set_max_regs_up<REGS_EPILOGUE>();
    EpilogueWarp<T, KIND, 0, CTAS, EPI_COLS(CAP_N), ROWS_ARE> ew(p, &tmap_out, tmem_base, CAP_N, unit, num_units, rank, warp - 4, warp & 3, lane, s_vec,
                                                       s_out, acc_full, acc_empty, fp_full, fp_drained, abort_flag);
    ew.run(n_local);
    if (p.dbg && warp == 4 && lane == 0) ew.write_counters((int)blockIdx.x);
  } else if (set_max_regs_down<REGS_ISSUE>(); warp == 0) {
    // ================= TMA producer =================
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    // The token operand A is read again by every column tile of the launch and fits in L2: its lines are marked to
    // be evicted last, so that data streaming through L2 meanwhile (the weights, the outputs, a tensor-parallel
    // rank's peer copies) does not push it out.
    const uint64_t keep = l2_policy_evict_last();
    const bool hint = p.l2_hint != 0;
    for_each_block<HAS_FP>(n_local, p.int_kb, p.fp_kb, [&](int j, auto is_fp, int kb) {
      constexpr bool fp = decltype(is_fp)::value;
      const int tile = unit + j * num_units;
      const int m0 = (tile % p.num_m_tiles) * TILE_M + rank * BLOCK_M;      // this CTA's rows of A
      const int n0 = (tile / p.num_m_tiles) * bn + rank * b_rows;           // this CTA's rows of B
      if (!mbar_wait_warp(smem_u32(empty_bar + stage), phase ^ 1, abort_flag, p.status)) return false;
      if (elected) {
        const uint32_t fb = smem_u32(full_bar + stage);
        const uint32_t sa = smem_u32(tiles + stage * STAGE_BYTES);
        if (rank == 0) mbar_expect_tx(fb, stage_tx);
        if (fp) {
          tma_load_2d<CTAS>(sa, &tmap_fa, fb, kb * 64, m0);
          tma_load_2d<CTAS>(sa + A_BYTES, &tmap_fb, fb, kb * 64, n0);
        } else {
          if (hint) tma_load_2d_policy<CTAS>(sa, &tmap_a, fb, kb * STAGE_K_BYTES, m0, keep);
          else tma_load_2d<CTAS>(sa, &tmap_a, fb, kb * STAGE_K_BYTES, m0);
          tma_load_2d<CTAS>(sa + A_BYTES, &tmap_b, fb, kb * STAGE_K_BYTES, n0);
        }
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
      return true;
    });
    __syncwarp();
  } else if (warp == 1) {
    // ================= MMA issuer (pair leader only) =================
    // The whole warp walks the loop and one elected lane issues.  Loop exits are warp votes, so stage, phase and the
    // descriptors made from them are uniform over the warp.  (With the loop inside a `lane == 0` branch whose exits
    // depended on that lane's waits, one instruction left every ~217 cycles: a 256 x 256 x 128 block took 850 to 970
    // cycles, now 512 to 545, the tensor pipe itself needing 512.  Llama-2-70B gate+up at 4096 tokens: 1845 -> 1440 us
    // sustained, 7B qkv at 2048 tokens: 122 -> 102 us.)
    if (rank == 0) {
      const bool elected = elect_one();
      const bool dbg = p.dbg != nullptr;
      const uint64_t da0 = make_smem_desc(smem_u32(tiles)), db0 = make_smem_desc(smem_u32(tiles) + A_BYTES);
      int stage = 0;
      uint32_t phase = 0;
      long long w_region = 0, w_full = 0;
      const long long t_begin = clock64();
      for_each_block<HAS_FP>(n_local, p.int_kb, p.fp_kb, [&](int j, auto is_fp, int kb) {
        constexpr bool fp = decltype(is_fp)::value;
        if (kb == 0) {
          const long long t0 = dbg ? clock64() : 0;
          uint32_t parity;
          const uint64_t *bar = region_barrier<HAS_FP>(j, fp, acc_empty, fp_drained, parity);
          if (bar != nullptr && !mbar_wait_warp(smem_u32(bar), parity, abort_flag, p.status)) return false;
          if (dbg) w_region += clock64() - t0;
        }
        const long long t1 = dbg ? clock64() : 0;
        if (!mbar_wait_warp(smem_u32(full_bar + stage), phase, abort_flag, p.status)) return false;
        if (dbg) w_full += clock64() - t1;
        tc_fence_after();
        if (elected) {
          // stage bases and 32-byte K steps inside the swizzled row are offsets of the 16-byte start-address field
          const uint64_t da = da0 + (uint32_t)(stage * (STAGE_BYTES >> 4)), db = db0 + (uint32_t)(stage * (STAGE_BYTES >> 4));
          const uint32_t d = tmem_base + ((fp ? j + 1 : j) & 1) * CAP_N;
#pragma unroll
          for (int k = 0; k < STAGE_K_BYTES / 32; ++k) {
            if (fp) mma_f16<CTAS>(d, da + 2 * k, db + 2 * k, p.idesc_fp, (k > 0 || kb > 0) ? 1u : 0u);
            else mma_i8<CTAS>(d, da + 2 * k, db + 2 * k, p.idesc_int, (k > 0 || kb > 0) ? 1u : 0u);
          }
          mma_commit<CTAS>(smem_u32(empty_bar + stage));    // stage reusable once these MMAs retire
          if (fp && kb == p.fp_kb - 1) mma_commit<CTAS>(smem_u32(fp_full + (j & 1)));
          if (!fp && kb == p.int_kb - 1) mma_commit<CTAS>(smem_u32(acc_full + (j & 1)));
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        return true;
      });
      if (dbg && lane == 0) {
        unsigned long long *d = p.dbg + (size_t)blockIdx.x * 16;
        d[0] = (unsigned long long)(clock64() - t_begin);   // MMA warp: issue loop
        d[1] = (unsigned long long)w_region;                // ... waiting for a free accumulator region
        d[2] = (unsigned long long)w_full;                  // ... waiting for operands
        d[3] = (unsigned long long)n_local;
      }
    }
  }

  // ---- teardown: every thread arrives here, also after an aborted wait
  if (*abort_flag) {
    // let bulk copies that are still in flight land before shared memory is released
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();          // no CTA leaves while its peer may still address it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<CTAS>(tmem_base, TMEM_ALLOC);
  }
}

// ---------------------------------------------------------------------------------------------
// Host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres);
    if (e == cudaSuccess && qres == cudaDriverEntryPointSuccess) fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

}  // namespace

int make_tmap(CUtensorMap *map, const void *base, CUtensorMapDataType dt, int elem_bytes, int rows, int cols,
              int box_rows, int box_row_bytes, long long pitch) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return QUIK_ERR_CUDA;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(pitch > 0 ? pitch : cols) * elem_bytes};
  cuuint32_t box[2] = {(cuuint32_t)(box_row_bytes / elem_bytes), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapSwizzle sw = box_row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  CUresult r = fn(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
    return QUIK_ERR_CUDA;
  }
  return QUIK_OK;
}

// m = 128 (one CTA) or 256 (CTA pair)
uint32_t make_idesc(int c_format, int ab_format, int m, int n) {
  uint32_t d = 0;
  d |= (uint32_t)c_format << 4;      // accumulator: 1 = F32, 2 = S32
  d |= (uint32_t)ab_format << 7;     // A format
  d |= (uint32_t)ab_format << 10;    // B format
  d |= (uint32_t)(n >> 3) << 17;     // N / 8
  d |= (uint32_t)(m >> 4) << 24;     // M / 16
  return d;
}

unsigned int *device_status_word() {
  static std::atomic<unsigned int *> cached[kMaxDevices];      // the address of a device's word never changes
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return nullptr;
  }
  unsigned int *known = cached[dev].load();
  if (known != nullptr) return known;
  void *p = nullptr;
  if (cudaGetSymbolAddress(&p, g_device_status) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  cached[dev].store(static_cast<unsigned int *>(p));
  return static_cast<unsigned int *>(p);
}

namespace {

constexpr size_t smem_bytes(int cap_n, int ctas) {
  return 1024 /*align slack*/ + (size_t)num_stages(cap_n, ctas) * stage_bytes(cap_n, ctas) + AUX_BYTES(cap_n) +
         EPI_WARPS * EPI_BUF_BYTES;
}

// Largest number of CTA pairs that can be resident at once (0 if pairs cannot be launched).
template <typename Kern>
int max_pairs(Kern kern, size_t smem) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * num_sms());
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// Units (CTAs, or CTA pairs) of one kernel instantiation that are resident at once on the current device.
// The shared-memory opt-in and the occupancy answer belong to a device, so they are kept per device ordinal.
template <typename T, int CAP_N, int KIND, int CTAS, int ROWS_ARE>
int resident_units(int *out) {
  static std::mutex mu;
  static int cached[kMaxDevices];       // 0 = not asked yet, -1 = cannot launch
  int dev = 0;
  QUIK_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return QUIK_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == 0) {
    auto kern = gemm_tcgen05_kernel<T, CAP_N, KIND, CTAS, ROWS_ARE>;
    constexpr size_t smem = smem_bytes(CAP_N, CTAS);
    cudaFuncAttributes at;
    QUIK_CUDA_TRY(cudaFuncGetAttributes(&at, kern));
    if (at.numRegs < REGS_LAUNCH) return QUIK_ERR_UNSUPPORTED;      // the epilogue warps would wait for registers for ever
    QUIK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int n = CTAS == 1 ? num_sms() : max_pairs(kern, smem);
    cached[dev] = n > 0 ? n : -1;
  }
  *out = cached[dev];
  return QUIK_OK;
}

template <typename T, int CAP_N, int KIND, int CTAS, int ROWS_ARE>
int launch_t(const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tfa, const CUtensorMap &tfb,
             const CUtensorMap &to, const GemmParams &p, cudaStream_t st) {
  auto kern = gemm_tcgen05_kernel<T, CAP_N, KIND, CTAS, ROWS_ARE>;
  constexpr size_t smem = smem_bytes(CAP_N, CTAS);
  int resident = 0;
  const int rc = resident_units<T, CAP_N, KIND, CTAS, ROWS_ARE>(&resident);
  if (rc != QUIK_OK) return rc;
  if (resident <= 0) return QUIK_ERR_UNSUPPORTED;
  const int units = p.num_tiles < resident ? p.num_tiles : resident;
  LaunchCfg lc(dim3(CTAS * units), dim3(NUM_THREADS), smem, st, CTAS);
  QUIK_CUDA_TRY(cudaLaunchKernelEx(&lc.cfg, kern, ta, tb, tfa, tfb, to, p));
  return check_launch("gemm_tcgen05_kernel");
}

// ---- tile shape per problem -------------------------------------------------------------------
// A launch is a number of waves of equally sized tiles over the resident units (CTAs or CTA pairs).  The time of a tile depends
// little on its width: a k-block of a pair moves 16 KB of A and 64 * block_n bytes of B per CTA from L2, 15 to 18 TB/s over the chip,
// which takes about 179 + 0.50 * block_n ns (single CTAs 200 + 0.70 * block_n); but its epilogue takes 2000 + 20 * block_n ns (six
// tenths of that without an outlier product; a fifth more in pairs, whose regions are free when both CTAs are done), and with few
// k-blocks that is the longer one.  Pairs also start and end 900 ns later.  So a narrower tile only pays where it saves a wave or where epilogues bound the launch; among
// equals the widest is taken, and pairs before singles.  Fitted to all widths of 24 problems of 200 to 4096 tokens, 896 to 18208 integer
// columns.  On 1686 drawn problems of 129 to 4096 tokens, the two narrowest widths of each number of waves timed for singles and
// pairs, the choice costs 0.9 % more than the best of them on average, 11 % at worst (one rule for singles and pairs and no epilogue:
// 3.4 and 23 %; constants refitted to 3985 others: 0.9).  Problems of one wave of 32-column tiles are where it errs most often, to
// either side by up to 5 %.  333 tokens through 11008 x 4096 33.5 us, now 29.1, 777 through 4096 x 6912 32.1, now 27.1.
double tile_cost(int M, int N, int kblocks, bool outliers, int ctas, int bn, int units) {
  const int tile_m = BLOCK_M * ctas;
  const long long tiles = (long long)((M + tile_m - 1) / tile_m) * ((N + bn - 1) / bn);
  const long long waves = (tiles + units - 1) / units;
  const double products = kblocks * (ctas == 2 ? 179.0 + 0.50 * bn : 200.0 + 0.70 * bn) + 800.0;
  const double epilogue = (2000.0 + 20.0 * bn) * (outliers ? 1.0 : 0.6) * (ctas == 2 ? 1.2 : 1.0);
  return (double)waves * (products > epilogue ? products : epilogue) + (ctas == 2 ? 900.0 : 0.0);
}

}  // namespace

void choose_tile(int M, int N, int int_kb, int fp_kb, int *ctas_out, int *bn_out) {
  const int forced_n = g_tile_n.load(), pair_mode = g_cta_pair.load();
  const int sms = num_sms();
  const int n16 = (N + 15) & ~15;
  double best = 0.0;
  int best_ctas = 1, best_bn = 128;
  bool have = false;
  for (int ctas = 2; ctas >= 1; --ctas) {
    if (ctas == 2 && (pair_mode == 1 || (pair_mode == 0 && M <= BLOCK_M))) continue;
    if (ctas == 1 && pair_mode == 2) continue;
    const int units = ctas == 2 ? sms / 2 : sms;
    for (int bn = 256; bn >= 32; bn -= 16) {
      int cand = bn;
      if (forced_n) {
        if (bn != 256) break;                       // one candidate only
        cand = forced_n;
      }
      if (cand > n16) cand = n16 < 32 ? 32 : n16;   // a tile wider than the matrix only wastes columns
      const double c = tile_cost(M, N, int_kb + fp_kb, fp_kb > 0, ctas, cand, units);
      if (!have || c < best) {
        have = true;
        best = c;
        best_ctas = ctas;
        best_bn = cand;
      }
    }
  }
  *ctas_out = best_ctas;
  *bn_out = best_bn;
}

void set_tile_n(int n) { g_tile_n.store(n); }
int get_tile_n() { return g_tile_n.load(); }
void set_debug_counters(void *buf) { g_dbg.store(static_cast<unsigned long long *>(buf)); }
unsigned long long *get_debug_counters() { return g_dbg.load(); }
void set_l2_hint(int on) { g_l2_hint.store(on ? 1 : 0); }
int get_l2_hint() { return g_l2_hint.load(); }
void set_cta_pair(int mode) { g_cta_pair.store(mode); }
int get_cta_pair() { return g_cta_pair.load(); }

int device_status_read(int clear) {
  unsigned int v = 0;
  QUIK_CUDA_TRY(cudaDeviceSynchronize());
  QUIK_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_device_status, sizeof(v)));
  if (clear && v) {
    unsigned int z = 0;
    QUIK_CUDA_TRY(cudaMemcpyToSymbol(g_device_status, &z, sizeof(z)));
  }
  return v ? QUIK_ERR_DEVICE_WAIT : QUIK_OK;
}

int launch_gemm_tcgen05(const int8_t *A, const int8_t *B, int M, int N, int K, const Epilogue &ep,
                        cudaStream_t st) {
  if (M == 0 || N == 0) return QUIK_OK;
  if (K % 16 != 0 || K <= 0) return QUIK_ERR_SHAPE;
  if (!aligned16(A) || !aligned16(B)) return QUIK_ERR_ALIGN;
  const bool has_fp = ep.mode == 1 && ep.fp_a != nullptr && ep.F > 0;
  if (ep.y != nullptr && (has_fp || ep.dtype != QUIK_F16)) return QUIK_ERR_UNSUPPORTED;      // no operator asks for it
  if (has_fp && (ep.F % 8 != 0 || !aligned16(ep.fp_a) || !aligned16(ep.fp_b))) return QUIK_ERR_ALIGN;

  GemmParams p{};
  p.int_kb = (K + STAGE_K_BYTES - 1) / STAGE_K_BYTES;
  p.fp_kb = has_fp ? (ep.F + 63) / 64 : 0;
  int ctas = 1, block_n = 128;
  choose_tile(M, N, p.int_kb, p.fp_kb, &ctas, &block_n);
  const int tile_m = BLOCK_M * ctas;
  const int m_tiles = (M + tile_m - 1) / tile_m;
  const int cap_n = block_n <= 128 ? 128 : 256;

  fill_epilogue_params(p, ep, M, N);
  if (p.status == nullptr) return QUIK_ERR_CUDA;
  p.block_n = block_n;
  p.split_n = split_columns(block_n, EPI_WARPS / 4);
  p.num_m_tiles = m_tiles;
  p.num_tiles = m_tiles * ((N + block_n - 1) / block_n);
  p.idesc_int = make_idesc(2, 1, tile_m, block_n);                              // S32 accumulate, signed 8-bit operands
  p.idesc_fp = make_idesc(1, ep.dtype == QUIK_BF16 ? 1 : 0, tile_m, block_n);   // F32 accumulate, F16 / BF16 operands
  p.l2_hint = g_l2_hint.load();

  CUtensorMap ta, tb, tfa, tfb;
  int rc;
  if ((rc = make_tmap(&ta, A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K, BLOCK_M)) != QUIK_OK) return rc;
  if ((rc = make_tmap(&tb, B, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K, block_n / ctas)) != QUIK_OK) return rc;
  if (has_fp) {
    const CUtensorMapDataType fdt = ep.dtype == QUIK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    if ((rc = make_tmap(&tfa, ep.fp_a, fdt, 2, M, ep.F, BLOCK_M)) != QUIK_OK) return rc;
    if ((rc = make_tmap(&tfb, ep.fp_b, fdt, 2, N, ep.F, block_n / ctas)) != QUIK_OK) return rc;
  } else {
    tfa = ta;
    tfb = tb;
  }
  // the result, where its rows allow bulk stores: boxes of 32 rows x 64 bytes
  CUtensorMap to = ta;
  if (p.vec_out) {
    if (ep.mode == 0) rc = make_tmap(&to, ep.C, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, M, N, 32, 64);
    else rc = make_tmap(&to, ep.out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, M, N, 32, 64, p.ldo);
    if (rc != QUIK_OK) return rc;
  }
#define QUIK_LAUNCH_R(T, K, C, R) \
  return cap_n == 256 ? launch_t<T, 256, K, C, R>(ta, tb, tfa, tfb, to, p, st) : launch_t<T, 128, K, C, R>(ta, tb, tfa, tfb, to, p, st)
#define QUIK_LAUNCH_C(T, K, C)                      \
  do {                                              \
    if (p.vec_out) QUIK_LAUNCH_R(T, K, C, ALIGNED); \
    QUIK_LAUNCH_R(T, K, C, UNALIGNED);              \
  } while (0)
#define QUIK_LAUNCH(T, K)                  \
  do {                                     \
    if (ctas == 2) QUIK_LAUNCH_C(T, K, 2); \
    QUIK_LAUNCH_C(T, K, 1);                \
  } while (0)
  if (ep.mode == 0) QUIK_LAUNCH(__half, 0);
  if (ep.dtype == QUIK_BF16) {
    if (has_fp) QUIK_LAUNCH(__nv_bfloat16, 2);
    QUIK_LAUNCH(__nv_bfloat16, 1);
  }
  if (has_fp) QUIK_LAUNCH(__half, 2);
  if (ep.y) QUIK_LAUNCH(__half, 3);
  QUIK_LAUNCH(__half, 1);
#undef QUIK_LAUNCH_R
#undef QUIK_LAUNCH_C
#undef QUIK_LAUNCH
}

}  // namespace quik
