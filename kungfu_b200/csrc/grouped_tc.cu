// Products of a mixture's experts over many rows, on tcgen05:  out[r, n] = sum_k x[r, k] w[e(r)][n, k]  for the sorted pairs r
// of a plan (grouped.cu), bfloat16 operands, 32-bit accumulation; gated: gate and up rows of an expert in two accumulators.
//
// A block owns 128 features of an expert x up to 128 of its rows (two neighbouring tiles of the plan's list): weights are the
// MMA's A operand (128 lanes), rows its N (64 or 128), K in stages of 64 through a TMA ring, one tile per block; roles as in
// gemm_tc.cu.  Rows that are read through the plan (one row per token) are first copied in sorted order, which costs less
// than a row-wise gather in every feature tile.  What bounds it is what an SM takes in: 48 KB a stage for 2.1 M multiply-adds.
// 128 rows for each of 32 experts of 2,048 x 2,048, grouped.cu's kernel -> this one: gate and up 276 -> 118 us, down 133 -> 57 us.  Its results
// are those of grouped.cu's tensor-core kernels bit for bit.
#include "common.cuh"
#include "tc_common.cuh"

namespace {

using namespace kf_tc;

// A test can make the producer leave out the loads of every stage from this one on (-1: never); see kf_test_grouped_give_up.
static __device__ int g_test_drop_from_stage = -1;

constexpr int GT_ROWS = 128, GT_PLAN = 64;                      // rows of a block; of a tile of the plan

struct GroupedTc {
  const int* tile_group; const int* tile_row0; const int* tile_nrows; const int* n_tiles;
  const int* row_index; const float* row_scale;                 // gated: gate and up of sorted row r times row_scale[row_index[r]]
  void* out;
  int* error_flag;
  int N, K, silu, stages;
  float limit;
};

// dst[r] = src[index[r] / div]: rows of 16-byte chunks
__global__ void __launch_bounds__(256) sorted_rows_kernel(const uint4* src, const int* index, int div, uint4* dst, int rows, int chunks) {
  kf_pdl_trigger();
  kf_pdl_wait();
  const int r = blockIdx.x;
  const uint4* from = src + (size_t)(index[r] / div) * chunks;
  for (int i = threadIdx.x; i < chunks; i += 256) dst[(size_t)r * chunks + i] = from[i];
}

// Warps of the epilogue.  An activation is a chain of an exponential and a division, 0.16 us a row with one warp per scheduler, which
// nothing hides: gated products have four (the product above 168 -> 118 us, N = K = 512 of two experts of 192 rows 24 -> 13 us).
template <int GATED> constexpr int EPI_WARPS = GATED ? 16 : 4;

template <int GATED, typename TO>
__global__ void __launch_bounds__(64 + 32 * EPI_WARPS<GATED>)
grouped_tc_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ GroupedTc p) {
  constexpr int NACC = GATED ? 2 : 1, A_BYTES = BM * BK * 2, B_BYTES = GT_ROWS * BK * 2, STAGE = NACC * A_BYTES + B_BYTES;
  constexpr int TMEM = 128 * NACC;
  const int drop = g_test_drop_from_stage;                        // asked for while the kernels ahead finish
  kf_pdl_wait();                                                  // the plan and the rows come from them
  const int ti = blockIdx.y;
  if (ti >= *p.n_tiles) return;
  const int g = p.tile_group[ti];
  int first = ti;
  while (first > 0 && p.tile_group[first - 1] == g) --first;
  if ((ti - first) & 1) return;                                   // the second of two tiles
  const int r0 = p.tile_row0[ti];
  const bool pair = ti + 1 < *p.n_tiles && p.tile_group[ti + 1] == g;
  const int nrows = p.tile_nrows[ti] + (pair ? p.tile_nrows[ti + 1] : 0);
  const int f0 = blockIdx.x * BM, nkb = (p.K + BK - 1) / BK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + (size_t)p.stages * STAGE);
  uint64_t* empty = full + p.stages;
  uint64_t* acc_full = empty + p.stages;
  uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
  volatile int* s_abort = (volatile int*)(tmem_slot + 1);
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  kf_pdl_trigger();                                               // after the allocation (tc_common.cuh); a block that left counts as triggered
  const int bytes = NACC * A_BYTES + (pair ? B_BYTES : B_BYTES / 2);
  int issued = 0;                                                 // stages this thread has asked for (the producer's count)
  auto give_up = [&](int code) { record_error(p.error_flag, 48 + code); *s_abort = 1; __threadfence_block(); };

  if (warp == 0) {
    if (lane == 0) {
      const int w0 = g * NACC * p.N + f0;                         // the expert's gate rows, then its up rows
      int s = 0;
      uint32_t ph = 1;
      const int last = drop >= 0 && drop < nkb ? drop : nkb;
      for (; issued < last; ++issued) {
        if (!mbar_wait(&empty[s], ph)) { give_up(ERR_WAIT_EMPTY); break; }
        const int i = issued;
        uint8_t* st = smem + (size_t)s * STAGE;
        mbar_expect_tx(&full[s], bytes);
        tma_load_2d(st, &tm_w, &full[s], i * BK, w0);
        if (GATED) tma_load_2d(st + A_BYTES, &tm_w, &full[s], i * BK, w0 + p.N);
        tma_load_2d(st + NACC * A_BYTES, &tm_x, &full[s], i * BK, r0);
        if (pair) tma_load_2d(st + NACC * A_BYTES + B_BYTES / 2, &tm_x, &full[s], i * BK, r0 + GT_PLAN);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc(pair ? GT_ROWS : GT_PLAN);
      const uint64_t da0 = umma_desc(smem), du0 = umma_desc(smem + A_BYTES), db0 = umma_desc(smem + NACC * A_BYTES);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait(&full[s], ph)) { give_up(ERR_WAIT_FULL); break; }
        const uint64_t so = (uint64_t)((uint32_t)s * (uint32_t)(STAGE >> 4));
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          umma(tmem, da0 + so + 2 * k, db0 + so + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
          if (GATED) umma(tmem + GT_ROWS, du0 + so + 2 * k, db0 + so + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&empty[s]);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      }
      umma_commit(acc_full);
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, f = f0 + quarter * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const bool ok = mbar_wait(acc_full, 0, 2) && !*s_abort;
    if (!ok && lane == 0) give_up(ERR_WAIT_ACC);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (__all_sync(0xffffffffu, ok)) {
      TO* out = (TO*)p.out + (size_t)r0 * p.N + f;
      for (int c0 = (warp - 2) / 4 * 16; c0 < nrows; c0 += EPI_WARPS<GATED> / 4 * 16) {
        float v[16], u[16];
        tmem_ld16(lane_addr + c0, v);
        if (GATED) {
          tmem_ld16(lane_addr + GT_ROWS + c0, u);
          if (p.row_scale)
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int r = r0 + min(c0 + j, nrows - 1);
              const float rs = p.row_scale[p.row_index ? p.row_index[r] : r];
              v[j] *= rs, u[j] *= rs;
            }
          if (p.silu) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = v[j] / (1.f + expf(-v[j])) * u[j];
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = kf_clamped_swish(v[j], u[j], p.limit);
          }
        }
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c0 + j < nrows && f < p.N) kf_store(out, (size_t)(c0 + j) * p.N, v[j]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // After a wait that ran out: loads that nobody waited for have landed before this block's shared memory becomes another's.
  if (threadIdx.x == 0 && *s_abort)
    for (int i = max(0, issued - p.stages); i < issued; ++i) mbar_wait(&full[i % p.stages], (uint32_t)(i / p.stages) & 1);
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM) : "memory");
  }
}

template <int GATED, typename TO>
int launch(const CUtensorMap& tw, const CUtensorMap& tx, GroupedTc p, int max_tiles, cudaStream_t s) {
  constexpr int STAGE = (GATED ? 2 : 1) * BM * BK * 2 + GT_ROWS * BK * 2;
  p.stages = GATED ? 4 : 3;                                       // gated: one block per SM; otherwise two, of 96 KB
  const size_t smem = (size_t)p.stages * STAGE + 1024 + 256;
  auto kernel = grouped_tc_kernel<GATED, TO>;
  static bool configured = false;                                 // per instantiation
  if (!configured) {
    if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      kf_record_cuda_error(cudaGetLastError());
      return KF_ERR_SETUP;
    }
    configured = true;
  }
  kf_launch(kernel, dim3(kf_ceil_div(p.N, BM), max_tiles), dim3(64 + 32 * EPI_WARPS<GATED>), smem, s, tw, tx, p);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

}  // namespace

// Whether this kernel takes a mixture's product: `pairs` rows over `groups` experts of [NW, K] bfloat16 weights, one behind the
// other.  From 64 rows an expert on average: below, the weights' bytes bound the product and the kernels of grouped.cu, which
// read only the experts and rows that exist, are the better ones.
KF_API int kf_grouped_tc_supported(const void* x, const void* w, long pairs, int groups, int N, int K) {
  return pairs >= 64l * groups && N >= 128 && K > 0 && K % 8 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 && tensor_maps_available();
}

// Whether it is also the faster one for these sizes.  A short K does not hide a block's start, the copy of gathered rows and the gated epilogue.
// Against grouped.cu's kernels, times here over times there at 64 to 320 rows for each of 2 to 96 experts, evenly spread and on a third of the
// experts: gathered and gated, K 256 0.6 to 2.0, 512 0.5 to 1.5, 768 0.4 to 1.0 from 384 features on (below to 1.2), 1,536 0.3 to 1.0 at any N; one of
// the two, 768 0.4 to 0.9 (to 1.2); neither, K 64 0.6 to 1.3, 128 0.5 to 1.2, 256 0.4 to 0.9.
KF_API int kf_grouped_tc_pays(int gathered, int gated, int N, int K) {
  return K >= (gathered || gated ? (N >= 384 ? 768 : 1536) : 256);
}

// x: [pairs, K], or with row_index one row per row_index[r] / row_div, copied to `sorted` [pairs, K] first.  gated: 0, 1 (the
// clamped form with `limit`) or 2 (silu(gate) * up), w [groups, 2N, K] then, else [groups, N, K].  out [pairs, N].
KF_API int kf_grouped_tc(const void* x, const int* row_index, int row_div, void* sorted, const void* w, void* out, int out_dtype,
                         const int* tile_group, const int* tile_row0, const int* tile_nrows, const int* n_tiles, int max_tiles,
                         int groups, int pairs, int N, int K, int gated, float limit, const float* row_scale, int* error_flag,
                         cudaStream_t stream) {
  if (pairs <= 0) return KF_OK;
  if (!kf_grouped_tc_supported(x, w, pairs, groups, N, K) || max_tiles < 1 || max_tiles > 65535 || (row_index && (!sorted || row_div < 1))) return KF_ERR_SIZE;
  if (row_index) {
    kf_launch(sorted_rows_kernel, dim3(pairs), dim3(256), 0, stream, (const uint4*)x, row_index, row_div, (uint4*)sorted, pairs, K / 8);
    KF_CHECK_LAUNCH();
    x = sorted;
  }
  CUtensorMap tw, tx;
  if (!tensor_map(w, (long)groups * (gated ? 2 : 1) * N, K, BM, &tw) || !tensor_map(x, pairs, K, GT_PLAN, &tx)) return KF_ERR_SETUP;
  const GroupedTc p{tile_group, tile_row0, tile_nrows, n_tiles, row_index, row_scale, out, error_flag, N, K, gated == 2, 0, limit};
  if (out_dtype == KF_BF16) return gated ? launch<1, __nv_bfloat16>(tw, tx, p, max_tiles, stream) : launch<0, __nv_bfloat16>(tw, tx, p, max_tiles, stream);
  if (out_dtype == KF_F32) return gated ? launch<1, float>(tw, tx, p, max_tiles, stream) : launch<0, float>(tw, tx, p, max_tiles, stream);
  return KF_ERR_DTYPE;
}

// For tests: as kf_test_gemm_give_up, for the experts' kernel.
KF_API int kf_test_grouped_give_up(unsigned long long limit_ns, int drop_from_stage) {
  const unsigned long long lim = limit_ns ? limit_ns : WAIT_LIMIT_NS;
  if (cudaMemcpyToSymbol(g_wait_limit_ns, &lim, sizeof(lim)) != cudaSuccess ||
      cudaMemcpyToSymbol(g_test_drop_from_stage, &drop_from_stage, sizeof(int)) != cudaSuccess) {
    kf_record_cuda_error(cudaGetLastError());
    return KF_ERR_SETUP;
  }
  return KF_OK;
}
