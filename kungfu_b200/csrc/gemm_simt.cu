// Generic matrix product  out[T, N] = x[T, K] . w[N, K]^T  with 32-bit FMA accumulation.
//
// This is the true 32-bit product of the engine (no tensor-core or reduced-precision mode) and the
// fallback for shapes and types the tensor-core kernel refuses.  Any T, N, K.  The order of an output's sum is
// fixed by (N, K) alone, so a row's result does not depend on T or on which other rows share the launch.
// `fma_tile_kernel` where both operands are 32-bit; `gemm_simt_kernel` (64 x 64 tiles, k ascending in one thread) for
// bfloat16 operands; `cols_kernel`, with the same bits, for a few 32-bit rows of a short K on bfloat16 weights.  Reference counterpart: the 32x64x64 shared-tile product in
// crates/kf-backend-cuda/src/kernels/quant.cuh:110-171.
#include "common.cuh"
#include <type_traits>

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TX, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TO* __restrict__ out,
                 int T, int N, int K, float softcap, long ldx) {
  kf_pdl_trigger();
  kf_pdl_wait();
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
  const int lr = tid >> 2, lk = (tid & 3) * 4;          // this thread loads row lr, k = lk..lk+3 of each tile
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    {
      const int r = row0 + lr;
      const TX* p = x + (size_t)r * ldx + k0 + lk;
#pragma unroll
      for (int u = 0; u < 4; ++u) xs[lk + u][lr] = (r < T && k0 + lk + u < K) ? kf_load(p, u) : 0.f;
      const int c = col0 + lr;
      const TW* q = w + (size_t)c * K + k0 + lk;
#pragma unroll
      for (int u = 0; u < 4; ++u) ws[lk + u][lr] = (c < N && k0 + lk + u < K) ? kf_load(q, u) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = row0 + ty * 4 + i;
    if (r >= T) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = col0 + tx * 4 + j;
      if (c < N) kf_store(out, (size_t)r * N + c, kf_softcap(acc[i][j], softcap));
    }
  }
}

// ---- both operands 32-bit ------------------------------------------------------------------------------------------------
// A block of 128 threads owns MT rows x 128 features.  Few rows are bound by the weights' bytes, many by the FMA pipe:
//   * tiles of 32 k of both operands travel through a ring of 16-byte cp.async copies (4-byte ones where a row's pitch or
//     base is not a multiple of 16 bytes), rows 144 bytes apart in shared memory, so that the eight rows that a quarter of
//     a warp reads 16 bytes of lie in different banks and nothing has to be transposed on the way in;
//   * a thread multiplies TM x TN outputs, each as a pair of sums over the even and the odd k: the packed FMA
//     (fma.rn.f32x2) takes two neighbouring k of both operands straight from those 16 bytes, which is two FMAs an issue
//     slot and 16 shared-memory loads for 256 of them at 8 x 8 outputs;
//   * MT = 1..8 rows (one feature a thread), 16, 32 or 64, so that a decode step does not multiply padding;
//   * K is cut into a cluster of up to eight blocks where the features alone leave SMs idle; the partial tiles meet in
//     shared memory in the order of the parts.  The cut depends on (N, K) only.
// Measured alone with a cold L2 (one B200), the generic kernel -> this one, error against 64 bits (2-norms) below:
//   18,432 x 2,304: 1 row 238 -> 47 us (3.6 TB/s), 64 rows 254 -> 140, 167 rows 756 -> 382, 2,048 rows 6.71 -> 3.81 ms (46 TFLOP/s)
//   2,304 x 9,216:  1 row 698 -> 33 us (2.6 TB/s), 64 rows 713 -> 133, 167 rows 668 -> 250, 2,048 rows 3.43 -> 2.08 ms
//   256,000 x 2,304: 1 row 2.54 -> 0.41 ms (5.8 TB/s);   error at K = 9,216 1.7e-6 -> 4.3e-7, at K = 2,304 8.6e-7 -> 2.2e-7 to 4.3e-7
constexpr int FN = 128, FK = 32, FLD = FK + 4, FTHREADS = 128;

template <int MT>
struct FmaShape {
  static constexpr int TM = MT < 8 ? MT : 8;
  static constexpr int ROWS = MT / TM;                      // threads along the rows
  static constexpr int COLS = FTHREADS / ROWS;              // and along the features
  static constexpr int TN = FN / COLS;
  static constexpr int STAGES = MT >= 32 ? 3 : 4;
  static constexpr int STAGE = (MT + FN) * FLD;             // floats
  static constexpr int RED_LD = FN + 8;
  static constexpr size_t SMEM = sizeof(float) * (STAGES * STAGE > MT * RED_LD ? STAGES * STAGE : MT * RED_LD);
};

__device__ __forceinline__ void fma_pair(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
template <bool VEC>
__device__ __forceinline__ void copy_chunk(float* dst, const float* src, int left) {      // left: valid floats from src on
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (VEC) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(left > 0 ? 16 : 0) : "memory");
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * u), "l"(left > u ? src + u : src), "r"(left > u ? 4 : 0) : "memory");
  }
}

template <int MT, bool VEC, typename TO>
__global__ void __launch_bounds__(FTHREADS, MT >= 64 ? 2 : 1)
fma_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, TO* __restrict__ out, int T, int N, int K,
                float softcap, long ldx, int splits) {
  using S = FmaShape<MT>;
  constexpr int TM = S::TM, TN = S::TN, ROWS = S::ROWS, COLS = S::COLS;
  kf_pdl_trigger();
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int z = blockIdx.x % splits;                        // the part of K; the blocks of a cluster are neighbours in x
  const int row0 = (blockIdx.x / splits) * MT, col0 = blockIdx.y * FN;
  const int tiles = (K + FK - 1) / FK, per = (tiles + splits - 1) / splits;
  const int first = z * per, n = max(0, min(tiles, first + per) - first);
  // which rows and features are this thread's: ty + ROWS * i, tx + COLS * j
  const int tx = MT >= 64 ? (lane & 7) + 8 * (warp & 1) : MT >= 32 ? (lane & 7) + 8 * warp : MT >= 16 ? (lane & 15) + 16 * warp : tid;
  const int ty = MT >= 64 ? (lane >> 3) + 4 * (warp >> 1) : MT >= 32 ? lane >> 3 : MT >= 16 ? lane >> 4 : 0;

  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  const int cr = tid >> 3, cc = (tid & 7) * 4;              // this thread copies 4 floats at column cc of rows cr, cr + 16, ...
  auto request = [&](int i) {
    if (i < n) {
      const int k = (first + i) * FK + cc;
      const int left = K - k;
      float* xs = sm + (i % S::STAGES) * S::STAGE;
      float* ws = xs + MT * FLD;
#pragma unroll
      for (int r = 0; r < FN; r += 16) {
        const int f = col0 + r + cr;
        const bool in = f < N && left > 0;
        copy_chunk<VEC>(ws + (r + cr) * FLD + cc, in ? w + (size_t)f * K + k : w, in ? left : 0);
      }
#pragma unroll
      for (int r = 0; r < MT; r += 16) {
        if (MT >= 16 || cr < MT) {
          const int t = row0 + r + cr;
          const bool in = t < T && left > 0;
          copy_chunk<VEC>(xs + (r + cr) * FLD + cc, in ? x + (size_t)t * ldx + k : x, in ? left : 0);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  kf_pdl_wait();
#pragma unroll
  for (int i = 0; i < S::STAGES - 1; ++i) request(i);
  for (int i = 0; i < n; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S::STAGES - 2) : "memory");
    __syncthreads();                                        // tile i is there, and everybody is done with tile i - 1
    request(i + S::STAGES - 1);
    const float* xs = sm + (i % S::STAGES) * S::STAGE + ty * FLD;
    const float* ws = sm + (i % S::STAGES) * S::STAGE + (MT + tx) * FLD;
#pragma unroll
    for (int k = 0; k < FK; k += 4) {
      ulonglong2 a[TM];
#pragma unroll
      for (int r = 0; r < TM; ++r) a[r] = *reinterpret_cast<const ulonglong2*>(xs + r * ROWS * FLD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + j * COLS * FLD + k);
#pragma unroll
        for (int r = 0; r < TM; ++r) fma_pair(acc[r][j], a[r].x, b.x);
#pragma unroll
        for (int r = 0; r < TM; ++r) fma_pair(acc[r][j], a[r].y, b.y);
      }
    }
  }

  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                          // the ring is free: it holds the block's partial tile now
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      sm[(ty + ROWS * i) * S::RED_LD + tx + COLS * j] =
          __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
  if (splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  // block z of the cluster sums the features [z * FN / splits, (z + 1) * FN / splits) of every row
  const int share = FN / splits;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  for (int e = tid; e < MT * share; e += FTHREADS) {
    const int r = e / share, c = z * share + e % share;
    const int t = row0 + r, f = col0 + c;
    if (t >= T || f >= N) continue;
    float v = 0.f;
    if (splits > 1) {
      float part[8];
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        part[p] = 0.f;
        if (p < splits) {
          uint32_t remote;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(base + 4u * (r * S::RED_LD + c)), "r"(p));
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[p]) : "r"(remote) : "memory");
        }
      }
      v = part[0];
#pragma unroll
      for (int p = 1; p < 8; ++p) if (p < splits) v += part[p];
    } else {
      v = sm[r * S::RED_LD + c];
    }
    kf_store(out, (size_t)t * N + f, kf_softcap(v, softcap));
  }
  if (splits > 1) {                                         // nobody leaves while a peer reads its shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// How many ways K is cut: until the feature tiles times the parts are about two blocks per SM, each part 256 k or more.
// A function of the weights' shape alone, so that a row's sum has the same order in every launch.
static int fma_splits(int N, int K) {
  int s = 1;
  while (s < 8 && (long)kf_ceil_div(N, FN) * s < 256 && K / (2 * s) >= 256) s *= 2;
  return s;
}

template <int MT, bool VEC, typename TO>
static int launch_fma(const float* x, const float* w, TO* out, int T, int N, int K, float softcap, long ldx, cudaStream_t s) {
  using S = FmaShape<MT>;
  auto kernel = fma_tile_kernel<MT, VEC, TO>;
  const cudaError_t e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (e != cudaSuccess) { kf_record_cuda_error(e); return KF_ERR_SETUP; }
  const int splits = fma_splits(N, K);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kf_ceil_div(T, MT) * splits, kf_ceil_div(N, FN));
  cfg.blockDim = dim3(FTHREADS);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (kf_pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = splits;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, kernel, x, w, out, T, N, K, softcap, ldx, splits);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

template <bool VEC, typename TO>
static int launch_fma_rows(const float* x, const float* w, TO* out, int T, int N, int K, float softcap, long ldx, cudaStream_t s) {
  if (T <= 1) return launch_fma<1, VEC>(x, w, out, T, N, K, softcap, ldx, s);
  if (T <= 2) return launch_fma<2, VEC>(x, w, out, T, N, K, softcap, ldx, s);
  if (T <= 4) return launch_fma<4, VEC>(x, w, out, T, N, K, softcap, ldx, s);
  if (T <= 8) return launch_fma<8, VEC>(x, w, out, T, N, K, softcap, ldx, s);
  if (T <= 16) return launch_fma<16, VEC>(x, w, out, T, N, K, softcap, ldx, s);
  if (T <= 32) return launch_fma<32, VEC>(x, w, out, T, N, K, softcap, ldx, s);
  return launch_fma<64, VEC>(x, w, out, T, N, K, softcap, ldx, s);
}

constexpr long MAX_GRID_Y = 65535;

template <typename TO>
static int launch_fma_any(const float* x, const float* w, TO* out, int T, int N, int K, float softcap, long ldx, cudaStream_t s) {
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  return vec ? launch_fma_rows<true>(x, w, out, T, N, K, softcap, ldx, s) : launch_fma_rows<false>(x, w, out, T, N, K, softcap, ldx, s);
}

// 32-bit rows x bfloat16 weights of few k and few rows (the second halves of factored projections in a decode step): bound by
// latency.  A thread owns a feature and two rows, its weights (at most 8 KV) requested before the grid dependency is waited
// for and held in registers, the rows in shared memory; k ascending, so the bits are those of `gemm_simt_kernel`.
// 2,048 features of 64 k at 8 rows, in place: 5.9 -> 2.5 us.
constexpr int CF = 32, CR = 8;

template <int KV, typename TO>
__global__ void __launch_bounds__(128)
cols_kernel(const float* x, const __nv_bfloat16* __restrict__ w, TO* __restrict__ out, int T, int N, int K, float softcap, long ldx) {
  kf_pdl_trigger();
  __shared__ __align__(16) float xs[CR][8 * KV];
  const int tid = threadIdx.x, f = blockIdx.x * CF + (tid & 31), r0 = blockIdx.y * CR, rg = 2 * (tid >> 5);
  uint4 wv[KV];
#pragma unroll
  for (int c = 0; c < KV; ++c)
    wv[c] = f < N && 8 * c < K ? *reinterpret_cast<const uint4*>(w + (size_t)f * K + 8 * c) : make_uint4(0u, 0u, 0u, 0u);
  kf_pdl_wait();
  x = kf_produced(x);
  for (int i = tid; i < CR * (K / 4); i += 128) {
    const int r = i / (K / 4), c = 4 * (i - r * (K / 4));
    *reinterpret_cast<float4*>(&xs[r][c]) = r0 + r < T ? *reinterpret_cast<const float4*>(x + (size_t)(r0 + r) * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  float acc[2] = {0.f, 0.f};
#pragma unroll
  for (int c = 0; c < KV; ++c) {
    if (8 * c >= K) break;
    const uint32_t u[4] = {wv[c].x, wv[c].y, wv[c].z, wv[c].w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float v = __uint_as_float(e & 1 ? u[e >> 1] & 0xffff0000u : u[e >> 1] << 16);
#pragma unroll
      for (int r = 0; r < 2; ++r) acc[r] = fmaf(xs[rg + r][8 * c + e], v, acc[r]);
    }
  }
  if (f >= N) return;
#pragma unroll
  for (int r = 0; r < 2; ++r)
    if (r0 + rg + r < T) kf_store(out, (size_t)(r0 + rg + r) * N + f, kf_softcap(acc[r], softcap));
}

template <typename TO>
static int launch_cols(const float* x, const __nv_bfloat16* w, TO* out, int T, int N, int K, float softcap, long ldx, cudaStream_t s) {
  const dim3 grid(kf_ceil_div(N, CF), kf_ceil_div(T, CR));
  if (K <= 64) kf_launch(cols_kernel<8, TO>, grid, dim3(128), 0, s, x, w, out, T, N, K, softcap, ldx);
  else kf_launch(cols_kernel<16, TO>, grid, dim3(128), 0, s, x, w, out, T, N, K, softcap, ldx);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

template <typename TX, typename TW>
static int launch(const TX* x, const TW* w, void* out, int out_dtype, int T, int N, int K, float softcap, cudaStream_t s,
                  long ldx = 0) {
  if (ldx <= 0) ldx = K;
  // the tiled kernel counts feature tiles in the grid's y; wider outputs than 65,535 of them stay with the generic kernel
  if constexpr (std::is_same<TX, float>::value && std::is_same<TW, float>::value) {
    if (kf_ceil_div(N, FN) <= MAX_GRID_Y) {
      if (out_dtype == KF_F32) return launch_fma_any(x, w, (float*)out, T, N, K, softcap, ldx, s);
      if (out_dtype == KF_BF16) return launch_fma_any(x, w, (__nv_bfloat16*)out, T, N, K, softcap, ldx, s);
      return KF_ERR_DTYPE;
    }
  }
  // few rows of a short K: beyond 64 rows the tiles of the generic kernel are full, and above 128 k the weights of a thread
  // no longer fit its registers
  if constexpr (std::is_same<TX, float>::value && std::is_same<TW, __nv_bfloat16>::value) {
    if (T <= 64 && K <= 128 && K % 8 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
      if (out_dtype == KF_F32) return launch_cols(x, w, (float*)out, T, N, K, softcap, ldx, s);
      if (out_dtype == KF_BF16) return launch_cols(x, w, (__nv_bfloat16*)out, T, N, K, softcap, ldx, s);
      return KF_ERR_DTYPE;
    }
  }
  dim3 grid(kf_ceil_div(N, BN), kf_ceil_div(T, BM));
  if (out_dtype == KF_F32)
    kf_launch(gemm_simt_kernel<TX, TW, float>, dim3(grid), dim3(256), 0, s, x, w, (float*)out, T, N, K, softcap, ldx);
  else if (out_dtype == KF_BF16)
    kf_launch(gemm_simt_kernel<TX, TW, __nv_bfloat16>, dim3(grid), dim3(256), 0, s, x, w, (__nv_bfloat16*)out, T, N, K, softcap, ldx);
  else
    return KF_ERR_DTYPE;
  KF_CHECK_LAUNCH();
  return KF_OK;
}

// softcap > 0 applies cap * tanh(v / cap) to every output element.
KF_API int kf_linear_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* out, int out_dtype,
                          int T, int N, int K, float softcap, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return KF_OK;
  if (K <= 0) return KF_ERR_SIZE;
  if (x_dtype == KF_F32 && w_dtype == KF_F32) return launch((const float*)x, (const float*)w, out, out_dtype, T, N, K, softcap, stream);
  if (x_dtype == KF_BF16 && w_dtype == KF_BF16) return launch((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, out_dtype, T, N, K, softcap, stream);
  if (x_dtype == KF_F32 && w_dtype == KF_BF16) return launch((const float*)x, (const __nv_bfloat16*)w, out, out_dtype, T, N, K, softcap, stream);
  if (x_dtype == KF_BF16 && w_dtype == KF_F32) return launch((const __nv_bfloat16*)x, (const float*)w, out, out_dtype, T, N, K, softcap, stream);
  return KF_ERR_DTYPE;
}

// The same product over a column range of a wider 32-bit matrix: x[t, k] = base[t * ldx + col0 + k].  The low-rank
// second halves of factored projections read their inputs this way, straight from the stacked projection's result.
KF_API int kf_linear_simt_cols(const float* base, long ldx, long col0, const void* w, int w_dtype, void* out, int out_dtype,
                               int T, int N, int K, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return KF_OK;
  if (K <= 0 || ldx < col0 + K) return KF_ERR_SIZE;
  if (w_dtype == KF_F32) return launch(base + col0, (const float*)w, out, out_dtype, T, N, K, 0.f, stream, ldx);
  if (w_dtype == KF_BF16) return launch(base + col0, (const __nv_bfloat16*)w, out, out_dtype, T, N, K, 0.f, stream, ldx);
  return KF_ERR_DTYPE;
}
