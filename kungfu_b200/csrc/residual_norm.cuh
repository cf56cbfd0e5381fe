// A row of the 32-bit residual stream is updated by a branch and, in the same pass, normed for what reads it next:
//   NORMED   x += rmsnorm(a) * g1          (post-norm, then the residual)
//   SCALED   x += a * g1                   (a factor per column)
//   PLAIN    x += a + b                    (branches side by side; b may be absent)
//   out = rmsnorm(x) * g2 (plus2 == 2: x as it is), copy = x, each in its own type, when asked for.
// One block per row, the row in registers as 16-byte vectors, so that every number is read and written once.  The gains do
// not depend on earlier kernels and are requested before the grid dependency is waited for; a and x at once after it; each
// sum costs one barrier (every warp adds the warps' sums itself).
// The kernel is bound by latency at a few rows and by bytes at many.  A few rows (`kf_residual_norm_threads`) take a thread
// per vector; many rows take four vectors a thread, so that an SM holds six or more rows at different stages of this chain
// where eight rows of two blocks, in step with one another, left the memory idle in turns.  The order of a row's sums is a
// function of H alone (`kf_row_sum`): a row has the same bits whatever else is in the step.
// Measured in place (one B200), the kernels it took the place of -> this one: NORMED at 2,048 rows of 2,304 20 -> 14 us
// (66 MB: 4.9 TB/s), SCALED at 8 rows of 2,048 4.5 -> 1.8 us, PLAIN at 8 rows 4.9 -> 2.1 us and at 2,048 rows 19 -> 14 us.
// The one order of the sums costs 0.4 us at 2,048 rows and 0.1 us at 512 in a chain of such kernels (8.9 -> 9.3 us); vectors dealt
// to the threads of a few rows so that both add up alike without exchanges cost those 0.35 us of 1.94 each.
#pragma once
#include "common.cuh"

enum KfResidualMode { KF_RES_NORMED = 0, KF_RES_SCALED = 1, KF_RES_PLAIN = 2 };

// four consecutive gains as they lie in memory, and their values
template <typename TW> struct KfRaw4;
template <> struct KfRaw4<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ float4 get() const { return v; }
};
template <> struct KfRaw4<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ float4 get() const {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
  }
};

__device__ __forceinline__ void kf_put4(float* o, float4 v) { *reinterpret_cast<float4*>(o) = v; }
__device__ __forceinline__ void kf_put4(__nv_bfloat16* o, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(o) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

__device__ __forceinline__ float kf_square4(float4 v) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x))); }

// The block's sum of a row of which thread t holds vectors t, t + blockDim.x, ...: part[k] is what vector t + k * blockDim.x
// adds.  In every thread; `red` holds 32 floats and is used for one sum only.  SHORT: at most 1,024 vectors; their sum has one
// order for both thread counts: 32 neighbouring vectors as a tree, then those sums as another.  With four vectors a thread (256 threads
// at most) a warp makes its four trees together: lanes 8 k .. 8 k + 7 go on with tree k after two exchanges.  Rows of more
// vectors always have four a thread, which are added first.
template <int NV, bool SHORT>
__device__ __forceinline__ float kf_row_sum(const float (&part)[NV], float* red) {
  static_assert(NV == 1 || NV == 4, "a vector per thread or four");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int n = blockDim.x >> 5;
  if (NV == 4 && SHORT) {
    const bool h16 = lane & 16, h8 = lane & 8;
    const float a = (h16 ? part[NV / 2] : part[0]) + __shfl_xor_sync(0xffffffffu, h16 ? part[0] : part[NV / 2], 16);
    const float b = (h16 ? part[NV - 1] : part[NV / 4]) + __shfl_xor_sync(0xffffffffu, h16 ? part[NV / 4] : part[NV - 1], 16);
    float v = (h8 ? b : a) + __shfl_xor_sync(0xffffffffu, h8 ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((lane & 7) == 0) red[warp + (lane >> 3) * n] = v;
    n *= 4;
  } else {
    float v = part[0];
#pragma unroll
    for (int k = 1; k < NV; ++k) v += part[k];
    v = kf_warp_sum(v);
    if (lane == 0) red[warp] = v;
  }
  __syncthreads();
  return kf_warp_sum(lane < n ? red[lane] : 0.f);
}

template <int MODE, typename TW1, typename TW2, typename TO, int NV, int MAXT>
__global__ void __launch_bounds__(MAXT)
residual_norm_kernel(const float* a, const float* b, const TW1* __restrict__ w1, float eps1, int plus1, float* x,
                     const TW2* __restrict__ w2, float eps2, int plus2, TO* __restrict__ out, TO* __restrict__ copy, int H) {
  kf_pdl_trigger();
  __shared__ float red1[32], red2[32];
  KfRaw4<TW1> r1[NV];
  KfRaw4<TW2> r2[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    if (i < H && MODE != KF_RES_PLAIN) r1[k].load(w1 + i);
    if (i < H && out != nullptr && plus2 != 2) r2[k].load(w2 + i);
  }
  kf_pdl_wait();
  a = kf_produced(a), b = kf_produced(b), x = kf_produced(x);
  const size_t base = (size_t)blockIdx.x * H;
  float4 v[NV], xv[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    v[k] = i < H ? *reinterpret_cast<const float4*>(a + base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    xv[k] = i < H ? *reinterpret_cast<const float4*>(x + base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (MODE == KF_RES_PLAIN && b != nullptr) {
    float4 u[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = 4 * (threadIdx.x + k * blockDim.x);
      u[k] = i < H ? *reinterpret_cast<const float4*>(b + base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k].x += u[k].x, v[k].y += u[k].y, v[k].z += u[k].z, v[k].w += u[k].w;
  }
  float inv = 1.f;
  if (MODE == KF_RES_NORMED) {
    float ss[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) ss[k] = kf_square4(v[k]);
    inv = 1.f / sqrtf(kf_row_sum<NV, NV == 1 || MAXT == 256>(ss, red1) / (float)H + eps1);
  }
  const float p1 = plus1 ? 1.f : 0.f;
  float ss[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    ss[k] = 0.f;
    if (i < H) {
      if (MODE == KF_RES_PLAIN) {
        v[k] = make_float4(v[k].x + xv[k].x, v[k].y + xv[k].y, v[k].z + xv[k].z, v[k].w + xv[k].w);
      } else {
        const float4 g = r1[k].get();
        v[k] = make_float4(fmaf(v[k].x * inv, g.x + p1, xv[k].x), fmaf(v[k].y * inv, g.y + p1, xv[k].y),
                           fmaf(v[k].z * inv, g.z + p1, xv[k].z), fmaf(v[k].w * inv, g.w + p1, xv[k].w));
      }
      kf_put4(x + base + i, v[k]);
      if (copy != nullptr) kf_put4(copy + base + i, v[k]);
      ss[k] = kf_square4(v[k]);
    }
  }
  if (out == nullptr) return;
  const float inv2 = plus2 == 2 ? 1.f : 1.f / sqrtf(kf_row_sum<NV, NV == 1 || MAXT == 256>(ss, red2) / (float)H + eps2);
  const float p2 = plus2 ? 1.f : 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = 4 * (threadIdx.x + k * blockDim.x);
    if (i < H) {
      const float4 g = plus2 == 2 ? make_float4(0.f, 0.f, 0.f, 0.f) : r2[k].get();
      kf_put4(out + base + i, make_float4(v[k].x * inv2 * (g.x + p2), v[k].y * inv2 * (g.y + p2), v[k].z * inv2 * (g.z + p2), v[k].w * inv2 * (g.w + p2)));
    }
  }
}

// Whether the kernel takes these rows: whole vectors on 16-byte boundaries (gains on boundaries of four of their own), and a
// row within 1,024 threads of four vectors.
static inline bool kf_residual_norm_takes(const void* a, const void* b, const void* w1, int w1_size, const void* x, const void* w2,
                                          int w2_size, const void* out, const void* copy, int out_size, int H) {
  return H % 4 == 0 && H <= 16384 && (((uintptr_t)a | (uintptr_t)b | (uintptr_t)x) & 15) == 0 &&
         ((uintptr_t)w1 & (4 * w1_size - 1)) == 0 && ((uintptr_t)w2 & (4 * w2_size - 1)) == 0 &&
         (((uintptr_t)out | (uintptr_t)copy) & (4 * out_size - 1)) == 0;
}

// Threads of a row: a vector each below 256 rows, four each from there on, or where a row has more than 1,024 vectors.
static inline int kf_residual_norm_threads(int T, int H, int* vectors) {
  const int n = H / 4;
  const bool one = T < 256 && n <= 1024;
  *vectors = one ? 1 : 4;
  const int t = one ? n : (n + 3) / 4;
  return (t + 31) / 32 * 32;
}

template <int MODE, typename TW1, typename TW2, typename TO>
static void kf_launch_residual_norm(const float* a, const float* b, const TW1* w1, float eps1, int plus1, float* x, const TW2* w2,
                                    float eps2, int plus2, TO* out, TO* copy, int T, int H, cudaStream_t s) {
  int nv;
  const int threads = kf_residual_norm_threads(T, H, &nv);
  if (nv == 1)
    kf_launch(residual_norm_kernel<MODE, TW1, TW2, TO, 1, 1024>, dim3(T), dim3(threads), 0, s, a, b, w1, eps1, plus1, x, w2, eps2, plus2, out, copy, H);
  else if (threads <= 256)
    kf_launch(residual_norm_kernel<MODE, TW1, TW2, TO, 4, 256>, dim3(T), dim3(threads), 0, s, a, b, w1, eps1, plus1, x, w2, eps2, plus2, out, copy, H);
  else
    kf_launch(residual_norm_kernel<MODE, TW1, TW2, TO, 4, 1024>, dim3(T), dim3(threads), 0, s, a, b, w1, eps1, plus1, x, w2, eps2, plus2, out, copy, H);
}
