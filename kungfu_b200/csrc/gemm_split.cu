// Product of 32-bit operands on the 5th-generation tensor cores:  out[T, N] = x[T, K] . w[N, K]^T  at 32-bit precision.
//
// A 32-bit number is the exact sum of three bfloat16 ones (its significand cut after 8, 16 and 24 bits; bfloat16 has the same
// exponents), and a product of two bfloat16 numbers is exact in 32 bits.  With x = x1 + x2 + x3 and w = w1 + w2 + w3 the six
// products x1 w1, x1 w2, x2 w1, x2 w2, x1 w3, x3 w1 hold all but 2^-21 of x w (the other three are left out).  What a
// tensor core adds up it may cut off instead of rounding, so an accumulator lives for 64 k only, and products of one size share
// one (x1 w1; x1 w2 + x2 w1; the other three); the sums are added in registers, rounded to nearest.
//
// Shape of the kernel (gemm_split_kernel): weights are the MMA's A operand (128 features = 128 lanes), rows of x its N.
//   warp 0      TMA: weights as they are, 128 x 64 floats a stage, and the three planes of x (cut by `split_rows_kernel`; up to
//               16 rows the summing warps cut x themselves, into shared memory, two chunks ahead)
//   warps 2-9   read the weights of a stage, cut them in registers and put the three planes into tensor memory (the MMA
//               takes A from there), so that the weights cross the memory system once, in 32 bits, and no copy is kept
//   warp 1      12 MMAs a chunk: the planes of x lie behind one another in shared memory as the accumulators do in tensor memory,
//               so that w1 meets all three planes of x in one MMA, w2 the first two and w3 the first.  An MMA with A in tensor
//               memory takes about 110 cycles however few rows it has, so their number is what counts
//   warps 10-.. add the finished accumulators to their sums in registers
// K is cut into parts (`split_parts`, from N and K alone) so that the feature tiles fill the SMs.  Up to 16 rows the parts of
// a tile are a cluster of CTAs, two of them to an SM, and meet in shared memory; beyond, a CTA walks (tile, part) units
// and leaves the parts' sums in memory for `sum_parts_kernel`.  Either way an output's sum is the chunks of a part in
// ascending k and the parts in ascending order, whatever T is, so a row does not depend on the rows beside it.
//
// A sum that is not finite, or below 2^-60 and not zero, is made again with plain FMAs by the thread that owns it: an infinity
// has no planes (its product with a plane of zeros would be NaN), and lower planes of numbers below 2^-110 leave bfloat16's range.
#include "common.cuh"
#include "tc_common.cuh"

namespace {

using namespace kf_tc;

constexpr int CK = 64;                                          // k of a chunk: the life of an accumulator
constexpr int W_STAGE = BM * CK * 4;                            // 32 KB: two boxes of 128 rows x 32 floats
constexpr int A_COLS = 3 * CK / 2;                              // tensor-memory columns of a chunk's three weight planes
constexpr int CUTTERS = 256;                                    // threads that cut weights: two per feature
constexpr int SMALL_T = 16, LARGE_T = 80;                      // rows of a tile, at most

__device__ __forceinline__ bool plain_needed(float v) { return !(fabsf(v) >= 8.67361738e-19f && fabsf(v) <= 3.4e38f) && v != 0.f; }   // 2^-60

// Two neighbours cut into three words of bfloat16 pairs; the cuts are exact.
__device__ __forceinline__ void cut_pair(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  p1 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
  a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
  p2 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
  a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
  p3 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// The three planes [3][T][pitch] of x [T, K], K a multiple of 4, zeros from K to the pitch.  A block per row.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* x, __nv_bfloat16* planes, int T, int K, int pitch) {
  kf_pdl_trigger();
  kf_pdl_wait();
  const int t = blockIdx.x;
  const float4* src = reinterpret_cast<const float4*>(x + (size_t)t * K);
#pragma unroll 4
  for (int i = threadIdx.x; i < pitch / 4; i += 256) {
    const float4 v = 4 * i < K ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    uint2 p[3];
    cut_pair(v.x, v.y, p[0].x, p[1].x, p[2].x);
    cut_pair(v.z, v.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(planes + ((size_t)j * T + t) * pitch + 4 * i) = p[j];
  }
}

__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t* r) {     // needs tcgen05.wait::ld before r is used
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}

__device__ __noinline__ float plain_sum(const float* x, const float* w, int n) {
  float v = 0.f;
  for (int i = 0; i < n; ++i) v = fmaf(x[i], w[i], v);
  return v;
}

// Whether the phase of this parity has completed, without waiting for it
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return done != 0;
}

struct SplitArgs {
  const float* x;
  const float* w;
  void* out;
  float* partial;                                                // [parts][T][N], where a launch leaves the parts' sums
  int* error_flag;
  float softcap;
  int T, N, K, parts, bn, w_stages;                              // bn: rows of a tile, a multiple of 16
};

// LARGE: a CTA per SM, up to 80 rows (the MMA takes 240), the sums in eight warps.  Otherwise two CTAs per SM, 16 rows, the sums in four.
template <bool LARGE>
struct SplitShape {
  static constexpr int MAX_T = LARGE ? LARGE_T : SMALL_T;
  static constexpr int SUM_GROUPS = LARGE ? 2 : 1;
  static constexpr int COLS = MAX_T / SUM_GROUPS;                // accumulator columns of a thread, at most
  static constexpr int BATCH = 8;                                // columns of every accumulator per wait on tensor memory
  static constexpr int THREADS_ = 64 + CUTTERS + 128 * SUM_GROUPS;
  static constexpr int TMEM = LARGE ? 512 : 256;
  static constexpr int X_STAGES = 2;
};
static_assert(2 * A_COLS + 3 * LARGE_T <= 512 && 3 * LARGE_T <= 256 && 2 * A_COLS + 3 * SMALL_T <= 256, "weight planes and accumulators fit tensor memory");

template <bool LARGE, typename TO>
__global__ void __launch_bounds__(SplitShape<LARGE>::THREADS_, LARGE ? 1 : 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ SplitArgs a) {
  using S = SplitShape<LARGE>;
  const int bn = LARGE ? a.bn : SMALL_T;
  const int ws = a.w_stages, x_stage = 3 * bn * CK * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sw = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sx = sw + (size_t)ws * W_STAGE;
  uint64_t* w_full = (uint64_t*)(sx + (size_t)S::X_STAGES * x_stage);
  uint64_t* w_empty = w_full + ws;
  uint64_t* x_full = w_empty + ws;
  uint64_t* x_empty = x_full + S::X_STAGES;
  uint64_t* a_full = x_empty + S::X_STAGES;                       // [2] weight planes of a chunk are in tensor memory
  uint64_t* done = a_full + 2;                                    // [2] its MMAs have ended
  uint64_t* acc_free = done + 2;                                  // [2] its accumulators have been read
  uint32_t* tmem_slot = (uint32_t*)(acc_free + 2);
  volatile int* s_abort = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (a.K + CK - 1) / CK;
  const int sets = 2 * A_COLS + 6 * bn <= S::TMEM ? 2 : 1;          // of accumulators, as tensor memory has room
  const int n_tt = (a.T + bn - 1) / bn, n_ft = (a.N + BM - 1) / BM;
  const int n_units = n_ft * n_tt * a.parts;                      // unit = ((feature tile) * n_tt + row tile) * parts + part

  if (threadIdx.x == 0) {
    for (int s = 0; s < ws; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], CUTTERS); }
    for (int s = 0; s < S::X_STAGES; ++s) { mbar_init(&x_full[s], LARGE ? 1 : 128); mbar_init(&x_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&a_full[b], CUTTERS); mbar_init(&done[b], 1); mbar_init(&acc_free[b], 128 * S::SUM_GROUPS); }
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(S::TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  kf_pdl_trigger();

  auto range = [&](int unit, int& first, int& last) {             // chunks of the unit's part
    const int z = unit % a.parts;
    first = (int)((long)z * chunks / a.parts);
    last = (int)((long)(z + 1) * chunks / a.parts);
  };
  auto give_up = [&](int code) { atomicExch(a.error_flag, 32 + code); *s_abort = 1; };

  if (warp == 0) {
    // ---- TMA: weights run ahead of x by as many stages as there are, and begin before the kernel ahead has ended ------------
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w) : "memory");
      if (LARGE) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_x) : "memory");
      auto load_w = [&](int unit, int c, int s) {
        const int f0 = unit / a.parts / n_tt * BM;
        mbar_expect_tx(&w_full[s], W_STAGE);
        tma_load_2d(sw + (size_t)s * W_STAGE, &tm_w, &w_full[s], c * CK, f0);
        tma_load_2d(sw + (size_t)s * W_STAGE + W_STAGE / 2, &tm_w, &w_full[s], c * CK + 32, f0);   // beyond K: zeros
      };
      // two walks over the same chunks, each as far ahead as its ring allows
      int wu = blockIdx.x, wc = 0, wl = 0, w_slot = 0, xu = blockIdx.x, xc = 0, xl = 0, x_slot = 0;
      uint32_t w_ph = 1, x_ph = 1;
      if (wu < n_units) { range(wu, wc, wl); xc = wc; xl = wl; }
      auto next_w = [&]() {
        load_w(wu, wc, w_slot);
        if (++w_slot == ws) { w_slot = 0; w_ph ^= 1; }
        if (++wc == wl) { wu += gridDim.x; if (wu < n_units) range(wu, wc, wl); }
      };
      for (int i = 0; i < ws && wu < n_units; ++i) next_w();      // the ring is empty: nothing to wait for
      if (!LARGE) {
        while (wu < n_units) {
          if (!mbar_wait(&w_empty[w_slot], w_ph)) { give_up(ERR_WAIT_EMPTY); break; }
          next_w();
        }
        xu = n_units;
      }
      if (LARGE) kf_pdl_wait();                                   // the planes of x come from the kernel ahead
      unsigned long long idle_since = 0;
      int idle = 0;
      while (xu < n_units) {                                      // the weights' walk is never behind
        if (mbar_test(&x_empty[x_slot], x_ph)) {
          const int t0 = (xu / a.parts % n_tt) * bn;
          mbar_expect_tx(&x_full[x_slot], x_stage);
          for (int p = 0; p < 3; ++p)
            tma_load_2d(sx + (size_t)x_slot * x_stage + (size_t)p * bn * CK * 2, &tm_x, &x_full[x_slot], xc * CK, p * a.T + t0);
          if (++x_slot == S::X_STAGES) { x_slot = 0; x_ph ^= 1; }
          if (++xc == xl) { xu += gridDim.x; if (xu < n_units) range(xu, xc, xl); }
          idle = 0;
        } else if (wu < n_units && mbar_test(&w_empty[w_slot], w_ph)) {
          next_w();
          idle = 0;
        } else if ((++idle & 255) == 0) {                         // bounded like every wait
          const unsigned long long now = global_ns();
          if (idle == 256) idle_since = now;
          else if (now - idle_since > g_wait_limit_ns) { give_up(ERR_WAIT_EMPTY); break; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMA issuer -------------------------------------------------------------------------------------------------------
    if (lane == 0) {
      const uint32_t idesc[3] = {umma_idesc(3 * bn), umma_idesc(2 * bn), umma_idesc(bn)};
      const uint64_t dx0 = umma_desc(sx);
      int c = 0, x_slot = 0;
      uint32_t x_ph = 0;
      bool ok = true;
      for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
        int first, last;
        range(unit, first, last);
        for (int i = first; i < last; ++i, ++c) {
          const int b = c & 1;
          if (!mbar_wait(&a_full[b], (uint32_t)(c >> 1) & 1) || !mbar_wait(&x_full[x_slot], x_ph) ||
              (c >= sets && !mbar_wait(&acc_free[c & (sets - 1)], (uint32_t)(c / sets - 1) & 1))) { give_up(ERR_WAIT_FULL); ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t wa = tmem + b * A_COLS, acc = tmem + 2 * A_COLS + (c & (sets - 1)) * 3 * bn;
          const uint64_t dx = dx0 + (uint64_t)((uint32_t)(x_slot * x_stage) >> 4);
#pragma unroll
          for (int k = 0; k < CK / UMMA_K; ++k)
#pragma unroll
            for (int q = 0; q < 3; ++q)                           // plane q of the weights, into the accumulators from number q on
              umma_ts(acc + q * bn, wa + q * (CK / 2) + k * (UMMA_K / 2), dx + 2 * k, idesc[q], (q > 0 || k > 0) ? 1u : 0u);
          umma_commit(&x_empty[x_slot]);
          umma_commit(&done[b]);
          if (++x_slot == S::X_STAGES) { x_slot = 0; x_ph ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp < 2 + CUTTERS / 32) {
    // ---- weights: two threads per feature, 32 k each at a time from shared memory into three planes of tensor memory ----------
    const int quarter = warp & 3, half = (warp - 2) >> 2, r = quarter * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    int c = 0, slot = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
      int first, last;
      range(unit, first, last);
      for (int i = first; i < last; ++i, ++c) {
        const int b = c & 1;
        ok = mbar_wait(&w_full[slot], ph) && (c < 2 || mbar_wait(&done[b], (uint32_t)((c >> 1) - 1) & 1)) && !*s_abort;
        if (!__all_sync(0xffffffffu, ok)) { if (lane == 0) give_up(ERR_WAIT_FULL); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint8_t* row = sw + (size_t)slot * W_STAGE + half * (W_STAGE / 2) + r * 128;
        const uint32_t dst = lane_addr + b * A_COLS + half * 16;
        uint32_t p1[16], p2[16], p3[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {                             // 16-byte piece j of a row stands at j ^ (row % 8)
          const float4 v = *reinterpret_cast<const float4*>(row + ((j ^ (r & 7)) << 4));
          cut_pair(v.x, v.y, p1[2 * j], p2[2 * j], p3[2 * j]);
          cut_pair(v.z, v.w, p1[2 * j + 1], p2[2 * j + 1], p3[2 * j + 1]);
        }
        tmem_st16(dst, p1);
        tmem_st16(dst + CK / 2, p2);
        tmem_st16(dst + CK, p3);
        mbar_arrive(&w_empty[slot]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(&a_full[b]);
        if (++slot == ws) { slot = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ---- sums: a thread per feature and a quarter of the rows (the small tile: all of them) --------------------------------------
    const int quarter = warp & 3, group = (warp - 2 - CUTTERS / 32) >> 2;
    const int fl = quarter * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const int cols = bn / S::SUM_GROUPS, col0 = group * cols;
    int c = 0;
    bool ok = true;
    kf_pdl_wait();                                                // before anything is written, and for x
    // The small tile: these 128 threads cut x.  Thread i has 4 floats at k 4 (i % 16) of rows i / 16 and i / 16 + 8; a chunk's
    // stage is its accumulator's number, free when its products are done; the next chunk's floats are on their way meanwhile.
    const int ct = threadIdx.x - 64 - CUTTERS, cj = ct & 15;
    int xu = blockIdx.x, xc = 0, xl = 0;
    float4 xv[2];
    auto ask_x = [&]() {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int t = (ct >> 4) + 8 * u, k = xc * CK + 4 * cj;
        xv[u] = xu < n_units && t < a.T && k < a.K ? *reinterpret_cast<const float4*>(a.x + (size_t)t * a.K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    auto cut_x = [&](int stage) {
      if (xu >= n_units) return;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int t = (ct >> 4) + 8 * u;
        uint2 q[3];
        cut_pair(xv[u].x, xv[u].y, q[0].x, q[1].x, q[2].x);
        cut_pair(xv[u].z, xv[u].w, q[0].y, q[1].y, q[2].y);
        uint8_t* dst = sx + (size_t)stage * x_stage + t * 128 + (((cj >> 1) ^ (t & 7)) << 4) + (cj & 1) * 8;
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(dst + e * (SMALL_T * CK * 2)) = q[e];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&x_full[stage]);
      if (++xc == xl) { xu += gridDim.x; if (xu < n_units) range(xu, xc, xl); }
      ask_x();
    };
    if (!LARGE) {
      if (xu < n_units) range(xu, xc, xl);
      ask_x();
      cut_x(0);
      cut_x(1);
    }
    for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
      int first, last;
      range(unit, first, last);
      float sum[S::COLS];
#pragma unroll
      for (int j = 0; j < S::COLS; ++j) sum[j] = 0.f;
      for (int i = first; i < last; ++i, ++c) {
        const int b = c & 1;
        ok = mbar_wait(&done[b], (uint32_t)(c >> 1) & 1) && !*s_abort;
        if (!__all_sync(0xffffffffu, ok)) { if (lane == 0) give_up(ERR_WAIT_ACC); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = lane_addr + 2 * A_COLS + (c & (sets - 1)) * 3 * bn + col0;
#pragma unroll
        for (int j0 = 0; j0 < S::COLS; j0 += S::BATCH) {
          if (j0 >= cols) break;
          uint32_t v[3][S::BATCH];
#pragma unroll
          for (int q = 0; q < 3; ++q) tmem_ld8_async(acc + q * bn + j0, v[q]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < S::BATCH; ++j) {
            asm volatile("" : "+r"(v[0][j]), "+r"(v[1][j]), "+r"(v[2][j]));      // not before the wait
            sum[j0 + j] += __uint_as_float(v[0][j]) + (__uint_as_float(v[1][j]) + __uint_as_float(v[2][j]));
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(&acc_free[c & (sets - 1)]);
        if (!LARGE) cut_x(b);                                     // for the chunk after next, while the next one's MMAs run
      }
      if (!ok) break;
      // ---- the unit's outputs: the parts of a product in a cluster through shared memory, else to memory -----------------------
      const int z = unit % a.parts, t0 = (unit / a.parts % n_tt) * bn, f = unit / a.parts / n_tt * BM + fl;
      const int k0 = first * CK, k1 = min(a.K, last * CK);
      const bool in_cluster = !LARGE && a.parts > 1;
      float* red = reinterpret_cast<float*>(sw);                  // [16][128]: the ring is free by then
      auto put = [&](int j, float v) {
        const int t = t0 + col0 + j;
        if (in_cluster) red[(col0 + j) * BM + fl] = v;
        else if (t < a.T && f < a.N) {
          if (a.parts > 1) a.partial[((size_t)z * a.T + t) * a.N + f] = v;
          else kf_store((TO*)a.out, (size_t)t * a.N + f, kf_softcap(v, a.softcap));
        }
      };
      unsigned long long again = 0ull;                            // columns whose sums are made again: rare
#pragma unroll
      for (int j = 0; j < S::COLS; ++j)
        if ((j & ~7) < cols) {
          put(j, sum[j]);
          if (plain_needed(sum[j])) again |= 1ull << j;
        }
      if (again && f < a.N) {
#pragma unroll 1
        for (int j = 0; j < cols; ++j)
          if ((again >> j & 1ull) && t0 + col0 + j < a.T)
            put(j, plain_sum(a.x + (size_t)(t0 + col0 + j) * a.K + k0, a.w + (size_t)f * a.K + k0, k1 - k0));
      }
    }
    __syncwarp();
  }
  if (!LARGE && a.parts > 1) {
    // ---- the cluster's parts: CTA z sums the rows t % parts == z out of its peers' shared memory, in the parts' order ---------
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int z = blockIdx.x % a.parts, f0 = blockIdx.x / a.parts * BM;
    if (warp >= 2 + CUTTERS / 32) {
      const int fl = threadIdx.x - 64 - CUTTERS, f = f0 + fl;
      const uint32_t red = smem_u32(sw);
      for (int t = z; t < min(a.T, SMALL_T); t += a.parts) {
        float part[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          part[p] = 0.f;
          if (p < a.parts) {
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(red + 4u * (uint32_t)(t * BM + fl)), "r"(p));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[p]) : "r"(remote) : "memory");
          }
        }
        float v = part[0];
#pragma unroll
        for (int p = 1; p < 8; ++p) if (p < a.parts) v += part[p];
        if (f < a.N && !*s_abort) kf_store((TO*)a.out, (size_t)t * a.N + f, kf_softcap(v, a.softcap));
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // nobody leaves while a peer reads its shared memory
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TMEM) : "memory");
  }
}

// out[i] = the parts' sums in ascending order, for outputs i of [T, N]
template <typename TO>
__global__ void __launch_bounds__(256)
sum_parts_kernel(const float* partial, TO* out, long n, int parts, float softcap) {
  kf_pdl_trigger();
  kf_pdl_wait();
  const long i = 4 * ((long)blockIdx.x * 256 + threadIdx.x);
  if (i + 3 < n && n % 4 == 0) {
    float4 v[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) if (p < parts) v[p] = __ldcs(reinterpret_cast<const float4*>(partial + p * n + i));
#pragma unroll
    for (int p = 1; p < 8; ++p)
      if (p < parts) { v[0].x += v[p].x; v[0].y += v[p].y; v[0].z += v[p].z; v[0].w += v[p].w; }
    const float r[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) kf_store(out, i + e, kf_softcap(r[e], softcap));
  } else {
    for (long e = i; e < min(i + 4, n); ++e) {
      float s = partial[e];
      for (int p = 1; p < parts; ++p) s += partial[p * n + e];
      kf_store(out, e, kf_softcap(s, softcap));
    }
  }
}

// Parts of K: as many (a power of two, at most eight) as give every SM of the GPU a (feature tile, part), each of four chunks
// or more.  From N and K alone: the order of an output's sum must not depend on T.
int split_parts(int N, int K) {
  const int chunks = kf_ceil_div(K, CK), tiles = kf_ceil_div(N, BM);
  int p = 1;
  while (p < 8 && (long)tiles * p * 2 <= 148 && chunks / (p * 2) >= 4) p *= 2;
  return p;
}

int split_pitch(int K) { return (K + 7) & ~7; }
long plane_floats(int T, int K) { return ((long)T * split_pitch(K) * 3 / 2 + 3) & ~3l; }

template <bool LARGE, typename TO>
int launch_split(const CUtensorMap& tw, const CUtensorMap& tx, SplitArgs a, cudaStream_t stream) {
  using S = SplitShape<LARGE>;
  constexpr size_t LIMIT = LARGE ? SMEM_LIMIT : 112 * 1024;       // two CTAs of the small one share an SM
  const size_t fixed = (size_t)S::X_STAGES * 3 * a.bn * CK * 2 + 1024 + 256;
  a.w_stages = (int)((LIMIT - fixed) / W_STAGE);
  if (a.w_stages > 6) a.w_stages = 6;
  const size_t smem = fixed + (size_t)a.w_stages * W_STAGE;
  auto kernel = gemm_split_kernel<LARGE, TO>;
  static bool configured = false;                                 // per instantiation
  if (!configured) {
    if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LIMIT) != cudaSuccess) {
      kf_record_cuda_error(cudaGetLastError());
      return KF_ERR_SETUP;
    }
    configured = true;
  }
  const bool cluster = !LARGE && a.parts > 1;
  const long units = (long)kf_ceil_div(a.N, BM) * kf_ceil_div(a.T, a.bn) * a.parts;
  const long resident = (long)kf_sm_count() * (LARGE ? 1 : 2);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(cluster || units < resident ? units : resident));   // in a cluster a CTA has one unit
  cfg.blockDim = dim3(S::THREADS_);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (kf_pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = a.parts;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, kernel, tw, tx, a);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

template <typename TO>
int linear_split(const float* x, const float* w, TO* out, int T, int N, int K, float softcap, float* scratch, int* error_flag,
                 cudaStream_t stream) {
  const int pitch = split_pitch(K);
  SplitArgs a = {};
  a.x = x, a.w = w, a.out = out, a.T = T, a.N = N, a.K = K, a.softcap = softcap, a.error_flag = error_flag;
  a.parts = split_parts(N, K);
  const bool large = T > SMALL_T;
  const int n_tt = kf_ceil_div(T, large ? LARGE_T : SMALL_T);
  a.bn = (kf_ceil_div(T, n_tt) + 15) & ~15;
  __nv_bfloat16* planes = (__nv_bfloat16*)scratch;
  a.partial = scratch + plane_floats(T, K);
  CUtensorMap tw, tx;
  if (!tensor_map_f32(w, N, K, BM, &tw)) return KF_ERR_SETUP;
  if (!large) return launch_split<false, TO>(tw, tw, a, stream);
  if (!tensor_map(planes, 3l * T, pitch, a.bn, &tx)) return KF_ERR_SETUP;
  kf_launch(split_rows_kernel, dim3(T), dim3(256), 0, stream, x, planes, T, K, pitch);
  KF_CHECK_LAUNCH();
  const int s = launch_split<true, TO>(tw, tx, a, stream);
  if (s != KF_OK || a.parts == 1) return s;
  const long n = (long)T * N;
  kf_launch(sum_parts_kernel<TO>, dim3(kf_ceil_div(n, 1024)), dim3(256), 0, stream, (const float*)a.partial, out, n, a.parts, softcap);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

}  // namespace

// Whether this product runs here: rows of whole 16 bytes on aligned bases, and weights of 4 Mi numbers or more (below, the
// launches around the product cost more than it saves).  T does not enter: see the order of a sum above.
KF_API int kf_linear_split_supported(const void* x, const void* w, int N, int K) {
  return K > 0 && K % 4 == 0 && (long)N * K >= (1l << 22) && N <= (1 << 24) && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 && tensor_maps_available();
}

// Floats of scratch that a call needs, and the kernels that it launches.
KF_API long kf_linear_split_scratch(int T, int N, int K) {
  const int parts = split_parts(N, K);
  return T <= SMALL_T ? 0 : plane_floats(T, K) + (parts > 1 ? (long)parts * T * N : 0);
}
KF_API int kf_linear_split_launches(int T, int N, int K) { return T <= SMALL_T ? 1 : split_parts(N, K) > 1 ? 3 : 2; }

// out[T, N] = x[T, K] . w[N, K]^T, all 32-bit (out may be bfloat16); softcap > 0 applies cap * tanh(v / cap).
KF_API int kf_linear_split(const float* x, const float* w, void* out, int out_dtype, int T, int N, int K, float softcap,
                           float* scratch, int* error_flag, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return KF_OK;
  if (!kf_linear_split_supported(x, w, N, K) || !scratch || !error_flag || ((uintptr_t)scratch & 15)) return KF_ERR_SIZE;
  if (out_dtype == KF_F32) return linear_split(x, w, (float*)out, T, N, K, softcap, scratch, error_flag, stream);
  if (out_dtype == KF_BF16) return linear_split(x, w, (__nv_bfloat16*)out, T, N, K, softcap, scratch, error_flag, stream);
  return KF_ERR_DTYPE;
}
