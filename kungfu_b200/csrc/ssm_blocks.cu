// The state-space recurrence of ssm.cu for prompts, as products over blocks of 128 rows.
//
// The walk of ssm.cu costs a row 3 N P packed multiply-adds per head and a chain over the rows.  Over a block of L = 128
// rows (of one request) with la_t the running sum of log decays, S_0 the state before the block and
//   dt_t, a   as there;   la_t = sum over s <= t of a dt_s  (a < 0)
// the same recurrence reads
//   y_t  = exp(la_t) S_0^T C_t + sum over s <= t of exp(la_t - la_s) dt_s (C_t . B_s) x_s + D x_t
//   S_L  = exp(la_L) S_0 + sum over s of exp(la_L - la_s) dt_s B_s x_s^T
// which are products of 128-row matrices: per row and head N P (state), N P (start state) and L P / 2 (inside the block)
// multiply-adds, and C_t . B_s once for all heads of a group.  Three kernels:
//   1. per (block, head): the block's own contribution to the state at its end; per (block, group): the table C_t . B_s;
//   2. the states at the blocks' starts, one after the other from the request's stored state, which takes the last one;
//   3. per (block, head): y.
// All products are 32-bit (packed FMAs, 8 x 8 outputs per thread); the running sums of log decays are kept as a pair of
// floats rounded from 64-bit sums, so that exp(la_t - la_s) does not lose what the sums have in common, and C_t . B_s is summed
// in 64 bits eight products at a time, because its error is that of every term inside a block.
// What bounds them is the FMA pipe (2.8 G multiply-adds at 2,048 rows of 64 heads x 64 x 128) at the rate that shared-memory
// reads leave it; the states between the kernels stay in L2.  One prompt of 2,048 rows: the walk 592 us, in chunks side by
// side 435 us, this 210 us with a cold L2.  Errors against 64 bits (2-norms; 128 to 2,048 rows, one to eight requests, decays of
// e^-0.01 to e^-3 a row): of y 6.9e-8 to 9.9e-8 (the walk 7.5e-8 to 2.9e-6), of the state 4.7e-8 to 1.5e-7 (4.9e-8 to 3.9e-6).
#include "common.cuh"

namespace {

constexpr int L = 128, THREADS = 128, PT = 64, NMAX = 128, LD = NMAX + 4;
constexpr int SMEM = (L + PT) * LD * (int)sizeof(float);       // 101,376 bytes: two blocks per SM

typedef unsigned long long pair_t;
__device__ __forceinline__ void fma2(pair_t& c, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ pair_t twice(float v) {
  pair_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float lo_of(pair_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(pair_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ pair_t pair_of(float lo, float hi) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void cp16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct Args {
  const float* xbc; int ld_x;
  const float* proj; int ld_p, dt_col0;
  const void* dt_bias; const void* a_log; const void* d_skip;
  float* state; float* y;
  int heads, groups, P, N, n_reqs;
  const int* req_state_slot;
  int write_state, max_blocks;
  const int* row_start; const int* n_rows;                      // per block
  const int* r_block0; const int* r_nblocks;                    // per request
  float* block_state; float* block_decay; float* table;         // [block, head, P, N], [block, head], [block, group, L, L]
};

// dt and the running sums of log decays of a block's rows (rows behind the last: dt 0, the sum stays).
template <typename TW>
__device__ __forceinline__ void decays(const Args& p, int row0, int rows, int h, float* s_dt, float* s_hi, float* s_lo, double* s_part) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  float dt = 0.f;
  if (t < rows) {
    const float z = p.proj[(size_t)(row0 + t) * p.ld_p + p.dt_col0 + h] + kf_load((const TW*)p.dt_bias, h);
    dt = z > 20.f ? z + log1pf(expf(-z)) : log1pf(expf(z));
  }
  const float a = -expf(kf_load((const TW*)p.a_log, h));
  double sum = fmax((double)a * (double)dt, -1e30);             // finite, so that differences of sums are numbers
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += v;
  }
  if (lane == 31) s_part[warp] = sum;
  __syncthreads();
  for (int w = 0; w < warp; ++w) sum += s_part[w];
  s_dt[t] = dt;
  s_hi[t] = (float)sum;
  s_lo[t] = (float)(sum - (double)(float)sum);
  __syncthreads();
}

// ---- 1: contributions to the state, and the tables C . B ---------------------------------------------------------------

template <typename TW>
__global__ void __launch_bounds__(THREADS, 2) ssm_block_state_kernel(const Args p) {
  kf_pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_dt[L], s_hi[L], s_lo[L];
  __shared__ double s_part[THREADS / 32];
  const int blk = blockIdx.x, rows = p.n_rows[blk];
  if (rows <= 0) return;
  const int row0 = p.row_start[blk], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, P = p.P, inner = p.heads * P;
  const int tx = (lane & 7) + 8 * (warp & 1), ty = (lane >> 3) + 4 * (warp >> 1);      // 16 x 8 threads
  const int cr = tid >> 3, cc = (tid & 7) * 4;                  // this thread copies rows cr + 16 i, four columns from cc + 32 j on
  int job = blockIdx.y;
  if (job < 3 * p.groups) {
    // The table of a group, 64 rows t x 64 columns s a job: (t, s) halves (0, 0), (1, 0) and (1, 1); nothing reads (0, 1).
    // Eight products at a time are summed in 32 bits, as four even and four odd states, and those sums in 64 bits: every
    // term of y that is made inside a block has one of these numbers in it.
    const int g = job / 3, th = (job % 3 + 1) >> 1, sh = job % 3 >> 1;
    if (64 * th >= rows) return;
    float* Cs = sm;                                             // [64][LD]
    float* Bs = sm + 64 * LD;                                   // [64][LD]
    const float* b0 = p.xbc + inner + g * N;
    const float* c0 = b0 + p.groups * N;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = cc + 32 * j;
#pragma unroll
      for (int r = cr; r < 64; r += 16) {
        const int t = 64 * th + r, s = 64 * sh + r;
        const bool in_b = n < N && s < rows, in_c = n < N && t < rows;
        cp16(Bs + r * LD + n, in_b ? b0 + (size_t)(row0 + s) * p.ld_x + n : p.xbc, in_b);
        cp16(Cs + r * LD + n, in_c ? c0 + (size_t)(row0 + t) * p.ld_x + n : p.xbc, in_c);
      }
      commit();
    }
    double sum[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] = 0.;
    auto slice = [&](int s) {
      for (int k0 = 32 * s; k0 < min(N, 32 * s + 32); k0 += 8) {
        pair_t acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
        for (int k = k0; k < k0 + 8; k += 4) {                  // columns from N on are zeros
          ulonglong2 a[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(Cs + (ty + 8 * i) * LD + k);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(Bs + (tx + 16 * j) * LD + k);
#pragma unroll
            for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
            for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].y, b.y);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) sum[i][j] += (double)lo_of(acc[i][j]) + (double)hi_of(acc[i][j]);
      }
    };
    wait_groups<3>(); __syncthreads(); slice(0);
    wait_groups<2>(); __syncthreads(); slice(1);
    wait_groups<1>(); __syncthreads(); slice(2);
    wait_groups<0>(); __syncthreads(); slice(3);
    float* out = p.table + ((size_t)blk * p.groups + g) * L * L + (size_t)64 * th * L + 64 * sh;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) out[(ty + 8 * i) * L + tx + 16 * j] = (float)sum[i][j];
    return;
  }
  job -= 3 * p.groups;
  const int ptiles = (P + PT - 1) / PT, h = job / ptiles, pb = job % ptiles * PT, g = h / (p.heads / p.groups);
  float* Bs = sm;                                               // [128][NMAX]
  float* Xs = sm + L * NMAX;                                    // [128][PT]
  const float* b0 = p.xbc + inner + g * N;
  const float* x0 = p.xbc + h * P + pb;
#pragma unroll
  for (int s = 0; s < 4; ++s) {                                 // 32 rows a group
#pragma unroll
    for (int r = 32 * s + cr; r < 32 * s + 32; r += 16) {
#pragma unroll
      for (int n = cc; n < NMAX; n += 32) {
        const bool in = r < rows && n < N;
        cp16(Bs + r * NMAX + n, in ? b0 + (size_t)(row0 + r) * p.ld_x + n : p.xbc, in);
      }
#pragma unroll
      for (int c = cc; c < PT; c += 32) {
        const bool in = r < rows && pb + c < P;
        cp16(Xs + r * PT + c, in ? x0 + (size_t)(row0 + r) * p.ld_x + c : p.xbc, in);
      }
    }
    commit();
  }
  decays<TW>(p, row0, rows, h, s_dt, s_hi, s_lo, s_part);
  const float end_hi = s_hi[L - 1], end_lo = s_lo[L - 1];
  if (tid == 0 && pb == 0) p.block_decay[(size_t)blk * p.heads + h] = expf(end_hi + end_lo);
  pair_t acc[8][4];                                             // p = 4 ty + (0..3) and 32 + those; pairs of n = 4 tx + .. and 64 + ..
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  auto slice = [&](int s) {
#pragma unroll
    for (int r = 32 * s + cr; r < 32 * s + 32; r += 16) {       // what this thread copied of x, times its row's weight
      const float w = s_dt[r] * expf((end_hi - s_hi[r]) + (end_lo - s_lo[r]));
#pragma unroll
      for (int c = cc; c < PT; c += 32) {
        float4* v = reinterpret_cast<float4*>(Xs + r * PT + c);
        float4 u = *v;
        u.x *= w; u.y *= w; u.z *= w; u.w *= w;
        *v = u;
      }
    }
    __syncthreads();
    if (32 * s >= rows) return;
#pragma unroll 4
    for (int r = 32 * s; r < 32 * s + 32; ++r) {
      const float4 xa = *reinterpret_cast<const float4*>(Xs + r * PT + 4 * ty), xb = *reinterpret_cast<const float4*>(Xs + r * PT + 32 + 4 * ty);
      const ulonglong2 ba = *reinterpret_cast<const ulonglong2*>(Bs + r * NMAX + 4 * tx), bb = *reinterpret_cast<const ulonglong2*>(Bs + r * NMAX + 64 + 4 * tx);
      const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const pair_t xx = twice(x[i]);
        fma2(acc[i][0], xx, ba.x);
        fma2(acc[i][1], xx, ba.y);
        fma2(acc[i][2], xx, bb.x);
        fma2(acc[i][3], xx, bb.y);
      }
    }
  };
  wait_groups<3>(); slice(0);
  wait_groups<2>(); slice(1);
  wait_groups<1>(); slice(2);
  wait_groups<0>(); slice(3);
  float* out = p.block_state + ((size_t)blk * p.heads + h) * P * N;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int pp = pb + 4 * ty + (i & 3) + (i >= 4 ? 32 : 0);
    if (pp >= P) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int n = 4 * tx + 64 * j;
      if (n < N)
        *reinterpret_cast<float4*>(out + (size_t)pp * N + n) =
            make_float4(lo_of(acc[i][2 * j]), hi_of(acc[i][2 * j]), lo_of(acc[i][2 * j + 1]), hi_of(acc[i][2 * j + 1]));
    }
  }
}

// ---- 2: the states at the blocks' starts ----------------------------------------------------------------------------------

__global__ void __launch_bounds__(256) ssm_block_fold_kernel(const Args p) {
  kf_pdl_trigger();
  kf_pdl_wait();
  const int req = blockIdx.x, h = blockIdx.y, PN = p.P * p.N, e = (blockIdx.z * 256 + threadIdx.x) * 4;
  const int n = p.r_nblocks[req];
  if (e >= PN || n <= 0) return;
  const int k0 = p.r_block0[req], slot = p.req_state_slot[req];
  float4* own = reinterpret_cast<float4*>(p.state + ((size_t)slot * p.heads + h) * PN + e);
  float4* at = reinterpret_cast<float4*>(p.block_state + ((size_t)k0 * p.heads + h) * PN + e);
  const size_t step = (size_t)p.heads * PN / 4;
  const float* dec = p.block_decay + (size_t)k0 * p.heads + h;
  float4 S = *own;
  for (int k = 0; k < n; k += 8) {                              // eight blocks' numbers asked for at once
    float4 add[8];
    float d[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u < n) add[u] = at[(k + u) * step], d[u] = dec[(size_t)(k + u) * p.heads];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u < n) {
        at[(k + u) * step] = S;
        S.x = fmaf(d[u], S.x, add[u].x); S.y = fmaf(d[u], S.y, add[u].y); S.z = fmaf(d[u], S.z, add[u].z); S.w = fmaf(d[u], S.w, add[u].w);
      }
  }
  if (p.write_state) *own = S;
}

// ---- 3: y -----------------------------------------------------------------------------------------------------------------

template <typename TW>
__global__ void __launch_bounds__(THREADS, 2) ssm_block_out_kernel(const Args p) {
  kf_pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_dt[L], s_hi[L], s_lo[L];
  __shared__ double s_part[THREADS / 32];
  const int blk = blockIdx.x, rows = p.n_rows[blk];
  if (rows <= 0) return;
  const int row0 = p.row_start[blk], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = p.N, P = p.P, inner = p.heads * P;
  const int ptiles = (P + PT - 1) / PT, h = blockIdx.y / ptiles, pb = blockIdx.y % ptiles * PT, g = h / (p.heads / p.groups);
  const int cr = tid >> 3, cc = (tid & 7) * 4;
  // 32 rows per warp; the later rows have more of the block's sum, so every other block deals the warps the other way round
  const int band = (blockIdx.x + blockIdx.y) & 1 ? 3 - warp : warp;
  const int tx = lane & 7, ty = lane >> 3;
  // this thread's rows: 32 band + ty + 4 i; its columns p: 4 tx + (0..3) and 32 + those
  float* Cs = sm;                                               // [128][LD]; then the weights of the rows s: [128][LD]
  float* Ss = sm + L * LD;                                      // [PT][LD], row 4 a + b of a half at 8 b + a; then x: [128][PT]
  const float* c0 = p.xbc + inner + (p.groups + g) * N;
  const float* s0 = p.block_state + ((size_t)blk * p.heads + h) * P * N;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = cc + 32 * j;
#pragma unroll
    for (int r = cr; r < L; r += 16) {
      const bool in = n < N && r < rows;
      cp16(Cs + r * LD + n, in ? c0 + (size_t)(row0 + r) * p.ld_x + n : p.xbc, in);
    }
#pragma unroll
    for (int r = cr; r < PT; r += 16) {
      const bool in = n < N && pb + r < P;
      cp16(Ss + ((r & 3) * 8 + ((r >> 2) & 7) + (r & 32)) * LD + n, in ? s0 + (size_t)(pb + r) * N + n : p.xbc, in);
    }
    commit();
  }
  decays<TW>(p, row0, rows, h, s_dt, s_hi, s_lo, s_part);
  // y of the thread's outputs: sums of at most 64 terms (as even and odd ones) or 32 are made apart and then added, as the
  // walk's lanes do, so that no chain is longer than those
  pair_t y[8][4];
  {
    pair_t acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    auto slice = [&](int s) {
      if (32 * band >= rows) return;
      for (int k = 32 * s; k < min(N, 32 * s + 32); k += 4) {
        ulonglong2 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(Cs + (32 * band + ty + 4 * i) * LD + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(Ss + ((j & 3) * 8 + tx + (j & 4) * 8) * LD + k);
#pragma unroll
          for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
          for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].y, b.y);
        }
      }
    };
    wait_groups<3>(); __syncthreads(); slice(0);
    wait_groups<2>(); __syncthreads(); slice(1);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[i][j] = pair_of(lo_of(acc[i][2 * j]) + hi_of(acc[i][2 * j]), lo_of(acc[i][2 * j + 1]) + hi_of(acc[i][2 * j + 1]));
        acc[i][2 * j] = acc[i][2 * j + 1] = 0ull;
      }
    wait_groups<1>(); __syncthreads(); slice(2);
    wait_groups<0>(); __syncthreads(); slice(3);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = 32 * band + ty + 4 * i;
      const float d = expf(s_hi[t] + s_lo[t]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        y[i][j] = pair_of(d * (lo_of(y[i][j]) + (lo_of(acc[i][2 * j]) + hi_of(acc[i][2 * j]))),
                          d * (hi_of(y[i][j]) + (lo_of(acc[i][2 * j + 1]) + hi_of(acc[i][2 * j + 1]))));
    }
  }
  __syncthreads();                                              // C and the start state are used up
  float* Ms = Cs;
  float* Xs = Ss;
  const float* t0 = p.table + ((size_t)blk * p.groups + g) * L * L;
  const float* x0 = p.xbc + h * P + pb;
#pragma unroll
  for (int s = 0; s < 4; ++s) {                                 // columns 32 s .. of the table from row 32 s on, and x of those rows
#pragma unroll
    for (int r = 32 * s + cr; r < L; r += 16) {
      const bool in = r < rows;
      cp16(Ms + r * LD + 32 * s + cc, in ? t0 + r * L + 32 * s + cc : p.xbc, in);
    }
#pragma unroll
    for (int r = 32 * s + cr; r < 32 * s + 32; r += 16)
#pragma unroll
      for (int c = cc; c < PT; c += 32) {
        const bool in = r < rows && pb + c < P;
        cp16(Xs + r * PT + c, in ? x0 + (size_t)(row0 + r) * p.ld_x + c : p.xbc, in);
      }
    commit();
  }
  auto inside = [&](int s) {
    bool bad = false;                                           // what this thread copied of x: numbers that are not finite
#pragma unroll
    for (int r = 32 * s + cr; r < 32 * s + 32; r += 16)
#pragma unroll
      for (int c = cc; c < PT; c += 32) {
        const float4 v = *reinterpret_cast<const float4*>(Xs + r * PT + c);
        bad |= !isfinite(v.x) | !isfinite(v.y) | !isfinite(v.z) | !isfinite(v.w);
      }
    // what this thread copied of the table becomes exp(la_t - la_s) dt_s (C_t . B_s), zero above the diagonal
    const int c = 32 * s + cc;
    if (32 * s < rows) {
      const float h0 = s_hi[c], h1 = s_hi[c + 1], h2 = s_hi[c + 2], h3 = s_hi[c + 3];
      const float l0 = s_lo[c], l1 = s_lo[c + 1], l2 = s_lo[c + 2], l3 = s_lo[c + 3];
      const float d0 = s_dt[c], d1 = s_dt[c + 1], d2 = s_dt[c + 2], d3 = s_dt[c + 3];
#pragma unroll
      for (int r = 32 * s + cr; r < L; r += 16) {
        float4* v = reinterpret_cast<float4*>(Ms + r * LD + c);
        const float th = s_hi[r], tl = s_lo[r];
        float4 u = *v;
        u.x = c <= r ? u.x * (d0 * expf((th - h0) + (tl - l0))) : 0.f;
        u.y = c + 1 <= r ? u.y * (d1 * expf((th - h1) + (tl - l1))) : 0.f;
        u.z = c + 2 <= r ? u.z * (d2 * expf((th - h2) + (tl - l2))) : 0.f;
        u.w = c + 3 <= r ? u.w * (d3 * expf((th - h3) + (tl - l3))) : 0.f;
        *v = u;
      }
    }
    bad = __syncthreads_or(bad);
    if (s > band || 32 * band >= rows) return;
    pair_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    if (bad && s == band) {
      // some x of these rows is not finite, and zero times it is not zero: each row takes its columns up to itself only.  (Left
      // out in the loop below, whoever is not finite, they cost 228 us of three kernels at 2,048 rows where this costs 212.)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = 32 * band + ty + 4 * i;
#pragma unroll 1
        for (int k = 32 * s; k <= row; ++k) {
          const pair_t m = twice(Ms[row * LD + k]);
          const ulonglong2 xa = *reinterpret_cast<const ulonglong2*>(Xs + k * PT + 4 * tx);
          const ulonglong2 xb = *reinterpret_cast<const ulonglong2*>(Xs + k * PT + 32 + 4 * tx);
          fma2(acc[i][0], m, xa.x);
          fma2(acc[i][1], m, xa.y);
          fma2(acc[i][2], m, xb.x);
          fma2(acc[i][3], m, xb.y);
        }
      }
    } else {
#pragma unroll 2
      for (int k = 32 * s; k < 32 * s + 32; k += 4) {
        float4 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(Ms + (32 * band + ty + 4 * i) * LD + k);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const ulonglong2 xa = *reinterpret_cast<const ulonglong2*>(Xs + (k + u) * PT + 4 * tx);
          const ulonglong2 xb = *reinterpret_cast<const ulonglong2*>(Xs + (k + u) * PT + 32 + 4 * tx);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const pair_t m = twice(u == 0 ? a[i].x : u == 1 ? a[i].y : u == 2 ? a[i].z : a[i].w);
            fma2(acc[i][0], m, xa.x);
            fma2(acc[i][1], m, xa.y);
            fma2(acc[i][2], m, xb.x);
            fma2(acc[i][3], m, xb.y);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(y[i][j]) : "l"(acc[i][j]));
  };
  wait_groups<3>(); inside(0);
  wait_groups<2>(); inside(1);
  wait_groups<1>(); inside(2);
  wait_groups<0>(); inside(3);
  kf_pdl_trigger();
  const float dsk = kf_load((const TW*)p.d_skip, h);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = 32 * band + ty + 4 * i;
    if (t >= rows) continue;
    float* yo = p.y + (size_t)(row0 + t) * inner + h * P + pb;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = 4 * tx + 32 * j;
      if (pb + c >= P) continue;
      const float4 x = *reinterpret_cast<const float4*>(Xs + t * PT + c);
      *reinterpret_cast<float4*>(yo + c) = make_float4(fmaf(dsk, x.x, lo_of(y[i][2 * j])), fmaf(dsk, x.y, hi_of(y[i][2 * j])),
                                                       fmaf(dsk, x.z, lo_of(y[i][2 * j + 1])), fmaf(dsk, x.w, hi_of(y[i][2 * j + 1])));
    }
  }
}

// Cuts the requests' rows into blocks.
__global__ void ssm_block_list_kernel(int n_reqs, const int* __restrict__ req_row_start, const int* __restrict__ req_n_rows, int max_blocks,
                                      int* __restrict__ row_start, int* __restrict__ n_rows, int* __restrict__ r_block0, int* __restrict__ r_nblocks) {
  kf_pdl_trigger();
  kf_pdl_wait();
  if (threadIdx.x != 0) return;
  int k = 0;
  for (int r = 0; r < n_reqs; ++r) {
    const int n = req_n_rows[r], nb = n > 0 ? (n + L - 1) / L : 0;
    r_block0[r] = k;
    r_nblocks[r] = nb;
    for (int c = 0; c < nb && k < max_blocks; ++c, ++k) {
      row_start[k] = req_row_start[r] + c * L;
      n_rows[k] = min(L, n - c * L);
    }
  }
  for (; k < max_blocks; ++k) n_rows[k] = 0;
}

template <typename TW>
int launch(const Args& a, cudaStream_t s) {
  const cudaError_t e1 = cudaFuncSetAttribute((const void*)ssm_block_state_kernel<TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  const cudaError_t e2 = cudaFuncSetAttribute((const void*)ssm_block_out_kernel<TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e1 != cudaSuccess || e2 != cudaSuccess) { kf_record_cuda_error(e1 != cudaSuccess ? e1 : e2); return KF_ERR_SETUP; }
  const int ptiles = kf_ceil_div(a.P, PT), PN = a.P * a.N;
  // without the programmatic-dependent-launch attribute: blocks of 100 KB that wait would keep the kernel before them off the SMs
  ssm_block_state_kernel<TW><<<dim3(a.max_blocks, 3 * a.groups + a.heads * ptiles), THREADS, SMEM, s>>>(a);
  kf_launch(ssm_block_fold_kernel, dim3(a.n_reqs, a.heads, kf_ceil_div(PN, 1024)), dim3(256), 0, s, a);
  ssm_block_out_kernel<TW><<<dim3(a.max_blocks, a.heads * ptiles), THREADS, SMEM, s>>>(a);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

}  // namespace

// Rows per block, and whether the kernels take these sizes (16-byte vectors everywhere; at most 128 states).
KF_API int kf_ssm_blocks_rows() { return L; }
KF_API int kf_ssm_blocks_supported(const float* xbc, int ld_x, const float* state, int heads, int groups, int P, int N) {
  return N >= 4 && N <= NMAX && N % 4 == 0 && P % 4 == 0 && ld_x % 4 == 0 && groups >= 1 && heads % groups == 0 &&
         (((uintptr_t)xbc | (uintptr_t)state) & 15) == 0 && 3L * groups + (long)heads * kf_ceil_div(P, PT) <= 65535;
}

// As kf_ssm_scan.  Scratch from the caller, with max_blocks >= rows / 128 + n_reqs: `list` 2 * max_blocks + 2 * n_reqs ints,
// `block_state` max_blocks * heads * P * N floats, `block_decay` max_blocks * heads floats, `table` max_blocks * groups *
// 128 * 128 floats; block_state, table and y on 16-byte boundaries.
KF_API int kf_ssm_scan_blocks(const float* xbc, int ld_x, const float* proj, int ld_p, int dt_col0, const void* dt_bias,
                              const void* a_log, const void* d_skip, int w_dtype, float* state, float* y, int heads, int groups,
                              int P, int N, int n_reqs, const int* req_row_start, const int* req_n_rows,
                              const int* req_state_slot, int write_state, int max_blocks, int* list, float* block_state,
                              float* block_decay, float* table, cudaStream_t stream) {
  if (n_reqs <= 0) return KF_OK;
  if (heads < 1 || P < 1 || max_blocks < 1 || !kf_ssm_blocks_supported(xbc, ld_x, state, heads, groups, P, N)) return KF_ERR_SIZE;
  if ((((uintptr_t)block_state | (uintptr_t)table | (uintptr_t)y) & 15) != 0) return KF_ERR_ALIGN;
  if (w_dtype != KF_F32 && w_dtype != KF_BF16) return KF_ERR_DTYPE;
  const Args a{xbc, ld_x, proj, ld_p, dt_col0, dt_bias, a_log, d_skip, state, y, heads, groups, P, N, n_reqs, req_state_slot,
               write_state, max_blocks, list, list + max_blocks, list + 2 * max_blocks, list + 2 * max_blocks + n_reqs,
               block_state, block_decay, table};
  kf_launch(ssm_block_list_kernel, dim3(1), dim3(32), 0, stream, n_reqs, req_row_start, req_n_rows, max_blocks, list,
            list + max_blocks, list + 2 * max_blocks, list + 2 * max_blocks + n_reqs);
  return w_dtype == KF_F32 ? launch<float>(a, stream) : launch<__nv_bfloat16>(a, stream);
}
