// Short causal convolution of a step's rows (see short_conv.cuh for the rule and the state), and the kernel that
// moves the state on after the step.
//
// kf_short_conv:        out[t][c] = act(conv(t, c) + out_bias[c]) for every row t of the step; rows of one request read
//                       the rows before them in the same step, or the state.
// kf_short_conv_commit: the state of every request of the step becomes its last taps-1 inputs, one thread per
//                       (request, channel).  It runs after every reader of the old state (stream order).
// Both skip padding (rows of request -1, requests without rows).
#include "short_conv.cuh"

enum { KF_CONV_ACT_NONE = 0, KF_CONV_ACT_SILU = 1 };

// VEC channels per thread (4 when every offset is a multiple of four floats: 16-byte loads and stores), `rows_per_block`
// rows per block.  A thread walks its rows with the last TAPS - 1 inputs in registers: a row is read once, four rows are
// asked for at a time, and a request's look-ups (where it starts, its slot) and the inputs before its first row here are
// fetched once per request, not per row.  What no earlier kernel of the step writes (taps, biases, the step's integers) is
// requested before the grid dependency is waited for, and with `early` the state too: the caller then says that nothing
// ahead of this kernel in the stream that may still be running writes it.  Bound by bytes at many rows, by latency at a few.
// Measured in place at 4,352 channels of four taps: 8 rows 5.3 -> 2.2 us, 2,048 rows 46 -> 25 us.
// `commit_state` (steps in which no request has more than one row, i.e. decoding): the thread that has just read a channel's
// tail also moves it on, which saves the commit kernel; with several rows per request other threads may still need the old
// tail, so the commit stays a kernel of its own there.
template <typename TW, int VEC, int TAPS>
__global__ void __launch_bounds__(256) short_conv_kernel(KfConvIn p, const TW* __restrict__ w, const TW* __restrict__ out_bias, int act,
                                  float* __restrict__ out, int ld_out, const int* __restrict__ row_req,
                                  const int* __restrict__ req_row_start, const int* __restrict__ req_state_slot, int T,
                                  int rows_per_block, float* commit_state, int early) {
  constexpr int H = TAPS > 1 ? TAPS - 1 : 1, U = 4;
  kf_pdl_trigger();
  if (!early) {
    kf_pdl_wait();
    p.state = kf_produced(p.state);
  }
  const int c0 = (blockIdx.y * blockDim.x + threadIdx.x) * VEC;
  if (c0 >= p.C) return;
  float wv[VEC][TAPS], bi[VEC], bo[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
#pragma unroll
    for (int j = 0; j < TAPS; ++j) wv[v][j] = kf_load(w, (size_t)(c0 + v) * TAPS + j);
    bi[v] = p.in_bias ? kf_load((const TW*)p.in_bias, c0 + v) : 0.f;
    bo[v] = out_bias ? kf_load(out_bias, c0 + v) : 0.f;
  }
  const int t0 = blockIdx.x * rows_per_block, t_end = min(T, t0 + rows_per_block);
  float h[H][VEC];                                          // h[k]: the input k + 1 rows before the current one
  auto take = [&](const float* src, float* u) {
    if (VEC == 4) { const float4 q = *reinterpret_cast<const float4*>(src); u[0] = q.x; u[1] = q.y; u[2] = q.z; u[VEC - 1] = q.w; }
    else u[0] = src[0];
  };
  int slot = 0;
  // the inputs before row t of request `req`: those of the state (which = 0), those of the step (1)
  auto before = [&](int req, int t, int which, const float* in) {
    const int row0 = req_row_start[req], i = t - row0;
    slot = req_state_slot[req];
#pragma unroll
    for (int k = 0; k < TAPS - 1; ++k) {
      const int idx = i - 1 - k;
      if (which && idx >= 0) {
        take(in + (size_t)(row0 + idx) * p.ld + p.col0 + c0, h[k]);
#pragma unroll
        for (int v = 0; v < VEC; ++v) h[k][v] += bi[v];
      } else if (!which && idx < 0) {
        take(p.state + ((size_t)slot * (TAPS - 1) + (TAPS - 1 + idx)) * p.C + c0, h[k]);
      }
    }
  };
  int cur = row_req[t0];
  if (cur >= 0) before(cur, t0, 0, nullptr);
  kf_pdl_wait();
  const float* in = kf_produced(p.in);
  if (cur >= 0) before(cur, t0, 1, in);
  for (int tb = t0; tb < t_end; tb += U) {
    float raw[U][VEC];
    int reqs[U];
#pragma unroll
    for (int r = 0; r < U; ++r) {
      reqs[r] = tb + r < t_end ? row_req[tb + r] : -1;
      if (tb + r < t_end) take(in + (size_t)(tb + r) * p.ld + p.col0 + c0, raw[r]);
    }
#pragma unroll
    for (int r = 0; r < U; ++r) {
      const int t = tb + r, req = reqs[r];
      if (req < 0) { cur = -1; continue; }
      if (req != cur) { before(req, t, 0, in); before(req, t, 1, in); cur = req; }
      float acc[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        raw[r][v] += bi[v];
        acc[v] = 0.f;
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) acc[v] = fmaf(wv[v][j], h[TAPS - 2 - j][v], acc[v]);
        acc[v] = fmaf(wv[v][TAPS - 1], raw[r][v], acc[v]);
      }
      if (TAPS > 1 && commit_state) {                       // one row per request: input j becomes tail entry j - 1
#pragma unroll
        for (int j = 1; j < TAPS; ++j) {
          const float* u = j == TAPS - 1 ? raw[r] : h[TAPS - 2 - j < 0 ? 0 : TAPS - 2 - j];
          float* dst = commit_state + ((size_t)slot * (TAPS - 1) + (j - 1)) * p.C + c0;
          if (VEC == 4) *reinterpret_cast<float4*>(dst) = make_float4(u[0], u[1], u[2], u[VEC - 1]);
          else dst[0] = u[0];
        }
      }
#pragma unroll
      for (int k = H - 1; k > 0; --k)
#pragma unroll
        for (int v = 0; v < VEC; ++v) h[k][v] = h[k - 1][v];
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        h[0][v] = raw[r][v];
        acc[v] += bo[v];
        if (act == KF_CONV_ACT_SILU) acc[v] = acc[v] / (1.f + expf(-acc[v]));
      }
      float* dst = out + (size_t)t * ld_out + c0;
      if (VEC == 4) *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[VEC - 1]);
      else dst[0] = acc[0];
    }
  }
}

template <typename TW>
__global__ void short_conv_commit_kernel(KfConvIn p, float* __restrict__ state, int n_reqs,
                                         const int* __restrict__ req_row_start, const int* __restrict__ req_n_rows,
                                         const int* __restrict__ req_state_slot) {
  kf_pdl_trigger();
  kf_pdl_wait();
  const int req = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (req >= n_reqs || c >= p.C) return;
  const int n = req_n_rows[req];
  if (n <= 0) return;
  const int row0 = req_row_start[req], slot = req_state_slot[req];
  float v[KF_MAX_TAPS - 1];
#pragma unroll
  for (int s = 0; s < KF_MAX_TAPS - 1; ++s)
    if (s < p.taps - 1) v[s] = kf_conv_input<TW>(p, row0, slot, n - (p.taps - 1) + s, c);   // old entries are read first
#pragma unroll
  for (int s = 0; s < KF_MAX_TAPS - 1; ++s)
    if (s < p.taps - 1) state[((size_t)slot * (p.taps - 1) + s) * p.C + c] = v[s];
}

// commit_inline: the step has no request with more than one row; the state is then moved on here and
// kf_short_conv_commit must not run for this step.  early: the state may be read before the kernels ahead have finished.
KF_API int kf_short_conv(const float* in, int ld, int col0, const void* in_bias, const void* w, const void* out_bias,
                         int w_dtype, int C, int taps, int act, float* state, float* out, int ld_out,
                         const int* row_req, const int* req_row_start, const int* req_state_slot, int T, int commit_inline,
                         int early, cudaStream_t stream) {
  if (T <= 0 || C <= 0) return KF_OK;
  if (taps < 1 || taps > KF_MAX_TAPS) return KF_ERR_SIZE;
  KfConvIn p{in, ld, col0, in_bias, state, C, taps};
  const bool vec = C % 4 == 0 && ld % 4 == 0 && col0 % 4 == 0 && ld_out % 4 == 0 &&
                   (((uintptr_t)in | (uintptr_t)out | (uintptr_t)state) & 15) == 0;
  const int per_thread = vec ? 4 : 1;
  const int threads = C / per_thread >= 256 ? 256 : 128;
  const int rows = T >= 1024 ? 16 : (T >= 64 ? 4 : 1);
  const dim3 grid(kf_ceil_div(T, rows), kf_ceil_div(C, threads * per_thread));
  float* commit = (commit_inline && taps > 1) ? state : nullptr;
#define KF_GO1(TW, VEC, TAPS)                                                                                           \
  kf_launch(short_conv_kernel<TW, VEC, TAPS>, grid, dim3(threads), 0, stream, p, (const TW*)w, (const TW*)out_bias, act, out, \
            ld_out, row_req, req_row_start, req_state_slot, T, rows, commit, early)
#define KF_GO(TW, VEC)                                                                                                  \
  switch (taps) {                                                                                                       \
    case 1: KF_GO1(TW, VEC, 1); break; case 2: KF_GO1(TW, VEC, 2); break; case 3: KF_GO1(TW, VEC, 3); break;            \
    case 4: KF_GO1(TW, VEC, 4); break; case 5: KF_GO1(TW, VEC, 5); break; case 6: KF_GO1(TW, VEC, 6); break;            \
    case 7: KF_GO1(TW, VEC, 7); break; default: KF_GO1(TW, VEC, 8); break;                                              \
  }
  if (w_dtype == KF_F32) { if (vec) { KF_GO(float, 4) } else { KF_GO(float, 1) } }
  else if (w_dtype == KF_BF16) { if (vec) { KF_GO(__nv_bfloat16, 4) } else { KF_GO(__nv_bfloat16, 1) } }
  else return KF_ERR_DTYPE;
#undef KF_GO
#undef KF_GO1
  KF_CHECK_LAUNCH();
  return KF_OK;
}

KF_API int kf_short_conv_commit(const float* in, int ld, int col0, const void* in_bias, int w_dtype, int C, int taps,
                                float* state, int n_reqs, const int* req_row_start, const int* req_n_rows,
                                const int* req_state_slot, cudaStream_t stream) {
  if (n_reqs <= 0 || C <= 0 || taps <= 1) return KF_OK;
  if (taps > KF_MAX_TAPS) return KF_ERR_SIZE;
  KfConvIn p{in, ld, col0, in_bias, state, C, taps};
  const int threads = C >= 256 ? 256 : 128;
  const dim3 grid(n_reqs, kf_ceil_div(C, threads));
  if (w_dtype == KF_F32)
    kf_launch(short_conv_commit_kernel<float>, grid, dim3(threads), 0, stream, p, state, n_reqs, req_row_start, req_n_rows,
              req_state_slot);
  else if (w_dtype == KF_BF16)
    kf_launch(short_conv_commit_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, p, state, n_reqs, req_row_start,
              req_n_rows, req_state_slot);
  else
    return KF_ERR_DTYPE;
  KF_CHECK_LAUNCH();
  return KF_OK;
}
