// Paged attention for any head size up to 512, any number of heads and groups, any page size, in exact 32-bit arithmetic
// (expf, tanhf, no fast-math).
//
// For the row at position p of request r: keys lo..p, lo = max(0, p - window + 1) on a windowed layer, else 0 (reference:
// window rule crates/kf-backend-cuda/src/kernels/attention.cu:156, scores/softcap :80-81, lane-per-key online softmax :68-103):
//   s_j = (q . k_j) * scale;  s_j = cap * tanh(s_j / cap) if cap > 0
//   o   = sum_j softmax(s)_j v_j,  zeros if no key is visible.
// keep_first > 0 (with a window): keys 0..keep_first-1 stay visible behind the window, at their true positions.
// sink != 0: the softmax's denominator has one more term, exp(0) (a key of score 0 without a value): the walk starts from
// maximum 0 and sum 1.
// window < 0: chunks of -window positions (kf_first_key).  sig_bias (one number per head, or null): no softmax; key j counts
// with sigmoid(s_j + sig_bias[h]), and the weights are not normalized.
// This is the engine's 32-bit attention and the fallback of the bfloat16 path for head sizes the tensor-core kernels do not
// take.
//
// A block owns up to 16 (row, query head) pairs over one stored head and walks the keys in runs of 32 from a multiple of 32:
//   * keys and values of a run are copied to shared memory once for all pairs (a warp per row, 16-byte cp.async where the
//     rows are 32-bit and aligned); the next run's keys are on their way during P V, its values during Q K^T;
//   * Q K^T: a warp has two pairs and a key per lane (packed FMAs over four elements at a time), so that the maximum and the
//     sum of a pair are shuffles inside its warp; P V: a thread has an element and all pairs (packed FMAs over two pairs).
// What bounds it is shared-memory reads (some 3,000 cycles a run of 32 keys for 16 pairs).  One warp per pair, one lane per
// key and the keys' rows straight from L2 took 172 us a launch where this takes 14 (one B200, 8 heads of 256 over 4: a
// prompt step of 167 rows up to position 97 and two decode steps).
// The order of every sum is fixed by (row, head) alone: the runs lie at multiples of 32, and a run that a row does not see
// leaves its maximum, sum and accumulators as they are.  So a row's result does not depend on how the step was cut, on
// what else is in the batch, or on how many rows a block has.
#include "common.cuh"
#include <type_traits>

constexpr int MAX_D_ALL = 512;
constexpr int NQ = 16, RUN = 32, ATHREADS = 256, PLD = NQ + 4;

__device__ __forceinline__ void fma_pair(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float lo_of(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

// floats between rows in shared memory: rows of eight neighbouring keys start in different banks
__host__ __device__ constexpr int row_pitch(int d) { return (d + 31) / 32 * 32 + 4; }

// DT: threads along the head's elements (64, 128 or 256), DPT: elements per thread.  At heads of 256, where shared memory allows two
// blocks per SM, the compiler is told so: left to itself it takes 79 registers and reads less ahead (eight rows of 2,048 keys
// 490 us, with 128 registers 442; a step of 97 and 60 rows 51 -> 45).  Below, its own choice of 62 to 64 is the better one.
template <typename TQ, typename TKV, int DT, int DPT>
__global__ void __launch_bounds__(ATHREADS, DT == 256 ? 2 : 0)
attention_generic_kernel(const TQ* __restrict__ q, TQ* __restrict__ out, const TKV* __restrict__ pages,
                         const int* __restrict__ items, const int* __restrict__ positions,
                         const int* __restrict__ row_req, const int* __restrict__ block_table, int table_stride,
                         int page_size, int nh, int nkv, int d, float scale, float softcap, int window, int vsplit,
                         int keep_first, int sink, const float* __restrict__ sig_bias, int T, int rows, int vec) {
  constexpr int PAIRS = NQ / (ATHREADS / DT) / 2;           // pairs of (row, head) pairs a thread accumulates
  kf_pdl_trigger();
  extern __shared__ __align__(16) float sm[];
  __shared__ int s_row[NQ], s_req[NQ], s_pos[NQ], s_lo[NQ], s_kept[NQ];
  __shared__ __align__(16) float s_p[RUN * PLD];
  __shared__ __align__(16) float s_corr[NQ];
  const int ld = row_pitch(d), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* const Ks = sm;
  float* const Vs = sm + RUN * ld;
  float* const Qs = sm + 2 * RUN * ld;

  const int group = nh / nkv, per = min(group, NQ), cuts = (group + per - 1) / per;
  const int y = blockIdx.x % (nkv * cuts), kvh = y / cuts;
  const int h0 = kvh * group + (y % cuts) * per, n_h = min(per, kvh * group + group - h0);
  const int it0 = blockIdx.x / (nkv * cuts) * rows;
  kf_pdl_wait();

  // pair p = row p / per of the block, head h0 + p % per; a pair without a row or head has s_row = -1
  if (tid < NQ) {
    const int i = tid / per, it = it0 + i;
    const bool in = i < rows && it < T && tid % per < n_h;
    const int t = in ? (items ? items[it] : it) : -1;       // `items` names the rows this launch handles
    const int req = in ? row_req[t] : -1, pos = req >= 0 ? positions[t] : -1;
    const int lo = kf_first_key(max(pos, 0), window);
    s_row[tid] = t, s_req[tid] = req, s_pos[tid] = pos, s_lo[tid] = lo;
    s_kept[tid] = min(keep_first, lo);                      // keys [0, kept) are seen behind the window
  }
  // shared memory starts as zeros: the padding of every row, and the values of keys that no row of the block sees
  for (int i = tid; i < (2 * RUN + NQ) * ld; i += ATHREADS) sm[i] = 0.f;
  __syncthreads();
  const KfHeadMap hm = kf_head_map(h0, kvh, nh, nkv, vsplit);
  for (int p = warp; p < NQ; p += ATHREADS / 32) {
    if (s_row[p] < 0) continue;
    const TQ* qr = q + ((size_t)s_row[p] * hm.n_query + kf_head_map(h0 + p % per, kvh, nh, nkv, vsplit).query) * d;
    for (int e = lane; e < d; e += 32) Qs[p * ld + e] = kf_load(qr, e);
  }

  const size_t head_stride = (size_t)page_size * d;
  unsigned long long acc[DPT][PAIRS];
#pragma unroll
  for (int e = 0; e < DPT; ++e)
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) acc[e][i] = 0ull;
  float m[2], l[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) m[u] = sink ? 0.f : -INFINITY, l[u] = sink ? 1.f : 0.f;
  const int p0 = 2 * warp;                                  // this warp's pairs in Q K^T: p0, p0 + 1
  const int de = tid % DT, pg = tid / DT * (2 * PAIRS);     // this thread's element and first pair in P V

  // the rows of a block may belong to several requests: neighbouring rows of one request are walked together
  for (int a = 0; a < rows;) {
    const int req = s_req[a * per];
    int b = a + 1;
    while (b < rows && s_req[b * per] == req) ++b;
    if (req >= 0) {
      int min_lo = s_lo[a * per], max_pos = -1, max_kept = 0;
      for (int i = a; i < b; ++i) {
        min_lo = min(min_lo, s_lo[i * per]);
        max_pos = max(max_pos, s_pos[i * per]);
        max_kept = max(max_kept, s_kept[i * per]);
      }
      const int* table = block_table + (size_t)req * table_stride;
      auto run_from = [&](int c) { return c * RUN < max_kept ? c : max(c, min_lo / RUN); };
      // copies the keys (which = 0) or values (1) of run c; keys that no row of the walk sees become zeros
      auto copy = [&](int c, int which) {
        if (c * RUN <= max_pos) {
          float* dst = which ? Vs : Ks;
          for (int u = warp; u < RUN; u += ATHREADS / 32) {
            const int j = c * RUN + u;
            const bool seen = j <= max_pos && (j >= min_lo || j < max_kept);
            if (seen) {
              const int page = table[j / page_size];
              const TKV* src = pages + (((size_t)page * 2 + which) * hm.n_stored + (which ? hm.value : hm.key)) * head_stride + (size_t)(j % page_size) * d;
              if (std::is_same<TKV, float>::value && vec) {
                for (int e = 4 * lane; e < d; e += 128)
                  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + u * ld + e)), "l"((const float*)src + e) : "memory");
              } else {
                for (int e = lane; e < d; e += 32) dst[u * ld + e] = kf_load(src, e);
              }
            } else {
              for (int e = lane; e < d; e += 32) dst[u * ld + e] = 0.f;
            }
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };

      int c = run_from(0);
      copy(c, 0);
      copy(c, 1);
      while (c * RUN <= max_pos) {
        const int next = run_from(c + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                    // the run's keys (and, the first time, q) are there
        unsigned long long dot[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
        if (s_row[p0] >= 0 || s_row[p0 + 1] >= 0) {
          const float* kr = Ks + lane * ld;
          const float* qa = Qs + p0 * ld;
#pragma unroll 8
          for (int e = 0; e < d; e += 4) {
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(kr + e);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(qa + u * ld + e);
              fma_pair(dot[u][0], x.x, k.x);
              fma_pair(dot[u][1], x.y, k.y);
            }
          }
        }
        float pv[2];
        bool see[2];
        bool all = true;                                    // every pair sees every key of the run
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int p = p0 + u, row = p / per, j = c * RUN + lane;
          const bool mine = s_row[p] >= 0 && row >= a && row < b;
          const bool seen = mine && j <= s_pos[p] && (j >= s_lo[p] || j < s_kept[p]);
          all = all && (s_row[p] < 0 || seen);
          see[u] = seen;
          const float sum = (lo_of(dot[u][0]) + hi_of(dot[u][0])) + (lo_of(dot[u][1]) + hi_of(dot[u][1]));
          const float s = seen ? kf_softcap(sum * scale, softcap) : -INFINITY;
          float corr = 1.f;
          if (sig_bias) {
            if (mine) l[u] = 1.f;
            pv[u] = seen ? 1.f / (1.f + expf(-(s + sig_bias[h0 + p % per]))) : 0.f;
          } else {
            const float m_new = fmaxf(m[u], kf_warp_max(s));
            pv[u] = seen ? expf(s - m_new) : 0.f;
            corr = (m[u] == -INFINITY) ? 0.f : expf(m[u] - m_new);
            l[u] = l[u] * corr + kf_warp_sum(pv[u]);
            m[u] = m_new;
          }
          if (lane == 0) s_corr[p] = corr;
        }
        // a weight below zero marks a key that its pair does not see (a seen one's may have underflowed to zero)
        *reinterpret_cast<float2*>(s_p + lane * PLD + p0) = make_float2(see[0] ? pv[0] : -1.f, see[1] ? pv[1] : -1.f);
        all = __syncthreads_and(all);                       // the keys are free, the weights are there
        copy(next, 0);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                    // the run's values are there
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
          const unsigned long long f = *reinterpret_cast<const unsigned long long*>(s_corr + pg + 2 * i);
#pragma unroll
          for (int e = 0; e < DPT; ++e) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[e][i]) : "l"(f));
        }
        if (all) {
#pragma unroll 4
          for (int u = 0; u < RUN; ++u) {
            unsigned long long w[PAIRS];
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) w[i] = *reinterpret_cast<const unsigned long long*>(s_p + u * PLD + pg + 2 * i);
#pragma unroll
            for (int e = 0; e < DPT; ++e) {
              const float v = de + e * DT < d ? Vs[u * ld + de + e * DT] : 0.f;
              const unsigned long long vv = pair_of(v, v);
#pragma unroll
              for (int i = 0; i < PAIRS; ++i) fma_pair(acc[e][i], w[i], vv);
            }
          }
        } else {
          // A key that a pair does not see is left out, not multiplied by zero: its value may be infinite.  One that it sees
          // is multiplied whatever its weight is, as above, so that a row's result does not depend on the block's other rows.
          for (int u = 0; u < RUN; ++u) {
            float v[DPT];
#pragma unroll
            for (int e = 0; e < DPT; ++e) v[e] = de + e * DT < d ? Vs[u * ld + de + e * DT] : 0.f;
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
              const float w0 = s_p[u * PLD + pg + 2 * i], w1 = s_p[u * PLD + pg + 2 * i + 1];
              if (!(w0 < 0.f)) {
#pragma unroll
                for (int e = 0; e < DPT; ++e) acc[e][i] = pair_of(fmaf(w0, v[e], lo_of(acc[e][i])), hi_of(acc[e][i]));
              }
              if (!(w1 < 0.f)) {
#pragma unroll
                for (int e = 0; e < DPT; ++e) acc[e][i] = pair_of(lo_of(acc[e][i]), fmaf(w1, v[e], hi_of(acc[e][i])));
              }
            }
          }
        }
        __syncthreads();                                    // the values and the weights are free
        copy(next, 1);
        c = next;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
    a = b;
  }

  if (lane < 2) s_corr[p0 + lane] = (lane ? l[1] : l[0]) > 0.f ? 1.f / (lane ? l[1] : l[0]) : 0.f;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2 * PAIRS; ++i) {
    const int p = pg + i;
    if (s_row[p] < 0) continue;
    TQ* o = out + ((size_t)s_row[p] * nh + h0 + p % per) * d;
#pragma unroll
    for (int e = 0; e < DPT; ++e) {
      const float v = (i & 1) ? hi_of(acc[e][i / 2]) : lo_of(acc[e][i / 2]);
      if (de + e * DT < d) kf_store(o, de + e * DT, s_req[p] < 0 ? 0.f : v * s_corr[p]);      // padding rows are zeros
    }
  }
}

template <typename TQ, typename TKV, int DT, int DPT>
static int launch(const void* q, void* out, const void* pages, const int* items, const int* positions, const int* row_req,
                  const int* block_table, int table_stride, int page_size, int nh, int nkv, int d, float scale, float softcap,
                  int window, int vsplit, int keep_first, int sink, const float* sig_bias, int T, cudaStream_t stream) {
  auto kernel = attention_generic_kernel<TQ, TKV, DT, DPT>;
  const size_t smem = sizeof(float) * (2 * RUN + NQ) * row_pitch(d);
  const cudaError_t e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(sizeof(float) * (2 * RUN + NQ) * row_pitch(DT * DPT)));
  if (e != cudaSuccess) { kf_record_cuda_error(e); return KF_ERR_SETUP; }
  const int group = nh / nkv, per = group < NQ ? group : NQ, cuts = kf_ceil_div(group, per);
  // Rows of a block share the copies of keys and values: as many as 16 pairs hold, while there are blocks for all SMs
  // (fewer rows only leave warps of a block without a pair, and a step of a few rows is bound by one block's walk).
  int rows = NQ / per;
  while (rows > 1 && (long)kf_ceil_div(T, rows) * nkv * cuts < kf_sm_count()) rows = (rows + 1) / 2;
  const long blocks = (long)kf_ceil_div(T, rows) * nkv * cuts;
  if (blocks > 0x7fffffffL) return KF_ERR_SIZE;
  const int vec = d % 4 == 0 && ((uintptr_t)pages & 15) == 0;
  kf_launch(kernel, dim3((unsigned)blocks), dim3(ATHREADS), smem, stream, (const TQ*)q, (TQ*)out, (const TKV*)pages, items,
            positions, row_req, block_table, table_stride, page_size, nh, nkv, d, scale, softcap, window, vsplit, keep_first,
            sink, sig_bias, T, rows, vec);
  KF_CHECK_LAUNCH();
  return KF_OK;
}

// items: rows of the step to process (null = rows 0..T-1); T is then the number of items.
KF_API int kf_attention_generic(const void* q, void* out, int q_dtype, const void* pages, int kv_dtype,
                                const int* items, const int* positions, const int* row_req, const int* block_table, int table_stride,
                                int page_size, int nh, int nkv, int d, float scale, float softcap, int window,
                                int vsplit, int keep_first, int sink, const float* sig_bias, int T, cudaStream_t stream) {
  if (T <= 0) return KF_OK;
  if (d < 1 || d > MAX_D_ALL || nkv < 1 || nh % nkv != 0 || page_size < 1 || !kf_head_map_ok(nh, nkv, vsplit)) return KF_ERR_SIZE;
#define KF_GO1(TQ, TKV, DT, DPT)                                                                              \
  return launch<TQ, TKV, DT, DPT>(q, out, pages, items, positions, row_req, block_table, table_stride, page_size, nh, nkv, d, \
                                  scale, softcap, window, vsplit, window > 0 ? keep_first : 0, sink, sig_bias, T, stream)
#define KF_GO(TQ, TKV) do { if (d <= 64) KF_GO1(TQ, TKV, 64, 1); if (d <= 128) KF_GO1(TQ, TKV, 128, 1); \
                            if (d <= 256) KF_GO1(TQ, TKV, 256, 1); KF_GO1(TQ, TKV, 256, 2); } while (0)
  if (q_dtype == KF_F32 && kv_dtype == KF_F32) KF_GO(float, float);
  if (q_dtype == KF_BF16 && kv_dtype == KF_BF16) KF_GO(__nv_bfloat16, __nv_bfloat16);
  return KF_ERR_DTYPE;
#undef KF_GO
#undef KF_GO1
}
