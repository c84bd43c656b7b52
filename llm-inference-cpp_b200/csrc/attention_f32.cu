// Causal grouped-query attention over the paged cache, 32-bit path: fp32 in, fp32 FMA arithmetic, fp32 out.
//
// Reference: src/model/transformer.cpp:263-282 (score[s] = dot(q, k_s) * scale for s = 0..pos, softmax, sum of p_s v_s).
//
// The order of every addition depends on the keys' absolute positions only, and is the same in both kernels of this file, so a
// position's result does not depend on how a step was cut or batched:
//   * a page is 64 positions anchored at 0, 64, ..; of a page the keys that the query sees (pos - window + 1 .. pos) count;
//   * score = (ascending fmaf chain over the head's entries) * scale; m = the page's largest score, p = exp(score - m),
//     l = ascending sum of p, a = ascending fmaf chain of p * v;
//   * pages join in ascending order: M' = max(M, m), L = L e^(M-M') + l e^(m-M'), A alike; the output is A * (1 / L).
// A page's m, l and a need nothing of the pages before it: that is what lets a decode step work on the pages side by side
// (attention_generic's one warp per query walks them one after another: 290 us a layer for four sequences of 30 to 400 positions
// and 15 heads of 64, prompt and decode steps together; these kernels 91 us for the prompts and 21 us a decode step).
//
//  * attention_f32_decode_kernel: a block per (token, kv head, up to four of its heads), a warp per page, lanes over keys, then
//    over entries;
//  * attention_f32_prompt_kernel: a block per 32 queries and head, a page's 32 x 64 scores and its sums as register tiles.
#include <math.h>

#include "common.cuh"
#include "sm100.cuh"
#include "step_meta.cuh"

namespace llmi {

constexpr int F32_PAGE = 64;
constexpr int F32_HEADS = 4;        // most heads of a block of the decode kernel
constexpr int F32_QUERIES = 32;     // queries of a block of the prompt kernel
constexpr int F32_SMEM_LIMIT = 220 * 1024;

__device__ __forceinline__ void cp_async_f4(float* dst, const float* src, bool real) {
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ float page_base(float m) { return m == -INFINITY ? 0.f : m; }
// the factors with which the running state and a page's sums enter the joined state
__device__ __forceinline__ void join_factors(float& M, float m, float& of_state, float& of_page) {
  const float joined = fmaxf(M, m);
  of_state = M == -INFINITY ? 0.f : expf(__fsub_rn(M, joined));
  of_page = m == -INFINITY ? 0.f : expf(__fsub_rn(m, joined));
  M = joined;
}
__device__ __forceinline__ float joined_sum(float state, float of_state, float page, float of_page) {
  return __fmaf_rn(state, of_state, __fmul_rn(page, of_page));
}

__host__ __device__ constexpr int f32_decode_warps(int hd) { return hd <= 64 ? 8 : 4; }      // at most
__host__ __device__ constexpr long f32_decode_floats(int hd, int heads, int warps) {
  return (long)heads * hd                                  // q
         + (long)warps * F32_PAGE * (hd + 4)               // keys of the warps' pages
         + (long)warps * heads * F32_PAGE                  // p
         + (long)warps * heads * (hd + 2)                  // the pages' a, m, l
         + (long)heads * hd + 2 * heads                    // A, M, L
         + 2L * warps * heads;                             // join factors
}

// NJ: entries of a head per lane (ceil(head_dim / 32)).  HEADS: heads of a block (the last block of a kv head may have fewer): four
// share the reads of a page's values; one or two where the device has SMs to spare, so that a warp's work on a page, which is all
// that a short sequence has, is as long as that of so many heads.  As many warps as a sequence has pages: a block's shared
// memory is theirs, so that several blocks of short sequences fit an SM.
template <int NJ, int HEADS>
__global__ void __launch_bounds__(256)
attention_f32_decode_kernel(const float* __restrict__ q, long ldq, float* __restrict__ out, long ldo, const float* __restrict__ k_cache,
                            const float* __restrict__ v_cache, const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ tok_pos,
                            PagedKV kv, int all_heads, float scale, int window) {
  extern __shared__ __align__(16) float f32_smem[];
  const int hd = kv.head_dim, pitch = hd + 4, n_warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x, t = blockIdx.y;
  const int first = blockIdx.z * HEADS, group = min(HEADS, all_heads - first);      // this block's heads of the kv head's
  float* k_s = f32_smem + warp * F32_PAGE * pitch;
  float* q_s = f32_smem + n_warps * F32_PAGE * pitch;
  float* p_s = q_s + group * hd + warp * HEADS * F32_PAGE;
  float* page_a = q_s + group * hd + n_warps * HEADS * F32_PAGE;          // [warp][group][hd]
  float* page_m = page_a + n_warps * group * hd;                          // [warp][group]
  float* page_l = page_m + n_warps * group;
  float* A = page_l + n_warps * group;                                    // [group][hd]
  float* M = A + group * hd;
  float* L = M + group;
  float* f_state = L + group;                                             // [warp][group]
  float* f_page = f_state + n_warps * group;
  pdl_launch_dependents();
  pdl_wait();

  const int seq = tok_seq[t];
  float* o = out + (size_t)t * ldo + ((size_t)kvh * all_heads + first) * hd;
  if (seq < 0) {
    for (int i = threadIdx.x; i < group * hd; i += blockDim.x) o[i] = 0.f;
    return;
  }
  const int pos = tok_pos[t];
  const int lo = first_visible(pos, window, 0);
  const int first_page = lo / F32_PAGE, last_page = pos / F32_PAGE;
  const float* qp = q + (size_t)t * ldq + ((size_t)kvh * all_heads + first) * hd;
  for (int i = threadIdx.x; i < group * hd; i += blockDim.x) {
    q_s[i] = qp[i];
    A[i] = 0.f;
  }
  for (int j = threadIdx.x; j < group; j += blockDim.x) {
    M[j] = -INFINITY;
    L[j] = 0.f;
  }
  __syncthreads();

  for (int base = first_page; base <= last_page; base += n_warps) {
    const int page = base + warp;
    if (page <= last_page) {
      const int k_lo = max(lo - page * F32_PAGE, 0), k_hi = min(pos - page * F32_PAGE, F32_PAGE - 1);     // keys k_lo..k_hi count
      const size_t at = kv_row_offset(kv, seq, page * F32_PAGE, kvh);
      const float* kp = k_cache + at;
      const float* vp = v_cache + at;
      const int chunks = hd >> 2;
      for (int i = lane; i < F32_PAGE * chunks; i += 32) {
        const int row = i / chunks, c = i - row * chunks;
        if (row >= k_lo && row <= k_hi) cp_async_f4(k_s + row * pitch + 4 * c, kp + row * hd + 4 * c, true);
      }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      const bool in0 = lane >= k_lo && lane <= k_hi, in1 = lane + 32 >= k_lo && lane + 32 <= k_hi;
      for (int j = 0; j < group; ++j) {
        const float* qh = q_s + j * hd;
        const float* k0 = k_s + lane * pitch;
        const float* k1 = k0 + 32 * pitch;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
        for (int d = 0; d < hd; d += 4) {
          const float4 a = *reinterpret_cast<const float4*>(qh + d);
          const float4 x = *reinterpret_cast<const float4*>(k0 + d);
          const float4 y = *reinterpret_cast<const float4*>(k1 + d);
          s0 = fmaf(a.x, x.x, s0);
          s1 = fmaf(a.x, y.x, s1);
          s0 = fmaf(a.y, x.y, s0);
          s1 = fmaf(a.y, y.y, s1);
          s0 = fmaf(a.z, x.z, s0);
          s1 = fmaf(a.z, y.z, s1);
          s0 = fmaf(a.w, x.w, s0);
          s1 = fmaf(a.w, y.w, s1);
        }
        s0 = in0 ? __fmul_rn(s0, scale) : -INFINITY;      // (rows of the tile that no key is in are never used)
        s1 = in1 ? __fmul_rn(s1, scale) : -INFINITY;
        const float m = warp_max(fmaxf(s0, s1)), mb = page_base(m);
        p_s[j * F32_PAGE + lane] = in0 ? expf(__fsub_rn(s0, mb)) : 0.f;
        p_s[j * F32_PAGE + lane + 32] = in1 ? expf(__fsub_rn(s1, mb)) : 0.f;
        if (lane == 0) page_m[warp * group + j] = m;
      }
      __syncwarp();
      float acc[HEADS][NJ], l[HEADS];
#pragma unroll
      for (int j = 0; j < HEADS; ++j) {
        l[j] = 0.f;
#pragma unroll
        for (int e = 0; e < NJ; ++e) acc[j][e] = 0.f;
      }
      const int n_keys = k_hi + 1;
#pragma unroll 8
      for (int kk = k_lo; kk < n_keys; ++kk) {
        float v[NJ];
#pragma unroll
        for (int e = 0; e < NJ; ++e) v[e] = lane + 32 * e < hd ? vp[kk * hd + lane + 32 * e] : 0.f;
#pragma unroll
        for (int j = 0; j < HEADS; ++j) {
          const float p = p_s[j * F32_PAGE + kk];           // (heads beyond the group: stale numbers that nobody reads on)
          l[j] = __fadd_rn(l[j], p);
#pragma unroll
          for (int e = 0; e < NJ; ++e) acc[j][e] = fmaf(p, v[e], acc[j][e]);
        }
      }
#pragma unroll
      for (int j = 0; j < HEADS; ++j) {
        if (j >= group) continue;
        if (lane == 0) page_l[warp * group + j] = l[j];
#pragma unroll
        for (int e = 0; e < NJ; ++e)
          if (lane + 32 * e < hd) page_a[(warp * group + j) * hd + lane + 32 * e] = acc[j][e];
      }
      __syncwarp();
    }
    __syncthreads();
    const int here = min(n_warps, last_page - base + 1);
    for (int j = threadIdx.x; j < group; j += blockDim.x) {
      float m_run = M[j], l_run = L[j];
      for (int w = 0; w < here; ++w) {
        float fs, fp;
        join_factors(m_run, page_m[w * group + j], fs, fp);
        l_run = joined_sum(l_run, fs, page_l[w * group + j], fp);
        f_state[w * group + j] = fs;
        f_page[w * group + j] = fp;
      }
      M[j] = m_run;
      L[j] = l_run;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < group * hd; i += blockDim.x) {
      const int j = i / hd;
      float a = A[i];
      for (int w = 0; w < here; ++w) a = joined_sum(a, f_state[w * group + j], page_a[w * group * hd + i], f_page[w * group + j]);
      A[i] = a;
    }
    // (a thread reads only its own A before the next round's second barrier; the pages' sums are written behind the barrier below)
    __syncthreads();
  }
  for (int i = threadIdx.x; i < group * hd; i += blockDim.x) o[i] = __fmul_rn(A[i], __fdiv_rn(1.0f, L[i / hd]));
}

__host__ __device__ constexpr long f32_prompt_floats(int hd) {
  return (long)(F32_QUERIES + 2 * F32_PAGE) * (hd + 4) + (long)F32_QUERIES * (F32_PAGE + 4);
}

// NV: pieces of four entries per thread (ceil(head_dim / 64)).
template <int NV>
__global__ void __launch_bounds__(128)
attention_f32_prompt_kernel(const float* __restrict__ q, long ldq, float* __restrict__ out, long ldo, const float* __restrict__ k_cache,
                            const float* __restrict__ v_cache, const int32_t* __restrict__ tok_pos, const int32_t* __restrict__ seq_q_start,
                            int n_seqs, PagedKV kv, int n_heads, float scale, int window) {
  extern __shared__ __align__(16) float f32_smem[];
  __shared__ int job_seq, job_block;
  const int hd = kv.head_dim, pitch = hd + 4;
  float* q_s = f32_smem;                                   // [32][pitch]
  float* k_s = q_s + F32_QUERIES * pitch;                  // [64][pitch]
  float* v_s = k_s + F32_PAGE * pitch;
  float* p_s = v_s + F32_PAGE * pitch;                     // [32][68]
  constexpr int PP = F32_PAGE + 4;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int h = blockIdx.x % n_heads, job = blockIdx.x / n_heads;
  pdl_launch_dependents();
  pdl_wait();
  // which 32 queries: block `job` of the sequences' blocks, counted in sequence order
  if (tid < 32) {
    if (tid == 0) job_seq = -1;
    __syncwarp();
    int before = 0;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
      const int s = s0 + tid;
      const int n = s < n_seqs ? (seq_q_start[s + 1] - seq_q_start[s] + F32_QUERIES - 1) / F32_QUERIES : 0;
      int incl = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (tid >= d) incl += up;
      }
      if (n > 0 && job >= before + incl - n && job < before + incl) {
        job_seq = s;
        job_block = job - (before + incl - n);
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
      if (job < before) break;
    }
  }
  __syncthreads();
  const int seq = job_seq;
  if (seq < 0) return;
  const int t0 = seq_q_start[seq] + job_block * F32_QUERIES;
  const int n_q = min(F32_QUERIES, seq_q_start[seq + 1] - t0);
  const int pos0 = tok_pos[t0];                            // the queries' positions are pos0, pos0 + 1, ..
  const int kvh = h / (n_heads / kv.n_kv_heads);
  const int chunks = hd >> 2;
  for (int i = tid; i < F32_QUERIES * chunks; i += 128) {
    const int r = i / chunks, c = i - r * chunks;
    const float4 z = r < n_q ? *reinterpret_cast<const float4*>(q + (size_t)(t0 + r) * ldq + (size_t)h * hd + 4 * c) : make_float4(0, 0, 0, 0);
    *reinterpret_cast<float4*>(q_s + r * pitch + 4 * c) = z;
  }
  float A[4][4 * NV], M[4], L[4];
  int lo[4], hi[4];                                        // positions that row ty + 8 i sees
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    M[i] = -INFINITY;
    L[i] = 0.f;
    const int r = ty + 8 * i;
    hi[i] = r < n_q ? pos0 + r : -1;
    lo[i] = r < n_q ? first_visible(pos0 + r, window, 0) : 0;
#pragma unroll
    for (int e = 0; e < 4 * NV; ++e) A[i][e] = 0.f;
  }
  const int last = pos0 + n_q - 1;
  const int lo_first = first_visible(pos0, window, 0), lo_last = first_visible(last, window, 0);
  for (int page = lo_first / F32_PAGE; page <= last / F32_PAGE; ++page) {
    const int key0 = page * F32_PAGE, n_keys = min(F32_PAGE, last - key0 + 1);
    const size_t at = kv_row_offset(kv, seq, key0, kvh);
    __syncthreads();                                       // nobody reads the page before any more
    for (int i = tid; i < F32_PAGE * chunks; i += 128) {
      const int r = i / chunks, c = i - r * chunks;
      cp_async_f4(k_s + r * pitch + 4 * c, k_cache + at + (r < n_keys ? r * hd + 4 * c : 0), r < n_keys);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = tid; i < F32_PAGE * chunks; i += 128) {
      const int r = i / chunks, c = i - r * chunks;
      cp_async_f4(v_s + r * pitch + 4 * c, v_cache + at + (r < n_keys ? r * hd + 4 * c : 0), r < n_keys);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    float s[4][4];                                         // row ty + 8 i, key tx + 16 j
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
    for (int d = 0; d < hd; d += 4) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(q_s + (ty + 8 * i) * pitch + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(k_s + (tx + 16 * j) * pitch + d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          s[i][j] = fmaf(a[i].x, b.x, s[i][j]);
          s[i][j] = fmaf(a[i].y, b.y, s[i][j]);
          s[i][j] = fmaf(a[i].z, b.z, s[i][j]);
          s[i][j] = fmaf(a[i].w, b.w, s[i][j]);
        }
      }
    }
    const bool whole = n_q == F32_QUERIES && key0 >= lo_last && key0 + F32_PAGE - 1 <= pos0;     // every query sees every key
    float m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = key0 + tx + 16 * j;
        s[i][j] = whole || (key >= lo[i] && key <= hi[i]) ? __fmul_rn(s[i][j], scale) : -INFINITY;
        m[i] = fmaxf(m[i], s[i][j]);
      }
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], d));
      const float mb = page_base(m[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = key0 + tx + 16 * j;
        p_s[(ty + 8 * i) * PP + tx + 16 * j] = whole || (key >= lo[i] && key <= hi[i]) ? expf(__fsub_rn(s[i][j], mb)) : 0.f;
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float a[4][4 * NV], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      l[i] = 0.f;
#pragma unroll
      for (int e = 0; e < 4 * NV; ++e) a[i][e] = 0.f;
    }
    for (int kk = 0; kk < n_keys; kk += 4) {
      float4 p4[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) p4[i] = *reinterpret_cast<const float4*>(p_s + (ty + 8 * i) * PP + kk);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 v[NV];
#pragma unroll
        for (int e = 0; e < NV; ++e)
          v[e] = 4 * tx + 64 * e < hd ? *reinterpret_cast<const float4*>(v_s + (kk + u) * pitch + 4 * tx + 64 * e) : make_float4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float p = u == 0 ? p4[i].x : u == 1 ? p4[i].y : u == 2 ? p4[i].z : p4[i].w;
          const int key = key0 + kk + u;
          if (whole || (key >= lo[i] && key <= hi[i])) {   // (a key that is not seen leaves the sums alone, whatever its row holds)
            l[i] = __fadd_rn(l[i], p);
#pragma unroll
            for (int e = 0; e < NV; ++e) {
              a[i][4 * e] = fmaf(p, v[e].x, a[i][4 * e]);
              a[i][4 * e + 1] = fmaf(p, v[e].y, a[i][4 * e + 1]);
              a[i][4 * e + 2] = fmaf(p, v[e].z, a[i][4 * e + 2]);
              a[i][4 * e + 3] = fmaf(p, v[e].w, a[i][4 * e + 3]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float fs, fp;
      join_factors(M[i], m[i], fs, fp);
      L[i] = joined_sum(L[i], fs, l[i], fp);
#pragma unroll
      for (int e = 0; e < 4 * NV; ++e) A[i][e] = joined_sum(A[i][e], fs, a[i][e], fp);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty + 8 * i;
    if (r >= n_q) continue;
    const float inv = __fdiv_rn(1.0f, L[i]);
#pragma unroll
    for (int e = 0; e < NV; ++e) {
      const int d = 4 * tx + 64 * e;
      if (d < hd)
        *reinterpret_cast<float4*>(out + (size_t)(t0 + r) * ldo + (size_t)h * hd + d) =
            make_float4(__fmul_rn(A[i][4 * e], inv), __fmul_rn(A[i][4 * e + 1], inv), __fmul_rn(A[i][4 * e + 2], inv), __fmul_rn(A[i][4 * e + 3], inv));
    }
  }
}

// Head sizes in whole 16-byte pieces up to 128; the generic kernel has the rest.
inline bool attention_f32_takes(int hd, int group) { return hd > 0 && hd <= 128 && hd % 4 == 0 && group > 0; }
static_assert(f32_decode_floats(64, F32_HEADS, f32_decode_warps(64)) * 4 <= F32_SMEM_LIMIT && f32_decode_floats(128, F32_HEADS, f32_decode_warps(128)) * 4 <= F32_SMEM_LIMIT);

template <typename K>
int f32_configure(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F32_SMEM_LIMIT) == cudaSuccess ? LLMI_OK : LLMI_ERR_LAUNCH;
}

template <int NJ>
int f32_configure_decode() {
  int rc = f32_configure(attention_f32_decode_kernel<NJ, 1>);
  if (rc == LLMI_OK) rc = f32_configure(attention_f32_decode_kernel<NJ, 2>);
  return rc == LLMI_OK ? f32_configure(attention_f32_decode_kernel<NJ, F32_HEADS>) : rc;
}

}  // namespace llmi

using namespace llmi;

LLMI_EXPORT int llmi_attention_f32_supported(int head_dim, int group) { return attention_f32_takes(head_dim, group) ? 1 : 0; }

// fp32 q [n_tokens, >= n_heads * head_dim] (row pitch ldq), out (row pitch ldo), caches of pages of 64.  `decode` 1: token by token
// (tok_seq -1: a row of zeros), max_pages: most pages that a token sees (0: not known); 0: the tokens of the sequences one after
// another as seq_q_start says, no padding rows.  Both may take a prompt.
LLMI_EXPORT int llmi_attention_f32(const float* q, long ldq, float* out, long ldo, const float* k_cache, const float* v_cache,
                                   const int32_t* tok_seq, const int32_t* tok_pos, const int32_t* seq_pages, int pages_stride, int page_size,
                                   const int32_t* seq_q_start, int n_seqs, int n_tokens, int decode, int max_pages, int n_heads,
                                   int n_kv_heads, int head_dim, float scale, int window, cudaStream_t stream) {
  if (n_tokens <= 0 || n_seqs <= 0 || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads != 0) return LLMI_ERR_BAD_SIZE;
  const int group = n_heads / n_kv_heads;
  if (page_size != F32_PAGE || !attention_f32_takes(head_dim, group)) return LLMI_ERR_UNSUPPORTED;
  if ((((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15) || ((ldq | ldo) & 3)) return LLMI_ERR_ALIGN;
  PagedKV kv{seq_pages, pages_stride, page_size, n_kv_heads, head_dim};
  static PerDevice<bool> configured;
  if (!configured.here()) {
    int rc = f32_configure_decode<1>();
    if (rc == LLMI_OK) rc = f32_configure_decode<2>();
    if (rc == LLMI_OK) rc = f32_configure_decode<4>();
    if (rc == LLMI_OK) rc = f32_configure(attention_f32_prompt_kernel<1>);
    if (rc == LLMI_OK) rc = f32_configure(attention_f32_prompt_kernel<2>);
    if (rc != LLMI_OK) return rc;
    configured.here() = true;
  }
  if (decode) {
    if (n_tokens > 65535) return LLMI_ERR_BAD_SIZE;
    int heads = 1;
    while (heads < F32_HEADS && heads < group && (long)n_tokens * n_kv_heads * ((group + heads - 1) / heads) > sm_count()) heads *= 2;
    const int splits = (group + heads - 1) / heads, most = f32_decode_warps(head_dim);
    if (splits > 65535) return LLMI_ERR_BAD_SIZE;
    const int warps = max_pages > 0 && max_pages < most ? max_pages : most;
    const dim3 grid(n_kv_heads, n_tokens, splits), block(32 * warps);
    const size_t smem = f32_decode_floats(head_dim, heads, warps) * sizeof(float);
#define LLMI_LAUNCH_HEADS(NJ, HEADS)                                                                                                    \
  launch_pdl(PDL_SMALL, attention_f32_decode_kernel<NJ, HEADS>, grid, block, smem, stream, q, ldq, out, ldo, k_cache, v_cache, tok_seq, \
             tok_pos, kv, group, scale, window)
#define LLMI_LAUNCH(NJ) (heads == 1 ? LLMI_LAUNCH_HEADS(NJ, 1) : heads == 2 ? LLMI_LAUNCH_HEADS(NJ, 2) : LLMI_LAUNCH_HEADS(NJ, F32_HEADS))
    if (head_dim <= 32) return LLMI_LAUNCH(1);
    if (head_dim <= 64) return LLMI_LAUNCH(2);
    return LLMI_LAUNCH(4);
#undef LLMI_LAUNCH
#undef LLMI_LAUNCH_HEADS
  }
  const long blocks = (long)(n_tokens / F32_QUERIES + n_seqs) * n_heads;      // at most so many blocks of 32 queries
  if (blocks > 0x7fffffffL) return LLMI_ERR_BAD_SIZE;
  const size_t smem = f32_prompt_floats(head_dim) * sizeof(float);
#define LLMI_LAUNCH(NV)                                                                                                              \
  launch_pdl(PDL_SMALL, attention_f32_prompt_kernel<NV>, dim3((unsigned)blocks), dim3(128), smem, stream, q, ldq, out, ldo, k_cache, \
             v_cache, tok_pos, seq_q_start, n_seqs, kv, n_heads, scale, window)
  return head_dim <= 64 ? LLMI_LAUNCH(1) : LLMI_LAUNCH(2);
#undef LLMI_LAUNCH
}
