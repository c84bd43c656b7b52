// A delta rule in its general form: a recurrent mixer whose per-head state S [D, Dv] changes per token by a diagonal
// decay plus a rank-one term, both read from the OLD state, and a write:
//     S <- diag(w) S + m (pᵀ S) + k vᵀ ;        o = Sᵀ r
// w, m, p, k, r are vectors over the D key channels, v over the Dv value channels.  With p = u (the unit key),
// m = -(a * u) and w a decay per channel this is the rule whose removal acts along the key's direction only
// (llmi_gdelta_prepare makes exactly these); other rules of the family differ in how w, m, p are made.
// Column j of S evolves alone:  s_j <- w * s_j + m (p . s_j) + k v_j,  o_j = s_j . r — so the state is kept column by
// column ([head][column][entry], fp32, one row of the cache's state slab per slot) and columns are spread over threads.
//
// Everything here is fp32 arithmetic.  Kernels, in the order of a step:
//   llmi_gdelta_prepare     per (token, head): the decay from a low-rank path, the removal rate, the unit key
//   llmi_dplr_recurrence    per (sequence, head, slice of columns): the recurrence over the step's tokens
//   (llmi_delta_finish of delta_rule.cu then norms and gates o)
// The recurrence treats a column alone and only continues what the slab holds: the result does not depend on how a
// prompt was cut or on what else is in the batch.
#include <math.h>

#include "common.cuh"
#include "recurrence.cuh"

namespace llmi {

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }

// dst = tanh(src) row by row (the input of the low-rank path's second product).
template <typename T>
__global__ void __launch_bounds__(256)
tanh_rows_kernel(const float* __restrict__ src, long ld, T* __restrict__ dst, int R, long total) {
  pdl_launch_dependents();
  pdl_wait();
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const long t = i / R;
    dst[i] = from_f32<T>(tanhf(src[t * ld + (i - t * R)]));
  }
}

// `proj`, one fp32 row per token:  [ r (H*D) | k (H*D) | v (H*Dv) | a (H*D) | gate (H*Dv) | low (R) ].
// `prep`, one fp32 row per token:  [ w (H*D) | p (H*D) | m (H*D) ]:
//   w = exp(-exp(-1/2) * sigmoid(w0 + W2 tanh(low)))   (W2 as w2t [R, H*D] fp32: neighbouring threads read neighbours)
//   p = k / sqrt(sum_head(k^2) + 1e-6),   m = -sigmoid(a + a_bias) * p
// With `z` (fp32 [T, ldz], the product W2 tanh(low) made by a matrix product beforehand: the way of a step of many
// tokens) the kernel adds w0 to it instead of walking the R entries itself.
__global__ void __launch_bounds__(128)
gdelta_prepare_kernel(const float* __restrict__ proj, long ld, int H, int D, int Dv, int R, const float* __restrict__ w2t,
                      const float* __restrict__ z_all, long ldz, const float* __restrict__ w0,
                      const float* __restrict__ a_bias, const int32_t* __restrict__ tok_seq, float* __restrict__ prep, long ldp) {
  extern __shared__ float low_s[];                       // tanh of the low-rank path's R entries
  __shared__ float scratch[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  if (tok_seq[t] < 0) return;
  const int HD = H * D;
  const float* row = proj + (size_t)t * ld;
  const float* low = row + 3 * (size_t)HD + 2 * (size_t)H * Dv;
  if (!z_all)
    for (int j = threadIdx.x; j < R; j += blockDim.x) low_s[j] = tanhf(low[j]);
  const float* k = row + HD + (size_t)h * D;
  float ss = 0.f;
  for (int d = threadIdx.x; d < D; d += blockDim.x) ss = fmaf(k[d], k[d], ss);
  ss = block_sum(ss, scratch);                           // (its barriers also publish low_s)
  const float inv = 1.0f / sqrtf(ss + 1e-6f);
  float* out = prep + (size_t)t * ldp + (size_t)h * D;
  const float* a = row + 2 * (size_t)HD + (size_t)H * Dv + (size_t)h * D;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const int c = h * D + d;
    float z = w0[c];
    if (z_all) {
      z += z_all[(size_t)t * ldz + c];
    } else {
      for (int j = 0; j < R; ++j) z = fmaf(w2t[(size_t)j * HD + c], low_s[j], z);
    }
    const float u = k[d] * inv;
    out[d] = expf(-0.6065306597126334f * sigmoid_f(z));
    out[HD + d] = u;
    out[2 * (size_t)HD + d] = -sigmoid_f(a[d] + a_bias[c]) * u;
  }
}

// The same for heads of 32, 64 or 128 entries on 16-byte rows, four entries a thread.  Many tokens (z given): D / 4 threads a head,
// a token's heads side by side (3,000 tokens of 32 heads of 64: 27 us, 100 with a block per token and head and an entry
// a thread).  A few: a block per (token, head) whose 128 threads cut the R rows of W2 into 512 / D segments of equal length, so
// that a row's loads are not behind one another (two tokens of 32 heads, R = 128: 2.9 us, 6.9 with one thread walking all rows);
// the segments' sums are added in ascending order behind w0.
__device__ __forceinline__ float4 gdelta_four(const float4& k, const float4& a, const float4& b, const float4& z, float inv, float4& u, float4& m) {
  u = make_float4(k.x * inv, k.y * inv, k.z * inv, k.w * inv);
  m = make_float4(-sigmoid_f(a.x + b.x) * u.x, -sigmoid_f(a.y + b.y) * u.y, -sigmoid_f(a.z + b.z) * u.z, -sigmoid_f(a.w + b.w) * u.w);
  const float c = -0.6065306597126334f;
  return make_float4(expf(c * sigmoid_f(z.x)), expf(c * sigmoid_f(z.y)), expf(c * sigmoid_f(z.z)), expf(c * sigmoid_f(z.w)));
}
// 1 / |k| of a head that L = D / 4 neighbouring lanes hold
template <int L>
__device__ __forceinline__ float gdelta_inverse(const float4& k) {
  float ss = fmaf(k.w, k.w, fmaf(k.z, k.z, fmaf(k.y, k.y, k.x * k.x)));
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  return 1.0f / sqrtf(ss + 1e-6f);
}

template <int D>
__global__ void __launch_bounds__(256)
gdelta_prepare_rows_kernel(const float* __restrict__ proj, long ld, int H, int Dv, const float* __restrict__ z_all, long ldz,
                           const float* __restrict__ w0, const float* __restrict__ a_bias, const int32_t* __restrict__ tok_seq,
                           float* __restrict__ prep, long ldp) {
  pdl_launch_dependents();
  const int t = blockIdx.x, HD = H * D, c = 4 * (blockIdx.y * 256 + threadIdx.x), at = c < HD ? c : 0;
  pdl_wait();
  if (tok_seq[t] < 0) return;
  const float* row = proj + (size_t)t * ld;
  const float4 k = *reinterpret_cast<const float4*>(row + HD + at);
  const float4 a = *reinterpret_cast<const float4*>(row + 2 * (size_t)HD + (size_t)H * Dv + at);
  const float4 zz = *reinterpret_cast<const float4*>(z_all + (size_t)t * ldz + at);
  const float4 b = *reinterpret_cast<const float4*>(a_bias + at), z0 = *reinterpret_cast<const float4*>(w0 + at);
  const float inv = gdelta_inverse<D / 4>(k);                 // (every lane takes part; a head's lanes are all in range or all not)
  if (c >= HD) return;
  float4 u, m;
  const float4 w = gdelta_four(k, a, b, make_float4(z0.x + zz.x, z0.y + zz.y, z0.z + zz.z, z0.w + zz.w), inv, u, m);
  float* out = prep + (size_t)t * ldp + c;
  *reinterpret_cast<float4*>(out) = w;
  *reinterpret_cast<float4*>(out + HD) = u;
  *reinterpret_cast<float4*>(out + 2 * (size_t)HD) = m;
}

template <int D>
__global__ void __launch_bounds__(128)
gdelta_prepare_walk_kernel(const float* __restrict__ proj, long ld, int H, int Dv, int R, const float* __restrict__ w2t,
                           const float* __restrict__ w0, const float* __restrict__ a_bias, const int32_t* __restrict__ tok_seq,
                           float* __restrict__ prep, long ldp) {
  constexpr int L = D / 4, SEGS = 128 / L, AHEAD = 16;
  extern __shared__ __align__(16) float low_s[];              // tanh of the low-rank path's R entries
  __shared__ float4 part[SEGS][L];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y, HD = H * D;
  if (tok_seq[t] < 0) return;
  const int lane = threadIdx.x % L, seg = threadIdx.x / L, c = h * D + 4 * lane;
  const int per = (R + SEGS - 1) / SEGS, j0 = min(R, seg * per), j1 = min(R, j0 + per);
  const float* row = proj + (size_t)t * ld;
  const float4 k = *reinterpret_cast<const float4*>(row + HD + c);
  const float4 a = *reinterpret_cast<const float4*>(row + 2 * (size_t)HD + (size_t)H * Dv + c);
  const float4 b = *reinterpret_cast<const float4*>(a_bias + c), z0 = *reinterpret_cast<const float4*>(w0 + c);
  const float* low = row + 3 * (size_t)HD + 2 * (size_t)H * Dv;
  float4 w[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (j0 + i < j1) w[i] = *reinterpret_cast<const float4*>(w2t + (size_t)(j0 + i) * HD + c);
  for (int j = threadIdx.x; j < R; j += 128) low_s[j] = tanhf(low[j]);
  __syncthreads();
  float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = j0; j < j1; j += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (j + i < j1) {
        const float l = low_s[j + i];
        z.x = fmaf(w[i].x, l, z.x); z.y = fmaf(w[i].y, l, z.y); z.z = fmaf(w[i].z, l, z.z); z.w = fmaf(w[i].w, l, z.w);
      }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (j + AHEAD + i < j1) w[i] = *reinterpret_cast<const float4*>(w2t + (size_t)(j + AHEAD + i) * HD + c);
  }
  part[seg][lane] = z;
  __syncthreads();
  const float inv = gdelta_inverse<L>(k);
  if (seg > 0) return;
  z = z0;
#pragma unroll
  for (int s = 0; s < SEGS; ++s) {
    const float4 v = part[s][lane];
    z = make_float4(z.x + v.x, z.y + v.y, z.z + v.z, z.w + v.w);
  }
  float4 u, m;
  const float4 decay = gdelta_four(k, a, b, z, inv, u, m);
  float* out = prep + (size_t)t * ldp + c;
  *reinterpret_cast<float4*>(out) = decay;
  *reinterpret_cast<float4*>(out + HD) = u;
  *reinterpret_cast<float4*>(out + 2 * (size_t)HD) = m;
}

template <int D>
int launch_gdelta_fours(const float* proj, long ld, int H, int Dv, int R, const float* w2t, const float* z, long ldz, const float* w0,
                        const float* a_bias, const int32_t* tok_seq, float* prep, long ldp, int n_tokens, cudaStream_t stream) {
  if (z)
    return launch_pdl(PDL_SMALL, gdelta_prepare_rows_kernel<D>, dim3(n_tokens, (H * D + 1023) / 1024), dim3(256), 0, stream, proj, ld, H, Dv, z,
                      ldz, w0, a_bias, tok_seq, prep, ldp);
  return launch_pdl(PDL_SMALL, gdelta_prepare_walk_kernel<D>, dim3(n_tokens, H), dim3(128), (size_t)R * sizeof(float), stream, proj, ld, H, Dv, R,
                    w2t, w0, a_bias, tok_seq, prep, ldp);
}

// The general form: one block per (head, sequence), one thread per column j of S, the column in shared memory
// (S_s[d][cols]: no two threads share a bank); any D and Dv.  The vectors of the next token are fetched while the
// current one is computed (two buffers, one barrier per token).
__global__ void __launch_bounds__(1024)
dplr_recurrence_kernel(const float* __restrict__ proj, long ld, const float* __restrict__ prep, long ldp, int H, int D,
                       int Dv, float* __restrict__ state, long state_stride, const int32_t* __restrict__ seq_q_start,
                       const int32_t* __restrict__ seq_slot, float* __restrict__ o_raw, long ldo, int write_state) {
  extern __shared__ float sm[];
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.x, seq = blockIdx.y;
  const int slot = seq_slot[seq];
  if (slot < 0) return;
  const int r0 = seq_q_start[seq], n = seq_q_start[seq + 1] - r0;
  if (n <= 0) return;
  const int cols = blockDim.x;                               // Dv rounded up to whole warps
  const int j = threadIdx.x;
  const bool live = j < Dv;
  float* vec = sm;                                           // [2][5*D]: w, p, m, k, r of a token
  float* S_s = sm + 10 * D;                                  // [D][cols]
  const int HD = H * D;
  float* S_g = state + (size_t)slot * state_stride + (size_t)h * D * Dv;
  if (live)
    for (int d = 0; d < D; ++d) S_s[(size_t)d * cols + j] = S_g[(size_t)j * D + d];
  auto fetch = [&](int i, int buf) {
    const float* pr = prep + (size_t)(r0 + i) * ldp + (size_t)h * D;
    const float* xr = proj + (size_t)(r0 + i) * ld + (size_t)h * D;
    float* dst = vec + buf * 5 * D;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
      dst[d] = pr[d];
      dst[D + d] = pr[HD + d];
      dst[2 * D + d] = pr[2 * (size_t)HD + d];
      dst[3 * D + d] = xr[HD + d];
      dst[4 * D + d] = xr[d];
    }
  };
  fetch(0, 0);
  for (int i = 0; i < n; ++i) {
    __syncthreads();                                         // buffer i&1 is filled; the other one is read out
    if (i + 1 < n) fetch(i + 1, (i + 1) & 1);
    if (!live) continue;
    const float v = proj[(size_t)(r0 + i) * ld + 2 * (size_t)HD + (size_t)h * Dv + j];
    const float* w = vec + (i & 1) * 5 * D;
    const float *p = w + D, *m = w + 2 * D, *k = w + 3 * D, *r = w + 4 * D;
    float dot = 0.f;
    for (int d = 0; d < D; ++d) dot = fmaf(S_s[(size_t)d * cols + j], p[d], dot);
    float o = 0.f;
    for (int d = 0; d < D; ++d) {
      const float s = fmaf(k[d], v, fmaf(m[d], dot, w[d] * S_s[(size_t)d * cols + j]));
      S_s[(size_t)d * cols + j] = s;
      o = fmaf(s, r[d], o);
    }
    o_raw[(size_t)(r0 + i) * ldo + (size_t)h * Dv + j] = o;
  }
  if (live && write_state)
    for (int d = 0; d < D; ++d) S_g[(size_t)j * D + d] = S_s[(size_t)d * cols + j];
}

// The form for D = 32, 64, 128 and Dv a multiple of 16.  A thread holds TWO neighbouring columns of S and a sixteenth
// of their entries (lane `sub` of sixteen: d = 64 i + 4 sub + 0..3, while d < D) in registers, as pairs of entries; partial
// sums over d are joined by join_four, a token's p . S beside the token before's S . r.  The recurrence is a chain over the
// tokens, so the work of a token is spread thin (16 columns a warp), a head's columns are cut into slices of 32 (or 16),
// every slice a block of its own (blockIdx.z), and what a token needs — w, p, m, k, r of the head, the slice's v — is
// copied into a ring of REC_STAGES batches of REC_BATCH tokens (cp.async, 16 bytes a copy, each thread's places worked out
// once), so that no load's latency lies on the chain from token to token; one barrier per batch.  (Two tokens per round of
// shuffles — the second one's sum over the state follows from the state before the first, (p_B * w_A) . S + (p_B . m_A)(p_A .
// S) + (p_B . k_A) v_A — was measured slower, 1.10 against 0.96 ms for 2,048 tokens: the time of a token is its
// instructions.)
// 1,300 tokens, two sequences, 32 heads of 64: 442 -> 251 ns a token; six of 400 1,094 -> 481 (same bits).
template <int D>
__global__ void __launch_bounds__(256)
dplr_recurrence_quad_kernel(const float* __restrict__ proj, long ld, const float* __restrict__ prep, long ldp, int H, int Dv,
                            float* __restrict__ state, long state_stride, const int32_t* __restrict__ seq_q_start,
                            const int32_t* __restrict__ seq_slot, float* __restrict__ o_raw, long ldo, int write_state) {
  extern __shared__ __align__(16) float sm[];
  const int h = blockIdx.x, seq = blockIdx.y;
  const int slot = seq_slot[seq];
  if (slot < 0) return;
  const int r0 = seq_q_start[seq], n = seq_q_start[seq + 1] - r0;
  if (n <= 0) return;
  constexpr int NI = (D + 63) / 64;                          // chunks of four entries per lane (D = 32: lanes 8..15 hold none)
  const int CB = blockDim.x >> 3;                            // columns of this block's slice (the launcher gives 8 CB threads)
  const int cg = threadIdx.x >> 4, sub = threadIdx.x & 15;   // my columns: col0, col0 + 1
  const int col0 = blockIdx.z * CB + 2 * cg;
  const bool holds = 4 * sub < D;
  const int HD = H * D;
  float* S_g = state + (size_t)slot * state_stride + (size_t)h * D * Dv + (size_t)col0 * D;     // [column][entry]
  // a token's place in the ring: [w | p | m | k | r (D each) | v of the slice (CB)]; all parts are whole 16-byte pieces
  constexpr int Q = D / 4;                                   // 16-byte pieces of one vector
  const int pieces = 5 * Q + CB / 4, pitch = 5 * D + CB;
  // My copies: piece (threadIdx.x + r blockDim.x) of a batch, counted over its tokens.  (CB = 16, D = 128: 4 x 164 pieces for
  // 128 threads.)
  constexpr int COPIES = 6;
  static_assert(REC_BATCH * (5 * Q + 4) <= COPIES * 128 && REC_BATCH * (5 * Q + 8) <= COPIES * 256, "every piece of a batch is somebody's copy");
  const float* src[COPIES];
  int dst[COPIES], of_token[COPIES];
#pragma unroll
  for (int r = 0; r < COPIES; ++r) {
    const int x = threadIdx.x + r * blockDim.x, u = x / pieces, e = x - u * pieces;
    of_token[r] = u < REC_BATCH ? u : 0x7fffffff / 2;        // (behind every sequence's end: never copied)
    const int tok = u < REC_BATCH ? u : 0, part = e / Q, off = 4 * (e - part * Q);
    const float* prow = prep + (size_t)(r0 + tok) * ldp + (size_t)h * D;
    const float* xrow = proj + (size_t)(r0 + tok) * ld;
    dst[r] = tok * pitch + 4 * e;
    if (part < 3) src[r] = prow + (size_t)part * HD + off;                                       // w, p, m
    else if (part == 3) src[r] = xrow + (size_t)h * D + HD + off;                               // k
    else if (part == 4) src[r] = xrow + (size_t)h * D + off;                                     // r
    else src[r] = xrow + 2 * (size_t)HD + (size_t)h * Dv + blockIdx.z * CB + 4 * (e - 5 * Q);
    if (part < 3) dst[r] |= 1 << 30;                         // from prep
  }
  const int stage_floats = REC_BATCH * pitch;
  const size_t advance_p = (size_t)REC_BATCH * ldp, advance_x = (size_t)REC_BATCH * ld;
  int asked = 0;                                             // tokens asked for so far (whole batches)
  auto issue = [&](int stage) {
    float* base = sm + stage * stage_floats;
#pragma unroll
    for (int r = 0; r < COPIES; ++r) {
      if (asked + of_token[r] < n) rec_copy16(base + (dst[r] & ~(1 << 30)), src[r]);
      src[r] += (dst[r] >> 30) ? advance_p : advance_x;
    }
    asked += REC_BATCH;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_wait();                                                // (so far: the step's sizes and this thread's places only)
  pdl_launch_dependents();
#pragma unroll
  for (int s = 0; s < REC_STAGES - 1; ++s) issue(s);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 S_r[2][NI][2];                                      // [column][chunk][pair of entries]
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const float4 v = holds ? *reinterpret_cast<const float4*>(S_g + c * D + 64 * i + 4 * sub) : zero;
      S_r[c][i][0] = make_float2(v.x, v.y);
      S_r[c][i][1] = make_float2(v.z, v.w);
    }
  float2 o_pend = make_float2(0.f, 0.f);                     // my parts of the token before's S . r, of both columns
  float* o_at = o_raw + (size_t)r0 * ldo + (size_t)h * Dv + col0 + (sub & 1);      // (lanes sub = 2, 3 write)
  int stage = 0;
  for (int i0 = 0; i0 < n; i0 += REC_BATCH) {
    asm volatile("cp.async.wait_group %0;" ::"n"(REC_STAGES - 2) : "memory");
    __syncthreads();                                         // this batch is there; the one before is read out
    issue(stage == 0 ? REC_STAGES - 1 : stage - 1);
    const float* in = sm + stage * stage_floats;
    stage = stage == REC_STAGES - 1 ? 0 : stage + 1;
    const int here = min(REC_BATCH, n - i0);
#pragma unroll
    for (int u = 0; u < REC_BATCH; ++u, in += pitch) {
      if (u >= here) break;
      float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < NI; ++c) {
        const float4 pp = holds ? *reinterpret_cast<const float4*>(in + D + 64 * c + 4 * sub) : zero;
#pragma unroll
        for (int col = 0; col < 2; ++col) {
          acc[col] = __ffma2_rn(S_r[col][c][0], make_float2(pp.x, pp.y), acc[col]);
          acc[col] = __ffma2_rn(S_r[col][c][1], make_float2(pp.z, pp.w), acc[col]);
        }
      }
      float dx = pair_sum(acc[0]), dy = pair_sum(acc[1]);
      const float o_before = join_four(dx, dy, o_pend.x, o_pend.y, sub);
      if (i0 + u > 0) {
        if ((sub & ~1) == 2) *o_at = o_before;
        o_at += ldo;
      }
      const float2 v = *reinterpret_cast<const float2*>(in + 5 * D + 2 * cg);
      const float2 d2[2] = {pair_of(dx), pair_of(dy)}, v2[2] = {pair_of(v.x), pair_of(v.y)};
      float2 o2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < NI; ++c) {
        const float4 ww = holds ? *reinterpret_cast<const float4*>(in + 64 * c + 4 * sub) : zero;
        const float4 mm = holds ? *reinterpret_cast<const float4*>(in + 2 * D + 64 * c + 4 * sub) : zero;
        const float4 kk = holds ? *reinterpret_cast<const float4*>(in + 3 * D + 64 * c + 4 * sub) : zero;
        const float4 rr = holds ? *reinterpret_cast<const float4*>(in + 4 * D + 64 * c + 4 * sub) : zero;
        const float2 wp[2] = {make_float2(ww.x, ww.y), make_float2(ww.z, ww.w)}, mp[2] = {make_float2(mm.x, mm.y), make_float2(mm.z, mm.w)};
        const float2 kp[2] = {make_float2(kk.x, kk.y), make_float2(kk.z, kk.w)}, rp[2] = {make_float2(rr.x, rr.y), make_float2(rr.z, rr.w)};
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int col = 0; col < 2; ++col) {
            S_r[col][c][e] = __ffma2_rn(kp[e], v2[col], __ffma2_rn(mp[e], d2[col], __fmul2_rn(wp[e], S_r[col][c][e])));
            o2[col] = __ffma2_rn(S_r[col][c][e], rp[e], o2[col]);
          }
      }
      o_pend = make_float2(pair_sum(o2[0]), pair_sum(o2[1]));       // joined over the lanes in the next token's rounds
    }
  }
  {
    float none = 0.f, none2 = 0.f;
    const float o_last = join_four(none, none2, o_pend.x, o_pend.y, sub);
    if ((sub & ~1) == 2) *o_at = o_last;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (write_state && holds) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int i = 0; i < NI; ++i)
        *reinterpret_cast<float4*>(S_g + c * D + 64 * i + 4 * sub) =
            make_float4(S_r[c][i][0].x, S_r[c][i][0].y, S_r[c][i][1].x, S_r[c][i][1].y);
  }
}

// The same for one token a sequence (the same bits): bound by the state's way in and out, so no ring; every vector straight into
// the registers, beside the state.  64 sequences, 32 heads of 64: 35.1 us in the form above, 14.8 so; 8 of 16
// heads of 128 7.0, 4.8.
template <int D>
__global__ void __launch_bounds__(256)
dplr_recurrence_one_kernel(const float* __restrict__ proj, long ld, const float* __restrict__ prep, long ldp, int H, int Dv,
                           float* __restrict__ state, long state_stride, const int32_t* __restrict__ seq_q_start,
                           const int32_t* __restrict__ seq_slot, float* __restrict__ o_raw, long ldo, int write_state) {
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.x, seq = blockIdx.y, slot = seq_slot[seq], row = seq_q_start[seq];
  if (slot < 0 || seq_q_start[seq + 1] <= row) return;
  constexpr int NI = (D + 63) / 64;
  const int CB = blockDim.x >> 3, cg = threadIdx.x >> 4, sub = threadIdx.x & 15, col0 = blockIdx.z * CB + 2 * cg, HD = H * D;
  const bool holds = 4 * sub < D;
  float* S_g = state + (size_t)slot * state_stride + (size_t)h * D * Dv + (size_t)col0 * D;
  const float* prow = prep + (size_t)row * ldp + (size_t)h * D + 4 * sub;
  const float* xrow = proj + (size_t)row * ld;
  float2 S_r[2][NI][2];
  rec_load_state<NI>(S_r, S_g, D, sub, holds);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 ww[NI], pp[NI], mm[NI], kk[NI], rr[NI];
#pragma unroll
  for (int c = 0; c < NI; ++c) {
    ww[c] = holds ? *reinterpret_cast<const float4*>(prow + 64 * c) : zero;
    pp[c] = holds ? *reinterpret_cast<const float4*>(prow + HD + 64 * c) : zero;
    mm[c] = holds ? *reinterpret_cast<const float4*>(prow + 2 * (size_t)HD + 64 * c) : zero;
    rr[c] = holds ? *reinterpret_cast<const float4*>(xrow + (size_t)h * D + 4 * sub + 64 * c) : zero;
    kk[c] = holds ? *reinterpret_cast<const float4*>(xrow + HD + (size_t)h * D + 4 * sub + 64 * c) : zero;
  }
  const float2 v = *reinterpret_cast<const float2*>(xrow + 2 * (size_t)HD + (size_t)h * Dv + col0);
  float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, o2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int c = 0; c < NI; ++c)
#pragma unroll
    for (int col = 0; col < 2; ++col) {
      acc[col] = __ffma2_rn(S_r[col][c][0], make_float2(pp[c].x, pp[c].y), acc[col]);
      acc[col] = __ffma2_rn(S_r[col][c][1], make_float2(pp[c].z, pp[c].w), acc[col]);
    }
  float dx = pair_sum(acc[0]), dy = pair_sum(acc[1]), none = 0.f, none2 = 0.f;
  join_four(dx, dy, 0.f, 0.f, sub);
  const float2 d2[2] = {pair_of(dx), pair_of(dy)}, v2[2] = {pair_of(v.x), pair_of(v.y)};
#pragma unroll
  for (int c = 0; c < NI; ++c) {
    const float2 wp[2] = {make_float2(ww[c].x, ww[c].y), make_float2(ww[c].z, ww[c].w)}, mp[2] = {make_float2(mm[c].x, mm[c].y), make_float2(mm[c].z, mm[c].w)};
    const float2 kp[2] = {make_float2(kk[c].x, kk[c].y), make_float2(kk[c].z, kk[c].w)}, rp[2] = {make_float2(rr[c].x, rr[c].y), make_float2(rr[c].z, rr[c].w)};
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int col = 0; col < 2; ++col) {
        S_r[col][c][e] = __ffma2_rn(kp[e], v2[col], __ffma2_rn(mp[e], d2[col], __fmul2_rn(wp[e], S_r[col][c][e])));
        o2[col] = __ffma2_rn(S_r[col][c][e], rp[e], o2[col]);
      }
  }
  if (write_state && holds) rec_store_state<NI>(S_r, S_g, D, sub);
  const float o = join_four(none, none2, pair_sum(o2[0]), pair_sum(o2[1]), sub);
  if ((sub & ~1) == 2) o_raw[(size_t)row * ldo + (size_t)h * Dv + col0 + (sub & 1)] = o;
}

template <int D>
int launch_dplr_quad(const float* proj, long ld, const float* prep, long ldp, int H, int Dv, float* state, long state_stride,
                     const int32_t* seq_q_start, const int32_t* seq_slot, float* o_raw, long ldo, int n_seqs, int write_state, int one,
                     cudaStream_t stream) {
  const int CB = Dv % 32 == 0 ? 32 : 16;                     // columns per block
  if (one)
    return launch_pdl(PDL_ATTENTION, dplr_recurrence_one_kernel<D>, dim3(H, n_seqs, Dv / CB), dim3(8 * CB), 0, stream, proj, ld, prep, ldp, H,
                      Dv, state, state_stride, seq_q_start, seq_slot, o_raw, ldo, write_state);
  const size_t smem = (size_t)REC_STAGES * REC_BATCH * (5 * D + CB) * sizeof(float);       // (at most 32 KB)
  return launch_pdl(PDL_ATTENTION, dplr_recurrence_quad_kernel<D>, dim3(H, n_seqs, Dv / CB), dim3(8 * CB), smem, stream, proj, ld,
                    prep, ldp, H, Dv, state, state_stride, seq_q_start, seq_slot, o_raw, ldo, write_state);
}

}  // namespace llmi

using namespace llmi;

// w2t: W2 transposed, fp32 [R, H*D]; z (optional): fp32 [T, ldz] = tanh(low) W2ᵀ made beforehand.
LLMI_EXPORT int llmi_gdelta_prepare(const float* proj, long ld, int H, int D, int Dv, int R, const float* w2t, const float* z,
                                    long ldz, const float* w0, const float* a_bias, const int32_t* tok_seq, float* prep, long ldp,
                                    int n_tokens, cudaStream_t stream) {
  if (n_tokens <= 0 || H <= 0 || H > 65535 || D <= 0 || Dv <= 0 || R <= 0 || R > 8192) return LLMI_ERR_BAD_SIZE;
  // Four entries a thread: always behind a product.  Walking W2's rows it pays a barrier and its segments' sum, and blocks of 128 threads
  // of many registers; the general form walks all R rows one behind the other.  R rows, blocks: general / fours, us: 16, 64 2.9 /
  // 2.8; 16, 256 3.0 / 3.5; 32, 256 3.4 / 3.4; 64, 512 4.6 / 3.8; 64, 1,024 5.4 / 6.0; 128, 1,024 8.3 / 6.4; 128, 2 6.4 / 2.7; 8, 128 2.6 / 2.9.
  const bool fours = z || (long)n_tokens * H <= 16L * R - 192;
  if (fours && ld % 4 == 0 && ldp % 4 == 0 && ldz % 4 == 0 && Dv % 4 == 0 && !((uintptr_t)proj & 15) && !((uintptr_t)prep & 15) && !((uintptr_t)z & 15) &&
      !((uintptr_t)w2t & 15) && !((uintptr_t)w0 & 15) && !((uintptr_t)a_bias & 15)) {
    if (D == 32) return launch_gdelta_fours<32>(proj, ld, H, Dv, R, w2t, z, ldz, w0, a_bias, tok_seq, prep, ldp, n_tokens, stream);
    if (D == 64) return launch_gdelta_fours<64>(proj, ld, H, Dv, R, w2t, z, ldz, w0, a_bias, tok_seq, prep, ldp, n_tokens, stream);
    if (D == 128) return launch_gdelta_fours<128>(proj, ld, H, Dv, R, w2t, z, ldz, w0, a_bias, tok_seq, prep, ldp, n_tokens, stream);
  }
  const int threads = D > 64 ? 128 : (D > 32 ? 64 : 32);
  return launch_pdl(PDL_SMALL, gdelta_prepare_kernel, dim3(n_tokens, H), dim3(threads), (size_t)R * sizeof(float), stream, proj, ld,
                    H, D, Dv, R, w2t, z, ldz, w0, a_bias, tok_seq, prep, ldp);
}

// dst [T, R] (type `dtype`, contiguous) = tanh(src[:, :R]); src fp32 rows of pitch ld.
LLMI_EXPORT int llmi_tanh_rows(int dtype, const float* src, long ld, void* dst, int n_rows, int R, cudaStream_t stream) {
  if (n_rows <= 0 || R <= 0) return LLMI_ERR_BAD_SIZE;
  const long total = (long)n_rows * R;
  const long want = (total + 255) / 256, most = (long)sm_count() * 16;
  const unsigned blocks = (unsigned)(want < most ? want : most);
  if (dtype == LLMI_DTYPE_F32)
    return launch_pdl(PDL_SMALL, tanh_rows_kernel<float>, dim3(blocks), dim3(256), 0, stream, src, ld, (float*)dst, R, total);
  if (dtype == LLMI_DTYPE_BF16)
    return launch_pdl(PDL_SMALL, tanh_rows_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, src, ld, (__nv_bfloat16*)dst, R, total);
  return LLMI_ERR_BAD_DTYPE;
}

// proj fp32 [T, ld]: r at column 0, k at H*D, v at 2*H*D; prep fp32 [T, ldp]: w at 0, p at H*D, m at 2*H*D;
// state fp32 [slots, state_stride >= H*D*Dv]; o_raw fp32 [T, ldo] receives Sᵀ r.  one: no sequence brings more than one token.
LLMI_EXPORT int llmi_dplr_recurrence(const float* proj, long ld, const float* prep, long ldp, int H, int D, int Dv, float* state,
                                     long state_stride, const int32_t* seq_q_start, const int32_t* seq_slot, float* o_raw,
                                     long ldo, int n_seqs, int write_state, int one, cudaStream_t stream) {
  if (n_seqs <= 0 || n_seqs > 65535 || H <= 0 || D <= 0 || Dv <= 0 || Dv > 1024) return LLMI_ERR_BAD_SIZE;
  if (Dv % 16 == 0 && ld % 4 == 0 && ldp % 4 == 0 && ldo % 4 == 0 && state_stride % 4 == 0 && !((uintptr_t)state & 15) &&
      !((uintptr_t)o_raw & 15) && !((uintptr_t)prep & 15) && !((uintptr_t)proj & 15)) {
#define LLMI_QUAD(DD)                                                                                                      \
  if (D == DD)                                                                                                             \
    return launch_dplr_quad<DD>(proj, ld, prep, ldp, H, Dv, state, state_stride, seq_q_start, seq_slot, o_raw, ldo, n_seqs, \
                                write_state, one, stream)
    LLMI_QUAD(32);
    LLMI_QUAD(64);
    LLMI_QUAD(128);
#undef LLMI_QUAD
  }
  const int cols = (Dv + 31) / 32 * 32;
  const size_t smem = ((size_t)10 * D + (size_t)D * cols) * sizeof(float);
  if (smem > 200 * 1024) return LLMI_ERR_BAD_SIZE;
  static PerDevice<size_t> allowed;
  if (smem > 48 * 1024 && allowed.here() < smem) {
    if (cudaFuncSetAttribute(dplr_recurrence_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return LLMI_ERR_BAD_SIZE;
    allowed.here() = smem;
  }
  return launch_pdl(PDL_ATTENTION, dplr_recurrence_kernel, dim3(H, n_seqs), dim3(cols), smem, stream, proj, ld, prep, ldp, H, D, Dv,
                    state, state_stride, seq_q_start, seq_slot, o_raw, ldo, write_state);
}
