// Latent attention of PROMPTS in its expanded form (bf16): tcgen05 tiles over keys and values that the latent rows are
// multiplied out into.
//
// The kernel of latent_attention_mma.cu works on the cached rows [c (C) | r (R)] themselves: a (query, key) pair costs
// 2 C + R products a head, which is the least that can be read for single tokens, but for prompts it is arithmetic that counts:
// with C = 512, R = 64 and heads of 128 the pair costs 320 once k = Uk c and v = Uv c have been made, a matrix product over
// the sequence's rows that every query shares.  So a prompt step takes four launches:
//
//   llmi_latent_expand_prepare   the sequences' rows out of their pages, sequence after sequence in whole pages of 64 (rows
//                                behind a sequence's end are zeros): c to [rows, C], r to [rows, 64]; the rotated part of the
//                                queries to [tokens, heads, 64] (R < 64: zeros behind)
//   a product                    [rows, C] x [heads x (D + Dv), C]: a row's [k | v] of every head
//   llmi_attention_expanded      causal attention, straight to the heads' values: the product with Uv behind the attention
//                                and the one with Uk before it fall away
//
// The attention is that of attention_prefill_tc.cu (see there for the barriers, the lazy scaling and the two threads of a
// query row), with these differences: a score's products run over D plain columns and one tile of 64 rotated ones that all
// heads share; keys and values are columns of one matrix, rows in order, so no page table; 128 queries and one head a block,
// one block per SM with 512 tensor-memory columns where D is 128.
// Measured (2,048 wide, 16 heads of 128, rank 512; layer by layer in a step): 3,059 tokens of two prompts took 753 us a layer in
// the attention on the latent rows, at 104 TFLOP/s of mma.sync; which steps go this way: kernels.latent_expanded_pages.
#include <cuda.h>
#include <math.h>

#include "common.cuh"
#include "sm100.cuh"
#include "step_meta.cuh"

namespace llmi {

constexpr int LX_PAGE = 64, LX_BM = 128, LX_ROT = 64;

// ---- rows out of their pages, rotated queries ----
struct ExpandParams {
  const __nv_bfloat16* cache;       // [page][1][64][C + R]
  const int32_t* seq_pages;
  int pages_stride;
  const int32_t* seq_q_start;
  const int32_t* seq_kv_len;
  int n_seqs, C, R;
  __nv_bfloat16* xc;                // [row_pages * 64, C]
  __nv_bfloat16* xr;                // [row_pages * 64, 64]
  int row_pages;                    // at least the sequences' pages
  const __nv_bfloat16* q;           // [tokens, H * (D + R)], row pitch ldq
  long ldq;
  __nv_bfloat16* qr;                // [tokens, H * 64]
  const float* inv_freq;
  const int32_t* tok_seq;
  const int32_t* tok_pos;
  int n_tokens, H, D, rot_dims, pairing;
  float amplitude;
};

// Blocks 0 .. row_pages - 1: a page each.  The others: 8 tokens each, a warp per token.
__global__ void __launch_bounds__(256) latent_expand_prepare_kernel(const ExpandParams p) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x < p.row_pages) {
    int page = blockIdx.x, seq = 0;
    for (; seq < p.n_seqs; ++seq) {
      const int n = p.seq_q_start[seq + 1] > p.seq_q_start[seq] ? (p.seq_kv_len[seq] + LX_PAGE - 1) / LX_PAGE : 0;
      if (page < n) break;
      page -= n;
    }
    const bool real = seq < p.n_seqs;
    const int live = real ? min(LX_PAGE, p.seq_kv_len[seq] - page * LX_PAGE) : 0;
    const int Dk = p.C + p.R, chunks = p.C / 8, rchunks = p.R / 8;
    const __nv_bfloat16* src = real ? p.cache + (size_t)p.seq_pages[(size_t)seq * p.pages_stride + page] * LX_PAGE * Dk : p.cache;
    const size_t row0 = (size_t)blockIdx.x * LX_PAGE;
    for (int r = warp; r < LX_PAGE; r += 8) {
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      const uint4* from = reinterpret_cast<const uint4*>(src + (size_t)r * Dk);
      uint4* to = reinterpret_cast<uint4*>(p.xc + (row0 + r) * p.C);
      for (int c = lane; c < chunks; c += 32) to[c] = r < live ? from[c] : zero;
      uint4* to_r = reinterpret_cast<uint4*>(p.xr + (row0 + r) * LX_ROT);
      if (lane < LX_ROT / 8) to_r[lane] = (r < live && lane < rchunks) ? from[chunks + lane] : zero;
    }
    return;
  }
  const int t = ((int)blockIdx.x - p.row_pages) * 8 + warp;
  if (t >= p.n_tokens || p.tok_seq[t] < 0) return;          // (rows of no sequence are in no tile that is stored)
  const float pos = (float)p.tok_pos[t];
  const int half = p.rot_dims / 2;
  // a lane's pair: one angle for all heads (lane < R / 2 <= 32; the pairs that turn, then the rest two by two)
  const bool turns = lane < half, has = lane < p.R / 2;
  const int a = turns ? (p.pairing ? 2 * lane : lane) : p.rot_dims + 2 * (lane - half);
  const int b = turns && !p.pairing ? lane + half : a + 1;
  float s = 0.f, co = 1.f;
  if (turns) {
    sincosf(pos * p.inv_freq[lane], &s, &co);
    s *= p.amplitude;
    co *= p.amplitude;
  }
  for (int h = 0; h < p.H; ++h) {
    const __nv_bfloat16* src = p.q + (size_t)t * p.ldq + (size_t)h * (p.D + p.R) + p.D;
    __nv_bfloat16* dst = p.qr + ((size_t)t * p.H + h) * LX_ROT;
    if (has) {
      const float u = __bfloat162float(src[a]), v = __bfloat162float(src[b]);
      dst[a] = turns ? __float2bfloat16_rn(rot_lo(u, v, co, s)) : src[a];
      dst[b] = turns ? __float2bfloat16_rn(rot_hi(u, v, co, s)) : src[b];
    } else {
      *reinterpret_cast<uint32_t*>(dst + 2 * lane) = 0u;    // entries R .. 63
    }
  }
}

// ---- the attention ----
constexpr int LX_SUB = LX_PAGE * 64 * 2;              // 8 KB: 64 rows x 64 columns of bf16, one swizzled sub-tile
constexpr float LX_LAZY = 8.0f;                       // the reference maximum follows the running one in steps of 2^8

// HD: plain entries of a head's key, and of its value.
template <int HD>
struct LxCfg {
  static constexpr int VSUB = HD / 64, QSUB = VSUB + 1;       // 64-column sub-tiles of V, of Q and K
  static constexpr int THREADS = 64 + 256;                    // producer warp, MMA warp, eight softmax warps
  static constexpr int STAGES = HD == 64 ? 2 : 3;
  static constexpr int K_TILE = QSUB * LX_SUB, STAGE = (QSUB + VSUB) * LX_SUB;
  static constexpr int QBYTES = 2 * QSUB * LX_SUB;
  static constexpr int TMEM_COLS = HD == 64 ? 256 : 512;      // S0, S1, the O's of the two key halves
  static constexpr int SMEM = QBYTES + STAGES * STAGE + 1024 + 128;
};

struct ExpandedParams {
  __nv_bfloat16* out;       // [tokens, n_heads * HD]
  long ldo;
  const int32_t* seq_q_start;
  const int32_t* seq_kv_len;
  int n_seqs, n_heads;
  float scale_log2;
  int* error_flag;
};

__device__ __forceinline__ void lx_tma(uint32_t dst, const CUtensorMap* map, int col, int row, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(col), "r"(row)
      : "memory");
}
// K-major operand tile (rows of 128 bytes, 128-byte swizzle, 8-row groups 1024 bytes apart)
__device__ __forceinline__ uint64_t lx_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
__device__ __forceinline__ void lx_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void lx_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 16 consecutive fp32 columns of this thread's TMEM lane; no wait
__device__ __forceinline__ void lx_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void lx_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 16 consecutive fp32 columns of this thread's TMEM lane, written; no wait
__device__ __forceinline__ void lx_st16(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
        "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
}
__device__ __forceinline__ void lx_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }


__device__ __forceinline__ void lx_mma_ts(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// 16 consecutive 32-bit columns of this thread's TMEM lane, written; no wait
__device__ __forceinline__ void lx_st16u(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

template <int HD>
__global__ void __launch_bounds__(LxCfg<HD>::THREADS, HD == 64 ? 2 : 1)
attention_expanded_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                          const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_r, ExpandedParams p, int q_pitch) {
  using C = LxCfg<HD>;
  constexpr int STAGES = C::STAGES, VSUB = C::VSUB, QSUB = C::QSUB, KEYS = 32;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = base;                                      // sub-tile u: + u * 16 KB; the rotated one last
  const uint32_t kv_smem = base + C::QBYTES;                         // stage s: K at + s * STAGE, V K_TILE further
  const uint32_t bars = kv_smem + STAGES * C::STAGE;
  // barriers: q_full, kv_full[stages], kv_empty[stages], s_full[2], p_ready[2], o_done, tmem slot
  const uint32_t q_full = bars;
  auto kv_full = [&](int s) { return bars + 8u * (1 + s); };
  auto kv_empty = [&](int s) { return bars + 8u * (1 + STAGES + s); };
  auto s_full = [&](int b) { return bars + 8u * (1 + 2 * STAGES + b); };
  auto p_ready = [&](int b) { return bars + 8u * (3 + 2 * STAGES + b); };
  const uint32_t o_done = bars + 8u * (5 + 2 * STAGES);
  const uint32_t tmem_slot = o_done + 8u;

  // The head is the fast grid index; blocks of 128 queries are counted from the last one of the last sequence backwards
  // (long jobs first).  row0: the sequence's first row among the expanded ones.
  int seq = p.n_seqs - 1, mb = 0, q_start = 0, q_len = 0, kv_len = 0;
  {
    int x = blockIdx.y;
    for (; seq >= 0; --seq) {
      q_start = p.seq_q_start[seq];
      q_len = p.seq_q_start[seq + 1] - q_start;
      const int n = (q_len + LX_BM - 1) / LX_BM;
      if (x < n) {
        mb = n - 1 - x;
        break;
      }
      x -= n;
    }
    if (seq < 0) return;
    kv_len = p.seq_kv_len[seq];
  }
  int row0 = 0;
  for (int s = 0; s < seq; ++s)
    if (p.seq_q_start[s + 1] > p.seq_q_start[s]) row0 += (p.seq_kv_len[s] + LX_PAGE - 1) / LX_PAGE * LX_PAGE;
  const int pos0 = kv_len - q_len, m0 = mb * LX_BM, first_q = pos0 + m0;
  const int n_pg = (first_q + min(LX_BM, q_len - m0) - 1) / LX_PAGE + 1;
  const int head = blockIdx.x;
  __shared__ float s_ml[2][LX_BM][2];      // (reference maximum, sum) of a row's two key halves

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_qr) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_kv) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_r) : "memory");
    mbar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(kv_full(s), 1);
      mbar_init(kv_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_full(b), 1);
      mbar_init(p_ready(b), 8);
    }
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(C::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
  pdl_launch_dependents();      // (only now: see attention_prefill_tc.cu)
  const uint32_t tmem_s = tmem, tmem_o = tmem + 128;

  if (warp == 0) {
    if (lane == 0) {
      // ---- producer ----
      pdl_wait();
      mbar_expect_tx(q_full, C::QBYTES);
#pragma unroll
      for (int u = 0; u < VSUB; ++u) lx_tma(q_smem + u * 2 * LX_SUB, &map_q, head * q_pitch + 64 * u, q_start + m0, q_full);
      lx_tma(q_smem + VSUB * 2 * LX_SUB, &map_qr, head * LX_ROT, q_start + m0, q_full);
      for (int j = 0; j < n_pg; ++j) {
        const int s = j % STAGES;
        if (j >= STAGES && !mbar_wait(kv_empty(s), ((j / STAGES) - 1) & 1, p.error_flag, 81)) break;
        const int row = row0 + j * LX_PAGE;
        const uint32_t k_tile = kv_smem + s * C::STAGE;
        mbar_expect_tx(kv_full(s), C::STAGE);
#pragma unroll
        for (int u = 0; u < VSUB; ++u) {
          lx_tma(k_tile + u * LX_SUB, &map_kv, head * 2 * HD + 64 * u, row, kv_full(s));
          lx_tma(k_tile + C::K_TILE + u * LX_SUB, &map_kv, head * 2 * HD + HD + 64 * u, row, kv_full(s));
        }
        lx_tma(k_tile + VSUB * LX_SUB, &map_r, 0, row, kv_full(s));
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issuer ----
      const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      const uint32_t idesc_o = idesc_s | (1u << 16);
      auto issue_s = [&](int j) {
        const uint32_t d = tmem_s + (uint32_t)(64 * (j & 1));
#pragma unroll
        for (int k4 = 0; k4 < QSUB * 4; ++k4) {
          const uint64_t a = lx_desc(q_smem + (k4 / 4) * 2 * LX_SUB), b = lx_desc(kv_smem + (j % STAGES) * C::STAGE + (k4 / 4) * LX_SUB);
          lx_mma(d, a + 2 * (k4 % 4), b + 2 * (k4 % 4), idesc_s, k4 > 0);
        }
        lx_commit(s_full(j & 1));
      };
      bool ok = mbar_wait(q_full, 0, p.error_flag, 82) && mbar_wait(kv_full(0), 0, p.error_flag, 83);
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_s(0);
      }
      for (int j = 0; j < n_pg && ok; ++j) {
        if (j + 1 < n_pg) {
          ok = mbar_wait(kv_full((j + 1) % STAGES), ((j + 1) / STAGES) & 1, p.error_flag, 84);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          issue_s(j + 1);
        }
        ok = mbar_wait(p_ready(j & 1), (j >> 1) & 1, p.error_flag, 86);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = tmem_s + (uint32_t)(64 * (j & 1));
        const uint32_t v_tile = kv_smem + (j % STAGES) * C::STAGE + C::K_TILE;
        // the keys of half h accumulate into their own O; P of half h lies at columns 32h.. of the S buffer
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int k4 = 0; k4 < 2; ++k4)
#pragma unroll
            for (int u = 0; u < VSUB; ++u)
              lx_mma_ts(tmem_o + (uint32_t)(HD * h + 64 * u), a + (uint32_t)(32 * h + 8 * k4),
                        lx_desc(v_tile + u * LX_SUB) + (uint64_t)((2 * h + k4) * ((16 * 128) >> 4)), idesc_o, (j > 0 || k4 > 0) ? 1u : 0u);
        lx_commit(o_done);
        lx_commit(kv_empty(j % STAGES));
      }
    }
  } else {
    // ---- softmax and output: two threads per query row, 32 keys of a page each ----
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const int row = quad * 32 + lane, qrow = m0 + row, qpos = pos0 + qrow;
    const bool row_ok = qrow < q_len;
    const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
    const uint32_t t_o = tmem_o + t_lane + (uint32_t)(HD * half);
    float m_run = -INFINITY, m_ref = -INFINITY, l_run = 0.f;   // maxima in base 2, scaled
    bool ok = true;
    for (int j = 0; j < n_pg && ok; ++j) {
      ok = mbar_wait(s_full(j & 1), (j >> 1) & 1, p.error_flag, 88);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t_s = tmem_s + t_lane + (uint32_t)(64 * (j & 1) + KEYS * half);
      float sc[KEYS];
#pragma unroll
      for (int c = 0; c < KEYS; c += 16) lx_ld16(t_s + (uint32_t)c, sc + c);
      lx_ld_wait();
      const int key0 = j * LX_PAGE + KEYS * half;
      if (key0 + KEYS - 1 > first_q) {
#pragma unroll
        for (int c = 0; c < KEYS; ++c)
          if (key0 + c > qpos) sc[c] = -INFINITY;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // four chains instead of one long one
#pragma unroll
      for (int c = 0; c < KEYS; c += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(mx4[u], fmaxf(sc[c + 2 * u], sc[c + 2 * u + 1]));
      }
      m_run = fmaxf(m_run, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2);
      float corr = 1.f;
      if (m_run > m_ref + LX_LAZY || m_ref == -INFINITY) {     // (both -inf: nothing seen yet, nothing to scale)
        corr = (m_ref == -INFINITY) ? 0.f : fast_exp2(m_ref - m_run);
        m_ref = m_run;
        l_run *= corr;
      }
      const float neg_ref = (m_ref == -INFINITY) ? 0.f : -m_ref;
      float2 sum2[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), neg2 = make_float2(neg_ref, neg_ref);
      uint32_t packed[KEYS / 2];
#pragma unroll
      for (int c = 0; c < KEYS; c += 2) {
        const float2 x = __ffma2_rn(make_float2(sc[c], sc[c + 1]), scale2, neg2);
        const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));          // 2^(-inf) = 0 for masked keys
        sum2[(c >> 1) & 3] = __fadd2_rn(sum2[(c >> 1) & 3], e);
        __nv_bfloat162 h = __floats2bfloat162_rn(e.x, e.y);
        packed[c >> 1] = *reinterpret_cast<uint32_t*>(&h);
      }
      {
        const float2 t = __fadd2_rn(__fadd2_rn(sum2[0], sum2[1]), __fadd2_rn(sum2[2], sum2[3]));
        l_run += t.x + t.y;
      }
      if (j >= 1) {
        // (waited for on every page: see attention_prefill_tc.cu)
        ok = mbar_wait(o_done, (j - 1) & 1, p.error_flag, 89);
        if (!ok) break;
        if (__any_sync(0xffffffffu, corr != 1.f)) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int c = 0; c < HD; c += 16) {
            float t[16];
            lx_ld16(t_o + (uint32_t)c, t);
            lx_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) t[e] *= corr;
            lx_st16(t_o + (uint32_t)c, t);
          }
        }
      }
      lx_st16u(t_s, packed);      // P over the first half of the S columns this thread has just read
      lx_st_wait();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready(j & 1));
    }
    // (a warp whose wait gave up still goes through the barrier below)
    const bool fine = __all_sync(0xffffffffu, ok && mbar_wait(o_done, (n_pg - 1) & 1, p.error_flag, 90));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    constexpr int DH = HD / 2;                                                // output columns per thread
    s_ml[half][row][0] = m_ref;
    s_ml[half][row][1] = l_run;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const float m_a = s_ml[0][row][0], m_b = s_ml[1][row][0], M = fmaxf(m_a, m_b);
    float w_a = (m_a == -INFINITY) ? 0.f : fast_exp2(m_a - M), w_b = (m_b == -INFINITY) ? 0.f : fast_exp2(m_b - M);
    const float inv = 1.f / (s_ml[0][row][1] * w_a + s_ml[1][row][1] * w_b);
    w_a *= inv;
    w_b *= inv;
    if (fine) {      // every lane takes part in the tensor-memory loads; only the rows that exist are stored
      const uint32_t t_mine = tmem_o + t_lane + (uint32_t)(DH * half);
      __nv_bfloat16* dst = p.out + (size_t)(q_start + qrow) * p.ldo + (size_t)head * HD + DH * half;
#pragma unroll 1
      for (int c0 = 0; c0 < DH; c0 += 32) {
        float o[32], ob[32];
        lx_ld16(t_mine + (uint32_t)c0, o);
        lx_ld16(t_mine + (uint32_t)(c0 + 16), o + 16);
        lx_ld16(t_mine + (uint32_t)(HD + c0), ob);
        lx_ld16(t_mine + (uint32_t)(HD + c0 + 16), ob + 16);
        lx_ld_wait();
#pragma unroll
        for (int c = 0; c < 32 && row_ok; c += 8) {
          uint32_t v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int x = c + 2 * e;
            __nv_bfloat162 h = __floats2bfloat162_rn(w_a * o[x] + w_b * ob[x], w_a * o[x + 1] + w_b * ob[x + 1]);
            v[e] = *reinterpret_cast<uint32_t*>(&h);
          }
          *reinterpret_cast<uint4*>(dst + c0 + c) = make_uint4(v[0], v[1], v[2], v[3]);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS));
}

typedef CUresult (*LxEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A bf16 matrix [rows, cols] with row pitch ld (elements): tiles of [box_rows, 64 columns], 128-byte swizzle.
static int lx_make_map(CUtensorMap* map, const void* ptr, long rows, long cols, long ld, int box_rows) {
  static LxEncodeFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return LLMI_ERR_DRIVER;
    fn = (LxEncodeFn)sym;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? LLMI_OK
             : LLMI_ERR_DRIVER;
}

template <int HD>
static int lx_launch(const CUtensorMap& mq, const CUtensorMap& mqr, const CUtensorMap& mkv, const CUtensorMap& mr, const ExpandedParams& p,
                     int q_pitch, int n_blocks, cudaStream_t stream) {
  using C = LxCfg<HD>;
  static PerDevice<bool> configured_on;
  bool& configured = configured_on.here();
  if (!configured) {
    if (cudaFuncSetAttribute(attention_expanded_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
      return LLMI_ERR_LAUNCH;
    configured = true;
  }
  return launch_pdl(PDL_ATTENTION, attention_expanded_kernel<HD>, dim3(p.n_heads, n_blocks), dim3(C::THREADS), C::SMEM, stream, mq, mqr, mkv,
                    mr, p, q_pitch);
}

}  // namespace llmi

using namespace llmi;

// Heads of D plain entries and values of D, D 64 or 128, a rotated part of up to 64.
LLMI_EXPORT int llmi_attention_expanded_supported(int D, int Dv, int R, int C, int page_size) {
  return (D == 64 || D == 128) && Dv == D && R >= 0 && R <= LX_ROT && R % 8 == 0 && C > 0 && C % 8 == 0 && page_size == LX_PAGE;
}

// cache [page][1][64][C + R]; xc [row_pages * 64, C], xr [row_pages * 64, 64]: the rows of the sequences that bring tokens, in
// sequence order, whole pages each; q [n_tokens, H * (D + R)] (row pitch ldq); qr [n_tokens, H * 64].
LLMI_EXPORT int llmi_latent_expand_prepare(const void* cache, const int32_t* seq_pages, int pages_stride, const int32_t* seq_q_start,
                                           const int32_t* seq_kv_len, int n_seqs, int C, int R, void* xc, void* xr, int row_pages,
                                           const void* q, long ldq, void* qr, const float* inv_freq, const int32_t* tok_seq,
                                           const int32_t* tok_pos, int n_tokens, int H, int D, int rot_dims, int pairing, float amplitude,
                                           cudaStream_t stream) {
  if (n_seqs <= 0 || row_pages <= 0 || n_tokens <= 0 || H <= 0 || rot_dims > R || (rot_dims & 1) || rot_dims < 0) return LLMI_ERR_BAD_SIZE;
  if (!llmi_attention_expanded_supported(D, D, R, C, LX_PAGE)) return LLMI_ERR_UNSUPPORTED;
  if (((uintptr_t)cache | (uintptr_t)xc | (uintptr_t)xr) & 15) return LLMI_ERR_ALIGN;
  const ExpandParams p{(const __nv_bfloat16*)cache, seq_pages, pages_stride, seq_q_start, seq_kv_len, n_seqs, C, R, (__nv_bfloat16*)xc,
                       (__nv_bfloat16*)xr, row_pages, (const __nv_bfloat16*)q, ldq, (__nv_bfloat16*)qr, inv_freq, tok_seq, tok_pos,
                       n_tokens, H, D, rot_dims, pairing, amplitude};
  return launch_pdl(PDL_SMALL, latent_expand_prepare_kernel, dim3(row_pages + (n_tokens + 7) / 8), dim3(256), 0, stream, p);
}

// kv [n_rows, H * 2 D]: [k | v] of every head; xr, q, qr as above; n_blocks: at least the blocks of 128 queries of the step.
LLMI_EXPORT int llmi_attention_expanded(const void* q, long ldq, const void* qr, const void* kv, long ldkv, const void* xr, long n_rows,
                                        void* out, long ldo, const int32_t* seq_q_start, const int32_t* seq_kv_len, int n_seqs,
                                        int n_tokens, int n_blocks, int H, int D, int R, float scale, int* error_flag, cudaStream_t stream) {
  if (n_seqs <= 0 || n_tokens <= 0 || n_blocks <= 0 || n_blocks > 65535 || H <= 0 || n_rows <= 0 || n_rows > 0x7fffffffL) return LLMI_ERR_BAD_SIZE;
  if (!llmi_attention_expanded_supported(D, D, R, 8, LX_PAGE) || !(scale > 0.f)) return LLMI_ERR_UNSUPPORTED;
  if ((((uintptr_t)q | (uintptr_t)qr | (uintptr_t)kv | (uintptr_t)xr | (uintptr_t)out) & 15) || (ldq & 7) || (ldkv & 7) || (ldo & 7)) return LLMI_ERR_ALIGN;
  CUtensorMap mq, mqr, mkv, mr;
  int rc = lx_make_map(&mq, q, n_tokens, (long)H * (D + R), ldq, LX_BM);
  if (rc == LLMI_OK) rc = lx_make_map(&mqr, qr, n_tokens, (long)H * LX_ROT, (long)H * LX_ROT, LX_BM);
  if (rc == LLMI_OK) rc = lx_make_map(&mkv, kv, n_rows, (long)H * 2 * D, ldkv, LX_PAGE);
  if (rc == LLMI_OK) rc = lx_make_map(&mr, xr, n_rows, LX_ROT, LX_ROT, LX_PAGE);
  if (rc != LLMI_OK) return rc;
  const ExpandedParams p{(__nv_bfloat16*)out, ldo, seq_q_start, seq_kv_len, n_seqs, H, scale * 1.4426950408889634f, error_flag};
  return D == 64 ? lx_launch<64>(mq, mqr, mkv, mr, p, D + R, n_blocks, stream) : lx_launch<128>(mq, mqr, mkv, mr, p, D + R, n_blocks, stream);
}
