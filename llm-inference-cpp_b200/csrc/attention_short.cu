// Attention of SHORT messages on top of long histories: the prompt step of a conversation that goes on (bf16, head size 64
// or 128, pages of 64).
//
// Same operation as attention_prefill_tc.cu (reference loop: src/model/transformer.cpp:263-282).  That kernel takes 128
// queries of one query head a block, which a message of a dozen tokens leaves nine tenths empty, and reads a kv head's
// pages once for each of its query heads.  What bounds this case is the read of the cache; so the rows of a tile are here
// the (position, head of the group) pairs of one kv head, 16 to 64 of them, and the arithmetic is mma.sync on fragments,
// as in attention_decode_mma.cu:
//
//   * a producer warp keeps a ring of cache pages full by TMA (128-byte swizzle);
//   * four consumer warps: ROWS = 16: every warp takes the 16 rows and 16 keys of a page; 32: two row groups, 32 keys each;
//     64: four row groups, all 64 keys.  S = Q K^T, softmax in the accumulator layout, O += P V, all in registers;
//   * a cluster of 1, 2, 4 or 8 blocks shares a (sequence, kv head, row tile): every block takes a run of its pages and
//     leaves (values, maximum, sum) in its shared memory; the cluster's warps then add them, a row a warp, in key order.  No workspace, no tickets.
//
// The weights (probabilities) meet V as bf16, as in the other tensor-core kernels — but for the decode steps of ungrouped heads
// of 128 (WIDE), whose weights are 32 bits wide in the kernel that has the rest of them (attention_decode.cu).  There a tile has ONE
// row, and the other fifteen are free: all of them hold its query, so that every thread group has its weights, and a weight goes
// in as three bf16 numbers that add up to it exactly, in three rows: no more matrix instructions than with one.  Every product is
// exact; the products of a page are summed by the matrix instruction and join the running sums by a rounded addition (running
// sums inside the instruction are cut off, not rounded).  Against 64 bits the same error as attention_decode.cu's, also where the
// values' weighted sum all but cancels (there, 64 sequences of 2,200: 1.671e-3 both, of which the output's rounding is all; bf16
// weights 0.7).  What it costs (with bf16 weights -> with these): 16 x 1 x 128, 64 sequences of 2,200 172 -> 180 us, 1 of 4,000 12.5
// -> 13.6.
//
// Measured against the tiles of 128 queries (kv heads x group x head size, positions, tokens; with about 8 us of launch):
// 64 sequences, 32 x 1 x 64, 1,500, 8: 239 -> 140 us (the read of the cache alone: 120 us); 24, 8 x 4 x 128, 2,200, 9:
// 191 -> 82 (33); 8, 32 x 1 x 64, 3,900, 16: 76 -> 61 (39); 1, 32 x 1 x 64, 4,000, 21: 27.5 -> 19.4 (5); 8, 5 x 3 x 64,
// 2,000, 16: 33 -> 20.5 (3).  Which kernel takes a step, and how many blocks share an item: attention_short_parts.
#include <cooperative_groups.h>
#include <cuda.h>
#include <math.h>
#include <type_traits>

#include "common.cuh"
#include "mma_sync.cuh"
#include "sm100.cuh"

namespace llmi {

namespace cg = cooperative_groups;

constexpr int SH_PAGE = 64;
constexpr int SH_CONSUMERS = 4;
constexpr int SH_THREADS = (SH_CONSUMERS + 1) * 32;
constexpr int SH_MAX_ROWS = 64;              // rows of the largest tile

struct ShortParams {
  const __nv_bfloat16* q;     // [tokens, >= n_heads * HD], rotated; row pitch ldq
  long ldq;
  __nv_bfloat16* out;
  long ldo;
  const int32_t* seq_pages;   // [n_seqs, pages_stride]
  const int32_t* seq_q_start; // [n_seqs + 1]
  const int32_t* seq_kv_len;  // [n_seqs]
  int pages_stride;
  int n_kv_heads, group, row_tiles;
  float scale_log2;
  int window;
  int* error_flag;
  // a decode step whose position encoding is done here (FUSE): `q` holds the un-rotated [q | k | v] rows
  const float* inv_freq;      // [HD / 2] when rotary_dim > 0
  int rotary_dim;             // HD or 0
  int n_heads, write_kv;
  __nv_bfloat16* k_cache_w;
  __nv_bfloat16* v_cache_w;
  int early;                  // rows of earlier steps were complete before the launch ahead began
};

template <int HD>
struct ShCfg {
  static constexpr int NSUB = HD / 64;
  static constexpr int SUB_BYTES = SH_PAGE * 64 * 2;
  static constexpr int TILE_BYTES = NSUB * SUB_BYTES;
  static constexpr int STAGE_BYTES = 2 * TILE_BYTES;
  static constexpr int STAGES = HD == 64 ? 4 : 3;
  static constexpr int OUT_PITCH = HD + 4;      // floats a row of the results: values, maximum, sum
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 16 * STAGES + 16;
  static_assert(SH_MAX_ROWS * OUT_PITCH * 4 <= STAGES * STAGE_BYTES, "the results lie where the ring was");
};

__device__ __forceinline__ uint32_t sh_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 sh_unpack(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
__device__ __forceinline__ void sh_tma(uint32_t dst, const CUtensorMap* map, int col, int row, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(col), "r"(row)
      : "memory");
}

// v as the sum of three bf16 numbers (8 + 8 + 8 bits; exact for |v| > 2^-110, where the last of them is no denormal number)
__device__ __forceinline__ void sh_split(float v, float& hi, float& mid, float& lo) {
  hi = __bfloat162float(__float2bfloat16_rn(v));
  const float rest = __fsub_rn(v, hi);
  mid = __bfloat162float(__float2bfloat16_rn(rest));
  lo = __fsub_rn(rest, mid);
}

// FUSE: one token a sequence; its q is rotated as it is read, its k (rotated) and v are made, appended to the cache and put into
// the newest page by the block that has that page (rope_store.cu's arithmetic: the same bits).  A tile is then 16 rows, and no two
// warps share keys.
template <int HD, int ROWS, bool FUSE, bool WIDE>
__global__ void __launch_bounds__(SH_THREADS, HD == 64 ? 3 : 2)
attention_short_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, ShortParams p) {
  using C = ShCfg<HD>;
  constexpr int WR = ROWS / 16, WK = SH_CONSUMERS / WR;      // row groups, key groups
  constexpr int KEYS = SH_PAGE / WK;                         // keys of a page per warp
  static_assert(!FUSE || ROWS == 16, "one warp has the keys of the step's own row");
  extern __shared__ uint8_t smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int parts = (int)cluster.num_blocks(), part = (int)cluster.block_rank();
  pdl_launch_dependents();
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = base + C::STAGES * C::STAGE_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (C::STAGES + s); };
  const uint32_t row_bar = bars + 16u * C::STAGES;
  float* results = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));     // [WK][ROWS][OUT_PITCH]

  // which (sequence, kv head, row tile); the same for all blocks of a cluster
  int item = blockIdx.x / parts;
  const int tile = item % p.row_tiles;
  item /= p.row_tiles;
  const int kvh = item % p.n_kv_heads, seq = item / p.n_kv_heads;
  const int G = p.group;
  const int q_start = p.seq_q_start[seq], q_len = FUSE ? 1 : p.seq_q_start[seq + 1] - q_start, kv_len = p.seq_kv_len[seq];
  const int row0 = tile * ROWS, rows = min(ROWS, q_len * G - row0);
  if (rows <= 0 || kv_len <= 0) return;
  const int pos0 = kv_len - q_len;
  const int first_q = pos0 + row0 / G, last_q = pos0 + (row0 + rows - 1) / G;      // positions of the tile's queries
  const int lo = (p.window > 0 && first_q - p.window + 1 > 0) ? first_q - p.window + 1 : 0;
  const int pg_first = lo / SH_PAGE, n_all = last_q / SH_PAGE - pg_first + 1;
  const int per = (n_all + parts - 1) / parts;
  const int pg0 = pg_first + part * per, n_pages = max(0, min(per, n_all - part * per));
  const int32_t* pages = p.seq_pages + (size_t)seq * p.pages_stride;

  // The step's own row of a fused decode step never comes from the cache: the producer warp, once it has asked for all pages, makes
  // it, appends it and puts it into the page that the copy engine brought.  So no page waits for the kernel before, and nothing for
  // the row's way out and back (the append, a fence, then the newest page's copy).  A token step, us a layer less: 9 heads of 64
  // over 3, one sequence of 100, 340, 1,000 positions 0.5, 0.5, 0.1; 15 over 5, eight sequences of 100, 340, 1,000 1.1, 0.7, 0.9; from
  // 3,900 positions on the same within 0.1.  Made by the consumer warp that has the row's keys, it cost 24 sequences of up to 3,900
  // positions 1.6 us a layer of 49.  (In attention_decode.cu, whose blocks are bound by the cache's read, a turn of eight sequences of
  // 3,900 positions took 36.9 ms instead of 31.4 so: their newest pages then compete with the product before.)
  const bool own_row = FUSE && p.write_kv;
  const int new_row = pos0 % SH_PAGE, new_page = n_all - 1 - part * per;      // (of this part's pages: its last, or none of them)
  const bool has_newest = own_row && n_pages > 0 && new_page == n_pages - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ float s_rot[FUSE ? HD : 1];                     // sines, then cosines, of the step's position
  const bool rotate = FUSE && p.rotary_dim > 0;
  if (rotate && threadIdx.x >= 32 && threadIdx.x < 32 + HD / 2) {
    const int j = threadIdx.x - 32;
    sincosf((float)pos0 * p.inv_freq[j], &s_rot[j], &s_rot[HD / 2 + j]);
  }
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), SH_CONSUMERS);
    }
    mbar_init(row_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == SH_CONSUMERS) {
    // ---- producer (lane 0 asks for the pages) ----
    bool waited = false, ok = true;
    for (int i = 0; i < n_pages && ok; ++i) {
      const int s = i % C::STAGES;
      const int page = pages[pg0 + i];
      // Where rows of earlier steps may be read ahead, only a page with rows of this step, written by a kernel before, waits.
      if (!waited && (!p.early || (!own_row && (pg0 + i + 1) * SH_PAGE > pos0))) {
        pdl_wait();
        waited = true;
      }
      if (lane == 0) {
        if (i >= C::STAGES && !mbar_wait(empty_bar(s), ((i / C::STAGES) - 1) & 1, p.error_flag, 77)) {
          ok = false;
        } else {
          const int row = (page * p.n_kv_heads + kvh) * SH_PAGE;
          mbar_expect_tx(full_bar(s), C::STAGE_BYTES);
#pragma unroll
          for (int u = 0; u < C::NSUB; ++u) {
            sh_tma(base + s * C::STAGE_BYTES + u * C::SUB_BYTES, &map_k, u * 64, row, full_bar(s));
            sh_tma(base + s * C::STAGE_BYTES + C::TILE_BYTES + u * C::SUB_BYTES, &map_v, u * 64, row, full_bar(s));
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    }
    if (has_newest && ok) {
      // entries j and j + HD / 2 of the new key and value, rounded as the cache has them
      constexpr int NP = HD / 64;
      __nv_bfloat16 kn[NP][2], vn[NP][2];
      pdl_wait();
      const __nv_bfloat16* row = p.q + (size_t)q_start * p.ldq;
      const __nv_bfloat16* ksrc = row + (size_t)(p.n_heads + kvh) * HD;
      const __nv_bfloat16* vsrc = row + (size_t)(p.n_heads + p.n_kv_heads + kvh) * HD;
      const size_t dst = (((size_t)pages[pg0 + new_page] * p.n_kv_heads + kvh) * SH_PAGE + new_row) * HD;
#pragma unroll
      for (int u = 0; u < NP; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          kn[u][h] = ksrc[lane + 32 * u + HD / 2 * h];
          vn[u][h] = vsrc[lane + 32 * u + HD / 2 * h];
        }
      const int s = new_page % C::STAGES;
      const uint32_t k_tile = base + s * C::STAGE_BYTES, v_tile = k_tile + C::TILE_BYTES;
      if (mbar_wait(full_bar(s), (new_page / C::STAGES) & 1, p.error_flag, 80)) {
#pragma unroll
        for (int u = 0; u < NP; ++u) {
          if (rotate) {
            const int j = lane + 32 * u;
            const float a = __bfloat162float(kn[u][0]), b = __bfloat162float(kn[u][1]), sn = s_rot[j], cs = s_rot[HD / 2 + j];
            kn[u][0] = __float2bfloat16_rn(rot_lo(a, b, cs, sn));
            kn[u][1] = __float2bfloat16_rn(rot_hi(a, b, cs, sn));
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = lane + 32 * u + HD / 2 * h;
            const uint32_t at = (uint32_t)((j / 64) * C::SUB_BYTES + new_row * 128 + (((j / 8 & 7) ^ (new_row & 7)) << 4) + (j & 7) * 2);
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(k_tile + at), "h"(__bfloat16_as_ushort(kn[u][h])) : "memory");
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(v_tile + at), "h"(__bfloat16_as_ushort(vn[u][h])) : "memory");
            p.k_cache_w[dst + j] = kn[u][h];
            p.v_cache_w[dst + j] = vn[u][h];
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(row_bar);
      }
    }
  } else {
    // ---- consumers: warp (wr, wk) has rows 16 wr .. and keys KEYS wk .. of every page ----
    const int wr = warp % WR, wk = warp / WR;
    const int gq = lane >> 2, t = lane & 3;                 // accumulator rows gq and gq + 8, columns 2t and 2t + 1
    pdl_wait();                                             // q comes from the kernel before
    const bool has_row = has_newest && wk == new_row / KEYS;      // the step's own row is one of my keys
    uint32_t qa[HD / 16][4];
    int qpos[2];
    {
      const __nv_bfloat16* src[2];
      bool live[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = wr * 16 + gq + 8 * h;
        live[h] = WIDE || r < rows;
        const int x = row0 + min(r, rows - 1), i = x / G;
        qpos[h] = pos0 + i;
        src[h] = p.q + (size_t)(q_start + i) * p.ldq + (size_t)(kvh * G + x - i * G) * HD;
      }
#pragma unroll
      for (int kc = 0; kc < HD / 16; ++kc)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          qa[kc][e] = live[e & 1] ? *reinterpret_cast<const uint32_t*>(src[e & 1] + kc * 16 + (e >> 1) * 8 + 2 * t) : 0u;
      if (rotate) {                                          // both entries of a pair are this thread's, HD / 32 chunks apart
#pragma unroll
        for (int kc = 0; kc < HD / 32; ++kc)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int dim = kc * 16 + (e >> 1) * 8 + 2 * t;
            const float2 a = sh_unpack(qa[kc][e]), b = sh_unpack(qa[kc + HD / 32][e]);
            const float s0 = s_rot[dim], c0 = s_rot[HD / 2 + dim], s1 = s_rot[dim + 1], c1 = s_rot[HD / 2 + dim + 1];
            qa[kc][e] = sh_pack(rot_lo(a.x, b.x, c0, s0), rot_lo(a.y, b.y, c1, s1));
            qa[kc + HD / 32][e] = sh_pack(rot_hi(a.x, b.x, c0, s0), rot_hi(a.y, b.y, c1, s1));
          }
      }
    }
    float o[HD / 8][4];
#pragma unroll
    for (int dc = 0; dc < HD / 8; ++dc)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[dc][e] = 0.f;
    float mrow[2] = {-INFINITY, -INFINITY}, lrow[2] = {0.f, 0.f};     // maxima scaled, in base 2
    const int mtx = lane >> 3, lr = lane & 7;
    for (int i = 0; i < n_pages; ++i) {
      const int s = i % C::STAGES;
      if (!mbar_wait(full_bar(s), (i / C::STAGES) & 1, p.error_flag, 78)) break;
      const uint32_t k_tile = base + s * C::STAGE_BYTES, v_tile = k_tile + C::TILE_BYTES;
      if (has_row && i == new_page && !mbar_wait(row_bar, 0, p.error_flag, 79)) break;      // (the row is in its place)
      const int key0 = (pg0 + i) * SH_PAGE + wk * KEYS;                  // this warp's first key
      const bool inside = key0 + KEYS - 1 <= first_q && (p.window <= 0 || key0 >= last_q - p.window + 1);
      if (key0 + KEYS > kv_len || key0 < lo) {
        // value rows that no query sees are cleared: their zero probabilities must not meet a NaN.  (Row groups that share
        // the keys write the same zeros; each reads behind its own.)
        for (int idx = lane; idx < KEYS * (HD / 8); idx += 32) {
          const int row = wk * KEYS + idx / (HD / 8), ch = idx % (HD / 8);
          const int key = (pg0 + i) * SH_PAGE + row;
          if (key < lo || key >= kv_len)
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(v_tile + (ch / 8) * C::SUB_BYTES + (uint32_t)(row * 128 + ((ch & 7) << 4))), "r"(0u)
                         : "memory");
        }
        __syncwarp();
      }
      float sc[KEYS / 8][4];
#pragma unroll
      for (int n = 0; n < KEYS / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[n][e] = 0.f;
#pragma unroll
      for (int kc = 0; kc < HD / 16; ++kc)
#pragma unroll
        for (int n = 0; n < KEYS / 8; n += 2) {
          const int row = wk * KEYS + n * 8 + (mtx >> 1) * 8 + lr, kch = (kc % 4) * 2 + (mtx & 1);
          uint32_t b0, b1, b2, b3;
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                       : "r"(k_tile + (kc / 4) * C::SUB_BYTES + (uint32_t)(row * 128 + ((kch ^ (row & 7)) << 4))));
          mma_bf16(sc[n], qa[kc], b0, b1);
          mma_bf16(sc[n + 1], qa[kc], b2, b3);
        }
      if (!inside) {
#pragma unroll
        for (int n = 0; n < KEYS / 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = key0 + n * 8 + 2 * t + (e & 1), at = qpos[e >> 1];
            if (key > at || (p.window > 0 && key < at - p.window + 1)) sc[n][e] = -INFINITY;
          }
      }
      float mx[2] = {-INFINITY, -INFINITY}, fix[2], neg[2];
#pragma unroll
      for (int n = 0; n < KEYS / 8; ++n) {
        mx[0] = fmaxf(mx[0], fmaxf(sc[n][0], sc[n][1]));
        mx[1] = fmaxf(mx[1], fmaxf(sc[n][2], sc[n][3]));
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
        const float mn = fmaxf(mrow[h], mx[h] * p.scale_log2);
        fix[h] = (mn == -INFINITY) ? 1.f : fast_exp2(mrow[h] - mn);
        neg[h] = (mn == -INFINITY) ? 0.f : -mn;
        mrow[h] = mn;
      }
      if (__any_sync(0xffffffffu, fix[0] != 1.f || fix[1] != 1.f)) {
        lrow[0] *= fix[0];
        lrow[1] *= fix[1];
#pragma unroll
        for (int dc = 0; dc < HD / 8; ++dc) {
          o[dc][0] *= fix[0];
          o[dc][1] *= fix[0];
          o[dc][2] *= fix[1];
          o[dc][3] *= fix[1];
        }
      }
#pragma unroll
      for (int kk = 0; kk < KEYS / 16; ++kk) {
        uint32_t pa[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const float* x = sc[kk * 2 + n];
          const float p0 = fast_exp2(fmaf(x[0], p.scale_log2, neg[0])), p1 = fast_exp2(fmaf(x[1], p.scale_log2, neg[0]));
          const float p2 = fast_exp2(fmaf(x[2], p.scale_log2, neg[1])), p3 = fast_exp2(fmaf(x[3], p.scale_log2, neg[1]));
          lrow[0] += p0 + p1;
          lrow[1] += p2 + p3;
          if (WIDE) {                                        // rows 0 (thread group 0), 1 (group 1) and 8 (group 0): the three parts
            float hi[2], mid[2], lo[2];
            sh_split(p0, hi[0], mid[0], lo[0]);
            sh_split(p1, hi[1], mid[1], lo[1]);
            pa[n * 2 + 0] = gq == 0 ? sh_pack(hi[0], hi[1]) : gq == 1 ? sh_pack(lo[0], lo[1]) : 0u;
            pa[n * 2 + 1] = gq == 0 ? sh_pack(mid[0], mid[1]) : 0u;
          } else {
            pa[n * 2 + 0] = sh_pack(p0, p1);
            pa[n * 2 + 1] = sh_pack(p2, p3);
          }
        }
#pragma unroll
        for (int dc = 0; dc < HD / 8; dc += 2) {
          const int key = wk * KEYS + kk * 16 + (mtx & 1) * 8 + lr;
          const int dchunk = dc + (mtx >> 1);
          uint32_t r0, r1, r2, r3;
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                       : "r"(v_tile + (dchunk / 8) * C::SUB_BYTES + (uint32_t)(key * 128 + (((dchunk & 7) ^ (key & 7)) << 4))));
          if (WIDE) {
            float f0[4] = {0.f, 0.f, 0.f, 0.f}, f1[4] = {0.f, 0.f, 0.f, 0.f};
            mma_bf16(f0, pa, r0, r1);
            mma_bf16(f1, pa, r2, r3);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              o[dc][e] = __fadd_rn(o[dc][e], f0[e]);
              o[dc + 1][e] = __fadd_rn(o[dc + 1][e], f1[e]);
            }
          } else {
            mma_bf16(o[dc], pa, r0, r1);
            mma_bf16(o[dc + 1], pa, r2, r3);
          }
        }
      }
      fence_reads_before_async_writes();
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_bar(s));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      lrow[h] += __shfl_xor_sync(0xffffffffu, lrow[h], 1);
      lrow[h] += __shfl_xor_sync(0xffffffffu, lrow[h], 2);
    }
    if (WIDE) {                                              // the row's three parts meet in the threads of row 0
#pragma unroll
      for (int dc = 0; dc < HD / 8; ++dc)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float lo = __shfl_down_sync(0xffffffffu, o[dc][e], 4);
          o[dc][e] = __fadd_rn(o[dc][e], __fadd_rn(o[dc][e + 2], lo));
        }
    }
    if (WK == 1 && parts == 1) {                            // a row's only piece: straight out
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = wr * 16 + gq + 8 * h, x = row0 + r, tok = x / G;
        if (r >= rows) continue;
        __nv_bfloat16* dst = p.out + (size_t)(q_start + tok) * p.ldo + (size_t)(kvh * G + x - tok * G) * HD + 2 * t;
        const float inv = 1.0f / lrow[h];
#pragma unroll
        for (int dc = 0; dc < HD / 8; ++dc)
          *reinterpret_cast<uint32_t*>(dst + dc * 8) = sh_pack(o[dc][2 * h] * inv, o[dc][2 * h + 1] * inv);
      }
      return;                                               // (nobody waits behind: the barriers below are skipped by all)
    }
    // this warp's rows to shared memory, where the ring was: every page that was asked for has been read by all warps
    asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float* mine = results + (size_t)(wk * ROWS + wr * 16 + gq + 8 * h) * C::OUT_PITCH;
#pragma unroll
      for (int dc = 0; dc < HD / 8; ++dc)
        *reinterpret_cast<float2*>(mine + dc * 8 + 2 * t) = make_float2(o[dc][2 * h], o[dc][2 * h + 1]);
      if (t == 0) {
        mine[HD] = mrow[h];
        mine[HD + 1] = lrow[h];
      }
    }
  }
  if (WK == 1 && parts == 1) return;           // (the producer)
  if (parts > 1) cluster.sync(); else __syncthreads();

  // ---- the cluster's rows dealt out over its warps, up to four rows of a warp at a time (a row is a chain of reads from
  // another SM and shuffles: one by one the 16 rows of a warp were 4 us); the pieces (block, key group) in that order ----
  if (warp < SH_CONSUMERS) {
    const int n_pieces = parts * WK, step = parts * SH_CONSUMERS;      // (at most 32 pieces)
    const int z = min(lane, n_pieces - 1);
    const float* mine = cluster.map_shared_rank(results, z / WK) + (size_t)(z % WK) * ROWS * C::OUT_PITCH;
    auto merge = [&](int r0, auto batch) {                             // rows r0, r0 + step, ..
      constexpr int RB = decltype(batch)::value;
      float w[RB], lw[RB], L[RB], acc[RB][HD / 32];
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        const float* at = mine + (size_t)(r0 + i * step) * C::OUT_PITCH;
        w[i] = lane < n_pieces ? at[HD] : -INFINITY;
        lw[i] = lane < n_pieces ? at[HD + 1] : 0.f;
        L[i] = 0.f;
#pragma unroll
        for (int u = 0; u < HD / 32; ++u) acc[i][u] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        const float M = warp_max(w[i]);
        w[i] = (w[i] == -INFINITY) ? 0.f : fast_exp2(w[i] - M);
        lw[i] *= w[i];
      }
#pragma unroll 2
      for (int b = 0; b < parts; ++b) {
        const float* from = cluster.map_shared_rank(results, b) + lane;
#pragma unroll
        for (int g = 0; g < WK; ++g)
#pragma unroll
          for (int i = 0; i < RB; ++i) {
            const float* at = from + (size_t)(g * ROWS + r0 + i * step) * C::OUT_PITCH;
            const float wz = __shfl_sync(0xffffffffu, w[i], b * WK + g);
            L[i] += __shfl_sync(0xffffffffu, lw[i], b * WK + g);
#pragma unroll
            for (int u = 0; u < HD / 32; ++u) acc[i][u] = fmaf(wz, at[32 * u], acc[i][u]);
          }
      }
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        const int x = row0 + r0 + i * step, tok = x / G;
        __nv_bfloat16* dst = p.out + (size_t)(q_start + tok) * p.ldo + (size_t)(kvh * G + x - tok * G) * HD + lane;
        const float inv = 1.0f / L[i];
#pragma unroll
        for (int u = 0; u < HD / 32; ++u) dst[32 * u] = __float2bfloat16_rn(acc[i][u] * inv);
      }
    };
    int r0 = part + parts * warp;
    for (; r0 + 3 * step < rows; r0 += 4 * step) merge(r0, std::integral_constant<int, 4>());
    for (; r0 + step < rows; r0 += 2 * step) merge(r0, std::integral_constant<int, 2>());
    if (r0 < rows) merge(r0, std::integral_constant<int, 1>());
  }
  if (parts > 1) cluster.sync();               // nobody's shared memory goes while it is read
}

typedef CUresult (*ShEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The cache of one layer as a matrix [pages * kv_heads * 64 rows, head_dim]: tiles of [64 rows, 64 columns].
static int sh_cache_map(CUtensorMap* map, const void* ptr, long rows, int head_dim) {
  static ShEncodeFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return LLMI_ERR_DRIVER;
    fn = (ShEncodeFn)sym;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)head_dim, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)head_dim * 2};
  const cuuint32_t box[2] = {64, 64};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? LLMI_OK
             : LLMI_ERR_DRIVER;
}

template <int HD, int ROWS, bool FUSE, bool WIDE>
static int sh_launch(const CUtensorMap& mk, const CUtensorMap& mv, const ShortParams& p, int n_items, int parts, cudaStream_t stream) {
  using C = ShCfg<HD>;
  static PerDevice<bool> configured_on;
  bool& configured = configured_on.here();
  if (!configured) {
    if (cudaFuncSetAttribute(attention_short_kernel<HD, ROWS, FUSE, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
      return LLMI_ERR_LAUNCH;
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_items * parts);
  cfg.blockDim = dim3(SH_THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled(PDL_ATTENTION) ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)parts;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  pairs_may_start_early = false;
  return cudaLaunchKernelEx(&cfg, attention_short_kernel<HD, ROWS, FUSE, WIDE>, mk, mv, p) == cudaSuccess ? LLMI_OK : LLMI_ERR_LAUNCH;
}

template <int HD>
static int sh_launch_rows(const CUtensorMap& mk, const CUtensorMap& mv, const ShortParams& p, int n_items, int rows, int parts,
                          bool wide, cudaStream_t stream) {
  if constexpr (HD == 128)
    if (wide)
      return p.k_cache_w ? sh_launch<HD, 16, true, true>(mk, mv, p, n_items, parts, stream)
                         : sh_launch<HD, 16, false, true>(mk, mv, p, n_items, parts, stream);
  if (p.k_cache_w) return sh_launch<HD, 16, true, false>(mk, mv, p, n_items, parts, stream);
  if (rows <= 16) return sh_launch<HD, 16, false, false>(mk, mv, p, n_items, parts, stream);
  if (rows <= 32) return sh_launch<HD, 32, false, false>(mk, mv, p, n_items, parts, stream);
  return sh_launch<HD, 64, false, false>(mk, mv, p, n_items, parts, stream);
}

}  // namespace llmi

using namespace llmi;

// q: [tokens, >= n_heads * head_dim] rotated queries, the cache complete; otherwise as llmi_attention_prefill.  max_q: the most
// tokens a sequence brings; parts: blocks that share a (sequence, kv head, row tile): 1, 2, 4 or 8.
// fuse = 1 (max_q 1, groups up to 16): a decode step as for llmi_attention_decode_fused — `q` is the step's un-rotated
// [q | k | v] rows, rotary_dim is head_dim or 0, the new k (rotated) and v are appended with write_kv.
// wide = 1 (max_q 1, ungrouped heads of 128): 32-bit weights.
// early = 1: what earlier steps left of the step's sequences was complete before the launch ahead began (a model's step: the copy of its
// index block lies between), so that it may be read before that launch has ended.
LLMI_EXPORT int llmi_attention_short(const void* q, long ldq, void* out, long ldo, void* k_cache, void* v_cache,
                                     long n_cache_pages, const int32_t* seq_pages, int pages_stride, const int32_t* seq_q_start,
                                     const int32_t* seq_kv_len, int n_seqs, int max_q, int n_heads, int n_kv_heads, int head_dim,
                                     float scale, int window, int parts, int fuse, const float* inv_freq, int rotary_dim,
                                     int write_kv, int wide, int early, int* error_flag, cudaStream_t stream) {
  if (n_seqs <= 0 || max_q <= 0 || n_heads <= 0 || n_kv_heads <= 0 || n_cache_pages <= 0) return LLMI_ERR_BAD_SIZE;
  if (n_heads % n_kv_heads || (parts != 1 && parts != 2 && parts != 4 && parts != 8)) return LLMI_ERR_BAD_SIZE;
  if (head_dim != 64 && head_dim != 128) return LLMI_ERR_UNSUPPORTED;
  if (((uintptr_t)q & 3) || (ldq & 1) || ((uintptr_t)out & 3) || (ldo & 1) || ((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15)) return LLMI_ERR_ALIGN;
  const int group = n_heads / n_kv_heads;
  if (fuse && (max_q != 1 || group > 16 || (rotary_dim != 0 && (rotary_dim != head_dim || !inv_freq)))) return LLMI_ERR_UNSUPPORTED;
  if (wide && (max_q != 1 || group != 1 || head_dim != 128)) return LLMI_ERR_UNSUPPORTED;
  const long rows = n_cache_pages * n_kv_heads * SH_PAGE, tile_rows = (long)max_q * group;
  const long tiles = (tile_rows + SH_MAX_ROWS - 1) / SH_MAX_ROWS, items = (long)n_seqs * n_kv_heads * tiles;
  if (rows > 0x7fffffffL || items * parts > 0x7fffffffL) return LLMI_ERR_BAD_SIZE;
  CUtensorMap mk, mv;
  int rc = sh_cache_map(&mk, k_cache, rows, head_dim);
  if (rc != LLMI_OK) return rc;
  rc = sh_cache_map(&mv, v_cache, rows, head_dim);
  if (rc != LLMI_OK) return rc;
  ShortParams p{(const __nv_bfloat16*)q, ldq, (__nv_bfloat16*)out, ldo, seq_pages, seq_q_start, seq_kv_len, pages_stride, n_kv_heads,
                group, (int)tiles, scale * 1.4426950408889634f, window, error_flag, inv_freq, fuse ? rotary_dim : 0, n_heads,
                write_kv ? 1 : 0, fuse ? (__nv_bfloat16*)k_cache : nullptr, fuse ? (__nv_bfloat16*)v_cache : nullptr, early};
  const int per_tile = (int)(tile_rows < SH_MAX_ROWS ? tile_rows : SH_MAX_ROWS);
  return head_dim == 64 ? sh_launch_rows<64>(mk, mv, p, (int)items, per_tile, parts, wide != 0, stream)
                        : sh_launch_rows<128>(mk, mv, p, (int)items, per_tile, parts, wide != 0, stream);
}
