// y = x · Wᵀ (+ bias) with fp32 FMA arithmetic on the CUDA cores.
//
// This is the true 32-bit matrix product of the library (no tensor-core mode, no
// reduced-precision inputs when T = float) and the fallback for bf16 shapes the
// tensor-core kernel refuses.  W is [out, in] row-major as the reference stores it
// (include/llmi/model/kernels.hpp:15-17; src/model/kernels.cpp:97-113), x is [rows, in].
//
// The order of additions, the same in every kernel of this file: k is cut into segments of SEG places anchored at 0; a
// segment's sum is one running fmaf chain from 0 in ascending k; an output is the sum of its segments' sums in ascending
// order.  So the value of y[r, o] does not depend on how many rows are in the call, where r lies or which of the kernels a
// call's size selects — and the segments of an output can be worked on at the same time.  (One chain over all of k, as
// before, left a decode step of the 32-bit path nothing to do in parallel but its outputs; against 64 bits the sum of
// segments is the nearer one.)
//
// Three kernels:
//  * linear_simt_kernel: any type, pitch and alignment (a tile of 64 x 64 outputs, scalar loads), and fp32 rows of short k;
//  * linear_f32_tile_kernel: fp32, 16-byte rows, many tokens: four segments of a 64 x 64 tile at a time;
//  * linear_f32_rows_kernel: fp32, 16-byte rows, few tokens: bound by reading w once.
#include "common.cuh"
#include "sm100.cuh"

namespace llmi {

constexpr int BM = 64, BN = 64, BK = 16;
constexpr int SEG = 256;          // k places of a segment (a multiple of BK)

// Output modes of the product.
constexpr int OUT_STORE = 0;      // y (type T) = acc
constexpr int OUT_STORE_F32 = 1;  // y (float) = acc
constexpr int OUT_ADD_F32 = 2;    // y (float) += acc       (residual sum kept in fp32)

template <typename T, int MODE>
__device__ __forceinline__ void put_output(void* yv, long at, int n, float v, const float* bias, const float* oscale) {
  if (bias) v = __fadd_rn(v, bias[n]);
  if (oscale) v = __fmul_rn(v, oscale[n]);
  if (MODE == OUT_STORE) {
    ((T*)yv)[at] = from_f32<T>(v);
  } else if (MODE == OUT_STORE_F32) {
    ((float*)yv)[at] = v;
  } else {
    float* p = (float*)yv + at;
    *p = __fadd_rn(*p, v);
  }
}

template <typename T, int MODE>
__global__ void __launch_bounds__(256)
linear_simt_kernel(const T* __restrict__ x, long ldx, const T* __restrict__ w, long ldw,
                   const float* __restrict__ bias, const float* __restrict__ oscale, void* __restrict__ yv, long ldy, int M, int N, int K,
                   long bx, long bw, long by) {
  // blockIdx.z numbers the products of a batch (one per head, say): operand b starts bx, bw, by elements further on
  x += (long)blockIdx.z * bx;
  w += (long)blockIdx.z * bw;
  yv = MODE == OUT_STORE ? (void*)((T*)yv + (long)blockIdx.z * by) : (void*)((float*)yv + (long)blockIdx.z * by);
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int lr = tid >> 2;        // row of the tile this thread loads
  const int lk = (tid & 3) * 4;   // first of its four k

  float acc[4][4], total[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = total[i][j] = 0.f;

  // The next k block is fetched into registers while the current one is multiplied, so that a block pays the
  // latency of global memory once, not once per k block.  The order of the additions is untouched.
  const int m_ld = m0 + lr, n_ld = n0 + lr;
  float a_next[4], b_next[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = k0 + lk + e;
      a_next[e] = (m_ld < M && k < K) ? to_f32(x[(long)m_ld * ldx + k]) : 0.f;
      b_next[e] = (n_ld < N && k < K) ? to_f32(w[(long)n_ld * ldw + k]) : 0.f;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      As[lk + e][lr] = a_next[e];
      Bs[lk + e][lr] = b_next[e];
    }
    __syncthreads();
    if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if ((k0 + BK) % SEG == 0 || k0 + BK >= K) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          total[i][j] = __fadd_rn(total[i][j], acc[i][j]);
          acc[i][j] = 0.f;
        }
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      put_output<T, MODE>(yv, (long)m * ldy + n, n, total[i][j], bias, oscale);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Many tokens.  Bound by the FMA pipes (128 a clock and SM; 74 TFLOP/s, of which 8 x 8 products out of registers alone reach
// 55).  800 tokens x 960 -> 5,120: 225 us, 35 TFLOP/s: a block takes 31 us for its 4 segments and the last of 7.03 waves is
// nearly empty.  (Two blocks of half the stages on an SM were slower, and so were tiles of 64 x 128: as many FMAs a clock, fewer
// tiles for the SMs.)  A block makes a tile of 64 x 64 outputs; its four groups of 64
// threads take segments 4r, 4r + 1, .. of round r, each thread 8 x 8 outputs in registers (one 16-byte shared load per 16
// FMAs where 4 x 4 outputs need two).  With the segments side by side a block keeps two warps of independent chains
// on every scheduler though its tile is small, and small tiles fill the 148 SMs at the widths of small models (600 tokens x
// 960 outputs are 150 tiles).  Operands go to shared memory as they lie (rows of 32 k places, 36 floats apart: a quarter
// warp's 16-byte loads touch 32 different banks) by cp.async, two stages a group.  A stage costs a barrier of the group, its copies'
// addresses and the first loads' latency, which two warps a scheduler do not cover: stages of 16 places, three of them, took 251
// us for those 800 tokens, and 3 to 11 % more over 65 to 1,500 tokens and the widths of 576 to 5,120 (four requests of the 360M
// shape in fp32 37.4 -> 35.7 ms).  The same chains: the same bits.
constexpr int TILE_STAGES = 2;
constexpr int TILE_BK = 32;            // k places of a stage
constexpr int TILE_PITCH = TILE_BK + 4;
constexpr int TILE_STAGE_FLOATS = (BM + BN) * TILE_PITCH;
constexpr int TOTAL_PITCH = BN + 8;
constexpr int TILE_SMEM = (4 * TILE_STAGES * TILE_STAGE_FLOATS + BM * TOTAL_PITCH) * (int)sizeof(float);

__device__ __forceinline__ void cp_async_16(float* dst, const float* src, bool real) {
  const int bytes = real ? 16 : 0;               // 0: the place is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void group_barrier(int group) { asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory"); }

template <int MODE>
__global__ void __launch_bounds__(256, 1)
linear_f32_tile_kernel(const float* __restrict__ x, long ldx, const float* __restrict__ w, long ldw, const float* __restrict__ bias,
                       const float* __restrict__ oscale, float* __restrict__ y, long ldy, int M, int N, int K, long bx, long bw, long by) {
  extern __shared__ __align__(16) float tile_smem[];
  x += (long)blockIdx.z * bx;
  w += (long)blockIdx.z * bw;
  y += (long)blockIdx.z * by;
  const int group = threadIdx.x >> 6, t = threadIdx.x & 63;
  const int tx = t & 7, ty = t >> 3;             // outputs (ty + 8 i, tx + 8 j)
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float* stages = tile_smem + group * TILE_STAGES * TILE_STAGE_FLOATS;
  float* total = tile_smem + 4 * TILE_STAGES * TILE_STAGE_FLOATS;
  for (int i = threadIdx.x; i < BM * TOTAL_PITCH; i += 256) total[i] = 0.f;

  const int n_seg = (K + SEG - 1) / SEG;
  for (int round = 0; round * 4 < n_seg; ++round) {
    const int seg = round * 4 + group;
    const int k_begin = seg * SEG, k_end = min(K, k_begin + SEG);
    const int steps = seg < n_seg ? (k_end - k_begin + TILE_BK - 1) / TILE_BK : 0;
    auto load = [&](int step) {
      float* s = stages + (step % TILE_STAGES) * TILE_STAGE_FLOATS;
      const int k = k_begin + step * TILE_BK + (t & 7) * 4;
#pragma unroll
      for (int e = 0; e < 16; ++e) {             // rows 0..63 of x, then 64 rows of w
        const int r = (t >> 3) + e * 8;
        const bool of_x = e < 8;
        const int row = of_x ? m0 + r : n0 + r - BM;
        const bool real = k < k_end && row < (of_x ? M : N);
        const float* src = of_x ? x + (long)row * ldx + k : w + (long)row * ldw + k;
        cp_async_16(s + r * TILE_PITCH + (t & 7) * 4, real ? src : x, real);
      }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
      if (s < steps) load(s);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int step = 0; step < steps; ++step) {
      asm volatile("cp.async.wait_group %0;" ::"n"(TILE_STAGES - 2) : "memory");
      group_barrier(group);                      // this step's rows are here, and everybody is done with the step before's
      if (step + TILE_STAGES - 1 < steps) load(step + TILE_STAGES - 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float* s = stages + (step % TILE_STAGES) * TILE_STAGE_FLOATS;
#pragma unroll 2
      for (int q = 0; q < TILE_BK / 4; ++q) {
        float4 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(s + (ty + 8 * i) * TILE_PITCH + 4 * q);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 b = *reinterpret_cast<const float4*>(s + (BM + tx + 8 * j) * TILE_PITCH + 4 * q);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
        }
      }
    }
    // the segments join the total one after another, in ascending order
    for (int g = 0; g < 4; ++g) {
      __syncthreads();
      if (g == group && seg < n_seg) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float* p = total + (ty + 8 * i) * TOTAL_PITCH + tx + 8 * j;
            *p = __fadd_rn(*p, acc[i][j]);
          }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < BM * BN; i += 256) {
    const int m = m0 + i / BN, n = n0 + i % BN;
    if (m < M && n < N) put_output<float, MODE>(y, (long)m * ldy + n, n, total[(i / BN) * TOTAL_PITCH + i % BN], bias, oscale);
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Few tokens.  Bound by reading w once, and by latency: a decode step of a small model is a chain of such products.  A block
// takes ROWS rows of w; rows and tokens go to shared memory in segments of 256 places (places 260 floats apart: a quarter
// warp's 16-byte loads of its four rows touch different banks), w, where the caller says that the kernel before does not write
// it (`early`: a model's weights), before that kernel has ended (a request step of the 360M shape 39.9 -> 38.9 ms).  A thread makes the sums of one segment for two rows and two (or four) tokens: 4 (6) shared loads of 16 bytes per 16
// (32) FMAs, which is what a block spends its time on: with one row a thread it is 1.5 (1.7) times as many.  A chain of 256
// FMAs is 1,024 clocks, half a microsecond, whatever K is, where one chain over K = 2,560 is 5 us.
// Four tokens, as they follow one another in a step (rows of w x K): 960 x 960 22.3 -> 6.0 us, 5,120 x 960 23.4 -> 11.3, 960 x
// 2,560 41.9 -> 7.1 against the form whose threads had one row, four tokens and x through L1.
constexpr int ROWS = 8;
constexpr int SEG_PITCH = SEG + 4;
constexpr int ROWS_PASS = 16;         // tokens in shared memory at a time
constexpr int ROWS_MAX_TOKENS = 64;
constexpr int ROWS_THREADS = 128;     // at least: an output of a pass per thread

template <int MODE, int TOKENS>
__global__ void __launch_bounds__(512)
linear_f32_rows_kernel(const float* __restrict__ x, long ldx, const float* __restrict__ w, long ldw, const float* __restrict__ bias,
                       const float* __restrict__ oscale, float* __restrict__ y, long ldy, int M, int N, int K, int staged, int pass,
                       int early, long bx, long bw, long by) {
  extern __shared__ __align__(16) float rows_smem[];
  x += (long)blockIdx.z * bx;
  w += (long)blockIdx.z * bw;
  y += (long)blockIdx.z * by;
  float* w_s = rows_smem;                                             // [staged][ROWS][SEG_PITCH]
  float* x_s = w_s + staged * ROWS * SEG_PITCH;                       // [staged][pass][SEG_PITCH]
  float* part = x_s + staged * pass * SEG_PITCH;                      // [staged][pass][ROWS]
  const int tid = threadIdx.x, n_threads = blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, n_warps = n_threads >> 5;
  const int n0 = blockIdx.x * ROWS, n_rows = min(ROWS, N - n0);
  const int n_seg = (K + SEG - 1) / SEG;
  const int groups = pass / TOKENS;                                   // groups of tokens of a pass
  const int row = tid & 3, tg = (tid >> 2) % groups, seg_lane = (tid >> 2) / groups;      // rows `row` and `row` + 4
  const int seg_lanes = (n_threads >> 2) / groups;
  pdl_launch_dependents();
  bool waited = !early;
  if (!early) pdl_wait();
  float total[ROWS_MAX_TOKENS / ROWS_PASS] = {};                      // this thread's output of every pass, over the rounds

  for (int s0 = 0; s0 < n_seg; s0 += staged) {
    const int here = min(staged, n_seg - s0);
    const int k0 = s0 * SEG, pieces = (min(K, (s0 + here) * SEG) - k0) / 4;      // pieces of 16 bytes of a row
    // (rows that do not exist repeat the last one: their sums go nowhere)
    for (int r = warp; r < ROWS; r += n_warps) {
      const float* src = w + (long)(n0 + min(r, n_rows - 1)) * ldw + k0;
      for (int q = lane; q < pieces; q += 32) cp_async_16(w_s + ((q / (SEG / 4)) * ROWS + r) * SEG_PITCH + (q % (SEG / 4)) * 4, src + 4 * q, true);
    }
    if (!waited) {
      pdl_wait();
      waited = true;
    }
#pragma unroll
    for (int turn = 0; turn < ROWS_MAX_TOKENS / ROWS_PASS; ++turn) {
      const int t0 = turn * pass;
      if (t0 >= M) break;
      for (int m = warp; m < pass; m += n_warps) {
        const float* src = x + (long)min(t0 + m, M - 1) * ldx + k0;
        for (int q = lane; q < pieces; q += 32) cp_async_16(x_s + ((q / (SEG / 4)) * pass + m) * SEG_PITCH + (q % (SEG / 4)) * 4, src + 4 * q, true);
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      for (int s = seg_lane; s < here; s += seg_lanes) {
        const int len = min(SEG, K - k0 - s * SEG);
        const float* wr = w_s + (s * ROWS + row) * SEG_PITCH;
        const float* xr = x_s + (s * pass + tg * TOKENS) * SEG_PITCH;
        float acc[2][TOKENS] = {};
#pragma unroll 4
        for (int k = 0; k < len; k += 4) {
          const float4 w0 = *reinterpret_cast<const float4*>(wr + k), w1 = *reinterpret_cast<const float4*>(wr + 4 * SEG_PITCH + k);
#pragma unroll
          for (int e = 0; e < TOKENS; ++e) {
            const float4 xv = *reinterpret_cast<const float4*>(xr + e * SEG_PITCH + k);
            acc[0][e] = fmaf(xv.x, w0.x, acc[0][e]);
            acc[1][e] = fmaf(xv.x, w1.x, acc[1][e]);
            acc[0][e] = fmaf(xv.y, w0.y, acc[0][e]);
            acc[1][e] = fmaf(xv.y, w1.y, acc[1][e]);
            acc[0][e] = fmaf(xv.z, w0.z, acc[0][e]);
            acc[1][e] = fmaf(xv.z, w1.z, acc[1][e]);
            acc[0][e] = fmaf(xv.w, w0.w, acc[0][e]);
            acc[1][e] = fmaf(xv.w, w1.w, acc[1][e]);
          }
        }
#pragma unroll
        for (int e = 0; e < TOKENS; ++e) {
          part[(s * pass + tg * TOKENS + e) * ROWS + row] = acc[0][e];
          part[(s * pass + tg * TOKENS + e) * ROWS + row + 4] = acc[1][e];
        }
      }
      __syncthreads();
      // this pass's outputs (token, row), a thread each: their segments in ascending order
      if (tid < pass * ROWS)
        for (int s = 0; s < here; ++s) total[turn] = __fadd_rn(total[turn], part[s * pass * ROWS + tid]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int turn = 0; turn < ROWS_MAX_TOKENS / ROWS_PASS; ++turn) {
    const int m = turn * pass + tid / ROWS, r = tid % ROWS;
    if (tid < pass * ROWS && m < M && r < n_rows) put_output<float, MODE>(y, (long)m * ldy + n0 + r, n0 + r, total[turn], bias, oscale);
  }
}

template <int MODE, int TOKENS>
int launch_linear_f32_rows(const float* x, long ldx, const float* w, long ldw, const float* bias, const float* oscale, float* y, long ldy,
                           int M, int N, int K, int early, cudaStream_t stream, int batch, long bx, long bw, long by) {
  static PerDevice<bool> configured;
  if (!configured.here()) {
    if (cudaFuncSetAttribute(linear_f32_rows_kernel<MODE, TOKENS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess)
      return LLMI_ERR_LAUNCH;
    configured.here() = true;
  }
  const int pass = M >= ROWS_PASS ? ROWS_PASS : (M + TOKENS - 1) / TOKENS * TOKENS;
  const int n_seg = (K + SEG - 1) / SEG, blocks = (N + ROWS - 1) / ROWS;
  // as many segments at a time as shared memory takes, in rounds of equal size: all of it where every block has an SM of
  // its own, else half, so that one block loads while another multiplies
  const int seg_bytes = ((ROWS + pass) * SEG_PITCH + pass * ROWS) * (int)sizeof(float);
  const int most = ((long)blocks * batch <= sm_count() ? 216 : 108) * 1024 / seg_bytes;
  const int rounds = (n_seg + most - 1) / most, staged = (n_seg + rounds - 1) / rounds;
  int threads = 4 * (pass / TOKENS) * staged;
  threads = threads < ROWS_THREADS ? ROWS_THREADS : (threads > 512 ? 512 : (threads + 31) / 32 * 32);
  return launch_pdl(PDL_GEMM, linear_f32_rows_kernel<MODE, TOKENS>, dim3(blocks, 1, batch), dim3(threads), (size_t)staged * seg_bytes, stream,
                    x, ldx, w, ldw, bias, oscale, y, ldy, M, N, K, staged, pass, early, bx, bw, by);
}

// Which kernel: fp32 rows that 16-byte copies can take go to the two fast ones.  Up to 8 tokens the rows kernel; up to 64 while
// the outputs are so few that the tiles leave SMs idle (rows / tiles: 64 x 1,600 of K = 960: 28.7 / 33.5 us, 64 x 960 of
// K = 2,560: 45 / 83, 32 x 3,072 of K = 576: 15.7 / 21.9; 48 x 3,072: 21.8 / 22.2, 24 x 5,120 of K = 960: 42 / 32).
constexpr long ROWS_MAX_OUTPUTS = 104 * 1024;
template <int MODE>
int launch_linear_f32(const float* x, long ldx, const float* w, long ldw, const float* bias, const float* oscale, float* y, long ldy,
                      int M, int N, int K, int early, cudaStream_t stream, int batch, long bx, long bw, long by) {
  if (M <= 8 || (M <= ROWS_MAX_TOKENS && (long)M * N * batch <= ROWS_MAX_OUTPUTS)) {
    if (M <= 8) return launch_linear_f32_rows<MODE, 2>(x, ldx, w, ldw, bias, oscale, y, ldy, M, N, K, early, stream, batch, bx, bw, by);
    return launch_linear_f32_rows<MODE, 4>(x, ldx, w, ldw, bias, oscale, y, ldy, M, N, K, early, stream, batch, bx, bw, by);
  }
  static PerDevice<bool> configured;
  if (!configured.here()) {
    if (cudaFuncSetAttribute(linear_f32_tile_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM) != cudaSuccess)
      return LLMI_ERR_LAUNCH;
    configured.here() = true;
  }
  linear_f32_tile_kernel<MODE><<<dim3((N + BN - 1) / BN, (M + BM - 1) / BM, batch), 256, TILE_SMEM, stream>>>(
      x, ldx, w, ldw, bias, oscale, y, ldy, M, N, K, bx, bw, by);
  return launch_status();
}

// fp32 rows of 16 bytes that linear_simt_kernel is the faster one for.  The tile kernel's four groups of threads take a segment each:
// with k up to one segment three of them wait.  (us, tile / plain: 1,000 tokens x 4,096 rows of k = 64 53 / 27, 256 126 / 81, 320 131 /
// 102, 512 about equal; x 320 rows of 64 9.3 / 6.7, of 256 19.7 / 16.5, of 320 equal; the rows kernel: 24 x 4,096 of 64 14.5 / 6.0, 40 x 1,024
// of 128 11.2 / 9.2, 24 x 320 of 128 equal.)
inline bool plain_is_faster(int M, int N, int K, int batch) {
  if (M <= 8) return false;
  if (K <= SEG) return !(M <= 24 && K >= 64 && (long)M * N * batch <= 16384);
  return K <= 3 * SEG / 2 && M > ROWS_MAX_TOKENS && (long)((N + BN - 1) / BN) * ((M + BM - 1) / BM) * batch > sm_count();
}

template <typename T>
int launch_linear_simt(const void* x, long ldx, const void* w, long ldw, const float* bias, const float* oscale, void* y, long ldy, int M,
                       int N, int K, int mode, int early, cudaStream_t stream, int batch = 1, long bx = 0, long bw = 0, long by = 0) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
  if (grid.y > 65535 || batch < 1 || batch > 65535) return LLMI_ERR_BAD_SIZE;
  pairs_may_start_early = false;
  const bool rows_of_16 = (((uintptr_t)x | (uintptr_t)w) & 15) == 0 && ((ldx | ldw | bx | bw | (long)K) & 3) == 0;
  const bool plain = plain_is_faster(M, N, K, batch);
#define LLMI_LAUNCH(MODE)                                                                                                     \
  if (sizeof(T) == 4 && rows_of_16 && !plain)                                                                                        \
    return launch_linear_f32<MODE>((const float*)x, ldx, (const float*)w, ldw, bias, oscale, (float*)y, ldy, M, N, K, early,  \
                                   stream, batch, bx, bw, by);                                                                        \
  linear_simt_kernel<T, MODE><<<grid, 256, 0, stream>>>((const T*)x, ldx, (const T*)w, ldw, bias, oscale, y, ldy, M, N, K, bx, bw, by)
  switch (mode) {
    case OUT_STORE: LLMI_LAUNCH(OUT_STORE); break;
    case OUT_STORE_F32: LLMI_LAUNCH(OUT_STORE_F32); break;
    case OUT_ADD_F32: LLMI_LAUNCH(OUT_ADD_F32); break;
    default: return LLMI_ERR_UNSUPPORTED;
  }
#undef LLMI_LAUNCH
  return launch_status();
}

}  // namespace llmi

using namespace llmi;

// x [M, K] (row pitch ldx), w [N, K] (row pitch ldw), y [M, N] (row pitch ldy), pitches in elements; y takes
// (x · wᵀ + bias) * oscale, both [N] or null.  early 1: the launch ahead does not write w (a model's weights), so that it may be
// read before that launch has ended.
LLMI_EXPORT int llmi_linear_simt(int dtype, const void* x, long ldx, const void* w, long ldw, const float* bias, const float* oscale,
                                 void* y, long ldy, int M, int N, int K, int mode, int early, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return LLMI_ERR_BAD_SIZE;
  if (dtype == LLMI_DTYPE_F32) return launch_linear_simt<float>(x, ldx, w, ldw, bias, oscale, y, ldy, M, N, K, mode, early, stream);
  if (dtype == LLMI_DTYPE_BF16)
    return launch_linear_simt<__nv_bfloat16>(x, ldx, w, ldw, bias, oscale, y, ldy, M, N, K, mode, early, stream);
  return LLMI_ERR_BAD_DTYPE;
}

// `batch` products of the same sizes in one launch: product b reads x + b*bx, w + b*bw and writes y + b*by (offsets in
// elements; rows may be strided, so the operands of a batch may interleave: the heads of one activation row).
// Arithmetic and order of additions are those of llmi_linear_simt.
LLMI_EXPORT int llmi_linear_simt_batched(int dtype, const void* x, long ldx, long bx, const void* w, long ldw, long bw,
                                         void* y, long ldy, long by, int batch, int M, int N, int K, int mode, int early,
                                         cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return LLMI_ERR_BAD_SIZE;
  if (dtype == LLMI_DTYPE_F32)
    return launch_linear_simt<float>(x, ldx, w, ldw, nullptr, nullptr, y, ldy, M, N, K, mode, early, stream, batch, bx, bw, by);
  if (dtype == LLMI_DTYPE_BF16)
    return launch_linear_simt<__nv_bfloat16>(x, ldx, w, ldw, nullptr, nullptr, y, ldy, M, N, K, mode, early, stream, batch, bx, bw, by);
  return LLMI_ERR_BAD_DTYPE;
}
