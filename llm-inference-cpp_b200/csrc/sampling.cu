// Next-token choice on the device: first-maximum argmax, and temperature / top-k / top-p
// sampling with an inverse-CDF draw.
//
// Reference semantics (src/model/sampling.cpp:11-76; include/llmi/model/sampling.hpp:11-24):
//   p = softmax(logits / temperature); order by p descending, equal values by ascending id;
//   keep the first k (top_k == 0 or > n keeps all); if top_p < 1 keep the shortest prefix whose
//   running sum reaches top_p (never fewer than one); renormalise by the kept sum; walk ids in
//   ascending order and return the first id whose running sum reaches u.
// Argmax returns the first maximum (src/model/transformer.cpp:22-24).
//
// A cluster of eight blocks takes a row; each block holds an eighth of the ids' probabilities in its shared memory, and
// sums, counts and maxima over the row go through the blocks' shared memories.  The kept set is found in one of two ways:
//
//  * with a top_k of at most 512 (what chats are sampled with): each block finds the top_k-th largest of its threads' own
//    maxima, a bound that at least top_k values reach; the largest bound of the eight lets few more than top_k values
//    through (where a peaked row has fewer probabilities above 0, the bound is the smallest number above 0: what is 0 is
//    never drawn and adds nothing to a mass).  Those (up to 1,024) go to the first block, which ranks them by (value descending, id ascending), cuts the
//    ranks after top_k and top_p, and draws from the kept ones in id order: no pass over the row per bit.
//  * otherwise: the kept set is { p > thr } plus the first n_eq ids with p == thr, and (thr, n_eq) is found by building
//    thr's bit pattern from the top bit down with counting (top-k) or mass (top-p) passes: probabilities are non-negative
//    floats, so their bit patterns order like their values.
//
// Counts are integers and masses are summed in double in a fixed order, so a row's result does not depend on which other
// rows are in the launch.
//
// What bounds it: one block per row, its 31 bits' passes for top_k and 31 more for top_p each over the whole row, took
// 304 us for a row of 49,152 with top_k 50 and top_p 0.95, a fifth of a decode step at batch 1.  This way 20 us (8 rows
// the same, 64 rows 43 us; peaked rows 20 and 37 us); the general way 56 us with top_k 0 and top_p 0.95.
//
// `probs` is caller-provided scratch of n_rows * vocab floats (used when an eighth of a row exceeds shared memory).
#include <cooperative_groups.h>
#include <math.h>

#include "common.cuh"

namespace llmi {

constexpr int SAMPLE_THREADS = 1024;

__global__ void __launch_bounds__(SAMPLE_THREADS)
argmax_kernel(const float* __restrict__ logits, long ld, int vocab, int32_t* __restrict__ out) {
  __shared__ float best_v[32];
  __shared__ int best_i[32];
  pdl_launch_dependents();
  pdl_wait();
  const float* row = logits + (size_t)blockIdx.x * ld;
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  if ((vocab & 3) == 0 && (((uintptr_t)row) & 15) == 0) {
    const float4* r4 = reinterpret_cast<const float4*>(row);
    for (int i = threadIdx.x; i < (vocab >> 2); i += blockDim.x) {   // ascending i: the first maximum stays
      const float4 v = r4[i];
      if (bi == 0x7fffffff || v.x > bv) { bv = v.x; bi = 4 * i; }
      if (v.y > bv) { bv = v.y; bi = 4 * i + 1; }
      if (v.z > bv) { bv = v.z; bi = 4 * i + 2; }
      if (v.w > bv) { bv = v.w; bi = 4 * i + 3; }
    }
  } else {
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      const float v = row[i];
      if (bi == 0x7fffffff || v > bv) { bv = v; bi = i; }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { best_v[warp] = bv; best_i[warp] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (best_v[w] > bv || (best_v[w] == bv && best_i[w] < bi)) { bv = best_v[w]; bi = best_i[w]; }
    out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
  }
}

namespace cg = cooperative_groups;

constexpr int SAMPLE_CLUSTER = 8;            // blocks per row (the largest portable cluster)
constexpr int SAMPLE_ROW_THREADS = 512;      // threads of each
constexpr int SAMPLE_WARPS = SAMPLE_ROW_THREADS / 32;
constexpr int SAMPLE_LIST = 1024;            // values that may pass the top-k bound

// Reductions over a block, and over the cluster, in a fixed order: lanes by butterfly, then the warps' results by butterfly
// again in every warp, then the blocks in rank order.  Every thread gets the result.  A block's part goes to a mailbox in
// every block of the cluster; two mailboxes take turns, so that one barrier a reduction is enough (a mailbox is written
// again only behind the next reduction's barrier, which no block reaches before it has read this one).
struct RowReduce {
  double* d;                                  // [32]
  double (*box)[SAMPLE_CLUSTER];              // [2][blocks]
  int parity;
  template <typename V> __device__ V block_sum(V v) {
    V* buf = reinterpret_cast<V*>(d);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) buf[warp] = v;
    __syncthreads();
    V t = lane < SAMPLE_WARPS ? buf[lane] : V(0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  }
  // every block's value, in rank order, for all of them: box[..][rank]
  __device__ const double* exchange(double v) {
    cg::cluster_group cluster = cg::this_cluster();
    parity ^= 1;
    if (threadIdx.x < SAMPLE_CLUSTER) *cluster.map_shared_rank(&box[parity][cluster.block_rank()], threadIdx.x) = v;
    cluster.sync();
    return box[parity];
  }
  __device__ double sum(double v) {
    const double* all = exchange(block_sum(v));
    double t = 0;
#pragma unroll
    for (int r = 0; r < SAMPLE_CLUSTER; ++r) t += all[r];
    return t;
  }
  __device__ long long count(int v) {         // exact: a count fits the mailbox's double
    const double* all = exchange((double)block_sum(v));
    double t = 0;
#pragma unroll
    for (int r = 0; r < SAMPLE_CLUSTER; ++r) t += all[r];
    return (long long)t;
  }
  __device__ float max(float v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) d[warp] = (double)v;
    __syncthreads();
    v = warp_max(lane < SAMPLE_WARPS ? (float)d[lane] : -INFINITY);
    const double* all = exchange((double)v);
#pragma unroll
    for (int r = 0; r < SAMPLE_CLUSTER; ++r) v = fmaxf(v, (float)all[r]);
    return v;
  }
  // Exclusive prefix sums over the threads of the block in thread order, and the block's total: lanes by shuffles, then
  // the warps' totals the same way.
  template <typename V> __device__ V block_scan(V v, V* total) {
    V* buf = reinterpret_cast<V*>(d);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    V incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    __syncthreads();
    if (lane == 31) buf[warp] = incl;
    __syncthreads();
    V w = lane < SAMPLE_WARPS ? buf[lane] : V(0);
    V wincl = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V up = __shfl_up_sync(0xffffffffu, wincl, o);
      if (lane >= o) wincl += up;
    }
    const V warp_base = __shfl_sync(0xffffffffu, wincl - w, warp);
    *total = __shfl_sync(0xffffffffu, wincl, SAMPLE_WARPS - 1);
    return warp_base + (incl - v);
  }
  // ... over the cluster's threads: blocks in rank order before them
  __device__ double scan(double v, double* total) {
    double mine;
    const double before = block_scan(v, &mine);
    const double* all = exchange(mine);
    const int rank = (int)cg::this_cluster().block_rank();
    double base = 0, t = 0;
#pragma unroll
    for (int r = 0; r < SAMPLE_CLUSTER; ++r) {
      if (r == rank) base = t;
      t += all[r];
    }
    *total = t;
    return base + before;
  }
};

// (three blocks an SM: with the 52 registers that are taken otherwise two, 64 rows 51 -> 59 us)
__global__ void __cluster_dims__(SAMPLE_CLUSTER, 1, 1) __launch_bounds__(SAMPLE_ROW_THREADS, 3)
sample_kernel(const float* __restrict__ logits, long ld, int vocab, float temperature, int top_k, float top_p,
              const double* __restrict__ uniforms, float* __restrict__ probs, int32_t* __restrict__ out, int chunk,
              int probs_in_smem) {
  __shared__ double red_d[32];
  __shared__ double red_box[2][SAMPLE_CLUSTER];
  __shared__ int result_first, result_last, n_list;
  __shared__ uint2 list[SAMPLE_LIST];         // (value's bits, id); in the first block: of the whole row
  __shared__ uint2 kept_list[SAMPLE_ROW_THREADS];
  extern __shared__ float smem_probs[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), seq = blockIdx.x / SAMPLE_CLUSTER;
  RowReduce red{red_d, red_box, 0};
  constexpr int NT = SAMPLE_ROW_THREADS;
  const int tid = threadIdx.x;
  const float* row = logits + (size_t)seq * ld;
  const int id0 = min(vocab, rank * chunk), n = min(vocab, id0 + chunk) - id0;      // this block's ids: id0 .. id0 + n - 1
  row += id0;
  float* p = probs_in_smem ? smem_probs : probs + (size_t)seq * vocab + id0;
  const uint32_t* pb = reinterpret_cast<const uint32_t*>(p);
  if (tid == 0) {
    result_first = 0x7fffffff;
    result_last = -1;
    n_list = 0;
  }
  pdl_launch_dependents();
  cluster.sync();                             // every block of the cluster runs: its shared memory may be written
  pdl_wait();

  // softmax(logits / temperature), denominator in double; the scaled logits wait in p for the maximum
  float mx = -INFINITY;
  for (int i = tid; i < n; i += NT) {
    const float x = row[i] / temperature;
    p[i] = x;
    mx = fmaxf(mx, x);
  }
  mx = red.max(mx);
  double part = 0;
  for (int i = tid; i < n; i += NT) {
    const float e = expf(p[i] - mx);
    p[i] = e;
    part += (double)e;
  }
  const double denom = red.sum(part);
  const float inv = (float)(1.0 / denom);
  uint32_t own = 0;                           // largest bit pattern among this thread's probabilities
  for (int i = tid; i < n; i += NT) {
    p[i] *= inv;
    own = max(own, pb[i]);
  }
  const long long k = (top_k <= 0 || top_k > vocab) ? vocab : top_k;

  if (k <= NT) {
    // ---- few candidates ----
    // the k-th largest of the threads' maxima (0 when fewer than that are above 0), bit by bit; at least k values of this
    // block, so of the row, reach it
    uint32_t bound = 0;
    for (int bit = 30; bit >= 0; --bit) {
      const uint32_t cand = bound | (1u << bit);
      if (__syncthreads_count(own >= cand) >= k) bound = cand;
    }
    const double* all = red.exchange((double)bound);
#pragma unroll
    for (int r = 0; r < SAMPLE_CLUSTER; ++r) bound = max(bound, (uint32_t)all[r]);
    bound = max(bound, 1u);                   // (the other ids of the k have probability 0)
    int* counter = cluster.map_shared_rank(&n_list, 0);
    uint2* dst = cluster.map_shared_rank(list, 0);
    if (own >= bound)
      for (int i = tid; i < n; i += NT)
        if (pb[i] >= bound) {
          const int at = atomicAdd(counter, 1);
          if (at < SAMPLE_LIST) dst[at] = make_uint2(pb[i], (uint32_t)(id0 + i));
        }
    cluster.sync();
    const int m = *counter;
    if (m <= SAMPLE_LIST) {
      cluster.sync();                         // every block has read the counter: the first may go on alone, and end
      if (rank != 0) return;
      // ranks by (value descending, id ascending); the first k of them, in rank order, into kept_list
      for (int i = tid; i < m; i += NT) {
        const uint2 me = list[i];
        int before = 0;
        for (int j = 0; j < m; ++j) {
          const uint2 o = list[j];
          before += o.x > me.x || (o.x == me.x && o.y < me.y);
        }
        if (before < k) kept_list[before] = me;
      }
      __syncthreads();
      const int found = (int)min(k, (long long)m);      // (fewer than k only where the others are 0)
      const bool in_k = tid < found;
      const uint2 me = in_k ? kept_list[tid] : make_uint2(0u, 0u);
      const double mine = in_k ? (double)__uint_as_float(me.x) : 0.0;
      int n_kept = found;
      if (top_p < 1.0f) {
        // the shortest prefix whose running sum reaches top_p (all of them when none does), at least one
        double total;
        const double upto = red.block_scan(mine, &total) + mine;
        const int below = __syncthreads_count(in_k && !(upto >= (double)top_p));
        n_kept = min(found, below + 1);
      }
      // the kept ones in id order
      const bool in = tid < n_kept;
      int before = 0;
      if (in)
        for (int j = 0; j < n_kept; ++j) before += kept_list[j].y < me.y;
      if (in) list[before] = me;
      __syncthreads();
      const uint2 at = in ? list[tid] : make_uint2(0u, 0u);
      const double v = in ? (double)__uint_as_float(at.x) : 0.0;
      double kept;
      const double cum = red.block_scan(v, &kept) + v;
      const double target = uniforms[seq] * kept;
      if (in && !(__uint_as_float(at.x) <= 0.f)) {
        if (cum >= target) atomicMin(&result_first, (int)at.y);
        atomicMax(&result_last, (int)at.y);
      }
      __syncthreads();
      if (tid == 0) out[seq] = result_first != 0x7fffffff ? result_first : (result_last >= 0 ? result_last : 0);
      return;
    }
    // (so many equal values at the bound: the general way)
  }
  __syncthreads();

  // ---- the general way ----
  // top-k: thr_k = the k-th largest value; n_eq = how many of the ties at thr_k are kept
  uint32_t thr = 0;
  long long n_eq;
  if (k < vocab) {
    for (int bit = 30; bit >= 0; --bit) {  // bit 31 is the sign: never set
      const uint32_t cand = thr | (1u << bit);
      int c = 0;
      for (int i = tid; i < n; i += NT) c += pb[i] >= cand;
      if (red.count(c) >= k) thr = cand;
    }
    int c = 0;
    for (int i = tid; i < n; i += NT) c += pb[i] > thr;
    n_eq = k - red.count(c);
  } else {
    int c = 0;
    for (int i = tid; i < n; i += NT) c += pb[i] == 0u;
    n_eq = red.count(c);  // thr = 0: everything is kept
  }

  // top-p inside the top-k set
  if (top_p < 1.0f) {
    const uint32_t thr_k = thr;
    const long long n_eq_k = n_eq;
    const double tie_mass_k = (double)n_eq_k * (double)__uint_as_float(thr_k);
    double m = 0;
    for (int i = tid; i < n; i += NT) m += pb[i] > thr_k ? (double)p[i] : 0.0;
    const double total_k = red.sum(m) + tie_mass_k;
    if (total_k >= (double)top_p) {
      // largest value v (>= thr_k) with mass{p >= v, in the set} >= top_p
      uint32_t t2 = 0;
      for (int bit = 30; bit >= 0; --bit) {
        const uint32_t cand = t2 | (1u << bit);
        double mm = 0;
        for (int i = tid; i < n; i += NT) mm += (pb[i] >= cand && pb[i] > thr_k) ? (double)p[i] : 0.0;
        mm = red.sum(mm);
        if (cand <= thr_k) mm += tie_mass_k;
        if (mm >= (double)top_p) t2 = cand;
      }
      if (t2 < thr_k) t2 = thr_k;
      double mg = 0;
      int ce = 0;
      for (int i = tid; i < n; i += NT) {
        mg += pb[i] > t2 ? (double)p[i] : 0.0;
        ce += pb[i] == t2;
      }
      mg = red.sum(mg);
      long long avail = red.count(ce);
      if (t2 == thr_k) avail = n_eq_k;
      const double tv = (double)__uint_as_float(t2);
      long long need = 1;
      double cum = mg + tv;
      while (cum < (double)top_p && need < avail) { cum += tv; ++need; }
      thr = t2;
      n_eq = need;
    }
  }

  // kept set = { p > thr } + the first n_eq ids with p == thr.  Each thread owns a contiguous id range; ranks of ties and
  // running sums come from scans over the threads in id order.
  const int own_ids = (n + NT - 1) / NT;
  const int i0 = min(n, tid * own_ids), i1 = min(n, i0 + own_ids);
  int eq_local = 0;
  for (int i = i0; i < i1; ++i) eq_local += pb[i] == thr;
  double eq_total;
  int eq_rank = (int)red.scan((double)eq_local, &eq_total);
  const int eq_rank0 = eq_rank;
  double local = 0;
  for (int i = i0; i < i1; ++i) {
    if (pb[i] > thr) local += (double)p[i];
    else if (pb[i] == thr) { if (eq_rank < n_eq) local += (double)p[i]; ++eq_rank; }
  }
  double kept;
  const double mass_before = red.scan(local, &kept);
  const double target = uniforms[seq] * kept;
  double cum = mass_before;
  eq_rank = eq_rank0;
  int first = 0x7fffffff, last = -1;
  for (int i = i0; i < i1; ++i) {
    bool in = false;
    if (pb[i] > thr) in = true;
    else if (pb[i] == thr) { in = eq_rank < n_eq; ++eq_rank; }
    if (!in || p[i] <= 0.f) continue;
    cum += (double)p[i];
    last = id0 + i;
    if (cum >= target && first == 0x7fffffff) first = id0 + i;
  }
  if (first != 0x7fffffff) atomicMin(cluster.map_shared_rank(&result_first, 0), first);
  if (last >= 0) atomicMax(cluster.map_shared_rank(&result_last, 0), last);
  cluster.sync();
  if (rank == 0 && tid == 0) out[seq] = result_first != 0x7fffffff ? result_first : (result_last >= 0 ? result_last : 0);
}

}  // namespace llmi

using namespace llmi;

LLMI_EXPORT int llmi_argmax(const float* logits, long ld, int n_rows, int vocab, int32_t* out, cudaStream_t stream) {
  if (n_rows <= 0 || vocab <= 0) return LLMI_ERR_BAD_SIZE;
  return launch_pdl(PDL_SMALL, argmax_kernel, n_rows, SAMPLE_THREADS, 0, stream, logits, ld, vocab, out);
}

// temperature must be > 0 (the caller maps temperature <= 0 to llmi_argmax, as the reference does).
LLMI_EXPORT int llmi_sample(const float* logits, long ld, int n_rows, int vocab, float temperature, int top_k,
                            float top_p, const double* uniforms, float* probs_scratch, int32_t* out,
                            cudaStream_t stream) {
  if (n_rows <= 0 || vocab <= 0) return LLMI_ERR_BAD_SIZE;
  if (!(temperature > 0.f)) return LLMI_ERR_UNSUPPORTED;
  if (n_rows > 0x7fffffff / SAMPLE_CLUSTER) return LLMI_ERR_BAD_SIZE;
  // an eighth of a row's probabilities per block, in shared memory up to 200 KB
  const int chunk = (vocab + SAMPLE_CLUSTER - 1) / SAMPLE_CLUSTER;
  const size_t bytes = (size_t)chunk * sizeof(float);
  static PerDevice<int> room_on;
  int& room = room_on.here();                 // 0: not asked yet, -1: none
  if (room == 0) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, current_device());
    room = v - 20 * 1024;                     // the kernel's static arrays take 12.8 KB
    if (room <= 0 || cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, room) != cudaSuccess) room = -1;
  }
  const int in_smem = room > 0 && bytes <= (size_t)room ? 1 : 0;
  return launch_pdl(PDL_SMALL, sample_kernel, n_rows * SAMPLE_CLUSTER, SAMPLE_ROW_THREADS, in_smem ? bytes : 0, stream, logits, ld,
                    vocab, temperature, top_k, top_p, uniforms, probs_scratch, out, chunk, in_smem);
}
