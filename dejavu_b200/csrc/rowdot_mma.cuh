// rowdot_mma: y[b, m] = act( w[idx[m], :] . x[b, :] + bias[idx[m]] ) for up to 32 rows of x on the tensor cores, fp16 or
// bf16 in. With this many rows of x the CUDA-core kernel would issue 8*B FMAs per 16-byte weight chunk, which no longer
// hides behind the HBM stream. Every gathered row is read once; the streaming is weight_ring.cuh's.
#pragma once
#include "rowdot.cuh"
#include "weight_ring.cuh"

namespace djv {

template <typename T, typename TO, int ACT>
struct RowdotSource {
  TO *Y;
  const T *W, *X;
  const void *idx;
  const T *bias;
  int M, N, idx64, B;
  long long ldw;
  float act_param;
  int first, last, rows, S, rank;  // rows of the cluster, of its tiles; the block's place in it
  // of the thread's pieces: the rows of the tile being copied, the row numbers of the one after it
  const T *row[WR_WP];
  long long next[WR_WP];
  int k;
  float bias0, bias1;

  __device__ __forceinline__ void look_up(int t) {
#pragma unroll
    for (int i = 0; i < WR_WP; ++i) {
      const int r = (int)threadIdx.x / WR_PPR + WR_RP * i, m = first + t * rows + r;
      next[i] = r < rows && m < last ? load_index(idx, m, idx64) : -1;
    }
  }
  __device__ __forceinline__ void seek(int t, int c) {
    if (c == 0) {
      if (t == 0) look_up(0);
#pragma unroll
      for (int i = 0; i < WR_WP; ++i) row[i] = next[i] < 0 ? nullptr : W + next[i] * ldw;
      look_up(t + 1);
    }
    k = (c * S + rank) * WR_K + (int)threadIdx.x % WR_PPR * 8;  // N % 8 == 0: a piece is inside the row or entirely outside
  }
  __device__ __forceinline__ const void *w(int i, bool &ok) const {
    ok = k < N;
    return row[i] != nullptr ? row[i] + (ok ? k : 0) : nullptr;
  }
  __device__ __forceinline__ const void *x(int i, bool &ok) const {
    const int b = (int)threadIdx.x / WR_PPR + WR_RP * i;
    ok = k < N;
    return b < B ? X + (size_t)b * N + (ok ? k : 0) : nullptr;
  }
  __device__ __forceinline__ void begin(int t) {  // (a thread finishes the same pair of every token)
    bias0 = bias1 = 0.f;
    if (is_glu(ACT) || bias == nullptr) return;
    const int pairs = WR_ROWS / 2 / S, m = first + t * rows + 2 * (rank * pairs + (int)threadIdx.x % pairs);
    if (m < last) bias0 = to_f(bias[load_index(idx, m, idx64)]);
    if (m + 1 < last) bias1 = to_f(bias[load_index(idx, m + 1, idx64)]);
  }
  __device__ __forceinline__ void store(int t, int pair, int b, float2 v) const {
    const int m = first + t * rows + 2 * pair;
    if (2 * pair >= rows) return;
    if constexpr (is_glu(ACT)) {  // rows 2i, 2i + 1 are the gate and up rows of output i (no bias in this form)
      if (m < last) Y[(size_t)b * (M / 2) + m / 2] = from_f<TO>(apply_glu<ACT>(v.x, v.y, act_param));
    } else {
      if (m < last) Y[(size_t)b * M + m] = from_f<TO>(apply_act_param<ACT>(v.x + bias0, act_param));
      if (m + 1 < last) Y[(size_t)b * M + m + 1] = from_f<TO>(apply_act_param<ACT>(v.y + bias1, act_param));
    }
  }
};

template <typename T, typename TO, int NT, int ACT, int PART>  // NT groups of 8 rows of x
__global__ void __launch_bounds__(WR_THREADS, WR_BPS)
rowdot_mma_kernel(TO *__restrict__ Y, const T *__restrict__ W, const T *__restrict__ X, const void *__restrict__ idx,
                  const T *__restrict__ bias, int M, int N, long long ldw, int idx64, int B, float act_param, int per, int rest) {
  extern __shared__ __align__(128) unsigned char wr_smem[];
  constexpr int UNIT = is_glu(ACT) ? 2 : 1;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), cl = blockIdx.x / S;
  const int first = (cl * per + min(cl, rest)) * UNIT, last = first + (per + (cl < rest ? 1 : 0)) * UNIT;
  const int tiles = ceil_div_dev(last - first, WR_ROWS), rows = ceil_div_dev(ceil_div_dev(last - first, tiles), 2) * 2;
  const int all = ceil_div_dev(N, WR_K), chunks = (all - rank + S - 1) / S;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (idx == nullptr) {  // the weights that fill the ring are asked for while the kernel before this one is still running
    constexpr int PL = WR_K / 64, LINES = (WeightRing<NT>::STAGES - 1) * PL;
    for (int l = threadIdx.x; l < WR_ROWS * LINES; l += WR_THREADS) {
      const int m = first + l / LINES, k = (l % LINES / PL * S + rank) * WR_K + l % PL * 64;
      if (l / LINES < rows && m < last && k < N) prefetch_l2(W + m * ldw + k);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  RowdotSource<T, TO, ACT> src{Y, W, X, idx, bias, M, N, idx64, B, ldw, act_param, first, last, rows, S, rank};
  weight_ring<T, NT, PART>(src, tiles, chunks, B, wr_smem);
}

// (internal linkage: each library prepares its own copy of the kernel)
template <typename T, typename TO, int NT, int ACT, int PART = 0>
static int launch_rowdot_mma(TO *Y, const T *W, const T *X, const void *idx, const T *bias, int M, int N, long long ldw,
                             int idx64, int B, float act_param, cudaStream_t st) {
  constexpr int UNIT = is_glu(ACT) ? 2 : 1;
  static DevicePrep prep;
  const int (*resident)[4];
  const cudaError_t prepared = prep.get([](int (&r)[4]) { return ring_residency<NT>(rowdot_mma_kernel<T, TO, NT, ACT, PART>, r); }, resident);
  if (prepared != cudaSuccess) {
    set_error("rowdot_mma: %s", cudaGetErrorString(prepared));
    return DJV_ERR_CUDA;
  }
  const RingPlan p = ring_plan(M / UNIT, UNIT, ceil_div(N, WR_K), *resident);
  djv::launch_kernel_cluster(rowdot_mma_kernel<T, TO, NT, ACT, PART>, dim3(p.clusters * p.S), dim3(WR_THREADS),
                             (size_t)WeightRing<NT>::BYTES, st, dim3(p.S), Y, W, X, idx, bias, M, N, ldw, idx64, B, act_param,
                             p.per, p.rest);
  count_launch();
  return DJV_OK;
}

}  // namespace djv
