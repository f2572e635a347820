// rowdot_mma: y[b, m] = act( w[idx[m], :] . x[b, :] + bias[idx[m]] ) for up to 32 rows of x on the tensor cores, fp16 or
// bf16 in. With this many rows of x the CUDA-core kernel would issue 8*B FMAs per 16-byte weight chunk, which no longer
// hides behind the HBM stream. Every gathered row is read once. Two forms: rowdot_mma_kernel, streamed by weight_ring.cuh, and
// rowdot_mma_short_kernel for products that are over before a ring has been worth filling.
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

// -------------------------------------------------------------------------------------------
// Short lists. A block owns 16 rows; its 8 warps split the columns (warp w takes 32-column blocks w, w + 8, ..), and so do the S
// blocks of a cluster where the tiles alone leave multiprocessors idle. Lane (g, t) loads 16 contiguous bytes of rows g and g + 8
// and of token rows g, 8 + g, ..: the order along k is the same on both sides. Bound by the chain row numbers, weights, sums of the
// warps, sums of the cluster: nothing is staged, so nothing has to fill and drain.
// -------------------------------------------------------------------------------------------
constexpr int MS_THREADS = 256;
constexpr int MS_WARPS = MS_THREADS / WARP;
constexpr int MS_ROWS = 16;
// A block asks for up to 8 KB of each of its rows before it waits for the kernel before it, a row a thread: a LayerNorm, under which
// HBM has little to do. 16 steps of 8 layers, 4096 wide, 16 sequences 11829 -> 11477 us, 12 sequences, 4 layers 6732 -> 6608. (The ring
// form, line by line of a list: up to 1 % slower with 5 and 8 sequences.)

template <typename T, typename TO, int NT, int ACT>  // NT groups of 8 activation rows
__global__ void __launch_bounds__(MS_THREADS, NT == 1 ? 5 : 1)
rowdot_mma_short_kernel(TO *__restrict__ Y, const T *__restrict__ W, const T *__restrict__ X,
                  const void *__restrict__ idx, const T *__restrict__ bias, int M, int N,
                  long long ldw, int idx64, int B, float act_param, int ahead) {
  __shared__ float red[MS_WARPS][NT][MS_ROWS][8];
  __shared__ float bsum[NT][MS_ROWS][8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int S = gridDim.y, sblk = blockIdx.y;
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP;
  const int g = lane / 4, t = lane % 4;
  const int m0 = blockIdx.x * MS_ROWS;
  const int m_lo = m0 + g, m_hi = m0 + g + 8;
  if (ahead > 0) {  // the block's share of its rows, of those below `ahead` (known to exist), while the kernel before this one runs
    const AheadSpan s = ahead_share(sblk, S, N * (int)sizeof(T));
    if (tid < MS_ROWS && m0 + tid < M && s.bytes > 0) {
      const long long r = load_index(idx, m0 + tid, idx64);
      if (ahead_takes(r, ahead)) bulk_prefetch_l2(reinterpret_cast<const char *>(W + r * ldw) + s.offset, s.bytes);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const long long r_lo = (m_lo < M) ? load_index(idx, m_lo, idx64) : -1;
  const long long r_hi = (m_hi < M) ? load_index(idx, m_hi, idx64) : -1;
  const T *w_lo = W + (r_lo < 0 ? 0 : r_lo) * ldw;
  const T *w_hi = W + (r_hi < 0 ? 0 : r_hi) * ldw;

  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

  const int kblocks = (N + 31) / 32;
  // weight and activation loads of U k-blocks are all issued before the first MMA needs them
  constexpr int U = 2;
  for (int kb0 = sblk * MS_WARPS + warp; kb0 < kblocks; kb0 += MS_WARPS * S * U) {
    uint4 a_lo[U], a_hi[U], xv[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (kb0 + u * MS_WARPS * S) * 32 + t * 8;
      const bool ok = k < N;  // N % 8 == 0: a 16-byte piece is inside the row or entirely outside
      a_lo[u] = (ok && r_lo >= 0) ? ld_stream16(w_lo + k) : make_uint4(0, 0, 0, 0);
      a_hi[u] = (ok && r_hi >= 0) ? ld_stream16(w_hi + k) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int tok = j * 8 + g;
        xv[u][j] = (ok && tok < B) ? ld_cached16(X + (size_t)tok * N + k) : make_uint4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        // blocks past the end of the row hold zeros on both sides and add nothing
        float s[4] = {};
        mma_m16n8k16_t<T>(s, a_lo[u].x, a_hi[u].x, a_lo[u].y, a_hi[u].y, xv[u][j].x, xv[u][j].y);
        mma_m16n8k16_t<T>(s, a_lo[u].z, a_hi[u].z, a_lo[u].w, a_hi[u].w, xv[u][j].z, xv[u][j].w);
        add_sums(acc[j], s);
      }
    }
  }
  // acc[j]: rows g (e 0,1) and g+8 (e 2,3), tokens j*8 + 2t (e 0,2) and j*8 + 2t+1 (e 1,3)
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    red[warp][j][g][2 * t] = acc[j][0];
    red[warp][j][g][2 * t + 1] = acc[j][1];
    red[warp][j][g + 8][2 * t] = acc[j][2];
    red[warp][j][g + 8][2 * t + 1] = acc[j][3];
  }
  __syncthreads();
  namespace cgx = cooperative_groups;
  cgx::cluster_group cluster = cgx::this_cluster();
  if (S > 1) {
    // this block's sums, then the cluster's
    for (int o = tid; o < NT * MS_ROWS * 8; o += MS_THREADS) {
      const int j = o / (MS_ROWS * 8), row = (o / 8) % MS_ROWS, c = o % 8;
      float s = 0.f;
#pragma unroll
      for (int w2 = 0; w2 < MS_WARPS; ++w2) s += red[w2][j][row][c];
      bsum[j][row][c] = s;
    }
    cluster.sync();
  }
  if (sblk == 0) {
    for (int o = tid; o < NT * MS_ROWS * 8; o += MS_THREADS) {
      const int j = o / (MS_ROWS * 8), row = (o / 8) % MS_ROWS, c = o % 8;
      const int m = m0 + row, tok = j * 8 + c;
      if (m < M && tok < B) {
        auto total = [&](int at) {  // sum of one (row, token) over the warps, and over the blocks of the cluster
          float s = 0.f;
          if (S > 1) {
            for (int q = 0; q < S; ++q) s += cluster.map_shared_rank(&bsum[0][0][0], q)[at];
          } else {
            const int jj = at / (MS_ROWS * 8), rr = (at / 8) % MS_ROWS, cc = at % 8;
#pragma unroll
            for (int w2 = 0; w2 < MS_WARPS; ++w2) s += red[w2][jj][rr][cc];
          }
          return s;
        };
        if (is_glu(ACT)) {
          // rows 2i, 2i + 1 are the gate and up rows of output i (no bias in this form)
          if (row % 2 == 0 && m + 1 < M)
            Y[(size_t)tok * (M / 2) + m / 2] = from_f<TO>(apply_glu<ACT>(total(o), total(o + 8), act_param));
        } else {
          float s = total(o);
          if (bias != nullptr) s += to_f(bias[load_index(idx, m, idx64)]);
          Y[(size_t)tok * M + m] = from_f<TO>(apply_act_param<ACT>(s, act_param));
        }
      }
    }
  }
  if (S > 1) cluster.sync();  // no block leaves while block 0 may still read its sums
}

// Blocks of the cluster that split the reduction; `bps` is the kernel's occupancy.
inline int rowdot_mma_short_split(int M, int N, int NT, int bps) {
  const int tiles = ceil_div(M, MS_ROWS);
  // Split the reduction over the S blocks of a cluster when the tiles alone leave multiprocessors idle.
  const int slots = sm_count() * bps;
  // Measured behaviour: the resident blocks run in waves; a wave costs a fixed ~5 us (row numbers, first loads,
  // reduction, cluster barriers) plus, per k-block of 32 columns a warp walks, the larger of a latency floor that
  // grows with the activation rows and the wave's bytes per k-block step (8 KB per block) over the HBM rate.
  // S in {1, 2, 4, 8} (other cluster sizes measured slower than either neighbour), every warp keeps >= 4 k-blocks.
  const int kblocks = (N + 31) / 32;
  int S = 1;
  double best = 1e30;
  for (int c = 1; c <= 8; c *= 2) {
    if (c > 1 && kblocks < MS_WARPS * c * 4) break;
    const double kb_per_warp = (double)ceil_div(kblocks, MS_WARPS * c);
    const double floor_us = 0.6 + 0.23 * NT;
    double t = 0.0;
    for (int left = tiles * c; left > 0; left -= slots) {
      const int nb = left < slots ? left : slots;
      const double bw_us = nb * 8192.0 / 6.5e6;
      t += 5.0 + kb_per_warp * (floor_us > bw_us ? floor_us : bw_us);
    }
    if (t < best - 1e-9) {
      best = t;
      S = c;
    }
  }
  return S;
}

// Which form. us, short / ring, bf16 with fp32 result, fp16 gathered with bias (64 matrices in turn: those below a million elements
// stay in L2; of 128 rows spread over 3072 x 768 and 8 rows of x the ring has 3.8, this form 4.2):
//   16 rows of x: 512 x 512 2.0 / 2.6, 2.5 / 3.6; 1024 x 1024 3.6 / 4.9, 4.3 / 5.4; 4096 x 1024 4.2 / 4.5, 4.9 / 5.6; 2048 x 2048
//     5.3 / 6.2, 6.1 / 7.6; 1024 x 4096 5.2 / 5.7, 6.0 / 7.4; 512 x 12288 6.5 / 7.4, 7.2 / 8.3. But 6144 x 1024 6.7 / 4.6, 8.3 / 6.1;
//     512 x 2048 4.6 / 4.5, 5.4 / 5.2; 3072 x 2048 6.1 / 5.8, 6.9 / 6.9; 1024 x 12288 9.6 / 8.2, 10.5 / 10.2.
//   8 rows: 256 x 1024 2.8 / 3.4, 3.1 / 4.1; 2048 x 512 2.8 / 3.1, 3.4 / 3.8; but 512 x 1024 4.2 / 3.9, 4.7 / 4.6; 2048 x 1024
//     4.6 / 4.4, 5.4 / 5.0; 1024 x 2048 5.6 / 4.5, 6.5 / 5.6. And short rows whose tiles fill the resident blocks once: 11264 x 2048
//     10.4 / 10.9, 11.1 / 13.3; 11264 x 768 5.4 / 5.9, 5.9 / 8.0; but 8192 x 2048 9.4 / 6.6, 10.1 / 8.5.
inline bool rowdot_mma_is_short(int M, int N, int NT, int blocks) {
  if (NT > 1) return N <= 1024 ? M <= 4096 : N <= 4096 ? M > 512 && M <= 2048 : M <= 512;
  const int tiles = ceil_div(M, MS_ROWS);
  return (N <= 512 && M <= 2048) || (N <= 1024 && M <= 256) || (N <= 2048 && tiles <= blocks && tiles * 10 >= blocks * 9);
}

// (internal linkage: each library prepares its own copy of the kernels)
template <typename T, typename TO, int NT, int ACT, int PART = 0>
static int launch_rowdot_mma(TO *Y, const T *W, const T *X, const void *idx, const T *bias, int M, int N, long long ldw,
                             int idx64, int B, float act_param, cudaStream_t st) {
  constexpr int UNIT = is_glu(ACT) ? 2 : 1;
  if constexpr (PART == 0) {
    static DevicePrep prep;
    const int (*fit)[4];
    const cudaError_t asked = prep.get([](int (&r)[4]) {
      return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r[0], rowdot_mma_short_kernel<T, TO, NT, ACT>, MS_THREADS, 0);
    }, fit);
    if (asked != cudaSuccess) {
      set_error("rowdot_mma: %s", cudaGetErrorString(asked));
      return DJV_ERR_CUDA;
    }
    const int per_sm = max(1, (*fit)[0]);
    if (rowdot_mma_is_short(M, N, NT, per_sm * sm_count())) {
      const int S = rowdot_mma_short_split(M, N, NT, per_sm);
      djv::launch_kernel_cluster(rowdot_mma_short_kernel<T, TO, NT, ACT>, dim3(ceil_div(M, MS_ROWS), S), dim3(MS_THREADS), 0, st,
                                 dim3(1, S, 1), Y, W, X, idx, bias, M, N, ldw, idx64, B, act_param, idx == nullptr ? M : early_rows(0));
      count_launch();
      return DJV_OK;
    }
  }
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
