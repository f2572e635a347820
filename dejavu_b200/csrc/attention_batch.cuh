// The projections of a decode step of several sequences that share one lazy-K/V state, on the tensor cores
// (mma.sync m16n8k16, fp16 in, fp32 accumulate): every selected head's weights are read from HBM once, whatever the batch.
//
//   qkv_batch_kernel   q, k, v of the heads in use: B x (1 + slots pending) token rows (of 2 and 3 sequences: see qkv_batch_takes)
//   out_proj_mma_kernel  output projection over the heads in use, up to 16 rows of the context
#pragma once
#include <cooperative_groups.h>

#include "attn_state.cuh"
#include "common.cuh"
#include "mma.cuh"

namespace djv {

// -------------------------------------------------------------------------------------------
// QKV projection. A cluster of S blocks owns one (head, q|k|v): all of its HD weight rows. Block s takes 64 of every
// 64 * S columns of the rows, and up to 64 token rows at a time go through them together; a stage of the ring is
// HD x 64 weights and 64 x 64 activations, brought in by cp.async, swizzled in 16-byte pieces for ldmatrix. The blocks
// of the cluster add up their sums through distributed shared memory, in rank order, each for a part of the rows.
//
// What bounds it: the weights from HBM, if the activations are not read too often. A block of 16 rows with all columns
// (the form before) reads the token rows again for every 16 rows, and the weights again for every 16 token rows.
// Splitting columns instead of rows over the device keeps the activations at 1 / 8 of that. The token rows of many sequences are
// shared out over several clusters per head. 16 sequences, 12 of 32 heads of 128, 4096 wide, mean over the steps of a window (16 to
// 256 token rows), with the step's opening: 38.3 -> 24.9 us, 5.8 of them the weights at copy rate.
// -------------------------------------------------------------------------------------------
constexpr int QB_THREADS = 256, QB_WARPS = QB_THREADS / WARP;
constexpr int QB_K = 64;       // columns of a stage: 128 bytes of a row
constexpr int QB_TOKENS = 64;  // token rows per pass
constexpr int QB_STAGES = 4;   // two blocks per multiprocessor: a cluster of 4 single ones does not fit everywhere

struct QkvBatchArgs {
  const __half *w, *bias;    // (3,nheads,hd,d), (3,nheads,hd) or null
  const __half *x;           // (B,d): the current tokens
  __half *x_ring;            // (B,16,d): the window; this kernel puts x into it
  int *state;
  __half *q, *k_cache, *v_cache;  // (B,nheads,hd), caches of S_cache positions
  int B, d, nheads, S_cache;
};

template <int HD>
struct QkvBatchSmem {
  static constexpr int W_BYTES = HD * QB_K * 2, STAGE = W_BYTES + QB_TOKENS * QB_K * 2;
  static constexpr int RED = QB_WARPS / (HD / 16) * (HD + 4) * QB_TOKENS * 4;  // the sums, where the ring was
  static constexpr size_t BYTES = QB_STAGES * STAGE > RED ? QB_STAGES * STAGE : RED;
};

// up to NT * 8 token rows: the block's share of the products, left where the ring was as [part of k][token][weight row]
template <int HD, int NT>
__device__ __forceinline__ void qkv_batch_products(const __half *w, const __half *const *rows_s, int nr, int d, int rank, int S,
                                                   unsigned char *ring) {
  constexpr int MT = HD / 16, KW = QB_WARPS / MT;  // tiles of 16 weight rows; warps that share one, by steps of k
  constexpr int WP = HD * 8 / QB_THREADS, XP = (NT * 64 + QB_THREADS - 1) / QB_THREADS;  // 16-byte pieces per thread and stage
  constexpr int STAGE = QkvBatchSmem<HD>::STAGE, W_BYTES = QkvBatchSmem<HD>::W_BYTES;
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP;
  const int mt = warp % MT, kw = warp / MT;
  const int r8 = tid / 8, ch = tid % 8;
  const uint32_t base = smem_addr(ring), piece = (uint32_t)(r8 * 128 + ((ch ^ (r8 & 7)) << 4));  // (r8 + 32 swizzles alike)
  const __half *xr[XP];
#pragma unroll
  for (int i = 0; i < XP; ++i) xr[i] = r8 + 32 * i < nr ? rows_s[r8 + 32 * i] : nullptr;
  const int chunks = (d + QB_K - 1) / QB_K, mine = rank < chunks ? (chunks - rank + S - 1) / S : 0;
  auto issue = [&](int it) {
    if (it < mine) {
      const uint32_t dst = base + (uint32_t)(it % QB_STAGES) * STAGE + piece;
      const int k = (it * S + rank) * QB_K + ch * 8;
      const bool ok = k < d;  // d % 8 == 0: a piece is inside the row or entirely outside
#pragma unroll
      for (int i = 0; i < WP; ++i)
        cp_async16_zfill(dst + i * 32 * 128, ok ? w + (size_t)(r8 + 32 * i) * d + k : w, ok ? 16 : 0);
#pragma unroll
      for (int i = 0; i < XP; ++i)
        if (r8 + 32 * i < NT * 8)
          cp_async16_zfill(dst + W_BYTES + i * 32 * 128, ok && xr[i] ? xr[i] + k : w, ok && xr[i] ? 16 : 0);
    }
    cp_async_commit();
  };
  float acc[NT][4] = {};
#pragma unroll
  for (int it = 0; it < QB_STAGES - 1; ++it) issue(it);
  const int ar = mt * 16 + (lane & 15), ac = lane >> 4;             // ldmatrix rows of the weights, of pairs of token tiles
  const int br = (lane & 7) + ((lane >> 4) << 3), bc = (lane >> 3) & 1;
  for (int it = 0; it < mine; ++it) {
    cp_async_wait<QB_STAGES - 2>();
    __syncthreads();  // everybody's copies of this stage have landed, and the stage before has been read
    issue(it + QB_STAGES - 1);
    const uint32_t wb = base + (uint32_t)(it % QB_STAGES) * STAGE, xb = wb + W_BYTES;
    float s[NT][4] = {};
#pragma unroll
    for (int ks = kw; ks < QB_K / 16; ks += KW) {
      uint32_t a[4];
      ldmatrix_x4(a, wb + ar * 128 + (((2 * ks + ac) ^ (ar & 7)) << 4));
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        uint32_t b[4];
        const int row = j * 8 + br;
        ldmatrix_x4(b, xb + row * 128 + (((2 * ks + bc) ^ (row & 7)) << 4));
        mma_m16n8k16(s[j], a[0], a[1], a[2], a[3], b[0], b[1]);
        mma_m16n8k16(s[j + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) add_sums(acc[j], s[j]);
  }
  cp_async_wait<0>();
  __syncthreads();
  float *red = reinterpret_cast<float *>(ring) + kw * NT * 8 * (HD + 4);  // (no two lanes of a store share a bank)
  const int g = lane / 4, t = lane % 4;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) red[(j * 8 + 2 * t + e % 2) * (HD + 4) + mt * 16 + g + e / 2 * 8] = acc[j][e];
}

template <int HD>
__global__ void __launch_bounds__(QB_THREADS, 2) qkv_batch_kernel(QkvBatchArgs a) {
  extern __shared__ __align__(128) unsigned char qb_ring[];
  __shared__ const __half *rows_s[QB_TOKENS];
  __shared__ int code_s[QB_TOKENS];  // (sequence << 4) | window slot of the pass's token rows
  pdl_prologue();
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int pair = blockIdx.x / S, i = pair / 3, qkv = pair % 3;
  // (one trip to memory for all of them: the lists have room for every i)
  const int n_eff = a.state[ST_NEFF], slot = a.state[ST_SLOT], base = a.state[ST_BASE], status = a.state[ST_STATUS];
  const int h = st_eff(a.state, a.nheads)[i];
  const unsigned mask = (qkv == 0) ? (1u << slot) : (unsigned)st_rowmask(a.state, a.nheads)[i];
  if (status == 0) {  // nobody reads row `slot` of a window in this kernel: the current tokens are taken from x
    const int per = a.d / 8;
    for (int b = gridDim.x - 1 - blockIdx.x + gridDim.x * blockIdx.y; b < a.B; b += gridDim.x * gridDim.y) {  // (the last blocks seldom have a head)
      const uint4 *src = reinterpret_cast<const uint4 *>(a.x + (size_t)b * a.d);
      uint4 *dst = reinterpret_cast<uint4 *>(a.x_ring + ((size_t)b * DJV_KV_WINDOW + slot) * a.d);
      for (int c = tid; c < per; c += QB_THREADS) dst[c] = src[c];
    }
  }
  if (i >= n_eff) return;  // (the same for all blocks of a cluster)
  const int pending = __popc(mask);
  const __half *w = a.w + ((size_t)qkv * a.nheads + h) * HD * a.d;
  const __half *bias = a.bias ? a.bias + ((size_t)qkv * a.nheads + h) * HD : nullptr;
  float *red = reinterpret_cast<float *>(qb_ring);
  for (int r0 = blockIdx.y * QB_TOKENS; r0 < a.B * pending; r0 += gridDim.y * QB_TOKENS) {
    const int nr = min(QB_TOKENS, a.B * pending - r0);
    if (tid < nr) {
      const int sq = (r0 + tid) / pending, s = (int)__fns(mask, 0, (r0 + tid) % pending + 1);
      code_s[tid] = (sq << 4) | s;
      rows_s[tid] = s == slot ? a.x + (size_t)sq * a.d : a.x_ring + ((size_t)sq * DJV_KV_WINDOW + s) * a.d;
    }
    __syncthreads();
    int tokens;
    if (nr <= 16) {
      qkv_batch_products<HD, 2>(w, rows_s, nr, a.d, rank, S, qb_ring);
      tokens = 16;
    } else if (nr <= 32) {
      qkv_batch_products<HD, 4>(w, rows_s, nr, a.d, rank, S, qb_ring);
      tokens = 32;
    } else {
      qkv_batch_products<HD, 8>(w, rows_s, nr, a.d, rank, S, qb_ring);
      tokens = 64;
    }
    cluster.sync();
    const int jn = HD / S / 4;  // groups of 4 weight rows that this block finishes
    for (int o = tid; o < jn * nr; o += QB_THREADS) {
      const int j = (rank * jn + o % jn) * 4, tok = o / jn;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int q = 0; q < S; ++q) {
        const float *part = cluster.map_shared_rank(red, q) + tok * (HD + 4) + j;
#pragma unroll
        for (int kw = 0; kw < QB_WARPS / (HD / 16); ++kw) {
          const float4 v = *reinterpret_cast<const float4 *>(part + (size_t)kw * tokens * (HD + 4));
          sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
      }
      if (bias) {
        sum.x += __half2float(bias[j]); sum.y += __half2float(bias[j + 1]);
        sum.z += __half2float(bias[j + 2]); sum.w += __half2float(bias[j + 3]);
      }
      __half2 out[2] = {__floats2half2_rn(sum.x, sum.y), __floats2half2_rn(sum.z, sum.w)};
      const size_t sq = (size_t)(code_s[tok] >> 4), bh = sq * a.nheads + h;
      const int pos = base + (code_s[tok] & (DJV_KV_WINDOW - 1));
      if (qkv == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) a.q[bh * HD + j + e] = reinterpret_cast<__half *>(out)[e];
      } else {
        __half *at = qkv == 1 ? a.k_cache + ((bh * (HD / 8) + j / 8) * a.S_cache + pos) * 8 + j % 8
                              : a.v_cache + (bh * a.S_cache + pos) * HD + j;
        *reinterpret_cast<uint2 *>(at) = *reinterpret_cast<uint2 *>(out);
      }
    }
    cluster.sync();  // the sums have been read by everybody: the ring may be used again, and no block leaves before
  }
}

// A few sequences stay with qkv_sparse_kernel, whose blocks take 8 to 32 rows with all columns each, so that a step is one wave of
// loads: two, and three of middling width, unless the rows are so few that it would put a block on each. us a step with its opening,
// qkv_sparse_kernel / qkv_batch_kernel, mean over a window: two sequences, 12 of 32 heads of 64, 2048 wide 10.4 / 11.1, 12 of 32 of
// 128, 4096 wide 15.0 / 17.3, 16 of 40, 5120 wide 21.5 / 20.7, 24 of 72, 9216 wide 43.2 / 51.7, one head of 64, 768 wide 12.7 / 7.9;
// three 11.4 / 11.4, 17.0 / 17.6, 24.9 / 21.2; four 12.3 / 11.6, 18.4 / 18.1, 28.2 / 23.0.
inline bool qkv_batch_takes(int B, int heads, int d, int hd) {
  return (long long)heads * 3 * hd < 2 * sm_count() || B > 3 || (B == 3 && (d <= 2048 || d > 4096));
}

// Blocks per cluster: the blocks run in rounds of what is resident, a round takes a block's column chunks, and the time of 4 to 6 of
// them for filling the ring and adding up, 8 in clusters of 8. us at heads of 128, 16 sequences, clusters of 1 / 2 / 4 / 8: 4096
// wide, 12 heads 82 / 49 / 32 / 28 (two sequences 31 / 20 / 17 / 20), 9216 wide, 24 heads 204 / 113 / 82 / 72 (65 / 45 / 53 / 52).
// Clusters per head (grid.y), each with a share of the passes over token rows: a window leaves up to 16 rows for each sequence,
// in a step with all heads for all of them. A cluster without rows is gone at once, and the weights come from L2 for all but the
// first. us for 1 / 2 / 4: 4 of 12 heads of 64, 768 wide, 32 sequences 17.8 / 13.0 / 11.3 (qkv_sparse_kernel 17.0), 64 sequences
// 29.5 / 20.1 / 14.7 (24.8); 12 of 32 of 128, 4096 wide, 16 sequences 31.6 / 24.9 / 24.7, 8 sequences 21.7 / 21.3 / 21.3.
struct QkvBatchPlan {
  int S, shares;
};
inline QkvBatchPlan qkv_batch_plan(int B, int heads, int d, int hd, const int (&resident)[4]) {
  const int chunks = ceil_div(d, QB_K), pairs = 3 * (heads > 0 ? heads : 1);
  QkvBatchPlan best{1, B < 8 ? 1 : B < 32 ? 2 : 4};
  const int chunk = B < 4 ? 2 : 3;
  long long least = -1;
  for (int i = 0, S = 1; i < 4 && S <= chunks && S * 4 <= hd; ++i, S *= 2) {
    if (resident[i] < 1) continue;
    const long long cost = (long long)ceil_div(pairs, resident[i]) * (chunk * ceil_div(chunks, S) + (S == 8 ? 18 : 12));
    if (least < 0 || cost < least) {
      least = cost;
      best.S = S;
    }
  }
  return best;
}

template <int HD>
static int launch_qkv_batch(const QkvBatchArgs &a, int heads, cudaStream_t st) {
  constexpr size_t smem = QkvBatchSmem<HD>::BYTES;
  static_assert(smem <= 113 * 1024, "shared memory of two blocks");
  static DevicePrep prep;
  const int (*resident)[4];
  const cudaError_t prepared = prep.get([](int (&r)[4]) {
    return cluster_residency(qkv_batch_kernel<HD>, QB_THREADS, (int)smem, 2, r);
  }, resident);
  if (prepared != cudaSuccess) {
    set_error("attn_step: %s", cudaGetErrorString(prepared));
    return DJV_ERR_CUDA;
  }
  const QkvBatchPlan p = qkv_batch_plan(a.B, heads, a.d, HD, *resident);
  djv::launch_kernel_cluster(qkv_batch_kernel<HD>, dim3(a.nheads * 3 * p.S, p.shares), dim3(QB_THREADS), smem, st, dim3(p.S), a);
  return DJV_OK;
}

// -------------------------------------------------------------------------------------------
// Output projection, weight in the (d, nheads, hd) layout, for 5..16 rows of the context: a block owns 16 output rows, its
// 8 warps split the 32-column pieces of the heads in use. Lane (g, t) loads 16 contiguous bytes of weight rows g and
// g + 8 and of context rows g and g + 8: the order along k is the same on both sides. (CUDA cores in slices of 8 and 4
// rows, each reading the weights again, took 23.6 us at 16 rows, 12 of 32 heads of 128, width 4096; this 8.2.)
// With the caller's word that the heads are known, the weights are asked for under the attention kernel: 16 steps of 8 layers with
// 16 sequences 11621 -> 11481 us.
// -------------------------------------------------------------------------------------------
constexpr int OM_THREADS = 256, OM_WARPS = OM_THREADS / WARP, OM_ROWS = 16;

template <int HD, int NT>
__global__ void __launch_bounds__(OM_THREADS)
out_proj_mma_kernel(__half *__restrict__ Y, const __half *__restrict__ W, const __half *__restrict__ X,
                    const int *__restrict__ head_idx, const int *__restrict__ n_active_dev, const __half *__restrict__ bias,
                    int B, int d, int nheads, int nnz, int early) {
  __shared__ float red[OM_WARPS][NT][OM_ROWS][8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (early) {  // the heads are known: their columns of the block's rows, while the attention before this kernel is still running
    const int n_pf = n_active_dev ? min(nnz, *n_active_dev) : nnz;
    for (int o = threadIdx.x; o < n_pf * OM_ROWS; o += OM_THREADS) {
      const int n = blockIdx.x * OM_ROWS + o % OM_ROWS, h = head_idx[o / OM_ROWS];
      if (n < d && ahead_takes(h, nheads)) bulk_prefetch_l2(W + ((size_t)n * nheads + h) * HD, HD * 2);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr int PIECES = HD / 32, U = NT == 1 ? 6 : 4;
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP, g = lane / 4, t = lane % 4;
  const int n0 = blockIdx.x * OM_ROWS;
  const bool ok_lo = n0 + g < d, ok_hi = n0 + g + 8 < d;
  const size_t ld = (size_t)nheads * HD;
  const __half *w_lo = W + (size_t)(n0 + g) * ld + t * 8, *w_hi = w_lo + 8 * ld, *xg = X + (size_t)g * ld + t * 8;
  const int total = (n_active_dev ? min(nnz, *n_active_dev) : nnz) * PIECES;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  float acc[NT][4] = {};
  for (int p0 = warp; p0 < total; p0 += OM_WARPS * U) {
    uint4 lo[U], hi[U], x[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = p0 + u * OM_WARPS;
      const bool ok = p < total;
      const size_t at = ok ? (size_t)head_idx[p / PIECES] * HD + p % PIECES * 32 : 0;
      lo[u] = ok && ok_lo ? ld_stream16(w_lo + at) : zero;
      hi[u] = ok && ok_hi ? ld_stream16(w_hi + at) : zero;
#pragma unroll
      for (int j = 0; j < NT; ++j) x[u][j] = ok && j * 8 + g < B ? ld_cached16(xg + j * 8 * ld + at) : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        float s[4] = {};
        mma_m16n8k16(s, lo[u].x, hi[u].x, lo[u].y, hi[u].y, x[u][j].x, x[u][j].y);
        mma_m16n8k16(s, lo[u].z, hi[u].z, lo[u].w, hi[u].w, x[u][j].z, x[u][j].w);
        add_sums(acc[j], s);
      }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) red[warp][j][g + e / 2 * 8][2 * t + e % 2] = acc[j][e];
  __syncthreads();
  for (int o = tid; o < NT * 8 * OM_ROWS; o += OM_THREADS) {
    const int r = o % OM_ROWS, b = o / OM_ROWS;
    if (b >= B || n0 + r >= d) continue;
    float s = 0.f;
#pragma unroll
    for (int w2 = 0; w2 < OM_WARPS; ++w2) s += red[w2][b / 8][r][b % 8];
    Y[(size_t)b * d + n0 + r] = __float2half_rn(s + (bias ? __half2float(bias[n0 + r]) : 0.f));
  }
}

}  // namespace djv
