// Products of a few rows of x with streamed weight rows on the tensor cores (mma.sync m16n8k16, 16-bit in, fp32
// accumulate): the engine of the products with up to 32 rows of x whose result elements belong to weight rows.
//
// A cluster of S blocks works through tiles of 32 weight rows; block s of it takes every S-th chunk of 128 columns. A
// stage of a block's ring is one chunk: 32 x 256 bytes of weights and 8 * NT x 256 bytes of activations, brought in by
// 16-byte asynchronous copies, 16 neighbouring lanes to a row, pieces swizzled for ldmatrix. Rows that a tile does not have
// are not copied: what is in their place meets no other row's sums, and copies of nothing took as long as copies (22016 x
// 4096, 8 rows of x: 36 us with them, 29.5 without). The ring runs on from one tile to the next, so the sums of a tile are
// added up (over the 4 warps that split a chunk's columns, then over the cluster through distributed shared memory, in rank
// order) while the next tile's weights are on their way. Two blocks per multiprocessor, each with 72, 48, 40 or 24 KB of weights in
// flight for up to 8, 16, 24 and 32 rows of x: activations and sums take the rest.
//
// The tensor cores' sums are short: 16 columns with up to 8 rows of x, 32 with more, join the others in fp32 (add_sums). Kept in
// the MMAs' accumulators from end to end of a row they were off by 1.0e-6 of the result at 4096 columns and 2.9e-6 at 11008;
// now 1.2e-7 to 1.5e-7 and 1.8e-7. With PART, the sums of PART chunks join before they meet the rest (0.9e-7 and 1.0e-7):
// where the CUDA cores, 1.0e-7 and 1.4e-7, had the product before. Cost with 8 rows of x 0 to 2 %, with 32 up to 5 %, of PART
// another 0 to 4 %.
//
// Bound by HBM from about 20 MB of weights on: bf16, 8 rows of x, us before (a block of 8 warps per 16 rows, fed straight
// from registers) / now, of which the weights at copy rate: 6144 x 4096 15.1 / 10.3 (7.7), 12352 x 4096 28.9 / 18.6 (15.5),
// 22016 x 4096 34.6 / 29.3 (27.7), 50272 x 2048 41.3 / 33.6 (31.6); 16 rows, 4096 gathered rows of 12288 24.4 / 20.3 (15.5).
// Short lists are over before a ring has been worth filling: those of the products take another form (rowdot_mma.cuh).
//
// What the weights are, which x meets them and where results go is the Source's business:
//   seek(t, c)            the copies that follow are those of chunk c (of this block) of tile t; called in order
//   w(i, ok), x(i, ok)    this thread's i-th 16-byte piece of them, null where there is no such row (token); !ok: zeros. Piece
//                         i is row (token) tid / 16 + 16 * i, columns (tid % 16) * 8 .. of the chunk
//   begin(t)              the products of tile t start
//   store(t, pair, b, v)  sums of weight rows 2 * pair, 2 * pair + 1 of tile t with token b
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "mma.cuh"

namespace djv {

constexpr int WR_THREADS = 256, WR_WARPS = WR_THREADS / WARP;
constexpr int WR_ROWS = 32;                     // weight rows of a tile, or fewer
constexpr int WR_K = 128;                       // columns of a chunk
constexpr int WR_BPS = 2;                       // blocks per multiprocessor
constexpr int WR_PPR = WR_K / 8, WR_RP = WR_THREADS / WR_PPR;  // 16-byte pieces of a row; rows that the block copies at once
constexpr int WR_KW = WR_WARPS / (WR_ROWS / 16);  // warps that share 16 rows, each with a quarter of a chunk's columns
constexpr int WR_WP = WR_ROWS / WR_RP;           // 16-byte pieces of weights per thread and chunk
constexpr int WR_MAX_S = 8;

template <int NT>
struct WeightRing {
  static constexpr int XP = ceil_div_dev(NT * 8, WR_RP);  // 16-byte pieces of x per thread and chunk
  static constexpr int W_BYTES = WR_ROWS * WR_K * 2, STAGE = W_BYTES + NT * 8 * WR_K * 2;
  static constexpr int PITCH = WR_ROWS + 4;                     // floats between the tokens of a sum
  static constexpr int RED = WR_KW * NT * 8 * PITCH;            // floats of one tile's sums
  static constexpr int STAGES = (226 * 1024 / WR_BPS - 1024 - 2 * RED * 4) / STAGE;
  static constexpr int BYTES = STAGES * STAGE + 2 * RED * 4;    // (two sets: a block may be a tile ahead of its cluster)
  static_assert(STAGES >= 3, "");
};

template <typename T, int NT, int PART = 0, class Source>
__device__ __forceinline__ void weight_ring(Source &src, int tiles, int chunks, int tokens, unsigned char *smem) {
  using R = WeightRing<NT>;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP;
  const int mt = warp / WR_KW, kw = warp % WR_KW;
  const int r0 = tid / WR_PPR, ch = tid % WR_PPR;
  const uint32_t base = smem_addr(smem), piece = (uint32_t)(r0 * WR_K * 2 + ((ch ^ (r0 & 7)) << 4));  // (r0 + 8 swizzles alike)
  float *red = reinterpret_cast<float *>(smem + R::STAGES * R::STAGE);
  int to = 0, tt = 0, tc = 0;  // stage, tile and chunk of the next copies
  auto issue = [&]() {
    if (tt < tiles && chunks > 0) {
      src.seek(tt, tc);
      const uint32_t dst = base + (uint32_t)to * R::STAGE + piece;
#pragma unroll
      for (int i = 0; i < WR_WP; ++i) {
        bool ok = true;
        const void *p = src.w(i, ok);
        if (p) cp_async16_zfill(dst + i * WR_RP * WR_K * 2, p, ok ? 16 : 0);
      }
#pragma unroll
      for (int i = 0; i < R::XP; ++i)
        if (r0 + WR_RP * i < NT * 8) {
          bool ok = true;
          const void *p = src.x(i, ok);
          if (p) cp_async16_zfill(dst + R::W_BYTES + i * WR_RP * WR_K * 2, p, ok ? 16 : 0);
        }
      if (++tc == chunks) {
        tc = 0;
        ++tt;
      }
    }
    to = to + 1 == R::STAGES ? 0 : to + 1;
    cp_async_commit();
  };
#pragma unroll 1
  for (int i = 0; i < R::STAGES - 1; ++i) issue();
  const int ar = mt * 16 + (lane & 15), ac = WR_PPR / WR_KW * kw + (lane >> 4);
  const int br = lane & 7, bc = WR_PPR / WR_KW * kw + (lane >> 3);
  const uint32_t a_off = (uint32_t)ar * WR_K * 2, b_off = R::W_BYTES + (uint32_t)br * WR_K * 2;
  int from = 0;
  auto chunk = [&](float (&acc)[NT][4]) {  // the next one's products
    cp_async_wait<R::STAGES - 2>();
    __syncthreads();  // everybody's copies of this stage have landed, and the stage before has been read
    issue();
    const uint32_t st = base + (uint32_t)from * R::STAGE;
    from = from + 1 == R::STAGES ? 0 : from + 1;
#pragma unroll
    for (int p = 0; p < WR_PPR / WR_KW; p += 4) {  // two steps of 16 columns
      uint32_t a0[4], a1[4];
      ldmatrix_x4(a0, st + a_off + (((ac + p) ^ (ar & 7)) << 4));
      ldmatrix_x4(a1, st + a_off + (((ac + p + 2) ^ (ar & 7)) << 4));
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        uint32_t b[4];
        ldmatrix_x4(b, st + b_off + j * 8 * WR_K * 2 + (((bc + p) ^ br) << 4));
        float s[4] = {};
        mma_m16n8k16_t<T>(s, a0[0], a0[1], a0[2], a0[3], b[0], b[1]);
        if (NT == 1) {
          add_sums(acc[j], s);
          s[0] = s[1] = s[2] = s[3] = 0.f;
        }
        mma_m16n8k16_t<T>(s, a1[0], a1[1], a1[2], a1[3], b[2], b[3]);
        add_sums(acc[j], s);
      }
    }
  };
  for (int t = 0; t < tiles; ++t) {
    src.begin(t);
    float acc[NT][4] = {};
    if constexpr (PART == 0) {
      for (int c = 0; c < chunks; ++c) chunk(acc);
    } else {
      for (int c = 0; c < chunks;) {
        float part[NT][4] = {};
#pragma unroll 1
        for (const int stop = min(c + PART, chunks); c < stop; ++c) chunk(part);
#pragma unroll
        for (int j = 0; j < NT; ++j) add_sums(acc[j], part[j]);
      }
    }
    float *mine = red + (t & 1) * R::RED;
    const int g = lane / 4, q = lane % 4;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        mine[(kw * NT * 8 + j * 8 + 2 * q + e % 2) * R::PITCH + mt * 16 + g + e / 2 * 8] = acc[j][e];
    __syncthreads();
    const int pairs = WR_ROWS / 2 / S;  // row pairs that this block finishes
    auto sums_of_warps = [&](int pair, int b) {
      float *at = mine + b * R::PITCH + 2 * pair;
      float2 v = *reinterpret_cast<const float2 *>(at);
#pragma unroll
      for (int k = 1; k < WR_KW; ++k) {
        const float2 p = *reinterpret_cast<const float2 *>(at + k * NT * 8 * R::PITCH);
        v.x += p.x;
        v.y += p.y;
      }
      return v;
    };
    if (S > 1) {
      for (int o = tid; o < WR_ROWS / 2 * tokens; o += WR_THREADS) {
        const int pair = o % (WR_ROWS / 2), b = o / (WR_ROWS / 2);
        *reinterpret_cast<float2 *>(mine + b * R::PITCH + 2 * pair) = sums_of_warps(pair, b);
      }
      cluster.sync();
    }
    for (int o = tid; o < pairs * tokens; o += WR_THREADS) {
      const int pair = rank * pairs + o % pairs, b = o / pairs;
      float2 v;
      if (S > 1) {
        v = make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < WR_MAX_S; ++s)
          if (s < S) {
            const float2 p = *reinterpret_cast<const float2 *>(cluster.map_shared_rank(mine, s) + b * R::PITCH + 2 * pair);
            v.x += p.x;
            v.y += p.y;
          }
      } else {
        v = sums_of_warps(pair, b);
      }
      src.store(t, pair, b, v);
    }
  }
  cp_async_wait<0>();
  if (S > 1) cluster.sync();  // no block leaves while another may still read its sums
}

// How `units` (rows, or pairs of rows that stay together) are dealt out: `clusters` clusters of S blocks, `per` units each,
// one more in the first `rest` ones.
struct RingPlan {
  int S, clusters, per, rest;
};

// The clusters that are resident at once (`resident[i]` of them of 2^i blocks) share the rows evenly. A tile costs its chunks,
// a chunk by its rows but not less than 20 of them, and about 3 chunks' time for sums and cluster barriers, 1 without a
// cluster.
inline RingPlan ring_plan(int units, int unit_rows, int chunks, const int (&resident)[4]) {
  RingPlan p{};
  long long least = -1;
  for (int i = 0, S = 1; S <= WR_MAX_S && S <= chunks; ++i, S *= 2) {
    if (resident[i] < 1) continue;
    const int clusters = max(1, min(resident[i], ceil_div(units * unit_rows, 16)));
    const int rows = ceil_div(units, clusters) * unit_rows, tiles = ceil_div(rows, WR_ROWS);
    const long long c = ceil_div(chunks, S), sums = (S > 1 ? 3 : 1) * 32;
    const long long cost = tiles * (c * max(ceil_div(rows, tiles), 20) + sums);
    if (least < 0 || cost < least) {
      least = cost;
      p = {S, clusters, units / clusters, units % clusters};
    }
  }
  return p;
}

// `more`: shared memory behind the ring
template <int NT, typename... P>
inline cudaError_t ring_residency(void (*kernel)(P...), int (&resident)[4], int more = 0) {
  return cluster_residency(kernel, WR_THREADS, WeightRing<NT>::BYTES + more, WR_BPS, resident);
}

}  // namespace djv
