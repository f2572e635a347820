// rowdot: y[b, m] = act(w[idx[m], :] . x[b, :] + bias[idx[m]]) for a few rows of x on the CUDA cores, for fp16, bf16
// and fp32 weights. Bound by HBM: every row of w is read exactly once.
#pragma once
#include "dtype.cuh"

namespace djv {

// Gated unit with a clamp: the gate is cut from above, the linear part on both sides, and one is added to it.
__device__ __forceinline__ float clamped_glu(float gate, float up, float limit) {
  const float g = fminf(gate, limit);
  const float u = fminf(fmaxf(up, -limit), limit);
  return g * sigmoid_f(1.702f * g) * (u + 1.f);
}

__device__ __forceinline__ float silu_glu(float gate, float up) { return gate * sigmoid_f(gate) * up; }

// gated units: two rows of the matrix make one output
__host__ __device__ constexpr bool is_glu(int act) { return act == DJV_ACT_CLAMPED_GLU || act == DJV_ACT_SILU_GLU; }
template <int ACT>
__device__ __forceinline__ float apply_glu(float gate, float up, float p) {
  return ACT == DJV_ACT_CLAMPED_GLU ? clamped_glu(gate, up, p) : silu_glu(gate, up);
}

// activations that take a constant, next to those that do not
template <int ACT>
__device__ __forceinline__ float apply_act_param(float v, float p) {
  if (ACT == DJV_ACT_SOFTCAP) return p * tanhf(v / p);
  return apply_act<ACT>(v);
}

// -------------------------------------------------------------------------------------------
// rowdot. A block owns a contiguous range of rows, the rows / blocks of them give or take one (pair, for gated units), and
// has 8 / WPR groups of WPR warps. A pass gives every group ROWS rows, whose 16-byte chunks its 32*WPR lanes stride over
// with U chunks in flight per lane per row. x is read through L1 (it is tiny and reused by every group); weights bypass L1.
//
// The grid is all blocks that are resident at once. Handing out rows in rounds instead (a grid of up to 6 blocks per
// multiprocessor of which 4 fit) left a part of the blocks without work in the last round: us before / now, bf16, 1 row of x:
// 12352 x 4096 23.2 / 16.3 (0.95 of the copy rate), 6144 x 4096 12.2 / 9.3, 22016 x 4096 gated 32.9 / 29.1, 50272 x 4096 66.0 / 58.3,
// 11264 x 2048 gated 8.9 / 9.1; 2 rows: 22016 x 4096 34.5 / 29.9, 4096 x 4096 8.3 / 8.1; fp16 gathered: 4096 x 12288 18.5 / 17.4 and
// with 2 rows 19.2 / 18.8. (Runs of different days differ by up to 5 %.) Short lists are bound by the chain launch, row numbers, x
// and first weights, sums, store: 2048 x 2048 2.8 / 2.9; gathered 384 x 768 2.5 / 2.7, 512 x 12288 with 2 rows 5.6 / 5.4.
// -------------------------------------------------------------------------------------------
constexpr int RD_THREADS = 256;
constexpr int RD_WARPS = RD_THREADS / WARP;
constexpr int RD_SPAN = 128;  // rows whose sums a block keeps before it finishes them
constexpr int RD_FEW = 8;     // as many as a block with 4 chunks per row can have

// What a block asks for before it waits for the kernel before it. Dense steps of one user are a chain of products and small kernels
// between them, under which HBM would be idle: RD_AHEAD bytes per block, twice as many where that is an eighth of its rows, by bulk
// prefetches (one thread an 8 KB piece). A decode step of 6 layers, 4096 wide, one / two rows of x, us: nothing 562.6 / 620.6, 16 rows
// of 8 KB line by line 568.4 / 624.3, 8 KB in bulk 554.1 / 615.6, 16 KB 547.3 / 607.3, 32 KB 542.1 / 596.3; 12 layers, 2048 wide 472.3,
// 464.9, 458.7, 451.7, 460.6; with routed experts, 2048 wide 568.1, 576.5, 564.5, 563.6, 569.9, 4096 wide 640.0, 646.0, 630.8, 629.9,
// 636.2; this rule 543.6 / 597.2, 455.4, 566.1, 626.2. Lines are an instruction each, and with more bytes the loads of the kernel
// before queue up behind them. In the sparse steps, fp16, whose side streams fill the gaps, neither form gains: 16 steps of 8 layers,
// 4096 wide, nothing 8058, line by line 8073, a bulk prefetch per row 8045; 4 layers 9216 wide 13528, 13565, 13550, in runs that differ
// by 0.1 to 0.4 %. Those keep the lines.
constexpr int RD_AHEAD = 16384;
template <typename T>
constexpr bool is_half = false;
template <>
constexpr bool is_half<__half> = true;

// Blocks per multiprocessor that the registers of a pass leave room for: ROWS * U 16-byte loads, ROWS * B sums.
__host__ __device__ constexpr int rd_blocks(int B) { return B == 1 ? 4 : B == 2 ? 3 : B <= 4 ? 2 : 1; }

template <typename T, typename TO, int B, int ACT, int WPR, int ROWS, int U, int BLOCKS, int SPAN>
__global__ void __launch_bounds__(RD_THREADS, BLOCKS)
rowdot_kernel(TO *__restrict__ Y, const T *__restrict__ W, const T *__restrict__ X,
              const void *__restrict__ idx, const T *__restrict__ bias, int M, int N,
              long long ldw, int idx64, int ahead, float act_param, int per_block, int rest) {
  constexpr int UNIT = is_glu(ACT) ? 2 : 1;  // rows 2i, 2i + 1 of the matrix are the gate and up rows of output i
  constexpr int GROUPS = RD_WARPS / WPR;
  constexpr int GLANES = WARP * WPR;
  __shared__ float red[B][SPAN][WPR];

  const int tid = threadIdx.x;
  const int warp = tid / WARP, lane = tid % WARP;
  const int group = warp / WPR, wig = warp % WPR;
  const int glane = wig * WARP + lane;
  const int nchunks = N / Chunk<T>::N;
  const uint4 *Xv = reinterpret_cast<const uint4 *>(X);
  const int units = M / UNIT;
  const int bx = blockIdx.x;
  const int first = (bx * per_block + min(bx, rest)) * UNIT;  // the first `rest` blocks have one more
  const int last = first + (per_block + (bx < rest ? 1 : 0)) * UNIT;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if constexpr (!is_half<T>) {
    // Weights are not produced by any kernel of a step, and a prefetch could not return a stale value anyway.
    const int row_bytes = nchunks * 16, pieces = ahead_pieces(row_bytes);
    const int total = (int)min((long long)(last - first) * pieces, max(1ll, (long long)ahead * pieces / row_bytes));
    for (int p = tid; p < total; p += RD_THREADS) {
      const AheadSpan s = ahead_piece(p, row_bytes);
      bulk_prefetch_l2(reinterpret_cast<const char *>(W + (first + s.row) * ldw) + s.offset, s.bytes);
    }
  } else if (ahead) {
    // 8 KB of each of 16 rows, line by line: of rows that are below `ahead`. A list that its maker is still writing (an event between
    // them may have become a programmatic edge of a graph) can hold anything. What it holds is only asked for, but asking for what no
    // page backs holds up the memory of the whole device: 16 steps of 2 layers, 4096 wide, two sequences, 7839 us, with the bound 4469.
    constexpr int LINES = 64, MAX_ROWS = 16;
    const int row_lines = (int)min((long long)LINES, ((long long)N * (int)sizeof(T) + 127) / 128);
    for (int m = first + warp; m < min(last, first + MAX_ROWS); m += RD_WARPS) {
      const long long r = load_index(idx, m, idx64);
      if (!ahead_takes(r, ahead)) continue;
      const char *w0 = reinterpret_cast<const char *>(W + r * ldw);
      for (int l = lane; l < row_lines; l += WARP) prefetch_l2(w0 + (size_t)l * 128);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // The bias of the output that this thread finishes first: its row number is asked for together with those of the first pass,
  // and it is on its way, unread, while that pass makes the products. (A thread without a row in that pass loads it at the end.)
  constexpr int SO = SPAN / UNIT;  // outputs of a span, for every row of x
  const int m_first = first + group * ROWS, m_bias = first + tid % SO;
  long long bias_row = -1;
  if (UNIT == 1 && bias != nullptr && m_first < last && m_bias < last && tid < SO * B) bias_row = load_index(idx, m_bias, idx64);
  T bias0 = T(0.f);

  for (int s0 = first; s0 < last; s0 += SPAN) {  // (the same trips for all threads of the block)
    const int s1 = min(last, s0 + SPAN);
    for (int m0 = s0 + group * ROWS; m0 < s1; m0 += GROUPS * ROWS) {
      const uint4 *wp[ROWS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        const long long r = m0 + j < s1 ? load_index(idx, m0 + j, idx64) : -1;
        wp[j] = r < 0 ? nullptr : reinterpret_cast<const uint4 *>(W + r * ldw);
      }
      if (UNIT == 1 && m0 == m_first && bias_row >= 0) bias0 = bias[bias_row];
      float acc[ROWS][B];
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
#pragma unroll
        for (int b = 0; b < B; ++b) acc[j][b] = 0.f;
      for (int c0 = glane; c0 < nchunks; c0 += GLANES * U) {
        uint4 wv[ROWS][U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + u * GLANES;
#pragma unroll
          for (int j = 0; j < ROWS; ++j)
            wv[j][u] = (c < nchunks && wp[j] != nullptr) ? ld_stream16(wp[j] + c) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + u * GLANES;
          if (c < nchunks) {
#pragma unroll
            for (int b = 0; b < B; ++b) {
              const uint4 xv = ld_cached16(Xv + (size_t)b * nchunks + c);
#pragma unroll
              for (int j = 0; j < ROWS; ++j) acc[j][b] = dot_chunk<T>(wv[j][u], xv, acc[j][b]);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const float v = warp_sum(acc[j][b]);
          if (lane == 0 && m0 + j < s1) red[b][m0 + j - s0][wig] = v;
        }
    }
    __syncthreads();
    const int outs = (s1 - s0) / UNIT;
    for (int o = tid; o < SO * B; o += RD_THREADS) {
      const int b = o / SO, i = o % SO;
      if (i >= outs) continue;
      float v[UNIT];
#pragma unroll
      for (int j = 0; j < UNIT; ++j) {
        const int row = i * UNIT + j;
        v[j] = 0.f;
#pragma unroll
        for (int w2 = 0; w2 < WPR; ++w2) v[j] += red[b][row][w2];
        if (UNIT == 1 && bias != nullptr)
          v[j] += to_f(s0 == first && o == tid && bias_row >= 0 ? bias0 : bias[load_index(idx, s0 + row, idx64)]);
      }
      const size_t at = (size_t)b * units + s0 / UNIT + i;
      if constexpr (is_glu(ACT)) Y[at] = from_f<TO>(apply_glu<ACT>(v[0], v[1], act_param));
      else Y[at] = from_f<TO>(apply_act_param<ACT>(v[0], act_param));
    }
    if (s1 < last) __syncthreads();  // red[] is reused by the next span
  }
}

// What a lane has under way of a pass: 4 rows x 2 chunks; 2 rows x 4 chunks where a block has few rows (RD_FEW_ROWS); for two rows
// of x also those with a block more per multiprocessor (RD_FOUR_BLOCKS).
enum RowdotForm { RD_FOUR_ROWS, RD_FEW_ROWS, RD_FOUR_BLOCKS };

struct RowdotPlan {
  int wpr, grid, per_block, rest, ahead;
  RowdotForm form;
};

// A block with p rows makes ceil(p / (groups * rows)) passes of ceil(nchunks / (32 * wpr * chunks)) trips of the chunk loop, and a
// pass costs about one trip on top (row pointers, sums of the warps, a block barrier at the end). The least is within 3 % of the
// best at every shape above; of equals the one with fewer lanes per row has more rows under way, but a block that is done after
// one pass of few rows wants all its warps in it.
inline long long rowdot_cost(int p, int nchunks, int rows, int &wpr) {
  static const int k_wpr = env_int("DJV_RD_WPR", 0);  // development knob
  long long best = -1;
  for (int w = 1; w <= 8; w *= 2) {
    const int at_once = RD_WARPS / w * rows;
    const long long cost = (long long)ceil_div(p, at_once) * (ceil_div(nchunks, WARP * w * (8 / rows)) + 1);
    if (best < 0 || cost < best || (rows == 2 && cost == best && p <= at_once && nchunks >= WARP * w)) {
      best = cost;
      wpr = w;
    }
  }
  if (k_wpr > 0) wpr = k_wpr;
  return best;
}

// Few rows: 2 per block, or up to 5 short ones with several rows of x. us, 4 x 2 / 2 x 4: two rows of x 512 x 12288 7.1 / 5.8,
// 512 x 9216 6.3 / 5.5, 2048 x 1024 2.5 / 2.4; three 512 x 12288 6.6 / 5.8, 512 x 4096 3.9 / 3.4; but 1024 x 12288 7.8 / 8.3 (two),
// 7.8 / 8.7 (three). A block more for two rows of x where that saves a tenth of the trips on a multiprocessor: 4096 x 4096
// 9.3 / 8.2, 4096 x 12288 21.9 / 19.6; but 12352 x 4096 17.9 / 21.3, 6144 x 4096 10.3 / 11.2.
inline RowdotPlan plan_rowdot(int M, int nchunks, int unit, int B) {
  const int units = M / unit;
  int slots = sm_count() * rd_blocks(B), p = ceil_div(units, slots) * unit;
  RowdotPlan r{};
  r.form = B <= 4 && (p <= 2 || (B > 1 && p <= 5 && nchunks <= 256)) ? RD_FEW_ROWS : RD_FOUR_ROWS;
  const int q = r.form == RD_FEW_ROWS ? max(2, p) : p;
  const long long cost = rowdot_cost(q, nchunks, r.form == RD_FEW_ROWS ? 2 : 4, r.wpr);
  if (B == 2 && r.form == RD_FOUR_ROWS) {
    const int more = sm_count() * 4;
    int wpr;
    if (rowdot_cost(ceil_div(units, more) * unit, nchunks, 2, wpr) * 4 * 10 <= cost * 3 * 9) {
      r.form = RD_FOUR_BLOCKS;
      r.wpr = wpr;
      slots = more;
    }
  }
  r.grid = max(1, min(slots, r.form == RD_FEW_ROWS ? ceil_div(M, q) : units));
  r.per_block = units / r.grid;
  r.rest = units % r.grid;
  r.ahead = (int)max((long long)RD_AHEAD, min(2ll * RD_AHEAD, (long long)r.per_block * unit * nchunks * 16 / 8));
  return r;
}

// launch(WPR, ROWS, U, BLOCKS, SPAN) with compile-time arguments
#define DJV_ROWDOT_WPR(plan, ROWS_, U_, BLOCKS_, SPAN_, LAUNCH)       \
  do {                                                                \
    switch ((plan).wpr) {                                             \
      case 1: LAUNCH(1, ROWS_, U_, BLOCKS_, SPAN_); break;            \
      case 2: LAUNCH(2, ROWS_, U_, BLOCKS_, SPAN_); break;            \
      case 4: LAUNCH(4, ROWS_, U_, BLOCKS_, SPAN_); break;            \
      default: LAUNCH(8, ROWS_, U_, BLOCKS_, SPAN_); break;           \
    }                                                                 \
  } while (0)
#define DJV_ROWDOT(plan, B_, LAUNCH)                                                  \
  do {                                                                                \
    if constexpr ((B_) <= 4) {                                                        \
      if ((plan).form == RD_FEW_ROWS) {                                               \
        DJV_ROWDOT_WPR(plan, 2, 4, rd_blocks(B_), RD_FEW, LAUNCH);                    \
        break;                                                                        \
      }                                                                               \
    }                                                                                 \
    if constexpr ((B_) == 2) {                                                        \
      if ((plan).form == RD_FOUR_BLOCKS) {                                            \
        DJV_ROWDOT_WPR(plan, 2, 4, 4, RD_SPAN, LAUNCH);                               \
        break;                                                                        \
      }                                                                               \
    }                                                                                 \
    DJV_ROWDOT_WPR(plan, 4, 2, rd_blocks(B_), RD_SPAN, LAUNCH);                       \
  } while (0)

}  // namespace djv
