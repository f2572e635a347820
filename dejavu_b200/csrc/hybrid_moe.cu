// Routed feed-forward: every token goes through the `top` experts with the largest router scores sigmoid(z); an expert is a
// gated unit whose input is the token's activation times its score.
//
// A prompt portion is sorted by expert on the device (no host synchronisation) and runs as grouped matrix products: this
// file has the sorting and a CUDA-core form of the product for any size, hybrid_moe_gemm.cu the tensor-core form. A decode
// step runs two kernels on the chosen experts' weights; a shared expert, which every token uses, runs in the same two.
#include <cooperative_groups.h>

#include "../../include/dejavu_b200_routed.h"
#include "hybrid_moe.cuh"
#include "rowdot.cuh"
#include "weight_ring.cuh"

namespace djv {

constexpr int MAX_TOP = 16, MAX_EXPERTS = 1024;

// The `top` largest of z[0 .. E) by one warp, ties to the lower index. Lane k < top returns (index, value) of place k.
__device__ __forceinline__ void warp_topk(const float *z, int E, int top, int &index, float &value) {
  const int lane = threadIdx.x % WARP;
  float last = INFINITY;  // the choice before, and its index: what comes after it in the order (value down, index up)
  int last_i = -1;
  index = 0;
  value = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += WARP) {
      const float v = z[e];
      const bool open = v < last || (v == last && e > last_i);
      if (open && (v > best || at == 0x7fffffff)) {
        best = v;
        at = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, at, o);
      if (oi != 0x7fffffff && (at == 0x7fffffff || ov > best || (ov == best && oi < at))) {
        best = ov;
        at = oi;
      }
    }
    last = best;
    last_i = at;
    if (lane == k) {
      index = at < E ? at : 0;  // (a row that is not a number chooses something inside the range)
      value = best;
    }
  }
}

// ---- prompt portions: sorting ------------------------------------------------------------------------------------
constexpr int RT_WARPS = 8, RT_TOKENS = 16;

// choices of every token, and each choice's place among its expert's rows
__global__ void __launch_bounds__(RT_WARPS * WARP) moe_route_kernel(const float *__restrict__ z, int n, int E, int top,
                                                                    int *__restrict__ expert, int *__restrict__ place,
                                                                    float *__restrict__ weight, int *__restrict__ count) {
  extern __shared__ int sm[];
  int *cnt = sm, *base = cnt + E, *pick = base + E, *own = pick + RT_TOKENS * top;  // [E], [E], [tokens][top] x2
  pdl_prologue();
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP;
  const int t0 = blockIdx.x * RT_TOKENS, tn = min(RT_TOKENS, n - t0);
  for (int e = tid; e < E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int t = warp; t < tn; t += RT_WARPS) {
    int e;
    float v;
    warp_topk(z + (size_t)(t0 + t) * E, E, top, e, v);
    if (lane < top) {
      pick[t * top + lane] = e;
      own[t * top + lane] = atomicAdd(cnt + e, 1);
      weight[(size_t)(t0 + t) * top + lane] = sigmoid_f(v);
    }
  }
  __syncthreads();
  for (int e = tid; e < E; e += blockDim.x) base[e] = cnt[e] ? atomicAdd(count + e, cnt[e]) : 0;
  __syncthreads();
  for (int i = tid; i < tn * top; i += blockDim.x) {
    expert[(size_t)t0 * top + i] = pick[i];
    place[(size_t)t0 * top + i] = base[pick[i]] + own[i];
  }
}

// rows in the order of their experts: copies of the activations, weights, and where each choice went (over `place`)
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) moe_scatter_kernel(T *__restrict__ xs, const T *__restrict__ x,
                                                          const int *__restrict__ expert, int *__restrict__ place,
                                                          const float *__restrict__ weight, float *__restrict__ ws,
                                                          const int *__restrict__ count, int *__restrict__ offsets, int n,
                                                          int E, int top, int D) {
  extern __shared__ int off[];  // E + 1
  pdl_prologue();
  const int tid = threadIdx.x, lane = tid % WARP;
  if (tid < WARP) {
    int run = 0;
    for (int e0 = 0; e0 < E; e0 += WARP) {
      const int c = e0 + lane < E ? count[e0 + lane] : 0;
      int s = c;
#pragma unroll
      for (int o = 1; o < WARP; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += up;
      }
      if (e0 + lane < E) off[e0 + lane] = run + s - c;
      run += __shfl_sync(0xffffffffu, s, WARP - 1);
    }
    if (lane == 0) off[E] = run;
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int e = tid; e <= E; e += blockDim.x) offsets[e] = off[e];
  const int step = gridDim.x * (blockDim.x / WARP);
  for (int i = blockIdx.x * (blockDim.x / WARP) + tid / WARP; i < n * top; i += step) {  // a warp per row
    const int to = off[expert[i]] + place[i];
    __syncwarp();  // everybody has read place[i]
    if (lane == 0) {
      place[i] = to;
      ws[to] = weight[i];
    }
    const T *src = x + (size_t)(i / top) * D;
    T *dst = xs + (size_t)to * D;
    if (VEC) {
      constexpr int U = 8;
      const int nch = D / Chunk<T>::N;
      for (int c0 = lane; c0 < nch; c0 += WARP * U) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (c0 + u * WARP < nch) v[u] = reinterpret_cast<const uint4 *>(src)[c0 + u * WARP];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (c0 + u * WARP < nch) reinterpret_cast<uint4 *>(dst)[c0 + u * WARP] = v[u];
      }
    } else {
      for (int c = lane; c < D; c += WARP) dst[c] = src[c];
    }
  }
}

// ---- prompt portions: grouped product on the CUDA cores ------------------------------------------------------------
constexpr int GG_M = 64, GG_N = 64, GG_K = 16, GG_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(GG_THREADS) moe_grouped_kernel(GroupedArgs a) {
  __shared__ float xs[GG_K][GG_M + 4], wsm[GG_K][GG_N + 4];
  __shared__ int found[4];
  pdl_prologue();
  const int tid = threadIdx.x;
  if (tid == 0) {
    int e, r0, r1;
    found[0] = grouped_tile(a.offsets, a.E, GG_M, blockIdx.y, e, r0, r1);
    found[1] = e;
    found[2] = r0;
    found[3] = r1;
  }
  __syncthreads();
  if (!found[0]) return;
  const int e = found[1], r0 = found[2], rows = min(GG_M, found[3] - r0), n0 = blockIdx.x * GG_N;
  const T *x = static_cast<const T *>(a.x) + (size_t)r0 * a.K;
  const T *w = static_cast<const T *>(a.w) + ((size_t)e * a.N + n0) * a.K;
  const int tm = tid / 16 * 4, tn = tid % 16 * 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < a.K; k0 += GG_K) {
    for (int i = tid; i < GG_M * GG_K; i += GG_THREADS) {
      const int r = i / GG_K, k = i % GG_K;
      xs[k][r] = r < rows && k0 + k < a.K ? to_f(x[(size_t)r * a.K + k0 + k]) : 0.f;
      wsm[k][r] = n0 + r < a.N && k0 + k < a.K ? to_f(w[(size_t)r * a.K + k0 + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GG_K; ++k) {
      float u[4], v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        u[i] = xs[k][tm + i];
        v[i] = wsm[k][tn + i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(u[i], v[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (tm + i >= rows) continue;
    const size_t r = (size_t)r0 + tm + i;
    const float s = a.scale ? a.scale[r] : 1.f;
    if (a.glu) {
#pragma unroll
      for (int j = 0; j < 4; j += 2)
        if (n0 + tn + j + 1 < a.N)
          static_cast<T *>(a.y)[r * (a.N / 2) + (n0 + tn + j) / 2] = from_f<T>(silu_glu(s * acc[i][j], s * acc[i][j + 1]));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n0 + tn + j < a.N) static_cast<T *>(a.y)[r * a.N + n0 + tn + j] = from_f<T>(s * acc[i][j]);
    }
  }
}

// ---- decode ----------------------------------------------------------------------------------------------------
struct MoeDecodeArgs {
  float *y;               // (B, D)
  void *act;              // (B, slots, ld_act): slot k < top is a token's k-th expert, slot top the shared one
  int *chosen;            // (B, top)
  const void *x;          // (B, D)
  const float *z;         // (B, E)
  const void *w_gu, *w_down;        // (E, 2F, D), (E, D, F)
  const void *shared_gu, *shared_down;  // (2F', D), (D, F'), or null
  const float *init;      // (B, D) added to y, or null
  int B, E, top, D, F, F_shared, ld_act;
};

constexpr int MO_THREADS = 256, MO_WARPS = MO_THREADS / WARP;

// dot products of R rows of w (stride ld) with x, N elements, by `lanes` lanes of which this is one: U 16-byte chunks per
// lane and row in flight
template <typename T, bool VEC, int R, int U>
__device__ __forceinline__ void warp_rows(const T *w, size_t ld, const T *x, int n, float (&acc)[R], int lane, int lanes) {
  if (VEC) {
    const int nch = n / Chunk<T>::N;
    for (int c0 = lane; c0 < nch; c0 += lanes * U) {
      uint4 v[R][U];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int c = c0 + u * lanes;
          v[r][u] = c < nch ? ld_stream16(reinterpret_cast<const uint4 *>(w + r * ld) + c) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + u * lanes;
        if (c < nch) {
          const uint4 xv = *(reinterpret_cast<const uint4 *>(x) + c);
#pragma unroll
          for (int r = 0; r < R; ++r) acc[r] = dot_chunk<T>(v[r][u], xv, acc[r]);
        }
      }
    }
  } else {
    for (int c = lane; c < n; c += lanes)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = fmaf(to_f(w[r * ld + c]), to_f(x[c]), acc[r]);
  }
}

// grid (B, tiles of outputs, slots): sequences that use the same weights run side by side
template <typename T, bool VEC>
__global__ void __launch_bounds__(MO_THREADS) moe_decode_up_kernel(MoeDecodeArgs a) {
  __shared__ int pick_s;
  __shared__ float weight_s;
  pdl_prologue();
  const int b = blockIdx.x, slot = blockIdx.z, lane = threadIdx.x % WARP, warp = threadIdx.x / WARP;
  const bool shared = slot == a.top;
  const int F = shared ? a.F_shared : a.F, o = blockIdx.y * MO_WARPS + warp;
  if ((int)blockIdx.y * MO_WARPS >= F) return;
  if (!shared) {
    if (warp == 0) {
      int e;
      float v;
      warp_topk(a.z + (size_t)b * a.E, a.E, slot + 1, e, v);
      if (lane == slot) {
        pick_s = e;
        weight_s = sigmoid_f(v);
        if (blockIdx.y == 0) a.chosen[b * a.top + slot] = e;
      }
    }
    __syncthreads();
  }
  if (o >= F) return;
  const float wt = shared ? 1.f : weight_s;
  const T *w = shared ? static_cast<const T *>(a.shared_gu) : static_cast<const T *>(a.w_gu) + (size_t)pick_s * 2 * a.F * a.D;
  float acc[2] = {0.f, 0.f};
  warp_rows<T, VEC, 2, 4>(w + (size_t)2 * o * a.D, a.D, static_cast<const T *>(a.x) + (size_t)b * a.D, a.D, acc, lane, WARP);
  acc[0] = warp_sum(acc[0]);
  acc[1] = warp_sum(acc[1]);
  if (lane == 0)
    static_cast<T *>(a.act)[((size_t)b * gridDim.z + slot) * a.ld_act + o] = from_f<T>(silu_glu(wt * acc[0], wt * acc[1]));
}

// WPR warps share a row of the result
template <typename T, bool VEC, int WPR>
__global__ void __launch_bounds__(MO_THREADS) moe_decode_down_kernel(MoeDecodeArgs a, int slots) {
  __shared__ float red[MO_WARPS];
  pdl_prologue();
  const int b = blockIdx.x, lane = threadIdx.x % WARP, warp = threadIdx.x / WARP;
  const int m = blockIdx.y * (MO_WARPS / WPR) + warp / WPR, part = warp % WPR;
  const T *act = static_cast<const T *>(a.act) + (size_t)b * slots * a.ld_act;
  float acc[1] = {0.f};
  if (m < a.D)
    for (int s = 0; s < slots; ++s) {
      const bool shared = s == a.top;
      const int F = shared ? a.F_shared : a.F;
      const T *w = shared ? static_cast<const T *>(a.shared_down) + (size_t)m * F
                          : static_cast<const T *>(a.w_down) + ((size_t)a.chosen[b * a.top + s] * a.D + m) * F;
      warp_rows<T, VEC, 1, 4>(w, 0, act + (size_t)s * a.ld_act, F, acc, part * WARP + lane, WPR * WARP);
    }
  float sum = warp_sum(acc[0]);
  if (WPR > 1) {
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    sum = 0.f;
#pragma unroll
    for (int x = 0; x < WPR; ++x) sum += red[warp / WPR * WPR + x];
  }
  if (lane == 0 && part == 0 && m < a.D) a.y[(size_t)b * a.D + m] = sum + (a.init ? a.init[(size_t)b * a.D + m] : 0.f);
}

// ---- decode, several rows: every weight row is read once -----------------------------------------------------------
// Streamed by weight_ring.cuh. The up stage goes through the gate and up rows of all experts that any sequence chose, one
// after another and the shared one last, dealt out evenly whatever expert they belong to; a sequence that did not choose the
// expert of a row does not store that row's product. The down stage adds all experts up in one accumulator: its columns are
// those of all experts in a row, and a sequence that did not choose an expert meets it with zeros.
// 8 sequences, 8 experts of 3648 x 4096 and the shared one, us: up 114 -> 87 (75 at copy rate), down 83 -> 51 (38). Before,
// a block took 16 rows and all columns, with no loads under way while it found its experts or added up. (Finding a chunk's
// expert by a division for every chunk cost the down stage 24 us.)
constexpr int MM_B = 32, MM_E = 1137;

// Who chose what, in the shared memory that two blocks per multiprocessor leave behind their rings: the experts in use in
// ascending order, a bit for every expert, and an expert's place among a sequence's choices, as a byte for every expert and sequence
// where there is room for that, else as the sequences' choices, which are looked through. (Bytes for 32 sequences whatever their
// number left room for one block from 57 experts on with 24 sequences, from 112 on with 8: 64 experts of 704 x 2048, 24 sequences,
// 171 us so, 101 now; 112 of 512 x 1024, 8 sequences, 52 and 26.)
template <int NT>
struct MoeTable {
  static constexpr int SEQS = NT * 8, BITS = (MM_E + 31) / 32 * 4, LIST = SEQS * MAX_TOP * 2, CHOICES = SEQS * MAX_TOP * 2;
  static constexpr int BYTES = 115344 - WeightRing<NT>::BYTES;  // (two blocks of 115344 bytes are resident, two of 115648 are not)
  static_assert(BYTES >= BITS + LIST + CHOICES, "");
  static bool has_places(int E) { return E * SEQS <= BYTES - BITS - LIST; }
};

template <int NT, bool PLACES>
struct MoeInUse {
  const signed char *places;  // [E][SEQS]
  const unsigned *choices;    // [B][pairs], two to a word
  const short *list;          // [n] experts in use
  int n, pairs;

  // the expert's place among the sequence's choices, or -1
  __device__ __forceinline__ int place(int e, int b) const {
    if (PLACES) return places[e * MoeTable<NT>::SEQS + b];
    int s = -1;
    for (int k = 0; k < pairs; ++k) {
      const unsigned two = choices[b * pairs + k];
      if ((two & 0xffffu) == (unsigned)e) s = 2 * k;
      if (two >> 16 == (unsigned)e) s = 2 * k + 1;
    }
    return s;
  }
};

// every block finds for itself
template <int NT, bool PLACES>
__device__ __forceinline__ MoeInUse<NT, PLACES> moe_in_use(const MoeDecodeArgs &a, unsigned char *table, int *n_s) {
  using Table = MoeTable<NT>;
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP, pairs = (a.top + 1) / 2, words = (a.E + 31) / 32;
  unsigned *bits = reinterpret_cast<unsigned *>(table);
  short *list = reinterpret_cast<short *>(table + Table::BITS);
  signed char *places = reinterpret_cast<signed char *>(table + Table::BITS + Table::LIST);
  unsigned short *choices = reinterpret_cast<unsigned short *>(places);
  for (int i = tid; i < words; i += WR_THREADS) bits[i] = 0u;
  if (PLACES)
    for (int i = tid; i < a.E * Table::SEQS / 4; i += WR_THREADS) reinterpret_cast<int *>(places)[i] = -1;
  __syncthreads();
  for (int b = warp; b < a.B; b += WR_WARPS) {
    int e;
    float v;
    warp_topk(a.z + (size_t)b * a.E, a.E, a.top, e, v);
    if (lane < a.top) atomicOr(bits + e / 32, 1u << e % 32);
    if (PLACES) {
      if (lane < a.top) places[e * Table::SEQS + b] = (signed char)lane;
    } else if (lane < 2 * pairs) {
      choices[b * 2 * pairs + lane] = lane < a.top ? (unsigned short)e : (unsigned short)0xffff;
    }
  }
  __syncthreads();
  if (warp == 0) {
    int n = 0;
    for (int w0 = 0; w0 < words; w0 += WARP) {
      unsigned m = w0 + lane < words ? bits[w0 + lane] : 0u;
      int at = __popc(m);  // experts of this lane and those before it
#pragma unroll
      for (int o = 1; o < WARP; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += up;
      }
      const int all = __shfl_sync(0xffffffffu, at, WARP - 1);
      at += n - __popc(m);
      for (; m; m &= m - 1) list[at++] = (short)((w0 + lane) * 32 + __ffs(m) - 1);
      n += all;
    }
    if (lane == 0) *n_s = n;
  }
  __syncthreads();
  return {places, reinterpret_cast<const unsigned *>(choices), list, *n_s, pairs};
}

template <int NT, bool PLACES>
struct MoeUpSource {
  const MoeDecodeArgs &a;
  const MoeInUse<NT, PLACES> used;
  int slots, first, last, rows, S, rank;  // units (pairs of rows) of the cluster; weight rows of its tiles
  const bf16 *row[WR_WP];
  int k;

  // the expert of a unit (E: the shared one), and the unit's number in it
  __device__ __forceinline__ int expert(int &unit) const {
    const int at = min(unit / a.F, used.n);
    unit -= at * a.F;
    return at < used.n ? used.list[at] : a.E;
  }
  __device__ __forceinline__ void seek(int t, int c) {
    if (c == 0)
#pragma unroll
      for (int i = 0; i < WR_WP; ++i) {
        const int r = (int)threadIdx.x / WR_PPR + WR_RP * i;
        int unit = first + (t * rows + r) / 2;
        const bool ok = r < rows && unit < last;
        row[i] = nullptr;
        if (ok) {
          const int e = expert(unit);
          row[i] = (e == a.E ? static_cast<const bf16 *>(a.shared_gu) : static_cast<const bf16 *>(a.w_gu) + (size_t)e * 2 * a.F * a.D) +
                   (size_t)(2 * unit + r % 2) * a.D;
        }
      }
    k = (c * S + rank) * WR_K + (int)threadIdx.x % WR_PPR * 8;
  }
  __device__ __forceinline__ const void *w(int i, bool &ok) const {
    ok = k < a.D;
    return row[i] != nullptr ? row[i] + (ok ? k : 0) : nullptr;
  }
  __device__ __forceinline__ const void *x(int i, bool &ok) const {
    const int b = (int)threadIdx.x / WR_PPR + WR_RP * i;
    ok = k < a.D;
    return b < a.B ? static_cast<const bf16 *>(a.x) + (size_t)b * a.D + (ok ? k : 0) : nullptr;
  }
  __device__ __forceinline__ void begin(int) {}
  __device__ __forceinline__ void store(int t, int pair, int b, float2 v) const {
    int unit = first + t * rows / 2 + pair;
    if (2 * pair >= rows || unit >= last) return;
    const int e = expert(unit), s = e == a.E ? a.top : used.place(e, b);
    if (s < 0) return;
    const float wt = e == a.E ? 1.f : sigmoid_f(a.z[(size_t)b * a.E + e]);
    static_cast<bf16 *>(a.act)[((size_t)b * slots + s) * a.ld_act + unit] = from_f<bf16>(silu_glu(wt * v.x, wt * v.y));
  }
};

template <int NT, bool PLACES>
struct MoeDownSource {
  const MoeDecodeArgs &a;
  const MoeInUse<NT, PLACES> used;
  int slots, first, last, rows, S, rank;  // rows of the cluster, of its tiles
  // the chunk's number in its expert, the expert's chunks, row length and place in the list (used.n: the shared one), and of
  // the thread's pieces the rows of weights and of activations (xs: whether the sequence chose the expert)
  int j, kf, F, at, k;
  const bf16 *row[WR_WP], *act[(MM_B + WR_RP - 1) / WR_RP];
  bool xs[(MM_B + WR_RP - 1) / WR_RP];

  __device__ __forceinline__ void enter(int t) {
    const bool shared = at == used.n;
    const int e = shared ? a.E : used.list[at];
    F = shared ? a.F_shared : a.F;
    kf = ceil_div_dev(F, WR_K);
    const bf16 *base = shared ? static_cast<const bf16 *>(a.shared_down) : static_cast<const bf16 *>(a.w_down) + (size_t)e * a.D * a.F;
#pragma unroll
    for (int i = 0; i < WR_WP; ++i) {
      const int r = (int)threadIdx.x / WR_PPR + WR_RP * i, m = first + t * rows + r;
      row[i] = r < rows && m < last ? base + (size_t)m * F : nullptr;
    }
#pragma unroll
    for (int i = 0; i < (MM_B + WR_RP - 1) / WR_RP; ++i) {
      const int b = (int)threadIdx.x / WR_PPR + WR_RP * i;
      const int s = b >= a.B ? -1 : shared ? a.top : used.place(e, b);
      xs[i] = s >= 0;
      act[i] = b < a.B ? static_cast<const bf16 *>(a.act) + ((size_t)b * slots + max(s, 0)) * a.ld_act : nullptr;
    }
  }
  __device__ __forceinline__ void seek(int t, int c) {
    if (c == 0) {
      j = rank;
      at = 0;
      enter(t);
    } else {
      j += S;
    }
    while (j >= kf && at < used.n) {  // (the list ends with the shared expert, or with the last chunk)
      j -= kf;
      ++at;
      enter(t);
    }
    k = j * WR_K + (int)threadIdx.x % WR_PPR * 8;
  }
  __device__ __forceinline__ const void *w(int i, bool &ok) const {
    ok = k < F;
    return row[i] != nullptr ? row[i] + (ok ? k : 0) : nullptr;
  }
  __device__ __forceinline__ const void *x(int i, bool &ok) const {
    ok = k < F && xs[i];
    return act[i] != nullptr ? act[i] + (ok ? k : 0) : nullptr;
  }
  __device__ __forceinline__ void begin(int) {}
  __device__ __forceinline__ void store(int t, int pair, int b, float2 v) const {
    const int at = first + t * rows + 2 * pair;
    if (2 * pair >= rows) return;
    const size_t o = (size_t)b * a.D + at;
    if (at < last) a.y[o] = v.x + (a.init ? a.init[o] : 0.f);
    if (at + 1 < last) a.y[o + 1] = v.y + (a.init ? a.init[o + 1] : 0.f);
  }
};

template <int NT, bool UP, bool PLACES>
__global__ void __launch_bounds__(WR_THREADS, WR_BPS) moe_ring_kernel(MoeDecodeArgs a, int slots) {
  extern __shared__ __align__(128) unsigned char wr_smem[];
  __shared__ int n_s;
  pdl_prologue();
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), cl = blockIdx.x / S, clusters = gridDim.x / S;
  const MoeInUse<NT, PLACES> used = moe_in_use<NT, PLACES>(a, wr_smem + WeightRing<NT>::BYTES, &n_s);
  const int n = used.n;
  const bool shared = a.shared_gu != nullptr;
  const int units = UP ? n * a.F + (shared ? a.F_shared : 0) : a.D, per = units / clusters, rest = units % clusters;
  const int first = cl * per + min(cl, rest), last = first + per + (cl < rest ? 1 : 0), rows_all = (last - first) * (UP ? 2 : 1);
  const int tiles = ceil_div_dev(rows_all, WR_ROWS), rows = tiles ? ceil_div_dev(ceil_div_dev(rows_all, tiles), 2) * 2 : 0;
  const int all = UP ? ceil_div_dev(a.D, WR_K) : n * ceil_div_dev(a.F, WR_K) + (shared ? ceil_div_dev(a.F_shared, WR_K) : 0);
  const int chunks = rank < all ? (all - rank + S - 1) / S : 0;
  if constexpr (UP) {
    MoeUpSource<NT, PLACES> src{a, used, slots, first, last, rows, S, rank};
    weight_ring<bf16, NT>(src, tiles, chunks, a.B, wr_smem);
  } else {
    MoeDownSource<NT, PLACES> src{a, used, slots, first, last, rows, S, rank};
    weight_ring<bf16, NT>(src, tiles, chunks, a.B, wr_smem);
  }
}

template <int NT, bool UP, bool PLACES>
static int launch_ring(const MoeDecodeArgs &a, int slots, cudaStream_t st) {
  static DevicePrep prep;
  const int (*resident)[4];
  const cudaError_t prepared = prep.get([](int (&r)[4]) { return ring_residency<NT>(moe_ring_kernel<NT, UP, PLACES>, r, MoeTable<NT>::BYTES); },
                                        resident);
  if (prepared != cudaSuccess) {
    set_error("moe_decode: %s", cudaGetErrorString(prepared));
    return DJV_ERR_CUDA;
  }
  // (which experts are in use is known on the device only: as many as there can be)
  const int n = a.E < a.B * a.top ? a.E : a.B * a.top, kf = ceil_div(a.F, WR_K), kf_shared = ceil_div(a.F_shared, WR_K);
  const RingPlan p = UP ? ring_plan(n * a.F + a.F_shared, 2, ceil_div(a.D, WR_K), *resident)
                        : ring_plan(a.D, 1, n * kf + kf_shared, *resident);
  djv::launch_kernel_cluster(moe_ring_kernel<NT, UP, PLACES>, dim3(p.clusters * p.S), dim3(WR_THREADS),
                             (size_t)(WeightRing<NT>::BYTES + MoeTable<NT>::BYTES), st, dim3(p.S), a, slots);
  count_launch();
  return DJV_OK;
}

template <int NT>
static int launch_mma(const MoeDecodeArgs &a, int slots, bool up, bool down, cudaStream_t st) {
  const bool places = MoeTable<NT>::has_places(a.E);
  const int rc = !up ? DJV_OK : places ? launch_ring<NT, true, true>(a, slots, st) : launch_ring<NT, true, false>(a, slots, st);
  if (rc || !down) return rc;
  return places ? launch_ring<NT, false, true>(a, slots, st) : launch_ring<NT, false, false>(a, slots, st);
}

// ---- decode, one row --------------------------------------------------------------------------------------------------
// The chosen experts' rows and the shared one's are dealt out evenly over the resident blocks, as the dense products' are
// (rowdot.cuh): a block per 8 outputs and expert, and 8 rows of the result per block, left a last round nearly empty, and a lane walked
// the experts one after another. Every block has a part of the shared expert, which it begins with: its rows are known while
// the router is still running, and are asked for ahead. Bound by HBM from about 50 MB on, below by the chain router scores, choices,
// weights, sums. A decode step, us before / now: 12 layers 2048 wide, 8 experts of 1856 and a shared one 566 / 540 (up 10.3 / 9.5
// of 7.0 at copy rate, down 9.5 / 5.8 of 3.5), 6 layers 4096 wide, experts of 3648 626 / 597.
constexpr int M1_SPAN = 64;  // outputs whose sums a block keeps before it finishes them

template <typename T, int WPR>
__global__ void __launch_bounds__(MO_THREADS, 4) moe_one_up_kernel(MoeDecodeArgs a) {
  constexpr int GROUPS = MO_WARPS / WPR, GLANES = WARP * WPR, U = 2, AT_ONCE = GROUPS * 2;
  static_assert(M1_SPAN % AT_ONCE == 0, "");
  __shared__ float red[M1_SPAN][2][WPR], weight_s[M1_SPAN];
  __shared__ T *out_s[M1_SPAN];
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP, group = warp / WPR, wig = warp % WPR, glane = wig * WARP + lane;
  const int nch = a.D / Chunk<T>::N, grid = gridDim.x, bx = blockIdx.x;
  auto part = [&](int n, int at, int &first, int &count) {  // of n outputs
    const int per = n / grid, rest = n % grid;
    first = at * per + min(at, rest);
    count = per + (at < rest ? 1 : 0);
  };
  int fs, ns, fe, ne;
  part(a.F_shared, bx, fs, ns);
  part(a.top * a.F, grid - 1 - bx, fe, ne);  // (those with one more are others than above)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int row_bytes = nch * 16, rows_ahead = min(2 * ns, max(1, RD_AHEAD / row_bytes));
  for (int r = tid; r < rows_ahead; r += MO_THREADS)
    for (int off = 0; off < row_bytes; off += AHEAD_PIECE)
      bulk_prefetch_l2(reinterpret_cast<const char *>(static_cast<const T *>(a.shared_gu) + ((size_t)2 * fs + r) * a.D) + off,
                       min(AHEAD_PIECE, row_bytes - off));
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int e_l = 0;  // of place `lane`: the expert, and its score
  float v_l = 0.f;
  bool known = false;
  if (bx == 0 && warp == 0) {
    warp_topk(a.z, a.E, a.top, e_l, v_l);
    known = true;
    if (lane < a.top) a.chosen[lane] = e_l;
  }
  const uint4 *xv = static_cast<const uint4 *>(a.x);
  const int n = ns + ne;
  for (int s0 = 0; s0 < n; s0 += M1_SPAN) {
    const int s1 = min(n, s0 + M1_SPAN);
    for (int i0 = s0 + group * 2; i0 < s1; i0 += AT_ONCE) {
      const uint4 *wp[2] = {nullptr, nullptr};  // gate row; the up row is behind it
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = i0 + q;
        if (i >= s1) continue;
        const T *w;
        T *out = static_cast<T *>(a.act);
        float wt = 1.f;
        if (i < ns) {
          w = static_cast<const T *>(a.shared_gu) + (size_t)2 * (fs + i) * a.D;
          out += (size_t)a.top * a.ld_act + fs + i;
        } else {
          if (!known) {
            warp_topk(a.z, a.E, a.top, e_l, v_l);
            known = true;
          }
          const int u = fe + i - ns, s = u / a.F, o = u - s * a.F;
          wt = sigmoid_f(__shfl_sync(0xffffffffu, v_l, s));
          w = static_cast<const T *>(a.w_gu) + ((size_t)__shfl_sync(0xffffffffu, e_l, s) * a.F + o) * 2 * a.D;
          out += (size_t)s * a.ld_act + o;
        }
        wp[q] = reinterpret_cast<const uint4 *>(w);
        if (wig == 0 && lane == 0) {
          weight_s[i - s0] = wt;
          out_s[i - s0] = out;
        }
      }
      float acc[4] = {};
      for (int c0 = glane; c0 < nch; c0 += GLANES * U) {
        uint4 v[4][U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + u * GLANES;
#pragma unroll
          for (int r = 0; r < 4; ++r)
            v[r][u] = c < nch && wp[r / 2] != nullptr ? ld_stream16(wp[r / 2] + (r % 2) * nch + c) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + u * GLANES;
          if (c < nch) {
            const uint4 x = ld_cached16(xv + c);
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r] = dot_chunk<T>(v[r][u], x, acc[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float t = warp_sum(acc[r]);
        if (lane == 0 && i0 + r / 2 < s1) red[i0 + r / 2 - s0][r % 2][wig] = t;
      }
    }
    __syncthreads();
    if (tid < s1 - s0) {
      float g = 0.f, u = 0.f;
#pragma unroll
      for (int k = 0; k < WPR; ++k) {
        g += red[tid][0][k];
        u += red[tid][1][k];
      }
      *out_s[tid] = from_f<T>(silu_glu(weight_s[tid] * g, weight_s[tid] * u));
    }
    if (s1 < n) __syncthreads();
  }
}

template <typename T, int WPR>
__global__ void __launch_bounds__(MO_THREADS, 4) moe_one_down_kernel(MoeDecodeArgs a) {
  constexpr int GROUPS = MO_WARPS / WPR, GLANES = WARP * WPR, U = 2, AT_ONCE = GROUPS * 4, N = Chunk<T>::N;
  static_assert(M1_SPAN % AT_ONCE == 0, "");
  __shared__ float red[M1_SPAN][WPR];
  __shared__ const T *base_s[MAX_TOP];  // row 0 of a choice's weights
  const int tid = threadIdx.x, warp = tid / WARP, lane = tid % WARP, group = warp / WPR, wig = warp % WPR, glane = wig * WARP + lane;
  const int grid = gridDim.x, bx = blockIdx.x, per = a.D / grid, rest = a.D % grid;
  const int first = bx * per + min(bx, rest), last = first + per + (bx < rest ? 1 : 0);
  const int nf = a.F / N, nfs = a.F_shared / N, nch = nfs + a.top * nf;  // chunks of a row: the shared expert's, the choices'
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (nfs > 0) {
    const int row_bytes = nfs * 16, rows_ahead = min(last - first, max(1, RD_AHEAD / row_bytes));
    for (int r = tid; r < rows_ahead; r += MO_THREADS)
      for (int off = 0; off < row_bytes; off += AHEAD_PIECE)
        bulk_prefetch_l2(reinterpret_cast<const char *>(static_cast<const T *>(a.shared_down) + (size_t)(first + r) * a.F_shared) + off,
                         min(AHEAD_PIECE, row_bytes - off));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid < a.top) base_s[tid] = static_cast<const T *>(a.w_down) + (size_t)a.chosen[tid] * a.D * a.F;
  __syncthreads();
  for (int s0 = first; s0 < last; s0 += M1_SPAN) {
    const int s1 = min(last, s0 + M1_SPAN);
    for (int m0 = s0 + group * 4; m0 < s1; m0 += AT_ONCE) {
      float acc[4] = {};
      for (int c0 = glane; c0 < nch; c0 += GLANES * U) {
        uint4 v[4][U];
        const uint4 *xp[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = c0 + u * GLANES;
          const T *w = static_cast<const T *>(a.shared_down), *act = static_cast<const T *>(a.act);
          int F = a.F_shared, k = c;  // chunk k of its part of the row
          if (c < nfs) {
            act += (size_t)a.top * a.ld_act;
          } else if (c < nch) {
            const int s = (c - nfs) / nf;
            k = c - nfs - s * nf;
            F = a.F;
            w = base_s[s];
            act += (size_t)s * a.ld_act;
          }
          xp[u] = reinterpret_cast<const uint4 *>(act) + k;
          const T *row = w + (size_t)m0 * F + k * N;
#pragma unroll
          for (int r = 0; r < 4; ++r)
            v[r][u] = c < nch && m0 + r < s1 ? ld_stream16(row + (size_t)r * F) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (c0 + u * GLANES < nch) {
            const uint4 x = ld_cached16(xp[u]);
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r] = dot_chunk<T>(v[r][u], x, acc[r]);
          }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float t = warp_sum(acc[r]);
        if (lane == 0 && m0 + r < s1) red[m0 + r - s0][wig] = t;
      }
    }
    __syncthreads();
    if (tid < s1 - s0) {
      float y = 0.f;
#pragma unroll
      for (int k = 0; k < WPR; ++k) y += red[tid][k];
      a.y[s0 + tid] = y + (a.init ? a.init[s0 + tid] : 0.f);
    }
    if (s1 < last) __syncthreads();
  }
}

// As plan_rowdot: the lanes that share a row by passes x trips.
template <typename T>
static int launch_one(const MoeDecodeArgs &a, bool up, bool down, cudaStream_t st) {
  constexpr int N = Chunk<T>::N;
  const int resident = 4 * sm_count();
  int wpr = 1;
#define DJV_GO(KERNEL_, GRID_)                                                                                       \
  switch (wpr) {                                                                                                     \
    case 1: djv::launch_kernel(KERNEL_<T, 1>, dim3(GRID_), dim3(MO_THREADS), 0, st, a); break;                       \
    case 2: djv::launch_kernel(KERNEL_<T, 2>, dim3(GRID_), dim3(MO_THREADS), 0, st, a); break;                       \
    case 4: djv::launch_kernel(KERNEL_<T, 4>, dim3(GRID_), dim3(MO_THREADS), 0, st, a); break;                       \
    default: djv::launch_kernel(KERNEL_<T, 8>, dim3(GRID_), dim3(MO_THREADS), 0, st, a); break;               \
  }                                                                                                                  \
  count_launch();
  if (up) {
    const int units = a.top * a.F + a.F_shared, grid = min(resident, units);
    rowdot_cost(2 * ceil_div(units, grid), a.D / N, 4, wpr);
    DJV_GO(moe_one_up_kernel, grid)
  }
  if (down) {
    const int grid = min(resident, a.D);
    rowdot_cost(ceil_div(a.D, grid), a.F_shared / N + a.top * (a.F / N), 4, wpr);
    DJV_GO(moe_one_down_kernel, grid)
  }
#undef DJV_GO
  return check_launch("moe_decode");
}

template <typename T>
static int launch_decode(const MoeDecodeArgs &a, bool up, bool down, cudaStream_t st) {
  const int slots = a.top + (a.shared_gu ? 1 : 0), fmax = a.F > a.F_shared || !a.shared_gu ? a.F : a.F_shared;
  constexpr int N = Chunk<T>::N;
  const bool vec_up = a.D % N == 0 && aligned16(a.x) && aligned16(a.w_gu) && aligned16(a.shared_gu);
  const bool vec_down = a.F % N == 0 && (!a.shared_gu || a.F_shared % N == 0) && a.ld_act % N == 0 && aligned16(a.act) &&
                        aligned16(a.w_down) && aligned16(a.shared_down);
  if (a.B == 1 && vec_up && vec_down && (long long)a.top * a.F + a.F_shared <= (1 << 28)) return launch_one<T>(a, up, down, st);
  if constexpr (sizeof(T) == 2) {
    // several rows share weights (both stages take this form or neither: they agree on where a choice's activations are)
    if (a.B >= 2 && a.B <= MM_B && vec_up && vec_down && a.E <= MM_E) {
      int rc;
      switch ((a.B + 7) / 8) {
        case 1: rc = launch_mma<1>(a, slots, up, down, st); break;
        case 2: rc = launch_mma<2>(a, slots, up, down, st); break;
        case 3: rc = launch_mma<3>(a, slots, up, down, st); break;
        default: rc = launch_mma<4>(a, slots, up, down, st); break;
      }
      return rc ? rc : check_launch("moe_decode");
    }
  }
  if (up) {
    const dim3 grid(a.B, ceil_div(fmax, MO_WARPS), slots);
    if (vec_up) djv::launch_kernel(moe_decode_up_kernel<T, true>, grid, dim3(MO_THREADS), 0, st, a);
    else djv::launch_kernel(moe_decode_up_kernel<T, false>, grid, dim3(MO_THREADS), 0, st, a);
    count_launch();
  }
  if (down) {
    // as many warps per row as still lets every block be resident at once and gives each lane work
    int wpr = 1;
    while (wpr < 4 && (long long)a.B * a.D * wpr * 2 <= (long long)8 * MO_WARPS * sm_count() && a.F / N >= WARP * wpr * 2) wpr *= 2;
    const dim3 grid(a.B, ceil_div(a.D, MO_WARPS / wpr));
    if (!vec_down) djv::launch_kernel(moe_decode_down_kernel<T, false, 1>, dim3(a.B, ceil_div(a.D, MO_WARPS)), dim3(MO_THREADS), 0, st, a, slots);
    else if (wpr == 1) djv::launch_kernel(moe_decode_down_kernel<T, true, 1>, grid, dim3(MO_THREADS), 0, st, a, slots);
    else if (wpr == 2) djv::launch_kernel(moe_decode_down_kernel<T, true, 2>, grid, dim3(MO_THREADS), 0, st, a, slots);
    else djv::launch_kernel(moe_decode_down_kernel<T, true, 4>, grid, dim3(MO_THREADS), 0, st, a, slots);
    count_launch();
  }
  return check_launch("moe_decode");
}

}  // namespace djv

using namespace djv;

extern "C" int djv_moe_route(int dtype, void *xs, const void *x, const float *z, int *expert, int *place, float *weight,
                             float *ws, int *count, int *offsets, int n, int E, int top, int D, void *stream) {
  DJV_REQUIRE(dtype == DJV_DTYPE_BF16 || dtype == DJV_DTYPE_F32, "moe_route: dtype %d", dtype);
  DJV_REQUIRE(xs && x && z && expert && place && weight && ws && count && offsets, "moe_route: null pointer");
  DJV_REQUIRE(n >= 1 && E >= 1 && E <= MAX_EXPERTS && top >= 1 && top <= E && top <= MAX_TOP && D >= 1 &&
                  (long long)n * top < (1ll << 31),
              "moe_route: n=%d, %d of %d experts, D=%d", n, top, E, D);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(count, 0, (size_t)E * 4, st) != cudaSuccess) return check_launch("moe_route");
  djv::launch_kernel(moe_route_kernel, dim3(ceil_div(n, RT_TOKENS)), dim3(RT_WARPS * WARP),
                     4 * (size_t)(2 * E + 2 * RT_TOKENS * top), st, z, n, E, top, expert, place, weight, count);
  const size_t sm = 4 * (size_t)(E + 1);
  const int blocks = ceil_div(n * top, 8), most = 8 * sm_count(), grid = blocks < most ? blocks : most;
  const bool vec = D % (16 / (int)dtype_bytes(dtype)) == 0 && aligned16(x) && aligned16(xs);
#define DJV_GO(T_, V_)                                                                                                \
  djv::launch_kernel(moe_scatter_kernel<T_, V_>, dim3(grid), dim3(256), sm, st, static_cast<T_ *>(xs),                \
                     static_cast<const T_ *>(x), static_cast<const int *>(expert), place,                             \
                     static_cast<const float *>(weight), ws, static_cast<const int *>(count), offsets, n, E, top, D)
  if (dtype == DJV_DTYPE_BF16) {
    if (vec) DJV_GO(bf16, true);
    else DJV_GO(bf16, false);
  } else {
    if (vec) DJV_GO(float, true);
    else DJV_GO(float, false);
  }
#undef DJV_GO
  count_launch(2);
  return check_launch("moe_route");
}

extern "C" int djv_moe_grouped(int dtype, void *y, const void *x, const void *w, const float *scale, const int *offsets,
                               int R, int E, int N, int K, int glu, void *stream) {
  DJV_REQUIRE(dtype == DJV_DTYPE_BF16 || dtype == DJV_DTYPE_F32, "moe_grouped: dtype %d", dtype);
  DJV_REQUIRE(y && x && w && offsets, "moe_grouped: null pointer");
  DJV_REQUIRE(R >= 1 && E >= 1 && E <= MAX_EXPERTS && N >= 1 && K >= 1 && (!glu || N % 2 == 0),
              "moe_grouped: R=%d E=%d N=%d K=%d", R, E, N, K);
  const GroupedArgs a{y, x, w, scale, offsets, R, E, N, K, glu};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (moe_grouped_tc_supported(dtype, a)) return moe_grouped_tc(a, st);
  const long long tiles = (long long)R / GG_M + E;  // no fewer than there can be
  DJV_REQUIRE(tiles <= 65535, "moe_grouped: %d rows are too many", R);
  const dim3 grid(ceil_div(N, GG_N), (unsigned)tiles);
  if (dtype == DJV_DTYPE_BF16) djv::launch_kernel(moe_grouped_kernel<bf16>, grid, dim3(GG_THREADS), 0, st, a);
  else djv::launch_kernel(moe_grouped_kernel<float>, grid, dim3(GG_THREADS), 0, st, a);
  count_launch();
  return check_launch("moe_grouped");
}

extern "C" int djv_moe_decode(int dtype, float *y, void *act, int *chosen, const void *x, const float *z, const void *w_gu,
                              const void *w_down, const void *shared_gu, const void *shared_down, const float *init, int B,
                              int E, int top, int D, int F, int F_shared, int ld_act, int stages, void *stream) {
  DJV_REQUIRE(dtype == DJV_DTYPE_BF16 || dtype == DJV_DTYPE_F32, "moe_decode: dtype %d", dtype);
  DJV_REQUIRE(y && act && chosen && x && z && w_gu && w_down && (!shared_gu) == (!shared_down), "moe_decode: null pointer");
  DJV_REQUIRE(B >= 1 && E >= 1 && top >= 1 && top <= E && top <= MAX_TOP && D >= 1 && F >= 1 && ld_act >= F &&
                  (!shared_gu || (F_shared >= 1 && ld_act >= F_shared)),
              "moe_decode: B=%d, %d of %d experts, D=%d F=%d + %d", B, top, E, D, F, F_shared);
  const MoeDecodeArgs a{y, act, chosen, x, z, w_gu, w_down, shared_gu, shared_down, init, B, E, top, D, F,
                        shared_gu ? F_shared : 0, ld_act};
  DJV_REQUIRE(ceil_div(F > a.F_shared ? F : a.F_shared, MO_WARPS) <= 65535 && ceil_div(D, MO_WARPS) <= 65535,
              "moe_decode: D=%d or F=%d is too large", D, F);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return dtype == DJV_DTYPE_BF16 ? launch_decode<bf16>(a, stages & 1, stages & 2, st)
                                 : launch_decode<float>(a, stages & 1, stages & 2, st);
}
