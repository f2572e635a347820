// Keys and values of a prompt into the caches of the decode kernels.
//   K cache (B,nheads,hd/8,S,8)   V cache (B,nheads,S,hd)   qkv (B,L,3,nheads,hd)
// A block takes 32 positions of one head. Both sides move whole lines: a position's hd values are read in a row; of the
// keys, 16-byte pieces change places in shared memory, so that 32 positions of one piece are written in a row. Bound by
// HBM: L = 1983, 32 heads of 128, inputs and caches rotating over more than L2: 32.5 MB read and as much written in 11.9 us,
// 0.84 of the copy rate (two permuting copies before: 42.3).
#include "common.cuh"

namespace djv {

constexpr int KS_POS = 32, KS_THREADS = 256;

template <int HD>
__global__ void __launch_bounds__(KS_THREADS)
kv_store_kernel(__half *__restrict__ k_cache, __half *__restrict__ v_cache, const __half *__restrict__ qkv, int L, int nheads, int S) {
  constexpr int P = HD / 8, N = KS_POS * P / KS_THREADS > 0 ? KS_POS * P / KS_THREADS : 1;  // pieces of a position, of a thread
  __shared__ uint4 ks[KS_POS][P + 1];
  pdl_prologue();
  const int tid = threadIdx.x, p0 = blockIdx.x * KS_POS, h = blockIdx.y, b = blockIdx.z;
  const size_t bh = (size_t)b * nheads + h, row = (size_t)3 * nheads * HD;
  const uint4 *src = reinterpret_cast<const uint4 *>(qkv + (size_t)b * L * row + (size_t)(nheads + h) * HD);
  uint4 k[N], v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int o = tid + i * KS_THREADS, pos = o / P, c = o % P;
    if (pos < KS_POS && p0 + pos < L) {
      const uint4 *at = src + (size_t)(p0 + pos) * (row / 8) + c;
      k[i] = ld_stream16(at);
      v[i] = ld_stream16(at + (size_t)nheads * P);
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int o = tid + i * KS_THREADS, pos = o / P, c = o % P;
    if (pos < KS_POS && p0 + pos < L) {
      ks[pos][c] = k[i];
      reinterpret_cast<uint4 *>(v_cache)[(bh * S + p0 + pos) * P + c] = v[i];
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int o = tid + i * KS_THREADS, pos = o % KS_POS, c = o / KS_POS;
    if (c < P && p0 + pos < L) reinterpret_cast<uint4 *>(k_cache)[(bh * P + c) * S + p0 + pos] = ks[pos][c];
  }
}

}  // namespace djv

using namespace djv;

extern "C" int djv_kv_store(void *k_cache, void *v_cache, const void *qkv, int B, int L, int nheads, int hd, int S, void *stream) {
  DJV_REQUIRE(k_cache && v_cache && qkv, "kv_store: null pointer");
  DJV_REQUIRE(hd == 32 || hd == 64 || hd == 128, "kv_store: head_dim %d not in {32,64,128}", hd);
  DJV_REQUIRE(B >= 1 && B <= 65535 && nheads >= 1 && nheads <= 65535 && L >= 1 && L <= S, "kv_store: B=%d L=%d nheads=%d S=%d", B, L,
              nheads, S);
  DJV_REQUIRE(aligned16(k_cache) && aligned16(v_cache) && aligned16(qkv), "kv_store: pointers must be 16-byte aligned");
  const dim3 grid(ceil_div(L, KS_POS), nheads, B);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  __half *k = static_cast<__half *>(k_cache), *v = static_cast<__half *>(v_cache);
  const __half *x = static_cast<const __half *>(qkv);
  if (hd == 128) djv::launch_kernel(kv_store_kernel<128>, grid, dim3(KS_THREADS), 0, st, k, v, x, L, nheads, S);
  else if (hd == 64) djv::launch_kernel(kv_store_kernel<64>, grid, dim3(KS_THREADS), 0, st, k, v, x, L, nheads, S);
  else djv::launch_kernel(kv_store_kernel<32>, grid, dim3(KS_THREADS), 0, st, k, v, x, L, nheads, S);
  count_launch();
  return check_launch("kv_store");
}
