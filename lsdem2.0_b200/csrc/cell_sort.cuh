// Pieces of the stable cell bucket sort, shared by the sort as separate launches (sort_scan.cu)
// and the sort inside the neighbour lists' rebuild (neighbours.cu).
#pragma once
#include "kernels.h"

namespace lsdem {

template <typename T>
__device__ T block_exclusive_scan(T v, T* smem_warp, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = (lane < (int)(blockDim.x >> 5)) ? smem_warp[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    smem_warp[lane] = w;
  }
  __syncthreads();
  T warp_off = warp > 0 ? smem_warp[warp - 1] : T(0);
  if (total) *total = smem_warp[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_off + x - v;
}

// Bucket of a key: 0 for -1 (outside the domain), 1 + key for a cell, and a
// last bucket for keys >= ncells (a centre rounding onto the upper domain face),
// which, as in the reference, sort after every cell, by key, and belong to none.
__device__ __forceinline__ int bucket_of(int k, int ncells) { return k < 0 ? 0 : (k >= ncells ? ncells + 1 : k + 1); }

// (key, index) order: a stable sort by key puts the keys past the last cell, which
// share the last bucket, in ascending key and then index order.
__device__ __forceinline__ bool key_idx_less(int ka, int a, int kb, int b) { return ka < kb || (ka == kb && a < b); }

// Compare-exchange of two (key, index) entries.
__device__ __forceinline__ void cx(int& ka, int& a, int& kb, int& b) {
  if (key_idx_less(kb, b, ka, a)) {
    const int t = a, tk = ka;
    a = b; ka = kb;
    b = t; kb = tk;
  }
}

// Bodies i0 to i1 of the first and last bucket (outside every cell) where these are longer than 64,
// by one block, in ascending index order from base0 and baseL on.
__device__ inline void special_buckets(const int* __restrict__ key, int i0, int i1, int ncells, const int* offs, int base0,
                                       int baseL, int* __restrict__ sorted_idx, int* sw) {
  const int L = ncells + 1;
  const bool long0 = offs[1] - offs[0] > 64, longL = offs[L + 1] - offs[L] > 64;
  if (!long0 && !longL) return;
  for (int t0 = i0; t0 < i1; t0 += blockDim.x) {
    const int i = t0 + threadIdx.x;
    const int b = i < i1 ? bucket_of(key[i], ncells) : -1;
    const int f0 = b == 0 && long0, fL = b == L && longL;
    int tot0, totL;
    const int r0 = block_exclusive_scan<int>(f0, sw, &tot0);
    const int rL = block_exclusive_scan<int>(fL, sw, &totL);
    if (f0) sorted_idx[base0 + r0] = i;
    if (fL) sorted_idx[baseL + rL] = i;
    base0 += tot0;
    baseL += totL;
  }
}

// A bucket of up to 8 members from s on, put in order in registers by one thread.
__device__ __forceinline__ void small_bucket(const int* __restrict__ key, bool bykey, int s, int L, int* sorted_idx) {
  int v[8], k[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = j < L ? sorted_idx[s + j] : 0x7fffffff;
    k[j] = (j < L && bykey) ? key[v[j]] : (j < L ? 0 : 0x7fffffff);
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) {
#pragma unroll
    for (int j = r & 1; j + 1 < 8; j += 2) cx(k[j], v[j], k[j + 1], v[j + 1]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < L) sorted_idx[s + j] = v[j];
}

// A bucket of 9 to 64 members, ranked in registers by one warp.
__device__ __forceinline__ void mid_bucket(const int* __restrict__ key, bool bykey, int s, int L, int* sorted_idx) {
  const int lane = threadIdx.x & 31;
  const int v0 = lane < L ? sorted_idx[s + lane] : 0x7fffffff;
  const int v1 = lane + 32 < L ? sorted_idx[s + 32 + lane] : 0x7fffffff;
  int r0 = 0, r1 = 0;
  if (bykey) {
    const int k0 = lane < L ? key[v0] : 0x7fffffff, k1 = lane + 32 < L ? key[v1] : 0x7fffffff;
    for (int j = 0; j < 32; ++j) {
      const int u0 = __shfl_sync(0xffffffffu, v0, j), u1 = __shfl_sync(0xffffffffu, v1, j);
      const int w0 = __shfl_sync(0xffffffffu, k0, j), w1 = __shfl_sync(0xffffffffu, k1, j);
      r0 += key_idx_less(w0, u0, k0, v0) + key_idx_less(w1, u1, k0, v0);
      r1 += key_idx_less(w0, u0, k1, v1) + key_idx_less(w1, u1, k1, v1);
    }
  } else {
    for (int j = 0; j < 32; ++j) {
      const int u0 = __shfl_sync(0xffffffffu, v0, j), u1 = __shfl_sync(0xffffffffu, v1, j);
      r0 += (u0 < v0) + (u1 < v0);
      r1 += (u0 < v1) + (u1 < v1);
    }
  }
  __syncwarp();
  if (lane < L) sorted_idx[s + r0] = v0;
  if (lane + 32 < L) sorted_idx[s + r1] = v1;
}

// A longer bucket, ranked by one block through tmp.
__device__ inline void big_bucket(const int* __restrict__ key, bool bykey, int s, int L, int* sorted_idx, int* tmp) {
  for (int k = threadIdx.x; k < L; k += blockDim.x) tmp[s + k] = sorted_idx[s + k];
  __syncthreads();
  for (int k = threadIdx.x; k < L; k += blockDim.x) {
    const int v = tmp[s + k], kv = bykey ? key[v] : 0;
    int r = 0;
    for (int m = 0; m < L; ++m) {
      const int u = tmp[s + m];
      r += bykey ? key_idx_less(key[u], u, kv, v) : u < v;
    }
    sorted_idx[s + r] = v;
  }
}

}  // namespace lsdem
