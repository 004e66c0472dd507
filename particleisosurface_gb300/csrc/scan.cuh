// Exclusive scan of a sequence given by an input functor: an int array, or
// flags worked out from node types, bitmap words and the like as they are read,
// so that no array of flags is written first.
//
// Up to 131072 elements take one launch: a block, or a cluster of 8 blocks that
// exchange their totals through distributed shared memory, holds the whole
// sequence in registers.  Longer ones take two: the tiles' sums, then the tiles,
// each of which adds up the sums before its own (a third launch scans the sums
// when there are more than 4096 tiles).  A frame runs 13 to 19 scans, nearly all
// of them short: as three launches each (tile sums, a scan of the sums, tiles)
// they took 140 us of a 2k-particle frame's 1.1 ms and 190 us of a 151k-particle
// frame's 1.8 ms, about 10 us a scan; one launch takes 3 to 5 us.
// Blocks of a cluster run at the same time by definition; no kernel waits on
// another launch, so nothing can spin.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace pisurf {

// int array; four(i) may load 16 bytes where the array allows it.
struct ScanInts {
  const int* p;
  __device__ int operator()(long long i) const { return p[i]; }
  __device__ int4 four(long long i) const {
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) return *reinterpret_cast<const int4*>(p + i);
    return make_int4(p[i], p[i + 1], p[i + 2], p[i + 3]);
  }
};

// f(i) for i < count, 0 at and past it (the sentinel whose place gets the
// total); f.four(i): elements i to i + 3, i a multiple of 4.
template <class F>
struct ScanOf {
  F f;
  long long count;
  __device__ int operator()(long long i) const { return i < count ? f(i) : 0; }
  __device__ int4 four(long long i) const {
    return i + 3 < count ? f.four(i) : make_int4((*this)(i), (*this)(i + 1), (*this)(i + 2), 0);
  }
};

template <class In>
__device__ __forceinline__ int4 scan_load(const In& in, long long i, long long n) {
  if (i + 3 < n) return in.four(i);
  return make_int4(i < n ? in(i) : 0, i + 1 < n ? in(i + 1) : 0, i + 2 < n ? in(i + 2) : 0, 0);
}

__device__ __forceinline__ void scan_store(int* out, long long i, long long n, int4 v) {
  if (i + 3 < n && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    *reinterpret_cast<int4*>(out + i) = v;
    return;
  }
  if (i < n) out[i] = v.x;
  if (i + 1 < n) out[i + 1] = v.y;
  if (i + 2 < n) out[i + 2] = v.z;
  if (i + 3 < n) out[i + 3] = v.w;
}

// Exclusive scan of a warp's 128 V elements from `base` on, in registers:
// v[k] becomes the exclusive sums of four elements; returns the warp's total.
template <class In, int V>
__device__ __forceinline__ int warp_scan(const In& in, long long base, long long n, int4 (&v)[V]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < V; ++k) v[k] = scan_load(in, base + (k * 32 + lane) * 4, n);
  int run = 0;
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int t = v[k].x + v[k].y + v[k].z + v[k].w;
    int inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const int e = run + inc - t;
    run += __shfl_sync(0xffffffffu, inc, 31);
    v[k] = make_int4(e, e + v[k].x, e + v[k].x + v[k].y, e + v[k].x + v[k].y + v[k].z);
  }
  return run;
}

// The block's warps' totals -> what comes before this warp; the block's total
// in *total.
template <int WARPS>
__device__ __forceinline__ int block_before(int mine, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_warp[warp] = mine;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const int t = s_warp[w];
    if (w < warp) before += t;
    all += t;
  }
  *total = all;
  return before;
}

// The whole sequence (at most CL * NT * 4 V elements) in one cluster.
template <class In, int NT, int V, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(NT)
    k_scan_one(In in, int* out, long long n, int* d_total) {
  launch_wait();
  namespace cg = cooperative_groups;
  __shared__ int s_warp[NT / 32];
  __shared__ int s_total;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long base = (long long)blockIdx.x * (NT * 4 * V) + warp * (128 * V);
  int4 v[V];
  const int mine = warp_scan<In, V>(in, base, n, v);
  int total;
  int before = block_before<NT / 32>(mine, s_warp, &total);
  if (CL > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    if (threadIdx.x == 0) s_total = total;
    cluster.sync();
    int ahead = 0;
    for (int q = 0; q < (int)blockIdx.x; ++q) ahead += *cluster.map_shared_rank(&s_total, q);
    before += ahead;
    total += ahead;
  }
  if (d_total && blockIdx.x == CL - 1 && threadIdx.x == 0) *d_total = total;
#pragma unroll
  for (int k = 0; k < V; ++k)
    scan_store(out, base + (k * 32 + lane) * 4, n,
               make_int4(v[k].x + before, v[k].y + before, v[k].z + before, v[k].w + before));
  if (CL > 1) cg::this_cluster().sync();  // the totals are read before their blocks end
}

// Longer sequences: tiles of 8192 elements.
constexpr int kTileThreads = 256, kTileV = 8;
constexpr int kScanTile = kTileThreads * 4 * kTileV;

template <class In>
__global__ void __launch_bounds__(kTileThreads) k_scan_sums(In in, long long n, int* sums) {
  launch_wait();
  __shared__ int s_warp[kTileThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = (long long)blockIdx.x * kScanTile;
  int acc = 0;
#pragma unroll
  for (int k = 0; k < kTileV; ++k) {
    const int4 v = scan_load(in, base + (k * kTileThreads + threadIdx.x) * 4, n);
    acc += v.x + v.y + v.z + v.w;
  }
  acc = __reduce_add_sync(0xffffffffu, acc);
  if (lane == 0) s_warp[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < kTileThreads / 32; ++w) t += s_warp[w];
    sums[blockIdx.x] = t;
  }
}

// scanned: sums[] already holds each tile's offset, else the tile adds up the
// sums before its own.
template <class In>
__global__ void __launch_bounds__(kTileThreads) k_scan_tiles(In in, int* out, long long n, const int* sums,
                                                             int scanned, int* d_total) {
  launch_wait();
  __shared__ int s_warp[kTileThreads / 32];
  __shared__ int s_pre[kTileThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = (long long)blockIdx.x * kScanTile + warp * (128 * kTileV);
  int4 v[kTileV];
  const int mine = warp_scan<In, kTileV>(in, base, n, v);
  int ahead = 0;
  if (scanned) {
    ahead = sums[blockIdx.x];
  } else {
    int part = 0;
    for (int i = threadIdx.x; i < (int)blockIdx.x; i += kTileThreads) part += sums[i];
    part = __reduce_add_sync(0xffffffffu, part);
    if (lane == 0) s_pre[warp] = part;
  }
  int total;
  int before = block_before<kTileThreads / 32>(mine, s_warp, &total);  // its barrier covers s_pre too
  if (!scanned)
    for (int w = 0; w < kTileThreads / 32; ++w) ahead += s_pre[w];
  before += ahead;
  if (d_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *d_total = ahead + total;
#pragma unroll
  for (int k = 0; k < kTileV; ++k)
    scan_store(out, base + (k * 32 + lane) * 4, n,
               make_int4(v[k].x + before, v[k].y + before, v[k].z + before, v[k].w + before));
}

constexpr long long kScanOneLaunch = 8LL * 512 * 4 * 8;  // elements one launch takes

// out[i] = sum of in(k), k < i, for i < n; the sum of all n in *d_total when
// given.  An int array may be scanned in place.  tmp: scan_tmp_ints(n) ints.
template <class In>
void exclusive_scan(const In& in, int* out, long long n, int* d_total, int* tmp, cudaStream_t s) {
  if (n <= 0) {
    if (d_total) PI_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), s));
    return;
  }
  // a block while 4 elements a thread hold the sequence; then the cluster, 4
  // elements a thread (8 SMs load at once) up to 32768, 32 above
  if (n <= 4096) {
    PI_LAUNCH((k_scan_one<In, 1024, 1, 1>), 1, 1024, 0, s, in, out, n, d_total);
    return;
  }
  if (n <= 8 * 4096) {
    PI_LAUNCH((k_scan_one<In, 1024, 1, 8>), 8, 1024, 0, s, in, out, n, d_total);
    return;
  }
  if (n <= kScanOneLaunch) {
    PI_LAUNCH((k_scan_one<In, 512, 8, 8>), 8, 512, 0, s, in, out, n, d_total);
    return;
  }
  const unsigned nt = div_up(n, kScanTile);
  PI_LAUNCH(k_scan_sums<In>, nt, kTileThreads, 0, s, in, n, tmp);
  const int scanned = nt > 4096 ? 1 : 0;
  if (scanned) exclusive_scan(ScanInts{tmp}, tmp, (long long)nt, nullptr, tmp + nt, s);
  PI_LAUNCH(k_scan_tiles<In>, nt, kTileThreads, 0, s, in, out, n, (const int*)tmp, scanned, d_total);
}

}  // namespace pisurf
