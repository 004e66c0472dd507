// Exclusive scan and stable LSD radix sort.
//
// The scan builds the cell offset tables, ranks the octree's INTERNAL nodes and
// numbers the extraction's vertices and triangles.  The radix sort orders
// particles by (grid, cell) where radii differ and in the build that allocates
// nothing (grid.cu's counting sort does the others), and the leaves' corners
// above D_max 14.
//
// Scan: scan.cuh.
// Radix sort: 8-bit digits; per pass a per-tile digit histogram, an exclusive
// scan of the digit-major histogram table, and a scatter in which each tile
// ranks its keys stably with warp match masks.  No kernel waits on another
// block, so nothing can spin.
#include "common.cuh"
#include "scan.cuh"

namespace pisurf {

std::atomic<unsigned long long> g_launches{0};

static constexpr int kThreads = 256;
static constexpr int kItems = 8;
static constexpr int kTile = kThreads * kItems;

size_t scan_tmp_ints(long long n) {
  const size_t nt = div_up(n > 0 ? n : 1, kScanTile);
  return nt + nt / kScanTile + 64;
}

void exclusive_scan_i32(const int* in, int* out, long long n, int* d_total, int* tmp, cudaStream_t s) {
  exclusive_scan(ScanInts{in}, out, n, d_total, tmp, s);
}

// ---------------------------------------------------------------------------
// radix sort
// ---------------------------------------------------------------------------
template <class K>
__global__ void k_rs_hist(const K* __restrict__ keys, long long n, int shift, int* __restrict__ hist,
                          int nt) {
  launch_wait();
  __shared__ int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  long long base = (long long)blockIdx.x * kTile;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    long long idx = base + (long long)i * kThreads + threadIdx.x;
    if (idx < n) atomicAdd(&h[(int)((keys[idx] >> shift) & 255)], 1);
  }
  __syncthreads();
  hist[(long long)threadIdx.x * nt + blockIdx.x] = h[threadIdx.x];
}

template <class K>
__global__ void k_rs_scatter(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                             K* __restrict__ kout, uint32_t* __restrict__ vout, long long n, int shift,
                             const int* __restrict__ offs, int nt) {
  launch_wait();
  __shared__ int run[256];
  __shared__ int wc[kThreads / 32][256];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  run[t] = offs[(long long)t * nt + blockIdx.x];
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) wc[w][t] = 0;
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
  long long base = (long long)blockIdx.x * kTile;
  for (int r = 0; r < kItems; ++r) {
    long long idx = base + (long long)r * kThreads + t;
    bool valid = idx < n;
    K key = valid ? kin[idx] : K(0);
    uint32_t val = valid ? vin[idx] : 0u;
    int d = valid ? (int)((key >> shift) & 255) : 256;
    unsigned peers = __match_any_sync(0xffffffffu, d);
    int leader = __ffs(peers) - 1;
    int rank = __popc(peers & lt);
    int cnt = __popc(peers);
    if (valid && lane == leader) wc[warp][d] = cnt;
    __syncthreads();
    if (valid) {
      int pos = run[d] + rank;
      for (int w = 0; w < warp; ++w) pos += wc[w][d];
      kout[pos] = key;
      vout[pos] = val;
    }
    __syncthreads();
    if (valid && lane == leader) {
      atomicAdd(&run[d], cnt);
      wc[warp][d] = 0;
    }
    __syncthreads();
  }
}

size_t radix_tmp_ints(long long n) {
  size_t nt = div_up(n > 0 ? n : 1, kTile);
  return 256 * nt + scan_tmp_ints((long long)(256 * nt)) + 32;
}

template <class K>
static void radix_sort(K** keys, uint32_t** vals, K** kalt, uint32_t** valt, long long n, int bits,
                       int* tmp, cudaStream_t s) {
  if (n <= 1 || bits <= 0) return;
  int nt = (int)div_up(n, kTile);
  int* hist = tmp;
  int* stmp = tmp + 256 * (size_t)nt;
  for (int shift = 0; shift < bits; shift += 8) {
    PI_LAUNCH(k_rs_hist<K>, nt, kThreads, 0, s, *keys, n, shift, hist, nt);
    exclusive_scan_i32(hist, hist, 256LL * nt, nullptr, stmp, s);
    PI_LAUNCH(k_rs_scatter<K>, nt, kThreads, 0, s, *keys, *vals, *kalt, *valt, n, shift, hist, nt);
    std::swap(*keys, *kalt);
    std::swap(*vals, *valt);
  }
}

void radix_sort_u32(uint32_t** keys, uint32_t** vals, uint32_t** kalt, uint32_t** valt, long long n,
                    int bits, int* tmp, cudaStream_t s) {
  radix_sort<uint32_t>(keys, vals, kalt, valt, n, bits, tmp, s);
}
void radix_sort_u64(uint64_t** keys, uint32_t** vals, uint64_t** kalt, uint32_t** valt, long long n,
                    int bits, int* tmp, cudaStream_t s) {
  radix_sort<uint64_t>(keys, vals, kalt, valt, n, bits, tmp, s);
}

}  // namespace pisurf
