// K1: hash grid.  loadRootBox (src/surface_reconstructor.cpp:30-49) and the
// constant-radius HashGrid (src/hash_grid.cpp:4-139): bounding box, cell keys,
// the particles in key order (equal keys by index), dense cell offset table,
// and the positions in cell order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <stdexcept>
#include <string>

#include "device.cuh"
#include "internal.h"

namespace pisurf {

// Order-preserving float <-> uint encoding for atomic min/max.
__device__ __forceinline__ unsigned fenc(float f) {
  unsigned b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
static inline float fdec(unsigned e) {
  unsigned b = (e & 0x80000000u) ? (e & 0x7fffffffu) : ~e;
  float f;
  std::memcpy(&f, &b, 4);
  return f;
}

// misc[0..5] = enc(min x, max x, min y, max y, min z, max z); misc[6] = count
// of non-finite coordinates.
__global__ void k_bbox(const float* __restrict__ xyz, long long n, unsigned* __restrict__ misc) {
  launch_wait();
  unsigned mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
  unsigned bad = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float v = xyz[3 * i + k];
      if (!isfinite(v)) {
        ++bad;
        continue;
      }
      unsigned e = fenc(v);
      mn[k] = min(mn[k], e);
      mx[k] = max(mx[k], e);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = min(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
      mx[k] = max(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
    }
  }
  for (int o = 16; o > 0; o >>= 1) bad += __shfl_xor_sync(0xffffffffu, bad, o);
  // the block's warps combine in shared memory, so that each block issues one
  // set of atomics (all blocks hit the same seven words)
  __shared__ unsigned s_v[32][7];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    for (int k = 0; k < 3; ++k) {
      s_v[warp][2 * k] = mn[k];
      s_v[warp][2 * k + 1] = mx[k];
    }
    s_v[warp][6] = bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    for (int w = 1; w < nw; ++w)
      for (int k = 0; k < 3; ++k) {
        s_v[0][2 * k] = min(s_v[0][2 * k], s_v[w][2 * k]);
        s_v[0][2 * k + 1] = max(s_v[0][2 * k + 1], s_v[w][2 * k + 1]);
      }
    for (int w = 1; w < nw; ++w) s_v[0][6] += s_v[w][6];
    for (int k = 0; k < 3; ++k) {
      atomicMin(misc + 2 * k, s_v[0][2 * k]);
      atomicMax(misc + 2 * k + 1, s_v[0][2 * k + 1]);
    }
    if (s_v[0][6]) atomicAdd(misc + 6, s_v[0][6]);
  }
}

__global__ void k_init_misc(unsigned* misc) {
  launch_wait();
  int t = threadIdx.x;
  if (t < 6) misc[t] = (t & 1) ? 0u : 0xffffffffu;
  if (t >= 6 && t < 16) misc[t] = 0;
}

// CalcXYZIdx + CalcCellHash (src/hash_grid.cpp:124-139) per particle; key -1
// outside the grid.  skey = key + 1 so that key -1 sorts first, as the
// reference's std::sort on long long keys does.
__global__ void k_keys(const float* __restrict__ xyz, long long n, float b0, float b2, float b4,
                       float cell, int nx, int ny, int nz, int* __restrict__ key,
                       uint32_t* __restrict__ skey, uint32_t* __restrict__ sidx) {
  launch_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
  int cx = (int)__fdiv_rn(__fsub_rn(x, b0), cell);
  int cy = (int)__fdiv_rn(__fsub_rn(y, b2), cell);
  int cz = (int)__fdiv_rn(__fsub_rn(z, b4), cell);
  int k = -1;
  if (cx >= 0 && cx < nx && cy >= 0 && cy < ny && cz >= 0 && cz < nz)
    k = (int)(((long long)cz * ny + cy) * nx + cx);
  key[i] = k;
  skey[i] = (uint32_t)(k + 1);
  sidx[i] = (uint32_t)i;
}

__global__ void k_cell_count(const int* __restrict__ key, long long n, int* __restrict__ cnt) {
  launch_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int k = key[i];
  if (k >= 0) atomicAdd(cnt + k, 1);
}

// ---------------------------------------------------------------------------
// The frame's hash order (IndexList): a counting sort by cell, since the cell
// counts are needed anyway.  Particles take places in their cell's range in any
// order, then each cell's few particles (8 on a liquid's lattice) are put in
// index order, which is what a stable sort by key gives.  Four launches with
// the scan, against fifteen for three 8-bit radix passes: 110 -> 25 us of a
// 151k-particle frame, 130 -> 55 us at 1M (a radix pass's time on such sizes is
// launches and block barriers).  Particles outside the grid (key -1) form a range
// of their own at the front, as the reference's sort puts them.
// ---------------------------------------------------------------------------
constexpr int kSmallCell = 256;   // larger cells are radix-sorted by a block each
constexpr int kHugeCell = 4096;   // still larger ones are split over blocks by index windows
constexpr int kWindowWords = 10240;  // bits of a window's particles, in shared memory
constexpr int kWindows = 32;         // windows at least

// Key, and the particle's place in its cell (cnt: cell counts, zeroed;
// *outside: particles of key -1).  A warp's particles of one cell add their
// number once: one by one, the additions of 1M particles in one cell took 0.9 ms.
__global__ void k_cell_place(const float* __restrict__ xyz, long long n, float b0, float b2, float b4, float cell,
                             int nx, int ny, int nz, int* __restrict__ key, int* __restrict__ cnt,
                             unsigned* __restrict__ outside, uint32_t* __restrict__ place) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int k = -2;  // a lane past the end
  if (i < n) {
    const int cx = (int)__fdiv_rn(__fsub_rn(xyz[3 * i], b0), cell);
    const int cy = (int)__fdiv_rn(__fsub_rn(xyz[3 * i + 1], b2), cell);
    const int cz = (int)__fdiv_rn(__fsub_rn(xyz[3 * i + 2], b4), cell);
    k = -1;
    if (cx >= 0 && cx < nx && cy >= 0 && cy < ny && cz >= 0 && cz < nz) k = (int)(((long long)cz * ny + cy) * nx + cx);
  }
  const unsigned peers = __match_any_sync(0xffffffffu, k);
  const int lead = __ffs(peers) - 1;
  int first = 0;
  if (lane == lead && k >= -1)
    first = k >= 0 ? atomicAdd(cnt + k, __popc(peers)) : (int)atomicAdd(outside, (unsigned)__popc(peers));
  first = __shfl_sync(0xffffffffu, first, lead);
  if (i >= n) return;
  key[i] = k;
  place[i] = (uint32_t)(first + __popc(peers & ((1u << lane) - 1u)));
}

// Sorted range of cell k (-1: the particles outside the grid).
__device__ __forceinline__ void cell_range(const int* __restrict__ off, long long cells, long long n, int k, int* s,
                                           int* e) {
  const int front = (int)(n - off[cells]);
  *s = k >= 0 ? front + off[k] : 0;
  *e = k >= 0 ? front + off[k + 1] : front;
}

__global__ void k_cell_scatter(const int* __restrict__ key, const uint32_t* __restrict__ place,
                               const int* __restrict__ off, long long cells, long long n, uint32_t* __restrict__ list) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s, e;
  cell_range(off, cells, n, key[i], &s, &e);
  list[s + place[i]] = (uint32_t)i;
}

__device__ __forceinline__ void put_particle(const float* __restrict__ xyz, uint32_t i, long long t,
                                             uint32_t* __restrict__ sidx, float4* __restrict__ pos) {
  sidx[t] = i;
  pos[t] = make_float4(xyz[3ll * i], xyz[3ll * i + 1], xyz[3ll * i + 2], 0.f);
}

// A thread per particle counts the lower indices of its cell; the first one of
// a cell above kSmallCell lists the cell instead (big: [0, listed), the cells
// above kHugeCell from its end; nbig: both counts).
__global__ void k_cell_sort(const float* __restrict__ xyz, const int* __restrict__ key,
                            const uint32_t* __restrict__ list, const int* __restrict__ off, long long cells,
                            long long n, uint32_t* __restrict__ sidx, float4* __restrict__ pos, int* __restrict__ big,
                            long long listed, unsigned* __restrict__ nbig) {
  launch_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const uint32_t i = list[t];
  const int k = key[i];
  int s, e;
  cell_range(off, cells, n, k, &s, &e);
  if (e - s > kSmallCell) {
    if (t == s) {
      if (e - s > kHugeCell)
        big[listed - 1 - atomicAdd(nbig + 1, 1u)] = k;
      else
        big[atomicAdd(nbig, 1u)] = k;
    }
    return;
  }
  int rank = 0;
  for (int u = s; u < e; ++u) rank += list[u] < i ? 1 : 0;
  put_particle(xyz, i, s + rank, sidx, pos);
}

// A window of a huge cell's particles, by a block: the indices of [w width,
// (w + 1) width) as bits, and the number of lower ones; what comes before a
// particle in the cell is then a count of bits.  Every window reads all of the
// cell's list, so that none waits for another.
constexpr int kBigThreads = 256;
__device__ void cell_window(const float* __restrict__ xyz, const uint32_t* __restrict__ list, long long n, int s, int e,
                            uint32_t w, uint32_t width, unsigned* bits, int* s_sum, uint32_t* __restrict__ sidx,
                            float4* __restrict__ pos) {
  constexpr int warps = kBigThreads / 32;
  const int x = threadIdx.x, lane = x & 31, warp = x >> 5;
  const int words = (int)(width / 32);
  const uint32_t lo = w * width;
  for (int k = x; k < words; k += kBigThreads) bits[k] = 0u;
  __syncthreads();
  int below = 0;
  auto take = [&](long long t, uint32_t i) {
    if (t < s || t >= e) return;
    if (i < lo)
      ++below;
    else if (i - lo < width)
      atomicOr(bits + ((i - lo) >> 5), 1u << (i & 31u));  // lo is a multiple of 32
  };
#pragma unroll 4
  for (long long q = s / 4 + x; q < (e + 3) / 4; q += kBigThreads) {
    if (4 * q + 3 < n) {
      const uint4 v = reinterpret_cast<const uint4*>(list)[q];
      take(4 * q, v.x), take(4 * q + 1, v.y), take(4 * q + 2, v.z), take(4 * q + 3, v.w);
    } else {
      for (long long t = 4 * q; t < n; ++t) take(t, list[t]);
    }
  }
  below = __reduce_add_sync(0xffffffffu, below);
  if (lane == 0) s_sum[warp] = below;
  __syncthreads();
  // a thread's run of words
  const int run = (words + kBigThreads - 1) / kBigThreads, k0 = min(x * run, words), k1 = min(k0 + run, words);
  int count = 0;
  for (int k = k0; k < k1; ++k) count += __popc(bits[k]);
  int inc = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s_sum[warps + warp] = inc;
  __syncthreads();
  long long at = s + inc - count;
  for (int k = 0; k < warps; ++k) at += s_sum[k] + (k < warp ? s_sum[warps + k] : 0);
  for (int k = k0; k < k1; ++k)
    for (unsigned b = bits[k]; b != 0u; b &= b - 1u)
      put_particle(xyz, lo + 32u * k + (uint32_t)(__ffs(b) - 1), at++, sidx, pos);
  __syncthreads();
}

// The listed cells.  Up to kHugeCell a block per cell, stable 8-bit radix passes
// over the particle indices (list and alt in turn; four passes end in list).
// Larger ones (a clump, or a lattice's face on the grid's upper bound, all of
// which has key -1) in windows: one block's passes, three barriers for 256
// particles each, took 390 us of a 1M lattice with 30,000 particles on the
// bound and 13.3 ms of 1M particles in one cell.
__global__ void __launch_bounds__(kBigThreads) k_cell_sort_big(const float* __restrict__ xyz, uint32_t* list,
                                                               uint32_t* alt, const int* __restrict__ off,
                                                               long long cells, long long n,
                                                               uint32_t* __restrict__ sidx, float4* __restrict__ pos,
                                                               const int* __restrict__ big, long long listed,
                                                               const unsigned* __restrict__ nbig) {
  launch_wait();
  constexpr int warps = kBigThreads / 32;
  __shared__ unsigned s_bits[kWindowWords];
  __shared__ int s_run[256];
  const int x = threadIdx.x, lane = x & 31, warp = x >> 5;
  // windows as wide as the bits allow, or narrower
  const uint32_t span = max((uint32_t)kWindows, (uint32_t)((n + 32ll * kWindowWords - 1) / (32ll * kWindowWords)));
  const uint32_t width = (uint32_t)((n + 32ll * span - 1) / (32ll * span)) * 32u;
  const uint32_t windows = (uint32_t)((n + width - 1) / width);
  for (long long t = blockIdx.x; t < (long long)nbig[1] * windows; t += gridDim.x) {
    int s, e;
    cell_range(off, cells, n, big[listed - 1 - t / windows], &s, &e);
    cell_window(xyz, list, n, s, e, (uint32_t)(t % windows), width, s_bits, s_run, sidx, pos);
  }
  int(*const s_cnt)[256] = reinterpret_cast<int(*)[256]>(s_bits);
  static_assert(warps * 256 <= kWindowWords && 2 * warps <= 256, "shared by the two paths");
  for (unsigned b = blockIdx.x; b < *nbig; b += gridDim.x) {
    int s, e;
    cell_range(off, cells, n, big[b], &s, &e);
    uint32_t *from = list + s, *to = alt + s;
    const int len = e - s;
    for (int shift = 0; shift < 32; shift += 8) {
      s_run[x] = 0;
      for (int w = 0; w < warps; ++w) s_cnt[w][x] = 0;
      __syncthreads();
      for (int j = x; j < len; j += kBigThreads) atomicAdd(&s_run[(from[j] >> shift) & 255u], 1);
      __syncthreads();
      if (warp == 0) {  // exclusive scan of the 256 counts, eight a lane
        int v[8], sum = 0;
        for (int q = 0; q < 8; ++q) v[q] = s_run[lane * 8 + q], sum += v[q];
        int inc = sum;
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += u;
        }
        int run = inc - sum;
        for (int q = 0; q < 8; ++q) s_run[lane * 8 + q] = run, run += v[q];
      }
      __syncthreads();
      for (int j0 = 0; j0 < len; j0 += kBigThreads) {
        const int j = j0 + x;
        const bool valid = j < len;
        const uint32_t v = valid ? from[j] : 0u;
        const int d = valid ? (int)((v >> shift) & 255u) : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const bool lead = valid && lane == __ffs(peers) - 1;
        if (lead) s_cnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
          int p = s_run[d] + __popc(peers & ((1u << lane) - 1u));
          for (int w = 0; w < warp; ++w) p += s_cnt[w][d];
          to[p] = v;
        }
        __syncthreads();
        if (lead) {
          atomicAdd(&s_run[d], __popc(peers));
          s_cnt[warp][d] = 0;
        }
        __syncthreads();
      }
      uint32_t* const tmp = from;
      from = to;
      to = tmp;
    }
    for (int j = x; j < len; j += kBigThreads) put_particle(xyz, from[j], s + j, sidx, pos);
    __syncthreads();
  }
}

void stage_upload_host(pi_frame* f, const float* xyz, long long n) {
  cudaStream_t s = f->ctx->stream;
  f->stage = 0;  // no particles until they are here: the results are of another count
  f->N = n;
  f->xyz.alloc(f->ctx, s, (size_t)n * 3);
  PI_CUDA(cudaMemcpyAsync(f->xyz.p, xyz, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, s));
}

void stage_upload_device(pi_frame* f, const float* d_xyz, long long n) {
  cudaStream_t s = f->ctx->stream;
  f->stage = 0;  // no particles until they are here: the results are of another count
  f->N = n;
  f->xyz.alloc(f->ctx, s, (size_t)n * 3);
  PI_CUDA(cudaMemcpyAsync(f->xyz.p, d_xyz, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, s));
}

long long grid_cell_counts(const float bounding[6], float cell, long long max_cells, int nn[3]) {
  double total = 1.0;
  for (int i = 0; i < 3; ++i) {
    // XYZCellNum (src/hash_grid.cpp:24-27): ceil of a float quotient; a
    // tiny radius makes it too large for an int, so it is checked as a float
    // (NaN and infinity fail the test too) before the conversion
    const float q = std::ceil((bounding[i * 2 + 1] - bounding[i * 2]) / cell);
    if (!(q <= (float)max_cells))
      throw std::length_error("hash grid axis of " + std::to_string(q) + " cells exceeds the limit of " +
                              std::to_string(max_cells) + " cells (radius too small for the particle box)");
    nn[i] = std::max(int(q), 1);
    total *= nn[i];
  }
  if (total > (double)max_cells)
    throw std::length_error("hash grid of " + std::to_string((long long)total) + " cells exceeds the limit of " +
                            std::to_string(max_cells) + " cells");
  return (long long)nn[0] * nn[1] * nn[2];
}

void stage_hashgrid(pi_frame* f) {
  cudaStream_t s = f->ctx->stream;
  f->f64_ready = false;
  const long long n = f->N;
  f->misc.alloc(f->ctx, s, 16);
  PI_LAUNCH(k_init_misc, 1, 32, 0, s, f->misc.p);
  int blocks = (int)std::min<long long>(div_up(n, 256), (long long)f->ctx->smCount * 2);
  PI_LAUNCH(k_bbox, blocks, 256, 0, s, f->xyz.p, n, f->misc.p);
  unsigned* const h = reinterpret_cast<unsigned*>(f->ctx->hpin + kPinReadOffset);
  PI_CUDA(cudaMemcpyAsync(h, f->misc.p, sizeof(unsigned) * 8, cudaMemcpyDeviceToHost, s));
  // the buffers that do not depend on the box, while it is worked out (under a
  // budget after it, which refuses positions that are not finite whatever is left)
  auto buffers = [&]() {
    f->key.alloc(f->ctx, s, n);
    f->sidx.alloc(f->ctx, s, n);
    f->u32a.alloc(f->ctx, s, n);
    f->u32b.alloc(f->ctx, s, n);
    f->u32c.alloc(f->ctx, s, n / kSmallCell + 1);  // a listed cell holds more than kSmallCell
    f->pos.alloc(f->ctx, s, n);
  };
  if (!f->ctx->budget) buffers();
  PI_CUDA(cudaStreamSynchronize(s));
  if (h[6]) throw std::invalid_argument("non-finite particle coordinate");
  float bb[6];
  for (int k = 0; k < 6; ++k) bb[k] = fdec(h[k]);
  f->singleLayer = (bb[0] == bb[1] || bb[2] == bb[3] || bb[4] == bb[5]);

  // HashGrid ctor (src/hash_grid.cpp:4-34), same float expressions.
  GridHost& g = f->g;
  const float cell = f->P.radius * 4.0f;
  g.cell = cell;
  for (int i = 0; i < 3; ++i) {
    float length = (std::ceil((bb[i * 2 + 1] - bb[i * 2]) / cell)) * cell;
    float center = (bb[i * 2] + bb[i * 2 + 1]) / 2;
    g.bounding[i * 2] = center - length / 2;
    g.bounding[i * 2 + 1] = center + length / 2;
  }
  int nn[3];
  // FindStartEnd stores keys in an int (src/hash_grid.cpp:105).
  g.cellNum = grid_cell_counts(g.bounding, cell, (1LL << 31) - 2, nn);
  g.nx = nn[0], g.ny = nn[1], g.nz = nn[2];
  if (f->ctx->budget) buffers();
  f->tmp.alloc(f->ctx, s, scan_tmp_ints(g.cellNum + 1));
  f->off.alloc(f->ctx, s, g.cellNum + 1);
  // misc[7]: particles outside the grid, misc[8], misc[9]: cells above kSmallCell
  // and kHugeCell (zeroed by k_init_misc)
  int* const big = reinterpret_cast<int*>(f->u32c.p);
  const long long listed = n / kSmallCell + 1;
  PI_CUDA(cudaMemsetAsync(f->off.p, 0, sizeof(int) * (g.cellNum + 1), s));
  PI_LAUNCH(k_cell_place, div_up(n, 256), 256, 0, s, f->xyz.p, n, g.bounding[0], g.bounding[2], g.bounding[4], cell,
            g.nx, g.ny, g.nz, f->key.p, f->off.p, f->misc.p + 7, f->u32b.p);
  exclusive_scan_i32(f->off.p, f->off.p, g.cellNum + 1, nullptr, f->tmp.p, s);
  PI_LAUNCH(k_cell_scatter, div_up(n, 256), 256, 0, s, f->key.p, f->u32b.p, f->off.p, g.cellNum, n, f->u32a.p);
  PI_LAUNCH(k_cell_sort, div_up(n, 256), 256, 0, s, f->xyz.p, f->key.p, f->u32a.p, f->off.p, g.cellNum, n, f->sidx.p,
            f->pos.p, big, listed, f->misc.p + 8);
  PI_LAUNCH(k_cell_sort_big, (int)std::min<long long>(n / kSmallCell, 4ll * f->ctx->smCount), kBigThreads, 0, s,
            f->xyz.p, f->u32a.p, f->u32b.p, f->off.p, g.cellNum, n, f->sidx.p, f->pos.p, big, listed, f->misc.p + 8);
  // the valid-key count (offset table total) reaches g.nInvalid in
  // resolve_pending; nothing before the end of the call reads it
  f->pin_pending |= 1 << kPinValid;
  // loadRootBox result kept for the octree root (resizeRootBoxConstR)
  for (int k2 = 0; k2 < 6; ++k2) f->bbox6[k2] = bb[k2];
}

}  // namespace pisurf
