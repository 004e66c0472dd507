// K6: dual-grid extraction, genIsoOurs state 1 (src/surface_reconstructor.cpp:290-323).
//
// The reference walks the octree recursively (include/traverse.h) and visits
// every interior octree vertex once with the 8 leaves around it
// (VisitorExtract::on_vert, src/visitorextract.cpp:229-256).  Those vertices
// are exactly the corners of leaves that lie strictly inside the root box, so
// here they are enumerated in parallel:
//   1. every leaf marks its interior corners (integer lattice at D_max) in
//      a Morton-indexed lattice bitmap (sort + unique above D_max = 14); the
//      set bits in index order are the dual vertices, in Z order;
//   2. per vertex, the leaf containing each of the 8 octants is found by
//      descending from the root; sign code, table[256] -> canonical case;
//   3. per non-trivial cell, the case triangles (src/visitorextract.cpp:95-199)
//      name leaf pairs; mesh vertices are deduplicated by the sorted leaf-id
//      pair, as Mesh::insert_vert keys them (src/global.cpp:13-32), the
//      first (lowest) slot of a key winning, through a hash table in L2;
//   4. each mesh vertex's leaf-to-leaf segment is bisected down to r/2 with a
//      field evaluation per step (a warp's vertices share the candidates,
//      group_field) and interpolated with the 0.1/0.9 snap (calc_vertices,
//      src/visitorextract.cpp:47-84);
//   5. triangles are oriented by the table's flip and deduplicated by their
//      sorted vertex triple, the first generated winning (Mesh::insert_tri,
//      src/global.cpp:34-53).
// The output order differs from the reference's traversal order; the mesh is
// the same set of vertices (by leaf-id pair) and triangles.
#include <algorithm>
#include <mutex>

#include "chunk.cuh"
#include "device.cuh"
#include "dmc.h"
#include "internal.h"
#include "scan.cuh"

namespace pisurf {

// The DMC table packed for device reads, one word per sign code: bits 3 c to
// 3 c + 2 the corner that canonical corner c is, bit 24 the flip, bits 25 to 28
// the triangles, bit 29 set unless all signs are equal; and the edges (0 to 11,
// four bits each) of its triangles' corners.  Plain loads: lanes read different
// entries, which the constant cache would serve one after another (as it did
// the eight corner words, the code, flip, count and edges of the unpacked
// table).
__device__ unsigned d_case[256];
__device__ unsigned long long d_edges[256];
constexpr unsigned kCaseFlip = 1u << 24, kCaseMixed = 1u << 29;
__device__ __forceinline__ int case_corner(unsigned cs, int c) { return (cs >> (3 * c)) & 7; }
__device__ __forceinline__ int case_triangles(unsigned cs) { return (cs >> 25) & 15; }

void dmc_host_table(int trans[256][8], bool flip[256], int code[256]) {
  DmcTables t;
  dmc_build(&t);
  for (int i = 0; i < 256; ++i) {
    for (int k = 0; k < 8; ++k) trans[i][k] = t.trans[i][k];
    flip[i] = t.flip[i] != 0;
    code[i] = t.code[i];
  }
}

static void upload_tables(int device) {
  static std::mutex mu;
  static bool done[128] = {false};
  std::lock_guard<std::mutex> lk(mu);
  if (device >= 0 && device < 128 && done[device]) return;
  DmcTables t;
  dmc_build(&t);
  unsigned cs[256];
  unsigned long long edges[256];
  for (int i = 0; i < 256; ++i) {
    const int code = t.code[i];
    const bool mixed = code != 0 && code != 255;
    cs[i] = (t.flip[i] ? kCaseFlip : 0u) | (mixed ? kCaseMixed | ((unsigned)t.ntri[code] << 25) : 0u);
    edges[i] = 0;
    for (int c = 0; c < 8; ++c) cs[i] |= (unsigned)t.trans[i][c] << (3 * c);
    if (mixed)
      for (int k = 0; k < 3 * t.ntri[code]; ++k) edges[i] |= (unsigned long long)t.tri[code][k] << (4 * k);
  }
  PI_CUDA(cudaMemcpyToSymbol(d_case, cs, sizeof(cs)));
  PI_CUDA(cudaMemcpyToSymbol(d_edges, edges, sizeof(edges)));
  // a copy from pageable memory may return before it has arrived, and the contexts'
  // streams do not wait for the default one
  PI_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
  if (device >= 0 && device < 128) done[device] = true;
}

__device__ __forceinline__ void edge_corners(int e, int* c0, int* c1) {
  const int axis = e >> 2, k = e & 3;
  const int u = axis == 0 ? 1 : 0, v = axis == 2 ? 1 : 2;
  *c0 = ((k & 1) << u) | (((k >> 1) & 1) << v);
  *c1 = *c0 | (1 << axis);
}

// Scan input: set bits of the bitmap words.
struct WordBits {
  const unsigned* bits;
  __device__ int operator()(long long i) const { return __popc(bits[i]); }
  __device__ int4 four(long long i) const {
    const uint4 b = *reinterpret_cast<const uint4*>(bits + i);
    return make_int4(__popc(b.x), __popc(b.y), __popc(b.z), __popc(b.w));
  }
};

// Interior corners of the leaves, key (x << 2B) | (y << B) | z, B = D_max + 1.  A
// thread per point of a family's 3 x 3 x 3 lattice (27 keys for eight leaves'
// 64 corners); boundary points, and those that are no leaf's corner, get the
// all-ones key.
__global__ void k_corner_keys(const int* __restrict__ nd_child, long long nf, const int4* __restrict__ nd_org,
                              int full, int B, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  launch_wait();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nf * 27) return;
  const long long first = 8 * (t / 27) + 1;  // the family's first node
  const int p = (int)(t % 27), ix = p % 3, iy = p / 3 % 3, iz = p / 9;
  const int4 o = nd_org[first];
  const int x = o.x + ix * o.w, y = o.y + iy * o.w, z = o.z + iz * o.w;
  bool leaf = false;  // of the children around the point
  for (int k = 0; k < 8; ++k) {
    const int dx = ix - (k & 1), dy = iy - ((k >> 1) & 1), dz = iz - (k >> 2);
    if ((unsigned)dx < 2u && (unsigned)dy < 2u && (unsigned)dz < 2u) leaf = leaf || nd_child[first + k] < 0;
  }
  uint64_t key;
  if (leaf && x > 0 && x < full && y > 0 && y < full && z > 0 && z < full)
    key = ((uint64_t)x << (2 * B)) | ((uint64_t)y << B) | (uint64_t)z;
  else
    key = (1ull << (3 * B)) - 1ull;
  keys[t] = key;
  vals[t] = (uint32_t)t;
}

// Morton code of three coordinates of up to 21 bits each (bit interleaving
// by the usual shift-and-mask steps), and its inverse.
__device__ __forceinline__ uint64_t spread3(uint64_t v) {
  v &= 0x1fffffull;
  v = (v | (v << 32)) & 0x1f00000000ffffull;
  v = (v | (v << 16)) & 0x1f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}
__device__ __forceinline__ uint64_t compact3(uint64_t v) {
  v &= 0x1249249249249249ull;
  v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ull;
  v = (v ^ (v >> 4)) & 0x100f00f00f00f00full;
  v = (v ^ (v >> 8)) & 0x1f0000ff0000ffull;
  v = (v ^ (v >> 16)) & 0x1f00000000ffffull;
  v = (v ^ (v >> 32)) & 0x1fffffull;
  return v;
}

// Interior leaf corners (coordinates 1 .. 2^D_max - 1) as bits of a lattice
// bitmap indexed by the Morton code of (x - 1, y - 1, z - 1).  The Morton
// range is cut into blocks of 2^bb codes (a 2^(bb/3)-cube of lattice
// points).  Up to D_max = 9 (2^27 bits) every block is stored (slot = block,
// slot and blist null); above it only the blocks that hold a corner, with
// consecutive slots in block order, so that work and memory follow the
// surface rather than the volume of the lattice.  Either way the set bits in
// slot order are the unique corners in Z order, which keeps the later
// per-vertex work spatially coherent (as the reference's recursive
// traversal is).
//
// The corners are taken family by family: the eight children of a node are
// consecutive (family f holds nodes 8 f + 1 to 8 f + 8), and when all eight are
// leaves, as nearly every family with a leaf is, their 64 corners are the 27
// points of a 3 x 3 x 3 lattice.  A point's Morton code is the OR of its
// coordinates' spread codes, so the points of one bitmap word are a product of
// per-axis sets and their bits come from shifts: two to eight words, and as many
// atomics, a family.  A lane per corner, merging the bits of equal words across
// the warp, took 438 us for the 4.4M leaves of a 1M dam-break frame (12 merge
// rounds a warp); a thread per family takes 37 us and needs no leaf list.

// The spread codes (x and shifts applied) of the three lattice coordinates
// o - 1, o + w - 1, o + 2 w - 1 of one axis; code[i] = -1 where the point is not
// interior.
__device__ __forceinline__ void axis_codes(int o, int w, int full, int shift, long long (&code)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int x = o + i * w;
    code[i] = x > 0 && x < full ? (long long)(spread3((uint64_t)(x - 1)) << shift) : -1;
  }
}

struct Family {
  int leaves;  // bit k: child k is a leaf
  long long cx[3], cy[3], cz[3];
};

__device__ __forceinline__ bool load_family(const int* __restrict__ nd_child, const int4* __restrict__ nd_org,
                                            long long nf, long long f, int full, Family& fam) {
  if (f >= nf) return false;
  fam.leaves = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) fam.leaves |= (nd_child[8 * f + 1 + k] < 0 ? 1 : 0) << k;
  if (fam.leaves == 0) return false;
  const int4 o = nd_org[8 * f + 1];
  axis_codes(o.x, o.w, full, 0, fam.cx);
  axis_codes(o.y, o.w, full, 1, fam.cy);
  axis_codes(o.z, o.w, full, 2, fam.cz);
  return true;
}

// visit(code) for every interior corner of the family's leaves, some of them
// more than once.
template <class V>
__device__ __forceinline__ void family_corners(const Family& fam, const V& visit) {
  for (int k = 0; k < 8; ++k) {
    if (!((fam.leaves >> k) & 1)) continue;
    for (int c = 0; c < 8; ++c) {
      // lattice index per axis: the child's octant bit plus the corner's
      const int ix = (k & 1) + (c & 1), iy = ((k >> 1) & 1) + ((c >> 1) & 1), iz = ((k >> 2) & 1) + ((c >> 2) & 1);
      const long long x = ix == 0 ? fam.cx[0] : ix == 1 ? fam.cx[1] : fam.cx[2];
      const long long y = iy == 0 ? fam.cy[0] : iy == 1 ? fam.cy[1] : fam.cy[2];
      const long long z = iz == 0 ? fam.cz[0] : iz == 1 ? fam.cz[1] : fam.cz[2];
      if (x >= 0 && y >= 0 && z >= 0) visit(x | y | z);
    }
  }
}

// The three points of one axis as bit sets `in` shifted by their low codes,
// those of equal high code (bits from 5 on) merged into the first: out[i] = 0
// where point i is merged into another or not interior.
__device__ __forceinline__ void merge_axis(unsigned in, const long long (&code)[3], unsigned (&out)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) out[i] = code[i] >= 0 ? in << (int)(code[i] & 31) : 0u;
#pragma unroll
  for (int i = 1; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < i; ++j)
      if (out[j] != 0u && out[i] != 0u && (code[j] >> 5) == (code[i] >> 5)) {
        out[j] |= out[i];
        out[i] = 0u;
      }
}

// used[block] = 1 for every block that holds a corner.
__global__ void k_block_mark(const int* __restrict__ nd_child, long long nf, const int4* __restrict__ nd_org, int full,
                             int bb, int* __restrict__ used) {
  launch_wait();
  Family fam;
  if (!load_family(nd_child, nd_org, nf, (long long)blockIdx.x * blockDim.x + threadIdx.x, full, fam)) return;
  long long last = -1;
  family_corners(fam, [&](long long code) {
    const long long b = code >> bb;
    if (b != last) used[b] = 1;
    last = b;
  });
}

// slot -> block (the inverse of the scan of used)
__global__ void k_block_list(long long nb, const int* __restrict__ used, const int* __restrict__ slot,
                             long long* __restrict__ blist) {
  launch_wait();
  const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nb && used[b]) blist[slot[b]] = b;
}

__global__ void k_corner_mark(const int* __restrict__ nd_child, long long nf, const int4* __restrict__ nd_org,
                              int full, int bb, const int* __restrict__ slot, unsigned* __restrict__ bits) {
  launch_wait();
  Family fam;
  if (!load_family(nd_child, nd_org, nf, (long long)blockIdx.x * blockDim.x + threadIdx.x, full, fam)) return;
  auto mark = [&](long long code, unsigned m) {  // code: of any point of the word
    const long long blk = slot ? (long long)slot[code >> bb] : code >> bb;
    atomicOr(bits + (blk << (bb - 5)) + ((code & ((1ll << bb) - 1)) >> 5), m);
  };
  if (fam.leaves != 0xff) {
    family_corners(fam, [&](long long code) { mark(code, 1u << (int)(code & 31)); });
    return;
  }
  unsigned mx[3];
  merge_axis(1u, fam.cx, mx);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (mx[i] == 0u) continue;
    unsigned my[3];
    merge_axis(mx[i], fam.cy, my);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (my[j] == 0u) continue;
      unsigned mz[3];
      merge_axis(my[j], fam.cz, mz);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (mz[k] != 0u) mark(fam.cx[i] | fam.cy[j] | fam.cz[k], mz[k]);
    }
  }
}

__global__ void k_bitmap_keys(const unsigned* __restrict__ bits, long long nw, const int* __restrict__ off, int bb,
                              const long long* __restrict__ blist, int B, uint64_t* __restrict__ out) {
  launch_wait();
  long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  unsigned b = bits[w];
  int o = off[w];
  const long long sl = w >> (bb - 5);
  const uint64_t base = ((uint64_t)(blist ? blist[sl] : sl) << bb) | ((uint64_t)(w & ((1LL << (bb - 5)) - 1)) << 5);
  while (b) {
    const int i = __ffs(b) - 1;
    b &= b - 1;
    const uint64_t idx = base | (uint64_t)i;
    const uint64_t x = compact3(idx) + 1, y = compact3(idx >> 1) + 1, z = compact3(idx >> 2) + 1;
    out[o++] = (x << (2 * B)) | (y << B) | z;
  }
}

__device__ __forceinline__ uint32_t mix64to32(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return (uint32_t)k;
}

// Deduplication by key with "first insertion wins" (Mesh::insert_vert /
// insert_tri, src/global.cpp:13-53): an open-addressing table of slot + 1
// per distinct key keeps the lowest slot (atomicMin), keys are compared
// through the slots' own key arrays.  The table has more entries than
// slots, so a probe always ends.
// An entry is lowered only where this slot is below what it holds (it never
// rises, so a stale read costs an atomic and nothing else): most of a key's six
// slots come after its first.  195 -> 168 us for the 12.9M slots of a 1M
// dam-break frame.  Homes that follow the leaf ids, so that neighbours share
// lines, were slower (212 us: the probes of near keys run into one another).
__global__ void k_vkey_insert(long long ns, const uint64_t* __restrict__ khi, const uint64_t* __restrict__ klo,
                              uint32_t mask, unsigned* __restrict__ tab, uint32_t* __restrict__ where) {
  launch_wait();
  long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ns) return;
  const uint64_t lo = klo[s], hi = khi ? khi[s] : 0ull;
  uint32_t h = mix64to32(lo ^ (hi * 0x9E3779B97F4A7C15ull)) & mask;
  for (uint32_t t = 0; t <= mask; ++t) {
    unsigned cur = tab[h];
    if (cur == 0u) {
      cur = atomicCAS(tab + h, 0u, (unsigned)s + 1u);
      if (cur == 0u) break;
    }
    const long long o = (long long)cur - 1;
    if (klo[o] == lo && (!khi || khi[o] == hi)) {
      if ((unsigned)s + 1u < cur) atomicMin(tab + h, (unsigned)s + 1u);  // the entry only ever falls
      break;
    }
    h = (h + 1u) & mask;
  }
  where[s] = h;
}

// Triangles: the sorted vertex triple of the oriented triangle is the key.
__device__ __forceinline__ void sorted3(const int* o, int& s0, int& s1, int& s2) {
  const int a = o[0], b = o[1], c = o[2];
  s0 = min(a, min(b, c));
  s2 = max(a, max(b, c));
  s1 = a + b + c - s0 - s2;
}

__global__ void k_tri_insert(long long nt, const int* __restrict__ otri, uint32_t mask, unsigned* __restrict__ tab,
                             uint32_t* __restrict__ where) {
  launch_wait();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  int s0, s1, s2;
  sorted3(otri + 3 * t, s0, s1, s2);
  // homes by the lowest vertex, whose triangles are near in the list: 109 us
  // scattered by a full mix, 91 us this way (4.3M triangles)
  uint32_t h = ((uint32_t)s0 * 4u + (mix64to32(((uint64_t)(uint32_t)s1 << 32) | (uint32_t)s2) & 3u)) & mask;
  for (uint32_t i = 0; i <= mask; ++i) {
    unsigned cur = tab[h];
    if (cur == 0u) {
      cur = atomicCAS(tab + h, 0u, (unsigned)t + 1u);
      if (cur == 0u) break;
    }
    int o0, o1, o2;
    sorted3(otri + 3 * ((long long)cur - 1), o0, o1, o2);
    if (o0 == s0 && o1 == s1 && o2 == s2) {
      if ((unsigned)t + 1u < cur) atomicMin(tab + h, (unsigned)t + 1u);
      break;
    }
    h = (h + 1u) & mask;
  }
  where[t] = h;
}

// flag[s] = 1 where slot s is its key's first (lowest) slot
__global__ void k_first_flag(long long n, const unsigned* __restrict__ tab, const uint32_t* __restrict__ where,
                             int* __restrict__ flag) {
  launch_wait();
  long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) flag[s] = tab[where[s]] == (unsigned)s + 1u ? 1 : 0;
  if (s == n) flag[s] = 0;
}

// The same as a scan input (a sequence the scan reads once).
struct FirstSlot {
  const unsigned* tab;
  const uint32_t* where;
  __device__ int operator()(long long i) const { return tab[where[i]] == (unsigned)i + 1u ? 1 : 0; }
  __device__ int4 four(long long i) const {
    return make_int4((*this)(i), (*this)(i + 1), (*this)(i + 2), (*this)(i + 3));
  }
};

// Ranks of the first slots among n: rank[n] and *total are their number.  The flags are
// worked out inside the scan while it reads them once; a longer scan reads its
// input twice, and the flags' random table reads are dearer than an array.
static void rank_first(long long n, const unsigned* tab, const uint32_t* where, int* rank, int* total, int* tmp,
                       cudaStream_t s) {
  if (n + 1 <= kScanOneLaunch) {
    exclusive_scan(ScanOf<FirstSlot>{{tab, where}, n}, rank, n + 1, total, tmp, s);
    return;
  }
  PI_LAUNCH(k_first_flag, div_up(n + 1, 256), 256, 0, s, n, tab, where, rank);
  exclusive_scan_i32(rank, rank, n + 1, total, tmp, s);
}

// slot -> vertex (numbered in order of first slots); vertex -> its first slot
__global__ void k_vertex_map(long long ns, const unsigned* __restrict__ tab, const uint32_t* __restrict__ where,
                             const int* __restrict__ rank, int* __restrict__ slot_vertex, int* __restrict__ rep) {
  launch_wait();
  long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ns) return;
  const long long first = (long long)tab[where[s]] - 1;
  const int v = rank[first];
  slot_vertex[s] = v;
  if (first == s) rep[v] = (int)s;
}

__global__ void k_tri_write(long long nt, const int* __restrict__ rank, const int* __restrict__ otri,
                            int* __restrict__ out) {
  launch_wait();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const int o = rank[t];
  if (rank[t + 1] == o) return;
  out[3 * o] = otri[3 * t];
  out[3 * o + 1] = otri[3 * t + 1];
  out[3 * o + 2] = otri[3 * t + 2];
}

__global__ void k_unique_flag(const uint64_t* __restrict__ keys, long long n, uint64_t invalid,
                              int* __restrict__ flag) {
  launch_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  if (i == n) {
    flag[i] = 0;
    return;
  }
  uint64_t k = keys[i];
  flag[i] = (k != invalid && (i == 0 || keys[i - 1] != k)) ? 1 : 0;
}

__global__ void k_unique_write(const uint64_t* __restrict__ keys, const int* __restrict__ scan, long long n,
                               uint64_t invalid, uint64_t* __restrict__ out) {
  launch_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t k = keys[i];
  if (k != invalid && (i == 0 || keys[i - 1] != k)) out[scan[i]] = k;
}

// One thread per dual vertex (a unique interior leaf corner): the eight leaves
// around it by descent from the root, then the DMC case.  Octant c of the corner
// is the lattice cell (x - 1 + bit), ..., and the child that holds a cell at
// depth d is bit D_max - 1 - d of its coordinates, so a step of the descent
// loads the child index alone: the nodes' origins, the other half of the loads
// and half of the instructions, are not needed (1M dam break, 5.8M corners:
// 336 -> 299 us; 187 with the table in plain loads).
__global__ void k_dual(const uint64_t* __restrict__ verts, long long nu, int B, const int* __restrict__ nd_child,
                       const float4* __restrict__ nd_v, int* __restrict__ cells,
                       uint8_t* __restrict__ procs, int* __restrict__ tcount, unsigned long long* __restrict__ ndual) {
  launch_wait();
  long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (u > nu) return;
  if (u == nu) {
    tcount[u] = 0;
    return;
  }
  const uint64_t key = verts[u];
  const uint64_t m = (1ull << B) - 1ull;
  const int x = (int)((key >> (2 * B)) & m), y = (int)((key >> B) & m), z = (int)(key & m);
  // x - 1 and x agree above the lowest set bit of x, so the eight cells share
  // the descent down to the highest of the three
  const int split = 31 - __clz((x & -x) | (y & -y) | (z & -z));
  int bit = B - 2;  // D_max - 1
  int start = 0;
  for (; bit > split; --bit) {
    const int ch = nd_child[start];
    if (ch < 0) break;
    start = ch + (((x >> bit) & 1) | (((y >> bit) & 1) << 1) | (((z >> bit) & 1) << 2));
  }
  // the eight descents below `start` advance in lockstep, so that their
  // loads are in flight together rather than one chain after another
  int n8[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) n8[c] = start;
  for (; bit >= 0; --bit) {
    int ch[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) ch[c] = nd_child[n8[c]];
    const int bx0 = ((x - 1) >> bit) & 1, by0 = (((y - 1) >> bit) & 1) << 1, bz0 = (((z - 1) >> bit) & 1) << 2;
    const int bx1 = (x >> bit) & 1, by1 = ((y >> bit) & 1) << 1, bz1 = ((z >> bit) & 1) << 2;
    bool more = false;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (ch[c] >= 0) {
        n8[c] = ch[c] + (((c & 1) ? bx1 : bx0) | ((c & 2) ? by1 : by0) | ((c & 4) ? bz1 : bz0));
        more = true;
      }
    if (!more) break;
  }
  int index = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c)
    if (nd_v[n8[c]].w > 0.f) index |= 1 << c;
  const unsigned cs = __ldg(d_case + index);
  if (cs & kCaseMixed) {
    int4* const out = reinterpret_cast<int4*>(cells + 8 * u);
    out[0] = make_int4(n8[0], n8[1], n8[2], n8[3]);
    out[1] = make_int4(n8[4], n8[5], n8[6], n8[7]);
    stripe_add(ndual, C_DUAL, 1ull);
  }
  procs[u] = (uint8_t)index;
  tcount[u] = (cs & kCaseMixed) ? case_triangles(cs) : 0;
}

// Triangle slots: the two leaves each triangle corner bisects and their sorted
// id pair.  The slots of a block's dual vertices are one run, so a thread takes
// every kSlotThreads-th slot of it, finds its dual vertex in the block's offsets,
// and the stores of a warp are contiguous (a thread per dual vertex stored up to
// 15 slots of its own, a line each: 160 us at 1M, 109 this way).
constexpr int kSlotThreads = 256;
__global__ void __launch_bounds__(kSlotThreads) k_tri_slots(long long nu, const int* __restrict__ cells,
                                                            const uint8_t* __restrict__ procs,
                                                            const int* __restrict__ toff,
                                                            const uint64_t* __restrict__ nd_id, int id_bits, int packed,
                                                            int* __restrict__ slotA, int* __restrict__ slotB,
                                                            uint64_t* __restrict__ khi, uint64_t* __restrict__ klo,
                                                            int8_t* __restrict__ tflip) {
  launch_wait();
  __shared__ int s_off[kSlotThreads + 1];
  const long long u0 = (long long)blockIdx.x * kSlotThreads;
  const int nloc = (int)(nu - u0 < kSlotThreads ? nu - u0 : kSlotThreads);
  for (int i = threadIdx.x; i <= kSlotThreads; i += kSlotThreads) s_off[i] = toff[u0 + min(i, nloc)];
  __syncthreads();
  const int first = s_off[0], total = 3 * (s_off[kSlotThreads] - first);
  for (int q = threadIdx.x; q < total; q += kSlotThreads) {
    const int t = first + q / 3, k = q % 3;
    int i = 0;  // the last vertex whose triangles start at or before t
#pragma unroll
    for (int o = kSlotThreads / 2; o > 0; o >>= 1)
      if (s_off[i + o] <= t) i += o;
    const long long u = u0 + i;
    const int index = procs[u];
    const unsigned cs = __ldg(d_case + index);
    const int e = (int)(__ldg(d_edges + index) >> (4 * (3 * (t - s_off[i]) + k))) & 15;
    int c0, c1;
    edge_corners(e, &c0, &c1);
    const int A = __ldg(cells + 8 * u + case_corner(cs, c0)), Bn = __ldg(cells + 8 * u + case_corner(cs, c1));
    const long long s = 3ll * first + q;
    slotA[s] = A;
    slotB[s] = Bn;
    const uint64_t ia = __ldg(nd_id + A), ib = __ldg(nd_id + Bn);
    const uint64_t lo = ia < ib ? ia : ib, hi = ia < ib ? ib : ia;
    if (packed) {
      klo[s] = (lo << id_bits) | hi;
    } else {
      khi[s] = lo;
      klo[s] = hi;
    }
    if (k == 0) tflip[t] = (cs & kCaseFlip) ? 1 : 0;
  }
}

struct BisectArgs {
  GridView g;  // the hash grid (constant radius); with a variable radius the grid the vertices are bucketed by
  PartView P;
  float iso;
  float rr;  // r / 2 (variable radius: the searcher's minimum radius / 2)
  const MultiGridView* mg;  // variable radius: the bins' grids, else null
};

// Vertices listed by the hash cell of their first bisection midpoint (count
// per cell, scan, place), so that neighbouring threads of k_bisect walk the
// same cells.  Order within a cell is arbitrary: each vertex's result
// depends on its own edge only.
__device__ __forceinline__ int vertex_cell(const BisectArgs& a, const float4& p, const float4& q, int ekx,
                                           int eky) {
  const float mx = __fmul_rn(__fadd_rn(p.x, q.x), 0.5f);
  const float my = __fmul_rn(__fadd_rn(p.y, q.y), 0.5f);
  const float mz = __fmul_rn(__fadd_rn(p.z, q.z), 0.5f);
  int cx, cy, cz;
  cell_of(a.g, mx, my, mz, cx, cy, cz);
  return ((cz + 2) * eky + (cy + 2)) * ekx + (cx + 2);
}

__global__ void k_vcell_count(BisectArgs a, long long nv, const int* __restrict__ rep, const int* __restrict__ slotA,
                              const int* __restrict__ slotB, const float4* __restrict__ nd_v, int ekx, int eky,
                              int* __restrict__ cnt, int* __restrict__ key) {
  launch_wait();
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int k = -1;
  if (v < nv) {
    const int s = rep[v];
    k = vertex_cell(a, nd_v[slotA[s]], nd_v[slotB[s]], ekx, eky);
  }
  const unsigned peers = __match_any_sync(0xffffffffu, k);
  if (k >= 0 && lane == __ffs(peers) - 1) atomicAdd(cnt + k, __popc(peers));
  if (v < nv) key[v] = k;
}

__global__ void k_vcell_place(long long nv, const int* __restrict__ key, const int* __restrict__ off,
                              int* __restrict__ fill, int* __restrict__ list) {
  launch_wait();
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int k = v < nv ? key[v] : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, k);
  if (k < 0) return;
  const int leader = __ffs(peers) - 1;
  int b = 0;
  if (lane == leader) b = atomicAdd(fill + k, __popc(peers));
  b = __shfl_sync(peers, b, leader);
  list[off[k] + b + __popc(peers & ((1u << lane) - 1u))] = (int)v;
}

template <bool VR>
__global__ void __launch_bounds__(128, 8) k_bisect(BisectArgs a, long long nv, int per_warp, const int* __restrict__ order, const int* __restrict__ rep,
                         const int* __restrict__ slotA,
                         const int* __restrict__ slotB, const float4* __restrict__ nd_v,
                         const uint64_t* __restrict__ nd_id, float* __restrict__ out,
                         uint64_t* __restrict__ vkeys, int2* __restrict__ vedge,
                         unsigned long long* __restrict__ counters) {
  launch_wait();
  __shared__ __align__(16) float s_stage[VR ? 1 : kGroupWarps][VR ? 1 : GroupRoom<32>::kFloats];
  const int lane = threadIdx.x & 31;
  const long long t = ((long long)blockIdx.x * kGroupWarps + (threadIdx.x >> 5)) * per_warp + lane;
  const bool valid = lane < per_warp && t < nv;
  long long v = 0;
  int A = 0, B = 0;
  float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
  if (valid) {
    v = order[t];
    const int s = rep[v];
    A = slotA[s], B = slotB[s];
    p = nd_v[A], q = nd_v[B];
  }
  const float dx = __fsub_rn(p.x, q.x), dy = __fsub_rn(p.y, q.y), dz = __fsub_rn(p.z, q.z);
  float d = __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fadd_rn(__fmul_rn(dy, dy), __fmul_rn(dz, dz))));
  long long pairs = 0;
  int steps = 0;
  // a warp steps until its last edge is short enough
  for (int it = 0; it < 64; ++it) {
    const bool go = d > a.rr;
    if (!__any_sync(0xffffffffu, go)) break;
    float4 m;
    m.x = __fmul_rn(__fadd_rn(p.x, q.x), 0.5f);
    m.y = __fmul_rn(__fadd_rn(p.y, q.y), 0.5f);
    m.z = __fmul_rn(__fadd_rn(p.z, q.z), 0.5f);
    if (VR) {
      m.w = go ? a.iso - field_sum_vr(*a.mg, a.P, m.x, m.y, m.z, &pairs) : 0.f;
    } else {
      m.w = a.iso - group_field<32>(a.g, a.P, m.x, m.y, m.z, go, s_stage[VR ? 0 : threadIdx.x >> 5], pairs);
    }
    if (go) {
      if ((m.w > 0.f) == (p.w > 0.f))
        p = m;
      else
        q = m;
      d = __fmul_rn(d, 0.5f);
      ++steps;
    }
  }
  // group_field books a window's pairs on the lanes that hold its rows, whether
  // they have a vertex or not: summed over the warp before those without leave
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    steps += __shfl_xor_sync(0xffffffffu, steps, o);
  }
  if (lane == 0 && steps > 0) {
    stripe_add(counters, C_BISECT_EVALS, (unsigned long long)steps);
    stripe_add(counters, C_BISECT_PAIRS, (unsigned long long)pairs);
  }
  if (!valid) return;
  vedge[v] = make_int2(A, B);
  const float ratio = __fdiv_rn(__fsub_rn(0.0f, p.w), __fsub_rn(q.w, p.w));
  float3 r;
  if (ratio < kAbove01) {  // (double)ratio < 0.1
    r = make_float3(p.x, p.y, p.z);
  } else if (ratio > kBelow09) {  // (double)ratio > 0.9
    r = make_float3(q.x, q.y, q.z);
  } else {
    r.x = __fadd_rn(p.x, __fmul_rn(__fsub_rn(q.x, p.x), ratio));
    r.y = __fadd_rn(p.y, __fmul_rn(__fsub_rn(q.y, p.y), ratio));
    r.z = __fadd_rn(p.z, __fmul_rn(__fsub_rn(q.z, p.z), ratio));
  }
  out[3 * v] = r.x;
  out[3 * v + 1] = r.y;
  out[3 * v + 2] = r.z;
  uint64_t ia = nd_id[A], ib = nd_id[B];
  vkeys[2 * v] = ia < ib ? ia : ib;
  vkeys[2 * v + 1] = ia < ib ? ib : ia;
}

// Oriented triangle in Mesh::insert_tri argument order.
__global__ void k_tri_orient(long long nt, const int* __restrict__ slot_vertex, const int8_t* __restrict__ tflip,
                             int* __restrict__ otri) {
  launch_wait();
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const int a = slot_vertex[3 * t], b = slot_vertex[3 * t + 1], c = slot_vertex[3 * t + 2];
  otri[3 * t] = tflip[t] ? a : c;
  otri[3 * t + 1] = b;
  otri[3 * t + 2] = tflip[t] ? c : a;
}

// Mask of the smallest power-of-two table with more than n entries.
static uint32_t table_mask(long long n) {
  uint32_t m = 1;
  while ((long long)m < n + 1) m <<= 1;
  return m - 1;
}

// A count the host waits for on stream st: a scan stores its total in a pinned
// word, an event follows it, and the caller may queue work that does not need
// the count before it waits for the event (no copy, no stream-wide wait).
struct CountReader {
  pi_frame* f;
  cudaStream_t st;
  int off;
  cudaEvent_t ev;
  int* word() const { return reinterpret_cast<int*>(f->ctx->hpin + off); }
  void stored() const { PI_CUDA(cudaEventRecord(ev, st)); }
  int wait() const {
    PI_CUDA(cudaEventSynchronize(ev));
    return *const_cast<const volatile int*>(word());
  }
};

// Steps 1-2 of the extraction, the mesh topology: it reads only the tree
// (nd_child, nd_org of the f->nNodes nodes), not the leaves' values.  Sets
// f->nLeaves, f->tp_uverts (the unique interior leaf corners as lattice
// keys, in Z order) and f->tp_nu.
static void extract_topology(pi_frame* f, cudaStream_t s, const CountReader& rd) {
  pi_ctx* c = f->ctx;
  const long long nn = f->nNodes;
  // 1. leaves: every INTERNAL node has eight children, so the counts follow
  const long long nf = (nn - 1) / 8;  // families
  f->nLeaves = nn - nf;
  DBuf<int> tmp;
  // 2. dual vertices = unique interior leaf corners
  const int B = f->dmax + 1;
  const int full = 1 << f->dmax;
  DBuf<uint64_t>& uverts = f->tp_uverts;
  long long nu = 0;
  // block size: 2^bb Morton codes, bb a multiple of 3 and at least 15 (32^3
  // points, 1024 words), so that at most 2^24 blocks cover the lattice; past
  // 2^18 codes a block (D_max > 14) the blocks grow too large and the corners
  // are sorted instead (below)
  const int bb = std::max(15, ((3 * f->dmax - 24 + 2) / 3) * 3);
  if (bb <= 18) {
    const long long nb = 1LL << std::max(0, 3 * f->dmax - bb);
    // up to 2^27 bits (16 MB) clearing and scanning the whole bitmap costs less
    // than the launches and the read that find the used blocks (40 us at D_max 9
    // against 60); at 2^30 bits it cost 230 us of a 1.7M-particle frame, the blocks 110
    const bool dense = f->dmax <= 9;
    long long nused = nb;
    DBuf<int> used, slot;
    DBuf<long long> blist;
    if (!dense) {
      used.alloc(c, s, nb + 1);
      if (tmp.n < scan_tmp_ints(nb + 1)) tmp.alloc(c, s, scan_tmp_ints(nb + 1));
      PI_CUDA(cudaMemsetAsync(used.p, 0, sizeof(int) * (nb + 1), s));
      PI_LAUNCH(k_block_mark, div_up(nf, 128), 128, 0, s, f->nd_child.p, nf, f->nd_org.p, full, bb, used.p);
      slot.alloc(c, s, nb + 1);
      exclusive_scan_i32(used.p, slot.p, nb + 1, rd.word(), tmp.p, s);
      rd.stored();
      nused = rd.wait();
      blist.alloc(c, s, nused > 0 ? nused : 1);
      PI_LAUNCH(k_block_list, div_up(nb, 256), 256, 0, s, nb, used.p, slot.p, blist.p);
    }
    const long long nw = nused << (bb - 5);
    DBuf<unsigned> bits;
    DBuf<int> cnt;
    bits.alloc(c, s, nw > 0 ? nw : 1);
    cnt.alloc(c, s, nw + 1);
    if (tmp.n < scan_tmp_ints(nw + 1)) tmp.alloc(c, s, scan_tmp_ints(nw + 1));
    PI_CUDA(cudaMemsetAsync(bits.p, 0, sizeof(unsigned) * (nw > 0 ? nw : 1), s));
    PI_LAUNCH(k_corner_mark, div_up(nf, 128), 128, 0, s, f->nd_child.p, nf, f->nd_org.p, full, bb,
              dense ? nullptr : slot.p, bits.p);
    exclusive_scan(ScanOf<WordBits>{{bits.p}, nw}, cnt.p, nw + 1, rd.word(), tmp.p, s);
    rd.stored();
    nu = rd.wait();
    if (uverts.n < (size_t)(nu > 0 ? nu : 1)) uverts.alloc(c, s, nu > 0 ? nu : 1);
    PI_LAUNCH(k_bitmap_keys, div_up(nw, 256), 256, 0, s, bits.p, nw, cnt.p, bb, dense ? nullptr : blist.p, B,
              uverts.p);
  } else {
    const long long nk = nf * 27;
    const uint64_t invalid = (1ull << (3 * B)) - 1ull;
    DBuf<uint64_t> keys, keys2;
    DBuf<uint32_t> vals, vals2;
    keys.alloc(c, s, nk);
    keys2.alloc(c, s, nk);
    vals.alloc(c, s, nk);
    vals2.alloc(c, s, nk);
    PI_LAUNCH(k_corner_keys, div_up(nk, 256), 256, 0, s, f->nd_child.p, nf, f->nd_org.p, full, B, keys.p, vals.p);
    DBuf<int> rtmp;
    rtmp.alloc(c, s, radix_tmp_ints(nk));
    uint64_t *kp = keys.p, *ka = keys2.p;
    uint32_t *vp = vals.p, *va = vals2.p;
    radix_sort_u64(&kp, &vp, &ka, &va, nk, 3 * B, rtmp.p, s);
    DBuf<int> uf;
    uf.alloc(c, s, nk + 1);
    tmp.alloc(c, s, scan_tmp_ints(nk + 1));
    PI_LAUNCH(k_unique_flag, div_up(nk + 1, 256), 256, 0, s, kp, nk, invalid, uf.p);
    exclusive_scan_i32(uf.p, uf.p, nk + 1, rd.word(), tmp.p, s);
    rd.stored();
    nu = rd.wait();
    if (uverts.n < (size_t)(nu > 0 ? nu : 1)) uverts.alloc(c, s, nu > 0 ? nu : 1);
    PI_LAUNCH(k_unique_write, div_up(nk, 256), 256, 0, s, kp, uf.p, nk, invalid, uverts.p);
  }
  f->tp_nu = nu;
}

void topology_start(pi_frame* f) {
  pi_ctx* c = f->ctx;
  cudaStream_t ts = c->topo_stream;
  PI_CUDA(cudaStreamWaitEvent(ts, c->ev_topo_in, 0));
  f->tp_inflight = true;
  try {
    extract_topology(f, ts, CountReader{f, ts, kPinTopoReadOffset, c->ev_topo_read});
  } catch (...) {
    cudaEventRecord(c->ev_topo_done, ts);  // what was launched is joined all the same
    throw;
  }
  PI_CUDA(cudaEventRecord(c->ev_topo_done, ts));
}

void topology_join(pi_frame* f) {
  if (!f->tp_inflight) return;
  PI_CUDA(cudaStreamWaitEvent(f->ctx->stream, f->ctx->ev_topo_done, 0));
  f->tp_inflight = false;
}

void topology_fence(pi_frame* f) {
  topology_join(f);
  pi_ctx* c = f->ctx;
  PI_CUDA(cudaEventRecord(c->ev_topo_in, c->stream));
  PI_CUDA(cudaStreamWaitEvent(c->topo_stream, c->ev_topo_in, 0));
}

void stage_extract(pi_frame* f) {
  pi_ctx* c = f->ctx;
  cudaStream_t s = c->stream;
  upload_tables(c->device);
  // steps 1-2: the topology, started beside the octree's last level or run
  // here
  if (f->tp_inflight)
    topology_join(f);
  else
    extract_topology(f, s, CountReader{f, s, kPinReadOffset, c->ev_read});
  const int B = f->dmax + 1;
  const long long nu = f->tp_nu;
  const uint64_t* const uverts = f->tp_uverts.p;
  DBuf<int> tmp;
  tmp.alloc(c, s, scan_tmp_ints(nu + 1));
  // 3. dual cells
  DBuf<int> cells, toff;
  DBuf<int8_t> procs;
  cells.alloc(c, s, nu * 8 > 0 ? nu * 8 : 1);
  procs.alloc(c, s, nu > 0 ? nu : 1);
  toff.alloc(c, s, nu + 1);
  if (tmp.n < scan_tmp_ints(nu + 1)) tmp.alloc(c, s, scan_tmp_ints(nu + 1));
  const CountReader rd{f, s, kPinReadOffset, c->ev_read};
  // k_dual reads the leaves' values: the octree's last QEF level, if it was
  // left running, ends here
  qef_join(f);
  counters_begin(f, &f->extract_counted, C_DUAL, C_BISECT_PAIRS);
  PI_LAUNCH(k_dual, div_up(nu + 1, 128), 128, 0, s, uverts, nu, B, f->nd_child.p, f->nd_v.p,
            cells.p, reinterpret_cast<uint8_t*>(procs.p), toff.p, f->dcount.p);
  exclusive_scan_i32(toff.p, toff.p, nu + 1, rd.word(), tmp.p, s);
  rd.stored();
  const long long nt0 = rd.wait();
  // 4. triangle slots and vertex keys (sorted leaf-id pairs)
  const int id_bits = 3 * f->dmax;
  const int packed = (2 * id_bits <= 64) ? 1 : 0;
  const long long ns = 3 * nt0;
  DBuf<int> slotA, slotB;
  DBuf<uint64_t> khi, klo;
  DBuf<int8_t> tflip;
  slotA.alloc(c, s, ns > 0 ? ns : 1);
  slotB.alloc(c, s, ns > 0 ? ns : 1);
  klo.alloc(c, s, ns > 0 ? ns : 1);
  if (!packed) khi.alloc(c, s, ns > 0 ? ns : 1);
  tflip.alloc(c, s, nt0 > 0 ? nt0 : 1);
  PI_LAUNCH(k_tri_slots, div_up(nu, kSlotThreads), kSlotThreads, 0, s, nu, cells.p,
            reinterpret_cast<const uint8_t*>(procs.p), toff.p, f->nd_id.p, id_bits, packed, slotA.p, slotB.p, khi.p,
            klo.p, tflip.p);
  cells.release();
  procs.release();
  toff.release();
  // 5. unique mesh vertices: first slot of each key, numbered in slot order
  DBuf<unsigned> vtab;
  DBuf<uint32_t> vwhere;
  DBuf<int> vrank, slot_vertex, rep;
  const uint32_t vmask = table_mask(ns);
  vtab.alloc(c, s, (size_t)vmask + 1);
  vwhere.alloc(c, s, ns > 0 ? ns : 1);
  vrank.alloc(c, s, ns + 1);
  if (tmp.n < scan_tmp_ints(ns + 1)) tmp.alloc(c, s, scan_tmp_ints(ns + 1));
  PI_CUDA(cudaMemsetAsync(vtab.p, 0, sizeof(unsigned) * ((size_t)vmask + 1), s));
  PI_LAUNCH(k_vkey_insert, div_up(ns, 256), 256, 0, s, ns, packed ? nullptr : khi.p, klo.p, vmask, vtab.p,
            vwhere.p);
  rank_first(ns, vtab.p, vwhere.p, vrank.p, rd.word(), tmp.p, s);
  rd.stored();
  slot_vertex.alloc(c, s, ns > 0 ? ns : 1);
  rep.alloc(c, s, ns > 0 ? ns : 1);  // room for a vertex per slot
  PI_LAUNCH(k_vertex_map, div_up(ns, 256), 256, 0, s, ns, vtab.p, vwhere.p, vrank.p, slot_vertex.p, rep.p);
  const long long nv = rd.wait();
  vtab.release();
  vwhere.release();
  vrank.release();
  khi.release();
  klo.release();
  // 6. triangles: first of each sorted vertex triple, in generation order
  // (they need the vertex numbering, not the positions, so they come before
  // the bisection and, for a host destination, their copy overlaps it)
  DBuf<int> otri, trank;
  DBuf<unsigned> ttab;
  DBuf<uint32_t> twhere;
  otri.alloc(c, s, nt0 * 3 > 0 ? nt0 * 3 : 3);
  PI_LAUNCH(k_tri_orient, div_up(nt0, 256), 256, 0, s, nt0, slot_vertex.p, tflip.p, otri.p);
  // nearly every triangle is distinct, so the table gets twice as many
  // entries as triangles (load at most 1/2; linear probing degrades fast
  // above that)
  const uint32_t tmask = table_mask(2 * nt0);
  ttab.alloc(c, s, (size_t)tmask + 1);
  twhere.alloc(c, s, nt0 > 0 ? nt0 : 1);
  trank.alloc(c, s, nt0 + 1);
  PI_CUDA(cudaMemsetAsync(ttab.p, 0, sizeof(unsigned) * ((size_t)tmask + 1), s));
  PI_LAUNCH(k_tri_insert, div_up(nt0, 256), 256, 0, s, nt0, otri.p, tmask, ttab.p, twhere.p);
  rank_first(nt0, ttab.p, twhere.p, trank.p, rd.word(), tmp.p, s);
  rd.stored();
  // room for every generated triangle and the splash icosahedra
  const long long nsp = f->P.splash ? f->nSplash : 0;
  const long long tcap = (nt0 + 20 * nsp) * 3;
  f->mt.alloc(c, s, tcap > 0 ? tcap : 3);
  PI_LAUNCH(k_tri_write, div_up(nt0, 256), 256, 0, s, nt0, trank.p, otri.p, f->mt.p);
  f->mv.alloc(c, s, (nv + 12 * nsp) * 3 > 0 ? (nv + 12 * nsp) * 3 : 3);
  f->mk.alloc(c, s, (nv + 12 * nsp) * 2 > 0 ? (nv + 12 * nsp) * 2 : 2);
  f->vedge.alloc(c, s, nv + 12 * nsp > 0 ? nv + 12 * nsp : 1);
  if (nsp > 0) PI_CUDA(cudaMemsetAsync(f->vedge.p + nv, 0xff, sizeof(int2) * 12 * nsp, s));
  const long long nt = rd.wait();
  // splash icosahedra after the surface (Mesh::AppendSplash_ConstR runs
  // after generate_mesh, src/surface_reconstructor.cpp:299-320)
  if (nsp > 0) splash_mesh(f, nv, nt);
  f->nT = nt + 20 * nsp;
  if (f->host_tris && f->nT > 0 && f->nT <= f->host_tcap) {
    PI_CUDA(cudaEventRecord(c->ev_tris_ready, s));
    PI_CUDA(cudaStreamWaitEvent(c->copy_stream, c->ev_tris_ready, 0));
    PI_CUDA(cudaMemcpyAsync(f->host_tris, f->mt.p, sizeof(int) * 3 * f->nT, cudaMemcpyDeviceToHost,
                            c->copy_stream));
    PI_CUDA(cudaEventRecord(c->ev_tris_copied, c->copy_stream));
    f->tris_sent = true;
  }
  // 7. vertex positions by bisection (the splash vertices follow them)
  f->nV = nv + 12 * nsp;
  const GridHost& gh = f->g;
  BisectArgs ba{GridView{gh.bounding[0], gh.bounding[2], gh.bounding[4], gh.cell, gh.nx, gh.ny, gh.nz, f->off.p},
                PartView{f->pos.p, f->xm.p, f->ga.p, f->gb.p, f->xlo.p}, f->iso, f->P.radius / 2, nullptr};
  if (f->varR) {
    // bucket the vertices by a grid over the root box; bisect down to half the
    // searcher's minimum radius (src/visitorextract.cpp:54)
    float bcell;
    const int bn = vr_bucket_grid(f, &bcell);
    ba.g = GridView{f->rootC[0] - f->rootH, f->rootC[1] - f->rootH, f->rootC[2] - f->rootH, bcell, bn, bn, bn, nullptr};
    ba.rr = f->vrMinR / 2;
    ba.mg = f->mgv.p;
  }
  {
    const int ekx = ba.g.nx + 4, eky = ba.g.ny + 4;
    const long long nc = (long long)ekx * eky * (ba.g.nz + 4);
    DBuf<int> vcnt, vfill, vkey, vorder;
    vcnt.alloc(c, s, nc + 1);
    vfill.alloc(c, s, nc);
    vkey.alloc(c, s, nv > 0 ? nv : 1);
    vorder.alloc(c, s, nv > 0 ? nv : 1);
    if (tmp.n < scan_tmp_ints(nc + 1)) tmp.alloc(c, s, scan_tmp_ints(nc + 1));
    PI_CUDA(cudaMemsetAsync(vcnt.p, 0, sizeof(int) * (nc + 1), s));
    PI_CUDA(cudaMemsetAsync(vfill.p, 0, sizeof(int) * nc, s));
    PI_LAUNCH(k_vcell_count, div_up(nv, 256), 256, 0, s, ba, nv, rep.p, slotA.p, slotB.p, f->nd_v.p, ekx, eky,
              vcnt.p, vkey.p);
    exclusive_scan_i32(vcnt.p, vcnt.p, nc + 1, nullptr, tmp.p, s);
    PI_LAUNCH(k_vcell_place, div_up(nv, 256), 256, 0, s, nv, vkey.p, vcnt.p, vfill.p, vorder.p);
    // vertices per warp: all its lanes filter the candidates of the vertices it
    // holds, so fewer of them shorten a warp's chain; halved while that leaves a
    // handful of warps per SM (5,000 vertices: 69 us with 32, 46 with 4)
    int per_warp = 32;
    while (!f->varR && per_warp > 4 && nv < 8LL * c->smCount * per_warp) per_warp /= 2;
    prof_begin(c, s, PG_BISECT);
    if (f->varR)
      PI_LAUNCH(k_bisect<true>, div_up(nv, 128), 128, 0, s, ba, nv, per_warp, vorder.p, rep.p, slotA.p, slotB.p, f->nd_v.p,
                f->nd_id.p, f->mv.p, f->mk.p, f->vedge.p, f->dcount.p);
    else
      PI_LAUNCH(k_bisect<false>, div_up(nv, per_warp * kGroupWarps), 32 * kGroupWarps, 0, s, ba, nv, per_warp, vorder.p, rep.p, slotA.p, slotB.p, f->nd_v.p,
                f->nd_id.p, f->mv.p, f->mk.p, f->vedge.p, f->dcount.p);
    prof_end(c, s, PG_BISECT);
  }
  counters_snapshot(f, kPinExtract);
}

}  // namespace pisurf
