// Warp-cooperative field evaluation for a chunk of query points that share
// one hash cell, hence one 27-cell candidate list (Evaluator::SingleEval,
// src/evaluator.cpp:60-87).  Lane l holds points l, l + 32, ... (K per lane).
//
// The warp tests 32 candidates at a time against the chunk's bounding box: a
// candidate whose support radius R (|G d| < 2h needs |d| < R, stored as
// R^2 * 1.002 in xm.w) does not reach the box contributes to no point.
// Survivors' records are staged in shared memory in candidate order and every
// lane walks them, so each point's compensated sum sees the in-support terms
// in candidate order (the same terms and order as field_sum).
#pragma once
#include "device.cuh"

namespace pisurf {

constexpr int kCandBuf = 96;  // staged candidate records per warp (default; k_q_eval tunes it)

// Order-preserving map of a float onto a signed int (for warp min / max).
__device__ __forceinline__ int fkey(float v) {
  const int i = __float_as_int(v);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float fkey_inv(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7fffffff); }

// 16-byte asynchronous copy global -> shared (cp.async, no register
// staging); completed by cp_async_wait_all before the records are read.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Per-warp staging buffer (shared memory): the staged candidates' records,
// one array of CB floats per component (structure of arrays), so that a
// component of two consecutive candidates is one 8-byte load feeding the
// packed FP32 instructions below.
enum : int {
  SC_X, SC_Y, SC_Z,        // centre, high part (xm)
  SC_LX, SC_LY, SC_LZ,     // centre, low part (xlo)
  SC_A0, SC_A1, SC_A2, SC_A3,  // A = G / h: a00 a01 a02 a11
  SC_B0, SC_B1, SC_B2,     // a12 a22 det * Sigma
  kStageComps
};
__host__ __device__ constexpr int stage_floats(int cb) { return kStageComps * cb; }  // per warp
constexpr int kStageFloats = stage_floats(kCandBuf);

struct ChunkStage {
  float* c;  // c[k * CB + t]: component k of staged candidate t
};

// 4-byte asynchronous copy global -> shared.
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

template <int CB>
__device__ __forceinline__ float2 ld_pair(const ChunkStage& st, int k, int t) {
  return *reinterpret_cast<const float2*>(st.c + k * CB + t);
}

// The staged candidates [0, nc) against the lane's K points: two consecutive
// candidates per step with Blackwell's packed FP32 instructions, each term
// added to the point's compensated sum (s, c) in candidate order.
template <int K, int CB>
__device__ __forceinline__ void eval_staged(const ChunkStage& st, int nc, const float2 (&QX)[K], const float2 (&QY)[K],
                                            const float2 (&QZ)[K], const bool (&slots)[K], float (&s)[K],
                                            float (&c)[K]) {
  const float2 M1 = make_float2(-1.0f, -1.0f);
  auto kahan = [&](int m, float term) {
    const float y = __fsub_rn(term, c[m]);
    const float tt = __fadd_rn(s[m], y);
    c[m] = __fsub_rn(__fsub_rn(tt, s[m]), y);
    s[m] = tt;
  };
#pragma unroll 1
  for (int t = 0; t < nc; t += 2) {
    const bool two = t + 1 < nc;  // warp-uniform: a second candidate in this pair
    const float2 X = ld_pair<CB>(st, SC_X, t), Y = ld_pair<CB>(st, SC_Y, t), Z = ld_pair<CB>(st, SC_Z, t);
    const float2 LX = ld_pair<CB>(st, SC_LX, t), LY = ld_pair<CB>(st, SC_LY, t), LZ = ld_pair<CB>(st, SC_LZ, t);
    const float2 A0 = ld_pair<CB>(st, SC_A0, t), A1 = ld_pair<CB>(st, SC_A1, t), A2 = ld_pair<CB>(st, SC_A2, t),
                 A3 = ld_pair<CB>(st, SC_A3, t);
    const float2 B0 = ld_pair<CB>(st, SC_B0, t), B1 = ld_pair<CB>(st, SC_B1, t), B2 = ld_pair<CB>(st, SC_B2, t);
#pragma unroll
    for (int m = 0; m < K; ++m) {
      if (!slots[m]) continue;  // warp-uniform
      // d = (q - x) - lo
      const float2 dx = __ffma2_rn(LX, M1, __ffma2_rn(X, M1, QX[m]));
      const float2 dy = __ffma2_rn(LY, M1, __ffma2_rn(Y, M1, QY[m]));
      const float2 dz = __ffma2_rn(LZ, M1, __ffma2_rn(Z, M1, QZ[m]));
      // u = A d (amul), s2 = |u|^2
      const float2 u0 = __ffma2_rn(A0, dx, __ffma2_rn(A1, dy, __fmul2_rn(A2, dz)));
      const float2 u1 = __ffma2_rn(A1, dx, __ffma2_rn(A3, dy, __fmul2_rn(B0, dz)));
      const float2 u2 = __ffma2_rn(A2, dx, __ffma2_rn(B0, dy, __fmul2_rn(B1, dz)));
      const float2 s2 = __ffma2_rn(u0, u0, __ffma2_rn(u1, u1, __fmul2_rn(u2, u2)));
      const bool in0 = s2.x < 4.0f, in1 = two && s2.y < 4.0f;
      if (in0 || in1) {
        // bspline_s2 on both: q = s2 / sqrt(s2), b1 = 1 + s2 (0.75 q - 1.5),
        // b2 = 0.25 (2 - q)^3, q <= 1 ? b1 : b2
        const float2 r = make_float2(rsqrtf(fmaxf(s2.x, 1e-30f)), rsqrtf(fmaxf(s2.y, 1e-30f)));
        const float2 q = __fmul2_rn(s2, r);
        const float2 b1 = __ffma2_rn(s2, __ffma2_rn(make_float2(0.75f, 0.75f), q, make_float2(-1.5f, -1.5f)),
                                     make_float2(1.0f, 1.0f));
        const float2 tq = __ffma2_rn(q, M1, make_float2(2.0f, 2.0f));
        const float2 b2 = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(0.25f, 0.25f), tq), tq), tq);
        const float2 term = __fmul2_rn(B2, make_float2(q.x <= 1.0f ? b1.x : b2.x, q.y <= 1.0f ? b1.y : b2.y));
        if (in0) kahan(m, term.x);
        if (in1) kahan(m, term.y);
      }
    }
  }
}

// The 27-cell candidates of a cell as one run of `total` places: the nine rows
// one after the other.  Lane r < 9 holds row r's range, so their offsets load
// together, and a batch of 32 candidates spans rows: a row holds 5 of the 49
// candidates of a dam-break frame's points, and row by row the filter ran nine
// batches of five lanes where two full ones do.  (1M frame, level D_max - 1:
// 712 -> 555 us; uniform grid of 150k particles 527 -> 450 us.)
struct CandidateRun {
  int total;
  int incl;   // places up to and with this lane's row
  int shift;  // place t of this lane's row is particle t + shift
  __device__ __forceinline__ CandidateRun(const GridView& g, int cx, int cy, int cz) {
    const int lane = threadIdx.x & 31;
    int s = 0, e = 0;
    if (lane >= 9 || !nb_row(g, cx, cy + lane % 3 - 1, cz + lane / 3 - 1, &s, &e)) s = e = 0;
    incl = e - s;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    total = __shfl_sync(0xffffffffu, incl, 8);
    shift = s - (incl - (e - s));
    if (lane >= 9) incl = 0x7fffffff;  // ends the search below
  }
  // particle at place t (any index for t >= total); every lane calls it
  __device__ __forceinline__ int at(int t) const {
    int r = 0;  // rows that end at or before t
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
      if (__shfl_sync(0xffffffffu, incl, r + o - 1) <= t) r += o;
    return t + __shfl_sync(0xffffffffu, shift, r);
  }
};

// Sums over the chunk's candidates for the K points of this lane.  act[m]
// marks the lane's valid points, and an invalid point's coordinates must be
// NaN (its s2 is then NaN and no term passes s2 < 4); slots[m]
// (warp-uniform) tells whether any lane holds a point m.  Returns the
// compensated sums in sum[]; adds the algorithmic candidate pairs of the
// lane's points to pairs.
//
// Two consecutive staged candidates are evaluated together with Blackwell's
// packed FP32 instructions (__ffma2_rn, __fmul2_rn, __fadd2_rn: two IEEE
// round-to-nearest operations per instruction, each element rounded as the
// scalar instruction rounds it), from the offset q - x through the kernel
// term det * Sigma * B(|A d|).  The expressions are those of field_sum (a - b
// as fma(b, -1, a), exact in the product, one rounding), so every term is
// bit for bit the scalar one; the compensated sum then takes the two terms
// one after the other, in candidate order.
// CB staged candidates per warp (a multiple of 32 above 32); the flush
// points move with it, the terms and their order do not.
template <int K, int CB = kCandBuf>
__device__ __forceinline__ void chunk_field(const GridView& g, const PartView& P, int cx, int cy, int cz,
                                            const float (&qx)[K], const float (&qy)[K], const float (&qz)[K],
                                            const bool (&act)[K], const bool (&slots)[K], const ChunkStage& st,
                                            float (&sum)[K], long long& pairs) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  // bounding box of the chunk's points
  const int kmin = 0x7fffffff, kmax = (int)0x80000000;
  int lx = kmin, ly = kmin, lz = kmin, hx = kmax, hy = kmax, hz = kmax;
  int nact = 0;
#pragma unroll
  for (int m = 0; m < K; ++m)
    if (act[m]) {
      lx = min(lx, fkey(qx[m]));
      ly = min(ly, fkey(qy[m]));
      lz = min(lz, fkey(qz[m]));
      hx = max(hx, fkey(qx[m]));
      hy = max(hy, fkey(qy[m]));
      hz = max(hz, fkey(qz[m]));
      ++nact;
    }
  const float blx = fkey_inv(__reduce_min_sync(0xffffffffu, lx));
  const float bly = fkey_inv(__reduce_min_sync(0xffffffffu, ly));
  const float blz = fkey_inv(__reduce_min_sync(0xffffffffu, lz));
  const float bhx = fkey_inv(__reduce_max_sync(0xffffffffu, hx));
  const float bhy = fkey_inv(__reduce_max_sync(0xffffffffu, hy));
  const float bhz = fkey_inv(__reduce_max_sync(0xffffffffu, hz));
  // the lane's points as packed pairs (q, q), built once per chunk
  float2 QX[K], QY[K], QZ[K];
#pragma unroll
  for (int m = 0; m < K; ++m) {
    QX[m] = make_float2(qx[m], qx[m]);
    QY[m] = make_float2(qy[m], qy[m]);
    QZ[m] = make_float2(qz[m], qz[m]);
  }
  // compensated sums (Kahan), updated only for in-support terms
  float s[K], c[K];
#pragma unroll
  for (int m = 0; m < K; ++m) s[m] = c[m] = 0.f;
  int nc = 0;
  auto flush = [&]() {
    cp_async_wait_all();
    __syncwarp();
    eval_staged<K, CB>(st, nc, QX, QY, QZ, slots, s, c);
    __syncwarp();
    nc = 0;
  };
  const CandidateRun run(g, cx, cy, cz);
  pairs += (long long)run.total * nact;
  // each batch's centres are loaded while the batch before is tested
  int j = run.at(lane);
  float4 x = make_float4(0.f, 0.f, 0.f, -1.f);
  if (lane < run.total) x = __ldg(P.xm + j);
  for (int t0 = 0; t0 < run.total; t0 += 32) {
    const int jn = run.at(t0 + 32 + lane);
    float4 xn = make_float4(0.f, 0.f, 0.f, -1.f);
    if (t0 + 32 + lane < run.total) xn = __ldg(P.xm + jn);
    const float ex = fmaxf(fmaxf(blx - x.x, x.x - bhx), 0.f);
    const float ey = fmaxf(fmaxf(bly - x.y, x.y - bhy), 0.f);
    const float ez = fmaxf(fmaxf(blz - x.z, x.z - bhz), 0.f);
    const bool pass = fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < x.w;  // x.w < 0 past the run's end
    const unsigned pm = __ballot_sync(0xffffffffu, pass);
    if (pass) {
      const int p = nc + __popc(pm & lt);
      float* const c0 = st.c + p;
      c0[SC_X * CB] = x.x;
      c0[SC_Y * CB] = x.y;
      c0[SC_Z * CB] = x.z;
      const float* ga = reinterpret_cast<const float*>(P.ga + j);
      const float* gb = reinterpret_cast<const float*>(P.gb + j);
      const float* gl = reinterpret_cast<const float*>(P.xlo + j);
      cp_async4(c0 + SC_LX * CB, gl);
      cp_async4(c0 + SC_LY * CB, gl + 1);
      cp_async4(c0 + SC_LZ * CB, gl + 2);
      cp_async4(c0 + SC_A0 * CB, ga);
      cp_async4(c0 + SC_A1 * CB, ga + 1);
      cp_async4(c0 + SC_A2 * CB, ga + 2);
      cp_async4(c0 + SC_A3 * CB, ga + 3);
      cp_async4(c0 + SC_B0 * CB, gb);
      cp_async4(c0 + SC_B1 * CB, gb + 1);
      cp_async4(c0 + SC_B2 * CB, gb + 2);
    }
    nc += __popc(pm);
    if (nc > CB - 32) flush();
    j = jn;
    x = xn;
  }
  flush();
#pragma unroll
  for (int m = 0; m < K; ++m) sum[m] = s[m];
}


// ---------------------------------------------------------------------------
// A point per lane, G lanes to a group: the group's points are near one another
// but not of one cell (sibling leaves, edge midpoints in cell order).  Points
// whose cells lie in a window of two cells per axis are evaluated together: the
// union of their candidates, at most four by four rows of four cells, is one run,
// filtered by the group's lanes against the points' box and staged as in
// chunk_field, and a staged candidate counts for a point only if its cell is one
// of the point's own 27 (a code of the window's outer cells against the lane's
// place in it).  Points outside the window are taken in another round.  Terms and
// order per point are field_sum's.
//
// A thread per point walking its own rows ran about 70 instructions per
// candidate of 32 points, most of them for lanes whose row was shorter, and
// waited for nine rows' offsets in turn.  Families of eight leaves take groups
// of eight: their box spans r against a reach of 4r and more, so few staged
// candidates are out of a lane's reach (leaf level 646 -> 454 us at 1M, 481 as
// whole warps; 37 -> 22 at 2k particles).  The edge midpoints of a cell are
// spread over 4r, where a warp's larger batches win (661 -> 586 us at 1M, 733 in
// eights; 1354 -> 984 on 500k sheets and filaments).
// ---------------------------------------------------------------------------
constexpr int kGroupWarps = 4;  // warps per block of the kernels on group_field
// Shared memory of a group: the staged components and codes, then 16 row
// records; the stride puts a warp's groups on different banks.
template <int G>
struct GroupRoom {
  static constexpr int kBuf = G == 32 ? 64 : 24;  // staged candidates
  static constexpr int kRows = (kStageComps + 1) * kBuf;
  static constexpr int kStride = G == 32 ? kRows + 64 : 424;
  static constexpr int kFloats = 32 / G * kStride;  // per warp
  static_assert(G == 8 || G == 32, "group sizes");
  static_assert(kRows % 4 == 0 && kStride % 4 == 0 && kRows + 64 <= kStride && kBuf >= 2 * G, "group layout");
};

// The staged candidates [0, nc) of the lane's group against its point; the
// groups' counts differ, the loop runs to the warp's largest.
template <int CB>
__device__ __forceinline__ void eval_coded(const float* st, int nc, const float2& QX, const float2& QY,
                                           const float2& QZ, int forbid, float& s, float& c) {
  const ChunkStage cs{const_cast<float*>(st)};
  const float2 M1 = make_float2(-1.0f, -1.0f);
  auto kahan = [&](float term) {
    const float y = __fsub_rn(term, c);
    const float tt = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(tt, s), y);
    s = tt;
  };
  const int most = __reduce_max_sync(0xffffffffu, nc);
#pragma unroll 1
  for (int t = 0; t < most; t += 2) {
    const int2 code = *reinterpret_cast<const int2*>(st + kStageComps * CB + t);
    const float2 X = ld_pair<CB>(cs, SC_X, t), Y = ld_pair<CB>(cs, SC_Y, t), Z = ld_pair<CB>(cs, SC_Z, t);
    const float2 LX = ld_pair<CB>(cs, SC_LX, t), LY = ld_pair<CB>(cs, SC_LY, t), LZ = ld_pair<CB>(cs, SC_LZ, t);
    const float2 A0 = ld_pair<CB>(cs, SC_A0, t), A1 = ld_pair<CB>(cs, SC_A1, t), A2 = ld_pair<CB>(cs, SC_A2, t),
                 A3 = ld_pair<CB>(cs, SC_A3, t);
    const float2 B0 = ld_pair<CB>(cs, SC_B0, t), B1 = ld_pair<CB>(cs, SC_B1, t), B2 = ld_pair<CB>(cs, SC_B2, t);
    // the expressions of eval_staged
    const float2 dx = __ffma2_rn(LX, M1, __ffma2_rn(X, M1, QX));
    const float2 dy = __ffma2_rn(LY, M1, __ffma2_rn(Y, M1, QY));
    const float2 dz = __ffma2_rn(LZ, M1, __ffma2_rn(Z, M1, QZ));
    const float2 u0 = __ffma2_rn(A0, dx, __ffma2_rn(A1, dy, __fmul2_rn(A2, dz)));
    const float2 u1 = __ffma2_rn(A1, dx, __ffma2_rn(A3, dy, __fmul2_rn(B0, dz)));
    const float2 u2 = __ffma2_rn(A2, dx, __ffma2_rn(B0, dy, __fmul2_rn(B1, dz)));
    const float2 s2 = __ffma2_rn(u0, u0, __ffma2_rn(u1, u1, __fmul2_rn(u2, u2)));
    const bool in0 = t < nc && s2.x < 4.0f && (code.x & forbid) == 0;
    const bool in1 = t + 1 < nc && s2.y < 4.0f && (code.y & forbid) == 0;
    if (in0 || in1) {
      const float2 r = make_float2(rsqrtf(fmaxf(s2.x, 1e-30f)), rsqrtf(fmaxf(s2.y, 1e-30f)));
      const float2 q = __fmul2_rn(s2, r);
      const float2 b1 = __ffma2_rn(s2, __ffma2_rn(make_float2(0.75f, 0.75f), q, make_float2(-1.5f, -1.5f)),
                                   make_float2(1.0f, 1.0f));
      const float2 tq = __ffma2_rn(q, M1, make_float2(2.0f, 2.0f));
      const float2 b2 = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(0.25f, 0.25f), tq), tq), tq);
      const float2 term = __fmul2_rn(B2, make_float2(q.x <= 1.0f ? b1.x : b2.x, q.y <= 1.0f ? b1.y : b2.y));
      if (in0) kahan(term.x);
      if (in1) kahan(term.y);
    }
  }
}

// Each lane's sum at its own point (0 for a lane without one); every lane of the
// warp calls it, smem holds the warp's GroupRoom<G>::kFloats of shared memory.
template <int G>
__device__ __forceinline__ float group_field(const GridView& g, const PartView& P, float qx, float qy, float qz,
                                             bool active, float* smem, long long& pairs) {
  using Room = GroupRoom<G>;
  constexpr int CB = Room::kBuf;
  constexpr unsigned ALL = 0xffffffffu, LANES = G == 32 ? ALL : (1u << (G & 31)) - 1u;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1), grp = lane & ~(G - 1);  // grp: the group's first lane
  float* const st = smem + lane / G * Room::kStride;
  int4* const rows = reinterpret_cast<int4*>(st + Room::kRows);
  // the group's bits of a ballot
  auto ballot = [&](bool p) { return (__ballot_sync(ALL, p) >> grp) & LANES; };
  int cx, cy, cz;
  cell_of(g, qx, qy, qz, cx, cy, cz);
  float s = 0.f, c = 0.f;
  bool waits = active;
  for (;;) {
    if (!__any_sync(ALL, waits)) break;
    const unsigned mine = ballot(waits);
    // the window's first cell: that of the group's first waiting point (in cell
    // order the lowest), for eight siblings the lowest within one of it per axis
    // (a group without a point runs along empty)
    const int lead = grp + (mine ? __ffs(mine) - 1 : 0);
    int bx = __shfl_sync(ALL, cx, lead), by = __shfl_sync(ALL, cy, lead), bz = __shfl_sync(ALL, cz, lead);
    if (G == 8) {
      const int ox = bx, oy = by, oz = bz;
      const bool near = waits && abs(cx - ox) <= 1 && abs(cy - oy) <= 1 && abs(cz - oz) <= 1;
      bx -= ballot(near && cx < ox) ? 1 : 0;
      by -= ballot(near && cy < oy) ? 1 : 0;
      bz -= ballot(near && cz < oz) ? 1 : 0;
    }
    const int lx = cx - bx, ly = cy - by, lz = cz - bz;
    const bool member = waits && (unsigned)lx < 2u && (unsigned)ly < 2u && (unsigned)lz < 2u;
    waits = waits && !member;
    const int ux = ballot(member && lx == 1) ? 1 : 0, uy = ballot(member && ly == 1) ? 1 : 0,
              uz = ballot(member && lz == 1) ? 1 : 0;
    const bool any = ballot(member) != 0u;
    // bounding box of the group's points
    float blx, bly, blz, bhx, bhy, bhz;
    if (G == 32) {
      const int kmin = 0x7fffffff, kmax = (int)0x80000000;
      blx = fkey_inv(__reduce_min_sync(ALL, member ? fkey(qx) : kmin));
      bly = fkey_inv(__reduce_min_sync(ALL, member ? fkey(qy) : kmin));
      blz = fkey_inv(__reduce_min_sync(ALL, member ? fkey(qz) : kmin));
      bhx = fkey_inv(__reduce_max_sync(ALL, member ? fkey(qx) : kmax));
      bhy = fkey_inv(__reduce_max_sync(ALL, member ? fkey(qy) : kmax));
      bhz = fkey_inv(__reduce_max_sync(ALL, member ? fkey(qz) : kmax));
    } else {
      const float inf = __int_as_float(0x7f800000);
      blx = member ? qx : inf, bly = member ? qy : inf, blz = member ? qz : inf;
      bhx = member ? qx : -inf, bhy = member ? qy : -inf, bhz = member ? qz : -inf;
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        blx = fminf(blx, __shfl_xor_sync(ALL, blx, o));
        bly = fminf(bly, __shfl_xor_sync(ALL, bly, o));
        blz = fminf(blz, __shfl_xor_sync(ALL, blz, o));
        bhx = fmaxf(bhx, __shfl_xor_sync(ALL, bhx, o));
        bhy = fmaxf(bhy, __shfl_xor_sync(ALL, bhy, o));
        bhz = fmaxf(bhz, __shfl_xor_sync(ALL, bhz, o));
      }
    }
    // rows (y, z) = (r % 4, r / 4) of the union, from the window's first cell
    // less one, two for each of the group's first eight lanes: [rs, re) the
    // particles, those below r1 in the first of the four cells, those from r3 on
    // in the last
    const int x0 = max(bx - 1, 0), x1 = min(bx + 1 + ux, g.nx - 1);
    int rs[2], re[2], r1[2], r3[2], code[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int r = 2 * sub + k, ry = r & 3, rz = r >> 2;
      const int y = by - 1 + ry, z = bz - 1 + rz;
      rs[k] = re[k] = r1[k] = r3[k] = 0;
      if (any && sub < 8 && ry <= 2 + uy && rz <= 2 + uz && x0 <= x1 && y >= 0 && y < g.ny && z >= 0 && z < g.nz) {
        const int* const row = g.off + ((long long)z * g.ny + y) * g.nx;
        rs[k] = __ldg(row + x0);
        re[k] = __ldg(row + x1 + 1);
        r1[k] = __ldg(row + min(max(bx, x0), x1 + 1));
        r3[k] = __ldg(row + min(max(bx + 2, x0), x1 + 1));
      }
      code[k] = (ry == 0 ? 4 : 0) | (ry == 3 ? 8 : 0) | (rz == 0 ? 16 : 0) | (rz == 3 ? 32 : 0);
    }
    const int n0 = re[0] - rs[0], n1 = re[1] - rs[1];
    int incl = n0 + n1;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int v = __shfl_up_sync(ALL, incl, o, G);
      if (sub >= o) incl += v;
    }
    const int total = __shfl_sync(ALL, incl, 7, G);
    const int mid = incl - n1, first = mid - n0;  // places where the lane's rows start: first, mid
    __syncwarp();  // the round before is done with the row records
    if (sub < 8) {
      rows[2 * sub] = make_int4(rs[0] - first, r1[0], r3[0], code[0]);
      rows[2 * sub + 1] = make_int4(rs[1] - mid, r1[1], r3[1], code[1]);
    }
    __syncwarp();
    // what a lane may not take: the first cell (row, layer) if it is in the
    // window's second, the last if it is in the first
    const int forbid = (lx == 1 ? 1 : 2) | (ly == 1 ? 4 : 8) | (lz == 1 ? 16 : 32);
    // the members' candidates, for the work counters: the rows that belong to the
    // 27 cells of each place in the window, times the members there
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int here = __popc(ballot(member && (lx | (ly << 1) | (lz << 2)) == k));
      if (G == 32 && here == 0) continue;  // warp-uniform
      const int no = ((k & 1) ? 1 : 2) | ((k & 2) ? 4 : 8) | ((k & 4) ? 16 : 32);
      int n = 0;
      if ((code[0] & no) == 0) n += (k & 1) ? re[0] - r1[0] : r3[0] - rs[0];
      if ((code[1] & no) == 0) n += (k & 1) ? re[1] - r1[1] : r3[1] - rs[1];
      pairs += (long long)here * n;
    }
    const float nan = __int_as_float(0x7fc00000);  // no term for a lane outside the round
    const float2 QX = member ? make_float2(qx, qx) : make_float2(nan, nan);
    const float2 QY = member ? make_float2(qy, qy) : make_float2(nan, nan);
    const float2 QZ = member ? make_float2(qz, qz) : make_float2(nan, nan);
    int nc = 0;
    auto flush = [&]() {
      cp_async_wait_all();
      __syncwarp();
      eval_coded<CB>(st, nc, QX, QY, QZ, forbid, s, c);
      __syncwarp();
      nc = 0;
    };
    // record of the row that holds place t
    auto row_at = [&](int t) {
      int l = 0;  // lanes whose rows end at or before t
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
        if (__shfl_sync(ALL, incl, l + o - 1, G) <= t) l += o;
      const int r = 2 * l + (t >= __shfl_sync(ALL, mid, l, G) ? 1 : 0);
      return rows[r];
    };
    const int most = __reduce_max_sync(ALL, total);
    int4 w = row_at(sub);
    int j = sub + w.x;
    float4 x = make_float4(0.f, 0.f, 0.f, -1.f);
    if (sub < total) x = __ldg(P.xm + j);
    for (int t0 = 0; t0 < most; t0 += G) {
      const int tn = t0 + G + sub;
      const int4 wn = row_at(tn);
      const int jn = tn + wn.x;
      float4 xn = make_float4(0.f, 0.f, 0.f, -1.f);
      if (tn < total) xn = __ldg(P.xm + jn);
      const float ex = fmaxf(fmaxf(blx - x.x, x.x - bhx), 0.f);
      const float ey = fmaxf(fmaxf(bly - x.y, x.y - bhy), 0.f);
      const float ez = fmaxf(fmaxf(blz - x.z, x.z - bhz), 0.f);
      const bool pass = fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < x.w;  // x.w < 0 past the run's end
      const unsigned pm = ballot(pass);
      if (pass) {
        float* const c0 = st + nc + __popc(pm & ((1u << sub) - 1u));
        c0[SC_X * CB] = x.x;
        c0[SC_Y * CB] = x.y;
        c0[SC_Z * CB] = x.z;
        c0[kStageComps * CB] = __int_as_float(w.w | (j < w.y ? 1 : 0) | (j >= w.z ? 2 : 0));
        const float* ga = reinterpret_cast<const float*>(P.ga + j);
        const float* gb = reinterpret_cast<const float*>(P.gb + j);
        const float* gl = reinterpret_cast<const float*>(P.xlo + j);
        cp_async4(c0 + SC_LX * CB, gl);
        cp_async4(c0 + SC_LY * CB, gl + 1);
        cp_async4(c0 + SC_LZ * CB, gl + 2);
        cp_async4(c0 + SC_A0 * CB, ga);
        cp_async4(c0 + SC_A1 * CB, ga + 1);
        cp_async4(c0 + SC_A2 * CB, ga + 2);
        cp_async4(c0 + SC_A3 * CB, ga + 3);
        cp_async4(c0 + SC_B0 * CB, gb);
        cp_async4(c0 + SC_B1 * CB, gb + 1);
        cp_async4(c0 + SC_B2 * CB, gb + 2);
      }
      nc += __popc(pm);
      if (__any_sync(ALL, nc > CB - G)) flush();
      w = wn;
      j = jn;
      x = xn;
    }
    flush();
  }
  return s;
}

// ---------------------------------------------------------------------------
// Bulk staging (configurations with `bulk` set in kEvalTable): each 27-cell
// row run is copied whole, in pieces of kBulkCap records, by 1D TMA bulk
// copies (cp.async.bulk, one per record array, completion counted on an
// mbarrier) into a per-warp AoS buffer; the warp then applies the same box
// test from shared memory and writes the survivors into the SoA buffer the
// evaluation loop reads.  Same candidates, same order, same values as
// chunk_field.  Waits are bounded: a wait that runs out counts
// C_STAGE_TIMEOUT (the host fails the frame), waits once more for the copies
// in flight and stops the warp.
// ---------------------------------------------------------------------------
constexpr int kBulkCap = 64;  // records per bulk piece

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(a) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ void mbar_expect(uint64_t* bar, unsigned tx) {
  const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }\n" ::"r"(b), "r"(tx)
               : "memory");
}

// 16-byte aligned global -> shared copy of `bytes` (a multiple of 16)
__device__ __forceinline__ void bulk_copy(float4* dst, const float4* src, unsigned bytes, uint64_t* bar) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(d),
               "l"(src), "r"(bytes), "r"(b)
               : "memory");
}

// Bounded wait for the barrier's phase `parity`; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
  const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
  for (int it = 0; it < (1 << 22); ++it) {
    unsigned done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }\n"
        : "=r"(done)
        : "r"(b), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

struct BulkStage {
  float4* rec;     // 4 x kBulkCap records: xm, xlo, ga, gb
  uint64_t* bar;   // the warp's barrier
  unsigned phase;  // parity of the next completion
};

// chunk_field with bulk staging; returns false after a wait ran out.
template <int K, int CB>
__device__ __forceinline__ bool chunk_field_bulk(const GridView& g, const PartView& P, int cx, int cy, int cz,
                                                 const float (&qx)[K], const float (&qy)[K], const float (&qz)[K],
                                                 const bool (&act)[K], const bool (&slots)[K], const ChunkStage& st,
                                                 BulkStage& bs, unsigned long long* counters, float (&sum)[K],
                                                 long long& pairs) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int kmin = 0x7fffffff, kmax = (int)0x80000000;
  int lx = kmin, ly = kmin, lz = kmin, hx = kmax, hy = kmax, hz = kmax;
  int nact = 0;
#pragma unroll
  for (int m = 0; m < K; ++m)
    if (act[m]) {
      lx = min(lx, fkey(qx[m]));
      ly = min(ly, fkey(qy[m]));
      lz = min(lz, fkey(qz[m]));
      hx = max(hx, fkey(qx[m]));
      hy = max(hy, fkey(qy[m]));
      hz = max(hz, fkey(qz[m]));
      ++nact;
    }
  const float blx = fkey_inv(__reduce_min_sync(0xffffffffu, lx));
  const float bly = fkey_inv(__reduce_min_sync(0xffffffffu, ly));
  const float blz = fkey_inv(__reduce_min_sync(0xffffffffu, lz));
  const float bhx = fkey_inv(__reduce_max_sync(0xffffffffu, hx));
  const float bhy = fkey_inv(__reduce_max_sync(0xffffffffu, hy));
  const float bhz = fkey_inv(__reduce_max_sync(0xffffffffu, hz));
  float2 QX[K], QY[K], QZ[K];
#pragma unroll
  for (int m = 0; m < K; ++m) {
    QX[m] = make_float2(qx[m], qx[m]);
    QY[m] = make_float2(qy[m], qy[m]);
    QZ[m] = make_float2(qz[m], qz[m]);
  }
  float s[K], c[K];
#pragma unroll
  for (int m = 0; m < K; ++m) s[m] = c[m] = 0.f;
  int nc = 0;
  auto flush = [&]() {
    __syncwarp();
    eval_staged<K, CB>(st, nc, QX, QY, QZ, slots, s, c);
    __syncwarp();
    nc = 0;
  };
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy) {
      int rs, re;
      if (!nb_row(g, cx, cy + dy, cz + dz, &rs, &re)) continue;
      pairs += (long long)(re - rs) * nact;
      for (int j0 = rs; j0 < re; j0 += kBulkCap) {
        const int cnt = min(kBulkCap, re - j0);
        const unsigned bytes = 16u * (unsigned)cnt;
        __syncwarp();  // every lane is done with the previous piece
        if (lane == 0) {
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
          mbar_expect(bs.bar, 4u * bytes);
          bulk_copy(bs.rec, P.xm + j0, bytes, bs.bar);
          bulk_copy(bs.rec + kBulkCap, P.xlo + j0, bytes, bs.bar);
          bulk_copy(bs.rec + 2 * kBulkCap, P.ga + j0, bytes, bs.bar);
          bulk_copy(bs.rec + 3 * kBulkCap, P.gb + j0, bytes, bs.bar);
        }
        if (!mbar_wait(bs.bar, bs.phase)) {
          if (lane == 0) stripe_add(counters, C_STAGE_TIMEOUT, 1ull);
          mbar_wait(bs.bar, bs.phase);  // the copies in flight, once more
          return false;
        }
        bs.phase ^= 1u;
        for (int k0 = 0; k0 < cnt; k0 += 32) {
          const int k = k0 + lane;
          bool pass = false;
          float4 x;
          if (k < cnt) {
            x = bs.rec[k];
            const float ex = fmaxf(fmaxf(blx - x.x, x.x - bhx), 0.f);
            const float ey = fmaxf(fmaxf(bly - x.y, x.y - bhy), 0.f);
            const float ez = fmaxf(fmaxf(blz - x.z, x.z - bhz), 0.f);
            pass = fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < x.w;
          }
          const unsigned pm = __ballot_sync(0xffffffffu, pass);
          if (pass) {
            float* const c0 = st.c + nc + __popc(pm & lt);
            const float4 l = bs.rec[kBulkCap + k], a = bs.rec[2 * kBulkCap + k], b = bs.rec[3 * kBulkCap + k];
            c0[SC_X * CB] = x.x;
            c0[SC_Y * CB] = x.y;
            c0[SC_Z * CB] = x.z;
            c0[SC_LX * CB] = l.x;
            c0[SC_LY * CB] = l.y;
            c0[SC_LZ * CB] = l.z;
            c0[SC_A0 * CB] = a.x;
            c0[SC_A1 * CB] = a.y;
            c0[SC_A2 * CB] = a.z;
            c0[SC_A3 * CB] = a.w;
            c0[SC_B0 * CB] = b.x;
            c0[SC_B1 * CB] = b.y;
            c0[SC_B2 * CB] = b.z;
          }
          nc += __popc(pm);
          if (nc > CB - 32) flush();
        }
      }
    }
  flush();
#pragma unroll
  for (int m = 0; m < K; ++m) sum[m] = s[m];
  return true;
}

}  // namespace pisurf
