// K3: anisotropic SPH field at points and particle normals.
//   - CalcParticlesNormal (src/evaluator.cpp:363-375): per particle the
//     poly6-gradient form sum_j det_j Sigma (-6 G_j d) (h^2 - |G_j d|^2)^2,
//     d = p_i - xmean_j (AnisotropicInterpolateGrad, :455-463, :408-415).
//   - SingleEval / SingleEvalWithGrad at arbitrary points (:60-125).
//   - HashGrid::GetPIdxList / GetInBoxParticles as device queries.
// The per-point field sum itself is field_sum() in device.cuh.
#include <cmath>
#include <vector>

#include "device.cuh"
#include "internal.h"

namespace pisurf {

// Gradient-form sums at a point; with four lanes to a point (walk_row) the even
// lanes hold x and y, the odd ones z.
template <int L>
struct GradSums {
  Kahan2 xy;
  Kahan x, y, z;
  // the term of candidate j at q, in all lanes
  template <bool SCALED>
  __device__ __forceinline__ void add(const PartView& P, int j, float qx, float qy, float qz, int sub) {
    const float4 c = __ldg(P.xm + j);
    const float dx = qx - c.x, dyy = qy - c.y, dzz = qz - c.z;
    const float4 a = __ldg(P.ga + j);
    const float4 b = __ldg(P.gb + j);
    const float4 lo = __ldg(P.xlo + j);
    float u0, u1, u2;
    amul(a, b, dx - lo.x, dyy - lo.y, dzz - lo.z, u0, u1, u2);
    const float s2 = fmaf(u0, u0, fmaf(u1, u1, u2 * u2));
    if (s2 < 1.0f) {
      const float om = 1.0f - s2;
      float f = b.z * om * om;
      if (SCALED) f *= b.w;
      if (L == 1) {
        x.add(u0 * f);
        y.add(u1 * f);
        z.add(u2 * f);
      } else {
        xy.add(__fmul2_rn(sub & 1 ? make_float2(u2, u2) : make_float2(u0, u1), make_float2(f, f)));
      }
    }
  }
  __device__ __forceinline__ void gather() {
    if (L == 1) return;
    x.s = xy.s.x, y.s = xy.s.y;
    z.s = __shfl_down_sync(0xffffffffu, xy.s.x, 1, 4);
  }
};

// A normal and its length, whose rounding is written out: the compiler's choice of
// which product to fuse moved with the code around it, and the lengths' last bits,
// and the node curvatures', with it.
__device__ __forceinline__ float4 with_length(float x, float y, float z) {
  return make_float4(x, y, z, sqrtf(fmaf(z, z, fmaf(y, y, __fmul_rn(x, x)))));
}

// |d| < R / 2: |A d| < 1 needs it.
__device__ __forceinline__ bool grad_reach(const float4* xm, float qx, float qy, float qz) {
  const float4 x = __ldg(xm);
  const float dx = qx - x.x, dyy = qy - x.y, dzz = qz - x.z;
  return fmaf(dx, dx, fmaf(dyy, dyy, dzz * dzz)) < 0.25f * x.w;
}

// Gradient-form sum at q (without the -6 h^5 factor): sum_j wdet_j u (1 - s2)^2
// with u = A_j (q - xmean_j), s2 = |u|^2 < 1.
template <int L>
__device__ __forceinline__ void grad_sum(const GridView& g, const PartView& P, float qx, float qy, float qz,
                                         bool valid, int sub, GradSums<L>& sum) {
  int cx, cy, cz;
  cell_of(g, qx, qy, qz, cx, cy, cz);
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy) {
      int s = 0, e = 0;
      if (!valid || !nb_row(g, cx, cy + dy, cz + dz, &s, &e)) {
        if (L == 1) continue;
        s = e = 0;
      }
      walk_row<L>(
          s, e, sub, [&](int j0, int k) { return grad_reach(P.xm + j0 + k, qx, qy, qz); },
          [&](int j) { sum.template add<false>(P, j, qx, qy, qz, sub); });
    }
  sum.gather();
}

template <int L>
__global__ void __launch_bounds__(128, 12) k_normals(GridView g, PartView P, long long n, float gscale, float4* __restrict__ nrm) {
  launch_wait();
  const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x & (L - 1);
  if (L == 1 && t >= n) return;
  const float4 p = t < n ? P.pos[t] : make_float4(0.f, 0.f, 0.f, 0.f);
  const bool splash = p.w != 0.f;  // a splash particle's normal stays zero
  if (t < n && splash && sub == 0) nrm[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (L == 1 && splash) return;
  GradSums<L> sum;
  grad_sum<L>(g, P, p.x, p.y, p.z, t < n && !splash, sub, sum);
  if (L > 1 && (sub != 0 || t >= n || splash)) return;
  const float gx = sum.x.s * gscale, gy = sum.y.s * gscale, gz = sum.z.s * gscale;
  nrm[t] = with_length(gx, gy, gz);
}

// field_sum and grad_sum at q in one walk: both need u = A_j d of the same
// candidates (s2 < 1 implies the |d| < R / 2 that grad_sum tests first).  Terms
// and orders are those of the two sums.
__device__ __forceinline__ float field_grad_sum(const GridView& g, const PartView& P, float qx, float qy, float qz,
                                                float& gx, float& gy, float& gz) {
  int cx, cy, cz;
  cell_of(g, qx, qy, qz, cx, cy, cz);
  Kahan acc, ax, ay, az;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy) {
      int s, e;
      if (!nb_row(g, cx, cy + dy, cz + dz, &s, &e)) continue;
      for (int j0 = s; j0 < e; j0 += 32) {
        const int cnt = min(32, e - j0);
        unsigned m = 0u;
        for (int k = 0; k < cnt; ++k) {
          const float4 x = __ldg(P.xm + j0 + k);
          const float dx = qx - x.x, dyy = qy - x.y, dzz = qz - x.z;
          const float e2 = fmaf(dx, dx, fmaf(dyy, dyy, dzz * dzz));
          m |= (e2 < x.w ? 1u : 0u) << k;
        }
        while (m) {
          const int j = j0 + __ffs(m) - 1;
          m &= m - 1u;
          const float4 x = __ldg(P.xm + j);
          const float dx = qx - x.x, dyy = qy - x.y, dzz = qz - x.z;
          const float4 a = __ldg(P.ga + j);
          const float4 b = __ldg(P.gb + j);
          const float4 lo = __ldg(P.xlo + j);
          float u0, u1, u2;
          amul(a, b, dx - lo.x, dyy - lo.y, dzz - lo.z, u0, u1, u2);
          const float s2 = fmaf(u0, u0, fmaf(u1, u1, u2 * u2));
          if (s2 < 4.0f) acc.add(b.z * bspline_s2(s2));
          if (s2 < 1.0f) {
            const float om = 1.0f - s2;
            const float f = b.z * om * om;
            ax.add(u0 * f);
            ay.add(u1 * f);
            az.add(u2 * f);
          }
        }
      }
    }
  gx = ax.s;
  gy = ay.s;
  gz = az.s;
  return acc.s;
}

// Hash cell of each point (over the grid grown by 2 cells, where cell_coord
// clamps) and its place among the cell's points, a warp's points of one cell
// with one addition.  A point with no cell of the grid beside its own has no
// candidate: it gets its value here and no place (x = -1).  All points outside
// would else add to the few cells that they are clamped to: 300k of them took
// 277 us, 65 in the caller's order; points in one cell 277, 70 in their order.
__global__ void k_point_cell(GridView g, const float* __restrict__ pts, long long m, int* __restrict__ cnt,
                             int2* __restrict__ at, float iso, float gscale, float* __restrict__ val,
                             float* __restrict__ grad) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int k = -1;
  if (i < m) {
    int cx, cy, cz;
    cell_of(g, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], cx, cy, cz);
    if (cx >= -1 && cx <= g.nx && cy >= -1 && cy <= g.ny && cz >= -1 && cz <= g.nz) {
      k = ((cz + 2) * (g.ny + 4) + (cy + 2)) * (g.nx + 4) + (cx + 2);
    } else {
      val[i] = iso;
      if (grad) grad[3 * i] = grad[3 * i + 1] = grad[3 * i + 2] = 0.0f * gscale;
    }
  }
  const unsigned peers = __match_any_sync(0xffffffffu, k);
  const int lead = __ffs(peers) - 1;
  int first = 0;
  if (lane == lead && k >= 0) first = atomicAdd(cnt + k, __popc(peers));
  first = __shfl_sync(0xffffffffu, first, lead);
  if (i < m) at[i] = make_int2(k, first + __popc(peers & ((1u << lane) - 1u)));
}

__global__ void k_point_order(const int2* __restrict__ at, const int* __restrict__ off, long long m,
                              int* __restrict__ order) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int2 a = at[i];
  if (a.x >= 0) order[off[a.x] + a.y] = (int)i;
}

// A thread per point, in the order given (null: as they come; *ordered points are
// in it).  Points in no
// order put every lane in a cell of its own, and each candidate load then
// fetches 32 lines; in cell order a warp's lanes read the same ones.  300k
// points around a 200k-particle frame with gradients: 438 us as they come, 141
// us in cell order with both sums in one walk, and 20 us for the ordering.
__global__ void __launch_bounds__(128) k_eval_points(GridView g, PartView P, const float* __restrict__ pts,
                                                     const int* __restrict__ order, const int* __restrict__ ordered,
                                                     long long m, float iso, float gscale, float* __restrict__ val,
                                                     float* __restrict__ grad) {
  launch_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (order ? *ordered : m)) return;
  const long long i = order ? order[t] : t;
  const float qx = pts[3 * i], qy = pts[3 * i + 1], qz = pts[3 * i + 2];
  if (!grad) {
    val[i] = iso - field_sum(g, P, qx, qy, qz, nullptr);
    return;
  }
  float gx, gy, gz;
  val[i] = iso - field_grad_sum(g, P, qx, qy, qz, gx, gy, gz);
  grad[3 * i] = gx * gscale;
  grad[3 * i + 1] = gy * gscale;
  grad[3 * i + 2] = gz * gscale;
}

static GridView gview(pi_frame* f) {
  const GridHost& gh = f->g;
  return GridView{gh.bounding[0], gh.bounding[2], gh.bounding[4], gh.cell, gh.nx, gh.ny, gh.nz, f->off.p};
}
static PartView pview(pi_frame* f) { return PartView{f->pos.p, f->xm.p, f->ga.p, f->gb.p, f->xlo.p}; }

// -6 h^5 with h = 2r (see AnisotropicInterpolateGrad in A = G / h units)
static float grad_scale(pi_frame* f) {
  double h = 2.0 * (double)f->P.radius;
  return (float)(-6.0 * h * h * h * h * h);
}

// ---- variable radius: the bins' candidate lists, per-particle scales ----

// Gradient-form sum with each term scaled by its particle's -6 h_j^5 (gb.w).
template <int L>
__device__ __forceinline__ void grad_sum_vr(const MultiGridView& m, const PartView& P, float qx, float qy, float qz,
                                            bool valid, int sub, GradSums<L>& sum) {
  for (int b = 0; b < m.nb; ++b) {
    const BinGrid g = m.g[b];
    const int cx = cell_coord(qx, g.b0, g.cell, g.nx), cy = cell_coord(qy, g.b2, g.cell, g.ny),
              cz = cell_coord(qz, g.b4, g.cell, g.nz);
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy) {
        int s = 0, e = 0;
        if (!valid || !bin_row(g, m.off, cx, cy + dy, cz + dz, &s, &e)) {
          if (L == 1) continue;
          s = e = 0;
        }
        walk_row<L>(
            s, e, sub, [&](int j0, int k) { return grad_reach(P.xm + j0 + k, qx, qy, qz); },
            [&](int j) { sum.template add<true>(P, j, qx, qy, qz, sub); });
      }
  }
  sum.gather();
}

template <int L>
__global__ void __launch_bounds__(128) k_vr_normals(const MultiGridView* __restrict__ mg, PartView P, long long n,
                                                    float4* __restrict__ nrm) {
  launch_wait();
  const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
  const int sub = threadIdx.x & (L - 1);
  if (L == 1 && t >= n) return;
  const float4 p = t < n ? P.pos[t] : make_float4(0.f, 0.f, 0.f, 0.f);
  GradSums<L> sum;
  grad_sum_vr<L>(*mg, P, p.x, p.y, p.z, t < n, sub, sum);
  if (L > 1 && (sub != 0 || t >= n)) return;
  const float gx = sum.x.s, gy = sum.y.s, gz = sum.z.s;
  nrm[t] = with_length(gx, gy, gz);
}

__global__ void k_vr_eval_points(const MultiGridView* __restrict__ mg, PartView P, const float* __restrict__ pts,
                                 long long m, float iso, float* __restrict__ val, float* __restrict__ grad) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const float qx = pts[3 * i], qy = pts[3 * i + 1], qz = pts[3 * i + 2];
  val[i] = iso - field_sum_vr(*mg, P, qx, qy, qz, nullptr);
  if (grad) {
    GradSums<1> sum;
    grad_sum_vr<1>(*mg, P, qx, qy, qz, true, 0, sum);
    grad[3 * i] = sum.x.s;
    grad[3 * i + 1] = sum.y.s;
    grad[3 * i + 2] = sum.z.s;
  }
}

__global__ void k_vr_nb_count(const MultiGridView* __restrict__ mg, const float* __restrict__ pts, long long m,
                              int* __restrict__ cnt) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const MultiGridView& v = *mg;
  int c = 0;
  for (int b = 0; b < v.nb; ++b) {
    const BinGrid g = v.g[b];
    const int cx = cell_coord(pts[3 * i], g.b0, g.cell, g.nx), cy = cell_coord(pts[3 * i + 1], g.b2, g.cell, g.ny),
              cz = cell_coord(pts[3 * i + 2], g.b4, g.cell, g.nz);
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy) {
        int s, e;
        if (bin_row(g, v.off, cx, cy + dy, cz + dz, &s, &e)) c += e - s;
      }
  }
  cnt[i] = c;
}

__global__ void k_vr_nb_fill(const MultiGridView* __restrict__ mg, const float* __restrict__ pts, long long m,
                             const int* __restrict__ off, const uint32_t* __restrict__ sidx, int* __restrict__ out) {
  launch_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const MultiGridView& v = *mg;
  int o = off[i];
  for (int b = 0; b < v.nb; ++b) {
    const BinGrid g = v.g[b];
    const int cx = cell_coord(pts[3 * i], g.b0, g.cell, g.nx), cy = cell_coord(pts[3 * i + 1], g.b2, g.cell, g.ny),
              cz = cell_coord(pts[3 * i + 2], g.b4, g.cell, g.nz);
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy) {
        int s, e;
        if (!bin_row(g, v.off, cx, cy + dy, cz + dz, &s, &e)) continue;
        for (int j = s; j < e; ++j) out[o++] = (int)sidx[j];
      }
  }
}

void stage_normals(pi_frame* f) {
  cudaStream_t s = f->ctx->stream;
  // a clump of less than a cell's neighbourhood: nearly every candidate is a
  // term, which four lanes work out four times over (20,000 particles in one
  // cell: 6.9 ms with four, 5.1 with one)
  const int lanes = !f->varR && f->g.cellNum < 27 ? 1 : particle_lanes(f);
  if (f->varR) {
    const auto normals = lanes == 4 ? k_vr_normals<4> : k_vr_normals<1>;
    PI_LAUNCH(normals, div_up(f->N * lanes, 128), 128, 0, s, f->mgv.p, pview(f), f->N, f->nrm.p);
    return;
  }
  const auto normals = lanes == 4 ? k_normals<4> : k_normals<1>;
  PI_LAUNCH(normals, div_up(f->N * lanes, 128), 128, 0, s, gview(f), pview(f), f->N, grad_scale(f), f->nrm.p);
}

// Cells of the grid grown by 2 on each side.
static long long point_cells(const pi_frame* f) {
  return (long long)(f->g.nx + 4) * (f->g.ny + 4) * (f->g.nz + 4);
}

// Whether consecutive points (h: the caller's, on the host) are mostly of
// different cells that have candidates: of 32 pairs spread over them, eight and
// more.  Points of one cell or in a scan's order read the same lines as they come,
// and points beyond the grid's reach read none.
static bool points_scattered(const pi_frame* f, const float* h, long long m) {
  const float lo[3] = {f->g.bounding[0], f->g.bounding[2], f->g.bounding[4]};
  const int n[3] = {f->g.nx, f->g.ny, f->g.nz};
  int apart = 0;
  for (int k = 0; k < 32; ++k) {
    const float* const p = h + (m - 1) * k / 32 * 3;
    bool reach = true, same = true;
    for (int ax = 0; ax < 3; ++ax) {
      const float q = std::floor((p[ax] - lo[ax]) / f->g.cell), r = std::floor((p[3 + ax] - lo[ax]) / f->g.cell);
      reach = reach && q >= -1.0f && q <= (float)n[ax];
      same = same && q == r;
    }
    apart += reach && !same ? 1 : 0;
  }
  return apart >= 8;
}

// Whether m points are put in cell order first: from the count where the five
// launches of the ordering (15 us) are less than the scattered loads they save,
// while the cells' table is no larger than the points' own arrays, and where the
// points are scattered.
static bool order_points(const pi_frame* f, const float* h_pts, long long m) {
  const long long nc = point_cells(f);
  if (m < 16384 || nc > 4 * m || m > 0x7fffffffLL || nc >= 0x7fffffffLL) return false;  // places and cells are ints
  return points_scattered(f, h_pts, m);
}

void eval_points(pi_frame* f, const float* h_pts, const float* d_pts, long long m, float* d_val, float* d_grad) {
  cudaStream_t s = f->ctx->stream;
  if (f->varR) {
    PI_LAUNCH(k_vr_eval_points, div_up(m, 128), 128, 0, s, f->mgv.p, pview(f), d_pts, m, f->iso, d_val, d_grad);
    return;
  }
  const GridView g = gview(f);
  DBuf<int> cnt, order, tmp;
  DBuf<int2> at;
  bool ordered = order_points(f, h_pts, m);
  const long long nc = point_cells(f);
  try {
    if (ordered) {
      cnt.alloc(f->ctx, s, nc + 1);
      at.alloc(f->ctx, s, m);
      order.alloc(f->ctx, s, m);
      tmp.alloc(f->ctx, s, scan_tmp_ints(nc + 1));
    }
  } catch (const NoMem&) {  // the caller's order needs none of them
    ordered = false;
    cnt.release(), at.release(), order.release(), tmp.release();
  }
  if (ordered) {
    PI_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int) * (nc + 1), s));
    PI_LAUNCH(k_point_cell, div_up(m, 256), 256, 0, s, g, d_pts, m, cnt.p, at.p, f->iso, grad_scale(f),
              d_val, d_grad);
    exclusive_scan_i32(cnt.p, cnt.p, nc + 1, nullptr, tmp.p, s);
    PI_LAUNCH(k_point_order, div_up(m, 256), 256, 0, s, at.p, cnt.p, m, order.p);
  }
  // the scan's last entry is the number of points that have a place
  PI_LAUNCH(k_eval_points, div_up(m, 128), 128, 0, s, g, pview(f), d_pts, order.p,
            ordered ? cnt.p + nc : nullptr, m, f->iso, grad_scale(f), d_val, d_grad);
}

// GetPIdxList: counts, then lists (particle indices through IndexList).
__global__ void k_nb_count(GridView g, const float* __restrict__ pts, long long m, int* __restrict__ cnt) {
  launch_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  int cx, cy, cz;
  cell_of(g, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], cx, cy, cz);
  int c = 0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy) {
      int s, e;
      if (nb_row(g, cx, cy + dy, cz + dz, &s, &e)) c += e - s;
    }
  cnt[i] = c;
}

__global__ void k_nb_fill(GridView g, const float* __restrict__ pts, long long m, const int* __restrict__ off,
                          const uint32_t* __restrict__ sidx, int* __restrict__ out) {
  launch_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  int cx, cy, cz;
  cell_of(g, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], cx, cy, cz);
  int o = off[i];
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy) {
      int s, e;
      if (!nb_row(g, cx, cy + dy, cz + dz, &s, &e)) continue;
      for (int j = s; j < e; ++j) out[o++] = (int)sidx[j];
    }
}

long long neighbors(pi_frame* f, const float* h_pts, long long m, long long* h_off, int* h_idx, long long cap) {
  cudaStream_t s = f->ctx->stream;
  DBuf<float> pts;
  DBuf<int> cnt, tmp;
  pts.alloc(f->ctx, s, m * 3);
  cnt.alloc(f->ctx, s, m + 1);
  tmp.alloc(f->ctx, s, scan_tmp_ints(m + 1));
  PI_CUDA(cudaMemcpyAsync(pts.p, h_pts, sizeof(float) * 3 * m, cudaMemcpyHostToDevice, s));
  GridView g = gview(f);
  PI_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int) * (m + 1), s));
  if (f->varR)
    PI_LAUNCH(k_vr_nb_count, div_up(m, 128), 128, 0, s, f->mgv.p, pts.p, m, cnt.p);
  else
    PI_LAUNCH(k_nb_count, div_up(m, 128), 128, 0, s, g, pts.p, m, cnt.p);
  int total = 0;
  exclusive_scan_i32(cnt.p, cnt.p, m + 1, nullptr, tmp.p, s);
  PI_CUDA(cudaMemcpyAsync(&total, cnt.p + m, sizeof(int), cudaMemcpyDeviceToHost, s));
  PI_CUDA(cudaStreamSynchronize(s));
  std::vector<int> offs(m + 1);
  PI_CUDA(cudaMemcpy(offs.data(), cnt.p, sizeof(int) * (m + 1), cudaMemcpyDeviceToHost));
  for (long long i = 0; i <= m; ++i) h_off[i] = offs[i];
  if (total > cap) return total;
  DBuf<int> out;
  out.alloc(f->ctx, s, total > 0 ? total : 1);
  if (f->varR)
    PI_LAUNCH(k_vr_nb_fill, div_up(m, 128), 128, 0, s, f->mgv.p, pts.p, m, cnt.p, f->sidx.p, out.p);
  else
    PI_LAUNCH(k_nb_fill, div_up(m, 128), 128, 0, s, g, pts.p, m, cnt.p, f->sidx.p, out.p);
  PI_CUDA(cudaMemcpyAsync(h_idx, out.p, sizeof(int) * total, cudaMemcpyDeviceToHost, s));
  PI_CUDA(cudaStreamSynchronize(s));
  return total;
}

// GetInBoxParticles (src/hash_grid.cpp:164-194): x outer, z inner, one
// thread walks the cell block (a query, not a hot path).
__global__ void k_in_box(GridView g, float b1x, float b1y, float b1z, float b2x, float b2y, float b2z,
                         float B1, float B3, float B5, const uint32_t* __restrict__ sidx, int* __restrict__ out,
                         long long cap, long long* __restrict__ total) {
  launch_wait();
  b1x = fmaxf(b1x, g.b0);
  b1y = fmaxf(b1y, g.b2);
  b1z = fmaxf(b1z, g.b4);
  b2x = fminf(b2x, B1);
  b2y = fminf(b2y, B3);
  b2z = fminf(b2z, B5);
  int mnx, mny, mnz, mxx, mxy, mxz;
  cell_of(g, b1x, b1y, b1z, mnx, mny, mnz);
  cell_of(g, b2x, b2y, b2z, mxx, mxy, mxz);
  long long k = 0;
  for (int x = mnx - 1; x <= mxx + 1; ++x)
    for (int y = mny - 1; y <= mxy + 1; ++y)
      for (int z = mnz - 1; z <= mxz + 1; ++z) {
        if (x < 0 || x >= g.nx || y < 0 || y >= g.ny || z < 0 || z >= g.nz) continue;
        long long c = ((long long)z * g.ny + y) * g.nx + x;
        for (int j = g.off[c]; j < g.off[c + 1]; ++j) {
          if (k < cap) out[k] = (int)sidx[j];
          ++k;
        }
      }
  *total = k;
}

long long in_box(pi_frame* f, const float* b1, const float* b2, int* h_idx, long long cap) {
  cudaStream_t s = f->ctx->stream;
  DBuf<int> out;
  DBuf<long long> tot;
  out.alloc(f->ctx, s, cap > 0 ? cap : 1);
  tot.alloc(f->ctx, s, 1);
  const GridHost& gh = f->g;
  PI_LAUNCH(k_in_box, 1, 1, 0, s, gview(f), b1[0], b1[1], b1[2], b2[0], b2[1], b2[2], gh.bounding[1],
            gh.bounding[3], gh.bounding[5], f->sidx.p, out.p, cap, tot.p);
  long long total = 0;
  PI_CUDA(cudaMemcpyAsync(&total, tot.p, sizeof(long long), cudaMemcpyDeviceToHost, s));
  PI_CUDA(cudaStreamSynchronize(s));
  if (total <= cap && total > 0)
    PI_CUDA(cudaMemcpy(h_idx, out.p, sizeof(int) * total, cudaMemcpyDeviceToHost));
  return total;
}

}  // namespace pisurf
