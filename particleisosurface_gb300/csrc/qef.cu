// K5: per-leaf QEF vertex, TNode::NodeCalcNode (src/iso_method_ours.cpp:101-174)
// with QEFNormal<float,4>::combineSelf (include/qefnorm.h:18-33) and
// calcErrorDMC (src/iso_method_ours.cpp:40-50).  In the reference both call
// sites are commented out (src/surface_reconstructor.cpp:258,270); pi_params.qef
// switches them on with the same semantics:
//   leaf by size:      node = QEF vertex if it lies in the cell, value
//                      f(node), zeroed if err / cellsize < 1e-4;
//   leaf by criteria:  node = QEF vertex if it lies in the cell, value
//                      f(node) (the later SingleEval undoes the zeroing).
// Gradients are the finite differences of GridEval (src/evaluator.cpp:293-359)
// over the 27 samples.  Accumulation and solve are FP64; the solve follows
// the pseudo-inverse rule of a Jacobi eigen-decomposition of the equilibrated
// symmetric 4x4 normal matrix (eigenvalues below 1e-12 of the largest are
// dropped), decided by LDL^T bounds where they settle it.  Where that matrix
// is singular the reference's Matrix4f::inverse yields non-finite values and
// the vertex is rejected; so is it here, and the number of singular leaves is
// counted.
#include <algorithm>
#include <cmath>

#include "device.cuh"
#include "internal.h"

namespace pisurf {

enum : int8_t { Q_EMPTY = 0, Q_INTERNAL = 1, Q_LEAF = 2 };

// Symmetric 4x4 Jacobi eigen-decomposition, A = V diag(w) V^T.
__device__ void sym_eig4(double A[4][4], double w[4], double V[4][4]) {
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) V[i][j] = (i == j) ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 20; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int p = 0; p < 4; ++p) {
      dia += fabs(A[p][p]);
      for (int q = p + 1; q < 4; ++q) off += fabs(A[p][q]);
    }
    if (off <= 1e-18 * dia || off == 0.0) break;
    for (int p = 0; p < 3; ++p)
      for (int q = p + 1; q < 4; ++q) {
        const double apq = A[p][q];
        if (fabs(apq) <= 1e-300) continue;
        const double theta = (A[q][q] - A[p][p]) / (2.0 * apq);
        double t = 1.0 / (fabs(theta) + sqrt(theta * theta + 1.0));
        if (theta < 0.0) t = -t;
        const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        for (int r = 0; r < 4; ++r) {
          const double arp = A[r][p], arq = A[r][q];
          A[r][p] = c * arp - s * arq;
          A[r][q] = s * arp + c * arq;
        }
        for (int r = 0; r < 4; ++r) {
          const double apr = A[p][r], aqr = A[q][r];
          A[p][r] = c * apr - s * aqr;
          A[q][r] = s * apr + c * aqr;
        }
        for (int r = 0; r < 4; ++r) {
          const double vrp = V[r][p], vrq = V[r][q];
          V[r][p] = c * vrp - s * vrq;
          V[r][q] = s * vrp + c * vrq;
        }
      }
  }
  for (int i = 0; i < 4; ++i) w[i] = A[i][i];
}

// d / 2 for a double d that is 0 or at least 2^-1021 in magnitude (here a
// difference of two floats, so at least 2^-149), exactly, on the integer
// pipe: the exponent field is decremented.
__device__ __forceinline__ double half_exact(double d) {
  const long long b = __double_as_longlong(d);
  return (b << 1) == 0 ? d : __longlong_as_double(b - (1LL << 52));
}

// (double)f on the integer pipe for a normal float f (the exponent rebased
// from 127 to 1023, the 23 fraction bits moved to the top of the 52), the
// hardware conversion for zero, subnormal, infinite and NaN inputs.
__device__ __forceinline__ double f2d_exact(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xffu;
  if (e == 0u || e == 0xffu) return (double)f;
  const unsigned hi = (u & 0x80000000u) | (((u >> 3) & 0x0fffffffu) + (896u << 20));
  return __hiloint2double((int)hi, (int)(u << 29));
}

// Equilibration scale of a diagonal entry v: about v^-1/2 from the FP32
// reciprocal square root when v converts to a normal float, the FP64 value
// otherwise, 1 for v <= 0.  Any positive scale gives the same solution.
__device__ __forceinline__ double equil_scale(double v) {
  if (!(v > 0.0)) return 1.0;
  const float vf = (float)v;
  if (vf >= 1.17549435e-38f && vf <= 3.0e38f) return (double)rsqrtf(vf);
  return 1.0 / sqrt(v);
}

struct QefArgs {
  GridView g;
  PartView P;
  float iso;
  float radius;
  long long lb, le;
  // the level's finite-difference step (every node of a level has the same
  // half size), in FP64, and its reciprocal
  double step, i1;
  int unit_exp;  // biased exponent of the sample values' unit (below); 0: no unit
};

// ---------------------------------------------------------------------------
// The normal equations in integers.  A sample value is the float iso - sum, and
// every such value is a whole multiple of unit = ulp(iso) / 2: a result of
// iso / 2 or more in magnitude has an ulp of at least that, and below it sum
// lies between iso / 2 and 3 iso / 2, so that the subtraction is exact on the
// grid of ulp(iso / 2).  In units, values within 8 times iso are integers below
// 2^28, differences and products are exact in 32 and 64 bits, and the sums over
// samples carry no rounding at all; only their combination with the positions
// is FP64.  Deep in dense particles, where every value of a leaf is larger, all
// are multiples of the smallest one's ulp, and that is the leaf's unit.  A leaf
// with a wider range than 28 bits takes the FP64 sums.
//
// FP64 issue bounds this kernel: GB300 has two FP64 lanes per SM and clock.
// The FP64 sums took about 460 instructions a leaf of 620 in all; these take 140,
// and their 1000 integer instructions run on pipes with 64 lanes.  1M dam
// break, 4.2M leaves: 5.4 -> 2.6 ms alone (with the accepted leaves apart).
// ---------------------------------------------------------------------------
constexpr int kSampleLow = -(1 << 28), kSampleHigh = 1 << 25;  // in units; no value exceeds iso

// v as a double, rounded once: 2^84 + high and 2^52 + low words are exact.
__device__ __forceinline__ double i64_to_double(long long v) {
  const double hi = __hiloint2double(0x45300000, (int)((unsigned)(v >> 32) ^ 0x80000000u));
  const double lo = __hiloint2double(0x43300000, (int)(unsigned)v);
  return (hi - 0x1.00000801p84) + lo;  // 2^84 + 2^63 + 2^52
}
__device__ __forceinline__ double i32_to_double(int v) {
  return __hiloint2double(0x43300000, (int)((unsigned)v ^ 0x80000000u)) - 0x1.000008p52;  // 2^52 + 2^31
}

// Twice the finite difference of sample i along the axis of the given stride
// (GridEval's, src/evaluator.cpp:185-240: one-sided at the ends, the mean of the
// two in the middle).
template <int STRIDE>
__device__ __forceinline__ int diff2(const int (&s)[27], int i) {
  const int d = (i / STRIDE) % 3;
  if (d == 0) return 2 * (s[i] - s[i + STRIDE]);
  if (d == 2) return 2 * (s[i - STRIDE] - s[i]);
  return s[i - STRIDE] - s[i + STRIDE];
}

// Sums over the samples of the products of two axes' differences, total and
// per plane of constant position along each of the two axes.
template <int S1, int S2>
__device__ __forceinline__ void cross_sums(const int (&s)[27], double& total, double (&by1)[3], double (&by2)[3]) {
  long long r1[3] = {0, 0, 0}, r2[3] = {0, 0, 0};
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 3; ++k2) {
      constexpr int S3 = 13 - S1 - S2;  // the third axis' stride (1, 3, 9)
      long long c = 0;
#pragma unroll
      for (int k3 = 0; k3 < 3; ++k3) {
        const int i = k1 * S1 + k2 * S2 + k3 * S3;
        c += (long long)diff2<S1>(s, i) * diff2<S2>(s, i);
      }
      r1[k1] += c;
      r2[k2] += c;
    }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    by1[k] = i64_to_double(r1[k]);
    by2[k] = i64_to_double(r2[k]);
  }
  total = by1[0] + by1[1] + by1[2];
}

// One axis: the sum of its squared differences, what they contribute to its
// right side through their own positions p, twice the sum of difference times
// value, and its differences' plane sums (for the last column).
template <int S>
__device__ __forceinline__ void axis_sums(const int (&s)[27], const double (&p)[3], double& square, double& right,
                                          double& first, double& moved) {
  long long sq[3] = {0, 0, 0}, gf = 0;
  int plane[3] = {0, 0, 0};
  constexpr int SA = S == 1 ? 3 : 1, SB = S == 9 ? 3 : 9;
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const int i = k * S + a * SA + b * SB;
        const int g = diff2<S>(s, i);
        sq[k] += (long long)g * g;
        gf += (long long)g * s[i];
        // values lie in [-2^28, 2^25]: moved up by 2^27, nine of them fit
        plane[k] += s[i] + (1 << 27);
      }
  const double q0 = i64_to_double(sq[0]), q1 = i64_to_double(sq[1]), q2 = i64_to_double(sq[2]);
  square = q0 + q1 + q2;
  right = fma(-p[2], q2, fma(-p[1], q1, fma(-p[0], q0, i64_to_double(2 * gf))));
  const double f0 = i32_to_double(plane[0]), f1 = i32_to_double(plane[1]), f2 = i32_to_double(plane[2]);
  const double d0 = f0 - f1, d2 = f1 - f2;  // half the end planes' sums
  first = d0 + d2;                          // the middle plane's sum, a third of all
  moved = fma(2.0, fma(p[2], d2, p[0] * d0), p[1] * first);
}

// The normal matrix and right side of the planes [g, -2 | 2 f - g.p] (g twice
// the differences, f the values, in units; p in steps): those of
// NodeCalcNode's planes times two, hence the same solution, its value in units.
__device__ __forceinline__ void integer_normal(const int (&s)[27], const double (&px)[3], const double (&py)[3],
                                               const double (&pz)[3], double (&A)[4][4], double (&B)[4]) {
  double right[3], first[3], moved[3];
  axis_sums<1>(s, px, A[0][0], right[0], first[0], moved[0]);
  axis_sums<3>(s, py, A[1][1], right[1], first[1], moved[1]);
  axis_sums<9>(s, pz, A[2][2], right[2], first[2], moved[2]);
  double u[3], v[3];
  cross_sums<1, 3>(s, A[0][1], u, v);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    right[0] = fma(-py[k], v[k], right[0]);
    right[1] = fma(-px[k], u[k], right[1]);
  }
  cross_sums<1, 9>(s, A[0][2], u, v);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    right[0] = fma(-pz[k], v[k], right[0]);
    right[2] = fma(-px[k], u[k], right[2]);
  }
  cross_sums<3, 9>(s, A[1][2], u, v);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    right[1] = fma(-pz[k], v[k], right[1]);
    right[2] = fma(-py[k], u[k], right[2]);
  }
  long long f = 0;
#pragma unroll
  for (int i = 0; i < 27; ++i) f += s[i];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    A[r][3] = -6.0 * first[r];  // -2 times the sum of the differences
    B[r] = -right[r];
  }
  A[3][3] = 108.0;
  B[3] = 2.0 * (i64_to_double(2 * f) - (moved[0] + moved[1] + moved[2]));
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < r; ++c) A[r][c] = A[c][r];
}

constexpr int kQefThreads = 64;

// LDL^T factorisation of the symmetric 4x4 A (no pivoting): pivots d, their
// reciprocals id, and M = L^-1 (unit lower triangular), so that
// A^-1 = M^T diag(id) M.  Returns 0 if a pivot is below `floor`, 1 otherwise.
__device__ int ldlt4(const double A[4][4], double floor, double d[4], double id[4], double M[4][4]) {
  double L[4][4] = {{1, 0, 0, 0}, {0, 1, 0, 0}, {0, 0, 1, 0}, {0, 0, 0, 1}};
  for (int j = 0; j < 4; ++j) {
    double dj = A[j][j];
    for (int k = 0; k < j; ++k) dj -= L[j][k] * L[j][k] * d[k];
    if (!(dj >= floor)) return 0;
    d[j] = dj;
    id[j] = 1.0 / dj;
    for (int i = j + 1; i < 4; ++i) {
      double l = A[i][j];
      for (int k = 0; k < j; ++k) l -= L[i][k] * L[j][k] * d[k];
      L[i][j] = l * id[j];
    }
  }
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) M[i][j] = i == j ? 1.0 : 0.0;
  for (int i = 1; i < 4; ++i)
    for (int j = 0; j < i; ++j) {
      double v = -L[i][j];
      for (int k = j + 1; k < i; ++k) v -= L[i][k] * M[k][j];
      M[i][j] = v;
    }
  return 1;
}

// The leaves of the level [lb, le), as offsets node - lb, so that k_qef's
// threads are all leaves: the FP64 pipe issues per warp instruction, and a
// thread that has no leaf would leave its lane of every FP64 instruction
// idle (on a level with few leaves most of them).  One atomic per warp;
// list[0] counts the leaves and they follow from list[1] (each warp's in
// node order; each leaf's result does not depend on the order).
__global__ void k_qef_pick(const int8_t* __restrict__ nd_type, long long lb, long long le, int* __restrict__ list) {
  launch_wait();
  const long long node = lb + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool leaf = node < le && nd_type[node] == Q_LEAF;
  const unsigned m = __ballot_sync(0xffffffffu, leaf);
  if (m == 0u) return;  // warp-uniform
  int base = 0;
  if (lane == 0) base = atomicAdd(list, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (leaf) list[1 + base + __popc(m & ((1u << lane) - 1u))] = (int)(node - lb);
}

// The same matrix from FP64 sums, for leaves whose values are not integers of
// the unit within range (or not finite).
__device__ __noinline__ void fp64_normal(const float* sv, const double (&px)[3], const double (&py)[3],
                                         const double (&pz)[3], double (&A)[4][4], double (&B)[4]) {
  double sd[27];
#pragma unroll
  for (int i = 0; i < 27; ++i) sd[i] = f2d_exact(sv[i]);
  // GridEval's finite differences (src/evaluator.cpp:185-240) are g = d / step
  // (one-sided) and g = d / (2 step) (central), d a difference of samples.
  // NodeCalcNode's residual of plane i at (x, v) is g.(x - p) - v + f, which
  // with y = x / step and q = p / step reads d'.(y - q) - v + f, d' = d or
  // d / 2: the same least-squares problem in the variables (y, v), solved
  // below and mapped back by x = step y.  So no sample difference is scaled
  // by the step; the central ones are halved on the integer pipe, and only
  // the nine lattice coordinates are multiplied (FP64 instructions bound this
  // kernel).  The pseudo-inverse rule sees the same equilibrated matrix: a
  // diagonal change of variables cancels in D A D.
  //
  // The plane's -1 entry makes q[3], q[7], q[10] minus the sums of the
  // differences over the 27 samples.  Along one row of three samples
  // s0, s1, s2 those are (s0 - s1) + (s0 - s2) / 2 + (s1 - s2) = 3 times the
  // central one, so each is taken as -3 times the sum over the 9 central
  // samples of its axis.
  double q[15];
  double cx = 0.0, cy = 0.0, cz = 0.0;
#pragma unroll
  for (int k = 0; k < 15; ++k) q[k] = 0.0;
#pragma unroll
  for (int i = 0; i < 27; ++i) {
    const int x = i % 3, y = (i / 3) % 3, z = i / 9;
    const double qx = px[x], qy = py[y], qz = pz[z];
    auto fd = [&](int d, int stride) {
      if (d == 0) return sd[i] - sd[i + stride];
      if (d == 2) return sd[i - stride] - sd[i];
      return half_exact(sd[i - stride] - sd[i + stride]);
    };
    const double gx = fd(x, 1), gy = fd(y, 3), gz = fd(z, 9);
    // plane [d', -1, f - q.d'] accumulated as QEFNormal::combineSelf
    const double w = fma(-qz, gz, fma(-qy, gy, fma(-qx, gx, sd[i])));
    const double pl[5] = {gx, gy, gz, -1.0, w};
    if (x == 1) cx += gx;
    if (y == 1) cy += gy;
    if (z == 1) cz += gz;
    int idx = 0;
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int s2 = r; s2 < 5; ++s2, ++idx)
        if (idx != 3 && idx != 7 && idx != 10 && idx != 12) q[idx] += pl[r] * pl[s2];
  }
  q[3] = -3.0 * cx;
  q[7] = -3.0 * cy;
  q[10] = -3.0 * cz;
  q[12] = 27.0;  // the (-1) x (-1) entry: 27 ones
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int idx = ((2 * 4 + 3 - r) * r) / 2;
#pragma unroll
    for (int s2 = r; s2 < 4; ++s2) A[r][s2] = A[s2][r] = q[idx + s2 - r];
    B[r] = -q[idx + 4 - r];
  }
}

// Solves a leaf: 1 with the vertex and the planes' value in v if it lies in the
// cell, 0 if not, -1 if the system is singular.
__device__ __forceinline__ int qef_vertex(const QefArgs& a, long long node, const float4* __restrict__ nd_c,
                                          const float* __restrict__ nd_samp, float4& v) {
  const float4 c = nd_c[node];
  const float h = c.w;
  const float mn[3] = {__fsub_rn(c.x, h), __fsub_rn(c.y, h), __fsub_rn(c.z, h)};
  const float mx[3] = {__fadd_rn(c.x, h), __fadd_rn(c.y, h), __fadd_rn(c.z, h)};
  const float* sv = nd_samp + node * 27;
  // sample positions (GenerateSampling): three per axis, in units of the
  // finite-difference step (times 1 / step, see below)
  const double i1 = a.i1;
  auto lattice = [&](int ax, int k) {
    return f2d_exact(__fadd_rn(__fmul_rn(1.0f - k * 0.5f, mn[ax]), __fmul_rn(k * 0.5f, mx[ax]))) * i1;
  };
  const double px[3] = {lattice(0, 0), lattice(0, 1), lattice(0, 2)};
  const double py[3] = {lattice(1, 0), lattice(1, 1), lattice(1, 2)};
  const double pz[3] = {lattice(2, 0), lattice(2, 1), lattice(2, 2)};
  double A[4][4], B[4];
  double vunit = 1.0;  // the solution's value is in this unit
  // the leaf's unit: the frame's, or the ulp of its smallest value where that is
  // coarser (all its values are multiples of it)
  float low = fabsf(sv[0]), si_f[27];
#pragma unroll
  for (int i = 0; i < 27; ++i) {
    si_f[i] = sv[i];
    low = fminf(low, fabsf(si_f[i]));
  }
  const int eu = max(a.unit_exp, (__float_as_int(low) >> 23) - 23);  // biased exponent of the unit
  const float inv_unit = __int_as_float((254 - eu) << 23);
  int si[27];
  bool whole = eu > 0 && eu < 254;
#pragma unroll
  for (int i = 0; i < 27; ++i) {
    const float m = si_f[i] * inv_unit;  // exact: a power of two
    whole = whole && m >= (float)kSampleLow && m <= (float)kSampleHigh;
    si[i] = (int)m;
  }
  if (whole) {
    integer_normal(si, px, py, pz, A, B);
    vunit = f2d_exact(__int_as_float(eu << 23));
  } else {
    fp64_normal(sv, px, py, pz, A, B);
  }
  // Equilibrate: the gradient rows are ~|f| / step while the w column is 1,
  // so A's condition number exceeds what FP32 or even FP64 resolves.  With
  // a positive diagonal D close to diag(A_ii)^-1/2 the solve is
  // (D A D) y = D B, x = D y: the same minimiser in exact arithmetic for any
  // such D, well conditioned unless the planes are degenerate.  D is taken
  // from the FP32 reciprocal square root (two conversions instead of an FP64
  // square root and division); the equilibrated diagonal is then 1 to about
  // 1e-7, and dmax, its largest entry, bounds the largest eigenvalue from
  // below.
  double D[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) D[r] = equil_scale(A[r][r]);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    B[r] *= D[r];
#pragma unroll
    for (int s2 = r; s2 < 4; ++s2) A[r][s2] = A[s2][r] = A[r][s2] * (D[r] * D[s2]);
  }
  const double dmax = fmax(fmax(A[0][0], A[1][1]), fmax(A[2][2], A[3][3]));
  // Pseudo-inverse rule: eigenvalues at most 1e-12 * max |eigenvalue| are
  // dropped, and a system with a dropped eigenvalue counts as singular (the
  // reference's Matrix4f::inverse gives non-finite values there and the
  // vertex is rejected).  Decided without an eigen-decomposition where the
  // bounds settle it: the smallest eigenvalue is at most every LDL^T pivot,
  // and at least min(d) / ||M||_F^2 and 1 / ||A^-1||_F (A^-1 = M^T D^-1 M,
  // so ||A^-1||_2 <= ||M||_2^2 / min(d)), while the largest lies in
  // [dmax, trace].  The first lower bound costs a few instructions and
  // settles the dam-break leaves with a margin of 1e6 or more; the second
  // needs the whole inverse and is the fallback.
  const double tr = A[0][0] + A[1][1] + A[2][2] + A[3][3];
  bool singular, solved = false;
  double xs[4] = {0.0, 0.0, 0.0, 0.0};
  double dd[4], id[4], M[4][4];
  const int ok = tr > 0.0 ? ldlt4(A, 1e-12 * dmax, dd, id, M) : 0;
  if (!(tr > 0.0) || !ok) {
    singular = true;  // a pivot below 1e-12 dmax <= 1e-12 * max eigenvalue
    solved = true;
  } else {
    singular = false;
    double m2 = 4.0;
#pragma unroll
    for (int r = 1; r < 4; ++r)
#pragma unroll
      for (int c2 = 0; c2 < r; ++c2) m2 = fma(M[r][c2], M[r][c2], m2);
    const double dmin = fmin(fmin(dd[0], dd[1]), fmin(dd[2], dd[3]));
    const double t = 1e-12 * tr;
    if (dmin > t * m2) {
      // x = M^T D^-1 M B: forward product, scaling, back product
      double z[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        double v = B[r];
#pragma unroll
        for (int k = 0; k < r; ++k) v = fma(M[r][k], B[k], v);
        z[r] = v * id[r];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        double v = z[r];
#pragma unroll
        for (int k = r + 1; k < 4; ++k) v = fma(M[k][r], z[k], v);
        xs[r] = v;
      }
      solved = true;
    } else {
      double Ai[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c2 = r; c2 < 4; ++c2) {
          double v = 0.0;
#pragma unroll
          for (int k = c2; k < 4; ++k) v += M[k][r] * id[k] * M[k][c2];
          Ai[r][c2] = Ai[c2][r] = v;
        }
      double f2 = 0.0, f2o = 0.0;  // ||A^-1||_F^2: diagonal, twice the upper part
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        f2 = fma(Ai[r][r], Ai[r][r], f2);
#pragma unroll
        for (int s2 = r + 1; s2 < 4; ++s2) f2o = fma(Ai[r][s2], Ai[r][s2], f2o);
      }
      f2 = fma(2.0, f2o, f2);
      if (f2 * t * t < 1.0) {  // smallest eigenvalue > 1e-12 * trace >= tolerance
#pragma unroll
        for (int r = 0; r < 4; ++r) xs[r] = Ai[r][0] * B[0] + Ai[r][1] * B[1] + Ai[r][2] * B[2] + Ai[r][3] * B[3];
        solved = true;
      }
    }
  }
  if (!solved) {
    // borderline conditioning: the eigen-decomposition decides
    double w[4], V[4][4];
    sym_eig4(A, w, V);
    double wmax = 0.0;
    for (int k = 0; k < 4; ++k) wmax = fmax(wmax, fabs(w[k]));
    const double tol = 1e-12 * wmax;
    singular = !(wmax > 0.0);
    for (int k = 0; k < 4; ++k) {
      if (fabs(w[k]) <= tol) {
        singular = true;
        continue;
      }
      double proj = 0.0;
      for (int r = 0; r < 4; ++r) proj += V[r][k] * B[r];
      proj /= w[k];
      for (int r = 0; r < 4; ++r) xs[r] += V[r][k] * proj;
    }
  }
  if (singular) return -1;
#pragma unroll
  for (int r = 0; r < 4; ++r) xs[r] *= D[r];
#pragma unroll
  for (int r = 0; r < 3; ++r) xs[r] *= a.step;  // x = step y
  bool in_cell = true;
#pragma unroll
  for (int r = 0; r < 3; ++r) in_cell = in_cell && xs[r] >= f2d_exact(mn[r]) && xs[r] <= f2d_exact(mx[r]);
  if (!in_cell) return 0;
  v = make_float4((float)xs[0], (float)xs[1], (float)xs[2], (float)(xs[3] * vunit));
  return 1;
}

constexpr int kAccepted = 1 << 31;  // mark of a list entry

// One thread per listed leaf: the vertex and whether it lies in the cell.  An
// accepted leaf's node gets the vertex and the planes' value there and its entry
// of the list is marked for k_qef_accept; the others keep their node.
// counters: singular systems, leaves solved
__global__ void __launch_bounds__(kQefThreads, 8) k_qef(QefArgs a, const int* __restrict__ count_ptr,
                                                        const int* __restrict__ start, int* __restrict__ list,
                                                        float4* __restrict__ nd_v,
                                                        const float4* __restrict__ nd_c,
                                                        const float* __restrict__ nd_samp,
                                                        unsigned long long* __restrict__ counters) {
  launch_wait();
  const int count = *count_ptr;
  if (start) list += *start;
  for (int t = blockIdx.x * kQefThreads + threadIdx.x; t < count; t += gridDim.x * kQefThreads) {
    const unsigned am = __activemask();  // the warp's lanes that hold a leaf
    if ((int)(threadIdx.x & 31) == __ffs(am) - 1) stripe_add(counters, C_QEF_LEAVES, (unsigned long long)__popc(am));
    const int leaf = list[t];
    const long long node = a.lb + leaf;
    float4 v;
    const int verdict = qef_vertex(a, node, nd_c, nd_samp, v);
    if (verdict < 0) stripe_add(counters, C_QEF_SINGULAR, 1ull);
    if (verdict > 0) {
      nd_v[node] = v;
      list[t] = leaf | kAccepted;
    }
  }
}

// The accepted leaves, a warp each: calcErrorDMC (src/iso_method_ours.cpp:40-50)
// with GridEval's float gradients, float as in the reference, a sample a lane
// and the sum in sample order; then SingleEval at the vertex, 32 candidates at a
// time, the terms added in candidate order.  In k_qef a lane did this alone for
// hundreds of candidates while its warp waited: a few accepted leaves made the
// coarse levels of a 500k-particle sheets frame take 965, 809 and 518 us.
// counters: QEF vertices accepted, field evaluations
__global__ void __launch_bounds__(128) k_qef_accept(QefArgs a, const int* __restrict__ count_ptr,
                                                    const int* __restrict__ start, const int* __restrict__ list,
                                                    float4* __restrict__ nd_v, const float4* __restrict__ nd_c,
                                                    const float* __restrict__ nd_samp,
                                                    unsigned long long* __restrict__ counters) {
  launch_wait();
  const int lane = threadIdx.x & 31;
  const int count = *count_ptr;
  if (start) list += *start;
  unsigned long long done = 0;
  // a warp takes 8 entries at a time: enough to skim the list, few enough to
  // spread a run of accepted ones
  for (int t0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 8; t0 < count; t0 += gridDim.x * 32) {
    const int entry = lane < 8 && t0 + lane < count ? list[t0 + lane] : 0;
    unsigned todo = __ballot_sync(0xffffffffu, entry < 0);
    for (; todo; todo &= todo - 1u) {
      const long long node = a.lb + (__shfl_sync(0xffffffffu, entry, __ffs(todo) - 1) & ~kAccepted);
      const float4 c = nd_c[node];
      float4 v = nd_v[node];
      const float h = c.w;
      const float cellsize = 2.0f * h;
      const float step = cellsize / 2;
      float term = 0.f;
      {
        const int i = min(lane, 26);
        const float mn[3] = {__fsub_rn(c.x, h), __fsub_rn(c.y, h), __fsub_rn(c.z, h)};
        const float mx[3] = {__fadd_rn(c.x, h), __fadd_rn(c.y, h), __fadd_rn(c.z, h)};
        const float* sv = nd_samp + node * 27;
        const int x = i % 3, y = (i / 3) % 3, z = i / 9;
        const float px = __fadd_rn(__fmul_rn(1.0f - x * 0.5f, mn[0]), __fmul_rn(x * 0.5f, mx[0]));
        const float py = __fadd_rn(__fmul_rn(1.0f - y * 0.5f, mn[1]), __fmul_rn(y * 0.5f, mx[1]));
        const float pz = __fadd_rn(__fmul_rn(1.0f - z * 0.5f, mn[2]), __fmul_rn(z * 0.5f, mx[2]));
        auto fdf = [&](int d, int stride) {
          if (d == 0) return (sv[i] - sv[i + stride]) / step;
          if (d == 2) return (sv[i - stride] - sv[i]) / step;
          return (sv[i - stride] - sv[i + stride]) / (step * 2);
        };
        const float gx = fdf(x, 1), gy = fdf(y, 3), gz = fdf(z, 9);
        const float d = gx * (v.x - px) + gy * (v.y - py) + gz * (v.z - pz) - v.w;
        term = d * d / (1.0f + gx * gx + gy * gy + gz * gz);
      }
      float err = 0.0f;
      for (int i = 0; i < 27; ++i) err = __fadd_rn(err, __shfl_sync(0xffffffffu, term, i));
      v.w = a.iso - field_sum_warp(a.g, a.P, v.x, v.y, v.z);
      // leaf by size keeps the zeroing (no SingleEval follows it)
      const bool leaf_by_size = cellsize - a.radius < kAbove1em8;
      if (leaf_by_size && err / cellsize < 0.0001f) v.w = 0.0f;
      if (lane == 0) nd_v[node] = v;
      ++done;
    }
  }
  if (lane == 0) {
    stripe_add(counters, C_QEF_EVALS, done);
    stripe_add(counters, C_QEF_ACCEPTED, done);
  }
}

// On the context's QEF stream, after the level's classification on the
// context stream: the FP64 pipe is busy with these leaves while the FP32
// pipes run the next level's sampling (or the mesh topology after the last
// level).  The leaf list is the QEF stream's own, allocated and freed in its
// order.
void qef_level(pi_frame* f, long long lb, long long le, int depth, int parts, int part) {
  pi_ctx* c = f->ctx;
  cudaStream_t s = c->qef_stream;
  PI_CUDA(cudaEventRecord(c->ev_qef_in, c->stream));
  PI_CUDA(cudaStreamWaitEvent(s, c->ev_qef_in, 0));
  f->qef_inflight = true;
  DBuf<int> list;
  const long long nl = le - lb;
  if (!parts) list.alloc(c, s, nl + 1);
  const GridHost& gh = f->g;
  // half size of the level's nodes (the root's halved exactly per level);
  // the step of GridEval is cellsize / 2 = that half size
  const float step = std::ldexp(f->rootH, -depth);
  // half an ulp of the iso value: 2^-24 of its power of two (where that is no
  // normal float, every leaf takes the FP64 sums)
  int iso_exp = 0;
  std::frexp(f->iso, &iso_exp);  // iso in [2^(iso_exp - 1), 2^iso_exp)
  const int unit_exp = std::isfinite(f->iso) && f->iso > 0.f ? std::max(0, iso_exp - 25 + 127) : 0;
  QefArgs qa{GridView{gh.bounding[0], gh.bounding[2], gh.bounding[4], gh.cell, gh.nx, gh.ny, gh.nz, f->off.p},
             PartView{f->pos.p, f->xm.p, f->ga.p, f->gb.p, f->xlo.p},
             f->iso,
             f->P.radius,
             lb,
             le,
             (double)step,
             1.0 / (double)step,
             unit_exp};
  // the leaves: the level's, listed here, or the part's nodes (on the leaf
  // level each becomes a leaf)
  const int* count = parts ? f->plist.p + part : list.p;
  const int* start = parts ? f->plist.p + 2 * (parts + 1) + part : nullptr;
  int* const leaves = parts ? f->pnodes.p : list.p + 1;
  if (!parts) {
    PI_CUDA(cudaMemsetAsync(list.p, 0, sizeof(int), s));
    PI_LAUNCH(k_qef_pick, div_up(nl, 256), 256, 0, s, f->nd_type.p, lb, le, list.p);
  }
  const long long share = part_share(nl, parts);
  prof_begin(f->ctx, s, PG_QEF);
  PI_LAUNCH(k_qef, div_up(share, kQefThreads), kQefThreads, 0, s, qa, count, start, leaves, f->nd_v.p, f->nd_c.p,
            f->nd_samp.p, f->dcount.p);
  PI_LAUNCH(k_qef_accept, (int)std::min<long long>(div_up(share, 32), 8LL * c->smCount), 128, 0, s, qa, count, start,
            (const int*)leaves, f->nd_v.p, f->nd_c.p, f->nd_samp.p, f->dcount.p);
  prof_end(f->ctx, s, PG_QEF);
  list.release();
  PI_CUDA(cudaEventRecord(c->ev_qef_done, s));
}

void qef_join(pi_frame* f) {
  if (!f->qef_inflight) return;
  PI_CUDA(cudaStreamWaitEvent(f->ctx->stream, f->ctx->ev_qef_done, 0));
  f->qef_inflight = false;
}

}  // namespace pisurf
