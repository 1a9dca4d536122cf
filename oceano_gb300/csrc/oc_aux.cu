// Cell-local kernels around the stage: transport speed (dt), velocity
// projection, vorticity indicator and L2 projection of the vortex.  One
// thread per cell, FP64, runtime degree; tables from this unit's constant copy.
#include "oc_kernels.cuh"

namespace oc {

// ---------------------------------------------------------------------------
// Transport speed (OceanDG.h:2505-2580): max over cells and Gauss-Lobatto p+2 points of
// sigma_max(J^-1) sqrt(g h) + |J^-1 u|_inf, sigma_max by the reference's five power
// iterations.  The result is FP64, but GB300 runs FP64 at 1/64 of the FP32 rate, and
// one FP64 evaluation per point cost 201 us on the 320x160 degree-3 mesh, against 9 us
// for reading the state.  So a first kernel bounds every point's speed from above and
// below in FP32, and only the points whose upper bound reaches the largest lower bound
// (of the mesh, or of the cell where every cell's speed is wanted) are evaluated in
// FP64 by a second one; sigma_max depends on the mesh alone and is computed once.  Five
// steps and one estimate, before -> after, us: 320x160 cells of degree 3 671 -> 489,
// 151x67 of degree 4 541 -> 377, random hp mesh 1441 -> 1158, 250x10 channel 238 -> 215.
// ---------------------------------------------------------------------------
__global__ void cell_sigma_kernel(int n, const double *geo, double *sigma) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const double *J = geo + 11 * (int64_t)c;
  double e0 = 1., e1 = 1.;
  for (int it = 0; it < 5; ++it) {
    const double a0 = J[6] * e0 + J[7] * e1, a1 = J[8] * e0 + J[9] * e1;
    e0 = J[6] * a0 + J[8] * a1;
    e1 = J[7] * a0 + J[9] * a1;
    double nrm = 0;
    nrm = mx<double>(nrm, fabs(e0));
    nrm = mx<double>(nrm, fabs(e1));
    e0 /= nrm;
    e1 /= nrm;
  }
  const double j0 = J[6] * e0 + J[7] * e1, j1 = J[8] * e0 + J[9] * e1;
  sigma[c] = sqrt((j0 * j0 + j1 * j1) / (e0 * e0 + e1 * e1));
}

// x rounded towards zero to FP32, by integer operations (values below the FP32 normal
// range count as zero, those above it as infinite, NaN stays)
__device__ __forceinline__ float truncated(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const unsigned ha = h & 0x7fffffffu;
  if (ha >= 0x47f00000u) return x != x ? __int_as_float(0x7fffffff)
                                          : __uint_as_float(0x7f800000u | (h & 0x80000000u));
  return __uint_as_float(
      ha < 0x38100000u ? 0u
                       : ((((h << 3) | (l >> 29)) & 0x7fffffffu) ^ 0x40000000u) | (h & 0x80000000u));
}

// Bounds of one cell: up, the largest upper bound of its points' speeds (infinite where a
// value is not finite); lo, the largest lower bound; mask, the points (gy G + gx) whose
// upper bound reaches the lower bounds met before them (the largest speed's among them).
// With z_i and q_i rounded to 2^-23 and the shape values to 2^-24, an interpolated value
// is within (2 + 2 + 2N + 2) 2^-24 Lambda max_i |v_i| < 2e-6 Lambda max_i |v_i| of the
// exact one; everything after that is within 1e-5 relative of the bounds' own terms.
template <int P>
__device__ __forceinline__ void speed_bounds(const AuxArgs &a, int c, int64_t zo, const double *z,
                                             const double *q, float &up, float &lo,
                                             unsigned long long &mask) {
  constexpr int N = P + 1, G = P + 2, NN = N * N;
  const DegTables<float> &tb = tab<float>(P);
  float v[3][NN], m[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < NN; ++i) {
    v[0][i] = truncated(z[zo + i]);
    v[1][i] = truncated(q[2 * zo + i]);
    v[2][i] = truncated(q[2 * zo + NN + i]);
  }
#pragma unroll
  for (int e = 0; e < 3; ++e)
#pragma unroll
    for (int i = 0; i < NN; ++i) m[e] = fmaxf(m[e], fabsf(v[e][i]));
  const double *J = a.geo + 11 * (int64_t)c;
  const float J0 = (float)J[6], J1 = (float)J[7], J2 = (float)J[8], J3 = (float)J[9];
  const float sigma = (float)a.sigma[c], g = (float)a.g, cu = (float)a.cu;
  const float E = 2e-6f * tb.lebG;
  const float dz = E * m[0];
  const float dj = E * fmaxf(m[1], m[2]) * fmaxf(fabsf(J0) + fabsf(J1), fabsf(J2) + fabsf(J3));
  const double *zb1 = a.sd1 ? a.sd1 + cell_data(a.err, a.sdo1, c, a.n_sd[1], G * G) : nullptr;
  // u = q f(h) with f = sqrt(2) h / sqrt(h^4 + max(h^4, cu^4)): increasing up to cu, 1/h above
  auto f = [&](float h) {
    const float h4 = h * h * h * h, c4 = cu * cu * cu * cu;
    return 1.41421356f * h * rcp_fast(sqrt_fast(h4 + fmaxf(h4, c4)));
  };
  up = lo = 0.f;
  mask = 0ull;
#pragma unroll 1
  for (int gy = 0; gy < G; ++gy) {
    float r[3][N];
#pragma unroll
    for (int e = 0; e < 3; ++e)
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        r[e][ix] = 0.f;
#pragma unroll
        for (int iy = 0; iy < N; ++iy) r[e][ix] += tb.BG[gy][iy] * v[e][iy * N + ix];
      }
#pragma unroll
    for (int gx = 0; gx < G; ++gx) {
      float zv = 0, q0 = 0, q1 = 0;
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        const float b = tb.BG[gx][ix];
        zv += b * r[0][ix];
        q0 += b * r[1][ix];
        q1 += b * r[2][ix];
      }
      const float zb = zb1 ? (float)zb1[gy * G + gx] : 0.f;
      const float h = zv + zb, dh = dz + 1e-6f * fabsf(zb);
      const float hu = fmaxf(h + dh, 1e-12f), hl = fmaxf(h - dh, 0.f);
      float fu, fl;
      if (hl > cu) {
        fu = rcp_fast(hl);
        fl = rcp_fast(hu);
      } else {
        fu = hu < cu ? f(hu) : rcp_fast(cu);
        const float fa = f(hl), fb = f(hu);
        fl = fa <= fb ? fa : fb <= fa ? fb : 0.f;
      }
      const float cq = fmaxf(fabsf(J0 * q0 + J1 * q1), fabsf(J2 * q0 + J3 * q1));
      float pu = (sigma * sqrt_fast(g * hu) + fu * (cq + dj)) * 1.00001f;
      float pl = (sigma * sqrt_fast(g * hl) + fl * fmaxf(cq - dj, 0.f)) * 0.99999f;
      // (fmaxf drops a NaN: a value that is not finite is found in the sums)
      if (!(fabsf(h) + fabsf(q0) + fabsf(q1) + pu + pl < INFINITY)) {
        pu = INFINITY;
        pl = 0.f;
      }
      if (pu >= lo) mask |= 1ull << (gy * G + gx);
      up = fmaxf(up, pu);
      lo = fmaxf(lo, pl);
    }
  }
}

// The FP64 speed at a point from its interpolated values.  Both ways of taking a cell's points
// (masked_speed, point_speed) interpolate by the same fused multiply-adds in the same order and
// end here, out of line, so that a point's speed does not depend on the cells that share its
// warp: the largest speed is the largest of the cells' own, bit for bit.
__device__ __noinline__ double speed_at(const AuxArgs &a, int c, double zv, double q0, double q1,
                                        double zb) {
  const double *J = a.geo + 11 * (int64_t)c;
  double v0, v1;
  velocity<double>(zv, q0, q1, zb, a.cu4, v0, v1);
  const double cs0 = J[6] * v0 + J[7] * v1, cs1 = J[8] * v0 + J[9] * v1;
  double conv = 0;
  conv = mx<double>(conv, fabs(cs0));
  conv = mx<double>(conv, fabs(cs1));
  return a.sigma[c] * sqrt(a.g * depth<double>(zv, zb)) + conv;
}

// FP64 speeds of the masked points of a cell: their maximum, or -1 where one is not finite
template <int P>
__device__ __forceinline__ double masked_speed(const AuxArgs &a, int c, int64_t zo,
                                               const double *z, const double *q,
                                               unsigned long long mask) {
  constexpr int N = P + 1, G = P + 2, NN = N * N;
  const DegTables<double> &tb = tab<double>(P);
  const double *zb1 = a.sd1 ? a.sd1 + cell_data(a.err, a.sdo1, c, a.n_sd[1], G * G) : nullptr;
  double local = 0;
  bool nonfinite = false;
#pragma unroll 1
  for (int gy = 0; gy < G; ++gy) {
    const unsigned row = (unsigned)(mask >> (gy * G)) & ((1u << G) - 1u);
    if (!row) continue;
    double r[3][N];
#pragma unroll
    for (int ix = 0; ix < N; ++ix) {
      r[0][ix] = r[1][ix] = r[2][ix] = 0;
#pragma unroll
      for (int iy = 0; iy < N; ++iy) {
        const double b = tb.BG[gy][iy];
        r[0][ix] = fma(b, z[zo + iy * N + ix], r[0][ix]);
        r[1][ix] = fma(b, q[2 * zo + iy * N + ix], r[1][ix]);
        r[2][ix] = fma(b, q[2 * zo + NN + iy * N + ix], r[2][ix]);
      }
    }
#pragma unroll 1
    for (int gx = 0; gx < G; ++gx) {
      if (!((row >> gx) & 1u)) continue;
      double zv = 0, q0 = 0, q1 = 0;
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        const double b = tb.BG[gx][ix];
        zv = fma(b, r[0][ix], zv);
        q0 = fma(b, r[1][ix], q0);
        q1 = fma(b, r[2][ix], q1);
      }
      const double sp = speed_at(a, c, zv, q0, q1, zb1 ? zb1[gy * G + gx] : 0.);
      // std::max keeps the running maximum when sp is NaN: check every point
      if (!isfinite(sp)) nonfinite = true;
      local = mx<double>(local, sp);
    }
  }
  return nonfinite || !isfinite(local) ? -1. : local;
}

// The cell of a thread: on a mesh of several degrees the blocks run over the concatenated
// degree groups, so that the cells of a warp have one degree (random hp mesh: bounds
// 81 us in index order); -1 past the end.
__device__ __forceinline__ int grouped_cell(const AuxArgs &a) {
  if (!a.group_cells[0]) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    return c < a.n_cells ? c : -1;
  }
  int b = blockIdx.x, k = 0;
  while (k < OC_MAXDEG - 1 && b >= a.group_blocks[k]) b -= a.group_blocks[k++];
  const int i = b * blockDim.x + threadIdx.x;
  return i < a.group_n[k] ? (int)checked(a.err, a.group_cells[k][i], a.n_cells, BS_CELL) : -1;
}

// lower: FP32 bits of the largest lower bound (non-negative, ordered like the values)
__global__ void __launch_bounds__(64) speed_bounds_kernel(const AuxArgs a, const double *z,
                                                          const double *q, float *up,
                                                          unsigned long long *mask,
                                                          unsigned *lower) {
  const int c = grouped_cell(a);
  float lo = 0.f;
  if (c >= 0) {
    const int p = checked_degree(a.err, a.deg[c]), N = p + 1;
    const int64_t zo = checked(a.err, a.off[c], a.n_dofs - N * N + 1, BS_OFFSET);
    float u = 0.f;
    unsigned long long m = 0ull;
    switch (p) {
      case 1: speed_bounds<1>(a, c, zo, z, q, u, lo, m); break;
      case 2: speed_bounds<2>(a, c, zo, z, q, u, lo, m); break;
      case 3: speed_bounds<3>(a, c, zo, z, q, u, lo, m); break;
      default: speed_bounds<4>(a, c, zo, z, q, u, lo, m); break;
    }
    up[c] = u;
    mask[c] = m;
  }
  const unsigned w = __reduce_max_sync(OC_FULL, __float_as_uint(lo));
  if ((threadIdx.x & 31) == 0 && w > 0u) atomicMax(lower, w);
}

// FP64 speed at point k = gy G + gx of a cell (rolled: a warp that comes here alone would
// otherwise wait for its instructions, 69 us for a few cells)
__device__ __forceinline__ double point_speed(const AuxArgs &a, int c, int p, int64_t zo,
                                              const double *z, const double *q, int k) {
  const int N = p + 1, G = p + 2, gy = k / G, gx = k - gy * G;
  const double *by = &a.gtabd[p - 1].BG[gy][0], *bx = &a.gtabd[p - 1].BG[gx][0];
  double zv = 0, q0 = 0, q1 = 0;
#pragma unroll 1
  for (int ix = 0; ix < N; ++ix) {
    double r0 = 0, r1 = 0, r2 = 0;
#pragma unroll 1
    for (int iy = 0; iy < N; ++iy) {
      const int64_t i = zo + iy * N + ix;
      r0 = fma(by[iy], z[i], r0);
      r1 = fma(by[iy], q[zo + i], r1);
      r2 = fma(by[iy], q[zo + N * N + i], r2);
    }
    zv = fma(bx[ix], r0, zv);
    q0 = fma(bx[ix], r1, q0);
    q1 = fma(bx[ix], r2, q1);
  }
  return speed_at(a, c, zv, q0, q1,
                  a.sd1 ? a.sd1[cell_data(a.err, a.sdo1, c, a.n_sd[1], G * G) + k] : 0.);
}

// The largest speed (atomicMax on the bits of a non-negative double), or with per_cell the
// largest speed of every cell; a point that is not finite raises the error flag and its
// cell counts as 0.  Up to kFewCells cells of a warp are taken one after the other, the
// lanes at their points; more (a flow whose speeds tie) by one thread each.
constexpr int kFewCells = 6;
__global__ void __launch_bounds__(64) speed_kernel(const AuxArgs a, const double *z,
                                                   const double *q, const float *up,
                                                   const unsigned long long *mask,
                                                   const unsigned *lower,
                                                   unsigned long long *out, double *per_cell) {
  const int c = grouped_cell(a), lane = threadIdx.x & 31;
  const bool take = c >= 0 && (per_cell || up[c] >= __uint_as_float(*lower));
  unsigned todo = __ballot_sync(OC_FULL, take);
  if (!todo) return;
  double local = 0;
  int p = 1;
  int64_t zo = 0;
  unsigned long long m = 0ull;
  if (take) {
    p = checked_degree(a.err, a.deg[c]);
    zo = checked(a.err, a.off[c], a.n_dofs - (p + 1) * (p + 1) + 1, BS_OFFSET);
    m = mask[c];
  }
  if (__popc(todo) <= kFewCells) {
    for (; todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const int cc = __shfl_sync(OC_FULL, c, src), pp = __shfl_sync(OC_FULL, p, src);
      const int64_t zz = __shfl_sync(OC_FULL, zo, src);
      const unsigned long long mm = __shfl_sync(OC_FULL, m, src);
      double sp = 0;
      bool bad = false;
      for (int k = lane; k < (pp + 2) * (pp + 2); k += 32)
        if ((mm >> k) & 1ull) {
          const double v = point_speed(a, cc, pp, zz, z, q, k);
          // std::max keeps the running maximum when v is NaN: check every point
          bad |= !isfinite(v);
          sp = mx<double>(sp, v);
        }
      for (int o = 16; o > 0; o >>= 1) sp = mx<double>(sp, __shfl_xor_sync(OC_FULL, sp, o));
      if (__any_sync(OC_FULL, bad)) sp = -1.;
      if (lane == src) local = sp;
    }
  } else if (take) {
    switch (p) {
      case 1: local = masked_speed<1>(a, c, zo, z, q, m); break;
      case 2: local = masked_speed<2>(a, c, zo, z, q, m); break;
      case 3: local = masked_speed<3>(a, c, zo, z, q, m); break;
      default: local = masked_speed<4>(a, c, zo, z, q, m); break;
    }
  }
  if (take) {
    if (local < 0) {
      atomicOr(a.err, ERR_NONFINITE);
      local = 0;
    }
    if (per_cell) per_cell[c] = local;
    if (local > 0) atomicMax(out, (unsigned long long)__double_as_longlong(local));
  }
}

// Values of the cell's fields at a row qy of Gauss p+1 points and the velocity there
// (OceanDG.h:2599-2662): call(qx, zeta, q0, q1, u, v) per point.
template <int P, class Fn>
__device__ __forceinline__ void velocity_row(const AuxArgs &a, const double *zc, const double *qc,
                                             const double *sd, int qy, Fn call) {
  constexpr int N = P + 1, NN = N * N;
  const DegTables<double> &tb = tab<double>(P);
  double r[3][N];
#pragma unroll
  for (int ix = 0; ix < N; ++ix) {
    r[0][ix] = r[1][ix] = r[2][ix] = 0;
#pragma unroll
    for (int iy = 0; iy < N; ++iy) {
      const double b = tb.BM[qy][iy];
      r[0][ix] += b * zc[iy * N + ix];
      r[1][ix] += b * qc[iy * N + ix];
      r[2][ix] += b * qc[NN + iy * N + ix];
    }
  }
#pragma unroll
  for (int qx = 0; qx < N; ++qx) {
    double zv = 0, q0 = 0, q1 = 0;
#pragma unroll
    for (int ix = 0; ix < N; ++ix) {
      const double b = tb.BM[qx][ix];
      zv += b * r[0][ix];
      q0 += b * r[1][ix];
      q1 += b * r[2][ix];
    }
    double u, v;
    velocity<double>(zv, q0, q1, sd ? sd[2 * (qy * N + qx)] : 0., a.cu4, u, v);
    call(qx, zv, q0, q1, u, v);
  }
}

// OceanDG.h:2599-2662 (degree >= 1 path): u = S^-1 (velocity at Gauss p+1), sum-factorised,
// one thread per cell
template <int P>
__device__ __forceinline__ void velocity_cell(const AuxArgs &a, int c, int64_t zo, const double *z,
                                              const double *q, double *u) {
  constexpr int N = P + 1, NN = N * N;
  const DegTables<double> &tb = tab<double>(P);
  const double *sd = a.sd2 ? a.sd2 + cell_data(a.err, a.sdo2, c, a.n_sd[2], 2 * NN) : nullptr;
  double o[2][NN];
#pragma unroll
  for (int i = 0; i < NN; ++i) o[0][i] = o[1][i] = 0;
#pragma unroll 1
  for (int qy = 0; qy < N; ++qy) {
    double r0[N], r1[N];
#pragma unroll
    for (int ix = 0; ix < N; ++ix) r0[ix] = r1[ix] = 0;
    velocity_row<P>(a, z + zo, q + 2 * zo, sd, qy,
                    [&](int qx, double, double, double, double u0, double u1) {
#pragma unroll
                      for (int ix = 0; ix < N; ++ix) {
                        r0[ix] += tb.Sinv[ix][qx] * u0;
                        r1[ix] += tb.Sinv[ix][qx] * u1;
                      }
                    });
#pragma unroll
    for (int iy = 0; iy < N; ++iy)
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        o[0][iy * N + ix] += tb.Sinv[iy][qy] * r0[ix];
        o[1][iy * N + ix] += tb.Sinv[iy][qy] * r1[ix];
      }
  }
#pragma unroll
  for (int i = 0; i < NN; ++i) {
    u[2 * zo + i] = o[0][i];
    u[2 * zo + NN + i] = o[1][i];
  }
}

__global__ void __launch_bounds__(64) velocity_field_kernel(const AuxArgs a, const double *z,
                                                            const double *q, double *u) {
  const int c = grouped_cell(a);
  if (c < 0) return;
  const int p = checked_degree(a.err, a.deg[c]), N = p + 1;
  const int64_t zo = checked(a.err, a.off[c], a.n_dofs - N * N + 1, BS_OFFSET);
  switch (p) {
    case 1: velocity_cell<1>(a, c, zo, z, q, u); break;
    case 2: velocity_cell<2>(a, c, zo, z, q, u); break;
    case 3: velocity_cell<3>(a, c, zo, z, q, u); break;
    default: velocity_cell<4>(a, c, zo, z, q, u); break;
  }
}

// Vorticity of the indicator features (hpTuner.h:247-305 of the velocity above) and the cell
// means of zeta and q, straight from the state: the nodal velocity is not formed, its
// values and derivatives at QGauss(nq) are B S^-1 and D S^-1 applied to the velocity at
// Gauss p+1 (BS, DS: [degree-1][8][OC_MAXN]).  FP64 pipe, one thread per cell.  (In two
// kernels, velocity by a sum over all node pairs into global memory and vorticity from
// it: 212 + 63 us on 125,000 cells of degrees 1 and 2.)
template <int P>
__device__ __forceinline__ float vorticity_cell(const AuxArgs &a, int c, int64_t zo,
                                                const double *z, const double *q, int nq,
                                                const double *BS, const double *DS,
                                                float *mean) {
  constexpr int N = P + 1, NN = N * N, NQ = OC_MAXDEG;
  const DegTables<double> &tb = tab<double>(P);
  const double *sd = a.sd2 ? a.sd2 + cell_data(a.err, a.sdo2, c, a.n_sd[2], 2 * NN) : nullptr;
  const double *Bp = BS + (P - 1) * 8 * OC_MAXN, *Dp = DS + (P - 1) * 8 * OC_MAXN;
  const double *J = a.geo + 11 * (int64_t)c;
  const double J0 = J[6], J1 = J[7], J2 = J[8], J3 = J[9];
  const bool rect = J1 == 0. && J2 == 0.;
  double w[NQ][NQ], m[3] = {0, 0, 0};
#pragma unroll
  for (int l = 0; l < NQ; ++l)
#pragma unroll
    for (int k = 0; k < NQ; ++k) w[l][k] = 0;
#pragma unroll 1
  for (int qy = 0; qy < N; ++qy) {
    double u[N], v[N], s[3] = {0, 0, 0};
    velocity_row<P>(a, z + zo, q + 2 * zo, sd, qy,
                    [&](int qx, double zv, double q0, double q1, double u0, double u1) {
                      u[qx] = u0;
                      v[qx] = u1;
                      s[0] += tb.wM[qx] * zv;
                      s[1] += tb.wM[qx] * q0;
                      s[2] += tb.wM[qx] * q1;
                    });
#pragma unroll
    for (int e = 0; e < 3; ++e) m[e] += tb.wM[qy] * s[e];
#pragma unroll
    for (int k = 0; k < NQ; ++k)
      if (k < nq) {
        // dv/dx - du/dy: x derivatives meet the values along y and the other way round
        double f = 0, g = 0;
#pragma unroll
        for (int qx = 0; qx < N; ++qx) {
          f += __ldg(Dp + k * OC_MAXN + qx) * v[qx];
          g += __ldg(Bp + k * OC_MAXN + qx) * u[qx];
        }
        f *= J0;
        g *= -J3;
        if (!rect) {
          double fu = 0, gv = 0;
#pragma unroll
          for (int qx = 0; qx < N; ++qx) {
            fu += __ldg(Dp + k * OC_MAXN + qx) * u[qx];
            gv += __ldg(Bp + k * OC_MAXN + qx) * v[qx];
          }
          f -= J1 * fu;
          g += J2 * gv;
        }
#pragma unroll
        for (int l = 0; l < NQ; ++l)
          if (l < nq)
            w[l][k] += __ldg(Bp + l * OC_MAXN + qy) * f + __ldg(Dp + l * OC_MAXN + qy) * g;
      }
  }
  float mv = 0.f;
#pragma unroll
  for (int l = 0; l < NQ; ++l)
#pragma unroll
    for (int k = 0; k < NQ; ++k)
      if (l < nq && k < nq) {
        const float x = (float)fabs(w[l][k]);
        mv = x > mv ? x : mv;
      }
#pragma unroll
  for (int e = 0; e < 3; ++e) mean[e] = (float)m[e];
  return mv;
}

// vorticity and means of every cell and the largest vorticity of each member (non-negative
// floats order like their bits; one atomic per member in a warp)
__global__ void __launch_bounds__(64) vorticity_means_kernel(
    const AuxArgs a, const double *z, const double *q, int nq, const double *BS, const double *DS,
    const int *info, int n_members, float *out, float *feat, unsigned *vmax) {
  const int c = grouped_cell(a);
  float w = 0.f;
  int m = -1;
  if (c >= 0) {
    const int p = checked_degree(a.err, a.deg[c]), N = p + 1;
    const int64_t zo = checked(a.err, a.off[c], a.n_dofs - N * N + 1, BS_OFFSET);
    float *mean = feat + 12 * (int64_t)c;
    switch (p) {
      case 1: w = vorticity_cell<1>(a, c, zo, z, q, nq, BS, DS, mean); break;
      case 2: w = vorticity_cell<2>(a, c, zo, z, q, nq, BS, DS, mean); break;
      case 3: w = vorticity_cell<3>(a, c, zo, z, q, nq, BS, DS, mean); break;
      default: w = vorticity_cell<4>(a, c, zo, z, q, nq, BS, DS, mean); break;
    }
    out[c] = w;
    m = info[6 * (int64_t)c + 5];
    if (m < 0 || m >= n_members) m = -1;
  }
  unsigned left = __ballot_sync(OC_FULL, m >= 0);
  while (left) {
    const int mm = __shfl_sync(OC_FULL, m, __ffs(left) - 1);
    const unsigned own = __reduce_max_sync(OC_FULL, m == mm ? __float_as_uint(w) : 0u);
    if ((threadIdx.x & 31) == 0) atomicMax(&vmax[mm], own);
    left &= ~__ballot_sync(OC_FULL, m == mm);
  }
}

// hpTuner.h:247-305: max over QGauss(nq) points of |dv/dx - du/dy|;
// B/D: [degree-1][nq*OC_MAXN] values/derivatives of the basis at the points
__global__ void vorticity_kernel(const AuxArgs a, const double *u, int nq, const double *B,
                                 const double *Dm, float *out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.n_cells) return;
  const int p = checked_degree(a.err, a.deg[c]), N = p + 1, n = N * N;
  const double *Bp = B + (p - 1) * 8 * OC_MAXN, *Dp = Dm + (p - 1) * 8 * OC_MAXN;
  const double *J = a.geo + 11 * (int64_t)c;
  const double *uc = u + 2 * checked(a.err, a.off[c], a.n_dofs - n + 1, BS_OFFSET);
  float mv = 0.f;
  for (int qy = 0; qy < nq; ++qy)
    for (int qx = 0; qx < nq; ++qx) {
      double ux = 0, uy = 0, vx = 0, vy = 0;
      for (int iy = 0; iy < N; ++iy)
        for (int ix = 0; ix < N; ++ix) {
          const double bx = Bp[qx * OC_MAXN + ix], by = Bp[qy * OC_MAXN + iy];
          const double dx = Dp[qx * OC_MAXN + ix], dy = Dp[qy * OC_MAXN + iy];
          const double uu = uc[iy * N + ix], vv = uc[n + iy * N + ix];
          ux += dx * by * uu;
          uy += bx * dy * uu;
          vx += dx * by * vv;
          vy += bx * dy * vv;
        }
      const double du_dy = J[7] * ux + J[9] * uy;  // physical d/dy of u
      const double dv_dx = J[6] * vx + J[8] * vy;  // physical d/dx of v
      const float w = (float)fabs(dv_dx - du_dy);
      mv = w > mv ? w : mv;
    }
  out[c] = mv;
}

// OceanDG.h:2241-2352 with the vortex exact solution as the projected function:
// zeta = S^-1 f0, q = S^-1 (f_{1,2} depth(f0, zb)) on Gauss p+1, accumulated
// point by point into the cell's own outputs
__global__ void project_vortex_kernel(const AuxArgs a, double time, double *z, double *q) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.n_cells) return;
  const int p = checked_degree(a.err, a.deg[c]), N = p + 1, n = N * N;
  const DegTables<double> &tb = tab<double>(p);
  const double *J = a.geo + 11 * (int64_t)c;
  const double *sd = a.sd2 ? a.sd2 + cell_data(a.err, a.sdo2, c, a.n_sd[2], 2 * n) : nullptr;
  const int64_t zo = checked(a.err, a.off[c], a.n_dofs - n + 1, BS_OFFSET);
  const VortexParams vp = vortex_params(a.vortex);
  double *zc = z + zo, *q0 = q + 2 * zo, *q1 = q + 2 * zo + n;
  for (int i = 0; i < n; ++i) zc[i] = 0.;
  for (int i = 0; i < 2 * n; ++i) q0[i] = 0.;
  for (int qy = 0; qy < N; ++qy)
    for (int qx = 0; qx < N; ++qx) {
      const double e0 = tb.xM[qx], e1 = tb.xM[qy];
      const double x = J[0] + J[2] * e0 + J[3] * e1, y = J[1] + J[4] * e0 + J[5] * e1;
      const double fz = vortex_value(vp, a.g, x, y, time, 0);
      const double hq = depth<double>(fz, sd ? sd[2 * (qy * N + qx)] : 0.);
      const double f1 = vortex_value(vp, a.g, x, y, time, 1) * hq;
      const double f2 = vortex_value(vp, a.g, x, y, time, 2) * hq;
      for (int iy = 0; iy < N; ++iy)
        for (int ix = 0; ix < N; ++ix) {
          const double s = tb.Sinv[iy][qy] * tb.Sinv[ix][qx];
          zc[iy * N + ix] += s * fz;
          q0[iy * N + ix] += s * f1;
          q1[iy * N + ix] += s * f2;
        }
    }
}

cudaError_t aux_upload_tables(const DegTables<double> *td, const DegTables<float> *tf) {
  cudaError_t e = cudaMemcpyToSymbol(c_tabd, td, sizeof(DegTables<double>) * OC_MAXDEG);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_tabf, tf, sizeof(DegTables<float>) * OC_MAXDEG);
}

// blocks of 64 for the kernels that take their cell by grouped_cell
static int grouped_grid(const AuxArgs &a) {
  if (!a.group_cells[0]) return (a.n_cells + 63) / 64;
  int grid = 0;
  for (int k = 0; k < OC_MAXDEG; ++k) grid += a.group_blocks[k];
  return grid;
}

cudaError_t launch_cell_sigma(int n, const double *geo, double *sigma, cudaStream_t st) {
  cell_sigma_kernel<<<(n + 127) / 128, 128, 0, st>>>(n, geo, sigma);
  return cudaGetLastError();
}

// work: the largest lower bound (FP32 bits) and, 8 bytes on, the result (FP64 bits); up, mask:
// per cell
cudaError_t launch_transport_speed(const AuxArgs &a, const double *z, const double *q, float *up,
                                   unsigned long long *mask, unsigned long long *work,
                                   double *per_cell, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(work, 0, 16, st);
  if (e != cudaSuccess) return e;
  const int grid = grouped_grid(a);
  unsigned *lower = reinterpret_cast<unsigned *>(work);
  speed_bounds_kernel<<<grid, 64, 0, st>>>(a, z, q, up, mask, lower);
  speed_kernel<<<grid, 64, 0, st>>>(a, z, q, up, mask, lower, work + 1, per_cell);
  return cudaGetLastError();
}

cudaError_t launch_velocity_field(const AuxArgs &a, const double *z, const double *q, double *u,
                                  cudaStream_t st) {
  velocity_field_kernel<<<grouped_grid(a), 64, 0, st>>>(a, z, q, u);
  return cudaGetLastError();
}

// compute_errors_hydro (OceanDG.h:2380-2459) with the vortex as exact solution:
// per cell the squared L2 errors of depth and discharge on the cell Gauss rule,
// written to part[2c], part[2c+1] (summed by errors_reduce_kernel in a fixed order).
__global__ void errors_kernel(const AuxArgs a, double time, const double *sd0, const int *sdo0,
                              const double *z, const double *q, double *part) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.n_cells) return;
  const int p = checked_degree(a.err, a.deg[c]), N = p + 1, n = N * N;
  const int Q = a.cell_rule ? p + 1 : (3 * p) / 2 + 1;
  const DegTables<double> &tb = tab<double>(p);
  // the cell Gauss rule's tables: floor(1.5 p) + 1 points, or the Gauss p+1 ones
  const double(*BQ)[OC_MAXN] = a.cell_rule ? tb.BM : tb.BQ;
  const double *xQ = a.cell_rule ? tb.xM : tb.xQ, *wQ = a.cell_rule ? tb.wM : tb.wQ;
  const double *J = a.geo + 11 * (int64_t)c;
  const int64_t zo = checked(a.err, a.off[c], a.n_dofs - n + 1, BS_OFFSET);
  const double *zc = z + zo, *q0 = q + 2 * zo, *q1 = q + 2 * zo + n;
  const double *sd = sd0 ? sd0 + cell_data(a.err, sdo0, c, a.n_sd[0], 5 * Q * Q) : nullptr;
  const VortexParams vp = vortex_params(a.vortex);
  double e0 = 0., e1 = 0.;
  for (int qy = 0; qy < Q; ++qy)
    for (int qx = 0; qx < Q; ++qx) {
      double zv = 0., a0 = 0., a1 = 0.;
      for (int iy = 0; iy < N; ++iy)
        for (int ix = 0; ix < N; ++ix) {
          const double b = BQ[qy][iy] * BQ[qx][ix];
          zv += b * zc[iy * N + ix];
          a0 += b * q0[iy * N + ix];
          a1 += b * q1[iy * N + ix];
        }
      const double x = J[0] + J[2] * xQ[qx] + J[3] * xQ[qy];
      const double y = J[1] + J[4] * xQ[qx] + J[5] * xQ[qy];
      const double zb = sd ? sd[5 * (qy * Q + qx)] : 0.;
      const double f0 = vortex_value(vp, a.g, x, y, time, 0);
      const double hq = depth<double>(f0, zb);
      const double jxw = wQ[qx] * wQ[qy] * J[10];
      const double d0 = hq - depth<double>(zv, zb);
      const double u = vortex_value(vp, a.g, x, y, time, 1) * hq - a0;
      const double v = vortex_value(vp, a.g, x, y, time, 2) * hq - a1;
      e0 += d0 * d0 * jxw;
      e1 += (u * u + v * v) * jxw;
    }
  part[2 * (int64_t)c] = e0;
  part[2 * (int64_t)c + 1] = e1;
}

// one block: strided partial sums, then a fixed tree (deterministic order)
__global__ void errors_reduce_kernel(int n, const double *part, double *out) {
  __shared__ double s0[256], s1[256];
  double a0 = 0., a1 = 0.;
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    a0 += part[2 * (int64_t)c];
    a1 += part[2 * (int64_t)c + 1];
  }
  s0[threadIdx.x] = a0;
  s1[threadIdx.x] = a1;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      s0[threadIdx.x] += s0[threadIdx.x + h];
      s1[threadIdx.x] += s1[threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sqrt(s0[0]);
    out[1] = sqrt(s1[0]);
  }
}

// prepare_for_conservative_coarsening (OceanDG.h:2732-2778) on marked cells
__global__ void conservative_coarsening_kernel(const AuxArgs a, const unsigned char *mark,
                                               double *z) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.n_cells || !mark[c]) return;
  const int p = checked_degree(a.err, a.deg[c]), N = p + 1, n = N * N, G = p + 2;
  const DegTables<double> &tb = tab<double>(p);
  const double det = a.geo[11 * (int64_t)c + 10];
  double *zc = z + checked(a.err, a.off[c], a.n_dofs - n + 1, BS_OFFSET);
  const double *sd = a.sd1 ? a.sd1 + cell_data(a.err, a.sdo1, c, a.n_sd[1], G * G) : nullptr;
  double area = 0., integral = 0.;
  for (int gy = 0; gy < G; ++gy)
    for (int gx = 0; gx < G; ++gx) {
      double zv = 0.;
      for (int iy = 0; iy < N; ++iy)
        for (int ix = 0; ix < N; ++ix) zv += tb.BG[gy][iy] * tb.BG[gx][ix] * zc[iy * N + ix];
      const double zb = sd ? sd[gy * G + gx] : 0.;
      const double mask = zv <= -zb ? 0. : 1.;
      const double jxw = tb.wG[gx] * tb.wG[gy] * det;
      area += mask * jxw;
      integral += zv * mask * jxw;
    }
  if (area > 0.) {
    const double v = integral * (1. / area);
    for (int i = 0; i < n; ++i) zc[i] = v;
  }
}

// one thread: an index outside its range through the bounds check (no access)
__global__ void bounds_selftest_kernel(int *err) { checked(err, 5, 3, BS_SELFTEST); }

cudaError_t launch_bounds_selftest(int *err, cudaStream_t st) {
  bounds_selftest_kernel<<<1, 1, 0, st>>>(err);
  return cudaGetLastError();
}

cudaError_t launch_errors(const AuxArgs &a, double time, const double *sd0, const int *sdo0,
                          const double *z, const double *q, double *part, double *out,
                          cudaStream_t st) {
  errors_kernel<<<(a.n_cells + 127) / 128, 128, 0, st>>>(a, time, sd0, sdo0, z, q, part);
  errors_reduce_kernel<<<1, 256, 0, st>>>(a.n_cells, part, out);
  return cudaGetLastError();
}

cudaError_t launch_conservative_coarsening(const AuxArgs &a, const unsigned char *mark, double *z,
                                           cudaStream_t st) {
  conservative_coarsening_kernel<<<(a.n_cells + 127) / 128, 128, 0, st>>>(a, mark, z);
  return cudaGetLastError();
}

// Indicator features of one cell (see oc_indicator_features in oceano_gpu.h); the means are
// there already (vorticity_means_kernel).
__global__ void features_kernel(const AuxArgs a, const float *w, const int *info, int n_members, const unsigned *vmax, float thr,
                                float *feat, float *flags, float *wn) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.n_cells) return;
  const int p = checked_degree(a.err, a.deg[c]);
  const int *inf = info + 6 * (int64_t)c;
  const int m = inf[5];
  const float mx = (m >= 0 && m < n_members) ? __uint_as_float(vmax[m]) : 0.f;
  const float inv = mx > 0.f ? 1.f / mx : 0.f;
  const float w0 = w[c] * inv;
  // vorticity magnitudes relative to the member maximum on a log10 scale: the
  // refinement threshold (1e-5 of the maximum) sits many decades below the bulk
  // of the values, where a linear feature is lost in the BF16 inputs
  float nb[4];
  for (int f = 0; f < 4; ++f) nb[f] = log10f(fabsf(inf[f] >= 0 ? w[inf[f]] * inv : w0) + 1e-12f);
  float *o = feat + 12 * (int64_t)c;
  o[3] = log10f(fabsf(w0) + 1e-12f);
  o[4] = 0.5f * (nb[1] - nb[0]);  // differences across the cell (faces 1-0, 3-2)
  o[5] = 0.5f * (nb[3] - nb[2]);
  o[6] = nb[0]; o[7] = nb[1]; o[8] = nb[2]; o[9] = nb[3];
  o[10] = (float)inf[4]; o[11] = (float)p;
  if (flags) flags[c] = w0 > thr ? 1.f : 0.f;
  if (wn) wn[c] = w0;
}

cudaError_t launch_features(const AuxArgs &a, const double *z, const double *q, int nq,
                            const double *BS, const double *DS, float *w, const int *info,
                            int n_members, unsigned *vmax, float thr, float *feat, float *flags,
                            float *wn, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(vmax, 0, sizeof(unsigned) * n_members, st);
  if (e != cudaSuccess) return e;
  vorticity_means_kernel<<<grouped_grid(a), 64, 0, st>>>(a, z, q, nq, BS, DS, info, n_members, w,
                                                         feat, vmax);
  features_kernel<<<(a.n_cells + 127) / 128, 128, 0, st>>>(a, w, info, n_members, vmax, thr, feat,
                                                           flags, wn);
  return cudaGetLastError();
}

cudaError_t launch_vorticity(const AuxArgs &a, const double *u, int nq, const double *B,
                             const double *D, float *out, cudaStream_t st) {
  vorticity_kernel<<<(a.n_cells + 127) / 128, 128, 0, st>>>(a, u, nq, B, D, out);
  return cudaGetLastError();
}

cudaError_t launch_project_vortex(const AuxArgs &a, double time, double *z, double *q,
                                  cudaStream_t st) {
  project_vortex_kernel<<<(a.n_cells + 127) / 128, 128, 0, st>>>(a, time, z, q);
  return cudaGetLastError();
}

}  // namespace oc
