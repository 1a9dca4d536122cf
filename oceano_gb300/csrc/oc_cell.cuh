// The stage of the mixed time step with four lanes per cell -- two or eight on some groups
// (cell_lanes in oc_api.cu) -- for the common case (operators without static
// data, friction model and ARK scheme; oc_kernels.cuh holds the general kernel, in
// which a team of T lanes shares a cell).
//
// A warp takes 8 cells of one degree, lane h of a cell its face h, its rows h, h + 4, ..
// of Gauss points and of nodes.  The lanes load their rows of the stage input into
// shared memory (one slot per cell) and the neighbours' traces with them, one face per
// lane.  Then every lane evaluates its face
// (own side as the minus side, outward normal), adds it to the cell's residual (faces
// 0, 1, then 2, 3: no two lanes share a node), and its rows of the discharge's cell
// integrals: interpolation, pointwise model and x-integrals, which meet in shared memory
// for the y-integrals.  The zeta cell integrals are linear in the discharge (two 1D
// matrices); they, the zeta sweeps and the discharge inverse are row-local up to one
// projection, summed over the four lanes by shuffles, and so is the Runge-Kutta update:
// a lane loads and stores its rows (vector accesses where rows are aligned).
//
// Bound by instruction issue and latency (degree 3, 320x160 cells, one internal stage: 51%
// of the issue slots, 14 of 16 possible warps per SM on average).  The team kernel issues 33.9 M warp
// instructions there, with 24 to 30 of 32 lanes at work and lanes that repeat a cell's
// whole chain of phases; here 8 cells x 4 lanes fill the warp, each phase's work is split
// by rows or faces, and fewer operations are left (z integrals, inverses and sweeps by
// rank-one forms, no flux ordering by side).  Rows in vector accesses and the update by
// rows in place of element-wise passes through shared memory: 109 -> 97 us per step at
// degree 3, 231 -> 199 on the random hp mesh.  With one lane per cell (three times the
// shared memory per warp, 168 registers) the same algorithm ran 33 / 59 / 102 / 173 us
// per step at degree 1 .. 4 on 51,200 cells against 41 / 67 / 97 / 193 (now 39 / 64 / 95 /
// 183), but 64 against 27 us on 3,200 cells of degree 3 and 370 against 199 us on the random
// hp mesh (now 202): one warp's chain is four times as long.  128 registers (8 blocks of 2
// warps); with 112, 9 blocks, degree 4 took 242 us and the hp mesh 289.
#pragma once
#include "oc_kernels.cuh"

namespace oc {

// Dimensions of the stage with LPC_ lanes per cell: 4, or 2 on large groups of degree 1 and 8
// on small ones of degree 4 (cell_lanes in oc_api.cu).
template <int P, int QR, int LPC_>
struct CellDims {
  static constexpr int N = P + 1, Q = QR ? P + 1 : (3 * P) / 2 + 1, G = P + 2, NN = N * N;
  static constexpr int LPC = LPC_, CPW = 32 / LPC;  // lanes per cell, cells per warp
  static constexpr int NR = (N + LPC - 1) / LPC;  // rows of nodes of a lane
  static constexpr int FL = LPC < 4 ? LPC : 4;    // lanes that take different faces
  static constexpr bool PAIR = LPC == 8;          // two lanes per face, half of the points each
  // shared memory: rows of nodes at a stride that vector loads can read (load_row)
  static constexpr int RS = N == 3 ? 4 : N == 5 ? 6 : N, NS = N * RS;
  // floats of a cell's slot: stage input 3 NS, residual 3 NS, x-integrals 4 N Q; the stride
  // mod 32 counted over the vector accesses to whole cells, rows and x-integrals and the
  // scalar ones to faces
  static constexpr int used = (6 * NS + 3) / 4 * 4 + 4 * N * Q;
  static constexpr int mod = PAIR ? 8 : P < 3 ? 12 : 4;
  static constexpr int S = used + (mod + 32 - used % 32) % 32;
  static constexpr int warp_bytes = CPW * S * 4;
};
// Stage inputs are read by plain loads: a read-only one (__ldg) is no ordinary memory
// access to the compiler, which may then issue it before the wait for the launch that
// wrote the value.

// x - ref in FP32 on the integer and FP32 pipes, from the top 24 bits of x, the next 23 and the
// last 6 as one float each, and ref cut the same way (SplitRef).  For neighbouring x and ref
// the three differences are exact and only the sums round, so that a deviation keeps its FP32
// precision however small it is.  (An FP64 subtraction and conversion per value run at 1/64
// of the FP32 rate: a third of the degree-3 stage 0, 77 us against 45 us for FP32 input.)
// Values below the FP32 normal range count as zero; `odd` collects those above it
// (infinities, NaN), which are converted by FP64 instructions.
__device__ __forceinline__ float split_deviation(double x, const SplitRef &ref, bool &odd) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const unsigned ha = h & 0x7fffffffu;
  odd |= ha >= 0x47f00000u;
  const unsigned fb =
      ((((h << 3) | (l >> 29)) & 0x7fffffffu) ^ 0x40000000u) | (h & 0x80000000u);
  const unsigned f = ha < 0x38100000u ? 0u : fb;
  const unsigned e = f & 0xff800000u;
  const float m = __uint_as_float(e | ((l >> 6) & 0x7fffffu)) - __uint_as_float(e);
  const float r = __uint_as_float(e | ((l << 17) & 0x7e0000u)) - __uint_as_float(e);
  return ((__uint_as_float(f) - ref.t[0]) + fmaf(m, 0x1p-23f, -ref.t[1])) +
         fmaf(r, 0x1p-46f, -ref.t[2]);
}
// (double)x by integer operations (values below the FP32 normal range count as zero)
__device__ __forceinline__ double widen(float x) {
  const unsigned u = __float_as_uint(x), m = u & 0x7fffffffu;
  const unsigned h = m < 0x00800000u ? 0u : (m >> 3) + (m < 0x7f800000u ? 0x38000000u : 0x70000000u);
  return __hiloint2double((int)((u & 0x80000000u) | h), h ? (int)(u << 29) : 0);
}
// isfinite by an integer operation: as a comparison it runs on the FP64 pipe, which with it and
// a conversion instruction in widen was 28% busy at the last stage (degree 3, 320x160 cells, cold
// caches: 48.6 us; 10% and 44.0 us without)
__device__ __forceinline__ bool finite(double x) {
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}
// n stage-input values (FP32 as stored, FP64 as deviations from ref): load(i, j) gives
// the address of value j of element i, or NULL
template <typename RIN, int NV, int NI, class Addr>
__device__ __forceinline__ void load_state(float (&v)[NV][NI], const SplitRef (&ref)[NV],
                                           Addr addr) {
  if constexpr (sizeof(RIN) == 4) {
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const RIN *p = addr(i, j);
        v[j][i] = p ? *p : 0.f;
      }
  } else {
    double x[NV][NI];
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const RIN *p = addr(i, j);
        x[j][i] = p ? *p : 1.;
      }
    bool odd = false;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int i = 0; i < NI; ++i) v[j][i] = split_deviation(x[j][i], ref[j], odd);
    if (odd)
#pragma unroll
      for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          bool o = false;
          split_deviation(x[j][i], ref[j], o);
          if (o)
            v[j][i] = (float)(x[j][i] - (((double)ref[j].t[0] + (double)ref[j].t[1]) +
                                         (double)ref[j].t[2]));
        }
  }
}

// The flat-bathymetry model of a launch.
struct FlatModel {
  float g, cu4, zbe;  // zbe = zb + zeta_ref
};

// One side of a face point: normal discharge deviation q.n - q_r.n, normal velocity
// deviation, normal velocity, depth and wave speed.  DEEP: the depth is known to lie
// above Threshold_for_wetdry, where the velocity is q / h and neither the depth nor the
// free surface is clipped.
struct FaceNormal {
  float n0, n1, urn;  // outward normal, u_r.n
};
struct FaceSide {
  float dqn, dun, un, h, c;
};
template <bool DEEP>
__device__ __forceinline__ FaceSide face_side(const RefStateF &rf, const FlatModel &m,
                                              const FaceNormal &f, float dh, float dq0,
                                              float dq1) {
  FaceSide s;
  s.dqn = dq0 * f.n0 + dq1 * f.n1;
  if constexpr (DEEP) {
    s.h = rf.hr + dh;
    s.dun = (s.dqn - f.urn * dh) * rcp_fast(s.h);
  } else {
    float du0, du1;
    vel_dev<float>(rf, m.cu4, dh, dq0, dq1, du0, du1, s.h);
    s.dun = du0 * f.n0 + du1 * f.n1;
  }
  s.un = f.urn + s.dun;
  s.c = fabsf(s.un) + sqrt_fast(m.g * s.h);
  return s;
}

// Lax-Friedrichs flux through a face with flat bathymetry (face_flux_dev with
// flat = true), the own cell as the minus side and n its outward normal: mass flux, and
// advective flux plus the own side's pressure flux, all times jw.  Swapping the sides
// and the normal changes exactly the signs.
template <bool DEEP>
__device__ __forceinline__ void flat_flux(const RefStateF &rf, const FlatModel &m,
                                          const FaceNormal &f, float jw, float zm, float dqm0,
                                          float dqm1, float zp, float dqp0, float dqp1, float &F,
                                          float &F0, float &F1) {
  const FaceSide a = face_side<DEEP>(rf, m, f, zm, dqm0, dqm1);
  const FaceSide b = face_side<DEEP>(rf, m, f, zp, dqp0, dqp1);
  const float hj = 0.5f * jw, lh = hj * fmaxf(a.c, b.c);
  const float jump = DEEP ? zm - zp : fmaxf(zm, -rf.hr) - fmaxf(zp, -rf.hr);
  F = hj * (a.dqn + b.dqn) + lh * jump;
  const float Xm0 = rf.qr0 * a.dun + dqm0 * a.un, Xm1 = rf.qr1 * a.dun + dqm1 * a.un;
  const float Xp0 = rf.qr0 * b.dun + dqp0 * b.un, Xp1 = rf.qr1 * b.dun + dqp1 * b.un;
  const float pj = (-0.5f * m.g * hj) * ((a.h + b.h) * jump);
  F0 = hj * (Xm0 + Xp0) + (lh * (dqm0 - dqp0) + pj * f.n0);
  F1 = hj * (Xm1 + Xp1) + (lh * (dqm1 - dqp1) + pj * f.n1);
}

// A lower bound of the depth where the nodal depths less h_r lie in [lo, hi] and the
// interpolation has the Lebesgue constant leb, above the wet/dry threshold cu (NaN: no)
__device__ __forceinline__ bool is_deep(const RefStateF &rf, float cu, float lo, float hi,
                                        float leb) {
  const float dmin = 0.5f * (hi + lo) - 0.5f * leb * (hi - lo);
  return rf.hr + dmin > 1.001f * cu + 1e-4f;
}

template <bool B>
struct BoolC {
  static constexpr bool value = B;
};

// The zeta solve of the lanes with `work` set, literally in FP64 over a flat bottom at 0
// (OceanDG.h:828-855, :1373-1507): zeta^n from u^n, rhs = b + int depth(zeta^n) phi over Gauss-Lobatto
// p+2, the epsilon lift of dry cells and at most max_iter lumped sweeps with the
// batch stop rule.  The result goes straight to the stage's outputs.  All lanes of
// the warp call (the norms of a batch are summed over its lanes); out of line and on
// the thread's stack, because only cells that are not fully wet come here.
template <int P, int LPC>
__device__ __noinline__ bool zeta_literal_cell(const StageArgs &a, int cell, int64_t zo,
                                               const float *b, bool work) {
  constexpr int N = P + 1, G = P + 2, NN = N * N;
  const DegTables<double> &tb = tab<double>(P);
  const double det = a.geo[11 * (int64_t)cell + 10];
  double z[NN], rhs[NN], r[NN], m[NN];
  for (int i = 0; i < NN; ++i) z[i] = work ? a.un_z[zo + i] : 1.0;
  // r = int o0(zeta) phi, m = int o1(zeta) phi over the Gauss-Lobatto points
  auto integrate = [&](auto fn) {
    for (int i = 0; i < NN; ++i) r[i] = m[i] = 0;
#pragma unroll 1
    for (int gy = 0; gy < G; ++gy) {
      double v[N], s0[N], s1[N];
      for (int ix = 0; ix < N; ++ix) {
        v[ix] = s0[ix] = s1[ix] = 0;
        for (int iy = 0; iy < N; ++iy) v[ix] += tb.BG[gy][iy] * z[iy * N + ix];
      }
#pragma unroll 1
      for (int gx = 0; gx < G; ++gx) {
        double x = 0, o0, o1;
        for (int ix = 0; ix < N; ++ix) x += tb.BG[gx][ix] * v[ix];
        fn(x, tb.wG[gx] * tb.wG[gy] * det, o0, o1);
        for (int ix = 0; ix < N; ++ix) {
          s0[ix] += tb.BG[gx][ix] * o0;
          s1[ix] += tb.BG[gx][ix] * o1;
        }
      }
      for (int iy = 0; iy < N; ++iy)
        for (int ix = 0; ix < N; ++ix) {
          r[iy * N + ix] += tb.BG[gy][iy] * s0[ix];
          m[iy * N + ix] += tb.BG[gy][iy] * s1[ix];
        }
    }
  };
  int ndry = 0;
  integrate([&](double v, double jxw, double &o0, double &o1) {
    o0 = depth<double>(v, 0.) * jxw;
    o1 = 0;
    ndry += v <= 0.;
  });
  for (int i = 0; i < NN; ++i) rhs[i] = (double)b[i] + r[i];
  if (ndry == G * G)
    for (int i = 0; i < NN; ++i) z[i] = 1e-09;
  bool active = work;
  const int lane = threadIdx.x & 31, W = a.batch, b0 = lane / LPC / W * W;
  for (int k = 0; k < a.max_iter; ++k) {
    if (!__any_sync(OC_FULL, active)) break;
    double part = 0;
    if (active) {
      ndry = 0;
      integrate([&](double v, double jxw, double &o0, double &o1) {
        const double msk = v <= 0. ? 0. : 1.;
        ndry += msk == 0.;
        o0 = -depth<double>(v, 0.) * jxw;
        o1 = msk * jxw;
      });
      for (int i = 0; i < NN; ++i) {
        const double old = z[i];
        z[i] = old + (ndry < G * G ? 1. / m[i] * (rhs[i] + r[i]) : 0.);
        part += fabs(old - z[i]);
      }
    }
    double bn = 0;
    for (int j = 0; j < W; ++j) {
      const double o = __shfl_sync(OC_FULL, part, min(LPC * (b0 + j), 31));
      if (LPC * (b0 + j) < 32) bn += o;
    }
    active = active && bn > 1e-12;
  }
  bool bad = false;
  if (work)
    for (int i = 0; i < NN; ++i) {
      if (a.out_z) a.out_z[zo + i] = z[i];
      if (a.out_rz) a.out_rz[zo + i] = (float)(z[i] - a.zeta_ref);
      bad |= a.last && !isfinite(z[i]);
    }
  return bad;
}

// The exact wetness check of the lanes with `check` set (zeta + zb above the threshold
// at every Gauss-Lobatto point of u^n, zn, and of the result zn + d), then the literal
// solve of those that are not fully wet.  Returns whether the literal solve wrote the
// lane's result; `bad` reports a non-finite one.  All lanes of the warp call.
template <int P, int LPC>
__device__ __noinline__ bool zeta_cold(const StageArgs &a, int cell, int64_t zo, const float *zn,
                                       const float *b, float det, bool check, bool *bad) {
  constexpr int N = P + 1, G = P + 2, NN = N * N;
  const DegTables<float> &tb = tab<float>(P);
  float d[NN], c[N], r[N], s = 0;
  const Sweeps<float> &sw = a.swf[P - 1];
  const float f = sw.one / det;
  for (int i = 0; i < N; ++i) c[i] = r[i] = 0;
  for (int iy = 0; iy < N; ++iy)
    for (int ix = 0; ix < N; ++ix) {
      const float u = b[iy * N + ix] * (tb.zi[ix] * tb.zi[iy] * f);
      d[iy * N + ix] = u;
      c[iy] += tb.zw[ix] * u;
      r[ix] += tb.zw[iy] * u;
    }
  for (int i = 0; i < N; ++i) s += tb.zw[i] * c[i];
  for (int iy = 0; iy < N; ++iy)
    for (int ix = 0; ix < N; ++ix)
      d[iy * N + ix] += sw.sb * (tb.zv[iy] * (r[ix] - s * tb.zv[ix]) +
                                 tb.zv[ix] * (c[iy] - s * tb.zv[iy])) +
                        sw.sg * s * tb.zv[ix] * tb.zv[iy];
  bool wet = true;
  const float thr = a.wet_thrf;
#pragma unroll 1
  for (int gy = 0; gy < G; ++gy) {
    float v0[N], v1[N];
    for (int ix = 0; ix < N; ++ix) {
      v0[ix] = v1[ix] = 0;
      for (int iy = 0; iy < N; ++iy) {
        v0[ix] += tb.BG[gy][iy] * zn[iy * N + ix];
        v1[ix] += tb.BG[gy][iy] * (zn[iy * N + ix] + d[iy * N + ix]);
      }
    }
#pragma unroll 1
    for (int gx = 0; gx < G; ++gx) {
      float x0 = 0, x1 = 0;
      for (int ix = 0; ix < N; ++ix) {
        x0 += tb.BG[gx][ix] * v0[ix];
        x1 += tb.BG[gx][ix] * v1[ix];
      }
      wet = wet && x0 + a.zreff > thr && x1 + a.zreff > thr;
    }
  }
  const bool work = check && !wet;
  if (__any_sync(OC_FULL, work)) *bad = zeta_literal_cell<P, LPC>(a, cell, zo, b, work) || *bad;
  return work;
}

// rows of nodes in shared memory, by vector accesses (stride CellDims::RS)
template <int N>
__device__ __forceinline__ void load_row(const float *p, float (&v)[N]) {
  if constexpr (N == 2) {
    const float2 a = *reinterpret_cast<const float2 *>(p);
    v[0] = a.x; v[1] = a.y;
  } else if constexpr (N == 5) {
    const float2 a = *reinterpret_cast<const float2 *>(p), b = *reinterpret_cast<const float2 *>(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = p[4];
  } else {
    const float4 a = *reinterpret_cast<const float4 *>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z;
    if constexpr (N == 4) v[3] = a.w;
  }
}
template <int N>
__device__ __forceinline__ void store_row(float *p, const float (&v)[N]) {
  if constexpr (N == 2) {
    *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
  } else if constexpr (N == 5) {
    *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    *reinterpret_cast<float2 *>(p + 2) = make_float2(v[2], v[3]);
    p[4] = v[4];
  } else {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], N == 4 ? v[N - 1] : 0.f);
  }
}
// a row of N values in a vector of the handle (FP32; cells of one degree with an even row
// length: aligned to the row, one vector access per lane, the warp's rows one after the other)
template <int N, bool ALIGNED>
__device__ __forceinline__ void get_row(const float *p, bool in, float (&v)[N]) {
  if constexpr (ALIGNED && (N == 2 || N == 4)) {
    if (in) load_row<N>(p, v);
    else
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = in ? p[i] : 0.f;
  }
}
template <int N, bool ALIGNED>
__device__ __forceinline__ void put_row(float *p, const float (&v)[N]) {
  if constexpr (ALIGNED && (N == 2 || N == 4)) {
    store_row<N>(p, v);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = v[i];
  }
}

// sum over the lanes of a cell
template <int LPC>
__device__ __forceinline__ float cell_sum(float v) {
#pragma unroll
  for (int o = 1; o < LPC; o <<= 1) v += __shfl_xor_sync(OC_FULL, v, o);
  return v;
}

// One row of Gauss points qy of the discharge's cell integrals (OceanDG.h:695-826) from
// the stage input U: the x-integrals of the row's terms, [x0 | y0 | x1 | y1][N] at Y
// (component, derivative in x or source: x, derivative in y: y).
template <int P, int QR, int LPC, bool DEEP>
__device__ __forceinline__ void point_row(const RefStateF &rf, const FlatModel &fm,
                                          const float *U, const float *Aj, const float *b,
                                          const float *d, float wy, float *Y) {
  using D = CellDims<P, QR, LPC>;
  constexpr int N = D::N, Q = D::Q, RS = D::RS, NS = D::NS;
  const DegTables<float> &tb = tab<float>(P);
  const auto &cBQ = QR ? tb.BM : tb.BQ;
  const auto &cDQ = QR ? tb.DM : tb.DQ;
  const auto &cwQ = QR ? tb.wM : tb.wQ;
  float vz[N], vy[N], v0[N], v1[N];
#pragma unroll
  for (int ix = 0; ix < N; ++ix) vz[ix] = vy[ix] = v0[ix] = v1[ix] = 0.f;
#pragma unroll
  for (int iy = 0; iy < N; ++iy) {
    float z[N], q0[N], q1[N];
    load_row<N>(U + iy * RS, z);
    load_row<N>(U + NS + iy * RS, q0);
    load_row<N>(U + 2 * NS + iy * RS, q1);
#pragma unroll
    for (int ix = 0; ix < N; ++ix) {
      vz[ix] += b[iy] * z[ix];
      vy[ix] += d[iy] * z[ix];
      v0[ix] += b[iy] * q0[ix];
      v1[ix] += b[iy] * q1[ix];
    }
  }
  float x0[N], y0[N], x1[N], y1[N];
#pragma unroll
  for (int ix = 0; ix < N; ++ix) x0[ix] = y0[ix] = x1[ix] = y1[ix] = 0.f;
  // velocity of the reference state in reference coordinates
  const float kA = Aj[0] * rf.ur0 + Aj[1] * rf.ur1, kB = Aj[2] * rf.ur0 + Aj[3] * rf.ur1;
  // (rolled: as fast as unrolled at degrees 1 to 3, degree 4 202 -> 193 us per step, and the
  // four degrees of an hp mesh fit the instruction cache better, 223 -> 212 us)
#pragma unroll 1
  for (int qx = 0; qx < Q; ++qx) {
    float z = 0, zx = 0, zy = 0, q0 = 0, q1 = 0;
#pragma unroll
    for (int ix = 0; ix < N; ++ix) {
      const float bx = cBQ[qx][ix];
      z += bx * vz[ix];
      zx += cDQ[qx][ix] * vz[ix];
      zy += bx * vy[ix];
      q0 += bx * v0[ix];
      q1 += bx * v1[ix];
    }
    // fluxes minus the reference flux (ShallowWater.h:378-403) in reference coordinates,
    // J^-1 (q_r du + dq (u_r + du)), and -g h grad(zeta) (:405-432), times JxW
    const float w = cwQ[qx] * wy;
    float h, A, B;
    if constexpr (DEEP) {
      h = rf.hr + z;
      const float wr = w * rcp_fast(h);
      A = ((Aj[0] * q0 + Aj[1] * q1) - kA * z) * wr;
      B = ((Aj[2] * q0 + Aj[3] * q1) - kB * z) * wr;
    } else {
      float du0, du1;
      vel_dev<float>(rf, fm.cu4, z, q0, q1, du0, du1, h);
      A = (Aj[0] * du0 + Aj[1] * du1) * w;
      B = (Aj[2] * du0 + Aj[3] * du1) * w;
    }
    const float Au = w * kA + A, Bu = w * kB + B;
    const float g00 = rf.qr0 * A + q0 * Au, g01 = rf.qr0 * B + q0 * Bu;
    const float g10 = rf.qr1 * A + q1 * Au, g11 = rf.qr1 * B + q1 * Bu;
    const float gh = (-fm.g * w) * h;
    const float s0 = gh * (Aj[0] * zx + Aj[2] * zy), s1 = gh * (Aj[1] * zx + Aj[3] * zy);
#pragma unroll
    for (int ix = 0; ix < N; ++ix) {
      const float bx = cBQ[qx][ix], dx = cDQ[qx][ix];
      x0[ix] += dx * g00;
      x0[ix] += bx * s0;
      y0[ix] += bx * g01;
      x1[ix] += dx * g10;
      x1[ix] += bx * s1;
      y1[ix] += bx * g11;
    }
  }
  float y[4 * N];
#pragma unroll
  for (int ix = 0; ix < N; ++ix) {
    y[ix] = x0[ix];
    y[N + ix] = y0[ix];
    y[2 * N + ix] = x1[ix];
    y[3 * N + ix] = y1[ix];
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
    *reinterpret_cast<float4 *>(Y + 4 * i) =
        make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
}

// One warp of cells (`blk`, n_group, group_cells, group_first as in stage_body).
// CONF: a conforming mesh of this degree alone (one slot per face, no degree jump).
template <int P, typename RIN, int QR, bool CONF, int LPC>
__device__ __forceinline__ void cell_body(const StageArgs &a, unsigned char *smem_raw,
                                          const int blk, const int n_group,
                                          const int *group_cells, const int group_first) {
  using D = CellDims<P, QR, LPC>;
  constexpr int N = D::N, Q = D::Q, G = D::G, NN = D::NN, S = D::S, RS = D::RS, NS = D::NS,
                CPW = D::CPW, NR = D::NR, FL = D::FL;
  constexpr bool PAIR = D::PAIR;
  const DegTables<float> &tb = tab<float>(P);
  const auto &cBQ = QR ? tb.BM : tb.BQ;
  const auto &cwQ = QR ? tb.wM : tb.wQ;
  // entries that differ by lane come from the global copy (L1)
  const DegTables<float> &gt = a.gtabf[P - 1];
  const float *gB = QR ? &gt.BM[0][0] : &gt.BQ[0][0], *gD = QR ? &gt.DM[0][0] : &gt.DQ[0][0],
              *gw = QR ? gt.wM : gt.wQ;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, h = lane % LPC,
            c = lane / LPC;
  const int cpw = CPW / a.batch * a.batch;  // whole batches of the zeta stop rule
  const int g0 = (blk * kCellWarps + warp) * cpw;
  const int nvalid = max(0, min(cpw, n_group - g0));
  const bool valid = c < nvalid;
  constexpr bool FIRST = sizeof(RIN) == 8;  // the FP64 stage input is stage 0's, u^n
  const int s = FIRST ? 0 : a.stage;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  float *SM = reinterpret_cast<float *>(smem_raw + warp * D::warp_bytes);
  float *U = SM + c * S, *RES = U + 3 * NS, *Y = U + (6 * NS + 3) / 4 * 4;  // the lane's cell
  // lanes past the last cell work on the group's first one and store nothing
  const int gi = valid ? g0 + c : 0;
  const int cell =
      (int)checked(a.err, group_cells ? group_cells[gi] : group_first + gi, a.n_cells, BS_CELL);
  const int64_t zo = checked(a.err, a.uniform_nn ? (int64_t)cell * a.uniform_nn : a.off[cell],
                             a.n_dofs - NN + 1, BS_OFFSET);
  const float *geo = a.geof + 11 * (int64_t)cell;
  // det J^-1, entries of J: cell integrals and face lengths by the same rounded numbers (with
  // J^-1 and det rounded apart they differed by 4e-8, the same way at every step), and their
  // determinant in two terms
  const float Aj[4] = {__ldg(geo + 5), -__ldg(geo + 3), -__ldg(geo + 4), __ldg(geo + 2)};
  const float d0 = __fmul_rn(Aj[0], Aj[3]), d1 = __fmul_rn(Aj[1], Aj[2]), det = __fsub_rn(d0, d1);
  const float detr = (fmaf(Aj[0], Aj[3], -d0) - fmaf(Aj[1], Aj[2], -d1)) +
                     __fsub_rn(__fsub_rn(d0, det), d1);
  // independent instances with their own step size: the residual carries dt_c / dt
  const float sc = a.cscalef ? __ldg(a.cscalef + cell) : 1.f;
  const FlatModel fm = {a.gf, a.cu4f, a.zreff};
  const SplitRef ref[3] = {a.zrefs, {{a.ref.qr0, 0.f, 0.f}}, {{a.ref.qr1, 0.f, 0.f}}};
  const float cu = a.cuf;
  const RIN *const rz = static_cast<const RIN *>(a.rz), *const rq = static_cast<const RIN *>(a.rq);
  // face records: slots 2f and 2f + 1 of face f (the second half of a hanging face)
  auto record = [&](int sl) {
    const int2 v = __ldg(reinterpret_cast<const int2 *>(a.cfrec) + (8 * (int64_t)cell + sl));
    FaceRec r;
    r.other = v.x;
    r.pk = valid ? v.y : 0;
#ifdef OC_BOUNDS_CHECK
    check_record(a, r, Q, nullptr, nullptr);
#endif
    return r;
  };
  FaceRec rec = record(2 * (h % FL)), rec2;
  rec2.pk = rec2.other = 0;
  if (!CONF) rec2 = record(2 * (h % FL) + 1);
  // the second lane of a face takes its nodes in the opposite order: by the symmetry of the
  // points its first half of them is then the other half, with the same table entries
  const bool rev = PAIR && h >= FL;
  // the lane's rows of nodes iy = h + 4 k: lumped mass, its inverse in two terms and the
  // highest mode there
  float l_r[NR], rl[NR], rll[NR], v_r[NR], w_r[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const int iy = min(h + LPC * k, N - 1);
    const bool in = h + LPC * k < N;
    l_r[k] = __ldg(gt.zl + iy);
    rl[k] = P == 1 ? 2.f : __ldg(gt.zi + iy);  // (1 / l = 2 at degree 1)
    rll[k] = P == 1 ? 0.f : __ldg(gt.zir + iy);
    v_r[k] = __ldg(gt.zv + iy);
    w_r[k] = in ? __ldg(gt.zw + iy) : 0.f;
  }
  __syncwarp();
  // from here on the previous launch's results are read (see stage_body)
  asm volatile("griddepcontrol.wait;\n" ::: "memory");

  // ---- stage input of the warp's cells and the neighbour traces, one memory round trip -------
  // A lane loads its rows; the rows of a cell and the cells of a warp follow one another in
  // memory.
  auto row_in = [&](int k) { return valid && h + LPC * k < N; };
  auto zrow = [&](int k) { return zo + (h + LPC * k) * N; };
  auto qrow = [&](int k, int e) { return 2 * zo + e * NN + (h + LPC * k) * N; };
  // neighbour trace of a slot: values at the face nodes (N of a conforming face)
  constexpr int NB = CONF ? N : OC_MAXN;
  auto load_trace = [&](const FaceRec &r, float (&t)[3][NB]) {
    const int Nn = CONF ? N : r.nb_deg() + 1, nf = r.nb_face();
    int base = nf == 0 ? 0 : nf == 1 ? Nn - 1 : nf == 2 ? 0 : (Nn - 1) * Nn;
    int st = nf < 2 ? Nn : 1;
    if (rev) {
      base += (Nn - 1) * st;
      st = -st;
    }
    const bool in = r.kind() == 1;
    const RIN *const tz = rz + ((int64_t)r.other + base), *const tq = rq + (2 * (int64_t)r.other + base);
    load_state<RIN>(t, ref, [&](int i, int k) -> const RIN * {
      if (!in || (!CONF && i >= Nn)) return nullptr;
      return k == 0 ? tz + i * st : tq + ((k - 1) * Nn * Nn + i * st);
    });
  };
  float nb[3][NB];
  // The cell's own reference state: the fluxes are taken minus their value at the mean of the
  // cell's nodes (a constant flux has no weak divergence), so that FP32 rounds tables, sums
  // and products against the variation over a cell.  c3: the mean's deviations from the
  // operator's reference state, in the units of the stage input; from here on U and the
  // traces hold depth and discharge less (h_r, q_r).  Where the mean is not deep the
  // operator's reference state serves (velocities by division).  Against one reference
  // state for all cells the rounded tables moved the state the same way at every step: with
  // this, det J^-1 and the inverse in two terms (below) and balance_tables, mixed against
  // FP64 after 1,003 steps of the 320x160 degree-3 vortex zeta 4.5e-10 -> 1.4e-10, discharge
  // 6.0e-9 -> 1.0e-9.
  RefStateF rf = a.ref;
  rf.rr0 = rf.rr1 = 0.f;  // (a constant in the velocity is a constant flux)
  float c3[3] = {rf.hr - fm.zbe, 0.f, 0.f};
  auto localise = [&](float (&t)[3][NB]) {
#pragma unroll
    for (int e = 0; e < 3; ++e)
#pragma unroll
      for (int i = 0; i < NB; ++i) t[e][i] -= c3[e];
  };
  {
    float v[3 * NR][N];
    if constexpr (sizeof(RIN) == 4) {
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        get_row<N, CONF>((const float *)rz + zrow(k), row_in(k), v[3 * k]);
        get_row<N, CONF>((const float *)rq + qrow(k, 0), row_in(k), v[3 * k + 1]);
        get_row<N, CONF>((const float *)rq + qrow(k, 1), row_in(k), v[3 * k + 2]);
      }
    } else {
      SplitRef rr[3 * NR];
#pragma unroll
      for (int e = 0; e < 3 * NR; ++e) rr[e] = ref[e % 3];
      load_state<RIN>(v, rr, [&](int i, int e) -> const RIN * {
        if (!row_in(e / 3)) return nullptr;
        return e % 3 == 0 ? rz + (zrow(e / 3) + i) : rq + (qrow(e / 3, e % 3 - 1) + i);
      });
    }
    load_trace(rec, nb);
    float mean[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 3; ++e) {
#pragma unroll
      for (int k = 0; k < NR; ++k)
        if (h + LPC * k < N)
#pragma unroll
          for (int i = 0; i < N; ++i) mean[e] += v[3 * k + e][i];
      mean[e] = cell_sum<LPC>(mean[e]) * (1.f / NN);
    }
    if (fm.zbe + mean[0] > 1.001f * cu + 1e-4f) {
#pragma unroll
      for (int e = 0; e < 3; ++e) c3[e] = mean[e];
      rf.hr = fm.zbe + mean[0];
      rf.qr0 += mean[1];
      rf.qr1 += mean[2];
      const float r = rcp_fast(rf.hr), u0 = rf.qr0 * r, u1 = rf.qr1 * r;
      rf.ur0 = u0 + fmaf(-u0, rf.hr, rf.qr0) * r;
      rf.ur1 = u1 + fmaf(-u1, rf.hr, rf.qr1) * r;
    }
    localise(nb);
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      if (FIRST && row_in(k)) {  // the FP32 u^n
        put_row<N, CONF>(a.out_unzf + zrow(k), v[3 * k]);
        put_row<N, CONF>(a.out_unqf + qrow(k, 0), v[3 * k + 1]);
        put_row<N, CONF>(a.out_unqf + qrow(k, 1), v[3 * k + 2]);
      }
      if (h + LPC * k < N)
#pragma unroll
        for (int e = 0; e < 3; ++e) {
#pragma unroll
          for (int i = 0; i < N; ++i) v[3 * k + e][i] -= c3[e];
          store_row<N>(U + e * NS + (h + LPC * k) * RS, v[3 * k + e]);
        }
    }
  }
  __syncwarp();

  // ---- zeta cell integrals (OceanDG.h:669-693) and nodal bounds of zeta, by rows -------------
  // int q . grad(phi) of a polynomial on an affine cell, exact in the Gauss rules:
  // (G (x) M) (J^-1 q)_x + (M (x) G) (J^-1 q)_y times det, M = L (I - beta v w^T)
  float zlo = U[0], zhi = zlo;  // depth less h_r
  {
    const float a0 = Aj[0] * sc, a1 = Aj[1] * sc, b0 = Aj[2] * sc, b1 = Aj[3] * sc;
    float o[NR][N], m[N];
#pragma unroll
    for (int ix = 0; ix < N; ++ix) m[ix] = 0.f;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const int iy = min(h + LPC * k, N - 1);
      float ta[N], t[N], z[N], q0[N], q1[N], my = 0;
      load_row<N>(U + iy * RS, z);
      load_row<N>(U + NS + iy * RS, q0);
      load_row<N>(U + 2 * NS + iy * RS, q1);
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        zlo = fminf(zlo, z[ix]);
        zhi = fmaxf(zhi, z[ix]);
        ta[ix] = a0 * q0[ix] + a1 * q1[ix];
        t[ix] = b0 * q0[ix] + b1 * q1[ix];
        my += tb.zw[ix] * t[ix];
      }
      my *= tb.zbeta;
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {  // G along x; M along x for the y term
        o[k][ix] = 0.f;
#pragma unroll
        for (int j = 0; j < N; ++j) o[k][ix] += tb.GD[ix][j] * ta[j];
        m[ix] += w_r[k] * o[k][ix];
        t[ix] = tb.zl[ix] * (t[ix] - tb.zv[ix] * my);
      }
      store_row<N>(Y + iy * RS, t);
    }
#pragma unroll
    for (int ix = 0; ix < N; ++ix) m[ix] = tb.zbeta * cell_sum<LPC>(m[ix]);
#pragma unroll
    for (int o = 1; o < LPC; o <<= 1) {
      zlo = fminf(zlo, __shfl_xor_sync(OC_FULL, zlo, o));
      zhi = fmaxf(zhi, __shfl_xor_sync(OC_FULL, zhi, o));
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const int iy = h + LPC * k;
      if (iy < N) {
        float v[N], zero[N];
#pragma unroll
        for (int ix = 0; ix < N; ++ix) {
          v[ix] = l_r[k] * (o[k][ix] - v_r[k] * m[ix]);  // M along y
          zero[ix] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const float g = __ldg(&gt.GD[iy][j]);
          float t[N];
          load_row<N>(Y + j * RS, t);
#pragma unroll
          for (int ix = 0; ix < N; ++ix) v[ix] += g * t[ix];
        }
        store_row<N>(RES + iy * RS, v);
        store_row<N>(RES + NS + iy * RS, zero);
        store_row<N>(RES + 2 * NS + iy * RS, zero);
      }
    }
  }

  // ---- the lane's faces: h, h + 2; h; or half of face h mod 4 (OceanDG.h:936-1050, :1105-1339) ----
#pragma unroll 1
  for (int fo = h % FL; fo < 4; fo += FL) {
    int fbase = fo == 0 ? 0 : fo == 1 ? N - 1 : fo == 2 ? 0 : (N - 1) * RS;
    int fstr = fo < 2 ? RS : 1;
    if (rev) {
      fbase += (N - 1) * fstr;
      fstr = -fstr;
    }
    // outward normal det J^-T n_ref / |.|, whose length is that of the face
    const float sg = fo & 1 ? 1.f : -1.f;
    float on0 = sg * (fo < 2 ? Aj[0] : Aj[2]), on1 = sg * (fo < 2 ? Aj[1] : Aj[3]);
    const float tl = sqrtf(on0 * on0 + on1 * on1), inv = 1.f / tl;
    on0 *= inv;
    on1 *= inv;
    const float full_len = tl * sc;
    const FaceNormal fn = {on0, on1, rf.ur0 * on0 + rf.ur1 * on1};
    float oz[N], o0[N], o1[N], cz[N], c0[N], c1[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int d = fbase + i * fstr;
      oz[i] = U[d];
      o0[i] = U[NS + d];
      o1[i] = U[2 * NS + d];
      cz[i] = c0[i] = c1[i] = 0.f;
    }
#pragma unroll 1
    for (int half = 0; half < (CONF ? 1 : 2); ++half) {
      const FaceRec r = rec;
      const int kind = r.kind();
      if (half && !__any_sync(OC_FULL, kind != 0)) break;
      if (half) {
        load_trace(r, nb);
        localise(nb);
      }
      const int Nn = CONF ? N : r.nb_deg() + 1;
      float lo = zlo, hi = zhi;  // nodal bounds of both sides
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (CONF || i < Nn) {
          lo = fminf(lo, nb[0][i]);
          hi = fmaxf(hi, nb[0][i]);
        }
      // the face points' 1D Lebesgue constants lie below the cells' 2D one at degree 4
      const bool deep = is_deep(rf, cu, lo, hi, 3.f);
      // conforming faces between cells of this degree: the rows from the constant bank;
      // the first and last Gauss-Lobatto points are nodes.  One choice for all faces of
      // the warp (hp meshes: two paths would run one after the other)
      const bool conf_path =
          CONF || __all_sync(OC_FULL, kind != 1 || (r.nb_deg() == P && r.orient() == 0 &&
                                                    r.sub() < 0));
      float len = full_len;
      if (conf_path && deep) {
        if (kind == 1) {
#pragma unroll
          for (int k = 0; k < (PAIR ? (G + 1) / 2 : G); ++k) {
            constexpr int L = N - 1;
            if (PAIR && G % 2 && k == G / 2 && rev) break;
            const bool end = k == 0 || k == G - 1;
            float z, q0, q1, zn, qn0, qn1;
            if (end) {
              z = oz[k ? L : 0]; q0 = o0[k ? L : 0]; q1 = o1[k ? L : 0];
              zn = nb[0][k ? L : 0]; qn0 = nb[1][k ? L : 0]; qn1 = nb[2][k ? L : 0];
            } else {
              z = q0 = q1 = zn = qn0 = qn1 = 0.f;
#pragma unroll
              for (int i = 0; i < N; ++i) {
                const float l = tb.F[0][G][k][i];
                z += l * oz[i]; q0 += l * o0[i]; q1 += l * o1[i];
                zn += l * nb[0][i]; qn0 += l * nb[1][i]; qn1 += l * nb[2][i];
              }
            }
            float F, F0, F1;
            flat_flux<true>(rf, fm, fn, -tb.wF[G][k] * len, z, q0, q1, zn, qn0, qn1, F, F0, F1);
            if (end) {
              cz[k ? L : 0] += F; c0[k ? L : 0] += F0; c1[k ? L : 0] += F1;
            } else {
#pragma unroll
              for (int i = 0; i < N; ++i) {
                const float l = tb.F[0][G][k][i];
                cz[i] += l * F; c0[i] += l * F0; c1[i] += l * F1;
              }
            }
          }
        }
      } else if (kind == 1) {
        // hanging faces, degree jumps, shallow water: trace rows from the global table copy
        const int side = r.side(), sub = r.sub(), nf = r.nf();
        const bool orient = r.orient() != 0;
        if (side == 1 && sub >= 0) len *= 0.5f;  // coarse side: the fine half-face
        const float *lo_ = &gt.F[side ? sub + 1 : 0][nf][0][0];
        const float *ln = &a.gtabf[Nn - 2].F[side ? 0 : sub + 1][nf][0][0];
        const float *wf = &gt.wF[nf][0];
        auto points = [&](auto DEEP) {
#pragma unroll 1
          for (int k = rev; k < nf; k += PAIR ? 2 : 1) {
            const int kn = orient ? nf - 1 - k : k;  // k: the own side's point order
            float l[N], z = 0, q0 = 0, q1 = 0, zn = 0, qn0 = 0, qn1 = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
              l[i] = __ldg(lo_ + k * OC_MAXN + (rev ? N - 1 - i : i));
              z += l[i] * oz[i]; q0 += l[i] * o0[i]; q1 += l[i] * o1[i];
            }
#pragma unroll
            for (int i = 0; i < NB; ++i) {  // rows are zero past the neighbour's nodes
              const float m =
                  rev ? i < Nn ? __ldg(ln + kn * OC_MAXN + Nn - 1 - i) : 0.f : __ldg(ln + kn * OC_MAXN + i);
              zn += m * nb[0][i]; qn0 += m * nb[1][i]; qn1 += m * nb[2][i];
            }
            float F, F0, F1;
            flat_flux<decltype(DEEP)::value>(rf, fm, fn, -__ldg(wf + k) * len, z, q0, q1, zn,
                                             qn0, qn1, F, F0, F1);
#pragma unroll
            for (int i = 0; i < N; ++i) {
              cz[i] += l[i] * F; c0[i] += l[i] * F0; c1[i] += l[i] * F1;
            }
          }
        };
        if (deep) points(BoolC<true>());
        else points(BoolC<false>());
      }
      if (kind == 2) {  // boundary face: Gauss n_q points
        const int bid = r.bid(), bkind = a.bc_kind[bid];
        if (bkind == 0) atomicOr(a.err, ERR_UNKNOWN_BID);
#pragma unroll 1
        for (int k = rev; k < Q; k += PAIR ? 2 : 1) {
          float z = 0, q0 = 0, q1 = 0;
#pragma unroll
          for (int i = 0; i < N; ++i) {
            const float l = PAIR ? __ldg(gB + k * OC_MAXN + (rev ? N - 1 - i : i)) : cBQ[k][i];
            z += l * oz[i]; q0 += l * o0[i]; q1 += l * o1[i];
          }
          float F, F0, F1;
          const float jxw = -(PAIR ? __ldg(gw + k) : cwQ[k]) * len;
          if (bkind == OC_BC_WALL_) {
            const float un = (rf.qr0 + q0) * on0 + (rf.qr1 + q1) * on1;
            flat_flux<false>(rf, fm, fn, jxw, z, q0, q1, z, q0 - 2.f * un * on0,
                             q1 - 2.f * un * on1, F, F0, F1);
          } else {
            const double sx = QR ? tab<double>(P).xM[k] : tab<double>(P).xQ[k];
            // (against the operator's reference state: the constant flux of the cell's own less
            // the operator's is taken off)
            boundary_flux<float, true>(a, bid, bkind, fo, sx, a.geo + 11 * (int64_t)cell,
                                       a.zeta_ref, 0, fm.g, fm.cu4, z + c3[0], q0 + c3[1],
                                       q1 + c3[2], on0, on1, F, F0, F1);
            const float dhc = c3[0] + (fm.zbe - a.ref.hr);
            const float ucn = ((c3[1] + (a.ref.rr0 - a.ref.ur0 * dhc)) * on0 +
                               (c3[2] + (a.ref.rr1 - a.ref.ur1 * dhc)) * on1) / rf.hr;
            const float un = a.ref.ur0 * on0 + a.ref.ur1 * on1 + ucn;
            F = (F - (c3[1] * on0 + c3[2] * on1)) * jxw;
            F0 = (F0 - (a.ref.qr0 * ucn + c3[1] * un)) * jxw;
            F1 = (F1 - (a.ref.qr1 * ucn + c3[2] * un)) * jxw;
          }
#pragma unroll
          for (int i = 0; i < N; ++i) {
            const float l = PAIR ? __ldg(gB + k * OC_MAXN + (rev ? N - 1 - i : i)) : cBQ[k][i];
            cz[i] += l * F; c0[i] += l * F0; c1[i] += l * F1;
          }
        }
      }
      rec = rec2;
    }
    if (fo + FL < 4) {  // the next face's trace, while this one's values are added
      rec = record(2 * (fo + FL));
      if (!CONF) rec2 = record(2 * (fo + FL) + 1);
      load_trace(rec, nb);
      localise(nb);
    }
    __syncwarp();
#pragma unroll
    for (int turn = 0; turn < LPC / 2; ++turn) {
      if ((h >> 1) == turn)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int d = fbase + i * fstr;
          RES[d] += cz[i];
          RES[NS + d] += c0[i];
          RES[2 * NS + d] += c1[i];
        }
      __syncwarp();
    }
  }

  // ---- the lane's rows of Gauss points ----------------------------------------------------------
  {
    const bool deep = is_deep(rf, cu, zlo, zhi, QR ? tb.lebQ1 : tb.lebQ);
    // not unrolled (instruction cache)
#pragma unroll 1
    for (int qy = h; qy < Q; qy += LPC) {
      float b[N], d[N];
#pragma unroll
      for (int iy = 0; iy < N; ++iy) {
        b[iy] = __ldg(gB + qy * OC_MAXN + iy);
        d[iy] = __ldg(gD + qy * OC_MAXN + iy);
      }
      const float wy = __ldg(gw + qy) * sc;
      if (deep)  // by lane, so that a result does not depend on the other cells of the warp
        point_row<P, QR, LPC, true>(rf, fm, U, Aj, b, d, wy, Y + qy * 4 * N);
      else
        point_row<P, QR, LPC, false>(rf, fm, U, Aj, b, d, wy, Y + qy * 4 * N);
    }
  }
  __syncwarp();

  // ---- y-integrals and the exact inverse mass of the discharge (OceanDG.h:1532-1571), by rows ---
  // ((I + alpha v w^T) (x) (I + alpha v w^T)) (L^-1 (x) L^-1) / det: the Gauss p+1 mass is
  // the exact one, a rank-one change of its Gauss-Lobatto lumping L (fill_tables)
  const float rdet = 1.f / det, rdetr = (fmaf(-det, rdet, 1.f) - detr * rdet) * rdet;
  float rq_[NR][2][N];  // the lane's rows of the residual
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const int iy = min(h + LPC * k, N - 1);
    load_row<N>(RES + NS + iy * RS, rq_[k][0]);
    load_row<N>(RES + 2 * NS + iy * RS, rq_[k][1]);
  }
  {
    float cr[2][N];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int ix = 0; ix < N; ++ix) cr[e][ix] = 0.f;
#pragma unroll
    for (int qy = 0; qy < Q; ++qy) {
      float y[4 * N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float4 v = *reinterpret_cast<const float4 *>(Y + qy * 4 * N + 4 * i);
        y[4 * i] = v.x; y[4 * i + 1] = v.y; y[4 * i + 2] = v.z; y[4 * i + 3] = v.w;
      }
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const int iy = min(h + LPC * k, N - 1);
        const float b = __ldg(gB + qy * OC_MAXN + iy), d = __ldg(gD + qy * OC_MAXN + iy);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int ix = 0; ix < N; ++ix) {
            rq_[k][e][ix] += b * y[2 * e * N + ix];
            rq_[k][e][ix] += d * y[(2 * e + 1) * N + ix];
          }
      }
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      // 1 / (l_i l_j det) in two terms: its rounding scaled the whole residual
      float f[N], fr[N];
      const float fy = rdet * rl[k],
                  fyr = fmaf(rdet, rl[k], -fy) + (rdetr * rl[k] + rdet * rll[k]);
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        f[ix] = P == 1 ? 4.f * rdet : fy * tb.zi[ix];
        fr[ix] = P == 1 ? 4.f * rdetr
                        : fmaf(fy, tb.zi[ix], -f[ix]) + (fyr * tb.zi[ix] + fy * tb.zir[ix]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float cc = 0;
#pragma unroll
        for (int ix = 0; ix < N; ++ix) {
          rq_[k][e][ix] = fmaf(rq_[k][e][ix], f[ix], rq_[k][e][ix] * fr[ix]);
          cc += tb.zw[ix] * rq_[k][e][ix];
        }
        cc *= tb.malpha;
#pragma unroll
        for (int ix = 0; ix < N; ++ix) {
          rq_[k][e][ix] += tb.zv[ix] * cc;
          cr[e][ix] += w_r[k] * rq_[k][e][ix];
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        const float t = tb.malpha * cell_sum<LPC>(cr[e][ix]);
#pragma unroll
        for (int k = 0; k < NR; ++k) rq_[k][e][ix] += v_r[k] * t;
      }
  }

  // ---- Runge-Kutta update, by rows -----------------------------------------------------------------
  // sum_j f_j k_j: the registers of the first two stages are read together (the second is the
  // first again, with coefficient 0, at s = 1)
  float fR[OC_MAXSTAGES];
  load_coefs<float>(a.dyn->ff, a.dyn->f, fR);
  float fs = fR[0];
#pragma unroll
  for (int j = 1; j < OC_MAXSTAGES; ++j)
    if (j == s) fs = fR[j];
  const int j2 = s > 1 ? 2 : 1;
  const float f1 = s > 0 ? fR[0] : 0.f, f2 = s > 1 ? fR[1] : 0.f, f3 = s > 2 ? fR[2] : 0.f;
  const bool wk = !a.last || a.write_kq_last;
  bool nonfinite = false;
  // value e of the row (0 zeta, 1 and 2 the discharge) with k in r: stores k, returns in r
  // sum_j f_j k_j and in un the FP32 u^n
  auto update = [&](int k, int e, float (&r)[N], float (&un)[N]) {
    const bool in = row_in(k);
    const int64_t o = e ? qrow(k, e - 1) : zrow(k);
    const float *k1p = static_cast<const float *>(e ? a.kq[1] : a.kz[1]) + o;
    const float *k2p = static_cast<const float *>(e ? a.kq[j2] : a.kz[j2]) + o;
    const float *k3p = static_cast<const float *>(e ? a.kq[3] : a.kz[3]) + o;
    float *ko = static_cast<float *>(e ? a.kq[s + 1] : a.kz[s + 1]) + o;
    float k1[N], k2[N], k3[N];
    get_row<N, CONF>(k1p, in && s > 0, k1);
    get_row<N, CONF>(k2p, in && s > 0, k2);
    get_row<N, CONF>(k3p, in && s > 2, k3);
    // (the last stage needs u^n in FP32 for the wetness of zeta alone; stage 0 wrote its row)
    const float *const unp = !FIRST ? (e ? a.un_qf : a.un_zf) : (e ? a.out_unqf : a.out_unzf);
    get_row<N, CONF>(unp + o, in && !(e && a.last), un);
    if (in && wk) put_row<N, CONF>(ko, r);
#pragma unroll
    for (int ix = 0; ix < N; ++ix)
      r[ix] = fs * r[ix] + f1 * k1[ix] + f2 * k2[ix] + f3 * k3[ix];
  };
  // u^n + up of a row: the FP32 stage input of the next stage; the last stage leaves up in the
  // residual slots for the FP64 result
  auto store = [&](int k, int e, const float (&up)[N], const float (&un)[N]) {
    if (a.last) {
      if (h + LPC * k < N) store_row<N>(RES + e * NS + (h + LPC * k) * RS, up);
    } else if (row_in(k)) {
      float v[N];
#pragma unroll
      for (int ix = 0; ix < N; ++ix) v[ix] = un[ix] + up[ix];
      put_row<N, CONF>((e ? a.out_rq : a.out_rz) + (e ? qrow(k, e - 1) : zrow(k)), v);
    }
  };
#pragma unroll
  for (int k = 0; k < NR; ++k)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float un[N];
      update(k, e + 1, rq_[k][e], un);
      store(k, e + 1, rq_[k][e], un);
    }

  // ---- the zeta sweeps in closed form (sweep_modes): rz_ is b = sum_j f_j k_j ---------------------
  bool literal = false;
  {
    float un[NR][N], rz_[NR][N];
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      load_row<N>(RES + min(h + LPC * k, N - 1) * RS, rz_[k]);
      update(k, 0, rz_[k], un[k]);
    }
    const Sweeps<float> &sums = a.swf[P - 1];
    const float f = sums.one * rdet;
    float u[NR][N], cy[NR], rr[N], sw = 0;
#pragma unroll
    for (int ix = 0; ix < N; ++ix) rr[ix] = 0.f;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const float fy = f * rl[k];
      cy[k] = 0.f;
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        u[k][ix] = rz_[k][ix] * (fy * tb.zi[ix]);
        cy[k] += tb.zw[ix] * u[k][ix];
        rr[ix] += w_r[k] * u[k][ix];
      }
      sw += w_r[k] * cy[k];
    }
    sw = cell_sum<LPC>(sw);
#pragma unroll
    for (int ix = 0; ix < N; ++ix) rr[ix] = cell_sum<LPC>(rr[ix]) - sw * tb.zv[ix];
    // fully wet where the nodal |zeta - zeta_ref| before and after stay below the
    // Lebesgue bound of the Gauss-Lobatto points (see stage_body)
    const float lim = (fm.zbe - a.wet_thrf) / tb.lebG * 0.999f;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const float cx = sums.sb * (cy[k] - sw * v_r[k]) + sums.sg * sw * v_r[k];
      const float cz = sums.sb * v_r[k];
#pragma unroll
      for (int ix = 0; ix < N; ++ix) {
        u[k][ix] += cz * rr[ix] + cx * tb.zv[ix];
        ok = ok && (!row_in(k) || (fabsf(un[k][ix]) < lim &&
                                   fabsf(un[k][ix] + u[k][ix]) < lim));
      }
    }
    unsigned bad = __ballot_sync(OC_FULL, valid && !ok);
    if (bad) {
      // the same bound about the cell's own level, for flows far from the reference level (with
      // a reference level of 0 every cell comes here; the margin: FP32 rounding of the
      // interpolation)
      float lo = INFINITY, hi = -INFINITY;
#pragma unroll
      for (int k = 0; k < NR; ++k)
#pragma unroll
        for (int ix = 0; ix < N; ++ix)
          if (row_in(k)) {
            const float x0 = un[k][ix], x1 = x0 + u[k][ix];
            lo = fminf(lo, fminf(x0, x1));
            hi = fmaxf(hi, fmaxf(x0, x1));
            if (!(fabsf(x0) < INFINITY && fabsf(x1) < INFINITY)) lo = -INFINITY;
          }
#pragma unroll
      for (int o = 1; o < LPC; o <<= 1) {
        lo = fminf(lo, __shfl_xor_sync(OC_FULL, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(OC_FULL, hi, o));
      }
      const float least = fm.zbe + 0.5f * ((hi + lo) - tb.lebG * (hi - lo));
      ok = least > a.wet_thrf + 1e-5f * fmaxf(fabsf(lo), fabsf(hi));
      bad = __ballot_sync(OC_FULL, valid && !ok);
    }
    if (bad) {  // lane 0 of each such cell, from zeta^n and b of the whole cell
      __syncwarp();
#pragma unroll
      for (int k = 0; k < NR; ++k)
        if (h + LPC * k < N)
#pragma unroll
          for (int ix = 0; ix < N; ++ix) {
            U[(h + LPC * k) * N + ix] = un[k][ix];
            RES[(h + LPC * k) * N + ix] = rz_[k][ix];
          }
      __syncwarp();
      const bool check = valid && h == 0 && ((bad >> (LPC * c)) & ((1u << LPC) - 1u));
      literal = zeta_cold<P, LPC>(a, cell, zo, U, RES, det, check, &nonfinite);
      literal = __shfl_sync(OC_FULL, (int)literal, lane - h) != 0;
    }
    if (a.last) __syncwarp();  // (RES may hold b)
#pragma unroll
    for (int k = 0; k < NR; ++k)
      if (!literal) store(k, 0, u[k], un[k]);
  }
  if (a.last) {
    // u^{n+1} = u^n + up in FP64, lane-contiguous: iteration i takes the cells jl + C i, lane
    // l < C NN the DoF l mod NN of one of them (whole lines: the result may be a host vector
    // that is written over the link, 294 against 420 us per step with rows of four values)
    constexpr int C = 32 / NN;
    const int jl = lane / NN, dl = lane - jl * NN;
    const float *const e0 = SM + 3 * NS + dl / N * RS + dl % N;
    __syncwarp();
#pragma unroll 2
    for (int i = 0; i < CPW; i += C) {
      const int jc = min(jl + i, CPW - 1);
      const int64_t oj = __shfl_sync(OC_FULL, (int)zo, jc * LPC);
      const bool lit = __shfl_sync(OC_FULL, (int)literal, jc * LPC) != 0;
      if (lane < C * NN && jl + i < nvalid) {
        const float *const up = e0 + jc * S;
        const int64_t oz = oj + dl, oq = 2 * oj + dl;
        const double z = a.un_z[oz] + widen(up[0]);
        const double q0 = a.un_q[oq] + widen(up[NS]), q1 = a.un_q[oq + NN] + widen(up[2 * NS]);
        if (!lit) a.out_z[oz] = z;
        a.out_q[oq] = q0;
        a.out_q[oq + NN] = q1;
        nonfinite |= !finite(q0) || !finite(q1) || (!lit && !finite(z));
      }
    }
  }
  report_nonfinite(a, nonfinite);
}

// resident blocks per SM (register cap)
#ifndef OC_CELL_BLOCKS
#define OC_CELL_BLOCKS 8
#endif
template <int P, typename RIN, int QR, bool CONF, int LPC>
__global__ void __launch_bounds__(32 * kCellWarps, OC_CELL_BLOCKS) cell_kernel(const StageArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cell_body<P, RIN, QR, CONF, LPC>(a, smem_raw, blockIdx.x, a.n_group, a.group_cells, a.group_first);
}

}  // namespace oc
