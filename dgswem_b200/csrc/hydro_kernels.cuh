// hydro_kernels.cuh -- sm_100a kernels of one RK stage of the p=1 DG hydro
// step.  Per stage: stage_p1 (tile kernel: edge fluxes once per edge in
// shared memory, volume integral, SSP combination; no atomics) ->
// node_minmax (slope limiter node pass) -> limit_wetdry (limiter element
// pass + WETDRY).  Every arithmetic sequence follows the reference routine
// named in its comment.  Compiled twice (kernels_fast.cu with FMA
// contraction, kernels_strict.cu without), see hydro_device.cuh.
#pragma once

#include <cuda_runtime.h>

#include "cr_math.cuh"
#include "hydro_device.cuh"

#ifndef DGSWEM_VARIANT
#error "define DGSWEM_VARIANT (fast or strict) before including hydro_kernels.cuh"
#endif

namespace dgswem {
namespace DGSWEM_VARIANT {

__constant__ BasisP1 cBasis;

// Arithmetic type of the stage kernel's edge and volume terms: FP64, or
// FP32 in the mixed-precision variant (kernels_mixed.cu), whose state,
// SSP combination, ocean depth-positivity fix, limiter and wet/dry stay FP64.
#ifdef DGSWEM_MIXED
typedef float real;
#else
typedef double real;
#endif
__constant__ BasisT<real> cBasisR;  // cBasis in that type

__device__ real gTab[54];  // BasisT::tr and sw, the stage kernel's per-lane tables

// RAMPDG of the stage: from device memory in a replayed CUDA graph (whose
// kernel arguments are fixed at capture), else the launch argument
__device__ __forceinline__ double stage_ramp(const StageArgs& A) { return A.ramp ? *A.ramp : A.rampdg; }

// Element geometry rows in the arithmetic type
__device__ __forceinline__ const real* egeo_r(const MeshView& m) {
#ifdef DGSWEM_MIXED
  return m.egeof;
#else
  return m.egeo;
#endif
}

// Physics constants of the stage kernel's terms in the arithmetic type
struct PhysR {
  real g, nleq, leq, nleqg, fg_l, tau_cap, cori, fric, cf;
};
__device__ __forceinline__ PhysR phys_r(const StageArgs& A) {
#ifdef DGSWEM_MIXED
  const PhysF& p = A.pf;
#else
  const Physics& p = A.ph;
#endif
  return PhysR{p.g, p.nleq, p.leq, p.nleqg, p.fg_l, p.tau_cap, p.cori, p.fric, p.cf};
}

// Asynchronous global -> shared copies (cp.async, completion by
// cp.async.wait_all): the data goes straight to shared memory.
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async8_s(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4_s(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}

// DEPTH**(1.D0/3.D0) of the Manning friction (rhs_dg_hydro.F).  The strict
// variant takes the correctly rounded value of the reference's expression
// (pow_third, cr_math.cuh: IEEE operations only, so the oracle's correctly
// rounded evaluation gives the same bits); the fast variant takes the cube
// root, which differs from it by less than an ulp's worth of the exponent's
// rounding (1/3 is not a double) and costs a fraction of it.
__device__ __forceinline__ double cube_root(double x) {
#ifdef DGSWEM_FAST_MATH
  return cbrt(x);
#else
  return pow_third(x);
#endif
}
__device__ __forceinline__ float cube_root(float x) { return cbrtf(x); }

template <class T>
struct Flux3T {
  T f, g, h;
};
struct alignas(2 * sizeof(real)) Real2 {
  real x, y;
};
using Flux3 = Flux3T<double>;

// Total depth HT = ZE*NLEQ + HB of numerical_flux.F's flux evaluation.
template <bool kNonlin, class T>
__device__ __forceinline__ T depth(const Physics& P, T ze, T hb) {
  return kNonlin ? ze + hb : ze * T(P.nleq) + hb;
}

// max(|un| + c, |un|) with c the square root of a real number: |un| + c, or
// |un| where c is NaN (a negative depth), since c >= 0 otherwise.  FP64 has no
// maximum instruction: a select on c costs half of fmax's compare, selects
// and NaN handling.  (c = NaN and |un| = NaN give NaN either way.)
__device__ __forceinline__ double side_speed(double a, double c) { return c == c ? a + c : a; }
__device__ __forceinline__ float side_speed(float a, float c) { return fmaxf(a + c, a); }

// a b, never fused with a sum
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
// a b + c: fused in the contracting builds (not left to the compiler, which
// may fuse another product of a sum of two), the product rounded by itself in
// the strict build
template <class T>
__device__ __forceinline__ T madd(T a, T b, T c) {
#ifdef DGSWEM_FAST_MATH
  return fma(a, b, c);
#else
  return c + a * b;
#endif
}

// 1 / d and sqrt(s) of both sides of an edge point (d = total depth, s =
// gravity wave speed squared), FP64, by cr_math.cuh's sequences where all four
// are in their range.  kTry: without a branch, ok reset where they are not --
// the stage kernel forms an edge's three points in one straight line, which
// the compiler interleaves, and redoes the edge out of line in that rare case;
// otherwise the operators take over here, out of line.
__device__ __noinline__ double rcp_any(double x) { return 1.0 / x; }
__device__ __noinline__ double quot_any(double a, double b) { return a / b; }
__device__ __noinline__ double sqrt_any(double x) { return sqrt(x); }
template <bool kTry>
__device__ __forceinline__ void side_terms(double di, double de, double si, double se, double& fi, double& fe,
                                           double& ci, double& ce, bool& ok) {
  const bool in = mid_range(di) && mid_range(de) && mid_range(si) && mid_range(se);
  if (kTry || __builtin_expect(in, 1)) {
    fi = rcp_from(di, rcp_seed(di));
    fe = rcp_from(de, rcp_seed(de));
    ci = sqrt_from(si, rsqrt_seed(si));
    ce = sqrt_from(se, rsqrt_seed(se));
    ok = ok && in;
  } else {
    fi = rcp_any(di);
    fe = rcp_any(de);
    ci = sqrt_any(si);
    ce = sqrt_any(se);
  }
}
template <bool kTry>
__device__ __forceinline__ void side_terms(float di, float de, float si, float se, float& fi, float& fe, float& ci,
                                           float& ce, bool&) {
  fi = 1.0f / di;
  fe = 1.0f / de;
  ci = sqrtf(si);
  ce = sqrtf(se);
}
// The larger speed of an edge point's two sides, skipping a NaN one (a side of
// depth zero without flow: its mass flux still takes the other side's speed).
// kTry: by one comparison, without FP64 fmax's NaN handling: a NaN speed needs a
// depth or a discharge for which side_terms resets ok, or that leaves no flux
// finite.
template <bool kTry>
__device__ __forceinline__ double larger(double a, double b) { return kTry ? (a > b ? a : b) : fmax(a, b); }
template <bool kTry>
__device__ __forceinline__ float larger(float a, float b) { return fmaxf(a, b); }

// numerical_flux.F:750-914, Local Lax-Friedrichs, in arithmetic type T.
// kNonlin specialises NLEQ=1, LEQ=0 (the products with 1 and sums with 0 it
// removes are exact).  ht_in / ht_ex: the total depths, depth(ze, hb) --
// passed in so that the mixed-precision kernels can supply them from FP32
// depth traces rather than from an FP32 sum of elevation and bathymetry.
template <bool kNonlin, class T, bool kTry = false>
__device__ __forceinline__ Flux3T<T> llf_ok(const Physics& P, T ze_in, T ze_ex, T qx_in, T qx_ex, T qy_in,
                                            T qy_ex, T hb_in, T hb_ex, T ht_in, T ht_ex, T sf_in, T sf_ex, T nx,
                                            T ny, T G, bool& ok) {
  const T NLEQ = kNonlin ? T(1) : T(P.nleq);
  const T LEQ = kNonlin ? T(0) : T(P.leq);
  const T nleqg = G * NLEQ;
  const T j1 = ze_ex - ze_in, j2 = qx_ex - qx_in, j3 = qy_ex - qy_in;
  const T nxsi = nx * sf_in, nxse = nx * sf_ex;
  T fh, fhe, ci, ce;
  side_terms<kTry>(kNonlin ? ht_in : NLEQ * ht_in + LEQ, kNonlin ? ht_ex : NLEQ * ht_ex + LEQ,
                   G * ht_in * madd(nxsi, nxsi, mul_rn(ny, ny)), G * ht_ex * madd(nxse, nxse, mul_rn(ny, ny)), fh, fhe, ci, ce, ok);
  T f1, fx1i, fy1i, ui, vi, fx2i, fy2i, fx3i, fy3i;
  {
    f1 = kNonlin ? T(1) : NLEQ + LEQ * hb_in;
    fx1i = qx_in * f1 * sf_in;
    fy1i = qy_in * f1;
    const T fu = kNonlin ? qx_in : NLEQ * qx_in;
    const T fv = kNonlin ? qy_in : NLEQ * qy_in;
    const T fg = nleqg * ze_in;
    ui = qx_in * fh;
    vi = qy_in * fh;
    const T huu = fu * ui, hvv = fv * vi, huv = fu * vi;
    const T gh2 = kNonlin ? fg * (T(0.5) * ze_in + hb_in) : fg * (T(0.5) * ze_in + hb_in) + T(P.fg_l) * ze_in;
    fx2i = (huu + gh2) * sf_in;
    fy2i = huv;
    fx3i = huv * sf_in;
    fy3i = hvv + gh2;
  }
  T fx1e, fy1e, ue, ve, fx2e, fy2e, fx3e, fy3e;
  {
    const T f1e = kNonlin ? T(1) : NLEQ + LEQ * hb_ex;
    fx1e = qx_ex * f1e * sf_ex;
    fy1e = qy_ex * f1e;
    const T fu = kNonlin ? qx_ex : NLEQ * qx_ex;
    const T fv = kNonlin ? qy_ex : NLEQ * qy_ex;
    const T fg = nleqg * ze_ex;
    ue = qx_ex * fhe;
    ve = qy_ex * fhe;
    const T huu = fu * ue, hvv = fv * ve, huv = fu * ve;
    const T gh2 = kNonlin ? fg * (T(0.5) * ze_ex + hb_ex) : fg * (T(0.5) * ze_ex + hb_ex) + T(P.fg_l) * ze_ex;
    fx2e = (huu + gh2) * sf_ex;
    fy2e = huv;
    fx3e = huv * sf_ex;
    fy3e = hvv + gh2;
  }
  const T f1a = T(0.5) * ((fx1i + fx1e) * nx + (fy1i + fy1e) * ny);
  const T f2a = T(0.5) * ((fx2i + fx2e) * nx + (fy2i + fy2e) * ny);
  const T f3a = T(0.5) * ((fx3i + fx3e) * nx + (fy3i + fy3e) * ny);
  const T uni = kNonlin ? ui * nx + vi * ny : (ui * nx + vi * ny) * NLEQ;
  const T une = kNonlin ? ue * nx + ve * ny : (ue * nx + ve * ny) * NLEQ;
  // max(|un+c|, |un|, |un-c|) over both sides.  For c >= 0 the rounded
  // |un| + c equals the rounded larger of |un + c| and |un - c| exactly, so
  // fmax(|un| + c, |un|) is the same value; with c = NaN (negative depth) both
  // forms reduce to |un|, as fmax skips NaN operands.
  const T eig = larger<kTry>(side_speed(fabs(uni), ci), side_speed(fabs(une), ce));
  Flux3T<T> r;
  r.f = f1a - T(0.5) * eig * j1;
  if (kNonlin) {
    r.g = f2a - T(0.5) * eig * j2;
    r.h = f3a - T(0.5) * eig * j3;
  } else {
    const T nx2 = NLEQ + LEQ * nx * nx, ny2 = NLEQ + LEQ * ny * ny, nxy = nx * ny;
    r.g = f2a - T(0.5) * eig * (j2 * nx2 + LEQ * j3 * nxy);
    r.h = f3a - T(0.5) * eig * (j3 * ny2 + LEQ * j2 * nxy);
  }
  return r;
}

template <bool kNonlin, class T>
__device__ __forceinline__ Flux3T<T> llf(const Physics& P, T ze_in, T ze_ex, T qx_in, T qx_ex, T qy_in, T qy_ex,
                                         T hb_in, T hb_ex, T ht_in, T ht_ex, T sf_in, T sf_ex, T nx, T ny, T G) {
  bool ok = true;
  return llf_ok<kNonlin, T>(P, ze_in, ze_ex, qx_in, qx_ex, qy_in, qy_ex, hb_in, hb_ex, ht_in, ht_ex, sf_in, sf_ex,
                            nx, ny, G, ok);
}

// Trace of the modal state at point j of local edge l (mode 1 is 1 there).
__device__ __forceinline__ void edge_trace(const BasisP1& B, const double* q, int l, int j, double& z,
                                           double& u, double& v) {
  const double p1 = B.phi_edge[l][j][1], p2 = B.phi_edge[l][j][2];
  z = q[0] + q[1] * p1 + q[2] * p2;
  u = q[3] + q[4] * p1 + q[5] * p2;
  v = q[6] + q[7] * p1 + q[8] * p2;
}

// Exterior (ghost) state of a boundary edge point from the in-side trace
// (land_edge_hydro.F:201-218, ocean_edge_hydro.F:148-177 and 255-259,
// flow_edge_hydro.F:126-150, radiation_edge_hydro.F:173-193,
// ebarrier_edge_hydro.F:120-160).  Point j of the edge, normal (nx, ny).
// The ocean elevation sum and its depth-positivity fix are FP64 in every
// variant.
__device__ __forceinline__ void ghost_state(const StageArgs& A, unsigned kind, int list, int j, real zi, real xi,
                                            real yi, real hbi, real nx, real ny, real& zx, real& xx, real& yx) {
  const Physics& P = A.ph;
  const real tx = -ny, ty = nx;
  zx = zi;
  xx = xi;
  yx = yi;
  if (kind == kOcean) {
    // endpoint values EMO*RFF*COS(ARGJ-EFA) come from the host for this stage
    double zsum = 0.0;
    for (int f = 0; f < A.m.nbfr; ++f) {
      const double* zg = A.ocean_zg + ((size_t)f * A.m.needs + list) * 2;
      zsum = zsum + (0.5 * (zg[0] + zg[1]) + 0.5 * (zg[1] - zg[0]) * cBasis.xegp[j]);
    }
    const double hbd = hbi;
    if (zsum * P.ifnlfa + hbd <= 0) zsum = fabs(hbd) + P.h0;
    zx = (real)zsum;
  } else if (kind == kLand) {
    const real qn = xi * nx + yi * ny, qt = xi * tx + yi * ty;
    const real qne = -qn, qte = qt, den = real(1) / (nx * ty - ny * tx);
    xx = (ty * qne - ny * qte) * den;
    yx = (-tx * qne + nx * qte) * den;
  } else if (kind == kFlow) {
    // per-point terms QNAM_GP*RFF*COS(ARG) come from the host for this stage
    real qne = 0;
    xx = 0;
    yx = 0;
    for (int f = 0; f < A.m.nffr; ++f) {
      qne = qne + (real)A.flow_qn[((size_t)f * A.m.nfeds + list) * 3 + j];
      xx = -(ty * qne - ny * real(0)) / (nx * ty - ny * tx);
      yx = -(-tx * qne + nx * real(0)) / (nx * ty - ny * tx);
    }
  } else if (kind == kRadiation) {
    const real qn = xi * nx + yi * ny, qt = xi * tx + yi * ty;
    const real qne = -qn + real(2) * sqrt(real(P.g) / (hbi + zi)) * zi, qte = qt,
               den = real(1) / (nx * ty - ny * tx);
    xx = (ty * qne - ny * qte) * den;
    yx = (-tx * qne + nx * qte) * den;
  } else if (kind == kEBarrier) {
    const real above = zi - (real)A.m.ebht[list];
    const real subsup = real(2) * above / real(3);
    real qne, qte;
    if (above < real(0.01)) {
      qne = -(xi * nx + yi * ny);
      qte = xi * tx + yi * ty;
    } else {
      qne = (real)stage_ramp(A) * (real)A.m.ebcfsp[list] * subsup * sqrt(subsup * real(P.g));
      qte = 0;
    }
    xx = (ty * qne - ny * qte) / (nx * ty - ny * tx);
    yx = (-tx * qne + nx * qte) / (nx * ty - ny * tx);
  }
}

__device__ __forceinline__ void edge_geometry(const double* xs, const double* ys, int l, double& xlen,
                                              double& nx, double& ny) {
  // calc_normal.F:41-48 on this element's counter-clockwise edge l
  const int a = (l + 1) % 3, b = (l + 2) % 3;
  const double dy = ys[b] - ys[a], dx = xs[b] - xs[a];
  xlen = sqrt(dy * dy + dx * dx);
  nx = (ys[b] - ys[a]) / xlen;
  ny = -(xs[b] - xs[a]) / xlen;
}

// ibarrier_edge_hydro.F:21-607 for one side of internal-barrier segment `seg`;
// both elements of a segment evaluate the whole weir logic and keep their
// own part, so no element writes another's right-hand side.
template <bool kNonlin>
__device__ __noinline__ void ibarrier_side(const StageArgs& A, int seg, int side, double* out9) {
  const BasisP1& B = cBasis;
  const Physics& P = A.ph;
  const MeshView& m = A.m;
  const int ne = m.ne;
  const int elb = m.ib_elem[2 * seg], elf = m.ib_elem[2 * seg + 1];
  const int ledb = m.ib_led[2 * seg], ledf = m.ib_led[2 * seg + 1];
  const int wdb = A.wd[elb], wdf = A.wd[elf];
  for (int c = 0; c < 9; ++c) out9[c] = 0.0;
  if (wdb == 0 && wdf == 0) return;
  double qb[9], qf[9], hbb[3], hbf[3], xb[3], yb[3], xf[3], yf[3];
  for (int c = 0; c < 9; ++c) { qb[c] = A.qin[(size_t)c * ne + elb]; qf[c] = A.qin[(size_t)c * ne + elf]; }
  for (int k = 0; k < 3; ++k) { hbb[k] = m.hb[(size_t)k * ne + elb]; hbf[k] = m.hb[(size_t)k * ne + elf]; }
  for (int v = 0; v < 3; ++v) {
    const int nb = m.nm[(size_t)v * ne + elb], nf = m.nm[(size_t)v * ne + elf];
    xb[v] = m.x[nb]; yb[v] = m.y[nb]; xf[v] = m.x[nf]; yf[v] = m.y[nf];
  }
  double lenb, nxb, nyb, lenf, nxf, nyf;
  edge_geometry(xb, yb, ledb, lenb, nxb, nyb);
  edge_geometry(xf, yf, ledf, lenf, nxf, nyf);
  const double txb = -nyb, tyb = nxb, txf = -nyf, tyf = nxf;
  const double areasb = (xb[0] - xb[2]) * (yb[1] - yb[2]) + (xb[2] - xb[1]) * (yb[0] - yb[2]);
  const double areasf = (xf[0] - xf[2]) * (yf[1] - yf[2]) + (xf[2] - xf[1]) * (yf[0] - yf[2]);
  for (int i = 0; i < 3; ++i) {
    const int gpb = i, gpf = 2 - i;
    double zeb, qxb, qyb, zef, qxf, qyf;
    edge_trace(B, qb, ledb, gpb, zeb, qxb, qyb);
    edge_trace(B, qf, ledf, gpf, zef, qxf, qyf);
    const double hbbp = hbb[0] + hbb[1] * B.phi_edge[ledb][gpb][1] + hbb[2] * B.phi_edge[ledb][gpb][2];
    const double hbfp = hbf[0] + hbf[1] * B.phi_edge[ledf][gpf][1] + hbf[2] * B.phi_edge[ledf][gpf][2];
    const double htb = depth<kNonlin>(P, zeb, hbbp), htf = depth<kNonlin>(P, zef, hbfp);
    const double sfb = m.sfac_edge ? m.sfac_edge[(size_t)(ledb * 3 + gpb) * ne + elb] : 1.0;
    const double sff = m.sfac_edge ? m.sfac_edge[(size_t)(ledf * 3 + gpf) * ne + elf] : 1.0;
    double aboveb = 0.0, abovef = 0.0;
    if (wdb == 1) aboveb = zeb - m.ibht[seg];
    if (wdf == 1) abovef = zef - m.ibht[seg];
    double qbn = 0.0, qfn = 0.0, qbt = 0.0, qft = 0.0;
    int weir = 0;
    if ((abovef <= 0.01 && aboveb <= 0.01) || fabs(abovef - aboveb) < 0.01) {
      qbn = -(qxb * nxb + qyb * nyb);
      qfn = -(qxf * nxf + qyf * nyf);
      qbt = qxb * txb + qyb * tyb;
      qft = qxf * txf + qyf * tyf;
    } else {
      const double ssf = 2.0 * abovef / 3.0, ssb = 2.0 * aboveb / 3.0;
      if (abovef > aboveb && abovef > 0.01) {
        weir = 1;
        qfn = (aboveb > ssf) ? stage_ramp(A) * m.ibcfsb[seg] * aboveb * sqrt(2.0 * P.g * (abovef - aboveb))
                             : stage_ramp(A) * m.ibcfsp[seg] * ssf * sqrt(ssf * P.g);
      } else if (aboveb > abovef && aboveb > 0.01) {
        weir = -1;
        qbn = (abovef > ssb) ? stage_ramp(A) * m.ibcfsb[seg] * abovef * sqrt(2.0 * P.g * (aboveb - abovef))
                             : stage_ramp(A) * m.ibcfsp[seg] * ssb * sqrt(ssb * P.g);
      }
    }
    Flux3 fb{0, 0, 0}, ff{0, 0, 0};
    double qxe = 0.0, qye = 0.0;
    bool done = false;
    if (weir <= 0) {
      qxe = (tyb * qbn - nyb * qbt) / (nxb * tyb - nyb * txb);
      qye = (-txb * qbn + nxb * qbt) / (nxb * tyb - nyb * txb);
      fb = llf<kNonlin>(P, zeb, zeb, qxb, qxe, qyb, qye, hbbp, hbbp, htb, htb, sfb, sfb, nxb, nyb, P.g);
      if (weir < 0) {  // the front side keeps the back side's exterior momentum
        ff = llf<kNonlin>(P, zef, zef, qxf, qxe, qyf, qye, hbfp, hbfp, htf, htf, sff, sff, nxf, nyf,
                          wdf == 0 ? 0.0 : P.g);
        done = true;
      }
    }
    if (!done && weir >= 0) {
      qxe = (tyf * qfn - nyf * qft) / (nxf * tyf - nyf * txf);
      qye = (-txf * qfn + nxf * qft) / (nxf * tyf - nyf * txf);
      ff = llf<kNonlin>(P, zef, zef, qxf, qxe, qyf, qye, hbfp, hbfp, htf, htf, sff, sff, nxf, nyf, P.g);
      if (weir > 0)
        fb = llf<kNonlin>(P, zeb, zeb, qxb, qxe, qyb, qye, hbbp, hbbp, htb, htb, sfb, sfb, nxb, nyb,
                          wdb == 0 ? 0.0 : P.g);
    }
    const Flux3 fo = side == 0 ? fb : ff;
    const int led = side == 0 ? ledb : ledf, gp = side == 0 ? gpb : gpf;
    const double areas = side == 0 ? areasb : areasf, len = side == 0 ? lenb : lenf;
    for (int k = 0; k < 3; ++k) {
      const double w = 2.0 * B.m_inv[k] / areas * len * B.phi_edge[led][gp][k] * B.wegp[gp];
      out9[k] = out9[k] - w * fo.f;
      out9[3 + k] = out9[3 + k] - w * fo.g;
      out9[6 + k] = out9[6 + k] - w * fo.h;
    }
  }
}

// Internal-barrier sides of one stage, one thread per (segment, side), into
// ib_rhs[(2*seg + side)*9 + c]; the stage kernel adds them at the edge's
// place in each element's sum.  Runs before stage_p1 on the same stream
// (both only read the stage's input state).  Segments without an opposite
// edge (ib_elem < 0) are skipped, as in the reference.
template <bool kNonlin>
__global__ void __launch_bounds__(128) ibarrier_sides(const __grid_constant__ StageArgs A) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= 2 * A.m.nibseg) return;
  const int seg = w >> 1, side = w & 1;
  if (A.m.ib_elem[2 * seg] < 0) return;
  ibarrier_side<kNonlin>(A, seg, side, A.ib_rhs + (size_t)w * 9);
}

// ---------------------------------------------------------------------------
// Tile stage kernel.  Block b owns tile b of the tile plan built at create:
// up to kTile consecutive elements (the shape's tile), and for them the edge
// tasks the tile evaluates (boundary edges, edges to out-of-tile elements,
// shared interior edges once) and the halo of out-of-tile neighbours those
// tasks read.  Three phases separated by barriers, kTile threads:
//   1. tile and halo elements: modal state, bathymetry modes and wet/dry flag
//      into shared memory; tile elements also the geometry rows the sums read;
//   2. one thread per edge task: its two elements' modes once into registers,
//      then the LLF flux at the three Lobatto points in the reference's own
//      in/ex orientation with its dry-side rules -> F, G, H per point in
//      shared memory (internal-barrier sides come from ibarrier_sides);
//   3. one thread per element: the nine right-hand sides, each in the
//      reference's order (boundary edges, interior edges in edge-number order
//      as the slot sum of add_internal_flux, rain, area points), the volume
//      fluxes and sources formed where they are added, then the SSP
//      combination.
// Work is split by edge and by element, not by point and mode, because the
// kernel is bound by instruction issue: a finer split repeats the loads of an
// element's modes, the task decode, the weights and the geometry for every
// point and mode (4,670 thread instructions an element and stage in the first
// stage, 1,550 of them FP64, against 2,135 and 1,185 here), and because the
// values of one edge or element give straight-line code whose long dependent
// chains (reciprocals, roots) the compiler interleaves: with a branch per
// operation, as the operators' range checks make, a block of the kernel took
// twice the cycles.  Three blocks of 128 threads with 158 registers and no
// spills: four blocks of 128 registers, five of 96 and six of 80 spill and are
// 11, 25 and 40 % slower.  On 1M elements (strict, wet/dry beach, mean of the
// two stages) 245 us before, 141.5 us now.
// internal_edge_hydro.F, *_edge_hydro.F, rhs_dg_hydro.F, DG_hydro_timestep.F:238-290
// ---------------------------------------------------------------------------

// resident stage threads per SM the register allocation targets (FP64: at most
// 168 registers a thread); a shape of T threads per block is compiled for that
// many over T resident blocks
#ifndef DGSWEM_STAGE_RESIDENT_THREADS
#define DGSWEM_STAGE_RESIDENT_THREADS 384
#endif
constexpr int stage_min_blocks(int threads) {
  return DGSWEM_STAGE_RESIDENT_THREADS / threads > 0 ? DGSWEM_STAGE_RESIDENT_THREADS / threads : 1;
}

// The 12 modal values (ZE, QX, QY, HB modes, contiguous) of shared-memory
// slot `slot` in the arithmetic type: the FP64 slots qs (stride kQStride),
// or their FP32 copy (stride kQfStride) in the mixed variant.
__device__ __forceinline__ void slot_values(const real* qt, int slot, real v[12]) {
#ifdef DGSWEM_MIXED
  const float4* q = reinterpret_cast<const float4*>(qt + slot * kQfStride);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float4 t = q[j];
    v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
  }
#else
  const double2* q = reinterpret_cast<const double2*>(qt + slot * kQStride);
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const double2 t = q[j];
    v[2 * j] = t.x; v[2 * j + 1] = t.y;
  }
#endif
}

// q0 + q1 p1 + q2 p2, a trace at Lobatto point I from a variable's three
// modes.  At the end points (vertices) p1 and p2 are 0, +-1 or 2
// (BasisT::tr): the products are exact and the fused form gives the bits of
// the separately rounded one.  At the midpoint they are +-1/2 (or -1 and 0),
// exact except for subnormal modes, which waves running into still water do
// reach: there the strict build rounds the products.
__device__ __forceinline__ real trace3(int I, const real* q, real p1, real p2) {
#ifndef DGSWEM_FAST_MATH
  if (I == 1) return q[0] + q[1] * p1 + q[2] * p2;
#endif
  return fma(q[2], p2, fma(q[1], p1, q[0]));
}

// One Lobatto point of an interior edge in the reference's in/ex orientation
// (internal_edge_hydro.F): the LLF flux of the two traces, then the dry-side
// rules of :212-302 -> o[0..4] = F, G_in, H_in, G_ex, H_ex.
template <bool kNonlin>
__device__ __forceinline__ void interior_point(const Physics& P, real zi, real zx, real xi, real xx, real yi,
                                           real yx, real hi, real hx, real hti, real htx, real sfi, real sfx,
                                           real nx, real ny, int wd_in, int wd_ex, real* o) {
  const Flux3T<real> f =
      llf<kNonlin, real>(P, zi, zx, xi, xx, yi, yx, hi, hx, hti, htx, sfi, sfx, nx, ny, real(P.g));
  o[0] = f.f; o[1] = f.g; o[2] = f.h; o[3] = f.g; o[4] = f.h;
  if ((wd_in == 0 || wd_ex == 0) && fabs(f.f) > real(1.0e-8)) {
    // internal_edge_hydro.F:212-302: mass flux out of / into a dry
    // element.  The four cases re-evaluate the flux once with changed
    // arguments: the dry side's state replaced by the wet side's with
    // reflected momentum (outflow from a dry element), or gravity off
    // (G = 0) for the dry side's momentum flux.
    const bool in_dry = wd_in == 0;
    const real F0 = f.f;
    const real tx = -ny, ty = nx, den = nx * ty - ny * tx;
    const bool reflect = in_dry ? F0 > real(0) : F0 < real(0);
    // the wet side, whose momentum is reflected onto the dry side
    const real qxw = in_dry ? xx : xi, qyw = in_dry ? yx : yi;
    const real qnw = qxw * nx + qyw * ny, qtw = qxw * tx + qyw * ty;
    const real qnr = -qnw, qtr = qtw;
    const real qxr = (ty * qnr - ny * qtr) / den, qyr = (-tx * qnr + nx * qtr) / den;
    real a_zi = zi, a_zx = zx, a_xi = xi, a_xx = xx, a_yi = yi, a_yx = yx;
    real a_hi = hi, a_hx = hx, a_ti = hti, a_tx = htx, a_si = sfi, a_sx = sfx, a_g = 0;
    if (reflect) {
      a_g = real(P.g);
      if (in_dry) {
        a_zi = zx; a_xi = qxr; a_yi = qyr; a_hi = hx; a_ti = htx; a_si = sfx;
      } else {
        a_zx = zi; a_xx = qxr; a_yx = qyr; a_hx = hi; a_tx = hti; a_sx = sfi;
      }
    }
    const Flux3T<real> r = llf<kNonlin, real>(P, a_zi, a_zx, a_xi, a_xx, a_yi, a_yx, a_hi, a_hx, a_ti, a_tx,
                                              a_si, a_sx, nx, ny, a_g);
    if (reflect) {
      o[0] = r.f;
      if (in_dry) { o[3] = r.g; o[4] = r.h; o[1] = 0; o[2] = 0; }
      else        { o[1] = r.g; o[2] = r.h; o[3] = 0; o[4] = 0; }
    } else {
      if (in_dry) { o[1] = r.g; o[2] = r.h; }
      else        { o[3] = r.g; o[4] = r.h; }
    }
  }
}

// Bathymetry hb and total depth ht at a trace point from elevation z and the
// slot's fourth trace w: w is HB in the FP64 kernels; the mixed kernels'
// FP32 slots hold the depth modes ZE + HB (summed in FP64, then rounded), so
// that a thin water column keeps FP32 relative accuracy instead of being the
// difference of two rounded values of metres.
template <bool kNonlin>
__device__ __forceinline__ void trace_depth(const Physics& P, real z, real w, real& hb, real& ht) {
#ifdef DGSWEM_MIXED
  hb = w - z;
  ht = kNonlin ? w : depth<kNonlin>(P, z, hb);
#else
  hb = w;
  ht = depth<kNonlin>(P, z, hb);
#endif
}

// The volume terms' reciprocal, square root and Manning friction G n^2 /
// depth^(1/3): FP64 by cr_math.cuh's sequences without a branch, ok reset where
// an argument is out of their range (a zero speed is in it), and by the
// operators, out of line, for those.
__device__ __forceinline__ double rcp_try(double x, bool& ok) {
  ok = ok && mid_range(x);
  return rcp_from(x, rcp_seed(x));
}
__device__ __forceinline__ double sqrt_try(double x, bool& ok) {
  ok = ok && (mid_range(x) || x == 0.0);
  const double r = sqrt_from(x, rsqrt_seed(x));
  return x == 0.0 ? x : r;
}
__device__ __forceinline__ double manning_try(double gn2, double depth, bool& ok) {
#ifdef DGSWEM_FAST_MATH
  return gn2 / cbrt(depth);
#else
  double c;
  const bool near = pow_third_try(depth, &c);
  ok = ok && near && mid_range(gn2) && mid_range(c);
  return quot_from(gn2, c, rcp_from(c, rcp_seed(c)));
#endif
}
__device__ __forceinline__ double rcp_slow(double x) { return rcp_any(x); }
__device__ __forceinline__ double sqrt_slow(double x) { return sqrt_any(x); }
__device__ __forceinline__ double manning_slow(double gn2, double depth) { return quot_any(gn2, cube_root(depth)); }
__device__ __forceinline__ float rcp_try(float x, bool&) { return 1.0f / x; }
__device__ __forceinline__ float sqrt_try(float x, bool&) { return sqrtf(x); }
__device__ __forceinline__ float manning_try(float gn2, float depth, bool&) { return gn2 / cube_root(depth); }
__device__ __forceinline__ float rcp_slow(float x) { return 1.0f / x; }
__device__ __forceinline__ float sqrt_slow(float x) { return sqrtf(x); }
__device__ __forceinline__ float manning_slow(float gn2, float depth) { return gn2 / cube_root(depth); }

// Adds the volume integral of element e (rhs_dg_hydro.F:58-470) to its nine
// right-hand sides from its 12 slot values q (ZE, QX, QY modes, then HB or, in
// the mixed variant, depth modes) and geometry rows.  What is the same at the
// three area points is formed once: the mode derivatives' products with the
// inverse Jacobian (drphi and dsphi are constants at p=1: modes 2 and 3 have
// d/dx = 3/2 dsdx and drdx + 1/2 dsdx), the bed slope, M_INV * WAGP, the
// vertices' wind stress and pressure scaled by the ramp (met_forcing.F:49-66).
// The three points' reciprocals, square roots and cube roots come first and in
// straight lines -- long dependent chains, which the compiler interleaves --
// with one test that they are all in range at the end (ok).
template <bool kNonlin, bool kSph, int kTile>
__device__ __forceinline__ void volume_sums(const StageArgs& A, const BasisT<real>& C, const real q[12],
                                            const real* geo, const double* met, int el, int e, real rhs[3][3]) {
  const MeshView& m = A.m;
  const Physics& P = A.ph;
  const PhysR R = phys_r(A);
  const int ne = m.ne;
  const real NLEQ = kNonlin ? real(1) : R.nleq, LEQ = kNonlin ? real(0) : R.leq;
#ifdef DGSWEM_MIXED
  const real hbe[3] = {q[9] - q[0], q[10] - q[1], q[11] - q[2]};  // the slot holds the depth modes ZE + HB
#else
  const real* hbe = q + 9;
#endif
  real zq[3], uq[3], vq[3], hq[3], depth[3], fh[3], tau[3];
  bool ok = true;
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    hq[I] = hbe[0] * C.phi_area[0][I] + hbe[1] * C.phi_area[1][I] + hbe[2] * C.phi_area[2][I];
    zq[I] = q[0] + q[1] * C.phi_area[1][I] + q[2] * C.phi_area[2][I];
    uq[I] = q[3] + q[4] * C.phi_area[1][I] + q[5] * C.phi_area[2][I];
    vq[I] = q[6] + q[7] * C.phi_area[1][I] + q[8] * C.phi_area[2][I];
#ifdef DGSWEM_MIXED
    depth[I] = kNonlin ? q[9] + q[10] * C.phi_area[1][I] + q[11] * C.phi_area[2][I] : zq[I] + hq[I];
#else
    depth[I] = zq[I] + hq[I];
#endif
    fh[I] = rcp_try(kNonlin ? depth[I] : NLEQ * depth[I] + LEQ, ok);
    tau[I] = m.fric ? (real)m.fric[e] : R.fric;
  }
  real gn2 = 0;
  if (m.manning) {
    const real nbar = geo[EGeo::kNbar * kTile + el];
    gn2 = R.g * (nbar * nbar);
#pragma unroll
    for (int I = 0; I < 3; ++I) {
      tau[I] = manning_try(gn2, depth[I], ok);
      tau[I] = tau[I] < R.cf ? R.cf : tau[I];
    }
  }
  if (P.iflinbf == 0) {
#pragma unroll
    for (int I = 0; I < 3; ++I) {
      const real u = uq[I] * fh[I], v = vq[I] * fh[I];
      tau[I] = tau[I] * sqrt_try(u * u + v * v, ok) * fh[I];
    }
  }
  if (__builtin_expect(!ok, 0)) {
#pragma unroll 1
    for (int I = 0; I < 3; ++I) {
      const real d = I == 0 ? depth[0] : I == 1 ? depth[1] : depth[2];
      const real f = rcp_slow(kNonlin ? d : NLEQ * d + LEQ);
      real t = m.fric ? (real)m.fric[e] : R.fric;
      if (m.manning) {
        t = manning_slow(gn2, d);
        if (t < R.cf) t = R.cf;
      }
      if (P.iflinbf == 0) {
        const real u = (I == 0 ? uq[0] : I == 1 ? uq[1] : uq[2]) * f;
        const real v = (I == 0 ? vq[0] : I == 1 ? vq[1] : vq[2]) * f;
        t = t * sqrt_slow(u * u + v * v) * f;
      }
#pragma unroll
      for (int J = 0; J < 3; ++J)
        if (I == J) { fh[J] = f; tau[J] = t; }
    }
  }
  if (P.iflinbf == 0) {
    real hyb = 1;
    if (P.ifhybf == 1) {  // hybrid friction factor from the element-mean depth
#ifdef DGSWEM_MIXED
      const real depth_c = q[9];
#else
      const real depth_c = q[9] + q[0];
#endif
      const real fh_c = real(1) / (kNonlin ? depth_c : real(P.nleq) * depth_c + real(P.leq));
      hyb = pow(real(1) + pow(real(P.hbreak) * fh_c, real(P.ftheta)), real(P.fgamma / P.ftheta));
    }
#pragma unroll
    for (int I = 0; I < 3; ++I) {
      if (P.ifhybf == 1) tau[I] = tau[I] * hyb;
      tau[I] = tau[I] < R.tau_cap ? tau[I] : R.tau_cap;
    }
  }
  const real drdx = geo[EGeo::kDrdx * kTile + el], dsdx = geo[EGeo::kDsdx * kTile + el];
  const real drdy = geo[EGeo::kDrdy * kTile + el], dsdy = geo[EGeo::kDsdy * kTile + el];
  const real x1 = real(1.5) * dsdx, x2 = drdx + real(0.5) * dsdx;
  const real y1 = real(1.5) * dsdy, y2 = drdy + real(0.5) * dsdy;
  const real dhx = madd(hbe[2], x2, hbe[1] * x1), dhy = madd(hbe[2], y2, hbe[1] * y1);
  const real xf1 = C.mw[1][0] * x1, yf1 = C.mw[1][0] * y1, xf2 = C.mw[2][0] * x2, yf2 = C.mw[2][0] * y2;
  const real cori = m.cori ? (real)m.cori[e] : R.cori;
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    const real sfq = kSph ? (real)m.sfac_area[(size_t)I * ne + e] : real(1);
    const real f1 = kNonlin ? real(1) : NLEQ + LEQ * hq[I];
    const real fx = uq[I] * f1 * sfq, fy = vq[I] * f1;
    const real fu = kNonlin ? uq[I] : NLEQ * uq[I], fv = kNonlin ? vq[I] : NLEQ * vq[I];
    const real fg = R.nleqg * zq[I];
    const real u = uq[I] * fh[I], v = vq[I] * fh[I];
    const real huu = fu * u, hvv = fv * v, huv = fu * v;
    const real gt = real(0.5) * zq[I] + hq[I];
    const real gh2 = kNonlin ? real(0) : fg * gt + R.fg_l * zq[I];
    const real gx = (kNonlin ? madd(fg, gt, huu) : huu + gh2) * sfq, gy = huv;
    const real hx = huv * sfq, hy = kNonlin ? madd(fg, gt, hvv) : hvv + gh2;
    real sx = -(tau[I] * uq[I]) + fg * dhx * sfq + cori * vq[I];
    real sy = -(tau[I] * vq[I]) + fg * dhy - cori * uq[I];
    if (P.nws != 0) {
      // met_forcing.F:49-66: the nodal fields are scaled by the ramp each stage
      const real drpsi[3] = {-0.5, 0.5, 0.0}, dspsi[3] = {-0.5, 0.0, 0.5};
      real dpsidx[3], dpsidy[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        dpsidx[a] = drpsi[a] * drdx + dspsi[a] * dsdx;
        dpsidy[a] = drpsi[a] * drdy + dspsi[a] * dsdy;
      }
      const real fw = real(1) / f1, r = (real)stage_ramp(A);
      const double* w = met + el;  // rows wsx, wsy, pr of vertices 1, 2, 3
      const real wx0 = r * (real)w[0], wx1 = r * (real)w[kTile], wx2 = r * (real)w[2 * kTile];
      const real wy0 = r * (real)w[3 * kTile], wy1 = r * (real)w[4 * kTile], wy2 = r * (real)w[5 * kTile];
      const real p0 = r * (real)w[6 * kTile], p1 = r * (real)w[7 * kTile], p2 = r * (real)w[8 * kTile];
      sx = sx + fw * (wx0 * C.psi[0][I] + wx1 * C.psi[1][I] + wx2 * C.psi[2][I]) -
           R.g * sfq * depth[I] * (p0 * dpsidx[0] + p1 * dpsidx[1] + p2 * dpsidx[2]);
      sy = sy + fw * (wy0 * C.psi[0][I] + wy1 * C.psi[1][I] + wy2 * C.psi[2][I]) -
           R.g * depth[I] * (p0 * dpsidy[0] + p1 * dpsidy[1] + p2 * dpsidy[2]);
    }
    const real s0 = C.srfac[0][I], s1 = C.srfac[1][I], s2 = C.srfac[2][I];
    rhs[1][0] = rhs[1][0] + s0 * sx;
    rhs[2][0] = rhs[2][0] + s0 * sy;
    rhs[0][1] = rhs[0][1] + xf1 * fx + yf1 * fy;
    rhs[1][1] = rhs[1][1] + xf1 * gx + yf1 * gy + s1 * sx;
    rhs[2][1] = rhs[2][1] + xf1 * hx + yf1 * hy + s1 * sy;
    rhs[0][2] = rhs[0][2] + xf2 * fx + yf2 * fy;
    rhs[1][2] = rhs[1][2] + xf2 * gx + yf2 * gy + s2 * sx;
    rhs[2][2] = rhs[2][2] + xf2 * hx + yf2 * hy + s2 * sy;
  }
}

// Phase 2 of the stage kernel: an edge task of the tile (word tk, normal
// (nx, ny) from the in to the ex side), its three Lobatto points.  o[3*point +
// {0, 1, 2}] = F, G, H of the in side, and of the ex side unless one of the two
// is dry: then xres holds the ex side's G and H, xo[2*point + {0, 1}].  tflag: 0, kTaskDry where both sides are dry (no flux), or
// kTaskTwo where one is (the dry-side rules of internal_edge_hydro.F:212-302).
constexpr int kTaskDry = 1, kTaskTwo = 2;

// Lobatto point I of a task the main path leaves out: an interior task with one
// dry side or with a value outside the range of llf_ok's sequences, or a
// boundary task.
template <bool kNonlin, bool kSph, int kTile>
__device__ __forceinline__ void edge_point_rare(const StageArgs& A, const real* tab, const real* qt, const int* wds,
                                                int tile0, int hbeg, uint2 tk, Real2 nrm, int I, real* o, real* xo) {
  const MeshView& m = A.m;
  const Physics& P = A.ph;
  const int ne = m.ne;
  const unsigned fl = tk.x, kind = fl & 7u;
  const int sin = (fl >> TaskBits::kInSlot) & 511, led_in = (fl >> TaskBits::kLedIn) & 3;
  const real nx = nrm.x, ny = nrm.y;
  const real* ti = tab + led_in * 6;
  real q[12];
  slot_values(qt, sin, q);
  const real pi1 = ti[2 * I], pi2 = ti[2 * I + 1];
  const real zi = trace3(I, q, pi1, pi2), xi = trace3(I, q + 3, pi1, pi2), yi = trace3(I, q + 6, pi1, pi2);
  real hi, hti, f[5];
  trace_depth<kNonlin>(P, zi, trace3(I, q + 9, pi1, pi2), hi, hti);
  const int gin = kSph ? (sin < kTile ? tile0 + sin : m.tile_halo[hbeg + sin - kTile]) : 0;
  const real sfi = kSph ? (real)m.sfac_edge[(size_t)(led_in * 3 + I) * ne + gin] : real(1);
  if (kind == kInterior) {
    const int sex = (fl >> TaskBits::kExSlot) & 511, led_ex = (fl >> TaskBits::kLedEx) & 3;
    const real* tx = tab + led_ex * 6 + 4;
    const real px1 = tx[-2 * I], px2 = tx[-2 * I + 1];
    slot_values(qt, sex, q);
    const real zx = trace3(I, q, px1, px2), xx = trace3(I, q + 3, px1, px2), yx = trace3(I, q + 6, px1, px2);
    real hx, htx;
    trace_depth<kNonlin>(P, zx, trace3(I, q + 9, px1, px2), hx, htx);
    const int gex = kSph ? (sex < kTile ? tile0 + sex : m.tile_halo[hbeg + sex - kTile]) : 0;
    const real sfx = kSph ? (real)m.sfac_edge[(size_t)(led_ex * 3 + 2 - I) * ne + gex] : real(1);
    interior_point<kNonlin>(P, zi, zx, xi, xx, yi, yx, hi, hx, hti, htx, sfi, sfx, nx, ny, wds[sin], wds[sex], f);
    xo[2 * I] = f[3];
    xo[2 * I + 1] = f[4];
  } else {
    real zx, xx, yx;
    ghost_state(A, kind, (int)tk.y, I, zi, xi, yi, hi, nx, ny, zx, xx, yx);
    // only the ocean ghost has its own elevation (the others copy zi)
    const real htx = kind == kOcean ? depth<kNonlin>(P, zx, hi) : hti;
    const Flux3T<real> r =
        llf<kNonlin, real>(P, zi, zx, xi, xx, yi, yx, hi, hi, hti, htx, sfi, sfi, nx, ny, real(P.g));
    f[0] = r.f; f[1] = r.g; f[2] = r.h;
  }
  o[3 * I] = f[0];
  o[3 * I + 1] = f[1];
  o[3 * I + 2] = f[2];
}

// Returns whether the task is left to edge_point_rare.
template <bool kNonlin, bool kSph, int kTile>
__device__ __forceinline__ bool edge_task(const StageArgs& A, const real* tab, const real* qt, const int* wds,
                                          int tile0, int hbeg, uint2 tk, real nx, real ny, real* o, int* flag) {
  const MeshView& m = A.m;
  const Physics& P = A.ph;
  const int ne = m.ne;
  const unsigned fl = tk.x, kind = fl & 7u;
  const int sin = (fl >> TaskBits::kInSlot) & 511;
  const int wd_in = wds[sin];
  // (barrier sides: ibarrier_sides, launched before this kernel)
  if (kind != kInterior) return kind != kIBarrier && wd_in != 0;
  const int sex = (fl >> TaskBits::kExSlot) & 511;
  const int wd_ex = wds[sex];
  const bool both = wd_in != 0 && wd_ex != 0, none = wd_in == 0 && wd_ex == 0;
  *flag = both ? 0 : none ? kTaskDry : kTaskTwo;
  if (!both) return !none;
  const int led_in = (fl >> TaskBits::kLedIn) & 3, led_ex = (fl >> TaskBits::kLedEx) & 3;
  const real* ti = tab + led_in * 6;
  const real* tx = tab + led_ex * 6 + 4;  // the ex side's points run backwards
  const int gin = kSph ? (sin < kTile ? tile0 + sin : m.tile_halo[hbeg + sin - kTile]) : 0;
  const int gex = kSph ? (sex < kTile ? tile0 + sex : m.tile_halo[hbeg + sex - kTile]) : 0;
  real qi[12], qx[12];
  slot_values(qt, sin, qi);
  slot_values(qt, sex, qx);
  bool ok = true;
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    const real pi1 = ti[2 * I], pi2 = ti[2 * I + 1], px1 = tx[-2 * I], px2 = tx[-2 * I + 1];
    const real zi = trace3(I, qi, pi1, pi2), xi = trace3(I, qi + 3, pi1, pi2), yi = trace3(I, qi + 6, pi1, pi2);
    const real zx = trace3(I, qx, px1, px2), xx = trace3(I, qx + 3, px1, px2), yx = trace3(I, qx + 6, px1, px2);
    real hi, hti, hx, htx;
    trace_depth<kNonlin>(P, zi, trace3(I, qi + 9, pi1, pi2), hi, hti);
    trace_depth<kNonlin>(P, zx, trace3(I, qx + 9, px1, px2), hx, htx);
    const real sfi = kSph ? (real)m.sfac_edge[(size_t)(led_in * 3 + I) * ne + gin] : real(1);
    const real sfx = kSph ? (real)m.sfac_edge[(size_t)(led_ex * 3 + 2 - I) * ne + gex] : real(1);
    const Flux3T<real> f = llf_ok<kNonlin, real, true>(P, zi, zx, xi, xx, yi, yx, hi, hx, hti, htx, sfi, sfx, nx, ny,
                                                       real(P.g), ok);
    o[3 * I] = f.f;
    o[3 * I + 1] = f.g;
    o[3 * I + 2] = f.h;
  }
  return !ok;
}

// The terms of earlier stages in an SSP combination of any form, in their
// order, into out (nine rows, row c at at(c)): term by term, the nine values of
// a stage's state and right-hand side fetched together.  h0: the step-start
// state, fetched by the caller where its coefficient is nonzero.  Bound by the
// latency of those loads: value by value, each with its own loop over the
// stages, a step of SSP(5,2) took 393 us on 200k elements (p=2: 916 us), this
// way 187 (501); SSP(3,2), 132 -> 100.
template <class Args, class At>
__device__ __forceinline__ void ssp_history(const Args& A, At at, double h0[9], double out[9]) {
#pragma unroll
  for (int c = 0; c < 9; ++c) out[c] = 0.0;
#pragma unroll 1
  for (int I = 0; I < A.irk - 1; ++I) {
    const double a = A.a[I], b = A.b[I];
    double r[9];
    if (I > 0 && a != 0.0)
#pragma unroll
      for (int c = 0; c < 9; ++c) h0[c] = A.qhist[I][at(c)];
    if (b != 0.0)
#pragma unroll
      for (int c = 0; c < 9; ++c) r[c] = A.rhist[I][at(c)];
    if (a != 0.0)
#pragma unroll
      for (int c = 0; c < 9; ++c) out[c] = madd(a, h0[c], out[c]);
    if (b != 0.0)
#pragma unroll
      for (int c = 0; c < 9; ++c) out[c] = madd(b, r[c], out[c]);
  }
}

// Phase 3 of the stage kernel: tile element el (global id e).
// The sums are in the arithmetic type, the SSP combination in FP64 (in the
// mixed variant: the RHS rounded to FP32, the stage states and their
// combination FP64).
template <bool kNonlin, bool kSph, int kTile>
__device__ __forceinline__ void element_sums(const StageArgs& A, const real* tab, const double* qs, const real* qt,
                                             const real* geo, const double* met, const real* res,
                                             const int* tflag, const int* wds,
                                             int tbeg, unsigned info, unsigned slots, int el, int e) {
  const BasisT<real>& C = cBasisR;
  const MeshView& m = A.m;
  const Physics& P = A.ph;
  const int ne = m.ne;
  const int wde = wds[el];
  real rhs[3][3], isum[3][3];  // [variable][mode]
#pragma unroll
  for (int V = 0; V < 3; ++V)
#pragma unroll
    for (int K = 0; K < 3; ++K) { rhs[V][K] = 0; isum[V][K] = 0; }
  // one interior edge l in the order of the sum, its flux at r: the nine
  // weights EDFAC * EDGEQ(l, point, mode), negative on the in side
  // (rhs_*_in(k) - w_in * flux), are powers of two times two numbers: EDGEQ is
  // 1/3 (rounded) times 1, 4, 1 for mode 1 and times the factors sw[..][0] for
  // mode 2, and is itself the power of two sw[..][1] for mode 3 (BasisT::sw,
  // checked when the tables are built).
  auto add_edge = [&](int l, const real v[3][3]) {
    const bool is_in = ei_flag(info, l) != 0;
    const real ed = geo[(EGeo::kEdfac + l) * kTile + el];
    const real a = ed * C.edgeq[0][0][0];
    const real wa = is_in ? -a : a, we = is_in ? -ed : ed;
    const real* sw = tab + 18 + (is_in ? 18 : 0) + l * 6;
    real acc[3][3];
#pragma unroll
    for (int I = 0; I < 3; ++I) {
      const real w[3] = {I == 1 ? real(4) * wa : wa, sw[2 * I] * wa, sw[2 * I + 1] * we};
#pragma unroll
      for (int V = 0; V < 3; ++V)
#pragma unroll
        for (int K = 0; K < 3; ++K) {
          acc[V][K] = I == 0 ? mul_rn(w[K], v[I][V]) : madd(w[K], v[I][V], acc[V][K]);
        }
    }
#pragma unroll
    for (int V = 0; V < 3; ++V)
#pragma unroll
      for (int K = 0; K < 3; ++K) isum[V][K] = isum[V][K] + acc[V][K];
  };
  bool plain = (info & 0x1ffu) == 0u;  // three interior edges (kInterior is 0), none with a dry side
  static_assert(kInterior == 0, "einfo's kind bits");
#pragma unroll
  for (int l = 0; l < 3; ++l) plain = plain && tflag[plain ? (slots >> (10 * l)) & kNoTask : 0] == 0;
  if (__builtin_expect(plain, 1)) {
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int l = ei_order(info, s);
      const real* r = res + ((slots >> (10 * l)) & kNoTask) * 9;
      real v[3][3];
#pragma unroll
      for (int I = 0; I < 3; ++I)
#pragma unroll
        for (int V = 0; V < 3; ++V) v[I][V] = r[3 * I + V];
      add_edge(l, v);
    }
  } else {
#pragma unroll 1
    for (int s = 0; s < 3; ++s) {
      const int l = ei_order(info, s);
      const unsigned kind = ei_kind(info, l);
      if (kind == kNone) continue;
      const int ti = (slots >> (10 * l)) & kNoTask;
      const real* r = res + ti * 9;
      if (kind == kIBarrier) {
        const double* o = A.ib_rhs + (size_t)m.tile_tasks[tbeg + ti].y * 9;
#pragma unroll
        for (int V = 0; V < 3; ++V)
#pragma unroll
          for (int K = 0; K < 3; ++K) rhs[V][K] = rhs[V][K] + (real)o[3 * V + K];
        continue;
      }
      if (kind == kInterior) {
        const int tf = tflag[ti];
        if (tf == kTaskDry) continue;
        real v[3][3];  // [point][F, G, H]
#pragma unroll
        for (int I = 0; I < 3; ++I)
#pragma unroll
          for (int V = 0; V < 3; ++V) v[I][V] = r[3 * I + V];
        if (tf == kTaskTwo && ei_flag(info, l) == 0) {
          const real* xr = reinterpret_cast<const real*>(A.xres) + (size_t)(tbeg + ti) * 6;
#pragma unroll
          for (int I = 0; I < 3; ++I) { v[I][1] = xr[2 * I]; v[I][2] = xr[2 * I + 1]; }
        }
        add_edge(l, v);
      } else if (wde != 0) {
        const real areas = egeo_r(m)[(size_t)EGeo::kAreas * ne + e];
        const real xlen = egeo_r(m)[(size_t)(EGeo::kXlen + l) * ne + e];
        const real wb[3] = {real(2) * C.m_inv[0] / areas * xlen, real(2) * C.m_inv[1] / areas * xlen,
                            real(2) * C.m_inv[2] / areas * xlen};
#pragma unroll
        for (int I = 0; I < 3; ++I)
#pragma unroll
          for (int K = 0; K < 3; ++K) {
            const real wk = wb[K] * C.phi_edge[l][I][K] * C.wegp[I];
#pragma unroll
            for (int V = 0; V < 3; ++V) rhs[V][K] = rhs[V][K] - wk * r[3 * I + V];
          }
      }
    }
  }
#pragma unroll
  for (int V = 0; V < 3; ++V)
#pragma unroll
    for (int K = 0; K < 3; ++K) rhs[V][K] = rhs[V][K] + isum[V][K];  // add_internal_flux
  if (P.rainfall == 1) {
    const real src = real(7.0556e-6);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int K = 0; K < 3; ++K) rhs[0][K] = rhs[0][K] + C.srfac[K][i] * src;
  }
  // the step-start state of the SSP combination, in one batch here: its latency
  // is covered by the volume terms (read where it is used, between stores that
  // the compiler cannot reorder, nine round trips cost 70 us of 260 at 1M
  // elements; after the volume terms 3 us; prefetched before the edge sums 3 us)
  double h0[9];
  if (A.irk > 1 && A.ca0 != 0.0)
#pragma unroll
    for (int c = 0; c < 9; ++c) h0[c] = A.qhist[0][(size_t)c * ne + e];
  if (wde != 0) {
    real q[12];
    slot_values(qt, el, q);
    volume_sums<kNonlin, kSph, kTile>(A, C, q, geo, met, el, e, rhs);
  }
  // SSP-RK combination (DG_hydro_timestep.F:238-290), zero coefficients
  // skipped: the stages whose nonzero terms are the current state and
  // right-hand side (the first), or those and the step-start state, without a
  // branch per term; any other stage by ssp_history
  bool bad = false;
  double out[9];
  if (A.ssp != kSspAny) {
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      double acc = 0.0;
      if (A.ssp == kSspTwo) acc = madd(A.ca0, h0[c], acc);
      acc = madd(A.ca, qs[el * kQStride + c], acc);
      out[c] = madd(A.cb, (double)rhs[c / 3][c % 3], acc);
    }
  } else {
    ssp_history(A, [&](int c) { return (size_t)c * ne + e; }, h0, out);
    if (A.ca != 0.0)
#pragma unroll
      for (int c = 0; c < 9; ++c) out[c] = madd(A.ca, qs[el * kQStride + c], out[c]);
    if (A.cb != 0.0)
#pragma unroll
      for (int c = 0; c < 9; ++c) out[c] = madd(A.cb, (double)rhs[c / 3][c % 3], out[c]);
  }
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    bad = bad || isnan(out[c]);
    A.qout[(size_t)c * ne + e] = out[c];
  }
  if (A.rout) {
#pragma unroll
    for (int c = 0; c < 9; ++c) A.rout[(size_t)c * ne + e] = (double)rhs[c / 3][c % 3];
  }
  if (bad) atomicOr(A.err, 1u);
}

template <bool kNonlin, bool kSph, int kTile, int kThreads>
__global__ void __launch_bounds__(kThreads, stage_min_blocks(kThreads))
    stage_p1(const __grid_constant__ StageArgs A) {
  static_assert(kTile % 32 == 0 && kThreads % kTile == 0, "tile shape");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const MeshView& m = A.m;
  const int ne = m.ne;
  const int tid = threadIdx.x;
  const int tile = A.tile_list ? A.tile_list[A.tile_off + (int)blockIdx.x] : (int)blockIdx.x;
  const int tile0 = tile * kTile, n = min(kTile, m.ne_tiled - tile0);
  const int hbeg = tile * m.max_halo, tbeg = tile * m.max_tasks;
  const int2 count = m.tile_count[tile];  // tasks, those of them that read no halo element
  const StageLayout L = stage_layout(kTile, m.max_halo, m.max_tasks, (unsigned)sizeof(real), A.ph.nws != 0);
  double* qs = reinterpret_cast<double*>(smem_raw + L.qs);
  real* geo = reinterpret_cast<real*>(smem_raw + L.geo);
#ifdef DGSWEM_MIXED
  real* qt = reinterpret_cast<real*>(smem_raw + L.qf);  // FP32 copy of the slots
#else
  const real* qt = qs;
#endif
  real* res = reinterpret_cast<real*>(smem_raw + L.res);
  real* tab = reinterpret_cast<real*>(smem_raw + L.tab);  // BasisT::tr, then BasisT::sw
  int* wds = reinterpret_cast<int*>(smem_raw + L.wd);
  int* tflag = reinterpret_cast<int*>(smem_raw + L.tflag);
  double* met = reinterpret_cast<double*>(smem_raw + L.met);  // nodal wind stress and pressure (NWS)
  int* rare = reinterpret_cast<int*>(smem_raw + L.rare);  // number, then ids, of the tasks left to edge_point_rare

  // ---- phase 1: tile and halo elements into shared memory ----
  if (tid < 54) {  // from global memory: constant loads by lane would be replayed 32 times
    if (sizeof(real) == 8)
      cp_async8(tab + tid, gTab + tid);
    else
      cp_async4(tab + tid, gTab + tid);
  }
  // Everything whose address is known: this thread's first task and its
  // element's edge info into registers, the tile's rows by cp.async, and the
  // halo ids, whose elements are copied once they and the tile are here.  The
  // first round of edge tasks reads only tile elements: the halo's second round
  // trip hides behind it.  (A block of more threads than tile elements, for
  // meshes of few tiles, lets the others fetch the halo meanwhile and has one
  // round of tasks.)
  uint2 tk = make_uint2(kIBarrier, 0u);
  Real2 nrm{};
  if (tid < m.max_tasks) {
    tk = m.tile_tasks[tbeg + tid];
    nrm = reinterpret_cast<const Real2*>(m.tile_nrm)[tbeg + tid];
  }
  if (tid == 0) rare[0] = 0;
  const int hj = kThreads > kTile ? tid - kTile : tid;
  const int hid = hj >= 0 && hj < m.max_halo ? m.tile_halo[hbeg + hj] : -1;
  unsigned info = 0, slots = 0;
  if (tid < n) {
    info = m.einfo[tile0 + tid];
    slots = m.eslot[tile0 + tid];
  }
  {
    constexpr int kStep = kThreads / kTile;  // thread t: element t % kTile of every kStep-th row
    const int w = tid % kTile, r0 = tid / kTile;
    if (w < n) {
      const size_t step = (size_t)kStep * ne;
      const int nrow = m.manning ? EGeo::kSmemRows : EGeo::kNbar;
      constexpr unsigned rb = sizeof(real);
      const unsigned gdst = smem_addr(geo) + (unsigned)((EGeo::kDrdx + r0) * kTile + w) * rb;
      const real* gsrc = egeo_r(m) + (size_t)(EGeo::kDrdx + r0) * ne + tile0 + w;
#pragma unroll
      for (int j = 0; j < (EGeo::kSmemRows - EGeo::kDrdx + kStep - 1) / kStep; ++j) {
        if (EGeo::kDrdx + r0 + j * kStep >= nrow) continue;
        if (rb == 8)
          cp_async8_s(gdst + rb * kStep * kTile * j, gsrc + j * step);
        else
          cp_async4_s(gdst + rb * kStep * kTile * j, gsrc + j * step);
      }
    }
  }
  int nd[3] = {0, 0, 0};
  if (A.ph.nws != 0 && tid < n) {
#pragma unroll
    for (int a = 0; a < 3; ++a) nd[a] = m.nm[(size_t)a * ne + tile0 + tid];
  }
  chain_wait();
  chain_next();
  if (tid < n) cp_async4(wds + tid, A.wd + tile0 + tid);
#ifdef DGSWEM_MIXED
  // one thread per tile or halo element: its 12 FP64 values into registers,
  // then its FP32 slot (ZE, QX, QY modes and the depth modes ZE + HB, FP64
  // sums) and, for a tile element, the FP64 state the SSP combination reads
  auto load_slot = [&](int j, int g) {
    double v[12];
#pragma unroll
    for (int r = 0; r < 9; ++r) v[r] = A.qin[(size_t)r * ne + g];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[9 + k] = m.hb[(size_t)k * ne + g];
    if (j < kTile) {
      double2* d = reinterpret_cast<double2*>(qs + j * kQStride);
#pragma unroll
      for (int i = 0; i < 5; ++i) d[i] = make_double2(v[2 * i], v[2 * i + 1]);
    } else {
      wds[j] = A.wd[g];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) v[9 + k] = v[k] + v[9 + k];
    float4* f = reinterpret_cast<float4*>(qt + j * kQfStride);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      f[i] = make_float4((float)v[4 * i], (float)v[4 * i + 1], (float)v[4 * i + 2], (float)v[4 * i + 3]);
  };
#else
  auto load_slot = [&](int j, int g) {
    const unsigned d = smem_addr(qs) + (unsigned)(j * kQStride) * 8u;
    const double* q0 = A.qin + g;
#pragma unroll
    for (int c = 0; c < 9; ++c) cp_async8_s(d + 8u * c, q0 + (size_t)c * ne);
    const double* h0 = m.hb + g;
#pragma unroll
    for (int k = 0; k < 3; ++k) cp_async8_s(d + 72u + 8u * k, h0 + (size_t)k * ne);
    if (j >= kTile) cp_async4(wds + j, A.wd + g);
  };
#endif
  bool halo_here = kThreads > kTile;
  if (kThreads > kTile) {  // the threads beyond the tile's copy the halo
    if (tid < kTile) {
      if (tid < n) load_slot(tid, tile0 + tid);
    } else {
      for (int j = tid - kTile; j < m.max_halo; j += kThreads - kTile) {
        const int g = j == tid - kTile ? hid : m.tile_halo[hbeg + j];
        if (g >= 0) load_slot(kTile + j, g);
      }
    }
    cp_async_wait_all();
    __syncthreads();
  } else {
    if (tid < n) load_slot(tid, tile0 + tid);
    cp_async_wait_all();
    __syncthreads();
    for (int j = tid; j < m.max_halo; j += kThreads) {
      const int g = j == tid ? hid : m.tile_halo[hbeg + j];
      if (g >= 0) load_slot(kTile + j, g);
    }
  }

  // the element's nodal wind stress and pressure, read in phase 3
  if (A.ph.nws != 0 && tid < n) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      cp_async8(met + a * kTile + tid, A.wsx + nd[a]);
      cp_async8(met + (3 + a) * kTile + tid, A.wsy + nd[a]);
      cp_async8(met + (6 + a) * kTile + tid, A.pr + nd[a]);
    }
  }

  // ---- phase 2: one thread per edge task (the next round's task is fetched
  // while this one's is evaluated) ----
  for (int t0 = 0; t0 < count.x; t0 += kThreads) {
    if (!halo_here && t0 + kThreads > count.y) {
      cp_async_wait_all();
      __syncthreads();
      halo_here = true;
    }
    const int t = t0 + tid;
    const uint2 tk0 = tk;
    const Real2 n0 = nrm;
    if (t + kThreads < count.x) {
      tk = m.tile_tasks[tbeg + t + kThreads];
      nrm = reinterpret_cast<const Real2*>(m.tile_nrm)[tbeg + t + kThreads];
    }
    if (t < count.x &&
        edge_task<kNonlin, kSph, kTile>(A, tab, qt, wds, tile0, hbeg, tk0, n0.x, n0.y, res + t * 9, tflag + t))
      rare[1 + atomicAdd(rare, 1)] = t;
  }
  cp_async_wait_all();
  __syncthreads();
  // the tasks left out, a thread per (task, point): in any order, each writes
  // its own values
  const int nrare = rare[0];
  if (nrare > 0) {
    for (int w = tid; w < 3 * nrare; w += kThreads) {
      const int i = w / 3, t = rare[1 + i];
      edge_point_rare<kNonlin, kSph, kTile>(A, tab, qt, wds, tile0, hbeg, m.tile_tasks[tbeg + t],
                                            reinterpret_cast<const Real2*>(m.tile_nrm)[tbeg + t], w - 3 * i,
                                            res + t * 9, reinterpret_cast<real*>(A.xres) + (size_t)(tbeg + t) * 6);
    }
    __syncthreads();
  }

  // ---- phase 3: one thread per element: sums in the reference's order, SSP ----
  if (tid < n)
    element_sums<kNonlin, kSph, kTile>(A, tab, qs, qt, geo, met, res, tflag, wds, tbeg, info, slots, tid, tile0 + tid);
}

// slopelimiter.F:3300-3404: min/max of element means over each node's star,
// stored as (min, max) pairs per variable, minmax[(var*NP + n)*2 + {0,1}]:
// the limiter pass gathers a node's bounds of a variable with one 16-byte
// load (one sector; six separate arrays took two 8-byte loads from two
// sectors), and this pass writes three coalesced pair arrays.
// Bound by the latency of its gathers: a star is read kStarBatch elements at a
// time, the last repeated to fill a batch, which leaves a minimum as it is
// (500k nodes: 21.1 us one at a time, 20.4 by three, 21.9 by four, 21.0 by six).
constexpr int kStarBatch = 3;
__global__ void node_minmax(const __grid_constant__ LimitArgs L) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int p0 = n < L.m.np ? L.m.star_ptr[n] : 0, p1 = n < L.m.np ? L.m.star_ptr[n + 1] : 0;
  chain_wait();
  chain_next();
  if (n >= L.m.np) return;
  const int ne = L.m.ne;
  double zmin = 99999., zmax = -99999., xmin = 99999., xmax = -99999., ymin = 99999., ymax = -99999.;
#pragma unroll 1
  for (int p = p0; p < p1; p += kStarBatch) {
    int e[kStarBatch];
    double zt[kStarBatch], xt[kStarBatch], yt[kStarBatch];
#pragma unroll
    for (int j = 0; j < kStarBatch; ++j) e[j] = L.m.star[min(p + j, p1 - 1)];
#pragma unroll
    for (int j = 0; j < kStarBatch; ++j) {
      zt[j] = L.q[e[j]];
      xt[j] = L.q[(size_t)3 * ne + e[j]];
      yt[j] = L.q[(size_t)6 * ne + e[j]];
    }
#pragma unroll
    for (int j = 0; j < kStarBatch; ++j) {
      zmin = zt[j] < zmin ? zt[j] : zmin; xmin = xt[j] < xmin ? xt[j] : xmin; ymin = yt[j] < ymin ? yt[j] : ymin;
      zmax = zt[j] > zmax ? zt[j] : zmax; xmax = xt[j] > xmax ? xt[j] : xmax; ymax = yt[j] > ymax ? yt[j] : ymax;
    }
  }
  const size_t np = (size_t)L.m.np;
  double2* o = reinterpret_cast<double2*>(L.minmax);
  o[n] = make_double2(zmin, zmax);
  o[np + n] = make_double2(xmin, xmax);
  o[2 * np + n] = make_double2(ymin, ymax);
}

// bounds (min, max) of variable var at node nd
__device__ __forceinline__ double2 node_bounds(const double* minmax, int np, int nd, int var) {
  return reinterpret_cast<const double2*>(minmax)[(size_t)var * np + nd];
}

// x / 3 in the arithmetic type: the correctly rounded FP64 quotient without
// a division (div3, cr_math.cuh), the FP32 division in the mixed variant
__device__ __forceinline__ double third_of(double x) { return div3(x); }
__device__ __forceinline__ float third_of(float x) { return x / 3.0f; }

// Whether a redistribution sweep of vertex values vx about the mean z0 would
// start from sumdif == +0 with every vx - vmin free of a sign bit: such a sweep
// changes no bit, as each redfac is +0 (the quotient of +0, or 0, capped by a
// non-negative redmax), so vx - redfac leaves vx (a -0 included) and the next
// sweep starts from the same values.  Stopping there gives the bits of running
// all three sweeps.
__device__ __forceinline__ bool sweep_idle(const real vx[3], const real vmin[3], real z0, real& sumdif) {
  const real sumloc = third_of(vx[0] + vx[1] + vx[2]);
  sumdif = (sumloc - z0) * real(3);
  return !signbit(sumdif) && sumdif == real(0) && !signbit(vx[0] - vmin[0]) && !signbit(vx[1] - vmin[1]) &&
         !signbit(vx[2] - vmin[2]);
}

// slopelimiter.F:3555-3677: the three sweeps that restore the element mean z0
__device__ __forceinline__ void sweeps(real vx[3], const real vmin[3], const real vmax[3], real z0) {
#pragma unroll 1
  for (int sweep = 0; sweep < 3; ++sweep) {
    real sumdif;
    if (sweep_idle(vx, vmin, z0, sumdif)) break;
    const real signdif = copysign(real(1), sumdif);
    real dif[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) dif[a] = (vx[a] - z0) * signdif;
    // sumdif is shared out over the vertices left with dif > 0, the next vertex
    // included: a third if all three have it, else a half or all of it (exact
    // scalings).  As selects: the branches on that count left a warp's 32 pairs
    // a few lanes at a time.  Only the third, a division, stays a branch.
    const bool up0 = dif[0] > 0, up1 = dif[1] > 0, up2 = dif[2] > 0, pos = signdif > 0;
    real first = sumdif * signdif;
    if (up0 && up1 && up2)
      first = third_of(first);
    else
      first = first * (up1 || up2 ? real(0.5) : real(1));
    const real half = up2 ? real(0.5) : real(1);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      real redfac = k == 0 ? first : k == 1 ? sumdif * signdif * half : sumdif * signdif;
      if (!(k == 0 ? up0 : k == 1 ? up1 : up2)) redfac = 0;
      const real redmax = pos ? vx[k] - vmin[k] : vmax[k] - vx[k];
      redfac = fmin(redfac, redmax);
      const real red = redfac * signdif;
      sumdif = sumdif - red;
      vx[k] = vx[k] - red;
    }
  }
}

// slopelimiter.F:3434-3779 (vertex clamp + 3 redistribution sweeps) followed
// by wetdry.F:61-548 for the same element.  The limiter arithmetic is in the
// arithmetic type (FP32 in the mixed variant, on deviations from the element
// mean, which it does not change), WETDRY in FP64.
// Many (element, variable) pairs need a sweep where waves cross the mesh, if
// only to take up a rounding of the mean; few near rest.  Run by the element's
// own thread, a variable at a time, those lanes kept the whole warp through up
// to nine sweeps (1,480 warp against 720 thread instructions an element).  So a
// warp of the FP64 builds first clamps all three variables, collects the pairs
// that need sweeps in shared memory, and then sweeps them 32 at a time: 68.0 ->
// 61.4 us on 1M elements, 1,260 warp instructions; 56.2 us with the sweep's
// shares as selects and blocks of 64, 54.4 with the clamp below.  The mixed
// variant, which sweeps only clamped variables, keeps them in place (34.9 us
// against 36.1 on 760k elements; 32.3 with the selects).
// Compiled per limiter shape (kLimitBlocks / kLimitMinBlocks).
constexpr int kLimitPairs = 96;  // (element, variable) pairs of a warp
template <int kBlock, int kMinBlocks>
__global__ void __launch_bounds__(kBlock, kMinBlocks) limit_wetdry(const __grid_constant__ LimitArgs L) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int ne = L.m.ne, np = L.m.np;
  const BasisP1& B = cBasis;
  const bool live = e < L.ne_act;
  int nd[3] = {0, 0, 0};
  if (live) {
#pragma unroll
    for (int v = 0; v < 3; ++v) nd[v] = L.m.nm[(size_t)v * ne + e];
  }
  chain_wait();
  chain_next();
  double q[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) q[c] = live ? L.q[(size_t)c * ne + e] : 0.0;
  // the element means (mode 1 of ZE, QX, QY) and WDFLG change only in
  // WETDRY: values whose bits did not change are not stored again (modes
  // 2-3 are rebuilt by the limiter and stored always)
  const double m0 = q[0], m3 = q[3], m6 = q[6];
#ifdef DGSWEM_MIXED
  // mixed variant: modes 2-3 of a variable are stored only where the
  // limiter rebuilt them or WETDRY changed a mode
  bool rebuilt[3] = {false, false, false}, wd_modes = false;
#endif
  if (L.slopeflag != 0) {
#ifndef DGSWEM_MIXED
    // pair i of the warp: the clamped vertex values and the (FP64) mean at
    // item[0..3][i], its places in the node bounds, which the owner has just
    // fetched, at node[0..2][i]
    __shared__ double items[kBlock / 32][4][kLimitPairs];
    __shared__ int nodes[kBlock / 32][3][kLimitPairs];
    double(*item)[kLimitPairs] = items[threadIdx.x / 32];
    int(*node)[kLimitPairs] = nodes[threadIdx.x / 32];
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    int npair = 0, at[3];
#endif
#pragma unroll
    for (int var = 0; var < 3; ++var) {
      double* zc = &q[3 * var];
#ifdef DGSWEM_MIXED
      // FP32 on deviations from the element mean (mode 1): vertex value -
      // mode 1 and bound - mode 1 (differences in FP64).  The sweeps and
      // the rebuild of modes 2-3 are the reference's with mode 1 = 0 (the
      // mean cancels exactly in both), so FP32 rounds only the small
      // deviations, not the full vertex values.  A variable whose three
      // vertex values lie within their bounds is left as it is: the clamp
      // changes nothing, and the sweeps and the rebuild are the identity in
      // exact arithmetic (the reference's FP64 rebuild returns the modes to
      // rounding), so its FP64 modes are kept rather than rounded to FP32.
      const real z0 = 0;
      real vmin[3], vmax[3], vx[3];
      bool clamped = false;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double2 bd = node_bounds(L.minmax, np, nd[a], var);
        vmin[a] = (real)(bd.x - zc[0]);
        vmax[a] = (real)(bd.y - zc[0]);
        const real v = (real)(B.phi_corner[a][1] * zc[1] + B.phi_corner[a][2] * zc[2]);
        vx[a] = fmax(fmin(v, vmax[a]), vmin[a]);
        clamped = clamped || v > vmax[a] || v < vmin[a];
      }
      if (!clamped) continue;
      rebuilt[var] = true;
      sweeps(vx, vmin, vmax, z0);
      zc[1] = -(real(1.0 / 6.0) * (vx[0] + vx[1])) + real(1.0 / 3.0) * vx[2];
      zc[2] = -(real(.5) * vx[0]) + real(.5) * vx[1];
#else
      const real z0 = zc[0];
      real vmin[3], vmax[3], vx[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double2 bd = node_bounds(L.minmax, np, nd[a], var);
        vmin[a] = bd.x;
        vmax[a] = bd.y;
        vx[a] = zc[0] + B.phi_corner[a][1] * zc[1] + B.phi_corner[a][2] * zc[2];
        // one comparison each (fmin and fmax also look for NaN bounds, which
        // node_minmax never leaves; a NaN vertex value takes the bound here
        // too): 1M elements 56.0 -> 54.4 us
        vx[a] = vx[a] <= vmax[a] ? vx[a] : vmax[a];
        vx[a] = vx[a] >= vmin[a] ? vx[a] : vmin[a];
      }
      bool sweep = live;
      real sumdif;
      if (sweep_idle(vx, vmin, z0, sumdif)) {
        sweep = false;
        zc[1] = -(real(1.0 / 6.0) * (vx[0] + vx[1])) + real(1.0 / 3.0) * vx[2];
        zc[2] = -(real(.5) * vx[0]) + real(.5) * vx[1];
      }
      const unsigned need = __ballot_sync(0xffffffffu, sweep);
      at[var] = sweep ? npair + __popc(need & below) : -1;
      npair += __popc(need);
      if (sweep) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          item[a][at[var]] = vx[a];
          node[a][at[var]] = var * np + nd[a];
        }
        item[3][at[var]] = z0;
      }
#endif
    }
#ifndef DGSWEM_MIXED
    __syncwarp();
    for (int i = threadIdx.x & 31; i < npair; i += 32) {
      real vx[3], vmin[3], vmax[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double2 bd = node_bounds(L.minmax, np, node[a][i], 0);
        vx[a] = item[a][i];
        vmin[a] = bd.x;
        vmax[a] = bd.y;
      }
      sweeps(vx, vmin, vmax, item[3][i]);
#pragma unroll
      for (int a = 0; a < 3; ++a) item[a][i] = vx[a];
    }
    __syncwarp();
#pragma unroll
    for (int var = 0; var < 3; ++var) {
      if (at[var] < 0) continue;
      const real v0 = item[0][at[var]], v1 = item[1][at[var]], v2 = item[2][at[var]];
      q[3 * var + 1] = -(real(1.0 / 6.0) * (v0 + v1)) + real(1.0 / 3.0) * v2;
      q[3 * var + 2] = -(real(.5) * v0) + real(.5) * v1;
    }
#endif
  }
  if (!live) return;
  if (L.wetdry) {
    const double H0 = L.ph.h0, ZERO = 1.0e-6, c13 = 1.0 / 3.0, c16 = 1.0 / 6.0;
    double dpn[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) dpn[v] = L.m.dp[nd[v]];
    const double dpe_min = fmin(fmin(dpn[0], dpn[1]), dpn[2]);
    int wd = L.wd[e];
    const int wd_read = wd;
    int ndry = 0, hmax_i = 0;
    double hmax = ZERO, ht[3], zn[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      zn[v] = q[0] + B.phi_corner[v][1] * q[1] + B.phi_corner[v][2] * q[2];
      ht[v] = dpn[v] + zn[v];
      if (ht[v] > hmax) { hmax_i = v; hmax = ht[v]; }
      if (ht[v] <= H0 + ZERO) ++ndry;
    }
    const double dp_avg = c13 * (dpn[0] + dpn[1] + dpn[2]);
    double zh[3] = {0.0, 0.0, 0.0};
    bool check = false;
    if (ndry == 0) {
      if (wd != 1) {
        zh[0] = zn[0]; zh[1] = zn[1]; zh[2] = zn[2];
        check = true;
      }
    } else {
#ifdef DGSWEM_MIXED
      wd_modes = true;
#endif
      const double ht_avg = q[0] + dp_avg;
      if (ndry == 3 || ht_avg <= H0 + ZERO) {  // cases 2 and 3A: flatten, stop flow
        q[0] = ht_avg - dp_avg;
        if (ht_avg < ZERO) q[0] = ZERO - dp_avg;
        q[1] = -L.m.hb[(size_t)ne + e];
        q[2] = -L.m.hb[(size_t)2 * ne + e];
#pragma unroll
        for (int c = 3; c < 9; ++c) q[c] = 0.0;
        if (ndry == 3) {
          wd = 0;
        } else {
          zh[0] = q[0]; zh[1] = q[0]; zh[2] = q[0];
          check = true;
        }
      } else {  // case 3B: move water to the dry vertices, momentum to the wet ones
        // vertices shallow -> deep: the reference's exchange sort of the
        // index list (pairs (1,2), (1,3), (2,3) in that order, swapping when
        // the first depth is larger), held as (depth, vertex) registers
        double s0 = ht[0], s1 = ht[1], s2 = ht[2];
        int j0 = 0, j1 = 1, j2 = 2;
        if (s0 > s1) { const double t = s0; s0 = s1; s1 = t; const int u = j0; j0 = j1; j1 = u; }
        if (s0 > s2) { const double t = s0; s0 = s2; s2 = t; const int u = j0; j0 = j2; j2 = u; }
        if (s1 > s2) { const double t = s1; s1 = s2; s2 = t; const int u = j1; j1 = j2; j2 = u; }
        const double d0 = fmax(H0, s0) - s0;
        const double d1 = fmax(H0, s1 - 0.5 * d0) - s1;
        const double d2 = -d0 - d1;
        double dh[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) dh[v] = j0 == v ? d0 : (j1 == v ? d1 : d2);
        int nd2 = 0;
        double qxs = 0.0, qys = 0.0, hmax2 = 0.0, hh[3], qxn[3], qyn[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          hh[v] = ht[v] + dh[v];
          if (hh[v] > hmax2) { hmax_i = v; hmax2 = hh[v]; }
          qxn[v] = q[3] + B.phi_corner[v][1] * q[4] + B.phi_corner[v][2] * q[5];
          qyn[v] = q[6] + B.phi_corner[v][1] * q[7] + B.phi_corner[v][2] * q[8];
          if (hh[v] <= H0 + 1.0e-10) { ++nd2; qxs = qxs + qxn[v]; qys = qys + qyn[v]; }
        }
        if (nd2 == 3) {
#pragma unroll
          for (int c = 3; c < 9; ++c) q[c] = 0.0;
        } else {
          // / (3 - nd2), nd2 in {0, 1, 2}: by 3 correctly rounded, by 2 and 1 exact
          qxs = nd2 == 0 ? div3(qxs) : nd2 == 1 ? qxs * 0.5 : qxs;
          qys = nd2 == 0 ? div3(qys) : nd2 == 1 ? qys * 0.5 : qys;
          double qxh[3], qyh[3];
#pragma unroll
          for (int v = 0; v < 3; ++v) {
            const bool dry = hh[v] <= H0 + 1.0e-10;
            qxh[v] = dry ? 0.0 : qxn[v] + qxs;
            qyh[v] = dry ? 0.0 : qyn[v] + qys;
          }
          q[3] = c13 * (qxh[0] + qxh[1] + qxh[2]);
          q[4] = -(c16 * (qxh[0] + qxh[1])) + c13 * qxh[2];
          q[5] = -(0.5 * qxh[0]) + 0.5 * qxh[1];
          q[6] = c13 * (qyh[0] + qyh[1] + qyh[2]);
          q[7] = -(c16 * (qyh[0] + qyh[1])) + c13 * qyh[2];
          q[8] = -(0.5 * qyh[0]) + 0.5 * qyh[1];
        }
#pragma unroll
        for (int v = 0; v < 3; ++v) zh[v] = hh[v] - dpn[v];
        q[1] = -(c16 * (zh[0] + zh[1])) + c13 * zh[2];
        q[2] = -(0.5 * zh[0]) + 0.5 * zh[1];
        check = true;
      }
    }
    if (check) {
      const double zmax = hmax_i == 0 ? zh[0] : (hmax_i == 1 ? zh[1] : zh[2]);
      if (zmax > (-dpe_min + H0)) {
        wd = 1;
      } else {
#pragma unroll
        for (int c = 3; c < 9; ++c) q[c] = 0.0;
        wd = 0;
#ifdef DGSWEM_MIXED
        wd_modes = true;
#endif
      }
    }
    if (wd != wd_read) L.wd[e] = wd;
  }
  auto same = [](double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); };
  if (!same(q[0], m0)) L.q[e] = q[0];
  if (!same(q[3], m3)) L.q[(size_t)3 * ne + e] = q[3];
  if (!same(q[6], m6)) L.q[(size_t)6 * ne + e] = q[6];
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    if (c % 3 == 0) continue;
#ifdef DGSWEM_MIXED
    if (!rebuilt[c / 3] && !wd_modes) continue;
#endif
    L.q[(size_t)c * ne + e] = q[c];
  }
}

// write_results.F:14-170 (modal2nodal) + NODECODE from the wet flags; node n
// of the device order writes its results at its input position
__global__ void modal2nodal_kernel(MeshView m, const double* __restrict__ q, const int* __restrict__ wd,
                                   double nleq, double leq, double* eta2, double* uu2, double* vv2,
                                   int* nodecode) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= m.np) return;
  const int ne = m.ne;
  const BasisP1& B = cBasis;
  double area_sum = 0.0;
  int wet = 0;
  for (int p = m.star_ptr[n]; p < m.star_ptr[n + 1]; ++p) {
    const int e = m.star[p];
    if (wd[e] == 0) continue;
    wet = 1;
    const int a = m.nm[e], b = m.nm[(size_t)ne + e], c = m.nm[(size_t)2 * ne + e];
    const double areas = (m.x[a] - m.x[c]) * (m.y[b] - m.y[c]) + (m.x[c] - m.x[b]) * (m.y[a] - m.y[c]);
    area_sum = area_sum + 0.5 * areas;
  }
  double et = 0.0, uu = 0.0, vv = 0.0;
  for (int p = m.star_ptr[n]; p < m.star_ptr[n + 1]; ++p) {
    const int e = m.star[p];
    if (wd[e] == 0) continue;
    const int a = m.nm[e], b = m.nm[(size_t)ne + e], c = m.nm[(size_t)2 * ne + e];
    const int K = (a == n) ? 0 : (b == n) ? 1 : 2;
    const double p1 = B.phi_corner[K][1], p2 = B.phi_corner[K][2];
    const double zd = q[e] + p1 * q[(size_t)ne + e] + p2 * q[(size_t)2 * ne + e];
    const double xd = q[(size_t)3 * ne + e] + p1 * q[(size_t)4 * ne + e] + p2 * q[(size_t)5 * ne + e];
    const double yd = q[(size_t)6 * ne + e] + p1 * q[(size_t)7 * ne + e] + p2 * q[(size_t)8 * ne + e];
    const double hd = m.hb[e] + p1 * m.hb[(size_t)ne + e] + p2 * m.hb[(size_t)2 * ne + e];
    const double areas = (m.x[a] - m.x[c]) * (m.y[b] - m.y[c]) + (m.x[c] - m.x[b]) * (m.y[a] - m.y[c]);
    const double w = 0.50 * areas / area_sum;
    const double fh = 1.0 / (nleq * (zd + hd) + leq);
    et = et + w * zd;
    uu = uu + w * xd * fh;
    vv = vv + w * yd * fh;
  }
  const int out = m.node_perm[n];  // results in the input node order
  if (eta2) eta2[out] = et;
  if (uu2) uu2[out] = uu;
  if (vv2) vv2[out] = vv;
  if (nodecode) nodecode[out] = wet;
}

// Fortran layout ZE(DOFH,NE) <-> state SoA q[c*NE+e] for one variable
// Host (Fortran) layout f[3*e + k] in input element order <-> device SoA
// q[(3*var + k)*NE + i] in device element order: i = inv[e], e = perm[i].
__global__ void fortran_to_soa(const double* __restrict__ f, double* __restrict__ q, int ne, int var,
                               const int* __restrict__ perm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ne) return;
  const int e = perm[i];
#pragma unroll
  for (int k = 0; k < 3; ++k) q[(size_t)(3 * var + k) * ne + i] = f[(size_t)3 * e + k];
}

__global__ void soa_to_fortran(const double* __restrict__ q, double* __restrict__ f, int ne, int var,
                               const int* __restrict__ inv) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int i = inv[e];
#pragma unroll
  for (int k = 0; k < 3; ++k) f[(size_t)3 * e + k] = q[(size_t)(3 * var + k) * ne + i];
}

// Halo of a partitioned handle: the states of stage buffer q (row stride ne)
// at local element ids idx[0..n) to / from a contiguous buffer.  kind 0: the
// element means of ZE, QX, QY (3 doubles); kind 1: the nine modal values and
// WDFLG (10 doubles, WDFLG as 0.0 / 1.0).
__global__ void halo_pack(const double* __restrict__ q, const int* __restrict__ wd, int ne,
                          const int* __restrict__ idx, int n, int kind, double* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int i = idx[j];
  if (kind == 0) {
#pragma unroll
    for (int v = 0; v < 3; ++v) out[(size_t)3 * j + v] = q[(size_t)(3 * v) * ne + i];
  } else {
#pragma unroll
    for (int c = 0; c < 9; ++c) out[(size_t)10 * j + c] = q[(size_t)c * ne + i];
    out[(size_t)10 * j + 9] = (double)wd[i];
  }
}

__global__ void halo_unpack(double* __restrict__ q, int* __restrict__ wd, int ne, const int* __restrict__ idx,
                            int n, int kind, const double* __restrict__ in) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int i = idx[j];
  if (kind == 0) {
#pragma unroll
    for (int v = 0; v < 3; ++v) q[(size_t)(3 * v) * ne + i] = in[(size_t)3 * j + v];
  } else {
#pragma unroll
    for (int c = 0; c < 9; ++c) q[(size_t)c * ne + i] = in[(size_t)10 * j + c];
    wd[i] = (int)in[(size_t)10 * j + 9];
  }
}

// dst[i] = src[idx[i]]: WDFLG between input and device element order
__global__ void gather_int(const int* __restrict__ src, int* __restrict__ dst, const int* __restrict__ idx, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

}  // namespace DGSWEM_VARIANT
}  // namespace dgswem
