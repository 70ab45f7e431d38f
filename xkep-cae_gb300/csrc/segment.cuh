// Segment-segment closest point in exact reference arithmetic, shared by the pair kernels and the
// pruning features.
#pragma once

#include "xk_common.cuh"

// _closest_point_segments_batch (geometry/_compute.py:55-151), operation for operation.
XK_D void closest_exact(const double* xA0, const double* xA1, const double* xB0, const double* xB1, double& s,
                        double& t, double& dist, double* normal, double* diff) {
  const double TOL = 1e-10;
  double dA[3], dB[3], w0[3];
  for (int i = 0; i < 3; ++i) {
    dA[i] = xsub(xA1[i], xA0[i]);
    dB[i] = xsub(xB1[i], xB0[i]);
    w0[i] = xsub(xA0[i], xB0[i]);
  }
  const double a = xdot_es(dA, dA), b = xdot_es(dA, dB), c = xdot_es(dB, dB);
  const double d = xdot_es(dA, w0), e = xdot_es(dB, w0);
  const double det = xsub(xmul(a, c), xmul(b, b));
  double ac = xmul(a, c);
  if (!(ac >= 1e-30)) ac = (ac != ac) ? ac : 1e-30;  // np.maximum keeps NaN
  const bool par = det < xmul(TOL, ac);
  const double sdet = par ? 1.0 : det;
  const double s_unc = par ? 0.0 : xdiv(xsub(xmul(b, e), xmul(c, d)), sdet);
  const double t_unc = par ? 0.0 : xdiv(xsub(xmul(a, e), xmul(b, d)), sdet);
  const bool cok = c > TOL, aok = a > TOL;
  const double sc = cok ? c : 1.0, sa = aok ? a : 1.0;
  s = par ? 0.0 : xclip01(s_unc);
  t = par ? (cok ? xclip01(xdiv(e, sc)) : 0.0) : xclip01(t_unc);
  const bool s_cl = (s_unc < 0.0) || (s_unc > 1.0);
  const bool t_cl = (t_unc < 0.0) || (t_unc > 1.0);
  if (s_cl && !par) t = cok ? xclip01(xdiv(xadd(xmul(b, s), e), sc)) : 0.0;
  if (t_cl && !par) {
    s = aok ? xclip01(xdiv(xsub(xmul(b, t), d), sa)) : 0.0;
    t = cok ? xclip01(xdiv(xadd(xmul(b, s), e), sc)) : 0.0;
  }
  for (int i = 0; i < 3; ++i) diff[i] = xsub(xadd(xA0[i], xmul(s, dA[i])), xadd(xB0[i], xmul(t, dB[i])));
  dist = xsqrt(xdot_es(diff, diff));
  const double sd = (dist >= 1e-30 || dist != dist) ? dist : 1e-30;
  for (int i = 0; i < 3; ++i) normal[i] = xdiv(diff[i], sd);
  if (dist < 1e-30) { normal[0] = 0.0; normal[1] = 0.0; normal[2] = 1.0; }
}

// Sign and range tests of doubles on their bits, in the integer pipe (the FP64 pipe also compares).
XK_D bool below0_64(double x) { return (unsigned long long)__double_as_longlong(x) > 0x8000000000000000ULL; }
XK_D bool above1_64(double x) { return __double_as_longlong(x) > 0x3ff0000000000000LL; }
XK_D bool outside01_64(double x) { return below0_64(x) || above1_64(x); }
XK_D double clip01_64(double x) { return below0_64(x) ? 0.0 : (above1_64(x) ? 1.0 : x); }

// The same closest point for the ordinary case (both segments longer than 2^-14, det > 1e-3 ac, finite): the
// operations of closest_exact in their order, each rounded on its own, so the same bits; the divides share
// their reciprocals and are skipped where the unclamped parameters stand.  False outside that case.
// From the segments' first points, their difference vectors and the squares of these (xdot_es).
XK_D bool closest_exact_fast(const double* xA, const double* dA, double a, const double* xB, const double* dB, double c,
                             double& s, double& t, double& dist, double* normal) {
  double w0[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) w0[i] = xsub(xA[i], xB[i]);
  const double b = xdot_es(dA, dB), d = xdot_es(dA, w0), e = xdot_es(dB, w0);
  const double ac = xmul(a, c), det = xsub(ac, xmul(b, b));
  if (!(in_range64<-29, 140>(a) && in_range64<-29, 140>(c) && __double2hiint(fma(-1e-3, ac, det)) > 0)) return false;
  const Divisor64 qd = divisor64(det);
  const double su = div64(xsub(xmul(b, e), xmul(c, d)), qd), tu = div64(xsub(xmul(a, e), xmul(b, d)), qd);
  s = clip01_64(su);
  t = clip01_64(tu);
  const bool s_cl = outside01_64(su), t_cl = outside01_64(tu);
  if (s_cl || t_cl) {
    const Divisor64 qc = divisor64(c);
    if (s_cl) t = clip01_64(div64(xadd(xmul(b, s), e), qc));
    if (t_cl) {
      s = clip01_64(div64(xsub(xmul(b, t), d), a));
      t = clip01_64(div64(xadd(xmul(b, s), e), qc));
    }
  }
  double diff[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) diff[i] = xsub(xadd(xA[i], xmul(s, dA[i])), xadd(xB[i], xmul(t, dB[i])));
  const double d2 = xdot_es(diff, diff);
  if (!in_range64<-190, 300>(d2)) return false;
  dist = sqrt64(d2);
  const Divisor64 q = divisor64(dist);
#pragma unroll
  for (int i = 0; i < 3; ++i) normal[i] = div64(diff[i], q);
  return true;
}
