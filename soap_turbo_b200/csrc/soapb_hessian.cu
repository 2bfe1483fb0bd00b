// soapb_hessian.cu -- the central-atom Hessian of soap_turbo
// (get_soap_central_hessian, src/soap_turbo.f90:1151-1700) in FP64:
//
//   hess(a, b, v, k2) = sum_d vecs(d, v, i) d^2 q_d / dr_ia dr_jb
//
// for every pair k2 = (site i, neighbour j), a of the central atom and b of
// the neighbour, the self pair's block being minus the sum of the others.
//
// k64_radial_d2 adds the second radial derivatives to the plain FP64 path's
// state (src/soap_turbo_radial.f90:838-861, 895-905, 917-956; unified filter
// seed only); k64_hgeo writes one geometry record per pair (pair_geometry,
// src/soap_turbo.f90:1537-1652); k64_hess is persistent, one CTA per site at a
// time, and follows the reference's two passes around the weight vectors' S
// matrices (see the kernel).  The angular factor Omega = C_k Q_l^m(t) w^m and
// its derivatives are rebuilt from the record where needed (Q_l^m = d^m P_l /
// dt^m, w = (x - iy)/r), as the reference does.  Every sum runs in a fixed order,
// so results repeat bit for bit.
#include "soapb_device.cuh"

namespace soapb {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr int kHessPC = 16;     // pairs per chunk of pass A
constexpr int kHessCols = 13;   // k-sums of a unit of pass B at most (odd: the transpose buffer's row stride)
constexpr int kHessChunk = 256; // pairs whose entries are listed at a time
constexpr int kHessSmemPair = 113 * 1024;  // shared memory of a CTA of which an SM holds two

#define CU_RET(x)                         \
  do {                                    \
    const cudaError_t e_ = (x);           \
    if (e_ != cudaSuccess) return e_;     \
  } while (0)

struct dcx {
  double re, im;
};
__device__ __forceinline__ dcx cx(double r, double i) { return dcx{r, i}; }
__device__ __forceinline__ dcx operator+(dcx a, dcx b) { return cx(a.re + b.re, a.im + b.im); }
__device__ __forceinline__ dcx operator-(dcx a, dcx b) { return cx(a.re - b.re, a.im - b.im); }
__device__ __forceinline__ dcx operator*(dcx a, dcx b) {
  return cx(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
__device__ __forceinline__ dcx operator*(double s, dcx a) { return cx(s * a.re, s * a.im); }

__device__ __forceinline__ double nv_tab(int n) { return n == -3 ? 1.0 : sqrt(1.0 / (double)(2 * n + 5)); }

// One (pair, species) radial expansion with its first and second r
// derivatives (process_block, src/soap_turbo_radial.f90:550-1002, unified
// seed), the polynomials kept whole to alpha + 4 as the reference does.
template <int AMAX>
__device__ void radial_pair_d2(const DevParams &P, const RadSp &S, const double *W, double r_in, bool is_central,
                               double *val, double *der, double *der2) {
  const double sqpi2 = 1.2533141373155002512, isq2 = 0.70710678118654752440;
  const double sq2pi = 0.79788456080286535588, sq8pi = 1.5957691216057307118;
  constexpr int NT = AMAX + 8;
  const int a = S.alpha, n_poly = S.n_poly, n_hi = n_poly + 4;
  const double c = S.c, rs = S.rs, dr = S.dr;
  const double rj = r_in * S.inv_rcut;
  double T1[NT], T2[NT], pol[NT], DT[NT], D2T[NT];  // index n + 3
#pragma unroll
  for (int t = 0; t < NT; ++t) T1[t] = T2[t] = pol[t] = DT[t] = D2T[t] = 0.0;
  const double sig = S.atom_sigma + c * rj, s2 = sig * sig;              // :560-570
  const double isig = 1.0 / sig, is2 = isig * isig, is3 = is2 * isig;
  double amp, ampd, ampd2;                                               // :589-635
  if (!P.scaling_poly) {
    amp = 1.0; ampd = 0.0; ampd2 = 0.0;
  } else if (S.amp_scaling == 0.0) {
    amp = isig; ampd = -c * is2; ampd2 = 2.0 * c * c * is3;
  } else if (S.amp_scaling == 1.0) {
    const double h = 1.0 + 2.0 * (rj * rj * rj) - 3.0 * rj * rj;
    const double hp = 6.0 * rj * rj - 6.0 * rj, hpp = 12.0 * rj - 6.0, g = isig * h;
    amp = (h <= 1.0e-10) ? 0.0 : g;
    ampd = (h <= 1.0e-10) ? 0.0 : hp * isig - c * isig * g;
    ampd2 = (h <= 1.0e-10) ? 0.0 : hpp * isig - 2.0 * c * hp * is2 + 2.0 * c * c * h * is3;
  } else {
    const double h = 1.0 + 2.0 * (rj * rj * rj) - 3.0 * rj * rj;
    if (h <= 1.0e-10) {
      amp = 0.0; ampd = 0.0; ampd2 = 0.0;
    } else {
      const double hp = 6.0 * rj * rj - 6.0 * rj, hpp = 12.0 * rj - 6.0, aa = S.amp_scaling;
      amp = isig * pow(h, aa);
      ampd = aa * pow(h, aa - 1.0) * hp * isig - c * isig * amp;
      ampd2 = (aa * (aa - 1.0) * pow(h, aa - 2.0) * hp * hp + aa * pow(h, aa - 1.0) * hpp) * isig -
              2.0 * c * aa * pow(h, aa - 1.0) * hp * is2 + 2.0 * c * c * pow(h, aa) * is3;
    }
  }
  if (S.do_central && S.cw != 1.0 && is_central) {                       // :638-646
    amp *= S.cw; ampd *= S.cw; ampd2 *= S.cw;
  }
  if (P.radial_enh == 1) {                                               // :651-670
    const double g = rj + sq2pi * sig, f = 1.0 + sq2pi * c;
    ampd2 = ampd2 * g + 2.0 * ampd * f;
    ampd = amp * f + ampd * g;
    amp = amp * g;
  } else if (P.radial_enh == 2) {
    const double g = rj * rj + s2 + sq8pi * sig * rj;
    const double f = 2.0 * rj + 2.0 * sig * c + sq8pi * sig + sq8pi * rj * c;
    const double h = 2.0 + 2.0 * c * c + 2.0 * sq8pi * c;
    ampd2 = ampd2 * g + 2.0 * ampd * f + amp * h;
    ampd = amp * f + ampd * g;
    amp = amp * g;
  }
  // inner overlap on [0, rcut_soft] (:676-698)
  const double es = exp(-0.5 * (rs - rj) * (rs - rj) * is2), e0 = exp(-0.5 * rj * rj * is2);
  double C1 = s2 * es;
  const double C2 = s2 * e0;
  T1[0] = 0.0;
  T1[1] = sqpi2 * sig * (erf((rs - rj) * isq2 * isig) + erf(rj * isq2 * isig));
  for (int n = -1; n <= n_hi; ++n) {
    if (n >= 0) C1 = C1 * dr;
    const double ra = n == -1 ? 0.0 : (double)(n + 1) * nv_tab(n - 2) / nv_tab(n);
    T1[n + 3] = s2 * ra * T1[n + 1] - nv_tab(n - 1) / nv_tab(n) * (rj - 1.0) * T1[n + 2] +
                (C1 - C2) * (1.0 / nv_tab(n));
  }
  double pref = 0.0;
  if (S.has_filter) {                                                    // :721-795
    const double q = S.q, drnf = S.drnf;
    const double iD = 1.0 / (s2 + q), sqiD = sqrt(iD);
    const double sgf = sig * drnf * sqiD, rjf = (s2 * rs + q * rj) * iD, sf2 = sgf * sgf;
    const bool keep = (rs - rj) < 4.0 * sig;
    const double isgf = 1.0 / sgf, isf2 = isgf * isgf;
    pref = keep ? exp(-0.5 * (rs - rj) * (rs - rj) * iD) : 0.0;
    double C2f = sf2 * exp(-0.5 * (rs - rjf) * (rs - rjf) * isf2);
    T2[0] = 0.0;
    T2[1] = sqpi2 * sgf * (erf((1.0 - rjf) * isq2 * isgf) - erf((rs - rjf) * isq2 * isgf));
    for (int n = -1; n <= n_hi; ++n) {
      if (n >= 0) C2f = C2f * dr;
      const double ra = n == -1 ? 0.0 : (double)(n + 1) * nv_tab(n - 2) / nv_tab(n);
      T2[n + 3] = sf2 * ra * T2[n + 1] - nv_tab(n - 1) / nv_tab(n) * (rjf - 1.0) * T2[n + 2] -
                  C2f * (1.0 / nv_tab(n));
      if (n == -1) T2[2] = T2[2] + sf2 * exp(-0.5 * (1.0 - rjf) * (1.0 - rjf) * isf2) * (1.0 / nv_tab(-1));
    }
  }
  for (int n = 1; n <= n_hi; ++n) pol[n + 3] = T1[n + 3] + pref * T2[n + 3];  // :808-812
  {                                                                      // :825-861
    const double f = 1.0 - rj;
    const double g0 = f * is2 + c * f * f * is3, g1 = -(is2 + 2.0 * c * f * is3), g2 = c * is3;
    const double is4 = is2 * is2, is5 = is4 * isig, is6 = is4 * is2;
    const double k0 = -is2, k1 = -4.0 * c * is3, k2 = (1.0 - 3.0 * c * c) * is4, k3 = 2.0 * c * is5,
                 k4 = c * c * is6;
    const double B0 = k0 + k1 * f + k2 * f * f + k3 * f * f * f + k4 * f * f * f * f;
    const double B1 = -(k1 + 2.0 * k2 * f + 3.0 * k3 * f * f + 4.0 * k4 * f * f * f);
    const double B2 = k2 + 3.0 * k3 * f + 6.0 * k4 * f * f, B3 = -(k3 + 4.0 * k4 * f), B4 = k4;
    for (int n = 1; n <= n_poly; ++n) {
      const double R1 = nv_tab(n + 1) / nv_tab(n), R2 = nv_tab(n + 2) / nv_tab(n);
      const double R3 = nv_tab(n + 3) / nv_tab(n), R4 = nv_tab(n + 4) / nv_tab(n);
      DT[n + 3] = g0 * pol[n + 3] + R1 * g1 * pol[n + 4] + R2 * g2 * pol[n + 5];
      D2T[n + 3] = B0 * pol[n + 3] + R1 * B1 * pol[n + 4] + R2 * B2 * pol[n + 5] + R3 * B3 * pol[n + 6] +
                   R4 * B4 * pol[n + 7];
    }
  }
  if (P.basis == 1) {                                                    // :875-908
    const double ss2 = S.sigma_sq0 + s2, iss = 1.0 / ss2, siss = sqrt(iss);
    const bool gm = rj < 4.0 * (S.atom_sigma + sig);
    const double ge = gm ? S.N_gauss * e0 : 0.0;
    const double M0 = gm ? exp(-0.5 * rj * rj * iss) * sqpi2 * sig * S.atom_sigma * siss *
                               (1.0 + erf(S.atom_sigma * isig * rj * isq2 * siss)) * S.N_gauss
                         : 0.0;
    pol[a + 3] = M0;
    const double sc0 = S.sigma_sq0 * s2 * iss, pp = s2 * rj * iss;
    const double M1 = sc0 * ge - pp * M0, M2 = sc0 * ge * (-rj) - pp * M1 + sc0 * M0;
    const double M3 = sc0 * ge * rj * rj - pp * M2 + 2.0 * sc0 * M1;
    const double M4 = sc0 * ge * (-rj * rj * rj) - pp * M3 + 3.0 * sc0 * M2;
    const double is4 = is2 * is2, is5 = is4 * isig, is6 = is4 * is2;
    DT[a + 3] = M1 * is2 + c * M2 * is3;
    D2T[a + 3] = -M0 * is2 - 4.0 * c * M1 * is3 + (1.0 - 3.0 * c * c) * M2 * is4 + 2.0 * c * M3 * is5 +
                 c * c * M4 * is6;
  }
  // transform from g_alpha to g_n (:911-976)
  for (int i = 0; i < a; ++i) {
    double v = 0.0, d = 0.0, d2 = 0.0;
    for (int m = 1; m <= a; ++m) {
      const double w = W[(m - 1) * a + i];
      v = v + w * pol[m + 3];
      d = d + w * (amp * DT[m + 3] + ampd * pol[m + 3]);
      d2 = d2 + w * (amp * D2T[m + 3] + 2.0 * ampd * DT[m + 3] + ampd2 * pol[m + 3]);
    }
    val[i] = amp * v * S.sqrt_rcut;
    der[i] = d * S.inv_sqrt_rcut;
    der2[i] = d2 * S.inv_sqrt_rcut * S.inv_rcut;
  }
}

// ---- second radial derivatives, one thread per pair; the values and first
// derivatives the FP64 descriptor path already holds are left as they are
template <int AMAX>
__global__ void k64_radial_d2(const DevParams P, const DevBatch B, double *rad_der2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= B.n_pairs) return;
  int lo = 0, hi = B.n_sites;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (B.off[mid] <= k) lo = mid; else hi = mid;
  }
  const bool is_self = (B.off[lo] == k);
  const double r = B.rjs[k];
  const unsigned bits = B.bits[k];
  double *r2o = rad_der2 + (size_t)k * P.n_max;
  unsigned todo = 0u;
  for (int s = 0; s < P.n_species; ++s) {
    const RadSp &S = P.rad[s];
    if (((bits >> s) & 1u) && r < S.rcut_hard && (!is_self || S.do_central)) todo |= 1u << s;
    else
      for (int n = 0; n < S.alpha; ++n) r2o[S.nbeg + n] = 0.0;
  }
  // one expansion per valid species; lanes of different species share it
  while (todo) {
    const int s = __ffs(todo) - 1;
    todo &= todo - 1u;
    const RadSp &S = P.rad[s];
    double val[AMAX], der[AMAX], der2[AMAX];
    radial_pair_d2<AMAX>(P, S, P.Wblk + (size_t)s * P.wstride, r, is_self, val, der, der2);
    for (int n = 0; n < S.alpha; ++n) r2o[S.nbeg + n] = der2[n] * S.gscale;
  }
}

// Per-pair record of the Hessian (pair_geometry, src/soap_turbo.f90:1537-1652),
// written once by k64_hgeo and read by k64_hess: offsets in doubles.
struct GeoLayout {
  int nh, invr, F, t, th, w, wh, Q, wp, size;
  __host__ __device__ explicit GeoLayout(int L) {
    const int L1 = L + 1, K = L1 * (L1 + 1) / 2;
    nh = 0;
    invr = 3;
    w = 4;        // 3 complex; the complex values at even offsets
    wh = w + 6;   // 9 complex
    wp = wh + 18; // L + 3 complex: w^m at m + 2, w^-2 = w^-1 = 0
    t = wp + 2 * (L + 3);
    th = t + 3;
    F = th + 9;   // F_l, F'_l, F''_l of each l
    Q = F + 3 * L1;  // K: Q_l^m(t) = d^m P_l / dt^m, and two pads (Q_l^m+1, Q_l^m+2 of the last k are read)
    size = Q + K + 2;
    size += size & 1;
  }
};

__device__ __forceinline__ dcx ldc(const double *p) { return cx(p[0], p[1]); }
__device__ __forceinline__ void stc(double *p, dcx v) {
  p[0] = v.re;
  p[1] = v.im;
}

// get_ilexp (src/soap_turbo_angular.f90:361-422) to lmax, for the F_l of the Hessian
__device__ void ilexp_to(int lmax, double x, double *out) {
  const double xcut = 1.0e-7, x2 = x * x, x4 = x2 * x2, inv_x2 = (x2 > 0.0) ? 1.0 / x2 : 0.0;
  double x2pow = x2 * x2, flm2, flm1, fact = 1.0;
  if (x > 0.0) {
    const double e2 = exp(-2.0 * x2);
    flm2 = fabs((1.0 - e2) / 2.0 / x2);
    flm1 = fabs((x2 - 1.0 + e2 * (x2 + 1.0)) / 2.0 / x4);
  } else {
    flm2 = 1.0;
    flm1 = 0.0;
  }
  for (int l = 0; l <= lmax; ++l) {
    if (l > 0) fact = fact * (2.0 * (double)l + 1.0);
    if (l == 0) {
      out[0] = (x < xcut) ? 1.0 - x2 : flm2;
    } else if (l == 1) {
      out[1] = (x2 / 1000.0 < xcut) ? (x2 - x4) / fact : flm1;
    } else {
      const double ratio = x2pow / fact;
      const double fl = (ratio * (double)l < xcut) ? ratio : fabs(flm2 - (2.0 * (double)l - 1.0) * inv_x2 * flm1);
      x2pow = x2pow * x2;
      flm2 = flm1;
      flm1 = fl;
      out[l] = fl;
    }
  }
}

// ---- pair geometry, one thread per pair: F_l and its first two r-derivatives,
// the unit vector, the gradients and Hessians of t = cos(theta) and
// w = (x - iy)/r, Q_l^m(t) and w^m.  good[k] = 0 for pairs the Hessian skips
// (beyond rcut_max, at the origin, or in no species).  A warp's records are built
// in shared memory (rows of odd length) and copied out side by side: written by
// their threads, a value at a time 1 KB apart, they took 121 us for 88 k pairs.
__device__ void pair_record(const DevParams &P, const DevBatch &B, int kk, double *g, int *good) {
  const int L = P.l_max;
  const GeoLayout Lg(L);
  const double rr = B.rjs[kk];
  const unsigned bits = B.bits[kk];
  const bool ok = rr < P.rcut_max && rr >= 1.0e-10 && bits != 0u;
  good[kk] = ok ? 1 : 0;
  if (!ok) return;
  const int isp = __ffs(bits) - 1;
  const double invr = 1.0 / rr, invr2 = invr * invr;
  g[Lg.invr] = invr;
  const double sscal = P.sig_t_c[isp], sig = P.sig_t[isp] + sscal * rr;
  const double amp = P.rcut2 / (sig * sig), ampd = -2.0 * sscal / sig * amp;
  const double ampdd = 6.0 * sscal * sscal / (sig * sig) * amp;
  const double xarg = rr / sig, invz = 1.0 / (xarg * xarg);
  double il[SOAPB_MAX_LMAX + 3];
  ilexp_to(L + 2, xarg, il);
  const double zp = 2.0 * rr / (sig * sig) - 2.0 * rr * rr * sscal / (sig * sig * sig);
  const double zp2 = 2.0 / (sig * sig) - 8.0 * rr * sscal / (sig * sig * sig) +
                     6.0 * rr * rr * sscal * sscal / (sig * sig * sig * sig);
  for (int l = 0; l <= L; ++l) {
    const double rl = (double)l;
    const double dil = il[l + 1] + (rl * invz - 1.0) * il[l];
    const double d2il = il[l + 2] + ((double)(2 * l + 1) * invz - 2.0) * il[l + 1] +
                        (rl * (rl - 1.0) * invz * invz - 2.0 * rl * invz + 1.0) * il[l];
    const double f0 = il[l], f1 = dil * zp, f2 = d2il * zp * zp + dil * zp2;
    g[Lg.F + 3 * l] = amp * f0;
    g[Lg.F + 3 * l + 1] = ampd * f0 + amp * f1;
    g[Lg.F + 3 * l + 2] = ampdd * f0 + 2.0 * ampd * f1 + amp * f2;
  }
  double nh[3];
  const double sin_t = sin(B.thetas[kk]), cos_t = cos(B.thetas[kk]);
  const double sin_f = sin(B.phis[kk]), cos_f = cos(B.phis[kk]);
  nh[0] = sin_t * cos_f;
  nh[1] = sin_t * sin_f;
  nh[2] = cos_t;
  for (int q = 0; q < 3; ++q) g[Lg.nh + q] = nh[q];
  const double tt = nh[2];
  const dcx wc = cx(nh[0], -nh[1]);
  const dcx ec[3] = {cx(1.0, 0.0), cx(0.0, -1.0), cx(0.0, 0.0)};
  for (int q = 0; q < 3; ++q) {
    g[Lg.t + q] = -tt * nh[q] * invr + (q == 2 ? invr : 0.0);
    stc(g + Lg.w + 2 * q, (-nh[q] * invr) * wc + invr * ec[q]);
  }
  for (int bb = 0; bb < 3; ++bb)
    for (int aa = 0; aa < 3; ++aa) {
      double th = (3.0 * tt * nh[aa] * nh[bb]) * invr2;
      dcx wh = invr2 * ((3.0 * nh[aa] * nh[bb]) * wc - nh[bb] * ec[aa] - nh[aa] * ec[bb]);
      if (bb == 2) th = th - nh[aa] * invr2;
      if (aa == 2) th = th - nh[bb] * invr2;
      if (aa == bb) {
        th = th - tt * invr2;
        wh = wh - invr2 * wc;
      }
      g[Lg.th + bb * 3 + aa] = th;
      stc(g + Lg.wh + 2 * (bb * 3 + aa), wh);
    }
  double *Qt = g + Lg.Q;
  Qt[0] = 1.0;
  if (L >= 1) {
    Qt[1] = tt;
    Qt[2] = 1.0;
  }
  for (int ll = 2; ll <= L; ++ll) {
    const int kbb = ll * (ll + 1) / 2;
    for (int mm = 0; mm <= ll - 2; ++mm) {
      const int kq = kbb + mm;
      Qt[kq] = ((double)(2 * ll - 1) * tt * Qt[kq - ll] - (double)(ll + mm - 1) * Qt[kq - 2 * ll + 1]) /
               (double)(ll - mm);
    }
    Qt[kbb + ll - 1] = (double)(2 * ll - 1) * tt * Qt[kbb - 1];
    Qt[kbb + ll] = (double)(2 * ll - 1) * Qt[kbb - 1];
  }
  Qt[Lg.size - Lg.Q - 1] = Qt[(L + 1) * (L + 2) / 2] = Qt[(L + 1) * (L + 2) / 2 + 1] = 0.0;
  dcx wpow = cx(1.0, 0.0);
  stc(g + Lg.wp, cx(0.0, 0.0));
  stc(g + Lg.wp + 2, cx(0.0, 0.0));
  stc(g + Lg.wp + 4, wpow);
  for (int mm = 1; mm <= L; ++mm) {
    wpow = wpow * wc;
    stc(g + Lg.wp + 2 * (mm + 2), wpow);
  }
}
__global__ void __launch_bounds__(32) k64_hgeo(const DevParams P, const DevBatch B, double *geo, int *good) {
  extern __shared__ double srec[];
  const int k0 = blockIdx.x * 32, lane = threadIdx.x, size = GeoLayout(P.l_max).size, row = size | 1;
  if (k0 + lane < B.n_pairs) pair_record(P, B, k0 + lane, srec + lane * row, good);
  __syncwarp();
  const int n = min(32, B.n_pairs - k0);
  double *o = geo + (size_t)k0 * size;
  for (int i = 0; i < n; ++i)
    for (int t = lane; t < size; t += 32) o[(size_t)i * size + t] = srec[i * row + t];
}

// Per-CTA global scratch of the Hessian kernel (hess_scratch_doubles)
struct HessScratch {
  double2 *G;     // (3, n_max, k_max) complex: sum_j d c_nlm / d r_j
  double *dp1;    // (n_soap, 3): d p / d r_i, unnormalised
  double *kept3;  // (3, n_kept)
  double *vk;     // (3, n_kept): weight vectors spread through the compression
};

__device__ HessScratch carve(double *base, const DevParams &P) {
  HessScratch h;
  h.G = (double2 *)base;
  h.dp1 = base + 6 * (size_t)P.n_max * P.k_max;
  h.kept3 = h.dp1 + 3 * (size_t)P.n_soap;
  h.vk = h.kept3 + 3 * (size_t)P.n_kept;
  return h;
}

// Shared memory of k64_hess, in doubles.
struct HessSmem {
  int Z, red, ck, rad, dot, list, total;
  int rows;  // radial indices whose tables it holds
};
__host__ __device__ inline HessSmem hess_smem(const DevParams &P, int n_vec, int threads) {
  HessSmem S;
  const int N = P.n_max, K = P.k_max, AB = P.amax_t;
  const int n_red = threads * kHessCols, n_rad = (threads / 16) * 4 * AB;
  const int n_dot = 4 + 4 * n_vec, n_list = (kHessChunk * P.n_species + 3) / 4, n_ck = K + (K + 1) / 2;
  // pass B: the tables of one weight vector, of every species where two CTAs
  // then still fit an SM, and the warps' transpose buffers
  int rows = (kHessSmemPair / 8 * (threads / 256) - n_red - n_rad - n_dot - n_list - n_ck - 4) / (8 * K);
  if (rows > N) rows = N;
  if (rows < AB) rows = AB;
  S.rows = rows;
  S.Z = 0;
  S.red = 8 * rows * K;
  const int b = S.red + n_red, a = kHessPC * (12 * K + 2 * AB);  // pass A: a chunk's angular factors and radial rows
  int o = ((a > b ? a : b) + 1) & ~1;
  S.rad = o;  o += n_rad;
  S.ck = o;   o += n_ck;
  S.dot = o;  o += n_dot;
  S.list = o; o += n_list;
  S.total = o;
  return S;
}

// Warp-wise dot product over fixed lane strides and a fixed shuffle tree.
__device__ __forceinline__ double warp_dot(const double *x, int sx, const double *y, int sy, int n) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int t = lane; t < n; t += 32) s += x[(size_t)t * sx] * y[(size_t)t * sy];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Weight vectors of one site: v < n_vec the caller's, v = n_vec the site's
// unnormalised p, v = n_vec + 1 + a the column a of dp1.  Of the first n_vec + 1
// the Hessian is formed; the last three give dp1 . dp_j.
__device__ __forceinline__ double weight(const double *vecs, const double *soap_i, double sv, const double *dp1,
                                         int n_vec, int ns, int site, int v, int o) {
  if (v < n_vec) return vecs[((size_t)site * n_vec + v) * ns + o];
  if (v == n_vec) return soap_i[o] * sv;
  return dp1[3 * o + (v - n_vec - 1)];
}

// Whether pair k takes part for species s: its radial row is not zero and it has a record.
__device__ __forceinline__ unsigned hess_species(const DevParams &P, const DevBatch &B, const int *good, int k) {
  if (!good[k]) return 0u;
  const double r = B.rjs[k];
  const unsigned bits = B.bits[k];
  unsigned ok = 0u;
  for (int s = 0; s < P.n_species; ++s)
    if (((bits >> s) & 1u) && r < P.rad[s].rcut_hard) ok |= 1u << s;
  return ok;
}

// The k-sums of a (pair, weight vector), from Omega = C Q_l^m(t) w^m and its
// derivatives in t and w (d Omega_a = Omega_t t_a + Omega_w w_a and so on, so that
// the Cartesian tensors t_a, w_a, t_ab, w_ab enter once per pair, not per k):
//   0  Re[(z2 - z1/r) Om]   1 Re[z1 Om]   2 Re[z1 Om_t]   3,4 z1 Om_w
//   5  Re[z0 Om_t]  6,7 z0 Om_w  8 Re[z0 Om_tt]  9,10 z0 Om_tw  11,12 z0 Om_ww
//   13 + 4 q: Re[gg1_q Om], Re[gg0_q Om_t], gg0_q Om_w (two)
// with z_i the radial contractions of Z_v and gg_q those of ZG_v's component q
// (:1378-1412, reassociated over k); a vector of which only v . dp_j is needed has
// four: Re[z1 Om], Re[z0 Om_t], z0 Om_w.
constexpr int kSumsFull = 25, kSumsLight = 4;

// The sums of pair records read at one Cartesian element.
__device__ __forceinline__ double re_prod(const double *s, const double *w) { return s[0] * w[0] - s[1] * w[1]; }
// v . dp_j (b) = n_b S2 + Re sum z0 dOm_b
__device__ __forceinline__ double first_der(double s_om, double s_t, const double *s_w, const double *g,
                                            const GeoLayout &Lg, int b) {
  return g[Lg.nh + b] * s_om + s_t * g[Lg.t + b] + re_prod(s_w, g + Lg.w + 2 * b);
}
__device__ __forceinline__ double second_der(const double *S, const double *g, const GeoLayout &Lg, int aa, int bb) {
  const double *t = g + Lg.t, *wa = g + Lg.w + 2 * aa, *wb = g + Lg.w + 2 * bb, *wh = g + Lg.wh + 2 * (bb * 3 + aa);
  const double na = g[Lg.nh + aa], nb = g[Lg.nh + bb];
  const double s3a = S[2] * t[aa] + re_prod(S + 3, wa), s3b = S[2] * t[bb] + re_prod(S + 3, wb);
  const double tw[2] = {t[aa] * wb[0] + t[bb] * wa[0], t[aa] * wb[1] + t[bb] * wa[1]};
  const double ww[2] = {wa[0] * wb[0] - wa[1] * wb[1], wa[0] * wb[1] + wa[1] * wb[0]};
  const double s4 = S[8] * t[aa] * t[bb] + S[5] * g[Lg.th + bb * 3 + aa] + re_prod(S + 9, tw) + re_prod(S + 11, ww) +
                    re_prod(S + 6, wh);
  const double *Sq = S + 13 + 4 * aa;
  const double s6 = Sq[1] * t[bb] + re_prod(Sq + 2, wb);
  return -(na * nb * S[0] + (aa == bb ? g[Lg.invr] * S[1] : 0.0) + na * s3b + nb * s3a + s4 + nb * Sq[0] + s6);
}

// ---- the Hessian, persistent, one CTA per site at a time.  Per site:
//  A  G(n,k) = sum_j d/dr_j [4 pi R_n F_l Omega_k] (:1305-1334), a species'
//     pairs in CSR order and its radial indices only (the others' R_n are
//     zero), with the pairs' angular factors A_j, B_j built in shared memory
//     chunk by chunk; then dp1 = d p / d r_i = -(d p / d c) G component by
//     component of p (the reference sums -dp_j over the pairs; the two agree to
//     rounding, since sum_j d c / d r_j = G);
//  B  per weight vector: the vector spread back through the compression into its
//     S_v(n, n', l) and applied to c_nlm (Z_v) and to G (ZG_v) (:1336-1376), the
//     tables in shared memory; then a half-warp per pair, lanes over k, contracts
//     its species' rows of them with the pair's R_n, R'_n, R''_n and Omega into the
//     k-sums above, Z_v and ZG_v as units of their own;
//  C  per pair: the second derivative hv and the first derivatives v . dp_j (what
//     the reference's self-test rebuilds, here the value used), and from them the
//     normalisation (:1414-1484).
// Sums run in a fixed order (pairs in CSR order, k within a lane, lanes through
// shared memory).
// What bounds it: instructions (280 k per site of 52 pairs, three species, one
// vector; a third of them FP64), issued at 38 % of the rate by 16 warps per SM that
// wait for the pair records, G and c_nlm from L1 and L2.  1.16 ms at 1679 such
// sites.  Against it, 3.07 ms: tables of every radial index read from L2 by every
// pair (190 KB each) and Cartesian tensors of Omega formed per k; 1.81 ms with the
// tables of a species and vector at a time in shared memory, and G beside them, the
// barriers between them taking a quarter of the time.
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k64_hess(const DevParams P, const DevBatch B, const double *rad,
                                                         const double *rad_der, const double *rad_der2,
                                                         const double *geo, const int *good, const double2 *cnk,
                                                         const double *norm, const double *soap, int n_vec,
                                                         const double *vecs, double *hess, double *sums,
                                                         double *scratch, size_t scratch_per_cta, int *ticket) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_site;
  __shared__ int s_base[SOAPB_MAX_SPECIES + 1];
  const int N = P.n_max, K = P.k_max, ns = P.n_soap, nk = P.n_kept, AB = P.amax_t, nsp = P.n_species;
  const int nvh = n_vec + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = lane >> 4, hl = lane & 15;
  constexpr int NW = NT / 32;
  const size_t sp_sums = (size_t)kSumsFull * nvh + 3 * kSumsLight;
  const GeoLayout Lg(P.l_max);
  const HessSmem Ly = hess_smem(P, n_vec, NT);
  const HessScratch h = carve(scratch + scratch_per_cta * blockIdx.x, P);
  double2 *G = h.G;
  const int RT = Ly.rows, NK = N * K;
  double2 *cab = (double2 *)(sm + Ly.Z);  // (pair, A_x, B_x, A_y, .., K): lanes over k side by side
  double *crr = sm + Ly.Z + (size_t)kHessPC * K * 12;
  double2 *sZ = (double2 *)(sm + Ly.Z), *sZG = sZ + (size_t)RT * K;  // (row, K); (q, row, K)
  double *red = sm + Ly.red + (size_t)warp * 32 * kHessCols;
  double *wrad = sm + Ly.rad + (size_t)(2 * warp + half) * 4 * AB;
  double *sdot = sm + Ly.dot;
  unsigned short *list = (unsigned short *)(sm + Ly.list);
  // per k: 4 pi (-1)^m preflm, and l | m << 8
  double *sck = sm + Ly.ck;
  int *klm = (int *)(sck + K);
  const double fourpi = 4.0 * kPi;
  for (int k = tid; k < K; k += NT) {
    const int lm = ((const int *)(P.blob + P.off_klm))[k];
    klm[k] = lm;
    sck[k] = ((lm >> 8) & 1) ? -fourpi * P.preflm64[k] : fourpi * P.preflm64[k];
  }

  for (;;) {
    __syncthreads();
    if (tid == 0) s_site = atomicAdd(ticket, 1);
    __syncthreads();
    const int site = s_site;
    if (site >= B.n_sites) break;
    const int p0 = B.off[site], p1 = min(B.off[site + 1], B.n_pairs);
    const double sv = norm[site], invs = 1.0 / sv, invs3 = invs / (sv * sv), invs5 = invs3 / (sv * sv);
    const double2 *c = cnk + (size_t)site * N * K;
    const double *soap_i = soap + (size_t)site * ns;
    // the entries of species [s_lo, s_hi) among the pairs [c0, c1), pair - c0, from
    // list[s_base[s]] on (every warp writes the same list); whether a pair has several
    auto build = [&](int s_lo, int s_hi, int c0, int c1) {
      __syncthreads();  // the list before is read
      unsigned long long v = 0ull;
      bool several = false;
      for (int t = 0; c0 + 32 * t < c1; ++t) {
        const int k = c0 + 32 * t + lane;
        const unsigned ok = k < c1 ? hess_species(P, B, good, k) : 0u;
        v |= (unsigned long long)ok << (8 * t);
        several |= (ok & (ok - 1u)) != 0u;
      }
      int e = 0;
      for (int s = s_lo; s < s_hi; ++s) {
        if (lane == 0) s_base[s] = e;
        for (int t = 0; c0 + 32 * t < c1; ++t) {
          const bool on = (v >> (8 * t + s)) & 1ull;
          const unsigned m = __ballot_sync(0xffffffffu, on);
          // bit 15: no earlier species of the pair
          if (on)
            list[e + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(
                (32 * t + lane) | ((((v >> (8 * t)) & ((1ull << s) - 1ull)) & 0xffull) ? 0 : 0x8000));
          e += __popc(m);
        }
      }
      if (lane == 0) s_base[s_hi] = e;
      __syncthreads();
      return __any_sync(0xffffffffu, several) != 0;
    };
    // species one at a time where the site takes several chunks, and where a pair's
    // sums come from several species (they are added in the species' order)
    const bool multi = p1 - p0 - 1 > kHessChunk;
    const bool apart = multi || build(0, nsp, p0 + 1, p1);
    // ---- A
    for (int t = tid; t < 3 * NK; t += NT) G[t] = make_double2(0.0, 0.0);
    for (int s = 0; s < nsp; ++s) {
      const int a = P.rad[s].alpha, nb = P.rad[s].nbeg;
      for (int c0 = p0 + 1; c0 < p1; c0 += kHessChunk) {
        if (multi) build(s, s + 1, c0, min(p1, c0 + kHessChunk));
        const int e0 = s_base[s], e1 = s_base[s + 1];
        for (int eb = e0; eb < e1; eb += kHessPC) {
          const int nc = min(kHessPC, e1 - eb);
          __syncthreads();  // the chunk before is read (and G is cleared)
          for (int t = tid; t < nc * 2 * a; t += NT) {
            const int pp = t / (2 * a), r = t - pp * 2 * a;
            const size_t j = c0 + (list[eb + pp] & 0x7fff);
            crr[pp * 2 * AB + (r < a ? r : AB + r - a)] = (r < a ? rad : rad_der)[j * N + nb + (r < a ? r : r - a)];
          }
          for (int t = tid; t < nc * K; t += NT) {
            const int pp = t / K, k = t - pp * K, lm = klm[k], l = lm & 0xff, m = lm >> 8;
            const double *g = geo + (size_t)(c0 + (list[eb + pp] & 0x7fff)) * Lg.size;
            const double C = sck[k];
            const double q0 = C * g[Lg.Q + k], q1 = (m < l) ? C * g[Lg.Q + k + 1] : 0.0;
            const dcx w0 = ldc(g + Lg.wp + 2 * (m + 2)), w1 = ldc(g + Lg.wp + 2 * (m + 1));
            const dcx Om = q0 * w0, Ot = q1 * w0, Ow = (q0 * (double)m) * w1;
            const double f0 = g[Lg.F + 3 * l], f1 = g[Lg.F + 3 * l + 1];
            double2 *o = cab + pp * 6 * K + k;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              const double nq = g[Lg.nh + q];
              const dcx d = (f1 * nq) * Om + f0 * (g[Lg.t + q] * Ot + Ow * ldc(g + Lg.w + 2 * q));
              o[2 * q * K] = make_double2(f0 * nq * Om.re, f0 * nq * Om.im);
              o[(2 * q + 1) * K] = make_double2(d.re, d.im);
            }
          }
          __syncthreads();
          // threads over (k, two radial indices)
          for (int it = tid; it < ((a + 1) >> 1) * K; it += NT) {
            const int n2 = it / K, k = it - n2 * K, n0 = 2 * n2, n1 = min(n0 + 1, a - 1);
            double2 *g0 = G + (nb + n0) * K + k, *g1 = G + (nb + n1) * K + k;
            double2 x[3], y[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              x[q] = g0[q * NK];
              y[q] = g1[q * NK];
            }
            for (int pp = 0; pp < nc; ++pp) {
              const double2 *f = cab + pp * 6 * K + k;
              const double *R = crr + pp * 2 * AB;
              const double r0 = R[n0], d0 = R[AB + n0], r1 = R[n1], d1 = R[AB + n1];
#pragma unroll
              for (int q = 0; q < 3; ++q) {
                const double2 A = f[2 * q * K], D = f[(2 * q + 1) * K];
                x[q].x = x[q].x + d0 * A.x + r0 * D.x;
                x[q].y = x[q].y + d0 * A.y + r0 * D.y;
                y[q].x = y[q].x + d1 * A.x + r1 * D.x;
                y[q].y = y[q].y + d1 * A.y + r1 * D.y;
              }
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              g0[q * NK] = x[q];
              if (n0 + 1 < a) g1[q * NK] = y[q];
            }
          }
        }
      }
    }
    __syncthreads();
    // dp1 in the kept components, then through the compression map
    for (int q = tid; q < nk; q += NT) {
      const int code = P.kept_nnl[q];
      const int n = code & 0xff, np = (code >> 8) & 0xff, l = code >> 16;
      const double base = (n == np) ? 1.0 : sqrt(2.0);
      double d[3] = {0.0, 0.0, 0.0};
      for (int m = 0; m <= l; ++m) {
        const int k = l * (l + 1) / 2 + m;
        const double w = base * ((m > 0) ? 2.0 : 1.0);
        const double2 a = c[(size_t)n * K + k], b = c[(size_t)np * K + k];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const double2 ga = G[e * NK + n * K + k], gb = G[e * NK + np * K + k];
          d[e] = d[e] - w * (ga.x * b.x + ga.y * b.y + a.x * gb.x + a.y * gb.y);
        }
      }
      for (int e = 0; e < 3; ++e) h.kept3[(size_t)e * nk + q] = d[e];
    }
    __syncthreads();
    for (int o = tid; o < ns; o += NT) {
      double d0 = 0.0, d1 = 0.0, d2 = 0.0;
      for (int t = P.pi_off[o]; t < P.pi_off[o + 1]; ++t) {
        const double e = P.pi_el64[t];
        const int q = P.pi_q[t];
        d0 = d0 + e * h.kept3[q];
        d1 = d1 + e * h.kept3[nk + q];
        d2 = d2 + e * h.kept3[2 * nk + q];
      }
      h.dp1[3 * o] = d0;
      h.dp1[3 * o + 1] = d1;
      h.dp1[3 * o + 2] = d2;
    }
    __syncthreads();
    // the site's dot products: t1 (3), then per v wp, u1 (3)
    for (int d = warp; d < 3 + 4 * n_vec; d += NW) {
      double r;
      if (d < 3) r = sv * warp_dot(soap_i, 1, h.dp1 + d, 3, ns);
      else {
        const int v = (d - 3) >> 2, e = (d - 3) & 3;
        const double *wv = vecs + ((size_t)site * n_vec + v) * ns;
        r = (e == 0) ? sv * warp_dot(wv, 1, soap_i, 1, ns) : warp_dot(wv, 1, h.dp1 + (e - 1), 3, ns);
      }
      if (lane == 0) sdot[d] = r;
    }
    // ---- B: a pass per vector of the Hessian, then one for the three columns of
    // dp1 together (their tables in ZG's place, their sums being the same)
    for (int v = 0; v <= nvh; ++v) {
      const bool full = v < nvh;
      const size_t off = (size_t)v * kSumsFull + (full ? 13 : 0);  // of the ZG sums
      __syncthreads();  // the vectors before are read
      for (int t = tid; t < (full ? nk : 3 * nk); t += NT) {
        const int w = t / nk, q = t - w * nk;
        double x = 0.0;
        for (int i = P.pj_off[q]; i < P.pj_off[q + 1]; ++i)
          x = x + P.pj_el64[i] * weight(vecs, soap_i, sv, h.dp1, n_vec, ns, site, v + w, P.pj_o[i]);
        h.vk[t] = x;
      }
      for (int s_lo = 0, s_hi; s_lo < nsp; s_lo = s_hi) {
        // as many species as the tables hold
        int n_rows = P.rad[s_lo].alpha;
        for (s_hi = s_lo + 1; !apart && s_hi < nsp && n_rows + P.rad[s_hi].alpha <= RT; ++s_hi) n_rows += P.rad[s_hi].alpha;
        const int nb = P.rad[s_lo].nbeg;
        __syncthreads();  // vk is complete, the tables before are read
        // S_v through the per-(l, n) lists of the kept components (2 v on the
        // diagonal, sqrt 2 v off it, np ascending)
        for (int it = tid; it < n_rows * K; it += NT) {
          const int n = it / K, k = it - n * K, l = klm[k] & 0xff;
          double2 z = make_double2(0.0, 0.0), b[3];
#pragma unroll
          for (int q = 0; q < 3; ++q) b[q] = z;
          const int li = l * N + nb + n, t1 = P.hl_off[li + 1];
          if (full) {
#pragma unroll 4
            for (int t = P.hl_off[li]; t < t1; ++t) {
              const int code = __ldg(P.hl_packed + t), np = code & 0xff;
              const double y = (code < 0 ? 2.0 : sqrt(2.0)) * h.vk[(code >> 8) & 0xffff];
              const double2 cc = c[np * K + k];
              const double2 *gg = G + np * K + k;
              z.x += y * cc.x;
              z.y += y * cc.y;
#pragma unroll
              for (int q = 0; q < 3; ++q) {
                const double2 gv = gg[q * NK];
                b[q].x += y * gv.x;
                b[q].y += y * gv.y;
              }
            }
            sZ[n * K + k] = z;
          } else {
#pragma unroll 4
            for (int t = P.hl_off[li]; t < t1; ++t) {
              const int code = __ldg(P.hl_packed + t), np = code & 0xff, q0 = (code >> 8) & 0xffff;
              const double f = code < 0 ? 2.0 : sqrt(2.0);
              const double2 cc = c[np * K + k];
#pragma unroll
              for (int q = 0; q < 3; ++q) {
                const double y = f * h.vk[q * nk + q0];
                b[q].x += y * cc.x;
                b[q].y += y * cc.y;
              }
            }
          }
#pragma unroll
          for (int q = 0; q < 3; ++q) sZG[(q * RT + n) * K + k] = b[q];
        }
        __syncthreads();
        for (int c0 = p0 + 1; c0 < p1; c0 += kHessChunk) {
          if (multi) build(s_lo, s_hi, c0, min(p1, c0 + kHessChunk));
          int n_two = 0;  // pairs of entries
          for (int s = s_lo; s < s_hi; ++s) n_two += (s_base[s + 1] - s_base[s] + 1) >> 1;
          // units: two pairs (one per half-warp), Z_v (all first) or ZG_v
          for (int u = warp; u < (full ? 2 : 1) * n_two; u += NW) {
            const bool zg = !full || u >= n_two;
            int e = u >= n_two ? u - n_two : u, s = s_lo;
            for (int m2; e >= (m2 = (s_base[s + 1] - s_base[s] + 1) >> 1); ++s) e -= m2;
            const int e0 = s_base[s], a = P.rad[s].alpha, row = P.rad[s].nbeg - nb;
            e = e0 + 2 * e + half;
            const bool pv = e < s_base[s + 1];
            const int code = list[pv ? e : e0], j = c0 + (code & 0x7fff);
            const double *g = geo + (size_t)j * Lg.size;
            // R_n, R'_n, R''_n side by side
            for (int t = hl; t < 3 * a; t += 16) {
              const int w = t / a, n = t - w * a;
              wrad[4 * n + w] = (w == 0 ? rad : (w == 1 ? rad_der : rad_der2))[(size_t)j * N + nb + row + n];
            }
            __syncwarp();
            double acc[kHessCols];
#pragma unroll
            for (int t = 0; t < kHessCols; ++t) acc[t] = 0.0;
            const double *gQ = g + Lg.Q, *gW = g + Lg.wp, *gF = g + Lg.F;
            for (int k = hl; k < K; k += 16) {
              const int lm = klm[k], l = lm & 0xff, m = lm >> 8;
              // Om = q0 w0, Om_t = q1 w0, Om_w = q0 w1, ...
              const double C = ((m > 0) ? 2.0 : 1.0) * sck[k];
              const double q0 = C * gQ[k], q1 = (m < l) ? C * gQ[k + 1] : 0.0;
              const double2 w0 = *(const double2 *)(gW + 2 * (m + 2)), v1 = *(const double2 *)(gW + 2 * (m + 1));
              const double f0 = gF[3 * l], f1 = gF[3 * l + 1];
              const dcx W0 = cx(w0.x, w0.y), W1 = cx((double)m * v1.x, (double)m * v1.y);
              const dcx Om = q0 * W0, Ot = q1 * W0, Ow = q0 * W1;
              if (zg) {
                double2 a0[3], a1[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) a0[q] = a1[q] = make_double2(0.0, 0.0);
                const double2 *z = sZG + row * K + k;
#pragma unroll 2
                for (int n = 0; n < a; ++n, z += K) {
                  const double2 r = *(const double2 *)(wrad + 4 * n);
#pragma unroll
                  for (int q = 0; q < 3; ++q) {
                    const double2 zz = z[q * RT * K];
                    a0[q].x += r.x * zz.x;
                    a0[q].y -= r.x * zz.y;
                    a1[q].x += r.y * zz.x;
                    a1[q].y -= r.y * zz.y;
                  }
                }
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                  const dcx z0 = cx(f0 * a0[q].x, f0 * a0[q].y);
                  const dcx z1 = cx(f0 * a1[q].x + f1 * a0[q].x, f0 * a1[q].y + f1 * a0[q].y);
                  acc[4 * q] += z1.re * Om.re - z1.im * Om.im;
                  acc[4 * q + 1] += z0.re * Ot.re - z0.im * Ot.im;
                  acc[4 * q + 2] += z0.re * Ow.re - z0.im * Ow.im;
                  acc[4 * q + 3] += z0.re * Ow.im + z0.im * Ow.re;
                }
                continue;
              }
              double2 a0 = make_double2(0.0, 0.0), a1 = a0, a2 = a0;
              const double2 *z = sZ + row * K + k;
#pragma unroll 4
              for (int n = 0; n < a; ++n, z += K) {
                const double2 zz = *z, r = *(const double2 *)(wrad + 4 * n);
                const double r2 = wrad[4 * n + 2];
                a0.x += r.x * zz.x;
                a0.y -= r.x * zz.y;
                a1.x += r.y * zz.x;
                a1.y -= r.y * zz.y;
                a2.x += r2 * zz.x;
                a2.y -= r2 * zz.y;
              }
              const dcx z0 = cx(f0 * a0.x, f0 * a0.y), z1 = cx(f0 * a1.x + f1 * a0.x, f0 * a1.y + f1 * a0.y);
              const double q2 = (m + 1 < l) ? C * gQ[k + 2] : 0.0, f2 = gF[3 * l + 2];
              const double2 v2 = *(const double2 *)(gW + 2 * m);
              const double mm = (double)(m * (m - 1)), invr = g[Lg.invr];
              const dcx W2 = cx(mm * v2.x, mm * v2.y);
              const dcx y = cx(f0 * a2.x + 2.0 * f1 * a1.x + f2 * a0.x - invr * z1.re,
                               f0 * a2.y + 2.0 * f1 * a1.y + f2 * a0.y - invr * z1.im);
              acc[0] += y.re * Om.re - y.im * Om.im;
              acc[1] += z1.re * Om.re - z1.im * Om.im;
              acc[2] += z1.re * Ot.re - z1.im * Ot.im;
              acc[3] += z1.re * Ow.re - z1.im * Ow.im;
              acc[4] += z1.re * Ow.im + z1.im * Ow.re;
              acc[5] += z0.re * Ot.re - z0.im * Ot.im;
              acc[6] += z0.re * Ow.re - z0.im * Ow.im;
              acc[7] += z0.re * Ow.im + z0.im * Ow.re;
              const dcx Ott = q2 * W0, Otw = q1 * W1, Oww = q0 * W2;
              acc[8] += z0.re * Ott.re - z0.im * Ott.im;
              acc[9] += z0.re * Otw.re - z0.im * Otw.im;
              acc[10] += z0.re * Otw.im + z0.im * Otw.re;
              acc[11] += z0.re * Oww.re - z0.im * Oww.im;
              acc[12] += z0.re * Oww.im + z0.im * Oww.re;
            }
            // the lanes' sums: lane t of a half adds column t of its half's 16 rows
            const int cols = zg ? 12 : 13;
#pragma unroll
            for (int t = 0; t < kHessCols; ++t)
              if (t < cols) red[lane * kHessCols + t] = acc[t];
            __syncwarp();
            if (pv && hl < cols) {
              double x = 0.0;
#pragma unroll
              for (int r = 0; r < 16; ++r) x += red[(16 * half + r) * kHessCols + hl];
              double *o = sums + (size_t)j * sp_sums + off - (zg ? 0 : 13) + hl;
              *o = (code & 0x8000) ? x : *o + x;
            }
            __syncwarp();
          }
        }
      }
    }
    __syncthreads();
    // ---- C: the normalisation (:1414-1484): t2 = p . dp_j, c12(b, a) = dp1(:, a) .
    // dp_j(:, b), u2 = w . dp_j.  Pairs the Hessian skips keep the zero blocks the
    // launcher cleared.
    for (int it = tid; it < (p1 - p0 - 1) * 9 * n_vec; it += NT) {
      const int jj = it / (9 * n_vec), t = it - jj * 9 * n_vec, v = t / 9, e = t - v * 9, bb = e / 3, aa = e - bb * 3;
      const int j = p0 + 1 + jj;
      if (!hess_species(P, B, good, j)) continue;
      const double *g = geo + (size_t)j * Lg.size, *S = sums + (size_t)j * sp_sums;
      const double *Sv = S + v * kSumsFull, *Sp = S + n_vec * kSumsFull, *Sc = S + nvh * kSumsFull + aa * kSumsLight;
      const double *t1 = sdot, *dv = sdot + 3 + 4 * v;
      const double wp = dv[0], *u1 = dv + 1;
      const double t2b = first_der(Sp[1], Sp[5], Sp + 6, g, Lg, bb), u2b = first_der(Sv[1], Sv[5], Sv + 6, g, Lg, bb);
      const double c12 = first_der(Sc[0], Sc[1], Sc + 2, g, Lg, bb);
      const double hvv = second_der(Sv, g, Lg, aa, bb), hvp = second_der(Sp, g, Lg, aa, bb);
      hess[((size_t)j * n_vec + v) * 9 + e] = hvv * invs - (u1[aa] * t2b + u2b * t1[aa]) * invs3 -
                                              wp * (c12 + hvp) * invs3 + 3.0 * wp * t1[aa] * t2b * invs5;
    }
    __syncthreads();
    // the self pair: minus the sum of the others (:1488-1495)
    if (p1 > p0)
      for (int t = warp; t < 9 * n_vec; t += NW) {
        double x = 0.0;
        for (int j = p0 + 1 + lane; j < p1; j += 32) x += hess[(size_t)j * n_vec * 9 + t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) hess[(size_t)p0 * n_vec * 9 + t] = -x;
      }
  }
}

}  // namespace

// Doubles per CTA, a multiple of 32 so that every CTA's region starts on a
// 256-byte boundary.
size_t hess_scratch_doubles(const DevParams &P) {
  const size_t n = 6 * (size_t)P.n_max * P.k_max + 3 * (size_t)P.n_soap + 6 * (size_t)P.n_kept;
  return (n + 31) / 32 * 32;
}

int hess_threads(const DevParams &P, int n_vec, int n_sites);

size_t hess_sums_doubles(int n_vec) { return (size_t)kSumsFull * (n_vec + 1) + 3 * kSumsLight; }

// At most 16 vectors in a launch, and no more than keep the pairs' sums within 4 GB
// (16 at 1.2 M pairs, 7 at 2.4 M), in chunks as even as they come.  A chunk forms a site's
// G and dp1 again: 17 vectors at 100 sites of one species take 1.2 times 16's time.
int hess_vecs(int n_vec, long long n_pairs) {
  constexpr size_t kBytes = (size_t)4 << 30;
  int most = 16;
  while (most > 1 && sizeof(double) * hess_sums_doubles(most) * (size_t)n_pairs > kBytes) --most;
  const int chunks = (n_vec + most - 1) / most;
  return (n_vec + chunks - 1) / chunks;
}

size_t hess_geo_doubles(const DevParams &P) { return (size_t)GeoLayout(P.l_max).size; }

size_t hess_smem_bytes(const DevParams &P, int n_vec, int n_sites) {
  return sizeof(double) * (size_t)hess_smem(P, n_vec, hess_threads(P, n_vec, n_sites)).total;
}

// One CTA of 512 threads an SM or two of 256.  512 where shared memory holds one CTA
// of 256 only; else up to one site per SM, and up to three where a site is some work
// (beyond, two CTAs of 256 have less of a last wave).  Calls of three vectors with 512 and
// 256 threads, us, at 148, 149, 296, 297, 444, 445 and 600 sites: one species, l_max 8 225
// and 281, 317 and 315, 353 and 348, 419 and 456, 485 and 561, 527 and 561, 697 and 715;
// two species of alpha 4, l_max 4 145 and 162, 193 and 175, 211 and 189, 250 and 239, 277
// and 290, 305 and 291, 384 and 349.  One species of alpha 10, l_max 12 (one CTA of
// either) 403 and 492 at 148, 666 and 851 at 296, 1376 and 1769 at 600.  150 sites of one
// species, l_max 6, with five vectors 300 and 313.
int hess_threads(const DevParams &P, int n_vec, int n_sites) {
  if (sizeof(double) * (size_t)hess_smem(P, n_vec, 256).total > kHessSmemPair) return 512;
  const int sms = sm_count(), most = P.n_max * P.k_max > 128 ? 3 * sms : sms;
  return n_sites <= most ? 512 : 256;
}

template <int NT>
static int hess_grid_of(const DevParams &P, int n_vec) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t sm = sizeof(double) * (size_t)hess_smem(P, n_vec, NT).total;
  auto kern = k64_hess<NT>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) return sms;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, sm);
  return sms * (per_sm > 0 ? per_sm : 1);
}
int hess_grid(const DevParams &P, int n_vec, int n_sites) {
  return hess_threads(P, n_vec, n_sites) == 512 ? hess_grid_of<512>(P, n_vec) : hess_grid_of<256>(P, n_vec);
}

cudaError_t launch_hessian(const DevParams &P, const DevBatch &B, cudaStream_t s, const Fp64Work &w,
                           double *rad_der2, double *geo, int *good, const double *soap, int n_vec,
                           const double *vecs, double *hess, double *sums, double *scratch, int grid, int *ticket,
                           int *launches, bool pair_state) {
  CU_RET(cudaMemsetAsync(hess, 0, sizeof(double) * 9 * (size_t)n_vec * B.n_pairs, s));
  CU_RET(cudaMemsetAsync(ticket, 0, sizeof(int), s));
  if (B.n_pairs > 0 && pair_state) {
    const int blocks = (B.n_pairs + 127) / 128;
    int amax = 0;
    for (int sp = 0; sp < P.n_species; ++sp) amax = amax > P.rad[sp].alpha ? amax : P.rad[sp].alpha;
    if (amax <= 8) k64_radial_d2<8><<<blocks, 128, 0, s>>>(P, B, rad_der2);
    else k64_radial_d2<16><<<blocks, 128, 0, s>>>(P, B, rad_der2);
    const size_t smg = 32 * sizeof(double) * (hess_geo_doubles(P) | 1);
    CU_RET(cudaFuncSetAttribute(k64_hgeo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smg));
    k64_hgeo<<<(B.n_pairs + 31) / 32, 32, smg, s>>>(P, B, geo, good);
    if (launches) *launches += 2;
  }
  if (B.n_sites > 0) {
    const size_t sm = hess_smem_bytes(P, n_vec, B.n_sites);
    const int threads = hess_threads(P, n_vec, B.n_sites);
    auto kern = threads == 512 ? k64_hess<512> : k64_hess<256>;
    CU_RET(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    const int g = grid < B.n_sites ? grid : B.n_sites;
    kern<<<g, threads, sm, s>>>(P, B, w.rad, w.rad_der, rad_der2, geo, good, (const double2 *)w.cnk, w.norm, soap,
                                n_vec, vecs, hess, sums, scratch, hess_scratch_doubles(P), ticket);
    if (launches) *launches += 1;
  }
  return cudaGetLastError();
}

}  // namespace soapb
