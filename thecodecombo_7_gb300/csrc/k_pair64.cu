// k_pair64.cu -- the FP64 drop-in's non-bonded pair loop of cnonbondnl
// (cnonbond_nblist.c:134-523, SPME + STYPE branch).
//
// Compiled with -fmad=false: where the reference's roundings matter they are
// kept; the pair loop fuses multiplies and adds by explicit fma().
//
// The FP64 pipe bounds the pair loop (two FP64 instructions per SM and clock,
// 1/64 of the FP32 rate), so it is written for the fewest FP64 instructions
// per pair within the cutoff:
//   - entries beyond the cutoff (42 % of a 12 A list at rc 10 A) are dropped by
//     an FP32 distance of 32-bit fixed-point coordinates, whose wrapped integer
//     difference is the minimum image; the margin covers its rounding, and the
//     FP64 distance decides what is left;
//   - the survivors are packed: a warp queues them in shared memory and
//     evaluates full batches of 32, pairs with an LJ term apart from the rest;
//   - erfc(kappa r)/r and the force factor are piecewise polynomials in r^2
//     (degree 6, 128 intervals per octave, below 1e-15 of the function:
//     k_pair_table), 12 fused multiply-adds in place of two exponentials, three
//     divisions, a root and the erfc fit;
//   - signs and comparisons on the bits of the doubles, in integer registers.
// What is left is 28 FP64 instructions per pair, against about 200: at 96,000
// sites 11.6 ms -> 1.32 ms a call, 94 % of the pipe's rate (1.71 ms with the
// image chosen by comparing FP64 separations, LJ by FP64 divisions and static
// strides); at 4,095 sites 577 -> 79 us, where the pipe's share is 52 us and
// the rest the ends of the uneven rows.
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "fe_device.cuh"

namespace fe {

struct PairParams {
  double3 L, H;
  double rc, rc2, kappa, kpi, epsRF, erfc_rc;
  // optional CHARMM switch (ron2 = 0: off): 1 / (rc^2 - ron^2)^3, rc^2 - 3 ron^2
  double ron2, inv_sw_den, sw_c0;
  int lj_form;          // 0 CHARMM (the reference's default build); 2 its BGO build
  int n, nt, max_nb;
  float3 sc;            // L / 2^32 per axis
  float rf2;            // rc2 with the FP32 test's margin
  int tab0;             // first interval of the table (r^2's high word >> kTabShift)
  int parts;            // warps that share a row
  int wide;             // the cutoff reaches half the box: images by the reference's rule
  int nexcl;            // excluded and 1-4 pairs, listed or not
  double rec_ew;        // erfc(kappa rc) / rc
  double qfe;           // QFACTOR / epsRF
};

// The table of the real-space functions over r^2: kTabOct octaves below rc^2
// (down to rc / 11), 2^kTabBits intervals per octave; an interval holds the
// coefficients of (F, E) in r^2 - centre, lowest first.  At relative
// half-width 2^-8 the interpolation error of exp(-kappa^2 r^2) at kappa r =
// 3.2 is (0.04)^7 / (7! 2^6) = 5e-16, falling with the seventh power of
// (kappa r)^2.  The whole table is 100 KB: one block per SM keeps it in
// shared memory.
constexpr int kTabBits = 7, kTabOct = 7, kTabDeg = 6, kTabShift = 20 - kTabBits;
constexpr int kTabN = (kTabOct << kTabBits) + 1, kTabRow = 2 * (kTabDeg + 1);
constexpr int kP64Warps = 16;
constexpr int kP64Units = 5;   // units per warp a small box's rows are split for
constexpr int kP64Queue = 64;  // entries of a queue: fewer than 32 kept + 32 new

// F = [erfc(kr) + 2 k/sqrt(pi) r exp(-(kr)^2)] / r^3 and E = erfc(kr) / r in
// the reference's terms (cnonbond_nblist.c:330-372)
__device__ __forceinline__ void pair_direct(double kappa, double kpi, double r2, double &F,
                                            double &E) {
  double dr = sqrt(r2);
  double dri = 1.0 / dr;
  double kr = kappa * dr;
  double erfckr = ref_erfc(kr);
  double g = 2.0 * kpi * dr * exp(-kr * kr);
  E = erfckr * dri;
  F = (dri / r2) * (erfckr + g);
}

// the double whose high word is the interval's first, plus half an interval
__device__ __forceinline__ double tab_centre(int hi) {
  return __hiloint2double((hi & ~((1 << kTabShift) - 1)) | (1 << (kTabShift - 1)), 0);
}

// F and E for the table, with the exponential's argument carried to twice the
// precision: exp(-(kappa r)^2) from the product's rounding error too, apart
// from the exponential of the fit's polynomial
__device__ __forceinline__ void pair_direct_fine(double kappa, double kpi, double r2, double &F,
                                                 double &E) {
  const double r = sqrt(r2), ri = 1.0 / r, z = kappa * r, t = 1.0 / (1.0 + 0.5 * z);
  const double k2 = kappa * kappa, k2l = fma(kappa, kappa, -k2);
  const double z2 = k2 * r2, z2l = fma(k2, r2, -z2) + k2l * r2;
  const double ex = exp(-z2) * (1.0 - z2l);
  double p = 0.17087277;
  p = fma(t, p, -0.82215223);
  p = fma(t, p, 1.48851587);
  p = fma(t, p, -1.13520398);
  p = fma(t, p, 0.27886807);
  p = fma(t, p, -0.18628806);
  p = fma(t, p, 0.09678418);
  p = fma(t, p, 0.37409196);
  p = fma(t, p, 1.00002368);
  p = fma(t, p, -1.26551223);
  const double er = t * exp(p) * ex;
  E = er * ri;
  F = (ri / r2) * fma(2.0 * kpi * r, ex, er);
}

// One thread per interval: Chebyshev interpolation at kTabDeg + 1 nodes
// (a_k = 2/m sum_j f(x_j) T_k(x_j), Clenshaw 1955), turned into powers of
// the offset from the centre; the centre is a node, whose value is the
// constant term.
__global__ void k_pair_table(double kappa, double kpi, int tab0, double *__restrict__ tab) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= kTabN) return;
  constexpr int m = kTabDeg + 1;
  static_assert(m % 2 == 1, "the centre of the interval is a node");
  const int hi = (tab0 + t) << kTabShift;
  const double c = tab_centre(hi), lo = __hiloint2double(hi, 0), h = c - lo;
  double f[2][m], a[2][m];
  for (int j = 0; j < m; j++) {
    double x = 2 * j + 1 == m ? 0.0 : cospi((j + 0.5) / m);
    pair_direct_fine(kappa, kpi, c + h * x, f[0][j], f[1][j]);
  }
  for (int w = 0; w < 2; w++)
    for (int k = 0; k < m; k++) {
      double s = 0.0;
      for (int j = 0; j < m; j++) s += f[w][j] * cospi(k * (j + 0.5) / m);
      a[w][k] = s * (k == 0 ? 1.0 : 2.0) / m;
    }
  // T_k in powers of x: T_0 = 1, T_1 = x, T_k = 2 x T_k-1 - T_k-2
  double T[m][m];
  for (int k = 0; k < m; k++)
    for (int p = 0; p < m; p++) {
      double v = k == p && k < 2 ? 1.0 : 0.0;
      if (k >= 2) v = (p > 0 ? 2.0 * T[k - 1][p - 1] : 0.0) - T[k - 2][p];
      T[k][p] = v;
    }
  for (int w = 0; w < 2; w++) {
    double ih = 1.0;
    for (int p = 0; p < m; p++) {
      double s = 0.0;
      for (int k = m - 1; k >= p; k--) s += a[w][k] * T[k][p];
      if (p == 0) s = f[w][m / 2];
      tab[(size_t)t * kTabRow + 2 * p + w] = s * ih;
      ih /= h;
    }
  }
}

// the pair loop's view of the sites (pair_fix_coord) and, optionally, the forces
// cleared
__global__ void k_pair_fix(int n, double3 invL, const double4 *__restrict__ pos,
                           const int *__restrict__ type, int4 *__restrict__ pfx,
                           double *__restrict__ ff_zero) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  pfx[i] = pair_fix_coord(pos[i], invL, type[i]);
  if (ff_zero) {
    ff_zero[3 * i] = 0.0;
    ff_zero[3 * i + 1] = 0.0;
    ff_zero[3 * i + 2] = 0.0;
  }
}

struct Pair64Acc {
  double fx, fy, fz, e_lj, e_ljs, e_real, qsum, e_intra;
};

// d > h: subtract l, d < -h: add l (the reference's image rule), compared in
// integer registers
__device__ __forceinline__ double img_shift(double d, double h, double l) {
  const bool far = (__double_as_longlong(d) & 0x7fffffffffffffffll) > __double_as_longlong(h);
  return far ? d - copysign(l, d) : d;
}
__device__ __forceinline__ double pair_sep(const PairParams &P, double4 pa, double4 pb, double &dx,
                                           double &dy, double &dz) {
  dx = img_shift(pa.x - pb.x, P.H.x, P.L.x);
  dy = img_shift(pa.y - pb.y, P.H.y, P.L.y);
  dz = img_shift(pa.z - pb.z, P.H.z, P.L.z);
  return fma(dz, dz, fma(dy, dy, dx * dx));
}

// Which image of site a pairs with b along an axis, from the fixed-point
// coordinates: 0 a itself, 1 a - L, 2 a + L
__device__ __forceinline__ int img_class(unsigned ua, unsigned ub) {
  const bool neg = (int)(ua - ub) < 0;
  return ua > ub ? (neg ? 1 : 0) : (neg || ua == ub ? 0 : 2);
}
// the row's site and its two images
struct RowSite {
  double4 p;
  double3 lo, hi;  // p - L, p + L
};
__device__ __forceinline__ double img_pick(int c, double x, double lo, double hi) {
  return c == 0 ? x : c == 1 ? lo : hi;
}

// F and E of r^2 <= rc^2 from the table; false closer than its first interval, or
// not a number (pair_direct has those)
__device__ __forceinline__ bool pair_table(const PairParams &P, const double *__restrict__ tab,
                                           double r2, double &F, double &E) {
  const int hi = __double2hiint(r2);
  const int t = (hi >> kTabShift) - P.tab0;
  if ((unsigned)t >= (unsigned)kTabN) return false;
  const double d = r2 - tab_centre(hi);
  const double2 *c = reinterpret_cast<const double2 *>(tab + t * kTabRow);
  // E, which falls as 1/r where F falls as 1/r^3, has reached FP64's rounding
  // one degree earlier: its last coefficient is left out
  double2 v = c[kTabDeg - 1];
  F = fma(c[kTabDeg].x, d, v.x);
  E = v.y;
#pragma unroll
  for (int k = kTabDeg - 2; k >= 0; k--) {
    v = c[k];
    F = fma(F, d, v.x);
    E = fma(E, d, v.y);
  }
  return true;
}

// 1 / x, x normal and positive: the hardware's 20-bit reciprocal (PTX
// rcp.approx.ftz.f64) and two Newton-Raphson steps, each doubling the digits
__device__ __forceinline__ double recip_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// LJ force factor and energies of one pair (cnonbond_nblist.c:277-328);
// lj = (eps, sigma^2, eps (sr12s - 2 sr6s) at rc) of the type pair
__device__ __forceinline__ double pair_lj(const PairParams &P, const double *__restrict__ lj,
                                          double dr2, Pair64Acc &A) {
  const double eps = lj[0], sig2 = lj[1];
  const double ri2 = recip_nr(dr2);
  const double sr2 = sig2 * ri2;
  const double sr6 = sr2 * sr2 * sr2;
  if (P.lj_form == 2) {
    // the BGO build (cnonbond_nblist.c:294-307): eps [13 (R/r)^12 -
    // 18 (R/r)^10 + 4 (R/r)^6], shifted sum at rc as the default form
    double sr12 = sr6 * sr6;
    double sr10 = sr6 * sr2 * sr2;
    double sr2s = sig2 / P.rc2;
    double sr6s = sr2s * sr2s * sr2s;
    double sr12s = sr6s * sr6s;
    double sr10s = sr6s * sr2s * sr2s;
    A.e_lj += eps * (13.0 * sr12 - 18.0 * sr10 + 4.0 * sr6);
    A.e_ljs += eps * (13.0 * sr12s - 18.0 * sr10s + 4.0 * sr6s);
    return eps * ri2 * (156.0 * sr12 - 180.0 * sr10 + 24.0 * sr6);
  }
  const double d = fma(sr6, sr6, -sr6);  // sr12 - sr6
  double flj = 12.0 * eps * ri2 * d;
  double elj = eps * (d - sr6);
  if (P.ron2 > 0.0) {
    if (__double_as_longlong(dr2) > __double_as_longlong(P.ron2)) {
      const double c = P.rc2 - dr2, ci = c * P.inv_sw_den;
      const double sw = c * ci * fma(2.0, dr2, P.sw_c0);
      const double dsw = 12.0 * ci * (dr2 - P.ron2);
      flj = fma(flj, sw, elj * dsw);
      elj = elj * sw;
    }
  } else {
    A.e_ljs += lj[2];
  }
  A.e_lj += elj;
  return flj;
}

// One pair of a batch: site a (position pa, charge factor qfa = qa QFACTOR /
// epsRF) with site b; img: the image of a on each axis (img_class, two bits
// each).  Adds to the lane's sums and to b's force.
template <bool WITH_LJ>
__device__ __forceinline__ void pair_eval(const PairParams &P, const double *__restrict__ tab,
                                          const RowSite &S, double qfa, bool live, int b, int img,
                                          bool lj, int ta, const double4 *__restrict__ pos,
                                          const int *__restrict__ type,
                                          const double *__restrict__ lj_tab,
                                          double *__restrict__ ff, Pair64Acc &A) {
  if (!live) return;
  const double4 pb = pos[b];
  double dx = img_pick(img & 3, S.p.x, S.lo.x, S.hi.x) - pb.x;
  double dy = img_pick((img >> 2) & 3, S.p.y, S.lo.y, S.hi.y) - pb.y;
  double dz = img_pick(img >> 4, S.p.z, S.lo.z, S.hi.z) - pb.z;
  double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  if (P.wide || __double_as_longlong(r2) > __double_as_longlong(P.rc2)) {
    // within the FP32 test's margin of the cutoff, or a site on a face whose
    // fixed-point coordinate rounded to the other one, or a cutoff that takes both
    // images of sites half a box apart: the reference's rule
    // (bits of a NaN may be above those of rc2: it goes on, into the energies)
    r2 = pair_sep(P, S.p, pb, dx, dy, dz);
    if (r2 > P.rc2) return;
  }
  const double qq = qfa * pb.w;
  double F, E;
  if (!pair_table(P, tab, r2, F, E)) {
    // without charge there is no real-space term, as the reference tests: sites
    // that coincide would give 0 times infinity
    if (qq != 0.0) {
      pair_direct(P.kappa, P.kpi, r2, F, E);
    } else {
      if (!(WITH_LJ && lj)) return;
      F = E = 0.0;
    }
  }
  A.e_real = fma(qq, E, A.e_real);
  A.qsum += qq;
  double force = qq * F;
  if (WITH_LJ && lj) force += pair_lj(P, lj_tab + 3 * (ta * P.nt + type[b]), r2, A);
  A.fx = fma(force, dx, A.fx);
  A.fy = fma(force, dy, A.fy);
  A.fz = fma(force, dz, A.fz);
  atomicAdd(&ff[3 * b], -(force * dx));
  atomicAdd(&ff[3 * b + 1], -(force * dy));
  atomicAdd(&ff[3 * b + 2], -(force * dz));
}

// sum over the warp of three values: lanes 0, 8 and 16 get x, y and z (six
// additions instead of fifteen)
__device__ __forceinline__ double warp_sum3(double x, double y, double z, int lane) {
  const unsigned full = 0xffffffffu;
  const bool h = lane & 16, g = lane & 8;
  double a = (h ? z : x) + __shfl_xor_sync(full, h ? x : z, 16);
  double b = (h ? 0.0 : y) + __shfl_xor_sync(full, h ? y : 0.0, 16);
  double c = (g ? b : a) + __shfl_xor_sync(full, g ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(full, c, o);
  return c;
}

// An excluded or 1-4 pair of the list (xint flags, cnonbond_nblist.c:245-263,
// 416-437): no LJ and no real-space term but the intra correction; a 1-4 pair
// keeps LJ, E14FAC of the real-space term and the rest of the correction.
__device__ __forceinline__ void pair_excluded(const PairParams &P,
                                              const double *__restrict__ tab, int a, int e,
                                              const double4 *__restrict__ pos,
                                              const int *__restrict__ type,
                                              const double *__restrict__ lj_tab,
                                              double *__restrict__ ff, Pair64Acc &A) {
  const int b = e >> 3, xflag = e & 7;
  const double4 pa = pos[a], pb = pos[b];
  double dx, dy, dz;
  const double r2 = pair_sep(P, pa, pb, dx, dy, dz);
  if (r2 > P.rc2) return;
  double F, E;
  if (!pair_table(P, tab, r2, F, E)) pair_direct(P.kappa, P.kpi, r2, F, E);
  const double dri = rsqrt(r2);
  double qqab = qfactor_mul(pa.w * pb.w), force = 0.0;
  if (xflag == 4) {
    const double qq = qqab * kE14FAC / P.epsRF;
    const int k = type[a] * P.nt + type[b];
    if (lj_tab[3 * k] != 0.0) force += pair_lj(P, lj_tab + 3 * k, r2, A);
    if (qq != 0.0) {
      A.e_real += qq * E;
      A.qsum += qq;
      force += qq * F;
    }
    qqab *= (1.0 - kE14FAC);
  }
  A.e_intra += qqab * (dri - E);
  force -= qqab * (dri * (dri * dri) - F);
  const double fx = force * dx, fy = force * dy, fz = force * dz;
  atomicAdd(&ff[3 * a], fx);
  atomicAdd(&ff[3 * a + 1], fy);
  atomicAdd(&ff[3 * a + 2], fz);
  atomicAdd(&ff[3 * b], -fx);
  atomicAdd(&ff[3 * b + 1], -fy);
  atomicAdd(&ff[3 * b + 2], -fz);
}

// One warp per row a of the half list (P.parts warps share a row of a small
// box), then one warp per 32 excluded pairs.  At most one block per SM.  Warp w
// of the grid's W takes unit w of every even W units and W - 1 - w of every odd
// one: rows grow shorter (entries have b > a), so a pair of turns costs every warp
// the same, and neighbours in a turn are on different SMs, whose FP64 pipes then
// finish together.  The units of a warp and with them the order of its energy
// sums are fixed: energies repeat bit for bit.  At 96,000 sites, ten steps take
// 18.23 ms, with units taken from a device counter, whose sums do not repeat,
// 18.14; at 4,095 sites, twenty steps, 3.07 and 3.09 (strides of W, whose every
// turn favours the same warps, left 40 % between the first and the last block).
__global__ void __launch_bounds__(kP64Warps * 32)
k_pair64(PairParams P, const double *__restrict__ gtab, const double4 *__restrict__ pos,
         const int4 *__restrict__ pfx, const int *__restrict__ type,
         const double *__restrict__ lj_tab,
         const int *__restrict__ count, const int *__restrict__ ent,
         const unsigned char *__restrict__ lj_on, const int2 *__restrict__ xl,
         double *__restrict__ ff, double *__restrict__ partials) {
  extern __shared__ double2 s_tab[];
  // a pair waits as b and, apart, its image classes: b takes up to 28 bits (the
  // list holds 8 b), so the two do not share a word
  __shared__ int s_q[kP64Warps][2][kP64Queue];
  __shared__ unsigned char s_img[kP64Warps][2][kP64Queue];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const double2 *g2 = reinterpret_cast<const double2 *>(gtab);
  for (int i = threadIdx.x; i < kTabN * kTabRow / 2; i += blockDim.x) s_tab[i] = g2[i];
  const double *tab = reinterpret_cast<const double *>(s_tab);
  int *qn = s_q[w][0], *ql = s_q[w][1];
  unsigned char *in = s_img[w][0], *il = s_img[w][1];
  __syncthreads();
  Pair64Acc A;
  A.e_lj = A.e_ljs = A.e_real = A.qsum = A.e_intra = 0.0;
  const unsigned full = 0xffffffffu, lt = (1u << lane) - 1u;
  const int nrow = (P.n - 1) * P.parts, nx = P.nexcl;
  const int nunit = nrow + (nx + 31) / 32, nwarp = gridDim.x * kP64Warps;
  const int rank = w * gridDim.x + blockIdx.x;
  for (int k = 0; k * nwarp < nunit; k++) {
    const int cur = k * nwarp + (k & 1 ? nwarp - 1 - rank : rank);
    if (cur >= nunit) break;
    if (cur >= nrow) {
      const int i = (cur - nrow) * 32 + lane;
      if (i < nx) {
        const int2 x = xl[i];
        if (x.y & 7) pair_excluded(P, tab, x.x, x.y, pos, type, lj_tab, ff, A);
      }
      continue;
    }
    const int a = cur / P.parts, part = cur - a * P.parts;
    RowSite S;
    S.p = pos[a];
    S.lo = make_double3(S.p.x - P.L.x, S.p.y - P.L.y, S.p.z - P.L.z);
    S.hi = make_double3(S.p.x + P.L.x, S.p.y + P.L.y, S.p.z + P.L.z);
    const int4 fa = pfx[a];
    const int ta = fa.w & INT_MAX, cnt = count[a];
    const double qfa = P.qfe * S.p.w;
    const int step = ((cnt + P.parts - 1) / P.parts + 31) & ~31;
    const int lo = min(part * step, cnt), hi = min(lo + step, cnt);
    const int *row = ent + (size_t)a * P.max_nb;
    A.fx = A.fy = A.fz = 0.0;
    int nn = 0, nl = 0;
    // the entry two chunks ahead and the coordinates one ahead are in flight
    int e1 = lo + lane < hi ? row[lo + lane] : a * 8;
    int e2 = lo + 32 + lane < hi ? row[lo + 32 + lane] : a * 8;
    int4 f1 = pfx[e1 >> 3];
    for (int base = lo; base < hi; base += 32) {
      const int i = base + lane;
      bool ok = i < hi;
      const int e = e1;
      const int4 fb = f1;
      e1 = e2;
      f1 = pfx[e1 >> 3];
      e2 = i + 64 < hi ? row[i + 64] : a * 8;
      const float dx = __int2float_rn((int)((unsigned)fa.x - (unsigned)fb.x)) * P.sc.x;
      const float dy = __int2float_rn((int)((unsigned)fa.y - (unsigned)fb.y)) * P.sc.y;
      const float dz = __int2float_rn((int)((unsigned)fa.z - (unsigned)fb.z)) * P.sc.z;
      ok = ok && (e & 7) == 0 && (dx * dx + dy * dy + dz * dz <= P.rf2 || (fa.w | fb.w) < 0);
      bool lj = false;
      if (ok) lj = lj_on[ta * P.nt + (fb.w & INT_MAX)] != 0;
      const unsigned ml = __ballot_sync(full, ok && lj), mn = __ballot_sync(full, ok && !lj);
      if (ok) {
        const int img = img_class((unsigned)fa.x, (unsigned)fb.x) |
                        img_class((unsigned)fa.y, (unsigned)fb.y) << 2 |
                        img_class((unsigned)fa.z, (unsigned)fb.z) << 4;
        const int at = lj ? nl + __popc(ml & lt) : nn + __popc(mn & lt);
        (lj ? ql : qn)[at] = e >> 3;
        (lj ? il : in)[at] = (unsigned char)img;
      }
      nl += __popc(ml);
      nn += __popc(mn);
      __syncwarp();
      if (nn >= 32) {
        nn -= 32;
        pair_eval<false>(P, tab, S, qfa, true, qn[nn + lane], in[nn + lane], false, ta, pos, type,
                         lj_tab, ff, A);
        __syncwarp();
      }
      if (nl >= 32) {
        nl -= 32;
        pair_eval<true>(P, tab, S, qfa, true, ql[nl + lane], il[nl + lane], true, ta, pos, type,
                        lj_tab, ff, A);
        __syncwarp();
      }
    }
    // what is left of both queues together
    if (nl == 0) {
      if (nn > 0)
        pair_eval<false>(P, tab, S, qfa, lane < nn, lane < nn ? qn[lane] : 0,
                         lane < nn ? in[lane] : 0, false, ta, pos, type, lj_tab, ff, A);
    } else {
      for (int o = lane; o - lane < nl + nn; o += 32) {
        const bool lj = o < nl;
        const bool live = o < nl + nn;
        const int q = lj ? ql[o] : live ? qn[o - nl] : 0;
        const int img = lj ? il[o] : live ? in[o - nl] : 0;
        pair_eval<true>(P, tab, S, qfa, live, q, img, lj, ta, pos, type, lj_tab, ff, A);
      }
    }
    __syncwarp();
    const double f = warp_sum3(A.fx, A.fy, A.fz, lane);
    if ((lane & 7) == 0 && lane < 24) atomicAdd(&ff[3 * a + (lane >> 3)], f);
  }
  double v[5] = {A.e_lj, A.e_ljs, A.e_real, A.qsum * P.rec_ew, A.e_intra};
  block_partials<5>(v, partials);
}

// Counts of the half list (instrumentation): entries, pairs within rc that
// the pair loop evaluates (not excluded), and those with an LJ term -- the
// units of the pair loop's algorithmic FLOP count.
__global__ void k_pair_counts(PairParams P, const double4 *__restrict__ pos,
                              const int *__restrict__ type, const double *__restrict__ lj_eps,
                              const double *__restrict__ lj_sig, const int *__restrict__ count,
                              const int *__restrict__ ent, unsigned long long *__restrict__ out) {
  unsigned long long c[4] = {0, 0, 0, 0};
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < P.n - 1; a += gridDim.x * blockDim.x) {
    double4 pa = pos[a];
    const int *row = ent + (size_t)a * P.max_nb;
    int cnt = count[a];
    c[0] += cnt;
    for (int bb = 0; bb < cnt; bb++) {
      int e = row[bb];
      int b = e >> 3, xflag = e & 7;
      double4 pb = pos[b];
      double dx = pa.x - pb.x, dy = pa.y - pb.y, dz = pa.z - pb.z;
      dx -= P.L.x * rint(dx / P.L.x);
      dy -= P.L.y * rint(dy / P.L.y);
      dz -= P.L.z * rint(dz / P.L.z);
      if (dx * dx + dy * dy + dz * dz > P.rc2) continue;
      if (xflag != 0 && xflag != 4) {
        c[3]++;
        continue;
      }
      c[1]++;
      int k = type[a] * P.nt + type[b];
      if (lj_eps[k] * lj_sig[k] != 0.0) c[2]++;
    }
  }
  for (int t = 0; t < 4; t++) atomicAdd(&out[t], c[t]);
}

int pair_counts64(Box *b, long long *out4) {
  PairParams P;
  P.L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  P.rc2 = b->p.rc * b->p.rc;
  P.n = b->n;
  P.nt = b->nt;
  P.max_nb = b->max_nb;
  unsigned long long *d = nullptr;
  FE_CUDA(cudaMalloc(&d, 4 * sizeof(unsigned long long)));
  cudaMemsetAsync(d, 0, 4 * sizeof(unsigned long long), b->stream);
  int blocks = (b->n + 255) / 256;
  k_pair_counts<<<blocks, 256, 0, b->stream>>>(P, b->pos_q, b->type, b->lj_eps, b->lj_sig,
                                               b->nl_count, b->nl_ent, d);
  cudaError_t e = cudaGetLastError();
  unsigned long long h[4] = {0, 0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, b->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
  cudaFree(d);
  if (e != cudaSuccess) return cuda_fail(e, "k_pair_counts");
  for (int t = 0; t < 4; t++) out4[t] = (long long)h[t];
  return FE_OK;
}

static double host_ref_erfc(double x) {
  // same function as ref_erfc (ewald.c:817-836), evaluated on the host once
  double z = fabs(x);
  double t = 1.0 / (1.0 + 0.5 * z);
  double v = t * exp(-z * z + -1.26551223 +
                     t * (1.00002368 + t * (0.37409196 + t * (0.09678418 +
                     t * (-0.18628806 + t * (0.27886807 + t * (-1.13520398 +
                     t * (1.48851587 + t * (-0.82215223 + t * 0.17087277)))))))));
  return x < 0 ? 2.0 - v : v;
}

static PairParams pair_params(Box *b) {
  PairParams P;
  P.L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  P.H = make_double3(b->p.L[0] / 2.0, b->p.L[1] / 2.0, b->p.L[2] / 2.0);
  P.rc = b->p.rc;
  P.rc2 = b->p.rc * b->p.rc;
  P.kappa = b->p.kappa;
  P.kpi = 1.0 * b->p.kappa / sqrt(kPI);
  P.epsRF = b->p.epsRF;
  P.erfc_rc = host_ref_erfc(b->p.kappa * b->p.rc);
  P.rec_ew = P.erfc_rc / P.rc;
  P.qfe = kELEC * kELEQ * kELEQ * kNA * 1.0E-3 / P.epsRF;
  P.ron2 = b->p.r_switch > 0.0 ? b->p.r_switch * b->p.r_switch : 0.0;
  const double w = P.rc2 - P.ron2;
  P.inv_sw_den = P.ron2 > 0.0 ? 1.0 / (w * w * w) : 0.0;
  P.sw_c0 = P.rc2 - 3.0 * P.ron2;
  P.lj_form = b->lj_form;
  P.n = b->n;
  P.nt = b->nt;
  P.max_nb = b->max_nb;
  P.sc = make_float3((float)(b->p.L[0] / 4294967296.0), (float)(b->p.L[1] / 4294967296.0),
                     (float)(b->p.L[2] / 4294967296.0));
  // the FP32 distance of two sites at rc is off by less than 2e-6 of rc (a
  // rounding of each 32-bit difference, product and sum) and 2 L / 2^32
  const double Lm = fmax(b->p.L[0], fmax(b->p.L[1], b->p.L[2]));
  const double rm = b->p.rc * (1.0 + 4e-6) + 4.0 * Lm / 4294967296.0;
  P.rf2 = (float)(rm * rm);
  int hi;
  {
    long long bits;
    memcpy(&bits, &P.rc2, sizeof bits);
    hi = (int)(bits >> 32);
  }
  P.tab0 = (hi >> kTabShift) - (kTabN - 1);
  P.parts = 1;
  const double Hm = 0.5 * fmin(b->p.L[0], fmin(b->p.L[1], b->p.L[2]));
  P.wide = b->p.rc >= Hm * (1.0 - 1e-6);  // (the images' rounding is 1e-9 of a box)
  P.nexcl = b->nexcl;
  return P;
}

constexpr size_t kP64Shm = sizeof(double) * kTabN * kTabRow;

int pair64_setup(Box *b) {
  FE_CUDA(cudaDeviceGetAttribute(&b->nsm, cudaDevAttrMultiProcessorCount, b->dev));
  FE_CUDA(cudaMalloc(&b->pair_tab, kP64Shm));
  {
    const size_t nt2 = (size_t)b->nt * b->nt;
    std::vector<unsigned char> on(nt2);
    std::vector<double> lj(3 * nt2);
    const double rc2 = b->p.rc * b->p.rc;
    for (size_t k = 0; k < nt2; k++) {
      const double eps = b->p.lj_eps[k], sig = b->p.lj_sig[k];
      on[k] = eps * sig != 0.0 ? 1 : 0;
      const double s2 = sig * sig / rc2, s6 = s2 * s2 * s2;
      lj[3 * k] = on[k] ? eps : 0.0;
      lj[3 * k + 1] = sig * sig;
      lj[3 * k + 2] = on[k] ? eps * (s6 * s6 - 2.0 * s6) : 0.0;
    }
    FE_CUDA(cudaMalloc(&b->lj_on, nt2));
    FE_CUDA(cudaMemcpy(b->lj_on, on.data(), nt2, cudaMemcpyHostToDevice));
    FE_CUDA(cudaMalloc(&b->lj_tab, sizeof(double) * 3 * nt2));
    FE_CUDA(cudaMemcpy(b->lj_tab, lj.data(), sizeof(double) * 3 * nt2, cudaMemcpyHostToDevice));
  }
  FE_CUDA(cudaFuncSetAttribute(k_pair64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kP64Shm));
  PairParams P = pair_params(b);
  k_pair_table<<<(kTabN + 31) / 32, 32, 0, b->stream>>>(P.kappa, P.kpi, P.tab0, b->pair_tab);
  FE_LAUNCH_CHECK("k_pair_table");
  return FE_OK;
}

int launch_pair_fix(Box *b, bool zero_forces) {
  const double3 invL = make_double3(1.0 / b->p.L[0], 1.0 / b->p.L[1], 1.0 / b->p.L[2]);
  k_pair_fix<<<(b->n + 63) / 64, 64, 0, b->stream>>>(b->n, invL, b->pos_q, b->type, b->pfx,
                                                   zero_forces ? b->ff : nullptr);
  FE_LAUNCH_CHECK("k_pair_fix");
  return FE_OK;
}

int launch_pair64(Box *b) {
  PairParams P = pair_params(b);
  // one block per SM (the table fills its shared memory); a box with few rows
  // splits them so that every warp gets some units to level the ends
  const int warps = b->nsm * kP64Warps, rows = b->n - 1;
  P.parts = kP64Units * warps / rows;
  if (P.parts < 1) P.parts = 1;
  if (P.parts > 8) P.parts = 8;
  int blocks = (rows * P.parts + kP64Warps - 1) / kP64Warps;
  if (blocks > b->nsm) blocks = b->nsm;
  if (blocks > kSumRows) blocks = kSumRows;
  k_pair64<<<blocks, kP64Warps * 32, kP64Shm, b->stream>>>(
      P, b->pair_tab, b->pos_q, b->pfx, b->type, b->lj_tab, b->nl_count, b->nl_ent, b->lj_on,
      b->xl, b->ff, b->part_pair);
  FE_LAUNCH_CHECK("k_pair64");
  b->n_pair = blocks;
  return FE_OK;
}

}  // namespace fe
