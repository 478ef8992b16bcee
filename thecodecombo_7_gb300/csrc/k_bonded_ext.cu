// k_bonded_ext.cu -- the bonded terms of forces() in FP64: for the drop-in
// bonds (cbond.c:27-180), bends (cbend.c:24-218), Urey-Bradley 1-3 terms
// (curey.c:37-106), proper torsions (ctorsion.c:63-246) and improper torsions
// (cimproper.c:55-221) in one launch (k_bonded64); for the mixed precision
// the last three (its bonds and bends are in its intramolecular kernel).
//
// One thread per term.  The torsion and improper geometry is the reference's
// (unit bond vectors, the two cross products with the central bond, the sign
// from their cross product along it, tau = sign * acos of the clamped
// cosine) and its force transformation onto the four sites; only the order of
// the final per-site sums differs (atomics).  The drop-in precision adds the
// forces to ff through FP64 atomics; the mixed precision adds them to the
// 64-bit fixed-point force sums (2^32 per kJ/mol/A, exact and order-free).
// Energies are summed exactly in 64-bit fixed point (2^-32 kJ/mol) and land in
// the slots SC_UREY, SC_TORS, SC_IMPR.  These terms are few (a few per
// molecule) and run once per force evaluation, so FP64 costs little here and
// keeps acos well conditioned near 0 and pi.
#include "fe_device.cuh"
#include "fe_mixed.h"

namespace fe {

constexpr double kExtFix = 4294967296.0;  // 2^32: the mixed force sums' scale

__device__ __forceinline__ void min_image3(double3 L, double3 H, double *d) {
  double l[3] = {L.x, L.y, L.z}, h[3] = {H.x, H.y, H.z};
#pragma unroll
  for (int c = 0; c < 3; c++) {
    if (d[c] > h[c]) d[c] -= l[c];
    else if (d[c] < -h[c]) d[c] += l[c];
  }
}

template <bool FIXED>
__device__ __forceinline__ void add_force(double *ff, unsigned long long *fix, int i, int c,
                                          double v) {
  if (FIXED)
    atomicAdd(&fix[3 * i + c], (unsigned long long)__double2ll_rn(v * kExtFix));
  else
    atomicAdd(&ff[3 * i + c], v);
}

struct ExtArgs {
  double3 L, H;
  int nbond, nbend, nurey, ntors, nimpr;  // terms evaluated of each kind
  const int *bond_ab, *bend_abc;
  const double *bond_req, *bond_k, *bend_t0, *bend_k;
  const int *urey_ab;
  const double *urey_seq, *urey_k;
  const int *tors_abcd;
  const double *tors_par;  // 18 per torsion: kphi[6], nphi[6], delphi[6]
  double *tors_tau;
  const int *impr_abcd;
  const double *impr_k, *impr_eq;
};

// the dihedral (a, b, c, d) and its generalised force fr = -dE/dtau applied
// to the four sites (ctorsion.c:80-246, cimproper.c:71-221)
struct Dihedral {
  double u[3], w[3];  // eab x ebc, ecd x ebc
  double rab, rbc, rcd, irab, irbc, ircd, cosb, cosc, isinb2, isinc2;
  double tau;
};

__device__ __forceinline__ void dihedral_geom(const double4 *__restrict__ pos, double3 L,
                                              double3 H, int ia, int ib, int ic, int id,
                                              Dihedral &D) {
  double4 A = pos[ia], B = pos[ib], Cc = pos[ic], Dd = pos[id];
  double dab[3] = {B.x - A.x, B.y - A.y, B.z - A.z};
  double dbc[3] = {Cc.x - B.x, Cc.y - B.y, Cc.z - B.z};
  double dcd[3] = {Dd.x - Cc.x, Dd.y - Cc.y, Dd.z - Cc.z};
  min_image3(L, H, dab);
  min_image3(L, H, dbc);
  min_image3(L, H, dcd);
  D.rab = sqrt(dab[0] * dab[0] + dab[1] * dab[1] + dab[2] * dab[2]);
  D.irab = 1.0 / D.rab;
  D.rbc = sqrt(dbc[0] * dbc[0] + dbc[1] * dbc[1] + dbc[2] * dbc[2]);
  D.irbc = 1.0 / D.rbc;
  D.rcd = sqrt(dcd[0] * dcd[0] + dcd[1] * dcd[1] + dcd[2] * dcd[2]);
  D.ircd = 1.0 / D.rcd;
  double eab[3], ebc[3], ecd[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    eab[c] = dab[c] * D.irab;
    ebc[c] = dbc[c] * D.irbc;
    ecd[c] = dcd[c] * D.ircd;
  }
  D.u[0] = eab[1] * ebc[2] - eab[2] * ebc[1];
  D.u[1] = eab[2] * ebc[0] - eab[0] * ebc[2];
  D.u[2] = eab[0] * ebc[1] - eab[1] * ebc[0];
  D.cosb = -(eab[0] * ebc[0] + eab[1] * ebc[1] + eab[2] * ebc[2]);
  D.isinb2 = 1.0 / (1.0 - D.cosb * D.cosb);
  D.w[0] = ecd[1] * ebc[2] - ecd[2] * ebc[1];
  D.w[1] = ecd[2] * ebc[0] - ecd[0] * ebc[2];
  D.w[2] = ecd[0] * ebc[1] - ecd[1] * ebc[0];
  D.cosc = -(ecd[0] * ebc[0] + ecd[1] * ebc[1] + ecd[2] * ebc[2]);
  D.isinc2 = 1.0 / (1.0 - D.cosc * D.cosc);
  double x0 = -(D.u[1] * D.w[2] - D.u[2] * D.w[1]);
  double x1 = -(D.u[2] * D.w[0] - D.u[0] * D.w[2]);
  double x2 = -(D.u[0] * D.w[1] - D.u[1] * D.w[0]);
  double num = x0 * ebc[0] + x1 * ebc[1] + x2 * ebc[2];
  double costau = -(D.u[0] * D.w[0] + D.u[1] * D.w[1] + D.u[2] * D.w[2]) * sqrt(D.isinb2) *
                  sqrt(D.isinc2);
  costau = fmin(1.0, fmax(-1.0, costau));
  D.tau = (num >= 0.0 ? 1.0 : -1.0) * acos(costau);
}

template <bool FIXED>
__device__ __forceinline__ void dihedral_force(const Dihedral &D, double fr, int ia, int ib,
                                               int ic, int id, double *ff,
                                               unsigned long long *fix) {
  double fa = -fr * D.irab * D.isinb2;
  double fb1 = fr * (D.rbc - D.rab * D.cosb) * D.irab * D.irbc * D.isinb2;
  double fb2 = fr * D.cosc * D.irbc * D.isinc2;
  double fc1 = fr * (D.rbc - D.rcd * D.cosc) * D.ircd * D.irbc * D.isinc2;
  double fc2 = fr * D.cosb * D.irbc * D.isinb2;
  double fd = -fr * D.ircd * D.isinc2;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    add_force<FIXED>(ff, fix, ia, c, fa * D.u[c]);
    add_force<FIXED>(ff, fix, ib, c, fb1 * D.u[c] + fb2 * D.w[c]);
    add_force<FIXED>(ff, fix, ic, c, fc1 * D.w[c] + fc2 * D.u[c]);
    add_force<FIXED>(ff, fix, id, c, fd * D.w[c]);
  }
}

// harmonic stretch (cbond.c, curey.c): E = k (r - r0)^2, its energy returned
template <bool FIXED>
__device__ __forceinline__ double stretch_term(const ExtArgs &a, const double4 *__restrict__ pos,
                                               const int *__restrict__ ab, double req, double k,
                                               double *ff, unsigned long long *fix) {
  int ia = ab[0], ib = ab[1];
  double4 A = pos[ia], B = pos[ib];
  double d[3] = {B.x - A.x, B.y - A.y, B.z - A.z};
  min_image3(a.L, a.H, d);
  double dr = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  double dri = 1.0 / dr;
  double rr = dr - req;
  double fr = -k * rr * 2.0;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    double f = fr * dri * d[c];
    add_force<FIXED>(ff, fix, ia, c, -f);
    add_force<FIXED>(ff, fix, ib, c, f);
  }
  return -(fr * rr * 0.5);
}

// cbend.c: E = k (theta - theta0)^2 (drop-in only)
__device__ __forceinline__ double bend_term(const ExtArgs &a, const double4 *__restrict__ pos,
                                            int u, double *ff) {
  int ia = a.bend_abc[3 * u], ib = a.bend_abc[3 * u + 1], ic = a.bend_abc[3 * u + 2];
  double4 A = pos[ia], B = pos[ib], Cc = pos[ic];
  double da[3] = {A.x - B.x, A.y - B.y, A.z - B.z}, dc[3] = {Cc.x - B.x, Cc.y - B.y, Cc.z - B.z};
  min_image3(a.L, a.H, da);
  min_image3(a.L, a.H, dc);
  double drai = 1.0 / sqrt(da[0] * da[0] + da[1] * da[1] + da[2] * da[2]);
  double erax = da[0] * drai, eray = da[1] * drai, eraz = da[2] * drai;
  double drci = 1.0 / sqrt(dc[0] * dc[0] + dc[1] * dc[1] + dc[2] * dc[2]);
  double ercx = dc[0] * drci, ercy = dc[1] * drci, ercz = dc[2] * drci;
  double cosphi = erax * ercx + eray * ercy + eraz * ercz;
  double phi = acos(cosphi);
  double isinphi = 1.0 / sqrt(1.0 - cosphi * cosphi);
  double rr = phi - a.bend_t0[u];
  double fr = -a.bend_k[u] * rr * 2.0;
  double irasin = drai * isinphi * fr;
  double ircsin = drci * isinphi * fr;
  double fxa = (erax * cosphi - ercx) * irasin;
  double fya = (eray * cosphi - ercy) * irasin;
  double fza = (eraz * cosphi - ercz) * irasin;
  double fxc = (ercx * cosphi - erax) * ircsin;
  double fyc = (ercy * cosphi - eray) * ircsin;
  double fzc = (ercz * cosphi - eraz) * ircsin;
  add_force<false>(ff, nullptr, ia, 0, fxa);
  add_force<false>(ff, nullptr, ia, 1, fya);
  add_force<false>(ff, nullptr, ia, 2, fza);
  add_force<false>(ff, nullptr, ib, 0, -(fxa + fxc));
  add_force<false>(ff, nullptr, ib, 1, -(fya + fyc));
  add_force<false>(ff, nullptr, ib, 2, -(fza + fzc));
  add_force<false>(ff, nullptr, ic, 0, fxc);
  add_force<false>(ff, nullptr, ic, 1, fyc);
  add_force<false>(ff, nullptr, ic, 2, fzc);
  return -fr * rr * 0.5;
}

// term t of the Urey-Bradley, torsion, improper sequence; its energy into e
template <bool FIXED>
__device__ __forceinline__ void ext_term(const ExtArgs &a, const double4 *__restrict__ pos, int t,
                                         double *ff, unsigned long long *fix, double &e_urey,
                                         double &e_tors, double &e_impr) {
  if (t < a.nurey) {
    e_urey += stretch_term<FIXED>(a, pos, a.urey_ab + 2 * t, a.urey_seq[t], a.urey_k[t], ff, fix);
  } else if (t < a.nurey + a.ntors) {
    int u = t - a.nurey;
    const int *q = a.tors_abcd + 4 * u;
    Dihedral D;
    dihedral_geom(pos, a.L, a.H, q[0], q[1], q[2], q[3], D);
    a.tors_tau[u] = D.tau;
    const double *kp = a.tors_par + 18 * u;
    double fr = 0.0, et = 0.0;
    for (int s = 0; s < 6; s++) {  // the series ends at the first zero kphi
      if (kp[s] == 0.0) break;
      double arg = kp[6 + s] * D.tau - kp[12 + s];
      double sn, cs;
      sincos(arg, &sn, &cs);
      fr += kp[s] * kp[6 + s] * sn;
      et += kp[s] * (1.0 + cs);
    }
    e_tors += et;
    dihedral_force<FIXED>(D, fr, q[0], q[1], q[2], q[3], ff, fix);
  } else {
    int u = t - a.nurey - a.ntors;
    const int *q = a.impr_abcd + 4 * u;
    Dihedral D;
    dihedral_geom(pos, a.L, a.H, q[0], q[1], q[2], q[3], D);
    double rr = D.tau - a.impr_eq[u];
    double fr = -2.0 * a.impr_k[u] * rr;
    e_impr += -fr * rr * 0.5;
    dihedral_force<FIXED>(D, fr, q[0], q[1], q[2], q[3], ff, fix);
  }
}

// the drop-in's terms: bonds, bends, then ext_term's
__global__ void k_bonded64(ExtArgs a, const double4 *__restrict__ pos, double *__restrict__ ff,
                           double *__restrict__ partials) {
  double e[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int tot = a.nbond + a.nbend + a.nurey + a.ntors + a.nimpr;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += gridDim.x * blockDim.x) {
    if (t < a.nbond)
      e[0] += stretch_term<false>(a, pos, a.bond_ab + 2 * t, a.bond_req[t], a.bond_k[t], ff,
                                  nullptr);
    else if (t < a.nbond + a.nbend)
      e[1] += bend_term(a, pos, t - a.nbond, ff);
    else
      ext_term<false>(a, pos, t - a.nbond - a.nbend, ff, nullptr, e[2], e[3], e[4]);
  }
  block_partials<5>(e, partials);
}

// the mixed precision's Urey-Bradley, torsion and improper terms
__global__ void __launch_bounds__(128)
k_bonded_ext(ExtArgs a, const double4 *__restrict__ pos, unsigned long long *__restrict__ fix,
             unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
             double *__restrict__ out) {
  double e[3] = {0.0, 0.0, 0.0};  // urey, torsion, improper
  const int tot = a.nurey + a.ntors + a.nimpr;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += gridDim.x * blockDim.x)
    ext_term<true>(a, pos, t, nullptr, fix, e[0], e[1], e[2]);
  block_fix_final<3>(e, 32, facc, ticket, out);
}

static ExtArgs ext_args(const Box *b, int kinds) {
  ExtArgs a;
  a.L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  a.H = make_double3(b->p.L[0] / 2.0, b->p.L[1] / 2.0, b->p.L[2] / 2.0);
  a.nbond = kinds & BK_BOND ? b->nbond : 0;
  a.nbend = kinds & BK_BEND ? b->nbend : 0;
  a.nurey = kinds & BK_UREY ? b->nurey : 0;
  a.ntors = kinds & BK_TORS ? b->ntors : 0;
  a.nimpr = kinds & BK_IMPR ? b->nimpr : 0;
  a.bond_ab = b->bond_ab;
  a.bend_abc = b->bend_abc;
  a.bond_req = b->bond_req;
  a.bond_k = b->bond_k;
  a.bend_t0 = b->bend_t0;
  a.bend_k = b->bend_k;
  a.urey_ab = b->urey_ab;
  a.urey_seq = b->urey_seq;
  a.urey_k = b->urey_k;
  a.tors_abcd = b->tors_abcd;
  a.tors_par = b->tors_par;
  a.tors_tau = b->tors_tau;
  a.impr_abcd = b->impr_abcd;
  a.impr_k = b->impr_k;
  a.impr_eq = b->impr_eq;
  return a;
}

// Few terms: one warp per block, so that their FP64 instructions (300 for a
// torsion) spread over the SMs' narrow FP64 pipes: 1,365 water molecules took
// 15 us in 16 blocks of 256 threads.
static void bonded_shape(int tot, int *blocks, int *threads) {
  *threads = tot <= 32 * 512 ? 32 : 128;
  *blocks = (tot + *threads - 1) / *threads;
  if (*blocks > kSumRows) *blocks = kSumRows;
  if (*blocks < 1) *blocks = 1;
}

int launch_bonded64(Box *b, int kinds, bool fast) {
  const ExtArgs a = ext_args(b, kinds);
  int blocks, threads;
  bonded_shape(a.nbond + a.nbend + a.nurey + a.ntors + a.nimpr, &blocks, &threads);
  k_bonded64<<<blocks, threads, 0, b->stream>>>(a, b->pos_q, b->ff,
                                                fast ? b->part_fast : b->part_bond);
  FE_LAUNCH_CHECK("k_bonded64");
  if (fast) {
    b->n_fast = blocks;
  } else {
    b->n_bond = blocks;
    b->bond_kinds = (unsigned)kinds;
  }
  return FE_OK;
}

int launch_bonded_ext_mixed(Box *b) {
  const ExtArgs a = ext_args(b, BK_UREY | BK_TORS | BK_IMPR);
  const int tot = a.nurey + a.ntors + a.nimpr;
  if (tot == 0) return FE_OK;
  int blocks, threads;
  bonded_shape(tot, &blocks, &threads);
  k_bonded_ext<<<blocks, threads, 0, b->stream>>>(a, b->pos_q, b->mx->fix, b->facc, b->ticket,
                                                  b->scal + SC_UREY);
  FE_LAUNCH_CHECK("k_bonded_ext");
  return FE_OK;
}

}  // namespace fe
