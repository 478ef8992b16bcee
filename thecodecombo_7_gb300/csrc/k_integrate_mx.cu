// k_integrate_mx.cu -- the integrator kernels of the mixed-precision step,
// compiled with FMA contraction: the FP64 update of positions and velocities
// (integrate_vverlet.c:54-83) and, for NVE, the tail of the step in one
// launch.  The drop-in's kernels of the same steps (k_integrate.cu) round each
// multiply and add separately as the reference's C does; the mixed path keeps
// FP64 state but needs no such parity, and on this GPU the FP64 pipe is what
// bounds these kernels, so fused multiply-adds cut their time.
#include "fe_device.cuh"
#include "fe_mixed.h"

namespace fe {

// Threads per block of the per-site kernels: the FP64 pipes bind them, so a
// small box spreads over the SMs.
static int mx_site_block(int n) { return n <= 32768 ? 64 : 256; }

__device__ __forceinline__ float mx_prepare(const MxPrepare &m, int i, double4 p) {
  const int s = m.iperm[i];
  const int4 q = fx_site(p, m.invL);
  m.posfx[s] = q;
  m.fix[3 * i] = 0ull;
  m.fix[3 * i + 1] = 0ull;
  m.fix[3 * i + 2] = 0ull;
  return m.snap ? fx_moved2(q, m.snap[s], m.sc) : 0.f;
}

// integrate_vverlet.c:54-83: half kick, drift (atom and atnopbc), pbc_all,
// after the Nose-Hoover scale of the velocities (scale, optional)
__global__ void k_vv1_mx(int n, double vscal, double dt, double dt_h, double3 L, double3 H,
                         const double *__restrict__ imass100, const double *__restrict__ ff,
                         double *__restrict__ vv, double4 *__restrict__ pos,
                         double *__restrict__ nopbc, int *__restrict__ status,
                         const double *__restrict__ scale, MxPrepare m) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  float d2 = 0.f;
  if (i < n) {
    double c = dt_h * imass100[i];
    double w0 = vv[3 * i], w1 = vv[3 * i + 1], w2 = vv[3 * i + 2];
    if (scale) {
      const double s = *scale;
      w0 = __dmul_rn(w0, s);
      w1 = __dmul_rn(w1, s);
      w2 = __dmul_rn(w2, s);
    }
    double v0 = vscal * (w0 + c * ff[3 * i]);
    double v1 = vscal * (w1 + c * ff[3 * i + 1]);
    double v2 = vscal * (w2 + c * ff[3 * i + 2]);
    vv[3 * i] = v0;
    vv[3 * i + 1] = v1;
    vv[3 * i + 2] = v2;
    nopbc[3 * i] += dt * v0;
    nopbc[3 * i + 1] += dt * v1;
    nopbc[3 * i + 2] += dt * v2;
    double4 p = pos[i];
    p.x += dt * v0;
    p.y += dt * v1;
    p.z += dt * v2;
    int bad = 0;
    p.x = pbc_wrap(p.x, H.x, L.x, &bad);
    p.y = pbc_wrap(p.y, H.y, L.y, &bad);
    p.z = pbc_wrap(p.z, H.z, L.z, &bad);
    if (bad) atomicOr(status, ST_PBC_LOOP);
    pos[i] = p;
    if (m.iperm) d2 = mx_prepare(m, i, p);
  }
  if (m.iperm && m.snap) fx_moved_max(d2, m.dmax2);
}

int launch_vv1_mx(Box *b, double vscal, bool scaled) {
  double3 L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  double3 H = make_double3(b->p.L[0] / 2.0, b->p.L[1] / 2.0, b->p.L[2] / 2.0);
  double dt = b->p.dt, dt_h = 0.5 * b->p.dt;
  const int tb = mx_site_block(b->n);
  k_vv1_mx<<<(b->n + tb - 1) / tb, tb, 0, b->stream>>>(
      b->n, vscal, dt, dt_h, L, H, b->imass100, b->ff, b->vv, b->pos_q, b->pos_nopbc, b->status,
      scaled ? b->scal + SC_NHC_SCALE : nullptr, mixed_prepare(b, b->have_list, b->mx->inner_on));
  FE_LAUNCH_CHECK("k_vv1_mx");
  return FE_OK;
}

// What the last block of a step's second half kick does with the kinetic tensor.
// nhc 0: the record.  1: the chain update that ends the step, whose velocity
// scale k_mx_scale_kinet / k_b_scale_kinet applies.  2: a step of the same run
// follows: the tensor of the scaled velocities is s^2 times this one, so the
// record and the chain update that opens the next step need no pass over the
// velocities, and the next first half kick applies both scales in one (4,095
// sites: 83 us a step with the pass between, 76 without).
__device__ __forceinline__ void vv2_end(const BIntArgs &a, int nhc) {
  if (nhc == 0) {
    record_dev(a.scal, a.rec, a.rec_cap, a.rec_counter);
    return;
  }
  nhc_chain_dev(a.nhc_M, a.nhc_Q, a.nfree, a.dt, a.zeta, a.scal);
  if (nhc == 1) return;
  const double s = a.scal[SC_NHC_SCALE], s2 = s * s;
  for (int i = 0; i < 6; i++) a.scal[SC_KEN + i] *= s2;
  a.scal[FE_EN_KINET] = a.scal[SC_KEN + 0] + a.scal[SC_KEN + 2] + a.scal[SC_KEN + 5];
  record_dev(a.scal, a.rec, a.rec_cap, a.rec_counter);
  nhc_chain_dev(a.nhc_M, a.nhc_Q, a.nfree, a.dt, a.zeta, a.scal);
  a.scal[SC_NHC_SCALE] *= s;
}

// Mixed precision: the tail of a step in one launch -- the FP64 forces from
// the fixed-point sums minus the mean reciprocal force (k_mx_finalize), the
// energy assembly in block 0 (k_mx_slots, k_assemble), the second half kick
// with uu = vv and the kinetic tensor (k_vv2_kinet); the last block finishes
// kinet and writes the step's record or updates the Nose-Hoover chain (vv2_end).
constexpr double kMxForceFix = 4294967296.0;  // 2^32 per kJ/mol/A

__device__ __forceinline__ void vv2_tail_body(const BIntArgs &a, VBlk vb, int nhc) {
  if (vb.id == 0 && threadIdx.x == 0) {
    mixed_slots_dev(a.scal, a.erfc_rc_over_rc, a.mixed_fused);
    assemble_dev(a.scal, a.fan, a.sewald, 1);
  }
  __shared__ double mean[3];
  if (threadIdx.x < 3) mean[threadIdx.x] = a.scal[SC_FMEAN + threadIdx.x] / kMxForceFix / (double)a.n;
  __syncthreads();
  double k[6] = {0, 0, 0, 0, 0, 0};
  for (int i = vb.id * blockDim.x + threadIdx.x; i < a.n; i += vb.n * blockDim.x) {
    double imass = a.imass100[i];
    double v[3];
    for (int c = 0; c < 3; c++) {
      double f = (double)(long long)a.fix[3 * i + c] * (1.0 / kMxForceFix) - mean[c];
      a.ff[3 * i + c] = f;
      v[c] = (a.vv[3 * i + c] + 1.0 * a.dt_h * imass * f);
      a.vv[3 * i + c] = v[c];
      a.uu[3 * i + c] = v[c];
    }
    double fac = a.mass[i];
    double sx = v[0] + v[0], sy = v[1] + v[1], sz = v[2] + v[2];
    k[0] += fac * sx * sx;
    k[1] += fac * sy * sx;
    k[2] += fac * sy * sy;
    k[3] += fac * sz * sx;
    k[4] += fac * sz * sy;
    k[5] += fac * sz * sz;
  }
  if (block_fix_final<6>(k, 20, a.facc, a.ticket, a.scal + SC_KEN, vb) && threadIdx.x == 0) {
    kinet_scalars(a.scal);
    vv2_end(a, nhc);
  }
}

__global__ void k_vv2_mx_tail(const __grid_constant__ BIntArgs a, int nhc) {
  vv2_tail_body(a, vblk_self(), nhc);
}

int launch_vv2_mx_tail(Box *b, int nhc) {
  BIntArgs a = make_bint_args(b);
  const int tb = mx_site_block(b->n);
  int blocks = (b->n + tb - 1) / tb;
  if (blocks > 512) blocks = 512;
  k_vv2_mx_tail<<<blocks, tb, 0, b->stream>>>(a, nhc);
  FE_LAUNCH_CHECK("k_vv2_mx_tail");
  return FE_OK;
}

// kinet of the velocities (k_kinet_fix): `scale`: after the chain's velocity
// scale (integrate_nhc.c:152-159), with the record; else with the chain update
// that opens a step (integrate_nhc.c:57-147)
__global__ void k_mx_scale_kinet(BIntArgs a, int scale) {
  const double s = scale ? a.scal[SC_NHC_SCALE] : 1.0;
  double k[6] = {0, 0, 0, 0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
    double v[3], u[3];
    for (int c = 0; c < 3; c++) {
      v[c] = a.vv[3 * i + c];
      u[c] = a.uu[3 * i + c];
      if (scale) {
        v[c] = __dmul_rn(v[c], s);
        u[c] = __dmul_rn(u[c], s);
        a.vv[3 * i + c] = v[c];
        a.uu[3 * i + c] = u[c];
      }
    }
    double fac = a.mass[i];
    double sx = v[0] + u[0], sy = v[1] + u[1], sz = v[2] + u[2];
    k[0] += fac * sx * sx;
    k[1] += fac * sy * sx;
    k[2] += fac * sy * sy;
    k[3] += fac * sz * sx;
    k[4] += fac * sz * sy;
    k[5] += fac * sz * sz;
  }
  if (block_fix_final<6>(k, 20, a.facc, a.ticket, a.scal + SC_KEN) && threadIdx.x == 0) {
    kinet_scalars(a.scal);
    if (scale) record_dev(a.scal, a.rec, a.rec_cap, a.rec_counter);
    else nhc_chain_dev(a.nhc_M, a.nhc_Q, a.nfree, a.dt, a.zeta, a.scal);
  }
}

int launch_mx_scale_kinet(Box *b, bool scale) {
  const int tb = mx_site_block(b->n);
  int blocks = (b->n + tb - 1) / tb;
  if (blocks > 512) blocks = 512;
  k_mx_scale_kinet<<<blocks, tb, 0, b->stream>>>(make_bint_args(b), scale ? 1 : 0);
  FE_LAUNCH_CHECK("k_mx_scale_kinet");
  return FE_OK;
}

// ---------------------------------------------------------------------------
// Integrator kernels of a batched step: every box of a replica batch in one
// launch per kernel (blocks of box r: off[r] .. off[r+1]-1).  The arithmetic
// is that of the single-box kernels above, site for site; the Nose-Hoover
// velocity scale is applied inside the next per-site pass instead of in a
// launch of its own, and the energy assembly rides on the second half kick.


// kinet (fixed point, as k_kinet_fix) and the first Nose-Hoover chain update
__global__ void k_b_kinet_nhc(const BIntArgs *__restrict__ A, const int *__restrict__ off,
                              int nbox) {
  const int r = vblk_box(off, nbox);
  const BIntArgs &a = A[r];
  const VBlk vb = vblk_of(off, r);
  double k[6] = {0, 0, 0, 0, 0, 0};
  for (int i = vb.id * blockDim.x + threadIdx.x; i < a.n; i += vb.n * blockDim.x) {
    double fac = a.mass[i];
    double sx = a.vv[3 * i] + a.uu[3 * i];
    double sy = a.vv[3 * i + 1] + a.uu[3 * i + 1];
    double sz = a.vv[3 * i + 2] + a.uu[3 * i + 2];
    k[0] += fac * sx * sx;
    k[1] += fac * sy * sx;
    k[2] += fac * sy * sy;
    k[3] += fac * sz * sx;
    k[4] += fac * sz * sy;
    k[5] += fac * sz * sz;
  }
  if (block_fix_final<6>(k, 20, a.facc, a.ticket, a.scal + SC_KEN, vb) && threadIdx.x == 0) {
    kinet_scalars(a.scal);
    nhc_chain_dev(a.nhc_M, a.nhc_Q, a.nfree, a.dt, a.zeta, a.scal);
  }
}

// [Nose-Hoover velocity scale, integrate_nhc.c:152-159] then the first half
// kick, drift and pbc_all (integrate_vverlet.c:54-83, vscal = 1) and what the
// force evaluation starts from
__global__ void k_b_vv1(const BIntArgs *__restrict__ A, const int *__restrict__ off, int nbox,
                        int nhc) {
  const int r = vblk_box(off, nbox);
  const BIntArgs &a = A[r];
  const VBlk vb = vblk_of(off, r);
  int i = vb.id * blockDim.x + threadIdx.x;
  float d2 = 0.f;
  if (i < a.n) {
    double v[3];
    for (int c = 0; c < 3; c++) v[c] = a.vv[3 * i + c];
    if (nhc) {
      double scale = a.scal[SC_NHC_SCALE];
      for (int c = 0; c < 3; c++) {
        v[c] = v[c] * scale;
        a.uu[3 * i + c] = a.uu[3 * i + c] * scale;
      }
    }
    double imass = a.imass100[i];
    for (int c = 0; c < 3; c++) {
      v[c] = 1.0 * (v[c] + a.dt_h * imass * a.ff[3 * i + c]);
      a.vv[3 * i + c] = v[c];
    }
    double ddx = a.dt * v[0], ddy = a.dt * v[1], ddz = a.dt * v[2];
    a.nopbc[3 * i] += ddx;
    a.nopbc[3 * i + 1] += ddy;
    a.nopbc[3 * i + 2] += ddz;
    double4 p = a.pos[i];
    p.x += ddx;
    p.y += ddy;
    p.z += ddz;
    int bad = 0;
    p.x = pbc_wrap(p.x, a.H.x, a.L.x, &bad);
    p.y = pbc_wrap(p.y, a.H.y, a.L.y, &bad);
    p.z = pbc_wrap(p.z, a.H.z, a.L.z, &bad);
    if (bad) atomicOr(a.status, ST_PBC_LOOP);
    a.pos[i] = p;
    d2 = mx_prepare(a.m, i, p);
  }
  if (a.m.snap) fx_moved_max(d2, a.m.dmax2);
}

// the end of a step, as k_vv2_mx_tail
__global__ void k_b_vv2(const BIntArgs *__restrict__ A, const int *__restrict__ off, int nbox,
                        int nhc) {
  const int r = vblk_box(off, nbox);
  vv2_tail_body(A[r], vblk_of(off, r), nhc);
}

// NHC: the second velocity scale, kinet of the scaled velocities and the record
__global__ void k_b_scale_kinet(const BIntArgs *__restrict__ A, const int *__restrict__ off,
                                int nbox) {
  const int r = vblk_box(off, nbox);
  const BIntArgs &a = A[r];
  const VBlk vb = vblk_of(off, r);
  double scale = a.scal[SC_NHC_SCALE];
  double k[6] = {0, 0, 0, 0, 0, 0};
  for (int i = vb.id * blockDim.x + threadIdx.x; i < a.n; i += vb.n * blockDim.x) {
    double v[3], u[3];
    for (int c = 0; c < 3; c++) {
      v[c] = a.vv[3 * i + c] * scale;
      u[c] = a.uu[3 * i + c] * scale;
      a.vv[3 * i + c] = v[c];
      a.uu[3 * i + c] = u[c];
    }
    double fac = a.mass[i];
    double sx = v[0] + u[0], sy = v[1] + u[1], sz = v[2] + u[2];
    k[0] += fac * sx * sx;
    k[1] += fac * sy * sx;
    k[2] += fac * sy * sy;
    k[3] += fac * sz * sx;
    k[4] += fac * sz * sy;
    k[5] += fac * sz * sz;
  }
  if (block_fix_final<6>(k, 20, a.facc, a.ticket, a.scal + SC_KEN, vb) && threadIdx.x == 0) {
    kinet_scalars(a.scal);
    record_dev(a.scal, a.rec, a.rec_cap, a.rec_counter);
  }
}

int launch_b_kinet_nhc(const BIntArgs *A, const int *off, int nbox, int blocks, cudaStream_t s) {
  k_b_kinet_nhc<<<blocks, 256, 0, s>>>(A, off, nbox);
  FE_LAUNCH_CHECK("k_b_kinet_nhc");
  return FE_OK;
}
int launch_b_vv1(const BIntArgs *A, const int *off, int nbox, int blocks, int nhc,
                 cudaStream_t s) {
  k_b_vv1<<<blocks, 256, 0, s>>>(A, off, nbox, nhc);
  FE_LAUNCH_CHECK("k_b_vv1");
  return FE_OK;
}
int launch_b_vv2(const BIntArgs *A, const int *off, int nbox, int blocks, int nhc,
                 cudaStream_t s) {
  k_b_vv2<<<blocks, 256, 0, s>>>(A, off, nbox, nhc);
  FE_LAUNCH_CHECK("k_b_vv2");
  return FE_OK;
}
int launch_b_scale_kinet(const BIntArgs *A, const int *off, int nbox, int blocks,
                         cudaStream_t s) {
  k_b_scale_kinet<<<blocks, 256, 0, s>>>(A, off, nbox);
  FE_LAUNCH_CHECK("k_b_scale_kinet");
  return FE_OK;
}

}  // namespace fe
