// k_mixed.cu -- the mixed-precision force engine: FP32 pair and SPME math,
// 64-bit fixed-point force sums (exact, so the result does not depend on the
// order of summation), FP64 integration and energy reductions.
//
// Layout (rebuilt with the list, every nlist steps):
//   * sites are sorted by a cell grid of edge h >= rlist/3 (cells assigned
//     from the same 32-bit fractions as below); perm[s] is the original
//     index of sorted slot s;
//   * every step, posfx[s] = (x, y, z) as unsigned 32-bit fractions of the box
//     length (x/L + 1/2 scaled by 2^32) and the charge: the difference of two
//     coordinates taken in 32-bit integer arithmetic wraps around, which IS the
//     minimum image for |d| < L/2, and converts to FP32 with a relative error
//     of 2^-24 (~2e-7 A at 3 A) -- no image shifts, no cell-relative frames;
//   * the OUTER list is full (both directions, no Newton-3 scatter): row s
//     holds every non-excluded j within rlist, pairs with an LJ term at the
//     front and the rest at the back.  It is built per unit of 8 sorted
//     sites (4 or 1 in small boxes): the candidates near the unit's bounding box
//     are loaded once and tested against all its sites;
//   * the pair kernel reads an INNER list (rc + skin, skin 0.8 A): it prunes
//     the outer rows into it while computing forces after every list
//     rebuild and whenever some site has moved skin/2 since the last prune
//     (measured every step against a snapshot of the positions), so every
//     pair within rc is always in it -- the forces are those of the outer
//     list, with ~27 % fewer entries walked (small boxes walk the outer rows);
//   * excluded / 1-4 pairs (xint) are handled with the bonded terms, one
//     thread per term when all molecules are alike, one per molecule when they
//     are contiguous runs of sites, else by kernels over the exclusion list
//     (cnonbond_nblist.c:245-263, 416-437 semantics);
//   * SPME spreading adds every site's spline contributions to 64-bit
//     fixed-point grid sums with integer reductions (order independent),
//     which the transform kernels (fe_fft.cuh) read, or a pass converts to the
//     FP32 grid for the library; at order 4 the spline weights are computed where
//     they are used (spreading, gather).
// In the pair kernel one warp walks a row (rows handed out from a device
// counter) with coalesced entry loads, two entries a lane at a time; the row's
// FP32 partial sums are added over the warp in a fixed order and converted once
// to the fixed-point accumulators (2^32 per kJ/mol/A) -- deterministic.
#include <algorithm>
#include <climits>
#include <cstring>
#include <cmath>
#include <vector>

#include "fe_device.cuh"
#include "fe_df.cuh"
#include "fe_mixed.h"

namespace fe {

constexpr double kFixScale = 4294967296.0;  // 2^32
constexpr float kFixScaleF = 4294967296.0f;
constexpr int kMxWarps = 8;                 // warps per block of the list build
constexpr int kMxMaxCellAtoms = 2048;       // sites per cell a sort block handles

__device__ __forceinline__ long long to_fix(float v) { return __float2ll_rn(v * kFixScaleF); }

// v in [-g, 2g) wrapped into [0, g) without a division
__device__ __forceinline__ int wrap1(int v, int g) { return v < 0 ? v + g : (v >= g ? v - g : v); }

// a fixed-point coordinate difference in A, in FP64 (the integer difference
// is exact; sd = L / 2^32 in double)
__device__ __forceinline__ double fx_delta_d(unsigned a, unsigned b, double sd) {
  return (double)(int)(a - b) * sd;
}

// ---------------------------------------------------------------------------
// sorting by cells

// cell of each site from the same 32-bit fractions the kernels see, so that
// cell membership and fixed-point coordinates always agree
__device__ __forceinline__ void k_mx_cell_body(VBlk vb_, int n, const double4 *__restrict__ pos, double3 invL, int3 nc,
                          int *__restrict__ cell_of, int *__restrict__ count) {
  int i = vb_.id * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = pos[i];
  int cx = (int)(((unsigned long long)frac32(p.x, invL.x) * (unsigned)nc.x) >> 32);
  int cy = (int)(((unsigned long long)frac32(p.y, invL.y) * (unsigned)nc.y) >> 32);
  int cz = (int)(((unsigned long long)frac32(p.z, invL.z) * (unsigned)nc.z) >> 32);
  int c = (cx * nc.y + cy) * nc.z + cz;
  cell_of[i] = c;
  atomicAdd(&count[c], 1);
}

__global__ void k_mx_cell(int n, const double4 *__restrict__ pos, double3 invL, int3 nc,
                          int *__restrict__ cell_of, int *__restrict__ count) {
  k_mx_cell_body(vblk_self(), n, pos, invL, nc, cell_of, count);
}

__device__ __forceinline__ void k_mx_fill_body(VBlk vb_, int n, const int *__restrict__ cell_of, const int *__restrict__ start,
                          int *__restrict__ fill, int *__restrict__ perm) {
  int i = vb_.id * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c = cell_of[i];
  int s = atomicAdd(&fill[c], 1);
  perm[start[c] + s] = i;
}

__global__ void k_mx_fill(int n, const int *__restrict__ cell_of, const int *__restrict__ start,
                          int *__restrict__ fill, int *__restrict__ perm) {
  k_mx_fill_body(vblk_self(), n, cell_of, start, fill, perm);
}

// order each cell's sites by original index (deterministic layout): cells of up
// to 32 sites by rank within one warp, larger ones by a bitonic sort
__device__ __forceinline__ void k_mx_cellsort_body(VBlk vb_, const int *__restrict__ start, int *__restrict__ perm,
                              int *__restrict__ iperm, int *__restrict__ cell_s,
                              const int *__restrict__ type, int *__restrict__ type_s,
                              int *__restrict__ status) {
  __shared__ int buf[kMxMaxCellAtoms];
  int c = vb_.id;
  int s0 = start[c], s1 = start[c + 1];
  int m = s1 - s0;
  if (m > kMxMaxCellAtoms) {
    if (threadIdx.x == 0) atomicOr(status, ST_CELL_OVERFLOW);
    m = kMxMaxCellAtoms;
  }
  if (m <= 32 && blockDim.x == 32) {
    // one site per lane: its rank among the cell's original indices
    const int lane = threadIdx.x;
    int v = lane < m ? perm[s0 + lane] : INT_MAX;
    int rank = 0;
#pragma unroll
    for (int src = 0; src < 32; src++) rank += __shfl_sync(0xffffffffu, v, src) < v ? 1 : 0;
    if (lane < m) {
      perm[s0 + rank] = v;
      iperm[v] = s0 + rank;
      cell_s[s0 + rank] = c;
      type_s[s0 + rank] = type[v];
    }
    return;
  }
  int P = 1;
  while (P < m) P <<= 1;
  for (int i = threadIdx.x; i < P; i += blockDim.x) buf[i] = i < m ? perm[s0 + i] : INT_MAX;
  __syncthreads();
  for (int k = 2; k <= P; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < P; i += blockDim.x) {
        int ixj = i ^ j;
        if (ixj > i) {
          int a = buf[i], b = buf[ixj];
          bool up = (i & k) == 0;
          if ((a > b) == up) {
            buf[i] = b;
            buf[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    int o = buf[i];
    perm[s0 + i] = o;
    iperm[o] = s0 + i;
    cell_s[s0 + i] = c;
    type_s[s0 + i] = type[o];
  }
}

__global__ void k_mx_cellsort(const int *__restrict__ start, int *__restrict__ perm,
                              int *__restrict__ iperm, int *__restrict__ cell_s,
                              const int *__restrict__ type, int *__restrict__ type_s,
                              int *__restrict__ status) {
  k_mx_cellsort_body(vblk_self(), start, perm, iperm, cell_s, type, type_s, status);
}

// sorted fixed-point coordinates and charge; with `snap`, also the largest
// squared displacement of any site since the inner list was last pruned
__device__ __forceinline__ void k_mx_convert_body(VBlk vb_, int n, const double4 *__restrict__ pos, const int *__restrict__ perm,
                             double3 invL, int4 *__restrict__ posfx,
                             const int4 *__restrict__ snap, float3 sc,
                             unsigned *__restrict__ dmax2) {
  int s = vb_.id * blockDim.x + threadIdx.x;
  float d2 = 0.f;
  if (s < n) {
    int4 q = fx_site(pos[perm[s]], invL);
    posfx[s] = q;
    if (snap) d2 = fx_moved2(q, snap[s], sc);
  }
  if (snap) fx_moved_max(d2, dmax2);
}

// fix_zero (optional): the force sums to clear for the evaluation that follows
__global__ void k_mx_convert(int n, const double4 *__restrict__ pos, const int *__restrict__ perm,
                             double3 invL, int4 *__restrict__ posfx,
                             const int4 *__restrict__ snap, float3 sc,
                             unsigned *__restrict__ dmax2, unsigned long long *__restrict__ fix_zero) {
  if (fix_zero) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) {
      fix_zero[3 * s] = 0ull;
      fix_zero[3 * s + 1] = 0ull;
      fix_zero[3 * s + 2] = 0ull;
    }
  }
  k_mx_convert_body(vblk_self(), n, pos, perm, invL, posfx, snap, sc, dmax2);
}

__device__ __forceinline__ int mx_is_excluded(const int *__restrict__ xs, const int *__restrict__ xp,
                                              int a, int b) {
  for (int p = xs[a]; p < xs[a + 1]; p++)
    if (xp[p] == b) return 1;
  return 0;
}

// ---------------------------------------------------------------------------
// lists

// Entries of a row so far: LJ pairs at the front (ascending), the rest at the back
// (descending).
struct RowCursor {
  int nlj, nnl;
};

__device__ __forceinline__ void row_close(const RowCursor &rc, int cap, int s, int lane,
                                          int *__restrict__ cnt_lj, int *__restrict__ cnt_nl,
                                          int *__restrict__ status) {
  if (lane != 0) return;
  if (rc.nlj + rc.nnl > cap) {
    atomicOr(status, ST_LIST_OVERFLOW);
    int keep = min(rc.nlj, cap);
    cnt_lj[s] = keep;
    cnt_nl[s] = cap - keep;
  } else {
    cnt_lj[s] = rc.nlj;
    cnt_nl[s] = rc.nnl;
  }
}

// Consecutive sorted sites one warp lists together.  More share a candidate's
// load among them, fewer make enough warps in small boxes, where the build waits
// for its warps.  50 steps (five builds) in us with units of 1, 2, 4 and 8:
//    4,095 sites  2931  3190  3450  3979      13,500  4509  4436  4412  4613
//    6,000        3408  3529  3793  4252      28,500  6987  6702  6601  6608
//    9,000        3527  3523  3496  4178      36,000  7973  7660  7521  7598
constexpr int kListUnitMax = 8;
static int list_unit(long sites) { return sites >= 48000 ? 8 : sites >= 7500 ? 4 : 1; }
// cells per rlist along each axis: finer cells trim the candidates of a unit
// (rlist/2: ~3000 per unit of 8 water sites, rlist/3: ~2250), coarser ones
// make fewer, longer contiguous ranges; 3 measured fastest of 2, 3, 4
constexpr double kListCellsPerReach = 3.0;
constexpr int kListExcl = 4;  // excluded partners per site handled by lane masks
constexpr int kListBlocksPerSM = 3;  // register budget of the list build (no spills at 74)
static_assert(kListUnitMax * kListExcl == 32, "one lane per (site, excluded partner)");

__device__ __forceinline__ float warp_fmin(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_fmax(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int wrap_mod(int v, int g) {
  v %= g;
  return v < 0 ? v + g : v;
}

// gap between the interval [lo, hi] and cell c of edge h along one axis
__device__ __forceinline__ float cell_gap(int c, float h, float lo, float hi) {
  return fmaxf(fmaxf(c * h - hi, lo - (c + 1) * h), 0.f);
}

// Appends one chunk's passing candidates to a row without divergent branches.
__device__ __forceinline__ void row_push_bf(bool ok, bool lj, int entry, unsigned lt, int cap,
                                            int *__restrict__ row, RowCursor &rc) {
  unsigned mlj = __ballot_sync(0xffffffffu, ok && lj);
  unsigned mnl = __ballot_sync(0xffffffffu, ok && !lj);
  if ((mlj | mnl) == 0u) return;  // warp-uniform: nothing to append
  int p = lj ? rc.nlj + __popc(mlj & lt) : rc.nnl + __popc(mnl & lt);
  int other = lj ? rc.nnl : rc.nlj;
  int idx = lj ? p : cap - 1 - p;
  if (ok && p + other < cap) row[idx] = entry;
  rc.nlj += __popc(mlj);
  rc.nnl += __popc(mnl);
}

// One chunk of candidates (one per lane) against every site of the unit.
// FAST: the FP32 frame of the unit's first site covers every pair, the
// sites have at most kListExcl excluded partners and nt <= 32; otherwise
// the exact fixed-point differences, the exclusion lists and the type table
// are used.  Sites past the end of the unit carry NaN offsets: no pair passes.
template <bool FAST, int kListUnit>
__device__ __forceinline__ void list_chunk(
    int j, int js, int4 pj, float fjx, float fjy, float fjz, int tj, unsigned mj, unsigned ebit,
    unsigned lanebit, unsigned lt, const float4 (&site)[kListUnit], const int4 (&spk)[kListUnit],
    float3 sc, float rl2, int nt, const unsigned char *__restrict__ lj_on,
    const int *__restrict__ xs, const int *__restrict__ xp, int ok_orig, int oj, int cap,
    int *__restrict__ row0, RowCursor (&rc)[kListUnit]) {
#pragma unroll
  for (int k = 0; k < kListUnit; k++) {
    unsigned exm = __shfl_sync(0xffffffffu, ebit, 4 * k);
    float4 si = site[k];
    int tik = __float_as_int(si.w);
    float dx, dy, dz;
    if (FAST) {
      dx = fjx - si.x;
      dy = fjy - si.y;
      dz = fjz - si.z;
    } else {
      int4 pik = spk[k];
      dx = fx_delta((unsigned)pj.x, (unsigned)pik.x, sc.x);
      dy = fx_delta((unsigned)pj.y, (unsigned)pik.y, sc.y);
      dz = fx_delta((unsigned)pj.z, (unsigned)pik.z, sc.z);
      if (si.x != si.x) dx = si.x;  // padding site
    }
    float r2 = dx * dx + dy * dy + dz * dz;
    bool ok = r2 < rl2 && js != k && (exm & lanebit) == 0u;
    bool lj;
    if (FAST) {
      lj = ((mj >> tik) & 1u) != 0u;
    } else {
      int oi = __shfl_sync(0xffffffffu, ok_orig, k);
      if (ok) ok = !mx_is_excluded(xs, xp, oi, oj);
      lj = lj_on[tik * nt + tj] != 0;
    }
    row_push_bf(ok, lj, j, lt, cap, row0 + (size_t)k * cap, rc[k]);
  }
}

// Outer list: one warp per UNIT of kListUnit consecutive sorted sites (mostly
// one or two neighbouring cells).  The warp takes the bounding box of the
// unit's sites (minimum-image offsets from its first site, in A), walks the
// cell columns within reach of it -- 32 columns at a time, one per lane, each
// with the z cells within rlist of the box as one or two contiguous sorted
// ranges -- and packs those ranges into full 32-lane chunks of candidates.
// Every candidate is loaded once and tested against all sites of the unit.
// Excluded partners are turned into per-chunk lane masks (lane 4k+q owns the
// q-th partner of site k and locates it among the candidates once per column
// batch), so the per-pair test is a distance, a mask bit and a ballot.
// Rows come out in a fixed (column, slot) order: deterministic.
template <int kListUnit>
__device__ __forceinline__ void k_mx_list_body(VBlk vb_, int n, const int4 *__restrict__ posfx, const int *__restrict__ perm,
          const int *__restrict__ iperm, const int *__restrict__ cell_s,
          const int *__restrict__ type_s, const int *__restrict__ cstart, int3 nc, float3 sc,
          float3 Lf, float rlist, int nt, const unsigned *__restrict__ lj_row,
          const unsigned char *__restrict__ lj_on, const int *__restrict__ xs,
          const int *__restrict__ xp, int cap, int *__restrict__ cnt_lj,
          int *__restrict__ cnt_nl, int *__restrict__ ent, int *__restrict__ status) {
  const unsigned full = 0xffffffffu;
  __shared__ float4 s_site[kMxWarps][kListUnit];
  __shared__ int4 s_pk[kMxWarps][kListUnit];
  int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  unsigned lanebit = 1u << lane, lt = lanebit - 1u;
  float rl2 = rlist * rlist;
  // reach of the cell walk: rlist plus a margin for the FP32 frame's rounding
  float ra = rlist + 1e-3f + 4e-6f * fmaxf(Lf.x, fmaxf(Lf.y, Lf.z));
  float ra2 = ra * ra;
  float3 hc = make_float3(Lf.x / nc.x, Lf.y / nc.y, Lf.z / nc.z);
  float3 ihc = make_float3(nc.x / Lf.x, nc.y / Lf.y, nc.z / Lf.z);
  int nunits = (n + kListUnit - 1) / kListUnit;
  for (int u = vb_.id * kMxWarps + wib; u < nunits; u += vb_.n * kMxWarps) {
    int s0 = u * kListUnit, nk = min(kListUnit, n - s0);
    int sl = s0 + min(lane, nk - 1);  // lanes past the unit repeat its last site
    int4 pk = posfx[sl];
    int tk = type_s[sl];
    int ok_orig = perm[sl];
    unsigned r0x = __shfl_sync(full, (unsigned)pk.x, 0), r0y = __shfl_sync(full, (unsigned)pk.y, 0),
             r0z = __shfl_sync(full, (unsigned)pk.z, 0);
    float ox = fx_delta((unsigned)pk.x, r0x, sc.x), oy = fx_delta((unsigned)pk.y, r0y, sc.y),
          oz = fx_delta((unsigned)pk.z, r0z, sc.z);
    float lox = warp_fmin(ox), hix = warp_fmax(ox), loy = warp_fmin(oy), hiy = warp_fmax(oy),
          loz = warp_fmin(oz), hiz = warp_fmax(oz);
    // the FP32 frame of the first site gives the minimum image of every pair
    // within reach when offsets + reach stay under half the box
    bool frame = fmaxf(-lox, hix) + ra < 0.5f * Lf.x && fmaxf(-loy, hiy) + ra < 0.5f * Lf.y &&
                 fmaxf(-loz, hiz) + ra < 0.5f * Lf.z;
    // the unit's sites for the per-pair tests: offsets and type, and the
    // fixed-point coordinates for units the FP32 frame does not cover
    __syncwarp();
    if (lane < kListUnit) {
      float pad = lane < nk ? 0.f : __int_as_float(0x7fc00000);  // NaN: no pair passes
      s_site[wib][lane] = make_float4(ox + pad, oy + pad, oz + pad, __int_as_float(tk));
      s_pk[wib][lane] = pk;
    }
    __syncwarp();
    // lane 4k+q: q-th excluded partner of site k (sorted slot, -1 if none)
    int ek = lane >> 2, eq = lane & 3, exs = -1;
    bool many_l = false;
    if (ek < nk) {
      int o = perm[s0 + ek];
      int a = xs[o], m = xs[o + 1] - a;
      if (eq < m) exs = iperm[xp[a + eq]];
      many_l = eq == 0 && m > kListExcl;
    }
    bool fast = frame && lj_row != nullptr && !__any_sync(full, many_l);
    int *row0 = ent + (size_t)s0 * cap;
    int ecx = 0, ecy = 0;
    if (exs >= 0) {
      int c = cell_s[exs];
      ecy = (c / nc.z) % nc.y;
      ecx = c / (nc.z * nc.y);
    }
    // cell window of the unit, unwrapped (the whole axis when it wraps onto itself)
    float X0 = __uint2float_rn(r0x) * sc.x, Y0 = __uint2float_rn(r0y) * sc.y,
          Z0 = __uint2float_rn(r0z) * sc.z;
    float Xlo = X0 + lox, Xhi = X0 + hix, Ylo = Y0 + loy, Yhi = Y0 + hiy, Zlo = Z0 + loz,
          Zhi = Z0 + hiz;
    int xa = __float2int_rd((Xlo - ra) * ihc.x), xb = __float2int_rd((Xhi + ra) * ihc.x);
    int ya = __float2int_rd((Ylo - ra) * ihc.y), yb = __float2int_rd((Yhi + ra) * ihc.y);
    bool allx = xb - xa + 1 >= nc.x, ally = yb - ya + 1 >= nc.y;
    if (allx) {
      xa = 0;
      xb = nc.x - 1;
    }
    if (ally) {
      ya = 0;
      yb = nc.y - 1;
    }
    int nx = xb - xa + 1, ny = yb - ya + 1, ncol = nx * ny;
    // column of the excluded partner within the window (-1: outside)
    int eqcol = -1;
    if (exs >= 0) {
      int dx = wrap_mod(ecx - xa, nc.x), dy = wrap_mod(ecy - ya, nc.y);
      if (dx < nx && dy < ny) eqcol = dx * ny + dy;
    }
    RowCursor rc[kListUnit];
#pragma unroll
    for (int k = 0; k < kListUnit; k++) rc[k] = {0, 0};
    for (int q0 = 0; q0 < ncol; q0 += 32) {
      int q = q0 + lane;
      int a0 = 0, la = 0, b0 = 0, lb = 0;
      if (q < ncol) {
        int x = xa + q / ny, y = ya + q % ny;
        float gx = allx ? 0.f : cell_gap(x, hc.x, Xlo, Xhi);
        float gy = ally ? 0.f : cell_gap(y, hc.y, Ylo, Yhi);
        float g2 = gx * gx + gy * gy;
        if (g2 < ra2) {
          float rho = sqrtf(ra2 - g2);
          int za = __float2int_rd((Zlo - rho) * ihc.z), zb = __float2int_rd((Zhi + rho) * ihc.z);
          const int *cs = cstart + (wrap_mod(x, nc.x) * nc.y + wrap_mod(y, nc.y)) * nc.z;
          if (zb - za + 1 >= nc.z) {
            a0 = cs[0];
            la = cs[nc.z] - a0;
          } else {
            int zaw = wrap_mod(za, nc.z), zbw = wrap_mod(zb, nc.z);
            a0 = cs[zaw];
            if (zaw <= zbw) {
              la = cs[zbw + 1] - a0;
            } else {
              la = cs[nc.z] - a0;
              b0 = cs[0];
              lb = cs[zbw + 1] - b0;
            }
          }
        }
      }
      // exclusive prefix of the columns' candidate counts
      int len = la + lb, incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += t;
      }
      int P = incl - len, T = __shfl_sync(full, incl, 31);
      // virtual index of this lane's excluded partner among the batch's candidates
      bool here = eqcol >= q0 && eqcol < q0 + 32;
      int src = here ? eqcol - q0 : 0;
      int eP = __shfl_sync(full, P, src), ea0 = __shfl_sync(full, a0, src),
          ela = __shfl_sync(full, la, src), eb0 = __shfl_sync(full, b0, src),
          elb = __shfl_sync(full, lb, src);
      int ve = -1;
      if (here) {
        if (exs >= ea0 && exs < ea0 + ela) ve = eP + exs - ea0;
        else if (exs >= eb0 && exs < eb0 + elb) ve = eP + ela + exs - eb0;
      }
      for (int vb = 0; vb < T; vb += 32) {
        int v = vb + lane;
        bool valid = v < T;
        int c = 0;
#pragma unroll
        for (int st = 16; st; st >>= 1) {
          int Pt = __shfl_sync(full, P, c + st);
          if (Pt <= v) c += st;
        }
        int Pc = __shfl_sync(full, P, c), a0c = __shfl_sync(full, a0, c),
            lac = __shfl_sync(full, la, c), b0c = __shfl_sync(full, b0, c);
        int off = v - Pc;
        int j = off < lac ? a0c + off : b0c + (off - lac);
        if (!valid) j = s0;
        int4 pj = posfx[j];
        int tj = type_s[j];
        float fjx = fx_delta((unsigned)pj.x, r0x, sc.x), fjy = fx_delta((unsigned)pj.y, r0y, sc.y),
              fjz = fx_delta((unsigned)pj.z, r0z, sc.z);
        unsigned te = (unsigned)(ve - vb);
        unsigned ebit = (ve >= 0 && te < 32u) ? 1u << te : 0u;
        ebit |= __shfl_xor_sync(full, ebit, 1);
        ebit |= __shfl_xor_sync(full, ebit, 2);
        int js = valid ? j - s0 : -1;  // this lane's candidate is site js of the unit
        if (fast) {
          list_chunk<true, kListUnit>(j, js, pj, fjx, fjy, fjz, tj, lj_row[tj], ebit, lanebit, lt,
                           s_site[wib], s_pk[wib], sc, valid ? rl2 : -1.f, nt, lj_on, xs, xp,
                           ok_orig, 0, cap, row0, rc);
        } else {
          list_chunk<false, kListUnit>(j, js, pj, fjx, fjy, fjz, tj, 0u, ebit, lanebit, lt, s_site[wib],
                            s_pk[wib], sc, valid ? rl2 : -1.f, nt, lj_on, xs, xp, ok_orig,
                            perm[j], cap, row0, rc);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kListUnit; k++)
      if (k < nk) row_close(rc[k], cap, s0 + k, lane - k, cnt_lj, cnt_nl, status);
  }
}

template <int kListUnit>
__global__ void __launch_bounds__(kMxWarps * 32, kListBlocksPerSM)
k_mx_list(int n, const int4 *__restrict__ posfx, const int *__restrict__ perm,
          const int *__restrict__ iperm, const int *__restrict__ cell_s,
          const int *__restrict__ type_s, const int *__restrict__ cstart, int3 nc, float3 sc,
          float3 Lf, float rlist, int nt, const unsigned *__restrict__ lj_row,
          const unsigned char *__restrict__ lj_on, const int *__restrict__ xs,
          const int *__restrict__ xp, int cap, int *__restrict__ cnt_lj,
          int *__restrict__ cnt_nl, int *__restrict__ ent, int *__restrict__ status) {
  k_mx_list_body<kListUnit>(vblk_self(), n, posfx, perm, iperm, cell_s, type_s, cstart, nc, sc, Lf, rlist, nt, lj_row, lj_on, xs, xp, cap, cnt_lj, cnt_nl, ent, status);
}


// ---------------------------------------------------------------------------
// pair kernel

// Warps resident per SM the pair kernel's registers (64) are sized for.
constexpr int kPairRW = 32;
// Rows a warp takes from the row counter at a time.  (Rows shared by two or four
// warps with a scalar walk, 48 resident, were faster in small boxes only than the
// same walk of whole rows; the packed walk of whole rows takes 46 us a step at
// 1,500 sites where they took 52, and 49 at 4,095 where they took 56.)
constexpr int kPairGrab = 2;
// Up to this many sites the outer list is walked every step.  The inner list's
// 27 % fewer entries save less there than its launches and pruning walks cost.
// 50 steps (five builds) in us, outer list and inner:
//    1,500 sites  2116  2236      8,100  3074  3162      12,000  4011  4015
//    4,095        2417  2633      9,000  3888  3478      18,000  5344  5142
//    6,000        2942  2996     10,500  4150  3585      36,000  7646  7190
constexpr int kInnerMinSites = 8192;

struct MxPair {
  int n, nt, cap;
  float rc2, c2k, qfe;  // c2k = 2 kappa / sqrt(pi); qfe = QFACTOR / epsRF
  float khalf, mk2;  // kappa / 2, -kappa^2 log2 e
  float ron2, inv_sw_den;  // switch start^2 and 1 / (rc^2 - ron^2)^3
  float3 sc;                   // L / 2^32 per axis
  int cubic;                   // Lx = Ly = Lz: distances formed in lattice units
  float s2;                    // sc.x^2 (cubic boxes)
  // inner list: radius^2 (rc + skin)^2, and the squared displacement that
  // forces a prune ((skin / 2)^2, less a rounding margin)
  float rp2, thresh2;
  int inner_on;                // 0: rows always come from the outer list
};


// the reference's erfc (ewald.c:817-836, Numerical Recipes "erfcc") in FP32;
// ex = exp(-z^2) is shared with the force term
__device__ __forceinline__ float erfc_nr_f(float z, float ex) {
  float t = __fdividef(1.0f, 1.0f + 0.5f * z);
  float p = fmaf(t, 0.17087277f, -0.82215223f);
  p = fmaf(t, p, 1.48851587f);
  p = fmaf(t, p, -1.13520398f);
  p = fmaf(t, p, 0.27886807f);
  p = fmaf(t, p, -0.18628806f);
  p = fmaf(t, p, 0.09678418f);
  p = fmaf(t, p, 0.37409196f);
  p = fmaf(t, p, 1.00002368f);
  p = fmaf(t, p, -1.26551223f);
  return t * ex * __expf(p);
}

// 2^x by the SFU's ex2.approx (PTX ISA): the exponential of the pair terms
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kLog2e = 1.44269504f;

// Two FP32 values in a register pair: sm_100's packed instructions work on both
// at the issue cost of one.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32x2 pack2(float a) { return pack2(a, a); }
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  float2 r = unpack2(v);
  return r.x + r.y;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The same fit as erfc_nr_f of two values, erfc(z) = t exp(-z^2 + P(t)), with the
// two exponents merged: t 2^(P(t) log2 e + q2); den = 1 + z / 2 and
// q2 = -z^2 log2 e given.
__device__ __forceinline__ f32x2 erfc_nr_q2(f32x2 den, f32x2 q2) {
  float2 d = unpack2(den);
  f32x2 t = pack2(rcp_approx(d.x), rcp_approx(d.y));
  f32x2 p = fma2(t, pack2(0.17087277f), pack2(-0.82215223f));
  p = fma2(t, p, pack2(1.48851587f));
  p = fma2(t, p, pack2(-1.13520398f));
  p = fma2(t, p, pack2(0.27886807f));
  p = fma2(t, p, pack2(-0.18628806f));
  p = fma2(t, p, pack2(0.09678418f));
  p = fma2(t, p, pack2(0.37409196f));
  p = fma2(t, p, pack2(1.00002368f));
  p = fma2(t, p, pack2(-1.26551223f));
  float2 x = unpack2(fma2(p, pack2(kLog2e), q2));
  return mul2(t, pack2(ex2_approx(x.x), ex2_approx(x.y)));
}

// a row's sums, each over the even and the odd entries
struct PairAcc {
  f32x2 fx, fy, fz, e_lj, e_ljs, e_real, qsum;
};

// two list entries of a row
struct PairTwo {
  f32x2 dx, dy, dz;  // separations: A, or (CUBIC) lattice units of L / 2^32
  float qa, qb;      // the entries' charges
  int ja, jb;        // sorted slots (the LJ types)
};

template <bool CUBIC>
__device__ __forceinline__ f32x2 mx_sep(unsigned i, unsigned a, unsigned b, float sc) {
  f32x2 d = pack2(__int2float_rn((int)(i - a)), __int2float_rn((int)(i - b)));
  return CUBIC ? d : mul2(d, pack2(sc));
}

// the LJ switch between ron and rc, on a pair's force and energy
__device__ __forceinline__ void mx_switch(const MxPair &P, float r2, float &f, float &e) {
  if (r2 > P.ron2) {
    float c = P.rc2 - r2;
    float sw = c * c * (P.rc2 + 2.f * r2 - 3.f * P.ron2) * P.inv_sw_den;
    float dsw = 12.f * c * (r2 - P.ron2) * P.inv_sw_den;
    f = f * sw + e * dsw;
    e = e * sw;
  }
}

// Two pairs at once: Ewald real space always, LJ when WITH_LJ.  A pair beyond the cutoff gets zero charge
// and LJ strength, an entry past the row's end (MASK: va, vb) a distance beyond
// the cutoff.  Returns the squared distances.
template <bool WITH_LJ, bool CUBIC, bool MASK>
__device__ __forceinline__ float2 mx_pair_two(const MxPair &P, float qi, const PairTwo &T, bool va,
                                              bool vb, const float *__restrict__ ljrow,
                                              const int *__restrict__ type_s, PairAcc &a) {
  f32x2 r2 = fma2(T.dx, T.dx, fma2(T.dy, T.dy, mul2(T.dz, T.dz)));
  if (CUBIC) r2 = mul2(pack2(P.s2), r2);
  float2 d = unpack2(r2);
  if (MASK) {
    if (!va) d.x = 4.f * P.rc2;
    if (!vb) d.y = 4.f * P.rc2;
    r2 = pack2(d.x, d.y);
  }
  const bool oa = d.x > P.rc2, ob = d.y > P.rc2;
  const f32x2 rinv = pack2(rsqrt_approx(d.x), rsqrt_approx(d.y));
  const f32x2 r = mul2(r2, rinv), rinv2 = mul2(rinv, rinv);
  const f32x2 qq = pack2(oa ? 0.f : qi * T.qa, ob ? 0.f : qi * T.qb);
  const f32x2 q2 = mul2(r2, pack2(P.mk2));
  const float2 q2s = unpack2(q2);
  const f32x2 ex = pack2(ex2_approx(q2s.x), ex2_approx(q2s.y));  // exp(-(kappa r)^2)
  const f32x2 erfckr = erfc_nr_q2(fma2(pack2(P.khalf), r, pack2(1.f)), q2);
  const f32x2 qr = mul2(qq, rinv);
  f32x2 F = mul2(mul2(qr, rinv2), fma2(mul2(pack2(P.c2k), r), ex, erfckr));
  a.e_real = fma2(qr, erfckr, a.e_real);
  a.qsum = add2(a.qsum, qq);
  if (WITH_LJ) {
    const float *la = ljrow + type_s[T.ja] * 3, *lb = ljrow + type_s[T.jb] * 3;
    const f32x2 eps = pack2(oa ? 0.f : la[0], ob ? 0.f : lb[0]);
    const f32x2 sr2 = mul2(pack2(la[1], lb[1]), rinv2);
    const f32x2 sr6 = mul2(mul2(sr2, sr2), sr2);
    const f32x2 sr12 = mul2(sr6, sr6);
    f32x2 flj = mul2(mul2(mul2(pack2(12.f), eps), rinv2), fma2(sr6, pack2(-1.f), sr12));
    f32x2 elj = mul2(eps, fma2(pack2(-2.f), sr6, sr12));
    if (P.ron2 > 0.f) {
      float2 f = unpack2(flj), e = unpack2(elj);
      mx_switch(P, d.x, f.x, e.x);
      mx_switch(P, d.y, f.y, e.y);
      flj = pack2(f.x, f.y);
      elj = pack2(e.x, e.y);
    } else {
      a.e_ljs = fma2(eps, pack2(la[2], lb[2]), a.e_ljs);
    }
    F = add2(F, flj);
    a.e_lj = add2(a.e_lj, elj);
  }
  a.fx = fma2(F, T.dx, a.fx);
  a.fy = fma2(F, T.dy, a.fy);
  a.fz = fma2(F, T.dz, a.fz);
  return d;
}

// appends one entry per lane (where ok) to an inner row
template <bool LJ>
__device__ __forceinline__ void inner_push(bool ok, int entry, unsigned lt, int cap,
                                           int *__restrict__ row, RowCursor &rc) {
  const unsigned m = __ballot_sync(0xffffffffu, ok);
  const int k = (LJ ? rc.nlj : rc.nnl) + __popc(m & lt), other = LJ ? rc.nnl : rc.nlj;
  if (ok && k + other < cap) row[LJ ? k : cap - 1 - k] = entry;
  if (LJ) rc.nlj += __popc(m);
  else rc.nnl += __popc(m);
}

// Walks a row's entries [b0, b1), two a lane at a time with packed
// arithmetic.  The scalar walk is bound by instruction issue (146 M instructions
// at 96,000 sites); this one takes 97 M and waits for its loads.  The next two
// entries' positions are requested once the current ones are spent and the two
// entries after with them, so both are in flight behind the arithmetic.  Staging
// positions in shared memory two iterations ahead waits less but takes 143 M
// instructions, and rows dealt to blocks in runs (L1 hits 77 % of the gathers,
// not 41 %) spill: both were slower.  96,000 sites: 358 us a step with the scalar
// walk, 320 with this one.
//
// PRUNE: also writes the inner row; entries within rc + skin are appended to
// `irow` (same LJ-front / rest-back layout, same order).
template <bool WITH_LJ, bool CUBIC, bool PRUNE>
__device__ __forceinline__ void mx_segment(const MxPair &P, int4 pi, float qi,
                                            const int *__restrict__ row, int b0, int b1, int lane,
                                            const int4 *__restrict__ posfx,
                                            const float *__restrict__ ljrow,
                                            const int *__restrict__ type_s, int self, unsigned lt,
                                            int *__restrict__ irow, RowCursor &rc, PairAcc &a) {
  if (b0 >= b1) return;  // the same for all lanes
  int i = b0 + lane;
  auto entry = [&](int k) { return k < b1 ? row[k] : self; };
  PairTwo T;
  T.ja = entry(i);
  T.jb = entry(i + 32);
  int4 pa = posfx[T.ja], pb = posfx[T.jb];
  int na = entry(i + 64), nb = entry(i + 96);
  while (true) {
    T.dx = mx_sep<CUBIC>((unsigned)pi.x, (unsigned)pa.x, (unsigned)pb.x, P.sc.x);
    T.dy = mx_sep<CUBIC>((unsigned)pi.y, (unsigned)pa.y, (unsigned)pb.y, P.sc.y);
    T.dz = mx_sep<CUBIC>((unsigned)pi.z, (unsigned)pa.z, (unsigned)pb.z, P.sc.z);
    T.qa = __int_as_float(pa.w);
    T.qb = __int_as_float(pb.w);
    if (b0 + 64 > b1) {  // the last, partial one
      const bool va = i < b1, vb = i + 32 < b1;
      float2 d = mx_pair_two<WITH_LJ, CUBIC, true>(P, qi, T, va, vb, ljrow, type_s, a);
      if (PRUNE) {
        inner_push<WITH_LJ>(va && d.x < P.rp2, T.ja, lt, P.cap, irow, rc);
        inner_push<WITH_LJ>(vb && d.y < P.rp2, T.jb, lt, P.cap, irow, rc);
      }
      return;
    }
    pa = posfx[na];
    pb = posfx[nb];
    const int ma = entry(i + 128), mb = entry(i + 160);
    float2 d = mx_pair_two<WITH_LJ, CUBIC, false>(P, qi, T, true, true, ljrow, type_s, a);
    if (PRUNE) {
      inner_push<WITH_LJ>(d.x < P.rp2, T.ja, lt, P.cap, irow, rc);
      inner_push<WITH_LJ>(d.y < P.rp2, T.jb, lt, P.cap, irow, rc);
    }
    b0 += 64;
    if (b0 >= b1) return;
    i += 64;
    T.ja = na;
    T.jb = nb;
    na = ma;
    nb = mb;
  }
}

// NW warps per block: a launch shape chosen by mixed_autotune.
// With an inner list two variants run one after the other every evaluation and
// read the same device state.  PRUNE walks the outer rows, rewrites the inner ones and
// adds its block sums to the energy accumulators; it returns at once when no
// prune is due.  The plain variant walks the inner rows (nothing when the
// PRUNE variant ran), finishes the energies and clears the state.  Without
// one (P.inner_on 0) the plain variant alone walks the outer rows; `need` then
// stays set, so that a later evaluation with an inner list prunes first.
template <int NW, bool PRUNE>
__device__ __forceinline__ void k_mx_pair_body(VBlk vb_, MxPair P, const int4 *__restrict__ posfx, const int *__restrict__ type_s,
          const int *__restrict__ perm, const int *__restrict__ cnt_lj,
          const int *__restrict__ cnt_nl, const int *__restrict__ ent,
          int *__restrict__ icnt_lj, int *__restrict__ icnt_nl, int *__restrict__ ient,
          int4 *__restrict__ snap, MxPruneState *__restrict__ ps,
          const float *__restrict__ lj_tab, unsigned long long *__restrict__ fix,
          unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
          double *__restrict__ out, int *__restrict__ status) {
  // prune (read the outer list, rewrite the inner one) after a list rebuild
  // or when some site has moved half the skin since the last prune; between
  // prunes no pair can come within rc from beyond rc + skin
  const bool due =
      P.inner_on && (ps->need != 0 || __uint_as_float(ps->dmax2) >= P.thresh2);
  if (PRUNE && !due) return;
  const bool work = PRUNE || !due;
  extern __shared__ float s_lj[];  // nt*nt*3: eps, sig^2, shift constant
  for (int i = threadIdx.x; i < P.nt * P.nt * 3; i += blockDim.x) s_lj[i] = lj_tab[i];
  __syncthreads();
  int lane = threadIdx.x & 31;
  unsigned lt = (1u << lane) - 1u;
  if (PRUNE && vb_.id == 0 && threadIdx.x == 0) atomicAdd(&ps->prunes, 1ull);
  const bool outer = PRUNE || !P.inner_on;
  const int *rlj = outer ? cnt_lj : icnt_lj;
  const int *rnl = outer ? cnt_nl : icnt_nl;
  const int *rent = outer ? ent : ient;
  // energies per row in FP32, then exact fixed-point sums across rows (kept in
  // shared memory): the totals do not depend on how rows are spread over warps
  // (the launch shape)
  __shared__ long long weq[NW][4];
  if (lane < 4) weq[threadIdx.x >> 5][lane] = 0;
  __syncwarp();
  // rows are taken kPairGrab at a time from a device counter: warps finish
  // together whatever their rows' lengths (the per-row energies are exact
  // fixed-point sums, so the results do not depend on which warp took a row)
  while (work) {
    int s0 = 0;
    if (lane == 0) s0 = atomicAdd(&ps->next_row, kPairGrab);
    s0 = __shfl_sync(0xffffffffu, s0, 0);
    if (s0 >= P.n) break;
    const int s1 = min(s0 + kPairGrab, P.n);
    for (int s = s0; s < s1; s++) {
      int4 pi = posfx[s];
      float qi = __int_as_float(pi.w) * P.qfe;
      const float *ljrow = s_lj + type_s[s] * P.nt * 3;
      const int *row = rent + (size_t)s * P.cap;
      const int nlj = rlj[s], nl0 = P.cap - rnl[s];
      float v[8];
      v[7] = 0.f;
      PairAcc a = {0, 0, 0, 0, 0, 0, 0};  // 0.f twice
      RowCursor rc = {0, 0};
      int *irow = PRUNE ? ient + (size_t)s * P.cap : nullptr;
      // The list streams from HBM: a row that some warp takes about one row's
      // time from now goes to L2 (16 lines of its back part and 16 of its front,
      // as far as this row's reach).  At 96,000 sites a step takes 308 us with
      // it, 320 without.
      const int ahead = s + vb_.n * NW;
      if (ahead < P.n) {
        const int k = lane < 16 ? nl0 + 32 * lane : 32 * (lane - 16);
        if (k < (lane < 16 ? P.cap : nlj))
          asm volatile("prefetch.global.L2 [%0];" ::"l"(rent + (size_t)ahead * P.cap + k));
      }
      if (P.cubic) {
        mx_segment<true, true, PRUNE>(P, pi, qi, row, 0, nlj, lane, posfx, ljrow, type_s, s, lt,
                                       irow, rc, a);
        mx_segment<false, true, PRUNE>(P, pi, qi, row, nl0, P.cap, lane, posfx, ljrow, type_s, s,
                                        lt, irow, rc, a);
      } else {
        mx_segment<true, false, PRUNE>(P, pi, qi, row, 0, nlj, lane, posfx, ljrow, type_s, s, lt,
                                        irow, rc, a);
        mx_segment<false, false, PRUNE>(P, pi, qi, row, nl0, P.cap, lane, posfx, ljrow, type_s, s,
                                         lt, irow, rc, a);
      }
      if (PRUNE) {
        row_close(rc, P.cap, s, lane, icnt_lj, icnt_nl, status);
        if (lane == 0) snap[s] = pi;
      }
      v[0] = sum2(a.fx);
      v[1] = sum2(a.fy);
      v[2] = sum2(a.fz);
      v[3] = sum2(a.e_lj);
      v[4] = sum2(a.e_ljs);
      v[5] = sum2(a.e_real);
      v[6] = sum2(a.qsum);
      // the row's sums in a fixed order of FP32 partial sums (deterministic),
      // each converted once to fixed point: halving exchanges leave the t-th on
      // lanes 4 t .. 4 t + 3, so one conversion serves all seven
#pragma unroll
      for (int h = 4; h > 0; h >>= 1) {
        const bool up = (lane & (4 * h)) != 0;
#pragma unroll
        for (int k = 0; k < h; k++)
          v[k] = (up ? v[k + h] : v[k]) +
                 __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + h], 4 * h);
      }
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
      const int t = lane >> 2;
      if ((lane & 3) == 0 && t < 7) {
        // lattice units to A; every pair is visited from both ends: half of each
        // row's energy
        const long long q = to_fix(v[0] * (t >= 3 ? 0.5f : P.cubic ? P.sc.x : 1.f));
        if (t < 3) atomicAdd(&fix[3 * perm[s] + t], (unsigned long long)q);
        else weq[threadIdx.x >> 5][t - 3] += q;
      }
    }
  }
  __syncwarp();
  long long eq[4] = {0, 0, 0, 0};
  if (lane == 0)
#pragma unroll
    for (int t = 0; t < 4; t++) eq[t] = weq[threadIdx.x >> 5][t];
  if (PRUNE) {
    block_fix_add<4>(eq, 32, facc);
    return;
  }
  // the last block: both variants have read the prune state and every row
  // has been taken, clear both
  if (block_fix_final<4>(eq, 32, facc, ticket, out, vb_) && threadIdx.x == 0) {
    if (P.inner_on) ps->need = 0;
    ps->dmax2 = 0u;
    ps->next_row = 0;
  }
}

template <int NW, bool PRUNE>
__global__ void __launch_bounds__(NW * 32, kPairRW / NW)
k_mx_pair(MxPair P, const int4 *__restrict__ posfx, const int *__restrict__ type_s,
          const int *__restrict__ perm, const int *__restrict__ cnt_lj,
          const int *__restrict__ cnt_nl, const int *__restrict__ ent,
          int *__restrict__ icnt_lj, int *__restrict__ icnt_nl, int *__restrict__ ient,
          int4 *__restrict__ snap, MxPruneState *__restrict__ ps,
          const float *__restrict__ lj_tab, unsigned long long *__restrict__ fix,
          unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
          double *__restrict__ out, int *__restrict__ status) {
  k_mx_pair_body<NW, PRUNE>(vblk_self(), P, posfx, type_s, perm, cnt_lj, cnt_nl, ent, icnt_lj, icnt_nl, ient, snap, ps, lj_tab, fix, facc, ticket, out, status);
}

// qq (1 - erfc(kappa r)) / r of an excluded pair in double-float, from the
// exact integer separation of the 32-bit fractional coordinates and the FP64
// charges (the term eewald_intra of cnonbond_nblist.c:416-437)
__device__ __forceinline__ dfl intra_energy_df(const DfIntra &D, int4 A, int4 B, double qa,
                                               double qb, float qscale,
                                               const float2 *__restrict__ exptab) {
  dfl r2 = {0.f, 0.f};
  int dd[3] = {(int)((unsigned)A.x - (unsigned)B.x), (int)((unsigned)A.y - (unsigned)B.y),
               (int)((unsigned)A.z - (unsigned)B.z)};
#pragma unroll
  for (int c = 0; c < 3; c++) {
    dfl d = df_mul(df_from_ll((long long)dd[c]), {D.sl[c].x, D.sl[c].y});
    r2 = df_add(r2, df_mul(d, d));
  }
  dfl r = df_sqrt(r2);
  dfl z = df_mul(r, {D.kappa.x, D.kappa.y});
  dfl erf = df_add({1.0f, 0.0f}, df_neg(df_erfc_nr(z, D.C, exptab)));
  dfl qq = df_mul(df_mul(df_from_double(qa), df_from_double(qb)), {D.qf.x, D.qf.y});
  qq = df_mul_f(qq, qscale);
  return df_mul(df_mul(qq, erf), df_recip(r));
}

__device__ __forceinline__ long long df_to_fixed(dfl v, int shift) {
  return to_fixed(v.hi, shift) + to_fixed(v.lo, shift);
}

// excluded and 1-4 pairs (xint), cnonbond_nblist.c:245-263 and 416-437:
// inside rc an excluded pair contributes no LJ and no real-space term but the
// intra correction -qq (1 - erfc(kr)) / r; a 1-4 pair gets LJ, real space
// scaled by E14FAC and the correction with (1 - E14FAC)
__global__ void k_mx_excl(int nexcl, const int *__restrict__ ab, const int *__restrict__ flag,
                          const int4 *__restrict__ posfx, const int *__restrict__ iperm,
                          const int *__restrict__ type, float3 sL, int nt, const float *__restrict__ lj_tab, float rc2, float kappa,
                          float c2k, float qf, float epsRF, const double4 *__restrict__ pos_q,
                          const float2 *__restrict__ exptab, DfIntra D,
                          unsigned long long *__restrict__ fix,
                          unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                          double *__restrict__ out) {
  float e_lj = 0.f, e_ljs = 0.f, e_real = 0.f, qsum = 0.f;
  long long q_intra = 0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nexcl; t += gridDim.x * blockDim.x) {
    int a = ab[2 * t], b = ab[2 * t + 1], xf = flag[t];
    if (xf == 0) continue;
    int4 A = posfx[iperm[a]], B = posfx[iperm[b]];
    float dx = fx_delta((unsigned)A.x, (unsigned)B.x, sL.x);
    float dy = fx_delta((unsigned)A.y, (unsigned)B.y, sL.y);
    float dz = fx_delta((unsigned)A.z, (unsigned)B.z, sL.z);
    float r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > rc2) continue;
    float rinv = rsqrtf(r2), r = r2 * rinv, rinv2 = rinv * rinv;
    float kr = kappa * r;
    float ex = __expf(-kr * kr);
    float erfckr = erfc_nr_f(kr, ex);
    float qqab = __int_as_float(A.w) * __int_as_float(B.w) * qf;
    float F = 0.f;
    float qcorr = qqab;
    if (xf == 4) {
      float qq = qqab * (float)kE14FAC / epsRF;
      F += qq * rinv * rinv2 * (erfckr + c2k * r * ex);
      e_real += qq * erfckr * rinv;
      qsum += qq;
      const float *lj = lj_tab + (type[a] * nt + type[b]) * 3;
      if (lj[0] != 0.f) {
        float sr2 = lj[1] * rinv2, sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6;
        F += 12.f * lj[0] * rinv2 * (sr12 - sr6);
        e_lj += lj[0] * (sr12 - 2.f * sr6);
        e_ljs += lj[0] * lj[2];
      }
      qcorr *= (1.f - (float)kE14FAC);
    }
    float erfkr = 1.f - erfckr;
    q_intra += df_to_fixed(intra_energy_df(D, A, B, pos_q[a].w, pos_q[b].w,
                                           xf == 4 ? (float)(1.0 - kE14FAC) : 1.f, exptab),
                           32);
    F -= qcorr * rinv * rinv2 * (erfkr - c2k * r * ex);
    long long fxq = to_fix(F * dx), fyq = to_fix(F * dy), fzq = to_fix(F * dz);
    atomicAdd(&fix[3 * a], (unsigned long long)fxq);
    atomicAdd(&fix[3 * a + 1], (unsigned long long)fyq);
    atomicAdd(&fix[3 * a + 2], (unsigned long long)fzq);
    atomicAdd(&fix[3 * b], (unsigned long long)(-fxq));
    atomicAdd(&fix[3 * b + 1], (unsigned long long)(-fyq));
    atomicAdd(&fix[3 * b + 2], (unsigned long long)(-fzq));
  }
  long long v[5] = {to_fixed(e_lj, 32), to_fixed(e_ljs, 32), to_fixed(e_real, 32),
                    to_fixed(qsum, 32), q_intra};
  block_fix_final<5>(v, 32, facc, ticket, out);
}

// bonded terms from the fixed-point coordinates (cbond.c, cbend.c): the
// stretch, the angle and the energies in FP64 as in intra_bond / intra_bend,
// the forces in FP32 (sd: the length scale L / 2^32 in FP64)
__global__ void k_mx_bonded(int nbond, int nbend, float3 sL, double3 sd,
                            const int4 *__restrict__ posfx,
                            const int *__restrict__ iperm,
                            const int *__restrict__ bond_ab, const double *__restrict__ bond_req,
                            const double *__restrict__ bond_k, const int *__restrict__ bend_abc,
                            const double *__restrict__ bend_t0, const double *__restrict__ bend_k,
                            unsigned long long *__restrict__ fix,
                            unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                            double *__restrict__ out) {
  double eb = 0.0, ea = 0.0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nbond + nbend;
       t += gridDim.x * blockDim.x) {
    if (t < nbond) {
      int ia = bond_ab[2 * t], ib = bond_ab[2 * t + 1];
      int4 A = posfx[iperm[ia]], B = posfx[iperm[ib]];
      float dx = fx_delta((unsigned)B.x, (unsigned)A.x, sL.x);
      float dy = fx_delta((unsigned)B.y, (unsigned)A.y, sL.y);
      float dz = fx_delta((unsigned)B.z, (unsigned)A.z, sL.z);
      float dr = sqrtf(dx * dx + dy * dy + dz * dz);
      const double ex = fx_delta_d((unsigned)B.x, (unsigned)A.x, sd.x);
      const double ey = fx_delta_d((unsigned)B.y, (unsigned)A.y, sd.y);
      const double ez = fx_delta_d((unsigned)B.z, (unsigned)A.z, sd.z);
      const double rrd = sqrt(ex * ex + ey * ey + ez * ez) - bond_req[t];
      eb += bond_k[t] * rrd * rrd;
      float fr = -(float)bond_k[t] * (float)rrd * 2.f;
      float s = fr / dr;
      long long fxq = to_fix(s * dx), fyq = to_fix(s * dy), fzq = to_fix(s * dz);
      atomicAdd(&fix[3 * ia], (unsigned long long)(-fxq));
      atomicAdd(&fix[3 * ia + 1], (unsigned long long)(-fyq));
      atomicAdd(&fix[3 * ia + 2], (unsigned long long)(-fzq));
      atomicAdd(&fix[3 * ib], (unsigned long long)fxq);
      atomicAdd(&fix[3 * ib + 1], (unsigned long long)fyq);
      atomicAdd(&fix[3 * ib + 2], (unsigned long long)fzq);
    } else {
      int u = t - nbond;
      int ia = bend_abc[3 * u], ib = bend_abc[3 * u + 1], ic = bend_abc[3 * u + 2];
      int4 A = posfx[iperm[ia]], B = posfx[iperm[ib]], Cc = posfx[iperm[ic]];
      float dax = fx_delta((unsigned)A.x, (unsigned)B.x, sL.x);
      float day = fx_delta((unsigned)A.y, (unsigned)B.y, sL.y);
      float daz = fx_delta((unsigned)A.z, (unsigned)B.z, sL.z);
      float dcx = fx_delta((unsigned)Cc.x, (unsigned)B.x, sL.x);
      float dcy = fx_delta((unsigned)Cc.y, (unsigned)B.y, sL.y);
      float dcz = fx_delta((unsigned)Cc.z, (unsigned)B.z, sL.z);
      float drai = rsqrtf(dax * dax + day * day + daz * daz);
      float erax = dax * drai, eray = day * drai, eraz = daz * drai;
      float drci = rsqrtf(dcx * dcx + dcy * dcy + dcz * dcz);
      float ercx = dcx * drci, ercy = dcy * drci, ercz = dcz * drci;
      const double pax = fx_delta_d((unsigned)A.x, (unsigned)B.x, sd.x);
      const double pay = fx_delta_d((unsigned)A.y, (unsigned)B.y, sd.y);
      const double paz = fx_delta_d((unsigned)A.z, (unsigned)B.z, sd.z);
      const double pcx = fx_delta_d((unsigned)Cc.x, (unsigned)B.x, sd.x);
      const double pcy = fx_delta_d((unsigned)Cc.y, (unsigned)B.y, sd.y);
      const double pcz = fx_delta_d((unsigned)Cc.z, (unsigned)B.z, sd.z);
      double cosd = (pax * pcx + pay * pcy + paz * pcz) /
                    sqrt((pax * pax + pay * pay + paz * paz) * (pcx * pcx + pcy * pcy + pcz * pcz));
      cosd = fmin(fmax(cosd, -1.0), 1.0);
      const double rrd = acos(cosd) - bend_t0[u];
      ea += bend_k[u] * rrd * rrd;
      float cosphi = (float)cosd;
      float isinphi = rsqrtf(fmaxf(1.f - cosphi * cosphi, 1e-20f));
      float fr = -(float)bend_k[u] * (float)rrd * 2.f;
      float irasin = drai * isinphi * fr, ircsin = drci * isinphi * fr;
      float fxa = (erax * cosphi - ercx) * irasin, fya = (eray * cosphi - ercy) * irasin,
            fza = (eraz * cosphi - ercz) * irasin;
      float fxc = (ercx * cosphi - erax) * ircsin, fyc = (ercy * cosphi - eray) * ircsin,
            fzc = (ercz * cosphi - eraz) * ircsin;
      long long ax = to_fix(fxa), ay = to_fix(fya), az = to_fix(fza);
      long long cx = to_fix(fxc), cy = to_fix(fyc), cz = to_fix(fzc);
      atomicAdd(&fix[3 * ia], (unsigned long long)ax);
      atomicAdd(&fix[3 * ia + 1], (unsigned long long)ay);
      atomicAdd(&fix[3 * ia + 2], (unsigned long long)az);
      atomicAdd(&fix[3 * ib], (unsigned long long)(-(ax + cx)));
      atomicAdd(&fix[3 * ib + 1], (unsigned long long)(-(ay + cy)));
      atomicAdd(&fix[3 * ib + 2], (unsigned long long)(-(az + cz)));
      atomicAdd(&fix[3 * ic], (unsigned long long)cx);
      atomicAdd(&fix[3 * ic + 1], (unsigned long long)cy);
      atomicAdd(&fix[3 * ic + 2], (unsigned long long)cz);
    }
  }
  double v[2] = {eb, ea};
  block_fix_final<2>(v, 32, facc, ticket, out);
}

// ---------------------------------------------------------------------------
// SPME in FP32

// B-spline weights of order p at fraction w (same recursion as
// pme_spline.c:10-49), FP32
__device__ __forceinline__ void fillspline_f(int order, float w, float *array, float *darray) {
  for (int i = 3; i <= order; i++) array[i] = 0.f;
  array[2] = w;
  array[1] = 1.f - w;
  array[0] = 0.f;
  for (int i = 3; i <= order - 1; i++) {
    float div = 1.f / (float)(i - 1);
    array[i] = div * w * array[i - 1];
    for (int j = 1; j <= (i - 2); j++)
      array[i - j] = div * ((w + j) * array[i - j - 1] + ((float)(i - j) - w) * array[i - j]);
    array[1] *= div * (1.f - w);
  }
  darray[0] = 0.f;
  darray[1] = -array[1];
  for (int i = 2; i <= order; i++) darray[i] = array[i - 1] - array[i];
  int kk = order;
  float div = 1.f / (float)(kk - 1);
  array[kk] = div * w * array[kk - 1];
  for (int i = 1; i <= (kk - 2); i++)
    array[kk - i] = div * ((w + i) * array[kk - i - 1] + ((float)(kk - i) - w) * array[kk - i]);
  array[1] *= div * (1.f - w);
}

// per sorted slot: origin cell and fraction exactly from the 32-bit
// fixed-point coordinate (u G / 2^32: integer part and remainder), FP32
// weights, binning
// B-spline weights and derivatives of every site and its integer spline
// origin (floor of u G, exact from the 32-bit fraction)
__device__ __forceinline__ void k_mx_splines_body(VBlk vb_, int n, int order, int3 G, const int4 *__restrict__ posfx,
                             int *__restrict__ floor3, float *__restrict__ sm,
                             float *__restrict__ sd) {
  int s = vb_.id * blockDim.x + threadIdx.x;
  if (s >= n) return;
  int4 p = posfx[s];
  unsigned u[3] = {(unsigned)p.x, (unsigned)p.y, (unsigned)p.z};
  int g[3] = {G.x, G.y, G.z};
  float mn[9], dmn[9];
  for (int d = 0; d < 3; d++) {
    unsigned long long t = (unsigned long long)u[d] * (unsigned)g[d];
    float w = (float)(unsigned)(t & 0xffffffffull) * 0x1p-32f;
    fillspline_f(order, w, mn, dmn);
    for (int m = 1; m <= order; m++) {
      sm[((size_t)s * order + (m - 1)) * 3 + d] = mn[m];
      sd[((size_t)s * order + (m - 1)) * 3 + d] = dmn[m];
    }
    floor3[3 * s + d] = (int)(t >> 32);
  }
}

__global__ void k_mx_splines(int n, int order, int3 G, const int4 *__restrict__ posfx,
                             int *__restrict__ floor3, float *__restrict__ sm,
                             float *__restrict__ sd) {
  k_mx_splines_body(vblk_self(), n, order, G, posfx, floor3, sm, sd);
}

// Spreading by fixed-point reductions: thread (site, mx) adds the
// contributions q wx wy wz of its site's spline slab mx (order x order
// points) to a 64-bit fixed-point grid (2^40 per unit) with fire-and-forget
// integer reductions.  Integer sums do not depend on the order of the
// additions, so the grid is bitwise reproducible; sites in sorted (spatial)
// order keep neighbouring threads on neighbouring grid lines.
constexpr float kSpRedFix = 1099511627776.0f;  // 2^40

__device__ __forceinline__ void k_mx_spread_red_body(VBlk vb_, int n, int order, int3 G, const int4 *__restrict__ posfx,
                                const float *__restrict__ sm, const int *__restrict__ floor3,
                                unsigned long long *__restrict__ gfix) {
  int t = vb_.id * blockDim.x + threadIdx.x;
  int s = t / order, mx = t - s * order;
  if (s >= n) return;
  const float *w = sm + (size_t)s * order * 3;
  float qwx = __int_as_float(posfx[s].w) * w[mx * 3];
  int x = floor3[3 * s] - order + 1 + mx, y0 = floor3[3 * s + 1] - order + 1,
      z0 = floor3[3 * s + 2] - order + 1;
  if (x < 0) x += G.x;
  unsigned long long *gx = gfix + (size_t)x * G.y * G.z;
  for (int my = 0; my < order; my++) {
    int y = y0 + my;
    if (y < 0) y += G.y;
    float v = qwx * w[my * 3 + 1];
    unsigned long long *gy = gx + (size_t)y * G.z;
    for (int mz = 0; mz < order; mz++) {
      int z = z0 + mz;
      if (z < 0) z += G.z;
      atomicAdd(gy + z, (unsigned long long)__float2ll_rn(v * w[mz * 3 + 2] * kSpRedFix));
    }
  }
}

__global__ void k_mx_spread_red(int n, int order, int3 G, const int4 *__restrict__ posfx,
                                const float *__restrict__ sm, const int *__restrict__ floor3,
                                unsigned long long *__restrict__ gfix) {
  k_mx_spread_red_body(vblk_self(), n, order, G, posfx, sm, floor3, gfix);
}

// Order 4 (the configured workloads): the spline weights are computed where
// they are used, from the site's 32-bit fixed-point coordinate, instead of
// being stored by a separate pass and read back (fillspline_f with a
// constant order unrolls into registers).
__device__ __forceinline__ void spline4_axis(unsigned u, int g, int &fl, float (&m)[5],
                                             float (&dm)[5]) {
  unsigned long long t = (unsigned long long)u * (unsigned)g;
  fl = (int)(t >> 32);
  fillspline_f(4, (float)(unsigned)(t & 0xffffffffull) * 0x1p-32f, m, dm);
}

__device__ __forceinline__ void k_mx_spread_o4_body(VBlk vb_, int n, int3 G,
                                                  const int4 *__restrict__ posfx,
                                                  unsigned long long *__restrict__ gfix) {
  int t = vb_.id * blockDim.x + threadIdx.x;
  int s = t >> 2, mx = t & 3;
  if (s >= n) return;
  int4 p = posfx[s];
  float wx[5], wy[5], wz[5], dd[5];
  int fx, fy, fz;
  spline4_axis((unsigned)p.x, G.x, fx, wx, dd);
  spline4_axis((unsigned)p.y, G.y, fy, wy, dd);
  spline4_axis((unsigned)p.z, G.z, fz, wz, dd);
  float w_mx = mx == 0 ? wx[1] : mx == 1 ? wx[2] : mx == 2 ? wx[3] : wx[4];
  float qwx = __int_as_float(p.w) * w_mx;
  int x = fx - 3 + mx, y0 = fy - 3, z0 = fz - 3;
  if (x < 0) x += G.x;
  unsigned long long *gx = gfix + (size_t)x * G.y * G.z;
#pragma unroll
  for (int my = 0; my < 4; my++) {
    int y = y0 + my;
    if (y < 0) y += G.y;
    float v = qwx * wy[my + 1];
    unsigned long long *gy = gx + (size_t)y * G.z;
#pragma unroll
    for (int mz = 0; mz < 4; mz++) {
      int z = z0 + mz;
      if (z < 0) z += G.z;
      atomicAdd(gy + z, (unsigned long long)__float2ll_rn(v * wz[mz + 1] * kSpRedFix));
    }
  }
}

__global__ void k_mx_spread_o4(int n, int3 G, const int4 *__restrict__ posfx,
                             unsigned long long *__restrict__ gfix) {
  k_mx_spread_o4_body(vblk_self(), n, G, posfx, gfix);
}

// FP32 grid from the fixed-point sums; the sums are cleared for the next step
// (two points per thread and iteration: 16-byte loads and stores)
__device__ __forceinline__ void k_mx_fix2grid_body(VBlk vb_, long K, unsigned long long *__restrict__ gfix,
                              float *__restrict__ grid) {
  const long K2 = K >> 1;
  longlong2 *g2 = reinterpret_cast<longlong2 *>(gfix);
  float2 *o2 = reinterpret_cast<float2 *>(grid);
  for (long i = (long)vb_.id * blockDim.x + threadIdx.x; i < K2;
       i += (long)vb_.n * blockDim.x) {
    longlong2 v = g2[i];
    o2[i] = make_float2(fft_fix((unsigned long long)v.x), fft_fix((unsigned long long)v.y));
    g2[i] = make_longlong2(0, 0);
  }
  if ((K & 1) && vb_.id == 0 && threadIdx.x == 0) {
    grid[K - 1] = fft_fix(gfix[K - 1]);
    gfix[K - 1] = 0ull;
  }
}

__global__ void k_mx_fix2grid(long K, unsigned long long *__restrict__ gfix,
                              float *__restrict__ grid) {
  k_mx_fix2grid_body(vblk_self(), K, gfix, grid);
}

__device__ __forceinline__ void k_mx_recip_body(VBlk vb_, long Kh, const float *__restrict__ eterm, const float *__restrict__ kw,
                           cufftComplex *__restrict__ gk, unsigned long long *__restrict__ facc,
                           unsigned *__restrict__ ticket, double *__restrict__ out) {
  float e = 0.f;
  for (long h = (long)vb_.id * blockDim.x + threadIdx.x; h < Kh;
       h += (long)vb_.n * blockDim.x) {
    cufftComplex v = gk[h];
    float et = eterm[h];
    e = fmaf(kw[h] * et, v.x * v.x + v.y * v.y, e);
    v.x *= et;
    v.y *= et;
    gk[h] = v;
  }
  float vv[1] = {e};
  block_fix_final<1>(vv, 24, facc, ticket, out, vb_);
}

// The transforms and the convolution between them (fe_fft.cuh): planes, x
// lines, planes; the energy sum as in k_mx_recip.
__global__ void __launch_bounds__(512) k_mx_fft_forward(FftBox<float> B) {
  extern __shared__ float4 fft_sh[];
  fft_forward_body<float>(B, blockIdx.x, reinterpret_cast<Cx<float> *>(fft_sh));
}
__global__ void __launch_bounds__(512) k_mx_fft_backward(FftBox<float> B) {
  extern __shared__ float4 fft_sh[];
  fft_backward_body<float>(B, blockIdx.x, reinterpret_cast<Cx<float> *>(fft_sh));
}
__global__ void __launch_bounds__(256)
k_mx_fft_convolve(FftBox<float> B, unsigned long long *__restrict__ facc,
                  unsigned *__restrict__ ticket, double *__restrict__ out) {
  extern __shared__ float4 fft_sh[];
  float v[1] = {fft_convolve_body<float>(B, blockIdx.x, reinterpret_cast<Cx<float> *>(fft_sh))};
  block_fix_final<1>(v, 24, facc, ticket, out);
}

__global__ void k_mx_recip(long Kh, const float *__restrict__ eterm, const float *__restrict__ kw,
                           cufftComplex *__restrict__ gk, unsigned long long *__restrict__ facc,
                           unsigned *__restrict__ ticket, double *__restrict__ out) {
  k_mx_recip_body(vblk_self(), Kh, eterm, kw, gk, facc, ticket, out);
}

__device__ __forceinline__ void k_mx_gather_body(VBlk vb_, int n, int order, int3 G, float3 gl, float qfe,
                            const int4 *__restrict__ posfx, const int *__restrict__ perm,
                            const int *__restrict__ floor3, const float *__restrict__ sm,
                            const float *__restrict__ sd, const float *__restrict__ grid,
                            unsigned long long *__restrict__ fix,
                            unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                            double *__restrict__ out) {
  long long sx = 0, sy = 0, sz = 0;
  for (int s = vb_.id * blockDim.x + threadIdx.x; s < n; s += vb_.n * blockDim.x) {
    float fxi = 0.f, fyi = 0.f, fzi = 0.f;
    const float *m = sm + (size_t)s * order * 3;
    const float *dm = sd + (size_t)s * order * 3;
    int xo = floor3[3 * s] - order, yo0 = floor3[3 * s + 1] - order, zo0 = floor3[3 * s + 2] - order;
    for (int xi = 1; xi <= order; xi++) {
      int x = wrap1(xo + xi, G.x);
      float mx = m[(xi - 1) * 3], dmx = dm[(xi - 1) * 3];
      for (int yi = 1; yi <= order; yi++) {
        int y = wrap1(yo0 + yi, G.y);
        float my = m[(yi - 1) * 3 + 1], dmy = dm[(yi - 1) * 3 + 1];
        const float *row = grid + ((long)x * G.y + y) * G.z;
        for (int zi = 1; zi <= order; zi++) {
          int z = wrap1(zo0 + zi, G.z);
          float mz = m[(zi - 1) * 3 + 2], dmz = dm[(zi - 1) * 3 + 2];
          float term = row[z];
          fxi -= dmx * my * mz * term;
          fyi -= mx * dmy * mz * term;
          fzi -= mx * my * dmz * term;
        }
      }
    }
    float fac = __int_as_float(posfx[s].w) * qfe;
    fxi *= fac * gl.x;
    fyi *= fac * gl.y;
    fzi *= fac * gl.z;
    int oi = perm[s];
    long long qx = to_fix(fxi), qy = to_fix(fyi), qz = to_fix(fzi);
    atomicAdd(&fix[3 * oi], (unsigned long long)qx);
    atomicAdd(&fix[3 * oi + 1], (unsigned long long)qy);
    atomicAdd(&fix[3 * oi + 2], (unsigned long long)qz);
    sx += qx;
    sy += qy;
    sz += qz;
  }
  long long v[3] = {sx, sy, sz};
  block_fix_final<3>(v, 0, facc, ticket, out, vb_);
}

__global__ void k_mx_gather(int n, int order, int3 G, float3 gl, float qfe,
                            const int4 *__restrict__ posfx, const int *__restrict__ perm,
                            const int *__restrict__ floor3, const float *__restrict__ sm,
                            const float *__restrict__ sd, const float *__restrict__ grid,
                            unsigned long long *__restrict__ fix,
                            unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                            double *__restrict__ out) {
  k_mx_gather_body(vblk_self(), n, order, G, gl, qfe, posfx, perm, floor3, sm, sd, grid, fix, facc, ticket, out);
}

// gather with the order-4 weights and derivatives computed in registers.  LANES
// threads per site: one, or in small boxes four, an x plane each (1,500 sites
// are 12 blocks of single threads, each with 64 loads and 600 operations).
template <int LANES>
__device__ __forceinline__ void k_mx_gather_o4_body(VBlk vb_, int n, int3 G, float3 gl, float qfe,
                                                  const int4 *__restrict__ posfx,
                                                  const int *__restrict__ perm,
                                                  const float *__restrict__ grid,
                                                  unsigned long long *__restrict__ fix,
                                                  unsigned long long *__restrict__ facc,
                                                  unsigned *__restrict__ ticket,
                                                  double *__restrict__ out) {
  long long sx = 0, sy = 0, sz = 0;
  const int sub = LANES == 1 ? 0 : (int)threadIdx.x % LANES, per = blockDim.x / LANES;
  for (int s0 = vb_.id * per; s0 < n; s0 += vb_.n * per) {
    const int s = s0 + threadIdx.x / LANES;
    if (LANES == 1 && s >= n) break;
    int4 p = posfx[min(s, n - 1)];
    float m[3][5], dm[3][5];
    int fl[3];
    spline4_axis((unsigned)p.x, G.x, fl[0], m[0], dm[0]);
    spline4_axis((unsigned)p.y, G.y, fl[1], m[1], dm[1]);
    spline4_axis((unsigned)p.z, G.z, fl[2], m[2], dm[2]);
    float fxi = 0.f, fyi = 0.f, fzi = 0.f;
    int xo = fl[0] - 4, yo0 = fl[1] - 4, zo0 = fl[2] - 4;
#pragma unroll
    for (int xi = 1; xi <= 4 / LANES; xi++) {
      int x = wrap1(xo + xi + sub, G.x);
      float mx = m[0][xi], dmx = dm[0][xi];
      if (LANES > 1) {
#pragma unroll
        for (int k = 2; k <= 4; k++)
          if (sub == k - 1) {
            mx = m[0][k];
            dmx = dm[0][k];
          }
      }
#pragma unroll
      for (int yi = 1; yi <= 4; yi++) {
        int y = wrap1(yo0 + yi, G.y);
        float my = m[1][yi], dmy = dm[1][yi];
        const float *row = grid + ((long)x * G.y + y) * G.z;
#pragma unroll
        for (int zi = 1; zi <= 4; zi++) {
          int z = wrap1(zo0 + zi, G.z);
          float mz = m[2][zi], dmz = dm[2][zi];
          float term = row[z];
          fxi -= dmx * my * mz * term;
          fyi -= mx * dmy * mz * term;
          fzi -= mx * my * dmz * term;
        }
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      fxi += __shfl_xor_sync(0xffffffffu, fxi, o);
      fyi += __shfl_xor_sync(0xffffffffu, fyi, o);
      fzi += __shfl_xor_sync(0xffffffffu, fzi, o);
    }
    if (s >= n || sub != 0) continue;
    float fac = __int_as_float(p.w) * qfe;
    fxi *= fac * gl.x;
    fyi *= fac * gl.y;
    fzi *= fac * gl.z;
    int oi = perm[s];
    long long qx = to_fix(fxi), qy = to_fix(fyi), qz = to_fix(fzi);
    atomicAdd(&fix[3 * oi], (unsigned long long)qx);
    atomicAdd(&fix[3 * oi + 1], (unsigned long long)qy);
    atomicAdd(&fix[3 * oi + 2], (unsigned long long)qz);
    sx += qx;
    sy += qy;
    sz += qz;
  }
  long long v[3] = {sx, sy, sz};
  block_fix_final<3>(v, 0, facc, ticket, out, vb_);
}

template <int LANES>
__global__ void k_mx_gather_o4(int n, int3 G, float3 gl, float qfe, const int4 *__restrict__ posfx,
                             const int *__restrict__ perm, const float *__restrict__ grid,
                             unsigned long long *__restrict__ fix,
                             unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                             double *__restrict__ out) {
  k_mx_gather_o4_body<LANES>(vblk_self(), n, G, gl, qfe, posfx, perm, grid, fix, facc, ticket, out);
}

// Sites up to which four lanes share a site's gather; above, single threads fill the
// SMs.  With four lanes and with one, us a step: 1,500 sites 42.2 and 44.5, 4,095 48.4
// and 50.5, 12,000 79.4 and 79.9, 16,200 101.0 and 100.6, 48,000 both 178.4, 96,000
// 302.6 and 297.7.
constexpr int kGatherLanesSites = 16384;

// FP64 forces from the fixed-point sums, minus the mean reciprocal force
__device__ __forceinline__ void k_mx_finalize_body(VBlk vb_, int n, const unsigned long long *__restrict__ fix,
                              const double *__restrict__ scal, double *__restrict__ ff) {
  __shared__ double mean[3];
  if (threadIdx.x < 3) mean[threadIdx.x] = scal[SC_FMEAN + threadIdx.x] / kFixScale / (double)n;
  __syncthreads();
  int i = vb_.id * blockDim.x + threadIdx.x;
  if (i >= 3 * n) return;
  ff[i] = (double)(long long)fix[i] * (1.0 / kFixScale) - mean[i % 3];
}

__global__ void k_mx_finalize(int n, const unsigned long long *__restrict__ fix,
                              const double *__restrict__ scal, double *__restrict__ ff) {
  k_mx_finalize_body(vblk_self(), n, fix, scal, ff);
}

// All intramolecular terms of one molecule per thread: the exclusion
// corrections of k_mx_excl and the bonds and bends of k_mx_bonded, same
// arithmetic, with the molecule's forces summed in registers and added to
// the fixed-point accumulators once (atomically: the pair kernel and the
// gather may run beside it).
// site a of a molecule's register arrays, selected without dynamic indexing
template <int NS>
__device__ __forceinline__ int4 intra_pick(const int4 (&P)[NS], int a) {
  int4 r = P[0];
#pragma unroll
  for (int i = 1; i < NS; i++)
    if (a == i) r = P[i];
  return r;
}
template <int NS>
__device__ __forceinline__ void intra_add(float (&F)[NS][3], int a, float x, float y, float z) {
#pragma unroll
  for (int i = 0; i < NS; i++)
    if (a == i) {
      F[i][0] += x;
      F[i][1] += y;
      F[i][2] += z;
    }
}

// NS: the largest molecule (sites) of the box, so that the molecule's
// positions and forces stay in registers
// The three kinds of intramolecular term, each adding to the molecule's
// force registers F and the thread's energy sums A.
struct IntraAcc {
  float e_lj = 0.f, e_ljs = 0.f, e_real = 0.f, qsum = 0.f;
  double eb = 0.0, ea = 0.0;  // bond and bend energies (FP64 geometry)
  long long q_intra = 0;
};


// excluded (xf 1-3) or 1-4 (xf 4) pair a-bq: the intra correction, and for
// 1-4 pairs the scaled real-space term and LJ (cnonbond_nblist.c:245-263,
// 416-437); qa, qb the FP64 charges, type_a / type_b the site types
template <int NS>
__device__ __forceinline__ void intra_excl(const int4 (&P)[NS], float (&F)[NS][3], int a, int bq,
                                           int xf, double qa, double qb, int type_a, int type_b,
                                           float3 sL, int nt, const float *__restrict__ lj_tab,
                                           float rc2, float kappa, float c2k, float qf,
                                           float epsRF, const float2 *__restrict__ exptab,
                                           const DfIntra &D, IntraAcc &A) {
  const int4 Pa = intra_pick(P, a), Pb = intra_pick(P, bq);
  float dx = fx_delta((unsigned)Pa.x, (unsigned)Pb.x, sL.x);
  float dy = fx_delta((unsigned)Pa.y, (unsigned)Pb.y, sL.y);
  float dz = fx_delta((unsigned)Pa.z, (unsigned)Pb.z, sL.z);
  float r2 = dx * dx + dy * dy + dz * dz;
  if (r2 > rc2) return;
  float rinv = rsqrtf(r2), r = r2 * rinv, rinv2 = rinv * rinv;
  float kr = kappa * r;
  float ex = __expf(-kr * kr);
  float erfckr = erfc_nr_f(kr, ex);
  float qqab = __int_as_float(Pa.w) * __int_as_float(Pb.w) * qf;
  float Fs = 0.f;
  float qcorr = qqab;
  if (xf == 4) {
    float qq = qqab * (float)kE14FAC / epsRF;
    Fs += qq * rinv * rinv2 * (erfckr + c2k * r * ex);
    A.e_real += qq * erfckr * rinv;
    A.qsum += qq;
    const float *lj = lj_tab + (type_a * nt + type_b) * 3;
    if (lj[0] != 0.f) {
      float sr2 = lj[1] * rinv2, sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6;
      Fs += 12.f * lj[0] * rinv2 * (sr12 - sr6);
      A.e_lj += lj[0] * (sr12 - 2.f * sr6);
      A.e_ljs += lj[0] * lj[2];
    }
    qcorr *= (1.f - (float)kE14FAC);
  }
  float erfkr = 1.f - erfckr;
  A.q_intra += df_to_fixed(
      intra_energy_df(D, Pa, Pb, qa, qb, xf == 4 ? (float)(1.0 - kE14FAC) : 1.f, exptab), 32);
  Fs -= qcorr * rinv * rinv2 * (erfkr - c2k * r * ex);
  intra_add(F, a, Fs * dx, Fs * dy, Fs * dz);
  intra_add(F, bq, -Fs * dx, -Fs * dy, -Fs * dz);
}

// cbond.c:27: E = k (r - r0)^2.  The stretch and the energy in FP64 from
// the exact fixed-point differences (a sum of ~1e5 small positive terms
// keeps 1e-7 only if each stretch does: FP32 lengths carry ~1e-7 of r, a
// few 1e-6 of r - r0); the force in FP32 along the FP32 bond vector.
template <int NS>
__device__ __forceinline__ void intra_bond(const int4 (&P)[NS], float (&F)[NS][3], int ia, int ib,
                                           double req, float kb, float3 sL, double3 sd,
                                           IntraAcc &A) {
  const int4 Pa = intra_pick(P, ia), Pb = intra_pick(P, ib);
  const double ex = fx_delta_d((unsigned)Pb.x, (unsigned)Pa.x, sd.x);
  const double ey = fx_delta_d((unsigned)Pb.y, (unsigned)Pa.y, sd.y);
  const double ez = fx_delta_d((unsigned)Pb.z, (unsigned)Pa.z, sd.z);
  const double rr = sqrt(ex * ex + ey * ey + ez * ez) - req;
  A.eb += (double)kb * rr * rr;
  float dx = fx_delta((unsigned)Pb.x, (unsigned)Pa.x, sL.x);
  float dy = fx_delta((unsigned)Pb.y, (unsigned)Pa.y, sL.y);
  float dz = fx_delta((unsigned)Pb.z, (unsigned)Pa.z, sL.z);
  float dr = sqrtf(dx * dx + dy * dy + dz * dz);
  float fr = -kb * (float)rr * 2.f;
  float sc = fr / dr;
  intra_add(F, ia, -sc * dx, -sc * dy, -sc * dz);
  intra_add(F, ib, sc * dx, sc * dy, sc * dz);
}

// cbend.c:24: E = k (theta - theta0)^2.  The angle and the energy in FP64
// (as the stretch above); the force in FP32 from the FP32 unit vectors.
template <int NS>
__device__ __forceinline__ void intra_bend(const int4 (&P)[NS], float (&F)[NS][3], int ia, int ib,
                                           int ic, double t0, float ka, float3 sL, double3 sd,
                                           IntraAcc &A) {
  const int4 Pa = intra_pick(P, ia), Pb = intra_pick(P, ib), Pc = intra_pick(P, ic);
  const double ax = fx_delta_d((unsigned)Pa.x, (unsigned)Pb.x, sd.x);
  const double ay = fx_delta_d((unsigned)Pa.y, (unsigned)Pb.y, sd.y);
  const double az = fx_delta_d((unsigned)Pa.z, (unsigned)Pb.z, sd.z);
  const double cx = fx_delta_d((unsigned)Pc.x, (unsigned)Pb.x, sd.x);
  const double cy = fx_delta_d((unsigned)Pc.y, (unsigned)Pb.y, sd.y);
  const double cz = fx_delta_d((unsigned)Pc.z, (unsigned)Pb.z, sd.z);
  double cosd = (ax * cx + ay * cy + az * cz) /
                sqrt((ax * ax + ay * ay + az * az) * (cx * cx + cy * cy + cz * cz));
  cosd = fmin(fmax(cosd, -1.0), 1.0);
  const double rr = acos(cosd) - t0;
  A.ea += (double)ka * rr * rr;
  float dax = fx_delta((unsigned)Pa.x, (unsigned)Pb.x, sL.x);
  float day = fx_delta((unsigned)Pa.y, (unsigned)Pb.y, sL.y);
  float daz = fx_delta((unsigned)Pa.z, (unsigned)Pb.z, sL.z);
  float dcx = fx_delta((unsigned)Pc.x, (unsigned)Pb.x, sL.x);
  float dcy = fx_delta((unsigned)Pc.y, (unsigned)Pb.y, sL.y);
  float dcz = fx_delta((unsigned)Pc.z, (unsigned)Pb.z, sL.z);
  float drai = rsqrtf(dax * dax + day * day + daz * daz);
  float erax = dax * drai, eray = day * drai, eraz = daz * drai;
  float drci = rsqrtf(dcx * dcx + dcy * dcy + dcz * dcz);
  float ercx = dcx * drci, ercy = dcy * drci, ercz = dcz * drci;
  float cosphi = (float)cosd;
  float isinphi = rsqrtf(fmaxf(1.f - cosphi * cosphi, 1e-20f));
  float fr = -ka * (float)rr * 2.f;
  float irasin = drai * isinphi * fr, ircsin = drci * isinphi * fr;
  float fxa = (erax * cosphi - ercx) * irasin, fya = (eray * cosphi - ercy) * irasin,
        fza = (eraz * cosphi - ercz) * irasin;
  float fxc = (ercx * cosphi - erax) * ircsin, fyc = (ercy * cosphi - eray) * ircsin,
        fzc = (ercz * cosphi - eraz) * ircsin;
  intra_add(F, ia, fxa, fya, fza);
  intra_add(F, ic, fxc, fyc, fzc);
  intra_add(F, ib, -(fxa + fxc), -(fya + fyc), -(fza + fzc));
}

template <int NS>
__device__ __forceinline__ void k_mx_intra_body(VBlk vb_, int nmol, const int *__restrict__ mol_first,
                           const int *__restrict__ mol_x, const int *__restrict__ mol_xi,
                           const int *__restrict__ mol_b, const int *__restrict__ mol_bi,
                           const int *__restrict__ mol_a, const int *__restrict__ mol_ai,
                           const int *__restrict__ ab, const int *__restrict__ flag,
                           const int *__restrict__ bond_ab, const double *__restrict__ bond_req,
                           const double *__restrict__ bond_k, const int *__restrict__ bend_abc,
                           const double *__restrict__ bend_t0, const double *__restrict__ bend_k,
                           const int4 *__restrict__ posfx, const int *__restrict__ iperm,
                           const int *__restrict__ type, float3 sL, int nt,
                           const float *__restrict__ lj_tab, float rc2, float kappa, float c2k,
                           float qf, float epsRF, const double4 *__restrict__ pos_q,
                           const float2 *__restrict__ exptab, DfIntra D,
                           unsigned long long *__restrict__ fix,
                           unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                           double *__restrict__ out) {
  IntraAcc A;
  // the length scale per axis, L / 2^32, in FP64 (hi + lo)
  const double3 sd = make_double3((double)D.sl[0].x + (double)D.sl[0].y,
                                  (double)D.sl[1].x + (double)D.sl[1].y,
                                  (double)D.sl[2].x + (double)D.sl[2].y);
  for (int m = vb_.id * blockDim.x + threadIdx.x; m < nmol; m += vb_.n * blockDim.x) {
    const int lb = mol_first[m];
    const int ns = mol_first[m + 1] - lb;
    int4 P[NS];
    float F[NS][3];
#pragma unroll
    for (int i = 0; i < NS; i++) {
      P[i] = i < ns ? posfx[iperm[lb + i]] : make_int4(0, 0, 0, 0);
      F[i][0] = F[i][1] = F[i][2] = 0.f;
    }
    const int tx0 = mol_x[m], tx1 = mol_x[m + 1];
#pragma unroll
    for (int t = tx0; t < tx1; t++) {
      int a, bq, xf;
      int x = mol_xi[t];
      a = ab[2 * x] - lb;
      bq = ab[2 * x + 1] - lb;
      xf = flag[x];
      if (xf == 0) continue;
      intra_excl<NS>(P, F, a, bq, xf, pos_q[lb + a].w, pos_q[lb + bq].w,
                     type[lb + a], type[lb + bq], sL, nt, lj_tab, rc2, kappa, c2k, qf, epsRF, exptab, D, A);
    }
    const int tb0 = mol_b[m], tb1 = mol_b[m + 1];
#pragma unroll
    for (int t = tb0; t < tb1; t++) {
      int ia, ib;
      double req;
      float kb;
      int u = mol_bi[t];
      ia = bond_ab[2 * u] - lb;
      ib = bond_ab[2 * u + 1] - lb;
      req = bond_req[u];
      kb = (float)bond_k[u];
      intra_bond<NS>(P, F, ia, ib, req, kb, sL, sd, A);
    }
    const int ta0 = mol_a[m], ta1 = mol_a[m + 1];
#pragma unroll
    for (int t = ta0; t < ta1; t++) {
      int ia, ib, ic;
      double t0;
      float ka;
      int u = mol_ai[t];
      ia = bend_abc[3 * u] - lb;
      ib = bend_abc[3 * u + 1] - lb;
      ic = bend_abc[3 * u + 2] - lb;
      t0 = bend_t0[u];
      ka = (float)bend_k[u];
      intra_bend<NS>(P, F, ia, ib, ic, t0, ka, sL, sd, A);
    }
#pragma unroll
    for (int i = 0; i < NS; i++)
      if (i < ns)
#pragma unroll
        for (int c = 0; c < 3; c++) {
          unsigned long long *q = fix + 3 * (size_t)(lb + i) + c;
          atomicAdd(q, (unsigned long long)to_fix(F[i][c]));
        }
  }
  long long v[7] = {to_fixed(A.e_lj, 32), to_fixed(A.e_ljs, 32), to_fixed(A.e_real, 32),
                    to_fixed(A.qsum, 32), A.q_intra, to_fixed(A.eb, 32), to_fixed(A.ea, 32)};
  block_fix_final<7>(v, 32, facc, ticket, out, vb_);
}

template <int NS>
__global__ void k_mx_intra(int nmol, const int *__restrict__ mol_first,
                           const int *__restrict__ mol_x, const int *__restrict__ mol_xi,
                           const int *__restrict__ mol_b, const int *__restrict__ mol_bi,
                           const int *__restrict__ mol_a, const int *__restrict__ mol_ai,
                           const int *__restrict__ ab, const int *__restrict__ flag,
                           const int *__restrict__ bond_ab, const double *__restrict__ bond_req,
                           const double *__restrict__ bond_k, const int *__restrict__ bend_abc,
                           const double *__restrict__ bend_t0, const double *__restrict__ bend_k,
                           const int4 *__restrict__ posfx, const int *__restrict__ iperm,
                           const int *__restrict__ type, float3 sL, int nt,
                           const float *__restrict__ lj_tab, float rc2, float kappa, float c2k,
                           float qf, float epsRF, const double4 *__restrict__ pos_q,
                           const float2 *__restrict__ exptab, DfIntra D,
                           unsigned long long *__restrict__ fix,
                           unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                           double *__restrict__ out) {
  k_mx_intra_body<NS>(vblk_self(), nmol, mol_first, mol_x, mol_xi, mol_b, mol_bi, mol_a, mol_ai, ab, flag, bond_ab, bond_req, bond_k, bend_abc, bend_t0, bend_k, posfx, iperm, type, sL, nt, lj_tab, rc2, kappa, c2k, qf, epsRF, pos_q, exptab, D, fix, facc, ticket, out);
}

// A box of identical molecules, one TERM per thread: warps take 32 molecules
// of one exclusion, bond or bend of the template, so a molecule's six terms
// (water) run side by side instead of one after another -- at 1,500 sites one
// thread per molecule kept 4 SMs busy for 25 us with FP64 roots and arc
// cosines.  Forces go to the fixed-point sums term by term.
__device__ __forceinline__ void k_mx_terms_body(
    VBlk vb_, int nmol, const IntraTpl &T, const int4 *__restrict__ posfx,
    const int *__restrict__ iperm, float3 sL, int nt, const float *__restrict__ lj_tab, float rc2,
    float kappa, float c2k, float qf, float epsRF, const double4 *__restrict__ pos_q,
    const float2 *__restrict__ exptab, const DfIntra &D, unsigned long long *__restrict__ fix,
    unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
    double *__restrict__ out) {
  IntraAcc A;
  const double3 sd = make_double3((double)D.sl[0].x + (double)D.sl[0].y,
                                  (double)D.sl[1].x + (double)D.sl[1].y,
                                  (double)D.sl[2].x + (double)D.sl[2].y);
  const int lane = threadIdx.x & 31, mw = (nmol + 31) / 32, nterm = T.nx + T.nb + T.na;
  const int wpb = blockDim.x >> 5;
  for (int w = vb_.id * wpb + (threadIdx.x >> 5); w < nterm * mw; w += vb_.n * wpb) {
    const int q = w / mw, m = (w - q * mw) * 32 + lane;  // bends first: the longest
    if (m >= nmol) continue;
    const int lb = m * T.ns;
    int s[3] = {0, 0, 0};
    int4 P[3];
    float F[3][3];
    int ns = 2;
    if (q < T.na) {
      s[0] = T.aa[q];
      s[1] = T.ab[q];
      s[2] = T.ac[q];
      ns = 3;
    } else if (q < T.na + T.nb) {
      s[0] = T.ba[q - T.na];
      s[1] = T.bb[q - T.na];
    } else {
      s[0] = T.xa[q - T.na - T.nb];
      s[1] = T.xb[q - T.na - T.nb];
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      P[i] = i < ns ? posfx[iperm[lb + s[i]]] : make_int4(0, 0, 0, 0);
      F[i][0] = F[i][1] = F[i][2] = 0.f;
    }
    if (q < T.na) {
      intra_bend<3>(P, F, 0, 1, 2, (double)T.at0[q] + (double)T.at0_lo[q], T.ak[q], sL, sd, A);
    } else if (q < T.na + T.nb) {
      const int t = q - T.na;
      intra_bond<3>(P, F, 0, 1, (double)T.breq[t] + (double)T.breq_lo[t], T.bk[t], sL, sd, A);
    } else {
      const int t = q - T.na - T.nb;
      if (T.xf[t] != 0)
        intra_excl<3>(P, F, 0, 1, T.xf[t], pos_q[lb + s[0]].w, pos_q[lb + s[1]].w, T.type[s[0]],
                      T.type[s[1]], sL, nt, lj_tab, rc2, kappa, c2k, qf, epsRF, exptab, D, A);
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
      if (i < ns)
#pragma unroll
        for (int c = 0; c < 3; c++)
          atomicAdd(fix + 3 * (size_t)(lb + s[i]) + c, (unsigned long long)to_fix(F[i][c]));
  }
  long long v[7] = {to_fixed(A.e_lj, 32), to_fixed(A.e_ljs, 32), to_fixed(A.e_real, 32),
                    to_fixed(A.qsum, 32), A.q_intra, to_fixed(A.eb, 32), to_fixed(A.ea, 32)};
  block_fix_final<7>(v, 32, facc, ticket, out, vb_);
}

__global__ void k_mx_terms(int nmol, const __grid_constant__ IntraTpl T,
                           const int4 *__restrict__ posfx,
                           const int *__restrict__ iperm, float3 sL, int nt,
                           const float *__restrict__ lj_tab, float rc2, float kappa, float c2k,
                           float qf, float epsRF, const double4 *__restrict__ pos_q,
                           const float2 *__restrict__ exptab, const __grid_constant__ DfIntra D,
                           unsigned long long *__restrict__ fix,
                           unsigned long long *__restrict__ facc, unsigned *__restrict__ ticket,
                           double *__restrict__ out) {
  k_mx_terms_body(vblk_self(), nmol, T, posfx, iperm, sL, nt, lj_tab, rc2, kappa, c2k, qf, epsRF,
                  pos_q, exptab, D, fix, facc, ticket, out);
}

// Up to this many sites the intramolecular terms run beside the pair kernel;
// above they follow it, as its blocks fill the SMs.  Beside it and after it, us a
// step: 1,500 sites 42.2 and 43.1, 4,095 48.4 and 53.7, 12,000 79.4 and 84.9, 16,200
// 101.0 and 98.7, 48,000 177.5 and 178.4, 96,000 304 and 298; only from 18,000
// (96.9 and 102.4) to 24,000 (108.1 and 114.3) is the line on the wrong side.
constexpr int kIntraBranchSites = 16384;

// blocks of k_mx_terms: a warp per 32 terms, blocks of two warps while those
// fit the SMs a few times (FP64 pipes bind: spread the warps)
constexpr int kTermThreads = 64;
static int term_blocks(const IntraTpl &T, int nmol) {
  const long warps = (long)(T.nx + T.nb + T.na) * ((nmol + 31) / 32);
  const long blocks = (warps + kTermThreads / 32 - 1) / (kTermThreads / 32);
  return (int)(blocks < 1 ? 1 : blocks > 1216 ? 1216 : blocks);
}

// combine the mixed kernels' sums into the reference's slots
__global__ void k_mx_slots(double *__restrict__ s, double erfc_rc_over_rc, int fused) {
  if (threadIdx.x != 0) return;
  mixed_slots_dev(s, erfc_rc_over_rc, fused);
}

// ---------------------------------------------------------------------------
// host side

// an inner list of rc + skin lies inside the outer one
static bool inner_possible(const Box *b) {
  return b->p.rc + b->mx->skin < (b->p.rclist < b->p.rclist_ew ? b->p.rclist : b->p.rclist_ew);
}

static int up(int **dst, const std::vector<int> &v) {
  FE_CUDA(cudaMalloc(dst, sizeof(int) * (v.empty() ? 1 : v.size())));
  if (!v.empty())
    FE_CUDA(cudaMemcpy(*dst, v.data(), sizeof(int) * v.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

// Largest plane (bytes of shared memory) the transform kernels take here: at
// 96^3 (76 KB, one plane per SM on 96 of them) they take 41 us where the
// library and its two passes take 49, but the step is 1 % slower (297.7 -> 300.5 us):
// the transforms run beside the pair kernel, whose blocks the wide ones displace.
// At 64^3 and below (34 KB) the replica batch gains 4 %.
constexpr size_t kMxPlaneMax = 48 * 1024;

struct BMxArgs;
// The transform kernels' shared memory, raised once to what any plan may take
// (one limit for all boxes, so that none lowers another's)
static int mx_fft_limits();

int mixed_setup(Box *b) {
  Mixed &M = *b->mx;
  int n = b->n;
  FE_CUDA(cudaDeviceGetAttribute(&M.nsm, cudaDevAttrMultiProcessorCount, b->dev));
  FE_CUDA(cudaStreamCreateWithFlags(&M.s2, cudaStreamNonBlocking));
  FE_CUDA(cudaEventCreateWithFlags(&M.ev_fork, cudaEventDisableTiming));
  FE_CUDA(cudaEventCreateWithFlags(&M.ev_join, cudaEventDisableTiming));
  FE_CUDA(cudaStreamCreateWithFlags(&M.s3, cudaStreamNonBlocking));
  FE_CUDA(cudaEventCreateWithFlags(&M.ev_intra, cudaEventDisableTiming));
  FE_CUDA(cudaMalloc(&M.facc3, sizeof(unsigned long long) * kFaccSlots));
  FE_CUDA(cudaMemset(M.facc3, 0, sizeof(unsigned long long) * kFaccSlots));
  FE_CUDA(cudaMalloc(&M.ticket3, sizeof(unsigned)));
  FE_CUDA(cudaMemset(M.ticket3, 0, sizeof(unsigned)));
  FE_CUDA(cudaMalloc(&M.facc2, sizeof(unsigned long long) * kFaccSlots));
  FE_CUDA(cudaMemset(M.facc2, 0, sizeof(unsigned long long) * kFaccSlots));
  FE_CUDA(cudaMalloc(&M.ticket2, sizeof(unsigned)));
  FE_CUDA(cudaMemset(M.ticket2, 0, sizeof(unsigned)));
  // cell grid of edge >= rlist / kListCellsPerReach
  double edge = (b->p.rclist > b->p.rclist_ew ? b->p.rclist : b->p.rclist_ew) / kListCellsPerReach;
  M.ncells = 1;
  for (int d = 0; d < 3; d++) {
    int m = (int)(b->p.L[d] / edge);
    M.nc[d] = m < 1 ? 1 : m;
    M.h[d] = b->p.L[d] / M.nc[d];
    M.ncells *= M.nc[d];
  }
  // the minimum image from wrapped 32-bit fractions needs |d| < L/2
  double rl = b->p.rclist;
  for (int d = 0; d < 3; d++)
    if (rl >= 0.5 * b->p.L[d]) {
      set_error("mixed precision needs rclist < L/2 in every direction");
      return FE_ERR_ARG;
    }
  FE_CUDA(cudaMalloc(&M.cell_count, sizeof(int) * M.ncells));
  // the counts are zero between list builds: each build clears them after
  // its scan (launch_mixed_list, k_b_mx_scan)
  FE_CUDA(cudaMemset(M.cell_count, 0, sizeof(int) * M.ncells));
  FE_CUDA(cudaMalloc(&M.cell_start, sizeof(int) * (M.ncells + 1)));
  FE_CUDA(cudaMalloc(&M.cell_fill, sizeof(int) * M.ncells));
  FE_CUDA(cudaMalloc(&M.cell_of, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.perm, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.iperm, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.cell_s, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.type_s, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.posfx, sizeof(int4) * n));
  // full-list row capacity: a sphere of rlist at the box's density, with margin
  double vol = b->p.L[0] * b->p.L[1] * b->p.L[2];
  double expect = 4.0 / 3.0 * kPI * rl * rl * rl * (double)n / vol;
  int cap = (int)(1.6 * expect + 64.0);
  if (b->p.max_neighbors > 0) cap = b->p.max_neighbors;
  cap = (cap + 31) / 32 * 32;
  if (cap > n) cap = (n + 31) / 32 * 32;
  M.cap = cap;
  FE_CUDA(cudaMalloc(&M.cnt_lj, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.cnt_nl, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.ent, sizeof(int) * (size_t)n * cap));
  FE_CUDA(cudaMalloc(&M.icnt_lj, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.icnt_nl, sizeof(int) * n));
  FE_CUDA(cudaMalloc(&M.ient, sizeof(int) * (size_t)n * cap));
  FE_CUDA(cudaMalloc(&M.snap, sizeof(int4) * n));
  FE_CUDA(cudaMalloc(&M.ps, sizeof(MxPruneState)));
  FE_CUDA(cudaMemset(M.ps, 0, sizeof(MxPruneState)));
  M.inner_on = n > kInnerMinSites && inner_possible(b);
  FE_CUDA(cudaMalloc(&M.fix, sizeof(unsigned long long) * 3 * n));
  // LJ table: eps, sig^2, and the energy shift constant (sr12s - 2 sr6s)
  int nt = b->nt;
  std::vector<double> eps(nt * nt), sig(nt * nt);
  FE_CUDA(cudaMemcpy(eps.data(), b->lj_eps, sizeof(double) * nt * nt, cudaMemcpyDeviceToHost));
  FE_CUDA(cudaMemcpy(sig.data(), b->lj_sig, sizeof(double) * nt * nt, cudaMemcpyDeviceToHost));
  std::vector<float> lj(nt * nt * 3);
  double rc2 = b->p.rc * b->p.rc;
  for (int k = 0; k < nt * nt; k++) {
    double s2 = sig[k] * sig[k];
    double sr2s = s2 / rc2, sr6s = sr2s * sr2s * sr2s;
    bool on = (eps[k] * sig[k]) != 0.0;
    lj[3 * k] = on ? (float)eps[k] : 0.f;
    lj[3 * k + 1] = (float)s2;
    lj[3 * k + 2] = (float)(sr6s * sr6s - 2.0 * sr6s);
  }
  FE_CUDA(cudaMalloc(&M.lj_tab, sizeof(float) * lj.size()));
  FE_CUDA(cudaMemcpy(M.lj_tab, lj.data(), sizeof(float) * lj.size(), cudaMemcpyHostToDevice));
  std::vector<unsigned char> on(nt * nt);
  for (int k = 0; k < nt * nt; k++) on[k] = lj[3 * k] != 0.f ? 1 : 0;
  FE_CUDA(cudaMalloc(&M.lj_on, on.size()));
  FE_CUDA(cudaMemcpy(M.lj_on, on.data(), on.size(), cudaMemcpyHostToDevice));
  if (nt <= 32) {  // lj_row[t'] bit t: pair (t, t') has an LJ term
    std::vector<unsigned> row(nt, 0u);
    for (int t = 0; t < nt; t++)
      for (int t2 = 0; t2 < nt; t2++)
        if (on[t * nt + t2]) row[t2] |= 1u << t;
    FE_CUDA(cudaMalloc(&M.lj_row, sizeof(unsigned) * nt));
    FE_CUDA(cudaMemcpy(M.lj_row, row.data(), sizeof(unsigned) * nt, cudaMemcpyHostToDevice));
  }
  // exclusion pair list (xint), for the correction kernel
  M.nexcl = b->p.nexcl;
  FE_CUDA(cudaMalloc(&M.excl_ab, sizeof(int) * 2 * (M.nexcl ? M.nexcl : 1)));
  FE_CUDA(cudaMalloc(&M.excl_flag, sizeof(int) * (M.nexcl ? M.nexcl : 1)));
  if (M.nexcl) {
    FE_CUDA(cudaMemcpy(M.excl_ab, b->p.excl_ab, sizeof(int) * 2 * M.nexcl, cudaMemcpyHostToDevice));
    FE_CUDA(cudaMemcpy(M.excl_flag, b->p.excl_flag, sizeof(int) * M.nexcl, cudaMemcpyHostToDevice));
  }  {
    // molecules for the fused intramolecular kernel: connected components of
    // bonds, bends and exclusions; usable when each is a contiguous run of
    // at most kIntraMaxSites sites
    std::vector<int> par(n);
    for (int i = 0; i < n; i++) par[i] = i;
    auto find = [&](int x) {
      while (par[x] != x) x = par[x] = par[par[x]];
      return x;
    };
    auto unite = [&](int x, int y) {
      x = find(x);
      y = find(y);
      if (x != y) par[x > y ? x : y] = x < y ? x : y;
    };
    const fe_box_params &pp = b->p;
    for (int t = 0; t < pp.nbond; t++) unite(pp.bond_ab[2 * t], pp.bond_ab[2 * t + 1]);
    for (int t = 0; t < pp.nbend; t++) {
      unite(pp.bend_abc[3 * t], pp.bend_abc[3 * t + 1]);
      unite(pp.bend_abc[3 * t + 1], pp.bend_abc[3 * t + 2]);
    }
    for (int t = 0; t < pp.nexcl; t++) unite(pp.excl_ab[2 * t], pp.excl_ab[2 * t + 1]);
    std::vector<int> first, mol_of(n);
    bool ok = true;
    for (int i = 0; i < n && ok; i++) {
      int r = find(i);
      if (i == 0 || r != find(i - 1)) {
        if (r != i) ok = false;  // a component that does not start here: not contiguous
        first.push_back(i);
      }
      mol_of[i] = (int)first.size() - 1;
    }
    first.push_back(n);
    int nm = (int)first.size() - 1;
    for (int m = 0; m < nm && ok; m++)
      if (first[m + 1] - first[m] > kIntraMaxSites) ok = false;
    if (ok && nm > 0) {
      auto csr = [&](int count, auto mol_fn, std::vector<int> &off, std::vector<int> &idx) {
        off.assign(nm + 1, 0);
        for (int t = 0; t < count; t++) off[mol_fn(t) + 1]++;
        for (int m = 0; m < nm; m++) off[m + 1] += off[m];
        std::vector<int> fill(off.begin(), off.end() - 1);
        idx.assign(count > 0 ? count : 1, 0);
        for (int t = 0; t < count; t++) idx[fill[mol_fn(t)]++] = t;
      };
      std::vector<int> xo, xi, bo, bi, ao, ai;
      csr(pp.nexcl, [&](int t) { return mol_of[pp.excl_ab[2 * t]]; }, xo, xi);
      csr(pp.nbond, [&](int t) { return mol_of[pp.bond_ab[2 * t]]; }, bo, bi);
      csr(pp.nbend, [&](int t) { return mol_of[pp.bend_abc[3 * t]]; }, ao, ai);
      int rc;
      if ((rc = up(&M.mol_first, first))) return rc;
      if ((rc = up(&M.mol_x, xo)) || (rc = up(&M.mol_xi, xi))) return rc;
      if ((rc = up(&M.mol_b, bo)) || (rc = up(&M.mol_bi, bi))) return rc;
      if ((rc = up(&M.mol_a, ao)) || (rc = up(&M.mol_ai, ai))) return rc;
      M.nmol = nm;
      M.intra_maxs = 1;
      for (int m = 0; m < nm; m++)
        if (first[m + 1] - first[m] > M.intra_maxs) M.intra_maxs = first[m + 1] - first[m];
      // all molecules alike?  (same size and, at the same relative sites,
      // the same exclusions, bonds, bends and site types)
      IntraTpl &T = M.tpl;
      memset(&T, 0, sizeof T);
      const int ns0 = first[1] - first[0];
      bool uni = xo[1] - xo[0] <= kTplTerms && bo[1] - bo[0] <= kTplTerms &&
                 ao[1] - ao[0] <= kTplTerms;
      T.ns = ns0;
      T.nx = xo[1] - xo[0];
      T.nb = bo[1] - bo[0];
      T.na = ao[1] - ao[0];
      for (int m = 0; m < nm && uni; m++) {
        const int lb = first[m];
        if (first[m + 1] - lb != ns0 || lb != m * ns0 || xo[m + 1] - xo[m] != T.nx ||
            bo[m + 1] - bo[m] != T.nb || ao[m + 1] - ao[m] != T.na) {
          uni = false;
          break;
        }
        for (int i = 0; i < ns0 && uni; i++) {
          if (m == 0) T.type[i] = pp.type[lb + i];
          else if (pp.type[lb + i] != T.type[i]) uni = false;
        }
        for (int k = 0; k < T.nx && uni; k++) {
          int x = xi[xo[m] + k];
          int a = pp.excl_ab[2 * x] - lb, c = pp.excl_ab[2 * x + 1] - lb, f = pp.excl_flag[x];
          if (m == 0) {
            T.xa[k] = a;
            T.xb[k] = c;
            T.xf[k] = f;
          } else if (a != T.xa[k] || c != T.xb[k] || f != T.xf[k]) {
            uni = false;
          }
        }
        for (int k = 0; k < T.nb && uni; k++) {
          int u = bi[bo[m] + k];
          int a = pp.bond_ab[2 * u] - lb, c = pp.bond_ab[2 * u + 1] - lb;
          float req = (float)pp.bond_req[u], kk = (float)pp.bond_k[u];
          float req_lo = (float)(pp.bond_req[u] - (double)req);
          if (m == 0) {
            T.ba[k] = a;
            T.bb[k] = c;
            T.breq[k] = req;
            T.breq_lo[k] = req_lo;
            T.bk[k] = kk;
          } else if (a != T.ba[k] || c != T.bb[k] || req != T.breq[k] ||
                     req_lo != T.breq_lo[k] || kk != T.bk[k]) {
            uni = false;
          }
        }
        for (int k = 0; k < T.na && uni; k++) {
          int u = ai[ao[m] + k];
          int a = pp.bend_abc[3 * u] - lb, c = pp.bend_abc[3 * u + 1] - lb,
              d = pp.bend_abc[3 * u + 2] - lb;
          float t0 = (float)pp.bend_theta0[u], kk = (float)pp.bend_k[u];
          float t0_lo = (float)(pp.bend_theta0[u] - (double)t0);
          if (m == 0) {
            T.aa[k] = a;
            T.ab[k] = c;
            T.ac[k] = d;
            T.at0[k] = t0;
            T.at0_lo[k] = t0_lo;
            T.ak[k] = kk;
          } else if (a != T.aa[k] || c != T.ab[k] || d != T.ac[k] || t0 != T.at0[k] ||
                     t0_lo != T.at0_lo[k] || kk != T.ak[k]) {
            uni = false;
          }
        }
      }
      M.uniform = uni;
    }
  }

  {
    // double-float constants of the intramolecular correction energy
    std::vector<float2> tab(kDfExpN);
    for (int k = kDfExpLo; k <= kDfExpHi; k++) {
      float hi, lo;
      df_split(exp((double)k / 64.0), hi, lo);
      tab[k - kDfExpLo] = make_float2(hi, lo);
    }
    FE_CUDA(cudaMalloc(&M.exptab, sizeof(float2) * kDfExpN));
    FE_CUDA(cudaMemcpy(M.exptab, tab.data(), sizeof(float2) * kDfExpN, cudaMemcpyHostToDevice));
    // ewald.c:817-836, constant term first
    const double c[10] = {-1.26551223, 1.00002368, 0.37409196, 0.09678418, -0.18628806,
                          0.27886807, -1.13520398, 1.48851587, -0.82215223, 0.17087277};
    for (int k = 0; k < 10; k++) df_split(c[k], M.dfi.C.c[k].x, M.dfi.C.c[k].y);
    df_split(b->p.kappa, M.dfi.kappa.x, M.dfi.kappa.y);
    df_split(kELEC * kELEQ * kELEQ * kNA * 1.0E-3, M.dfi.qf.x, M.dfi.qf.y);
    for (int d = 0; d < 3; d++) df_split(b->p.L[d] / kFixScale, M.dfi.sl[d].x, M.dfi.sl[d].y);
  }

  // SPME, FP32
  long K = b->K, Kh = b->Kh;
  std::vector<double> et(Kh), kw(Kh);
  FE_CUDA(cudaMemcpy(et.data(), b->eterm, sizeof(double) * Kh, cudaMemcpyDeviceToHost));
  FE_CUDA(cudaMemcpy(kw.data(), b->kweight, sizeof(double) * Kh, cudaMemcpyDeviceToHost));
  std::vector<float> etf(Kh), kwf(Kh);
  for (long i = 0; i < Kh; i++) {
    etf[i] = (float)et[i];
    kwf[i] = (float)kw[i];
  }
  FE_CUDA(cudaMalloc(&M.eterm32, sizeof(float) * Kh));
  FE_CUDA(cudaMalloc(&M.kw32, sizeof(float) * Kh));
  FE_CUDA(cudaMemcpy(M.eterm32, etf.data(), sizeof(float) * Kh, cudaMemcpyHostToDevice));
  FE_CUDA(cudaMemcpy(M.kw32, kwf.data(), sizeof(float) * Kh, cudaMemcpyHostToDevice));
  FE_CUDA(cudaMalloc(&M.grid32, sizeof(float) * K));
  FE_CUDA(cudaMalloc(&M.grid32k, sizeof(cufftComplex) * Kh));
  FE_CUDA(cudaMalloc(&M.floor3, sizeof(int) * 3 * n));
  FE_CUDA(cudaMalloc(&M.gfix, sizeof(unsigned long long) * b->K));
  FE_CUDA(cudaMemset(M.gfix, 0, sizeof(unsigned long long) * b->K));
  FE_CUDA(cudaMalloc(&M.sm, sizeof(float) * 3 * (size_t)n * b->order));
  FE_CUDA(cudaMalloc(&M.sd, sizeof(float) * 3 * (size_t)n * b->order));
  std::vector<Cx<float>> tw;
  M.fft_own = fft_plan<float>(b->G, &M.fft, &tw) &&
              fft_plane_smem<float>(b->G[1], b->G[2]) <= kMxPlaneMax;
  if (M.fft_own) {
    FE_CUDA(cudaMalloc(&M.fft_tw, sizeof(Cx<float>) * tw.size()));
    FE_CUDA(cudaMemcpy(M.fft_tw, tw.data(), sizeof(Cx<float>) * tw.size(),
                       cudaMemcpyHostToDevice));
    fft_set_twiddles<float>(&M.fft, M.fft_tw);
    M.fft.fix = M.gfix;
    M.fft.real = M.grid32;
    M.fft.spec = reinterpret_cast<Cx<float> *>(M.grid32k);
    M.fft.eterm = M.eterm32;
    M.fft.kw = M.kw32;
    return mx_fft_limits();
  }
  cufftResult r = cufftPlan3d(&M.plan_r2c, b->G[0], b->G[1], b->G[2], CUFFT_R2C);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftPlan3d R2C");
  r = cufftPlan3d(&M.plan_c2r, b->G[0], b->G[1], b->G[2], CUFFT_C2R);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftPlan3d C2R");
  M.plans = true;
  return FE_OK;
}

__global__ void k_b_mx_fft_forward(const BMxArgs *A, const int *off, int nbox);
__global__ void k_b_mx_fft_backward(const BMxArgs *A, const int *off, int nbox);
__global__ void k_b_mx_fft_convolve(const BMxArgs *A, const int *off, int nbox);

static int mx_fft_limits() {
  const int lim = (int)kFftSmemMax;
  FE_CUDA(cudaFuncSetAttribute(k_mx_fft_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  FE_CUDA(cudaFuncSetAttribute(k_mx_fft_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  FE_CUDA(cudaFuncSetAttribute(k_mx_fft_convolve, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  FE_CUDA(cudaFuncSetAttribute(k_b_mx_fft_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  FE_CUDA(cudaFuncSetAttribute(k_b_mx_fft_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  FE_CUDA(cudaFuncSetAttribute(k_b_mx_fft_convolve, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  return FE_OK;
}

void mixed_free(Box *b) {
  if (!b->mx) return;
  Mixed &M = *b->mx;
  void *ptrs[] = {M.cell_count, M.cell_start, M.cell_fill, M.cell_of, M.perm, M.iperm, M.cell_s,
                  M.type_s, M.posfx, M.cnt_lj, M.cnt_nl, M.ent, M.icnt_lj, M.icnt_nl,
                  M.ient, M.snap, M.ps, M.fix, M.lj_tab, M.lj_on, M.lj_row, M.excl_ab, M.excl_flag, M.eterm32, M.kw32,
                  M.grid32, M.grid32k, M.floor3, M.gfix, M.sm, M.sd, M.mol_first, M.mol_x,
                  M.mol_xi, M.mol_b, M.mol_bi, M.mol_a, M.mol_ai, M.exptab, M.facc2, M.ticket2,
                  M.fft_tw, M.facc3, M.ticket3};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (M.ev_fork) cudaEventDestroy(M.ev_fork);
  if (M.ev_join) cudaEventDestroy(M.ev_join);
  if (M.s2) cudaStreamDestroy(M.s2);
  if (M.ev_intra) cudaEventDestroy(M.ev_intra);
  if (M.s3) cudaStreamDestroy(M.s3);
  if (M.plans) {
    cufftDestroy(M.plan_r2c);
    cufftDestroy(M.plan_c2r);
  }
  delete b->mx;
  b->mx = nullptr;
}

void mixed_counts(Box *b, const int **lj, const int **rest) {
  *lj = b->mx->cnt_lj;
  *rest = b->mx->cnt_nl;
}

// possible: the radii leave room for an inner list.  Whether a small box has one
// is its own steps' affair (kInnerMinSites) and its batch's.
void mixed_inner_counts(Box *b, const int **lj, const int **rest, bool *possible) {
  *lj = b->mx->icnt_lj;
  *rest = b->mx->icnt_nl;
  *possible = inner_possible(b);
}

MxPruneState *mixed_prune_state(Box *b) { return b->mx->ps; }

static float3 fix_scale(Box *b) {
  return make_float3((float)(b->p.L[0] / kFixScale), (float)(b->p.L[1] / kFixScale),
                     (float)(b->p.L[2] / kFixScale));
}

static int launch_convert(Box *b, bool zero_forces = false) {
  Mixed &M = *b->mx;
  double3 invL = make_double3(1.0 / b->p.L[0], 1.0 / b->p.L[1], 1.0 / b->p.L[2]);
  k_mx_convert<<<(b->n + 255) / 256, 256, 0, b->stream>>>(
      b->n, b->pos_q, M.perm, invL, M.posfx, M.inner_on ? M.snap : nullptr, fix_scale(b),
      &M.ps->dmax2, zero_forces ? M.fix : nullptr);
  FE_LAUNCH_CHECK("k_mx_convert");
  return FE_OK;
}



int launch_mixed_list(Box *b) {
  Mixed &M = *b->mx;
  int n = b->n;
  double3 L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  double3 invL = make_double3(1.0 / b->p.L[0], 1.0 / b->p.L[1], 1.0 / b->p.L[2]);
  int3 nc = make_int3(M.nc[0], M.nc[1], M.nc[2]);
  k_mx_cell<<<(n + 255) / 256, 256, 0, b->stream>>>(n, b->pos_q, invL, nc, M.cell_of,
                                                    M.cell_count);
  FE_LAUNCH_CHECK("k_mx_cell");
  k_cell_scan_ext(M.cell_count, M.ncells, M.cell_start, M.cell_fill, b->stream);
  FE_CUDA(cudaMemsetAsync(M.cell_count, 0, sizeof(int) * M.ncells, b->stream));
  k_mx_fill<<<(n + 255) / 256, 256, 0, b->stream>>>(n, M.cell_of, M.cell_start, M.cell_fill, M.perm);
  FE_LAUNCH_CHECK("k_mx_fill");
  k_mx_cellsort<<<M.ncells, 32, 0, b->stream>>>(M.cell_start, M.perm, M.iperm, M.cell_s,
                                                 b->type, M.type_s, b->status);
  FE_LAUNCH_CHECK("k_mx_cellsort");
  int rc = launch_convert(b);
  if (rc) return rc;
  float3 Lf = make_float3((float)b->p.L[0], (float)b->p.L[1], (float)b->p.L[2]);
  float rl = (float)(b->p.rclist < b->p.rclist_ew ? b->p.rclist : b->p.rclist_ew);
  const int unit = list_unit(n), units = (n + unit - 1) / unit;
  const int want = (units + kMxWarps - 1) / kMxWarps;
  const int blocks = want < M.nsm * 8 ? want : M.nsm * 8;
#define FE_LIST(U)                                                                               \
  k_mx_list<U><<<blocks, kMxWarps * 32, 0, b->stream>>>(                                         \
      n, M.posfx, M.perm, M.iperm, M.cell_s, M.type_s, M.cell_start, nc, fix_scale(b), Lf, rl,   \
      b->nt, M.lj_row, M.lj_on, b->x_start, b->x_partner, M.cap, M.cnt_lj, M.cnt_nl, M.ent,      \
      b->status)
  if (unit == 8) FE_LIST(8);
  else if (unit == 4) FE_LIST(4);
  else FE_LIST(1);
#undef FE_LIST
  FE_LAUNCH_CHECK("k_mx_list");
  // the inner list and its snapshot belong to the old sort: prune next
  FE_CUDA(cudaMemsetAsync(&M.ps->need, 0x01, sizeof(int), b->stream));
  b->have_list = true;
  return FE_OK;
}

static int pair_blocks(Box *b, int nw) {
  int blocks = (b->n + nw - 1) / nw;
  const int most = b->mx->nsm * kPairRW / nw;  // one resident wave
  return blocks > most ? most : blocks;
}

MxPair mx_pair_params(Box *b) {
  Mixed &M = *b->mx;
  MxPair P;
  P.n = b->n;
  P.nt = b->nt;
  P.cap = M.cap;
  P.rc2 = (float)(b->p.rc * b->p.rc);
  P.khalf = (float)(0.5 * b->p.kappa);
  P.mk2 = (float)(-b->p.kappa * b->p.kappa * 1.4426950408889634);
  P.c2k = (float)(2.0 * b->p.kappa / sqrt(kPI));
  double qf = kELEC * kELEQ * kELEQ * kNA * 1.0E-3;
  P.qfe = (float)(qf / b->p.epsRF);
  double ron2 = b->p.r_switch > 0.0 ? b->p.r_switch * b->p.r_switch : 0.0;
  double rc2 = b->p.rc * b->p.rc;
  P.ron2 = (float)ron2;
  P.inv_sw_den = ron2 > 0.0 ? (float)(1.0 / ((rc2 - ron2) * (rc2 - ron2) * (rc2 - ron2))) : 0.f;
  P.sc = fix_scale(b);
  P.cubic = (b->p.L[0] == b->p.L[1] && b->p.L[1] == b->p.L[2]) ? 1 : 0;
  P.s2 = P.sc.x * P.sc.x;
  double rp = b->p.rc + M.skin, hs = 0.5 * M.skin - 1e-4;
  P.rp2 = (float)(rp * rp);
  P.thresh2 = (float)(hs * hs);
  P.inner_on = M.inner_on ? 1 : 0;
  return P;
}

int launch_mx_pair_only(Box *b) {
  Mixed &M = *b->mx;
  MxPair P = mx_pair_params(b);
  size_t shm = sizeof(float) * (b->nt * b->nt * 3);
  int nw = M.tune_nw, blocks = M.tune_blocks > 0 ? M.tune_blocks : pair_blocks(b, nw);
#define FE_PAIR_ARGS                                                                          \
  P, M.posfx, M.type_s, M.perm, M.cnt_lj, M.cnt_nl, M.ent, M.icnt_lj, M.icnt_nl, M.ient, M.snap, \
      M.ps, M.lj_tab, M.fix, b->facc, b->ticket, b->scal + SC_MX_PAIR, b->status
  if (M.inner_on) {
    // the pruning variant: 64 registers, one resident wave of 8-warp blocks
    k_mx_pair<8, true><<<M.nsm * 4, 256, shm, b->stream>>>(FE_PAIR_ARGS);
    FE_LAUNCH_CHECK("k_mx_pair<prune>");
  }
#define FE_PAIR_LAUNCH(NWV) \
  k_mx_pair<NWV, false><<<blocks, NWV * 32, shm, b->stream>>>(FE_PAIR_ARGS)
  if (nw == 4) FE_PAIR_LAUNCH(4);
  else if (nw == 16) FE_PAIR_LAUNCH(16);
  else FE_PAIR_LAUNCH(8);
#undef FE_PAIR_LAUNCH
#undef FE_PAIR_ARGS
  FE_LAUNCH_CHECK("k_mx_pair");
  return FE_OK;
}

// Chooses the pair kernel's launch shape for this box: warps per block in
// {4, 8, 16} and the grid size
// (multiples of the SM count, or one warp per row), each timed with CUDA
// events on the box's stream over the current (inner) list; the fastest is
// kept.
// Forces and energies must be recomputed after.
int mixed_autotune(Box *b, int *nw_out, int *rw_out, int *blocks_out, double *us_out) {
  Mixed &M = *b->mx;
  int nsm = 0;
  FE_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, b->dev));
  const int nws[3] = {4, 8, 16};
  cudaEvent_t e0, e1;
  FE_CUDA(cudaEventCreate(&e0));
  FE_CUDA(cudaEventCreate(&e1));
  int best_nw = M.tune_nw, best_blocks = M.tune_blocks;
  float best = 1e30f;
  int rc = FE_OK;
  for (int c = 0; c < 3 && rc == FE_OK; c++) {
    int nw = nws[c];
    int full = (b->n + nw - 1) / nw;
    int grids[6] = {nsm * 4, nsm * 8, nsm * 12, nsm * 16, nsm * 24, full};
    for (int g = 0; g < 6 && rc == FE_OK; g++) {
      int blocks = grids[g] < full ? grids[g] : full;
      M.tune_nw = nw;
      M.tune_blocks = blocks;
      if ((rc = launch_mx_pair_only(b))) break;  // warm-up
      cudaEventRecord(e0, b->stream);
      for (int r = 0; r < 3 && rc == FE_OK; r++) rc = launch_mx_pair_only(b);
      cudaEventRecord(e1, b->stream);
      cudaError_t e = cudaEventSynchronize(e1);
      if (e != cudaSuccess) {
        rc = cuda_fail(e, "mixed_autotune");
        break;
      }
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best) {
        best = ms;
        best_nw = nw;
        best_blocks = blocks;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  M.tune_nw = best_nw;
  M.tune_blocks = best_blocks;
  if (rc) return rc;
  if (nw_out) *nw_out = best_nw;
  if (rw_out) *rw_out = kPairRW;
  if (blocks_out) *blocks_out = best_blocks;
  if (us_out) *us_out = 1000.0 * best / 3.0;
  return FE_OK;
}

static int spread_on(Box *b, cudaStream_t st) {
  Mixed &M = *b->mx;
  int3 G = make_int3(b->G[0], b->G[1], b->G[2]);
  long nt = (long)b->n * b->order;
  if (b->order == 4) {
    k_mx_spread_o4<<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(b->n, G, M.posfx, M.gfix);
    FE_LAUNCH_CHECK("k_mx_spread_o4");
  } else {
    k_mx_spread_red<<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(
        b->n, b->order, G, M.posfx, M.sm, M.floor3, M.gfix);
    FE_LAUNCH_CHECK("k_mx_spread_red");
  }
  return FE_OK;
}

static int fix2grid_on(Box *b, cudaStream_t st) {
  Mixed &M = *b->mx;
  k_mx_fix2grid<<<M.nsm * 8, 256, 0, st>>>(b->K, M.gfix, M.grid32);
  FE_LAUNCH_CHECK("k_mx_fix2grid");
  return FE_OK;
}

int launch_mx_spread_only(Box *b) {
  int rc = spread_on(b, b->stream);
  return rc ? rc : fix2grid_on(b, b->stream);
}

// The charge sums convolved in reciprocal space: grid sums in, potential grid
// out, the energy sum into SC_ENREC
static int convolve_on(Box *b, cudaStream_t st, unsigned long long *facc, unsigned *ticket) {
  Mixed &M = *b->mx;
  if (M.fft_own) {
    const int gx = b->G[0], gy = b->G[1], gz = b->G[2];
    const int pt = fft_plane_threads(gy, gz);
    const size_t ps = fft_plane_smem<float>(gy, gz);
    k_mx_fft_forward<<<gx, pt, ps, st>>>(M.fft);
    FE_LAUNCH_CHECK("k_mx_fft_forward");
    k_mx_fft_convolve<<<fft_line_blocks(gy, gz, M.fft.tile), fft_line_threads(gx, M.fft.tile),
                        fft_line_smem<float>(gx, M.fft.tile), st>>>(M.fft, facc, ticket,
                                                                    b->scal + SC_ENREC);
    FE_LAUNCH_CHECK("k_mx_fft_convolve");
    k_mx_fft_backward<<<gx, pt, ps, st>>>(M.fft);
    FE_LAUNCH_CHECK("k_mx_fft_backward");
    return FE_OK;
  }
  int rc = fix2grid_on(b, st);
  if (rc) return rc;
  cufftResult r = cufftSetStream(M.plan_r2c, st);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftSetStream");
  r = cufftExecR2C(M.plan_r2c, M.grid32, M.grid32k);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftExecR2C");
  int kb = (int)((b->Kh + 255) / 256);
  if (kb > 1024) kb = 1024;
  k_mx_recip<<<kb, 256, 0, st>>>(b->Kh, M.eterm32, M.kw32, M.grid32k, facc, ticket,
                                 b->scal + SC_ENREC);
  FE_LAUNCH_CHECK("k_mx_recip");
  r = cufftSetStream(M.plan_c2r, st);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftSetStream");
  r = cufftExecC2R(M.plan_c2r, M.grid32k, M.grid32);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftExecC2R");
  return FE_OK;
}

// The reciprocal-space forces and energy (pme_calc's work) on stream st with
// the reduction slots facc / ticket: [splines,] spreading, FFT, convolution,
// inverse FFT, gather.  It reads the fixed-point coordinates and adds to the
// force sums with integer atomics, so it may run beside the pair kernel.
static int spme_on(Box *b, cudaStream_t st, unsigned long long *facc, unsigned *ticket) {
  Mixed &M = *b->mx;
  const int n = b->n;
  int rc;
  int3 G = make_int3(b->G[0], b->G[1], b->G[2]);
  if (b->order != 4) {  // order 4 computes its weights inside spreading and gathering
    k_mx_splines<<<(n + 127) / 128, 128, 0, st>>>(n, b->order, G, M.posfx, M.floor3, M.sm,
                                                  M.sd);
    FE_LAUNCH_CHECK("k_mx_splines");
  }
  if ((rc = spread_on(b, st))) return rc;
  if ((rc = convolve_on(b, st, facc, ticket))) return rc;
  double qf = kELEC * kELEQ * kELEQ * kNA * 1.0E-3;
  float3 gl = make_float3((float)(b->G[0] / b->p.L[0]), (float)(b->G[1] / b->p.L[1]),
                          (float)(b->G[2] / b->p.L[2]));
  int gb = (n + 127) / 128;
  if (gb > 1024) gb = 1024;
  float qfe = (float)(qf / b->p.epsRF);
  if (b->order == 4) {
    if (n <= kGatherLanesSites)
      k_mx_gather_o4<4><<<std::min((4 * n + 127) / 128, 1024), 128, 0, st>>>(
          n, G, gl, qfe, M.posfx, M.perm, M.grid32, M.fix, facc, ticket, b->scal + SC_FMEAN);
    else
      k_mx_gather_o4<1><<<gb, 128, 0, st>>>(n, G, gl, qfe, M.posfx, M.perm, M.grid32, M.fix, facc,
                                            ticket, b->scal + SC_FMEAN);
    FE_LAUNCH_CHECK("k_mx_gather_o4");
  } else {
    k_mx_gather<<<gb, 128, 0, st>>>(n, b->order, G, gl, qfe, M.posfx, M.perm, M.floor3, M.sm,
                                    M.sd, M.grid32, M.fix, facc, ticket, b->scal + SC_FMEAN);
    FE_LAUNCH_CHECK("k_mx_gather");
  }
  return FE_OK;
}

// The intramolecular terms (exclusion corrections, 1-4 pairs, bonds, bends)
// on stream st with the reduction slots facc / ticket: one thread per
// molecule when the topology allows, else kernels over the exclusion and
// bonded lists.  Integer atomics into the force sums.
static int intra_on(Box *b, cudaStream_t st, unsigned long long *facc, unsigned *ticket) {
  Mixed &M = *b->mx;
  double qf = kELEC * kELEQ * kELEQ * kNA * 1.0E-3;
  // intramolecular terms: one thread per molecule when the topology allows,
  // else the exclusion and bonded kernels
  float3 sL = fix_scale(b);
  const DfIntra &dfi = M.dfi;
  if (M.nmol > 0) {
    const int mb = std::min((M.nmol + 31) / 32, 8192);  // one warp a block: FP64 pipes bind
#define FE_INTRA_ARGS                                                                           \
  M.nmol, M.mol_first, M.mol_x, M.mol_xi, M.mol_b, M.mol_bi, M.mol_a, M.mol_ai, M.excl_ab,        \
      M.excl_flag, b->bond_ab, b->bond_req, b->bond_k, b->bend_abc, b->bend_t0, b->bend_k,        \
      M.posfx, M.iperm, b->type, sL, b->nt, M.lj_tab, (float)(b->p.rc * b->p.rc),                 \
      (float)b->p.kappa, (float)(2.0 * b->p.kappa / sqrt(kPI)), (float)qf, (float)b->p.epsRF,     \
      b->pos_q, M.exptab, dfi, M.fix, facc, ticket, b->scal + SC_MX_INTRA
    if (M.uniform) {
      k_mx_terms<<<term_blocks(M.tpl, M.nmol), kTermThreads, 0, st>>>(
          M.nmol, M.tpl, M.posfx, M.iperm, sL, b->nt, M.lj_tab, (float)(b->p.rc * b->p.rc),
          (float)b->p.kappa, (float)(2.0 * b->p.kappa / sqrt(kPI)), (float)qf,
          (float)b->p.epsRF, b->pos_q, M.exptab, dfi, M.fix, facc, ticket,
          b->scal + SC_MX_INTRA);
    }
    else if (M.intra_maxs <= 3) k_mx_intra<3><<<mb, 32, 0, st>>>(FE_INTRA_ARGS);
    else if (M.intra_maxs <= 4) k_mx_intra<4><<<mb, 32, 0, st>>>(FE_INTRA_ARGS);
    else k_mx_intra<kIntraMaxSites><<<mb, 32, 0, st>>>(FE_INTRA_ARGS);
#undef FE_INTRA_ARGS
    FE_LAUNCH_CHECK("k_mx_intra");
  } else {
    int xb = (M.nexcl + 255) / 256;
    if (xb > 1024) xb = 1024;
    if (xb < 1) xb = 1;
    k_mx_excl<<<xb, 256, 0, st>>>(M.nexcl, M.excl_ab, M.excl_flag, M.posfx, M.iperm,
                                         b->type, sL, b->nt, M.lj_tab,
                                         (float)(b->p.rc * b->p.rc), (float)b->p.kappa,
                                         (float)(2.0 * b->p.kappa / sqrt(kPI)), (float)qf,
                                         (float)b->p.epsRF, b->pos_q, M.exptab, dfi, M.fix,
                                         facc, ticket, b->scal + SC_MX_EXCL);
    FE_LAUNCH_CHECK("k_mx_excl");
    int tot = b->nbond + b->nbend;
    int bb = (tot + 255) / 256;
    if (bb > 1024) bb = 1024;
    if (bb < 1) bb = 1;
    const double3 sd = make_double3((double)dfi.sl[0].x + (double)dfi.sl[0].y,
                                    (double)dfi.sl[1].x + (double)dfi.sl[1].y,
                                    (double)dfi.sl[2].x + (double)dfi.sl[2].y);
    k_mx_bonded<<<bb, 256, 0, st>>>(b->nbond, b->nbend, sL, sd, M.posfx, M.iperm, b->bond_ab,
                                           b->bond_req, b->bond_k, b->bend_abc, b->bend_t0,
                                           b->bend_k, M.fix, facc, ticket,
                                           b->scal + SC_BOND);
    FE_LAUNCH_CHECK("k_mx_bonded");
  }
  return FE_OK;
}

int forces_mixed(Box *b, bool prepared) {
  Mixed &M = *b->mx;
  int n = b->n;
  int rc;
  if (!prepared && (rc = launch_convert(b, true))) return rc;  // also clears the force sums
  // reciprocal space on the second stream and, in boxes that leave SMs free,
  // the intramolecular terms on the third, beside the pair kernel
  FE_CUDA(cudaEventRecord(M.ev_fork, b->stream));
  FE_CUDA(cudaStreamWaitEvent(M.s2, M.ev_fork, 0));
  if ((rc = spme_on(b, M.s2, M.facc2, M.ticket2))) return rc;
  FE_CUDA(cudaEventRecord(M.ev_join, M.s2));
  const bool branch = n <= kIntraBranchSites;
  if (branch) {
    FE_CUDA(cudaStreamWaitEvent(M.s3, M.ev_fork, 0));
    if ((rc = intra_on(b, M.s3, M.facc3, M.ticket3))) return rc;
    FE_CUDA(cudaEventRecord(M.ev_intra, M.s3));
  }
  if ((rc = launch_mx_pair_only(b))) return rc;
  if (!branch && (rc = intra_on(b, b->stream, M.facc3, M.ticket3))) return rc;
  // Urey-Bradley, torsions and impropers (FP64, into the fixed-point sums)
  if ((rc = launch_bonded_ext_mixed(b))) return rc;
  if (branch) FE_CUDA(cudaStreamWaitEvent(b->stream, M.ev_intra, 0));
  FE_CUDA(cudaStreamWaitEvent(b->stream, M.ev_join, 0));
  if (b->fold_tail) return FE_OK;  // finalised inside the second half kick
  k_mx_finalize<<<(3 * n + 255) / 256, 256, 0, b->stream>>>(n, M.fix, b->scal, b->ff);
  FE_LAUNCH_CHECK("k_mx_finalize");
  return launch_mixed_assemble(b);
}

// ---------------------------------------------------------------------------
// Replica batches: every box's force evaluation in one launch per kernel.
// Box r of a launch owns blocks off[r] .. off[r+1]-1 and runs the same kernel
// body as its own launch would, on its own buffers (the per-box arguments
// are kept in device memory); its reductions finish in its own last block.
// Where the transform kernels do not take every box's grid, the grids of boxes of
// equal shape sit side by side so that one batched library plan transforms them.

struct BMxArgs {
  int n, nt, nmol, order;
  const double4 *pos;
  const int *perm, *iperm, *type, *type_s;
  double3 invL;
  int4 *posfx;
  int4 *snap;
  float3 sc;
  MxPruneState *ps;
  // facc2 / ticket2: the reciprocal branch's, facc3 / ticket3: the intramolecular one's
  unsigned long long *fix, *facc, *facc2, *facc3;
  unsigned *ticket, *ticket2, *ticket3;
  double *scal;
  int *status;
  // pair
  MxPair P;
  const int *cnt_lj, *cnt_nl, *ent;
  int *icnt_lj, *icnt_nl, *ient;
  const float *lj_tab;
  // intramolecular
  const int *mol_first, *mol_x, *mol_xi, *mol_b, *mol_bi, *mol_a, *mol_ai, *excl_ab, *excl_flag;
  const int *bond_ab, *bend_abc;
  const double *bond_req, *bond_k, *bend_t0, *bend_k;
  float rc2, kappa, c2k, qf, epsRF;
  const float2 *exptab;
  DfIntra D;
  IntraTpl tpl;
  // list rebuild
  int3 nc;
  int ncells;
  int *cell_count, *cell_start, *cell_fill, *cell_of, *cell_s;
  int *perm_w, *iperm_w, *type_s_w;
  float3 Lf;
  float rlist;
  const unsigned *lj_row;
  const unsigned char *lj_on;
  const int *x_start, *x_partner;
  int cap;
  int *cnt_lj_w, *cnt_nl_w, *ent_w;
  // SPME
  int3 G;
  long K, Kh;
  int *floor3;
  float *sm, *sd;
  unsigned long long *gfix;
  float *grid32;
  cufftComplex *grid32k;
  const float *eterm32, *kw32;
  FftBox<float> fft;
  float3 gl;
  float qfe;
};

template <bool PRUNE>
__global__ void __launch_bounds__(256, kPairRW / 8)
k_b_mx_pair(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_pair_body<8, PRUNE>(
      vblk_of(off, r), a.P, a.posfx, a.type_s, a.perm, a.cnt_lj, a.cnt_nl, a.ent, a.icnt_lj,
      a.icnt_nl, a.ient, a.snap, a.ps, a.lj_tab, a.fix, a.facc, a.ticket, a.scal + SC_MX_PAIR,
      a.status);
}

template <int NS>
__global__ void k_b_mx_intra(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                             int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_intra_body<NS>(vblk_of(off, r), a.nmol, a.mol_first, a.mol_x, a.mol_xi, a.mol_b, a.mol_bi,
                      a.mol_a, a.mol_ai, a.excl_ab, a.excl_flag, a.bond_ab, a.bond_req, a.bond_k,
                      a.bend_abc, a.bend_t0, a.bend_k, a.posfx, a.iperm, a.type, a.sc, a.nt,
                      a.lj_tab, a.rc2, a.kappa, a.c2k, a.qf, a.epsRF, a.pos, a.exptab, a.D, a.fix,
                      a.facc3, a.ticket3, a.scal + SC_MX_INTRA);
}

__global__ void k_b_mx_terms(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                             int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_terms_body(vblk_of(off, r), a.nmol, a.tpl, a.posfx, a.iperm, a.sc, a.nt, a.lj_tab, a.rc2,
                  a.kappa, a.c2k, a.qf, a.epsRF, a.pos, a.exptab, a.D, a.fix, a.facc3, a.ticket3,
                  a.scal + SC_MX_INTRA);
}

__global__ void k_b_mx_splines(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                               int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_splines_body(vblk_of(off, r), a.n, a.order, a.G, a.posfx, a.floor3, a.sm, a.sd);
}

__global__ void k_b_mx_spread(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                              int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_spread_red_body(vblk_of(off, r), a.n, a.order, a.G, a.posfx, a.sm, a.floor3, a.gfix);
}

__global__ void k_b_mx_spread_o4(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                               int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_spread_o4_body(vblk_of(off, r), a.n, a.G, a.posfx, a.gfix);
}

__global__ void k_b_mx_gather_o4(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                               int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_gather_o4_body<1>(vblk_of(off, r), a.n, a.G, a.gl, a.qfe, a.posfx, a.perm, a.grid32, a.fix,
                    a.facc2, a.ticket2, a.scal + SC_FMEAN);
}

__global__ void k_b_mx_fix2grid(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                                int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_fix2grid_body(vblk_of(off, r), a.K, a.gfix, a.grid32);
}

__global__ void k_b_mx_recip(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                             int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_recip_body(vblk_of(off, r), a.Kh, a.eterm32, a.kw32, a.grid32k, a.facc2, a.ticket2,
                  a.scal + SC_ENREC);
}

__global__ void __launch_bounds__(512)
k_b_mx_fft_forward(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  extern __shared__ float4 fft_sh[];
  const int r = vblk_box(off, nbox);
  fft_forward_body<float>(A[r].fft, vblk_of(off, r).id, reinterpret_cast<Cx<float> *>(fft_sh));
}
__global__ void __launch_bounds__(512)
k_b_mx_fft_backward(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  extern __shared__ float4 fft_sh[];
  const int r = vblk_box(off, nbox);
  fft_backward_body<float>(A[r].fft, vblk_of(off, r).id, reinterpret_cast<Cx<float> *>(fft_sh));
}
__global__ void __launch_bounds__(256)
k_b_mx_fft_convolve(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  extern __shared__ float4 fft_sh[];
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  const VBlk vb = vblk_of(off, r);
  float v[1] = {fft_convolve_body<float>(a.fft, vb.id, reinterpret_cast<Cx<float> *>(fft_sh))};
  block_fix_final<1>(v, 24, a.facc2, a.ticket2, a.scal + SC_ENREC, vb);
}

__global__ void k_b_mx_gather(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                              int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_gather_body(vblk_of(off, r), a.n, a.order, a.G, a.gl, a.qfe, a.posfx, a.perm, a.floor3,
                   a.sm, a.sd, a.grid32, a.fix, a.facc2, a.ticket2, a.scal + SC_FMEAN);
}

// list rebuild of every box: cells, scan, fill, sort within cells, the
// fixed-point coordinates and the outer list (launch_mixed_list for each box)
__global__ void k_b_mx_cell(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_cell_body(vblk_of(off, r), a.n, a.pos, a.invL, a.nc, a.cell_of, a.cell_count);
}

// exclusive prefix of the cell counts (one block of 1024 threads per box,
// as k_cell_scan); fill counters cleared, counts cleared for the next build
__global__ void __launch_bounds__(1024) k_b_mx_scan(const BMxArgs *__restrict__ A) {
  const BMxArgs &a = A[blockIdx.x];
  int t = threadIdx.x, T = blockDim.x;
  int chunk = (a.ncells + T - 1) / T;
  int lo = min(t * chunk, a.ncells), hi = min(lo + chunk, a.ncells);
  int sum = 0;
  for (int c = lo; c < hi; c++) sum += a.cell_count[c];
  int total;
  int acc = block_exclusive_scan(sum, &total);
  if (t == 0) a.cell_start[a.ncells] = total;
  for (int c = lo; c < hi; c++) {
    a.cell_start[c] = acc;
    a.cell_fill[c] = 0;
    acc += a.cell_count[c];
    a.cell_count[c] = 0;
  }
}

__global__ void k_b_mx_fill(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_fill_body(vblk_of(off, r), a.n, a.cell_of, a.cell_start, a.cell_fill, a.perm_w);
}

__global__ void k_b_mx_cellsort(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                                int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  const VBlk vb = vblk_of(off, r);
  // the inner list and its snapshot belong to the old sort: prune next
  if (vb.id == 0 && threadIdx.x == 0) a.ps->need = 1;
  k_mx_cellsort_body(vb, a.cell_start, a.perm_w, a.iperm_w, a.cell_s, a.type, a.type_s_w,
                     a.status);
}

__global__ void k_b_mx_convert_only(const BMxArgs *__restrict__ A, const int *__restrict__ off,
                                    int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_convert_body(vblk_of(off, r), a.n, a.pos, a.perm, a.invL, a.posfx,
                    a.P.inner_on ? a.snap : nullptr, a.sc, &a.ps->dmax2);
}

template <int kListUnit>
__global__ void __launch_bounds__(kMxWarps * 32, kListBlocksPerSM)
k_b_mx_list(const BMxArgs *__restrict__ A, const int *__restrict__ off, int nbox) {
  const int r = vblk_box(off, nbox);
  const BMxArgs &a = A[r];
  k_mx_list_body<kListUnit>(vblk_of(off, r), a.n, a.posfx, a.perm, a.iperm, a.cell_s, a.type_s,
                 a.cell_start, a.nc, a.sc, a.Lf, a.rlist, a.nt, a.lj_row, a.lj_on, a.x_start,
                 a.x_partner, a.cap, a.cnt_lj_w, a.cnt_nl_w, a.ent_w, a.status);
}

struct BMxGroup {
  int G[3];
  int count = 0;
  float *real = nullptr;
  cufftComplex *cplx = nullptr;
  cufftHandle r2c = 0, c2r = 0;
  bool plans = false;
};

// block offsets of one kernel over the batch (device copy)
struct BMxRange {
  int *d_off = nullptr;
  int total = 0;
};

struct BMxPlan {
  int nbox = 0;
  BMxArgs *d_args = nullptr;
  BMxRange convert, prune, pair, intra, splines, spread, fix2grid, recip, gather;
  BMxRange cell, fill, cellsort, list;
  // every box's grid takes the transform kernels: planes and x tiles of all boxes
  bool fft_own = true;
  BMxRange planes, lines, terms;
  // Every box has identical molecules and their terms alone don't fill the SMs:
  // k_b_mx_terms (168,000 sites: 760 us a step with it, 752 by molecule)
  bool uniform = true;
  bool inner_on = false;  // some box has an inner list
  std::vector<char> inner;  // which
  bool branch = true;  // intramolecular terms beside the pair kernel
  int unit = 8;  // sites per warp of the list build
  cudaStream_t s3 = nullptr;
  cudaEvent_t ev_intra = nullptr;
  size_t plane_shm = 0, line_shm = 0;
  int intra_ns = 3;
  bool order4 = true;  // every box has B-spline order 4: weights computed in place
  // the reciprocal branch's stream and its fork / join events
  cudaStream_t s2 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  size_t pair_shm = 0;
  std::vector<BMxGroup> groups;
};

static int bmx_range(BMxRange &R, const std::vector<int> &blocks) {
  std::vector<int> off(blocks.size() + 1, 0);
  for (size_t r = 0; r < blocks.size(); r++) off[r + 1] = off[r] + blocks[r];
  R.total = off.back();
  FE_CUDA(cudaMalloc(&R.d_off, sizeof(int) * off.size()));
  FE_CUDA(cudaMemcpy(R.d_off, off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

void mixed_batch_free(BMxPlan *P) {
  if (!P) return;
  cudaFree(P->d_args);
  BMxRange *rs[] = {&P->convert, &P->prune, &P->pair, &P->intra, &P->splines, &P->spread,
                    &P->fix2grid, &P->recip, &P->gather, &P->cell, &P->fill,
                    &P->cellsort, &P->list, &P->planes, &P->lines, &P->terms};
  for (BMxRange *r : rs) cudaFree(r->d_off);
  if (P->ev_fork) cudaEventDestroy(P->ev_fork);
  if (P->ev_join) cudaEventDestroy(P->ev_join);
  if (P->s2) cudaStreamDestroy(P->s2);
  if (P->s3) cudaStreamDestroy(P->s3);
  if (P->ev_intra) cudaEventDestroy(P->ev_intra);
  for (BMxGroup &g : P->groups) {
    if (g.plans) {
      cufftDestroy(g.r2c);
      cufftDestroy(g.c2r);
    }
    cudaFree(g.real);
    cudaFree(g.cplx);
  }
  delete P;
}

MxPrepare mixed_prepare(Box *b, bool have_list, bool inner_on) {
  MxPrepare m;
  Mixed &M = *b->mx;
  m.iperm = have_list ? M.iperm : nullptr;
  m.posfx = M.posfx;
  m.snap = inner_on ? M.snap : nullptr;
  m.dmax2 = &M.ps->dmax2;
  m.fix = M.fix;
  m.invL = make_double3(1.0 / b->p.L[0], 1.0 / b->p.L[1], 1.0 / b->p.L[2]);
  m.sc = fix_scale(b);
  return m;
}

void mixed_bint_fields(Box *b, BIntArgs *a) {
  if (!b->mx) return;
  a->erfc_rc_over_rc = b->mx->erfc_rc_over_rc;
  a->mixed_fused = b->mx->nmol > 0 ? 1 : 0;
  a->fix = b->mx->fix;
}

bool mixed_batch_inner(const BMxPlan *P, int r) { return P->inner[r]; }

// The batched force evaluation needs mixed-precision boxes whose molecules
// are contiguous runs of sites (the fused intramolecular kernel); otherwise
// FE_ERR_ARG and the batch steps box by box.
int mixed_batch_plan(Box *const *boxes, int nbox, BMxPlan **out) {
  *out = nullptr;
  for (int r = 0; r < nbox; r++)
    if (!boxes[r]->mx || boxes[r]->mx->nmol == 0 || boxes[r]->mx->intra_maxs > kIntraMaxSites) {
      set_error("batched force evaluation: mixed-precision boxes of contiguous molecules only");
      return FE_ERR_ARG;
    }
  for (int r = 0; r < nbox; r++)
    if (boxes[r]->nurey + boxes[r]->ntors + boxes[r]->nimpr > 0) {
      set_error("batched force evaluation: boxes with Urey-Bradley, torsion or improper terms "
                "run box by box");
      return FE_ERR_ARG;
    }
  BMxPlan *P = new BMxPlan();
  P->nbox = nbox;
  FE_CUDA(cudaStreamCreateWithFlags(&P->s2, cudaStreamNonBlocking));
  FE_CUDA(cudaStreamCreateWithFlags(&P->s3, cudaStreamNonBlocking));
  FE_CUDA(cudaEventCreateWithFlags(&P->ev_intra, cudaEventDisableTiming));
  FE_CUDA(cudaEventCreateWithFlags(&P->ev_fork, cudaEventDisableTiming));
  FE_CUDA(cudaEventCreateWithFlags(&P->ev_join, cudaEventDisableTiming));
  std::vector<BMxArgs> args(nbox);
  std::vector<int> bconv, bprune, bpair, bintra, bspl, bspr, bf2g, brec, bgat;
  std::vector<int> bcell, bfill, bsort, blist, bplane, bline, bterms;
  double qf = kELEC * kELEQ * kELEQ * kNA * 1.0E-3;
  int rc = FE_OK;
  long sites = 0;
  for (int r = 0; r < nbox; r++) sites += boxes[r]->n;
  for (int r = 0; r < nbox && rc == FE_OK; r++) {
    Box *b = boxes[r];
    Mixed &M = *b->mx;
    BMxArgs &a = args[r];
    memset(&a, 0, sizeof a);
    a.n = b->n;
    a.nt = b->nt;
    a.nmol = M.nmol;
    a.order = b->order;
    a.pos = b->pos_q;
    a.perm = M.perm;
    a.iperm = M.iperm;
    a.type = b->type;
    a.type_s = M.type_s;
    a.invL = make_double3(1.0 / b->p.L[0], 1.0 / b->p.L[1], 1.0 / b->p.L[2]);
    a.posfx = M.posfx;
    a.snap = M.snap;
    a.sc = fix_scale(b);
    a.ps = M.ps;
    a.fix = M.fix;
    a.facc = b->facc;
    a.ticket = b->ticket;
    a.facc2 = M.facc2;
    a.ticket2 = M.ticket2;
    a.facc3 = M.facc3;
    a.ticket3 = M.ticket3;
    a.tpl = M.tpl;
    if (!M.uniform || sites > kIntraBranchSites) P->uniform = false;
    a.scal = b->scal;
    a.status = b->status;
    a.P = mx_pair_params(b);
    // rows and lists as one box of all the batch's sites would have them
    a.P.inner_on = sites > kInnerMinSites && inner_possible(b) ? 1 : 0;
    P->inner.push_back(a.P.inner_on != 0);
    P->branch = sites <= kIntraBranchSites;
    if (a.P.inner_on) P->inner_on = true;
    a.cnt_lj = M.cnt_lj;
    a.cnt_nl = M.cnt_nl;
    a.ent = M.ent;
    a.icnt_lj = M.icnt_lj;
    a.icnt_nl = M.icnt_nl;
    a.ient = M.ient;
    a.lj_tab = M.lj_tab;
    a.mol_first = M.mol_first;
    a.mol_x = M.mol_x;
    a.mol_xi = M.mol_xi;
    a.mol_b = M.mol_b;
    a.mol_bi = M.mol_bi;
    a.mol_a = M.mol_a;
    a.mol_ai = M.mol_ai;
    a.excl_ab = M.excl_ab;
    a.excl_flag = M.excl_flag;
    a.bond_ab = b->bond_ab;
    a.bend_abc = b->bend_abc;
    a.bond_req = b->bond_req;
    a.bond_k = b->bond_k;
    a.bend_t0 = b->bend_t0;
    a.bend_k = b->bend_k;
    a.rc2 = (float)(b->p.rc * b->p.rc);
    a.kappa = (float)b->p.kappa;
    a.c2k = (float)(2.0 * b->p.kappa / sqrt(kPI));
    a.qf = (float)qf;
    a.epsRF = (float)b->p.epsRF;
    a.exptab = M.exptab;
    a.D = M.dfi;
    a.G = make_int3(b->G[0], b->G[1], b->G[2]);
    a.K = b->K;
    a.Kh = b->Kh;
    a.floor3 = M.floor3;
    a.sm = M.sm;
    a.sd = M.sd;
    a.gfix = M.gfix;
    a.fft = M.fft;
    if (!M.fft_own) P->fft_own = false;
    a.eterm32 = M.eterm32;
    a.kw32 = M.kw32;
    a.gl = make_float3((float)(b->G[0] / b->p.L[0]), (float)(b->G[1] / b->p.L[1]),
                       (float)(b->G[2] / b->p.L[2]));
    a.qfe = (float)(qf / b->p.epsRF);
    a.nc = make_int3(M.nc[0], M.nc[1], M.nc[2]);
    a.ncells = M.ncells;
    a.cell_count = M.cell_count;
    a.cell_start = M.cell_start;
    a.cell_fill = M.cell_fill;
    a.cell_of = M.cell_of;
    a.cell_s = M.cell_s;
    a.perm_w = M.perm;
    a.iperm_w = M.iperm;
    a.type_s_w = M.type_s;
    a.Lf = make_float3((float)b->p.L[0], (float)b->p.L[1], (float)b->p.L[2]);
    a.rlist = (float)(b->p.rclist < b->p.rclist_ew ? b->p.rclist : b->p.rclist_ew);
    a.lj_row = M.lj_row;
    a.lj_on = M.lj_on;
    a.x_start = b->x_start;
    a.x_partner = b->x_partner;
    a.cap = M.cap;
    a.cnt_lj_w = M.cnt_lj;
    a.cnt_nl_w = M.cnt_nl;
    a.ent_w = M.ent;
    // the grid of equal shapes side by side (the group buffers are set below)
    int gi = -1;
    for (size_t g = 0; g < P->groups.size(); g++)
      if (P->groups[g].G[0] == b->G[0] && P->groups[g].G[1] == b->G[1] &&
          P->groups[g].G[2] == b->G[2])
        gi = (int)g;
    if (gi < 0) {
      P->groups.push_back(BMxGroup());
      gi = (int)P->groups.size() - 1;
      for (int d = 0; d < 3; d++) P->groups[gi].G[d] = b->G[d];
    }
    a.grid32 = reinterpret_cast<float *>((size_t)gi);                        // group index,
    a.grid32k = reinterpret_cast<cufftComplex *>((size_t)P->groups[gi].count);  // slot in it
    P->groups[gi].count++;
    if (M.intra_maxs > P->intra_ns) P->intra_ns = M.intra_maxs;
    size_t shm = sizeof(float) * (b->nt * b->nt * 3);
    if (shm > P->pair_shm) P->pair_shm = shm;
    int nsm = M.nsm > 0 ? M.nsm : 152;
    bconv.push_back((b->n + 255) / 256);
    bprune.push_back(std::max(1, std::min(4 * nsm, b->n / 160)));
    bpair.push_back(std::max(1, std::min(2048, b->n / 80)));
    bintra.push_back(std::min(2048, (M.nmol + 127) / 128));
    bterms.push_back(term_blocks(M.tpl, M.nmol));
    bspl.push_back((b->n + 127) / 128);
    bspr.push_back((int)(((long)b->n * b->order + 255) / 256));
    bf2g.push_back((int)std::min<long>(8L * nsm, (b->K / 2 + 255) / 256 + 1));
    brec.push_back((int)std::min<long>(1024L, (b->Kh + 255) / 256));
    bgat.push_back(std::min(1024, (b->n + 127) / 128));
    if (M.fft_own) {
      bplane.push_back(b->G[0]);
      bline.push_back(fft_line_blocks(b->G[1], b->G[2], M.fft.tile));
      P->plane_shm = std::max(P->plane_shm, fft_plane_smem<float>(b->G[1], b->G[2]));
      P->line_shm = std::max(P->line_shm, fft_line_smem<float>(b->G[0], M.fft.tile));
    }
    if (b->order != 4) P->order4 = false;
    bcell.push_back((b->n + 255) / 256);
    bfill.push_back((b->n + 255) / 256);
    bsort.push_back(M.ncells);
    P->unit = list_unit(sites);
    int units = (b->n + P->unit - 1) / P->unit;
    int lb = (units + kMxWarps - 1) / kMxWarps;
    blist.push_back(std::max(1, std::min(lb, nsm * 8)));
  }
  // The transform kernels work on each box's own grids; with a size they do
  // not take among the boxes, all use the library:
  // group buffers and batched plans; each box's grid points into its group.
  // Real grids start every Kpad floats (K rounded up to 4: 16-byte aligned,
  // as the grid kernels' paired float stores need for odd K).
  if (P->fft_own) {
    P->groups.clear();
    for (int r = 0; r < nbox; r++) {
      args[r].grid32 = boxes[r]->mx->grid32;
      args[r].grid32k = boxes[r]->mx->grid32k;
    }
    if (rc == FE_OK) rc = bmx_range(P->planes, bplane);
    if (rc == FE_OK) rc = bmx_range(P->lines, bline);
  }
  for (BMxGroup &g : P->groups) {
    if (rc) break;
    long K = (long)g.G[0] * g.G[1] * g.G[2], Kh = (long)g.G[0] * g.G[1] * (g.G[2] / 2 + 1);
    long Kpad = (K + 3) / 4 * 4;
    if (cudaMalloc(&g.real, sizeof(float) * Kpad * g.count) != cudaSuccess ||
        cudaMalloc(&g.cplx, sizeof(cufftComplex) * Kh * g.count) != cudaSuccess) {
      rc = cuda_fail(cudaGetLastError(), "batch grid buffers");
      break;
    }
    int nn[3] = {g.G[0], g.G[1], g.G[2]};
    int nh[3] = {g.G[0], g.G[1], g.G[2] / 2 + 1};
    cufftResult fr = cufftPlanMany(&g.r2c, 3, nn, nn, 1, (int)Kpad, nh, 1, (int)Kh, CUFFT_R2C,
                                   g.count);
    if (fr == CUFFT_SUCCESS)
      fr = cufftPlanMany(&g.c2r, 3, nn, nh, 1, (int)Kh, nn, 1, (int)Kpad, CUFFT_C2R, g.count);
    if (fr != CUFFT_SUCCESS) {
      rc = cufft_fail(fr, "cufftPlanMany (batch)");
      break;
    }
    g.plans = true;
  }
  if (rc == FE_OK && !P->fft_own)
    for (int r = 0; r < nbox; r++) {
      size_t gi = reinterpret_cast<size_t>(args[r].grid32);
      size_t slot = reinterpret_cast<size_t>(args[r].grid32k);
      BMxGroup &g = P->groups[gi];
      long K = (long)g.G[0] * g.G[1] * g.G[2], Kh = (long)g.G[0] * g.G[1] * (g.G[2] / 2 + 1);
      long Kpad = (K + 3) / 4 * 4;
      args[r].grid32 = g.real + slot * Kpad;
      args[r].grid32k = g.cplx + slot * Kh;
    }
  if (rc == FE_OK && cudaMalloc(&P->d_args, sizeof(BMxArgs) * nbox) != cudaSuccess)
    rc = cuda_fail(cudaGetLastError(), "batch arguments");
  if (rc == FE_OK &&
      cudaMemcpy(P->d_args, args.data(), sizeof(BMxArgs) * nbox, cudaMemcpyHostToDevice) !=
          cudaSuccess)
    rc = cuda_fail(cudaGetLastError(), "batch arguments");
  if (rc == FE_OK) rc = bmx_range(P->convert, bconv);
  if (rc == FE_OK) rc = bmx_range(P->prune, bprune);
  if (rc == FE_OK) rc = bmx_range(P->pair, bpair);
  if (rc == FE_OK) rc = bmx_range(P->intra, bintra);
  if (rc == FE_OK) rc = bmx_range(P->terms, bterms);
  if (rc == FE_OK) rc = bmx_range(P->splines, bspl);
  if (rc == FE_OK) rc = bmx_range(P->spread, bspr);
  if (rc == FE_OK) rc = bmx_range(P->fix2grid, bf2g);
  if (rc == FE_OK) rc = bmx_range(P->recip, brec);
  if (rc == FE_OK) rc = bmx_range(P->gather, bgat);
  if (rc == FE_OK) rc = bmx_range(P->cell, bcell);
  if (rc == FE_OK) rc = bmx_range(P->fill, bfill);
  if (rc == FE_OK) rc = bmx_range(P->cellsort, bsort);
  if (rc == FE_OK) rc = bmx_range(P->list, blist);
  if (rc) {
    mixed_batch_free(P);
    return rc;
  }
  *out = P;
  return FE_OK;
}

// The list rebuild of every box (launch_mixed_list for each); the cell
// counts are zero on entry and left at zero by the scan.
int mixed_batch_list(BMxPlan *P, cudaStream_t s) {
  const int nb = P->nbox;
  k_b_mx_cell<<<P->cell.total, 256, 0, s>>>(P->d_args, P->cell.d_off, nb);
  FE_LAUNCH_CHECK("k_b_mx_cell");
  k_b_mx_scan<<<nb, 1024, 0, s>>>(P->d_args);
  FE_LAUNCH_CHECK("k_b_mx_scan");
  k_b_mx_fill<<<P->fill.total, 256, 0, s>>>(P->d_args, P->fill.d_off, nb);
  FE_LAUNCH_CHECK("k_b_mx_fill");
  k_b_mx_cellsort<<<P->cellsort.total, 32, 0, s>>>(P->d_args, P->cellsort.d_off, nb);
  FE_LAUNCH_CHECK("k_b_mx_cellsort");
  k_b_mx_convert_only<<<P->convert.total, 256, 0, s>>>(P->d_args, P->convert.d_off, nb);
  FE_LAUNCH_CHECK("k_b_mx_convert_only");
  if (P->unit == 8) k_b_mx_list<8><<<P->list.total, kMxWarps * 32, 0, s>>>(P->d_args, P->list.d_off, nb);
  else if (P->unit == 4) k_b_mx_list<4><<<P->list.total, kMxWarps * 32, 0, s>>>(P->d_args, P->list.d_off, nb);
  else k_b_mx_list<1><<<P->list.total, kMxWarps * 32, 0, s>>>(P->d_args, P->list.d_off, nb);
  FE_LAUNCH_CHECK("k_b_mx_list");
  return FE_OK;
}

// One force evaluation of every box (forces_mixed for each, energies
// assembled later by the batched second half kick).
// Force sums of every box from the coordinates k_b_vv1 prepared; k_b_vv2 turns
// them into forces.
int mixed_batch_forces(BMxPlan *P, cudaStream_t s) {
  const int nb = P->nbox;
  // reciprocal space of every box on the second stream, beside the pair kernel
  cudaStream_t s2 = P->s2;
  FE_CUDA(cudaEventRecord(P->ev_fork, s));
  FE_CUDA(cudaStreamWaitEvent(s2, P->ev_fork, 0));
  if (P->order4) {
    k_b_mx_spread_o4<<<P->spread.total, 256, 0, s2>>>(P->d_args, P->spread.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_spread_o4");
  } else {
    k_b_mx_splines<<<P->splines.total, 128, 0, s2>>>(P->d_args, P->splines.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_splines");
    k_b_mx_spread<<<P->spread.total, 256, 0, s2>>>(P->d_args, P->spread.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_spread");
  }
  if (P->fft_own) {
    k_b_mx_fft_forward<<<P->planes.total, 512, P->plane_shm, s2>>>(P->d_args, P->planes.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_fft_forward");
    k_b_mx_fft_convolve<<<P->lines.total, 256, P->line_shm, s2>>>(P->d_args, P->lines.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_fft_convolve");
    k_b_mx_fft_backward<<<P->planes.total, 512, P->plane_shm, s2>>>(P->d_args, P->planes.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_fft_backward");
  } else {
    k_b_mx_fix2grid<<<P->fix2grid.total, 256, 0, s2>>>(P->d_args, P->fix2grid.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_fix2grid");
    for (BMxGroup &g : P->groups) {
      cufftResult r = cufftSetStream(g.r2c, s2);
      if (r == CUFFT_SUCCESS) r = cufftExecR2C(g.r2c, g.real, g.cplx);
      if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftExecR2C (batch)");
    }
    k_b_mx_recip<<<P->recip.total, 256, 0, s2>>>(P->d_args, P->recip.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_recip");
    for (BMxGroup &g : P->groups) {
      cufftResult r = cufftSetStream(g.c2r, s2);
      if (r == CUFFT_SUCCESS) r = cufftExecC2R(g.c2r, g.cplx, g.real);
      if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftExecC2R (batch)");
    }
  }
  if (P->order4) {
    k_b_mx_gather_o4<<<P->gather.total, 128, 0, s2>>>(P->d_args, P->gather.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_gather_o4");
  } else {
    k_b_mx_gather<<<P->gather.total, 128, 0, s2>>>(P->d_args, P->gather.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_gather");
  }
  FE_CUDA(cudaEventRecord(P->ev_join, s2));
  // the intramolecular terms on the third, or after the pair kernel, as in
  // forces_mixed
  cudaStream_t s3 = P->branch ? P->s3 : s;
  auto intra = [&]() -> int {
    if (P->uniform) k_b_mx_terms<<<P->terms.total, kTermThreads, 0, s3>>>(P->d_args, P->terms.d_off, nb);
    else if (P->intra_ns <= 3) k_b_mx_intra<3><<<P->intra.total, 128, 0, s3>>>(P->d_args, P->intra.d_off, nb);
    else if (P->intra_ns <= 4) k_b_mx_intra<4><<<P->intra.total, 128, 0, s3>>>(P->d_args, P->intra.d_off, nb);
    else k_b_mx_intra<kIntraMaxSites><<<P->intra.total, 128, 0, s3>>>(P->d_args, P->intra.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_intra");
    return FE_OK;
  };
  int rc = FE_OK;
  if (P->branch) {
    FE_CUDA(cudaStreamWaitEvent(s3, P->ev_fork, 0));
    if ((rc = intra())) return rc;
    FE_CUDA(cudaEventRecord(P->ev_intra, s3));
  }
  // real space
  if (P->inner_on) {
    k_b_mx_pair<true><<<P->prune.total, 256, P->pair_shm, s>>>(P->d_args, P->prune.d_off, nb);
    FE_LAUNCH_CHECK("k_b_mx_pair<prune>");
  }
  k_b_mx_pair<false><<<P->pair.total, 256, P->pair_shm, s>>>(P->d_args, P->pair.d_off, nb);
  FE_LAUNCH_CHECK("k_b_mx_pair");
  if (P->branch) FE_CUDA(cudaStreamWaitEvent(s, P->ev_intra, 0));
  else if ((rc = intra())) return rc;
  FE_CUDA(cudaStreamWaitEvent(s, P->ev_join, 0));
  return FE_OK;
}

int launch_mixed_assemble(Box *b) {
  k_mx_slots<<<1, 32, 0, b->stream>>>(b->scal, b->mx->erfc_rc_over_rc, b->mx->nmol > 0 ? 1 : 0);
  FE_LAUNCH_CHECK("k_mx_slots");
  return launch_assemble_energies(b, 1);
}

}  // namespace fe
