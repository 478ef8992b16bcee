// k_nblist.cu -- the Verlet-list build of nblist(ibox) (nblist.c:32-592) on
// the device.  Compiled with -fmad=false: the distance test below performs
// exactly the reference's roundings, so the pair set is bit-exact.
//
// Layout: a cell grid whose edge is at least half of max(rclist, rclist_ew)
// (the whole of it where the box is so sparse that finer cells would outnumber
// its sites), binned as CSR (count -> scan -> fill) with a sorted copy of the
// sites' 32-bit fixed-point coordinates.  One warp per site a walks the cell
// columns within reach (z neighbours are contiguous) and tests every b > a by
// an FP32 distance, 1/64 of the FP64 test's cost on this part; only candidates
// within the FP32 test's margin of the cutoff, and those of sites outside the
// box, take the reference's FP64 test, so the pair set is still the
// reference's.  The row is sorted by b -- bitonic in registers, consecutive
// keys per lane so that two thirds of the steps stay within a lane -- and
// written into the padded row nl_ent[a * max_nb ...], the layout of the
// reference's nlist[k].list[a][max_num_neighbors], with the xint flag packed
// as entry = b * 8 + xflag (nblist.c:149-183).
#include <climits>
#include <cmath>

#include "fe_device.cuh"

namespace fe {

constexpr int kListWarps = 4;        // warps per block
constexpr int kListBuf = 2048;       // candidates a warp can hold (per row)

// 32-bit fixed-point coordinates (x / L + 1/2 as a fraction of 2^32); w = the
// site, with the top bit set when it lies outside the box
__global__ void k_cell_count(const double4 *__restrict__ pos, int n, double3 L, int3 nc,
                             int4 *__restrict__ fx, int *__restrict__ cell_of,
                             int *__restrict__ cell_count) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = pos[i];
  const double s = 4294967296.0;
  unsigned ux = (unsigned)(unsigned long long)__double2ll_rn((p.x / L.x + 0.5) * s);
  unsigned uy = (unsigned)(unsigned long long)__double2ll_rn((p.y / L.y + 0.5) * s);
  unsigned uz = (unsigned)(unsigned long long)__double2ll_rn((p.z / L.z + 0.5) * s);
  bool in = fabs(p.x) <= 0.5 * L.x && fabs(p.y) <= 0.5 * L.y && fabs(p.z) <= 0.5 * L.z;
  int cx = (int)(((unsigned long long)ux * (unsigned)nc.x) >> 32);
  int cy = (int)(((unsigned long long)uy * (unsigned)nc.y) >> 32);
  int cz = (int)(((unsigned long long)uz * (unsigned)nc.z) >> 32);
  int c = (cx * nc.y + cy) * nc.z + cz;
  fx[i] = make_int4((int)ux, (int)uy, (int)uz, in ? i : i | INT_MIN);
  cell_of[i] = c;
  atomicAdd(&cell_count[c], 1);
}

// exclusive scan of cell_count into cell_start[0..ncells] (one block)
__global__ void k_cell_scan(const int *__restrict__ count, int ncells, int *__restrict__ start,
                            int *__restrict__ fill) {
  int t = threadIdx.x, T = blockDim.x;
  int chunk = (ncells + T - 1) / T;
  int lo = min(t * chunk, ncells), hi = min(lo + chunk, ncells);
  int s = 0;
  for (int c = lo; c < hi; c++) s += count[c];
  int total;
  int acc = block_exclusive_scan(s, &total);
  if (t == 0) start[ncells] = total;
  for (int c = lo; c < hi; c++) {
    start[c] = acc;
    fill[c] = 0;
    acc += count[c];
  }
}

__global__ void k_cell_fill(int n, const int *__restrict__ cell_of, const int *__restrict__ start,
                            int *__restrict__ fill, const int4 *__restrict__ fx,
                            int4 *__restrict__ sorted) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c = cell_of[i];
  int s = atomicAdd(&fill[c], 1);
  sorted[start[c] + s] = fx[i];
}

// the xint entry of the pair, -1 without one
__device__ __forceinline__ int excl_entry_of(const int *__restrict__ xs,
                                             const int *__restrict__ xp, int a, int b) {
  // the last matching entry wins, as in the hash scan of nblist.c:160-172
  int f = -1;
  for (int p = xs[a]; p < xs[a + 1]; p++)
    if (xp[p] == b) f = p;
  return f;
}

// nblist.c:116-145,178: component rejections, then dr2, in FP64
__device__ __forceinline__ bool list_test(double4 pa, double4 pb, double3 L, double hx, double hy,
                                          double hz, double rcut, double rcut2, double rcut2_ew) {
  double dx = fabs(pa.x - pb.x);
  if (dx > hx) dx -= L.x;
  if (dx > rcut) return false;
  double dy = fabs(pa.y - pb.y);
  if (dy > hy) dy -= L.y;
  if (dy > rcut) return false;
  double dz = fabs(pa.z - pb.z);
  if (dz > hz) dz -= L.z;
  if (dz > rcut) return false;
  double dr2 = dx * dx + dy * dy + dz * dz;
  return (dr2 < rcut2_ew) && (dr2 < rcut2);
}

__device__ __forceinline__ void list_order(int &a, int &b, bool up) {
  int lo = min(a, b), hi = max(a, b);
  a = up ? lo : hi;
  b = up ? hi : lo;
}

// bitonic sort of 32 R keys of a warp, lane l holding keys l R .. l R + R - 1
template <int R>
__device__ __forceinline__ void list_sort(int (&v)[R], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= R) {  // partner in another lane
        const bool up = ((lane * R) & k) == 0, lower = (lane & (j / R)) == 0;
#pragma unroll
        for (int r = 0; r < R; r++) {
          int o = __shfl_xor_sync(0xffffffffu, v[r], j / R);
          v[r] = up == lower ? min(v[r], o) : max(v[r], o);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++)
          if ((r & j) == 0) {
            const bool up = k < R ? (r & k) == 0 : ((lane * R) & k) == 0;
            list_order(v[r], v[r | j], up);
          }
      }
    }
  }
}

template <int R>
__device__ __forceinline__ void list_sort_buf(int *buf, int count, int lane) {
  int v[R];
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = lane * R + r < count ? buf[lane * R + r] : INT_MAX;
  __syncwarp();
  list_sort<R>(v, lane);
#pragma unroll
  for (int r = 0; r < R; r++)
    if (lane * R + r < count) buf[lane * R + r] = v[r];
  __syncwarp();
}

struct ListParams {
  double3 L;
  double rcut, rcut2, rcut2_ew;
  int3 nc;
  int reach;      // cells per cutoff: neighbours within +-reach
  float3 sc;      // L / 2^32 per axis
  float3 h;       // cell edges
  float ra2;      // columns further than this are out of reach
  float in2, out2;  // FP32 distances surely inside / outside the cutoff
  int n, max_nb;
};

// first cell and number of cells of the neighbourhood of cell c along an axis
__device__ __forceinline__ void list_window(int c, int nc, int reach, int &first, int &count) {
  if (nc > 2 * reach) {
    first = c - reach;
    count = 2 * reach + 1;
  } else {
    first = 0;
    count = nc;
  }
}
// gap between coordinate x in [0, L) and cell c (unwrapped) of edge h
__device__ __forceinline__ float list_gap(float x, int c, float h) {
  return fmaxf(fmaxf(c * h - x, x - (c + 1) * h), 0.f);
}

__global__ void __launch_bounds__(kListWarps * 32)
k_list(ListParams P, const double4 *__restrict__ pos, const int4 *__restrict__ fx,
       const int *__restrict__ cell_of, const int *__restrict__ cstart,
       const int4 *__restrict__ sorted, const int *__restrict__ xs, const int *__restrict__ xp,
       const int *__restrict__ xf, const int *__restrict__ xi, int *__restrict__ count,
       int *__restrict__ ent, int2 *__restrict__ xl, int *__restrict__ status) {
  __shared__ int sbuf[kListWarps][kListBuf];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int *buf = sbuf[w];
  const unsigned lt = (1u << lane) - 1u;
  const double hx = P.L.x / 2.0, hy = P.L.y / 2.0, hz = P.L.z / 2.0;
  const int3 nc = P.nc;
  for (int a = blockIdx.x * kListWarps + w; a < P.n; a += gridDim.x * kListWarps) {
    const int4 fa = fx[a];
    const bool aout = fa.w < 0;
    const int ca = cell_of[a];
    int x0, nx, y0, ny, z0, nz;
    list_window(ca / (nc.z * nc.y), nc.x, P.reach, x0, nx);
    list_window((ca / nc.z) % nc.y, nc.y, P.reach, y0, ny);
    list_window(ca % nc.z, nc.z, P.reach, z0, nz);
    const bool allx = nc.x <= 2 * P.reach, ally = nc.y <= 2 * P.reach;
    const float X = __uint2float_rn((unsigned)fa.x) * P.sc.x,
                Y = __uint2float_rn((unsigned)fa.y) * P.sc.y;
    // the z window as one or two runs of cells
    int za = z0 < 0 ? z0 + nc.z : z0, zn = min(nz, nc.z - za), zr = nz - zn;
    int cnt = 0;
    for (int ix = 0; ix < nx; ix++) {
      const int xu = x0 + ix, xc = xu < 0 ? xu + nc.x : xu >= nc.x ? xu - nc.x : xu;
      const float gx = allx ? 0.f : list_gap(X, xu, P.h.x);
      for (int iy = 0; iy < ny; iy++) {
        const int yu = y0 + iy, yc = yu < 0 ? yu + nc.y : yu >= nc.y ? yu - nc.y : yu;
        const float gy = ally ? 0.f : list_gap(Y, yu, P.h.y);
        if (gx * gx + gy * gy > P.ra2) continue;
        const int *cs = cstart + (xc * nc.y + yc) * nc.z;
        const int a0 = cs[za], la = cs[za + zn] - a0;
        const int b0 = zr > 0 ? cs[0] : 0, lb = zr > 0 ? cs[zr] - b0 : 0;
        for (int base = 0; base < la + lb; base += 32) {
          const int v = base + lane;
          bool ok = false;
          int b = 0;
          if (v < la + lb) {
            const int4 f = sorted[v < la ? a0 + v : b0 + (v - la)];
            b = f.w & INT_MAX;
            if (b > a) {
              const float dx = __int2float_rn((int)((unsigned)fa.x - (unsigned)f.x)) * P.sc.x;
              const float dy = __int2float_rn((int)((unsigned)fa.y - (unsigned)f.y)) * P.sc.y;
              const float dz = __int2float_rn((int)((unsigned)fa.z - (unsigned)f.z)) * P.sc.z;
              const float r2 = dx * dx + dy * dy + dz * dz;
              ok = r2 < P.out2;
              if (ok && (r2 > P.in2 || aout || f.w < 0))
                ok = list_test(pos[a], pos[b], P.L, hx, hy, hz, P.rcut, P.rcut2, P.rcut2_ew);
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, ok);
          if (ok) {
            const int p = cnt + __popc(m & lt);
            if (p < kListBuf) buf[p] = b;
          }
          cnt += __popc(m);
        }
      }
    }
    __syncwarp();
    const int mcount = cnt < kListBuf ? cnt : kListBuf;
    if (mcount <= 128) list_sort_buf<4>(buf, mcount, lane);
    else if (mcount <= 256) list_sort_buf<8>(buf, mcount, lane);
    else if (mcount <= 512) list_sort_buf<16>(buf, mcount, lane);
    else if (mcount <= 1024) list_sort_buf<32>(buf, mcount, lane);
    else {
      for (int i = mcount + lane; i < kListBuf; i += 32) buf[i] = INT_MAX;
      __syncwarp();
      for (int k = 2; k <= kListBuf; k <<= 1)
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
          for (int i = lane; i < kListBuf; i += 32) {
            int ixj = i ^ jj;
            if (ixj > i) {
              int vi = buf[i], vj = buf[ixj];
              if ((vi > vj) == ((i & k) == 0)) {
                buf[i] = vj;
                buf[ixj] = vi;
              }
            }
          }
          __syncwarp();
        }
    }
    int rowlen = mcount < P.max_nb ? mcount : P.max_nb;
    if (cnt > P.max_nb || cnt > kListBuf) {
      if (lane == 0) atomicOr(status, ST_LIST_OVERFLOW);
    }
    int *row = ent + (size_t)a * P.max_nb;
    for (int i = lane; i < rowlen; i += 32) {
      int b = buf[i];
      const int x = excl_entry_of(xs, xp, a, b);
      const int e = b * 8 + (x < 0 ? 0 : xf[x]);
      row[i] = e;
      if (e & 7) xl[xi[x]] = make_int2(a, e);
    }
    if (lane == 0) count[a] = rowlen;
    __syncwarp();
  }
}

void k_cell_scan_ext(const int *count, int ncells, int *start, int *fill, cudaStream_t s) {
  k_cell_scan<<<1, 1024, 0, s>>>(count, ncells, start, fill);
  ++g_launches;
}

int nblist_setup(Box *b) {
  double cut = b->p.rclist > b->p.rclist_ew ? b->p.rclist : b->p.rclist_ew;
  cut *= (1.0 + 1e-6);  // cells come from 32-bit fractions
  // cells of half a cutoff (2900 candidates per site of water instead of 5100
  // with whole ones), unless that makes far more cells than sites
  for (b->list_reach = 2; b->list_reach > 0; b->list_reach--) {
    double cells = 1.0;
    for (int d = 0; d < 3; d++) {
      double m = floor(b->p.L[d] * b->list_reach / cut);
      b->nc[d] = m < 1.0 ? 1 : m > 1024.0 ? 1024 : (int)m;
      cells *= b->nc[d];
    }
    b->ncells = b->nc[0] * b->nc[1] * b->nc[2];
    if (cells <= 4.0 * b->n + 4096.0 || b->list_reach == 1) break;
  }
  // the cell counts and, after them, the excluded pairs: one memset
  const size_t xl0 = ((size_t)b->ncells + 1) & ~(size_t)1;
  b->cell_bytes = sizeof(int) * xl0 + sizeof(int2) * (size_t)b->nexcl;
  FE_CUDA(cudaMalloc(&b->cell_count, b->cell_bytes));
  FE_CUDA(cudaMemset(b->cell_count, 0, b->cell_bytes));
  b->xl = reinterpret_cast<int2 *>(b->cell_count + xl0);
  FE_CUDA(cudaMalloc(&b->cell_start, sizeof(int) * (b->ncells + 1)));
  FE_CUDA(cudaMalloc(&b->cell_fill, sizeof(int) * b->ncells));
  FE_CUDA(cudaMalloc(&b->cell_sorted, sizeof(int4) * b->n));
  FE_CUDA(cudaMalloc(&b->pfx, sizeof(int4) * b->n));
  FE_CUDA(cudaMalloc(&b->cell_of, sizeof(int) * b->n));
  int mnb = b->p.max_neighbors;
  if (mnb <= 0) mnb = b->n < 2000 ? b->n : 1500;  // allocate.c:321-322
  if (mnb > kListBuf) mnb = kListBuf;
  if (mnb < 1) mnb = 1;
  b->max_nb = mnb;
  FE_CUDA(cudaMalloc(&b->nl_count, sizeof(int) * b->n));
  FE_CUDA(cudaMalloc(&b->nl_ent, sizeof(int) * (size_t)b->n * mnb));
  FE_CUDA(cudaMemsetAsync(b->nl_count, 0, sizeof(int) * b->n, b->stream));
  return FE_OK;
}

// nblist.c:607-647 (DLIST): whether any site of [lb, ub) has moved more than
// (rclist - rc) / 4 from its position at the last list build, along one axis
// or in distance, with the reference's per-axis image rule (|d| > half box:
// subtract the box length)
__global__ void k_nl_check(int lb, int ub, double3 L, double3 H, double rcut, double rcut2,
                           const double4 *__restrict__ pos, const double4 *__restrict__ pos0,
                           int *__restrict__ flag) {
  int i = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ub) return;
  double4 p = pos[i], q = pos0[i];
  double dx = fabs(p.x - q.x);
  if (dx > H.x) dx -= L.x;
  double dy = fabs(p.y - q.y);
  if (dy > H.y) dy -= L.y;
  double dz = fabs(p.z - q.z);
  if (dz > H.z) dz -= L.z;
  if (dx > rcut || dy > rcut || dz > rcut || dx * dx + dy * dy + dz * dz > rcut2) atomicOr(flag, 1);
}

int launch_nl_check(Box *b, int lb, int ub, int *dflag) {
  if (ub <= lb) return FE_OK;
  double3 L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  double3 H = make_double3(b->p.L[0] / 2.0, b->p.L[1] / 2.0, b->p.L[2] / 2.0);
  double rcut = (b->p.rclist - b->p.rc) / 4.0;
  k_nl_check<<<(ub - lb + 255) / 256, 256, 0, b->stream>>>(lb, ub, L, H, rcut, rcut * rcut,
                                                           b->pos_q, b->pos_list0, dflag);
  FE_LAUNCH_CHECK("k_nl_check");
  return FE_OK;
}

int launch_nblist(Box *b) {
  int n = b->n;
  double3 L = make_double3(b->p.L[0], b->p.L[1], b->p.L[2]);
  int3 nc = make_int3(b->nc[0], b->nc[1], b->nc[2]);
  FE_CUDA(cudaMemsetAsync(b->cell_count, 0, b->cell_bytes, b->stream));
  k_cell_count<<<(n + 63) / 64, 64, 0, b->stream>>>(b->pos_q, n, L, nc, b->pfx, b->cell_of,
                                                   b->cell_count);
  FE_LAUNCH_CHECK("k_cell_count");
  k_cell_scan<<<1, 1024, 0, b->stream>>>(b->cell_count, b->ncells, b->cell_start, b->cell_fill);
  FE_LAUNCH_CHECK("k_cell_scan");
  k_cell_fill<<<(n + 255) / 256, 256, 0, b->stream>>>(n, b->cell_of, b->cell_start, b->cell_fill,
                                                      b->pfx, b->cell_sorted);
  FE_LAUNCH_CHECK("k_cell_fill");
  ListParams P;
  P.L = L;
  P.rcut = b->p.rclist;
  P.rcut2 = b->p.rclist * b->p.rclist;
  P.rcut2_ew = b->p.rclist_ew * b->p.rclist_ew;
  P.nc = nc;
  P.reach = b->list_reach;
  P.sc = make_float3((float)(L.x / 4294967296.0), (float)(L.y / 4294967296.0),
                     (float)(L.z / 4294967296.0));
  P.h = make_float3((float)(L.x / nc.x), (float)(L.y / nc.y), (float)(L.z / nc.z));
  // The FP32 distance of two sites at the cutoff rl is within 2e-6 rl (a
  // rounding of each 32-bit difference, product and sum) and 2 L / 2^32 of
  // the FP64 one; twice that on either side goes to the FP64 test.
  const double rl = fmin(b->p.rclist, b->p.rclist_ew), Lm = fmax(L.x, fmax(L.y, L.z));
  const double eps = 4e-6 * rl + 4.0 * Lm / 4294967296.0;
  P.in2 = (float)((rl - eps) * (rl - eps));
  P.out2 = (float)((rl + eps) * (rl + eps));
  const double ra = rl + eps + 1e-5 * Lm;  // FP32 site and cell-edge coordinates
  P.ra2 = (float)(ra * ra);
  P.n = n;
  P.max_nb = b->max_nb;
  int blocks = (n + kListWarps - 1) / kListWarps;
  if (blocks > 152 * 16) blocks = 152 * 16;
  k_list<<<blocks, kListWarps * 32, 0, b->stream>>>(
      P, b->pos_q, b->pfx, b->cell_of, b->cell_start, b->cell_sorted, b->x_start, b->x_partner,
      b->x_flag, b->x_pair, b->nl_count, b->nl_ent, b->xl, b->status);
  FE_LAUNCH_CHECK("k_list");
  b->have_list = true;
  return FE_OK;
}

}  // namespace fe
