// k_spme.cu -- FP64 smooth particle-mesh Ewald of pme_calc (pme_calc.c:18-279)
// on the device: B-spline weights (pme_spline.c:10-49, pme_qgrid.c:26-70),
// spreading, real<->complex transforms, the reciprocal-space convolution
// and the force gather with mean-force removal.
//
// The FP64 pipe (two instructions per SM and clock) bounds spreading and
// gathering, so both run on groups of four lanes per site (eight above order
// 4), one x plane each: lanes 0 to 2 form the weights of one axis each where
// they are used and pass them on by shuffles, instead of a pass that stores
// them and two that read them back.  Spreading adds each FP64 product to the grid
// as an integer (fix_of): sums of integers do not depend on the order of arrival,
// so the grid, the reciprocal energy and its forces repeat bit for bit.
//
// FFT: three kernels of this project (fe_fft.cuh) on grids whose planes they
// hold, else the library.  The reference transforms the real charge grid Q with FFTW_BACKWARD,
// scales by eterm (index 0 left alone), transforms FFTW_FORWARD and reads the
// real part.  For real Q that equals  real_out = C2R(eterm * R2C(Q))  with
// the library's conventions (R2C: exp(-i...), C2R: exp(+i...), both unnormalised),
// which is what runs here on the half spectrum.  |S|^2 is the same for both
// signs, so the energy sum is unchanged (weight 2 for the mirrored half).
#include <cmath>
#include <vector>

#include "fe_device.cuh"
#include "fe_fft.cuh"

namespace fe {

constexpr int kMaxOrder = 8;
// Largest plane (bytes of shared memory) the transform kernels take in FP64:
// all that fits.  96^3 (153 KB): 207 us against the library's 231 with its
// convolution; 32^3: 40 against 65 (both bound by latency and the FP64 pipe).
constexpr size_t kFft64PlaneMax = 224 * 1024;

// pme_spline.c:10-49, same operation order; array/darray indices 0..order
__host__ __device__ inline void fillspline(int order, double w, double *array, double *darray) {
  for (int i = 3; i <= order; i++) array[i] = 0.0;
  array[2] = w;
  array[1] = 1.0 - w;
  array[0] = 0.0;
  for (int i = 3; i <= order - 1; i++) {
    double div = (double)(1.0 / (i - 1));
    array[i] = div * w * array[i - 1];
    double di = (double)(i);
    for (int j = 1; j <= (i - 2); j++) {
      double dj = (double)(j);
      array[i - j] = div * ((w + dj) * array[i - j - 1] + (di - dj - w) * array[i - j]);
    }
    array[1] *= div * (1.0 - w);
  }
  darray[0] = 0.0;
  darray[1] = -array[1];
  for (int i = 2; i <= order; i++) darray[i] = array[i - 1] - array[i];
  int kk = order;
  double div = (double)(1.0 / (kk - 1));
  array[kk] = div * w * array[kk - 1];
  double dkk = (double)(kk);
  for (int i = 1; i <= (kk - 2); i++) {
    double di = (double)(i);
    array[kk - i] = div * ((w + di) * array[kk - i - 1] + (dkk - di - w) * array[kk - i]);
  }
  array[1] *= div * (1.0 - w);
}

__device__ __forceinline__ int wrapg(int v, int g) {
  v %= g;
  return v < 0 ? v + g : v;
}

// Lanes per site: one per x plane of its spline
constexpr int spme_lanes(int order) { return order <= 4 ? 4 : 8; }

// weights (and derivatives) of the P grid points f - P + 1 .. f at fraction w:
// order 4 in closed form, others by the recursion (unrolled)
template <int P, bool DERIV>
__device__ __forceinline__ void spline_axis(double w, double (&m)[P], double (&d)[P]) {
  if (P == 4) {
    const double t = 1.0 - w, w2 = w * w, t2 = t * t, s = 1.0 / 6.0;
    m[0] = t2 * t * s;
    m[1] = fma(w2, fma(0.5, w, -1.0), 2.0 / 3.0);
    m[2] = fma(t2, fma(0.5, t, -1.0), 2.0 / 3.0);
    m[3] = w2 * w * s;
    if (DERIV) {
      d[0] = -0.5 * t2;
      d[1] = w * fma(1.5, w, -2.0);
      d[2] = -t * fma(1.5, t, -2.0);
      d[3] = 0.5 * w2;
    }
    return;
  }
  double a[P + 1], da[P + 1];
  fillspline(P, w, a, da);
#pragma unroll
  for (int k = 0; k < P; k++) {
    m[k] = a[k + 1];
    d[k] = da[k + 1];
  }
}

// The group's site: lane 0, 1, 2 of the group forms the axis x, y, z (scaled
// coordinate G (x / L + 1/2), pme_qgrid.c:27-33; origin its integer part);
// every lane gets the first grid index of each axis, all y and z weights and
// the x weight of its own plane.
template <int P, bool DERIV>
struct SpmeSite {
  int x, y0, z0;  // own x plane, first y and z (may be negative: add G)
  double wx, dx, wy[P], wz[P], dy[P], dz[P];
};

template <int P, bool DERIV>
__device__ __forceinline__ void spme_site(const double4 &p, int3 G, double3 GL, int sub,
                                          SpmeSite<P, DERIV> &S) {
  constexpr int W = spme_lanes(P);
  const unsigned full = 0xffffffffu;
  const double x = sub == 0 ? p.x : sub == 1 ? p.y : p.z;
  const int g = sub == 0 ? G.x : sub == 1 ? G.y : G.z;
  const double u = fma(x, sub == 0 ? GL.x : sub == 1 ? GL.y : GL.z, 0.5 * g);
  const int f = (int)u;
  const int first = wrapg(f, g) - P + 1;
  double m[P], d[P];
  spline_axis<P, DERIV>(u - (double)f, m, d);
  S.x = __shfl_sync(full, first, 0, W) + sub;
  if (S.x < 0) S.x += G.x;
  S.y0 = __shfl_sync(full, first, 1, W);
  S.z0 = __shfl_sync(full, first, 2, W);
  S.wx = S.dx = 0.0;
#pragma unroll
  for (int k = 0; k < P; k++) {
    double v = __shfl_sync(full, m[k], 0, W);
    if (k == sub) S.wx = v;
    S.wy[k] = __shfl_sync(full, m[k], 1, W);
    S.wz[k] = __shfl_sync(full, m[k], 2, W);
    if (DERIV) {
      v = __shfl_sync(full, d[k], 0, W);
      if (k == sub) S.dx = v;
      S.dy[k] = __shfl_sync(full, d[k], 1, W);
      S.dz[k] = __shfl_sync(full, d[k], 2, W);
    }
  }
}

// threads of a block: gathering and, as atomics bind it and a small box has few
// sites, spreading (4,095 sites, 20 steps: 3,055 us with 32, 3,105 with 64 or 128)
constexpr int kSpmeBlock = 128, kSpreadBlock = 32;

// The charge grid as integers: K counts of 2^-unit, modulo 2^64; K counts of their
// overflows; whether there are any; how many values had no place in a count.  The
// unit (Box::fix_u) is 2^-59 of the power of two above the largest charge, where the
// roundings to it leave a point no further from the sum of its products than FP64
// additions do (water at 2.1, 1.04 and 0.70 points per A: 0.9, 2.1 and 2.9 e-18 e rms
// against 0.9, 3.6 and 10 e-18); a point overflows at 16 times that charge.  At
// 96,000 sites, 10 steps, the counts cost 0.1 ms of 18.3 over FP64 reductions, whose
// sums do not repeat.
struct FixGrid {
  unsigned long long *sum;
  int *carry;  // K, then `overflows` and `bad`
  long K;
  int t0;      // unit - 1075
  __host__ __device__ int *overflows() const { return carry + K; }
  __host__ __device__ int *bad() const { return carry + K + 1; }
};

// v in units, to nearest; on the bits of v, in integer registers: one FP64
// instruction takes the time of 32 of those.  `top` keeps the largest shift: above
// kFixTop a value was not a number, or beyond 2^62 units.
constexpr int kFixTop = 9;
__device__ __forceinline__ long long fix_of(double v, int t0, int &top) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const int s = (int)(bits >> 52 & 0x7ff) + t0;
  const unsigned long long m = (bits & 0xfffffffffffffull) << 9 | 1ull << 61;
  top = max(top, s);
  // (shifts of 64 and more leave nothing: m < 2^62, so 63 does as well)
  const int r = min(max(kFixTop - s, 0), 63);
  const long long a = (long long)((m >> r) + (r > 0 ? m >> (r - 1) & 1ull : 0ull));
  return (long long)bits < 0 ? -a : a;
}

// pme_qgrid.c:77-112: the grid gets q mm[x] mm[y] mm[z] of every site; `at`
// keeps the positions it was spread from, for the gather
template <int P>
__global__ void __launch_bounds__(kSpreadBlock)
k_spread(int n, int3 G, double3 GL, const double4 *__restrict__ pos, double4 *__restrict__ at,
         FixGrid F) {
  constexpr int W = spme_lanes(P);
  const int t = blockIdx.x * kSpreadBlock + threadIdx.x, i = t / W, sub = t % W;
  const double4 p = pos[min(i, n - 1)];
  SpmeSite<P, false> S;
  spme_site<P, false>(p, G, GL, sub, S);
  if (i >= n || sub >= P) return;
  if (sub == 0) at[i] = p;
  const double qx = p.w * S.wx;
  int top = 0;
#pragma unroll
  for (int a = 0; a < P; a++) {
    const int y = S.y0 + a < 0 ? S.y0 + a + G.y : S.y0 + a;
    const double qy = qx * S.wy[a];
    const size_t row = ((size_t)S.x * G.y + y) * G.z;
    long long add[P], old[P];
#pragma unroll
    for (int b = 0; b < P; b++) {
      const int z = S.z0 + b < 0 ? S.z0 + b + G.z : S.z0 + b;
      add[b] = fix_of(qy * S.wz[b], F.t0, top);
      old[b] = (long long)atomicAdd(F.sum + row + z, (unsigned long long)add[b]);
    }
#pragma unroll
    for (int b = 0; b < P; b++) {
      // an addition that changed the sum's sign against both operands'
      const long long now = (long long)((unsigned long long)old[b] + (unsigned long long)add[b]);
      if (((old[b] ^ now) & (add[b] ^ now)) < 0) {
        const int z = S.z0 + b < 0 ? S.z0 + b + G.z : S.z0 + b;
        atomicAdd(F.carry + row + z, add[b] < 0 ? -1 : 1);
        *F.overflows() = 1;
      }
    }
  }
  if (top > kFixTop) *F.bad() = 1;
}

// the FP64 grid from the counts; all NaN where a value had no place in them
__global__ void k_fix_grid(FixGrid F, int unit, double *__restrict__ grid) {
  const double add = *F.bad() ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
  const bool over = *F.overflows();
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < F.K;
       i += (long)gridDim.x * blockDim.x) {
    double v = fft_fix64((long long)F.sum[i], unit) + add;
    if (over) v += scalbn((double)F.carry[i], 64 - unit);
    grid[i] = v;
  }
}

// half spectrum: energy sum and scaling by eterm (pme_calc.c:52-93)
__global__ void k_recip(long Kh, const double *__restrict__ eterm, const double *__restrict__ kw,
                        cufftDoubleComplex *__restrict__ gk, double *__restrict__ partials) {
  double e = 0.0;
  for (long h = (long)blockIdx.x * blockDim.x + threadIdx.x; h < Kh;
       h += (long)gridDim.x * blockDim.x) {
    cufftDoubleComplex v = gk[h];
    double et = eterm[h];
    double struc2 = fma(v.x, v.x, v.y * v.y);
    e = fma(kw[h], et * struc2, e);
    v.x *= et;
    v.y *= et;
    gk[h] = v;
  }
  double vv[1] = {e};
  block_partials<1>(vv, partials);
}

// pme_force (pme_calc.c:122-265): per-site gather from the convolved grid.
// Each lane sums its x plane, z first (two sums per point, weight and
// derivative), so a site takes 176 fused multiply-adds for its 64 points.
template <int P>
__global__ void __launch_bounds__(kSpmeBlock)
k_gather(int n, int3 G, double3 GL, double qfe, const double4 *__restrict__ pos,
         const double *__restrict__ grid, double *__restrict__ fp,
         double *__restrict__ partials) {
  constexpr int W = spme_lanes(P);
  const int sub = threadIdx.x % W;
  double s[3] = {0.0, 0.0, 0.0};
  const int ngrp = gridDim.x * (kSpmeBlock / W);
  // whole warps go round together (the weights pass between lanes)
  for (int i0 = blockIdx.x * (kSpmeBlock / W) + (threadIdx.x & ~31) / W; i0 < n; i0 += ngrp) {
    const int i = i0 + (threadIdx.x & 31) / W;
    const double4 p = pos[min(i, n - 1)];
    SpmeSite<P, true> S;
    spme_site<P, true>(p, G, GL, sub, S);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    if (sub < P) {
      const double *gx = grid + (size_t)S.x * G.y * G.z;
#pragma unroll
      for (int a = 0; a < P; a++) {
        const int y = S.y0 + a < 0 ? S.y0 + a + G.y : S.y0 + a;
        const double *gy = gx + (size_t)y * G.z;
        double b0 = 0.0, b1 = 0.0;
#pragma unroll
        for (int b = 0; b < P; b++) {
          const int z = S.z0 + b < 0 ? S.z0 + b + G.z : S.z0 + b;
          const double v = gy[z];
          b0 = fma(S.wz[b], v, b0);
          b1 = fma(S.dz[b], v, b1);
        }
        a0 = fma(S.wy[a], b0, a0);
        a1 = fma(S.dy[a], b0, a1);
        a2 = fma(S.wy[a], b1, a2);
      }
    }
    a0 *= S.dx;
    a1 *= S.wx;
    a2 *= S.wx;
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, o);
      a1 += __shfl_xor_sync(0xffffffffu, a1, o);
      a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    // lane 0, 1, 2 of the group finishes x, y, z
    const double f = (sub == 0 ? a0 : sub == 1 ? a1 : a2) *
                     (-(p.w * qfe) * (sub == 0 ? GL.x : sub == 1 ? GL.y : GL.z));
    if (i < n && sub < 3) {
      fp[3 * i + sub] = f;
      s[0] += f;
    }
  }
  // the lane's sum belongs to one component
  const double v = s[0];
  s[0] = sub == 0 ? v : 0.0;
  s[1] = sub == 1 ? v : 0.0;
  s[2] = sub == 2 ? v : 0.0;
  block_partials<3>(s, partials);
}

__global__ void __launch_bounds__(512) k_fft_forward(FftBox<double> B, const int *bad) {
  extern __shared__ double2 fft_sh[];
  fft_forward_body<double>(B, blockIdx.x, reinterpret_cast<Cx<double> *>(fft_sh));
  // a value without a place in the counts: from this element (which this thread
  // wrote) the x lines and the way back carry NaN to every point and to the energy
  if (threadIdx.x == 0 && *bad) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    B.spec[(size_t)blockIdx.x * B.dy.n * (B.dz.n / 2 + 1)] = {nan, nan};
  }
}
__global__ void __launch_bounds__(512) k_fft_backward(FftBox<double> B) {
  extern __shared__ double2 fft_sh[];
  fft_backward_body<double>(B, blockIdx.x, reinterpret_cast<Cx<double> *>(fft_sh));
}
__global__ void __launch_bounds__(256)
k_fft_convolve(FftBox<double> B, int blocks, double *__restrict__ partials) {
  extern __shared__ double2 fft_sh[];
  double v[1] = {0.0};
  for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
    v[0] += fft_convolve_body<double>(B, blk, reinterpret_cast<Cx<double> *>(fft_sh));
    __syncthreads();  // the tile's lines are read before the next tile's arrive
  }
  block_partials<1>(v, partials);
}

void spme_free(Box *b) {
  delete b->fft;
  b->fft = nullptr;
}

static size_t fix_bytes(const Box *b) {
  return sizeof(unsigned long long) * b->K + sizeof(int) * (b->K + 2);
}
static FixGrid fix_grid(const Box *b) {
  return FixGrid{b->grid_fix, reinterpret_cast<int *>(b->grid_fix + b->K), b->K, b->fix_u - 1075};
}

int spme_setup(Box *b) {
  int GX = b->p.grid[0], GY = b->p.grid[1], GZ = b->p.grid[2];
  b->G[0] = GX;
  b->G[1] = GY;
  b->G[2] = GZ;
  b->order = b->p.order;
  b->K = (long)GX * GY * GZ;
  b->Kh = (long)GX * GY * (GZ / 2 + 1);
  int order = b->order;
  // B-spline moduli (pme_setup.c:86-130), host arithmetic as the reference
  double mn[kMaxOrder + 2], dmn[kMaxOrder + 2];
  fillspline(order, 0.0, mn, dmn);
  int gm = GX > GY ? (GX > GZ ? GX : GZ) : (GY > GZ ? GY : GZ);
  std::vector<double> barr(gm + 8, 0.0);
  for (int i = 2; i <= order + 1; i++) barr[i] = mn[i - 1];
  auto dftmod = [&](int grid) {
    std::vector<double> bm(grid + 2, 0.0);
    double twopi = 2.0 * kPI;
    for (int i = 1; i <= grid; i++) {
      double sum1 = 0.0, sum2 = 0.0;
      for (int j = 1; j <= grid; j++) {
        double arg = twopi * (i - 1) * (j - 1) / grid;
        sum1 += barr[j] * cos(arg);
        sum2 += barr[j] * sin(arg);
      }
      bm[i] = sum1 * sum1 + sum2 * sum2;
    }
    return bm;
  };
  std::vector<double> bx = dftmod(GX), by = dftmod(GY), bz = dftmod(GZ);
  // eterm on the half spectrum (pme_calc.c:52-71)
  double blx = b->p.L[0], bly = b->p.L[1], blz = b->p.L[2];
  double vol = blx * bly * blz;
  double kap = b->p.kappa;
  double fac = kPI * kPI / kap / kap;
  int GZh = GZ / 2 + 1;
  std::vector<double> et(b->Kh), kw(b->Kh);
  for (int k1 = 0; k1 < GX; k1++)
    for (int k2 = 0; k2 < GY; k2++)
      for (int k3 = 0; k3 < GZh; k3++) {
        long h = ((long)k1 * GY + k2) * GZh + k3;
        if (k1 == 0 && k2 == 0 && k3 == 0) {
          et[h] = 1.0;  // the reference never scales index 0
          kw[h] = 0.0;
          continue;
        }
        int mx = k1 - (k1 > GX / 2 ? GX : 0);
        int my = k2 - (k2 > GY / 2 ? GY : 0);
        int mz = k3 - (k3 > GZ / 2 ? GZ : 0);
        double mhatx = mx / blx, mhaty = my / bly, mhatz = mz / blz;
        double mm = mhatx * mhatx + mhaty * mhaty + mhatz * mhatz;
        double bb = bx[k1 + 1] * by[k2 + 1] * bz[k3 + 1];
        double den = kPI * vol * mm * bb;
        et[h] = exp(-fac * mm) / den;
        kw[h] = (k3 == 0 || (GZ % 2 == 0 && k3 == GZ / 2)) ? 1.0 : 2.0;
      }
  FE_CUDA(cudaMalloc(&b->eterm, sizeof(double) * b->Kh));
  FE_CUDA(cudaMalloc(&b->kweight, sizeof(double) * b->Kh));
  FE_CUDA(cudaMemcpy(b->eterm, et.data(), sizeof(double) * b->Kh, cudaMemcpyHostToDevice));
  FE_CUDA(cudaMemcpy(b->kweight, kw.data(), sizeof(double) * b->Kh, cudaMemcpyHostToDevice));
  FE_CUDA(cudaMalloc(&b->grid, sizeof(double) * b->K));
  if (b->prec == FE_PREC_FP64) FE_CUDA(cudaMalloc(&b->grid_fix, fix_bytes(b)));
  int e = 0;  // |q| < 2^e; a weight is at most 8 (order 3, just outside the box)
  if (std::isfinite(b->qmax)) frexp(b->qmax, &e);
  b->fix_u = 59 - e;
  FE_CUDA(cudaMalloc(&b->grid_k, sizeof(cufftDoubleComplex) * b->Kh));
  FE_CUDA(cudaMalloc(&b->fp, sizeof(double) * 3 * b->n));
  FE_CUDA(cudaMalloc(&b->pos_pme, sizeof(double4) * b->n));
  FE_CUDA(cudaMemset(b->pos_pme, 0, sizeof(double4) * b->n));
  FftBox<double> F{};
  std::vector<Cx<double>> tw;
  if (fft_plan<double>(b->G, &F, &tw) && fft_plane_smem<double>(GY, GZ) <= kFft64PlaneMax) {
    FE_CUDA(cudaMalloc(&b->fft_tw, sizeof(Cx<double>) * tw.size()));
    FE_CUDA(cudaMemcpy(b->fft_tw, tw.data(), sizeof(Cx<double>) * tw.size(),
                       cudaMemcpyHostToDevice));
    fft_set_twiddles<double>(&F, (const Cx<double> *)b->fft_tw);
    F.fix = b->grid_fix;
    F.unit = b->fix_u;
    F.carry = fix_grid(b).carry;
    F.real = b->grid;
    F.spec = reinterpret_cast<Cx<double> *>(b->grid_k);
    F.eterm = b->eterm;
    F.kw = b->kweight;
    b->fft = new FftBox<double>(F);
    const int lim = (int)kFftSmemMax;
    FE_CUDA(cudaFuncSetAttribute(k_fft_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
    FE_CUDA(cudaFuncSetAttribute(k_fft_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
    FE_CUDA(cudaFuncSetAttribute(k_fft_convolve, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
    return FE_OK;
  }
  cufftResult r = cufftPlan3d(&b->plan_r2c, GX, GY, GZ, CUFFT_D2Z);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftPlan3d D2Z");
  r = cufftPlan3d(&b->plan_c2r, GX, GY, GZ, CUFFT_Z2D);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftPlan3d Z2D");
  b->plans = true;
  return FE_OK;
}

// f<order>(...) for the box's order
#define SPME_ORDER(order, CALL) \
  switch (order) {              \
    case 3: CALL(3); break;     \
    case 4: CALL(4); break;     \
    case 5: CALL(5); break;     \
    case 6: CALL(6); break;     \
    case 7: CALL(7); break;     \
    default: CALL(8); break;    \
  }

static double3 grid_per_length(const Box *b) {
  return make_double3(b->G[0] / b->p.L[0], b->G[1] / b->p.L[1], b->G[2] / b->p.L[2]);
}

// the counts from the current positions
static int launch_spread64(Box *b) {
  const int3 G = make_int3(b->G[0], b->G[1], b->G[2]);
  const double3 GL = grid_per_length(b);
  FE_CUDA(cudaMemsetAsync(b->grid_fix, 0, fix_bytes(b), b->stream));
  const int per = kSpreadBlock / spme_lanes(b->order), blocks = (b->n + per - 1) / per;
#define SPREAD(P)                                                                       \
  k_spread<P><<<blocks, kSpreadBlock, 0, b->stream>>>(b->n, G, GL, b->pos_q, b->pos_pme, \
                                                      fix_grid(b))
  SPME_ORDER(b->order, SPREAD)
#undef SPREAD
  FE_LAUNCH_CHECK("k_spread");
  return FE_OK;
}

// the charge grid (pme_qgrid.c:20-118)
int launch_charge_grid64(Box *b) {
  // (a mixed box has the counts from its first call of fe_charge_grid)
  if (!b->grid_fix) FE_CUDA(cudaMalloc(&b->grid_fix, fix_bytes(b)));
  int rc = launch_spread64(b);
  if (rc) return rc;
  const long want = (b->K + 255) / 256, most = 4L * b->nsm;
  k_fix_grid<<<(int)(want < most ? want : most), 256, 0, b->stream>>>(fix_grid(b), b->fix_u,
                                                                      b->grid);
  FE_LAUNCH_CHECK("k_fix_grid");
  return FE_OK;
}

int launch_pme64(Box *b, cudaEvent_t ev_recip) {
  int rc = b->fft ? launch_spread64(b) : launch_charge_grid64(b);
  if (rc) return rc;
  if (b->fft) {
    const int gx = b->G[0], gy = b->G[1], gz = b->G[2];
    const int pt = fft_plane_threads(gy, gz), tiles = fft_line_blocks(gy, gz, b->fft->tile);
    const size_t ps = fft_plane_smem<double>(gy, gz);
    k_fft_forward<<<gx, pt, ps, b->stream>>>(*b->fft, fix_grid(b).bad());
    FE_LAUNCH_CHECK("k_fft_forward");
    const int blocks = tiles < kSumRows ? tiles : kSumRows;
    k_fft_convolve<<<blocks, fft_line_threads(gx, b->fft->tile),
                     fft_line_smem<double>(gx, b->fft->tile), b->stream>>>(*b->fft, tiles,
                                                                          b->part_recip);
    FE_LAUNCH_CHECK("k_fft_convolve");
    b->n_recip = blocks;
    if (ev_recip) FE_CUDA(cudaEventRecord(ev_recip, b->stream));
    k_fft_backward<<<gx, pt, ps, b->stream>>>(*b->fft);
    FE_LAUNCH_CHECK("k_fft_backward");
    return launch_pme_gather64(b);
  }
  cufftResult r = cufftSetStream(b->plan_r2c, b->stream);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftSetStream");
  r = cufftExecD2Z(b->plan_r2c, b->grid, b->grid_k);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftExecD2Z");
  int blocks = (int)((b->Kh + 127) / 128);
  if (blocks > kSumRows) blocks = kSumRows;
  k_recip<<<blocks, 128, 0, b->stream>>>(b->Kh, b->eterm, b->kweight, b->grid_k, b->part_recip);
  FE_LAUNCH_CHECK("k_recip");
  b->n_recip = blocks;
  if (ev_recip) FE_CUDA(cudaEventRecord(ev_recip, b->stream));
  r = cufftSetStream(b->plan_c2r, b->stream);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftSetStream");
  r = cufftExecZ2D(b->plan_c2r, b->grid_k, b->grid);
  if (r != CUFFT_SUCCESS) return cufft_fail(r, "cufftExecZ2D");
  return launch_pme_gather64(b);
}

// pme_force (pme_calc.c:122-206): the reciprocal forces into fp from the
// convolved grid at the positions of the last charge_grid; launch_apply_pme or
// launch_tail64 sums their partials and removes the mean
int launch_pme_gather64(Box *b) {
  const int3 G = make_int3(b->G[0], b->G[1], b->G[2]);
  const double3 GL = grid_per_length(b);
  const double qfe = kELEC * kELEQ * kELEQ * kNA * 1.0E-3 / b->p.epsRF;
  const int per = kSpmeBlock / spme_lanes(b->order);
  int blocks = (b->n + per - 1) / per;
  if (blocks > kSumRows) blocks = kSumRows;
#define GATHER(P)                                                                               \
  k_gather<P><<<blocks, kSpmeBlock, 0, b->stream>>>(b->n, G, GL, qfe, b->pos_pme, b->grid, b->fp, \
                                                    b->part_gather)
  SPME_ORDER(b->order, GATHER)
#undef GATHER
  FE_LAUNCH_CHECK("k_gather");
  b->n_gather = blocks;
  return FE_OK;
}

}  // namespace fe
