// fe_fft.cuh -- the 3-D transforms of SPME as three kernels: real planes to
// the half spectrum (z and y), the x lines there and back with the convolution
// between, and the planes back to real.  The library's transform takes three
// launches each way and the convolution one; on the grids of small boxes
// (24^3 to 40^3) each is a launch's latency, and on larger ones a pass over
// the grid.
//
// A block transforms a whole plane (or a tile of x lines) in shared memory by
// the self-sorting Stockham scheme (Cooley & Tukey 1965, radices 2, 3, 4, 5 and
// 8), ping-pong between two buffers.  Elements are [index][line], so that a
// warp's lanes work on neighbouring lines and touch neighbouring words in
// every pass.  Two real rows make one complex line of the z transform.  Forward
// exp(-i..), backward exp(+i..), both unnormalised, half spectrum
// [x][y][z <= Gz/2]: the library's conventions.
//
// Sizes whose factors are 2, 3 and 5 and whose planes fit (fft_plan); others
// keep the library.  FP64 sources are compiled without contraction, so the
// products are fused by hand.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "fe_device.cuh"

namespace fe {

template <typename T>
struct Cx {
  T x, y;
};

__device__ __forceinline__ float fft_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fft_fma(double a, double b, double c) { return fma(a, b, c); }

template <typename T>
__device__ __forceinline__ Cx<T> operator+(Cx<T> a, Cx<T> b) {
  return {a.x + b.x, a.y + b.y};
}
template <typename T>
__device__ __forceinline__ Cx<T> operator-(Cx<T> a, Cx<T> b) {
  return {a.x - b.x, a.y - b.y};
}
template <typename T>
__device__ __forceinline__ Cx<T> cx_mul(Cx<T> a, Cx<T> b) {
  return {fft_fma(a.x, b.x, -(a.y * b.y)), fft_fma(a.x, b.y, a.y * b.x)};
}
// a times -i (forward) or +i (backward)
template <bool INV, typename T>
__device__ __forceinline__ Cx<T> cx_rot(Cx<T> a) {
  return INV ? Cx<T>{-a.y, a.x} : Cx<T>{a.y, -a.x};
}

template <bool INV, typename T>
__device__ __forceinline__ void fft2(Cx<T> &a, Cx<T> &b) {
  Cx<T> t = a - b;
  a = a + b;
  b = t;
}
template <bool INV, typename T>
__device__ __forceinline__ void fft4(Cx<T> &a, Cx<T> &b, Cx<T> &c, Cx<T> &d) {
  Cx<T> s = a + c, u = a - c, v = b + d, w = cx_rot<INV>(b - d);
  a = s + v;
  b = u + w;
  c = s - v;
  d = u - w;
}

// the R-point transform in registers, outputs in order
template <int R, bool INV, typename T>
__device__ __forceinline__ void fft_small(Cx<T> (&v)[R]) {
  if constexpr (R == 2) {
    fft2<INV>(v[0], v[1]);
  } else if constexpr (R == 3) {
    const T h = (T)0.86602540378443864676;  // sin(2 pi / 3)
    Cx<T> s = v[1] + v[2], d = v[1] - v[2];
    Cx<T> m = {fft_fma((T)-0.5, s.x, v[0].x), fft_fma((T)-0.5, s.y, v[0].y)};
    Cx<T> r = cx_rot<INV>(Cx<T>{h * d.x, h * d.y});
    v[0] = v[0] + s;
    v[1] = m + r;
    v[2] = m - r;
  } else if constexpr (R == 4) {
    fft4<INV>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 5) {
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410,
            s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
    Cx<T> a = v[1] + v[4], b = v[1] - v[4], c = v[2] + v[3], d = v[2] - v[3];
    Cx<T> p = {fft_fma(c1, a.x, fft_fma(c2, c.x, v[0].x)),
               fft_fma(c1, a.y, fft_fma(c2, c.y, v[0].y))};
    Cx<T> q = {fft_fma(c2, a.x, fft_fma(c1, c.x, v[0].x)),
               fft_fma(c2, a.y, fft_fma(c1, c.y, v[0].y))};
    Cx<T> r = cx_rot<INV>(Cx<T>{fft_fma(s1, b.x, s2 * d.x), fft_fma(s1, b.y, s2 * d.y)});
    Cx<T> t = cx_rot<INV>(Cx<T>{fft_fma(s2, b.x, -(s1 * d.x)), fft_fma(s2, b.y, -(s1 * d.y))});
    v[0] = v[0] + (a + c);
    v[1] = p + r;
    v[2] = q + t;
    v[3] = q - t;
    v[4] = p - r;
  } else {
    static_assert(R == 8, "radices 2, 3, 4, 5, 8");
    const T h = (T)0.70710678118654752440;
    fft4<INV>(v[0], v[2], v[4], v[6]);
    fft4<INV>(v[1], v[3], v[5], v[7]);
    // odd half times w8^k: w8 = h (1 -+ i)
    Cx<T> r1 = cx_rot<INV>(v[3]), r3 = cx_rot<INV>(v[7]);
    Cx<T> o1 = {h * (v[3].x + r1.x), h * (v[3].y + r1.y)};
    Cx<T> o2 = cx_rot<INV>(v[5]);
    Cx<T> o3 = {h * (r3.x - v[7].x), h * (r3.y - v[7].y)};
    Cx<T> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = e0 + o0;
    v[1] = e1 + o1;
    v[2] = e2 + o2;
    v[3] = e3 + o3;
    v[4] = e0 - o0;
    v[5] = e1 - o1;
    v[6] = e2 - o2;
    v[7] = e3 - o3;
  }
}

constexpr int kFftMaxFactors = 8;
// one axis: its length, radices and exp(-2 pi i t / n), t < n
struct FftDim {
  int n, nf;
  int f[kFftMaxFactors];
  const void *tw;
};

// q = w / d for 0 <= w < 2^20 and small d, by the FP32 reciprocal: the
// quotient of w + 1/2 stays 1/(2d) away from an integer, its error below that
__device__ __forceinline__ int fft_div(int w, float inv) {
  return __float2int_rd(((float)w + 0.5f) * inv);
}

// one pass of radix R over nb lines: butterflies j < n / R of every line
template <int R, bool INV, typename T>
__device__ __forceinline__ void fft_pass(const Cx<T> *__restrict__ in, Cx<T> *__restrict__ out,
                                         int n, int L, int nb, int ld, float inv_nb,
                                         const Cx<T> *__restrict__ tw) {
  const int m = n / R, step = m / L;  // twiddle exp(-2 pi i k r / (L R)) = tw[k r step]
  const float inv_L = 1.0f / (float)L;
  for (int w = threadIdx.x; w < nb * m; w += blockDim.x) {
    const int j = fft_div(w, inv_nb), b = w - j * nb;
    const int jl = L == 1 ? j : fft_div(j, inv_L), k = j - jl * L;
    Cx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = in[(j + r * m) * ld + b];
    if (L > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        Cx<T> t = tw[k * r * step];
        if (INV) t.y = -t.y;
        v[r] = cx_mul(v[r], t);
      }
    }
    fft_small<R, INV, T>(v);
    Cx<T> *o = out + (jl * L * R + k) * ld + b;
#pragma unroll
    for (int r = 0; r < R; r++) o[r * L * ld] = v[r];
  }
}

// nb lines of length D.n in `a` (element i of line b at a[i ld + b]); returns
// the buffer that holds the result (a or s)
template <bool INV, typename T>
__device__ __forceinline__ Cx<T> *fft_lines(Cx<T> *a, Cx<T> *s, const FftDim &D, int nb, int ld,
                                            const Cx<T> *tw) {
  const float inv_nb = 1.0f / (float)nb;
  int L = 1;
  for (int p = 0; p < D.nf; p++) {
    const int R = D.f[p];
    __syncthreads();
    if (R == 8) fft_pass<8, INV, T>(a, s, D.n, L, nb, ld, inv_nb, tw);
    else if (R == 4) fft_pass<4, INV, T>(a, s, D.n, L, nb, ld, inv_nb, tw);
    else if (R == 5) fft_pass<5, INV, T>(a, s, D.n, L, nb, ld, inv_nb, tw);
    else if (R == 3) fft_pass<3, INV, T>(a, s, D.n, L, nb, ld, inv_nb, tw);
    else fft_pass<2, INV, T>(a, s, D.n, L, nb, ld, inv_nb, tw);
    L *= R;
    Cx<T> *t = a;
    a = s;
    s = t;
  }
  __syncthreads();
  return a;
}

// One box's transforms.
template <typename T>
struct FftBox {
  FftDim dx, dy, dz;
  int tile;              // x lines of a block of the middle kernel
  unsigned long long *fix;  // fixed-point charge sums (fft_load); or
  T *real;               // the real grid, in (when fix is null) and out
  int unit;              // FP64: the sums count 2^-unit
  const int *carry;      // FP64: their overflows, and whether there are any
  Cx<T> *spec;           // half spectrum
  const T *eterm, *kw;
};

__host__ __device__ inline int fft_odd(int v) { return v | 1; }
// elements of one of the two buffers of a plane / of an x tile
__host__ __device__ inline int fft_plane_elems(int gy, int gz) {
  const int z = gz * fft_odd((gy + 1) / 2), y = gy * fft_odd(gz / 2 + 1);
  return z > y ? z : y;
}
template <typename T>
size_t fft_plane_smem(int gy, int gz) {
  return sizeof(Cx<T>) * (2 * (size_t)fft_plane_elems(gy, gz) + gy + gz);
}
template <typename T>
size_t fft_line_smem(int gx, int tile) {
  return sizeof(Cx<T>) * ((size_t)2 * gx * fft_odd(tile) + gx);
}

template <typename T>
__device__ __forceinline__ const Cx<T> *fft_twiddles(const FftDim &D, Cx<T> *sh) {
  const Cx<T> *g = reinterpret_cast<const Cx<T> *>(D.tw);
  for (int i = threadIdx.x; i < D.n; i += blockDim.x) sh[i] = g[i];
  return sh;
}

// a fixed-point grid sum (2^40 per unit) as FP32: the upper 32 bits hold value
// x 2^8 and convert exactly while |value| < 2^16, the lower 32 with one
// rounding, one fused multiply-add joins them
__device__ __forceinline__ float fft_fix(unsigned long long u) {
  return fmaf((float)(int)(u >> 32), 0x1p-8f, __uint2float_rn((unsigned)u) * 0x1p-40f);
}

// v counts of 2^-unit as FP64, rounded to nearest in integer registers (the FP64 pipe
// is the pair loop's)
__device__ __forceinline__ double fft_fix64(long long v, int unit) {
  const unsigned long long m = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  if (m == 0) return 0.0;
  const int z = __clzll((long long)m);
  const unsigned long long top = m << z, cut = top & 0x7ff;
  unsigned long long r = top >> 11;
  r += cut > 0x400 || (cut == 0x400 && (r & 1));
  r += (unsigned long long)(1085 - z - unit) << 52;
  return __longlong_as_double((long long)(r | (v < 0 ? 1ull << 63 : 0ull)));
}

// Value i of the real grid's sums: FP32 ones count 2^-40 (the transform clears them);
// FP64 ones come with a count of overflows, looked at where there are any.
__device__ __forceinline__ bool fft_overflows(const FftBox<float> &) { return false; }
__device__ __forceinline__ bool fft_overflows(const FftBox<double> &B) {
  return B.fix && B.carry[(size_t)B.dx.n * B.dy.n * B.dz.n];
}
__device__ __forceinline__ float fft_load(const FftBox<float> &B, size_t i, bool) {
  return B.fix ? fft_fix(B.fix[i]) : B.real[i];
}
__device__ __forceinline__ double fft_load(const FftBox<double> &B, size_t i, bool overflows) {
  if (!B.fix) return B.real[i];
  const double v = fft_fix64((long long)B.fix[i], B.unit);
  return overflows ? v + scalbn((double)B.carry[i], 64 - B.unit) : v;
}

// plane x: real -> half spectrum over (y, z)
template <typename T>
__device__ __forceinline__ void fft_forward_body(const FftBox<T> &B, int x, Cx<T> *sh) {
  const int gy = B.dy.n, gz = B.dz.n, zh = gz / 2 + 1, np = (gy + 1) / 2;
  const int elems = fft_plane_elems(gy, gz), lz = fft_odd(np), ly = fft_odd(zh);
  Cx<T> *a = sh, *s = sh + elems;
  const Cx<T> *twz = fft_twiddles<T>(B.dz, sh + 2 * elems);
  const Cx<T> *twy = fft_twiddles<T>(B.dy, sh + 2 * elems + gz);
  // rows 2p and 2p + 1 as the real and imaginary part of line p
  const float inv_gz = 1.0f / (float)gz;
  const size_t base = (size_t)x * gy * gz;
  const bool over = fft_overflows(B);
  // (eight loads a thread in flight: a store to the sums or to the plane between
  // them would hold each back until the last has arrived)
  for (int w0 = threadIdx.x; w0 < 2 * np * gz; w0 += 8 * blockDim.x) {
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int w = w0 + u * blockDim.x;
      v[u] = (T)0;
      if (w < gy * gz) v[u] = fft_load(B, base + w, over);
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int w = w0 + u * blockDim.x;
      if (w >= 2 * np * gz) break;
      const int y = fft_div(w, inv_gz), z = w - y * gz;
      if (sizeof(T) == sizeof(float) && B.fix && w < gy * gz) B.fix[base + w] = 0ull;
      Cx<T> *e = a + z * lz + (y >> 1);
      if (y & 1) e->y = v[u];
      else e->x = v[u];
    }
  }
  Cx<T> *f = fft_lines<false, T>(a, s, B.dz, np, lz, twz);
  Cx<T> *g = f == a ? s : a;
  // the two rows' spectra: A = (Z[k] + Z*[-k]) / 2, B = (Z[k] - Z*[-k]) / 2i
  const float inv_np = 1.0f / (float)np;
  for (int w = threadIdx.x; w < np * zh; w += blockDim.x) {
    const int k = fft_div(w, inv_np), p = w - k * np;
    const Cx<T> u = f[k * lz + p], v = f[(k == 0 ? 0 : gz - k) * lz + p];
    const T h = (T)0.5;
    g[(2 * p) * ly + k] = {h * (u.x + v.x), h * (u.y - v.y)};
    if (2 * p + 1 < gy) g[(2 * p + 1) * ly + k] = {h * (u.y + v.y), h * (v.x - u.x)};
  }
  Cx<T> *r = fft_lines<false, T>(g, f, B.dy, zh, ly, twy);
  const float inv_zh = 1.0f / (float)zh;
  Cx<T> *o = B.spec + (size_t)x * gy * zh;
  for (int w = threadIdx.x; w < gy * zh; w += blockDim.x) {
    const int y = fft_div(w, inv_zh);
    o[w] = r[y * ly + (w - y * zh)];
  }
}

// plane x: half spectrum -> real over (y, z)
template <typename T>
__device__ __forceinline__ void fft_backward_body(const FftBox<T> &B, int x, Cx<T> *sh) {
  const int gy = B.dy.n, gz = B.dz.n, zh = gz / 2 + 1, np = (gy + 1) / 2;
  const int elems = fft_plane_elems(gy, gz), lz = fft_odd(np), ly = fft_odd(zh);
  Cx<T> *a = sh, *s = sh + elems;
  const Cx<T> *twz = fft_twiddles<T>(B.dz, sh + 2 * elems);
  const Cx<T> *twy = fft_twiddles<T>(B.dy, sh + 2 * elems + gz);
  const float inv_zh = 1.0f / (float)zh, inv_np = 1.0f / (float)np, inv_gz = 1.0f / (float)gz;
  const Cx<T> *in = B.spec + (size_t)x * gy * zh;
  for (int w = threadIdx.x; w < gy * zh; w += blockDim.x) {
    const int y = fft_div(w, inv_zh);
    a[y * ly + (w - y * zh)] = in[w];
  }
  Cx<T> *f = fft_lines<true, T>(a, s, B.dy, zh, ly, twy);
  Cx<T> *g = f == a ? s : a;
  // line p: Z = A + i B with both rows' Hermitian halves (the imaginary parts
  // of k = 0 and k = gz / 2, which a real row has not, left out)
  for (int w = threadIdx.x; w < np * zh; w += blockDim.x) {
    const int k = fft_div(w, inv_np), p = w - k * np;
    Cx<T> u = f[(2 * p) * ly + k];
    Cx<T> v = 2 * p + 1 < gy ? f[(2 * p + 1) * ly + k] : Cx<T>{(T)0, (T)0};
    if (k == 0 || 2 * k == gz) {
      g[k * lz + p] = {u.x, v.x};
    } else {
      g[k * lz + p] = {u.x - v.y, u.y + v.x};
      g[(gz - k) * lz + p] = {u.x + v.y, v.x - u.y};
    }
  }
  Cx<T> *r = fft_lines<true, T>(g, f, B.dz, np, lz, twz);
  T *o = B.real + (size_t)x * gy * gz;
  for (int w = threadIdx.x; w < gy * gz; w += blockDim.x) {
    const int y = fft_div(w, inv_gz), z = w - y * gz;
    const Cx<T> e = r[z * lz + (y >> 1)];
    o[w] = (y & 1) ? e.y : e.x;
  }
}

// `tile` x lines from line q0 of the (y, z) plane: forward, the convolution
// (pme_calc.c:52-93), backward; returns the thread's share of the energy sum
template <typename T>
__device__ __forceinline__ T fft_convolve_body(const FftBox<T> &B, int blk, Cx<T> *sh) {
  const int gx = B.dx.n, lines = B.dy.n * (B.dz.n / 2 + 1), nt = B.tile, lt = fft_odd(nt);
  const int q0 = blk * nt, nb = min(nt, lines - q0);
  Cx<T> *a = sh, *s = sh + gx * lt;
  const Cx<T> *tw = fft_twiddles<T>(B.dx, sh + 2 * gx * lt);
  const float inv_nb = 1.0f / (float)nb;
  for (int w = threadIdx.x; w < gx * nb; w += blockDim.x) {
    const int i = fft_div(w, inv_nb), b = w - i * nb;
    a[i * lt + b] = B.spec[(size_t)i * lines + q0 + b];
  }
  Cx<T> *f = fft_lines<false, T>(a, s, B.dx, nb, lt, tw);
  T e = (T)0;
  for (int w = threadIdx.x; w < gx * nb; w += blockDim.x) {
    const int i = fft_div(w, inv_nb), b = w - i * nb;
    const size_t h = (size_t)i * lines + q0 + b;
    Cx<T> v = f[i * lt + b];
    const T et = B.eterm[h];
    e = fft_fma(B.kw[h] * et, fft_fma(v.x, v.x, v.y * v.y), e);
    f[i * lt + b] = {v.x * et, v.y * et};
  }
  Cx<T> *r = fft_lines<true, T>(f, f == a ? s : a, B.dx, nb, lt, tw);
  for (int w = threadIdx.x; w < gx * nb; w += blockDim.x) {
    const int i = fft_div(w, inv_nb), b = w - i * nb;
    B.spec[(size_t)i * lines + q0 + b] = r[i * lt + b];
  }
  return e;
}

// ---- host side ----

constexpr size_t kFftSmemMax = 224 * 1024;

// radices of n, largest first; false when a prime above 5 is left
inline bool fft_factor(int n, FftDim *D) {
  D->n = n;
  D->nf = 0;
  for (int r : {8, 4, 5, 3, 2})
    while (n % r == 0 && D->nf < kFftMaxFactors) {
      // 2 x 8 is dearer than 4 x 4
      if (r == 8 && n == 16) break;
      D->f[D->nf++] = r;
      n /= r;
    }
  return n == 1;
}

// Plans a box: sizes that factor, planes and tiles that fit in shared memory.
// tw: gx + gy + gz twiddles for the device, in that order.  Every axis at least
// 4 and at most 256 (indices of a plane stay below fft_div's limit).
template <typename T>
bool fft_plan(const int *G, FftBox<T> *B, std::vector<Cx<T>> *tw) {
  for (int d = 0; d < 3; d++)
    if (G[d] < 4 || G[d] > 256) return false;
  if (!fft_factor(G[0], &B->dx) || !fft_factor(G[1], &B->dy) || !fft_factor(G[2], &B->dz))
    return false;
  // lines per block of the middle kernel: 64-byte rows at least, wider while
  // that still leaves two blocks an SM
  const int lines = G[1] * (G[2] / 2 + 1);
  B->tile = 8;
  if (lines / 16 >= 304) B->tile = 16;
  if (fft_plane_smem<T>(G[1], G[2]) > kFftSmemMax || fft_line_smem<T>(G[0], B->tile) > kFftSmemMax)
    return false;
  tw->clear();
  for (int d = 0; d < 3; d++)
    for (int t = 0; t < G[d]; t++) {
      const long double a = -2.0L * 3.14159265358979323846264338327950288L * t / G[d];
      tw->push_back({(T)cosl(a), (T)sinl(a)});
    }
  return true;
}

template <typename T>
void fft_set_twiddles(FftBox<T> *B, const Cx<T> *dev) {
  B->dx.tw = dev;
  B->dy.tw = dev + B->dx.n;
  B->dz.tw = dev + B->dx.n + B->dy.n;
}

// threads of a block: a plane's passes have gy gz / 8 to / 16 butterflies
inline int fft_plane_threads(int gy, int gz) { return gy * gz >= 2048 ? 512 : 256; }
inline int fft_line_threads(int gx, int tile) { return gx * tile > 512 ? 256 : 128; }

inline int fft_line_blocks(int gy, int gz, int tile) {
  return (gy * (gz / 2 + 1) + tile - 1) / tile;
}

}  // namespace fe
