// Dynamic Smagorinsky eddy viscosity on the device: LES = 2 (coefficient
// averaged in z, subgrid.f90:261-414 sgs_dynamic_Smagorinsky) and LES = 3
// (pointwise coefficient, subgrid.f90:420-583 _noaverage).
//
// The model runs in FP64 in both precisions.  The source makes some sixty
// whole-array passes (interpolations, 24 filters, 34 ghost fills, two rates of
// strain, contractions); here they are four kernels and, for LES = 2, a fifth:
//   k_dyn_strain   |S| and |S| Sij of U, V, W;
//   k_dyn_filter   filtered face velocities hat(U), hat(V), hat(W);
//   k_dyn_strain   4 |hat(S)| hat(Sij) of those;
//   k_dyn_contract the 15 filters of Lij and Mij (hat(ui uj), hat(ui),
//                  hat(|S| Sij)), the contractions Mij Lij and Mij Mij and, for
//                  LES = 3, nu_t with its clipping and ghosts;
//   k_dyn_zavg     LES = 2: the z averages, nu_t, clipping and ghosts.
// Ghost entries (apply_Neumann_bc_x / apply_periodic_bc_x,
// boundary_conditions.f90:295-344; apply_periodic_bc_z, :732-760; one process)
// are never stored: a reader takes the interior entry that the source's copies
// would have left there, by index (xmap, zmap, zmap_w).
// The filter of filter_xzy (subgrid.f90:140-184, fil_size = 2) is the product
// of (1,4,1)/6 along x, y and z (one-sided 2/3, 1/3 at the first and last row
// of its y section), applied as three sums.
//
// Work arrays are dense (nxg,nyg) planes, i fastest, Fortran indices.
#include "kernels.cuh"
#include "strain.cuh"

namespace blgpu {
namespace {

// |S|; |S| Sij; 4 |hat S| hat Sij; hat(U), hat(V), hat(W) and, once those are
// used, Mij Lij and Mij Mij of LES = 2 in the first two of them
enum { W_S, W_SS, W_M = W_SS + 6, W_F = W_M + 6, W_COUNT = W_F + 3 };

struct P6 {
  double *p[6];
};
struct P3 {
  double *p[3];
};

__device__ __forceinline__ long long dix(int i, int j, int k, const Geo &g) {
  return ((long long)(k - 1) * g.nyg + (j - 1)) * (long long)g.nxg + (i - 1);
}

// the column whose entry the source's x ghost fill leaves at column i of an
// array of n1 columns: Neumann, periodic for a face array (n1 = nx, id 1) or
// periodic for a centre array (n1 = nxg, id 2)
__device__ __forceinline__ int xmap(int i, int n1, int periodic, bool face) {
  if (!periodic) return i <= 1 ? 2 : i >= n1 ? n1 - 1 : i;
  if (face) return i <= 1 ? n1 - 1 : i >= n1 ? 2 : i;
  return i <= 1 ? n1 - 2 : i >= n1 ? 3 : i == n1 - 1 ? 2 : i;
}
// the plane left at plane k by apply_periodic_bc_z: centre arrays (n3 = nzg
// planes, two copies above) and W faces (n3 = nz)
__device__ __forceinline__ int zmap(int k, int nzg) { return k <= 1 ? nzg - 2 : k == nzg - 1 ? 2 : k >= nzg ? 3 : k; }
__device__ __forceinline__ int zmap_w(int k, int nz) { return k <= 1 ? nz - 1 : k >= nz ? 2 : k; }

// velocities of the box around (i,j), as FP64
template <typename T> struct LdBox {
  const T *U, *V, *W;
  long long c, px, pl;  // c: box index of (i-1, j, k = 0)
  int nz;
  __device__ LdBox(const Geo &g, const T *u, const T *v, const T *w, int i, int j, int)
      : U(u), V(v), W(w), c(bidx(g, i - 1, j, 0)), px(g.px), pl(g.plane), nz(g.nz) {}
  __device__ __forceinline__ void pre(int k) const {
    const long long o = c + 1 + min(k, nz) * pl;
    prefetch_l1(U + o);
    prefetch_l1(V + o);
    prefetch_l1(W + o);
  }
  __device__ __forceinline__ double at(const T *a, int s, int dj, int k) const {
    return (double)__ldg(a + c + s + dj * px + k * pl);
  }
  __device__ __forceinline__ double u(int s, int dj, int k) const { return at(U, s, dj, k); }
  __device__ __forceinline__ double v(int s, int dj, int k) const { return at(V, s, dj, k); }
  __device__ __forceinline__ double w(int s, int dj, int k) const { return at(W, s, dj, k); }
};

// the filtered velocities around (i,j), ghosts by index
struct LdHat {
  const double *U, *V, *W;
  int xu[2], xc[3], j, nxg, nz, nzg;
  long long pl;
  __device__ LdHat(const Geo &g, const double *u, const double *v, const double *w, int i, int j_, int periodic)
      : U(u), V(v), W(w), j(j_), nxg(g.nxg), nz(g.nz), nzg(g.nzg), pl((long long)g.nxg * g.nyg) {
    for (int s = 0; s < 2; ++s) xu[s] = xmap(i - 1 + s, g.nx, periodic, true) - 1;
    for (int s = 0; s < 3; ++s) xc[s] = xmap(i - 1 + s, g.nxg, periodic, false) - 1;
  }
  __device__ __forceinline__ void pre(int k) const {  // interior planes only
    const long long o = (min(k, nz - 1) - 1) * pl + (j - 1) * nxg;
    prefetch_l1(U + o + xu[1]);
    prefetch_l1(V + o + xc[1]);
    prefetch_l1(W + o + xc[1]);
  }
  __device__ __forceinline__ double u(int s, int dj, int k) const {
    return __ldg(U + (zmap(k, nzg) - 1) * pl + (j + dj - 1) * nxg + xu[s]);
  }
  __device__ __forceinline__ double v(int s, int dj, int k) const {
    return __ldg(V + (zmap(k, nzg) - 1) * pl + (j + dj - 1) * nxg + xc[s]);
  }
  __device__ __forceinline__ double w(int s, int dj, int k) const {
    return __ldg(W + (zmap_w(k, nz) - 1) * pl + (j + dj - 1) * nxg + xc[s]);
  }
};

// scale |S| Sij of every cell (i = 2..nxg-1, j = 2..nyg-1, k = 2..nzg-1) and,
// unless null, |S|
template <typename T, typename LD>
__global__ void __launch_bounds__(128) k_dyn_strain(Geo g, const T *__restrict__ U, const T *__restrict__ V,
                                                    const T *__restrict__ W, int periodic, double scale, P6 out,
                                                    double *__restrict__ S, int kchunk) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2, j = blockIdx.y * blockDim.y + threadIdx.y + 2;
  if (i > g.nxg - 1 || j > g.nyg - 1) return;
  const int k0 = 2 + blockIdx.z * kchunk, k1 = min(k0 + kchunk - 1, g.nzg - 1);
  const LD ld(g, U, V, W, i, j, periodic);
  StrainColumn<double, LD> col(ld, g.ax.F, g.ax.rF, g.ax.C, g.ax.rC, g.ay.F, g.ay.rF, g.ay.C, g.ay.rC, g.az.F, g.az.rF,
                               g.az.C, g.az.rC, i, j);
  col.start(k0);
  for (int k = k0; k <= k1; ++k) {
    double s[6];
    const double n = col.cell(k, s);
    const long long c = dix(i, j, k, g);
    const double f = scale * n;
#pragma unroll
    for (int m = 0; m < 6; ++m) out.p[m][c] = f * s[m];
    if (S) S[c] = n;
  }
}

constexpr double F1 = 1.0 / 6.0, F2 = 2.0 / 3.0;

// y weights of row j of the section ja..jb, and the rows they belong to
struct YW {
  double a, b, c;
  int jm, jp;
  __device__ YW(int j, int ja, int jb)
      : a(j == ja ? 0.0 : j == jb ? 1.0 / 3.0 : F1), b(F2), c(j == ja ? 1.0 / 3.0 : j == jb ? 0.0 : F1),
        jm(j == ja ? j : j - 1), jp(j == jb ? j : j + 1) {}
  __device__ __forceinline__ double operator()(double m, double o, double p) const {
    return __fma_rn(c, p, __fma_rn(a, m, b * o));
  }
};
__device__ __forceinline__ double f141(double m, double o, double p) { return __fma_rn(F1, m + p, F2 * o); }

// hat(U), hat(V), hat(W) on the interior of their own x and z ranges and all
// rows; blockIdx.z = 3 chunk + component
template <typename T>
__global__ void __launch_bounds__(256) k_dyn_filter(Geo g, const T *__restrict__ U, const T *__restrict__ V,
                                                    const T *__restrict__ W, P3 out, int kchunk) {
  const int q = blockIdx.z % 3;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 2, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int n1 = q == 0 ? g.nx : g.nxg, n2 = q == 1 ? g.ny : g.nyg, n3 = q == 2 ? g.nz : g.nzg;
  const int k0 = 2 + (blockIdx.z / 3) * kchunk, k1 = min(k0 + kchunk - 1, n3 - 1);
  if (i > n1 - 1 || j > n2 || k0 > k1) return;
  const T *__restrict__ a = q == 0 ? U : q == 1 ? V : W;
  const YW y(j, 1, n2);
  const long long om = bidx(g, i, y.jm, 0), oo = bidx(g, i, j, 0), op = bidx(g, i, y.jp, 0);
  auto plane = [&](int k) {  // the x and y sums of plane k
    const T *p = a + k * g.plane;
    double v[3];
#pragma unroll
    for (int s = 0; s < 3; ++s)
      v[s] = y((double)__ldg(p + om + s - 1), (double)__ldg(p + oo + s - 1), (double)__ldg(p + op + s - 1));
    return f141(v[0], v[1], v[2]);
  };
  double lo = plane(k0 - 1), mid = plane(k0);
  double *__restrict__ o = q == 0 ? out.p[0] : q == 1 ? out.p[1] : out.p[2];
  for (int k = k0; k <= k1; ++k) {
    prefetch_l1(a + oo + min(k + 3, n3) * g.plane);
    const double hi = plane(k + 1);
    o[dix(i, j, k, g)] = f141(lo, mid, hi);
    lo = mid;
    mid = hi;
  }
}

// nu_t(i,j,k) into the box: clipped, its Neumann rows (j = 1, nyg), and for
// LES = 3 the periodic x and z ghosts that take their value from it; an entry
// that the source's ghost copies overwrite is not written
template <typename T>
__device__ __forceinline__ void put_rows(const Geo &g, T *__restrict__ nut, int i, int j, int k, double v) {
  const T t = (T)(v > 0.0 ? v : 0.0);
  nut[bidx(g, i, j, k)] = t;
  if (j == 2) nut[bidx(g, i, 1, k)] = t;
  if (j == g.nyg - 1) nut[bidx(g, i, g.nyg, k)] = t;
}
template <typename T>
__device__ __forceinline__ void put_periodic(const Geo &g, T *__restrict__ nut, int i, int j, int k, double v) {
  const int gi = i == g.nxg - 2 ? 1 : i == 2 ? g.nxg - 1 : i == 3 ? g.nxg : 0;
  const int gk = k == g.nzg - 2 ? 1 : k == 2 ? g.nzg - 1 : k == 3 ? g.nzg : 0;
  if (i == g.nxg - 1 || k == g.nzg - 1) return;
  put_rows(g, nut, i, j, k, v);
  if (gi) put_rows(g, nut, gi, j, k, v);
  if (gk) put_rows(g, nut, i, j, gk, v);
  if (gi && gk) put_rows(g, nut, gi, j, gk, v);
}

// Lij, Mij and their contractions.  A warp owns 32 columns of one row j and
// gives its 30 inner ones; it walks up k.  Per plane a lane forms the y sums
// of the 15 filtered quantities at its own column (the centre velocities are
// averaged from the box there), the x sums take the two neighbours' by
// shuffles, and the z sums two planes carried in registers.  LES = 3 stores
// nu_t, LES = 2 Mij Lij and Mij Mij.
constexpr int DC_ROWS = 4;

template <typename T>
__global__ void __launch_bounds__(32 * DC_ROWS, 3)
    k_dyn_contract(Geo g, const T *__restrict__ U, const T *__restrict__ V, const T *__restrict__ W, P6 SS, P6 M0,
                   const double *__restrict__ S, int model, double *__restrict__ ml_out, double *__restrict__ mm_out,
                   T *__restrict__ nut, int kchunk) {
  const int lane = threadIdx.x, i = 1 + blockIdx.x * 30 + lane, j = blockIdx.y * DC_ROWS + threadIdx.y + 2;
  const int k0 = 2 + blockIdx.z * kchunk, k1 = min(k0 + kchunk - 1, g.nzg - 1);
  if (j > g.nyg - 1) return;  // whole warps
  const int periodic = model == 3;
  const int ic = min(i, g.nxg);                       // lanes past the last column repeat it
  const int im = xmap(ic, g.nxg, periodic, false);
  const bool moved = im != ic;
  const YW y(j, 2, g.nyg - 1);
  const int rows[3] = {y.jm, j, y.jp};
  auto U_ = [&](int x, int r, int k) { return (double)__ldg(U + bidx(g, x, r, k)); };
  auto V_ = [&](int x, int r, int k) { return (double)__ldg(V + bidx(g, x, r, k)); };
  auto W_ = [&](int x, int r, int k) { return (double)__ldg(W + bidx(g, x, r, k)); };
  const bool out = lane >= 1 && lane <= 30 && i <= g.nxg - 1;
  double lo[15], mid[15];
#pragma unroll
  for (int q = 0; q < 15; ++q) lo[q] = mid[q] = 0.0;
  for (int kk = k0 - 1; kk <= k1 + 1; ++kk) {
    const int km = zmap(kk, g.nzg);
    if (kk < k1) {  // row j two planes ahead (the block's other rows come from its other warps)
      const int kn = zmap(kk + 2, g.nzg);
      const long long b = bidx(g, ic, j, kn), c = dix(im, j, kn, g), o = dix(ic, j, kk + 1, g);
      prefetch_l1(U + b);
      prefetch_l1(V + b);
      prefetch_l1(W + b);
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        prefetch_l1(SS.p[m] + c);
        prefetch_l1(M0.p[m] + o);
      }
    }
    double v[15];
    {
      double a[3], b[3], c[3];  // centre velocities at (im, rows, km): the products' entries
      double vb = V_(im, rows[0] - 1, km);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        a[r] = 0.5 * (U_(im - 1, rows[r], km) + U_(im, rows[r], km));
        const double vt = V_(im, rows[r], km);
        // rows ja and jb repeat a row with a zero weight
        b[r] = 0.5 * ((r > 0 && rows[r] == rows[r - 1] ? V_(im, rows[r] - 1, km) : vb) + vt);
        vb = vt;
        c[r] = 0.5 * (W_(im, rows[r], km - 1) + W_(im, rows[r], km));
      }
      v[0] = y(a[0] * a[0], a[1] * a[1], a[2] * a[2]);
      v[1] = y(b[0] * b[0], b[1] * b[1], b[2] * b[2]);
      v[2] = y(c[0] * c[0], c[1] * c[1], c[2] * c[2]);
      v[3] = y(a[0] * b[0], a[1] * b[1], a[2] * b[2]);
      v[4] = y(a[0] * c[0], a[1] * c[1], a[2] * c[2]);
      v[5] = y(b[0] * c[0], b[1] * c[1], b[2] * c[2]);
      // the velocities alone: u with x ghosts only, v with none, w with z ghosts only
      if (kk != km) {
#pragma unroll
        for (int r = 0; r < 3; ++r) a[r] = 0.5 * (U_(im - 1, rows[r], kk) + U_(im, rows[r], kk));
      }
      if (kk != km || moved) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          b[r] = 0.5 * (V_(ic, rows[r] - 1, kk) + V_(ic, rows[r], kk));
          c[r] = 0.5 * (W_(ic, rows[r], km - 1) + W_(ic, rows[r], km));
        }
      }
      v[6] = y(a[0], a[1], a[2]);
      v[7] = y(b[0], b[1], b[2]);
      v[8] = y(c[0], c[1], c[2]);
    }
    const long long om = dix(im, rows[0], km, g), oo = dix(im, j, km, g), op = dix(im, rows[2], km, g);
#pragma unroll
    for (int m = 0; m < 6; ++m) v[9 + m] = y(__ldg(SS.p[m] + om), __ldg(SS.p[m] + oo), __ldg(SS.p[m] + op));
#pragma unroll
    for (int q = 0; q < 15; ++q)
      v[q] = f141(__shfl_up_sync(0xffffffffu, v[q], 1), v[q], __shfl_down_sync(0xffffffffu, v[q], 1));
    const int k = kk - 1;
    if (kk >= k0 + 1 && out) {
      double f[15];
#pragma unroll
      for (int q = 0; q < 15; ++q) f[q] = f141(lo[q], mid[q], v[q]);
      const long long c = dix(i, j, k, g);
      const double L[6] = {f[0] - f[6] * f[6], f[1] - f[7] * f[7], f[2] - f[8] * f[8],
                           f[3] - f[6] * f[7], f[4] - f[6] * f[8], f[5] - f[7] * f[8]};
      double ml = 0.0, mm = 0.0;
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        const double M = M0.p[m][c] - f[9 + m], t = m < 3 ? M : 2.0 * M;
        ml = __fma_rn(t, L[m], ml);
        mm = __fma_rn(t, M, mm);
      }
      if (model == 2) {
        ml_out[c] = ml;
        mm_out[c] = mm;
      } else {
        put_periodic(g, nut, i, j, k, -0.5 * (ml / mm) * S[c]);
      }
    }
#pragma unroll
    for (int q = 0; q < 15; ++q) {
      lo[q] = mid[q];
      mid[q] = v[q];
    }
  }
}

// LES = 2: <Mij Lij> / <Mij Mij> over k = 2..nzg-2, summed in k order, and
// nu_t; the x and z ghosts stay zero as in the source
template <typename T>
__global__ void __launch_bounds__(128) k_dyn_zavg(Geo g, const double *__restrict__ ml, const double *__restrict__ mm,
                                                  const double *__restrict__ S, T *__restrict__ nut) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y + 2;
  if (i > g.nxg) return;
  const long long pl = (long long)g.nxg * g.nyg, c = dix(i, j, 1, g);
  if (i == 1 || i == g.nxg) {
    for (int k = 1; k <= g.nzg; ++k) put_rows(g, nut, i, j, k, 0.0);
    return;
  }
  double a = 0.0, b = 0.0;
#pragma unroll 8
  for (int k = 2; k <= g.nzg - 2; ++k) {
    a += __ldg(ml + c + (k - 1) * pl);
    b += __ldg(mm + c + (k - 1) * pl);
  }
  const double cz = (a / (double)(g.nzg - 3)) / (b / (double)(g.nzg - 3));
  put_rows(g, nut, i, j, 1, 0.0);
#pragma unroll 4
  for (int k = 2; k <= g.nzg - 1; ++k) put_rows(g, nut, i, j, k, -0.5 * cz * __ldg(S + c + (k - 1) * pl));
  put_rows(g, nut, i, j, g.nzg, 0.0);
}

}  // namespace

size_t dyn_smagorinsky_work_bytes(int nxg, int nyg, int nzg) {
  return (size_t)W_COUNT * (size_t)nxg * nyg * nzg * sizeof(double);
}

template <typename T>
int launch_dyn_smagorinsky(const Geo &g, const T *U, const T *V, const T *W, double *work, int model, T *nut,
                           cudaStream_t st) {
  const size_t n = (size_t)g.nxg * g.nyg * g.nzg;
  double *w[W_COUNT];
  for (int q = 0; q < W_COUNT; ++q) w[q] = work + (size_t)q * n;
  P6 SS, M;
  for (int m = 0; m < 6; ++m) { SS.p[m] = w[W_SS + m]; M.p[m] = w[W_M + m]; }
  const P3 F{{w[W_F], w[W_F + 1], w[W_F + 2]}};
  const int periodic = model == 3, nk = g.nzg - 2, kc = 16;
  const dim3 sb(32, 4), sg((g.nxg - 2 + 31) / 32, (g.nyg - 2 + 3) / 4, (nk + kc - 1) / kc);
  k_dyn_strain<T, LdBox<T>><<<sg, sb, 0, st>>>(g, U, V, W, periodic, 1.0, SS, w[W_S], kc);
  const dim3 fb(32, 8), fg((g.nxg - 2 + 31) / 32, (g.nyg + 7) / 8, 3 * ((nk + kc - 1) / kc));
  k_dyn_filter<T><<<fg, fb, 0, st>>>(g, U, V, W, F, kc);
  k_dyn_strain<double, LdHat><<<sg, sb, 0, st>>>(g, w[W_F], w[W_F + 1], w[W_F + 2], periodic, 4.0, M, nullptr, kc);
  const int cc = 32;
  const dim3 cb(32, DC_ROWS), cg((g.nxg - 2 + 29) / 30, (g.nyg - 2 + DC_ROWS - 1) / DC_ROWS, (nk + cc - 1) / cc);
  k_dyn_contract<T><<<cg, cb, 0, st>>>(g, U, V, W, SS, M, w[W_S], model, w[W_F], w[W_F + 1], nut, cc);
  if (model != 2) return 4;
  k_dyn_zavg<T><<<dim3((g.nxg + 127) / 128, g.nyg - 2), 128, 0, st>>>(g, w[W_F], w[W_F + 1], w[W_S], nut);
  return 5;
}

template int launch_dyn_smagorinsky<double>(const Geo &, const double *, const double *, const double *, double *,
                                            int, double *, cudaStream_t);
template int launch_dyn_smagorinsky<float>(const Geo &, const float *, const float *, const float *, double *, int,
                                           float *, cudaStream_t);

}  // namespace blgpu
