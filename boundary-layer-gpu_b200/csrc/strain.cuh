// strain.cuh -- the rate of strain of compute_Sij (subgrid.f90:672-730) along
// a column of cells, shared by the Smagorinsky kernels.
//
// compute_Sij takes the diagonal terms at the cell centre and averages the
// off-diagonal ones from the four surrounding cell edges.  A thread owns the
// column (i,j) and walks up k: the edge values above cell k (the ones of
// index k+1 of the xz and yz edges) are those below cell k+1 and are carried,
// and so are the velocities of plane k+1, so a cell costs 17 loads and 19
// quotients where its 12 edges taken one by one cost 48 and 24.
// Every quotient is the source's a/b formed by Markstein's correction from
// the tabulated reciprocal (mdiv, common.cuh): RN(a/b) in FP64, within
// (1/2 + 2^-20) ulp of a/b in FP32.
//
// LD supplies the velocities as R: u(s, dj, k) is U(i-1+s, j+dj, k), s = 0, 1;
// v(s, dj, k) is V(i-1+s, j+dj, k), s = 0..2; w(s, dj, k) is W(i-1+s, j+dj, k),
// s = 0..2 (Fortran indices; LD may map ghost columns and planes); pre(k) starts
// the three fields' lines of plane k on their way.  Loads are what the kernels
// wait for most: 4.4 cycles of the 8.7 between a warp's instructions in the
// FP64 Smagorinsky kernel, 3.4 and 3.8 of about 8 in the dynamic model's.
#pragma once
#include "common.cuh"

namespace blgpu {

// the FP32 form of mdiv, three instructions.  b and rb are the FP64 spacing
// and its reciprocal, each rounded to FP32, so rb is within 2^-23 of 1/b but
// not its rounding: the result is RN(a/b + e), |e| < 2^-20 ulp
__device__ __forceinline__ float mdiv(float a, float b, float rb) {
  const float q = __fmul_rn(a, rb);
  return __fmaf_rn(__fmaf_rn(-q, b, a), rb, q);
}

__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

template <typename R, typename LD> struct StrainColumn {
  const LD &d;
  // spacings and reciprocals: x(i)-x(i-1), y(j)-y(j-1) and the centre spacings
  // below and above (xg: i, i+1; yg: j, j+1)
  R xF, rxF, yF, ryF, cx0, rcx0, cx1, rcx1, cy0, rcy0, cy1, rcy1;
  const R *zF, *rzF, *zC, *rzC;
  // carried: the xz and yz edges below cell k, the velocities of plane k the
  // edges above plane k-1 needed, and W(i,j,k-1)
  R e5a, e5b, e6a, e6b, u0, u1, v0, v1, wb;

  __device__ __forceinline__ StrainColumn(const LD &ld, const R *xF_, const R *xrF_, const R *xC, const R *xrC,
                                          const R *yF_, const R *yrF_, const R *yC, const R *yrC, const R *zF_,
                                          const R *zrF_, const R *zC_, const R *zrC_, int i, int j)
      : d(ld), xF(xF_[i]), rxF(xrF_[i]), yF(yF_[j]), ryF(yrF_[j]), cx0(xC[i - 1]), rcx0(xrC[i - 1]), cx1(xC[i]),
        rcx1(xrC[i]), cy0(yC[j - 1]), rcy0(yrC[j - 1]), cy1(yC[j]), rcy1(yrC[j]), zF(zF_), rzF(zrF_), zC(zC_),
        rzC(zrC_) {}

  // edges between planes k-1 and k from W of plane k-1 and u, v of both:
  // E5(i), E5(i+1) and E6(j), E6(j+1)
  __device__ __forceinline__ void edges_below(int k, R ub0, R ub1, R vb0, R vb1, R ut0, R ut1, R vt0, R vt1, R wm, R wc,
                                              R we, R ws, R wn) {
    const R h = (R)0.5, dz = zC[k - 1], rdz = rzC[k - 1];
    e5a = h * (mdiv(ut0 - ub0, dz, rdz) + mdiv(wc - wm, cx0, rcx0));
    e5b = h * (mdiv(ut1 - ub1, dz, rdz) + mdiv(we - wc, cx1, rcx1));
    e6a = h * (mdiv(vt0 - vb0, dz, rdz) + mdiv(wc - ws, cy0, rcy0));
    e6b = h * (mdiv(vt1 - vb1, dz, rdz) + mdiv(wn - wc, cy1, rcy1));
  }

  // to the state below cell k
  __device__ __forceinline__ void start(int k) {
    u0 = d.u(0, 0, k); u1 = d.u(1, 0, k); v0 = d.v(1, -1, k); v1 = d.v(1, 0, k);
    wb = d.w(1, 0, k - 1);
    edges_below(k, d.u(0, 0, k - 1), d.u(1, 0, k - 1), d.v(1, -1, k - 1), d.v(1, 0, k - 1), u0, u1, v0, v1,
                d.w(0, 0, k - 1), wb, d.w(2, 0, k - 1), d.w(1, -1, k - 1), d.w(1, 1, k - 1));
  }

  // s[0..5] = S11 S22 S33 S12 S13 S23 of cell k and |S|; moves up one cell
  __device__ __forceinline__ R cell(int k, R (&s)[6]) {
    const R h = (R)0.5, q = (R)0.25;
    d.pre(k + 3);
    const R us0 = d.u(0, -1, k), us1 = d.u(1, -1, k), un0 = d.u(0, 1, k), un1 = d.u(1, 1, k);
    const R vw0 = d.v(0, -1, k), vw1 = d.v(0, 0, k), ve0 = d.v(2, -1, k), ve1 = d.v(2, 0, k);
    const R wm = d.w(0, 0, k), wc = d.w(1, 0, k), we = d.w(2, 0, k), ws = d.w(1, -1, k), wn = d.w(1, 1, k);
    const R ut0 = d.u(0, 0, k + 1), ut1 = d.u(1, 0, k + 1), vt0 = d.v(1, -1, k + 1), vt1 = d.v(1, 0, k + 1);
    s[0] = mdiv(u1 - u0, xF, rxF);
    s[1] = mdiv(v1 - v0, yF, ryF);
    s[2] = mdiv(wc - wb, zF[k], rzF[k]);
    // xy edges (i,j), (i+1,j), (i,j+1), (i+1,j+1)
    const R a = h * (mdiv(u0 - us0, cy0, rcy0) + mdiv(v0 - vw0, cx0, rcx0));
    const R b = h * (mdiv(u1 - us1, cy0, rcy0) + mdiv(ve0 - v0, cx1, rcx1));
    const R c = h * (mdiv(un0 - u0, cy1, rcy1) + mdiv(v1 - vw1, cx0, rcx0));
    const R e = h * (mdiv(un1 - u1, cy1, rcy1) + mdiv(ve1 - v1, cx1, rcx1));
    s[3] = q * (a + b + c + e);
    const R p5a = e5a, p5b = e5b, p6a = e6a, p6b = e6b;
    edges_below(k + 1, u0, u1, v0, v1, ut0, ut1, vt0, vt1, wm, wc, we, ws, wn);
    s[4] = q * (p5a + p5b + e5a + e5b);
    s[5] = q * (p6a + p6b + e6a + e6b);
    u0 = ut0; u1 = ut1; v0 = vt0; v1 = vt1; wb = wc;
    R S = 0;
#pragma unroll
    for (int m = 0; m < 6; ++m) S = S + (m < 3 ? (R)2 : (R)4) * s[m] * s[m];
    return sqrt(S);
  }
};

// |S| of cell (i,j,k) by divisions.  mdiv forms a NaN where a difference or its
// quotient is infinite and the division gives an infinity, so a caller that
// keeps |S| of such cells (a run that has blown up) takes it from here where
// cell() returned a NaN.  It does so after its column and in a function of its
// own (512 x 96 x 256, FP64: 242 -> 240 us per launch; inlined after the
// column 303, called cell by cell 253).
template <typename R, typename LD>
__device__ __forceinline__ R strain_divided(const LD &d, const R *xF, const R *xC, const R *yF, const R *yC,
                                            const R *zF, const R *zC, int i, int j, int k) {
  const R h = (R)0.5, q = (R)0.25;
  // xy edge (i + s, j + t), xz edge (i + s, k + t), yz edge (j + s, k + t)
  auto xy = [&](int s, int t) {
    return h * ((d.u(s, t, k) - d.u(s, t - 1, k)) / yC[j - 1 + t] +
                (d.v(1 + s, t - 1, k) - d.v(s, t - 1, k)) / xC[i - 1 + s]);
  };
  auto xz = [&](int s, int t) {
    return h * ((d.u(s, 0, k + t) - d.u(s, 0, k + t - 1)) / zC[k - 1 + t] +
                (d.w(1 + s, 0, k + t - 1) - d.w(s, 0, k + t - 1)) / xC[i - 1 + s]);
  };
  auto yz = [&](int s, int t) {
    return h * ((d.v(1, s - 1, k + t) - d.v(1, s - 1, k + t - 1)) / zC[k - 1 + t] +
                (d.w(1, s, k + t - 1) - d.w(1, s - 1, k + t - 1)) / yC[j - 1 + s]);
  };
  const R m[6] = {(d.u(1, 0, k) - d.u(0, 0, k)) / xF[i], (d.v(1, 0, k) - d.v(1, -1, k)) / yF[j],
                  (d.w(1, 0, k) - d.w(1, 0, k - 1)) / zF[k], q * (xy(0, 0) + xy(1, 0) + xy(0, 1) + xy(1, 1)),
                  q * (xz(0, 0) + xz(1, 0) + xz(0, 1) + xz(1, 1)), q * (yz(0, 0) + yz(1, 0) + yz(0, 1) + yz(1, 1))};
  R S = 0;
#pragma unroll
  for (int e = 0; e < 6; ++e) S = S + (e < 3 ? (R)2 : (R)4) * m[e] * m[e];
  return sqrt(S);
}

}  // namespace blgpu
