// zsum.cu -- the mixed form's z transforms as FP32 products for the lengths
// beyond the tensor-core kernels (M/2+1 > 96; their tables of 4 x Q columns
// fill tensor memory at Q = 96).
//
// The real DFT over the half spectrum is two square products of order
// Q = M/2+1 (the algebra of zdft_tc.cu): forward X_k = f_k + f_{M-k} and
// Y_k = f_k - f_{M-k} (X_0 = f_0, X_{M/2} = f_{M/2}, Y = 0 there) give
//   Re C_m = sum_k X_k cos(2 pi m k / M),  Im C_m = sum_k Y_k (-sin);
// inverse X_k = Re C_k, Y_k = Im C_k (halved and zero at k = 0 and M/2) give
//   f_m, f_{M-m} = 2/M (sum_k X_k cos +- sum_k Y_k (-sin)).
// A CTA owns one row b and 64 kx columns; X and Y stay in shared memory, the
// tables stream through it in slabs of 16 k by 128 rows (double-buffered
// cp.async).  A thread forms 8 rows x 4 columns of both products with row
// pairs in FP32x2 multiply-adds: per k six 16-byte shared loads for 64
// multiply-adds.  Bounded by FP32 arithmetic (Q^2 multiply-adds per column
// and product): 1.6e9 at 512 x 96 x 256, 44 us at one per lane and clock.
// The direct sums (k_dft_z_*: one column group per lane, the table through L1)
// lose at every length they hold; us per launch at 258 x 65 x nz, forward /
// inverse, sums -> products: nz = 195 68 / 54 -> 33 / 31, 226 79 / 62 ->
// 37 / 35, 258 106 / 103 -> 68 / 66, 322 154 / 140 -> 99 / 94, 402 237 / 236 ->
// 118 / 109 (from Q = 145 on one CTA fits an SM); 514 and 769, which the sums
// do not hold: 217 / 202 and 311 / 290.
#include <cmath>
#include <vector>

#include "kernels.cuh"
#include "tma.cuh"

namespace blgpu {
namespace {

constexpr int ZC = 64;    // kx columns per CTA
constexpr int ZM = 128;   // rows per CTA and table pitch unit
constexpr int ZK = 16;    // k per table slab
constexpr int ZT = 256;   // threads

__device__ __forceinline__ void cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tma::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// tab[k][2][pitch]: cos and -sin of 2 pi m k / M, k < kpad (a multiple of ZK)
template <bool INV>
__global__ void __launch_bounds__(ZT, 2) k_zsum(Spec s, float *__restrict__ R, float2 *__restrict__ C,
                                                const float *__restrict__ tab, int pitch, int kpad) {
  extern __shared__ __align__(16) float zs_sm[];
  float *X = zs_sm, *Y = X + kpad * ZC, *T = Y + kpad * ZC;  // T[2][ZK][2][ZM]
  const int M = s.M, Q = s.MH, H = (M - 1) / 2;
  const bool even = (M & 1) == 0;
  const int b = blockIdx.y, x0 = blockIdx.x * ZC, m0 = blockIdx.z * ZM;
  const int tid = threadIdx.x;
  auto slab = [&](int q) {  // table rows k = q ZK .. of columns m0 .. m0 + ZM - 1
    float *dst = T + (q & 1) * (ZK * 2 * ZM);
    const float *src = tab + (size_t)q * ZK * 2 * pitch + m0;
    for (int e = tid; e < ZK * 2 * (ZM / 4); e += ZT) {
      const int r = e / (ZM / 4), c = e % (ZM / 4);
      cp16(dst + r * ZM + 4 * c, src + (size_t)r * pitch + 4 * c);
    }
    cp_commit();
  };
  slab(0);
  // X and Y of the CTA's columns; columns past N hold what R or C hold there
  // (never stored), columns past the pitch zeros
  for (int e = tid; e < kpad * (ZC / 4); e += ZT) {
    const int k = e / (ZC / 4), c = 4 * (e % (ZC / 4)), x = x0 + c;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), m = p;
    if (k < Q && x < s.rx) {
      const bool edge = k == 0 || (even && k == M / 2);
      if (!INV) {
        const float *r = R + (size_t)b * M * s.rx + x;
        p = __ldg(reinterpret_cast<const float4 *>(r + (size_t)k * s.rx));
        if (!edge) {
          const float4 f = p, w = __ldg(reinterpret_cast<const float4 *>(r + (size_t)(M - k) * s.rx));
          p = make_float4(f.x + w.x, f.y + w.y, f.z + w.z, f.w + w.w);
          m = make_float4(f.x - w.x, f.y - w.y, f.z - w.z, f.w - w.w);
        }
      } else {
        const float4 *r = reinterpret_cast<const float4 *>(C + ((size_t)b * Q + k) * s.rx + x);
        const float4 u = __ldg(r), v = __ldg(r + 1);
        const float h = edge ? 0.5f : 1.f;
        p = make_float4(h * u.x, h * u.z, h * v.x, h * v.z);
        if (!edge) m = make_float4(u.y, u.w, v.y, v.w);
      }
    }
    *reinterpret_cast<float4 *>(X + k * ZC + c) = p;
    *reinterpret_cast<float4 *>(Y + k * ZC + c) = m;
  }
  // warp: 32 rows (4 groups of 8) x 32 columns (8 groups of 4)
  const int warp = tid >> 5, lane = tid & 31;
  const int mr = 32 * (warp >> 1) + 8 * (lane >> 3), cc = 32 * (warp & 1) + 4 * (lane & 7);
  float2 re[4][4], im[4][4];  // [row pair][column]
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) re[r][c] = im[r][c] = make_float2(0.f, 0.f);
  const int nslab = kpad / ZK;
  for (int q = 0; q < nslab; ++q) {
    if (q + 1 < nslab) {
      slab(q + 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    const float *tq = T + (q & 1) * (ZK * 2 * ZM) + mr;
    const float *xq = X + q * ZK * ZC + cc, *yq = Y + q * ZK * ZC + cc;
#pragma unroll 2
    for (int k = 0; k < ZK; ++k) {
      const float4 c0 = *reinterpret_cast<const float4 *>(tq + k * 2 * ZM);
      const float4 c1 = *reinterpret_cast<const float4 *>(tq + k * 2 * ZM + 4);
      const float4 n0 = *reinterpret_cast<const float4 *>(tq + k * 2 * ZM + ZM);
      const float4 n1 = *reinterpret_cast<const float4 *>(tq + k * 2 * ZM + ZM + 4);
      const float4 xv = *reinterpret_cast<const float4 *>(xq + k * ZC);
      const float4 yv = *reinterpret_cast<const float4 *>(yq + k * ZC);
      const float2 cs[4] = {make_float2(c0.x, c0.y), make_float2(c0.z, c0.w), make_float2(c1.x, c1.y),
                            make_float2(c1.z, c1.w)};
      const float2 sn[4] = {make_float2(n0.x, n0.y), make_float2(n0.z, n0.w), make_float2(n1.x, n1.y),
                            make_float2(n1.z, n1.w)};
      const float xs[4] = {xv.x, xv.y, xv.z, xv.w}, ys[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 xx = make_float2(xs[c], xs[c]), yy = make_float2(ys[c], ys[c]);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          re[r][c] = __ffma2_rn(cs[r], xx, re[r][c]);
          im[r][c] = __ffma2_rn(sn[r], yy, im[r][c]);
        }
      }
    }
    __syncthreads();  // slab q read by all before q + 2 takes its place
  }
  const int x = x0 + cc;
  if (x >= s.N) return;
  const bool full = x + 3 < s.N;
  const float sc = 2.0f / (float)M;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int m = m0 + mr + r;
    if (m >= Q) break;
    float a[4], d[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      a[c] = (r & 1) ? re[r >> 1][c].y : re[r >> 1][c].x;
      d[c] = (r & 1) ? im[r >> 1][c].y : im[r >> 1][c].x;
    }
    if (!INV) {
      float2 *o = C + ((size_t)b * Q + m) * s.rx + x;
      if (full) {
        reinterpret_cast<float4 *>(o)[0] = make_float4(a[0], d[0], a[1], d[1]);
        reinterpret_cast<float4 *>(o)[1] = make_float4(a[2], d[2], a[3], d[3]);
      } else {
        for (int c = 0; c < 4 && x + c < s.N; ++c) o[c] = make_float2(a[c], d[c]);
      }
    } else {
      const bool two = m >= 1 && m <= H;  // rows m and M - m
      float *o = R + ((size_t)b * M + m) * s.rx + x;
      float *w = R + ((size_t)b * M + (M - m)) * s.rx + x;
      float f[4], h[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        f[c] = (a[c] + d[c]) * sc;
        h[c] = (a[c] - d[c]) * sc;
      }
      if (full) {
        *reinterpret_cast<float4 *>(o) = make_float4(f[0], f[1], f[2], f[3]);
        if (two) *reinterpret_cast<float4 *>(w) = make_float4(h[0], h[1], h[2], h[3]);
      } else {
        for (int c = 0; c < 4 && x + c < s.N; ++c) {
          o[c] = f[c];
          if (two) w[c] = h[c];
        }
      }
    }
  }
}

int kpad_of(const Spec &s) { return (s.MH + ZK - 1) / ZK * ZK; }
int pitch_of(const Spec &s) { return (s.MH + ZM - 1) / ZM * ZM; }
size_t zsum_smem(const Spec &s) { return ((size_t)2 * kpad_of(s) * ZC + 2 * ZK * 2 * ZM) * sizeof(float); }

}  // namespace

// M = 192 .. 767: above the tensor-core lengths, to the columns that fit a CTA
bool zsum_serves(const Spec &s) { return s.MH > 96 && zsum_smem(s) <= 227 * 1024; }

void zsum_tables(const Spec &s, std::vector<float> &t) {
  const int kp = kpad_of(s), pitch = pitch_of(s);
  t.assign((size_t)kp * 2 * pitch, 0.f);
  for (int k = 0; k < s.MH; ++k)
    for (int m = 0; m < s.MH; ++m) {
      const double a = 2.0 * M_PI * (double)(((long long)m * k) % s.M) / (double)s.M;
      t[((size_t)k * 2) * pitch + m] = (float)cos(a);
      t[((size_t)k * 2 + 1) * pitch + m] = (float)-sin(a);
    }
}

void launch_zsum(const Spec &s, float *R, float2 *C, const float *tab, int inverse, cudaStream_t st) {
  const size_t sm = zsum_smem(s);
  const dim3 grid((s.N + ZC - 1) / ZC, s.NM, pitch_of(s) / ZM);
  auto *k = inverse ? k_zsum<true> : k_zsum<false>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k<<<grid, ZT, sm, st>>>(s, R, C, tab, pitch_of(s), kpad_of(s));
}

}  // namespace blgpu
