// Sparse k-pair contraction (alg_sparseP / alg_Pin_is_sparse): only the stored elements of P1, P2.
//
// The reference keeps, per pair, the elements with |P| > thr_sparseP (default 1e-40) in COO form and
// multiplies them with sparse_zgemm (comm/sparse_matrix.cpp:6-40; sparse2D.h:9-200; the branch of
// evolve_eph.cpp:67-82, phases per element by compute_sPt, evolve_eph.cpp:194-203). Here the phases
// are factorised per k as in the dense forms (rt = conj(D) o rho, st = conj(D) o (1 - rho), the
// finish multiplies by D), and the products are regrouped by the k-point they update:
//
//   every pair (k, k') gives a forward contribution to target k from source k' with
//     X-matrix P1 (read by rows: X_k[a] += sum_b P1[a][b] rt_k'[b]) and
//     Y-matrix P2 (read by columns: Y_k[b] += sum_a st_k'[a] P2[a][b]);
//   a pair with k < k' also gives a reverse contribution to target k' from source k with
//     X-matrix conj(P2) (rows) and Y-matrix conj(P1) (columns)        (evolve_eph.cpp:101-106).
//
// Every output element (k, X or Y, a) is owned by one thread, which runs over its products of all
// the contributions to k: no atomics, and a fixed order of the sums. Each stored element is kept
// twice (once per direction, the reverse copy conjugated), which the forward/reverse symmetry of
// the dense kernels avoids; the sparse form pays where the fill is low enough (bench --sparse).
//
// Layout (ELL, lane-interleaved): the products of thread lane l of k-point k are a list of
// (element value, index into the coordinate array rs) -- the index names the source k-point, rt or
// st, and the element's other band-pair index. The lists of the 2 nb^2 threads of a k-point are
// padded with zeros to the longest one, L_k, and stored interleaved: product j of lane l at
// base_k + j (2 nb^2) + l. Consecutive threads then read consecutive values (coalesced), and the
// loads of a thread's products do not depend on each other.
//
// Arithmetic. On the FP64 pipe (1.7 multiply-adds per clock and SM) the products of 60k nb = 4 pairs with 18 % of
// the elements stored take 128 us against 28 us of HBM time (9.4M products of 20 bytes). k_pairs_sparse_fx multiplies on the integer pipes, as
// dmd_pairs_fx.cuh does. Neighbours in a list come from different pairs, so nothing is scaled by blocks here: an element
// keeps its own exponent (the larger of its two parts) in the low bits of its index word, a coordinate is
// aligned when it is loaded, and a thread's sums move their exponent T up when a product or the sum itself outgrows it:
//   element   p = q 2^(emax - d - 60),  q = h 2^32 + l,  |q| <= 2^60 (FP64 keeps 53 bits)
//   coordinate r = m 2^(f - 1075);  R = (m 2^6) >> (T - (f - d)) = rh 2^32 + rl,  |R| < 2^59
//   sum       (A0 + A1 2^-32) 2^(emax + T - 1077),  A0 += h rh,  A1 += h rl + l rh, exact in 64 bits for the 8 real
//             terms of 4 products (A0 2^58 beside the 2^61 at which it is shifted, A1 8 (2^59 + 2^58))
// It takes 51 us there (47 % of the HBM rate: what bounds it is the latency of index, then coordinate, with 21 warps
// per SM; the next chunk's index words are loaded ahead: 10 us of the step's 267); an RK4 step of 2000 k-points went from
// 702 to 257 us, of 100 from 206 to 60.
// The dropped l rl is at most 2^-57 of the largest product, the bits lost to a shift 2^-56 of it, and a sum is rounded
// to FP64 once.
#pragma once
#include <climits>
#include <type_traits>

#include "dmd_common.cuh"
#include "dmd_pairs_fx.cuh"

namespace dmd {

constexpr int kSpPBits = 60;     // element bits
constexpr int kSpDBits = 11;     // exponent bits of an index word
constexpr unsigned kSpDMax = (1u << kSpDBits) - 1;
constexpr int kSpT0 = 64;        // lowest T: zeros (f = 0) shift to 0

// Elements to fixed point in place, emax = fx_expo of the largest; the exponents into the index words
__global__ void k_sparse_quantise(long long n, int emax, double2* __restrict__ val, int* __restrict__ gidx) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 v = val[i];
  const int d = emax - fx_expo(fmax(fabs(v.x), fabs(v.y)));  // 0 to 1924
  const int2 x = fx_digits(v.x, kSpPBits - emax + d), y = fx_digits(v.y, kSpPBits - emax + d);
  // (the imaginary digits are negated: not from the smallest integer)
  reinterpret_cast<int4*>(val)[i] = make_int4(x.x, x.y, y.x, max(y.y, -INT_MAX));
  gidx[i] = (int)((unsigned)gidx[i] << kSpDBits | (unsigned)d);
}

// (a0 2^32 + a1) >> s for a folded sum (a1 < 2^32)
__device__ __forceinline__ void sp_shift(long long& a0, unsigned& a1, int s) {
  if (s < 32) {
    a1 = __funnelshift_r(a1, (unsigned)a0, s);
    a0 >>= s;
  } else {
    a1 = (unsigned)(a0 >> min(s - 32, 63));
    a0 >>= min(s, 63);
  }
}
// digits of a coordinate aligned to T: n = T - (f - d) >= 0
__device__ __forceinline__ int2 sp_digits(double x, int n) {
  const int hi = __double2hiint(x);
  const long long m = ((long long)((hi & 0xfffff) | 0x100000) << 38 | (long long)(unsigned)__double2loint(x) << 6) >> min(n, 63);
  const long long q = hi < 0 ? -m : m;  // (the shift first: towards zero, so that -0 gives 0)
  const int l = (int)q;
  return make_int2((int)(q >> 32) + (int)((unsigned)l >> 31), l);
}

template <int NB, int S>
__global__ void __launch_bounds__(256) k_pairs_sparse_fx(int nk, int emax, const long long* __restrict__ base,
                                                         const int* __restrict__ len, const int4* __restrict__ val,
                                                         const unsigned* __restrict__ gidx, const double2* __restrict__ rs,
                                                         double2* __restrict__ acc) {
  constexpr int TPR = 2 * NB * NB, GS = 256 / S;
  __shared__ double2 part[S > 1 ? 256 : 1];
  const int s = threadIdx.x / GS;
  const long long g = blockIdx.x * (long long)GS + threadIdx.x % GS;
  const long long k = g / TPR;
  const int l = (int)(g - k * TPR);
  const int L = k < nk ? len[k] : 0;
  const int4* vp = val + (k < nk ? base[k] + l : 0);
  const unsigned* ip = gidx + (k < nk ? base[k] + l : 0);
  long long x0 = 0, x1 = 0, y0 = 0, y1 = 0;  // A0, A1 of the real and the imaginary part
  int T = kSpT0, top = 0;
  unsigned un[4];  // the next chunk's index words
  auto index = [&](int j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) un[i] = j + i < L ? __ldcs(ip + (size_t)(j + i) * TPR) : 0u;
  };
  auto chunk = [&](int j, auto tail) {
    int4 v[4];
    unsigned u[4];
    double2 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool ok = !decltype(tail)::value || j + i < L;
      u[i] = un[i];
      r[i] = ok ? __ldg(rs + (u[i] >> kSpDBits)) : mk2(0.0, 0.0);
      v[i] = ok ? __ldcs(vp + (size_t)(j + i) * TPR) : make_int4(0, 0, 0, 0);
    }
    index(j + 4 * S);
    int gx[4], gy[4], gm = T;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = (int)(u[i] & kSpDMax);
      const int fx = (__double2hiint(r[i].x) >> 20) & 0x7ff, fy = (__double2hiint(r[i].y) >> 20) & 0x7ff;
      top = max(top, max(fx, fy));
      gx[i] = fx - d;
      gy[i] = fy - d;
      gm = max(gm, max(gx[i], gy[i]));
    }
    const int hx = (int)(x0 >> 32), hy = (int)(y0 >> 32);
    if (gm > T || max(hx ^ (hx >> 31), hy ^ (hy >> 31)) >= 1 << 29) {
      const int n = max(gm - T, 3);
      unsigned lx = (unsigned)x1, ly = (unsigned)y1;
      sp_shift(x0, lx, n);
      sp_shift(y0, ly, n);
      x1 = lx;
      y1 = ly;
      T += n;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int2 c = sp_digits(r[i].x, T - gx[i]), e = sp_digits(r[i].y, T - gy[i]);
      fx_mad(x0, x1, v[i].x, v[i].y, c);
      fx_mad(x0, x1, -v[i].z, -v[i].w, e);
      fx_mad(y0, y1, v[i].x, v[i].y, e);
      fx_mad(y0, y1, v[i].z, v[i].w, c);
    }
    x1 = fx_fold(x0, x1);
    y1 = fx_fold(y0, y1);
  };
  int j = 4 * s;
  index(j);
  for (; j + 4 <= L; j += 4 * S) chunk(j, std::false_type());
  if (j < L) chunk(j, std::true_type());
  double2 sum;
  if (top == 0x7ff) {  // an infinite or NaN coordinate: in FP64
    sum = mk2(0.0, 0.0);
    for (j = 4 * s; j < L; j += 4 * S)
      for (int i = j; i < min(j + 4, L); ++i) {
        const int4 v = vp[(size_t)i * TPR];
        const unsigned u = ip[(size_t)i * TPR];
        const int e = emax - (int)(u & kSpDMax) + kFxPBits - kSpPBits;
        sum = cfma(mk2(fx_decode(v.x, v.y, e), fx_decode(v.z, v.w, e)), rs[u >> kSpDBits], sum);
      }
  } else {
    const int e = emax + T - 1077;
    sum = mk2(scalbn(fma((double)(unsigned)x1, 0x1p-32, (double)x0), e), scalbn(fma((double)(unsigned)y1, 0x1p-32, (double)y0), e));
  }
  if constexpr (S > 1) {
    part[threadIdx.x] = sum;
    __syncthreads();
    if (s) return;
#pragma unroll
    for (int i = 1; i < S; ++i) sum = mk2(sum.x + part[i * GS + threadIdx.x].x, sum.y + part[i * GS + threadIdx.x].y);
  }
  if (k < nk) acc[(size_t)k * TPR + l] = sum;
}

template <int NB>
__global__ void __launch_bounds__(256) k_pairs_sparse(int nk, const long long* __restrict__ base,
                                                      const int* __restrict__ len, const double2* __restrict__ val,
                                                      const int* __restrict__ gidx, const double2* __restrict__ rs,
                                                      double2* __restrict__ acc) {
  constexpr int TPR = 2 * NB * NB;
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long k = g / TPR;
  if (k >= nk) return;
  const int l = (int)(g - k * TPR);
  const int L = len[k];
  const double2* vp = val + base[k] + l;
  const int* ip = gidx + base[k] + l;
  double2 s0 = mk2(0.0, 0.0), s1 = mk2(0.0, 0.0);
  int j = 0;
  for (; j + 4 <= L; j += 4) {
    const double2 v0 = __ldg(vp + (size_t)j * TPR), v1 = __ldg(vp + (size_t)(j + 1) * TPR);
    const double2 v2 = __ldg(vp + (size_t)(j + 2) * TPR), v3 = __ldg(vp + (size_t)(j + 3) * TPR);
    const int i0 = __ldg(ip + (size_t)j * TPR), i1 = __ldg(ip + (size_t)(j + 1) * TPR);
    const int i2 = __ldg(ip + (size_t)(j + 2) * TPR), i3 = __ldg(ip + (size_t)(j + 3) * TPR);
    s0 = cfma(v0, __ldg(rs + i0), s0);
    s1 = cfma(v1, __ldg(rs + i1), s1);
    s0 = cfma(v2, __ldg(rs + i2), s0);
    s1 = cfma(v3, __ldg(rs + i3), s1);
  }
  for (; j < L; ++j) s0 = cfma(__ldg(vp + (size_t)j * TPR), __ldg(rs + __ldg(ip + (size_t)j * TPR)), s0);
  acc[(size_t)k * TPR + l] = mk2(s0.x + s1.x, s0.y + s1.y);
}

}  // namespace dmd
