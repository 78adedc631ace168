// The FP64 k-pair contraction on the integer pipes: block-scaled fixed point (layout in dmd_layout.h,
// coordinates and sums as in dmd_pairs_cb.cuh).
//
// Why. This part multiplies FP64 at 1.7 lanes per clock and SM, but adds a 32 x 32 -> 64-bit integer
// product (mad.wide) at 61 (both measured). The contraction needs 16 nb^4 flops per pair: 2.35 ms on the FP64
// pipe for 9.7M nb = 2 pairs, 0.75 ms of HBM time. In two-digit fixed point a multiply-add is three
// mad.wide, a third of the HBM time. Measured per RK4 step, 2.5M nb = 2 pairs (1.27 GB a launch): 920 us (the
// FP64 pipe: 3.3 ms); 409k nb = 4 pairs (3.35 GB): 2.26 ms, 6.0 TB/s; 70k nb = 2 pairs in L2: 83 us (330). What bounds it
// is the issue rate (50 %): per row block and matrix 192 mad.wide of some 750 instructions, the rest mainly
// the cross-lane sums of the forward partials.
//
// Operators. The elements of a row block's line (Q1 row or Q2 column: the elements of one output, for up
// to 32 / 8 pairs) are split in two groups -- products with a diagonal and with an off-diagonal
// coordinate, which differ by the spin mixing -- and each group shares a binary exponent ex:
//   q = p 2^(61 - ex) rounded to an integer = h 2^32 + l,  l signed,  |h| <= 2^29
// in the 8 bytes of the double that it replaces: 61 bits below the group's largest element (FP64 keeps 53
// below each element). An element of the layout is (re_h, re_l, im_h, im_l).
// Coordinates. 59 bits (the rows' of nb = 4: 57) below the largest one of their group: the column's over the
// work item's 32 (8) columns; a row's times the line's 2^ex over the item's rows (so the reverse sums,
// which run over the item's rows, need no shift per row block). Built from the FP64 coordinates once per
// item (columns) or row block (rows).
// Sums. With rh, rl the digits of a coordinate, A0 += h rh and A1 += h rl + l rh are exact in 64 bits: A0
// takes the 64 (96) terms of a forward sum over the warp or the 128 (512) of a reverse sum over an
// item, A1 four lines' terms of 2^60 + 2^58 before it is folded into A0. What is dropped is l rl, at most 2^-58 of
// the group's largest product. A forward sum is rounded to 2^-56 of it per lane and added over the
// warp as integers, so a row block's sum is rounded to FP64 once; then one FP64 reduction in L2 per row
// block and value (the FP64 kernel issues one per pair and value). Reverse sums keep A1's remainder and are exact
// to the end of the item.
//
// Weak sums. All this is relative to the largest product that an item's exponents allow, which need not be near the ones
// that a sum has: a cold state's occupations range over tens of bits within 32 columns, and detailed balance pairs the large ones with
// small elements. So a sum is checked when it is known: a row block's forward sums against the unit of their exponents
// (error 2^-55 of it, root mean square), a column's reverse sums against theirs (2^-56.5; nb = 4 2^-54.5), over the lines and
// elements of the matrix. Below 2^-7 (2^-8; nb = 4 2^-7) of it they are not added but listed, and the gated launch sums them in
// FP64: each k-point's own largest sum keeps some 2^-48, as FP64 sums of a few hundred terms do. At 300 K next to none is listed. The check
// takes 1 to 4 % of the main launch (2.5M pairs 205 -> 212 us, 70k 13.4 -> 13.8, 46k nb = 4 pairs 91.9 -> 93.5); an evaluation with
// some sums listed 2 to 3 us more, one of uniformly random exponents over 60 bits 300 us in place of 218 (the FP64 pipe: 800).
// A state with a non-finite coordinate has no scale: the prep kernel raises bit 1 of the flag, the first
// launch returns and the gated one (which otherwise carries the anti-Hermitian part of a state that is not Hermitian,
// bit 0) contracts in FP64 from the decoded elements, so NaN and infinities spread as they do in FP64. Operators
// with a non-finite element are never converted (dmd_api.cu). Row blocks are split where their pairs are of too uneven strength
// for one exponent (k_fx_class).
#pragma once
#include <type_traits>

#include "dmd_common.cuh"
#include "dmd_layout.h"
#include "dmd_pairs_cb.cuh"
#include "dmd_tma.cuh"

namespace dmd {

constexpr int kFxPBits = 61;         // operator bits
constexpr int kFxCBits = 59;         // column coordinate bits
constexpr int kFxBase = 32;          // digit base 2^32
constexpr int kFxExZero = -20000;    // exponent of a group without a nonzero element
// Bits below the unit from which on sums are listed. A column that lies that far below by its elements alone (k_fx_static) is weak here
// and most often not elsewhere: it is listed where its sum lies kFxWeakMore bits lower still, or fx_weak_most below the unit.
constexpr int kFxWeakRow = 7, kFxWeakMore = 5;
__host__ __device__ constexpr int fx_weak_column(int nb) { return nb == 2 ? 8 : 7; }  // (the row digits: fx_row_bits)
__host__ __device__ constexpr int fx_weak_most(int nb) { return fx_weak_column(nb) + 4; }

// a listed sum: row block x's lines of flush z, or item x's columns z (bits), of column block y; w: matrix, 2: columns
typedef int4 FxWeak;

// bits of the row coordinates: a reverse sum's 128 (nb = 2) or 512 (nb = 4) products stay below 2^63
// in units of 2^32
__host__ __device__ constexpr int fx_row_bits(int nb) { return nb == 2 ? 59 : 57; }

// e with |x| < 2^e (0 and tiny values: -900, far below any scale that matters and safe to invert)
__device__ __forceinline__ int fx_expo(double x) {
  const int f = ((__double2hiint(x) >> 20) & 0x7ff) - 1022;
  return f < -900 ? -900 : f;
}
// whether these are zero in every lane
__device__ __forceinline__ bool fx_all_zero(double a, double b, double c, double d) {
  const long long u = __double_as_longlong(a) | __double_as_longlong(b) | __double_as_longlong(c) | __double_as_longlong(d);
  return !__any_sync(0xffffffffu, (u << 1) != 0);
}
// x 2^s rounded to an integer (|x 2^s| < 2^62) and split into signed digits: q = h 2^32 + l. Integer
// arithmetic: the FP64 pipe's conversions and products would cost as much as the item's sums.
__device__ __forceinline__ int2 fx_digits(double x, int s) {
  const long long b = __double_as_longlong(x);
  const int f = (int)(b >> 52) & 0x7ff;
  long long q = (b & 0xfffffffffffffLL) | (f ? 1LL << 52 : 0LL);
  const int sh = (f ? f : 1) - 1075 + s;  // <= 9
  q = sh >= 0 ? q << sh : (sh < -54 ? 0LL : (q + (1LL << (-sh - 1))) >> -sh);
  if (b < 0) q = -q;
  const int l = (int)q;
  return make_int2((int)((q - l) >> kFxBase), l);
}
// x 2^e for a converted integer x (0 or 1 <= |x| <= 2^63): an addition to the exponent field where every such
// result is normal
__device__ __forceinline__ double fx_scale(double x, int e) {
  if (e < -1000 || e > 900) return scalbn(x, e);
  const int hi = __double2hiint(x);
  return __hiloint2double(hi ? hi + (int)((unsigned)e << 20) : 0, __double2loint(x));
}
__device__ __forceinline__ double fx_decode(int h, int l, int ex) {
  // (a group's exponent is kFxExZero or above -900: the factor is a normal number, and short code matters where this is
  // called: as scalbn the listed sums' 50 KB of instructions took longer to fetch than to run)
  return (double)((long long)h * (1LL << kFxBase) + l) * __hiloint2double(ex < -900 ? 0 : (ex - kFxPBits + 1023) << 20, 0);
}
__device__ __forceinline__ void fx_mul(long long& a0, long long& a1, int h, int l, int2 r, long long a1_0) {
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(a0) : "r"(h), "r"(r.x));
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(a1) : "r"(h), "r"(r.y), "l"(a1_0));
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a1) : "r"(l), "r"(r.x));
}
__device__ __forceinline__ int4 fx_lds(uint32_t addr) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void fx_mad(long long& a0, long long& a1, int h, int l, int2 r) {
  // asm: written as 64-bit sums of products the compiler regroups them into trees with extra adds and moves
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a0) : "r"(h), "r"(r.x));
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a1) : "r"(h), "r"(r.y));
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a1) : "r"(l), "r"(r.x));
}
// carries of a1 into a0; returns a1's remainder in [0, 2^32)
__device__ __forceinline__ unsigned fx_fold(long long& a0, long long a1) {
  a0 += a1 >> kFxBase;
  return (unsigned)a1;
}

// Whether line element b of a pair's quarter qg, at step i of the loop, is a diagonal coordinate's: nb = 2
// walks b = 0..3 (diagonal: 0 and 3); nb = 4 walks its quarter from the diagonal element b = 4 qg + qg on
template <int NB>
__host__ __device__ constexpr int fx_group(int i) {
  return NB == 2 ? ((i == 1 || i == 2) ? 1 : 0) : (i == 0 ? 0 : 1);
}

// Which pairs of a row block may share its exponents. An element is off by at most 2^-62 of its group's largest in the
// block; a group within kFxSpread = 10 bits of it by 2^-51 of its own largest, in a sum of FP64's 2^-53 per term. A pair
// goes to a row block of its own (class 1, 2, ... by the same rule among those left) where the largest element of a matrix lies
// further below the block's, or a group that is no weaker than the others of its row's or column's k-point (spin-flip elements; kmax, within
// kFxSame bits): a single small element beside larger ones of the same sum may lose its low bits. At 300 K that makes 0.1 to 1 % more
// row blocks (2^8 would make 2 to 10 %; counting every small group 33 % where 82 % of the elements are zero).
// One warp per row block: nb = 2 a lane per pair, nb = 4 four lanes, 8 lines each. First (pass 0) kmax[k][line][group] and, in
// `bad`: [0] a non-finite element or a group below 2^-900, where fx_expo stops, [1] 1100 + the largest element's exponent.
constexpr int kFxSpread = 10, kFxSame = 4, kFxKmax0 = 30000;
template <int NB>
__global__ void __launch_bounds__(128) k_fx_class(long long nrb, const RowBlock* __restrict__ rbs, const int* __restrict__ rbJ,
                                                  const double2* __restrict__ P, int pass, int* __restrict__ kmax,
                                                  uint8_t* __restrict__ cls, int* __restrict__ bad) {
  constexpr int NB2 = NB * NB, NE = 2 * NB2 * NB2, S = NB == 2 ? 32 : 8, LPL = 8;
  constexpr unsigned FULL = 0xffffffffu;
  const long long r = blockIdx.x * 4LL + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31, slot = lane % S;
  if (r >= nrb) return;
  const RowBlock b = rbs[r];
  const int n = __popc(b.mask);
  const double2* p = P + (size_t)b.pair0 * NE + (size_t)(lane / S) * LPL * NB2 * n + slot;
  int ex[LPL][2], top = -1100;
  bool ok = true;
#pragma unroll
  for (int L = 0; L < LPL; ++L) {
    double mx[2] = {0.0, 0.0};
    if (slot < n) {
#pragma unroll
      for (int e = 0; e < NB2; ++e) {
        const double2 v = p[(size_t)(L * NB2 + e) * n];
        ok = ok && isfinite(v.x) && isfinite(v.y);
        double& m = mx[e / NB == e % NB ? 0 : 1];
        m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
      }
    }
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      ex[L][g] = mx[g] > 0.0 ? fx_expo(mx[g]) : kFxExZero;
      ok = ok && ex[L][g] != -900;
      top = max(top, ex[L][g]);
    }
  }
  int col = 0;  // the slot's column
  for (int i = 0, q = -1; i < S; ++i)
    if ((b.mask >> i) & 1u && ++q == slot) col = rbJ[r] * S + i;
  constexpr int NG = 4 * NB2;  // groups of a pair
  int* const krow = kmax + (size_t)b.row * NG + (lane / S) * LPL * 2;
  int* const kcol = kmax + (size_t)col * NG + (lane / S) * LPL * 2;
  if (!pass) {
    if (!ok) *bad = 1;
    top = __reduce_max_sync(FULL, top);
    if (lane == 0) atomicMax(bad + 1, top + 1100);
#pragma unroll
    for (int i = 0; i < 2 * LPL; ++i) {
      const int e = ex[i / 2][i % 2];
      int m = slot < n ? e : kFxExZero;
#pragma unroll
      for (int o = 1; o < S; o <<= 1) m = max(m, __shfl_xor_sync(FULL, m, o));
      if (slot == 0 && m != kFxExZero) atomicMax(&krow[i], m + kFxKmax0);
      if (slot < n && e != kFxExZero && ((b.revmask >> (col % S)) & 1u)) atomicMax(&kcol[i], e + kFxKmax0);
    }
    return;
  }
  unsigned same = 0;  // groups as strong as the others of a k-point
  if (slot < n) {
#pragma unroll
    for (int i = 0; i < 2 * LPL; ++i) {
      const int e = ex[i / 2][i % 2] + kFxKmax0 + kFxSame;
      if (e >= krow[i] || (((b.revmask >> (col % S)) & 1u) && e >= kcol[i])) same |= 1u << i;
    }
  }
  int most[2] = {kFxExZero, kFxExZero};  // the pair's largest of each matrix (nb = 4: of the lane's)
#pragma unroll
  for (int i = 0; i < 2 * LPL; ++i) {
    int& q = most[NB == 2 ? i / (2 * NB2) : 0];
    q = max(q, ex[i / 2][i % 2]);
  }
  if (NB == 4) most[0] = max(most[0], __shfl_xor_sync(FULL, most[0], 8));
  bool open = slot < n;
  for (int c = 0; __any_sync(FULL, open); ++c) {
    bool in = open;
#pragma unroll
    for (int L = 0; L < LPL; ++L)
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        int m = open ? ex[L][g] : kFxExZero;
#pragma unroll
        for (int o = 1; o < S; o <<= 1) m = max(m, __shfl_xor_sync(FULL, m, o));
        if (ex[L][g] != kFxExZero) in = in && !(m - ex[L][g] > kFxSpread && ((same >> (2 * L + g)) & 1u));
      }
#pragma unroll
    for (int q = 0; q < (NB == 2 ? 2 : 1); ++q) {
      int m = open ? most[q] : kFxExZero;
#pragma unroll
      for (int o = 1; o < S; o <<= 1) m = max(m, __shfl_xor_sync(FULL, m, o));
      in = in && (most[q] == kFxExZero || m - most[q] <= kFxSpread);
    }
    unsigned take = __ballot_sync(FULL, in);
    if (S == 8) take = take & take >> 8 & take >> 16 & take >> 24 & 0xffu;  // all lines of a pair
    if (take == 0u) {  // every pair left is weak in some line: the first one alone
      const unsigned left = __ballot_sync(FULL, open);
      take = left & -left;
    }
    if (open && (take >> slot) & 1u) {
      open = false;
      if (lane == slot) cls[b.pair0 + slot] = (uint8_t)c;
    }
  }
}

// Row blocks whose pairs have several classes (list: their indices): the elements to the new blocks' order, in place,
// one block of threads each; shared memory: the row block's elements (nb = 2: 32 pairs of 512 bytes, nb = 4: 8 of 8 KB)
constexpr int kFxSplitBytes = 64 << 10;
template <int NB>
__global__ void __launch_bounds__(256) k_fx_split(const int* __restrict__ list, const RowBlock* __restrict__ rbs,
                                                  const uint8_t* __restrict__ cls, double2* __restrict__ P) {
  constexpr int NE = 2 * NB * NB * NB * NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int off[32], cnt[32];  // of a slot's class: first pair's element in the row block; pairs
  double2* const buf = (double2*)smem_raw;
  const RowBlock b = rbs[list[blockIdx.x]];
  const int n = __popc(b.mask);
  double2* const p = P + (size_t)b.pair0 * NE;
  for (int t = threadIdx.x; t < n * NE; t += blockDim.x) buf[t] = p[t];
  if (threadIdx.x < n) {
    const int c = cls[b.pair0 + threadIdx.x];
    int below = 0, same = 0, before = 0;
    for (int i = 0; i < n; ++i) {
      const int ci = cls[b.pair0 + i];
      below += ci < c;
      same += ci == c;
      before += ci == c && i < (int)threadIdx.x;
    }
    off[threadIdx.x] = below * NE + before;
    cnt[threadIdx.x] = same;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < n * NE; t += blockDim.x) {
    const int s = t % n, e = t / n;
    p[off[s] + e * cnt[s]] = buf[t];
  }
}

// FP64 elements to fixed point in place, one warp per row block; ex: [row block][line][group]; rbz: the row blocks without
// reverse terms of pairs that are zero throughout (their sums are zero, not weak)
template <int NB>
__global__ void __launch_bounds__(128) k_fx_quantise(long long nrb, const RowBlock* __restrict__ rbs,
                                                     unsigned char* __restrict__ P, int16_t* __restrict__ ex,
                                                     RowBlock* __restrict__ rbz) {
  constexpr int NB2 = NB * NB, NL = 2 * NB2;
  const long long r = blockIdx.x * 4LL + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= nrb) return;
  const RowBlock b = rbs[r];
  const int n = __popc(b.mask), m = NB2 * n;
  double2* p = (double2*)P + (size_t)b.pair0 * 2 * NB2 * NB2;
  unsigned nonzero = 0;  // by slot
  for (int L = 0; L < NL; ++L, p += m) {
    double mx[2] = {0.0, 0.0};
    for (int t = lane; t < m; t += 32) {
      const int e = t / n;
      const int g = (e / NB == e % NB) ? 0 : 1;
      const double v = fmax(fabs(p[t].x), fabs(p[t].y));
      if (v > 0.0) nonzero |= 1u << (t - e * n);
      if (g) mx[1] = fmax(mx[1], v);
      else mx[0] = fmax(mx[0], v);
    }
    int E[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      int e = kFxExZero;
      if (mx[g] > 0.0) e = fx_expo(mx[g]);
      E[g] = __reduce_max_sync(0xffffffffu, e);
    }
    if (lane < 2) ex[(r * NL + L) * 2 + lane] = (int16_t)(lane ? E[1] : E[0]);
    for (int t = lane; t < m; t += 32) {
      const int e = t / n;
      const int g = (e / NB == e % NB) ? 0 : 1;
      const int s = E[g] == kFxExZero ? 0 : kFxPBits - E[g];
      const int2 x = fx_digits(p[t].x, s), y = fx_digits(p[t].y, s);
      reinterpret_cast<int4*>(p)[t] = make_int4(x.x, x.y, y.x, y.y);
    }
  }
  nonzero = __reduce_or_sync(0xffffffffu, nonzero);
  const int slot = __popc(b.mask & ((1u << lane) - 1u));
  const unsigned keep = __ballot_sync(0xffffffffu, (b.mask >> lane) & (nonzero >> slot) & 1u);
  if (lane == 0) rbz[r] = {b.row, b.mask, b.revmask & keep, b.pair0};
}

// How far a column's elements lie below the item's largest where the coordinates are alike: st[item][matrix][column], in bits,
// from the lines of the diagonal coordinates (the off-diagonal ones are mostly small). kFxNone: no element at all. One warp per item.
constexpr int kFxNone = 127;
template <int NB>
__global__ void __launch_bounds__(128) k_fx_static(const WorkItem* __restrict__ items, int nitems, const RowBlock* __restrict__ rbz,
                                                   const int4* __restrict__ P, const int16_t* __restrict__ ex,
                                                   int8_t* __restrict__ st) {
  constexpr int NB2 = NB * NB, NB4 = NB2 * NB2, W = 128 / NB2, NL = 2 * NB2;
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, qg = lane / W, sl = lane % W;
  if (item >= nitems) return;
  const WorkItem w = items[item];
  for (int m = 0; m < 2; ++m) {
    int own = kFxExZero, all = kFxExZero, any = kFxExZero;  // the column's and the item's largest; the column's of every line
    for (int rb = w.rb0; rb < w.rb1; ++rb) {
      const RowBlock b = rbz[rb];
      const int n = __popc(b.mask), slot = __popc(b.mask & ((1u << sl) - 1u));
      for (int a = 0; a < NB2; ++a) {
        const bool diag = a / NB == a % NB;
        const int16_t* x = ex + ((size_t)rb * NL + m * NB2 + a) * 2;
        if (diag) all = max(all, max((int)x[0], (int)x[1]));
        if (!((b.revmask >> sl) & 1u)) continue;
        for (int i = 0; i < 4; ++i) {
          const int e = 4 * qg + i;
          const int4 v = P[(size_t)b.pair0 * 2 * NB4 + ((size_t)(m * NB2 + a) * NB2 + e) * n + slot];
          const long long p = (long long)v.x * (1LL << kFxBase) + v.y, q = (long long)v.z * (1LL << kFxBase) + v.w;
          const unsigned long long u = (unsigned long long)(p < 0 ? -p : p) | (unsigned long long)(q < 0 ? -q : q);
          if (u == 0ull) continue;
          const int t = 64 - __clzll((long long)u) + x[e / NB == e % NB ? 0 : 1] - kFxPBits;
          any = max(any, t);
          if (diag) own = max(own, t);
        }
      }
    }
#pragma unroll
    for (int o = W; o < 32; o <<= 1) {
      own = max(own, __shfl_xor_sync(0xffffffffu, own, o));
      any = max(any, __shfl_xor_sync(0xffffffffu, any, o));
    }
    if (qg) continue;
    st[((size_t)item * 2 + m) * W + sl] =
        (int8_t)(any == kFxExZero ? kFxNone : own == kFxExZero ? kFxNone - 1 : min(max(all - own, 0), kFxNone - 1));
  }
}

// bytes between the (line, re | im) rows of a chunk's forward sums: 32 lanes of 16 bytes and 64 more, so that the
// 32 8-byte reads of a step fall on all banks twice
constexpr int kFxFwdStride = 32 * 16 + 64;

// Shared memory of a warp: a ring of two chunks of two lines; the row digits and the forward exponents -- of
// every row block of the item for nb = 2 (lane r makes row block r's when the item starts), of the one at work
// for nb = 4, whose row blocks are 4 times the work and digits; then zeros.
template <int NB>
struct FxSmem {
  static constexpr int NB2 = NB * NB, G = NB2 / 4, W = 32 / G;
  static constexpr bool kItemDigits = NB == 2;
  static constexpr int stage_bytes = 2 * NB2 * W * 16;
  static constexpr int row_bytes = NB2 * 16;  // a row block's digits: int4 (diagonal h, l, off-diagonal h, l) per line
  static constexpr int dig = 2 * stage_bytes;
  static constexpr int zero = dig + (kItemDigits ? kMaxRowBlocksPerItem : 1) * row_bytes;
  static constexpr int exps = zero + row_bytes;
  static constexpr int NF = NB == 2 ? 1 : 2;  // flushes of forward sums per row block
  static constexpr int top = exps + (kItemDigits ? kMaxRowBlocksPerItem * NB2 * 4 : 0);  // their largest units: int per flush
  static constexpr int fwd = top + kMaxRowBlocksPerItem * NF * 4;                        // forward sums of a chunk
  static constexpr int bars = fwd + 4 * kFxFwdStride;
  static constexpr int warp_bytes = (bars + 16 + 127) / 128 * 128;
  static constexpr size_t cta_bytes = 4 * (size_t)warp_bytes;
};

// a and b summed over the lane pairs that differ in `bit`: the lane with the bit clear gets a's sum
__device__ __forceinline__ long long fx_merge(long long a, long long b, int bit, int lane) {
  const bool up = lane & bit;
  const long long keep = up ? b : a, send = up ? a : b;
  return keep + __shfl_xor_sync(0xffffffffu, send, bit);
}

// FP64 contraction of one work item from the decoded elements (non-finite states), straight from global
// memory: the sums of both parts of the state, with FP64 atomics per pair
template <int NB>
__device__ __noinline__ void fx_item_f64(const WorkItem w, const RowBlock* rbs, const int4* P, const int16_t* ex,
                                         const double* rs0, size_t half, bool anti, double* acc, int nk, int lane) {
  constexpr int NB2 = NB * NB, NB4 = NB2 * NB2, W = 128 / NB2, NL = 2 * NB2;
  const int qg = lane / W, sl = lane % W, col = w.J * W + sl;
  if (col >= nk) return;
  for (int part = 0; part < (anti ? 2 : 1); ++part) {
    const double* rs = rs0 + (part ? half : 0);
    const double* rc = rs + (size_t)col * 2 * NB2;
    for (int rb = w.rb0; rb < w.rb1; ++rb) {
      const RowBlock b = rbs[rb];
      if (!((b.mask >> sl) & 1u)) continue;
      const bool rev = (b.revmask >> sl) & 1u;
      const int n = __popc(b.mask), slot = __popc(b.mask & ((1u << sl) - 1u));
      const double* rr = rs + (size_t)b.row * 2 * NB2;
      for (int L = 0; L < NL; ++L) {
        const int m = L / NB2, a = L % NB2;
        const double kr = m ? rr[a] : rr[NB2 + a];  // r_k[j] or s_k[a]
        double fx = 0.0, fy = 0.0;
        for (int i = 0; i < 4; ++i) {
          const int e = 4 * qg + i;
          const int g = (e / NB == e % NB) ? 0 : 1;
          const int4 v = P[(size_t)b.pair0 * 2 * NB4 + ((size_t)L * NB2 + e) * n + slot];
          const int x = ex[((size_t)rb * NL + L) * 2 + g];
          const double px = fx_decode(v.x, v.y, x), py = fx_decode(v.z, v.w, x);
          const double c = m ? rc[NB2 + e] : rc[e];
          fx = fma(px, c, fx);
          fy = fma(py, c, fy);
          if (rev) {  // conj(p) times the row's coordinate, to the other sum of the column
            const double vx = px * kr, vy = -py * kr;
            double* d = acc + (size_t)col * 4 * NB2 + (m ? 0 : 2 * NB2) + 2 * e;
            atomicAdd(d, part ? -vy : vx);
            atomicAdd(d + 1, part ? vx : vy);
          }
        }
        double* d = acc + (size_t)b.row * 4 * NB2 + 2 * L;
        atomicAdd(d, part ? -fy : fx);
        atomicAdd(d + 1, part ? fx : fy);
      }
    }
  }
}

// The same for listed sums of one part (x i: imag), in pieces that a warp has in flight at once: line L of row block rb, and
// row block rb's share of the reverse sums of the columns in `cols`
template <int NB>
__device__ __noinline__ void fx_row_f64(const int rb, const int J, const int L, const RowBlock* rbs, const int4* P, const int16_t* ex,
                                        const double* rs, bool imag, double* acc, int nk, int lane) {
  constexpr int NB2 = NB * NB, NB4 = NB2 * NB2, W = 128 / NB2, NL = 2 * NB2;
  const int qg = lane / W, sl = lane % W, col = J * W + sl;
  const RowBlock b = rbs[rb];
  const int n = __popc(b.mask), slot = __popc(b.mask & ((1u << sl) - 1u));
  double x = 0.0, y = 0.0;
  if (((b.mask >> sl) & 1u) && col < nk) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = 4 * qg + i;
      const int4 v = P[(size_t)b.pair0 * 2 * NB4 + ((size_t)L * NB2 + e) * n + slot];
      const int xe = ex[((size_t)rb * NL + L) * 2 + ((e / NB == e % NB) ? 0 : 1)];
      const double c = rs[(size_t)col * 2 * NB2 + (L < NB2 ? 0 : NB2) + e];
      x = fma(fx_decode(v.x, v.y, xe), c, x);
      y = fma(fx_decode(v.z, v.w, xe), c, y);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
  }
  if (lane == 0) {
    double* d = acc + (size_t)b.row * 4 * NB2 + 2 * L;
    atomicAdd(d, imag ? -y : x);
    atomicAdd(d + 1, imag ? x : y);
  }
}
template <int NB>
__device__ __noinline__ void fx_column_f64(const int rb, const int J, const int m, const unsigned cols, const RowBlock* rbs,
                                           const int4* P, const int16_t* ex, const double* rs, bool imag, double* acc, int nk,
                                           int lane) {
  constexpr int NB2 = NB * NB, NB4 = NB2 * NB2, W = 128 / NB2, NL = 2 * NB2;
  const int qg = lane / W, sl = lane % W, col = J * W + sl;
  const RowBlock b = rbs[rb];
  if (!((cols & b.revmask) >> sl & 1u) || col >= nk) return;
  const int n = __popc(b.mask), slot = __popc(b.mask & ((1u << sl) - 1u));
  double x[4] = {0.0, 0.0, 0.0, 0.0}, y[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int a = 0; a < NB2; ++a) {
    const int L = m * NB2 + a;
    const double kr = rs[(size_t)b.row * 2 * NB2 + (m ? a : NB2 + a)];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = 4 * qg + i;
      const int4 v = P[(size_t)b.pair0 * 2 * NB4 + ((size_t)L * NB2 + e) * n + slot];
      const int xe = ex[((size_t)rb * NL + L) * 2 + ((e / NB == e % NB) ? 0 : 1)];
      x[i] = fma(fx_decode(v.x, v.y, xe), kr, x[i]);
      y[i] = fma(-fx_decode(v.z, v.w, xe), kr, y[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    double* d = acc + (size_t)col * 4 * NB2 + (m ? 0 : 2 * NB2) + 2 * (4 * qg + i);
    atomicAdd(d, imag ? -y[i] : x[i]);
    atomicAdd(d + 1, imag ? x[i] : y[i]);
  }
}

// One warp per work item and matrix (Q1 or Q2): lane (qg, sl) owns column W J + sl and the quarter qg of
// every line. With both matrices in one warp the reverse sums and the column's digits took 168 registers and
// left 12 warps per SM, too few to cover the multiply-adds' latency; one matrix fits 4 CTAs. Chunks of
// two lines (4 KB) stream through a per-warp ring of two bulk copies. The forward sums (line, re | im,
// group) of a chunk are added over the warp through shared memory, 8 lanes' entries by each lane, and the two
// bits of lanes that remain by exchanges that halve the values, so that lane (group, re | im, line) ends with its
// total. (Exchanges alone, 8 instructions per value and level, took a sixth of the kernel's instructions.)
template <int NB, bool IMAG>
__device__ __forceinline__ void fx_item(unsigned char* const wbase, const int item, const WorkItem w, const int m, const RowBlock* __restrict__ rbs,
                                        const int4* __restrict__ P, const int16_t* __restrict__ ex, const int8_t* __restrict__ st,
                                        const double* __restrict__ rs, double* __restrict__ acc, int nk, int lane,
                                        unsigned int* __restrict__ flag, FxWeak* __restrict__ weak, unsigned nweak,
                                        unsigned int* __restrict__ errflag) {
  typedef FxSmem<NB> S;
  constexpr int NB2 = S::NB2, NB4 = NB2 * NB2, W = S::W;
  constexpr int LF = NB == 2 ? 4 : 8;  // lines per forward flush
  constexpr int NF = NB2 / LF;         // flushes per row block
  constexpr int CPR = NB2 / 2;         // chunks (two lines) per row block
  constexpr int RB = fx_row_bits(NB);
  constexpr unsigned FULL = 0xffffffffu;
  const int qg = lane / W, sl = lane % W;
  const uint32_t sbase = smem_u32(wbase);
  uint64_t* const bar = (uint64_t*)(wbase + S::bars);
  const int nrb = w.rb1 - w.rb0;  // <= kMaxRowBlocksPerItem = 32
  RowBlock mine;                  // lane r: the item's row block r
  mine.row = 0;
  mine.mask = 0;
  mine.revmask = 0;
  mine.pair0 = 0;
  if (lane < nrb) mine = rbs[w.rb0 + lane];
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  // the column's coordinates: r for Q1's forward sums, s for Q2's; the rows': s for Q1, r for Q2
  const int col = w.J * W + sl;
  const int co = m ? NB2 : 0, ro = m ? 0 : NB2;
  double cv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int b = NB == 2 ? i : 4 * qg + ((i + qg) & 3);
    cv[i] = col < nk ? rs[(size_t)col * 2 * NB2 + co + b] : 0.0;
  }
  __syncwarp();
  const uint64_t pol = policy_evict_first();
  // address of a row block's lines of this matrix and bytes of a chunk of it (0 past the item's end)
  const char* const mysrc = (const char*)(P + (size_t)mine.pair0 * 2 * NB4 + (size_t)m * NB4 * __popc(mine.mask));
  const int mylen = 2 * NB2 * 16 * __popc(mine.mask);
  auto copy = [&](const char* src, int len, int q) {  // chunk q of a row block into stage q % 2
    if (lane == 0 && len > 0) {
      mbar_arrive_expect_tx(&bar[q & 1], len);
      bulk_g2s(wbase + (q & 1) * S::stage_bytes, src + (size_t)q * len, len, &bar[q & 1], pol);
    }
  };
  const char* src = (const char*)__shfl_sync(FULL, (unsigned long long)mysrc, 0);
  int len = __shfl_sync(FULL, mylen, 0);
  copy(src, len, 0);
  copy(src, len, 1);

  // the largest row coordinate times its line's scale, per group: the reverse sums' exponents
  int eS0 = -30000, eS1 = -30000;
  const double* const rr = rs + (size_t)mine.row * 2 * NB2 + ro;
  const short2* const xr = (const short2*)ex + ((size_t)(w.rb0 + (lane < nrb ? lane : 0)) * 2 + m) * NB2;
  int xm[NF][2];  // the largest exponents of lane r's row block's flushes
#pragma unroll
  for (int f = 0; f < NF; ++f) xm[f][0] = xm[f][1] = kFxExZero;
  int em = -900;
  if (lane < nrb) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
#pragma unroll 4
      for (int a = f * LF; a < (f + 1) * LF; ++a) {
        const int e = fx_expo(rr[a]);
        const short2 x = xr[a];
        eS0 = max(eS0, e + x.x);
        eS1 = max(eS1, e + x.y);
        em = max(em, e);
        xm[f][0] = max(xm[f][0], x.x);
        xm[f][1] = max(xm[f][1], x.y);
      }
    }
  }
  eS0 = __reduce_max_sync(FULL, eS0);
  eS1 = __reduce_max_sync(FULL, eS1);
  bool row_zero = !__any_sync(FULL, em > -900);  // perhaps: every row coordinate is zero
  if (row_zero) {
    long long u = 0;
    for (int a = 0; a < NB2; ++a) u |= lane < nrb ? __double_as_longlong(rr[a]) << 1 : 0;
    row_zero = !__any_sync(FULL, u != 0);
  }
  const int lg = lane & 1, lri = (lane >> 1) & 1, ll = (lane >> 2) % LF;
  int2 cd[4];  // the column's digits
  int eR;      // their exponent, of this lane's group
  {
    int e[2] = {-900, -900};
#pragma unroll
    for (int i = 0; i < 4; ++i) e[fx_group<NB>(i)] = max(e[fx_group<NB>(i)], fx_expo(cv[i]));
    e[0] = __reduce_max_sync(FULL, e[0]);
    e[1] = __reduce_max_sync(FULL, e[1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) cd[i] = fx_digits(cv[i], kFxCBits - e[fx_group<NB>(i)]);
    eR = (lg ? e[1] : e[0]) + 2 * kFxBase - kFxPBits - kFxCBits;  // of the forward sums' unit
    // the exponent field (1022 + e of a double below 2^e) that one of a flush's sums has to exceed
    const bool zero = max(e[0], e[1]) == -900 && fx_all_zero(cv[0], cv[1], cv[2], cv[3]);  // no sum is weak
    if (lane < nrb) {
#pragma unroll
      for (int f = 0; f < NF; ++f)
        ((int*)(wbase + S::top))[lane * NF + f] = zero ? -1 : max(xm[f][0] + e[0], xm[f][1] + e[1]) + 1022 - kFxWeakRow;
    }
  }
  short exn[NF];   // nb = 4: lane (group, re | im, line of a flush): its lines' exponents and row coordinates,
  double rown[NF]; // one row block ahead
  auto fetch = [&](int rbi) {
    const int row = __shfl_sync(FULL, mine.row, rbi);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      exn[f] = ex[(((size_t)(w.rb0 + rbi) * 2 + m) * NB2 + f * LF + ll) * 2 + lg];
      rown[f] = rs[(size_t)row * 2 * NB2 + ro + f * LF + ll];
    }
  };
  if constexpr (S::kItemDigits) {  // lanes (row block of 4, line, group)
    const int a = (lane >> 1) & 3;
    for (int r0 = 0; r0 < nrb; r0 += 4) {
      const int r = r0 + (lane >> 3), row = __shfl_sync(FULL, mine.row, r & 31);
      if (r < nrb) {
        const short x = ex[(((size_t)(w.rb0 + r) * 2 + m) * NB2 + a) * 2 + lg];
        ((int2*)(wbase + S::dig))[r * 8 + (lane & 7)] =
            fx_digits(rs[(size_t)row * 2 * NB2 + ro + a], RB + x - (lg ? eS1 : eS0));
        ((short*)(wbase + S::exps))[r * 8 + (lane & 7)] = x;
      }
    }
  } else if (nrb > 0) {
    fetch(0);
  }
  for (int i = lane; i < NB2; i += 32) ((int4*)(wbase + S::zero))[i] = make_int4(0, 0, 0, 0);
  __syncwarp();

  // the column's reverse sums [step][re | im]: B0 2^32 + Br, with the low products of four lines at work in B1
  long long B0[4][2], B1[4][2];
  unsigned Br[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) B0[i][0] = B0[i][1] = Br[i][0] = Br[i][1] = 0;
  bool any_rev = false;
  unsigned weak_rows = 0;  // flushes whose sums are too small for their unit (nb = 4: items hold at most 16 row blocks)
  int cfail = -1;
#pragma unroll 1
  for (int rbi = 0; rbi < nrb; ++rbi) {
    const int brow = __shfl_sync(FULL, mine.row, rbi);
    const unsigned bmask = __shfl_sync(FULL, mine.mask, rbi);
    const unsigned brev = __shfl_sync(FULL, mine.revmask, rbi);
    const bool active = (bmask >> sl) & 1u, rev = (brev >> sl) & 1u;
    any_rev |= rev;
    const char* nsrc = (const char*)__shfl_sync(FULL, (unsigned long long)mysrc, (rbi + 1) & 31);
    const int nlen = __shfl_sync(FULL, rbi + 1 < nrb ? mylen : 0, (rbi + 1) & 31);
    short exv[NF];
    if constexpr (S::kItemDigits) {
      exv[0] = ((const short*)(wbase + S::exps))[(rbi * NB2 + ll) * 2 + lg];
    } else {
      __syncwarp();  // the previous row block's digits have been read
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        exv[f] = exn[f];
        const int2 d = fx_digits(rown[f], RB + exv[f] - (lg ? eS1 : eS0));
        if (lri == 0) ((int2*)(wbase + S::dig))[(f * LF + ll) * 2 + lg] = d;
      }
      if (rbi + 1 < nrb) fetch(rbi + 1);
      __syncwarp();
    }
    // lanes without a reverse term read zero digits, lanes without a pair zero elements
    const uint32_t dg = sbase + (rev ? S::dig + (S::kItemDigits ? rbi * S::row_bytes : 0) : S::zero);
    const uint32_t ns = active ? __popc(bmask) * 16 : 0;
    const uint32_t s0 = active ? sbase + __popc(bmask & ((1u << sl) - 1u)) * 16 : sbase + S::zero;
    const uint32_t s1 = active ? s0 + S::stage_bytes : s0;
    // forward sums: lane reads value lane % 8 of lanes 4 k + lane / 8
    const uint32_t fsum = sbase + S::fwd + ((lane >> 1) & 3) * kFxFwdStride + (lane >> 3) * 16 + (lane & 1) * 8;
    uint32_t eo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) eo[i] = (NB == 2 ? i : 4 * qg + ((i + qg) & 3)) * ns;

    // one line: forward sums of the two groups (to the chunk's buffer), reverse sums
    auto line = [&](uint32_t sp, int L) {
      const int4 rd = fx_lds(dg + L * 16);  // the row coordinate's digits for both groups
      long long A0[2][2], A1[2][2];         // [group][re | im]; A1 starts at half of A0's unit
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        constexpr int gr[4] = {fx_group<NB>(0), fx_group<NB>(1), fx_group<NB>(2), fx_group<NB>(3)};
        const int g = gr[i];
        const int4 p = fx_lds(sp + eo[i]);
        if (i < 2) {  // the first of its group
          fx_mul(A0[g][0], A1[g][0], p.x, p.y, cd[i], 1LL << (kFxBase - 1));
          fx_mul(A0[g][1], A1[g][1], p.z, p.w, cd[i], 1LL << (kFxBase - 1));
        } else {
          fx_mad(A0[g][0], A1[g][0], p.x, p.y, cd[i]);
          fx_mad(A0[g][1], A1[g][1], p.z, p.w, cd[i]);
        }
        const int2 d = g ? make_int2(rd.z, rd.w) : make_int2(rd.x, rd.y);
        fx_mad(B0[i][0], B1[i][0], p.x, p.y, d);
        fx_mad(B0[i][1], B1[i][1], p.z, p.w, d);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const long long t0 = A0[0][x] + (A1[0][x] >> kFxBase), t1 = A0[1][x] + (A1[1][x] >> kFxBase);
        asm volatile("st.shared.v2.s64 [%0], {%1, %2};" ::"r"(sbase + S::fwd + lane * 16 + ((L & 1) * 2 + x) * kFxFwdStride),
                     "l"(t0), "l"(t1)
                     : "memory");
      }
    };
    // the two lines of chunk q: lane (part of 4, line, re | im, group) returns its value's sum over 8 lanes;
    // false when the copy did not arrive
    auto two = [&](int q, long long& v) -> bool {
      const int c = rbi * CPR + q;
      if (!__all_sync(FULL, mbar_wait_bounded(&bar[q & 1], (unsigned)(c >> 1) & 1u, errflag))) {
        cfail = c;
        return false;
      }
      const uint32_t sp = (q & 1) ? s1 : s0;
      line(sp, 2 * q);
      line(sp + NB2 * ns, 2 * q + 1);
      // the stage is free once every lane has read it: order those reads before the next bulk copy into it
      fence_proxy_async();
      __syncwarp();
      if (q + 2 < CPR) copy(src, len, q + 2);
      else copy(nsrc, nlen, q + 2 - CPR);
      v = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        long long o;
        asm volatile("ld.shared.s64 %0, [%1];" : "=l"(o) : "r"(fsum + k * 64));
        v += o;
      }
      __syncwarp();
      return true;
    };
    auto four = [&](int q, long long& v) -> bool {  // two chunks from q on, merged over the parts' first bit
      long long a, b;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        B1[i][0] = Br[i][0];
        B1[i][1] = Br[i][1];
      }
      if (!two(q, a) || !two(q + 1, b)) return false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        Br[i][0] = fx_fold(B0[i][0], B1[i][0]);
        Br[i][1] = fx_fold(B0[i][1], B1[i][1]);
      }
      v = fx_merge(a, b, 8, lane);
      return true;
    };
    bool ok = true;
#pragma unroll 1
    for (int f = 0; f < NF; ++f) {
      long long v, u;
      if (!(ok = four(f * LF / 2, v))) break;
      if constexpr (LF == 8) {
        if (!(ok = four(f * LF / 2 + 2, u))) break;
        v = fx_merge(v, u, 16, lane);
      } else {
        u = __shfl_xor_sync(FULL, v, 16);
        v += u;
      }
      // the totals of the flush's lines to the row's sums (x i in the anti-Hermitian pass)
      double d = fx_scale((double)v, (NF == 1 || f == 0 ? exv[0] : exv[NF - 1]) + eR);
      // (no branch here: 2 % on 2.5M pairs)
      const bool add = __any_sync(FULL, ((__double2hiint(d) >> 20) & 0x7ff) > ((const int*)(wbase + S::top))[rbi * NF + f]);
      if (!add) weak_rows |= 1u << (rbi * NF + f);
      d += __shfl_xor_sync(FULL, d, 1);
      if (add && lg == 0 && lane < 4 * LF) {
        double* dst = acc + (size_t)brow * 4 * NB2 + 2 * (m * NB2 + f * LF + ll);
        if (IMAG) atomicAdd(dst + (lri ^ 1), lri ? -d : d);
        else atomicAdd(dst + lri, d);
      }
    }
    if (!ok) break;
    src = nsrc;
    len = nlen;
  }
  if (cfail >= 0) {  // drain the copies still in flight (bounded), then leave
    if (lane == 0) {
      const int clast = (cfail + 2 < CPR * nrb ? cfail + 2 : CPR * nrb) - 1;
      for (int i = cfail; i <= clast; ++i)  mbar_wait_bounded(&bar[i & 1], (unsigned)(i >> 1) & 1u, nullptr, 1u << 16);
    }
    __syncwarp();
    return;
  }
  // weak sums are left to the gated launch; in that launch they are summed at once
  auto list = [&](int x, int z, int kind) {
    if (lane == 0) {
      const unsigned i = atomicAdd(flag, DMD_HFLAG_WEAK) / DMD_HFLAG_WEAK;
      if (i < nweak) weak[i] = make_int4(x, w.J, z, m | kind);
      else atomicOr(errflag, DMD_DEVERR_LIST);
    }
  };
  for (unsigned u = weak_rows; u; u &= u - 1) {
    const int q = __ffs(u) - 1, rb = w.rb0 + q / NF, f = q % NF;
    if (IMAG) {
      for (int l = 0; l < LF; ++l) fx_row_f64<NB>(rb, w.J, m * NB2 + f * LF + l, rbs, P, ex, rs, true, acc, nk, lane);
    } else {
      list(rb, f, 0);
    }
  }
  // the column block's sums (Y' from Q1, X' from Q2) through the now free first stage, so that a warp's
  // reductions touch consecutive doubles (one lane per column would touch 32 sectors each)
  if (__any_sync(FULL, any_rev)) {
    double2* const out = (double2*)wbase + (size_t)sl * NB2;
    int got = 0;  // as for the forward sums, over the column's elements
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = NB == 2 ? i : 4 * qg + ((i + qg) & 3);
      const int e = (fx_group<NB>(i) ? eS1 : eS0) + 2 * kFxBase - kFxPBits - RB;  // of B0's unit
      double v[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        // B0 2^32 + Br to 64 bits: below 2^46 with 16 bits of Br, else rounded to B0's unit
        const int h = (int)(B0[i][x] >> 32);
        const bool low = (unsigned)(h ^ (h >> 31)) < (1u << 14);
        const long long q = low ? (long long)((unsigned long long)B0[i][x] << 16 | Br[i][x] >> 16) : B0[i][x] + (Br[i][x] >> 31);
        v[x] = fx_scale((double)q, low ? e - 16 : e);
        got = max(got, (__double2hiint(v[x]) >> 20) & 0x7ff);
      }
      // conj(p): the imaginary sum has the opposite sign
      out[b] = IMAG ? mk2(v[1], v[0]) : mk2(v[0], -v[1]);
    }
#pragma unroll
    for (int o = W; o < 32; o <<= 1) got = max(got, __shfl_xor_sync(FULL, got, o));
    const int below = max(eS0, eS1) + 1022 - got;
    bool small = any_rev && !row_zero && below >= fx_weak_column(NB);
    unsigned cols = __ballot_sync(FULL, small);
    if (cols) {
      const int s = st[((size_t)item * 2 + m) * W + sl];
      small = small && s != kFxNone && below >= min(max(s + kFxWeakMore, fx_weak_column(NB)), fx_weak_most(NB));
      cols = __ballot_sync(FULL, small);
    }
    if (cols) {
      if (small) {
#pragma unroll
        for (int i = 0; i < 4; ++i) out[4 * qg + i] = mk2(0.0, 0.0);
      }
      const int z = (int)(W == 32 ? cols : cols & ((1u << (W & 31)) - 1u));
      if (IMAG) {
        for (int rb = w.rb0; rb < w.rb1; ++rb) fx_column_f64<NB>(rb, w.J, m, (unsigned)z, rbs, P, ex, rs, true, acc, nk, lane);
      } else {
        list(item, z, 2);
      }
    }
    __syncwarp();
    constexpr int R = 2 * NB2;  // reals per column: consecutive lanes take consecutive reals of one or more columns
    double* const dst = acc + (size_t)w.J * W * 4 * NB2 + (m ? 0 : R);
#pragma unroll
    for (int i = 0; i < W * R / 32; ++i) {
      const int idx = i * 32 + lane, cc = idx / R;
      if (w.J * W + cc < nk) atomicAdd(dst + (size_t)cc * 4 * NB2 + idx % R, ((const double*)wbase)[idx]);
    }
  }
}

// IMAG: the gated launch behind every evaluation's first one, for the anti-Hermitian part (sums times i), the listed sums and
// non-finite states. It costs 2.5 us where there is nothing to do; in the same launch, as a second pass of the warp or
// as blocks that return at once, it cost the pass that always runs 3 to 50 % from 400k pairs on. rbz: the row blocks without the
// reverse terms of zero pairs; rbs: with them (a non-finite coordinate times zero is NaN).
template <int NB, int MINB, bool IMAG>
__global__ void __launch_bounds__(128, MINB) k_pairs_fx(const WorkItem* __restrict__ items, int nitems,
                                                        const RowBlock* __restrict__ rbs, const RowBlock* __restrict__ rbz,
                                                        const int4* __restrict__ P, const int16_t* __restrict__ ex,
                                                        const int8_t* __restrict__ st, const double* __restrict__ rs, size_t half,
                                                        double* __restrict__ acc,
                                                        int nk, unsigned int* flag, FxWeak* weak, unsigned nweak,
                                                        unsigned int* __restrict__ errflag) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const unsigned fl = *flag;
  if (IMAG ? fl == 0u : (fl & DMD_HFLAG_NONFINITE) != 0u) return;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int task = blockIdx.x * 4 + wib, item = task >> 1, m = task & 1;
  if (IMAG && !(fl & DMD_HFLAG_NONFINITE)) {
    const unsigned n = min(fl / DMD_HFLAG_WEAK, nweak);
    constexpr int NB2 = NB * NB, LF = NB == 2 ? 4 : 8, PARTS = NB == 2 ? 16 : 8;  // a warp per line or row block of a listed sum
    for (unsigned long long i = task; i < (unsigned long long)n * PARTS; i += gridDim.x * 4) {
      const FxWeak u = weak[i / PARTS];
      const int part = (int)(i % PARTS), mu = u.w & 1;
      if (u.w & 2) {
        const WorkItem w = items[u.x];
        for (int rb = w.rb0 + part; rb < w.rb1; rb += PARTS)
          fx_column_f64<NB>(rb, w.J, mu, (unsigned)u.z, rbs, P, ex, rs, false, acc, nk, lane);
        __syncwarp();
      } else if (part < LF) {
        fx_row_f64<NB>(u.x, u.y, mu * NB2 + u.z * LF + part, rbs, P, ex, rs, false, acc, nk, lane);
      }
    }
    if (!(fl & DMD_HFLAG_NONHERM)) return;
  }
  if (item >= nitems) return;
  const WorkItem w = items[item];
  if (IMAG && (fl & DMD_HFLAG_NONFINITE)) {
    if (m == 0) fx_item_f64<NB>(w, rbs, P, ex, rs, half, (fl & DMD_HFLAG_NONHERM) != 0u, acc, nk, lane);
    return;
  }
  fx_item<NB, IMAG>(smem_raw + (size_t)wib * FxSmem<NB>::warp_bytes, item, w, m, rbz, P, ex, st, rs + (IMAG ? half : 0), acc, nk, lane,
                    flag, weak, nweak, errflag);
}

}  // namespace dmd
