// Batched form of the k-pair contraction on the tensor cores (tcgen05), nb = 2 and nb = 4.
//
// With many states sharing P the contraction is a GEMM. Every stored pair (k1, k2) is kept twice, as
// directed operators (row <- column): (k1 <- k2) with A = Q1, B = Q2 and, when the pair carries the
// reverse term, (k2 <- k1) with A = conj(Q2), B = conj(Q1) (Q1, Q2: the Hermitian-coordinate
// operators of dmd_pairs_cb.cuh). Then for every row k
//   X'_k[a] = sum_c sum_j A_kc[a][j] r_c[j],      Y'_k[j] = sum_c sum_a B_kc[a][j] s_c[a]
// and no reverse sums remain. The batched form runs in the deviation form, where s = -r (or s = 0 in
// the linearized form), so both sums contract the same coordinates: Y'_k[j] = -sum B_kc[a][j] r_c[a].
// Rows (energy-rank positions) are grouped in tiles of TR = 64 / nb^2 (16 for nb = 2, 4 for nb = 4),
// columns in groups of CG = 32 / nb^2 (8, 2); a tile's operators over one column group form a dense
// block (zeros where a row and a column have no pair; rows of an energy window pair with nearly the
// same columns, so the blocks are nearly full). For a tile and up to 128 states one CTA computes
//   D[q][n] = sum_(c, j) R[q][(c, j)] * B[(c, j)][n],  n < 128: (r, a, re|im) of X', n >= 128: (r, j, re|im) of -Y'
// (M = 128 states, N = 256, K = CG columns x nb^2 = 32 per group) as tcgen05 MMAs accumulating in tensor
// memory over all of the tile's column groups, then writes each row's sums once (FP32, as the
// tensor memory holds them): no atomics.
// Operands are bf16 hi + lo splits (x = hi + lo, 16 significant bits); the product keeps
// hi*hi + hi*lo + lo*hi. Every operand row holds [hi (32) | lo (32)] = 128 bytes, so a tile is a
// 128-byte-swizzled K-major tile and the three products are MMAs over K slices paired through
// descriptor offsets (hi: +0, +32 B; lo: +64, +96 B). Operand blocks are laid out in HBM exactly as
// the MMA reads them (swizzle included), so two bulk copies fill a pipeline stage. Warp 0 (one lane)
// produces, warp 1 (one lane) issues MMAs, the other lanes of both warps park at __syncwarp (a lane
// polling an mbarrier would hold up the working lane of its warp), and all four warps write the sums
// through shared memory in 512-byte rows.
#pragma once
#include <cuda_bf16.h>

#include "dmd_common.cuh"
#include "dmd_kernels.cuh"
#include "dmd_pairs_cb.cuh"
#include "dmd_tc.cuh"
#include "dmd_tma.cuh"

namespace dmd {

struct TcTile {
  int32_t g0, g1;  // column groups [g0, g1)
  int64_t boff;    // index of the tile's first operator block
};

constexpr int TC_K = 32, TC_N = 128, TC_M = 128;
// rows per tile and columns per group for nb2 = nb^2 coordinates per k-point
__host__ __device__ constexpr int tc_tr(int nb2) { return 64 / nb2; }
__host__ __device__ constexpr int tc_cg(int nb2) { return 32 / nb2; }
constexpr int TC_PLANE = 8192;                     // bf16 per 128-row tile (128 rows x [hi 32 | lo 32])
constexpr int TC_BLOCK = 2 * TC_PLANE;             // bf16 per operator block: X rows, then Y rows (256)
constexpr int TC_ABLOCK = TC_PLANE;                // bf16 per coordinate block: R (128 states)
constexpr uint32_t TC_BLOCK_BYTES = 2 * TC_BLOCK;  // 32 KB
constexpr uint32_t TC_ABLOCK_BYTES = 2 * TC_ABLOCK;  // 16 KB
constexpr uint32_t TC_STAGE_BYTES = TC_ABLOCK_BYTES + TC_BLOCK_BYTES;
constexpr int TC_NST = 4;                          // pipeline stages of (coordinate block, operator block)
// dynamic shared memory of a CTA with nst stages (2 stages leave room for 2 CTAs per SM)
__host__ __device__ constexpr size_t tc_smem_bytes(int nst) { return (size_t)nst * TC_STAGE_BYTES + 1024 + 128; }
constexpr size_t TC_SMEM_BYTES = tc_smem_bytes(TC_NST);

// element (row, kk) of a tile: kk < 32 the hi part, kk + 32 the lo part of K index kk
__host__ __device__ __forceinline__ int tc_ci(int row, int kk) { return tc_sw128(row, kk); }

// r coordinates (FP32, [part][q][pos][2 NB2] as written by k_prep_herm, the first NB2 of each 2 NB2)
// -> coordinate blocks [part][group][mblock][128 x (hi 32 | lo 32)]; entries of padding states stay
// zero. Part 1 (anti-Hermitian) is packed only when *gate is set.
template <int NB>
__global__ void k_pack_tc(int nk, int nrhs, int ngroups, int nmb, const float* __restrict__ rs,
                          uint16_t* __restrict__ A, const unsigned int* __restrict__ gate) {
  constexpr int NB2 = NB * NB, CG = tc_cg(NB2);
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const int part = blockIdx.y;
  if (part == 1 && *gate == 0u) return;
  const size_t per = (size_t)nrhs * nk * NB2;
  if (idx >= per) return;
  const int e = (int)(idx % NB2), p = (int)((idx / NB2) % nk), q = (int)(idx / ((size_t)NB2 * nk));
  const float v = rs[(size_t)part * 2 * per + ((size_t)q * nk + p) * 2 * NB2 + e];
  const __nv_bfloat16 hi = __float2bfloat16_rn(v);
  const __nv_bfloat16 lo = __float2bfloat16_rn(__fsub_rn(v, __bfloat162float(hi)));
  const int g = p / CG, kk = (p % CG) * NB2 + e, mb = q / TC_M, m = q % TC_M;
  uint16_t* blk = A + (((size_t)part * ngroups + g) * nmb + mb) * TC_ABLOCK;
  blk[tc_ci(m, kk)] = __bfloat16_as_ushort(hi);
  blk[tc_ci(m, kk + 32)] = __bfloat16_as_ushort(lo);
}

// IMAG: the anti-Hermitian pass (sums times i, added); otherwise acc = sums (stored). acc is FP32,
// [state][position][X' (NB2) | Y' (NB2)], astride float2 per state. ysign: -1 (Y' = -D_Y, s = -r) or 0
// (linearized form, s = 0).
template <bool IMAG, int NST = TC_NST, int NB = 2>
__global__ void __launch_bounds__(128, 1) k_pairs_tc(const TcTile* __restrict__ tiles, int ntiles,
                                                     const uint16_t* __restrict__ B, const uint16_t* __restrict__ A,
                                                     int nmb, int nrhs, int nk, float2* __restrict__ acc,
                                                     size_t astride, float ysign,
                                                     const unsigned int* __restrict__ gate,
                                                     unsigned int* __restrict__ errflag) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (gate && *gate == 0u) return;
  // swizzled operand tiles start on 1024-byte boundaries (1 KB of slack is allocated)
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  // the CTAs of one tile (all state blocks) are adjacent, so its operator blocks are read from HBM once
  const int t = blockIdx.x / nmb, mb = blockIdx.x % nmb;
  if (t >= ntiles) return;
  const TcTile tile = tiles[t];
  const int nch = tile.g1 - tile.g0;
  uint64_t* full = (uint64_t*)(smem + NST * TC_STAGE_BYTES);
  uint64_t* empty = full + NST;
  uint64_t* done = empty + NST;
  uint32_t* tslot = (uint32_t*)(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tc_alloc(tslot, 256);  // D: X' in columns [0, 128), -Y' in [128, 256)
    tc_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  if (nch > 0) {
    if (warp == 0) {
      if (lane == 0) {  // producer: coordinate block + operator block per column group
        const uint64_t pol_a = policy_evict_last(), pol_b = policy_evict_first();
        int issued = 0;
        for (int i = 0; i < nch; ++i) {
          const int s = i % NST;
          if (i >= NST && !mbar_wait_bounded(&empty[s], (uint32_t)((i / NST - 1) & 1), errflag)) break;
          unsigned char* st = smem + (size_t)s * TC_STAGE_BYTES;
          mbar_arrive_expect_tx(&full[s], TC_STAGE_BYTES);
          bulk_g2s(st, A + ((size_t)(tile.g0 + i) * nmb + mb) * TC_ABLOCK, TC_ABLOCK_BYTES, &full[s], pol_a);
          bulk_g2s(st + TC_ABLOCK_BYTES, B + (size_t)(tile.boff + i) * TC_BLOCK, TC_BLOCK_BYTES, &full[s], pol_b);
          ++issued;
        }
        mbar_wait_bounded(done, 0, errflag);
        // no bulk copy into this CTA's shared memory outlives it (all landed unless a wait gave up)
        for (int j = issued > NST ? issued - NST : 0; j < issued; ++j)
          mbar_wait_bounded(&full[j % NST], (uint32_t)((j / NST) & 1), errflag);
      }
      __syncwarp();
    } else if (warp == 1) {
      if (lane == 0) {  // MMA issuer
        constexpr uint32_t idesc = tc_idesc_bf16(TC_M, 2 * TC_N);
        constexpr uint32_t SBO = 1024, LO = 64;  // bytes: 8-row atoms; hi -> lo slice of a row
        for (int i = 0; i < nch; ++i) {
          const int s = i % NST;
          if (!mbar_wait_bounded(&full[s], (uint32_t)((i / NST) & 1), errflag)) break;
          tc_fence_after();
          const uint32_t a0 = smem_u32(smem + (size_t)s * TC_STAGE_BYTES), b0 = a0 + TC_ABLOCK_BYTES;
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {  // K = 32 as two MMAs of K = 16 (32 bytes of the row apart)
            const uint32_t ko = ks * 32;
            const uint32_t accum = (i | ks) != 0;  // the tile's first MMA overwrites the accumulator
            tc_mma(tmem, tc_desc_sw128(a0 + ko, SBO), tc_desc_sw128(b0 + ko, SBO), idesc, accum);  // hi x hi
            tc_mma(tmem, tc_desc_sw128(a0 + LO + ko, SBO), tc_desc_sw128(b0 + ko, SBO), idesc, 1);  // lo x hi
            tc_mma(tmem, tc_desc_sw128(a0 + ko, SBO), tc_desc_sw128(b0 + LO + ko, SBO), idesc, 1);  // hi x lo
          }
          tc_commit(&empty[s]);  // the stage is free once these MMAs have read it
        }
        tc_commit(done);  // arrives when every MMA issued above has completed (also after a failure)
      }
      __syncwarp();
    }
    // all MMAs complete before TMEM is read (bounded; a timeout sets the flag)
    mbar_wait_bounded(done, 0, errflag);
  }
  tc_fence_after();
  // epilogue: TMEM lane 32 w + l holds state q = 128 mb + 32 w + l. 32 TMEM columns hold RPC rows of
  // the tile (4 for nb = 2, 1 for nb = 4) x NB2 elements x (re, im); per such chunk a thread writes its
  // state's RPC x 2 NB2 sums into shared memory (a row of 33 float2 per state), then the warp stores
  // each state's 256 contiguous bytes with one coalesced instruction.
  constexpr int NB2 = NB * NB, RPC = 16 / NB2, TR = tc_tr(NB2);
  float2* wsm = (float2*)smem + (size_t)warp * 32 * 33;
  const int qb = mb * TC_M + warp * 32;
  const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
  for (int rq = 0; rq < 4; ++rq) {
    float vx[32], vy[32];
    if (nch > 0) {
      tc_ld32(lane_addr + rq * 32, vx);
      tc_ld32(lane_addr + 128 + rq * 32, vy);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) vx[i] = vy[i] = 0.f;
    }
    float2* my = wsm + lane * 33;
#pragma unroll
    for (int rr = 0; rr < RPC; ++rr)
#pragma unroll
      for (int a = 0; a < NB2; ++a) {
        my[rr * 2 * NB2 + a] = make_float2(vx[rr * 2 * NB2 + 2 * a], vx[rr * 2 * NB2 + 2 * a + 1]);
        my[rr * 2 * NB2 + NB2 + a] =
            make_float2(ysign * vy[rr * 2 * NB2 + 2 * a], ysign * vy[rr * 2 * NB2 + 2 * a + 1]);
      }
    __syncwarp();
    // lane l covers row p0 + l / (2 NB2), element l % (2 NB2) of every state of the warp
    const int p = t * TR + rq * RPC + lane / (2 * NB2);
    if (p < nk) {
      for (int j = 0; j < 32 && qb + j < nrhs; ++j) {
        const float2 v = wsm[j * 33 + lane];
        float2* dst = acc + (size_t)(qb + j) * astride + (size_t)p * 2 * NB2 + lane % (2 * NB2);
        if (IMAG) {
          const float2 o = *dst;
          *dst = make_float2(o.x - v.y, o.y + v.x);
        } else {
          *dst = v;
        }
      }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tc_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------------------
// RK4 stage of the nb = 2 batch in one kernel behind the contraction: the split finish (k_finish<2, 2, true>), the
// update, and the next stage's coordinates straight into the operand blocks. As three kernels (finish, k_prep_tc,
// k_pack_tc: 72 + 24 + 15 us per evaluation of 96 states on 5000 k-points, more than the contraction's 64) the state went
// through memory three times, each thread reloaded its k-point's constants for every state, and the FP64 pipe did 60
// operations per state and k-point.
// A warp takes one state's elements of a column group's 8 energy ranks, a lane per element (a thread per k-point needs 128
// registers: 16 warps per SM and 75 us), and walks states with the k-points' constants and phases in registers; its
// stores are whole 64-byte halves of an operand row. It takes 43 to 50 us there, the FP64 pipe 64 % busy (the update's own
// multiply-adds and the exact splits); the RK4 step went from 700 to 484 us (1000 k-points, 16 states: 85 us).
// Slopes are kept in FP32, which holds them exactly (the finish forms them in FP32; no coherent or drift term here). Conversions and comparisons of doubles run on the FP64 pipe too
// (with them it was 79 % busy): they are integer operations here, and each real takes one fused multiply-add.
// ---------------------------------------------------------------------------------------------
struct TcStage {
  const int* inv;          // energy rank -> k
  uint16_t* A;             // coordinate blocks, part 0
  int nmb;
  float2* ph_next;         // the next evaluation's phases (two buffers in turn: FinishArgs::ph32 is the other one)
  unsigned int* hflag;     // the next evaluation's flag
  int phase;
  TimeArg ta;              // the next evaluation's time
};

// (float)x, round to nearest even, in integer arithmetic; outside FP32's normal range (zeros apart) the conversion
static __device__ __noinline__ float narrow_rare(double x) { return (float)x; }
__device__ __forceinline__ float narrow(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), sgn = hi & 0x80000000u;
  const unsigned e = hi - sgn - (897u << 20);  // exponent (and mantissa) above the smallest normal
  if (e >= (254u << 20)) return ((hi - sgn) | lo) ? narrow_rare(x) : __int_as_float((int)hi);
  // 29 bits go: half a unit less one, and one more where the last bit kept is odd
  const unsigned long long m =
      ((unsigned long long)(hi - sgn) << 32 | lo) - (896ull << 52) + 0xfffffffull + ((lo >> 29) & 1u);
  return __int_as_float((int)(sgn | (unsigned)(m >> 29)));
}
// (double)x
static __device__ __noinline__ double widen_rare(float x) { return (double)x; }
__device__ __forceinline__ double widen(float x) {
  const unsigned b = (unsigned)__float_as_int(x), sgn = b & 0x80000000u, u = b - sgn;
  if (u - 0x800000u >= 0x7f000000u) return u ? widen_rare(x) : __hiloint2double((int)b, 0);
  return __hiloint2double((int)(sgn | ((u >> 3) + (896u << 20))), (int)(b << 29));
}
// x == y, x == -y (NaN as equal patterns) and x != 0
__device__ __forceinline__ bool same(double x, double y) {
  const long long a = __double_as_longlong(x), b = __double_as_longlong(y);
  return a == b || ((a | b) << 1) == 0;
}
__device__ __forceinline__ bool opposite(double x, double y) {
  const long long a = __double_as_longlong(x), b = __double_as_longlong(y);
  return (a ^ b) == (long long)0x8000000000000000ull || ((a | b) << 1) == 0;
}
__device__ __forceinline__ bool nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }

__device__ __forceinline__ void tc_store4(uint16_t* blk, int m, int kk, const float* r) {
  uint32_t h[2], l[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const __nv_bfloat162 hi = __floats2bfloat162_rn(r[2 * i], r[2 * i + 1]);
    const __nv_bfloat162 lo =
        __floats2bfloat162_rn(__fsub_rn(r[2 * i], __low2float(hi)), __fsub_rn(r[2 * i + 1], __high2float(hi)));
    h[i] = *reinterpret_cast<const uint32_t*>(&hi);
    l[i] = *reinterpret_cast<const uint32_t*>(&lo);
  }
  *reinterpret_cast<uint2*>(blk + tc_ci(m, kk)) = make_uint2(h[0], h[1]);  // 4 elements: half of a swizzled 16-byte unit
  *reinterpret_cast<uint2*>(blk + tc_ci(m, kk + 32)) = make_uint2(l[0], l[1]);
}

// the anti-Hermitian part's coordinate blocks, from the stage's input; gated
__global__ void __launch_bounds__(128) k_anti_tc2(FinishArgs a, TcStage p, uint16_t* __restrict__ A1) {
  if (*a.hflag == 0u) return;
  const int pr = blockIdx.x * 8 + (threadIdx.x & 7);
  if (pr >= a.nk) return;
  const int k = p.inv[pr];
  const float2 D = p.phase ? a.ph32[(size_t)k * 4 + 1] : make_float2(1.f, 0.f);
  for (int q = threadIdx.x >> 3; q < a.nrhs; q += 16) {
    const double2* y = a.y + (size_t)q * a.sstride + (size_t)k * 4;
    const double2 y1 = y[1], y2 = y[2];
    // A_ij = (rho_ij - conj(rho_ji)) / (2i), times conj(D)
    const float2 af = make_float2((float)__dmul_rn(__dadd_rn(y1.y, y2.y), 0.5), (float)__dmul_rn(__dsub_rn(y2.x, y1.x), 0.5));
    const float r[4] = {(float)y[0].y, __fmaf_rn(D.x, af.x, D.y * af.y), __fmaf_rn(D.x, af.y, -D.y * af.x), (float)y[3].y};
    tc_store4(A1 + ((size_t)blockIdx.x * p.nmb + q / TC_M) * TC_ABLOCK, q % TC_M, (threadIdx.x & 7) * 4, r);
  }
}

__device__ __forceinline__ float2 quad_get(float2 v, int lane) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

// A grid of one wave: every warp takes an equal run of the (column group, state) tasks, states innermost, and reloads
// the constants where its run enters a group (equal shares of a group's states per block leave a second, nearly empty
// wave or too few warps: 67 and 84 us).
constexpr int kTcStageCtas = 8;
__global__ void __launch_bounds__(128, kTcStageCtas) k_stage_tc2(FinishArgs a, TcStage p, int ngroups) {
  const int lane = threadIdx.x & 31, e = lane & 3, i = e >> 1, j = e & 1, l0 = lane - e, tl = l0 + 2 * j + i;
  if (a.hflag && blockIdx.x == 0 && threadIdx.x == 0) *a.hflag = 0u;  // every pair launch of this evaluation has completed
  const long long tasks = (long long)ngroups * a.nrhs, warps = 4LL * gridDim.x, w = 4LL * blockIdx.x + (threadIdx.x >> 5);
  const long long t1 = tasks * (w + 1) / warps;
  const float2 zero = make_float2(0.f, 0.f), one = make_float2(1.f, 0.f);
  const float pf = (float)(a.prefac * 0.5);
  const double hs = a.tref[a.stage == 2 ? 1 : a.stage == 3 ? 3 : 2];  // h, h/6, h/2
  const size_t n = a.sstride * a.nrhs;
  float2* const K = (float2*)a.K;
  double2* const out = a.stage < 3 ? a.ytmp : a.ybase;
  // element (rank, e) of a row: 4 ranks of 4 elements per swizzled 16-byte unit and half
  const int kk = (lane >> 2) * 4 + e;
  int group = -1, pr = 0;
  bool live = false, flag = false;
  size_t ke = 0;
  float2 x0 = zero, y0 = zero, v0 = zero, D = one, dn = one;
  double fi = 0.0;
  float ffi = 0.f, ffj = 0.f;
  const long long t0 = tasks * w / warps;
  int gt = (int)(t0 / a.nrhs), q = (int)(t0 - (long long)gt * a.nrhs) - 1;
  for (int left = (int)(t1 - t0); left > 0; --left) {
    if (++q == a.nrhs) {
      q = 0;
      ++gt;
    }
    if (gt != group) {  // this element's constants
      group = gt;
      pr = gt * 8 + (lane >> 2);
      live = pr < a.nk;
      if (!live) pr = a.nk - 1;
      const int k = p.inv[pr];
      ke = (size_t)k * 4 + e;
      x0 = a.x0y0 ? a.x0y0[(size_t)k * 8 + e] : zero;
      y0 = a.x0y0 ? a.x0y0[(size_t)k * 8 + 4 + e] : zero;
      v0 = a.v0 ? a.v0[ke] : zero;
      fi = a.fref[2 * (size_t)k + i];
      ffi = (float)fi;
      ffj = (float)a.fref[2 * (size_t)k + j];
      D = (a.phase && i != j) ? a.ph32[ke] : one;
      if (p.phase) {  // D(0, 1) of the next time
        const double x = (a.ew[2 * (size_t)k] - a.ew[2 * (size_t)k + 1]) * eval_time(p.ta);
        float sn, cs;
        sincosf((float)fma(-6.283185307179586, rint(x * 0.15915494309189535), x), &sn, &cs);
        dn = make_float2(cs, sn);
        if (live && q == 0) p.ph_next[ke] = i == j ? one : (i < j ? dn : make_float2(cs, -sn));
      }
    }
    const size_t el = (size_t)q * a.sstride + ke;
    const float2* Xs = (const float2*)a.acc + (size_t)q * a.astride + (size_t)pr * 8 + e;
    float2 X = Xs[0], Y = Xs[4];
    const double2 y = a.y[el], yb = a.stage == 0 ? y : a.ybase[el];
    // X = (M^H)^-1 X'
    const float2 xo = quad_get(X, tl), yo = quad_get(Y, tl);
    if (i < j) {
      X = make_float2(0.5f * (X.x - xo.y), 0.5f * (X.y + xo.x));
      Y = make_float2(0.5f * (Y.x - yo.y), 0.5f * (Y.y + yo.x));
    } else if (i > j) {
      X = make_float2(0.5f * (xo.x + X.y), 0.5f * (xo.y - X.x));
      Y = make_float2(0.5f * (yo.x + Y.y), 0.5f * (yo.y - Y.x));
    }
    // herm_up(rho - F): upper triangle, real diagonal (the diagonal difference in FP64)
    float2 dh = i == j ? make_float2(narrow(__dsub_rn(y.x, fi)), 0.f) : make_float2(narrow(y.x), narrow(y.y));
    const float2 dho = quad_get(dh, tl);
    if (i > j) dh = make_float2(dho.x, -dho.y);
    const float2 PXd = fmul(D, X), PYd = fmul(D, Y), PXt = ffma(D, x0, PXd), PYt = ffma(D, y0, PYd);
    float2 c;
    if (a.lin) {
      c = PXd;
    } else {
      c = make_float2((1.f - ffi) * PXd.x - ffj * PYd.x, (1.f - ffi) * PXd.y - ffj * PYd.y);
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const float2 d1 = quad_get(dh, l0 + 2 * i + l), m = quad_get(PYt, l0 + 2 * i + l);
        c = ffma(make_float2(-d1.x, -d1.y), quad_get(PXt, l0 + 2 * l + j), c);
        c = ffma(make_float2(-m.x, -m.y), quad_get(dh, l0 + 2 * l + j), c);
      }
    }
    // (prefac/2)(c + c^dagger) + D o V0; the (1, 0) element is the exact conjugate of the (0, 1) one
    const float2 co = quad_get(c, tl);
    float2 f = make_float2(pf * (c.x + co.x), pf * (c.y - co.y));
    if (a.v0) f = ffma(D, v0, f);
    const float2 fo = quad_get(f, tl);
    if (i > j) f = make_float2(fo.x, -fo.y);
    double2 yn;
    if (a.stage < 3) {
      yn = mk2(fma(hs, widen(f.x), yb.x), fma(hs, widen(f.y), yb.y));
    } else {  // y + h/6 (k1 + 2 k2 + 2 k3 + k4): the sum to 2^-71 of its largest term, as three floats
      const float2 k1 = K[el], k2 = K[n + el], k3 = K[2 * n + el];
      auto sum = [&](float u, float v, float w, float x, double base) {
        float s, t, r, q, low, rest;
        two_sum(u, __fadd_rn(v, v), s, t);
        two_sum(s, __fadd_rn(w, w), s, r);
        two_sum(s, x, s, q);
        two_sum(t, r, low, rest);
        two_sum(low, q, low, t);
        return fma(hs, widen(s), fma(hs, widen(low), fma(hs, widen(__fadd_rn(rest, t)), base)));
      };
      yn = mk2(sum(k1.x, k2.x, k3.x, f.x, yb.x), sum(k1.y, k2.y, k3.y, f.y, yb.y));
    }
    if (live) {
      out[el] = yn;
      if (a.stage < 3) K[(size_t)a.stage * n + el] = f;
    }
    // the next evaluation's coordinates: conj(D) o (rho - diag(f)), element (0, 1) real part, (1, 0) imaginary part
    const double2 yt = mk2(__shfl_sync(0xffffffffu, yn.x, tl), __shfl_sync(0xffffffffu, yn.y, tl));
    flag |= live && (i == j ? nonzero(yn.y) : (!same(yn.x, yt.x) || !opposite(yn.y, yt.y)));
    float r;
    if (i == j) {
      r = narrow(__dsub_rn(yn.x, fi));
    } else {
      const float ax = narrow(yn.x), ay = narrow(yn.y), bx = narrow(yt.x), by = narrow(yt.y);
      const float2 hf = make_float2(0.5f * (ax + bx), i < j ? 0.5f * (ay - by) : 0.5f * (by - ay));
      r = i < j ? __fmaf_rn(dn.x, hf.x, dn.y * hf.y) : __fmaf_rn(dn.x, hf.y, -dn.y * hf.x);
    }
    const __nv_bfloat16 hi = __float2bfloat16_rn(r), lo = __float2bfloat16_rn(__fsub_rn(r, __bfloat162float(hi)));
    if (live) {
      uint16_t* const blk = p.A + ((size_t)gt * p.nmb + q / TC_M) * TC_ABLOCK;
      blk[tc_ci(q % TC_M, kk)] = __bfloat16_as_ushort(hi);
      blk[tc_ci(q % TC_M, kk + 32)] = __bfloat16_as_ushort(lo);
    }
  }
  if (__any_sync(0xffffffffu, flag) && lane == 0) atomicOr(p.hflag, 1u);
}

}  // namespace dmd
