// Row-tile machinery shared by the two Arnoldi variants (Householder in
// krylov.cu, modified Gram-Schmidt in krylov_mgs.cu): the operator applied
// to a tile of rows, deterministic block and grid reductions, FP32<->FP64
// conversions on the integer pipes, and the unsolved-pattern prefill of the
// sync-free solves' outputs.
#pragma once

#include <algorithm>

#include "internal.h"

namespace lace {

constexpr int kTPB = 256;   // threads per block of the row-tile kernels

// operator row i of the tile: CSR (LPR lanes per row) or BCSR (thread/row)
struct OpView {
  int bs;
  const int *row, *col;
  const double *val;
  const int *sell_ptr, *sell_col;  // sliced ELL (CSR row pointers give the row lengths)
  const double *sell_val;
};

template <int LPR, typename ZT>
__device__ __forceinline__ void tile_apply(const OpView &op, int n, int base, int tr,
                                           const ZT *__restrict__ z, double *sw) {
  if (op.bs == 0 && op.sell_ptr != nullptr) {
    // sliced ELL: warp w takes the 32-row slices w, w+8, ... of the tile; entry
    // t of the slice's rows is one coalesced load, four entries in flight
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int t0 = wid * 32; t0 < tr; t0 += kTPB) {
      const int i = base + t0 + lane;
      double s = 0.0;
      if (i < n) {
        const int len = op.row[i + 1] - op.row[i];
        const int *cp = op.sell_col + op.sell_ptr[(base + t0) >> 5] + lane;
        const double *vp = op.sell_val + (cp - op.sell_col);
        for (int t = 0; t < len; t += 4) {
          int c[4];
          double v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (t + u < len) {
              c[u] = cp[32 * (t + u)];
              v[u] = vp[32 * (t + u)];
            }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (t + u < len) s = fma(v[u], to_f64(z[c[u]]), s);
        }
      }
      sw[t0 + lane] = s;
    }
  } else if (op.bs == 0) {
    const int sub = threadIdx.x & (LPR - 1);
    const int grp = threadIdx.x / LPR;
    constexpr int G = kTPB / LPR;
    for (int t = grp; t < tr; t += G) {
      const int i = base + t;
      double s = 0.0;
      if (i < n) {
        const int e = op.row[i + 1];
        for (int p = op.row[i] + sub; p < e; p += LPR) s = fma(op.val[p], to_f64(z[op.col[p]]), s);
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, LPR);
      if (sub == 0) sw[t] = s;
    }
  } else {
    const int bs = op.bs, ld = bs * bs;
    for (int t = threadIdx.x; t < tr; t += kTPB) {
      const int i = base + t;
      double s = 0.0;
      if (i < n) {
        const int I = i / bs, r = i - I * bs;
        for (int p = op.row[I]; p < op.row[I + 1]; ++p) {
          const double *blk = op.val + (size_t)p * ld + r * bs;
          const ZT *zj = z + (size_t)op.col[p] * bs;
          for (int c = 0; c < bs; ++c) s = fma(blk[c], to_f64(zj[c]), s);
        }
      }
      sw[t] = s;
    }
  }
}

__device__ __forceinline__ double block_sum(double v, double *scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kTPB / 32; ++w) t += scratch[w];
  return t;  // valid in thread 0
}

// last block: sred[k] = sum over blocks of partials[b*kLdT + k], k < count;
// warp w takes k = w, w+8, ..., its lanes stride over the blocks (fixed
// order, so the result is deterministic)
__device__ __forceinline__ void fold_partials(const double *partials, int count, double *sred) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = wid; k < count; k += kTPB / 32) {
    double s = strided_sum(partials + k, kLdT, lane, 32, (int)gridDim.x);
    s = warp_sum(s);
    if (lane == 0) sred[k] = s;
  }
}

// FP64 -> FP32 with integer operations, rounding toward zero (the FP64 unit,
// which also converts, is the scarce one).  Finite values only: below the
// FP32 normal range they become 0, above it NaN.
__device__ __forceinline__ float dtof_rz(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hi = (unsigned)(b >> 32);
  const int e = (int)((hi >> 20) & 0x7ffu) - 896;
  const unsigned m = ((hi & 0xfffffu) << 3) | ((unsigned)b >> 29);
  const unsigned mag = e <= 0 ? 0u : (e >= 255 ? 0x7fc00000u : (((unsigned)e << 23) | m));
  return __uint_as_float((hi & 0x80000000u) | mag);
}

// Double-float values: an FP64 value x as hi = dtof_rz(x) and lo =
// dtof_rz(x - hi), about 48 bits together (finite |x| < 2^128; lo of values
// near the FP32 underflow flushes to 0), so that products and sums of FP64
// data run on the FP32 unit - 64 times the FP64 unit's rate on this part -
// with FP64-like accuracy.  Conversions use integer operations.
__device__ __forceinline__ float2 df_split(double x) {
  const float h = dtof_rz(x);
  return make_float2(h, dtof_rz(x - to_f64(h)));
}
__device__ __forceinline__ double df_join(float2 v) { return to_f64(v.x) + to_f64(v.y); }
// (sh, sl) += (ah + al) * (bh + bl): the high product exactly (an FMA gives
// its rounding error), the cross terms in FP32, al*bl dropped (2^-48
// relative), the high parts summed error-free (TwoSum), the rest into sl
__device__ __forceinline__ void df_mac(float ah, float al, float bh, float bl, float &sh, float &sl) {
  const float p = ah * bh;
  const float pe = fmaf(ah, bl, fmaf(al, bh, fmaf(ah, bh, -p)));
  const float t = sh + p;
  const float z = t - sh;
  const float e = (sh - (t - z)) + (p - z);
  sh = t;
  sl += e + pe;
}// (sh, sl) += (ah + al) * b for an FP32 b
__device__ __forceinline__ void df_mac1(float ah, float al, float b, float &sh, float &sl) {
  const float p = ah * b;
  const float pe = fmaf(al, b, fmaf(ah, b, -p));
  const float t = sh + p;
  const float z = t - sh;
  const float e = (sh - (t - z)) + (p - z);
  sh = t;
  sl += e + pe;
}

// pair arithmetic for values kept as pairs: h + l as an unevaluated sum
// renormalised (TwoSum: exact for any magnitudes), a + b (the high parts
// summed error-free, the low parts added) and a * b (the high product
// exactly, the cross terms in FP32, a.lo * b.lo dropped)
__device__ __forceinline__ float2 df_renorm(float h, float l) {
  const float t = h + l, z = t - h;
  return make_float2(t, (h - (t - z)) + (l - z));
}
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
  const float t = a.x + b.x, z = t - a.x;
  const float e = (a.x - (t - z)) + (b.x - z);
  return df_renorm(t, e + (a.y + b.y));
}
__device__ __forceinline__ float2 df_mul(float2 a, float2 b) {
  const float p = a.x * b.x;
  const float e = fmaf(a.x, b.y, fmaf(a.y, b.x, fmaf(a.x, b.x, -p)));
  const float s = p + e;  // |e| <= |p| up to rounding: Fast2Sum
  return make_float2(s, e - (s - p));
}

// the unsolved pattern (all ones) into row i of an FP32 or FP64 vector: the
// sync-free solve that writes the vector polls it until the pattern is gone
__device__ __forceinline__ void mark_unsolved(void *x, int f32, size_t i) {
  if (f32) reinterpret_cast<unsigned *>(x)[i] = ~0u;
  else reinterpret_cast<unsigned long long *>(x)[i] = ~0ull;
}

// the vectors the next step's two solves write, marked unsolved (null: none)
struct Prefill {
  void *t, *z;
  int t_f32, z_f32;
};

__device__ __forceinline__ void prefill_row(const Prefill &f, size_t i) {
  if (f.t) mark_unsolved(f.t, f.t_f32, i);
  if (f.z) mark_unsolved(f.z, f.z_f32, i);
}

// ------------------------------------- persistent (cooperative) kernels

// Sums over a cooperatively launched grid without a barrier: every block
// stores its partial sums with a tag, and every block reads all of them until
// the tags are there, so a sum costs one trip through L2 and back instead of
// an arrival, a generation and then the read (each a trip of its own, behind a
// fence of every thread: a Gram-Schmidt sum took 5.5 us of an otherwise empty
// step on 152 blocks).  A 64-bit value is two 64-bit words of a tag and 32 bits
// each, so that a word is its own ready flag.  A launch's tags start from the
// epoch the last one left (one tag per fold); two phases of slots take turns, so
// a block may run one fold ahead.  Bounded: a wait that gives up sets
// kStatusSpinTimeout, and every block leaves at its next fold.
constexpr int kFoldCap = 2 * kLdT;  // values of one fold at most
struct FoldSlots {
  unsigned *epoch;
  ulonglong2 *slot;  // two phases of kFoldCap x gridDim.x, two of kFoldCap sums, kLdT single values
};
inline size_t fold_bytes(int blocks) { return 16 + sizeof(ulonglong2) * (2 * (size_t)kFoldCap * (blocks + 1) + kLdT); }
static inline FoldSlots fold_slots(void *buf) { return FoldSlots{(unsigned *)buf, (ulonglong2 *)((char *)buf + 16)}; }

__device__ __forceinline__ void tag_put(ulonglong2 *p, double v, unsigned tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | (b & 0xffffffffull)), "l"(t | (b >> 32))
               : "memory");
}
__device__ __forceinline__ ulonglong2 tag_load(const ulonglong2 *p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool tag_is(ulonglong2 v, unsigned tag) {
  return (unsigned)(v.x >> 32) == tag && (unsigned)(v.y >> 32) == tag;
}
__device__ __forceinline__ double tag_value(ulonglong2 v) {
  return __longlong_as_double((long long)((v.x & 0xffffffffull) | (v.y << 32)));
}
__device__ __forceinline__ bool tag_gave_up(int spins, Control *ctrl) {
  if (spins <= kMaxSpins && !((spins & 1023) == 1023 && (ld_relaxed(&ctrl->status) & kStatusSpinTimeout))) return false;
  atomicOr(&ctrl->status, kStatusSpinTimeout);
  return true;
}
// one tagged value, waited for
__device__ __forceinline__ double tag_get(const ulonglong2 *p, unsigned tag, Control *ctrl, bool &ok) {
  ulonglong2 v = tag_load(p);
  for (int spins = 0; !tag_is(v, tag); ++spins) {
    if (tag_gave_up(spins, ctrl)) {
      ok = false;
      break;
    }
    v = tag_load(p);
  }
  return tag_value(v);
}
// the lane's part of a sum over the blocks: p[b] for b = lane, lane + 32, ...
// added in that order
__device__ __forceinline__ double tag_lane_sum(const ulonglong2 *p, int blocks, unsigned tag, Control *ctrl, bool &ok) {
  double t = 0.0;
  for (int b0 = threadIdx.x & 31; b0 < blocks; b0 += 160) {
    ulonglong2 v[5];
    for (int spins = 0;; ++spins) {
      bool wait = false;
#pragma unroll
      for (int u = 0; u < 5; ++u)
        if (b0 + 32 * u < blocks) v[u] = tag_load(p + b0 + 32 * u);
#pragma unroll
      for (int u = 0; u < 5; ++u)
        if (b0 + 32 * u < blocks) wait |= !tag_is(v[u], tag);
      if (!wait) break;
      if (tag_gave_up(spins, ctrl)) {
        ok = false;
        break;
      }
    }
#pragma unroll
    for (int u = 0; u < 5; ++u)
      if (b0 + 32 * u < blocks) t += tag_value(v[u]);
  }
  return t;
}

// ------------------------------------- shared by the one-kernel steps

// sum_k V[k][i] c[k] over k < ncols: eight independent loads in flight
__device__ __forceinline__ double vcomb8(const double *__restrict__ V, size_t ldv, int i, int ncols,
                                         const double *c) {
  double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  int k = 0;
  for (; k + 8 <= ncols; k += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = fma(V[(size_t)(k + u) * ldv + i], c[k + u], a[u]);
  }
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (k + u < ncols) a[u] = fma(V[(size_t)(k + u) * ldv + i], c[k + u], a[u]);
  return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

// rows i, i+1 (i even, i+1 < n): sum_k V[k][i..i+1] c[k] over k < ncols with
// 16-byte loads, a batch of eight columns in flight before any use
__device__ __forceinline__ double2 vcomb8x2(const double *__restrict__ V, size_t ldv, int i, int ncols,
                                           const double *c) {
  // two accumulators per row: the FP64 unit is the scarce one, so few
  // closing additions matter more than a short dependency chain
  double2 a[2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int k = 0; k < ncols; k += 8) {
    // a partial batch skips its missing columns
    double2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u < ncols) v[u] = __ldg(reinterpret_cast<const double2 *>(V + (size_t)(k + u) * ldv + i));
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k + u < ncols) {
        a[u & 1].x = fma(v[u].x, c[k + u], a[u & 1].x);
        a[u & 1].y = fma(v[u].y, c[k + u], a[u & 1].y);
      }
  }
  return make_double2(a[0].x + a[1].x, a[0].y + a[1].y);
}

// block partial sums sacc[k] = sum over this block's rows i > lo of
// V[k][i] w[i], k < jp1: up to 32 columns as (column, row group) pairs over
// the 32 warps, more as up to five columns per warp; lanes walk rows
__device__ __forceinline__ void hh_block_dots(const double *__restrict__ V, size_t ldv, int jp1, int r0, int r1,
                                              int lo, const double *sw, double *swarp, double *sacc) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nsl = r1 > r0 ? (r1 - r0 + 31) >> 5 : 0;
  if (jp1 <= 32) {
    // row groups per column: no more than have eight slices each to load at once
    // (every group costs a warp's FP64 sum and an addition)
    const int G = max(1, min(32 / jp1, nsl >> 3));
    double acc = 0.0;
    if (wid < G * jp1) {
      // a warp streams its column over 1/G of the rows: eight rows per lane
      // in flight (one block per SM has few warps to hide the latency)
      const int k = wid % jp1, g = wid / jp1;
      const double *Vk = V + (size_t)k * ldv + r0;
      for (int sl0 = g; sl0 < nsl; sl0 += 8 * G) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int t = 32 * (sl0 + u * G) + lane;
          v[u] = (sl0 + u * G < nsl && r0 + t < r1) ? Vk[t] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int t = 32 * (sl0 + u * G) + lane;
          const int i = r0 + t;
          acc = fma(v[u], (sl0 + u * G < nsl && i < r1 && i > lo) ? sw[t] : 0.0, acc);
        }
      }
      acc = warp_sum(acc);
    }
    if (lane == 0) swarp[wid] = acc;
    __syncthreads();
    if (threadIdx.x < jp1) {
      double t = 0.0;
      for (int g = 0; g < G; ++g) t += swarp[g * jp1 + threadIdx.x];
      sacc[threadIdx.x] = t;
    }
  } else {
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int sl0 = 0; sl0 < nsl; sl0 += 4) {
      // four rows per lane for each of the warp's columns in flight
      double wv[4];
      int ii[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = 32 * (sl0 + u) + lane;
        const int i = r0 + t;
        const bool ok = sl0 + u < nsl && i < r1 && i > lo;
        wv[u] = ok ? sw[t] : 0.0;
        ii[u] = ok ? i : r0;
      }
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        const int k = wid + 32 * c;
        if (32 * c < jp1 && k < jp1) {
          double v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = V[(size_t)k * ldv + ii[u]];
#pragma unroll
          for (int u = 0; u < 4; ++u) acc[c] = fma(v[u], wv[u], acc[c]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const int k = wid + 32 * c;
      if (32 * c < jp1) {  // warp-uniform
        const double v = warp_sum(acc[c]);
        if (lane == 0 && k < jp1) swarp[k] = v;
      }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < jp1; k += blockDim.x) sacc[k] = swarp[k];
  }
  __syncthreads();
}

// sres[k] = sum over the grid of the blocks' sacc[k], k < nv, the same in
// every block.  One or two values: every block adds all partial sums (a warp
// per value).  More: block k adds value k's and hands the sum out, two trips
// through L2 - every block adding every value costs ten FP64 instructions of a
// warp per value and block, 16 cycles of the SM's FP64 unit each (at 31 values
// 5 us more).  ntop > 0: the rows top0..top1-1 of w that this block owns go out
// as well, and sres gets rows 0..ntop-1 from position nv on.
__device__ __forceinline__ bool hh_grid_fold(const double *sacc, int nv, const FoldSlots &f, unsigned tag, Control *ctrl,
                                             double *sres, const double *stop = nullptr, int top0 = 0, int top1 = 0,
                                             int ntop = 0) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int G = gridDim.x;
  ulonglong2 *P = f.slot + (size_t)(tag & 1) * kFoldCap * G;
  ulonglong2 *R = f.slot + (2 * (size_t)G + (tag & 1)) * kFoldCap, *top = f.slot + (2 * (size_t)G + 2) * kFoldCap;
  for (int k = top0 + (int)threadIdx.x; k < top1; k += blockDim.x) tag_put(top + k, stop[k - top0], tag);
  for (int k = threadIdx.x; k < nv; k += blockDim.x) tag_put(P + (size_t)k * G + blockIdx.x, sacc[k], tag);
  bool ok = true;
  const bool all = nv <= 2;
  for (int k = all ? wid : (int)blockIdx.x + wid * G; k < nv; k += (int)(blockDim.x >> 5) * (all ? 1 : G)) {
    const double t = warp_sum(tag_lane_sum(P + (size_t)k * G, G, tag, ctrl, ok));
    if (lane == 0) {
      if (all) sres[k] = t;
      else tag_put(R + k, t, tag);
    }
  }
  if (!all)
    for (int k = threadIdx.x; k < nv; k += blockDim.x) sres[k] = tag_get(R + k, tag, ctrl, ok);
  for (int k = threadIdx.x; k < ntop; k += blockDim.x) sres[nv + k] = tag_get(top + k, tag, ctrl, ok);
  return __syncthreads_and(ok);
}

// ------------------------------------------------------------ host side

static inline OpView opview(const ArnoldiArgs &a) {
  return OpView{a.bs, a.row, a.col, a.val, a.sell_ptr, a.sell_col, a.sell_val};
}

static inline int rowgrid(int n) {
  int g = (n + kTPB - 1) / kTPB;
  return std::min(g, num_sms() * 8);
}

// the outputs of step j's two solves (the L solve's vector and column j of Z)
static inline Prefill prefill_for(const ArnoldiArgs &a, int j) {
  if (!a.prefill || j >= a.m) return Prefill{nullptr, nullptr, 0, 0};
  void *zj = (char *)a.Z + (size_t)j * a.ldz * (a.z_f32 ? 4 : 8);
  return Prefill{a.fill_t, zj, a.fill_t_f32, a.z_f32};
}

// One wave: as many blocks as are resident at once (the passes loop over
// their row tiles), so no partly filled last wave, and the last block folds
// few partial sums.  Never more than the ArnoldiArgs grid the partial-sum
// buffer is sized for.
template <typename K>
static inline int wave_grid(K kernel, int cap) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTPB, 0) != cudaSuccess || per_sm <= 0) {
    cudaGetLastError();
    return cap;
  }
  return std::max(1, std::min(cap, per_sm * num_sms()));
}

// Rows of w (or u) per block of a one-kernel step, a multiple of 32: as many
// blocks as SMs, but at least 256 rows each - more blocks on a small system only
// make every sum over them longer.
static inline int step_rows(int n, int sms) { return std::max(256, ((n + sms - 1) / sms + 31) / 32 * 32); }

}  // namespace lace
