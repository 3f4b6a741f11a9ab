// Batched solves, a thread-block cluster for each (system, right-hand side).
//
// A cluster takes a job from the queue (largest systems first) and carries it
// through ParILU(0) and FGMRES-Householder; clusters never wait for one another.
// Its CTAs share the rows of the vectors and of the basis (the dot products and
// combinations are bound by the FP64 units, two multiply-adds a clock and SM, so
// the CTAs of a cluster divide that time), add their partial sums through
// distributed shared memory, and each form the small matrices for themselves.
// The triangular solves push values to shared-memory slots as sptrsv_push.cu
// does, on as few of the cluster's CTAs as hold the slots: a level of a 2D grid
// costs 0.15 us that way where one barrier per level and dependencies read from
// global memory took 1 us and more.  A row marks its slots unsolved again
// when it has read them, so both triangles use the same slots and no solve
// needs a fill.
//
// The arithmetic is that of the single-CTA form (batch_persist.cu: ParILU as
// src/parilu_v0_3.cpp:62-108 in synchronous form, FGMRES as
// src/fgmres_householder_restart.cpp), which still takes the systems whose slots
// fit no cluster or whose rows have too many dependants - but for U's entries,
// scaled by the rounded reciprocal pivot (one rounding more each; a division by the
// pivot would be on the chain of every level: 37 -> 44 ms below, in FP64 47 -> 87).
// Over 4,500 random pairs the residuals are 1.001 times that form's in the
// geometric mean, in FP64 1.000; the error of the case below against 64 bits is the
// same.
//
// Time of 24 systems of 1,089 to 9,025 rows, four right-hand sides each, FP32
// factors, FGMRES(30) to 1e-12: 264 ms with a CTA per system and its four
// right-hand sides in lockstep, 37 ms here (FP64 factors 47).  A direction of the
// largest on four CTAs: 130k cycles of triangular solves (2 x 189 levels), 115k of
// FP64 work (its floor 85k), 20k of small matrices and barriers.
#include <algorithm>

#include <cooperative_groups.h>

#include "context.h"
#include "krylov_tile.cuh"
#include "perdevice.h"
#include "push.cuh"

namespace lace {

namespace {

constexpr int kCT = 32 * kPushW;          // threads per CTA
constexpr int kLd = kBatchMaxM + 2;       // the small matrices' largest leading dimension
constexpr int kCMax = 8;                  // CTAs per cluster at most
constexpr size_t kCSmemMax = 200 * 1024;  // dynamic shared memory: slots, rows of w, T and R

// eight FP64 sums over the warp, reduce-scatter: afterwards lane l holds the
// total of value sum8_slot(l)
__device__ __forceinline__ double sum8(double (&a)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 4; h >= 1; h >>= 1) {
    const bool hi = lane & (4 * h);
#pragma unroll
    for (int c = 0; c < h; ++c) {
      const double send = hi ? a[c] : a[c + h];
      const double got = __shfl_xor_sync(0xffffffffu, send, 4 * h);
      a[c] = (hi ? a[c + h] : a[c]) + got;
    }
  }
  a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
  a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
  return a[0];
}
__device__ __forceinline__ int sum8_slot(int lane) {
  return (((lane >> 4) & 1) << 2) | (((lane >> 3) & 1) << 1) | ((lane >> 2) & 1);
}

// f(0) ... f(min(n, 8) - 1), highest first: a jump into straight-line code, because an FP64 instruction that is
// only switched off by its predicate costs as much as one that runs (the second
// set of dot products took 50k cycles at 2,256 rows a CTA that way, the first
// 33k)
template <typename Fn>
__device__ __forceinline__ void upto8(int n, Fn f) {
  switch (n) {
    default: f(7); [[fallthrough]];
    case 7: f(6); [[fallthrough]];
    case 6: f(5); [[fallthrough]];
    case 5: f(4); [[fallthrough]];
    case 4: f(3); [[fallthrough]];
    case 3: f(2); [[fallthrough]];
    case 2: f(1); [[fallthrough]];
    case 1: f(0);
  }
}

// one triangle's plan for the warp: its groups, and their values
template <typename FT>
struct Tri {
  const int *slot, *rc, *dst;  // of the system's first group
  FT *val, *rd;                // this cluster's
  int gb, ge;
};

// x = T^{-1} b on the slots; the caller has synchronised the cluster
template <typename FT, int K, bool LOWER>
__device__ void push_tri(const Tri<FT> &T, const FT *b, FT *x, unsigned base, int rank, int *status) {
  const int lane = threadIdx.x & 31;
  struct Rec {
    int slot, rc, dst[K];
    FT v[K], d;
  } cur, nxt;
  auto load = [&](Rec &r, int g) {
    r.slot = T.slot[g];
    r.rc = T.rc[(size_t)g * 32 + lane];
#pragma unroll
    for (int t = 0; t < K; ++t) {
      r.dst[t] = T.dst[((size_t)g * K + t) * 32 + lane];
      r.v[t] = T.val[((size_t)g * K + t) * 32 + lane];
    }
    r.d = LOWER ? (FT)1 : T.rd[(size_t)g * 32 + lane];
  };
  bool gave_up = false;
  if (T.gb < T.ge) load(cur, T.gb);
  for (int g = T.gb; g < T.ge; ++g) {
    const int row = cur.rc < 0 ? -1 : cur.rc & 0x7ffffff, cnt = cur.rc < 0 ? 0 : cur.rc >> 27;
    FT y = row >= 0 ? __ldcg(b + row) : (FT)0;
    if (g + 1 < T.ge) load(nxt, g + 1);
    Slot dst[K];
    unsigned a[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
      dst[t] = slot_of(base, rank, cur.dst[t]);
      a[t] = base + (unsigned)(((t < cnt ? cur.slot + t : 0) * 32 + lane) * (int)sizeof(FT));
    }
    if (!LOWER) y *= cur.d;
    FT s[K];
    for (int polls = 0;;) {
      bool ok = false;
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // four polls between the limit's tests
        unsigned m = 0;
#pragma unroll
        for (int t = 0; t < K; ++t) {
          s[t] = ld_slot(a[t], (FT)0);
          m = max(m, head(s[t]));
        }
        ok = __all_sync(0xffffffffu, m != 0xffffffffu);
        if (ok) break;
      }
      if (ok || gave_up) break;
      polls += 4;
      if ((polls & 1023) == 0) {
        if (polls > kMaxSpins && lane == 0) atomicOr(status, kStatusSpinTimeout);
        gave_up = __any_sync(0xffffffffu, polls > kMaxSpins || (*(const volatile int *)status & kStatusSpinTimeout));
      }
    }
#pragma unroll
    for (int t = 0; t < K; ++t) y = fma(-cur.v[t], s[t], y);
    if (head(y) == 0xffffffffu) y = (FT)NAN;  // a solved value never carries the mark
#pragma unroll
    for (int t = 0; t < K; ++t) push(dst[t], y);
#pragma unroll
    for (int t = 0; t < K; ++t)
      if (t < cnt) st_mark(a[t], (FT)0);
    if (row >= 0) x[row] = y;
    cur = nxt;
  }
}

template <typename FT, int K>
__global__ void __launch_bounds__(kCT, 1) k_batch_cluster(CBatch P) {
  extern __shared__ __align__(16) unsigned char smem_c[];
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), C = P.C, cluster = blockIdx.x / C;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gw = rank * kPushW + warp;
  const int m = P.m, ld = m + 2;
  // partial sums and the rows of w that every CTA needs, from all CTAs; two sets in turn
  __shared__ double xch[2][kCMax][kLd], xw[2][kLd], xv[2][kLd];
  __shared__ double sred[(kLd / 8 + 1) * kPushW * 8];
  __shared__ double sg[kLd], scs[kLd], ssn[kLd], sc[kLd], ss[kLd], sd[kLd], srho[kLd], sh[kLd];
  __shared__ double s_dd, s_ia, s_rtol;
  __shared__ int s_job, s_live, s_step, s_conv;
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem_c);
  double *ws = reinterpret_cast<double *>(smem_c + P.slot_bytes);
  double *Tm = ws + P.rbmax, *Rm = Tm + (size_t)ld * ld;
  const size_t nmax = P.nmax;
  double *V = P.V + (size_t)cluster * (m + 1) * nmax;
  FT *Z = (FT *)P.Z + (size_t)cluster * m * nmax;
  FT *Q = (FT *)P.Q + (size_t)cluster * nmax, *Tt = (FT *)P.Tt + (size_t)cluster * nmax;
  FT *F0 = (FT *)P.F + (size_t)cluster * 2 * P.fstride;
  Tri<FT> L, U;
  L.val = (FT *)P.val + (size_t)cluster * P.vstride;
  U.val = L.val + (size_t)P.gmax[0] * K * 32;
  U.rd = U.val + (size_t)P.gmax[1] * K * 32;
  L.rd = U.rd;
  // slot row 0 stays 0, the others are unsolved between the solves
  for (unsigned k = tid; k < P.slot_bytes / 16; k += kCT) {
    const unsigned v = k < 2 * sizeof(FT) ? 0u : 0xffffffffu;
    reinterpret_cast<uint4 *>(smem_c)[k] = make_uint4(v, v, v, v);
  }
  int buf = 0;

  // partial sums of nc columns over this CTA's rows, then over the cluster:
  // column k < ncols is V_k . w over rows >= lo, column ncols (if any) w . w
  auto sums = [&](int ncols, int nc, int lo, int r0, int nloc) {
    for (int k0 = 0, ch = 0; k0 < nc; k0 += 8, ++ch) {
      double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      for (int i = tid; i < nloc; i += kCT) {
        if (r0 + i < lo) continue;
        const double wi = ws[i];
        const double *v = V + (size_t)k0 * nmax + r0 + i;
        double t[8];
        upto8(nc - k0, [&](int c) { t[c] = k0 + c < ncols ? v[(size_t)c * nmax] : wi; });
        upto8(nc - k0, [&](int c) { a[c] = fma(t[c], wi, a[c]); });
      }
      const double v = sum8(a);
      if ((lane & 3) == 0) sred[(ch * kPushW + warp) * 8 + sum8_slot(lane)] = v;
    }
    __syncthreads();
    for (int k = tid; k < nc; k += kCT) {
      double t = 0.0;
      for (int w = 0; w < kPushW; ++w) t += sred[((k >> 3) * kPushW + w) * 8 + (k & 7)];
      for (int r = 0; r < C; ++r) *cl.map_shared_rank(&xch[buf][rank][k], r) = t;
    }
  };
  auto total = [&](int k) {
    double t = 0.0;
    for (int r = 0; r < C; ++r) t += xch[buf][r][k];
    return t;
  };

  for (;;) {
    {
      int jb = 0;
      if (rank == 0 && tid == 0) jb = atomicAdd(P.next, 1);
      __syncwarp();
      jb = __shfl_sync(0xffffffffu, jb, 0);
      if (rank == 0 && tid < C) *cl.map_shared_rank(&s_job, tid) = jb;
      __syncwarp();
    }
    cl.sync();
    const int job = s_job;
    if (job >= P.njobs) break;  // the same for the whole cluster
    const int sys = P.jsys[job], rhs = P.jrhs[job];
    const int n = P.n[sys], R0 = P.roff[sys], e0 = P.Arow[R0], e1 = P.Arow[R0 + n];
    const int rb = max(((n + C - 1) / C + 31) / 32 * 32, (m + 2 + 31) / 32 * 32);  // rows a CTA
    const int r0 = rank * rb, nloc = max(0, min(n - r0, rb));
    const double *b = P.b + (size_t)rhs * P.N + R0;
    double *x = P.x + (size_t)rhs * P.N + R0;
    // ---- ParILU(0) into the cluster's buffers: F = A, then the synchronous sweeps
    FT *Fa = F0 - e0, *Fb = F0 + P.fstride - e0;
    for (int p = e0 + rank * kCT + tid; p < e1; p += C * kCT) Fa[p] = (FT)P.Aval[p];
    cl.sync();
    for (int sw = 0; sw < P.sweeps; ++sw) {
      for (int p = e0 + rank * kCT + tid; p < e1; p += C * kCT) {
        FT s = (FT)P.Aval[p];
        for (int q = P.pptr[p]; q < P.pptr[p + 1]; ++q) {
          const int2 pr = P.pairs[q];
          s = fma(-__ldcg(Fa + pr.x), __ldcg(Fa + pr.y), s);
        }
        const int d = P.dpos[p];
        Fb[p] = d >= 0 ? s / __ldcg(Fa + d) : s;
      }
      cl.sync();
      FT *t = Fa;
      Fa = Fb;
      Fb = t;
    }
    // the factor values in the order the warp's groups use them, U's scaled by
    // the reciprocal diagonal
    for (int up = 0; up < 2; ++up) {
      Tri<FT> &T = up ? U : L;
      const int *wp = P.wptr[up] + (size_t)sys * (C * kPushW + 1) + gw;
      const size_t g0 = P.goff[up][sys];
      T.gb = wp[0];
      T.ge = wp[1];
      T.slot = P.slot[up] + g0;
      T.rc = P.rc[up] + g0 * 32;
      T.dst = P.dst[up] + g0 * K * 32;
      const int *map = P.map[up] + g0 * K * 32, *dmap = P.dmap[up] + g0 * 32;
      for (int g = T.gb; g < T.ge; ++g) {
        FT rd = (FT)1;
        if (up) {
          const int dm = dmap[(size_t)g * 32 + lane];
          rd = dm >= 0 ? (FT)1 / __ldcg(Fa + dm) : (FT)0;
          T.rd[(size_t)g * 32 + lane] = rd;
        }
#pragma unroll
        for (int t = 0; t < K; ++t) {
          const int mp = map[((size_t)g * K + t) * 32 + lane];
          T.val[((size_t)g * K + t) * 32 + lane] = mp >= 0 ? __ldcg(Fa + mp) * rd : (FT)0;
        }
      }
    }
    // ---- FGMRES-Householder
    bool first = true;
    int iters = 0, conv = 0;
    for (int cyc = 0; cyc < P.restart_max; ++cyc) {
      // r = b - A x, its norm
      for (int i = tid; i < nloc; i += kCT) {
        const int r = r0 + i;
        double s = b[r];
        for (int p = P.Arow[R0 + r]; p < P.Arow[R0 + r + 1]; ++p)
          s = fma(-P.Aval[p], __ldcg(x + (P.Acol[p] - R0)), s);
        ws[i] = s;
      }
      sums(0, 1, 0, r0, nloc);
      if (rank == 0 && tid < C) *cl.map_shared_rank(&xw[buf][0], tid) = ws[0];
      cl.sync();
      if (tid == 0) {
        const double rn2 = total(0), rnorm = sqrt(rn2);
        if (first) s_rtol = P.rtol * rnorm;
        s_step = 0;
        s_conv = s_live = 0;  // s_conv: 1 converged, -1 not finite
        if (rnorm < s_rtol || rnorm == 0.0) {
          s_conv = 1;
        } else if (!(rnorm >= s_rtol)) {
          s_conv = -1;
        } else {
          const double w0 = xw[buf][0];
          const double dd = mysgn(w0) * rnorm;
          const double alpha = sqrt(2.0 * (rn2 + fabs(w0) * rnorm));
          s_dd = dd;
          s_ia = alpha > 0.0 ? 1.0 / alpha : 0.0;
          sg[0] = -dd;
          Tm[0] = 2.0;
          s_live = 1;
        }
      }
      buf ^= 1;
      first = false;
      __syncthreads();
      if (!s_live) {
        conv = s_conv;
        break;
      }
      // v_0 = (r + dd e_0) / alpha, q_0 = -r / dd
      {
        const double dd = s_dd, ia = s_ia, rdd = 1.0 / dd;
        for (int i = tid; i < nloc; i += kCT) {
          const double wi = ws[i];
          V[r0 + i] = (r0 + i == 0 ? wi + dd : wi) * ia;
          Q[r0 + i] = (FT)(-wi * rdd);
        }
      }
      for (int j = 0;; ++j) {
        const int jp1 = j + 1;
        FT *zj = Z + (size_t)j * nmax;
        // ---- z_j = U^-1 L^-1 q_j, w = A z_j
        cl.sync();
        push_tri<FT, K, true>(L, Q, Tt, base, rank, P.status);
        cl.sync();
        push_tri<FT, K, false>(U, Tt, zj, base, rank, P.status);
        cl.sync();
        for (int i = tid; i < nloc; i += kCT) {
          double s = 0.0;
          for (int p = P.Arow[R0 + r0 + i]; p < P.Arow[R0 + r0 + i + 1]; ++p)
            s = fma(P.Aval[p], to_f64(__ldcg(zj + (P.Acol[p] - R0))), s);
          ws[i] = s;
        }
        // ---- s = V^T w, y = T^T s, w -= V y
        sums(jp1, jp1, 0, r0, nloc);
        cl.sync();
        for (int k = tid; k < jp1; k += kCT) ss[k] = total(k);
        buf ^= 1;
        __syncthreads();
        for (int e = tid; e < 4 * ((jp1 + 7) & ~7); e += kCT) {  // four threads an entry, whole warps
          const int k = e >> 2;
          double y = 0.0;
          if (k < jp1)
            for (int l = e & 3; l <= k; l += 4) y = fma(Tm[l + k * ld], ss[l], y);
          y += __shfl_xor_sync(0xffffffffu, y, 1);
          y += __shfl_xor_sync(0xffffffffu, y, 2);
          if (k < jp1 && (e & 3) == 0) sd[k] = y;
        }
        __syncthreads();
        for (int i = tid; i < nloc; i += kCT) {
          double s = ws[i];
          const double *v = V + r0 + i;
          for (int k0 = 0; k0 < jp1; k0 += 8) {
            double t[8];
            upto8(jp1 - k0, [&](int c) { t[c] = v[(size_t)(k0 + c) * nmax]; });
            upto8(jp1 - k0, [&](int c) { s = fma(-t[c], sd[k0 + c], s); });
          }
          ws[i] = s;
        }
        // ---- V^T w over rows > j, ||w_{j+1:}||^2; the first rows of w and row j + 1 of V to all CTAs
        sums(jp1, jp1 + 1, jp1, r0, nloc);
        if (rank == 0)
          for (int e = tid; e < (jp1 + 1) * C; e += kCT) {
            const int k = e / C, r = e % C;
            *cl.map_shared_rank(&xw[buf][k], r) = k < n ? ws[k] : 0.0;
            *cl.map_shared_rank(&xv[buf][k], r) = k < jp1 && jp1 < n ? V[(size_t)k * nmax + jp1] : 0.0;
          }
        cl.sync();
        // ---- the new reflector, T's column, c = T_{j+1} rho, Givens
        for (int k = tid - 32; k >= 0 && k < jp1; k += kCT) {
          ss[k] = total(k);
          srho[k] = xv[buf][k];
          sh[k] = xw[buf][k];
        }
        if (tid == 0) {
          const double nrm2 = jp1 < n ? total(jp1) : 0.0;
          const double wn = sqrt(nrm2);
          const double wj1 = jp1 < n ? xw[buf][jp1] : 0.0;
          const double dd = mysgn(wj1) * wn;
          const double alpha = sqrt(2.0 * (nrm2 + fabs(wj1) * wn));
          s_dd = dd;
          s_ia = alpha > 0.0 ? 1.0 / alpha : 0.0;
          srho[jp1] = (wj1 + dd) * s_ia;
        }
        buf ^= 1;
        __syncthreads();
        if (tid < jp1) sd[tid] = (ss[tid] + s_dd * srho[tid]) * s_ia;
        __syncthreads();
        for (int e = tid; e < 4 * ((jp1 + 7) & ~7); e += kCT) {
          const int k = e >> 2;
          double t = 0.0;
          if (k < jp1)
            for (int l = k + (e & 3); l < jp1; l += 4) t = fma(Tm[k + l * ld], sd[l], t);
          t += __shfl_xor_sync(0xffffffffu, t, 1);
          t += __shfl_xor_sync(0xffffffffu, t, 2);
          if (k < jp1 && (e & 3) == 0) Tm[k + jp1 * ld] = -2.0 * t;
        }
        // (the rotations meanwhile, in a warp that has no entry: at most 66 x 4 threads have)
        if (tid == kCT - 1) {
          Tm[jp1 + jp1 * ld] = 2.0;
          const double dd = s_dd;
          double *Rj = Rm + (size_t)j * ld;
          double a0 = sh[0];
          for (int k = 0; k < j; ++k) {
            const double a1 = sh[k + 1], c = scs[k], s = ssn[k];
            Rj[k] = c * a0 + s * a1;
            a0 = -s * a0 + c * a1;
          }
          double cg_, sn;
          givens_rot(a0, -dd, 4.9406564584124654e-324, &cg_, &sn);
          scs[j] = cg_;
          ssn[j] = sn;
          Rj[j] = cg_ * a0 - sn * dd;
          const double gj = sg[j];
          sg[jp1] = -sn * gj;
          sg[j] = cg_ * gj;
          const double resid = fabs(sg[jp1]);
          // a column that is not finite, or that the least squares cannot divide by,
          // ends the solve; the update takes the columns before it
          const bool bad = !(resid == resid) || !(fabs(Rj[j]) > 0.0);
          s_step = bad ? j : jp1;
          if (bad || resid < s_rtol || j == m - 1) {
            s_live = 0;
            s_conv = bad ? -1 : resid < s_rtol ? 1 : 0;
          }
        }
        __syncthreads();
        if (!s_live) break;  // the same for the whole cluster
        for (int e = tid; e < 4 * ((jp1 + 1 + 7) & ~7); e += kCT) {
          const int k = e >> 2;
          double t = 0.0;
          if (k <= jp1)
            for (int l = k + (e & 3); l <= jp1; l += 4) t = fma(Tm[k + l * ld], srho[l], t);
          t += __shfl_xor_sync(0xffffffffu, t, 1);
          t += __shfl_xor_sync(0xffffffffu, t, 2);
          if (k <= jp1 && (e & 3) == 0) sc[k] = t;
        }
        __syncthreads();
        // ---- v_{j+1} and q_{j+1} = e_{j+1} - V_{j+1} c
        {
          const double dd = s_dd, ia = s_ia, cj = sc[jp1];
          for (int i = tid; i < nloc; i += kCT) {
            const int r = r0 + i;
            const double wi = ws[i];
            const double vi = r > j ? (r == jp1 ? wi + dd : wi) * ia : 0.0;
            double *v = V + r;
            double acc = (r == jp1 ? 1.0 : 0.0) - vi * cj;
            for (int k0 = 0; k0 < jp1; k0 += 8) {
              double t[8];
              upto8(jp1 - k0, [&](int c) { t[c] = v[(size_t)(k0 + c) * nmax]; });
              upto8(jp1 - k0, [&](int c) { acc = fma(-t[c], sc[k0 + c], acc); });
            }
            v[(size_t)jp1 * nmax] = vi;
            Q[r] = (FT)acc;
          }
        }
      }
      // ---- least squares R y = g (a lane a row, the columns from the last), x += Z y
      const int ns = s_step;
      __syncthreads();
      if (warp == 0) {
        for (int i = lane; i < ns; i += 32) sd[i] = sg[i] / Rm[i + i * ld];
        __syncwarp();
        for (int jj = ns - 1; jj > 0; --jj) {
          const double yj = sd[jj];
          for (int i = lane; i < jj; i += 32) sd[i] = sd[i] - Rm[i + jj * ld] * yj / Rm[i + i * ld];
          __syncwarp();
        }
      }
      __syncthreads();
      for (int i = tid; i < nloc; i += kCT) {
        double s = x[r0 + i];
        const FT *z = Z + r0 + i;
        for (int k0 = 0; k0 < ns; k0 += 8) {
          FT t[8];
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (k0 + c < ns) t[c] = __ldcg(z + (size_t)(k0 + c) * nmax);
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (k0 + c < ns) s = fma(to_f64(t[c]), sd[k0 + c], s);
        }
        x[r0 + i] = s;
      }
      iters += ns;
      conv = s_conv;
      cl.sync();  // x is read across the cluster's rows, sd and s_conv are written again
      if (conv) break;
    }
    if (rank == 0 && tid == 0) {
      P.iters[sys * P.nrhs + rhs] = iters;
      P.conv[sys * P.nrhs + rhs] = conv > 0;
    }
  }
  cl.sync();  // no CTA leaves while another may still write to it
}

template <typename FT, int K>
int launch_t(cudaStream_t s, const CBatch &P, int clusters, int *room) {
  const auto fn = k_batch_cluster<FT, K>;
  static PerDevice limits;
  if (!limits.done([&] {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCSmemMax) == cudaSuccess;
      }))
    return DEV_ERR_UNKNOWN;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * P.C));
  cfg.blockDim = dim3(kCT);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)P.C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = P.C > 1 ? 1 : 0;
  if (room) {
    *room = num_sms();
    if (P.C > 1 && cudaOccupancyMaxActiveClusters(room, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      *room = 0;
    }
    return 0;
  }
  return cudaLaunchKernelEx(&cfg, fn, P) == cudaSuccess ? 0 : DEV_ERR_UNKNOWN;
}

}  // namespace

size_t batch_cluster_smem(size_t slot_bytes, int nmax, int m, int C, int *rbmax) {
  const int rb = std::max(((nmax + C - 1) / C + 31) / 32 * 32, (m + 2 + 31) / 32 * 32);
  *rbmax = rb;
  return slot_bytes + 8 * ((size_t)rb + 2 * (size_t)(m + 2) * (m + 2));
}
size_t batch_cluster_smem_max() { return kCSmemMax; }

int launch_batch_cluster(cudaStream_t s, const CBatch &P, int clusters, int *room) {
  if (P.f32) return P.K == 2 ? launch_t<float, 2>(s, P, clusters, room) : launch_t<float, 4>(s, P, clusters, room);
  return P.K == 2 ? launch_t<double, 2>(s, P, clusters, room) : launch_t<double, 4>(s, P, clusters, room);
}

}  // namespace lace
