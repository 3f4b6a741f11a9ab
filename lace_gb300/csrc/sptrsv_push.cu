// SpTRSV of any sparse triangle that fits one thread-block cluster: rows push
// their values to the rows that wait for them.
//
// Rows are taken in level order, 32 at a time (a group: a lane each; 32 / BS
// block rows of BS lanes each for blocked factors), and every off-diagonal
// entry has a slot of its own in the shared memory of the CTA that solves its
// row.  A solved row is written straight into the slots of its entries - its
// own CTA's shared memory or, over the cluster, another's - and a slot is its
// own ready flag (the unsolved mark, as in the other sync-free solves), so a
// level of the wavefront costs one store into shared memory, near or far, the
// poll that sees it and the multiply-adds; nothing on the chain reads global
// memory, and there is no barrier between levels.  A group's entries, slots and
// destinations are loaded while its warp still waits for the entries to fill.
//
// A warp takes its groups in level order, so the lowest unsolved group can
// always proceed.  The groups of a level go to the CTAs in stretches, so that
// neighbouring rows, and most pushes, stay in one CTA.
//
// Bound: the number of levels times the hand-over between SMs, about 0.2 us.
// Pairs of triangles, the block-scheduled solves' time first: 48^3 in level
// order, FP32, 325 -> 66 us; 66^3 422 -> 85; 30^3 198 -> 38; 32^3 blocks of 5 x 5
// 192 -> 65.  The schedule is tuned by time, and this one is a candidate
// wherever no row has more than eight entries or dependants (four in blocked
// factors) and the slots fit: about 290,000 rows of a 7-point stencil in FP32.
#include <algorithm>

#include <cooperative_groups.h>

#include "context.h"
#include "perdevice.h"
#include "push.cuh"

namespace lace {

namespace {

constexpr size_t kPushSmemMax = 220 * 1024;

struct PushArgs {
  const int *wptr;  // groups of each warp of the cluster
  const int *slot;  // per group: its first slot row (a row: 32 slots)
  const int *rc;    // per group and row: row | entries << 27, -1: none
  const int *dst;   // per group, dependant and row
  const void *val, *rd;  // CT, per group, entry (component) and lane
  const void *b;
  void *x;
  int in_f32, out_f32, early;
  unsigned fill;  // 16-byte words of a CTA's slots
  const int *done;
  int *status;
};

// a group's entries and destinations, loaded one group ahead
template <typename CT, int BS, int K, bool UNIT>
struct PushRec {
  int slot, rc, dst[K];
  CT v[K][BS], d[BS];
  __device__ __forceinline__ void load(const PushArgs &A, int g, int lane) {
    constexpr int RPG = 32 / BS;
    const int r = lane / BS;
    const bool on = lane < RPG * BS;
    slot = A.slot[g];
    rc = on ? A.rc[(size_t)g * RPG + r] : -1;
#pragma unroll
    for (int t = 0; t < K; ++t) {
      dst[t] = on ? A.dst[((size_t)g * K + t) * RPG + r] : -1;
#pragma unroll
      for (int e = 0; e < BS; ++e) v[t][e] = ((const CT *)A.val)[(((size_t)g * K + t) * BS + e) * 32 + lane];
    }
#pragma unroll
    for (int e = 0; e < BS; ++e) d[e] = UNIT ? (CT)1 : ((const CT *)A.rd)[((size_t)g * BS + e) * 32 + lane];
  }
};

template <typename CT, int BS, int K, bool UNIT>
__global__ void __launch_bounds__(32 * kPushW, 1) k_sptrsv_push(PushArgs A) {
  extern __shared__ __align__(16) unsigned char smem_p[];
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem_p);
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, comp = lane % BS;
  constexpr bool kAhead = K * BS * sizeof(CT) <= 96;  // registers for two groups
  // the second triangle of a pair starts under the first one's solve; what it
  // reads of earlier kernels is in place (the first one waited for them)
  if (!A.early) asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (A.done != nullptr && *(volatile const int *)A.done) {  // the same for every CTA
    if (A.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  const int gb = A.wptr[rank * kPushW + warp], ge = A.wptr[rank * kPushW + warp + 1];
  // slot row 0 stays 0: the slots of the entries a row does not have
  for (unsigned k = threadIdx.x; k < A.fill; k += 32 * kPushW) {
    const unsigned m = k < 2 * sizeof(CT) ? 0u : 0xffffffffu;
    reinterpret_cast<uint4 *>(smem_p)[k] = make_uint4(m, m, m, m);
  }
  using Rec = PushRec<CT, BS, K, UNIT>;
  Rec cur, nxt;
  if (gb < ge) cur.load(A, gb, lane);
  cl.sync();  // every slot of the cluster is unsolved
  if (A.early) asm volatile("griddepcontrol.wait;" ::: "memory");
  bool gave_up = false;
  for (int g = gb; g < ge; ++g) {
    const int row = cur.rc < 0 ? -1 : (cur.rc & 0x7ffffff) * BS + comp, cnt = cur.rc < 0 ? 0 : cur.rc >> 27;
    CT rhs = (CT)0;
    if (row >= 0) rhs = A.in_f32 ? (CT)((const float *)A.b)[row] : (CT)((const double *)A.b)[row];
    if (kAhead && g + 1 < ge) nxt.load(A, g + 1, lane);
    Slot dst[K];
    unsigned a[K];
#pragma unroll
    for (int t = 0; t < K; ++t) {
      dst[t] = slot_of(base + comp * (unsigned)sizeof(CT), rank, cur.dst[t]);
      a[t] = base + (unsigned)(((t < cnt ? cur.slot + t : 0) * 32 + lane) * (int)sizeof(CT));
    }
    if (BS == 1 && !UNIT) rhs *= cur.d[0];
    // The wait: nothing in the loop but the loads, their test and a count (with
    // the sums and the limit's tests inside, a poll took 0.13 us and a level of
    // a 64 x 64 grid 0.27 us).
    CT s[K];
    for (int polls = 0;;) {
      bool ok = false;
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // four polls between the limit's tests
        unsigned m = 0;
#pragma unroll
        for (int t = 0; t < K; ++t) {
          s[t] = ld_slot(a[t], (CT)0);
          m = max(m, head(s[t]));
        }
        ok = __all_sync(0xffffffffu, m != 0xffffffffu);
        if (ok) break;
      }
      if (ok || gave_up) break;
      polls += 4;
      if ((polls & 1023) == 0) {
        if (polls > kMaxSpins && lane == 0) atomicOr(A.status, kStatusSpinTimeout);  // the solve is reported as failed
        gave_up = __any_sync(0xffffffffu, polls > kMaxSpins || (*(const volatile int *)A.status & kStatusSpinTimeout));
      }
    }
    CT x = rhs;
    if (BS == 1) {
#pragma unroll
      for (int t = 0; t < K; ++t) x = fma(-cur.v[t][0], s[t], x);
    } else {
      const int l0 = lane - comp;
#pragma unroll
      for (int t = 0; t < K; ++t) {
        CT p = (CT)0;
#pragma unroll
        for (int e = 0; e < BS; ++e) p = fma(cur.v[t][e], __shfl_sync(0xffffffffu, s[t], (l0 + e) & 31), p);
        x -= p;
      }
      if (!UNIT) {
        CT p = (CT)0;
#pragma unroll
        for (int e = 0; e < BS; ++e) p = fma(cur.d[e], __shfl_sync(0xffffffffu, x, (l0 + e) & 31), p);
        x = p;
      }
    }
    if (head(x) == 0xffffffffu) x = (CT)NAN;  // a solved value never carries the mark
#pragma unroll
    for (int t = 0; t < K; ++t) push(dst[t], x);
    if (row >= 0) {
      if (A.out_f32) ((float *)A.x)[row] = (float)x;
      else ((double *)A.x)[row] = (double)x;
    }
    if (kAhead) cur = nxt;
    else if (g + 1 < ge) cur.load(A, g + 1, lane);
  }
  cl.sync();  // no CTA leaves while another may still write to it
}

// a plan's values from the triangle's: the entries scaled by the reciprocal
// diagonal (a blocked triangle's as they are, its inverse diagonal blocks in rd)
template <typename VT, typename CT>
__global__ void k_push_values(int lanes, int bs, int K, int unit, const int *__restrict__ map,
                              const int *__restrict__ dmap, const VT *__restrict__ val, const VT *__restrict__ dinv,
                              CT *__restrict__ out, CT *__restrict__ rd) {
  const int RPG = 32 / bs, LD = bs * bs;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < lanes; q += gridDim.x * blockDim.x) {
    const int g = q >> 5, lane = q & 31, r = lane / bs, c = lane % bs;
    const bool on = lane < RPG * bs;
    const int dm = on ? dmap[(size_t)g * RPG + r] : -1;
    CT f = (CT)1;
    if (!unit)
      for (int e = 0; e < bs; ++e) {
        const CT w = dm < 0 ? (CT)0 : bs == 1 ? (CT)1 / cvt<CT>(val[dm]) : cvt<CT>(dinv[(size_t)dm * LD + c * bs + e]);
        rd[((size_t)g * bs + e) * 32 + lane] = w;
        if (bs == 1) f = w;
      }
    for (int t = 0; t < K; ++t) {
      const int m = on ? map[((size_t)g * K + t) * RPG + r] : -1;
      for (int e = 0; e < bs; ++e)
        out[(((size_t)g * K + t) * bs + e) * 32 + lane] = m < 0 ? (CT)0 : cvt<CT>(val[(size_t)m * LD + c * bs + e]) * f;
    }
  }
}

// launches the solve, or with clusters set asks how many of its clusters the device holds
template <typename CT, int BS, int K, bool UNIT>
int launch_t(cudaStream_t s, const PushPlan &p, const PushArgs &a, int *clusters) {
  const auto fn = k_sptrsv_push<CT, BS, K, UNIT>;
  static PerDevice limits;
  if (!limits.done([&] {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPushSmemMax) == cudaSuccess &&
               cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
      }))
    return DEV_ERR_UNKNOWN;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.C);
  cfg.blockDim = dim3(32 * kPushW);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)p.C;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = p.C > 1 ? 2 : 1;
  if (clusters) {
    *clusters = 1;
    if (p.C > 1 && cudaOccupancyMaxActiveClusters(clusters, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      *clusters = 0;
    }
    return 0;
  }
  return cudaLaunchKernelEx(&cfg, fn, a) == cudaSuccess ? 0 : DEV_ERR_UNKNOWN;
}

template <typename CT, int BS, int K>
int launch_u(cudaStream_t s, const PushPlan &p, const PushArgs &a, int *clusters) {
  return p.unit ? launch_t<CT, BS, K, true>(s, p, a, clusters) : launch_t<CT, BS, K, false>(s, p, a, clusters);
}

template <typename CT, int BS>
int launch_k(cudaStream_t s, const PushPlan &p, const PushArgs &a, int *clusters) {
  if constexpr (BS == 1)
    if (p.K == 8) return launch_u<CT, 1, 8>(s, p, a, clusters);
  return p.K == 3 ? launch_u<CT, BS, 3>(s, p, a, clusters) : launch_u<CT, BS, 4>(s, p, a, clusters);
}

template <typename CT>
int launch_ct(cudaStream_t s, const PushPlan &p, const PushArgs &a, int *clusters) {
  switch (p.bs) {
    case 1: return launch_k<CT, 1>(s, p, a, clusters);
    case 2: return launch_k<CT, 2>(s, p, a, clusters);
    case 3: return launch_k<CT, 3>(s, p, a, clusters);
    case 4: return launch_k<CT, 4>(s, p, a, clusters);
    case 5: return launch_k<CT, 5>(s, p, a, clusters);
    case 6: return launch_k<CT, 6>(s, p, a, clusters);
    case 7: return launch_k<CT, 7>(s, p, a, clusters);
    default: return launch_k<CT, 8>(s, p, a, clusters);
  }
}

}  // namespace

// Rows by level, groups by CTA and warp, slots and destinations: 0, or 1 where
// the triangle does not fit C CTAs, 2 where it fits no number of them.
int push_plan_host(const Pattern &T, bool lower, int bs, size_t ct, int C, PushHost &h) {
  const int n = T.n, RPG = 32 / bs, LD = bs * bs;
  if ((long long)((int)T.idx.size() - n) * bs * (long long)ct > (long long)C * (long long)kPushSmemMax) return 1;
  std::vector<int> lev(n), out(n, 0);
  int depth = 0, deg = 0;
  for (int k = 0; k < n; ++k) {
    const int i = lower ? k : n - 1 - k;
    int l = 0, c = 0;
    for (int e = T.ptr[i]; e < T.ptr[i + 1]; ++e) {
      const int j = T.idx[e];
      if (j == i) continue;
      l = std::max(l, lev[j] + 1);
      deg = std::max(deg, ++out[j]);
      ++c;
    }
    lev[i] = l;
    depth = std::max(depth, l + 1);
    deg = std::max(deg, c);
    if (deg > (bs == 1 ? 8 : 4) || n >= 1 << 27) return 2;
  }
  if (deg > h.K) h.K = deg <= 3 ? 3 : deg <= 4 ? 4 : 8;
  const int K = h.K;
  std::vector<int> lp(depth + 1, 0), rows(n);
  for (int i = 0; i < n; ++i) ++lp[lev[i] + 1];
  for (int l = 0; l < depth; ++l) lp[l + 1] += lp[l];
  std::vector<int> at(lp.begin(), lp.end() - 1);
  for (int k = 0; k < n; ++k) {
    const int i = lower ? k : n - 1 - k;
    rows[at[lev[i]]++] = i;
  }
  // groups: CTA, warp, first slot row, entries of the longest row
  struct G {
    int cta, warp, first, rows, slot, kin;
  };
  std::vector<G> gs;
  std::vector<int> taken(C, 0), srows(C, 1);  // slot row 0: zeros
  for (int l = 0; l < depth; ++l) {
    const int ng = (lp[l + 1] - lp[l] + RPG - 1) / RPG;
    for (int k = 0; k < ng; ++k) {
      G g;
      g.cta = (int)(((long long)k * C + l % C) / ng);  // stretches; the odd one out moves with the level
      g.warp = taken[g.cta]++ % kPushW;
      g.first = lp[l] + k * RPG;
      g.rows = std::min(RPG, lp[l + 1] - g.first);
      g.kin = 0;
      for (int r = 0; r < g.rows; ++r) g.kin = std::max(g.kin, T.ptr[rows[g.first + r] + 1] - T.ptr[rows[g.first + r]] - 1);
      g.slot = srows[g.cta];
      srows[g.cta] += g.kin;
      gs.push_back(g);
    }
  }
  const int top = *std::max_element(srows.begin(), srows.end());
  if ((size_t)top * 32 * ct > kPushSmemMax) return 1;
  h.smem = (size_t)top * 32 * ct;
  h.groups = (int)gs.size();
  h.levels = depth;
  // warps' groups one after the other, in level order
  h.wptr.assign((size_t)C * kPushW + 1, 0);
  for (const G &g : gs) ++h.wptr[g.cta * kPushW + g.warp + 1];
  for (int w = 0; w < C * kPushW; ++w) h.wptr[w + 1] += h.wptr[w];
  std::vector<int> fill(h.wptr.begin(), h.wptr.end() - 1), pos(n), cta(n), slot(n);
  const size_t ng = gs.size();
  h.slot.resize(ng);
  h.rc.assign(ng * RPG, -1);
  h.dmap.assign(ng * RPG, -1);
  h.map.assign(ng * K * RPG, -1);
  h.dst.assign(ng * K * RPG, -1);
  for (const G &g : gs) {
    const int q = fill[g.cta * kPushW + g.warp]++;
    h.slot[q] = g.slot;
    for (int r = 0; r < g.rows; ++r) {
      const int i = rows[g.first + r];
      pos[i] = q * RPG + r;
      cta[i] = g.cta;
      slot[i] = g.slot * 32 + r * bs;
    }
  }
  std::fill(out.begin(), out.end(), 0);
  for (int i = 0; i < n; ++i) {
    const size_t q = pos[i] / RPG, r = pos[i] % RPG;
    int t = 0;
    for (int e = T.ptr[i]; e < T.ptr[i + 1]; ++e) {
      const int j = T.idx[e];
      if (j == i) {
        h.dmap[pos[i]] = bs == 1 ? e : i;
        continue;
      }
      const size_t u = out[j]++, qj = pos[j] / RPG, rj = pos[j] % RPG;
      h.map[(q * K + t) * RPG + r] = e;
      h.dst[(qj * K + u) * RPG + rj] = (cta[i] << 24) | (int)((slot[i] + t * 32) * ct);
      ++t;
    }
    h.rc[pos[i]] = i | t << 27;
  }
  return 0;
}

int push_plan_upload(cudaStream_t s, const PushHost &h, int bs, size_t ct, int C, bool unit, PushPlan &p) {
  p.valid = false;
  p.bs = bs;
  p.C = C;
  p.K = h.K;
  p.groups = h.groups;
  p.smem = h.smem;
  p.unit = unit ? 1 : 0;
  p.ct = ct;
  const size_t lanes = (size_t)h.groups * 32;
  auto up = [&](DBuf &d, const std::vector<int> &v) { return d.upload(v.data(), 4 * v.size(), s); };
  if (up(p.wptr, h.wptr) || up(p.slot, h.slot) || up(p.rc, h.rc) || up(p.dst, h.dst) || up(p.map, h.map) ||
      up(p.dmap, h.dmap) || p.val.ensure(ct * lanes * h.K * bs) || p.rd.ensure(ct * lanes * bs))
    return DEV_ERR_DEVICE_ALLOC;
  if (cudaStreamSynchronize(s) != cudaSuccess) return DEV_ERR_UNKNOWN;
  PushArgs a = {};
  int clusters = 0;
  const int rc = ct == 4 ? launch_ct<float>(s, p, a, &clusters) : launch_ct<double>(s, p, a, &clusters);
  if (rc) return rc;
  p.vals_version = -1;
  p.valid = clusters > 0;
  return 0;
}

void launch_push_values(cudaStream_t s, PushPlan &p, const void *val, const void *dinv, VType vt) {
  const int lanes = p.groups * 32, grid = std::max(1, std::min((lanes + 255) / 256, num_sms() * 8));
  const int *map = (const int *)p.map.p, *dmap = (const int *)p.dmap.p;
  switch (vt) {
    case VType::F64:
      k_push_values<double, double><<<grid, 256, 0, s>>>(lanes, p.bs, p.K, p.unit, map, dmap, (const double *)val,
                                                         (const double *)dinv, (double *)p.val.p, (double *)p.rd.p);
      break;
    case VType::F32:
      k_push_values<float, float><<<grid, 256, 0, s>>>(lanes, p.bs, p.K, p.unit, map, dmap, (const float *)val,
                                                       (const float *)dinv, (float *)p.val.p, (float *)p.rd.p);
      break;
    case VType::BF16:
      k_push_values<__nv_bfloat16, float><<<grid, 256, 0, s>>>(lanes, p.bs, p.K, p.unit, map, dmap,
                                                               (const __nv_bfloat16 *)val, (const __nv_bfloat16 *)dinv,
                                                               (float *)p.val.p, (float *)p.rd.p);
      break;
  }
}

int launch_push(cudaStream_t s, const PushPlan &p, const void *b, int in_f32, void *x, int out_f32, int early,
                int *status, const int *done) {
  PushArgs a;
  a.wptr = (const int *)p.wptr.p;
  a.slot = (const int *)p.slot.p;
  a.rc = (const int *)p.rc.p;
  a.fill = (unsigned)(p.smem / 16);
  a.dst = (const int *)p.dst.p;
  a.val = p.val.p;
  a.rd = p.rd.p;
  a.b = b;
  a.x = x;
  a.in_f32 = in_f32;
  a.out_f32 = out_f32;
  a.early = early;
  a.done = done;
  a.status = status;
  return p.ct == 4 ? launch_ct<float>(s, p, a, nullptr) : launch_ct<double>(s, p, a, nullptr);
}

}  // namespace lace
