// Batched solves (lace_gpu_batch_*): many independent systems, several
// right-hand sides each.
//
// lace_gpu_batch_create assembles the systems into one block-diagonal CSR
// operator on the batch's context (so the context's pattern analysis builds
// the A-order ParILU records for all of them at once) and, per system, the
// level sets of its two triangles.  lace_gpu_batch_solve then runs the whole
// solve - every system's ParILU sweeps and FGMRES-Householder for every
// (system, rhs) pair - as one persistent launch, captured in a CUDA graph when
// the context's options ask for graphs: a cluster of CTAs per pair
// (batch_cluster.cu), or, where a system's triangles do not fit a cluster's
// shared memory or the jobs fill the chip anyway, a CTA per system and up to four
// of its right-hand sides (batch_persist.cu).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <atomic>
#include <numeric>
#include <thread>
#include <vector>

#include "context.h"

using namespace lace;

struct lace_gpu_batch {
  lace_gpu_ctx *ctx = nullptr;
  int nsys = 0, nrhs = 0, N = 0, nmax = 0;
  std::vector<int> n, row_off;
  DBuf dn, droff, lsys, lptr, lrows, usys, uptr, urows;  // per system and its levels
  DBuf cL, fL, cU, fU, dU;                               // level-ordered row records (columns, A positions)
  int w = 0;                                             // record width
  DBuf vrec;                                             // per CTA: the records' factor values
  DBuf jsys, jrhs, jnr;                                  // jobs: (system, first rhs, rhs count)
  int njobs = 0;
  size_t nnzmax = 0;                                     // the largest system's entries
  DBuf F;                                                // per CTA: factor values in A's order, twice
  DBuf V, W, Tm, Rm, Z, Q, Tt, ctl;                              // per-CTA workspace, queue and results
  int grid = 0, m = 0, f32 = -1;
  // the cluster form: the block-diagonal pattern, and per triangle (0 L, 1 U)
  // the systems' plans one after the other
  std::vector<int> hrow, hcol;
  int C = 0, K = 2, plan_ct = 0, plan_m = 0, clusters = 0, gmax[2] = {0, 0}, rbmax = 0;
  size_t slot_bytes = 0, csmem = 0;
  DBuf wptr[2], goff[2], pslot[2], rc[2], dst[2], map[2], dmap[2], cjsys, cjrhs, vals;
};

namespace {

constexpr int kSplitRows = 16384;  // single-CTA form: systems from here on give each right-hand side its own job

// levels of one triangle of system rows [r0, r0 + n) (global indices in
// the block-diagonal CSR): lower: a row's level is one more than the largest
// level of the columns left of it; upper: of the columns right of it.  Rows
// grouped by level in ascending order; ptr gets the level boundaries
// (relative to the concatenated rows), one entry per level start.
void levels(const std::vector<int> &row, const std::vector<int> &col, int r0, int n, bool lower,
            std::vector<int> &lev, std::vector<int> &ptr, std::vector<int> &rows) {
  int depth = 0;
  for (int k = 0; k < n; ++k) {
    const int i = lower ? r0 + k : r0 + n - 1 - k;
    int l = 0;
    for (int p = row[i]; p < row[i + 1]; ++p) {
      const int c = col[p];
      if (lower ? c < i : c > i) l = std::max(l, lev[c - r0] + 1);
    }
    lev[i - r0] = l;
    depth = std::max(depth, l + 1);
  }
  std::vector<int> cnt(depth + 1, 0);
  for (int k = 0; k < n; ++k) ++cnt[lev[k] + 1];
  for (int l = 0; l < depth; ++l) cnt[l + 1] += cnt[l];
  const int base = (int)rows.size();
  rows.resize(base + n);
  std::vector<int> fill(cnt.begin(), cnt.end() - 1);
  for (int k = 0; k < n; ++k) rows[base + fill[lev[k]]++] = r0 + k;  // ascending rows within a level
  for (int l = 0; l < depth; ++l) ptr.push_back(base + cnt[l]);
}

}  // namespace

extern "C" int lace_gpu_batch_create(lace_gpu_batch **out, lace_gpu_ctx *ctx, int nsys, const int *n,
                                     const int *row_off, const int *nnz_off, const int *row, const int *col,
                                     const double *val, int nrhs) {
  if (!out || !ctx || !n || !row_off || !nnz_off || !row || !col || !val) return set_err(DEV_ERR_INVALID_PTR);
  if (nsys < 1 || nrhs < 1 || nrhs > 64) return set_err(DEV_ERR_ILLEGAL_VALUE);
  cudaSetDevice(ctx->device);
  auto *B = new lace_gpu_batch();
  B->ctx = ctx;
  B->nsys = nsys;
  B->nrhs = nrhs;
  B->n.assign(n, n + nsys);
  B->row_off.assign(row_off, row_off + nsys);
  // block-diagonal S: system s occupies rows row_off[s] .. row_off[s]+n[s]
  int N = 0;
  for (int s = 0; s < nsys; ++s) {
    if (row_off[s] != N || n[s] < 1) {
      delete B;
      return set_err(DEV_ERR_ILLEGAL_VALUE);
    }
    N += n[s];
    B->nmax = std::max(B->nmax, n[s]);
  }
  B->N = N;
  std::vector<int> Sr(N + 1, 0);
  long long nnz = 0;
  for (int s = 0; s < nsys; ++s) nnz += row[row_off[s] + s + n[s]] - row[row_off[s] + s];
  if (nnz > 0x7fffffffLL) {
    delete B;
    return set_err(DEV_ERR_NOT_SUPPORTED);
  }
  std::vector<int> Sc(nnz);
  std::vector<double> Sv(nnz);
  long long p = 0;
  for (int s = 0; s < nsys; ++s) {
    // system s's row pointers are local, stored at row[row_off[s] + s .. + n[s]]
    const int *rp = row + row_off[s] + s;
    for (int i = 0; i < n[s]; ++i) {
      for (int e = rp[i]; e < rp[i + 1]; ++e) {
        const int c = col[nnz_off[s] + e];
        if (c < 0 || c >= n[s]) {
          delete B;
          return set_err(DEV_ERR_ILLEGAL_VALUE);
        }
        Sc[p] = c + row_off[s];
        Sv[p] = val[nnz_off[s] + e];
        ++p;
      }
      Sr[row_off[s] + i + 1] = (int)p;
    }
  }
  int rc = lace_gpu_upload_csr_host(ctx, N, (int)nnz, Sr.data(), Sc.data(), Sv.data());
  if (rc) {
    delete B;
    return rc;
  }
  // per system: the triangles' levels; the queue order, largest first
  std::vector<int> lev(B->nmax), lsys(nsys + 1), usys(nsys + 1), lptr, lrows, uptr, urows;
  lrows.reserve(N);
  urows.reserve(N);
  for (int s = 0; s < nsys; ++s) {
    lsys[s] = (int)lptr.size();
    levels(Sr, Sc, row_off[s], n[s], true, lev, lptr, lrows);
    usys[s] = (int)uptr.size();
    levels(Sr, Sc, row_off[s], n[s], false, lev, uptr, urows);
  }
  lsys[nsys] = (int)lptr.size();
  usys[nsys] = (int)uptr.size();
  lptr.push_back(N);
  uptr.push_back(N);
  // level-ordered records of the two triangles: for the k-th row of the
  // level order, its off-diagonal entries' local columns and A positions
  // (W of them, -1 beyond the row's count) and, for U, its diagonal's position
  std::vector<int> dpos_row(N), sys_of(N);
  int W = 0;
  for (int s = 0; s < nsys; ++s)
    for (int i = row_off[s]; i < row_off[s] + n[s]; ++i) {
      sys_of[i] = s;
      int d = -1;
      for (int q = Sr[i]; q < Sr[i + 1]; ++q)
        if (Sc[q] == i) d = q;
      if (d < 0) {  // the upload checked this already
        delete B;
        return set_err(DEV_ERR_NOT_SUPPORTED);
      }
      dpos_row[i] = d;
      W = std::max(W, std::max(d - Sr[i], Sr[i + 1] - d - 1));
    }
  if (W > kBatchMaxW) {
    delete B;
    return set_err(DEV_ERR_NOT_SUPPORTED);
  }
  W = std::max(W, 1);
  B->w = W;
  std::vector<int> cLh((size_t)N * W, -1), fLh((size_t)N * W, -1), cUh((size_t)N * W, -1), fUh((size_t)N * W, -1),
      dUh(N);
  for (int k = 0; k < N; ++k) {
    const int gl = lrows[k], gu = urows[k];
    const int rl = row_off[sys_of[gl]], ru = row_off[sys_of[gu]];
    for (int q = Sr[gl], w = 0; q < dpos_row[gl]; ++q, ++w) {
      cLh[(size_t)k * W + w] = Sc[q] - rl;
      fLh[(size_t)k * W + w] = q;
    }
    for (int q = dpos_row[gu] + 1, w = 0; q < Sr[gu + 1]; ++q, ++w) {
      cUh[(size_t)k * W + w] = Sc[q] - ru;
      fUh[(size_t)k * W + w] = q;
    }
    dUh[k] = dpos_row[gu];
  }
  // jobs, largest systems first: a system of at least kSplitRows rows gives
  // each right-hand side its own job (its FGMRES processes run on different
  // SMs: the longest of them sets the launch's time), a smaller one takes its
  // right-hand sides in groups of up to four (the operator, factor and
  // level-barrier work shared)
  std::vector<int> order(nsys);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return n[a] > n[b]; });
  std::vector<int> jsys, jrhs, jnr;
  const int R = batch_persist_rhs();
  for (int s : order) {
    const int g = n[s] >= kSplitRows ? 1 : R;
    for (int r = 0; r < nrhs; r += g) {
      jsys.push_back(s);
      jrhs.push_back(r);
      jnr.push_back(std::min(g, nrhs - r));
    }
    B->nnzmax = std::max(B->nnzmax, (size_t)(Sr[row_off[s] + n[s]] - Sr[row_off[s]]));
  }
  B->njobs = (int)jsys.size();
  cudaStream_t st = ctx->stream;
  if (B->dn.upload(n, 4 * (size_t)nsys, st) || B->droff.upload(row_off, 4 * (size_t)nsys, st) ||
      B->jsys.upload(jsys.data(), 4 * jsys.size(), st) || B->jrhs.upload(jrhs.data(), 4 * jrhs.size(), st) ||
      B->jnr.upload(jnr.data(), 4 * jnr.size(), st) || B->lsys.upload(lsys.data(), 4 * lsys.size(), st) ||
      B->usys.upload(usys.data(), 4 * usys.size(), st) || B->lptr.upload(lptr.data(), 4 * lptr.size(), st) ||
      B->uptr.upload(uptr.data(), 4 * uptr.size(), st) || B->lrows.upload(lrows.data(), 4 * lrows.size(), st) ||
      B->urows.upload(urows.data(), 4 * urows.size(), st) || B->cL.upload(cLh.data(), 4 * cLh.size(), st) ||
      B->fL.upload(fLh.data(), 4 * fLh.size(), st) || B->cU.upload(cUh.data(), 4 * cUh.size(), st) ||
      B->fU.upload(fUh.data(), 4 * fUh.size(), st) || B->dU.upload(dUh.data(), 4 * dUh.size(), st)) {
    delete B;
    return set_err(DEV_ERR_DEVICE_ALLOC);
  }
  if (cudaStreamSynchronize(st) != cudaSuccess) {
    delete B;
    return set_err(DEV_ERR_UNKNOWN);
  }
  B->hrow = std::move(Sr);
  B->hcol = std::move(Sc);
  *out = B;
  return DEV_SUCCESS;
}

// CTAs per cluster (1, 2, 4, 8) by the time the queue takes: per search
// direction a job costs 26 ns a row divided over the CTAs (the FP64 units'
// share at 15 basis vectors), 0.18 us a level of its triangles and 10 us of
// barriers and small matrices (all measured), and a grid's directions grow with
// its side; the clusters side by side take the jobs' sum, and none less than
// the largest job.  24 systems of up to 9,025 rows, four right-hand sides: C = 1,
// 2, 4, 8 at 93, 45, 37 and 75 ms.
static double cluster_cost(const lace_gpu_batch *B, const std::vector<int> &levels, int C) {
  double sum = 0.0, top = 0.0;
  for (int s = 0; s < B->nsys; ++s) {
    const double t = std::sqrt((double)B->n[s]) * (0.026 * B->n[s] / C + 0.18 * levels[s] + 10.0);
    sum += t * B->nrhs;
    top = std::max(top, t);
  }
  return std::max(top, sum / std::max(1, num_sms() / C));
}

// The same of the single-CTA form: per direction 16.5 ns a row and right-hand
// side and 0.72 us a level, its right-hand sides in lockstep, one job an SM.  It
// stays the better one where the jobs fill the chip (a level's barrier serves four
// right-hand sides): 256 systems of 1,024 to 65,536 rows, four right-hand sides,
// 3.6 s against 5.2 on clusters; the 24 systems above 264 ms against 37.
static double persist_cost(const lace_gpu_batch *B, const std::vector<int> &levels) {
  double sum = 0.0, top = 0.0;
  for (int s = 0; s < B->nsys; ++s) {
    const int g = B->n[s] >= kSplitRows ? 1 : batch_persist_rhs();
    for (int r = 0; r < B->nrhs; r += g) {
      const double t =
          std::sqrt((double)B->n[s]) * (0.0165 * B->n[s] * std::min(g, B->nrhs - r) + 0.72 * levels[s] + 10.0);
      sum += t;
      top = std::max(top, t);
    }
  }
  return std::max(top, sum / std::max(1, num_sms()));
}

// The cluster form's plans for value size ct and m directions (C = 0: the
// batch does not fit it, or the single-CTA form is the better one).
static int cluster_plan(lace_gpu_batch *B, int m, size_t ct) {
  if (B->plan_ct == (int)ct && B->plan_m == m) return 0;
  B->C = 0;
  B->plan_ct = 0;
  lace_gpu_ctx *c = B->ctx;
  const int nsys = B->nsys;
  // the triangles of each system and their entries' positions in A
  struct Sys {
    Pattern T[2];
    std::vector<int> pos[2];
    PushHost h[2];
    int levels = 0, fit = 0;
  };
  std::vector<Sys> S(nsys);
  auto parallel = [&](auto fn) {
    std::atomic<int> next{0};
    auto work = [&] {
      for (int s; (s = next.fetch_add(1)) < nsys;) fn(s);
    };
    std::vector<std::thread> th;
    const int k = std::min(nsys, std::max(1, std::min(16, (int)std::thread::hardware_concurrency())));
    for (int i = 1; i < k; ++i) th.emplace_back(work);
    work();
    for (auto &x : th) x.join();
  };
  parallel([&](int s) {
    const int n = B->n[s], r0 = B->row_off[s];
    for (int up = 0; up < 2; ++up) {
      Pattern &T = S[s].T[up];
      T.n = n;
      T.ptr.assign(1, 0);
      for (int i = 0; i < n; ++i) {
        for (int p = B->hrow[r0 + i]; p < B->hrow[r0 + i + 1]; ++p) {
          const int j = B->hcol[p] - r0;
          if (up ? j < i : j > i) continue;
          T.idx.push_back(j);
          S[s].pos[up].push_back(p);
        }
        T.ptr.push_back((int)T.idx.size());
      }
      std::vector<int> lev(n, 0);
      int d = 0;
      for (int k = 0; k < n; ++k) {
        const int i = up ? n - 1 - k : k;
        for (int e = T.ptr[i]; e < T.ptr[i + 1]; ++e)
          if (T.idx[e] != i) lev[i] = std::max(lev[i], lev[T.idx[e]] + 1);
        d = std::max(d, lev[i] + 1);
      }
      S[s].levels += d;
    }
  });
  std::vector<int> levels(nsys);
  for (int s = 0; s < nsys; ++s) levels[s] = S[s].levels;
  std::vector<int> order{1, 2, 4, 8};
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return cluster_cost(B, levels, a) < cluster_cost(B, levels, b); });
  const double other = persist_cost(B, levels);
  for (int C : order) {
    if (cluster_cost(B, levels, C) >= other) break;
    int rb = 0;
    const size_t rest = batch_cluster_smem(0, B->nmax, m, C, &rb);
    if (rest + 1024 > batch_cluster_smem_max()) continue;
    const size_t cap = batch_cluster_smem_max() - rest;
    size_t most = 0;  // slots of the largest triangle, without the groups' padding
    for (auto &y : S)
      for (auto &T : y.T) most = std::max(most, T.idx.size() - (size_t)T.n);
    if (most * ct > cap * C) continue;
    int K = 2;
    for (bool again = true; again;) {
      again = false;
      parallel([&](int s) {
        // the fewest CTAs that hold the slots of both triangles
        Sys &y = S[s];
        y.fit = 0;
        for (int ctas = 1; ctas <= C && !y.fit; ctas *= 2) {
          int no = 0;
          for (int up = 0; up < 2 && !no; ++up) {
            y.h[up] = PushHost();
            y.h[up].K = K;
            no = push_plan_host(y.T[up], up == 0, 1, ct, ctas, y.h[up]);
            if (!no && y.h[up].smem > cap) no = 1;
          }
          if (!no) y.fit = ctas;
          if (no == 2) break;
        }
      });
      int kmax = K;
      for (auto &y : S)
        if (y.fit) kmax = std::max({kmax, y.h[0].K, y.h[1].K});
      if (kmax > 4) return 0;
      if (kmax > K) {
        K = 4;
        again = true;
      }
    }
    bool fit = true;
    for (auto &y : S) fit = fit && y.fit;
    if (!fit) continue;
    B->slot_bytes = 256;
    for (int up = 0; up < 2; ++up) {
      std::vector<int> wptr, goff, slot, rc, dst, map, dmap;
      B->gmax[up] = 0;
      for (int s = 0; s < nsys; ++s) {
        const PushHost &h = S[s].h[up];
        goff.push_back((int)slot.size());
        B->gmax[up] = std::max(B->gmax[up], h.groups);
        B->slot_bytes = std::max(B->slot_bytes, h.smem);
        wptr.insert(wptr.end(), h.wptr.begin(), h.wptr.end());
        wptr.resize((size_t)(s + 1) * (C * kPushW + 1), h.groups);  // CTAs without groups
        slot.insert(slot.end(), h.slot.begin(), h.slot.end());
        rc.insert(rc.end(), h.rc.begin(), h.rc.end());
        dst.insert(dst.end(), h.dst.begin(), h.dst.end());
        for (int e : h.map) map.push_back(e < 0 ? -1 : S[s].pos[up][e]);
        for (int e : h.dmap) dmap.push_back(e < 0 ? -1 : S[s].pos[up][e]);
      }
      auto send = [&](DBuf &d, const std::vector<int> &v) { return d.upload(v.data(), 4 * v.size(), c->stream); };
      if (send(B->wptr[up], wptr) || send(B->goff[up], goff) || send(B->pslot[up], slot) || send(B->rc[up], rc) ||
          send(B->dst[up], dst) || send(B->map[up], map) || send(B->dmap[up], dmap) ||
          cudaStreamSynchronize(c->stream) != cudaSuccess)
        return DEV_ERR_DEVICE_ALLOC;
    }
    // jobs, largest systems first
    std::vector<int> by(nsys), js, jr;
    std::iota(by.begin(), by.end(), 0);
    std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return B->n[a] > B->n[b]; });
    for (int s : by)
      for (int r = 0; r < B->nrhs; ++r) {
        js.push_back(s);
        jr.push_back(r);
      }
    if (B->cjsys.upload(js.data(), 4 * js.size(), c->stream) || B->cjrhs.upload(jr.data(), 4 * jr.size(), c->stream) ||
        cudaStreamSynchronize(c->stream) != cudaSuccess)
      return DEV_ERR_DEVICE_ALLOC;
    B->csmem = batch_cluster_smem(B->slot_bytes, B->nmax, m, C, &B->rbmax);
    B->K = K;
    CBatch P = {};
    P.C = C;
    P.K = K;
    P.f32 = ct == 4;
    P.smem = B->csmem;
    int room = 0;
    const int rc = launch_batch_cluster(c->stream, P, 1, &room);
    if (rc) return rc;
    if (room < 1) continue;
    B->clusters = std::max(1, std::min(nsys * B->nrhs, std::min(room, num_sms() / C)));
    B->C = C;
    break;
  }
  B->plan_ct = (int)ct;
  B->plan_m = m;
  return 0;
}

extern "C" int lace_gpu_batch_destroy(lace_gpu_batch *B) {
  if (B) {
    cudaSetDevice(B->ctx->device);
    cudaStreamSynchronize(B->ctx->stream);
  }
  delete B;
  return DEV_SUCCESS;
}

// the per-CTA workspace for search_max m: one CTA per SM (the kernel's
// register budget), at most one per system
static int batch_workspace(lace_gpu_batch *B, int m, bool f32) {
  if (m == B->m && (int)f32 == B->f32) return 0;
  B->m = 0;  // until all of it is there
  const int prc = cluster_plan(B, m, f32 ? 4 : 8);
  if (prc) return prc;
  if (B->C) {
    const size_t G = (size_t)B->clusters, nmax = (size_t)B->nmax, fb = f32 ? 4 : 8;
    int rc = 0;
    rc |= B->F.ensure(fb * G * 2 * (B->nnzmax + 4));
    rc |= B->vals.ensure(fb * G * 32 * ((size_t)(B->gmax[0] + B->gmax[1]) * B->K + B->gmax[1]));
    rc |= B->Z.ensure(fb * G * m * nmax);
    rc |= B->Q.ensure(fb * G * nmax);
    rc |= B->Tt.ensure(fb * G * nmax);
    rc |= B->ctl.ensure(4 * (2 + 2 * (size_t)B->nsys * B->nrhs));
    rc |= B->V.ensure(8 * G * (m + 1) * nmax);
    if (rc) return DEV_ERR_DEVICE_ALLOC;
    B->m = m;
    B->f32 = f32;
    return 0;
  }
  const int R = batch_persist_rhs();
  B->grid = std::max(1, std::min(B->njobs, num_sms()));
  const size_t G = (size_t)B->grid, nmax = (size_t)B->nmax, ld = (size_t)m + 2;
  const size_t fb = f32 ? 4 : 8;
  int rc = 0;
  rc |= B->F.ensure(fb * G * 2 * (B->nnzmax + 4));
  rc |= B->vrec.ensure(fb * G * (2 * (size_t)B->w + 1) * nmax);
  rc |= B->V.ensure(8 * G * R * (m + 1) * nmax);
  rc |= B->W.ensure(8 * G * R * nmax);
  rc |= B->Tm.ensure(8 * G * R * ld * ld);
  rc |= B->Rm.ensure(8 * G * R * ld * ld);
  rc |= B->Z.ensure(fb * G * R * m * nmax);
  rc |= B->Q.ensure(fb * G * R * nmax);
  rc |= B->Tt.ensure(fb * G * R * nmax);
  rc |= B->ctl.ensure(4 * (2 + 2 * (size_t)B->nsys * B->nrhs));
  if (rc) return DEV_ERR_DEVICE_ALLOC;
  B->m = m;
  B->f32 = f32;
  return 0;
}

extern "C" int lace_gpu_batch_solve(lace_gpu_batch *B, int sweeps, int search_max, int restart_max, double rtol,
                                    const double *b, double *x, int *iters_out) {
  if (!B || !b || !x) return set_err(DEV_ERR_INVALID_PTR);
  if (search_max < 1 || search_max > kBatchMaxM || sweeps < 0 || restart_max < 1)
    return set_err(DEV_ERR_NOT_SUPPORTED);
  lace_gpu_ctx *c = B->ctx;
  cudaSetDevice(c->device);
  if (c->opt.trsv_mode != LACE_TRSV_SYNCFREE) return set_err(DEV_ERR_NOT_SUPPORTED);
  if (!c->sweep_ao) return set_err(DEV_ERR_NOT_SUPPORTED);  // the A-order records
  const bool f32 = c->vtype() != VType::F64;
  int rc = batch_workspace(B, search_max, f32);
  if (rc) return set_err(rc);
  cudaStream_t s = c->stream;
  const size_t pairs = (size_t)B->nsys * B->nrhs;
  int *ctl = (int *)B->ctl.p;
  if (cudaMemsetAsync(ctl, 0, B->ctl.bytes, s) != cudaSuccess) return set_err(DEV_ERR_UNKNOWN);
  CBatch P = {};
  if (B->C) {
    P.nrhs = B->nrhs;
    P.m = search_max;
    P.restart_max = restart_max;
    P.sweeps = sweeps;
    P.N = B->N;
    P.njobs = (int)pairs;
    P.C = B->C;
    P.K = B->K;
    P.f32 = f32 ? 1 : 0;
    P.rtol = rtol;
    P.jsys = (const int *)B->cjsys.p;
    P.jrhs = (const int *)B->cjrhs.p;
    P.n = (const int *)B->dn.p;
    P.roff = (const int *)B->droff.p;
    P.Arow = (const int *)c->Arow.p;
    P.Acol = (const int *)c->Acol.p;
    P.Aval = (const double *)c->Aval.p;
    P.pptr = (const int *)c->sw_pptr.p;
    P.dpos = (const int *)c->sw_dpos.p;
    P.pairs = (const int2 *)c->sw_pairs.p;
    for (int up = 0; up < 2; ++up) {
      P.wptr[up] = (const int *)B->wptr[up].p;
      P.goff[up] = (const int *)B->goff[up].p;
      P.slot[up] = (const int *)B->pslot[up].p;
      P.rc[up] = (const int *)B->rc[up].p;
      P.dst[up] = (const int *)B->dst[up].p;
      P.map[up] = (const int *)B->map[up].p;
      P.dmap[up] = (const int *)B->dmap[up].p;
      P.gmax[up] = B->gmax[up];
    }
    P.vstride = 32 * ((size_t)(B->gmax[0] + B->gmax[1]) * B->K + B->gmax[1]);
    P.fstride = B->nnzmax + 4;
    P.nmax = (size_t)B->nmax;
    P.smem = B->csmem;
    P.slot_bytes = (unsigned)B->slot_bytes;
    P.rbmax = B->rbmax;
    P.V = (double *)B->V.p;
    P.F = B->F.p;
    P.val = B->vals.p;
    P.Z = B->Z.p;
    P.Q = B->Q.p;
    P.Tt = B->Tt.p;
    P.b = b;
    P.x = x;
    P.next = ctl;
    P.iters = ctl + 1;
    P.conv = ctl + 1 + pairs;
    P.status = ctl + 1 + 2 * pairs;
  }
  PBatchHost h;
  h.nsys = B->nsys;
  h.nrhs = B->nrhs;
  h.m = search_max;
  h.restart_max = restart_max;
  h.sweeps = sweeps;
  h.N = B->N;
  h.grid = B->grid;
  h.f32 = f32 ? 1 : 0;
  h.rtol = rtol;
  h.njobs = B->njobs;
  h.jsys = (const int *)B->jsys.p;
  h.jrhs = (const int *)B->jrhs.p;
  h.jnr = (const int *)B->jnr.p;
  h.n = (const int *)B->dn.p;
  h.roff = (const int *)B->droff.p;
  h.lsys = (const int *)B->lsys.p;
  h.usys = (const int *)B->usys.p;
  h.Arow = (const int *)c->Arow.p;
  h.Acol = (const int *)c->Acol.p;
  h.Aval = (const double *)c->Aval.p;
  h.pptr = (const int *)c->sw_pptr.p;
  h.dpos = (const int *)c->sw_dpos.p;
  h.diag = (const int *)c->sw_diag.p;
  h.pairs = (const int2 *)c->sw_pairs.p;
  h.F = B->F.p;
  h.fstride = B->nnzmax + 4;
  h.lptr = (const int *)B->lptr.p;
  h.w = B->w;
  h.cL = (const int *)B->cL.p;
  h.fL = (const int *)B->fL.p;
  h.cU = (const int *)B->cU.p;
  h.fU = (const int *)B->fU.p;
  h.dU = (const int *)B->dU.p;
  h.vrec = B->vrec.p;
  h.lrows = (const int *)B->lrows.p;
  h.uptr = (const int *)B->uptr.p;
  h.urows = (const int *)B->urows.p;
  h.b = b;
  h.x = x;
  h.nmax = (size_t)B->nmax;
  h.V = (double *)B->V.p;
  h.W = (double *)B->W.p;
  h.Tm = (double *)B->Tm.p;
  h.Rm = (double *)B->Rm.p;
  h.Z = B->Z.p;
  h.Q = B->Q.p;
  h.Tt = B->Tt.p;
  h.next = ctl;
  h.iters = ctl + 1;
  h.conv = ctl + 1 + pairs;
  cudaGraphExec_t ge = nullptr;
  if (c->opt.use_graph) {
    // the one launch, captured and replayed as a graph
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return set_err(DEV_ERR_UNKNOWN);
    rc = B->C ? launch_batch_cluster(s, P, B->clusters, nullptr) : launch_batch_persist(s, h);
    const cudaError_t ce = cudaStreamEndCapture(s, &g);
    if (rc || ce != cudaSuccess) return set_err(rc ? rc : DEV_ERR_UNKNOWN);
    const cudaError_t ie = cudaGraphInstantiate(&ge, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) return set_err(DEV_ERR_UNKNOWN);
    if (cudaGraphLaunch(ge, s) != cudaSuccess) {
      cudaGraphExecDestroy(ge);
      return set_err(DEV_ERR_UNKNOWN);
    }
  } else {
    rc = B->C ? launch_batch_cluster(s, P, B->clusters, nullptr) : launch_batch_persist(s, h);
    if (rc) return set_err(rc);
  }
  std::vector<int> res(2 * pairs + 1);
  const bool ok = cudaMemcpyAsync(res.data(), ctl + 1, 4 * res.size(), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
                  cudaStreamSynchronize(s) == cudaSuccess;
  if (ge) cudaGraphExecDestroy(ge);
  if (!ok) return set_err(DEV_ERR_UNKNOWN);
  if (res[2 * pairs] & kStatusSpinTimeout) return set_err(DEV_ERR_INTERNAL_LIMIT);
  bool all = true;
  for (size_t k = 0; k < pairs; ++k) {
    if (iters_out) iters_out[k] = res[k];
    all = all && res[pairs + k];
  }
  return all ? DEV_SUCCESS : DEV_NOTCONVERGED;
}
