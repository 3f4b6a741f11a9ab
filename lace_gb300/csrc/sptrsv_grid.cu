// SpTRSV on the factors of a lexicographic grid stencil (5-point in 2D,
// 7-point in 3D): the wavefront carried in registers.
//
// When every row of a triangle depends on exactly its existing neighbours at
// distances 1, nx and nx*ny (the pattern ILU(0) keeps of a 5- or 7-point
// stencil in natural order; checked on the device, entry by entry), the
// rows are a box of lines along x, and the solve is a wavefront over them.
// A warp takes a tile of 32 neighbouring lines, a lane each, and walks along x,
// each line one step behind the lines before it in y and in z: the neighbours a
// row needs are then values formed one step earlier by the lanes before it (a
// shuffle each), the neighbour in x is the lane's own register, and a step is
// three multiply-adds - no scan, no shared-memory or L2 round trip inside a
// tile, at any line length.  Only the tile's first lines in y and z need other
// tiles' results, four steps at a time, from face buffers whose entries are
// their own ready flags (the unsolved mark; the one consumer of an entry puts
// the mark back after reading it, so no fill pass is needed between solves).  A
// tile publishes its last lines in its own CTA's shared memory, in the next
// CTA's of its thread-block cluster, or through global memory, where helper
// warps of the receiving CTA poll for them and copy them on.  Clusters take
// their tiles by ticket in order, so a cluster only ever waits for tiles that
// running clusters hold.
//
// Factor values are kept in the order the lanes use them (per tile and block
// of four steps, one vector of four per lane and coefficient, scaled by the
// reciprocal diagonal) and arrive through a ring of cp.async stages, as does
// the vector between the two triangles (the same order; the upper triangle
// walks it backwards).  The right-hand side of the lower triangle and the
// solution of the upper one are in row order: a CTA stages its tiles' lines in
// shared memory, read and written a line at a time (lane by lane, row order
// costs 32 sectors an access, which bound the solve itself).
//
// Bound: the dependency chain, (nx + ny + nz) steps of a shuffle and dependent
// multiply-adds plus one hand-over per tile boundary.
#include <algorithm>
#include <type_traits>

#include <cooperative_groups.h>

#include "context.h"
#include "perdevice.h"

namespace lace {

namespace {

constexpr int kGW = 4;       // most warps (tiles) per CTA
constexpr int kGHelpers = 4;  // most helper warps per CTA

// blocks of four steps in flight per warp (a block takes 0.2 us in FP32, 0.7 us in FP64)
template <typename CT>
constexpr int kGD = sizeof(CT) == 4 ? 6 : 4;

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The unsolved mark of a face entry: for FP32 all ones (an FP32 operation
// that gives a NaN gives the canonical 0x7fffffff, and every published value
// comes out of a multiply-add); for FP64, whose NaNs keep their payloads, a
// signalling NaN, which no arithmetic instruction returns, told apart by its
// high word.
constexpr unsigned kMark32 = 0xffffffffu;
constexpr unsigned long long kMark64 = 0xfff7ffffffffffffull;
__device__ __forceinline__ bool unsolved(float v) { return __float_as_uint(v) == kMark32; }
__device__ __forceinline__ bool unsolved(double v) { return __double2hiint(v) == (int)(kMark64 >> 32); }
template <int N>
__device__ __forceinline__ bool any_unsolved(const float (&f)[N][4]) {
  unsigned m = 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    m = __vimax3_u32(m, __float_as_uint(f[k][0]), __float_as_uint(f[k][1]));
    m = __vimax3_u32(m, __float_as_uint(f[k][2]), __float_as_uint(f[k][3]));
  }
  return m == kMark32;
}
template <int N>
__device__ __forceinline__ bool any_unsolved(const double (&f)[N][4]) {
  bool w = false;
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int u = 0; u < 4; ++u) w |= unsolved(f[k][u]);
  return w;
}

// four entries at a shared-memory address, where p; v keeps its values otherwise
__device__ __forceinline__ void ld_face(int p, unsigned a, float (&v)[4]) {
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %4, 0; @q ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%5]; }"
               : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3])
               : "r"(p), "r"(a));
}
__device__ __forceinline__ void ld_face(int p, unsigned a, double (&v)[4]) {
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %4, 0; @q ld.volatile.shared.v2.f64 {%0, %1}, [%5]; "
               "@q ld.volatile.shared.v2.f64 {%2, %3}, [%5 + 16]; }"
               : "+d"(v[0]), "+d"(v[1]), "+d"(v[2]), "+d"(v[3])
               : "r"(p), "r"(a));
}
__device__ __forceinline__ void clear_face(int p, unsigned a, float) {
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %0, 0; @q st.volatile.shared.v4.u32 [%1], {%2, %2, %2, %2}; }" ::"r"(p),
               "r"(a), "r"(kMark32));
}
__device__ __forceinline__ void clear_face(int p, unsigned a, double) {
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %0, 0; @q st.volatile.shared.v2.u64 [%1], {%2, %2}; "
               "@q st.volatile.shared.v2.u64 [%1 + 16], {%2, %2}; }" ::"r"(p),
               "r"(a), "l"(kMark64));
}
// four solved entries for the next tile (shared or global memory), where p
__device__ __forceinline__ void publish(int p, float *d, const float (&v)[4]) {
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %0, 0; @q st.relaxed.gpu.v4.f32 [%1], {%2, %3, %4, %5}; }" ::"r"(p), "l"(d),
               "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
}
__device__ __forceinline__ void publish(int p, double *d, const double (&v)[4]) {
  asm volatile("{ .reg .pred q; setp.ne.s32 q, %0, 0; @q st.relaxed.gpu.v2.f64 [%1], {%2, %3}; "
               "@q st.relaxed.gpu.v2.f64 [%1 + 16], {%4, %5}; }" ::"r"(p), "l"(d), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]));
}
// global face entries, past the L1
__device__ __forceinline__ void ld_far(const float *p, float (&v)[4]) {
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "l"(p));
}
__device__ __forceinline__ void ld_far(const double *p, double (&v)[4]) {
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "l"(p + 2));
}
__device__ __forceinline__ void clear_far(float *p) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %1, %1, %1};" ::"l"(p), "r"(kMark32));
}
__device__ __forceinline__ void clear_far(double *p) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %1};" ::"l"(p), "l"(kMark64));
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %1};" ::"l"(p + 2), "l"(kMark64));
}
__device__ __forceinline__ void st_near(unsigned a, const float (&v)[4]) {
  asm volatile("st.volatile.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
}
__device__ __forceinline__ void st_near(unsigned a, const double (&v)[4]) {
  asm volatile("st.volatile.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]));
  asm volatile("st.volatile.shared.v2.f64 [%0], {%1, %2};" ::"r"(a + 16), "d"(v[2]), "d"(v[3]));
}

__global__ void k_fill_mark(void *p, int f32, size_t count) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < count; k += (size_t)gridDim.x * blockDim.x)
    if (f32) reinterpret_cast<unsigned *>(p)[k] = kMark32;
    else reinterpret_cast<unsigned long long *>(p)[k] = kMark64;
}

struct GridArgs {
  GridShape g;
  const void *coef;   // CT, see GridPlan
  void *face;         // CT, see GridPlan
  const void *b;      // right-hand side (lower: rows) and solution (upper: rows), else CT in tile order
  void *x;
  int rows_f32;       // the type of the rows: FP32, else FP64
  int early;          // the kernel before this one is the pair's first triangle
  int *tickets;
  int *dirty;         // set when a wait gave up: the faces may hold stale values
  const int *done;
  int *status;
};

// a wait that gives up: the solve is reported as failed, and so is every
// later one until the host has cleared the faces
__device__ __forceinline__ bool gave_up(int spins, int *status, int *dirty) {
  if (spins <= kMaxSpins && !((spins & 1023) == 1023 && (*(volatile const int *)status & kStatusSpinTimeout))) return false;
  atomicOr(status, kStatusSpinTimeout);
  atomicExch(dirty, 1);
  return true;
}

// The helper warps of a CTA: four lanes per face row that comes from another
// cluster, each copying every fourth block of the row from the global face
// buffer to the shared one as it is solved and marking it unsolved again
// behind it, so that the tiles' own warps only ever poll shared memory.
template <typename CT>
__device__ void grid_helper(const GridArgs &A, int sy_, int sz_, bool fary, bool farz, unsigned sface, int h,
                            bool lower, int Y0, int Z0, int rows) {
  const GridShape &g = A.g;
  const int LY = 1 << g.lyl, LZ = 32 >> g.lyl, T4 = 4 * g.nb, row = h >> 2;
  const bool isz = row >= g.wz * LZ;  // rows towards y first, then those towards z
  const int r = isz ? row - g.wz * LZ : row;
  const int wy = isz ? r / LY : 0, wz = isz ? 0 : r / LZ;
  const int ly = isz ? r % LY : 0, lz = isz ? 0 : r % LZ;
  const int ty = sy_ * g.wy + wy, tz = sz_ * g.wz + wz;
  const int yv = ty * LY + ly - Y0, zv = tz * LZ + lz - Z0;
  bool act = row < g.wz * LZ + (g.nz > 1 ? g.wy * LY : 0) && yv >= 0 && yv < g.ny && zv >= 0 && zv < g.nz;
  act = act && (isz ? farz && zv > 0 : fary && yv > 0);
  const int s = ly + lz + g.first(lower, ty, tz);
  int kb = (s >> 2) + (h & 3);
  const int ke = act ? (s + g.nx - 1) >> 2 : -1;
  const int frow = isz ? LZ + ly : lz;
  CT *src = (CT *)A.face + ((size_t)(tz * (g.sy * g.wy) + ty) * rows + frow) * T4;
  const unsigned dst = sface + (unsigned)(((wz * g.wy + wy) * rows + frow) * T4 * (int)sizeof(CT));
  for (int spins = 0; kb <= ke; ++spins) {
    CT v[4];
    ld_far(src + 4 * kb, v);
    // all four, on the line or not (see waits below)
    bool ok = true;
#pragma unroll
    for (int u = 0; u < 4; ++u) ok = ok && !unsolved(v[u]);
    if (ok) {
      st_near(dst + 4 * kb * (int)sizeof(CT), v);
      clear_far(src + 4 * kb);
      kb += 4;
      spins = 0;
    } else if (gave_up(spins, A.status, A.dirty)) {
      break;
    }
  }
}

// the coefficients and right-hand side of four steps, and the values of the
// neighbouring tiles, in the lanes that take them (0 in the others)
template <typename CT>
struct GridBlk {
  CT cx[4], cy[4], cz[4], v[4], f[2][4];
};

// a block of four steps in the row-order staging of a warp: 4 values a lane,
// and a pad that spreads a line's consecutive steps over all banks
constexpr int kGPad = 132;

// the ring of a warp: a block's coefficients, and the upper triangle's
// right-hand side
template <typename CT, bool HASZ, bool LOWER, bool UNIT>
__host__ __device__ constexpr int grid_stage_bytes() {
  return (3 + (HASZ ? 1 : 0) - (UNIT ? 1 : 0) + (LOWER ? 0 : 1)) * 128 * (int)sizeof(CT);
}

// Time a pair of triangles (L, then U; calls one after the other), with the
// block-scheduled kernels and with this one: 128^3 FP32 228 -> 116 us (DRAM 85 MB,
// the chain is the bound), 64^3 116 -> 57 us, 64^2 50 -> 20 us; 128^3 FP64 679 -> 375
// us; 93 x 70 x 51 in FP64, whose lines are no multiple of a chunk, 12,220 -> 159 us.
template <typename CT, bool HASZ, bool LOWER, bool UNIT>
__global__ void __launch_bounds__(32 * (kGW + kGHelpers)) k_sptrsv_grid(GridArgs A) {
  constexpr int D = kGD<CT>;
  constexpr int K = 3 + (HASZ ? 1 : 0) - (UNIT ? 1 : 0);  // coefficients: x, y, [z], [reciprocal diagonal]
  constexpr int VB = 4 * sizeof(CT);                      // bytes of a lane's vector
  constexpr unsigned kStage = grid_stage_bytes<CT, HASZ, LOWER, UNIT>(), kRing = D * kStage;
  constexpr int DIR = LOWER ? 1 : -1;
  extern __shared__ __align__(16) unsigned char smem_g[];
  __shared__ int s_tile;
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const GridShape &g = A.g;
  const int rank = (int)cl.block_rank(), csize = g.cy * g.cz, ry_ = rank % g.cy, rz_ = rank / g.cy;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gw = g.wy * g.wz;
  const int LY = 1 << g.lyl, LZ = 32 >> g.lyl, ly = lane & (LY - 1), lz = lane >> g.lyl;
  const int wy = warp % g.wy, wz = warp / g.wy;
  const int TY = g.sy * g.wy, T4 = 4 * g.nb, nb = g.nb;
  const int rows = LZ + (HASZ ? LY : 0);  // face rows of a tile: LZ towards y, LY towards z
  const int n = g.nx * g.ny * g.nz;
  // the padded lines of the last tiles come last for a lower triangle, first
  // for an upper one (its tiles are the lower's, walked backwards)
  const int Y0 = LOWER ? 0 : TY * LY - g.ny, Z0 = LOWER ? 0 : g.sz * g.wz * LZ - g.nz;
  CT *sface = reinterpret_cast<CT *>(smem_g + (size_t)gw * kRing);
  CT *const stage = sface + (size_t)gw * rows * T4;  // the tiles' lines, kGPad values a block
  const int ngroups = (g.sy / g.cy) * (g.sz / g.cz);
  const bool one_round = ngroups * csize <= (int)gridDim.x;  // a ticket each
  // What does not depend on earlier kernels, then the wait for them.  After it,
  // the next kernel may start in the SMs this one leaves free (it waits for this
  // one's end itself); what a kernel whose predecessor waited here reads of
  // still earlier ones is in place without a wait.
  if (!A.early) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  const int done = A.done != nullptr ? *(volatile const int *)A.done : 0;
  // An earlier solve gave up.  The one cluster of a small box sets the flag itself
  // only after all of its CTAs have read it here; of several clusters another may
  // have set it meanwhile, so that their CTAs leave or stay together by what
  // comes with the ticket.
  const int dirty = ngroups > 1 ? 0 : *(volatile const int *)A.dirty;
  if (A.early && (done || dirty)) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (done) return;  // the same for every CTA
  if (dirty) {
    if (threadIdx.x == 0) atomicOr(A.status, kStatusSpinTimeout);
    return;
  }
  for (int k = threadIdx.x; k < gw * rows * T4; k += blockDim.x) {
    if constexpr (sizeof(CT) == 4) reinterpret_cast<unsigned *>(sface)[k] = kMark32;
    else reinterpret_cast<unsigned long long *>(sface)[k] = kMark64;
  }
  bool waited = !A.early, gone = false;  // gone: this warp gave up a wait
  while (true) {
    int tk = 0;
    if (ngroups > 1) {
      if (rank == 0 && threadIdx.x == 0) {
        const int gone = *(volatile const int *)A.dirty;
        tk = atomicAdd(&A.tickets[0], 1);
        if (gone) {
          atomicOr(A.status, kStatusSpinTimeout);
          tk = ngroups;
        }
      }
      __syncwarp();
      tk = __shfl_sync(0xffffffffu, tk, 0);
    }
    cl.sync();  // every CTA of the cluster is done with its last tiles, its faces are unsolved
    if (ngroups > 1) {
      if (rank == 0 && (int)threadIdx.x < csize) *(volatile int *)cl.map_shared_rank(&s_tile, threadIdx.x) = tk;
      __syncwarp();
      cl.sync();
      tk = *(const volatile int *)&s_tile;
    }
    if (tk >= ngroups) {  // the same for the whole cluster
      // the kernel after this one may count on the one before it having ended
      if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
      break;
    }
    const int gy = g.sy / g.cy;
    const int sy_ = tk % gy * g.cy + ry_, sz_ = tk / gy * g.cz + rz_;  // this CTA's super-tile
    const int ty = sy_ * g.wy + wy, tz = sz_ * g.wz + wz;
    const int yv = ty * LY + ly - Y0, zv = tz * LZ + lz - Z0;  // this lane's line
    const bool lane_ok = yv >= 0 && yv < g.ny && zv >= 0 && zv < g.nz;
    // the lines of the CTA's tiles between rows and the staging, a warp a line
    int2 *const tab = reinterpret_cast<int2 *>(stage + (size_t)gw * nb * kGPad);
    if (warp < gw) {  // a line's first step (past every step: no line) and the row of step 0
      const int s = ly + lz + g.first(LOWER, ty, tz), lin = g.nx * (yv + g.ny * zv);
      tab[threadIdx.x] = make_int2(lane_ok ? s : 1 << 29, (LOWER ? lin : n - 1 - lin) - DIR * s);
    }
    __syncthreads();
    // four lines and five times 32 steps of each a warp at a time, all loads in
    // flight before the first store
    auto lines_in = [&](auto rt) {
      using RT = decltype(rt);
      const RT *b = (const RT *)A.b;
      for (int l = 4 * warp; l < gw * 32; l += blockDim.x >> 3)
        for (int t0 = lane; t0 < T4; t0 += 160) {
          RT v[4][5];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int2 e = tab[l + k];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
              const int t = t0 + 32 * q;
              v[k][q] = (unsigned)(t - e.x) < (unsigned)g.nx ? b[e.y + DIR * t] : (RT)0;
            }
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            CT *const st = stage + ((l + k) >> 5) * nb * kGPad + ((l + k) & 31) * 4;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
              const int t = t0 + 32 * q;
              if (t < T4) st[(t >> 2) * kGPad + (t & 3)] = (CT)v[k][q];
            }
          }
        }
    };
    auto lines_out = [&](auto rt) {
      using RT = decltype(rt);
      RT *x = (RT *)A.x;
      for (int l = warp; l < gw * 32; l += blockDim.x >> 5) {
        const int2 e = tab[l];
        if (e.x >= T4) continue;  // no line here
        const CT *const st = stage + (l >> 5) * nb * kGPad + (l & 31) * 4;
        for (int t0 = e.x + lane; t0 < e.x + g.nx; t0 += 128) {
          CT v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int t = t0 + 32 * q;
            if (t < T4) v[q] = st[(t >> 2) * kGPad + (t & 3)];
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int t = t0 + 32 * q;
            if ((unsigned)(t - e.x) < (unsigned)g.nx) x[e.y + DIR * t] = (RT)v[q];
          }
        }
      }
    };
    if constexpr (LOWER) {
      if (A.rows_f32) lines_in(0.f);
      else lines_in(0.0);
      __syncthreads();
    }
    if (warp >= gw) {
      grid_helper<CT>(A, sy_, sz_, ry_ == 0, rz_ == 0, smem_u32(sface), (warp - gw) * 32 + lane, LOWER, Y0, Z0, rows);
    } else if (__any_sync(0xffffffffu, lane_ok)) {
      const int tile = tz * TY + ty;
      const int XO = g.first(LOWER, ty, tz);
      const int s = ly + lz + XO;  // this lane's first step
      // blocks in which every line of the tile is inside the box
      const int kin0 = (LY + LZ - 2 + XO + 3) >> 2, kin1 = (g.nx + XO) >> 2;
      const unsigned nx = lane_ok ? (unsigned)g.nx : 0u;  // valid steps: 0 <= t - s < nx
      auto valid = [&](int t) { return (unsigned)(t - s) < nx; };
      // faces: rows read by this lane, rows it writes for the next tiles
      const int needY = lane_ok && ly == 0 && yv > 0, needZ = HASZ && lane_ok && lz == 0 && zv > 0;
      const int pubY = lane_ok && ly == LY - 1 && yv + 1 < g.ny, pubZ = HASZ && lane_ok && lz == LZ - 1 && zv + 1 < g.nz;
      unsigned srcY = smem_u32(sface + (size_t)(warp * rows + lz) * T4);
      unsigned srcZ = HASZ ? smem_u32(sface + (size_t)(warp * rows + LZ + ly) * T4) : 0u;
      // the next tiles' faces: in this CTA's shared memory, the next CTA's of the
      // cluster, or global memory; the next tile's step for the same x is a
      // multiple of four steps earlier
      CT *gf = (CT *)A.face, *dstY, *dstZ;
      if (wy + 1 < g.wy) dstY = sface + (size_t)((warp + 1) * rows + lz) * T4;
      else if (ry_ + 1 < g.cy) dstY = cl.map_shared_rank(sface, rank + 1) + (size_t)(wz * g.wy * rows + lz) * T4;
      else dstY = gf + ((size_t)(tile + 1) * rows + lz) * T4;
      if (wz + 1 < g.wz) dstZ = sface + (size_t)((warp + g.wy) * rows + LZ + ly) * T4;
      else if (rz_ + 1 < g.cz) dstZ = cl.map_shared_rank(sface, rank + g.cy) + (size_t)(wy * rows + LZ + ly) * T4;
      else dstZ = gf + ((size_t)(tile + TY) * rows + LZ + ly) * T4;
      dstY -= LY - 1 + XO - g.first(LOWER, ty + 1, tz);
      dstZ -= LZ - 1 + XO - g.first(LOWER, ty, tz + 1);
      const CT *coef = (const CT *)A.coef + (size_t)tile * nb * K * 128 + lane * 4;
      // tile-order vectors are in the lower triangle's order; an upper triangle's
      // tiles, blocks and lanes count from the other end
      const CT *bt = (const CT *)A.b + ((size_t)(g.tiles() - tile) * nb * 32 - 1 - lane) * 4;
      CT *xt = (CT *)A.x + ((size_t)tile * nb * 32 + lane) * 4;
      const unsigned ring = smem_u32(smem_g) + warp * kRing + lane * VB;
      CT *const st = stage + (size_t)warp * nb * kGPad + lane * 4;

      // block kb's coefficients, and right-hand side, into the ring stage at byte o
      auto issue_c = [&](int kb, unsigned o) {
        const CT *c = coef + (size_t)kb * (K * 128);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          cp16(ring + o + k * 32 * VB, c + k * 128);
          if (sizeof(CT) == 8) cp16(ring + o + k * 32 * VB + 16, c + k * 128 + 2);
        }
      };
      auto issue_b = [&](int kb, unsigned o) {
        if constexpr (!LOWER) {
          const CT *p = bt - (size_t)kb * 128;
          cp16(ring + o + K * 32 * VB, p);
          if (sizeof(CT) == 8) cp16(ring + o + K * 32 * VB + 16, p + 2);
        }
      };
      using Blk = GridBlk<CT>;
      auto fetch = [&](int kb, unsigned o, Blk &B) {
        const CT *c = reinterpret_cast<const CT *>(smem_g + warp * kRing + o + lane * VB);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          B.cx[u] = c[u];
          B.cy[u] = c[128 + u];
          if (HASZ) B.cz[u] = c[256 + u];
          const CT b = LOWER ? st[kb * kGPad + u] : c[K * 128 + 3 - u];
          B.v[u] = UNIT ? b : b * c[(K - 1) * 128 + u];
        }
      };
      auto faces = [&](int on, Blk &B) {
        ld_face(needY & on, srcY, B.f[0]);
        if (HASZ) ld_face(needZ & on, srcZ, B.f[1]);
      };
      // Whether some entry of block kb's faces is unsolved, where the lane's line
      // has a step in the block.  A block with an entry on the line is written
      // whole, in FP64 by two stores that nothing orders: with the entries off
      // the line not waited for, the second store could land after the block was
      // marked unsolved again, and its value be taken for a solved one by the
      // next tile that uses this face.
      auto waits = [&](auto edge, int kb, const Blk &B) {
        if constexpr (!decltype(edge)::value) return any_unsolved(B.f);
        bool on = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) on |= valid(4 * kb + u);
        return on && any_unsolved(B.f);
      };
      auto poll = [&](auto edge, int kb, Blk &B) {
        for (int spins = 0;; ++spins) {
          faces(1, B);
          if (!__any_sync(0xffffffffu, waits(edge, kb, B))) break;
          // the whole warp or none of it: the lanes' steps shuffle
          if ((spins & 1023) == 1023 && __any_sync(0xffffffffu, gave_up(spins, A.status, A.dirty))) {
            gone = true;
            break;
          }
        }
      };
      CT x = (CT)0;
      unsigned wst = (D - 1) * kStage, rst = 0;  // ring stages written and read next
      // One block of four steps: the steps on B, and between them the copy of
      // the block D - 1 ahead and the next block's data (on its way since D - 2
      // blocks) and faces into Bn.  Straight-line code up to the test for an
      // unsolved face, so that all of it fills the gaps of the steps' chain.
      // EDGE: some line is outside the box in some step of this block or the
      // next, or the copy ahead would leave the tile.
      auto block = [&](auto edge, int kb, Blk &B, Blk &Bn) {
        constexpr bool EDGE = decltype(edge)::value;
        const int t0 = 4 * kb, more = kb + 1 < nb;
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) in[u] = EDGE ? valid(t0 + u) : lane_ok;
        CT out[4], sy, sz = (CT)0;
        // a step: its shuffles, other work while they are on their way, its sums
        auto shuffle = [&]() {
          sy = __shfl_up_sync(0xffffffffu, x, 1);
          if (HASZ) sz = __shfl_up_sync(0xffffffffu, x, LY);
        };
        auto step = [&](int u) {
          CT acc = fma(-B.cx[u], x, B.v[u]);
          if (HASZ) {
            sz = lz == 0 ? (!EDGE || in[u] ? B.f[1][u] : (CT)0) : sz;
            acc = fma(-B.cz[u], sz, acc);
          }
          sy = ly == 0 ? (!EDGE || in[u] ? B.f[0][u] : (CT)0) : sy;
          out[u] = x = fma(-B.cy[u], sy, acc);
        };
        shuffle();
        clear_face(needY, srcY, (CT)0);
        srcY += VB;
        if (HASZ) {
          clear_face(needZ, srcZ, (CT)0);
          srcZ += VB;
        }
        const int ahead = EDGE ? min(kb + D - 1, nb - 1) : kb + D - 1;
        step(0);
        shuffle();
        issue_c(ahead, wst);
        issue_b(ahead, wst);
        cp_commit();
        step(1);
        shuffle();
        cp_wait<D - 2>();
        wst = wst + kStage == kRing ? 0u : wst + kStage;
        rst = rst + kStage == kRing ? 0u : rst + kStage;
        fetch(EDGE ? min(kb + 1, nb - 1) : kb + 1, rst, Bn);
        step(2);
        shuffle();
        faces(EDGE ? more : 1, Bn);
        step(3);
        const int some = EDGE ? in[0] | in[1] | in[2] | in[3] : 1;
        publish(pubY & some, dstY + t0, out);
        if (HASZ) publish(pubZ & some, dstZ + t0, out);
        if constexpr (LOWER) {
#pragma unroll
          for (int u = 0; u < 4; ++u) out[u] = in[u] ? out[u] : (CT)0;
        }
        CT *d = LOWER ? xt + (size_t)kb * 128 : st + kb * kGPad;
        if constexpr (sizeof(CT) == 4) {
          *reinterpret_cast<float4 *>(d) = make_float4(out[0], out[1], out[2], out[3]);
        } else {
          *reinterpret_cast<double2 *>(d) = make_double2(out[0], out[1]);
          *reinterpret_cast<double2 *>(d + 2) = make_double2(out[2], out[3]);
        }
        if (__any_sync(0xffffffffu, waits(edge, kb + 1, Bn) && more)) poll(edge, kb + 1, Bn);
      };
#pragma unroll
      for (int kb = 0; kb < D - 1; ++kb) issue_c(min(kb, nb - 1), kb * kStage);
      if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
      // the first group holds all coefficients so far and block 0's right-hand
      // side, the next ones their block's
#pragma unroll
      for (int kb = 0; kb < D - 1; ++kb) {
        issue_b(min(kb, nb - 1), kb * kStage);
        cp_commit();
      }
      cp_wait<D - 2>();
      Blk B0, B1;
#pragma unroll
      for (int u = 0; u < 4; ++u) B0.f[0][u] = B0.f[1][u] = B1.f[0][u] = B1.f[1][u] = (CT)0;
      fetch(0, 0, B0);
      poll(std::true_type{}, 0, B0);
      int kb = 0;
      // inner blocks two at a time; the blocks at the lines' ends one at a time
      while (kb < nb) {
        if (kb >= kin0 && kb + 2 < kin1 && kb + D < nb) {
          block(std::false_type{}, kb, B0, B1);
          block(std::false_type{}, kb + 1, B1, B0);
          kb += 2;
        } else {
          block(std::true_type{}, kb, B0, B1);
          B0 = B1;
          ++kb;
        }
      }
      cp_wait<0>();
    }
    if (!waited) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      waited = true;
    }
    // A tile whose warp has read all its faces has no more of them to come.  A
    // warp that gave up stays, and its CTA's shared memory with it, until every
    // warp of the cluster has published.  (Everyone waiting: 128^3 FP32 119.0 us a
    // pair, like this 116.3.  A round that another follows ends at the loop's top.)
    if (one_round && csize > 1) {
      __syncwarp();
      cl.barrier_arrive();
    }
    if constexpr (!LOWER) {
      __syncthreads();
      if (A.rows_f32) lines_out(0.f);
      else lines_out(0.0);
    }
    if (one_round) {
      __syncwarp();
      if (gone && csize > 1) cl.barrier_wait();
      break;
    }
    if constexpr (!LOWER) __syncthreads();
  }
  // the CTA that leaves last re-arms the tickets
  if (ngroups > 1 && threadIdx.x == 0 && atomicAdd(&A.tickets[1], 1) == (int)gridDim.x - 1) {
    A.tickets[0] = 0;
    A.tickets[1] = 0;
    __threadfence();
  }
}

// a line's place in tile order: the element of x = 0 is at
// base + (t / 4) * 128 + t % 4 with t = t0, the others at t = t0 + x
struct GridLine {
  size_t base;
  int t0;
};
// logical line (Y, Z) of a triangle's own order (lower: the box's lines)
__device__ __forceinline__ GridLine grid_line(const GridShape &g, bool lower, int Y, int Z) {
  const int LY = 1 << g.lyl, LZ = 32 >> g.lyl, TY = g.sy * g.wy;
  if (!lower) {
    Y += TY * LY - g.ny;
    Z += g.sz * g.wz * LZ - g.nz;
  }
  const int ty = Y >> g.lyl, tz = Z / LZ, yl = Y & (LY - 1), zl = Z & (LZ - 1);
  return GridLine{((size_t)(tz * TY + ty) * g.nb * 32 + (yl | zl << g.lyl)) * 4, yl + zl + g.first(lower, ty, tz)};
}

// a vector from rows to tile order, and back: a warp per line
template <typename ST, typename CT>
__global__ void k_grid_in(GridShape g, const ST *__restrict__ b, CT *__restrict__ t, const int *done) {
  if (done != nullptr && *(volatile const int *)done) return;
  const int lane = threadIdx.x & 31, lines = g.ny * g.nz;
  for (int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < lines; l += (gridDim.x * blockDim.x) >> 5) {
    const GridLine p = grid_line(g, true, l % g.ny, l / g.ny);
    for (int x = lane; x < g.nx; x += 32) {
      const int tt = p.t0 + x;
      t[p.base + (size_t)(tt >> 2) * 128 + (tt & 3)] = (CT)b[(size_t)l * g.nx + x];
    }
  }
}
template <typename CT, typename OT>
__global__ void k_grid_out(GridShape g, const CT *__restrict__ t, OT *__restrict__ x_, const int *done) {
  if (done != nullptr && *(volatile const int *)done) return;
  const int lane = threadIdx.x & 31, lines = g.ny * g.nz;
  for (int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < lines; l += (gridDim.x * blockDim.x) >> 5) {
    const GridLine p = grid_line(g, true, l % g.ny, l / g.ny);
    for (int x = lane; x < g.nx; x += 32) {
      const int tt = p.t0 + x;
      x_[(size_t)l * g.nx + x] = (OT)t[p.base + (size_t)(tt >> 2) * 128 + (tt & 3)];
    }
  }
}

// the plan's values from the triangle's CSR values, a warp per line
template <typename VT, typename CT>
__global__ void k_grid_values(GridShape g, int lower, int unit, const int *__restrict__ row,
                              const int *__restrict__ col, const VT *__restrict__ val, CT *__restrict__ coef) {
  const int n = g.nx * g.ny * g.nz, K = g.coefs(unit), hz = g.nz > 1, lane = threadIdx.x & 31, lines = g.ny * g.nz;
  for (int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < lines; l += (gridDim.x * blockDim.x) >> 5) {
    const GridLine p = grid_line(g, lower != 0, l % g.ny, l / g.ny);
    // the vectors' (tile, block, lane) order with K planes a block
    const size_t blk = p.base / 128, in = p.base % 128;
    for (int X = lane; X < g.nx; X += 32) {
      const int lin = l * g.nx + X, i = lower ? lin : n - 1 - lin, t = p.t0 + X;
      CT cx = (CT)0, cy = (CT)0, cz = (CT)0, dg = (CT)1;
      for (int e = row[i]; e < row[i + 1]; ++e) {
        const int d = lower ? i - col[e] : col[e] - i;
        const CT v = cvt<CT>(val[e]);
        if (d == 0) dg = v;
        else if (d == 1) cx = v;
        else if (d == g.nx) cy = v;
        else cz = v;
      }
      const CT rd = unit ? (CT)1 : (CT)1 / dg;
      CT *c = coef + (blk + (t >> 2)) * K * 128 + in + (t & 3);
      c[0] = cx * rd;
      c[128] = cy * rd;
      if (hz) c[256] = cz * rd;
      if (!unit) c[(K - 1) * 128] = rd;
    }
  }
}

// *bad |= some row does not have exactly the grid's neighbours
__global__ void k_grid_check(GridShape g, int lower, const int *__restrict__ row, const int *__restrict__ col,
                             int *bad) {
  const int n = g.nx * g.ny * g.nz;
  bool b = false;
  for (int lin = blockIdx.x * blockDim.x + threadIdx.x; lin < n; lin += gridDim.x * blockDim.x) {
    const int i = lower ? lin : n - 1 - lin;
    const int X = lin % g.nx, Y = (lin / g.nx) % g.ny, Z = lin / (g.nx * g.ny);
    int want = 1 | (X > 0 ? 2 : 0) | (Y > 0 ? 4 : 0) | (Z > 0 ? 8 : 0), got = 0, cnt = 0;
    for (int e = row[i]; e < row[i + 1]; ++e, ++cnt) {
      const int d = lower ? i - col[e] : col[e] - i;
      got |= d == 0 ? 1 : (d == 1 ? 2 : (d == g.nx ? 4 : (g.nz > 1 && d == g.nx * g.ny ? 8 : 16)));
    }
    b |= got != want || cnt != __popc(want);
  }
  if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1);
}

constexpr size_t kGridSmemMax = 220 * 1024;
// shared memory of a CTA: the warps' rings, face rows and lines
size_t smem_bytes(const GridShape &g, int stage, size_t ct) {
  return (size_t)g.wy * g.wz * ((ct == 4 ? kGD<float> : kGD<double>) * (size_t)stage + ct * ((size_t)g.face_rows() * 4 * g.nb + (size_t)g.nb * kGPad) + 256);
}
// face rows a CTA gets from other clusters, at most
int helper_rows(const GridShape &g) { return g.wz * (32 >> g.lyl) + (g.nz > 1 ? g.wy << g.lyl : 0); }

template <typename CT, bool HASZ, bool LOWER, bool UNIT>
int launch_t(cudaStream_t s, const GridArgs &a) {
  const auto fn = k_sptrsv_grid<CT, HASZ, LOWER, UNIT>;
  static PerDevice limits;
  if (!limits.done([&] {
        return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGridSmemMax) == cudaSuccess;
      }))
    return DEV_ERR_UNKNOWN;
  const size_t sm = smem_bytes(a.g, grid_stage_bytes<CT, HASZ, LOWER, UNIT>(), sizeof(CT));
  // the lines' copies want all the warps the registers allow
  const int warps = kGW + kGHelpers, csize = a.g.cy * a.g.cz;
  const int groups = a.g.sy * a.g.sz / csize;
  const int room = std::max(1, num_sms() * (int)std::max<size_t>(1, kGridSmemMax / sm) / csize);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(std::min(groups, room) * csize));
  cfg.blockDim = dim3((unsigned)(32 * warps));
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)csize;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = csize > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, fn, a) == cudaSuccess ? 0 : DEV_ERR_UNKNOWN;
}

template <typename CT, bool HASZ>
int launch_ct(cudaStream_t s, const GridArgs &a, int lower, int unit) {
  if (lower) return unit ? launch_t<CT, HASZ, true, true>(s, a) : launch_t<CT, HASZ, true, false>(s, a);
  return unit ? launch_t<CT, HASZ, false, true>(s, a) : launch_t<CT, HASZ, false, false>(s, a);
}

}  // namespace

bool grid_shape(int n, int d1, int d2, int d3, size_t ct, GridShape &g) {
  // distances 1, nx[, nx * ny] with whole lines and planes
  if (d1 != 1 || d2 < 2 || n < 1 || n % d2) return false;
  g.nx = d2;
  if (d3 > 0) {
    if (d3 <= d2 || d3 % d2 || n % d3) return false;
    g.ny = d3 / d2;
    g.nz = n / d3;
  } else {
    g.ny = n / d2;
    g.nz = 1;
  }
  // Lanes, warps as wy x wz tiles, CTAs as cy x cz super-tiles: the split with
  // the least time in hand-overs on the way from the first to the last line (in
  // ns, from time stamps of a 128^3 solve: between warps of a CTA, CTAs of a
  // cluster, clusters), then the fewest tiles.  Up to four warps a CTA in FP32
  // (one a scheduler: 128^3 122 us a pair, two 133, one 161, when it was first
  // chosen) and two in FP64 (the FP64 unit takes no more); fewer where their lines
  // do not fit its shared memory: a CTA holds whole lines, up to about 1,500 rows
  // in FP32 and 715 in FP64, and longer ones go to the chunks.  Clusters of up to
  // eight (128^3: 122 us, four 131).
  const long long kWarpHop = 500, kCtaHop = 550, kFarHop = 1800;
  long long best = -1;
  GridShape pick = g;
  for (int gw = ct == 4 ? kGW : 2; gw >= 1; gw >>= 1)
    for (int l = 0; l <= 5; ++l)
      for (int w = 1; w <= gw; w <<= 1)
        for (int cy = 1; cy <= 8; cy <<= 1)
          for (int cz = 1; cy * cz <= 8; cz <<= 1) {
            GridShape c = g;
            c.lyl = l;
            c.wy = w;
            c.wz = gw / w;
            c.cy = cy;
            c.cz = cz;
            if (g.nz == 1 && (l < 5 || c.wz > 1 || cz > 1)) continue;
            const int LY = 1 << l, LZ = 32 >> l;
            const int ty = (g.ny + LY - 1) / LY, tz = (g.nz + LZ - 1) / LZ;
            c.sy = (ty + w * cy - 1) / (w * cy) * cy;
            c.sz = (tz + c.wz * cz - 1) / (c.wz * cz) * cz;
            c.nb = (g.nx + LY + LZ - 2 + 3 + 3) / 4;
            if (c.sy > 0xffff || c.sz > 0x7fff || 4 * helper_rows(c) > 32 * kGHelpers ||
                smem_bytes(c, 5 * 128 * (int)ct, ct) > kGridSmemMax)
              continue;
            auto hops = [&](int t, int wn, int cn) {  // t tiles in a row
              const long long far = (t - 1) / (wn * cn), cta = (t - 1) / wn - far;
              return far * kFarHop + cta * kCtaHop + (t - 1 - far - cta) * kWarpHop;
            };
            const long long cost = (hops(ty, w, cy) + hops(tz, c.wz, cz)) * 1000 + std::min(999, c.tiles() / 8);
            if (best < 0 || cost < best) {
              best = cost;
              pick = c;
            }
          }
  if (best < 0) return false;
  g = pick;
  // Against the block-scheduled solve of the same triangle (both in ns, from
  // measured solves): its chunks of 32 rows are a wavefront step each where
  // they do not straddle two lines, and one chain where they do; a line's step
  // here is a quarter of a block.  Long and thin boxes of aligned lines stay
  // with the chunks.
  const bool f64 = ct == 8;
  const long long chunk = f64 ? 1280 : 430;
  const long long there = d2 % 32 == 0 ? ((long long)g.nx / 32 + g.ny + g.nz) * chunk : (long long)n / 32 * (f64 ? 590 : 500);
  const long long here = ((long long)g.nx + g.ny + g.nz) * (f64 ? 180 : 50) + best / 1000 + 4000;
  return here <= there;
}

int grid_check(cudaStream_t s, const GridShape &g, bool lower, const int *row, const int *col, int *flag, bool *ok) {
  if (cudaMemsetAsync(flag, 0, 4, s) != cudaSuccess) return DEV_ERR_UNKNOWN;
  const int n = g.nx * g.ny * g.nz;
  k_grid_check<<<std::max(1, std::min((n + 255) / 256, num_sms() * 8)), 256, 0, s>>>(g, lower ? 1 : 0, row, col, flag);
  int f = 1;
  if (cudaMemcpyAsync(&f, flag, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
    return DEV_ERR_UNKNOWN;
  *ok = f == 0;
  return 0;
}

// buffers of one triangle's plan; the padding of the coefficients stays 0
int grid_prepare(cudaStream_t s, const GridShape &g, bool lower, bool unit, VType vt, GridPlan &p) {
  const size_t ct = vt == VType::F64 ? 8 : 4;
  p.valid = false;
  p.g = g;
  p.lower = lower ? 1 : 0;
  p.unit = unit ? 1 : 0;
  p.ct = ct;
  const size_t cb = (size_t)g.tiles() * g.nb * g.coefs(unit) * 128 * ct;
  const size_t fb = (size_t)g.tiles() * g.face_rows() * 4 * g.nb * ct;
  if (p.coef.ensure(cb) || p.face.ensure(fb) || p.ctl.ensure(16))
    return DEV_ERR_DEVICE_ALLOC;
  if (cudaMemsetAsync(p.coef.p, 0, cb, s) != cudaSuccess ||
      grid_clear_faces(s, p))
    return DEV_ERR_UNKNOWN;
  p.vals_version = -1;
  p.valid = true;
  return 0;
}

// the faces unsolved and the tickets re-armed, as every finished solve leaves them
int grid_clear_faces(cudaStream_t s, GridPlan &p) {
  const GridShape &g = p.g;
  const size_t count = (size_t)g.tiles() * g.face_rows() * 4 * g.nb;
  const int grid = (int)std::max<size_t>(1, std::min<size_t>((size_t)num_sms() * 4, (count + 255) / 256));
  k_fill_mark<<<grid, 256, 0, s>>>(p.face.p, p.ct == 4, count);
  return cudaMemsetAsync(p.ctl.p, 0, 16, s) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : DEV_ERR_UNKNOWN;
}

void launch_grid_values(cudaStream_t s, GridPlan &p, const int *row, const int *col, const void *val, VType vt) {
  const GridShape &g = p.g;
  const int grid = std::max(1, std::min((g.ny * g.nz + 7) / 8, num_sms() * 16));
  switch (vt) {
    case VType::F64:
      k_grid_values<double, double><<<grid, 256, 0, s>>>(g, p.lower, p.unit, row, col, (const double *)val,
                                                         (double *)p.coef.p);
      break;
    case VType::F32:
      k_grid_values<float, float><<<grid, 256, 0, s>>>(g, p.lower, p.unit, row, col, (const float *)val,
                                                       (float *)p.coef.p);
      break;
    case VType::BF16:
      k_grid_values<__nv_bfloat16, float><<<grid, 256, 0, s>>>(g, p.lower, p.unit, row, col,
                                                               (const __nv_bfloat16 *)val, (float *)p.coef.p);
      break;
  }
}

// x = T^{-1} b: a lower triangle from rows to tile order, an upper one from
// tile order to rows
static int grid_solve(cudaStream_t s, GridPlan &p, const void *b, void *x, int rows_f32, int early, int *status,
                      const int *done) {
  GridArgs a;
  a.g = p.g;
  a.coef = p.coef.p;
  a.face = p.face.p;
  a.b = b;
  a.x = x;
  a.rows_f32 = rows_f32;
  a.early = early;
  a.tickets = (int *)p.ctl.p;
  a.dirty = (int *)p.ctl.p + 2;
  a.done = done;
  a.status = status;
  if (p.ct == 4)
    return p.g.nz > 1 ? launch_ct<float, true>(s, a, p.lower, p.unit) : launch_ct<float, false>(s, a, p.lower, p.unit);
  return p.g.nz > 1 ? launch_ct<double, true>(s, a, p.lower, p.unit) : launch_ct<double, false>(s, a, p.lower, p.unit);
}

int launch_grid_pair(cudaStream_t s, GridPlan &p1, GridPlan &p2, const void *b, int in_f32, void *t, void *x, int out_f32,
                     int *status, const int *done) {
  const int rc = grid_solve(s, p1, b, t, in_f32, 0, status, done);
  return rc ? rc : grid_solve(s, p2, t, x, out_f32, 1, status, done);
}

int launch_grid_tri(cudaStream_t s, GridPlan &p, const void *b, int in_f32, void *t, void *x, int out_f32, int *status,
                    const int *done) {
  const int grid = std::max(1, std::min((p.g.ny * p.g.nz + 7) / 8, num_sms() * 16));
  if (p.lower) {
    const int rc = grid_solve(s, p, b, t, in_f32, 0, status, done);
    if (rc) return rc;
    if (p.ct == 8 && out_f32) k_grid_out<double, float><<<grid, 256, 0, s>>>(p.g, (const double *)t, (float *)x, done);
    else if (p.ct == 8) k_grid_out<double, double><<<grid, 256, 0, s>>>(p.g, (const double *)t, (double *)x, done);
    else if (out_f32) k_grid_out<float, float><<<grid, 256, 0, s>>>(p.g, (const float *)t, (float *)x, done);
    else k_grid_out<float, double><<<grid, 256, 0, s>>>(p.g, (const float *)t, (double *)x, done);
    return 0;
  }
  if (p.ct == 8 && in_f32) k_grid_in<float, double><<<grid, 256, 0, s>>>(p.g, (const float *)b, (double *)t, done);
  else if (p.ct == 8) k_grid_in<double, double><<<grid, 256, 0, s>>>(p.g, (const double *)b, (double *)t, done);
  else if (in_f32) k_grid_in<float, float><<<grid, 256, 0, s>>>(p.g, (const float *)b, (float *)t, done);
  else k_grid_in<double, float><<<grid, 256, 0, s>>>(p.g, (const double *)b, (float *)t, done);
  return grid_solve(s, p, t, x, out_f32, 0, status, done);
}

}  // namespace lace
