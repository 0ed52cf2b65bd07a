// Prisms, quads and curved triangles: upload, sampled boxes, their own
// LBVH, and the primitive pass of a trace call.
//
// The reference traces every primitive kind in one BVH walk
// (FEM-AABB/raytracer.cu:255-347). Here the hexahedra go through their own
// engine first; the primitive pass then visits, per query, the primitives
// whose box the ray meets in ascending (box entry, index) order, each on the
// segment [0.001, closest hit so far] that starts at the hexahedra's hit,
// and keeps a primitive hit when it is nearer. One thread per query, until the
// query has spent kPrimBudget solver iterations; those queries' searches are then
// dealt over the lanes of warps. The per-primitive solves are short, branchy
// FP32 Newton loops whose start search the reference defines by exact
// comparisons. This file is compiled
// without multiply-add contraction (see ho_prim.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ho_host.h"
#include "ho_prim.cuh"
#include "ho_trace.cuh"

namespace ho {

namespace {

#define PR_TRY(x)                            \
  do {                                       \
    cudaError_t e__ = (x);                   \
    if (e__ != cudaSuccess) return int(e__); \
  } while (0)

constexpr int kPrimThreads = 128;
// Resident blocks per SM the register budget is sized for (80 registers a
// thread; measured faster than 64, 128 or an unbounded 208 despite spills),
// and candidates collected per walk of the primitive tree (a ray with more
// walks again; 16 halves the node visits but measured no faster).
#ifndef HO_PRIM_MIN_BLOCKS
#define HO_PRIM_MIN_BLOCKS 6
#endif
#ifndef HO_PRIM_CAND_K
#define HO_PRIM_CAND_K 8
#endif
constexpr int kPrimCandK = HO_PRIM_CAND_K;

__global__ void prim_setup_kernel(PrimRec* __restrict__ recs, const float* __restrict__ pool, int64_t n,
                                  float* __restrict__ box) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const PrimRec p = recs[i];
  float lo[3], hi[3];
  pr_box(p, pool, lo, hi);
  for (int a = 0; a < 3; ++a) {
    recs[i].lo[a] = lo[a];
    recs[i].hi[a] = hi[a];
    box[6 * i + a] = lo[a];
    box[6 * i + 3 + a] = hi[a];
  }
}

// Interpolation on [-1.05, 1.05] at n points and the change to the Bernstein
// basis of degree n - 1 there: a polynomial lies between its Bernstein
// coefficients' extremes. amp: the change's infinity norm, for the rounding.
struct PrimMats {
  float node[kPrimMaxModes + 1][kPrimMaxModes];
  float inv[kPrimMaxModes + 1][kPrimMaxModes * kPrimMaxModes];
  float amp[kPrimMaxModes + 1];
};

// One block per primitive, once per scene: the oriented bounds over r, s (, t)
// in [-1.05, 1.05], the widest range that a hit or a quad's containment test
// accepts (a linear triangle clamps its point into the triangle: its
// vertices), along the rows of the inverse Jacobian at the centre.
__global__ void __launch_bounds__(64) prim_cull_kernel(const PrimRec* __restrict__ recs, const float* __restrict__ pool,
                                                       const PrimMats* __restrict__ mats, PrimCull* __restrict__ cull,
                                                       float* __restrict__ start) {
  constexpr int kMost = kPrimMaxModes * kPrimMaxModes * kPrimMaxModes;
  __shared__ float pt[2][3][kMost];
  __shared__ float red[64];
  const PrimRec& p = recs[blockIdx.x];
  const bool curved = pr_curved(p);
  if (p.kind == kPrimPrism && threadIdx.x < 7) {  // the points of the prism solver's starts
    const float3 X = pr_point(p, pool, pr_prism_start(threadIdx.x));
    float* x = start + 21 * static_cast<int64_t>(blockIdx.x) + 3 * threadIdx.x;
    x[0] = X.x;
    x[1] = X.y;
    x[2] = X.z;
  }
  int dim[3] = {1, 1, 1};
  if (p.kind == kPrimTri) {
    dim[0] = 3;
  } else {
    for (int a = 0; a < (p.kind == kPrimPrism ? 3 : 2); ++a) dim[a] = curved ? max(2, static_cast<int>(pmode(p.gm, a))) : 2;
  }
  const int n = dim[0] * dim[1] * dim[2];
  float amp = 1.f;
  int cur = 0;
  if (p.kind == kPrimTri) {
    if (threadIdx.x < 3)
      for (int a = 0; a < 3; ++a) pt[0][a][threadIdx.x] = p.v[3 * threadIdx.x + a];
    __syncthreads();
  } else {
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      const int i = q % dim[0], j = (q / dim[0]) % dim[1], k = q / (dim[0] * dim[1]);
      const float3 X = pr_point(p, pool, make_float3(mats->node[dim[0]][i], mats->node[dim[1]][j],
                                                     p.kind == kPrimPrism ? mats->node[dim[2]][k] : 0.f));
      pt[0][0][q] = X.x;
      pt[0][1][q] = X.y;
      pt[0][2][q] = X.z;
    }
    __syncthreads();
    int stride = 1;
    for (int ax = 0; ax < (p.kind == kPrimPrism ? 3 : 2); ++ax) {
      const float* M = mats->inv[dim[ax]];
      amp *= mats->amp[dim[ax]];
      for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const int at = (q / stride) % dim[ax], base = q - at * stride;
        for (int a = 0; a < 3; ++a) {
          float v = 0.f;
          for (int r = 0; r < dim[ax]; ++r) v += M[at * kPrimMaxModes + r] * pt[cur][a][base + r * stride];
          pt[cur ^ 1][a][q] = v;
        }
      }
      stride *= dim[ax];
      cur ^= 1;
      __syncthreads();
    }
  }
  // directions: rows of the inverse of the tangents at the centre (a surface's
  // third tangent: its normal)
  float3 t[3];
  if (p.kind == kPrimTri) {
    t[0] = pr_sub(pr_vert(p, 1), pr_vert(p, 0));
    t[1] = pr_sub(pr_vert(p, 2), pr_vert(p, 0));
  } else {
    float3 X;
    pr_geom(p, pool, make_float3(0.f, 0.f, 0.f), X, t);
  }
  if (p.kind != kPrimPrism) t[2] = pr_cross(t[0], t[1]);
  const float3 c[3] = {pr_cross(t[1], t[2]), pr_cross(t[2], t[0]), pr_cross(t[0], t[1])};
  const float det = pr_dot(t[0], c[0]);
  const float inv = 1.0f / det;
  PrimCull out;
  float size = 0.f;
  bool ok = !(p.kind == kPrimTri && curved) && fabsf(det) > 1e-30f && fabsf(inv) < 1e30f;
  const auto block_max = [&](float x) {
    red[threadIdx.x] = x == x ? x : FLT_MAX;  // a NaN counts as infinite
    __syncthreads();
    for (int h = 32; h > 0; h >>= 1) {
      if (threadIdx.x < h) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + h]);
      __syncthreads();
    }
    const float r = red[0];
    __syncthreads();
    return r;
  };
  for (int a = 0; a < 3; ++a) {
    float m = 0.f;
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      const float v = fabsf(pt[cur][a][q]);
      m = v <= FLT_MAX ? fmaxf(m, v) : FLT_MAX;
    }
    size = fmaxf(size, block_max(m));
  }
  ok = ok && size < 1e15f;
  for (int k = 0; k < 3; ++k) {
    const float mv[3] = {c[k].x * inv, c[k].y * inv, c[k].z * inv};
    const float m1 = fabsf(mv[0]) + fabsf(mv[1]) + fabsf(mv[2]);
    float lo = FLT_MAX, hi = -FLT_MAX;
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      const float v = mv[0] * pt[cur][0][q] + mv[1] * pt[cur][1][q] + mv[2] * pt[cur][2][q];
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
    const float slack = m1 * size * 1e-6f * (2.f + amp);
    out.lo[k] = -block_max(-lo) - slack;
    out.hi[k] = block_max(hi) + slack;
    for (int a = 0; a < 3; ++a) out.m[3 * k + a] = mv[a];
    ok = ok && m1 < 1e20f && fabsf(out.lo[k]) < 1e25f && fabsf(out.hi[k]) < 1e25f;
  }
  out.size = ok ? size : -1.f;
  if (threadIdx.x == 0) cull[blockIdx.x] = out;
}

struct PrimParams {
  const BNode* __restrict__ nodes;
  const PrimRec* __restrict__ prims;
  const PrimCull* __restrict__ cull;
  const float* __restrict__ start;  // per prism: the points of its solver's 7 starts
  const float* __restrict__ geom;
  const float* __restrict__ field;
  const float* __restrict__ rays;
  int64_t n_rays;
  CamArgs cam;
  const ViewDesc* views;
  int n_views;
  float iso[8];
  uint32_t iso_mask;
  ho_hit* __restrict__ hits;
  uint8_t* __restrict__ rgb;
  int64_t n_queries;
  bool fresh;
  DevStats* stats;
  struct PrimHeavy* heavy;  // queries handed to prim_heavy_kernel (nullptr: none are)
  unsigned heavy_cap;       // the most that fit
  unsigned* heavy_ctr;      // their count (it may pass heavy_cap), and the next to take
};

// A primitive whose bounds the ray misses is no candidate, nor a prism whose
// starts all end at once.
struct PrimKeep {
  const PrimParams& P;
  float3 o, d;
  float tmax;
  __device__ __forceinline__ bool operator()(int e) const {
    if (!pr_may_hit(P.cull[e], o, d, 0.001f, tmax, kPrimTol)) return false;
    const PrimRec& p = P.prims[e];
    return p.kind != kPrimPrism || pr_prism_begins(p, P.start + 21 * static_cast<int64_t>(e), o, d, 0.001f, tmax);
  }
};

// A query's answer so far and where its candidate walk stands.
struct PrimState {
  float best;  // closest hit so far
  int win;     // its primitive (-1: none of this pass)
  float3 x;
  float kt;  // last visited key (entry, index)
  int ke;
};
// A query handed to prim_heavy_kernel.
struct PrimHeavy {
  int32_t q;
  uint32_t iters;
  PrimState s;
};
static_assert(sizeof(PrimHeavy) == 36, "what a handed-over query takes, below");
// Iterations after which a query is handed over. A quad's or a triangle's
// start search takes 1,000 to 4,000 iterations when it finds nothing; on one
// thread a ray that passes several such surfaces ran for hundreds of
// milliseconds after the others had ended. (32, 96 and 1,024 measure within 2%.)
constexpr uint32_t kPrimBudget = 256;
// Most queries handed over in a call (36 bytes each); the others run to their
// end where they are.
constexpr int64_t kPrimHeavyMost = int64_t(1) << 22;

__device__ __forceinline__ ho_hit prim_base(const PrimParams& P, int64_t q) {
  if (!P.fresh) return P.hits[q];
  ho_hit h;
  h.t = FLT_MAX;
  h.elem = -1;
  h.face = -1;
  h.kind = HO_HIT_MISS;
  for (int a = 0; a < 3; ++a) h.xi[a] = h.n[a] = 0.f;
  h.u = 0.f;
  h.flags = 0;
  h.iters = 0;
  return h;
}

// The hit record and the pixel of a finished query.
__device__ __forceinline__ void prim_finish(const PrimParams& P, int64_t q, float3 d, ho_hit h, const PrimState& s,
                                            uint32_t iters, bool incomplete) {
  if (s.win >= 0) {
    const PrimRec& p = P.prims[s.win];
    const float3 n = pr_normal(p, P.geom, s.x, d);
    h.t = s.best;
    h.elem = p.local;
    h.face = -1;
    h.kind = static_cast<int16_t>(HO_HIT_PRISM + p.kind);
    h.xi[0] = s.x.x;
    h.xi[1] = s.x.y;
    h.xi[2] = s.x.z;
    h.n[0] = n.x;
    h.n[1] = n.y;
    h.n[2] = n.z;
    h.u = pr_field(p, P.field, s.x);
    h.flags = 0;
  }
  h.iters += iters;
  if (incomplete) h.flags |= HO_FLAG_INCOMPLETE;
  if (P.hits && (P.fresh || s.win >= 0 || incomplete)) P.hits[q] = h;
  if (P.rgb && P.rays == nullptr && (P.fresh || s.win >= 0)) {
    HitState v;
    v.t = h.t;
    v.elem = h.elem;
    v.face = h.face;
    v.kind = h.kind;
    v.n = make_float3(h.n[0], h.n[1], h.n[2]);
    shade(v, d, P.rgb + 3 * q);
  }
}

// The j-th of a walk's candidates, from registers.
__device__ __forceinline__ void walk_entry(const float (&bt)[kPrimCandK], const int (&be)[kPrimCandK], int j, float& ct,
                                           int& ce) {
  ct = bt[0];
  ce = be[0];
#pragma unroll
  for (int m = 1; m < kPrimCandK; ++m)
    if (j == m) {
      ct = bt[m];
      ce = be[m];
    }
}

// The candidates of a query in (box entry, index) order on [0.001, closest hit
// so far], from where its walk stands. Hands over after kPrimBudget iterations
// when there is room (returns false, with the place in the list).
__device__ __forceinline__ bool prim_walk(const PrimParams& P, float3 o, float3 d, PrimState& s, PrimWork& pw,
                                          unsigned& cand, Work& w, bool& incomplete, unsigned& place) {
  const uint32_t iters0 = pw.iters;
  bool asked = false;
  for (;;) {
    float bt[kPrimCandK];
    int be[kPrimCandK];
    bool overflow;
    if (!collect_in<kPrimCandK>(P.nodes, o, d, s.best, s.kt, s.ke, bt, be, overflow, w, PrimKeep{P, o, d, s.best})) {
      atomicOr(&P.stats->status, kStatusStackOverflow);
      incomplete = true;
      return true;
    }
    bool done = false;
#pragma unroll 1
    for (int j = 0; j < kPrimCandK; ++j) {
      float ct;
      int ce;
      walk_entry(bt, be, j, ct, ce);
      if (ce == INT_MAX || ct > s.best) {
        done = true;
        break;
      }
      if (P.heavy && !asked && pw.iters - iters0 > kPrimBudget) {
        asked = true;
        place = atomicAdd(P.heavy_ctr, 1u);
        if (place < P.heavy_cap) return false;
      }
      const PrimRec& p = P.prims[ce];  // read in place: the solvers take it by reference
      float te, tx, th;
      float3 xh;
      ++cand;
      if (pr_slab(o, d, p.lo, p.hi, 0.001f, s.best, te, tx) &&
          pr_hit(p, P.cull[ce], P.start + 21 * static_cast<int64_t>(ce), P.geom, o, d, 0.001f, s.best, th, xh, pw) &&
          th > 0.001f && th < s.best) {
        s.best = th;
        s.win = ce;
        s.x = xh;
      }
      s.kt = ct;
      s.ke = ce;
    }
    if (done || !overflow) return true;
  }
}

__global__ void __launch_bounds__(kPrimThreads, HO_PRIM_MIN_BLOCKS) prim_trace_kernel(PrimParams P) {
  PrimWork pw;
  unsigned cand = 0;
  Work w;
  const int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q < P.n_queries) {
    float3 o, d;
    float iso;
    bool iso_on;
    query_ray_from(P.rays, P.n_rays, P.cam, P.iso, P.iso_mask, P.views, P.n_views, q, o, d, iso, iso_on);
    const ho_hit h = prim_base(P, q);
    PrimState s;
    s.best = h.kind != HO_HIT_MISS ? h.t : FLT_MAX;
    s.win = -1;
    s.x = make_float3(0.f, 0.f, 0.f);
    s.kt = -FLT_MAX;
    s.ke = -1;
    bool incomplete = false;
    unsigned place = 0;
    if (prim_walk(P, o, d, s, pw, cand, w, incomplete, place)) {
      prim_finish(P, q, d, h, s, pw.iters, incomplete);
    } else {
      PrimHeavy v;
      v.q = static_cast<int32_t>(q);
      v.iters = pw.iters;
      v.s = s;
      P.heavy[place] = v;
    }
  }
  // counters: summed over the warp when all its lanes are here together
  // (the last block's tail warp is partial), else added one by one
  const unsigned long long v[4] = {cand, pw.iters, pw.flops, w.nodes};
  const bool whole = __activemask() == 0xffffffffu;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    unsigned long long x = v[k];
    if (whole) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
      if ((threadIdx.x & 31) != 0) x = 0;
    }
    if (x) atomicAdd(&P.stats->c[ST_PRIM_CAND + k], x);
  }
}

__device__ __forceinline__ float3 shfl_f3(float3 v, int src) {
  return make_float3(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                     __shfl_sync(0xffffffffu, v.z, src));
}

// The handed-over queries: up to 16 per warp, a lane each, in rounds. In a
// round every lane walks to its query's next candidate; prisms are solved lane
// by lane; the start searches of the surface candidates, 36 to 108 independent
// solves each, are dealt over all lanes, in order and packed (a query's success
// with the lowest number is the start that the loops of pr_hit_surface would stop
// at); the Newtons that follow run a lane each. A lane whose query has ended takes the
// next; with few queries a warp takes fewer, so that all warps have some. What
// bounds it is the issue rate of the searches' chains and their unequal lengths
// (18 of at most 30 iterations on average, a pass takes its longest). 4,138
// curved triangles at 960 x 540 ran 97 ms with a warp to each query, whose lanes
// mostly waited (8 of 40 searches in a second pass, one lane's Newton on all);
// 70 / 59 / 51 / 49 / 53 ms with 2 / 4 / 8 / 16 / 32 queries a warp. Six or eight
// blocks an SM with fewer registers: 59 and 60 ms.
__global__ void __launch_bounds__(kPrimThreads, 4) prim_heavy_kernel(PrimParams P) {
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ unsigned spent[kPrimThreads];  // iterations for the lane's query
  const int lane = threadIdx.x & 31, first = threadIdx.x & ~31;
  const unsigned n = min(*P.heavy_ctr, P.heavy_cap), warps = gridDim.x * (kPrimThreads / 32);
  const int width = static_cast<int>(min(16u, (n + warps - 1u) / warps));
  PrimWork pw;
  unsigned cand = 0;
  Work w;
  bool have = false, drained = lane >= width, overflow = true, incomplete = false;
  PrimHeavy v;
  float3 o = make_float3(0.f, 0.f, 0.f), d = o;
  float bt[kPrimCandK];
  int be[kPrimCandK], at = kPrimCandK;
  for (;;) {
    if (!have && !drained) {
      const unsigned k = atomicAdd(P.heavy_ctr + 1, 1u);
      if (k < n) {
        v = P.heavy[k];
        float iso;
        bool iso_on;
        query_ray_from(P.rays, P.n_rays, P.cam, P.iso, P.iso_mask, P.views, P.n_views, v.q, o, d, iso, iso_on);
        have = overflow = true;
        incomplete = false;
        at = kPrimCandK;
        spent[threadIdx.x] = v.iters;
      } else {
        drained = true;
      }
    }
    if (!__any_sync(kAll, have)) break;
    // -- the query's next candidate, or its end
    int ce = -1;
    bool surface = false;
    float enter = 0.f, exit = 0.f;
    if (have) {
      PrimState& s = v.s;
      bool end = false;
      while (ce < 0 && !end) {
        if (at == kPrimCandK) {
          if (!overflow) break;
          if (!collect_in<kPrimCandK>(P.nodes, o, d, s.best, s.kt, s.ke, bt, be, overflow, w,
                                      PrimKeep{P, o, d, s.best})) {
            atomicOr(&P.stats->status, kStatusStackOverflow);
            incomplete = end = true;
            break;
          }
          at = 0;
        }
        float ct;
        int e;
        walk_entry(bt, be, at, ct, e);
        if (e == INT_MAX || ct > s.best) {
          end = true;
          break;
        }
        ++at;
        ++cand;
        s.kt = ct;
        s.ke = e;
        const PrimRec& p = P.prims[e];
        if (pr_slab(o, d, p.lo, p.hi, 0.001f, s.best, enter, exit) &&
            (p.kind == kPrimPrism || pr_may_hit(P.cull[e], o, d, 0.001f, s.best, kPrimTol))) {
          ce = e;
          surface = p.kind != kPrimPrism;
        }
      }
      if (ce < 0) {
        prim_finish(P, v.q, d, prim_base(P, v.q), s, spent[threadIdx.x], incomplete);
        have = false;
      }
    }
    __syncwarp();
    bool hit = false;
    float th = 0.f;
    float3 xh = make_float3(0.f, 0.f, 0.f);
    const uint32_t own = pw.iters;
    if (ce >= 0 && !surface)
      hit = pr_hit_prism(P.prims[ce], P.cull[ce], P.start + 21 * static_cast<int64_t>(ce), P.geom, o, d, 0.001f, v.s.best,
                         th, xh, pw);
    __syncwarp();
    // -- the surfaces' start searches
    int base = 0, total = 0;
    bool started = false;
    float r = 0.f, t = 0.f;
    if (surface) {
      const bool quad = P.prims[ce].kind == kPrimQuad;
      float3 plane;
      total = (quad ? 99 : 36) + (pr_plane_point(P.prims[ce], o, d, enter, exit, plane) ? (quad ? 9 : 4) : 0);
    }
    const uint32_t before = pw.iters;
    if (ce >= 0) atomicAdd(&spent[threadIdx.x], before - own);
    for (;;) {
      const int rem = total - base;
      int incl = rem;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(kAll, incl, off);
        if (lane >= off) incl += x;
      }
      const int all = __shfl_sync(kAll, incl, 31);
      if (all == 0) break;
      const int excl = incl - rem;
      int q = 0;  // the query of this lane's solve: the first whose solves go past the lane
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(kAll, incl, q + step - 1) <= lane) q += step;
      const int k = __shfl_sync(kAll, base, q) + lane - __shfl_sync(kAll, excl, q);
      const int e = __shfl_sync(kAll, ce, q);
      const float3 qo = shfl_f3(o, q), qd = shfl_f3(d, q);
      const float qen = __shfl_sync(kAll, enter, q), qex = __shfl_sync(kAll, exit, q);
      bool ok = false;
      float rr = 0.f, ss = 0.f;
      PrimWork job;
      if (lane < all) {
        const PrimRec& p = P.prims[e];
        const bool quad = p.kind == kPrimQuad;
        const int starts = quad ? 9 : 4, points = quad ? 11 : 9;
        float3 x;
        if (k < points * starts) x = pr_segment_point(qo, qd, qen, qex, k / starts, points - 1);
        else pr_plane_point(p, qo, qd, qen, qex, x);
        if (!quad || pr_near(P.cull[e], x, kPrimNear)) {
          ok = pr_project(p, P.geom, x, k % starts, rr, ss, job) && pr_on_surface(p, P.geom, x, rr, ss, job);
        }
      }
      __syncwarp();
      const unsigned m = __ballot_sync(kAll, ok);
      const int hi = min(incl, 32);
      const bool mine = rem > 0 && excl < 32;
      const unsigned f = mine ? m & (kAll >> (32 - hi)) & (kAll << excl) : 0u;
      const int src = f ? __ffs(f) - 1 : 0;
      const float r1 = __shfl_sync(kAll, rr, src), s1 = __shfl_sync(kAll, ss, src);
      // counted are the solves up to the success, whatever ran beside them
      const unsigned fq = __shfl_sync(kAll, f, q);
      if (job.iters && (fq == 0u || lane < __ffs(fq))) {
        pw.iters += job.iters;
        pw.flops += job.flops;
        atomicAdd(&spent[first + q], job.iters);
      }
      if (f) {
        started = true;
        r = r1;
        t = s1;
        base = total;
      } else if (mine) {
        base += hi - excl;
      }
    }
    // -- their Newtons
    if (surface) {
      const PrimRec& p = P.prims[ce];
      const float2 rs = make_float2(r, t);
      t = 0.5f * (enter + exit);
      if (started || p.kind != kPrimQuad) t = pr_param(o, d, pr_point(p, P.geom, make_float3(rs.x, rs.y, 0.f)));
      const uint32_t it0 = pw.iters;
      hit = pr_surface_newton(p, P.geom, o, d, 0.001f, v.s.best, rs.x, rs.y, t, th, xh, pw);
      atomicAdd(&spent[threadIdx.x], pw.iters - it0);
    }
    if (hit && th > 0.001f && th < v.s.best) {
      v.s.best = th;
      v.s.win = ce;
      v.s.x = xh;
    }
    __syncwarp();
  }
  const unsigned long long c[4] = {cand, pw.iters, pw.flops, w.nodes};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    unsigned long long x = c[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(kAll, x, off);
    if (lane == 0 && x) atomicAdd(&P.stats->c[ST_PRIM_CAND + k], x);
  }
}

// Host copy of the primitives, kind-major, with modes packed and offsets
// rebased; a geometry whose modes do not make it curved for its kind is
// kept linear, as the reference's HasHighOrderGeom decides.
void pack_prims(const HostPrims& hp, std::vector<PrimRec>& recs, int64_t counts[3]) {
  recs.clear();
  counts[0] = counts[1] = counts[2] = 0;
  for (int k = 0; k < 3; ++k)
    for (int64_t i = 0; i < hp.size(); ++i) {
      if (hp.kind[i] != k) continue;
      PrimRec r;
      std::memset(&r, 0, sizeof(r));
      std::copy(hp.verts.begin() + 18 * i, hp.verts.begin() + 18 * i + 18, r.v);
      r.kind = k;
      r.local = static_cast<int32_t>(counts[k]++);
      const uint32_t* g = hp.gmodes.data() + 3 * i;
      const uint32_t* f = hp.fmodes.data() + 3 * i;
      const bool curved = hp.goff[i] >= 0 && g[0] > 0 && g[1] > 0 && (k != kPrimPrism || g[2] > 0);
      r.gm = curved ? (g[0] | g[1] << 8 | (k == kPrimPrism ? g[2] : 0u) << 16) : 0u;
      r.goff = curved ? hp.goff[i] : -1;
      r.fm = f[0] | f[1] << 8 | (k == kPrimPrism ? f[2] : 0u) << 16;
      r.foff = hp.foff[i];
      recs.push_back(r);
    }
}

}  // namespace

void prims_free(ho_context* c) {
  cudaFree(c->d_prims);
  cudaFree(c->d_pcull);
  cudaFree(c->d_pstart);
  cudaFree(c->d_pgeom);
  cudaFree(c->d_pfield);
  cudaFree(c->d_pbox);
  cudaFree(c->d_pnodes);
  c->d_prims = c->d_pcull = nullptr;
  c->d_pstart = nullptr;
  c->d_pgeom = c->d_pfield = c->d_pbox = nullptr;
  c->d_pnodes = nullptr;
  c->n_prims = c->n_pnodes = 0;
  c->pbvh_depth = 0;
  c->prim_counts[0] = c->prim_counts[1] = c->prim_counts[2] = 0;
}

int prims_build(ho_context* c) {
  prims_free(c);
  const HostPrims& hp = c->hs.prims;
  if (hp.size() == 0) return 0;
  std::vector<PrimRec> recs;
  pack_prims(hp, recs, c->prim_counts);
  const int64_t n = static_cast<int64_t>(recs.size());
  cudaStream_t s = c->stream;
  const size_t ng = std::max<size_t>(hp.geom.size(), 1), nf = std::max<size_t>(hp.field.size(), 1);
  PR_TRY(cudaMalloc(&c->d_prims, n * sizeof(PrimRec)));
  PR_TRY(cudaMalloc(&c->d_pgeom, ng * sizeof(float)));
  PR_TRY(cudaMalloc(&c->d_pfield, nf * sizeof(float)));
  PR_TRY(cudaMalloc(&c->d_pbox, n * 6 * sizeof(float)));
  PR_TRY(cudaMemcpyAsync(c->d_prims, recs.data(), n * sizeof(PrimRec), cudaMemcpyHostToDevice, s));
  if (!hp.geom.empty())
    PR_TRY(cudaMemcpyAsync(c->d_pgeom, hp.geom.data(), hp.geom.size() * sizeof(float), cudaMemcpyHostToDevice, s));
  if (!hp.field.empty())
    PR_TRY(cudaMemcpyAsync(c->d_pfield, hp.field.data(), hp.field.size() * sizeof(float), cudaMemcpyHostToDevice, s));
  prim_setup_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, s>>>(static_cast<PrimRec*>(c->d_prims),
                                                                           c->d_pgeom, n, c->d_pbox);
  PR_TRY(cudaGetLastError());
  {
    PrimMats M;
    std::memset(&M, 0, sizeof(M));
    std::vector<double> B, V;
    for (int m = 2; m <= kPrimMaxModes; ++m) {
      // Bernstein polynomials at Chebyshev-Lobatto points, inverted
      std::vector<double> x(m);
      B.assign(static_cast<size_t>(m) * m, 0.0);
      for (int r = 0; r < m; ++r) {
        x[r] = 0.5 - 0.5 * std::cos(M_PI * r / (m - 1));
        M.node[m][r] = static_cast<float>(-1.05 + 2.1 * x[r]);
        double binom = 1.0;
        for (int k = 0; k < m; ++k) {
          if (k > 0) binom = binom * (m - k) / k;
          B[r * m + k] = binom * std::pow(x[r], k) * std::pow(1.0 - x[r], m - 1 - k);
        }
      }
      invert_dense(B, m, V);
      for (int k = 0; k < m; ++k) {
        double row = 0.0;
        for (int r = 0; r < m; ++r) {
          M.inv[m][k * kPrimMaxModes + r] = static_cast<float>(V[k * m + r]);
          row += std::fabs(V[k * m + r]);
        }
        M.amp[m] = std::max(M.amp[m], static_cast<float>(row));
      }
    }
    PrimMats* dm = nullptr;
    PR_TRY(cudaMalloc(&c->d_pcull, n * sizeof(PrimCull)));
    PR_TRY(cudaMalloc(&c->d_pstart, std::max<int64_t>(c->prim_counts[0], 1) * 21 * sizeof(float)));
    PR_TRY(cudaMalloc(&dm, sizeof(PrimMats)));
    cudaError_t e = cudaMemcpyAsync(dm, &M, sizeof(M), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
      prim_cull_kernel<<<static_cast<unsigned>(n), 64, 0, s>>>(static_cast<const PrimRec*>(c->d_prims), c->d_pgeom, dm,
                                                               static_cast<PrimCull*>(c->d_pcull), c->d_pstart);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(dm);
    PR_TRY(e);
  }
  float bounds[6];
  const int rc = build_tree(c->d_pbox, nullptr, n, s, &c->d_pnodes, &c->n_pnodes, &c->pbvh_depth, bounds);
  if (rc) return rc;
  c->n_prims = n;
  c->device_bytes += n * static_cast<int64_t>(sizeof(PrimRec) + sizeof(PrimCull) + 24 + sizeof(BNode)) +
                     static_cast<int64_t>((ng + nf) * sizeof(float));
  return 0;
}

int launch_prims(ho_context* c, const TraceArgs& a, ho_hit* hits, bool fresh, DevStats* stats, cudaStream_t s,
                 bool may_allocate) {
  PrimParams P;
  P.nodes = c->d_pnodes;
  P.prims = static_cast<const PrimRec*>(c->d_prims);
  P.cull = static_cast<const PrimCull*>(c->d_pcull);
  P.start = c->d_pstart;
  P.geom = c->d_pgeom;
  P.field = c->d_pfield;
  P.rays = a.rays;
  P.n_rays = a.n_rays;
  P.cam = cam_args(a);
  P.views = a.views;
  P.n_views = a.n_views;
  for (int i = 0; i < 8; ++i) P.iso[i] = i < a.n_iso ? a.iso[i] : 0.f;
  P.iso_mask = a.iso_on_mask;
  P.hits = hits;
  P.rgb = a.rgb;
  P.n_queries = a.rays ? a.n_rays * a.n_iso
                       : (a.views ? a.n_queries_views : static_cast<int64_t>(a.width) * a.height * a.n_iso);
  P.fresh = fresh;
  P.stats = stats ? stats : c->d_stats;
  if (P.n_queries == 0) return 0;
  const int64_t blocks = (P.n_queries + kPrimThreads - 1) / kPrimThreads;
  P.heavy = nullptr;
  P.heavy_cap = 0;
  P.heavy_ctr = nullptr;
  // The list is the context's. A call that the caller is capturing does not
  // use it (the graph would keep its address), nor one for which there is no
  // memory: their queries all run on one thread each. Calls on other streams
  // wait for the list's last reader.
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  PR_TRY(cudaStreamIsCapturing(s, &cs));
  if (may_allocate && cs == cudaStreamCaptureStatusNone) {
    const int64_t places = std::min(P.n_queries, kPrimHeavyMost);
    const size_t want = 16 + static_cast<size_t>(places) * sizeof(PrimHeavy);
    if (!c->pheavy_done) PR_TRY(cudaEventCreateWithFlags(&c->pheavy_done, cudaEventDisableTiming));
    if (want > c->pheavy_cap) {
      cudaFree(c->d_pheavy);
      c->d_pheavy = nullptr;
      c->pheavy_cap = 0;
      if (cudaMalloc(&c->d_pheavy, want) == cudaSuccess) {
        c->pheavy_cap = want;
      } else {
        cudaGetLastError();
        c->d_pheavy = nullptr;
      }
    }
    if (c->d_pheavy) {
      P.heavy_ctr = static_cast<unsigned*>(c->d_pheavy);
      P.heavy = reinterpret_cast<PrimHeavy*>(static_cast<char*>(c->d_pheavy) + 16);
      P.heavy_cap = static_cast<unsigned>(places);
      PR_TRY(cudaStreamWaitEvent(s, c->pheavy_done, 0));
      PR_TRY(cudaMemsetAsync(P.heavy_ctr, 0, 2 * sizeof(unsigned), s));
    }
  }
  prim_trace_kernel<<<static_cast<unsigned>(blocks), kPrimThreads, 0, s>>>(P);
  PR_TRY(cudaGetLastError());
  if (P.heavy) {
    int dev = 0, sms = 0;
    PR_TRY(cudaGetDevice(&dev));
    PR_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t most = (P.n_queries * 32 + kPrimThreads - 1) / kPrimThreads;
    prim_heavy_kernel<<<static_cast<unsigned>(std::min<int64_t>(most, sms * 4)), kPrimThreads, 0, s>>>(P);
    PR_TRY(cudaGetLastError());
    PR_TRY(cudaEventRecord(c->pheavy_done, s));
    ++c->launches;
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ho
