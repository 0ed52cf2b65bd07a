// Host side of the element-major intersection rounds (batched and learned
// modes) and the small kernels between rounds: gather each ray's next
// candidate, bucket the pairs by element (counting sort), cut the buckets
// into batches, and write the final results.
#include <cuda_runtime.h>

#include <algorithm>

#include "ho_check.cuh"
#include "ho_host.h"
#include "ho_rounds.cuh"

namespace ho {

// Exclusive scan of the per-element pair counts in two launches over tiles of
// kScanTile values (1024 threads, 4 consecutive values each): the tiles'
// sums, then every tile's scan from its offset (the sum of the tiles before
// it, which each block adds up itself). One block carrying a running total
// through all the tiles takes time linear in the tile count (0.12 ms per
// round at 262,144 elements under a profiler; in the benchmark's graph the
// difference did not show).
constexpr int kScanTile = 4096;

__device__ __forceinline__ uint32_t block_sum_1024(uint32_t x, uint32_t* wsum) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  if (lane == 0) wsum[wid] = x;
  __syncthreads();
  uint32_t t = lane < 32 ? wsum[lane] : 0u;
  if (wid == 0) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane == 0) wsum[0] = t;
  }
  __syncthreads();
  const uint32_t total = wsum[0];
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(1024) tile_sum_kernel(const uint32_t* __restrict__ in, int64_t len,
                                                        uint32_t* __restrict__ sums) {
  __shared__ uint32_t wsum[32];
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * kScanTile + static_cast<int64_t>(threadIdx.x) * 4;
  uint32_t t = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) t += i0 + k < len ? in[i0 + k] : 0u;
  const uint32_t total = block_sum_1024(t, wsum);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) tile_scan_kernel(const uint32_t* __restrict__ in, int64_t len,
                                                         const uint32_t* __restrict__ sums, uint32_t* __restrict__ out) {
  __shared__ uint32_t wsum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // this tile's offset: the sums of the tiles before it
  uint32_t pre = 0;
  for (unsigned b = threadIdx.x; b < blockIdx.x; b += blockDim.x) pre += sums[b];
  const uint32_t offset = block_sum_1024(pre, wsum);
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * kScanTile + static_cast<int64_t>(threadIdx.x) * 4;
  uint32_t v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = i0 + k < len ? in[i0 + k] : 0u;
  const uint32_t t = v[0] + v[1] + v[2] + v[3];
  uint32_t x = t;  // inclusive scan over the warp
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint32_t ws = wsum[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, ws, off);
      if (lane >= off) ws += y;
    }
    wsum[lane] = ws;
  }
  __syncthreads();
  uint32_t run = offset + (wid > 0 ? wsum[wid - 1] : 0u) + (x - t);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i0 + k < len) out[i0 + k] = run;
    run += v[k];
  }
}

__global__ void round_init_kernel(RayState* __restrict__ st, const uint8_t* __restrict__ kovf,
                                  const unsigned* __restrict__ qcount) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= *qcount) return;
  RayState r;
  r.best = miss_state();
  r.tie = miss_state();
  r.cursor = 0;
  r.pass = 0;
  r.kt = -FLT_MAX;
  r.ke = -1;
  r.done = 0;
  r.ovf = kovf[i];
  r.its = 0;
  r.seen = 0;
  st[i] = r;
}

// One thread per ray in flight: its next ordered candidate whose padded box
// the ray meets before the closest hit so far (the candidate loop of the
// reference's traversal, FEM-AABB/raytracer.cu:117-356, in ascending
// (entry t, element) order). A ray whose list was cut at kCandK walks the
// tree again for the candidates after the last visited one. limit: visited
// candidates of a ray before the tail takes it (0: no tail), counted whether
// they were solved or ended here, so which of the two kernels solves a
// candidate does not depend on how many ended here (their face Newtons
// differ in the last bits on a few rays).
// settle: before the tail, rays go on past the candidates that end here and
// stop before the first that has to be solved (no pairs are written), so the
// tail's list holds only rays with something left to solve.
__global__ void round_gather_kernel(TraceParams P, RayState* __restrict__ st, RoundPair* __restrict__ pairs,
                                    int32_t* __restrict__ pkey, uint32_t* __restrict__ prank,
                                    uint32_t* __restrict__ kcount, unsigned* __restrict__ ctr, int limit,
                                    bool settle) {
  const unsigned item = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  bool live = item < *P.qcount && !st[item].done;
  if (!__any_sync(kFull, live)) return;
  Work w;
  RoundPair p;
  int elem = -1;
  if (live) {
    RayState& r = st[item];
    float3 o, d;
    float iso;
    bool iso_on;
    query_ray(P, P.work[item], o, d, iso, iso_on);
    float2* kb = P.kbuf + static_cast<int64_t>(item) * kCandK;
    const float best_t = r.best.t;
    int cursor = r.cursor, pass = r.pass, ke = r.ke, seen = r.seen;
    float kt = r.kt;
    bool ovf = r.ovf != 0, done = false;
    for (int guard = 0; guard < (1 << 20) && (limit == 0 || seen < limit); ++guard) {
      if (cursor >= kCandK) {
        if (!ovf) {
          done = true;
          break;
        }
        float bt[kCandK];
        int be[kCandK];
        if (!collect(P, o, d, best_t, kt, ke, bt, be, ovf, w)) {
          atomicOr(&P.stats->status, kStatusStackOverflow);
          r.best.flags |= HO_FLAG_INCOMPLETE;
          done = true;
          break;
        }
        for (int j = 0; j < kCandK; ++j) kb[j] = make_float2(bt[j], __int_as_float(be[j]));
        cursor = 0;
        ++pass;
        ++w.restarts;
        r.best.flags |= HO_FLAG_OVERFLOW;
      }
      const float2 c = kb[cursor];
      const float ct = c.x;
      const int ce = __float_as_int(c.y);
      if (ce == INT_MAX || ct > best_t) {
        done = true;
        break;
      }
      const int j = cursor, e0 = ke;
      const float k0 = kt;
      ++cursor;
      kt = ct;
      ke = ce;
      const float* b = P.box + 6 * static_cast<int64_t>(ce);
      const float lo[3] = {__ldg(b), __ldg(b + 1), __ldg(b + 2)};
      const float hi[3] = {__ldg(b + 3), __ldg(b + 4), __ldg(b + 5)};
      float te, tx;
      if (!ray_box(o, d, lo, hi, 0.001f, best_t, te, tx)) continue;
      ++seen;
      // a candidate that can hold neither a root nor a face hit ends here,
      // without a place in a round
      Pred pr;
      pr.on = false;
      if (P.pred && pass == 0 && j < kPredK && item < P.pred_items &&
          P.cand_e[static_cast<int64_t>(item) * kPredK + j] == ce) {
        const float* y = P.pred + (static_cast<int64_t>(item) * kPredK + j) * kMlpOut;
        pr.on = true;
        pr.xi_in = make_float3(y[0], y[1], y[2]);
        pr.v = make_float3(y[3], y[4], y[5]);
        pr.k = __ldg(P.desc + static_cast<int64_t>(ce) * kDescFloats + 45);
        pr.te = te;
      }
      const bool scan = iso_on && needs_iso(P, ce, o, d, te, tx, iso, pr);
      if (!scan && !any_face(P.fbox, ce, o, d, best_t)) {
        ++w.cand;
        w.culled += 6;
        continue;
      }
      if (settle) {
        cursor = j;
        kt = k0;
        ke = e0;
        break;
      }
      p.item = static_cast<int32_t>(item);
      p.j = (pass == 0 ? j : kPairPred) | (scan ? 0 : kPairNoIso);
      p.te = te;
      p.tx = tx;
      elem = ce;
      break;
    }
    r.cursor = cursor;
    r.pass = pass;
    r.kt = kt;
    r.ke = ke;
    r.seen = seen;
    r.ovf = ovf ? 1 : 0;
    if (done) r.done = 1;
  }
  const unsigned m = __ballot_sync(kFull, elem >= 0);
  if (m) {
    const int leader = __ffs(m) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(ctr, static_cast<unsigned>(__popc(m)));
    base = __shfl_sync(kFull, base, leader);
    if (elem >= 0) {
      const unsigned k = base + __popc(m & ((1u << lane) - 1u));
      // element-sorted with the pairs that search for an isosurface apart
      const int key = 2 * elem + (p.j & kPairNoIso ? 0 : 1);
      pairs[k] = p;
      pkey[k] = key;
      prank[k] = atomicAdd(&kcount[key], 1u);
    }
  }
  const unsigned nodes = __reduce_add_sync(kFull, w.nodes), restarts = __reduce_add_sync(kFull, w.restarts),
                 cand = __reduce_add_sync(kFull, w.cand), culled = __reduce_add_sync(kFull, w.culled);
  if (lane == 0) {
    if (nodes) atomicAdd(&P.stats->c[ST_NODES], static_cast<unsigned long long>(nodes));
    if (restarts) atomicAdd(&P.stats->c[ST_RESTART], static_cast<unsigned long long>(restarts));
    if (cand) atomicAdd(&P.stats->c[ST_CAND], static_cast<unsigned long long>(cand));
    if (culled) atomicAdd(&P.stats->c[ST_CULLED], static_cast<unsigned long long>(culled));
  }
}

// Lists rays (all queued ones, or the *n_from of `from`) for the passes after the
// rounds, so that those passes' threads are all busy. flight (or nullptr): the
// rays still in flight, for the tail (counted in the work counters too). The
// others' hits go to the check's list: from its front those that the check's
// shorter path answers, face hits away from the face's edges, from its back the
// others, so that a warp of the check mostly runs one path (a 1920 x 1080
// picture of 3 isovalues, 1.54 M hits: check 4.2 -> 1.9 ms, tie pass 0.51 ->
// 0.43 ms).
__global__ void ray_list_kernel(const unsigned* __restrict__ n_from, const uint32_t* __restrict__ from,
                                const RayState* __restrict__ st, uint32_t* __restrict__ flight,
                                unsigned* __restrict__ n_flight, CheckLists L, DevStats* stats) {
  const int lane = threadIdx.x & 31;
  const unsigned n = *n_from;
  for (uint64_t k = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; (k & ~31ull) < n;
       k += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    int to = -1;  // 0: in flight, 1: front, 2: back
    unsigned i = 0;
    if (k < n) {
      i = from ? from[k] : static_cast<unsigned>(k);
      const HitState& b = st[i].best;
      if (flight && !st[i].done) to = 0;
      else if (b.kind != HO_HIT_MISS) to = b.kind == HO_HIT_FACE && normal_on_face(b.face, b.xi) ? 1 : 2;
    }
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      const unsigned m = __ballot_sync(kFull, to == w);
      if (!m) continue;
      unsigned* ctr = w == 0 ? n_flight : (w == 1 ? L.n_front : L.n_back);
      const int leader = __ffs(m) - 1;
      unsigned base = 0;
      if (lane == leader) {
        base = atomicAdd(ctr, static_cast<unsigned>(__popc(m)));
        if (w == 0) atomicAdd(&stats->c[ST_TAIL], static_cast<unsigned long long>(__popc(m)));
      }
      const unsigned at = __shfl_sync(kFull, base, leader) + __popc(m & ((1u << lane) - 1u));
      if (to == w) (w == 0 ? flight[at] : (w == 1 ? L.list[at] : L.list[L.cap - 1 - at])) = i;
    }
  }
}

// Also tallies the round (non-empty rounds and pairs) into the work counters.
__global__ void round_scatter_kernel(const RoundPair* __restrict__ pairs, const int32_t* __restrict__ pkey,
                                     const uint32_t* __restrict__ prank, const uint32_t* __restrict__ koff,
                                     const unsigned* __restrict__ ctr, RoundPair* __restrict__ sorted,
                                     DevStats* stats) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned n_pairs = *ctr;
  if (k == 0 && n_pairs > 0) {
    atomicAdd(&stats->c[ST_ROUNDS], 1ull);
    atomicAdd(&stats->c[ST_PAIRS], static_cast<unsigned long long>(n_pairs));
  }
  if (k >= n_pairs) return;
  sorted[koff[pkey[k]] + prank[k]] = pairs[k];
}

// Ctr layout: [0] pairs of the round, [4..5] the tail's list count and cursor,
// [6..9] the check's front, back, failure and tie counts, [10..13] the same of
// the check of the tail's rays,
// and per order n (2..9) the batch count, region start, write cursor of the
// face batches, take cursor, and count and write cursor of the isosurface
// batches, which come first in the region.
constexpr int kCtrOrderNb = 16, kCtrOrderOff = 26, kCtrOrderCur = 36, kCtrOrderNext = 46, kCtrIsoNb = 56,
              kCtrIsoCur = 66, kCtrWords = 80;

// Batches per SM that a round's pairs are spread over, before batches grow.
constexpr unsigned kSpreadPerSm = 16;
// HO_OPT_ROUND_CHUNK where it asks for a fixed batch size, else 0. The size that
// the option reports while unset asks for the rule below, so that a program that
// puts an option's value back, or the autotuner when no fixed size is faster,
// does not take the rule from later, smaller calls.
static int fixed_chunk(const ho_context* c) {
  return c->round_chunk == round_batch_default(c->N, c->use_tc) ? 0 : c->round_chunk;
}
// Pairs per batch of a key: the fixed size, else the slots, or fewer while
// the round has less than `spread` full batches (16 warps an SM). A warp's lanes
// are fed by a batch's pairs, so a full batch keeps them busiest; but a round
// that cannot fill the device lasts as long as its longest batch, and a batch of
// one or two pairs, with the warp to itself, is several times shorter. Calls
// before (full batches only) and after: 777 rays 1.81 -> 1.18 ms, a 256 x 256
// picture 3.5 -> 2.5 ms, four path bounces 14.4 -> 12.7 ms; 4 or more batches a
// resident warp change nothing (1920 x 1080: 15.3 ms either way); 64 an SM:
// 2.6 ms and 13.0 ms for the second and third.
__device__ __forceinline__ int batch_size(int chunk, int order, bool tc, bool faces, unsigned pairs, unsigned spread) {
  if (chunk > 0) return chunk;
  const int most = faces ? face_slots(order) : round_batch_default(order, tc);
  return tc ? most : max(1, min(most, static_cast<int>((pairs + spread - 1) / spread)));
}
// Does a key's batch take the face layout?
__device__ __forceinline__ bool face_batch(int64_t key, bool tc, const float* __restrict__ cull) {
  return !tc && !(key & 1) && __ldg(cull + (key >> 1) * kCullFloats + 12) >= 0.f;
}

// Batches per order: a key's pairs (key 2 e: element e's pairs without an
// isosurface search, 2 e + 1: with one) in batches of its element's order's
// size. A warp step costs what its most expensive lane does, an isosurface
// sample several times a face step, so the two kinds share no batch; the
// isosurface batches, the longer ones, come first.
__global__ void round_batch_count_kernel(const uint32_t* __restrict__ kcount, const uint8_t* __restrict__ order,
                                         const float* __restrict__ cull, int64_t n_elem, int chunk, bool tc,
                                         unsigned spread, unsigned* __restrict__ ctr) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= 2 * n_elem) return;
  const int c = static_cast<int>(kcount[k]);
  if (c == 0) return;
  const int n = order[k >> 1];
  const int B = batch_size(chunk, n, tc, face_batch(k, tc, cull), ctr[0], spread);
  const unsigned nb = static_cast<unsigned>((c + B - 1) / B);
  atomicAdd(&ctr[kCtrOrderNb + n], nb);
  if (k & 1) atomicAdd(&ctr[kCtrIsoNb + n], nb);
}

// Region start of each order's batches (orders in increasing n).
__global__ void round_order_offsets_kernel(unsigned* __restrict__ ctr) {
  unsigned run = 0;
  for (int n = 0; n < 10; ++n) {
    ctr[kCtrOrderOff + n] = run;
    ctr[kCtrOrderCur + n] = ctr[kCtrIsoNb + n];
    ctr[kCtrIsoCur + n] = 0;
    ctr[kCtrOrderNext + n] = 0;
    run += ctr[kCtrOrderNb + n];
  }
}

// Each key's pairs in batches, written into its order's region.
__global__ void round_batch_kernel(const uint32_t* __restrict__ kcount, const uint32_t* __restrict__ koff,
                                   const uint8_t* __restrict__ order, const float* __restrict__ cull, int64_t n_elem,
                                   int chunk, bool tc, unsigned spread, RoundBatch* __restrict__ batches,
                                   unsigned* __restrict__ ctr) {
  const int64_t key = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (key >= 2 * n_elem) return;
  const int c = static_cast<int>(kcount[key]);
  if (c == 0) return;
  const int n = order[key >> 1];
  const bool faces = face_batch(key, tc, cull);
  const int B = batch_size(chunk, n, tc, faces, ctr[0], spread);
  const int nb = (c + B - 1) / B;
  const unsigned base = ctr[kCtrOrderOff + n] + atomicAdd(&ctr[(key & 1 ? kCtrIsoCur : kCtrOrderCur) + n],
                                                          static_cast<unsigned>(nb));
  for (int k = 0; k < nb; ++k) {
    RoundBatch bt;
    bt.elem = static_cast<int32_t>(key >> 1);
    bt.first = static_cast<int32_t>(koff[key]) + k * B;
    bt.count = min(B, c - k * B);
    bt.faces = faces ? 1 : 0;
    batches[base + k] = bt;
  }
}

// The queued rays' answers into the call's outputs, and the count of the grazing
// hits.
__global__ void round_finish_kernel(TraceParams P, const RayState* __restrict__ st) {
  const unsigned item = blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= *P.qcount) return;
  const int64_t q = P.work[item];
  float3 o, d;
  float iso;
  bool iso_on;
  query_ray(P, q, o, d, iso, iso_on);
  const HitState& b = st[item].best;
  write_result(P, q, d, b, static_cast<uint32_t>(st[item].its));
  const unsigned act = __activemask();
  const unsigned g = __ballot_sync(act, is_grazing(b, d));
  if (g && static_cast<int>(threadIdx.x & 31) == __ffs(act) - 1)
    atomicAdd(&P.stats->c[ST_GRAZING], static_cast<unsigned long long>(__popc(g)));
}

// Grow-only device buffer of `want` elements of `size` bytes.
template <typename T>
static cudaError_t grow(T*& p, size_t& cap, size_t want, size_t size) {
  if (p && cap >= want) return cudaSuccess;
  cudaFree(p);
  p = nullptr;
  cap = 0;
  void* q = nullptr;
  const cudaError_t e = cudaMalloc(&q, std::max<size_t>(want, 1) * size);
  if (e == cudaSuccess) {
    p = static_cast<T*>(q);
    cap = want;
  }
  return e;
}

#define RT_TRY(x)                        \
  do {                                   \
    const cudaError_t e_ = (x);          \
    if (e_ != cudaSuccess) return int(e_); \
  } while (0)

static int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Scratch for up to n_cap queued rays (all queries of the call), allocated
// before any stream capture.
int prepare_rounds(ho_context* c, int64_t n_cap) {
  const size_t n = static_cast<size_t>(std::max<int64_t>(n_cap, 1));
  const int64_t n_elem = c->n_elem;
  RoundBufs& rb = c->rounds;
  RT_TRY(grow(rb.state, rb.state_cap, n, sizeof(RayState)));
  RT_TRY(grow(rb.pairs, rb.pairs_cap, 2 * n, sizeof(RoundPair)));
  RT_TRY(grow(rb.pkey, rb.pkey_cap, n, sizeof(int32_t)));
  RT_TRY(grow(rb.prank, rb.prank_cap, n, sizeof(uint32_t)));
  RT_TRY(grow(rb.batches, rb.batches_cap, n, sizeof(RoundBatch)));
  RT_TRY(grow(rb.kcount, rb.kcount_cap, static_cast<size_t>(2 * n_elem), sizeof(uint32_t)));
  RT_TRY(grow(rb.koff, rb.koff_cap, static_cast<size_t>(2 * n_elem), sizeof(uint32_t)));
  RT_TRY(grow(rb.tile_sums, rb.tile_sums_cap, static_cast<size_t>((2 * n_elem + kScanTile - 1) / kScanTile),
              sizeof(uint32_t)));
  RT_TRY(grow(rb.ctr, rb.ctr_cap, kCtrWords, sizeof(unsigned)));
  RT_TRY(grow(rb.fail, rb.fail_cap, n, sizeof(uint32_t)));
  if (!c->check_stream) RT_TRY(cudaStreamCreateWithFlags(&c->check_stream, cudaStreamNonBlocking));
  if (!c->check_fork) RT_TRY(cudaEventCreateWithFlags(&c->check_fork, cudaEventDisableTiming));
  if (!c->check_done) RT_TRY(cudaEventCreateWithFlags(&c->check_done, cudaEventDisableTiming));
  if (__builtin_popcount(c->orders) > 1) {  // streams and events of the orders' launches
    if (!c->order_fork) RT_TRY(cudaEventCreateWithFlags(&c->order_fork, cudaEventDisableTiming));
    for (int m = kMinModes; m <= kMaxModes; ++m) {
      if (!c->order_streams[m]) RT_TRY(cudaStreamCreateWithFlags(&c->order_streams[m], cudaStreamNonBlocking));
      if (!c->order_done[m]) RT_TRY(cudaEventCreateWithFlags(&c->order_done[m], cudaEventDisableTiming));
    }
  }
  return 0;
}

// The check's residuals for caller-given hits (ho_hit_residuals).
int launch_residuals(ho_context* c, int64_t n, const float* rays, const ho_hit* hits, double* out, cudaStream_t s) {
  cudaError_t e;
  switch (c->N) {
    case 2: e = launch_residuals_n<2>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 3: e = launch_residuals_n<3>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 4: e = launch_residuals_n<4>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 5: e = launch_residuals_n<5>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 6: e = launch_residuals_n<6>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 7: e = launch_residuals_n<7>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 8: e = launch_residuals_n<8>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    case 9: e = launch_residuals_n<9>(c->d_rec, c->d_flags, n, rays, hits, out, s); break;
    default: e = cudaErrorInvalidValue; break;
  }
  return int(e);
}

// Scratch of the check's launches: in the pair-key and failure buffers, or, for
// the rays that the tail finished (second), in the pair buffer. All are idle
// after the rounds. The counters are to be zeroed.
static CheckLists check_lists(ho_context* c, int64_t n_cap, bool second) {
  RoundBufs& rb = c->rounds;
  CheckLists L;
  L.cap = n_cap;
  L.list = second ? static_cast<uint32_t*>(rb.pairs) : reinterpret_cast<uint32_t*>(rb.pkey);
  L.fail = second ? static_cast<uint32_t*>(rb.pairs) + n_cap : rb.fail;
  unsigned* ctr = rb.ctr + (second ? 10 : 6);
  L.n_front = ctr;
  L.n_back = ctr + 1;
  L.n_fail = ctr + 2;
  L.n_tie = ctr + 3;
  return L;
}
static_assert(2 * sizeof(RoundPair) >= 2 * sizeof(uint32_t), "the pair buffer holds two lists");

// FP64 check of the listed rays' hits, plain fallback of the failures; without
// the check, the hits are only completed.
static int enqueue_check(ho_context* c, const TraceParams& P, const RoundParams& R, const CheckLists& L, cudaStream_t s,
                         int64_t threads) {
  cudaError_t e;
  if (!c->fp64_check) {
    c->launches += 1;
    switch (c->N) {
      case 2: e = launch_post_n<2>(P, R.state, L, threads, s); break;
      case 3: e = launch_post_n<3>(P, R.state, L, threads, s); break;
      case 4: e = launch_post_n<4>(P, R.state, L, threads, s); break;
      case 5: e = launch_post_n<5>(P, R.state, L, threads, s); break;
      case 6: e = launch_post_n<6>(P, R.state, L, threads, s); break;
      case 7: e = launch_post_n<7>(P, R.state, L, threads, s); break;
      case 8: e = launch_post_n<8>(P, R.state, L, threads, s); break;
      case 9: e = launch_post_n<9>(P, R.state, L, threads, s); break;
      default: e = cudaErrorInvalidValue; break;
    }
    return int(e);
  }
  c->launches += 3;  // check, tie rule, fallback
  const int sms = sm_count();
  switch (c->N) {
    case 2: e = launch_check_n<2>(P, R.state, L, threads, sms, s); break;
    case 3: e = launch_check_n<3>(P, R.state, L, threads, sms, s); break;
    case 4: e = launch_check_n<4>(P, R.state, L, threads, sms, s); break;
    case 5: e = launch_check_n<5>(P, R.state, L, threads, sms, s); break;
    case 6: e = launch_check_n<6>(P, R.state, L, threads, sms, s); break;
    case 7: e = launch_check_n<7>(P, R.state, L, threads, sms, s); break;
    case 8: e = launch_check_n<8>(P, R.state, L, threads, sms, s); break;
    case 9: e = launch_check_n<9>(P, R.state, L, threads, sms, s); break;
    default: e = cudaErrorInvalidValue; break;
  }
  return int(e);
}

// The check of every queued ray with a hit.
static int enqueue_check_all(ho_context* c, const TraceParams& P, const RoundParams& R, cudaStream_t s, int64_t n_cap) {
  const CheckLists L = check_lists(c, n_cap, false);
  RT_TRY(cudaMemsetAsync(L.n_front, 0, 4 * sizeof(unsigned), s));
  ray_list_kernel<<<static_cast<unsigned>((n_cap + 255) / 256), 256, 0, s>>>(P.qcount, nullptr, R.state, nullptr, nullptr,
                                                                             L, P.stats);
  RT_TRY(cudaGetLastError());
  ++c->launches;
  return enqueue_check(c, P, R, L, s, n_cap);
}

static RoundParams round_params(ho_context* c, const TraceParams& P) {
  RoundBufs& rb = c->rounds;
  RoundParams R;
  R.rec = P.rec;
  R.fbox = P.fbox;
  R.flags = P.flags;
  R.cull = P.cull;
  R.rays = P.rays;
  R.n_rays = P.n_rays;
  R.cam = P.cam;
  for (int i = 0; i < 8; ++i) R.iso[i] = P.iso[i];
  R.iso_on_mask = P.iso_on_mask;
  R.views = P.views;
  R.n_views = P.n_views;
  R.work = P.work;
  R.state = static_cast<RayState*>(rb.state);
  R.pairs = static_cast<RoundPair*>(rb.pairs) + rb.pairs_cap / 2;
  R.batches = static_cast<RoundBatch*>(rb.batches);
  R.batch_base = rb.ctr + kCtrOrderOff + c->N;
  R.n_batches = rb.ctr + kCtrOrderNb + c->N;
  R.next_batch = rb.ctr + kCtrOrderNext + c->N;
  R.crec = c->d_crec;
  R.coff = c->d_coff;
  R.stats = P.stats;
  R.desc = P.desc;
  R.cand_e = P.cand_e;
  R.pred = P.pred;
  R.pred_items = P.pred_items;
  R.warm_cap = c->warm_cap;
  return R;
}

// Records an event on s; inside a stream capture the event becomes an event
// record node of the graph, so its time is taken when the graph runs.
static cudaError_t record_event(cudaEvent_t ev, cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &cs);
  if (e != cudaSuccess) return e;
  return cudaEventRecordWithFlags(ev, s, cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal
                                                                               : cudaEventRecordDefault);
}

// The next pair of timing events of this call (created on first use).
static cudaError_t next_events(ho_context* c, cudaEvent_t* a, cudaEvent_t* b) {
  while (static_cast<int>(c->round_events.size()) < c->round_events_used + 2) {
    cudaEvent_t ev = nullptr;
    const cudaError_t e = cudaEventCreate(&ev);
    if (e != cudaSuccess) return e;
    c->round_events.push_back(ev);
  }
  *a = c->round_events[c->round_events_used];
  *b = c->round_events[c->round_events_used + 1];
  c->round_events_used += 2;
  return cudaSuccess;
}

// One round: gather each ray's next pair, bucket by element, intersect. Every
// launch has a fixed size and reads its counts on the device, so rounds can
// be enqueued (and captured) without reading anything back.
static int enqueue_round(ho_context* c, const TraceParams& P, const RoundParams& R, cudaStream_t s, bool learned,
                         int64_t n_cap, int limit) {
  RoundBufs& rb = c->rounds;
  const int64_t n_elem = c->n_elem;
  RoundPair* gathered = static_cast<RoundPair*>(rb.pairs);
  const unsigned gi = static_cast<unsigned>((n_cap + 255) / 256);
  const int64_t n_keys = 2 * n_elem;
  RT_TRY(cudaMemsetAsync(rb.kcount, 0, static_cast<size_t>(n_keys) * sizeof(uint32_t), s));
  RT_TRY(cudaMemsetAsync(rb.ctr, 0, kCtrWords * sizeof(unsigned), s));
  round_gather_kernel<<<gi, 256, 0, s>>>(P, R.state, gathered, rb.pkey, rb.prank, rb.kcount, rb.ctr, limit,
                                      false);
  {
    const unsigned tiles = static_cast<unsigned>((n_keys + kScanTile - 1) / kScanTile);
    if (tiles > 0) {
      tile_sum_kernel<<<tiles, 1024, 0, s>>>(rb.kcount, n_keys, rb.tile_sums);
      tile_scan_kernel<<<tiles, 1024, 0, s>>>(rb.kcount, n_keys, rb.tile_sums, rb.koff);
    }
  }
  round_scatter_kernel<<<gi, 256, 0, s>>>(gathered, rb.pkey, rb.prank, rb.koff, rb.ctr,
                                          const_cast<RoundPair*>(R.pairs), P.stats);
  const unsigned ge = static_cast<unsigned>((n_keys + 255) / 256);
  // with the network's predictions, a solve's restarts depend on what else its
  // warp runs: full batches for every call size
  const unsigned spread = learned ? 1u : kSpreadPerSm * static_cast<unsigned>(sm_count());
  const int chunk = fixed_chunk(c);
  round_batch_count_kernel<<<ge, 256, 0, s>>>(rb.kcount, c->d_cord, c->d_cull, n_elem, chunk, c->use_tc, spread, rb.ctr);
  round_order_offsets_kernel<<<1, 1, 0, s>>>(rb.ctr);
  round_batch_kernel<<<ge, 256, 0, s>>>(rb.kcount, rb.koff, c->d_cord, c->d_cull, n_elem, chunk, c->use_tc, spread,
                                        const_cast<RoundBatch*>(R.batches), rb.ctr);
  RT_TRY(cudaGetLastError());
  c->launches += 7 + __builtin_popcount(c->orders);
  // One launch per element order present in the scene. Each ends with a few
  // warps on its longest pairs; on streams of their own (in a captured call,
  // branches of the graph) one order's blocks take the room that another's
  // leave, where one after the other each would wait for the last pair before.
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  if (c->time_rounds) {
    RT_TRY(next_events(c, &t0, &t1));
    RT_TRY(record_event(t0, s));
  }
  const bool fork = __builtin_popcount(c->orders) > 1;
  if (fork) RT_TRY(cudaEventRecord(c->order_fork, s));
  cudaError_t e = cudaSuccess;
  bool first = true;
  for (int n = kMaxModes; n >= kMinModes && e == cudaSuccess; --n) {
    if (!((c->orders >> n) & 1u)) continue;
    RoundParams Rn = R;
    Rn.batch_base = rb.ctr + kCtrOrderOff + n;
    Rn.n_batches = rb.ctr + kCtrOrderNb + n;
    Rn.next_batch = rb.ctr + kCtrOrderNext + n;
    // the first (largest) order stays on the call's stream
    cudaStream_t so = first ? s : c->order_streams[n];
    if (!first) RT_TRY(cudaStreamWaitEvent(so, c->order_fork, 0));
    switch (n) {
      case 2: e = launch_round_n<2>(Rn, so, learned, c->use_tc); break;
      case 3: e = launch_round_n<3>(Rn, so, learned, c->use_tc); break;
      case 4: e = launch_round_n<4>(Rn, so, learned, c->use_tc); break;
      case 5: e = launch_round_n<5>(Rn, so, learned, c->use_tc); break;
      case 6: e = launch_round_n<6>(Rn, so, learned, c->use_tc); break;
      case 7: e = launch_round_n<7>(Rn, so, learned, c->use_tc); break;
      case 8: e = launch_round_n<8>(Rn, so, learned, c->use_tc); break;
      case 9: e = launch_round_n<9>(Rn, so, learned, c->use_tc); break;
      default: e = cudaErrorInvalidValue; break;
    }
    if (!first && e == cudaSuccess) e = cudaEventRecord(c->order_done[n], so);
    if (!first && e == cudaSuccess) e = cudaStreamWaitEvent(s, c->order_done[n], 0);
    first = false;
  }
  RT_TRY(e);
  if (t1) RT_TRY(record_event(t1, s));
  return 0;
}

// The tail and the check: every ray still in flight is finished by the
// warp-per-ray kernel; afterwards no round has pairs left (ctr[0] = 0). The tail
// is a few long chains that leave most of the device idle, so the check of the
// rays that the rounds finished runs beside it, on a stream of its own (a branch
// of the graph in a captured call); the tail's rays are checked after it. The
// tail is enqueued first: its blocks then have their places, and the check's
// fill the rest.
static int enqueue_tail_and_check(ho_context* c, const TraceParams& P, const RoundParams& R, cudaStream_t s, bool learned,
                                  int64_t n_cap) {
  RoundBufs& rb = c->rounds;
  unsigned* n_list = rb.ctr + 4;
  unsigned* next = rb.ctr + 5;
  const unsigned gi = static_cast<unsigned>((n_cap + 255) / 256);
  const CheckLists first = check_lists(c, n_cap, false), second = check_lists(c, n_cap, true);
  RT_TRY(cudaMemsetAsync(rb.ctr + 4, 0, 10 * sizeof(unsigned), s));
  round_gather_kernel<<<gi, 256, 0, s>>>(P, R.state, static_cast<RoundPair*>(rb.pairs), rb.pkey, rb.prank, rb.kcount,
                                         rb.ctr, 0, true);
  ray_list_kernel<<<gi, 256, 0, s>>>(P.qcount, nullptr, R.state, rb.prank, n_list, first, P.stats);
  RT_TRY(cudaGetLastError());
  RT_TRY(cudaEventRecord(c->check_fork, s));
  cudaError_t e;
  switch (c->N) {
    case 2: e = launch_tail_n<2>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 3: e = launch_tail_n<3>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 4: e = launch_tail_n<4>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 5: e = launch_tail_n<5>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 6: e = launch_tail_n<6>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 7: e = launch_tail_n<7>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 8: e = launch_tail_n<8>(P, R.state, rb.prank, n_list, next, learned, s); break;
    case 9: e = launch_tail_n<9>(P, R.state, rb.prank, n_list, next, learned, s); break;
    default: e = cudaErrorInvalidValue; break;
  }
  RT_TRY(e);
  RT_TRY(cudaStreamWaitEvent(c->check_stream, c->check_fork, 0));
  int rc = enqueue_check(c, P, R, first, c->check_stream, n_cap);
  RT_TRY(cudaEventRecord(c->check_done, c->check_stream));
  if (rc) return rc;
  const int64_t few = std::min<int64_t>(n_cap, static_cast<int64_t>(sm_count()) * 1024);
  ray_list_kernel<<<static_cast<unsigned>((few + 255) / 256), 256, 0, s>>>(n_list, rb.prank, R.state, nullptr, nullptr,
                                                                           second, P.stats);
  RT_TRY(cudaGetLastError());
  rc = enqueue_check(c, P, R, second, s, few);
  if (rc) return rc;
  RT_TRY(cudaStreamWaitEvent(s, c->check_done, 0));
  RT_TRY(cudaMemsetAsync(rb.ctr, 0, sizeof(unsigned), s));
  c->launches += 4;
  return 0;
}

// The state init and `rounds` rounds, then, with the tail, the tail, the check
// and the final write-out of the queued rays. Without it rays may still be in
// flight after the rounds, and finish_rounds ends the call.
int enqueue_rounds(ho_context* c, const TraceParams& P, cudaStream_t s, bool learned, int64_t n_cap, int rounds) {
  const RoundParams R = round_params(c, P);
  const unsigned gi = static_cast<unsigned>((n_cap + 255) / 256);
  round_init_kernel<<<gi, 256, 0, s>>>(R.state, P.kovf, P.qcount);
  RT_TRY(cudaGetLastError());
  c->launches += 2;  // init and finish
  // with the tail, a fixed number of rounds (the tail finishes every ray)
  if (c->tail_after > 0) rounds = std::min(c->round_count, c->tail_after);
  for (int r = 0; r < rounds; ++r) {
    const int rc = enqueue_round(c, P, R, s, learned, n_cap, c->tail_after > 0 ? rounds : 0);
    if (rc) return rc;
  }
  if (c->tail_after == 0) return 0;
  const int rc = enqueue_tail_and_check(c, P, R, s, learned, n_cap);
  if (rc) return rc;
  round_finish_kernel<<<gi, 256, 0, s>>>(P, R.state);
  RT_TRY(cudaGetLastError());
  return 0;
}

// After the enqueued rounds ran: without the tail, one more round while the last
// one still found pairs (with a read-back each), then the check and the final
// write-out. The check polishes a ray's hit, and a ray in flight compares its
// next candidates with that hit, so no ray is checked before all are done: its
// answer would depend on how many rounds the call before had needed.
int finish_rounds(ho_context* c, const TraceParams& P, cudaStream_t s, bool learned, int64_t n_cap) {
  const RoundParams R = round_params(c, P);
  for (int guard = 0; guard < 100000; ++guard) {
    unsigned last = 0;
    unsigned long long rounds = 0;
    RT_TRY(cudaMemcpyAsync(&last, c->rounds.ctr, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    RT_TRY(cudaMemcpyAsync(&rounds, &P.stats->c[ST_ROUNDS], sizeof(rounds), cudaMemcpyDeviceToHost, s));
    RT_TRY(cudaStreamSynchronize(s));
    c->rounds_needed = static_cast<int>(rounds);
    if (last == 0) break;
    const int rc = enqueue_round(c, P, R, s, learned, n_cap, 0);
    if (rc) return rc;
  }
  if (c->tail_after > 0) return 0;
  const int rc = enqueue_check_all(c, P, R, s, n_cap);
  if (rc) return rc;
  round_finish_kernel<<<static_cast<unsigned>((n_cap + 255) / 256), 256, 0, s>>>(P, R.state);
  RT_TRY(cudaGetLastError());
  return 0;
}

}  // namespace ho
