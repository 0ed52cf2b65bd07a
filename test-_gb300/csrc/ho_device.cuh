// Device-side element math for curved hexahedra with Modified-A modal
// geometry and field. All arithmetic FP32; templated on N = modes per
// direction so every tensor loop unrolls.
//
// Algorithm steps follow the reference's per-element functions
// (paths relative to the reference project root):
//   basis            FEM-AABB/fem/ModalBasis.cuh:16-70
//   map / Jacobian   FEM-AABB/fem/HexElement.cu:8-206  (here sum-factorised)
//   inverse map      FEM-AABB/fem/HexElement.cu:227-272
//   field, gradient  FEM-AABB/fem/HexElement.cu:274-330
//   isosurface scan  FEM-AABB/fem/RayIsosurface.cu:44-188
//   padded box       FEM-AABB/high_order.h:51-113
//   slab test        FEM-AABB/high_order.h:115-152
//   face Newton      FEM-AABB/high_order.h:164-304
//   nearest face     FEM-AABB/high_order.h:409-465
//   hex hit policy   FEM-AABB/raytracer.cu:184-254
#pragma once

#include <cfloat>
#include <cstdint>

#include "ho_layout.h"

namespace ho {

// ---------------------------------------------------------------------------
// Work counters kept in registers per thread and flushed once per thread.
// ---------------------------------------------------------------------------
struct Work {
  uint32_t cand = 0, geom = 0, map = 0, field = 0, newton = 0, face = 0, culled = 0, nodes = 0, restarts = 0;
  uint32_t accepted = 0, rejected = 0;
  // SM cycles by phase (warp kernels, counted on lane 0): traversal, isosurface
  // scan, bracket refinement, face search
  unsigned long long cyc[4] = {0, 0, 0, 0};
  // round kernel: loop steps and busy lanes over them (counted on lane 0)
  unsigned long long steps = 0, lanes = 0;
  // round kernel: algorithmic FP32 flops of the evaluations and solves done
  unsigned long long flops = 0;
};

// Algorithmic flops of one sum-factorised point evaluation of `comps`
// components (value and three partials each) at n modes per direction: the
// 1-D basis values and derivatives (3 x 8n) plus 2(2n^3 + 3n^2 + 4n) per
// component; and of one 3x3 Newton solve and update.
__host__ __device__ constexpr unsigned long long eval_flops(int n, int comps) {
  return 3ull * 8 * n + 2ull * comps * (2ull * n * n * n + 3ull * n * n + 4ull * n);
}
constexpr unsigned long long kSolveFlops = 60;
// One evaluation on a face (face_eval): two axes' basis values, and per
// component 4n^2 + 6n.
__host__ __device__ constexpr unsigned long long face_eval_flops(int n) {
  return 2ull * 8 * n + 3ull * (4ull * n * n + 6ull * n);
}

// ---------------------------------------------------------------------------
// 1-D Modified-A basis: phi_0 = (1-x)/2, phi_1 = (1+x)/2,
// phi_i = (1-x^2)/4 * P^{(1,1)}_{i-2}(x). P^{(1,1)} by the three-term
// recurrence P_m = A_m x P_{m-1} - B_m P_{m-2}, A_m = (2m+1)(m+1)/(m(m+2)),
// B_m = (m+1)/(m+2), P_0 = 1, P_1 = 2x (the alpha = beta = 1 case of the
// general recurrence in ModalBasis.cuh:16-41); derivatives by differentiating
// the same recurrence.
// ---------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void basis_val(float x, float (&a)[N]) {
  a[0] = 0.5f * (1.0f - x);
  if (N > 1) a[1] = 0.5f * (1.0f + x);
  const float w = 0.25f * (1.0f - x * x);
  float pm2 = 1.0f, pm1 = 2.0f * x;
#pragma unroll
  for (int i = 2; i < N; ++i) {
    const int m = i - 2;
    float p;
    if (m == 0) p = 1.0f;
    else if (m == 1) p = pm1;
    else {
      const float A = float((2 * m + 1) * (m + 1)) / float(m * (m + 2));
      const float B = float(m + 1) / float(m + 2);
      p = A * x * pm1 - B * pm2;
      pm2 = pm1;
      pm1 = p;
    }
    a[i] = w * p;
  }
}

template <int N>
__device__ __forceinline__ void basis_val_der(float x, float (&a)[N], float (&d)[N]) {
  a[0] = 0.5f * (1.0f - x);
  d[0] = -0.5f;
  if (N > 1) {
    a[1] = 0.5f * (1.0f + x);
    d[1] = 0.5f;
  }
  const float w = 0.25f * (1.0f - x * x);
  const float hx = -0.5f * x;
  float pm2 = 1.0f, pm1 = 2.0f * x, qm2 = 0.0f, qm1 = 2.0f;
#pragma unroll
  for (int i = 2; i < N; ++i) {
    const int m = i - 2;
    float p, q;
    if (m == 0) {
      p = 1.0f;
      q = 0.0f;
    } else if (m == 1) {
      p = pm1;
      q = qm1;
    } else {
      const float A = float((2 * m + 1) * (m + 1)) / float(m * (m + 2));
      const float B = float(m + 1) / float(m + 2);
      p = A * x * pm1 - B * pm2;
      q = A * (pm1 + x * qm1) - B * qm2;
      pm2 = pm1;
      pm1 = p;
      qm2 = qm1;
      qm1 = q;
    }
    a[i] = w * p;
    d[i] = hx * p + w * q;
  }
}

// ---------------------------------------------------------------------------
// Sum-factorised tensor contractions. Coefficient index ((k*N)+j)*N+i,
// i fastest (HexElement.cu:14-26). One component per call.
//
// Code size matters more than call overhead here: a fully unrolled N^3
// contraction is thousands of instructions, and inlining it at every call
// site overflows the instruction cache. So the i and j loops are unrolled
// (basis values in registers), the k loop is rolled (its basis values come
// from the caller's per-lane local array), and the routines are out of line.
// ---------------------------------------------------------------------------
template <int N>
struct Basis {
  float ar[N], dr[N], as[N], ds[N], at[N], dt[N];
};

// Where an element record lives: global memory (read-only path) or a warp's
// shared-memory staging slot. Offsets are in floats.
template <bool SM>
struct CoefRef;
template <>
struct CoefRef<false> {
  const float* __restrict__ p;
  __device__ __forceinline__ float4 ld4(int off) const { return __ldg(reinterpret_cast<const float4*>(p + off)); }
  __device__ __forceinline__ float ld(int off) const { return __ldg(p + off); }
  __device__ __forceinline__ CoefRef at(int off) const { return CoefRef{p + off}; }
};
template <>
struct CoefRef<true> {
  uint32_t a;  // shared-space byte address
  __device__ __forceinline__ float4 ld4(int off) const {
    float4 v;
    asm("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a + 4u * off));
    return v;
  }
  __device__ __forceinline__ float ld(int off) const {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a + 4u * off));
    return v;
  }
  __device__ __forceinline__ CoefRef at(int off) const { return CoefRef{a + 4u * static_cast<uint32_t>(off)}; }
};

// One coefficient row (N values) into registers, RS/4 vector loads.
template <int N, bool SM>
__device__ __forceinline__ void load_row(const CoefRef<SM>& c, int off, float (&r)[row_stride(N)]) {
#pragma unroll
  for (int q = 0; q < row_stride(N) / 4; ++q) {
    const float4 v = c.ld4(off + 4 * q);
    r[4 * q] = v.x;
    r[4 * q + 1] = v.y;
    r[4 * q + 2] = v.z;
    r[4 * q + 3] = v.w;
  }
}

// value and the three reference-space partials: out = {v, dv/dr, dv/ds, dv/dt}
template <int N, bool SM>
__device__ __noinline__ void contract_vd(CoefRef<SM> c, const Basis<N>* __restrict__ B, float* __restrict__ out) {
  constexpr int RS = row_stride(N);
  float ar[N], dr[N], as[N], ds[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    ar[i] = B->ar[i];
    dr[i] = B->dr[i];
    as[i] = B->as[i];
    ds[i] = B->ds[i];
  }
  float v = 0.f, vr = 0.f, vs = 0.f, vt = 0.f;
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    const float tk = B->at[k], dtk = B->dt[k];
    float q0 = 0.f, q1 = 0.f, q2 = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      float row[RS];
      load_row<N, SM>(c, (k * N + j) * RS, row);
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        s0 = fmaf(row[i], ar[i], s0);
        s1 = fmaf(row[i], dr[i], s1);
      }
      q0 = fmaf(s0, as[j], q0);
      q1 = fmaf(s1, as[j], q1);
      q2 = fmaf(s0, ds[j], q2);
    }
    v = fmaf(q0, tk, v);
    vr = fmaf(q1, tk, vr);
    vs = fmaf(q2, tk, vs);
    vt = fmaf(q0, dtk, vt);
  }
  out[0] = v;
  out[1] = vr;
  out[2] = vs;
  out[3] = vt;
}

// value only
template <int N, bool SM>
__device__ __noinline__ float contract_v(CoefRef<SM> c, const Basis<N>* __restrict__ B) {
  constexpr int RS = row_stride(N);
  float ar[N], as[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    ar[i] = B->ar[i];
    as[i] = B->as[i];
  }
  float v = 0.0f;
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    const float tk = B->at[k];
    float q0 = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      float row[RS];
      load_row<N, SM>(c, (k * N + j) * RS, row);
      float s0 = 0.f;
#pragma unroll
      for (int i = 0; i < N; ++i) s0 = fmaf(row[i], ar[i], s0);
      q0 = fmaf(s0, as[j], q0);
    }
    v = fmaf(q0, tk, v);
  }
  return v;
}

// Element record (record_floats(N) floats): x, y, z geometry blocks then the
// field block, in global memory (SM = false) or a shared-memory slot.
template <int N, bool SM = false>
struct Elem {
  CoefRef<SM> c;
  bool has_field;
  __device__ __forceinline__ CoefRef<SM> fld() const { return c.at(3 * block_floats(N)); }
};

// x(xi) and J (row-major J[row=x,y,z][col=r,s,t]).
template <int N, bool SM>
__device__ __noinline__ void geom_eval_raw(CoefRef<SM> c, float3 xi, float* __restrict__ xJ) {
  Basis<N> B;
  basis_val_der<N>(xi.x, B.ar, B.dr);
  basis_val_der<N>(xi.y, B.as, B.ds);
  basis_val_der<N>(xi.z, B.at, B.dt);
#pragma unroll 1
  for (int comp = 0; comp < 3; ++comp) contract_vd<N, SM>(c.at(comp * block_floats(N)), &B, xJ + 4 * comp);
}

template <int N, bool SM>
__device__ __forceinline__ void geom_eval(const Elem<N, SM>& e, float3 xi, float3& x, float (&J)[9], Work& w) {
  float r[12];
  geom_eval_raw<N, SM>(e.c, xi, r);
  x = make_float3(r[0], r[4], r[8]);
  J[0] = r[1]; J[1] = r[2]; J[2] = r[3];
  J[3] = r[5]; J[4] = r[6]; J[5] = r[7];
  J[6] = r[9]; J[7] = r[10]; J[8] = r[11];
  ++w.geom;
}

template <int N, bool SM>
__device__ __noinline__ float3 geom_map_raw(CoefRef<SM> c, float3 xi) {
  Basis<N> B;
  basis_val<N>(xi.x, B.ar);
  basis_val<N>(xi.y, B.as);
  basis_val<N>(xi.z, B.at);
  const float x = contract_v<N, SM>(c, &B);
  const float y = contract_v<N, SM>(c.at(block_floats(N)), &B);
  const float z = contract_v<N, SM>(c.at(2 * block_floats(N)), &B);
  return make_float3(x, y, z);
}

template <int N, bool SM>
__device__ __forceinline__ float3 geom_map(const Elem<N, SM>& e, float3 xi, Work& w) {
  ++w.map;
  return geom_map_raw<N, SM>(e.c, xi);
}

// u(xi) and grad_xi u
template <int N, bool SM>
__device__ __noinline__ void field_eval_raw(CoefRef<SM> c, float3 xi, float* __restrict__ ug) {
  Basis<N> B;
  basis_val_der<N>(xi.x, B.ar, B.dr);
  basis_val_der<N>(xi.y, B.as, B.ds);
  basis_val_der<N>(xi.z, B.at, B.dt);
  contract_vd<N, SM>(c, &B, ug);
}

template <int N, bool SM>
__device__ __forceinline__ void field_eval(const Elem<N, SM>& e, float3 xi, float& u, float3& g, Work& w) {
  float r[4];
  field_eval_raw<N, SM>(e.fld(), xi, r);
  u = r[0];
  g = make_float3(r[1], r[2], r[3]);
  ++w.field;
}

template <int N, bool SM>
__device__ __noinline__ float field_value_raw(CoefRef<SM> c, float3 xi) {
  Basis<N> B;
  basis_val<N>(xi.x, B.ar);
  basis_val<N>(xi.y, B.as);
  basis_val<N>(xi.z, B.at);
  return contract_v<N, SM>(c, &B);
}

template <int N, bool SM>
__device__ __forceinline__ float field_value(const Elem<N, SM>& e, float3 xi) {
  return field_value_raw<N, SM>(e.fld(), xi);
}

// Components [c0, c1) of one point evaluation, out of line: 0-2 are x, y, z
// (value and the three partials), 3 is the field. The basis values stay in
// registers: the rolled k loop picks at[k] / dt[k] with a predicated select
// instead of reading them back from the stack, and one loop body serves all
// components, so the code stays small. Same FMA order as contract_vd.
template <int N, bool SM>
__device__ __noinline__ void eval_comps(CoefRef<SM> c, float3 xi, int c0, int c1, float4* __restrict__ out) {
  constexpr int RS = row_stride(N);
  float ar[N], dr[N], as[N], ds[N], at[N], dt[N];
  basis_val_der<N>(xi.x, ar, dr);
  basis_val_der<N>(xi.y, as, ds);
  basis_val_der<N>(xi.z, at, dt);
#pragma unroll 1
  for (int comp = c0; comp < c1; ++comp) {
    const CoefRef<SM> cc = c.at(comp * block_floats(N));
    float v = 0.f, vr = 0.f, vs = 0.f, vt = 0.f;
#pragma unroll 1
    for (int k = 0; k < N; ++k) {
      float tk = at[0], dtk = dt[0];
#pragma unroll
      for (int m = 1; m < N; ++m)
        if (k == m) {
          tk = at[m];
          dtk = dt[m];
        }
      float q0 = 0.f, q1 = 0.f, q2 = 0.f;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        float row[RS];
        load_row<N, SM>(cc, (k * N + j) * RS, row);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          s0 = fmaf(row[i], ar[i], s0);
          s1 = fmaf(row[i], dr[i], s1);
        }
        q0 = fmaf(s0, as[j], q0);
        q1 = fmaf(s1, as[j], q1);
        q2 = fmaf(s0, ds[j], q2);
      }
      v = fmaf(q0, tk, v);
      vr = fmaf(q1, tk, vr);
      vs = fmaf(q2, tk, vs);
      vt = fmaf(q0, dtk, vt);
    }
    out[comp] = make_float4(v, vr, vs, vt);
  }
}

// One component of a point evaluation by 8 adjacent lanes (the warp is
// converged, a group's lanes pass the same arguments): lane s of the group
// contracts the slabs k = s, s + 8, and every lane then folds all slabs in the
// order of k. Same FMAs in the same order as eval_comps. A bracket's refinement
// in the tail is a chain of such evaluations: tail of 1 M scattered rays 2.3 ->
// 2.0 ms, of a mixed-order 1024 x 1024 picture of 3 isovalues 2.6 -> 1.8 ms.
template <int N, bool SM>
__device__ __noinline__ float4 eval_slabs(CoefRef<SM> c, float3 xi, int comp) {
  constexpr int RS = row_stride(N), G = 8, S = (N + G - 1) / G;
  const int lane = threadIdx.x & 31, sub = lane & (G - 1), base = lane - sub;
  float ar[N], dr[N], as[N], ds[N], at[N], dt[N];
  basis_val_der<N>(xi.x, ar, dr);
  basis_val_der<N>(xi.y, as, ds);
  basis_val_der<N>(xi.z, at, dt);
  const CoefRef<SM> cc = c.at(comp * block_floats(N));
  float q0[S], q1[S], q2[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int k = sub + s * G;
    q0[s] = q1[s] = q2[s] = 0.f;
    if (k < N) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        float row[RS];
        load_row<N, SM>(cc, (k * N + j) * RS, row);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          s0 = fmaf(row[i], ar[i], s0);
          s1 = fmaf(row[i], dr[i], s1);
        }
        q0[s] = fmaf(s0, as[j], q0[s]);
        q1[s] = fmaf(s1, as[j], q1[s]);
        q2[s] = fmaf(s0, ds[j], q2[s]);
      }
    }
  }
  __syncwarp();
  float v = 0.f, vr = 0.f, vs = 0.f, vt = 0.f;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int src = base + k % G;
    const float p0 = __shfl_sync(0xffffffffu, q0[k / G], src), p1 = __shfl_sync(0xffffffffu, q1[k / G], src),
                p2 = __shfl_sync(0xffffffffu, q2[k / G], src);
    v = fmaf(p0, at[k], v);
    vr = fmaf(p1, at[k], vr);
    vs = fmaf(p2, at[k], vs);
    vt = fmaf(p0, dt[k], vt);
  }
  return make_float4(v, vr, vs, vt);
}

// Adjugate / determinant inverse, no singular guard (HexElement.cu:208-225).
__device__ __forceinline__ void invert3(const float (&J)[9], float (&K)[9]) {
  const float c0 = J[4] * J[8] - J[5] * J[7];
  const float c1 = J[5] * J[6] - J[3] * J[8];
  const float c2 = J[3] * J[7] - J[4] * J[6];
  const float det = J[0] * c0 + J[1] * c1 + J[2] * c2;
  const float id = 1.0f / det;
  K[0] = c0 * id;
  K[1] = (J[2] * J[7] - J[1] * J[8]) * id;
  K[2] = (J[1] * J[5] - J[2] * J[4]) * id;
  K[3] = c1 * id;
  K[4] = (J[0] * J[8] - J[2] * J[6]) * id;
  K[5] = (J[2] * J[3] - J[0] * J[5]) * id;
  K[6] = c2 * id;
  K[7] = (J[1] * J[6] - J[0] * J[7]) * id;
  K[8] = (J[0] * J[4] - J[1] * J[3]) * id;
}

// Inverse map x(xi) = p by Newton from xi0 (the reference always starts at
// 0), at most 50 iterations, converged when every |delta| < 1e-5.
// A NaN iterate can never converge, so it stops early with the same answer.
template <int N, bool SM>
__device__ __forceinline__ bool inverse_map(const Elem<N, SM>& e, float3 p, float3& xi, Work& w,
                                            float3 xi0 = make_float3(0.f, 0.f, 0.f), int max_it = 50) {
  xi = xi0;
  for (int it = 0; it < max_it; ++it) {
    ++w.newton;
    float3 x;
    float J[9], K[9];
    geom_eval<N>(e, xi, x, J, w);
    const float rx = x.x - p.x, ry = x.y - p.y, rz = x.z - p.z;
    invert3(J, K);
    const float d0 = K[0] * rx + K[1] * ry + K[2] * rz;
    const float d1 = K[3] * rx + K[4] * ry + K[5] * rz;
    const float d2 = K[6] * rx + K[7] * ry + K[8] * rz;
    xi.x -= d0;
    xi.y -= d1;
    xi.z -= d2;
    if (fabsf(d0) < 1e-5f && fabsf(d1) < 1e-5f && fabsf(d2) < 1e-5f) return true;
    if (!(fabsf(d0) + fabsf(d1) + fabsf(d2) < FLT_MAX)) return false;  // NaN / Inf
  }
  return false;
}

// f(t) = u(x(t)) - iso and df/dt with the world gradient
// (RayIsosurface.cu:44-65).
struct Sample {
  float3 xi;
  float f, df;
  float3 g;
};

// The batched engines' form of a sample (AH = true in sample_along): every
// Newton iteration also evaluates the field (value and xi-gradient) at its
// point, and when the step converges (all components below 1e-5) the sample
// is taken to first order at the converged point, u(xi - step) = u(xi) -
// grad u . step (error O(|step|^2), below 1e-9), with the gradient mapped by
// the iteration's inverse Jacobian. The reference evaluates the field and the
// Jacobian once more at the converged point (sample_along with AH = false);
// the round kernel and the warp-per-ray kernel both use this form, with the
// same arithmetic, so they give the same answers.
// U: all 32 lanes call it with the same arguments, so 8 lanes share each
// component and take the others by shuffles
// (the tail of 12 views of mixed orders 13.3 -> 10.8 ms).
template <int N, bool SM, bool U = false>
__device__ __forceinline__ bool sample_ahead(const Elem<N, SM>& e, float3 o, float3 d, float t, float iso, Sample& s,
                                             Work& w, float3 xi0, int max_it) {
  float3 xi = xi0;
  for (int it = 1;; ++it) {
    float4 r[4];
    if constexpr (U) {
      const float4 v = eval_slabs<N, SM>(e.c, xi, (threadIdx.x >> 3) & 3);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        r[k] = make_float4(__shfl_sync(0xffffffffu, v.x, 8 * k), __shfl_sync(0xffffffffu, v.y, 8 * k),
                           __shfl_sync(0xffffffffu, v.z, 8 * k), __shfl_sync(0xffffffffu, v.w, 8 * k));
    } else {
      eval_comps<N, SM>(e.c, xi, 0, 4, r);
    }
    w.flops += eval_flops(N, 4);
    ++w.geom;
    ++w.field;
    const float J[9] = {r[0].y, r[0].z, r[0].w, r[1].y, r[1].z, r[1].w, r[2].y, r[2].z, r[2].w};
    const float u = r[3].x;
    const float3 gr = make_float3(r[3].y, r[3].z, r[3].w);
    float K[9];
    invert3(J, K);
    ++w.newton;
    w.flops += kSolveFlops;
    const float rx = r[0].x - (o.x + t * d.x), ry = r[1].x - (o.y + t * d.y), rz = r[2].x - (o.z + t * d.z);
    const float d0 = K[0] * rx + K[1] * ry + K[2] * rz;
    const float d1 = K[3] * rx + K[4] * ry + K[5] * rz;
    const float d2 = K[6] * rx + K[7] * ry + K[8] * rz;
    xi.x -= d0;
    xi.y -= d1;
    xi.z -= d2;
    if (fabsf(d0) < 1e-5f && fabsf(d1) < 1e-5f && fabsf(d2) < 1e-5f) {
      s.xi = xi;
      s.g = make_float3(K[0] * gr.x + K[3] * gr.y + K[6] * gr.z, K[1] * gr.x + K[4] * gr.y + K[7] * gr.z,
                        K[2] * gr.x + K[5] * gr.y + K[8] * gr.z);
      s.f = (u - (gr.x * d0 + gr.y * d1 + gr.z * d2)) - iso;
      s.df = s.g.x * d.x + s.g.y * d.y + s.g.z * d.z;
      return true;
    }
    s.xi = xi;
    if (!(fabsf(d0) + fabsf(d1) + fabsf(d2) < FLT_MAX)) return false;
    if (it >= max_it) return false;
  }
}

template <int N, bool SM, bool AH = false, bool U = false>
__device__ __forceinline__ bool sample_along(const Elem<N, SM>& e, float3 o, float3 d, float t, float iso, Sample& s,
                                             Work& w, float3 xi0 = make_float3(0.f, 0.f, 0.f), int max_it = 50) {
  if constexpr (AH) return sample_ahead<N, SM, U>(e, o, d, t, iso, s, w, xi0, max_it);
  const float3 p = make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
  if (!inverse_map<N>(e, p, s.xi, w, xi0, max_it)) return false;
  float u;
  float3 gr;
  field_eval<N>(e, s.xi, u, gr, w);
  float3 x;
  float J[9], K[9];
  geom_eval<N>(e, s.xi, x, J, w);
  invert3(J, K);
  s.g = make_float3(K[0] * gr.x + K[3] * gr.y + K[6] * gr.z, K[1] * gr.x + K[4] * gr.y + K[7] * gr.z,
                    K[2] * gr.x + K[5] * gr.y + K[8] * gr.z);
  s.f = u - iso;
  s.df = s.g.x * d.x + s.g.y * d.y + s.g.z * d.z;
  return true;
}

// Learned-mode sample: Newton from a predicted xi with a short iteration cap;
// if that does not converge the plain cold-start solve answers (the fallback
// the learned guess never replaces).
constexpr int kWarmCap = 4;
template <int N, bool SM, bool AH = false, bool U = false>
__device__ __forceinline__ bool sample_warm(const Elem<N, SM>& e, float3 o, float3 d, float t, float iso, Sample& s,
                                            Work& w, bool warm, float3 xi0) {
  if (warm) {
    if (sample_along<N, SM, AH, U>(e, o, d, t, iso, s, w, xi0, kWarmCap)) {
      ++w.accepted;
      return true;
    }
    ++w.rejected;
  }
  return sample_along<N, SM, AH, U>(e, o, d, t, iso, s, w);
}

__device__ __forceinline__ float3 lerp3(float3 a, float3 b, float u) {
  return make_float3(a.x + u * (b.x - a.x), a.y + u * (b.y - a.y), a.z + u * (b.z - a.z));
}

// At most 20 safeguarded Newton/bisection steps on a bracket [lt, rt] whose
// left sample is ls; done when |f| < 1e-5, else the midpoint with the left
// sample's xi and gradient (RayIsosurface.cu:121-177).
template <int N, bool SM, bool AH = false, bool U = false>
__device__ __forceinline__ bool refine_bracket(const Elem<N, SM>& e, float3 o, float3 d, float iso, float lt, float rt,
                                               Sample ls, float& th, float3& xh, float3& gh, Work& w,
                                               bool warm = false, float3 rxi = make_float3(0.f, 0.f, 0.f)) {
  for (int it = 0; it < 20; ++it) {
    const float mt = 0.5f * (lt + rt);
    Sample ms;
    if (!sample_warm<N, SM, AH, U>(e, o, d, mt, iso, ms, w, warm, lerp3(ls.xi, rxi, 0.5f))) return false;
    float ct = mt;
    if (fabsf(ms.df) > 1e-8f) {
      const float nt = mt - ms.f / ms.df;
      if (nt > lt && nt < rt) ct = nt;
    }
    Sample cs;
    if (!sample_warm<N, SM, AH, U>(e, o, d, ct, iso, cs, w, warm, ms.xi)) {
      ct = mt;  // keep the failed solve's xi, as the reference does
      cs.f = ms.f;
      cs.g = ms.g;
    }
    if (fabsf(cs.f) < 1e-5f) {
      th = ct;
      xh = cs.xi;
      gh = cs.g;
      return true;
    }
    if (ls.f * cs.f <= 0.0f) {
      rt = ct;
      rxi = cs.xi;
    } else {
      lt = ct;
      ls = cs;
    }
  }
  th = 0.5f * (lt + rt);
  xh = ls.xi;
  gh = ls.g;
  return true;
}

// First sign change over 17 uniform samples of [t0,t1], then the bracket
// refinement (RayIsosurface.cu:67-188). One thread.
template <int N, bool SM>
__device__ bool find_iso(const Elem<N, SM>& e, float3 o, float3 d, float t0, float t1, float iso, float& th, float3& xh,
                         float3& gh, Work& w) {
  bool have = false;
  float tp = t0;
  Sample sp;
  sp.f = 0.f;
  sp.xi = make_float3(0.f, 0.f, 0.f);
  sp.g = sp.xi;
  for (int i = 0; i <= 16; ++i) {
    const float t = t0 + (t1 - t0) * (float(i) / 16.0f);
    Sample s;
    if (!sample_along<N>(e, o, d, t, iso, s, w)) continue;
    if (!have) {
      have = true;
      tp = t;
      sp = s;
      continue;
    }
    if (sp.f * s.f <= 0.0f) return refine_bracket<N>(e, o, d, iso, tp, t, sp, th, xh, gh, w);
    tp = t;
    sp = s;
  }
  return false;
}

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float3 shfl3(float3 v, int src) {
  return make_float3(__shfl_sync(kFull, v.x, src), __shfl_sync(kFull, v.y, src), __shfl_sync(kFull, v.z, src));
}

// Warp version: the 17 samples are independent inverse-map solves, so lane i
// solves sample i; the first sample i (in order) that succeeded and whose
// previous successful sample has f(prev)*f(i) <= 0 is found with ballots —
// the same bracket the sequential scan stops at. The refinement is then run
// by every lane on identical data (uniform control flow); its work is
// counted in wu, which only lane 0 reports. Call with all 32 lanes. The
// samples take the field with every Newton iteration (sample_ahead), as the
// round kernel does.
// Learned prediction for one candidate: xi at the segment entry te and
// d xi / d t there (scaled by the element size: xi(t) ~ xi_in + (t-te)*k*v).
struct Pred {
  bool on;
  float3 xi_in, v;
  float k, te;
  __device__ __forceinline__ float3 at(float t) const {
    const float u = (t - te) * k;
    return make_float3(xi_in.x + u * v.x, xi_in.y + u * v.y, xi_in.z + u * v.z);
  }
};

template <int N, bool L, bool SM>
__device__ bool find_iso_warp(const Elem<N, SM>& e, float3 o, float3 d, float t0, float t1, float iso, float& th,
                              float3& xh, float3& gh, Work& w, Work& wu, const Pred& pr) {
  const int lane = threadIdx.x & 31;
  Sample s;
  s.f = 0.f;
  s.df = 0.f;
  s.xi = make_float3(0.f, 0.f, 0.f);
  s.g = s.xi;
  const long long c0 = clock64();
  const float t = t0 + (t1 - t0) * (float(lane) / 16.0f);
  bool ok = false;
  if (!L || !pr.on) {
    if (lane <= 16) ok = sample_along<N, SM, true>(e, o, d, t, iso, s, w);
  } else {
    // learned: Newton from the predicted xi, short cap
    if (lane <= 16) ok = sample_along<N, SM, true>(e, o, d, t, iso, s, w, pr.at(t), kWarmCap);
    // a sample that missed the cap restarts from its converged neighbours'
    // xi (interpolated in t), then, failing that, from the plain cold start
    const unsigned cm = __ballot_sync(kFull, ok && lane <= 16);
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned below = cm & lt_mask, above = cm & ~lt_mask & ~(1u << lane) & 0x1FFFFu;
    const int lb = below ? 31 - __clz(below) : lane, la = above ? __ffs(above) - 1 : lane;
    const float3 xb = shfl3(s.xi, lb), xa = shfl3(s.xi, la);
    const float tb = __shfl_sync(kFull, t, lb), ta = __shfl_sync(kFull, t, la);
    if (lane <= 16) {
      if (ok) {
        ++w.accepted;
      } else {
        float3 g0 = pr.at(t);
        if (below && above) g0 = lerp3(xb, xa, (t - tb) / (ta - tb));
        else if (below) g0 = make_float3(xb.x + (t - tb) * pr.k * pr.v.x, xb.y + (t - tb) * pr.k * pr.v.y,
                                         xb.z + (t - tb) * pr.k * pr.v.z);
        else if (above) g0 = make_float3(xa.x + (t - ta) * pr.k * pr.v.x, xa.y + (t - ta) * pr.k * pr.v.y,
                                         xa.z + (t - ta) * pr.k * pr.v.z);
        ok = (cm != 0u) && sample_along<N, SM, true>(e, o, d, t, iso, s, w, g0, kWarmCap);
        if (!ok) {
          ++w.rejected;
          ok = sample_along<N, SM, true>(e, o, d, t, iso, s, w);
        }
      }
    }
  }
  wu.cyc[1] += clock64() - c0;
  const unsigned okm = __ballot_sync(kFull, ok);
  const unsigned below = okm & ((1u << lane) - 1u);
  const int prev = below ? 31 - __clz(below) : lane;
  const float pf = __shfl_sync(kFull, s.f, prev);
  const bool sc = ok && below != 0u && pf * s.f <= 0.0f;
  const unsigned scm = __ballot_sync(kFull, sc);
  if (scm == 0u) return false;
  const int ri = __ffs(scm) - 1;
  const int li = 31 - __clz(okm & ((1u << ri) - 1u));
  const float lt = __shfl_sync(kFull, t, li), rt = __shfl_sync(kFull, t, ri);
  Sample ls;
  ls.f = __shfl_sync(kFull, s.f, li);
  ls.df = __shfl_sync(kFull, s.df, li);
  ls.xi = shfl3(s.xi, li);
  ls.g = shfl3(s.g, li);
  const float3 rxi = shfl3(s.xi, ri);
  const long long c1 = clock64();
  const bool found = refine_bracket<N, SM, true, true>(e, o, d, iso, lt, rt, ls, th, xh, gh, wu, L && pr.on, rxi);
  wu.cyc[2] += clock64() - c1;
  return found;
}

// True when the isosurface search of a candidate's segment [te, tx] cannot
// find a sign change that is an isosurface point of the element, from the
// element's certificate (cull_kernel in ho_build.cu has the proof, and what it
// leaves open for restarted network starts): every sample whose Newton solve
// converges has xi within delta of y = K (x - x0), which is linear in t, and a
// field value within H of the trilinear interpolant of the element's corner
// values there.
// So u - iso keeps one sign over the segment when those bounds clear the
// isovalue on one side over the boxes around its four quarters (a trilinear
// function on a box has its extremes at the box's corners), and the 17
// samples, whatever subset of them converges, bracket nothing. A NaN
// anywhere fails the comparisons: the search then runs.
__device__ __forceinline__ bool iso_excluded(const float* __restrict__ cull, int elem, float3 o, float3 d, float te,
                                             float tx, float iso, bool warm, const Pred& pr) {
  const float4* c4 = reinterpret_cast<const float4*>(cull + static_cast<int64_t>(elem) * kCullFloats);
  const float4 k0 = __ldg(c4), k1 = __ldg(c4 + 1), k2 = __ldg(c4 + 2), k3 = __ldg(c4 + 3);
  if (!(k3.x >= 0.f)) return false;
  if (warm) {  // the network's starts must lie where the certificate's Newton bound holds
    const float3 a = pr.at(te), b = pr.at(tx);
    const float m = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(b.x))),
                          fmaxf(fabsf(b.y), fabsf(b.z)));
    if (!(m <= k3.z)) return false;
  }
  const float K[9] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w, k2.x};
  const float3 q = make_float3(o.x - k2.y, o.y - k2.z, o.z - k2.w);
  // rounding of the sample points o + t d and of y (the candidate's box keeps
  // a margin of 0.01 in y for it)
  const float kn = fmaxf(fabsf(K[0]) + fabsf(K[1]) + fabsf(K[2]),
                         fmaxf(fabsf(K[3]) + fabsf(K[4]) + fabsf(K[5]), fabsf(K[6]) + fabsf(K[7]) + fabsf(K[8])));
  const float big = fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z))) + fmaxf(fabsf(te), fabsf(tx)) *
                        fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)));
  const float slop = 1e-6f * big * kn;
  if (!(slop <= 5e-3f)) return false;
  const float dl = k3.x + slop;
  float y0[3], ys[3];  // y at te, and over a quarter of the segment
  const float qt = 0.25f * (tx - te);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    y0[a] = K[3 * a] * (q.x + te * d.x) + K[3 * a + 1] * (q.y + te * d.y) + K[3 * a + 2] * (q.z + te * d.z);
    ys[a] = (K[3 * a] * d.x + K[3 * a + 1] * d.y + K[3 * a + 2] * d.z) * qt;
  }
  const float4 f0 = __ldg(c4 + 4), f1 = __ldg(c4 + 5);
  const float lim_lo = iso - k3.y, lim_hi = iso + k3.y;
  bool above = true, below = true;
#pragma unroll 1
  for (int s = 0; s < 4 && (above || below); ++s) {
    float w[3][2];  // interpolation weights of the box's two sides per axis
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float p = y0[a] + s * ys[a], r = p + ys[a];
      w[a][0] = 0.5f + 0.5f * (fminf(p, r) - dl);
      w[a][1] = 0.5f + 0.5f * (fmaxf(p, r) + dl);
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const float e0 = f0.x + w[0][x] * (f0.y - f0.x), e1 = f0.z + w[0][x] * (f0.w - f0.z),
                  e2 = f1.x + w[0][x] * (f1.y - f1.x), e3 = f1.z + w[0][x] * (f1.w - f1.z);
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const float g0 = e0 + w[1][y] * (e1 - e0), g1 = e2 + w[1][y] * (e3 - e2);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const float v = g0 + w[2][z] * (g1 - g0);
          above = above && v > lim_hi;
          below = below && v < lim_lo;
        }
      }
    }
  }
  return above || below;
}

// Slab test clipped to [tmin, tmax] (high_order.h:115-152).
__device__ __forceinline__ bool ray_box(float3 o, float3 d, const float* lo, const float* hi, float tmin, float tmax,
                                        float& te, float& tx) {
  te = tmin;
  tx = tmax;
  const float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (fabsf(dd[a]) < 1e-8f) {
      if (oo[a] < lo[a] || oo[a] > hi[a]) return false;
      continue;
    }
    const float inv = 1.0f / dd[a];
    float a0 = (lo[a] - oo[a]) * inv, a1 = (hi[a] - oo[a]) * inv;
    if (a0 > a1) {
      const float tmp = a0;
      a0 = a1;
      a1 = tmp;
    }
    te = fmaxf(te, a0);
    tx = fminf(tx, a1);
  }
  return tx >= te;
}

// Face table (high_order.h:164-184): fixed axis, fixed value, free axes.
__device__ __forceinline__ void face_param(int f, int& fixed, float& val, int& ua, int& va) {
  switch (f) {
    case 0: fixed = 2; val = -1.f; ua = 0; va = 1; break;
    case 1: fixed = 1; val = -1.f; ua = 0; va = 2; break;
    case 2: fixed = 0; val = 1.f; ua = 1; va = 2; break;
    case 3: fixed = 1; val = 1.f; ua = 0; va = 2; break;
    case 4: fixed = 0; val = -1.f; ua = 1; va = 2; break;
    default: fixed = 2; val = 1.f; ua = 0; va = 1; break;
  }
}

__device__ __forceinline__ float getc(float3 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }
__device__ __forceinline__ void setc(float3& v, int a, float s) {
  if (a == 0) v.x = s;
  else if (a == 1) v.y = s;
  else v.z = s;
}

// Point and the two tangents of face f (face_param's free axes ua < va) at
// its free coordinates (u, v), components [c0, c1) (0-2: x, y, z, 3: the field):
// out[c] = {x_c, dx_c/du, dx_c/dv, 0}.
//
// On a face the fixed coordinate is exactly -1 or 1, where one vertex mode is
// exactly 1 and every other mode exactly 0, so of the contraction over three
// axes (eval_comps) only the face's own N x N coefficients contribute, and the
// Newton needs no derivative across the face. The sums over the free axes run
// in eval_comps' order, and adding a product with 0 or multiplying by 1 is
// exact, so the values are eval_comps' to the last bit at 1 / N of its
// multiply-adds. The face solves are most of the round kernel's steps; their
// evaluations' cost was 2 (2N^3 + 3N^2) operations a component.
template <int N, bool SM>
__device__ __noinline__ void face_eval(CoefRef<SM> c, int f, float u, float v, int c0, int c1,
                                       float4* __restrict__ out) {
  constexpr int RS = row_stride(N);
  int fixed, ua, va;
  float val;
  face_param(f, fixed, val, ua, va);
  const int m = val < 0.f ? 0 : 1;
  const int sf = fixed == 0 ? 1 : (fixed == 1 ? RS : N * RS);  // strides of the three axes' modes
  const int su = ua == 0 ? 1 : RS, sv = va == 1 ? RS : N * RS;
  float pu[N], du[N], pv[N], dv[N];
  basis_val_der<N>(u, pu, du);
  basis_val_der<N>(v, pv, dv);
#pragma unroll 1
  for (int comp = c0; comp < c1; ++comp) {
    const CoefRef<SM> cc = c.at(comp * block_floats(N) + m * sf);
    float x = 0.f, xu = 0.f, xv = 0.f;
#pragma unroll 1
    for (int b = 0; b < N; ++b) {
      float pb = pv[0], db = dv[0];
#pragma unroll
      for (int k = 1; k < N; ++k)
        if (b == k) {
          pb = pv[k];
          db = dv[k];
        }
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int a = 0; a < N; ++a) {
        const float w = cc.ld(b * sv + a * su);
        s0 = fmaf(w, pu[a], s0);
        s1 = fmaf(w, du[a], s1);
      }
      x = fmaf(s0, pb, x);
      xu = fmaf(s1, pb, xu);
      xv = fmaf(s0, db, xv);
    }
    out[comp] = make_float4(x, xu, xv, 0.f);
  }
}

// True when no seed of face f can be accepted on the ray's [tmin, tmax], by the
// element's certificate (cull_kernel). Let z = xi' - xi for a point xi of the
// cube with position X, a parameter t, and an accepted (xi', t') on the face:
// G(xi') - G(xi) = e + w (t' - t) + a term of size eps, where e = K (o + t d -
// X), w = K d and eps covers the acceptance tolerance 1e-4 and rounding, and z
// differs from it by at most b = beta |z| <= beta / (1 - beta) (|e| + |w| |t' -
// t| + eps). z's component across the face is known (across), which bounds t'
// - t when the ray is not nearly parallel to the face; the other two must
// bring xi' into [-1.001, 1.001]. With xi = 0 this is a slab test in the
// element's own frame; with the last iterate of a failed seed, e is small and
// so is what the curvature leaves open.
static __device__ __noinline__ bool face_impossible(const float* __restrict__ cert, int f, float3 o, float3 d, float3 xi,
                                             float3 X, float t, float across, float tmin, float tmax) {
  const float4* c4 = reinterpret_cast<const float4*>(cert);
  const float4 k0 = __ldg(c4), k1 = __ldg(c4 + 1), k2 = __ldg(c4 + 2), k3 = __ldg(c4 + 3);
  if (!(k3.x >= 0.f)) return false;
  const float K[9] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w, k2.x};
  const float beta = k3.w, bp = beta / (1.f - beta);
  const float kn = fmaxf(fabsf(K[0]) + fabsf(K[1]) + fabsf(K[2]),
                         fmaxf(fabsf(K[3]) + fabsf(K[4]) + fabsf(K[5]), fabsf(K[6]) + fabsf(K[7]) + fabsf(K[8])));
  const float big = fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z))) +
                    fabsf(t) * fmaxf(fabsf(d.x), fmaxf(fabsf(d.y), fabsf(d.z)));
  const float eps = kn * (1.05e-4f + 2e-6f * big);
  const float3 q = make_float3(o.x + t * d.x - X.x, o.y + t * d.y - X.y, o.z + t * d.z - X.z);
  float e[3], w[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    e[a] = K[3 * a] * q.x + K[3 * a + 1] * q.y + K[3 * a + 2] * q.z;
    w[a] = K[3 * a] * d.x + K[3 * a + 1] * d.y + K[3 * a + 2] * d.z;
  }
  int fixed, ua, va;
  float val;
  face_param(f, fixed, val, ua, va);
  const float en = fmaxf(fabsf(e[0]), fmaxf(fabsf(e[1]), fabsf(e[2])));
  const float wn = fmaxf(fabsf(w[0]), fmaxf(fabsf(w[1]), fabsf(w[2])));
  const float ef = (fixed == 0 ? e[0] : (fixed == 1 ? e[1] : e[2])) - across;
  const float wf = fixed == 0 ? w[0] : (fixed == 1 ? w[1] : w[2]);
  const float steep = fabsf(wf) - bp * wn;
  if (!(steep > 1e-3f * wn)) return false;
  const float s0 = -ef / wf, h = (bp * (en + wn * fabsf(s0) + eps) + eps) / steep;
  const float tol = 2e-6f * big;
  const float lo = fmaxf(s0 - h, tmin - t - tol), hi = fminf(s0 + h, tmax - t + tol);
  if (lo > hi) return true;
  const float z = bp * (en + wn * fmaxf(fabsf(lo), fabsf(hi)) + eps) + eps;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int a = k == 0 ? ua : va;
    const float ea = a == 0 ? e[0] : (a == 1 ? e[1] : e[2]), wa = a == 0 ? w[0] : (a == 1 ? w[1] : w[2]);
    const float p = getc(xi, a) + ea, r0 = wa * lo, r1 = wa * hi;
    if (p + fmaxf(r0, r1) + z < -1.001f || p + fminf(r0, r1) - z > 1.001f) return true;
  }
  return false;
}

// Iterations after which a first seed is asked whether the face can be hit at
// all: a seed that converges takes about 7 (its steps are clamped to 0.25),
// one that sticks at the clamps of u, v or tau runs all its 50.
constexpr int kSeedPatience = 8;

// One seed of the ray / curved-face Newton in (u,v,tau): at most 50
// iterations, accept when max|X-Y| < 1e-4 with u,v in [-1.001,1.001] and tau
// in [tmin,tmax]; step clamp 0.25, divergence break after 5 iterations
// (high_order.h:213-300).
template <int N, bool SM>
__device__ bool face_newton(const Elem<N, SM>& e, float3 o, float3 d, int f, float3 p, float tau, float tmin, float tmax,
                            float& th, float3& xh, Work& w, int max_it, const float* cert = nullptr, bool* none = nullptr);

template <int N, bool SM>
__device__ bool face_seed(const Elem<N, SM>& e, float3 o, float3 d, int f, int si, int sj, float tmin, float tmax,
                          float& th, float3& xh, Work& w, const float* cert = nullptr, bool* none = nullptr) {
  int fixed, ua, va;
  float val;
  face_param(f, fixed, val, ua, va);
  const float dd = d.x * d.x + d.y * d.y + d.z * d.z;
  float3 p = make_float3(0.f, 0.f, 0.f);
  setc(p, fixed, val);
  setc(p, ua, si == 0 ? -0.8f : (si == 1 ? 0.0f : 0.8f));
  setc(p, va, sj == 0 ? -0.8f : (sj == 1 ? 0.0f : 0.8f));
  const float3 x0 = geom_map<N>(e, p, w);
  const float3 df = make_float3(x0.x - o.x, x0.y - o.y, x0.z - o.z);
  float tau = dd > 0.f ? (df.x * d.x + df.y * d.y + df.z * d.z) / dd : 0.f;
  tau = fminf(fmaxf(tau, tmin), tmax);
  return face_newton<N>(e, o, d, f, p, tau, tmin, tmax, th, xh, w, 50, cert, none);
}

// The (u,v,tau) Newton of one seed from a given start point.
template <int N, bool SM>
__device__ bool face_newton(const Elem<N, SM>& e, float3 o, float3 d, int f, float3 p, float tau, float tmin, float tmax,
                            float& th, float3& xh, Work& w, int max_it, const float* cert, bool* none) {
  int fixed, ua, va;
  float val;
  face_param(f, fixed, val, ua, va);
  float prev = FLT_MAX;
  for (int it = 0; it < max_it; ++it) {
    ++w.face;
    float3 X;
    float J[9];
    geom_eval<N>(e, p, X, J, w);
    const float rx = X.x - (o.x + tau * d.x), ry = X.y - (o.y + tau * d.y), rz = X.z - (o.z + tau * d.z);
    const float m = fmaxf(fabsf(rx), fmaxf(fabsf(ry), fabsf(rz)));
    bool ended = false;
    if (m < 1e-4f) {
      const float pu = getc(p, ua), pv = getc(p, va);
      if (pu >= -1.001f && pu <= 1.001f && pv >= -1.001f && pv <= 1.001f && tau >= tmin && tau <= tmax) {
        th = tau;
        xh = p;
        return true;
      }
      ended = true;
    } else if (it > 5 && m > prev * 1.5f) {
      ended = true;
    }
    // a first seed that ends without a hit, or takes long: none may have one
    if (cert && (ended || it == kSeedPatience) && face_impossible(cert, f, o, d, p, X, tau, 0.f, tmin, tmax)) {
      *none = true;
      return false;
    }
    if (ended) return false;
    prev = m;
    const float A[9] = {J[ua], J[va], -d.x, J[3 + ua], J[3 + va], -d.y, J[6 + ua], J[6 + va], -d.z};
    float K[9];
    invert3(A, K);
    const float du = -(K[0] * rx + K[1] * ry + K[2] * rz);
    const float dv = -(K[3] * rx + K[4] * ry + K[5] * rz);
    const float dtau = -(K[6] * rx + K[7] * ry + K[8] * rz);
    const float mx = fmaxf(fabsf(du), fmaxf(fabsf(dv), fabsf(dtau)));
    const float sc = mx > 0.25f ? 0.25f / mx : 1.0f;
    float nu = getc(p, ua) + du * sc, nv = getc(p, va) + dv * sc;
    tau = fminf(fmaxf(tau + dtau * sc, tmin), tmax);
    nu = fminf(fmaxf(nu, -1.5f), 1.5f);  // fminf/fmaxf drop a NaN, as on the host
    nv = fminf(fmaxf(nv, -1.5f), 1.5f);
    setc(p, ua, nu);
    setc(p, va, nv);
    setc(p, fixed, val);
  }
  return false;
}

// Ray against one curved face: the 9 seeds {-0.8,0,0.8}^2 in order (v outer,
// u inner); the first seed accepted answers (high_order.h:189-304).
template <int N, bool SM>
__device__ bool hit_face(const Elem<N, SM>& e, float3 o, float3 d, int f, float tmin, float tmax, float& th, float3& xh,
                         Work& w) {
  for (int sj = 0; sj < 3; ++sj)
    for (int si = 0; si < 3; ++si)
      if (face_seed<N>(e, o, d, f, si, sj, tmin, tmax, th, xh, w)) return true;
  return false;
}

// Nearest boundary-face hit over the 6 faces. A face is skipped when the
// segment [tmin,tmax] misses that face's hull box: the box bounds the face
// over u,v in [-1.001,1.001] and is inflated past the 1e-4 acceptance
// tolerance plus rounding, so no seed could have been accepted there and the
// reference's answer for the face is "no hit" (exact culling).
// The reference's padded-box pre-test (high_order.h:420-431) is the same box
// the candidate was admitted with, so it always passes here.
template <int N, bool SM>
__device__ bool hit_hex(const Elem<N, SM>& e, const float* __restrict__ fbox, float3 o, float3 d, float tmin, float tmax,
                        float& th, float3& xh, int& face, Work& w) {
  bool any = false;
  float best = tmax;
  for (int f = 0; f < 6; ++f) {
    const float* b = fbox + 6 * f;
    const float lo[3] = {__ldg(b + 0), __ldg(b + 1), __ldg(b + 2)};
    const float hi[3] = {__ldg(b + 3), __ldg(b + 4), __ldg(b + 5)};
    float a0, a1;
    if (!ray_box(o, d, lo, hi, tmin, tmax, a0, a1)) {
      ++w.culled;
      continue;
    }
    float tf;
    float3 xf;
    if (hit_face<N>(e, o, d, f, tmin, tmax, tf, xf, w)) {
      if (tf > tmin && tf < best) {
        best = tf;
        xh = xf;
        face = f;
        any = true;
      }
    }
  }
  if (any) th = best;
  return any;
}

__device__ __forceinline__ float3 normalize3(float3 v) {
  const float l = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
  const float s = 1.0f / l;
  return make_float3(v.x * s, v.y * s, v.z * s);
}
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

struct HitState {
  float t;
  int elem, face, kind;
  float3 xi, n;
  float u;
  uint32_t flags;
};

// Internal flag of a HitState: the face hit's normal (from the Jacobian at xi)
// and the field value at xi are still to be filled in (fill_hit).
constexpr uint32_t kFlagPost = 0x80000000u;

// Unit normal of a face hit from the Jacobian's columns (the face's two
// tangents), against the ray.
__device__ __forceinline__ float3 face_normal(const float (&J)[9], float3 xi, float3 d) {
  const float3 dr = make_float3(J[0], J[3], J[6]), ds = make_float3(J[1], J[4], J[7]),
               dt = make_float3(J[2], J[5], J[8]);
  float3 n;
  if (fabsf(xi.x) > 0.9f) n = cross3(ds, dt);
  else if (fabsf(xi.y) > 0.9f) n = cross3(dr, dt);
  else n = cross3(dr, ds);
  n = normalize3(n);
  if (n.x * d.x + n.y * d.y + n.z * d.z > 0.f) n = make_float3(-n.x, -n.y, -n.z);
  return n;
}

// Does face_normal take a hit on face f from the face's own two tangents?
__device__ __forceinline__ bool normal_on_face(int f, float3 xi) {
  int fixed, ua, va;
  float val;
  face_param(f, fixed, val, ua, va);
  return fixed == 0 || (!(fabsf(xi.x) > 0.9f) && (fixed == 1 || !(fabsf(xi.y) > 0.9f)));
}

// What a hit committed with kFlagPost lacks, from the Jacobian and the field
// value at its xi.
__device__ __forceinline__ void fill_hit(HitState& h, const float (&J)[9], float u, float3 d) {
  if (h.kind == HO_HIT_FACE) h.n = face_normal(J, h.xi, d);
  h.u = u;
  h.flags &= ~kFlagPost;
}

// Two candidates' hits this close in t claim one surface point: a face shared
// by two elements, an edge of two faces, a root in the overlap of two padded
// boxes. The reference keeps whichever its visit order and FP32 rounding put
// first. A hit that displaces the best one by less than this keeps the
// displaced hit as the ray's tie partner, and the final FP64 check decides
// between the two (fp64_tie_rule).
constexpr float kTieT = 1e-4f;

// The best hit (t = best_t; a miss has FLT_MAX) is about to become a hit at
// t_new < best_t: keep the old one as the tie partner when it is within
// kTieT, else drop the partner (it lies behind the old best, so further than
// kTieT from the new hit too). Blind stores: no read of the partner.
__device__ __forceinline__ void note_tie(const HitState& best, float best_t, float t_new, HitState* tie) {
  if (!tie) return;
  if (best_t - t_new <= kTieT) *tie = best;
  else tie->kind = HO_HIT_MISS;
}

// Per-candidate policy of the reference's hex branch: iso search on the
// padded-box segment when enabled; if it finds nothing, nearest curved face.
template <int N, bool SM>
__device__ void visit_candidate(const Elem<N, SM>& e, const float* __restrict__ fbox, int eidx, float3 o, float3 d,
                                float te, float tx, float iso, bool iso_on, HitState& best, Work& w,
                                HitState* tie = nullptr) {
  ++w.cand;
  float th;
  float3 xi, g;
  if (iso_on && e.has_field && find_iso<N>(e, o, d, te, tx, iso, th, xi, g, w)) {
    if (th > 0.001f && th < best.t) {
      float3 n = normalize3(g);
      if (n.x * d.x + n.y * d.y + n.z * d.z > 0.f) n = make_float3(-n.x, -n.y, -n.z);
      note_tie(best, best.t, th, tie);
      best.t = th;
      best.elem = eidx;
      best.face = -1;
      best.kind = HO_HIT_ISO;
      best.xi = xi;
      best.n = n;
      best.u = field_value<N>(e, xi);
    }
    return;
  }
  int face = -1;
  if (hit_hex<N>(e, fbox, o, d, 0.001f, best.t, th, xi, face, w)) {
    if (th > 0.001f && th < best.t) {
      float3 x;
      float J[9];
      geom_eval<N>(e, xi, x, J, w);
      const float3 n = face_normal(J, xi, d);
      note_tie(best, best.t, th, tie);
      best.t = th;
      best.elem = eidx;
      best.face = face;
      best.kind = HO_HIT_FACE;
      best.xi = xi;
      best.n = n;
      best.u = e.has_field ? field_value<N>(e, xi) : 0.f;
    }
  }
}

// Face test of one face against [tmin,tmax] through its hull box (exact cull).
__device__ __forceinline__ bool face_may_hit(const float* __restrict__ fbox, int f, float3 o, float3 d, float tmin,
                                             float tmax) {
  const float* b = fbox + 6 * f;
  const float lo[3] = {__ldg(b + 0), __ldg(b + 1), __ldg(b + 2)};
  const float hi[3] = {__ldg(b + 3), __ldg(b + 4), __ldg(b + 5)};
  float a0, a1;
  return ray_box(o, d, lo, hi, tmin, tmax, a0, a1);
}

// The same, with the entry into the hull box.
__device__ __forceinline__ bool face_entry(const float* __restrict__ fbox, int f, float3 o, float3 d, float tmin,
                                           float tmax, float& te) {
  const float* b = fbox + 6 * f;
  const float lo[3] = {__ldg(b + 0), __ldg(b + 1), __ldg(b + 2)};
  const float hi[3] = {__ldg(b + 3), __ldg(b + 4), __ldg(b + 5)};
  float a1;
  return ray_box(o, d, lo, hi, tmin, tmax, te, a1);
}

// The same from the element's centre: t at the closest approach to it.
__device__ __forceinline__ bool face_excluded(const float* __restrict__ cert, int f, float3 o, float3 d, float tmin,
                                              float tmax) {
  const float3 x0 = make_float3(__ldg(cert + 9), __ldg(cert + 10), __ldg(cert + 11));
  const float dd = d.x * d.x + d.y * d.y + d.z * d.z;
  const float t = ((x0.x - o.x) * d.x + (x0.y - o.y) * d.y + (x0.z - o.z) * d.z) / dd;
  int fixed, ua, va;
  float val;
  face_param(f, fixed, val, ua, va);
  return face_impossible(cert, f, o, d, make_float3(0.f, 0.f, 0.f), x0, t, val, tmin, tmax);
}

// How far a face may be entered and still give a hit at or before hi: hi and
// the rounding of the slab test far from the ray's origin (the hull boxes'
// own inflation covers the solver's tolerance).
__device__ __forceinline__ float seed_reach(float hi) { return fminf(hi + 1e-6f * fabsf(hi), FLT_MAX); }

// Where the predicted xi-line enters [-1,1]^3: face, start point, t.
__device__ __forceinline__ bool predicted_entry(const Pred& pr, float tmin, float tmax, int& face, float3& p,
                                                float& tau) {
  const float a[3] = {pr.xi_in.x, pr.xi_in.y, pr.xi_in.z};
  const float v[3] = {pr.v.x * pr.k, pr.v.y * pr.k, pr.v.z * pr.k};
  float enter = -FLT_MAX, leave = FLT_MAX;
  int ax = -1;
  float side = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (fabsf(v[c]) < 1e-12f) {
      if (fabsf(a[c]) > 1.f) return false;
      continue;
    }
    const float t0 = pr.te + (-1.f - a[c]) / v[c], t1 = pr.te + (1.f - a[c]) / v[c];
    const float lo = fminf(t0, t1), hi = fmaxf(t0, t1);
    if (lo > enter) {
      enter = lo;
      ax = c;
      side = (t0 < t1) ? -1.f : 1.f;
    }
    leave = fminf(leave, hi);
  }
  if (ax < 0 || enter > leave || enter > tmax || leave < tmin) return false;
  // face table (high_order.h:164-184): (axis, side) -> face index
  face = ax == 2 ? (side < 0.f ? 0 : 5) : (ax == 1 ? (side < 0.f ? 1 : 3) : (side < 0.f ? 4 : 2));
  tau = fminf(fmaxf(enter, tmin), tmax);
  p = pr.at(tau);
  setc(p, ax, side);
  return true;
}

// Warp version of hit_hex: the (face, seed) Newton solves of a step are
// independent, so they are spread over the lanes. For each face the lowest
// seed index that was accepted answers — the seed the sequential loop would
// stop at — and faces are then compared in index order as the reference does.
template <int N, bool L, bool SM>
__device__ bool hit_hex_warp(const Elem<N, SM>& e, const float* __restrict__ fbox, const float* __restrict__ cert, float3 o, float3 d, float tmin,
                             float tmax, float& th, float3& xh, int& face, Work& w, Work& wu, const Pred& pr) {
  const int lane = threadIdx.x & 31;
  // learned: one Newton solve from the predicted element entry; faces whose
  // hull box misses [tmin, t_learned] cannot hold a nearer hit and are skipped
  int lf = -1;
  float lt = 0.f;
  float3 lx = make_float3(0.f, 0.f, 0.f);
  if (L && pr.on) {
    float3 p0;
    float tau0;
    int f0;
    if (predicted_entry(pr, tmin, tmax, f0, p0, tau0) &&
        face_newton<N>(e, o, d, f0, p0, tau0, tmin, tmax, lt, lx, wu, kWarmCap)) {
      lf = f0;
      ++wu.accepted;
    } else {
      ++wu.rejected;
    }
  }
  // the seeds as next_seeds (ho_rounds.cuh) orders them, spread over the lanes;
  // seed 0 of all faces at once, since a step costs the warp the same
  const bool staged = __ldg(cert + 12) >= 0.f;
  unsigned todo = lf >= 0 ? 63u & ~(1u << lf) : 63u, tried = 0u, found = 0u;
  float tv[6];
  float3 xv[6];
  for (;;) {
    float hi = lf >= 0 ? fminf(tmax, lt) : tmax;
#pragma unroll
    for (int f = 0; f < 6; ++f)
      if (((found >> f) & 1u) && tv[f] > tmin) hi = fminf(hi, tv[f]);
    todo &= ~found;
    for (int f = 0; f < 6; ++f) {
      if (!((todo >> f) & 1u)) continue;
      if (!face_may_hit(fbox, f, o, d, tmin, seed_reach(hi)) ||
          (staged && face_excluded(cert, f, o, d, tmin, seed_reach(hi)))) {
        ++wu.culled;
        todo &= ~(1u << f);
      }
    }
    if (todo == 0u) break;
    // fresh: seed 0 (all seeds without a certificate); rest: seeds 1-8
    const unsigned now = todo;
    const unsigned rest = now & tried, fresh = now & ~tried;
    const int per = staged ? 1 : 9, n_fresh = per * __popc(fresh), T = n_fresh + 8 * __popc(rest);
    unsigned dead = 0u;
    for (int base = 0; base < T; base += 32) {
      const int k = base + lane;
      bool ok = false, none = false;
      float ts = 0.f;
      float3 xs = make_float3(0.f, 0.f, 0.f);
      int f = -1;
      if (k < T) {
        unsigned m = k < n_fresh ? fresh : rest;
        const int slot = k < n_fresh ? k / per : (k - n_fresh) >> 3;
        for (int q = 0; q < slot; ++q) m &= m - 1u;
        f = __ffs(m) - 1;
        const int sd = k < n_fresh ? k - slot * per : 1 + ((k - n_fresh) & 7);
        ok = face_seed<N>(e, o, d, f, sd % 3, sd / 3, tmin, tmax, ts, xs, w, staged && sd == 0 ? cert : nullptr, &none);
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 6; ++q) {  // each face's lowest accepted seed
        if (__any_sync(kFull, none && f == q)) dead |= 1u << q;
        const unsigned b = __ballot_sync(kFull, ok && f == q);
        if (b == 0u || ((found >> q) & 1u)) continue;
        const int src = __ffs(b) - 1;
        found |= 1u << q;
        tv[q] = __shfl_sync(kFull, ts, src);
        xv[q] = shfl3(xs, src);
      }
    }
    todo &= ~(staged ? rest | dead : now);
    tried |= now;
  }
  bool any = false;
  float best = tmax;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    if (f != lf && !((found >> f) & 1u)) continue;
    const float tf = f == lf ? lt : tv[f];
    if (tf > tmin && tf < best) {
      best = tf;
      xh = f == lf ? lx : xv[f];
      face = f;
      any = true;
    }
  }
  if (any) th = best;
  return any;
}

// Warp version of visit_candidate: every lane holds the same `best`.
template <int N, bool L, bool SM>
__device__ void visit_warp(const Elem<N, SM>& e, const float* __restrict__ fbox, const float* __restrict__ cert, int eidx, float3 o, float3 d, float te,
                           float tx, float iso, bool iso_on, HitState& best, Work& w, Work& wu, const Pred& pr,
                           HitState* tie = nullptr) {
  ++wu.cand;
  float th;
  float3 xi, g;
  if (iso_on && e.has_field && find_iso_warp<N, L>(e, o, d, te, tx, iso, th, xi, g, w, wu, pr)) {
    if (th > 0.001f && th < best.t) {
      float3 n = normalize3(g);
      if (n.x * d.x + n.y * d.y + n.z * d.z > 0.f) n = make_float3(-n.x, -n.y, -n.z);
      note_tie(best, best.t, th, tie);
      best.t = th;
      best.elem = eidx;
      best.face = -1;
      best.kind = HO_HIT_ISO;
      best.flags &= ~kFlagPost;
      best.xi = xi;
      best.n = n;
      float4 r[4];  // the field at the root: what fill_hit gives the round kernel's hits
      eval_comps<N, SM>(e.c, xi, 3, 4, r);
      best.u = r[3].x;
    }
    return;
  }
  int face = -1;
  const long long c0 = clock64();
  const bool fh = hit_hex_warp<N, L>(e, fbox, cert, o, d, 0.001f, best.t, th, xi, face, w, wu, pr);
  wu.cyc[3] += clock64() - c0;
  if (fh) {
    if (th > 0.001f && th < best.t) {
      // geometry (and field) at the hit: what fill_hit gives the round kernel's hits
      float4 r[4];
      eval_comps<N, SM>(e.c, xi, 0, e.has_field ? 4 : 3, r);
      ++wu.geom;
      const float J[9] = {r[0].y, r[0].z, r[0].w, r[1].y, r[1].z, r[1].w, r[2].y, r[2].z, r[2].w};
      const float3 n = face_normal(J, xi, d);
      note_tie(best, best.t, th, tie);
      best.t = th;
      best.elem = eidx;
      best.face = face;
      best.kind = HO_HIT_FACE;
      best.flags &= ~kFlagPost;
      best.xi = xi;
      best.n = n;
      best.u = e.has_field ? r[3].x : 0.f;
    }
  }
}

}  // namespace ho
