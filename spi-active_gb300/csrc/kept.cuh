// kept.cuh -- substeps kept by a forward pass for the sweeps that follow it (adjoint.cu, sensitivity.cu).
//
// Per rollout and physics substep, 736 bytes in 16-byte fields: per leg the factorisation of its equations
// (K', y, L, D^-1), its joint state and its foot contact's height and branch; for the base its state,
// its acceleration and the Cholesky factor of its articulated inertia. A warp's accesses to a field are
// contiguous; they are written and read once, past the caches.
#pragma once

#include <cuda_runtime.h>

#include "adjoint.cuh"
#include "rollout.cuh"

namespace spi {

constexpr int kLegFields = 9;                       // 16-byte fields per leg and kept substep
constexpr int kBaseFields = 10;                     // and per rollout
constexpr size_t kKeptBytes = 16 * (4 * kLegFields + kBaseFields);   // per rollout and substep

__device__ __forceinline__ float scalar_value(float x) { return x; }

// Cholesky factor of a 6x6 symmetric positive definite matrix: the strict lower triangle by rows and
// the inverse diagonal.
struct Factor6 {
  float l[15], inv[6];
  template <class T> __device__ __forceinline__ void put_factor(const T (*Mx)[6], const T* invL) {
    int k = 0;
#pragma unroll
    for (int i = 1; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) l[k++] = scalar_value(Mx[i][j]);
#pragma unroll
    for (int i = 0; i < 6; ++i) inv[i] = scalar_value(invL[i]);
  }
  __device__ __forceinline__ SV<float> solve(const SV<float>& b) const {
    float x[6] = {b.w.x, b.w.y, b.w.z, b.v.x, b.v.y, b.v.z};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      float a = x[i];
#pragma unroll
      for (int k = 0; k < i; ++k) a = a - l[i * (i - 1) / 2 + k] * x[k];
      x[i] = a * inv[i];
    }
#pragma unroll
    for (int i = 5; i >= 0; --i) {
      float a = x[i];
#pragma unroll
      for (int k = i + 1; k < 6; ++k) a = a - l[k * (k - 1) / 2 + i] * x[k];
      x[i] = a * inv[i];
    }
    SV<float> r;
    r.w = v3(x[0], x[1], x[2]);
    r.v = v3(x[3], x[4], x[5]);
    return r;
  }
};

// A rollout's kept substeps: leg fields [slot][field][4 rollouts], base fields [slot][field][rollouts].
struct Kept {
  float4* leg;     // at this lane
  float4* base;    // at this lane's rollout
  size_t leg_slot, base_slot;   // 16-byte fields from one slot to the next (of the whole batch)
  size_t leg_field, base_field;
  // legs, base: the batch's fields for `rollouts` rollouts
  __device__ __forceinline__ static Kept of(float4* legs, float4* base, size_t rollouts, size_t rollout, int leg) {
    return Kept{legs + 4 * rollout + leg, base + rollout, 4 * rollouts * kLegFields, rollouts * kBaseFields, 4 * rollouts,
                rollouts};
  }
  __device__ __forceinline__ float4* leg_at(int slot, int f) const { return leg + slot * leg_slot + f * leg_field; }
  __device__ __forceinline__ float4* base_at(int slot, int f) const { return base + slot * base_slot + f * base_field; }
};

__device__ __forceinline__ void keep_state(const Kept& k, int slot, int leg, const BaseState<float>& B) {
  if (leg != 0) return;
  __stcs(k.base_at(slot, 0), make_float4(B.p.x, B.p.y, B.p.z, B.qx));
  __stcs(k.base_at(slot, 1), make_float4(B.qy, B.qz, B.qw, B.nu.w.x));
  __stcs(k.base_at(slot, 2), make_float4(B.nu.w.y, B.nu.w.z, B.nu.v.x, B.nu.v.y));
}
__device__ __forceinline__ void keep_legs(const Kept& k, int slot, const float d[3], const LegState<float>& L,
                                          float zf = 0.f, float branch = 0.f) {
  __stcs(k.leg_at(slot, 6), make_float4(d[0], d[1], d[2], L.q[0]));
  __stcs(k.leg_at(slot, 7), make_float4(L.q[1], L.q[2], L.qd[0], L.qd[1]));
  __stcs(k.leg_at(slot, 8), make_float4(L.qd[2], zf, branch, 0.f));
}
// The base acceleration and the Cholesky factor of a kept substep (nuz: the state's last value).
__device__ __forceinline__ void keep_solve(const Kept& k, int slot, int leg, float nuz, const SV<float>& a0,
                                           const Factor6& fac) {
  if (leg != 0) return;
  __stcs(k.base_at(slot, 3), make_float4(nuz, a0.w.x, a0.w.y, a0.w.z));
  __stcs(k.base_at(slot, 4), make_float4(a0.v.x, a0.v.y, a0.v.z, fac.l[0]));
#pragma unroll
  for (int f = 0; f < 3; ++f)
    __stcs(k.base_at(slot, 5 + f), make_float4(fac.l[4 * f + 1], fac.l[4 * f + 2], fac.l[4 * f + 3], fac.l[4 * f + 4]));
  __stcs(k.base_at(slot, 8), make_float4(fac.l[13], fac.l[14], fac.inv[0], fac.inv[1]));
  __stcs(k.base_at(slot, 9), make_float4(fac.inv[2], fac.inv[3], fac.inv[4], fac.inv[5]));
}
// The state and, for WORK, the factorisations of a kept substep.
template <bool WORK>
__device__ __forceinline__ void load_kept(const Kept& k, int slot, BaseState<float>& B, LegState<float>& L,
                                          adj::SolveWork<float>& W, Factor6& fac, SV<float>& a0) {
  const float4 b0 = __ldcs(k.base_at(slot, 0)), b1 = __ldcs(k.base_at(slot, 1)), b2 = __ldcs(k.base_at(slot, 2)),
               b3 = __ldcs(k.base_at(slot, 3));
  const float4 l6 = __ldcs(k.leg_at(slot, 6)), l7 = __ldcs(k.leg_at(slot, 7)), l8 = __ldcs(k.leg_at(slot, 8));
  if (WORK) {
    float l[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 u = __ldcs(k.leg_at(slot, 2 * c)), v = __ldcs(k.leg_at(slot, 2 * c + 1));
      W.Kp[c].w = v3(u.x, u.y, u.z);
      W.Kp[c].v = v3(u.w, v.x, v.y);
      W.y[c] = v.z;
      l[c] = v.w;
    }
    W.l10 = l[0]; W.l20 = l[1]; W.l21 = l[2];
    W.i[0] = l6.x; W.i[1] = l6.y; W.i[2] = l6.z;
    float v[24];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const float4 u = __ldcs(k.base_at(slot, 4 + f));
      v[4 * f] = u.x; v[4 * f + 1] = u.y; v[4 * f + 2] = u.z; v[4 * f + 3] = u.w;
    }
    a0.w = v3(b3.y, b3.z, b3.w);
    a0.v = v3(v[0], v[1], v[2]);
#pragma unroll
    for (int i = 0; i < 15; ++i) fac.l[i] = v[3 + i];
#pragma unroll
    for (int i = 0; i < 6; ++i) fac.inv[i] = v[18 + i];
  }
  B.p = v3(b0.x, b0.y, b0.z);
  B.qx = b0.w; B.qy = b1.x; B.qz = b1.y; B.qw = b1.z;
  B.nu.w = v3(b1.w, b2.x, b2.y);
  B.nu.v = v3(b2.z, b2.w, b3.x);
  B.R = quat_to_R(B.qx, B.qy, B.qz, B.qw);
  L.q[0] = l6.w; L.q[1] = l7.x; L.q[2] = l7.y;
  L.qd[0] = l7.z; L.qd[1] = l7.w; L.qd[2] = l8.x;
}

// Asynchronous copies of kept fields to shared memory (16 bytes each).
__device__ __forceinline__ void copy_async(float4* dst, const float4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// A kept substep of one rollout in shared memory, as one lane of its quad sees it: the lane's leg's fields and
// the base's.
struct KeptView {
  const float4* leg;
  const float4* base;
  __device__ __forceinline__ float4 legf(int i) const { return leg[i]; }
  __device__ __forceinline__ float4 basef(int i) const { return base[i]; }
  __device__ __forceinline__ BaseState<float> state() const {
    const float4 b0 = basef(0), b1 = basef(1), b2 = basef(2);
    BaseState<float> B;
    B.p = v3(b0.x, b0.y, b0.z);
    B.qx = b0.w; B.qy = b1.x; B.qz = b1.y; B.qw = b1.z;
    B.nu.w = v3(b1.w, b2.x, b2.y);
    B.nu.v = v3(b2.z, b2.w, basef(3).x);
    B.R = quat_to_R(B.qx, B.qy, B.qz, B.qw);
    return B;
  }
  __device__ __forceinline__ SV<float> accel() const {
    const float4 u = basef(3), v = basef(4);
    SV<float> a;
    a.w = v3(u.y, u.z, u.w);
    a.v = v3(v.x, v.y, v.z);
    return a;
  }
  __device__ __forceinline__ Factor6 factor() const {
    float v[24];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const float4 u = basef(4 + f);
      v[4 * f] = u.x; v[4 * f + 1] = u.y; v[4 * f + 2] = u.z; v[4 * f + 3] = u.w;
    }
    Factor6 r;
#pragma unroll
    for (int i = 0; i < 15; ++i) r.l[i] = v[3 + i];
#pragma unroll
    for (int i = 0; i < 6; ++i) r.inv[i] = v[18 + i];
    return r;
  }
  __device__ __forceinline__ adj::SolveWork<float> work() const {
    adj::SolveWork<float> W;
    float l[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 u = legf(2 * c), v = legf(2 * c + 1);
      W.Kp[c].w = v3(u.x, u.y, u.z);
      W.Kp[c].v = v3(u.w, v.x, v.y);
      W.y[c] = v.z;
      l[c] = v.w;
    }
    W.l10 = l[0]; W.l20 = l[1]; W.l21 = l[2];
    const float4 d = legf(6);
    W.i[0] = d.x; W.i[1] = d.y; W.i[2] = d.z;
    return W;
  }
  __device__ __forceinline__ LegState<float> leg_state() const {
    const float4 u = legf(6), v = legf(7);
    LegState<float> L;
    L.q[0] = u.w; L.q[1] = v.x; L.q[2] = v.y;
    L.qd[0] = v.z; L.qd[1] = v.w; L.qd[2] = legf(8).x;
    return L;
  }
};

}  // namespace spi
