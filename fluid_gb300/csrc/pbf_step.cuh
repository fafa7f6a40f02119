// The arithmetic of one step's phases, one particle at a time: what a pass sums over the
// neighbours and what it makes of the sums. Shared by the per-phase kernels (pbf_kernels.cu) and
// the whole-step kernel of small scenes (pbf_small.cu), which give the same bits: every rounding
// of the sums is explicit.
#pragma once

#include "pbf_device.cuh"

namespace pbf {

// Order-preserving unsigned image of a float (a total order, NaN included).
__device__ __forceinline__ uint32_t order_bits(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Rank of each lane's key among the cell's particles (particles.cpp:254-265 have no grid): one
// atomic on the cell's count per run of equal keys among consecutive lanes (the slots are still
// mostly in the cell order of the last step; measured 38 against 42 us a step for one atomic
// per distinct key of the warp by __match_any_sync on scrambled cells). All lanes of the warp
// call it; dead lanes carry the key 0xffffffff, a run of their own.
__device__ __forceinline__ uint32_t count_rank(uint32_t key, bool live, uint32_t* cell_count) {
  const unsigned lane = lane_id();
  const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
  const bool head = lane == 0 || prev != key;
  const unsigned heads = __ballot_sync(0xffffffffu, head);
  const unsigned upto = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);  // lanes 0..lane
  const int start = 31 - __clz(heads & upto);                            // this lane's run head
  const unsigned above = heads & ~upto;
  const int next = above ? __ffs(above) - 1 : 32;                        // the next run's head
  uint32_t base = 0;
  if (head && live) base = atomicAdd(&cell_count[key], static_cast<uint32_t>(next - static_cast<int>(lane)));
  base = __shfl_sync(0xffffffffu, base, start);
  return base + (lane - static_cast<unsigned>(start));
}

// Density and lambda (particles.cpp:185-204).
struct LambdaSum {
  float qsum = 0.f, g2 = 0.f;
  float3 gs = make_float3(0.f, 0.f, 0.f);
  __device__ __forceinline__ void add(const float4& xi, const float4& xj, const DevParams& P) {
    const Pair p = pair_of(xi, xj, P.h, P.h2);
    qsum = __fmaf_rn(__fmul_rn(p.q, p.q), p.q, qsum);
    gs = fma3(p.r, p.s, gs);
    g2 = __fmaf_rn(__fmul_rn(p.s, p.s), p.r2, g2);
  }
  __device__ __forceinline__ float lambda(const DevParams& P, float* rho_out) const {
    const float rho = __fmul_rn(P.poly6_c, qsum);
    const float kg = __fmul_rn(P.spiky_c, P.inv_rho0);
    const float denom = __fmaf_rn(__fmul_rn(kg, kg), __fadd_rn(g2, dot3_rn(gs, gs)), P.epsilon);
    *rho_out = rho;
    return -__fdiv_rn(__fmaf_rn(rho, P.inv_rho0, -1.0f), denom);
  }
};

// Delta p = sum of (lambda_i + lambda_j + s_corr) grad W over rho0 (particles.cpp:206-213); N4
// specialises the tensile exponent N = 4 of particles.cpp:40.
template <bool N4>
__device__ __forceinline__ float3 delta_term(const float4& xi, const float4& xj, float wt, const DevParams& P,
                                             float* c) {
  const Pair p = pair_of(xi, xj, P.h, P.h2);
  const float a = __fmul_rn(wt, __fmul_rn(__fmul_rn(p.q, p.q), p.q));  // W / W(dq)
  float an;
  if (N4) {
    const float a2 = __fmul_rn(a, a);
    an = __fmul_rn(a2, a2);
  } else {
    an = a;
    for (int e = 1; e < P.scorr_n; ++e) an = __fmul_rn(an, a);
  }
  const float coef = __fmaf_rn(-P.scorr_k, an, __fadd_rn(xi.w, xj.w));  // lambda_i + lambda_j + s_corr
  *c = __fmul_rn(coef, p.s);
  return p.r;
}
template <bool N4>
struct DeltaSum {
  float3 dp = make_float3(0.f, 0.f, 0.f);
  __device__ __forceinline__ void add(const float4& xi, const float4& xj, float wt, const DevParams& P) {
    float c;
    const float3 r = delta_term<N4>(xi, xj, wt, P, &c);
    dp = fma3(r, c, dp);
  }
  __device__ __forceinline__ float3 delta(const DevParams& P) const {
    const float sc = __fmul_rn(P.spiky_c, P.inv_rho0);
    return make_float3(__fmul_rn(dp.x, sc), __fmul_rn(dp.y, sc), __fmul_rn(dp.z, sc));
  }
};

// Velocity, vorticity, XSPH and the reported density (particles.cpp:215-234).
struct XD {
  float4 x, d;  // a neighbour's x* and displacement
};
struct XsphTerm {
  float3 vij, w;  // u_j - u_i; its cross product with the spiky direction
  float q3;
};
__device__ __forceinline__ XsphTerm xsph_term(const float4& xi, const float3& vi, const XD& a, float inv_dt,
                                              const DevParams& P) {
  const Pair p = pair_of(xi, a.x, P.h, P.h2);
  XsphTerm t;
  t.vij = make_float3(__fmaf_rn(a.d.x, inv_dt, -vi.x), __fmaf_rn(a.d.y, inv_dt, -vi.y),
                      __fmaf_rn(a.d.z, inv_dt, -vi.z));
  t.q3 = __fmul_rn(__fmul_rn(p.q, p.q), p.q);
  const float3 rs = make_float3(__fmul_rn(p.r.x, p.s), __fmul_rn(p.r.y, p.s), __fmul_rn(p.r.z, p.s));
  t.w = make_float3(__fmaf_rn(t.vij.y, rs.z, -__fmul_rn(t.vij.z, rs.y)),
                    __fmaf_rn(t.vij.z, rs.x, -__fmul_rn(t.vij.x, rs.z)),
                    __fmaf_rn(t.vij.x, rs.y, -__fmul_rn(t.vij.y, rs.x)));
  return t;
}
struct XsphSum {
  float qsum = 0.f;
  float3 visc = make_float3(0.f, 0.f, 0.f), w = make_float3(0.f, 0.f, 0.f);
  __device__ __forceinline__ void add(const float4& xi, const float3& vi, const XD& a, float inv_dt,
                                      const DevParams& P) {
    const XsphTerm t = xsph_term(xi, vi, a, inv_dt, P);
    visc = fma3(t.vij, t.q3, visc);
    qsum = __fadd_rn(qsum, t.q3);
    w = make_float3(__fadd_rn(w.x, t.w.x), __fadd_rn(w.y, t.w.y), __fadd_rn(w.z, t.w.z));
  }
  __device__ __forceinline__ float rho(const DevParams& P) const { return __fmul_rn(P.poly6_c, qsum); }
  __device__ __forceinline__ float3 velocity(const float3& vi, const DevParams& P) const {
    return fma3(visc, __fmul_rn(P.xsph_c, P.poly6_c), vi);
  }
  __device__ __forceinline__ float4 omega(const DevParams& P) const {  // w: its length
    const float3 o = make_float3(__fmul_rn(w.x, P.spiky_c), __fmul_rn(w.y, P.spiky_c), __fmul_rn(w.z, P.spiky_c));
    return make_float4(o.x, o.y, o.z, __fsqrt_rn(dot3_rn(o, o)));
  }
};

// Vorticity confinement (particles.cpp:236-248).
__device__ __forceinline__ float3 vort_term(const float4& xi, const float4& xj, const DevParams& P, float* c) {
  const Pair p = pair_of(xi, xj, P.h, P.h2);
  *c = __fmul_rn(xj.w, p.s);  // |omega_j| s
  return p.r;
}
struct VortSum {
  float3 eta = make_float3(0.f, 0.f, 0.f);
  __device__ __forceinline__ void add(const float4& xi, const float4& xj, const DevParams& P) {
    float c;
    const float3 r = vort_term(xi, xj, P, &c);
    eta = fma3(r, c, eta);
  }
  __device__ __forceinline__ float3 location(const DevParams& P) const {
    return make_float3(__fmul_rn(eta.x, P.spiky_c), __fmul_rn(eta.y, P.spiky_c), __fmul_rn(eta.z, P.spiky_c));
  }
};
// v + dt eps (eta / |eta|) x omega
__device__ __forceinline__ float3 confined(const float3& v, const float3& eta, const float4& wi, float dt,
                                           const DevParams& P) {
  const float en = __fsqrt_rn(dot3_rn(eta, eta));
  if (!(en > kEps)) return v;
  const float ie = __fdiv_rn(1.0f, en);
  const float3 nh = make_float3(__fmul_rn(eta.x, ie), __fmul_rn(eta.y, ie), __fmul_rn(eta.z, ie));
  const float3 c = make_float3(__fmaf_rn(nh.y, wi.z, -__fmul_rn(nh.z, wi.y)),
                               __fmaf_rn(nh.z, wi.x, -__fmul_rn(nh.x, wi.z)),
                               __fmaf_rn(nh.x, wi.y, -__fmul_rn(nh.y, wi.x)));
  return fma3(c, __fmul_rn(dt, P.vort_eps), v);
}

}  // namespace pbf
