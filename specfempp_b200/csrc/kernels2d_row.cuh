// Row form of the owner-computes element kernel (single shot; isotropic P-SV,
// SH, poroelastic and acoustic media, one launch for both media of a model).
//
// One thread per element row (the five points of a row iz), E elements per
// block (5 E threads).  The xi-direction contractions of the gradient and of
// the divergence run on the row in registers with warp-uniform coefficients
// (constant bank), the gamma-direction ones read columns of the element's
// displacement and F1 in shared memory, so a point needs a fifth of the
// shared-memory and coefficient loads of the point-per-thread kernel.  Per
// point the operations and their order are those of elastic_block<E, EK, true>
// and acoustic_block<E, true> (components paired in FFMA2 for P-SV and
// poroelastic media, the two directions paired for the scalar ones; FFMA2
// rounds each lane as fmaf), so the results are the same bits.
//
// What bounded it (element launch of the fluid-solid 400x200 model, 2.0 M
// element points, each launch chained to the one before, so that they overlap;
// one after another 27.0 us before and 18.4 us now, acoustic 125 k elements 21
// us, poroelastic 22.5 k elements 12.3 us):
// * 24.9 us: the geometry and material words, 28 of 52 B an element point.
//   The specialisations below: 19.2 us.
// * the coefficient rows of a thread (its iz) from the constant bank: threads
//   of a warp hold different iz, indexed constant loads are served one
//   address at a time and the compiler reloads them at every use (the
//   indexed-constant unit 77% busy in the acoustic rows, 43.5 us for 125 k
//   elements).  From global memory, held in registers: 15.9 us here, 19.3 us
//   there.
// * a row per thread makes every load of a warp stride five points and cost
//   several wavefronts of the L1: the block's points are gathered into shared
//   memory, and its results scattered from there, with consecutive threads on
//   consecutive points, and per-point words arrive by 16-byte cp.async; rows
//   are then read at a stride of five words, which no two lanes map to one
//   bank.  That takes 12% off the poroelastic kernel (10.6 -> 9.4 us, 22.5 k
//   elements) and nothing from the others.
//
// The kernel is specialised on what the mesh lets it not load (chosen for the
// whole mesh at set-up, RowClass in host2d.hpp):
//   GEO 1  every element is a rectangle along the axes: xi_z and gamma_x are
//          exactly zero and xi_x, gamma_z, |J| one value an element.  Three
//          words an element in place of five a point, and the products with
//          the zero words drop out; x + 0 and x * 0 change no bit of a finite
//          result, so this is the general kernel's arithmetic.
//   MAT 1  the material words are one value an element (layered models).
// An element's values are one 32-byte record (64 bytes poroelastic), read by
// its five threads from the same sectors.
// Reference: include/kokkos_kernels/impl/compute_stiffness_interaction.tpp:140-247,
// include/algorithms/gradient.hpp:40-82, divergence.hpp:41-74,
// include/medium/dim2/*/isotropic/stress.hpp,
// include/boundary_conditions/stacey/stacey.tpp:50-80, 130-146, 291-326,
// include/kokkos_kernels/impl/compute_source_interaction.tpp:17-104.
#pragma once

#include "kernels2d_batched.cuh"

namespace sfg {
namespace dev {

// n floats (a multiple of 4, both ends 16-byte aligned) into shared memory by
// all threads of the block; cp_async_wait before the barrier that publishes it.
template <int THREADS>
__device__ __forceinline__ void cp_async_block(float *dst, const float *src, int n) {
  for (int i = threadIdx.x; i < n / 4; i += THREADS)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst + 4 * i))),
                 "l"(src + 4 * i)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Geometry of a row's points: the block's staged arrays [5][25 E] (GEO 0) or
// the element's record.
template <int E, int GEO>
struct RowGeo {
  const float *s;      // staged xi_x of the row's first point; the others 25 E floats apart
  __device__ __forceinline__ void stage(const MedArgs &A, size_t p0, float *sg) const {
    constexpr int N = NP * E;
    cp_async_block<NG * E>(sg, A.xix + p0, N);
    cp_async_block<NG * E>(sg + N, A.xiz + p0, N);
    cp_async_block<NG * E>(sg + 2 * N, A.gax + p0, N);
    cp_async_block<NG * E>(sg + 3 * N, A.gaz + p0, N);
    cp_async_block<NG * E>(sg + 4 * N, A.jac + p0, N);
  }
  __device__ __forceinline__ void load(const MedArgs &, size_t, const float *sg, int row) { s = sg + row; }
  struct Pt {
    float xix, xiz, gax, gaz, jac;
    // physical derivatives from the reference ones
    __device__ __forceinline__ float ddx(float dxi, float dga) const { return xix * dxi + gax * dga; }
    __device__ __forceinline__ float ddz(float dxi, float dga) const { return xiz * dxi + gaz * dga; }
    // F0, F1 of one component from its stress row (sx, sz)
    __device__ __forceinline__ float f0(float sx, float sz) const { return jac * (sx * xix + sz * xiz); }
    __device__ __forceinline__ float f1(float sx, float sz) const { return jac * (sx * gax + sz * gaz); }
  };
  __device__ __forceinline__ Pt at(int ix) const {
    constexpr int N = NP * E;
    return Pt{s[ix], s[N + ix], s[2 * N + ix], s[3 * N + ix], s[4 * N + ix]};
  }
  __device__ __forceinline__ float j(int ix) const { return s[4 * NP * E + ix]; }
};

template <int E>
struct RowGeo<E, 1> {
  struct Pt {
    float xix, gaz, jac;
    __device__ __forceinline__ float ddx(float dxi, float) const { return xix * dxi; }
    __device__ __forceinline__ float ddz(float, float dga) const { return gaz * dga; }
    __device__ __forceinline__ float f0(float sx, float) const { return jac * (sx * xix); }
    __device__ __forceinline__ float f1(float, float sz) const { return jac * (sz * gaz); }
  } p;
  __device__ __forceinline__ void stage(const MedArgs &, size_t, float *) const {}
  __device__ __forceinline__ void load(const MedArgs &A, size_t rec, const float *, int) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(A.erec + rec));
    p.xix = t.x; p.gaz = t.y; p.jac = t.z;
  }
  __device__ __forceinline__ Pt at(int) const { return p; }
  __device__ __forceinline__ float j(int) const { return p.jac; }
};

// Two material words of a row's points (MAT 0, staged [2][25 E]) or of the
// element (MAT 1).
template <int E, int MAT>
struct RowMat {
  const float *s;
  __device__ __forceinline__ void stage(const MedArgs &A, size_t p0, float *sg) const {
    cp_async_block<NG * E>(sg, A.prop0 + p0, NP * E);
    cp_async_block<NG * E>(sg + NP * E, A.prop1 + p0, NP * E);
  }
  __device__ __forceinline__ void load(const MedArgs &, size_t, const float *sg, int row) { s = sg + row; }
  __device__ __forceinline__ float c0(int ix) const { return s[ix]; }
  __device__ __forceinline__ float mu(int ix) const { return s[NP * E + ix]; }
};

template <int E>
struct RowMat<E, 1> {
  float c0_, mu_;
  __device__ __forceinline__ void stage(const MedArgs &, size_t, float *) const {}
  __device__ __forceinline__ void load(const MedArgs &A, size_t rec, const float *, int) {
    const float2 t = __ldg(reinterpret_cast<const float2 *>(A.erec + rec + 4));
    c0_ = t.x; mu_ = t.y;
  }
  __device__ __forceinline__ float c0(int) const { return c0_; }
  __device__ __forceinline__ float mu(int) const { return mu_; }
};

// Shared floats of a block: displacement (later the results) and F1, the
// poroelastic fluid velocity, then the staged words.
template <int E, int EK, int GEO, int MAT>
__host__ __device__ constexpr int row_smem() {
  constexpr int nc = EK == 4 ? 4 : (EK == 0 ? 2 : 1);
  return NP * E * (2 * nc + (EK == 4 ? 2 : 0) + (GEO ? 0 : 5) + (MAT ? 0 : 2));
}

// P-SV (EK 0) and poroelastic (EK 4) rows: NH component pairs.
template <int E, int EK, int GEO, int MAT>
__device__ __forceinline__ void pair_rows(const StiffArgs &S, const MedArgs &A, int ebase, float *smem) {
  constexpr int NH = EK == 4 ? 2 : 1, T = NG * E;
  const int tid = threadIdx.x;
  const int le = tid / NG, iz = tid - le * NG;
  const int e = ebase + le;
  const bool act = e < A.e1;
  float2 *sub = reinterpret_cast<float2 *>(smem), *sF1b = sub + NP * E * NH;     // [25 E][NH]
  float2 *sv = sF1b + NP * E * NH;                                               // poroelastic [25 E]
  float *sg = smem + NP * E * (4 * NH + (EK == 4 ? 2 : 0));
  float *sm = sg + (GEO ? 0 : 5 * NP * E);
  float2 *su = sub + le * NP * NH, *sF1 = sF1b + le * NP * NH;
  const size_t ee = act ? e : A.e0, p0 = size_t(ebase) * NP, pend = size_t(A.e1) * NP;
  const size_t rec = ee * (EK == 4 ? 16 : 8);
  RowGeo<E, GEO> G;
  RowMat<E, MAT> M;
  // static words before the wait: staged arrays, records, this thread's five
  // points' indices
  G.stage(A, p0, sg);
  M.stage(A, p0, sm);
  int g[NG], sl[NG];
#pragma unroll
  for (int k = 0; k < NG; ++k) {
    const size_t p = p0 + tid + k * T;
    g[k] = p < pend ? __ldg(A.ibool + p) : -1;
    sl[k] = p < pend ? __ldg(A.slot + p) : 0;
  }
  G.load(A, rec, sg, tid * NG);
  M.load(A, rec, sm, tid * NG);
  float4 pw0, pw1;     // poroelastic: C, M, phi / tort, rho_f / rho_bar; eta_f k^-1 (xx, xz, zz)
  if (EK == 4) {
    pw0 = __ldg(reinterpret_cast<const float4 *>(A.erec + rec + 8));
    pw1 = __ldg(reinterpret_cast<const float4 *>(A.erec + rec + 12));
  }
  float hz[NG];
  ld_row5(t_rows[iz], hz);
  pdl_wait();
  pdl_release();
  if (NH == 1) {
    float2 t[NG];
#pragma unroll
    for (int k = 0; k < NG; ++k) t[k] = g[k] >= 0 ? ld_dep2(A.u + size_t(g[k]) * 2) : make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < NG; ++k) sub[tid + k * T] = t[k];
  } else {
    float4 t[NG];
    float2 v[NG];
#pragma unroll
    for (int k = 0; k < NG; ++k) {
      t[k] = g[k] >= 0 ? ld_dep4(A.u + size_t(g[k]) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[k] = g[k] >= 0 ? ld_dep2(A.v + size_t(g[k]) * 4 + 2) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < NG; ++k) {
      sub[(tid + k * T) * 2] = make_float2(t[k].x, t[k].y);
      sub[(tid + k * T) * 2 + 1] = make_float2(t[k].z, t[k].w);
      sv[tid + k * T] = v[k];
    }
  }
  if (GEO == 0 || MAT == 0) cp_async_wait();
  __syncthreads();
  // xi derivatives of the row's points (components paired)
  float2 ur[NG][NH];
#pragma unroll
  for (int h = 0; h < NH; ++h) {
    float2 x[NG];
#pragma unroll
    for (int l = 0; l < NG; ++l) x[l] = su[(iz * NG + l) * NH + h];
#pragma unroll
    for (int ix = 0; ix < NG; ++ix) {
      float2 px = make_float2(0.f, 0.f);
#pragma unroll
      for (int l = 0; l < NG; ++l) px = fma2(f2(c_hp[ix * NG + l]), x[l], px);
      ur[ix][h] = px;
    }
  }
#pragma unroll
  for (int ix = 0; ix < NG; ++ix) {
    float2 pg[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      pg[h] = make_float2(0.f, 0.f);
#pragma unroll
      for (int l = 0; l < NG; ++l) pg[h] = fma2(f2(hz[l]), su[(l * NG + ix) * NH + h], pg[h]);
    }
    const auto P = G.at(ix);
    const float c0 = M.c0(ix), mu = M.mu(ix);
    const float du00 = P.ddx(ur[ix][0].x, pg[0].x), du01 = P.ddz(ur[ix][0].x, pg[0].x);
    const float du10 = P.ddx(ur[ix][0].y, pg[0].y), du11 = P.ddz(ur[ix][0].y, pg[0].y);
    const float lam = c0 - 2.f * mu;
    if (EK == 0) {
      const float sxx = c0 * du00 + lam * du11;
      const float szz = c0 * du11 + lam * du00;
      const float sxz = mu * (du01 + du10);
      // stress rows (sxx, sxz) of x and (sxz, szz) of z
      ur[ix][0] = make_float2(P.f0(sxx, sxz), P.f0(sxz, szz));
      sF1[iz * NG + ix] = make_float2(P.f1(sxx, sxz), P.f1(sxz, szz));
    } else {
      const float du20 = P.ddx(ur[ix][NH - 1].x, pg[NH - 1].x);
      const float du31 = P.ddz(ur[ix][NH - 1].y, pg[NH - 1].y);
      const float l2m = lam + 2.0f * mu;   // c0 = H_Biot, mu = mu_G
      const float dw = du20 + du31;
      const float sxx = l2m * du00 + lam * du11 + pw0.x * dw;
      const float szz = l2m * du11 + lam * du00 + pw0.x * dw;
      const float sxz = mu * (du01 + du10);
      const float sp = pw0.x * (du00 + du11) + pw0.y * dw;
      const float pt = pw0.z, rr = pw0.w;
      const float tx = sxx - pt * sp, tz = szz - pt * sp, qx = sp - rr * sxx, qs = -1.0f * rr * sxz, qz = sp - rr * szz;
      ur[ix][0] = make_float2(P.f0(tx, sxz), P.f0(sxz, tz));
      ur[ix][NH - 1] = make_float2(P.f0(qx, qs), P.f0(qs, qz));
      sF1[(iz * NG + ix) * NH] = make_float2(P.f1(tx, sxz), P.f1(sxz, tz));
      sF1[(iz * NG + ix) * NH + NH - 1] = make_float2(P.f1(qx, qs), P.f1(qs, qz));
    }
  }
  float wz[NG];
  ld_row5(t_rows[5 + iz], wz);
  const float wiz = ld_w(iz);
  const int bs = act ? __ldg(A.bc_slot + e) : -1;
  const int src = act ? __ldg(A.src_head + e) : -1;
  __syncthreads();
#pragma unroll
  for (int ix = 0; ix < NG; ++ix) {
    const int q = iz * NG + ix;
    float a[2 * NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      float2 t1 = make_float2(0.f, 0.f), t2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int l = 0; l < NG; ++l) {
        t1 = fma2(ur[l][h], f2(c_hpw[l * NG + ix]), t1);
        t2 = fma2(sF1[(l * NG + ix) * NH + h], f2(wz[l]), t2);
      }
      a[2 * h] = -(wiz * t1.x + c_w[ix] * t2.x);
      a[2 * h + 1] = -(wiz * t1.y + c_w[ix] * t2.y);
    }
    if (EK == 4) {
      // viscous damping of the fluid motion; factor w_x w_z |J|
      const float2 vf = sv[le * NP + q];
      const float fac = c_w[ix] * wiz * G.j(ix);
      const float viscx = fac * ((pw1.x * vf.x) + (pw1.y * vf.y));
      const float viscz = fac * ((pw1.y * vf.x) + (pw1.z * vf.y));
      a[0] += pw0.z * viscx;
      a[1] += pw0.z * viscz;
      a[2 * NH - 2] -= viscx;
      a[2 * NH - 1] -= viscz;
    }
    if (EK == 0 && bs >= 0) {
      const size_t k = size_t(bs) * NP + q;
      const float wq = A.bc_w[k];
      if (wq != 0.f) {
        const float nx = A.bc_nx[k], nz = A.bc_nz[k], j1 = A.bc_j1[k];
        const float2 vv = ld_dep2(A.v + size_t(__ldg(A.ibool + ee * NP + q)) * 2);
        const float rvp = A.bc_imp0[k], rvs = A.bc_imp1[k];
        const float vn = vv.x * nx + vv.y * nz;
        const float fx = ((vn * nx / (j1 * j1)) * (rvp - rvs)) + vv.x * rvs;
        const float fz = ((vn * nz / (j1 * j1)) * (rvp - rvs)) + vv.y * rvs;
        a[0] += -1.f * fx * j1 * wq;
        a[1] += -1.f * fz * j1 * wq;
      }
    }
    if (src >= 0) {
      const int step = ld_dep(S.step);
      for (int s = src; s >= 0; s = S.src_next[s]) {
        const float f = step < S.nstep ? ld_dep(S.stf + size_t(step) * S.nsrc + s) : 0.f;
        a[0] += f * S.src_arr[(size_t(s) * 2 + 0) * NP + q];
        a[1] += f * S.src_arr[(size_t(s) * 2 + 1) * NP + q];
        if (EK == 4) {
          a[2 * NH - 2] += f * S.src_arr2[(size_t(s) * 2 + 0) * NP + q];
          a[2 * NH - 1] += f * S.src_arr2[(size_t(s) * 2 + 1) * NP + q];
        }
      }
    }
    // the displacement has been read by all: its place takes the results
    su[q * NH] = make_float2(a[0], a[1]);
    if (NH == 2) su[q * NH + NH - 1] = make_float2(a[2 * NH - 2], a[2 * NH - 1]);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NG; ++k) {
    if (g[k] < 0) continue;
    if (NH == 1) {
      reinterpret_cast<float2 *>(A.r)[sl[k]] = sub[tid + k * T];
    } else {
      const float2 x = sub[(tid + k * T) * 2], y = sub[(tid + k * T) * 2 + 1];
      reinterpret_cast<float4 *>(A.r)[sl[k]] = make_float4(x.x, x.y, y.x, y.y);
    }
  }
}

// Scalar rows: acoustic (SH false: sigma = rho^-1 grad chi) and SH (sigma =
// mu grad u_y), the two derivative directions paired.
template <int E, bool SH, int GEO, int MAT>
__device__ __forceinline__ void scalar_rows(const StiffArgs &S, const MedArgs &A, int ebase, float *smem) {
  constexpr int T = NG * E;
  const int tid = threadIdx.x;
  const int le = tid / NG, iz = tid - le * NG;
  const int e = ebase + le;
  const bool act = e < A.e1;
  float *su = smem + le * NP, *sF1 = smem + (E + le) * NP;     // [25] u, F1
  float *sg = smem + 2 * NP * E, *sm = sg + (GEO ? 0 : 5 * NP * E);
  const size_t ee = act ? e : A.e0, p0 = size_t(ebase) * NP, pend = size_t(A.e1) * NP, rec = ee * 8;
  RowGeo<E, GEO> G;
  RowMat<E, MAT> M;
  G.stage(A, p0, sg);
  M.stage(A, p0, sm);
  int g[NG], sl[NG];
#pragma unroll
  for (int k = 0; k < NG; ++k) {
    const size_t p = p0 + tid + k * T;
    g[k] = p < pend ? __ldg(A.ibool + p) : -1;
    sl[k] = p < pend ? __ldg(A.slot + p) : 0;
  }
  G.load(A, rec, sg, tid * NG);
  M.load(A, rec, sm, tid * NG);
  float hz[NG];
  ld_row5(t_rows[iz], hz);
  pdl_wait();
  pdl_release();
  {
    float t[NG];
#pragma unroll
    for (int k = 0; k < NG; ++k) t[k] = g[k] >= 0 ? ld_dep(A.u + g[k]) : 0.f;
#pragma unroll
    for (int k = 0; k < NG; ++k) smem[tid + k * T] = t[k];
  }
  if (GEO == 0 || MAT == 0) cp_async_wait();
  __syncthreads();
  float ur[NG], f0[NG];
#pragma unroll
  for (int l = 0; l < NG; ++l) ur[l] = su[iz * NG + l];
#pragma unroll
  for (int ix = 0; ix < NG; ++ix) {
    float2 d = make_float2(0.f, 0.f);
#pragma unroll
    for (int l = 0; l < NG; ++l) d = fma2(make_float2(c_hp[ix * NG + l], hz[l]), make_float2(ur[l], su[l * NG + ix]), d);
    const auto P = G.at(ix);
    const float k = SH ? M.mu(ix) : M.c0(ix);
    const float s0 = k * P.ddx(d.x, d.y);
    const float s1 = k * P.ddz(d.x, d.y);
    f0[ix] = P.f0(s0, s1);
    sF1[iz * NG + ix] = P.f1(s0, s1);
  }
  float wz[NG];
  ld_row5(t_rows[5 + iz], wz);
  const float wiz = ld_w(iz);
  const int bs = act ? __ldg(A.bc_slot + e) : -1;
  const int src = act ? __ldg(A.src_head + e) : -1;
  __syncthreads();
#pragma unroll
  for (int ix = 0; ix < NG; ++ix) {
    const int q = iz * NG + ix;
    float2 t = make_float2(0.f, 0.f);
#pragma unroll
    for (int l = 0; l < NG; ++l)
      t = fma2(make_float2(f0[l], sF1[l * NG + ix]), make_float2(c_hpw[l * NG + ix], wz[l]), t);
    float a = -(wiz * t.x + c_w[ix] * t.y);
    if (bs >= 0) {
      const size_t k = size_t(bs) * NP + q;
      const float wq = A.bc_w[k];
      if (wq != 0.f)
        a += -1.f * (wq * A.bc_j1[k]) * (SH ? A.bc_imp1[k] : A.bc_imp0[k]) * ld_dep(A.v + __ldg(A.ibool + ee * NP + q));
      if (!SH) a *= A.bc_keep[k];   // acoustic free surface (Dirichlet) zeroes the element term
    }
    if (src >= 0) {
      const int step = ld_dep(S.step);
      for (int s = src; s >= 0; s = S.src_next[s]) {
        const float f = step < S.nstep ? ld_dep(S.stf + size_t(step) * S.nsrc + s) : 0.f;
        a += f * S.src_arr[(size_t(s) * 2) * NP + q];
      }
    }
    su[q] = a;      // the displacement has been read by all
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NG; ++k)
    if (g[k] >= 0) A.r[sl[k]] = smem[tid + k * T];
}

// Resident blocks that the registers are held to.
template <int E, int EK, int GEO, int MAT>
__host__ __device__ constexpr int row_min_blocks() {
  constexpr int threads = (NG * E + 31) / 32 * 32;
  constexpr int regs = EK == 4 ? 112 : (EK == 0 ? 72 : 56);   // 64 / 48 and 88 / 72 measured equal or slower
  return 65536 / (threads * regs);
}

// The first blocks take receivers and the recording of a step, the next el.nblocks elastic
// elements (EK 0 P-SV, 1 SH, 4 poroelastic; 5 none), the others acoustic ones
// (EK 0 and 5).
template <int E, int EK, int GEO, int MAT>
__global__ void __launch_bounds__(NG * E, row_min_blocks<E, EK, GEO, MAT>()) k_stiffness_row(StiffArgs S) {
  __shared__ __align__(16) float smem[row_smem<E, EK, GEO, MAT>()];
  const int b = int(blockIdx.x) - S.rec_blocks - S.save_blocks;
  if (b < 0) {
    leading_block(S, smem);
  } else if (EK != 5 && b < S.el.nblocks) {
    if (EK == 1) scalar_rows<E, true, GEO, MAT>(S, S.el, S.el.e0 + b * E, smem);
    else pair_rows<E, EK == 4 ? 4 : 0, GEO, MAT>(S, S.el, S.el.e0 + b * E, smem);
  } else if (EK == 0 || EK == 5) {
    scalar_rows<E, false, GEO, MAT>(S, S.ac, S.ac.e0 + (b - S.el.nblocks) * E, smem);
  }
}

}  // namespace dev
}  // namespace sfg
