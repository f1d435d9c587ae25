// Batched-shot kernels of the 2D elastic time step (FP32).
//
// S independent shots (different sources, same mesh and model) advance in one
// launch per colour.  Fields are [point][component][shot], so the 32 lanes of
// a warp are 32 shots of one GLL point: the index, Jacobian and material
// loads of a point are warp-uniform (one transaction serves all shots) and
// the field loads are 128-byte coalesced.  A block is one element: 25 warps,
// one per GLL point, over a tile of up to 32 shots.  The Lagrange
// coefficients a warp needs are warp-uniform too and come from constant
// memory.
//
// Per shot the arithmetic is the single-shot element kernel's, operation for
// operation (same explicit FMAs in the contractions, everything else rounded
// separately), so a batched run gives the same bits as S separate runs.
// Reference: as kernels2d.cuh (compute_stiffness_interaction.tpp:140-247,
// stacey.tpp:50-80, compute_source_interaction.tpp:17-104, newmark.tpp:10-128,
// compute_seismogram.tpp:19-171).
#pragma once

#include "kernels2d.cuh"

namespace sfg {
namespace dev {

__constant__ float c_hp[NP];    // hp[i*5+j] = l'_j(xi_i)
__constant__ float c_hpw[NP];   // hp[l*5+i] * w[l]
__constant__ float c_w[NG];

// The same coefficients in global memory, for threads of a warp that need
// different rows: indexed constant-bank loads are served one address at a
// time (the indexed-constant unit was 77% busy in the acoustic row kernel,
// whose compiler reloads them at every use), a row here is two L1 hits and
// stays in registers.  Row i: l'_l(xi_i) over l; row 5 + i: hpw[l*5+i] over l;
// [10][i]: w.
__device__ __align__(16) float t_rows[11][8];

__device__ __forceinline__ void ld_row5(const float *row, float (&h)[NG]) {
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(h[0]), "=f"(h[1]), "=f"(h[2]), "=f"(h[3])
               : "l"(row));
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(h[4]) : "l"(row + 4));
}
__device__ __forceinline__ float ld_w(int i) {
  float x;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(x) : "l"(&t_rows[10][i]));
  return x;
}

struct BatchArgs {
  const int *__restrict__ ibool;
  const float *__restrict__ xix, *__restrict__ xiz, *__restrict__ gax, *__restrict__ gaz,
      *__restrict__ jac, *__restrict__ prop0, *__restrict__ prop1;
  const int *__restrict__ bc_slot;
  const float *__restrict__ bc_w, *__restrict__ bc_nx, *__restrict__ bc_nz, *__restrict__ bc_j1,
      *__restrict__ bc_imp0, *__restrict__ bc_imp1;
  const int *__restrict__ src_head, *__restrict__ src_next, *__restrict__ src_shot;
  const float *__restrict__ src_arr;   // [nsrc][2][25]
  const float *__restrict__ stf;       // [nstep][nsrc]
  int nsrc, nstep;
  const int *__restrict__ step;
  const float *__restrict__ u, *__restrict__ v;   // [nglob][NC][S]
  float *__restrict__ accum;
  float *__restrict__ r;               // owner-computes: [slot[element*25 + point]][NC][S]
  const int *__restrict__ slot;
  const float *__restrict__ erec;      // per-element records (RowClass)
  int e0;                              // first element of the colour
  int S;                               // shots
  int nspec_b;                         // elements (persistent kernel)
};

// grid: (elements of the colour, shot tiles of 32); block: 25 warps x 32 lanes.
// LOCAL: write the element's contribution to its own slot of A.r instead of
// adding it into the accumulator (then e0 = 0 and the grid covers all elements).
template <int NC, bool LOCAL>
__global__ void __launch_bounds__(NP * 32) k_stiffness_batched(BatchArgs A) {
  __shared__ float su[NC][NP][32];
  __shared__ float sF[NC][2][NP][32];
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int shot = blockIdx.y * 32 + lane;
  const bool act = shot < A.S;
  const int e = A.e0 + blockIdx.x;
  const size_t p = size_t(e) * NP + q;
  const int iz = q / NG, ix = q - iz * NG;
  const int g = __ldg(A.ibool + p);
  const float xix = __ldg(A.xix + p), xiz = __ldg(A.xiz + p), gax = __ldg(A.gax + p),
              gaz = __ldg(A.gaz + p), jac = __ldg(A.jac + p);
  const float c0 = __ldg(A.prop0 + p), mu = __ldg(A.prop1 + p);
  float uu[NC], acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const size_t k = (size_t(g) * NC + c) * A.S + shot;
    uu[c] = act ? A.u[k] : 0.f;
    acc[c] = (act && !LOCAL) ? A.accum[k] : 0.f;
    su[c][q][lane] = uu[c];
  }
  const int bs = __ldg(A.bc_slot + e);
  const int src = __ldg(A.src_head + e);
  __syncthreads();
  float dxi[NC], dga[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    dxi[c] = 0.f;
    dga[c] = 0.f;
#pragma unroll
    for (int l = 0; l < NG; ++l) {
      dxi[c] = fmaf(c_hp[ix * NG + l], su[c][iz * NG + l][lane], dxi[c]);
      dga[c] = fmaf(c_hp[iz * NG + l], su[c][l * NG + ix][lane], dga[c]);
    }
  }
  float Sx[NC], Sz[NC];
  if (NC == 2) {
    const float du00 = xix * dxi[0] + gax * dga[0], du01 = xiz * dxi[0] + gaz * dga[0];
    const float du10 = xix * dxi[NC - 1] + gax * dga[NC - 1];
    const float du11 = xiz * dxi[NC - 1] + gaz * dga[NC - 1];
    const float lam = c0 - 2.f * mu;
    const float sxx = c0 * du00 + lam * du11;
    const float szz = c0 * du11 + lam * du00;
    const float sxz = mu * (du01 + du10);
    Sx[0] = sxx; Sz[0] = sxz; Sx[NC - 1] = sxz; Sz[NC - 1] = szz;
  } else {
    Sx[0] = mu * (xix * dxi[0] + gax * dga[0]);
    Sz[0] = mu * (xiz * dxi[0] + gaz * dga[0]);
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    sF[c][0][q][lane] = jac * (Sx[c] * xix + Sz[c] * xiz);
    sF[c][1][q][lane] = jac * (Sx[c] * gax + Sz[c] * gaz);
  }
  __syncthreads();
  if (!act) return;
  float a[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    float t1 = 0.f, t2 = 0.f;
#pragma unroll
    for (int l = 0; l < NG; ++l) {
      t1 = fmaf(sF[c][0][iz * NG + l][lane], c_hpw[l * NG + ix], t1);
      t2 = fmaf(sF[c][1][l * NG + ix][lane], c_hpw[l * NG + iz], t2);
    }
    a[c] = -(c_w[iz] * t1 + c_w[ix] * t2);
  }
  if (bs >= 0) {
    const size_t k = size_t(bs) * NP + q;
    const float wq = A.bc_w[k];
    if (wq != 0.f) {
      const float nx = A.bc_nx[k], nz = A.bc_nz[k], j1 = A.bc_j1[k];
      if (NC == 2) {
        const float vx = A.v[(size_t(g) * NC) * A.S + shot];
        const float vz = A.v[(size_t(g) * NC + NC - 1) * A.S + shot];
        const float rvp = A.bc_imp0[k], rvs = A.bc_imp1[k];
        const float vn = vx * nx + vz * nz;
        const float fx = ((vn * nx / (j1 * j1)) * (rvp - rvs)) + vx * rvs;
        const float fz = ((vn * nz / (j1 * j1)) * (rvp - rvs)) + vz * rvs;
        a[0] += -1.f * fx * j1 * wq;
        a[NC - 1] += -1.f * fz * j1 * wq;
      } else {
        a[0] += -1.f * (wq * j1) * A.bc_imp1[k] * A.v[size_t(g) * A.S + shot];
      }
    }
  }
  if (src >= 0) {
    const int step = *A.step;
    for (int s = src; s >= 0; s = A.src_next[s]) {
      if (A.src_shot[s] != shot) continue;
      const float f = step < A.nstep ? A.stf[size_t(step) * A.nsrc + s] : 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) a[c] += f * A.src_arr[(size_t(s) * 2 + c) * NP + q];
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (LOCAL) A.r[(size_t(__ldg(A.slot + p)) * NC + c) * A.S + shot] = a[c];
    else A.accum[(size_t(g) * NC + c) * A.S + shot] = acc[c] + a[c];
  }
}

// Owner-computes update for [point][NC][S] fields: a thread takes V shots (as
// one vector; V divides S) of both components of a point, so that all its
// field loads are in flight together and the contribution range is read once;
// the contributions are summed in colour order (bitwise the colour passes'
// sum), then M^-1, corrector and optional predictor.  One component and one
// vector a thread, with three divisions for its index, reached 0.61 of the
// DRAM's cycles.
template <int V> struct ShotVec { float x[V]; };
template <int V>
__device__ __forceinline__ ShotVec<V> ld_shots(const float *p) {
  ShotVec<V> r;
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    r.x[0] = t.x; r.x[1] = t.y; r.x[2] = t.z; r.x[3] = t.w;
  } else if constexpr (V == 2) {
    const float2 t = *reinterpret_cast<const float2 *>(p);
    r.x[0] = t.x; r.x[1] = t.y;
  } else {
    r.x[0] = *p;
  }
  return r;
}
template <int V>
__device__ __forceinline__ void st_shots(float *p, const ShotVec<V> &r) {
  if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(r.x[0], r.x[1], r.x[2], r.x[3]);
  else if constexpr (V == 2) *reinterpret_cast<float2 *>(p) = make_float2(r.x[0], r.x[1]);
  else *p = r.x[0];
}

template <int NC, int V>
__global__ void __launch_bounds__(256) k_update_batched_gather(UpdateArgs A, int S) {
  const int SV = S / V, n = A.n / (NC * V);
  const int stride = gridDim.x * blockDim.x;
  bool bad = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int g = i / SV, s = (i - g * SV) * V;
    const size_t o = size_t(g) * NC * S + s;
    const int k0 = A.inv_start[g], k1 = A.inv_start[g + 1];
    ShotVec<V> u[NC], v[NC], acc[NC];
    float mi[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      u[c] = ld_shots<V>(A.u + o + size_t(c) * S);
      v[c] = ld_shots<V>(A.v + o + size_t(c) * S);
      mi[c] = A.minv[size_t(g) * NC + c];
#pragma unroll
      for (int w = 0; w < V; ++w) acc[c].x[w] = 0.f;
    }
    for (int k = k0; k < k1; ++k) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const ShotVec<V> t = ld_shots<V>(A.r + (size_t(k) * NC + c) * S + s);
#pragma unroll
        for (int w = 0; w < V; ++w) acc[c].x[w] = acc[c].x[w] + t.x[w];
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      ShotVec<V> a;
#pragma unroll
      for (int w = 0; w < V; ++w) {
        a.x[w] = __fmul_rn(acc[c].x[w], mi[c]);
        v[c].x[w] = newmark_correct(v[c].x[w], a.x[w], A.dt2);
        if (A.predict) newmark_predict(u[c].x[w], v[c].x[w], a.x[w], A.dt, A.dt2, A.dtsq2);
        bad |= !isfinite(u[c].x[w]);
      }
      if (A.predict) st_shots<V>(A.u + o + size_t(c) * S, u[c]);
      st_shots<V>(A.v + o + size_t(c) * S, v[c]);
      if (A.a_store) st_shots<V>(A.a_store + o + size_t(c) * S, a);
    }
  }
  if (bad) *A.flag = 1;
  if (A.advance && blockIdx.x == 0 && threadIdx.x == 0) *A.step += 1;
}

// ---------------------------------------------------------------------------
// Quad-shot form (S a multiple of 4): each thread carries 4 consecutive shots
// of one GLL point as a float4, so it has four times the field bytes in
// flight of the one-shot-per-lane kernel.  Block: one element, 25 points x T
// threads (T = shots in the tile / 4, at most 8); grid: (elements, shot tiles).
// Per shot the operations are those of k_stiffness_batched.
template <int NC, bool LOCAL>
__global__ void __launch_bounds__(NP * 8) k_stiffness_batched4(BatchArgs A, int T) {
  __shared__ float4 su[NC][NP][8];
  __shared__ float4 sF[NC][2][NP][8];
  const int q = threadIdx.x / T, j = threadIdx.x - q * T;
  const int shot0 = (blockIdx.y * T + j) * 4;
  const bool act = shot0 < A.S;
  const int e = A.e0 + blockIdx.x;
  const size_t p = size_t(e) * NP + q;
  const int iz = q / NG, ix = q - iz * NG;
  const int g = __ldg(A.ibool + p);
  const float xix = __ldg(A.xix + p), xiz = __ldg(A.xiz + p), gax = __ldg(A.gax + p),
              gaz = __ldg(A.gaz + p), jac = __ldg(A.jac + p);
  const float c0 = __ldg(A.prop0 + p), mu = __ldg(A.prop1 + p);
  float4 acc4[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const size_t k = (size_t(g) * NC + c) * A.S + shot0;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    su[c][q][j] = act ? *reinterpret_cast<const float4 *>(A.u + k) : z;
    acc4[c] = (act && !LOCAL) ? *reinterpret_cast<const float4 *>(A.accum + k) : z;
  }
  const int bs = __ldg(A.bc_slot + e);
  const int src = __ldg(A.src_head + e);
  __syncthreads();
  float a[NC][4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    float dxi[NC], dga[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      dxi[c] = 0.f;
      dga[c] = 0.f;
#pragma unroll
      for (int l = 0; l < NG; ++l) {
        dxi[c] = fmaf(c_hp[ix * NG + l], (&su[c][iz * NG + l][j].x)[w], dxi[c]);
        dga[c] = fmaf(c_hp[iz * NG + l], (&su[c][l * NG + ix][j].x)[w], dga[c]);
      }
    }
    float Sx[NC], Sz[NC];
    if (NC == 2) {
      const float du00 = xix * dxi[0] + gax * dga[0], du01 = xiz * dxi[0] + gaz * dga[0];
      const float du10 = xix * dxi[NC - 1] + gax * dga[NC - 1];
      const float du11 = xiz * dxi[NC - 1] + gaz * dga[NC - 1];
      const float lam = c0 - 2.f * mu;
      const float sxx = c0 * du00 + lam * du11;
      const float szz = c0 * du11 + lam * du00;
      const float sxz = mu * (du01 + du10);
      Sx[0] = sxx; Sz[0] = sxz; Sx[NC - 1] = sxz; Sz[NC - 1] = szz;
    } else {
      Sx[0] = mu * (xix * dxi[0] + gax * dga[0]);
      Sz[0] = mu * (xiz * dxi[0] + gaz * dga[0]);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      a[c][w] = jac * (Sx[c] * xix + Sz[c] * xiz);       // F0 for now
      (&sF[c][1][q][j].x)[w] = jac * (Sx[c] * gax + Sz[c] * gaz);
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) sF[c][0][q][j] = make_float4(a[c][0], a[c][1], a[c][2], a[c][3]);
  __syncthreads();
  if (!act) return;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      float t1 = 0.f, t2 = 0.f;
#pragma unroll
      for (int l = 0; l < NG; ++l) {
        t1 = fmaf((&sF[c][0][iz * NG + l][j].x)[w], c_hpw[l * NG + ix], t1);
        t2 = fmaf((&sF[c][1][l * NG + ix][j].x)[w], c_hpw[l * NG + iz], t2);
      }
      a[c][w] = -(c_w[iz] * t1 + c_w[ix] * t2);
    }
  }
  if (bs >= 0) {
    const size_t k = size_t(bs) * NP + q;
    const float wq = A.bc_w[k];
    if (wq != 0.f) {
      const float nx = A.bc_nx[k], nz = A.bc_nz[k], j1 = A.bc_j1[k];
      if (NC == 2) {
        const float4 vx4 = *reinterpret_cast<const float4 *>(A.v + (size_t(g) * NC) * A.S + shot0);
        const float4 vz4 = *reinterpret_cast<const float4 *>(A.v + (size_t(g) * NC + NC - 1) * A.S + shot0);
        const float rvp = A.bc_imp0[k], rvs = A.bc_imp1[k];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const float vx = (&vx4.x)[w], vz = (&vz4.x)[w];
          const float vn = vx * nx + vz * nz;
          const float fx = ((vn * nx / (j1 * j1)) * (rvp - rvs)) + vx * rvs;
          const float fz = ((vn * nz / (j1 * j1)) * (rvp - rvs)) + vz * rvs;
          a[0][w] += -1.f * fx * j1 * wq;
          a[NC - 1][w] += -1.f * fz * j1 * wq;
        }
      } else {
        const float4 v4 = *reinterpret_cast<const float4 *>(A.v + size_t(g) * A.S + shot0);
#pragma unroll
        for (int w = 0; w < 4; ++w) a[0][w] += -1.f * (wq * j1) * A.bc_imp1[k] * (&v4.x)[w];
      }
    }
  }
  if (src >= 0) {
    const int step = *A.step;
    for (int s = src; s >= 0; s = A.src_next[s]) {
      const int w = A.src_shot[s] - shot0;
      if (w < 0 || w > 3) continue;
      const float f = step < A.nstep ? A.stf[size_t(step) * A.nsrc + s] : 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float add = f * A.src_arr[(size_t(s) * 2 + c) * NP + q];
        // the one-shot kernel adds sources in chain order; so does this loop
        if (w == 0) a[c][0] += add;
        else if (w == 1) a[c][1] += add;
        else if (w == 2) a[c][2] += add;
        else a[c][3] += add;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (LOCAL) {
      *reinterpret_cast<float4 *>(A.r + (size_t(__ldg(A.slot + p)) * NC + c) * A.S + shot0) =
          make_float4(a[c][0], a[c][1], a[c][2], a[c][3]);
    } else {
      *reinterpret_cast<float4 *>(A.accum + (size_t(g) * NC + c) * A.S + shot0) =
          make_float4(acc4[c].x + a[c][0], acc4[c].y + a[c][1], acc4[c].z + a[c][2], acc4[c].w + a[c][3]);
    }
  }
}

// Thread form of the owner-computes batched element kernel: one thread per
// element and shot, the element's 25 points in registers.  The lanes of a
// warp are the shots of one element (of 32 / G elements when the shots fill
// only G < 32 lanes), so every field access is coalesced over shots and the
// contractions need neither shared memory nor barriers: the xi derivatives
// replace the displacement row by row, the gamma derivatives are formed
// column by column, F0 and F1 replace them, and the divergence contracts F0
// rows and F1 columns in place (two components paired in FFMA2, which rounds
// each lane as fmaf).  The block's index, slot, geometry and material words
// are staged once in shared memory and read as broadcasts.  GEO 1, MAT 1: as
// in the row kernel, words that are one value an element come from its record.
// The row form read every gamma column from shared memory once a row (63% of
// the L1's wavefronts, 122 instructions a point of 32 shots); this form
// executes about half.  Per shot the operations and their order are those of
// k_stiffness_batched (same bits).
template <int GEO, int MAT>
constexpr int bt_words() { return 2 + (GEO ? 0 : 5) + (MAT ? 0 : 2); }   // staged words a point

// One component pair (P-SV) or one component (SH) of a thread's shot.
template <int NC> struct BtV;
template <> struct BtV<2> { float2 v; };
template <> struct BtV<1> { float v; };
__device__ __forceinline__ void bt_fma(BtV<2> &a, float h, const BtV<2> &x) { a.v = fma2(f2(h), x.v, a.v); }
__device__ __forceinline__ void bt_fma(BtV<1> &a, float h, const BtV<1> &x) { a.v = fmaf(h, x.v, a.v); }
__device__ __forceinline__ void bt_zero(BtV<2> &a) { a.v = make_float2(0.f, 0.f); }
__device__ __forceinline__ void bt_zero(BtV<1> &a) { a.v = 0.f; }
template <int NC>
__device__ __forceinline__ float bt_get(const BtV<NC> &a, int c);
template <>
__device__ __forceinline__ float bt_get<2>(const BtV<2> &a, int c) { return c ? a.v.y : a.v.x; }
template <>
__device__ __forceinline__ float bt_get<1>(const BtV<1> &a, int) { return a.v; }

// out_i = sum_l coef(i, l) x_l over the five values of a line, in place; DIV:
// the divergence's weighted derivatives hpw[l*5+i], else hp[i*5+l].
template <int NC, bool DIV>
__device__ __forceinline__ void bt_line(BtV<NC> &x0, BtV<NC> &x1, BtV<NC> &x2, BtV<NC> &x3, BtV<NC> &x4) {
  const BtV<NC> x[NG] = {x0, x1, x2, x3, x4};
  BtV<NC> o[NG];
#pragma unroll
  for (int i = 0; i < NG; ++i) {
    bt_zero(o[i]);
#pragma unroll
    for (int l = 0; l < NG; ++l) bt_fma(o[i], DIV ? c_hpw[l * NG + i] : c_hp[i * NG + l], x[l]);
  }
  x0 = o[0]; x1 = o[1]; x2 = o[2]; x3 = o[3]; x4 = o[4];
}

constexpr int BT_THREADS = 128;

// G lanes per element (a power of two, at least the shots of the tile or 32).
template <int NC, int GEO, int MAT>
__global__ void __launch_bounds__(BT_THREADS, 4) k_stiffness_batched_t(BatchArgs A, int G) {
  extern __shared__ __align__(16) float btsm[];
  const int NE = BT_THREADS / G;                  // elements of the block
  const int NPB = NE * NP;
  const int e0 = blockIdx.x * NE;
  {
    const size_t p0 = size_t(e0) * NP;
    const int n = min(NE, A.nspec_b - e0) * NP;
    int *si = reinterpret_cast<int *>(btsm);
    for (int i = threadIdx.x; i < n; i += BT_THREADS) {
      si[i] = __ldg(A.ibool + p0 + i);
      si[NPB + i] = __ldg(A.slot + p0 + i);
      int w = 2;
      if (GEO == 0) {
        btsm[w++ * NPB + i] = __ldg(A.xix + p0 + i);
        btsm[w++ * NPB + i] = __ldg(A.xiz + p0 + i);
        btsm[w++ * NPB + i] = __ldg(A.gax + p0 + i);
        btsm[w++ * NPB + i] = __ldg(A.gaz + p0 + i);
        btsm[w++ * NPB + i] = __ldg(A.jac + p0 + i);
      }
      if (MAT == 0) {
        btsm[w++ * NPB + i] = __ldg(A.prop0 + p0 + i);
        btsm[w++ * NPB + i] = __ldg(A.prop1 + p0 + i);
      }
    }
  }
  const int le = threadIdx.x / G, shot = blockIdx.y * 32 + (threadIdx.x - le * G);
  const int e = e0 + le;
  const bool act = e < A.nspec_b && shot < A.S;
  float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 m2 = make_float2(0.f, 0.f);
  if (GEO == 1 && act) g4 = __ldg(reinterpret_cast<const float4 *>(A.erec + size_t(e) * 8));
  if (MAT == 1 && act) m2 = __ldg(reinterpret_cast<const float2 *>(A.erec + size_t(e) * 8 + 4));
  __syncthreads();
  if (!act) return;
  const int *sg = reinterpret_cast<const int *>(btsm) + le * NP, *ss = sg + NPB;
  const float *sw = btsm + 2 * NPB + le * NP;
  BtV<NC> U[NP], D[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const float *u = A.u + size_t(sg[q]) * NC * A.S + shot;
    if constexpr (NC == 2) U[q].v = make_float2(u[0], u[A.S]);
    else U[q].v = u[0];
  }
#pragma unroll
  for (int ix = 0; ix < NG; ++ix) {
#pragma unroll
    for (int iz = 0; iz < NG; ++iz) D[iz * NG + ix] = U[iz * NG + ix];
    bt_line<NC, false>(D[ix], D[5 + ix], D[10 + ix], D[15 + ix], D[20 + ix]);
  }
#pragma unroll
  for (int iz = 0; iz < NG; ++iz) bt_line<NC, false>(U[5 * iz], U[5 * iz + 1], U[5 * iz + 2], U[5 * iz + 3], U[5 * iz + 4]);
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    float xix, xiz = 0.f, gax = 0.f, gaz, jac;
    if (GEO == 1) { xix = g4.x; gaz = g4.y; jac = g4.z; }
    else { xix = sw[q]; xiz = sw[NPB + q]; gax = sw[2 * NPB + q]; gaz = sw[3 * NPB + q]; jac = sw[4 * NPB + q]; }
    float c0, mu;
    if (MAT == 1) { c0 = m2.x; mu = m2.y; }
    else { c0 = sw[(GEO ? 0 : 5) * NPB + q]; mu = sw[(GEO ? 1 : 6) * NPB + q]; }
    // x + 0 and x * 0 of the rectangle's zero words change no bit
    auto ddx = [&](float dxi, float dga) { return GEO ? xix * dxi : xix * dxi + gax * dga; };
    auto ddz = [&](float dxi, float dga) { return GEO ? gaz * dga : xiz * dxi + gaz * dga; };
    auto f0 = [&](float sx, float sz) { return GEO ? jac * (sx * xix) : jac * (sx * xix + sz * xiz); };
    auto f1 = [&](float sx, float sz) { return GEO ? jac * (sz * gaz) : jac * (sx * gax + sz * gaz); };
    if constexpr (NC == 2) {
      const float2 dx = U[q].v, dg = D[q].v;
      const float du00 = ddx(dx.x, dg.x), du01 = ddz(dx.x, dg.x), du10 = ddx(dx.y, dg.y), du11 = ddz(dx.y, dg.y);
      const float lam = c0 - 2.f * mu;
      const float sxx = c0 * du00 + lam * du11;
      const float szz = c0 * du11 + lam * du00;
      const float sxz = mu * (du01 + du10);
      U[q].v = make_float2(f0(sxx, sxz), f0(sxz, szz));
      D[q].v = make_float2(f1(sxx, sxz), f1(sxz, szz));
    } else {
      const float sx = mu * ddx(U[q].v, D[q].v), sz = mu * ddz(U[q].v, D[q].v);
      U[q].v = f0(sx, sz);
      D[q].v = f1(sx, sz);
    }
  }
#pragma unroll
  for (int iz = 0; iz < NG; ++iz) bt_line<NC, true>(U[5 * iz], U[5 * iz + 1], U[5 * iz + 2], U[5 * iz + 3], U[5 * iz + 4]);
#pragma unroll
  for (int ix = 0; ix < NG; ++ix) bt_line<NC, true>(D[ix], D[5 + ix], D[10 + ix], D[15 + ix], D[20 + ix]);
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int iz = q / NG, ix = q - iz * NG;
    float *r = A.r + size_t(ss[q]) * NC * A.S + shot;
#pragma unroll
    for (int c = 0; c < NC; ++c)
      r[size_t(c) * A.S] = -(c_w[iz] * bt_get<NC>(U[q], c) + c_w[ix] * bt_get<NC>(D[q], c));
  }
  const int bs = __ldg(A.bc_slot + e), src = __ldg(A.src_head + e);
  if (bs < 0 && src < 0) return;
  // boundary and source elements: the Stacey traction, then the sources, onto
  // the thread's own results
  const int step = *A.step;
  for (int q = 0; q < NP; ++q) {
    float *r = A.r + size_t(ss[q]) * NC * A.S + shot;
    const size_t g = size_t(sg[q]) * NC;
    float a[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) a[c] = r[size_t(c) * A.S];
    if (bs >= 0) {
      const size_t k = size_t(bs) * NP + q;
      const float wq = A.bc_w[k];
      if (wq != 0.f) {
        const float nx = A.bc_nx[k], nz = A.bc_nz[k], j1 = A.bc_j1[k];
        if (NC == 2) {
          const float vx = A.v[g * A.S + shot], vz = A.v[(g + NC - 1) * A.S + shot];
          const float rvp = A.bc_imp0[k], rvs = A.bc_imp1[k];
          const float vn = vx * nx + vz * nz;
          const float fx = ((vn * nx / (j1 * j1)) * (rvp - rvs)) + vx * rvs;
          const float fz = ((vn * nz / (j1 * j1)) * (rvp - rvs)) + vz * rvs;
          a[0] += -1.f * fx * j1 * wq;
          a[NC - 1] += -1.f * fz * j1 * wq;
        } else {
          a[0] += -1.f * (wq * j1) * A.bc_imp1[k] * A.v[g * A.S + shot];
        }
      }
    }
    for (int s = src; s >= 0; s = A.src_next[s]) {
      if (A.src_shot[s] != shot) continue;
      const float f = step < A.nstep ? A.stf[size_t(step) * A.nsrc + s] : 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) a[c] += f * A.src_arr[(size_t(s) * 2 + c) * NP + q];
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) r[size_t(c) * A.S] = a[c];
  }
}

// Quad-shot updates (S a multiple of 4): flat float4 index over [nglob][NC][S].
__global__ void __launch_bounds__(256) k_update_batched4(UpdateArgs A, int S) {
  const int n4 = A.n >> 2;
  const int stride = gridDim.x * blockDim.x;
  bool bad = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
    const float mi = A.minv[(4 * i) / S];
    float4 ac = reinterpret_cast<const float4 *>(A.accum)[i];
    float4 uu = reinterpret_cast<float4 *>(A.u)[i];
    float4 vv = reinterpret_cast<float4 *>(A.v)[i];
    float *pa = &ac.x, *pu = &uu.x, *pv = &vv.x;
    float a[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      a[w] = __fmul_rn(pa[w], mi);
      pv[w] = newmark_correct(pv[w], a[w], A.dt2);
      if (A.predict) newmark_predict(pu[w], pv[w], a[w], A.dt, A.dt2, A.dtsq2);
      bad |= !isfinite(pu[w]);
    }
    if (A.predict) reinterpret_cast<float4 *>(A.u)[i] = uu;
    reinterpret_cast<float4 *>(A.v)[i] = vv;
    reinterpret_cast<float4 *>(A.accum)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (A.a_store) reinterpret_cast<float4 *>(A.a_store)[i] = make_float4(a[0], a[1], a[2], a[3]);
  }
  if (bad) *A.flag = 1;
  if (A.advance && blockIdx.x == 0 && threadIdx.x == 0) *A.step += 1;
}

// a = accum * M^-1 (M^-1 shared by the shots); corrector; optional fused
// predictor; accumulator clear.  Flat index i over [nglob][NC][S].
__global__ void __launch_bounds__(256) k_update_batched(UpdateArgs A, int S) {
  const int stride = gridDim.x * blockDim.x;
  bool bad = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += stride) {
    const float a = __fmul_rn(A.accum[i], A.minv[i / S]);
    float vv = newmark_correct(A.v[i], a, A.dt2);
    float uu = A.u[i];
    if (A.predict) newmark_predict(uu, vv, a, A.dt, A.dt2, A.dtsq2);
    A.u[i] = uu;
    A.v[i] = vv;
    A.accum[i] = 0.f;
    if (A.a_store) A.a_store[i] = a;
    bad |= !isfinite(uu);
  }
  if (bad) *A.flag = 1;
  if (A.advance && blockIdx.x == 0 && threadIdx.x == 0) *A.step += 1;
}

// One block per receiver, lanes over shots (tiles of 32): displacement,
// velocity (corrected) or acceleration interpolated with the receiver's
// Lagrange weights.  seis is [S][nsig][ntypes][nrec][2].
__global__ void __launch_bounds__(32) k_receivers_batched(RecArgs A, int S) {
  const int step = *A.step;
  if (step % A.nsb != 0) return;
  const int isig = step / A.nsb;
  if (isig >= A.nsig) return;
  const int r = A.rec_list[blockIdx.x];
  const int ce = A.rec_elem[r];
  const int NC = A.ncomp;
  for (int s0 = 0; s0 < S; s0 += 32) {
    const int shot = s0 + threadIdx.x;
    if (shot >= S) continue;
    for (int t = 0; t < A.ntypes; ++t) {
      float tr[2] = {0.f, 0.f};
      for (int c = 0; c < NC; ++c) {
        // the 25 weighted values, summed in the order of the single-shot
        // kernel's xor butterfly (lane i + lane i^o), so traces match it bitwise
        float x[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) x[q] = 0.f;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const int g = A.ibool[size_t(ce) * NP + q];
          const size_t k = (size_t(g) * NC + c) * S + shot;
          float sum = 0.f;
          if (A.types[t] == 0) {                 // displacement: no sum
          } else if (A.cpl.inv_start) {
            for (int j = A.cpl.inv_start[g]; j < A.cpl.inv_start[g + 1]; ++j)
              sum = sum + A.cpl.r[(size_t(j) * NC + c) * S + shot];
          } else {
            sum = A.accum[k];
          }
          const float acc = __fmul_rn(sum, A.minv[size_t(g) * NC + c]);
          float val;
          switch (A.types[t]) {
            case 0: val = A.u[k]; break;
            case 1: val = newmark_correct(A.v[k], acc, A.dt2); break;
            default: val = acc; break;
          }
          x[q] = A.rec_h[size_t(r) * NP + q] * val;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < o; ++i) x[i] = x[i] + x[i + o];
        tr[c] = x[0];
      }
      float *dst = A.seis + (((size_t(shot) * A.nsig + isig) * A.ntypes + t) * A.nrec_total + r) * 2;
      dst[0] = tr[0];
      dst[1] = NC > 1 ? tr[1] : 0.f;
    }
  }
}

}  // namespace dev
}  // namespace sfg
