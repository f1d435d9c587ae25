// sm_100a kernels of the 3D elastic spectral-element time step (FP32).
//
// One step is two launches: [layer kernel] -> [finish kernel] (-> [late
// receivers] where velocity or acceleration is recorded).
// * Layer kernel (k_layer3d): a block owns a tile of 4 x 2 elements in (x, y)
//   and marches L element layers up in z, one thread per (x, y) column of an
//   element's five points.  Per layer the tile's displacement planes arrive by
//   cp.async while the layer below is computed; the 5-term Lagrange-derivative
//   contractions (include/algorithms/gradient.hpp:103-156), the isotropic
//   stress (include/medium/dim3/elastic/isotropic/stress.hpp:46-99), F_k =
//   |J| sigma . grad(xi_k) (core/specfem/point/stress.hpp:217-240) and the
//   divergence with its weight products (include/algorithms/divergence.hpp:
//   90-137) run on whole columns (components in pairs, FFMA2); the epilogue
//   applies the absorbing-face traction -C v and point sources.  The tile's
//   contributions are then summed per unique point in shared memory (x
//   neighbours, then y, then the layer below) and every point that no other
//   tile touches is finished at once: a = sum * M^-1, Newmark corrector, next
//   predictor (newmark.tpp:10-128).  Only the tile's shared points pass through
//   memory: 23 of an inner tile's 128 columns, and of the others the plane
//   between two marches, 1 - (105/128) (1 - 1/(4 L)) of all points for marches
//   of L layers (38% for one, 28% for two, 23% for four).
// * Finish kernel (k_finish3d): sums the tiles' parts of the shared points in
//   tile order (across a z boundary of two blocks of one tile: lower plus
//   upper first), finishes them, and takes the receivers that read only the
//   displacement.
// The order of every sum depends on the tiles alone, so the number of layers
// a block marches changes no bit.
//
// The old displacement and velocity are read and the new ones written to a
// second pair of buffers, so that neighbouring tiles, and the receivers of
// the finish kernel, read the step's own fields whatever the order of blocks.
//
// Why this split: a kernel per element with its contributions in memory moves
// 12 B a contribution out and back (3.9 contributions' worth a point counting
// index arrays, 185 B a point and step); marching tiles move 60 B of fields and
// M^-1 and 15.5 B of material a point, and at the shared points the tiles' parts
// out and back and the fields once more.  The metric terms are folded (|J| into grad xi, 1/|J| into the moduli), which drops the
// Jacobian word and nine products a point; a mesh of boxes along the axes
// (GEO 1, decided for the whole mesh at set-up) keeps three metric words an
// element.
//
// Measured, 48x48x32 boxes with moduli per point (4.8 M points): step 370 ->
// 291 us; layer kernel 232 us and finish kernel 64 us one after another (2
// layers a block; they overlap in a step).  Deformed, general metric: step 406
// us, layer kernel 349 us.
// 13x11x9: 17.9 -> 17.3 us.  The layer kernel is bound by shared memory (its
// wavefronts take 67% of the L1's cycles) and by the barriers of a layer at
// two blocks a SM; three blocks at 80 registers spill and take 250 us.  The
// finish kernel waits for scattered 12-byte accesses at 45% of the DRAM.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sfg3 {
namespace dev {

constexpr int NG = 5;
constexpr int NQ = 125;
constexpr int TX = 4, TY = 2;                        // elements of a tile
constexpr int CX = 4 * TX + 1, CY = 4 * TY + 1;      // point columns of a tile
constexpr int NCOL = CX * CY;
constexpr int NEDGE = 2 * CX + 2 * (CY - 2);         // columns on the tile's rim
constexpr int TILE_THREADS = TX * TY * NG * NG;
constexpr int CS = 20;                               // floats a column in shared memory (15 used; 20: no bank conflicts)

__constant__ float c3_hp[NG * NG];    // hp[i*5+j] = l'_j(xi_i)
__constant__ float c3_hpw[NG * NG];   // hp[l*5+i] * w[l]
__constant__ float c3_w[NG];
// The same, for threads of a warp that need different rows (indexed constant
// loads serialise).  Row i: l'_l(xi_i) over l; row 5 + i: hpw[l*5+i] over l.
__device__ __align__(16) float t3_rows[10][8];

__device__ __forceinline__ void ld_row5(const float *row, float (&h)[NG]) {
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(h[0]), "=f"(h[1]), "=f"(h[2]), "=f"(h[3])
               : "l"(row));
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(h[4]) : "l"(row + 4));
}

// A column's 15 values: (x, y) of plane iz at 2 iz, z of plane iz at 10 + iz.
__host__ __device__ constexpr int cpos(int iz, int c) { return c < 2 ? 2 * iz + c : 10 + iz; }

struct Step3Args {
  // mesh
  int nex, ney, nez, nbx, nby, L, nchunk;
  int NX, NY, NZ;                     // lattice points
  size_t nloc;
  const float *__restrict__ g9;       // GEO 0: [9][nspec*125] |J| d xi_k / d x_j, k-major
  const float4 *__restrict__ ediag;   // GEO 1: [nspec] |J| d xi_k / d x_k
  const float *__restrict__ c0, *__restrict__ mu;   // (lambda + 2 mu) / |J|, mu / |J| [nspec*125]
  const float *__restrict__ minv;     // [nglob][3]
  const int *__restrict__ bc_slot;    // [nspec]: absorbing data slot or -1
  const float *__restrict__ bc_c;     // [slot][6][125]: C xx yy zz xy xz yz
  const int *__restrict__ src_head, *__restrict__ src_next;
  const float *__restrict__ src_arr;  // [nsrc][3][125]
  const float *stf;                   // [nstep][nsrc]
  int nsrc, nstep;
  // fields: old (the step's predicted state) and new, [nglob][3]
  const float *uo, *vo;
  float *un, *vn, *a_store;
  // the tiles' parts of shared points: rim columns of every plane, all
  // columns of the planes between two blocks of a tile
  float *rim;                         // [tile][NZ][NEDGE][3]
  float *lower, *upper;               // [tile][nchunk][NCOL][3]
  float dt, dt2, dtsq2;
  int predict;
  // step[0]: the step counter, advanced by the finish kernel; step[1]: the
  // step being taken, set by the layer kernel and read by the receivers
  int *flag, *step;
  int advance;
  // receivers
  const int *__restrict__ rec_elem;
  const float *__restrict__ rec_h;    // [nrec][125]
  const int *__restrict__ types;      // per type: 0 displacement, 1 velocity, 2 acceleration
  int ntypes, nrec, nsig, rec_blocks;
  float *seis;                        // [nsig][ntypes][nrec][3]
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// data that the step's kernels write: never through the read-only cache
__device__ __forceinline__ float ld_dep(const float *p) {
  float x;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(x) : "l"(p) : "memory");
  return x;
}
// the same past the L1 (before the wait: complete, but written by any SM)
__device__ __forceinline__ float ld_l2(const float *p) {
  float x;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(x) : "l"(p) : "memory");
  return x;
}
__device__ __forceinline__ int ld_dep(const int *p) {
  int x;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
  return x;
}
__device__ __forceinline__ void cp4(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

struct Col { float2 p[8]; };          // 15 values and a pad

__device__ __forceinline__ Col ld_col(const float *s) {
  Col c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 t = reinterpret_cast<const float4 *>(s)[i];
    c.p[2 * i] = make_float2(t.x, t.y);
    c.p[2 * i + 1] = make_float2(t.z, t.w);
  }
  return c;
}
__device__ __forceinline__ void st_col(float *s, const Col &c) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    reinterpret_cast<float4 *>(s)[i] = make_float4(c.p[2 * i].x, c.p[2 * i].y, c.p[2 * i + 1].x, c.p[2 * i + 1].y);
}
__device__ __forceinline__ float cget(const Col &c, int i) { return i & 1 ? c.p[i >> 1].y : c.p[i >> 1].x; }
__device__ __forceinline__ void cset(Col &c, int i, float v) {
  if (i & 1) c.p[i >> 1].y = v;
  else c.p[i >> 1].x = v;
}
__device__ __forceinline__ void col_fma(Col &acc, float h, const Col &x) {
#pragma unroll
  for (int i = 0; i < 8; ++i) acc.p[i] = __ffma2_rn(f2(h), x.p[i], acc.p[i]);
}
__device__ __forceinline__ void col_add(Col &acc, const Col &x) {
#pragma unroll
  for (int i = 0; i < 8; ++i) { acc.p[i].x = acc.p[i].x + x.p[i].x; acc.p[i].y = acc.p[i].y + x.p[i].y; }
}
__device__ __forceinline__ Col col_zero() {
  Col c;
#pragma unroll
  for (int i = 0; i < 8; ++i) c.p[i] = make_float2(0.f, 0.f);
  return c;
}
// out plane iz = sum_l coef(iz, l) in plane l.  Warp-uniform coefficients are
// operands straight from the constant bank; paired they would first have to
// be moved to register pairs (layer kernel 242 -> 228 us at 48x48x32).
template <bool DIV>
__device__ __forceinline__ Col col_z(const Col &x) {
  Col o = col_zero();
#pragma unroll
  for (int iz = 0; iz < NG; ++iz) {
    float2 t = make_float2(0.f, 0.f);
    float z = 0.f;
#pragma unroll
    for (int l = 0; l < NG; ++l) {
      const float h = DIV ? c3_hpw[l * NG + iz] : c3_hp[iz * NG + l];
      t = make_float2(fmaf(h, x.p[l].x, t.x), fmaf(h, x.p[l].y, t.y));
      z = fmaf(h, cget(x, 10 + l), z);
    }
    o.p[iz] = t;
    cset(o, 10 + iz, z);
  }
  return o;
}

__device__ __forceinline__ float dot3(float a0, float b0, float a1, float b1, float a2, float b2) {
  return fmaf(a2, b2, fmaf(a1, b1, a0 * b0));
}

// Isotropic stress, moduli divided by |J| and derivatives multiplied by it.
__device__ __forceinline__ void stress3(const float du[3][3], float c0, float mu, float sig[3][3]) {
  const float lam = c0 - 2.f * mu;
  sig[0][0] = fmaf(c0, du[0][0], lam * (du[1][1] + du[2][2]));
  sig[1][1] = fmaf(c0, du[1][1], lam * (du[0][0] + du[2][2]));
  sig[2][2] = fmaf(c0, du[2][2], lam * (du[0][0] + du[1][1]));
  sig[0][1] = sig[1][0] = mu * (du[0][1] + du[1][0]);
  sig[0][2] = sig[2][0] = mu * (du[0][2] + du[2][0]);
  sig[1][2] = sig[2][1] = mu * (du[1][2] + du[2][1]);
}

__device__ __forceinline__ void nm_predict(float &u, float &v, float a, float dt, float dt2, float dtsq2) {
  u = __fadd_rn(u, __fadd_rn(__fmul_rn(dt, v), __fmul_rn(dtsq2, a)));
  v = __fadd_rn(v, __fmul_rn(dt2, a));
}

// a = sum * M^-1, corrector, next predictor of one component.
__device__ __forceinline__ bool finish_value(const Step3Args &A, size_t i, float sum, float u, float v, float mi) {
  const float a = __fmul_rn(sum, mi);
  float vv = __fadd_rn(v, __fmul_rn(A.dt2, a));
  if (A.predict) nm_predict(u, vv, a, A.dt, A.dt2, A.dtsq2);
  A.un[i] = u;
  A.vn[i] = vv;
  if (A.a_store) A.a_store[i] = a;
  return !isfinite(u);
}

__device__ __forceinline__ int rim_index(int tx, int ty) {
  if (ty == 0) return tx;
  if (ty == CY - 1) return CX + tx;
  return 2 * CX + 2 * (ty - 1) + (tx ? 1 : 0);
}

// Shared memory of k_layer3d, floats: U planes of two layers, F of the
// element columns (two directions), v and M^-1 of four planes
// ([value][column]: consecutive threads on consecutive banks).
constexpr int L3_U = NCOL * CS, L3_F = TILE_THREADS * CS, L3_V = 24 * NCOL;
constexpr int L3_SMEM = (2 * L3_U + 2 * L3_F + L3_V) * int(sizeof(float));

template <int GEO>
__global__ void __launch_bounds__(TILE_THREADS, 2) k_layer3d(const __grid_constant__ Step3Args A) {
  extern __shared__ __align__(16) float sm3[];
  float *sU = sm3, *sF0 = sm3 + 2 * L3_U, *sF1 = sF0 + L3_F, *sV = sF1 + L3_F;
  const int tid = threadIdx.x;
  const int tile = blockIdx.x, bx = tile % A.nbx, by = tile / A.nbx, chunk = blockIdx.y;
  const int z0 = chunk * A.L, z1 = min(z0 + A.L, A.nez);
  // this thread's element column
  const int le = tid / (NG * NG), cq = tid - le * (NG * NG);
  const int iy = cq / NG, ix = cq - iy * NG;
  const int lx = le % TX, ly = le / TX;
  const int nax = min(TX, A.nex - bx * TX), nay = min(TY, A.ney - by * TY);
  const bool act = lx < nax && ly < nay;
  // this thread's point column of the tile
  const int ty = tid / CX, tx = tid - ty * CX;
  const bool col = tid < NCOL && tx <= 4 * nax && ty <= 4 * nay;
  const size_t plane = size_t(A.NX) * A.NY * 3;
  const size_t gcol = (size_t(by * 4 * TY + ty) * A.NX + bx * 4 * TX + tx) * 3;
  const bool rim = (tx == 0 && bx > 0) || (tx == CX - 1 && bx < A.nbx - 1) || (ty == 0 && by > 0) ||
                   (ty == CY - 1 && by < A.nby - 1);
  // what no kernel of the step writes, requested before the wait: the
  // coefficient rows of this thread, and the first layer's moduli and flags
  float hx[NG], hy[NG], kx[NG], ky[NG];
  ld_row5(t3_rows[ix], hx);
  ld_row5(t3_rows[iy], hy);
  ld_row5(t3_rows[5 + ix], kx);
  ld_row5(t3_rows[5 + iy], ky);
  const float wx = c3_w[ix], wy = c3_w[iy], wyx = wy * wx;
  float c0[NG], mu[NG];
  float4 dg = make_float4(0.f, 0.f, 0.f, 0.f);
  int bs = -1, src = -1;
  auto element = [&](int ez) { return (ez * A.ney + by * TY + ly) * A.nex + bx * TX + lx; };
  auto fetch_words = [&](int ez) {
    if (!act) return;
    const size_t e = size_t(element(ez)), pe = e * NQ + cq;
#pragma unroll
    for (int iz = 0; iz < NG; ++iz) { c0[iz] = __ldg(A.c0 + pe + iz * 25); mu[iz] = __ldg(A.mu + pe + iz * 25); }
    if (GEO == 1) dg = __ldg(A.ediag + e);
  };
#pragma unroll
  for (int iz = 0; iz < NG; ++iz) c0[iz] = mu[iz] = 0.f;
  fetch_words(z0);
  if (act) { bs = __ldg(A.bc_slot + element(z0)); src = __ldg(A.src_head + element(z0)); }
  pdl_wait();
  pdl_release();
  // planes 1..4 (and plane 0 of the first layer) of layer ez into U buffer b
  auto fetch_u = [&](int ez, int b, bool first) {
    if (!col) return;
    const float *src = A.uo + gcol + size_t(4 * ez) * plane;
    float *dst = sU + b * L3_U + tid * CS;
#pragma unroll
    for (int iz = 0; iz < NG; ++iz) {
      if (iz == 0 && !first) continue;
#pragma unroll
      for (int c = 0; c < 3; ++c) cp4(dst + cpos(iz, c), src + iz * plane + c);
    }
  };
  auto fetch_v = [&](int ez) {
    if (!col || rim) return;
    const size_t g = gcol + size_t(4 * ez) * plane;
    float *dst = sV + tid;
#pragma unroll
    for (int iz = 0; iz < 4; ++iz)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        cp4(dst + (iz * 3 + c) * NCOL, A.vo + g + iz * plane + c);
        cp4(dst + (12 + iz * 3 + c) * NCOL, A.minv + g + iz * plane + c);
      }
  };
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) A.step[1] = ld_dep(A.step);
  float carry[3] = {0.f, 0.f, 0.f};
  bool bad = false;
  fetch_u(z0, 0, true);
  cp_commit();
  for (int ez = z0; ez < z1; ++ez) {
    const int b = (ez - z0) & 1;
    float *U = sU + b * L3_U;
    const size_t pe = size_t(act ? element(ez) : 0) * NQ + cq;
    cp_wait<0>();
    __syncthreads();
    // the next layer's displacement, and this layer's v and M^-1
    fetch_v(ez);
    cp_commit();
    if (ez + 1 < z1) {
      fetch_u(ez + 1, b ^ 1, false);
      if (col) {   // its plane 0 is this layer's plane 4
        float *n = sU + (b ^ 1) * L3_U + tid * CS;
        const float *o = U + tid * CS;
#pragma unroll
        for (int c = 0; c < 3; ++c) n[cpos(0, c)] = o[cpos(4, c)];
      }
    }
    cp_commit();
    if (GEO == 0 && act && ez + 1 < z1) {
      // the next layer's metric terms into the L2: 9 x 125 floats an element
      const float *n = A.g9 + size_t(element(ez + 1)) * NQ;
      for (int i = cq; i < 9 * 16; i += 25)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(n + size_t(i >> 4) * A.nloc + min((i & 15) * 8, NQ - 1)));
    }
    Col dx = col_zero(), dy = col_zero(), dz;
    {
      const float *row = U + ((ly * 4 + iy) * CX + lx * 4) * CS;
#pragma unroll
      for (int l = 0; l < NG; ++l) col_fma(dx, hx[l], ld_col(row + l * CS));
      const float *clm = U + (ly * 4 * CX + lx * 4 + ix) * CS;
#pragma unroll
      for (int l = 0; l < NG; ++l) col_fma(dy, hy[l], ld_col(clm + l * CX * CS));
      dz = col_z<false>(ld_col(row + ix * CS));
    }
    // per plane: derivatives, stress, F in place of the derivatives
#pragma unroll
    for (int iz = 0; iz < NG; ++iz) {
      float du[3][3], sig[3][3];
      if (GEO == 1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          du[c][0] = dg.x * cget(dx, cpos(iz, c));
          du[c][1] = dg.y * cget(dy, cpos(iz, c));
          du[c][2] = dg.z * cget(dz, cpos(iz, c));
        }
        stress3(du, c0[iz], mu[iz], sig);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          cset(dx, cpos(iz, c), dg.x * sig[c][0]);
          cset(dy, cpos(iz, c), dg.y * sig[c][1]);
          cset(dz, cpos(iz, c), dg.z * sig[c][2]);
        }
      } else {
        float gi[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) gi[k] = __ldg(A.g9 + size_t(k) * A.nloc + pe + iz * 25);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            du[c][j] = dot3(cget(dx, cpos(iz, c)), gi[j], cget(dy, cpos(iz, c)), gi[3 + j], cget(dz, cpos(iz, c)), gi[6 + j]);
        stress3(du, c0[iz], mu[iz], sig);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          cset(dx, cpos(iz, c), dot3(sig[c][0], gi[0], sig[c][1], gi[1], sig[c][2], gi[2]));
          cset(dy, cpos(iz, c), dot3(sig[c][0], gi[3], sig[c][1], gi[4], sig[c][2], gi[5]));
          cset(dz, cpos(iz, c), dot3(sig[c][0], gi[6], sig[c][1], gi[7], sig[c][2], gi[8]));
        }
      }
    }
    st_col(sF0 + tid * CS, dx);
    st_col(sF1 + tid * CS, dy);
    if (ez + 1 < z1) fetch_words(ez + 1);      // for the next layer
    const Col t3 = col_z<true>(dz);
    __syncthreads();
    Col a;
    {
      Col t1 = col_zero(), t2 = col_zero();
      const float *row = sF0 + (le * 25 + iy * NG) * CS, *clm = sF1 + (le * 25 + ix) * CS;
#pragma unroll
      for (int l = 0; l < NG; ++l) col_fma(t1, kx[l], ld_col(row + l * CS));
#pragma unroll
      for (int l = 0; l < NG; ++l) col_fma(t2, ky[l], ld_col(clm + l * NG * CS));
      a = col_zero();
#pragma unroll
      for (int iz = 0; iz < NG; ++iz) {
        const float wzy = c3_w[iz] * wy, wzx = c3_w[iz] * wx;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int i = cpos(iz, c);
          cset(a, i, -dot3(wzy, cget(t1, i), wzx, cget(t2, i), wyx, cget(t3, i)));
        }
      }
    }
    if (bs >= 0) {
#pragma unroll
      for (int iz = 0; iz < NG; ++iz) {
        const float *C = A.bc_c + size_t(bs) * 6 * NQ + iz * 25 + cq;
        const float cxx = C[0], cyy = C[NQ], czz = C[2 * NQ], cxy = C[3 * NQ], cxz = C[4 * NQ], cyz = C[5 * NQ];
        if (cxx != 0.f || cyy != 0.f || czz != 0.f) {
          const float *v = A.vo + (size_t(4 * ez + iz) * A.NX * A.NY + size_t((by * TY + ly) * 4 + iy) * A.NX +
                                   (bx * TX + lx) * 4 + ix) * 3;
          const float vx = ld_dep(v), vy = ld_dep(v + 1), vz = ld_dep(v + 2);
          cset(a, cpos(iz, 0), cget(a, cpos(iz, 0)) - (cxx * vx + cxy * vy + cxz * vz));
          cset(a, cpos(iz, 1), cget(a, cpos(iz, 1)) - (cxy * vx + cyy * vy + cyz * vz));
          cset(a, cpos(iz, 2), cget(a, cpos(iz, 2)) - (cxz * vx + cyz * vy + czz * vz));
        }
      }
    }
    if (src >= 0) {
      const int step = ld_dep(A.step);
      for (int s = src; s >= 0; s = A.src_next[s]) {
        const float f = step < A.nstep ? ld_dep(A.stf + size_t(step) * A.nsrc + s) : 0.f;
#pragma unroll
        for (int iz = 0; iz < NG; ++iz)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            cset(a, cpos(iz, c), cget(a, cpos(iz, c)) + f * A.src_arr[(size_t(s) * 3 + c) * NQ + iz * 25 + cq]);
      }
    }
    if (act && ez + 1 < z1) { bs = __ldg(A.bc_slot + element(ez + 1)); src = __ldg(A.src_head + element(ez + 1)); }
    __syncthreads();               // F is read: its place takes the contributions
    if (act) st_col(sF0 + tid * CS, a);
    cp_wait<1>();                  // this layer's v and M^-1 (own copies)
    __syncthreads();
    if (col) {
      // the tile's sum at each of the column's points: x neighbours, then y
      Col s;
      const int ex1 = min(tx >> 2, nax - 1), ey1 = min(ty >> 2, nay - 1);
      const bool px = (tx & 3) == 0 && tx > 0 && tx < 4 * nax, py = (ty & 3) == 0 && ty > 0 && ty < 4 * nay;
      auto part = [&](int eyy) {
        const int jy = ty - 4 * eyy;
        Col r = ld_col(sF0 + ((eyy * TX + (px ? ex1 - 1 : ex1)) * 25 + jy * NG + tx - 4 * (px ? ex1 - 1 : ex1)) * CS);
        if (px) col_add(r, ld_col(sF0 + ((eyy * TX + ex1) * 25 + jy * NG) * CS));
        return r;
      };
      s = part(py ? ey1 - 1 : ey1);
      if (py) col_add(s, part(ey1));
      const Col u = ld_col(U + tid * CS);
      const float *vm = sV + tid;
#pragma unroll
      for (int iz = 0; iz < 4; ++iz) {
        float t[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) t[c] = cget(s, cpos(iz, c));
        if (iz == 0 && ez > z0) {
#pragma unroll
          for (int c = 0; c < 3; ++c) t[c] = carry[c] + t[c];
        }
        if (iz == 0 && ez == z0 && z0 > 0) {
          float *d = A.upper + ((size_t(tile) * A.nchunk + chunk) * NCOL + tid) * 3;
          d[0] = t[0]; d[1] = t[1]; d[2] = t[2];
        } else if (rim) {
          float *d = A.rim + ((size_t(tile) * A.NZ + 4 * ez + iz) * NEDGE + rim_index(tx, ty)) * 3;
          d[0] = t[0]; d[1] = t[1]; d[2] = t[2];
        } else {
          const size_t g = gcol + size_t(4 * ez + iz) * plane;
#pragma unroll
          for (int c = 0; c < 3; ++c)
            bad |= finish_value(A, g + c, t[c], cget(u, cpos(iz, c)), vm[(iz * 3 + c) * NCOL],
                                vm[(12 + iz * 3 + c) * NCOL]);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) carry[c] = cget(s, cpos(4, c));
      if (ez + 1 == z1) {
        // the top plane of the block
        if (z1 < A.nez) {
          float *d = A.lower + ((size_t(tile) * A.nchunk + chunk) * NCOL + tid) * 3;
          d[0] = carry[0]; d[1] = carry[1]; d[2] = carry[2];
        } else if (rim) {
          float *d = A.rim + ((size_t(tile) * A.NZ + 4 * z1) * NEDGE + rim_index(tx, ty)) * 3;
          d[0] = carry[0]; d[1] = carry[1]; d[2] = carry[2];
        } else {
          const size_t g = gcol + size_t(4 * z1) * plane;
#pragma unroll
          for (int c = 0; c < 3; ++c)
            bad |= finish_value(A, g + c, carry[c], cget(u, cpos(4, c)), ld_dep(A.vo + g + c), __ldg(A.minv + g + c));
        }
      }
    }
  }
  if (bad) *A.flag = 1;
}

// One receiver by 128 threads (q = thread, red [3][128]): Lagrange
// interpolation with a fixed-order tree sum.  late: the velocity and
// acceleration types, else the displacement ones.
__device__ __forceinline__ void receive3(const Step3Args &A, int rr, int q, float (*red)[128], bool on, bool late) {
  const int e = on ? A.rec_elem[rr] : 0;
  const int ex = e % A.nex, ey = (e / A.nex) % A.ney, ez = e / (A.nex * A.ney);
  const int ix = q % NG, iy = (q / NG) % NG, iz = q / (NG * NG);
  const size_t g = ((size_t(4 * ez + iz) * A.NY + 4 * ey + iy) * A.NX + 4 * ex + ix) * 3;
  // the old fields and the weight before the wait
  float fo[3] = {0.f, 0.f, 0.f}, h = 0.f;
  if (on && q < NQ) {
    h = A.rec_h[size_t(rr) * NQ + q];
#pragma unroll
    for (int c = 0; c < 3; ++c) fo[c] = ld_l2((late ? A.vo : A.uo) + g + c);
  }
  pdl_wait();
  pdl_release();
  const int step = on ? ld_dep(A.step + 1) : 0;
  for (int t = 0; t < A.ntypes; ++t) {
    const int ty = A.types[t];
    if ((ty != 0) != late) continue;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float val = 0.f;
      if (on && q < NQ) {
        float f = fo[c];
        if (late) {
          const float a = ld_dep(A.a_store + g + c);
          f = ty == 2 ? a : __fadd_rn(fo[c], __fmul_rn(A.dt2, a));
        }
        val = h * f;
      }
      red[c][q] = val;
    }
    __syncthreads();
    for (int o = 64; o > 0; o >>= 1) {
      if (q < o)
#pragma unroll
        for (int c = 0; c < 3; ++c) red[c][q] = red[c][q] + red[c][q + o];
      __syncthreads();
    }
    if (on && q < 3 && step < A.nsig) A.seis[((size_t(step) * A.ntypes + t) * A.nrec + rr) * 3 + q] = red[q][0];
    __syncthreads();
  }
}

// Planes a block of the finish kernel takes of a tile's rim: many where that
// still gives every SM a few blocks.
__host__ __device__ inline int finish_planes(int ntile, int NZ) { return ntile * (NZ / 32) >= 3 * 148 ? 32 : 8; }
constexpr int FIN_RUN = 2;            // planes a thread takes of one column

// The tiles' sum of one shared point (column (tx, ty) of the tile, lattice
// plane gz): the tiles' parts in tile order, across a plane between two
// chunks the lower plus the upper part of each tile.
__device__ __forceinline__ void shared_sum(const Step3Args &A, int tile, int tx, int ty, bool left, bool below, int gz,
                                           float s[3]) {
  const int kk = gz > 0 && gz < A.NZ - 1 && gz % (4 * A.L) == 0 ? gz / (4 * A.L) : -1;
  bool first = true;
#pragma unroll
  for (int dy = 1; dy >= 0; --dy)
#pragma unroll
    for (int dx = 1; dx >= 0; --dx) {
      if ((dx && !left) || (dy && !below)) continue;
      const int t = tile - dx - dy * A.nbx;
      const int cx = dx ? CX - 1 : tx, cy = dy ? CY - 1 : ty;
      float p[3];
      if (kk >= 0) {
        const float *lo = A.lower + ((size_t(t) * A.nchunk + kk - 1) * NCOL + cy * CX + cx) * 3;
        const float *up = A.upper + ((size_t(t) * A.nchunk + kk) * NCOL + cy * CX + cx) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) p[c] = ld_dep(lo + c) + ld_dep(up + c);
      } else {
        const float *r = A.rim + ((size_t(t) * A.NZ + gz) * NEDGE + rim_index(cx, cy)) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) p[c] = ld_dep(r + c);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) s[c] = first ? p[c] : s[c] + p[c];
      first = false;
    }
}

// The shared points.  Blocks: rec_blocks with two receivers each, then (tile,
// group of finish_planes planes), then (tile, plane between two chunks).  A
// point is about 18 loads that depend on nothing but its place, so the kernel
// lives on loads in flight: a thread takes FIN_RUN planes of one column and
// issues the fields of all of them before the first sum.
__global__ void __launch_bounds__(256) k_finish3d(const __grid_constant__ Step3Args A) {
  __shared__ float red[2][3][128];
  const int tid = threadIdx.x;
  const int ntile = A.nbx * A.nby, FIN_PLANES = finish_planes(ntile, A.NZ), ngroup = (A.NZ + FIN_PLANES - 1) / FIN_PLANES;
  int b = int(blockIdx.x) - A.rec_blocks;
  if (b < 0) {
    const int rr = blockIdx.x * 2 + (tid >> 7);
    receive3(A, rr, tid & 127, red[tid >> 7], rr < A.nrec, false);
    return;
  }
  const bool rimrun = b < ntile * ngroup;
  if (!rimrun) b -= ntile * ngroup;
  const int tile = b % ntile, k = b / ntile;       // k: plane group, or chunk boundary
  const int bx = tile % A.nbx, by = tile / A.nbx;
  // the tile's own columns: its low rim, and its high end on the mesh boundary
  const int nax = min(TX, A.nex - bx * TX), nay = min(TY, A.ney - by * TY);
  const int ncx = 4 * nax + (bx == A.nbx - 1), ncy = 4 * nay + (by == A.nby - 1);
  const int nl = bx > 0 ? ncy : 0, nb = by > 0 ? ncx - (bx > 0) : 0;   // columns x = 0, then y = 0
  const int per = rimrun ? nl + nb : ncx * ncy;
  const int planes = rimrun ? min(FIN_PLANES, A.NZ - k * FIN_PLANES) : 1;
  const int runs = (planes + FIN_RUN - 1) / FIN_RUN;
  const size_t plane = size_t(A.NX) * A.NY * 3;
  bool bad = false;
  bool waited = false;
  for (int i = tid; i < per * runs; i += blockDim.x) {
    const int run = i / per, j = i - run * per;
    const int gz0 = rimrun ? k * FIN_PLANES + run * FIN_RUN : 4 * A.L * (k + 1);
    const int n = rimrun ? min(FIN_RUN, planes - run * FIN_RUN) : 1;
    int tx, ty;
    if (rimrun) {
      if (j < nl) { tx = 0; ty = j; }
      else { tx = j - nl + (bx > 0); ty = 0; }
    } else {
      tx = j % ncx; ty = j / ncx;
    }
    const bool left = tx == 0 && bx > 0, below = ty == 0 && by > 0;
    if (!rimrun && (left || below)) continue;    // in the rim run
    const size_t g = ((size_t(gz0) * A.NY + by * 4 * TY + ty) * A.NX + bx * 4 * TX + tx) * 3;
    float u[FIN_RUN][3], v[FIN_RUN][3], mi[FIN_RUN][3], s[FIN_RUN][3];
#pragma unroll
    for (int r = 0; r < FIN_RUN; ++r)
      if (r < n)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const size_t o = g + r * plane + c;
          u[r][c] = ld_l2(A.uo + o); v[r][c] = ld_l2(A.vo + o); mi[r][c] = __ldg(A.minv + o);
        }
    if (!waited) { pdl_wait(); pdl_release(); waited = true; }
#pragma unroll
    for (int r = 0; r < FIN_RUN; ++r)
      if (r < n) shared_sum(A, tile, tx, ty, left, below, gz0 + r, s[r]);
#pragma unroll
    for (int r = 0; r < FIN_RUN; ++r)
      if (r < n)
#pragma unroll
        for (int c = 0; c < 3; ++c) bad |= finish_value(A, g + r * plane + c, s[r][c], u[r][c], v[r][c], mi[r][c]);
  }
  if (!waited) { pdl_wait(); pdl_release(); }
  if (bad) *A.flag = 1;
  if (A.advance && rimrun && b == 0 && tid == 0) A.step[0] += 1;
}

// Velocity and acceleration receivers, after the finish kernel: a block of 128
// threads a receiver, from the old velocity and the stored acceleration.
__global__ void __launch_bounds__(128) k_receivers3d(const __grid_constant__ Step3Args A) {
  __shared__ float red[3][128];
  receive3(A, blockIdx.x, threadIdx.x, red, true, true);
}

__global__ void __launch_bounds__(256) k_predict3d(float *__restrict__ u, float *__restrict__ v,
                                                   const float *__restrict__ a, size_t n, float dt, float dt2,
                                                   float dtsq2) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    float uu = u[i], vv = v[i];
    nm_predict(uu, vv, a[i], dt, dt2, dtsq2);
    u[i] = uu;
    v[i] = vv;
  }
}

}  // namespace dev
}  // namespace sfg3
