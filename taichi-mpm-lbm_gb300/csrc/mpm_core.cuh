// MLS-MPM building blocks shared by the single-solver kernels (mpm.cu) and the batched
// kernels (batch.cu): solver parameters, particle views, B-spline weights, the polar
// rotation, and the per-CTA bodies of P2G (optionally with the penalty coupling folded in),
// grid update + G2P and the block clear.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "coupling_core.cuh"
#include "fsi_common.cuh"

namespace fsi {
namespace {

constexpr int kTileCap = 2048;  // nodes per shared tile

struct Mpm {
  int nx, ny, nz;
  int n;  // particles
  float dt, dx, inv_dx, mu, lam, g[3], damping;
  int bw, apic;
  float lower, upper[3];
  long long cap;
  int nbx, nby, nbz;  // 4^3 block grid
  int material;       // FSI_MATERIAL_*
  int threads;        // threads per block of the tiled P2G / G2P (128, 256 or 512)
  int fold;           // coupled tiled substep: 0 by particle count, 1 in P2G, 2 separate,
                      // 3 separate force and spread kernels
};

struct PView {
  float* __restrict__ x;
  float* __restrict__ v;
  float* __restrict__ C;
  float* __restrict__ F;
  const float* __restrict__ mass;
  const float* __restrict__ vol;
  const int32_t* __restrict__ active;
  float* __restrict__ fp;
  const float* __restrict__ mu;   // per-particle Lame parameters, or NULL
  const float* __restrict__ lam;
};

__device__ __forceinline__ void base_fx(const Mpm& m, const float x[3], int base[3], float fx[3]) {
  // base = trunc(x * inv_dx - 0.5) (cast toward zero), fx = x * inv_dx - base (mpm3d.py:239-240).
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float gpos = __fmul_rn(x[a], m.inv_dx);
    base[a] = base_cell(__fsub_rn(gpos, 0.5f));
    fx[a] = __fsub_rn(gpos, (float)base[a]);
  }
}


__device__ __forceinline__ float dot3r(float a0, float a1, float a2, float b0, float b1, float b2) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a0, b0), __fmul_rn(a1, b1)), __fmul_rn(a2, b2));
}

// out = A B for row-major 3x3, sequential sum over k.
__device__ __forceinline__ void matmul3(const float* A, const float* B, float* out) {
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      out[3 * a + b] = dot3r(A[3 * a], A[3 * a + 1], A[3 * a + 2], B[b], B[3 + b], B[6 + b]);
}

__device__ __forceinline__ float det3(const float* a) {
  const float t0 = __fsub_rn(__fmul_rn(a[4], a[8]), __fmul_rn(a[7], a[5]));
  const float t1 = __fsub_rn(__fmul_rn(a[1], a[8]), __fmul_rn(a[7], a[2]));
  const float t2 = __fsub_rn(__fmul_rn(a[1], a[5]), __fmul_rn(a[4], a[2]));
  float d = __fsub_rn(__fmul_rn(a[0], t0), __fmul_rn(a[3], t1));
  return __fadd_rn(d, __fmul_rn(a[6], t2));
}

// Rotation of the polar decomposition by one-sided Jacobi SVD (Hestenes 1958):
// orthogonalise the columns of A = F V by plane rotations; R = U V^T with
// U = A column-normalised, the smallest column flipped if U V^T is improper.
__device__ void polar_jacobi(const float* F, float* R) {
  float A[9], V[9] = {1.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f, 1.f};
#pragma unroll
  for (int i = 0; i < 9; ++i) A[i] = F[i];
  for (int sweep = 0; sweep < 8; ++sweep) {
    float off = 0.f;
#pragma unroll
    for (int pq = 0; pq < 3; ++pq) {
      const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
      const float alpha = dot3r(A[p], A[3 + p], A[6 + p], A[p], A[3 + p], A[6 + p]);
      const float beta = dot3r(A[q], A[3 + q], A[6 + q], A[q], A[3 + q], A[6 + q]);
      const float gamma = dot3r(A[p], A[3 + p], A[6 + p], A[q], A[3 + q], A[6 + q]);
      if (gamma == 0.f) continue;
      off = fmaxf(off, fabsf(gamma) / sqrtf(alpha * beta));
      const float zeta = (beta - alpha) / (2.f * gamma);
      const float t = copysignf(1.f, zeta) / (fabsf(zeta) + sqrtf(1.f + zeta * zeta));
      const float c = 1.f / sqrtf(1.f + t * t), s = c * t;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float ap = A[3 * r + p], aq = A[3 * r + q];
        A[3 * r + p] = c * ap - s * aq;
        A[3 * r + q] = s * ap + c * aq;
        const float vp = V[3 * r + p], vq = V[3 * r + q];
        V[3 * r + p] = c * vp - s * vq;
        V[3 * r + q] = s * vp + c * vq;
      }
    }
    if (off < 1e-7f) break;
  }
  float nrm[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) nrm[c] = sqrtf(A[c] * A[c] + A[3 + c] * A[3 + c] + A[6 + c] * A[6 + c]);
  float U[9];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) U[3 * r + c] = nrm[c] > 0.f ? A[3 * r + c] / nrm[c] : (r == c ? 1.f : 0.f);
  if (det3(U) * det3(V) < 0.f) {
    int cmin = 0;
    if (nrm[1] < nrm[cmin]) cmin = 1;
    if (nrm[2] < nrm[cmin]) cmin = 2;
#pragma unroll
    for (int r = 0; r < 3; ++r) U[3 * r + cmin] = -U[3 * r + cmin];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      R[3 * a + b] = U[3 * a] * V[3 * b] + U[3 * a + 1] * V[3 * b + 1] + U[3 * a + 2] * V[3 * b + 2];
}

// Rotation of F = R S by Newton's iteration X <- (z X + X^{-T}/z)/2 with
// Frobenius-norm scaling z = (|X^{-1}|_F / |X|_F)^{1/2} (Higham, SIAM J. Sci.
// Stat. Comput. 7, 1986). Used for det F > 0, where R is the unique rotation
// the reference obtains as U V^T from ti.svd (mpm3d.py:245-246); inverted or
// degenerate F fall back to the Jacobi SVD.
__device__ void polar_rotation(const float* F, float* R) {
  float X[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) X[i] = F[i];
  if (!(det3(F) > 1e-20f)) {
    polar_jacobi(F, R);
    return;
  }
  bool scale = true;
  for (int it = 0; it < 16; ++it) {
    float Cf[9];
    Cf[0] = X[4] * X[8] - X[5] * X[7];
    Cf[1] = X[5] * X[6] - X[3] * X[8];
    Cf[2] = X[3] * X[7] - X[4] * X[6];
    Cf[3] = X[2] * X[7] - X[1] * X[8];
    Cf[4] = X[0] * X[8] - X[2] * X[6];
    Cf[5] = X[1] * X[6] - X[0] * X[7];
    Cf[6] = X[1] * X[5] - X[2] * X[4];
    Cf[7] = X[2] * X[3] - X[0] * X[5];
    Cf[8] = X[0] * X[4] - X[1] * X[3];
    const float det = X[0] * Cf[0] + X[1] * Cf[1] + X[2] * Cf[2];
    float z = 1.f;
    if (scale) {
      float nx2 = 0.f, nc2 = 0.f;
#pragma unroll
      for (int i = 0; i < 9; ++i) { nx2 += X[i] * X[i]; nc2 += Cf[i] * Cf[i]; }
      z = sqrtf(sqrtf(nc2 / nx2) / fabsf(det));
    }
    const float a = 0.5f * z, b = 0.5f / (z * det);
    float d2 = 0.f, n2 = 0.f;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const float xn = a * X[i] + b * Cf[i];
      const float dd = xn - X[i];
      d2 += dd * dd;
      n2 += xn * xn;
      X[i] = xn;
    }
    if (d2 < 1e-4f * n2) scale = false;
    if (d2 <= 1e-13f * n2) break;
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) R[i] = X[i];
}

__device__ __forceinline__ bool inside(const Mpm& m, int i, int j, int k) {
  return 0 <= i && i < m.nx && 0 <= j && j < m.ny && 0 <= k && k < m.nz;
}

__device__ __forceinline__ long long node_index(const Mpm& m, int i, int j, int k) {
  return ((long long)i * m.ny + j) * m.nz + k;
}

__device__ __forceinline__ void mark_block(const Mpm& m, uint8_t* dirty, int i, int j, int k) {
  dirty[((long long)(i >> 2) * m.nby + (j >> 2)) * m.nbz + (k >> 2)] = 1;
}

// Block-wide bounding box of the stencils of this CTA's active particles.
struct Box {
  int lo[3], ext[3];
  int vol;
};

// The part in the grid of the box [sh[0..2], sh[3..5]]; vol: its nodes, at most kTileCap + 1.
template <class G>
__device__ __forceinline__ Box box_of(const G& m, const int* sh) {
  Box box;
  const int n[3] = {m.nx, m.ny, m.nz};
  long long vol = 1;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int lo = max(sh[a], 0), hi = min(sh[3 + a], n[a] - 1);
    box.lo[a] = lo;
    box.ext[a] = hi >= lo ? hi - lo + 1 : 0;
    vol *= box.ext[a];
  }
  box.vol = vol > (long long)kTileCap ? kTileCap + 1 : (int)vol;
  return box;
}

template <class G>
__device__ bool cta_box(const G& m, bool act, const int base[3], Box& box, int* sh) {
  // sh: 6 ints of shared scratch
  if (threadIdx.x < 3) { sh[threadIdx.x] = 0x7fffffff; sh[3 + threadIdx.x] = -0x7fffffff; }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int lo = act ? base[a] : 0x7fffffff;
    int hi = act ? base[a] + 2 : -0x7fffffff;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) { atomicMin(&sh[a], lo); atomicMax(&sh[3 + a], hi); }
  }
  __syncthreads();
  if (sh[0] == 0x7fffffff) return false;  // no active particle
  box = box_of(m, sh);
  return true;
}

// For a CTA whose box is too large, the usual reason being that its particles end one body and
// begin the next: cuts it in two where consecutive particles are farthest apart. Returns this
// thread's part (false: before the cut) and both boxes; every thread calls it.
// sh: 13 ints of shared scratch, last: 4 ints per warp.
template <class G>
__device__ bool cut_boxes(const G& m, bool act, const int base[3], Box box[2], int* sh, int (*last)[4]) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  __syncthreads();  // the whole box's scratch is no longer read
  if (t < 12) sh[t] = t % 6 < 3 ? 0x7fffffff : -0x7fffffff;
  if (t == 12) sh[12] = 0;
  if (lane == 31) {
    last[warp][0] = base[0]; last[warp][1] = base[1]; last[warp][2] = base[2]; last[warp][3] = act;
  }
  __syncthreads();
  int before[4] = {base[0], base[1], base[2], act};
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    before[a] = __shfl_up_sync(0xffffffffu, before[a], 1);
    if (lane == 0 && warp > 0) before[a] = last[warp - 1][a];
  }
  int far = 0;  // distance << 10 | thread
  if (act && t > 0 && before[3]) {
    // each term below 2^20, whatever the coordinates
    unsigned d = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned u = base[a] > before[a] ? (unsigned)base[a] - (unsigned)before[a]
                                             : (unsigned)before[a] - (unsigned)base[a];
      d += min(u, 0x7ffffu);
    }
    far = (int)(min(d, 0x1fffffu) << 10) | t;
  }
  far = __reduce_max_sync(0xffffffffu, far);
  if (lane == 0) atomicMax(&sh[12], far);
  __syncthreads();
  const bool part = t >= (sh[12] & 1023);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const bool mine = act && part == (h == 1);
      const int lo = __reduce_min_sync(0xffffffffu, mine ? base[a] : 0x7fffffff);
      const int hi = __reduce_max_sync(0xffffffffu, mine ? base[a] + 2 : -0x7fffffff);
      if (lane == 0) { atomicMin(&sh[6 * h + a], lo); atomicMax(&sh[6 * h + 3 + a], hi); }
    }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    box[h] = box_of(m, sh + 6 * h);
    if (sh[6 * h] == 0x7fffffff) box[h].vol = 0;
  }
  return part;
}

// Shared scratch of stage_stencils.
struct StageScratch {
  int box[16], last[16][4];
};

// The 3-vectors of a CTA's stencil nodes in shared memory: node (i, j, k) of this thread's stencil
// is at t0 + i s0 + j s1 + k. ok: the stencils fit the tile.
struct Staged {
  const float (*tile)[kTileCap];
  bool any, ok;  // any: the CTA has an active particle
  int t0, s0, s1;
  __device__ __forceinline__ void operator()(int i, int j, int k, float v[3]) const {
    const int t = t0 + i * s0 + j * s1 + k;
    v[0] = tile[0][t]; v[1] = tile[1][t]; v[2] = tile[2][t];
  }
};

// Stages the box of the CTA's stencils (two boxes where it ends one body and begins the next), every
// node once: load(i, j, k, v). Every thread calls it.
template <class G, class Load>
__device__ __forceinline__ Staged stage_stencils(const G& m, bool act, const int base[3],
                                                 float (*tile)[kTileCap], StageScratch& sc, Load load) {
  Staged st;
  st.tile = tile;
  st.ok = false;
  Box box;
  st.any = cta_box(m, act, base, box, sc.box);
  if (!st.any) return st;
  // A box's nodes into the tile from `at`. Quotients of t < kTileCap by float reciprocals: (t + 1/2) / e
  // is at least 1 / (2 e) from an integer, its rounding error below 2^-22 t / e.
  auto stage = [&](const Box& b, int at) {
    const int e12 = b.ext[1] * b.ext[2];
    const float r12 = 1.f / (float)e12, r2 = 1.f / (float)b.ext[2];
    for (int t = threadIdx.x; t < b.vol; t += blockDim.x) {
      const int ti = (int)(((float)t + 0.5f) * r12), r = t - ti * e12;
      const int tj = (int)(((float)r + 0.5f) * r2), tk = r - tj * b.ext[2];
      float v[3];
      load(b.lo[0] + ti, b.lo[1] + tj, b.lo[2] + tk, v);
      tile[0][at + t] = v[0]; tile[1][at + t] = v[1]; tile[2][at + t] = v[2];
    }
  };
  st.ok = box.vol <= kTileCap;
  int off = 0;  // this thread's box in the tile
  if (st.ok) {
    stage(box, 0);
  } else {
    Box two[2];
    const bool part = cut_boxes(m, act, base, two, sc.box, sc.last);
    st.ok = two[0].vol + two[1].vol <= kTileCap;
    if (st.ok) {
      stage(two[0], 0);
      stage(two[1], two[0].vol);
      box = part ? two[1] : two[0];
      off = part ? two[0].vol : 0;
    }
  }
  __syncthreads();
  st.s1 = box.ext[2];
  st.s0 = box.ext[1] * box.ext[2];
  st.t0 = off + (base[0] - box.lo[0]) * st.s0 + (base[1] - box.lo[1]) * st.s1 + (base[2] - box.lo[2]);
  return st;
}

__device__ __forceinline__ void load_particle_x(const PView& P, long long cap, int p, float x[3]) {
  x[0] = P.x[p]; x[1] = P.x[cap + p]; x[2] = P.x[2 * cap + p];
}

// The once-per-particle part of P2G for active particle p (mpm3d.py:242-252):
// F <- (I + dt C) F (written back), the stress, and affine = stress term + m C.
__device__ __forceinline__ void p2g_stress_affine(const Mpm& m, const PView& P, int p,
                                                  float affine[9], float& mass) {
  const long long cap = m.cap;
  float Cp[9], Fp[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) { Cp[i] = P.C[i * cap + p]; Fp[i] = P.F[i * cap + p]; }
  // F <- (I + dt C) F (mpm3d.py:243)
  float A[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) A[i] = __fadd_rn((i % 4 == 0) ? 1.f : 0.f, __fmul_rn(m.dt, Cp[i]));
  float Fn[9];
  matmul3(A, Fp, Fn);
#pragma unroll
  for (int i = 0; i < 9; ++i) P.F[i * cap + p] = Fn[i];
  const float J = det3(Fn);
  const float mu = P.mu ? P.mu[p] : m.mu;
  const float lam = P.lam ? P.lam[p] : m.lam;
  float Ft[9], S[9];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) Ft[3 * a + b] = Fn[3 * b + a];
  if (m.material == FSI_MATERIAL_NEO_HOOKEAN) {
    // Kirchhoff stress of compressible Neo-Hookean: mu (F F^T - I) + lam ln(J) I.
    matmul3(Fn, Ft, S);
#pragma unroll
    for (int i = 0; i < 9; ++i) S[i] = __fmul_rn(mu, __fsub_rn(S[i], (i % 4 == 0) ? 1.f : 0.f));
    const float ll = __fmul_rn(lam, logf(J));
    S[0] = __fadd_rn(S[0], ll); S[4] = __fadd_rn(S[4], ll); S[8] = __fadd_rn(S[8], ll);
  } else {
    // Fixed-corotated: 2 mu (F - R) F^T + lam J (J - 1) I (mpm3d.py:247-251)
    float R[9];
    polar_rotation(Fn, R);
    const float twomu = __fmul_rn(2.f, mu);
    float Pm[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) Pm[i] = __fmul_rn(twomu, __fsub_rn(Fn[i], R[i]));
    matmul3(Pm, Ft, S);
    const float lj = __fmul_rn(__fmul_rn(lam, J), __fsub_rn(J, 1.f));
    S[0] = __fadd_rn(S[0], lj); S[4] = __fadd_rn(S[4], lj); S[8] = __fadd_rn(S[8], lj);
  }
  float coef = __fmul_rn(__fmul_rn(__fmul_rn(-m.dt, P.vol[p]), 4.f), m.inv_dx);
  coef = __fmul_rn(coef, m.inv_dx);
  mass = P.mass[p];
#pragma unroll
  for (int i = 0; i < 9; ++i) affine[i] = __fadd_rn(__fmul_rn(coef, S[i]), __fmul_rn(mass, Cp[i]));
}

// Exclusive scan over the block (blockDim.x a multiple of 32, at most 1024 threads).
// `ws` is 32 ints of shared scratch; *total receives the block's sum.
__device__ __forceinline__ int block_excl_scan(int v, int* ws, int* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) ws[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int s = lane < nw ? ws[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    ws[lane] = s;
  }
  __syncthreads();
  const int excl = incl - v + (wid > 0 ? ws[wid - 1] : 0);
  *total = ws[nw - 1];
  __syncthreads();
  return excl;
}

// Whether the scatter beside a lattice of this population storage sums in runs (p2g_runs_body, the
// coupling staged), or in the order of the tile (p2g_tile_body, the coupling read directly). A 16-bit
// lattice turns last-bit differences of the reaction into whole quanta of its populations, so the sums
// that feed it keep their order: with runs, C of 6 to 24 FP16 scenes after 8 steps is 2.3e-5 from the
// tile's, with the tile 1.7e-5 from itself. The tile costs 335 us for 64 scenes, runs 109. FP32
// lattices pass the differences on as they are: 2.1e-5 against 1.4e-5, over 80 substeps.
inline bool scatter_in_runs(int32_t storage) { return storage == FSI_STORAGE_F32; }

// ------------------------------------------------- P2G of a CTA's particles, in runs
//
// The scatter sums what a CTA's particles add to a node before anything is added in global
// memory. Each thread writes its particle's record (weights, affine, momentum) into shared
// memory at the particle's place in base-cell order: a counting sort over the base cells of the
// CTA's bounding box, integers only, ties in thread order. The records are then cut into equal
// runs, one per group of nine lanes: lane (ox, oy) of a group walks its run and keeps the sums
// of the nodes (ox, oy, 0..2) of the current base cell in registers. A step to the next cell
// along z retires one node and shifts the other two, any other step retires all three. A
// retired node is one vector reduction into global memory.
//
// Why: particles of a body are stored cell by cell, so 256 of them fill 80 to 120 base cells,
// and a float atomic in shared memory is a compare-and-swap loop. A tile of nodes in shared
// memory takes 108 of them per particle (27 nodes, four components); here there are none, and
// about 5 vector reductions per particle. Measured, one launch for 2,097,152 / 502,304
// particles: 359 / 115 us with the tile, 188 / 49 us with runs. Adding the runs up once more per
// node in shared memory, for one reduction per node and CTA, took 340 us: its barriers, and runs
// cut at the ends of lines.
constexpr int kScatterCells = 2048;  // base cells of the bounding box that the sort counts

// A particle's record in shared memory, as float offsets: 0-2 wx, 3 mass, 4-6 wy, 7 cell key,
// 8-10 wz, 11 fz, 12-20 affine, 21-23 m v + dt f, 24-25 fx, fy. 28 floats: 16 bytes short of 128,
// so records of neighbouring places start on different banks.
constexpr int kRecFloats = 28;

// Shared memory of the P2G of kT threads (dynamic: 29 KB for 256 threads).
template <int kT>
struct __align__(16) ScatterSmem {
  // the sort's counts, then the records
  float rec[kT * kRecFloats > kScatterCells ? kT * kRecFloats : kScatterCells];
  int16_t arrived[kT];
  int ws[32];
  int box[8];
};

// A CTA's particles in base-cell order.
struct CellOrder {
  int lo[3];     // lowest base cell
  int ext[3];    // base cells of the bounding box
  int count;     // particles
  int pos;       // this thread's place
  uint32_t key;  // its cell relative to lo: x, y, z in 10 bits each
  bool fits;     // the box fits the sort
};

// `in`: this thread's particle takes part, with base cell `base` in [-2, n) on each axis. Every
// thread of the CTA calls it; it ends after a barrier that follows the last read of the counts.
template <int kT>
__device__ __forceinline__ CellOrder cell_order(bool in, const int base[3], ScatterSmem<kT>& sm) {
  int* const cnt = reinterpret_cast<int*>(sm.rec);
  int* const sh = sm.box;
  CellOrder o;
  if (threadIdx.x < 3) { sh[threadIdx.x] = 0x7fffffff; sh[3 + threadIdx.x] = -0x7fffffff; }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int lo = __reduce_min_sync(0xffffffffu, in ? base[a] : 0x7fffffff);
    const int hi = __reduce_max_sync(0xffffffffu, in ? base[a] : -0x7fffffff);
    if ((threadIdx.x & 31) == 0) { atomicMin(&sh[a], lo); atomicMax(&sh[3 + a], hi); }
  }
  o.count = __syncthreads_count(in);
  o.pos = 0;
  o.key = 0;
  long long cells = 1;
  bool narrow = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o.lo[a] = sh[a];
    o.ext[a] = o.count ? sh[3 + a] - sh[a] + 1 : 0;
    cells *= o.ext[a];
    narrow = narrow && o.ext[a] < 1023;
  }
  o.fits = narrow && cells <= kScatterCells;
  if (!o.fits || o.count == 0) return o;
  const int nc = (int)cells;
  for (int c = threadIdx.x; c < nc; c += kT) cnt[c] = 0;
  __syncthreads();
  int cell = 0, slot = 0;
  if (in) {
    const int l0 = base[0] - o.lo[0], l1 = base[1] - o.lo[1], l2 = base[2] - o.lo[2];
    o.key = ((uint32_t)l0 << 20) | ((uint32_t)l1 << 10) | (uint32_t)l2;
    cell = (l0 * o.ext[1] + l1) * o.ext[2] + l2;
    slot = atomicAdd(&cnt[cell], 1);
  }
  __syncthreads();
  const int per = (nc + kT - 1) / kT;
  const int c0 = threadIdx.x * per;
  int sum = 0;
  for (int c = c0; c < min(c0 + per, nc); ++c) sum += cnt[c];
  int total;
  int run = block_excl_scan(sum, sm.ws, &total);
  for (int c = c0; c < min(c0 + per, nc); ++c) {
    const int v = cnt[c];
    cnt[c] = run;
    run += v;
  }
  __syncthreads();
  // order of arrival within the cell -> thread order
  const int start = cnt[cell], end = cell + 1 < nc ? cnt[cell + 1] : o.count;
  if (in) sm.arrived[start + slot] = (int16_t)threadIdx.x;
  __syncthreads();
  if (in) {
    o.pos = start;
    for (int s = start; s < end; ++s) o.pos += sm.arrived[s] < (int)threadIdx.x;
  }
  return o;
}

// Adds the records in `rec` (in cell order) into the grid.
template <int kT>
__device__ __forceinline__ void scatter_runs(const Mpm& m, const CellOrder& o, const float* rec,
                                             float4* __restrict__ grid) {
  constexpr int kGroups = kT / 32 * 3;
  constexpr uint32_t kNone = 0xfffffff0u;  // no cell: neither it nor the next is a key
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = lane / 9, r9 = lane - 9 * grp;
  const int ox = r9 / 3, oy = r9 - 3 * ox;
  const int per = (o.count + kGroups - 1) / kGroups;
  int q = (warp * 3 + grp) * per;
  const int end = grp < 3 ? min(q + per, o.count) : q;  // lanes 27-31 have no group
  const float fox = (float)ox, foy = (float)oy;
  float am[3][4];
#pragma unroll
  for (int z = 0; z < 3; ++z) am[z][0] = am[z][1] = am[z][2] = am[z][3] = 0.f;
  uint32_t cur = kNone;
  bool row = false;    // the lane's (x, y) lies in the grid
  int k0 = 0;          // z of the current base cell
  long long node = 0;  // index of node (ox, oy, 0) of the current base cell
  auto retire = [&](int z) {
    if (row && k0 + z >= 0 && k0 + z < m.nz)
      red_add_v4(grid + node + z, am[z][0], am[z][1], am[z][2], am[z][3]);
  };
  for (; q < end; ++q) {
    const float* r = rec + q * kRecFloats;
    const uint32_t key = __float_as_uint(r[7]);
    if (key != cur) {
      if (key == cur + 1u) {
        retire(0);
#pragma unroll
        for (int a = 0; a < 4; ++a) { am[0][a] = am[1][a]; am[1][a] = am[2][a]; am[2][a] = 0.f; }
        ++k0;
        ++node;
      } else {
        if (cur != kNone) {
          retire(0); retire(1); retire(2);
#pragma unroll
          for (int z = 0; z < 3; ++z) am[z][0] = am[z][1] = am[z][2] = am[z][3] = 0.f;
        }
        const int i = o.lo[0] + (int)(key >> 20) + ox, j = o.lo[1] + (int)((key >> 10) & 1023u) + oy;
        k0 = o.lo[2] + (int)(key & 1023u);
        row = i >= 0 && i < m.nx && j >= 0 && j < m.ny;
        node = node_index(m, i, j, k0);
      }
      cur = key;
    }
    const float wxy = __fmul_rn(r[ox], r[4 + oy]);
    const float4 wz = *reinterpret_cast<const float4*>(r + 8);
    const float w[3] = {__fmul_rn(wxy, wz.x), __fmul_rn(wxy, wz.y), __fmul_rn(wxy, wz.z)};
    const float2 f = *reinterpret_cast<const float2*>(r + 24);
    const float d0 = __fsub_rn(fox, f.x), d1 = __fsub_rn(foy, f.y);
    const float4 a0 = *reinterpret_cast<const float4*>(r + 12);
    const float4 a1 = *reinterpret_cast<const float4*>(r + 16);
    const float4 a2 = *reinterpret_cast<const float4*>(r + 20);
    const float mass = r[3];
    // m v + dt f + A (node - x): the terms of ox and oy once for the three oz
    const float p0 = fmaf(a0.x, d0, fmaf(a0.y, d1, a2.y));
    const float p1 = fmaf(a0.w, d0, fmaf(a1.x, d1, a2.z));
    const float p2 = fmaf(a1.z, d0, fmaf(a1.w, d1, a2.w));
#pragma unroll
    for (int z = 0; z < 3; ++z) {
      const float d2 = __fsub_rn((float)z, wz.w);
      am[z][0] = fmaf(w[z], fmaf(a0.z, d2, p0), am[z][0]);
      am[z][1] = fmaf(w[z], fmaf(a1.y, d2, p1), am[z][1]);
      am[z][2] = fmaf(w[z], fmaf(a2.x, d2, p2), am[z][2]);
      am[z][3] = fmaf(w[z], mass, am[z][3]);
    }
  }
  if (cur != kNone) { retire(0); retire(1); retire(2); }
}

// Whether a stencil with this base cell has a node in the grid.
__device__ __forceinline__ bool stencil_in_grid(int nx, int ny, int nz, const int base[3]) {
  return base[0] >= -2 && base[0] < nx && base[1] >= -2 && base[1] < ny && base[2] >= -2 &&
         base[2] < nz;
}

// Marks the 4^3 node blocks that the stencils of the base cells lo .. lo + ext - 1 overlap.
__device__ __forceinline__ void mark_cells(const Mpm& m, uint8_t* __restrict__ dirty,
                                           const int lo[3], const int ext[3]) {
  const int n[3] = {m.nx, m.ny, m.nz};
  int b0[3], nb[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b0[a] = max(lo[a], 0) >> 2;
    nb[a] = (min(lo[a] + ext[a] + 1, n[a] - 1) >> 2) - b0[a] + 1;
  }
  for (int t = threadIdx.x; t < nb[0] * nb[1] * nb[2]; t += blockDim.x) {
    const int bi = b0[0] + t / (nb[1] * nb[2]), bj = b0[1] + (t / nb[2]) % nb[1], bk = b0[2] + t % nb[2];
    dirty[((long long)bi * m.nby + bj) * m.nbz + bk] = 1;
  }
}

// P2G of particle p (this thread) within its CTA of kT threads, in runs; every thread calls it.
// A CTA whose bounding box does not fit the sort (particles of two bodies far apart, or
// scattered ones) adds each contribution straight into global memory.
// Odd lanes walk the stencil backwards where contributions are added singly: the two particles of
// a sub-cell pair, which share a base cell, then add into different nodes at each step.
template <int kT>
__device__ __forceinline__ void p2g_runs_body(const Mpm& m, const PView& P, float4* __restrict__ grid,
                                              uint8_t* __restrict__ dirty, int p,
                                              ScatterSmem<kT>& sm) {
  const long long cap = m.cap;
  bool act = false;
  int base[3] = {0, 0, 0};
  float fx[3] = {0.f, 0.f, 0.f};
  if (p < m.n) {
    float x[3];  // beside the flag, not after it
    load_particle_x(P, cap, p, x);
    act = P.active[p] != 0;
    if (act) base_fx(m, x, base, fx);
  }
  const bool in = act && stencil_in_grid(m.nx, m.ny, m.nz, base);
  const CellOrder o = cell_order(in, base, sm);
  float affine[9], mv[3], dtf[3], mass = 0.f;
  if (act) {
    p2g_stress_affine(m, P, p, affine, mass);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mv[a] = __fmul_rn(mass, P.v[a * cap + p]);
      dtf[a] = __fmul_rn(m.dt, P.fp[a * cap + p]);
    }
  }
  if (o.count == 0) return;  // no stencil of this CTA reaches the grid
  if (o.fits) {
    if (in) {
      float* r = sm.rec + o.pos * kRecFloats;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        r[i] = bspline_w(fx[0], i);
        r[4 + i] = bspline_w(fx[1], i);
        r[8 + i] = bspline_w(fx[2], i);
      }
      r[3] = mass;
      r[7] = __uint_as_float(o.key);
      r[11] = fx[2];
#pragma unroll
      for (int i = 0; i < 9; ++i) r[12 + i] = __fmul_rn(affine[i], m.dx);
#pragma unroll
      for (int a = 0; a < 3; ++a) r[21 + a] = __fadd_rn(mv[a], dtf[a]);
      r[24] = fx[0];
      r[25] = fx[1];
    }
    __syncthreads();
    scatter_runs<kT>(m, o, sm.rec, grid);
    mark_cells(m, dirty, o.lo, o.ext);
    return;
  }
  if (!in) return;
  const bool rev = (threadIdx.x & 1) != 0;
#pragma unroll 1
  for (int t = 0; t < 27; ++t) {
    const int s = rev ? 26 - t : t;
    const int oi = s / 9, oj = (s / 3) % 3, ok = s % 3;
    const int i = base[0] + oi, j = base[1] + oj, k = base[2] + ok;
    if (!inside(m, i, j, k)) continue;
    const float w = __fmul_rn(__fmul_rn(bspline_w(fx[0], oi), bspline_w(fx[1], oj)), bspline_w(fx[2], ok));
    const float d[3] = {__fmul_rn(__fsub_rn((float)oi, fx[0]), m.dx),
                        __fmul_rn(__fsub_rn((float)oj, fx[1]), m.dx),
                        __fmul_rn(__fsub_rn((float)ok, fx[2]), m.dx)};
    float add[3];  // rounded term by term like the reference
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float ad = dot3r(affine[3 * a], affine[3 * a + 1], affine[3 * a + 2], d[0], d[1], d[2]);
      add[a] = __fmul_rn(w, __fadd_rn(__fadd_rn(mv[a], ad), dtf[a]));
    }
    red_add_v4(grid + node_index(m, i, j, k), add[0], add[1], add[2], __fmul_rn(w, mass));
    mark_block(m, dirty, i, j, k);
  }
}

// P2G of particle p (this thread) within its CTA through a tile of nodes in shared memory: every
// term rounded like the reference's, one addition per node and CTA into global memory. Every thread
// of the CTA calls it. It serves the launches whose sums have to stay as they are:
// kCoupled: with the penalty coupling folded in (_compute_coupling_forces_kernel,
// fsi/coupling.py:332-406), for launches of few particles only, where one launch less counts. The
// particle's coupling force is formed first (it is P2G's dt f term), and the fluid reaction and solid
// fraction are spread into fa->accum beside the grid scatter.
// Its loop of 27 paced steps also fixes the order in which CTAs reach a node in practice: over 47
// pairs of equal three-step runs of the 4,096-particle smoke scene the lattices were the same bit
// for bit, against 15 pairs that differ when the coupling is a kernel of its own, and 3 to 14 of
// 23 with P2G in runs here (which takes 12 to 15 us for this launch's 27).
// Not kCoupled: beside 16-bit lattices (scatter_in_runs).
// kExtTile: the tile is the caller's shared memory `ext` (4 x kTileCap floats).
template <bool kCoupled, bool kExtTile = false>
__device__ __forceinline__ void p2g_tile_body(const Mpm& m, const PView& P,
                                              float4* __restrict__ grid,
                                              uint8_t* __restrict__ dirty, int p,
                                              const ForceArgs* fa, float (*ext)[kTileCap] = nullptr) {
  __shared__ float own[kExtTile ? 1 : 4][kExtTile ? 1 : kTileCap];
  float (*tile)[kTileCap] = kExtTile ? ext : reinterpret_cast<float (*)[kTileCap]>(own);
  __shared__ int sh[8];
  const long long cap = m.cap;
  const bool act = p < m.n && P.active[p] != 0;

  int base[3] = {0, 0, 0};
  float fx[3] = {0.f, 0.f, 0.f};
  float affine[9], mv[3], dtf[3], mass = 0.f;
  // coupling: in-grid fluid stencil nodes (bit 9i + 3j + k), valid weight, force, volume
  uint32_t usable = 0;
  float valid = 0.f, pf[3] = {0.f, 0.f, 0.f}, vp = 0.f;
  if (kCoupled) {
    bool partial = false, clipped = false, unsupported = false;
    if (act) {
      int cb[3];
      float cw[3][3];
      if (!coupling_particle<false>(*fa, p, cb, cw, usable, valid, pf, partial, clipped,
                                    unsupported)) {
        usable = 0;
        pf[0] = pf[1] = pf[2] = 0.f;
      }
      vp = P.vol[p];
    } else if (p < m.n) {
      P.fp[p] = 0.f; P.fp[cap + p] = 0.f; P.fp[2 * cap + p] = 0.f;
    }
    warp_count(&fa->cnt->unsupported, unsupported);
    warp_count(&fa->cnt->partial, partial);
    warp_count(&fa->cnt->clipped, clipped);
  }
  if (act) {
    float x[3];
    load_particle_x(P, cap, p, x);
    base_fx(m, x, base, fx);
    p2g_stress_affine(m, P, p, affine, mass);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mv[a] = __fmul_rn(mass, P.v[a * cap + p]);
      dtf[a] = __fmul_rn(m.dt, kCoupled ? pf[a] : P.fp[a * cap + p]);
    }
  }

  Box box;
  if (!cta_box(m, act, base, box, sh)) return;
  const bool use_tile = box.vol <= kTileCap;
  if (use_tile) {
    for (int t = threadIdx.x; t < box.vol; t += blockDim.x) {
      tile[0][t] = 0.f; tile[1][t] = 0.f; tile[2][t] = 0.f; tile[3][t] = 0.f;
    }
    __syncthreads();
  }

  if (act) {
    // Per-axis stencil terms, once per particle: weights, offsets (i - fx) dx, in-grid tests
    // and the node's place in the tile (or grid). Odd lanes walk the stencil backwards (their
    // axis terms are stored reversed), so the two particles of a sub-cell pair, which share a
    // base cell, add into different nodes at each step.
    const bool rev = (threadIdx.x & 1) != 0;
    float wa[3][3], da[3][3];
    bool ina[3][3];
    int oa[3][3];  // axis offset of stencil step s: the node index is base + oa
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int s3 = 0; s3 < 3; ++s3) {
        const int o = rev ? 2 - s3 : s3;
        oa[a][s3] = o;
        wa[a][s3] = bspline_w(fx[a], o);
        da[a][s3] = __fmul_rn(__fsub_rn((float)o, fx[a]), m.dx);
        const int n = base[a] + o;
        ina[a][s3] = n >= 0 && n < (a == 0 ? m.nx : (a == 1 ? m.ny : m.nz));
      }
    const int st1 = use_tile ? box.ext[2] : m.nz;
    const long long st0 = use_tile ? (long long)box.ext[1] * box.ext[2] : (long long)m.ny * m.nz;
    const long long t0 = use_tile
        ? ((long long)(base[0] - box.lo[0]) * box.ext[1] + (base[1] - box.lo[1])) * box.ext[2] + (base[2] - box.lo[2])
        : ((long long)base[0] * m.ny + base[1]) * m.nz + base[2];
    const long long g0 = ((long long)base[0] * m.ny + base[1]) * m.nz + base[2];  // lattice node
    const long long gs0 = (long long)m.ny * m.nz;
#pragma unroll
    for (int si = 0; si < 3; ++si) {
      if (!ina[0][si]) continue;
#pragma unroll
      for (int sj = 0; sj < 3; ++sj) {
        if (!ina[1][sj]) continue;
        const float wxy = __fmul_rn(wa[0][si], wa[1][sj]);
        // dot3r's ((A0 d0 + A1 d1) + A2 d2): the first two terms are shared by the 3 k.
        float pa[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
          pa[a] = __fadd_rn(__fmul_rn(affine[3 * a], da[0][si]), __fmul_rn(affine[3 * a + 1], da[1][sj]));
#pragma unroll
        for (int sk = 0; sk < 3; ++sk) {
          if (!ina[2][sk]) continue;
          const float w = __fmul_rn(wxy, wa[2][sk]);
          float add[3];
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const float ad = __fadd_rn(pa[a], __fmul_rn(affine[3 * a + 2], da[2][sk]));
            add[a] = __fmul_rn(w, __fadd_rn(__fadd_rn(mv[a], ad), dtf[a]));
          }
          const float addm = __fmul_rn(w, mass);
          const long long t = t0 + oa[0][si] * st0 + oa[1][sj] * st1 + oa[2][sk];
          if (kCoupled && (usable >> (9 * oa[0][si] + 3 * oa[1][sj] + oa[2][sk])) & 1u) {
            float4 c = coupling_spread_terms(fa->c, w, valid, pf, vp);
            if (!fa->c.build_fraction) c.w = 0.f;
            red_add_v4(fa->accum + g0 + oa[0][si] * gs0 + oa[1][sj] * m.nz + oa[2][sk],
                       c.x, c.y, c.z, c.w);
          }
          if (use_tile) {
            atomicAdd(&tile[0][t], add[0]);
            atomicAdd(&tile[1][t], add[1]);
            atomicAdd(&tile[2][t], add[2]);
            atomicAdd(&tile[3][t], addm);
          } else {
            red_add_v4(grid + t, add[0], add[1], add[2], addm);
            mark_block(m, dirty, base[0] + oa[0][si], base[1] + oa[1][sj], base[2] + oa[2][sk]);
          }
        }
      }
    }
  }

  if (use_tile) {
    __syncthreads();
    if (box.vol == 0) return;  // every stencil node lies outside the grid
    const int e12 = box.ext[1] * box.ext[2];
    for (int t = threadIdx.x; t < box.vol; t += blockDim.x) {
      const float a = tile[0][t], b = tile[1][t], c = tile[2][t], d = tile[3][t];
      if (a == 0.f && b == 0.f && c == 0.f && d == 0.f) continue;
      const int ti = t / e12, r = t - ti * e12, tj = r / box.ext[2], tk = r - tj * box.ext[2];
      red_add_v4(grid + node_index(m, box.lo[0] + ti, box.lo[1] + tj, box.lo[2] + tk), a, b, c, d);
    }
    // Mark the 4^3 blocks overlapped by the box.
    const int b0[3] = {box.lo[0] >> 2, box.lo[1] >> 2, box.lo[2] >> 2};
    const int b1[3] = {(box.lo[0] + box.ext[0] - 1) >> 2, (box.lo[1] + box.ext[1] - 1) >> 2,
                       (box.lo[2] + box.ext[2] - 1) >> 2};
    const int nbx = b1[0] - b0[0] + 1, nby = b1[1] - b0[1] + 1, nbz = b1[2] - b0[2] + 1;
    for (int t = threadIdx.x; t < nbx * nby * nbz; t += blockDim.x) {
      const int bi = b0[0] + t / (nby * nbz), bj = b0[1] + (t / nbz) % nby, bk = b0[2] + t % nbz;
      dirty[((long long)bi * m.nby + bj) * m.nbz + bk] = 1;
    }
  }
}

// Grid update of one node (mpm3d.py:268-288): v = p/m + dt g, then per-axis
// walls within boundary_width: outward velocity becomes -damping * v.
__device__ __forceinline__ void grid_op(const Mpm& m, float4 node, int i, int j, int k, float v[3]) {
  v[0] = node.x; v[1] = node.y; v[2] = node.z;
  if (!(node.w > 0.f)) return;
#pragma unroll
  for (int a = 0; a < 3; ++a) v[a] = __fdiv_rn(v[a], node.w);
#pragma unroll
  for (int a = 0; a < 3; ++a) v[a] = __fadd_rn(v[a], __fmul_rn(m.dt, m.g[a]));
  const int idx[3] = {i, j, k};
  const int n[3] = {m.nx, m.ny, m.nz};
  const float nd = -m.damping;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (idx[a] < m.bw && v[a] < 0.f) v[a] = __fmul_rn(nd, v[a]);
    if (idx[a] >= n[a] - m.bw && v[a] > 0.f) v[a] = __fmul_rn(nd, v[a]);
  }
}

// G2P of particle p from grid velocities: v and the APIC C in the reference's node order, then
// advection and clamp. row(i, j, in)(k, v): the velocity v of node k of the stencil row (i, j), whose
// nodes lie in the grid where in[k]. kInside: the whole stencil lies in the grid.
template <bool kInside, class Row>
__device__ __forceinline__ void g2p_gather(const Mpm& m, const PView& P, int p, const int base[3],
                                           const float fx[3], Row row) {
  const long long cap = m.cap;
  float nv[3] = {0.f, 0.f, 0.f};
  float nc[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float four_inv_dx = __fmul_rn(4.f, m.inv_dx);
  // Per-axis stencil terms, once per particle; the sums run in the reference's node order.
  float wa[3][3];
  bool ina[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      wa[a][o] = bspline_w(fx[a], o);
      const int n = base[a] + o;
      ina[a][o] = kInside || (n >= 0 && n < (a == 0 ? m.nx : (a == 1 ? m.ny : m.nz)));
    }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (!ina[0][i]) continue;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (!ina[1][j]) continue;
      const float wxy = __fmul_rn(wa[0][i], wa[1][j]);
      auto node = row(i, j, ina[2]);
      // Node offsets made again for each row: nine of them held through the gather spill.
      float f[3] = {fx[0], fx[1], fx[2]};
      asm volatile("" : "+f"(f[0]), "+f"(f[1]), "+f"(f[2]));
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (!ina[2][k]) continue;
        const float w = __fmul_rn(wxy, wa[2][k]);
        float gv[3];
        node(k, gv);
        const float dpos[3] = {__fsub_rn((float)i, f[0]), __fsub_rn((float)j, f[1]),
                               __fsub_rn((float)k, f[2])};
#pragma unroll
        for (int a = 0; a < 3; ++a) nv[a] = __fadd_rn(nv[a], __fmul_rn(w, gv[a]));
        const float s = __fmul_rn(four_inv_dx, w);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b)
            nc[3 * a + b] = __fadd_rn(nc[3 * a + b], __fmul_rn(s, __fmul_rn(gv[a], dpos[b])));
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) P.v[a * cap + p] = nv[a];
#pragma unroll
  for (int i = 0; i < 9; ++i) P.C[i * cap + p] = m.apic ? nc[i] : 0.f;
  float x[3];  // read again: not held in registers through the gather
  load_particle_x(P, cap, p, x);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float xa = __fadd_rn(x[a], __fmul_rn(m.dt, nv[a]));
    xa = fminf(fmaxf(xa, m.lower), m.upper[a]);
    P.x[a * cap + p] = xa;
  }
}

// Grid update + G2P of particle p (this thread) within its CTA; every thread calls it.
// Bound by issue: 945 of about 1,500 instructions a warp are the 27 nodes' rounded products and
// sums, at 71 % of the issue slots; the rest stages the box, with some ten shared-memory wavefronts
// a node less than a gather straight from the grid (16 a load: the eight particles of a cell read
// four lines). 2,097,152 particles: 144 us with the tile and the grid behind one test per node,
// quotients by integer division and boxes held through the gather; 109 as it is. Velocities made
// by a pass of their own over the dirty blocks gave 105 + 10.
// A CTA that ends one body and begins the next has a box between the two that does not fit; it
// stages two boxes instead. Gathering such a CTA straight from the grid, 27 grid updates a particle
// in a row, took 12 us, longer than the whole launch of a few bodies (now 5).
// kExtTile: the tile is the caller's shared memory `ext` (3 x kTileCap floats) instead of a
// static array of its own.
template <bool kExtTile = false>
__device__ __forceinline__ void g2p_body(const Mpm& m, const PView& P,
                                         const float4* FSI_LAUNCH_RO grid, int p,
                                         float (*ext)[kTileCap] = nullptr) {
  __shared__ float own[kExtTile ? 1 : 3][kExtTile ? 1 : kTileCap];
  float (*tile)[kTileCap] = kExtTile ? ext : reinterpret_cast<float (*)[kTileCap]>(own);
  __shared__ StageScratch scratch;
  bool act = false;
  int base[3] = {0, 0, 0};
  float fx[3] = {0.f, 0.f, 0.f};
  if (p < m.n) {
    float x[3];  // beside the flag, not after it
    load_particle_x(P, m.cap, p, x);
    act = P.active[p] != 0;
    if (act) base_fx(m, x, base, fx);
  }
  const Staged st = stage_stencils(m, act, base, tile, scratch, [&](int i, int j, int k, float v[3]) {
    grid_op(m, grid[node_index(m, i, j, k)], i, j, k, v);
  });
  if (!act) return;
  if (st.ok) {
    auto staged = [&](int i, int j, const bool*) { return [&st, i, j](int k, float v[3]) { st(i, j, k, v); }; };
    if (stencil_inside(m, base))
      g2p_gather<true>(m, P, p, base, fx, staged);
    else
      g2p_gather<false>(m, P, p, base, fx, staged);
  } else {
    // The three nodes of a row are loaded together: one node after another, the 27 latencies of a
    // single such CTA outlast a small launch.
    const long long t0 = ((long long)base[0] * m.ny + base[1]) * m.nz + base[2];
    g2p_gather<false>(m, P, p, base, fx, [&](int i, int j, const bool in[3]) {
      const long long t = t0 + (long long)i * m.ny * m.nz + (long long)j * m.nz;
      struct { float4 n[3]; } r;
#pragma unroll
      for (int k = 0; k < 3; ++k) r.n[k] = in[k] ? grid[t + k] : make_float4(0.f, 0.f, 0.f, 0.f);
      return [&m, &base, r, i, j](int k, float v[3]) {
        grid_op(m, r.n[k], base[0] + i, base[1] + j, base[2] + k, v);
      };
    });
  }
}

// Inputs of coupling_particle loaded before the staging, so that its round trips to memory cover
// theirs.
struct CouplingInputs : Staged {
  static constexpr bool kStages = true;
  static constexpr int kBatch = 3;
  float xs[3], vs[3], ms, vl;
  uint32_t fl;
  __device__ __forceinline__ float x(const ForceArgs&, int, int ax) const { return xs[ax]; }
  __device__ __forceinline__ float v(const ForceArgs&, int, int ax) const { return vs[ax]; }
  __device__ __forceinline__ float mass(const ForceArgs&, int) const { return ms; }
  __device__ __forceinline__ float vol(const ForceArgs&, int) const { return vl; }
  __device__ __forceinline__ uint32_t flag(const ForceArgs&, long long) const { return fl; }
};

// coupling_forces_body with the lattice velocities of the CTA's stencils staged in shared memory;
// every thread calls it. tile: 3 x kTileCap floats of shared memory.
// Read directly, each of the 27 loads of a warp takes 16 wavefronts (as in g2p_body) and the warps
// wait on them: 88 us for 502,304 particles, 79 staged. What is left is the spread's 27 vector
// reductions a particle (58 us without them) and the issue of some 2,000 instructions a
// warp. Summing the reductions in runs first took the kernel without staging from 86 to 65 us; it was
// tried beside FP16 lattices, which amplify another order of that sum, and not yet beside FP32 alone.
__device__ __forceinline__ void coupling_staged_body(const ForceArgs& a, int p, float (*tile)[kTileCap],
                                                     StageScratch& scratch) {
  CouplingInputs in;
  bool act = false;
  in.ms = in.vl = 0.f;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) in.xs[ax] = in.vs[ax] = 0.f;
  if (p < a.n) {  // together, whether active or not
    act = a.active[p] != 0;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) { in.xs[ax] = a.x[ax * a.cap + p]; in.vs[ax] = a.v[ax * a.cap + p]; }
    in.ms = a.mass[p];
    in.vl = a.vol[p];
  }
  int base[3] = {0, 0, 0};
  float fx[3];
  if (act) stencil_base(a.c.inv_dx, in.xs, base, fx);
  in.fl = 0;
  if (act && stencil_inside(a.g, base))
    in.fl = a.flags[((long long)(base[0] + 1) * a.g.ny + base[1] + 1) * a.g.nz + base[2] + 1];
  static_cast<Staged&>(in) =
      stage_stencils(a.g, act, base, tile, scratch, [&](int i, int j, int k, float v[3]) {
        const float4 u = a.macro[((long long)i * a.g.ny + j) * a.g.nz + k];
        v[0] = u.x; v[1] = u.y; v[2] = u.z;
      });
  coupling_forces_body<false>(a, p, in);
}

// The dirty ones of the 4^3 node blocks [b0, b0 + kBlock) (each of the CTA's kBlock threads looks
// at one), listed in shared memory by their first node, so that the whole CTA works on them:
// a body's blocks lie together.
struct DirtyList {
  int n;
  int3 first[kBlock];
};

__device__ __forceinline__ void list_dirty(const Mpm& m, const uint8_t* dirty, long long b, DirtyList& l) {
  __syncthreads();  // a previous list is no longer read
  if (threadIdx.x == 0) l.n = 0;
  __syncthreads();
  const bool d = b < (long long)m.nbx * m.nby * m.nbz && dirty[b] != 0;
  const unsigned mask = __ballot_sync(0xffffffffu, d);
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0 && mask) at = atomicAdd(&l.n, __popc(mask));
  at = __shfl_sync(0xffffffffu, at, 0) + __popc(mask & ((1u << lane) - 1u));
  if (d) {
    const int bi = (int)(b / ((long long)m.nby * m.nbz)), r = (int)(b - (long long)bi * m.nby * m.nbz);
    const int bj = r / m.nbz, bk = r - bj * m.nbz;
    l.first[at] = make_int3(4 * bi, 4 * bj, 4 * bk);
  }
  __syncthreads();
}

// Node e of the list: its coordinates, and whether it lies in the grid.
__device__ __forceinline__ bool list_node(const Mpm& m, const DirtyList& l, int e, int& i, int& j, int& k) {
  if (e >= 64 * l.n) return false;
  const int3 f = l.first[e >> 6];
  i = f.x + ((e >> 4) & 3); j = f.y + ((e >> 2) & 3); k = f.z + (e & 3);
  return i < m.nx && j < m.ny && k < m.nz;
}

// Zeroes the dirty blocks and their flags.
__device__ __forceinline__ void clear_dirty_body(const Mpm& m, float4* __restrict__ grid,
                                                 uint8_t* __restrict__ dirty, long long b, DirtyList& l) {
  list_dirty(m, dirty, b, l);
  for (int e = threadIdx.x; e < 64 * l.n; e += kBlock) {
    int i, j, k;
    if (list_node(m, l, e, i, j, k)) grid[node_index(m, i, j, k)] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (b < (long long)m.nbx * m.nby * m.nbz && dirty[b] != 0) dirty[b] = 0;
}

// Host-side validation of a solver descriptor and its particle arrays.
int make_mpm(const fsi_mpm_desc* d, const fsi_particles* p, Mpm& m, PView& v) {
  FSI_REQUIRE(d && p, "NULL descriptor");
  FSI_REQUIRE(d->nx > 4 && d->ny > 4 && d->nz > 4, "grid %dx%dx%d too small", d->nx, d->ny, d->nz);
  FSI_REQUIRE(d->num_particles >= 0 && d->num_particles <= p->capacity,
              "num_particles %d outside [0, capacity %lld]", d->num_particles,
              (long long)p->capacity);
  FSI_REQUIRE(p->x && p->v && p->C && p->F && p->mass && p->volume && p->active && p->force,
              "NULL particle array");
  m.nx = d->nx; m.ny = d->ny; m.nz = d->nz;
  m.n = d->num_particles;
  m.dt = d->dt; m.dx = d->dx; m.inv_dx = d->inv_dx; m.mu = d->mu; m.lam = d->lam;
  for (int a = 0; a < 3; ++a) { m.g[a] = d->gravity[a]; m.upper[a] = d->clamp_upper[a]; }
  m.damping = d->boundary_damping; m.bw = d->boundary_width; m.apic = d->apic;
  m.lower = d->clamp_lower;
  m.cap = p->capacity;
  m.nbx = (d->nx + 3) / 4; m.nby = (d->ny + 3) / 4; m.nbz = (d->nz + 3) / 4;
  FSI_REQUIRE(d->material == FSI_MATERIAL_FIXED_COROTATED || d->material == FSI_MATERIAL_NEO_HOOKEAN,
              "unknown material %d", d->material);
  FSI_REQUIRE((p->mu == nullptr) == (p->lam == nullptr), "per-particle mu and lam go together");
  m.material = d->material;
  FSI_REQUIRE(d->launch_threads == 0 || d->launch_threads == 128 || d->launch_threads == 256 ||
                  d->launch_threads == 512,
              "launch_threads %d is not 0, 128, 256 or 512", d->launch_threads);
  FSI_REQUIRE(d->coupling_fold >= 0 && d->coupling_fold <= 3, "coupling_fold %d outside 0..3",
              d->coupling_fold);
  m.threads = d->launch_threads ? d->launch_threads : kBlock;
  m.fold = d->coupling_fold;
  v.x = p->x; v.v = p->v; v.C = p->C; v.F = p->F; v.mass = p->mass; v.vol = p->volume;
  v.active = p->active; v.fp = p->force; v.mu = p->mu; v.lam = p->lam;
  return FSI_OK;
}

}  // namespace
}  // namespace fsi
