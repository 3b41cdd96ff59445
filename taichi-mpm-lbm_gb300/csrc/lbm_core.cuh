// Lattice Boltzmann building blocks shared by the single-lattice kernels (lbm.cu) and the
// batched kernels (batch.cu): geometry, storage forms, macroscopic fields, the MRT
// collision in the exact and fast forms, and the fused AA-pattern step of a thread's cells.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include "fsi_common.cuh"
#include "lbm_formulas.cuh"
#include "lbm_vec.cuh"

namespace fsi {
namespace {


struct LbmGeom {
  int nx, ny, nz;
  long long n;  // cells
};

__host__ LbmGeom geom_of(const fsi_lbm_desc* d) {
  return LbmGeom{d->nx, d->ny, d->nz, (long long)d->nx * d->ny * d->nz};
}

// Launch shape of the cell kernels: x = z (contiguous, coalesced), y = y rows, z = x planes,
// so a thread knows (i, j, k) without integer division.
struct CellLaunch {
  dim3 grid, block;
};

CellLaunch cell_launch(const LbmGeom& g) {
  int bz = ((g.nz + 31) / 32) * 32;
  if (bz > kBlock) bz = kBlock;
  int by = kBlock / bz;
  if (by > g.ny) by = g.ny;
  return CellLaunch{dim3((g.nz + bz - 1) / bz, (g.ny + by - 1) / by, g.nx), dim3(bz, by, 1)};
}

// Signed 32-bit offsets from a cell to its +-1 neighbours on each axis, periodic wrap included
// (lbm3d.py:335-350). A neighbour index is then one three-operand add.
struct Deltas {
  uint32_t c;
  int xp, xm, yp, ym, zp, zm;
  __device__ __forceinline__ Deltas() {}
  __device__ __forceinline__ Deltas(const LbmGeom& g, int i, int j, int k) {
    const int nyz = g.ny * g.nz;
    c = (uint32_t)((i * g.ny + j) * g.nz + k);
    xp = i == g.nx - 1 ? -(g.nx - 1) * nyz : nyz;
    xm = i == 0 ? (g.nx - 1) * nyz : -nyz;
    yp = j == g.ny - 1 ? -(g.ny - 1) * g.nz : g.nz;
    ym = j == 0 ? (g.ny - 1) * g.nz : -g.nz;
    zp = k == g.nz - 1 ? -(g.nz - 1) : 1;
    zm = k == 0 ? g.nz - 1 : -1;
  }
  // Index of x + s * e_q.
  __device__ __forceinline__ uint32_t nb(int q, int s) const {
    const int dx = s * ex(q), dy = s * ey(q), dz = s * ez(q);
    const int ox = dx > 0 ? xp : (dx < 0 ? xm : 0);
    const int oy = dy > 0 ? yp : (dy < 0 ? ym : 0);
    const int oz = dz > 0 ? zp : (dz < 0 ? zm : 0);
    return c + (uint32_t)(ox + oy + oz);
  }
};

// Flag bits of the 8 corner neighbours x + (+-1, +-1, +-1) of the cell of d (periodic wrap),
// from the 0/1 solid mask.
__device__ __forceinline__ uint32_t corner_flag_bits(const int32_t* __restrict__ solid,
                                                     const Deltas& d) {
  uint32_t f = 0;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t nb = d.c + (uint32_t)((a ? d.xp : d.xm) + (b ? d.yp : d.ym) + (c ? d.zp : d.zm));
        if (solid[nb] != 0) f |= 1u << (kFlagCornerShift + 4 * a + 2 * b + c);
      }
  return f;
}

// ------------------------------------------------------------- storage forms
// ld(p, i, s) returns population i as float given its rest-equilibrium shift s = w_q rho0;
// st(p, i, v, s) stores population value v.
template <int kStore>
struct Store;

template <>
struct Store<FSI_STORAGE_F32> {
  using T = float;
  static __device__ __forceinline__ float ld(const T* p, uint32_t i, float) { return p[i]; }
  static __device__ __forceinline__ void st(T* p, uint32_t i, float v, float) { p[i] = v; }
  static __device__ __forceinline__ float2 ld2(const T* p, uint32_t i0, uint32_t i1, float) {
    return make_float2(p[i0], p[i1]);
  }
  static __device__ __forceinline__ void st2(T* p, uint32_t i0, uint32_t i1, float2 v, float) {
    p[i0] = v.x;
    p[i1] = v.y;
  }
  // Slots i and i + 1, i even, in one access.
  static __device__ __forceinline__ float2 ldp(const T* p, uint32_t i, float) {
    return *reinterpret_cast<const float2*>(p + i);
  }
  static __device__ __forceinline__ void stp(T* p, uint32_t i, float2 v, float) {
    *reinterpret_cast<float2*>(p + i) = v;
  }
};

constexpr float kF16Scale = 4096.0f;  // deviations of order 1e-8..1e-1 map into FP16's normal range

template <>
struct Store<FSI_STORAGE_F16> {
  using T = __half;
  static __device__ __forceinline__ float ld(const T* p, uint32_t i, float s) {
    return fmaf(__half2float(p[i]), 1.0f / kF16Scale, s);
  }
  static __device__ __forceinline__ void st(T* p, uint32_t i, float v, float s) {
    p[i] = __float2half_rn((v - s) * kF16Scale);
  }
  // Two values at once: one packed conversion and one packed fma / sub+mul per pair.
  static __device__ __forceinline__ float2 unpack(__half2 h, float s) {
    return vfma(__half22float2(h), make_float2(1.0f / kF16Scale, 1.0f / kF16Scale), make_float2(s, s));
  }
  static __device__ __forceinline__ __half2 pack(float2 v, float s) {
    return __float22half2_rn(vmul(vsub(v, s), kF16Scale));
  }
  static __device__ __forceinline__ float2 ld2(const T* p, uint32_t i0, uint32_t i1, float s) {
    return unpack(__halves2half2(p[i0], p[i1]), s);
  }
  static __device__ __forceinline__ void st2(T* p, uint32_t i0, uint32_t i1, float2 v, float s) {
    const __half2 h = pack(v, s);
    p[i0] = __low2half(h);
    p[i1] = __high2half(h);
  }
  static __device__ __forceinline__ float2 ldp(const T* p, uint32_t i, float s) {
    return unpack(*reinterpret_cast<const __half2*>(p + i), s);
  }
  static __device__ __forceinline__ void stp(T* p, uint32_t i, float2 v, float s) {
    *reinterpret_cast<__half2*>(p + i) = pack(v, s);
  }
};

template <>
struct Store<FSI_STORAGE_BF16> {
  using T = __nv_bfloat16;
  static __device__ __forceinline__ float ld(const T* p, uint32_t i, float s) {
    return __bfloat162float(p[i]) + s;
  }
  static __device__ __forceinline__ void st(T* p, uint32_t i, float v, float s) {
    p[i] = __float2bfloat16_rn(v - s);
  }
  static __device__ __forceinline__ float2 ld2(const T* p, uint32_t i0, uint32_t i1, float s) {
    return vadd(__bfloat1622float2(__halves2bfloat162(p[i0], p[i1])), s);
  }
  static __device__ __forceinline__ void st2(T* p, uint32_t i0, uint32_t i1, float2 v, float s) {
    const __nv_bfloat162 h = __float22bfloat162_rn(vsub(v, s));
    p[i0] = __low2bfloat16(h);
    p[i1] = __high2bfloat16(h);
  }
  static __device__ __forceinline__ float2 ldp(const T* p, uint32_t i, float s) {
    return vadd(__bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + i)), s);
  }
  static __device__ __forceinline__ void stp(T* p, uint32_t i, float2 v, float s) {
    *reinterpret_cast<__nv_bfloat162*>(p + i) = __float22bfloat162_rn(vsub(v, s));
  }
};

// The 19 storage shifts w_q rho0 by their three values.
struct Shifts {
  float w0, w1, w2;
  __device__ __forceinline__ float operator[](int q) const { return q == 0 ? w0 : (q < 7 ? w1 : w2); }
};

// Post-stream F_q(x) of a fluid cell in a state of the given parity.
template <int kStore>
__device__ __forceinline__ float gather32(const typename Store<kStore>::T* FSI_LAUNCH_RO pops,
                                          uint32_t n, const Deltas& d, uint32_t fl, int q,
                                          int parity, float shift) {
  if (parity == 0 || q == 0 || ((fl >> opp(q)) & 1u)) return Store<kStore>::ld(pops, q * n + d.c, shift);
  return Store<kStore>::ld(pops, opp(q) * n + d.nb(q, -1), shift);
}

// Storage index of F_q(x) in a state of the given parity (the slot a gather reads).
__device__ __forceinline__ uint32_t slot32(uint32_t n, const Deltas& d, uint32_t fl, int q,
                                           int parity) {
  if (parity == 0 || q == 0 || ((fl >> opp(q)) & 1u)) return q * n + d.c;
  return opp(q) * n + d.nb(q, -1);
}

// ---------------------------------------------------------------- macro fields
// rho and u as update_macro computes them (lbm3d.py:409-425): sequential sums
// in q order, then u = u / rho, u = u + (force * 0.5) / rho.
template <class V>
__device__ __forceinline__ void macro_of(const V (&F)[19], V gx, V gy, V gz, V& rho, V& ux, V& uy,
                                         V& uz) {
  V r = F[0];
#pragma unroll
  for (int q = 1; q < 19; ++q) r = vadd(r, F[q]);
  V x = vsub(F[1], F[2]);
  x = vadd(x, F[7]); x = vsub(x, F[8]); x = vadd(x, F[9]); x = vsub(x, F[10]);
  x = vadd(x, F[11]); x = vsub(x, F[12]); x = vadd(x, F[13]); x = vsub(x, F[14]);
  V y = vsub(F[3], F[4]);
  y = vadd(y, F[7]); y = vsub(y, F[8]); y = vsub(y, F[9]); y = vadd(y, F[10]);
  y = vadd(y, F[15]); y = vsub(y, F[16]); y = vadd(y, F[17]); y = vsub(y, F[18]);
  V z = vsub(F[5], F[6]);
  z = vadd(z, F[11]); z = vsub(z, F[12]); z = vsub(z, F[13]); z = vadd(z, F[14]);
  z = vadd(z, F[15]); z = vsub(z, F[16]); z = vsub(z, F[17]); z = vadd(z, F[18]);
  x = vdiv(x, r); y = vdiv(y, r); z = vdiv(z, r);
  x = vadd(x, vdiv(vmul(gx, 0.5f), r));
  y = vadd(y, vdiv(vmul(gy, 0.5f), r));
  z = vadd(z, vdiv(vmul(gz, 0.5f), r));
  rho = r; ux = x; uy = y; uz = z;
}

// The same quantities from the moments m = M F of mrt_forward: its rows 0, 3, 5 and 7 are
// update_macro's sums of f, e_x f, e_y f and e_z f, term for term in q order (the formula
// generator's self-check asserts it), so rho and j are the same values.
template <class V>
__device__ __forceinline__ void macro_of_moments(const V (&m)[19], V gx, V gy, V gz, V& rho,
                                                 V& ux, V& uy, V& uz) {
  const V r = m[0];
  V x = vdiv(m[3], r), y = vdiv(m[5], r), z = vdiv(m[7], r);
  x = vadd(x, vdiv(vmul(gx, 0.5f), r));
  y = vadd(y, vdiv(vmul(gy, 0.5f), r));
  z = vadd(z, vdiv(vmul(gz, 0.5f), r));
  rho = r; ux = x; uy = y; uz = z;
}

// The same quantities with fused operations and one reciprocal (fast forms).
template <class V>
__device__ __forceinline__ void macro_fast(const V (&F)[19], V gx, V gy, V gz, V& rho, V& ux,
                                           V& uy, V& uz) {
  const V P0 = vadd(F[1], F[2]), P1 = vadd(F[3], F[4]), P2 = vadd(F[5], F[6]);
  const V P3 = vadd(F[7], F[8]), P4 = vadd(F[9], F[10]), P5 = vadd(F[11], F[12]);
  const V P6 = vadd(F[13], F[14]), P7 = vadd(F[15], F[16]), P8 = vadd(F[17], F[18]);
  const V r = vadd(vadd(vadd(vadd(F[0], P0), vadd(P1, P2)), vadd(vadd(P3, P4), vadd(P5, P6))),
                   vadd(P7, P8));
  const V D3 = vsub(F[7], F[8]), D4 = vsub(F[9], F[10]), D5 = vsub(F[11], F[12]);
  const V D6 = vsub(F[13], F[14]), D7 = vsub(F[15], F[16]), D8 = vsub(F[17], F[18]);
  const V jx = vadd(vadd(vsub(F[1], F[2]), vadd(D3, D4)), vadd(D5, D6));
  const V jy = vadd(vadd(vsub(F[3], F[4]), vsub(D3, D4)), vadd(D7, D8));
  const V jz = vadd(vadd(vsub(F[5], F[6]), vsub(D5, D6)), vsub(D7, D8));
  const V inv = vrcp(r);
  rho = r;
  ux = vmul(vfma(0.5f, gx, jx), inv);
  uy = vmul(vfma(0.5f, gy, jy), inv);
  uz = vmul(vfma(0.5f, gz, jz), inv);
}

template <bool kFast, class V>
__device__ __forceinline__ void macro_any(const V (&F)[19], V gx, V gy, V gz, V& rho, V& ux,
                                          V& uy, V& uz) {
  if (kFast) macro_fast(F, gx, gy, gz, rho, ux, uy, uz);
  else macro_of(F, gx, gy, gz, rho, ux, uy, uz);
}

// Sum of the non-zero terms e_c * v_c in x, y, z order (Taichi Vector.dot with
// exact zero products dropped).
template <class V>
__device__ __forceinline__ V edot(int q, V vx, V vy, V vz) {
  V s = splat<V>(0.0f);
  bool first = true;
  if (ex(q) != 0) { s = ex(q) > 0 ? vx : vneg(vx); first = false; }
  if (ey(q) != 0) { V t = ey(q) > 0 ? vy : vneg(vy); s = first ? t : vadd(s, t); first = false; }
  if (ez(q) != 0) { V t = ez(q) > 0 ? vz : vneg(vz); s = first ? t : vadd(s, t); }
  return s;
}

// MRT collision with Guo forcing of one fluid cell (or two, V = float2) in the reference's
// order (lbm3d.py:276-333), given the moments mF = M F of its populations (mrt_forward, which
// the caller also reads rho and j from). SG[k] is the forcing weight 1 - 0.5 S[k] of the reference,
// evaluated once per launch: 0.5 S[k] is an exact scaling, so 1 - 0.5 S[k] has a single
// rounding wherever it is computed.
template <class V>
__device__ __forceinline__ void collide_cell(const V (&mF)[19], V ux, V uy, V uz, V gx, V gy, V gz,
                                             const float* __restrict__ S,
                                             const float* __restrict__ SG, V (&out)[19]) {
  // Guo source terms t_q = w_q ((e_q - u).G + (e_q.u)(e_q.G)) (lbm3d.py:276-283).
  // (e - u_c) G_c takes three values per axis, for e = -1, 0, +1.
  const V dx[3] = {vmul(vsub(-1.0f, ux), gx), vmul(vneg(ux), gx), vmul(vsub(1.0f, ux), gx)};
  const V dy[3] = {vmul(vsub(-1.0f, uy), gy), vmul(vneg(uy), gy), vmul(vsub(1.0f, uy), gy)};
  const V dz[3] = {vmul(vsub(-1.0f, uz), gz), vmul(vneg(uz), gz), vmul(vsub(1.0f, uz), gz)};
  // (e.u)(e.G) of q and of opp(q) are the same rounded product: both dot products change
  // sign together and (-x)(-y) = xy. They can differ only in the sign of an exact zero,
  // which the forcing moments g = M t then carry only into sums that are non-zero or +0.
  V t[19], b[19];
#pragma unroll
  for (int q = 0; q < 19; ++q) {
    const V a = vadd(vadd(dx[ex(q) + 1], dy[ey(q) + 1]), dz[ez(q) + 1]);
    if (q == 0) {
      t[q] = vmul(weight_of(q), a);
    } else {
      b[q] = (q & 1) ? vmul(edot(q, ux, uy, uz), edot(q, gx, gy, gz)) : b[q - 1];
      t[q] = vmul(weight_of(q), vadd(a, b[q]));
    }
  }
  V g[19], m[19];
  mrt_forward(t, g);
#pragma unroll
  for (int k = 0; k < 19; ++k) m[k] = mF[k];
  // Relaxation towards meq (lbm3d.py:285-326). S_0 = S_3 = S_5 = S_7 = 0: those
  // moments only receive the forcing term.
  const V uxx = vmul(ux, ux), uyy = vmul(uy, uy), uzz = vmul(uz, uz);
  V meq[19];
#pragma unroll
  for (int k = 0; k < 19; ++k) meq[k] = splat<V>(0.0f);
  meq[1] = vadd(vadd(uxx, uyy), uzz);
  meq[9] = vsub(vsub(vmul(vmul(2.0f, ux), ux), uyy), uzz);
  meq[11] = vsub(uyy, uzz);
  meq[13] = vmul(ux, uy);
  meq[14] = vmul(uy, uz);
  meq[15] = vmul(ux, uz);
#pragma unroll
  for (int k = 0; k < 19; ++k) {
    if (k == 0 || k == 3 || k == 5 || k == 7) {
      m[k] = vadd(m[k], g[k]);
    } else {
      const bool has_eq = (k == 1 || k == 9 || k == 11 || k == 13 || k == 14 || k == 15);
      const V d = has_eq ? vsub(m[k], meq[k]) : m[k];
      m[k] = vsub(m[k], vmul(S[k], d));
      m[k] = vadd(m[k], vmul(SG[k], g[k]));  // SG[k] = 1 - S[k]/2, rounded once
    }
  }
  mrt_inverse(m, out);
}

struct StepArgs {
  LbmGeom g;
  void* __restrict__ pops;
  float4* __restrict__ macro;
  const float* __restrict__ force;
  const float* __restrict__ force_prev;
  const uint32_t* __restrict__ flags;
  float s[19];
  float sg[19];     // 1 - s_k / 2, the weight of the forcing moment g_k (host-rounded once)
  float shift[19];  // w_q rho0, the storage offset of the deviation forms
  int write_faces;
};

// Cells per thread of the step kernel: the exact form evaluates one cell per thread in
// scalar float arithmetic; the fast forms evaluate the two cells (i, j, k) and (i, j + 1, k)
// of a thread together in packed float2 arithmetic (half the floating-point instructions).
// The exact form stays scalar because the assembler's optimisation of packed f32x2 code
// was observed to change rounding (a single-use product merged into the following
// subtraction), which would break bit-identity with the reference's float32 operations.
template <bool kFast>
struct StepLanes {
  static constexpr int n = kFast ? 2 : 1;
  using V = typename std::conditional<kFast, float2, float>::type;
};

constexpr int kStepBlock = 128;

// Minimum resident 128-thread blocks per SM of the step kernel (caps its registers at
// 65536 / (128 * n)). From a sweep on the 256^3 channel with spheres, us per step with rho and u
// read / recomputed:
//   exact, even   640/610 at 5, 617/610 at 6, 615/608 at 7, 613/595 at 8
//          odd    672/685 at 6, 644/649 at 7, 624/639 at 8, 607/639 at 9
//   FP16,  even   443/408 at 4, 394/408 at 5, 363/373 at 6, 361/357 at 7
//          odd    515/539 at 4, 474/473 at 5, 531/476 at 6, 556/451 at 7
//   BF16 within 5 % of FP16; fast FP32, even 452/473 at 6 and 472/474 at 5, odd 551/558 at 4,
//   543/514 at 5, 637/548 at 6.
template <int kStore, bool kFast, bool kOdd, bool kRecompute>
constexpr int step_min_blocks() {
  if (!kFast) return kOdd ? 9 : 8;
  if (kStore != FSI_STORAGE_F32) return kOdd && !kRecompute ? 5 : 7;
  return kOdd ? 5 : 6;
}

// Launch shape of the step kernel: x = z (contiguous), y = groups of `lanes` rows, z = x planes.
CellLaunch step_launch(const LbmGeom& g, int lanes) {
  int bz = ((g.nz + 31) / 32) * 32;
  if (bz > kStepBlock) bz = kStepBlock;
  const int rows = (g.ny + lanes - 1) / lanes;
  int by = kStepBlock / bz;
  if (by > rows) by = rows;
  return CellLaunch{dim3((g.nz + bz - 1) / bz, (rows + by - 1) / by, g.nx), dim3(bz, by, 1)};
}

// Storage index that the odd step reads F_q(x) from, and that it writes f*_q(x) to.
__device__ __forceinline__ uint32_t odd_src(const Deltas& d, uint32_t fl, int q, uint32_t n) {
  return ((fl >> opp(q)) & 1u) ? q * n + d.c : opp(q) * n + d.nb(q, -1);
}
__device__ __forceinline__ uint32_t odd_dst(const Deltas& d, uint32_t fl, int q, uint32_t n) {
  return ((fl >> q) & 1u) ? opp(q) * n + d.c : q * n + d.nb(q, +1);
}

// One step of the cells (ci[l], cj[l], ck[l]) of the lanes of one thread; a lane with
// has[l] false is treated like a solid cell (read from another lane, never stored).
// Args is StepArgs (one lattice, parameters in the kernel's parameter space) or any type
// with the same members (a lattice of a batch, whose rates and shifts are pointers).
template <int kStore, bool kFast, bool kOdd, bool kRecompute, class Args>
__device__ __forceinline__ void step_cells(const Args& a,
                                           const int (&ci)[StepLanes<kFast>::n],
                                           const int (&cj)[StepLanes<kFast>::n],
                                           const int (&ck)[StepLanes<kFast>::n],
                                           const bool (&has)[StepLanes<kFast>::n]) {
  using St = Store<kStore>;
  constexpr int L = StepLanes<kFast>::n;
  using V = typename StepLanes<kFast>::V;
  using Ln = Lanes<V>;
  uint32_t fl[L];
  bool live[L];
  bool any = false;
#pragma unroll
  for (int l = 0; l < L; ++l) {
    fl[l] = has[l] ? a.flags[(uint32_t)((ci[l] * a.g.ny + cj[l]) * a.g.nz + ck[l])] : kFlagSolid;
    live[l] = !(fl[l] & kFlagSolid);
    any = any || live[l];
  }
  if (!any) return;
  // A solid (or missing) lane reads the cells of the live lane and is never stored. It takes that
  // lane's coordinates here, before anything is derived from them: picked by an index chosen at
  // run time, the neighbour offsets would live in local memory.
  int i[L], j[L], k[L];
#pragma unroll
  for (int l = 0; l < L; ++l) { i[l] = ci[l]; j[l] = cj[l]; k[l] = ck[l]; }
  if constexpr (L == 2) {
    const uint32_t f0 = fl[0];
    if (!live[0]) { fl[0] = fl[1]; i[0] = ci[1]; j[0] = cj[1]; k[0] = ck[1]; }
    if (!live[1]) { fl[1] = f0; i[1] = ci[0]; j[1] = cj[0]; k[1] = ck[0]; }
  }
  Deltas d[L];
#pragma unroll
  for (int l = 0; l < L; ++l) d[l] = Deltas(a.g, i[l], j[l], k[l]);
  const uint32_t n = (uint32_t)a.g.n;
  typename St::T* __restrict__ pops = reinterpret_cast<typename St::T*>(a.pops);

  V F[19];
#pragma unroll
  for (int q = 0; q < 19; ++q) {
    uint32_t sl[L];
#pragma unroll
    for (int l = 0; l < L; ++l) {
      // F_q(x) = f*_q(x - e_q) in slot opp(q) there, or f*_opp(q)(x) in slot q here when
      // x - e_q is solid (half-way bounce-back).
      sl[l] = (!kOdd || q == 0) ? q * n + d[l].c : odd_src(d[l], fl[l], q, n);
    }
    if constexpr (L == 2) {
      F[q] = St::ld2(pops, sl[0], sl[1], a.shift[q]);
    } else {
      F[q] = St::ld(pops, sl[0], a.shift[q]);
    }
  }
  // Exact form: the moments M F, from which both rho, j and the collision start.
  V mF[19];
  if (!kFast) mrt_forward(F, mF);

  uint32_t c[L];
#pragma unroll
  for (int l = 0; l < L; ++l) c[l] = d[l].c;
  V gx, gy, gz, rho, ux, uy, uz;
#pragma unroll
  for (int l = 0; l < L; ++l) {
    Ln::set(gx, l, a.force[c[l]]);
    Ln::set(gy, l, a.force[n + c[l]]);
    Ln::set(gz, l, a.force[2 * n + c[l]]);
  }
  if (kRecompute) {
    V px, py, pz;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      Ln::set(px, l, a.force_prev[c[l]]);
      Ln::set(py, l, a.force_prev[n + c[l]]);
      Ln::set(pz, l, a.force_prev[2 * n + c[l]]);
    }
    if (kFast) macro_fast(F, px, py, pz, rho, ux, uy, uz);
    else macro_of_moments(mF, px, py, pz, rho, ux, uy, uz);
    if (a.write_faces) {
#pragma unroll
      for (int l = 0; l < L; ++l)
        if (live[l] && (fl[l] & (kFlagFaceLeft | kFlagFaceRight)))
          a.macro[d[l].c] = make_float4(Ln::get(ux, l), Ln::get(uy, l), Ln::get(uz, l),
                                        Ln::get(rho, l));
    }
  } else {
#pragma unroll
    for (int l = 0; l < L; ++l) {
      const float4 m = a.macro[c[l]];
      Ln::set(ux, l, m.x); Ln::set(uy, l, m.y); Ln::set(uz, l, m.z); Ln::set(rho, l, m.w);
    }
  }

  V out[19];
  if (kFast) mrt_collide_fast(F, rho, ux, uy, uz, gx, gy, gz, a.s, out);
  else collide_cell(mF, ux, uy, uz, gx, gy, gz, a.s, a.sg, out);

  // The stores address what the loads did. Seen as the same expressions, up to 19 64-bit
  // addresses per lane and the neighbour offsets would be kept from one to the other across the
  // collision, in registers that the loads in flight need; coordinates that only now become
  // known make them again. (Exact form at 256^3: even steps 641 -> 608 us, 771 -> 615 with rho and
  // u read. Its odd step with rho and u recomputed is short of issue slots instead: 639 us as it
  // is, 647 with the offsets made again.)
  if constexpr (kFast || !kOdd || !kRecompute) {
#pragma unroll
    for (int l = 0; l < L; ++l) {
      asm volatile("" : "+r"(j[l]), "+r"(k[l]));
      d[l] = Deltas(a.g, i[l], j[l], k[l]);
    }
  }
#pragma unroll
  for (int q = 0; q < 19; ++q) {
    // f*_q goes to slot opp(q) of this cell (even step, or odd-step bounce-back) or to slot q
    // of x + e_q (odd step). w_q = w_opp(q), so either slot's storage shift is shift[q].
    uint32_t t[L];
#pragma unroll
    for (int l = 0; l < L; ++l)
      t[l] = (!kOdd || q == 0) ? opp(q) * n + d[l].c : odd_dst(d[l], fl[l], q, n);
    if constexpr (L == 2) {
      if (live[0] && live[1]) {
        St::st2(pops, t[0], t[1], out[q], a.shift[q]);
        continue;
      }
    }
#pragma unroll
    for (int l = 0; l < L; ++l)
      if (live[l]) St::st(pops, t[l], Ln::get(out[q], l), a.shift[q]);
  }
}

template <int kStore, bool kFast, bool kOdd, bool kRecompute>
__global__ void __launch_bounds__(kStepBlock, (step_min_blocks<kStore, kFast, kOdd, kRecompute>()))
    lbm_step_kernel(StepArgs a) {
  constexpr int L = StepLanes<kFast>::n;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = L * (blockIdx.y * blockDim.y + threadIdx.y);
  const int i = blockIdx.z;
  if (k >= a.g.nz || j >= a.g.ny) return;
  int ci[L], cj[L], ck[L];
  bool has[L];
#pragma unroll
  for (int l = 0; l < L; ++l) {
    ci[l] = i; cj[l] = j + l; ck[l] = k;
    has[l] = j + l < a.g.ny;
  }
  step_cells<kStore, kFast, kOdd, kRecompute, StepArgs>(a, ci, cj, ck, has);
}

// Minimum resident blocks per SM of the even step by pairs. us per step at 256^3 with rho and u
// read / recomputed, by blocks: FP16 331/322 at 5, 334/316 at 6, 312/314 at 7, 312/322 at 8; BF16
// 318/316, 291/308, 284/317, 294/316; fast FP32 430/405, 428/423, 430/419, 446/497.
template <int kStore, bool kRecompute>
constexpr int even_min_blocks() {
  if (kStore != FSI_STORAGE_F32) return 7;
  return kRecompute ? 5 : 6;
}

// An even step of the cells c and c + 1, c even (as is the lattice's cell count), in the fast form.
// An even step reads and writes a cell's own slots only, so any two neighbours in memory make a
// pair, whose populations, forces and flags move in one access each: at 256^3 FP16 312 us, against
// 358 for the two rows of step_cells with as many accesses again, 39 packings and their addresses.
// (An odd step's pairs of neighbours along z gained nothing: ten of its directions stay apart.)
template <int kStore, bool kRecompute, class Args>
__device__ __forceinline__ void step_even_pair(const Args& a, uint32_t c) {
  using St = Store<kStore>;
  const uint32_t n = (uint32_t)a.g.n;
  typename St::T* __restrict__ pops = reinterpret_cast<typename St::T*>(a.pops);
  const uint2 fl = *reinterpret_cast<const uint2*>(a.flags + c);
  const bool live0 = !(fl.x & kFlagSolid), live1 = !(fl.y & kFlagSolid);
  if (!live0 && !live1) return;
  float2 F[19];
#pragma unroll
  for (int q = 0; q < 19; ++q) F[q] = St::ldp(pops, q * n + c, a.shift[q]);
  auto pair = [&](const float* p) { return *reinterpret_cast<const float2*>(p + c); };
  const float2 gx = pair(a.force), gy = pair(a.force + n), gz = pair(a.force + 2 * n);
  float2 rho, ux, uy, uz;
  if (kRecompute) {
    macro_fast(F, pair(a.force_prev), pair(a.force_prev + n), pair(a.force_prev + 2 * n), rho, ux, uy, uz);
    if (a.write_faces) {
      constexpr uint32_t face = kFlagFaceLeft | kFlagFaceRight;
      if (live0 && (fl.x & face)) a.macro[c] = make_float4(ux.x, uy.x, uz.x, rho.x);
      if (live1 && (fl.y & face)) a.macro[c + 1] = make_float4(ux.y, uy.y, uz.y, rho.y);
    }
  } else {
    const float4 m0 = a.macro[c], m1 = a.macro[c + 1];
    ux = make_float2(m0.x, m1.x); uy = make_float2(m0.y, m1.y); uz = make_float2(m0.z, m1.z);
    rho = make_float2(m0.w, m1.w);
  }
  float2 out[19];
  mrt_collide_fast(F, rho, ux, uy, uz, gx, gy, gz, a.s, out);
  asm volatile("" : "+r"(c));  // the stores' addresses made again, as in step_cells
  if (live0 && live1) {
#pragma unroll
    for (int q = 0; q < 19; ++q) St::stp(pops, opp(q) * n + c, out[q], a.shift[q]);
  } else {  // a solid cell is never stored
    c += live0 ? 0 : 1;
#pragma unroll
    for (int q = 0; q < 19; ++q) St::st(pops, opp(q) * n + c, live0 ? out[q].x : out[q].y, a.shift[q]);
  }
}

// Whether an even step may take its cells in pairs: an even number of cells, and arrays that start
// where two values do.
inline bool even_pairs(long long n, const void* pops, const void* flags, const void* force,
                       const void* force_prev) {
  const uintptr_t at = (uintptr_t)pops | (uintptr_t)flags | (uintptr_t)force | (uintptr_t)force_prev;
  return n % 2 == 0 && (at & 7) == 0;
}

template <int kStore, bool kRecompute>
__global__ void __launch_bounds__(kStepBlock, (even_min_blocks<kStore, kRecompute>()))
    lbm_even_pair_kernel(StepArgs a) {
  const uint32_t c = 2 * (blockIdx.x * kStepBlock + threadIdx.x);
  if (c < (uint32_t)a.g.n) step_even_pair<kStore, kRecompute>(a, c);
}

// numpy float32 norm of a 3-vector: sqrt((x*x + y*y) + z*z).
__device__ __forceinline__ float norm3_ref(float x, float y, float z) {
  return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

template <int kStore>
constexpr bool macro_by_pairs(bool odd_state) {
  return kStore != FSI_STORAGE_F32 || !odd_state;
}

// update_macro of the cells c and c + 1, c even (as is the lattice's cell count), in the fast form;
// their fluid rho (0 on solid cells) and |u| in mass / vmax. In an even state both cells' slots come
// in one access each; in an odd one a thread has twice the loads in flight. 64 scenes in FP16, by
// cells 531 us: 323 in an even state, 336 in an odd one. 192x96x96 cells in FP32, by cells 32 us: 30
// and 36, so FP32 takes pairs in even states only (macro_by_pairs).
template <int kStore, bool kOddState, class S>
__device__ __forceinline__ void macro_pair(const LbmGeom& g, const typename Store<kStore>::T* FSI_LAUNCH_RO pops,
                                           const float* FSI_LAUNCH_RO force, const uint32_t* __restrict__ flags,
                                           uint32_t c, const S& shift, float rho0, float4* macro,
                                           float (&mass)[2], float (&vmax)[2]) {
  const uint32_t n = (uint32_t)g.n;
  const uint2 fl = *reinterpret_cast<const uint2*>(flags + c);
  const bool solid0 = fl.x & kFlagSolid, solid1 = fl.y & kFlagSolid;
  float2 rho = splat<float2>(rho0), ux = splat<float2>(0.f), uy = ux, uz = ux;
  if (!solid0 || !solid1) {
    float2 F[19];
    if constexpr (kOddState) {
      const uint32_t nyz = (uint32_t)(g.ny * g.nz);
      Deltas d[2];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const uint32_t i = (c + l) / nyz, r = c + l - i * nyz, j = r / (uint32_t)g.nz;
        d[l] = Deltas(g, (int)i, (int)j, (int)(r - j * g.nz));
      }
#pragma unroll
      for (int q = 0; q < 19; ++q)
        F[q] = Store<kStore>::ld2(pops, slot32(n, d[0], fl.x, q, 1), slot32(n, d[1], fl.y, q, 1), shift[q]);
    } else {
#pragma unroll
      for (int q = 0; q < 19; ++q) F[q] = Store<kStore>::ldp(pops, q * n + c, shift[q]);
    }
    auto pair = [&](const float* p) { return *reinterpret_cast<const float2*>(p + c); };
    macro_fast(F, pair(force), pair(force + n), pair(force + 2 * n), rho, ux, uy, uz);
  }
  if (solid0) { rho.x = rho0; ux.x = uy.x = uz.x = 0.f; }
  if (solid1) { rho.y = rho0; ux.y = uy.y = uz.y = 0.f; }
  macro[c] = make_float4(ux.x, uy.x, uz.x, rho.x);
  macro[c + 1] = make_float4(ux.y, uy.y, uz.y, rho.y);
  mass[0] = solid0 ? 0.f : rho.x;
  mass[1] = solid1 ? 0.f : rho.y;
  vmax[0] = norm3_ref(ux.x, uy.x, uz.x);
  vmax[1] = norm3_ref(ux.y, uy.y, uz.y);
}

__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}

// Adds this block's sums of `s` (float32 within a warp, float64 across warps) into
// sums[0..NS) and, when max_out is not NULL, raises *max_out to the block maximum of `mx`.
// Every thread of the block must call it; each instantiation owns its shared scratch.
template <int NS>
__device__ void block_accumulate(double* __restrict__ sums, const float (&s)[NS],
                                 double* __restrict__ max_out, float mx) {
  float v[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) v[i] = s[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < NS; ++i) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  __shared__ double sh[NS][kBlock / 32];
  __shared__ float shm[kBlock / 32];
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  const int nwarps = (blockDim.x * blockDim.y + 31) / 32;
  if ((t & 31) == 0) {
#pragma unroll
    for (int i = 0; i < NS; ++i) sh[i][t >> 5] = (double)v[i];
    shm[t >> 5] = mx;
  }
  __syncthreads();
  if (t == 0) {
    float m = 0.f;
    for (int w = 0; w < nwarps; ++w) m = fmaxf(m, shm[w]);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      double acc = 0.0;
      for (int w = 0; w < nwarps; ++w) acc += sh[i][w];
      atomicAdd(sums + i, acc);
    }
    if (max_out) atomic_max_nonneg(max_out, (double)m);
  }
}

}  // namespace
}  // namespace fsi
