// What the residual kernels share, templated on the arithmetic type: the tile
// layout, the line operators of quadrilaterals (D = 2) and hexahedra (D = 3) of
// order P = N - 1, the 2D faces and the RK update of a point.  The kernels are in
// quad_kernels.cuh, hex_kernels.cuh and tri_kernels.cuh.
//
// Data layout in HBM is tile-major structure-of-arrays: TW consecutive
// elements form a tile and every per-element array is stored as
//   [tile][point][component][TW]
// so one CTA reads its whole tile as one contiguous chunk and, inside it, the
// TW elements of a (point, component) pair sit in one 32- or 64-byte run.
//
// Reference: the residual is FRSolver::compute_residual (src/solver.cpp:1494-
// 1645).  Its dense operator products (src/elements.cpp:1337-1501) are applied
// here as line operators: every nonzero of oppE, oppD, oppD_fpts, oppDiv and
// oppDiv_fpts for quads and hexes lies on the line of points through a
// solution point (src/elements.cpp:592-655), and the nonzeros are summed in the
// same order as the reference's row-major products.
#pragma once

#include <cstdint>

#include "physics.cuh"

namespace zb {
namespace dev {

constexpr int TW = 8;  // elements per tile

template <int D, int N>
struct Shape
{
  static constexpr int S = (D == 2) ? N * N : N * N * N;
  static constexpr int NF = (D == 2) ? N : N * N;  // flux points per face
  static constexpr int Fp = 2 * D * NF;
  static constexpr int V = D + 2;
  static constexpr int NM = D * D + 1;  // adjugate entries + |J|
  static constexpr int NT = (D == 2) ? ((S * TW <= 128) ? 128 : 256) : 256;
};

// Prefetch `bytes` (a multiple of 16, 16-byte aligned) from global memory
// into L2 without waiting: one bulk request, no registers held
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes)
{
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

template <typename T, int N>
struct LineOpsT
{
  T Dm[N * N];  // Dm[i*N+m] = l'_{m+1}(x_i) on [-1, x, 1]
  T Em[N], Ep[N], Dbm[N], Dbp[N];
};

// T: storage type of state, traces and metrics; A: arithmetic type.
template <typename T, typename A>
struct Args
{
  const T *U;        // [tile][S][V][TW]
  const T *Ufp;      // [tile][Fp][V][TW] extrapolated state (this stage)
  T *Ufp_next;       // extrapolation of the updated state (next stage)
  const T *mets;     // [tile][S][NM][TW]: adj[d1][d2] (reference inv_jaco), |J|
  const T *fgeo;     // [tile][Fp][D+1][TW]: face unit normal (left side), own dA
  const int *nbr;    // [tile][Fp][TW]: 2*partner+slot, or -1-bc
  T *divF;           // [tile][S][V][TW] residual of this stage
  A *divF_vol;       // NS: volume part of the residual (arithmetic type: it cancels
                     // against the surface part)
  T *Fvn;            // NS: viscous normal flux at own flux points
  const double *dt_dev;  // optional: the step as computed on the device (CFL, global)
  const double *dt_ele;  // optional: per-element step [tile * TW + lane] (CFL, local)
  T *Fcom;           // NS hexahedra, LDG beta = +-1/2, optional: common flux (convective
                     // + viscous, not dA-scaled) at the flux points whose side supplies
                     // the LDG normal flux; the partner reads it from there
  T *dU_out;         // NS, optional: physical gradient [tile][D][S][V][TW] (the
                     // reference keeps it in dU_spts for diagnostics)
  // RK update fused into the last kernel of a stage
  int rk_mode;       // 0: none; 1: U = U_ini - a dt/|J| divF; 2: final combination
  int save_ini;      // stage 0: write U_ini = U before updating
  int extrap_next;   // write Ufp_next from the updated state
  int nprev;         // final stage: number of earlier divF registers
  T *Uout;           // updated state (may alias U)
  T *U_ini;          // RK start state
  T *Ucomp;          // compensated-summation remainder (final stage, nullptr = off)
  const T *divF_prev[6];
  A rk_coef[6];      // a_s (mode 1: [0]) or b_s (mode 2)
  A dt;
  int64_t ntiles;
  const A *dops;     // triangles: dense operators (TriOps layout), nullptr otherwise
  int *err;          // tensor-core kernels: set when a completion wait gave up
  Phys<A> ph;
};

// Flux point f -> normal dimension, side (-1/+1), first spt of its line and
// stride along the line (orderings of src/quads.cpp:108-148, src/hexas.cpp:148-205).
template <int D, int N>
__device__ __forceinline__ void fpt_line(int f, int &dim, int &side, int &base, int &stride)
{
  if (D == 2)
  {
    const int face = f / N, j = f % N;
    switch (face)
    {
      case 0: dim = 1; side = -1; base = j; stride = N; break;
      case 1: dim = 0; side = 1; base = N * j; stride = 1; break;
      case 2: dim = 1; side = 1; base = N - 1 - j; stride = N; break;
      default: dim = 0; side = -1; base = N * (N - 1 - j); stride = 1; break;
    }
  }
  else
  {
    constexpr int N2 = N * N;
    const int face = f / N2, r = f % N2, j = r / N, k = r % N;
    switch (face)
    {
      case 0: dim = 2; side = -1; base = k + N * j; stride = N2; break;
      case 1: dim = 2; side = 1; base = (N - 1 - k) + N * j; stride = N2; break;
      case 2: dim = 0; side = -1; base = N * k + N2 * j; stride = 1; break;
      case 3: dim = 0; side = 1; base = N * (N - 1 - k) + N2 * j; stride = 1; break;
      case 4: dim = 1; side = -1; base = (N - 1 - k) + N2 * j; stride = N; break;
      default: dim = 1; side = 1; base = k + N2 * j; stride = N; break;
    }
  }
}

// Solution point s: line coordinate along dimension d and the flux points at
// the -/+ ends of that line.
template <int D, int N>
__device__ __forceinline__ void spt_ends(int s, int d, int &i, int &fm, int &fp)
{
  if (D == 2)
  {
    const int ix = s % N, iy = s / N;
    if (d == 0) { i = ix; fm = 3 * N + (N - 1 - iy); fp = N + iy; }
    else { i = iy; fm = ix; fp = 2 * N + (N - 1 - ix); }
  }
  else
  {
    constexpr int N2 = N * N;
    const int ix = s % N, iy = (s / N) % N, iz = s / N2;
    if (d == 0) { i = ix; fm = 2 * N2 + iz * N + iy; fp = 3 * N2 + iz * N + (N - 1 - iy); }
    else if (d == 1) { i = iy; fm = 4 * N2 + iz * N + (N - 1 - ix); fp = 5 * N2 + iz * N + ix; }
    else { i = iz; fm = iy * N + ix; fp = N2 + iy * N + (N - 1 - ix); }
  }
}

template <int N>
__device__ __forceinline__ constexpr int pow_n(int d)
{
  return d == 0 ? 1 : (d == 1 ? N : N * N);
}

// Face id -> (dimension, side) for summing surface terms in flux point order.
template <int D>
__device__ __forceinline__ void face_dim_side(int face, int &dim, int &side)
{
  if (D == 2)
  {
    dim = (face == 0 || face == 2) ? 1 : 0;
    side = (face == 1 || face == 2) ? 1 : -1;
  }
  else
  {
    dim = (face < 2) ? 2 : (face < 4 ? 0 : 1);
    side = (face % 2 == 0) ? -1 : 1;
  }
}

template <typename A, int N>
__device__ __forceinline__ void load_ops(A *sops, const LineOpsT<A, N> &ops, int tid, int nth)
{
  const A *src = reinterpret_cast<const A *>(&ops);
  constexpr int n = N * N + 4 * N;
  for (int i = tid; i < n; i += nth) sops[i] = src[i];
}

// Barrier of the threads running one tile: the whole block (bar == 0) or a
// warp-aligned group of nth threads on named barrier `bar` (batched stages).
__device__ __forceinline__ void group_sync(int bar, int nth)
{
  if (bar == 0)
    __syncthreads();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nth) : "memory");
}

// Shared-memory views of the line operators
template <typename A, int N>
struct SOps
{
  const A *Dm, *Em, *Ep, *Dbm, *Dbp;
  __device__ SOps(const A *p) : Dm(p), Em(p + N * N), Ep(p + N * N + N), Dbm(p + N * N + 2 * N), Dbp(p + N * N + 3 * N) {}
};

// extrapolate component v of the tile state in smem (layout [S][V][TW]) to flux point f
template <typename A, int D, int N>
__device__ __forceinline__ A extrap_smem(const A *sX, const SOps<A, N> &o, int f, int v, int l, int nv)
{
  int dim, side, base, stride;
  fpt_line<D, N>(f, dim, side, base, stride);
  const A *E = side < 0 ? o.Em : o.Ep;
  A acc = E[0] * sX[((base)*nv + v) * TW + l];
#pragma unroll
  for (int m = 1; m < N; m++) acc += E[m] * sX[((base + m * stride) * nv + v) * TW + l];
  return acc;
}

// read the neighbour's copy of a [tile][Fp][V][TW] array
template <typename T, typename A, int V>
__device__ __forceinline__ void gather_fpt(const T *src, int pidx, A out[V])
{
  const int64_t row = (int64_t)(pidx / TW) * V;
  const int lane = pidx % TW;
#pragma unroll
  for (int v = 0; v < V; v++) out[v] = (A)src[(row + v) * TW + lane];
}

// Shared-memory tile arrays of the 2D kernels (states, common solutions,
// gradients, fluxes) keep the variables of one (point, element) in 16-byte
// groups, [P][4/W][TW][W] with W = 16 / sizeof(A): FP32 holds all four
// variables in one group, FP64 two groups of two.  One 16-byte load per group
// fetches a point's variables where the global [P][V][TW] order takes four
// loads, and the eight elements of a warp's point read 128 contiguous bytes
// per group (no bank conflicts).
template <typename A>
struct TVec
{
  static constexpr int W = 16 / (int)sizeof(A), G = 4 / W;
};

// offset of (point p, element l, variable v)
template <typename A>
__device__ __forceinline__ int tix(int p, int l, int v)
{
  return ((p * TVec<A>::G + v / TVec<A>::W) * TW + l) * TVec<A>::W + v % TVec<A>::W;
}

// offset of (point p, element l)'s first group
template <typename A>
__device__ __forceinline__ int tvl(int p, int l)
{
  return tix<A>(p, l, 0);
}

__device__ __forceinline__ void ld4(const float *p, float x[4])
{
  const float4 q = *reinterpret_cast<const float4 *>(p);
  x[0] = q.x;
  x[1] = q.y;
  x[2] = q.z;
  x[3] = q.w;
}

// the second group of two doubles sits TW groups further on
__device__ __forceinline__ void ld4(const double *p, double x[4])
{
  const double2 a = *reinterpret_cast<const double2 *>(p);
  const double2 b = *reinterpret_cast<const double2 *>(p + 2 * TW);
  x[0] = a.x;
  x[1] = a.y;
  x[2] = b.x;
  x[3] = b.y;
}

__device__ __forceinline__ void st4(float *p, const float x[4])
{
  *reinterpret_cast<float4 *>(p) = make_float4(x[0], x[1], x[2], x[3]);
}

__device__ __forceinline__ void st4(double *p, const double x[4])
{
  *reinterpret_cast<double2 *>(p) = make_double2(x[0], x[1]);
  *reinterpret_cast<double2 *>(p + 2 * TW) = make_double2(x[2], x[3]);
}

// ---------------------------------------------------------------------------
// Common convective flux at one own flux point (Rusanov or Roe) plus ghost
// states on boundaries; returns the outward, dA-scaled own-side value in Fc
// (src/faces.cpp:1243-1364, 1616-1640).  For viscous runs the LDG part is
// added by the caller.
// ---------------------------------------------------------------------------
template <typename T, typename A, int D>
__device__ __forceinline__ void conv_common(const Args<T, A> &a, const A Uo[D + 2], const A Un[D + 2], int code,
                                            const A n[D], A UL[D + 2], A UR[D + 2], A UB[D + 2], A F[D + 2])
{
  if (code >= 0)
  {
    const int slot = code & 1;
#pragma unroll
    for (int v = 0; v < D + 2; v++)
    {
      UL[v] = slot ? Un[v] : Uo[v];
      UR[v] = slot ? Uo[v] : Un[v];
      UB[v] = UR[v];
    }
  }
  else
  {
    A Ua[D + 2], URa[D + 2], UBa[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; v++) UL[v] = Uo[v];
    to_abs<A, D>(Uo, Ua, a.ph);
    ghost_state<A, D>(-code - 1, Ua, n, URa, UBa, a.ph);
    to_stored<A, D>(URa, UR, a.ph);
    to_stored<A, D>(UBa, UB, a.ph);
  }
  if (a.ph.fconv == 2)
    roe<A, D>(UL, UR, n, F, a.ph);
  else
    rusanov<A, D>(UL, UR, n, F, a.ph);
}

// time step of element (tile, lane): per element, device-computed or fixed
template <typename T, typename A>
__device__ __forceinline__ A step_dt(const Args<T, A> &a, int64_t tile, int l)
{
  if (a.dt_ele) return (A)a.dt_ele[tile * TW + l];
  if (a.dt_dev) return (A)a.dt_dev[0];
  return a.dt;
}

// ---------------------------------------------------------------------------
// 2D faces (quadrilaterals and triangles: four variables, Fp flux points per
// element)
// ---------------------------------------------------------------------------

// LDG common solution at own flux point f (flip_beta = 1) from the traces
template <typename T, typename A>
__device__ __forceinline__ void common_solution_2d(const Args<T, A> &a, int64_t tile, int Fp, int f, int l, int code,
                                                   const A Uo[4], A UC[4])
{
  const A beta = a.ph.ldg_b;
  if (code >= 0)
  {
    const int slot = code & 1;
    if ((beta == A(0.5) && slot) || (beta == A(-0.5) && !slot))
    {
      // beta = +1/2 (-1/2) takes the right (left) trace: the own one, no gather
#pragma unroll
      for (int v = 0; v < 4; v++) UC[v] = Uo[v];
      return;
    }
    A Un[4];
    gather_fpt<T, A, 4>(a.Ufp, code >> 1, Un);
#pragma unroll
    for (int v = 0; v < 4; v++)
    {
      const A ul = slot ? Un[v] : Uo[v];
      const A ur = slot ? Uo[v] : Un[v];
      if (beta == A(0.5))
        UC[v] = ur;
      else if (beta == A(-0.5))
        UC[v] = ul;
      else
        UC[v] = A(0.5) * (ul + ur) - beta * (ul - ur);
    }
    return;
  }
  A n[2], Ua[4], URa[4], UBa[4];
  const T *g = a.fgeo + (tile * Fp + f) * (int64_t)3 * TW + l;
  n[0] = g[0];
  n[1] = g[TW];
  to_abs<A, 2>(Uo, Ua, a.ph);
  ghost_state<A, 2>(-code - 1, Ua, n, URa, UBa, a.ph);
  to_stored<A, 2>(UBa, UC, a.ph);
}

// whether this side forms the viscous normal flux of a point: not where
// one-sided LDG takes the partner's
template <typename A>
__device__ __forceinline__ bool own_visc_flux(A beta, int code)
{
  return !(code >= 0 && ((beta == A(0.5) && (code & 1)) || (beta == A(-0.5) && !(code & 1))));
}

// viscous normal flux at own flux point f from its trace and gradient trace
// (boundaries: of the prescribed state UC and gradient)
template <typename T, typename A>
__device__ __forceinline__ void visc_face_2d(const Args<T, A> &a, int64_t tile, int Fp, int f, int l, int code,
                                             const A Uf[4], const A dUf[4][2], const A UC[4])
{
  A n[2], Ua[4], Fn[4];
  const T *g = a.fgeo + (tile * Fp + f) * (int64_t)3 * TW + l;
  n[0] = g[0];
  n[1] = g[TW];
  to_abs<A, 2>(Uf, Ua, a.ph);
  if (code >= 0)
    visc_normal<A, 2>(Ua, dUf, n, Fn, a.ph);
  else
  {
    A UB[4], dUB[4][2];
    if constexpr (Pert<A>::on)
    {
      A UR[4];
      ghost_state<A, 2>(-code - 1, Ua, n, UR, UB, a.ph);
    }
    else
    {
      // the prescribed state is the point's common solution
#pragma unroll
      for (int v = 0; v < 4; v++) UB[v] = UC[v];
    }
    ghost_grad<A, 2>(-code - 1, Ua, dUf, n, dUB);
    visc_normal<A, 2>(UB, dUB, n, Fn, a.ph);
  }
  T *out = a.Fvn + (tile * Fp + f) * (int64_t)4 * TW + l;
#pragma unroll
  for (int v = 0; v < 4; v++) out[v * TW] = Fn[v];
}

// convective (VISC: + LDG viscous) common flux at own flux point f, dA-scaled
// and signed for this element
template <typename T, typename A, bool VISC>
__device__ __forceinline__ void common_flux_2d(const Args<T, A> &a, int64_t tile, int Fp, int f, int l, A out[4])
{
  constexpr int V = 4;
  const int code = a.nbr[(tile * Fp + f) * (int64_t)TW + l];
  const T *g = a.fgeo + (tile * Fp + f) * (int64_t)3 * TW + l;
  const A n[2] = {g[0], g[TW]};
  const A dA = g[2 * TW];
  A Uo[V], Un[V], UL[V], UR[V], UB[V], Fc[V];
  const T *uo = a.Ufp + (tile * Fp + f) * (int64_t)V * TW + l;
#pragma unroll
  for (int v = 0; v < V; v++) Uo[v] = uo[v * TW];
  if (code >= 0) gather_fpt<T, A, V>(a.Ufp, code >> 1, Un);
  A F1[V], F2[V];
  const A beta = a.ph.ldg_b, tau = a.ph.ldg_tau;
  if (VISC)
  {
    // the viscous normal flux of the side(s) LDG takes, loaded with the traces
    const bool own = own_visc_flux(beta, code);
    const T *fvo = a.Fvn + (tile * Fp + f) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) F1[v] = F2[v] = A(0);
    if (own)
    {
#pragma unroll
      for (int v = 0; v < V; v++) F1[v] = fvo[v * TW];
    }
    if (code >= 0 && (!own || (beta != A(0.5) && beta != A(-0.5)))) gather_fpt<T, A, V>(a.Fvn, code >> 1, F2);
  }
  conv_common<T, A, 2>(a, Uo, Un, code, n, UL, UR, UB, Fc);
  const bool right = (code >= 0) && (code & 1);
  if (VISC)
  {
#pragma unroll
    for (int v = 0; v < V; v++)
    {
      const A FnL = right ? F2[v] : F1[v], FnR = right ? F1[v] : F2[v];
      if (code >= 0)
        Fc[v] += A(0.5) * (FnL + FnR) + tau * (UL[v] - UR[v]) + beta * (FnL - FnR);
      else
        Fc[v] += FnL + tau * (UL[v] - UB[v]);
    }
  }
#pragma unroll
  for (int v = 0; v < V; v++) out[v] = right ? -Fc[v] * dA : Fc[v] * dA;
}

// ---------------------------------------------------------------------------
// Store the residual of one point and apply the optional RK update
// (src/solver.cpp:2916-2937, 3040-3094).  rk_load fetches what the update
// needs besides the residual, ahead of the barrier before the surface terms.
// ---------------------------------------------------------------------------
template <typename A, int V>
struct RkIn
{
  A detJ, u_ini[V];
};

template <typename T, typename A, int S, int V, int NM>
__device__ __forceinline__ void rk_load(const Args<T, A> &a, int64_t tile, int s, int l, RkIn<A, V> &in)
{
  constexpr int D = NM == 5 ? 2 : 3;
  const int64_t base = (tile * S + s) * (int64_t)V * TW;
  in.detJ = a.mets[((tile * S + s) * NM + D * D) * TW + l];
#pragma unroll
  for (int v = 0; v < V; v++) in.u_ini[v] = a.save_ini ? (A)a.U[base + v * TW + l] : (A)a.U_ini[base + v * TW + l];
}

// unew: the updated state as stored
template <typename T, typename A, int S, int V>
__device__ __forceinline__ void store_rk(const Args<T, A> &a, int64_t tile, int s, int l, const A res[V],
                                         const RkIn<A, V> &in, A unew[V])
{
  constexpr int MAXPREV = 3;
  const int64_t base = (tile * S + s) * (int64_t)V * TW;
  if (a.rk_mode == 0)
  {
#pragma unroll
    for (int v = 0; v < V; v++) a.divF[base + v * TW + l] = res[v];
    return;
  }
  // every load of the point before the first store: a load cannot move above
  // a store that may alias it, so interleaving them serialises the accesses
  const A dtv = step_dt(a, tile, l);
  const bool fast = a.rk_mode == 1 || a.nprev <= MAXPREV;
  A prev[MAXPREV][V], comp[V];
#pragma unroll
  for (int v = 0; v < V; v++) comp[v] = (a.rk_mode == 2 && a.Ucomp) ? (A)a.Ucomp[base + v * TW + l] : A(0);
  if (a.rk_mode == 2 && fast)
  {
#pragma unroll
    for (int st = 0; st < MAXPREV; st++)
      if (st < a.nprev)
      {
#pragma unroll
        for (int v = 0; v < V; v++) prev[st][v] = (A)a.divF_prev[st][base + v * TW + l];
      }
  }
#pragma unroll
  for (int v = 0; v < V; v++) a.divF[base + v * TW + l] = res[v];
  const A c = dtv / in.detJ;
#pragma unroll
  for (int v = 0; v < V; v++)
  {
    const int64_t idx = base + v * TW + l;
    if (a.save_ini) a.U_ini[idx] = in.u_ini[v];
    A u;
    if (a.rk_mode == 1)
      u = in.u_ini[v] - a.rk_coef[0] * c * res[v];
    else if (a.Ucomp)
    {
      // Kahan-compensated accumulation of the step increment; the
      // remainder includes the rounding of the stored state
      A delta = A(0);
      if (fast)
      {
#pragma unroll
        for (int st = 0; st < MAXPREV; st++)
          if (st < a.nprev) delta -= a.rk_coef[st] * c * prev[st][v];
      }
      else
        for (int st = 0; st < a.nprev; st++) delta -= a.rk_coef[st] * c * (A)a.divF_prev[st][idx];
      delta -= a.rk_coef[a.nprev] * c * res[v];
      const A y = delta - comp[v];
      u = (A)(T)(in.u_ini[v] + y);
      a.Ucomp[idx] = (T)((u - in.u_ini[v]) - y);
    }
    else
    {
      // reference order: U = U_ini; U -= b_s dt/|J| divF_s for s = 0..
      u = in.u_ini[v];
      if (fast)
      {
#pragma unroll
        for (int st = 0; st < MAXPREV; st++)
          if (st < a.nprev) u -= a.rk_coef[st] * c * prev[st][v];
      }
      else
        for (int st = 0; st < a.nprev; st++) u -= a.rk_coef[st] * c * a.divF_prev[st][idx];
      u -= a.rk_coef[a.nprev] * c * res[v];
    }
    a.Uout[idx] = u;
    unew[v] = (A)(T)u;
  }
}

}  // namespace dev
}  // namespace zb
