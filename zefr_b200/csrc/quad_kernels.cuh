// Tensor-product DFR residual kernels for quadrilaterals of order P = N - 1.
//
// One CTA per tile of TW elements; in the standalone kernels a thread owns one
// solution point and one flux point, so what a pass computed stays in registers
// for the next: the gradient kernel needs two barriers where looping over
// points pass by pass took four, and reads metrics, codes and traces once.
// The tile arrays in shared memory hold a point's four variables in 16-byte
// groups (TVec).  Line operators and summation order as described in
// dfr_kernels.cuh.  Measured against the pass-by-pass kernels (scalar shared
// reads, 128 or 256 threads, 3 CTAs of 142-156 registers per SM in FP64), us,
// 140^2 elements, Navier-Stokes Roe, gradient / face with RK update: FP64 P3
// 36 -> 23 / 36 -> 27, P4 72 -> 45 / 63 -> 50; mixed P3 26 -> 15 / 20 -> 17,
// P4 48 -> 23 / 31 -> 24.  Euler P4: FP64 75 -> 50, mixed 39 -> 23.5.
#pragma once

#include "dfr_kernels.cuh"

namespace zb {
namespace dev {

template <int N>
struct QuadShape
{
  static constexpr int S = N * N, Fp = 4 * N, V = 4, NM = 5;
  static constexpr int items = (S > Fp ? S : Fp) * TW;
  static constexpr int NT = (items + 31) / 32 * 32;  // a thread per solution point and per flux point
};

// CTAs per SM the registers are held to, as resident threads.  These kernels
// are bound by latency (a chain of gathers, two barriers and FP64 divisions
// per tile).  FP32 P4, 140^2 elements, us at 1024 / 1280 / 1536 threads:
// gradient 24.2 / 23.1 / 24.3, Euler 25.2 / 23.5 / 23.8, face with RK update
// 23.7 / 23.7 / 25.9 (P2: 14.2 / 15.3 / 17.0).  FP64 at 512, 640 and 768 is
// within 1% of itself; 512 spills least.  512 threads are one CTA of P5's 288,
// too few for the FP64 face kernel where an SM has more than one tile to do:
// `face_many` CTAs then (P5: two of 96 registers, some spilled).  P5 FP64 face,
// n^2 elements, LDG beta 0.3 Rusanov, us at one -> two: n 60 14.2 -> 12.5 (with
// the RK update 17.3 -> 15.1), n 140 51.5 -> 43.4 (73.3 -> 59.5); beta 0.5 Roe
// n 140 51.6 -> 50.9 (75.2 -> 68.3); n 24, fewer tiles than SMs, 8.9 -> 10.1.
template <typename A, int N>
struct QuadOcc
{
  static constexpr int nt = QuadShape<N>::NT;
  static constexpr bool f64 = sizeof(A) == 8;
  static constexpr int grad = (f64 ? 512 : 1280) / nt, face = (f64 ? 512 : 1024) / nt,
                       euler = (f64 ? 512 : 1280) / nt;
  static constexpr int face_many = face > 1 ? face : 2;
};

// X_v(f) of the four variables of a shared tile array at flux point f
template <typename A, int N>
__device__ __forceinline__ void quad_extrap4(const A *sX, const SOps<A, N> &o, int f, int l, A out[4])
{
  int dim, side, base, stride;
  fpt_line<2, N>(f, dim, side, base, stride);
  const A *E = side < 0 ? o.Em : o.Ep;
#pragma unroll
  for (int m = 0; m < N; m++)
  {
    A x[4];
    ld4(sX + tvl<A>(base + m * stride, l), x);
    const A e = E[m];
#pragma unroll
    for (int v = 0; v < 4; v++) out[v] = m == 0 ? e * x[v] : out[v] + e * x[v];
  }
}

// transformed flux F~_d = adj[d][.] . F into point d * S + s of sF
template <typename A>
__device__ __forceinline__ void quad_transform(const A F[4][2], const A adj[2][2], A *sF, int S, int s, int l)
{
#pragma unroll
  for (int d1 = 0; d1 < 2; d1++)
  {
    A t[4];
#pragma unroll
    for (int v = 0; v < 4; v++) t[v] = F[v][0] * adj[d1][0] + F[v][1] * adj[d1][1];
    st4(sF + tvl<A>(d1 * S + s, l), t);
  }
}

// volume divergence of the transformed flux at solution point s
template <typename A, int N>
__device__ __forceinline__ void quad_divergence(const A *sF, const SOps<A, N> &o, int s, int l, A vol[4])
{
  constexpr int S = N * N;
#pragma unroll
  for (int v = 0; v < 4; v++) vol[v] = A(0);
#pragma unroll
  for (int d = 0; d < 2; d++)
  {
    int i, fm, fp;
    spt_ends<2, N>(s, d, i, fm, fp);
    const int st = pow_n<N>(d), b = s - i * st;
#pragma unroll
    for (int m = 0; m < N; m++)
    {
      A x[4];
      ld4(sF + tvl<A>(d * S + b + m * st, l), x);
      const A c = o.Dm[i * N + m];
#pragma unroll
      for (int v = 0; v < 4; v++) vol[v] += c * x[v];
    }
  }
}

// surface terms of solution point s in ascending face order
template <typename A, int N>
__device__ __forceinline__ void quad_surface(const A *sFc, const SOps<A, N> &o, int s, int l, A surf[4])
{
#pragma unroll
  for (int v = 0; v < 4; v++) surf[v] = A(0);
#pragma unroll
  for (int face = 0; face < 4; face++)
  {
    int dim, side, i, fm, fp;
    face_dim_side<2>(face, dim, side);
    spt_ends<2, N>(s, dim, i, fm, fp);
    const A c = side < 0 ? -o.Dbm[i] : o.Dbp[i];
    A x[4];
    ld4(sFc + tvl<A>(side < 0 ? fm : fp, l), x);
#pragma unroll
    for (int v = 0; v < 4; v++) surf[v] += c * x[v];
  }
}

// traces of the updated state (sU, shared) for the next stage
template <typename T, typename A, int N>
__device__ __forceinline__ void quad_extrap_next(const Args<T, A> &a, int64_t tile, const A *sU, const SOps<A, N> &o,
                                                 int f, int l)
{
  A x[4];
  quad_extrap4<A, N>(sU, o, f, l, x);
  T *out = a.Ufp_next + (tile * QuadShape<N>::Fp + f) * (int64_t)4 * TW + l;
#pragma unroll
  for (int v = 0; v < 4; v++) out[v * TW] = x[v];
}

// ---------------------------------------------------------------------------
// Extrapolate the state to flux points: U_fpts = oppE U_spts (src/elements.cpp:1337-1360)
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(256) k_extrap(const T *__restrict__ U, T *__restrict__ Ufp, int64_t ntiles,
                                                const __grid_constant__ LineOpsT<A, N> ops)
{
  using G = QuadShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V;
  const int64_t total = ntiles * Fp * TW;
  for (int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gid < total; gid += (int64_t)gridDim.x * blockDim.x)
  {
    const int l = (int)(gid % TW);
    const int f = (int)((gid / TW) % Fp);
    const int64_t tile = gid / ((int64_t)TW * Fp);
    int dim, side, base, stride;
    fpt_line<2, N>(f, dim, side, base, stride);
    const T *Ut = U + tile * (int64_t)S * V * TW;
    T *out = Ufp + (tile * Fp + f) * (int64_t)V * TW;
#pragma unroll
    for (int v = 0; v < V; v++)
    {
      A acc = (side < 0 ? ops.Em[0] : ops.Ep[0]) * (A)Ut[((base)*V + v) * TW + l];
#pragma unroll
      for (int m = 1; m < N; m++)
        acc += (side < 0 ? ops.Em[m] : ops.Ep[m]) * (A)Ut[((base + m * stride) * V + v) * TW + l];
      out[v * TW + l] = (T)acc;
    }
  }
}

// ---------------------------------------------------------------------------
// Euler: volume flux, common flux and divergence of one tile, run by NTH
// threads (0: the runtime count nth) synchronised on barrier `bar`.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N, int NTH = 0>
__device__ __forceinline__ void euler_tile(const Args<T, A> &a, const LineOpsT<A, N> &ops, int64_t tile,
                                           unsigned char *smem_raw, int tid, int nth, int bar)
{
  using G = QuadShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, NM = G::NM;
  if (NTH) nth = NTH;
  A *sU = reinterpret_cast<A *>(smem_raw);  // [S] points: the updated state
  A *sF = sU + S * V * TW;                  // [2 S] points: transformed flux
  A *sFc = sF + 2 * S * V * TW;             // [Fp] points: common flux
  A *sops = sFc + Fp * V * TW;
  load_ops<A, N>(sops, ops, tid, nth);
  SOps<A, N> o(sops);
  // transformed volume flux F~ = adj F (src/elements.cpp:1588-1699)
  for (int it = tid; it < S * TW; it += nth)
  {
    const int s = it / TW, l = it % TW;
    const T *u = a.U + (tile * S + s) * (int64_t)V * TW + l;
    const T *m = a.mets + (tile * S + s) * (int64_t)NM * TW + l;
    A U[V], F[V][2], P, Pp;
#pragma unroll
    for (int v = 0; v < V; v++) U[v] = u[v * TW];
    const A adj[2][2] = {{m[0], m[TW]}, {m[2 * TW], m[3 * TW]}};
    flux_conv_stored<A, 2>(U, F, P, Pp, a.ph);
    quad_transform<A>(F, adj, sF, S, s, l);
  }
  // common flux at the tile's flux points
  for (int it = tid; it < Fp * TW; it += nth)
  {
    const int f = it / TW, l = it % TW;
    A out[V];
    common_flux_2d<T, A, false>(a, tile, Fp, f, l, out);
    st4(sFc + tvl<A>(f, l), out);
  }
  group_sync(bar, nth);
  for (int it = tid; it < S * TW; it += nth)
  {
    const int s = it / TW, l = it % TW;
    RkIn<A, V> in;
    if (a.rk_mode) rk_load<T, A, S, V, NM>(a, tile, s, l, in);
    A vol[V], surf[V], unew[V];
    quad_divergence<A, N>(sF, o, s, l, vol);
    quad_surface<A, N>(sFc, o, s, l, surf);
#pragma unroll
    for (int v = 0; v < V; v++) vol[v] += surf[v];
    store_rk<T, A, S, V>(a, tile, s, l, vol, in, unew);
    if (a.extrap_next) st4(sU + tvl<A>(s, l), unew);
  }
  if (a.extrap_next)
  {
    group_sync(bar, nth);
    for (int it = tid; it < Fp * TW; it += nth) quad_extrap_next<T, A, N>(a, tile, sU, o, it / TW, it % TW);
  }
}

// Shared memory of euler_tile (elements of the arithmetic type)
template <int N>
constexpr int euler_smem_elems()
{
  return (QuadShape<N>::S * 4 * 3 + QuadShape<N>::Fp * 4) * TW + N * N + 4 * N;
}

template <typename T, typename A, int N>
__global__ void __launch_bounds__(QuadShape<N>::NT, QuadOcc<A, N>::euler)
    k_euler(const __grid_constant__ Args<T, A> a, const __grid_constant__ LineOpsT<A, N> ops)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t tile = blockIdx.x;
  if (tile >= a.ntiles) return;
  euler_tile<T, A, N, QuadShape<N>::NT>(a, ops, tile, smem_raw, threadIdx.x, QuadShape<N>::NT, 0);
}

// ---------------------------------------------------------------------------
// Navier-Stokes kernel 1: common solution, corrected gradient, viscous normal
// flux at own flux points, volume flux and its divergence
// (src/solver.cpp:1540-1600; src/elements.cpp:1393-1447, 1588-1699;
//  src/faces.cpp:1366-1474, 508-710).  A thread keeps its point's state,
// metrics and gradient in registers from the gradient to the flux, so the flux
// is formed before the faces read the gradient and two barriers suffice; it
// keeps its flux point's code, trace and common solution likewise.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(QuadShape<N>::NT, QuadOcc<A, N>::grad)
    k_ns_grad(const __grid_constant__ Args<T, A> a, const __grid_constant__ LineOpsT<A, N> ops)
{
  using G = QuadShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, NM = G::NM, D = 2, NT = G::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sU = reinterpret_cast<A *>(smem_raw);  // [S] points
  A *sUC = sU + S * V * TW;                 // [Fp] points
  A *sdU = sUC + Fp * V * TW;               // [D S] points: physical gradient
  A *sF = sdU + D * S * V * TW;             // [D S] points: transformed flux
  A *sops = sF + D * S * V * TW;
  load_ops<A, N>(sops, ops, threadIdx.x, NT);
  const int64_t tile = blockIdx.x;
  if (tile >= a.ntiles) return;
  SOps<A, N> o(sops);
  const int p = threadIdx.x / TW, l = threadIdx.x % TW;  // solution point and flux point of this thread
  const bool has_s = p < S, has_f = p < Fp;
  A U[V], adj[D][D], det = A(1), Uf[V], UC[V];
  int code = 0;
  if (has_s)
  {
    const T *u = a.U + (tile * S + p) * (int64_t)V * TW + l;
    const T *m = a.mets + (tile * S + p) * (int64_t)NM * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) U[v] = u[v * TW];
#pragma unroll
    for (int d1 = 0; d1 < D; d1++)
#pragma unroll
      for (int d2 = 0; d2 < D; d2++) adj[d1][d2] = m[(d1 * D + d2) * TW];
    det = m[D * D * TW];
    st4(sU + tvl<A>(p, l), U);
  }
  if (has_f)
  {
    code = a.nbr[(tile * Fp + p) * (int64_t)TW + l];
    const T *uo = a.Ufp + (tile * Fp + p) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) Uf[v] = uo[v * TW];
    common_solution_2d<T, A>(a, tile, Fp, p, l, code, Uf, UC);
    st4(sUC + tvl<A>(p, l), UC);
  }
  __syncthreads();
  if (has_s)
  {
    // corrected reference gradient, transformed to physical space
    A tdU[V][D], dU[V][D];
#pragma unroll
    for (int d = 0; d < D; d++)
    {
      int i, fm, fp;
      spt_ends<2, N>(p, d, i, fm, fp);
      const int st = pow_n<N>(d), b = p - i * st;
#pragma unroll
      for (int v = 0; v < V; v++) tdU[v][d] = A(0);
#pragma unroll
      for (int m = 0; m < N; m++)
      {
        A x[V];
        ld4(sU + tvl<A>(b + m * st, l), x);
        const A c = o.Dm[i * N + m];
#pragma unroll
        for (int v = 0; v < V; v++) tdU[v][d] += c * x[v];
      }
      A xm[V], xp[V];
      ld4(sUC + tvl<A>(fm, l), xm);
      ld4(sUC + tvl<A>(fp, l), xp);
      const A cm = o.Dbm[i], cp = o.Dbp[i];
#pragma unroll
      for (int v = 0; v < V; v++) tdU[v][d] += cm * xm[v] + cp * xp[v];
    }
    const A inv_det = A(1) / det;
#pragma unroll
    for (int d1 = 0; d1 < D; d1++)
    {
      A g[V];
#pragma unroll
      for (int v = 0; v < V; v++)
      {
        g[v] = (tdU[v][0] * adj[0][d1] + tdU[v][1] * adj[1][d1]) * inv_det;
        dU[v][d1] = g[v];
      }
      st4(sdU + tvl<A>(d1 * S + p, l), g);
      if (a.dU_out)
      {
        T *out = a.dU_out + ((tile * D + d1) * S + p) * (int64_t)V * TW + l;
#pragma unroll
        for (int v = 0; v < V; v++) out[v * TW] = (T)g[v];
      }
    }
    // flux, transformed: F~ = adj (F_conv + F_visc)
    A F[V][D], P, Pp, Ua[V];
    flux_conv_stored<A, D>(U, F, P, Pp, a.ph);
    to_abs<A, D>(U, Ua, a.ph);
    flux_visc_add<A, D>(Ua, dU, F, a.ph);
    quad_transform<A>(F, adj, sF, S, p, l);
  }
  __syncthreads();
  if (has_f && own_visc_flux(a.ph.ldg_b, code))
  {
    A dUf[V][D];
#pragma unroll
    for (int d = 0; d < D; d++)
    {
      A x[V];
      quad_extrap4<A, N>(sdU + d * S * V * TW, o, p, l, x);
#pragma unroll
      for (int v = 0; v < V; v++) dUf[v][d] = x[v];
    }
    visc_face_2d<T, A>(a, tile, Fp, p, l, code, Uf, dUf, UC);
  }
  if (has_s)
  {
    A vol[V];
    quad_divergence<A, N>(sF, o, p, l, vol);
    A *out = a.divF_vol + (tile * S + p) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) out[v * TW] = vol[v];
  }
}

// Shared memory of the gradient and face kernels (elements)
template <int N>
constexpr int quad_grad_smem_elems()
{
  return (QuadShape<N>::S * 4 * 5 + QuadShape<N>::Fp * 4) * TW + N * N + 4 * N;
}
template <int N>
constexpr int quad_face_smem_elems()
{
  return (QuadShape<N>::S * 4 + QuadShape<N>::Fp * 4) * TW + N * N + 4 * N;
}

// ---------------------------------------------------------------------------
// Navier-Stokes kernel 2: convective + LDG common flux, surface correction,
// optional RK update (src/faces.cpp:1476-1614; src/elements.cpp:1476-1501).
// The point's volume residual and update inputs load while the face flux is
// formed.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N, int MINB>
__global__ void __launch_bounds__(QuadShape<N>::NT, MINB)
    k_ns_face(const __grid_constant__ Args<T, A> a, const __grid_constant__ LineOpsT<A, N> ops)
{
  using G = QuadShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, NM = G::NM, NT = G::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sFc = reinterpret_cast<A *>(smem_raw);  // [Fp] points
  A *sUnew = sFc + Fp * V * TW;              // [S] points
  A *sops = sUnew + S * V * TW;
  load_ops<A, N>(sops, ops, threadIdx.x, NT);
  const int64_t tile = blockIdx.x;
  if (tile >= a.ntiles) return;
  SOps<A, N> o(sops);
  const int p = threadIdx.x / TW, l = threadIdx.x % TW;
  const bool has_s = p < S, has_f = p < Fp;
  RkIn<A, V> in;
  A res[V];
  if (has_s)
  {
    const A *dv = a.divF_vol + (tile * S + p) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) res[v] = dv[v * TW];
    if (a.rk_mode) rk_load<T, A, S, V, NM>(a, tile, p, l, in);
  }
  if (has_f)
  {
    A out[V];
    common_flux_2d<T, A, true>(a, tile, Fp, p, l, out);
    st4(sFc + tvl<A>(p, l), out);
  }
  __syncthreads();
  if (has_s)
  {
    A surf[V], unew[V];
    quad_surface<A, N>(sFc, o, p, l, surf);
#pragma unroll
    for (int v = 0; v < V; v++) res[v] += surf[v];
    store_rk<T, A, S, V>(a, tile, p, l, res, in, unew);
    if (a.extrap_next) st4(sUnew + tvl<A>(p, l), unew);
  }
  if (a.extrap_next)
  {
    __syncthreads();
    if (has_f) quad_extrap_next<T, A, N>(a, tile, sUnew, o, p, l);
  }
}

}  // namespace dev
}  // namespace zb
