// Flux-reconstruction residual kernels for triangles of order P = N - 1 with
// dense operators (S = N(N+1)/2 solution points, Fp = 3N flux points).
//
// Same tile-major layout, face codes and pointwise physics as the tensor-
// product kernels (dfr_kernels.cuh); the operators are the reference's dense
// oppE, oppD, oppD_fpts, oppDiv, oppDiv_fpts (src/elements.cpp:656-744),
// applied as the reference's products apply them (src/elements.cpp:
// 1337-1501): one sum over the whole row in ascending column order, the
// flux-point (correction) sum added after the solution-point sum.
#pragma once

#include "dfr_kernels.cuh"

namespace zb {
namespace dev {

template <int N>
struct TriShape
{
  static constexpr int D = 2, V = 4, NM = 5;
  static constexpr int S = N * (N + 1) / 2;
  static constexpr int Fp = 3 * N;
  static constexpr int NT = 128;
  // dense operator block: oppE [Fp][S], oppD [D][S][S], oppD_fpts [D][S][Fp],
  // oppDiv [S][D*S], oppDiv_fpts [S][Fp]
  static constexpr int OE = 0, OD = OE + Fp * S, ODF = OD + D * S * S, ODV = ODF + D * S * Fp,
                       ODVF = ODV + S * D * S, NOPS = ODVF + S * Fp;
  // the tile arrays that follow the operator block in shared memory start on
  // a 16-byte boundary
  static constexpr int OPS_PAD = ((NOPS + 3) / 4) * 4;
  static_assert(V == 4, "the shared tile arrays hold four variables per point");
};

// global [S][V][TW] tile -> the shared layout above
template <typename T, typename A, int S>
__device__ __forceinline__ void load_tile_vl(const T *__restrict__ src, A *dst)
{
  for (int i = threadIdx.x; i < S * 4 * TW; i += blockDim.x)
  {
    const int l = i % TW, v = (i / TW) % 4, p = i / (4 * TW);
    dst[tix<A>(p, l, v)] = src[i];
  }
}

// X_v(f) = sum_s E[f][s] Y_v(s) for the four variables of a shared tile array
template <typename A, int N>
__device__ __forceinline__ void tri_extrap4(const A *sY, const A *E, int f, int l, A out[4])
{
  constexpr int S = TriShape<N>::S;
#pragma unroll
  for (int v = 0; v < 4; v++) out[v] = A(0);
#pragma unroll
  for (int t = 0; t < S; t++)
  {
    A x[4];
    ld4(sY + tvl<A>(t, l), x);
    const A e = E[f * S + t];
#pragma unroll
    for (int v = 0; v < 4; v++) out[v] += e * x[v];
  }
}

template <typename A, int N>
__device__ __forceinline__ void load_tri_ops(A *sops, const A *g)
{
  for (int i = threadIdx.x; i < TriShape<N>::NOPS; i += blockDim.x) sops[i] = g[i];
}

template <typename T, typename A, int N>
__global__ void __launch_bounds__(128) k_tri_extrap(const T *__restrict__ U, T *__restrict__ Ufp, int64_t ntiles,
                                                    const A *__restrict__ dops)
{
  using G = TriShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V;
  __shared__ A sE[Fp * S];
  for (int i = threadIdx.x; i < Fp * S; i += blockDim.x) sE[i] = dops[G::OE + i];
  __syncthreads();
  const int64_t total = ntiles * Fp * TW;
  for (int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gid < total; gid += (int64_t)gridDim.x * blockDim.x)
  {
    const int l = (int)(gid % TW);
    const int f = (int)((gid / TW) % Fp);
    const int64_t tile = gid / ((int64_t)TW * Fp);
    const T *Ut = U + tile * (int64_t)S * V * TW;
    T *out = Ufp + (tile * Fp + f) * (int64_t)V * TW;
#pragma unroll
    for (int v = 0; v < V; v++)
    {
      A acc = A(0);
#pragma unroll
      for (int t = 0; t < S; t++) acc += sE[f * S + t] * (A)Ut[(t * V + v) * TW + l];
      out[v * TW + l] = (T)acc;
    }
  }
}

template <typename T, typename A, int N>
__device__ __forceinline__ void tri_extrap_next(const Args<T, A> &a, int64_t tile, const A *sUnew, const A *E)
{
  using G = TriShape<N>;
  constexpr int Fp = G::Fp, V = G::V;
  for (int it = threadIdx.x; it < Fp * TW; it += blockDim.x)
  {
    const int f = it / TW, l = it % TW;
    A x[V];
    tri_extrap4<A, N>(sUnew, E, f, l, x);
    T *out = a.Ufp_next + (tile * Fp + f) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) out[v * TW] = (T)x[v];
  }
}

// transformed flux F~_d = adj[d][.] . F at solution point s into sF [D*S] points
template <typename A>
__device__ __forceinline__ void tri_transform(const A F[4][2], const A adj[2][2], A *sF, int S, int s, int l)
{
#pragma unroll
  for (int d1 = 0; d1 < 2; d1++)
  {
    A Ft[4];
#pragma unroll
    for (int v = 0; v < 4; v++) Ft[v] = F[v][0] * adj[d1][0] + F[v][1] * adj[d1][1];
    st4(sF + tvl<A>(d1 * S + s, l), Ft);
  }
}

// divF(s) = sum_k oppDiv[s][k] F~(k) + sum_f oppDiv_fpts[s][f] Fc(f), then store / RK
template <typename T, typename A, int N>
__device__ __forceinline__ void tri_finish(const Args<T, A> &a, int64_t tile, int s, int l, const A *sF,
                                           const A *sFc, const A *ops, A *sUnew, const A *vol_in)
{
  using G = TriShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, D = 2;
  A vol[V], surf[V];
#pragma unroll
  for (int v = 0; v < V; v++)
  {
    surf[v] = A(0);
    vol[v] = A(0);
  }
  if (vol_in)
  {
#pragma unroll
    for (int v = 0; v < V; v++) vol[v] = vol_in[v];
  }
  else
  {
    const A *Dv = ops + G::ODV + s * D * S;
#pragma unroll
    for (int k = 0; k < D * S; k++)
    {
      A x[4];
      ld4(sF + tvl<A>(k, l), x);
#pragma unroll
      for (int v = 0; v < V; v++) vol[v] += Dv[k] * x[v];
    }
  }
  const A *Dvf = ops + G::ODVF + s * Fp;
#pragma unroll
  for (int f = 0; f < Fp; f++)
  {
    A x[4];
    ld4(sFc + tvl<A>(f, l), x);
#pragma unroll
    for (int v = 0; v < V; v++) surf[v] += Dvf[f] * x[v];
  }
  A res[V], unew[V];
#pragma unroll
  for (int v = 0; v < V; v++) res[v] = vol[v] + surf[v];
  RkIn<A, V> in;
  if (a.rk_mode) rk_load<T, A, S, V, 5>(a, tile, s, l, in);
  store_rk<T, A, S, V>(a, tile, s, l, res, in, unew);
  if (sUnew) st4(sUnew + tvl<A>(s, l), unew);
}

// ---------------------------------------------------------------------------
// Euler: volume flux, common flux and divergence of one tile.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(128) k_tri_euler(const __grid_constant__ Args<T, A> a)
{
  using G = TriShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, D = 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sops = reinterpret_cast<A *>(smem_raw);
  A *sU = sops + G::OPS_PAD;  // [S] points: the updated state
  A *sF = sU + S * V * TW;
  A *sFc = sF + D * S * V * TW;
  load_tri_ops<A, N>(sops, a.dops);
  const int64_t tile = blockIdx.x;
  if (tile >= a.ntiles) return;
  for (int it = threadIdx.x; it < S * TW; it += blockDim.x)
  {
    const int s = it / TW, l = it % TW;
    const T *u = a.U + (tile * S + s) * (int64_t)V * TW + l;
    const T *m = a.mets + (tile * S + s) * (int64_t)5 * TW + l;
    A U[V], F[V][D], P, Pp;
#pragma unroll
    for (int v = 0; v < V; v++) U[v] = u[v * TW];
    const A adj[2][2] = {{m[0], m[TW]}, {m[2 * TW], m[3 * TW]}};
    flux_conv_stored<A, D>(U, F, P, Pp, a.ph);
    tri_transform<A>(F, adj, sF, S, s, l);
  }
  for (int it = threadIdx.x; it < Fp * TW; it += blockDim.x)
  {
    const int f = it / TW, l = it % TW;
    A out[V];
    common_flux_2d<T, A, false>(a, tile, Fp, f, l, out);
    st4(sFc + tvl<A>(f, l), out);
  }
  __syncthreads();
  for (int it = threadIdx.x; it < S * TW; it += blockDim.x)
  {
    const int s = it / TW, l = it % TW;
    tri_finish<T, A, N>(a, tile, s, l, sF, sFc, sops, a.extrap_next ? sU : nullptr, nullptr);
  }
  if (a.extrap_next)
  {
    __syncthreads();
    tri_extrap_next<T, A, N>(a, tile, sU, sops + G::OE);
  }
}

// ---------------------------------------------------------------------------
// Navier-Stokes kernel 1: LDG common solution, corrected gradient, own viscous
// normal flux, volume flux and its divergence.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(128) k_tri_ns_grad(const __grid_constant__ Args<T, A> a)
{
  using G = TriShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, D = 2, NM = 5;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sops = reinterpret_cast<A *>(smem_raw);
  A *sU = sops + G::OPS_PAD;    // [S] points
  A *sUC = sU + S * V * TW;      // [Fp] points
  A *sdU = sUC + Fp * V * TW;    // [D*S] points: physical gradient
  A *sF = sdU + D * S * V * TW;  // [D*S] points: transformed flux
  load_tri_ops<A, N>(sops, a.dops);
  const int64_t tile = blockIdx.x;
  if (tile >= a.ntiles) return;
  load_tile_vl<T, A, S>(a.U + tile * (int64_t)S * V * TW, sU);
  for (int it = threadIdx.x; it < Fp * TW; it += blockDim.x)
  {
    const int f = it / TW, l = it % TW;
    const int code = a.nbr[(tile * Fp + f) * (int64_t)TW + l];
    A Uo[V], UC[V];
    const T *uo = a.Ufp + (tile * Fp + f) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) Uo[v] = uo[v * TW];
    common_solution_2d<T, A>(a, tile, Fp, f, l, code, Uo, UC);
    st4(sUC + tvl<A>(f, l), UC);
  }
  __syncthreads();
  // gradient: oppD U + oppD_fpts Ucomm, then physical; the point's flux right
  // after it, from registers, so the faces need not wait before it
  for (int it = threadIdx.x; it < S * TW; it += blockDim.x)
  {
    const int s = it / TW, l = it % TW;
    A tdU[V][D];
#pragma unroll
    for (int d = 0; d < D; d++)
    {
      const A *Dd = sops + G::OD + (d * S + s) * S;
      const A *Df = sops + G::ODF + (d * S + s) * Fp;
      A acc[V], cor[V];
#pragma unroll
      for (int v = 0; v < V; v++)
      {
        acc[v] = A(0);
        cor[v] = A(0);
      }
#pragma unroll
      for (int t = 0; t < S; t++)
      {
        A x[4];
        ld4(sU + tvl<A>(t, l), x);
#pragma unroll
        for (int v = 0; v < V; v++) acc[v] += Dd[t] * x[v];
      }
#pragma unroll
      for (int f = 0; f < Fp; f++)
      {
        A x[4];
        ld4(sUC + tvl<A>(f, l), x);
#pragma unroll
        for (int v = 0; v < V; v++) cor[v] += Df[f] * x[v];
      }
#pragma unroll
      for (int v = 0; v < V; v++) tdU[v][d] = acc[v] + cor[v];
    }
    const T *m = a.mets + (tile * S + s) * (int64_t)NM * TW + l;
    A adj[D][D];
#pragma unroll
    for (int d1 = 0; d1 < D; d1++)
#pragma unroll
      for (int d2 = 0; d2 < D; d2++) adj[d1][d2] = m[(d1 * D + d2) * TW];
    const A inv_det = A(1) / m[D * D * TW];
    A dU[V][D];
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
      st4(sdU + tvl<A>(d1 * S + s, l), g);
      if (a.dU_out)
      {
        T *out = a.dU_out + ((tile * D + d1) * S + s) * (int64_t)V * TW + l;
#pragma unroll
        for (int v = 0; v < V; v++) out[v * TW] = (T)g[v];
      }
    }
    A U[V], F[V][D], P, Pp, Ua[V];
    ld4(sU + tvl<A>(s, l), U);
    flux_conv_stored<A, D>(U, F, P, Pp, a.ph);
    to_abs<A, D>(U, Ua, a.ph);
    flux_visc_add<A, D>(Ua, dU, F, a.ph);
    tri_transform<A>(F, adj, sF, S, s, l);
  }
  __syncthreads();
  // own viscous normal flux at flux points
  for (int it = threadIdx.x; it < Fp * TW; it += blockDim.x)
  {
    const int f = it / TW, l = it % TW;
    const int code = a.nbr[(tile * Fp + f) * (int64_t)TW + l];
    if (!own_visc_flux(a.ph.ldg_b, code)) continue;
    A Uf[V], dUf[V][D], UC[V];
    const T *uo = a.Ufp + (tile * Fp + f) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) Uf[v] = uo[v * TW];
    ld4(sUC + tvl<A>(f, l), UC);
#pragma unroll
    for (int d = 0; d < D; d++)
    {
      A x[V];
      tri_extrap4<A, N>(sdU + d * S * V * TW, sops + G::OE, f, l, x);
#pragma unroll
      for (int v = 0; v < V; v++) dUf[v][d] = x[v];
    }
    visc_face_2d<T, A>(a, tile, Fp, f, l, code, Uf, dUf, UC);
  }
  for (int it = threadIdx.x; it < S * TW; it += blockDim.x)
  {
    const int s = it / TW, l = it % TW;
    A vol[V];
#pragma unroll
    for (int v = 0; v < V; v++) vol[v] = A(0);
    const A *Dv = sops + G::ODV + s * D * S;
#pragma unroll
    for (int k = 0; k < D * S; k++)
    {
      A x[V];
      ld4(sF + tvl<A>(k, l), x);
#pragma unroll
      for (int v = 0; v < V; v++) vol[v] += Dv[k] * x[v];
    }
    A *out = a.divF_vol + (tile * S + s) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) out[v * TW] = vol[v];
  }
}

// ---------------------------------------------------------------------------
// Navier-Stokes kernel 2: convective + LDG common flux, correction, RK.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(128) k_tri_ns_face(const __grid_constant__ Args<T, A> a)
{
  using G = TriShape<N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sops = reinterpret_cast<A *>(smem_raw);
  A *sFc = sops + G::OPS_PAD;   // [Fp] points
  A *sUnew = sFc + Fp * V * TW;  // [S] points: the updated state
  load_tri_ops<A, N>(sops, a.dops);
  const int64_t tile = blockIdx.x;
  if (tile >= a.ntiles) return;
  for (int it = threadIdx.x; it < Fp * TW; it += blockDim.x)
  {
    const int f = it / TW, l = it % TW;
    A out[V];
    common_flux_2d<T, A, true>(a, tile, Fp, f, l, out);
    st4(sFc + tvl<A>(f, l), out);
  }
  __syncthreads();
  for (int it = threadIdx.x; it < S * TW; it += blockDim.x)
  {
    const int s = it / TW, l = it % TW;
    A vol[V];
    const A *dv = a.divF_vol + (tile * S + s) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++) vol[v] = dv[v * TW];
    tri_finish<T, A, N>(a, tile, s, l, nullptr, sFc, sops, a.extrap_next ? sUnew : nullptr, vol);
  }
  if (a.extrap_next)
  {
    __syncthreads();
    tri_extrap_next<T, A, N>(a, tile, sUnew, sops + G::OE);
  }
}

}  // namespace dev
}  // namespace zb
