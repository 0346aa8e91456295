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
  // dense operator block: oppE [Fp][S], oppD [D][S][S], oppD_fpts [D][S][Fp],
  // oppDiv [S][D*S], oppDiv_fpts [S][Fp]
  static constexpr int OE = 0, OD = OE + Fp * S, ODF = OD + D * S * S, ODV = ODF + D * S * Fp,
                       ODVF = ODV + S * D * S, NOPS = ODVF + S * Fp;
  // the tile arrays that follow the operator block in shared memory start on
  // a 16-byte boundary
  static constexpr int OPS_PAD = ((NOPS + 3) / 4) * 4;
  static_assert(V == 4, "the shared tile arrays hold four variables per point");
};

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

// Launch shape: a thread per solution point and per flux point of a tile, the
// CTAs resident and walking the tiles, so a kernel's operators are copied to
// shared memory once per CTA and not once per tile (all five, at P4 14 KB in
// FP64 beside 4 KB of state per tile; P8 104 KB).  minb: CTAs per SM the
// registers and the shared memory allow, as resident threads.  Against one
// 128-thread CTA per tile (with whole flux matrices per face point), us,
// Navier-Stokes Roe gradient / face with RK update and Euler Roe with RK update,
// 2 x 110^2 elements (P8: 2 x 60^2):
//   FP64  P1 31 -> 15 / 35 -> 18, 31 -> 17;  P3 47 -> 32 / 44 -> 30, 46 -> 32;
//         P5 108 -> 93 / 90 -> 65, 111 -> 85;  P8 248 -> 107 / 123 -> 51, 165 -> 83
//   mixed P1 16 -> 12 / 17 -> 13, 17 -> 13;  P3 25 -> 21 / 22 -> 20, 25 -> 22;
//         P5 59 -> 51 / 39 -> 38, 50 -> 43;  P8 73 -> 56 / 46 -> 28, 68 -> 44
// The FP64 face kernel's 400 threads (168 registers) spill 130-160 bytes at most
// orders; 256 threads (222 registers) spill none and take longer: P1 17.9 -> 21.3,
// P3 30.4 -> 38.9, P5 65 -> 94.
template <typename A, int N>
struct TriRun
{
  using G = TriShape<N>;
  static constexpr int items = (G::S > G::Fp ? G::S : G::Fp) * TW;
  static constexpr int NT = (items + 31) / 32 * 32;
  static constexpr bool f64 = sizeof(A) == 8;
  // The operators of a kernel as one block, the two dimensions' rows of oppD,
  // oppD_fpts and oppDiv interleaved pairwise: element (row, column, d) at
  // 2 (row * columns + column) + d.  The blocks follow the plain operators in
  // Args::dops (tri_operator_blocks arranges them).
  static constexpr int pad(int n) { return (n + 3) / 4 * 4; }
  static constexpr int GU = 0, GF = GU + 2 * G::S * G::S, GDV = GF + 2 * G::S * G::Fp, GE = GDV + 2 * G::S * G::S,
                       grad_ops = pad(GE + G::Fp * G::S);
  static constexpr int FDVF = 0, FE = pad(G::S * G::Fp), face_ops = pad(FE + G::Fp * G::S);
  static constexpr int EDV = 0, EDVF = 2 * G::S * G::S, EE = pad(EDVF + G::S * G::Fp), euler_ops = pad(EE + G::Fp * G::S);
  static constexpr int GRAD_AT = pad(G::NOPS), FACE_AT = GRAD_AT + grad_ops, EULER_AT = FACE_AT + face_ops;
  static constexpr int grad_smem = (grad_ops + (5 * G::S + G::Fp) * 4 * TW) * (int)sizeof(A);
  static constexpr int face_smem = (face_ops + (G::S + G::Fp) * 4 * TW) * (int)sizeof(A);
  static constexpr int euler_smem = (euler_ops + (3 * G::S + G::Fp) * 4 * TW) * (int)sizeof(A);
  static constexpr int extrap_smem = (pad(G::Fp * G::S) + G::S * 4 * TW) * (int)sizeof(A);
  static constexpr int fit(int threads, int smem)
  {
    const int by_smem = 225 * 1024 / (smem + 1024), by_threads = threads / NT;
    const int n = by_smem < by_threads ? by_smem : by_threads;
    return n < 1 ? 1 : n > 24 ? 24 : n;
  }
  static constexpr int grad_minb = fit(f64 ? 512 : 1280, grad_smem);
  static constexpr int face_minb = fit(f64 ? 400 : 1024, face_smem);
  static constexpr int euler_minb = fit(f64 ? 512 : 1280, euler_smem);
  static constexpr int extrap_minb = fit(1536, extrap_smem);
};

// a pair of coefficients (dimension 0, dimension 1) with one load
__device__ __forceinline__ void ld2(const float *p, float &a, float &b)
{
  const float2 q = *reinterpret_cast<const float2 *>(p);
  a = q.x;
  b = q.y;
}
__device__ __forceinline__ void ld2(const double *p, double &a, double &b)
{
  const double2 q = *reinterpret_cast<const double2 *>(p);
  a = q.x;
  b = q.y;
}

// copy an operator block (a multiple of 16 bytes, 16-byte aligned) to shared memory
template <typename A>
__device__ __forceinline__ void load_block(A *dst, const A *src, int n, int nt)
{
  const float4 *g = reinterpret_cast<const float4 *>(src);
  float4 *d = reinterpret_cast<float4 *>(dst);
  for (int i = threadIdx.x; i < n * (int)sizeof(A) / 16; i += nt) d[i] = g[i];
}

// vol = sum_t (oppDiv[s][t] F~_0(t) + oppDiv[s][S + t] F~_1(t)); dv: the row's pairs
template <typename A, int N>
__device__ __forceinline__ void tri_divergence(const A *sF, const A *dv, int l, A vol[4])
{
  constexpr int S = TriShape<N>::S;
#pragma unroll
  for (int v = 0; v < 4; v++) vol[v] = A(0);
#pragma unroll
  for (int t = 0; t < S; t++)
  {
    A c0, c1, x0[4], x1[4];
    ld2(dv + 2 * t, c0, c1);
    ld4(sF + tvl<A>(t, l), x0);
    ld4(sF + tvl<A>(S + t, l), x1);
#pragma unroll
    for (int v = 0; v < 4; v++) vol[v] += c0 * x0[v] + c1 * x1[v];
  }
}

// surf = sum_f oppDiv_fpts[s][f] Fc(f)
template <typename A, int N>
__device__ __forceinline__ void tri_surface(const A *sFc, const A *dvf, int l, A surf[4])
{
  constexpr int Fp = TriShape<N>::Fp;
#pragma unroll
  for (int v = 0; v < 4; v++) surf[v] = A(0);
#pragma unroll
  for (int f = 0; f < Fp; f++)
  {
    A x[4];
    ld4(sFc + tvl<A>(f, l), x);
#pragma unroll
    for (int v = 0; v < 4; v++) surf[v] += dvf[f] * x[v];
  }
}

// traces of the updated state (sU, shared) for the next stage
template <typename T, typename A, int N>
__device__ __forceinline__ void tri_extrap_next(const Args<T, A> &a, int64_t tile, const A *sU, const A *E, int f,
                                                int l)
{
  A x[4];
  tri_extrap4<A, N>(sU, E, f, l, x);
  T *out = a.Ufp_next + (tile * TriShape<N>::Fp + f) * (int64_t)4 * TW + l;
#pragma unroll
  for (int v = 0; v < 4; v++) out[v * TW] = (T)x[v];
}

// State -> flux points (U_fpts = oppE U_spts), a thread per (flux point, element)
// reading its S values of every variable through L1.
template <typename T, typename A, int N>
__global__ void __launch_bounds__(128) k_tri_extrap_direct(const T *__restrict__ U, T *__restrict__ Ufp, int64_t ntiles,
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
    const int l = (int)(gid % TW), f = (int)((gid / TW) % Fp);
    const int64_t tile = gid / ((int64_t)TW * Fp);
    const T *u = U + tile * (int64_t)S * V * TW + l;
    T *out = Ufp + (tile * Fp + f) * (int64_t)V * TW + l;
#pragma unroll
    for (int v = 0; v < V; v++)
    {
      A acc = A(0);
#pragma unroll
      for (int t = 0; t < S; t++) acc += sE[f * S + t] * (A)u[(t * V + v) * TW];
      out[v * TW] = (T)acc;
    }
  }
}

// The same with the tile's state in shared memory: a flux point reads S 16-byte
// groups there instead of 4 S values, for two barriers per tile.  us, 2 n^2
// triangles, direct -> this form, FP64 and mixed: P4 n 110 18.6 -> 14.6 and 12.7
// -> 10.8, P3 n 110 12.6 -> 10.5 and 10.1 -> 8.7, P2 n 60 8.6 -> 6.6 and 7.0 ->
// 6.6, n 130 the same.  On large meshes the barriers outweigh the little work per
// tile: at P1 past 14 tiles per SM (n 90 the same, n 110 7.3 -> 8.6 and 6.6 ->
// 8.6, n 300 13.1 -> 16.0 and 11.6 -> 13.7), at P2 past 56 (n 160 12.7 -> 11.7 and
// 10.1 -> 10.2, n 300 24.9 -> 26.9 and 17.2 -> 19.4).
template <int N>
constexpr bool tri_extrap_direct(int64_t ntiles)
{
  return (N == 2 && ntiles > 148 * 14) || (N == 3 && ntiles > 148 * 56);
}

template <typename T, typename A, int N>
__global__ void __launch_bounds__(TriRun<A, N>::NT) k_tri_extrap(const T *__restrict__ U, T *__restrict__ Ufp,
                                                                 int64_t ntiles, const A *__restrict__ dops)
{
  using G = TriShape<N>;
  using R = TriRun<A, N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sE = reinterpret_cast<A *>(smem_raw);
  A *sU = sE + R::pad(Fp * S);
  load_block<A>(sE, dops + R::FACE_AT + R::FE, R::pad(Fp * S), R::NT);
  const int p = threadIdx.x / TW, l = threadIdx.x % TW;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
  {
    if (p < S)
    {
      const T *u = U + (tile * S + p) * (int64_t)V * TW + l;
      const A x[V] = {u[0], u[TW], u[2 * TW], u[3 * TW]};
      st4(sU + tvl<A>(p, l), x);
    }
    __syncthreads();
    if (p < Fp)
    {
      A x[V];
      tri_extrap4<A, N>(sU, sE, p, l, x);
      T *out = Ufp + (tile * Fp + p) * (int64_t)V * TW + l;
#pragma unroll
      for (int v = 0; v < V; v++) out[v * TW] = (T)x[v];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Euler: volume flux, common flux and divergence of one tile.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(TriRun<A, N>::NT, TriRun<A, N>::euler_minb)
    k_tri_euler(const __grid_constant__ Args<T, A> a)
{
  using G = TriShape<N>;
  using R = TriRun<A, N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, D = 2, NT = R::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sops = reinterpret_cast<A *>(smem_raw);
  A *sU = sops + R::euler_ops;  // [S] points: the updated state
  A *sF = sU + S * V * TW;
  A *sFc = sF + D * S * V * TW;
  load_block<A>(sops, a.dops + R::EULER_AT, R::euler_ops, NT);
  const int p = threadIdx.x / TW, l = threadIdx.x % TW;
  const bool has_s = p < S, has_f = p < Fp;
  for (int64_t tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x)
  {
    if (has_s)
    {
      const T *u = a.U + (tile * S + p) * (int64_t)V * TW + l;
      const T *m = a.mets + (tile * S + p) * (int64_t)5 * TW + l;
      A U[V], F[V][D], P, Pp;
#pragma unroll
      for (int v = 0; v < V; v++) U[v] = u[v * TW];
      const A adj[2][2] = {{m[0], m[TW]}, {m[2 * TW], m[3 * TW]}};
      flux_conv_stored<A, D>(U, F, P, Pp, a.ph);
      tri_transform<A>(F, adj, sF, S, p, l);
    }
    if (has_f)
    {
      A out[V];
      common_flux_2d<T, A, false>(a, tile, Fp, p, l, out);
      st4(sFc + tvl<A>(p, l), out);
    }
    __syncthreads();
    if (has_s)
    {
      RkIn<A, V> in;
      if (a.rk_mode) rk_load<T, A, S, V, 5>(a, tile, p, l, in);
      A res[V], surf[V], unew[V];
      tri_divergence<A, N>(sF, sops + R::EDV + 2 * p * S, l, res);
      tri_surface<A, N>(sFc, sops + R::EDVF + p * Fp, l, surf);
#pragma unroll
      for (int v = 0; v < V; v++) res[v] += surf[v];
      store_rk<T, A, S, V>(a, tile, p, l, res, in, unew);
      if (a.extrap_next) st4(sU + tvl<A>(p, l), unew);
    }
    __syncthreads();
    // the next tile's sU is written only after its own barrier, past this read
    if (a.extrap_next && has_f) tri_extrap_next<T, A, N>(a, tile, sU, sops + R::EE, p, l);
  }
}

// ---------------------------------------------------------------------------
// Navier-Stokes kernel 1: LDG common solution, corrected gradient, own viscous
// normal flux, volume flux and its divergence.  A point's flux follows its
// gradient from registers, so the faces need not wait before it.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(TriRun<A, N>::NT, TriRun<A, N>::grad_minb)
    k_tri_ns_grad(const __grid_constant__ Args<T, A> a)
{
  using G = TriShape<N>;
  using R = TriRun<A, N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, D = 2, NM = 5, NT = R::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sops = reinterpret_cast<A *>(smem_raw);
  A *sU = sops + R::grad_ops;    // [S] points
  A *sUC = sU + S * V * TW;      // [Fp] points
  A *sdU = sUC + Fp * V * TW;    // [D*S] points: physical gradient
  A *sF = sdU + D * S * V * TW;  // [D*S] points: transformed flux
  load_block<A>(sops, a.dops + R::GRAD_AT, R::grad_ops, NT);
  const int p = threadIdx.x / TW, l = threadIdx.x % TW;
  const bool has_s = p < S, has_f = p < Fp;
  for (int64_t tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x)
  {
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
      // oppD U, and apart from it oppD_fpts Ucomm, both dimensions at once
      A g0[V], g1[V], c0[V], c1[V];
#pragma unroll
      for (int v = 0; v < V; v++) g0[v] = g1[v] = c0[v] = c1[v] = A(0);
      const A *Dd = sops + R::GU + 2 * p * S;
#pragma unroll
      for (int t = 0; t < S; t++)
      {
        A k0, k1, x[4];
        ld2(Dd + 2 * t, k0, k1);
        ld4(sU + tvl<A>(t, l), x);
#pragma unroll
        for (int v = 0; v < V; v++)
        {
          g0[v] += k0 * x[v];
          g1[v] += k1 * x[v];
        }
      }
      const A *Df = sops + R::GF + 2 * p * Fp;
#pragma unroll
      for (int f = 0; f < Fp; f++)
      {
        A k0, k1, x[4];
        ld2(Df + 2 * f, k0, k1);
        ld4(sUC + tvl<A>(f, l), x);
#pragma unroll
        for (int v = 0; v < V; v++)
        {
          c0[v] += k0 * x[v];
          c1[v] += k1 * x[v];
        }
      }
#pragma unroll
      for (int v = 0; v < V; v++)
      {
        g0[v] += c0[v];
        g1[v] += c1[v];
      }
      const A inv_det = A(1) / det;
      A dU[V][D];
#pragma unroll
      for (int d1 = 0; d1 < D; d1++)
      {
        A g[V];
#pragma unroll
        for (int v = 0; v < V; v++)
        {
          g[v] = (g0[v] * adj[0][d1] + g1[v] * adj[1][d1]) * inv_det;
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
      A F[V][D], P, Pp, Ua[V];
      flux_conv_stored<A, D>(U, F, P, Pp, a.ph);
      to_abs<A, D>(U, Ua, a.ph);
      flux_visc_add<A, D>(Ua, dU, F, a.ph);
      tri_transform<A>(F, adj, sF, S, p, l);
    }
    __syncthreads();
    // own viscous normal flux at flux points
    if (has_f && own_visc_flux(a.ph.ldg_b, code))
    {
      A x0[V], x1[V], dUf[V][D];
#pragma unroll
      for (int v = 0; v < V; v++) x0[v] = x1[v] = A(0);
      const A *E = sops + R::GE + p * S;
#pragma unroll
      for (int t = 0; t < S; t++)
      {
        A y0[4], y1[4];
        ld4(sdU + tvl<A>(t, l), y0);
        ld4(sdU + tvl<A>(S + t, l), y1);
        const A e = E[t];
#pragma unroll
        for (int v = 0; v < V; v++)
        {
          x0[v] += e * y0[v];
          x1[v] += e * y1[v];
        }
      }
#pragma unroll
      for (int v = 0; v < V; v++)
      {
        dUf[v][0] = x0[v];
        dUf[v][1] = x1[v];
      }
      visc_face_2d<T, A>(a, tile, Fp, p, l, code, Uf, dUf, UC);
    }
    if (has_s)
    {
      A vol[V];
      tri_divergence<A, N>(sF, sops + R::GDV + 2 * p * S, l, vol);
      A *out = a.divF_vol + (tile * S + p) * (int64_t)V * TW + l;
#pragma unroll
      for (int v = 0; v < V; v++) out[v * TW] = vol[v];
    }
    // the next tile writes sU and sUC, last read before the barrier above, and
    // sdU and sF only after its own first barrier
  }
}

// ---------------------------------------------------------------------------
// Navier-Stokes kernel 2: convective + LDG common flux, correction, RK.
// ---------------------------------------------------------------------------
template <typename T, typename A, int N>
__global__ void __launch_bounds__(TriRun<A, N>::NT, TriRun<A, N>::face_minb)
    k_tri_ns_face(const __grid_constant__ Args<T, A> a)
{
  using G = TriShape<N>;
  using R = TriRun<A, N>;
  constexpr int S = G::S, Fp = G::Fp, V = G::V, NT = R::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *sops = reinterpret_cast<A *>(smem_raw);
  A *sFc = sops + R::face_ops;   // [Fp] points
  A *sUnew = sFc + Fp * V * TW;  // [S] points: the updated state
  load_block<A>(sops, a.dops + R::FACE_AT, a.extrap_next ? R::face_ops : R::FE, NT);
  const int p = threadIdx.x / TW, l = threadIdx.x % TW;
  const bool has_s = p < S, has_f = p < Fp;
  for (int64_t tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x)
  {
    RkIn<A, V> in;
    A res[V];
    if (has_s)
    {
      const A *dv = a.divF_vol + (tile * S + p) * (int64_t)V * TW + l;
#pragma unroll
      for (int v = 0; v < V; v++) res[v] = dv[v * TW];
      if (a.rk_mode) rk_load<T, A, S, V, 5>(a, tile, p, l, in);
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
      tri_surface<A, N>(sFc, sops + R::FDVF + p * Fp, l, surf);
#pragma unroll
      for (int v = 0; v < V; v++) res[v] += surf[v];
      store_rk<T, A, S, V>(a, tile, p, l, res, in, unew);
      if (a.extrap_next) st4(sUnew + tvl<A>(p, l), unew);
    }
    __syncthreads();
    // the next tile's sUnew is written only after its own barrier, past this read
    if (a.extrap_next && has_f) tri_extrap_next<T, A, N>(a, tile, sUnew, sops + R::FE, p, l);
  }
}

}  // namespace dev
}  // namespace zb
