// Launches of the hexahedral residual kernels of one arithmetic type.
#pragma once
#include "ctx_impl.cuh"
#include "hex_kernels.cuh"
#include "time_kernels.cuh"

namespace zb {

// column-mapped kernels: TW x N^2 threads per tile, times the threads that share
// a column
template <typename T, typename A, int N, int ZS, int MINB>
static void launch_euler_hex(Ctx &c, const Args<T, A> &a, const LineOpsT<A, N> &ops)
{
  using G = Shape<3, N>;
  const size_t smem = (size_t)(4 * G::S * G::V + G::Fp * G::V) * TW * sizeof(A);
  set_smem(dev::k_hex_euler<T, A, N, ZS, MINB>, smem);
  ProfScope ps(c, ZB_K_EULER);
  dev::k_hex_euler<T, A, N, ZS, MINB><<<(unsigned)c.ntiles, TW * N * N * ZS, smem, c.stream>>>(a, ops);
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N, int MINB>
static void launch_grad_hex(Ctx &c, const Args<T, A> &a, const LineOpsT<A, N> &ops)
{
  using G = Shape<3, N>;
  const size_t smem = (size_t)((4 * G::S * G::V + G::Fp * G::V) * TW + 3 * N * TW) * sizeof(A);  // + sX padding
  set_smem(dev::k_hex_ns_grad<T, A, N, MINB>, smem);
  ProfScope ps(c, ZB_K_NS_GRAD);
  dev::k_hex_ns_grad<T, A, N, MINB>
      <<<(unsigned)c.ntiles, TW * N * N * dev::HexNsShape<A, N>::grad_zs, smem, c.stream>>>(a, ops);
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N, bool ONE, bool RK>
static void launch_face_hex(Ctx &c, const Args<T, A> &a, const LineOpsT<A, N> &ops)
{
  using G = Shape<3, N>;
  const size_t smem = (size_t)(G::Fp * G::V + (RK && !ONE ? G::S * G::V : 0)) * TW * sizeof(A);
  set_smem(dev::k_hex_ns_face<T, A, N, ONE, RK>, smem);
  ProfScope ps(c, ZB_K_NS_FACE);
  dev::k_hex_ns_face<T, A, N, ONE, RK>
      <<<(unsigned)c.ntiles, TW * N * N * dev::HexFaceShape<A, N, ONE, RK>::zs, smem, c.stream>>>(a, ops);
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N>
static void launch_extrap_hex(Ctx &c)
{
  ProfScope ps(c, ZB_K_EXTRAP);
  dev::k_hex_extrap<T, A, N><<<(unsigned)c.ntiles, TW * N * N, 0, c.stream>>>((const T *)c.U, (T *)c.Ufp[c.cur],
                                                                              c.ntiles, line_ops<A, N>(c.plan));
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N>
static void launch_stage_hex(Ctx &c, const StageCfg &sc)
{
  const Args<T, A> a = make_args<T, A>(c, sc);
  const LineOpsT<A, N> ops = line_ops<A, N>(c.plan);
  if (!c.plan.params.viscous)
  {
    using E = dev::HexEulerShape<A, N>;
    if (E::few(c.ntiles))
      launch_euler_hex<T, A, N, E::few_zs, E::few_minb>(c, a, ops);
    else
      launch_euler_hex<T, A, N, E::zs, E::minb>(c, a, ops);
  }
  else
  {
    using G1 = dev::HexNsShape<A, N>;
    if (!sc.face_only)
    {
      if (c.ntiles > (int64_t)148 * G1::grad_few)
        launch_grad_hex<T, A, N, G1::grad_minb>(c, a, ops);
      else
        launch_grad_hex<T, A, N, G1::grad_few>(c, a, ops);
    }
    if (sc.grad_only) return;
    if (a.Fcom)
      a.rk_mode ? launch_face_hex<T, A, N, true, true>(c, a, ops) : launch_face_hex<T, A, N, true, false>(c, a, ops);
    else
      a.rk_mode ? launch_face_hex<T, A, N, false, true>(c, a, ops) : launch_face_hex<T, A, N, false, false>(c, a, ops);
  }
  if (sc.extrap_next)
  {
    if (a.Fcom)
      c.ufp_valid = false;  // the state changed and no traces were stored
    else
      c.cur ^= 1;
  }
}

template <typename T, typename A, int N>
static void bind_hex_order(Ctx &c)
{
  c.launch_extrap = &launch_extrap_hex<T, A, N>;
  c.launch_stage = &launch_stage_hex<T, A, N>;
  c.launch_dt = &launch_dt_impl<T, A, 3, N>;
}

template <typename T, typename A>
static void bind_hex(Ctx &c)
{
  switch (c.N)
  {
    case 2: bind_hex_order<T, A, 2>(c); break;
    case 3: bind_hex_order<T, A, 3>(c); break;
    case 4: bind_hex_order<T, A, 4>(c); break;
    case 5: bind_hex_order<T, A, 5>(c); break;
    default: break;
  }
}

}  // namespace zb
