// Launches of the triangle residual kernels.
#include "ctx_impl.cuh"
#include "tri_kernels.cuh"
#include "tri_tc_kernels.cuh"

namespace zb {

// Triangles: dense-operator kernels (tri_kernels.cuh)
template <typename T, typename A, int N>
static void launch_extrap_tri(Ctx &c)
{
  using R = dev::TriRun<A, N>;
  const T *U = (const T *)c.U;
  T *Ufp = (T *)c.Ufp[c.cur];
  const A *ops = (const A *)c.dops;
  ProfScope ps(c, ZB_K_EXTRAP);
  if (dev::tri_extrap_direct<N>(c.ntiles))
  {
    if constexpr (N <= 3)
      dev::k_tri_extrap_direct<T, A, N>
          <<<grid_for(c.ntiles * dev::TriShape<N>::Fp * TW, 128), 128, 0, c.stream>>>(U, Ufp, c.ntiles, ops);
  }
  else
  {
    set_smem(dev::k_tri_extrap<T, A, N>, R::extrap_smem);
    const unsigned grid = (unsigned)std::min<int64_t>(c.ntiles, (int64_t)148 * R::extrap_minb);
    dev::k_tri_extrap<T, A, N><<<grid, R::NT, R::extrap_smem, c.stream>>>(U, Ufp, c.ntiles, ops);
  }
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N>
static void launch_stage_tri(Ctx &c, const StageCfg &sc)
{
  using R = dev::TriRun<A, N>;
  const auto grid = [&](int minb) { return (unsigned)std::min<int64_t>(c.ntiles, (int64_t)148 * minb); };
  const Args<T, A> a = make_args<T, A>(c, sc);
  if (c.tc_err_host && *c.tc_err_host)
  {
    *c.tc_err_host = 0;
    ZB_THROW(ZB_ERR_CUDA, "a tensor-core completion wait of an earlier launch timed out");
  }
  if (!c.plan.params.viscous)
  {
    set_smem(dev::k_tri_euler<T, A, N>, R::euler_smem);
    ProfScope ps(c, ZB_K_EULER);
    dev::k_tri_euler<T, A, N><<<grid(R::euler_minb), R::NT, R::euler_smem, c.stream>>>(a);
    c.launches++;
    CK(cudaGetLastError());
  }
  else
  {
    if (!sc.face_only)
    {
      ProfScope ps(c, ZB_K_NS_GRAD);
      bool launched = false;
      if constexpr (std::is_same<A, float>::value && N <= 5)
      {
        if (c.plan.params.tensor_ops)
        {
          using C = dev::TriTc<N>;
          set_smem(dev::k_tri_ns_grad_tc<N>, C::SMEM);
          const int64_t groups = (c.ntiles + C::TILES - 1) / C::TILES;
          dev::k_tri_ns_grad_tc<N><<<(unsigned)groups, C::NT, C::SMEM, c.stream>>>(a);
          launched = true;
        }
      }
      if (!launched)
      {
        set_smem(dev::k_tri_ns_grad<T, A, N>, R::grad_smem);
        dev::k_tri_ns_grad<T, A, N><<<grid(R::grad_minb), R::NT, R::grad_smem, c.stream>>>(a);
      }
      c.launches++;
      CK(cudaGetLastError());
    }
    if (sc.grad_only) return;
    set_smem(dev::k_tri_ns_face<T, A, N>, R::face_smem);
    ProfScope ps(c, ZB_K_NS_FACE);
    dev::k_tri_ns_face<T, A, N><<<grid(R::face_minb), R::NT, R::face_smem, c.stream>>>(a);
    c.launches++;
    CK(cudaGetLastError());
  }
  if (sc.extrap_next) c.cur ^= 1;
}

template <typename T, typename A>
static void bind_tri_t(Ctx &c)
{
#define ZB_BIND_TRI(NN)                             \
  case NN:                                          \
    c.launch_extrap = &launch_extrap_tri<T, A, NN>; \
    c.launch_stage = &launch_stage_tri<T, A, NN>;   \
    break;
  switch (c.N)
  {
    ZB_BIND_TRI(2) ZB_BIND_TRI(3) ZB_BIND_TRI(4) ZB_BIND_TRI(5) ZB_BIND_TRI(6) ZB_BIND_TRI(7) ZB_BIND_TRI(8)
    ZB_BIND_TRI(9)
    default: break;
  }
#undef ZB_BIND_TRI
}

void bind_tri(Ctx &c)
{
  if (c.prec == ZB_FP64)
    bind_tri_t<double, double>(c);
  else
    bind_tri_t<float, float>(c);
}

}  // namespace zb
