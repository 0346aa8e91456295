// Launches of the quadrilateral residual kernels.
#include "ctx_impl.cuh"
#include "quad_kernels.cuh"
#include "time_kernels.cuh"

namespace zb {

template <typename T, typename A, int N>
static void launch_extrap_quad(Ctx &c)
{
  const int64_t work = c.ntiles * dev::QuadShape<N>::Fp * TW;
  ProfScope ps(c, ZB_K_EXTRAP);
  dev::k_extrap<T, A, N><<<grid_for(work, 256), 256, 0, c.stream>>>((const T *)c.U, (T *)c.Ufp[c.cur], c.ntiles,
                                                                       line_ops<A, N>(c.plan));
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N, int MINB>
static void launch_face_quad(Ctx &c, const Args<T, A> &a, const LineOpsT<A, N> &ops)
{
  const size_t smem = dev::quad_face_smem_elems<N>() * sizeof(A);
  set_smem(dev::k_ns_face<T, A, N, MINB>, smem);
  ProfScope ps(c, ZB_K_NS_FACE);
  dev::k_ns_face<T, A, N, MINB><<<(unsigned)c.ntiles, dev::QuadShape<N>::NT, smem, c.stream>>>(a, ops);
  c.launches++;
  CK(cudaGetLastError());
}

template <typename T, typename A, int N>
static void launch_stage_quad(Ctx &c, const StageCfg &sc)
{
  constexpr int NT = dev::QuadShape<N>::NT;
  const Args<T, A> a = make_args<T, A>(c, sc);
  const LineOpsT<A, N> ops = line_ops<A, N>(c.plan);
  if (!c.plan.params.viscous)
  {
    const size_t smem = dev::euler_smem_elems<N>() * sizeof(A);
    set_smem(dev::k_euler<T, A, N>, smem);
    ProfScope ps(c, ZB_K_EULER);
    dev::k_euler<T, A, N><<<(unsigned)c.ntiles, NT, smem, c.stream>>>(a, ops);
    c.launches++;
    CK(cudaGetLastError());
  }
  else
  {
    const size_t smem1 = dev::quad_grad_smem_elems<N>() * sizeof(A);
    set_smem(dev::k_ns_grad<T, A, N>, smem1);
    if (!sc.face_only)
    {
      ProfScope ps(c, ZB_K_NS_GRAD);
      dev::k_ns_grad<T, A, N><<<(unsigned)c.ntiles, NT, smem1, c.stream>>>(a, ops);
      c.launches++;
      CK(cudaGetLastError());
    }
    if (sc.grad_only) return;
    using O = dev::QuadOcc<A, N>;
    if (c.ntiles > 148)
      launch_face_quad<T, A, N, O::face_many>(c, a, ops);
    else
      launch_face_quad<T, A, N, O::face>(c, a, ops);
  }
  if (sc.extrap_next) c.cur ^= 1;
}

template <typename T, typename A, int N>
static void bind_quad_order(Ctx &c)
{
  c.launch_extrap = &launch_extrap_quad<T, A, N>;
  c.launch_stage = &launch_stage_quad<T, A, N>;
  c.launch_dt = &launch_dt_impl<T, A, 2, N>;
}

template <typename T, typename A>
static void bind_quad_t(Ctx &c)
{
  switch (c.N)
  {
    case 2: bind_quad_order<T, A, 2>(c); break;
    case 3: bind_quad_order<T, A, 3>(c); break;
    case 4: bind_quad_order<T, A, 4>(c); break;
    case 5: bind_quad_order<T, A, 5>(c); break;
    case 6: bind_quad_order<T, A, 6>(c); break;
    default: break;
  }
}

void bind_quad(Ctx &c)
{
  if (c.prec == ZB_FP64)
    bind_quad_t<double, double>(c);
  else
    bind_quad_t<float, float>(c);
}

}  // namespace zb
