// Host-side check of the launch shapes that are written as rules: wherever a
// kernel's registers are held to a number of CTAs per SM, that many fit the
// SM's 228 KB of shared memory (1 KB of it reserved per CTA) and its 2,048
// threads; a tighter bound only spills registers.
#include <cstdio>

#include "../../zefr_b200/csrc/hex_kernels.cuh"
#include "../../zefr_b200/csrc/quad_kernels.cuh"
#include "../../zefr_b200/csrc/tri_adjoint.cuh"

using namespace zb::dev;

static int g_bad = 0;

static void held(const char *what, int N, int esz, int ctas, size_t smem, int threads)
{
  if (ctas <= 1) return;
  if (ctas * (smem + 1024) > 228 * 1024 || ctas * threads > 2048)
  {
    std::printf("%s P%d, %d-byte values: %d CTAs of %zu bytes and %d threads\n", what, N - 1, esz, ctas, smem, threads);
    g_bad++;
  }
}

template <typename A, int N>
static void tri_forward()
{
  using R = TriRun<A, N>;
  held("tri gradient", N, sizeof(A), R::grad_minb, R::grad_smem, R::NT);
  held("tri face", N, sizeof(A), R::face_minb, R::face_smem, R::NT);
  held("tri Euler", N, sizeof(A), R::euler_minb, R::euler_smem, R::NT);
}

template <int N>
static void tri()
{
  tri_forward<double, N>();
  tri_forward<float, N>();
  held("tri adjoint", N, 8, TriAdjRun<N>::minb, TriAdjRun<N>::ns1_smem, TriAdjRun<N>::ns1_nt);
}

template <typename A, int N>
static void quad()
{
  using O = QuadOcc<A, N>;
  held("quad gradient", N, sizeof(A), O::grad, quad_grad_smem_elems<N>() * sizeof(A), QuadShape<N>::NT);
  held("quad face", N, sizeof(A), O::face_many, quad_face_smem_elems<N>() * sizeof(A), QuadShape<N>::NT);
  held("quad Euler", N, sizeof(A), O::euler, euler_smem_elems<N>() * sizeof(A), QuadShape<N>::NT);
}

int main()
{
  tri<2>();
  tri<3>();
  tri<4>();
  tri<5>();
  tri<6>();
  tri<7>();
  tri<8>();
  tri<9>();
  quad<double, 2>();
  quad<double, 3>();
  quad<double, 4>();
  quad<double, 5>();
  quad<double, 6>();
  quad<float, 2>();
  quad<float, 3>();
  quad<float, 4>();
  quad<float, 5>();
  quad<float, 6>();
  std::printf("%d shapes held too tight\n", g_bad);
  return g_bad ? 1 : 0;
}
