// Host-side check of the boundary face reverse (bnd_face_vjp) and its
// free-stream part against forward-mode dual numbers through the whole face
// function: common flux with the ghost state, viscous normal flux of the
// prescribed state and gradient, LDG penalty.  The reverse adds to sums that
// already hold values, as in the kernels, and the Rusanov dissipation is scaled
// by 1 - rus_k.  Prints the worst relative error and exits non-zero above 1e-12
// (values and weights of order one; a few hundred rounded operations of 1e-16
// each).
#include <cstdio>
#include <cstring>
#include <random>

#include "../../zefr_b200/csrc/adjoint.cuh"

using namespace zb::dev;
using DD = Dual<double>;

static double g_worst = 0.0;

static void record(int bc, double a, double b)
{
  const double e = std::fabs(a - b) / std::fmax(1.0, std::fmax(std::fabs(a), std::fabs(b)));
  if (!(e <= g_worst)) g_worst = e;
  if (!(e <= 1e-12)) std::printf("MISMATCH bc %d: %.17g vs %.17g\n", bc, a, b);
}

template <int D, bool VISC>
static void face(int bc, const DD U[D + 2], const DD dU[D + 2][D], const DD n[D], const Phys<DD> &ph, DD F[D + 2])
{
  constexpr int V = D + 2;
  conv_face<D, DD>(bc, U, U, n, F, ph);
  if (!VISC) return;
  DD UR[V], UB[V], dUB[V][D], Fn[V];
  ghost_state<DD, D>(bc, U, n, UR, UB, ph);
  ghost_grad<DD, D>(bc, U, dU, n, dUB);
  visc_normal<DD, D>(UB, dUB, n, Fn, ph);
  for (int v = 0; v < V; v++) F[v] += Fn[v] + ph.ldg_tau * (U[v] - UB[v]);
}

template <int D, bool VISC>
static void check(std::mt19937_64 &rng, int bc, int fconv, bool sutherland, double mach, double rus_k)
{
  constexpr int V = D + 2;
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  Phys<double> ph;
  std::memset(&ph, 0, sizeof(ph));
  ph.gamma = 1.4;
  ph.prandtl = 0.71;
  ph.mu = 0.31;
  ph.rt = 0.7;
  ph.c_sth = 0.37;
  ph.fix_vis = sutherland ? 0 : 1;
  ph.fconv = fconv;
  ph.ldg_tau = 0.1;
  ph.rus_k = rus_k;
  ph.rho_fs = 1.1;
  ph.P_fs = 0.9;
  ph.T_wall = 1.2;
  ph.R_ref = 0.8;
  double n[D], nn = 0.0, U[V], dU[V][D], w[V], m2 = 0.0;
  for (int d = 0; d < D; d++)
  {
    ph.V_fs[d] = mach * u(rng);
    ph.V_wall[d] = 0.3 * u(rng);
    n[d] = u(rng);
    nn += n[d] * n[d];
  }
  for (int d = 0; d < D; d++) n[d] /= std::sqrt(nn);
  U[0] = 1.0 + 0.3 * u(rng);
  for (int d = 0; d < D; d++)
  {
    U[d + 1] = mach * u(rng);
    m2 += U[d + 1] * U[d + 1];
  }
  U[V - 1] = 2.5 + 0.5 * m2 / U[0] + 0.2 * u(rng);
  for (int v = 0; v < V; v++)
  {
    w[v] = u(rng);
    for (int d = 0; d < D; d++) dU[v][d] = u(rng);
  }
  // the sums before the call
  double Ub0[V], dUb0[V][D], pb0[5], Ub[V], dUb[V][D], pb[5];
  for (int v = 0; v < V; v++)
  {
    Ub[v] = Ub0[v] = u(rng);
    for (int d = 0; d < D; d++) dUb[v][d] = dUb0[v][d] = u(rng);
  }
  for (int k = 0; k < 5; k++) pb[k] = pb0[k] = u(rng);
  bnd_face_vjp<D, VISC>(bc, U, dU, n, w, ph, Ub, dUb, pb);
  const int np = bc_uses_freestream(bc) ? 5 : 0;
  for (int k = 0; k < V + V * D + np; k++)
  {
    const int kp = k - V - V * D;
    if (kp >= 1 && kp <= 3 && kp > D) continue;
    Phys<DD> q = dual_phys(ph);
    if (kp >= 0) seed_param(q, kp);
    DD L[V], dL[V][D], nd[D], F[V];
    for (int d = 0; d < D; d++) nd[d] = DD(n[d]);
    for (int v = 0; v < V; v++)
    {
      L[v] = DD(U[v], v == k ? 1.0 : 0.0);
      for (int d = 0; d < D; d++) dL[v][d] = DD(dU[v][d], k == V + v * D + d ? 1.0 : 0.0);
    }
    face<D, VISC>(bc, L, dL, nd, q, F);
    double acc = 0.0;
    for (int v = 0; v < V; v++) acc += w[v] * F[v].d;
    const int v = (k - V) / D, d = (k - V) % D;
    record(bc, kp >= 0 ? pb[kp] : k < V ? Ub[k] : dUb[v][d],
           (kp >= 0 ? pb0[kp] : k < V ? Ub0[k] : dUb0[v][d]) + acc);
  }
  // parameters that the face does not depend on keep their sums
  for (int k = 0; k < 5; k++)
    if (np == 0 || (k >= 1 && k <= 3 && k > D)) record(bc, pb[k], pb0[k]);
}

int main()
{
  std::mt19937_64 rng(7);
  const int bcs[] = {2, 3, 4, 5, 6, 7, 8, 9, 11};
  for (int rep = 0; rep < 200; rep++)
    for (int bc : bcs)
      for (int fconv : {0, 2})
      {
        const double mach = rep % 2 ? 0.4 : 2.0;  // sub- and supersonic far fields
        const double rus_k = rep % 4 < 2 ? 0.0 : 0.35;
        check<2, true>(rng, bc, fconv, rep % 3 == 0, mach, rus_k);
        check<3, true>(rng, bc, fconv, rep % 3 == 1, mach, rus_k);
        check<2, false>(rng, bc, fconv, false, mach, rus_k);
        check<3, false>(rng, bc, fconv, false, mach, rus_k);
      }
  std::printf("worst relative error %.3g\n", g_worst);
  return g_worst <= 1e-12 ? 0 : 1;
}
