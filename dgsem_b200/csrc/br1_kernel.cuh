// Viscous flux of the Navier-Stokes equations from the BR1 lifted gradient,
// one kernel per stage, 2D (periodic or with wall faces) and 3D (periodic):
//   q = (v, T = p / rho) at nodes       compressible_navier_stokes2D.hpp:56-69, 3D :55-70
//   weak-form volume term with Dhat     parabolic_gradient.hpp:509-532, 3D :17-95
//   interface average q^ = (q- + q+)/2  parabolic_gradient.hpp:620-686, 3D :159-307
//   lifting, transform with Ja, * 1/J   parabolic_gradient.hpp:573-585, 712-818, 3D :100-437
//   -F_v at the node                    compressible_navier_stokes2D.hpp:71-106, 3D :72-124
// Output: the contravariant flux visc[e][dir][r][node] = Ja^dir . (-F_v)_r at
// every node, r = 0 .. DIM-1 the momentum rows, DIM the energy row (the mass
// row is zero).  That is all the stage kernel needs: its volume term is a
// Dhat product of visc^dir along the line, and the one-sided interface flux
// -F_v . n of the high-side element at its low face (parabolic_viscous.hpp:
// 570-585) is that element's visc^dir there.  So the flux is formed once per
// node instead of once per node, face and neighbour, and 6 (2D) or 12 (3D)
// doubles per node are written and read.
//
// The kernel is a line sweep (stage_line_kernel.cuh): a warp owns whole
// elements, a lane one line per direction; the derivative of q along the line
// with the averages at its two ends goes to a shared plane per direction, and
// the lanes then combine the directions node by node.  B200, us per stage,
// gradient kernel + stage kernel before (one thread per node, the divergent
// faces inside every warp: 7.8 M warp instructions for the gradient of TGV
// 16^3; -F_v recomputed at every face) -> now:
//   3D Taylor-Green 16^3, n = 4    63.1 -> 30.5 (line sweep; node shape 43)
//   2D 32 x 32, n = 5 (adjoint)    14.6 -> 11.8 (node shape)
#pragma once

#include "stage_line_kernel.cuh"

namespace dgsem {

__device__ __forceinline__ void ns_gradient_variables(const double* u, double gamma,
                                                      double* q) {
  const double rho = u[0];
  const double inv_rho = recip(rho);
  const double v1 = u[1] * inv_rho;
  const double v2 = u[2] * inv_rho;
  const double p = (gamma - 1.0) * (u[3] - 0.5 * (u[1] * u[1] + u[2] * u[2]) * inv_rho);
  q[0] = rho;
  q[1] = v1;
  q[2] = v2;
  q[3] = p * inv_rho;
}

template <int N>
struct ViscArgs {
  const double* u;
  double* visc;  // [E][DIM][DIM + 1][ND] (may be null)
  double* grad;  // adjoint (2D): velocity gradient [E][2][2][ND] (may be null)
  int nelem;
  double gamma, mu, kappa;
  DeviceTables tab;
  const int* info;    // element info (MeshView::info)
  const double* mij;  // -1/J per node
  BasisConst<N> basis;
  int bc_kind[6];  // BcKind per face; faces without a neighbour are walls (2D)
};

template <int DIM, int N>
struct ViscShape {
  using G = LineGeo<DIM, N>;
  static constexpr int NQ = DIM + 1;  // v, T
  static constexpr int WPB = 4;
  static constexpr int EPB = G::EPW * WPB;
  static constexpr int WARP_DOUBLES = (NQ + DIM * NQ) * G::PLANE;
  static constexpr size_t smem_bytes = sizeof(double) * (size_t)WARP_DOUBLES * WPB;
};

// (v, T) from conserved variables.
template <int DIM>
__device__ __forceinline__ void visc_variables(const double* u, double gm1, double* q) {
  const double inv = recip(u[0]);
#pragma unroll
  for (int d = 0; d < DIM; ++d) q[d] = __dmul_rn(u[1 + d], inv);
  const double m2 = line_dot<DIM>(u + 1, q);
  q[DIM] = __dmul_rn(__dmul_rn(gm1, __fma_rn(-0.5, m2, u[DIM + 1])), inv);
}

template <int DIM, int N>
__device__ __forceinline__ void viscous_flux_body(const ViscArgs<N>& p) {
  using S = ViscShape<DIM, N>;
  using G = LineGeo<DIM, N>;
  constexpr int NV = G::NV, ND = G::ND, NF = G::NF, PLANE = G::PLANE, NQ = S::NQ;
  extern __shared__ __align__(128) double smem_visc[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* Q = smem_visc + warp * S::WARP_DOUBLES;
  double* Dq = Q + NQ * PLANE;  // [dir][var]
  const int e0 = (int)blockIdx.x * S::EPB, eb = min(S::EPB, p.nelem - e0);
  const int ew = e0 + warp * G::EPW, ne = min(G::EPW, p.nelem - ew);
  const int el = lane / NF, line = lane - el * NF;
  const bool act = el < ne;
  const int e = act ? ew + el : 0;
  const int* info = p.info + (int64_t)e * 12;
  int row[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) row[c] = __ldg(info + 3 + c);
  stage_dependency_sync();
  const double gm1 = p.gamma - 1.0;
  LinePos<DIM, N> pos;

  // ---- (v, T) of the x lines ----------------------------------------------
  if (act) {
    pos.set(0, el, line);
    const double* src = p.u + (int64_t)e * (NV * ND) + N * line;
    double u[NV][N];
    if ((reinterpret_cast<uintptr_t>(p.u) & line_vec_mask<N>()) == 0) {
#pragma unroll
      for (int v = 0; v < NV; ++v) load_xline<N, true>(src + v * ND, u[v]);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) load_xline<N, false>(src + v * ND, u[v]);
    }
    double q[NQ][N];
#pragma unroll
    for (int m = 0; m < N; ++m) {
      double un[NV], qn[NQ];
#pragma unroll
      for (int v = 0; v < NV; ++v) un[v] = u[v][m];
      visc_variables<DIM>(un, gm1, qn);
#pragma unroll
      for (int v = 0; v < NQ; ++v) q[v][m] = qn[v];
    }
#pragma unroll
    for (int v = 0; v < NQ; ++v) store_line<true, N>(Q + v * PLANE, pos.off, q[v]);
  }
  __syncthreads();  // the block's planes are published

  // ---- derivative along every line, with the averages at its ends ----------
#pragma unroll(N > 4 ? 1 : DIM)
  for (int dir = 0; dir < DIM; ++dir) {
    if (!act) break;
    pos.set(dir, el, line);
    int nb[2];
    nb[0] = __ldg(info + 6 + 2 * dir);
    nb[1] = __ldg(info + 7 + 2 * dir);
    double hat[2][NQ];  // far-side values
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int be = nb[s] - e0;
      if (dir == 0 && be >= 0 && be < eb) {
        const int w = be / G::EPW;
        const double* T = smem_visc + w * S::WARP_DOUBLES +
                          LinePos<DIM, N>::slot(0, be - w * G::EPW, line, s ? 0 : N - 1);
#pragma unroll
        for (int v = 0; v < NQ; ++v) hat[s][v] = T[v * PLANE];
      } else {
        const double* T = p.u + (int64_t)max(nb[s], 0) * (NV * ND) + pos.first +
                          (s ? 0 : (N - 1) * pos.stride);
        double un[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) un[v] = __ldg(T + v * ND);
        visc_variables<DIM>(un, gm1, hat[s]);
      }
    }
    double q[NQ][N];
#pragma unroll
    for (int v = 0; v < NQ; ++v) load_line<false, N>(Q + v * PLANE, pos.off, q[v]);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int m = s ? N - 1 : 0;
      if (DIM == 2 && nb[s] < 0) {
        // wall: q^ = q of the wall state (navier_stokes_wall_boundary.hpp:
        // 82-99 no-slip: velocity zero; :162-190 slip: the normal velocity
        // removed along the element's own face normal)
#pragma unroll
        for (int v = 0; v < NQ; ++v) hat[s][v] = q[v][m];
        if (p.bc_kind[2 * dir + s] == BC_NS_NOSLIP_ADIABATIC_WALL) {
          hat[s][0] = 0.0;
          hat[s][1] = 0.0;
        } else {
          double n[2];
#pragma unroll
          for (int c = 0; c < 2; ++c)
            n[c] = __ldg(p.tab.ja[dir][c] + (int64_t)row[c] * ND + pos.first + m * pos.stride);
          const double vn = (q[0][m] * n[0] + q[1][m] * n[1]) / (n[0] * n[0] + n[1] * n[1]);
          hat[s][0] -= vn * n[0];
          hat[s][1] -= vn * n[1];
        }
      } else {
#pragma unroll
        for (int v = 0; v < NQ; ++v) hat[s][v] = 0.5 * (q[v][m] + hat[s][v]);
      }
    }
#pragma unroll
    for (int v = 0; v < NQ; ++v) {
      double d[N];
#pragma unroll
      for (int m = 0; m < N; ++m) {
        double s = __dmul_rn(p.basis.Dhat[m][0], q[v][0]);
#pragma unroll
        for (int k = 1; k < N; ++k) s = __fma_rn(p.basis.Dhat[m][k], q[v][k], s);
        d[m] = s;
      }
      d[0] = __fma_rn(-p.basis.lhat_l0, hat[0][v], d[0]);
      d[N - 1] = __fma_rn(p.basis.lhat_rN, hat[1][v], d[N - 1]);
      store_line<false, N>(Dq + (dir * NQ + v) * PLANE, pos.off, d);
    }
  }
  __syncwarp();

  // ---- gradient, -F_v and its contravariant components, node by node along
  // the lines of the last direction (their nodes are contiguous over lanes) ---
  if (!act) return;
  pos.set(DIM - 1, el, line);
#pragma unroll(N > 4 ? 2 : N)
  for (int m = 0; m < N; ++m) {
    int o = LinePos<DIM, N>::slot(DIM - 1, el, line, m);
    const int node = pos.first + m * pos.stride;
    double ja[DIM][DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int c = 0; c < DIM; ++c)
        ja[a][c] = __ldg(p.tab.ja[a][c] + (int64_t)row[c] * ND + node);
    const double inv_j = -__ldg(p.mij + (int64_t)e * ND + node);
    double g[DIM][NQ];  // d q_v / d x_c
#pragma unroll
    for (int v = 0; v < NQ; ++v) {
      double d[DIM];
#pragma unroll
      for (int a = 0; a < DIM; ++a) d[a] = Dq[(a * NQ + v) * PLANE + o];
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        double s = __dmul_rn(ja[0][c], d[0]);
#pragma unroll
        for (int a = 1; a < DIM; ++a) s = __fma_rn(ja[a][c], d[a], s);
        g[c][v] = __dmul_rn(s, inv_j);
      }
    }
    if constexpr (DIM == 2) {
      if (p.grad) {
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
          for (int c = 0; c < 2; ++c)
            p.grad[(((int64_t)e * 2 + v) * 2 + c) * ND + node] = g[c][v];
      }
    }
    if (!p.visc) continue;
    // -F_v: w[c][r] = -mu tau_rc, energy -mu (v . tau_c + kappa dT/dx_c)
    double w[DIM][NQ];
    double trace = g[0][0];
#pragma unroll
    for (int c = 1; c < DIM; ++c) trace += g[c][c];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      double en = __dmul_rn(p.kappa, g[c][DIM]);
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        // (4 d_c v_c - 2 sum of the others) / 3 = 2 d_c v_c - 2/3 trace
        const double tau = r == c ? __fma_rn(-2.0 / 3.0, trace, 2.0 * g[c][c]) : g[c][r] + g[r][c];
        en = __fma_rn(Q[r * PLANE + o], tau, en);
        w[c][r] = -(p.mu * tau);
      }
      w[c][DIM] = -(p.mu * en);
    }
    double* out = p.visc + (int64_t)e * (DIM * NQ * ND) + node;
#pragma unroll
    for (int a = 0; a < DIM; ++a)
#pragma unroll
      for (int r = 0; r < NQ; ++r) {
        double s = __dmul_rn(ja[a][0], w[0][r]);
#pragma unroll
        for (int c = 1; c < DIM; ++c) s = __fma_rn(ja[a][c], w[c][r], s);
        out[(a * NQ + r) * ND] = s;
      }
  }
}

template <int DIM, int N>
__global__ void __launch_bounds__(32 * ViscShape<DIM, N>::WPB, 4)
    viscous_flux_kernel(const ViscArgs<N> p) {
  viscous_flux_body<DIM, N>(p);
}

}  // namespace dgsem
