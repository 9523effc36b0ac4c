// Shared parts of the fused DGSEM stage kernels for sm_100a: one launch
// computes, per element,
//   RHS(u_in) = -1/J [ sum_dir V_dir(u_in) + surface lift ]
// and writes either du or the SSPRK3 stage value a*u_n + b*u_in + c*du.
// Here: launch arguments, element and node indices, the Hennemann-Gassner
// indicator, the fused diagnostics, boundary states and the interface flux of
// the node-parallel kernels.  The kernels: stage_line_kernel.cuh (line
// sweeps), stage_node_kernel.cuh, stage_node2_kernel.cuh, stage_pipe_kernel.cuh
// (one or two nodes per thread).
// Reference path replaced (one Kokkos kernel per item, :line):
//   deep_copy(du, 0)                         solver/structured_solver.hpp:469
//   HGIndicator2D                            subcell_limiting/indicator.hpp:337-418
//   VolumeIntegralSplit / FinitVolumeIntegral space_integral/volume_flux.hpp:221-511
//   VolumeIntegralShockCapturingHG blend     space_integral/volume_flux.hpp:817-842
//   InterfaceHelper::interface_flux          space_integral/surface_flux.hpp:45-271
//   BC_Apply (Dirichlet/Outflow/Mixed)       boundary_condition/*.hpp
//   SurfaceIntegral::integral                space_integral/surface_integral.hpp:35-154
//   JacobianProjFunctor                      space_integral/jacobian.hpp:76-101
//   parallel_ma2 / parallel_ma3              time_integrator/SSPRK3.hpp:12-143
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "physics.cuh"

namespace dgsem {

__host__ __device__ constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }

template <int N>
struct BasisConst {
  double Dsplit[N][N];
  double Dvol[N][N];  // Dsplit / 4 (Kennedy-Gruber) or / 2: line_pair_flux
  double Dhat[N][N];
  double Vinv[N][N];
  double inv_w[N];
  double w[N];     // quadrature weights (fused diagnostics)
  double lhat_l0;  // l_0(-1) / w_0
  double lhat_rN;  // l_N(+1) / w_N
};

struct DeviceTables {
  const double* ja[3][3];  // ja[a][c]: [eidx_c][node]
  const double* jdiag[3];  // [e_a * n + i]
  const double* coord[3];  // [e_a * n + i]
  const double* fv[3][3];  // FV subcell normals [eidx_c][f * n^(d-1) + line]
};

enum BcKind : int {
  BC_PERIODIC = 0,
  BC_DIRICHLET_DMR = 1,
  BC_OUTFLOW = 2,
  BC_MIXED_DMR_WALL = 3,
  BC_DIRICHLET_CONST = 4,
  BC_SLIP_WALL = 5,
  BC_NS_NOSLIP_ADIABATIC_WALL = 6,  // navier_stokes_wall_boundary.hpp:33-132
  BC_NS_SLIP_ADIABATIC_WALL = 7     // navier_stokes_wall_boundary.hpp:134-219
};

struct BcParams {
  int kind[6];
  double state[4];     // DIRICHLET_CONST conserved state
  double dmr_post[4];  // conserved post-shock state
  double dmr_pre[4];   // conserved pre-shock state
  double sqrt3;
};

// Per-mesh data of one stage launch.  Single-mesh launches read it from the
// kernel parameters; in batched launches each block copies its mesh's view
// from the per-tile mesh list into shared memory at start.
struct MeshView {
  const double* u_in;
  const double* u_n;
  double* out;
  double c;  // out = a*u_n + b*u_in + c*du  (c = stage factor * this mesh's dt)
  int cells[3];
  int nelem;
  int periodic[3];
  DeviceTables tab;
  // element info, 12 ints per element, and -1/J per node.  The line shapes
  // need them (tables 32-byte aligned: they are read as vectors); the
  // node-parallel kernels compute them where they are null
  const int* info;
  const double* mij;
};

// Copies the view of mesh m into shared memory, one 8-byte word per thread
// (the block's first sizeof(MeshView) / 8 threads); the caller synchronises.
__device__ __forceinline__ void copy_mesh_view(MeshView* dst, const MeshView* meshes, int m,
                                               int tid) {
  static_assert(sizeof(MeshView) % 8 == 0, "mesh view words");
  constexpr int MW = int(sizeof(MeshView) / 8);
  if (tid < MW)
    reinterpret_cast<unsigned long long*>(dst)[tid] =
        __ldg(reinterpret_cast<const unsigned long long*>(meshes + m) + tid);
}

template <int N>
struct StageArgs {
  MeshView mesh;           // single-mesh launches
  const MeshView* meshes;  // batched launches: mesh table
  const int* tile_mesh;    // batched launches: mesh of each block
  const int* tile_e0;      // batched launches: first element of each block
  double a, b;             // out = a*u_n + b*u_in + c*du
  double t;                // stage time when t_dev is null
  const double* t_dev;     // optional device clock: stage time = *t_dev + t
  double gamma, inv_gm1;
  double alpha_max, alpha_min, atol, hg_threshold, hg_s;
  double* alpha_out;       // optional per-element alpha
  unsigned int* nonfinite;
  const double* visc;      // Navier-Stokes contravariant viscous flux (br1_kernel.cuh)
  BcParams bc;
  BasisConst<N> basis;
  // Failure-path testing only (both 0 in normal use): bound of the tile-copy
  // waits in ns (0 = 1 s) and, when skip_tile_copy is set, the node-parallel
  // kernel arms its u_n barrier without issuing the copy, so that the wait
  // runs out with nothing in flight.
  unsigned long long wait_limit_ns;
  int skip_tile_copy;
  // Fused diagnostics: when non-null, every block writes the volume
  // integrals (volume, kinetic energy, entropy) of the nodes it stores to
  // diag[3 * slot] (slot = block, or tile of a persistent launch).
  double* diag;
};

// ---------------------------------------------------------------------------
// Fused per-step diagnostics (analyzer/volume_average_euler.hpp:29-53 with the
// weights of analyzer/volume_weighted_analyzer_functor.hpp:80,104): for one
// node of the output state, volume weight w = (w_i w_j [w_k]) / |1/J|,
// kinetic energy density |m|^2 / (2 rho), entropy density
// -rho (ln p - gamma ln rho) / (gamma - 1).
// ---------------------------------------------------------------------------
template <int DIM, int N>
__device__ __forceinline__ void diag_add_node(const double* val, const BasisConst<N>& B, int node,
                                              double inv_j, double gamma, double inv_gm1,
                                              double* acc) {
  constexpr int NV = DIM + 2;
  const int in = node % N, jn = (node / N) % N, kn = node / (N * N);
  double wq = B.w[in] * B.w[jn];
  if (DIM == 3) wq = wq * B.w[kn];
  const double w = wq / fabs(inv_j);
  double m2 = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) m2 += val[1 + d] * val[1 + d];
  const double ke = 0.5 * m2 / val[0];
  const double p = (gamma - 1.0) * (val[NV - 1] - ke);
  // 1 / (gamma - 1) from the launch arguments: within an ulp of the division
  const double s = -val[0] * (log(p) - gamma * log(val[0])) * inv_gm1;
  acc[0] += w;
  acc[1] += w * ke;
  acc[2] += w * s;
}

// Sums acc[3] over the block in a fixed order and stores the result at
// out[0..2]; every thread of the block calls it (the caller makes the
// scratch free with a barrier first).  Whole warps: a warp shuffle tree,
// then the warps in order (`red` holds 3 * NT / 32 doubles); otherwise every
// thread's values in thread order (`red` holds 3 * NT doubles).
template <int NT>
__device__ __forceinline__ void diag_block_store(double* acc, double* red, double* out) {
  if constexpr (NT % 32 == 0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], o);
    }
    __syncthreads();
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < 3; ++k) red[3 * warp + k] = acc[k];
    __syncthreads();
    if (threadIdx.x == 0) {
      double s[3] = {0.0, 0.0, 0.0};
      for (int w = 0; w < NT / 32; ++w)
#pragma unroll
        for (int k = 0; k < 3; ++k) s[k] += red[3 * w + k];
#pragma unroll
      for (int k = 0; k < 3; ++k) out[k] = s[k];
    }
  } else {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) red[3 * threadIdx.x + k] = acc[k];
    __syncthreads();
    if (threadIdx.x == 0) {
      double s[3] = {0.0, 0.0, 0.0};
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int k = 0; k < 3; ++k) s[k] += red[3 * t + k];
#pragma unroll
      for (int k = 0; k < 3; ++k) out[k] = s[k];
    }
  }
}

// Node index of position m along line `line` in direction dir.
template <int DIM, int N>
__device__ __forceinline__ int line_node(int dir, int line, int m) {
  if (DIM == 2) return dir == 0 ? m + N * line : line + N * m;
  if (dir == 0) return m + N * line;
  if (dir == 1) return (line % N) + N * m + N * N * (line / N);
  return line + N * N * m;
}

__device__ __forceinline__ double ja_at(const double* tab, int64_t eidx, int nd,
                                        int node) {
  return __ldg(tab + eidx * nd + node);
}

// ---------------------------------------------------------------------------
// Double Mach reflection state (examples/Euler2D/double_mach_reflection/
// double_mach_reflection_structured.cpp:9-32); the shock position is
// evaluated without contraction so the pre/post decision matches the
// reference's host arithmetic.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void dmr_state(const BcParams& bc, double x, double y,
                                          double t, double* u) {
  const double shock = __dadd_rn(
      1.0 / 6.0, __ddiv_rn(__dadd_rn(y, __dmul_rn(20.0, t)), bc.sqrt3));
  const double* s = (x < shock) ? bc.dmr_post : bc.dmr_pre;
#pragma unroll
  for (int q = 0; q < 4; ++q) u[q] = s[q];
}

// MixedDirichletSlipWallBC::reflect_state (dirichlet_boundary.hpp:207-220).
__device__ __forceinline__ void reflect_state(const double* ui, const double* n,
                                              double* uw) {
  const double rho = ui[0];
  const double vx = ui[1] / rho;
  const double vy = ui[2] / rho;
  const double nn2 = __fma_rn(n[1], n[1], __dmul_rn(n[0], n[0]));
  const double vn = __fma_rn(vy, n[1], __dmul_rn(vx, n[0])) / nn2;
  uw[0] = rho;
  uw[1] = __dmul_rn(rho, __fma_rn(-2.0 * vn, n[0], vx));
  uw[2] = __dmul_rn(rho, __fma_rn(-2.0 * vn, n[1], vy));
  uw[3] = ui[3];
}

// ---------------------------------------------------------------------------
// Hennemann-Gassner indicator for one element (indicator.hpp:337-418, 2D).
// Evaluated with explicitly rounded products and sums (no contraction) in
// the reference's order, so alpha and the troubled-cell flag match.
// ---------------------------------------------------------------------------
// Indicator variable rho * p with gamma fixed to 1.4 (indicator.hpp:148-161).
__device__ __forceinline__ double hg_node_value(double rho, double m1, double m2,
                                                double E) {
  const double u_vel = __ddiv_rn(m1, rho);
  const double v_vel = __ddiv_rn(m2, rho);
  const double vv = __dadd_rn(__dmul_rn(u_vel, u_vel), __dmul_rn(v_vel, v_vel));
  const double p = __dmul_rn(1.4 - 1.0, __dsub_rn(E, __dmul_rn(__dmul_rn(0.5, rho), vv)));
  return __dmul_rn(p, rho);
}

// Indicator variable rho * p of a 3D node with gamma fixed to 1.4
// (indicator.hpp:187-210).
__device__ __forceinline__ double hg_node_value_3d(double rho, double m1, double m2, double m3,
                                                   double E) {
  const double u_vel = __ddiv_rn(m1, rho);
  const double v_vel = __ddiv_rn(m2, rho);
  const double w_vel = __ddiv_rn(m3, rho);
  const double vv = __dadd_rn(__dadd_rn(__dmul_rn(u_vel, u_vel), __dmul_rn(v_vel, v_vel)),
                              __dmul_rn(w_vel, w_vel));
  const double p = __dmul_rn(1.4 - 1.0, __dsub_rn(E, __dmul_rn(__dmul_rn(0.5, rho), vv)));
  return __dmul_rn(p, rho);
}

// Modal energies -> logistic alpha with clipping (indicator.hpp:385-416).
__device__ __forceinline__ double hg_alpha_from_energies(double total, double c1, double c2,
                                                         double threshold, double s,
                                                         double alpha_min,
                                                         double alpha_max) {
  const double e1 = (total != 0.0) ? __ddiv_rn(__dsub_rn(total, c1), total) : 0.0;
  const double e2 = (c1 != 0.0) ? __ddiv_rn(__dsub_rn(c1, c2), c1) : 0.0;
  const double energy = fmax(e1, e2);
  double alpha = __ddiv_rn(
      1.0, __dadd_rn(1.0, exp(__dmul_rn(__ddiv_rn(-s, threshold),
                                        __dsub_rn(energy, threshold)))));
  if (alpha < alpha_min) alpha = 0.0;
  if (alpha > 1.0 - alpha_min) alpha = 1.0;
  return fmin(alpha_max, alpha);
}

// Sequential energy sums over m2[j*N + i] in the reference's order
// (total over all modes, clip1 over j,i < N-1, clip2 over j,i < N-2).
template <int N, class Modes>
__device__ __forceinline__ void hg_energy_sums(const Modes& m2, double* total, double* c1,
                                               double* c2) {
  double t = 0.0, a = 0.0, b = 0.0;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) t = __dadd_rn(t, m2[j * N + i]);
#pragma unroll
  for (int j = 0; j + 1 < N; ++j)
#pragma unroll
    for (int i = 0; i + 1 < N; ++i) a = __dadd_rn(a, m2[j * N + i]);
#pragma unroll
  for (int j = 0; j + 2 < N; ++j)
#pragma unroll
    for (int i = 0; i + 2 < N; ++i) b = __dadd_rn(b, m2[j * N + i]);
  *total = t;
  *c1 = a;
  *c2 = b;
}

// The 3D energy sums over m2[k*N*N + j*N + i] in the reference's order and
// coverage (indicator.hpp:494-544): clip2 over i, j, k < N-2; clip1 adds the
// index-(N-2) layers; total adds the layer k = N-1 and the rows j = N-1 of
// k < N-1.
template <int N, class Modes>
__device__ __forceinline__ void hg_energy_sums_3d(const Modes& m2, double* total, double* c1,
                                                  double* c2) {
  auto at = [&](int k, int j, int i) { return m2[(k * N + j) * N + i]; };
  double b = 0.0;
#pragma unroll
  for (int k = 0; k + 2 < N; ++k)
#pragma unroll
    for (int j = 0; j + 2 < N; ++j)
#pragma unroll
      for (int i = 0; i + 2 < N; ++i) b = __dadd_rn(b, at(k, j, i));
  double a = b;
  if (N >= 2) {
#pragma unroll
    for (int j = 0; j + 1 < N; ++j)
#pragma unroll
      for (int i = 0; i + 1 < N; ++i) a = __dadd_rn(a, at(N - 2, j, i));
#pragma unroll
    for (int k = 0; k + 2 < N; ++k)
#pragma unroll
      for (int i = 0; i + 1 < N; ++i) a = __dadd_rn(a, at(k, N - 2, i));
#pragma unroll
    for (int k = 0; k + 2 < N; ++k)
#pragma unroll
      for (int j = 0; j + 2 < N; ++j) a = __dadd_rn(a, at(k, j, N - 2));
  }
  double t = a;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) t = __dadd_rn(t, at(N - 1, j, i));
#pragma unroll
  for (int k = 0; k + 1 < N; ++k)
#pragma unroll
    for (int i = 0; i < N; ++i) t = __dadd_rn(t, at(k, N - 1, i));
  *total = t;
  *c1 = a;
  *c2 = b;
}

// Single-thread 3D indicator (standalone indicator kernel), ND = N^3 the
// stride between variables: the dimension-wise modal transform
// (indicator.hpp:69-111) in the reference's order, then the energies.
template <int N>
__device__ double hg_alpha_3d(const double* us_el, int ND, const BasisConst<N>& B,
                              double threshold, double s, double alpha_min, double alpha_max) {
  double a[N * N * N], b[N * N * N];
  for (int node = 0; node < N * N * N; ++node)
    a[node] = hg_node_value_3d(us_el[node], us_el[ND + node], us_el[2 * ND + node],
                               us_el[3 * ND + node], us_el[4 * ND + node]);
  for (int k = 0; k < N; ++k)
    for (int j = 0; j < N; ++j)
      for (int i = 0; i < N; ++i) {
        double r = 0.0;
        for (int ii = 0; ii < N; ++ii)
          r = __dadd_rn(r, __dmul_rn(B.Vinv[i][ii], a[(k * N + j) * N + ii]));
        b[(k * N + j) * N + i] = r;
      }
  for (int k = 0; k < N; ++k)
    for (int j = 0; j < N; ++j)
      for (int i = 0; i < N; ++i) {
        double r = 0.0;
        for (int jj = 0; jj < N; ++jj)
          r = __dadd_rn(r, __dmul_rn(B.Vinv[j][jj], b[(k * N + jj) * N + i]));
        a[(k * N + j) * N + i] = r;
      }
  for (int k = 0; k < N; ++k)
    for (int j = 0; j < N; ++j)
      for (int i = 0; i < N; ++i) {
        double r = 0.0;
        for (int kk = 0; kk < N; ++kk)
          r = __dadd_rn(r, __dmul_rn(B.Vinv[k][kk], a[(kk * N + j) * N + i]));
        b[(k * N + j) * N + i] = __dmul_rn(r, r);
      }
  double total, c1, c2;
  hg_energy_sums_3d<N>(b, &total, &c1, &c2);
  return hg_alpha_from_energies(total, c1, c2, threshold, s, alpha_min, alpha_max);
}

// Single-thread version (standalone indicator kernel).  ND is the stride
// between variables of the element's state.
template <int N>
__device__ double hg_alpha_2d(const double* us_el, int ND, const BasisConst<N>& B,
                              double threshold, double s, double alpha_min,
                              double alpha_max) {
  double ind[N][N];
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int node = j * N + i;
      ind[j][i] = hg_node_value(us_el[node], us_el[ND + node], us_el[2 * ND + node],
                                us_el[3 * ND + node]);
    }
  double tmp[N][N];
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      double r = 0.0;
#pragma unroll
      for (int ii = 0; ii < N; ++ii) r = __dadd_rn(r, __dmul_rn(B.Vinv[i][ii], ind[j][ii]));
      tmp[j][i] = r;
    }
  double m2[N * N];
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      double r = 0.0;
#pragma unroll
      for (int jj = 0; jj < N; ++jj) r = __dadd_rn(r, __dmul_rn(B.Vinv[j][jj], tmp[jj][i]));
      m2[j * N + i] = __dmul_rn(r, r);
    }
  double total, c1, c2;
  hg_energy_sums<N>(m2, &total, &c1, &c2);
  return hg_alpha_from_energies(total, c1, c2, threshold, s, alpha_min, alpha_max);
}

// ---------------------------------------------------------------------------
// Shared by the stage kernels
// ---------------------------------------------------------------------------
// Programmatic dependent launch: the stage kernels are launched with
// programmatic stream serialization, so a stage kernel may be scheduled while
// the previous kernel on its stream is still draining.  Each block waits for
// that kernel's completion and memory flush before it reads or writes anything
// a kernel of a step writes (launch_stage_kernel lists what may be read
// earlier), then lets the next kernel be scheduled.  Both instructions are
// no-ops in a normal launch.
__device__ __forceinline__ void stage_dependency_sync() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The u tile [el][var][node] of a block in two steps: issue() starts every
// global load of this thread for a full tile (ne == EPB) into registers,
// store() writes them to the shared tile `us` (a partial tile is loaded and
// stored in store()).  Work placed between the two overlaps the loads' latency,
// and the block waits for one global round trip instead of one per loop
// iteration.
template <int NV, int ND, int EPB, int NT>
struct ElementTileLoad {
  static constexpr int TILE = EPB * NV * ND, PER = (TILE + NT - 1) / NT;
  double v[PER];
  __device__ __forceinline__ void issue(const double* src, int ne, int tid) {
    if (ne != EPB) return;
#pragma unroll
    for (int r = 0; r < PER; ++r)
      if (TILE % NT == 0 || tid + r * NT < TILE) v[r] = __ldg(src + tid + r * NT);
  }
  __device__ __forceinline__ void store(const double* src, double* us, int ne, int tid) const {
    if (ne == EPB) {
#pragma unroll
      for (int r = 0; r < PER; ++r) {
        const int idx = tid + r * NT;
        if (TILE % NT == 0 || idx < TILE) us[idx] = v[r];
      }
    } else {
      for (int idx = tid; idx < ne * NV * ND; idx += NT) us[idx] = __ldg(src + idx);
    }
  }
};

// Element index over the axes != c of the element whose coordinate along
// `dir` is replaced by `pos` (the neighbour across a face of direction dir).
template <int DIM>
__device__ __forceinline__ int eidx_other_shift(const int* I, int c, int dir, int pos,
                                                int c0, int c1) {
  if (c == dir) return I[3 + c];
  if (DIM == 2) return pos;
  const int ax0 = (c == 0) ? 1 : 0;  // first axis != c
  const int ax1 = (c == 2) ? 1 : 2;  // second axis != c
  const int i0 = (ax0 == dir) ? pos : I[ax0];
  const int i1 = (ax1 == dir) ? pos : I[ax1];
  return i0 + (ax0 == 0 ? c0 : c1) * i1;
}

// Interface or boundary flux f* at face node `line` of the face (dir, side)
// of element `el` (surface_flux.hpp:45-271, boundary_set.hpp:70-86), with
// this element's state at the face node given as `so`.
template <int DIM, int N, int VF, int SF, bool NS>
__device__ __forceinline__ void element_face_flux_state(
    const StageArgs<N>& p, const MeshView& M, const FaceState<DIM>& so, const double* us_el,
    int e_own, const int* I, int dir, int side, int line, double gamma, double t_stage, int c0,
    int c1, int c2, double* f) {
  constexpr int NV = DIM + 2, ND = ipow(N, DIM);
  const int own_node = line_node<DIM, N>(dir, line, side ? N - 1 : 0);
  const int face = 2 * dir + side;
  const int en = I[6 + face];
  // the state on the far side of the face (neighbour trace or boundary
  // state) and the face normal; one flux evaluation follows for both cases
  double ux[NV], nrm[DIM];
  const int nb_node = line_node<DIM, N>(dir, line, side ? 0 : N - 1);
  if (en >= 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) ux[q] = __ldg(M.u_in + ((int64_t)en * NV + q) * ND + nb_node);
    // normal: Ja^dir of the element on the high side at its low-face node
    const int r_node = line_node<DIM, N>(dir, line, 0);
    const int cells[3] = {c0, c1, c2};
    int npos = I[dir] + 1;
    if (npos >= cells[dir]) npos = 0;
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const int eo = side ? eidx_other_shift<DIM>(I, c, dir, npos, c0, c1) : I[3 + c];
      nrm[c] = ja_at(M.tab.ja[dir][c], eo, ND, r_node);
    }
  } else {
    // boundary face (boundary_helper.hpp:93-146): own metric at the boundary
    // node; the inner state is the left state on high faces.
#pragma unroll
    for (int c = 0; c < DIM; ++c) nrm[c] = ja_at(M.tab.ja[dir][c], I[3 + c], ND, own_node);
    const int kind = p.bc.kind[face];
    if (DIM == 2) {
      const double x = __ldg(M.tab.coord[0] + I[0] * N + (own_node % N));
      const double y = __ldg(M.tab.coord[1] + I[1] * N + (own_node / N));
      if (kind == BC_DIRICHLET_DMR || (kind == BC_MIXED_DMR_WALL && x < 1.0 / 6.0)) {
        dmr_state(p.bc, x, y, t_stage, ux);
      } else if (kind == BC_DIRICHLET_CONST) {
#pragma unroll
        for (int q = 0; q < NV; ++q) ux[q] = p.bc.state[q];
      } else if (kind == BC_OUTFLOW) {
        // outflow_boundary.hpp:79-104: average along the line normal to the face
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          double acc = 0.0;
#pragma unroll
          for (int m = 0; m < N; ++m)
            acc += us_el[q * ND + line_node<DIM, N>(dir, line, m)];
          ux[q] = acc / (double)N;
        }
      } else {  // slip wall / wall branch of the mixed BC
        reflect_state(so.u, nrm, ux);
      }
    } else {  // 3D meshes are periodic: no boundary faces
#pragma unroll
      for (int q = 0; q < NV; ++q) ux[q] = so.u[q];
    }
  }
  const FaceState<DIM> sx = prepare_face<DIM>(ux, gamma);
  if (side) {
    surface_flux<DIM, SF>(so, sx, nrm, gamma, f);
  } else {
    surface_flux<DIM, SF>(sx, so, nrm, gamma, f);
  }
  if constexpr (NS) {
    // the one-sided viscous interface flux -F_v . n of the high-side (primary)
    // element at its low-face node (parabolic_viscous.hpp:570-585) is its
    // contravariant viscous flux there (br1_kernel.cuh); lifted with the same
    // factors as the inviscid flux
    constexpr int NQ = DIM + 1;
    const int eh = en >= 0 && side ? en : e_own;
    const int node = en >= 0 ? line_node<DIM, N>(dir, line, 0) : own_node;
    const double* V = p.visc + ((int64_t)eh * DIM + dir) * (NQ * ND) + node;
    if (en >= 0) {
#pragma unroll
      for (int r = 0; r < NQ; ++r) f[1 + r] += __ldg(V + r * ND);
    } else if (p.bc.kind[face] == BC_NS_NOSLIP_ADIABATIC_WALL) {
      // NSNoSlipAdiabaticWallBC::apply_viscous_device (navier_stokes_wall_
      // boundary.hpp:101-131): the inner -F_v . n on the momentum, no mass or
      // energy flux (adiabatic); the slip wall adds nothing
#pragma unroll
      for (int r = 0; r < DIM; ++r) f[1 + r] += __ldg(V + r * ND);
    }
  }
}

}  // namespace dgsem
