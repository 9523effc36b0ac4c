// Line-sweep form of the fused stage kernel (launch shapes 0-2): split form,
// optionally with Hennemann-Gassner shock capturing and with the viscous terms
// (br1_kernel.cuh), 2D and 3D, the same
// right-hand side and SSPRK3 epilogue as stage_node_kernel.cuh.
//
// One warp works on EPW = 32 / n^(d-1) whole elements and on nothing else:
// no block barrier orders anything, only __syncwarp.
//   load   a lane reads one x line of the state per variable (32-byte vectors
//          for n = 4, 8), prepares its n nodes and publishes them in shared
//          memory;
//   sweep  for each direction a lane owns one line of n nodes: the two-point
//          fluxes of its n (n - 1) / 2 pairs, the shock-capturing blend and
//          the surface fluxes of the line's two ends, added to a per-warp sum
//          R in shared memory;
//   store  -1/J, SSPRK3 combination and store, by x lines (n even, vectors)
//          or by lines of the last direction (n odd).
//
// Why lines: a line evaluates each two-point flux once for both of its nodes
// with no exchange (one thread per node evaluates or fetches n - 1 per node),
// each end face belongs to the line that holds its own state, and the pairs
// of a line are independent instruction streams that cover the FP64 latency.
// That halves the instructions per node; what then bounds the kernel is the
// latency of its global loads, so
//   * the loads a direction needs (neighbour traces, metric terms, normals)
//     are issued together before its volume term, u_n is brought into L2 at
//     kernel start, and the state is read once (everything later comes from
//     shared memory);
//   * the volume term is one straight block without branches: reciprocals and
//     roots are branch-free (physics.cuh: recip_ulp, root) and the logarithmic
//     means take their series for every pair; a line with a pair outside the
//     series' range repeats its volume term (LineMean).
//
// Shared memory of a warp, planes of doubles [slot][element][node]: the NV
// conserved variables, 1 / (2 rho), p, Chandrashekar: rho / p; then the NV
// planes of R.  Node positions are swizzled for n = 4 (LinePos), otherwise
// x lines have an odd stride, so that the lines of every direction fall on
// distinct banks.
//
// Measured against the former line-per-direction kernel (one thread per line,
// one direction per thread, block barriers, 7.5 M warp instructions per TGV
// 16^3 stage, here 4.4 M) and against one thread per node, B200, us per stage
// (the sweep when it was first measured; with the rounded reciprocals 0.5-2 %
// more):
//   KH 1024^2 Ranocha        1181 -> 432   (thread per node 708)
//   TGV 16^3 Kennedy-Gruber  23.3 -> 13.4  (17.9)
//   TGV 32^3 Chandrashekar    365 -> 97    (181)
//   3D shock capturing n = 5, 1287 elements  29.3 -> 19.0
// ncu on TGV 32^3 Chandrashekar: FP64 pipe 50-52 % of the time, 6.7-8.9 TB/s out
// of L2, 0.42-0.43 instructions per cycle and scheduler; the longest stall is the
// global load (1.6-2.0 of 6.5-6.8 cycles between a warp's instructions).
//
// Scaling by powers of two is exact, so averages are formed from halved
// velocities and the pair normal Ja_i + Ja_k, and the factors are collected
// in the constants Dvol = Dsplit * (1/4 or 1/2).
#pragma once

#include <type_traits>

#include "stage_kernel.cuh"
#include "tma.cuh"

namespace dgsem {

template <int DIM, int N>
struct LineGeo {
  static constexpr int NV = DIM + 2;
  static constexpr int ND = ipow(N, DIM);
  static constexpr int NF = ipow(N, DIM - 1);  // lines per direction
  static constexpr int EPW = 32 / NF;          // elements per warp
  static constexpr bool SWZ = N == 4;
  static constexpr int LS = SWZ ? 4 : (N % 2 ? N : N + 1);  // stride of x lines
  static constexpr int PL = LS * NF;                        // one element's plane
  static constexpr int PLANE = EPW * PL;                    // one warp's plane
  static_assert(EPW >= 1, "an element's lines fit one warp");
};

// Planes published per node (after the NV conserved variables).
template <int DIM, int VF>
struct LineSlots {
  static constexpr int HINV = DIM + 2;  // 1 / (2 rho)
  static constexpr int P = DIM + 3;
  static constexpr int B = DIM + 4;     // Chandrashekar: rho / p
  static constexpr int NS = VF == VF_CHANDRASHEKAR ? DIM + 5 : DIM + 4;
};

template <int DIM, int N, int VF>
struct LineShape {
  using G = LineGeo<DIM, N>;
  static constexpr int WARP_DOUBLES = (LineSlots<DIM, VF>::NS + G::NV) * G::PLANE;
  static constexpr size_t smem_bytes(int warps) {
    return sizeof(double) * (size_t)WARP_DOUBLES * warps;
  }
};

// A lane's line along one direction: positions of its nodes in a shared
// plane, and their node indices first + m * stride.
// n = 4: the node (i, j, k) (2D: k = the element in the warp) sits at
// 16 k + 4 (j ^ k) + (i ^ 2 (k & 1)): 16 lanes reading one node of their y or
// z lines (64 bits each) and 8 lanes reading half of their x lines (128 bits
// each) fall on distinct banks.
template <int DIM, int N>
struct LinePos {
  int off[N];
  int first, stride;

  static __device__ __forceinline__ int slot(int dir, int el, int line, int m) {
    using G = LineGeo<DIM, N>;
    const int lo = line % N, hi = DIM == 3 ? line / N : 0;
    const int i = dir == 0 ? m : lo;
    const int j = dir == 0 ? lo : dir == 1 ? m : hi;
    const int k = dir == 2 ? m : hi;
    if constexpr (G::SWZ) {
      const int kk = DIM == 2 ? (el & 3) : k;
      const int base = DIM == 2 ? 16 * el : 64 * el + 16 * k;
      return base + 4 * (j ^ kk) + (i ^ (2 * (kk & 1)));
    } else {
      return el * G::PL + (j + N * k) * G::LS + i;
    }
  }

  __device__ __forceinline__ void set(int dir, int el, int line) {
    const int lo = line % N, hi = DIM == 3 ? line / N : 0;
    stride = dir == 0 ? 1 : dir == 1 ? N : N * N;
    first = dir == 0 ? N * line : dir == 1 ? lo + N * N * hi : line;
#pragma unroll
    for (int m = 0; m < N; ++m) off[m] = slot(dir, el, line, m);
  }
};

// The n values of an x line (contiguous in memory) from global memory.  VEC:
// 32-byte vectors (n a multiple of 4) or 16-byte vectors (n even); the caller
// has checked the alignment (line_vec_mask).
template <int N, bool VEC>
__device__ __forceinline__ void load_xline(const double* src, double* v) {
  if constexpr (VEC && N % 4 == 0) {
#pragma unroll
    for (int m = 0; m < N; m += 4)
      asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                   : "=d"(v[m]), "=d"(v[m + 1]), "=d"(v[m + 2]), "=d"(v[m + 3])
                   : "l"(src + m)
                   : "memory");
  } else if constexpr (VEC && N % 2 == 0) {
#pragma unroll
    for (int m = 0; m < N; m += 2) {
      const double2 d = *reinterpret_cast<const double2*>(src + m);
      v[m] = d.x;
      v[m + 1] = d.y;
    }
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) v[m] = src[m];
  }
}

template <int N, bool VEC>
__device__ __forceinline__ void store_xline(double* dst, const double* v) {
  if constexpr (VEC && N % 4 == 0) {
#pragma unroll
    for (int m = 0; m < N; m += 4)
      asm volatile("st.global.v4.f64 [%4], {%0,%1,%2,%3};" ::"d"(v[m]), "d"(v[m + 1]),
                   "d"(v[m + 2]), "d"(v[m + 3]), "l"(dst + m)
                   : "memory");
  } else if constexpr (VEC && N % 2 == 0) {
#pragma unroll
    for (int m = 0; m < N; m += 2)
      *reinterpret_cast<double2*>(dst + m) = make_double2(v[m], v[m + 1]);
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) dst[m] = v[m];
  }
}

// Address bits that must be zero for the vector accesses to x lines.
template <int N>
__host__ __device__ constexpr unsigned line_vec_mask() {
  return N % 4 == 0 ? 31u : N % 2 == 0 ? 15u : 0u;
}

// One line's values of one plane.  XL: an x line; at n = 4 its halves are two
// aligned 16-byte pieces.
template <bool XL, int N>
__device__ __forceinline__ void load_line(const double* plane, const int* off, double* v) {
  if constexpr (XL && N == 4) {
    const double2 a = *reinterpret_cast<const double2*>(plane + off[0]);
    const double2 b = *reinterpret_cast<const double2*>(plane + off[2]);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) v[m] = plane[off[m]];
  }
}

template <bool XL, int N>
__device__ __forceinline__ void store_line(double* plane, const int* off, const double* v) {
  if constexpr (XL && N == 4) {
    *reinterpret_cast<double2*>(plane + off[0]) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(plane + off[2]) = make_double2(v[2], v[3]);
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m) plane[off[m]] = v[m];
  }
}

// Node data of the two-point fluxes.
template <int DIM>
struct LineNode {
  double rho;
  double hv[DIM];  // v / 2
  double p;
  double x;  // Kennedy-Gruber: e / 2; Chandrashekar: rho / p
  double y;  // Chandrashekar: |v|^2 / 4
};

// a . b with one rounding order: sums of products are written as explicit
// multiply-adds, so that every instantiation of the kernel gives the same bits.
template <int DIM>
__device__ __forceinline__ double line_dot(const double* a, const double* b) {
  double r = __dmul_rn(a[0], b[0]);
#pragma unroll
  for (int d = 1; d < DIM; ++d) r = __fma_rn(a[d], b[d], r);
  return r;
}

// The result of line_pair_flux carries a power of two that Dvol takes out:
// Kennedy-Gruber 4 f, Chandrashekar and Ranocha 2 f.
template <int VF>
struct LineScale {
  static constexpr double value = VF == VF_KENNEDY_GRUBER ? 0.25 : 0.5;
};

// How a line evaluates the logarithmic means of its pairs, from f^2 =
// ((a - b) / (a + b))^2 of both means:
//   MEAN_SHORT    f^2 < 1e-4: the reference's series (4 terms)
//   MEAN_LONG     f^2 < 1/16 (a ratio of up to 5/3 between two nodes): the
//                 same series atanh(f) / f = sum f^2k / (2k + 1) to 13 terms
//                 (remainder below 1e-17).  The reference takes the logarithm
//                 here, whose argument b / a near 1 costs it up to 50 units in
//                 the last place; the two agree to that
//   MEAN_GENERAL  any pair: the reference's rule with the logarithm
// A line takes the same form for all of its pairs, so each form is one block
// of straight code.  The sums' reciprocals are recip_ulp's (at most 0.501 units
// in the last place; the node kernels' shared ones, two_reciprocals, 1.5): with
// rounded ones KH 1024^2 took 503 us per stage instead of 494, a stage of 64
// batched meshes 694 instead of 674.
enum LineMean : int { MEAN_SHORT, MEAN_LONG, MEAN_GENERAL };

__device__ __forceinline__ double line_atanh_series(double t) {
  double r = 1.0 / 25.0;
#pragma unroll
  for (int k = 11; k >= 0; --k) r = __fma_rn(r, t, 1.0 / (2 * k + 1));
  return r;
}

// Two-point volume flux of two nodes of a line, ns = Ja_i + Ja_k.  *range
// keeps the largest high word of the f^2 seen (MEAN_SHORT; the caller compares
// it with the range of the form).
template <int DIM, int VF, int MEAN>
__device__ __forceinline__ void line_pair_flux(const LineNode<DIM>& L, const LineNode<DIM>& R,
                                               const double* ns, double inv_gm1, int* range,
                                               double* f) {
  const double rs = L.rho + R.rho;
  double va[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) va[d] = L.hv[d] + R.hv[d];
  if constexpr (VF == VF_KENNEDY_GRUBER) {
    const double ps = L.p + R.p;
    const double ea = L.x + R.x;
    const double vn = line_dot<DIM>(va, ns);
    const double f1 = __dmul_rn(rs, vn);
    f[0] = f1;
#pragma unroll
    for (int d = 0; d < DIM; ++d) f[1 + d] = __fma_rn(f1, va[d], __dmul_rn(ps, ns[d]));
    f[DIM + 1] = __dmul_rn(__fma_rn(rs, ea, ps), vn);
    return;
  }
  // a, b: the arguments of the inverse logarithmic mean
  double a, b;
  if constexpr (VF == VF_CHANDRASHEKAR) {
    a = L.x;
    b = R.x;
  } else {
    a = __dmul_rn(L.rho, R.p);
    b = __dmul_rn(R.rho, L.p);
  }
  const double s = a + b;
  const double is = recip_ulp(s);
  double rho_mean, im;
  if constexpr (MEAN == MEAN_GENERAL) {
    rho_mean = ln_mean_rs(L.rho, R.rho, rs, recip_ulp(rs));
    im = inv_ln_mean_rs(a, b, is);
  } else if constexpr (MEAN == MEAN_LONG) {
    const double t = (L.rho - R.rho) * recip_ulp(rs), g2 = __dmul_rn(t, t);
    const double w = (a - b) * is, f2 = __dmul_rn(w, w);
    rho_mean = __dmul_rn(0.5 * rs, recip_ulp(line_atanh_series(g2)));
    im = __dmul_rn(2.0 * is, line_atanh_series(f2));
  } else {
    const double t = (L.rho - R.rho) * recip_ulp(rs), g2 = __dmul_rn(t, t);
    const double w = (a - b) * is, f2 = __dmul_rn(w, w);
    // both are >= 0 or NaN: compared on the high words, no FP64 compare
    *range = max(*range, max(__double2hiint(g2), __double2hiint(f2)));
    rho_mean = __dmul_rn(
        rs, __fma_rn(g2, __fma_rn(g2, __fma_rn(g2, -22.0 / 945.0, -2.0 / 45.0), -1.0 / 6.0), 0.5));
    im = __dmul_rn(
        is, __fma_rn(f2, __fma_rn(f2, __fma_rn(f2, 2.0 / 7.0, 2.0 / 5.0), 2.0 / 3.0), 2.0));
  }
  if constexpr (VF == VF_CHANDRASHEKAR) {
    // numerical_flux.hpp:436-500 with b = rho / p = 2 beta
    const double pm = __dmul_rn(rs, is);
    const double f1 = __dmul_rn(rho_mean, line_dot<DIM>(va, ns));
    f[0] = f1;
    double fe = __dmul_rn(f1, __fma_rn(inv_gm1, im, -(L.y + R.y)));
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double fm = __fma_rn(f1, va[d], __dmul_rn(pm, ns[d]));
      f[1 + d] = fm;
      fe = __fma_rn(fm, va[d], fe);
    }
    f[DIM + 1] = fe;
  } else {  // Ranocha
    const double vi = line_dot<DIM>(L.hv, ns), vk = line_dot<DIM>(R.hv, ns);
    const double irp = __dmul_rn(__dmul_rn(L.p, R.p), im);
    const double pa = 0.5 * (L.p + R.p);
    const double f1 = __dmul_rn(rho_mean, vi + vk);
    f[0] = f1;
#pragma unroll
    for (int d = 0; d < DIM; ++d) f[1 + d] = __fma_rn(f1, va[d], __dmul_rn(pa, ns[d]));
    f[DIM + 1] = __fma_rn(
        f1, __fma_rn(2.0, line_dot<DIM>(L.hv, R.hv), __dmul_rn(irp, inv_gm1)),
        __fma_rn(L.p, vk, __dmul_rn(R.p, vi)));
  }
}

// State of one side of a face: conserved variables, v / 2, p, a^2 / 4.
template <int DIM>
struct LineFace {
  double u[DIM + 2];
  double hv[DIM];
  double p;
  double qa2;
};

template <int DIM>
__device__ __forceinline__ void line_face_prepare(LineFace<DIM>& s, double gamma) {
  const double hinv = 0.5 * recip(s.u[0]);
#pragma unroll
  for (int d = 0; d < DIM; ++d) s.hv[d] = __dmul_rn(s.u[1 + d], hinv);
  const double ke = line_dot<DIM>(s.u + 1, s.hv);
  s.p = __dmul_rn(gamma - 1.0, s.u[DIM + 1] - ke);
  s.qa2 = __dmul_rn(__dmul_rn(0.5 * gamma, s.p), hinv);
}

// Local Lax-Friedrichs flux (llf_flux on halved data): with h = v.n / 2 and
// lambda / 2 = max |h| + sqrt(max(a^2 / 4) |n|^2),
//   f = h_L u_L + h_R u_R + pressure terms - lambda / 2 (u_R - u_L).
template <int DIM>
__device__ __forceinline__ void line_llf(const LineFace<DIM>& L, const LineFace<DIM>& R,
                                         const double* n, double* f) {
  const double hL = line_dot<DIM>(L.hv, n), hR = line_dot<DIM>(R.hv, n);
  const double nn = line_dot<DIM>(n, n);
  const double hlam = fmax(fabs(hL), fabs(hR)) + root(fmax(L.qa2, R.qa2) * nn);
  const double pa = 0.5 * (L.p + R.p);
  f[0] = __fma_rn(-hlam, R.u[0] - L.u[0], __fma_rn(hR, R.u[0], __dmul_rn(hL, L.u[0])));
#pragma unroll
  for (int d = 0; d < DIM; ++d)
    f[1 + d] = __fma_rn(
        -hlam, R.u[1 + d] - L.u[1 + d],
        __fma_rn(pa, n[d], __fma_rn(hR, R.u[1 + d], __dmul_rn(hL, L.u[1 + d]))));
  f[DIM + 1] = __fma_rn(
      -hlam, R.u[DIM + 1] - L.u[DIM + 1],
      __fma_rn(hR, R.u[DIM + 1] + R.p, __dmul_rn(hL, L.u[DIM + 1] + L.p)));
}

template <int DIM, int SF>
__device__ __forceinline__ void line_surface_flux(const LineFace<DIM>& L, const LineFace<DIM>& R,
                                                  const double* n, double gamma, double* f) {
  if constexpr (SF == SF_HLLC && DIM == 2) {
    FaceState<2> l, r;  // the HLLC flux works on the conserved variables
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      l.u[q] = L.u[q];
      r.u[q] = R.u[q];
    }
    hllc_flux_2d(l, r, n, gamma, f);
  } else {
    line_llf<DIM>(L, R, n, f);
  }
}

// Everything a lane needs to know about its element.
template <int DIM>
struct LineElement {
  int e;            // element index in its mesh
  int row[DIM];     // rows of the metric tables per axis (element info 3-5)
  const int* info;  // element info of the element
};

// State beyond a boundary face of a 2D mesh (boundary_helper.hpp:93-146; see
// element_face_flux_state); `U` the element's planes of conserved variables.
template <int N>
__device__ __forceinline__ void line_boundary_state(const StageArgs<N>& p, const MeshView& M,
                                                    const LineElement<2>& E,
                                                    const LinePos<2, N>& pos, const double* U,
                                                    int face, double t_stage, const double* ui,
                                                    const double* nrm, double* ux) {
  constexpr int PLANE = LineGeo<2, N>::PLANE;
  const int node = pos.first + ((face & 1) ? N - 1 : 0) * pos.stride;
  const int kind = p.bc.kind[face];
  // row[c] = index over the axes other than c
  const double x = __ldg(M.tab.coord[0] + E.row[1] * N + node % N);
  const double y = __ldg(M.tab.coord[1] + E.row[0] * N + node / N);
  if (kind == BC_DIRICHLET_DMR || (kind == BC_MIXED_DMR_WALL && x < 1.0 / 6.0)) {
    dmr_state(p.bc, x, y, t_stage, ux);
  } else if (kind == BC_DIRICHLET_CONST) {
#pragma unroll
    for (int q = 0; q < 4; ++q) ux[q] = p.bc.state[q];
  } else if (kind == BC_OUTFLOW) {
    // outflow_boundary.hpp:79-104: average along the line normal to the face
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double s = 0.0;
#pragma unroll
      for (int m = 0; m < N; ++m) s += U[q * PLANE + pos.off[m]];
      ux[q] = s / (double)N;
    }
  } else {  // slip wall / wall branch of the mixed BC
    reflect_state(ui, nrm, ux);
  }
}

// Node data at position `o` of the planes P.
template <int DIM, int VF, int PLANE>
__device__ __forceinline__ LineNode<DIM> line_node_data(const double* P, int o) {
  using K = LineSlots<DIM, VF>;
  LineNode<DIM> q;
  const double hinv = P[K::HINV * PLANE + o];
  q.rho = P[o];
#pragma unroll
  for (int d = 0; d < DIM; ++d) q.hv[d] = __dmul_rn(P[(1 + d) * PLANE + o], hinv);
  q.p = P[K::P * PLANE + o];
  q.x = VF == VF_KENNEDY_GRUBER   ? __dmul_rn(P[(DIM + 1) * PLANE + o], hinv)
        : VF == VF_CHANDRASHEKAR ? P[K::B * PLANE + o]
                                 : 0.0;
  q.y = VF == VF_CHANDRASHEKAR ? line_dot<DIM>(q.hv, q.hv) : 0.0;
  return q;
}

// Metric terms of a line.
template <int DIM, int N, bool XL>
__device__ __forceinline__ void line_metrics(const MeshView& M, const LineElement<DIM>& E, int dir,
                                             const LinePos<DIM, N>& pos, double (*ja)[DIM]) {
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    const double* J = M.tab.ja[dir][c] + (int64_t)E.row[c] * LineGeo<DIM, N>::ND + pos.first;
    if constexpr (XL) {
      double v[N];
      load_xline<N, true>(J, v);
#pragma unroll
      for (int m = 0; m < N; ++m) ja[m][c] = v[m];
    } else {
#pragma unroll
      for (int m = 0; m < N; ++m) ja[m][c] = __ldg(J + m * pos.stride);
    }
  }
}

// The neighbours across a line's ends and the normal of its high face: Ja^dir
// of the element on the high side at its low face (at a boundary the line's
// own last node).  The component along dir does not depend on the position
// along dir.
template <int DIM, int N>
__device__ __forceinline__ void line_ends(const MeshView& M, const LineElement<DIM>& E, int dir,
                                          const LinePos<DIM, N>& pos, int* nb, double* nh) {
  constexpr int ND = LineGeo<DIM, N>::ND;
  nb[0] = __ldg(E.info + 6 + 2 * dir);
  nb[1] = __ldg(E.info + 7 + 2 * dir);
  const int cd = M.cells[dir];
  const int step = nb[1] > E.e ? 1 : 1 - cd;  // the neighbour's position along dir
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    // stride of dir in the rows of axis c
    const int st = DIM == 2 ? 1
                   : c == 0 ? (dir == 1 ? 1 : M.cells[1])
                            : (dir == 0 ? 1 : M.cells[0]);
    const int shift = c == dir || nb[1] < 0 ? 0 : step * st;
    nh[c] = __ldg(M.tab.ja[dir][c] + (int64_t)(E.row[c] + shift) * ND + pos.first +
                  (nb[1] < 0 ? (N - 1) * pos.stride : 0));
  }
}

// The neighbours' conserved states at a line's ends.
template <int DIM, int N>
__device__ __forceinline__ void line_traces(const MeshView& M, const LinePos<DIM, N>& pos,
                                            const int* nb, double (*tr)[DIM + 2]) {
  constexpr int NV = DIM + 2, ND = LineGeo<DIM, N>::ND;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const double* T = M.u_in + (int64_t)max(nb[s], 0) * (NV * ND) + pos.first +
                      (s ? 0 : (N - 1) * pos.stride);
#pragma unroll
    for (int v = 0; v < NV; ++v) tr[s][v] = __ldg(T + v * ND);
  }
}

// Every pair of the line once, with one form of the means.
template <int DIM, int N, int VF, int MEAN>
__device__ __forceinline__ int line_pairs(const StageArgs<N>& p, const LineNode<DIM>* q,
                                          const double (*ja)[DIM], double (*acc)[DIM + 2]) {
  constexpr int NV = DIM + 2;
#pragma unroll
  for (int m = 0; m < N; ++m)
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[m][v] = 0.0;
  int range = 0;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (k <= i) continue;
      double ns[DIM], f[NV];
#pragma unroll
      for (int c = 0; c < DIM; ++c) ns[c] = ja[i][c] + ja[k][c];
      line_pair_flux<DIM, VF, MEAN>(q[i], q[k], ns, p.inv_gm1, &range, f);
      const double dik = p.basis.Dvol[i][k], dki = p.basis.Dvol[k][i];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        acc[i][v] = __fma_rn(dik, f[v], acc[i][v]);
        acc[k][v] = __fma_rn(dki, f[v], acc[k][v]);
      }
    }
  return range;
}

// Node data of a line.
template <int DIM, int N, int VF, bool XL>
__device__ __forceinline__ void line_nodes(const double* P, const LinePos<DIM, N>& pos,
                                           LineNode<DIM>* q) {
  using K = LineSlots<DIM, VF>;
  constexpr int NV = DIM + 2, PLANE = LineGeo<DIM, N>::PLANE;
  double hinv[N], t[N];
  load_line<XL, N>(P + K::HINV * PLANE, pos.off, hinv);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    if (v == NV - 1 && VF != VF_KENNEDY_GRUBER) continue;
    load_line<XL, N>(P + v * PLANE, pos.off, t);
    if (v == 0) {
#pragma unroll
      for (int m = 0; m < N; ++m) q[m].rho = t[m];
    } else if (v <= DIM) {
#pragma unroll
      for (int m = 0; m < N; ++m) q[m].hv[v - 1] = __dmul_rn(t[m], hinv[m]);
    } else if (VF == VF_KENNEDY_GRUBER) {
#pragma unroll
      for (int m = 0; m < N; ++m) q[m].x = __dmul_rn(t[m], hinv[m]);
    }
  }
  load_line<XL, N>(P + K::P * PLANE, pos.off, t);
#pragma unroll
  for (int m = 0; m < N; ++m) q[m].p = t[m];
  if constexpr (VF == VF_CHANDRASHEKAR) {
    load_line<XL, N>(P + K::B * PLANE, pos.off, t);
#pragma unroll
    for (int m = 0; m < N; ++m) {
      q[m].x = t[m];
      q[m].y = line_dot<DIM>(q[m].hv, q[m].hv);
    }
  }
}

// Adds `scale` times the volume term of a line outside the short series' range
// to its line of R: with the long series, or (not `series`) the general means,
// the latter rolled up for n > 4.  A function of its own, called by few lines
// and last, when little is live: inlined, its code cost the kernels' main path
// registers (TGV 32^3 Chandrashekar 96 -> 111 us per stage, KH 1024^2 445 ->
// 471).
template <int DIM, int N, int VF>
__device__ __noinline__ void line_volume_steep(const StageArgs<N>* p, const MeshView* M,
                                               LineElement<DIM> E, int dir, int el, int line,
                                               const double* P, double* R, bool series,
                                               double scale) {
  using G = LineGeo<DIM, N>;
  constexpr int NV = G::NV, PLANE = G::PLANE;
  LinePos<DIM, N> pos;
  pos.set(dir, el, line);
  LineNode<DIM> q[N];
  double ja[N][DIM], acc[N][NV];
  if (series || N <= 4) {
    line_nodes<DIM, N, VF, false>(P, pos, q);
    line_metrics<DIM, N, false>(*M, E, dir, pos, ja);
    if (series)
      line_pairs<DIM, N, VF, MEAN_LONG>(*p, q, ja, acc);
    else if constexpr (N <= 4)
      line_pairs<DIM, N, VF, MEAN_GENERAL>(*p, q, ja, acc);
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int m = 0; m < N; ++m) {
        double* r = R + v * PLANE + pos.off[m];
        *r = __fma_rn(scale, acc[m][v], *r);
      }
    return;
  }
#pragma unroll 1
  for (int i = 0; i + 1 < N; ++i) {
    const int oi = LinePos<DIM, N>::slot(dir, el, line, i);
    const LineNode<DIM> L = line_node_data<DIM, VF, PLANE>(P, oi);
#pragma unroll 1
    for (int k = i + 1; k < N; ++k) {
      const int ok = LinePos<DIM, N>::slot(dir, el, line, k);
      const LineNode<DIM> Q = line_node_data<DIM, VF, PLANE>(P, ok);
      double ns[DIM], f[NV];
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        const double* J = M->tab.ja[dir][c] + (int64_t)E.row[c] * G::ND + pos.first;
        ns[c] = __ldg(J + i * pos.stride) + __ldg(J + k * pos.stride);
      }
      line_pair_flux<DIM, VF, MEAN_GENERAL>(L, Q, ns, p->inv_gm1, nullptr, f);
      const double dik = __dmul_rn(scale, p->basis.Dvol[i][k]);
      const double dki = __dmul_rn(scale, p->basis.Dvol[k][i]);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        R[v * PLANE + oi] = __fma_rn(dik, f[v], R[v * PLANE + oi]);
        R[v * PLANE + ok] = __fma_rn(dki, f[v], R[v * PLANE + ok]);
      }
    }
  }
}

// Volume term of a line.  Returns 0, or for a line outside the short series'
// range 1 (long series) or 2 (general means); acc is then zero and the caller
// adds the term with line_volume_steep after everything else.
template <int DIM, int N, int VF, bool XL>
__device__ __forceinline__ int line_volume(const StageArgs<N>& p, const LinePos<DIM, N>& pos,
                                           const double* P, const double (*ja)[DIM],
                                           LineNode<DIM>* q, double (*acc)[DIM + 2]) {
  line_nodes<DIM, N, VF, XL>(P, pos, q);
  const int range = line_pairs<DIM, N, VF, MEAN_SHORT>(p, q, ja, acc);
  constexpr int kShortRange = 0x3f1a36e2, kLongRange = 0x3fb00000;  // high words: 1e-4, 1/16
  if (VF == VF_KENNEDY_GRUBER || range < kShortRange) return 0;
#pragma unroll
  for (int m = 0; m < N; ++m)
#pragma unroll
    for (int v = 0; v < DIM + 2; ++v) acc[m][v] = 0.0;
  return range < kLongRange ? 1 : 2;
}

// Shock-capturing blend of a troubled line (volume_flux.hpp:817-842): (1 -
// alpha) DG + alpha FV, the FV subcell fluxes (:457-509 in 2D, :521-630 in 3D)
// once per interface.
template <int DIM, int N, int VF>
__device__ __forceinline__ void line_blend(const StageArgs<N>& p, const MeshView& M,
                                           const LineElement<DIM>& E, int dir, int line,
                                           const LinePos<DIM, N>& pos, const double* P,
                                           double alpha, double (*acc)[DIM + 2]) {
  using G = LineGeo<DIM, N>;
  using K = LineSlots<DIM, VF>;
  constexpr int NV = G::NV, NF = G::NF, PLANE = G::PLANE;
  const double one_m = 1.0 - alpha;
#pragma unroll
  for (int m = 0; m < N; ++m)
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[m][v] = __dmul_rn(acc[m][v], one_m);
  auto node = [&](int m) {
    LineFace<DIM> s;
#pragma unroll
    for (int v = 0; v < NV; ++v) s.u[v] = P[v * PLANE + pos.off[m]];
    const double hinv = P[K::HINV * PLANE + pos.off[m]];
#pragma unroll
    for (int d = 0; d < DIM; ++d) s.hv[d] = __dmul_rn(s.u[1 + d], hinv);
    s.p = P[K::P * PLANE + pos.off[m]];
    s.qa2 = __dmul_rn(__dmul_rn(0.5 * p.gamma, s.p), hinv);
    return s;
  };
  LineFace<DIM> L = node(0);
#pragma unroll
  for (int m = 1; m < N; ++m) {
    const LineFace<DIM> S = node(m);
    double nrm[DIM], f[NV];
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      nrm[c] = __ldg(M.tab.fv[dir][c] + (int64_t)E.row[c] * (N - 1) * NF + (m - 1) * NF + line);
    line_llf<DIM>(L, S, nrm, f);
    const double wl = alpha * p.basis.inv_w[m - 1], wr = -alpha * p.basis.inv_w[m];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      acc[m - 1][v] = __fma_rn(wl, f[v], acc[m - 1][v]);
      acc[m][v] = __fma_rn(wr, f[v], acc[m][v]);
    }
    L = S;
  }
}

// Surface fluxes at both ends of a line (surface_flux.hpp:45-271): `take(s, f)`
// receives the flux of the low (s = 0) and the high face.  jlo, nh: normals of
// the low and high face; tr: far states, at boundary faces of 2D meshes
// replaced by the boundary states.
template <int DIM, int N, int VF, int SF, class Take>
__device__ __forceinline__ void line_faces(const StageArgs<N>& p, const MeshView& M,
                                           const LineElement<DIM>& E, int dir,
                                           const LinePos<DIM, N>& pos, const double* P,
                                           const int* nb, double (*tr)[DIM + 2],
                                           const double* jlo, const double* nh, double t_stage,
                                           Take&& take) {
  using K = LineSlots<DIM, VF>;
  constexpr int NV = DIM + 2, PLANE = LineGeo<DIM, N>::PLANE;
  const double gamma = p.gamma;
  if constexpr (DIM == 2) {
    if ((nb[0] | nb[1]) < 0) {
#pragma unroll 1
      for (int s = 0; s < 2; ++s) {
        if ((s ? nb[1] : nb[0]) >= 0) continue;
        double ui[NV], ux[NV], nrm[DIM];
#pragma unroll
        for (int v = 0; v < NV; ++v) ui[v] = P[v * PLANE + (s ? pos.off[N - 1] : pos.off[0])];
#pragma unroll
        for (int c = 0; c < DIM; ++c) nrm[c] = s ? nh[c] : jlo[c];
        line_boundary_state<N>(p, M, E, pos, P, 2 * dir + s, t_stage, ui, nrm, ux);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          tr[0][v] = s ? tr[0][v] : ux[v];
          tr[1][v] = s ? ux[v] : tr[1][v];
        }
      }
    }
  }
  auto face = [&](int s) {
    LineFace<DIM> own, far;
    double nrm[DIM], f[NV];
    const int o = s ? pos.off[N - 1] : pos.off[0];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      own.u[v] = P[v * PLANE + o];
      far.u[v] = s ? tr[1][v] : tr[0][v];
    }
#pragma unroll
    for (int c = 0; c < DIM; ++c) nrm[c] = s ? nh[c] : jlo[c];
    if constexpr (!(SF == SF_HLLC && DIM == 2)) {
      const double hinv = P[K::HINV * PLANE + o];
#pragma unroll
      for (int d = 0; d < DIM; ++d) own.hv[d] = __dmul_rn(own.u[1 + d], hinv);
      own.p = P[K::P * PLANE + o];
      own.qa2 = __dmul_rn(__dmul_rn(0.5 * gamma, own.p), hinv);
      line_face_prepare<DIM>(far, gamma);
    }
    // own state left of the face at the high end, right of it at the low end
    if (s)
      line_surface_flux<DIM, SF>(own, far, nrm, gamma, f);
    else
      line_surface_flux<DIM, SF>(far, own, nrm, gamma, f);
    take(s, f);
  };
  if constexpr (SF == SF_HLLC && DIM == 2) {
    // the longer flux once, for both ends in turn
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
      LineFace<DIM> l, r;
      double nrm[DIM], f[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double own = P[v * PLANE + (s ? pos.off[N - 1] : pos.off[0])];
        l.u[v] = s ? own : tr[0][v];
        r.u[v] = s ? tr[1][v] : own;
      }
#pragma unroll
      for (int c = 0; c < DIM; ++c) nrm[c] = s ? nh[c] : jlo[c];
      line_surface_flux<DIM, SF>(l, r, nrm, gamma, f);
      take(s, f);
    }
  } else {
    face(0);
    face(1);
  }
}

// Lifts a face flux into the line's end node (surface_integral.hpp:35-154).
template <int N, int NV>
__device__ __forceinline__ void line_lift(const StageArgs<N>& p, int s, const double* f,
                                          double (*acc)[NV]) {
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    acc[0][v] = s ? acc[0][v] : __fma_rn(-f[v], p.basis.lhat_l0, acc[0][v]);
    acc[N - 1][v] = s ? __fma_rn(f[v], p.basis.lhat_rN, acc[N - 1][v]) : acc[N - 1][v];
  }
}

// Viscous terms of a line, outside the shock-capturing blend (the reference
// adds the parabolic terms separately, structured_solver.hpp:437-480): Dhat
// product of the contravariant flux along the line (parabolic_viscous.hpp:
// 398-466) and the one-sided interface fluxes of the high-side elements, the
// line's own at its low end (br1_kernel.cuh).
template <int DIM, int N, bool XL>
__device__ __forceinline__ void line_viscous(const StageArgs<N>& p, const LineElement<DIM>& E,
                                             int dir, const LinePos<DIM, N>& pos, const int* nb,
                                             double (*acc)[DIM + 2]) {
  constexpr int NQ = DIM + 1, ND = LineGeo<DIM, N>::ND;
  const double* V = p.visc + ((int64_t)E.e * DIM + dir) * (NQ * ND) + pos.first;
  const double* Vn = p.visc + ((int64_t)max(nb[1], 0) * DIM + dir) * (NQ * ND) + pos.first;
  bool lo = true, hi = true;
  if (DIM == 2 && (nb[0] | nb[1]) < 0) {
    // no-slip walls: the inner flux on the momentum rows; slip walls: none
    lo = nb[0] >= 0 || p.bc.kind[2 * dir] == BC_NS_NOSLIP_ADIABATIC_WALL;
    hi = nb[1] >= 0 || p.bc.kind[2 * dir + 1] == BC_NS_NOSLIP_ADIABATIC_WALL;
  }
#pragma unroll
  for (int r = 0; r < NQ; ++r) {
    double w[N];
    if constexpr (XL) {
      load_xline<N, true>(V + r * ND, w);
    } else {
#pragma unroll
      for (int m = 0; m < N; ++m) w[m] = __ldg(V + r * ND + m * pos.stride);
    }
    double wl = w[0], wh = __ldg(Vn + r * ND);
    if constexpr (DIM == 2) {
      wh = nb[1] >= 0 ? wh : w[N - 1];
      wl = !lo || (nb[0] < 0 && r == DIM) ? 0.0 : wl;
      wh = !hi || (nb[1] < 0 && r == DIM) ? 0.0 : wh;
    }
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
      for (int k = 0; k < N; ++k)
        acc[m][1 + r] = __fma_rn(p.basis.Dhat[m][k], w[k], acc[m][1 + r]);
    acc[0][1 + r] = __fma_rn(-wl, p.basis.lhat_l0, acc[0][1 + r]);
    acc[N - 1][1 + r] = __fma_rn(wh, p.basis.lhat_rN, acc[N - 1][1 + r]);
  }
}

// One direction of a lane's line; its contribution is added to R (written by
// the first direction).
template <int DIM, int N, int VF, int SF, bool HG, bool NS, bool XL>
__device__ __forceinline__ void line_sweep(const StageArgs<N>& p, const MeshView& M,
                                           const LineElement<DIM>& E, int dir, int el, int line,
                                           const double* P, double* R, double alpha,
                                           double t_stage) {
  constexpr int NV = DIM + 2, PLANE = LineGeo<DIM, N>::PLANE;
  LinePos<DIM, N> pos;
  pos.set(dir, el, line);
  // the direction's global loads, requested together before the volume term
  int nb[2];
  double ja[N][DIM], nh[DIM], tr[2][NV], acc[N][NV];
  line_metrics<DIM, N, XL>(M, E, dir, pos, ja);
  line_ends<DIM, N>(M, E, dir, pos, nb, nh);
  line_traces<DIM, N>(M, pos, nb, tr);
  LineNode<DIM> q[N];
  const int steep = line_volume<DIM, N, VF, XL>(p, pos, P, ja, q, acc);
  const bool troubled = HG && fabs(alpha - 0.0) > p.atol;
  if constexpr (HG) {
    if (troubled)
      line_blend<DIM, N, VF>(p, M, E, dir, line, pos, P, alpha, acc);
  }
  line_faces<DIM, N, VF, SF>(p, M, E, dir, pos, P, nb, tr, ja[0], nh, t_stage,
                             [&](int s, const double* f) { line_lift<N, NV>(p, s, f, acc); });
  if constexpr (NS) line_viscous<DIM, N, XL>(p, E, dir, pos, nb, acc);
  if (steep) {
    // the direction's terms in R, R's former line in acc
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int m = 0; m < N; ++m) {
        double* r = R + v * PLANE + pos.off[m];
        const double t = *r;
        *r = acc[m][v];
        acc[m][v] = t;
      }
    line_volume_steep<DIM, N, VF>(&p, &M, E, dir, el, line, P, R, steep == 1,
                                  troubled ? 1.0 - alpha : 1.0);
  }
  if (steep && dir == 0) return;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    double r[N];
    if (dir > 0) {
      load_line<XL, N>(R + v * PLANE, pos.off, r);
#pragma unroll
      for (int m = 0; m < N; ++m) acc[m][v] += r[m];
    }
#pragma unroll
    for (int m = 0; m < N; ++m) r[m] = acc[m][v];
    store_line<XL, N>(R + v * PLANE, pos.off, r);
  }
}

// Node data published per node: 1 / (2 rho), p, Chandrashekar rho / p, and
// with shock capturing the indicator variable rho p (hg_node_value[_3d],
// indicator.hpp:148-161, :187-210, gamma = 1.4, every operation rounded as
// written there; quotient_r needs the rounded reciprocal).
template <int DIM, int VF, bool HG>
__device__ __forceinline__ void line_prepare_node(const double* u, double gamma, double& hinv,
                                                  double& pr, double& b, double& ind) {
  const double inv = HG ? 1.0 / u[0] : recip(u[0]);
  hinv = 0.5 * inv;
  double hv[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) hv[d] = __dmul_rn(u[1 + d], hinv);
  pr = __dmul_rn(gamma - 1.0, u[DIM + 1] - line_dot<DIM>(u + 1, hv));
  if constexpr (VF == VF_CHANDRASHEKAR) b = quotient(u[0], pr);
  if constexpr (HG) {
    double vv = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double vd = quotient_r(u[1 + d], u[0], inv);
      const double v2 = __dmul_rn(vd, vd);
      vv = d == 0 ? v2 : __dadd_rn(vv, v2);
    }
    ind = __dmul_rn(
        __dmul_rn(1.4 - 1.0, __dsub_rn(u[DIM + 1], __dmul_rn(__dmul_rn(0.5, u[0]), vv))), u[0]);
  }
}

// Squared modes of one element in node order, read through a plane.
template <int DIM, int N>
struct LineModes {
  const double* plane;
  int el;
  __device__ __forceinline__ double operator[](int node) const {
    LinePos<DIM, N> pos;
    pos.set(0, el, node / N);
    return plane[pos.off[node % N]];
  }
};

// Hennemann-Gassner alpha of the lane's element (indicator.hpp:337-418, 3D
// :430-585): modal transform line by line in the planes S, the energies by the
// element's first lane in the reference's order, every operation rounded as
// written there (identical alpha and troubled-cell flags).  `ind`: the
// indicator variable on the lane's x line.
template <int DIM, int N>
__device__ __forceinline__ double line_alpha(const StageArgs<N>& p, double* S, int el, int line,
                                             bool act, int e, double* ind) {
  using G = LineGeo<DIM, N>;
  auto modal = [&](double* v) {  // v <- Vinv v, sums in index order from 0
    double w[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      double r = 0.0;
#pragma unroll
      for (int k = 0; k < N; ++k) r = __dadd_rn(r, __dmul_rn(p.basis.Vinv[i][k], v[k]));
      w[i] = r;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = w[i];
  };
  LinePos<DIM, N> pos;
  if (act) {
    pos.set(0, el, line);
    modal(ind);
    store_line<true, N>(S, pos.off, ind);
  }
  __syncwarp();
#pragma unroll
  for (int dir = 1; dir < DIM; ++dir) {
    if (act) {
      pos.set(dir, el, line);
      double v[N];
      load_line<false, N>(S, pos.off, v);
      modal(v);
      if (dir == DIM - 1) {
#pragma unroll
        for (int m = 0; m < N; ++m) v[m] = __dmul_rn(v[m], v[m]);
      }
      store_line<false, N>(S, pos.off, v);
    }
    __syncwarp();
  }
  double alpha = 0.0;
  if (act && line == 0) {
    double total, c1, c2;
    const LineModes<DIM, N> m2{S, el};
    if constexpr (DIM == 2)
      hg_energy_sums<N>(m2, &total, &c1, &c2);
    else
      hg_energy_sums_3d<N>(m2, &total, &c1, &c2);
    alpha = hg_alpha_from_energies(total, c1, c2, p.hg_threshold, p.hg_s, p.alpha_min,
                                   p.alpha_max);
    if (p.alpha_out) p.alpha_out[e] = alpha;
  }
  alpha = __shfl_sync(0xffffffffu, alpha, min(el, G::EPW - 1) * G::NF);
  __syncwarp();  // the planes are free again
  return alpha;
}

template <int DIM, int N, int VF, int SF, bool HG, bool NS, bool BATCH, int WPB>
__device__ __forceinline__ void stage_line_body(const StageArgs<N>& p) {
  using G = LineGeo<DIM, N>;
  using K = LineSlots<DIM, VF>;
  constexpr int NV = G::NV, ND = G::ND, NF = G::NF, EPW = G::EPW, PLANE = G::PLANE;
  constexpr int EPB = EPW * WPB;
  // Directions share one copy of the code where a copy each would not stay in
  // the instruction cache.
  constexpr bool ROLL = N > 4;
  constexpr bool XSTORE = N % 2 == 0;  // store by x lines
  extern __shared__ __align__(128) double smem_line[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* P = smem_line + warp * LineShape<DIM, N, VF>::WARP_DOUBLES;
  double* R = P + K::NS * PLANE;

  __shared__ MeshView mesh_s;
  int e0;
  // the tile list, the mesh views and the mesh tables are written by the host
  // or by the context's creation only: they are read before the wait
  if constexpr (BATCH) {
    static_assert(32 * WPB >= int(sizeof(MeshView) / 8), "block narrower than the mesh view");
    e0 = p.tile_e0[blockIdx.x];
    copy_mesh_view(&mesh_s, p.meshes, p.tile_mesh[blockIdx.x], tid);
    __syncthreads();
  } else {
    e0 = (int)blockIdx.x * EPB;
  }
  const MeshView& M = BATCH ? mesh_s : p.mesh;
  const int ew = e0 + warp * EPW;         // the warp's first element
  const int ne = min(EPW, M.nelem - ew);  // its elements (may be <= 0)
  const int el = lane / NF, line = lane - el * NF;
  const bool act = el < ne;
  LineElement<DIM> E;
  E.e = act ? ew + el : 0;
  E.info = M.info + (int64_t)E.e * 12;
#pragma unroll
  for (int c = 0; c < DIM; ++c) E.row[c] = __ldg(E.info + 3 + c);
  stage_dependency_sync();
  const double gamma = p.gamma;
  const double t_stage = p.t_dev ? (*p.t_dev + p.t) : p.t;
  const bool vec = ((reinterpret_cast<uintptr_t>(M.u_in) | reinterpret_cast<uintptr_t>(M.u_n) |
                     reinterpret_cast<uintptr_t>(M.out)) &
                    line_vec_mask<N>()) == 0;
  const int64_t ebase = (int64_t)E.e * (NV * ND);

  // ---- load, node data, publish --------------------------------------------
  double ind[N];  // indicator variable rho p (shock capturing)
  if (act) {
    LinePos<DIM, N> pos;
    pos.set(0, el, line);
    double u[NV][N];
    const double* src = M.u_in + ebase + N * line;
    if (vec) {
#pragma unroll
      for (int v = 0; v < NV; ++v) load_xline<N, true>(src + v * ND, u[v]);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) load_xline<N, false>(src + v * ND, u[v]);
    }
    // u_n is needed at the end only: bring the warp's tile into L2 now
    if (p.a != 0.0 && lane == 0 && (NV * ND) % 2 == 0 &&
        (reinterpret_cast<uintptr_t>(M.u_n) & 15u) == 0)
      bulk_prefetch_l2(M.u_n + ebase, (uint32_t)ne * NV * ND * sizeof(double));
    double hinv[N], pr[N], b[N];
#pragma unroll
    for (int m = 0; m < N; ++m) {
      double un[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) un[v] = u[v][m];
      line_prepare_node<DIM, VF, HG>(un, gamma, hinv[m], pr[m], b[m], ind[m]);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) store_line<true, N>(P + v * PLANE, pos.off, u[v]);
    store_line<true, N>(P + K::HINV * PLANE, pos.off, hinv);
    store_line<true, N>(P + K::P * PLANE, pos.off, pr);
    if constexpr (VF == VF_CHANDRASHEKAR) store_line<true, N>(P + K::B * PLANE, pos.off, b);
  }
  double alpha = 0.0;
  if constexpr (HG) alpha = line_alpha<DIM, N>(p, R, el, line, act, E.e, ind);

  // ---- directions ------------------------------------------------------------
  if constexpr (ROLL) {
#pragma unroll 1
    for (int dir = 0; dir < DIM; ++dir) {
      __syncwarp();
      if (act)
        line_sweep<DIM, N, VF, SF, HG, NS, false>(p, M, E, dir, el, line, P, R, alpha, t_stage);
    }
  } else {
    __syncwarp();
    if (act)
      line_sweep<DIM, N, VF, SF, HG, NS, true>(p, M, E, 0, el, line, P, R, alpha, t_stage);
#pragma unroll
    for (int dir = 1; dir < DIM; ++dir) {
      __syncwarp();
      if (act)
        line_sweep<DIM, N, VF, SF, HG, NS, false>(p, M, E, dir, el, line, P, R, alpha, t_stage);
    }
  }
  __syncwarp();

  // ---- -1/J, SSPRK3 combination, store -----------------------------------------
  double dacc[3] = {0.0, 0.0, 0.0};
  if (act) {
    bool bad = false;
    double mij[N], un[NV][N], vals[N][NV];
    const double* mij_e = M.mij + (int64_t)E.e * ND;
    LinePos<DIM, N> pos;
    pos.set(XSTORE ? 0 : DIM - 1, el, line);
    if constexpr (XSTORE) {
      load_xline<N, true>(mij_e + pos.first, mij);
      if (p.a != 0.0) {
        const double* src = M.u_n + ebase + pos.first;
        if (vec) {
#pragma unroll
          for (int v = 0; v < NV; ++v) load_xline<N, true>(src + v * ND, un[v]);
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) load_xline<N, false>(src + v * ND, un[v]);
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < N; ++m) mij[m] = __ldg(mij_e + pos.first + m * pos.stride);
      if (p.a != 0.0) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
          for (int m = 0; m < N; ++m)
            un[v][m] = M.u_n[ebase + v * ND + pos.first + m * pos.stride];
      }
    }
    double cm[N];
#pragma unroll
    for (int m = 0; m < N; ++m) cm[m] = __dmul_rn(M.c, mij[m]);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double r[N], ui[N];
      load_line<XSTORE, N>(R + v * PLANE, pos.off, r);
      if (p.b != 0.0) load_line<XSTORE, N>(P + v * PLANE, pos.off, ui);
#pragma unroll
      for (int m = 0; m < N; ++m) {
        double val = __dmul_rn(r[m], cm[m]);
        if (p.b != 0.0) val = __fma_rn(p.b, ui[m], val);
        if (p.a != 0.0) val = __fma_rn(p.a, un[v][m], val);
        bad |= !isfinite(val);
        vals[m][v] = val;
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double r[N];
#pragma unroll
      for (int m = 0; m < N; ++m) r[m] = vals[m][v];
      double* dst = M.out + ebase + v * ND + pos.first;
      if constexpr (XSTORE) {
        if (vec)
          store_xline<N, true>(dst, r);
        else
          store_xline<N, false>(dst, r);
      } else {
#pragma unroll
        for (int m = 0; m < N; ++m) dst[m * pos.stride] = r[m];
      }
    }
    if (bad) atomicOr(p.nonfinite, 1u);
    if constexpr (!BATCH) {
      if (p.diag) {
#pragma unroll
        for (int m = 0; m < N; ++m)
          diag_add_node<DIM, N>(vals[m], p.basis, pos.first + m * pos.stride, -mij[m], gamma,
                                p.inv_gm1, dacc);
      }
    }
  }
  if constexpr (!BATCH) {
    if (p.diag) {
      __shared__ double red[3 * WPB];
      diag_block_store<32 * WPB>(dacc, red, p.diag + 3 * (int64_t)blockIdx.x);
    }
  }
}

// MINB resident blocks per SM are requested from the register allocator.
template <int DIM, int N, int VF, int SF, bool HG, bool NS, bool BATCH, int WPB, int MINB>
__global__ void __launch_bounds__(32 * WPB, MINB) stage_line_kernel(const __grid_constant__ StageArgs<N> p) {
  stage_line_body<DIM, N, VF, SF, HG, NS, BATCH, WPB>(p);
}

// ---------------------------------------------------------------------------
// The same arithmetic with a block per group of EPW elements, for meshes that
// do not fill the GPU with one warp per group: the warps of the block take
//   load   the group's nodes, one per thread;
//   sweep  warp d < DIM: volume term of direction d; warp DIM + d: the face
//          fluxes of direction d (into F); with shock capturing one more warp:
//          alpha; then warp d: blend, lifting, viscous terms -> its planes R_d;
//   store  the group's nodes, one per thread: R_0 + R_1 [+ R_2], -1/J, SSPRK3
//          combination.
// The chain of dependent instructions of a lane is about half of the line
// sweep's; every sum is formed in the same order, so the results are the line
// sweep's bit for bit.
// ---------------------------------------------------------------------------
template <int DIM, int N, int VF, bool HG>
struct SplitShape {
  using G = LineGeo<DIM, N>;
  static constexpr int WARPS = 2 * DIM + (HG ? 1 : 0);
  static constexpr int NT = 32 * WARPS;
  static constexpr int NS = LineSlots<DIM, VF>::NS;
  static constexpr int FACE = 32 * G::NV;  // one (direction, side): [var][lane]
  static constexpr int DOUBLES = (NS + DIM * G::NV + (HG ? 1 : 0)) * G::PLANE + DIM * 2 * FACE;
  static constexpr size_t smem_bytes = sizeof(double) * (size_t)DOUBLES;
  static_assert(!HG || G::EPW <= 16, "alpha per element");
};

template <int DIM, int N, int VF, int SF, bool HG, bool NS, bool BATCH>
__device__ __forceinline__ void stage_split_body(const StageArgs<N>& p) {
  using G = LineGeo<DIM, N>;
  using K = LineSlots<DIM, VF>;
  using S = SplitShape<DIM, N, VF, HG>;
  constexpr int NV = G::NV, ND = G::ND, NF = G::NF, EPW = G::EPW, PLANE = G::PLANE, NT = S::NT;
  constexpr int PASSES = (EPW * ND + NT - 1) / NT;
  extern __shared__ __align__(128) double smem_split[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* P = smem_split;
  double* R = P + K::NS * PLANE;                  // [dir][var]
  double* F = R + DIM * NV * PLANE;               // [dir][side][var][lane]
  double* I = F + DIM * 2 * S::FACE;              // indicator plane (HG)
  __shared__ double alpha_s[HG ? EPW : 1];

  __shared__ MeshView mesh_s;
  int e0;
  // tables are read before the wait (see stage_line_body)
  if constexpr (BATCH) {
    static_assert(NT >= int(sizeof(MeshView) / 8), "block narrower than the mesh view");
    e0 = p.tile_e0[blockIdx.x];
    copy_mesh_view(&mesh_s, p.meshes, p.tile_mesh[blockIdx.x], tid);
    __syncthreads();
  } else {
    e0 = (int)blockIdx.x * EPW;
  }
  const MeshView& M = BATCH ? mesh_s : p.mesh;
  const int ne = min(EPW, M.nelem - e0);
  const int el = lane / NF, line = lane - el * NF;
  const bool act = el < ne;
  const int dir = warp % DIM;
  const bool volume = warp < DIM, faces = !volume && warp < 2 * DIM;
  LineElement<DIM> E;
  E.e = act ? e0 + el : e0;
  E.info = M.info + (int64_t)E.e * 12;
#pragma unroll
  for (int c = 0; c < DIM; ++c) E.row[c] = __ldg(E.info + 3 + c);
  LinePos<DIM, N> pos;
  pos.set(dir, el, line);
  int nb[2];
  double ja[N][DIM], nh[DIM], tr[2][NV];
  if (volume) {
    line_metrics<DIM, N, false>(M, E, dir, pos, ja);
    nb[0] = __ldg(E.info + 6 + 2 * dir);
    nb[1] = __ldg(E.info + 7 + 2 * dir);
  } else if (faces) {
    line_ends<DIM, N>(M, E, dir, pos, nb, nh);
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      ja[0][c] = __ldg(M.tab.ja[dir][c] + (int64_t)E.row[c] * ND + pos.first);
  }
  stage_dependency_sync();
  const double gamma = p.gamma;
  const double t_stage = p.t_dev ? (*p.t_dev + p.t) : p.t;
  const int64_t gbase = (int64_t)e0 * (NV * ND);
  const bool with_n = p.a != 0.0;

  // ---- load, node data, publish --------------------------------------------
  int opos[PASSES];
#pragma unroll
  for (int k = 0; k < PASSES; ++k) {
    const int t = tid + k * NT, te = t / ND, node = t - te * ND;
    opos[k] = te < ne ? LinePos<DIM, N>::slot(0, te, node / N, node % N) : -1;
    if (opos[k] < 0) continue;
    const int o = opos[k];
    double u[NV], hinv, pr, b = 0.0, ind = 0.0;
    const double* src = M.u_in + gbase + (int64_t)te * (NV * ND) + node;
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = __ldg(src + v * ND);
    line_prepare_node<DIM, VF, HG>(u, gamma, hinv, pr, b, ind);
#pragma unroll
    for (int v = 0; v < NV; ++v) P[v * PLANE + o] = u[v];
    P[K::HINV * PLANE + o] = hinv;
    P[K::P * PLANE + o] = pr;
    if constexpr (VF == VF_CHANDRASHEKAR) P[K::B * PLANE + o] = b;
    if constexpr (HG) I[o] = ind;
  }
  if (faces) line_traces<DIM, N>(M, pos, nb, tr);
  __syncthreads();

  // ---- volume terms, face fluxes, alpha --------------------------------------
  double acc[N][NV];
  int steep = 0;
  double* Rd = R + dir * (NV * PLANE);
  if (volume) {
    if (act) {
      LineNode<DIM> q[N];
      steep = line_volume<DIM, N, VF, false>(p, pos, P, ja, q, acc);
      // A steep line's term in straight code right here (this kernel's chain is
      // short: the call of line_volume_steep cost KH 64^2 1.0 of 5.8 us), kept
      // in R_d until the other terms are there: the same sum in the same order.
      // Long lines take the call at the end like the line sweep.
      if ((steep == 1 && N <= (DIM == 2 ? 6 : 4)) || (steep == 2 && N <= 4)) {
        // copies the compiler cannot relate to the first pass, or it would
        // keep that pass's intermediate values in registers
#pragma unroll
        for (int m = 0; m < N; ++m) {
          asm volatile("" : "+d"(q[m].rho), "+d"(q[m].p), "+d"(q[m].x), "+d"(q[m].y));
#pragma unroll
          for (int d = 0; d < DIM; ++d) asm volatile("" : "+d"(q[m].hv[d]), "+d"(ja[m][d]));
        }
        if constexpr (N <= (DIM == 2 ? 6 : 4)) {
          if (steep == 1)
            line_pairs<DIM, N, VF, MEAN_LONG>(p, q, ja, acc);
          else if constexpr (N <= 4)
            line_pairs<DIM, N, VF, MEAN_GENERAL>(p, q, ja, acc);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
          for (int m = 0; m < N; ++m) {
            Rd[v * PLANE + pos.off[m]] = acc[m][v];
            acc[m][v] = 0.0;
          }
        steep = 4;
      }
    }
  } else if (faces) {
    if (act)
      line_faces<DIM, N, VF, SF>(p, M, E, dir, pos, P, nb, tr, ja[0], nh, t_stage,
                                 [&](int s, const double* f) {
#pragma unroll
                                   for (int v = 0; v < NV; ++v)
                                     F[(dir * 2 + s) * S::FACE + v * 32 + lane] = f[v];
                                 });
  } else if constexpr (HG) {
    double ind[N];
    LinePos<DIM, N> px;
    px.set(0, el, line);
    if (act) load_line<true, N>(I, px.off, ind);
    const double a = line_alpha<DIM, N>(p, I, el, line, act, E.e, ind);
    if (act && line == 0) alpha_s[el] = a;
  }
  // u_n and -1/J of the thread's nodes, on their way during the barrier
  double un[PASSES][NV], mij[PASSES];
#pragma unroll
  for (int k = 0; k < PASSES; ++k) {
    if (opos[k] < 0) continue;
    const int t = tid + k * NT, te = t / ND, node = t - te * ND;
    mij[k] = __ldg(M.mij + (int64_t)e0 * ND + t);
    if (with_n) {
#pragma unroll
      for (int v = 0; v < NV; ++v)
        un[k][v] = M.u_n[gbase + (int64_t)te * (NV * ND) + v * ND + node];
    }
  }
  __syncthreads();
  if (volume && act) {
    const double alpha = HG ? alpha_s[el] : 0.0;
    const bool troubled = HG && fabs(alpha - 0.0) > p.atol;
    if constexpr (HG) {
      if (troubled)
        line_blend<DIM, N, VF>(p, M, E, dir, line, pos, P, alpha, acc);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      double f[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) f[v] = F[(dir * 2 + s) * S::FACE + v * 32 + lane];
      line_lift<N, NV>(p, s, f, acc);
    }
    if constexpr (NS) line_viscous<DIM, N, false>(p, E, dir, pos, nb, acc);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double r[N];
#pragma unroll
      for (int m = 0; m < N; ++m)
        r[m] = steep == 4
                   ? __fma_rn(troubled ? 1.0 - alpha : 1.0, Rd[v * PLANE + pos.off[m]], acc[m][v])
                   : acc[m][v];
      store_line<false, N>(Rd + v * PLANE, pos.off, r);
    }
    if (steep == 1 || steep == 2)
      line_volume_steep<DIM, N, VF>(&p, &M, E, dir, el, line, P, Rd, steep == 1,
                                    troubled ? 1.0 - alpha : 1.0);
  }
  __syncthreads();

  // ---- -1/J, SSPRK3 combination, store -----------------------------------------
  double dacc[3] = {0.0, 0.0, 0.0};
  bool bad = false;
#pragma unroll
  for (int k = 0; k < PASSES; ++k) {
    const int o = opos[k];
    if (o < 0) continue;
    const int t = tid + k * NT, te = t / ND, node = t - te * ND;
    const double cm = __dmul_rn(M.c, mij[k]);
    double vals[NV];
    double* dst = M.out + gbase + (int64_t)te * (NV * ND) + node;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double r = R[v * PLANE + o];
#pragma unroll
      for (int d = 1; d < DIM; ++d) r = R[(d * NV + v) * PLANE + o] + r;
      double val = __dmul_rn(r, cm);
      if (p.b != 0.0) val = __fma_rn(p.b, P[v * PLANE + o], val);
      if (with_n) val = __fma_rn(p.a, un[k][v], val);
      bad |= !isfinite(val);
      dst[v * ND] = val;
      vals[v] = val;
    }
    if constexpr (!BATCH) {
      if (p.diag) diag_add_node<DIM, N>(vals, p.basis, node, -mij[k], gamma, p.inv_gm1, dacc);
    }
  }
  if (bad) atomicOr(p.nonfinite, 1u);
  if constexpr (!BATCH) {
    if (p.diag) {
      __shared__ double red[3 * S::WARPS];
      diag_block_store<NT>(dacc, red, p.diag + 3 * (int64_t)blockIdx.x);
    }
  }
}

template <int DIM, int N, int VF, int SF, bool HG, bool NS, bool BATCH, int MINB>
__global__ void __launch_bounds__(SplitShape<DIM, N, VF, HG>::NT, MINB)
    stage_split_kernel(const __grid_constant__ StageArgs<N> p) {
  stage_split_body<DIM, N, VF, SF, HG, NS, BATCH>(p);
}

}  // namespace dgsem
