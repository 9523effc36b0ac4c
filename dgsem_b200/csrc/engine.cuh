// Type-erased solver engine: one instantiation per supported template
// combination (dimension, nodes per direction, volume flux, surface flux,
// shock capturing, Navier-Stokes).  Each engine carries several launch shapes
// of the same right-hand side; shapes 0-2 give the same bits, the others agree
// with them to rounding (other orders of summation, and logarithms where 0-2
// take a series).  So the autotuner's choice (capi.cu: dgsem_autotune), which is
// by time, can change the last bits of a result; a fixed shape never does.
// The C ABI context owns one engine.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <memory>
#include <utility>

#include "br1_kernel.cuh"
#include "stage_kernel.cuh"
#include "stage_line_kernel.cuh"
#include "stage_node2_kernel.cuh"
#include "stage_node_kernel.cuh"
#include "stage_pipe_kernel.cuh"
#include "tables.hpp"

namespace dgsem {

// Everything an engine needs that does not depend on its template arguments.
struct EngineConfig {
  int ndims;
  int n;
  int64_t cells[3];
  int periodic[3];
  int64_t nelem;
  double gamma;
  double mu, prandtl;
  double alpha_max, alpha_min, atol;
  double hg_threshold, hg_s;
  DeviceTables tab;
  BcParams bc;
  BasisTables basis;
  unsigned int* nonfinite;  // device flag
  double* visc;             // Navier-Stokes contravariant viscous flux (br1_kernel.cuh)
  double* grad;             // adjoint: velocity gradient written with it (may be null)
  // per-element info (node_element_info layout, 12 ints per element) and
  // -1/J per node [E][n^d], computed once per context.  The line shapes and the
  // viscous flux kernel read them unconditionally; null only in the shared
  // configuration of a batch group, whose launches take them from the mesh views
  const int* elem_info;
  const double* mij;
  // failure-path testing (StageArgs::wait_limit_ns / skip_tile_copy)
  unsigned long long wait_limit_ns;
  int skip_tile_copy;
};

// Launch-shape variants: 0-2 line shapes (stage_line_kernel.cuh), 3-4
// node-parallel (stage_node_kernel.cuh), 5 persistent node-parallel with TMA
// tile streaming (stage_pipe_kernel.cuh; single-mesh launches; split form
// without shock capturing or viscous terms, an even number of doubles per
// element), 6 two nodes per thread (stage_node2_kernel.cuh; 3D, n = 2 or 4,
// split form without shock capturing or viscous terms).
constexpr int kNumVariants = 7;

class EngineBase {
 public:
  virtual ~EngineBase() = default;
  // out = a*u_n + b*u_in + c*RHS(u_in, t); alpha_out optional; diag
  // optional: per-block volume integrals of `out` (StageArgs::diag), as many
  // slots as diag_slots() returns.
  virtual cudaError_t stage(const EngineConfig& cfg, const double* u_n,
                            const double* u_in, double* out, double a, double b,
                            double c, double t, const double* t_dev,
                            double* alpha_out, cudaStream_t s, double* diag = nullptr) = 0;
  // number of diag slots (blocks) the last stage launch with diag wrote
  virtual int64_t last_diag_slots() const = 0;
  // Fills the per-mesh tables of the stage kernels (EngineConfig::
  // elem_info / MeshView::info, 12 ints per element; ::mij, -1/J per node)
  // of the mesh `m` (its cells, periodicity, element count and metric
  // tables) on stream s.
  virtual cudaError_t build_mesh_tables(const MeshView& m, int* info, double* mij,
                                        cudaStream_t s) const = 0;
  // Batched launch over a tile list (mesh index and first element per block)
  // of meshes sharing this engine's scheme and degree; per-mesh data in
  // `meshes` (device array).  Tiles are built with elements_per_block().
  virtual cudaError_t batch_stage(const EngineConfig& cfg, const MeshView* meshes,
                                  const int* tile_mesh, const int* tile_e0, int ntiles,
                                  double a, double b, double t, const double* t_dev,
                                  cudaStream_t s) = 0;
  virtual int kernels_per_stage() const = 0;
  virtual int elements_per_block() const = 0;
  virtual int threads_per_block() const = 0;
  virtual size_t smem_bytes() const = 0;
  // launch-shape variant in [0, num_variants())
  virtual void set_variant(int v) = 0;
  virtual int variant() const = 0;
  // elements of the mesh (of all meshes of a batch group): launch shape 0
  // depends on it
  virtual void set_mesh_size(int64_t nelem) = 0;
  virtual int num_variants() const = 0;
  // stage kernel that the current launch shape runs
  virtual const char* kernel_name() const = 0;
};

std::unique_ptr<EngineBase> make_engine(int ndims, int n, int vf, int sf,
                                        bool hg, bool ns);

// Nodal initial condition on one mesh (capi.cu).
cudaError_t launch_initial(int kind, int ndims, int n, const int64_t* cells, int64_t nelem,
                           const DeviceTables& tab, const BcParams& bc, double gamma,
                           const double* params, double* u, cudaStream_t s);

template <int N>
inline void fill_basis_const(const BasisTables& b, BasisConst<N>* out) {
  for (int i = 0; i < N; ++i) {
    for (int j = 0; j < N; ++j) {
      out->Dsplit[i][j] = b.Dsplit[i][j];
      out->Dhat[i][j] = b.Dhat[i][j];
      out->Vinv[i][j] = b.Vinv[i][j];
    }
    out->inv_w[i] = b.inv_weights[i];
    out->w[i] = b.weights[i];
  }
  out->lhat_l0 = b.lhat_left[0];
  out->lhat_rN = b.lhat_right[N - 1];
}

// The arguments of one stage launch that do not depend on the mesh.
template <int N>
inline StageArgs<N> stage_args_common(const EngineConfig& cfg, double a, double b, double t,
                                      const double* t_dev, double* alpha_out) {
  StageArgs<N> args{};
  args.a = a;
  args.b = b;
  args.t = t;
  args.t_dev = t_dev;
  args.gamma = cfg.gamma;
  args.inv_gm1 = 1.0 / (cfg.gamma - 1.0);
  args.alpha_max = cfg.alpha_max;
  args.alpha_min = cfg.alpha_min;
  args.atol = cfg.atol;
  args.hg_threshold = cfg.hg_threshold;
  args.hg_s = cfg.hg_s;
  args.alpha_out = alpha_out;
  args.nonfinite = cfg.nonfinite;
  args.visc = cfg.visc;
  args.bc = cfg.bc;
  args.wait_limit_ns = cfg.wait_limit_ns;
  args.skip_tile_copy = cfg.skip_tile_copy;
  fill_basis_const<N>(cfg.basis, &args.basis);
  return args;
}

// Line shapes (stage_line_kernel.cuh): 0 = the split or the sweep form by the
// mesh's size (Engine::split_waves), 1 = split, 2 = sweep with another
// register cap than 0's.  Resident blocks per SM requested from the register
// allocator: the sweeps get 168 registers (12 warps per SM) where a line's
// data fit them, 255 (8 warps) at long lines, and shape 2 128 (16 warps) at
// short ones (2D n = 2: 111 us per stage of 640 000 elements against 116).
template <int DIM, int N, int V>
struct LineLaunch {
  static constexpr int WPB = 2;
  static constexpr bool LONG = N > 5 || (DIM == 3 && N == 5);
  static constexpr int MINB = V == 0 ? (LONG ? 4 : 6) : N <= 4 ? 8 : LONG ? 6 : 4;
  static constexpr int NT = 32 * WPB;
};
template <int DIM, int N, bool HG>
struct SplitLaunch {
  static constexpr int MINB = DIM == 3 ? 2 : N <= 4 ? (HG ? 3 : 4) : N <= 6 ? (HG ? 2 : 3) : 2;
};

// Fraction of the lanes of its warps that a block of `threads` threads uses.
constexpr double lane_use(int threads) { return double(threads) / (((threads + 31) / 32) * 32); }

// Elements per block of the node-parallel shapes: 128 / n^d (about 128
// threads), unless that leaves more than 5 % of the block's warp lanes idle
// (n^d = 36, 49 in 2D; 27 in 3D); then the smallest count up to 256 threads
// that fills at least 95 % of them (a partly filled warp costs a whole
// warp's issue slots).
constexpr int node_elements_per_block(int nd) {
  const int e0 = 128 / nd > 0 ? 128 / nd : 1;
  if (lane_use(e0 * nd) >= 0.95) return e0;
  for (int e = e0 + 1; e * nd <= 256; ++e)
    if (lane_use(e * nd) >= 0.95) return e;
  return e0;
}

// Node-parallel variants: one thread per node; variant 3 caps registers at
// ~72 per thread (7 resident blocks of 128 threads), variant 4 leaves them to
// the compiler.
template <int DIM, int N>
struct NodeLaunch {
  static constexpr int ND = ipow(N, DIM);
  static constexpr int EPB = node_elements_per_block(ND);
  static constexpr int NT = EPB * ND;
  static constexpr int MINB = 65536 / (NT * 72) > 1 ? 65536 / (NT * 72) : 1;
};

// Launches a stage kernel with programmatic stream serialization: the GPU
// may schedule its blocks while the previous kernel on `s` drains (hiding the
// launch gap between the three stages of a step); griddepcontrol.wait
// (stage_dependency_sync) holds every block until that kernel has completed and
// flushed its writes.  After a copy, a memset or an event the launch is ordered
// as usual.  Before the wait a kernel reads only what no kernel of a step
// writes: its arguments, the metric tables, element info and -1/J
// (element_tables_kernel writes the last two at creation, which ends with a
// device synchronisation), mesh views and tile lists (host copies).  Whoever
// writes one of these on the device has to synchronise before the next launch.
template <class... P, class... A>
void launch_stage_kernel(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                         cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Contravariant viscous flux of u into `visc` (and the adjoint's velocity
// gradient into `grad`); either output may be null.
template <int DIM, int N>
inline void launch_viscous_flux(const EngineConfig& cfg, const double* u, double* visc,
                                double* grad, cudaStream_t s) {
  using S = ViscShape<DIM, N>;
  ViscArgs<N> a{};
  a.u = u;
  a.visc = visc;
  a.grad = grad;
  a.nelem = (int)cfg.nelem;
  a.gamma = cfg.gamma;
  a.mu = cfg.mu;
  a.kappa = cfg.gamma / ((cfg.gamma - 1.0) * cfg.prandtl);
  a.tab = cfg.tab;
  a.info = cfg.elem_info;
  a.mij = cfg.mij;
  fill_basis_const<N>(cfg.basis, &a.basis);
  for (int f = 0; f < 2 * DIM; ++f) a.bc_kind[f] = cfg.bc.kind[f];
  const unsigned blocks = (unsigned)((cfg.nelem + S::EPB - 1) / S::EPB);
  launch_stage_kernel(viscous_flux_kernel<DIM, N>, blocks, 32 * S::WPB, S::smem_bytes, s, a);
}

template <int DIM, int N>
inline void set_viscous_flux_attributes() {
  cudaFuncSetAttribute(viscous_flux_kernel<DIM, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)ViscShape<DIM, N>::smem_bytes);
}

template <int DIM, int N, int VF, int SF, bool HG, bool NS = false>
class Engine final : public EngineBase {
 public:
  static constexpr bool kBatch = !NS && !HG;

  using LG = LineGeo<DIM, N>;
  using SSh = SplitShape<DIM, N, VF, HG>;
  template <int V, bool B>
  static auto line_kernel() {
    using L = LineLaunch<DIM, N, V>;
    return stage_line_kernel<DIM, N, VF, SF, HG, NS, B, L::WPB, L::MINB>;
  }
  template <bool B>
  static auto split_kernel() {
    return stage_split_kernel<DIM, N, VF, SF, HG, NS, B, SplitLaunch<DIM, N, HG>::MINB>;
  }
  static constexpr int LINE_WPB = LineLaunch<DIM, N, 0>::WPB;
  static constexpr int LINE_NT = LineLaunch<DIM, N, 0>::NT;
  static constexpr int LINE_EPB = LG::EPW * LINE_WPB;
  static constexpr size_t LINE_SMEM = LineShape<DIM, N, VF>::smem_bytes(LINE_WPB);
  // whether the current line shape runs in the split form
  bool use_split() const { return variant_ == 1 || (variant_ == 0 && split_); }

  // Loads and configures the kernels of one launch shape (and of its batched
  // and fallback forms), once per engine: only shapes that are selected, since
  // a kernel's code goes to the device at its first use.  On the device the
  // engine was created for, whichever is current in the call that selects.
  void load_variant(int v) {
    if (loaded_ & (1u << v)) return;
    loaded_ |= 1u << v;
    int current = device_;
    cudaGetDevice(&current);
    if (current != device_) cudaSetDevice(device_);
    auto attr = [](auto kernel, size_t smem) {
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    };
    auto node = [&](auto cap) {
      constexpr bool CAP = decltype(cap)::value;
      attr(node_kernel<false, CAP>(), NSh::smem_bytes);
      if constexpr (kBatch) attr(node_kernel<true, CAP>(), NSh::smem_bytes);
    };
    auto sweep = [&](auto v_c) {
      constexpr int V = decltype(v_c)::value;
      attr(line_kernel<V, false>(), LINE_SMEM);
      if constexpr (kBatch) attr(line_kernel<V, true>(), LINE_SMEM);
    };
    if constexpr (NS) set_viscous_flux_attributes<DIM, N>();
    if (v == 1 || (v == 0 && split_)) {
      attr(split_kernel<false>(), SSh::smem_bytes);
      if constexpr (kBatch) attr(split_kernel<true>(), SSh::smem_bytes);
    } else if (v == 0) {
      sweep(std::integral_constant<int, 0>{});
    } else if (v == 2) {
      sweep(std::integral_constant<int, 2>{});
    } else if (v == 4) {
      node(std::false_type{});
    } else {
      node(std::true_type{});  // 3; 5 and 6 fall back to it
    }
    if constexpr (kPipe)
      if (v == 5) attr(pipe_kernel(), PSh::smem_bytes);
    if constexpr (kNode2)
      if (v == 6) attr(node2_kernel(), Node2Shape<N, VF>::smem_bytes);
    if (current != device_) cudaSetDevice(current);
  }

  // Shape 0 runs the split form on meshes that give the sweep fewer than
  // split_waves() waves: `nelem` / EPW warps on WPB * MINB warp slots per SM.
  // A sweep's time is one lane's chain per wave; the split form's chain is about
  // half of it, but its blocks fill the GPU sooner.  Both give the same bits.
  // Measured on a B200 (1776 slots, 1184 at long lines) at 14 sizes of 0.1 to 3.3
  // waves per form; split / sweep time on both sides of the line, at waves:
  //   2D Chandrashekar, vortex    n = 4: 0.94 at 0.95, 1.07 at 1.20
  //                               n = 2, 3, 5-8: 0.94-1.04 at 0.95, 1.01-1.16 at 1.2
  //      Ranocha, HLLC (KH), n = 4  0.88, 0.91 at 0.70, 1.03, 1.10 at 0.95
  //      Kennedy-Gruber           n = 2, 3: 0.87, 0.83 at 0.70, 1.00 at 0.85
  //                               n = 4, 5, 6: 0.95, 0.79, 0.94 at 0.50, 1.15, 0.95,
  //                               0.98 at 0.70, 1.27, 1.16, 1.17 at 0.85
  //                               n = 7, 8: 0.75, 0.68 at 0.20, 1.16, 1.06 at 0.50
  //      viscous                  n = 3: 0.92 at 0.70, 1.00 at 0.85
  //                               n = 4, 5, 8: 1.01, 0.98, 1.02 at 0.70
  //   3D n = 2, 4                 0.94, 0.94 at 0.35, 0.98, 1.08 at 0.50
  //      n = 3                    0.89 at 0.20, 1.13 at 0.35 (Kennedy-Gruber 0.90 at 0.50)
  //      n = 5                    0.97 at 0.68, 1.12 at 0.84 (0.91 at 1.02, where the
  //                               sweep starts its second wave); viscous 0.96, 1.05
  // With shock capturing the line depends on the flow, because steep lines
  // lengthen the sweep's chain: the two crossings are, in waves,
  //   2D, Kelvin-Helmholtz / double Mach   n = 2, 3, 4: 0.8, 0.8, 0.7 / 1.0, 1.6, 2.0
  //                               n = 5: 0.6 / 1.7;  n = 6, 8: 0.3, 0.3 / 1.7, 2.2
  //   2D viscous KH               n = 3, 4, 5, 8: 0.3, 0.2, 0.3, 0.5
  //   3D Taylor-Green             n = 2, 3, 4, 5: 0.27, 0.27, 0.3, 0.55
  // and the line lies where neither loses more than 1.45 (2D) or 1.2 (3D).
  void set_mesh_size(int64_t nelem) override {
    using L = LineLaunch<DIM, N, 0>;
    int sms = 0;
    cudaGetDevice(&device_);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_);
    const int64_t warps = (nelem + LG::EPW - 1) / LG::EPW;
    split_ = (double)warps < split_waves() * (sms * L::WPB * L::MINB);
    loaded_ &= ~1u;
    load_variant(variant_);
  }
  static constexpr double split_waves() {
    if (DIM == 3) return N <= 4 ? 0.4 : HG ? 0.6 : 0.7;
    if (HG) return N <= 4 ? 1.13 : N > 5 ? 0.68 : NS ? 0.45 : 0.6;
    if (NS) return N <= 3 ? 0.8 : 0.7;
    if (VF == VF_KENNEDY_GRUBER) return N <= 3 ? 0.85 : N <= 6 ? 0.68 : 0.4;
    return N <= 5 ? 1.0 : 0.95;
  }

  // node-parallel shapes: split form with shock capturing or with the
  // Navier-Stokes viscous terms; batched node launches with neither
  static constexpr bool kNode = true;
  using NL = NodeLaunch<DIM, N>;
  using NSh = NodeShape<DIM, N, VF, NL::EPB, HG, NS>;
  template <bool B, bool CAP>
  static auto node_kernel() {
    if constexpr (CAP)
      return stage_node_kernel_capped<DIM, N, VF, SF, NL::EPB, B, NL::MINB, HG, NS>;
    else
      return stage_node_kernel<DIM, N, VF, SF, NL::EPB, B, HG, NS>;
  }
  // launches without u_n (a == 0) request the smaller shared-memory size
  static size_t node_smem(const StageArgs<N>& args) {
    return args.a != 0.0 ? NSh::smem_bytes : NSh::smem_bytes_base;
  }
  template <bool CAP>
  void launch_node(const StageArgs<N>& args, int64_t nelem, cudaStream_t s) const {
    if constexpr (kNode) {
      const int64_t blocks = (nelem + NL::EPB - 1) / NL::EPB;
      last_grid_ = blocks;
      launch_stage_kernel(node_kernel<false, CAP>(), (unsigned)blocks, NL::NT, node_smem(args), s,
                          args);
    }
  }
  template <bool CAP>
  void launch_node_batch(const StageArgs<N>& args, int ntiles, cudaStream_t s) const {
    if constexpr (kBatch)
      launch_stage_kernel(node_kernel<true, CAP>(), (unsigned)ntiles, NL::NT, node_smem(args), s,
                          args);
  }

  // shape 6: two nodes per thread (3D, n = 2 or 4, split form)
  static constexpr bool kNode2 = DIM == 3 && (N == 2 || N == 4) && !HG && !NS;
  template <int NN = N>
  static auto node2_kernel() {
    return stage_node2_kernel<NN, VF, SF>;
  }
  void launch_node2(const StageArgs<N>& args, int64_t nelem, cudaStream_t s) const {
    if constexpr (kNode2) {
      using S2 = Node2Shape<N, VF>;
      const int64_t blocks = (nelem + Node2Launch<N>::EPB - 1) / Node2Launch<N>::EPB;
      last_grid_ = blocks;
      launch_stage_kernel(node2_kernel(), (unsigned)blocks, Node2Launch<N>::NT,
                          args.a != 0.0 ? S2::smem_bytes : S2::smem_bytes_base, s, args);
    } else {
      launch_node<true>(args, nelem, s);
    }
  }

  using PSh = PipeShape<DIM, N, VF, NL::EPB>;
  static constexpr bool kPipe = kBatch && PSh::kSupported;
  static auto pipe_kernel() {
    return stage_pipe_kernel<DIM, N, VF, SF, NL::EPB, PSh::MINB>;
  }
  // Persistent launch: as many blocks as fit on the device at once.  Falls
  // back to the node-parallel shape when a state pointer is not 16-byte
  // aligned (bulk copies need it).
  void launch_pipe(const StageArgs<N>& args, int64_t nelem, cudaStream_t s) const {
    if constexpr (kPipe) {
      const uintptr_t al = reinterpret_cast<uintptr_t>(args.mesh.u_in) |
                           reinterpret_cast<uintptr_t>(args.mesh.u_n);
      if (al & 15u) {
        launch_node<true>(args, nelem, s);
        return;
      }
      if (pipe_blocks_ == 0) {
        int dev = 0, nsm = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pipe_kernel(), PSh::NT,
                                                      PSh::smem_bytes);
        pipe_blocks_ = (nsm > 0 ? nsm : 1) * (per_sm > 0 ? per_sm : 1);
      }
      const int64_t ntiles = (nelem + NL::EPB - 1) / NL::EPB;
      const int64_t blocks = ntiles < pipe_blocks_ ? ntiles : pipe_blocks_;
      last_grid_ = blocks;
      launch_stage_kernel(pipe_kernel(), (unsigned)blocks, PSh::NT, PSh::smem_bytes, s, args,
                          (int)ntiles);
    } else {
      launch_node<true>(args, nelem, s);
    }
  }

  StageArgs<N> common_args(const EngineConfig& cfg, double a, double b, double t,
                           const double* t_dev, double* alpha_out) const {
    StageArgs<N> args = stage_args_common<N>(cfg, a, b, t, t_dev, alpha_out);
    for (int i = 0; i < N; ++i)
      for (int j = 0; j < N; ++j)
        args.basis.Dvol[i][j] = LineScale<VF>::value * args.basis.Dsplit[i][j];
    return args;
  }

  // line shapes; `grid` blocks of elements_per_block() elements
  template <bool B>
  void launch_line(const StageArgs<N>& args, unsigned grid, cudaStream_t s) const {
    if (use_split())
      launch_stage_kernel(split_kernel<B>(), grid, SSh::NT, SSh::smem_bytes, s, args);
    else if (variant_ == 2)
      launch_stage_kernel(line_kernel<2, B>(), grid, LINE_NT, LINE_SMEM, s, args);
    else
      launch_stage_kernel(line_kernel<0, B>(), grid, LINE_NT, LINE_SMEM, s, args);
  }

  cudaError_t stage(const EngineConfig& cfg, const double* u_n,
                    const double* u_in, double* out, double a, double b,
                    double c, double t, const double* t_dev,
                    double* alpha_out, cudaStream_t s, double* diag = nullptr) override {
    StageArgs<N> args = common_args(cfg, a, b, t, t_dev, alpha_out);
    args.diag = diag;
    args.mesh.u_in = u_in;
    args.mesh.u_n = u_n;
    args.mesh.out = out;
    args.mesh.c = c;
    for (int i = 0; i < 3; ++i) {
      args.mesh.cells[i] = (int)cfg.cells[i];
      args.mesh.periodic[i] = cfg.periodic[i];
    }
    args.mesh.nelem = (int)cfg.nelem;
    args.mesh.tab = cfg.tab;
    args.mesh.info = cfg.elem_info;
    args.mesh.mij = cfg.mij;
    if constexpr (NS) launch_viscous_flux<DIM, N>(cfg, u_in, cfg.visc, cfg.grad, s);
    switch (variant_) {
      case 3: launch_node<true>(args, cfg.nelem, s); break;
      case 4: launch_node<false>(args, cfg.nelem, s); break;
      case 5: launch_pipe(args, cfg.nelem, s); break;
      case 6: launch_node2(args, cfg.nelem, s); break;
      default: {
        last_grid_ = (cfg.nelem + elements_per_block() - 1) / elements_per_block();
        launch_line<false>(args, (unsigned)last_grid_, s);
        break;
      }
    }
    if (diag) last_diag_slots_ = last_grid_;
    return cudaGetLastError();
  }

  cudaError_t batch_stage(const EngineConfig& cfg, const MeshView* meshes,
                          const int* tile_mesh, const int* tile_e0, int ntiles,
                          double a, double b, double t, const double* t_dev,
                          cudaStream_t s) override {
    if constexpr (!kBatch) {
      return cudaErrorNotSupported;
    } else {
      StageArgs<N> args = common_args(cfg, a, b, t, t_dev, nullptr);
      args.meshes = meshes;
      args.tile_mesh = tile_mesh;
      args.tile_e0 = tile_e0;
      switch (variant_) {
        case 3:
        case 5:
        case 6: launch_node_batch<true>(args, ntiles, s); break;
        case 4: launch_node_batch<false>(args, ntiles, s); break;
        default: launch_line<true>(args, (unsigned)ntiles, s); break;
      }
      return cudaGetLastError();
    }
  }

  cudaError_t build_mesh_tables(const MeshView& m, int* info, double* mij,
                                cudaStream_t s) const override {
    const int64_t nodes = (int64_t)m.nelem * ipow(N, DIM);
    const unsigned blocks = (unsigned)std::min<int64_t>((nodes + 255) / 256, 4096);
    element_tables_kernel<DIM, N, 12><<<blocks, 256, 0, s>>>(m, info, mij);
    return cudaGetLastError();
  }

  int kernels_per_stage() const override { return NS ? 2 : 1; }
  int64_t last_diag_slots() const override { return last_diag_slots_; }
  int elements_per_block() const override {
    if constexpr (kNode2)
      if (variant_ == 6) return Node2Launch<N>::EPB;
    if (variant_ >= 3) return NL::EPB;
    return use_split() ? LG::EPW : LINE_EPB;
  }
  int threads_per_block() const override {
    if (variant_ >= 3) return NL::NT;
    return use_split() ? SSh::NT : LINE_NT;
  }
  size_t smem_bytes() const override {
    if constexpr (kNode2)
      if (variant_ == 6) return Node2Shape<N, VF>::smem_bytes;
    if (variant_ >= 3) return NSh::smem_bytes;
    return use_split() ? SSh::smem_bytes : LINE_SMEM;
  }
  void set_variant(int v) override {
    variant_ = (v >= 0 && v < num_variants()) ? v : 0;
    load_variant(variant_);
  }
  int variant() const override { return variant_; }
  const char* kernel_name() const override {
    if (kNode2 && variant_ == 6) return "stage_node2_kernel";
    if (kPipe && variant_ == 5) return "stage_pipe_kernel";
    if (variant_ >= 3) return "stage_node_kernel";
    return use_split() ? "stage_split_kernel" : "stage_line_kernel";
  }
  // shapes 5 and 6 exist for single-mesh launches; batched launches run them as 3
  int num_variants() const override { return kNode2 ? 7 : kPipe ? 6 : kNode ? 5 : 3; }

 private:
  int variant_ = 0;
  bool split_ = false;   // shape 0 runs the split form (set_mesh_size)
  unsigned loaded_ = 0;  // launch shapes configured so far (load_variant)
  int device_ = 0;       // device of the creation (set_mesh_size)
  mutable int64_t pipe_blocks_ = 0;
  mutable int64_t last_grid_ = 0;  // blocks of the last single-mesh stage launch
  int64_t last_diag_slots_ = 0;
};

}  // namespace dgsem
