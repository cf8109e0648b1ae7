// Launch entry points of the per-atom passes, one translation unit per precision.
#pragma once
#include <cuda_runtime.h>

#include "efs_kernels.cuh"
#include "grad_kernels.cuh"

namespace sus2g {

struct GradLaunch {
  int grid = 0, block = 0, warps = 0;
  int acc_cols = 0;  // lane-private accumulator columns (0: shuffle-tree reductions)
  int part = 0;      // GradPart: the whole pass, or its per-atom or per-edge part
  size_t smem = 0;
};

// Launch shape of grad_pass_kernel<L, Real, mode> or of one part of it (GradPart; grid sized from
// occupancy x SM count).
template <typename Real>
GradLaunch grad_pass_config(int L, int mode, const DevModel<Real>& dm, int natoms, int sm_count, int part = 0);
// Launches it with that shape (a.slots must hold cfg.grid * cfg.warps slices).
template <typename Real>
int launch_grad_pass(int L, int mode, const GradArgs<Real>& a, const GradLaunch& cfg, cudaStream_t stream);

// The kernels of the split gradient (grad_edge.cuh, grad_graph.cuh).  Launch shapes: GradLaunch with
// grid 0 where the kernel does not take the model; the edge, graph and gate-weight kernels write
// one slice per block.
constexpr int kDualAtoms = 16;  // centres per block of the graph kernel: half a row of 32
template <typename Real>
GradLaunch grad_edge_config(int L, int mode, const DevModel<Real>& dm, int natoms, int sm_count);
template <typename Real>
int launch_grad_edge(int L, int mode, const GradArgs<Real>& a, const GradLaunch& cfg, cudaStream_t stream);
GradLaunch grad_moment_config(int L, int mode, const DevModel<float>& dm, int natoms, int sm_count);
int launch_grad_moment(int L, int mode, const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t stream);
bool grad_graph_fits(const DevModel<float>& dm, bool gated);
GradLaunch grad_graph_config(int mode, const DevModel<float>& dm, int natoms, int sm_count);
int launch_grad_graph(int mode, const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t stream);
int launch_lhm_sum(const GradArgs<float>& a, int Lp, cudaStream_t stream);
GradLaunch grad_gate_weight_config(const DevModel<float>& dm, int natoms, int sm_count);
int launch_grad_gate_weight(const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t stream);
template <typename Real, int L>
GradLaunch grad_edge_config_l(int mode, const DevModel<Real>& dm, int natoms, int sm_count);
template <typename Real, int L>
int launch_grad_edge_l(int mode, const GradArgs<Real>& a, const GradLaunch& cfg, cudaStream_t stream);
template <int L>
GradLaunch grad_moment_config_l(int mode, const DevModel<float>& dm, int natoms, int sm_count);
template <int L>
int launch_grad_moment_l(int mode, const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t stream);

// Warps per block (`most` or 2) of a launch whose n warps, one centre each, are resident at once: what
// leaves the fullest SM with fewer warps, an odd block counted as the next even one (it leaves one of
// the SM's four schedulers a warp short).  884 centres in blocks of 4 put 8 warps on some of 152 SMs
// and 4 on the others, in blocks of 2 at most 6: FP64 per-edge gradient 509 -> 481 and 465 -> 440 us, gate
// forward 229 -> 158 us (blocks of 3: 561, 524 and 193), per-atom gradient parts 317 -> 269 and 300 -> 252 us;
// FP32 passes, bound by latency there, gain 0 to 4%.
inline int spread_warps(int n, int most, int sm_count) {
  auto load = [&](int w) { return ((n + w - 1) / w + sm_count - 1) / sm_count * ((w + 1) / 2 * 2); };
  return most > 2 && load(2) < load(most) ? 2 : most;
}

// Launches atom_pass_kernel<L, Real, mode, Kahan = (Real is float)> sized as a multiple of the SM
// count, with the register budget of `blocks` resident blocks per SM (3 or 4; 0 = the default),
// as a programmatic dependent launch when pdl is set (the kernel stages its model tables while
// the previous kernel of the stream drains).  Returns the warps per block of the launch (0: no
// centres, nothing launched) or throws on a configuration error.
template <typename Real>
int launch_atom_pass(int L, int mode, const PassArgs<Real>& args, int sm_count, cudaStream_t stream,
                     int blocks = 0, bool pdl = false);

// The per-atom graph kernel of a split pass (graph_block_kernel<gm>: 0 energy pass, 1 gate forward,
// 2 gate reverse): returns 1 or throws.
int launch_atom_graph(const PassArgs<float>& args, int sm_count, cudaStream_t stream, int gm);
// Warps per block of that kernel (and of the gradient's) for a program of so many slots.
int graph_program_warps(int nslots, int F, int S);
// Whether a pass's nodes fit that kernel's shared memory (the pass runs fused otherwise).
bool graph_block_fits(const BlockProg& g, int F, int S);
// The per-atom gate-signal adjoints a.hbar from the per-edge contributions (hbar_sum_kernel).
int launch_hbar_sum(const PassArgs<float>& args, cudaStream_t stream);

// Per-L entry points, explicitly instantiated in the pass_fp*_l* / grad_fp*_l* units.
template <typename Real, int L>
int launch_atom_pass_l(int mode, const PassArgs<Real>& a, int sm_count, cudaStream_t s, int blocks, bool pdl);
template <typename Real, int L>
GradLaunch grad_pass_config_l(int mode, const DevModel<Real>& dm, int natoms, int sm_count, int part);
template <typename Real, int L>
int launch_grad_pass_l(int mode, const GradArgs<Real>& a, const GradLaunch& cfg, cudaStream_t s);

}  // namespace sus2g
