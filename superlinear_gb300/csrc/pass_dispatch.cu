// Run-time selection of the per-L pass and gradient units (instantiated in pass_fp*_l*.cu and
// grad_fp*_l*.cu); this unit sees only their declarations.
#include <algorithm>
#include <stdexcept>
#include <string>

#include "grad_edge.cuh"
#include "grad_graph.cuh"
#include "graph_block.cuh"
#include "pass_launch.h"

namespace sus2g {

template <typename Real>
int launch_atom_pass(int L, int mode, const PassArgs<Real>& a, int sm_count, cudaStream_t s, int blocks, bool pdl) {
  if (a.dm.K > kMaxK) throw std::runtime_error("sh_k_max above " + std::to_string(kMaxK) + " is not supported");
  switch (L) {
    case 0: return launch_atom_pass_l<Real, 0>(mode, a, sm_count, s, blocks, pdl);
    case 1: return launch_atom_pass_l<Real, 1>(mode, a, sm_count, s, blocks, pdl);
    case 2: return launch_atom_pass_l<Real, 2>(mode, a, sm_count, s, blocks, pdl);
    case 3: return launch_atom_pass_l<Real, 3>(mode, a, sm_count, s, blocks, pdl);
    case 4: return launch_atom_pass_l<Real, 4>(mode, a, sm_count, s, blocks, pdl);
    case 5: return launch_atom_pass_l<Real, 5>(mode, a, sm_count, s, blocks, pdl);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}

template <typename Real>
GradLaunch grad_pass_config(int L, int mode, const DevModel<Real>& dm, int natoms, int sm_count, int part) {
  switch (L) {
    case 0: return grad_pass_config_l<Real, 0>(mode, dm, natoms, sm_count, part);
    case 1: return grad_pass_config_l<Real, 1>(mode, dm, natoms, sm_count, part);
    case 2: return grad_pass_config_l<Real, 2>(mode, dm, natoms, sm_count, part);
    case 3: return grad_pass_config_l<Real, 3>(mode, dm, natoms, sm_count, part);
    case 4: return grad_pass_config_l<Real, 4>(mode, dm, natoms, sm_count, part);
    case 5: return grad_pass_config_l<Real, 5>(mode, dm, natoms, sm_count, part);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}

template <typename Real>
int launch_grad_pass(int L, int mode, const GradArgs<Real>& a, const GradLaunch& cfg, cudaStream_t s) {
  switch (L) {
    case 0: return launch_grad_pass_l<Real, 0>(mode, a, cfg, s);
    case 1: return launch_grad_pass_l<Real, 1>(mode, a, cfg, s);
    case 2: return launch_grad_pass_l<Real, 2>(mode, a, cfg, s);
    case 3: return launch_grad_pass_l<Real, 3>(mode, a, cfg, s);
    case 4: return launch_grad_pass_l<Real, 4>(mode, a, cfg, s);
    case 5: return launch_grad_pass_l<Real, 5>(mode, a, cfg, s);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}

namespace {
template <int GM>
int launch_graph(const PassArgs<float>& a, int sm_count, cudaStream_t s) {
  const BlockProg& g = GM == 0 ? a.dm.outer.block : a.dm.gate.block;
  auto kern = graph_block_kernel<GM>;
  const size_t smem = graph_block_bytes(g.nslots, a.dm.F, a.dm.S);
  static LargestPerDevice allowed;
  cudaError_t err = allow_shared_memory(kern, smem, allowed);
  if (err != cudaSuccess) throw std::runtime_error(std::string("graph kernel shared memory: ") + cudaGetErrorString(err));
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, g.warps * kWarp, smem);
  if (per_sm < 1) throw std::runtime_error("graph kernel does not fit on an SM");
  const int need = (a.natoms + kGraphAtoms - 1) / kGraphAtoms;
  kern<<<std::max(1, std::min(need, per_sm * sm_count)), g.warps * kWarp, smem, s>>>(a);
  err = cudaGetLastError();
  if (err != cudaSuccess) throw std::runtime_error(std::string("graph kernel launch: ") + cudaGetErrorString(err));
  return 1;
}
}  // namespace

int graph_program_warps(int nslots, int F, int S) { return graph_block_warps(graph_block_bytes(nslots, F, S)); }

bool graph_block_fits(const BlockProg& g, int F, int S) {
  return g.nslots > 0 && graph_block_bytes(g.nslots, F, S) <= 227 * 1024;
}

int launch_atom_graph(const PassArgs<float>& a, int sm_count, cudaStream_t s, int gm) {
  if (a.natoms == 0) return 0;
  switch (gm) {
    case 0: return launch_graph<0>(a, sm_count, s);
    case 1: return launch_graph<1>(a, sm_count, s);
    case 2: return launch_graph<2>(a, sm_count, s);
  }
  throw std::runtime_error("graph kernel: unknown pass");
}

int launch_hbar_sum(const PassArgs<float>& a, cudaStream_t s) {
  if (a.natoms == 0) return 0;
  const unsigned blocks = static_cast<unsigned>((static_cast<long long>(a.natoms) * kWarp + 255) / 256);
  hbar_sum_kernel<<<blocks, 256, 0, s>>>(a);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) throw std::runtime_error(std::string("gate-signal adjoint launch: ") + cudaGetErrorString(err));
  return 1;
}

template <typename Real>
GradLaunch grad_edge_config(int L, int mode, const DevModel<Real>& dm, int natoms, int sm_count) {
  switch (L) {
    case 0: return grad_edge_config_l<Real, 0>(mode, dm, natoms, sm_count);
    case 1: return grad_edge_config_l<Real, 1>(mode, dm, natoms, sm_count);
    case 2: return grad_edge_config_l<Real, 2>(mode, dm, natoms, sm_count);
    case 3: return grad_edge_config_l<Real, 3>(mode, dm, natoms, sm_count);
    case 4: return grad_edge_config_l<Real, 4>(mode, dm, natoms, sm_count);
    case 5: return grad_edge_config_l<Real, 5>(mode, dm, natoms, sm_count);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}
template <typename Real>
int launch_grad_edge(int L, int mode, const GradArgs<Real>& a, const GradLaunch& cfg, cudaStream_t s) {
  switch (L) {
    case 0: return launch_grad_edge_l<Real, 0>(mode, a, cfg, s);
    case 1: return launch_grad_edge_l<Real, 1>(mode, a, cfg, s);
    case 2: return launch_grad_edge_l<Real, 2>(mode, a, cfg, s);
    case 3: return launch_grad_edge_l<Real, 3>(mode, a, cfg, s);
    case 4: return launch_grad_edge_l<Real, 4>(mode, a, cfg, s);
    case 5: return launch_grad_edge_l<Real, 5>(mode, a, cfg, s);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}
GradLaunch grad_moment_config(int L, int mode, const DevModel<float>& dm, int natoms, int sm_count) {
  switch (L) {
    case 0: return grad_moment_config_l<0>(mode, dm, natoms, sm_count);
    case 1: return grad_moment_config_l<1>(mode, dm, natoms, sm_count);
    case 2: return grad_moment_config_l<2>(mode, dm, natoms, sm_count);
    case 3: return grad_moment_config_l<3>(mode, dm, natoms, sm_count);
    case 4: return grad_moment_config_l<4>(mode, dm, natoms, sm_count);
    case 5: return grad_moment_config_l<5>(mode, dm, natoms, sm_count);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}
int launch_grad_moment(int L, int mode, const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t s) {
  switch (L) {
    case 0: return launch_grad_moment_l<0>(mode, a, cfg, s);
    case 1: return launch_grad_moment_l<1>(mode, a, cfg, s);
    case 2: return launch_grad_moment_l<2>(mode, a, cfg, s);
    case 3: return launch_grad_moment_l<3>(mode, a, cfg, s);
    case 4: return launch_grad_moment_l<4>(mode, a, cfg, s);
    case 5: return launch_grad_moment_l<5>(mode, a, cfg, s);
  }
  throw std::runtime_error("sh_l_max above 5 is not supported");
}

namespace {
void (*graph_gradient_kernel(int mode))(GradArgs<float>) {
  return mode == kGradOuter ? grad_graph_kernel<kGradOuter>
                            : mode == kGradGateForward ? grad_graph_kernel<kGradGateForward> : grad_graph_kernel<kGradGateReverse>;
}
void check_gradient(cudaError_t err, const char* what) {
  if (err != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(err));
}
}  // namespace

bool grad_graph_fits(const DevModel<float>& dm, bool gated) {
  auto fits = [&](const BlockProg& g) { return g.nslots > 0 && dual_block_bytes(g.nslots, dm.F, dm.S) <= 227 * 1024; };
  return fits(dm.outer.dual) && (!gated || fits(dm.gate.dual));
}
GradLaunch grad_graph_config(int mode, const DevModel<float>& dm, int natoms, int sm_count) {
  auto kern = graph_gradient_kernel(mode);
  GradLaunch cfg;
  const BlockProg& g = (mode == kGradOuter ? dm.outer : dm.gate).dual;
  cfg.warps = g.warps;
  cfg.block = g.warps * kWarp;
  cfg.smem = dual_block_bytes(g.nslots, dm.F, dm.S);
  static LargestPerDevice allowed[3];
  check_gradient(allow_shared_memory(kern, cfg.smem, allowed[mode]), "gradient graph shared memory");
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, cfg.block, cfg.smem);
  if (per_sm < 1) throw std::runtime_error("gradient graph kernel does not fit on an SM");
  cfg.grid = std::max(1, std::min((natoms + kDualAtoms - 1) / kDualAtoms, per_sm * sm_count));
  return cfg;
}
int launch_grad_graph(int mode, const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t s) {
  if (a.natoms == 0) return 0;
  graph_gradient_kernel(mode)<<<cfg.grid, cfg.block, cfg.smem, s>>>(a);
  check_gradient(cudaGetLastError(), "gradient graph launch");
  return 1;
}
int launch_lhm_sum(const GradArgs<float>& a, int Lp, cudaStream_t s) {
  if (a.natoms == 0) return 0;
  lhm_sum_kernel<float><<<static_cast<unsigned>((static_cast<long long>(a.natoms) * kWarp + 255) / 256), 256, 0, s>>>(a, Lp);
  check_gradient(cudaGetLastError(), "gate-signal adjoint launch");
  return 1;
}
GradLaunch grad_gate_weight_config(const DevModel<float>& dm, int natoms, int sm_count) {
  const int tile = gate_weight_tile(dm.F, dm.Q);
  auto kern = tile == 4 ? grad_gate_weight_kernel<4> : grad_gate_weight_kernel<2>;
  GradLaunch cfg;
  cfg.warps = kGwThreads32 / kWarp;
  cfg.block = kGwThreads32;
  cfg.smem = gate_weight_bytes(dm.F, dm.Q);
  if (cfg.smem > 227 * 1024) throw std::runtime_error("gate weight gradient: radial functions + gate scalars exceed the shared-memory staging");
  static LargestPerDevice allowed[2];
  check_gradient(allow_shared_memory(kern, cfg.smem, allowed[tile == 4]), "gate weight shared memory");
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, cfg.block, cfg.smem);
  cfg.grid = std::max(1, std::min((natoms + kDualAtoms - 1) / kDualAtoms, std::max(1, per_sm) * sm_count));
  return cfg;
}
int launch_grad_gate_weight(const GradArgs<float>& a, const GradLaunch& cfg, cudaStream_t s) {
  if (a.natoms == 0) return 0;
  auto kern = gate_weight_tile(a.dm.F, a.dm.Q) == 4 ? grad_gate_weight_kernel<4> : grad_gate_weight_kernel<2>;
  kern<<<cfg.grid, cfg.block, cfg.smem, s>>>(a);
  check_gradient(cudaGetLastError(), "gate weight launch");
  return 1;
}

template int launch_atom_pass<float>(int, int, const PassArgs<float>&, int, cudaStream_t, int, bool);
template int launch_atom_pass<double>(int, int, const PassArgs<double>&, int, cudaStream_t, int, bool);
template GradLaunch grad_edge_config<float>(int, int, const DevModel<float>&, int, int);
template GradLaunch grad_edge_config<double>(int, int, const DevModel<double>&, int, int);
template int launch_grad_edge<float>(int, int, const GradArgs<float>&, const GradLaunch&, cudaStream_t);
template int launch_grad_edge<double>(int, int, const GradArgs<double>&, const GradLaunch&, cudaStream_t);
template GradLaunch grad_pass_config<float>(int, int, const DevModel<float>&, int, int, int);
template GradLaunch grad_pass_config<double>(int, int, const DevModel<double>&, int, int, int);
template int launch_grad_pass<float>(int, int, const GradArgs<float>&, const GradLaunch&, cudaStream_t);
template int launch_grad_pass<double>(int, int, const GradArgs<double>&, const GradLaunch&, cudaStream_t);

}  // namespace sus2g
