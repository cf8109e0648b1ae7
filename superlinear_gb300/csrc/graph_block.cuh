// The per-atom part of a split pass (FP32 engines), a block for 32 centres: for the energy pass
// (Static or Effect outer), moments a.mom -> the graph program forward -> readout (site energy,
// descriptors) -> the program's reverse -> adjoint moments a.amom; for the Effect gate passes, the
// gate graph forward with the gate-signal projection, or the gate-signal adjoint's projection and
// the gate graph reverse.
//
// What bounds it: issue slots for the program's terms T[target] += c X[a] v[b], and at few centres
// the latency of the steps.  With lanes over a program's terms (run_prog, one centre per warp) a
// 16-byte record serves one term of one centre, and its two node reads hit scattered banks.  Here
// lanes are centres: node values lie [slot][32 centres] in shared memory, every node read is one
// conflict-free row, a 16-byte unit serves two terms of 32 centres (about 9 instructions a term),
// and a block's 16 (or 32) warps share the target lists of a step, longest first, with a barrier per step.
// Only the nodes of this pass take slots, and an adjoint takes its node's slot when the reverse
// never reads the value, which keeps two blocks per SM at L4/K8.  Every list is summed chunk by
// chunk in run_prog's order and the gate-signal adjoints as in the fused pass, so that split and fused
// passes give the same bits: the number of centres chooses between them, and a frame's results
// must not depend on the frames it is evaluated with.
// Effect L4/K8/R2/O3, 110,592 atoms: the outer pass's graph about 1.0 ms one centre a warp, 0.9 ms
// two, 0.2 ms here; 8,000 atoms 78 -> 41 us (one wave, cold program).
#pragma once
#include "efs_kernels.cuh"

namespace sus2g {

// Warps of a block: 16, or 32 where shared memory admits one block per SM.
__host__ __device__ inline int graph_block_warps(size_t bytes) { return bytes > 113 * 1024 ? 2 * kGraphWarps : kGraphWarps; }

// Shared memory of a block: the slots, then hbar [F][32] (gate reverse) or the readout's scalars
// [S][33] (energy pass).
__host__ __device__ inline size_t graph_block_bytes(int nslots, int F, int S) {
  const int more = F * kGraphAtoms > S * (kGraphAtoms + 1) ? F * kGraphAtoms : S * (kGraphAtoms + 1);
  return sizeof(float) * (static_cast<size_t>(nslots) * kGraphAtoms + more);
}

// A warp's units [p0, p1), four at a time with the next four loading.  A unit that closes a step
// carries the block's barrier: every warp's stream has one per step.
__device__ __forceinline__ void run_block_steps(const int4* units, int p0, int p1, float* s, int lane) {
  constexpr int D = 4;
  constexpr unsigned kSlotMask = 0xfffu << 7;
  const unsigned lane4 = 4u * lane;
  const char* base = reinterpret_cast<const char*>(s);
  auto at = [&](unsigned off) { return *reinterpret_cast<const float*>(base + off); };
  int4 cur[D], nxt[D];
#pragma unroll
  for (int u = 0; u < D; ++u) nxt[u] = __ldg(units + p0 + u);  // (streams are whole fours)
  float sum = 0.f, acc = 0.f;
  for (int p = p0; p < p1; p += D) {
#pragma unroll
    for (int u = 0; u < D; ++u) cur[u] = nxt[u];
    if (p + D < p1)
#pragma unroll
      for (int u = 0; u < D; ++u) nxt[u] = __ldg(units + p + D + u);
#pragma unroll
    for (int u = 0; u < D; ++u) {
      const unsigned x = static_cast<unsigned>(cur[u].x), z = static_cast<unsigned>(cur[u].z);
      const float xa = at((x & kSlotMask) | lane4), va = at(((x >> 13) & kSlotMask) | lane4);
      const float xb = at((z & kSlotMask) | lane4), vb = at(((z >> 13) & kSlotMask) | lane4);
      acc = fmaf(__int_as_float(cur[u].y) * xa, va, acc);
      acc = fmaf(__int_as_float(cur[u].w) * xb, vb, acc);
      if (z & (kUnitChunkEnd | kUnitListEnd | kUnitStepEnd)) {
        if (z & kUnitChunkEnd) {
          sum += acc;
          acc = 0.f;
        }
        if (z & kUnitListEnd) {
          float* t = reinterpret_cast<float*>(reinterpret_cast<char*>(s) + ((((x & 0x7fu) << 7) | ((z & 0x1fu) << 14)) | lane4));
          *t += sum;
          sum = 0.f;
        }
        if (z & kUnitStepEnd) asm volatile("bar.sync 0;" ::: "memory");
      }
    }
  }
}

// Rows [32][n] of a per-centre array (row stride ld) into or out of slots: a lane moves its centre's
// row in 16-byte units (the rows' lines stay in L1 between a warp's accesses).
template <typename Put>
__device__ __forceinline__ void centre_rows(const float* rows, int ld, int n, int na, int warp, int warps, int lane, Put&& put) {
  const float* row = rows + static_cast<size_t>(min(lane, na - 1)) * ld;
  if (n % 4 == 0 && ld % 4 == 0) {
    for (int t = 4 * warp; t < n; t += 4 * warps) {
      const float4 w = *reinterpret_cast<const float4*>(row + t);
      put(t, w.x); put(t + 1, w.y); put(t + 2, w.z); put(t + 3, w.w);
    }
  } else {
    for (int t = warp; t < n; t += warps) put(t, row[t]);
  }
}

// GM: 0 the energy pass (Static or Effect outer tables), 1 the gate forward pass (the values that
// the gate reverse reads to a.gkeep, gate signals to a.hsig), 2 the gate reverse pass (per-atom
// gate-signal adjoints in a.hbar, or a.hbar_atom for caller edges).
template <int GM>
__global__ void __launch_bounds__(2 * kGraphWarps * kWarp, 1) graph_block_kernel(PassArgs<float> a) {
  constexpr int A = kGraphAtoms;
  const DevModel<float>& dm = a.dm;
  const BlockProg& g = GM == 0 ? dm.outer.block : dm.gate.block;
  const int KH = dm.K * dm.H, C = dm.C, F = dm.F, Q = dm.Q;
  const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = warp_lane();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s = reinterpret_cast<float*>(smem_raw);  // [nslots][32]
  float* more = s + g.nslots * A;                 // hbar [F][32], or the scalars [S][33]
  pdl_launch_dependents();
  const int p0 = g.begin[4 * warp], p1 = g.begin[4 * warp + 1], p2 = g.begin[4 * warp + 3];
  pdl_wait();
  for (int blk = blockIdx.x; blk * A < a.natoms; blk += gridDim.x) {
    const int n0 = blk * A, na = min(A, a.natoms - n0);
    const size_t n = static_cast<size_t>(n0 + min(lane, na - 1));  // the lane's centre
    __syncthreads();  // the slots of the previous centres are free
    if (warp == 0) s[g.one * A + lane] = 1.f;
    if constexpr (GM == 2) {
      if (a.hbar_atom) {
        for (int mu = warp; mu < F; mu += warps) more[mu * A + lane] = static_cast<float>(a.hbar_atom[n * F + mu]);
      } else {
        centre_rows(a.hbar + static_cast<size_t>(n0) * F, F, F, na, warp, warps, lane,
                    [&](int mu, float x) { more[mu * A + lane] = x; });
      }
      for (int q = warp; q < g.nkeep; q += warps)
        s[g.keep[q] * A + lane] = a.gkeep[(static_cast<size_t>(blk) * g.nkeep + q) * A + lane];
      for (int q = warp; q < g.nzero_adj; q += warps) s[g.zero_adj[q] * A + lane] = 0.f;
      __syncthreads();
      for (int q = warp; q < Q; q += warps) {
        const float* w = dm.gate_wmat_t + static_cast<size_t>(q) * F;
        float sum = 0.f;
#pragma unroll 8
        for (int mu = 0; mu < F; ++mu) sum = fmaf(more[mu * A + lane], __ldg(w + mu), sum);
        s[g.seed_adj[q] * A + lane] = sum;
      }
      __syncthreads();
    } else {
      centre_rows(a.mom + static_cast<size_t>(n0) * KH, KH, KH, na, warp, warps, lane, [&](int t, float x) {
        const int slot = g.basic_slot[t];
        if (slot >= 0) s[slot * A + lane] = x;
      });
      for (int q = warp; q < g.nzero_v; q += warps) s[g.zero_v[q] * A + lane] = 0.f;
      __syncthreads();
      run_block_steps(g.units, p0, p1, s, lane);
    }
    if constexpr (GM == 1) {
      for (int q = warp; q < g.nkeep; q += warps)
        a.gkeep[(static_cast<size_t>(blk) * g.nkeep + q) * A + lane] = s[g.keep[q] * A + lane];
      // four signals at a time: each gate scalar is read once for them
      for (int mu = 4 * warp; mu < F; mu += 4 * warps) {
        float h[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int q = 0; q < Q; ++q) {
          const float x = s[g.seed_v[q] * A + lane];
          const float* w = dm.gate_wmat_t + static_cast<size_t>(q) * F + mu;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (mu + i < F) h[i] = fmaf(__ldg(w + i), x, h[i]);
        }
        if (lane < na)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (mu + i < F) a.hsig[n * F + mu + i] = h[i];
      }
      continue;
    }
    if constexpr (GM == 0) {
      // adjoint seeds and the scalars, lanes over centres; then the readout as readout_seeds sums
      // it, a warp per centre and lanes over the scalars (33 floats a row: conflict-free both ways)
      const int ti = C == 1 ? 0 : species_of(a.types, static_cast<int>(n), C);
      const float coef_r = static_cast<float>(dm.species_readout ? 1.0 : dm.species[ti]);
      const float* lin = dm.linear + (dm.species_readout ? ti * dm.S : 0);
      for (int q = warp; q < dm.S; q += warps) {
        more[q * (A + 1) + lane] = s[g.seed_v[q] * A + lane];
        s[g.seed_adj[q] * A + lane] = coef_r * lin[q];
      }
      for (int q = warp; q < g.nzero_adj; q += warps) s[g.zero_adj[q] * A + lane] = 0.f;
      __syncthreads();
      for (int c = warp; c < na; c += warps) {
        const int tc = __shfl_sync(0xffffffffu, ti, c);
        const int off = dm.species_readout ? tc * dm.S : 0;
        float ehi = 0.f, elo = 0.f;
        for (int q = lane; q < dm.S; q += kWarp) {
          const float vv = more[q * (A + 1) + c];
          csum_add_prod(ehi, elo, dm.linear[off + q], vv);
          if (a.desc) a.desc[static_cast<size_t>(n0 + c) * dm.S + q] = static_cast<double>(vv);
        }
        const double es = warp_csum(ehi, elo);
        if (lane == 0)
          a.site_energy[n0 + c] = dm.species[tc] + dm.shift[tc] + (dm.species_readout ? 1.0 : dm.species[tc]) * es;
      }
    }
    run_block_steps(g.units, p1, p2, s, lane);
    if (lane < na) {
      float* row = a.amom + n * KH;
      auto get = [&](int t) {
        const int slot = g.basic_adj[t];
        return slot >= 0 ? s[slot * A + lane] : 0.f;
      };
      if (KH % 4 == 0) {
        for (int t = 4 * warp; t < KH; t += 4 * warps)
          *reinterpret_cast<float4*>(row + t) = make_float4(get(t), get(t + 1), get(t + 2), get(t + 3));
      } else {
        for (int t = warp; t < KH; t += warps) row[t] = get(t);
      }
    }
  }
}

// The gate-signal adjoint of every centre: the F contributions of its edges (stored at the reverse
// edges by the outer pass) summed per column, warp per centre, in the fused gate reverse pass's order
// (row_group_sums).  Bound by the read of the [E][F] contributions.
static __global__ void __launch_bounds__(256) hbar_sum_kernel(PassArgs<float> a) {
  const int F = a.dm.F, lane = warp_lane();
  const int atom = static_cast<int>((static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) / kWarp);
  pdl_launch_dependents();
  pdl_wait();
  if (atom >= a.natoms) return;
  const int e0 = a.row[atom], n = a.row_end[atom] - e0;
  const float* rows = a.hcontrib + static_cast<size_t>(e0) * F;
  float* out = a.hbar + static_cast<size_t>(atom) * F;
  if (row_groups_ok(F)) {
    row_group_sums(rows, F, n, lane, [&](int c, float4 t) { reinterpret_cast<float4*>(out)[c] = t; });
  } else {
    for (int mu = lane; mu < F; mu += kWarp) out[mu] = column_sum<float>(rows + mu, F, n);
  }
}

}  // namespace sus2g
