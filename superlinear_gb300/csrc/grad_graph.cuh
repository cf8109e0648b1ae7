// The per-atom part of the split parameter gradient (FP32 engines): the pass's graph program on
// values and tangents and its reverse on their adjoints, a block for 16 centres -- lanes 0-15 of a
// node's row hold the centres' values (adjoints lambda), lanes 16-31 their tangents (adjoints mu) --
// in the layout and with the program units of graph_block.cuh.  A term reads two rows and the
// partner halves by shuffle:
//   forward   v[t] += c v_x v_y,  vd[t] += c (v_x vd_y + vd_x v_y)
//   reverse   lam[t] += c (lam_x v_y + mu_x vd_y),  mu[t] += c mu_x v_y
// Bound by issue slots; the one-centre-per-warp program walk it replaces spent most of its time
// waiting for program records (long scoreboard 3.3-9.4 per issue) at 6 (L5) to 16 warps per SM.
#pragma once
#include "grad_kernels.cuh"
#include "graph_block.cuh"
#include "pass_launch.h"

namespace sus2g {

template <bool REV>
__device__ __forceinline__ void run_dual_steps(const int4* units, int p0, int p1, float* s, int lane) {
  constexpr int D = 4;
  constexpr unsigned kSlotMask = 0xfffu << 7;
  const unsigned lane4 = 4u * lane;
  const bool val = lane < kDualAtoms;
  const char* base = reinterpret_cast<const char*>(s);
  auto at = [&](unsigned off) { return *reinterpret_cast<const float*>(base + off); };
  float sum = 0.f, acc = 0.f;
  auto term = [&](unsigned w, int cbits) {
    const float x = at((w & kSlotMask) | lane4), y = at(((w >> 13) & kSlotMask) | lane4);
    const float sx = __shfl_xor_sync(0xffffffffu, x, kDualAtoms), sy = __shfl_xor_sync(0xffffffffu, y, kDualAtoms);
    const float b1 = val ? y : sy, b2 = REV ? (val ? sy : 0.f) : (val ? 0.f : y);
    acc = fmaf(__int_as_float(cbits), fmaf(x, b1, sx * b2), acc);
  };
  int4 nxt[D];
#pragma unroll
  for (int u = 0; u < D; ++u) nxt[u] = __ldg(units + p0 + u);
  for (int p = p0; p < p1; p += D) {
    int4 cur[D];
#pragma unroll
    for (int u = 0; u < D; ++u) cur[u] = nxt[u];
    if (p + D < p1)
#pragma unroll
      for (int u = 0; u < D; ++u) nxt[u] = __ldg(units + p + D + u);
#pragma unroll
    for (int u = 0; u < D; ++u) {
      const unsigned x = static_cast<unsigned>(cur[u].x), z = static_cast<unsigned>(cur[u].z);
      term(x, cur[u].y);
      term(z, cur[u].w);
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

// Shared memory: the rows, then hb [F][32] (gate reverse) or the readout's scalars [S][33], then the
// centres' energy weights and species.
__host__ __device__ inline size_t dual_block_bytes(int nslots, int F, int S) {
  return graph_block_bytes(nslots, F, S) + kDualAtoms * (sizeof(double) * 2 + sizeof(int)) + 8;
}

template <int MODE>
__global__ void __launch_bounds__(2 * kGraphWarps * kWarp, 1) grad_graph_kernel(GradArgs<float> a) {
  constexpr int A = kDualAtoms, W = kWarp;
  const DevModel<float>& dm = a.dm;
  const PassTables<float>& pt = MODE == kGradOuter ? dm.outer : dm.gate;
  const PassGradLayout& gl = MODE == kGradOuter ? dm.grad.outer : dm.grad.gate;
  const BlockProg& g = pt.dual;
  const int KH = dm.K * dm.H, C = dm.C, F = dm.F, Q = dm.Q, NS = dm.S;
  const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = warp_lane(), half = lane / A, c0 = lane % A;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s = reinterpret_cast<float*>(smem_raw);
  float* more = s + g.nslots * W;
  double* s_ew = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(smem_raw) + graph_block_bytes(g.nslots, F, NS) + 7) & ~uintptr_t(7));
  double* s_sp = s_ew + A;
  int* s_type = reinterpret_cast<int*>(s_sp + A);
  const int* begin = g.begin + 4 * warp;
  const int p0 = begin[0], p1 = begin[1], p2 = begin[2], p3 = begin[3];
  double* slot = a.slots + static_cast<size_t>(blockIdx.x) * dm.grad.nparams;
  for (int blk = blockIdx.x; blk * A < a.natoms; blk += gridDim.x) {
    const int n0 = blk * A, na = min(A, a.natoms - n0);
    const bool on = c0 < na;
    const size_t n = static_cast<size_t>(n0 + min(c0, na - 1));  // the lane's centre
    __syncthreads();
    if (warp == 0) s[g.one * W + lane] = half ? 0.f : 1.f;
    if constexpr (MODE == kGradGateReverse) {
      for (int mu = warp; mu < F; mu += warps)
        more[mu * W + lane] = static_cast<float>(a.lh_atom[n * 2 * F + half * F + mu]);
      for (int q = warp; q < g.nkeep; q += warps)
        s[g.keep[q] * W + lane] = a.gkeep[(static_cast<size_t>(blk) * g.nkeep + q) * W + lane];
      for (int q = warp; q < g.nzero_adj; q += warps) s[g.zero_adj[q] * W + lane] = 0.f;
      __syncthreads();
      for (int q = warp; q < Q; q += warps) {
        const float* w = dm.gate_wmat_t + static_cast<size_t>(q) * F;
        float sum = 0.f;
#pragma unroll 8
        for (int mu = 0; mu < F; ++mu) sum = fmaf(more[mu * W + lane], __ldg(w + mu), sum);
        s[g.seed_adj[q] * W + lane] = sum;
      }
      __syncthreads();
    } else {
      const float* row = a.mom + (n * 2 + half) * KH;
      auto put = [&](int t, float x) {
        const int to = g.basic_slot[t];
        if (to >= 0) s[to * W + lane] = x;
      };
      if (KH % 4 == 0) {
        for (int t = 4 * warp; t < KH; t += 4 * warps) {
          const float4 w = *reinterpret_cast<const float4*>(row + t);
          put(t, w.x); put(t + 1, w.y); put(t + 2, w.z); put(t + 3, w.w);
        }
      } else {
        for (int t = warp; t < KH; t += warps) put(t, row[t]);
      }
      for (int q = warp; q < g.nzero_v; q += warps) s[g.zero_v[q] * W + lane] = 0.f;
      if (MODE == kGradOuter && threadIdx.x < A) {
        s_type[threadIdx.x] = C == 1 ? 0 : species_of(a.types, static_cast<int>(n), C);
        s_ew[threadIdx.x] = a.ew[n];
      }
      __syncthreads();
      run_dual_steps<false>(g.units, p0, p1, s, lane);
    }
    if constexpr (MODE == kGradGateForward) {
      for (int q = warp; q < g.nkeep; q += warps)
        a.gkeep[(static_cast<size_t>(blk) * g.nkeep + q) * W + lane] = s[g.keep[q] * W + lane];
      // the gate scalars and their tangents, for the projection weights' gradient
      for (int q = warp; q < Q; q += warps)
        a.gscal[(static_cast<size_t>(blk) * Q + q) * W + lane] = on ? s[g.seed_v[q] * W + lane] : 0.f;
      float* out = half ? a.hsigd : a.hsig;
      for (int mu = 4 * warp; mu < F; mu += 4 * warps) {
        float h[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int q = 0; q < Q; ++q) {
          const float x = s[g.seed_v[q] * W + lane];
          const float* w = dm.gate_wmat_t + static_cast<size_t>(q) * F + mu;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (mu + i < F) h[i] = fmaf(__ldg(w + i), x, h[i]);
        }
        if (on)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (mu + i < F) out[n * F + mu + i] = h[i];
      }
      continue;
    }
    if constexpr (MODE == kGradOuter) {
      // seeds, the scalars copied to padded rows, then the readout's gradient in FP64
      const int ti = s_type[c0];
      const double coef = dm.species_readout ? 1.0 : dm.species[ti], ew = s_ew[c0];
      const double seed_d = half ? coef : ew * coef;
      const float* lin = dm.linear + (dm.species_readout ? ti * NS : 0);
      for (int q = warp; q < NS; q += warps) {
        more[q * (W + 1) + lane] = s[g.seed_v[q] * W + lane];
        s[g.seed_adj[q] * W + lane] = static_cast<float>(seed_d * static_cast<double>(lin[q]));
      }
      for (int q = warp; q < g.nzero_adj; q += warps) s[g.zero_adj[q] * W + lane] = 0.f;
      __syncthreads();
      // a warp per centre: sum of the weighted scalars (shared readout only)
      {
        double sp = 0.0;
        if (!dm.species_readout && warp < na)
          for (int q = lane; q < NS; q += kWarp)
            sp += static_cast<double>(dm.linear[q]) *
                  (s_ew[warp] * static_cast<double>(more[q * (W + 1) + warp]) + static_cast<double>(more[q * (W + 1) + A + warp]));
        sp = warp_sum(sp);
        if (lane == 0 && warp < A) s_sp[warp] = sp;
      }
      __syncthreads();
      for (int q = threadIdx.x; q < NS; q += blockDim.x) {
        const float* m = more + q * (W + 1);
        for (int t = 0; t < C; ++t) {
          const double ct = dm.species_readout ? 1.0 : dm.species[t];
          double sum = 0.0;
          bool any = false;
          for (int c = 0; c < na; ++c)
            if (s_type[c] == t) {
              sum += ct * (s_ew[c] * static_cast<double>(m[c]) + static_cast<double>(m[A + c]));
              any = true;
            }
          if (any) slot[dm.grad.linear_off + (dm.species_readout ? t * NS : 0) + q] += sum;
        }
      }
      const int t = blockDim.x - 1 - threadIdx.x;
      if (t < C) {
        double se = 0.0, ss = 0.0;
        for (int c = 0; c < na; ++c)
          if (s_type[c] == t) { se += s_ew[c]; ss += s_ew[c] + s_sp[c]; }
        slot[dm.grad.shift_off + t] += se;
        slot[dm.grad.species_off + t] += ss;
      }
    }
    run_dual_steps<true>(g.units, p1, p2, s, lane);
    if (p2 < p3) {  // (every warp has units in the contraction's reverse step, or none)
      if (gl.rw_off >= 0) {
        // rank-weight gradients, read before the contraction's reverse: the two halves' products add
        for (int w = warp; w < gl.nw; w += warps) {
          float hi = 0.f, lo = 0.f;
          for (int p = gl.w_begin[w]; p < gl.w_begin[w + 1]; ++p) {
            const float x = s[g.rank_adj[p] * W + lane], v = s[g.rank_v[p] * W + lane];
            if (on) csum_add_prod(hi, lo, x, v);
          }
          const double sum = warp_csum(hi, lo);
          if (lane == 0) slot[gl.rw_off + w] += sum;
        }
      }
      __syncthreads();
      for (int q = warp; q < g.nzero_late; q += warps) s[g.zero_late[q] * W + lane] = 0.f;
      __syncthreads();
      run_dual_steps<true>(g.units, p2, p3, s, lane);
    }
    if (on) {
      float* row = a.abar + (n * 2 + half) * KH;
      auto get = [&](int t) {
        const int from = g.basic_adj[t];
        return from >= 0 ? s[from * W + lane] : 0.f;
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

// Gate projection weights: dJ/dW[mu][q] = sum over centres of lambda_h[mu] g[q] + mu_h[mu] gdot[q], an
// (F x 2N) (2N x Q) product over chunks of 16 centres (the 32 columns of a.gscal's rows against
// a.lh_atom's).  A thread owns T x T outputs -- mu = tm + i Tm, q = tq + j Tq, so that neighbouring
// threads read neighbouring rows -- sums a chunk in FP32 packed pairs and adds it to compensated
// totals, which go to the block's slice at the end.  T = 4 where that still fills the block's 512
// threads (12 x 36 tiles at L5/K8), else 2 (8 x 30 at L3/K4).
constexpr int kGwThreads32 = 512;
constexpr int kGwStride = 36;
__host__ __device__ inline size_t gate_weight_bytes(int F, int Q) { return sizeof(float) * kGwStride * static_cast<size_t>(F + Q); }
__host__ __device__ inline int gate_weight_tile(int F, int Q) { return ((F + 3) / 4) * ((Q + 3) / 4) >= kGwThreads32 / 2 ? 4 : 2; }
template <int T>
__global__ void __launch_bounds__(kGwThreads32) grad_gate_weight_kernel(GradArgs<float> a) {
  constexpr int A = kDualAtoms, S = kGwStride, NW = kGwThreads32 / kWarp;
  const int F = a.dm.F, Q = a.dm.Q, Tm = (F + T - 1) / T, Tq = (Q + T - 1) / T;
  const int warp = threadIdx.x / kWarp, lane = warp_lane();
  extern __shared__ __align__(16) float gw_rows[];
  float* sh = gw_rows;           // [F][S] lambda (columns 0-15), mu (16-31)
  float* sg = sh + F * S;        // [Q][S] gate scalars and tangents
  double* slot = a.slots + static_cast<size_t>(blockIdx.x) * a.dm.grad.nparams + a.dm.grad.gate_w_off;
  const int nblk = (a.natoms + A - 1) / A;
  for (int t0 = 0; t0 < Tm * Tq; t0 += kGwThreads32) {
    const bool mine = t0 + static_cast<int>(threadIdx.x) < Tm * Tq;
    const int t = mine ? t0 + threadIdx.x : 0, tm = t / Tq, tq = t - tm * Tq;
    float hi[T][T], lo[T][T];
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) hi[i][j] = lo[i][j] = 0.f;
    for (int blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
      __syncthreads();
      for (int c = warp; c < A; c += NW) {
        const int n = blk * A + c;
        for (int m = lane; m < 2 * F; m += kWarp)
          sh[(m < F ? m * S : (m - F) * S + A) + c] =
              n < a.natoms ? static_cast<float>(a.lh_atom[static_cast<size_t>(n) * 2 * F + m]) : 0.f;
      }
      for (int q = warp; q < Q; q += NW) sg[q * S + lane] = a.gscal[(static_cast<size_t>(blk) * Q + q) * kWarp + lane];
      __syncthreads();
      if (!mine) continue;
      Pair<float> acc[T][T];
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j] = {0.f, 0.f};
#pragma unroll 2
      for (int c = 0; c < kWarp; c += 4) {
        Pair<float> x0[T], x1[T], y0[T], y1[T];
#pragma unroll
        for (int i = 0; i < T; ++i) {
          load_quad(sh + min(tm + i * Tm, F - 1) * S + c, x0[i], x1[i]);
          load_quad(sg + min(tq + i * Tq, Q - 1) * S + c, y0[i], y1[i]);
        }
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) {
            acc[i][j] = fma2(x0[i], y0[j], acc[i][j]);
            acc[i][j] = fma2(x1[i], y1[j], acc[i][j]);
          }
      }
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) csum_add(hi[i][j], lo[i][j], acc[i][j].x + acc[i][j].y);
    }
    if (mine)
#pragma unroll
      for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) {
          const int mu = tm + i * Tm, q = tq + j * Tq;
          if (mu < F && q < Q) slot[mu * Q + q] += double(hi[i][j]) + double(lo[i][j]);
        }
  }
}

}  // namespace sus2g
