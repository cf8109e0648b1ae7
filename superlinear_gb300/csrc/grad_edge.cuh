// Kernels of the split parameter gradient: the edge->moment sums with tangents, and the per-edge
// parameter contributions (see grad_kernels.cuh for the method).
//
// What bounds them: instruction issue at 9 to 16 resident warps per SM.  Both stage the batch's 32
// edges by column (stage_stride) and reduce with 128-bit reads and packed pairs, as the E/F passes
// do.  The parameter kernel writes per radial channel k, for every l, the adjoints alpha_l, beta_l of
// the Chebyshev sums' values and slopes and the factors' contributions to columns beside T_b and
// dT_b/dxi and one indicator column per neighbour species; every parameter's batch sum is then the
// dot product of two columns (two pairs for a Chebyshev coefficient: sum_e alpha_l T_b + beta_l D_b),
// one parameter per lane.  Sums run over the warp's whole share of centres -- compensated FP32 (hi,
// lo) in FP32 engines -- and reach the block's FP64 slice once, at the end.
// Against a lane-private shared-memory accumulator per (parameter, lane), read and written for
// every edge and summed over the lanes per batch and channel: per-edge part of the outer / gate pass
// 516 -> 285 / 294 -> 194 us (256 frames, Effect L3/K4/R2/O2), 1621 -> 992 / 770 -> 387 us (96 frames,
// Effect L5/K8/R2/O2, three species).  The moments with tangents, the block graph kernel
// (grad_graph.cuh) and the adjoint sums replaced per-atom parts (gate forward, outer, gate reverse)
// of 255 + 341 + 158 us (L3) and 1196 + 1714 + 1165 us (L5) by 155 + 238 + 110 and 412 + 563 + 350 us.
#pragma once
#include "grad_kernels.cuh"

namespace sus2g {

// ---------------------------------------------------------------------------------------------
// Geometry of one edge with its tangent direction, shared by both kernels.
// ---------------------------------------------------------------------------------------------
// The centre's inputs: force weight and the frame's stress weights.
template <typename Real>
struct CentreWeights {
  double fx, fy, fz;
  Real s[9];
};
template <typename Real>
__device__ __forceinline__ CentreWeights<Real> centre_weights(const GradArgs<Real>& a, int atom) {
  CentreWeights<Real> w;
  const double* sw = a.sw + 9 * static_cast<size_t>(a.frame_of[atom]);
#pragma unroll
  for (int q = 0; q < 9; ++q) w.s[q] = Real(sw[q]);
  const double* f = a.fw + 3 * static_cast<size_t>(atom);
  w.fx = f[0]; w.fy = f[1]; w.fz = f[2];
  return w;
}

// One edge's record, neighbour and the neighbour's force weight.
template <typename Real>
struct GradEdge {
  typename Vec4<Real>::type d;
  int j, tj;
  double fx, fy, fz;
};
template <typename Real>
__device__ __forceinline__ GradEdge<Real> load_grad_edge(const GradArgs<Real>& a, int e, int C) {
  GradEdge<Real> x;
  x.d = a.d4[e];
  x.j = a.nbr[e];
  x.tj = C == 1 ? 0 : species_of(a.types, x.j, C);
  const double* f = a.fw + 3 * static_cast<size_t>(x.j);
  x.fx = f[0]; x.fy = f[1]; x.fz = f[2];
  return x;
}

// r, dr along the edge's direction w = fw_i - fw_j + S d, and harmonics with tangents.
template <int L, typename Real>
__device__ __forceinline__ void edge_tangent(const GradEdge<Real>& x, const CentreWeights<Real>& c, Real& r, Real& rdot,
                                             Real* Y, Real* Yd) {
  const Real dx = x.d.x, dy = x.d.y, dz = x.d.z;
  r = x.d.w;
  const Real ir = Real(1) / r;
  const Real ux = dx * ir, uy = dy * ir, uz = dz * ir;
  const Real wx = Real(c.fx - x.fx) + c.s[0] * dx + c.s[1] * dy + c.s[2] * dz;
  const Real wy = Real(c.fy - x.fy) + c.s[3] * dx + c.s[4] * dy + c.s[5] * dz;
  const Real wz = Real(c.fz - x.fz) + c.s[6] * dx + c.s[7] * dy + c.s[8] * dz;
  rdot = ux * wx + uy * wy + uz * wz;
  sph_values<L, Real>(ux, uy, uz, Y);
  sph_tangent<L, Real>(ux, uy, uz, (wx - ux * rdot) * ir, (wy - uy * rdot) * ir, (wz - uz * rdot) * ir, Yd);
}

// ---------------------------------------------------------------------------------------------
// Edge->moment sums with tangents: A = sum_e u Y, Adot = sum_e (udot Y + u Ydot), to
// a.mom [N][2][K H].  Columns: u [F], udot [F], Y [H], Ydot [H].
// ---------------------------------------------------------------------------------------------
template <typename Real>
__host__ __device__ inline int grad_moment_warp_size(int L, int K) {
  const int H = (L + 1) * (L + 1), F = K * (L + 1);
  // the unused slots of the last channel group reach at most G (L + 1) columns past the u columns
  const int reach = moment_slots(L, K) * (H <= kWarp ? kWarp / H : 1) * (L + 1);
  return round4((max(2 * F + 2 * H, F + reach)) * stage_stride<Real>());
}

template <int NS, int STEP, int TAIL, typename Real, int N>
__device__ __forceinline__ void moment_batch_dual(const Real* u, int ud, const Real* y, int yd, const Real* ut,
                                                  const Real* yt, int nb, Pair<Real> (&part)[N], Pair<Real> (&dot)[N]) {
#pragma unroll
  for (int s = 0; s < N; ++s) part[s] = dot[s] = {Real(0), Real(0)};
  for (int q = 0; q < nb; q += 4) {
    Pair<Real> y0, y1, d0, d1, u0, u1, v0, v1;
    load_quad(y + q, y0, y1);
    load_quad(y + yd + q, d0, d1);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      load_quad(u + s * STEP + q, u0, u1);
      load_quad(u + s * STEP + ud + q, v0, v1);
      part[s] = fma2(u0, y0, part[s]);
      dot[s] = fma2(v0, y0, dot[s]);
      part[s] = fma2(u1, y1, part[s]);
      dot[s] = fma2(v1, y1, dot[s]);
      dot[s] = fma2(u0, d0, dot[s]);
      dot[s] = fma2(u1, d1, dot[s]);
    }
    if constexpr (TAIL) {
      load_quad(yt + q, y0, y1);
      load_quad(yt + yd + q, d0, d1);
      load_quad(ut + q, u0, u1);
      load_quad(ut + ud + q, v0, v1);
      part[N - 1] = fma2(u0, y0, part[N - 1]);
      dot[N - 1] = fma2(v0, y0, dot[N - 1]);
      part[N - 1] = fma2(u1, y1, part[N - 1]);
      dot[N - 1] = fma2(v1, y1, dot[N - 1]);
      dot[N - 1] = fma2(u0, d0, dot[N - 1]);
      dot[N - 1] = fma2(u1, d1, dot[N - 1]);
    }
  }
}

// Register budgets: 128 (blocks of up to 128 threads, four per SM) up to L = 3; at L = 4 and 5 168,
// which spill less, in blocks of up to 384 threads (shared memory admits 9 to 12 warps per SM there,
// most of them in one block with one copy of the tables).  FP64: 255.
__host__ __device__ constexpr int grad_max_warps(int L, bool fp32) { return fp32 && L >= 4 ? 12 : 4; }
__host__ __device__ constexpr int grad_min_blocks(int L, bool fp32) { return !fp32 ? 2 : L >= 4 ? 1 : 4; }

template <int L, typename Real, int MODE, int BF>
__global__ void __launch_bounds__(kWarp * grad_max_warps(L, sizeof(Real) == 4), grad_min_blocks(L, sizeof(Real) == 4)) grad_moment_kernel(GradArgs<Real> a) {
  constexpr int Lp = L + 1, H = Lp * Lp, S = stage_stride<Real>();
  constexpr bool KAHAN = sizeof(Real) == 4;
  using MI = MomentItems<L>;
  constexpr int NS = MI::KS + (MI::kTail ? 1 : 0);
  const DevModel<Real>& dm = a.dm;
  const PassTables<Real>& pt = MODE == kGradOuter ? dm.outer : dm.gate;
  const bool effect_outer = MODE == kGradOuter && dm.gated;
  const int C = dm.C, F = dm.F, B = BF ? BF : dm.B, K = dm.K;
  const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = warp_lane();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Real* s_coeff = reinterpret_cast<Real*>(smem_raw);
  Real* s_scal = s_coeff + F * B;
  Real* s_w0 = s_scal + 2 * dm.nblk * C * C;
  Real* s_w1 = s_w0 + C * F;
  Real* s_wa = s_w1 + C * F;
  Real* stage = reinterpret_cast<Real*>(smem_raw) + round4(pass_table_size<Real>(C, F, B, dm.nblk)) +
                grad_moment_warp_size<Real>(L, K) * warp;
  for (int q = threadIdx.x; q < F * B; q += blockDim.x) s_coeff[q] = pt.coeff[q];
  for (int q = threadIdx.x; q < 2 * dm.nblk * C * C; q += blockDim.x) s_scal[q] = pt.scal[q];
  for (int q = threadIdx.x; q < C * F; q += blockDim.x) {
    s_w0[q] = pt.wcenter[q];
    s_w1[q] = pt.wsource[q];
    s_wa[q] = pt.wadd ? pt.wadd[q] : Real(0);
  }
  __syncthreads();

  const bool item_on = lane < MI::G * H;
  const int lm = H <= kWarp ? (item_on ? lane % H : 0) : lane, kg = H <= kWarp && item_on ? lane / H : 0;
  auto l_of = [](int h) {
    int l = 0;
#pragma unroll
    for (int q = 1; q < Lp; ++q) l += h >= q * q;
    return l;
  };
  const Real* col_u = stage + (kg * Lp + l_of(lm)) * S;
  const Real* col_y = stage + (2 * F + lm) * S;
  constexpr int TW = MI::kTail ? MI::kTail : 1;
  const int lmt = kWarp + lane % TW, kt = lane / TW;
  const Real* col_ut = stage + (min(kt, K - 1) * Lp + L) * S;
  const Real* col_yt = stage + (2 * F + lmt) * S;
  auto item_of = [&](int q) {
    if (MI::kTail && q == MI::KS) return kt < K ? kt * H + lmt : -1;
    const int k = kg + q * MI::G;
    return (H > kWarp || item_on) && k < K ? k * H + lm : -1;
  };
  const bool half_slots = MI::KS >= 2 && moment_slots(L, K) < MI::KS;

  for (int atom = blockIdx.x * warps + warp; atom < a.natoms; atom += gridDim.x * warps) {
    const int ti = C == 1 ? 0 : species_of(a.types, atom, C);
    const int e0 = a.row[atom], e1 = a.row_end[atom];
    const CentreWeights<Real> cw = centre_weights<Real>(a, atom);
    Real acc[NS], cmp[NS], accd[NS], cmpd[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) acc[q] = cmp[q] = accd[q] = cmpd[q] = Real(0);
    GradEdge<Real> cur{};
    if (e0 + lane < e1) cur = load_grad_edge<Real>(a, e0 + lane, C);
    for (int base = e0; base < e1; base += kWarp) {
      const int e = base + lane, nb = min(kWarp, e1 - base);
      GradEdge<Real> nxt = cur;
      if (e + kWarp < e1) nxt = load_grad_edge<Real>(a, e + kWarp, C);
      if (effect_outer) {
        rows_to_cols<Real>(stage, a.hsig, F, cur.j, nb, lane);
        rows_to_cols<Real>(stage + F * S, a.hsigd, F, cur.j, nb, lane);
      }
      Real* col = stage + lane;
      if (e < e1) {
        Real r, rdot;
        {
          Real Y[H], Yd[H];
          edge_tangent<L, Real>(cur, cw, r, rdot, Y, Yd);
#pragma unroll
          for (int h = 0; h < H; ++h) {
            col[(2 * F + h) * S] = Y[h];
            col[(2 * F + H + h) * S] = Yd[h];
          }
        }
        const Envelopes<Real> env = edge_envelopes<Real>(dm, r);
        const Real* w0 = s_w0 + ti * F;
        const Real* w1 = s_w1 + cur.tj * F;
        const Real* wa = s_wa + cur.tj * F;
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
          Real R[Lp], Rd[Lp];
          radial_channel<L, Real, true, BF>(dm, s_coeff, s_scal, ti * C + cur.tj, r, env, k, R, Rd);
          Real* ck = col + k * Lp * S;
#pragma unroll
          for (int l = 0; l < Lp; ++l) {
            const int m = k * Lp + l;
            const Real x0 = w0[m];
            Real x3 = w1[m], x3d = Real(0);
            if (effect_outer) {
              const Real al = wa[m];
              x3 += al * ck[l * S];
              x3d = al * ck[(F + l) * S];
            }
            ck[l * S] = x0 * x3 * R[l];
            ck[(F + l) * S] = x0 * (x3d * R[l] + x3 * Rd[l] * rdot);
          }
        }
      } else {
        for (int q = 0; q < 2 * F + 2 * H; ++q) col[q * S] = Real(0);
      }
      __syncwarp();
      Pair<Real> part[NS], dot[NS];
      if (half_slots)
        moment_batch_dual<MI::KS >= 2 ? MI::KS / 2 : MI::KS, MI::G * Lp * S, MI::kTail>(col_u, F * S, col_y, H * S, col_ut,
                                                                                        col_yt, nb, part, dot);
      else
        moment_batch_dual<MI::KS, MI::G * Lp * S, MI::kTail>(col_u, F * S, col_y, H * S, col_ut, col_yt, nb, part, dot);
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        kadd<Real, KAHAN>(acc[q], cmp[q], part[q].x + part[q].y);
        kadd<Real, KAHAN>(accd[q], cmpd[q], dot[q].x + dot[q].y);
      }
      __syncwarp();
      cur = nxt;
    }
    Real* out = a.mom + static_cast<size_t>(atom) * 2 * K * H;
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const int t = item_of(q);
      if (t >= 0) { out[t] = acc[q]; out[K * H + t] = accd[q]; }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Per-edge parameter contributions from the moment adjoints a.abar [N][2][K H].
// ---------------------------------------------------------------------------------------------
// Columns of one radial channel: alpha, beta [Lp], T, D [B], centre and neighbour factor [Lp], warp
// slope and shift; Effect outer: gate additive factor [Lp] and the neighbours' h and hdot [2 Lp],
// which the channel's gate-signal adjoints lambda, mu overwrite; then the indicators of
// the neighbour's species [C] and ones (the only columns whose number is not compiled in).
struct GradCols {
  int beta, T, D, x0, xj, sc, al, h, ind;  // column offsets (alpha 0)
};
__host__ __device__ constexpr GradCols grad_cols(int Lp, int B, bool effect_outer) {
  GradCols g{};
  g.beta = Lp;
  g.T = 2 * Lp;
  g.D = g.T + B;
  g.x0 = g.D + B;
  g.xj = g.x0 + Lp;
  g.sc = g.xj + Lp;
  g.al = g.sc + 2;
  g.h = g.al + (effect_outer ? Lp : 0);
  g.ind = g.h + (effect_outer ? 2 * Lp : 0);
  return g;
}
// Parameters per channel: Chebyshev; per neighbour species (neighbour factor, additive factor);
// per centre species (centre factor, warp slope and shift per neighbour species).
struct GradItems { int ncoef, nj, nc; };
__host__ __device__ inline GradItems grad_items(int Lp, int B, int C, bool effect_outer) {
  return {Lp * B, C * Lp * (effect_outer ? 2 : 1), Lp + 2 * C};
}
// Accumulators of a warp: [K][ncoef + nj] and [C][K][nc], each (hi, lo) in FP32 engines.
template <typename Real>
__host__ __device__ inline int grad_edge_acc(const GradItems& n, int K, int C) {
  return (sizeof(Real) == 4 ? 2 : 1) * K * (n.ncoef + n.nj + C * n.nc);
}
template <typename Real>
__host__ __device__ inline int grad_edge_warp_floats(int L, int K, int B, int C, bool effect_outer) {
  return round4((grad_cols(L + 1, B, effect_outer).ind + C + 1) * stage_stride<Real>()) + 2 * K * round4((L + 1) * (L + 1)) +
         round4(grad_edge_acc<Real>(grad_items(L + 1, B, C, effect_outer), K, C));
}
// The block's item table: (column a, column b) of the nj + nc single dot products.
__host__ __device__ inline int grad_edge_items(const GradItems& n) { return round4(n.nj + n.nc); }

template <typename Real>
__device__ __forceinline__ void acc_add(Real* acc, int i, Real x) {
  if constexpr (sizeof(Real) == 4) {
    Pair<Real>* p = reinterpret_cast<Pair<Real>*>(acc) + i;
    Pair<Real> v = *p;
    csum_add(v.x, v.y, x);
    *p = v;
  } else {
    acc[i] += x;
  }
}
template <typename Real>
__device__ __forceinline__ double acc_get(const Real* acc, int i) {
  if constexpr (sizeof(Real) == 4) return double(acc[2 * i]) + double(acc[2 * i + 1]);
  else return acc[i];
}

// One value from global to shared memory, asynchronously (joined by cp_async_commit / cp_async_wait).
template <typename Real>
__device__ __forceinline__ void cp_async_value(Real* dst, const Real* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(sizeof(Real)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// sum_q x[q] y[q] over a batch's columns, and sum_q x[q] y[q] + z[q] w[q] (sixteen edges at a time:
// the columns of edges past the batch are zero).
template <typename Real>
__device__ __forceinline__ Real col_dot(const Real* x, const Real* y, int nb) {
  Pair<Real> s{Real(0), Real(0)}, t = s, x0, x1, y0, y1;
#pragma unroll 1
  for (int q0 = 0; q0 < nb; q0 += 16)
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
      load_quad(x + q0 + q, x0, x1);
      load_quad(y + q0 + q, y0, y1);
      s = fma2(x0, y0, s);
      t = fma2(x1, y1, t);
    }
  return (s.x + s.y) + (t.x + t.y);
}
template <typename Real>
__device__ __forceinline__ Real col_dot(const Real* x, const Real* y, const Real* z, const Real* w, int nb) {
  Pair<Real> s{Real(0), Real(0)}, t = s, x0, x1, y0, y1, z0, z1, w0, w1;
#pragma unroll 1
  for (int q0 = 0; q0 < nb; q0 += 16)
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
      load_quad(x + q0 + q, x0, x1);
      load_quad(y + q0 + q, y0, y1);
      load_quad(z + q0 + q, z0, z1);
      load_quad(w + q0 + q, w0, w1);
      s = fma2(x0, y0, s);
      t = fma2(z0, w0, t);
      s = fma2(x1, y1, s);
      t = fma2(z1, w1, t);
    }
  return (s.x + s.y) + (t.x + t.y);
}

// EFFECT: the outer pass of a gated model (gate signals in, their adjoints out).
template <int L, typename Real, int MODE, int BF, bool EFFECT>
__global__ void __launch_bounds__(kWarp * grad_max_warps(L, sizeof(Real) == 4), grad_min_blocks(L, sizeof(Real) == 4)) grad_edge_kernel(GradArgs<Real> a) {
  constexpr int Lp = L + 1, H = Lp * Lp, H4 = round4(H), NPH = (H + 1) / 2, S = stage_stride<Real>();
  constexpr int B = BF, NP = BF / 2, NC = (Lp * B + kWarp - 1) / kWarp;
  static_assert(BF > 0 && BF % 2 == 0, "compiled basis sizes only");
  const DevModel<Real>& dm = a.dm;
  const PassTables<Real>& pt = MODE == kGradOuter ? dm.outer : dm.gate;
  const PassGradLayout& gl = MODE == kGradOuter ? dm.grad.outer : dm.grad.gate;
  const int C = dm.C, F = dm.F, K = dm.K, C2 = C * C;
  const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = warp_lane();
  constexpr GradCols g = grad_cols(Lp, B, EFFECT);
  const GradItems n = grad_items(Lp, B, C, EFFECT);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Real* s_coeff = reinterpret_cast<Real*>(smem_raw);
  Real* s_scal = s_coeff + F * B;
  Real* s_w0 = s_scal + 2 * dm.nblk * C2;
  Real* s_w1 = s_w0 + C * F;
  Real* s_wa = s_w1 + C * F;
  int* s_item = reinterpret_cast<int*>(reinterpret_cast<Real*>(smem_raw) + round4(pass_table_size<Real>(C, F, B, dm.nblk)));
  const int wfloats = grad_edge_warp_floats<Real>(L, K, B, C, EFFECT);
  Real* stage = reinterpret_cast<Real*>(s_item + grad_edge_items(n)) + wfloats * warp;
  Real* abl = stage + round4((g.ind + C + 1) * S);  // [K][H4]
  Real* abm = abl + K * H4;
  Real* acc = abm + K * H4;             // [K][ncoef + nj], [C][K][nc]
  const int naccs = grad_edge_acc<Real>(n, K, C), acc_c = K * (n.ncoef + n.nj);

  for (int q = threadIdx.x; q < F * B; q += blockDim.x) s_coeff[q] = pt.coeff[q];
  for (int q = threadIdx.x; q < 2 * dm.nblk * C2; q += blockDim.x) s_scal[q] = pt.scal[q];
  for (int q = threadIdx.x; q < C * F; q += blockDim.x) {
    s_w0[q] = pt.wcenter[q];
    s_w1[q] = pt.wsource[q];
    s_wa[q] = pt.wadd ? pt.wadd[q] : Real(0);
  }
  // items: neighbour species (t, xj_l), then (t, al_l); centre species: x0_l, then (t, slope), (t, shift)
  for (int q = threadIdx.x; q < n.nj + n.nc; q += blockDim.x) {
    int ca, cb;
    if (q < n.nj) {
      const int t = (q / Lp) % C, l = q % Lp;
      ca = (q < C * Lp ? g.xj : g.al) + l;
      cb = g.ind + t;
    } else if (q < n.nj + Lp) {
      ca = g.x0 + q - n.nj;
      cb = g.ind + C;
    } else {
      const int i = q - n.nj - Lp;
      ca = g.sc + i % 2;
      cb = g.ind + i / 2;
    }
    s_item[q] = ca | (cb << 16);
  }
  for (int q = lane; q < naccs; q += kWarp) acc[q] = Real(0);
  __syncthreads();

  for (int atom = blockIdx.x * warps + warp; atom < a.natoms; atom += gridDim.x * warps) {
    const int ti = C == 1 ? 0 : species_of(a.types, atom, C);
    const int e0 = a.row[atom], e1 = a.row_end[atom];
    const CentreWeights<Real> cw = centre_weights<Real>(a, atom);
    {
      const Real* src = a.abar + static_cast<size_t>(atom) * 2 * K * H;
      for (int t = lane; t < K * H; t += kWarp) {
        abl[t / H * H4 + t % H] = src[t];
        abm[t / H * H4 + t % H] = src[K * H + t];
      }
    }
    GradEdge<Real> cur{};
    if (e0 + lane < e1) cur = load_grad_edge<Real>(a, e0 + lane, C);
    for (int base = e0; base < e1; base += kWarp) {
      const int e = base + lane, nb = min(kWarp, e1 - base);
      const bool valid = e < e1;
      GradEdge<Real> nxt = cur;
      if (e + kWarp < e1) nxt = load_grad_edge<Real>(a, e + kWarp, C);
      Real* col = stage + lane;
      const int tj = cur.tj, rv = EFFECT && valid ? a.rev[e] : 0;
      Real r = Real(1), rdot = Real(0), Y[2 * NPH], Yd[2 * NPH];
      Y[2 * NPH - 1] = Yd[2 * NPH - 1] = Real(0);
      __syncwarp();
      for (int t = 0; t < C; ++t) col[(g.ind + t) * S] = valid && tj == t ? Real(1) : Real(0);
      col[(g.ind + C) * S] = valid ? Real(1) : Real(0);
      if (valid) edge_tangent<L, Real>(cur, cw, r, rdot, Y, Yd);
      else for (int q = 0; q < g.ind; ++q) col[q * S] = Real(0);
      const Envelopes<Real> env = edge_envelopes<Real>(dm, r);
      // Effect outer pass: the neighbours' h and hdot of channel k as (edge, l) elements, Lp
      // consecutive values per edge, the next channel's copied during this one's batch sums
      int hq[Lp];
      auto fetch_h = [&](int k) {
#pragma unroll
        for (int i = 0; i < Lp; ++i) {
          const int q = (i * kWarp + lane) / Lp, l = (i * kWarp + lane) % Lp;
          Real* dst = stage + (g.h + l) * S + q;
          if (q < nb) {
            cp_async_value(dst, a.hsig + hq[i] + k * Lp);
            cp_async_value(dst + Lp * S, a.hsigd + hq[i] + k * Lp);
          }
        }
        cp_async_commit();
      };
      Real* col_h = col + g.h * S;
      if constexpr (EFFECT) {
#pragma unroll
        for (int i = 0; i < Lp; ++i)
          hq[i] = __shfl_sync(0xffffffffu, cur.j, (i * kWarp + lane) / Lp) * F + (i * kWarp + lane) % Lp;
        fetch_h(0);
      }
#pragma unroll 1
      for (int k = 0; k < K; ++k) {
        if constexpr (EFFECT) {
          cp_async_wait<0>();
          __syncwarp();
        }
        if (valid) {
          // SU_l = sum_m lambda Y + mu Ydot, TT_l = sum_m mu Y
          Pair<Real> SU[Lp], TT[Lp];
#pragma unroll
          for (int l = 0; l < Lp; ++l) SU[l] = TT[l] = {Real(0), Real(0)};
#pragma unroll
          for (int h0 = 0; h0 < H; h0 += 4) {
            Pair<Real> Al[2], Am[2];
            load_quad(abl + k * H4 + h0, Al[0], Al[1]);
            load_quad(abm + k * H4 + h0, Am[0], Am[1]);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int h = h0 + 2 * u;
              if (h < H) {
                int la = 0, lb = 0;
#pragma unroll
                for (int q = 1; q < Lp; ++q) { la += h >= q * q; lb += h + 1 >= q * q; }
                const Pair<Real> y{Y[h], Y[h + 1]}, yd{Yd[h], Yd[h + 1]};
                if (h + 1 < H && la == lb) {
                  SU[la] = fma2(Al[u], y, SU[la]);
                  SU[la] = fma2(Am[u], yd, SU[la]);
                  TT[la] = fma2(Am[u], y, TT[la]);
                } else {
                  SU[la].x += Al[u].x * y.x + Am[u].x * yd.x;
                  TT[la].x += Am[u].x * y.x;
                  if (h + 1 < H) {
                    SU[lb].y += Al[u].y * y.y + Am[u].y * yd.y;
                    TT[lb].y += Am[u].y * y.y;
                  }
                }
              }
            }
          }
          const int sb = scaling_block(dm.scaling_mode, k, 0, Lp);
          const WarpVar<Real> wv = warp_var<Real>(r, s_scal[2 * sb * C2 + ti * C + tj], s_scal[(2 * sb + 1) * C2 + ti * C + tj]);
          Pair<Real> T[NP], D[NP], DD[NP];
          cheb_pairs<Real, NP, true>(wv.xi, B, T, D);
          {
            // DD_b = 4 D_b-1 + 2 xi DD_b-1 - DD_b-2, from DD_2 = 4
            Real p2 = Real(0), p1 = Real(4);
            DD[0] = {Real(0), Real(0)};
            DD[1].x = p1;
#pragma unroll
            for (int b = 3; b < B; ++b) {
              const Real db = b & 1 ? D[b / 2].x : D[b / 2 - 1].y;  // D_b-1
              const Real v = Real(4) * db + (Real(2) * wv.xi * p1 - p2);
              p2 = p1; p1 = v;
              if (b & 1) DD[b / 2].y = v;
              else DD[b / 2].x = v;
            }
          }
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            col[(g.T + 2 * p) * S] = T[p].x;
            col[(g.T + 2 * p + 1) * S] = T[p].y;
            col[(g.D + 2 * p) * S] = D[p].x;
            col[(g.D + 2 * p + 1) * S] = D[p].y;
          }
          Real g1 = Real(0), g2 = Real(0), g3 = Real(0);
#pragma unroll
          for (int l = 0; l < Lp; ++l) {
            const int m = k * Lp + l;
            Real cc[B];
            load_coeff_row<Real, B, B>(s_coeff + m * B, B, cc);
            // (T_0 = 1, D_0 = DD_0 = DD_1 = 0 and D_1 = 1 need no product)
            Pair<Real> sa{cc[0], cc[1] * T[0].y}, sd{Real(0), cc[1]}, se{Real(0), Real(0)};
#pragma unroll
            for (int p = 1; p < NP; ++p) {
              const Pair<Real> c{cc[2 * p], cc[2 * p + 1]};
              sa = fma2(c, T[p], sa);
              sd = fma2(c, D[p], sd);
              se = fma2(c, DD[p], se);
            }
            const Real cT = sa.x + sa.y, cD = sd.x + sd.y, cDD = se.x + se.y;
            const Real f = l == 0 ? env.f0 : env.f1, fd = l == 0 ? env.fd0 : env.fd1;
            const Real R = f * cT, Rd = fd * cT + f * cD * wv.xr;
            const Real su = SU[l].x + SU[l].y, tt = TT[l].x + TT[l].y;
            const Real x0 = s_w0[ti * F + m];
            Real x3 = s_w1[tj * F + m], x3d = Real(0), al = Real(0), hv = Real(0), hdv = Real(0);
            if constexpr (EFFECT) {
              al = s_wa[tj * F + m];
              hv = col_h[l * S];
              hdv = col_h[(Lp + l) * S];
              x3 += al * hv;
              x3d = al * hdv;
            }
            const Real RT = R * tt, Qv = R * su + Rd * rdot * tt;
            const Real dRd = x0 * x3 * rdot * tt;
            const Real dR = x0 * (x3 * su + x3d * tt);
            const Real al_ = dR * f + dRd * fd, fr = dRd * f;
            col[l * S] = al_;
            col[(g.beta + l) * S] = fr * wv.xr;
            col[(g.x0 + l) * S] = x3 * Qv + x3d * RT;
            col[(g.xj + l) * S] = x0 * Qv;
            g1 += al_ * cD;
            g2 += fr * cD;
            g3 += fr * cDD;
            if constexpr (EFFECT) {
              col[(g.al + l) * S] = x0 * (Qv * hv + RT * hdv);
              col_h[l * S] = x0 * al * Qv;
              col_h[(Lp + l) * S] = x0 * al * RT;
            }
          }
          // warp slope and shift of the pair (t_i, t_j)
          col[g.sc * S] = wv.xs * (g1 + wv.xr * g3) + wv.xrs * g2;
          col[(g.sc + 1) * S] = wv.xg * (g1 + wv.xr * g3) + wv.xrg * g2;
        }
        __syncwarp();
        if constexpr (EFFECT) {
          // the gate-signal adjoints of this channel: 2 Lp consecutive values of the reverse edge's row
          const Real* out = stage + g.h * S;
#pragma unroll
          for (int i = 0; i < 2 * Lp; ++i) {
            const int q = (i * kWarp + lane) / (2 * Lp), c = (i * kWarp + lane) % (2 * Lp);
            const int row = __shfl_sync(0xffffffffu, rv, q);
            if (q < nb) a.lhm[static_cast<size_t>(row) * 2 * F + k * 2 * Lp + c] = out[c * S + q];
          }
          __syncwarp();
          if (k + 1 < K) fetch_h(k + 1);
        }
        // batch sums: Chebyshev coefficients (l, b), then the single products
#pragma unroll
        for (int s = 0; s < NC; ++s) {
          const int it = lane + kWarp * s;
          if (it < Lp * B) {
            const int l = it / B, b = it % B;
            acc_add(acc, k * (n.ncoef + n.nj) + it,
                    col_dot(stage + l * S, stage + (g.T + b) * S, stage + (g.beta + l) * S, stage + (g.D + b) * S, nb));
          }
        }
        for (int it = lane; it < n.nj + n.nc; it += kWarp) {
          const int w = s_item[it];
          const Real x = col_dot(stage + (w & 0xffff) * S, stage + (w >> 16) * S, nb);
          if (it < n.nj) acc_add(acc, k * (n.ncoef + n.nj) + n.ncoef + it, x);
          else acc_add(acc, acc_c + (ti * K + k) * n.nc + it - n.nj, x);
        }
        __syncwarp();
      }
      cur = nxt;
    }
  }
  // the block's slice: a thread per parameter adds the warps' sums in warp order
  __syncthreads();
  double* slot = a.slots + static_cast<size_t>(blockIdx.x) * dm.grad.nparams;
  const Real* acc0 = acc - static_cast<size_t>(warp) * wfloats;
  auto block_sum = [&](int i) {
    double v = 0.0;
    for (int w = 0; w < warps; ++w) v += acc_get(acc0 + static_cast<size_t>(w) * wfloats, i);
    return v;
  };
  for (int i = threadIdx.x; i < K * (n.ncoef + n.nj); i += blockDim.x) {
    const int k = i / (n.ncoef + n.nj), it = i - k * (n.ncoef + n.nj);
    int p;
    if (it < n.ncoef) {
      p = gl.coeff_off + (k * Lp + it / B) * gl.coeff_stride + it % B;
    } else {
      const int q = it - n.ncoef, t = (q / Lp) % C, m = k * Lp + q % Lp;
      p = q < C * Lp ? gl.wc_off + t * gl.wc_t_stride + m * gl.wc_mu_stride : gl.add_off + t * F + m;
    }
    slot[p] += block_sum(i);
  }
  __syncthreads();
  // centre-species sums (in the "pair" map a warp parameter appears under every k: one thread's)
  for (int i = threadIdx.x; i < C * n.nc; i += blockDim.x) {
    const int t = i / n.nc, it = i - t * n.nc;
    for (int k = 0; k < K; ++k) {
      int p;
      if (it < Lp) {
        p = gl.wc_off + t * gl.wc_t_stride + (k * Lp + it) * gl.wc_mu_stride;
      } else {
        const int sb = scaling_block(dm.scaling_mode, k, 0, Lp), q = it - Lp;
        p = gl.scal_off + (2 * sb + q % 2) * C2 + t * C + q / 2;
      }
      slot[p] += block_sum(acc_c + (t * K + k) * n.nc + it);
    }
  }
}

// The gate-signal adjoints (dJ/dh, dJ/dhdot) of every centre: its edges' rows summed per column, warp
// per centre (as hbar_sum_kernel); rows hold [k][lambda_l, mu_l], the sums go out as [lambda F, mu F]
// with the objective's own dJ/dh added.
template <typename Real>
__global__ void __launch_bounds__(256) lhm_sum_kernel(GradArgs<Real> a, int Lp) {
  constexpr int V = 16 / sizeof(Real);
  using W = typename RowUnit<Real>::type;
  const int F = a.dm.F, lane = warp_lane();
  const int atom = static_cast<int>((static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) / kWarp);
  if (atom >= a.natoms) return;
  const int e0 = a.row[atom], n = a.row_end[atom] - e0;
  const Real* rows = a.lhm + static_cast<size_t>(e0) * 2 * F;
  double* out = a.lh_atom + static_cast<size_t>(atom) * 2 * F;
  auto put = [&](int c, Real x) {
    const int k = c / (2 * Lp), i = c - k * 2 * Lp, m = k * Lp + (i < Lp ? i : i - Lp);
    double v = double(x);
    if (i < Lp && a.extra_h) v += a.extra_h[static_cast<size_t>(atom) * F + m];
    out[i < Lp ? m : F + m] = v;
  };
  if ((2 * F) % V != 0 || 2 * F / V > kWarp) {
    for (int c = lane; c < 2 * F; c += kWarp) put(c, column_sum<Real>(rows + c, 2 * F, n));
    return;
  }
  const int nc = 2 * F / V, groups = kWarp / nc, grp = lane / nc, c = lane - grp * nc;
  const W* src = reinterpret_cast<const W*>(rows) + c;
  Real t[V], own[V];
#pragma unroll
  for (int i = 0; i < V; ++i) t[i] = Real(0);
  if (grp < groups) {
    for (int e = grp; e < n; e += 8 * groups) {
      W w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e + u * groups < n) w[u] = src[static_cast<size_t>(e + u * groups) * nc];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e + u * groups < n) {
          t[0] += w[u].x; t[1] += w[u].y;
          if constexpr (V == 4) { t[2] += w[u].z; t[3] += w[u].w; }
        }
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) own[i] = t[i];
  for (int q = 1; q < groups; ++q)
#pragma unroll
    for (int i = 0; i < V; ++i) t[i] += __shfl_sync(0xffffffffu, own[i], min(lane + q * nc, kWarp - 1));
  if (lane < nc)
#pragma unroll
    for (int i = 0; i < V; ++i) put(V * c + i, t[i]);
}

}  // namespace sus2g
