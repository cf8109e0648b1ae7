// Warp-per-atom passes of the SUS2-SH energy / force / virial evaluation.
//
// Algorithm (per centre atom i, edges e = (i -> j, d) sorted by centre):
//   forward   A_i[k,l,m] = sum_e x0(t_i,mu) x3(t_j,mu) R_mu(r_e) Y_lm(d_e),  mu = k (L+1) + l
//             (sus2_sl_kernel.cpp:340-354 forward_moments, :165-216 edge_basis)
//   contract  ranked K -> rank contraction (sus2_sl_kernel.cpp:104-105, 217-221)
//   graph     v[out] += c v[a] v[b] over the pass's product range (:308-313)
//   readout   E_i = species + shift + sum_q rho_q v[map q]            (:556)
//   reverse   adjoint of readout, graph and contraction (:527-528), then per edge
//             g_e = dE/dd_e = sum_b Abar[b] x0 x3 (R'_mu d/r Y_h + R_mu grad Y_h)  (:356-380)
//   Effect    gate pass first (x0 x1 = gate type factors, gate radial / warp), h_i = W g_i
//             (:447-455); outer x3 = tau_j + alpha_j h_j; the outer reverse also emits
//             hbar_j[mu] += Abar x0 alpha R Y (:368), gathered per atom and pushed back through
//             the gate graph (:558-559).
//
// GPU mapping: one warp owns one centre atom at a time.  Lanes take edges (32 per batch); each
// lane evaluates Y_lm and the radial functions of its edge in registers and stages u_mu =
// x0 x3 R_mu and Y_h in shared memory, one column per quantity; lanes then switch to owning (k, lm)
// moment items and reduce over the staged edges in a fixed order: plain sums over each batch of
// <= 32 edges (even and odd edges apart, then together), then a Kahan-compensated add of the batch
// partial into the atom's moment (FP32 bulk) -- no atomics, deterministic.
//
// What bounds it: instruction issue and the latency of dependent steps at 12 to 16 resident warps
// per SM (DRAM 1-12% busy), so the per-edge loops are written for few instructions: staged
// columns read four edges at a time with one Y read per channel group, packed FP32 pairs over
// edges (moments), basis index (radial sums) and harmonics (adjoints), gate-signal rows moved as
// whole sectors.  Against one row per edge with scalar reads of both factors: gate forward 133.7 ->
// 72.2 M warp instructions and 266 -> 183 us, outer 259 -> 195 M and 533 -> 435 us, gate reverse
// 149 -> 124 M and 259 -> 241 us (Effect L4/K8/R2/O3, 8,000 atoms); Static L3/K4/O2, 32,768 atoms:
// step 782 -> 680 us.  The rank contraction and the product graph, forward and reverse, run as the
// pass's lane-balanced graph program (GraphProg) over shared-memory node arrays.  The adjoint
// pass recomputes Y and R per edge instead of storing them and writes g_e per edge; forces are
// gathered per atom through the reverse-edge permutation by a separate kernel.
#pragma once
#include <type_traits>

#include "basis.cuh"

namespace sus2g {

enum PassMode : int {
  kModeStatic = 0, kModeGateForward = 1, kModeOuter = 2, kModeGateReverse = 3,
  // the Static pass split at the per-atom boundary into three kernels: the edge->moment forward
  // (moments to a.mom), the per-atom graph (graph_block_kernel: readout, adjoint moments to
  // a.amom) and the per-edge adjoint (from a.amom)
  kModeStaticFwd = 4, kModeStaticRev = 5,
  // the Effect outer pass compiled with the neighbours' gate-signal rows h_j brought into shared
  // memory by 1-D bulk async copies, one 32-edge batch ahead (a kernel variant of kModeOuter)
  kModeOuterBulk = 6,
  // the Effect outer pass split like the Static pass (forward with h_j, per-atom graph kernel,
  // adjoint writing the hbar contributions)
  kModeOuterFwd = 7, kModeOuterRev = 8,
  // the Effect gate passes split the same way: the gate forward pass's edge->moment part (the
  // per-atom gate graph and gate-signal projection then run in graph_block_kernel), and the gate
  // reverse pass's per-edge adjoint (after graph_block_kernel gathered the gate-signal adjoint and
  // ran the gate graph's reverse)
  kModeGateFwdEdges = 9, kModeGateRevEdges = 10
};

template <typename Real>
struct PassArgs {
  DevModel<Real> dm;
  int natoms;
  const int* types;
  const int* row;          // [natoms] first edge of each centre
  const int* row_end;      // [natoms] one past its last edge (row + 1 for CSR layouts)
  const int* nbr;          // [E]
  const int* rev;          // [E] reverse edge
  const typename Vec4<Real>::type* d4;  // [E] (dx, dy, dz, r)
  Real* g;                 // [E][3] dE/dd per edge (written by static/outer, accumulated by gate reverse)
  Real* hsig;              // [natoms][F] gate signal h (written by gate forward)
  Real* hcontrib;          // [E][F] per-edge hbar contributions, stored at the reverse edge
  Real* gmom;              // [natoms][M] gate moment values (gate forward -> gate reverse)
  const double* hbar_atom; // [natoms][F] gate-signal adjoint already summed per atom (caller edges), or null
  Real* gkeep;             // [natoms / 32][nkeep][32] gate values the reverse reads (split gate passes)
  Real* hbar;              // [natoms][F] the same, as hbar_atom, by hbar_sum_kernel (split gate reverse pass)
  double* site_energy;     // [natoms]
  double* virial;          // [natoms][6] (xx, yy, zz, xy, xz, yz), minus d (x) g
  double* desc;            // [natoms][S] scalar moments (descriptors), or null
  Real* mom;               // [natoms][K H] moments (split Static pass: forward -> graph kernel)
  Real* amom;              // [natoms][K H] their adjoints (graph kernel -> per-edge adjoint)
  int* error;
  int moment_mma;          // FP32 engines: 1 = edge->moment batch sums on the tensor cores (3xTF32 mma.sync)
  int atom_order;          // 0: warps take centres grid-strided; 1: each warp a contiguous run of
                           // centres; 2: warps take the next centre from a device counter as they
                           // finish -- dynamic balance for uneven centres
  int* work;               // atom_order 2: {next centre, warps done}, zero at launch; the last warp
                           // to finish zeroes both for the next launch
  int h_bulk;              // Effect outer pass: neighbours' h_j rows staged by bulk async copies (pass_h_bulk)
  int grid_mode;           // 0: all resident blocks; 1: the fewest blocks that keep the same atoms per warp
  int block_warps;         // launch shape: warps per block (1 .. kPassWarps; 0 = spread_warps); the kernel
                           // reads its block size from blockDim
  Real* keep;              // [keep_rows][kKeepBatches][2 F + H][32]: R, R', Y per edge (pass_keeps)
  int keep_rows;
};

template <typename Real>
__host__ __device__ inline int pass_table_size(int C, int F, int B, int nblk) {
  return F * B + 2 * nblk * C * C + 3 * C * F;
}
__host__ __device__ constexpr int round4(int n) { return (n + 3) & ~3; }
// Staged edge columns of the forward reduction: column c holds one quantity of the batch's 32 edges
// (u_mu at columns [0, F), Y_h at [F, F + H)), so that a lane writes its edge's values without bank
// conflicts and the reduction reads four edges of a column with one 128-bit access.  The column
// stride is a multiple of 16 bytes and odd in 16-byte units: the 128-bit reads of neighbouring
// columns hit distinct bank groups.
template <typename Real>
__host__ __device__ constexpr int stage_stride() { return sizeof(Real) == 4 ? 36 : 34; }
// Moment items of a lane: harmonic lm (all of l's (2 l + 1) functions are neighbouring lanes) and
// radial channels k = kg + s G, s < slots; G channel groups of H lanes fit in a warp.  A lane's Y
// value serves every channel it owns, and its u columns of one step are G (L + 1) columns apart.
template <int L>
struct MomentItems {
  static constexpr int Lp = L + 1, H = Lp * Lp;
  static constexpr int G = H <= kWarp ? kWarp / H : 1;
  static constexpr int KS = (kMaxK + G - 1) / G;
  static constexpr int kTail = H > kWarp ? H - kWarp : 0;  // harmonics past the warp width: one (k, lm) item a lane
  static_assert(kTail == 0 || kWarp / (kTail ? kTail : 1) >= kMaxK, "tail items");
};
// Slots a pass runs: half of KS when the model's channels fit there (two compiled trip counts).
__host__ __device__ constexpr int moment_slots(int L, int K) {
  const int H = (L + 1) * (L + 1), G = H <= kWarp ? kWarp / H : 1, KS = (kMaxK + G - 1) / G, nk = (K + G - 1) / G;
  return KS >= 2 && nk <= KS / 2 ? KS / 2 : KS;
}
// Staged columns: F + H, and at least those the unused slots of the last channel group reach.
__host__ __device__ constexpr int stage_cols(int L, int K) {
  const int H = (L + 1) * (L + 1), G = H <= kWarp ? kWarp / H : 1;
  const int need = K * (L + 1) + H, reach = moment_slots(L, K) * G * (L + 1);
  return need > reach ? need : reach;
}
// E/F/virial pass tables: radial coefficients [F][B], warp (slope, shift) [2 nblk][C^2], and per
// species pair (t_i, t_j) the products x0(t_i) x1(t_j) and x0(t_i) wadd(t_j) [C^2][F] each.
__host__ __device__ inline int efs_table_size(int C, int F, int B, int nblk) {
  return round4(F * B + 2 * nblk * C * C + 2 * C * C * F);
}
// Per-warp scratch: the staged edge columns, overlaid by the node values v [M + 1] (v[M] = 1, the
// graph program's constant node) and the node adjoints [M + 1] (they live between the forward
// reduction and the per-edge adjoint, when the columns are free); the moment adjoints abar
// [K][round4(H)], hbar [F] and the graph program's partial slots [parts].
template <typename Real>
__host__ __device__ inline int pass_warp_size(int L, int M, int K, int parts) {
  const int H = (L + 1) * (L + 1), stage = stage_cols(L, K) * stage_stride<Real>(), nodes = 2 * (M + 1);
  return round4(round4(stage > nodes ? stage : nodes) + K * round4(H) + K * (L + 1) + parts + 4);
}
// Whether the Effect outer pass can stage the neighbours' gate-signal rows h_j with bulk async
// copies: a row must be a whole number of 16-byte units (the copy's size and alignment rule).
// The host launches the kModeOuterBulk variant only then, and sizes its scratch by the same test.
template <typename Real>
__host__ __device__ constexpr bool h_rows_bulk_ok(int F) {
  return (F * static_cast<int>(sizeof(Real))) % 16 == 0;
}
template <typename Real>
__host__ __device__ inline bool pass_h_bulk(int mode, int flag, int F) {
  return (mode == kModeOuter || mode == kModeOuterBulk) && flag != 0 && h_rows_bulk_ok<Real>(F);
}
// Per-warp scratch with the h_j staging area appended: 32 rows of F (one per lane, 16-byte
// aligned) and the warp's mbarrier (4 values, 16 bytes or more).
template <typename Real>
__host__ __device__ inline int pass_warp_stride(int L, int M, int K, int parts, bool h_bulk) {
  return pass_warp_size<Real>(L, M, K, parts) + (h_bulk ? kWarp * K * (L + 1) + 4 : 0);
}

// Kahan-compensated accumulation for the FP32 bulk form (explicitly rounded steps, never fused
// with the caller's multiplies); plain sums in FP64.
template <typename Real, bool KAHAN>
__device__ __forceinline__ void kadd(Real& s, Real& c, Real x) {
  if constexpr (KAHAN && sizeof(Real) == 4) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  } else if constexpr (KAHAN) {
    const Real y = x - c;
    const Real t = s + y;
    c = (t - s) - y;
    s = t;
  } else {
    s += x;
  }
}

// ---------------------------------------------------------------------------------------------
// Per-edge radial functions of one pass: R_mu and (optionally) dR_mu/dr for all (k, l).
// The warp (slope, shift) depends on (scaling block, t_i, t_j); the Chebyshev part is shared by
// every l of a block and only the envelope differs between l = 0 and l > 0 with two cutoffs.
// ---------------------------------------------------------------------------------------------
// One row of radial coefficients (16-byte aligned when BF > 0: rows of BF = 8 values from an
// aligned table) into registers, with 128-bit loads where the size allows.
template <typename Real, int BF, int NBM>
__device__ __forceinline__ void load_coeff_row(const Real* c, int B, Real (&cc)[NBM]) {
  if constexpr (BF > 0 && sizeof(Real) == 4 && BF % 4 == 0) {
    const float4* c4 = reinterpret_cast<const float4*>(c);
#pragma unroll
    for (int q = 0; q < BF / 4; ++q) {
      const float4 v = c4[q];
      cc[4 * q] = v.x; cc[4 * q + 1] = v.y; cc[4 * q + 2] = v.z; cc[4 * q + 3] = v.w;
    }
  } else if constexpr (BF > 0 && sizeof(Real) == 8 && BF % 2 == 0) {
    const double2* c2 = reinterpret_cast<const double2*>(c);
#pragma unroll
    for (int q = 0; q < BF / 2; ++q) {
      const double2 v = c2[q];
      cc[2 * q] = v.x; cc[2 * q + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int b = 0; b < NBM; ++b) cc[b] = b < B ? c[b] : Real(0);
  }
}

// One edge's inputs: the record (d, r), the neighbour and its species.
template <typename Real>
struct EdgeIn {
  typename Vec4<Real>::type d;
  int j, tj;
};
// (species indices are clamped to [0, C): an index out of range, which the edge build or the
// caller-edge checks report, must not reach the per-species tables within the same step)
__device__ __forceinline__ int species_of(const int* types, int i, int C) { return min(max(types[i], 0), C - 1); }

template <typename Real>
__device__ __forceinline__ EdgeIn<Real> load_edge(const typename Vec4<Real>::type* d4, const int* nbr,
                                                  const int* types, int e, int C) {
  EdgeIn<Real> x;
  x.d = d4[e];
  x.j = nbr[e];
  // one species: no neighbour-type load (it would wait on the neighbour index just loaded)
  x.tj = C == 1 ? 0 : species_of(types, x.j, C);
  return x;
}

// Rows of a per-atom or per-edge array [.][F] against the staged columns of a batch's nb edges: row
// index r of lane q's edge <-> column entries stage[mu * stride + q].  Eight edges by four 16-byte
// units per access: each row's 64 consecutive bytes are whole sectors, where one row per lane
// would touch 32 lines per access and write half sectors.  Rows that are not whole 16-byte units
// go value by value, one row per lane.
template <typename Real>
struct RowUnit { using type = typename std::conditional<sizeof(Real) == 4, float4, double2>::type; };
template <typename Real>
__device__ __forceinline__ void rows_to_cols(Real* stage, const Real* rows, int F, int r, int nb, int lane) {
  constexpr int V = 16 / sizeof(Real), S = stage_stride<Real>();
  using W = typename RowUnit<Real>::type;
  if (F % V == 0) {
    const int nc = F / V, q8 = lane & 7;
    const W* src[4];
#pragma unroll
    for (int qb = 0; qb < 4; ++qb)
      src[qb] = reinterpret_cast<const W*>(rows + static_cast<size_t>(__shfl_sync(0xffffffffu, r, 8 * qb + q8)) * F);
    for (int c = lane >> 3; c < nc; c += 4) {
      W w[4];
#pragma unroll
      for (int qb = 0; qb < 4; ++qb)
        if (8 * qb + q8 < nb) w[qb] = src[qb][c];
#pragma unroll
      for (int qb = 0; qb < 4; ++qb)
        if (8 * qb + q8 < nb) {
          Real* d = stage + V * c * S + 8 * qb + q8;
          d[0] = w[qb].x;
          d[S] = w[qb].y;
          if constexpr (V == 4) { d[2 * S] = w[qb].z; d[3 * S] = w[qb].w; }
        }
    }
  } else if (lane < nb) {
    for (int mu = 0; mu < F; ++mu) stage[mu * S + lane] = rows[static_cast<size_t>(r) * F + mu];
  }
  __syncwarp();
}
template <typename Real>
__device__ __forceinline__ void cols_to_rows(Real* rows, const Real* stage, int F, int r, int nb, int lane) {
  constexpr int V = 16 / sizeof(Real), S = stage_stride<Real>();
  using W = typename RowUnit<Real>::type;
  __syncwarp();
  if (F % V == 0) {
    const int nc = F / V, q8 = lane & 7;
    W* dst[4];
#pragma unroll
    for (int qb = 0; qb < 4; ++qb)
      dst[qb] = reinterpret_cast<W*>(rows + static_cast<size_t>(__shfl_sync(0xffffffffu, r, 8 * qb + q8)) * F);
    for (int c = lane >> 3; c < nc; c += 4) {
#pragma unroll
      for (int qb = 0; qb < 4; ++qb)
        if (8 * qb + q8 < nb) {
          const Real* d = stage + V * c * S + 8 * qb + q8;
          W w;
          w.x = d[0];
          w.y = d[S];
          if constexpr (V == 4) { w.z = d[2 * S]; w.w = d[3 * S]; }
          dst[qb][c] = w;
        }
    }
  } else if (lane < nb) {
    for (int mu = 0; mu < F; ++mu) rows[static_cast<size_t>(r) * F + mu] = stage[mu * S + lane];
  }
  __syncwarp();
}

// The F columns of a row-major per-edge array [n][F] summed over the rows: 32 / W groups of
// W = F / 4 lanes take the rows in turn, a lane reading one 16-byte unit of its row, four rows in
// flight; the groups' sums are added in group order.  put(c, t) on lane c < W receives columns
// 4 c .. 4 c + 3.  For rows of whole units (row_groups_ok).  Bound by the rows' latency; a lane summing two
// columns row after row (column_sums_2) took the fused gate reverse pass 31.3 us, this 28.5 (Effect L3/K4,
// 1,400 atoms).
__host__ __device__ constexpr bool row_groups_ok(int F) { return F % 4 == 0 && F / 4 <= kWarp; }
template <typename Put>
__device__ __forceinline__ void row_group_sums(const float* rows, int F, int n, int lane, Put&& put) {
  const int nc = F / 4, groups = kWarp / nc, grp = lane / nc, c = lane - grp * nc;
  const float4* src = reinterpret_cast<const float4*>(rows) + c;
  float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
  if (grp < groups) {
    for (int e = grp; e < n; e += 4 * groups) {
      float4 w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e + u * groups < n) w[u] = src[static_cast<size_t>(e + u * groups) * nc];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e + u * groups < n) { t.x += w[u].x; t.y += w[u].y; t.z += w[u].z; t.w += w[u].w; }
    }
  }
  const float4 own = t;
  for (int q = 1; q < groups; ++q) {
    const int from = min(lane + q * nc, kWarp - 1);
    t.x += __shfl_sync(0xffffffffu, own.x, from);
    t.y += __shfl_sync(0xffffffffu, own.y, from);
    t.z += __shfl_sync(0xffffffffu, own.z, from);
    t.w += __shfl_sync(0xffffffffu, own.w, from);
  }
  if (lane < nc) put(c, t);
}

// Four consecutive values of a 16-byte aligned shared-memory column as two pairs.
template <typename Real>
__device__ __forceinline__ void load_quad(const Real* p, Pair<Real>& a, Pair<Real>& b) {
  if constexpr (sizeof(Real) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = {v.x, v.y};
    b = {v.z, v.w};
  } else {
    const double2 v = reinterpret_cast<const double2*>(p)[0], w = reinterpret_cast<const double2*>(p)[1];
    a = {v.x, v.y};
    b = {w.x, w.y};
  }
}

// Edge->moment sums of one staged batch: part[s] = sum_q u[q][k_s, l] Y[q][lm] over the batch's
// edges (rounded up to four: the entries past nb are zero), even and odd edges in the two halves.
// Per four edges a lane reads Y once and one u column per channel, 128 bits each, and issues two
// packed multiply-adds per channel.
template <int NS, int STEP, int TAIL, typename Real, int N>
__device__ __forceinline__ void moment_batch(const Real* u, const Real* y, const Real* ut, const Real* yt, int nb,
                                             Pair<Real> (&part)[N]) {
#pragma unroll
  for (int s = 0; s < N; ++s) part[s] = {Real(0), Real(0)};
#pragma unroll 2
  for (int q = 0; q < nb; q += 4) {
    Pair<Real> y0, y1, u0, u1;
    load_quad(y + q, y0, y1);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      load_quad(u + s * STEP + q, u0, u1);
      part[s] = fma2(u0, y0, part[s]);
      part[s] = fma2(u1, y1, part[s]);
    }
    if constexpr (TAIL) {
      load_quad(yt + q, y0, y1);
      load_quad(ut + q, u0, u1);
      part[N - 1] = fma2(u0, y0, part[N - 1]);
      part[N - 1] = fma2(u1, y1, part[N - 1]);
    }
  }
}

// Envelopes of an edge's l = 0 and l > 0 functions, times the model's scaling.
template <typename Real>
struct Envelopes { Real f0, fd0, f1, fd1; };
template <typename Real>
__device__ __forceinline__ Envelopes<Real> edge_envelopes(const DevModel<Real>& dm, Real r) {
  Envelopes<Real> e;
  envelope<Real>(r, dm.rmax, dm.poly, dm.cutoff_p, e.f0, e.fd0);
  if (dm.split) envelope<Real>(r, dm.rang, dm.poly, dm.cutoff_p, e.f1, e.fd1);
  else { e.f1 = e.f0; e.fd1 = e.fd0; }
  e.f0 *= dm.scaling; e.fd0 *= dm.scaling; e.f1 *= dm.scaling; e.fd1 *= dm.scaling;
  return e;
}

// Chebyshev values T_b(xi) and derivatives D_b = dT_b / dxi (DERIV) of one warp as pairs over b.
template <typename Real, int NP, bool DERIV>
__device__ __forceinline__ void cheb_pairs(Real xi, int B, Pair<Real> (&T)[NP], Pair<Real> (&D)[NP]) {
  Real t2 = Real(1), t1 = xi, d2 = Real(0), d1 = Real(1);
  const Real x2 = xi + xi;
  T[0] = {t2, t1};
  D[0] = {d2, d1};
#pragma unroll
  for (int b = 2; b < 2 * NP; ++b) {
    Real t = Real(0), d = Real(0);
    if (b < B) {
      t = x2 * t1 - t2;
      if (DERIV) d = Real(2) * t1 + (x2 * d1 - d2);
      t2 = t1; t1 = t;
      d2 = d1; d1 = d;
    }
    if (b & 1) { T[b / 2].y = t; D[b / 2].y = d; }
    else { T[b / 2].x = t; D[b / 2].x = d; }
  }
}

// sum_b c_b T_b and sum_b c_b D_b of one radial function: the even and odd terms are the halves of
// the packed sums.
template <typename Real, int BF, int NP, bool DERIV>
__device__ __forceinline__ void cheb_dot(const Real* c, int B, const Pair<Real> (&T)[NP], const Pair<Real> (&D)[NP],
                                         Real& a, Real& ad) {
  Real cc[2 * NP];
  load_coeff_row<Real, BF, 2 * NP>(c, B, cc);
  // (T_0 = 1, D_0 = 0 and D_1 = 1 need no product)
  Pair<Real> sa{cc[0], cc[1] * T[0].y}, sd{Real(0), cc[1]};
#pragma unroll
  for (int p = 1; p < NP; ++p) {
    if (2 * p < B) {
      sa = fma2(Pair<Real>{cc[2 * p], cc[2 * p + 1]}, T[p], sa);
      if (DERIV) sd = fma2(Pair<Real>{cc[2 * p], cc[2 * p + 1]}, D[p], sd);
    }
  }
  a = sa.x + sa.y;
  ad = sd.x + sd.y;
}

// The radial functions R_mu (and dR_mu/dr) of channel k for every l.  Beyond a cutoff the envelope
// and its slope are exactly zero, so the l > 0 functions of a two-cutoff model vanish by themselves
// outside the angular cutoff.  The warp is shared by the l of a channel unless the model's scaling
// map gives each l its own (then a rolled loop: one copy of the warp's code).
template <int L, typename Real, bool DERIV, int BF>
__device__ __forceinline__ void radial_channel(const DevModel<Real>& dm, const Real* s_coeff, const Real* s_scal,
                                               int pair, Real r, const Envelopes<Real>& env, int k, Real (&R)[L + 1],
                                               Real (&Rd)[L + 1]) {
  constexpr int Lp = L + 1, NP = ((BF ? BF : kMaxB) + 1) / 2;
  const int B = BF ? BF : dm.B, C2 = dm.C * dm.C;
  Pair<Real> T[NP], D[NP];
  auto warp = [&](int sb) {
    const Real slope = s_scal[2 * sb * C2 + pair], shift = s_scal[(2 * sb + 1) * C2 + pair];
    const Real xi = tanh(slope * (r - shift) * Real(0.5));
    cheb_pairs<Real, NP, DERIV>(xi, B, T, D);
    return (Real(1) - xi * xi) * slope * Real(0.5);  // dxi / dr
  };
  if (dm.scaling_mode == 2 || dm.scaling_mode == 0) {
    const Real xr = warp(scaling_block(dm.scaling_mode, k, 0, Lp));
    const Real fx0 = env.f0 * xr, fx1 = env.f1 * xr;
#pragma unroll
    for (int l = 0; l < Lp; ++l) {
      Real a, ad;
      cheb_dot<Real, BF, NP, DERIV>(s_coeff + (k * Lp + l) * B, B, T, D, a, ad);
      R[l] = (l == 0 ? env.f0 : env.f1) * a;
      if (DERIV) Rd[l] = (l == 0 ? env.fd0 : env.fd1) * a + (l == 0 ? fx0 : fx1) * ad;
    }
  } else {
#pragma unroll 1
    for (int l = 0; l < Lp; ++l) {
      const Real xr = warp(scaling_block(dm.scaling_mode, k, l, Lp));
      Real a, ad;
      cheb_dot<Real, BF, NP, DERIV>(s_coeff + (k * Lp + l) * B, B, T, D, a, ad);
      const Real f = l == 0 ? env.f0 : env.f1, fd = l == 0 ? env.fd0 : env.fd1;
      const Real v = f * a, vd = fd * a + f * xr * ad;
#pragma unroll
      for (int q = 0; q < Lp; ++q)
        if (q == l) {
          R[q] = v;
          if (DERIV) Rd[q] = vd;
        }
    }
  }
}

// Steps [s0, s1) of a pass's graph program (GraphProg, device_common.cuh) on the warp's node
// arrays: forward steps add into v, reverse steps into adj (DIR 1 / 2: the range holds forward /
// reverse steps only).  Each lane runs its term stream (one
// coalesced row per term), adding chunk sums to their target node or partial slot at the chunk's
// last term; then the lanes combine the partial slots of lists that were cut into several chunks.
template <typename Real, int DIR = 0>
__device__ __forceinline__ void run_prog(const GraphProg<Real>& g, int s0, int s1, Real* v, Real* adj, Real* parts,
                                         int lane) {
  for (int st = s0; st < s1; ++st) {
    const int4 info = g.steps[st];
    const bool rev = DIR == 2 || (DIR == 0 && (info.w & 1));
    Real* T = rev ? adj : v;
    const Real* X = rev ? adj : v;
    const ProgRec<Real>* r = g.rows + static_cast<size_t>(info.x) * kWarp + lane;
    Real acc = Real(0);
#pragma unroll 4
    for (int i = 0; i < info.y; ++i) {
      const ProgRec<Real> p = load_rec<Real>(r + static_cast<size_t>(i) * kWarp);
      acc += p.c * X[p.ab & 0xffffu] * v[p.ab >> 16];
      if (p.flush != kProgNoFlush) {
        if (p.flush >= 0) T[p.flush] += acc;
        else parts[-p.flush - 2] = acc;
        acc = Real(0);
      }
    }
    const int comb_end = info.w >> 1;
    if (comb_end > info.z) {
      __syncwarp();
      for (int q = info.z + lane; q < comb_end; q += kWarp) {
        const int4 e = g.comb[q];
        Real s = Real(0);
        for (int p = e.y; p < e.z; ++p) s += parts[p];
        T[e.x] += s;
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// Edge->moment batch sums on the tensor cores (FP32 engines, optional): the batch's staged rows
// form the products D[mu][lm] = sum_q u[q][mu] Y[q][lm] (q < 32 edges), computed as m16n8k8 TF32
// mma.sync tiles with each operand split into a TF32 head and a TF32 tail (3xTF32: head*head +
// head*tail + tail*head, about FP32 accuracy); the entries with l(mu) = l(lm) are the moment
// partials, written to part[k][lm].  Edges past the batch are zero; tile columns past F / H repeat the
// last one and are discarded.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned tf32_head(float x) {
  unsigned h;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
  return h;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
template <int L>
__device__ __forceinline__ void moments_mma_batch(const float* stage, int F, float* part, int lane) {
  constexpr int Lp = L + 1, H = Lp * Lp, S = stage_stride<float>();
  const int g = lane >> 2, t = lane & 3;
  const int mtiles = (F + 15) / 16;
  constexpr int ntiles = (H + 7) / 8;
  for (int mt = 0; mt < mtiles; ++mt) {
#pragma unroll
    for (int nt = 0; nt < ntiles; ++nt) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ks = 0; ks < kWarp / 8; ++ks) {
        const float* a0 = stage + min(16 * mt + g, F - 1) * S + 8 * ks + t;
        const float* a1 = stage + min(16 * mt + g + 8, F - 1) * S + 8 * ks + t;
        const float* b0 = stage + (F + min(8 * nt + g, H - 1)) * S + 8 * ks + t;
        const float av[4] = {a0[0], a1[0], a0[4], a1[4]};
        const float bv[2] = {b0[0], b0[4]};
        unsigned ah[4], al[4], bh[2], bl[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          ah[i] = tf32_head(av[i]);
          al[i] = tf32_head(av[i] - __uint_as_float(ah[i]));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          bh[i] = tf32_head(bv[i]);
          bl[i] = tf32_head(bv[i] - __uint_as_float(bh[i]));
        }
        mma_tf32(d, al, bh);
        mma_tf32(d, ah, bl);
        mma_tf32(d, ah, bh);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int mu = 16 * mt + g + 8 * (i >> 1), lm = 8 * nt + 2 * t + (i & 1);
        if (mu < F && lm < H) {
          int l = 0;
          while ((l + 1) * (l + 1) <= lm) ++l;
          if (mu % Lp == l) part[(mu / Lp) * H + lm] = d[i];
        }
      }
    }
  }
  __syncwarp();
}

// Readout of one centre and the adjoint seeds: E_i = species + shift + coef sum_q linear_q
// v[map q] into a.site_energy (the sum in compensated FP32 with exact products for the FP32 bulk
// form, FP64 otherwise), the scalar moments into a.desc when requested, adj zeroed and seeded with
// coef linear in Real (the reference's readout, sus2_sl_kernel.cpp:556).
template <typename Real>
__device__ __forceinline__ void readout_seeds(const PassArgs<Real>& a, int atom, int ti, const Real* v, Real* adj,
                                              int lane) {
  const DevModel<Real>& dm = a.dm;
  const int M = dm.M;
  const double coef = dm.species_readout ? 1.0 : dm.species[ti];
  const Real coef_r = Real(coef);
  const int off = dm.species_readout ? ti * dm.S : 0;
  for (int q = lane; q <= M; q += kWarp) adj[q] = Real(0);
  __syncwarp();
  double es64 = 0.0;
  float ehi = 0.f, elo = 0.f;
  for (int q = lane; q < dm.S; q += kWarp) {
    const int node = dm.scalar_map[q];
    const Real lin = dm.linear[off + q], vv = v[node];
    if (sizeof(Real) == 4) csum_add_prod(ehi, elo, float(lin), float(vv));
    else es64 += double(lin) * double(vv);
    adj[node] = coef_r * lin;
    if (a.desc) a.desc[static_cast<size_t>(atom) * dm.S + q] = double(vv);
  }
  const double es = sizeof(Real) == 4 ? warp_csum(ehi, elo) : warp_sum(es64);
  if (lane == 0) a.site_energy[atom] = dm.species[ti] + dm.shift[ti] + coef * es;
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// The pass kernel.
// ---------------------------------------------------------------------------------------------
constexpr int kPassWarps = 4;
// FP64: the forward keeps R, R' and Y of a centre's first kKeepBatches batches of 32 edges for its
// adjoint -- the fused Static and outer passes in rows of the resident warps (they stay in L2), the
// gate passes, two kernels, in rows of the centres.  The FP64 pipe is busy 85% of those passes, and
// most of that is the radial functions: Static L3/K4/O2, 4,096 atoms 1,099 -> 752 us.  (FP32 passes
// gain nothing: 57 -> 64 us; their recomputation is cheaper than the traffic.)
constexpr int kKeepBatches = 4;
template <typename Real>
__host__ __device__ constexpr bool pass_keeps(int mode) {
  return sizeof(Real) == 8 && (mode == kModeStatic || mode == kModeOuter || mode == kModeOuterBulk ||
                               mode == kModeGateForward || mode == kModeGateReverse);
}
__host__ __device__ inline size_t pass_keep_values(int L, int F) {
  return static_cast<size_t>(kKeepBatches) * (2 * F + (L + 1) * (L + 1)) * kWarp;
}
// Minimum resident blocks per SM (the register budget: 4 blocks = 128 registers, 3 = 168).  Both
// budgets are compiled for the B = 8 passes and the engine's autotuner times them on the caller's
// layout; without tuning: 4 for the FP32 kernels up to L = 3 and the L = 4 gate passes, 3
// otherwise (measured: the L = 4 outer pass spills and runs slower at 128 registers; the FP64
// kernels spill more).
__host__ __device__ constexpr int default_min_blocks(int L, bool fp32, int mode) {
  return (fp32 && (L <= 3 || (L == 4 && mode != kModeOuter && mode != kModeOuterBulk))) ? 4 : 3;
}

template <int L, typename Real, int MODE, bool KAHAN, int BF, int MINB>
__global__ void __launch_bounds__(kPassWarps * kWarp, MINB) atom_pass_kernel(PassArgs<Real> a) {
  constexpr int Lp = L + 1, H = Lp * Lp, H4 = round4(H), NPH = (H + 1) / 2;
  constexpr int S = stage_stride<Real>();
  using MI = MomentItems<L>;
  constexpr int NS = MI::KS + (MI::kTail ? 1 : 0);  // moment item slots of a lane
  using V4 = typename Vec4<Real>::type;
  const DevModel<Real>& dm = a.dm;
  const bool gate_pass = MODE == kModeGateForward || MODE == kModeGateReverse || MODE == kModeGateFwdEdges ||
                         MODE == kModeGateRevEdges;
  // the gate reverse pass adds its edge gradients and virials to the outer pass's
  constexpr bool kGateRev = MODE == kModeGateReverse || MODE == kModeGateRevEdges;
  const PassTables<Real>& pt = gate_pass ? dm.gate : dm.outer;
  const int C = dm.C, F = dm.F, B = BF ? BF : dm.B, K = dm.K, M = dm.M, NB = dm.NB;
  const int warps = blockDim.x / kWarp, warp = threadIdx.x / kWarp, lane = warp_lane();
  // Effect outer pass, bulk variant: the neighbours' h_j rows of a 32-edge batch are brought into
  // hbuf by bulk async copies (one row per lane), issued while the batch before is still being
  // worked on (a constant false in every other variant)
  constexpr bool kBulk = MODE == kModeOuterBulk;
  const bool hb_on = kBulk && h_rows_bulk_ok<Real>(F);

  extern __shared__ __align__(16) unsigned char smem_raw[];
  Real* sm = reinterpret_cast<Real*>(smem_raw);
  Real* s_coeff = sm;
  Real* s_scal = s_coeff + F * B;
  Real* s_pw = s_scal + 2 * dm.nblk * C * C;        // [C^2][F] x0(t_i) x1(t_j)
  Real* s_pa = s_pw + C * C * F;                    // [C^2][F] x0(t_i) wadd(t_j)
  const int wsize = pass_warp_size<Real>(L, M, K, dm.prog_parts);
  Real* wbase = sm + efs_table_size(C, F, B, dm.nblk) + pass_warp_stride<Real>(L, M, K, dm.prog_parts, hb_on) * warp;
  Real* stage = wbase;                              // columns [F + H][S]: u_mu, then Y_h
  Real* v = wbase;                                  // [M + 1], v[M] = 1 (over the free columns)
  Real* adj = v + M + 1;                            // [M + 1]
  Real* abar = wbase + round4(max(stage_cols(L, K) * S, 2 * (M + 1)));  // [K][H4]
  Real* hbar = abar + K * H4;                       // [F]
  Real* parts = hbar + F;                           // [prog_parts]
  Real* hbuf = wbase + wsize;                       // [32][F] h_j rows of one batch (hb_on)
  unsigned long long* hb_bar = reinterpret_cast<unsigned long long*>(hbuf + kWarp * F);

  // the next kernel may be scheduled as soon as every block has started; the model tables staged
  // here are written only by host uploads, which completed before the launch chain began, so
  // they are read before the wait for the previous kernel's edges and signals
  pdl_launch_dependents();
  for (int q = threadIdx.x; q < F * B; q += blockDim.x) s_coeff[q] = pt.coeff[q];
  for (int q = threadIdx.x; q < 2 * dm.nblk * C * C; q += blockDim.x) s_scal[q] = pt.scal[q];
  for (int q = threadIdx.x; q < C * C * F; q += blockDim.x) {
    const int pair = q / F, mu = q - pair * F, ti = pair / C, tj = pair - ti * C;
    const Real x0 = pt.wcenter[ti * F + mu];
    s_pw[q] = x0 * pt.wsource[tj * F + mu];
    s_pa[q] = pt.wadd ? x0 * pt.wadd[tj * F + mu] : Real(0);
  }
  __syncthreads();
  pdl_wait();
  const bool effect_outer = MODE == kModeOuter || MODE == kModeOuterBulk || MODE == kModeOuterFwd || MODE == kModeOuterRev;
  // the two per-edge kernels of a split pass: forward only (moments out), adjoint only (moment
  // adjoints in)
  constexpr bool kFwdOnly = MODE == kModeStaticFwd || MODE == kModeOuterFwd || MODE == kModeGateFwdEdges;
  constexpr bool kRevOnly = MODE == kModeStaticRev || MODE == kModeOuterRev || MODE == kModeGateRevEdges;
  // the h_j copies of a batch: lane 0 orders the warp's reads of hbuf before the async writes and
  // announces the bytes, every lane with an edge copies its row; the caller has synchronised the
  // warp after its last reads of hbuf
  unsigned hb_parity = 0;
  if (hb_on) {
    if (lane == 0) mbar_init(hb_bar, 1);
    __syncwarp();
  }
  auto hb_issue = [&](bool has_edge, int j, int nedges) {
    if (lane == 0) {
      fence_proxy_async_smem();
      mbar_arrive_expect(hb_bar, static_cast<unsigned>(nedges * F * sizeof(Real)));
    }
    __syncwarp();
    if (has_edge) bulk_copy_g2s(hbuf + lane * F, a.hsig + (size_t)j * F, F * sizeof(Real), hb_bar);
  };
  // waits for the batch's rows; on a copy that does not complete (bounded wait) records the error,
  // waits once more for the copies in flight and returns false: the warp then leaves the kernel
  auto hb_arrived = [&]() {
    const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(hb_bar, hb_parity));
    if (!ok) {
      if (lane == 0) record_error(a.error, kErrAsyncCopy);
      mbar_wait_bounded(hb_bar, hb_parity);
    }
    hb_parity ^= 1u;
    return ok;
  };

  // the lane's moment items (MomentItems): slot q < KS is (k = kg + q G, lm), the tail slot of L = 5
  // is (kt, lmt); item_of gives the slot's index k H + lm, -1 when it is none of the model's
  const bool item_on = lane < MI::G * H;
  const int lm = H <= kWarp ? (item_on ? lane % H : 0) : lane, kg = H <= kWarp && item_on ? lane / H : 0;
  auto l_of = [](int h) {
    int l = 0;
#pragma unroll
    for (int q = 1; q < Lp; ++q) l += h >= q * q;
    return l;
  };
  const Real* col_u = stage + (kg * Lp + l_of(lm)) * S;
  const Real* col_y = stage + (F + lm) * S;
  constexpr int TW = MI::kTail ? MI::kTail : 1;
  const int lmt = kWarp + lane % TW, kt = lane / TW;
  const Real* col_ut = stage + (min(kt, K - 1) * Lp + L) * S;
  const Real* col_yt = stage + (F + lmt) * S;
  auto item_of = [&](int q) {
    if (MI::kTail && q == MI::KS) return kt < K ? kt * H + lmt : -1;
    const int k = kg + q * MI::G;
    return (H > kWarp || item_on) && k < K ? k * H + lm : -1;
  };
  const bool half_slots = MI::KS >= 2 && moment_slots(L, K) < MI::KS;

  // centres of this warp: grid-strided, one contiguous run (neighbouring centres share their
  // neighbours' rows in L1), or taken one at a time from a device counter
  const int gwarp = blockIdx.x * warps + warp, nwarps = gridDim.x * warps;
  const int per_warp = (a.natoms + nwarps - 1) / nwarps;
  const bool dynamic = a.atom_order == 2;
  auto grab = [&]() {
    int x = 0;
    if (lane == 0) x = atomicAdd(a.work, 1);
    return __shfl_sync(0xffffffffu, x, 0);
  };
  const int atom_first = dynamic ? grab() : (a.atom_order ? gwarp * per_warp : gwarp);
  const int atom_stop = a.atom_order == 1 ? min(a.natoms, atom_first + per_warp) : a.natoms;
  const int atom_step = a.atom_order == 1 ? 1 : nwarps;
  // the dynamic order's reset: every warp counts itself done after its last take (ordered after
  // it by the fence), and the last one zeroes the pair, when no take of this launch is pending
  auto finish_dynamic = [&]() {
    if (dynamic && lane == 0) {
      __threadfence();
      if (atomicAdd(a.work + 1, 1) == nwarps - 1) {
        atomicExch(a.work, 0);
        atomicExch(a.work + 1, 0);
      }
    }
  };
  for (int atom = atom_first; atom < atom_stop; atom = dynamic ? grab() : atom + atom_step) {
    const int ti = C == 1 ? 0 : species_of(a.types, atom, C);
    const int e0 = a.row[atom], e1 = a.row_end[atom];
    // the kept functions, a lane per column (batches past keep_batches evaluate them again)
    constexpr bool kKeep = pass_keeps<Real>(MODE);
    const int keep_row = gate_pass ? atom : blockIdx.x * warps + warp;
    const int keep_batches = kKeep && keep_row < a.keep_rows ? kKeepBatches : 0;
    Real* kept = kKeep ? a.keep + static_cast<size_t>(keep_row) * pass_keep_values(L, F) + lane : nullptr;
    // per-atom virial: FP64 for the FP64 form; compensated FP32 (hi, lo) for the FP32 bulk form
    double vir[6] = {0, 0, 0, 0, 0, 0};
    float vhi[6] = {0, 0, 0, 0, 0, 0}, vlo[6] = {0, 0, 0, 0, 0, 0};

    // edge inputs of the lane's edge in the last batch: left by the forward loop, which the
    // per-edge adjoint then starts from (it runs the batches in reverse order)
    EdgeIn<Real> cur{};
    const int nbat = (e1 - e0 + kWarp - 1) / kWarp;
    // the gate reverse pass starts with the per-atom work: its first edge batch loads meanwhile
    if ((MODE == kModeGateReverse || kRevOnly) && nbat > 0 && e0 + (nbat - 1) * kWarp + lane < e1)
      cur = load_edge<Real>(a.d4, a.nbr, a.types, e0 + (nbat - 1) * kWarp + lane, C);
    if (kRevOnly) {
      // ---------------- split pass, per-edge part: adjoint moments from the graph kernel ----------
      for (int t = lane; t < K * H; t += kWarp) abar[t / H * H4 + t % H] = a.amom[static_cast<size_t>(atom) * (K * H) + t];
      __syncwarp();
    } else if (MODE != kModeGateReverse) {
      // ---------------- forward moments ----------------
      Real acc[NS], cmp[NS];
#pragma unroll
      for (int q = 0; q < NS; ++q) { acc[q] = Real(0); cmp[q] = Real(0); }
      // the next batch's edge inputs are loaded while the current batch is evaluated
      if (e0 + lane < e1) cur = load_edge<Real>(a.d4, a.nbr, a.types, e0 + lane, C);
      if (hb_on && nbat > 0) hb_issue(e0 + lane < e1, cur.j, min(kWarp, e1 - e0));
      for (int base = e0; base < e1; base += kWarp) {
        const int e = base + lane, nb = min(kWarp, e1 - base);
        const bool more = base + kWarp < e1;
        EdgeIn<Real> nxt = cur;
        if (more && e + kWarp < e1) nxt = load_edge<Real>(a.d4, a.nbr, a.types, e + kWarp, C);
        if (hb_on && !hb_arrived()) return;
        // Effect: the neighbours' gate signals h_j, from the bulk-copied batch rows or brought into
        // the u columns (each value read once before its u_mu overwrites it)
        if (effect_outer && !hb_on) rows_to_cols<Real>(stage, a.hsig, F, cur.j, nb, lane);
        Real* col = stage + lane;
        const int kb = (base - e0) / kWarp;
        const bool keep = kKeep && kb < keep_batches;
        Real* kq = kKeep ? kept + static_cast<size_t>(kb) * (2 * F + H) * kWarp : nullptr;
        if (e < e1) {
          const V4 dv = cur.d;
          const Real r = dv.w, ir = Real(1) / r;
          {
            Real Y[H];
            sph_values<L, Real>(dv.x * ir, dv.y * ir, dv.z * ir, Y);
            // (with two cutoffs the l > 0 functions beyond the angular one meet u = 0)
#pragma unroll
            for (int h = 0; h < H; ++h) {
              col[(F + h) * S] = Y[h];
              if (kKeep && keep) kq[(2 * F + h) * kWarp] = Y[h];
            }
          }
          const int pair = ti * C + cur.tj;
          const Real* pw = s_pw + pair * F;
          const Real* pa = s_pa + pair * F;
          const Real* hj = hbuf + lane * F;
          const Envelopes<Real> env = edge_envelopes<Real>(dm, r);
#pragma unroll 1
          for (int k = 0; k < K; ++k) {
            Real R[Lp], Rd[Lp];
            if (!keep) radial_channel<L, Real, false, BF>(dm, s_coeff, s_scal, pair, r, env, k, R, Rd);
            Real* ck = col + k * Lp * S;
            if (kKeep && keep) {
              radial_channel<L, Real, true, BF>(dm, s_coeff, s_scal, pair, r, env, k, R, Rd);
#pragma unroll
              for (int l = 0; l < Lp; ++l) {
                kq[(k * Lp + l) * kWarp] = R[l];
                kq[(F + k * Lp + l) * kWarp] = Rd[l];
              }
            }
#pragma unroll
            for (int l = 0; l < Lp; ++l) {
              Real w = pw[k * Lp + l];
              if (effect_outer) w += pa[k * Lp + l] * (hb_on ? hj[k * Lp + l] : ck[l * S]);
              ck[l * S] = w * R[l];
            }
          }
        } else {
          for (int q = 0; q < F + H; ++q) col[q * S] = Real(0);
        }
        __syncwarp();
        // the next batch's h_j rows travel while this batch is reduced
        if (hb_on && more) hb_issue(e + kWarp < e1, nxt.j, min(kWarp, e1 - base - kWarp));
        // plain sums over the batch's (<= 32) staged edges, then a compensated add of the batch
        // partial into the atom's running moment
        Pair<Real> part[NS];
        if (sizeof(Real) == 4 && a.moment_mma) {
          // tensor-core batch sums into the abar rows (free until the reverse), then each lane
          // reads its items
          moments_mma_batch<L>(reinterpret_cast<const float*>(stage), F, reinterpret_cast<float*>(abar), lane);
#pragma unroll
          for (int q = 0; q < NS; ++q) part[q] = {item_of(q) >= 0 ? abar[item_of(q)] : Real(0), Real(0)};
        } else if (half_slots) {
          moment_batch<MI::KS >= 2 ? MI::KS / 2 : MI::KS, MI::G * Lp * S, MI::kTail>(col_u, col_y, col_ut, col_yt, nb, part);
        } else {
          moment_batch<MI::KS, MI::G * Lp * S, MI::kTail>(col_u, col_y, col_ut, col_yt, nb, part);
        }
#pragma unroll
        for (int q = 0; q < NS; ++q) kadd<Real, KAHAN>(acc[q], cmp[q], part[q].x + part[q].y);
        __syncwarp();
        if (more) cur = nxt;
      }
      if (kFwdOnly) {
        // split pass, forward part: the moments go to the graph kernel
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          const int t = item_of(q);
          if (t >= 0) a.mom[static_cast<size_t>(atom) * (K * H) + t] = acc[q];
        }
        continue;
      }
      for (int q = lane; q <= M; q += kWarp) v[q] = q < M ? Real(0) : Real(1);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        const int t = item_of(q);
        if (t >= 0) {
          const int b = dm.basic_of[t];
          if (b >= 0) v[b] = acc[q];
        }
      }
      __syncwarp();
      run_prog<Real, 1>(pt.prog, 0, pt.prog.nfwd, v, adj, parts, lane);

      if (MODE == kModeGateForward) {
        for (int q = lane; q < M; q += kWarp) a.gmom[(size_t)atom * M + q] = v[q];
        // the gate scalars gathered once into the (here unused) hbar row when they fit, so that
        // each signal's sum reads its weights and the scalars without a node-index load between
        const bool staged = dm.Q <= F;
        if (staged)
          for (int q = lane; q < dm.Q; q += kWarp) hbar[q] = v[dm.gate_nodes[q]];
        __syncwarp();
        for (int mu = lane; mu < F; mu += kWarp) {
          Real h = Real(0);
          for (int q = 0; q < dm.Q; ++q)
            h += dm.gate_wmat_t[q * F + mu] * (staged ? hbar[q] : v[dm.gate_nodes[q]]);
          a.hsig[(size_t)atom * F + mu] = h;
        }
        __syncwarp();
        continue;
      }

      // ---------------- readout and seeds ----------------
      readout_seeds<Real>(a, atom, ti, v, adj, lane);
    } else {
      // ---------------- gate reverse: gather hbar, project, load gate values ----------------
      if (sizeof(Real) == 4 && !a.hbar_atom && row_groups_ok(F)) {  // in the split pass's order (hbar_sum_kernel)
        row_group_sums(reinterpret_cast<const float*>(a.hcontrib + (size_t)e0 * F), F, e1 - e0, lane,
                       [&](int c, float4 t) { reinterpret_cast<float4*>(hbar)[c] = t; });
      } else if (!a.hbar_atom && F <= 2 * kWarp) {
        column_sums_2<Real>(a.hcontrib + (size_t)e0 * F, F, e1 - e0, hbar, lane);
      } else {
        for (int mu = lane; mu < F; mu += kWarp) {
          if (a.hbar_atom) {
            hbar[mu] = Real(a.hbar_atom[(size_t)atom * F + mu]);
          } else {
            hbar[mu] = column_sum<Real>(a.hcontrib + (size_t)e0 * F + mu, F, e1 - e0);
          }
        }
      }
      for (int q = lane; q <= M; q += kWarp) {
        v[q] = q < M ? a.gmom[(size_t)atom * M + q] : Real(1);
        adj[q] = Real(0);
      }
      __syncwarp();
      for (int q = lane; q < dm.Q; q += kWarp) {
        Real s = Real(0);
        for (int mu = 0; mu < F; ++mu) s += hbar[mu] * dm.gate_wmat[mu * dm.Q + q];
        adj[dm.gate_nodes[q]] += s;
      }
      __syncwarp();
    }

    // ---------------- reverse graph and contraction ----------------
    if (!kRevOnly) {
      run_prog<Real, 2>(pt.prog, pt.prog.nfwd, pt.prog.nsteps, v, adj, parts, lane);
      for (int t = lane; t < K * H; t += kWarp) {
        const int b = dm.basic_of[t];
        abar[t / H * H4 + t % H] = b >= 0 ? adj[b] : Real(0);
      }
      __syncwarp();
    }

    // ---------------- per-edge adjoint ----------------
    // batches in reverse order, the next one's edge inputs loaded while the current one runs
    // (with bulk-copied h_j rows the last forward batch's rows are still in hbuf: the first
    // adjoint batch uses them, and each batch's copies for the one after are issued mid-batch)
    for (int bt = nbat - 1; bt >= 0; --bt) {
      const int e = e0 + bt * kWarp + lane, nb = min(kWarp, e1 - e0 - bt * kWarp);
      const bool valid = e < e1;
      EdgeIn<Real> nxt = cur;
      if (bt > 0) nxt = load_edge<Real>(a.d4, a.nbr, a.types, e - kWarp, C);
      if (hb_on && bt < nbat - 1 && !hb_arrived()) return;
      // Effect: h_j in the columns (or the bulk-copied batch rows); each value is read before the
      // hbar contribution overwrites it, and the contributions go out as rows
      if (effect_outer && !hb_on) rows_to_cols<Real>(stage, a.hsig, F, cur.j, nb, lane);
      if (!effect_outer && !valid) { cur = nxt; continue; }
      const V4 dv = cur.d;
      const int tj = cur.tj;
      cur = nxt;
      Real r = Real(1), ir = Real(1), ux = Real(0), uy = Real(0), uz = Real(0), s = Real(0);
      // P[h] = sum_k w R_kl(h) abar[k][h] feeds the angular gradient; the radial-derivative term
      // sum_h Qd[h] Y[h], Qd[h] = sum_k w R'_kl(h) abar[k][h], is summed per (k, l) as
      // w R'_kl S_kl with S_kl = sum_{h in l} abar[k][h] Y[h] (no per-h Qd registers).  Both run on
      // pairs of harmonics (2 p, 2 p + 1): of one l (one packed step), or of two neighbouring l.
      Pair<Real> P[NPH];
      if (valid) {
        r = dv.w;
        ir = Real(1) / r;
        ux = dv.x * ir; uy = dv.y * ir; uz = dv.z * ir;
        Real Y[2 * NPH];
        Y[2 * NPH - 1] = Real(0);
        const bool have = kKeep && bt < keep_batches;
        const Real* kq = kKeep ? kept + static_cast<size_t>(bt) * (2 * F + H) * kWarp : nullptr;
        if (kKeep && have) {
#pragma unroll
          for (int h = 0; h < H; ++h) Y[h] = kq[(2 * F + h) * kWarp];
        } else {
          sph_values<L, Real>(ux, uy, uz, Y);
        }
#pragma unroll
        for (int p = 0; p < NPH; ++p) P[p] = {Real(0), Real(0)};
        const int pair = ti * C + tj;
        const Real* pw = s_pw + pair * F;
        const Real* pa = s_pa + pair * F;
        const Real* hj = hbuf + lane * F;
        Real* col = stage + lane;
        const Envelopes<Real> env = edge_envelopes<Real>(dm, r);
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
          Real R[Lp], Rd[Lp];
          if (kKeep && have) {
#pragma unroll
            for (int l = 0; l < Lp; ++l) {
              R[l] = kq[(k * Lp + l) * kWarp];
              Rd[l] = kq[(F + k * Lp + l) * kWarp];
            }
          } else {
            radial_channel<L, Real, true, BF>(dm, s_coeff, s_scal, pair, r, env, k, R, Rd);
          }
          Real* ck = col + k * Lp * S;
          Real wR[Lp];
          Pair<Real> Sl[Lp];
#pragma unroll
          for (int l = 0; l < Lp; ++l) {
            Real w = pw[k * Lp + l];
            if (effect_outer) {
              const Real wa = pa[k * Lp + l];
              w += wa * (hb_on ? hj[k * Lp + l] : ck[l * S]);
              ck[l * S] = wa * R[l];
            }
            wR[l] = w * R[l];
            Rd[l] *= w;
            Sl[l] = {Real(0), Real(0)};
          }
          const Real* ab = abar + k * H4;
#pragma unroll
          for (int h0 = 0; h0 < H; h0 += 4) {
            Pair<Real> A[2];
            load_quad(ab + h0, A[0], A[1]);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int h = h0 + 2 * u;
              if (h < H) {
                const int la = l_of(h), lb = h + 1 < H ? l_of(h + 1) : la;
                P[h / 2] = fma2(Pair<Real>{wR[la], wR[lb]}, A[u], P[h / 2]);
                if (h + 1 < H && la == lb) {
                  Sl[la] = fma2(A[u], Pair<Real>{Y[h], Y[h + 1]}, Sl[la]);
                } else {
                  Sl[la].x += A[u].x * Y[h];
                  if (h + 1 < H) Sl[lb].y += A[u].y * Y[h + 1];
                }
              }
            }
          }
#pragma unroll
          for (int l = 0; l < Lp; ++l) {
            const Real sum = Sl[l].x + Sl[l].y;
            s += Rd[l] * sum;
            if (effect_outer) ck[l * S] *= sum;
          }
        }
      }
      // the next (earlier, full) batch's h_j rows travel while this one finishes
      if (hb_on && bt > 0) {
        __syncwarp();
        hb_issue(true, cur.j, kWarp);
      }
      if (effect_outer) {
        cols_to_rows<Real>(a.hcontrib, stage, F, valid ? a.rev[e] : 0, nb, lane);
        if (!valid) continue;
      }
      Real gx = Real(0), gy = Real(0), gz = Real(0);
      sph_grad_dot<L, Real>(ux, uy, uz, reinterpret_cast<const Real*>(P), gx, gy, gz);
      const Real ug = ux * gx + uy * gy + uz * gz;
      const Real Gx = ux * s + (gx - ux * ug) * ir;
      const Real Gy = uy * s + (gy - uy * ug) * ir;
      const Real Gz = uz * s + (gz - uz * ug) * ir;
      Real* ge = a.g + (size_t)e * 3;
      if (kGateRev) {
        ge[0] += Gx; ge[1] += Gy; ge[2] += Gz;
      } else {
        ge[0] = Gx; ge[1] = Gy; ge[2] = Gz;
      }
      if (sizeof(Real) == 4) {
        const float dx = float(dv.x), dy = float(dv.y), dz = float(dv.z);
        csum_add_prod(vhi[0], vlo[0], -dx, float(Gx)); csum_add_prod(vhi[1], vlo[1], -dy, float(Gy));
        csum_add_prod(vhi[2], vlo[2], -dz, float(Gz)); csum_add_prod(vhi[3], vlo[3], -dx, float(Gy));
        csum_add_prod(vhi[4], vlo[4], -dx, float(Gz)); csum_add_prod(vhi[5], vlo[5], -dy, float(Gz));
      } else {
        const double dx = dv.x, dy = dv.y, dz = dv.z;
        vir[0] -= dx * double(Gx); vir[1] -= dy * double(Gy); vir[2] -= dz * double(Gz);
        vir[3] -= dx * double(Gy); vir[4] -= dx * double(Gz); vir[5] -= dy * double(Gz);
      }
    }
    // per-atom virial: one lane of four writes a component (FP32 bulk: compensated warp totals in
    // FP32, then one conversion to FP64)
    double* vo = a.virial + (size_t)atom * 6;
    const int vc = warp_sums_index(lane);
    double total;
    if (sizeof(Real) == 4) {
      float h, l;
      warp_csums(vhi, vlo, lane, h, l);
      total = double(h) + double(l);
    } else {
      total = warp_sums(vir, lane);
    }
    if ((lane & 3) == 0 && vc < 6) vo[vc] = kGateRev ? vo[vc] + total : total;
    __syncwarp();
  }
  finish_dynamic();
}

}  // namespace sus2g
