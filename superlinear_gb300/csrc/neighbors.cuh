// Periodic directed-edge builder (CSR by centre) and the small gather / reduction kernels.
//
// Edge set: every (i, j, image n) with |x_j - x_i + n.cell|^2 < r_c^2 except i == j with n = 0,
// i.e. the reference's neighbourhoods including self images in small cells
// (src/neighborhoods.cpp:145-350; the standalone harness enumerates images the same way,
// interfaces/lammps/tests/embedded_efs.cpp:49-66).  Two enumerations produce that set:
//   * image scan (small frames): for each j of the frame the image range
//     ceil(-f - reach) .. floor(-f + reach) per axis, f = (x_j - x_i) . inv(cell),
//     reach_q = r_c |inv(cell)[:, q]|  -- the harness's own bounds;
//   * cell list (frames whose perpendicular widths are all >= 3 r_c): fractional bins of width
//     >= r_c / 2, the 125 bins within two of the centre's with periodic wrap; each (j, n) is
//     found exactly once.
// Afterwards each centre's edges are sorted by (j, n) -- the image-scan order -- and every edge
// gets the index of its reverse edge (j -> i, -n) by binary search, which makes the force gather
// F_i = sum_{e out of i} (g_e - g_rev(e)) atomic-free and deterministic.
#pragma once
#include "device_common.cuh"

namespace sus2g {

struct FramePlan {
  double cell[9];   // rows are lattice vectors
  double inv[9];    // inverse of the row matrix: frac_q = sum_a x_a inv[a][q]
  double reach[3];
  int a0, a1;       // atom range
  int use_bins;
  int nb[3];
  int bin0;         // first bin index of this frame in the global bin arrays
  int cap;          // cell-list frames: edge slots per centre in the padded staging buffers
  long long pad0;   // cell-list frames: first padded slot of the frame (centre i: pad0 + (i - a0) cap)
  float cellf[9];   // FP32 copy of the cell for the candidate prefilter
  float celll[9];   // cell - cellf: with cellf the double-float form of the cell rows
  double band;      // |r^2 error| bound of the FP32 prefilter; candidates within it get the FP64 test
  float screen2;    // FP32 prefilter threshold r_c^2 + band
  float lo2, hi2;   // FP32 engines: r^2 below lo2 is inside, above hi2 outside, else the FP64 test
  float invf[9], reachf[3], rc2f;  // FP32 copies for the image scan's FP32 ranges and bound
};

// Per-atom integer cell offsets floor(frac) (FP64 arithmetic) and bin coordinates (10 bits each),
// written by the binning kernel for cell-list frames; the offsets also per bin slot.
struct __align__(16) AtomOff { int x, y, z, bin; };
// One bin slot (atoms grouped by bin): the exact position wrapped into the home cell,
// x - floor(frac) . cell (FP64), and the atom's index: the exact test forms x_j + n.cell - x_i as
// wrapped x_j + ((w + off_i) . cell - x_i), whose second term is one constant per (centre,
// neighbouring bin).
struct __align__(16) BinPos { double x, y, z; int j, pad; };
// The wrapped position as double-float parts x = xh + xl (xh = fl32(x)).
struct __align__(16) BinPosF { float xh, yh, zh; int j; float xl, yl, zl; int pad; };

__device__ __forceinline__ unsigned long long edge_key(int j, int n0, int n1, int n2) {
  return (static_cast<unsigned long long>(j) << 21) |
         (static_cast<unsigned long long>(n0 + 64) << 14) |
         (static_cast<unsigned long long>(n1 + 64) << 7) |
         static_cast<unsigned long long>(n2 + 64);
}

// Cell-list frames, one warp per centre i.  Bins are at least r_c / 2 wide, so every neighbour lies
// in the 5 x 5 x 5 bins around the centre's bin (about 2.3x fewer candidates than 27 bins of width
// r_c).  Each lane owns four of those 125 bins and walks them two at a time (independent loads in
// flight): a candidate is one 16-byte load, and the FP32 prefilter adds the bin's wrap shift to the
// wrapped position's leading part.  Candidates that pass are appended to a per-warp ring in shared
// memory and whenever 32 are queued the warp tests a full warp of them:
//   * FP64 engines: x_j + n.cell - x_i and r^2 in FP64;
//   * FP32 engines: the same vector from double-float (hi, lo) parts in FP32 arithmetic, with the
//     FP64 test only for the rare entries whose FP32 r^2 lies within 1e-4 relative of r_c^2
//     (FP64 runs at 1/64 of the FP32 rate on this GPU).
// Either way the accepted set is exactly {r^2 < r_c^2} in FP64.  The vector's periodic part
// depends only on the wrap w in {-1, 0, 1}^3 of the neighbouring bin: entry k < 27 of the shift
// table holds (w_k + off_i) . cell - x_i.  Accepted edges of each round are reported through
// Round(mask, lane_accepted, j, packed image, x, y, z, r) (Real components and distance), so the
// caller can count or write them with one ballot per round.
constexpr int kEdgeQueue = 128;                    // ring entries: at most 31 + 64 are waiting
constexpr int kBinReach = 2;                       // bins on each side of the centre's bin
constexpr int kBinSpan = 2 * kBinReach + 1;        // 5
constexpr int kBinStencil = kBinSpan * kBinSpan * kBinSpan;  // 125
constexpr int kBinsPerLane = 4;                    // 32 x 4 >= 125
// double-float sum (ah + al) + (bh + bl), rounded to FP32 (two-sum of the high parts)
__device__ __forceinline__ float df_add(float ah, float al, float bh, float bl) {
  const float s = ah + bh;
  const float v = s - ah;
  const float e = (ah - (s - v)) + (bh - v);
  return s + (e + (al + bl));
}

// Double-float accumulation (h, l) += (bh, bl) (Knuth two-sum of the leading parts, the trailing
// parts added once): absolute error a few 2^-48 of the operands' magnitudes.
__device__ __forceinline__ void df_acc(float& h, float& l, float bh, float bl) {
  const float s = h + bh;
  const float v = s - h;
  const float e = (h - (s - v)) + (bh - v) + (l + bl);
  h = s + e;
  l = e - (h - s);
}

// (h, l) += m (ch, cl) for a small integer m (|m| <= 64): m ch is split exactly by an FMA.
__device__ __forceinline__ void df_acc_mul(float& h, float& l, float m, float ch, float cl) {
  const float p = m * ch;
  const float pe = fmaf(m, ch, -p);
  df_acc(h, l, p, fmaf(m, cl, pe));
}

// Per-warp shared tables of the fill.  Per wrap w in {-1, 0, 1}^3 of a neighbouring bin (index
// (w0 + 1) 9 + (w1 + 1) 3 + (w2 + 1)) the exact shift (w + off_i) . cell - x_i: its leading FP32
// part, and the trailing part (FP32 engines) or the FP64 value.  The ring: (bin slot, wrap index |
// (w0 + 1) << 5 | (w1 + 1) << 7 | (w2 + 1) << 9).
template <typename Real> struct BinWalk {
  float4 hi[27];
  typename Vec4<Real>::type lo[27];
  int2 queue[kEdgeQueue];
};

template <typename Real, typename Round>
__device__ __forceinline__ void warp_bin_edges(int i, const FramePlan& fp, const double* pos, double rc2,
                                               const int* bin_count, int bin_cap, const AtomOff* bin_off,
                                               const BinPos* bin_pos, const BinPosF* bin_posf, const int* rec_of,
                                               const AtomOff* off, int* error, BinWalk<Real>& walk, Round&& round) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const AtomOff oi = off[i];
  const int bi0 = oi.bin >> 20, bi1 = (oi.bin >> 10) & 1023, bi2 = oi.bin & 1023;
  const double* c = fp.cell;
  const int self_rec = rec_of[i];  // the centre's own bin slot
  // lane k < 27: wrap k.  Its shift (w + off_i) . cell - x_i = w . cell - (x_i wrapped into the home
  // cell): FP64 engines in FP64; FP32 engines as double-float parts from the cell's and the centre
  // slot's (hi, lo) parts in FP32 arithmetic (their exact FP64 shift is formed only for the rare
  // entries near the cutoff)
  if (lane < 27) {
    const int w0 = lane / 9 - 1, w1 = (lane / 3) % 3 - 1, w2 = lane % 3 - 1;
    typename Vec4<Real>::type lo;
    float4 hi;
    lo.w = 0;
    if constexpr (sizeof(Real) == 8) {
      const double a0 = w0 + oi.x, a1 = w1 + oi.y, a2 = w2 + oi.z;
      lo.x = a0 * c[0] + a1 * c[3] + a2 * c[6] - pos[3 * i];
      lo.y = a0 * c[1] + a1 * c[4] + a2 * c[7] - pos[3 * i + 1];
      lo.z = a0 * c[2] + a1 * c[5] + a2 * c[8] - pos[3 * i + 2];
      hi = make_float4(static_cast<float>(lo.x), static_cast<float>(lo.y), static_cast<float>(lo.z), 0.f);
    } else {
      const BinPosF me = bin_posf[self_rec];
      const float* cf = fp.cellf;
      const float* cl = fp.celll;
      float h[3], l[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        // w0 row0 + w1 row1 + w2 row2 - x_i, each term an exact (hi, lo) pair
        float sh = -(q == 0 ? me.xh : (q == 1 ? me.yh : me.zh));
        float sl = -(q == 0 ? me.xl : (q == 1 ? me.yl : me.zl));
        const int wq[3] = {w0, w1, w2};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const float th = static_cast<float>(wq[r]) * cf[3 * r + q], tl = static_cast<float>(wq[r]) * cl[3 * r + q];
          const float s2 = sh + th, v = s2 - sh;
          const float e = (sh - (s2 - v)) + (th - v);
          const float rest = e + (sl + tl);
          sh = s2 + rest;
          sl = rest - (sh - s2);
        }
        h[q] = sh;
        l[q] = sl;
      }
      hi = make_float4(h[0], h[1], h[2], 0.f);
      lo.x = l[0]; lo.y = l[1]; lo.z = l[2];
    }
    walk.hi[lane] = hi;
    walk.lo[lane] = lo;
  }
  __syncwarp();
  const float screen = fp.screen2, lo2 = fp.lo2, hi2 = fp.hi2;
  int head = 0, tail = 0;  // warp-uniform ring positions
  // test of the ring's first n entries (one per lane) and the round callback
  auto drain = [&](int n) {
    bool ok = false;
    int j = 0, image = 0;
    Real vx = 0, vy = 0, vz = 0, r2 = 0;
    if (lane < n) {
      const int2 q = walk.queue[(head + lane) & (kEdgeQueue - 1)];
      const int k = q.y & 31;
      const AtomOff oj = bin_off[q.x];
      const int n0 = ((q.y >> 5) & 3) - 1 + oi.x - oj.x, n1 = ((q.y >> 7) & 3) - 1 + oi.y - oj.y,
                n2 = ((q.y >> 9) & 3) - 1 + oi.z - oj.z;
      image = ((n0 + 64) << 14) | ((n1 + 64) << 7) | (n2 + 64);
      const bool self = q.x == self_rec && k == 13;
      const bool packable = (((n0 + 64) | (n1 + 64) | (n2 + 64)) & ~127) == 0;
      if (!packable) record_error(error, kErrImageRange);
      if constexpr (sizeof(Real) == 8) {
        const BinPos bp = bin_pos[q.x];
        const auto w = walk.lo[k];
        j = bp.j;
        vx = bp.x + w.x;
        vy = bp.y + w.y;
        vz = bp.z + w.z;
        r2 = vx * vx + vy * vy + vz * vz;
        ok = r2 < rc2;
      } else {
        const BinPosF bp = bin_posf[q.x];
        const float4 h = walk.hi[k];
        const EdgeF l = walk.lo[k];
        j = bp.j;
        vx = df_add(bp.xh, bp.xl, h.x, l.x);
        vy = df_add(bp.yh, bp.yl, h.y, l.y);
        vz = df_add(bp.zh, bp.zl, h.z, l.z);
        r2 = vx * vx + vy * vy + vz * vz;
        ok = r2 < lo2;
        if (!ok && r2 < hi2) {
          // near the cutoff: the FP64 test decides, x_j + (w + off_i) . cell - x_i in FP64
          const BinPos bd = bin_pos[q.x];
          const double a0 = n0 + oj.x, a1 = n1 + oj.y, a2 = n2 + oj.z;
          const double dx = bd.x + (a0 * c[0] + a1 * c[3] + a2 * c[6] - pos[3 * i]);
          const double dy = bd.y + (a0 * c[1] + a1 * c[4] + a2 * c[7] - pos[3 * i + 1]);
          const double dz = bd.z + (a0 * c[2] + a1 * c[5] + a2 * c[8] - pos[3 * i + 2]);
          const double d2 = dx * dx + dy * dy + dz * dz;
          ok = d2 < rc2;
          vx = static_cast<float>(dx); vy = static_cast<float>(dy); vz = static_cast<float>(dz);
          r2 = static_cast<float>(d2);
        }
      }
      ok = ok && !self && packable;
    }
    head += n;
    const unsigned mask = __ballot_sync(0xffffffffu, ok);
    if constexpr (sizeof(Real) == 8) round(mask, ok, j, image, vx, vy, vz, sqrt(r2));
    else round(mask, ok, j, image, vx, vy, vz, sqrtf(r2));
  };
  // prefilter of slot `rec` of a bin with shift h, and its place in the ring
  auto screen_candidate = [&](bool have, int rec, const float4& h, int wrap) {
    bool pass = false;
    if (have) {
      const float4 p = *reinterpret_cast<const float4*>(bin_posf + rec);
      const float x = p.x + h.x, y = p.y + h.y, z = p.z + h.z;
      pass = x * x + y * y + z * z < screen;
    }
    const unsigned m = __ballot_sync(0xffffffffu, pass);
    if (pass) walk.queue[(tail + __popc(m & below)) & (kEdgeQueue - 1)] = make_int2(rec, wrap);
    tail += __popc(m);
  };
#pragma unroll 1
  for (int u = 0; u < kBinsPerLane; u += 2) {
    int first[2], len[2], wrap[2];
    float4 h[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int sl = kBinsPerLane * lane + u + p;
      first[p] = 0; len[p] = 0; wrap[p] = 13;
      if (sl < kBinStencil) {
        int w[3], at[3] = {bi0 + sl / (kBinSpan * kBinSpan) - kBinReach, bi1 + (sl / kBinSpan) % kBinSpan - kBinReach,
                           bi2 + sl % kBinSpan - kBinReach};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          w[q] = 1;
          if (at[q] < 0) { w[q] = 0; at[q] += fp.nb[q]; }
          else if (at[q] >= fp.nb[q]) { w[q] = 2; at[q] -= fp.nb[q]; }
        }
        const int bin = fp.bin0 + (at[0] * fp.nb[1] + at[1]) * fp.nb[2] + at[2];
        first[p] = bin * bin_cap;
        len[p] = min(bin_count[bin], bin_cap);
        wrap[p] = (w[0] * 9 + w[1] * 3 + w[2]) | (w[0] << 5) | (w[1] << 7) | (w[2] << 9);
      }
      h[p] = walk.hi[wrap[p] & 31];
    }
    const int most = __reduce_max_sync(0xffffffffu, max(len[0], len[1]));
    for (int t = 0; t < most; ++t) {
      screen_candidate(t < len[0], first[0] + t, h[0], wrap[0]);
      screen_candidate(t < len[1], first[1] + t, h[1], wrap[1]);
      __syncwarp();
      while (tail - head >= 32) drain(32);
      __syncwarp();  // the ring's read entries may be overwritten
    }
  }
  if (tail > head) drain(tail - head);
  __syncwarp();
}

}  // namespace sus2g
