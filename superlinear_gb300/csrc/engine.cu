// Host orchestration of the GPU engine: device tables, edge building, pass launches, force gather
// and per-frame reductions.
#include "engine.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <map>
#include <cstring>
#include <numeric>
#include <stdexcept>
#include <string>

#include "neighbors.cuh"
#include "pass_launch.h"

namespace sus2g {

#define SUS2G_CUDA(call)                                                                      \
  do {                                                                                        \
    cudaError_t err__ = (call);                                                               \
    if (err__ != cudaSuccess)                                                                 \
      throw Error(10, std::string("CUDA error: ") + cudaGetErrorString(err__) + " at " #call); \
  } while (0)

void DevBuf::ensure(size_t n) {
  if (n <= bytes && ptr) return;
  release();
  const size_t want = std::max<size_t>(n, 256);
  SUS2G_CUDA(cudaMalloc(&ptr, want));
  bytes = want;
}
bool DevBuf::try_ensure(size_t n) {
  if (n <= bytes && ptr) return true;
  release();
  const size_t want = std::max<size_t>(n, 256);
  const cudaError_t err = cudaMalloc(&ptr, want);
  if (err == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    ptr = nullptr;
    return false;
  }
  SUS2G_CUDA(err);
  bytes = want;
  return true;
}
void DevBuf::release() {
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
  bytes = 0;
}

// ------------------------------------------------------------------------------------------------
// edge building kernels
// ------------------------------------------------------------------------------------------------
namespace {

// Frame of every atom; with posh / posl (batches with image-scan frames) also its position
// as double-float parts x = xh + xl, xh = fl32(x), for the image scan's FP32 arithmetic.
__global__ void k_frame_of(const FramePlan* plans, int nframes, int* frame_of, const double* pos, float4* posh,
                           float4* posl) {
  const int f = blockIdx.x;
  if (f >= nframes) return;
  for (int i = plans[f].a0 + threadIdx.x; i < plans[f].a1; i += blockDim.x) {
    frame_of[i] = f;
    if (posh) {
      const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
      const float xh = static_cast<float>(x), yh = static_cast<float>(y), zh = static_cast<float>(z);
      posh[i] = make_float4(xh, yh, zh, 0.f);
      posl[i] = make_float4(static_cast<float>(x - xh), static_cast<float>(y - yh), static_cast<float>(z - zh), 0.f);
    }
  }
}

// Cell-list binning in one pass: per atom the wrapped fractions and integer cell offsets, its bin
// (bins of frame f are bin0 .. bin0 + nb0 nb1 nb2 - 1) and its record in the bin's fixed-capacity
// slots bin bcap .. bin bcap + bcap - 1 (order inside a bin is arbitrary: each centre's edges are
// sorted by (j, image) afterwards).  A bin that receives more than bcap atoms raises *bin_over to
// its count; the host then grows bcap and repeats the step.  With find_frame the atom's frame is
// found here (binary search over the frames' first atoms) and written to frame_of.
__global__ void k_bin_place(const FramePlan* plans, int nframes, bool find_frame, int* frame_of, const double* pos,
                            int natoms, int bcap, int* rec_of, int* bin_count, AtomOff* off, AtomOff* bin_off,
                            BinPos* bin_pos, BinPosF* bin_posf, int* bin_over,
                            int* error, const int* types, int C) {
  pdl_launch_dependents();  // the fill kernel's blocks may become resident while this grid runs
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natoms) return;
  int f;
  if (find_frame) {
    // last frame whose first atom is <= i (an empty frame shares its first atom with the next one)
    int lo = 0, hi = nframes - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (plans[mid].a0 <= i) lo = mid; else hi = mid - 1;
    }
    f = lo;
    frame_of[i] = f;
  } else {
    f = frame_of[i];
  }
  const FramePlan& fp = plans[f];
  if (types[i] < 0 || types[i] >= C) record_error(error, kErrBadSpecies);
  if (!fp.use_bins) return;
  const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  // fractional coordinates, checked before any conversion to an integer: a non-finite coordinate,
  // or one more than 2^30 cells from the home cell, is reported and the atom binned inertly at
  // fraction 0 of bin 0 with non-finite wrapped positions (every distance test then rejects it)
  double sq[3];
  bool finite = true;
  for (int q = 0; q < 3; ++q) {
    sq[q] = x * fp.inv[q] + y * fp.inv[3 + q] + z * fp.inv[6 + q];
    finite = finite && fabs(sq[q]) < 1073741824.0;  // false for NaN and infinities too
  }
  if (!finite) record_error(error, kErrBadPosition);
  int b[3], o[3];
  for (int q = 0; q < 3; ++q) {
    const double fl = finite ? floor(sq[q]) : 0.0;
    const double w = finite ? sq[q] - fl : 0.0;
    o[q] = static_cast<int>(fl);
    b[q] = max(0, min(static_cast<int>(w * fp.nb[q]), fp.nb[q] - 1));
  }
  off[i] = AtomOff{o[0], o[1], o[2], (b[0] << 20) | (b[1] << 10) | b[2]};
  const int bin = fp.bin0 + (b[0] * fp.nb[1] + b[1]) * fp.nb[2] + b[2];
  const int slot = atomicAdd(bin_count + bin, 1);
  if (slot >= bcap) { atomicMax(bin_over, slot + 1); rec_of[i] = 0; return; }
  const long long rec = static_cast<long long>(bin) * bcap + slot;
  rec_of[i] = static_cast<int>(rec);
  bin_off[rec] = AtomOff{o[0], o[1], o[2], 0};
  const double* c = fp.cell;
  const double a0 = o[0], a1 = o[1], a2 = o[2];
  const double bad = finite ? 0.0 : nan("");
  const double wx = x - (a0 * c[0] + a1 * c[3] + a2 * c[6]) + bad;
  const double wy = y - (a0 * c[1] + a1 * c[4] + a2 * c[7]) + bad;
  const double wz = z - (a0 * c[2] + a1 * c[5] + a2 * c[8]) + bad;
  bin_pos[rec] = BinPos{wx, wy, wz, i, 0};
  const float hx = static_cast<float>(wx), hy = static_cast<float>(wy), hz = static_cast<float>(wz);
  bin_posf[rec] = BinPosF{hx, hy, hz, i, static_cast<float>(wx - hx), static_cast<float>(wy - hy),
                          static_cast<float>(wz - hz), 0};
}

constexpr int kFillWarps = 8;
// A centre's edges between the walk and the sort: the first kStage of them in shared memory, the
// rest in its padded slots of the staging buffers.
template <typename Real> struct EdgeStage {
  static constexpr int kStage = sizeof(Real) == 4 ? 128 : 64;
  typename Vec4<Real>::type d4[kStage];
  int j[kStage], image[kStage];
};

// rank[u] = how many of the centre's n words come before mine[u].  A cell-list frame is at least
// 3 r_c wide, so a neighbour appears once per centre and its index alone is the order.
template <int U, typename Real>
__device__ __forceinline__ void rank_neighbours(int n, const EdgeStage<Real>& st, const int* rest, const int (&mine)[U],
                                                int (&rank)[U]) {
  const int staged = min(n, EdgeStage<Real>::kStage);
#pragma unroll
  for (int u = 0; u < U; ++u) rank[u] = 0;
  int t = 0;
  for (; t + 4 <= staged; t += 4) {
    const int4 o = *reinterpret_cast<const int4*>(st.j + t);
#pragma unroll
    for (int u = 0; u < U; ++u) rank[u] += (o.x < mine[u]) + (o.y < mine[u]) + (o.z < mine[u]) + (o.w < mine[u]);
  }
  for (; t < n; ++t) {
    const int o = t < staged ? st.j[t] : rest[t];
#pragma unroll
    for (int u = 0; u < U; ++u) rank[u] += o < mine[u];
  }
}

// The order of a centre's n <= 128 edges: perm[rank] = place in the stage (32 U places).
template <int U, typename Real>
__device__ __forceinline__ void order_edges(int lane, int n, const EdgeStage<Real>& st, const int* rest, int* perm) {
  int mine[U], rank[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int q = u * kWarp + lane;
    mine[u] = q >= n ? 0 : q < EdgeStage<Real>::kStage ? st.j[q] : rest[q];
  }
  rank_neighbours<U, Real>(n, st, rest, mine, rank);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u * kWarp + lane < n) perm[rank[u]] = u * kWarp + lane;
}

template <typename Real>
__device__ __forceinline__ void order_any(int lane, int n, const EdgeStage<Real>& st, const int* rest, int* perm) {
  switch ((n + kWarp - 1) / kWarp) {
    case 0: break;
    case 1: order_edges<1, Real>(lane, n, st, rest, perm); break;
    case 2: order_edges<2, Real>(lane, n, st, rest, perm); break;
    case 3: order_edges<3, Real>(lane, n, st, rest, perm); break;
    default: order_edges<4, Real>(lane, n, st, rest, perm);
  }
}

// Cell-list frames: one warp per centre over its 125 stencil bins (warp_bin_edges), one pass.  The
// centre's edges are staged, put in order by neighbour and written once, coalesced, to its padded
// slots pad0 + (i - a0) cap .. + cap; a count above cap is clamped to cap and raises *overflow to
// the full count, which the host reads with the step's error check (it then grows the capacity and
// repeats the step).
// Bound by the instructions of the walk and the sort.  32,768 atoms of 92 edges: 164 us with 64-bit
// keys ranked four per lane for any count, staging in global memory and a fractional prefilter; 118 us
// so.
template <typename Real>
__global__ void __launch_bounds__(kFillWarps * kWarp, 4)
k_edge_fill_bins(const FramePlan* plans, const int* frame_of, const double* pos, int natoms, double rc2,
                 const int* bin_count, int bin_cap, const AtomOff* bin_off, const BinPos* bin_pos,
                 const BinPosF* bin_posf, const int* rec_of, const AtomOff* off,
                 int* counts, int* nbr,
                 typename Vec4<Real>::type* d4, unsigned long long* key, int* overflow, int* error, int* row,
                 int* row_end, unsigned long long* key_out, int* nbr_out, typename Vec4<Real>::type* d4_out) {
  using Stage = EdgeStage<Real>;
  __shared__ __align__(16) BinWalk<Real> walks[kFillWarps];
  __shared__ __align__(16) Stage stages[kFillWarps];
  pdl_wait();  // the bins and frame map of the previous kernel
  pdl_launch_dependents();
  const int i = static_cast<int>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / kWarp);
  if (i >= natoms) return;
  const FramePlan& fp = plans[frame_of[i]];
  if (!fp.use_bins) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x / kWarp;
  const unsigned below = (1u << lane) - 1u;
  const long long pad = fp.pad0 + static_cast<long long>(i - fp.a0) * fp.cap;
  const int cap = fp.cap;
  Stage& st = stages[w];
  int cursor = 0;
  warp_bin_edges<Real>(i, fp, pos, rc2, bin_count, bin_cap, bin_off, bin_pos, bin_posf, rec_of, off, error, walks[w],
                       [&](unsigned mask, bool ok, int j, int image, Real x, Real y, Real z, Real r) {
                         if (ok) {
                           const int k = cursor + __popc(mask & below);
                           typename Vec4<Real>::type v;
                           v.x = x; v.y = y; v.z = z; v.w = r;
                           if (k < Stage::kStage) {
                             st.d4[k] = v;
                             st.j[k] = j;
                             st.image[k] = image;
                           } else if (k < cap) {
                             d4[pad + k] = v;
                             nbr[pad + k] = j;
                             key[pad + k] = static_cast<unsigned long long>(image);
                           }
                         }
                         cursor += __popc(mask);
                       });
  const int n = min(cursor, cap);
  if (lane == 0) {
    counts[i] = n;
    if (cursor > cap) atomicMax(overflow, cursor);
    row[i] = static_cast<int>(pad);
    row_end[i] = static_cast<int>(pad) + n;
  }
  const int* rest = nbr + pad;
  auto write = [&](int to, int from) {
    const bool staged = from < Stage::kStage;
    const int j = staged ? st.j[from] : rest[from];
    const unsigned long long image = staged ? static_cast<unsigned long long>(st.image[from]) : key[pad + from];
    key_out[pad + to] = (static_cast<unsigned long long>(j) << 21) | image;
    nbr_out[pad + to] = j;
    d4_out[pad + to] = staged ? st.d4[from] : d4[pad + from];
  };
  if (n <= 4 * kWarp) {
    int* perm = reinterpret_cast<int*>(walks[w].queue);  // (the ring is empty)
    order_any<Real>(lane, n, st, rest, perm);
    __syncwarp();
    for (int q = lane; q < n; q += kWarp) write(q, perm[q]);
  } else {
    for (int q = lane; q < n; q += kWarp) {
      const int mine[1] = {q < Stage::kStage ? st.j[q] : rest[q]};
      int rank[1];
      rank_neighbours<1, Real>(n, st, rest, mine, rank);
      write(rank[0], q);
    }
  }
}

// Periodic frames too small for cell lists (a perpendicular width below 3 r_c, or at most 512
// atoms): warp per centre i, lanes over the frame's atoms j.  For each j the image range per axis
// is ceil(-f - reach) .. floor(-f + reach), f = (x_j - x_i) . inv(cell), and every image n in it
// with r^2 = |x_j + n.cell - x_i|^2 < r_c^2 in FP64 is an edge.  As in the cell-list fill, a lane walks
// its images with an FP32 prefilter, what passes waits in a ring, and a full warp of it is tested:
//   * dx = x_j - x_i in double-float (hi, lo) parts; f = dx_hi . inv(cell) in FP32 errs by at most
//     ~7 2^-24 S, S = sum |dx_r inv_rq|; widening reach by 1e-4 + 1e-6 S keeps every image of the
//     FP64 range.
//   * Prefilter: dx_hi + n.cell_hi errs by less than 16 2^-24 M, M = |dx| + sum_r |n_r| |cell_r| (one
//     norms), so nothing within r_c is lost above (r_c + 16 2^-24 M)^2 (1 + 1e-4).
//   * FP64 engines then test in FP64.  FP32 engines accumulate the vector as double-float pairs
//     (exact two-sums, m cell_hi split exactly by an FMA): absolute error a few dozen 2^-48 of M;
//     rounded once to FP32, with M <= 1e6 r_c, r^2 near r_c^2 errs by well under 1e-6 r_c^2, so r^2
//     below lo2 = (1 - 1e-4) r_c^2 is inside and above hi2 = (1 + 1e-4) r_c^2 outside in FP64 too,
//     and the band takes the FP64 test.  The accepted set is the FP64 set.
//   * Non-finite positions, ranges outside the packable [-64, 63] and larger M take the FP64 loop per
//     lane, which reports the first two.
// The accepted edges are staged, put in order by (j, n) -- in 31 bits up to 1,024 atoms -- and written
// once to the centre's padded slots, as by the cell-list kernel.
// Bound by instructions: with every image's vector formed in place by its lane and 64-bit keys,
// 17,544 atoms of 256 frames took 98 us and 3,840 of 64 frames 39 us (FP64, 884 of 12 frames: 67 us);
// so 75, 26 and 34 us.
template <typename Real>
__global__ void __launch_bounds__(kFillWarps * kWarp)
k_edge_image_fill(const FramePlan* plans, const int* frame_of, const double* pos, const float4* posh,
                  const float4* posl, const int* types, int C, int natoms, double rc2, int* counts,
                  int* nbr, typename Vec4<Real>::type* d4, unsigned long long* key, int* overflow, int* error, int* row,
                  int* row_end, unsigned long long* key_out, int* nbr_out, typename Vec4<Real>::type* d4_out) {
  using Stage = EdgeStage<Real>;
  __shared__ __align__(16) Stage stages[kFillWarps];
  __shared__ int2 queues[kFillWarps][kEdgeQueue];  // (j, packed image)
  __shared__ int cursors[kFillWarps];
  pdl_wait();  // the frame map (and, in mixed batches, the cell-list fill) of the previous kernels
  pdl_launch_dependents();
  const int i = static_cast<int>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / kWarp);
  if (i >= natoms) return;
  const FramePlan& fp = plans[frame_of[i]];
  if (fp.use_bins) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x / kWarp;
  const unsigned below = (1u << lane) - 1u;
  const long long pad = fp.pad0 + static_cast<long long>(i - fp.a0) * fp.cap;
  const int cap = fp.cap;
  Stage& st = stages[w];
  int2* queue = queues[w];
  int& cursor = cursors[w];
  if (lane == 0) cursor = 0;
  __syncwarp();
  const double xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
  // a non-finite centre is reported and gets no edges; a non-finite neighbour is skipped (it
  // reports itself as a centre); image ranges are clamped to the packable [-64, 63] before any
  // conversion to an integer, and a range that reaches past it is reported
  const bool centre_ok = isfinite(xi) && isfinite(yi) && isfinite(zi);
  if (lane == 0 && !centre_ok) record_error(error, kErrBadPosition);
  if (lane == 0 && (types[i] < 0 || types[i] >= C)) record_error(error, kErrBadSpecies);
  const double* c = fp.cell;
  const double* inv = fp.inv;
  const float4 cih = posh[i], cil = posl[i];
  float ch[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) ch[q] = fp.cellf[q];
  const float rcf = sqrtf(fp.rc2f);
  // frames of at most 1,024 atoms: j and the image in one staged word (see the sort below)
  const bool one_word = fp.a1 - fp.a0 <= 1024;
  auto stage_edge = [&](int k, int j, int image, Real x, Real y, Real z, Real r2) {
    typename Vec4<Real>::type v;
    v.x = x; v.y = y; v.z = z;
    if constexpr (sizeof(Real) == 4) v.w = sqrtf(r2);
    else v.w = sqrt(r2);
    const int word = one_word ? ((j - fp.a0) << 21) | image : j;
    if (k < Stage::kStage) {
      st.d4[k] = v;
      st.j[k] = word;
      st.image[k] = image;
    } else if (k < cap) {
      d4[pad + k] = v;
      nbr[pad + k] = word;
      key[pad + k] = static_cast<unsigned long long>(image);
    }
  };
  auto exact = [&](int j, int a, int b, int cc, double& vx, double& vy, double& vz) {
    const double dx = pos[3 * j] - xi, dy = pos[3 * j + 1] - yi, dz = pos[3 * j + 2] - zi;
    vx = dx + a * c[0] + b * c[3] + cc * c[6];
    vy = dy + a * c[1] + b * c[4] + cc * c[7];
    vz = dz + a * c[2] + b * c[5] + cc * c[8];
    return vx * vx + vy * vy + vz * vz;
  };
  int head = 0, tail = 0;  // warp-uniform ring positions
  auto drain = [&](int n) {
    bool ok = false;
    int j = 0, image = 0;
    Real vx = 0, vy = 0, vz = 0, r2 = 0;
    if (lane < n) {
      const int2 q = queue[(head + lane) & (kEdgeQueue - 1)];
      j = q.x;
      image = q.y;
      const int a = (image >> 14) - 64, b = ((image >> 7) & 127) - 64, cc = (image & 127) - 64;
      if constexpr (sizeof(Real) == 8) {
        r2 = exact(j, a, b, cc, vx, vy, vz);
        ok = r2 < rc2;
      } else {
        const float4 hj = posh[j], lj = posl[j];
        const float* cl = fp.celll;
        float xh = hj.x, xl = lj.x, yh = hj.y, yl = lj.y, zh = hj.z, zl = lj.z;
        df_acc(xh, xl, -cih.x, -cil.x);
        df_acc(yh, yl, -cih.y, -cil.y);
        df_acc(zh, zl, -cih.z, -cil.z);
        const float m[3] = {static_cast<float>(a), static_cast<float>(b), static_cast<float>(cc)};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          df_acc_mul(xh, xl, m[r], ch[3 * r], cl[3 * r]);
          df_acc_mul(yh, yl, m[r], ch[3 * r + 1], cl[3 * r + 1]);
          df_acc_mul(zh, zl, m[r], ch[3 * r + 2], cl[3 * r + 2]);
        }
        vx = xh + xl; vy = yh + yl; vz = zh + zl;
        r2 = vx * vx + vy * vy + vz * vz;
        ok = r2 < fp.lo2;
        if (!ok && r2 < fp.hi2) {
          double ex, ey, ez;
          const double d2 = exact(j, a, b, cc, ex, ey, ez);
          ok = d2 < rc2;
          vx = static_cast<float>(ex); vy = static_cast<float>(ey); vz = static_cast<float>(ez);
          r2 = static_cast<float>(d2);
        }
      }
      ok = ok && !(j == i && a == 0 && b == 0 && cc == 0);
    }
    head += n;
    const unsigned mask = __ballot_sync(0xffffffffu, ok);
    const int k0 = cursor;
    __syncwarp();
    if (lane == 0) cursor = k0 + __popc(mask);
    if (ok) stage_edge(k0 + __popc(mask & below), j, image, vx, vy, vz, r2);
    __syncwarp();
  };
  for (int j0 = fp.a0; centre_ok && j0 < fp.a1; j0 += kWarp) {
    const int j = j0 + lane;
    int lo[3] = {0, 0, 0}, hi[3] = {-1, -1, -1};
    float xh = 0.f, yh = 0.f, zh = 0.f, screen = 0.f;
    if (j < fp.a1) {
      const float4 hj = posh[j], lj = posl[j];
      float xl = lj.x, yl = lj.y, zl = lj.z;
      xh = hj.x; yh = hj.y; zh = hj.z;
      df_acc(xh, xl, -cih.x, -cil.x);
      df_acc(yh, yl, -cih.y, -cil.y);
      df_acc(zh, zl, -cih.z, -cil.z);
      bool fast = true;
      float m = fabsf(xh) + fabsf(yh) + fabsf(zh);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const float t0 = xh * fp.invf[q], t1 = yh * fp.invf[3 + q], t2 = zh * fp.invf[6 + q];
        const float f = t0 + t1 + t2, S = fabsf(t0) + fabsf(t1) + fabsf(t2);
        const float reach = fp.reachf[q] + 1e-4f + 1e-6f * S;
        const float l = ceilf(-f - reach), h = floorf(-f + reach);
        if (l >= -64.0f && h <= 63.0f) {
          lo[q] = static_cast<int>(l);
          hi[q] = static_cast<int>(h);
          m += static_cast<float>(max(abs(lo[q]), abs(hi[q]))) * (fabsf(ch[3 * q]) + fabsf(ch[3 * q + 1]) + fabsf(ch[3 * q + 2]));
        } else {
          fast = false;
        }
      }
      fast = fast && m * m <= 1e12f * fp.rc2f;
      const float lim = rcf + 9.6e-7f * m;
      screen = lim * lim * 1.0001f;
      if (!fast) {
        // FP64 test of every image, by this lane
        const double dx = pos[3 * j] - xi, dy = pos[3 * j + 1] - yi, dz = pos[3 * j + 2] - zi;
        const bool finite = isfinite(dx) && isfinite(dy) && isfinite(dz);
        for (int q = 0; finite && q < 3; ++q) {
          const double f = dx * inv[q] + dy * inv[3 + q] + dz * inv[6 + q];
          double l = ceil(-f - fp.reach[q]), h = floor(-f + fp.reach[q]);
          if (l < -64.0 || h > 63.0) {
            record_error(error, kErrImageRange);
            l = fmax(l, -64.0);
            h = fmin(h, 63.0);
          }
          lo[q] = static_cast<int>(l);
          hi[q] = static_cast<int>(fmax(h, l - 1.0));
        }
        for (int a = lo[0]; finite && a <= hi[0]; ++a)
          for (int b = lo[1]; b <= hi[1]; ++b)
            for (int cc = lo[2]; cc <= hi[2]; ++cc) {
              if (i == j && a == 0 && b == 0 && cc == 0) continue;
              double vx, vy, vz;
              const double r2 = exact(j, a, b, cc, vx, vy, vz);
              if (r2 < rc2)
                stage_edge(atomicAdd(&cursor, 1), j, ((a + 64) << 14) | ((b + 64) << 7) | (cc + 64), Real(vx), Real(vy), Real(vz), Real(r2));
            }
        hi[0] = lo[0] - 1;  // nothing left for the walk
      }
    }
    __syncwarp();
    const int mine = max(0, hi[0] - lo[0] + 1) * max(0, hi[1] - lo[1] + 1) * max(0, hi[2] - lo[2] + 1);
    const int most = __reduce_max_sync(0xffffffffu, mine);
    int a = lo[0], b = lo[1], cc = lo[2];
    for (int t = 0; t < most; ++t) {
      const float fa = static_cast<float>(a), fb = static_cast<float>(b), fc = static_cast<float>(cc);
      const float vx = fmaf(fa, ch[0], fmaf(fb, ch[3], fmaf(fc, ch[6], xh)));
      const float vy = fmaf(fa, ch[1], fmaf(fb, ch[4], fmaf(fc, ch[7], yh)));
      const float vz = fmaf(fa, ch[2], fmaf(fb, ch[5], fmaf(fc, ch[8], zh)));
      const bool pass = t < mine && vx * vx + vy * vy + vz * vz < screen;
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      if (pass)
        queue[(tail + __popc(m & below)) & (kEdgeQueue - 1)] = make_int2(j, ((a + 64) << 14) | ((b + 64) << 7) | (cc + 64));
      tail += __popc(m);
      if (++cc > hi[2]) {
        cc = lo[2];
        if (++b > hi[1]) { b = lo[1]; ++a; }
      }
      __syncwarp();
      if (tail - head >= 32) drain(32);
    }
  }
  if (tail > head) drain(tail - head);
  __syncwarp();
  const int total = cursor, n = min(total, cap);
  if (lane == 0) {
    counts[i] = n;
    if (total > cap) atomicMax(overflow, total);
    row[i] = static_cast<int>(pad);
    row_end[i] = static_cast<int>(pad) + n;
  }
  const int* rest = nbr + pad;
  auto word_of = [&](int q) { return q < Stage::kStage ? st.j[q] : rest[q]; };
  auto image_of = [&](int q) { return q < Stage::kStage ? st.image[q] : static_cast<int>(key[pad + q]); };
  auto write = [&](int to, int from) {
    const int word = word_of(from), j = one_word ? fp.a0 + (word >> 21) : word;
    key_out[pad + to] = (static_cast<unsigned long long>(j) << 21) | static_cast<unsigned long long>(image_of(from));
    nbr_out[pad + to] = j;
    d4_out[pad + to] = from < Stage::kStage ? st.d4[from] : d4[pad + from];
  };
  if (one_word && n <= 4 * kWarp) {
    int* perm = reinterpret_cast<int*>(queue);  // (the ring is empty)
    order_any<Real>(lane, n, st, rest, perm);
    __syncwarp();
    for (int q = lane; q < n; q += kWarp) write(q, perm[q]);
  } else if (one_word) {
    for (int q = lane; q < n; q += kWarp) {
      const int mine[1] = {word_of(q)};
      int rank[1];
      rank_neighbours<1, Real>(n, st, rest, mine, rank);
      write(rank[0], q);
    }
  } else {
    for (int q = lane; q < n; q += kWarp) {
      const int j = word_of(q), image = image_of(q);
      int rank = 0;
      for (int t = 0; t < n; ++t) {
        const int o = word_of(t);
        rank += o < j || (o == j && image_of(t) < image);
      }
      write(rank, q);
    }
  }
}

// Sort one centre's edges of a user edge list by key into CSR order (warp per centre, rank sort;
// keys within a centre are unique).  Keys of centres with at most `stage` edges are staged in
// shared memory (the rank loop then reads broadcast shared memory); longer lists rank from global
// memory.  Periodic batches are sorted inside their fill kernels.
constexpr int kSortWarps = 8;
template <typename Real>
__global__ void __launch_bounds__(kSortWarps * kWarp)
k_edge_sort(const int* row, int natoms, int stage, const unsigned long long* key_in, const int* nbr_in,
            const typename Vec4<Real>::type* d4_in, unsigned long long* key_out, int* nbr_out,
            typename Vec4<Real>::type* d4_out) {
  extern __shared__ unsigned long long sort_keys[];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x & 31;
  if (warp >= natoms) return;
  const int e0 = row[warp], n = row[warp + 1] - e0;
  const long long in0 = e0;
  const unsigned long long* K = key_in;
  const int* NB = nbr_in;
  const typename Vec4<Real>::type* D = d4_in;
  const unsigned long long* src = K + in0;
  if (n <= stage) {
    unsigned long long* sk = sort_keys + (threadIdx.x / kWarp) * stage;
    for (int q = lane; q < n; q += kWarp) sk[q] = src[q];
    __syncwarp();
    src = sk;
  }
  // up to kSortPer keys per lane per pass: their payloads load while the ranks are counted
  constexpr int kSortPer = 4;
  for (int q0 = 0; q0 < n; q0 += kSortPer * kWarp) {
    unsigned long long k[kSortPer];
    int nb[kSortPer], rank[kSortPer];
    typename Vec4<Real>::type d[kSortPer];
#pragma unroll
    for (int u = 0; u < kSortPer; ++u) {
      const int q = q0 + u * kWarp + lane;
      k[u] = ~0ull;
      rank[u] = 0;
      if (q < n) {
        k[u] = src[q];
        nb[u] = NB[in0 + q];
        d[u] = D[in0 + q];
      }
    }
    for (int t = 0; t < n; ++t) {
      const unsigned long long kt = src[t];
#pragma unroll
      for (int u = 0; u < kSortPer; ++u) rank[u] += kt < k[u];
    }
#pragma unroll
    for (int u = 0; u < kSortPer; ++u) {
      if (q0 + u * kWarp + lane < n) {
        key_out[e0 + rank[u]] = k[u];
        nbr_out[e0 + rank[u]] = nb[u];
        d4_out[e0 + rank[u]] = d[u];
      }
    }
  }
}

// Reverse edge of every edge (warp per centre i): for e = (i -> j, n) the edge (j -> i, -n) is
// found by binary search in j's sorted keys.
// Up to kRevPer searches per lane run interleaved, so their dependent loads overlap.
// It also clears the first nzero bin counters (their last reader, the fill kernel, is done), so
// that the next step's binning starts from zero without a memset.
__global__ void k_reverse(const int* row, const int* row_end, const unsigned long long* key, int natoms, int* rev,
                          int* error, int* zero, int nzero) {
  constexpr int kRevPer = 4;
  const long long tid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (long long q = tid; q < nzero; q += static_cast<long long>(gridDim.x) * blockDim.x) zero[q] = 0;
  const int i = static_cast<int>(tid / kWarp);
  const int lane = threadIdx.x & 31;
  if (i >= natoms) return;
  const int end = row_end[i];
  for (int base = row[i]; base < end; base += kRevPer * kWarp) {
    int lo[kRevPer], hi[kRevPer], found[kRevPer];
    unsigned long long want[kRevPer];
#pragma unroll
    for (int u = 0; u < kRevPer; ++u) {
      const int e = base + u * kWarp + lane;
      lo[u] = 0; hi[u] = -1; found[u] = -1; want[u] = 0;
      if (e < end) {
        const unsigned long long k = key[e];
        const int j = static_cast<int>(k >> 21);
        const int n0 = static_cast<int>((k >> 14) & 127) - 64, n1 = static_cast<int>((k >> 7) & 127) - 64,
                  n2 = static_cast<int>(k & 127) - 64;
        want[u] = edge_key(i, -n0, -n1, -n2);
        lo[u] = row[j];
        hi[u] = row_end[j] - 1;
      }
    }
    bool active = true;
    while (active) {
      active = false;
#pragma unroll
      for (int u = 0; u < kRevPer; ++u) {
        if (lo[u] <= hi[u]) {
          const int mid = (lo[u] + hi[u]) >> 1;
          const unsigned long long km = key[mid];
          if (km == want[u]) { found[u] = mid; hi[u] = lo[u] - 1; }
          else if (km < want[u]) lo[u] = mid + 1;
          else hi[u] = mid - 1;
          active = active || lo[u] <= hi[u];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kRevPer; ++u) {
      const int e = base + u * kWarp + lane;
      if (e < end) {
        if (found[u] < 0) record_error(error, kErrReverseEdge);
        rev[e] = found[u] < 0 ? e : found[u];
      }
    }
  }
}

// F_i = sum over i's edges of (g_e - g_rev(e)), warp per atom: FP64 accumulation for FP64 edge
// gradients, compensated FP32 (two-sum, FP64 result) for FP32 ones.
template <typename Real>
__global__ void k_force_gather(const int* row, const int* row_end, const int* rev, const Real* g, int natoms,
                               double* force) {
  pdl_wait();  // the pass's dE/dd per edge
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x & 31;
  if (warp >= natoms) return;
  double f[3] = {0, 0, 0};
  float hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0};
  for (int e = row[warp] + lane; e < row_end[warp]; e += kWarp) {
    const int r = rev[e];
    for (int c = 0; c < 3; ++c) {
      if (sizeof(Real) == 4) {
        csum_add(hi[c], lo[c], float(g[3 * (size_t)e + c]));
        csum_add(hi[c], lo[c], -float(g[3 * (size_t)r + c]));
      } else {
        f[c] += double(g[3 * (size_t)e + c]) - double(g[3 * (size_t)r + c]);
      }
    }
  }
  for (int c = 0; c < 3; ++c) f[c] = sizeof(Real) == 4 ? warp_csum(hi[c], lo[c]) : warp_sum(f[c]);
  if (lane == 0)
    for (int c = 0; c < 3; ++c) force[3 * (size_t)warp + c] = f[c];
}


// Caller edges: incoming lists.  in(j) = the edges whose neighbour is j, sorted by edge index, so
// that per-atom sums over them run in a fixed order (no floating-point atomics).
__global__ void k_fill_in(const int* nbr, const int* edges, const int* in_row, int* cursor, int* in_tmp) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= *edges) return;
  const int j = nbr[e];
  in_tmp[in_row[j] + atomicSub(cursor + j, 1) - 1] = e;
}
// warp per atom: rank sort of the (unique) edge indices of in(j)
__global__ void k_sort_in(const int* in_row, int nall, const int* in_tmp, int* in_edge) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x & 31;
  if (j >= nall) return;
  const int b = in_row[j], n = in_row[j + 1] - b;
  for (int q = lane; q < n; q += kWarp) {
    const int x = in_tmp[b + q];
    int rank = 0;
    for (int t = 0; t < n; ++t) rank += in_tmp[b + t] < x;
    in_edge[b + rank] = x;
  }
}

// hbar[j][mu] = sum over in(j), in edge order, of the per-edge contributions hc[e][mu]
// (compensated FP32 for FP32 contributions, FP64 result).
template <typename Real>
__global__ void k_hbar_gather(const int* in_row, const int* in_edge, const Real* hc, int nall, int F, double* hbar) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<long long>(nall) * F) return;
  const int j = static_cast<int>(t / F), mu = static_cast<int>(t - static_cast<long long>(j) * F);
  double acc = 0.0;
  float hi = 0.f, lo = 0.f;
  for (int q = in_row[j]; q < in_row[j + 1]; ++q) {
    const Real v = hc[static_cast<size_t>(in_edge[q]) * F + mu];
    if (sizeof(Real) == 4) csum_add(hi, lo, float(v));
    else acc += double(v);
  }
  hbar[t] = sizeof(Real) == 4 ? double(hi) + double(lo) : acc;
}

// Caller edges: F_i = sum_{e in out(i)} g_e - sum_{e in in(i)} g_e for every atom (ghosts have
// no out-edges), warp per atom, fixed order.
template <typename Real>
__global__ void k_force_gather_user(const int* row, int nowned, const int* in_row, const int* in_edge, const Real* g,
                                    int nall, double* force) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
  const int lane = threadIdx.x & 31;
  if (i >= nall) return;
  double f[3] = {0, 0, 0};
  float hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0};
  auto add = [&](int e, float sign) {
    for (int c = 0; c < 3; ++c) {
      if (sizeof(Real) == 4) csum_add(hi[c], lo[c], sign * float(g[3 * (size_t)e + c]));
      else f[c] += double(sign) * double(g[3 * (size_t)e + c]);
    }
  };
  if (i < nowned)
    for (int e = row[i] + lane; e < row[i + 1]; e += kWarp) add(e, 1.f);
  for (int q = in_row[i] + lane; q < in_row[i + 1]; q += kWarp) add(in_edge[q], -1.f);
  for (int c = 0; c < 3; ++c) f[c] = sizeof(Real) == 4 ? warp_csum(hi[c], lo[c]) : warp_sum(f[c]);
  if (lane == 0)
    for (int c = 0; c < 3; ++c) force[3 * (size_t)i + c] = f[c];
}

// Row pack / unpack of per-atom vectors for the caller's halo exchange: buf[k][w] = v[atom_k][w]
// (atoms[k], or first + k when atoms is null); mode 0 copies buf into v, mode 1 adds it.
template <typename T>
__global__ void k_rows_pack(const T* v, int width, int n, const int* atoms, int first, double* buf) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<long long>(n) * width) return;
  const int k = static_cast<int>(t / width), w = static_cast<int>(t - static_cast<long long>(k) * width);
  const int atom = atoms ? atoms[k] : first + k;
  buf[t] = double(v[static_cast<size_t>(atom) * width + w]);
}
template <typename T>
__global__ void k_rows_unpack(T* v, int width, int n, const int* atoms, int first, const double* buf, int add) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<long long>(n) * width) return;
  const int k = static_cast<int>(t / width), w = static_cast<int>(t - static_cast<long long>(k) * width);
  const int atom = atoms ? atoms[k] : first + k;
  T& dst = v[static_cast<size_t>(atom) * width + w];
  dst = add ? T(double(dst) + buf[t]) : T(buf[t]);
}

__global__ void k_iota(int* v, long long n) {
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e < n) v[e] = static_cast<int>(e);
}

// Per-frame energy and virial (FP64), one launch: block (f, slice) sums the site energies and
// per-atom virials of its atoms (a fixed strided order per thread, then shuffle trees and the
// block's warps in order) into partial[f][slice][7] and copies the site energies out when asked;
// the block of frame f that arrives last (arrivals[f], reset by that block) adds the frame's
// slices in slice order.  The result does not depend on which block arrives last.
constexpr int kFrameThreads = 256;
__global__ void __launch_bounds__(kFrameThreads)
k_frame_reduce(const FramePlan* plans, int nframes, int S, const double* site, const double* vir_atom,
               double* site_out, double* partial, unsigned* arrivals, double* energy, double* virial) {
  const int f = blockIdx.x, sl = blockIdx.y;
  if (f >= nframes) return;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int i = plans[f].a0 + sl * kFrameThreads + threadIdx.x; i < plans[f].a1; i += S * kFrameThreads) {
    const double e = site[i];
    acc[0] += e;
    if (site_out) site_out[i] = e;
    for (int c = 0; c < 6; ++c) acc[1 + c] += vir_atom[6 * (size_t)i + c];
  }
  __shared__ double sh[kFrameThreads / kWarp][7];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x / kWarp;
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    double v = acc[c];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sh[warp][c] = v;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double v = 0.0;
    for (int w = 0; w < kFrameThreads / kWarp; ++w) v += sh[w][threadIdx.x];
    partial[(static_cast<size_t>(f) * S + sl) * 7 + threadIdx.x] = v;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(arrivals + f, 1u) == static_cast<unsigned>(S - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  // warp c < 7 sums component c over the S <= 64 slices: lane q holds slices q and q + 32, then a
  // fixed shuffle tree (all loads in flight at once)
  if (warp < 7) {
    const int c = warp;
    const double* pf = partial + static_cast<size_t>(f) * S * 7 + c;
    double v = lane < S ? __ldcg(pf + 7 * lane) : 0.0;
    if (lane + kWarp < S) v += __ldcg(pf + 7 * (lane + kWarp));
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) {
      if (c == 0) {
        if (energy) energy[f] = v;
      } else if (virial) {
        virial[6 * f + c - 1] = v;
      }
    }
  }
  if (threadIdx.x == 0) arrivals[f] = 0u;
}

// Caller-provided edges (owned centres, LAMMPS layout): *flag = 1 when an index is out of range or a
// length is not well inside (0, 1e150).
__global__ void k_check_user_edges(const int* ei, const int* ej, const double* d, long long n, int nowned, int nall, int* flag) {
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int i = ei[e], j = ej[e];
  const double x = d[3 * e], y = d[3 * e + 1], z = d[3 * e + 2], r2 = x * x + y * y + z * z;
  if (i < 0 || i >= nowned || j < 0 || j >= nall || !(r2 > 1e-290) || !(r2 < 1e299)) *flag = 1;
}
// Counts per centre and per neighbour.  An edge with a centre or neighbour index out of range is
// flagged and left out here and by the scatter below alike, so that no row keeps an unfilled slot.
__global__ void k_count_user_edges(const int* ei, const int* ej, long long n, int* out_count, int* in_count, int nowned,
                                   int nall, int* error) {
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int i = ei[e], j = ej[e];
  if (i < 0 || i >= nowned || j < 0 || j >= nall) { record_error(error, kErrEdgeCapacity); return; }
  atomicAdd(out_count + i, 1);
  atomicAdd(in_count + j, 1);
}

template <typename Real>
__global__ void k_scatter_user_edges(const int* ei, const int* ej, const double* d, long long n, const int* row,
                                     int* cursor, int* nbr, typename Vec4<Real>::type* d4, unsigned long long* key,
                                     int nowned, int nall, int* error) {
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int i = ei[e], j = ej[e];
  if (i < 0 || i >= nowned || j < 0 || j >= nall) { record_error(error, kErrEdgeCapacity); return; }
  const double x = d[3 * e], y = d[3 * e + 1], z = d[3 * e + 2];
  const double r2 = x * x + y * y + z * z;
  if (!(r2 > 0) || !(r2 < 1e300)) record_error(error, kErrBadDistance);
  // the counts run down to zero as the rows fill (the order within a row is made by the sort)
  const int p = row[i] + atomicSub(cursor + i, 1) - 1;
  nbr[p] = j;
  typename Vec4<Real>::type v;
  // FP32 records: the distance from the rounded r^2 (an FP32 square root; the FP64 one costs tens
  // of FP64-pipe instructions)
  if constexpr (sizeof(Real) == 4) {
    v.x = edge_component(x); v.y = edge_component(y); v.z = edge_component(z);
    v.w = sqrtf(static_cast<float>(r2));
  } else {
    v.x = x; v.y = y; v.z = z;
    v.w = sqrt(r2);
  }
  d4[p] = v;
  // Order key: neighbour, then the caller's edge index (unique, deterministic).
  key[p] = (static_cast<unsigned long long>(j) << 32) | static_cast<unsigned long long>(e & 0xffffffffLL);
}

// Exclusive scans of n counts each into row[0..n] on the device: block 0 the out-edges, block 1 the
// in-edges (each thread scans a contiguous chunk, then the chunk totals are scanned in shared
// memory).  Totals above 2^31 - 1 are flagged.
__global__ void k_exclusive_scans(const int* out_counts, const int* in_counts, int n, int* out_row, int* in_row, int* error) {
  const int* counts = blockIdx.x ? in_counts : out_counts;
  int* row = blockIdx.x ? in_row : out_row;
  __shared__ long long part[1024];
  const int t = threadIdx.x, T = blockDim.x;
  const long long chunk = (static_cast<long long>(n) + T - 1) / T;
  const long long a = t * chunk, b = min(static_cast<long long>(n), a + chunk);
  long long s = 0;
  for (long long i = a; i < b; ++i) s += counts[i];
  part[t] = s;
  __syncthreads();
  for (int off = 1; off < T; off <<= 1) {
    const long long v = t >= off ? part[t - off] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  long long run = part[t] - s;
  for (long long i = a; i < b; ++i) {
    row[i] = static_cast<int>(run);
    run += counts[i];
  }
  if (t == T - 1) {
    if (part[t] > 2147483647LL) record_error(error, kErrEdgeCapacity);
    row[n] = static_cast<int>(min(part[t], 2147483647LL));
  }
}

void invert3(const double* c, double* inv) {
  // inverse of the row matrix c (rows = lattice vectors)
  const double det = c[0] * (c[4] * c[8] - c[5] * c[7]) - c[1] * (c[3] * c[8] - c[5] * c[6]) + c[2] * (c[3] * c[7] - c[4] * c[6]);
  if (!(std::fabs(det) > 0) || !std::isfinite(det)) throw Error(4, "invalid (singular) cell");
  const double id = 1.0 / det;
  inv[0] = (c[4] * c[8] - c[5] * c[7]) * id;
  inv[1] = (c[2] * c[7] - c[1] * c[8]) * id;
  inv[2] = (c[1] * c[5] - c[2] * c[4]) * id;
  inv[3] = (c[5] * c[6] - c[3] * c[8]) * id;
  inv[4] = (c[0] * c[8] - c[2] * c[6]) * id;
  inv[5] = (c[2] * c[3] - c[0] * c[5]) * id;
  inv[6] = (c[3] * c[7] - c[4] * c[6]) * id;
  inv[7] = (c[1] * c[6] - c[0] * c[7]) * id;
  inv[8] = (c[0] * c[4] - c[1] * c[3]) * id;
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// model tables
// ------------------------------------------------------------------------------------------------
// A pass's graph program on the host (GraphProg, device_common.cuh).  Its structure depends on the
// model topology only and is built once per engine; each upload fills the coefficients: a fixed
// product coefficient, or the current rank weight w[widx] of a contraction row.
struct HostProg {
  std::vector<std::array<int, 4>> steps, comb;
  struct Rec { unsigned ab; int flush; int widx; double cfix; };
  std::vector<Rec> rows;  // [row][kWarp]
  int nfwd = 0, max_parts = 0;
  bool gate = false;
};

// The block program (BlockProg, graph_block.cuh) of a pass: its slots, and the lists of build_prog's
// steps -- term by term and chunk by chunk in that program's order -- dealt to a block's warps.
struct HostBlockProg {
  struct Term { int a, b, widx; double c; };
  struct Unit { Term t[2]; int target; bool chunk_end, list_end, step_end; };
  std::vector<Unit> units;
  std::vector<int> begin, basic_slot, basic_adj, zero_v, zero_adj, seed_v, seed_adj, keep, zero_late, rank_v, rank_adj;
  int nslots = 0, one = 0, warps = 0;
};

namespace {

struct Packer {
  std::vector<int> ints;
  int add_int(const std::vector<int>& v) { int o = static_cast<int>(ints.size()); ints.insert(ints.end(), v.begin(), v.end()); return o; }
};

// Offsets of a pass's parameter-dependent values in the value table.
struct PassOffsets { int coeff, scal, wc, wa; };
struct ValueOffsets {
  PassOffsets outer, gate;
  int linear, wmat, wmat_t, outer_w, gate_w;
};

// The parameter-dependent values in the device table's order (offsets are the same at every call).
template <typename Real>
ValueOffsets pack_values(const Model& m, std::vector<Real>& out) {
  out.clear();
  const int C = m.C, F = m.F, B = m.B;
  auto add = [&](const std::vector<double>& v) {
    const int o = static_cast<int>(out.size());
    for (double x : v) out.push_back(static_cast<Real>(x));
    return o;
  };
  auto pass = [&](bool gate) {
    PassOffsets o{};
    const bool own_radial = gate && m.gate_shared_radial;
    o.coeff = static_cast<int>(out.size());
    for (int mu = 0; mu < F; ++mu)
      for (int b = 0; b < B; ++b)
        out.push_back(static_cast<Real>(own_radial ? m.gate_radial[static_cast<size_t>(mu) * B + b]
                                                   : m.radial[static_cast<size_t>(mu) * (B + C) + b]));
    o.scal = add(gate && m.gate_decoupled ? m.gate_scal : m.scal);
    o.wc = static_cast<int>(out.size());
    for (int t = 0; t < C; ++t)
      for (int mu = 0; mu < F; ++mu)
        out.push_back(static_cast<Real>(gate ? m.gate_type[static_cast<size_t>(t) * F + mu]
                                             : m.radial[static_cast<size_t>(mu) * (B + C) + B + t]));
    o.wa = static_cast<int>(out.size());
    for (size_t q = 0; q < static_cast<size_t>(C) * F; ++q) out.push_back(static_cast<Real>(!gate && m.gated ? m.gate_add[q] : 0.0));
    return o;
  };
  ValueOffsets o{};
  o.outer = pass(false);
  o.gate = m.gated ? pass(true) : o.outer;
  o.linear = add(m.linear);
  o.wmat = static_cast<int>(out.size());
  if (m.gated)
    for (int mu = 0; mu < F; ++mu)
      for (int q = 0; q < m.Q; ++q) out.push_back(static_cast<Real>(m.gate_weight(mu, q)));
  o.wmat_t = static_cast<int>(out.size());
  if (m.gated)
    for (int q = 0; q < m.Q; ++q)
      for (int mu = 0; mu < F; ++mu) out.push_back(out[static_cast<size_t>(o.wmat) + static_cast<size_t>(mu) * m.Q + q]);
  o.outer_w = add(m.outer_w);
  o.gate_w = add(m.gate_w);
  return o;
}

// A program coefficient that is a rank weight: its place in the program image, and the weight.
struct WeightPatch { size_t at; int widx; bool gate; };
// One value of the device tables copied to its other places (rank weights into the programs).
struct ValueCopy { void* to; const void* from; };
template <typename Real>
__global__ void k_copy_values(const ValueCopy* list, int n) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) *static_cast<Real*>(list[q].to) = *static_cast<const Real*>(list[q].from);
}

// ---- per-atom graph program (see GraphProg in device_common.cuh) ----
struct ProgGroup {
  int target;
  std::vector<std::array<int, 2>> ab;
  std::vector<double> c;   // fixed coefficient (when widx < 0)
  std::vector<int> widx;   // rank-weight index, or -1
};

// One step: the groups' term lists cut into chunks of about total / 32 terms (at least 4), dealt
// longest first to the least-loaded lane; lists of several chunks sum through partial slots.
// Each lane's chunks become one term stream, stored lane-major and padded with zero terms.
void add_prog_step(HostProg& hp, const std::vector<ProgGroup>& groups, bool reverse, int one) {
  long long total = 0;
  for (const auto& g : groups) total += static_cast<long long>(g.ab.size());
  if (total == 0) return;
  const int T = std::max(4, static_cast<int>((total + kWarp - 1) / kWarp));
  struct Ch { int g, tb, te, flush; };
  std::vector<Ch> chs;
  const int comb_begin = static_cast<int>(hp.comb.size());
  int parts = 0;
  for (size_t gi = 0; gi < groups.size(); ++gi) {
    const int n = static_cast<int>(groups[gi].ab.size());
    if (!n) continue;
    if (n <= T) {
      chs.push_back({static_cast<int>(gi), 0, n, groups[gi].target});
      continue;
    }
    const int k = (n + T - 1) / T, slot0 = parts;
    for (int j = 0; j < k; ++j) chs.push_back({static_cast<int>(gi), j * n / k, (j + 1) * n / k, -(parts++ + 2)});
    hp.comb.push_back({groups[gi].target, slot0, parts, 0});
  }
  std::vector<int> order(chs.size());
  for (size_t i = 0; i < chs.size(); ++i) order[i] = static_cast<int>(i);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return chs[x].te - chs[x].tb > chs[y].te - chs[y].tb; });
  std::vector<int> lane_of(chs.size());
  long long load[kWarp] = {0};
  for (int i : order) {
    int best = 0;
    for (int l = 1; l < kWarp; ++l)
      if (load[l] < load[best]) best = l;
    lane_of[i] = best;
    load[best] += chs[i].te - chs[i].tb;
  }
  // Rows are filled one at a time: each lane takes a term of its current chunk (a chunk's terms
  // may be summed in any order), choosing the one whose two node reads share a shared-memory
  // bank (node index mod 32; equal nodes broadcast) with the fewest other lanes' reads of this
  // row, so that the warp's two loads per row are mostly conflict-free.
  std::vector<std::vector<int>> lane_chunks(kWarp);
  for (size_t i = 0; i < chs.size(); ++i) lane_chunks[lane_of[i]].push_back(static_cast<int>(i));
  std::vector<size_t> next_chunk(kWarp, 0);
  std::vector<std::vector<int>> pool(kWarp);  // remaining term indices of the lane's current chunk
  std::vector<int> cur(kWarp, -1);
  auto refill = [&](int l) {
    if (next_chunk[l] < lane_chunks[l].size()) {
      cur[l] = lane_chunks[l][next_chunk[l]++];
      for (int q = chs[cur[l]].tb; q < chs[cur[l]].te; ++q) pool[l].push_back(q);
    }
  };
  for (int l = 0; l < kWarp; ++l) refill(l);
  const int first = static_cast<int>(hp.rows.size() / kWarp);
  const HostProg::Rec pad{static_cast<unsigned>(one) | (static_cast<unsigned>(one) << 16), kProgNoFlush, -1, 0.0};
  struct Banks {  // distinct nodes read per bank in one row (at most one per lane)
    int n[kWarp], node[kWarp][kWarp];
    bool seen(int x) const {
      const unsigned b = static_cast<unsigned>(x) % kWarp;
      for (int q = 0; q < n[b]; ++q)
        if (node[b][q] == x) return true;
      return false;
    }
    int cost(int x) const { return n[static_cast<unsigned>(x) % kWarp] == 0 || seen(x) ? 0 : n[static_cast<unsigned>(x) % kWarp]; }
    void read(int x) {
      const unsigned b = static_cast<unsigned>(x) % kWarp;
      if (!seen(x)) node[b][n[b]++] = x;
    }
  };
  Banks bank_a, bank_b;
  int len = 0;
  for (;;) {
    bool any = false;
    for (int l = 0; l < kWarp; ++l) any = any || !pool[l].empty();
    if (!any) break;
    std::fill(bank_a.n, bank_a.n + kWarp, 0);
    std::fill(bank_b.n, bank_b.n + kWarp, 0);
    for (int l = 0; l < kWarp; ++l) {
      if (pool[l].empty()) { hp.rows.push_back(pad); continue; }
      const ProgGroup& g = groups[chs[cur[l]].g];
      size_t best = 0;
      int best_cost = 1 << 30;
      for (size_t k = 0; k < pool[l].size() && best_cost > 0; ++k) {  // (the first free one is best)
        const int c = bank_a.cost(g.ab[pool[l][k]][0]) + bank_b.cost(g.ab[pool[l][k]][1]);
        if (c < best_cost) { best_cost = c; best = k; }
      }
      const int q = pool[l][best];
      pool[l].erase(pool[l].begin() + static_cast<long>(best));
      const int a = g.ab[q][0], b = g.ab[q][1];
      bank_a.read(a);
      bank_b.read(b);
      const bool last = pool[l].empty();
      hp.rows.push_back({static_cast<unsigned>(a) | (static_cast<unsigned>(b) << 16), last ? chs[cur[l]].flush : kProgNoFlush,
                         g.widx[q], g.c[q]});
      if (last) refill(l);
    }
    ++len;
  }
  hp.steps.push_back({first, len, comb_begin, (static_cast<int>(hp.comb.size()) << 1) | (reverse ? 1 : 0)});
  hp.max_parts = std::max(hp.max_parts, parts);
}

// The pass's rank contraction and product graph as a program: forward (contraction, graph levels
// 1..L), then reverse (graph levels L-1..0, contraction); node M is the constant 1.
HostProg build_prog(const Model& m, bool gate) {
  if (m.M + 1 > 65535) throw Error(3, "SUS2 model: too many moment nodes for the per-atom program");
  HostProg hp;
  hp.gate = gate;
  const int one = m.M;
  const auto& rows = gate ? m.gate_rows : m.outer_rows;
  const GraphSchedule& g = gate ? m.gate_graph : m.outer_graph;
  std::vector<std::vector<int>> by_dst(m.M), by_src(m.M);
  for (int q = 0; q < static_cast<int>(rows.size()); ++q) {
    by_dst[rows[q].dst].push_back(q);
    by_src[rows[q].src].push_back(q);
  }
  std::vector<int> dsts;
  for (int d = 0; d < m.M; ++d)
    if (!by_dst[d].empty()) dsts.push_back(d);
  {
    std::vector<ProgGroup> gs;
    for (int d : dsts) {
      ProgGroup pg{d, {}, {}, {}};
      for (int q : by_dst[d]) { pg.ab.push_back({rows[q].src, one}); pg.c.push_back(1.0); pg.widx.push_back(rows[q].widx); }
      gs.push_back(std::move(pg));
    }
    add_prog_step(hp, gs, false, one);
  }
  for (int lv = 0; lv < g.levels; ++lv) {
    std::vector<ProgGroup> gs;
    for (int q = g.level_begin[lv]; q < g.level_begin[lv + 1]; ++q) {
      ProgGroup pg{g.out_nodes[q], {}, {}, {}};
      for (int p = g.out_begin[q]; p < g.out_begin[q + 1]; ++p) {
        const Product& pr = m.products[g.fprod[p]];
        pg.ab.push_back({pr.a, pr.b});
        pg.c.push_back(pr.c);
        pg.widx.push_back(-1);
      }
      gs.push_back(std::move(pg));
    }
    add_prog_step(hp, gs, false, one);
  }
  hp.nfwd = static_cast<int>(hp.steps.size());
  for (int lv = static_cast<int>(g.rlevel_begin.size()) - 2; lv >= 0; --lv) {
    std::vector<ProgGroup> gs;
    for (int q = g.rlevel_begin[lv]; q < g.rlevel_begin[lv + 1]; ++q) {
      ProgGroup pg{g.in_nodes[q], {}, {}, {}};
      for (int e = g.in_begin[q]; e < g.in_begin[q + 1]; ++e) {
        pg.ab.push_back({g.rprod_out[e], g.rprod_other[e]});
        pg.c.push_back(g.rprod_c[e]);
        pg.widx.push_back(-1);
      }
      gs.push_back(std::move(pg));
    }
    add_prog_step(hp, gs, true, one);
  }
  {
    std::vector<ProgGroup> gs;
    for (int b = 0; b < m.NB; ++b) {
      ProgGroup pg{b, {}, {}, {}};
      for (int q : by_src[b]) { pg.ab.push_back({rows[q].dst, one}); pg.c.push_back(1.0); pg.widx.push_back(rows[q].widx); }
      gs.push_back(std::move(pg));
    }
    add_prog_step(hp, gs, true, one);
  }
  return hp;
}

// dual: the gradient's program.  Its rank-weight gradients read the contraction's source values just
// before the contraction's reverse, the last step, which the streams then set apart.
HostBlockProg build_block_prog(const Model& m, const HostProg& hp, const std::vector<int>& basic_of, bool dual) {
  HostBlockProg bp;
  const int nsteps = static_cast<int>(hp.steps.size());
  const std::vector<int>& seeds = hp.gate ? m.gate_nodes : m.scalar_map;
  const int one = m.M;
  // each step's target lists from the lane streams: a chunk is a lane's terms up to a flush (rows
  // first .. first + n - 1 of that lane), a list its chunks begin .. end - 1
  struct Chunk { int lane, first, n; };
  struct List { int target, begin, end; };
  std::vector<Chunk> chunks;
  std::vector<std::vector<List>> steps(nsteps);
  chunks.reserve(hp.rows.size() / 2);
  auto rec = [&](const Chunk& c, int i) -> const HostProg::Rec& { return hp.rows[static_cast<size_t>(c.first + i) * kWarp + c.lane]; };
  std::vector<char> in_v(m.M, 0), in_adj(m.M, 0), rev_b(m.M, 0), early(m.M, 0), rank_src(m.M, 0);
  const std::vector<ContractionRow>& rank_rows = hp.gate ? m.gate_rows : m.outer_rows;
  const bool apart = dual && !rank_rows.empty();
  if (dual)
    for (const auto& r : rank_rows)
      if (r.widx >= 0) rank_src[r.src] = 1;
  for (int st = 0; st < nsteps; ++st) {
    const auto& info = hp.steps[st];
    const bool rev = (info[3] & 1) != 0;
    std::vector<Chunk> parts;
    const bool last = apart && st + 1 == nsteps;
    auto mark = [&](int target) {
      (rev ? in_adj : in_v)[target] = 1;
      if (rev && !last) early[target] = 1;
    };
    for (int lane = 0; lane < kWarp; ++lane) {
      Chunk c{lane, info[0], 0};
      for (int i = 0; i < info[1]; ++i) {
        ++c.n;
        const int flush = rec(c, c.n - 1).flush;
        if (flush == kProgNoFlush) continue;
        for (int k = 0; k < c.n; ++k) {
          const unsigned ab = rec(c, k).ab;
          const int x = static_cast<int>(ab & 0xffffu), y = static_cast<int>(ab >> 16);
          if (x != one) mark(x);
          if (y != one) { in_v[y] = 1; if (rev) rev_b[y] = 1; }
        }
        if (flush >= 0) {
          mark(flush);
          const int b = static_cast<int>(chunks.size());
          chunks.push_back(c);
          steps[st].push_back({flush, b, b + 1});
        } else {
          if (static_cast<size_t>(-flush - 2) >= parts.size()) parts.resize(static_cast<size_t>(-flush - 1));
          parts[-flush - 2] = c;
        }
        c = Chunk{lane, c.first + c.n, 0};  // (what follows a lane's last flush is padding)
      }
    }
    for (int q = info[2]; q < (info[3] >> 1); ++q) {
      const auto& c = hp.comb[q];
      const int b = static_cast<int>(chunks.size());
      for (int p = c[1]; p < c[2]; ++p) chunks.push_back(parts[p]);
      mark(c[0]);
      steps[st].push_back({c[0], b, static_cast<int>(chunks.size())});
    }
  }
  // slots: moments in (k, h) order, the other values, the constant, then adjoints; an adjoint takes
  // its node's value slot when the reverse never reads the value
  std::vector<int> vslot(m.M, -1), aslot(m.M, -1);
  int n = 0;
  std::vector<char> is_basic(m.M, 0), is_seed(m.M, 0);
  for (int b : basic_of)
    if (b >= 0) { is_basic[b] = 1; in_adj[b] = 1; if (vslot[b] < 0) vslot[b] = n++; }
  for (int q : seeds) { is_seed[q] = 1; in_v[q] = in_adj[q] = early[q] = 1; }
  for (int q = 0; q < m.M; ++q)
    if (in_v[q] && vslot[q] < 0) {
      vslot[q] = n++;
      bp.zero_v.push_back(vslot[q]);
    }
  bp.one = n++;
  for (int q = 0; q < m.M; ++q)
    if (in_adj[q]) {
      const bool share = vslot[q] >= 0 && !rev_b[q] && !(rank_src[q] && early[q]);
      aslot[q] = share ? vslot[q] : n++;
      if (share && rank_src[q]) bp.zero_late.push_back(aslot[q]);
      else if (!is_seed[q]) bp.zero_adj.push_back(aslot[q]);
    }
  if (n > kGraphMaxSlots) return HostBlockProg{};
  bp.nslots = n;
  const int warps = bp.warps = graph_program_warps(n, m.F, m.S);
  for (int b : basic_of) {
    bp.basic_slot.push_back(b >= 0 ? vslot[b] : -1);
    bp.basic_adj.push_back(b >= 0 ? aslot[b] : -1);
  }
  for (int q : seeds) { bp.seed_v.push_back(vslot[q]); bp.seed_adj.push_back(aslot[q]); }
  for (int q = 0; q < m.M; ++q)
    if (rev_b[q] || rank_src[q]) bp.keep.push_back(vslot[q]);
  if (dual) {
    std::vector<const ContractionRow*> by_weight;
    for (const auto& r : rank_rows)
      if (r.widx >= 0 && r.widx < static_cast<int>((hp.gate ? m.gate_w : m.outer_w).size())) by_weight.push_back(&r);
    std::stable_sort(by_weight.begin(), by_weight.end(), [](const ContractionRow* x, const ContractionRow* y) { return x->widx < y->widx; });
    for (const ContractionRow* r : by_weight) {
      bp.rank_v.push_back(vslot[r->src]);
      bp.rank_adj.push_back(aslot[r->dst]);
    }
  }
  // streams: lists longest first onto the least-loaded warp
  const HostBlockProg::Term pad{bp.one, bp.one, -1, 0.0};
  std::vector<std::vector<HostBlockProg::Unit>> stream(warps);
  std::vector<int> fwd_end(warps, 0), last_begin(warps, -1);
  auto fours = [&](std::vector<HostBlockProg::Unit>& v) {
    while (v.size() % 4) v.push_back({{pad, pad}, 0, false, false, false});
  };
  for (int st = 0; st < nsteps; ++st) {
    const bool rev = (hp.steps[st][3] & 1) != 0;
    std::vector<size_t> cost, order;
    for (const List& l : steps[st]) {
      size_t c = 1;
      for (int q = l.begin; q < l.end; ++q) c += static_cast<size_t>((chunks[q].n + 1) / 2);
      order.push_back(cost.size());
      cost.push_back(c);
    }
    std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) { return cost[x] > cost[y]; });
    if (apart && st + 1 == nsteps)
      for (int w = 0; w < warps; ++w) {
        fours(stream[w]);
        last_begin[w] = static_cast<int>(stream[w].size());
      }
    std::vector<size_t> load(warps, 0);
    for (size_t q : order) {
      const int w = static_cast<int>(std::min_element(load.begin(), load.end()) - load.begin());
      load[w] += cost[q];
      const List& l = steps[st][q];
      for (int c = l.begin; c < l.end; ++c) {
        const Chunk& ch = chunks[c];
        for (int i = 0; i < ch.n; i += 2) {
          HostBlockProg::Unit u{{pad, pad}, 0, false, false, false};
          for (int k = 0; k < 2 && i + k < ch.n; ++k) {
            const HostProg::Rec& t = rec(ch, i + k);
            const int x = static_cast<int>(t.ab & 0xffffu), y = static_cast<int>(t.ab >> 16);
            u.t[k] = {x == one ? bp.one : (rev ? aslot : vslot)[x], y == one ? bp.one : vslot[y], t.widx, t.cfix};
          }
          if (i + 2 >= ch.n) {
            u.chunk_end = true;
            u.list_end = c + 1 == l.end;
            u.target = (rev ? aslot : vslot)[l.target];
          }
          stream[w].push_back(u);
        }
      }
    }
    // the step's last unit carries the barrier (a unit of its own for a warp without lists)
    for (int w = 0; w < warps; ++w) {
      if (load[w] == 0) stream[w].push_back({{pad, pad}, 0, false, false, false});
      stream[w].back().step_end = true;
      if (st + 1 == hp.nfwd) {
        fours(stream[w]);
        fwd_end[w] = static_cast<int>(stream[w].size());
      }
    }
  }
  for (int w = 0; w < warps; ++w) {
    fours(stream[w]);
    const int first = static_cast<int>(bp.units.size());
    bp.begin.push_back(first);
    bp.begin.push_back(first + fwd_end[w]);
    bp.begin.push_back(first + (last_begin[w] >= 0 ? last_begin[w] : static_cast<int>(stream[w].size())));
    bp.units.insert(bp.units.end(), stream[w].begin(), stream[w].end());
    bp.begin.push_back(static_cast<int>(bp.units.size()));
  }
  bp.units.insert(bp.units.end(), 4, {{pad, pad}, 0, false, false, false});  // (an empty last stream's first read)
  return bp;
}

// Serialises the block programs into one 16-byte aligned device image and binds them.
void upload_block_progs(const Model& m, const HostBlockProg* const (&progs)[2], DevBuf& buf, cudaStream_t s,
                        BlockProg (&out)[2], std::vector<WeightPatch>& patches) {
  std::vector<unsigned char> img;
  auto put = [&](const void* p, size_t n) {
    const size_t o = (img.size() + 15) & ~size_t(15);
    img.resize(o + std::max<size_t>(n, 16));
    if (n) std::memcpy(img.data() + o, p, n);
    return o;
  };
  size_t off[2][12];
  for (int k = 0; k < 2; ++k) {
    const HostBlockProg& bp = *progs[k];
    const std::vector<double>& w = k ? m.gate_w : m.outer_w;
    std::vector<int4> units(bp.units.size());
    for (size_t q = 0; q < units.size(); ++q) {
      const auto& u = bp.units[q];
      unsigned x[2];
      float c[2];
      for (int i = 0; i < 2; ++i) {
        x[i] = (static_cast<unsigned>(u.t[i].a) << 7) | (static_cast<unsigned>(u.t[i].b) << 20);
        c[i] = static_cast<float>(u.t[i].widx >= 0 ? w[u.t[i].widx] : u.t[i].c);
      }
      x[0] |= static_cast<unsigned>(u.target) & 127u;
      x[1] |= static_cast<unsigned>(u.target) >> 7;
      if (u.chunk_end) x[1] |= kUnitChunkEnd;
      if (u.list_end) x[1] |= kUnitListEnd;
      if (u.step_end) x[1] |= kUnitStepEnd;
      int y[2];
      std::memcpy(y, c, sizeof(y));
      units[q] = make_int4(static_cast<int>(x[0]), y[0], static_cast<int>(x[1]), y[1]);
    }
    off[k][0] = put(units.data(), sizeof(int4) * units.size());
    for (size_t q = 0; q < units.size(); ++q)
      for (int i = 0; i < 2; ++i)
        if (bp.units[q].t[i].widx >= 0)
          patches.push_back({off[k][0] + sizeof(int4) * q + sizeof(int) * (i ? 3 : 1), bp.units[q].t[i].widx, k == 1});
    const std::vector<int>* lists[] = {&bp.begin, &bp.basic_slot, &bp.basic_adj, &bp.zero_v, &bp.zero_adj, &bp.seed_v, &bp.seed_adj,
                                       &bp.keep, &bp.zero_late, &bp.rank_v, &bp.rank_adj};
    for (int i = 0; i < 11; ++i) off[k][1 + i] = put(lists[i]->data(), sizeof(int) * lists[i]->size());
  }
  buf.ensure(img.size());
  SUS2G_CUDA(cudaMemcpyAsync(buf.ptr, img.data(), img.size(), cudaMemcpyHostToDevice, s));
  SUS2G_CUDA(cudaStreamSynchronize(s));
  const unsigned char* base = static_cast<const unsigned char*>(buf.ptr);
  for (int k = 0; k < 2; ++k) {
    const HostBlockProg& bp = *progs[k];
    auto ints = [&](int i) { return reinterpret_cast<const int*>(base + off[k][i]); };
    BlockProg g;
    g.nslots = bp.nslots; g.one = bp.one; g.warps = bp.warps;
    g.nzero_v = static_cast<int>(bp.zero_v.size());
    g.nzero_adj = static_cast<int>(bp.zero_adj.size());
    g.nkeep = static_cast<int>(bp.keep.size());
    g.units = reinterpret_cast<const int4*>(base + off[k][0]);
    g.begin = ints(1); g.basic_slot = ints(2); g.basic_adj = ints(3); g.zero_v = ints(4); g.zero_adj = ints(5);
    g.seed_v = ints(6); g.seed_adj = ints(7);
    g.nzero_late = static_cast<int>(bp.zero_late.size());
    g.keep = ints(8); g.zero_late = ints(9); g.rank_v = ints(10); g.rank_adj = ints(11);
    out[k] = g;
  }
}

// Serialises the programs of the passes into one 16-byte aligned device image and binds them.
template <typename Real>
void upload_progs(const Model& m, const std::vector<const HostProg*>& progs, DevBuf& buf, cudaStream_t s,
                  std::vector<GraphProg<Real>>& out, std::vector<WeightPatch>& patches) {
  std::vector<unsigned char> img;
  auto put = [&](const void* p, size_t n) {
    const size_t o = (img.size() + 15) & ~size_t(15);
    img.resize(o + n);
    if (n) std::memcpy(img.data() + o, p, n);
    return o;
  };
  struct Off { size_t steps, comb, rows; };
  std::vector<Off> offs;
  for (const HostProg* hp : progs) {
    Off o{};
    o.steps = put(hp->steps.data(), sizeof(int4) * hp->steps.size());
    o.comb = put(hp->comb.data(), sizeof(int4) * hp->comb.size());
    const std::vector<double>& w = hp->gate ? m.gate_w : m.outer_w;
    std::vector<ProgRec<Real>> rows(hp->rows.size());
    for (size_t q = 0; q < rows.size(); ++q) {
      const HostProg::Rec& x = hp->rows[q];
      rows[q] = ProgRec<Real>{};
      rows[q].ab = x.ab;
      rows[q].flush = x.flush;
      rows[q].c = static_cast<Real>(x.widx >= 0 ? w[x.widx] : x.cfix);
    }
    o.rows = put(rows.data(), sizeof(ProgRec<Real>) * rows.size());
    for (size_t q = 0; q < rows.size(); ++q)
      if (hp->rows[q].widx >= 0)
        patches.push_back({o.rows + static_cast<size_t>(reinterpret_cast<const char*>(&rows[q].c) - reinterpret_cast<const char*>(rows.data())),
                         hp->rows[q].widx, hp->gate});
    offs.push_back(o);
  }
  if (img.empty()) img.resize(16);
  buf.ensure(img.size());
  SUS2G_CUDA(cudaMemcpyAsync(buf.ptr, img.data(), img.size(), cudaMemcpyHostToDevice, s));
  SUS2G_CUDA(cudaStreamSynchronize(s));
  const unsigned char* base = static_cast<const unsigned char*>(buf.ptr);
  out.clear();
  for (size_t k = 0; k < progs.size(); ++k) {
    GraphProg<Real> g;
    g.nsteps = static_cast<int>(progs[k]->steps.size());
    g.nfwd = progs[k]->nfwd;
    g.max_parts = progs[k]->max_parts;
    g.steps = reinterpret_cast<const int4*>(base + offs[k].steps);
    g.comb = reinterpret_cast<const int4*>(base + offs[k].comb);
    g.rows = reinterpret_cast<const ProgRec<Real>*>(base + offs[k].rows);
    out.push_back(g);
  }
}

template <typename Real>
PassTables<Real> bind_pass(const PassOffsets& o, int ndst, const Real* R) {
  PassTables<Real> t{};
  t.coeff = R + o.coeff; t.scal = R + o.scal; t.wcenter = t.wsource = R + o.wc; t.wadd = R + o.wa;
  t.ndst = ndst;
  return t;
}

}  // namespace

Engine::Engine(const Model& model, int device, int precision) : model_(model), device_(device), precision_(precision) {
  if (precision != kFP64 && precision != kFP32) throw Error(1, "precision must be 0 (FP64) or 1 (FP32 bulk)");
  pdl_ = default_pdl();
  SUS2G_CUDA(cudaSetDevice(device));
  SUS2G_CUDA(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device));
  SUS2G_CUDA(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking));
  stream_ = own_stream_;
  // the second stream runs the reverse-edge search beside the first pass: at the most urgent
  // priority, so that its blocks take SM slots ahead of that pass's pending blocks
  int least = 0;
  SUS2G_CUDA(cudaDeviceGetStreamPriorityRange(&least, &urgent_priority_));
  SUS2G_CUDA(cudaStreamCreateWithPriority(&aux_stream_, cudaStreamNonBlocking, urgent_priority_));
  for (cudaEvent_t* e : {&ev_fork_, &ev_rev_, &ev_fork2_, &ev_join2_})
    SUS2G_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  // scalar readout and gate nodes are written with plain stores; duplicates would race
  auto unique = [](std::vector<int> v) { std::sort(v.begin(), v.end()); return std::adjacent_find(v.begin(), v.end()) == v.end(); };
  if (!unique(model_.scalar_map)) throw Error(3, "SUS2 model: duplicate entries in alpha_moment_mapping");
  if (model_.gated && !unique(model_.gate_nodes)) throw Error(3, "SUS2 model: duplicate gate scalar moments");
  if (model_.K > kMaxK) throw Error(3, "SUS2 model: sh_k_max above 8 is not supported by the GPU engine");
  plans_ = new std::vector<FramePlan>();
  weight_copies_ = new std::vector<ValueCopy>();
  SUS2G_CUDA(cudaMallocHost(&host_total_, 8 * sizeof(int)));
  // [0] error code, [1] cell-list edge capacity overflow (largest count), [2] bin capacity overflow
  error_.ensure(3 * sizeof(int));
  SUS2G_CUDA(cudaMemsetAsync(error_.ptr, 0, 3 * sizeof(int), stream_));
  // the dynamic centre order's counters: zero now; each launch's last warp zeroes its pair again
  work_.ensure(sizeof(int) * kWorkInts);
  SUS2G_CUDA(cudaMemsetAsync(work_.ptr, 0, sizeof(int) * kWorkInts, stream_));
  upload_model();
}

Engine::~Engine() {
  reset_step_graph();
  delete plans_;
  delete static_cast<std::vector<ValueCopy>*>(weight_copies_);
  if (host_total_) cudaFreeHost(host_total_);
  if (pinned_) cudaFreeHost(pinned_);
  for (cudaEvent_t e : event_pool_) cudaEventDestroy(e);
  if (precision_ == kFP32) delete static_cast<DevModel<float>*>(dev_model_);
  else delete static_cast<DevModel<double>*>(dev_model_);
  for (cudaEvent_t e : {ev_fork_, ev_rev_, ev_fork2_, ev_join2_})
    if (e) cudaEventDestroy(e);
  if (aux_stream_) cudaStreamDestroy(aux_stream_);
  if (own_stream_) cudaStreamDestroy(own_stream_);
}

// Work on the second stream forks from the engine stream after an event and joins it back
// before the first consumer; the stage timer keeps everything on one stream.
bool Engine::may_fork() const { return !timing_; }

void Engine::wait_reverse() {
  if (!rev_pending_) return;
  SUS2G_CUDA(cudaStreamWaitEvent(stream_, ev_rev_, 0));
  rev_pending_ = false;
}

namespace {
// basic index of (k, l, m) at k H + l l + l + m, -1 when absent
std::vector<int> basic_table(const Model& m) {
  std::vector<int> t(static_cast<size_t>(m.K) * m.H, -1);
  for (int b = 0; b < m.NB; ++b) {
    const auto& q = m.basic[b];
    t[static_cast<size_t>(q[0]) * m.H + q[1] * q[1] + q[1] + q[2]] = b;
  }
  return t;
}
}  // namespace

// The device tables at the current parameters.  The first call builds and uploads the structure
// (index lists, graph programs, gradient layout); later ones send the parameter-dependent values and
// copy the rank weights into the programs on the device.
template <typename Real>
void Engine::upload_tables() {
  const Model& m = model_;
  const cudaStream_t us = stream_;
  // species and shift (FP64), then the values; the host copies die at return, hence the
  // synchronisation at the end (which also orders the tables before work on any later stream)
  std::vector<Real> values;
  const ValueOffsets vo = pack_values<Real>(m, values);
  const size_t dbl_bytes = sizeof(double) * 2 * static_cast<size_t>(m.C), bytes = dbl_bytes + sizeof(Real) * values.size();
  std::vector<unsigned char> img(bytes);
  std::memcpy(img.data(), m.species.data(), dbl_bytes / 2);
  std::memcpy(img.data() + dbl_bytes / 2, m.shift.data(), dbl_bytes / 2);
  std::memcpy(img.data() + dbl_bytes, values.data(), sizeof(Real) * values.size());
  tab_value_.ensure(bytes);
  SUS2G_CUDA(cudaMemcpyAsync(tab_value_.ptr, img.data(), bytes, cudaMemcpyHostToDevice, us));
  const Real* R = reinterpret_cast<const Real*>(tab_value_.as<unsigned char>() + dbl_bytes);
  if (dev_model_) {
    static_cast<DevModel<Real>*>(dev_model_)->scaling = Real(m.scaling);
    copy_weights<Real>();
    SUS2G_CUDA(cudaStreamSynchronize(us));
    return;
  }
  Packer pk;
  const int o_basic = pk.add_int(basic_table(m)), o_map = pk.add_int(m.scalar_map), o_nodes = pk.add_int(m.gate_nodes);
  // parameter-gradient layout: block offsets in the trainer's order and rank-weight row lists
  std::map<std::string, int> off;
  for (const auto& b : m.layout()) off[b.name] = b.offset;
  auto block = [&](const char* n) { auto it = off.find(n); return it == off.end() ? -1 : it->second; };
  auto weight_rows = [&](const std::vector<ContractionRow>& rows, int nw, int& o_begin, int& o_src, int& o_dst) {
    std::vector<std::vector<const ContractionRow*>> of(nw);
    for (const auto& r : rows)
      if (r.widx >= 0 && r.widx < nw) of[r.widx].push_back(&r);
    std::vector<int> begin{0}, src, dst;
    for (const auto& list : of) {
      for (const ContractionRow* r : list) { src.push_back(r->src); dst.push_back(r->dst); }
      begin.push_back(static_cast<int>(src.size()));
    }
    o_begin = pk.add_int(begin);
    o_src = pk.add_int(src);
    o_dst = pk.add_int(dst);
  };
  GradLayout gl{};
  int ow_b = 0, ow_s = 0, ow_d = 0, gw_b = 0, gw_s = 0, gw_d = 0;
  gl.shift_off = block("shift_coeffs");
  gl.species_off = block("species_coeffs");
  gl.linear_off = block("moment_coeffs");
  gl.gate_w_off = block("two_layer_gate_weights");
  gl.nparams = m.param_count();
  gl.outer.coeff_off = block("radial_coeffs");
  gl.outer.coeff_stride = m.B + m.C;
  gl.outer.scal_off = block("scal_coeffs");
  gl.outer.wc_off = block("radial_coeffs") + m.B;
  gl.outer.wc_mu_stride = m.B + m.C;
  gl.outer.wc_t_stride = 1;
  gl.outer.add_off = block("two_layer_gate_additive_coeffs");
  gl.outer.rw_off = block("outer_k_rank1_weights");
  gl.outer.nw = static_cast<int>(m.outer_w.size());
  weight_rows(m.outer_rows, gl.outer.nw, ow_b, ow_s, ow_d);
  if (m.gated) {
    gl.gate.coeff_off = m.gate_shared_radial ? block("two_layer_gate_radial_coeffs") : block("radial_coeffs");
    gl.gate.coeff_stride = m.gate_shared_radial ? m.B : m.B + m.C;
    gl.gate.scal_off = m.gate_decoupled ? block("two_layer_gate_scaling_coeffs") : block("scal_coeffs");
    gl.gate.wc_off = block("two_layer_gate_type_coeffs");
    gl.gate.wc_mu_stride = 1;
    gl.gate.wc_t_stride = m.F;
    gl.gate.add_off = -1;
    gl.gate.rw_off = block("two_layer_gate_k_rank_weights");
    gl.gate.nw = static_cast<int>(m.gate_w.size());
    weight_rows(m.gate_rows, gl.gate.nw, gw_b, gw_s, gw_d);
  }
  if (pk.ints.empty()) pk.ints.push_back(0);
  tab_int_.ensure(sizeof(int) * pk.ints.size());
  // stream-ordered copies: the engine stream is non-blocking, so a legacy-stream copy would not
  // order against its next kernel; the host vectors die at return, hence the synchronisation below
  SUS2G_CUDA(cudaMemcpyAsync(tab_int_.ptr, pk.ints.data(), sizeof(int) * pk.ints.size(), cudaMemcpyHostToDevice, us));
  const int* I = tab_int_.as<int>();
  auto* dm = new DevModel<Real>();
  dev_model_ = dm;
  dm->C = m.C; dm->L = m.L; dm->K = m.K; dm->B = m.B; dm->F = m.F; dm->H = m.H; dm->M = m.M; dm->NB = m.NB;
  dm->S = m.S; dm->Q = m.Q; dm->nblk = m.nblk; dm->scaling_mode = m.scaling_mode;
  dm->rmax = Real(m.max_dist); dm->rang = Real(m.angular); dm->scaling = Real(m.scaling);
  dm->split = m.split; dm->poly = m.poly_cutoff; dm->cutoff_p = m.cutoff_p; dm->gated = m.gated;
  dm->species_readout = m.species_readout;
  dm->basic_of = I + o_basic;
  auto ndst = [](const std::vector<ContractionRow>& rows) {
    std::vector<int> d;
    for (const auto& r : rows) d.push_back(r.dst);
    std::sort(d.begin(), d.end());
    return static_cast<int>(std::unique(d.begin(), d.end()) - d.begin());
  };
  dm->outer = bind_pass<Real>(vo.outer, ndst(m.outer_rows), R);
  dm->gate = m.gated ? bind_pass<Real>(vo.gate, ndst(m.gate_rows), R) : dm->outer;
  weight_value_[0] = R + vo.outer_w;
  weight_value_[1] = R + vo.gate_w;
  prog_[0].reset(new HostProg(build_prog(m, false)));
  prog_[1].reset(new HostProg(m.gated ? build_prog(m, true) : HostProg{}));
  {
    std::vector<GraphProg<Real>> bound;
    std::vector<WeightPatch> patches;
    upload_progs<Real>(m, {prog_[0].get(), prog_[1].get()}, tab_prog_, us, bound, patches);
    add_weight_copies<Real>(tab_prog_.ptr, &patches);
    dm->outer.prog = bound[0];
    dm->gate.prog = m.gated ? bound[1] : bound[0];
    dm->prog_parts = std::max(bound[0].max_parts, m.gated ? bound[1].max_parts : 0);
  }
  dm->linear = R + vo.linear;
  dm->species = tab_value_.as<double>();
  dm->shift = tab_value_.as<double>() + m.C;
  dm->scalar_map = I + o_map;
  dm->gate_wmat = R + vo.wmat;
  dm->gate_wmat_t = R + vo.wmat_t;
  dm->gate_nodes = I + o_nodes;
  gl.outer.w_begin = I + ow_b; gl.outer.w_src = I + ow_s; gl.outer.w_dst = I + ow_d;
  gl.gate.w_begin = I + gw_b; gl.gate.w_src = I + gw_s; gl.gate.w_dst = I + gw_d;
  dm->grad = gl;
  if (sizeof(Real) == 4 && m.B == 8) upload_block_programs(false);
  SUS2G_CUDA(cudaStreamSynchronize(us));
}

// The places of a program image that hold rank weights join the list of copies (sent to the device
// at the next parameter upload: an engine that never gets one needs no list there).
template <typename Real>
void Engine::add_weight_copies(void* image, const void* weight_patches) {
  auto& list = *static_cast<std::vector<ValueCopy>*>(weight_copies_);
  for (const WeightPatch& p : *static_cast<const std::vector<WeightPatch>*>(weight_patches))
    list.push_back({static_cast<unsigned char*>(image) + p.at, static_cast<const Real*>(weight_value_[p.gate ? 1 : 0]) + p.widx});
}
template <typename Real>
void Engine::copy_weights() {
  const auto& list = *static_cast<std::vector<ValueCopy>*>(weight_copies_);
  const int n = static_cast<int>(list.size());
  if (n == 0) return;
  if (copies_sent_ != list.size()) {
    tab_copies_.ensure(sizeof(ValueCopy) * list.size());
    SUS2G_CUDA(cudaMemcpyAsync(tab_copies_.ptr, list.data(), sizeof(ValueCopy) * list.size(), cudaMemcpyHostToDevice, stream_));
    copies_sent_ = list.size();
  }
  k_copy_values<Real><<<(n + 255) / 256, 256, 0, stream_>>>(tab_copies_.as<ValueCopy>(), n);
  SUS2G_CUDA(cudaGetLastError());
}

// The block programs of the split passes, built with the tables, or (dual) of the split gradient,
// built at its first use.
void Engine::upload_block_programs(bool dual) {
  const Model& m = model_;
  auto* dm = static_cast<DevModel<float>*>(dev_model_);
  const std::vector<int> basic_of = basic_table(m);
  HostBlockProg host[2];
  host[0] = build_block_prog(m, *prog_[0], basic_of, dual);
  if (m.gated) host[1] = build_block_prog(m, *prog_[1], basic_of, dual);
  BlockProg blocks[2];
  const HostBlockProg* const hosts[2] = {&host[0], &host[1]};
  DevBuf& buf = dual ? tab_dual_ : tab_block_;
  std::vector<WeightPatch> patches;
  upload_block_progs(m, hosts, buf, stream_, blocks, patches);
  add_weight_copies<float>(buf.ptr, &patches);
  (dual ? dm->outer.dual : dm->outer.block) = blocks[0];
  (dual ? dm->gate.dual : dm->gate.block) = blocks[1];
  if (dual) have_dual_ = true;
}

// Takes the parameters (and scaling) of a model of the same structure, as a new engine for it would
// start: settings at their defaults, no geometry, the caller's stream released.
bool Engine::take_params(const Model& m) {
  if (!model_.same_structure(m)) return false;
  SUS2G_CUDA(cudaSetDevice(device_));
  // what was queued on any stream that the engine was given may still read the tables (the caller's
  // stream itself may be gone by now, so it is not named here)
  SUS2G_CUDA(cudaDeviceSynchronize());
  rev_pending_ = false;
  reset_step_graph();
  stream_ = own_stream_;
  std::vector<double> p(static_cast<size_t>(m.param_count()));
  m.get_params(p.data());
  model_.set_params(p.data());
  model_.scaling = m.scaling;
  step_graphs_ = true;
  pdl_ = default_pdl();
  moment_mma_ = false;
  grad_split_ = true;
  set_timing(false);
  open_stage_ = -1;
  for (int q = 0; q < 4; ++q) {
    pass_blocks_[q] = pass_grid_[q] = pass_order_[q] = pass_stage_[q] = 0;
    pass_wpb_[q] = 0;
  }
  std::fill(std::begin(ran_warps_), std::end(ran_warps_), 0);
  static_split_ = gate_split_ = -1;
  split_blocks_ = gate_split_blocks_[0] = gate_split_blocks_[1] = 0;
  gate_ran_split_ = false;
  staged_ = 0;
  desc_out_ = nullptr;
  natoms_ = nframes_ = ncentres_ = bins_frames_ = 0;
  nedges_ = exact_edges_ = 0;
  nedges_exact_ = true;
  user_edges_ = padded_ = clear_bins_ = false;
  plans_->clear();
  launches_ = 0;
  ++edge_generation_;
  SUS2G_CUDA(cudaMemsetAsync(error_.ptr, 0, 3 * sizeof(int), stream_));
  upload_model();
  return true;
}

void Engine::upload_model() {
  SUS2G_CUDA(cudaSetDevice(device_));
  // work already queued on the engine's stream may still read the tables being replaced
  if (stream_) SUS2G_CUDA(cudaStreamSynchronize(stream_));
  reset_step_graph();  // a captured step holds the old tables' values
  if (precision_ == kFP32) upload_tables<float>();
  else upload_tables<double>();
}

long long Engine::nedges() {
  wait_reverse();
  if (!nedges_exact_ && user_edges_) {
    int total = 0;
    SUS2G_CUDA(cudaMemcpyAsync(&total, row_.as<int>() + natoms_, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    SUS2G_CUDA(cudaStreamSynchronize(stream_));
    exact_edges_ = total;
    nedges_exact_ = true;
  }
  if (!nedges_exact_) {
    // padded layout: the sum of the per-centre counts
    std::vector<int> counts(static_cast<size_t>(std::max(0, ncentres_)));
    if (ncentres_)
      SUS2G_CUDA(cudaMemcpyAsync(counts.data(), counts_.ptr, sizeof(int) * ncentres_, cudaMemcpyDeviceToHost, stream_));
    SUS2G_CUDA(cudaStreamSynchronize(stream_));
    exact_edges_ = 0;
    for (int c : counts) exact_edges_ += c;
    nedges_exact_ = true;
  }
  return exact_edges_;
}

void Engine::copy_edges(long long cap, int* centre, int* neighbour, double* d, long long* count) {
  const long long total = nedges();
  *count = total;
  const int nc = ncentres_;
  std::vector<int> row(static_cast<size_t>(nc) + 1), row_end(static_cast<size_t>(nc));
  std::vector<int> nbr(static_cast<size_t>(std::max<long long>(1, nedges_)));
  const size_t rec = precision_ == kFP32 ? sizeof(EdgeF) : sizeof(EdgeD);
  std::vector<unsigned char> d4(rec * static_cast<size_t>(std::max<long long>(1, nedges_)));
  if (nc) {
    SUS2G_CUDA(cudaMemcpyAsync(row.data(), row_.ptr, sizeof(int) * nc, cudaMemcpyDeviceToHost, stream_));
    SUS2G_CUDA(cudaMemcpyAsync(row_end.data(), d_row_end(), sizeof(int) * nc, cudaMemcpyDeviceToHost, stream_));
  }
  if (nedges_) {
    SUS2G_CUDA(cudaMemcpyAsync(nbr.data(), nbr_.ptr, sizeof(int) * nedges_, cudaMemcpyDeviceToHost, stream_));
    SUS2G_CUDA(cudaMemcpyAsync(d4.data(), d4_.ptr, rec * nedges_, cudaMemcpyDeviceToHost, stream_));
  }
  SUS2G_CUDA(cudaStreamSynchronize(stream_));
  long long k = 0;
  for (int i = 0; i < nc; ++i)
    for (int e = row[i]; e < row_end[i]; ++e, ++k) {
      if (k >= cap) continue;
      if (centre) centre[k] = i;
      if (neighbour) neighbour[k] = nbr[e];
      if (d) {
        if (precision_ == kFP32) {
          const EdgeF& x = reinterpret_cast<const EdgeF*>(d4.data())[e];
          d[3 * k] = x.x; d[3 * k + 1] = x.y; d[3 * k + 2] = x.z;
        } else {
          const EdgeD& x = reinterpret_cast<const EdgeD*>(d4.data())[e];
          d[3 * k] = x.x; d[3 * k + 1] = x.y; d[3 * k + 2] = x.z;
        }
      }
    }
  if (k != total) throw Error(20, "edge rows disagree with the edge count");
}

void* Engine::pinned(size_t bytes) {
  if (bytes > pinned_bytes_) {
    if (pinned_) cudaFreeHost(pinned_);
    pinned_ = nullptr;
    pinned_bytes_ = 0;
    SUS2G_CUDA(cudaMallocHost(&pinned_, bytes));
    pinned_bytes_ = bytes;
  }
  return pinned_;
}

void Engine::check_device_error() {
  enqueue_error_read();
  SUS2G_CUDA(cudaStreamSynchronize(stream_));
  check_error_read();
}

void Engine::enqueue_error_read() {
  wait_reverse();
  SUS2G_CUDA(cudaMemcpyAsync(host_total_ + 4, error_.ptr, 3 * sizeof(int), cudaMemcpyDeviceToHost, stream_));
}

void Engine::check_error_read() {
  const int h = host_total_[4], over = host_total_[5], bin_over = host_total_[6];
  if (over > 0 || bin_over > 0) {
    SUS2G_CUDA(cudaMemsetAsync(error_.ptr, 0, 3 * sizeof(int), stream_));
    if (over > 0) {
      cap_scale_ *= 2.0;
      min_cap_ = std::max(min_cap_, over);
    }
    if (bin_over > 0) {
      bin_cap_scale_ *= 2.0;
      min_bin_cap_ = std::max(min_bin_cap_, bin_over);
    }
    reset_step_graph();
    throw EdgeOverflow();
  }
  if (h) {
    SUS2G_CUDA(cudaMemsetAsync(error_.ptr, 0, sizeof(int), stream_));
    // a warp that left a pass early (a bounded wait that gave up) did not count itself done
    SUS2G_CUDA(cudaMemsetAsync(work_.ptr, 0, sizeof(int) * kWorkInts, stream_));
    static const char* msg[] = {"", "neighbour list capacity or centre index out of range",
                                "periodic image index outside [-64, 63]", "a directed edge has no reverse partner",
                                "zero or non-finite edge length", "non-finite atom coordinate",
                                "atom species index out of range",
                                "a bulk asynchronous copy into shared memory did not complete"};
    throw Error(20 + h, std::string("device check failed: ") + (h > 0 && h < 8 ? msg[h] : "unknown"));
  }
}

cudaEvent_t Engine::take_event() {
  if (event_next_ == event_pool_.size()) {
    cudaEvent_t e;
    SUS2G_CUDA(cudaEventCreate(&e));
    event_pool_.push_back(e);
  }
  return event_pool_[event_next_++];
}

void Engine::mark_begin(int stage) {
  if (!timing_) return;
  open_stage_ = stage;
  open_event_ = take_event();
  SUS2G_CUDA(cudaEventRecord(open_event_, stream_));
}

void Engine::mark_end() {
  if (!timing_ || open_stage_ < 0) return;
  cudaEvent_t e = take_event();
  SUS2G_CUDA(cudaEventRecord(e, stream_));
  marks_.push_back({open_stage_, {open_event_, e}});
  open_stage_ = -1;
}

void Engine::set_timing(bool on) {
  timing_ = on;
  marks_.clear();
  event_next_ = 0;
  for (int i = 0; i < 8; ++i) { stage_ms_[i] = 0; stage_count_[i] = 0; }
}

void Engine::take_stage_times(double* ms, int* counts) {
  SUS2G_CUDA(cudaStreamSynchronize(stream_));
  for (const auto& m : marks_) {
    float t = 0;
    SUS2G_CUDA(cudaEventElapsedTime(&t, m.second.first, m.second.second));
    stage_ms_[m.first] += t;
    stage_count_[m.first] += 1;
  }
  marks_.clear();
  event_next_ = 0;
  for (int i = 0; i < 8; ++i) {
    if (ms) ms[i] = stage_ms_[i];
    if (counts) counts[i] = stage_count_[i];
    stage_ms_[i] = 0;
    stage_count_[i] = 0;
  }
}

void Engine::build_edges(int nframes, const int* frame_natoms, const double* cells, const double* d_pos,
                         const int* d_types) {
  SUS2G_CUDA(cudaSetDevice(device_));
  ++edge_generation_;
  if (nframes < 0) throw Error(1, "negative frame count");
  const double rc = model_.max_dist, rc2 = rc * rc;
  std::vector<FramePlan>& plans = *plans_;
  plans.assign(nframes, FramePlan{});
  int a = 0, bins = 0, bin_cap = min_bin_cap_;
  long long pad_total = 0;
  bins_frames_ = 0;
  for (int f = 0; f < nframes; ++f) {
    FramePlan& fp = plans[f];
    if (frame_natoms[f] < 0) throw Error(1, "negative atom count");
    std::memcpy(fp.cell, cells + 9 * f, sizeof(fp.cell));
    invert3(fp.cell, fp.inv);
    double width[3];
    for (int q = 0; q < 3; ++q) {
      // |column q of inv| = 1 / perpendicular width of the cell along reciprocal direction q
      const double n = std::sqrt(fp.inv[q] * fp.inv[q] + fp.inv[3 + q] * fp.inv[3 + q] + fp.inv[6 + q] * fp.inv[6 + q]);
      fp.reach[q] = rc * n;
      width[q] = 1.0 / n;
    }
    fp.a0 = a;
    fp.a1 = a + frame_natoms[f];
    a = fp.a1;
    fp.use_bins = frame_natoms[f] > 512 && width[0] >= 3 * rc && width[1] >= 3 * rc && width[2] >= 3 * rc;
    fp.bin0 = bins;
    if (fp.use_bins) {
      ++bins_frames_;
      // bins at least r_c / 2 wide (the 5 x 5 x 5 stencil of the fill kernel); widths >= 3 r_c
      // give at least 6 bins per axis, so the periodic stencil never holds a bin twice
      for (int q = 0; q < 3; ++q) fp.nb[q] = std::max(6, std::min(512, static_cast<int>(width[q] / (0.5 * rc))));
      // FP32 prefilter: |error of r^2| <= 2 r_c |error of d| near the cutoff; d is the rounded wrapped
      // position (below the row norms' sum S per component) plus the rounded shift (below 2 S):
      // |error of d| <= 3^1/2 2^-24 (3 S + r_c) < 3.3e-7 S (the widths give S >= 9 r_c); the band is
      // more than twice what that and r^2's own rounding need
      double rows = 0;
      for (int q = 0; q < 3; ++q)
        rows += std::sqrt(fp.cell[3 * q] * fp.cell[3 * q] + fp.cell[3 * q + 1] * fp.cell[3 * q + 1] + fp.cell[3 * q + 2] * fp.cell[3 * q + 2]);
      fp.band = 2.0 * rc * (4.0 * 6.0e-8 * rows) * 4.0 + 1e-6;
      fp.screen2 = static_cast<float>(rc2 + fp.band);
      bins += fp.nb[0] * fp.nb[1] * fp.nb[2];
      // bin capacity: twice the frame's mean atoms per bin plus 8 (grown after an overflow)
      const double per_bin = frame_natoms[f] / static_cast<double>(fp.nb[0] * fp.nb[1] * fp.nb[2]);
      bin_cap = std::max(bin_cap, static_cast<int>(std::min(1.0e6, std::ceil(bin_cap_scale_ * per_bin) + 8.0)));
    }
    // FP32 cell rows (hi, lo) and the band of r^2 around r_c^2 that FP32 engines decide in FP64
    // (the cell-list fill's double-float r^2 is within ~1e-6 relative of the exact one, the
    // image scan's FP32 r^2 within ~5e-5)
    for (int q = 0; q < 9; ++q) {
      fp.cellf[q] = static_cast<float>(fp.cell[q]);
      fp.celll[q] = static_cast<float>(fp.cell[q] - static_cast<double>(fp.cellf[q]));
    }
    fp.lo2 = static_cast<float>(rc2 * (1.0 - 1e-4));
    fp.hi2 = static_cast<float>(rc2 * (1.0 + 1e-4));
    for (int q = 0; q < 9; ++q) fp.invf[q] = static_cast<float>(fp.inv[q]);
    for (int q = 0; q < 3; ++q) fp.reachf[q] = static_cast<float>(fp.reach[q]);
    fp.rc2f = static_cast<float>(rc2);
    // padded edge slots of every frame: cap_scale x the mean neighbour count of the frame's density
    // + 64 per centre (grown after an overflow)
    const double vol = std::abs(fp.cell[0] * (fp.cell[4] * fp.cell[8] - fp.cell[5] * fp.cell[7]) -
                                fp.cell[1] * (fp.cell[3] * fp.cell[8] - fp.cell[5] * fp.cell[6]) +
                                fp.cell[2] * (fp.cell[3] * fp.cell[7] - fp.cell[4] * fp.cell[6]));
    const double mean = vol > 0 ? frame_natoms[f] / vol * (4.0 / 3.0) * 3.141592653589793 * rc * rc2 : 0.0;
    fp.cap = std::max(min_cap_, static_cast<int>(std::min(1.0e6, std::ceil(cap_scale_ * mean) + 64.0)));
    fp.pad0 = pad_total;
    pad_total += static_cast<long long>(frame_natoms[f]) * fp.cap;
  }
  natoms_ = ncentres_ = a;
  nframes_ = nframes;
  d_types_ = d_types;
  user_edges_ = false;
  cudaStream_t s = stream_;
  mark_begin(0);
  plan_.ensure(sizeof(FramePlan) * std::max(1, nframes));
  // (a captured step leaves the plans out: they are on the device already, identical by the step key)
  if (nframes && !capturing_)
    SUS2G_CUDA(cudaMemcpyAsync(plan_.ptr, plans.data(), sizeof(FramePlan) * nframes, cudaMemcpyHostToDevice, s));
  frame_of_.ensure(sizeof(int) * std::max(1, a));
  counts_.ensure(sizeof(int) * (a + 1));
  row_.ensure(sizeof(int) * (a + 1));
  {
    // bin counters: zero at the start of a binning pass; the reverse-edge kernel of the previous
    // step cleared the ones it used, so only new or reallocated entries need a memset
    const void* before = bin_count_.ptr;
    bin_count_.ensure(sizeof(int) * (bins + 1));
    if (bin_count_.ptr != before) bin_zeroed_ = 0;
  }
  // batches with cell lists only: the binning kernel finds each atom's frame itself
  const bool find_frame = bins && bins_frames_ == nframes;
  if (nframes && !find_frame) {
    const bool split = bins_frames_ < nframes;
    if (split) posf_.ensure(2 * sizeof(float4) * std::max(1, a));
    k_frame_of<<<nframes, 256, 0, s>>>(plan_.as<FramePlan>(), nframes, frame_of_.as<int>(), d_pos,
                                       split ? posf_.as<float4>() : nullptr, split ? posf_.as<float4>() + a : nullptr);
    ++launches_;
  }
  if (bins) {
    if (bin_zeroed_ < bins + 1) SUS2G_CUDA(cudaMemsetAsync(bin_count_.ptr, 0, sizeof(int) * (bins + 1), s));
    bin_zeroed_ = 0;          // counted into from here on
    bins_used_ = bins + 1;    // cleared again by this step's reverse-edge kernel
    off_.ensure(sizeof(AtomOff) * a);
    rec_of_.ensure(sizeof(int) * a);
    const size_t slots = static_cast<size_t>(bins) * bin_cap;
    bin_off_.ensure(sizeof(AtomOff) * slots);
    bin_pos_.ensure(sizeof(BinPos) * slots);
    bin_posf_.ensure(sizeof(BinPosF) * slots);
    // one warp per block: each atom costs ~40 FP64 operations (1/64 of the FP32 rate on this
    // GPU), so small frames are spread over as many SMs as possible (4,096 atoms: 128 SMs)
    k_bin_place<<<(a + kWarp - 1) / kWarp, kWarp, 0, s>>>(plan_.as<FramePlan>(), nframes, find_frame, frame_of_.as<int>(), d_pos, a,
                                               bin_cap, rec_of_.as<int>(), bin_count_.as<int>(),
                                               off_.as<AtomOff>(), bin_off_.as<AtomOff>(), bin_pos_.as<BinPos>(),
                                               bin_posf_.as<BinPosF>(), error_.as<int>() + 2, error_.as<int>(), d_types,
                                               model_.C);
    ++launches_;
  }
  const unsigned warp_blocks = static_cast<unsigned>((static_cast<long long>(a) * kWarp + 255) / 256);
  const size_t rsz = precision_ == kFP32 ? sizeof(EdgeF) : sizeof(EdgeD);
  const FramePlan* P = plan_.as<FramePlan>();
  const int* FO = frame_of_.as<int>();
  const AtomOff* BO = bin_off_.as<AtomOff>();
  const BinPos* BP = bin_pos_.as<BinPos>();
  const BinPosF* BPF = bin_posf_.as<BinPosF>();
  const AtomOff* OF = off_.as<AtomOff>();
  int* overflow = error_.as<int>() + 1;
  // every periodic batch: the fill kernels (cell lists and image scan) write each centre's edges
  // to its padded slots and sort them there into the final arrays; no compaction, no host
  // synchronisation.  The edge arrays are sized by the padded capacity, the exact total is the sum
  // of the counts, and an overflow is reported by the step's check_device_error.
  const size_t slots = static_cast<size_t>(std::max<long long>(1, pad_total));
  if (pad_total > 2147483647LL) throw Error(4, "edge build: more than 2^31 - 1 edge slots");
  pad_nbr_.ensure(sizeof(int) * slots);
  pad_d4_.ensure(rsz * slots);
  pad_key_.ensure(sizeof(unsigned long long) * slots);
  nbr_.ensure(sizeof(int) * slots);
  rev_.ensure(sizeof(int) * slots);
  d4_.ensure(rsz * slots);
  key_.ensure(sizeof(unsigned long long) * slots);
  row_end_.ensure(sizeof(int) * std::max(1, a));
  if (a) {
    int* RW = row_.as<int>();
    int* RE = row_end_.as<int>();
    unsigned long long* KO = key_.as<unsigned long long>();
    int* NO = nbr_.as<int>();
    if (bins) {
      if (precision_ == kFP32)
        SUS2G_CUDA(launch_kernel((pdl_ & kPdlFill) != 0, k_edge_fill_bins<float>, dim3(warp_blocks), dim3(kFillWarps * kWarp), 0, s,
            P, FO, d_pos, a, rc2, bin_count_.as<int>(), bin_cap, BO, BP, BPF, rec_of_.as<int>(), OF,
            counts_.as<int>(), pad_nbr_.as<int>(), pad_d4_.as<EdgeF>(), pad_key_.as<unsigned long long>(), overflow,
            error_.as<int>(), RW, RE, KO, NO, d4_.as<EdgeF>()));
      else
        SUS2G_CUDA(launch_kernel((pdl_ & kPdlFill) != 0, k_edge_fill_bins<double>, dim3(warp_blocks), dim3(kFillWarps * kWarp), 0, s,
            P, FO, d_pos, a, rc2, bin_count_.as<int>(), bin_cap, BO, BP, BPF, rec_of_.as<int>(), OF,
            counts_.as<int>(), pad_nbr_.as<int>(), pad_d4_.as<EdgeD>(), pad_key_.as<unsigned long long>(), overflow,
            error_.as<int>(), RW, RE, KO, NO, d4_.as<EdgeD>()));
      ++launches_;
    }
    if (bins_frames_ < nframes) {
      if (precision_ == kFP32)
        SUS2G_CUDA(launch_kernel((pdl_ & kPdlFill) != 0, k_edge_image_fill<float>, dim3(warp_blocks), dim3(kFillWarps * kWarp), 0, s,
            P, FO, d_pos, posf_.as<float4>(), posf_.as<float4>() + a, d_types, model_.C, a, rc2, counts_.as<int>(),
            pad_nbr_.as<int>(), pad_d4_.as<EdgeF>(),
            pad_key_.as<unsigned long long>(), overflow, error_.as<int>(), RW, RE, KO, NO, d4_.as<EdgeF>()));
      else
        SUS2G_CUDA(launch_kernel((pdl_ & kPdlFill) != 0, k_edge_image_fill<double>, dim3(warp_blocks), dim3(kFillWarps * kWarp), 0, s,
            P, FO, d_pos, posf_.as<float4>(), posf_.as<float4>() + a, d_types, model_.C, a, rc2, counts_.as<int>(), pad_nbr_.as<int>(),
            pad_d4_.as<EdgeD>(),
            pad_key_.as<unsigned long long>(), overflow, error_.as<int>(), RW, RE, KO, NO, d4_.as<EdgeD>()));
      ++launches_;
    }
  }
  nedges_ = pad_total;
  nedges_exact_ = false;
  padded_ = true;
  clear_bins_ = bins > 0;
  finalize_edges();
  mark_end();
}

void Engine::finalize_edges() {
  cudaStream_t s = stream_;
  const int a = ncentres_;
  // (periodic batches were sorted by their fill kernels)
  if (a && !padded_) {
    const int blocks = (a + kSortWarps - 1) / kSortWarps;
    // centres with at most 128 edges rank from shared memory
    constexpr int stage = 128;
    const size_t smem = sizeof(unsigned long long) * kSortWarps * stage;
    if (precision_ == kFP32)
      k_edge_sort<float><<<blocks, kSortWarps * kWarp, smem, s>>>(
          row_.as<int>(), a, stage, tmp_key_.as<unsigned long long>(), tmp_nbr_.as<int>(), tmp_d4_.as<EdgeF>(),
          key_.as<unsigned long long>(), nbr_.as<int>(), d4_.as<EdgeF>());
    else
      k_edge_sort<double><<<blocks, kSortWarps * kWarp, smem, s>>>(
          row_.as<int>(), a, stage, tmp_key_.as<unsigned long long>(), tmp_nbr_.as<int>(), tmp_d4_.as<EdgeD>(),
          key_.as<unsigned long long>(), nbr_.as<int>(), d4_.as<EdgeD>());
    ++launches_;
  }
  if (user_edges_) {
    const int nall = natoms_;
    if (nedges_) {
      const unsigned eb = static_cast<unsigned>((nedges_ + 255) / 256);
      if (model_.gated) {  // the outer pass stores its gate-signal adjoints at the edges themselves
        k_iota<<<eb, 256, 0, s>>>(rev_.as<int>(), nedges_);
        ++launches_;
      }
      k_fill_in<<<eb, 256, 0, s>>>(nbr_.as<int>(), row_.as<int>() + nall, in_row_.as<int>(), counts_.as<int>() + nall + 1,
                                   tmp_nbr_.as<int>());
      k_sort_in<<<static_cast<unsigned>((static_cast<long long>(nall) * kWarp + 255) / 256), 256, 0, s>>>(
          in_row_.as<int>(), nall, tmp_nbr_.as<int>(), in_edge_.as<int>());
      launches_ += 2;
    }
  } else if (nedges_ && a) {
    // reverse edges on the second stream: the Static pass and the Effect gate-forward pass do not
    // read them, so they overlap; wait_reverse() joins before the first reader
    // (FP32 engines only: the FP64 pass is long enough that the overlap gains nothing, and its
    // persistent grid loses SMs to the reverse kernel while that runs)
    cudaStream_t rs = s;
    if (may_fork() && precision_ == kFP32) {
      SUS2G_CUDA(cudaEventRecord(ev_fork_, s));
      SUS2G_CUDA(cudaStreamWaitEvent(aux_stream_, ev_fork_, 0));
      rs = aux_stream_;
    }
    SUS2G_CUDA(launch_kernel_priority(rs != s ? urgent_priority_ : 0, k_reverse,
        dim3(static_cast<unsigned>((static_cast<long long>(a) * kWarp + 255) / 256)), dim3(256), 0, rs,
        row_.as<int>(), d_row_end(), key_.as<unsigned long long>(), a, rev_.as<int>(), error_.as<int>(),
        bin_count_.as<int>(), clear_bins_ ? bins_used_ : 0));
    ++launches_;
    if (clear_bins_) bin_zeroed_ = bins_used_;
    if (rs != s) {
      SUS2G_CUDA(cudaEventRecord(ev_rev_, rs));
      rev_pending_ = true;
    }
  }
}

bool Engine::edges_plain(int nowned, int nall, int nedges, const int* d_i, const int* d_j, const double* d_d) {
  if (nedges <= 0) return true;
  SUS2G_CUDA(cudaSetDevice(device_));
  edge_flag_.ensure(sizeof(int));
  SUS2G_CUDA(cudaMemsetAsync(edge_flag_.ptr, 0, sizeof(int), stream_));
  k_check_user_edges<<<static_cast<unsigned>((static_cast<long long>(nedges) + 255) / 256), 256, 0, stream_>>>(
      d_i, d_j, d_d, nedges, nowned, nall, edge_flag_.as<int>());
  SUS2G_CUDA(cudaGetLastError());
  SUS2G_CUDA(cudaMemcpyAsync(host_total_ + 7, edge_flag_.ptr, sizeof(int), cudaMemcpyDeviceToHost, stream_));
  SUS2G_CUDA(cudaStreamSynchronize(stream_));
  return host_total_[7] == 0;
}
void Engine::set_edges(int nowned, int nall, const int* d_types, int nedges, const int* d_i, const int* d_j, const double* d_d) {
  SUS2G_CUDA(cudaSetDevice(device_));
  ++edge_generation_;
  clear_bins_ = false;
  padded_ = false;
  if (nowned < 0 || nall < nowned || nedges < 0) throw Error(1, "invalid atom layout");
  cudaStream_t s = stream_;
  ncentres_ = nowned;
  natoms_ = nall;
  nframes_ = 1;
  d_types_ = d_types;
  user_edges_ = true;
  std::vector<FramePlan>& plans = *plans_;
  plans.assign(1, FramePlan{});
  plans[0].a0 = 0;
  plans[0].a1 = nowned;
  plan_.ensure(sizeof(FramePlan));
  SUS2G_CUDA(cudaMemcpyAsync(plan_.ptr, plans.data(), sizeof(FramePlan), cudaMemcpyHostToDevice, s));
  // counts of out- and in-edges, both rows by one scan launch (ghosts have no out-edges), then the
  // scatter; the row ends -- the edges that are in range -- stay on the device
  const size_t E = std::max(1, nedges);
  const size_t rsz = precision_ == kFP32 ? sizeof(EdgeF) : sizeof(EdgeD);
  counts_.ensure(sizeof(int) * 2 * (nall + 1));
  row_.ensure(sizeof(int) * (nall + 1));
  in_row_.ensure(sizeof(int) * (nall + 1));
  in_edge_.ensure(sizeof(int) * E);
  nbr_.ensure(sizeof(int) * E); tmp_nbr_.ensure(sizeof(int) * E);
  if (model_.gated) rev_.ensure(sizeof(int) * E);
  d4_.ensure(rsz * E); tmp_d4_.ensure(rsz * E);
  key_.ensure(sizeof(unsigned long long) * E); tmp_key_.ensure(sizeof(unsigned long long) * E);
  int* out_count = counts_.as<int>();
  int* in_count = out_count + nall + 1;
  SUS2G_CUDA(cudaMemsetAsync(counts_.ptr, 0, sizeof(int) * 2 * (nall + 1), s));
  const unsigned eb = static_cast<unsigned>((static_cast<long long>(nedges) + 255) / 256);
  if (nedges) {
    k_count_user_edges<<<eb, 256, 0, s>>>(d_i, d_j, nedges, out_count, in_count, nowned, nall, error_.as<int>());
    ++launches_;
  }
  k_exclusive_scans<<<2, 1024, 0, s>>>(out_count, in_count, nall, row_.as<int>(), in_row_.as<int>(), error_.as<int>());
  ++launches_;
  if (nedges) {
    if (precision_ == kFP32)
      k_scatter_user_edges<float><<<eb, 256, 0, s>>>(d_i, d_j, d_d, nedges, row_.as<int>(), out_count,
          tmp_nbr_.as<int>(), tmp_d4_.as<EdgeF>(), tmp_key_.as<unsigned long long>(), nowned, nall, error_.as<int>());
    else
      k_scatter_user_edges<double><<<eb, 256, 0, s>>>(d_i, d_j, d_d, nedges, row_.as<int>(), out_count,
          tmp_nbr_.as<int>(), tmp_d4_.as<EdgeD>(), tmp_key_.as<unsigned long long>(), nowned, nall, error_.as<int>());
    ++launches_;
  }
  nedges_ = nedges;
  nedges_exact_ = false;
  finalize_edges();
}

template <typename Real>
PassArgs<Real> Engine::pass_args() {
  const Model& m = model_;
  const int N = natoms_;
  const size_t E = std::max<long long>(1, nedges_);
  g_.ensure(sizeof(Real) * 3 * E);
  site_.ensure(sizeof(double) * std::max(1, N));
  vir_atom_.ensure(sizeof(double) * 6 * std::max(1, N));
  PassArgs<Real> a{};
  a.dm = *static_cast<DevModel<Real>*>(dev_model_);
  a.moment_mma = moment_mma_ ? 1 : 0;
  a.natoms = ncentres_;
  a.types = d_types_;
  a.row = row_.as<int>();
  a.row_end = d_row_end();
  a.nbr = nbr_.as<int>();
  a.rev = rev_.as<int>();
  a.d4 = static_cast<const typename Vec4<Real>::type*>(d4_.ptr);
  a.g = g_.as<Real>();
  a.site_energy = site_.as<double>();
  a.virial = vir_atom_.as<double>();
  a.desc = desc_out_;
  a.error = error_.as<int>();
  if (m.gated) {
    hsig_.ensure(sizeof(Real) * static_cast<size_t>(std::max(1, N)) * m.F);
    hcontrib_.ensure(sizeof(Real) * E * m.F);
    // (a split gate pass keeps its own values, launch_gate_split)
    if (!use_gate_split<Real>()) gmom_.ensure(sizeof(Real) * static_cast<size_t>(std::max(1, N)) * m.M);
    a.hsig = hsig_.as<Real>();
    a.hcontrib = hcontrib_.as<Real>();
    a.gmom = gmom_.as<Real>();
  }
  return a;
}

template <typename Real>
void Engine::run_efs(double* d_energy, double* d_forces, double* d_virial, double* d_site, int stages) {
  const Model& m = model_;
  cudaStream_t s = stream_;
  const int N = natoms_;
  PassArgs<Real> a = pass_args<Real>();
  // stage 1: gate forward (Effect) -- gate signals of the centre atoms
  if (stages & kStageGate) {
    // every centre's site energy, virial and gate signal is written by the passes; only caller
    // layouts with ghosts have rows that must start at zero
    const bool ghosts = user_edges_ && N > ncentres_;
    if (ghosts) {
      SUS2G_CUDA(cudaMemsetAsync(site_.ptr, 0, sizeof(double) * std::max(1, N), s));
      SUS2G_CUDA(cudaMemsetAsync(vir_atom_.ptr, 0, sizeof(double) * 6 * std::max(1, N), s));
    }
    if (m.gated) {
      // ghost rows (caller edges) are filled by the caller's forward exchange
      if (ghosts)
        SUS2G_CUDA(cudaMemsetAsync(hsig_.ptr, 0, sizeof(Real) * static_cast<size_t>(std::max(1, N)) * m.F, s));
      mark_begin(2);
      gate_ran_split_ = use_gate_split<Real>();
      if (gate_ran_split_) launches_ += launch_gate_split<Real>(0, a, (pdl_ & kPdlFirstPass) != 0);
      else launches_ += launch_pass<Real>(kModeGateForward, a, (pdl_ & kPdlFirstPass) != 0);
      mark_end();
    }
  }
  // stage 2: Static pass, or Effect outer pass and the gate-signal adjoint per atom
  if (stages & kStageOuter) {
    if (m.gated) wait_reverse();  // the outer pass writes the gate-signal adjoints at reverse edges
    mark_begin(1);
    const int mode = m.gated ? kModeOuter : kModeStatic;
    if (use_static_split<Real>())
      launches_ += launch_static_split<Real>(a, (pdl_ & (m.gated ? kPdlBetweenPasses : kPdlFirstPass)) != 0);
    else launches_ += launch_pass<Real>(mode, a, (pdl_ & (m.gated ? kPdlBetweenPasses : kPdlFirstPass)) != 0);
    mark_end();
    if (m.gated && user_edges_) {
      hbar_atom_.ensure(sizeof(double) * static_cast<size_t>(std::max(1, N)) * m.F);
      const long long n = static_cast<long long>(N) * m.F;
      if (n) {
        k_hbar_gather<Real><<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(
            in_row_.as<int>(), in_edge_.as<int>(), hcontrib_.as<Real>(), N, m.F, hbar_atom_.as<double>());
        ++launches_;
      }
    }
  }
  // stage 3: Effect gate reverse, forces, per-frame energy and virial
  if (stages & kStageFinish) {
    if (m.gated) {
      if (user_edges_) a.hbar_atom = hbar_atom_.as<double>();
      mark_begin(3);
      if (gate_ran_split_) launches_ += launch_gate_split<Real>(1, a, (pdl_ & kPdlBetweenPasses) != 0);
      else launches_ += launch_pass<Real>(kModeGateReverse, a, (pdl_ & kPdlBetweenPasses) != 0);
      mark_end();
    }
    wait_reverse();
    mark_begin(4);
    // frame-reduction buffers first: the arrival counters must be zero before the reduction
    // starts on either stream
    int S = 1;
    if (nframes_) {
      int largest = 0;
      for (const FramePlan& fp : *plans_) largest = std::max(largest, fp.a1 - fp.a0);
      S = std::max(1, std::min(64, (largest + kFrameThreads - 1) / kFrameThreads));
      frame_partial_.ensure(sizeof(double) * 7 * static_cast<size_t>(nframes_) * S);
      if (nframes_ > arrivals_frames_) {
        // arrival counters start at zero; each launch leaves them at zero
        frame_arrivals_.ensure(sizeof(unsigned) * nframes_);
        SUS2G_CUDA(cudaMemsetAsync(frame_arrivals_.ptr, 0, sizeof(unsigned) * nframes_, s));
        arrivals_frames_ = nframes_;
      }
    }
    // the per-frame reduction (site energies and virials) runs on the second stream beside the
    // force gather
    cudaStream_t fs = s;
    if (may_fork() && nframes_ && d_forces && N) {
      SUS2G_CUDA(cudaEventRecord(ev_fork2_, s));
      SUS2G_CUDA(cudaStreamWaitEvent(aux_stream_, ev_fork2_, 0));
      fs = aux_stream_;
    }
    if (d_forces && N) {
      if (user_edges_)
        k_force_gather_user<Real><<<static_cast<unsigned>((static_cast<long long>(N) * kWarp + 255) / 256), 256, 0, s>>>(
            row_.as<int>(), ncentres_, in_row_.as<int>(), in_edge_.as<int>(), g_.as<Real>(), N, d_forces);
      else
        SUS2G_CUDA(launch_kernel((pdl_ & kPdlGather) != 0, k_force_gather<Real>, dim3((N * kWarp + 255) / 256), dim3(256), 0, s,
                                 row_.as<int>(), d_row_end(), rev_.as<int>(), g_.as<Real>(), ncentres_, d_forces));
      ++launches_;
    }
    if (nframes_) {
      k_frame_reduce<<<dim3(nframes_, S), kFrameThreads, 0, fs>>>(
          plan_.as<FramePlan>(), nframes_, S, site_.as<double>(), vir_atom_.as<double>(), d_site,
          frame_partial_.as<double>(), frame_arrivals_.as<unsigned>(), d_energy, d_virial);
      ++launches_;
    } else if (d_site && N) {
      SUS2G_CUDA(cudaMemcpyAsync(d_site, site_.ptr, sizeof(double) * ncentres_, cudaMemcpyDeviceToDevice, s));
    }
    if (fs != s) {
      SUS2G_CUDA(cudaEventRecord(ev_join2_, fs));
      SUS2G_CUDA(cudaStreamWaitEvent(s, ev_join2_, 0));
    }
    mark_end();
  }
}

namespace {
// grad[p] += sum over gradient slices, in two fixed-order levels: block (x, c) sums slices
// c, c + G, c + 2G, ... (G = gridDim.y) of parameters 32 x .. 32 x + 31 in 8 interleaved lanes
// per parameter, combined in shared memory in lane order, into part[c][p]; k_slot_finish adds
// the G partials in order.
constexpr int kSlotGroups = 32;
__global__ void k_slot_partial(const double* slots, int nslots, int nparams, double* part) {
  __shared__ double sh[8][33];
  const int p = blockIdx.x * 32 + threadIdx.x, g = threadIdx.y, c = blockIdx.y, G = gridDim.y;
  double s = 0.0;
  if (p < nparams)
    for (int w = c + G * g; w < nslots; w += 8 * G) s += slots[static_cast<size_t>(w) * nparams + p];
  sh[g][threadIdx.x] = s;
  __syncthreads();
  if (g == 0 && p < nparams) {
    double t = 0.0;
    for (int q = 0; q < 8; ++q) t += sh[q][threadIdx.x];
    part[static_cast<size_t>(c) * nparams + p] = t;
  }
}
__global__ void k_slot_finish(const double* part, int groups, int nparams, double* grad) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nparams) return;
  double s = 0.0;
  for (int c = 0; c < groups; ++c) s += part[static_cast<size_t>(c) * nparams + p];
  grad[p] += s;
}

// Gate projection weights: dJ/dW[mu][q] = sum_atoms lambda_h[mu] g[node q] + mu_h[mu] gdot[node q],
// a (2F x N) . (N x Q) product reduced over atoms.  Block b takes the atom chunks b, b + grid, ...,
// stages each chunk's lambda / mu rows and gate-node values in shared memory, and adds its partial
// sums into its own slot row (reduced later in fixed order with the other parameter slots), so the
// result is deterministic.  Outputs are taken kGwTile at a time (one per thread and repeat).
constexpr int kGwChunk = 32;
constexpr int kGwThreads = 256;
constexpr int kGwPer = 4;  // outputs per thread per tile
template <typename Real>
__global__ void __launch_bounds__(kGwThreads) k_gate_weight_grad(int natoms, int F, int Q, int M, const int* nodes,
                                                                 const double* lh, const Real* gmom,
                                                                 const Real* gmomd, double* slots, int nparams,
                                                                 int gw_off) {
  // staging and chunk sums in the compute precision (FP32 bulk: the products and each 32-atom
  // chunk's sum in FP32, the chunk partials added in FP64; FP64 plain: FP64 throughout)
  extern __shared__ double gw_sh[];
  Real* sl = reinterpret_cast<Real*>(gw_sh);   // [kGwChunk][2F]
  Real* sg = sl + kGwChunk * 2 * F;            // [kGwChunk][2Q]
  const int FQ = F * Q;
  double* out = slots + static_cast<size_t>(blockIdx.x) * nparams + gw_off;
  for (int tile = 0; tile < FQ; tile += kGwThreads * kGwPer) {
    double acc[kGwPer];
#pragma unroll
    for (int k = 0; k < kGwPer; ++k) acc[k] = 0.0;
    for (int base = blockIdx.x * kGwChunk; base < natoms; base += gridDim.x * kGwChunk) {
      const int n = min(kGwChunk, natoms - base);
      __syncthreads();
      for (int t = threadIdx.x; t < n * 2 * F; t += blockDim.x) sl[t] = Real(lh[static_cast<size_t>(base) * 2 * F + t]);
      for (int t = threadIdx.x; t < n * Q; t += blockDim.x) {
        const int a = t / Q, q = t - a * Q;
        const size_t o = static_cast<size_t>(base + a) * M + nodes[q];
        sg[a * 2 * Q + q] = gmom[o];
        sg[a * 2 * Q + Q + q] = gmomd[o];
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kGwPer; ++k) {
        const int t = tile + k * kGwThreads + threadIdx.x;
        if (t < FQ) {
          const int m = t / Q, q = t - m * Q;
          Real v = Real(0);
          for (int a = 0; a < n; ++a)
            v += sl[a * 2 * F + m] * sg[a * 2 * Q + q] + sl[a * 2 * F + F + m] * sg[a * 2 * Q + Q + q];
          acc[k] += double(v);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kGwPer; ++k) {
      const int t = tile + k * kGwThreads + threadIdx.x;
      if (t < FQ) out[t] += acc[k];
    }
  }
}
}  // namespace

template <typename Real>
void Engine::run_grad(const double* ew, const double* fw, const double* sw, double* grad,
                      const double* extra_h) {
  const Model& m = model_;
  if (user_edges_) throw Error(1, "the parameter gradient runs on periodic frames (build_edges)");
  if (m.body_combo) throw Error(1, "the parameter gradient of mu-body-linear-combo gates is not implemented");
  cudaStream_t s = stream_;
  const int N = natoms_, P = m.param_count();
  const size_t E = std::max<long long>(1, nedges_);
  if constexpr (sizeof(Real) == 4)
    if (m.B == 8 && !have_dual_) upload_block_programs(true);
  const DevModel<Real>& dm = *static_cast<DevModel<Real>*>(dev_model_);
  GradArgs<Real> a{};
  a.dm = dm;
  a.natoms = ncentres_;
  a.types = d_types_;
  a.row = row_.as<int>();
  a.row_end = d_row_end();
  a.nbr = nbr_.as<int>();
  a.rev = rev_.as<int>();
  a.d4 = static_cast<const typename Vec4<Real>::type*>(d4_.ptr);
  a.frame_of = frame_of_.as<int>();
  a.ew = ew;
  a.fw = fw;
  a.sw = sw;
  a.extra_h = extra_h;
  a.error = error_.as<int>();
  // the outer and gate reverse passes whole, or split into their per-atom and per-edge parts
  // (basis size 8) through the moment adjoints in gabar_.  Split, the per-edge part runs as
  // grad_edge_kernel where the model's warps are per channel and its sums fit in shared memory, and
  // FP32 engines run the per-atom part as the edge->moment kernel and the block graph kernel where
  // the nodes fit; the other forms of grad_pass_kernel cover what is left.
  const bool split = grad_split_ && m.B == 8;
  const int part1 = split ? kGradAtomPart : kGradWhole;
  bool dual = false;
  if constexpr (sizeof(Real) == 4) dual = split && grad_graph_fits(dm, m.gated);
  GradLaunch gm_o{}, gm_g{}, gg[3] = {}, ge_o{}, ge_g{}, gw{}, co{}, co2{}, cf{}, cr{}, cr2{};
  int nslots = 0;
  auto slices = [&](const GradLaunch& c, bool per_block) { nslots = std::max(nslots, per_block ? c.grid : c.grid * c.warps); };
  if (split) {
    ge_o = grad_edge_config<Real>(m.L, kGradOuter, dm, ncentres_, sm_count_);
    if (m.gated) ge_g = grad_edge_config<Real>(m.L, kGradGateReverse, dm, ncentres_, sm_count_);
    slices(ge_o, true);
    slices(ge_g, true);
  }
  if constexpr (sizeof(Real) == 4)
    if (dual) {
      gm_o = grad_moment_config(m.L, kGradOuter, dm, ncentres_, sm_count_);
      for (int q = 0; q < (m.gated ? 3 : 1); ++q) {
        gg[q] = grad_graph_config(q, dm, ncentres_, sm_count_);
        slices(gg[q], true);
      }
      if (m.gated) {
        gm_g = grad_moment_config(m.L, kGradGateForward, dm, ncentres_, sm_count_);
        gw = grad_gate_weight_config(dm, ncentres_, sm_count_);
        slices(gw, true);
      }
    }
  if (!dual) {
    co = grad_pass_config<Real>(m.L, kGradOuter, dm, ncentres_, sm_count_, part1);
    slices(co, false);
    if (m.gated) {
      cf = grad_pass_config<Real>(m.L, kGradGateForward, dm, ncentres_, sm_count_);
      cr = grad_pass_config<Real>(m.L, kGradGateReverse, dm, ncentres_, sm_count_, part1);
      slices(cf, false);
      slices(cr, false);
    }
  }
  if (split && !ge_o.grid) {
    co2 = grad_pass_config<Real>(m.L, kGradOuter, dm, ncentres_, sm_count_, kGradEdgePart);
    slices(co2, false);
  }
  if (split && m.gated && !ge_g.grid) {
    cr2 = grad_pass_config<Real>(m.L, kGradGateReverse, dm, ncentres_, sm_count_, kGradEdgePart);
    slices(cr2, false);
  }
  const size_t NC = static_cast<size_t>(std::max(1, ncentres_)), KH2 = 2 * static_cast<size_t>(m.K) * m.H;
  if (split) {
    gabar_.ensure(sizeof(Real) * NC * KH2);
    a.abar = gabar_.as<Real>();
  }
  slots_.ensure(sizeof(double) * static_cast<size_t>(nslots) * P);
  SUS2G_CUDA(cudaMemsetAsync(slots_.ptr, 0, sizeof(double) * static_cast<size_t>(nslots) * P, s));
  a.slots = slots_.as<double>();
  if (m.gated) {
    const size_t NF = static_cast<size_t>(std::max(1, N)) * m.F, NM = static_cast<size_t>(std::max(1, N)) * m.M;
    hsig_.ensure(sizeof(Real) * NF);
    hsigd_.ensure(sizeof(Real) * NF);
    lhm_.ensure(sizeof(Real) * E * 2 * m.F);
    lh_atom_.ensure(sizeof(double) * 2 * NF);
    a.hsig = hsig_.as<Real>();
    a.hsigd = hsigd_.as<Real>();
    a.lhm = lhm_.as<Real>();
    a.lh_atom = lh_atom_.as<double>();
    if (!dual) {
      gmom_.ensure(sizeof(Real) * NM);
      gmomd_.ensure(sizeof(Real) * NM);
      a.gmom = gmom_.as<Real>();
      a.gmomd = gmomd_.as<Real>();
    }
  }
  if constexpr (sizeof(Real) == 4)
    if (dual) {
      const size_t blocks = (NC + kDualAtoms - 1) / kDualAtoms;
      gdmom_.ensure(sizeof(Real) * NC * KH2);
      a.mom = gdmom_.as<Real>();
      if (m.gated) {
        gdkeep_.ensure(sizeof(Real) * blocks * kWarp * std::max(1, dm.gate.dual.nkeep));
        gdscal_.ensure(sizeof(Real) * blocks * kWarp * std::max(1, m.Q));
        a.gkeep = gdkeep_.as<Real>();
        a.gscal = gdscal_.as<Real>();
        launches_ += launch_grad_moment(m.L, kGradGateForward, a, gm_g, s);
        launches_ += launch_grad_graph(kGradGateForward, a, gg[kGradGateForward], s);
      }
      launches_ += launch_grad_moment(m.L, kGradOuter, a, gm_o, s);
      launches_ += launch_grad_graph(kGradOuter, a, gg[kGradOuter], s);
    }
  if (!dual) {
    if (m.gated) launches_ += launch_grad_pass<Real>(m.L, kGradGateForward, a, cf, s);
    launches_ += launch_grad_pass<Real>(m.L, kGradOuter, a, co, s);
  }
  if (ge_o.grid) launches_ += launch_grad_edge<Real>(m.L, kGradOuter, a, ge_o, s);
  else if (split) launches_ += launch_grad_pass<Real>(m.L, kGradOuter, a, co2, s);
  if (m.gated) {
    if constexpr (sizeof(Real) == 4)
      if (dual) {
        launches_ += launch_lhm_sum(a, m.L + 1, s);
        launches_ += launch_grad_graph(kGradGateReverse, a, gg[kGradGateReverse], s);
      }
    if (!dual) launches_ += launch_grad_pass<Real>(m.L, kGradGateReverse, a, cr, s);
    if (ge_g.grid) launches_ += launch_grad_edge<Real>(m.L, kGradGateReverse, a, ge_g, s);
    else if (split) launches_ += launch_grad_pass<Real>(m.L, kGradGateReverse, a, cr2, s);
    const int gw_off = dm.grad.gate_w_off;
    if (N && gw_off >= 0) {
      if constexpr (sizeof(Real) == 4)
        if (dual) launches_ += launch_grad_gate_weight(a, gw, s);
      if (!dual) {
        const int blocks = std::max(1, std::min(nslots, (ncentres_ + kGwChunk - 1) / kGwChunk));
        const size_t smem = sizeof(Real) * kGwChunk * 2 * (m.F + m.Q);
        if (smem > 200 * 1024) throw Error(3, "gate weight gradient: radial functions + gate scalars exceed the shared-memory staging");
        static LargestPerDevice allowed;
        SUS2G_CUDA(allow_shared_memory(k_gate_weight_grad<Real>, smem, allowed));
        k_gate_weight_grad<Real><<<blocks, kGwThreads, smem, s>>>(ncentres_, m.F, m.Q, m.M, dm.gate_nodes,
                                                                  lh_atom_.as<double>(), gmom_.as<Real>(),
                                                                  gmomd_.as<Real>(), slots_.as<double>(), P, gw_off);
        ++launches_;
      }
    }
  }
  slot_part_.ensure(sizeof(double) * kSlotGroups * static_cast<size_t>(P));
  k_slot_partial<<<dim3((P + 31) / 32, kSlotGroups), dim3(32, 8), 0, s>>>(slots_.as<double>(), nslots, P,
                                                                         slot_part_.as<double>());
  k_slot_finish<<<(P + 255) / 256, 256, 0, s>>>(slot_part_.as<double>(), kSlotGroups, P, grad);
  launches_ += 2;
}

void Engine::combination_grad(const double* d_ew, const double* d_fw, const double* d_sw, double* d_grad,
                              const double* d_extra_h) {
  SUS2G_CUDA(cudaSetDevice(device_));
  wait_reverse();
  if (precision_ == kFP32) run_grad<float>(d_ew, d_fw, d_sw, d_grad, d_extra_h);
  else run_grad<double>(d_ew, d_fw, d_sw, d_grad, d_extra_h);
}

const void* Engine::d_gate_additive() const {
  if (!model_.gated) return nullptr;
  if (precision_ == kFP32) return static_cast<const DevModel<float>*>(dev_model_)->outer.wadd;
  return static_cast<const DevModel<double>*>(dev_model_)->outer.wadd;
}

int Engine::gate_additive_offset() const {
  if (!model_.gated) return -1;
  if (precision_ == kFP32) return static_cast<const DevModel<float>*>(dev_model_)->grad.outer.add_off;
  return static_cast<const DevModel<double>*>(dev_model_)->grad.outer.add_off;
}

int Engine::static_pass_external(int natoms, const int* types, const int* row, const int* nbr, const void* d4, float* g,
                                 double* site, double* vir, int* error) {
  if (precision_ != kFP32 || model_.gated) throw Error(1, "external Static pass needs a Static model on an FP32 engine");
  PassArgs<float> a{};
  a.dm = *static_cast<DevModel<float>*>(dev_model_);
  a.natoms = natoms;
  a.types = types;
  a.row = row;
  a.row_end = row + 1;
  a.nbr = nbr;
  a.rev = nullptr;
  a.d4 = static_cast<const EdgeF*>(d4);
  a.g = g;
  a.site_energy = site;
  a.virial = vir;
  a.error = error;
  return launch_atom_pass<float>(model_.L, kModeStatic, a, sm_count_, stream_) ? 1 : 0;
}

void Engine::efs(double* d_energy, double* d_forces, double* d_virial, double* d_site) {
  SUS2G_CUDA(cudaSetDevice(device_));
  if (model_.gated && user_edges_ && ncentres_ != natoms_)
    throw Error(1, "Effect models on a ghost layout need the caller's gate-signal exchange: use the staged calls");
  if (precision_ == kFP32) run_efs<float>(d_energy, d_forces, d_virial, d_site, kStageAll);
  else run_efs<double>(d_energy, d_forces, d_virial, d_site, kStageAll);
}

// The energy pass (Static, or the Effect outer pass) split at the per-atom boundary (FP32
// engines, basis size 8): edge->moment forward, per-atom graph kernel, per-edge adjoint -- three
// launches through device moment arrays; the forward and adjoint kernels take the fused pass's
// tile shape.
template <typename Real>
bool Engine::use_static_split() const {
  return sizeof(Real) == 4 && model_.B == 8 && wants_split(static_split_) && split_fits(false);
}
bool Engine::split_fits(bool gate) const {
  if (precision_ != kFP32) return false;
  const auto* dm = static_cast<const DevModel<float>*>(dev_model_);
  return graph_block_fits(gate ? dm->gate.block : dm->outer.block, model_.F, model_.S);
}
template <typename Real>
int Engine::launch_static_split(PassArgs<Real> a, bool pdl) {
  if constexpr (sizeof(Real) == 4) {
    const size_t n = static_cast<size_t>(std::max(1, ncentres_)) * model_.K * model_.H;
    // a block of the graph kernel reads its centres' moments before it writes their adjoints
    mom_.ensure(sizeof(Real) * n);
    a.mom = a.amom = mom_.as<Real>();
    const int mode = model_.gated ? kModeOuter : kModeStatic;
    a.grid_mode = pass_grid_[mode];
    a.atom_order = pass_order_[mode];
    a.block_warps = pass_wpb_[mode];
    int k = launch_shape<Real>(model_.gated ? kModeOuterFwd : kModeStaticFwd, a, split_blocks_, pdl);
    k += launch_atom_graph(a, sm_count_, stream_, 0);
    k += launch_shape<Real>(model_.gated ? kModeOuterRev : kModeStaticRev, a, split_blocks_, false);
    return k;
  } else {
    throw Error(1, "the split passes run on FP32 engines");
  }
}

// The Effect gate passes split at the per-atom boundary (FP32 engines, basis size 8): which 0 =
// the gate forward pass (edge->moment kernel, then the per-atom gate graph and gate-signal
// projection), 1 = the gate reverse pass (per-atom sums of the gate-signal adjoints, their
// projection and the gate graph reverse, then the per-edge adjoint); the per-edge kernels take the
// fused pass's grid and centre order and their own register budget.
template <typename Real>
bool Engine::use_gate_split() const {
  return sizeof(Real) == 4 && model_.B == 8 && model_.gated && wants_split(gate_split_) && split_fits(true);
}
// Without a choice by the caller or the autotuner the passes run split from this many centres on.  A
// fused pass whose centres all have a resident warp (12 to 16 per SM) hides the per-atom work
// behind other warps' edges and saves two launches; past that every further round pays for it.
// Step times fused / split, us: Static L2 4,096 centres 101 / 106, 10,648 193 / 187; Static L3 4,096
// 120 / 119, 10,648 242 / 232, 110,592 1990 / 1806; Effect L3 2,016 148 / 159, 4,096 228 / 211,
// 110,592 4240 / 3427; Effect L4 1,000 234 / 263, 2,016 341 / 307, 110,592 10406 / 8490; Effect L5
// 1,000 229 / 257, 2,016 418 / 344, 32,768 3622 / 2780.
bool Engine::auto_split() const {
  return ncentres_ >= sm_count_ * (model_.L >= 4 ? 12 : model_.gated ? 24 : 40);
}
template <typename Real>
int Engine::launch_gate_split(int which, PassArgs<Real> a, bool pdl) {
  if constexpr (sizeof(Real) == 4) {
    const size_t n = static_cast<size_t>(std::max(1, ncentres_)) * model_.K * model_.H;
    const int mode = which == 0 ? kModeGateForward : kModeGateReverse;
    a.grid_mode = pass_grid_[mode];
    a.atom_order = pass_order_[mode];
    a.block_warps = pass_wpb_[mode];
    int k = 0;
    // moments or their adjoints; the gate values kept for the reverse, then the adjoints of h
    mom_.ensure(sizeof(Real) * n);
    a.mom = a.amom = mom_.as<Real>();
    const size_t nkeep = static_cast<size_t>((std::max(1, ncentres_) + kGraphAtoms - 1) / kGraphAtoms) * kGraphAtoms *
                         std::max(1, a.dm.gate.block.nkeep);
    gkeep_.ensure(sizeof(Real) * (nkeep + static_cast<size_t>(std::max(1, ncentres_)) * model_.F));
    a.gkeep = gkeep_.as<Real>();
    a.hbar = gkeep_.as<Real>() + nkeep;
    if (which == 0) {
      k += launch_shape<Real>(kModeGateFwdEdges, a, gate_split_blocks_[0], pdl);
      k += launch_atom_graph(a, sm_count_, stream_, 1);
    } else {
      if (!a.hbar_atom) k += launch_hbar_sum(a, stream_);
      k += launch_atom_graph(a, sm_count_, stream_, 2);
      k += launch_shape<Real>(kModeGateRevEdges, a, gate_split_blocks_[1], false);
    }
    return k;
  } else {
    throw Error(1, "the split passes run on FP32 engines");
  }
}

// One per-atom pass in the tile shape chosen for its mode (the defaults until autotune runs).
template <typename Real>
int Engine::launch_pass(int mode, PassArgs<Real> a, bool pdl) {
  a.grid_mode = pass_grid_[mode];
  a.atom_order = pass_order_[mode];
  a.h_bulk = pass_stage_[mode];
  a.block_warps = pass_wpb_[mode];
  return launch_shape<Real>(mode, a, pass_blocks_[mode], pdl);
}

// One pass launch in the shape already set in `a` (budget `blocks`); the dynamic centre order
// takes its mode's counter pair.
template <typename Real>
int Engine::launch_shape(int mode, PassArgs<Real> a, int blocks, bool pdl) {
  // the dynamic order's counter pair of this mode (zero between launches: the launch's last
  // warp resets it, so no memset sits between this launch and its predecessor)
  if (a.atom_order == 2) a.work = work_.as<int>() + 2 * mode;
  // FP64: the kept functions' rows, for up to 16 resident warps per SM (fused passes) or for the
  // centres of layouts up to kKeepCentres (gate passes); larger ones, and any on a device without the
  // room, evaluate them again in the reverse
  if (pass_keeps<Real>(mode)) {
    const bool gate = mode == kModeGateForward || mode == kModeGateReverse;
    DevBuf& buf = gate ? keep_gate_ : keep_;
    a.keep_rows = !gate ? std::min(16 * sm_count_, (ncentres_ + 3) / 4 * 4) : ncentres_ <= kKeepCentres ? ncentres_ : 0;
    const size_t bytes = sizeof(Real) * pass_keep_values(model_.L, model_.F) * a.keep_rows;
    if (!keep_size_[gate].holds(buf.bytes, bytes, [&](size_t n) { return buf.try_ensure(n); })) a.keep_rows = 0;
    a.keep = buf.as<Real>();
  }
  const int warps = launch_atom_pass<Real>(model_.L, mode, a, sm_count_, stream_, blocks, pdl);
  if (warps) ran_warps_[mode] = warps;
  return warps ? 1 : 0;
}

void Engine::pass_shape(int mode, int* shape4) const {
  const bool gate = mode == kModeGateForward || mode == kModeGateReverse;
  const bool runs = mode == kModeStatic ? !model_.gated : model_.gated;
  const bool fp32 = precision_ == kFP32;
  const bool split = runs && (gate ? (fp32 ? use_gate_split<float>() : use_gate_split<double>())
                                   : (fp32 ? use_static_split<float>() : use_static_split<double>()));
  int kernel = mode;  // whose launch has the pass's block size
  if (split) kernel = mode == kModeStatic ? kModeStaticFwd : mode == kModeOuter ? kModeOuterFwd
                                          : mode == kModeGateForward ? kModeGateFwdEdges : kModeGateRevEdges;
  shape4[0] = !split ? pass_blocks_[mode] : gate ? gate_split_blocks_[mode == kModeGateForward ? 0 : 1] : split_blocks_;
  shape4[1] = pass_grid_[mode];
  shape4[2] = pass_order_[mode] + (split ? 4 : 0) + (pass_stage_[mode] ? 8 : 0);
  shape4[3] = pass_wpb_[mode] ? pass_wpb_[mode] : ran_warps_[kernel] ? ran_warps_[kernel] : kPassWarps;
}

// Pass-kernel autotuner: on the current layout (the last evaluation's edges), times each pass the
// model runs in every tile shape -- register budget (3 or 4 resident blocks per SM), grid (all
// resident blocks, or the fewest that keep the same centres per warp), centre order (grid-
// strided, contiguous runs per warp, or taken from a device counter) and, for the Effect outer
// pass, the staging of the neighbours' gate-signal rows (plain loads or bulk async copies) --
// `reps` launches each after one warm-up launch, and keeps the fastest shape per pass; then, for
// FP32 models of basis size 8, the pass split at the per-atom boundary in the chosen grid and
// order with either budget, kept where faster.  ms_out[2 mode + (budget - 3)] = the best time of
// each budget (fused).
// The passes read the state the evaluation before them left (gate signals, node adjoints), so a
// full evaluation runs first; the gate reverse pass accumulates into the edge gradients, so the
// next evaluation recomputes them.
template <typename Real>
void Engine::autotune_passes(int reps, int* blocks_out, double* ms_out) {
  const Model& m = model_;
  cudaStream_t s = stream_;
  const int N = natoms_;
  double* scratch = static_cast<double*>(io(7, sizeof(double) * (7 * static_cast<size_t>(std::max(1, nframes_)) +
                                                                  4 * static_cast<size_t>(std::max(1, N)))));
  run_efs<Real>(scratch, scratch + 7 * std::max(1, nframes_), scratch + std::max(1, nframes_), nullptr, kStageAll);
  PassArgs<Real> a = pass_args<Real>();
  if (m.gated) {  // the fused gate passes are timed too
    gmom_.ensure(sizeof(Real) * static_cast<size_t>(std::max(1, N)) * m.M);
    a.gmom = gmom_.as<Real>();
  }
  const int modes_static[] = {kModeStatic};
  const int modes_gated[] = {kModeGateForward, kModeOuter, kModeGateReverse};
  const int* modes = m.gated ? modes_gated : modes_static;
  const int nmodes = m.gated ? 3 : 1;
  for (int q = 0; q < 4; ++q) { blocks_out[q] = 0; ms_out[2 * q] = ms_out[2 * q + 1] = 0.0; }
  cudaEvent_t e0 = take_event(), e1 = take_event();
  auto timed = [&](auto&& launch) {  // milliseconds per launch, after one warm-up
    launch();
    SUS2G_CUDA(cudaEventRecord(e0, s));
    for (int r = 0; r < reps; ++r) launch();
    SUS2G_CUDA(cudaEventRecord(e1, s));
    SUS2G_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    SUS2G_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    return double(ms) / std::max(1, reps);
  };
  double gate_gain = 0.0;  // milliseconds the split gate passes save together
  for (int k = 0; k < nmodes; ++k) {
    const int mode = modes[k];
    double best = 0.0;
    int choice = 0, choice_grid = 0, choice_order = 0, choice_stage = 0, choice_wpb = kPassWarps;
    // h_j staging by bulk copies: the outer pass only (basis size 8), where a row is whole
    // 16-byte units
    const int stages = pass_h_bulk<Real>(mode, 1, m.F) && m.B == 8 ? 2 : 1;
    for (int blocks = 3; blocks <= 4; ++blocks)
      for (int grid = 0; grid <= 1; ++grid)
        for (int order = 0; order <= 2; ++order)
          for (int stage = 0; stage < stages; ++stage)
          for (int wpb = 2; wpb <= kPassWarps; wpb += 2) {
            a.grid_mode = grid;
            a.atom_order = order;
            a.h_bulk = stage;
            a.block_warps = wpb;
            const double per = timed([&] { launch_shape<Real>(mode, a, blocks, false); });
            double& slot = ms_out[2 * mode + (blocks - 3)];
            if (slot == 0.0 || per < slot) slot = per;
            if (choice == 0 || per < best) {
              best = per; choice = blocks; choice_grid = grid; choice_order = order; choice_stage = stage;
              choice_wpb = wpb;
            }
          }
    a.h_bulk = 0;
    pass_blocks_[mode] = choice;
    pass_grid_[mode] = choice_grid;
    pass_order_[mode] = choice_order;
    pass_stage_[mode] = choice_stage;
    pass_wpb_[mode] = choice_wpb;
    blocks_out[mode] = choice;
    if ((mode == kModeStatic || mode == kModeOuter) && sizeof(Real) == 4 && m.B == 8) {
      // the fused energy pass (Static, or Effect outer) against its three-kernel split, in the
      // chosen grid and centre order, the split kernels with either register budget
      static_split_ = 0;
      if (split_fits(false)) {
        double split_best = 0.0;
        int split_choice = 0;
        for (int blocks = 3; blocks <= 4; ++blocks) {
          split_blocks_ = blocks;
          const double per = timed([&] { launch_static_split<Real>(a, false); });
          if (split_choice == 0 || per < split_best) { split_best = per; split_choice = blocks; }
        }
        split_blocks_ = split_choice;
        static_split_ = split_best < best ? 1 : 0;
      }
    }
    if ((mode == kModeGateForward || mode == kModeGateReverse) && sizeof(Real) == 4 && m.B == 8 && split_fits(true)) {
      // each gate pass against its split (per-edge kernel with either budget, per-atom kernel)
      const int which = mode == kModeGateForward ? 0 : 1;
      double split_best = 0.0;
      int split_choice = 0;
      for (int blocks = 3; blocks <= 4; ++blocks) {
        gate_split_blocks_[which] = blocks;
        const double per = timed([&] { launch_gate_split<Real>(which, a, false); });
        if (split_choice == 0 || per < split_best) { split_best = per; split_choice = blocks; }
      }
      gate_split_blocks_[which] = split_choice;
      gate_gain += best - split_best;
    }
  }
  // the two gate passes take the same form (the split ones share the kept gate values)
  gate_split_ = gate_gain > 0.0 ? 1 : 0;
  event_next_ = 0;
  reset_step_graph();  // a captured step holds the previous budgets
  // graphs captured elsewhere (a trainer's evaluation graph) hold them too: a new edge generation
  // makes their owners rebind and capture again
  ++edge_generation_;
}

void Engine::autotune(int reps, int* blocks_out, double* ms_out) {
  SUS2G_CUDA(cudaSetDevice(device_));
  if (natoms_ <= 0 || ncentres_ <= 0) throw Error(1, "autotune needs an evaluated layout: evaluate once first");
  if (timing_) throw Error(1, "autotune: turn the stage timer off first");
  wait_reverse();
  if (precision_ == kFP32) autotune_passes<float>(reps, blocks_out, ms_out);
  else autotune_passes<double>(reps, blocks_out, ms_out);
  check_device_error();
}

void Engine::set_pass_shape(int mode, int blocks, int grid, int order, int stage, int warps) {
  if (mode < 0 || mode > 3) throw Error(1, "pass shape: mode must be 0 .. 3");
  if (blocks != 0 && blocks != 3 && blocks != 4) throw Error(1, "pass shape: blocks per SM must be 0, 3 or 4");
  if (grid < 0 || grid > 1 || order < 0 || order > 2) throw Error(1, "pass shape: grid 0 .. 1, order 0 .. 2");
  if (stage < 0 || stage > 1) throw Error(1, "pass shape: staging 0 or 1");
  if (warps < 1 || warps > kPassWarps) throw Error(1, "pass shape: warps per block 1 .. 4");
  pass_wpb_[mode] = warps;
  pass_blocks_[mode] = blocks;
  pass_grid_[mode] = grid;
  pass_order_[mode] = order;
  pass_stage_[mode] = stage;
  // a pinned shape is the fused pass's
  if ((mode == kModeStatic || mode == kModeOuter) && static_split_ < 0) static_split_ = 0;
  if ((mode == kModeGateForward || mode == kModeGateReverse) && gate_split_ < 0) gate_split_ = 0;
  reset_step_graph();
  ++edge_generation_;  // graphs captured by other owners hold the previous shape
}

void Engine::reset_step_graph() {
  if (step_exec_) cudaGraphExecDestroy(step_exec_);
  if (step_graph_) cudaGraphDestroy(step_graph_);
  step_exec_ = nullptr;
  step_graph_ = nullptr;
  step_key_.clear();
}

void Engine::step_frames(int nframes, const int* frame_natoms, const double* cells, const double* d_pos,
                         const int* d_types, double* d_energy, double* d_forces, double* d_virial, double* d_site) {
  SUS2G_CUDA(cudaSetDevice(device_));
  // layout key: everything the captured launches depend on besides device memory contents
  std::vector<double> key;
  key.reserve(16 + 10 * static_cast<size_t>(std::max(0, nframes)));
  auto ptr = [](const void* p) { return static_cast<double>(reinterpret_cast<uintptr_t>(p)); };
  key.push_back(nframes);
  for (int f = 0; f < nframes; ++f) {
    key.push_back(frame_natoms[f]);
    for (int q = 0; q < 9; ++q) key.push_back(cells[9 * f + q]);
  }
  for (const void* p : {static_cast<const void*>(d_pos), static_cast<const void*>(d_types),
                        static_cast<const void*>(d_energy), static_cast<const void*>(d_forces),
                        static_cast<const void*>(d_virial), static_cast<const void*>(d_site),
                        static_cast<const void*>(stream_)})
    key.push_back(ptr(p));
  key.push_back(cap_scale_);
  key.push_back(min_cap_);
  key.push_back(bin_cap_scale_);
  key.push_back(min_bin_cap_);
  // the same layout as the previous step, with no other edge build, staged call or parameter
  // upload since (those may have regrown the buffers whose addresses a graph holds)
  const bool same = step_graphs_ && !timing_ && key == step_key_ && edge_generation_ == step_gen_;
  if (same && step_exec_) {
    SUS2G_CUDA(cudaGraphLaunch(step_exec_, stream_));
    launches_ += step_launches_;
    step_gen_ = ++edge_generation_;  // the replay rebuilds the edge arrays
    nedges_exact_ = false;
    return;
  }
  // periodic batches build their edges without host synchronisation: the second step of a layout
  // is captured and launched, later ones replay (a one-off layout is never captured)
  if (same && nframes > 0) {
    reset_step_graph();
    const int before = launches_;
    capturing_ = true;
    cudaGraph_t graph = nullptr;
    cudaError_t err = cudaStreamBeginCapture(stream_, cudaStreamCaptureModeRelaxed);
    if (err == cudaSuccess) {
      try {
        build_edges(nframes, frame_natoms, cells, d_pos, d_types);
        efs(d_energy, d_forces, d_virial, d_site);
      } catch (...) {
        capturing_ = false;
        cudaStreamEndCapture(stream_, &graph);
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        launches_ = before;
        throw;
      }
      err = cudaStreamEndCapture(stream_, &graph);
    }
    capturing_ = false;
    step_launches_ = launches_ - before;
    launches_ = before;  // the capture ran nothing
    if (err == cudaSuccess && graph && cudaGraphInstantiate(&step_exec_, graph, 0) == cudaSuccess) {
      step_graph_ = graph;
      SUS2G_CUDA(cudaGraphLaunch(step_exec_, stream_));
      launches_ += step_launches_;
      step_key_ = key;
      step_gen_ = edge_generation_;
      return;
    }
    // capture refused (e.g. a legacy-stream caller): run this step eagerly and stop capturing
    cudaGetLastError();
    if (graph) cudaGraphDestroy(graph);
    step_exec_ = nullptr;
    step_graphs_ = false;
  } else {
    reset_step_graph();
  }
  build_edges(nframes, frame_natoms, cells, d_pos, d_types);
  efs(d_energy, d_forces, d_virial, d_site);
  step_key_ = key;
  step_gen_ = edge_generation_;
}

void Engine::stage_begin(int nowned, int nall, const int* d_types, int nedges, const int* d_i, const int* d_j,
                         const double* d_d) {
  set_edges(nowned, nall, d_types, nedges, d_i, d_j, d_d);
  if (precision_ == kFP32) run_efs<float>(nullptr, nullptr, nullptr, nullptr, kStageGate);
  else run_efs<double>(nullptr, nullptr, nullptr, nullptr, kStageGate);
  staged_ = 1;
}

void Engine::stage_outer() {
  SUS2G_CUDA(cudaSetDevice(device_));
  if (staged_ != 1) throw Error(1, "staged evaluation: outer() needs begin() first");
  if (precision_ == kFP32) run_efs<float>(nullptr, nullptr, nullptr, nullptr, kStageOuter);
  else run_efs<double>(nullptr, nullptr, nullptr, nullptr, kStageOuter);
  staged_ = 2;
}

void Engine::stage_finish(double* d_energy, double* d_forces, double* d_virial, double* d_site) {
  SUS2G_CUDA(cudaSetDevice(device_));
  if (staged_ != 2) throw Error(1, "staged evaluation: finish() needs outer() first");
  if (precision_ == kFP32) run_efs<float>(d_energy, d_forces, d_virial, d_site, kStageFinish);
  else run_efs<double>(d_energy, d_forces, d_virial, d_site, kStageFinish);
  staged_ = 0;
}

void Engine::stage_rows(int which, int op, int n, const int* d_atoms, int first, double* d_buf) {
  SUS2G_CUDA(cudaSetDevice(device_));
  if (!model_.gated || n <= 0) return;
  const int W = model_.F;
  // forward exchange (h) between begin and outer; reverse exchange (hbar) between outer and finish
  if (which == 0 && staged_ != 1) throw Error(1, "staged evaluation: the gate-signal exchange runs between begin() and outer()");
  if (which == 1 && staged_ != 2) throw Error(1, "staged evaluation: the adjoint exchange runs between outer() and finish()");
  if (!d_atoms && (first < 0 || first + n > natoms_)) throw Error(1, "staged evaluation: atom range outside the layout");
  const long long t = static_cast<long long>(n) * W;
  const unsigned blocks = static_cast<unsigned>((t + 255) / 256);
  cudaStream_t s = stream_;
  if (which == 0) {
    if (op == 0) {
      if (precision_ == kFP32) k_rows_pack<float><<<blocks, 256, 0, s>>>(hsig_.as<float>(), W, n, d_atoms, first, d_buf);
      else k_rows_pack<double><<<blocks, 256, 0, s>>>(hsig_.as<double>(), W, n, d_atoms, first, d_buf);
    } else {
      if (precision_ == kFP32) k_rows_unpack<float><<<blocks, 256, 0, s>>>(hsig_.as<float>(), W, n, d_atoms, first, d_buf, 0);
      else k_rows_unpack<double><<<blocks, 256, 0, s>>>(hsig_.as<double>(), W, n, d_atoms, first, d_buf, 0);
    }
  } else {
    if (op == 0) k_rows_pack<double><<<blocks, 256, 0, s>>>(hbar_atom_.as<double>(), W, n, d_atoms, first, d_buf);
    else k_rows_unpack<double><<<blocks, 256, 0, s>>>(hbar_atom_.as<double>(), W, n, d_atoms, first, d_buf, 1);
  }
  ++launches_;
}

}  // namespace sus2g
