// The per-atom Verlet list from atoms sorted by cell, shared by the
// reference-layout launcher (FP32) and the plain form (FP64): neighbors[k * n + i]
// in the reference's candidate order (27 cells in dz, dy, dx order, members in
// sorted order; neighbor/verlet_list.cu:154-327).  Both users are compiled
// without contraction, so the pair predicate rounds as the reference's.
//
// k_list_cells, a block per home cell (list_grid): the 27 cells' atoms are staged in shared
// memory once for the cell's atoms, a warp takes one home atom at a time, its
// lanes test 32 candidates and a ballot compacts the hits in candidate order.
// The thread-per-atom form it stands beside follows two dependent loads per
// candidate (sorted index -> position) and was bound by their latency: 100,000
// atoms, rc + skin 2.8 at density 0.85, 212 us against 115 (now bound by issue,
// 71 % active).  It remains where cells are
// mostly empty (list_by_cells): there a block per cell would find nothing to do.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

namespace fmd {
namespace cells {

constexpr int kThreads = 128, kWarps = kThreads / 32;
constexpr int kWin = 768;   // candidates staged per window (a multiple of 32): one 27-cell stencil of a dense melt
constexpr int kGroup = 64;  // home atoms per pass

// Cells hold four atoms or more on average, and the 27 cells are distinct.
inline bool list_by_cells(int n, int nx) { return nx >= 3 && (int64_t)n >= 4ll * nx * nx * nx; }

// A block per home cell and kGroup of its atoms on average: a box of few cells
// with many atoms each would leave most SMs without a block (20,000 atoms in 27
// cells, rc + skin 9: 19.3 ms with one block per cell, 2.9 now, 7.0 with a
// thread per atom).
inline dim3 list_grid(int n, int ncell) {
  const long long per_cell = ((long long)n + ncell - 1) / ncell;
  const long long groups = (per_cell + kGroup - 1) / kGroup;
  return dim3((unsigned)ncell, (unsigned)(groups < 65535 ? groups : 65535));
}

// Key bits of ncell cell numbers (radix passes over the others are left out).
inline int key_bits(int ncell) {
  int b = 1;
  while (b < 31 && (1 << b) < ncell) ++b;
  return b;
}

__device__ __forceinline__ float from_index(int i, float) { return __int_as_float(i); }
__device__ __forceinline__ double from_index(int i, double) { return (double)i; }
__device__ __forceinline__ int to_index(float w) { return __float_as_int(w); }
__device__ __forceinline__ int to_index(double w) { return (int)w; }
__device__ __forceinline__ float image(float d, float L, float inv_L) { return d - L * rintf(d * inv_L); }
__device__ __forceinline__ double image(double d, double L, double inv_L) { return d - L * rint(d * inv_L); }

// Positions in sorted order, .w = the atom's index; the cells' ranges.
template <typename V4, typename Real>
__global__ void k_sorted(const V4* pos, const int* sorted, const int* scid, int* start, int* end, V4* spos, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c = scid[k], i = sorted[k];
  if (k == 0 || scid[k - 1] != c) start[c] = k;
  if (k == n - 1 || scid[k + 1] != c) end[c] = k + 1;
  V4 p = pos[i];
  p.w = from_index(i, Real());
  spos[k] = p;
}

// One home atom against the staged window; NEAR: every separation in the
// window is below half a box, so the minimum image is the difference itself.
template <bool NEAR, typename V4, typename Real>
__device__ __forceinline__ int test_window(const V4* s_c, int wn, V4 pi, int i, int excluded, int ne, Real rcs2,
                                           Real L, Real inv_L, int* nbr, int64_t n, int max_nbr, int count, int lane) {
  const uint32_t below = (1u << lane) - 1u;
  // room for every lane of every batch: no test per hit
  const bool roomy = count + ((wn + 31) & ~31) <= max_nbr;
  int* const out = nbr + i;
#pragma unroll 2
  for (int c0 = 0; c0 < wn; c0 += 32) {
    const V4 c = s_c[c0 + lane];
    Real dx = pi.x - c.x, dy = pi.y - c.y, dz = pi.z - c.z;
    if (!NEAR) {
      dx = image(dx, L, inv_L);
      dy = image(dy, L, inv_L);
      dz = image(dz, L, inv_L);
    }
    const Real r2 = dx * dx + dy * dy + dz * dz;
    const int j = to_index(c.w);
    bool hit = r2 < rcs2 && j != i;  // the window's padding is NaN: never
    for (int e = 0; e < ne; ++e) {  // every lane takes part in the shuffles
      const int out = __shfl_sync(0xFFFFFFFFu, excluded, e);
      hit &= out != j;
    }
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
    const int at = count + __popc(m & below);
    if (hit && (roomy || at < max_nbr)) out[at * n] = j;
    count += __popc(m);
  }
  return count;
}

template <typename V4, typename Real>
__global__ void __launch_bounds__(kThreads) k_list_cells(const V4* spos, const int* start, const int* end,
                                                         const int* eoff, const int* elist, int* nbr, int* cnt, int n,
                                                         int nx, Real rcs2, Real L, Real inv_L, int max_nbr,
                                                         int* overflow, int overflow_bit) {
  const int hs = start[blockIdx.x], nh = end[blockIdx.x] - hs;
  if (nh <= (int)blockIdx.y * kGroup) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cx = blockIdx.x % nx, cy = (blockIdx.x / nx) % nx, cz = blockIdx.x / (nx * nx);
  __shared__ V4 s_c[kWin];
  __shared__ int s_ns[27], s_off[28], s_cnt[kGroup];
  if (warp == 0) {
    int m = 0;
    if (lane < 27) {
      int x = cx + lane % 3 - 1, y = cy + (lane / 3) % 3 - 1, z = cz + lane / 9 - 1;
      x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
      y = y < 0 ? y + nx : (y >= nx ? y - nx : y);
      z = z < 0 ? z + nx : (z >= nx ? z - nx : z);
      const int c = (z * nx + y) * nx + x;
      s_ns[lane] = start[c];
      m = end[c] - s_ns[lane];
    }
    int incl = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane < 27) s_off[lane + 1] = incl;
    if (lane == 0) s_off[0] = 0;
  }
  // Within 0.24 L of the home cell's centre on every axis, two positions are
  // less than 0.48 L apart: the image is the difference itself.  Positions
  // outside the box, and cells across a face, take the general form.
  const Real cell = L / (Real)nx, reach = (Real)0.24 * L;
  const Real ox = ((Real)cx + (Real)0.5) * cell, oy = ((Real)cy + (Real)0.5) * cell, oz = ((Real)cz + (Real)0.5) * cell;
  auto near_home = [&](const V4& p) { return fabs(p.x - ox) < reach && fabs(p.y - oy) < reach && fabs(p.z - oz) < reach; };
  __syncthreads();
  const int total = s_off[27];
  for (int hg = blockIdx.y * kGroup; hg < nh; hg += gridDim.y * kGroup) {
    const int gn = min(kGroup, nh - hg);
    for (int w0 = 0; w0 < total; w0 += kWin) {
      const int wn = min(kWin, total - w0);
      __syncthreads();  // the previous window is no longer read
      bool near = true;
      for (int t = warp; t < 27; t += kWarps) {
        const int lo = max(s_off[t], w0), hi = min(s_off[t + 1], w0 + wn);
        for (int k = lo + lane; k < hi; k += 32) {
          const V4 p = spos[s_ns[t] + (k - s_off[t])];
          near = near && near_home(p);
          s_c[k - w0] = p;
        }
      }
      const int padded = (wn + 31) & ~31;
      if (wn + (int)threadIdx.x < padded) {
        V4 none;
        none.x = none.y = none.z = (Real)NAN;
        none.w = from_index(-1, Real());
        s_c[wn + threadIdx.x] = none;
      }
      near = __syncthreads_and(near);
      for (int a = warp; a < gn; a += kWarps) {
        const V4 pi = spos[hs + hg + a];
        const int i = to_index(pi.w);
        const int e0 = eoff ? eoff[i] : 0, ne = eoff ? eoff[i + 1] - e0 : 0;
        int count = w0 == 0 ? 0 : s_cnt[a];
        if (ne <= 32) {
          const int excluded = lane < ne ? elist[e0 + lane] : -1;
          if (near && near_home(pi))
            count = test_window<true, V4, Real>(s_c, wn, pi, i, excluded, ne, rcs2, L, inv_L, nbr, n, max_nbr, count, lane);
          else
            count = test_window<false, V4, Real>(s_c, wn, pi, i, excluded, ne, rcs2, L, inv_L, nbr, n, max_nbr, count, lane);
        } else {  // more exclusions than lanes: each hit walks the list
          for (int c0 = 0; c0 < wn; c0 += 32) {
            const V4 c = s_c[c0 + lane];
            const Real dx = image(pi.x - c.x, L, inv_L), dy = image(pi.y - c.y, L, inv_L), dz = image(pi.z - c.z, L, inv_L);
            const Real r2 = dx * dx + dy * dy + dz * dz;
            const int j = to_index(c.w);
            bool hit = r2 < rcs2 && j != i && c0 + lane < wn;
            for (int e = 0; hit && e < ne; ++e) hit = elist[e0 + e] != j;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
            const int at = count + __popc(m & ((1u << lane) - 1u));
            if (hit && at < max_nbr) nbr[(int64_t)at * n + i] = j;
            count += __popc(m);
          }
        }
        if (lane == 0) {
          s_cnt[a] = count;
          if (w0 + kWin >= total) {
            cnt[i] = min(count, max_nbr);
            if (count > max_nbr && overflow) atomicOr(overflow, overflow_bit);
          }
        }
        __syncwarp();
      }
    }
  }
}

}  // namespace cells
}  // namespace fmd
