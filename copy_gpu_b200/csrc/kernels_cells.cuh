// kernels_cells.cuh -- cell binning, deterministic cell sort and the full neighbour list.
//
// Reference: ContPointLocator::Build + BinPointsWorklet (rbmd/framework/locator/
// ContPointLocator.cxx:38-92) does bin -> SortByKey -> Lower/UpperBounds with library calls.
// Here: fused bin + per-cell atomic count (in the integrator or k_bin), one-block scan, atomic
// scatter, then a warp per cell ranks its atoms by caller id so the slot order is deterministic
// (a stable sort by (cell, id)), and the same warp gathers the slot-ordered caches.
#pragma once
#include "common.cuh"

namespace rbmd {

// cell index of a position, BinPointsWorklet semantics (truncate, clamp to [0, dims-1])
// Cell index of coordinate x along axis d, unclamped to the box but bounded, so that sums with stencil
// offsets and cell counts stay in 32 bits for an atom far outside (an overflowed sum read cell_start out
// of range).  No pair is accepted so far out, whatever cells are searched.
constexpr int kCellIndexMax = 1 << 30;
template <class R>
__device__ __forceinline__ int cell_index(const RepDev& rp, int d, R x) {
  const int c = (int)div_rn(sub_rn(x, Traits<R>::lo(rp, d)), Traits<R>::dx(rp, d));
  return max(-kCellIndexMax, min(kCellIndexMax, c));
}

template <class R>
__device__ __forceinline__ int cell_of_pos(const RepDev& rp, R x, R y, R z) {
  R p[3] = {x, y, z};
  int ijk[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int c = (int)div_rn(sub_rn(p[d], Traits<R>::lo(rp, d)), Traits<R>::dx(rp, d));
    c = max(c, 0);
    c = min(c, rp.dims[d] - 1);
    ijk[d] = c;
  }
  return rp.cell_base + ijk[0] + ijk[1] * rp.dims[0] + ijk[2] * rp.dims[0] * rp.dims[1];
}

// Verlet-skin rebuild flags: rebuild[r] for replica r and rebuild[n_replicas] for "any replica";
// a replica whose atoms all stayed within skin/2 keeps its cells, slots and list.
// rebuild (nullable): bin only the atoms of rebuilding replicas.  xref (nullable): the positions of
// this build, in caller order, so consecutive here (the cell sort would scatter them).
template <class R>
__global__ void k_bin(int n, const double* __restrict__ pos, const int* __restrict__ rep_of,
                      const RepDev* __restrict__ reps, int* __restrict__ cell_of,
                      int* __restrict__ cell_count, uint32_t* status, const int* __restrict__ rebuild,
                      double* __restrict__ xref) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rep_of ? rep_of[i] : 0;
  if (rebuild && !rebuild[r]) return;
  const RepDev& rp = reps[r];
  double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  if (!isfinite(x) || !isfinite(y) || !isfinite(z)) set_flag(status, kFlagNonFinite);
  if (xref) { xref[3 * i] = x; xref[3 * i + 1] = y; xref[3 * i + 2] = z; }
  int c = cell_of_pos<R>(rp, (R)x, (R)y, (R)z);
  cell_of[i] = c;
  atomicAdd(&cell_count[c], 1);
}

// Exclusive scan of the cell counts in two parallel passes: k_cell_block_sums reduces blocks of
// kScanBlock cells; k_cell_scan gives each block its prefix (sum of the preceding block sums)
// and scans its cells.  cell_start[ncell] = n; scatter cursors are cleared; over-full cells flag.
// `rebuild` (nullable, the "any replica" flag): skip the pass when every list is reused.  Cells
// of replicas that keep their list keep their counts, so their starts come out unchanged.
constexpr int kScanBlock = 4096;

// Number of replicas whose list is rebuilt in this pass (the list-build counter counts replica
// lists: with one replica, the number of rebuilding passes).
__device__ __forceinline__ unsigned long long rebuilt_replicas(const int* rebuild, int n_rep) {
  if (!rebuild) return (unsigned long long)n_rep;
  unsigned long long c = 0;
  for (int r = 0; r < n_rep; ++r) c += rebuild[r] != 0;
  return c;
}

// Zero the cell counts of the rebuilding replicas (all of them when rebuild is null).
__global__ void k_zero_counts(int ncell, const int* __restrict__ cell_rep, const int* __restrict__ rebuild,
                              int* __restrict__ cell_count) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  if (rebuild && !rebuild[cell_rep ? cell_rep[c] : 0]) return;
  cell_count[c] = 0;
}

__global__ void __launch_bounds__(1024) k_cell_block_sums(int ncell, const int* __restrict__ count,
                                                          int* __restrict__ block_sums,
                                                          const int* __restrict__ rebuild,
                                                          uint32_t* status) {
  if (rebuild && !*rebuild) return;
  __shared__ int red[32];
  const int b0 = blockIdx.x * kScanBlock;
  int s = 0, mx = 0;
  for (int c = b0 + threadIdx.x; c < min(ncell, b0 + kScanBlock); c += blockDim.x) {
    const int v = count[c];
    s += v;
    mx = max(mx, v);
  }
  if (mx > kMaxCellAtoms) set_flag(status, kFlagCellOverflow);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    block_sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(1024) k_cell_scan(int ncell, const int* __restrict__ count,
                                                    const int* __restrict__ block_sums,
                                                    int* __restrict__ start, int* __restrict__ cursor,
                                                    const int* __restrict__ rebuild) {
  if (rebuild && !*rebuild) return;
  __shared__ int warp_sums[32];
  __shared__ int base_sh;
  const int t = threadIdx.x, nt = blockDim.x;
  const int b0 = blockIdx.x * kScanBlock, b1 = min(ncell, b0 + kScanBlock);
  if (t < 32) {
    int v = 0;
    for (int b = t; b < (int)blockIdx.x; b += 32) v += block_sums[b];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (t == 0) base_sh = v;
  }
  // each thread owns kScanBlock / nt consecutive cells
  const int per = kScanBlock / nt;
  const int c0 = b0 + t * per;
  int local = 0;
  for (int c = c0; c < min(b1, c0 + per); ++c) local += count[c];
  const int lane = t & 31, w = t >> 5;
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sums[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int v = lane < (nt >> 5) ? warp_sums[lane] : 0;
    int inc2 = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc2, o);
      if (lane >= o) inc2 += y;
    }
    warp_sums[lane] = inc2 - v;
  }
  __syncthreads();
  int run = base_sh + warp_sums[w] + incl - local;
  for (int c = c0; c < min(b1, c0 + per); ++c) {
    start[c] = run;
    cursor[c] = 0;
    run += count[c];
  }
  if (b1 == ncell && t == nt - 1) start[ncell] = run;
}

__global__ void k_scatter(int n, const int* __restrict__ cell_of, const int* __restrict__ start,
                          int* __restrict__ cursor, int* __restrict__ tmp_slot_atom,
                          const int* __restrict__ rep_of, const int* __restrict__ rebuild) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (rebuild && !rebuild[rep_of ? rep_of[i] : 0]) return;
  int c = cell_of[i];
  int s = start[c] + atomicAdd(&cursor[c], 1);
  tmp_slot_atom[s] = i;
}

// Total order of positions for the cell sort: IEEE bits mapped so that unsigned comparison
// follows the float order (NaNs land at the ends, so a rank is always a permutation).
__device__ __forceinline__ uint32_t ord_key(float x) {
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ unsigned long long ord_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// One warp per cell: rank the cell's atoms by caller id (ids are distinct), or with sort_x by
// (x in the run precision, caller id), and gather the slot-ordered caches.  With sort_x every
// row of consecutive x cells is ordered by x, which lets the list build skip the candidates
// beyond the cutoff in x by binary search.  Cells above kMaxCellAtoms keep the scatter order
// (flagged by the scan).
// SPLIT (cells of many atoms): a cell is shared by nparts warps, each ranking its share of the
// atoms against all of them (30,000 water atoms fill 216 cells, 54 blocks of one warp per cell:
// 37 -> 16 us with parts).  Without it no index is divided: the warps of empty cells, most of a dilute
// or droplet system, do little else (300,000 atoms at 0.05 atoms a cell, whole sort: 1887 us with 64-bit
// divisions, 1239 without any).
constexpr int kSortWarps = 4;   // warps per block of k_cell_sort_gather

template <class R, bool SPLIT>
__global__ void __launch_bounds__(32 * kSortWarps) k_cell_sort_gather(
    int ncell, int nparts, const int* __restrict__ start, const int* __restrict__ tmp_slot_atom,
    const double* __restrict__ pos, const double* __restrict__ charge,
    const int* __restrict__ type, const int* __restrict__ mol, const int* __restrict__ rep_of,
    const RepDev* __restrict__ reps, int* __restrict__ slot_atom, int* __restrict__ atom_slot,
    typename Traits<R>::V4* __restrict__ pos4, void* __restrict__ frac_out,
    int2* __restrict__ meta, const int* __restrict__ rebuild, int sort_x, const int* __restrict__ cell_rep) {
  using Key = decltype(ord_key((R)0));
  __shared__ int ids[kSortWarps][kMaxCellAtoms];
  __shared__ Key keys[kSortWarps][kMaxCellAtoms];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned item = blockIdx.x * kSortWarps + w;   // below 2^32: ncell + atoms / 32 warps
  int cell = (int)item, part = 0;
  if (SPLIT) {
    cell = (int)(item / (unsigned)nparts);
    part = (int)(item % (unsigned)nparts);
  }
  if (cell >= ncell) return;
  if (rebuild && !rebuild[cell_rep ? cell_rep[cell] : 0]) return;
  const int s0 = start[cell], n = start[cell + 1] - s0;
  int k0 = 0, k1 = n;
  if (SPLIT) {
    k0 = (int)((long long)n * part / nparts);
    k1 = (int)((long long)n * (part + 1) / nparts);
  }
  if (k0 == k1) return;
  const bool sortable = n <= kMaxCellAtoms;
  if (sortable)
    for (int k = lane; k < n; k += 32) {
      const int id = tmp_slot_atom[s0 + k];
      ids[w][k] = id;
      if (sort_x) keys[w][k] = ord_key((R)pos[3 * id]);
    }
  __syncwarp();
  for (int k = k0 + lane; k < k1; k += 32) {
    int id = sortable ? ids[w][k] : tmp_slot_atom[s0 + k];
    int rank = k;
    if (sortable) {
      rank = 0;
      if (sort_x) {
        const Key kk = keys[w][k];
        for (int m = 0; m < n; ++m) {
          const Key km = keys[w][m];
          rank += km < kk || (km == kk && ids[w][m] < id);
        }
      } else {
        for (int m = 0; m < n; ++m) rank += ids[w][m] < id;
      }
    }
    const int slot = s0 + rank;
    slot_atom[slot] = id;
    atom_slot[id] = slot;
    const double x = pos[3 * id], y = pos[3 * id + 1], z = pos[3 * id + 2];
    const double q = charge ? charge[id] : 0.0;
    typename Traits<R>::V4 v;
    v.x = (R)x; v.y = (R)y; v.z = (R)z; v.w = (R)q;
    pos4[slot] = v;
    if (meta) meta[slot] = make_int2(type ? type[id] : 0, mol ? mol[id] : id);
    if (frac_out) {
      const RepDev& rp = reps[rep_of ? rep_of[id] : 0];
      double u[3] = {(x - rp.lo_d[0]) / rp.box_d[0], (y - rp.lo_d[1]) / rp.box_d[1],
                     (z - rp.lo_d[2]) / rp.box_d[2]};
      if (sizeof(R) == 4) {
        uint32_t U[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          U[d] = turn32(u[d] - floor(u[d]));
        }
        Frac32 fr{U[0], U[1], U[2], (float)q};
        reinterpret_cast<Frac32*>(frac_out)[slot] = fr;
      } else {
        unsigned long long U[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          U[d] = turn64(u[d] - floor(u[d]));
        }
        Frac64 fr{U[0], U[1], U[2], q};
        reinterpret_cast<Frac64*>(frac_out)[slot] = fr;
      }
    }
  }
}

// Refresh the slot caches from the master positions without re-binning (list reuse with skin).
// With xref (positions at the last build) the cached position is unwrapped: xref plus the
// minimum-image displacement since the build.  A listed pair's stored image shift then stays
// valid however often either atom crossed a face, so the pair kernels need no minimum-image
// step; the displacement is below skin/2, far under half a box.
template <class R>
__global__ void k_regather(int n, const int* __restrict__ slot_atom, const double* __restrict__ pos,
                           const double* __restrict__ charge, const int* __restrict__ rep_of,
                           const RepDev* __restrict__ reps, typename Traits<R>::V4* __restrict__ pos4,
                           void* __restrict__ frac_out, const double* __restrict__ xref,
                           const int* __restrict__ rebuild) {
  int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= n) return;
  int id = slot_atom[slot];
  if (rebuild && rebuild[rep_of ? rep_of[id] : 0]) return;   // the cell sort refreshed these caches
  const double x = pos[3 * id], y = pos[3 * id + 1], z = pos[3 * id + 2];
  const double q = charge ? charge[id] : 0.0;
  typename Traits<R>::V4 v;
  if (xref) {
    const RepDev& rp = reps[rep_of ? rep_of[id] : 0];
    double u[3] = {x, y, z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double r0 = xref[3 * id + d];
      double dd = u[d] - r0;
      if (fabs(dd) > 0.5 * rp.box_d[d]) dd -= (dd > 0 ? rp.box_d[d] : -rp.box_d[d]);
      u[d] = r0 + dd;
    }
    v.x = (R)u[0]; v.y = (R)u[1]; v.z = (R)u[2];
  } else {
    v.x = (R)x; v.y = (R)y; v.z = (R)z;
  }
  v.w = (R)q;
  pos4[slot] = v;
  if (frac_out) {
    const RepDev& rp = reps[rep_of ? rep_of[id] : 0];
    double u[3] = {(x - rp.lo_d[0]) / rp.box_d[0], (y - rp.lo_d[1]) / rp.box_d[1],
                   (z - rp.lo_d[2]) / rp.box_d[2]};
    if (sizeof(R) == 4) {
      uint32_t U[3];
      for (int d = 0; d < 3; ++d) {
        U[d] = turn32(u[d] - floor(u[d]));
      }
      reinterpret_cast<Frac32*>(frac_out)[slot] = Frac32{U[0], U[1], U[2], (float)q};
    } else {
      unsigned long long U[3];
      for (int d = 0; d < 3; ++d) {
        U[d] = turn64(u[d] - floor(u[d]));
      }
      reinterpret_cast<Frac64*>(frac_out)[slot] = Frac64{U[0], U[1], U[2], q};
    }
  }
}

// Periodic cell index: v mod d in [0, d).  Stencil rows stay within one period of the box for
// atoms inside or near it, where one compare and add replace the integer division; atoms
// further out take the division.
__device__ __forceinline__ int wrap_cell(int v, int d) {
  if (v >= 0 && v < d) return v;
  if (v < 0 && v >= -d) return v + d;
  if (v >= d && v < 2 * d) return v - d;
  return ((v % d) + d) % d;
}

// 1e-4 threshold of the neighbour predicate: the reference compares a float against the double
// literal 0.0001; for float x, (double)x > 1e-4 <=> x > 1e-4f (1e-4f < 1e-4 < nextafterf(1e-4f)).
__device__ __forceinline__ bool gt_small(float x) { return x > 1.0e-4f; }
__device__ __forceinline__ bool gt_small(double x) { return x > 1.0e-4; }
// cut2 - d2 of a candidate: the list keeps it above 1e-4 (ComputeNeighboursWorklet); the
// "ORIGINAL" neighbour type, which leaves the cutoff to the force function, keeps d2 < cut2
template <class R>
__device__ __forceinline__ bool inside_cut(R margin, int orig) { return orig ? margin > (R)0 : gt_small(margin); }

// Full Verlet list of slot i with the predicate of ComputeNeighboursWorklet
// (rbmd/framework/run/worklet/RunWorklet.cpp:40-96): rc^2 - d^2 > 1e-4 && d^2 > 1e-4 on
// r = (p_j - offset) - p_i with uncontracted float ops and the reference's cell-based periodic
// offsets (PeriodicCoordOffset).  Traversal: for each of the (2nc+1)^2 (y, z) neighbour rows the
// x cells ci-nc .. ci+nc are consecutive cell indices, hence one contiguous slot range when no x
// wrap occurs; rows that wrap in x are walked cell by cell.  The pair set equals the
// reference's 27-cell stencil; the order inside a row differs (sets are order-free).
template <class R>
__device__ __forceinline__ int nlist_range(int s, const int s1, const typename Traits<R>::V4* __restrict__ pos4,
                                           const R* pix, const R* off, int code, R cut2, int idx, int cap,
                                           int stride, int i, int* __restrict__ nbr, int orig) {
#pragma unroll 4
  for (; s < s1; ++s) {
    const typename Traits<R>::V4 pj = pos4[s];
    const R r0 = sub_rn(sub_rn(pj.x, off[0]), pix[0]);
    const R r1 = sub_rn(sub_rn(pj.y, off[1]), pix[1]);
    const R r2 = sub_rn(sub_rn(pj.z, off[2]), pix[2]);
    const R d2 = add_rn(add_rn(mul_rn(r0, r0), mul_rn(r1, r1)), mul_rn(r2, r2));
    if (inside_cut(sub_rn(cut2, d2), orig) && gt_small(d2)) {
      if (idx < cap) __stcs(nbr + nbr_at(idx, i, stride), (s << kShiftBits) | code);
      ++idx;
    }
  }
  return idx;
}

// Per-thread traversal of slot i's 27-cell stencil straight from global memory; returns the
// number of pairs found (entries beyond cap are counted, not stored).
// First slot s in [lo, hi) with pos4[s].x >= bound (the range is ordered by x).
template <class R>
__device__ __forceinline__ int lower_x(const typename Traits<R>::V4* __restrict__ pos4, int lo, int hi, R bound) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (pos4[mid].x < bound) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// trim_x: cells are ordered by x (k_cell_sort_gather with sort_x), so each contiguous x range
// is cut to the candidates with |x_j' - x_i| below the cutoff plus a rounding margin before the
// exact predicate runs; the accepted pairs and their order are unchanged.
template <class R>
__device__ int nlist_thread(int i, const typename Traits<R>::V4 pi, const RepDev& rp,
                            const typename Traits<R>::V4* __restrict__ pos4,
                            const int* __restrict__ cell_start, int num_cycles, R rc, int cap, int stride,
                            int* __restrict__ nbr, bool trim_x = false, int orig = 0) {
  const R pix[3] = {pi.x, pi.y, pi.z};
  const R xm = rc + (fabs(pix[0]) + (R)2 * rc) * (R)1e-5 + (R)1e-6;   // cutoff + margin in x
  int ci[3];
#pragma unroll
  for (int d = 0; d < 3; ++d)
    ci[d] = cell_index<R>(rp, d, pix[d]);
  const R cut2 = mul_rn(rc, rc);
  const int nc = num_cycles;
  const int dx0 = rp.dims[0], dx1 = rp.dims[1], dx2 = rp.dims[2];
  const bool x_contig = ci[0] - nc >= 0 && ci[0] + nc < dx0;
  int idx = 0;
  for (int b = -nc; b <= nc; ++b) {
    const int nby = ci[1] + b;
    const int wy = wrap_cell(nby, dx1), dy = wy - nby;
    for (int c = -nc; c <= nc; ++c) {
      R off[3];
      const int nbz = ci[2] + c;
      const int wz = wrap_cell(nbz, dx2), dz = wz - nbz;
      off[1] = mul_rn(Traits<R>::dx(rp, 1), (R)dy);
      off[2] = mul_rn(Traits<R>::dx(rp, 2), (R)dz);
      const int code_yz = ((dy > 0 ? 1 : (dy < 0 ? 2 : 0)) << 2) | ((dz > 0 ? 1 : (dz < 0 ? 2 : 0)) << 4);
      const int row = rp.cell_base + wy * dx0 + wz * dx0 * dx1;
      if (x_contig) {
        off[0] = (R)0;
        int s0 = cell_start[row + ci[0] - nc], s1 = cell_start[row + ci[0] + nc + 1];
        if (trim_x) {
          s0 = lower_x<R>(pos4, s0, s1, pix[0] - xm);
          s1 = lower_x<R>(pos4, s0, s1, pix[0] + xm);
        }
        idx = nlist_range<R>(s0, s1, pos4, pix, off, code_yz, cut2, idx, cap, stride, i, nbr, orig);
      } else {
        for (int a = -nc; a <= nc; ++a) {
          const int nbx = ci[0] + a;
          const int wx = wrap_cell(nbx, dx0);
          const int ddx = wx - nbx;
          off[0] = mul_rn(Traits<R>::dx(rp, 0), (R)ddx);
          const int code = code_yz | (ddx > 0 ? 1 : (ddx < 0 ? 2 : 0));
          int s0 = cell_start[row + wx], s1 = cell_start[row + wx + 1];
          if (trim_x) {
            const R xw = xm + fabs(off[0]) * (R)1e-5;   // the shifted bound rounds at |x_i + offset|
            s0 = lower_x<R>(pos4, s0, s1, pix[0] + off[0] - xw);
            s1 = lower_x<R>(pos4, s0, s1, pix[0] + off[0] + xw);
          }
          idx = nlist_range<R>(s0, s1, pos4, pix, off, code, cut2, idx, cap, stride, i, nbr, orig);
        }
      }
    }
  }
  return idx;
}

// Count of slot i's row; a last chunk that is not full is filled with the slot itself (distance
// 0, which no pair predicate accepts), so that a pass may evaluate whole chunks.
__device__ __forceinline__ void nlist_finish(int i, int idx, int cap, int stride, int* __restrict__ nbr,
                                             int* __restrict__ count, int* __restrict__ max_count,
                                             uint32_t* status) {
  count[i] = idx;
  for (int p = idx; p < cap && (p & (kNbrChunk - 1)) != 0; ++p) nbr[nbr_at(p, i, stride)] = i << kShiftBits;
  if (idx > cap) {
    set_flag(status, kFlagListOverflow);
    atomicMax(max_count, idx);
  }
}

template <class R>
__global__ void __launch_bounds__(256) k_nlist(
    int n, const typename Traits<R>::V4* __restrict__ pos4, const int* __restrict__ cell_start,
    const RepDev* __restrict__ reps, const int* __restrict__ rep_of_slot, int num_cycles, R rc,
    int cap, int stride, int* __restrict__ nbr, int* __restrict__ count, int* __restrict__ max_count,
    uint32_t* status, const int* __restrict__ rebuild, unsigned long long* __restrict__ nbuilds,
    int trim_x, int n_rep, int orig) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && nbuilds) atomicAdd(nbuilds, rebuilt_replicas(rebuild, n_rep));
  if (i >= n) return;
  const int r = rep_of_slot ? rep_of_slot[i] : 0;
  if (rebuild && !rebuild[r]) return;
  const RepDev& rp = reps[r];
  const int idx = nlist_thread<R>(i, pos4[i], rp, pos4, cell_start, num_cycles, rc, cap, stride, nbr,
                                  trim_x != 0, orig);
  nlist_finish(i, idx, cap, stride, nbr, count, max_count, status);
}

// Warp-per-atom list build for systems with few atoms and many candidates per atom (long
// cutoffs): the 32 lanes test consecutive candidates of a cell range together and a ballot
// compacts the accepted ones in candidate order, so the list equals k_nlist's entry for entry.
template <class R>
__global__ void __launch_bounds__(256) k_nlist_warp(
    int n, const typename Traits<R>::V4* __restrict__ pos4, const int* __restrict__ cell_start,
    const RepDev* __restrict__ reps, const int* __restrict__ rep_of_slot, R rc, int cap, int stride,
    int* __restrict__ nbr, int* __restrict__ count, int* __restrict__ max_count, uint32_t* status,
    const int* __restrict__ rebuild, unsigned long long* __restrict__ nbuilds, int n_rep, int orig) {
  using V4 = typename Traits<R>::V4;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i == 0 && lane == 0 && nbuilds) atomicAdd(nbuilds, rebuilt_replicas(rebuild, n_rep));
  if (i >= n) return;
  const int r = rep_of_slot ? rep_of_slot[i] : 0;
  if (rebuild && !rebuild[r]) return;
  const RepDev& rp = reps[r];
  const V4 pi = pos4[i];
  const R pix[3] = {pi.x, pi.y, pi.z};
  int ci[3];
#pragma unroll
  for (int d = 0; d < 3; ++d)
    ci[d] = cell_index<R>(rp, d, pix[d]);
  const R cut2 = mul_rn(rc, rc);
  const int dx0 = rp.dims[0], dx1 = rp.dims[1], dx2 = rp.dims[2];
  const bool x_contig = ci[0] - 1 >= 0 && ci[0] + 1 < dx0;
  const unsigned below = (1u << lane) - 1u;
  int idx = 0;
  // (no x-window search here: a serial binary search per row costs the warp more latency than
  // the 32-wide candidate test it would save)
  auto scan = [&](int s0, int s1, R o0, R o1, R o2, int code) {
    for (int base = s0; base < s1; base += 32) {
      const int sj = base + lane;
      bool ok = false;
      if (sj < s1) {
        const V4 pj = pos4[sj];
        const R r0 = sub_rn(sub_rn(pj.x, o0), pix[0]);
        const R r1 = sub_rn(sub_rn(pj.y, o1), pix[1]);
        const R r2 = sub_rn(sub_rn(pj.z, o2), pix[2]);
        const R d2 = add_rn(add_rn(mul_rn(r0, r0), mul_rn(r1, r1)), mul_rn(r2, r2));
        ok = inside_cut(sub_rn(cut2, d2), orig) && gt_small(d2);
      }
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        const int at = idx + __popc(m & below);
        if (at < cap) __stcs(nbr + nbr_at(at, i, stride), (sj << kShiftBits) | code);
      }
      idx += __popc(m);
    }
  };
  for (int b = -1; b <= 1; ++b)
    for (int c = -1; c <= 1; ++c) {
      const int nby = ci[1] + b, nbz = ci[2] + c;
      const int wy = wrap_cell(nby, dx1), wz = wrap_cell(nbz, dx2);
      const int dy = wy - nby, dz = wz - nbz;
      const R o1 = mul_rn(Traits<R>::dx(rp, 1), (R)dy), o2 = mul_rn(Traits<R>::dx(rp, 2), (R)dz);
      const int code_yz = ((dy > 0 ? 1 : (dy < 0 ? 2 : 0)) << 2) | ((dz > 0 ? 1 : (dz < 0 ? 2 : 0)) << 4);
      const int row = rp.cell_base + wy * dx0 + wz * dx0 * dx1;
      if (x_contig) {
        scan(cell_start[row + ci[0] - 1], cell_start[row + ci[0] + 2], (R)0, o1, o2, code_yz);
      } else {
        for (int a = -1; a <= 1; ++a) {
          const int nbx = ci[0] + a;
          const int wx = wrap_cell(nbx, dx0);
          const int ddx = wx - nbx;
          scan(cell_start[row + wx], cell_start[row + wx + 1], mul_rn(Traits<R>::dx(rp, 0), (R)ddx), o1, o2,
               code_yz | (ddx > 0 ? 1 : (ddx < 0 ? 2 : 0)));
        }
      }
    }
  if (lane == 0) nlist_finish(i, idx, cap, stride, nbr, count, max_count, status);
}

// ---- cell-cooperative list build ------------------------------------------------------------
// One warp per cell (or per 1/nparts of a cell's atoms): the candidates of the cell's 27-cell
// stencil, flattened in k_nlist's walk order, are held 32 * KC at a time in the registers of the
// lanes, each shifted by its periodic offset once, and every atom of the cell is tested against
// them by a broadcast read of its position: one coalesced load serves all atoms of the cell, no
// lane diverges in the tests, and two candidates share one packed instruction.  A ballot gives
// the accept bits of (atom, 32 candidates); lane k keeps the bits of atom k, and after a batch of
// kCellBatch candidates (a whole stencil at the densities of the benchmarks) every lane takes its
// accepted entries in candidate order, four per 16-byte store, all lanes in step.  Same float operations per pair
// and same order as k_nlist, so the list is identical entry for entry.  d2_max: the predicate
// rc^2 - d^2 > 1e-4 (or > 0) as one comparison of d^2 (pair_d2_max).  one = 1, unknown to the
// compiler: the sums of squares are written as m * one + t, because ptxas contracts a packed
// multiply and add even with explicit .rn (two pairs at the cutoff changed sides), and m * one
// + t rounds as the plain sum.  An atom whose own cell index
// differs from the cell it was binned into (binning clamps positions at the faces) takes
// k_nlist's path on its lane.  Bound by issue (packed tests, ballots and the walk over the bits).
// Measured per build: 200,000 electrolyte atoms at rc 2.5 in FP32 98 us (a shared-memory staged
// build with one thread per atom: 190), 50,021 in FP64 53 us (119); averaged over the steps of a
// run with list reuse 1,000,000 atoms 96 us (k_nlist: 154), 512 replicas 331 us (staged: 719).
// Two cells in turn per warp for such batches, whose steps rebuild about one replica in five, made
// the step 3 % slower.
constexpr int kCellWarps = 4;
constexpr int kCellBatch = 768;   // candidates whose accept bits are kept before entries are written

template <class R> struct __align__(16) CellWarpMem {
  struct __align__(16) XY { Pair<R> x, y; } xy[32];   // the atoms' -x and -y, each twice
  Pair<R> z[32];
  R off[3][27];        // periodic offset of each non-empty stencil cell
  int start[27];       // its first slot
  int code[27];        // its image code
  int pre[27];         // candidates before it
  int ent[kCellBatch];                      // list entry of each candidate of the batch
  unsigned word[kCellBatch / 32][32];       // accept bits [32 candidates][atom], first candidate on top
};

template <class R, int KC>
__global__ void __launch_bounds__(32 * kCellWarps) k_nlist_cell(
    int ncell, int nparts, const typename Traits<R>::V4* __restrict__ pos4, const int* __restrict__ cell_start,
    const RepDev* __restrict__ reps, const int* __restrict__ cell_rep, R rc, R d2_max, R one, int cap, int stride,
    int* __restrict__ nbr, int* __restrict__ count, int* __restrict__ max_count, uint32_t* status,
    const int* __restrict__ rebuild, unsigned long long* __restrict__ nbuilds, int n_rep, int orig) {
  static_assert(KC == 2 || KC == 4, "candidates per lane");
  using V4 = typename Traits<R>::V4;
  constexpr unsigned full = 0xffffffffu;
  __shared__ CellWarpMem<R> mem[kCellWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long item = (long long)blockIdx.x * kCellWarps + w;
  if (item == 0 && lane == 0 && nbuilds) atomicAdd(nbuilds, rebuilt_replicas(rebuild, n_rep));
  const int cell = (int)(item / nparts), part = (int)(item % nparts);
  if (cell >= ncell) return;   // uniform across the warp; the kernel has no block barrier
  const int r = cell_rep ? cell_rep[cell] : 0;
  if (rebuild && !rebuild[r]) return;
  const int s0 = cell_start[cell], ns = cell_start[cell + 1] - s0;
  const int a0 = s0 + (int)((long long)ns * part / nparts), a1 = s0 + (int)((long long)ns * (part + 1) / nparts);
  if (a0 == a1) return;
  CellWarpMem<R>& M = mem[w];
  const RepDev& rp = reps[r];
  const int d0 = rp.dims[0], d1 = rp.dims[1], d2n = rp.dims[2];
  const int cl = cell - rp.cell_base;
  const int cx = cl % d0, cy = (cl / d0) % d1, cz = cl / (d0 * d1);
  // the non-empty stencil cells in walk order: y outermost, then z, then x
  int cnt = 0, st = 0, dx = 0, dy = 0, dz = 0;
  if (lane < 27) {
    const int nbx = cx + lane % 3 - 1, nbz = cz + (lane / 3) % 3 - 1, nby = cy + lane / 9 - 1;
    const int wx = wrap_cell(nbx, d0), wy = wrap_cell(nby, d1), wz = wrap_cell(nbz, d2n);
    dx = wx - nbx;
    dy = wy - nby;
    dz = wz - nbz;
    const int c = rp.cell_base + wx + wy * d0 + wz * d0 * d1;
    st = cell_start[c];
    cnt = cell_start[c + 1] - st;
  }
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(full, incl, 31);
  const unsigned some = __ballot_sync(full, cnt > 0);
  const int nseg = __popc(some);
  if (cnt > 0) {
    const int at = __popc(some & ((1u << lane) - 1u));
    M.off[0][at] = mul_rn(Traits<R>::dx(rp, 0), (R)dx);
    M.off[1][at] = mul_rn(Traits<R>::dx(rp, 1), (R)dy);
    M.off[2][at] = mul_rn(Traits<R>::dx(rp, 2), (R)dz);
    M.start[at] = st;
    M.code[at] = (dx > 0 ? 1 : (dx < 0 ? 2 : 0)) | ((dy > 0 ? 1 : (dy < 0 ? 2 : 0)) << 2) |
                 ((dz > 0 ? 1 : (dz < 0 ? 2 : 0)) << 4);
    M.pre[at] = incl - cnt;
  }
  __syncwarp();
  // lane l holds the first candidate of segment l + 1, the rest never start
  const int next_pre = lane + 1 < nseg ? M.pre[lane + 1] : 1 << 30;
  const R d2_lo = (R)1.0e-4;                 // gt_small
  const Pair<R> unit = both<R>(one);
  int4* out = reinterpret_cast<int4*>(nbr);
  int strays = 0;   // atoms whose own cell is another: after the others
  for (int g0 = a0; g0 < a1; g0 += 32) {
    const int m = min(32, a1 - g0);
    const int i = g0 + min(lane, m - 1);
    const V4 pi = pos4[i];
    const int ci0 = (int)div_rn(sub_rn(pi.x, Traits<R>::lo(rp, 0)), Traits<R>::dx(rp, 0));
    const int ci1 = (int)div_rn(sub_rn(pi.y, Traits<R>::lo(rp, 1)), Traits<R>::dx(rp, 1));
    const int ci2 = (int)div_rn(sub_rn(pi.z, Traits<R>::lo(rp, 2)), Traits<R>::dx(rp, 2));
    const bool valid = lane < m, mine = valid && ci0 == cx && ci1 == cy && ci2 == cz;
    __syncwarp();
    M.xy[lane].x = both<R>(-pi.x);
    M.xy[lane].y = both<R>(-pi.y);
    M.z[lane] = both<R>(-pi.z);
    int idx = 0, have = 0;                     // pairs found; entries of the open chunk in ch
    int ch[4] = {0, 0, 0, 0};
    int4* dst = out + i;
    int row4 = 0;                              // first row of the open chunk
    for (int b0 = 0; b0 < total; b0 += kCellBatch) {
      const int b1 = min(total, b0 + kCellBatch);
      __syncwarp();
      for (int base = b0; base < b1; base += 32 * KC) {
        R px[KC], py[KC], pz[KC];
#pragma unroll
        for (int k = 0; k < KC; ++k) {
          const int q = base + 32 * k + 31 - lane;
          px[k] = (R)INFINITY;                 // past the last candidate: never accepted
          py[k] = pz[k] = (R)0;
          // segments starting at or before q: those before this group of 32, and a mask of the others
          const int q0 = base + 32 * k, rel = next_pre - q0;
          const unsigned starts = __reduce_or_sync(full, rel >= 0 && rel < 32 ? 1u << rel : 0u);
          const int sg = __popc(__ballot_sync(full, rel < 0)) + __popc(starts & (full >> lane));
          if (q < b1) {
            const int s = M.start[sg] + (q - M.pre[sg]);
            const V4 pj = pos4[s];
            px[k] = sub_rn(pj.x, M.off[0][sg]);
            py[k] = sub_rn(pj.y, M.off[1][sg]);
            pz[k] = sub_rn(pj.z, M.off[2][sg]);
            M.ent[q - b0] = (s << kShiftBits) | M.code[sg];
          }
        }
        unsigned word[KC];
#pragma unroll
        for (int k = 0; k < KC; ++k) word[k] = 0;
#pragma unroll 2
        for (int a = 0; a < m; ++a) {
          const typename CellWarpMem<R>::XY o = M.xy[a];
          const Pair<R> oz = M.z[a];
#pragma unroll
          for (int h = 0; h < KC; h += 2) {
            const Pair<R> dx = add2(Pair<R>{px[h], px[h + 1]}, o.x), dy = add2(Pair<R>{py[h], py[h + 1]}, o.y),
                          dz = add2(Pair<R>{pz[h], pz[h + 1]}, oz);
            const Pair<R> dd = fma2(mul2(dz, dz), unit, fma2(mul2(dy, dy), unit, mul2(dx, dx)));
            const unsigned ba = __ballot_sync(full, dd.x > d2_lo && dd.x <= d2_max);
            const unsigned bb = __ballot_sync(full, dd.y > d2_lo && dd.y <= d2_max);
            if (a == lane) {
              word[h] = ba;
              word[h + 1] = bb;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < KC; ++k) M.word[(base - b0) / 32 + k][lane] = word[k];
      }
      __syncwarp();
      if (mine) {
        const int nw = (b1 - b0 + 31) / 32;
        int found = 0;
        for (int k = 0; k < nw; ++k) found += __popc(M.word[k][lane]);
        idx += found;
        int wi = 0;
        unsigned bits = M.word[0][lane];
        auto next = [&]() -> int {             // entry of the next accepted candidate
          while (bits == 0) bits = M.word[++wi][lane];
          const int c = __clz(bits);
          bits ^= 0x80000000u >> c;
          return M.ent[32 * wi + c];
        };
        const int all = have + found;
        for (int t = 0; t < all >> 2; ++t) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k >= have) ch[k] = next();
          have = 0;
          if (row4 < cap) __stcs(dst, make_int4(ch[0], ch[1], ch[2], ch[3]));
          dst += stride;
          row4 += 4;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (k >= have && k < (all & 3)) ch[k] = next();
        have = all & 3;
      }
    }
    if (mine) {   // the last chunk, filled with the slot itself (see nlist_finish)
      if (have > 0 && row4 < cap) {
        const int self = i << kShiftBits;
        __stcs(dst, make_int4(ch[0], have > 1 ? ch[1] : self, have > 2 ? ch[2] : self, self));
      }
      count[i] = idx;
      if (idx > cap) {
        set_flag(status, kFlagListOverflow);
        atomicMax(max_count, idx);
      }
    }
    strays |= __any_sync(full, valid && !mine);
  }
  if (!strays) return;
  for (int i = a0 + lane; i < a1; i += 32) {
    const V4 pi = pos4[i];
    if ((int)div_rn(sub_rn(pi.x, Traits<R>::lo(rp, 0)), Traits<R>::dx(rp, 0)) == cx &&
        (int)div_rn(sub_rn(pi.y, Traits<R>::lo(rp, 1)), Traits<R>::dx(rp, 1)) == cy &&
        (int)div_rn(sub_rn(pi.z, Traits<R>::lo(rp, 2)), Traits<R>::dx(rp, 2)) == cz)
      continue;
    const int idx = nlist_thread<R>(i, pi, rp, pos4, cell_start, 1, rc, cap, stride, nbr, false, orig);
    nlist_finish(i, idx, cap, stride, nbr, count, max_count, status);
  }
}

// Fixed-point fractional coordinates + charge of the charged atoms (qidx: their caller ids,
// grouped per replica), the input of every k-space phase: U_d = floor(frac((x_d - lo_d)/L_d)
// * 2^32) (2^64 for FP64), so integer phases m . U mod 2^32 are exact.  Uncharged atoms add
// nothing to rho_k or the k-space force and are left out.
template <class R> struct FracT;
template <> struct FracT<float> { using T = Frac32; };
template <> struct FracT<double> { using T = Frac64; };

template <class R>
__device__ __forceinline__ typename FracT<R>::T frac_of(const RepDev& rp, const double* __restrict__ pos,
                                                        const double* __restrict__ charge, int id) {
  double u[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    u[d] = (pos[3 * id + d] - rp.lo_d[d]) / rp.box_d[d];
    u[d] -= floor(u[d]);
  }
  const double q = charge[id];
  if constexpr (sizeof(R) == 4) return Frac32{turn32(u[0]), turn32(u[1]), turn32(u[2]), (float)q};
  else return Frac64{turn64(u[0]), turn64(u[1]), turn64(u[2]), q};
}

template <class R>
__global__ void k_frac(int nq, const int* __restrict__ qidx, const double* __restrict__ pos,
                       const double* __restrict__ charge, const int* __restrict__ rep_of,
                       const RepDev* __restrict__ reps, void* __restrict__ frac_out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nq) return;
  const int id = qidx[c];
  reinterpret_cast<typename FracT<R>::T*>(frac_out)[c] = frac_of<R>(reps[rep_of ? rep_of[id] : 0], pos, charge, id);
}

}  // namespace rbmd
