// Cell lists and per-particle neighbour lists for large particle counts.
//
// The reference finds LJ pairs with a head/linked-list cell list of
// 16-grid-unit cells and a 27-cell scan (md_force.cxx:23-134).  Here the
// same idea serves every pair search of the step at once: after the
// position update the particles are binned into cells at least as wide as
// the longest pair range in use (the LJ cutoff, the overlap of two profile
// supports 2(RADIUS+HXI), and the near-contact range when a correction
// network is attached), and each particle gets the list of the particles
// within that range, in increasing index order.  The LJ force, the
// deterministic phi/up scatter and the near-contact pair search then read
// the lists instead of scanning all particles.  The LJ force keeps the
// reference's pair multiplicity of its own 16-unit cells (the kernel
// computes it per pair), so results do not depend on the cells used here.
//
// Five launches: count, scan, fill, sort (each cell's members by index, so
// the lists do not depend on atomic ordering) and the neighbour lists.
#pragma once

#include <cuda_runtime.h>

#include "particle_kernels.cuh"

namespace kapsel {

struct CellPar {
  int lc[3];         // cells per axis
  double inv_cl[3];  // 1 / cell length
  int ncell;
  double r2list;     // squared neighbour range
};

__device__ __forceinline__ void cell_coords(const double *x, const CellPar &c, int ci[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int k = (int)(x[d] * c.inv_cl[d]);
    ci[d] = k < 0 ? 0 : (k >= c.lc[d] ? c.lc[d] - 1 : k);
  }
}

__global__ void k_cell_count(PPar p, CellPar c, const DPart *__restrict__ parts, int *__restrict__ cellof,
                             int *__restrict__ count) {
  pdl_begin();
  parts = pdl_fresh(parts);
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= p.Np) return;
  int ci[3];
  cell_coords(parts[n].x, c, ci);
  const int cell = (ci[0] * c.lc[1] + ci[1]) * c.lc[2] + ci[2];
  cellof[n] = cell;
  atomicAdd(count + cell, 1);
}

// Exclusive scan of the per-cell counts (one block of 1024 threads): start
// and cursor, and the counts cleared for the next build.  One round of the
// block takes eight neighbouring cells a thread, since a round's barriers and
// loads are what it costs (9000 cells, one a thread: 14.5 us).
constexpr int SCAN_CELLS = 8;
__global__ void __launch_bounds__(1024) k_cell_scan(CellPar c, int *__restrict__ count, int *__restrict__ start,
                                                    int *__restrict__ cursor) {
  __shared__ int wsum[32];
  pdl_begin();
  count = pdl_fresh(count);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry = 0;  // counts before this pass of the loop, the same in every thread
  for (int base = 0; base < c.ncell; base += SCAN_CELLS * blockDim.x) {
    const int i0 = base + SCAN_CELLS * threadIdx.x;
    int v[SCAN_CELLS], sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_CELLS; ++k) v[k] = i0 + k < c.ncell ? count[i0 + k] : 0;
#pragma unroll
    for (int k = 0; k < SCAN_CELLS; ++k) sum += v[k];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    const int warps_before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    int ex = carry + (warp > 0 ? warps_before : 0) + incl - sum;
#pragma unroll
    for (int k = 0; k < SCAN_CELLS; ++k)
      if (i0 + k < c.ncell) {
        start[i0 + k] = ex;
        cursor[i0 + k] = ex;
        count[i0 + k] = 0;
        ex += v[k];
      }
    carry += __shfl_sync(0xffffffffu, w, 31);
    __syncthreads();  // wsum is written again
  }
  if (threadIdx.x == 0) start[c.ncell] = carry;
}

__global__ void k_cell_fill(PPar p, const int *__restrict__ cellof, int *__restrict__ cursor, int *__restrict__ list) {
  pdl_begin();
  cellof = pdl_fresh(cellof);
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= p.Np) return;
  list[atomicAdd(cursor + cellof[n], 1)] = n;
}

// Members of each cell in increasing particle index (a cell holds a few).
__global__ void k_cell_sort(CellPar c, const int *__restrict__ start, int *__restrict__ list) {
  pdl_begin();
  start = pdl_fresh(start);
  list = pdl_fresh(list);
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= c.ncell) return;
  const int b = start[cell], e = start[cell + 1];
  for (int i = b + 1; i < e; ++i) {
    const int v = list[i];
    int k = i - 1;
    while (k >= b && list[k] > v) {
      list[k + 1] = list[k];
      --k;
    }
    list[k + 1] = v;
  }
}

// Neighbour list of each particle: count, then up to NBL_MAX indices in
// increasing order, of the particles within the list range (minimum image).
// More neighbours than NBL_MAX: KAPSEL_ERANGE in the status word.  One warp
// per particle: the lanes read the bounds of the (up to 27) neighbouring cells
// together, share the members of all of them out among themselves, append the
// hits (ballot), then each lane places its entries by rank.  The chain of
// dependent loads is what it costs, and cell after cell it was 27 times as long
// (8600 particles at 256^3, the five launches with the position update, timed
// alone: 82 -> 54 us; the step, with the launches chained, 1154 -> 1131).
constexpr int NBL_WARPS = 4;  // particles per block
__global__ void __launch_bounds__(NBL_WARPS * 32) k_neighbor_lists(PPar p, CellPar c, const DPart *__restrict__ parts,
                                                                   const int *__restrict__ start,
                                                                   const int *__restrict__ list, int *__restrict__ nbl,
                                                                   int *__restrict__ status) {
  __shared__ int cand[NBL_WARPS][NBL_MAX];
  pdl_begin();
  parts = pdl_fresh(parts);
  start = pdl_fresh(start);
  list = pdl_fresh(list);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * NBL_WARPS + warp;
  if (n >= p.Np) return;  // a whole warp: no later block-wide barrier
  int *cw = cand[warp];
  const double xn[3] = {parts[n].x[0], parts[n].x[1], parts[n].x[2]};
  int ci[3];
  cell_coords(xn, c, ci);
  // lane q < 27: cell (ox, oy, oz); each distinct neighbouring cell once
  // (fewer than 3 cells on an axis)
  int first = 0, len = 0;
  if (lane < 27) {
    const int o[3] = {lane / 9 - 1, lane / 3 % 3 - 1, lane % 3 - 1};
    int cc[3];
    bool use = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if ((c.lc[d] == 1 && o[d] != 0) || (c.lc[d] == 2 && o[d] == -1)) use = false;
      cc[d] = (ci[d] + o[d] + c.lc[d]) % c.lc[d];
    }
    if (use) {
      const int cell = (cc[0] * c.lc[1] + cc[1]) * c.lc[2] + cc[2];
      first = start[cell];
      len = start[cell + 1] - first;
    }
  }
  int incl = len;  // members of the cells up to this lane's
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const int base = first - (incl - len), total = __shfl_sync(0xffffffffu, incl, 31);
  int cnt = 0;
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int t = t0 + lane;
    int q = 0;  // cells that end at or before member t
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
      if (__shfl_sync(0xffffffffu, incl, q + s - 1) <= t) q += s;
    const int at = __shfl_sync(0xffffffffu, base, q) + t;
    int j = -1;
    bool hit = false;
    if (t < total) {
      j = list[at];
      if (j != n) {
        double s = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double dd = parts[j].x[d] - xn[d];
          dd -= nint_d(dd * p.invL[d]) * p.L[d];
          s += dd * dd;
        }
        hit = s < c.r2list;
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
    if (hit && pos < NBL_MAX) cw[pos] = j;
    cnt += __popc(bal);
  }
  __syncwarp();
  if (cnt > NBL_MAX) {
    if (lane == 0) atomicExch(status, -6);
    cnt = NBL_MAX;
  }
  // increasing index order: each entry's rank among the distinct indices
  int *out = nbl + (size_t)n * (NBL_MAX + 1);
  for (int q = lane; q < cnt; q += 32) {
    const int v = cw[q];
    int r = 0;
    for (int t = 0; t < cnt; ++t) r += cw[t] < v;
    out[1 + r] = v;
  }
  if (lane == 0) out[0] = cnt;
}

}  // namespace kapsel
