// smac_coarse_cluster.cuh -- the coarse grids of the V-cycle in one thread-block
// cluster, held in distributed shared memory.
//
// Below about 64^3 cells a separately launched sweep is bound by latency, not
// bytes: every grid of the V-cycle's lower half costs its launches' ramp and
// the z-march's dependent steps (about 7 us per sweep at 32^3 and at 16^3
// alike), and the single-CTA kernel for the grids of <= 4096 cells waits on L2
// at every one of its ~50 steps.  This kernel runs the whole lower part of
// the V-cycle -- from the first grid of <= 32768 cells down to the coarsest --
// in one cluster of KCL CTAs:
//   - every grid's cells, right-hand side and face weights live in shared
//     memory, the planes of a grid spread over the ranks in chunks (plane k in
//     rank k / chunk); a rank reads the x of a neighbour's plane through
//     distributed shared memory (the only remote reads) and the restriction
//     writes a coarse right-hand side into the rank that owns it;
//   - the steps of the spread grids are separated by cluster barriers, the
//     steps of the grids of <= KCL_SOLO cells, held whole by rank 0, by
//     __syncthreads in rank 0 while the other ranks wait at the next cluster
//     barrier;
//   - the chunks halve with the grids (a coarse plane is in the rank of its
//     two children), so a rank's residual and its cells' weights are local.
// The operation sequence and every operation are those of the single-CTA
// kernel (k_coarse_vcycle) and of the separately launched sweeps they
// replace (each of those equal to two half-sweeps, bit for bit), so the
// V-cycle's result is the same bit for bit.
#pragma once

#include <cooperative_groups.h>
#include <cuda_pipeline.h>

#include "smac_kernels.cuh"

namespace smac {

constexpr int KCL = 8;           // CTAs in the cluster (the portable maximum)
// threads per CTA: 512, 128 registers a thread (at 1024 the phases' state
// spills at 64 registers)
#ifndef SMAC_KCL_NT32
#define SMAC_KCL_NT32 512
#endif
template <class T> __host__ __device__ constexpr int kcl_threads() { return sizeof(T) == 8 ? 512 : SMAC_KCL_NT32; }
constexpr int KCL_SOLO = 512;    // grids of at most this many cells are held and swept by rank 0
constexpr int KCL_TOP = 32768;   // the set starts at the first grid of at most this many cells
constexpr int MAX_CLL = 12;

// One grid of the set.  Every rank lays out the same arrays at the same
// shared-memory offsets (in elements of T), sized for one chunk of planes:
//   x, rhs  chunk planes of nx*ny cells;
//   bx      chunk planes of ny rows of nx+1 x-faces;
//   by      chunk planes of ny+1 rows of nx y-faces;
//   bz      chunk+1 planes of nx*ny z-faces (also the top face of the last plane).
struct ClusterLevel {
  Geom g;             // the grid's padded layout in global memory
  int cx, cy, cz;     // how this grid was coarsened from the one above
  int chunk;          // planes per rank (nz for a grid held by rank 0)
  int ox, orhs, obx, oby, obz;
  const void* bx;     // weights, stored as T
  const void* by;
  const void* bz;
};
struct ClusterSet {
  ClusterLevel L[MAX_CLL];
  int n;        // grids in the set
  int scratch;  // offset of the residuals of a chunk of cells (-1: no room)
  int nd;       // the first nd are spread over the ranks, the rest held by rank 0
  const void* rhs0;  // right-hand side of L[0] (global, padded layout)
  void* x0;          // its result (global, padded layout; the pads are not written)
};

// A grid of the set as the phases use it, passed by value (registers): its
// dimensions, chunk and shared-memory offsets.
struct ClGrid {
  int nx, ny, nz, chunk, ox, orhs, obx, oby, obz, cx, cy, cz;
};
__device__ __forceinline__ ClGrid cl_grid(const ClusterLevel& L) {
  return ClGrid{L.g.nx, L.g.ny, L.g.nz, L.chunk, L.ox, L.orhs, L.obx, L.oby, L.obz, L.cx, L.cy, L.cz};
}

template <class T>
struct ClusterView {
  T* local;  // this rank's shared memory
  int me;
  // element `off` of rank r's shared memory (a distributed-shared-memory
  // address for another rank)
  __device__ __forceinline__ T* at(int r, int off) const {
    T* p = local + off;
    return r == me ? p : cooperative_groups::this_cluster().map_shared_rank(p, r);
  }
  __device__ __forceinline__ int p0(const ClGrid& L) const { return min(L.nz, me * L.chunk); }
  __device__ __forceinline__ int p1(const ClGrid& L) const { return min(L.nz, (me + 1) * L.chunk); }
  // x of cell (i, j, k) of grid L, in whichever rank holds plane k; 0 outside the grid
  __device__ __forceinline__ T x(const ClGrid& L, int i, int j, int k) const {
    if (i < 0 || j < 0 || k < 0 || i >= L.nx || j >= L.ny || k >= L.nz) return (T)0;
    const int r = k / L.chunk;
    return *at(r, L.ox + ((k - r * L.chunk) * L.ny + j) * L.nx + i);
  }
  __device__ __forceinline__ T* rhsp(const ClGrid& L, int i, int j, int k) const {  // any rank
    const int r = k / L.chunk;
    return at(r, L.orhs + ((k - r * L.chunk) * L.ny + j) * L.nx + i);
  }
};

// Copies planes of rows of rl elements (global row j of plane k at src + base +
// k ps + j px, rpp rows per plane) into dst, row after row.  The warps take a
// plane's rows in turn and the lanes a row's elements, by asynchronous element
// copies (all of a thread's copies in flight; the caller waits).
template <class T>
__device__ __forceinline__ void cl_copy_rows(T* dst, const T* src, int base, int planes, int rl, int rpp, int px,
                                             int ps) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = 0; k < planes; ++k) {
    const T* sp = src + base + k * ps;
    T* d = dst + k * rpp * rl;
#pragma unroll 2
    for (int j = w; j < rpp; j += nw)
      for (int i = lane; i < rl; i += 32) __pipeline_memcpy_async(d + j * rl + i, sp + j * px + i, sizeof(T));
  }
}

// The weights of this rank's planes of grid L, or its right-hand side, into
// shared memory.
template <class T>
__device__ __noinline__ void cl_stage(ClusterView<T> V, const ClusterLevel& Lp) {
  const ClGrid L = cl_grid(Lp);
  const Geom& g = Lp.g;
  const int k0 = V.p0(L), np = V.p1(L) - k0;
  if (np <= 0) return;
  const int b = g.idx(0, 0, k0);
  cl_copy_rows<T>(V.local + L.obx, (const T*)Lp.bx, b, np, L.nx + 1, L.ny, g.px, g.ps);
  cl_copy_rows<T>(V.local + L.oby, (const T*)Lp.by, b, np, L.nx, L.ny + 1, g.px, g.ps);
  cl_copy_rows<T>(V.local + L.obz, (const T*)Lp.bz, b, np + 1, L.nx, L.ny, g.px, g.ps);  // z-faces k0..k0+np
}
template <class T>
__device__ __forceinline__ void cl_stage_rhs(ClusterView<T> V, const ClusterLevel& Lp, const T* rhs0) {
  const ClGrid L = cl_grid(Lp);
  const Geom& g = Lp.g;
  const int k0 = V.p0(L), np = V.p1(L) - k0;
  if (np <= 0) return;
  cl_copy_rows<T>(V.local + L.orhs, rhs0, g.idx(0, 0, k0), np, L.nx, L.ny, g.px, g.ps);
}

// The six neighbours (x-, x+, y-, y+, z-, z+) of the own cell (i, j, k) of
// grid L at local offset c (plane kk of the rank's np planes); 0 outside the
// grid.  Only the planes below the first and above the last own plane come
// from another rank: the last plane of rank me-1 and the first of rank me+1
// (every spread grid has the same chunk in every rank; a grid of rank 0 has
// all its planes).
template <class T>
__device__ __forceinline__ void cl_nb(const ClusterView<T>& V, const ClGrid& L, int i, int j, int k, int kk, int np,
                                      int c, T (&n)[6]) {
  const int nx = L.nx, ny = L.ny, pl = nx * ny;
  const T* x = V.local + L.ox;
  n[0] = i > 0 ? x[c - 1] : (T)0;
  n[1] = i + 1 < nx ? x[c + 1] : (T)0;
  n[2] = j > 0 ? x[c - nx] : (T)0;
  n[3] = j + 1 < ny ? x[c + nx] : (T)0;
  n[4] = (T)0;
  if (k > 0) n[4] = kk > 0 ? x[c - pl] : *V.at(V.me - 1, L.ox + (L.chunk - 1) * pl + j * nx + i);
  n[5] = (T)0;
  if (k + 1 < L.nz) n[5] = kk + 1 < np ? x[c + pl] : *V.at(V.me + 1, L.ox + j * nx + i);
}

template <class T>
__device__ __forceinline__ void cl_weights(const ClusterView<T>& V, const ClGrid& L, int i, int j, int kk, int c,
                                           T& wxm, T& wxp, T& wym, T& wyp, T& wzm, T& wzp) {
  const int nx = L.nx, ny = L.ny;
  const T* bx = V.local + L.obx + (kk * ny + j) * (nx + 1) + i;
  const T* by = V.local + L.oby + (kk * (ny + 1) + j) * nx + i;
  const T* bz = V.local + L.obz + c;
  wxm = bx[0];
  wxp = bx[1];
  wym = by[0];
  wyp = by[nx];
  wzm = bz[0];
  wzp = bz[nx * ny];
}

// A thread's items t, t + blockDim, ... of the (pair, row, plane) box of this
// rank's planes: the first one's coordinates and the steps to the next, found
// once per grid (they take six integer divisions).
struct ClItems {
  int total, tx, j, kk, sx, sj, sk;
};
template <class T>
__device__ __forceinline__ ClItems cl_items(const ClusterView<T>& V, const ClGrid& L) {
  const int half = (L.nx + 1) / 2, t = threadIdx.x, s = blockDim.x;
  return ClItems{half * L.ny * max(0, V.p1(L) - V.p0(L)), t % half, (t / half) % L.ny, t / (half * L.ny),
                 s % half, (s / half) % L.ny, s / (half * L.ny)};
}

// Half-sweep of colour `colour` over this rank's planes of grid L: the
// operations of cta_half_sweep.  The items' coordinates advance by carries.
template <class T>
__device__ __noinline__ void cl_half_sweep(ClusterView<T> V, ClGrid L, ClItems I, int colour, bool zero_init) {
  typedef acc_t<T> A;
  const int nx = L.nx, ny = L.ny, k0 = V.p0(L), np = V.p1(L) - k0;
  const int half = (nx + 1) / 2;
  int tx = I.tx, j = I.j, kk = I.kk;
  for (int t = threadIdx.x; t < I.total; t += blockDim.x) {
    const int k = k0 + kk;
    const int i = 2 * tx + ((2 * tx + j + k + colour) & 1);
    if (i < nx) {
      const int c = (kk * ny + j) * nx + i;
      T wxm, wxp, wym, wyp, wzm, wzp, n[6] = {(T)0, (T)0, (T)0, (T)0, (T)0, (T)0};
      cl_weights(V, L, i, j, kk, c, wxm, wxp, wym, wyp, wzm, wzp);
      const A bv = (A)V.local[L.orhs + c];  // (no mean shift below the finest grid)
      if (!zero_init) cl_nb(V, L, i, j, k, kk, np, c, n);
      V.local[L.ox + c] = (T)Stencil<T, T>::gs(bv, (A)wxm, (A)wxp, (A)wym, (A)wyp, (A)wzm, (A)wzp, (A)n[0], (A)n[1],
                                               (A)n[2], (A)n[3], (A)n[4], (A)n[5]);
    }
    tx += I.sx;
    int cy = tx >= half;
    tx -= cy ? half : 0;
    j += I.sj + cy;
    cy = j >= ny;
    j -= cy ? ny : 0;
    kk += I.sk + cy;
  }
}

// x += P xc on every own cell: the prolongation of Lc's x, ahead of the first
// post-smoothing sweep (whose first half-sweep reads the sum at the
// neighbours, and overwrites the rest).  A coarse plane of a spread grid is in
// the rank of its children, a grid of rank 0 is read from there.
template <class T>
__device__ __noinline__ void cl_prolong(ClusterView<T> V, ClGrid L, ClGrid Lc, bool lc_spread) {
  typedef acc_t<T> A;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int k0 = V.p0(L), np = V.p1(L) - k0, K0 = lc_spread ? V.p0(Lc) : 0;
  const T* xc = V.at(lc_spread ? V.me : 0, Lc.ox);
  for (int kk = 0; kk < np; ++kk) {
    const T* pc = xc + ((Lc.cz ? (k0 + kk) >> 1 : k0 + kk) - K0) * Lc.ny * Lc.nx;
    for (int j = w; j < L.ny; j += nw) {
      const T* row = pc + (Lc.cy ? j >> 1 : j) * Lc.nx;
      T* x = V.local + L.ox + (kk * L.ny + j) * L.nx;
      for (int i = lane; i < L.nx; i += 32) x[i] = (T)Ar<A>::add((A)x[i], (A)row[Lc.cx ? i >> 1 : i]);
    }
  }
}

// Residual of fine cell (i, j, k) (plane kk of the rank's np) added to acc:
// the operations of cta_resid_restrict.
template <class T>
__device__ __forceinline__ void cl_resid_add(const ClusterView<T>& V, const ClGrid& L, int i, int j, int k, int kk,
                                             int np, acc_t<T>& acc) {
  typedef acc_t<T> A;
  const int c = (kk * L.ny + j) * L.nx + i;
  T wxm, wxp, wym, wyp, wzm, wzp, xn[6];
  cl_weights(V, L, i, j, kk, c, wxm, wxp, wym, wyp, wzm, wzp);
  cl_nb(V, L, i, j, k, kk, np, c, xn);
  const A bv = (A)V.local[L.orhs + c];  // (no mean shift below the finest grid)
  const A ax = Stencil<T, T>::apply((A)V.local[L.ox + c], (A)wxm, (A)wxp, (A)wym, (A)wyp, (A)wzm, (A)wzp, (A)xn[0],
                                    (A)xn[1], (A)xn[2], (A)xn[3], (A)xn[4], (A)xn[5]);
  acc = Ar<A>::add(acc, Ar<A>::add(bv, -ax));
}

// Residual of grid L restricted to grid Lc (the operations of
// cta_resid_restrict): each rank takes the coarse cells whose children lie in
// its planes and writes them into the rank that holds their plane.
template <class T>
__device__ __noinline__ void cl_resid_restrict(ClusterView<T> V, ClGrid L, ClGrid Lc) {
  typedef acc_t<T> A;
  const int rx = Lc.cx ? 2 : 1, ry = Lc.cy ? 2 : 1, rz = Lc.cz ? 2 : 1;
  // coarse planes whose first child plane is in [k0, k1)
  const int k0 = V.p0(L), k1 = V.p1(L), np = k1 - k0;
  const int K0 = (k0 + rz - 1) / rz, K1 = min(Lc.nz, (k1 + rz - 1) / rz);
  const int total = Lc.nx * Lc.ny * max(0, K1 - K0);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int I = t % Lc.nx, J = (t / Lc.nx) % Lc.ny, K = K0 + t / (Lc.nx * Lc.ny);
    A acc = (A)0;
    for (int dk = 0; dk < rz; ++dk)
      for (int dj = 0; dj < ry; ++dj)
        for (int di = 0; di < rx; ++di) {
          const int i = (Lc.cx ? 2 * I : I) + di, j = (Lc.cy ? 2 * J : J) + dj, k = (Lc.cz ? 2 * K : K) + dk;
          if (i >= L.nx || j >= L.ny || k >= L.nz) continue;  // no such child (odd extent)
          cl_resid_add(V, L, i, j, k, k - k0, np, acc);
        }
    *V.rhsp(Lc, I, J, K) = (T)Ar<A>::div(acc, (A)(rx * ry * rz));
  }
}

// The same in two passes where the shared memory has room for the residuals of
// a chunk (at `scratch`): every own cell's residual, row by row without bank
// conflicts, then the children's sums.
template <class T>
__device__ __noinline__ void cl_resid_restrict2(ClusterView<T> V, ClGrid L, ClGrid Lc, int scratch) {
  typedef acc_t<T> A;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nx = L.nx, ny = L.ny, k0 = V.p0(L), k1 = V.p1(L), np = k1 - k0;
  T* res = V.local + scratch;
  for (int kk = 0; kk < np; ++kk)
    for (int j = w; j < ny; j += nw)
      for (int i = lane; i < nx; i += 32) {
        A r = (A)0;
        cl_resid_add(V, L, i, j, k0 + kk, kk, np, r);
        res[(kk * ny + j) * nx + i] = (T)r;
      }
  __syncthreads();
  const int rx = Lc.cx ? 2 : 1, ry = Lc.cy ? 2 : 1, rz = Lc.cz ? 2 : 1;
  const int K0 = (k0 + rz - 1) / rz, K1 = min(Lc.nz, (k1 + rz - 1) / rz);
  for (int K = K0; K < K1; ++K)
    for (int J = w; J < Lc.ny; J += nw)
      for (int I = lane; I < Lc.nx; I += 32) {
        A acc = (A)0;
        for (int dk = 0; dk < rz; ++dk)
          for (int dj = 0; dj < ry; ++dj)
            for (int di = 0; di < rx; ++di) {
              const int i = (Lc.cx ? 2 * I : I) + di, j = (Lc.cy ? 2 * J : J) + dj, k = (Lc.cz ? 2 * K : K) + dk;
              if (i >= nx || j >= ny || k >= L.nz) continue;  // no such child (odd extent)
              acc = Ar<A>::add(acc, (A)res[((k - k0) * ny + j) * nx + i]);
            }
        *V.rhsp(Lc, I, J, K) = (T)Ar<A>::div(acc, (A)(rx * ry * rz));
      }
}

// nhalf half-sweeps of a grid held whole by rank 0 (nx*ny*nz <= KCL_SOLO <=
// blockDim.x): thread t keeps cell t's weights, rhs and reciprocal diagonal in
// registers across the half-sweeps, which read the neighbours' x from shared
// memory and end at a barrier of the warps that own cells (the others wait at
// the one after the last).  Half-sweep h has colour c0 ^ (h & 1) before
// swap_at and (1 - c0) ^ ((h - swap_at) & 1) from there (the coarsest grid's
// backward pairs); the first may start from zero (zero_first).  The operations
// are those of cl_half_sweep.  Called by every thread of rank 0.
template <class T>
__device__ __noinline__ void cl_solo_run(ClusterView<T> V, ClGrid L, int nhalf, int c0, int swap_at, bool zero_first) {
  typedef acc_t<T> A;
  const int nx = L.nx, ny = L.ny, nz = L.nz, pl = nx * ny, cells = pl * nz;
  const int t = threadIdx.x, nthreads = (cells + 31) & ~31;
  if (t < nthreads) {
    const bool own = t < cells;
    const int c = own ? t : 0;
    const int k = c / pl, j = (c - k * pl) / nx, i = c - k * pl - j * nx;
    T wxm, wxp, wym, wyp, wzm, wzp;
    cl_weights(V, L, i, j, k, c, wxm, wxp, wym, wyp, wzm, wzp);
    const A bv = (A)V.local[L.orhs + c];  // (no mean shift below the finest grid)
    const A d = Stencil<T, T>::diag((A)wxm, (A)wxp, (A)wym, (A)wyp, (A)wzm, (A)wzp);
    const A rd = d > (A)0 ? Ar<A>::rcp(d) : (A)0;
    T* x = V.local + L.ox + c;
    for (int h = 0; h < nhalf; ++h) {
      const int colour = h < swap_at ? (c0 ^ (h & 1)) : ((1 - c0) ^ ((h - swap_at) & 1));
      if (own && ((i + j + k + colour) & 1) == 0) {
        A n[6] = {(A)0, (A)0, (A)0, (A)0, (A)0, (A)0};
        if (!(h == 0 && zero_first)) {
          if (i > 0) n[0] = (A)x[-1];
          if (i + 1 < nx) n[1] = (A)x[1];
          if (j > 0) n[2] = (A)x[-nx];
          if (j + 1 < ny) n[3] = (A)x[nx];
          if (k > 0) n[4] = (A)x[-pl];
          if (k + 1 < nz) n[5] = (A)x[pl];
        }
        const A v = Stencil<T, T>::offsum(bv, (A)wxm, (A)wxp, (A)wym, (A)wyp, (A)wzm, (A)wzp, n[0], n[1], n[2], n[3],
                                          n[4], n[5]);
        *x = d > (A)0 ? (T)Ar<A>::mul(v, rd) : (T)0;
      }
      if (nthreads <= 32) __syncwarp();
      else asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
    }
  }
  __syncthreads();
}

// The lower part of the V-cycle: pre-smoothing (nu1 sweeps from zero) and
// restriction down the set, coarse_pairs symmetric sweep pairs on the
// coarsest grid, prolongation and post-smoothing (nu2 sweeps) back up; the
// sequence of k_coarse_vcycle.  The set's first grid is not the finest
// (no mean shift is applied).
template <class T>
__global__ void __cluster_dims__(KCL, 1, 1) __launch_bounds__(kcl_threads<T>())
    k_coarse_cluster(const __grid_constant__ ClusterSet set, int nu1, int nu2, int coarse_pairs, const Scalars* s) {
  static_assert(KCL_SOLO <= kcl_threads<T>(), "a rank-0 grid needs a thread per cell");
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char cl_smem[];
  cg::cluster_group cl = cg::this_cluster();
  ClusterView<T> V;
  V.me = (int)cl.block_rank();
  V.local = reinterpret_cast<T*>(cl_smem);
  const int n = set.n, nd = set.nd;
  // The weights, which no kernel of the solve writes, are staged while the
  // previous kernel drains; the first grid's rhs, its output, after the wait.
  for (int q = 0; q < n; ++q) cl_stage<T>(V, set.L[q]);
  pdl_enter();
  if (s && s->done) {  // the same flag for every rank: all return, or none
    __pipeline_commit();
    __pipeline_wait_prior(0);  // no copy into this CTA's shared memory outlives it
    return;
  }
  cl_stage_rhs<T>(V, set.L[0], (const T*)set.rhs0);
  __pipeline_commit();
  __pipeline_wait_prior(0);
  cl.sync();
  auto restrict_to = [&](const ClGrid& L, int q) {  // grid q's residual to grid q + 1
    const ClGrid C = cl_grid(set.L[q + 1]);
    if (set.scratch >= 0) cl_resid_restrict2<T>(V, L, C, set.scratch);
    else cl_resid_restrict<T>(V, L, C);
  };
  // down the spread grids
  for (int q = 0; q < nd; ++q) {
    const ClGrid L = cl_grid(set.L[q]);
    const ClItems I = cl_items<T>(V, L);
    for (int h = 0; h < 2 * nu1; ++h) {
      cl_half_sweep<T>(V, L, I, h & 1, h == 0);
      cl.sync();
    }
    restrict_to(L, q);
    cl.sync();
  }
  // the grids of rank 0: down, the coarsest, up
  if (V.me == 0) {
    for (int q = nd; q < n - 1; ++q) {
      const ClGrid L = cl_grid(set.L[q]);
      cl_solo_run<T>(V, L, 2 * nu1, 0, 2 * nu1, true);
      restrict_to(L, q);
      __syncthreads();
    }
    cl_solo_run<T>(V, cl_grid(set.L[n - 1]), 4 * coarse_pairs, 0, 2 * coarse_pairs, true);
    for (int q = n - 2; q >= nd; --q) {
      const ClGrid L = cl_grid(set.L[q]);
      cl_prolong<T>(V, L, cl_grid(set.L[q + 1]), false);
      __syncthreads();
      cl_solo_run<T>(V, L, 2 * nu2, 1, 2 * nu2, false);
    }
  }
  cl.sync();
  // up the spread grids
  for (int q = nd - 1; q >= 0; --q) {
    const ClGrid L = cl_grid(set.L[q]);
    const ClItems I = cl_items<T>(V, L);
    if (q + 1 < n) {
      cl_prolong<T>(V, L, cl_grid(set.L[q + 1]), q + 1 < nd);
      cl.sync();
    }
    for (int h = 0; h < 2 * nu2; ++h) {
      cl_half_sweep<T>(V, L, I, (h & 1) ^ 1, false);
      cl.sync();
    }
  }
  // the first grid's x back to global memory (own planes; after the last
  // barrier no rank reads another's shared memory)
  {
    const ClusterLevel& Lp = set.L[0];
    const ClGrid L = cl_grid(Lp);
    const Geom& g = Lp.g;
    const int k0 = V.p0(L), np = V.p1(L) - k0;
    T* x0 = reinterpret_cast<T*>(set.x0);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int r = w; r < max(0, np) * L.ny; r += nw) {
      const int j = r % L.ny, k = k0 + r / L.ny;
      const T* src = V.local + L.ox + r * L.nx;
      T* dst = x0 + g.idx(0, j, k);
      for (int i = lane; i < L.nx; i += 32) dst[i] = src[i];
    }
  }
}

}  // namespace smac
