// shl_contact.cu -- linked-cell self-contact candidate list on the device.
//
// compute_shell_shell_contact_candidates (ShellSystem.C:1910-2135) with
// compute_bounding_box (2544-2587), as a pipeline of kernels that all return
// immediately unless the device flag ctl->rebuild is set (so the pipeline can
// be captured into a CUDA graph and skipped on device):
//
//   k_rb_aabb      per-face AABBs and sizes, per-block bounds
//   k_rb_bounds    shell bounds, avg_elem_size (fixed-order sum), cell size,
//                  d_max, cell counts; TOO_MANY_CELLS check (k_rb_grids and
//                  k_rb_grid_scan per shell for a batch)
//   k_rb_clear     clear the cell histogram and the per-face counters
//   k_rb_count     cell ranges per face, cell histogram (counting sort, pass 1);
//                  keep flags of the old list (ShellSystem.C:2016-2027)
//   scan           cell_count -> cell_start
//   k_rb_fill      scatter faces into their cells (counting sort, pass 2)
//   k_rb_cand      per (cell, face e1) entry: faces e2 > e1 in the cell, emitted
//                  from the lowest shared cell only, not topologically close, not
//                  in the kept list, not AABB-apart by d_max, not certainly apart
//                  along the line of centroids (a conservative prefilter)
//   k_rb_narrow    per candidate: closest points, accept d2 <= d2_max (SMOOTH:
//                  k_limit_coeffs and k_smooth_search)
//   scan, k_rb_scatter_new  accepted pairs grouped by eid1 (counting sort)
//   scan           per-face pair counts -> segment offsets
//   k_rb_assemble  kept old pairs + new pairs of each face, merged in e2 order
//   k_rb_copyback  scratch list -> list; its last block ends the pass
//   k_csr_*, scan  each node's (pair, role) entries, sorted
//
// The resulting list equals, as a set, the reference's list at the same state
// (the reference's cell-membership test is reproduced with the same rounded
// operations); it is stored sorted by (eid1, eid2), which fixes the order the
// per-node gather adds contact forces in.  The reference's slot order depends
// on OpenMP scheduling and is not reproduced.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "shl_cells.h"
#include "shl_geom.h"
#include "shl_internal.cuh"
#include "shl_pairs.cuh"

namespace shl {

namespace {

__device__ __forceinline__ bool rb_off(const Ctl* ctl) { return ctl->rebuild == 0 || ctl->halted != 0; }

__device__ __forceinline__ bool last_block_rb(uint32_t* counter) {
  __shared__ bool is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t t = atomicAdd(counter, 1u);
    is_last = (t == gridDim.x - 1);
    if (is_last) *counter = 0;
  }
  __syncthreads();
  return is_last;
}

__device__ __forceinline__ void set_error(Ctl* ctl, int code) {
  atomicMax(&ctl->error, code);
  ctl->rebuild = 0;
}

// The cell grid that face f is binned in: the control block's for a single
// shell, its shell's for a batch with self-contact (ShellCell).
struct GridView {
  double cell_size, d_max, d2_max;
  const double* bmin;
  uint32_t ny, nz, base;
};
__device__ __forceinline__ GridView grid_of(const DevBuf& b, const StepConst& sc, uint32_t f) {
  GridView g;
  if (sc.n_cs) {
    const ShellCell& s = b.shc[b.face_shell[f]];
    g.cell_size = s.cell_size; g.d_max = s.d_max; g.d2_max = s.d2_max; g.bmin = s.bmin;
    g.ny = s.ncd[1]; g.nz = s.ncd[2]; g.base = s.cell_base;
  } else {
    const Ctl* ctl = b.ctl;
    g.cell_size = ctl->cell_size; g.d_max = ctl->d_max; g.d2_max = ctl->d2_max; g.bmin = ctl->bmin;
    g.ny = ctl->ncd[1]; g.nz = ctl->ncd[2]; g.base = 0;
  }
  return g;
}

// face f takes part in the current pass (a batch rebuilds only the shells whose trigger fired)
__device__ __forceinline__ bool face_in_pass(const DevBuf& b, const StepConst& sc, uint32_t f) {
  return sc.n_cs == 0 || b.shc[b.face_shell[f]].rebuild != 0;
}

// Cell size, d_max and cell counts of a shell from its bounds and average
// element size (ShellSystem.C:1929-1969), rounded operation by operation.
// Returns the number of cells (0 with TOO_MANY_CELLS registered).
__device__ uint64_t grid_setup(const double* bmin, const double* bmax, double avg, double cell_size_mult,
                               double cell_margin, double thickness, int smooth, double* cell_size_out,
                               double* d_max_out, uint32_t* ncd) {
  double cell_size = __dmul_rn(cell_size_mult, avg);
  const double tolerance = __dmul_rn(cell_margin, cell_size);
  cell_size = __dadd_rn(cell_size, tolerance);
  double d_max = __dadd_rn(thickness, tolerance);
  // SMOOTH: the limit surfaces may be closer than the facets (ShellSystem.C:1940-1944)
  if (smooth) d_max = __dadd_rn(d_max, avg);
  *cell_size_out = cell_size;
  *d_max_out = d_max;
  uint64_t n_cells = 1;
  for (int c = 0; c < 3; ++c) {
    const double sz = __dsub_rn(bmax[c], bmin[c]);
    const double q = __dadd_rn(__ddiv_rn(__dadd_rn(sz, d_max), cell_size), 1.0);
    const int ncd_c = (q < 2147483647.0) ? (int)q : 2147483647;
    ncd[c] = (uint32_t)ncd_c;
    n_cells *= (uint64_t)(uint32_t)ncd_c;
  }
  return n_cells;
}

// ------------------------------------------------------------------ AABB --
__global__ void __launch_bounds__(kBlock) k_rb_aabb(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  __shared__ double sh_min[3][kBlock], sh_max[3][kBlock];
  const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
  double lo[3] = {SHL_DBL_MAX, SHL_DBL_MAX, SHL_DBL_MAX}, hi[3] = {-SHL_DBL_MAX, -SHL_DBL_MAX, -SHL_DBL_MAX};
  // a batch: only the shells of this pass (nothing else reads a face's box)
  if (f < sc.F && face_in_pass(b, sc, f)) {
    for (int k = 0; k < 3; ++k) {
      const double* q = b.p + 3 * (size_t)b.tri[3 * (size_t)f + k];
      for (int c = 0; c < 3; ++c) {
        if (q[c] < lo[c]) lo[c] = q[c];
        if (q[c] > hi[c]) hi[c] = q[c];
      }
    }
    for (int c = 0; c < 3; ++c) {
      b.bmin[3 * (size_t)f + c] = lo[c];
      b.bmax[3 * (size_t)f + c] = hi[c];
    }
    // BoundingBox::max_size
    double dmax = __dsub_rn(hi[0], lo[0]);
    const double d1 = __dsub_rn(hi[1], lo[1]), d2 = __dsub_rn(hi[2], lo[2]);
    if (d1 > dmax) dmax = d1;
    if (d2 > dmax) dmax = d2;
    b.fsize[f] = dmax;
  }
  if (sc.n_cs) return;  // a batch: per-shell grids (k_rb_grids)
  for (int c = 0; c < 3; ++c) {
    sh_min[c][threadIdx.x] = lo[c];
    sh_max[c][threadIdx.x] = hi[c];
  }
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st)
      for (int c = 0; c < 3; ++c) {
        sh_min[c][threadIdx.x] = fmin(sh_min[c][threadIdx.x], sh_min[c][threadIdx.x + st]);
        sh_max[c][threadIdx.x] = fmax(sh_max[c][threadIdx.x], sh_max[c][threadIdx.x + st]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int c = 0; c < 3; ++c) {
      b.partial[(size_t)blockIdx.x * 8 + c] = sh_min[c][0];
      b.partial[(size_t)blockIdx.x * 8 + 3 + c] = sh_max[c][0];
    }
}

// The shell's bounds, average element size and cell grid (ShellSystem.C:1910-1969)
// from k_rb_aabb's per-block bounds and face sizes.  The 1024 lanes of the
// fixed-order sum of shl_geom.h are added on kBoundsBlocks SMs (a lane's sum
// is a chain of F / 1024 FP64 additions: on one SM the 1024 chains took most of
// a pass's bounds step); the last block adds the lanes in the fixed tree and
// makes the grid.
constexpr int kBoundsBlocks = 16;
__global__ void __launch_bounds__(kBlock) k_rb_bounds(DevBuf b, StepConst sc, uint32_t n_parts) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl) || sc.n_cs) return;  // a batch: per-shell grids (k_rb_grids)
  __shared__ double sh_min[3][kBlock], sh_max[3][kBlock];
  __shared__ double lanes[SHL_SUM_LANES];
  {
    constexpr uint32_t per_block = SHL_SUM_LANES / kBoundsBlocks;
    const uint32_t l = blockIdx.x * per_block + threadIdx.x;
    if (threadIdx.x < per_block) {
      double acc = 0.0;
#pragma unroll 4
      for (uint32_t i = l; i < sc.F; i += SHL_SUM_LANES) acc = __dadd_rn(acc, __ldcg(&b.fsize[i]));
      b.sum_lanes[l] = acc;
    }
  }
  if (!last_block_rb(&ctl->cnt[5])) return;
  // shell bounds (exact min/max)
  for (int c = 0; c < 3; ++c) {
    double mn = SHL_DBL_MAX, mx = -SHL_DBL_MAX;
    for (uint32_t k = threadIdx.x; k < n_parts; k += blockDim.x) {
      mn = fmin(mn, __ldcg(&b.partial[(size_t)k * 8 + c]));
      mx = fmax(mx, __ldcg(&b.partial[(size_t)k * 8 + 3 + c]));
    }
    sh_min[c][threadIdx.x] = mn;
    sh_max[c][threadIdx.x] = mx;
  }
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st)
      for (int c = 0; c < 3; ++c) {
        sh_min[c][threadIdx.x] = fmin(sh_min[c][threadIdx.x], sh_min[c][threadIdx.x + st]);
        sh_max[c][threadIdx.x] = fmax(sh_max[c][threadIdx.x], sh_max[c][threadIdx.x + st]);
      }
    __syncthreads();
  }
  // avg_elem_size: the fixed-order sum of shl_geom.h (1024 lanes, then a tree)
  for (uint32_t l = threadIdx.x; l < SHL_SUM_LANES; l += blockDim.x) lanes[l] = __ldcg(&b.sum_lanes[l]);
  __syncthreads();
  for (uint32_t st = SHL_SUM_LANES / 2; st > 0; st >>= 1) {
    for (uint32_t l = threadIdx.x; l < st; l += blockDim.x) lanes[l] = __dadd_rn(lanes[l], lanes[l + st]);
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  ctl->du_sum = 0.0;
  for (int c = 0; c < 3; ++c) {
    ctl->bmin[c] = sh_min[c][0];
    ctl->bmax[c] = sh_max[c][0];
  }
  const double avg = __ddiv_rn(lanes[0], (double)sc.F);
  ctl->avg_elem_size = avg;
  const uint64_t n_cells = grid_setup(ctl->bmin, ctl->bmax, avg, sc.cell_size_mult, sc.cell_margin, sc.thickness,
                                      sc.smooth, &ctl->cell_size, &ctl->d_max, ctl->ncd);
  ctl->d2_max = __dmul_rn(ctl->d_max, ctl->d_max);
  if (n_cells > sc.n_cells_max) {
    atomicMax(&ctl->problem, (int)SHL_TOO_MANY_CELLS);
    ctl->rebuild = 0;
    return;
  }
  if (n_cells > sc.n_cells_cap) {
    set_error(ctl, SHL_ERR_CAPACITY);
    return;
  }
  ctl->n_cells = (uint32_t)n_cells;
  ctl->n_old = ctl->n_pairs;
  ctl->n_new = 0;
  ctl->n_rebuilds += 1;
}

// ------------------------------------------------------- batch grids --
// One block per shell of a batch with self-contact: the shell's bounds and
// average element size (the fixed-order sum of shl_geom.h over the shell's own
// faces, so every value equals that of the shell run alone), its cell size,
// d_max and cell counts.  Shells whose trigger did not fire keep their list.
// 1024 threads, one per lane of the sum: with 256 the chains of a 20,000-face
// shell took 100 us.
__global__ void __launch_bounds__(SHL_SUM_LANES) k_rb_grids(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  ShellCell& S = b.shc[blockIdx.x];
  if (!S.rebuild) {
    if (threadIdx.x == 0) S.n_cells = 0;
    return;
  }
  __shared__ double sh_box[6][SHL_SUM_LANES / 32];
  __shared__ double lanes[SHL_SUM_LANES];
  const uint32_t f0 = S.face_first, nf = S.face_end - S.face_first;
  double box[6];  // the lower corner, and the upper one's negative
  for (int c = 0; c < 6; ++c) box[c] = SHL_DBL_MAX;
  double acc = 0.0;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < nf; i += SHL_SUM_LANES) {
    for (int c = 0; c < 3; ++c) {
      box[c] = fmin(box[c], b.bmin[3 * (size_t)(f0 + i) + c]);
      box[3 + c] = fmin(box[3 + c], -b.bmax[3 * (size_t)(f0 + i) + c]);
    }
    acc = __dadd_rn(acc, __ldcg(&b.fsize[f0 + i]));
  }
  lanes[threadIdx.x] = acc;
  for (int c = 0; c < 6; ++c) {
    for (int o = 16; o > 0; o >>= 1) box[c] = fmin(box[c], __shfl_xor_sync(0xffffffffu, box[c], o));
    if ((threadIdx.x & 31u) == 0) sh_box[c][threadIdx.x >> 5] = box[c];
  }
  __syncthreads();
  double sh_min[3], sh_max[3];
  if (threadIdx.x == 0)
    for (int c = 0; c < 3; ++c) {
      double lo = SHL_DBL_MAX, hi = SHL_DBL_MAX;
      for (int w = 0; w < SHL_SUM_LANES / 32; ++w) {
        lo = fmin(lo, sh_box[c][w]);
        hi = fmin(hi, sh_box[3 + c][w]);
      }
      sh_min[c] = lo;
      sh_max[c] = -hi;
    }
  for (uint32_t st = SHL_SUM_LANES / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) lanes[threadIdx.x] = __dadd_rn(lanes[threadIdx.x], lanes[threadIdx.x + st]);
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  S.du_sum = 0.0;
  for (int c = 0; c < 3; ++c) {
    S.bmin[c] = sh_min[c];
    S.bmax[c] = sh_max[c];
  }
  const double avg = __ddiv_rn(lanes[0], (double)nf);
  S.avg_elem_size = avg;
  const uint64_t n_cells = grid_setup(S.bmin, S.bmax, avg, S.cell_size_mult, sc.cell_margin, S.thickness, sc.smooth,
                                      &S.cell_size, &S.d_max, S.ncd);
  S.d2_max = __dmul_rn(S.d_max, S.d_max);
  S.n_rebuilds += 1;
  if (n_cells > S.n_cells_max) {
    atomicMax(&ctl->problem, (int)SHL_TOO_MANY_CELLS);
    ctl->rebuild = 0;
    S.n_cells = 0;
    return;
  }
  S.n_cells = n_cells > sc.n_cells_cap ? sc.n_cells_cap + 1u : (uint32_t)n_cells;
}

// first cell of each shell's grid (exclusive scan over the shells), the pass's
// cell count and the list counters (one block)
__global__ void __launch_bounds__(1024) k_rb_grid_scan(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  const uint32_t n = sc.n_cs;
  const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint32_t s0 = threadIdx.x * per;
  uint64_t tot = 0;
  for (uint32_t k = 0; k < per; ++k)
    if (s0 + k < n) tot += b.shc[s0 + k].n_cells;
  __shared__ unsigned long long sh[1024];
  sh[threadIdx.x] = tot;
  __syncthreads();
  for (uint32_t o = 1; o < blockDim.x; o <<= 1) {
    const unsigned long long y = threadIdx.x >= o ? sh[threadIdx.x - o] : 0ull;
    __syncthreads();
    sh[threadIdx.x] += y;
    __syncthreads();
  }
  uint64_t run = sh[threadIdx.x] - tot;
  for (uint32_t k = 0; k < per; ++k)
    if (s0 + k < n) {
      ShellCell& S = b.shc[s0 + k];
      S.cell_base = run < 0xFFFFFFFFull ? (uint32_t)run : 0xFFFFFFFFu;
      run += S.n_cells;
    }
  if (threadIdx.x != blockDim.x - 1) return;
  const unsigned long long all = sh[blockDim.x - 1];
  if (all > sc.n_cells_cap) {
    set_error(ctl, SHL_ERR_CAPACITY);
    return;
  }
  ctl->n_cells = (uint32_t)all;
  ctl->n_old = ctl->n_pairs;
  ctl->n_new = 0;
  ctl->n_rebuilds += 1;
}

// ---------------------------------------------------------------- clear --
__global__ void k_rb_clear(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  const uint32_t n_cells = ctl->n_cells;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_cells; i += stride) {
    b.cell_count[i] = 0;
    b.cell_fill[i] = 0;
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < sc.F; i += stride) {
    b.seg_count[i] = 0;
    b.new_cnt[i] = 0;
    b.new_fill[i] = 0;
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * sc.V; i += stride) b.p32[i] = (float)b.p[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->n_cand = 0;
}

// ---------------------------------------------------------------- count --
// A face covers from eight cells (elements the size of a cell) to hundreds (a
// coarse shell: level 3 with cells of 2h, 350 cells per face), so a group of G
// lanes takes a face and walks its cells together.  With one thread per face, the
// 1,280 faces of a level-3 shell took 58 us to count and 352 us to fill, a warp
// per face 8 and 15 us.  Above kWideFaces the faces fill the GPU: a thread per
// face counts (level 6: 19 us, 29 with eight lanes, whose divisions are spread
// thinner), eight lanes fill (14 us, a thread 23).
constexpr uint32_t kWideFaces = 8192;

// the cells lo..hi of a face, G lanes at a time: calls at(cell)
template <int G, class Fn>
__device__ __forceinline__ void walk_cells(const GridView& g, const int* lo, const int* hi, uint32_t sub, Fn at) {
  const int l[3] = {lo[0], lo[1], lo[2]}, h[3] = {hi[0], hi[1], hi[2]};  // at() stores: not to be read again
  const uint32_t total = shl_cells_covered(l, h);
  for (uint32_t q = sub; q < total; q += G) at(g.base + shl_cells_at(q, l, h, g.ny, g.nz));
}

// cell ranges (ShellSystem.C:1982-1983) and histogram of the faces (G = 1 or a
// whole warp), keep flags of the old pairs
template <int G>
__global__ void __launch_bounds__(kBlock) k_rb_count(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  const uint32_t stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t sub = t0 % G;
  // all lanes of a warp run the same trips (the range is exchanged by shuffles)
  for (uint32_t w0 = (t0 & ~31u) / G; w0 < sc.F; w0 += stride / G) {
    const uint32_t f = w0 + (t0 & 31u) / G;
    const bool on = f < sc.F && face_in_pass(b, sc, f);
    const GridView g = grid_of(b, sc, on ? f : 0u);
    int lo[3], hi[3];
    if (G == 1) {
      for (int c = 0; on && c < 3; ++c) {
        lo[c] = (int)__ddiv_rn(__dsub_rn(b.bmin[3 * (size_t)f + c], g.bmin[c]), g.cell_size);
        hi[c] = (int)__ddiv_rn(__dadd_rn(__dsub_rn(b.bmax[3 * (size_t)f + c], g.bmin[c]), g.d_max), g.cell_size);
        b.cell_lo[4 * (size_t)f + c] = lo[c];
        b.cell_hi[3 * (size_t)f + c] = hi[c];
      }
      if (on) walk_cells<G>(g, lo, hi, 0, [&](uint32_t cell) { atomicAdd(&b.cell_count[cell], 1u); });
      continue;
    }
    int r = 0;
    if (on && sub < 6) {
      // lane c the range's start on axis c, lane 3 + c its end
      const uint32_t c = sub % 3u;
      const double cs = g.cell_size;
      if (sub < 3) {
        r = (int)__ddiv_rn(__dsub_rn(b.bmin[3 * (size_t)f + c], g.bmin[c]), cs);
        b.cell_lo[4 * (size_t)f + c] = r;
      } else {
        r = (int)__ddiv_rn(__dadd_rn(__dsub_rn(b.bmax[3 * (size_t)f + c], g.bmin[c]), g.d_max), cs);
        b.cell_hi[3 * (size_t)f + c] = r;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      lo[c] = __shfl_sync(0xffffffffu, r, c);
      hi[c] = __shfl_sync(0xffffffffu, r, 3 + c);
    }
    if (on) walk_cells<G>(g, lo, hi, sub, [&](uint32_t cell) { atomicAdd(&b.cell_count[cell], 1u); });
  }
  const uint32_t n_old = ctl->n_old;
  for (uint32_t j = t0; j < n_old; j += stride) {
    // ShellSystem.C:2020: drop unless sticking or still within d_max; a shell
    // of a batch that is not rebuilt keeps its whole list
    const uint32_t e1 = b.pe1[0][j];
    const bool keep = !face_in_pass(b, sc, e1) || b.pstick[0][j] != 0 || !(b.pd2[0][j] > grid_of(b, sc, e1).d2_max);
    b.pkeep[j] = keep ? 1 : 0;
    if (keep) atomicAdd(&b.seg_count[b.pe1[0][j]], 1u);
  }
}

// ----------------------------------------------------------------- scan --
// Exclusive scan of in[0..n) into out[0..n) (+ out[n] = total if with_end),
// gated by *gate; two launches.  n may be far below its capacity (the cells of a
// batch of which one shell is rebuilt; no pass at all), so the blocks are at most
// kScanBlocks and take every gridDim.x-th tile (a block per tile of the capacity:
// 68 us for the 100,000 tiles of a 256-shell batch that had nothing to scan).
constexpr uint32_t kScanBlocks = 152 * 8;
__global__ void __launch_bounds__(kBlock) k_scan_tiles(const uint32_t* gate, const Ctl* ctl, const uint32_t* in,
                                                       uint32_t* out, const uint32_t* n_ptr, uint32_t n_const,
                                                       uint32_t* tile_sums) {
  if (*gate == 0 || ctl->halted) return;
  const uint32_t n = n_ptr ? *n_ptr : n_const;
  constexpr int PER = kScanTile / kBlock;
  __shared__ uint32_t wsum[kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t tile = blockIdx.x; (uint64_t)tile * kScanTile < n; tile += gridDim.x) {
    uint32_t v[PER];
    uint32_t sum = 0;
    const uint32_t i0 = tile * kScanTile + threadIdx.x * PER;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const uint32_t x = (i0 + k < n) ? in[i0 + k] : 0u;
      v[k] = sum;
      sum += x;
    }
    // exclusive scan of the per-thread sums over the block
    uint32_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    __syncthreads();  // the previous tile's sums have been read
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = (lane < kBlock / 32) ? wsum[lane] : 0u;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      if (lane < kBlock / 32) wsum[lane] = w;
    }
    __syncthreads();
    const uint32_t excl = incl - sum + (warp > 0 ? wsum[warp - 1] : 0u);
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (i0 + k < n) out[i0 + k] = v[k] + excl;
    if (threadIdx.x == kBlock - 1) tile_sums[tile] = excl + sum;
  }
}

// Each tile's offset is the sum of the tiles before it, added up by the block that
// takes the tile (from its previous tile on); block 0 adds all of them: the total,
// out[n] and the capacity check.
__global__ void __launch_bounds__(kBlock) k_scan_add(const uint32_t* gate, Ctl* ctl, uint32_t* out,
                                                     const uint32_t* n_ptr, uint32_t n_const,
                                                     const uint32_t* tile_sums, uint32_t* total, int with_end,
                                                     uint32_t cap, int cap_error) {
  if (*gate == 0 || ctl->halted) return;
  const uint32_t n = n_ptr ? *n_ptr : n_const;
  __shared__ uint32_t wsum[kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the block's sum of tile_sums[from, to), in every thread
  auto block_total = [&](uint32_t from, uint32_t to) {
    uint32_t s = 0;
    for (uint32_t t = from + threadIdx.x; t < to; t += blockDim.x) s += tile_sums[t];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if (lane == 0) wsum[warp] = s;
    __syncthreads();
    s = 0;
    for (int w = 0; w < kBlock / 32; ++w) s += wsum[w];
    return s;
  };
  uint32_t add = 0, done = 0;  // the offset of tile `done`
  for (uint32_t tile = blockIdx.x; (uint64_t)tile * kScanTile < n; tile += gridDim.x) {
    add += block_total(done, tile);
    done = tile;
    if (tile == 0) continue;
    const uint32_t base = tile * kScanTile;
    for (uint32_t i = base + threadIdx.x; i < base + kScanTile && i < n; i += blockDim.x) out[i] += add;
  }
  if (blockIdx.x != 0) return;
  add += block_total(done, (n + kScanTile - 1) / kScanTile);
  if (threadIdx.x != 0) return;
  *total = add;
  if (with_end) out[n] = add;
  if (cap_error && add > cap) {
    atomicMax(&ctl->error, (int)SHL_ERR_CAPACITY);
    ctl->rebuild = 0;
    ctl->csr_dirty = 0;
  }
}

void launch_scan(const uint32_t* gate, Ctl* ctl, const uint32_t* in, uint32_t* out, const uint32_t* n_ptr,
                 uint32_t n_const, uint32_t n_cap, uint32_t* tile_sums, uint32_t* total, bool with_end,
                 uint32_t cap, bool cap_error, cudaStream_t s) {
  const uint32_t nt = (n_cap + kScanTile - 1) / kScanTile;
  const uint32_t grid = std::min(nt > 0 ? nt : 1u, kScanBlocks);
  k_scan_tiles<<<grid, kBlock, 0, s>>>(gate, ctl, in, out, n_ptr, n_const, tile_sums);
  k_scan_add<<<grid, kBlock, 0, s>>>(gate, ctl, out, n_ptr, n_const, tile_sums, total, with_end ? 1 : 0, cap,
                                     cap_error ? 1 : 0);
}

// ----------------------------------------------------------------- fill --
template <int G>
__global__ void __launch_bounds__(kBlock) k_rb_fill(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  const uint32_t stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t f = t0 / G; f < sc.F; f += stride / G) {
    if (!face_in_pass(b, sc, f)) continue;
    const GridView g = grid_of(b, sc, f);
    walk_cells<G>(g, b.cell_lo + 4 * (size_t)f, b.cell_hi + 3 * (size_t)f, t0 % G, [&](uint32_t cell) {
      const uint32_t pos = b.cell_start[cell] + atomicAdd(&b.cell_fill[cell], 1u);
      b.cell_items[pos] = f;
      b.entry_cell[pos] = cell;
    });
  }
}

__device__ __forceinline__ bool sorted_contains(const uint32_t* a, uint32_t lo, uint32_t hi, uint32_t x) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    const uint32_t y = a[mid];
    if (y == x) return true;
    if (y < x) lo = mid + 1; else hi = mid;
  }
  return false;
}

// index of x in a[lo..hi), or hi if absent
__device__ __forceinline__ uint32_t sorted_find(const uint32_t* a, uint32_t lo, uint32_t hi, uint32_t x) {
  const uint32_t end = hi;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    const uint32_t y = a[mid];
    if (y == x) return mid;
    if (y < x) lo = mid + 1; else hi = mid;
  }
  return end;
}

// ---------------------------------------------------------------- pairs --
// Conservative separating-axis tests in FP32 on FP32 copies of the positions:
// true only when the triangles are certainly farther apart than d_max.  For an
// axis a (any vector, unnormalised, |a| = L) the projections of the two
// triangles onto a are separated by more than d_max L, allowing for the
// rounding of the FP32 projections (including the rounding of the positions to
// FP32): at most 32 eps32 L S with S the largest coordinate magnitude.  The
// remaining relative margin (1e-5) is far above the rounding of the FP64
// closest-point solve, so a pair rejected here is one the exact path would
// reject too (d^2 > d_max^2).  The axes: the line of centroids, the two face
// normals and the in-plane normals of the six edges (n x e), which separate
// neighbouring, nearly coplanar faces of a smooth surface.
__device__ __forceinline__ bool apart_on_axis(const float* a, const float* const* P1, const float* const* P2,
                                              float d_max, float S) {
  const float L2 = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
  if (!(L2 > 0.f)) return false;
  float mn1 = 3.0e38f, mx1 = -3.0e38f, mn2 = 3.0e38f, mx2 = -3.0e38f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float q1 = a[0] * P1[k][0] + a[1] * P1[k][1] + a[2] * P1[k][2];
    const float q2 = a[0] * P2[k][0] + a[1] * P2[k][1] + a[2] * P2[k][2];
    mn1 = fminf(mn1, q1);
    mx1 = fmaxf(mx1, q1);
    mn2 = fminf(mn2, q2);
    mx2 = fmaxf(mx2, q2);
  }
  const float L = sqrtf(L2);
  const float gap = fmaxf(mn2 - mx1, mn1 - mx2) - 32.f * 5.9604645e-8f * L * S;
  return gap > d_max * L * (1.f + 1e-5f);
}

// the line of centroids (S: the largest coordinate magnitude, for the next test)
__device__ __forceinline__ bool apart_centroids32(const float* const* P1, const float* const* P2, float d_max,
                                                  float& S) {
  float d[3];
  S = 0.f;
  for (int c = 0; c < 3; ++c) {
    d[c] = (P2[0][c] + P2[1][c] + P2[2][c]) - (P1[0][c] + P1[1][c] + P1[2][c]);
    for (int k = 0; k < 3; ++k) S = fmaxf(S, fmaxf(fabsf(P1[k][c]), fabsf(P2[k][c])));
  }
  return apart_on_axis(d, P1, P2, d_max, S);
}

// the face normals and the in-plane edge normals
__device__ __forceinline__ bool apart_faces32(const float* const* P1, const float* const* P2, float d_max, float S) {
  const float* const* T[2] = {P1, P2};
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const float* const* P = T[t];
    float e[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) e[k][c] = P[(k + 1) % 3][c] - P[k][c];
    const float n[3] = {e[0][1] * e[2][2] - e[0][2] * e[2][1], e[0][2] * e[2][0] - e[0][0] * e[2][2],
                        e[0][0] * e[2][1] - e[0][1] * e[2][0]};
    if (apart_on_axis(n, P1, P2, d_max, S)) return true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float m[3] = {n[1] * e[k][2] - n[2] * e[k][1], n[2] * e[k][0] - n[0] * e[k][2],
                          n[0] * e[k][1] - n[1] * e[k][0]};
      if (apart_on_axis(m, P1, P2, d_max, S)) return true;
    }
  }
  return false;
}

// The filters of a pair (e1 < e2) that shares a cell, after the cell tests: not
// topologically close, not in the kept list, not AABB-apart by d_max
// (ShellSystem.C:2047-2060), and not certainly apart by the separating-axis
// tests.  They are conjunctive, so their order leaves the result unchanged; the
// cheap and decisive ones come first.
__device__ __forceinline__ bool cand_passes(const DevBuf& b, const StepConst& sc, uint32_t e1, uint32_t e2) {
  // faces sharing a node are neighbours in the mesh, always in the close list (ShellSystem.C:657-678)
  uint32_t t1[3], t2[3];
  for (int q = 0; q < 3; ++q) {
    t1[q] = b.tri[3 * (size_t)e1 + q];
    t2[q] = b.tri[3 * (size_t)e2 + q];
  }
  for (int q = 0; q < 3; ++q)
    if (t2[q] == t1[0] || t2[q] == t1[1] || t2[q] == t1[2]) return false;
  const double d_max = sc.n_cs ? b.shc[b.face_shell[e1]].d_max : b.ctl->d_max;
  bool apart = false;
  for (int c = 0; c < 3; ++c) {
    const double mn1 = b.bmin[3 * (size_t)e1 + c], mx1 = b.bmax[3 * (size_t)e1 + c];
    const double mn2 = b.bmin[3 * (size_t)e2 + c], mx2 = b.bmax[3 * (size_t)e2 + c];
    apart = apart || mn1 > __dadd_rn(mx2, d_max) || mn2 > __dadd_rn(mx1, d_max);
  }
  if (apart) return false;
  if (!sc.smooth) {  // facet bounds; SMOOTH distances are between limit surfaces
    const float* Q1[3];
    const float* Q2[3];
    for (int q = 0; q < 3; ++q) {
      Q1[q] = b.p32 + 3 * (size_t)t1[q];
      Q2[q] = b.p32 + 3 * (size_t)t2[q];
    }
    float S = 0.f;
    if (apart_centroids32(Q1, Q2, (float)d_max, S) || apart_faces32(Q1, Q2, (float)d_max, S)) return false;
  }
  if (sorted_contains(b.close_list, b.close_ptr[e1], b.close_ptr[e1 + 1], e2)) return false;
  const uint32_t o1 = b.pair_ptr[0][e1 + 1];
  const uint32_t at = sorted_find(b.pe2[0], b.pair_ptr[0][e1], o1, e2);
  return !(at < o1 && b.pkeep[at]);
}

// Candidate pairs of the (cell, face) entries: faces e2 > e1 in the cell, emitted
// from the lowest shared cell only, that pass the filters above.  A lane walks its
// entry's cell; one check in twelve passes the cell tests, and the filters behind
// them are a chain of scattered loads, so with both in one loop every trip of a
// warp paid for the filters with a few lanes in them.  The pairs that pass are
// queued per warp in shared memory and filtered 32 at a time: a level-6 sphere's
// 13 M checks 200 -> 81 us, a folded shell 0.91 -> 0.51 ms.  (Checking four faces
// at a time in the old loop: 188 us, and 1.15 ms in the folded shell.)
constexpr int kCandBlock = 256;
constexpr uint32_t kCandQueue = 64;
__global__ void __launch_bounds__(kCandBlock) k_rb_cand(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  __shared__ uint2 queues[kCandBlock / 32][kCandQueue];
  uint2* queue = queues[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  const uint32_t n_entries = ctl->n_entries;
  uint32_t queued = 0;
  // the filters of the queue's last 32 (or all remaining) pairs
  auto drain = [&](uint32_t n) {
    __syncwarp();
    const uint2 pr = lane < n ? queue[queued - n + lane] : make_uint2(0u, 0u);
    const bool ok = lane < n && cand_passes(b, sc, pr.x, pr.y);
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    queued -= n;
    if (!m) return;
    uint32_t off = 0;
    if (lane == 0) off = atomicAdd(&ctl->n_cand, (uint32_t)__popc(m));
    off = __shfl_sync(0xffffffffu, off, 0);
    if (off + (uint32_t)__popc(m) > sc.cand_cap) {
      if (lane == 0) set_error(ctl, SHL_ERR_CAPACITY);
    } else if (ok) {
      const uint32_t at = off + (uint32_t)__popc(m & below);
      b.cand_e1[at] = pr.x;
      b.cand_e2[at] = pr.y;
    }
  };
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t j0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); j0 < n_entries; j0 += stride) {
    const uint32_t j = j0 + lane;
    uint32_t e1 = 0, s0 = 0, cnt = 0, cx = 0, cy = 0, cz = 0;
    int4 lo1 = make_int4(0, 0, 0, 0);
    if (j < n_entries) {
      e1 = b.cell_items[j];
      const GridView g = grid_of(b, sc, e1);
      const uint32_t cell = b.entry_cell[j], local = cell - g.base;
      cz = local % g.nz;
      cy = (local / g.nz) % g.ny;
      cx = local / (g.nz * g.ny);
      lo1 = reinterpret_cast<const int4*>(b.cell_lo)[e1];
      s0 = b.cell_start[cell];
      cnt = b.cell_count[cell];
    }
    const uint32_t trips = __reduce_max_sync(0xffffffffu, cnt);
    uint32_t next = cnt > 0 ? b.cell_items[s0] : 0u;
    for (uint32_t k = 0; k < trips; ++k) {
      const uint32_t e2 = next;
      if (k + 1 < cnt) next = b.cell_items[s0 + k + 1];
      bool pass = false;
      if (k < cnt && e2 > e1) {
        const int4 lo2 = reinterpret_cast<const int4*>(b.cell_lo)[e2];
        pass = (uint32_t)max(lo1.x, lo2.x) == cx && (uint32_t)max(lo1.y, lo2.y) == cy && (uint32_t)max(lo1.z, lo2.z) == cz;
      }
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      if (pass) queue[queued + (uint32_t)__popc(m & below)] = make_uint2(e1, e2);
      queued += (uint32_t)__popc(m);
      if (queued >= 32) drain(32);
    }
  }
  if (queued > 0) drain(queued);
}

// the acceptance of a candidate at squared distance d2 (ShellSystem.C:2082)
__device__ __forceinline__ void narrow_accept(const DevBuf& b, const StepConst& sc, Ctl* ctl, uint32_t i, uint32_t e1,
                                              double d2) {
  const double d2_max = sc.n_cs ? b.shc[b.face_shell[e1]].d2_max : ctl->d2_max;
  if (d2 <= 0.0) atomicMax(&ctl->problem, (int)SHL_CONTACT_PROBLEM);
  const bool ok = !(d2 > d2_max);
  b.cand_d2[i] = d2;
  b.cand_ok[i] = ok ? 1 : 0;
  if (ok) {
    atomicAdd(&b.new_cnt[e1], 1u);
    atomicAdd(&b.seg_count[e1], 1u);
  }
}

// closest-point test of each candidate (rounded operation by operation)
__global__ void __launch_bounds__(kBlock) k_rb_narrow(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  extern __shared__ __align__(16) unsigned char pair_smem[];
  PairWork& work = *reinterpret_cast<PairWork*>(pair_smem);
  const uint32_t n = min(ctl->n_cand, sc.cand_cap);
  for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
    const uint32_t i = i0 + threadIdx.x;
    const bool active = i < n;
    const uint32_t ii = active ? i : i0;
    const uint32_t e1 = b.cand_e1[ii], e2 = b.cand_e2[ii];
    const double* P1[3];
    const double* P2[3];
    for (int q = 0; q < 3; ++q) {
      P1[q] = b.p + 3 * (size_t)b.tri[3 * (size_t)e1 + q];
      P2[q] = b.p + 3 * (size_t)b.tri[3 * (size_t)e2 + q];
    }
    shl_pair_geom g;
    pair_compute_block(active, P1, P2, work, &g);
    if (active) narrow_accept(b, sc, ctl, i, e1, g.d2);
  }
}

// The power form of each regular patch at the current positions, and of the
// irregular patches' subdivision children (sc.irr_levels levels, three children
// each; a thread per child and component).  A search evaluates a patch many
// times: formed in the search, an irregular patch's control points (12 table rows
// of N + 6 nodes) and coefficients took about 35 us per evaluation of one lane,
// and the few pairs next to an irregular vertex held the whole launch.
__global__ void __launch_bounds__(kBlock) k_limit_coeffs(DevBuf b, StepConst sc, bool rebuild) {
  const Ctl* ctl = b.ctl;
  if (rebuild ? rb_off(ctl) : (ctl->halted != 0 || ctl->paused != 0)) return;
  const uint32_t n_irr = (sc.F - sc.irr_first) * (uint32_t)sc.irr_levels * 9u;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < sc.F + n_irr; t += gridDim.x * blockDim.x) {
    if (t < n_irr) {
      const int c = (int)(t % 3u), k = (int)(t / 3u % 3u);
      const uint32_t q = t / 9u;
      const int slot = (int)(q % (uint32_t)sc.irr_levels), n = slot == sc.irr_levels - 1 ? SHL_SMOOTH_LEVELS : 1 + slot;
      shl_limit_patch lp;
      smooth_patch(b, sc, b.perm[sc.irr_first + q / (uint32_t)sc.irr_levels], lp);
      SHL_TABLE signed char BC[12][15] = SHL_BOX_COEFFS;
      double P[15];
#pragma unroll
      for (int m = 0; m < 15; ++m) P[m] = 0.0;
#pragma unroll
      for (int s = 0; s < 12; ++s) {
        const double Q = shl_limit_child_point(&lp, n, k, s, c);
#pragma unroll
        for (int m = 0; m < 15; ++m)
          if (BC[s][m] != 0) P[m] = SHL_FMA((double)BC[s][m], Q, P[m]);
      }
      double* out = b.icoef + SHL_LIMIT_NCOEF * (size_t)(t / 3u) + c;
      const double twelfth = 1.0 / 12.0;
#pragma unroll
      for (int m = 0; m < 15; ++m) out[3 * m] = SHL_MUL(P[m], twelfth);
      continue;
    }
    const uint32_t e = t - n_irr;
    if ((b.fsm[e] & 0xff) != 6) continue;
    shl_limit_patch lp;
    smooth_patch(b, sc, e, lp);
    double P[15][3];
    shl_limit_coeffs_regular(&lp, P);
    double* out = b.lcoef + SHL_LIMIT_NCOEF * (size_t)e;
    for (int m = 0; m < 15; ++m)
      for (int c = 0; c < 3; ++c) out[3 * m + c] = P[m][c];
  }
}

// the place of subdivision level n among a patch's stored levels, the first
// levels - 1 and the last one (the patch's corner, where many a search ends), or -1
__device__ __forceinline__ int stored_slot(int n, int levels) {
  return n == SHL_SMOOTH_LEVELS ? levels - 1 : (n < levels ? n - 1 : -1);
}

// a patch's limit surface at (v, w) from the stored power forms; deep: also the
// levels of an irregular patch beyond them (the form is made here; the lanes of
// a batch evaluate theirs together)
template <int ORDER, bool DEEP>
__device__ __noinline__ void limit_at(const DevBuf& b, const StepConst& sc, uint32_t e, double v, double w, double out[6][3]) {
  double j1 = 1.0;
  const double* coef = b.lcoef + SHL_LIMIT_NCOEF * (size_t)e;
  double P[15][3];
  if ((b.fsm[e] & 0xff) != 6) {
    int n, k;
    shl_limit_child(&v, &w, &n, &k, &j1);
    const int slot = stored_slot(n, sc.irr_levels);
    if (DEEP && slot < 0) {
      shl_limit_patch lp;
      smooth_patch(b, sc, e, lp);
      shl_limit_coeffs_child(&lp, n, k, P);
      coef = &P[0][0];
    } else {
      coef = b.icoef +
             SHL_LIMIT_NCOEF * ((size_t)((b.inv_perm[e] - sc.irr_first) * (uint32_t)sc.irr_levels + (uint32_t)slot) * 3 + (size_t)k);
    }
  }
  shl_limit_poly(reinterpret_cast<const double(*)[3]>(coef), v, w, ORDER, j1, out);
}

// SMOOTH closest-point searches in phase-coherent batches.  A search alternates
// between the order-2 evaluation of an iterate with its Newton step (about 1200
// FP64 operations) and the order-0 evaluation of a line-search trial (about 180),
// and takes from one to several hundred of them.  With one search per lane the
// lanes of a warp sit in different phases, and every trip pays for both with a
// third of the lanes busy in each.  Here a warp owns kSearchPool searches, kept
// in shared memory as resumable states (shl_smooth_state), and per trip runs up
// to 32 of them that are in the same phase.  A search whose next point lies in an
// irregular patch beyond the stored children makes a power form for it, which
// costs more than the rest of a trip; those are classes of their own, again one
// per phase (as one class, for every search with an irregular patch, they made
// batches and irregular meshes up to 1.9 times slower than a search per lane).
// With more searches than lanes there is nearly always a full batch of one class.  A finished
// search's slot is refilled from a queue shared by the grid (ctl->cnt[7]; the
// last warp to leave resets it).  A search's result does not depend on the lane
// or the order that runs it.  Folded level-5 shell, 1.4 M candidates at 5.9
// Newton iterates each: 100 -> 44 ms for a list build's searches (64 ms from the
// batches, 51 with the irregular children stored, 44 with the failing shifts of
// shl_smooth_direction passed over and the evaluation out of line), 8.6 -> 3.1 ms
// per step.  Pools of 64, 96 and 128 searches and two to four blocks per SM are
// within 3 %.  What is left is the FP64 pipe (57-80 % busy) and, in the list
// build, instruction fetches of the divergent Newton step.
//   REBUILD: the candidates of a linked-cell pass, each from (1/3, 1/3, 1/3,
//   1/3) as a new SmoothShellShellContact (SmoothShellShellContact.C:9-14),
//   then k_rb_narrow's acceptance;
//   else: the pairs of the list from their previous solution; x, d2 and
//   dc = p2 - p1 go to pvw, pd2 and the pair's force slots 0-2 for
//   k_contact_force.
constexpr int kSearchBlock = 128;
constexpr int kSearchPool = 64;  // searches per warp (a multiple of 32)
enum : uint8_t { kSearchEmpty = 0, kSearchNewton = 1, kSearchTrial = 2, kSearchDeep = 2 };  // + kSearchDeep: 3, 4
constexpr int kSearchClasses = 5;
struct SearchPool {
  double x[4][kSearchPool], xt[4][kSearchPool], d[4][kSearchPool], p1[3][kSearchPool], p2[3][kSearchPool];
  double f[kSearchPool], alpha[kSearchPool], gd[kSearchPool], dn[kSearchPool];
  uint32_t j[kSearchPool], e1[kSearchPool], e2[kSearchPool];
  uint8_t cls[kSearchPool], it[kSearchPool], ls[kSearchPool], shifted[kSearchPool], after_accept[kSearchPool];
  uint8_t irregular[kSearchPool];  // bit 0 / 1: element 1 / 2 has an irregular patch
  uint8_t batch[32];
};

// One trip of the pool's slot s, whose next evaluation is a Newton iterate's
// (phase SHL_SMOOTH_EVAL_FGH) or a trial's (SHL_SMOOTH_EVAL_TRIAL).
template <bool REBUILD, bool DEEP>
__device__ __forceinline__ void search_trip(const DevBuf& b, const StepConst& sc, Ctl* ctl, SearchPool& w, uint32_t s,
                                            int phase) {
  const uint32_t e1 = w.e1[s], e2 = w.e2[s];
  shl_smooth_state st;
  st.phase = phase;
  st.it = w.it[s];
  st.after_accept = w.after_accept[s];
#pragma unroll
  for (int k = 0; k < 4; ++k) st.x[k] = w.x[k][s];
  if (phase == SHL_SMOOTH_EVAL_TRIAL) {
    st.f = w.f[s];
    st.alpha = w.alpha[s];
    st.gd = w.gd[s];
    st.dn = w.dn[s];
    st.ls = w.ls[s];
    st.shifted = w.shifted[s];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      st.xt[k] = w.xt[k][s];
      st.d[k] = w.d[k][s];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      st.p1[c] = w.p1[c][s];
      st.p2[c] = w.p2[c][s];
    }
  }
  {
    const double* pt = phase == SHL_SMOOTH_EVAL_FGH ? st.x : st.xt;
    double ev1[6][3], ev2[6][3];
    if (phase == SHL_SMOOTH_EVAL_FGH) {
      limit_at<2, DEEP>(b, sc, e1, pt[0], pt[1], ev1);
      limit_at<2, DEEP>(b, sc, e2, pt[2], pt[3], ev2);
    } else {
      limit_at<0, DEEP>(b, sc, e1, pt[0], pt[1], ev1);
      limit_at<0, DEEP>(b, sc, e2, pt[2], pt[3], ev2);
    }
    shl_smooth_take(&st, ev1, ev2);
  }
  if (st.phase == SHL_SMOOTH_DONE) {
    const uint32_t j = w.j[s];
    w.cls[s] = kSearchEmpty;
    if (REBUILD) {
      for (int k = 0; k < 4; ++k) b.cand_x[4 * (size_t)j + k] = st.x[k];
      narrow_accept(b, sc, ctl, j, e1, st.f);
    } else {
      for (int k = 0; k < 4; ++k) b.pvw[0][4 * (size_t)j + k] = st.x[k];
      b.pd2[0][j] = st.f;
      double* out = b.pforce + kPairOut * (size_t)j;
      for (int c = 0; c < 3; ++c) out[c] = SHL_SUB(st.p2[c], st.p1[c]);
    }
    return;
  }
  w.it[s] = (uint8_t)st.it;
  w.after_accept[s] = (uint8_t)st.after_accept;
#pragma unroll
  for (int k = 0; k < 4; ++k) w.x[k][s] = st.x[k];
  if (st.phase == SHL_SMOOTH_EVAL_TRIAL) {
    w.alpha[s] = st.alpha;
    w.ls[s] = (uint8_t)st.ls;
#pragma unroll
    for (int k = 0; k < 4; ++k) w.xt[k][s] = st.xt[k];
    if (phase == SHL_SMOOTH_EVAL_FGH) {
      w.f[s] = st.f;
      w.gd[s] = st.gd;
      w.dn[s] = st.dn;
      w.shifted[s] = (uint8_t)st.shifted;
#pragma unroll
      for (int k = 0; k < 4; ++k) w.d[k][s] = st.d[k];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        w.p1[c][s] = st.p1[c];
        w.p2[c][s] = st.p2[c];
      }
    }
  }
  w.cls[s] = st.phase == SHL_SMOOTH_EVAL_TRIAL ? kSearchTrial : kSearchNewton;
}

// a search of the shallow classes moves to the deep ones if its next point lies in
// an irregular patch beyond the stored levels
__device__ __noinline__ void deepen(SearchPool& w, uint32_t s, int levels) {
  const unsigned irr = w.irregular[s], cls = w.cls[s];
  if (irr == 0 || cls == kSearchEmpty) return;
  const double(*pt)[kSearchPool] = cls == kSearchTrial ? w.xt : w.x;
  for (int k = 0; k < 2; ++k) {
    if (!(irr >> k & 1u)) continue;
    double v = pt[2 * k][s], x = pt[2 * k + 1][s];
    if (stored_slot(shl_rescale_irregular(&v, &x), levels) < 0) {
      w.cls[s] = (uint8_t)(cls + kSearchDeep);
      return;
    }
  }
}

// trips of the deep classes, out of line: they are rare on most meshes, and their
// copy of the evaluation would crowd the others out of the instruction cache
template <bool REBUILD>
__device__ __noinline__ void search_trip_deep(const DevBuf& b, const StepConst& sc, Ctl* ctl, SearchPool& w, uint32_t s,
                                              int phase) {
  search_trip<REBUILD, true>(b, sc, ctl, w, s, phase);
}

// DEEP: not every level of every irregular patch is stored (sc.irr_levels).  With
// all of them, the deep classes and their calls are left out of the kernel, which
// as a branch of it cost a sphere's searches 2 to 4 %.
template <bool REBUILD, bool DEEP>
__global__ void __launch_bounds__(kSearchBlock, 2) k_smooth_search(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  uint32_t* queue = &ctl->cnt[7];
  uint32_t* left = &ctl->cnt[8];
  const bool off = REBUILD ? rb_off(ctl) : (ctl->halted != 0 || ctl->paused != 0);
  const uint32_t n = off ? 0u : (REBUILD ? min(ctl->n_cand, sc.cand_cap) : ctl->n_pairs);
  extern __shared__ __align__(16) unsigned char search_smem[];
  SearchPool& w = reinterpret_cast<SearchPool*>(search_smem)[threadIdx.x >> 5];
  constexpr int R = kSearchPool / 32;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  bool more = n > 0;
#pragma unroll
  for (int r = 0; r < R; ++r) w.cls[32 * r + lane] = kSearchEmpty;
  __syncwarp();
  while (n > 0) {
    // slots of each class
    uint8_t cl[R];
    constexpr int kClasses = DEEP ? kSearchClasses : kSearchTrial + 1;
    unsigned count[kClasses] = {};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      cl[r] = w.cls[32 * r + lane];
#pragma unroll
      for (int k = 0; k < kClasses; ++k) count[k] += __popc(__ballot_sync(0xffffffffu, cl[r] == k));
    }
    if (more && count[kSearchEmpty] >= 16) {
      // refill the empty slots
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(queue, count[kSearchEmpty]);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (!(base + count[kSearchEmpty] < n)) more = false;  // the queue is empty for every warp
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const unsigned idle = __ballot_sync(0xffffffffu, cl[r] == kSearchEmpty);
        const uint32_t i = base + (uint32_t)__popc(idle & below);
        base += (uint32_t)__popc(idle);
        if (cl[r] != kSearchEmpty || i >= n) continue;
        const uint32_t s = 32 * r + lane;
        uint32_t e1, e2;
        double x0[4];
        if (REBUILD) {
          e1 = b.cand_e1[i];
          e2 = b.cand_e2[i];
          for (int k = 0; k < 4; ++k) x0[k] = 1.0 / 3.0;
        } else {
          e1 = b.pe1[0][i];
          e2 = b.pe2[0][i];
          for (int k = 0; k < 4; ++k) x0[k] = b.pvw[0][4 * (size_t)i + k];
        }
        shl_smooth_state st;
        shl_smooth_start(&st, x0);
        w.j[s] = i;
        w.e1[s] = e1;
        w.e2[s] = e2;
        for (int k = 0; k < 4; ++k) w.x[k][s] = st.x[k];
        w.it[s] = 0;
        w.after_accept[s] = 0;
        w.cls[s] = kSearchNewton;
        if (DEEP) {
          w.irregular[s] = (uint8_t)(((b.fsm[e1] & 0xff) != 6 ? 1u : 0u) | ((b.fsm[e2] & 0xff) != 6 ? 2u : 0u));
          deepen(w, s, sc.irr_levels);
        }
      }
      __syncwarp();
      continue;
    }
    // the largest class runs a batch
    int pick = kSearchNewton;
#pragma unroll
    for (int k = kSearchTrial; k < kClasses; ++k)
      if (count[k] > count[pick]) pick = k;
    if (count[pick] == 0) break;  // no search left (the queue is empty: an empty pool would have been refilled)
    uint32_t pos = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned m = __ballot_sync(0xffffffffu, cl[r] == pick);
      const uint32_t q = pos + (uint32_t)__popc(m & below);
      if (cl[r] == pick && q < 32) w.batch[q] = (uint8_t)(32 * r + lane);
      pos += (uint32_t)__popc(m);
    }
    __syncwarp();
    if (lane < count[pick]) {
      const uint32_t s = w.batch[lane];
      if (pick == kSearchNewton)
        search_trip<REBUILD, false>(b, sc, ctl, w, s, SHL_SMOOTH_EVAL_FGH);
      else if (pick == kSearchTrial)
        search_trip<REBUILD, false>(b, sc, ctl, w, s, SHL_SMOOTH_EVAL_TRIAL);
      else if (DEEP)
        search_trip_deep<REBUILD>(b, sc, ctl, w, s,
                                  pick == kSearchTrial + kSearchDeep ? SHL_SMOOTH_EVAL_TRIAL : SHL_SMOOTH_EVAL_FGH);
      if (DEEP) deepen(w, s, sc.irr_levels);
    }
    __syncwarp();
  }
  if (lane == 0) {
    __threadfence();
    const uint32_t warps = gridDim.x * (kSearchBlock / 32);
    if (atomicAdd(left, 1u) == warps - 1) {
      atomicExch(queue, 0u);
      atomicExch(left, 0u);
    }
  }
}

// accepted candidates grouped by eid1 (counting sort; order inside a group is
// fixed later by the assembly)
__global__ void __launch_bounds__(kBlock) k_rb_scatter_new(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  const uint32_t n = min(ctl->n_cand, sc.cand_cap);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!b.cand_ok[i]) continue;
    const uint32_t e1 = b.cand_e1[i];
    const uint32_t pos = b.new_off[e1] + atomicAdd(&b.new_fill[e1], 1u);
    b.new_e2[pos] = b.cand_e2[i];
    b.new_d2[pos] = b.cand_d2[i];
    if (sc.smooth)
      for (int k = 0; k < 4; ++k) b.new_x[4 * (size_t)pos + k] = b.cand_x[4 * (size_t)i + k];
  }
}

// -------------------------------------------------------------- assemble --
// one face's segment of the new list, serially: the face's new pairs sorted
// by e2 in place (insertion sort), merged with its kept old pairs
__device__ void assemble_serial(const DevBuf& b, const StepConst& sc, uint32_t e1) {
  uint32_t dst = b.pair_ptr[1][e1];
  const uint32_t o0 = b.pair_ptr[0][e1], o1 = b.pair_ptr[0][e1 + 1];
  const uint32_t nn = b.new_cnt[e1];
  const uint32_t off = nn ? b.new_off[e1] : 0u;
  uint32_t* ne2 = b.new_e2 + off;
  double* nd2 = b.new_d2 + off;
  double* nx = sc.smooth ? b.new_x + 4 * (size_t)off : nullptr;
  for (uint32_t k = 1; k < nn; ++k) {
    const uint32_t x = ne2[k];
    const double d = nd2[k];
    double xs[4];
    if (nx)
      for (int c = 0; c < 4; ++c) xs[c] = nx[4 * k + c];
    uint32_t q = k;
    while (q > 0 && ne2[q - 1] > x) {
      ne2[q] = ne2[q - 1];
      nd2[q] = nd2[q - 1];
      if (nx)
        for (int c = 0; c < 4; ++c) nx[4 * q + c] = nx[4 * (q - 1) + c];
      --q;
    }
    ne2[q] = x;
    nd2[q] = d;
    if (nx)
      for (int c = 0; c < 4; ++c) nx[4 * q + c] = xs[c];
  }
  uint32_t io = o0, in = 0;
  for (;;) {
    while (io < o1 && !b.pkeep[io]) ++io;
    const bool have_old = io < o1, have_new = in < nn;
    if (!have_old && !have_new) break;
    const bool take_old = have_old && (!have_new || b.pe2[0][io] < ne2[in]);
    b.pe1[1][dst] = e1;
    if (take_old) {
      b.pe2[1][dst] = b.pe2[0][io];
      b.pstick[1][dst] = b.pstick[0][io];
      b.pd2[1][dst] = b.pd2[0][io];
      for (int c = 0; c < 3; ++c) b.porig[1][3 * (size_t)dst + c] = b.porig[0][3 * (size_t)io + c];
      if (nx)
        for (int c = 0; c < 4; ++c) b.pvw[1][4 * (size_t)dst + c] = b.pvw[0][4 * (size_t)io + c];
      ++io;
    } else {
      b.pe2[1][dst] = ne2[in];
      b.pstick[1][dst] = 0;
      b.pd2[1][dst] = nd2[in];
      for (int c = 0; c < 3; ++c) b.porig[1][3 * (size_t)dst + c] = 0.0;
      if (nx)
        for (int c = 0; c < 4; ++c) b.pvw[1][4 * (size_t)dst + c] = nx[4 * in + c];
      ++in;
    }
    ++dst;
  }
}

// The new list, face by face (segments of eid1): the kept old pairs (in e2
// order already) merged with the face's new pairs sorted by e2, a new pair
// before an old one of the same e2.  One warp per face: the new pairs' keys
// (e2, index) are sorted in shared memory (bitonic), and every pair's place
// follows from ranks, an old pair's = its rank among the kept old ones + the
// new pairs of e2 <= its e2, a new pair's = its rank among the new ones + the
// kept old pairs of e2 < its e2; the same list as the serial merge, which
// takes a face with more than kAsmCap old or new pairs.
constexpr int kAsmWarps = 4;
constexpr uint32_t kAsmCap = 512;
__global__ void __launch_bounds__(32 * kAsmWarps) k_rb_assemble(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  __shared__ unsigned long long skey[kAsmWarps][kAsmCap];
  __shared__ uint32_t skept[kAsmWarps][kAsmCap + 1];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  unsigned long long* key = skey[w];
  uint32_t* kept = skept[w];
  // each warp reads the segments of 32 consecutive faces at once and merges
  // the faces that have old or new pairs, one after the other
  for (uint32_t fbase = (blockIdx.x * kAsmWarps + w) * 32; fbase < sc.F; fbase += gridDim.x * kAsmWarps * 32) {
    const uint32_t mine = fbase + lane;
    uint32_t my_o0 = 0, my_no = 0, my_nn = 0;
    if (mine < sc.F) {
      my_o0 = b.pair_ptr[0][mine];
      my_no = b.pair_ptr[0][mine + 1] - my_o0;
      my_nn = b.new_cnt[mine];
    }
    const bool big = my_nn > kAsmCap || my_no > kAsmCap;
    if (big) assemble_serial(b, sc, mine);
    unsigned todo = __ballot_sync(0xffffffffu, !big && (my_no > 0 || my_nn > 0));
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t e1 = fbase + (uint32_t)src;
      const uint32_t o0 = __shfl_sync(0xffffffffu, my_o0, src);
      const uint32_t no = __shfl_sync(0xffffffffu, my_no, src);
      const uint32_t nn = __shfl_sync(0xffffffffu, my_nn, src);
      const uint32_t dst = b.pair_ptr[1][e1];
      const uint32_t off = nn ? b.new_off[e1] : 0u;
      // the new pairs' keys, sorted
      uint32_t P = 32;
      while (P < nn) P <<= 1;
      for (uint32_t i = lane; i < P; i += 32)
        key[i] = i < nn ? ((unsigned long long)b.new_e2[off + i] << 32) | i : ~0ull;
      __syncwarp();
      if (nn > 1)
        for (uint32_t k = 2; k <= P; k <<= 1)
          for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t t = lane; t < P / 2; t += 32) {
              const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
              const unsigned long long x = key[i], y = key[i + j];
              if (((i & k) == 0) == (x > y)) {
                key[i] = y;
                key[i + j] = x;
              }
            }
            __syncwarp();
          }
      // kept old pairs before each old position (exclusive prefix count)
      uint32_t run = 0;
      for (uint32_t base = 0; base < no; base += 32) {
        const uint32_t i = base + lane;
        const bool kp = i < no && b.pkeep[o0 + i];
        const unsigned m = __ballot_sync(0xffffffffu, kp);
        if (i < no) kept[i] = run + (uint32_t)__popc(m & ((1u << lane) - 1u));
        run += (uint32_t)__popc(m);
      }
      if (lane == 0) kept[no] = run;
      __syncwarp();
      // kept old pairs
      for (uint32_t i = lane; i < no; i += 32) {
        const uint32_t io = o0 + i;
        if (!b.pkeep[io]) continue;
        const uint32_t x = b.pe2[0][io];
        uint32_t lo = 0, hi = nn;  // new pairs with e2 <= x
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if ((uint32_t)(key[mid] >> 32) <= x) lo = mid + 1;
          else hi = mid;
        }
        const uint32_t d = dst + kept[i] + lo;
        b.pe1[1][d] = e1;
        b.pe2[1][d] = x;
        b.pstick[1][d] = b.pstick[0][io];
        b.pd2[1][d] = b.pd2[0][io];
        for (int c = 0; c < 3; ++c) b.porig[1][3 * (size_t)d + c] = b.porig[0][3 * (size_t)io + c];
        if (sc.smooth)
          for (int c = 0; c < 4; ++c) b.pvw[1][4 * (size_t)d + c] = b.pvw[0][4 * (size_t)io + c];
      }
      // new pairs
      for (uint32_t r = lane; r < nn; r += 32) {
        const unsigned long long kr = key[r];
        const uint32_t x = (uint32_t)(kr >> 32), k = off + (uint32_t)(kr & 0xffffffffu);
        uint32_t lo = 0, hi = no;  // old pairs (kept or not) with e2 < x
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (b.pe2[0][o0 + mid] < x) lo = mid + 1;
          else hi = mid;
        }
        const uint32_t d = dst + r + kept[lo];
        b.pe1[1][d] = e1;
        b.pe2[1][d] = x;
        b.pstick[1][d] = 0;
        b.pd2[1][d] = b.new_d2[k];
        for (int c = 0; c < 3; ++c) b.porig[1][3 * (size_t)d + c] = 0.0;
        if (sc.smooth)
          for (int c = 0; c < 4; ++c) b.pvw[1][4 * (size_t)d + c] = b.new_x[4 * (size_t)k + c];
      }
      __syncwarp();
    }
  }
}

__global__ void k_rb_copyback(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (rb_off(ctl)) return;
  const uint32_t n = ctl->n_next;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
    b.pe1[0][j] = b.pe1[1][j];
    b.pe2[0][j] = b.pe2[1][j];
    b.pstick[0][j] = b.pstick[1][j];
    b.pd2[0][j] = b.pd2[1][j];
    for (int c = 0; c < 3; ++c) b.porig[0][3 * (size_t)j + c] = b.porig[1][3 * (size_t)j + c];
    if (sc.smooth)
      for (int c = 0; c < 4; ++c) b.pvw[0][4 * (size_t)j + c] = b.pvw[1][4 * (size_t)j + c];
  }
  for (uint32_t f = blockIdx.x * blockDim.x + threadIdx.x; f <= sc.F; f += stride) b.pair_ptr[0][f] = b.pair_ptr[1][f];
  // the last block ends the pass (every block has read its flag); a batch also
  // clears its shells' flags
  if (!last_block_rb(&ctl->cnt[10])) return;
  for (uint32_t s = threadIdx.x; s < sc.n_cs; s += blockDim.x) b.shc[s].rebuild = 0;
  if (threadIdx.x != 0) return;
  ctl->n_pairs = ctl->n_next;
  ctl->rebuild = 0;
  ctl->csr_dirty = 1;
}

// ------------------------------------------------------------ contact CSR --
__device__ __forceinline__ bool csr_off(const Ctl* ctl) { return ctl->csr_dirty == 0 || ctl->halted != 0; }

__global__ void k_csr_clear(DevBuf b, StepConst sc) {
  if (csr_off(b.ctl)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) b.ctl->cnt[9] = 0;  // k_csr_sort's list of large nodes
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < sc.V; i += stride) {
    b.csr_count[i] = 0;
    b.csr_fill[i] = 0;
  }
}

__global__ void k_csr_count(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (csr_off(ctl)) return;
  const uint32_t n = ctl->n_pairs;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
    const uint32_t e[2] = {b.pe1[0][j], b.pe2[0][j]};
    for (int r = 0; r < 6; ++r) atomicAdd(&b.csr_count[b.tri[3 * (size_t)e[r / 3] + r % 3]], 1u);
  }
}

__global__ void k_csr_fill(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (csr_off(ctl)) return;
  const uint32_t n = ctl->n_pairs;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
    const uint32_t e[2] = {b.pe1[0][j], b.pe2[0][j]};
    for (int r = 0; r < 6; ++r) {
      const uint32_t nd = b.tri[3 * (size_t)e[r / 3] + r % 3];
      const uint32_t pos = b.csr_ptr[nd] + atomicAdd(&b.csr_fill[nd], 1u);
      b.csr_ent[pos] = j * 8u + (uint32_t)r;
    }
  }
}

// Sort each node's entries (deterministic order for the gather): by one warp in
// registers up to kCsrSortCap entries (a few hundred in a contact-heavy state, up
// to about a thousand with SMOOTH contact), by a block of k_csr_sort_big in
// shared memory up to kCsrSortBigCap, in place by one thread beyond.
constexpr int kCsrSortWarps = 4;
constexpr int kCsrSortNodes = 8;  // nodes per warp
constexpr uint32_t kCsrSortCap = 1024;
constexpr uint32_t kCsrSortBigCap = 16384;
constexpr int kCsrSortBigBlock = 1024;

__device__ void csr_sort_serial(const DevBuf& b, uint32_t k0, uint32_t k1) {
  for (uint32_t k = k0 + 1; k < k1; ++k) {
    const uint32_t x = b.csr_ent[k];
    uint32_t q = k;
    while (q > k0 && b.csr_ent[q - 1] > x) {
      b.csr_ent[q] = b.csr_ent[q - 1];
      --q;
    }
    b.csr_ent[q] = x;
  }
}

// the nodes that k_csr_sort listed (in csr_fill, free after k_csr_fill; count in ctl->cnt[9])
__global__ void __launch_bounds__(kCsrSortBigBlock) k_csr_sort_big(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (csr_off(ctl)) return;
  extern __shared__ uint32_t big[];
  const uint32_t n_big = min(ctl->cnt[9], sc.V);
  for (uint32_t q = blockIdx.x; q < n_big; q += gridDim.x) {
    const uint32_t nd = b.csr_fill[q];
    const uint32_t k0 = b.csr_ptr[nd], k1 = b.csr_ptr[nd + 1];
    const uint32_t n = k1 - k0;
    if (n > kCsrSortBigCap) {
      if (threadIdx.x == 0) csr_sort_serial(b, k0, k1);
      __syncthreads();
      continue;
    }
    uint32_t P = kCsrSortCap;
    while (P < n) P <<= 1;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) big[i] = i < n ? b.csr_ent[k0 + i] : 0xffffffffu;
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1)
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {
        for (uint32_t t = threadIdx.x; t < P / 2; t += blockDim.x) {
          const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
          const uint32_t x = big[i], y = big[i + j];
          if (((i & k) == 0) == (x > y)) {
            big[i] = y;
            big[i + j] = x;
          }
        }
        __syncthreads();
      }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) b.csr_ent[k0 + i] = big[i];
    __syncthreads();
  }
  if (last_block_rb(&ctl->cnt[11]) && threadIdx.x == 0) ctl->csr_dirty = 0;
}

// Bitonic sort of n <= 32 E entries by one warp, in registers: element
// lane * E + r lies in register r of its lane, so the network's strides below E
// compare registers of one lane and the larger ones take one shuffle each.
template <int E>
__device__ __forceinline__ void warp_sort_segment(uint32_t* ent, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t x[E];
#pragma unroll
  for (int r = 0; r < E; ++r) x[r] = (uint32_t)r * 32u + lane < n ? ent[(uint32_t)r * 32u + lane] : 0xffffffffu;
  __syncwarp();
#pragma unroll
  for (int k = 2; k <= 32 * E; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j < E) {
#pragma unroll
        for (int r = 0; r < E; ++r) {
          if (r & j) continue;
          const bool up = k < E ? (r & k) == 0 : (lane & (uint32_t)(k / E)) == 0;
          const uint32_t lo = min(x[r], x[r | j]), hi = max(x[r], x[r | j]);
          x[r] = up ? lo : hi;
          x[r | j] = up ? hi : lo;
        }
      } else {
        const bool up = (lane & (uint32_t)(k / E)) == 0, first = (lane & (uint32_t)(j / E)) == 0;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const uint32_t y = __shfl_xor_sync(0xffffffffu, x[r], j / E);
          x[r] = up == first ? min(x[r], y) : max(x[r], y);
        }
      }
    }
#pragma unroll
  for (int r = 0; r < E; ++r)
    if (lane * E + r < n) ent[lane * E + r] = x[r];
  __syncwarp();
}

// One warp takes kCsrSortNodes consecutive nodes.  The sort is a chain of
// dependent compares, so it wants many warps and no shared memory: in shared
// memory, with 32 nodes per warp (8 warps per SM), a folded level-6 shell (41 k
// nodes, 250 entries each) took 1.37 ms, now 0.33; with SMOOTH contact (level 5, 630
// each) 2.15 ms, now 0.14 and 0.09 in k_csr_sort_big.
__global__ void __launch_bounds__(32 * kCsrSortWarps) k_csr_sort(DevBuf b, StepConst sc) {
  Ctl* ctl = b.ctl;
  if (csr_off(ctl)) return;
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  for (uint32_t base = (blockIdx.x * kCsrSortWarps + w) * kCsrSortNodes; base < sc.V;
       base += gridDim.x * kCsrSortWarps * kCsrSortNodes) {
    const uint32_t me = base + lane;
    uint32_t k0 = 0, n = 0;
    if (lane < kCsrSortNodes && me < sc.V) {
      k0 = b.csr_ptr[me];
      n = b.csr_ptr[me + 1] - k0;
    }
    // larger segments than the registers hold go to the list of k_csr_sort_big
    if (n > kCsrSortCap) b.csr_fill[atomicAdd(&ctl->cnt[9], 1u)] = me;
    unsigned todo = __ballot_sync(0xffffffffu, n >= 2 && n <= kCsrSortCap);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      uint32_t* ent = b.csr_ent + __shfl_sync(0xffffffffu, k0, src);
      const uint32_t sn = __shfl_sync(0xffffffffu, n, src);
      if (sn <= 32) warp_sort_segment<1>(ent, sn);
      else if (sn <= 64) warp_sort_segment<2>(ent, sn);
      else if (sn <= 128) warp_sort_segment<4>(ent, sn);
      else if (sn <= 256) warp_sort_segment<8>(ent, sn);
      else if (sn <= 512) warp_sort_segment<16>(ent, sn);
      else warp_sort_segment<32>(ent, sn);
    }
  }
}

inline uint32_t nblk(uint32_t n, uint32_t bs = kBlock) { return n == 0 ? 1 : (n + bs - 1) / bs; }

}  // namespace

constexpr size_t kSearchSmem = sizeof(SearchPool) * (kSearchBlock / 32);

// a grid that the SMs hold at once (the queue hands out the pairs)
template <bool REBUILD, bool DEEP>
static uint32_t search_grid() {
  static const uint32_t g = [] {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_smooth_search<REBUILD, DEEP>, kSearchBlock, kSearchSmem);
    return (uint32_t)(sms > 0 ? sms : 152) * (uint32_t)(per_sm > 0 ? per_sm : 1);
  }();
  return g;
}

template <bool REBUILD, bool DEEP>
static void launch_search(const DevBuf& b, const StepConst& sc, cudaStream_t s) {
  k_smooth_search<REBUILD, DEEP><<<search_grid<REBUILD, DEEP>(), kSearchBlock, kSearchSmem, s>>>(b, sc);
}

void launch_smooth_search(const DevBuf& b, const StepConst& sc, bool rebuild, cudaStream_t s) {
  uint32_t g = nblk(sc.F);
  if (g > 8 * 152) g = 8 * 152;
  if (sc.F > sc.irr_first && g < 152) g = 152;  // the irregular children, hundreds per face
  k_limit_coeffs<<<g, kBlock, 0, s>>>(b, sc, rebuild);
  const bool deep = sc.irr_levels < SHL_SMOOTH_LEVELS;
  if (rebuild)
    deep ? launch_search<true, true>(b, sc, s) : launch_search<true, false>(b, sc, s);
  else
    deep ? launch_search<false, true>(b, sc, s) : launch_search<false, false>(b, sc, s);
}

// kernels that take more than the default 48 KB of shared memory; called once
// per device before their first launch
cudaError_t init_contact_kernels() {
  const auto set = [](const void* f, size_t bytes) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  cudaError_t e = set((const void*)k_rb_narrow, sizeof(PairWork));
  if (e == cudaSuccess) e = set((const void*)k_csr_sort_big, kCsrSortBigCap * 4);
  if (e == cudaSuccess) e = set((const void*)k_smooth_search<true, true>, kSearchSmem);
  if (e == cudaSuccess) e = set((const void*)k_smooth_search<true, false>, kSearchSmem);
  if (e == cudaSuccess) e = set((const void*)k_smooth_search<false, true>, kSearchSmem);
  if (e == cudaSuccess) e = set((const void*)k_smooth_search<false, false>, kSearchSmem);
  return e;
}

void launch_contact_csr(const DevBuf& b, const StepConst& sc, cudaStream_t s) {
  const uint32_t gV = nblk(sc.V);
  uint32_t gP = nblk(sc.pairs_cap);
  if (gP > 8 * 152) gP = 8 * 152;
  k_csr_clear<<<gV, kBlock, 0, s>>>(b, sc);
  k_csr_count<<<gP, kBlock, 0, s>>>(b, sc);
  launch_scan(&b.ctl->csr_dirty, b.ctl, b.csr_count, b.csr_ptr, nullptr, sc.V, sc.V, b.scan_block, &b.ctl->n_csr,
              true, sc.csr_cap, true, s);
  k_csr_fill<<<gP, kBlock, 0, s>>>(b, sc);
  {
    const uint32_t g = std::min((sc.V + kCsrSortNodes * kCsrSortWarps - 1) / (kCsrSortNodes * kCsrSortWarps), 16u * 152u);
    k_csr_sort<<<g ? g : 1, 32 * kCsrSortWarps, 0, s>>>(b, sc);
    k_csr_sort_big<<<152, kCsrSortBigBlock, kCsrSortBigCap * 4, s>>>(b, sc);
  }
}

void launch_rebuild(const DevBuf& b, const StepConst& sc, cudaStream_t s) {
  const uint32_t gF = nblk(sc.F);
  k_rb_aabb<<<gF, kBlock, 0, s>>>(b, sc);
  if (!sc.n_cs) k_rb_bounds<<<kBoundsBlocks, kBlock, 0, s>>>(b, sc, gF);
  if (sc.n_cs) {
    k_rb_grids<<<sc.n_cs, SHL_SUM_LANES, 0, s>>>(b, sc);
    k_rb_grid_scan<<<1, 1024, 0, s>>>(b, sc);
  }
  {
    uint32_t g = nblk(sc.n_cells_cap > sc.F ? sc.n_cells_cap : sc.F);
    if (g > 16 * 152) g = 16 * 152;
    k_rb_clear<<<g, kBlock, 0, s>>>(b, sc);
  }
  const bool wide = sc.F <= kWideFaces;
  const uint32_t g_cells = std::min<uint32_t>(nblk(sc.F * (wide ? 32u : 8u)), 16 * 152);
  {
    uint32_t g = nblk(sc.pairs_cap) > g_cells ? nblk(sc.pairs_cap) : g_cells;
    if (g > 16 * 152) g = 16 * 152;
    if (wide)
      k_rb_count<32><<<g, kBlock, 0, s>>>(b, sc);
    else
      k_rb_count<1><<<g, kBlock, 0, s>>>(b, sc);
  }
  launch_scan(&b.ctl->rebuild, b.ctl, b.cell_count, b.cell_start, &b.ctl->n_cells, 0, sc.n_cells_cap, b.scan_block,
              &b.ctl->n_entries, false, sc.entries_cap, true, s);
  if (wide)
    k_rb_fill<32><<<g_cells, kBlock, 0, s>>>(b, sc);
  else
    k_rb_fill<8><<<g_cells, kBlock, 0, s>>>(b, sc);
  {
    uint32_t g = nblk(sc.entries_cap);
    if (g > 16 * 152) g = 16 * 152;
    k_rb_cand<<<g, kCandBlock, 0, s>>>(b, sc);
    uint32_t gc = nblk(sc.cand_cap);
    if (gc > 16 * 152) gc = 16 * 152;
    if (sc.smooth)
      launch_smooth_search(b, sc, true, s);
    else
      k_rb_narrow<<<gc, kBlock, sizeof(PairWork), s>>>(b, sc);
    launch_scan(&b.ctl->rebuild, b.ctl, b.new_cnt, b.new_off, nullptr, sc.F, sc.F, b.scan_block, &b.ctl->n_new,
                false, sc.pairs_cap, true, s);
    k_rb_scatter_new<<<gc, kBlock, 0, s>>>(b, sc);
  }
  launch_scan(&b.ctl->rebuild, b.ctl, b.seg_count, b.pair_ptr[1], nullptr, sc.F, sc.F, b.scan_block, &b.ctl->n_next,
              true, sc.pairs_cap, true, s);
  {
    uint32_t g = (sc.F + 32 * kAsmWarps - 1) / (32 * kAsmWarps);
    if (g > 16 * 152) g = 16 * 152;
    k_rb_assemble<<<g ? g : 1, 32 * kAsmWarps, 0, s>>>(b, sc);
  }
  {
    uint32_t g = nblk(sc.pairs_cap > sc.F + 1 ? sc.pairs_cap : sc.F + 1);
    if (g > 8 * 152) g = 8 * 152;
    k_rb_copyback<<<g, kBlock, 0, s>>>(b, sc);
  }
  launch_contact_csr(b, sc, s);
}

}  // namespace shl
