// A whole PCG solve as one persistent kernel: one CTA per SM, each owning a
// run of matrix chunks (fem_asm.cu) and their rows; the phases of an
// iteration are separated by grid-wide barriers instead of kernel
// boundaries.
//
//   A   z = S r + P y_c, p = z + beta p, q = K p, p.q           | barrier
//   B   x += alpha p, r -= alpha q, ||r||^2, S r, r.S r, shares
//       of P^T r                                               | barrier
//   C1  r_c                                                    | barrier
//   C2  y_c = Ac^-1 r_c, r_c.y_c                               | barrier
//
// (r.z = r.S r + r_c.y_c, so no phase of its own forms z before beta is known.
// A small coarse space: every CTA adds up r_c itself, no barrier after C1.)
// (Jacobi: A and B with z = D^-1 r.)  The sums are FP64 in a fixed order and
// the stopping tests those of the kernel chain; the scalars differ from the
// chain's in rounding (its r.z is one sum over z, and its q comes by
// recurrence).
//
// What bounds it: up to some 65,000 rows (a coarse space of full rows) the
// matrix stays in shared memory for the whole solve and the phases' latencies
// are left: 2,700 cycles per barrier and about 2,500 of dependent loads and sums
// per phase, 35,000 cycles (18 us) an iteration at 16,000 rows against 30 us
// for the chain's seven kernels (42,000 with z in a phase of its own, a barrier
// more, and one warp per slice).  At 121,000 rows and 4-voxel cells the planes,
// tables and rings take all of it: the matrix (55 MB) and the packed BF16
// coarse inverse (61 MB) stream once per iteration, 72 MB of that from HBM
// (half of the sectors hit L2), 81,000 cycles (42 us) against 70 us, HBM 21 %
// and L2 17 % busy.  All 128 registers are in use: loads held over a barrier
// beyond those of A spill and cost more than they hide (the first row of C2:
// 92,000 cycles).
//
// The reference factorises the assembled tangent on the host
// (backend/fea/fem/solver/static_solver.py:399-462).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>

#include "fem_bulk.cuh"
#include "fem_lattice.cuh"
#include "fem_pcg.h"

namespace femb200 {

// ───────────────────────── tables (host) ─────────────────────────

bool pcg_coarse_tables(const std::vector<int>& cta_row, const std::vector<int>& halo_ptr,
                       const std::vector<int>& halo, const std::vector<int>& node_cell,
                       const std::vector<int>& cell_corner, int n_cn, int parts, PcgCoarseHost* o) {
  const int G = (int)cta_row.size() - 1, Nn = cta_row[G], n_dof = 3 * n_cn, nb = (n_dof + 63) / 64;
  std::vector<std::vector<int>> tabs(G, std::vector<int>(kTabWords, 0));
  // a list of CTA g: its place in the header words and its length
  auto put = [&](int g, int word, const std::vector<int>& v) {
    tabs[g][word] = (int)tabs[g].size();
    tabs[g].insert(tabs[g].end(), v.begin(), v.end());
  };
  // Per CTA: its rows by cell (segments), and the coarse nodes that its columns
  // (its rows, then its halo) interpolate from, ascending, so that neighbouring
  // threads read neighbouring words of y_c.  By distinct cell, of which a CTA
  // has few: sorting the rows and looking up every column's corners took 6 ms
  // on one core at 51,000 rows, this 2.
  const int n_cells = (int)(cell_corner.size() / 8);
  std::vector<std::vector<int>> shares(n_cn), loc(G);
  o->seg_rows.resize(Nn);
  o->col_corners.resize((size_t)Nn + halo.size());
  std::vector<int> cell_at(n_cells, -1), cell_rows(n_cells, 0), local(n_cn, -1), cells, lg, sptr;
  std::vector<uint4> cell_cc(n_cells);
  for (int g = 0; g < G; ++g) {
    const int r0 = cta_row[g], r1 = cta_row[g + 1], nh = halo_ptr[g + 1] - halo_ptr[g];
    const int* hal = halo.data() + halo_ptr[g];
    cells.clear();
    for (int r = r0; r < r1; ++r) {
      const int c = node_cell[r];
      if (cell_at[c] != g) {
        cell_at[c] = g;
        cell_rows[c] = 0;
        cells.push_back(c);
      }
      ++cell_rows[c];
    }
    std::sort(cells.begin(), cells.end());
    const size_t row_cells = cells.size();
    sptr.assign(1, 0);
    tabs[g][TAB_SEG0] = o->n_seg;
    tabs[g][TAB_SROW] = r0;
    for (int c : cells) {
      for (int q = 0; q < 8; ++q) shares[cell_corner[8 * (size_t)c + q]].push_back(o->n_seg * 8 + q);
      const int at = sptr.back();
      sptr.push_back(at + cell_rows[c]);
      cell_rows[c] = at;  // from here on the place of the cell's next row
      ++o->n_seg;
    }
    for (int r = r0; r < r1; ++r) o->seg_rows[r0 + cell_rows[node_cell[r]]++] = r;
    tabs[g][TAB_NSEG] = (int)row_cells;
    put(g, TAB_SPTR, sptr);
    for (int k = 0; k < nh; ++k) {
      const int c = node_cell[hal[k]];
      if (cell_at[c] != g) {
        cell_at[c] = g;
        cells.push_back(c);
      }
    }
    lg.clear();
    for (int c : cells)
      for (int q = 0; q < 8; ++q) {
        int& l = local[cell_corner[8 * (size_t)c + q]];
        if (l < 0) {
          l = 0;
          lg.push_back(cell_corner[8 * (size_t)c + q]);
        }
      }
    if (lg.size() > 65536) return false;
    std::sort(lg.begin(), lg.end());
    for (size_t k = 0; k < lg.size(); ++k) local[lg[k]] = (int)k;
    for (int c : cells) {
      uint32_t idx[8];
      for (int q = 0; q < 8; ++q) idx[q] = (uint32_t)local[cell_corner[8 * (size_t)c + q]];
      cell_cc[c] = make_uint4(idx[0] | idx[1] << 16, idx[2] | idx[3] << 16, idx[4] | idx[5] << 16, idx[6] | idx[7] << 16);
    }
    uint4* cc = o->col_corners.data() + r0 + halo_ptr[g];
    for (int r = r0; r < r1; ++r) *cc++ = cell_cc[node_cell[r]];
    for (int k = 0; k < nh; ++k) *cc++ = cell_cc[node_cell[hal[k]]];
    for (int n : lg) local[n] = -1;
    tabs[g][TAB_NLOC] = (int)lg.size();
    put(g, TAB_LOC, lg);
    o->max_loc = std::max(o->max_loc, (int)lg.size());
    loc[g] = lg;
  }
  // the shares of a coarse node lie together: each share's place
  std::vector<int> place(8 * (size_t)o->n_seg);
  o->cn_ptr.assign(1, 0);
  for (int c = 0, at = 0; c < n_cn; ++c) {
    for (int j : shares[c]) place[j] = at++;
    o->cn_ptr.push_back(at);
  }
  for (int g = 0; g < G; ++g) {
    const int c0 = (int)((int64_t)n_cn * g / G), c1 = (int)((int64_t)n_cn * (g + 1) / G);
    tabs[g][TAB_CN0] = c0;
    tabs[g][TAB_NCN] = c1 - c0;
    put(g, TAB_CPTR, std::vector<int>(o->cn_ptr.begin() + c0, o->cn_ptr.begin() + c1 + 1));
    const size_t s0 = 8 * (size_t)tabs[g][TAB_SEG0], n8 = 8 * (size_t)tabs[g][TAB_NSEG];
    put(g, TAB_SPOS, std::vector<int>(place.begin() + s0, place.begin() + s0 + n8));
  }
  if (parts) {
    // tiles in super-blocks of about one CTA's share, so that a CTA touches
    // few row blocks; cut into equal runs
    const int64_t n_tiles = (int64_t)nb * (nb + 1) / 2;
    int sb = 1;
    while ((int64_t)(sb + 1) * (sb + 1) <= (n_tiles + G - 1) / G + sb) ++sb;
    std::vector<int2> order;
    order.reserve((size_t)n_tiles);
    const int T = (nb + sb - 1) / sb;
    for (int bi = 0; bi < T; ++bi)
      for (int bj = 0; bj <= bi; ++bj)
        for (int I = bi * sb; I < std::min(nb, (bi + 1) * sb); ++I)
          for (int J = bj * sb; J < std::min(I + 1, (bj + 1) * sb); ++J) order.push_back(make_int2(I, J));
    std::vector<std::vector<int>> yparts(nb);
    for (int g = 0; g < G; ++g) {
      const size_t t0 = (size_t)(n_tiles * g / G), t1 = (size_t)(n_tiles * (g + 1) / G);
      std::map<int, int> lb;
      for (size_t t = t0; t < t1; ++t) {
        lb.emplace(order[t].x, 0);
        lb.emplace(order[t].y, 0);
      }
      int k = 0;
      for (auto& kv : lb) kv.second = k++;
      std::vector<std::vector<int>> outs(k);
      std::vector<int> tl, blk, optr(1, 0), olist;
      for (size_t t = t0; t < t1; ++t) {
        const int I = order[t].x, J = order[t].y, lt = (int)(t - t0);
        const int li = lb[I], lj = lb[J];
        tl.push_back(I * (I + 1) / 2 + J);
        tl.push_back(li | (lj << 16));
        outs[li].push_back((1 + parts) * lt);
        if (I != J)
          for (int h = 1; h <= parts; ++h) outs[lj].push_back((1 + parts) * lt + h);
      }
      tabs[g][TAB_BLK0] = o->n_parts;
      for (auto& kv : lb) {
        yparts[kv.first].push_back(o->n_parts++);
        blk.push_back(kv.first);
        olist.insert(olist.end(), outs[kv.second].begin(), outs[kv.second].end());
        optr.push_back((int)olist.size());
      }
      tabs[g][TAB_NT] = (int)(t1 - t0);
      tabs[g][TAB_NL] = k;
      put(g, TAB_TILES, tl);
      put(g, TAB_BLK, blk);
      put(g, TAB_OPTR, optr);
      put(g, TAB_OLIST, olist);
      o->max_lblk = std::max(o->max_lblk, k);
      o->max_tiles = std::max(o->max_tiles, (int)(t1 - t0));
    }
    for (int g = 0; g < G; ++g) {
      std::map<int, int> at;
      std::vector<int> yidx, yptr(1, 0), ylist;
      for (int cn : loc[g])
        for (int d = 0; d < 3; ++d) {
          const int dof = 3 * cn + d, blk = dof >> 6;
          if (at.emplace(blk, (int)yptr.size() - 1).second) {
            ylist.insert(ylist.end(), yparts[blk].begin(), yparts[blk].end());
            yptr.push_back((int)ylist.size());
          }
          yidx.push_back(at[blk] << 6 | (dof & 63));
        }
      put(g, TAB_YIDX, yidx);
      put(g, TAB_YPTR, yptr);
      put(g, TAB_YLIST, ylist);
    }
  }
  o->tab_ptr.assign(1, 0);
  for (int g = 0; g < G; ++g) {
    while (tabs[g].size() % 4) tabs[g].push_back(0);
    o->tab.insert(o->tab.end(), tabs[g].begin(), tabs[g].end());
    o->tab_ptr.push_back((int)o->tab.size());
    o->max_tab = std::max(o->max_tab, (int)tabs[g].size());
  }
  return true;
}

// ───────────────────────── kernel ─────────────────────────

namespace {

constexpr int kWarps = kPcgThreads / 32;

// This CTA's sum of v over its threads, in thread 0.
__device__ __forceinline__ double cta_sum(double v, double* sred) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < kWarps ? sred[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  return t;
}

// The same for two sums at once.
__device__ __forceinline__ void cta_sum2(double& v, double& w, double* sv, double* sw) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_down_sync(0xffffffffu, v, o);
    w += __shfl_down_sync(0xffffffffu, w, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = v;
    sw[threadIdx.x >> 5] = w;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < kWarps ? sv[threadIdx.x] : 0.0;
    w = threadIdx.x < kWarps ? sw[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1) {
      v += __shfl_down_sync(0xffffffffu, v, o);
      w += __shfl_down_sync(0xffffffffu, w, o);
    }
  }
}

// Grid-wide barrier number `epoch` (1, 2, ...): every CTA's earlier writes
// are visible to all after it.  Bounded: false if the others did not arrive
// within some seconds.  (About 2,700 cycles with 148 CTAs; 1,860 of them are
// the arrivals' and the polls' round trips, the rest the writes' way to L2.
// Polling every CTA's tagged post instead of one counter took 10,000, a
// leader that gathers and broadcasts 5,000, clusters in front 4,500.)
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int epoch) {
  bool ok = true;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int want = epoch * gridDim.x;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    ok = false;
    for (int i = 0; i < (1 << 23); ++i) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - want) >= 0) {
        ok = true;
        break;
      }
    }
  }
  return __syncthreads_and(ok) != 0;
}

// Grid-wide sums: thread 0 of every CTA stores its share before a barrier;
// after it each thread reads one share (sum_load, issued with the phase's
// other loads), and sum_end adds them in the same order in every CTA.
__device__ __forceinline__ double sum_load(const double* slot) {
  double t = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kPcgThreads) t += __ldcg(slot + i);
  return t;
}

__device__ __forceinline__ double sum_end(double t, double* sred) {
  const int nw = min(kWarps, ((int)gridDim.x + 31) >> 5);
  if ((int)(threadIdx.x >> 5) < nw) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = t;
  }
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < nw; ++w) s += sred[w];
  return s;
}

__device__ __forceinline__ void tile_row(const uint4 w, float a[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 f = __bfloat1622float2(h[k]);
    a[2 * k] = f.x;
    a[2 * k + 1] = f.y;
  }
}

// x as three BF16 parts: x = hi + mid + lo to FP32's 24 bits.
__device__ __forceinline__ void split3(float x, __nv_bfloat16 (&p)[3]) {
  p[0] = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(p[0]);
  p[1] = __float2bfloat16_rn(r);
  p[2] = __float2bfloat16_rn(r - __bfloat162float(p[1]));
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The sum of an accumulator's columns 0..2 (the three parts of x), rows
// lane / 4 and lane / 4 + 8, in the lanes with lane % 4 == 0.
__device__ __forceinline__ void mma_rowsum(const float (&c)[4], float& lo, float& hi) {
  lo = c[0] + c[1] + __shfl_down_sync(0xffffffffu, c[0], 1);
  hi = c[2] + c[3] + __shfl_down_sync(0xffffffffu, c[2], 1);
}

// 32 rows of a 64 x 64 BF16 tile (a 4 KB part in shared memory) by one warp:
// u = A xj for those rows, v = A^T xi over them, on the tensor cores with x's
// three parts as columns 0..2 of B (exact products, FP32 sums): 16 MMAs
// where the FMA form took 19,000 cycles per 50 tiles of a CTA.  xj3 / xi3:
// the parts of x, [3][64] BF16 of the column block, [3][64] of the row block
// at this part's first row.
__device__ __forceinline__ void tile_part16(const unsigned char* part, const __nv_bfloat16* xj3,
                                            const __nv_bfloat16* xi3, float* u_out, float* v_out) {
  const int lane = threadIdx.x & 31, n = lane >> 2, k2 = 2 * (lane & 3);
  const uint32_t base = bulk::smem_addr(part);
  // B fragments: column n of x (zero for n > 2), rows k2, k2 + 1 and + 8
  uint32_t bj[4][2], bi[2][2];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      bj[s][h] = n < 3 ? *reinterpret_cast<const uint32_t*>(xj3 + 64 * n + 16 * s + 8 * h + k2) : 0u;
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      bi[s][h] = n < 3 ? *reinterpret_cast<const uint32_t*>(xi3 + 64 * n + 16 * s + 8 * h + k2) : 0u;
  // u: rows 16 m .. + 15, columns 16 s .. + 15 (all fragments in flight)
  {
    uint32_t f[2][4][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const uint32_t row = (uint32_t)(16 * m + (lane & 15)), chunk = (uint32_t)(2 * s + (lane >> 4));
        ldsm4(f[m][s], base + 128u * row + 16u * (chunk ^ (row & 7u)));
      }
    float c[2][4] = {};
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int m = 0; m < 2; ++m) mma16816(c[m], f[m][s], bj[s][0], bj[s][1]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      float lo, hi;
      mma_rowsum(c[m], lo, hi);
      if ((lane & 3) == 0) {
        u_out[16 * m + n] = lo;
        u_out[16 * m + n + 8] = hi;
      }
    }
  }
  // v: columns 16 m .. + 15 (rows of A^T), rows 16 s .. + 15 of the part;
  // transposed 8 x 8 blocks: (cols 0-7, rows 0-7), (cols 8-15, rows 0-7),
  // (cols 0-7, rows 8-15), (cols 8-15, rows 8-15)
  {
    uint32_t f[4][2][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const uint32_t row = (uint32_t)(16 * s + (lane & 7) + 8 * (lane >> 4));
        const uint32_t chunk = (uint32_t)(2 * m + ((lane >> 3) & 1));
        ldsm4t(f[m][s], base + 128u * row + 16u * (chunk ^ (row & 7u)));
      }
    float c[4][4] = {};
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int m = 0; m < 4; ++m) mma16816(c[m], f[m][s], bi[s][0], bi[s][1]);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float lo, hi;
      mma_rowsum(c[m], lo, hi);
      if ((lane & 3) == 0) {
        v_out[16 * m + n] = lo;
        v_out[16 * m + n + 8] = hi;
      }
    }
  }
}

// 16 rows of a 64 x 64 FP32 tile (a 4 KB part) by one warp: u = A xj for
// those rows, v = A^T xi over them.  Lane l covers columns 8 (l % 8) .. + 7 of
// rows 4 k + l / 8; the sums are completed by reduce-scatters over the lanes
// of a row and of a column group.
__device__ __forceinline__ void tile_part32(const unsigned char* part, const float* xj, const float* xi, float* u_out,
                                            float* v_out) {
  const int lane = threadIdx.x & 31, q = lane >> 3, cg8 = lane & 7;
  float x8[8], v[8], u[4];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x8[k] = xj[8 * cg8 + k];
    v[k] = 0.f;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4* A = reinterpret_cast<const float4*>(part) + (4 * k + q) * 16 + 2 * cg8;
    const float4 f0 = A[0], f1 = A[1];
    const float a[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
    const float xr = xi[4 * k + q];
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      s += a[e] * x8[e];
      v[e] += a[e] * xr;
    }
    u[k] = s;
  }
#pragma unroll
  for (int o = 4, w = 2; w >= 1; o >>= 1, w >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const float send = up ? u[k] : u[k + w];
      const float keep = up ? u[k + w] : u[k];
      u[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  u[0] += __shfl_xor_sync(0xffffffffu, u[0], 1);
  if ((cg8 & 1) == 0) u_out[4 * (cg8 >> 1) + q] = u[0];
#pragma unroll
  for (int o = 16, w = 4; o >= 8; o >>= 1, w >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const float send = up ? v[k] : v[k + w];
      const float keep = up ? v[k + w] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  reinterpret_cast<float2*>(v_out)[4 * cg8 + q] = make_float2(v[0], v[1]);
}

}  // namespace

template <bool TL>
__global__ void __launch_bounds__(kPcgThreads, 1) pcg_kernel(const __grid_constant__ PcgArgs a) {
  extern __shared__ __align__(128) unsigned char s_dyn[];
  // per warp: its ring stages, then its resident slices
  __shared__ __align__(8) uint64_t bars[3 * kWarps];
  __shared__ double sred[2][kWarps], ssum[3][kWarps];
  float* scratch = reinterpret_cast<float*>(s_dyn + a.mat_bytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = (int)gridDim.x, g = (int)blockIdx.x;
  // static words: first steps of the slices, halo nodes, coarse tables
  int* s_step = reinterpret_cast<int*>(s_dyn + a.mat_bytes + a.scratch_bytes);
  int* s_halo = s_step + a.as.max_slices + 1;
  int* tab = s_halo + a.as.max_halo;
  uint2* s_items = reinterpret_cast<uint2*>(s_dyn + a.mat_bytes + a.scratch_bytes + a.items_off);
  const int sl0 = a.as.cta_slice[g], nsl = a.as.cta_slice[g + 1] - sl0;
  const int nh = a.as.halo_ptr[g + 1] - a.as.halo_ptr[g];
  for (int k = tid; k <= nsl; k += kPcgThreads) s_step[k] = a.as.slice_step[sl0 + k];
  for (int k = tid; k < nh; k += kPcgThreads) s_halo[k] = a.as.halo[a.as.halo_ptr[g] + k];
  if (TL)
    for (int k = a.t.tab_ptr[g] + tid; k < a.t.tab_ptr[g + 1]; k += kPcgThreads) tab[k - a.t.tab_ptr[g]] = a.t.tab[k];
  if (tid == 0) {
    for (int k = 0; k < 3 * kWarps; ++k) bulk::bar_init(&bars[k], 1);
    bulk::bar_init_fence();
  }
  __syncthreads();
  const int row0 = a.as.cta_row[g], row1 = a.as.cta_row[g + 1], nrow = row1 - row0;
  const bool tiles = TL && a.c.full_ld == 0;
  const int nt = tiles ? tab[TAB_NT] : 0;
  unsigned int epoch = 0;
  bool ok = true;
  float4 *r4 = reinterpret_cast<float4*>(a.r), *x4 = reinterpret_cast<float4*>(a.x);
  float4 *p4 = reinterpret_cast<float4*>(a.p), *q4 = reinterpret_cast<float4*>(a.q);
  float4 *z4 = reinterpret_cast<float4*>(a.z), *pn4 = reinterpret_cast<float4*>(a.p2);
  const float4* d4 = reinterpret_cast<const float4*>(a.dinv);
  const float4* o4 = reinterpret_cast<const float4*>(a.boff);

  // This warp's items: slices warp, warp + 16, ... of the CTA (those below
  // a.resident stay in shared memory) in pieces of kPcgPiece steps, then the
  // 4 KB parts of the CTA's tiles (parts warp, warp + 16, ...).  The streamed
  // ones come through the warp's ring in that order, iteration after
  // iteration, each copy issued when its stage is free again: the memory
  // pipe works through the phases that read no matrix, too.
  const int res = min(a.resident, nsl), ns = a.stages;
  const int pshift = a.c.Ainv16 ? 1 : 2, parts = 1 << pshift;  // parts of a tile
  const unsigned char* tile_base = a.c.Ainv16 ? reinterpret_cast<const unsigned char*>(a.c.Ainv16)
                                              : reinterpret_cast<const unsigned char*>(a.c.Ainv32t);
  unsigned char* ring = s_dyn + a.res_bytes + (size_t)warp * ns * a.stage_bytes;
  uint64_t* bar = bars + 3 * warp;
  // the warp's list of streamed items: the first step and the bytes of a piece
  // of the matrix, or the index of a 4 KB tile part and 0
  uint2* items = s_items + (size_t)warp * a.max_items;
  int n_items = 0, n_mat = 0;
  {
    for (int s = warp; s < nsl; s += kWarps)
      if (s >= res)
        for (int t = s_step[s]; t < s_step[s + 1]; t += kPcgPiece) {
          const int n = min(kPcgPiece, s_step[s + 1] - t);
          if (lane == 0) items[n_items] = make_uint2((uint32_t)t, (uint32_t)(n * kAsmStepBytes));
          ++n_items;
        }
    n_mat = n_items;
    for (int k = warp; k < nt * parts; k += kWarps) {
      const int id = (tab + tab[TAB_TILES])[2 * (k >> pshift)];
      if (lane == 0) items[n_items] = make_uint2((uint32_t)id * parts + (k & (parts - 1)), 0u);
      ++n_items;
    }
    __syncwarp();
  }
  const bool any = n_items > 0;
  const uint64_t pol_mat = bulk::policy_evict_last(), pol_tile = bulk::policy_evict_first();
  // the next item to copy (the initial residual has no A phase: its items
  // start at the tiles) and its stage; the next stage to take and its parity
  int inext = n_mat, istage = 0, tstage = 0;
  uint32_t tparity = 0;
  auto issue = [&]() {
    if (lane == 0) {
      if (inext >= n_items) inext = 0;
      const uint2 it = items[inext];
      unsigned char* dst = ring + (size_t)istage * a.stage_bytes;
      if (it.y)
        bulk::load_hint(dst, a.as.words + (size_t)it.x * kAsmStepWords, it.y, bar + istage, pol_mat);
      else
        bulk::load_hint(dst, tile_base + 4096 * (size_t)it.x, 4096u, bar + istage, pol_tile);
      ++inext;
      if (++istage == ns) istage = 0;
    }
  };
  // the stage of the next streamed item, when it has landed
  auto take = [&]() {
    ok = bulk::wait(bar + tstage, tparity) && ok;
    unsigned char* buf = ring + (size_t)tstage * a.stage_bytes;
    if (++tstage == ns) {
      tstage = 0;
      tparity ^= 1u;
    }
    return buf;
  };
  bool loaded = false;   // this warp has waited for its resident slices
  uint32_t total = 0;    // bytes of those it copies itself
  {
    for (int s = warp; s < res; s += kWarps) total += (uint32_t)((s_step[s + 1] - s_step[s]) * kAsmStepBytes);
    if (total > 0 && lane == 0) {
      bulk::expect(bar + 2, total);
      for (int s = warp; s < res; s += kWarps)
        if (s_step[s + 1] > s_step[s])
          bulk::copy(s_dyn + (size_t)(s_step[s] - s_step[0]) * kAsmStepBytes,
                     a.as.words + (size_t)s_step[s] * kAsmStepWords,
                     (uint32_t)((s_step[s + 1] - s_step[s]) * kAsmStepBytes), bar + 2);
    }
    if (any)
      for (int k = 0; k < ns; ++k) issue();
  }

  double rz = 0.0, nrz = 0.0, rr0 = 0.0, tol2 = 0.0, rr = 0.0, pAp = 0.0, alpha = 0.0, beta = 0.0;
  bool first = true;  // the iteration after the initial residual: beta = 0, the old p and q are not read
  int iter = 0, done = 0, status = 0;
  double *part_a = a.part, *part_b = a.part + G, *part_d = a.part + 2 * G, *part_e = a.part + 3 * G;
  // this CTA's share of a sum (thread 0 stores it)
  auto post = [&](double* slot, double v, double* sh) {
    const double t = cta_sum(v, sh);
    if (tid == 0) slot[g] = t;
  };

  // lattice coordinates of the rows of three of the CTA's segments
  constexpr int kSegs = 3;
  float4 lt[kSegs];
  const int nseg = TL ? tab[TAB_NSEG] : 0;
  const int* sptr = TL ? tab + tab[TAB_SPTR] : nullptr;
  const float4* lat = TL ? a.t.seg_lat + tab[TAB_SROW] : nullptr;
  auto seg_load = [&](int s0) {
#pragma unroll
    for (int u = 0; u < kSegs; ++u) {
      const int s = s0 + u * kWarps, j = s < nseg ? sptr[s] + lane : 0;
      lt[u] = s < nseg && j < sptr[s + 1] ? __ldg(lat + j) : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    }
  };

  // The operands of this thread's first kCols columns of A, loaded under the
  // barrier in front of it: S r, the old p, and (two levels) the lattice
  // coordinates, the corners' places in s_yc and the fixed bits
  constexpr int kCols = TL ? 2 : 4;
  const int nc = nrow + nh, col0 = row0 + a.as.halo_ptr[g];
  float4 zv[kCols], pv[kCols], lv[kCols];
  uint4 cv[kCols];
  int fv[kCols];
  auto col_load = [&](int i0, const float4* pold, bool no_p) {
#pragma unroll
    for (int u = 0; u < kCols; ++u) {
      const int i = i0 + u * kPcgThreads;
      if (i < nc) {
        const int n = i < nrow ? row0 + i : s_halo[i - nrow];
        zv[u] = z4[n];
        pv[u] = no_p ? make_float4(0.f, 0.f, 0.f, 0.f) : pold[n];
        if (TL) {
          lv[u] = __ldg(a.c.node_lat + n);
          cv[u] = __ldg(a.t.col_corners + col0 + i);
          fv[u] = (int)a.m.fixed[n];
        }
      }
    }
  };
  // B: rows of this thread
  constexpr int kRows = 1;
  float *px = scratch, *py = px + a.as.max_cols, *pz = py + a.as.max_cols;
  float4 rv[kRows], xv[kRows], dv[kRows], ov[kRows];
  auto row_load = [&](int i0, bool init) {
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int n = row0 + i0 + u * kPcgThreads;
      if (n < row1) {
        if (!init) {
          rv[u] = r4[n];
          xv[u] = x4[n];
        }
        dv[u] = d4[n];
        ov[u] = o4 ? o4[n] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  };
  // Few slices: 2^split warps share the steps of one (a lone warp walks a
  // row's entries one dependent load after another: 4,800 cycles for a slice
  // that takes 1,000 of the SM's shared-memory time)
  int split = 0;
  if (res == nsl && nsl > 0)
    while (nsl << (split + 1) <= kWarps) ++split;
  float* s_split = scratch + 3 * a.as.max_cols + (TL ? 4 * a.t.max_loc : 0);  // [kWarps][3][32]

  for (bool init = true;; init = false) {
    if (!init) {
      // ── A: z = S r + P y_c, p = z + beta p, q = K p ──
      // The CTA's columns of p (its rows, then its halo) go to shared memory
      // as three planes (gathering z by 16-byte loads per entry took 32 L1
      // cycles a warp, 34,000 cycles a product at 820 rows per CTA); the
      // rows' p also to the other buffer: neighbours still read the old one.
      // Every CTA forms z and p of its halo itself, from the same operands in
      // the same order as their owner: a sixth phase with its barrier cost
      // more (5,000 cycles) than the halo's interpolation.
      const float4* po4 = p4;
      p4 = pn4;
      pn4 = const_cast<float4*>(po4);
      const double lz = sum_load(part_d) + (TL ? sum_load(part_e) : 0.0);
      float *sx = scratch, *sy = sx + a.as.max_cols, *sz = sy + a.as.max_cols;
      float4* s_yc = reinterpret_cast<float4*>(sz + a.as.max_cols);  // y_c of the coarse nodes these columns use
      if (TL) {
        if (a.c.full_ld) {
          const int* loc = tab + tab[TAB_LOC];
          for (int k = tid; k < 3 * tab[TAB_NLOC]; k += kPcgThreads)
            reinterpret_cast<float*>(s_yc + k / 3)[k % 3] = __ldcg(a.c.yc + 3 * loc[k / 3] + k % 3);
        } else {
          const int *yidx = tab + tab[TAB_YIDX], *yptr = tab + tab[TAB_YPTR], *ylist = tab + tab[TAB_YLIST];
          for (int k = tid; k < 3 * tab[TAB_NLOC]; k += kPcgThreads) {
            const int id = yidx[k], j1 = yptr[(id >> 6) + 1];
            float s = 0.f;
            constexpr int kU = 24;
            for (int j = yptr[id >> 6]; j < j1; j += kU) {
              float v[kU];
#pragma unroll
              for (int u = 0; u < kU; ++u)
                v[u] = j + u < j1 ? __ldcg(a.t.ypart + 64 * (size_t)ylist[j + u] + (id & 63)) : 0.f;
#pragma unroll
              for (int u = 0; u < kU; ++u) s += v[u];
            }
            reinterpret_cast<float*>(s_yc + k / 3)[k % 3] = s;
          }
        }
      } else {
        col_load(tid, po4, first);
      }
      nrz = sum_end(lz, ssum[2]);  // (its barrier also covers s_yc)
      beta = first ? 0.0 : nrz / rz;
      const float bt = (float)beta;
      for (int i0 = tid; i0 < nc; i0 += kCols * kPcgThreads) {
        if (i0 != tid) col_load(i0, po4, first);
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
          const int i = i0 + u * kPcgThreads;
          if (i < nc) {
            float z0 = zv[u].x, z1 = zv[u].y, z2 = zv[u].z;
            if (TL) {
              const uint32_t cpk[4] = {cv[u].x, cv[u].y, cv[u].z, cv[u].w};
              float c0 = 0.f, c1 = 0.f, c2 = 0.f;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const float4 y = s_yc[(cpk[k >> 1] >> (16 * (k & 1))) & 0xffffu];
                const float w = tri_weight(lv[u].x, lv[u].y, lv[u].z, k);
                c0 += w * y.x;
                c1 += w * y.y;
                c2 += w * y.z;
              }
              z0 = (fv[u] & 1) ? 0.f : z0 + c0;
              z1 = (fv[u] & 2) ? 0.f : z1 + c1;
              z2 = (fv[u] & 4) ? 0.f : z2 + c2;
            }
            const float4 v = make_float4(z0 + bt * pv[u].x, z1 + bt * pv[u].y, z2 + bt * pv[u].z, 0.f);
            sx[i] = v.x;
            sy[i] = v.y;
            sz[i] = v.z;
            if (i < nrow) p4[row0 + i] = v;
          }
        }
      }
      rz = nrz;
      if (!isfinite(nrz) || (TL && !(nrz > 0.0))) {
        done = status = 3;
        break;
      }
      if (!TL && first && !(nrz > 0.0)) {  // a zero preconditioned residual
        done = 1;
        break;
      }
      __syncthreads();
      double pap = 0.0;
      for (int s = warp >> split; s < nsl; s += kWarps >> split) {
        int t0 = s_step[s], t1 = s_step[s + 1];
        if (split) {
          const int n = t1 - t0, h = warp & ((1 << split) - 1);
          t1 = t0 + (n * (h + 1) >> split);
          t0 += n * h >> split;
        }
        const int node = __ldg(a.as.slice_rows + 32 * (size_t)(sl0 + s) + lane);
        const int la = node >= 0 ? node - row0 : 0;
        const float xa = sx[la], ya = sy[la], za = sz[la];
        float y0 = 0.f, y1 = 0.f, y2 = 0.f;
        if (s < res && !loaded && s_step[s + 1] > s_step[s]) {
          ok = bulk::wait(bars + 3 * (s % kWarps) + 2, 0u) && ok;
          loaded = true;
        }
        for (int t = t0; t < t1; t += kPcgPiece) {
          const unsigned char* buf = s < res ? s_dyn + (size_t)(t - s_step[0]) * kAsmStepBytes : take();
#pragma unroll
          for (int u = 0; u < kPcgPiece; ++u)
            if (t + u < t1) {
              const unsigned char* w = buf + u * kAsmStepBytes;
              const int lb = reinterpret_cast<const uint16_t*>(w)[lane];
              const float4 A = reinterpret_cast<const float4*>(w + 64)[lane];
              const float4 B = reinterpret_cast<const float4*>(w + 576)[lane];
              const float C = reinterpret_cast<const float*>(w + 1088)[lane];
              const float d0 = sx[lb] - xa, d1 = sy[lb] - ya, d2 = sz[lb] - za;
              y0 += A.x * d0 + A.y * d1 + A.z * d2;
              y1 += A.w * d0 + B.x * d1 + B.y * d2;
              y2 += B.z * d0 + B.w * d1 + C * d2;
            }
          if (s >= res) {
            __syncwarp();  // the piece is read
            issue();
          }
        }
        if (split) {
          float* o = s_split + 96 * warp + lane;
          o[0] = y0;
          o[32] = y1;
          o[64] = y2;
        } else if (node >= 0) {
          q4[node] = make_float4(y0, y1, y2, 0.f);
          pap += (double)y0 * xa + (double)y1 * ya + (double)y2 * za;
        }
      }
      if (split) {
        __syncthreads();
        if (warp < nsl) {  // a warp per slice adds its parts
          const int node = __ldg(a.as.slice_rows + 32 * (size_t)(sl0 + warp) + lane);
          float y[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            y[d] = 0.f;
            for (int h = 0; h < 1 << split; ++h) y[d] += s_split[96 * ((warp << split) + h) + 32 * d + lane];
          }
          if (node >= 0) {
            const int la = node - row0;
            q4[node] = make_float4(y[0], y[1], y[2], 0.f);
            pap += (double)y[0] * sx[la] + (double)y[1] * sy[la] + (double)y[2] * sz[la];
          }
        }
      }
      if (!ok) pap = __longlong_as_double(0x7ff8000000000000LL);
      post(part_a, pap, sred[0]);
      if (TL) seg_load(warp);  // in flight under the barrier
      if (!grid_barrier(a.bar, ++epoch)) break;
    } else if (TL) {
      seg_load(warp);
    }

    // ── B: x, r, ||r||^2, S r and r.S r ──
    // (p comes from the planes, whose own rows then take r for the restriction)
    const double la = init ? 0.0 : sum_load(part_a);
    float4 qv[kRows];
    auto q_load = [&](int i0) {
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (i0 + u * kPcgThreads < nrow) qv[u] = q4[row0 + i0 + u * kPcgThreads];
    };
    if (!init) {
      row_load(tid, false);
      q_load(tid);
      pAp = sum_end(la, ssum[0]);
      if (!(pAp > 0.0) || !isfinite(pAp)) {
        done = status = 3;
        alpha = 0.0;
        break;
      }
      alpha = rz / pAp;
    }

    const float al = (float)alpha;
    double lrr = 0.0, lrz = 0.0;
    for (int i0 = tid; i0 < nrow; i0 += kRows * kPcgThreads) {
      if (init || i0 != tid) row_load(i0, init);
      if (!init && i0 != tid) q_load(i0);
#pragma unroll
      for (int u = 0; u < kRows; ++u) {
        const int i = i0 + u * kPcgThreads, n = row0 + i;
        if (i >= nrow) break;
        float4 r = rv[u];
        if (init) {
          r = make_float4((float)a.b[3 * (size_t)n], (float)a.b[3 * (size_t)n + 1], (float)a.b[3 * (size_t)n + 2],
                          0.f);
          x4[n] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
          r.x -= al * qv[u].x; r.y -= al * qv[u].y; r.z -= al * qv[u].z;
          x4[n] = make_float4(xv[u].x + al * px[i], xv[u].y + al * py[i], xv[u].z + al * pz[i], 0.f);
        }
        r4[n] = r;
        if (TL) {
          px[i] = r.x;
          py[i] = r.y;
          pz[i] = r.z;
        }
        lrr += (double)r.x * r.x + (double)r.y * r.y + (double)r.z * r.z;
        float4 sv = make_float4(dv[u].x * r.x, dv[u].y * r.y, dv[u].z * r.z, 0.f);
        if (o4) {
          sv.x += ov[u].x * r.y + ov[u].y * r.z;
          sv.y += ov[u].x * r.x + ov[u].z * r.z;
          sv.z += ov[u].y * r.x + ov[u].z * r.y;
        }
        z4[n] = sv;
        lrz += (double)r.x * sv.x + (double)r.y * sv.y + (double)r.z * sv.z;
      }
    }
    cta_sum2(lrr, lrz, sred[0], sred[1]);
    if (tid == 0) {
      part_b[g] = lrr;
      part_d[g] = lrz;
    }
    if (TL) {
      // restricted shares of the CTA's rows, a warp per cell, three cells in
      // flight (the residuals above are this CTA's own, ordered by the sums'
      // barrier)
      for (int s0 = warp; s0 < nseg; s0 += kSegs * kWarps) {
        if (s0 != warp) seg_load(s0);
        float3 sr[kSegs];
#pragma unroll
        for (int u = 0; u < kSegs; ++u) {
          const int i = __float_as_int(lt[u].w) - row0;
          sr[u] = i >= 0 ? make_float3(px[i], py[i], pz[i]) : make_float3(0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kSegs; ++u) {
          const int s = s0 + u * kWarps;
          if (s >= nseg) break;
          float acc[32];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float w = tri_weight(lt[u].x, lt[u].y, lt[u].z, k);
            acc[4 * k] = w * sr[u].x;
            acc[4 * k + 1] = w * sr[u].y;
            acc[4 * k + 2] = w * sr[u].z;
            acc[4 * k + 3] = 0.f;
          }
          for (int j = sptr[s] + 32 + lane; j < sptr[s + 1]; j += 32) {
            const float4 l = __ldg(lat + j);
            const int i = __float_as_int(l.w) - row0;
            const float3 v = make_float3(px[i], py[i], pz[i]);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float w = tri_weight(l.x, l.y, l.z, k);
              acc[4 * k] += w * v.x;
              acc[4 * k + 1] += w * v.y;
              acc[4 * k + 2] += w * v.z;
            }
          }
          // reduce-scatter over the warp: lane k ends with word k of the 8 float4 shares
#pragma unroll
          for (int o = 16; o >= 1; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < o; ++k) {
              const float send = up ? acc[k] : acc[k + o];
              const float keep = up ? acc[k + o] : acc[k];
              acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          }
          reinterpret_cast<float*>(a.t.seg_r + (tab + tab[TAB_SPOS])[8 * s + (lane >> 2)])[lane & 3] = acc[0];
        }
      }
    }
    if (!grid_barrier(a.bar, ++epoch)) break;
    const double lr = sum_load(part_b);
    const bool merged = TL && a.t.merged;
    if (TL) {
      // ── C1: r_c from its shares (before the stopping test: the shares of
      // ||r||^2 arrive under it), a warp per coarse node where that is one
      // round, else eight lanes; merged, every CTA adds up all of r_c for
      // itself and the barrier falls away ──
      const int* cptr = merged ? a.t.cn_ptr : tab + tab[TAB_CPTR];
      const int ncn = merged ? a.c.n_cn : tab[TAB_NCN];
      const int lanes = ncn <= kWarps ? 32 : 8, per = 32 / lanes, sub = lane & (lanes - 1);
      float* out = merged ? scratch : a.c.rc + 3 * tab[TAB_CN0];
      const int n4 = (ncn + per - 1) & ~(per - 1);
      // (merged: the CTAs start at different nodes, so that they do not all
      // read the same words of L2 at once)
      const int rot = merged ? (int)((int64_t)g * n4 / G) & ~(per - 1) : 0;
      for (int kr = tid / lanes; kr < n4; kr += kPcgThreads / lanes) {
        const int k = kr + rot < n4 ? kr + rot : kr + rot - n4;
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        if (k < ncn) {
          const int j1 = cptr[k + 1];
          constexpr int kU = 4;
          for (int j = cptr[k] + sub; j < j1; j += lanes * kU) {
            float4 v[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u)
              v[u] = j + lanes * u < j1 ? __ldcg(a.t.seg_r + j + lanes * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < kU; ++u) {
              v0 += v[u].x;
              v1 += v[u].y;
              v2 += v[u].z;
            }
          }
        }
        for (int o = lanes / 2; o > 0; o >>= 1) {
          v0 += __shfl_xor_sync(0xffffffffu, v0, o);
          v1 += __shfl_xor_sync(0xffffffffu, v1, o);
          v2 += __shfl_xor_sync(0xffffffffu, v2, o);
        }
        if (k < ncn && sub < 3) out[3 * k + sub] = sub == 0 ? v0 : (sub == 1 ? v1 : v2);
      }
      if (merged)
        for (int k = 3 * ncn + tid; k < a.c.full_ld; k += kPcgThreads) scratch[k] = 0.f;
    }
    rr = sum_end(lr, ssum[1]);
    if (init) {
      rr0 = rr;
      tol2 = a.rtol * a.rtol * rr;
      if (!isfinite(rr)) {
        done = status = 3;
        break;
      }
      if (rr == 0.0) {
        done = 1;
        break;
      }
    } else {
      ++iter;
      if (!isfinite(rr)) {
        done = status = 3;
        break;
      }
      if (rr <= tol2) {
        done = 1;
        break;
      }
      if (iter >= a.max_iter) {
        done = 2;
        break;
      }
    }
    if (TL) {
      if (!merged && !grid_barrier(a.bar, ++epoch)) break;
      // ── C2: y_c = Ac^-1 r_c, and r_c.y_c = r.P y_c ──
      double lrc = 0.0;
      if (a.c.full_ld) {
        // full rows, a warp each
        const int ld = a.c.full_ld, nd = a.c.n_dof;
        // (r_c is zero beyond n_dof)
        if (!merged) {
          for (int k = tid; k < ld / 4; k += kPcgThreads)
            reinterpret_cast<float4*>(scratch)[k] = __ldcg(reinterpret_cast<const float4*>(a.c.rc) + k);
          __syncthreads();
        }  // (merged: the stopping test's sum had the barrier)
        for (int row = g * kWarps + warp; row < nd; row += G * kWarps) {
          float s = 0.f;
          if (a.c.Afull16) {
            const uint4* A = reinterpret_cast<const uint4*>(a.c.Afull16 + (size_t)row * ld);
            constexpr int kU = 6;
            for (int k0 = lane; k0 < ld / 8; k0 += 32 * kU) {
              uint4 w[kU];
#pragma unroll
              for (int u = 0; u < kU; ++u)
                w[u] = k0 + 32 * u < ld / 8 ? __ldg(A + k0 + 32 * u) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                const int k = min(k0 + 32 * u, ld / 8 - 1);
                float v[8];
                tile_row(w[u], v);
                const float4 x0 = reinterpret_cast<const float4*>(scratch)[2 * k];
                const float4 x1 = reinterpret_cast<const float4*>(scratch)[2 * k + 1];
                s += v[0] * x0.x + v[1] * x0.y + v[2] * x0.z + v[3] * x0.w;
                s += v[4] * x1.x + v[5] * x1.y + v[6] * x1.z + v[7] * x1.w;
              }
            }
          } else {
            const float4* A = reinterpret_cast<const float4*>(a.c.Afull32 + (size_t)row * ld);
            constexpr int kU = 12;
            for (int k0 = lane; k0 < ld / 4; k0 += 32 * kU) {
              float4 w[kU];
#pragma unroll
              for (int u = 0; u < kU; ++u)
                w[u] = k0 + 32 * u < ld / 4 ? __ldg(A + k0 + 32 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                const float4 x = reinterpret_cast<const float4*>(scratch)[min(k0 + 32 * u, ld / 4 - 1)];
                s += w[u].x * x.x + w[u].y * x.y + w[u].z * x.z + w[u].w * x.w;
              }
            }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0) {
            a.c.yc[row] = s;
            lrc += (double)s * scratch[row];
          }
        }
      } else {
        // this CTA's tiles, 4 KB parts from the warps' rings; outputs staged
        // (per tile u, then v of each part) and added per row block
        const int b0 = tab[TAB_BLK0], nl = tab[TAB_NL], batch = a.tile_batch, per = 64 * (1 + parts);
        const int *ids = tab + tab[TAB_TILES], *blk = tab + tab[TAB_BLK], *optr = tab + tab[TAB_OPTR],
                  *olist = tab + tab[TAB_OLIST];
        float* s_x = scratch;                     // [nl][64] r_c of the local blocks (BF16: [nl][3][64] parts)
        float* s_y = s_x + 96 * a.t.max_lblk;     // [nl][64] sums
        float* s_out = s_y + 64 * a.t.max_lblk;   // [batch][1 + parts][64] tile outputs
        __nv_bfloat16* s_x3 = reinterpret_cast<__nv_bfloat16*>(s_x);
        for (int k = tid; k < 16 * nl; k += kPcgThreads) {
          const float4 v = __ldcg(reinterpret_cast<const float4*>(a.c.rc + 64 * blk[k >> 4]) + (k & 15));
          if (a.c.Ainv16) {
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat16 p3[3];
              split3(x[e], p3);
#pragma unroll
              for (int h = 0; h < 3; ++h) s_x3[64 * (3 * (k >> 4) + h) + 4 * (k & 15) + e] = p3[h];
            }
          } else {
            reinterpret_cast<float4*>(s_x)[k] = v;
          }
          reinterpret_cast<float4*>(s_y)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        for (int tb = 0; tb < nt; tb += batch) {
          const int te = min(nt, tb + batch);
          // (the batch is a multiple of 16 tiles: every warp keeps its order of parts)
          for (int k = tb * parts + warp; k < te * parts; k += kWarps) {
            const int t = k >> pshift, h = k & (parts - 1), ij = ids[2 * t + 1], rows = 64 >> pshift;
            const int bi = ij & 0xffff, bj = ij >> 16;
            float* out = s_out + per * (t - tb);
            const unsigned char* buf = take();
            if (a.c.Ainv16)
              tile_part16(buf, s_x3 + 192 * bj, s_x3 + 192 * bi + rows * h, out + rows * h, out + 64 * (1 + h));
            else
              tile_part32(buf, s_x + 64 * bj, s_x + 64 * bi + rows * h, out + rows * h, out + 64 * (1 + h));
            __syncwarp();
            issue();
          }
          __syncthreads();
          for (int k = tid; k < 16 * nl; k += kPcgThreads) {
            float4 s = reinterpret_cast<const float4*>(s_y)[k];
            const int j1 = optr[(k >> 4) + 1], o0 = tb * (1 + parts), o1 = te * (1 + parts);
            constexpr int kU = 4;
            for (int j = optr[k >> 4]; j < j1; j += kU) {
              float4 v[kU];
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                const int o = j + u < j1 ? olist[j + u] : -1;
                v[u] = o >= o0 && o < o1 ? reinterpret_cast<const float4*>(s_out)[16 * (o - o0) + (k & 15)]
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
              }
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w;
              }
            }
            reinterpret_cast<float4*>(s_y)[k] = s;
          }
          __syncthreads();
        }
        for (int k = tid; k < 16 * nl; k += kPcgThreads)
          reinterpret_cast<float4*>(a.t.ypart + 64 * (size_t)b0)[k] = reinterpret_cast<const float4*>(s_y)[k];
        // (BF16: the three parts add up to r_c exactly)
        for (int k = tid; k < 64 * nl; k += kPcgThreads) {
          const __nv_bfloat16* x3 = s_x3 + 192 * (k >> 6) + (k & 63);
          const float x = a.c.Ainv16 ? __bfloat162float(x3[0]) + (__bfloat162float(x3[64]) + __bfloat162float(x3[128]))
                                     : s_x[k];
          lrc += (double)x * s_y[k];
        }
      }
      post(part_e, lrc, sred[0]);
      col_load(tid, p4, init);
      if (!grid_barrier(a.bar, ++epoch)) break;
    }
    first = init;
  }
  // copies still in flight land before the CTA's shared memory goes away
  if (any)
    for (int k = 0; k < ns; ++k) take();
  if (total > 0) bulk::wait(bar + 2, 0u);
  if (g == 0 && tid == 0) {
    CGState* st = a.cg;
    st->rz = rz;
    st->pAp = pAp;
    st->rr = rr;
    st->rr0 = rr0;
    st->tol2 = tol2;
    st->alpha = alpha;
    st->beta = beta;
    st->iter = iter;
    st->max_iter = a.max_iter;
    st->zsel = st->n_alt = st->locked = st->trips = 0;
    st->done = done;       // 0: a barrier gave up
    st->status = status;
  }
}

// ───────────────────────── launcher ─────────────────────────

bool pcg_plan(PcgArgs& a, bool two_level, const std::vector<int>& prefix, size_t* smem) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t limit = (size_t)optin - 2048;  // less the kernel's static shared memory
  const bool tiles = two_level && a.c.full_ld == 0;
  const size_t parts = a.c.Ainv16 ? 2 : 4;
  a.max_items = a.as.max_pieces + (tiles ? (int)((a.t.max_tiles * parts + kWarps - 1) / kWarps) : 0);
  size_t tab = sizeof(int) * (size_t)(a.as.max_slices + 1 + a.as.max_halo + (two_level ? a.t.max_tab : 0));
  tab = (tab + 7) & ~(size_t)7;
  a.items_off = (uint32_t)tab;
  tab += sizeof(uint2) * kWarps * (size_t)a.max_items;
  size_t base = sizeof(float) * 3 * (size_t)a.as.max_cols;
  if (two_level) base += sizeof(float) * 4 * (size_t)a.t.max_loc;
  base += sizeof(float) * 96 * kWarps;  // few slices: the warps' parts
  if (two_level) base = std::max(base, sizeof(float) * (size_t)a.c.full_ld);
  const int nsl = a.as.max_slices;
  // the coarse tiles staged at once: all of the CTA's, or as many as fit
  for (int batch = tiles ? (a.t.max_tiles + kWarps - 1) / kWarps * kWarps : 0;; batch -= kWarps) {
    size_t scratch = base;
    if (tiles)
      scratch = std::max(scratch, sizeof(float) * (160 * (size_t)a.t.max_lblk + 64 * (1 + parts) * (size_t)batch));
    scratch = (scratch + 127) & ~(size_t)127;
    // all slices resident and rings for the tiles, if any; else rings of two
    // stages or one for both, and as many resident slices as then fit
    for (int mode = 0; mode < 4; ++mode) {
      const bool all = mode < 2;
      const int ns = mode % 2 ? 1 : 2;
      const size_t stage = all ? (tiles ? 4096 : 0) : std::max<size_t>(tiles ? 4096 : 0, (kPcgPiece * kAsmStepBytes + 127) & ~127);
      const size_t ring = stage * ns * kWarps;
      if (scratch + tab + ring > limit) continue;
      const size_t room = limit - scratch - tab - ring;
      int res = 0;
      while (res < nsl && (((size_t)prefix[res + 1] * kAsmStepBytes + 127) & ~(size_t)127) <= room) ++res;
      if (all && res < nsl) continue;
      a.resident = res;
      a.stages = stage ? ns : 0;
      a.stage_bytes = (uint32_t)stage;
      a.res_bytes = (uint32_t)(((size_t)prefix[res] * kAsmStepBytes + 127) & ~(size_t)127);
      a.mat_bytes = a.res_bytes + (uint32_t)ring;
      a.scratch_bytes = (uint32_t)scratch;
      a.tile_batch = batch;
      *smem = a.mat_bytes + scratch + tab;
      return true;
    }
    if (batch <= kWarps) break;
  }
  return false;
}

__global__ void pcg_seg_lat_kernel(const int* seg_rows, const float4* node_lat, int n, float4* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int node = seg_rows[i];
  const float4 l = node_lat[node];
  out[i] = make_float4(l.x, l.y, l.z, __int_as_float(node));
}

void launch_pcg_seg_lat(const int* seg_rows, const float4* node_lat, int n, float4* out, cudaStream_t s) {
  pcg_seg_lat_kernel<<<(n + 255) / 256, 256, 0, s>>>(seg_rows, node_lat, n, out);
}

cudaError_t launch_pcg(const PcgArgs& a, bool two_level, size_t smem, cudaStream_t s) {
  const void* fn = two_level ? reinterpret_cast<const void*>(pcg_kernel<true>)
                             : reinterpret_cast<const void*>(pcg_kernel<false>);
  raise_smem_limit(fn);
  PcgArgs arg = a;
  void* params[] = {&arg};
  return cudaLaunchCooperativeKernel(fn, dim3(a.as.grid), dim3(kPcgThreads), params, smem, s);
}

}  // namespace femb200
