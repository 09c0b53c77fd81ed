// Assembled tangent: the off-diagonal 3 x 3 blocks K_ab of K_T, once per
// tangent state, and the product
//
//   (K x)_a = sum_{b != a} K_ab (x_b - x_a).
//
// Rigid translations leave every element stress-free, so the diagonal block
// is K_aa = -sum_b K_ab: it is neither stored nor read, and the difference
// form keeps the element pass's accuracy for smooth x (no cancellation of
// large K_aa x_a against the rest).
//
// Storage.  The rows (internal node order) are dealt out in runs to the CTAs
// of the persistent PCG kernel (fem_pcg.cu).  A CTA's rows, longest first, are
// cut into slices of 32, one row per lane; a slice's step k holds the rows'
// k-th entries side by side (kAsmStepBytes: columns, then the blocks'
// components), so a warp's reads are conflict-free, a row's sum stays in its
// lane's registers in the order of its entries, and a run of steps is one
// contiguous piece for a bulk copy.  Columns are local to the CTA: its rows,
// then a list of halo nodes.  Padding slots hold zero blocks on the row
// itself.  On the 64-voxel vertebral body 38 bytes x 1.4 M entries stream
// once per product, against 45 MB of element data, 36 MB of slot vectors
// written and read again and eight 16-byte vertex gathers per element.  (An
// entry-per-thread form, products added per row through shared memory, took
// 38 shared-memory cycles per 32 entries where this takes 20.)
//
// Rows of fixed DOFs are stored as zeros (K_ff x for x zero on fixed DOFs).
//
// The reference assembles its tangent with scatter-adds on the host
// (backend/fea/fem/solver/assembly.py:20-287); here each undirected edge's
// block is a fixed-order sum over the elements on it (one thread per edge, no
// atomics: bitwise reproducible), written to both of its rows.
#include <cuda_runtime.h>

#include <algorithm>

#include "fem_asm.h"

namespace femb200 {

// ───────────────────────── tables ─────────────────────────
//
// The first solve of a context pays for them, so the neighbour lists, halos,
// columns and edge lists are derived on the device and the host only deals out
// the rows: 2.0 ms at 74,600 hexes, where the neighbours and halos on the host
// took 16 ms with sixteen cores and 67 with one, more than a whole solve.

void asm_cta_rows(const std::vector<int>& deg, int sms, AsmHost* out) {
  const int Nn = (int)deg.size(), G = std::max(1, std::min(sms, Nn / kAsmMinRows));
  out->grid = G;
  out->cta_row.assign(G + 1, Nn);
  out->cta_row[0] = 0;
  // runs of rows with equal entries (a row counts as 4 more) per CTA
  int64_t total = 4 * (int64_t)Nn, at = 0;
  for (int d : deg) total += d;
  int g = 1;
  for (int a = 0; a < Nn && g < G; ++a) {
    at += deg[a] + 4;
    while (g < G && at * G >= total * g) out->cta_row[g++] = a + 1;
  }
  // at least one row each
  for (int k = 1; k < G; ++k) out->cta_row[k] = std::max(out->cta_row[k], out->cta_row[k - 1] + 1);
  for (int k = G - 1; k > 0; --k) out->cta_row[k] = std::min(out->cta_row[k], out->cta_row[k + 1] - 1);
}

bool asm_slices(const std::vector<int>& deg, AsmHost* out) {
  const int Nn = (int)deg.size(), G = out->grid;
  constexpr int kWarps = kPcgThreads / 32;
  out->slot0.assign(Nn, 0u);
  out->cta_slice.assign(1, 0);
  out->slice_step.assign(1, 0);
  out->slice_rows.reserve((size_t)Nn + 32 * (size_t)G);
  std::vector<int> order, first, prefix(1, 0);
  int64_t steps = 0;
  for (int g = 0; g < G; ++g) {
    const int r0 = out->cta_row[g], r1 = out->cta_row[g + 1], rows = r1 - r0;
    // longest rows first, else in their order
    int lo = deg[r0], hi = deg[r0];
    for (int r = r0; r < r1; ++r) {
      lo = std::min(lo, deg[r]);
      hi = std::max(hi, deg[r]);
    }
    first.assign(hi - lo + 2, 0);
    for (int r = r0; r < r1; ++r) ++first[hi - deg[r] + 1];
    for (size_t k = 1; k < first.size(); ++k) first[k] += first[k - 1];
    order.resize(rows);
    for (int r = r0; r < r1; ++r) order[first[hi - deg[r]]++] = r;
    const int64_t step0 = steps;
    int pieces[kWarps] = {}, n = 0;
    for (int i = 0; i < rows; i += 32, ++n) {
      const int d = deg[order[i]];
      for (int l = 0; l < 32; ++l) {
        const int r = i + l < rows ? order[i + l] : -1;
        out->slice_rows.push_back(r);
        if (r >= 0) out->slot0[r] = (uint32_t)(steps * 32 + l);
      }
      steps += d;
      if (steps >= (1LL << 27)) return false;
      out->slice_step.push_back((int)steps);
      if ((int)prefix.size() == n + 1) prefix.push_back(prefix.back());
      prefix[n + 1] = std::max(prefix[n + 1], (int)(steps - step0));
      pieces[n % kWarps] += (d + kPcgPiece - 1) / kPcgPiece;
    }
    out->cta_slice.push_back((int)out->slice_step.size() - 1);
    out->max_slices = std::max(out->max_slices, n);
    for (int w : pieces) out->max_pieces = std::max(out->max_pieces, w);
    for (size_t k = n + 1; k < prefix.size(); ++k) prefix[k] = std::max(prefix[k], (int)(steps - step0));
  }
  out->prefix = prefix;
  return true;
}

// A warp per node: the other vertices of its elements, each at the place that
// the smaller ones and the earlier equal ones leave it, then without repeats.
template <int SH>
__global__ void __launch_bounds__(128) asm_neighbours_kernel(const MeshDev m, int* cand, int* cols, int* counts) {
  constexpr int kN = 1 << SH, kOther = kN - 1;
  constexpr unsigned kFull = 0xffffffffu;
  const int a = blockIdx.x * 4 + ((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (a >= m.n_nodes) return;
  const int s0 = m.node_row[a], ns = m.node_row[a + 1] - s0, n = ns * kOther;
  const int base = m.blk_ptr[a / m.nb];
  cand += (size_t)s0 * kOther;
  cols += (size_t)s0 * kOther;
  for (int j = lane; j < ns; j += 32) {
    const uint32_t code = m.node_slots[s0 + j];
    const int la = (int)(code & (uint32_t)kOther);
    const int* cn = reinterpret_cast<const int*>(m.conn) + kN * (size_t)m.blk_elems[base + (int)(code >> SH)];
#pragma unroll
    for (int k = 0; k < kN; ++k)
      if (k != la) cand[kOther * j + (k < la ? k : k - 1)] = cn[k];
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    const int v = cand[i];
    int at = 0;
    for (int j = 0; j < n; ++j) {
      const int w = cand[j];
      at += w < v || (w == v && j < i);
    }
    cols[at] = v;
  }
  __syncwarp();
  int deg = 0, up = 0, len = 0, carry = -1;
  for (int c = 0; c < n; c += 32) {
    const bool in = c + lane < n;
    const int v = in ? cols[c + lane] : -1;
    int prev = __shfl_up_sync(kFull, v, 1);
    if (lane == 0) prev = carry;
    carry = __shfl_sync(kFull, v, 31);
    const bool first = in && v != prev;
    const unsigned mask = __ballot_sync(kFull, first);
    if (first) cols[deg + __popc(mask & ((1u << lane) - 1u))] = v;  // (below the next chunk)
    deg += __popc(mask);
    up += __popc(__ballot_sync(kFull, first && v > a));
    len += __popc(__ballot_sync(kFull, in && v > a));
    __syncwarp();
  }
  if (lane == 0) {
    counts[a] = deg;
    counts[m.n_nodes + a] = up;
    counts[2 * (size_t)m.n_nodes + a] = len;
  }
}

// The halo of one CTA of the solve: its rows' columns outside its run, marked.
__global__ void __launch_bounds__(256) asm_halo_mark_kernel(const MeshDev m, const __grid_constant__ AsmLists t,
                                                            const int* cta_row, uint32_t* bits0, uint32_t* bits1,
                                                            int* count) {
  __shared__ int s_n;
  const int g = blockIdx.x, r0 = cta_row[g], r1 = cta_row[g + 1], words = (m.n_nodes + 31) / 32;
  uint32_t* bits = (g & 1 ? bits1 : bits0) + (size_t)(g >> 1) * words;
  if (threadIdx.x == 0) s_n = 0;
  for (int r = r0 + (int)threadIdx.x; r < r1; r += 256) {
    const int* c = t.cols + (size_t)m.node_row[r] * (m.npe - 1);
    const int deg = t.deg[r];
    for (int k = 0; k < deg; ++k) {
      const int n = c[k];
      if (n < r0 || n >= r1) atomicOr(bits + (n >> 5), 1u << (n & 31));
    }
  }
  __syncthreads();
  int n = 0;
  for (int w = threadIdx.x; w < words; w += 256) n += __popc(__ldcg(bits + w));
  atomicAdd(&s_n, n);
  __syncthreads();
  if (threadIdx.x == 0) count[g] = s_n;
}

// ... and listed: each thread a run of words, after the marks of the runs before it.
__global__ void __launch_bounds__(256) asm_halo_list_kernel(int n_nodes, const uint32_t* bits0,
                                                            const uint32_t* bits1, const int* halo_ptr, int* halo) {
  __shared__ int s_n[256];
  const int g = blockIdx.x, tid = threadIdx.x, words = (n_nodes + 31) / 32;
  const uint32_t* bits = (g & 1 ? bits1 : bits0) + (size_t)(g >> 1) * words;
  const int w0 = (int)((int64_t)words * tid / 256), w1 = (int)((int64_t)words * (tid + 1) / 256);
  int n = 0;
  for (int w = w0; w < w1; ++w) n += __popc(bits[w]);
  s_n[tid] = n;
  __syncthreads();
  int at = halo_ptr[g];
  for (int k = 0; k < tid; ++k) at += s_n[k];
  for (int w = w0; w < w1; ++w)
    for (uint32_t b = bits[w]; b; b &= b - 1u) halo[at++] = 32 * w + __ffs((int)b) - 1;
}

// Edges to higher nodes, their slots and their (element, vertex pair) lists,
// a thread per node: the elements on the node in its slot order.
template <int SH>
__global__ void __launch_bounds__(128) asm_list_kernel(const MeshDev m, const __grid_constant__ AsmLists t, uint2* edges,
                                                       uint32_t* eptr, uint32_t* list) {
  const int a = blockIdx.x * 128 + threadIdx.x;
  if (a >= m.n_nodes) return;
  constexpr int kN = 1 << SH;
  const int s0 = m.node_row[a], s1 = m.node_row[a + 1], deg = t.deg[a];
  const int* ca = t.cols + (size_t)s0 * (kN - 1);
  const uint32_t e0 = t.erow[a], ne = t.erow[a + 1] - e0;
  uint32_t l = t.lrow[a];
  const int up = deg - (int)ne;
  const int base = m.blk_ptr[a / m.nb];
  for (uint32_t q = 0; q < ne; ++q) {
    const int b = ca[up + (int)q];
    const int* cb = t.cols + (size_t)m.node_row[b] * (kN - 1);
    int lo = 0, hi = t.deg[b];
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (cb[mid] < a)
        lo = mid + 1;
      else
        hi = mid;
    }
    edges[e0 + q] = make_uint2(t.slot0[a] + 32u * (uint32_t)(up + (int)q), t.slot0[b] + 32u * (uint32_t)lo);
    eptr[e0 + q] = l;
    for (int j = s0; j < s1; ++j) {
      const uint32_t code = m.node_slots[j];
      const uint32_t e = (uint32_t)m.blk_elems[base + (int)(code >> SH)], la = code & (uint32_t)(kN - 1);
      const int* cn = reinterpret_cast<const int*>(m.conn) + kN * (size_t)e;
#pragma unroll
      for (int k = 0; k < kN; ++k)
        if (cn[k] == b) list[l++] = (e * kN + la) * kN + (uint32_t)k;
    }
  }
  if (a == m.n_nodes - 1) eptr[e0 + ne] = l;
}

// Local columns of the steps; one CTA per CTA of the solve, a warp per slice.
__global__ void __launch_bounds__(512) asm_fill_kernel(const MeshDev m, const __grid_constant__ AsmDev S,
                                                       const __grid_constant__ AsmLists t) {
  const int g = blockIdx.x, lane = threadIdx.x & 31, r0 = S.cta_row[g], r1 = S.cta_row[g + 1];
  const int* halo = S.halo + S.halo_ptr[g];
  const int nh = S.halo_ptr[g + 1] - S.halo_ptr[g];
  for (int s = S.cta_slice[g] + ((int)threadIdx.x >> 5); s < S.cta_slice[g + 1]; s += 16) {
    const int r = S.slice_rows[32 * (size_t)s + lane], deg = r >= 0 ? t.deg[r] : 0;
    const int* c = t.cols + (r >= 0 ? (size_t)m.node_row[r] * (m.npe - 1) : 0);
    const int t0 = S.slice_step[s], t1 = S.slice_step[s + 1];
    for (int k = t0; k < t1; ++k) {
      const int n = k - t0 < deg ? c[k - t0] : r;  // padding: the row itself
      int l = n < 0 ? 0 : n - r0;
      if (n >= 0 && (n < r0 || n >= r1)) {
        int lo = 0, hi = nh;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (halo[mid] < n)
            lo = mid + 1;
          else
            hi = mid;
        }
        l = r1 - r0 + lo;
      }
      reinterpret_cast<uint16_t*>(S.words + (size_t)k * kAsmStepWords)[lane] = (uint16_t)l;
    }
  }
}

// ───────────────────────── assembly ─────────────────────────

// One thread per edge (a, b), a < b: K_ab summed over the elements on the
// edge in ascending element order, and K_ba = K_ab^T.  Column i of an
// element's block is the force at a under the unit displacement e_i of b.
// Bound by the scattered element loads (L1); each edge has about five
// elements, which neighbouring threads share.
template <int MODEL>
__global__ void __launch_bounds__(128) asm_edge_kernel(const __grid_constant__ AsmArgs a) {
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= a.s.n_edges) return;
  const MeshDev& m = a.m;
  const uint2 ed = __ldg(a.s.edges + t);
  const uint32_t l0 = __ldg(a.s.eptr + t), l1 = __ldg(a.s.eptr + t + 1);
  float K[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) K[k] = 0.f;
  int na = 0, nb = 0;
  for (uint32_t l = l0; l < l1; ++l) {
    const uint32_t en = __ldg(a.s.list + l);
    const int e = (int)(en >> 4), la = (int)(en >> 2) & 3, lb = (int)en & 3;
    const int4 cn = __ldg(m.conn + e);
    const int nid[4] = {cn.x, cn.y, cn.z, cn.w};
    na = la == 0 ? cn.x : (la == 1 ? cn.y : (la == 2 ? cn.z : cn.w));
    nb = lb == 0 ? cn.x : (lb == 1 ? cn.y : (lb == 2 ? cn.z : cn.w));
    float xv[4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 X = __ldg(m.X32 + nid[k]);
      xv[k][0] = X.x;
      xv[k][1] = X.y;
      xv[k][2] = X.z;
    }
    TetGeom<float> g;
    tet_geom(xv[0], xv[1], xv[2], xv[3], g);
    float wa[3], wb[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float w0 = -(g.c[0][j] + g.c[1][j] + g.c[2][j]);
      wa[j] = la == 0 ? w0 : (la == 1 ? g.c[0][j] : (la == 2 ? g.c[1][j] : g.c[2][j]));
      wb[j] = (lb == 0 ? w0 : (lb == 1 ? g.c[0][j] : (lb == 2 ? g.c[1][j] : g.c[2][j]))) * g.inv_det;
      wa[j] *= g.s6;
    }
    const DevMat<float>& mat = a.matF[__ldg(m.mat_id + e)];
    const float scale = __ldg(m.scale + e);
    float pay[kPay];
    {
      const int npay = model_pay_words(MODEL >= 0 ? MODEL : mat.model);
#pragma unroll
      for (int k = 0; k < kPay; ++k)
        pay[k] = (k < npay) ? __ldg(a.payload + (size_t)k * m.n_elems + e) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      float dF[9], dP[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) dF[k] = 0.f;
#pragma unroll
      for (int j = 0; j < 3; ++j) dF[3 * i + j] = wb[j];
      dP_any<MODEL>(mat, scale, pay, dF, dP);
#pragma unroll
      for (int r = 0; r < 3; ++r) K[3 * r + i] += dP[3 * r] * wa[0] + dP[3 * r + 1] * wa[1] + dP[3 * r + 2] * wa[2];
    }
  }
  asm_store(a.s, ed.x, K[0], K[1], K[2], K[3], K[4], K[5], K[6], K[7], K[8], m.fixed[na]);
  asm_store(a.s, ed.y, K[0], K[3], K[6], K[1], K[4], K[7], K[2], K[5], K[8], m.fixed[nb]);
}

// Smoother from the assembled blocks: K_aa = -sum_b K_ab, inverted as
// diag_store does (the 3 x 3 block, or its diagonal).  A warp per slice, a
// lane per row.
template <bool BLOCK>
__global__ void __launch_bounds__(128) asm_diag_kernel(const __grid_constant__ AsmArgs a, float* dinv, float* boff) {
  const int s = blockIdx.x * 4 + ((int)threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= a.s.n_slices) return;
  const int node = __ldg(a.s.slice_rows + 32 * (size_t)s + lane);
  float k[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) k[c] = 0.f;
  const int t1 = __ldg(a.s.slice_step + s + 1);
#pragma unroll 4
  for (int t = __ldg(a.s.slice_step + s); t < t1; ++t) {
    const uint32_t* w = a.s.words + (size_t)t * kAsmStepWords;
    const float4 A = __ldg(reinterpret_cast<const float4*>(w + 16) + lane);
    const float4 B = __ldg(reinterpret_cast<const float4*>(w + 144) + lane);
    k[0] += A.x; k[1] += A.y; k[2] += A.z; k[3] += A.w;
    k[4] += B.x; k[5] += B.y; k[6] += B.z; k[7] += B.w;
    k[8] += __ldg(reinterpret_cast<const float*>(w + 272) + lane);
  }
  if (node < 0) return;
  const float acc6[6] = {-k[0], -0.5f * (k[1] + k[3]), -0.5f * (k[2] + k[6]), -k[4], -0.5f * (k[5] + k[7]), -k[8]};
  const float acc3[3] = {-k[0], -k[4], -k[8]};
  diag_store<BLOCK>(BLOCK ? acc6 : acc3, a.m.fixed[node], node, dinv, boff);
}

// ───────────────────────── launchers ─────────────────────────

void launch_asm_neighbours(const MeshDev& m, int* cand, int* cols, int* counts, cudaStream_t s) {
  const int g = (m.n_nodes + 3) / 4;
  if (m.npe == 8)
    asm_neighbours_kernel<3><<<g, 128, 0, s>>>(m, cand, cols, counts);
  else
    asm_neighbours_kernel<2><<<g, 128, 0, s>>>(m, cand, cols, counts);
}

void launch_asm_halo_mark(const MeshDev& m, const AsmLists& t, const int* cta_row, int grid, uint32_t* bits0,
                          uint32_t* bits1, int* count, cudaStream_t s) {
  asm_halo_mark_kernel<<<grid, 256, 0, s>>>(m, t, cta_row, bits0, bits1, count);
}

void launch_asm_halo_list(int n_nodes, const uint32_t* bits0, const uint32_t* bits1, const int* halo_ptr, int grid,
                          int* halo, cudaStream_t s) {
  asm_halo_list_kernel<<<grid, 256, 0, s>>>(n_nodes, bits0, bits1, halo_ptr, halo);
}

void launch_asm_lists(const MeshDev& m, const AsmLists& t, uint2* edges, uint32_t* eptr, uint32_t* list, cudaStream_t s) {
  const int g = (m.n_nodes + 127) / 128;
  if (m.npe == 8)
    asm_list_kernel<3><<<g, 128, 0, s>>>(m, t, edges, eptr, list);
  else
    asm_list_kernel<2><<<g, 128, 0, s>>>(m, t, edges, eptr, list);
}

void launch_asm_fill(const MeshDev& m, const AsmDev& S, const AsmLists& t, cudaStream_t s) {
  asm_fill_kernel<<<S.grid, 512, 0, s>>>(m, S, t);
}

void launch_asm(const AsmArgs& a, int model, cudaStream_t s) {
  if (a.m.npe == 8) {
    launch_asm_hex(a, model, s);
    return;
  }
  const int g = (a.s.n_edges + 127) / 128;
  switch (model) {
    case M_LE: asm_edge_kernel<M_LE><<<g, 128, 0, s>>>(a); break;
    case M_NH: asm_edge_kernel<M_NH><<<g, 128, 0, s>>>(a); break;
    case M_MR: asm_edge_kernel<M_MR><<<g, 128, 0, s>>>(a); break;
    case M_J2: asm_edge_kernel<M_J2><<<g, 128, 0, s>>>(a); break;
    case M_TI: asm_edge_kernel<M_TI><<<g, 128, 0, s>>>(a); break;
    case M_FMR: asm_edge_kernel<M_FMR><<<g, 128, 0, s>>>(a); break;
    default: asm_edge_kernel<-1><<<g, 128, 0, s>>>(a); break;
  }
}

void launch_asm_diag(const AsmArgs& a, float* dinv, float* boff, cudaStream_t s) {
  if (boff)
    asm_diag_kernel<true><<<(a.s.n_slices + 3) / 4, 128, 0, s>>>(a, dinv, boff);
  else
    asm_diag_kernel<false><<<(a.s.n_slices + 3) / 4, 128, 0, s>>>(a, dinv, boff);
}

}  // namespace femb200
