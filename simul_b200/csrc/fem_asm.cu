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
#include <mutex>

#include "fem_asm.h"

namespace femb200 {

// ───────────────────────── tables (host) ─────────────────────────

bool build_asm_host(const int4* conn4, int Nn, int Ne, int npe, int sms, AsmHost* out) {
  const int* conn = &conn4[0].x;
  // node -> (element, vertex), elements ascending
  std::vector<int> arow(Nn + 1, 0);
  for (int64_t i = 0; i < (int64_t)npe * Ne; ++i) arow[conn[i] + 1]++;
  for (int i = 0; i < Nn; ++i) arow[i + 1] += arow[i];
  std::vector<uint32_t> acol(arow[Nn]);
  {
    std::vector<int> fill(arow.begin(), arow.end() - 1);
    for (int e = 0; e < Ne; ++e)
      for (int k = 0; k < npe; ++k) acol[fill[conn[(size_t)npe * e + k]]++] = (uint32_t)e * npe + k;
  }
  // neighbours of each node (ascending), edges to higher nodes and the
  // (element, vertex pair) lists of those edges: count, then fill
  std::vector<int64_t> nrow(Nn + 1, 0), erow(Nn + 1, 0), lrow(Nn + 1, 0);
  struct Part {
    int a0;
    std::vector<int> cols;
  };
  std::vector<Part> found;  // the neighbours, by the threads' runs of nodes
  std::mutex mu;
  parallel_ranges(Nn, [&](int a0, int a1) {
    Part p{a0, {}};
    p.cols.reserve((size_t)(a1 - a0) * (npe == 8 ? 27 : 15));
    // (rows are short: scanning the ones found so far beats sorting all repeats)
    for (int a = a0; a < a1; ++a) {
      const size_t base = p.cols.size();
      int64_t l = 0;
      for (int j = arow[a]; j < arow[a + 1]; ++j) {
        const int* cn = conn + (size_t)npe * (acol[j] / npe);
        for (int k = 0; k < npe; ++k) {
          const int b = cn[k];
          if (b == a) continue;
          l += b > a;
          size_t q = base;
          while (q < p.cols.size() && p.cols[q] != b) ++q;
          if (q == p.cols.size()) p.cols.push_back(b);
        }
      }
      std::sort(p.cols.begin() + base, p.cols.end());
      nrow[a + 1] = (int64_t)(p.cols.size() - base);
      erow[a + 1] = p.cols.end() - std::upper_bound(p.cols.begin() + base, p.cols.end(), a);
      lrow[a + 1] = l;
    }
    std::lock_guard<std::mutex> lock(mu);
    found.push_back(std::move(p));
  });
  for (int a = 0; a < Nn; ++a) {
    nrow[a + 1] += nrow[a];
    erow[a + 1] += erow[a];
    lrow[a + 1] += lrow[a];
  }
  const int64_t nnz = nrow[Nn];
  if (nnz > 0x7fffffffLL || lrow[Nn] > 0x7fffffffLL || (uint64_t)Ne * npe * npe > 0xffffffffULL) return false;
  out->cols.resize((size_t)nnz);
  out->row.assign(nrow.begin(), nrow.end());
  parallel_ranges((int)found.size(), [&](int p0, int p1) {
    for (int p = p0; p < p1; ++p)
      std::copy(found[p].cols.begin(), found[p].cols.end(), out->cols.begin() + nrow[found[p].a0]);
  }, 1);
  // runs of rows with equal entries (a row counts as 4 more) per CTA
  const int G = std::max(1, std::min(sms, Nn / kAsmMinRows));
  out->grid = G;
  out->cta_row.assign(G + 1, Nn);
  out->cta_row[0] = 0;
  {
    const int64_t total = nnz + 4 * (int64_t)Nn;
    int g = 1;
    for (int a = 0; a < Nn && g < G; ++a)
      while (g < G && (nrow[a + 1] + 4 * (int64_t)(a + 1)) * G >= total * g) out->cta_row[g++] = a + 1;
    // at least one row each
    for (int k = 1; k < G; ++k) out->cta_row[k] = std::max(out->cta_row[k], out->cta_row[k - 1] + 1);
    for (int k = G - 1; k > 0; --k) out->cta_row[k] = std::min(out->cta_row[k], out->cta_row[k + 1] - 1);
  }
  // slices; halos
  std::vector<uint32_t>& slot0 = out->slot0;
  slot0.assign(Nn, 0u);
  std::vector<std::vector<int>> halo(G), order(G);
  parallel_ranges(G, [&](int g0, int g1) {
    for (int g = g0; g < g1; ++g) {
      const int r0 = out->cta_row[g], r1 = out->cta_row[g + 1];
      for (int64_t j = nrow[r0]; j < nrow[r1]; ++j)
        if (out->cols[j] < r0 || out->cols[j] >= r1) halo[g].push_back(out->cols[j]);
      std::sort(halo[g].begin(), halo[g].end());
      halo[g].erase(std::unique(halo[g].begin(), halo[g].end()), halo[g].end());
      for (int r = r0; r < r1; ++r) order[g].push_back(r);
      std::stable_sort(order[g].begin(), order[g].end(),
                       [&](int a, int b) { return nrow[a + 1] - nrow[a] > nrow[b + 1] - nrow[b]; });
    }
  }, 1);
  out->cta_slice.assign(1, 0);
  out->slice_step.assign(1, 0);
  out->halo_ptr.assign(1, 0);
  std::vector<std::vector<int>> csteps(G);
  int64_t steps = 0;
  for (int g = 0; g < G; ++g) {
    const int rows = (int)order[g].size();
    csteps[g].push_back(0);
    for (int i = 0; i < rows; i += 32) {
      const int deg = (int)(nrow[order[g][i] + 1] - nrow[order[g][i]]);
      for (int l = 0; l < 32; ++l) {
        const int r = i + l < rows ? order[g][i + l] : -1;
        out->slice_rows.push_back(r);
        if (r >= 0) slot0[r] = (uint32_t)(steps * 32 + l);
      }
      steps += deg;
      if (steps >= (1LL << 27)) return false;
      out->slice_step.push_back((int)steps);
      csteps[g].push_back(csteps[g].back() + deg);
    }
    out->cta_slice.push_back((int)out->slice_step.size() - 1);
    out->max_slices = std::max(out->max_slices, (int)csteps[g].size() - 1);
    out->max_halo = std::max(out->max_halo, (int)halo[g].size());
    out->max_cols = std::max(out->max_cols, rows + (int)halo[g].size());
    out->halo.insert(out->halo.end(), halo[g].begin(), halo[g].end());
    out->halo_ptr.push_back((int)out->halo.size());
  }
  for (int g = 0; g < G; ++g) {
    constexpr int kWarps = kPcgThreads / 32;
    int n[kWarps] = {};
    for (size_t k = 0; k + 1 < csteps[g].size(); ++k)
      n[k % kWarps] += (csteps[g][k + 1] - csteps[g][k] + kPcgPiece - 1) / kPcgPiece;
    for (int w : n) out->max_pieces = std::max(out->max_pieces, w);
  }
  if (out->max_cols > 65536) return false;
  out->prefix.assign(out->max_slices + 1, 0);
  for (int g = 0; g < G; ++g)
    for (int k = 0; k <= out->max_slices; ++k)
      out->prefix[k] = std::max(out->prefix[k], csteps[g][std::min(k, (int)csteps[g].size() - 1)]);
  out->erow.assign(erow.begin(), erow.end());
  out->lrow.assign(lrow.begin(), lrow.end());
  return true;
}

// Edges to higher nodes, their slots and their (element, vertex pair) lists,
// a thread per node: the elements on the node in its slot order.  (On the host
// this took a third of the tables' time, and its upload as long as the rest.)
template <int SH>
__global__ void __launch_bounds__(128) asm_list_kernel(const MeshDev m, const __grid_constant__ AsmLists t, uint2* edges,
                                                       uint32_t* eptr, uint32_t* list) {
  const int a = blockIdx.x * 128 + threadIdx.x;
  if (a >= m.n_nodes) return;
  constexpr int kN = 1 << SH;
  const int j0 = t.row[a], deg = t.row[a + 1] - j0;
  const uint32_t e0 = t.erow[a], ne = t.erow[a + 1] - e0;
  uint32_t l = t.lrow[a];
  const int up = deg - (int)ne;
  const int base = m.blk_ptr[a / m.nb], s0 = m.node_row[a], s1 = m.node_row[a + 1];
  for (uint32_t q = 0; q < ne; ++q) {
    const int b = t.cols[j0 + up + (int)q];
    int lo = t.row[b], hi = t.row[b + 1];
    const int b0 = lo;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (t.cols[mid] < a)
        lo = mid + 1;
      else
        hi = mid;
    }
    edges[e0 + q] = make_uint2(t.slot0[a] + 32u * (uint32_t)(up + (int)q), t.slot0[b] + 32u * (uint32_t)(lo - b0));
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
__global__ void __launch_bounds__(512) asm_fill_kernel(const __grid_constant__ AsmDev S, const int* row, const int* cols) {
  const int g = blockIdx.x, lane = threadIdx.x & 31, r0 = S.cta_row[g], r1 = S.cta_row[g + 1];
  const int* halo = S.halo + S.halo_ptr[g];
  const int nh = S.halo_ptr[g + 1] - S.halo_ptr[g];
  for (int s = S.cta_slice[g] + ((int)threadIdx.x >> 5); s < S.cta_slice[g + 1]; s += 16) {
    const int r = S.slice_rows[32 * (size_t)s + lane];
    const int j0 = r >= 0 ? row[r] : 0, deg = r >= 0 ? row[r + 1] - j0 : 0;
    const int t0 = S.slice_step[s], t1 = S.slice_step[s + 1];
    for (int t = t0; t < t1; ++t) {
      const int n = t - t0 < deg ? cols[j0 + t - t0] : r;  // padding: the row itself
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
      reinterpret_cast<uint16_t*>(S.words + (size_t)t * kAsmStepWords)[lane] = (uint16_t)l;
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

void launch_asm_lists(const MeshDev& m, const AsmLists& t, uint2* edges, uint32_t* eptr, uint32_t* list, cudaStream_t s) {
  const int g = (m.n_nodes + 127) / 128;
  if (m.npe == 8)
    asm_list_kernel<3><<<g, 128, 0, s>>>(m, t, edges, eptr, list);
  else
    asm_list_kernel<2><<<g, 128, 0, s>>>(m, t, edges, eptr, list);
}

void launch_asm_fill(const AsmDev& S, const int* row, const int* cols, cudaStream_t s) {
  asm_fill_kernel<<<S.grid, 512, 0, s>>>(S, row, cols);
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
