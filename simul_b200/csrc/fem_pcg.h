// Tables and launcher of the persistent PCG kernel (fem_pcg.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "fem_asm.h"
#include "fem_internal.h"

namespace femb200 {

// Static words of one CTA for the two-level phases, copied to shared memory
// once per launch: a header of kTabWords, then the lists it points at.
enum {
  TAB_CN0, TAB_NCN,            // coarse nodes whose residual this CTA adds up
  TAB_CPTR,                    // [ncn + 1] into seg_r
  TAB_SEG0, TAB_NSEG,          // segments: the CTA's rows of one lattice cell
  TAB_SPTR,                    // [nseg + 1] into the CTA's run of seg_lat
  TAB_SROW,                    // start of that run
  TAB_SPOS,                    // [nseg * 8] places of the segments' shares in seg_r
  TAB_LOC, TAB_NLOC,           // coarse nodes that the CTA's columns interpolate from
  TAB_TILES, TAB_NT,           // tile mode: (tile index, local row block | local column block << 16) pairs
  TAB_BLK, TAB_NL, TAB_BLK0,   // row blocks the tiles touch; first of the CTA's parts in ypart
  TAB_OPTR, TAB_OLIST,         // a block's tile outputs, ascending: local tile * (1 + parts) + (0: rows, else columns)
  TAB_YIDX,                    // [nloc * 3] list index of each local coarse DOF's block << 6 | place in the block
  TAB_YPTR, TAB_YLIST,         // parts of the blocks those DOFs lie in
  kTabWords = 24
};

// Device tables of the two-level phases.
struct PcgDev {
  const int* tab_ptr;        // [grid + 1] into tab
  const int* tab;
  const float4* seg_lat;     // [Nn] rows grouped by (CTA, cell): lattice coordinates, node (w, int bits)
  float4* seg_r;             // [n_seg * 8] restricted residual shares (segment, corner), by coarse node
  const int* cn_ptr;         // [n_cn + 1] each coarse node's shares
  int merged;                // every CTA adds up all of r_c
  float* ypart;              // tile mode: [parts][64] each CTA's part of y_c
  const uint4* col_corners;  // each CTA's columns (rows, then halo; CTA g's start at cta_row[g] + halo_ptr[g]):
                             // the cell's eight corners, 16-bit indices into the CTA's coarse nodes
  int max_tab, max_lblk, max_loc, max_tiles;  // largest per CTA (shared memory)
};

struct PcgCoarseHost {
  std::vector<int> tab_ptr, tab, seg_rows, cn_ptr;
  std::vector<uint4> col_corners;
  int n_seg = 0, n_parts = 0, max_tab = 0, max_lblk = 0, max_loc = 0, max_tiles = 0;
};
// node_cell / cell_corner: the lattice cell of each node, the cells' corner coarse nodes.
// False if a CTA's columns need more than 65536 coarse nodes.
// parts: 4 KB parts of a packed tile (0: the product runs on full rows).
// cta_row: [grid + 1] first row of each CTA; halo_ptr, halo: its other columns.
bool pcg_coarse_tables(const std::vector<int>& cta_row, const std::vector<int>& halo_ptr,
                       const std::vector<int>& halo, const std::vector<int>& node_cell, const std::vector<int>& cell_corner,
                       int n_cn, int parts, PcgCoarseHost* out);
// seg_lat from the rows in segment order and their lattice coordinates
void launch_pcg_seg_lat(const int* seg_rows, const float4* node_lat, int n, float4* out, cudaStream_t s);

struct PcgArgs {
  MeshDev m;
  AsmDev as;
  CoarseDev c;               // two-level: lattice and inverse
  PcgDev t;
  const double* b;           // right-hand side (3 doubles per node, fixed DOFs zero)
  float *r, *x, *q, *z;      // float4 per node
  float *p, *p2;             // the direction's two buffers
  const float* dinv;
  const float* boff;         // null: diagonal smoother
  CGState* cg;
  double* part;              // [4][grid] shares of the grid-wide sums
  unsigned int* bar;         // barrier arrivals (zero at launch)
  double rtol;
  int max_iter;
  int resident;              // the first slices of every CTA stay in shared memory
  int stages;                // ring stages per warp for the other slices and the coarse tiles (0: none)
  uint32_t stage_bytes;
  uint32_t res_bytes;        // shared memory of the resident slices; the rings follow
  uint32_t mat_bytes;        // both
  uint32_t scratch_bytes;    // phase-local arrays; the CTA's static words follow
  uint32_t items_off;        // the warps' item lists among the static words, max_items each
  int max_items;
  int tile_batch;            // tiles a CTA stages before it adds them up
};

// Shares of r_c (16 bytes each) up to which every CTA reads them all: up to
// here that takes 3,000 cycles, as the phase of its own without its barrier
// (4,000 more); 8,000 shares took 16,000.
constexpr int kPcgMergedShares = 2048;

// Shared memory of a launch (the split of the args above).  False if it does
// not fit.
bool pcg_plan(PcgArgs& a, bool two_level, const std::vector<int>& prefix, size_t* smem);
// One cooperative launch runs the whole solve (cg holds its end state).
cudaError_t launch_pcg(const PcgArgs& a, bool two_level, size_t smem, cudaStream_t s);

}  // namespace femb200
