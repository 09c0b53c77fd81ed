// Tables and launchers of the assembled tangent (fem_asm.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "fem_internal.h"

namespace femb200 {

// A CTA of the persistent solve takes at least this many rows (two warps').
constexpr int kAsmMinRows = 64;

// A node's elements are sorted by one warp (asm_neighbours_kernel), in the
// square of their number: above this many the mesh is refused.
constexpr int kAsmMaxValence = 8192;

// The rows dealt out to the CTAs and cut into slices, from the nodes' numbers
// of neighbours.
struct AsmHost {
  int grid = 0;
  std::vector<int> cta_row;        // [grid + 1] first row of each CTA
  std::vector<int> cta_slice;      // [grid + 1]
  std::vector<int> slice_step;     // [slices + 1] first step of each slice
  std::vector<int> slice_rows;     // [slices * 32] node of each lane, -1: none
  std::vector<uint32_t> slot0;     // slot (step * 32 + lane) of each row's first entry (entry k: + 32 k)
  std::vector<int> prefix;         // prefix[k]: most steps that the first k slices of a CTA have
  int max_slices = 0, max_pieces = 0;
};

// For a grid of at most `sms` CTAs.
void asm_cta_rows(const std::vector<int>& deg, int sms, AsmHost* out);
// False where the mesh does not fit the format (2^27 steps).
bool asm_slices(const std::vector<int>& deg, AsmHost* out);

struct AsmArgs {
  MeshDev m;
  AsmDev s;
  const DevMat<float>* matF;
  const float* payload;
};

// One block into its slot, rows of fixed DOFs (bits of fx) as zeros.
static __device__ __forceinline__ void asm_store(const AsmDev& S, uint32_t slot, float k00, float k01, float k02, float k10,
                                          float k11, float k12, float k20, float k21, float k22, int fx) {
  uint32_t* w = S.words + (size_t)(slot >> 5) * kAsmStepWords;
  const int lane = (int)(slot & 31u);
  if (fx & 1) k00 = k01 = k02 = 0.f;
  if (fx & 2) k10 = k11 = k12 = 0.f;
  if (fx & 4) k20 = k21 = k22 = 0.f;
  reinterpret_cast<float4*>(w + 16)[lane] = make_float4(k00, k01, k02, k10);
  reinterpret_cast<float4*>(w + 144)[lane] = make_float4(k11, k12, k20, k21);
  reinterpret_cast<float*>(w + 272)[lane] = k22;
}

// Neighbour lists on the device, and where the edges go.
struct AsmLists {
  const int* cols;       // node a's neighbours, ascending, from node_row[a] * (npe - 1) on
  const int* deg;        // [Nn] their number
  const uint32_t* erow;  // [Nn + 1] edges to higher nodes before each node
  const uint32_t* lrow;  // [Nn + 1] (element, vertex pair) entries before each node's edges
  const uint32_t* slot0;
};
// neighbours of every node; counts: [3][Nn] their number, those of higher
// nodes, and the (element, vertex pair) entries of the edges to them.  cand and
// cols: [node_row[Nn] * (npe - 1)]
void launch_asm_neighbours(const MeshDev& m, int* cand, int* cols, int* counts, cudaStream_t s);
// the columns of each CTA's rows outside its run, as one bit per node and their
// number; then as ascending lists.  bits0 and bits1 take half the CTAs each:
// [(grid + 1) / 2][(Nn + 31) / 32], zeroed
void launch_asm_halo_mark(const MeshDev& m, const AsmLists& t, const int* cta_row, int grid, uint32_t* bits0,
                          uint32_t* bits1, int* count, cudaStream_t s);
void launch_asm_halo_list(int n_nodes, const uint32_t* bits0, const uint32_t* bits1, const int* halo_ptr, int grid,
                          int* halo, cudaStream_t s);
// the edges' slots, and per edge the elements on it as (element * npe +
// vertex a) * npe + vertex b
void launch_asm_lists(const MeshDev& m, const AsmLists& t, uint2* edges, uint32_t* eptr, uint32_t* list, cudaStream_t s);
// local columns of every slot of the steps, from the neighbour lists
void launch_asm_fill(const MeshDev& m, const AsmDev& S, const AsmLists& t, cudaStream_t s);
// values at the tangent state of `payload`
void launch_asm(const AsmArgs& a, int model, cudaStream_t s);
// HEX8: places of the elements' blocks in s.list (hpos, [32 Ne], preset to
// kNoPlace), and the two assembly kernels (fem_hex8.cu)
constexpr uint32_t kNoPlace = 0xffffffffu;
void launch_asm_hex_places(const uint32_t* list, size_t n, uint32_t* hpos, cudaStream_t s);
void launch_asm_hex(const AsmArgs& a, int model, cudaStream_t s);
// dinv (and boff: nodal 3 x 3 block inverse) from the assembled blocks
void launch_asm_diag(const AsmArgs& a, float* dinv, float* boff, cudaStream_t s);

}  // namespace femb200
