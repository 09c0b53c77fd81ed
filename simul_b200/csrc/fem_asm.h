// Tables and launchers of the assembled tangent (fem_asm.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "fem_internal.h"

namespace femb200 {

// A CTA of the persistent solve takes at least this many rows (two warps').
constexpr int kAsmMinRows = 64;

struct AsmHost {
  std::vector<int> cols;           // neighbours of each node, ascending (CSR with row)
  std::vector<int> row;
  std::vector<int2> entry;         // per slot of a step (step * 32 + lane): node, column (-1: padding)
  std::vector<uint2> edges;        // slots of (a, b) and (b, a) of each edge a < b
  std::vector<uint32_t> eptr;      // [edges + 1] into list
  std::vector<uint32_t> list;      // (element * npe + vertex a) * npe + vertex b, per edge
  int grid = 0;
  std::vector<int> cta_row;        // [grid + 1] first row of each CTA
  std::vector<int> cta_slice;      // [grid + 1]
  std::vector<int> slice_step;     // [slices + 1] first step of each slice
  std::vector<int> slice_rows;     // [slices * 32] node of each lane, -1: none
  std::vector<int> halo_ptr, halo;
  std::vector<int> prefix;         // prefix[k]: most steps that the first k slices of a CTA have
  int max_slices = 0, max_halo = 0, max_cols = 0, max_pieces = 0;
};

// Tables for a grid of at most `sms` CTAs.  False where the mesh does not fit
// the format (2^27 steps, 65,536 columns of a CTA, 32-bit lists).
bool build_asm_host(const int4* conn, int Nn, int Ne, int npe, int sms, AsmHost* out);

struct AsmArgs {
  MeshDev m;
  AsmDev s;
  const DevMat<float>* matF;
  const float* payload;
};

// local columns of every slot (row: CTA of each node's row; cols: the slots' columns, -1: padding)
void launch_asm_fill(const AsmDev& S, const int2* entry, cudaStream_t s);
// values at the tangent state of `payload`
void launch_asm(const AsmArgs& a, int model, cudaStream_t s);
// dinv (and boff: nodal 3 x 3 block inverse) from the assembled blocks
void launch_asm_diag(const AsmArgs& a, float* dinv, float* boff, cudaStream_t s);

}  // namespace femb200
