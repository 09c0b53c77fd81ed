// Tables and launchers of the assembled tangent (fem_asm.cu).
#pragma once
#include <algorithm>
#include <cstdint>
#include <exception>
#include <system_error>
#include <thread>
#include <vector>

#include "fem_internal.h"

namespace femb200 {

// A CTA of the persistent solve takes at least this many rows (two warps').
constexpr int kAsmMinRows = 64;

// f(begin, end) over [0, n) on up to 16 host threads, `grain` or more each.  A
// thread that cannot be had leaves its range to the caller's; an exception of
// any range is thrown here once all have ended.
template <typename F>
void parallel_ranges(int n, F f, int grain = 1024) {
  const int hw = std::max(1, (int)std::thread::hardware_concurrency());
  const int nt = std::max(1, std::min(std::min(hw, 16), n / grain));
  std::vector<std::exception_ptr> err(nt);
  auto part = [&](int t) {
    try {
      f((int)((int64_t)n * t / nt), (int)((int64_t)n * (t + 1) / nt));
    } catch (...) {
      err[t] = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(nt);
  int started = 1;
  try {
    for (; started < nt; ++started) pool.emplace_back(part, started);
  } catch (const std::system_error&) {
  }
  part(0);
  for (int t = started; t < nt; ++t) part(t);
  for (auto& th : pool) th.join();
  for (auto& e : err)
    if (e) std::rethrow_exception(e);
}

struct AsmHost {
  std::vector<int> cols;           // neighbours of each node, ascending (CSR with row)
  std::vector<int> row;
  std::vector<uint32_t> erow;      // [Nn + 1] edges to higher nodes before each node
  std::vector<uint32_t> lrow;      // [Nn + 1] (element, vertex pair) entries before each node's edges
  std::vector<uint32_t> slot0;     // slot (step * 32 + lane) of each row's first entry (entry k: + 32 k)
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

// AsmHost's lists on the device
struct AsmLists {
  const int *row, *cols;
  const uint32_t *erow, *lrow, *slot0;
};
// the edges' slots, and per edge the elements on it as (element * npe +
// vertex a) * npe + vertex b
void launch_asm_lists(const MeshDev& m, const AsmLists& t, uint2* edges, uint32_t* eptr, uint32_t* list, cudaStream_t s);
// local columns of every slot of the steps, from the neighbour lists
void launch_asm_fill(const AsmDev& S, const int* row, const int* cols, cudaStream_t s);
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
