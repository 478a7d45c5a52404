// launch_shape.h -- block sizes of the warp integrator (host code).
#pragma once

#include <cstddef>
#include <vector>

#include "../../include/pdrgpu.h"

namespace pdr {

// Warps of an SM in the 168-register variants (2 and 3), in one block by default:
// its warps then share one copy of the term tables.  FP64, 32,768 cells: 1,024 ms
// (three 4-warp blocks 1,025, six 2-warp blocks 1,028); 2,500: 102 to 105 (104 to
// 109, 105 to 113); from 16 to 1,824 cells the three differ by less than two runs
// of one of them.
constexpr int WARPS_168 = 12;

// register variant: the caller's, or the fastest measured (mixed 128 registers
// with 16 warps per SM, FP64 168 registers)
inline int warp_variant(const pdr_chem_opts &o, bool mixed) {
  return (o.reg_variant >= 0 && o.reg_variant <= 3) ? o.reg_variant : (mixed ? 1 : 2);
}

// Warps per block of variant rv; 0: the caller's number is refused (at most 8, and
// 4 in variants 2 and 3).  By default 8, and in variants 2 and 3 the SM's twelve
// where one warp's arrays (per_warp bytes) leave room for that beside the term
// tables in a block's `optin` bytes, else 4.  A caller who counts blocks
// (blocks_per_sm) counts 4-warp blocks there.
inline int warp_block(const pdr_chem_opts &o, int rv, size_t per_warp, size_t tables, size_t optin) {
  if (o.warps_per_block > (rv >= 2 ? 4 : 8)) return 0;
  if (o.warps_per_block > 0) return o.warps_per_block;
  if (rv < 2) return 8;
  return o.blocks_per_sm <= 0 && per_warp * WARPS_168 + tables + 1024 <= optin ? WARPS_168 : 4;
}

// The shapes that the autotuner times; warps_per_block 0 is the variant's default
// block.  The 12-warp blocks of variant 2, the FP64 default, are among them where
// the sample fills one on every SM it may use: smaller samples cannot tell them from
// the others (see WARPS_168).  (Variant 3 is 3 % slower in blocks of any size.)
struct WarpCandidate {
  int warps_per_block, reg_variant, refill;
};
inline std::vector<WarpCandidate> warp_candidates(int ncell_sample, int sms) {
  std::vector<WarpCandidate> c = {{4, 0, 0}, {2, 0, 0}, {4, 1, 0}, {8, 1, 0}, {4, 2, 0}, {2, 2, 0}, {4, 3, 0}, {4, 1, 1}};
  if (ncell_sample >= WARPS_168 * sms) c.push_back({0, 2, 0});
  return c;
}

}  // namespace pdr
