// Host check of the warp integrator's block sizes (launch_shape.h): what a caller's
// options give, what is refused, and that the autotuner reaches the default shape
// of either precision.
#include "../../3d-pdr_gb300/csrc/launch_shape.h"

#include <cstdio>

using namespace pdr;

static int bad = 0;
static void expect(const char *what, int got, int want) {
  if (got == want) return;
  std::printf("%s: %d, not %d\n", what, got, want);
  bad++;
}

int main() {
  const size_t optin = 227 * 1024, tables = 20000, per_warp = 14000;
  pdr_chem_opts o{};
  o.reg_variant = -1;
  auto block = [&](int wpb, int rv, int bps, size_t pw) {
    o.warps_per_block = wpb;
    o.blocks_per_sm = bps;
    return warp_block(o, rv, pw, tables, optin);
  };
  expect("FP64 variant", warp_variant(o, false), 2);
  expect("mixed variant", warp_variant(o, true), 1);
  // defaults
  for (int rv : {0, 1}) expect("default, variants 0 and 1", block(0, rv, 0, per_warp), 8);
  for (int rv : {2, 3}) {
    expect("default, variants 2 and 3", block(0, rv, 0, per_warp), 12);
    expect("default, a network whose arrays are larger", block(0, rv, 0, 20000), 4);
    // a caller who counts blocks counts 4-warp blocks, as blocks_per_sm 1 and 2 of the 12 warps an SM holds
    for (int bps : {1, 2, 3}) expect("blocks counted", block(0, rv, bps, per_warp), 4);
  }
  // the caller's own
  for (int rv = 0; rv < 4; rv++)
    for (int wpb = 1; wpb <= 13; wpb++) expect("explicit", block(wpb, rv, 0, per_warp), wpb <= (rv < 2 ? 8 : 4) ? wpb : 0);
  // the autotuner: each candidate is accepted, and with a sample that fills the SMs the defaults are among them
  for (int n : {64, 1823, 1824, 32768}) {
    bool fp64 = false, mixed = false;
    for (const WarpCandidate &c : warp_candidates(n, 152)) {
      const int b = block(c.warps_per_block, c.reg_variant, 0, per_warp);
      if (b < 1) expect("candidate", b, c.warps_per_block);
      fp64 |= c.reg_variant == 2 && b == 12 && c.refill == 0;
      mixed |= c.reg_variant == 1 && b == 8 && c.refill == 0;
    }
    expect("the autotuner reaches the FP64 default", fp64, n >= 1824);
    expect("the autotuner reaches the mixed default", mixed, 1);
  }
  std::printf("%s\n", bad ? "WRONG" : "ok");
  return bad != 0;
}
