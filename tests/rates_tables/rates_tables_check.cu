// Host check of the tables that the rate kernels read with 16-byte loads: the
// types they are made of must carry that alignment themselves, whatever else
// the linker places beside them.
// Usage: rates_tables_check; exit 0 when every check holds.
#include "../../3d-pdr_gb300/csrc/rates.cu"

#include <cstddef>
#include <cstdio>

namespace pdr {
int cuda_fail(cudaError_t, const char *) { return -1; }
void set_error(const std::string &) {}
}  // namespace pdr

using namespace pdr;

static int check_alignment() {
  int bad = 0;
  auto at_16 = [&](const char *what, size_t align, size_t size, size_t offset) {
    if (align % 16 == 0 && size % 16 == 0 && offset % 16 == 0) return;
    std::printf("%s: alignment %zu, size %zu, offset %zu\n", what, align, size, offset);
    bad++;
  };
  at_16("row of 2^(j/1024)", alignof(fp64::ExpRow), sizeof(fp64::ExpRow), 0);
  at_16("CO shielding patches", alignof(ShieldFast), sizeof(ShieldFast), offsetof(ShieldFast, patch));
  at_16("a patch", 16, sizeof(ShieldFast::patch[0][0]), 0);
  return bad;
}

int main() {
  const int bad = check_alignment();
  std::printf("alignment: %s\n", bad ? "WRONG" : "ok");
  return bad ? 1 : 0;
}
