// Host checks of the constant tables of the rate kernels.
//  align    the types read with 16-byte loads carry that alignment themselves,
//           whatever else the linker places beside them;
//  threads  the first calls of several host threads, on one device and on
//           several, upload the tables that a single thread uploads, and no call
//           returns before its device has them.  The copy to the device is
//           replaced by one that records its bytes.
// Usage: rates_tables_check align|threads; exit 0 when every check holds.
#include "../../3d-pdr_gb300/csrc/rates.cu"

#include <atomic>
#include <chrono>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <map>
#include <thread>

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

// ---- the copies to the device, recorded ----
static thread_local int t_device = 0;          // the device this thread has set
static std::mutex g_copies;
static std::map<std::pair<int, const void *>, std::vector<unsigned char>> g_device;   // (device, symbol) -> bytes

extern "C" cudaError_t cudaMemcpyToSymbol(const void *symbol, const void *src, size_t n, size_t, cudaMemcpyKind) {
  std::vector<unsigned char> bytes(n);
  std::memcpy(bytes.data(), src, n);
  std::this_thread::sleep_for(std::chrono::microseconds(200));   // a copy takes its time
  std::lock_guard<std::mutex> lk(g_copies);
  g_device[{t_device, symbol}] = bytes;
  return cudaSuccess;
}

static int check_threads() {
  // the tables of one thread alone
  t_device = 63;
  if (upload_shield_tables(63) != 0) return 1;
  const auto want_shield = g_device[{63, (const void *)&c_shield}], want_fast = g_device[{63, (const void *)&d_shield}];
  if (want_shield.size() != sizeof(ShieldTables) || want_fast.size() != sizeof(ShieldFast)) return 1;
  std::atomic<int> bad{0};
  // 30 devices; in every round two of them get their first calls from eight threads at once
  for (int round = 0; round < 30; round++) {
    std::atomic<int> ready{0};
    std::vector<std::thread> th;
    for (int k = 0; k < 8; k++)
      th.emplace_back([&, k] {
        const int dev = 2 * round + (k & 1);
        t_device = dev;
        ready++;
        while (ready < 8) {}
        if (upload_shield_tables(dev) != 0) bad++;
        std::lock_guard<std::mutex> lk(g_copies);
        if (g_device[{dev, (const void *)&c_shield}] != want_shield) bad++;
        if (g_device[{dev, (const void *)&d_shield}] != want_fast) bad++;
      });
    for (auto &t : th) t.join();
  }
  return bad;
}

int main(int argc, char **argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what != "align" && what != "threads") { std::printf("usage: rates_tables_check align|threads\n"); return 2; }
  const int bad = what == "align" ? check_alignment() : check_threads();
  std::printf("%s: %s (%d)\n", what.c_str(), bad ? "WRONG" : "ok", bad);
  return bad ? 1 : 0;
}
