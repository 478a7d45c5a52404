// Host check of the rounds in which the block integrator eliminates the leaf
// columns of its sparse Newton matrix (pdr_net.cpp gather_plan): FP32 matrices
// over each network's pattern, eliminated round by round as the device does it,
// against a row-by-row elimination.  The two take the same products in the same
// order, so every stored value agrees bit for bit.
// Usage: gather_check <data dir> <network>...; exit 0 when every check holds.
#include "../../3d-pdr_gb300/csrc/pdr_net.cpp"

#include <cmath>
#include <cstring>
#include <random>

namespace pdr {
int cuda_fail(cudaError_t, const char *) { return -1; }
void set_error(const std::string &) {}
}  // namespace pdr

using namespace pdr;

static int check_network(const std::string &dir, const std::string &name) {
  HostNet h;
  std::string err = load_network((dir + "/species_" + name + ".d").c_str(), (dir + "/rates_" + name + ".d").c_str(),
                                 (dir + "/layout_" + name + ".d").c_str(), h);
  if (!err.empty()) { std::printf("%s: load: %s\n", name.c_str(), err.c_str()); return 1; }
  const int n = h.neq, ONE = n + 1;
  std::vector<std::pair<int, int>> ent;
  for (auto &t : stoichiometry(h)) {
    if (h.ode_kind[t.r] == ODE_XRAY) continue;
    const int a = h.ra[t.r], b = (h.ode_kind[t.r] == ODE_BI) ? h.rb[t.r] : ONE;
    if (a <= n) ent.push_back({t.i, a});
    if (b <= n) ent.push_back({t.i, b});
  }
  const int G = std::max(64, (n + 31) / 32 * 32);
  SparsePlan sp;
  if (!sparse_plan(n, ent, h.xe, G, sp) || !gather_plan(sp, G)) { std::printf("%s: no plan\n", name.c_str()); return 1; }
  const int N = sp.N, a = sp.a, total = sp.total, ngroup = (int)sp.g_group.size() - 2;
  int bad = 0;
  if ((int)sp.g_elem.size() != (sp.nround + 1) * G || (int)sp.g_prod.size() != 4 * (ngroup + 2) * G) bad++;
  std::mt19937 rng(7);
  std::uniform_real_distribution<float> U(-1.0f, 1.0f);
  for (int trial = 0; trial < 3; trial++) {
    std::vector<float> A(total + 1, 0.0f), B;
    for (int i = 0; i < N; i++)
      for (int j = 0; j < N; j++)
        if (sp.F[i].test(j)) A[sp.loc(i, j)] = U(rng) + (i == j ? 6.0f : 0.0f);
    B = A;
    // row by row
    std::vector<float> dinv(a, 0.0f), piv(a, 0.0f);
    for (int i = 0; i < N; i++) {
      for (int k = 0; k < std::min(i, a); k++) {
        if (!sp.F[i].test(k)) continue;
        float &l = A[sp.loc(i, k)];
        l *= dinv[k];
        for (int j = k + 1; j < N; j++)
          if (sp.F[k].test(j)) {
            float &v = A[sp.loc(i, j)];
            v = std::fma(-l, A[sp.loc(k, j)], v);
          }
      }
      if (i < a) dinv[i] = 1.0f / A[sp.loc(i, i)];
    }
    // round by round; what a round stores is seen after the next barrier only
    std::vector<float> seen = B, seen_piv = piv, s(G);
    int round = 0;
    for (int t = 0; t < G; t++) s[t] = seen[sp.g_elem[t].x & 0xffff];
    for (int g = 0; g < ngroup; g++) {
      for (int t = 0; t < G; t++)
        for (int c = 0; c < 4; c++) {
          const unsigned w = sp.g_prod[(size_t)(4 * g + c) * G + t];
          s[t] = std::fma(-seen[w & 0xffff], seen[w >> 16], s[t]);
        }
      if (sp.g_group[g] & 1) {
        for (int t = 0; t < G; t++) {
          const int2 el = sp.g_elem[(size_t)round * G + t];
          const int kind = el.x >> 16;
          if (kind == 3) s[t] *= seen_piv[el.y];
          if (kind == 2) piv[el.y] = 1.0f / s[t];
          if (kind) B[el.x & 0xffff] = s[t];
        }
        round++;
        if (sp.g_group[g] & 2) { seen = B; seen_piv = piv; }
        for (int t = 0; t < G; t++) s[t] = seen[sp.g_elem[(size_t)round * G + t].x & 0xffff];
      }
    }
    if (round != sp.nround || std::memcmp(seen.data(), A.data(), 4 * (size_t)total) ||
        std::memcmp(seen_piv.data(), dinv.data(), 4 * (size_t)a))
      bad++;
    for (float v : A) bad += !std::isfinite(v);
  }
  std::printf("%s: %d rounds, %d groups of four products, %d failures\n", name.c_str(), sp.nround, ngroup, bad);
  return bad ? 1 : 0;
}

int main(int argc, char **argv) {
  int rc = argc > 2 ? 0 : 1;
  for (int k = 2; k < argc; k++) rc |= check_network(argv[1], argv[k]);
  return rc;
}
