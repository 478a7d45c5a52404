// Host check of the warp integrator's packed term tables (pdr_net.cpp,
// WarpTables::wtab): the device allocations are redirected to host memory, the
// right-hand side and the Jacobian assembly are replayed from the packed words
// lane by lane as chem_warp.cu runs them, and compared with a direct evaluation
// from the stoichiometry on seeded states.  Shared memory starts as NaN, so a
// value that is read before it is written shows.
// Usage: packed_check <species> <rates> <layout or -> <warp|block>
//   warp:  the network has packed tables, and they replay the stoichiometry
//   block: the network is beyond the packed fields: it loads, and has block tables only
// Exit 0 when every check holds.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

static cudaError_t host_malloc(void **p, size_t n) {
  *p = std::malloc(n ? n : 1);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
static cudaError_t host_copy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
#define cudaMalloc(p, n) host_malloc((void **)(p), (n))
#define cudaMemcpy(d, s, n, k) host_copy((d), (s), (n), (k))
#include "../../3d-pdr_gb300/csrc/pdr_net.cpp"
#undef cudaMalloc
#undef cudaMemcpy

#include <cmath>
#include <cstdio>
#include <random>

namespace pdr {
int cuda_fail(cudaError_t, const char *) { return -1; }
void set_error(const std::string &) {}
}  // namespace pdr

using namespace pdr;

static const double STALE = std::nan("");

static int replay(const HostNet &h, const WarpTables &T, std::mt19937_64 &rng) {
  const int n = h.neq, ONE = n + 1, W = 32, ld = W + 1;
  const auto terms = stoichiometry(h);
  const unsigned char *pl = reinterpret_cast<const unsigned char *>(T.wtab + T.wt_pl);
  const unsigned short *rab = reinterpret_cast<const unsigned short *>(T.wtab + T.wt_rab);
  const int *rt = T.wtab + T.wt_rt, *ht = T.wtab + T.wt_h, *pk = T.wtab + T.wt_pk, *bnd = T.wtab + T.wt_bnd;
  std::uniform_real_distribution<double> U(0.0, 1.0);
  int bad = 0;
  for (int trial = 0; trial < 4; trial++) {
    std::vector<double> x(n), rate(h.nreac);
    for (auto &v : x) v = std::pow(10.0, -20.0 * U(rng));
    for (auto &v : rate) v = std::pow(10.0, -8.0 - 12.0 * U(rng));
    const double nH = std::pow(10.0, 2.0 + 3.0 * U(rng));
    double xe = 0.0;
    for (int j = 0; j < n; j++) xe += h.xe[j] * x[j];
    std::vector<double> xs(x);
    xs.push_back(xe);
    xs.push_back(1.0);
    std::vector<double> kn(T.nkn + 1, 0.0);
    for (int r = 0; r < T.nreac; r++) kn[r] = rate[r] * (T.nh_mask[r] != 0.0 ? nH : 1.0);
    for (int e = 0; e < T.nkext; e++) {
      double k = 0.0;
      for (int q = T.kext_ptr[e]; q < T.kext_ptr[e + 1]; q++) k = std::fma((double)T.kext_rn[q].y, kn[T.kext_rn[q].x], k);
      kn[T.nreac + e] = k;
    }
    // the direct evaluation
    std::vector<double> f(n, 0.0), scale(n, 0.0), J((size_t)n * (n + 1), 0.0), js(n, 0.0);
    for (const Term &t : terms) {
      const int a = h.ra[t.r], b = (h.ode_kind[t.r] == ODE_BI) ? h.rb[t.r] : ONE;
      const double phi = kn[t.r] * xs[a] * xs[b], da = t.nu * kn[t.r] * xs[b], db = t.nu * kn[t.r] * xs[a];
      f[t.i] += t.nu * phi;
      scale[t.i] += std::fabs(t.nu * phi);
      J[(size_t)t.i * (n + 1) + a] += da;
      js[t.i] += std::fabs(da);
      if (b != ONE) {
        J[(size_t)t.i * (n + 1) + b] += db;
        js[t.i] += std::fabs(db);
      }
    }
    // rhs(): x_e's tree beside the pair products, the electron's pairs after it
    std::vector<double> P(T.nop, STALE), part(T.nparts + 1, STALE), v(W, 0.0);
    for (int j = 0; j < n; j++) P[j] = x[j];
    P[ONE] = 1.0;
    part[T.nparts] = 0.0;
    for (int j = 0; j < n; j++) v[j] = h.xe[j] * x[j];
    for (int k = 0; k < T.pk_len; k++) {
      const int o = k < 5 ? 16 >> k : 0;
      if (k == 5) P[n] = v[0];
      std::vector<double> nv(v), nP(P);
      for (int l = 0; l < W; l++) {
        const PairWord d(pk[k * W + l]);
        if (l < o) nv[l] = v[l] + v[l + o];
        else if (d.operand()) nP[d.operand()] = P[d.a()] * P[d.b()];
      }
      v = nv;
      P = nP;
    }
    for (int l = 0; l < W; l++) {
      double s = 0.0;
      int slot = pl[l];
      for (int t = 0; t < T.rhs_len4; t++) {
        const TermWord d((unsigned)rt[t * W + l]);
        if (d.rate() > T.nkn || d.operand() >= T.nop || slot > T.nparts) return 1000;
        s = std::fma(d.negative() ? -kn[d.rate()] : kn[d.rate()], P[d.operand()], s);
        if (d.last()) {
          part[slot++] = s;
          s = 0.0;
        }
      }
    }
    for (int i = 0; i < n; i++) {
      double got = 0.0;
      for (int k = 1; k <= T.plist_len; k++) got += part[pl[k * W + i]];
      if (!(std::fabs(got - f[i]) <= 1e-14 * scale[i] + 1e-300)) {
        if (bad < 5) std::printf("RHS species %d: %.17g vs %.17g (scale %.3g)\n", i, got, f[i], scale[i]);
        bad++;
      }
    }
    // assemble(), FP64 form
    std::vector<double> D(2 * (size_t)T.nreac, STALE), row((size_t)n * ld, 0.0), slots(T.nslots + 1, STALE);
    for (int r = 0; r < T.nreac; r++) {
      const int sa = rab[r] & 0xff, sb = rab[r] >> 8;
      D[r] = kn[r] * xs[sb];
      D[T.nreac + r] = (sb == ONE) ? 0.0 : kn[r] * xs[sa];
    }
    for (int l = 0; l < W; l++) {
      double s = 0.0;
      for (int t = 0; t < T.hlen4; t++) {
        const JacWord d(ht[t * W + l]);
        if (d.index() >= 2 * T.nreac) return 1001;
        s = std::fma((double)d.nu(), D[d.index()], s);
        if (d.kind()) {
          auto &to = d.kind() == 1 ? row : slots;
          if (d.kind() == 3 || d.target() >= (int)to.size()) return 1002;
          to[d.target()] = s;
          s = 0.0;
        }
      }
    }
    for (int b = 0; b < T.nbnd; b++) {
      const unsigned w = (unsigned)bnd[b];
      double acc = 0.0;
      for (unsigned q = (w >> 11) & 0xff; q < (w >> 19); q++) acc += slots[q];
      row[w & 0x7ff] = acc;
    }
    for (int i = 0; i < n; i++)
      for (int j = 0; j <= n; j++) {
        const double g = row[(size_t)i * ld + j], w = J[(size_t)i * (n + 1) + j];
        if (!(std::fabs(g - w) <= 1e-14 * js[i] + 1e-300)) {
          if (bad < 5) std::printf("J(%d,%d): %.17g vs %.17g\n", i, j, g, w);
          bad++;
        }
      }
  }
  return bad;
}

int main(int argc, char **argv) {
  if (argc != 5) { std::printf("usage: packed_check <species> <rates> <layout or -> <warp|block>\n"); return 2; }
  const bool warp = std::strcmp(argv[4], "warp") == 0;
  pdr_net net;
  const std::string err = load_network(argv[1], argv[2], std::strcmp(argv[3], "-") ? argv[3] : nullptr, net.host);
  if (!err.empty()) { std::printf("load: %s\n", err.c_str()); return 1; }
  const int rc = build_device_tables(&net);
  std::printf("neq %d nreac %d: rc %d, warp tables %d, block tables %d, pair rounds %d\n", net.host.neq, net.host.nreac, rc,
              (int)net.warp_ok, (int)net.cta_ok, net.warp.pk_len);
  if (rc != 0 || !net.cta_ok || net.warp_ok != warp) return 1;
  if (!warp) return 0;
  std::mt19937_64 rng(20261205u);
  const int bad = replay(net.host, net.warp, rng);
  std::printf("replay: %s (%d)\n", bad ? "MISMATCH" : "ok", bad);
  return bad ? 1 : 0;
}
