// Host side of the in-place mixed-radix kernels: the choice of radices, the
// schedule and its twiddles, and the precision dispatch.
#include <algorithm>
#include <cstring>

#include "hostfft.h"
#include "ipfft.h"

namespace b2f {

// Thread instructions per point of one radix-R stage: about 9 for the
// shared-memory traffic, twiddle product and indexing, plus the butterfly
// (radix 16, 10.5 by count, is priced at 8: its 16 sub-lines store whole
// 128-byte segments and its half-warps never straddle two lines).
static double ip_stage_cost(uint32_t R) {
  static const double bf[17] = {0,    0,    2.0,  5.3,  4.0,  8.0,  7.3,  12.0, 6.5,
                                10.5, 10.0, 19.0, 9.3,  22.0, 14.0, 13.3, 8.0};
  return 9.0 + bf[R];
}

double ip_cost(const std::vector<uint32_t>& radices) {
  double c = 0;
  for (uint32_t R : radices) c += ip_stage_cost(R);
  return c;
}

namespace {
struct Search {
  size_t min_stages;
  std::vector<uint32_t> cur, best;
  double best_cost = 1e300;
  // radices in non-increasing order, bounded by the best found so far
  void go(uint64_t n, uint32_t top, double cost) {
    if (n == 1) {
      if (cur.size() >= min_stages && cost < best_cost) {
        best_cost = cost;
        best = cur;
      }
      return;
    }
    for (uint32_t R = top; R >= 2; --R) {
      if (n % R) continue;
      const double c = cost + ip_stage_cost(R);
      if (c >= best_cost) continue;
      cur.push_back(R);
      go(n / R, R, c);
      cur.pop_back();
    }
  }
};
}  // namespace

std::vector<uint32_t> ip_radices(uint64_t n, size_t min_stages) {
  uint64_t m = n;
  for (uint64_t p : {2, 3, 5, 7, 11, 13})
    while (m % p == 0) m /= p;
  if (n < 2 || m != 1) return {};
  Search s;
  s.min_stages = min_stages;
  s.go(n, 16, 0.0);
  return s.best;
}

bool ip_schedule(uint64_t n, bool row, bool conv, int pair, IpSched& sc,
                 std::vector<uint32_t>& radices, std::vector<std::complex<double>>& tw) {
  // a row line has a lead stage and at least one more, a convolution its
  // first stage and its centre
  std::vector<uint32_t> r = ip_radices(n, row || conv ? 2 : 1);
  if (r.empty()) return false;
  std::memset(&sc, 0, sizeof(sc));
  sc.N = (uint32_t)n;
  sc.R0 = 1;
  radices.clear();
  // rows lead with the largest radix (16 whenever it is one of them: 128-byte
  // f32 segments in the last stage's stores); the others ascend
  if (row) {
    sc.R0 = r.front();
    r.erase(r.begin());
    radices.push_back(sc.R0);
  }
  std::sort(r.begin(), r.end());
  if (r.size() > (size_t)kIpMaxStages) return false;
  radices.insert(radices.end(), r.begin(), r.end());
  sc.NS = (uint32_t)(n / sc.R0);
  sc.nst = (uint32_t)r.size();
  sc.dNS = make_fastdiv(sc.NS);
  sc.dR0 = make_fastdiv(sc.R0);
  // W_L^{r i}: r in groups of `pair` (zero-filled), i < m inside a group
  const RootProduct root(n);
  auto table = [&](uint32_t R, uint64_t L) {
    const uint64_t m = L / R, u = n / L;
    for (uint32_t q = 1; q < R; q += pair)
      for (uint64_t i = 0; i < m; ++i)
        for (int j = 0; j < pair; ++j)  // (q + j) i < L
          tw.push_back(q + j < R ? root((q + j) * i * u) : std::complex<double>(0.0, 0.0));
  };
  if (row) {
    sc.tw0 = (uint32_t)tw.size();
    table(sc.R0, n);
  }
  uint64_t L = sc.NS;
  for (uint32_t s = 0; s < sc.nst; ++s) {
    IpStage& st = sc.st[s];
    st.R = r[s];
    st.L = (uint32_t)L;
    st.m = (uint32_t)(L / r[s]);
    st.nj = sc.NS / r[s];
    st.dm = make_fastdiv(st.m);
    st.dR = make_fastdiv(r[s]);
    st.tw = (uint32_t)tw.size();
    table(r[s], L);
    L /= r[s];
  }
  return true;
}

uint32_t ip_frequency(const IpSched& sc, uint32_t k0, uint32_t pos) {
  uint32_t f = 0, x = pos;
  for (int s = (int)sc.nst - 1; s >= 0; --s) {
    f = f * sc.st[s].R + x % sc.st[s].R;
    x /= sc.st[s].R;
  }
  return k0 + sc.R0 * f;
}

cudaError_t launch_ip_f32(IpKind, bool, const IpParams&, unsigned, unsigned, size_t, cudaStream_t);
cudaError_t launch_ip_f64(IpKind, bool, const IpParams&, unsigned, unsigned, size_t, cudaStream_t);

cudaError_t launch_ip(Prec p, IpKind kind, bool col, const IpParams& prm, unsigned grid,
                      unsigned threads, size_t smem, cudaStream_t st) {
  switch (p) {
    case PREC_F32: return launch_ip_f32(kind, col, prm, grid, threads, smem, st);
    case PREC_F64: return launch_ip_f64(kind, col, prm, grid, threads, smem, st);
    case PREC_DF64: break;  // the ping-pong engine
  }
  return cudaErrorInvalidValue;
}

}  // namespace b2f
