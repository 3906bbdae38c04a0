// Parameters of the in-place mixed-radix kernels (ipfft.cuh) and the host
// side that prepares them (ipfft.cu).
#pragma once
#include <complex>
#include <vector>

#include "kernels.h"

namespace b2f {

// Stages on a sub-line: the longest one-CTA line of small primes (7^5, 5^6)
// has fewer.
constexpr int kIpMaxStages = 8;

// One in-place stage of radix R on sub-lines: blocks of L values, the R
// inputs (and outputs) of a butterfly m = L / R apart, nj butterflies a
// sub-line.  tw: W_L^{r i} for i < m, r = 1..R-1.
struct IpStage {
  uint32_t R, m, L, nj, tw;
  FastDiv dm, dR;
};

// A length-N transform: for rows a lead stage of radix R0 that splits the
// line into R0 sub-lines of NS = N / R0 values (twiddles W_N^{r i} at tw0),
// for columns R0 = 1; then nst stages on the sub-lines.  Decimation in
// frequency: value `pos` of sub-line k0 ends up holding frequency
// k0 + R0 * f, f the digit reversal of pos over the stage radices.
struct IpSched {
  uint32_t N, R0, NS, nst, tw0;
  FastDiv dNS, dR0;
  IpStage st[kIpMaxStages];
};

struct IpParams {
  const void* in;
  void* out;
  const void* tw;
  uint32_t G;       // lines (rows) or adjacent columns a CTA
  uint32_t lam;     // sub-lines a CTA, G * R0
  uint32_t pitch;   // rows: values between sub-lines (odd), columns: unused
  uint32_t LDl;     // rows: values between lines
  uint32_t flags;
  uint32_t n;       // points of the line in memory (N, or fewer for a convolution)
  FastDiv dlam, dG, dn;
  LineIO io;
  FastDiv d_tw;     // PF_TW_STORE, as LinesParams
  uint64_t tw_store_M;
  const void* tws_a;
  const void* tws_b;
  FastDiv d_tws;
  double scale;
  IpSched sc;
  const uint32_t* perm;  // Rader: g^q mod p
  const void* bhat;      // convolutions: spectrum / N at the position of each frequency, [pos][k0]
  const void* chirp;     // Bluestein: exp(-i pi k^2 / n)
  const void* rtw;       // real transforms: W_{2N}^k, k < N
  uint64_t nlines;       // real transforms: lines
};

enum IpKind : int { IP_LINES = 0, IP_RADER = 1, IP_BLUE = 2, IP_R2C = 3, IP_C2R = 4 };

// The radices of an in-place transform of 13-smooth n (at least `min_stages`
// of them), cheapest by the per-point estimate ip_cost; empty when there is
// none.
std::vector<uint32_t> ip_radices(uint64_t n, size_t min_stages);
// Estimated thread instructions per point of those stages.
double ip_cost(const std::vector<uint32_t>& radices);
// The schedule of length n (rows: with a lead stage) and its twiddles in
// the layout of a precision with `pair` values per 16 bytes.
bool ip_schedule(uint64_t n, bool row, bool conv, int pair, IpSched& sc,
                 std::vector<uint32_t>& radices, std::vector<std::complex<double>>& tw);
// Frequency held by value pos of sub-line k0.
uint32_t ip_frequency(const IpSched& sc, uint32_t k0, uint32_t pos);
// Values between the sub-lines of a row: odd, so that adjacent sub-lines fall
// into different banks.
inline uint32_t ip_pitch(uint32_t ns) { return ns | 1u; }

cudaError_t launch_ip(Prec p, IpKind kind, bool col, const IpParams& prm, unsigned grid,
                      unsigned threads, size_t smem, cudaStream_t st);
// Resident threads per SM the kernels of a precision are built for.
inline uint32_t ip_threads_per_sm(Prec p) { return p == PREC_F32 ? 1024u : 512u; }

}  // namespace b2f
