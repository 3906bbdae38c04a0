// Long lines of a batch (a line, or a Bluestein convolution, too long for
// one CTA's shared memory): two or three HBM passes of a persistent kernel.
//
// A length T = N1 * N2 FFT (T = N, or the convolution length M) runs as
//   column pass: for each n2, FFT_N1 over n1 of x[N2 n1 + n2], times
//                W_T^{n2 k1}, into the scratch row k1 (natural [k1][n2]);
//   row pass:    for each k1, FFT_N2 over n2 of scratch row k1, giving
//                X[k1 + N1 k2].
// A task is G adjacent columns or rows of one line (up to 4,384 values), on
// the in-place stages of ipfft.cuh: columns interleaved, first stage from
// and last stage to global memory in segments of G values; rows with a lead
// stage along the row, the last stage storing G adjacent rows' outputs
// together.
//
// Bluestein lines (convolution M = N1 N2) take three passes: the chirped
// column pass; a middle row pass that runs the forward row FFT, multiplies
// by the chirp spectrum, and runs the row half of the inverse FFT
// (y[N2 n1 + n2] = sum_k1 W_N1^{-n1 k1} W_M^{-n2 k1} sum_k2 W_N2^{-n2 k2} Y[k1 + N1 k2],
// computed on conjugates with the forward codelets) in place on the rows,
// never leaving the digit-reversed order in between; and the inverse column
// pass, chirped into the output.  One scratch region of M values per line.
//
// Up to kLongSpread tasks a resident CTA are dealt out, task k of CTA b being
// b + k * gridDim.x: a batch with fewer tasks than CTAs has one a CTA.  More
// come from a work queue in chunks of consecutive tasks (mostly one line),
// which evens out what tasks of many lengths take.  A task's record and length
// descriptor arrive by asynchronous copies two and three tasks ahead, the
// two-level tables of its length (W_M, and the chirp) when they differ from
// the last task's.  The data itself is not prefetched: four CTAs of 256
// threads and 64 registers share an SM and cover each other's loads (fetching
// the next task's data or tables into L2 ahead cost its instructions and 3 %
// instead).
//
// What bounds it: instruction issue, 339 thread instructions per point of
// the first 4,000 lines of the mixed workload (540 with the earlier ping-pong
// stages and 16 warps an SM) at 43-46 % of the issue slots, behind loads,
// barriers and, as neighbouring tasks run other radices, instruction fetch.
// All 20,000 lines: 4.32 -> 3.08 ms; 512 x 65536: 404 -> 244 us; 512 x 65521 (Bluestein): 1994
// -> 1026; 1118 x 30011: 1676 -> 853; 6706 x 5003: 2122 -> 931.
#pragma once
#include "batch.cuh"
#include "ipfft.cuh"

namespace b2f {

constexpr uint32_t kLongThreads = 256;
constexpr uint32_t kLongChunk = 4;  // consecutive tasks per work-queue claim
// Tasks a resident CTA up to which they are dealt out.  A CTA holds four to
// eight tasks of the queue from its start, so that small batches ran theirs
// one after the other in a quarter of the CTAs: us from the queue / dealt out,
// without a counter to zero, one line of 3,001 points 56.9 / 19.0, 300 of 6,000
// 67.8 / 22.8, 64 of 65,536 87.7 / 39.6.  With 20 to 32 tasks a CTA dealing is still ahead (20,000 lines
// of up to 15,000 points 783 / 752, 2,400 of 20,000 442 / 412); at 40 to 65
// the queue is (10,000 of up to 65,536 1597 / 1631, 4,800 of 10,007 1273 /
// 1316), at 100 neither (20,000 of up to 65,536).
constexpr uint32_t kLongSpread = 32;
// k_long_pass claims the first two chunks before its loop and every later
// one when the chunk before it opens (three tasks ahead): that covers every
// chunk only when a chunk holds at least three tasks
static_assert(kLongChunk >= 3, "the prologue claims chunks 0 and 1 only");
// Values a task holds in shared memory: sixteen columns of 272 points or rows of 256.  With
// the tables (at most 2048 values) four CTAs share an SM.
constexpr uint32_t kLongTaskValues = 4384;

enum LongPassKind : uint32_t {
  LP_COL = 0,    // smooth line, column pass: x -> scratch
  LP_ROW = 1,    // smooth line, row pass: scratch -> out
  LP_BCOL1 = 2,  // Bluestein, chirped column pass: x -> scratch
  LP_BMID = 3,   // Bluestein, rows: FFT, spectrum product, inverse-row FFT, in place
  LP_BCOL3 = 4,  // Bluestein, inverse column pass, chirped: scratch -> out
};

struct LongLenDesc {
  uint32_t N, M, N1, N2;
  uint32_t blue;
  float scale;
  const c32* bhat;  // Bluestein: spectrum of the conjugate chirp / M, row k1 at k1 * N2 in the
                    // order the row's frequencies take ([pos][k0])
  // two-level tables (offsets into the twiddle table) with rows of
  // L = 2^tsplit >= sqrt(M): W_M^j = W_M^{L a} * W_M^b, j = a L + b,
  // a < tn = ceil(M / L) <= 512, b < L <= 512; the Bluestein chirp W_2N^q
  // likewise with rows of 2^csplit >= sqrt(2N)
  uint32_t ta, tb, tn, tsplit;
  uint32_t ca, cb, cn, csplit;
  uint32_t minv, mshift;  // n^2 mod 2N (mod_square)
  IpRows c, r;            // columns of N1, rows of N2
};

// One task: G adjacent columns or rows of one line.  Self-contained, so
// that the kernel can prefetch it with asynchronous copies (no dependent
// load of a line record).
struct LongTask {
  uint64_t base;     // complex offset of the line in the input buffer
  uint64_t scratch;  // complex offset of its scratch region (M values)
  uint32_t len;      // index into the length table
  uint32_t g0;       // first column (column passes) or row (row passes) of the task
  uint64_t obase;    // complex offset of the line in the output buffer
};
static_assert(sizeof(LongTask) == 32, "task records are copied as four 8-byte words");

struct LongParams {
  const c32* in;
  c32* out;
  c32* scratch;
  const c32* tw;
  const LongLenDesc* lens;
  const LongTask* tasks;
  uint32_t ntasks;
  uint32_t phase;    // 1: column pass, 2: row pass, 3: Bluestein inverse columns
  uint32_t inverse;
  uint32_t cap;      // complex elements of the data buffer
  unsigned int* counter;  // work queue: chunks of kLongChunk tasks handed out in order
};

FFT_D void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
FFT_D void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// W^j from a two-level table in shared memory (a shift and a mask).
struct TwoLevel {
  const c32* hi;
  const c32* lo;
  uint32_t sh;
  FFT_D c32 at(uint32_t j) const { return cmul(hi[j >> sh], lo[j & ((1u << sh) - 1)]); }
};

// n^2 mod m for n < 2^17, m = 2N < 2^19: the quotient estimate is
// umulhi(n^2 / 4, minv) >> mshift with minv = (2^(32+b) - 1) / m, 2^b <= m <
// 2^(b+1), mshift = b - 2.  Before the shift it is short by less than 3
// (the two dropped bits, minv's and umulhi's truncation), so after it by at
// most 1 when 2^mshift >= 3: one conditional subtraction.
FFT_D uint32_t mod_square(uint32_t n, uint32_t m, uint32_t minv, uint32_t mshift) {
  const uint64_t sq = (uint64_t)n * n;
  const uint32_t q = __umulhi((uint32_t)(sq >> 2), minv) >> mshift;
  const uint32_t r = (uint32_t)sq - q * m;
  return r >= m ? r - m : r;
}

// The chirp exp(-i pi n^2 / N).
struct LongChirp {
  TwoLevel t;
  uint32_t N, minv, mshift;
  FFT_D c32 at(uint32_t n) const { return t.at(mod_square(n, 2 * N, minv, mshift)); }
};

// ---- global memory ends; g counts the task's columns or rows
struct LongColLoad {  // point i of column g at src[N2 i + g]
  const c32* src;
  uint32_t N2;
  bool cj;
  template <int R>
  FFT_D void load(c32* v, uint32_t g, uint32_t i, uint32_t step) const {
    const c32* a = src + (uint64_t)N2 * i + g;
    const uint64_t d = (uint64_t)N2 * step;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = a[q * d];
    if (cj) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q].im = -v[q].im;
    }
  }
};

struct LongChirpLoad {  // the same of the chirped, zero-padded line; c0: first column
  const c32* src;
  LongChirp ch;
  uint32_t N2, c0;
  bool cj;
  template <int R>
  FFT_D void load(c32* v, uint32_t g, uint32_t i, uint32_t step) const {
    const uint32_t n = N2 * i + c0 + g, dn = N2 * step;
    // M >= 2N - 1: rows below N1 / 2 hold data, so the first half of a
    // butterfly's points, rounded up
    constexpr int H = (R + 1) / 2;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = czero<float>();
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (n + q * dn < ch.N) v[q] = src[n + q * dn];
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (n + q * dn < ch.N) {
        if (cj) v[q].im = -v[q].im;
        v[q] = cmul(v[q], ch.at(n + q * dn));
      }
  }
};

struct LongColStore {  // scratch[N2 k + c] = v * W_M^{c k}
  c32* dst;  // scratch + first column
  TwoLevel t;
  uint32_t N2, c0;
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t k, uint32_t step) const {
    const uint32_t c = c0 + g;
    uint32_t e = c * k;  // c k < M
    const uint32_t de = c * step;
    c32* a = dst + (uint64_t)N2 * k + g;
    const uint64_t d = (uint64_t)N2 * step;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      *a = cmul(v[q], t.at(e));
      e += de;
      a += d;
    }
  }
};

struct LongRowStore {  // out[k1 + N1 k], scaled, conjugated back for inverse transforms
  c32* dst;  // out + first row
  uint32_t N1;
  float sc, sci;
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t k, uint32_t step) const {
    c32* a = dst + (uint64_t)N1 * k + g;
    const uint64_t d = (uint64_t)N1 * step;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      *a = c32{v[q].re * sc, v[q].im * sci};
      a += d;
    }
  }
};

struct LongMidStore {  // scratch row k1, position i: v * W_M^{i k1}
  c32* dst;  // scratch row of the task's first row
  TwoLevel t;
  uint32_t N2, k0;
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t i, uint32_t step) const {
    const uint32_t k1 = k0 + g;
    uint32_t e = i * k1;
    const uint32_t de = step * k1;
    c32* a = dst + (uint64_t)N2 * g + i;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      a[q * step] = cmul(v[q], t.at(e));
      e += de;
    }
  }
};

struct LongChirpStore {  // out[n] = conj(v) * chirp(n), n = N2 k + c < N
  c32* dst;  // out
  LongChirp ch;
  uint32_t N2, c0;
  float sc, sci;
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t k, uint32_t step) const {
    const uint32_t n0 = N2 * k + c0 + g, dn = N2 * step;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const uint32_t n = n0 + q * dn;
      if (n < ch.N) {
        const c32 x = cmul(conj(v[q]), ch.at(n));
        dst[n] = c32{x.re * sc, x.im * sci};
      }
    }
  }
};

struct LongConvOp {
  const c32* bhat;  // spectrum of the task's first row
  uint32_t N2;
  FFT_D const c32* spectrum(uint32_t g) const { return bhat + (uint64_t)g * N2; }
  FFT_D void dc(uint32_t, c32, c32&) const {}
};

FFT_D void long_copy(c32* dst, const c32* src, uint32_t n) {
  for (uint32_t e = threadIdx.x; e < n; e += kLongThreads) cp_async8(dst + e, src + e);
}

// Issues the copies of a length's two-level tables that phase PH reads into
// T: W_M at 0 and tn, the chirp behind it (or at 0 when the phase needs no
// W_M).
template <uint32_t PH>
FFT_D void long_tables(const LongParams& p, const LongLenDesc& d, c32* T) {
  if (PH != 3) {
    long_copy(T, p.tw + d.ta, d.tn);
    long_copy(T + d.tn, p.tw + d.tb, 1u << d.tsplit);
    T += d.tn + (1u << d.tsplit);
  }
  if ((PH == 1 && d.blue) || PH == 3) {
    long_copy(T, p.tw + d.ca, d.cn);
    long_copy(T + d.cn, p.tw + d.cb, 1u << d.csplit);
  }
}

// One task of phase PH; the tables have been issued as a cp.async group of
// their own when `fresh` (one younger group may be in flight).  The caller
// synchronises before and after.
template <uint32_t PH>
FFT_D void long_task(const LongParams& p, const LongLenDesc& d, const LongTask& ln, c32* sm,
                     const c32* T, bool fresh) {
  const uint32_t tid = threadIdx.x, g0 = ln.g0;
  const bool inv = p.inverse != 0;
  const TwoLevel tw{T, T + d.tn, d.tsplit};
  if (fresh && (PH == 1 && d.blue)) {  // the chirp tables serve the first loads
    cp_async_wait<1>();
    __syncthreads();
    fresh = false;
  }
  auto landed = [&] {
    if (fresh) {
      cp_async_wait<1>();
      __syncthreads();
    }
  };
  if constexpr (PH == 1) {
    const Ip<float, true, IpRows> ip{d.c, sm, p.tw, tid, kLongThreads, min(d.c.G, d.N2 - g0)};
    if (d.blue) {
      const c32* Tc = T + d.tn + (1u << d.tsplit);
      const LongChirp ch{{Tc, Tc + d.cn, d.csplit}, d.N, d.minv, d.mshift};
      ip.first(LongChirpLoad{p.in + ln.base, ch, d.N2, g0, inv});
    } else {
      ip.first(LongColLoad{p.in + ln.base + g0, d.N2, inv});
    }
    landed();
    ip.forward_mids();
    ip.last(LongColStore{p.scratch + ln.scratch + g0, tw, d.N2, g0});
  } else if constexpr (PH == 2) {
    const Ip<float, false, IpRows> ip{d.r, sm, p.tw, tid, kLongThreads, min(d.r.G, d.N1 - g0)};
    c32* rows = p.scratch + ln.scratch + (uint64_t)g0 * d.N2;
    ip.first(IpLoad<float>{rows, (int64_t)d.N2, 1, 0});
    landed();
    ip.forward_mids();
    if (d.blue) {
      ip.centre(LongConvOp{d.bhat + (uint64_t)g0 * d.N2, d.N2});
      ip.inverse_mids();
      ip.final_dit(LongMidStore{rows, tw, d.N2, g0});
    } else {
      ip.last(LongRowStore{p.out + ln.obase + g0, d.N1, d.scale, inv ? -d.scale : d.scale});
    }
  } else {
    const Ip<float, true, IpRows> ip{d.c, sm, p.tw, tid, kLongThreads, min(d.c.G, d.N2 - g0)};
    ip.first(LongColLoad{p.scratch + ln.scratch + g0, d.N2, false});
    landed();
    ip.forward_mids();
    const LongChirp ch{{T, T + d.cn, d.csplit}, d.N, d.minv, d.mshift};
    ip.last(LongChirpStore{p.out + ln.obase, ch, d.N2, g0, d.scale, inv ? -d.scale : d.scale});
  }
}

// Persistent kernel of one long-line phase PH (= p.phase).  Tasks that are
// not DEALT out (kernels of their own: asking at run time costs the 20,000
// mixed lines 1 %) come in chunks of kLongChunk consecutive ones from
// a work queue (one atomicAdd per chunk), claimed a chunk ahead: the claim for
// the CTA's chunk c + 1 is issued when it starts using chunk c and its result
// is stored after that iteration's task, so the atomic's latency is hidden
// too.  While iteration k runs task k, asynchronous copies bring the length
// descriptor of task k + 2 (a ring of three) and the record of task k + 3 (a
// ring of four).
// Dynamic shared memory: p.cap values of data, then the tables.
template <uint32_t PH, bool DEALT>
__global__ void __launch_bounds__(kLongThreads, 4) k_long_pass(const __grid_constant__ LongParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LongLenDesc s_len[3];
  __shared__ LongTask s_task[4];
  __shared__ uint32_t s_chunk[4];  // first task of the CTA's chunk c, at c % 4
  static_assert(sizeof(LongLenDesc) % 8 == 0, "descriptors are copied as 8-byte words");
  c32* const data = reinterpret_cast<c32*>(smem_raw);
  c32* const tab = data + p.cap;
  const uint32_t tid = threadIdx.x;
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  // the CTA's k-th task (of the queue: its chunk claimed and visible); kNone
  // from the first one past the end (the queue hands out chunks in increasing order)
  auto task_of = [&](uint32_t k) -> uint32_t {
    const uint64_t t = DEALT ? blockIdx.x + (uint64_t)k * gridDim.x
                             : (uint64_t)s_chunk[(k / kLongChunk) & 3] + k % kLongChunk;
    return t < p.ntasks ? (uint32_t)t : kNone;
  };
  if (tid == 0 && !DEALT) {
    s_chunk[0] = atomicAdd(p.counter, 1u) * kLongChunk;
    s_chunk[1] = atomicAdd(p.counter, 1u) * kLongChunk;
  }
  __syncthreads();
  uint32_t held = kNone;  // length whose tables are in `tab`
  uint32_t ring0 = kNone, ring1 = kNone, ring2 = kNone;  // length each descriptor slot holds
  // record of task k into s_task[k % 4]
  auto fetch_task = [&](uint32_t k) {
    const uint32_t t = task_of(k);
    if (t != kNone && tid < 4)
      cp_async8(reinterpret_cast<uint64_t*>(&s_task[k & 3]) + tid,
                reinterpret_cast<const uint64_t*>(p.tasks + t) + tid);
  };
  // length descriptor of task k (whose record has landed) into s_len[k % 3],
  // unless that slot holds it already
  auto fetch_len = [&](uint32_t k) {
    if (task_of(k) == kNone) return;
    const uint32_t len = s_task[k & 3].len, r = k % 3;
    const uint32_t had = r == 0 ? ring0 : (r == 1 ? ring1 : ring2);
    if (had == len) return;
    if (r == 0) ring0 = len;
    else if (r == 1) ring1 = len;
    else ring2 = len;
    const uint64_t* src = reinterpret_cast<const uint64_t*>(p.lens + len);
    uint64_t* dst = reinterpret_cast<uint64_t*>(&s_len[r]);
    for (uint32_t i = tid; i < sizeof(LongLenDesc) / 8; i += kLongThreads)
      cp_async8(dst + i, src + i);
  };
  fetch_task(0);
  fetch_task(1);
  fetch_task(2);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  fetch_len(0);
  fetch_len(1);
  cp_async_commit();
#pragma unroll 1
  for (uint32_t k = 0; task_of(k) != kNone; ++k) {
    cp_async_wait<0>();
    __syncthreads();  // task k's and k + 1's descriptors and k + 2's record have landed, and
                      // every thread is past task k - 1
    // task k + 3 opens chunk c = (k + 3) / kLongChunk: claim chunk c + 1
    const bool claim = tid == 0 && !DEALT && (k + 3) % kLongChunk == 0;
    const uint32_t claimed = claim ? atomicAdd(p.counter, 1u) * kLongChunk : 0u;
    const LongLenDesc& d = s_len[k % 3];
    const LongTask& ln = s_task[k & 3];
    const bool fresh = ln.len != held;
    if (fresh) {
      held = ln.len;
      long_tables<PH>(p, d, tab);
      cp_async_commit();
    }
    fetch_len(k + 2);
    fetch_task(k + 3);
    cp_async_commit();
    long_task<PH>(p, d, ln, data, tab, fresh);
    // first read at iteration k + 4, after the barriers between
    if (claim) s_chunk[((k + 3) / kLongChunk + 1) & 3] = claimed;
  }
  cp_async_wait<0>();
}

}  // namespace b2f
