// Batched launch of many 1D f32 lines of mixed lengths: the device side.
//
// Persistent kernels share one execute call:
//  - k_batch_cta: each CTA repeatedly takes the next task from an atomic
//    counter; a task is up to G lines of one length whose FFT (mixed radix,
//    Rader or Bluestein, on the in-place stages of ipfft.cuh) fits one CTA's
//    share of the shared memory;
//  - k_long_pass (longpass.cuh): the longer lines, as column and row passes
//    through a scratch region;
//  - k_batch_cluster<P> (optional route for the longer lines): a thread-block cluster of P CTAs takes one long line
//    at a time and transforms it in a single HBM pass, the CTAs exchanging
//    data through distributed shared memory:
//      n = m + L*r (r = CTA rank, m < L = T/P),   k = P*k1 + k2,
//      X[P k1 + k2] = sum_m W_L^{m k1} [ W_T^{m k2} sum_r W_P^{r k2} x[m + L r] ],
//    i.e. a cross-CTA radix-P step with the W_T^{m k2} twiddle, a local
//    length-L FFT in each CTA, and a transposed read-out.  Bluestein lines
//    run their forward FFT this way, multiply by the chirp spectrum in the
//    transposed order, and run the inverse FFT in the mirrored order (local
//    FFT first, then the cross-CTA step), so the convolution never leaves
//    the chip.
// Work queue polls are bounded: a task index is taken with one atomicAdd and
// nothing ever waits on another CTA except the cluster barriers, which every
// CTA of a cluster reaches the same number of times.
#pragma once
#include <cooperative_groups.h>

#include "ipfft.cuh"

namespace b2f {

enum BatchKind : uint32_t {
  BK_MIXED = 0,     // one CTA, mixed radix
  BK_RADER = 1,     // one CTA, Rader
  BK_BLUE = 2,      // one CTA, Bluestein
  BK_CL_MIXED = 3,  // cluster, mixed radix (T = N)
  BK_CL_BLUE = 4,   // cluster, Bluestein (T = convolution length)
  BK_LONG = 5,      // long line: two passes N = N1*N2 through scratch (k_long_pass)
  BK_LONG_BLUE = 6, // long Bluestein line: three passes over M = N1*N2 (k_long_pass)
};

// What the in-place stages (Ip) read of a schedule: rows of one line or of
// several, or adjacent columns.
struct IpRows {
  IpSched sc;
  uint32_t G, lam, pitch, LDl, flags;
  FastDiv dlam, dG;
};

struct BatchLen {
  uint32_t kind;
  uint32_t N;     // line length
  uint32_t M;     // transform length: N, p-1, or the convolution length
  uint32_t G;     // lines per task (CTA kinds)
  uint32_t LD;    // shared-memory line pitch (cluster kinds, lines of up to 16 points)
  uint32_t P;     // cluster ranks in use (cluster kinds)
  uint32_t L;     // M / P (cluster kinds)
  float scale;    // normalisation of this length (f32, as the reference)
  const c32* bhat;        // [pos][k0] (CTA kinds), natural (cluster kinds)
  const uint32_t* perm;   // Rader: g^q mod p
  const c32* chirp;       // CTA Bluestein: exp(-i pi n^2 / N)
  FastDiv dN;
  // two-level table of the cross-CTA twiddle W_M^j of the cluster kinds,
  // j = a*L + b (offsets into BatchParams::tw): ta[a] = W_M^{a L}, tb[b] = W_M^b.
  uint32_t ta, tb;
  FastDiv dB;
  IpRows ip;      // CTA kinds above 16 points: the transform of length M on G lines
  Schedule sch;   // ping-pong schedule (cluster kinds: length L; lines of up to 16 points: N)
};

struct BatchTask {
  uint32_t len;    // index into the length table
  uint32_t first;  // first line (sorted order)
  uint32_t count;  // lines in the task
  uint32_t pad;
};

struct BatchParams {
  const c32* in;
  c32* out;
  const c32* tw;         // stage and inter-pass twiddle tables (FP64-built, rounded once)
  const BatchLen* lens;
  const BatchTask* tasks;
  const uint64_t* line_off;  // complex offset of each line in `in` (sorted order)
  const uint64_t* line_off_out;  // its offset in `out`, or null: the same as in `in`
  uint32_t ntasks;
  uint32_t inverse;
  unsigned int* counter;
};

constexpr int kBatchMaxG = 256;

// Asynchronous 8-byte global -> shared copy (sm_80+ LDGSTS): every thread
// keeps all of its loads in flight instead of waiting on each one.
FFT_D void cp_async8(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

template <class T>
FFT_D void copy_words(T* dst, const T* src, uint32_t tid, uint32_t nthreads) {
  static_assert(sizeof(T) % 4 == 0, "word copy");
  const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
  uint32_t* d = reinterpret_cast<uint32_t*>(dst);
  for (uint32_t i = tid; i < sizeof(T) / 4; i += nthreads) d[i] = s[i];
}

// W_T^j from the two-level table: j = a*B + b.
FFT_D c32 tw2(const BatchParams& bp, const BatchLen& L, uint32_t j, uint32_t B) {
  const uint32_t a = fdiv(j, L.dB), b = j - a * B;
  return cmul(bp.tw[L.ta + a], bp.tw[L.tb + b]);
}

// --------------------------------------------------------------- CTA tasks
// Global memory ends of the in-place stages: line g at base[g].
struct BatchLoad {
  const c32* in;
  const int64_t* base;
  bool cj;
  template <int R>
  FFT_D void load(c32* v, uint32_t g, uint32_t i, uint32_t step) const {
    const c32* a = in + base[g] + i;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = a[q * step];
    if (cj) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q].im = -v[q].im;
    }
  }
};

struct BatchStore {
  c32* out;
  const int64_t* base;
  float sc, sci;  // sci: scale of the imaginary part, negated for inverse transforms
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t k, uint32_t step) const {
    c32* a = out + base[g] + k;
#pragma unroll
    for (int q = 0; q < R; ++q) a[q * step] = c32{v[q].re * sc, v[q].im * sci};
  }
};

struct BatchScatter {  // Rader: conv = conj(v) at r -> point g^-r of the staged line
  c32* stage;
  const uint32_t* perm;
  uint32_t n;
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t r, uint32_t step) const {
    uint32_t j[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const uint32_t rr = r + q * step;
      j[q] = __ldg(perm + (rr ? n - 1 - rr : 0));
    }
#pragma unroll
    for (int q = 0; q < R; ++q) stage[g * n + j[q]] = conj(v[q]);
  }
};

struct BatchChirpLoad {
  const c32* in;
  const int64_t* base;
  const c32* chirp;
  uint32_t n;
  bool cj;
  template <int R>
  FFT_D void load(c32* v, uint32_t g, uint32_t i, uint32_t step) const {
    const c32* a = in + base[g];
    constexpr int H = (R + 1) / 2;  // as IpChirpLoad
    c32 w[H];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = czero<float>();
#pragma unroll
    for (int q = 0; q < H; ++q) {
      w[q] = czero<float>();
      if (i + q * step < n) {
        v[q] = a[i + q * step];
        w[q] = chirp[i + q * step];
      }
    }
#pragma unroll
    for (int q = 0; q < H; ++q) {
      if (cj) v[q].im = -v[q].im;
      if (i + q * step < n) v[q] = cmul(v[q], w[q]);
    }
  }
};

struct BatchChirpStore {
  c32* out;
  const int64_t* base;
  const c32* chirp;
  uint32_t n;
  float sc, sci;
  template <int R>
  FFT_D void store(c32* v, uint32_t g, uint32_t k, uint32_t step) const {
    c32* a = out + base[g];
    constexpr int H = (R + 1) / 2;
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (k + q * step < n) {
        const c32 x = cmul(conj(v[q]), chirp[k + q * step]);
        a[k + q * step] = c32{x.re * sc, x.im * sci};
      }
  }
};

// Lines of up to 16 points: one or two ping-pong stages.
FFT_D void batch_tiny(const BatchParams& bp, const BatchLen& L, const int64_t* base,
                      const int64_t* obase, uint32_t cnt, c32* A, c32* B, uint32_t tid, uint32_t T) {
  constexpr int PAD = PadOf<float>::value;
  const uint32_t N = L.N, LD = L.LD;
  const bool inv = bp.inverse;
  for (uint32_t e = tid; e < cnt * N; e += T) {
    const uint32_t c = fdiv(e, L.dN), n = e - c * N;
    c32 v = bp.in[base[c] + n];
    if (inv) v.im = -v.im;
    A[c * LD + pidx<PAD>(n)] = v;
  }
  __syncthreads();
  const c32* r = fft_lines_smem<float>(A, B, L.sch, cnt, LD, tid, T, bp.tw);
  const float sc = L.scale;
  for (uint32_t e = tid; e < cnt * N; e += T) {
    const uint32_t c = fdiv(e, L.dN), n = e - c * N;
    c32 v = r[c * LD + pidx<PAD>(n)];
    v.re *= sc;
    v.im = inv ? -v.im * sc : v.im * sc;
    bp.out[obase[c] + n] = v;
  }
}

// The task's lines on the in-place stages; `buf`: cnt * LDl values of data,
// then for Rader the staged lines and x[0], X[0] of each.
FFT_D void batch_lines(const BatchParams& bp, const BatchLen& L, const int64_t* base,
                       const int64_t* obase, uint32_t cnt, c32* buf, uint32_t tid, uint32_t T) {
  const bool inv = bp.inverse;
  const float sc = L.scale, sci = inv ? -L.scale : L.scale;
  const Ip<float, false, IpRows> ip{L.ip, buf, bp.tw, tid, T, cnt};
  if (L.kind == BK_MIXED) {
    ip.first(BatchLoad{bp.in, base, inv});
    ip.forward_mids();
    ip.last(BatchStore{bp.out, obase, sc, sci});
  } else if (L.kind == BK_BLUE) {
    ip.first(BatchChirpLoad{bp.in, base, L.chirp, L.N, inv});
    ip.forward_mids();
    ip.centre(IpConvOp<float>{L.bhat});
    ip.inverse_mids();
    ip.final_dit(BatchChirpStore{bp.out, obase, L.chirp, L.N, sc, sci});
  } else {  // Rader
    const uint32_t n = L.N;
    c32* stage = buf + cnt * L.ip.LDl;
    c32* x0 = stage + cnt * n;
    c32* X0 = x0 + cnt;
    for (uint32_t e = tid; e < cnt * n; e += T) {
      const uint32_t c = fdiv(e, L.dN), i = e - c * n;
      c32 v = bp.in[base[c] + i];
      if (inv) v.im = -v.im;
      stage[e] = v;
      if (i == 0) x0[c] = v;
    }
    __syncthreads();
    ip.first(IpGather<float, false>{stage, L.perm, n, 0});
    ip.forward_mids();
    ip.centre(IpRaderOp<float>{L.bhat, x0, X0});
    ip.inverse_mids();
    ip.final_dit(BatchScatter{stage, L.perm, n});
    for (uint32_t c = tid; c < cnt; c += T) stage[c * n] = X0[c];
    __syncthreads();
    for (uint32_t e = tid; e < cnt * n; e += T) {
      const uint32_t c = fdiv(e, L.dN);
      const c32 v = stage[e];
      bp.out[obase[c] + (e - c * n)] = c32{v.re * sc, v.im * sci};
    }
  }
}

// make_fastdiv for d < 2^16 on the device (the sub-lines of a task vary with
// its line count).
FFT_D FastDiv fastdiv_small(uint32_t d) {
  FastDiv f;
  f.d = d;
  const uint32_t l = d > 1 ? 32 - __clz(d - 1) : 0;
  if ((d & (d - 1)) == 0) {
    f.mul = 0;
    f.shift = l;
  } else {
    f.mul = (uint32_t)(((1ull << (31 + l)) + d - 1) / d);
    f.shift = l - 1;
  }
  return f;
}

// Persistent CTA kernel: 256 threads, four CTAs an SM; dynamic shared memory
// holds the largest task.  Issue-bound; with padded addresses, chirps and
// their 64-bit modulos recomputed per point the short lines took 317 thread
// instructions a point and Bluestein lines above 1,400 points the three-pass
// route: 964 lines of up to 2,293 points 95 -> 31 us, 1,300 of up to 1,849
// 91 -> 26 us.
__global__ void __launch_bounds__(256, 4) k_batch_cta(const __grid_constant__ BatchParams bp,
                                                   uint32_t buf_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BatchLen s_len;
  __shared__ int64_t s_base[kBatchMaxG];
  __shared__ int64_t s_obase[kBatchMaxG];
  __shared__ uint32_t s_task;
  uint32_t s_len_idx = 0xFFFFFFFFu;  // length descriptor currently in s_len (same in every thread)
  c32* A = reinterpret_cast<c32*>(smem_raw);
  const uint32_t tid = threadIdx.x, T = blockDim.x;
  // a task for every CTA: no atomic to wait for, no counter to zero
  const bool queue = gridDim.x < bp.ntasks;
  uint32_t t = blockIdx.x;
  if (queue) {
    if (tid == 0) s_task = atomicAdd(bp.counter, 1u);
    __syncthreads();
    t = s_task;
  }
  while (t < bp.ntasks) {
    const BatchTask task = bp.tasks[t];
    if (task.len != s_len_idx) copy_words(&s_len, bp.lens + task.len, tid, T);
    s_len_idx = task.len;
    for (uint32_t c = tid; c < task.count; c += T) {
      s_base[c] = (int64_t)bp.line_off[task.first + c];
      s_obase[c] = (int64_t)(bp.line_off_out ? bp.line_off_out : bp.line_off)[task.first + c];
    }
    __syncthreads();  // s_task read, s_len and the line offsets written
    uint32_t next = 0;
    if (tid == 0) {
      if (queue) next = atomicAdd(bp.counter, 1u);
      const uint32_t lam = task.count * s_len.ip.sc.R0;  // the sub-lines of this task's lines
      if (lam != s_len.ip.lam) {
        s_len.ip.lam = lam;
        s_len.ip.dlam = fastdiv_small(lam);
      }
    }
    __syncthreads();
    if (s_len.ip.sc.N)
      batch_lines(bp, s_len, s_base, s_obase, task.count, A, tid, T);
    else
      batch_tiny(bp, s_len, s_base, s_obase, task.count, A, A + buf_elems / 2, tid, T);
    if (!queue) break;
    if (tid == 0) s_task = next;
    __syncthreads();
    t = s_task;
  }
}

// ---------------------------------------------------------- cluster tasks
template <int P>
FFT_D void cluster_radix_p(cooperative_groups::cluster_group& cl, c32* src_local, c32* dst_local,
                           uint32_t Lr, uint32_t Mt, uint32_t rank, uint32_t tid, uint32_t T,
                           bool twiddle_first, const BatchParams& bp, const BatchLen& L) {
  // For m in this CTA's share: v[r] = src[r][m]; (twiddle_first: v[r] *= W_Mt^{m r});
  // DFT_P; (else: v[k2] *= W_Mt^{m k2}); dst[k2][m] = v[k2].
  constexpr int PAD = PadOf<float>::value;
  const uint32_t m0 = (uint32_t)(((uint64_t)rank * Lr) / P);
  const uint32_t m1 = (uint32_t)(((uint64_t)(rank + 1) * Lr) / P);
  for (uint32_t m = m0 + tid; m < m1; m += T) {
    c32 v[P];
    const uint32_t pm = pidx<PAD>(m);
#pragma unroll
    for (int r = 0; r < P; ++r) v[r] = cl.map_shared_rank(src_local, r)[pm];
    if (twiddle_first) {
#pragma unroll
      for (int r = 1; r < P; ++r) v[r] = cmul(v[r], tw2(bp, L, m * r, Lr));
    }
    dft<float, P>(v);
    if (!twiddle_first) {
#pragma unroll
      for (int r = 1; r < P; ++r) v[r] = cmul(v[r], tw2(bp, L, m * r, Lr));
    }
#pragma unroll
    for (int r = 0; r < P; ++r) cl.map_shared_rank(dst_local, r)[pm] = v[r];
  }
}

template <int P>
__global__ void __launch_bounds__(512, 1) k_batch_cluster(const __grid_constant__ BatchParams bp,
                                                          uint32_t buf_elems) {
  namespace cg = cooperative_groups;
  constexpr int PAD = PadOf<float>::value;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ BatchLen s_len;
  __shared__ uint32_t s_task;
  c32* A = reinterpret_cast<c32*>(smem_raw);
  c32* B = A + buf_elems;
  const uint32_t tid = threadIdx.x, T = blockDim.x;
  const uint32_t rank = cl.block_rank();
  for (;;) {
    if (rank == 0 && tid == 0) s_task = atomicAdd(bp.counter, 1u);
    cl.sync();
    const uint32_t t = *cl.map_shared_rank(&s_task, 0);
    cl.sync();  // rank 0 may not leave or move on while others read its slot
    if (t >= bp.ntasks) break;
    const BatchTask task = bp.tasks[t];
    copy_words(&s_len, bp.lens + task.len, tid, T);
    __syncthreads();
    const BatchLen& L = s_len;
    const uint32_t N = L.N, Mt = L.M, Lr = L.L;
    const bool inv = bp.inverse;
    const bool blue = L.kind == BK_CL_BLUE;
    const int64_t base = (int64_t)bp.line_off[task.first];
    const bool active = rank < L.P;  // ranks beyond P idle through the task
    // 1. this CTA's contiguous chunk n = rank*L + m
    if (active) {
      for (uint32_t m = tid; m < Lr; m += T) {
        const uint32_t n = rank * Lr + m;
        c32 v = czero<float>();
        if (n < N) {
          v = bp.in[base + n];
          if (inv) v.im = -v.im;
          if (blue) v = cmul(v, chirp<float>(n, N));
        }
        A[pidx<PAD>(m)] = v;
      }
    }
    cl.sync();
    // 2. cross-CTA radix-P step, twiddle after: A (all ranks) -> B (all ranks)
    if (L.P == P) {
      cluster_radix_p<P>(cl, A, B, Lr, Mt, rank, tid, T, false, bp, L);
    } else if (active) {
      switch (L.P) {
        case 2: cluster_radix_p<2>(cl, A, B, Lr, Mt, rank, tid, T, false, bp, L); break;
        case 3: cluster_radix_p<3>(cl, A, B, Lr, Mt, rank, tid, T, false, bp, L); break;
        case 4: cluster_radix_p<4>(cl, A, B, Lr, Mt, rank, tid, T, false, bp, L); break;
        case 5: cluster_radix_p<5>(cl, A, B, Lr, Mt, rank, tid, T, false, bp, L); break;
        case 7: cluster_radix_p<7>(cl, A, B, Lr, Mt, rank, tid, T, false, bp, L); break;
        default: break;
      }
    }
    cl.sync();
    // 3. local FFT_L of B (every rank runs it so barriers match; idle ranks on garbage)
    c32* r = fft_lines_smem<float>(B, A, L.sch, 1, L.LD, tid, T, bp.tw);
    c32* o = (r == A) ? B : A;
    if (!blue) {
      cl.sync();
      // 4. output n = P*k1 + k2 of this rank's chunk from rank k2, slot k1
      if (active) {
        const float sc = L.scale;
        for (uint32_t m = tid; m < Lr; m += T) {
          const uint32_t n = rank * Lr + m;
          const uint32_t k1 = n / L.P, k2 = n - k1 * L.P;
          c32 v = cl.map_shared_rank(r, k2)[pidx<PAD>(k1)];
          v.re *= sc;
          v.im = inv ? -v.im * sc : v.im * sc;
          bp.out[base + n] = v;
        }
      }
      cl.sync();
      continue;
    }
    // Bluestein: r holds F[P*k1 + rank] at slot k1; product with the chirp
    // spectrum, conjugated for the inverse through the forward kernels
    if (active) {
      for (uint32_t k1 = tid; k1 < Lr; k1 += T) {
        c32 v = cmul(r[pidx<PAD>(k1)], L.bhat[(uint64_t)k1 * L.P + rank]);
        v.im = -v.im;
        r[pidx<PAD>(k1)] = v;
      }
    }
    __syncthreads();
    // inverse in the mirrored order: local FFT_L first ...
    c32* r2 = fft_lines_smem<float>(r, o, L.sch, 1, L.LD, tid, T, bp.tw);
    c32* o2 = (r2 == r) ? o : r;
    cl.sync();
    // ... then the twiddle and the cross-CTA radix-P step: r2 -> o2
    if (L.P == P) {
      cluster_radix_p<P>(cl, r2, o2, Lr, Mt, rank, tid, T, true, bp, L);
    } else if (active) {
      switch (L.P) {
        case 2: cluster_radix_p<2>(cl, r2, o2, Lr, Mt, rank, tid, T, true, bp, L); break;
        case 3: cluster_radix_p<3>(cl, r2, o2, Lr, Mt, rank, tid, T, true, bp, L); break;
        case 4: cluster_radix_p<4>(cl, r2, o2, Lr, Mt, rank, tid, T, true, bp, L); break;
        case 5: cluster_radix_p<5>(cl, r2, o2, Lr, Mt, rank, tid, T, true, bp, L); break;
        case 7: cluster_radix_p<7>(cl, r2, o2, Lr, Mt, rank, tid, T, true, bp, L); break;
        default: break;
      }
    }
    cl.sync();
    // rank r holds y[r*L + m]; the convolution is conj(y)
    if (active) {
      const float sc = L.scale;
      for (uint32_t m = tid; m < Lr; m += T) {
        const uint32_t n = rank * Lr + m;
        if (n < N) {
          c32 w = o2[pidx<PAD>(m)];
          w.im = -w.im;
          c32 v = cmul(w, chirp<float>(n, N));
          v.re *= sc;
          v.im = inv ? -v.im * sc : v.im * sc;
          bp.out[base + n] = v;
        }
      }
    }
    cl.sync();
  }
}

}  // namespace b2f
