// In-place mixed-radix kernels: lines of any 13-smooth length (and the
// Rader, Bluestein and packed real transforms built on them), one pass
// through HBM, one shared-memory buffer.
//
// Every stage reads the R inputs of a butterfly, transforms them in
// registers and writes the R outputs back where the inputs were (decimation
// in frequency, twiddles after the butterfly), so a line needs one buffer,
// a stage one barrier, and the R addresses of a butterfly serve its loads
// and its stores.  The frequencies end up digit-reversed; the last stage
// goes from registers to global memory at the right frequency, so the
// reversal costs a few integer instructions a butterfly.  A convolution
// (Rader, Bluestein) never undoes it: its spectrum table is stored in that
// order, the last forward stage, the product and the first inverse stage
// are one step on R registers, and the inverse runs the mirrored stages
// (decimation in time, twiddles before the butterfly) back to natural order.
//
// Rows (lines contiguous in memory): a lead stage of radix R0 (16 when the
// length allows) reads global memory with adjacent threads on adjacent
// points and splits the line into R0 sub-lines of odd pitch.  From then on
// adjacent threads take adjacent sub-lines at one position: free of bank
// conflicts whatever the radices, twiddles shared by the half-warp, and the
// last stage's stores cover R0 adjacent frequencies.
// Columns (adjacent lines in memory): G columns interleaved, adjacent
// threads on adjacent columns all the way, first stage from and last stage
// to global memory.
//
// What bounds it: instruction issue (50-68 % of the issue slots, 45 % of the
// warps active) and, for lines that leave one CTA an SM, the latency of its
// phases; a point costs one shared load and store a stage, about half a
// 16-byte twiddle load and the butterfly.  Thread instructions per point and
// time against the ping-pong engine (k_lines, k_rader, k_bluestein), f32,
// about 33 M points: 1009 (Rader) 330 -> 236, 589 -> 343 us; 4099 (Bluestein
// over 9216) 695 -> 434, 1368 -> 566 us; 15015 in one pass instead of two
// 393 -> 132, 838 -> 249 us; 8 x 1920 x 1080 real there and back (1920 packed
// rows, 1080 columns) 385 -> 207 us.
#pragma once
#include "ipfft.h"
#include "kernels_impl.cuh"

namespace b2f {

// v[r] *= W_L^{r i}, r = 1..R-1, from the stage's table: two f32 twiddles
// (r, r + 1) of one i share 16 bytes, adjacent i adjacent.
template <class S, int R>
FFT_D void ip_twiddle(C<S>* v, const C<S>* __restrict__ tw, uint32_t i, uint32_t m) {
  if constexpr (sizeof(S) == 4) {
    const float4* __restrict__ t = reinterpret_cast<const float4*>(tw) + i;
#pragma unroll
    for (int r = 1; r < R; r += 2) {
      const float4 w = __ldg(t);
      t += m;
      v[r] = cmul(v[r], C<S>{w.x, w.y});
      if (r + 1 < R) v[r + 1] = cmul(v[r + 1], C<S>{w.z, w.w});
    }
  } else {
    const double2* __restrict__ t = reinterpret_cast<const double2*>(tw) + i;
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const double2 w = __ldg(t);
      t += m;
      v[r] = cmul(v[r], C<S>{w.x, w.y});
    }
  }
}

template <class F>
FFT_D void ip_radix(uint32_t R, F f) {
  switch (R) {
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 9: f(std::integral_constant<int, 9>()); break;
    case 10: f(std::integral_constant<int, 10>()); break;
    case 11: f(std::integral_constant<int, 11>()); break;
    case 12: f(std::integral_constant<int, 12>()); break;
    case 13: f(std::integral_constant<int, 13>()); break;
    case 14: f(std::integral_constant<int, 14>()); break;
    case 15: f(std::integral_constant<int, 15>()); break;
    case 16: f(std::integral_constant<int, 16>()); break;
    default: break;
  }
}

// The lines of one CTA in shared memory; P: IpParams, or the part of it
// that the stages read (sc, G, lam, pitch, LDl, flags, dlam, dG).
template <class S, bool COL, class P = IpParams>
struct Ip {
  const P& p;
  C<S>* sm;
  const C<S>* tw;
  uint32_t tid, T, nvalid;

  FFT_D uint32_t is() const { return COL ? p.G : 1u; }
  // sub-line lam -> line g and sub-line k0 of it; its first value
  FFT_D C<S>* sub(uint32_t lam, uint32_t& g, uint32_t& k0) const {
    if constexpr (COL) {
      g = lam;
      k0 = 0;
      return sm + lam;
    } else {
      g = fdiv(lam, p.sc.dR0);
      k0 = lam - g * p.sc.R0;
      return sm + g * p.LDl + k0 * p.pitch;
    }
  }
  // f(jj, lam) over the nj butterflies of every sub-line
  template <class F>
  FFT_D void each(uint32_t nj, F f) const {
    const uint32_t total = p.lam * nj;
#pragma unroll 1
    for (uint32_t e = tid; e < total; e += T) {
      const uint32_t jj = fdiv(e, p.dlam);
      f(jj, e - jj * p.lam);
    }
  }

  // One stage in place: forward (DIF) or the mirrored one (DIT).
  template <bool DIT>
  FFT_D void stage(const IpStage& s) const {
    ip_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const uint32_t step = s.m * is();
      const C<S>* t = tw + s.tw;
      each(s.nj, [&](uint32_t jj, uint32_t lam) {
        uint32_t g, k0;
        C<S>* a = sub(lam, g, k0);
        if (g >= nvalid) return;
        const uint32_t b = fdiv(jj, s.dm), i = jj - b * s.m;
        a += (b * s.L + i) * is();
        C<S> v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = a[q * step];
        if (DIT) ip_twiddle<S, R>(v, t, i, s.m);
        dft<S, R>(v);
        if (!DIT) ip_twiddle<S, R>(v, t, i, s.m);
#pragma unroll
        for (int q = 0; q < R; ++q) a[q * step] = v[q];
      });
    });
  }

  // The lead stage (rows) or stage 0 (columns) from global memory:
  // ld.load<R>(v, g, i, step) fetches points i, i + step, ... of line g.
  template <class Ld>
  FFT_D void first(const Ld& ld) const {
    if constexpr (COL) {
      const IpStage& s = p.sc.st[0];
      ip_radix(s.R, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const uint32_t step = s.m * is();
        each(s.nj, [&](uint32_t i, uint32_t g) {
          if (g >= nvalid) return;
          C<S> v[R];
          ld.template load<R>(v, g, i, s.m);
          dft<S, R>(v);
          ip_twiddle<S, R>(v, tw + s.tw, i, s.m);
          C<S>* a = sm + i * is() + g;
#pragma unroll
          for (int q = 0; q < R; ++q) a[q * step] = v[q];
        });
      });
    } else {
      const uint32_t NS = p.sc.NS;
      ip_radix(p.sc.R0, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const uint32_t total = nvalid * NS;
#pragma unroll 1
        for (uint32_t e = tid; e < total; e += T) {
          const uint32_t g = fdiv(e, p.sc.dNS), i = e - g * NS;
          C<S> v[R];
          ld.template load<R>(v, g, i, NS);
          dft<S, R>(v);
          ip_twiddle<S, R>(v, tw + p.sc.tw0, i, NS);
          C<S>* a = sm + g * p.LDl + i;
#pragma unroll
          for (int q = 0; q < R; ++q) a[q * p.pitch] = v[q];
        }
      });
    }
    __syncthreads();
  }

  // The mirrored lead stage (rows) or stage 0 (columns) to global memory:
  // st.store<R>(v, g, i, step) takes points i, i + step, ... of line g.
  template <class St>
  FFT_D void final_dit(const St& st) const {
    if constexpr (COL) {
      const IpStage& s = p.sc.st[0];
      ip_radix(s.R, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const uint32_t step = s.m * is();
        each(s.nj, [&](uint32_t i, uint32_t g) {
          if (g >= nvalid) return;
          C<S> v[R];
          const C<S>* a = sm + i * is() + g;
#pragma unroll
          for (int q = 0; q < R; ++q) v[q] = a[q * step];
          ip_twiddle<S, R>(v, tw + s.tw, i, s.m);
          dft<S, R>(v);
          st.template store<R>(v, g, i, s.m);
        });
      });
    } else {
      const uint32_t NS = p.sc.NS;
      ip_radix(p.sc.R0, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const uint32_t total = nvalid * NS;
#pragma unroll 1
        for (uint32_t e = tid; e < total; e += T) {
          const uint32_t g = fdiv(e, p.sc.dNS), i = e - g * NS;
          const C<S>* a = sm + g * p.LDl + i;
          C<S> v[R];
#pragma unroll
          for (int q = 0; q < R; ++q) v[q] = a[q * p.pitch];
          ip_twiddle<S, R>(v, tw + p.sc.tw0, i, NS);
          dft<S, R>(v);
          st.template store<R>(v, g, i, NS);
        }
      });
    }
  }

  // The last forward stage (m = 1), registers to global memory:
  // st.store<R>(v, g, k, step) takes frequencies k, k + step, ... of line
  // g.  Rows walk the sub-lines' frequencies in order (R0 adjacent
  // frequencies of each across the threads) or, with PF_CFIRST_STORE, take
  // adjacent lines first; columns walk the blocks in memory order.
  template <class St>
  FFT_D void last(const St& st) const {
    const uint32_t nst = p.sc.nst;
    const IpStage& s = p.sc.st[nst - 1];
    ip_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      each(s.nj, [&](uint32_t jj, uint32_t lam) {
        uint32_t g, k0;
        const C<S>* a;
        if (!COL && (p.flags & PF_CFIRST_STORE)) {
          k0 = fdiv(lam, p.dG);
          g = lam - k0 * p.G;
          a = sm + g * p.LDl + k0 * p.pitch;
        } else {
          a = sub(lam, g, k0);
        }
        if (g >= nvalid) return;
        uint32_t b, f;
        if constexpr (COL) {
          b = jj;
          f = 0;
          uint32_t x = b;
#pragma unroll 1
          for (int t = (int)nst - 2; t >= 0; --t) {
            const uint32_t q = fdiv(x, p.sc.st[t].dR);
            f = f * p.sc.st[t].R + (x - q * p.sc.st[t].R);
            x = q;
          }
        } else {
          f = jj;
          b = 0;
          uint32_t x = f;
#pragma unroll 1
          for (uint32_t t = 0; t + 1 < nst; ++t) {
            const uint32_t q = fdiv(x, p.sc.st[t].dR);
            b = b * p.sc.st[t].R + (x - q * p.sc.st[t].R);
            x = q;
          }
        }
        a += b * R * is();
        C<S> v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = a[q * is()];
        dft<S, R>(v);
        const uint32_t R0 = COL ? 1u : p.sc.R0;
        st.template store<R>(v, g, k0 + R0 * f, R0 * s.nj);
      });
    });
  }

  // Stages after the first up to the one before the last, forward.
  FFT_D void forward_mids() const {
#pragma unroll 1
    for (uint32_t t = COL ? 1 : 0; t + 1 < p.sc.nst; ++t) {
      stage<false>(p.sc.st[t]);
      __syncthreads();
    }
  }

  // A convolution's centre: last forward stage, product with the spectrum
  // (op.spectrum(g), [pos][k0]; op.dc sees frequency 0 first), conjugate,
  // first inverse stage.
  template <class Op>
  FFT_D void centre(const Op& op) const {
    const IpStage& s = p.sc.st[p.sc.nst - 1];
    const uint32_t R0 = COL ? 1u : p.sc.R0;
    ip_radix(s.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      each(s.nj, [&](uint32_t b, uint32_t lam) {
        uint32_t g, k0;
        C<S>* a = sub(lam, g, k0);
        if (g >= nvalid) return;
        a += b * R * is();
        C<S> v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = a[q * is()];
        dft<S, R>(v);
        const C<S>* __restrict__ w = op.spectrum(g) + (b * R) * R0 + k0;
        const C<S> v0 = v[0];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = conj(cmul(v[q], w[q * R0]));
        if (b == 0 && k0 == 0) op.dc(g, v0, v[0]);
        dft<S, R>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) a[q * is()] = v[q];
      });
    });
    __syncthreads();
  }

  // The mirrored stages back to the one after the final one.
  FFT_D void inverse_mids() const {
#pragma unroll 1
    for (int t = (int)p.sc.nst - 2; t >= (COL ? 1 : 0); --t) {
      stage<true>(p.sc.st[t]);
      __syncthreads();
    }
  }
};

// ------------------------------------------------------- global memory ends
template <class S>
struct IpLoad {  // points of the lines, conjugated for inverse transforms
  const C<S>* in;
  int64_t dl, es;
  uint32_t flags;
  template <int R>
  FFT_D void load(C<S>* v, uint32_t g, uint32_t i, uint32_t step) const {
    const C<S>* a = in + (int64_t)g * dl + (int64_t)i * es;
    const int64_t d = (int64_t)step * es;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = a[q * d];
    if (flags & PF_CONJ_IN) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q].im = -v[q].im;
    }
  }
};

template <class S>
struct IpStore {  // four-step twiddle, scale, conjugation, as asked by the flags
  const IpParams& p;
  C<S>* out;
  int64_t dl, es;
  uint64_t c0;
  S sc;
  template <int R>
  FFT_D void store(C<S>* v, uint32_t g, uint32_t k, uint32_t step) const {
    const uint32_t fl = p.flags;
    if (fl & PF_TW_STORE) {
      const uint32_t row = fdiv((uint32_t)(c0 + g), p.d_tw);
      const C<S>* __restrict__ ta = (const C<S>*)p.tws_a;
      const C<S>* __restrict__ tb = (const C<S>*)p.tws_b;
      if (p.tw_store_M <= 0xFFFFFFFFull) {
        // row k < M: a 32-bit exponent stepped through the split tables
        uint32_t m = row * k;
        const uint32_t dm = row * step, sh = p.d_tws.shift, msk = (1u << sh) - 1;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          v[q] = cmul(v[q], cmul(ta[m >> sh], tb[m & msk]));
          m += dm;
        }
      } else {
#pragma unroll
        for (int q = 0; q < R; ++q)
          v[q] = cmul(v[q], tw_two_level(ta, tb, (uint64_t)row * (k + q * step), p.d_tws));
      }
    }
    if (fl & PF_SCALE) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = cscale(v[q], sc);
    }
    if (fl & PF_CONJ_OUT) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q].im = -v[q].im;
    }
    C<S>* a = out + (int64_t)g * dl + (int64_t)k * es;
    const int64_t d = (int64_t)step * es;
#pragma unroll
    for (int q = 0; q < R; ++q) a[q * d] = v[q];
  }
};

// f32: 64 registers, so that 1024 threads share an SM; f64: 128 and 512.
template <class S>
struct IpBounds {
  static constexpr int threads = sizeof(S) == 4 ? 1024 : 512;
};

template <class S, bool COL>
__global__ void __launch_bounds__(IpBounds<S>::threads)
    k_ip_lines(const __grid_constant__ IpParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Group g = group_of(p.io, p.G, blockIdx.x);
  const Ip<S, COL> ip{p, reinterpret_cast<C<S>*>(smem_raw), (const C<S>*)p.tw, threadIdx.x,
                      blockDim.x, g.nvalid};
  ip.first(IpLoad<S>{(const C<S>*)p.in + g.in0, g.dl_in, p.io.in_es, p.flags});
  ip.forward_mids();
  ip.last(IpStore<S>{p, (C<S>*)p.out + g.out0, g.dl_out, p.io.out_es, g.c0,
                         Scalar<S>::from_double(p.scale)});
}

// ------------------------------------------------------------------ Rader
// X[0] = sum x; X[g^-r] = x[0] + (a (*) b)[r] with a[q] = x[g^q] and b[q] =
// W_p^{g^-q}, a cyclic convolution of N = p - 1 points
// (src/runtime/rader_axis.rs:1228-1336 builds the same pieces).  x[0] goes
// into frequency 0 of the product, which adds it to every output.  Rows
// pass through a staging buffer of natural order on both sides, so that
// global memory is read and written in order and the permutations stay in
// shared memory; columns write the permuted rows directly.
template <class S, bool COL>
struct IpGather {
  const C<S>* stage;
  const uint32_t* perm;
  uint32_t n, G;
  template <int R>
  FFT_D void load(C<S>* v, uint32_t g, uint32_t i, uint32_t step) const {
    uint32_t j[R];
#pragma unroll
    for (int q = 0; q < R; ++q) j[q] = __ldg(perm + i + q * step);
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = COL ? stage[j[q] * G + g] : stage[g * n + j[q]];
  }
};

template <class S, bool COL>
struct IpScatter {  // conv = conj(v) at r -> point g^-r
  const IpParams& p;
  C<S>* stage;
  C<S>* out;  // columns
  int64_t dl, es;
  S sc;
  template <int R>
  FFT_D void store(C<S>* v, uint32_t g, uint32_t r, uint32_t step) const {
    const uint32_t N = p.sc.N;
    uint32_t j[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const uint32_t rr = r + q * step;
      j[q] = __ldg(p.perm + (rr ? N - rr : 0));
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      v[q].im = -v[q].im;
      if constexpr (COL) {
        if (p.flags & PF_SCALE) v[q] = cscale(v[q], sc);
        if (p.flags & PF_CONJ_OUT) v[q].im = -v[q].im;
        out[(int64_t)g * dl + (int64_t)j[q] * es] = v[q];
      } else {
        stage[g * p.n + j[q]] = v[q];
      }
    }
  }
};

template <class S>
struct IpRaderOp {
  const C<S>* bhat;
  const C<S>* x0;
  C<S>* X0;
  FFT_D const C<S>* spectrum(uint32_t) const { return bhat; }
  // X[0] = x[0] + A[0]; the product's conjugate gets conj(x[0])
  FFT_D void dc(uint32_t g, C<S> a0, C<S>& prod) const {
    const C<S> x = x0[g];
    X0[g] = x + a0;
    prod = prod + conj(x);
  }
};

template <class S, bool COL>
__global__ void __launch_bounds__(IpBounds<S>::threads)
    k_ip_rader(const __grid_constant__ IpParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C<S>* sm = reinterpret_cast<C<S>*>(smem_raw);
  C<S>* stage = sm + (COL ? p.G * p.sc.N : p.G * p.LDl);
  C<S>* x0 = stage + p.G * p.n;
  C<S>* X0 = x0 + p.G;
  const uint32_t tid = threadIdx.x, T = blockDim.x, n = p.n, G = p.G;
  const Group g = group_of(p.io, G, blockIdx.x);
  const Ip<S, COL> ip{p, sm, (const C<S>*)p.tw, tid, T, g.nvalid};
  {
    const C<S>* in = (const C<S>*)p.in + g.in0;
    const bool cj = p.flags & PF_CONJ_IN;
    for_each_elem_batched<BatchU<S>::value, C<S>>(
        n, p.dn, COL ? G : g.nvalid, p.dG, COL, tid, T,
        [&](uint32_t c, uint32_t i) {
          return c < g.nvalid ? in[(int64_t)c * g.dl_in + (int64_t)i * p.io.in_es] : czero<S>();
        },
        [&](uint32_t c, uint32_t i, C<S> v) {
          if (c >= g.nvalid) return;
          if (cj) v.im = -v.im;
          stage[COL ? i * G + c : c * n + i] = v;
          if (i == 0) x0[c] = v;
        });
  }
  __syncthreads();
  ip.first(IpGather<S, COL>{stage, p.perm, n, G});
  ip.forward_mids();
  ip.centre(IpRaderOp<S>{(const C<S>*)p.bhat, x0, X0});
  ip.inverse_mids();
  const S sc = Scalar<S>::from_double(p.scale);
  C<S>* out = (C<S>*)p.out + g.out0;
  ip.final_dit(IpScatter<S, COL>{p, stage, out, g.dl_out, p.io.out_es, sc});
  if constexpr (COL) {
    for (uint32_t c = tid; c < g.nvalid; c += T) {
      C<S> v = X0[c];
      if (p.flags & PF_SCALE) v = cscale(v, sc);
      if (p.flags & PF_CONJ_OUT) v.im = -v.im;
      out[(int64_t)c * g.dl_out] = v;
    }
  } else {
    for (uint32_t c = tid; c < g.nvalid; c += T) stage[c * n] = X0[c];
    __syncthreads();
    for_each_elem(n, p.dn, g.nvalid, p.dG, false, tid, T, [&](uint32_t c, uint32_t i) {
      C<S> v = stage[c * n + i];
      if (p.flags & PF_SCALE) v = cscale(v, sc);
      if (p.flags & PF_CONJ_OUT) v.im = -v.im;
      out[(int64_t)c * g.dl_out + (int64_t)i * p.io.out_es] = v;
    });
  }
}

// -------------------------------------------------------------- Bluestein
// X[k] = c_k * sum_j (x_j c_j) conj(c_{k-j}), c_k = exp(-i pi k^2 / n), as a
// cyclic convolution of N >= 2n - 1 points (src/runtime/bluestein_axis.rs:
// 825-867): the chirp on the first stage's loads (points past n are zeros
// that nothing loads) and on the last stage's stores.
template <class S>
struct IpChirpLoad {
  const C<S>* in;
  const C<S>* chirp;
  int64_t dl, es;
  uint32_t n, flags;
  template <int R>
  FFT_D void load(C<S>* v, uint32_t g, uint32_t i, uint32_t step) const {
    const C<S>* a = in + (int64_t)g * dl + (int64_t)i * es;
    const int64_t d = (int64_t)step * es;
    // N >= 2n - 1: at most the first half of a butterfly's points, rounded
    // up, holds data (N even: n <= N / 2; N odd: n <= (N + 1) / 2 and R odd)
    constexpr int H = (R + 1) / 2;
    C<S> w[H];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = czero<S>();
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (i + q * step < n) {
        v[q] = a[q * d];
        w[q] = chirp[i + q * step];
      } else {
        w[q] = czero<S>();
      }
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (i + q * step < n) {
        if (flags & PF_CONJ_IN) v[q].im = -v[q].im;
        v[q] = cmul(v[q], w[q]);
      }
  }
};

template <class S>
struct IpChirpStore {
  C<S>* out;
  const C<S>* chirp;
  int64_t dl, es;
  uint32_t n, flags;
  S sc;
  template <int R>
  FFT_D void store(C<S>* v, uint32_t g, uint32_t i, uint32_t step) const {
    C<S>* a = out + (int64_t)g * dl + (int64_t)i * es;
    const int64_t d = (int64_t)step * es;
    constexpr int H = (R + 1) / 2;
#pragma unroll
    for (int q = 0; q < H; ++q)
      if (i + q * step < n) {
        C<S> x = cmul(conj(v[q]), chirp[i + q * step]);
        if (flags & PF_SCALE) x = cscale(x, sc);
        if (flags & PF_CONJ_OUT) x.im = -x.im;
        a[q * d] = x;
      }
  }
};

template <class S>
struct IpConvOp {
  const C<S>* bhat;
  FFT_D const C<S>* spectrum(uint32_t) const { return bhat; }
  FFT_D void dc(uint32_t, C<S>, C<S>&) const {}
};

template <class S, bool COL>
__global__ void __launch_bounds__(IpBounds<S>::threads)
    k_ip_blue(const __grid_constant__ IpParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Group g = group_of(p.io, p.G, blockIdx.x);
  const Ip<S, COL> ip{p, reinterpret_cast<C<S>*>(smem_raw), (const C<S>*)p.tw, threadIdx.x,
                      blockDim.x, g.nvalid};
  const C<S>* chirp = (const C<S>*)p.chirp;
  ip.first(IpChirpLoad<S>{(const C<S>*)p.in + g.in0, chirp, g.dl_in, p.io.in_es, p.n, p.flags});
  ip.forward_mids();
  ip.centre(IpConvOp<S>{(const C<S>*)p.bhat});
  ip.inverse_mids();
  ip.final_dit(IpChirpStore<S>{(C<S>*)p.out + g.out0, chirp, g.dl_out, p.io.out_es, p.n,
                                   p.flags, Scalar<S>::from_double(p.scale)});
}

// ------------------------------------------------------------------- real
// Even lengths 2N: R2C takes the line as N packed pairs, and X[k], X[N-k]
// come from Z[k], Z[N-k] (k_r2c_fx states the formulas); the last stage
// leaves Z in natural order in a second buffer.  C2R builds Z from the
// packed spectrum on the first stage's loads.
template <class S>
struct IpNatStore {
  C<S>* nat;
  uint32_t ld;
  template <int R>
  FFT_D void store(C<S>* v, uint32_t g, uint32_t k, uint32_t step) const {
#pragma unroll
    for (int q = 0; q < R; ++q) nat[g * ld + k + q * step] = v[q];
  }
};

template <class S>
__global__ void __launch_bounds__(IpBounds<S>::threads)
    k_ip_r2c(const __grid_constant__ IpParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C<S>* sm = reinterpret_cast<C<S>*>(smem_raw);
  C<S>* nat = sm + p.G * p.LDl;
  const uint32_t tid = threadIdx.x, T = blockDim.x, h = p.sc.N;
  const uint64_t l0 = (uint64_t)blockIdx.x * p.G;
  const uint32_t nvalid = p.nlines - l0 < p.G ? (uint32_t)(p.nlines - l0) : p.G;
  const Ip<S, false> ip{p, sm, (const C<S>*)p.tw, tid, T, nvalid};
  ip.first(IpLoad<S>{(const C<S>*)p.in + l0 * h, (int64_t)h, 1, 0});
  ip.forward_mids();
  ip.last(IpNatStore<S>{nat, h});
  __syncthreads();
  const C<S>* __restrict__ rtw = (const C<S>*)p.rtw;
  const S half = Scalar<S>::from_double(0.5), sc = Scalar<S>::from_double(p.scale);
  C<S>* out = (C<S>*)p.out + l0 * (h + 1);
  // pairs k <= h / 2 (p.dn divides by h / 2 + 1)
  const uint32_t K = h / 2 + 1;
  for_each_elem(K, p.dn, nvalid, p.dG, false, tid, T, [&](uint32_t c, uint32_t k) {
    const C<S>* z = nat + c * h;
    const C<S> a = z[k], b = conj(z[k == 0 ? 0 : h - k]);
    const C<S> E = cscale(a + b, half);
    const C<S> WO = cmul(cscale(mul_neg_i(a - b), half), rtw[k]);
    C<S> xk = E + WO, xh = conj(E - WO);
    if (p.flags & PF_SCALE) {
      xk = cscale(xk, sc);
      xh = cscale(xh, sc);
    }
    C<S>* o = out + (uint64_t)c * (h + 1);
    o[k] = xk;
    if (h - k != k) o[h - k] = xh;
  });
}

template <class S>
struct IpC2rLoad {
  const C<S>* in;
  const C<S>* rtw;
  uint32_t h;
  template <int R>
  FFT_D void load(C<S>* v, uint32_t g, uint32_t i, uint32_t step) const {
    const C<S>* x = in + (uint64_t)g * (h + 1);
    C<S> y[R], w[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const uint32_t n = i + q * step;
      v[q] = x[n];
      y[q] = x[h - n];
      w[q] = rtw[n];
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      C<S> xk = v[q], xh = y[q];
      if (i + q * step == 0) {
        xk.im = Scalar<S>::zero();
        xh.im = Scalar<S>::zero();
      }
      const C<S> P = xk + conj(xh), Q = xk - conj(xh);
      v[q] = conj(P + mul_i(cmulc(Q, w[q])));
    }
  }
};

template <class S>
__global__ void __launch_bounds__(IpBounds<S>::threads)
    k_ip_c2r(const __grid_constant__ IpParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t h = p.sc.N;
  const uint64_t l0 = (uint64_t)blockIdx.x * p.G;
  const uint32_t nvalid = p.nlines - l0 < p.G ? (uint32_t)(p.nlines - l0) : p.G;
  const Ip<S, false> ip{p, reinterpret_cast<C<S>*>(smem_raw), (const C<S>*)p.tw, threadIdx.x,
                        blockDim.x, nvalid};
  ip.first(IpC2rLoad<S>{(const C<S>*)p.in + l0 * (h + 1), (const C<S>*)p.rtw, h});
  ip.forward_mids();
  ip.last(IpStore<S>{p, (C<S>*)p.out + l0 * h, (int64_t)h, 1, 0, Scalar<S>::from_double(p.scale)});
}

}  // namespace b2f
