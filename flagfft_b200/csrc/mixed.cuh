// Mixed-radix tile passes of any radix sequence with direct global access.
//
// The passes whose length has no compile-time sequence (rows.cuh) and the
// on-chip real transforms run here.  Against the general ping-pong tile body
// (tile_impl.cuh) a pass
//   * reads the first Stockham stage's butterfly inputs straight from global
//     memory and writes the last stage's outputs straight to it, so a
//     transform of S stages crosses shared memory S - 1 times, not S + 1;
//   * runs the butterflies of the tile's W transforms as one flat index space
//     over the CTA's threads (butterfly e is j = e mod L/R of transform
//     e / (L/R)), so no stage leaves a fixed share of the threads idle when
//     its radix differs from the largest one;
//   * keeps the first stage's outputs transposed, output q of butterfly j at
//     q * P0 + j with P0 = L/R0 rounded up to odd: the stride-R0 writes that
//     a natural order would make collide on the banks for every even R0, and
//     the second stage's reads step the same layout without a division per
//     element (its index j + r L/R1 has the same residue mod R0 for every r);
//   * packs a real transform's pairs on its load or store and does the
//     Hermitian post / pre step from shared memory, both bins of a pair (k,
//     n/2 - k) from one twiddle.
// A convolution's inverse chain runs the radices reversed, so that its first
// stage happens in the registers of the forward chain's last: one of its
// round trips less.
// Measured on one B200 against the ping-pong and in-place bodies these passes
// ran on before: C2C 1200 x 4096 inverse 70.7 -> 25.7 us (3.1 TB/s of input
// and output), D2Z + Z2D 1500 x 1024 42.9 -> 24.9 us; the joined stages took
// 600 uneven transforms in one batch plan from 113.2 to 109.3 us.  What bounds
// it now is the shared-memory and codelet instruction stream of 16 to 24 warps
// per SM, not HBM: over ten tile shapes and four radix chains the two calls
// above moved by 2% from the shape choose_mixed takes (exec.cpp).
#pragma once

#include "tile_impl.cuh"

namespace ffb {
namespace mixed {

// Elements of one buffer (the transposed layout needs L + R0, a Rader core's
// real forms L + 1), and of one transform's slot (odd, so consecutive slots
// start on different banks).
FFB_HD int buf_len(const Core &c) { return c.L + c.radix[0] + 1; }
FFB_HD int slot_len(const Core &c, int nbuf) { return (nbuf * buf_len(c)) | 1; }

// Buffers a pass needs: a complex transform of at most two stages writes
// shared memory once; everything else alternates between two.
FFB_HD int buffers(const Core &c, CoreKind kind, IoKind io) {
  return kind == CoreKind::Dit && io == IoKind::C2C && c.nst <= 2 ? 1 : 2;
}

template <typename T>
inline size_t smem_bytes(const TileArgs<T> &a, CoreKind kind, IoKind io, int W) {
  // (two more elements per transform hold a Rader core's x0 and X0)
  return ((size_t)W * slot_len(a.core, buffers(a.core, kind, io)) + (kind == CoreKind::Rader ? 2 * (size_t)W : 0)) *
         sizeof(cpx<T>);
}

// One CTA tile: the pass, its bases and what of it is live.
template <typename T>
struct Tile {
  const TileArgs<T> *a;
  const void *in;  // transform 0 of the tile
  void *out;
  long long g0;
  int wlive, slot, blen, io, nl;  // nl: logical length of the core's transform (Bluestein n, Rader p)
  cpx<T> *sm;
  cpx<T> *extra;  // Rader: x0 of transform w at w, X0 at W + w
  FFB_HD int wc(int w) const { return w < wlive ? w : wlive - 1; }
  FFB_HD cpx<T> *buf(int w, int b) const { return sm + w * slot + b * blen; }
};

template <typename T>
FFB_HD cpx<T> ld_pair(const T *p, bool aligned) {
  if (aligned) return ldg_c(reinterpret_cast<const cpx<T> *>(p));
  return mk(ldg_v(p), ldg_v(p + 1));
}
template <typename T>
FFB_HD void st_pair(T *p, cpx<T> v, bool aligned) {
  if (aligned) {
    *reinterpret_cast<cpx<T> *>(p) = v;
  } else {
    p[0] = v.x;
    p[1] = v.y;
  }
}

// Core input i of transform w (already clamped to a live one) as the pass's
// IoKind presents it; zb: the buffer with the Hermitian pre step's result.
template <typename T, bool REAL>
FFB_HD cpx<T> core_input(const Tile<T> &t, int w, int i, const cpx<T> *zb) {
  const TileArgs<T> &a = *t.a;
  if constexpr (!REAL) {
    return ldg_c(reinterpret_cast<const cpx<T> *>(t.in) + w * a.ig + (long long)i * a.ii);
  } else {
    if (t.io == (int)IoKind::R2C)
      return ld_pair<T>(reinterpret_cast<const T *>(t.in) + w * a.ig + 2 * (long long)i, a.pair_aligned != 0);
    if (t.io == (int)IoKind::C2R) return zb[i];
    if (t.io == (int)IoKind::R2CFull) return mk(ldg_v(reinterpret_cast<const T *>(t.in) + w * a.ig + i), (T)0);
    // C2RFull: Hermitian expansion of the half spectrum
    const int n = a.n, half = n / 2;
    const bool mirror = i > half;
    cpx<T> v = ldg_c(reinterpret_cast<const cpx<T> *>(t.in) + w * a.ig + (mirror ? n - i : i));
    if (mirror) v.y = -v.y;
    if (i == 0 || ((n & 1) == 0 && i == half)) v.y = (T)0;
    return v;
  }
}

// First-stage reader of the forward chain: elements j + r * nb of transform w.
template <typename T, int KIND, bool REAL>
struct Source {
  const Tile<T> *t;
  int zbuf;
  template <int R>
  FFB_HD void get(int w, int j, int nb, cpx<T> (&v)[R]) const {
    const TileArgs<T> &a = *t->a;
    const int wc = t->wc(w);
    const cpx<T> *zb = t->buf(w, zbuf);
    if constexpr (KIND == 1) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = j + r * nb;
        v[r] = i < t->nl ? cmul(core_input<T, REAL>(*t, wc, i, zb), ldg_c(a.chirp + i)) : mk((T)0, (T)0);
      }
    } else if constexpr (KIND == 2) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = core_input<T, REAL>(*t, wc, ldg_v(a.perm_in + j + r * nb), zb);
    } else if constexpr (!REAL) {
      const cpx<T> *p = reinterpret_cast<const cpx<T> *>(t->in) + wc * a.ig + (long long)j * a.ii;
      const long long step = (long long)nb * a.ii;
      if (KIND == 0 && a.chirp_mode == 1) {
        const long long n = a.n, c0 = (long long)j * a.cj_e + (t->g0 + wc) * a.cj_g, cs = (long long)nb * a.cj_e;
#pragma unroll
        for (int r = 0; r < R; ++r)
          v[r] = c0 + r * cs < n ? cmul(ldg_c(p + r * step), ldg_c(a.chirp + c0 + r * cs)) : mk((T)0, (T)0);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ldg_c(p + r * step);
      }
    } else if (t->io == (int)IoKind::R2C) {
      const T *p = reinterpret_cast<const T *>(t->in) + wc * a.ig + 2 * j;
      if (a.pair_aligned) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ldg_c(reinterpret_cast<const cpx<T> *>(p + 2 * r * nb));
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = mk(ldg_v(p + 2 * r * nb), ldg_v(p + 2 * r * nb + 1));
      }
    } else if (t->io == (int)IoKind::C2R) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = zb[j + r * nb];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = core_input<T, true>(*t, wc, j + r * nb, zb);
    }
  }
};

// Four-step post-twiddle W_N^{g k} from the two split tables, m = g * k < N.
template <typename T>
FFB_HD cpx<T> post_twiddle(const TileArgs<T> &a, cpx<T> v, long long g, int k) {
  const uint32_t m = (uint32_t)(g * (long long)k);
  const uint32_t hi = fdiv(m, a.ptw_div);
  cpx<T> t = cmul(ldg_c(a.ptw_hi + hi), ldg_c(a.ptw_lo + (m - hi * a.ptw_div.d)));
  if (a.inv) t.y = -t.y;
  return cmul(v, t);
}

// Result k of transform w (natural order): global memory, or for the real
// forward pass shared memory, where the Hermitian post step takes it.
template <typename T, bool REAL>
FFB_HD void put_result(const Tile<T> &t, int w, int k, cpx<T> v, cpx<T> *zb) {
  const TileArgs<T> &a = *t.a;
  if constexpr (!REAL) {
    reinterpret_cast<cpx<T> *>(t.out)[w * a.og + (long long)k * a.ok] =
        a.post_twiddle ? post_twiddle(a, v, t.g0 + w, k) : v;
  } else {
    if (t.io == (int)IoKind::R2C) {
      zb[k] = v;
    } else if (t.io == (int)IoKind::C2R) {
      st_pair<T>(reinterpret_cast<T *>(t.out) + w * a.og + 2 * (long long)k, v, a.pair_aligned != 0);
    } else if (t.io == (int)IoKind::R2CFull) {
      if (k <= a.n / 2) reinterpret_cast<cpx<T> *>(t.out)[w * a.og + k] = v;
    } else {
      reinterpret_cast<T *>(t.out)[w * a.og + k] = v.x;
    }
  }
}

// Last-stage writer: outputs j + q * nb of transform w.
template <typename T, int KIND, bool REAL>
struct Sink {
  const Tile<T> *t;
  int zbuf;
  template <int R>
  FFB_HD void put(int w, int j, int nb, const cpx<T> (&v)[R]) const {
    const TileArgs<T> &a = *t->a;
    if (w >= t->wlive) return;
    cpx<T> *zb = t->buf(w, zbuf);
    if constexpr (KIND == 1) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int k = j + q * nb;
        if (k < t->nl) put_result<T, REAL>(*t, w, k, cmul(v[q], ldg_c(a.chirp + k)), zb);
      }
    } else if constexpr (KIND == 2) {
      const cpx<T> x0 = t->extra[w];
#pragma unroll
      for (int q = 0; q < R; ++q) put_result<T, REAL>(*t, w, ldg_v(a.perm_out + j + q * nb), x0 + v[q], zb);
    } else if constexpr (KIND == 0 && !REAL) {
      if (a.chirp_mode == 2) {
        const long long n = a.n, g = t->g0 + w;
        cpx<T> *p = reinterpret_cast<cpx<T> *>(t->out) + w * a.og;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const int k = j + q * nb;
          const long long c = (long long)k * a.cj_e + g * a.cj_g;
          if (c < n) p[(long long)k * a.ok] = cmul(v[q], ldg_c(a.chirp + c));
        }
      } else if (a.post_twiddle) {
#pragma unroll
        for (int q = 0; q < R; ++q) put_result<T, false>(*t, w, j + q * nb, v[q], zb);
      } else {
        cpx<T> *p = reinterpret_cast<cpx<T> *>(t->out) + w * a.og + (long long)j * a.ok;
        const long long step = (long long)nb * a.ok;
#pragma unroll
        for (int q = 0; q < R; ++q) p[q * step] = v[q];
      }
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) put_result<T, REAL>(*t, w, j + q * nb, v[q], zb);
    }
  }
};

// The forward chain's last stage of a convolution: times the kernel spectrum
// (natural order), then the inverse chain's first stage -- its radices are the
// forward chain's reversed, so butterfly j takes the same R values -- into
// shared memory in that stage's transposed layout; a Rader core's X0 = x0 +
// DC on the way.
template <typename T, int KIND>
struct KernelSink {
  const Tile<T> *t;
  int b;
  template <int R>
  FFB_HD void put(int w, int j, int nb, const cpx<T> (&v)[R]) const {
    const TileArgs<T> &a = *t->a;
    const cpx<T> *kern = a.kern;
    if constexpr (KIND == 3) kern += (t->g0 + t->wc(w)) * a.kern_stride;
    cpx<T> *p = t->buf(w, b) + j;
    if constexpr (KIND == 2) {
      if (j == 0) t->extra[a.W + w] = v[0] + t->extra[w];
    }
    cpx<T> y[R];
#pragma unroll
    for (int q = 0; q < R; ++q) y[q] = cmul(v[q], ldg_c(kern + j + q * nb));
    dft_fixed<R, true, T>(y);
#pragma unroll
    for (int q = 0; q < R; ++q) p[q * (nb | 1)] = y[q];
  }
};

// Radix sets of the kernels.  The codelets a kernel holds set its registers,
// and those its warps per SM: set 0 leaves out the large ones (single
// precision 11, 13, 17, 19; double everything above 10), which takes the
// kernel from 128 / 255 registers to 80 / 128 -- three / two 256-thread CTAs
// per SM instead of two / one.  The executor picks a chain from set 0
// whenever the length has one.
template <typename T>
FFB_HD constexpr bool in_set(int set, int R) {
  return set == 1 || R <= 10 || (sizeof(T) == 4 && (R == 12 || R == 15 || R == 16));
}
#define FFB_MIXED_CASE(R, CALL) \
  case R:                       \
    if constexpr (in_set<T>(SET, R)) CALL(R) break;
#define FFB_MIXED_SWITCH(R_, CALL)                                                                       \
  switch (R_) {                                                                                          \
    FFB_MIXED_CASE(2, CALL) FFB_MIXED_CASE(3, CALL) FFB_MIXED_CASE(4, CALL) FFB_MIXED_CASE(5, CALL)      \
    FFB_MIXED_CASE(6, CALL) FFB_MIXED_CASE(7, CALL) FFB_MIXED_CASE(8, CALL) FFB_MIXED_CASE(9, CALL)      \
    FFB_MIXED_CASE(10, CALL) FFB_MIXED_CASE(11, CALL) FFB_MIXED_CASE(12, CALL) FFB_MIXED_CASE(13, CALL)  \
    FFB_MIXED_CASE(15, CALL) FFB_MIXED_CASE(16, CALL) FFB_MIXED_CASE(17, CALL) FFB_MIXED_CASE(19, CALL)  \
    default: break;                                                                                      \
  }

template <int R, bool INV, typename T>
FFB_HD void twiddled_dft(cpx<T> (&v)[R], const cpx<T> *row, int Ns) {
#pragma unroll
  for (int r = 1; r < R; ++r) v[r] = cmul(v[r], ldg_c(row + (r - 1) * Ns));
  dft_fixed<R, INV, T>(v);
}

// All stages of core c in direction INV: stage 0 reads through src, the last
// writes through sink, the ones between alternate between the two buffers;
// stage 0 writes buffer b.  A single codelet (SINGLE: batch programs, whose
// convolution rows may be one too) reads and writes with nothing between.
// wfast_in / wfast_out: consecutive threads take consecutive transforms in the
// first / last stage (strided layouts).  START = 1: stage 0 is already in
// buffer b.
template <bool INV, int SET, typename T, bool SINGLE = false, int START = 0, class X, class Src, class MakeSink>
FFB_HD void run_chain(const Tile<T> &t, const Core &c, const cpx<T> *__restrict__ tw, const X &x, const Src &src,
                      const MakeSink &make_sink, int b, bool wfast_in, bool wfast_out) {
  const TileArgs<T> &a = *t.a;
  const int W = a.W, L = c.L, R0 = c.radix[0], nb0 = L / R0, P0 = nb0 | 1, S = c.nst;
  const int t0 = x.tid(), nt = x.nthreads();
  auto split = [&](int e, int s, int nb, bool wfast, int &w, int &j) FFB_INL {
    if (wfast) {
      j = (int)fdiv((uint32_t)e, a.wdiv);
      w = e - j * W;
    } else {
      w = (int)fdiv((uint32_t)e, c.rdiv[s]);
      j = e - w * nb;
    }
  };
  if (S == 1) {
    if constexpr (SINGLE) {
      const auto sink = make_sink(b);
#define FFB_MIXED_ONLY(R)                                                       \
  {                                                                             \
    _Pragma("unroll 1") for (int e = t0; e < W; e += nt) {                      \
      cpx<T> v[R];                                                              \
      if constexpr (START == 0) {                                               \
        src.template get<R>(e, 0, 1, v);                                        \
        dft_fixed<R, INV, T>(v);                                                \
      } else {                                                                  \
        const cpx<T> *p = t.buf(e, b);                                          \
        _Pragma("unroll") for (int r = 0; r < R; ++r) v[r] = p[r];              \
      }                                                                         \
      sink.template put<R>(e, 0, 1, v);                                         \
    }                                                                           \
  }
      FFB_MIXED_SWITCH(R0, FFB_MIXED_ONLY)
#undef FFB_MIXED_ONLY
    }
    return;
  }
  // stage 0: unit twiddles, output q of butterfly j at q * P0 + j
#define FFB_MIXED_FIRST(R)                                        \
  {                                                               \
    _Pragma("unroll 1") for (int e = t0; e < W * nb0; e += nt) {  \
      int w, j;                                                   \
      split(e, 0, nb0, wfast_in, w, j);                           \
      cpx<T> v[R];                                                \
      src.template get<R>(w, j, nb0, v);                          \
      dft_fixed<R, INV, T>(v);                                    \
      cpx<T> *p = t.buf(w, b) + j;                                \
      _Pragma("unroll") for (int q = 0; q < R; ++q) p[q * P0] = v[q]; \
    }                                                             \
  }
  if constexpr (START == 0) {
    FFB_MIXED_SWITCH(R0, FFB_MIXED_FIRST)
    x.sync();
  }
#undef FFB_MIXED_FIRST
  for (int s = 1; s < S - 1; ++s) {
    const int Ns = c.span[s];
    const cpx<T> *blk = tw + c.twoff[s];
#define FFB_MIXED_MID(R)                                                      \
  {                                                                           \
    const int nb = L / R, step = s == 1 ? nb / R0 : nb;                       \
    _Pragma("unroll 1") for (int e = t0; e < W * nb; e += nt) {               \
      int w, j;                                                               \
      split(e, s, nb, false, w, j);                                           \
      const int g = (int)fdiv((uint32_t)j, c.sdiv[s]), k = j - g * Ns;        \
      const cpx<T> *rp = t.buf(w, b) + (s == 1 ? k * P0 + g : j);             \
      cpx<T> v[R];                                                            \
      _Pragma("unroll") for (int r = 0; r < R; ++r) v[r] = rp[r * step];      \
      twiddled_dft<R, INV, T>(v, blk + k, Ns);                                \
      cpx<T> *wp = t.buf(w, 1 - b) + g * Ns * R + k;                          \
      _Pragma("unroll") for (int q = 0; q < R; ++q) wp[q * Ns] = v[q];        \
    }                                                                         \
  }
    FFB_MIXED_SWITCH(c.radix[s], FFB_MIXED_MID)
#undef FFB_MIXED_MID
    x.sync();
    b = 1 - b;
  }
  const int s = S - 1;
  const cpx<T> *blk = tw + c.twoff[s];
  const auto sink = make_sink(1 - b);
#define FFB_MIXED_LAST(R)                                                \
  {                                                                      \
    const int nb = L / R, step = s == 1 ? nb / R0 : nb, rs = s == 1 ? P0 : 1; \
    _Pragma("unroll 1") for (int e = t0; e < W * nb; e += nt) {          \
      int w, j;                                                          \
      split(e, s, nb, wfast_out, w, j);                                  \
      const cpx<T> *rp = t.buf(w, b) + j * rs;                           \
      cpx<T> v[R];                                                       \
      _Pragma("unroll") for (int r = 0; r < R; ++r) v[r] = rp[r * step]; \
      twiddled_dft<R, INV, T>(v, blk + j, nb);                           \
      sink.template put<R>(w, j, nb, v);                                 \
    }                                                                    \
  }
  FFB_MIXED_SWITCH(c.radix[s], FFB_MIXED_LAST)
#undef FFB_MIXED_LAST
}

// Buffer the last stage of a chain that starts in buffer b reads.
FFB_HD int last_buffer(const Core &c, int b) { return (c.nst & 1) ? 1 - b : b; }

// One CTA tile of a pass: KIND 0 a Dit core in direction INV, 1 a fused
// Bluestein, 2 a fused Rader, 3 a convolution row; REAL: any of the real
// IoKinds (io), else complex in and out.
template <typename T, int KIND, bool REAL, bool INV, int SET, bool SINGLE = false, class X>
FFB_HD void body(const TileArgs<T> &a, int io, long long bx, long long by, cpx<T> *sm, const X &x) {
  const bool real_in = REAL && (io == (int)IoKind::R2C || io == (int)IoKind::R2CFull);
  const bool real_out = REAL && (io == (int)IoKind::C2R || io == (int)IoKind::C2RFull);
  const bool half = REAL && (io == (int)IoKind::R2C || io == (int)IoKind::C2R);
  const int W = a.W;
  const int nbuf = buffers(a.core, (CoreKind)KIND, (IoKind)io);
  Tile<T> t;
  t.a = &a;
  t.g0 = bx * W;
  t.in = reinterpret_cast<const unsigned char *>(a.in) +
         (by * a.ib + t.g0 * a.ig) * (long long)(real_in ? sizeof(T) : sizeof(cpx<T>));
  t.out = reinterpret_cast<unsigned char *>(a.out) +
          (by * a.ob + t.g0 * a.og) * (long long)(real_out ? sizeof(T) : sizeof(cpx<T>));
  t.wlive = (int)((a.G - t.g0) < W ? (a.G - t.g0) : W);
  t.slot = slot_len(a.core, nbuf);
  t.blen = buf_len(a.core);
  t.io = io;
  t.nl = half ? a.n / 2 : a.n;
  t.sm = sm;
  t.extra = sm + (size_t)W * t.slot;
  const int t0 = x.tid(), nt = x.nthreads();

  int b = 0;  // buffer the first stage writes
  if constexpr (REAL) {
    if (io == (int)IoKind::C2R) {
      // Hermitian pre step, both bins of a pair: with S = X_k + conj X_m,
      // D = X_k - conj X_m, m = n/2 - k and y = conj(W_n^k) D,
      //   Z_k = S + i y,  Z_m = conj(S - i y);
      // Im X_0 and Im X_{n/2} are ignored
      const int h = t.nl, pairs = h / 2 + 1;
      for (int e = t0; e < W * pairs; e += nt) {
        const int w = (int)fdiv((uint32_t)e, a.pairs_div), k = e - w * pairs, m = h - k;
        const cpx<T> *row = reinterpret_cast<const cpx<T> *>(t.in) + t.wc(w) * a.ig;
        cpx<T> xk = ldg_c(row + k), xm = ldg_c(row + m);
        if (k == 0) {
          xk.y = (T)0;
          xm.y = (T)0;
        }
        const cpx<T> sv = mk(xk.x + xm.x, xk.y - xm.y), d = mk(xk.x - xm.x, xk.y + xm.y);
        const cpx<T> wk = ldg_c(a.rtw + k);
        const cpx<T> y = mk(d.x * wk.x + d.y * wk.y, d.y * wk.x - d.x * wk.y);
        cpx<T> *z = t.buf(w, 0);
        z[k] = mk(sv.x - y.y, sv.y + y.x);
        if (m != k && k != 0) z[m] = mk(sv.x + y.y, y.x - sv.y);
      }
      x.sync();
      b = 1;
    }
  }
  if constexpr (KIND == 2) {
    for (int w = t0; w < W; w += nt) t.extra[w] = core_input<T, REAL>(t, t.wc(w), 0, t.buf(w, 0));
    // (the first barrier of the chain comes before x0 is read)
  }
  const bool win = a.wfast != 0, wout = a.ok > a.og;
  const Source<T, KIND, REAL> src{&t, 0};
  if constexpr (KIND == 0) {
    run_chain<INV, SET, T, SINGLE>(t, a.core, a.tw, x, src, [&](int ob) FFB_INL { return Sink<T, KIND, REAL>{&t, ob}; }, b, win,
                      wout);
    b = 1 - last_buffer(a.core, b);  // where a shared-memory result is
  } else {
    run_chain<false, SET, T, SINGLE>(t, a.core, a.tw, x, src,
                                     [&](int ob) FFB_INL { return KernelSink<T, KIND>{&t, ob}; }, b, win, false);
    x.sync();
    b = 1 - last_buffer(a.core, b);  // the product, through the inverse chain's first stage
    run_chain<true, SET, T, SINGLE, 1>(t, a.core2, a.tw2, x, src,
                                       [&](int ob) FFB_INL { return Sink<T, KIND, REAL>{&t, ob}; }, b, false, wout);
    b = 1 - last_buffer(a.core2, b);
    if constexpr (KIND == 2) {
      for (int w = t0; w < t.wlive; w += nt) put_result<T, REAL>(t, w, 0, t.extra[W + w], t.buf(w, b));
    }
  }
  if constexpr (REAL) {
    if (io == (int)IoKind::R2C) {
      // Hermitian post step, both bins of a pair: E = (Z_k + conj Z_m) / 2,
      // O = -i (Z_k - conj Z_m) / 2, X_k = E + W_n^k O, X_m = conj(E - W_n^k O)
      x.sync();
      const int h = t.nl, pairs = h / 2 + 1;
      for (int e = t0; e < t.wlive * pairs; e += nt) {
        const int w = (int)fdiv((uint32_t)e, a.pairs_div), k = e - w * pairs, m = h - k;
        const cpx<T> *z = t.buf(w, b);
        const cpx<T> zk = z[k], zm = z[k == 0 ? 0 : m];
        const cpx<T> ev = mk((zk.x + zm.x) * (T)0.5, (zk.y - zm.y) * (T)0.5);
        const cpx<T> od = mk((zk.y + zm.y) * (T)0.5, (zm.x - zk.x) * (T)0.5);
        const cpx<T> wo = cmul(ldg_c(a.rtw + k), od);
        cpx<T> *row = reinterpret_cast<cpx<T> *>(t.out) + w * a.og;
        row[k] = ev + wo;
        if (m != k) row[m] = mk(ev.x - wo.x, wo.y - ev.y);
      }
    }
  }
}

// Threads per CTA at most, and the CTAs of that size per SM a radix set's
// registers leave room for.
constexpr int kMaxThreads = 256;
template <typename T>
FFB_HD constexpr int min_blocks(int set) {
  return (sizeof(T) == 4 ? 2 : 1) + (set == 0 ? 1 : 0);
}

template <typename T, int KIND, bool REAL, bool INV, int SET>
__global__ void __launch_bounds__(kMaxThreads, min_blocks<T>(SET)) k_mixed(const __grid_constant__ TileArgs<T> a,
                                                                          int io) {
  pdl_entry();
  extern __shared__ __align__(16) unsigned char smraw[];
  body<T, KIND, REAL, INV, SET>(a, io, (long long)blockIdx.x, (long long)blockIdx.y,
                                reinterpret_cast<cpx<T> *>(smraw), tile::DevX{1, 0});
}

template <typename T, int KIND, bool REAL, bool INV, int SET>
cudaError_t launch_set(const TileArgs<T> &a, int io, size_t smem, cudaStream_t s) {
  const long long tiles = (a.G + a.W - 1) / a.W;
#ifndef FFB_HOST_EMULATION
  cudaError_t e = set_smem_limit_once<k_mixed<T, KIND, REAL, INV, SET>>(232448);
  if (e != cudaSuccess) return e;
  return launch_pdl(k_mixed<T, KIND, REAL, INV, SET>, dim3((unsigned)tiles, (unsigned)a.nbatch),
                    dim3((unsigned)a.mixed), smem, s, a, io);
#else
  std::vector<unsigned char> buf(smem + 64);
  cpx<T> *sm = reinterpret_cast<cpx<T> *>(buf.data());
  for (long long by = 0; by < a.nbatch; ++by)
    for (long long bx = 0; bx < tiles; ++bx) {
      std::memset(buf.data(), 0xff, buf.size());
      body<T, KIND, REAL, INV, SET>(a, io, bx, by, sm, tile::HostX{});
    }
  return cudaSuccess;
#endif
}
template <typename T, int KIND, bool REAL, bool INV>
cudaError_t launch_one(const TileArgs<T> &a, int io, size_t smem, cudaStream_t s) {
  return a.mixed_set == 0 ? launch_set<T, KIND, REAL, INV, 0>(a, io, smem, s)
                          : launch_set<T, KIND, REAL, INV, 1>(a, io, smem, s);
}

// Launches core kind K over a pass (TileArgs::mixed threads per CTA).
template <typename T, int K>
cudaError_t launch(const TileArgs<T> &a0, IoKind io, size_t smem, cudaStream_t s) {
  TileArgs<T> a = a0;
  if (io == IoKind::C2C) {
    if constexpr (K == 0)
      return a.inv ? launch_one<T, 0, false, true>(a, 0, smem, s) : launch_one<T, 0, false, false>(a, 0, smem, s);
    else
      return launch_one<T, K, false, false>(a, 0, smem, s);
  }
  if constexpr (K == 3) {
    return cudaErrorInvalidValue;
  } else {
    // the rows of reals move as pairs when every row starts on a pair
    const void *base = io == IoKind::R2C ? a.in : a.out;
    const long long dist = io == IoKind::R2C ? a.ig : a.og;
    a.pair_aligned = reinterpret_cast<uintptr_t>(base) % sizeof(cpx<T>) == 0 && dist % 2 == 0;
    if constexpr (K == 0)
      return a.inv ? launch_one<T, 0, true, true>(a, (int)io, smem, s)
                   : launch_one<T, 0, true, false>(a, (int)io, smem, s);
    else
      return launch_one<T, K, true, false>(a, (int)io, smem, s);
  }
}

}  // namespace mixed
}  // namespace ffb
