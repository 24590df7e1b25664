// Real row passes with the whole shape fixed at compile time.
//
// An even-length real transform whose half length is one of the compile-time
// radix sequences runs the row kernel's stages (rows.cuh) on its rows read as
// complex pairs.  Forward (R2C): the first stage reads the pairs straight from
// global memory, the last writes its results to the row's shared buffer, and
// the Hermitian post step takes both bins of a pair (k, L - k) from there to
// global memory.  Inverse (C2R): the pre step fills the buffer from both bins
// of a pair, the stages run from it, and the last writes pairs of reals.
// Against the mixed-radix tile kernel every index is a constant and a row
// keeps one buffer instead of two.
//
// Measured on one B200 (in-place tiles, mixed-radix tiles, here): R2C + C2R
// 2048 x 8192 254 -> 103 -> 60.2 us (4.5 TB/s of input and output); 512 x 10000
// forward 37.7 -> 8.9 here.  What bounds it is the Hermitian step's extra round
// trip through shared memory.
#pragma once

#include "rows.cuh"

namespace ffb {
namespace rrows {

using rows::Seq;
using rows::slot_len;
using rows::SmemIO;

// Pairs (k, L - k), k = 0 .. L/2, a thread has in flight.
constexpr int kUnroll = 4;

// Post step of R2C: with E = (Z_k + conj Z_m) / 2, O = -i (Z_k - conj Z_m) / 2
// and m = L - k: X_k = E + W_n^k O, X_m = conj(E - W_n^k O).
template <typename T, int L, class X>
FFB_HD void post(const TileArgs<T> &a, cpx<T> *out, int wlive, const cpx<T> *sm, int nthr, const X &x) {
  constexpr int pairs = L / 2 + 1;
  x.each(nthr, [&](int tid) FFB_INL {
#pragma unroll 2
    for (int e = tid; e < wlive * pairs; e += nthr) {
      const int w = e / pairs, k = e - w * pairs, m = L - k;
      const cpx<T> *z = sm + w * slot_len<L>();
      const cpx<T> zk = z[pp_pos(k)], zm = z[k == 0 ? 0 : pp_pos(m)];
      const cpx<T> ev = mk((zk.x + zm.x) * (T)0.5, (zk.y - zm.y) * (T)0.5);
      const cpx<T> od = mk((zk.y + zm.y) * (T)0.5, (zm.x - zk.x) * (T)0.5);
      const cpx<T> wo = cmul(ldg_c(a.rtw + k), od);
      cpx<T> *row = out + w * a.og;
      row[k] = ev + wo;
      if (m != k) row[m] = mk(ev.x - wo.x, wo.y - ev.y);
    }
  });
}

// Pre step of C2R: with S = X_k + conj X_m, D = X_k - conj X_m and y =
// conj(W_n^k) D: Z_k = S + i y, Z_m = conj(S - i y); Im X_0 and Im X_L are
// ignored.
template <typename T, int L, class X>
FFB_HD void pre(const TileArgs<T> &a, const cpx<T> *in, int W, int wlive, cpx<T> *sm, int nthr, const X &x) {
  constexpr int pairs = L / 2 + 1;
  x.each(nthr, [&](int tid) FFB_INL {
#pragma unroll 1
    for (int e0 = tid; e0 < W * pairs; e0 += kUnroll * nthr) {
      cpx<T> xk[kUnroll], xm[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int e = e0 + u * nthr;
        if (e >= W * pairs) continue;
        const int w = e / pairs, k = e - w * pairs;
        const cpx<T> *row = in + (w < wlive ? w : wlive - 1) * a.ig;
        xk[u] = rows::ld_stream(row + k);
        xm[u] = rows::ld_stream(row + (L - k));
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int e = e0 + u * nthr;
        if (e >= W * pairs) continue;
        const int w = e / pairs, k = e - w * pairs, m = L - k;
        if (k == 0) {
          xk[u].y = (T)0;
          xm[u].y = (T)0;
        }
        const cpx<T> s = mk(xk[u].x + xm[u].x, xk[u].y - xm[u].y), d = mk(xk[u].x - xm[u].x, xk[u].y + xm[u].y);
        const cpx<T> wk = ldg_c(a.rtw + k);
        const cpx<T> y = mk(d.x * wk.x + d.y * wk.y, d.y * wk.x - d.x * wk.y);
        cpx<T> *z = sm + w * slot_len<L>();
        z[pp_pos(k)] = mk(s.x - y.y, s.y + y.x);
        if (m != k && k != 0) z[pp_pos(m)] = mk(s.x + y.y, y.x - s.y);
      }
    }
  });
}

// One CTA tile of W rows; INV: C2R, else R2C.  Dead rows of the last tile
// compute on the last live row's data and store nothing.
template <typename T, bool INV, int L, int TPT, class X, int... Rs>
FFB_HD void body(const TileArgs<T> &a, int W, long long bx, long long by, cpx<T> *sm, const X &x) {
  using Q = Seq<Rs...>;
  const int nthr = W * TPT;
  const long long g0 = bx * W;
  const int wlive = (int)((a.G - g0) < W ? (a.G - g0) : W);
  const TileArgs<T> *ap = &a;
  auto smem_io = [&](int, cpx<T> *buf) FFB_INL { return SmemIO<T>{buf}; };
  if constexpr (!INV) {
    const T *in = reinterpret_cast<const T *>(a.in) + by * a.ib + g0 * a.ig;
    cpx<T> *out = reinterpret_cast<cpx<T> *>(a.out) + by * a.ob + g0 * a.og;
    auto first = [&](int w, cpx<T> *) FFB_INL {
      const int wc = w < wlive ? w : wlive - 1;
      return rows::GlobalIn<T, 3>{ap, reinterpret_cast<const cpx<T> *>(in + wc * a.ig), g0 + wc};
    };
    rows::run_chain<T, false, L, TPT, false, true, Q, 0>(x, nthr, a.tw, sm, first, smem_io);
    x.sync();
    post<T, L>(a, out, wlive, sm, nthr, x);
  } else {
    const cpx<T> *in = reinterpret_cast<const cpx<T> *>(a.in) + by * a.ib + g0 * a.ig;
    T *out = reinterpret_cast<T *>(a.out) + by * a.ob + g0 * a.og;
    pre<T, L>(a, in, W, wlive, sm, nthr, x);
    x.sync();
    auto last = [&](int w, cpx<T> *) FFB_INL {
      return rows::GlobalOut<T, 3>{ap, reinterpret_cast<cpx<T> *>(out + w * a.og), g0 + w, w < wlive};
    };
    rows::run_chain<T, true, L, TPT, true, false, Q, 0>(x, nthr, a.tw, sm, smem_io, last);
  }
}

template <typename T, bool INV, int MB, int L, int TPT, int... Rs>
__global__ void __launch_bounds__(tile::TileBounds<T>::kMaxThreads, MB)
    k_rrows(const __grid_constant__ TileArgs<T> a, int W) {
  pdl_entry();
  extern __shared__ __align__(16) unsigned char smraw[];
  body<T, INV, L, TPT, rows::DevT, Rs...>(a, W, (long long)blockIdx.x, (long long)blockIdx.y,
                                          reinterpret_cast<cpx<T> *>(smraw), rows::DevT{});
}

// Rows per CTA: the executor's rule for row passes (about 128 threads, no more
// than keeps two CTAs per SM busy); 0 when no CTA holds a row.
template <typename T, int L>
long long rows_per_cta(const TileArgs<T> &a, int tpt) {
  const size_t per = slot_len<L>() * sizeof(cpx<T>);
  if (per > 232448) return 0;
  return std::max<long long>(
      1, std::min<long long>({128 / tpt, (long long)(110 * 1024 / per), a.nbatch * a.G / (2 * 148), (long long)a.G}));
}

// Many rows: the 64-register form (rows.cuh rows_dense says when and why).
// Measured (us, R2C / C2R): 2048 x 8192 31.0 / 35.1 -> 29.5 / 32.8, 8192 x 1024
// 18.5 / 24.6 -> 17.3 / 19.1, 16384 x 512 27.1 / 31.4 -> 22.5 / 25.7; 1024 x 64
// 4.2 / 4.6 -> 6.2 / 6.3, 3072 x 2000 14.2 / 14.5 -> 17.9 / 16.9
template <typename T, int L>
constexpr bool has_dense() {
  return sizeof(T) == 4 && (L & (L - 1)) == 0 && L >= 512 && L <= 8192;
}
template <typename T, int L>
bool run_dense(const TileArgs<T> &a) {
  return has_dense<T, L>() && a.nbatch * a.G * (long long)L >= rows::kDensePoints;
}

template <typename T, bool INV, int L, int... Rs>
cudaError_t launch_seq(const TileArgs<T> &a, cudaStream_t s) {
  if constexpr (slot_len<L>() * sizeof(cpx<T>) > 232448) {  // (no CTA holds such a row)
    (void)a;
    (void)s;
    return cudaErrorNotSupported;
  } else {
  constexpr int TPT = rows::rows_tpt<T, L, Rs...>();
  const size_t per = slot_len<L>() * sizeof(cpx<T>);
  const long long W = rows_per_cta<T, L>(a, TPT);
  const long long tiles = (a.G + W - 1) / W;
#ifndef FFB_HOST_EMULATION
  const dim3 grid((unsigned)tiles, (unsigned)a.nbatch), block((unsigned)(W * TPT));
  if constexpr (has_dense<T, L>()) {
    if (run_dense<T, L>(a)) {
      cudaError_t e = set_smem_limit_once<k_rrows<T, INV, 2, L, TPT, Rs...>>(232448);
      if (e != cudaSuccess) return e;
      return launch_pdl(k_rrows<T, INV, 2, L, TPT, Rs...>, grid, block, (size_t)W * per, s, a, (int)W);
    }
  }
  constexpr int MB = rows::rows_min_blocks<T, 0, L>();
  cudaError_t e = set_smem_limit_once<k_rrows<T, INV, MB, L, TPT, Rs...>>(232448);
  if (e != cudaSuccess) return e;
  return launch_pdl(k_rrows<T, INV, MB, L, TPT, Rs...>, grid, block, (size_t)W * per, s, a, (int)W);
#else
  (void)s;
  std::vector<unsigned char> buf((size_t)W * per + 64);
  cpx<T> *sm = reinterpret_cast<cpx<T> *>(buf.data());
  for (long long by = 0; by < a.nbatch; ++by)
    for (long long bx = 0; bx < tiles; ++bx) {
      std::memset(buf.data(), 0xff, buf.size());
      body<T, INV, L, TPT, rows::HostT, Rs...>(a, (int)W, bx, by, sm, rows::HostT{});
    }
  return cudaSuccess;
#endif
  }
}

// Half-length real rows whose distances keep every row on a pair (the base
// address is checked at launch).
template <typename T>
bool layout_fits(const TileArgs<T> &a, IoKind io) {
  const bool inv = io == IoKind::C2R;
  const long long dist = inv ? a.og : a.ig, bdist = inv ? a.ob : a.ib;
  return dist % 2 == 0 && (a.nbatch <= 1 || bdist % 2 == 0) && (inv ? a.ii : a.ok) == 1 && (inv ? a.ok : a.ii) == 2 &&
         a.nbatch <= 65535;
}

// Shape of the row kernel that runs the pass (rows and threads per CTA, shared
// memory, the 64-register form); false when none does.
template <typename T>
bool shape(const TileArgs<T> &a, IoKind io, TileKernel *k) {
  if (!layout_fits(a, io)) return false;
#define FFB_RROWS_SHAPE(L, ...)                                                \
  if (tile::core_is<L, __VA_ARGS__>(a.core)) {                                 \
    const int tpt = rows::rows_tpt<T, L, __VA_ARGS__>();                       \
    k->W = (int)rows_per_cta<T, L>(a, tpt);                                    \
    k->threads = k->W * tpt;                                                   \
    k->smem = (size_t)k->W * slot_len<L>() * sizeof(cpx<T>);                   \
    k->dense = run_dense<T, L>(a);                                             \
    return k->W > 0;                                                           \
  }
  FFB_FIXED_SEQUENCES(FFB_RROWS_SHAPE)
#undef FFB_RROWS_SHAPE
  return false;
}

// Launches a half-length real pass (IoKind R2C or C2R of a Dit core) on the
// row kernel of its core's sequence; cudaErrorNotSupported when the core is
// not one, or a row of reals does not start on a pair (the mixed-radix or the
// in-place tiles then take it).
template <typename T>
cudaError_t launch(const TileArgs<T> &a, IoKind io, cudaStream_t s) {
  const bool inv = io == IoKind::C2R;
  if (reinterpret_cast<uintptr_t>(inv ? a.out : a.in) % sizeof(cpx<T>) != 0 || !layout_fits(a, io))
    return cudaErrorNotSupported;
#define FFB_RROWS_TRY(L, ...)                \
  if (tile::core_is<L, __VA_ARGS__>(a.core)) \
    return inv ? launch_seq<T, true, L, __VA_ARGS__>(a, s) : launch_seq<T, false, L, __VA_ARGS__>(a, s);
  FFB_FIXED_SEQUENCES(FFB_RROWS_TRY)
#undef FFB_RROWS_TRY
  return cudaErrorNotSupported;
}

}  // namespace rrows
}  // namespace ffb
