// Wide column passes: many columns of long compile-time sequences (1024, 1536,
// 2048, 4096 points) in single precision.
//
// A strided pass over transforms of L points (element i of transform g at
// g + i * ii: a column of a row-major matrix) is coalesced only when a CTA
// moves several adjacent columns at once.  The column kernel of tcols.cuh
// holds 8192 points a tile and three tiles; here a persistent CTA of up to
// 512 threads walks tiles of W adjacent columns with W * L = 16384 points (32
// to 128 bytes of every row, twice its segments) through one landing buffer:
//   * a tile lands in shared memory by one TMA tensor copy while the tile
//     before it is transformed: the last warp that has taken a tile to
//     registers issues the next tile's copy over it;
//   * a thread holds sixteen elements of two columns as packed pairs
//     (packed.cuh), half the arithmetic instructions;
//   * between stages the values change threads through an exchange buffer of
//     half a tile, real parts first, then imaginary parts (a barrier on each
//     side), so landing buffer, exchange and twiddle table fit one SM;
//   * the last stage writes its results, with the optional four-step
//     post-twiddle, straight to global memory: whole W-column segments of a
//     row, or runs of a transform's elements for a row-layout output.
// In the exchange element i of column pair p is at p * (L + PAD) + (i ^
// ((i >> 4) & 15)): the radix-16 Stockham strides then fall on distinct
// banks, and PAD puts the column pairs of one wavefront on distinct banks.
//
// Measured on one B200 against tcols.cuh's kernel: the passes of R2C + C2R
// 2^24 x 4 (2048 and 4096 points) 1003 -> 821 us with the Hermitian passes,
// 2-D 4096 x 4096 164 -> 142 us.  A pass moves 3.2 to 3.3 TB/s (537 MB each of
// the four of 2^24 x 4 in 163 us, the 268 MB of 4096 x 4096 in 85); a plain copy
// of the same 32-byte row segments moves 4.3, one of 128-byte segments 5.1, so
// what bounds it is the strided traffic, then the lockstep of one CTA's
// stages.  Tried and not kept: thread copies (cp.async) instead of TMA, which
// hold the warps at the load unit at sixteen lines an instruction (2-D 4096 x
// 4096 167 us); the same kernel in double precision, no faster than tcols
// (Z2Z 2-D 2048 x 2048 58.7 -> 64.6 us, D2Z 3 * 2^20 x 2 82.7 -> 82.4); tiles
// of a quarter of the columns for small passes (C2C 2^19 x 1 20 -> 30 us).
#pragma once

#include "packed.cuh"
#include "rows.cuh"
#include "tma.cuh"

namespace ffb {
namespace wcols {

using C32 = cpx<float>;
using rows::Seq;

// Shared-memory twiddle table of sequence Q, as pairs (rows::TW_PAIRS): stage
// s > 0 block at tw_off_of(s), of 2 * floor(R_s / 2) * span_s entries (stage 0
// reads none).
template <class Q>
FFB_HD constexpr int tw_off_of(int s) {
  int o = 0;
  for (int i = 1; i < s; ++i) o += 2 * (Q::r(i) / 2) * Q::span(i);
  return o;
}

template <int L, int... Rs>
struct Shape {
  using Q = Seq<Rs...>;
  static constexpr int TPT = L / 16;           // threads per column pair
  static constexpr int P = 512 / TPT / 2 * 2;  // column pairs per tile
  static constexpr int W = 2 * P;              // columns per tile
  static constexpr int NT = P * TPT;
  static constexpr int RL = Q::r(Q::n - 1);  // last radix
  static constexpr int RB = 256;             // rows per box dimension of a tile copy
  static constexpr int PAD = 16 / P;         // column pairs of one 16-lane wavefront on distinct banks
  static constexpr size_t align128(size_t b) { return (b + 127) / 128 * 128; }
  static constexpr size_t head = 128;  // mbarrier and the count of warps that have taken a tile
  static constexpr size_t tile_bytes = (size_t)L * W * sizeof(C32);
  static constexpr size_t ex_at = head + tile_bytes;
  static constexpr size_t ptw_at = ex_at + align128((size_t)P * (L + PAD) * sizeof(F2));
  // the four-step twiddles W_N^{g q Ns} of the tile's columns
  static constexpr size_t tw_at = ptw_at + align128((size_t)W * RL * sizeof(C32));
  static constexpr size_t smem = tw_at + align128((size_t)tw_off_of<Q>(Q::n) * sizeof(C32));
  static_assert(Q::r(0) == 16 && L % 256 == 0, "the first radix gives the threads per column");
  static_assert(NT % 32 == 0 && NT <= 512 && W * RL <= NT, "one CTA of whole warps");
  static_assert(smem <= 232448, "tile, exchange and tables must fit one CTA's shared memory");
};

// Kernel arguments: the pass, the input's tensor map (device build) and view.
struct alignas(64) Args {
#ifndef FFB_HOST_EMULATION
  CUtensorMap in_map;
#endif
  tma::View in_view;
  TileArgs<float> a;
  long long tiles_per_batch;  // ceil(G / W)
  long long total_tiles;      // tiles_per_batch * nbatch
  int out_aligned;            // adjacent outputs of a column pair go in one 16-byte store (column outputs: always)
};

// W_N^m (conjugated for the inverse) from the two split tables, m < N.
FFB_HD C32 split_root(const TileArgs<float> &a, uint32_t m) {
  const uint32_t hi = fdiv(m, a.ptw_div);
  C32 t = cmul(ldg_c(a.ptw_hi + hi), ldg_c(a.ptw_lo + (m - hi * a.ptw_div.d)));
  if (a.inv) t.y = -t.y;
  return t;
}

// 16 bytes of shared memory: two neighbouring elements.
FFB_HD void lds_pair(const C32 *e, C32 &a, C32 &b) {
#ifdef __CUDA_ARCH__
  const float4 v = *reinterpret_cast<const float4 *>(e);
  a = mk(v.x, v.y);
  b = mk(v.z, v.w);
#else
  a = e[0];
  b = e[1];
#endif
}

// One stage of a thread: U butterflies of radix R (butterfly t + u * TPT, past
// the last one unused).
template <class Sh, int S>
struct StageOf {
  static constexpr int R = Sh::Q::r(S), Ns = Sh::Q::span(S);
  static constexpr int nb = Sh::TPT * 16 / R;  // butterflies per column
  static constexpr int U = (nb + Sh::TPT - 1) / Sh::TPT;
  struct Regs {
    cpx<F2> x[U][R];
  };
  static FFB_HD constexpr bool live(int t, int u) { return nb % Sh::TPT == 0 || t + u * Sh::TPT < nb; }
};

// Thread tid's column pair and index among the pair's threads: column pairs
// fastest where the access runs ALONG a row of the matrix.
template <class Sh, bool ALONG>
FFB_HD void place(int tid, int &p, int &t) {
  p = ALONG ? tid % Sh::P : tid / Sh::TPT;
  t = ALONG ? tid / Sh::P : tid % Sh::TPT;
}

FFB_HD constexpr int swz(int i) { return i ^ ((i >> 4) & 15); }

// One half (0 real, 1 imaginary) of stage S's outputs into the exchange.
template <class Sh, int S, int HALF>
FFB_HD void put_half(int tid, const typename StageOf<Sh, S>::Regs &st, F2 *ex) {
  using O = StageOf<Sh, S>;
  int p, t;
  place<Sh, true>(tid, p, t);
  F2 *b = ex + p * (Sh::TPT * 16 + Sh::PAD);
#pragma unroll
  for (int u = 0; u < O::U; ++u) {
    if (!O::live(t, u)) continue;
    const int j = t + u * Sh::TPT, k = O::Ns == 1 ? 0 : j % O::Ns, base = (j - k) * O::R + k;
#pragma unroll
    for (int q = 0; q < O::R; ++q) {
      const F2 v = HALF == 0 ? st.x[u][q].x : st.x[u][q].y;
      if constexpr (O::Ns == 1 && O::R == 16) {
        b[(base + (j & 15)) ^ q] = v;  // swz(16 j + q)
      } else if constexpr (O::Ns == 16 && O::R == 16) {
        b[(base ^ q) + 16 * q] = v;  // swz(base + 16 q): (base >> 4) & 15 is 0
      } else {
        b[swz(base + q * O::Ns)] = v;
      }
    }
  }
}
// One half of stage S's inputs from the exchange: elements j + r * nb.
template <class Sh, int S, int HALF, bool ALONG>
FFB_HD void get_half(int tid, typename StageOf<Sh, S>::Regs &st, const F2 *ex) {
  using O = StageOf<Sh, S>;
  int p, t;
  place<Sh, ALONG>(tid, p, t);
  const F2 *b = ex + p * (Sh::TPT * 16 + Sh::PAD);
#pragma unroll
  for (int u = 0; u < O::U; ++u) {
    if (!O::live(t, u)) continue;
    const int j = t + u * Sh::TPT;
#pragma unroll
    for (int r = 0; r < O::R; ++r) {
      // swz(j + r nb): nb is a multiple of 16, so the block index is j / 16 + r nb / 16
      const F2 v = b[(j ^ (((j >> 4) + r * (O::nb / 16)) & 15)) + r * O::nb];
      if constexpr (HALF == 0)
        st.x[u][r].x = v;
      else
        st.x[u][r].y = v;
    }
  }
}

// Stage S's twiddles and codelets on the values in registers.
template <bool INV, class Sh, int S, bool ALONG>
FFB_HD void stage_math(int tid, typename StageOf<Sh, S>::Regs &st, const C32 *tw) {
  using O = StageOf<Sh, S>;
  int p, t;
  place<Sh, ALONG>(tid, p, t);
#pragma unroll
  for (int u = 0; u < O::U; ++u) {
    if (!O::live(t, u)) continue;
    if constexpr (O::Ns > 1) {
      const C32 *row = tw + tw_off_of<typename Sh::Q>(S) + 2 * ((t + u * Sh::TPT) % O::Ns);
#pragma unroll
      for (int r = 1; r < O::R; r += 2) {
        C32 w0, w1;
        lds_pair(row + (r - 1) * O::Ns, w0, w1);
        st.x[u][r] = mul_tw(st.x[u][r], w0);
        if (r + 1 < O::R) st.x[u][r + 1] = mul_tw(st.x[u][r + 1], w1);
      }
    }
    dft_swapped<O::R, INV>(st.x[u]);
  }
}

// Stage 0's inputs from the landed tile ([row][W columns]).
template <class Sh>
FFB_HD void take_tile(int tid, typename StageOf<Sh, 0>::Regs &st, const C32 *land) {
  int p, t;
  place<Sh, true>(tid, p, t);
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    C32 c0, c1;
    lds_pair(land + (t + r * StageOf<Sh, 0>::nb) * Sh::W + p * 2, c0, c1);
    st.x[0][r] = mk(F2(c0.x, c1.x), F2(c0.y, c1.y));
  }
}

// The last stage's results to global memory, times the post-twiddle W_N^{g k}
// as W^{g j} W^{g q Ns}.  ptw: the second factors, entry q * W + column.
template <bool INV, class Sh, bool OUT_ROWS>
FFB_HD void write_out(int tid, const typename StageOf<Sh, Sh::Q::n - 1>::Regs &st, const Args &args, long long b,
                      long long g0, const C32 *ptw) {
  using O = StageOf<Sh, Sh::Q::n - 1>;
  const TileArgs<float> &a = args.a;
  int p, t;
  place<Sh, !OUT_ROWS>(tid, p, t);
  const long long g = g0 + p * 2;
  if (g >= a.G) return;
  // (a copied row has an even length, so both columns of a pair are live; the
  // branches stay, without them the 1536-point kernel runs 5% longer: 2-D 1536 x
  // 16384 210 -> 224 us)
  const bool both = g + 1 < a.G;
#pragma unroll
  for (int u = 0; u < O::U; ++u) {
    if (!O::live(t, u)) continue;
    const int j = t + u * Sh::TPT;  // nb == Ns in the last stage: outputs j + q * nb
    cpx<F2> t0;
    if (a.post_twiddle) {
      const C32 w0 = split_root(a, (uint32_t)(g * j));
      const C32 w1 = both ? split_root(a, (uint32_t)((g + 1) * j)) : w0;  // dead columns: no reads past the tables
      t0 = mk(F2(w0.x, w1.x), F2(w0.y, w1.y));
    }
    C32 *out = reinterpret_cast<C32 *>(a.out) + b * a.ob + g * a.og + (long long)j * a.ok;
    const long long step = (long long)O::nb * a.ok;
#pragma unroll
    for (int q = 0; q < O::R; ++q) {
      cpx<F2> v = st.x[u][q];
      if (a.post_twiddle) {
        cpx<F2> w = t0;
        if (q > 0) {
          C32 w0, w1;
          lds_pair(ptw + q * Sh::W + p * 2, w0, w1);
          w = mul_each(t0, mk(F2(w0.x, w1.x), F2(w0.y, w1.y)));
        }
        v = mul_each(v, w);
      }
      C32 *o = out + q * step;
      C32 c0, c1;
      v.x.get(c0.x, c1.x);
      v.y.get(c0.y, c1.y);
      if (!OUT_ROWS && args.out_aligned && both) {
#ifdef __CUDA_ARCH__
        *reinterpret_cast<float4 *>(o) = make_float4(c0.x, c0.y, c1.x, c1.y);
#else
        o[0] = c0;
        o[1] = c1;
#endif
      } else {
        o[0] = c0;
        if (both) o[a.og] = c1;
      }
    }
  }
}

// W_N^{g q Ns} of the tile's columns (entry q * W + column), one per thread.
template <class Sh>
FFB_HD void fill_ptw(int tid, const TileArgs<float> &a, long long g0, C32 *ptw) {
  constexpr int Ns = Sh::Q::span(Sh::Q::n - 1);
  if (!a.post_twiddle || tid >= Sh::W * Sh::RL) return;
  const int q = tid / Sh::W;
  const long long g = g0 + tid % Sh::W;
  if (g < a.G) ptw[tid] = split_root(a, (uint32_t)(g * (long long)(q * Ns)));
}

// From stage S's outputs, their real parts already in the exchange, to the
// tile's results: the exchange to stage S + 1, its twiddles and codelets, and
// so on; the last stage writes global memory.  Every step begins with a
// barrier.  Stages take their column pairs fastest over the threads, except
// the last one of a row-layout output.
#pragma nv_exec_check_disable
template <bool INV, class Sh, bool OUT_ROWS, int S, class X, class St>
FFB_HD void exchange(const X &x, const St &s1, F2 *ex, const C32 *tw, const Args &args, long long b, long long g0,
                     const C32 *ptw) {
  constexpr int N = Sh::Q::n;
  static_assert(S + 1 < N, "a sequence has two stages or more");
  constexpr bool last = S + 2 == N, along = !(last && OUT_ROWS);
  using From = typename StageOf<Sh, S>::Regs;
  using To = typename StageOf<Sh, S + 1>::Regs;
  struct Both {
    From f;
    To t;
  };
  auto s2 = x.step(
      Sh::NT,
      [&](int tid, const From &v) FFB_INL {
        Both r;
        r.f = v;
        get_half<Sh, S + 1, 0, along>(tid, r.t, ex);
        return r;
      },
      s1);
  auto s3 = x.step(
      Sh::NT,
      [&](int tid, const Both &v) FFB_INL {
        put_half<Sh, S, 1>(tid, v.f, ex);
        return v.t;
      },
      s2);
  if constexpr (last) {
    x.last(
        Sh::NT,
        [&](int tid, const To &v) FFB_INL {
          To r = v;
          get_half<Sh, S + 1, 1, along>(tid, r, ex);
          stage_math<INV, Sh, S + 1, along>(tid, r, tw);
          write_out<INV, Sh, OUT_ROWS>(tid, r, args, b, g0, ptw);
        },
        s3);
  } else {
    auto s4 = x.step(
        Sh::NT,
        [&](int tid, const To &v) FFB_INL {
          To r = v;
          get_half<Sh, S + 1, 1, along>(tid, r, ex);
          stage_math<INV, Sh, S + 1, along>(tid, r, tw);
          return r;
        },
        s3);
    auto s5 = x.step(
        Sh::NT,
        [&](int tid, const To &v) FFB_INL {
          put_half<Sh, S + 1, 0>(tid, v, ex);
          return v;
        },
        s4);
    exchange<INV, Sh, OUT_ROWS, S + 1>(x, s5, ex, tw, args, b, g0, ptw);
  }
}

// The shared-memory twiddle table from the host's block.
template <class Sh>
FFB_HD void fill_twiddles(C32 *tws, const C32 *g, int tid) {
  using Q = typename Sh::Q;
#pragma unroll
  for (int st = 1; st < Q::n; ++st) {  // (unrolled: the radices fold to constants)
    const int R = Q::r(st), Ns = Q::span(st), pairs = R / 2;
    C32 *blk = tws + tw_off_of<Q>(st);
    const C32 *src = g + Q::twoff(st);
    for (int e = tid; e < 2 * pairs * Ns; e += Sh::NT) {
      const int h = e & 1, mk_ = e >> 1, m = mk_ / Ns, k = mk_ - m * Ns, r = 2 * m + h + 1;
      blk[e] = r <= R - 1 ? ldg_c(src + (r - 1) * Ns + k) : mk(1.0f, 0.0f);
    }
  }
}

#ifndef FFB_HOST_EMULATION

// Device counter of waits that gave up (copies that never landed).
static __device__ int g_wcols_wait_failures;

// Warps' arrival at a tile taken to registers: true for the last one's lane 0.
template <int WARPS>
__device__ __forceinline__ bool last_reader(unsigned *readers) {
  __syncwarp();
  if ((threadIdx.x & 31) != 0) return false;
  __threadfence_block();
  const bool last = (atomicAdd(readers, 1u) + 1) % WARPS == 0;
  if (last) __threadfence_block();
  return last;
}

// One CTA per SM walks tiles blockIdx.x, + gridDim.x, ...: neighbouring CTAs
// take neighbouring columns, whose copies share lines in L2.  `full` counts a
// landed tile's bytes; every wait on it is bounded: a wait that gives up is
// counted in g_wcols_wait_failures, the threads leave the loop together and
// thread 0 lets the copies in flight land before the CTA ends.
template <bool INV, int L, bool OUT_ROWS, int... Rs>
__global__ void __launch_bounds__(Shape<L, Rs...>::NT, 1) k_wcols(const __grid_constant__ Args p) {
  pdl_entry();
  using Sh = Shape<L, Rs...>;
  constexpr int WARPS = Sh::NT / 32;
  extern __shared__ __align__(1024) unsigned char smraw[];
  uint64_t *full = reinterpret_cast<uint64_t *>(smraw);
  unsigned *readers = reinterpret_cast<unsigned *>(smraw + 16);
  C32 *land = reinterpret_cast<C32 *>(smraw + Sh::head);
  F2 *ex = reinterpret_cast<F2 *>(smraw + Sh::ex_at);
  C32 *ptw = reinterpret_cast<C32 *>(smraw + Sh::ptw_at);
  C32 *tw = reinterpret_cast<C32 *>(smraw + Sh::tw_at);
  const int tid = (int)threadIdx.x;
  const long long first = blockIdx.x, step = gridDim.x;
  auto issue = [&](long long q) {
    const long long b = q / p.tiles_per_batch, g0 = (q - b * p.tiles_per_batch) * Sh::W;
    tma::mbar_expect_tx(full, (uint32_t)Sh::tile_bytes);
    tma::load_4d(land, &p.in_map, (int)(2 * g0), 0, 0, (int)b, full);
  };
  if (tid == 0) {
    tma::mbar_init(full, 1);
    *readers = 0;
    tma::fence_mbar_init();
    if (first < p.total_tiles) issue(first);
  }
  fill_twiddles<Sh>(tw, p.a.tw, tid);
  __syncthreads();  // mbarrier initialised, twiddles in place
  const rows::DevT x{};
  int i = 0;
  bool failed = false;
  for (long long q = first; q < p.total_tiles; q += step, ++i) {
    const bool ok = tma::mbar_wait(full, (uint32_t)(i & 1));
    typename StageOf<Sh, 0>::Regs st;
    take_tile<Sh>(tid, st, land);
    if (last_reader<WARPS>(readers) && ok && q + step < p.total_tiles) issue(q + step);
    stage_math<INV, Sh, 0, true>(tid, st, tw);
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    const long long b = q / p.tiles_per_batch, g0 = (q - b * p.tiles_per_batch) * Sh::W;
    // (the barrier above ends the previous tile's reads of ptw; those of the
    // exchange order its use in the last stage)
    fill_ptw<Sh>(tid, p.a, g0, ptw);
    put_half<Sh, 0, 0>(tid, st, ex);
    exchange<INV, Sh, OUT_ROWS, 0>(x, st, ex, tw, p, b, g0, ptw);
  }
  if (failed && tid == 0) {
    atomicAdd(&g_wcols_wait_failures, 1);
    // tile i's copy, and the next one where every warp had taken tile i
    tma::mbar_wait(full, (uint32_t)(i & 1));
    if (*readers == (unsigned)((i + 1) * WARPS)) tma::mbar_wait(full, (uint32_t)((i + 1) & 1));
  }
}

#endif  // !FFB_HOST_EMULATION

}  // namespace wcols
}  // namespace ffb
