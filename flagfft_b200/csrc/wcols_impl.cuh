// Host side of the wide column passes (wcols.cuh): which passes take them, the
// tile view and the launch; part of k_f32_tcols.cu, beside the column kernel
// whose views and tensor maps it shares.  The host-emulation build runs the
// same tile loop on the CPU.
#pragma once

#include "tcols_impl.cuh"
#include "wcols.cuh"

namespace ffb {
namespace wcols {

// Tiles per SM from which a pass runs here and not on the column kernel,
// whose 64 KB groups keep three copies in flight and fill the SMs from half
// as many columns.  Measured (us, column kernel -> here): 1.7 tiles per SM
// (C2C 2^22 x 1) 45.0 -> 46.0, (2-D 2048 x 2048) 31.9 -> 33.1; 6.9 (2-D 4096 x
// 4096) 164 -> 142; 13.8 (R2C + C2R 2^24 x 4) 1003 -> 821.
constexpr long long kMinTilesPerSm = 4;

#ifndef FFB_HOST_EMULATION
inline long long min_tiles() { return kMinTilesPerSm * tcols::sm_count(); }
#else
inline long long min_tiles() { return kMinTilesPerSm; }  // (so small passes exercise it)
#endif

// False when the pass has too few tiles, or a layout or buffer the tensor
// copy or the writer does not take.
template <int L, class Sh>
bool make_args(const TileArgs<float> &a, Args *p, bool *out_rows) {
  if (a.G < Sh::W || a.G >= (1ll << 30) || a.nbatch * (a.G / Sh::W) < min_tiles()) return false;
  if (a.ig != 1 || a.ii < a.G || a.G % 2 != 0) return false;
  *out_rows = a.ok == 1 && a.og >= L;
  // rows of 1024 points: the column kernel writes them faster (C2C 2^20 x 16 140
  // us here, 132 there, R2C 2^21 x 16 197 / 187; 1536 x 2048 points x 8 210 / 224,
  // 2^22 x 8 262 / 290)
  if (*out_rows && L < 1536) return false;
  if (!*out_rows && (a.og != 1 || a.ok < a.G)) return false;
  // outputs off 16 bytes, two stores for one: the tile kernel is faster (C2C
  // 2^24 x 4 2044 us here, 1601 there, 2^23 x 4 882 / 764)
  p->out_aligned = reinterpret_cast<uintptr_t>(a.out) % 16 == 0 && a.ok % 2 == 0 && (a.nbatch == 1 || a.ob % 2 == 0);
  if (!*out_rows && !p->out_aligned) return false;
  int in_rows = 0;
  if (!tcols::make_view<float, L, Sh::W, Sh::RB>(a.in, a.nbatch, a.G, a.ib, a.ig, a.ii, &p->in_view, &in_rows) || in_rows)
    return false;
  p->a = a;
  p->tiles_per_batch = (a.G + Sh::W - 1) / Sh::W;
  p->total_tiles = p->tiles_per_batch * a.nbatch;
  return true;
}

#ifndef FFB_HOST_EMULATION

template <bool INV, int L, int... Rs>
cudaError_t launch_seq(const TileArgs<float> &a, cudaStream_t s) {
  using Sh = Shape<L, Rs...>;
  Args p{};
  bool out_rows = false;
  if (!make_args<L, Sh>(a, &p, &out_rows)) return cudaErrorNotSupported;
  if (!tcols::encode<float>(p.in_view, &p.in_map)) return cudaErrorNotSupported;
  const long long ctas = std::min<long long>(p.total_tiles, tcols::sm_count());
  cudaError_t e;
#define FFB_WCOLS_GO(OR)                                                                                     \
  {                                                                                                          \
    auto k = k_wcols<INV, L, OR, Rs...>;                                                                     \
    if ((e = set_smem_limit_once<k_wcols<INV, L, OR, Rs...>>((int)Sh::smem)) != cudaSuccess) return e;       \
    return launch_pdl(k, dim3((unsigned)ctas), dim3(Sh::NT), Sh::smem, s, p);                                \
  }
  if constexpr (L >= 1536) {
    if (out_rows) FFB_WCOLS_GO(true)
  }
  FFB_WCOLS_GO(false)
#undef FFB_WCOLS_GO
}

#else  // FFB_HOST_EMULATION

// The kernel's shared-memory image and its tile loop, every step over all
// threads in turn.
template <bool INV, int L, bool OR, class Sh>
void emulate(const Args &p) {
  std::vector<unsigned char> image(Sh::smem + 1024, 0xff);
  unsigned char *base = image.data() + (1024 - (reinterpret_cast<uintptr_t>(image.data()) & 1023));
  C32 *land = reinterpret_cast<C32 *>(base + Sh::head);
  F2 *ex = reinterpret_cast<F2 *>(base + Sh::ex_at);
  C32 *ptw = reinterpret_cast<C32 *>(base + Sh::ptw_at);
  C32 *tw = reinterpret_cast<C32 *>(base + Sh::tw_at);
  for (int t = 0; t < Sh::NT; ++t) fill_twiddles<Sh>(tw, p.a.tw, t);
  const rows::HostT x{};
  for (long long q = 0; q < p.total_tiles; ++q) {
    const long long b = q / p.tiles_per_batch, g0 = (q - b * p.tiles_per_batch) * Sh::W;
    std::memset(base, 0xff, Sh::tw_at);
    tma::emulate_box(p.in_view, (int)(2 * g0), 0, 0, (int)b, land, true);
    auto st = x.first(Sh::NT, [&](int tid) {
      typename StageOf<Sh, 0>::Regs r;
      take_tile<Sh>(tid, r, land);
      stage_math<INV, Sh, 0, true>(tid, r, tw);
      return r;
    });
    for (int t = 0; t < Sh::NT; ++t) fill_ptw<Sh>(t, p.a, g0, ptw);
    for (int t = 0; t < Sh::NT; ++t) put_half<Sh, 0, 0>(t, st[(size_t)t], ex);
    exchange<INV, Sh, OR, 0>(x, st, ex, tw, p, b, g0, ptw);
  }
}

template <bool INV, int L, int... Rs>
cudaError_t launch_seq(const TileArgs<float> &a, cudaStream_t) {
  using Sh = Shape<L, Rs...>;
  Args p{};
  bool out_rows = false;
  if (!make_args<L, Sh>(a, &p, &out_rows)) return cudaErrorNotSupported;
  if (out_rows)
    emulate<INV, L, true, Sh>(p);
  else
    emulate<INV, L, false, Sh>(p);
  return cudaSuccess;
}

#endif

// Threads and shared memory of the kernel for a pass whose buffers keep the
// copy rules; false when the column kernel takes it.
inline bool shape_any(const TileArgs<float> &a, int *threads, size_t *smem) {
  if (a.chirp_mode != 0 || a.nbatch <= 0) return false;
  alignas(16) static unsigned char probe[16];
  TileArgs<float> b = a;
  b.in = b.out = probe;
  Args p{};
  bool out_rows = false;
#define FFB_WCOLS_SHAPE(L, ...)                      \
  if (tile::core_is<L, __VA_ARGS__>(a.core)) {       \
    *threads = Shape<L, __VA_ARGS__>::NT;            \
    *smem = Shape<L, __VA_ARGS__>::smem;             \
    return make_args<L, Shape<L, __VA_ARGS__>>(b, &p, &out_rows); \
  }
  FFB_TCOLS_SEQUENCES(FFB_WCOLS_SHAPE)
#undef FFB_WCOLS_SHAPE
  return false;
}

// cudaErrorNotSupported: the column kernel takes the pass.
inline cudaError_t launch_any(const TileArgs<float> &a, cudaStream_t s) {
  if (a.chirp_mode != 0 || a.nbatch <= 0) return cudaErrorNotSupported;
#define FFB_WCOLS_TRY(L, ...)               \
  if (tile::core_is<L, __VA_ARGS__>(a.core)) \
    return a.inv ? launch_seq<true, L, __VA_ARGS__>(a, s) : launch_seq<false, L, __VA_ARGS__>(a, s);
  FFB_TCOLS_SEQUENCES(FFB_WCOLS_TRY)
#undef FFB_WCOLS_TRY
  return cudaErrorNotSupported;
}

}  // namespace wcols
}  // namespace ffb
