// Dispatch of the tensor-core kernel (mma_cl_kernel.cuh): which form of it a call takes.  The
// segmented forms are launched from mma_cl_seg.cu, a translation unit of its own because the register
// allocation that suits their step loop (ptxas --register-usage-level) does not suit the others; for the
// same reason the forms with tiles narrower than 56 channels are launched from mma_cl_narrow.cu.
#include "mma_cl_kernel.cuh"
#include "tmem_ema.cuh"

namespace mega {

// us of the fused pair with real poles as this kernel's chain, from 130 timings (4 to 64 sequences, 128 to 32768 positions, 256 to 2048
// channels on one B200) and 4300 of up to 67 M elements (20 to 6000 positions; these to 0.86 - 1.06 of the time, one in twenty outside):
// a block's start and end, then ns a position by the tiles of 16 channels and 8 sequences, of the wide tiles by waves of them (40 x 94 x
// 1736 with SiLU 38 us, 25 x 1621 x 1528 197; 64 x 8192 x 2048 1.41 ms in a row, with SiLU 1.52).
double mma_chain_us(const StreamArgs& a, bool xn) {
  const double groups = (a.B + kSeq - 1) / kSeq, tiles = ((a.D + 15) / 16) * groups, wide = ((a.D + 63) / 64) * groups, less = ((a.D + 55) / 56) * groups;
  const int v = (xn ? 1 : 0) + (a.mask ? 2 : 0);
  if (wide >= 148. || less >= 148.) {
    static const double kWave[4] = {83., 112., 97., 125.};
    const double w7 = std::ceil(less / 148.), waves = v != 0 ? w7 : std::min(std::ceil(wide / 148.), w7);   // (masks and xn: 56 channels alone)
    const int nsteps = (a.L + kStep - 1) / kStep;
    double us = waves * (27. + a.L * kWave[v] * (waves < 2. ? 1.1 : 1.) * (a.silu ? 1.07 : 1.) * 1e-3), best = waves * 0.96;
    if (v == 0 && wide > 148.)   // in runs, where mma_cl_try takes them
      for (int n = 2; n <= 8; n *= 2)
        if (const double cost = std::ceil(wide * n / 148.) / n; nsteps % n == 0 && nsteps / n >= 64 && cost * 1.02 < best) {
          best = cost * 1.02;
          us = 60. + a.L * cost * (a.silu ? 117. : 93.) * 1e-3;
        }
    return us;
  }
  static const double kFew[4] = {31.3, 48.5, 49., 64.}, kMore[4] = {51., 67.5, 62.5, 81.}, kMany[4] = {1., 1.28, 1.17, 1.53};
  if (tiles <= 148.) return (v == 0 ? 11. : 14.3) + a.L * kFew[v] * 1e-3;
  return tiles <= 296. ? 15.4 + a.L * kMore[v] * 1e-3 : 20.4 + a.L * std::min(0.3 * tiles, 109.) * kMany[v] * 1e-3;
}

// ... and of the EMA by itself: 16-channel tiles while each of them has an SM (16 x 4096 x 1024 101 us, 14 x 3140 x 712 81); between
// that and the segmented form 80 - 170 ns a position.
double mma_ema_chain_us(const StreamArgs& a) {
  const double L = a.L, n = (double)a.B * a.D * L, tiles = ((a.D + 15) / 16) * (double)((a.B + 7) / 8);
  if (a.cplx) return 95. + std::max(L * 29e-3, n / 700e3);
  if (a.mask) return 6. + std::max(L * 42e-3, n / 1300e3);
  const double ns = tiles > 148. && tiles <= 600. ? 0.28 * tiles : 23.2;
  return 6. + std::max(L * ns * 1e-3, n / 1300e3);
}

// Envelope: bf16, channel stride 1, ndim <= 16, a padding mask only with real poles, a
// normalised-copy output (strided like y) only together with the normalisation and distinct from x
// and y, B >= 4 (rows of the MMAs are sequences) unless the pipelined form applies, L < 2^24, and L
// a multiple of 32 when a state is exported.  Returns false, launching nothing, outside of it.
bool mma_cl_try(int dtype, const void* x, void* y, void* xn, long long xsb, long long xsl, long long xsd,
                long long ysb, long long ysl, long long ysd, bool norm, const StreamArgs& a_arg, cudaStream_t s) {
  if (g_options[OPT_DISABLE_MMA].load() != 0) return false;
  StreamArgs a_in = a_arg;
  {
    const int lim = g_options[OPT_WAIT_LIMIT].load(), wh = g_options[OPT_WITHHOLD_LOAD].load();
    a_in.wait_limit = lim > 0 ? (long long)lim : 4000000000LL;
    a_in.withhold_step = wh > 0 ? wh : -1;
  }
  if (dtype != MEGA_BF16 || xsd != 1 || ysd != 1) return false;
  // a padding mask: real poles only
  const bool masked = a_in.mask != nullptr;
  if (masked && a_in.cplx) return false;
  const bool want_xn = xn != nullptr;  // second output: the normalised activations, strided like y
  if (want_xn && (!norm || xn == y || xn == x)) return false;
  const bool ema = a_in.N > 0;  // N = 0: TimestepNorm alone
  if (!ema && (!norm || want_xn || a_in.silu || a_in.h_in || a_in.h_out)) return false;
  const int forced = g_options[OPT_MMA_TILE].load();
  const bool forced_pipe = forced == 222 || forced == 224 || forced == 422 || forced == 124;
  // fewer than 4 sequences leave most rows of the MMAs empty: only the pipelined form, which fills the SMs
  // from the sequence length, is then worth more than the SIMT kernels
  const bool can_pipe = ema && !want_xn && !a_in.cplx && !(a_in.mask != nullptr);
  if (a_in.N > 16 || a_in.N < 0 || (a_in.B < 4 && !(forced_pipe || (forced == 0 && can_pipe))) ||
      a_in.L >= (1 << 24) || a_in.D < 8)
    return false;
  if (a_in.h_out && (a_in.L % kStep) != 0) return false;
  if ((a_in.B + kSeq - 1) / kSeq > 65535) return false;
  // TimestepNorm -> EMA with real poles: statistics by scalar arithmetic and accumulators in tensor memory (16 x 4096 x 1024 88 us
  // against 142, with the second output 107 against 208, masked 106 against 195; 64 x 8192 x 2048 in a row 1.25 ms against 1.41, with
  // SiLU 1.47 against 1.52), or this kernel's chain (some ragged or short shapes).  The power cap takes most of the gain back where
  // all SMs are busy for long: 64 x 32768 x 2048 4.6 to 4.7 ms in a run of 20 launches, 5.1 to 5.2 in a long loop, the chain 5.15 and 5.2.
  // The EMA by itself: 16 x 4096 x 1024 74 us (98 here), 8 x 2000 x 1024 27 (51), 64 x 4096 x 2048 531 (468).
  if (ema && !a_in.cplx && (norm || !masked)) {
    const int asked = forced == 14 ? 4 : forced == 16 ? 9 : forced == 162 ? 10 : forced == 164 ? 12 : forced == 168 ? 16 : 0;
    // (of two that take about as long the one whose variance is 2e-7 off, here 3e-4)
    const bool better = forced == 0 && tmem_ema_us(a_in, norm, want_xn) < (norm ? mma_chain_us(a_in, want_xn) : 0.97 * mma_ema_chain_us(a_in));
    if ((asked > 0 || better) && tmem_ema_try(dtype, x, y, xn, xsb, xsl, ysb, ysl, norm, a_in, s, asked))
      return true;
  }
  // Tile width.  Large problems: 64 channels, or 56 when that fills the 148 SMs in fewer or
  // fuller waves (one CTA per SM; e.g. D = 2048 with 64 sequences: 37 x 8 = 296 CTAs = two full
  // waves).  Problems too small to give every SM a wide tile: 32 or 16 channels per CTA, so
  // that the few (8 sequences x 8 channels) strips there are spread over the SMs; a strip is
  // a serial chain along the sequence, so its speed depends on how few warps share its SM.
  // With the normalisation (three quarters of a step's instructions) such problems take the
  // 16-channel tile with two warps per column: a warp then walks 4 channels per step, e.g.
  // B = 16, L = 4096, D = 1024: 0.29 -> 0.17 ms; B = 8, L = 8192, D = 1024: 0.55 -> 0.30 ms.
  const long long seq_groups = (a_in.B + kSeq - 1) / kSeq;
  auto ctas = [&](int ch) -> long long { return ((a_in.D + ch - 1) / ch) * seq_groups; };
  auto waves_cost = [&](int ch) -> double {
    const long long waves = (ctas(ch) + 147) / 148;
    return (double)waves * ch;  // time ~ waves x work per CTA
  };
  int tile = g_options[OPT_MMA_TILE].load();
  // segmented form (64-channel tile, the sequence in 2, 4 or 8 runs): real EMA, no second output, no mask
  if (tile == 82 || tile == 84 || tile == 88) {
    const int n_seg = tile - 80;
    tile = 0;
    if (can_pipe && a_in.B >= 4) {
      if (mma_cl_segmented(dtype, x, y, xsb, xsl, ysb, ysl, norm, a_in, n_seg, s)) return true;
    } else if (!ema && norm && !masked && a_in.B >= 4) {  // TimestepNorm alone
      if (mma_cl_segmented(dtype, x, y, xsb, xsl, ysb, ysl, true, a_in, n_seg, s)) return true;
    }
  }
  // pipelined forms (real EMA, with or without the normalisation, no second output)
  if ((tile == 222 || tile == 224 || tile == 422 || tile == 124) && (a_in.cplx || !ema || want_xn || masked)) tile = 0;
  if (tile == 71 && (a_in.cplx || !ema || want_xn || masked)) tile = 0;
  if (tile != 2 && tile != 4 && tile != 7 && tile != 8 && tile != 22 && tile != 222 && tile != 224 && tile != 422 &&
      tile != 124 && tile != 71) {
    // (the EMA alone is closer to the memory bound and prefers the 128-byte rows of the 64-channel
    // tile: 1.71 against 2.02 ms at B = 64, L = 16384, D = 2048, unless 56 channels save a wave)
    if (ctas(64) >= 148 || ctas(56) >= 148) {
      tile = waves_cost(56) * (norm ? 1.0 : 1.15) < waves_cost(64) ? 7 : 8;
      // More than one wave: whole waves waste the SMs that the last one leaves idle.  The segmented
      // form takes ceil(items x runs / SMs) / runs waves of 64-channel steps instead (a step of the
      // 56- and of the 64-channel tile take about the same time); it pays when that saves 4 %.
      if (can_pipe && a_in.B >= 4 && ctas(64) > 148) {
        const int nsteps = (a_in.L + kStep - 1) / kStep;
        const double plain = (double)((ctas(tile == 7 ? 56 : 64) + 147) / 148);
        int best = 0;
        double best_cost = plain * 0.96;
        for (int n_seg = 2; n_seg <= 8; n_seg *= 2) {
          if (nsteps % n_seg != 0 || nsteps / n_seg < 64) continue;
          const double cost = (double)((ctas(64) * n_seg + 147) / 148) / n_seg * 1.02;
          if (cost < best_cost) {
            best_cost = cost;
            best = n_seg;
          }
        }
        if (best != 0) {
          if (mma_cl_segmented(dtype, x, y, xsb, xsl, ysb, ysl, norm, a_in, best, s)) return true;
        }
      }
    }
    else if (can_pipe && (ctas(16) <= 148 || a_in.B < 4))
      // too few strips for the SMs: four groups of warps per 16-channel strip set, pipelined along the
      // sequence (B = 8, L = 32768, D = 2048: 1.21 -> 1.05 ms; B = 16, L = 4096, D = 1024: 0.168 -> 0.143 ms;
      // the EMA alone on that shape: 0.153 -> 0.102 ms)
      tile = 224;
    else if (norm) tile = 22;  // 16 channels, two warps per column: twice the strips, half as long a step
    else tile = ctas(32) >= 111 ? 4 : 2;
  }
  // The tile code as the forms allow it; everything narrower than 56 channels (and the complex forms, which
  // always run the 16-channel tile) is launched from mma_cl_narrow.cu.
  if (masked || want_xn) tile = (tile == 7 || tile == 8) ? 7 : 22;
  else if (!ema && (tile == 2 || tile == 4)) tile = 22;
  if (a_in.cplx || !(tile == 7 || tile == 8 || tile == 71))
    return mma_cl_narrow(tile, dtype, x, y, xn, xsb, xsl, ysb, ysl, norm, a_in, s);
  if (masked) {  // 56-channel tile
    if (!norm)  // the EMA alone
      return a_in.silu ? launch_variant<false, 7, true, 1, false, true, false, 1, true>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s)
                       : launch_variant<false, 7, false, 1, false, true, false, 1, true>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s);
#define MEGA_MASKED(SILU, XN, EMA) \
  launch_variant<true, 7, SILU, 1, XN, EMA, false, 1, true>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s, xn, ysb, ysl)
    if (!ema) return MEGA_MASKED(false, false, false);
    if (want_xn) return a_in.silu ? MEGA_MASKED(true, true, true) : MEGA_MASKED(false, true, true);
    return a_in.silu ? MEGA_MASKED(true, false, true) : MEGA_MASKED(false, false, true);
#undef MEGA_MASKED
  }
  if (!ema) {
    // more than one wave of wide tiles: the segmented form, as for the fused pair
    if (a_in.B >= 4 && ctas(64) > 148 && g_options[OPT_MMA_TILE].load() == 0) {
      const int nsteps = (a_in.L + kStep - 1) / kStep;
      const double plain = (double)((ctas(tile == 7 ? 56 : 64) + 147) / 148);
      int best = 0;
      double best_cost = plain * 0.96;
      for (int n_seg = 2; n_seg <= 8; n_seg *= 2) {
        if (nsteps % n_seg != 0 || nsteps / n_seg < 64) continue;
        const double cost = (double)((ctas(64) * n_seg + 147) / 148) / n_seg * 1.02;
        if (cost < best_cost) {
          best_cost = cost;
          best = n_seg;
        }
      }
      if (best != 0 && mma_cl_segmented(dtype, x, y, xsb, xsl, ysb, ysl, true, a_in, best, s)) return true;
    }
    return tile == 7 ? launch_variant<true, 7, false, 1, false, false>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s)
                     : launch_variant<true, 8, false, 1, false, false>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s);
  }
  if (want_xn)  // 56-channel tiles (the 64-channel tile has no room for the two extra buffers)
    return a_in.silu ? launch_variant<true, 7, true, 1, true>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s, xn, ysb, ysl)
                     : launch_variant<true, 7, false, 1, true>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s, xn, ysb, ysl);
#define MEGA_MMA_VARIANT(NORM, SILU)                                                           \
  (tile == 71 ? launch_variant<NORM, 7, SILU, 1, false, true, false, 1, false, true>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s) \
   : tile == 7 ? launch_variant<NORM, 7, SILU>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s)        \
               : launch_variant<NORM, 8, SILU>(dtype, x, y, xsb, xsl, ysb, ysl, a_in, s))
  if (norm) return a_in.silu ? MEGA_MMA_VARIANT(true, true) : MEGA_MMA_VARIANT(true, false);
  return a_in.silu ? MEGA_MMA_VARIANT(false, true) : MEGA_MMA_VARIANT(false, false);
#undef MEGA_MMA_VARIANT
}

cudaError_t mma_cl_read_device_error(int* v, bool reset) {
  int v2 = 0;
  cudaError_t e = read_device_error(v, reset);
  if (e == cudaSuccess) e = mma_cl_seg_read_device_error(&v2, reset);
  if (e == cudaSuccess && *v == 0) *v = v2;
  if (e == cudaSuccess) e = tmem_ema_read_device_error(&v2, reset);
  if (e == cudaSuccess && *v == 0) *v = v2;
  if (e == cudaSuccess) e = mma_cl_narrow_read_device_error(&v2, reset);
  if (e == cudaSuccess && *v == 0) *v = v2;
  return e;
}

}  // namespace mega
