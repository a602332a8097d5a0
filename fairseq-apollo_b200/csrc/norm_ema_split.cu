// TimestepNorm -> causal EMA in forms that are parallel over time (norm_ema_split.cuh).
//
// The fused kernels move every element once, but a sequence is one chain of steps to them: with few sequences and
// channels they leave the SMs idle.  Two ways fill the SMs whatever the shape: the scan (scan_ema.cu), whose walks
// normalise their inputs as they read them, and, for bf16, TimestepNorm by itself (scan_norm.cu) followed by the
// tensor-core kernel alone, which runs in half the time of the fused one, or by the products of chunks (chunk_ema.cu; in bf16
// 14 x 3140 x 712 with the second output 250 us as a chain, 154 so); the normalised activations then go to their own output, or
// through y in place.
#include <cmath>

#include "chunk_ema.cuh"
#include "common.cuh"
#include "norm_ema_split.cuh"
#include "scan_cluster.cuh"
#include "scan_ema.cuh"
#include "scan_norm.cuh"
#include "scratch.cuh"
#include "tmem_ema.cuh"
#include "walk.cuh"

namespace mega {

namespace {

// Times in us from a grid of shapes on one B200 (L in positions, n in elements): a chain costs so much per position
// until the channels fill the device, then so much per element.
double longer(double chain_ns, double per_us, double L, double n) {
  const double a = L * chain_ns * 1e-3, b = n / per_us;
  return a > b ? a : b;
}

bool mma_takes(int dtype, const StreamArgs& a, bool want_xn) {
  const bool pipes = !want_xn && !a.cplx && a.mask == nullptr;   // forms pipelined along the sequence: any batch
  return dtype == MEGA_BF16 && g_options[OPT_DISABLE_MMA].load() == 0 && !(a.mask && a.cplx) && (a.B >= 4 || pipes) &&
         !(a.cplx && a.h_out && a.L % 32 != 0);   // (it cannot stop a state in mid-step; a real layer's head still runs there)
}

// (a part for the launch and, on the tensor-core kernel with complex poles, for its coefficients; long chains of the forms with
// a second output or a mask fall behind the short ones' rate.  With real poles mma_cl_try has a faster form since (tmem_ema.cu), whose
// roundings are the same: these times of the chain are left to say which calls round their operands to bf16, the others' results stay)
double fused_chain_us(int dtype, const StreamArgs& a, bool want_xn) {
  const double L = a.L, n = (double)a.B * a.D * a.L;
  if (mma_takes(dtype, a, want_xn)) {
    // (both a mask and the second output: 11 x 1894 x 464 153 us, 6 x 4999 x 2048 387, 16 x 4096 x 1024 257)
    if (a.mask && want_xn) return 15.0 + longer(65.0, 290e3, L, n);
    // (complex: 34 x 185 x 480 with the second output 76 us, 13 x 319 x 320 76, 9 x 2831 x 136 with it 205)
    const double fixed = a.cplx ? 68.0 : want_xn ? 15.0 : a.mask ? 13.0 : 11.0;
    const double chain = a.cplx ? (want_xn ? 46.0 : 36.0) : want_xn ? 44.0 : a.mask ? 42.0 : 30.0;
    const double rate = a.cplx ? (want_xn ? 300e3 : 480e3) : want_xn ? 500e3 : a.mask ? 520e3 : 600e3;
    const double far = L * 1e-3 * (a.cplx ? (want_xn ? 75.0 : 62.0) : want_xn || a.mask ? 50.0 : 34.0);
    const double near = fixed + longer(chain, rate, L, n);
    // (complex, once not every tile of 16 channels and 8 sequences has an SM: 26 x 443 x 1464 with the second output 217 us,
    // 9 x 3282 x 1944 279)
    const double tiles = ((a.D + 15) / 16) * (double)((a.B + 7) / 8);
    const double crowd = a.cplx && tiles > 148.0 ? 66.0 + L * 1e-3 * (tiles > 300.0 ? 0.8 * tiles : want_xn ? 90.0 : 65.0) : 0.0;
    return fmax(near, fmax(far, crowd));
  }
  // The streamed chain: ns a position by the blocks (128 channels of a sequence) that share an SM, from 310 shapes of 36 to 885
  // blocks and 64 to 3000 positions, to a tenth up to two blocks: 17 x 190 x 1024 fp32 27 us, 5 x 139 x 2000 fp16 with a state and
  // the second output 24, 28 x 1486 x 488 fp32 with the second output 190; complex 41 x 335 x 128 64, 24 x 1213 x 976 301.
  const double blocks = (double)a.B * ((a.D + 127) / 128) / 148.0, per = blocks <= 1.0 ? 1.0 : fmax(2.0, ceil(blocks - 0.2));
  double ns = a.cplx ? (per < 2 ? 175.0 : per < 3 ? 250.0 : per < 4 ? 340.0 : 130.0 * per)
                     : (per < 2 ? 125.0 : per < 3 ? 150.0 : per < 4 ? 195.0 : 78.0 * per);
  if (a.h_in || a.h_out) ns *= 1.09;
  if (a.mask) ns *= 1.03;
  if (dtype == MEGA_F32 && want_xn && blocks > 1.5) ns *= 1.4;
  return 4.0 * per + L * ns * 1e-3;
}

// The EMA of the normalised activations where TimestepNorm has left them.
ScanArgs behind_norm(const ScanArgs& ea, const void* mid) {
  ScanArgs a = ea;
  a.x = mid;
  a.xsb = ea.ysb;
  a.xsl = ea.ysl;
  a.xn = nullptr;
  a.prev_count = nullptr;
  return a;
}
// TimestepNorm, then the tensor-core kernel alone: where the fused call would run on it too (both round the normalised
// activations to bf16), without a mask (that form gains little) and at lengths that it can stop at
double mma_us(int dtype, const StreamArgs& a, bool want_xn) {
  if (!mma_takes(dtype, a, want_xn) || a.mask || (a.h_out && a.L % 32 != 0)) return 1e30;
  const double L = a.L, n = (double)a.B * a.D * a.L;
  return 10.0 + n / 700e3 + (a.cplx ? 54.0 + longer(28.0, 600e3, L, n) : longer(22.0, 1300e3, L, n));
}

// (in one launch, or as the scan's five)
double scan_us(int dtype, const ScanArgs& ea, bool want_xn) {
  const double n = (double)ea.B * ea.D * ea.L, one = scan_cluster_us(dtype, ea);
  // (padding masks: 33 x 1282 x 456 fp32 199 us, 16 x 4096 x 1024 fp16 475, with the second output 5 x 4079 x 536 201, complex
  // 1 x 9084 x 728 152)
  const double masked = !ea.mask ? 1.0 : ea.cplx ? 1.15 : want_xn ? 1.45 : dtype == MEGA_F32 ? 1.2 : 1.1;
  // (real: 10 x 985 x 1200 fp16 87 us, 60 x 2033 x 344 fp32 with the second output 268)
  return one < 1e29 ? one : (ea.cplx ? 45.0 : 38.0) + masked * n / (ea.cplx ? (want_xn ? 78e3 : 88e3) : (want_xn ? 160e3 : 165e3));
}

// TimestepNorm in fp32, then the products of chunks (chunk_ema.cu): the normalised activations lie in scratch memory, for fp32
// calls in xn or, in place, in y.  (moments and normalised activations of 6 x 4999 x 2048 bf16: 125 us)
constexpr double kWideMost = 62e6;   // elements of scratch memory: what the pool keeps between calls (scratch.cuh)
double chunk_us(int dtype, const ScanArgs& ea) {
  ScanArgs a = ea;
  a.prev_count = nullptr;
  a.mask = nullptr;
  const double n = (double)a.B * a.D * a.L;
  if (dtype != MEGA_F32 && n > kWideMost) return 1e30;
  return 12.0 + n / (dtype == MEGA_F32 ? 480e3 : 540e3) + chunk_ema_fwd_us(MEGA_F32, a);
}
bool norm_chunk_try(int dtype, const ScanArgs& ea, long long xsd, long long ysd, cudaStream_t s) {
  if (!rows_ok(dtype, ea.y, ea.ysb, ea.ysl, ysd) || (ea.xn && !rows_ok(dtype, ea.xn, ea.ysb, ea.ysl, ysd))) return false;
  ScanNormArgs na{};
  na.x = ea.x; na.B = ea.B; na.D = ea.D; na.L = ea.L;
  na.xsb = ea.xsb; na.xsl = ea.xsl; na.ysb = ea.ysb; na.ysl = ea.ysl;
  na.prev_count = ea.prev_count; na.prev_mean = ea.prev_mean; na.prev_var = ea.prev_var; na.gamma = ea.gamma; na.beta = ea.beta;
  na.eps = ea.eps; na.count_out = ea.count_out; na.mean_out = ea.mean_out; na.var_out = ea.var_out; na.mask = ea.mask;
  ScanArgs a = ea;
  a.prev_count = nullptr;
  a.xn = nullptr;
  a.mask = nullptr;   // (the norm has zeroed what is padded)
  if (dtype == MEGA_F32) {
    na.y = ea.xn ? ea.xn : ea.y;
    a.x = na.y;
    a.xsb = ea.ysb;
    a.xsl = ea.ysl;
    return scan_norm_fwd_try(dtype, na, xsd, ysd, s) && chunk_ema_fwd_try(dtype, dtype, a, 1, ysd, s, true);
  }
  const size_t n = (size_t)ea.B * ea.L * ea.D;
  Scratch sc(Scratch::padded(n * 4), s);
  if (!sc) return false;
  na.wide = sc.take<float>(n);
  na.y = ea.xn;
  a.x = na.wide;
  a.xsb = (long long)ea.L * ea.D;
  a.xsl = ea.D;
  return scan_norm_fwd_try(dtype, na, xsd, ysd, s) && chunk_ema_fwd_try(MEGA_F32, dtype, a, 1, ysd, s, true);
}

}  // namespace

bool norm_ema_split_try(int dtype, const void* x, void* y, void* xn, long long xsb, long long xsl, long long xsd,
                        long long ysb, long long ysl, long long ysd, const StreamArgs& a, cudaStream_t s) {
  const int asked = g_options[OPT_SPLIT].load(), forced = asked == 4 ? 0 : asked;   // (4 is about TimestepNorm by itself)
  if (forced == 1 || g_options[OPT_DISABLE_STREAM].load() != 0 || g_options[OPT_DISABLE_MMA].load() != 0 ||
      g_options[OPT_MMA_TILE].load() != 0)   // (a kernel asked for by name)
    return false;
  if (x == y || xn == y || xn == x || a.N < 1 || a.N > 16 || a.count_offset != 0) return false;
  ScanArgs ea{};
  ea.x = x; ea.y = y; ea.xn = xn; ea.B = a.B; ea.D = a.D; ea.L = a.L; ea.N = a.N;
  ea.xsb = xsb; ea.xsl = xsl; ea.ysb = ysb; ea.ysl = ysl;
  ea.p = a.p; ea.q = a.q; ea.g = a.g; ea.omega = a.omega; ea.mask = a.mask; ea.h_in = a.h_in; ea.h_out = a.h_out;
  ea.cplx = a.cplx; ea.silu = a.silu;
  ea.prev_count = a.prev_count; ea.prev_mean = a.prev_mean; ea.prev_var = a.prev_var; ea.gamma = a.gamma; ea.beta = a.beta;
  ea.eps = a.eps; ea.count_out = a.count_out; ea.mean_out = a.mean_out; ea.var_out = a.var_out;
  // (the margins: more launches on a host that is not ahead of the device; the fixed parts of the forms in several launches hold
  // some 10 us for it too; the models are good to a tenth: of 900 shapes 6 take a form more than 3 % slower than
  // the one they took before there were products of chunks)
  // (a prompt that comes in chunks keeps to the tensor-core kernel, and its rounding, unless much is gained)
  const bool prompt = dtype == MEGA_BF16 && a.h_out && !a.mask && !a.cplx && mma_takes(dtype, a, xn != nullptr);
  const double fused = fused_chain_us(dtype, a, xn != nullptr), scan = scan_us(dtype, ea, xn != nullptr) + (prompt ? 25.0 : 0.0),
               chain = mma_us(dtype, a, xn != nullptr) + 25.0;
  // The products of chunks behind TimestepNorm in bf16: for calls that would run on the tensor-core kernel in one of its two ways,
  // whose roundings these are too (complex 4 x 4096 x 1024 263 us fused, 103 so; real 142 and 94).
  const bool rounds = chain < 1e29 && (scan > 0.9 * fused || chain < scan);
  const double chunks = rounds ? 15.0 + (double)a.B * a.D * a.L / 700e3 + chunk_ema_fwd_us(dtype, behind_norm(ea, ea.y)) : 1e30;
  const double mma = chunks < chain ? chunks : chain;
  // (of what rounds to bf16 the fused kernel with accumulators in tensor memory, where it is the faster one: 8 x 8192 x 1024 with the
  // second output and SiLU 253 us as norm and products of chunks, 161 so).  It writes 16-byte pieces, as does what follows on
  // TimestepNorm by itself; for other outputs there is the scan (8 x 8192 x 1024 370 us; a thread per row 2046).
  // Statistics updated in place: TimestepNorm by itself may not overwrite them before the EMA behind it has been taken, so these calls
  // are the scan's too, in fp32 throughout.
  ScanNormArgs na{};
  na.x = x; na.y = xn ? xn : y; na.B = a.B; na.D = a.D; na.L = a.L;
  na.xsb = xsb; na.xsl = xsl; na.ysb = ysb; na.ysl = ysl;
  na.prev_count = a.prev_count; na.prev_mean = a.prev_mean; na.prev_var = a.prev_var; na.gamma = a.gamma;
  na.beta = a.beta; na.eps = a.eps; na.count_out = a.count_out; na.mean_out = a.mean_out; na.var_out = a.var_out;
  const bool parts = rows_ok(dtype, y, ysb, ysl, ysd) && (!xn || rows_ok(dtype, xn, ysb, ysl, ysd)) && !stats_in_place(na);
  const bool whole = parts && !a.cplx && mma_takes(dtype, a, xn != nullptr) && tmem_ema_us(a, true, xn != nullptr) < 0.95 * mma;
  if (forced == 0) {   // (what stands in mean_out and the like once the norm has run is what the forms below write too)
    const double chunk = chunk_us(dtype, ea), by_scan = scan - (prompt ? 25.0 : 0.0);
    if ((chunk < 0.88 * (by_scan < mma ? by_scan : mma) && chunk < 0.88 * fused) || (chunk < 1e29 && g_options[OPT_CHUNK].load() == 2))
      if (norm_chunk_try(dtype, ea, xsd, ysd, s)) return true;
  }
  // (a scan in one launch is worth its estimate where that is a launch's fixed part: 28 x 66 x 88 fp32 9.2 us, as a chain 11.4)
  const double n = (double)a.B * a.D * a.L, margin = n < 4e5 && scan < 45.0 ? 1.0 : 0.9;
  if (forced == 0 && (scan < mma ? scan : mma) > margin * fused) return false;
  if (forced == 0 && mma < scan && whole) return false;
  if (mma < scan && forced != 3 && parts) {
    void* mid = xn ? xn : y;
    const bool normed = (xsd == 1 && ysd == 1 && tmem_norm_us(a) < 0.9 * scan_norm_us(na) && tmem_norm_try(dtype, x, mid, xsb, xsl, ysb, ysl, a, s)) ||
                        scan_norm_fwd_try(dtype, na, xsd, ysd, s);
    if (normed &&
        ((chunks < chain && chunk_ema_fwd_try(dtype, dtype, behind_norm(ea, mid), 1, ysd, s, true)) ||
         mma_cl_try(dtype, mid, y, nullptr, ysb, ysl, ysd, ysb, ysl, ysd, false, a, s)))
      return true;   // (were the second one refused, the next form starts from x again)
  }
  return scan_ema_fwd_try(dtype, ea, xsd, ysd, s);
}

}  // namespace mega
