// The causal EMA and its backward as matrix products of chunks, parallel over time: real or complex poles, channels contiguous.
//
// With chunks of 16 positions, h the poles' states and everything below a matrix of the channel,
//   states   h' = q^16 h + V x         V (16 x poles): q^(15-k)
//   outputs  y  = T x + G h            T (16 x 16): the taps, omega on its diagonal; G (poles x 16): c q^(j+1)
// Backward: dx is the layer itself run over dy in reversed time, its states h the adjoint.  Of the parameters' gradients the sums
// over time sum_t dy_t (state of x)_t are, by adjointness, sum_t x_t h_t, and the same with the derivative s = dh/dq in h's place
// (s' = q^16 s + 16 q^15 h + U dy, U the derivative of V).  With l = sum_j q^j x_j and w = sum_j j q^(j-1) x_j of a chunk (V and
// U against x in the other order) and R_k the correlation of x and dy at lag k within chunks,
//   sum_t x_t h_t = q A1 + sum_k q^k R_k,               A1 = sum over chunks of l h
//   sum_t x_t s_t = q A2 + A1 + sum_k k q^(k-1) R_k,    A2 = sum over chunks of l s + w h.
// So nothing is computed per position and pole: 16 + 16 + 16 multiply-adds per element forward (real), 48 + 16 more backward, all
// on the tensor pipe.
//
// fp32 on the bf16 tensor pipe: matrices, states and fp32 inputs go in as three bf16 parts, of whose products all but
// those below 2^-24 are taken (split_mma.cuh); a bf16 input is one part, an fp16 one two.
//
// A sequence is cut into segments that run at the same time: (1) every segment but the last folds its inputs into a state
// of its own, (2) a small launch carries the states over the segments, (3) outputs, and the sums of the parameters'
// gradients.  A block takes eight segments of 16 (8) adjacent channels in tiles of 64 or 128 positions.  The tile comes with
// asynchronous copies, is turned into rows along time as bf16 parts, and then a warp owns a channel: the rows of
// its products are two consecutive chunks of the eight segments, so that states stay in a thread; matrices live in registers
// (complex: some in shared memory) for the whole segment.  Two buffers let half of the warps turn tiles while the others
// multiply.
//
// bf16 calls that would otherwise go to the tensor-core kernel take the leading parts alone, as that one does (lean_call).
// What bounds it (backward of 16 x 4096 x 1024 bf16, 227 us for both of its walks in one): the tensor pipe is busy 47 % of the
// time, issue slots 45 %, shared memory 32 %, DRAM 21 %; 16 warps per SM at 128 registers do not hide the chain of products.
// Complex outputs of fp32 inputs (6 x 4999 x 2048, 344 us; 374 under the profiler before half of the warps turned while others
// multiplied): 46, 47, 35 and 12 %.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "chunk_ema.cuh"
#include "common.cuh"
#include "scan_cluster.cuh"
#include "scratch.cuh"
#include "split_mma.cuh"
#include "stream_cl.cuh"
#include "tma.cuh"
#include "tmem_ema.cuh"
#include "walk.cuh"

namespace mega {

namespace {

// local states; with their derivatives; outputs; sums of the parameters' gradients; those and the outputs (the input's gradient)
enum Mode { kLocal, kLocalSens, kEmit, kGrad, kBoth };

struct ChunkArgs {
  ScanArgs a;
  const void* in;           // what is walked, and its strides
  long long isb, isl;
  const void* beside;       // with the sums: what it is correlated with
  long long bsb, bsl;
  int T, S;                 // steps of a segment (a multiple of 64), segments of a sequence
  int walked;               // of them, those that this launch takes
  int rev;                  // time runs backwards
  int parts;                // values per (sequence, segment) in the carry array
  float* carry;             // [B][S][parts][D][16]: what a segment starts from (of segment 0: a state that comes in, or unused)
  const unsigned char* frag;   // [D][blocks] of kBlockBytes
  int blocks;
  const float* pow;         // [D][6][16]: q^16 (re, im), 16 q^15 (re, im), what rounding took from q^16 relative to it (re, im)
};

template <typename T>
constexpr int kPartsOf = sizeof(T) == 4 ? 3 : std::is_same<T, __half>::value ? 2 : 1;

// blocks of a channel: V, [U], T (two), G
template <bool kC>
struct Blocks {
  static constexpr int v = kC ? 4 : 2, g = kC ? 4 : 2;
};

template <typename In, typename Out, bool kC, int kMode, bool kMask, bool kLean = false>
struct Form {
  static constexpr int kP = kPartsOf<In>;
  static_assert(kMode != kBoth || (kP == 1 && !kC), "the sums and the outputs in one: what registers and shared memory hold");
  static_assert(kMode != kGrad || kP > 1 || kC, "real one-part sums come with the outputs");
  // positions of a tile (what shared memory holds), and bytes of a row: eight rows hit different banks
  static constexpr int kTile = kMode < kGrad && (kP == 1 || (kP == 2 && !kC)) ? 128 : 64;
  static constexpr int kRow = 2 * kTile + 16;
  static constexpr int kCh = kMode == kGrad && kP == 3 ? 8 : 16;   // channels of a block, and its warps
  static constexpr int kThreads = 32 * kCh;
  static constexpr int kIns = kMode >= kGrad ? 2 : 1;
  static constexpr int kPlane = kCh * 8 * kRow;                    // bytes of one part of a tile
  static constexpr int kBufs = (kMode == kGrad && (kP == 3 || (kP == 2 && kC))) || (kMode == kLocalSens && kP == 3 && kC) ? 1 : 2;
  static constexpr int kV = Blocks<kC>::v;
  static constexpr int kRegs = kLean ? (kMode == kEmit ? kV + 2 + Blocks<kC>::g : kV) : kMode == kBoth ? 2 + Blocks<kC>::g : kMode == kEmit ? (kC ? Blocks<kC>::g : 2 * kV + 2) : kMode == kLocal ? kV : kC ? 0 : 2 * kV;
  static constexpr int kAll = kMode == kBoth ? 2 * kV + 2 + Blocks<kC>::g : kMode == kEmit ? kV + 2 + Blocks<kC>::g : kMode == kLocal ? kV : 2 * kV;
  static constexpr int kShared = kAll - kRegs;                     // matrices in shared memory (the first ones)
  static constexpr int kE = 16 / (int)sizeof(In), kPos = kTile / (4 * kE);  // channels of a 16-byte piece; positions of a thread
  static constexpr int kSlot = kIns * kPos * kThreads * 16;        // bytes of a tile as it arrives
  static constexpr int stage = kBufs * kIns * kP * kPlane;
  static constexpr int kRests = kLean ? 0 : kCh * 16 * (kC ? 8 : 4);  // of q^16
  static constexpr int fixed = stage + kShared * kCh * kBlockBytes + (kMask ? 512 : 0) + kRests;
  static constexpr int kSlots = fixed + 2 * kSlot <= (kCh == 8 ? 112 : 226) * 1024 ? 2 : 1;
  static constexpr int mats = stage + kSlots * kSlot;
  static constexpr int bits = mats + kShared * kCh * kBlockBytes;  // padded positions: a word for 32 of them, two sets
  static constexpr int kBits = 8 * kTile / 32;                     // words of a set
  static constexpr int rests = bits + (kMask ? 2 * kBits * 4 : 0);
  static constexpr int total = rests + kRests;
  static constexpr int kPerSm = kCh == 8 && total <= 112 * 1024 ? 2 : 1;
  static_assert(total <= 227 * 1024, "a block's shared memory");
};

// byte offset of (channel, segment, 16-position block): blocks of a row in an order that differs between the channels a
// warp writes at once
template <int kRow>
__device__ __forceinline__ int row_at(int ch, int seg, int blk) { return (ch * 8 + seg) * kRow + ((blk ^ ((ch >> 2) & 3)) << 5); }

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ void ldmatrix(uint32_t (&f)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldmatrix_t(uint32_t (&f)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(at) : "memory");
}

// the lower bf16 of a pair (as a shift it would become a multiplication, which costs more issue slots)
__device__ __forceinline__ float lower(uint32_t p) { return __uint_as_float(prmt(p, 0u, 0x1044)); }
// scalar form of split3: next to other fp32 work a packed operation costs what it saves
__device__ __forceinline__ void split(float lo, float hi, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = bf16_pair(lo, hi);
  lo -= lower(p0);
  hi -= __uint_as_float(p0 & 0xffff0000u);
  p1 = bf16_pair(lo, hi);
  p2 = bf16_pair(lo - lower(p1), hi - __uint_as_float(p1 & 0xffff0000u));
}
// silu without a division's slow path (inside the walk that cost half of its time: 607 us where this takes 340, 6 x 4999 x 2048
// complex): the reciprocal to one unit, for fp32 outputs to a half by a Newton step (the clamp keeps that from an infinity)
template <typename T>
__device__ __forceinline__ float silu_of(float v) {
  const float d = sizeof(T) == 4 ? fminf(1.f + __expf(-v), 1e38f) : 1.f + __expf(-v);
  float r = rcp_approx(d);
  if (sizeof(T) == 4) r = fmaf(r, fmaf(-d, r, 1.f), r);
  return v * r;
}
// Product j, smallest first, of those of a (kP parts) with a block: the leading one is the last.  (Callers go through the
// products of several independent sums in turn, so that none waits for the one before it.)
template <int kP>
constexpr int kTerms = kP == 1 ? 3 : kP == 2 ? 5 : 6;
template <int kP>
__device__ __forceinline__ void term(int j, bool onto, float (&d)[4], const uint32_t (&a)[kP][4], const Frag& b) {
  constexpr int kOf[3][6][2] = {{{0, 2}, {0, 1}, {0, 0}}, {{0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}}, {{0, 2}, {2, 0}, {1, 1}, {1, 0}, {0, 1}, {0, 0}}};
  const int p = kOf[kP - 1][j][0], q = kOf[kP - 1][j][1];
  const uint32_t b0 = q == 0 ? b.u.x : q == 1 ? b.u.z : b.v.x, b1 = q == 0 ? b.u.y : q == 1 ? b.u.w : b.v.y;
  if (onto) mma(d, a[p], b0, b1);
  else mma0(d, a[p], b0, b1);
}

// A thread's share of the tiles: kPos positions of kE channels of one segment.
template <typename E, int kCh, int kTile>
struct Share {
  static constexpr int kRow = 2 * kTile + 16;
  static constexpr int kE = 16 / (int)sizeof(E), kPos = kTile / (4 * kE), kCols = kCh / kE, kGroups = kTile / kPos;
  int left;         // positions of the segment from the share's next piece on (<= 0: none)
  int at[2];        // where its channels' rows take them: the first four, the others
  long long step;   // bytes from a position to the next
  char* next;
  __device__ __forceinline__ Share(const ChunkArgs& s, int id, const void* base, long long sb, long long sl, bool back) {
    const int col = id % kCols, pg = id / kCols % kGroups, seg = id / (kCols * kGroups);
    const int row = blockIdx.y * 8 + seg, c = blockIdx.x * kCh + col * kE;
    const int b = row / s.walked, first = (row - b * s.walked) * s.T;
    const bool ok = b < s.a.B && c < s.a.D;
    const int t = first + pg * kPos, pos = pg * kPos, in = back ? 16 - kPos - (pos & 15) : pos & 15;
    left = ok ? min(s.T, s.a.L - first) - pos : 0;
    step = (s.rev ? -sl : sl) * (long long)sizeof(E);
    next = (char*)base + (ok ? b * sb + (s.rev ? s.a.L - 1 - t : t) * sl + c : 0) * (long long)sizeof(E);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      at[i] = row_at<kRow>(col * kE + (kE == 8 ? 4 * i : 0), seg, pos >> 4) + in * 2 - (kE == 8 ? 4 * i * 8 * kRow : 0);
  }
  __device__ __forceinline__ int row(int j) const { return at[j >> 2] + j * 8 * kRow; }   // of channel j
  __device__ __forceinline__ void advance() {
    left -= kTile;
    next += kTile * step;
  }
  // its pieces of a tile on their way (zeros where the segment has ended: nothing is read there)
  __device__ __forceinline__ void fetch(uint32_t slot) {
    const char* from = next;
#pragma unroll
    for (int k = 0; k < kPos; ++k, from += step)
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(slot + k * 32 * kCh * 16), "l"(from), "r"(k < left ? 16 : 0)
                   : "memory");
    advance();
  }
};

// kPos 16-bit values of a row, kPos / 2 words
template <int kPos>
struct alignas(2 * kPos) Words {
  uint32_t v[kPos / 2];
};

// A thread's pieces into the rows of the buffer; kBack: the positions of a 16-position block in reversed order.
template <typename E, int kCh, int kTile, int kP, int kPlane, bool kBack>
__device__ __forceinline__ void turn(const Share<E, kCh, kTile>& sh, const unsigned char* slot, unsigned char* buf) {
  constexpr int kPos = Share<E, kCh, kTile>::kPos, kE = Share<E, kCh, kTile>::kE;
  uint32_t w[kPos][4];
#pragma unroll
  for (int k = 0; k < kPos; ++k) {
    const uint4 v = *reinterpret_cast<const uint4*>(slot + (kBack ? kPos - 1 - k : k) * 32 * kCh * 16);
    w[k][0] = v.x; w[k][1] = v.y; w[k][2] = v.z; w[k][3] = v.w;
  }
#pragma unroll
  for (int j = 0; j < kE; ++j) {
    Words<kPos> part[kP];
#pragma unroll
    for (int i = 0; i < kPos / 2; ++i) {
      if constexpr (sizeof(E) == 4) {
        split(__uint_as_float(w[2 * i][j & 3]), __uint_as_float(w[2 * i + 1][j & 3]), part[0].v[i], part[1 % kP].v[i], part[2 % kP].v[i]);
      } else {
        uint32_t v = prmt(w[2 * i][j >> 1], w[2 * i + 1][j >> 1], j & 1 ? 0x7632 : 0x5410);
        if constexpr (kP == 2) {   // fp16: its leading eight bits, and the rest
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
          v = bf16_pair(f.x, f.y);
          part[1].v[i] = bf16_pair(f.x - __uint_as_float(v << 16), f.y - __uint_as_float(v & 0xffff0000u));
        }
        part[0].v[i] = v;
      }
    }
#pragma unroll
    for (int p = 0; p < kP; ++p) *reinterpret_cast<Words<kPos>*>(buf + sh.row(j) + p * kPlane) = part[p];
  }
}

// A thread's share of the outputs, from the rows of the buffer (fp32: upper and lower halves in the first two parts).
template <typename E, int kCh, int kTile, int kPlane>
__device__ __forceinline__ void put(Share<E, kCh, kTile>& sh, const unsigned char* buf) {
  constexpr int kPos = Share<E, kCh, kTile>::kPos, kE = Share<E, kCh, kTile>::kE;
  Words<kPos> hi[kE], lo[sizeof(E) == 4 ? kE : 1];
#pragma unroll
  for (int j = 0; j < kE; ++j) {
    hi[j] = *reinterpret_cast<const Words<kPos>*>(buf + sh.row(j));
    if constexpr (sizeof(E) == 4) lo[j] = *reinterpret_cast<const Words<kPos>*>(buf + sh.row(j) + kPlane);
  }
  char* to = sh.next;
#pragma unroll
  for (int k = 0; k < kPos; ++k, to += sh.step) {
    auto word = [&](int i) {
      if constexpr (sizeof(E) == 4) return prmt(lo[i].v[k >> 1], hi[i].v[k >> 1], k & 1 ? 0x7632 : 0x5410);
      else return prmt(hi[2 * i].v[k >> 1], hi[2 * i + 1].v[k >> 1], k & 1 ? 0x7632 : 0x5410);
    };
    if (k < sh.left) *reinterpret_cast<uint4*>(to) = make_uint4(word(0), word(1), word(2), word(3));
  }
  sh.advance();
}

// ---- the matrices of a channel --------------------------------------------------------------------------------
// A warp per channel; powers in double, rounded once.  sens: U behind V; outs: T and G behind those; gain: the input gain p
// is V's (states as the layer exports them) instead of G's; om: omega on T's diagonal.
struct PrepArgs {
  const float *p, *q, *g, *omega;
  int D, N, sens, outs, gain, om, blocks;
  unsigned char* frag;
  float* pow;
};
template <bool kC>
__global__ void __launch_bounds__(128) chunk_prepare_kernel(PrepArgs a) {
  __shared__ double2 table[4][17][16], weight[4][16];
  __shared__ float taps[4][16], gains[4][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = blockIdx.x * 4 + warp;
  if (d >= a.D) return;
  double2(&pw)[17][16] = table[warp];
  const int n = lane & 15;
  const size_t at = (size_t)d * a.N + n;
  const bool live = n < a.N;
  double qr = 0., qi = 0., wr = 0., wi = 0.;   // pole; output weight p g
  if (live) {
    const double p = a.p[at];
    qr = kC ? a.q[2 * at] : a.q[at];
    wr = p * (kC ? a.g[2 * at] : a.g[at]);
    if (kC) {
      qi = a.q[2 * at + 1];
      wi = p * a.g[2 * at + 1];
    }
  }
  // (what the blocks below take from here: read from memory for each of their entries it was half of the kernel's 8.4 us)
  if (lane < 16) {
    gains[warp][n] = a.gain && live ? a.p[at] : 1.f;
    weight[warp][n] = !a.gain || !live ? make_double2(wr, wi) : make_double2(kC ? a.g[2 * at] : a.g[at], kC ? a.g[2 * at + 1] : 0.f);
  }
  double vr = 1., vi = 0.;
  for (int e = 0; e <= 16; ++e) {
    if (lane < 16) pw[e][n] = make_double2(vr, vi);
    if (e < 16 && a.outs) {
      double tap = wr * vr - wi * vi;
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) tap += __shfl_xor_sync(0xffffffffu, tap, s);
      if (lane == 0) taps[warp][e] = (float)(e == 0 && a.om ? tap + a.omega[d] : tap);
    }
    const double r = vr * qr - vi * qi;
    vi = vr * qi + vi * qr;
    vr = r;
  }
  __syncwarp();
  if (lane < 16) {
    float* pc = a.pow + (size_t)d * 96 + n;
    const double2 w = pw[16][n];
    const float r = (float)w.x, i = (float)w.y;
    pc[0] = r;
    pc[16] = i;
    pc[32] = (float)(16. * pw[15][n].x);
    pc[48] = (float)(16. * pw[15][n].y);
    const double m = (double)r * r + (double)i * i;   // (w - v) / v, v = r + i I; none for poles that forget sooner than they are corrected
    const bool some = m > 0.81;
    pc[64] = some ? (float)(((w.x - r) * r + (w.y - i) * i) / m) : 0.f;
    pc[80] = some ? (float)(((w.y - i) * r - (w.x - r) * i) / m) : 0.f;
  }
  constexpr int kV = Blocks<kC>::v;
  const int g = lane >> 2, t = lane & 3;
  const int us = kV, ts = us + (a.sens ? kV : 0), gs = ts + 2;
#pragma unroll 2
  for (int blk = 0; blk < a.blocks; ++blk) {
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 2 * t + (i & 1) + 8 * (i >> 1);
      double x;
      if (blk < ts) {
        const int nt = blk < us ? blk : blk - us, pole = 8 * (nt & 1) + g, e = 15 - k;
        const bool sens = blk >= us;
        const double2 w = pw[sens ? max(e - 1, 0) : e][pole];
        x = nt < 2 ? w.x : w.y;
        if (sens) x *= e;
        x = pole >= a.N ? 0. : x * gains[warp][pole];
      } else if (blk < gs) {
        const int lag = 8 * (blk - ts) + g - k;
        x = lag >= 0 ? taps[warp][lag] : 0.f;
      } else {
        const int kt = (blk - gs) >> 1, j = 8 * ((blk - gs) & 1) + g;
        const double2 w = pw[j + 1][k], c = weight[warp][k];
        x = kt == 0 ? c.x * w.x - c.y * w.y : -(c.x * w.y + c.y * w.x);
      }
      v[i] = (float)x;
    }
    store_frag(a.frag + ((size_t)d * a.blocks + blk) * kBlockBytes, v);
  }
}

// ---- what the products cannot give -----------------------------------------------------------------------------
// An infinity, a NaN or a value that bf16 rounds to an infinity makes NaN of all products that it enters, where the recurrence
// leaves finite states and outputs, or infinite ones, as they follow.  Here it is, position by position in fp32: n positions from
// `first` on (in the order they are walked) of the row of a quad (none where n is 0), from and to the states of a lane's poles;
// each(k, y) for outputs from the first such value on.  The whole warp takes part, for `most` positions.
template <typename In, bool kC, bool kSens, int kRe, typename Each>
__device__ __forceinline__ void one_by_one(const ChunkArgs& s, int b, int d, int first, int n, int most, float (&h)[kRe][4],
                                           float (*sens)[4], Each each) {
  const ScanArgs& a = s.a;
  const int t = threadIdx.x & 3;
  const bool gain = a.h_in || a.h_out;   // (the states are the layer's own then: see chunk_prepare_kernel)
  float fr[4], fi[4], u[4], c[4], ci[4], z = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // (poles there are not: states and weights of zero)
    const int m = 8 * (i >> 1) + 2 * t + (i & 1);
    const size_t at = (size_t)d * a.N + min(m, a.N - 1);
    const float p = __ldg(a.p + at);
    fr[i] = m < a.N ? __ldg(a.q + kRe * at) : 0.f;
    fi[i] = kC && m < a.N ? __ldg(a.q + kRe * at + 1) : 0.f;
    u[i] = gain ? p : 1.f;
    c[i] = m < a.N ? (gain ? 1.f : p) * __ldg(a.g + kRe * at) : 0.f;
    ci[i] = kC && m < a.N ? (gain ? 1.f : p) * __ldg(a.g + kRe * at + 1) : 0.f;
    z = fmaf(h[0][i], 0.f, fmaf(h[kRe - 1][i], 0.f, z));
  }
  const unsigned quad = 15u << (threadIdx.x & 28);
  bool on = (__ballot_sync(0xffffffffu, z != z) & quad) != 0u;
  const float om = __ldg(a.omega + d);
  const long long step = s.rev ? -s.isl : s.isl;
  const In* x = reinterpret_cast<const In*>(s.in) + b * s.isb + (long long)(s.rev ? a.L - 1 - first : first) * s.isl + d;
  const unsigned char* pad = a.mask ? a.mask + (size_t)b * a.L + (s.rev ? a.L - 1 - first : first) : nullptr;
#pragma unroll 1
  for (int k0 = 0; k0 < most; k0 += 8) {
    float v[8];
    bool skip[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int at = k0 + k;
      v[k] = at < n ? Elem<In>::ld(x + at * step) : 0.f;
      skip[k] = pad && at < n && __ldg(pad + (s.rev ? -at : at)) != 0;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in_row = k0 + k < n;
      const float in = skip[k] && !s.rev ? 0.f : v[k];
      on = on || (bf16_pair(in, in) & 0x7f80u) == 0x7f80u;
      float out = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (!in_row || 8 * (i >> 1) + 2 * t + (i & 1) >= a.N) continue;
        float &re = h[0][i], &im = h[kRe - 1][i];
        if (kSens) {
          float &sr = sens[0][i], &si = sens[kRe - 1][i];
          const float r = kC ? fmaf(fr[i], sr, fmaf(-fi[i], si, re)) : fmaf(fr[i], sr, re);
          if (kC) si = fmaf(fr[i], si, fmaf(fi[i], sr, im));
          sr = r;
        }
        const float w = u[i] * in, r = kC ? fmaf(fr[i], re, fmaf(-fi[i], im, w)) : fmaf(fr[i], re, w);
        if (kC) im = fmaf(fr[i], im, fi[i] * re);
        re = r;
        out = fmaf(c[i], re, kC ? fmaf(-ci[i], im, out) : out);
      }
#pragma unroll
      for (int m = 1; m < 4; m <<= 1) out += __shfl_xor_sync(0xffffffffu, out, m);
      if (on && in_row) each(k0 + k, fmaf(om, v[k], skip[k] && s.rev ? 0.f : out));
    }
  }
}

// ---- the walk ----------------------------------------------------------------------------------------------
// kMask: padded positions are zero to the states (and to the correlations), omega x takes them as they are; in reversed time,
// where outputs are the input's gradient, it is the outputs at padded positions that are omega dy alone.
// kLean: leading parts alone (bf16 forward: what the tensor-core kernel that walks a sequence as one chain takes too).
template <typename In, typename Out, bool kC, int kMode, bool kMask, bool kLean>
__global__ void __launch_bounds__(Form<In, Out, kC, kMode, kMask, kLean>::kThreads, Form<In, Out, kC, kMode, kMask, kLean>::kPerSm)
    chunk_kernel(ChunkArgs s) {
  using F = Form<In, Out, kC, kMode, kMask, kLean>;
  constexpr int kFrom = kLean ? kTerms<kPartsOf<In>> - 1 : 0, kFromH = kLean ? kTerms<3> - 1 : 0;   // first products taken
  constexpr int kP = F::kP, kV = F::kV, kPlane = F::kPlane, kCh = F::kCh, kTile = F::kTile, kRow = F::kRow;
  constexpr int kRe = kC ? 2 : 1;      // real numbers of a value
  constexpr bool kSums = kMode >= kGrad, kOuts = kMode == kEmit || kMode == kBoth;
  constexpr bool kSens = kMode == kLocalSens || kSums;
  constexpr int kTs = kMode == kBoth ? 2 * kV : kV;   // T's first block
  constexpr bool kWide = kOuts && sizeof(Out) == 4;   // leading products by themselves: the tensor pipe truncates its sums
  constexpr bool kApart = kWide || (kOuts && kMask);   // omega x in fp32
  extern __shared__ __align__(16) unsigned char smem[];
  const ScanArgs& a = s.a;
  int tid;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));   // (read once: it is used in every tile)
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int d = blockIdx.x * kCh + warp, dc = min(d, a.D - 1);
  Share<In, kCh, kTile> sh(s, tid, s.in, s.isb, s.isl, false);
  Share<In, kCh, kTile> sg(s, tid, s.beside, s.bsb, s.bsl, true);
  Share<Out, kCh, kTile> so(s, tid, a.y, a.ysb, a.ysl, false);
  // the row of this lane's states (found again where it is asked for: that leaves registers to the walk), and the longest one
  struct Row {
    int b, seg, len;
    bool live;
  };
  auto own_row = [&]() -> Row {
    int y;
    asm volatile("mov.u32 %0, %%ctaid.y;" : "=r"(y));
    Row r;
    r.b = (y * 8 + g) / s.walked;
    r.seg = y * 8 + g - r.b * s.walked;
    r.live = r.b < a.B && d < a.D;
    r.len = r.b < a.B ? min(s.T, a.L - r.seg * s.T) : 0;
    return r;
  };
  const Row row0 = own_row();
  const int most = __reduce_max_sync(0xffffffffu, row0.len);
  const int steps = (most + 31) / 32, tiles = (most + kTile - 1) / kTile;

  const uint32_t stage = smem_u32(smem) + F::stage + tid * 16;
  auto issue = [&](int tile) {
    if (tile < tiles) {
      const uint32_t slot = stage + tile % F::kSlots * F::kSlot;
      sh.fetch(slot);
      if constexpr (F::kIns == 2) sg.fetch(slot + F::kSlot / 2);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i < F::kSlots; ++i) issue(i);

  // matrices and powers
  const unsigned char* mats = s.frag + (size_t)dc * s.blocks * kBlockBytes;
  const unsigned char* own = smem + F::mats + warp * F::kShared * kBlockBytes;
  const int skip = kMode == kEmit ? s.blocks - F::kAll : 0;   // (U, where the call has it, lies between V and T)
  if constexpr (F::kShared > 0) {
    unsigned char* to = smem + F::mats + warp * F::kShared * kBlockBytes;
    for (int blk = 0; blk < F::kShared; ++blk) {
      const unsigned char* from = mats + (blk >= kV ? blk + skip : blk) * kBlockBytes;
      reinterpret_cast<uint4*>(to + blk * kBlockBytes)[lane] = __ldg(reinterpret_cast<const uint4*>(from) + lane);
      reinterpret_cast<uint2*>(to + blk * kBlockBytes + 512)[lane] = __ldg(reinterpret_cast<const uint2*>(from + 512) + lane);
    }
    __syncwarp();
  }
  Frag held[F::kRegs > 0 ? F::kRegs : 1];
#pragma unroll
  for (int i = 0; i < F::kRegs; ++i) {
    const int blk = F::kShared + i, at = blk >= kV ? blk + skip : blk;
    held[i] = {__ldg(reinterpret_cast<const uint4*>(mats + at * kBlockBytes) + lane),
               __ldg(reinterpret_cast<const uint2*>(mats + at * kBlockBytes + 512) + lane)};
  }
  auto matrix = [&](int blk) -> Frag {   // (blk is a constant wherever this is called)
    if (blk < F::kShared) return load_frag(own + blk * kBlockBytes);
    return held[blk - F::kShared];
  };
  // poles of a lane: 8 i + 2 t + e
  float qr[4], qi[kC ? 4 : 1], ur[kSens ? 4 : 1], ui[kSens && kC ? 4 : 1];
  const float* pw = s.pow + (size_t)dc * 96;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = 8 * (i >> 1) + 2 * t + (i & 1);
    qr[i] = __ldg(pw + n);
    if (kC) qi[kC ? i : 0] = __ldg(pw + 16 + n);
    if (kSens) ur[kSens ? i : 0] = __ldg(pw + 32 + n);
    if (kSens && kC) ui[kSens && kC ? i : 0] = __ldg(pw + 48 + n);
  }
  const float om = kApart ? __ldg(a.omega + dc) : 0.f;
  // q^16 rounded to fp32 is off by the same 2^-25 in every chunk, which adds up to 2^-25 / (1 - q^16) of a state; so every
  // 512 positions the states get what it lacks, for the 32 chunks to come at once (a pole at 0.9999: 6e-6 from float64 without, a
  // recurrence in fp32 1.4e-6, so 4e-7; at each tile of 64 it cost a backward 5 %)
  if constexpr (!kLean) {
    if (lane < 16) {
      float* rest = reinterpret_cast<float*>(smem + F::rests) + warp * 16 * kRe;
      rest[kRe * lane] = __ldg(pw + 64 + lane);
      if (kC) rest[kRe * lane + kRe - 1] = __ldg(pw + 80 + lane);
    }
    __syncwarp();
  }

  // states that the segment starts from
  auto carry_at = [&](int b, int at, int part) { return s.carry + (((size_t)(b * s.S + at) * s.parts + part) * a.D + d) * 16 + 2 * t; };
  float h[kRe][4], sn[kSens ? kRe : 1][4];
  auto start = [&](const Row& r) {
    const int b = r.b, seg = r.seg;
#pragma unroll
    for (int c = 0; c < kRe; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        h[c][i] = 0.f;
        if (kSens) sn[kSens ? c : 0][i] = 0.f;
      }
    if (!(kOuts || kSums) || !r.live) return;
    // (the first segment's too lies with the others, of one segment where h_out is h_in: that is written while this is read)
    const bool given = kMode == kEmit && a.h_in != nullptr;
    if (seg > 0 || (given && s.carry)) {
#pragma unroll
      for (int c = 0; c < kRe; ++c)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float2 v = __ldg(reinterpret_cast<const float2*>(carry_at(b, seg, c) + 8 * k));
          h[c][2 * k] = v.x;
          h[c][2 * k + 1] = v.y;
          if (kSens) {
            const float2 u = __ldg(reinterpret_cast<const float2*>(carry_at(b, seg, kRe + c) + 8 * k));
            sn[kSens ? c : 0][2 * k] = u.x;
            sn[kSens ? c : 0][2 * k + 1] = u.y;
          }
        }
    } else if (given) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = 8 * (i >> 1) + 2 * t + (i & 1);
        const size_t at = ((size_t)b * a.D + d) * a.N + n;
        if (n < a.N) {
          h[0][i] = __ldg(a.h_in + kRe * at);
          if (kC) h[kRe - 1][i] = __ldg(a.h_in + kRe * at + 1);
        }
      }
    }
  };
  start(row0);
  // q^16 h + v of pole i
  auto next = [&](int i, float& re, float& im, float vr, float vi) {
    if (kC) {
      const float r = fmaf(qr[i], re, fmaf(-qi[kC ? i : 0], im, vr));
      im = fmaf(qi[kC ? i : 0], re, fmaf(qr[i], im, vi));
      re = r;
    } else {
      re = fmaf(qr[i], re, vr);
    }
  };
  auto settle = [&](float chunks) {
    int id;   // (read again, and the loads volatile: nothing of this is kept in a register beside the products)
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(id));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t at = smem_u32(smem) + F::rests + ((id >> 5) * 16 + 8 * (i >> 1) + 2 * (id & 3) + (i & 1)) * (4 * kRe);
      float er, ei = 0.f;
      if (kC) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(er), "=f"(ei) : "r"(at));
      else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(er) : "r"(at));
      er *= chunks;
      ei *= chunks;
      auto more = [&](float& re, float& im) {
        if (kC) {
          const float r = re;
          re = fmaf(er, r, fmaf(-ei, im, r));
          im = fmaf(er, im, fmaf(ei, r, im));
        } else {
          re = fmaf(er, re, re);
        }
      };
      more(h[0][i], h[kRe - 1][i]);
      if (kSens) more(sn[0][i], sn[kSens ? kRe - 1 : 0][i]);
    }
  };
  // kSums: A1 and A2 of the lane's poles, R of its entries
  float a1[kSums ? kRe : 1][4] = {}, a2[kSums ? kRe : 1][4] = {}, R[kSums ? 8 : 1] = {};

  float beside = 0.f;   // of omega, at padded positions
  // columns 8 k .. of the products of two inputs with the 16 chunks as the reduction (parts' products below 2^-24 left out)
  auto correlate = [](float (&r)[4], const uint32_t (&x)[kP][4], const uint32_t (&y)[kP][4], int k) {
    bool onto = false;
#pragma unroll
    for (int o = 2 * kP - 2; o >= 0; --o)
#pragma unroll
      for (int p = 0; p < kP; ++p)
        if (o <= 2 && o - p >= 0 && o - p < kP) {
          if (onto) mma(r, x[p], y[o - p][2 * k], y[o - p][2 * k + 1]);
          else mma0(r, x[p], y[o - p][2 * k], y[o - p][2 * k + 1]);
          onto = true;
        }
  };

  // eight rows of 16 bytes each: segments, their first or second chunk, lower or upper half of it
  const int blk_in = (lane >> 3) & 1;
  const uint32_t frag_row = smem_u32(smem) + (warp * 8 + (lane & 7)) * kRow + (lane >> 4) * 16;
  const int swz = ((warp >> 2) & 3) << 5;
  unsigned char* mine = smem + (warp * 8 + g) * kRow + 4 * t;   // (of the rows g and g + 8: outputs)
  const int final = kMode == kEmit && a.h_out != nullptr && row0.live && row0.seg == s.S - 1 ? (row0.len - 1) / 32 : -1;   // step whose end leaves

  // kStep steps of 32 positions at a time: their products do not wait for each other, only their states do
  constexpr int kStep = kMode == kBoth || (kC && (kMode == kGrad || kP == 3)) ? 1 : 2;   // (what registers hold; at the cap of 128, 21 of the 50 forms spill 4 to 116 bytes all the same)
  auto multiply = [&](int tile) {
    const int buf = tile % F::kBufs * F::kIns * kP * kPlane;
    const int n = min(kTile / 32, steps - kTile / 32 * tile), last = final - kTile / 32 * tile;
#pragma unroll 1
    for (int s0 = 0; s0 < n; s0 += kStep) {
      const int first = (s0 << 6) ^ swz;   // of the first step's two blocks; the other one lies 32 bytes up or down
      auto rows = [&](int st) { return frag_row + buf + ((first ^ (st << 6)) ^ (blk_in << 5)); };
      uint32_t f[kStep][kP][4];
#pragma unroll
      for (int st = 0; st < kStep; ++st)
#pragma unroll
        for (int p = 0; p < kP; ++p) ldmatrix(f[st][p], rows(st) + p * kPlane);
      // bits of the segment's row in a step; what they leave of the lane's words of a fragment
      const uint32_t* bits = kMask ? reinterpret_cast<const uint32_t*>(smem + F::bits) + (tile & 1) * F::kBits + s0 : nullptr;
      auto keep = [&](uint32_t w, int i) {   // word i: rows g and g + 8 (the step's chunks), then their upper halves
        const uint32_t two = w >> (16 * (i & 1) + 8 * (i >> 1) + 2 * t) & 3u;
        return (two & 1u ? 0u : 0xffffu) | (two & 2u ? 0u : 0xffff0000u);
      };
      uint32_t padded[kStep];
      bool some = false;
      if constexpr (kMask) {
#pragma unroll
        for (int st = 0; st < kStep; ++st) {
          padded[st] = bits[g * (kTile / 32) + st];
          some = some || padded[st] != 0u;
        }
        some = __any_sync(0xffffffffu, some);
      }
      if (kMask && some && !kSums && !(kMode == kEmit && s.rev)) {
#pragma unroll
        for (int st = 0; st < kStep; ++st)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t m = keep(padded[st], i);
#pragma unroll
            for (int p = 0; p < kP; ++p) f[st][p][i] &= m;
          }
      }
      // outputs of a step, from the states that enter its chunks
      auto emit = [&](int st, const float (&enter)[2][kRe][4], bool any_odd) {
        // entering states: the A operand of G as they stand
        uint32_t hp[kRe][3][4];
#pragma unroll
        for (int c = 0; c < kRe; ++c)
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int r = 0; r < 2; ++r)
              if (kLean) hp[c][0][2 * k + r] = bf16_pair(enter[k][c][2 * r], enter[k][c][2 * r + 1]);
              else split(enter[k][c][2 * r], enter[k][c][2 * r + 1], hp[c][0][2 * k + r], hp[c][1][2 * k + r], hp[c][2][2 * k + r]);
        // T's zeros would carry a NaN or an infinity to the positions before it: such a chunk takes its outputs from the finite
        // values ahead of the first one, and is NaN from there on, as are all later states (until one_by_one())
        int bad[2];
        if (any_odd) {
          bad[0] = bad[1] = 16;
#pragma unroll
          for (int i = 3; i >= 0; --i) {   // (rows g, g + 8, then their upper halves)
#pragma unroll
            for (int e = 1; e >= 0; --e)
              if (((f[st][0][i] >> (16 * e)) & 0x7f80u) == 0x7f80u) bad[i & 1] = 8 * (i >> 1) + 2 * t + e;
          }
#pragma unroll
          for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int m = 1; m < 4; m <<= 1) bad[r] = min(bad[r], __shfl_xor_sync(0xffffffffu, bad[r], m));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int pos = 8 * (i >> 1) + 2 * t, from = i & 1 ? bad[1] : bad[0];
            const uint32_t keep = pos + 1 < from ? ~0u : pos < from ? 0xffffu : 0u;
#pragma unroll
            for (int p = 0; p < kP; ++p) f[st][p][i] &= keep;
          }
        }
        float y[2][4];
#pragma unroll
        for (int j = kFrom; j < kTerms<kP> - 1; ++j)
#pragma unroll
          for (int k = 0; k < 2; ++k) term<kP>(j, j > kFrom, y[k], f[st], matrix(kTs + k));
#pragma unroll
        for (int j = kFromH; j < kTerms<3> - 1; ++j)
#pragma unroll
          for (int c = 0; c < kRe; ++c)
#pragma unroll
            for (int k = 0; k < 2; ++k) term<3>(j, true, y[k], hp[c], matrix(kTs + 2 + 2 * c + k));
#pragma unroll
        for (int c = 0; c <= kRe; ++c)
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const Frag m = matrix(c < kRe ? kTs + 2 + 2 * c + k : kTs + k);
            const uint32_t(&p)[4] = c < kRe ? hp[c < kRe ? c : 0][0] : f[st][0];
            if (kWide) {   // (by themselves, so that what truncates is small)
              float l[4];
              mma0(l, p, m.u.x, m.u.y);
#pragma unroll
              for (int i = 0; i < 4; ++i) y[k][i] += l[i];
            } else if (kLean && c == 0) {
              mma0(y[k], p, m.u.x, m.u.y);
            } else {
              mma(y[k], p, m.u.x, m.u.y);
            }
          }
        if (kApart) {
          uint32_t own_x[kMask ? kP : 1][4];   // as they came
          if constexpr (kMask) {
#pragma unroll
            for (int p = 0; p < kP; ++p) ldmatrix(own_x[p], rows(st) + p * kPlane);
          }
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              float x0 = 0.f, x1 = 0.f;
#pragma unroll
              for (int p = kP - 1; p >= 0; --p) {
                const uint32_t w = kMask ? own_x[kMask ? p : 0][2 * k + r] : f[st][p][2 * k + r];
                x0 += __uint_as_float(w << 16);
                x1 += __uint_as_float(w & 0xffff0000u);
              }
              if (kMask && some && s.rev) {
                const uint32_t m = keep(padded[st], 2 * k + r);
                if (!(m & 0xffffu)) y[k][2 * r] = 0.f;
                if (!(m & 0xffff0000u)) y[k][2 * r + 1] = 0.f;
              }
              y[k][2 * r] = fmaf(om, x0, y[k][2 * r]);
              y[k][2 * r + 1] = fmaf(om, x1, y[k][2 * r + 1]);
            }
        }
        if (a.silu) {
#pragma unroll
          for (int i = 0; i < 8; ++i) y[i >> 2][i & 3] = silu_of<Out>(y[i >> 2][i & 3]);
        }
        if (any_odd) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (8 * (i >> 2) + 2 * t + (i & 1) >= bad[(i >> 1) & 1] &&
                !(kMask && s.rev && !(keep(padded[st], 2 * (i >> 2) + ((i >> 1) & 1)) >> (16 * (i & 1)) & 1u)))
              y[i >> 2][i & 3] = __int_as_float(0x7fffffff);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float y0 = y[k][2 * r], y1 = y[k][2 * r + 1];
            unsigned char* to = mine + buf + ((first ^ (st << 6)) ^ (r << 5)) + 16 * k;
            if constexpr (sizeof(Out) == 4) {
              *reinterpret_cast<uint32_t*>(to) = prmt(__float_as_uint(y0), __float_as_uint(y1), 0x7632);
              *reinterpret_cast<uint32_t*>(to + kPlane) = prmt(__float_as_uint(y0), __float_as_uint(y1), 0x5410);
            } else if constexpr (std::is_same<Out, __half>::value) {
              *reinterpret_cast<__half2*>(to) = __floats2half2_rn(y0, y1);
            } else {
              *reinterpret_cast<uint32_t*>(to) = bf16_pair(y0, y1);
            }
          }
      };
      if constexpr (kMode == kLocal || kMode == kLocalSens) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {   // eight poles at a time
          float v[kStep][kRe][4], u[kStep][kSens ? kRe : 1][4];
#pragma unroll
          for (int j = kFrom; j < kTerms<kP>; ++j)
#pragma unroll
            for (int c = 0; c < kRe; ++c)
#pragma unroll
              for (int st = 0; st < kStep; ++st) {
                term<kP>(j, j > kFrom, v[st][c], f[st], matrix(2 * c + k));
                if (kSens) term<kP>(j, j > 0, u[st][kSens ? c : 0], f[st], matrix((kSens ? kV : 0) + 2 * c + k));
              }
#pragma unroll
          for (int m = 0; m < 4 * kStep; ++m) {   // (in the order of time: steps, chunks, for two poles)
            const int st = m >> 2, i = 2 * k + (m & 1), at = m & 3;
            if (kSens) {   // s' = q^16 s + 16 q^15 h + U x
              float xr = u[st][0][at], xi = kC ? u[st][kSens ? kRe - 1 : 0][at] : 0.f;
              xr = fmaf(ur[kSens ? i : 0], h[0][i], xr);
              if (kC) {
                xr = fmaf(-ui[kSens && kC ? i : 0], h[kRe - 1][i], xr);
                xi = fmaf(ur[kSens ? i : 0], h[kRe - 1][i], fmaf(ui[kSens && kC ? i : 0], h[0][i], xi));
              }
              next(i, sn[0][i], sn[kSens ? kRe - 1 : 0][i], xr, xi);
            }
            next(i, h[0][i], h[kRe - 1][i], v[st][0][at], v[st][kRe - 1][at]);
          }
        }
      } else if constexpr (kMode == kEmit) {
        float v[kStep][2][kRe][4];
        float odd = 0.f;   // NaN where a row holds an infinity or a NaN
#pragma unroll
        for (int j = kFrom; j < kTerms<kP>; ++j)
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int c = 0; c < kRe; ++c)
#pragma unroll
              for (int st = 0; st < kStep; ++st) term<kP>(j, j > kFrom, v[st][k][c], f[st], matrix(2 * c + k));
#pragma unroll
        for (int st = 0; st < kStep; ++st) {
          odd = fmaf(v[st][0][0][0], 0.f, fmaf(v[st][0][0][2], 0.f, odd));
          // (a state that is exported is that of the segment's last position, wherever in a step it lies: position by position)
          if (s0 + st == last) {
            const Row r = own_row();
            const int b = r.b, len = r.len;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int m = 8 * (i >> 1) + 2 * t + (i & 1);
              const size_t row_n = (size_t)d * a.N + m;
              if (m >= a.N) continue;
              const float p = __ldg(a.p + row_n), fr = __ldg(a.q + kRe * row_n), fi = kC ? __ldg(a.q + kRe * row_n + 1) : 0.f;
              float re = h[0][i], im = h[kRe - 1][i];
              for (int k = 0; k < len - 32 * final; ++k) {
                const unsigned char* from = smem + buf + row_at<kRow>(warp, g, 2 * (s0 + st) + (k >> 4)) + (k & 15) * 2;
                float x = 0.f;
#pragma unroll
                for (int pl = kP - 1; pl >= 0; --pl) x += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(from + pl * kPlane));
                x = kMask && (padded[st] >> k & 1u) ? 0.f : x * p;
                const float r = kC ? fmaf(fr, re, fmaf(-fi, im, x)) : fmaf(fr, re, x);
                if (kC) im = fmaf(fr, im, fi * re);
                re = r;
              }
              const size_t o = ((size_t)b * a.D + d) * a.N + m;
              a.h_out[kRe * o] = re;
              if (kC) a.h_out[kRe * o + 1] = im;
            }
          }
#pragma unroll
          for (int m = 0; m < 8; ++m) {   // what enters the chunks, in the place of what they add
            const int i = m & 3, k = i >> 1, at = 2 * (m >> 2) + (i & 1);
            const float vr = v[st][k][0][at], vi = v[st][k][kRe - 1][at];
            v[st][k][0][at] = h[0][i];
            if (kC) v[st][k][kRe - 1][at] = h[kRe - 1][i];
            next(i, h[0][i], h[kRe - 1][i], vr, vi);
          }
        }
        __syncwarp();
        const bool any_odd = __any_sync(0xffffffffu, odd != odd);
#pragma unroll
        for (int st = 0; st < kStep; ++st) emit(st, v[st], any_odd);
        __syncwarp();
      } else {
        uint32_t e[kStep][kP][4];
#pragma unroll
        for (int st = 0; st < kStep; ++st)
#pragma unroll
          for (int p = 0; p < kP; ++p) ldmatrix(e[st][p], rows(st) + (kP + p) * kPlane);
        if (kMask && some) {   // (its blocks lie in reversed order)
#pragma unroll
          for (int st = 0; st < kStep; ++st)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t two = padded[st] >> (16 * (i & 1) + 14 - 8 * (i >> 1) - 2 * t) & 3u;
              const uint32_t m = (two & 2u ? 0u : 0xffffu) | (two & 1u ? 0u : 0xffff0000u);
#pragma unroll
              for (int p = 0; p < kP; ++p) e[st][p][i] &= m;
            }
        }
        float enter[kMode == kBoth ? kStep : 1][2][kRe][4], odd = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          float v[kStep][kRe][4], u[kStep][kRe][4], l[kStep][kRe][4], w[kStep][kRe][4];
#pragma unroll
          for (int c = 0; c < kRe; ++c) {
            const Frag mv = matrix(2 * c + k), mu = matrix(kV + 2 * c + k);
#pragma unroll
            for (int j = 0; j < kTerms<kP>; ++j)
#pragma unroll
              for (int st = 0; st < kStep; ++st) {
                term<kP>(j, j > 0, v[st][c], f[st], mv);
                term<kP>(j, j > 0, l[st][c], e[st], mv);
                term<kP>(j, j > 0, u[st][c], f[st], mu);
                term<kP>(j, j > 0, w[st][c], e[st], mu);
              }
          }
#pragma unroll
          for (int o = 0; o < 4 * kStep; ++o) {   // (in the order of time: steps, chunks, for two poles)
            const int st = o >> 2, m = o & 3, i = 2 * k + (o & 1);
            if (kMode == kBoth) {
              enter[kMode == kBoth ? st : 0][k][0][m] = h[0][i];
              if (k == 0 && !(o & 1)) odd = fmaf(v[st][0][m], 0.f, odd);
            }
            float &hr = h[0][i], &hi = h[kRe - 1][i], &sr = sn[0][i], &si = sn[kSens ? kRe - 1 : 0][i];
            const float lr = l[st][0][m], li = l[st][kRe - 1][m], wr = w[st][0][m], wi = w[st][kRe - 1][m];
            float xr = u[st][0][m], xi = u[st][kRe - 1][m];
            constexpr int im = kSums ? kRe - 1 : 0;
            if (kC) {
              a1[0][i] = fmaf(lr, hr, fmaf(-li, hi, a1[0][i]));
              a1[im][i] = fmaf(lr, hi, fmaf(li, hr, a1[im][i]));
              a2[0][i] = fmaf(lr, sr, fmaf(-li, si, fmaf(wr, hr, fmaf(-wi, hi, a2[0][i]))));
              a2[im][i] = fmaf(lr, si, fmaf(li, sr, fmaf(wr, hi, fmaf(wi, hr, a2[im][i]))));
              xr = fmaf(ur[kSens ? i : 0], hr, fmaf(-ui[kSens && kC ? i : 0], hi, xr));
              xi = fmaf(ur[kSens ? i : 0], hi, fmaf(ui[kSens && kC ? i : 0], hr, xi));
            } else {
              a1[0][i] = fmaf(lr, hr, a1[0][i]);
              a2[0][i] = fmaf(lr, sr, fmaf(wr, hr, a2[0][i]));
              xr = fmaf(ur[kSens ? i : 0], hr, xr);
            }
            next(i, sr, si, xr, xi);
            next(i, hr, hi, v[st][0][m], v[st][kRe - 1][m]);
          }
        }
        // both with the 16 chunks as the reduction: entry (i, j) is the sum of the products of positions i and 15 - j
#pragma unroll
        for (int st = 0; st < kStep; ++st) {
          uint32_t ft[kP][4];
#pragma unroll
          for (int p = 0; p < kP; ++p) {
            uint32_t m[4];
            ldmatrix_t(m, rows(st) + p * kPlane);
            ft[p][0] = m[0]; ft[p][1] = m[2]; ft[p][2] = m[1]; ft[p][3] = m[3];
            ldmatrix_t(e[st][p], rows(st) + (kP + p) * kPlane);
          }
          if (kMask && some) {   // the padded positions' own products are omega's alone
            uint32_t only[kP][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {   // (a position of a chunk of the segments 2t and 2t + 1)
              const int at = 16 * (i & 1) + 15 - g - 8 * (i >> 1);
              const uint32_t m = (bits[2 * t * (kTile / 32) + st] >> at & 1u ? 0u : 0xffffu) |
                                 (bits[(2 * t + 1) * (kTile / 32) + st] >> at & 1u ? 0u : 0xffff0000u);
#pragma unroll
              for (int p = 0; p < kP; ++p) {
                only[p][i] = e[st][p][i] & ~m;
                e[st][p][i] &= m;
              }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              float r[4];
              correlate(r, ft, only, k);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (8 * k + 2 * t + (i & 1) == 15 - g - 8 * (i >> 1)) beside += r[i];
            }
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            float r[4];
            correlate(r, ft, e[st], k);
#pragma unroll
            for (int i = 0; i < 4; ++i) R[(kSums ? 4 * k + i : 0)] += r[i];   // (in fp32: the tensor pipe truncates its sums)
          }
        }
        if constexpr (kMode == kBoth) {
          __syncwarp();
          const bool any_odd = __any_sync(0xffffffffu, odd != odd);
#pragma unroll
          for (int st = 0; st < kStep; ++st) emit(st, enter[st], any_odd);
          __syncwarp();
        }
      }
    }
  };
  // padded positions of a tile: a word for 32 positions of a row, in the order they are walked; read a tile ahead
  constexpr int kVotes = F::kBits / kCh;   // words of a warp
  bool pad[kMask ? kVotes : 1];
  auto look = [&](int tile) {
    if constexpr (kMask) {
#pragma unroll
      for (int i = 0; i < kVotes; ++i) {
        const int word = warp * kVotes + i, r = blockIdx.y * 8 + word / (kTile / 32), bb = r / s.walked, first = (r - bb * s.walked) * s.T;
        const int pos = tile * kTile + word % (kTile / 32) * 32 + lane, at = first + pos;
        pad[i] = bb < a.B && pos < s.T && at < a.L && __ldg(a.mask + (size_t)bb * a.L + (s.rev ? a.L - 1 - at : at)) != 0;
      }
    }
  };
  look(0);
  auto arrive = [&](int tile) {   // the tile's rows, and the copies of one further on
    if constexpr (kMask) {
      uint32_t* bits = reinterpret_cast<uint32_t*>(smem + F::bits) + (tile & 1) * F::kBits;
#pragma unroll
      for (int i = 0; i < kVotes; ++i) {
        const uint32_t v = __ballot_sync(0xffffffffu, pad[i]);
        if (lane == 0) bits[warp * kVotes + i] = v;
      }
      look(tile + 1);
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(F::kSlots - 1) : "memory");
    if (tile < tiles) {
      const unsigned char* slot = smem + F::stage + tid * 16 + tile % F::kSlots * F::kSlot;
      unsigned char* buf = smem + tile % F::kBufs * F::kIns * kP * kPlane;
      turn<In, kCh, kTile, kP, kPlane, false>(sh, slot, buf);
      if constexpr (F::kIns == 2) turn<In, kCh, kTile, kP, kPlane, true>(sg, slot + F::kSlot / 2, buf + kP * kPlane);
    }
    issue(tile + F::kSlots);
  };
  auto leave = [&](int tile) {
    if constexpr (kOuts)
      if (tile >= 0) put<Out, kCh, kTile, kPlane>(so, smem + tile % F::kBufs * F::kIns * kP * kPlane);
  };
  // (a thread takes outputs from where it puts inputs, unless their types differ in size)
  constexpr bool kSame = !kOuts || sizeof(In) == sizeof(Out);
  if constexpr (F::kBufs == 2) {
    arrive(0);
    __syncthreads();
    for (int i = 0; i < tiles; ++i) {
      if constexpr (!kLean)
        if (i % (512 / kTile) == 0) settle(2 * min(16, steps - kTile / 32 * i));
      if constexpr (!kSame) {   // (and half and half from there on: complex 6 x 4999 x 2048 from fp32 344 us, all turning first 359)
        leave(i - 1);
        __syncthreads();
      }
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        if (((warp >> 2) & 1) == half) {
          if (d < a.D) multiply(i);
        } else {
          if constexpr (kSame) leave(i - 1);
          arrive(i + 1);
        }
      }
      __syncthreads();
    }
    leave(tiles - 1);
  } else {
    for (int i = 0; i < tiles; ++i) {
      if constexpr (!kLean)
        if (i % (512 / kTile) == 0) settle(2 * min(16, steps - kTile / 32 * i));
      arrive(i);
      __syncthreads();
      if (d < a.D) multiply(i);
      __syncthreads();
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");

  // (a state that is not finite stays so: such a row is gone through once more)
  float z = 0.f;
#pragma unroll
  for (int i = 0; i < 4 * kRe; ++i) z = fmaf(h[i >> 2][i & 3], 0.f, z);
  const unsigned odd = __ballot_sync(0xffffffffu, z != z);   // (of all lanes, also those without a row)
  const Row end = own_row();
  const int b = end.b, seg = end.seg, len = end.len;
  const bool odd_row = end.live && (odd >> (lane & 28) & 15u) != 0u;
  const bool again = kMode != kGrad && __any_sync(0xffffffffu, odd_row);
  if constexpr (kOuts) {
    __syncthreads();   // (the block's outputs are there)
    if (again && s.in != a.y) {   // (in place the inputs are gone: NaN from there on)
      const int first = seg * s.T;
      Out* y = reinterpret_cast<Out*>(a.y) + b * a.ysb + d;
      if (odd_row) start(end);
      one_by_one<In, kC, false>(s, b, d, first, odd_row ? len : 0, most, h, sn, [&](int k, float v) {
        if (a.silu) v = silu_of<Out>(v);
        if ((k & 3) == t) Elem<Out>::st(y + (s.rev ? a.L - 1 - first - k : first + k) * a.ysl, v);
      });
      if (odd_row && final >= 0) {
#pragma unroll
        for (int i = 0; i < 4 * kRe; ++i) {
          const int m = 8 * ((i >> 1) & 1) + 2 * t + (i & 1);
          if (m < a.N) a.h_out[kRe * (((size_t)b * a.D + d) * a.N + m) + (i >> 2)] = h[i >> 2][i & 3];
        }
      }
    }
  }
  if constexpr (kMode == kLocal || kMode == kLocalSens) {   // what the segment behind it starts from
    if (again) {
      if (odd_row) start(end);
      one_by_one<In, kC, kSens>(s, b, d, seg * s.T, odd_row ? len : 0, most, h, sn, [](int, float) {});
    }
    if (end.live) {
#pragma unroll
      for (int c = 0; c < kRe; ++c)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          *reinterpret_cast<float2*>(carry_at(b, seg + 1, c) + 8 * k) = make_float2(h[c][2 * k], h[c][2 * k + 1]);
          if (kSens)
            *reinterpret_cast<float2*>(carry_at(b, seg + 1, kRe + c) + 8 * k) =
                make_float2(sn[kSens ? c : 0][2 * k], sn[kSens ? c : 0][2 * k + 1]);
        }
    }
  }
  if constexpr (kSums) {   // sums over the rows, then the channel's gradients, a lane per pole
    __syncthreads();   // (the buffers are free)
    float* red = reinterpret_cast<float*>(smem) + warp * (16 * 17 + 4 * 16);
    float* sums = red + 16 * 17;   // [a1, a2][re, im][16]
#pragma unroll
    for (int c = 0; c < kRe; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int m = 4; m < 32; m <<= 1) {
          a1[c][i] += __shfl_xor_sync(0xffffffffu, a1[c][i], m);
          a2[c][i] += __shfl_xor_sync(0xffffffffu, a2[c][i], m);
        }
        if (g == 0) {
          sums[c * 16 + 8 * (i >> 1) + 2 * t + (i & 1)] = a1[c][i];
          sums[(2 + c) * 16 + 8 * (i >> 1) + 2 * t + (i & 1)] = a2[c][i];
        }
      }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      red[(g + 8 * ((i >> 1) & 1)) * 17 + 8 * (i >> 2) + 2 * t + (i & 1)] = R[(kSums ? i : 0)];
    __syncwarp();
    float lag = 0.f;
    if (lane < 16)
      for (int i = 0; i < 16 - lane; ++i) lag += red[i * 17 + 15 - i - lane];
    const int n = lane & 15;
    const size_t at = (size_t)dc * a.N + min(n, a.N - 1);
    const double fr = a.q[kRe * at], fi = kC ? a.q[kRe * at + 1] : 0.;
    double er = 0., ei = 0., dr = 0., di = 0.;   // sum of q^k R_k and its derivative
    for (int k = 15; k >= 0; --k) {
      const double v = __shfl_sync(0xffffffffu, lag, k);
      const double t0 = dr * fr - di * fi + er, t1 = dr * fi + di * fr + ei;
      dr = t0;
      di = t1;
      const double t2 = er * fr - ei * fi + v;
      ei = er * fi + ei * fr;
      er = t2;
    }
    if (lane < 16 && n < a.N && d < a.D) {
      const double s1r = sums[n], s1i = kC ? sums[16 + n] : 0., s2r = sums[32 + n], s2i = kC ? sums[48 + n] : 0.;
      const float hr = (float)(er + fr * s1r - fi * s1i), sr = (float)(dr + s1r + fr * s2r - fi * s2i);
      const float p = __ldg(a.p + at);
      if (kC) {
        const float hi = (float)(ei + fr * s1i + fi * s1r), si = (float)(di + s1i + fr * s2i + fi * s2r);
        const float gr = __ldg(a.g + 2 * at), gi = __ldg(a.g + 2 * at + 1);
        atomicAdd(a.dp + at, gr * hr - gi * hi);
        atomicAdd(a.dg + 2 * at, p * hr);
        atomicAdd(a.dg + 2 * at + 1, -p * hi);
        atomicAdd(a.dq + 2 * at, p * (gr * sr - gi * si));
        atomicAdd(a.dq + 2 * at + 1, -p * (gi * sr + gr * si));
      } else {
        const float gn = __ldg(a.g + at);
        atomicAdd(a.dp + at, gn * hr);
        atomicAdd(a.dg + at, p * hr);
        atomicAdd(a.dq + at, p * gn * sr);
      }
    }
    if (kMask) {
#pragma unroll
      for (int m = 1; m < 32; m <<= 1) beside += __shfl_xor_sync(0xffffffffu, beside, m);
    }
    if (lane == 0 && d < a.D) atomicAdd(a.domega + d, kMask ? lag + beside : lag);
  }
}

// ---- the carry ---------------------------------------------------------------------------------------------
// A thread per (sequence, channel, pole): what every segment starts from, in the place of what the segment before it adds;
// of the first one a state that comes in.
// kSens: its derivative too.
template <bool kC, bool kSens>
__global__ void __launch_bounds__(128) chunk_carry_kernel(ChunkArgs s) {
  const ScanArgs& a = s.a;
  constexpr int kRe = kC ? 2 : 1;
  const int i = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;   // channel and pole
  if (i >= a.D * 16) return;
  const int d = i >> 4, n = i & 15;
  const bool in = n < a.N;
  const size_t at = (size_t)d * a.N + n;
  const double qr = in ? (double)a.q[kRe * at] : 0., qi = in && kC ? (double)a.q[kRe * at + 1] : 0.;
  double ur = 1., ui = 0.;   // q^(T-1)
  double br = qr, bi = qi;
  for (int e = s.T - 1; e > 0; e >>= 1) {
    if (e & 1) {
      const double r = ur * br - ui * bi;
      ui = ur * bi + ui * br;
      ur = r;
    }
    const double r = br * br - bi * bi;
    bi = 2. * br * bi;
    br = r;
  }
  const double wr = ur * qr - ui * qi, wi = ur * qi + ui * qr;
  const float fr = (float)wr, fi = (float)wi, gr = (float)(s.T * ur), gi = (float)(s.T * ui);
  const float er = (float)(wr - fr), ei = (float)(wi - fi);   // (the same rounding in every segment: see settle())
  const size_t val = (size_t)a.D * 16, step = val * s.parts;
  float* v = s.carry + ((size_t)b * s.S + 1) * step + i;
  float hr = 0.f, hi = 0.f, sr = 0.f, si = 0.f;
  if (!kSens && a.h_in) {
    const size_t o = ((size_t)b * a.D + d) * a.N + n;
    if (in) {
      hr = __ldcg(a.h_in + kRe * o);
      if (kC) hi = __ldcg(a.h_in + kRe * o + 1);
    }
    float* first = v - step;
    first[0] = hr;
    if (kC) first[val] = hi;
  }
  constexpr int kB = 4;   // segments whose loads go out together
  for (int k0 = 1; k0 < s.S; k0 += kB, v += kB * step) {
    float lr[kB], li[kB], mr[kB], mi[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const float* p = v + (size_t)min(u, s.S - 1 - k0) * step;
      lr[u] = __ldcg(p);
      if (kC) li[u] = __ldcg(p + val);
      if (kSens) {
        mr[u] = __ldcg(p + kRe * val);
        if (kC) mi[u] = __ldcg(p + (kRe + 1) * val);
      }
    }
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      if (k0 + u >= s.S) break;
      float* p = v + (size_t)u * step;
      if (kSens) {
        float x = fmaf(gr, hr, mr[u]), y = 0.f;
        if (kC) {
          x = fmaf(-gi, hi, x);
          y = fmaf(gr, hi, fmaf(gi, hr, mi[u]));
        }
        x = fmaf(er, sr, kC ? fmaf(-ei, si, x) : x);
        const float r = kC ? fmaf(fr, sr, fmaf(-fi, si, x)) : fmaf(fr, sr, x);
        if (kC) si = fmaf(fi, sr, fmaf(fr, si, fmaf(ei, sr, fmaf(er, si, y))));
        sr = r;
        p[kRe * val] = sr;
        if (kC) p[(kRe + 1) * val] = si;
      }
      const float x = fmaf(er, hr, kC ? fmaf(-ei, hi, lr[u]) : lr[u]);
      float r = kC ? fmaf(fr, hr, fmaf(-fi, hi, x)) : fmaf(fr, hr, x);
      if (!kC && fabsf(hr) == INFINITY && qr != 0.) r = hr + lr[u];   // (whatever is left of q^T: T is even)
      if (kC) hi = fmaf(fi, hr, fmaf(fr, hi, fmaf(ei, hr, fmaf(er, hi, li[u]))));
      hr = r;
      p[0] = hr;
      if (kC) p[val] = hi;
    }
  }
}

// ---- launches ----------------------------------------------------------------------------------------------
template <typename In, typename Out, bool kC, int kMode, bool kMask, bool kLean = false>
void run(const ChunkArgs& s, cudaStream_t st) {
  using F = Form<In, Out, kC, kMode, kMask, kLean>;
  const dim3 grid((s.a.D + F::kCh - 1) / F::kCh, (unsigned)(((long long)s.a.B * s.walked + 7) / 8));
  launch(chunk_kernel<In, Out, kC, kMode, kMask, kLean>, grid, F::kThreads, F::total, (void*)st, s);
}

// Steps of a segment: a multiple of 64 (two steps of the tensor products) that minimises rounds of blocks over the SMs x
// (steps + what a block's start and end cost beside them), the launch of the local states counted as 0.45 of the others
// (measured: 0.4 - 0.5).  Returns that cost.
double pick(const ScanArgs& a, ChunkArgs& s) {
  const long long cols = (a.D + 15) / 16;
  double best = 1e30;
  auto consider = [&](int t) {
    const int n = (int)(((long long)a.L + t - 1) / t);
    const double rounds = ceil((double)(cols * (((long long)a.B * n + 7) / 8)) / 148.0);
    const double local = n > 1 ? ceil((double)(cols * (((long long)a.B * (n - 1) + 7) / 8)) / 148.0) : 0.;
    const double cost = (rounds + 0.45 * local) * (t + 96.0);
    if (cost < best) {
      best = cost;
      s.T = t;
      s.S = n;
    }
  };
  if (const int asked = g_options[OPT_CHUNK_STEPS].load(); asked > 0) {
    consider((std::min(asked, 1 << 24) + 63) / 64 * 64);
    return best;
  }
  for (int S = 1; S <= 1024; ++S) {
    const int t = (int)((((long long)a.L + S - 1) / S + 63) / 64 * 64);
    consider(t);
    if (t == 64) break;
  }
  return best;
}

bool envelope(int dtype, const ScanArgs& a) {
  return g_options[OPT_CHUNK].load() != 1 && g_options[OPT_DISABLE_STREAM].load() == 0 && !a.bidir && !a.prev_count && a.N >= 1 &&
         a.N <= 16 && a.B <= 65535 && a.L >= 1 && a.L < 0x7fffff00 && pieces_ok(dtype, a.D);
}

// Times in us, fitted to a grid of 38 shapes on one B200 (1 to 64 sequences, 209 to 32768 positions, 128 to 2048 channels).  Here:
// a part for the launches and the blocks' start, some 10 us more of it than the device takes, for a host that is not far ahead;
// and ns per unit of pick()'s cost by the number of parts of a value and the kind of poles, which over 600 more shapes is 4 to
// 12 % off (standard deviation, by form).  So near a border the choice is between forms that differ by a tenth.
double chunk_us(int dtype, const ScanArgs& a, bool bwd, bool lean, double cost, bool segmented) {
  static const double kFwd[2][3] = {{25., 32., 43.}, {44., 54., 64.}}, kBwd[2][3] = {{48., 75., 102.}, {97., 140., 168.}};
  static const double kLeanFwd[2] = {17., 22.5};
  const int parts = dtype == MEGA_BF16 ? 0 : dtype == MEGA_F16 ? 1 : 2, c = a.cplx ? 1 : 0;
  return (bwd ? (segmented ? 32. : 20.) : (segmented ? 22. : 14.)) +
         (lean ? kLeanFwd[c] : bwd ? kBwd[c][parts] : kFwd[c][parts]) * 1e-3 * cost * (segmented ? 1. : a.cplx ? 1.14 : 1.07) *
             (a.mask ? (bwd ? 1.22 : a.cplx ? 1.22 : 1.36) : 1.) * (lean && a.D % 16 ? 1.2 : 1.);   // (16 channels in two sectors)
}
// bf16 calls without states or mask that are too long for a cluster go to the tensor-core kernel, which takes leading parts alone
// and walks a sequence as one chain: here they take leading parts alone too (lean), in a quarter of the products and the same
// distance from float64 (2.8e-3 before the outputs are rounded): real 16 x 4096 x 1024 102 us as a chain, 90 here (123 in all
// parts); 32 x 2048 x 1024 164 and 95; 8 x 8192 x 1024 186 and 137; complex 4 x 4096 x 1024 219 and 60.
bool chain_takes(const ScanArgs& a) { return a.L < (1 << 24) && (!a.cplx || a.B >= 4); }   // (mma_cl_try)
bool lean_call(int dtype, const ScanArgs& a) {
  return dtype == MEGA_BF16 && !a.mask && !a.h_in && !a.h_out && g_options[OPT_DISABLE_MMA].load() == 0 &&
         (g_options[OPT_CHUNK].load() == 3 || (g_options[OPT_CHUNK].load() == 0 && chain_takes(a) && !scan_cluster_first(dtype, a, 1, 1)));
}
double chain_us(const ScanArgs& a, bool lean) {
  StreamArgs t{};
  t.B = a.B; t.L = a.L; t.D = a.D; t.N = a.N;
  t.mask = a.mask;
  t.cplx = a.cplx;
  t.silu = a.silu;
  const double us = mma_ema_chain_us(t);
  // (what takes leading parts alone may as well do so with accumulators in tensor memory: 16 x 4096 x 1024 74 us for 90, 8 x 8192 x 1024
  // 87 for 135; a call with states, which is here in all parts, keeps to those)
  return lean && !a.cplx ? std::min(us, 1.05 * tmem_ema_us(t, false, false)) : us;
}
// The form that a call takes otherwise: the scan backward (real bf16 16 x 4096 x 1024: 517 us against 233 here, complex 1481
// against 459, fp32 539 against 505); forward the cluster kernel, the scan (fp32 complex of that size: 565 against 385; real fp32
// of 4 sequences 86 against 90), or in bf16 the tensor-core kernel, which walks a sequence as one chain.
double other_us(int dtype, const ScanArgs& a, bool bwd, bool lean) {
  const double L = a.L, n = (double)a.B * a.D * L;
  if (bwd) return a.cplx ? 59. + n / 47e3 : 40. + n / 125e3;
  if (dtype == MEGA_BF16 && g_options[OPT_DISABLE_MMA].load() == 0 && chain_takes(a) &&
      !(a.cplx && (a.mask || (a.h_out && a.L % 32 != 0))))
    return scan_cluster_first(dtype, a, 1, 1) ? 0.9 * scan_cluster_us(dtype, a) : chain_us(a, lean);
  const double one = scan_cluster_us(dtype, a);
  return one < 1e29 ? 0.9 * one : std::min(scan_ema_fwd_us(a), a.cplx ? 25. + n / 123e3 : 15. + n / 270e3);
}
bool pays(int dtype, const ScanArgs& a, bool bwd, bool lean, double cost, bool segmented) {
  if (g_options[OPT_CHUNK].load() >= 2) return true;
  // (a prompt whose state leaves at a length that is no multiple of 32: the tensor-core kernel's head, then a tail)
  if (dtype == MEGA_BF16 && !a.cplx && a.h_out && a.L % 32 != 0) return false;
  return g_options[OPT_MMA_TILE].load() == 0 && chunk_us(dtype, a, bwd, lean, cost, segmented) < 0.93 * other_us(dtype, a, bwd, lean);
}

template <typename In, typename Out, bool kC, bool kMask, bool kLean = false>
bool fwd(int dtype, const ScanArgs& a, bool asked, cudaStream_t st) {
  ChunkArgs s{};
  s.a = a;
  const double cost = pick(a, s);
  if ((long long)a.B * s.S > 8LL * 65535 || !(asked || pays(dtype, a, false, kLean, cost, s.S > 1))) return false;
  const bool state = a.h_in || a.h_out;
  constexpr int kBlocks = 2 * Blocks<kC>::v + 2;
  s.blocks = kBlocks;
  s.parts = kC ? 2 : 1;
  const bool slots = s.S > 1 || (a.h_in && a.h_in == a.h_out);
  const size_t frag = (size_t)a.D * kBlocks * kBlockBytes, carry = slots ? (size_t)a.B * s.S * s.parts * a.D * 16 : 0;
  Scratch sc(Scratch::padded(frag) + Scratch::padded((size_t)a.D * 96 * 4) + Scratch::padded(carry * 4), st);
  if (!sc) return false;
  unsigned char* fr = sc.take<unsigned char>(frag);
  float* pow = sc.take<float>((size_t)a.D * 96);
  s.frag = fr;
  s.pow = pow;
  s.carry = carry ? sc.take<float>(carry) : nullptr;
  const PrepArgs p{a.p, a.q, a.g, a.omega, a.D, a.N, 0, 1, state ? 1 : 0, sizeof(Out) == 4 || kMask ? 0 : 1, kBlocks, fr, pow};
  launch(chunk_prepare_kernel<kC>, (unsigned)((a.D + 3) / 4), 128, 0, (void*)st, p);
  s.in = a.x;
  s.isb = a.xsb;
  s.isl = a.xsl;
  if (s.S > 1) {
    s.walked = s.S - 1;
    run<In, In, kC, kLocal, kMask, kLean>(s, st);
  }
  if (slots) launch(chunk_carry_kernel<kC, false>, dim3((a.D * 16 + 127) / 128, a.B), 128, 0, (void*)st, s);
  s.walked = s.S;
  run<In, Out, kC, kEmit, kMask, kLean>(s, st);
  g_last_kernel.store("chunk_ema", std::memory_order_relaxed);
  return true;
}

template <typename T, bool kC, bool kMask>
bool bwd(int dtype, const ScanArgs& a, cudaStream_t st) {
  ChunkArgs s{};
  s.a = a;
  const double cost = pick(a, s);
  if ((long long)a.B * s.S > 8LL * 65535 || !pays(dtype, a, true, false, cost, s.S > 1)) return false;
  constexpr int kRe = kC ? 2 : 1, kBlocks = 3 * Blocks<kC>::v + 2;
  s.blocks = kBlocks;
  s.parts = 2 * kRe;
  const size_t frag = (size_t)a.D * kBlocks * kBlockBytes, carry = s.S > 1 ? (size_t)a.B * s.S * s.parts * a.D * 16 : 0;
  Scratch sc(Scratch::padded(frag) + Scratch::padded((size_t)a.D * 96 * 4) + Scratch::padded(carry * 4), st);
  if (!sc) return false;
  unsigned char* fr = sc.take<unsigned char>(frag);
  float* pow = sc.take<float>((size_t)a.D * 96);
  s.frag = fr;
  s.pow = pow;
  s.carry = carry ? sc.take<float>(carry) : nullptr;
  const PrepArgs p{a.p, a.q, a.g, a.omega, a.D, a.N, 1, 1, 0, sizeof(T) == 4 || kMask ? 0 : 1, kBlocks, fr, pow};
  launch(chunk_prepare_kernel<kC>, (unsigned)((a.D + 3) / 4), 128, 0, (void*)st, p);
  s.in = a.dy;   // (walked backwards: its states are the adjoint)
  s.isb = a.gsb;
  s.isl = a.gsl;
  s.beside = a.x;
  s.bsb = a.xsb;
  s.bsl = a.xsl;
  s.rev = 1;
  if (s.S > 1) {
    s.walked = s.S - 1;
    run<T, T, kC, kLocalSens, false>(s, st);
    launch(chunk_carry_kernel<kC, true>, dim3((a.D * 16 + 127) / 128, a.B), 128, 0, (void*)st, s);
  }
  s.walked = s.S;
  // (real bf16: one launch reads dy once for both, 16 x 4096 x 1024 241 -> 233 us, 4 x 4096 x 1024 131 -> 109 with the local states
  // of dy alone)
  if constexpr (kPartsOf<T> == 1 && !kC) {
    run<T, T, kC, kBoth, kMask>(s, st);
  } else {   // (more parts or poles than registers and shared memory hold at once)
    run<T, T, kC, kGrad, kMask>(s, st);
    run<T, T, kC, kEmit, kMask>(s, st);
  }
  g_last_kernel.store("chunk_ema", std::memory_order_relaxed);
  return true;
}

}  // namespace

// (in place: a block reads a tile before it writes it, and no other block reads it once the local states are there)
bool chunk_ema_fwd_try(int dtype, int out_dtype, const ScanArgs& a, long long xsd, long long ysd, cudaStream_t s, bool asked) {
  if (!envelope(dtype, a) || !pieces_ok(out_dtype, a.D) || !rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) ||
      !rows_ok(out_dtype, a.y, a.ysb, a.ysl, ysd))
    return false;
#define MEGA_FWD(IN, OUT, MASK) return a.cplx ? fwd<IN, OUT, true, MASK>(dtype, a, asked, s) : fwd<IN, OUT, false, MASK>(dtype, a, asked, s)
#define MEGA_FWD_SAME(TY) if (a.mask) MEGA_FWD(TY, TY, true); else MEGA_FWD(TY, TY, false)
  if (dtype == MEGA_F32 && out_dtype == MEGA_BF16 && !a.mask) MEGA_FWD(float, __nv_bfloat16, false);
  if (dtype == MEGA_F32 && out_dtype == MEGA_F16 && !a.mask) MEGA_FWD(float, __half, false);
  if (dtype != out_dtype) return false;
  switch (dtype) {
    case MEGA_F32: MEGA_FWD_SAME(float);
    case MEGA_BF16:
      if (lean_call(dtype, a))
        return a.cplx ? fwd<__nv_bfloat16, __nv_bfloat16, true, false, true>(dtype, a, asked, s)
                      : fwd<__nv_bfloat16, __nv_bfloat16, false, false, true>(dtype, a, asked, s);
      MEGA_FWD_SAME(__nv_bfloat16);
    case MEGA_F16: MEGA_FWD_SAME(__half);
    default: return false;
  }
#undef MEGA_FWD_SAME
#undef MEGA_FWD
}

double chunk_ema_fwd_us(int dtype, const ScanArgs& a) {
  if (!envelope(dtype, a)) return 1e30;
  ChunkArgs s{};
  const double cost = pick(a, s);
  return chunk_us(dtype, a, false, lean_call(dtype, a), cost, s.S > 1);
}

bool chunk_ema_bwd_try(int dtype, const ScanArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s) {
  if (!envelope(dtype, a) || a.h_in || a.h_out || a.silu || !rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) ||
      !rows_ok(dtype, a.dy, a.gsb, a.gsl, gsd) || !rows_ok(dtype, a.y, a.ysb, a.ysl, ysd))
    return false;
  switch (dtype) {
#define MEGA_BWD(TY)                                                                                            \
  return a.mask ? (a.cplx ? bwd<TY, true, true>(dtype, a, s) : bwd<TY, false, true>(dtype, a, s))                \
                : (a.cplx ? bwd<TY, true, false>(dtype, a, s) : bwd<TY, false, false>(dtype, a, s))
    case MEGA_F32: MEGA_BWD(float);
    case MEGA_BF16: MEGA_BWD(__nv_bfloat16);
    case MEGA_F16: MEGA_BWD(__half);
#undef MEGA_BWD
    default: return false;
  }
}

}  // namespace mega
