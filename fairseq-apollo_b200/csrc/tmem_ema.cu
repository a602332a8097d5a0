// TimestepNorm -> causal EMA, and either by itself, for bf16 activations with contiguous channels and real poles: the statistics in plain
// fp32, a thread per channel of a sequence, the EMA in tcgen05 products with accumulators in tensor memory.
//
// A block walks 16 channels of 8 (4) sequences in tiles of 256 positions = 16 chunks of 16.  For one channel the (sequence, chunk) pairs
// of a tile are the 128 rows of its products; with h the states that enter a chunk and everything else a matrix of the channel,
//   local  v = V x         V (16 poles x 16): p q^(15-k)
//   carry  h' = q^16 h + v
//   output y = T x + G h   T (16 x 16): the taps, omega on the diagonal; G (16 x 16 poles): g q^(j+1)
//   - the normalised rows go to shared memory as 16-byte pieces along time (K-major), which serve as A of T x and as B of V x;
//   - V x is taken the other way round, poles on the rows: eight channels share an accumulator of 128 rows x 128
//     columns, and V's of eight channels under each other are one operand, of whose products with a channel's rows only the channel's
//     own 16 rows are written.  So a thread holds one pole and reads a sequence's chunks as columns in the order of time: the carry
//     stays inside it, one multiply-add per chunk;
//   - the states go back as bf16, eight chunks to a 16-byte piece (MN-major), over the rows of x that are no longer needed, and G h is
//     added to T x;
//   - an output's thread holds a (sequence, chunk) row, reads two positions of the 16 channels at a time and writes 32 bytes each;
//   - the outputs of eight channels have one of two places, with SiLU, whose outputs take long, one of three: T x of the next tile's
//     first eight does not wait for them then (16 x 4096 x 1024 126 -> 112 us, 8 x 8192 x 1024 192 -> 174, with the second output 200 ->
//     178; a place is free once its last values are in registers: 109, 159 and 161).  Tensor memory has room for that where V is in shared memory, from where it costs the plain form 89 -> 98 us.
// The statistics are a chain along time, 12 to 13 instructions a position.  One warp to a scheduler issues 0.4 of them a cycle (41 cycles
// a position), so three groups of warps take the parts of 32 positions in turn: a group sums its part about a centre of its own before
// the state of the part before is there, hands the state on, and normalises (28 cycles).  Warps: 12 of the statistics (ahead by up to
// two tiles), 4 of states, 4 of outputs (8 with SiLU), one that fetches x (TMA), one that issues products, 2 for the normalised
// activations as an output.  Everything is exchanged over mbarriers, the statistics over named barriers of two warps.
//
// What bounds it (16 x 4096 x 1024, 88 us against 142 in the forms of mma_cl_kernel.cuh; 67 for the statistics by themselves): issue
// slots and latency at 22 warps, 0.65 instructions per scheduler and cycle; the products' reads of shared memory 12 us, the outputs 4.
// Two things that cost much: outputs that may stay in L1 (103 us; no_allocate), and code that does not fit the instruction cache (the
// same walk in 250 KB of code 512 us; what is rare is out of line).  Over all SMs for long the power cap takes 12 % of the clock.
//
// The EMA by itself (x turned into rows in the statistics' place) takes 74 us there, 98 as a chain of mma_cl_kernel.cuh and 83 as products
// of chunks with their matrices; 8 x 8192 x 1024 87 for 135 (95 with two places of outputs; eight sequences to a
// block gain nothing from the third).  What is left is the chain from products to states to products to outputs
// of a tile; without its outputs, or without its states, it takes a fifth less each.  Without states of the layer the input gain is
// G's, as in the products of chunks, whose distance from float64 this has (2.296e-3; 2.304e-3 with the gain in V, as in the chain;
// behind the norm 2.865e-3 and 2.871e-3, the chain 2.869e-3).
//
// An infinity or a NaN among a chunk's rows would make NaN of the outputs ahead of it too: it goes to the products as zero, and the
// outputs from there on are written as NaN (the EMA by itself: as the recurrence has them).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "scratch.cuh"
#include "split_mma.cuh"
#include "stream_cl.cuh"
#include "tma.cuh"
#include "tmem_ema.cuh"
#include "umma.cuh"

namespace mega {

namespace {

enum Form { kPair, kNormOnly, kEmaOnly };   // TimestepNorm -> EMA; either by itself
constexpr int kMostQ = 8, kCh = 16, kTile = 256, kChunk = 16, kPart = 32;   // kPart: positions of a stage of x
constexpr int kStages = 4;   // of x, two parts each
constexpr int kPlane = 4096 + 16, kBuf = kCh * kPlane;   // rows of a channel (16 bytes on: eight channels hit different banks); of a tile
constexpr int kMat = 1024;                               // T and G of a channel
enum { kOffX = 0, kOffOp = kOffX + kStages * 2 * kPart * kMostQ * kCh * 2, kOffMat = kOffOp + 2 * kBuf, kOffInv = kOffMat + kCh * kMat,
       kOffMail = kOffInv + 16 * 64 * 4, kOffTaps = kOffMail + 4 * 32 * 8, kOffBad = kOffTaps + kCh * 16 * 4, kOffBar = kOffBad + kMostQ * kCh * 4,
       kOffV = kOffBar + 40 * 8 + 32, kOffEnd = kOffV + 2 * 4096 };   // kOffV: V of 8 channels under each other, twice
static_assert(kOffV % 16 == 0 && kOffEnd <= 227 * 1024, "shared memory");
// barriers
enum { kXFull = 0, kXEmpty = kStages, kOpFull = 2 * kStages, kOpEmpty = kOpFull + 2, kHDone = kOpEmpty + 2, kHRead, kTDone, kYDone = kTDone + 2, kYRead, kReady, kEnd, kXnRead, kBars = kXnRead + 2 };
static_assert(kBars <= 40, "barriers");
// columns of tensor memory: local states of eight channels; outputs of eight channels, two or three times (and V)
constexpr int kColH = 0, kColY = 128;
// kQ: sequences of a block, eight or (few of them: more blocks, each with half of the work) four.
// Warps: four of the states, four or (SiLU; four sequences, of which half of the warps have rows) eight of the outputs, twelve of the
// statistics in groups, x, products, and two for the normalised activations where they are an output.
// TimestepNorm by itself has the statistics' warps, x, and four (two) that write what they leave; the EMA by itself eight that turn x into
// rows in the place of the statistics'.
template <int kQ, bool kSilu, bool kXn, int kForm>
struct Roles {
  static constexpr bool kEma = kForm != kNormOnly;
  static constexpr int kWarps = kForm == kEmaOnly ? 8 : 12;           // that write rows
  static constexpr int kPer = kQ / 2, kGroups = kWarps / kPer;           // of a group (two sequences each); groups
  static constexpr int kOut = 4, kOuts = kForm == kEmaOnly ? 4 : kSilu || kQ == 4 ? 2 : 1, kStats = kEma ? kOut + 4 * kOuts : 0, kLoad = kStats + kWarps;
  static constexpr int kMma = kLoad + 1, kCopy = kMma + (kEma ? 1 : 0), kCopies = !kXn ? 0 : kEma || kQ == 4 ? 2 : 4;
  static constexpr int kThreads = 32 * (kCopy + kCopies);
  static constexpr int kStep = kQ * kCh * 2, kStageBytes = 2 * kPart * kStep;   // bytes from a position of x to the next; of a stage
};

struct TmemArgs {
  StreamArgs a;
  __nv_bfloat16 *y, *xn;
  long long ysb, ysl;
  const __nv_bfloat16* x;   // (beside the tensor map: for values that are not finite)
  long long xsb, xsl;
  int wide;   // outputs: 32-byte pieces
  // Sequences in runs: a work item is (run, group of sequences, tile of channels); blocks draw items in that order, and one starts
  // from what the item of the run before has left behind its flag.
  int tiles_d, per_run, runs, run_len;   // run_len: whole tiles
  int* sched;                            // the next item; flags of the items (1: its state is there, 2: it gave up)
  float4* state;                         // [B][D] the means behind the last three parts, squared deviations
  float* h;                              // [B][D][16]
};

__device__ __forceinline__ bool tried(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// A wait that gives up raises `gone`; from then on no wait lasts, and everything runs out on whatever the buffers hold.
// (out of line: the roles' code together has to stay within the instruction cache, about 32 KB)
__device__ __noinline__ void wait_on(uint32_t bar, uint32_t parity, long long limit, volatile int* gone) {
  const long long start = clock64();
  while (!*gone) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i) {   // (polling takes issue slots and shared memory from the other warps)
      __nanosleep(40);
      if (tried(bar, parity)) return;
    }
    if (clock64() - start > limit) {
      g_device_error = 1;
      *gone = 1;
    }
  }
}
__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ float minus_bf16(unsigned short x, float c) {   // x - c
  float d;
  asm("sub.f32.bf16 %0, %1, %2;" : "=f"(d) : "h"(x), "f"(c));
  return d;
}
template <int N>
__device__ __forceinline__ void landed(float (&v)[N]) {   // (the registers of a load from tensor memory, once it has been waited for)
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+f"(v[i]));
}
__device__ __forceinline__ void store32(void* to, const uint32_t (&w)[8]) {
  asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
               "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
// 16 channels of a position, or eight where the others are not there
__device__ __forceinline__ void store_channels(__nv_bfloat16* to, bool wide, bool both, const uint32_t (&w)[8]) {
  if (wide) {
    store32(to, w);
    return;
  }
  asm volatile("st.global.L1::no_allocate.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
  if (both)
    asm volatile("st.global.L1::no_allocate.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(to + 8), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
__device__ __forceinline__ float ex2_approx(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// silu of two values: 1 + exp(-v) by way of a power of two, and the reciprocal to one unit
__device__ __forceinline__ uint32_t silu_pair(float a, float b) {
  const f32x2 v = pack2(a, b), x = mul2(v, pack2(-1.44269504f, -1.44269504f));
  float xa, xb, da, db;
  unpack2(x, xa, xb);
  unpack2(add2(pack2(ex2_approx(xa), ex2_approx(xb)), pack2(1.f, 1.f)), da, db);
  unpack2(mul2(v, pack2(rcp_approx(da), rcp_approx(db))), a, b);
  return bf16_pair(a, b);
}

// byte of row (sequence, chunk) in a plane; a row's second eight values lie 128 bytes on
__device__ __forceinline__ int row_of(int s, int chunk) { return (2 * s + (chunk >> 3)) * 256 + (chunk & 7) * 16; }

// one position of a channel, dev from some c: the sums about c with it, and its normalised value
__device__ __forceinline__ float normed(float dev, float inv, float eps, float w, float bb, float& s1, float& s2) {
  s1 += dev;
  s2 = fmaf(dev, dev, s2);
  const float u = s1 * inv, v = fmaxf(fmaf(-u, u, fmaf(s2, inv, eps)), eps);
  return fmaf(dev - u, rsqrt_approx(v) * w, bb);
}
// two positions, the later one's sums behind the earlier one's; what does not depend on the order in packed arithmetic
__device__ __forceinline__ void normed2(float dev_a, float dev_b, f32x2 inv, float eps, f32x2 eps2, f32x2 w, f32x2 bb, float& s1, float& s2,
                                        float& out_a, float& out_b) {
  const float s1a = s1 + dev_a, s2a = fmaf(dev_a, dev_a, s2);
  s1 = s1a + dev_b;
  s2 = fmaf(dev_b, dev_b, s2a);
  const f32x2 u = mul2(pack2(s1a, s1), inv), q = fma2(pack2(s2a, s2), inv, eps2);
  float ua, ub, va, vb;
  unpack2(u, ua, ub);
  const f32x2 v = fma2(pack2(-ua, -ub), u, q);
  unpack2(v, va, vb);
  const f32x2 r = mul2(pack2(rsqrt_approx(fmaxf(va, eps)), rsqrt_approx(fmaxf(vb, eps))), w);
  unpack2(fma2(sub2(pack2(dev_a, dev_b), u), r, bb), out_a, out_b);
}
// A part with padded positions (bits of pad; nothing but zeros comes of them) or without a mean to begin with (fresh: its first
// value is the centre).  Returns the mean and the squared deviations behind it.
__device__ __noinline__ float2 few(const unsigned char* from, int step, const float* invs, unsigned char* to, unsigned pad, bool fresh, float c, float s2,
                                   float eps, float w, float bb) {
  float s1 = 0.f, u = 0.f;
#pragma unroll 1
  for (int i = 0; i < kPart; ++i) {
    float out = 0.f;
    if (!(pad >> i & 1u)) {
      const unsigned short v = *reinterpret_cast<const unsigned short*>(from + i * step);
      if (fresh) c = __uint_as_float((uint32_t)v << 16);
      fresh = false;
      out = normed(minus_bf16(v, c), invs[i], eps, w, bb, s1, s2);
      u = s1 * invs[i];
    }
    *reinterpret_cast<__nv_bfloat16*>(to + (i >> 4) * 16 + (i >> 3 & 1) * 128 + (i & 7) * 2) = __float2bfloat16_rn(out);
  }
  return make_float2(c + u, fmaf(-u, s1, s2));
}
// What is not finite among a part's values: zero to the products, and noted.
__device__ __noinline__ void odd_values(unsigned char* rows, int t0, bool live, int* first, volatile int* any) {
#pragma unroll 1
  for (int i = 0; i < kPart; ++i) {
    unsigned short* at = reinterpret_cast<unsigned short*>(rows + (i >> 4) * 16 + (i >> 3 & 1) * 128) + (i & 7);
    if ((*at & 0x7f80u) != 0x7f80u) continue;
    *at = 0;
    if (live) {
      atomicMin(first, t0 + i);
      *any = 1;
    }
  }
}
__device__ __forceinline__ void zero_row(unsigned char* to) {
  *reinterpret_cast<uint4*>(to) = make_uint4(0u, 0u, 0u, 0u);
  *reinterpret_cast<uint4*>(to + 128) = make_uint4(0u, 0u, 0u, 0u);
}
// What a channel's statistics leave behind: of the call, or for the next run (slot: of the group's mean).  Out of line, as are the others
// above: nothing of it is held in registers beside the walk.
__device__ __noinline__ void finish(const TmemArgs& t, int b, int d, float mean, float dev2, int seen) {
  const StreamArgs& a = t.a;
  const size_t at = (size_t)b * a.D + d;
  const long long count = a.prev_count[b] + a.count_offset + seen;
  a.mean_out[at] = seen > 0 ? mean : a.prev_mean[at];
  a.var_out[at] = seen > 0 ? not_negative(dev2 / (float)count) : a.prev_var[at];
  if (d == 0) a.count_out[b] = count;
}
__device__ __noinline__ void hand_on(const TmemArgs& t, int b, int d, int slot, float mean, float dev2) {   // (whole tiles, three groups: slots 0, 1, 2)
  float* to = reinterpret_cast<float*>(t.state + (size_t)b * t.a.D + d);
  to[slot] = mean;
  if (slot == 2) to[3] = dev2;
}

// The EMA by itself: outputs from an infinity or a NaN on, and the state, are the recurrence's, position by position in fp32 (in place,
// where the inputs are gone: NaN); so are those of a row whose state is not finite to begin with or in the end.  first: the first of the
// block's positions to be written.
__device__ __noinline__ void one_by_one(const TmemArgs& t, int run, int begin, int len, int b, int d, int first, bool silu) {
  const StreamArgs& a = t.a;
  if (b >= a.B || d >= a.D || first >= len) return;
  const bool in_place = t.x == t.y;
  const size_t o = (size_t)b * a.D + d;
  float h[16], p[16], q[16], g[16];
#pragma unroll
  for (int n = 0; n < 16; ++n) {
    const bool in = n < a.N;
    const size_t c = (size_t)d * a.N + (in ? n : 0);
    const bool apart = !a.h_in && !a.h_out;   // (as the states of the runs are)
    p[n] = !in ? 0.f : apart ? 1.f : a.p[c];
    q[n] = in ? a.q[c] : 0.f;
    g[n] = !in ? 0.f : apart ? a.p[c] * a.g[c] : a.g[c];
    h[n] = !in ? 0.f : run > 0 ? __ldcg(t.h + o * 16 + n) : a.h_in ? a.h_in[o * a.N + n] : 0.f;
  }
  const float om = a.omega[d];
  const __nv_bfloat16* x = t.x + b * t.xsb + (long long)begin * t.xsl + d;
  __nv_bfloat16* y = t.y + b * t.ysb + (long long)begin * t.ysl + d;
#pragma unroll 1
  for (int i = 0; i < len; ++i) {
    const float v = in_place ? __int_as_float(0x7fffffff) : __bfloat162float(x[i * t.xsl]);
    float out = om * v;
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      if (n >= a.N) break;
      h[n] = fmaf(q[n], h[n], p[n] * v);
      out = fmaf(g[n], h[n], out);
    }
    if (i >= first) y[i * t.ysl] = __float2bfloat16_rn(silu ? siluf_(out) : out);
  }
  float* to = run < t.runs - 1 ? t.h : a.h_out;
  const int pitch = run < t.runs - 1 ? 16 : a.N;
  if (to)
#pragma unroll
    for (int n = 0; n < 16; ++n)
      if (n < a.N) to[o * pitch + n] = h[n];
}

template <int kQ, bool kSilu, bool kXn, bool kMask, int kForm>
__global__ void __launch_bounds__(Roles<kQ, kSilu, kXn, kForm>::kThreads, 1) tsn_ema_tmem_kernel(const __grid_constant__ CUtensorMap tx, const __grid_constant__ TmemArgs t) {
  extern __shared__ __align__(128) unsigned char smem[];
  using R = Roles<kQ, kSilu, kXn, kForm>;
  constexpr bool kEma = R::kEma;
  static_assert(kForm != kEmaOnly || (!kXn && !kMask), "x as it is, whole");
  constexpr int kGroups = R::kGroups, kPer = R::kPer, kStep = R::kStep;
  constexpr bool kThree = kSilu || (kForm == kEmaOnly && kQ == 4), kVShared = kThree && kQ == 8;   // places of the outputs; V in shared memory
  constexpr int kColV = kQ == 4 ? 64 : 384;
  const StreamArgs& a = t.a;
  const uint32_t base = smem_u32(smem);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  int* bad = reinterpret_cast<int*>(smem + kOffBad);   // [sequence][channel]: first position that is not finite
  volatile int* gone = reinterpret_cast<volatile int*>(smem + kOffBar + kBars * 8);
  volatile int* any_bad = gone + 1;
  uint32_t* tm_slot = reinterpret_cast<uint32_t*>(smem + kOffBar + kBars * 8 + 8);
  auto bar = [&](int i) { return base + kOffBar + i * 8; };
  const long long limit = a.wait_limit;
  auto wait = [&](int i, int phase) {
    if (!tried(bar(i), phase & 1)) wait_on(bar(i), phase & 1, limit, gone);
  };
  auto settle = [&](int i, int phase) {   // what the block itself has under way: however short the limit of the other waits is
    const long long start = clock64();
    while (!tried(bar(i), phase & 1) && clock64() - start < 2 * limit + 4000000) {}
  };
  auto wait_all = [&](int i, int phase) {   // (a whole warp)
    wait(i, phase);
    __syncwarp();
  };

  int* drawn = reinterpret_cast<int*>(smem + kOffBar + kBars * 8 + 12);
  if (tid == 0) *drawn = t.runs > 1 ? atomicAdd(t.sched, 1) : (int)blockIdx.x;
  __syncwarp();   // (lane 0 comes from a branch of its own)
  if (kEma && warp == 0) tm_alloc(smem_u32(tm_slot), 512);
  if (tid == 32) {
    auto init = [&](int i, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar(i)), "r"(n) : "memory"); };
    for (int i = 0; i < kStages; ++i) {
      init(kXFull + i, 1);
      init(kXEmpty + i, 2 * kPer);   // (two parts)
    }
    for (int i = 0; i < 2; ++i) {
      init(kOpFull + i, R::kWarps);
      init(kOpEmpty + i, kEma ? 1 : R::kCopies);
      init(kXnRead + i, 2);
    }
    init(kHDone, 1);
    init(kHRead, 4);
    init(kTDone, 1);
    init(kTDone + 1, 1);
    init(kYDone, 1);
    init(kYRead, kPer * R::kOuts);
    init(kReady, 4);
    init(kEnd, 1);
    *gone = 0;
    *any_bad = 0;
    mbar_fence_init();
  }
  if (tid < kQ * kCh) bad[tid] = 0x7fffffff;
  tm_before();
  __syncthreads();
  tm_after();
  const uint32_t tm = kEma ? __shfl_sync(0xffffffffu, *tm_slot, 0) : 0u;   // (uniform to the compiler: what issues products needs it in uniform registers)
  const int item = *drawn, run = item / t.per_run, place = item - run * t.per_run;
  const int d0 = place % t.tiles_d * kCh, b0 = place / t.tiles_d * kQ;
  const int begin = run * t.run_len, len = min(a.L - begin, t.run_len);   // the block's positions
  const int tiles = (len + kTile - 1) / kTile, parts = (len + kPart - 1) / kPart;
  if (run > 0) {
    if (tid == 0) {
      const long long start = clock64();
      int flag = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(flag) : "l"(t.sched + 1 + item - t.per_run) : "memory");
        if (flag != 0) break;
        __nanosleep(200);
        if (clock64() - start > limit) {
          g_device_error = 1;
          break;
        }
      }
      if (flag != 1) *gone = 1;
    }
    __syncthreads();
  }

  if (kForm == kEmaOnly && warp >= R::kStats && warp < R::kLoad) {
    // ---- x into rows: a thread per channel of a sequence, the groups' warps take the parts in turn -----------------------------
    const int nw = (warp - R::kStats) % kPer, own = (warp - R::kStats) / kPer, ch = lane & 15, s = 2 * nw + (lane >> 4);
    const bool live = d0 + ch < a.D && b0 + s < a.B;
    const unsigned char* from = smem + kOffX + nw * 64 + lane * 2;
    int part = own;
#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
      if (tile >= 2) wait_all(kOpEmpty + (tile & 1), (tile >> 1) - 1);
      unsigned char* plane = smem + kOffOp + (tile & 1) * kBuf + ch * kPlane + row_of(s, 0);
      const int end = min(8 * tile + 8, parts);
#pragma unroll 1
      for (; part < end; part += kGroups) {
        wait_all(kXFull + (part >> 1) % kStages, (part >> 1) / kStages);
        const unsigned char* v = from + (part & (2 * kStages - 1)) * (R::kStageBytes / 2);
        unsigned char* to = plane + (part & 4) * 64 + (part & 3) * 32;
        uint32_t w[kPart / 2], odd = 0u;
#pragma unroll
        for (int i = 0; i < kPart / 2; ++i) {
          w[i] = __byte_perm(*reinterpret_cast<const unsigned short*>(v + 2 * i * kStep), *reinterpret_cast<const unsigned short*>(v + (2 * i + 1) * kStep), 0x5410);
          odd |= (w[i] & 0x7f807f80u) + 0x00800080u;   // (bits 15 and 31: an exponent of ones)
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(to + (q >> 1) * 16 + (q & 1) * 128) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        if (odd & 0x80008000u) odd_values(to, part * kPart, live, bad + s * kCh + ch, any_bad);
        __syncwarp();
        if (lane == 0) arrive(bar(kXEmpty + (part >> 1) % kStages));
      }
      if (end == parts && part - kGroups == parts - 1) {   // (behind the end: zeros)
#pragma unroll 1
        for (int r = 2 * ((parts - 1) & 7) + 2; r < 16; ++r) zero_row(plane + (r >> 3) * 256 + (r & 7) * 16);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) arrive(bar(kOpFull + (tile & 1)));
    }
  } else if (kForm != kEmaOnly && warp >= R::kStats && warp < R::kLoad) {
    // ---- statistics: three (four sequences to a block: six) threads per channel of a sequence, which take the parts in turn ---------
    const int nw = (warp - R::kStats) % kPer, own = (warp - R::kStats) / kPer, ch = lane & 15, s = 2 * nw + (lane >> 4), d = d0 + ch, b = b0 + s;
    const bool live = d < a.D && b < a.B;
    const float eps = a.eps, w = live ? __ldg(a.gamma + d) : 0.f, bb = live ? __ldg(a.beta + d) : 0.f;
    const float n0 = b < a.B ? (float)(a.prev_count[b] + a.count_offset) : 1.f;
    // the mean and the squared deviations so far, as handed from part to part
    const size_t at = live ? (size_t)b * a.D + d : 0;
    float mean = live ? a.prev_mean[at] : 0.f, dev2 = (live ? a.prev_var[at] : 1.f) * n0;
    float c = mean;   // what deviations are taken from
    if (run > 0 && live) {   // (so that the bits are those of one run)
      const float4 m = __ldcg(t.state + at);
      mean = m.z;
      dev2 = m.w;
      c = own == 0 ? m.x : own == 1 ? m.y : m.z;
    }
    // values that are not finite come with sums that are not, unless the parameters make them
    bool odd = live && !(eps >= 1e-12f && fabsf(w) <= 1e10f && fabsf(bb) <= 1e37f);
    float* tab = reinterpret_cast<float*>(smem + kOffInv) + (kPer * own + nw) * 64 + (lane >> 4) * 32;
    float2* mail = reinterpret_cast<float2*>(smem + kOffMail) + nw * 32 + lane;
    const unsigned char* from = smem + kOffX + nw * 64 + lane * 2;
    const unsigned char* mrow = kMask && b < a.B ? a.mask + (size_t)b * a.L : nullptr;
    auto mask_at = [&](int part) -> unsigned {   // bit i: the part's position i is padded, of the lane's sequence
      const int t0 = part * kPart;
      if constexpr (kMask) {
        const int p = t0 + ch;
        const unsigned lo = __ballot_sync(0xffffffffu, mrow == nullptr || p >= len || __ldg(mrow + p) != 0);
        const unsigned hi = __ballot_sync(0xffffffffu, mrow == nullptr || p + 16 >= len || __ldg(mrow + p + 16) != 0);
        return lane & 16 ? __byte_perm(lo, hi, 0x7632) : __byte_perm(lo, hi, 0x5410);
      } else {
        return len - t0 >= 32 ? 0u : ~((1u << max(len - t0, 0)) - 1u);
      }
    };
    const f32x2 eps2 = pack2(eps, eps), w2 = pack2(w, w), bb2 = pack2(bb, bb);
    int seen = 0;
    if (kMask)
      for (int i = 0; i < own; ++i) seen += 32 - __popc(mask_at(i));
    const int plain = kMask ? 0 : len / kPart;   // parts that are whole
    // the mean and the squared deviations go from a part to the next by shared memory and a barrier of the two warps (every wait of
    // theirs that could last is bounded, so both come)
    const int mine = 1 + kPer * own + nw, theirs = 1 + kPer * ((own + 1) % kGroups) + nw;
    int part = own;
#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
      if (tile >= 2) wait_all(kOpEmpty + (tile & 1), (tile >> 1) - 1);
      unsigned char* plane = smem + kOffOp + (tile & 1) * kBuf + ch * kPlane + row_of(s, 0);
      const int first = part, end = min(8 * tile + 8, parts);
#pragma unroll 1
      for (; part < end; part += kGroups) {
        if (!kMask) seen = begin + part * kPart;
        const unsigned pad = mask_at(part);
        // 1 / count of the part's positions, for the whole warp
        tab[ch] = rcp_approx(n0 + (float)(seen + __popc(~pad & ((2u << ch) - 1u))));
        tab[ch + 16] = rcp_approx(n0 + (float)(seen + __popc(~pad & (~0u >> (15 - ch)))));
        const float n = n0 + (float)seen;
        wait_all(kXFull + (part >> 1) % kStages, (part >> 1) / kStages);
        const unsigned char* v = from + (part & (2 * kStages - 1)) * (R::kStageBytes / 2);
        unsigned char* to = plane + (part & 4) * 64 + (part & 3) * 32;
        auto take = [&]() {   // the state that the part before left
          if (part == 0) return;
          asm volatile("bar.sync %0, 64;" ::"r"(mine) : "memory");
          const float2 m = *mail;
          mean = m.x;
          dev2 = m.y;
        };
        auto give = [&]() {
          if (part == parts - 1) return;
          *mail = make_float2(mean, dev2);
          asm volatile("bar.arrive %0, 64;" ::"r"(theirs) : "memory");
        };
        auto whole = [&](auto some) {   // some: positions are padded (zeros; the counts know of them)
          constexpr bool kSome = decltype(some)::value;
          // (the first time: any value of the channel is as good a centre as its mean)
          if (!kSome && part < kGroups && run == 0) c = __uint_as_float((uint32_t)*reinterpret_cast<const unsigned short*>(v) << 16);
          float dev[kPart], t1[2] = {0.f, 0.f}, t2[2] = {0.f, 0.f};
#pragma unroll
          for (int i = 0; i < kPart; ++i) {
            dev[i] = minus_bf16(*reinterpret_cast<const unsigned short*>(v + i * kStep), c);
            if (kSome && (pad >> i & 1u)) dev[i] = 0.f;
            t1[i & 1] += dev[i];
            t2[i & 1] = fmaf(dev[i], dev[i], t2[i & 1]);
          }
          take();
          const float off = mean - c;
          float s1 = n * off, s2 = fmaf(s1, off, dev2);
          const float e1 = s1 + (t1[0] + t1[1]), ue = e1 * tab[kPart - 1];
          mean = c + ue;
          dev2 = fmaf(-e1, ue, s2 + (t2[0] + t2[1]));
          give();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float out[8];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const ulonglong2 inv = reinterpret_cast<const ulonglong2*>(tab)[2 * q + j];
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const int at = 8 * q + 4 * j + 2 * i;
                normed2(dev[at], dev[at + 1], i ? inv.y : inv.x, eps, eps2, w2, bb2, s1, s2, out[4 * j + 2 * i], out[4 * j + 2 * i + 1]);
                if (kSome && (pad >> at & 1u)) out[4 * j + 2 * i] = 0.f;
                if (kSome && (pad >> at & 2u)) out[4 * j + 2 * i + 1] = 0.f;
              }
            }
            *reinterpret_cast<uint4*>(to + (q >> 1) * 16 + (q & 1) * 128) =
                make_uint4(bf16_pair(out[0], out[1]), bf16_pair(out[2], out[3]), bf16_pair(out[4], out[5]), bf16_pair(out[6], out[7]));
          }
        };
        if (kMask ? !__any_sync(0xffffffffu, pad != 0u || n == 0.f) : part < plain && (part > 0 || !__any_sync(0xffffffffu, n == 0.f))) {
          whole(std::false_type{});
        } else if (kMask && !__any_sync(0xffffffffu, n == 0.f)) {
          whole(std::true_type{});
        } else {
          take();
          const float2 after = few(v, R::kStep, tab, to, pad, n == 0.f, mean, dev2, eps, w, bb);
          mean = after.x;
          dev2 = after.y;
          give();
        }
        c = mean;
        if (kMask) {
          seen += 32 - __popc(pad);
          if (part == parts - 1 && live && !*gone) finish(t, b, d, mean, dev2, seen);
#pragma unroll 1
          for (int i = 1; i < kGroups; ++i) seen += 32 - __popc(mask_at(part + i));
        }
        __syncwarp();
        if (lane == 0) arrive(bar(kXEmpty + (part >> 1) % kStages));
      }
      if (kEma && (odd || !(fabsf(dev2) < 3e38f))) {
#pragma unroll 1
        for (int i = first; i < part; i += kGroups) odd_values(plane + (i & 4) * 64 + (i & 3) * 32, i * kPart, live, bad + s * kCh + ch, any_bad);
      }
      if (kEma && !kMask && end == parts && run < t.runs - 1 && live && !*gone) hand_on(t, b, d, part - parts, c, dev2);
      if (end == parts && part - kGroups == parts - 1) {   // (behind the end: zeros)
        if (!kMask && run == t.runs - 1 && live && !*gone) finish(t, b, d, mean, dev2, a.L);
#pragma unroll 1
        for (int r = 2 * ((parts - 1) & 7) + 2; r < 16; ++r) zero_row(plane + (r >> 3) * 256 + (r & 7) * 16);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) arrive(bar(kOpFull + (tile & 1)));
    }
  } else if (kEma && warp < 4) {
    // ---- states and outputs -------------------------------------------------------------------------------------
    const int half = lane >> 4, pole = lane & 15;
    const uint32_t quarter = tm + ((uint32_t)warp << 21);
    // states of channel 2 warp + half, four sequences at a time, then of channel 8 + that: they take turns as the first set
    float q16 = 0.f, q16_other = 0.f, h[kQ / 2][4];
    auto turn_states = [&]() {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float v = h[0][i];
#pragma unroll
        for (int k = 1; k < kQ / 2; ++k) h[k - 1][i] = h[k][i];
        h[kQ / 2 - 1][i] = v;
      }
    };
    auto turn_pole = [&]() {
      const float q = q16;
      q16 = q16_other;
      q16_other = q;
    };
#pragma unroll 1
    for (int g = 0; g < 2; ++g) {   // the matrices of channel 8 g + 2 warp + half, from this lane's pole
      const int ch = 8 * g + 2 * warp + half, d = d0 + ch;
      const bool in = d < a.D && pole < a.N;
      const size_t o = in ? (size_t)d * a.N + pole : 0;
      const float gain = in ? __ldg(a.p + o) : 0.f, q = in ? __ldg(a.q + o) : 0.f;
      const bool apart = !a.h_in && !a.h_out;   // the input gain is G's
      const float p = apart ? (in ? 1.f : 0.f) : gain, gm = !in ? 0.f : apart ? gain * __ldg(a.g + o) : __ldg(a.g + o);
      double q2 = (double)q * q;
      q2 *= q2;
      q2 *= q2;
      q16 = (float)(q2 * q2);
      unsigned char* mat = smem + kOffMat + ch * kMat;
      float* taps = reinterpret_cast<float*>(smem + kOffTaps) + ch * 16;
      float pw = 1.f, vk[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        vk[15 - e] = p * pw;
        float tap = p * gm * pw;
#pragma unroll
        for (int m = 8; m > 0; m >>= 1) tap += __shfl_xor_sync(0xffffffffu, tap, m);
        if (pole == e) taps[e] = e == 0 && d < a.D ? tap + __ldg(a.omega + d) : tap;
        pw *= q;
        *reinterpret_cast<__nv_bfloat16*>(mat + 512 + (e >> 3) * 256 + (pole >> 3) * 128 + (e & 7) * 16 + (pole & 7) * 2) =
            __float2bfloat16_rn(gm * pw);
      }
      if constexpr (kVShared) {
        unsigned char* v = smem + kOffV + g * 4096 + (2 * warp + half) * 512 + (pole >> 3) * 256 + (pole & 7) * 16;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<uint4*>(v + i * 128) = make_uint4(bf16_pair(vk[8 * i], vk[8 * i + 1]), bf16_pair(vk[8 * i + 2], vk[8 * i + 3]),
                                                              bf16_pair(vk[8 * i + 4], vk[8 * i + 5]), bf16_pair(vk[8 * i + 6], vk[8 * i + 7]));
      } else {
        uint32_t words[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) words[i] = bf16_pair(vk[2 * i], vk[2 * i + 1]);
        tm_st8(quarter + kColV + 8 * g, words);
      }
      __syncwarp();
      float row[16];   // row `pole` of T
#pragma unroll
      for (int k = 0; k < 16; ++k) row[k] = k <= pole ? taps[max(pole - k, 0)] : 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<uint4*>(mat + (pole >> 3) * 256 + i * 128 + (pole & 7) * 16) =
            make_uint4(bf16_pair(row[8 * i], row[8 * i + 1]), bf16_pair(row[8 * i + 2], row[8 * i + 3]),
                       bf16_pair(row[8 * i + 4], row[8 * i + 5]), bf16_pair(row[8 * i + 6], row[8 * i + 7]));
#pragma unroll 1
      for (int hf = 0; hf < kQ / 4; ++hf) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int sq = b0 + 4 * hf + i;
          const size_t o = (size_t)sq * a.D + d;
          h[0][i] = !in || sq >= a.B ? 0.f : run > 0 ? __ldcg(t.h + o * 16 + pole) : a.h_in ? a.h_in[o * a.N + pole] : 0.f;
          if (kForm == kEmaOnly && !(fabsf(h[0][i]) <= 3.4e38f)) {   // (one_by_one)
            h[0][i] = 0.f;
            bad[(4 * hf + i) * kCh + ch] = 0;
            *any_bad = 1;
          }
        }
        turn_states();
      }
      turn_pole();
    }
    if (!kVShared) {
      tm_wait_st();
      tm_before();
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) arrive(bar(kReady));

#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
      unsigned char* op = smem + kOffOp + (tile & 1) * kBuf;
      const int last = min(15, (len - tile * kTile + kChunk - 1) / kChunk - 1);   // the tile's last chunk
#pragma unroll 1
      for (int unit = 0; unit < kQ / 2; ++unit) {
        const int g = unit / (kQ / 4), hf = unit % (kQ / 4), ch = 8 * g + 2 * warp + half;
        if (hf == 0) {
          wait_all(kHDone, g);
          tm_after();
        }
        unsigned char* to = op + ch * kPlane + (pole >> 3) * 128 + (pole & 7) * 16 + hf * 2048;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float v[32];
          tm_ld32(quarter + kColH + 64 * hf + 32 * j, v);
          tm_wait_ld();
          landed(v);
          if (j == 0 && hf == 0) {   // (x is still read until then)
            wait_all(kTDone + g, tile);
            if (kXn && g == 0) wait_all(kXnRead + (tile & 1), tile >> 1);
          }
          auto carry = [&](auto stops) {   // stops: chunks behind the last one, whose local states are zero, leave the states as they are
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t w[8];
              float hs = h[0][2 * j + i], enter = 0.f;
#pragma unroll
              for (int c = 0; c < 16; ++c) {
                if (c & 1) w[c >> 1] = bf16_pair(enter, hs);
                else enter = hs;
                hs = fmaf(decltype(stops)::value && c > last ? 1.f : q16, hs, v[16 * i + c]);
              }
              h[0][2 * j + i] = hs;
              *reinterpret_cast<uint4*>(to + (2 * j + i) * 512) = make_uint4(w[0], w[1], w[2], w[3]);
              *reinterpret_cast<uint4*>(to + (2 * j + i) * 512 + 256) = make_uint4(w[4], w[5], w[6], w[7]);
            }
          };
          if (last < 15) carry(std::true_type{});
          else carry(std::false_type{});
        }
        if (hf == kQ / 4 - 1) {
          fence_proxy_async();
          tm_before();
          __syncwarp();
          if (lane == 0) arrive(bar(kHRead));
        }
        turn_states();
        if (hf == kQ / 4 - 1) turn_pole();
      }
    }
    const bool on = run < t.runs - 1;
    if ((on || a.h_out || kForm == kEmaOnly) && !*gone) {
#pragma unroll 1
      for (int unit = 0; unit < kQ / 2; ++unit) {
        const int ch = 8 * (unit / (kQ / 4)) + 2 * warp + half, d = d0 + ch;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int s = 4 * (unit % (kQ / 4)) + i;
          const size_t o = (size_t)(b0 + s) * a.D + d;
          bool redo = false;
          if constexpr (kForm == kEmaOnly) {   // (one_by_one; in place only where an input was the reason)
            const unsigned odd = __ballot_sync(0xffffffffu, !(fabsf(h[0][i]) <= 3.4e38f));
            redo = bad[s * kCh + ch] < len;
            if (!redo && t.x != t.y && (odd >> (16 * half) & 0xffffu)) {
              redo = true;
              if (pole == 0) bad[s * kCh + ch] = 0;
              *any_bad = 1;
            }
            __syncwarp();
          }
          if (d < a.D && pole < a.N && b0 + s < a.B && !redo) {
            if (on) t.h[o * 16 + pole] = h[0][i];
            else if (a.h_out) a.h_out[o * a.N + pole] = bad[s * kCh + ch] < len ? __int_as_float(0x7fffffff) : h[0][i];
          }
        }
        turn_states();
      }
    }
  } else if (kEma && warp < R::kStats) {
    // ---- outputs: a thread per sequence and chunk ----------------------------------------------------------------
    const int half = lane >> 4, chunk = lane & 15, s_out = 2 * (warp & 3) + half, b = b0 + s_out;
    const uint32_t quarter = tm + ((uint32_t)(warp & 3) << 21);
    constexpr int kMine = kChunk / R::kOuts;   // positions
    const int first = ((warp - R::kOut) >> 2) * kMine;
#pragma unroll 1
    for (int tile = 0; (warp & 3) < kPer && tile < tiles; ++tile) {
      const int t0 = tile * kTile + chunk * kChunk;
      const long long row = (long long)b * t.ysb + (long long)(begin + t0) * t.ysl + d0;
      wait_all(kYDone, tile);
      tm_after();
      const int rows = *gone ? 0 : a.B;   // (nothing is stored once a wait has run out)
      const bool full = t.wide != 0 && b0 + kQ <= rows && (tile + 1) * kTile <= len;
      __nv_bfloat16* to = t.y + row + first * t.ysl;
      const uint32_t y0 = 128 * (kThree ? 2 * tile % 3 : 0), y1 = 128 * (kThree ? (2 * tile + 1) % 3 : 1);
#pragma unroll 1
      for (int i = first; i < first + kMine; i += 2) {
        float v[2 * kCh];
        uint32_t w[2][8];
#pragma unroll
        for (int c = 0; c < kCh; ++c) tm_ld2(quarter + kColY + (c < 8 ? y0 : y1) + 16 * (c & 7) + i, v + 2 * c);
        tm_wait_ld();
        landed(v);
        if (i == first + kMine - 2) {   // (the next products need not wait for what is on its way to memory)
          tm_before();
          __syncwarp();
          if (lane == 0) arrive(bar(kYRead));
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
#pragma unroll
          for (int c = 0; c < 8; ++c) w[k][c] = kSilu ? silu_pair(v[4 * c + k], v[4 * c + 2 + k]) : bf16_pair(v[4 * c + k], v[4 * c + 2 + k]);
          if (full) store32(to, w[k]);
          else if (b < rows && t0 + i + k < len) store_channels(to, t.wide != 0, d0 + 8 < a.D, w[k]);
          to += t.ysl;
        }
      }
      if (kForm != kEmaOnly && *any_bad && b < rows) {
        for (int c = 0; c < kCh && d0 + c < a.D; ++c)
          for (int k = max(bad[s_out * kCh + c] - t0, first); k < first + kMine && t0 + k < len; ++k) {
            t.y[row + k * t.ysl + c] = __ushort_as_bfloat16(0x7fff);
            if (kXn && !(kMask && __ldg(a.mask + (size_t)b * a.L + t0 + k))) t.xn[row + k * t.ysl + c] = __ushort_as_bfloat16(0x7fff);   // (padded: zero)
          }
      }
    }
  } else if (warp == R::kLoad) {
    // ---- x ------------------------------------------------------------------------------------------------------
    if (lane == 0) {
      prefetch_tensormap(&tx);
      const int stages = (parts + 1) / 2;
      int k = 0;
      for (; k < stages; ++k) {
        const int st = k % kStages;
        if (k >= kStages) wait(kXEmpty + st, k / kStages - 1);
        if (*gone) break;
        uint64_t* full = reinterpret_cast<uint64_t*>(smem + kOffBar) + kXFull + st;
        mbar_expect_tx(full, R::kStageBytes);
        if (k != a.withhold_step) tma_load_3d(smem + kOffX + st * R::kStageBytes, &tx, d0, b0, begin + k * 2 * kPart, full);
      }
      // (what is on its way arrives before the block ends, also where others leave without having waited for it)
      for (int i = max(k - kStages, 0); i < k; ++i)
        if (i != a.withhold_step) settle(kXFull + i % kStages, i / kStages);
    }
  } else if (warp >= R::kCopy) {
    // ---- the normalised activations as an output, before states take their place --------------------------------------
    const int chunk = lane & 15;
#pragma unroll 1
    for (int tile = 0; kXn && tile < tiles; ++tile) {
      const int t0 = tile * kTile + chunk * kChunk;
      wait_all(kOpFull + (tile & 1), tile >> 1);
      const int rows = *gone ? 0 : a.B;
      const bool full = t.wide != 0 && b0 + kQ <= rows && (tile + 1) * kTile <= len;
#pragma unroll 1
      for (int i = 0; i < 2 * kQ / (kXn ? R::kCopies : 1); ++i) {   // two sequences, four of their 16 positions
        const int s = kQ / R::kCopies * (warp - R::kCopy) + 2 * (i >> 2) + (lane >> 4), b = b0 + s, k0 = 4 * (i & 3);
        const unsigned char* from = smem + kOffOp + (tile & 1) * kBuf + row_of(s, chunk) + (k0 >> 3) * 128 + (k0 & 4) * 2;
        uint2 v[kCh];
#pragma unroll
        for (int c = 0; c < kCh; ++c) v[c] = *reinterpret_cast<const uint2*>(from + c * kPlane);
        __nv_bfloat16* to = t.xn + (long long)b * t.ysb + (long long)(begin + t0 + k0) * t.ysl + d0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t w[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) w[c] = __byte_perm(k < 2 ? v[2 * c].x : v[2 * c].y, k < 2 ? v[2 * c + 1].x : v[2 * c + 1].y, k & 1 ? 0x7632 : 0x5410);
          if (full) store32(to, w);
          else if (b < rows && t0 + k0 + k < len) store_channels(to, t.wide != 0, d0 + 8 < a.D, w);
          to += t.ysl;
        }
      }
      __syncwarp();
      if (lane == 0) arrive(bar((kEma ? kXnRead : kOpEmpty) + (tile & 1)));
    }
  } else if (kEma && umma_elect()) {
    // ---- products -----------------------------------------------------------------------------------------------
    constexpr uint32_t kLocal = umma_idesc(128, 16 * kQ, false), kTaps = umma_idesc(128, 16, false), kStates = umma_idesc(128, 16, true);
    wait(kReady, 0);
    tm_after();
    const uint64_t rows0 = umma_desc(base + kOffOp, 128, 256), mats0 = umma_desc(base + kOffMat, 128, 256);
    const uint64_t v0 = umma_desc(base + kOffV, 128, 256);
    auto local = [&](uint64_t op, int g) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if constexpr (kVShared) umma_16_rows(tm + kColH, v0 + g * (4096 / 16), op + (8 * g + j) * kPlane / 16, kLocal, j);
        else umma_16_rows(tm + kColH, tm + kColV + 8 * g, op + (8 * g + j) * kPlane / 16, kLocal, j);
      }
      umma_commit(bar(kHDone));
    };
    auto taps = [&](uint64_t op, int g, uint32_t y) {   // T x
#pragma unroll
      for (int j = 0; j < 8; ++j) umma(y + 16 * j, op + (8 * g + j) * kPlane / 16, mats0 + (8 * g + j) * kMat / 16, kTaps, false);
      umma_commit(bar(kTDone + g));
    };
    auto outs = [&](uint64_t op, int g, uint32_t y) {   // G h
#pragma unroll
      for (int j = 0; j < 8; ++j)
        umma(y + 16 * j, op + (8 * g + j) * kPlane / 16, mats0 + ((8 * g + j) * kMat + 512) / 16, kStates, true);
    };
#pragma unroll 1
    for (int tile = 0; tile < tiles && !*gone; ++tile) {   // (once a wait has run out no more are issued: what is under way ends soon)
      const uint64_t op = rows0 + (tile & 1) * (kBuf / 16);
      const uint32_t y0 = tm + kColY + 128 * (kThree ? 2 * tile % 3 : 0), y1 = tm + kColY + 128 * (kThree ? (2 * tile + 1) % 3 : 1);
      wait(kOpFull + (tile & 1), tile >> 1);
      tm_after();
      local(op, 0);
      if (!kThree) {
        if (tile > 0) wait(kYRead, tile - 1);
        tm_after();
      }
      taps(op, 0, y0);   // (three places: of two tiles ago, whose outputs the tile before has waited for)
      if (!kThree) taps(op, 1, y1);
      wait(kHRead, 0);
      tm_after();
      local(op, 1);
      if (kThree) {
        if (tile > 0) wait(kYRead, tile - 1);
        tm_after();
        taps(op, 1, y1);
      }
      outs(op, 0, y0);
      wait(kHRead, 1);
      tm_after();
      outs(op, 1, y1);
      umma_commit(bar(kYDone));
      umma_commit(bar(kOpEmpty + (tile & 1)));
    }
    // (nothing may be under way when the block ends)
    umma_commit(bar(kEnd));
    settle(kEnd, 0);
  }
  __syncwarp();   // (one lane has issued products, or fetched x: barriers are for warps that are together again)
  if constexpr (kForm == kEmaOnly) {   // what the products cannot give
    __syncthreads();
    if (*any_bad && !*gone && tid < kQ * kCh) one_by_one(t, run, begin, len, b0 + tid / kCh, d0 + tid % kCh, bad[tid], kSilu);
    __syncwarp();
  }
  tm_before();
  __syncthreads();
  tm_after();
  if (kEma && warp == 0) tm_free(tm, 512);
  if (run < t.runs - 1 && tid == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(t.sched + 1 + item), "r"(*gone ? 2 : 1) : "memory");
  }
}

template <int kQ, bool kSilu, bool kXn, bool kMask, int kForm = kPair>
void launch_form(const CUtensorMap& tx, const TmemArgs& t, cudaStream_t s) {
  const unsigned grid = (unsigned)(t.per_run * t.runs);
  launch(tsn_ema_tmem_kernel<kQ, kSilu, kXn, kMask, kForm>, grid, Roles<kQ, kSilu, kXn, kForm>::kThreads, kOffEnd, (void*)s, tx, t);
}

}  // namespace

namespace {

// us of a call in so many runs, from 200 timings (1 to 64 sequences, 128 to 32768 positions, 256 to 2048 channels on one B200) and, of
// the pair, 4300 of 20 to 6000 positions (to 0.9 - 1.1 of the time, one in ten outside): a block's start and end, then ns a position, and
// rounds of blocks over the SMs.  A tile that is not whole takes some part of a whole one's time.
double runs_us(const StreamArgs& a, bool norm, bool xn, int runs, int q) {
  const double tiles = (double)((a.D + kCh - 1) / kCh) * ((a.B + q - 1) / q) * runs;
  const int len = ((a.L + kTile - 1) / kTile + runs - 1) / runs * kTile;
  const double rounds = std::max(std::ceil(tiles / 148.), (double)runs);   // (a sequence's runs follow one another)
  if (!norm) {   // (13 with states of the layer; several rounds at the clock that the power cap leaves)
    double ns = q == 4 ? (a.silu ? 13.4 : 9.6) : a.silu ? 18.3 : 15.9;
    if (a.D % kCh) ns = std::max(ns, 28.5 * (q == 4 ? 0.7 : 1.));
    return 4. + rounds * ((a.h_in || a.h_out ? 13. : 6.) + len * ns * (rounds > 2. ? 1.04e-3 : 1e-3));
  }
  // [sequences of a block][outputs in 32- or 16-byte pieces][SiLU + 2 second output]; with masks that pad something
  // (16 x 4096 x 1024 88 us, SiLU 107, second output 107, both 124; 8 x 8192 x 1024 112, 159 with SiLU; 24 x 1500 x 1000 103 and 138)
  static const double kNs[2][2][4] = {{{12.2, 18.1, 14.7, 18.5}, {16., 18.3, 22., 24.3}}, {{18.7, 23.3, 23.5, 27.4}, {25.5, 28.4, 38., 40.}}};
  const bool pieces = a.D % kCh != 0;
  const double ns = kNs[q == 8][pieces][(a.silu ? 1 : 0) + (xn ? 2 : 0)] + (!a.mask ? 0. : q == 4 ? 3. : pieces ? 6.5 : 5.);
  const double steps = runs > 1 ? len : 0.5 * (a.L + len);
  return (runs > 1 ? 6. : 3.5) + rounds * (7.5 + (a.silu ? 1. : 0.) + (xn ? 2. : 0.) - (a.mask ? 1. : 0.) + steps * ns * 1e-3);
}
// with the limit of its waits, and the load that a test withholds
StreamArgs bounded(StreamArgs a) {
  const int limit = g_options[OPT_WAIT_LIMIT].load(), withheld = g_options[OPT_WITHHOLD_LOAD].load();
  a.wait_limit = limit > 0 ? (long long)limit : 4000000000LL;
  a.withhold_step = withheld > 0 ? withheld : -1;
  return a;
}
// sequences of a block: four where that gives all blocks an SM at once (a position takes 12 - 23 ns for 20 - 32: 8 x 8192 x 1024 112 us
// against 176, 4 x 4096 x 1024 60 against 88; in two rounds 16 x 4096 x 1024 118 against 91)
int sequences_of(const StreamArgs& a) { return (long long)((a.D + kCh - 1) / kCh) * ((a.B + 3) / 4) <= 148 ? 4 : 8; }
// runs: what balances the blocks' rounds (16 x 8192 x 5120 in two: 4.5 rounds of the sequence for 5; 26 x 2208 x 640 97 us, in one 106)
int runs_of(const StreamArgs& a, bool norm, bool xn) {
  int best = 1;
  if (a.mask) return best;   // (the positions that count are known to the run before alone)
  double least = (norm ? 0.98 : 0.95) * runs_us(a, norm, xn, 1, 8);
  for (int n = 2; n <= 8; n *= 2)
    if (const double us = runs_us(a, norm, xn, n, 8); a.L >= 1024 * n && us < least) {
      least = us;
      best = n;
    }
  return best;
}

}  // namespace

double tmem_ema_us(const StreamArgs& a, bool norm, bool xn) {
  const int q = sequences_of(a);
  const double us = runs_us(a, norm, xn, q == 8 ? runs_of(a, norm, xn) : 1, q);
  return norm && us > 400. ? 1.06 * us : us;   // (at the clock that the power cap leaves: 64 x 8192 x 2048 1.25 ms in a row, one at a time 1.17)
}

bool tmem_ema_try(int dtype, const void* x, void* y, void* xn, long long xsb, long long xsl, long long ysb, long long ysl, bool norm,
                  const StreamArgs& a, cudaStream_t s, int asked) {
  if (!norm && (a.mask || xn)) return false;
  if (dtype != MEGA_BF16 || a.cplx || a.N < 1 || a.N > 16 || a.D % 8 != 0 || (a.h_out && a.L % kChunk != 0) || a.L >= (1 << 24)) return false;
  if (!aligned_to(y, 16) || (xn && !aligned_to(xn, 16)) || ysb % 8 != 0 || ysl % 8 != 0) return false;
  const int q = asked == 4 ? 4 : asked > 0 ? 8 : sequences_of(a);
  const long long per_run = (long long)((a.D + kCh - 1) / kCh) * ((a.B + q - 1) / q);
  if (per_run > (1 << 24)) return false;
  CUtensorMap tx;
  if (!make_tensor_map_3d(&tx, dtype, x, a.D, a.B, a.L, xsb, xsl, kCh, q, 2 * kPart, CU_TENSOR_MAP_SWIZZLE_NONE)) return false;
  TmemArgs t{};
  t.a = bounded(a);
  t.x = reinterpret_cast<const __nv_bfloat16*>(x);
  t.xsb = xsb;
  t.xsl = xsl;
  t.y = reinterpret_cast<__nv_bfloat16*>(y);
  t.xn = reinterpret_cast<__nv_bfloat16*>(xn);
  t.ysb = ysb;
  t.ysl = ysl;
  t.wide = a.D % 16 == 0 && ysb % 16 == 0 && ysl % 16 == 0 && aligned_to(y, 32) && (!xn || aligned_to(xn, 32));
  t.tiles_d = (a.D + kCh - 1) / kCh;
  t.per_run = (int)per_run;
  t.runs = q == 4 || a.mask ? 1 : asked > 0 ? asked - 8 : runs_of(a, norm, xn != nullptr);
  const int tiles = (a.L + kTile - 1) / kTile, run_tiles = (tiles + t.runs - 1) / t.runs;
  t.runs = (tiles + run_tiles - 1) / run_tiles;
  t.run_len = run_tiles * kTile;
  auto go = [&]() {
    if (!norm) {
      if (q == 4) a.silu ? launch_form<4, true, false, false, kEmaOnly>(tx, t, s) : launch_form<4, false, false, false, kEmaOnly>(tx, t, s);
      else a.silu ? launch_form<8, true, false, false, kEmaOnly>(tx, t, s) : launch_form<8, false, false, false, kEmaOnly>(tx, t, s);
      return;
    }
#define MEGA_TMEM_OF(Q, SILU, XN) (a.mask ? launch_form<Q, SILU, XN, true>(tx, t, s) : launch_form<Q, SILU, XN, false>(tx, t, s))
#define MEGA_TMEM(SILU, XN) (q == 4 ? MEGA_TMEM_OF(4, SILU, XN) : MEGA_TMEM_OF(8, SILU, XN))
    if (a.silu) xn ? MEGA_TMEM(true, true) : MEGA_TMEM(true, false);
    else xn ? MEGA_TMEM(false, true) : MEGA_TMEM(false, false);
#undef MEGA_TMEM
#undef MEGA_TMEM_OF
  };
  if (t.runs == 1) {
    go();
  } else {
    const size_t flags = 1 + (size_t)per_run * t.runs, rows = (size_t)a.B * a.D;
    Scratch sc(Scratch::padded(flags * 4) + Scratch::padded(rows * 16) + Scratch::padded(rows * 64), s);
    if (!sc) return false;
    t.sched = sc.take<int>(flags);
    t.state = sc.take<float4>(rows);
    t.h = sc.take<float>(rows * 16);
    if (cudaMemsetAsync(t.sched, 0, flags * 4, s) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    go();
  }
  static const char* const kNames[9] = {"", "tsn_ema_mma tmem", "tsn_ema_mma tmem segmented runs=2", "tsn_ema_mma tmem segmented runs=3",
                                        "tsn_ema_mma tmem segmented runs=4", "tsn_ema_mma tmem segmented runs=5", "tsn_ema_mma tmem segmented runs=6",
                                        "tsn_ema_mma tmem segmented runs=7", "tsn_ema_mma tmem segmented runs=8"};
  g_last_kernel.store(!norm ? "ema_mma tmem" : a.mask ? "tsn_ema_mma tmem mask" : kNames[std::min(t.runs, 8)], std::memory_order_relaxed);
  return true;
}

// (16 x 4096 x 1024 67 us, masked 93; 8 x 8192 x 1024 82 and 115; 64 x 4096 x 2048 469 and 626, in a row 518 and 632; 24 x 1500 x 1000
// 76 and 92)
double tmem_norm_us(const StreamArgs& a) {
  const int q = sequences_of(a);
  const double tiles = (double)((a.D + kCh - 1) / kCh) * ((a.B + q - 1) / q), rounds = std::ceil(tiles / 148.);
  const int len = (a.L + kTile - 1) / kTile * kTile;
  const double ns = ((q == 4 ? 8.5 : 14.8) + (a.mask ? (q == 4 ? 4.5 : 6.) : 0.)) * (a.D % kCh ? 1.35 : 1.);
  return 4. + rounds * (5. + len * ns * 1e-3);
}

bool tmem_norm_try(int dtype, const void* x, void* y, long long xsb, long long xsl, long long ysb, long long ysl, const StreamArgs& a,
                   cudaStream_t s) {
  if (dtype != MEGA_BF16 || a.D % 8 != 0 || a.L >= (1 << 24) || x == y) return false;
  if (!aligned_to(y, 16) || ysb % 8 != 0 || ysl % 8 != 0) return false;
  const int q = sequences_of(a);
  const long long blocks = (long long)((a.D + kCh - 1) / kCh) * ((a.B + q - 1) / q);
  if (blocks > (1 << 24)) return false;
  CUtensorMap tx;
  if (!make_tensor_map_3d(&tx, dtype, x, a.D, a.B, a.L, xsb, xsl, kCh, q, 2 * kPart, CU_TENSOR_MAP_SWIZZLE_NONE)) return false;
  TmemArgs t{};
  t.a = bounded(a);
  t.xn = reinterpret_cast<__nv_bfloat16*>(y);
  t.ysb = ysb;
  t.ysl = ysl;
  t.wide = a.D % 16 == 0 && ysb % 16 == 0 && ysl % 16 == 0 && aligned_to(y, 32);
  t.tiles_d = (a.D + kCh - 1) / kCh;
  t.per_run = (int)blocks;
  t.runs = 1;
  t.run_len = (a.L + kTile - 1) / kTile * kTile;
  if (q == 4) a.mask ? launch_form<4, false, true, true, kNormOnly>(tx, t, s) : launch_form<4, false, true, false, kNormOnly>(tx, t, s);
  else a.mask ? launch_form<8, false, true, true, kNormOnly>(tx, t, s) : launch_form<8, false, true, false, kNormOnly>(tx, t, s);
  g_last_kernel.store("tsn_ema_mma tmem norm", std::memory_order_relaxed);
  return true;
}

cudaError_t tmem_ema_read_device_error(int* v, bool reset) { return read_device_error(v, reset); }

}  // namespace mega
