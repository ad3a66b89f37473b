// A stack of transformer layers over few rows as one resident kernel (ttb_chain_forward).
//
// What bounds it: a decoding step or a request of a few tokens is a chain of dependent operations, five a layer, each of which moves
// a few megabytes of weights and computes next to nothing. Here one grid of one CTA per SM runs all of them (GPT-2 small, one row, us a step: layer by
// layer 398, this kernel 171; its weights stream in 38). An operation takes 2 to 2.5 us: 1.0 to 1.3 from the last CTA's store to the other SMs having its
// result, and as much again of instructions that depend on one another. So
//   * No barriers. The operations hand their results on through memory that the call has filled with a word which no result can be
//     (TTB_CHAIN_UNWRITTEN); a reader asks for the words that it needs until they are others. A barrier over the grid was a flush, an atomic and a poll, 1.0
//     us, and the rows' way from L2 behind it as much again: 278 us a step then, 235 with nothing else changed. (ttb_chain_forward, whose callers place
//     results as they like, still has them.)
//   * Nothing is spilled (but 20 bytes by the kernel for 64 rows and depths that are no whole number of steps). With 227 KB of shared memory a spill does not stay in L1: 200 us with 320 bytes of them, 175 without. A third warpgroup, of which one
//     warp sends for weights, gives its registers to the two that compute.
//   * Few instructions. Every operation runs through its own once, behind all those of the others, so that fetching them counts: 1 to 3 cycles each
//     while a layer's fit in 32 KB, 6 and more beyond (measured on straight code), and a jump 30 to 100. One function for all products, steps of K that are jumped
//     over together, what does not depend on the operations before ahead of the wait for them: 175 -> 158.
//   * Weights. The output columns of a product are dealt out in units of eight (eight rows of W[N,K]: contiguous memory), as evenly as
//     they go over the CTAs. One warp copies the units that the CTA will read next into a shared-memory ring (cp.async.bulk) until it is full: about a layer
//     ahead of the arithmetic. Norm weights and biases travel the same way, and cached keys and values are brought to L2. (By a computing warp at the barriers,
//     the vocabulary's 77 MB took 37 us; now 20.)
//   * The products run on mma.sync m16n8k16, the columns of two units as its m and eight rows as its n: 128-row tcgen05 tiles would be empty but for a few
//     rows, and the round trip through tensor memory is longer than the whole product. The warps split K; the order of k inside a 32-wide chunk is permuted
//     alike for both operands so that each thread loads 16 bytes at a time: rows straight from global memory into fragments (no warp reads what another does),
//     W from the ring without bank conflicts (row pitch 64 bytes past a multiple of 128). Partial sums meet in shared memory.
//   * A layer norm in front of a product: every CTA normalises all rows itself into shared memory, which is cheaper than handing them on.
//   * Attention: the warps of a CTA share a (row, head), or several; scores on mma.sync, online softmax, merged through shared memory.
// us a step, before / now: GPT-2 small 1 row 278 / 158, 8 rows 291 / 187, 16 rows 325 / 224, 24 rows 391 / 285, 32 rows 427 / 335, 64 rows 627 / 567 (the
// operations alone, 30 cached tokens). From 16 rows on, what every CTA reads of the rows counts: 24 rows of an FFN's 3072 columns are 147 KB for each.
#include <algorithm>
#include <initializer_list>
#include <vector>

#include "ttb_chain_rules.cuh"
#include "ttb_common.cuh"
#include "ttb_sm100.cuh"

using namespace ttb;

namespace {

using chain::kWarps;                            // the operations are bound by what every warp has to do anyway: fewer warps, with more registers
constexpr int kThreads = kWarps * 32;            // of the warps that compute
constexpr int kBlock = kThreads + 128;          // and a warpgroup of which one warp sends for weights
// Registers: 384 threads are launched with 168 each; the third warpgroup gives 128 of its own up and the others take 64 more, so that nothing is
// spilled: with 227 KB of shared memory there is no room for spills in L1, and each is a trip to L2.
constexpr int kFeedRegisters = 40, kComputeRegisters = 232;
static_assert(kThreads * kComputeRegisters + 128 * kFeedRegisters <= kBlock * 168, "what the block was launched with");
constexpr int kGroup = 4;                       // most units of eight columns that a CTA computes at a time
constexpr int kRowPad = 64;                     // bytes between rows in shared memory, for the banks
constexpr int kNormed = 1024;                   // most columns of a layer norm
constexpr int kParamSlots = 3;
constexpr int kBars = 16;                       // groups of units that may be on their way
using chain::kBiasUnits;
constexpr int kParamBytes = 2 * kNormed * 2 + kBiasUnits * 16;
constexpr int kSmemLimit = 227 * 1024;
constexpr int kHeadDim = 64;
constexpr float kLog2e = 1.4426950408889634f;

struct ChainParams {
  ttb_chain_op ops[TTB_CHAIN_MAX_OPS];  // `reserved` holds what kGroupMask and the constants beside it say
  int n_ops;
  int ring_bytes, a_bytes, sums_bytes;  // shared memory of the weights' ring, of the normalised rows and of partial sums
  int* counter;  // arrivals at the grid's barrier
  int* status;
};
constexpr int kOpWords = sizeof(ttb_chain_op) / 4;
// ttb_chain_op::reserved: the units of a group, whether the operation begins with a barrier over the grid, whether its rows (A, or q with the keys
// beside it) and its residual are waited for word by word, and whether there is a layer norm.
constexpr int kGroupMask = 7, kBarrier = 1 << 3, kRowsFlow = 1 << 4, kResidualFlows = 1 << 5, kNorm = 1 << 6;
constexpr uint32_t kUnwritten = TTB_CHAIN_UNWRITTEN;  // a word of the flow that nobody has written yet
constexpr int kMostTries = 1 << 21;                   // of a wait for such words: a trip to L2 each, about a second

// What a CTA has to do of an operation.
struct Todo {
  // ttb_chain_op::reserved and kind (below 0: nothing); the units of a product (CTA r also writes normalised row r), or how many (row, head) pairs
  // and the logarithm of the warps for each
  int how, kind, lo, hi;
  __device__ __forceinline__ explicit Todo(const ttb_chain_op& op) {
    how = op.reserved;
    kind = op.kind;
    lo = hi = 0;
    if (kind == TTB_CHAIN_LINEAR) {
      const ttb_chain_linear& o = op.u.linear;
      const uint32_t units = ((uint32_t)o.N + 7) >> 3;
      lo = (int)chain::first_unit(units, blockIdx.x, gridDim.x);
      hi = (int)chain::first_unit(units, blockIdx.x + 1, gridDim.x);
      if (hi == lo && !(o.gamma && o.normed && (int)blockIdx.x < o.M)) kind = -1;
    } else {
      lo = (op.u.attention.rows * op.u.attention.heads - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
      if (lo <= 0) kind = -1;
      hi = lo <= 1 ? 3 : lo <= 2 ? 2 : lo <= 4 ? 1 : 0;
      static_assert(kWarps == 8, "warps a pair: 8, 4, 2, 1");
    }
  }
};

struct Shared {
  ttb_chain_op ops[TTB_CHAIN_MAX_OPS];   // (read from the kernel's parameters, every operation's first use would miss the constant cache)
  int4 todo[TTB_CHAIN_MAX_OPS];
  uint8_t params[kParamSlots][kParamBytes];
  uint64_t full[kBars];
  int bytes_done, params_done, groups_done;  // what of the rings all warps are done with
  volatile int abort_flag;                   // a wait of this CTA has run out
  volatile int gave_up[2];                   // one of a warp that computes, by the barrier ahead of which it did: all of them see the same behind it
};
constexpr int kSharedBytes = (sizeof(Shared) + 127) / 128 * 128;

// The thread's number, read anew in every operation: what the compiler derives from it ahead of the loop over the operations it
// has to spill.
__device__ __forceinline__ int thread() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// a / b for 0 <= a < 2^16, 0 < b: the quotient's error stays below the half that is added.
__device__ __forceinline__ int div_small(int a, int b) { return (int)__fdividef((float)a + 0.5f, (float)b); }

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 pack(const float (&f)[8]) {
  uint4 r;
  __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
  return r;
}
__device__ __forceinline__ float gelu16(float x) {  // the form of the tensor-core Linear's 16-bit outputs
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(0.7978845608028654f * (x + 0.044715f * x * x * x)));
  return 0.5f * x * (1.0f + y);
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Element offset of token j of sequence b in a paged cache ([pages, B, 16, H]).
__device__ __forceinline__ long long cache_row(int j, int b, int B, int H) { return (((long long)(j >> 4) * B + b) * 16 + (j & 15)) * H; }

// ---------------------------------------------------------------------------------------------
// between CTAs
// ---------------------------------------------------------------------------------------------
// What one CTA writes and others read goes past L1, a word at a time: each word is there or it is not, whatever the order in which they arrive.
__device__ __forceinline__ uint4 load16(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t load4(const void* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store16(void* p, const uint4& v) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void store4(void* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
// The greatest of the words so far: kUnwritten if one of them has not been written.
__device__ __forceinline__ void look(uint32_t& top, const uint4& v) { top = max(max(top, max(v.x, v.y)), max(v.z, v.w)); }

// After a look that found something missing: whether to look again. All lanes of a warp call it. Where it gives up, `tries` is kMostTries.
[[nodiscard]] __device__ __forceinline__ bool again(bool missing, int& tries, Shared& sm) {
  if (!__any_sync(0xffffffffu, missing)) return false;
  if (sm.abort_flag) tries = kMostTries - 1;
  if (++tries < kMostTries) return true;
  sm.abort_flag = 1;
  return false;
}
// Waits for sixteen bytes of the warp's: while there is nothing, many rows are too much to ask for again and again.
[[nodiscard]] __device__ __forceinline__ bool wait_ahead(const void* p, Shared& sm) {
  uint4 v;
  int tries = 0;
  do v = load16(p);
  while (again(max(max(v.x, v.y), max(v.z, v.w)) == kUnwritten, tries, sm));
  return tries < kMostTries;
}
// The same for a word of one thread. Out of line: a row of an operation before the last is nearly always there.
__device__ __noinline__ uint32_t wait_word(const void* p, Shared& sm, int phase) {
  uint32_t v = kUnwritten;
#pragma unroll 1
  for (int tries = 0; v == kUnwritten; ++tries) {
    if (tries == kMostTries || sm.abort_flag) {
      sm.abort_flag = sm.gave_up[phase] = 1;
      break;
    }
    v = load4(p);
  }
  return v;
}

// A barrier of the warps that compute.
__device__ __forceinline__ void sync_warps() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }

// ---------------------------------------------------------------------------------------------
// loads ahead
// ---------------------------------------------------------------------------------------------
// A bounded wait (each attempt suspends the thread for up to 20 us, 2^17 of them are some seconds).
[[nodiscard]] __device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int tries = 0; tries < (1 << 17); ++tries) {
    if (sm100::mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// Waits until fewer than `most` of the `issued` things are in use, or `all` that there were are done with. Bounded by the waits of the warps that use them, which raise the flag.
[[nodiscard]] __device__ __forceinline__ bool wait_slots(const int& done, int issued, int most, Shared& sm, int all = -1) {
  const uint32_t at = sm100::smem_u32(&done);
#pragma unroll 1
  for (int tries = 0; tries < (1 << 27); ++tries) {
    int n;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(n) : "r"(at) : "memory");
    if (issued - n < most || n == all) return true;
    if (sm.abort_flag) return false;
    __nanosleep(20);
  }
  sm.abort_flag = 1;
  return false;
}

// Brings the keys and values that an earlier launch has written, and that this CTA will read, to L2.
__device__ __forceinline__ void prefetch_keys(const ttb_chain_attention& o, int thread, int threads) {
  if (o.keys == TTB_CHAIN_KEYS_ROWS) return;
  const int H = o.heads * kHeadDim;
  const bool cached = o.keys == TTB_CHAIN_KEYS_CACHE;
  const int n = cached ? o.past : o.length;
#pragma unroll 1
  for (int unit = blockIdx.x; unit < o.rows * o.heads; unit += gridDim.x) {
    const int row = div_small(unit, o.heads), h = unit - row * o.heads;
#pragma unroll 1
    for (int j = thread; j < n; j += threads) {
      const long long at = cached ? cache_row(j, row, o.rows, H) + h * kHeadDim : ((long long)unit * o.length + j) * kHeadDim;
      prefetch_l2(static_cast<const __half*>(cached ? o.k_cache : o.k) + at);
      prefetch_l2(static_cast<const __half*>(cached ? o.v_cache : o.v) + at);
    }
  }
}

// Bytes of a unit's weights in the ring.
__device__ __host__ __forceinline__ int unit_bytes(int K) { return 8 * (K * 2 + kRowPad); }

// Where the weights of a group lie in the ring: one piece, at the ring's start where there is no room at its end. The warp that sends for them and those that
// read them go the same way.
struct RingAt {
  int start = 0, end = 0;  // the piece's offset; bytes taken so far, with those left out
  int next = 0;
  __device__ __forceinline__ void take(int bytes, int ring_bytes) {
    if (next + bytes > ring_bytes) {
      end += ring_bytes - next;
      next = 0;
    }
    start = next;
    next += bytes;
    end += bytes;
  }
};

// The warp that sends for what the operations need ahead of the arithmetic: in the order in which the CTA will read it, as far as the rings
// have room. What a group of units needs is counted on one barrier. Returns how many groups it has sent for. (By one of the computing warps, at the grid's
// barrier, it was on the way of every operation.)
__device__ __forceinline__ int feed(const ChainParams& prm, Shared& sm, uint32_t ring) {
  const int lane = threadIdx.x & 31;
  int groups = 0, params = 0;
  RingAt at;
#pragma unroll 1
  for (int op = 0; op < prm.n_ops; ++op) {
    const int4 todo = sm.todo[op];
    if (todo.y != TTB_CHAIN_LINEAR) {
      if (todo.y == TTB_CHAIN_ATTENTION) prefetch_keys(sm.ops[op].u.attention, lane, 32);
      continue;
    }
    const ttb_chain_linear& o = sm.ops[op].u.linear;
    const int group = todo.x & kGroupMask, lo = todo.z, hi = todo.w, K = o.K, N = o.N;
    int first = lo;
#pragma unroll 1
    do {
      const int nu = min(group, hi - first);
      const int before = at.end;
      at.take(nu * unit_bytes(K), prm.ring_bytes);
      if (!wait_slots(sm.groups_done, groups, kBars, sm) || !wait_slots(sm.bytes_done, at.end, prm.ring_bytes + 1, sm, before) ||
          (first == lo && !wait_slots(sm.params_done, params, kParamSlots, sm)))
        return groups;
      const uint32_t bar = sm100::smem_u32(&sm.full[groups % kBars]);
      const int rows = min(nu * 8, N - first * 8);
      if (lane == 0) {
        const uint32_t norm = first == lo && o.gamma ? (uint32_t)K * 2 : 0, bias = first == lo && o.bias ? (uint32_t)(hi - lo) * 16 : 0;
        const uint32_t dst = sm100::smem_u32(sm.params[params % kParamSlots]);
        sm100::mbar_expect_tx(bar, 2 * norm + bias + (uint32_t)(rows * K * 2));
        if (norm) {
          sm100::bulk_load_1d(dst, o.gamma, norm, bar);
          sm100::bulk_load_1d(dst + kNormed * 2, o.beta, norm, bar);
        }
        if (bias) sm100::bulk_load_1d(dst + kNormed * 4, static_cast<const char*>(o.bias) + (size_t)lo * 16, bias, bar);
      }
      __syncwarp();
      if (lane < rows)
        sm100::bulk_load_1d(ring + at.start + lane * (K * 2 + kRowPad), static_cast<const __half*>(o.W) + (long long)(first * 8 + lane) * K, (uint32_t)K * 2, bar);
      ++groups;
      first += group;
    } while (first < hi);
    ++params;
  }
  return groups;
}

// What a CTA has read of its rings, and which half of the sums' memory its next ones go to.
struct Read {
  int groups = 0, params = 0, red = 0;
  RingAt w;
};

// What every operation of a CTA works with.
struct Place {
  uint32_t ring, rows;  // shared memory of the weights and of the normalised rows
  float* red;           // two halves: of partial sums of a group of units, or of attention states; warps may still read the one before
  int ring_bytes;
};

// Tells the warp that sends for weights what all warps are done with; by one thread, behind a barrier of the warps that read it.
__device__ __forceinline__ void release(const Read& read, int params, Shared& sm) {
  if (threadIdx.x == kThreads - 32) {  // (of the warp with the least to do behind that barrier)
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(sm100::smem_u32(&sm.bytes_done)), "r"(read.w.end) : "memory");
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(sm100::smem_u32(&sm.params_done)), "r"(params) : "memory");
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(sm100::smem_u32(&sm.groups_done)), "r"(read.groups) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// products
// ---------------------------------------------------------------------------------------------
// The layout of a product: RT tiles of eight rows. On mma.sync m16n8k16 two units of eight output columns are the m and a tile of rows is the n. The
// warps are RG groups of TW tiles, and in a group share K. A chunk is 32 of K: thread t of a quad holds 8 of them, in 16 bytes, for
// column g of each unit and row g of each tile. Chunk c belongs to share c % KW; a warp works on CPW of its chunks at a time, of which K is
// a whole number (EXACT) or not.
template <int RT, int CPW> struct Layout {
  static constexpr int RG = RT <= 4 ? 1 : RT / 2, TW = RT / RG, KW = kWarps / RG;
  static constexpr int kStep = 32 * KW * CPW;                               // of K, that all warps work on at a time
  // steps of K whose rows (up to 64 registers) are held at a time
  static constexpr int kMost = (RT == 8 && CPW == 2 ? 12 : 16) / (CPW * TW), kHeld = kMost >= 4 ? (CPW > 3 ? 3 : 4) : kMost > 1 ? kMost : 1;
  static constexpr int kItems = (kGroup * RT + kWarps - 1) / kWarps;        // (unit, tile) pairs that a warp finishes
  static constexpr int kRed = kGroup * RT * KW * 64;                        // sums: [unit][tile][share][column][row]
  // Two places for the sums, so that a warp need not wait for those that still read the ones before; with many tiles, one, and a barrier.
  static constexpr int kPlaces = RT <= 3 ? 2 : 1;
  static_assert(RG * TW == RT && kHeld >= 1 && kRed >= kWarps * (kHeadDim + 2));
};

// Two fp32 numbers that one instruction works on.
struct Two {
  unsigned long long v;
  __device__ __forceinline__ Two() {}
  __device__ __forceinline__ Two(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ float2 get() const {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
  }
};
__device__ __forceinline__ Two operator+(Two a, Two b) {
  Two r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Two operator*(Two a, Two b) {
  Two r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) {
  Two r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ void unpack2(const uint4& q, Two (&f)[4]) {
  const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __half22float2(h[i]);
    f[i] = Two(v.x, v.y);
  }
}

// Layer norm of the operation's rows into shared memory (64 bytes past a multiple of 128 between rows, as in the ring): rows warp, warp + 8,
// ... by a warp, R of them at a time.
template <int R, int kIters>  // kIters: 16-byte pieces of a row per lane
__device__ __forceinline__ bool normalise(const ttb_chain_linear& o, bool flows, Shared& sm, uint32_t a_smem, uint32_t params) {
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, K = o.K, M = o.M;
  if (warp >= M) return true;
  const uint32_t gamma = params + lane * 16;
  const float inv_k = __fdividef(1.f, (float)K), eps = o.eps;
  int tries = 0;
  bool there_yet = true, there[kIters];
#pragma unroll
  for (int i = 0; i < kIters; ++i) there[i] = i * 256 + lane * 8 < K;
  Two ga[kIters][4], be[kIters][4];
  if (R == 1)
#pragma unroll
    for (int i = 0; i < kIters; ++i) {
      unpack2(lds128(gamma + i * 512), ga[i]);
      unpack2(lds128(gamma + kNormed * 2 + i * 512), be[i]);
    }
#pragma unroll 1
  for (int row0 = warp; row0 < M; row0 += kWarps * R) {
    const __half* src = static_cast<const __half*>(o.A) + (long long)row0 * o.lda + lane * 8;
    uint4 x[R][kIters];
    uint32_t top;
    if (flows && M > 2 && row0 == warp) there_yet = wait_ahead(src, sm);
    do {
      top = 0;
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < kIters; ++i) {  // (lanes beyond the row hold zeros)
          x[r][i] = make_uint4(0, 0, 0, 0);
          if ((R == 1 || row0 + r * kWarps < M) && there[i]) x[r][i] = load16(src + (long long)r * kWarps * o.lda + i * 256);
        }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < kIters; ++i) look(top, x[r][i]);
    } while (flows && again(top == kUnwritten, tries, sm));
    Two f[R][kIters][4];
    float sum[R], sq[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      Two t(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kIters; ++i) {
        unpack2(x[r][i], f[r][i]);
        t = t + ((f[r][i][0] + f[r][i][1]) + (f[r][i][2] + f[r][i][3]));
      }
      sum[r] = t.get().x + t.get().y;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], d);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float mean = sum[r] * inv_k;
      Two t(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kIters; ++i) {
        const Two minus(there[i] ? -mean : 0.f, there[i] ? -mean : 0.f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          f[r][i][e] = f[r][i][e] + minus;
          t = fma2(f[r][i][e], f[r][i][e], t);
        }
      }
      sq[r] = t.get().x + t.get().y;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) sq[r] += __shfl_xor_sync(0xffffffffu, sq[r], d);
#pragma unroll
    for (int r = 0; r < R; ++r) sq[r] = rsqrtf(sq[r] * inv_k + eps);
    const uint32_t to = a_smem + row0 * (K * 2 + kRowPad) + lane * 16;
#pragma unroll
    for (int i = 0; i < kIters; ++i) {
      if (R > 1) {
        unpack2(lds128(gamma + i * 512), ga[i]);
        unpack2(lds128(gamma + kNormed * 2 + i * 512), be[i]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const Two scale(sq[r], sq[r]);
        float y[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = fma2(f[r][i][e] * scale, ga[i][e], be[i][e]).get();
          y[2 * e] = v.x;
          y[2 * e + 1] = v.y;
        }
        const uint4 q = pack(y);
        if ((R == 1 || row0 + r * kWarps < M) && there[i])
          asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + r * kWarps * (K * 2 + kRowPad) + i * 512), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
        x[r][i] = q;
      }
    }
    if (o.normed)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (const int row = row0 + r * kWarps; row < M && chain::writes_row(row, (int)blockIdx.x))
#pragma unroll
          for (int i = 0; i < kIters; ++i)
            if (there[i]) store16(static_cast<__half*>(o.normed) + (long long)row * K + i * 256 + lane * 8, x[r][i]);
  }
  return there_yet && tries < kMostTries;
}

// Steps of K one behind the other, as far as there are any: a step that is not there is jumped over together with those behind it.
template <int S> struct Step {
  static constexpr int value = S;
};
template <int S, int N, typename F, typename G> __device__ __forceinline__ void steps(const F& there, const G& body) {
  body(Step<S>());
  if constexpr (S + 1 < N) {
    if (there(S + 1)) steps<S + 1, N>(there, body);
  }
}

__device__ __noinline__ void store_halves(__half* out, float2 y, int columns) {
  if (columns > 0) out[0] = __float2half_rn(y.x);
  if (columns > 1) out[1] = __float2half_rn(y.y);
}

// A product. What does not depend on the operations before comes first, while their results are on their way. False: a wait has run out.
template <int RT, int CPW, bool EXACT>
__device__ __forceinline__ bool linear(const ttb_chain_linear& o, const int4& todo, const Place& at, Shared& sm, Read& read) {
  using L = Layout<RT, CPW>;
  constexpr int KW = L::KW, TW = L::TW, kNext = KW * 64;  // bytes from one of a warp's chunks to the next
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int how = todo.x, lo = todo.z, hi = todo.w, group = how & kGroupMask;
  const int rg = warp % L::RG, share = warp / L::RG, M = o.M, K = o.K, N = o.N, act = o.act, pitch = K * 2 + kRowPad;
  const uint32_t lane_at = g * pitch + share * 64 + t * 16;
  const uint32_t params = sm100::smem_u32(sm.params[read.params % kParamSlots]);
  const uint32_t bias_at = o.bias ? params + kNormed * 4 : 0;
  ++read.params;
  int u0 = lo;
  bool ok = true;
#pragma unroll 1
  do {
    const int nu = min(group, hi - u0);
    read.w.take(nu * 8 * pitch, at.ring_bytes);
    ok = wait(sm100::smem_u32(&sm.full[read.groups % kBars]), (read.groups / kBars) & 1, &sm.abort_flag) && ok;
    ++read.groups;
    // what the epilogue needs: of (unit, tile) warp, warp + 8, ..: two columns of a row a thread
    const __half* res_at[L::kItems];
    __half* out_at[L::kItems];
    uint32_t res[L::kItems], bias[L::kItems];
    int columns[L::kItems];  // of the two that are there
#pragma unroll
    for (int it = 0; it < L::kItems; ++it) {
      const int u = (warp + it * kWarps) / RT, row = ((warp + it * kWarps) % RT) * 8 + t * 2 + (g & 1), col = (u0 + u) * 8 + (g & 6);
      columns[it] = u < nu && row < M ? N - col : 0;
      res_at[it] = static_cast<const __half*>(o.residual) + (long long)row * o.ldr + col;
      out_at[it] = static_cast<__half*>(o.out) + (long long)row * o.ldo + col;
      res[it] = bias[it] = 0;
      if (o.residual && columns[it] > 0) res[it] = load4(res_at[it]);
      if (bias_at && columns[it] > 0) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(bias[it]) : "r"(bias_at + (col - lo * 8) * 2));
    }
    const bool pairs = ((o.ldo | N) & 1) == 0 && (reinterpret_cast<uintptr_t>(o.out) & 3) == 0;
    float* red = at.red + (L::kPlaces == 2 ? read.red * L::kRed : 0);
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += L::kHeld * L::kStep) {
      // step `s` of K, and chunk i of it, are there
      auto step = [&](int s) { return k0 + s * L::kStep < K; };
      auto chunk = [&](int s, int i) { return EXACT || k0 + s * L::kStep + (i * KW + share) * 32 < K; };
      const uint32_t w_at = at.ring + read.w.start + lane_at + k0 * 2;
      // Weights of two units in a step. (The sums of a second unit that is not there are not read.)
      auto weights = [&](int s, int unit, uint4 (&a)[CPW], uint4 (&b)[CPW]) {
        const uint32_t first = w_at + unit * 8 * pitch, second = first + 8 * pitch;
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
          b[i] = make_uint4(0, 0, 0, 0);
          if (!EXACT) a[i] = b[i];
          if (chunk(s, i)) {
            a[i] = lds128(first + (s * CPW + i) * kNext);
            if (unit + 1 < nu) b[i] = lds128(second + (s * CPW + i) * kNext);
          }
        }
      };
      if ((how & kNorm) && u0 == lo && k0 == 0) {
        ok = normalise<(RT > 1 ? 2 : 1), (EXACT && RT <= 4 ? CPW : 4)>(o, how & kRowsFlow, sm, at.rows, params) && ok;
        sync_warps();
      }
      uint4 x[L::kHeld * CPW][TW];
      if (how & kNorm) {  // (rows that are not there leave sums that nobody reads)
        const uint32_t from = at.rows + rg * TW * 8 * pitch + lane_at + k0 * 2;
        steps<0, L::kHeld>(step, [&](auto at_step) {
          constexpr int s = decltype(at_step)::value;
#pragma unroll
          for (int i = 0; i < CPW; ++i)
#pragma unroll
            for (int r = 0; r < TW; ++r) {
              if (!EXACT) x[s * CPW + i][r] = make_uint4(0, 0, 0, 0);
              if (chunk(s, i)) x[s * CPW + i][r] = lds128(from + r * 8 * pitch + (s * CPW + i) * kNext);
            }
        });
      } else {
        const char* from[TW];  // (again the last row for those that are not there)
#pragma unroll
        for (int r = 0; r < TW; ++r) from[r] = static_cast<const char*>(o.A) + (long long)min((rg * TW + r) * 8 + g, M - 1) * o.lda * 2 + share * 64 + t * 16 + k0 * 2;
        uint32_t top;
        int tries = 0;
        do {
          top = 0;
          steps<0, L::kHeld>(step, [&](auto at_step) {
            constexpr int s = decltype(at_step)::value;
#pragma unroll
            for (int i = 0; i < CPW; ++i)
#pragma unroll
              for (int r = 0; r < TW; ++r) {
                if (!EXACT) x[s * CPW + i][r] = make_uint4(0, 0, 0, 0);
                if (chunk(s, i)) x[s * CPW + i][r] = load16(from[r] + (s * CPW + i) * kNext);
              }
          });
          steps<0, L::kHeld>(step, [&](auto at_step) {
            constexpr int s = decltype(at_step)::value;
#pragma unroll
            for (int i = 0; i < CPW; ++i)
#pragma unroll
              for (int r = 0; r < TW; ++r) look(top, x[s * CPW + i][r]);
          });
        } while ((how & kRowsFlow) && again(top == kUnwritten, tries, sm));
        ok = ok && tries < kMostTries;
      }
      if (L::kPlaces == 1 && k0 == 0 && !((how & kNorm) && u0 == lo)) sync_warps();
#pragma unroll 1
      for (int unit = 0; unit < nu; unit += 2) {
        constexpr int kChains = TW == 1 ? 2 : 1;  // of sums: an mma waits 20 cycles for the one before it
        float acc[kChains][TW][4];
#pragma unroll
        for (int c = 0; c < kChains; ++c)
#pragma unroll
          for (int r = 0; r < TW; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[c][r][e] = 0.f;
        steps<0, L::kHeld>(step, [&](auto at_step) {
          constexpr int s = decltype(at_step)::value;
          uint4 a[CPW], b[CPW];
          weights(s, unit, a, b);
#pragma unroll
          for (int i = 0; i < CPW; ++i) {
#pragma unroll
            for (int r = 0; r < TW; ++r) mma16816(acc[0][r], a[i].x, b[i].x, a[i].y, b[i].y, x[s * CPW + i][r].x, x[s * CPW + i][r].y);
#pragma unroll
            for (int r = 0; r < TW; ++r) mma16816(acc[kChains - 1][r], a[i].z, b[i].z, a[i].w, b[i].w, x[s * CPW + i][r].z, x[s * CPW + i][r].w);
          }
        });
#pragma unroll
        for (int r = 0; r < TW; ++r) {
          if (kChains == 2)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[0][r][e] += acc[kChains - 1][r][e];
          float2* dst = reinterpret_cast<float2*>(red + ((unit * RT + rg * TW + r) * KW + share) * 64) + lane;
          if (k0 > 0) {  // the sums of the steps before, by this thread
            const float2 before = dst[0], other = dst[RT * KW * 32];
            acc[0][r][0] += before.x;
            acc[0][r][1] += before.y;
            acc[0][r][2] += other.x;
            acc[0][r][3] += other.y;
          }
          dst[0] = make_float2(acc[0][r][0], acc[0][r][1]);
          dst[RT * KW * 32] = make_float2(acc[0][r][2], acc[0][r][3]);
        }
      }
    }
    if (!ok) sm.gave_up[read.red] = 1;
    sync_warps();
    const int stop = sm.gave_up[read.red];
    read.red ^= 1;
    release(read, read.params - (u0 + group < hi ? 1 : 0), sm);
#pragma unroll
    for (int it = 0; it < L::kItems; ++it) {
      const int tile = warp + it * kWarps;
      if (tile < nu * RT) {  // (a whole warp)
        const float* src = red + tile * KW * 64 + lane * 2;
        float2 v[2] = {};
#pragma unroll
        for (int j = 0; j < KW; ++j) {
          const float2 y = *reinterpret_cast<const float2*>(src + j * 64);
          v[j & 1].x += y.x;
          v[j & 1].y += y.y;
        }
        v[0].x += v[1].x;
        v[0].y += v[1].y;
        // column g, rows 2 t and 2 t + 1 -> columns g and g + 1 of one of the rows
        const float other = __shfl_xor_sync(0xffffffffu, (g & 1) ? v[0].x : v[0].y, 4);
        const float2 add = __half22float2(*reinterpret_cast<const __half2*>(&bias[it]));
        float2 y = make_float2(((g & 1) ? other : v[0].x) + add.x, ((g & 1) ? v[0].y : other) + add.y);
        if (act == TTB_CHAIN_ACT_GELU) {
          y.x = gelu16(y.x);
          y.y = gelu16(y.y);
        } else if (act == TTB_CHAIN_ACT_RELU) {
          y.x = fmaxf(y.x, 0.f);
          y.y = fmaxf(y.y, 0.f);
        }
        if ((how & kResidualFlows) && res[it] == kUnwritten) res[it] = wait_word(res_at[it], sm, read.red);
        const float2 before = __half22float2(*reinterpret_cast<const __half2*>(&res[it]));
        y.x += before.x;
        y.y += before.y;
        const __half2 q = __floats2half2_rn(y.x, y.y);
        if (pairs) {
          if (columns[it] > 0) store4(out_at[it], *reinterpret_cast<const uint32_t*>(&q));
        } else if (columns[it] > 0) {
          store_halves(out_at[it], y, columns[it]);
        }
      }
    }
    if (stop) return false;
    u0 += group;
  } while (u0 < hi);
  return true;
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------
// (row, head) pairs go round the CTAs; a CTA's warps are shared out among as many of its pairs as they serve at once, each taking
// every W-th page of 16 keys, the next page on its way while one is worked on. A new token over a cache is a page of its own. The scores
// run on mma.sync, keys as its m and the query as every one of its columns, so that all lanes of a quad have those of keys g and g + 8; probabilities and
// values stay in fp32: eight lanes a value, four values at a time.
__device__ __forceinline__ bool attention(const ttb_chain_attention& o, const int4& todo, float* sums, int half, Shared& sm, Read& read) {
  constexpr int kState = kHeadDim + 2;
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, kg = lane >> 3, sub = lane & 7;
  const int heads = o.heads, H = heads * kHeadDim, keys = o.keys, length = o.length, rows = o.rows;
  const bool flows = todo.x & kRowsFlow;
  const int mine = todo.z, W = 1 << todo.w, S = kWarps >> todo.w, place = warp >> todo.w, wi = warp & (W - 1);  // warps a pair, pairs at once
#pragma unroll 1
  for (int first = 0; first < mine; first += S) {
    const bool active = first + place < mine;
    const int unit = active ? (first + place) * (int)gridDim.x + (int)blockIdx.x : 0;
    const int row = div_small(unit, heads), h = unit - row * heads;
    const __half* qrow = static_cast<const __half*>(o.q) + (long long)row * o.ldq + h * kHeadDim;
    // key j of the row: k0 + (j / 16) * page + (j % 16) * pitch
    const __half *k0 = static_cast<const __half*>(o.k), *v0 = static_cast<const __half*>(o.v);
    long long at = (long long)unit * length * kHeadDim;
    int seq = row, n = length, pitch = kHeadDim, last = -1;  // last: the page of the new token
    long long page = 16 * kHeadDim;
    if (keys == TTB_CHAIN_KEYS_CACHE) {
      k0 = static_cast<const __half*>(o.k_cache);
      v0 = static_cast<const __half*>(o.v_cache);
      at = (long long)row * 16 * H + h * kHeadDim;
      n = o.past;
      pitch = H;
      page = 16ll * rows * H;
      last = (n + 15) >> 4;
    } else if (keys == TTB_CHAIN_KEYS_ROWS) {
      seq = div_small(row, length);
      k0 = static_cast<const __half*>(o.q) + H;
      v0 = k0 + H;
      pitch = o.ldq;
      at = (long long)(seq * length) * pitch + h * kHeadDim;
      n = o.causal ? row - seq * length + 1 : length;
      page = 16ll * pitch;
    }
    k0 += at;
    v0 += at;
    const int pages = last >= 0 ? last + 1 : (n + 15) >> 4;
    const float* mask = o.mask ? o.mask + (long long)seq * o.mask_pitch : nullptr;
    float* scores = o.probs && h == 0 ? o.scores + (long long)row * length : nullptr;
    const float scale = o.scale * kLog2e;
    float m = -INFINITY, l = 0.f;
    Two acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = Two(0.f, 0.f);
    int tries = 0;
    if (active) {
      uint4 q[2], kn[4], vn[4];  // kn: keys g and g + 8, t-th eights of both halves; vn: values kg, kg + 4, .., eight dimensions
#pragma unroll 1
      for (int p = wi - W; p < pages; p += W) {
        uint4 kr[4], vr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          kr[i] = kn[i];
          vr[i] = vn[i];
        }
        if (p + W < pages) {  // the next page is on its way while this one (there is none at first) is worked on
          const bool fresh = p + W == last, wait = flows && (fresh || keys == TTB_CHAIN_KEYS_ROWS);
          const int there = fresh ? 1 : min(16, n - (p + W) * 16);
          const __half* kp = (fresh ? qrow + H : k0 + (p + W) * page) + t * 8;
          const __half* vp = (fresh ? qrow + 2 * H : v0 + (p + W) * page) + sub * 8;
          uint32_t top;
          do {
#pragma unroll
            for (int i = 0; i < 4; ++i) kn[i] = load16(kp + min(g + (i & 1) * 8, there - 1) * pitch + (i >> 1) * 32);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              vn[u] = make_uint4(0, 0, 0, 0);
              if (kg + u * 4 < there) vn[u] = load16(vp + (kg + u * 4) * pitch);
            }
            if (!wait) break;
            top = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              look(top, kn[i]);
              look(top, vn[i]);
            }
          } while (again(top == kUnwritten, tries, sm));
        }
        if (p < 0) {  // (cached keys are on their way before the query is there)
          uint32_t top;
          do {
            top = 0;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              q[i] = load16(qrow + t * 8 + i * 32);
              look(top, q[i]);
            }
          } while (flows && again(top == kUnwritten, tries, sm));
          continue;
        }
        const int j0 = p == last ? n : p * 16, there = p == last ? 1 : min(16, n - j0);
        float sc[4] = {};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma16816(sc, kr[2 * i].x, kr[2 * i + 1].x, kr[2 * i].y, kr[2 * i + 1].y, q[i].x, q[i].y);
          mma16816(sc, kr[2 * i].z, kr[2 * i + 1].z, kr[2 * i].w, kr[2 * i + 1].w, q[i].z, q[i].w);
        }
        float pr[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          pr[i] = -INFINITY;
          if (g + i * 8 < there) {
            pr[i] = sc[2 * i] * scale;
            if (mask) pr[i] += mask[j0 + g + i * 8] * kLog2e;
            if (scores && t == 0) scores[j0 + g + i * 8] = pr[i];
          }
        }
        float top = fmaxf(pr[0], pr[1]);
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
        top = fmaxf(top, m);
        const float base = top == -INFINITY ? 0.f : top, keep = ex2f(m - base);
        m = top;
        pr[0] = ex2f(pr[0] - base);
        pr[1] = ex2f(pr[1] - base);
        l = l * keep + (pr[0] + pr[1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] = acc[e] * Two(keep, keep);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float pu = __shfl_sync(0xffffffffu, pr[u >> 1], (kg + (u & 1) * 4) * 4);
          Two f[4];
          unpack2(vr[u], f);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] = fma2(f[e], Two(pu, pu), acc[e]);
        }
      }
#pragma unroll
      for (int d = 4; d < 32; d <<= 1) l += __shfl_xor_sync(0xffffffffu, l, d);
    }
    float* red = sums + read.red * half;
    if (half == 0) sync_warps();
    float* state = red + warp * kState;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 v = acc[e].get();
#pragma unroll
      for (int d = 8; d < 32; d <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
      }
      if (lane < 8) *reinterpret_cast<float2*>(state + 2 + lane * 8 + e * 2) = v;
    }
    if (lane == 0) *reinterpret_cast<float2*>(state) = make_float2(m, l);
    if (tries == kMostTries) sm.gave_up[read.red] = 1;
    sync_warps();
    if (sm.gave_up[read.red]) return false;
    read.red ^= 1;
    if (active && (wi == 0 || scores)) {
      const float* st = red + place * W * kState;
      const int used = min(W, pages);  // warps that have seen a key
      float2 theirs[kWarps], part[kWarps];
#pragma unroll
      for (int i = 0; i < kWarps; ++i) {
        theirs[i] = make_float2(-INFINITY, 0.f);
        part[i] = make_float2(0.f, 0.f);
        if (i < used) {
          theirs[i] = *reinterpret_cast<const float2*>(st + i * kState);
          part[i] = *reinterpret_cast<const float2*>(st + i * kState + 2 + lane * 2);
        }
      }
      float top = theirs[0].x, sum = 0.f;
#pragma unroll
      for (int i = 1; i < kWarps; ++i) top = fmaxf(top, theirs[i].x);
      const float base = top == -INFINITY ? 0.f : top;
      float2 v = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kWarps; ++i) {
        const float f = ex2f(theirs[i].x - base);
        sum = fmaf(theirs[i].y, f, sum);
        v.x = fmaf(f, part[i].x, v.x);
        v.y = fmaf(f, part[i].y, v.y);
      }
      const float inv = 1.f / sum;
      if (wi == 0) {
        const __half2 y = __floats2half2_rn(v.x * inv, v.y * inv);
        store4(static_cast<__half*>(o.out) + (long long)row * o.ldo + h * kHeadDim + lane * 2, *reinterpret_cast<const uint32_t*>(&y));
      }
      if (scores)
#pragma unroll 1
        for (int j = wi * 32 + lane; j < n; j += W * 32)
          static_cast<__half*>(o.probs)[(long long)row * length + j] = __float2half_rn(ex2f(scores[j] - base) * inv);
    }
    // the new token's key and value are filed by the pair's last warp, behind what others wait for (pairs of the same row write its other heads)
    if (active && wi == W - 1 && o.k_cache && keys != TTB_CHAIN_KEYS_MEMORY) {
      const int sequences = keys == TTB_CHAIN_KEYS_CACHE ? rows : div_small(rows, length), token = keys == TTB_CHAIN_KEYS_CACHE ? n : row - seq * length;
      uint4 newest;
      tries = 0;
      do newest = load16(qrow + (lane & 8 ? 2 * H : H) + sub * 8);
      while (flows && again(max(max(newest.x, newest.y), max(newest.z, newest.w)) == kUnwritten, tries, sm));
      if (tries == kMostTries) sm.gave_up[read.red] = 1;
      if (lane < 16)
        *reinterpret_cast<uint4*>(static_cast<__half*>(lane < 8 ? o.k_cache : o.v_cache) + cache_row(token, seq, sequences, H) + h * kHeadDim + sub * 8) = newest;
    }
  }
  return true;
}

// ---------------------------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------------------------
template <int RT, int CPW, bool EXACT>
__global__ void __launch_bounds__(kBlock, 1) chain_kernel(const __grid_constant__ ChainParams prm) {
  using L = Layout<RT, CPW>;
  extern __shared__ __align__(128) uint8_t smem[];
  Shared& sm = *reinterpret_cast<Shared*>(smem);
  Place at;
  at.red = reinterpret_cast<float*>(smem + kSharedBytes);
  at.rows = sm100::smem_u32(smem) + kSharedBytes + prm.sums_bytes;
  at.ring = at.rows + prm.a_bytes;
  at.ring_bytes = prm.ring_bytes;
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int i = 0; i < kBars; ++i) sm100::mbar_init(sm100::smem_u32(&sm.full[i]), 1);
    sm.bytes_done = sm.params_done = sm.groups_done = 0;
    sm.abort_flag = sm.gave_up[0] = sm.gave_up[1] = 0;
    sm100::mbar_init_fence();
  }
  {
    const uint32_t* from = reinterpret_cast<const uint32_t*>(prm.ops);
    asm volatile("" : "+l"(from));  // as memory: a constant load with an address for each thread would go one thread after the other
    uint32_t* to = reinterpret_cast<uint32_t*>(sm.ops);
#pragma unroll 1
    for (int i = tid; i < prm.n_ops * kOpWords; i += kBlock) to[i] = from[i];
  }
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < prm.n_ops; i += kBlock) {
    const Todo d(sm.ops[i]);
    sm.todo[i] = make_int4(d.how, d.kind, d.lo, d.hi);
  }
  __syncthreads();
  if (tid >= kThreads) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFeedRegisters));
    if (tid >= kThreads + 32) return;
    const int groups = feed(prm, sm, at.ring);
    // every copy lands before the CTA's shared memory goes, also where a wait has run out
#pragma unroll 1
    for (int i = max(0, groups - kBars); i < groups; ++i) {
      const uint32_t bar = sm100::smem_u32(&sm.full[i % kBars]);
      const long long t0 = clock64();
      while (!sm100::mbar_try_wait(bar, (i / kBars) & 1) && clock64() - t0 < sm100::kWaitCycles) {
      }
    }
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kComputeRegisters));
  Read read;
#pragma unroll 1
  for (int i = 0; i < prm.n_ops; ++i) {
    const int4 todo = sm.todo[i];
    bool ok = true;
    if (todo.x & kBarrier) {  // everything that this CTA has written becomes visible to the others, and theirs to it
      sync_warps();
      if (tid == 0) {
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(prm.counter) : "memory");
        const int target = (int)gridDim.x * i;
        const long long t0 = clock64();
        while (sm100::ld_acquire_gpu(prm.counter) < target) {
          if (sm.abort_flag) break;
          if (clock64() - t0 > sm100::kWaitCycles) sm.abort_flag = 1;
        }
        if (sm.abort_flag) sm.gave_up[read.red] = 1;
      }
      sync_warps();
      ok = !sm.gave_up[read.red];
    }
    if (!ok) break;
    if (todo.y == TTB_CHAIN_LINEAR) ok = linear<RT, CPW, EXACT>(sm.ops[i].u.linear, todo, at, sm, read);
    else if (todo.y == TTB_CHAIN_ATTENTION) ok = attention(sm.ops[i].u.attention, todo, at.red, L::kPlaces == 2 ? L::kRed : 0, sm, read);
    if (!ok) break;
  }
  if (sm.abort_flag) atomicExch(prm.status, (int)TTB_ERR_DEVICE_WAIT);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// Which kernel runs a chain: tiles of eight rows and chunks of K a warp.
int row_tiles(int rows) { return rows <= 8 ? 1 : rows <= 16 ? 2 : rows <= 24 ? 3 : rows <= 32 ? 4 : 8; }
int share_of(int tiles) { return tiles <= 4 ? kWarps : 2 * kWarps / tiles; }  // Layout::KW
// Layout::kPlaces * kRed words; as many as `group` units need where there is one place.
int sums_of(int tiles, int group) { return (tiles <= 3 ? 2 * kGroup : std::max(group, 2)) * tiles * share_of(tiles) * 64 * 4; }

// Whether a chain takes a product so deep: the depth is a whole number of parts of 256 to 1024 columns, in 64s.
bool depth_fits(int64_t K) {
  if (K <= 0 || K > 8192 || K % 64 != 0) return false;
  for (int64_t parts = (K + 1023) / 1024; K / parts >= 256; ++parts)
    if (K % parts == 0 && (K / parts) % 64 == 0) return true;
  return false;
}

// How a chain of products so deep runs: the chunks of K that a warp works on at a time (Layout::CPW), and whether every product is a whole number of them for
// all warps (EXACT); chunks = 0: the ring does not hold a unit of the deepest. The rest of the shared memory is the ring.
struct Plan {
  int tiles = 0, chunks = 0, group = 0, ring_bytes = 0, a_bytes = 0;
  bool exact = false;
};
Plan plan_of_tiles(int tiles, const std::vector<int64_t>& depths, int normed_k) {
  Plan p;
  p.tiles = tiles;
  p.a_bytes = normed_k ? tiles * 8 * (normed_k * 2 + kRowPad) : 0;
  int64_t deepest = 0;
  for (int64_t K : depths) deepest = std::max(deepest, K);
  for (p.group = kGroup; p.group > 0; p.group -= 2) {  // sums of fewer units at a time, where the ring would have no room for a unit otherwise
    p.ring_bytes = kSmemLimit - kSharedBytes - sums_of(tiles, p.group) - p.a_bytes;
    if (unit_bytes((int)deepest) <= p.ring_bytes) break;
  }
  if (p.group <= 0) return p;
  for (int chunks = 4; chunks >= 2 && !p.exact; --chunks) {
    p.chunks = chunks;
    p.exact = tiles > 4 || normed_k <= 256 * chunks;  // (rows are normalised in pieces of 256)
    for (int64_t K : depths) p.exact = p.exact && K % (32 * share_of(tiles) * chunks) == 0;
  }
  if (!p.exact) p.chunks = 4;
  return p;
}
// The kernel for so many rows, or one for more that leaves the ring more room.
Plan plan_of(int rows, const std::vector<int64_t>& depths, int normed_k) {
  const int tiles = row_tiles(rows);
  Plan p = plan_of_tiles(tiles, depths, normed_k);
  if (!p.chunks && tiles < 4) p = plan_of_tiles(4, depths, normed_k);
  if (!p.chunks && tiles < 8) p = plan_of_tiles(8, depths, normed_k);
  return p;
}

template <int RT, int CPW, bool EXACT> cudaError_t launch(ttb_ctx* ctx, const ChainParams& prm) {
  const int smem = kSharedBytes + prm.sums_bytes + prm.a_bytes + prm.ring_bytes;
  cudaError_t e = cudaFuncSetAttribute(chain_kernel<RT, CPW, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctx->sm_count);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;  // the whole grid is resident, or the launch fails
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, chain_kernel<RT, CPW, EXACT>, prm);
}
template <int RT> cudaError_t launch(ttb_ctx* ctx, const Plan& plan, const ChainParams& prm) {
  if (!plan.exact) return launch<RT, 4, false>(ctx, prm);
  return plan.chunks == 2 ? launch<RT, 2, true>(ctx, prm) : plan.chunks == 3 ? launch<RT, 3, true>(ctx, prm) : launch<RT, 4, true>(ctx, prm);
}

}  // namespace

extern "C" int64_t ttb_chain_rows(int64_t hidden, int64_t inner) {
  if (hidden > kNormed || (hidden != 0 && !depth_fits(hidden)) || !depth_fits(inner)) return 0;
  for (int rows : {64, 32, 24, 16, 8})
    if (plan_of(rows, {hidden, inner}, (int)hidden).chunks) return rows;
  return 0;
}
static_assert(TTB_CHAIN_MAX_ROWS == 64, "the most rows of the widest kernel");

namespace {

// `flow`: the memory through which the operations hand their results on, none: they meet at barriers, counted in `counter`.
int chain_forward(ttb_ctx* ctx, int dtype, const ttb_chain_op* ops, int n_ops, int* counter, void* flow, size_t flow_bytes) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, dtype == TTB_F16, "chain_forward: dtype must be F16");
  TTB_REQUIRE(ctx, ops && (counter || flow) && n_ops > 0 && n_ops <= TTB_CHAIN_MAX_OPS, "chain_forward: 1 to %d operations", TTB_CHAIN_MAX_OPS);
  TTB_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(flow) & 15) == 0 && flow_bytes % 4 == 0, "chain_forward: the flow starts on 16 bytes and is of whole words");
  const uintptr_t flow0 = reinterpret_cast<uintptr_t>(flow), flow1 = flow0 + flow_bytes;
  auto flows = [&](const void* p) { return reinterpret_cast<uintptr_t>(p) - flow0 < flow1 - flow0; };
  // Every word of the flow is written once: the results lie in it one behind the other.
  uintptr_t filled = flow0;
  auto fill = [&](const void* p, int64_t rows, int64_t pitch, int64_t columns) {
    if (!p || !flows(p)) return true;
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    if (at < filled || columns % 2 != 0 || pitch % 2 != 0 || (at & 3) != 0) return false;
    filled = at + ((rows - 1) * pitch + columns) * 2;
    return filled <= flow1;
  };
  auto aligned = [](std::initializer_list<const void*> ps) {
    uintptr_t x = 0;
    for (const void* p : ps) x |= reinterpret_cast<uintptr_t>(p);
    return (x & 15) == 0;
  };
  ChainParams prm{};
  int rows = 0, normed_k = 0;
  std::vector<int64_t> depths;
  for (int i = 0; i < n_ops; ++i) {
    prm.ops[i] = ops[i];
    if (ops[i].kind == TTB_CHAIN_LINEAR) {
      const ttb_chain_linear& o = ops[i].u.linear;
      TTB_REQUIRE(ctx, o.M > 0 && o.M <= TTB_CHAIN_MAX_ROWS && o.N >= 0 && o.N <= (1 << 24) && depth_fits(o.K), "chain_forward: operation %d: bad shape %d x %d x %d", i,
                  o.M, o.N, o.K);
      TTB_REQUIRE(ctx, o.A && o.lda >= o.K && o.lda % 8 == 0 && (o.N == 0 || (o.W && o.out && o.ldo >= o.N)) && (!o.residual || (o.ldr >= o.N && o.ldr % 2 == 0)),
                  "chain_forward: operation %d: missing operand or bad pitch", i);
      TTB_REQUIRE(ctx, aligned({o.A, o.W, o.gamma, o.beta, o.bias, o.normed}) && (reinterpret_cast<uintptr_t>(o.residual) & 3) == 0 &&
                  (reinterpret_cast<uintptr_t>(o.out) & 1) == 0, "chain_forward: operation %d: misaligned operand", i);
      TTB_REQUIRE(ctx, !o.gamma || (o.beta && o.K <= kNormed), "chain_forward: operation %d: a layer norm takes at most %d columns and both of its weights", i, kNormed);
      TTB_REQUIRE(ctx, o.N > 0 || (o.gamma && o.normed), "chain_forward: operation %d does nothing", i);
      TTB_REQUIRE(ctx, !o.normed || chain::rows_have_writers(o.M, ctx->sm_count), "chain_forward: operation %d: more rows than SMs", i);
      TTB_REQUIRE(ctx, (!o.bias && !o.residual) || o.N % 8 == 0, "chain_forward: operation %d: a bias or residual needs a width that is a multiple of 8", i);
      TTB_REQUIRE(ctx, !o.bias || o.N <= chain::bias_columns(ctx->sm_count), "chain_forward: operation %d: too wide for a bias", i);
      TTB_REQUIRE(ctx, o.act >= 0 && o.act <= TTB_CHAIN_ACT_RELU, "chain_forward: operation %d: unknown activation", i);
      TTB_REQUIRE(ctx, fill(o.normed, o.M, o.K, o.K) && fill(o.out, o.M, o.ldo, o.N), "chain_forward: operation %d: results lie in the flow in order, in whole words", i);
      prm.ops[i].reserved = (o.gamma ? kNorm : 0) | (flows(o.A) ? kRowsFlow : 0) | (o.residual && flows(o.residual) ? kResidualFlows : 0);
      rows = std::max(rows, (int)o.M);
      if (std::find(depths.begin(), depths.end(), o.K) == depths.end()) depths.push_back(o.K);
      if (o.gamma) normed_k = std::max(normed_k, (int)o.K);
    } else {
      TTB_REQUIRE(ctx, ops[i].kind == TTB_CHAIN_ATTENTION, "chain_forward: operation %d: unknown kind", i);
      const ttb_chain_attention& o = ops[i].u.attention;
      const int H = o.heads * kHeadDim;
      TTB_REQUIRE(ctx, o.rows > 0 && o.rows <= TTB_CHAIN_MAX_ROWS && o.heads > 0 && o.heads <= 256 && o.past >= 0 && o.q && o.out, "chain_forward: operation %d: bad shape", i);
      TTB_REQUIRE(ctx, o.ldq % 8 == 0 && o.ldo % 2 == 0 && o.ldo >= H && aligned({o.q, o.k, o.v, o.k_cache, o.v_cache}) && (reinterpret_cast<uintptr_t>(o.out) & 3) == 0,
                  "chain_forward: operation %d: misaligned operand", i);
      switch (o.keys) {
        case TTB_CHAIN_KEYS_ROWS:
          TTB_REQUIRE(ctx, o.length > 0 && o.rows % o.length == 0 && o.ldq >= 3 * H && !o.k_cache == !o.v_cache, "chain_forward: operation %d: bad rows", i);
          break;
        case TTB_CHAIN_KEYS_CACHE:
          TTB_REQUIRE(ctx, o.k_cache && o.v_cache && o.ldq >= 3 * H, "chain_forward: operation %d: bad cache", i);
          break;
        case TTB_CHAIN_KEYS_MEMORY:
          TTB_REQUIRE(ctx, o.k && o.v && o.length > 0 && o.ldq >= H, "chain_forward: operation %d: bad memory", i);
          break;
        default: TTB_REQUIRE(ctx, false, "chain_forward: operation %d: unknown keys", i);
      }
      TTB_REQUIRE(ctx, !o.mask || o.mask_pitch >= (o.keys == TTB_CHAIN_KEYS_CACHE ? o.past + 1 : o.length), "chain_forward: operation %d: the mask is too short", i);
      TTB_REQUIRE(ctx, !o.probs || (o.keys == TTB_CHAIN_KEYS_MEMORY && o.scores), "chain_forward: operation %d: probabilities need a memory and scratch", i);
      TTB_REQUIRE(ctx, fill(o.out, o.rows, o.ldo, H), "chain_forward: operation %d: results lie in the flow in order, in whole words", i);
      TTB_REQUIRE(ctx, !flow || (!flows(o.k) && !flows(o.v) && !flows(o.k_cache) && !flows(o.v_cache)), "chain_forward: operation %d: keys in the flow", i);
      prm.ops[i].reserved = flows(o.q) ? kRowsFlow : 0;
    }
    if (!flow && i > 0) prm.ops[i].reserved |= kBarrier;
  }
  DeviceGuard g(ctx->device);
  prm.n_ops = n_ops;
  prm.counter = counter;
  prm.status = ctx->d_status;
  const Plan plan = plan_of(rows, depths, normed_k);
  TTB_REQUIRE(ctx, plan.chunks > 0, "chain_forward: an operation is too deep");
  prm.ring_bytes = plan.ring_bytes;
  prm.a_bytes = plan.a_bytes;
  prm.sums_bytes = sums_of(plan.tiles, plan.group);
  for (int i = 0; i < n_ops; ++i)
    if (ops[i].kind == TTB_CHAIN_LINEAR)  // a group's weights fit in the ring
      prm.ops[i].reserved |= std::min(plan.group, prm.ring_bytes / unit_bytes(ops[i].u.linear.K));
  if (flow) TTB_CUDA(ctx, cudaMemsetAsync(flow, TTB_CHAIN_UNWRITTEN & 0xff, flow_bytes, ctx->stream));
  else TTB_CUDA(ctx, cudaMemsetAsync(counter, 0, TTB_CHAIN_WORKSPACE, ctx->stream));
  switch (plan.tiles) {
    case 1: TTB_CUDA(ctx, launch<1>(ctx, plan, prm)); break;
    case 2: TTB_CUDA(ctx, launch<2>(ctx, plan, prm)); break;
    case 3: TTB_CUDA(ctx, launch<3>(ctx, plan, prm)); break;
    case 4: TTB_CUDA(ctx, launch<4>(ctx, plan, prm)); break;
    default: TTB_CUDA(ctx, launch<8>(ctx, plan, prm));
  }
  return launched(ctx, "chain_forward");
}

}  // namespace

extern "C" int ttb_chain_forward(ttb_ctx* ctx, int dtype, const ttb_chain_op* ops, int n_ops, void* workspace) {
  return chain_forward(ctx, dtype, ops, n_ops, static_cast<int*>(workspace), nullptr, 0);
}

extern "C" int ttb_chain_forward_flow(ttb_ctx* ctx, int dtype, const ttb_chain_op* ops, int n_ops, void* flow, int64_t flow_bytes) {
  if (ctx) TTB_REQUIRE(ctx, flow && flow_bytes > 0, "chain_forward_flow: no flow");
  return chain_forward(ctx, dtype, ops, n_ops, nullptr, flow, (size_t)flow_bytes);
}
