// A stack of transformer layers over few rows as one resident kernel (ttb_chain_forward).
//
// What bounds it: a decoding step or a request of a few tokens is a chain of dependent operations, five a layer, each of which moves
// a few megabytes of weights and computes next to nothing. As separate kernels each cost 4.8 us (GPT-2 small, one row: 89 kernels, 428 us
// a step; its weights stream in 38 us). Here one grid of one CTA per SM runs all of them with a barrier over the grid between two,
// and what does not depend on the operation before is fetched ahead of it:
//   * Weights. The output columns of a product are dealt out in units of eight (eight rows of W[N,K]: contiguous memory), as evenly as
//     they go over the CTAs. While a CTA waits at the barrier, one of its warps copies the units that it will read next into a
//     shared-memory ring (cp.async.bulk) until the ring is full: about a layer ahead of the arithmetic. Norm weights and biases
//     travel the same way, and cached keys and values are brought to L2.
//   * The products run on mma.sync m16n8k16 with the eight columns of a unit as its n: 128-row tcgen05 tiles would be empty but for a few
//     rows, and the round trip through tensor memory is longer than the whole product. The warps split the rows (16 each)
//     and K; the order of k inside a 32-wide chunk is permuted alike for both operands so that each thread loads 16 bytes at a time: A straight
//     from global memory into fragments (no warp reads what another does), W from the ring without bank conflicts (row pitch 64
//     bytes past a multiple of 128). Partial sums meet in shared memory.
//   * A layer norm in front of a product: every CTA normalises all rows itself into shared memory, which is cheaper than a barrier.
//   * Attention: the warps of a CTA share a (row, head), or several; eight lanes a key, online softmax, merged through shared memory.
//   * Code. Every operation runs through its instructions once, so that fetching them counts: loops over what differs from call to call are
//     not unrolled and waits and copies are functions (167 -> 67 KB for 16 rows: 306 -> 286 us a step of the above, 349 -> 320 of 8 rows
//     with 300 cached tokens).
// Now 286 us a step (layer by layer 414 on the same GPU): 60 operations of 2.9 to 3.5 us, of which the barrier itself is 1.0, the rows' way from L2 (and
// their layer norm) 0.9 to 1.0, the products 0.3 to 0.6 and the epilogue 0.3; the vocabulary's product, the embedding and the launch are the rest.
#include <algorithm>
#include <initializer_list>

#include "ttb_chain_rules.cuh"
#include "ttb_common.cuh"
#include "ttb_sm100.cuh"

using namespace ttb;

namespace {

using chain::kWarps;                            // the operations are bound by what every warp has to do anyway: fewer warps, with more registers
constexpr int kThreads = kWarps * 32;
constexpr int kGroup = 4;                       // most units of eight columns that a CTA computes at a time
constexpr int kRowPad = 64;                     // bytes between the rows of a ring slot, for the banks
constexpr int kPart = 1024;                     // most of K in a slot
constexpr int kMaxSlots = 24;
constexpr int kParamSlots = 4;
using chain::kBiasUnits;
constexpr int kParamBytes = 2 * kPart * 2 + kBiasUnits * 16;
constexpr int kSmemLimit = 227 * 1024;
constexpr int kHeadDim = 64;
constexpr float kLog2e = 1.4426950408889634f;

struct ChainParams {
  ttb_chain_op ops[TTB_CHAIN_MAX_OPS];  // linear: `reserved` is the part of K in a ring slot, and << 16 the units of a group
  int n_ops, slots, slot_bytes;
  int a_bytes;   // shared memory of the normalised rows
  int* counter;  // arrivals at the grid's barrier
  int* status;
};
constexpr int kOpWords = sizeof(ttb_chain_op) / 4;

// Position in a ring: slot and the parity of its current use.
struct Cursor {
  int slot = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next(int slots) {
    if (++slot == slots) {
      slot = 0;
      parity ^= 1;
    }
  }
};
// How far the copies have got: the next one is unit `first + unit`, part `batch + k` of K, of operation `op`.
struct Feed {
  int op = 0, begun = 0, first = 0, unit = 0, batch = 0, k = 0;
  int issued = 0, p_issued = 0;
  Cursor w, p;
};

// The units of a product that belong to this CTA, and whether it takes part in the operation at all: CTA r also writes normalised row r.
struct Share {
  int lo, hi;
  bool writes, part, params;  // params: norm weights or a bias come with it
  __device__ __forceinline__ Share() {}
  __device__ __forceinline__ explicit Share(const ttb_chain_linear& o) {
    const uint32_t units = ((uint32_t)o.N + 7) >> 3;
    lo = (int)chain::first_unit(units, blockIdx.x, gridDim.x);
    hi = (int)chain::first_unit(units, blockIdx.x + 1, gridDim.x);
    writes = o.gamma && o.normed && (int)blockIdx.x < o.M;
    part = hi > lo || writes;
    params = part && (o.gamma || (o.bias && hi > lo));
  }
};

struct Shared {
  ttb_chain_op ops[TTB_CHAIN_MAX_OPS];   // (read from the kernel's parameters, every operation's first use would miss the constant cache)
  Share share[TTB_CHAIN_MAX_OPS];
  float red[kWarps * kGroup * 128];      // partial sums of a group of units, or attention states
  uint8_t params[kParamSlots][kParamBytes];
  uint64_t full[kMaxSlots], pfull[kParamSlots];
  Feed feed;
  volatile int abort_flag;
};
constexpr int kSharedBytes = (sizeof(Shared) + 127) / 128 * 128;

// The thread's number, read anew in every operation: what the compiler derives from it ahead of the loop over the operations it
// has to spill, and a spill costs a trip to L2 here, since the barrier's acquire empties the L1 cache.
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
__device__ __forceinline__ void unpack(const uint4& r, float (&f)[8]) {
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __half22float2(h[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
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
// loads ahead
// ---------------------------------------------------------------------------------------------
// A bounded wait (each attempt suspends the thread for up to 20 us, 2^17 of them are some seconds) without a call: what is live around a
// call would be spilled, and a spill costs a trip to L2 here, since the barrier's acquire empties the L1 cache.
[[nodiscard]] __device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int tries = 0; tries < (1 << 17); ++tries) {
    if (sm100::mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// Waits, whatever the abort flag says, for a use of a slot whose copies have been issued.
__device__ __forceinline__ void drain(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!sm100::mbar_try_wait(bar, parity) && clock64() - t0 < sm100::kWaitCycles) {
  }
}

// Issues the weight copies of the operation that `f` is at, as far as the ring has room; true: all of them are on their way.
__device__ __forceinline__ bool feed_units(const ttb_chain_linear& o, int ks, int group, int hi, const ChainParams& prm, Shared& sm, uint32_t ring, int kpb,
                                           int consumed, Feed& f) {
  const int lane = threadIdx.x & 31, parts = div_small(o.K, ks);
#pragma unroll 1
  while (f.first < hi) {  // groups of units; in a group all units of one batch of parts of K, then of the next
    if (f.issued - consumed >= prm.slots) return false;
    const uint32_t bar = sm100::smem_u32(&sm.full[f.w.slot]);
    const int row0 = (f.first + f.unit) * 8, rows = min(8, o.N - row0);
    if (lane == 0) sm100::mbar_expect_tx(bar, (uint32_t)(rows * ks * 2));
    __syncwarp();
    if (lane < rows)
      sm100::bulk_load_1d(ring + f.w.slot * prm.slot_bytes + lane * (ks * 2 + kRowPad),
                          static_cast<const __half*>(o.W) + (long long)(row0 + lane) * o.K + (f.batch + f.k) * ks, (uint32_t)ks * 2, bar);
    f.w.next(prm.slots);
    ++f.issued;
    if (++f.k == min(kpb, parts - f.batch)) {
      f.k = 0;
      if (++f.unit == min(group, hi - f.first)) {
        f.unit = 0;
        f.batch += kpb;
        if (f.batch >= parts) {
          f.batch = 0;
          f.first += group;
        }
      }
    }
  }
  return true;
}

// Issues the copies that the rings have room for, in the order in which the CTA will read them. One warp calls it, where all warps
// have passed a barrier behind their last read of `consumed` slots and `p_consumed` norm and bias slots.
__device__ __noinline__ void feed(const ChainParams& prm, Shared& sm, uint32_t ring, int kpb, int consumed, int p_consumed) {
  const int lane = threadIdx.x & 31;
  Feed f = sm.feed;
  __syncwarp();
#pragma unroll 1
  for (; f.op < prm.n_ops; ++f.op) {
    if (sm.ops[f.op].kind != TTB_CHAIN_LINEAR) continue;
    const ttb_chain_linear& o = sm.ops[f.op].u.linear;
    const Share s = sm.share[f.op];
    if (!f.begun) {
      if (s.params) {
        if (f.p_issued - p_consumed >= kParamSlots) break;
        if (lane == 0) {
          const uint32_t bar = sm100::smem_u32(&sm.pfull[f.p.slot]), dst = sm100::smem_u32(sm.params[f.p.slot]);
          const uint32_t norm = o.gamma ? (uint32_t)o.K * 2 : 0, bias = o.bias ? (uint32_t)(s.hi - s.lo) * 16 : 0;
          sm100::mbar_expect_tx(bar, 2 * norm + bias);
          if (norm) {
            sm100::bulk_load_1d(dst, o.gamma, norm, bar);
            sm100::bulk_load_1d(dst + kPart * 2, o.beta, norm, bar);
          }
          if (bias) sm100::bulk_load_1d(dst + kPart * 4, static_cast<const char*>(o.bias) + (size_t)s.lo * 16, bias, bar);
        }
        f.p.next(kParamSlots);
        ++f.p_issued;
      }
      f.begun = 1;
      f.first = s.lo;
      f.unit = f.k = f.batch = 0;
    }
    if (!feed_units(o, sm.ops[f.op].reserved & 0xffff, sm.ops[f.op].reserved >> 16, s.hi, prm, sm, ring, kpb, consumed, f)) break;
    f.begun = 0;
  }
  if (lane == 0) sm.feed = f;
  __syncwarp();
}

// Waits for the next n slots of the ring.
[[nodiscard]] __device__ __noinline__ bool wait_slots(int n, int slots, Shared& sm, Cursor w) {
  bool ok = true;
#pragma unroll 1
  for (int i = 0; ok && i < n; ++i) {
    ok = wait(sm100::smem_u32(&sm.full[w.slot]), w.parity, &sm.abort_flag);
    w.next(slots);
  }
  return ok;
}

// Waits for the norm weights, bias and weights with which the CTA's share of an operation begins. One warp does it for all of them, ahead of
// a barrier of the CTA and mostly in the shadow of the grid's.
[[nodiscard]] __device__ __forceinline__ bool wait_ahead(const ttb_chain_op& op, const Share& s, int slots, Shared& sm, Cursor w, const Cursor& p) {
  if (op.kind != TTB_CHAIN_LINEAR || !s.part) return true;
  const bool ok = !s.params || wait(sm100::smem_u32(&sm.pfull[p.slot]), p.parity, &sm.abort_flag);
  return ok && wait_slots(min(op.reserved >> 16, s.hi - s.lo) * div_small(op.u.linear.K, op.reserved & 0xffff), slots, sm, w);
}

// Brings the keys and values that an earlier launch has written, and that this CTA reads two operations later, to L2.
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

// ---------------------------------------------------------------------------------------------
// products
// ---------------------------------------------------------------------------------------------
// What a CTA has read of its rings.
struct Read {
  Cursor w, p;
  int slots = 0, params = 0;
};

// The layout of a product: MT tiles of 16 rows, and the warps are MT tiles x KW shares of K. A chunk is 32 of K: thread t of a quad
// holds 8 of them, in 16 bytes, for its rows g and g + 8. Chunk c of a ring slot's part of K belongs to share c % KW, CPK of them
// to a warp at most.
template <int MT> struct Layout {
  static constexpr int KW = kWarps / MT, CPK = kPart / 32 / KW;
  static constexpr int kBatch = CPK <= 8 ? 16 / CPK : 1;  // parts of K whose fragments (up to 128 registers) are held at a time
  static constexpr int kItems = (MT * 16 * kGroup * 4 + kThreads - 1) / kThreads;  // pairs of output columns per thread and group
};

// Pair `it` of a thread: its row and its unit in the group.
__device__ __forceinline__ int item_row(int tid, int it) { return ((tid + it * kThreads) >> 8) * 16 + ((tid >> 2) & 15); }
__device__ __forceinline__ int item_unit(int tid) { return (tid >> 6) & 3; }

template <int MT> __device__ __forceinline__ void fetch_residual(const ttb_chain_linear& o, int u0, int nu, __half2 (&res)[Layout<MT>::kItems]) {
#pragma unroll
  for (int it = 0; it < Layout<MT>::kItems; ++it) res[it] = __half2();
  if (!o.residual) return;
  const int tid = thread();
#pragma unroll
  for (int it = 0; it < Layout<MT>::kItems; ++it)
    if (item_row(tid, it) < o.M && item_unit(tid) < nu)
      res[it] = *reinterpret_cast<const __half2*>(static_cast<const __half*>(o.residual) + (long long)item_row(tid, it) * o.ldr + (u0 + item_unit(tid)) * 8 +
                                                  (tid & 3) * 2);
}

// Adds up the shares of a group's sums and finishes them.
template <int MT>
__device__ __forceinline__ void epilogue(const ttb_chain_linear& o, const Shared& sm, const uint8_t* bias, int u0, int nu,
                                         const __half2 (&res)[Layout<MT>::kItems]) {
  constexpr int KW = Layout<MT>::KW;
  const bool pairs = ((o.ldo | o.N) & 1) == 0 && (reinterpret_cast<uintptr_t>(o.out) & 3) == 0;
  const int tid = thread(), u = item_unit(tid), cp = tid & 3;
#pragma unroll
  for (int it = 0; it < Layout<MT>::kItems; ++it) {
    const int row = item_row(tid, it);
    if (row < o.M && u < nu) {
      const float* src = sm.red + ((row >> 4) * kGroup + u) * KW * 128 + (tid & 63) * 2;
      float2 v[2] = {};
#pragma unroll
      for (int j = 0; j < KW; ++j) {
        const float2 x = *reinterpret_cast<const float2*>(src + j * 128);
        v[j & 1].x += x.x;
        v[j & 1].y += x.y;
      }
      v[0].x += v[1].x;
      v[0].y += v[1].y;
      if (o.bias) {
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(bias + u * 16 + cp * 4));
        v[0].x += b.x;
        v[0].y += b.y;
      }
      if (o.act == TTB_CHAIN_ACT_GELU) {
        v[0].x = gelu16(v[0].x);
        v[0].y = gelu16(v[0].y);
      } else if (o.act == TTB_CHAIN_ACT_RELU) {
        v[0].x = fmaxf(v[0].x, 0.f);
        v[0].y = fmaxf(v[0].y, 0.f);
      }
      if (o.residual) {
        const float2 r = __half22float2(res[it]);
        v[0].x += r.x;
        v[0].y += r.y;
      }
      const int col = (u0 + u) * 8 + cp * 2;
      __half* out = static_cast<__half*>(o.out) + (long long)row * o.ldo + col;
      if (pairs) {
        if (col < o.N) *reinterpret_cast<__half2*>(out) = __floats2half2_rn(v[0].x, v[0].y);
      } else {
        if (col < o.N) out[0] = __float2half_rn(v[0].x);
        if (col + 1 < o.N) out[1] = __float2half_rn(v[0].y);
      }
    }
  }
}

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

// Layer norm of the operation's rows into shared memory, a warp per row (64 bytes past a multiple of 128 between rows, as in the ring).
// The next row of a warp is on its way while one is normalised.
__device__ __forceinline__ void normalise(const ttb_chain_linear& o, const Share& s, Shared& sm, uint32_t a_smem, const Read& read) {
  constexpr int kIters = kPart / 256;  // 16-byte pieces of a row per lane
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, K = o.K, M = o.M;
  const __half* src = static_cast<const __half*>(o.A) + (long long)warp * o.lda + lane * 8;
  const uint32_t gamma = sm100::smem_u32(sm.params[read.p.slot]) + lane * 16;
  const float inv_k = __fdividef(1.f, (float)K), eps = o.eps;
  uint4 next[kIters];
#pragma unroll
  for (int i = 0; i < kIters; ++i) {
    next[i] = make_uint4(0, 0, 0, 0);
    if (warp < M && i * 256 + lane * 8 < K) next[i] = *reinterpret_cast<const uint4*>(src + i * 256);
  }
#pragma unroll 1
  for (int row = warp; row < M; row += kWarps) {
    Two f[kIters][4], sum(0.f, 0.f), sq(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kIters; ++i) {  // (lanes beyond the row hold zeros)
      unpack2(next[i], f[i]);
      sum = sum + ((f[i][0] + f[i][1]) + (f[i][2] + f[i][3]));
    }
    src += (long long)kWarps * o.lda;
    if (row + kWarps < M)
#pragma unroll
      for (int i = 0; i < kIters; ++i)
        if (i * 256 + lane * 8 < K) next[i] = *reinterpret_cast<const uint4*>(src + i * 256);
    const float mean = warp_sum(sum.get().x + sum.get().y) * inv_k;
    const Two minus(-mean, -mean);
#pragma unroll
    for (int i = 0; i < kIters; ++i)
      if (i * 256 + lane * 8 < K)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          f[i][e] = f[i][e] + minus;
          sq = fma2(f[i][e], f[i][e], sq);
        }
    const float rstd = rsqrtf(warp_sum(sq.get().x + sq.get().y) * inv_k + eps);
    const Two scale(rstd, rstd);
    const uint32_t to = a_smem + row * (K * 2 + kRowPad) + lane * 16;
#pragma unroll
    for (int i = 0; i < kIters; ++i)
      if (i * 256 + lane * 8 < K) {
        Two ga[4], be[4];
        unpack2(lds128(gamma + i * 512), ga);
        unpack2(lds128(gamma + kPart * 2 + i * 512), be);
        float y[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = fma2(f[i][e] * scale, ga[e], be[e]).get();
          y[2 * e] = v.x;
          y[2 * e + 1] = v.y;
        }
        const uint4 q = pack(y);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + i * 512), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
        if (s.writes && chain::writes_row(row, (int)blockIdx.x)) *reinterpret_cast<uint4*>(static_cast<__half*>(o.normed) + (long long)row * K + i * 256 + lane * 8) = q;
      }
  }
}

// Product of the rows that normalise() has left in shared memory; K is one part.
template <int MT>
__device__ __forceinline__ bool linear_norm(const ttb_chain_linear& o, const Share& s, int ks, int group, const ChainParams& prm, Shared& sm, uint32_t a_smem, uint32_t ring,
                                            Read& read) {
  constexpr int KW = Layout<MT>::KW, CPK = Layout<MT>::CPK;
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int mt = warp % MT, share = warp / MT, chunks = ks / 32;
  normalise(o, s, sm, a_smem, read);
  bool ok = true;
  const uint32_t lane_at = g * (ks * 2 + kRowPad) + share * 64 + t * 16;
  const uint32_t w_lane = ring + lane_at, a_lane = a_smem + mt * 16 * (ks * 2 + kRowPad) + lane_at, a_eight = 8 * (ks * 2 + kRowPad);
  const bool low = mt * 16 < o.M, high = mt * 16 + 8 < o.M;  // rows of the tile's halves (rows that are not there leave sums that nobody reads)
  __syncthreads();
#pragma unroll 1
  for (int u0 = s.lo; u0 < s.hi; u0 += group) {
    const int nu = min(group, s.hi - u0);
    if (u0 != s.lo) ok = wait_slots(nu, prm.slots, sm, read.w) && ok;
    uint32_t at[kGroup];
    float acc[kGroup][4];
#pragma unroll
    for (int u = 0; u < kGroup; ++u) {
      at[u] = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[u][e] = 0.f;
      if (u < nu) {
        at[u] = w_lane + read.w.slot * prm.slot_bytes;
        read.w.next(prm.slots);
        ++read.slots;
      }
    }
    if (low)
#pragma unroll
      for (int i = 0; i < CPK; ++i)
        if (i * KW + share < chunks) {
          uint4 b[kGroup], x = lds128(a_lane + i * KW * 64), y = make_uint4(0, 0, 0, 0);
          if (high) y = lds128(a_lane + a_eight + i * KW * 64);
#pragma unroll
          for (int u = 0; u < kGroup; ++u)
            b[u] = u < nu ? lds128(at[u] + i * KW * 64) : make_uint4(0, 0, 0, 0);
#pragma unroll
          for (int u = 0; u < kGroup; ++u)
            if (u < nu) mma16816(acc[u], x.x, y.x, x.y, y.y, b[u].x, b[u].y);
#pragma unroll
          for (int u = 0; u < kGroup; ++u)
            if (u < nu) mma16816(acc[u], x.z, y.z, x.w, y.w, b[u].z, b[u].w);
        }
    float2* dst = reinterpret_cast<float2*>(sm.red + (mt * kGroup * KW + share) * 128 + g * 8 + t * 2);
#pragma unroll
    for (int u = 0; u < kGroup; ++u)
      if (u < nu) {
        dst[u * KW * 64] = make_float2(acc[u][0], acc[u][1]);
        dst[u * KW * 64 + 32] = make_float2(acc[u][2], acc[u][3]);
      }
    __syncthreads();
    __half2 res[Layout<MT>::kItems];
    fetch_residual<MT>(o, u0, nu, res);
    epilogue<MT>(o, sm, sm.params[read.p.slot] + kPart * 4 + (u0 - s.lo) * 16, u0, nu, res);
    if (u0 + group < s.hi) {
      if (warp == kWarps - 1) feed(prm, sm, ring, Layout<MT>::kBatch, read.slots, read.params);  // behind a wide product, such as a vocabulary
      __syncthreads();  // the next group's partial sums take the same place
    }
  }
  read.p.next(kParamSlots);
  ++read.params;
  return ok;
}

// Product of rows as they are, K in up to eight parts.
template <int MT>
__device__ __forceinline__ bool linear_plain(const ttb_chain_linear& o, const Share& s, int ks, int group, const ChainParams& prm, Shared& sm, uint32_t ring, Read& read) {
  constexpr int KW = Layout<MT>::KW, CPK = Layout<MT>::CPK, kBatch = Layout<MT>::kBatch;
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int mt = warp % MT, share = warp / MT, chunks = ks / 32, parts = div_small(o.K, ks);
  const int r0 = mt * 16 + g, r1 = r0 + 8, M = o.M;
  const bool high = mt * 16 + 8 < M;  // rows in the tile's upper half
  const __half* a_lane = static_cast<const __half*>(o.A) + (long long)r0 * o.lda + share * 32 + t * 8;
  const uint32_t w_lane = ring + g * (ks * 2 + kRowPad) + share * 64 + t * 16;
  bool ok = true;
#pragma unroll 1
  for (int u0 = s.lo; u0 < s.hi; u0 += group) {
    const int nu = min(group, s.hi - u0);
    if (u0 != s.lo) ok = wait_slots(nu * parts, prm.slots, sm, read.w) && ok;
    __half2 res[Layout<MT>::kItems];
#pragma unroll 1
    for (int kb = 0; kb < parts; kb += kBatch) {
      uint4 a0[kBatch * CPK], a1[kBatch * CPK];
#pragma unroll
      for (int kl = 0; kl < kBatch; ++kl) {
        const __half* p0 = a_lane + (kb + kl) * ks;
        const __half* p1 = p0 + 8ll * o.lda;
#pragma unroll
        for (int i = 0; i < CPK; ++i) {
          a0[kl * CPK + i] = a1[kl * CPK + i] = make_uint4(0, 0, 0, 0);
          if (kb + kl < parts && i * KW + share < chunks) {
            if (r0 < M) a0[kl * CPK + i] = *reinterpret_cast<const uint4*>(p0 + i * KW * 32);
            if (high && r1 < M) a1[kl * CPK + i] = *reinterpret_cast<const uint4*>(p1 + i * KW * 32);
          }
        }
      }
      if (kb == 0) fetch_residual<MT>(o, u0, nu, res);  // what the epilogue adds is on its way before the products
#pragma unroll 1
      for (int u = 0; u < nu; ++u) {
        float acc[2][4] = {};  // two chains of sums
#pragma unroll
        for (int kl = 0; kl < kBatch; ++kl)
          if (kb + kl < parts) {
            const uint32_t at = w_lane + read.w.slot * prm.slot_bytes;
#pragma unroll
            for (int i = 0; i < CPK; ++i)
              if (i * KW + share < chunks) {
                const uint4 b = lds128(at + i * KW * 64);
                const uint4 &x = a0[kl * CPK + i], &y = a1[kl * CPK + i];
                mma16816(acc[0], x.x, y.x, x.y, y.y, b.x, b.y);
                mma16816(acc[1], x.z, y.z, x.w, y.w, b.z, b.w);
              }
            read.w.next(prm.slots);
            ++read.slots;
          }
        float2* dst = reinterpret_cast<float2*>(sm.red + ((mt * kGroup + u) * KW + share) * 128 + g * 8 + t * 2);
        float2 v0 = make_float2(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]), v1 = make_float2(acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
        if (kb > 0) {  // the sums of the parts before, by this thread
          const float2 p0 = dst[0], p1 = dst[32];
          v0 = make_float2(v0.x + p0.x, v0.y + p0.y);
          v1 = make_float2(v1.x + p1.x, v1.y + p1.y);
        }
        dst[0] = v0;
        dst[32] = v1;
      }
    }
    __syncthreads();
    epilogue<MT>(o, sm, sm.params[read.p.slot] + kPart * 4 + (u0 - s.lo) * 16, u0, nu, res);
    if (u0 + group < s.hi) {
      if (warp == kWarps - 1) feed(prm, sm, ring, kBatch, read.slots, read.params);
      __syncthreads();
    }
  }
  if (o.bias) {
    read.p.next(kParamSlots);
    ++read.params;
  }
  return ok;
}

// ---------------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------------
// (row, head) pairs go round the CTAs; a CTA's warps are shared out among as many of its pairs as they serve at once, each taking
// every W-th page of 16 keys: four keys a load, the next page on its way while one is worked on.
__device__ __forceinline__ void attention(const ttb_chain_attention& o, Shared& sm) {
  constexpr int kState = kHeadDim + 2;
  const int tid = thread(), warp = tid >> 5, lane = tid & 31, sub = lane & 7, kg = lane >> 3;
  const int heads = o.heads, H = heads * kHeadDim, total = o.rows * heads, keys = o.keys;
  const int mine = div_small(total - (int)blockIdx.x + (int)gridDim.x - 1, gridDim.x);  // pairs of this CTA
  if (total <= (int)blockIdx.x) return;
  const int W = max(1, div_small(kWarps, mine)), S = div_small(kWarps, W);  // warps a pair, pairs at once
  const int place = div_small(warp, W), wi = warp - place * W;
#pragma unroll 1
  for (int first = 0; first < mine; first += S) {
    const bool active = place < S && first + place < mine;
    const int unit = active ? (first + place) * (int)gridDim.x + (int)blockIdx.x : 0;
    const int row = div_small(unit, heads), h = unit - row * heads;
    const __half* qrow = static_cast<const __half*>(o.q) + (long long)row * o.ldq + h * kHeadDim;
    int seq = row, place_in = o.past, n = o.past + 1;  // of the row: its sequence, its position, the keys it sees
    // key j of the row: k0 + (j / 16) * page + (j % 16) * pitch
    const __half *k0, *v0;
    long long page;
    int pitch = H;
    if (keys == TTB_CHAIN_KEYS_CACHE) {
      k0 = static_cast<const __half*>(o.k_cache) + (long long)row * 16 * H + h * kHeadDim;
      v0 = static_cast<const __half*>(o.v_cache) + (long long)row * 16 * H + h * kHeadDim;
      page = 16ll * o.rows * H;
    } else if (keys == TTB_CHAIN_KEYS_ROWS) {
      seq = div_small(row, o.length);
      place_in = row - seq * o.length;
      n = o.causal ? place_in + 1 : o.length;
      pitch = o.ldq;
      page = 16ll * pitch;
      k0 = static_cast<const __half*>(o.q) + (long long)(seq * o.length) * pitch + H + h * kHeadDim;
      v0 = k0 + H;
    } else {
      n = o.length;
      pitch = kHeadDim;
      page = 16 * kHeadDim;
      k0 = static_cast<const __half*>(o.k) + (long long)unit * n * kHeadDim;
      v0 = static_cast<const __half*>(o.v) + (long long)unit * n * kHeadDim;
    }
    const float* mask = o.mask ? o.mask + (long long)seq * o.mask_pitch : nullptr;
    float* scores = o.probs && h == 0 ? o.scores + (long long)row * o.length : nullptr;
    float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    if (active) {
      float q[8];
      unpack(*reinterpret_cast<const uint4*>(qrow + sub * 8), q);
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] *= o.scale * kLog2e;
      // the new token's key and value are filed by the warp with the fewest keys (pairs of the same row write its other heads)
      const bool files = wi == W - 1 && lane < 16 && o.k_cache && keys != TTB_CHAIN_KEYS_MEMORY;
      uint4 newest = make_uint4(0, 0, 0, 0), *file_to = nullptr;
      if (files) {
        const int sequences = keys == TTB_CHAIN_KEYS_CACHE ? o.rows : div_small(o.rows, o.length);
        newest = *reinterpret_cast<const uint4*>(qrow + (lane < 8 ? H : 2 * H) + sub * 8);
        file_to = reinterpret_cast<uint4*>(static_cast<__half*>(lane < 8 ? o.k_cache : o.v_cache) + cache_row(place_in, seq, sequences, H) + h * kHeadDim + sub * 8);
      }
      const int fresh = keys == TTB_CHAIN_KEYS_CACHE ? n - 1 : -1;  // the key that is not in the cache yet
      const __half *kp = k0 + wi * page + (long long)kg * pitch + sub * 8, *vp = v0 + wi * page + (long long)kg * pitch + sub * 8;
      uint4 kr[4], vr[4], kn[4], vn[4];
#pragma unroll 1
      for (int j0 = (wi - W) * 16; j0 < n; j0 += 16 * W) {
        // the next page is on its way while this one (there is none at first) is worked on
        const int j1 = j0 + 16 * W + kg;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          kn[u] = vn[u] = make_uint4(0, 0, 0, 0);
          const int j = j1 + u * 4;
          if (j < n) {
            kn[u] = *reinterpret_cast<const uint4*>(j == fresh ? qrow + H + sub * 8 : kp + u * 4 * pitch);
            vn[u] = *reinterpret_cast<const uint4*>(j == fresh ? qrow + 2 * H + sub * 8 : vp + u * 4 * pitch);
          }
        }
        kp += W * page;
        vp += W * page;
        if (j0 >= 0) {
          float sc[4], top = m;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float f[8], dot[2];
            unpack(kr[u], f);
            dot[0] = q[0] * f[0];
            dot[1] = q[1] * f[1];
#pragma unroll
            for (int e = 2; e < 8; ++e) dot[e & 1] = fmaf(q[e], f[e], dot[e & 1]);
            sc[u] = dot[0] + dot[1];
          }
#pragma unroll
          for (int d = 1; d < 8; d <<= 1)
#pragma unroll
            for (int u = 0; u < 4; ++u) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], d);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = j0 + u * 4 + kg;
            if (j < n) {
              if (mask) sc[u] += mask[j] * kLog2e;
              if (scores && sub == 0) scores[j] = sc[u];
            } else {
              sc[u] = -INFINITY;
            }
            top = fmaxf(top, sc[u]);
          }
          const float base = top == -INFINITY ? 0.f : top, keep = ex2f(m - base);
          m = top;
          l *= keep;
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] *= keep;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float pr = ex2f(sc[u] - base);
            float f[8];
            unpack(vr[u], f);
            l += pr;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = fmaf(pr, f[e], acc[e]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          kr[u] = kn[u];
          vr[u] = vn[u];
        }
      }
      if (files) *file_to = newest;
    }
    // the four groups of a warp, then the warps
#pragma unroll
    for (int d = 8; d <= 16; d <<= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m, d), lo = __shfl_xor_sync(0xffffffffu, l, d);
      const float top = fmaxf(m, mo), base = top == -INFINITY ? 0.f : top;
      const float a = ex2f(m - base), b = ex2f(mo - base);
      m = top;
      l = l * a + lo * b;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = acc[e] * a + __shfl_xor_sync(0xffffffffu, acc[e], d) * b;
    }
    float* state = sm.red + warp * kState;
    if (lane < 8) {
#pragma unroll
      for (int e = 0; e < 8; ++e) state[2 + lane * 8 + e] = acc[e];
      if (lane == 0) {
        state[0] = m;
        state[1] = l;
      }
    }
    __syncthreads();
    if (active && (wi == 0 || scores)) {
      const float* st = sm.red + place * W * kState;
      const int used = min(W, (n + 15) >> 4);  // warps that have seen a key
      const float mine_m = lane < used ? st[lane * kState] : -INFINITY, mine_l = lane < used ? st[lane * kState + 1] : 0.f;
      const float top = warp_max(mine_m), base = top == -INFINITY ? 0.f : top;
      const float factor = ex2f(mine_m - base), inv = 1.f / warp_sum(mine_l * factor);
      if (wi == 0) {
        float2 v = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int i = 0; i < used; ++i) {
          const float f = __shfl_sync(0xffffffffu, factor, i);
          v.x = fmaf(f, st[i * kState + 2 + lane * 2], v.x);
          v.y = fmaf(f, st[i * kState + 3 + lane * 2], v.y);
        }
        *reinterpret_cast<__half2*>(static_cast<__half*>(o.out) + (long long)row * o.ldo + h * kHeadDim + lane * 2) = __floats2half2_rn(v.x * inv, v.y * inv);
      }
      if (scores)
#pragma unroll 1
        for (int j = wi * 32 + lane; j < n; j += W * 32)
          static_cast<__half*>(o.probs)[(long long)row * o.length + j] = __float2half_rn(ex2f(scores[j] - base) * inv);
    }
    if (first + S < mine) __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------------------------
template <int MT>
__global__ void __launch_bounds__(kThreads, 1) chain_kernel(const __grid_constant__ ChainParams prm) {
  extern __shared__ __align__(128) uint8_t smem[];
  Shared& sm = *reinterpret_cast<Shared*>(smem);
  const uint32_t rows = sm100::smem_u32(smem) + kSharedBytes, ring = rows + prm.a_bytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < prm.slots; ++i) sm100::mbar_init(sm100::smem_u32(&sm.full[i]), 1);
    for (int i = 0; i < kParamSlots; ++i) sm100::mbar_init(sm100::smem_u32(&sm.pfull[i]), 1);
    sm.feed = Feed();
    sm.abort_flag = 0;
    sm100::mbar_init_fence();
  }
  {
    const uint32_t* from = reinterpret_cast<const uint32_t*>(prm.ops);
    asm volatile("" : "+l"(from));  // as memory: a constant load with an address for each thread would go one thread after the other
    uint32_t* to = reinterpret_cast<uint32_t*>(sm.ops);
#pragma unroll 1
    for (int i = tid; i < prm.n_ops * kOpWords; i += kThreads) to[i] = from[i];
  }
  __syncthreads();
#pragma unroll 1
  for (int i = tid; i < prm.n_ops; i += kThreads)
    if (sm.ops[i].kind == TTB_CHAIN_LINEAR) sm.share[i] = Share(sm.ops[i].u.linear);
  __syncthreads();
  Read read;
  if (warp == kWarps - 1) {
    feed(prm, sm, ring, Layout<MT>::kBatch, 0, 0);
    if (!wait_ahead(sm.ops[0], sm.share[0], prm.slots, sm, read.w, read.p) && lane == 0) atomicExch(prm.status, (int)TTB_ERR_DEVICE_WAIT);
  }
  __syncthreads();
#pragma unroll 1
  for (int i = 0; !sm.abort_flag;) {
    const ttb_chain_op& op = sm.ops[i];
    bool ok = true;
    if (op.kind == TTB_CHAIN_ATTENTION) {
      attention(op.u.attention, sm);
    } else if (const Share s = sm.share[i]; s.part) {
      if (op.u.linear.gamma) ok = linear_norm<MT>(op.u.linear, s, op.reserved & 0xffff, op.reserved >> 16, prm, sm, rows, ring, read);
      else ok = linear_plain<MT>(op.u.linear, s, op.reserved & 0xffff, op.reserved >> 16, prm, sm, ring, read);
    }
    if (!ok) atomicExch(prm.status, (int)TTB_ERR_DEVICE_WAIT);
    if (++i == prm.n_ops) break;
    // Everything this CTA has written becomes visible to the others, and theirs to it. Meanwhile the other warps see to what comes next.
    __syncthreads();
    if (tid == 0) {
      asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(prm.counter) : "memory");
      const int target = (int)gridDim.x * i;
      const long long t0 = clock64();
      // (polling without the acquire and fencing once behind it takes 1000 cycles longer: a fence makes a trip of its own)
      while (sm100::ld_acquire_gpu(prm.counter) < target) {
        if (sm.abort_flag) break;
        if (clock64() - t0 > sm100::kWaitCycles) {
          sm.abort_flag = 1;
          atomicExch(prm.status, (int)TTB_ERR_DEVICE_WAIT);
        }
      }
    } else if (warp == kWarps - 1) {
      feed(prm, sm, ring, Layout<MT>::kBatch, read.slots, read.params);
    } else if (warp == kWarps - 2) {
      if (!wait_ahead(sm.ops[i], sm.share[i], prm.slots, sm, read.w, read.p) && lane == 0) atomicExch(prm.status, (int)TTB_ERR_DEVICE_WAIT);
    } else if (warp >= 1 && i + 1 < prm.n_ops && sm.ops[i + 1].kind == TTB_CHAIN_ATTENTION) {
      prefetch_keys(sm.ops[i + 1].u.attention, tid - 32, (kWarps - 3) * 32);
    }
    __syncthreads();
  }
  if (warp == kWarps - 1) {  // every copy lands before the CTA's shared memory goes, also where a wait has run out
    const Feed f = sm.feed;
#pragma unroll 1
    for (int s = 0; s < prm.slots; ++s)
      if (s < f.issued) drain(sm100::smem_u32(&sm.full[s]), s < f.w.slot ? f.w.parity : f.w.parity ^ 1);
#pragma unroll 1
    for (int s = 0; s < kParamSlots; ++s)
      if (s < f.p_issued) drain(sm100::smem_u32(&sm.pfull[s]), s < f.p.slot ? f.p.parity : f.p.parity ^ 1);
  }
}

// The part of K that a ring slot holds: the largest divisor of K up to kPart that is a multiple of 64. 0: none that is worth a slot.
int part_of(int64_t K) {
  for (int64_t parts = (K + kPart - 1) / kPart; parts > 0 && K / parts >= 256; ++parts)
    if (K % parts == 0 && (K / parts) % 64 == 0) return (int)(K / parts);
  return 0;
}

// Shared memory for `rows` rows of normed_k normalised columns; the rest is the ring, of parts of `part`.
void ring_of(int rows, int normed_k, int part, ChainParams* prm) {
  prm->slot_bytes = 8 * (part * 2 + kRowPad);
  prm->a_bytes = normed_k ? (rows <= 16 ? 16 : rows <= 32 ? 32 : 64) * (normed_k * 2 + kRowPad) : 0;
  prm->slots = std::max(0, std::min(kMaxSlots, (kSmemLimit - kSharedBytes - prm->a_bytes) / prm->slot_bytes));
}

template <int MT> cudaError_t launch(ttb_ctx* ctx, const ChainParams& prm, int smem) {
  cudaError_t e = cudaFuncSetAttribute(chain_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctx->sm_count);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;  // the whole grid is resident, or the launch fails
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, chain_kernel<MT>, prm);
}

}  // namespace

extern "C" int64_t ttb_chain_rows(int64_t hidden, int64_t inner) {
  const int part_h = hidden <= kPart ? part_of(hidden) : 0, part_i = inner <= 8192 ? part_of(inner) : 0;
  if (part_h != hidden || part_i == 0) return 0;
  ChainParams prm;
  for (int rows = TTB_CHAIN_MAX_ROWS; rows >= 16; rows /= 2) {
    ring_of(rows, (int)hidden, std::max(part_h, part_i), &prm);
    if (prm.slots >= inner / part_i) return rows;
  }
  return 0;
}

extern "C" int ttb_chain_forward(ttb_ctx* ctx, int dtype, const ttb_chain_op* ops, int n_ops, void* workspace) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, dtype == TTB_F16, "chain_forward: dtype must be F16");
  TTB_REQUIRE(ctx, ops && workspace && n_ops > 0 && n_ops <= TTB_CHAIN_MAX_OPS, "chain_forward: 1 to %d operations", TTB_CHAIN_MAX_OPS);
  auto aligned = [](std::initializer_list<const void*> ps) {
    uintptr_t x = 0;
    for (const void* p : ps) x |= reinterpret_cast<uintptr_t>(p);
    return (x & 15) == 0;
  };
  ChainParams prm{};
  int rows = 0, part = 256, normed_k = 0;
  for (int i = 0; i < n_ops; ++i) {
    prm.ops[i] = ops[i];
    if (ops[i].kind == TTB_CHAIN_LINEAR) {
      const ttb_chain_linear& o = ops[i].u.linear;
      const int ks = part_of(o.K);
      TTB_REQUIRE(ctx, o.M > 0 && o.M <= TTB_CHAIN_MAX_ROWS && o.N >= 0 && o.N <= (1 << 24) && o.K > 0 && o.K <= 8192 && ks > 0, "chain_forward: operation %d: bad shape %d x %d x %d", i,
                  o.M, o.N, o.K);
      TTB_REQUIRE(ctx, o.A && o.lda >= o.K && o.lda % 8 == 0 && (o.N == 0 || (o.W && o.out && o.ldo >= o.N)) && (!o.residual || (o.ldr >= o.N && o.ldr % 2 == 0)),
                  "chain_forward: operation %d: missing operand or bad pitch", i);
      TTB_REQUIRE(ctx, aligned({o.A, o.W, o.gamma, o.beta, o.bias, o.normed}) && (reinterpret_cast<uintptr_t>(o.residual) & 3) == 0 &&
                  (reinterpret_cast<uintptr_t>(o.out) & 1) == 0, "chain_forward: operation %d: misaligned operand", i);
      TTB_REQUIRE(ctx, !o.gamma || (o.beta && ks == o.K), "chain_forward: operation %d: a layer norm takes at most %d columns and both of its weights", i, kPart);
      TTB_REQUIRE(ctx, o.N > 0 || (o.gamma && o.normed), "chain_forward: operation %d does nothing", i);
      TTB_REQUIRE(ctx, !o.normed || chain::rows_have_writers(o.M, ctx->sm_count), "chain_forward: operation %d: more rows than SMs", i);
      TTB_REQUIRE(ctx, (!o.bias && !o.residual) || o.N % 8 == 0, "chain_forward: operation %d: a bias or residual needs a width that is a multiple of 8", i);
      TTB_REQUIRE(ctx, !o.bias || o.N <= chain::bias_columns(ctx->sm_count), "chain_forward: operation %d: too wide for a bias", i);
      TTB_REQUIRE(ctx, o.act >= 0 && o.act <= TTB_CHAIN_ACT_RELU, "chain_forward: operation %d: unknown activation", i);
      prm.ops[i].reserved = ks;
      rows = std::max(rows, (int)o.M);
      part = std::max(part, ks);
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
    }
  }
  DeviceGuard g(ctx->device);
  prm.n_ops = n_ops;
  ring_of(rows, normed_k, part, &prm);
  prm.counter = static_cast<int*>(workspace);
  prm.status = ctx->d_status;
  for (int i = 0; i < n_ops; ++i)
    if (ops[i].kind == TTB_CHAIN_LINEAR) {  // a group's weights fit in the ring: they are all read before a slot is free again
      const int group = std::min(kGroup, prm.slots / (ops[i].u.linear.K / prm.ops[i].reserved));
      TTB_REQUIRE(ctx, group > 0, "chain_forward: operation %d is too deep", i);
      prm.ops[i].reserved |= group << 16;
    }
  TTB_CUDA(ctx, cudaMemsetAsync(workspace, 0, TTB_CHAIN_WORKSPACE, ctx->stream));
  const int smem = kSharedBytes + prm.a_bytes + prm.slots * prm.slot_bytes;
  if (rows <= 16) TTB_CUDA(ctx, launch<1>(ctx, prm, smem));
  else if (rows <= 32) TTB_CUDA(ctx, launch<2>(ctx, prm, smem));
  else TTB_CUDA(ctx, launch<4>(ctx, prm, smem));
  return launched(ctx, "chain_forward");
}
