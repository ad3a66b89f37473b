// Tensor-core Linear for sm_100a: out[M,N] = epilogue(sum over passes of A_p[M,K] . W_p[N,K]^T).
//
// One persistent CTA (or CTA pair) per SM, 320 to 384 threads in three roles:
//   warp 0      : TMA producer  - cp.async.bulk.tensor loads of 128-byte-swizzled K-major tiles into a
//                 shared-memory ring, completion signalled on "full" mbarriers
//   warp 1      : MMA issuer    - one elected thread issues tcgen05.mma (128 x BN x 32 bytes of K per instruction)
//                 from shared-memory descriptors into a TMEM accumulator; tcgen05.commit releases ring
//                 slots ("empty" mbarriers) and publishes finished accumulators ("tmem_full")
//   warp 10     : second issuer on tiles of up to 128 columns, with an accumulator of its own (every other k-block)
//   warp 11     : second producer on tiles of up to 64 columns, which loads W while warp 0 loads A
//   warps 2..9  : epilogue      - tcgen05.ld the accumulator (one row per thread), apply scale/bias/activation/
//                 residual in fp32, convert, stage through a swizzled shared-memory tile and TMA-store it
// Two accumulators (of BN TMEM columns, twice as many with two issuers) let the epilogue of tile i overlap the MMAs of tile i+1.
//
// Operand kinds: fp16, bf16 (kind::f16), int8 (kind::i8, int32 accumulator) and fp32 read as tf32 (kind::tf32).
// A launch may run up to three passes over K into the same accumulator, each pass reading the first or the second
// of two A maps and of two W maps. That is how operands wider than the tensor core's formats are used at full accuracy:
//   bf16 activations kept as hi + lo planes :  A_hi.W + A_lo.W                       (2 passes)
//   fp32 as three tf32 products             :  A_hi.W_hi + A_lo.W_hi + A_hi.W_lo     (3 passes)
//   fp32 as three fp16 products             :  the same, of rows that are scaled into fp16's range; the epilogue takes the scales out again
// fp16 planes hold as many bits as tf32 ones (an element to 2^-23, or to 2^-39 of its row's largest) at half the bytes and twice the rate, and a sum is
// half as many instructions, each of which truncates it: us, tf32 / fp16 planes, and error against 64 bits: 128 x 768 x 768 8.9 / 8.0, 8.3e-7 / 6.2e-7; 128 x 2304 x
// 768 11.3 / 7.9, 1.5e-6 both; 527 x 768 x 3072 33.9 / 19.6, 1.1e-5 / 5.6e-6; 3000 x 2304 x 768 45.0 / 27.8, 2.8e-6 / 1.5e-6; 3000 x 768 x 3072 63.9 / 32.2. With a row's
// elements up to 2^20 apart, and the weights' as far the other way, the errors stay so; beyond, where fp16 planes have fewer bits of the small ones, tf32 planes are
// closer (2^24 apart: 128 x 768 x 768 8.3e-7 / 1.1e-5).
// Products of few tiles with a long K are split along K over the CTAs of a cluster: every CTA accumulates its K range
// in its own TMEM, the others hand their partial tile to the first CTA through distributed shared memory, and that CTA
// adds them in rank order and runs the epilogue, so the result does not depend on timing.
// Every mbarrier wait is bounded: on expiry the CTA raises a flag, all roles fall through to the common
// teardown (TMEM is released), and the host sees TTB_ERR_DEVICE_WAIT in the status word.
#include <cuda.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <unordered_map>

#include "ttb_common.cuh"
#include "ttb_ring.cuh"
#include "ttb_sm100.cuh"

using namespace ttb;
using namespace ttb::sm100;

namespace {

constexpr int BM = 128;          // rows of A per tile == TMEM lanes
constexpr int BK_BYTES = 128;    // bytes of K per ring slot row: one 128-byte swizzle span
constexpr int UMMA_K_BYTES = 32; // K bytes consumed by one tcgen05.mma (16 x 16-bit, 32 x 8-bit, 8 x tf32)
constexpr int kThreads = 320;    // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue (two per TMEM lane quarter)
constexpr int kMaxSplit = 4;     // CTAs of a cluster that may share one tile's K range (clusters of 6 pack badly into the GPCs:
                                 // 24 of them did not fit the chip at once and the launch took two waves)

constexpr int kPrefetchBlocks = 16;  // k-blocks of the first tile's weights that are sent for ahead of the wait: K = 1024 in 16 bits

// TWO = a pair of CTAs (one cluster of two SMs) computes a 256 x BN tile with cta_group::2 MMAs: each CTA stages its
// own 128 rows of A and its own half (BN/2 rows) of W, so a k-block costs 32 KB of L2->SM traffic per CTA instead of 48.
// SK = split-K over a cluster (BN = 32 only): a shorter ring, plus room for the partial tiles of the other CTAs.
constexpr int kLnMaxTiles = 4;  // kernels with the LayerNorm epilogue: N-tiles of 256 per row, N <= 1024
// PA, PB = planes of A and W that one ring slot holds (see Planes).
template <int BN, bool TWO = false, bool SK = false, int PA = 1, int PB = 1> struct Cfg {
  static constexpr int A_BYTES = BM * BK_BYTES;
  static constexpr int B_BYTES = (TWO ? BN / 2 : BN) * BK_BYTES;
  static constexpr int STAGE_BYTES = PA * A_BYTES + PB * B_BYTES;
  static constexpr int STAGES = SK ? 4 : (192 * 1024 / STAGE_BYTES < 8 ? 192 * 1024 / STAGE_BYTES : 8);
  // Two MMA-issuing warps with an accumulator each (even and odd k-blocks) wherever a k-block's MMAs are short: see the issuer.
  static constexpr int ISSUERS = (!TWO && BN <= 128) ? 2 : 1;
  // Two TMA-issuing warps, one per operand, on the narrowest tiles: see the producer.
  static constexpr int PRODUCERS = (!TWO && BN <= 64) ? 2 : 1;
  static constexpr int THREADS = kThreads + 32 * (ISSUERS - 1) + 32 * (PRODUCERS - 1);
  static constexpr int TMEM_COLS = 2 * ISSUERS * BN;
  static_assert(PRODUCERS == 1 || ISSUERS == 2, "warp numbers: 10 issues, 11 loads");
  static_assert(TMEM_COLS >= 32 && TMEM_COLS <= 512, "TMEM allocation");
  static_assert(ISSUERS == 1 || STAGES >= ring::kMinStages, "two issuers tell a slot's uses apart by parity: see ttb_ring.cuh");
  // Epilogue staging: per epilogue warp one [32 rows x 128 B] swizzled tile that its TMA stores read (BN >= 64 only).
  static constexpr int STAGING_BYTES = (BN >= 64) ? 8 * 4096 : 0;
  static constexpr int REDUCE_BYTES = SK ? (kMaxSplit - 1) * BM * BN * 4 : 0;  // [slot][column][row] 32-bit words
  static constexpr int BAR_BYTES = 256;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + STAGING_BYTES + REDUCE_BYTES + BAR_BYTES + 1024;  // + slack for 1024-byte alignment
};

// Output of the wider tiles: STORE_DIRECT, each thread its own row from registers; STORE_TMA, through shared memory and TMA
// stores (16-byte-aligned rows of a multiple of 16 bytes); STORE_WORDS, through shared memory and word stores, 128 consecutive
// bytes of one row per instruction whatever the row's alignment.
enum { STORE_DIRECT = 0, STORE_TMA = 1, STORE_WORDS = 2 };

// Products over two planes of an operand (bf16 hi + lo; fp32 as three products). On tiles of up to 128 columns, which are bound
// by their loads, a ring slot holds both planes of a k-block and all its products are issued from there, so that no plane is
// fetched twice: fp32 520 x 768 x 3072 51.2 -> 44.7 us, 128 x 768 x 3072 27 -> 17.9, bf16 3200 x 768 x 3072 45 -> 39. Tiles of 256
// columns, bound by the MMAs, run the products as passes over K: with slots twice the size they have too few of them (bf16
// 9000 x 2304 x 768 50.6 us in passes, 60.1 from shared slots).
template <int BN, bool TWO, int KIND, typename OutT, int VAR> struct Planes {
  static constexpr bool split = KIND == KIND_F16 && VAR == 5;  // VAR_SPLIT
  static constexpr bool shared = !TWO && BN <= 128 && (KIND == KIND_TF32 || split || (KIND == KIND_BF16 && (sizeof(OutT) == 4 || VAR == 1)));
  static constexpr int A = shared ? 2 : 1;
  static constexpr int B = (shared && (KIND == KIND_TF32 || split)) ? 2 : 1;
};

struct GemmParams {
  int M, N, K;             // K in elements, per pass
  int a_rows;              // single CTAs: rows of A that a tile's load brings (fewer than BM when M is smaller; the rest is never read back)
  int npass;               // 1..3 passes over K into one accumulator
  int pass_a, pass_b;      // bit p set: pass p reads the second A map / the second W map
  void* out;
  long long ldo;
  void* out_lo;            // plane that receives what is left of v after it has been stored and read by a product (same pitch as out), or null
  const void* bias;        // OutT[N] or null
  const void* residual;    // OutT[M, ldr] or null
  long long ldr;
  const float* row_scale;  // int8, symmetric: per-row activation scale; fp32 as fp16 planes: what a row of them was divided by
  const float* col_scale;  // fp32 as fp16 planes: the same of W's rows
  const float* w_scale;    // int8: device scalar, weight scale
  const float* act_qparams;  // int8, affine per tensor: device [scale, zero point]; null selects the symmetric form
  const int* col_sum;        // int8, affine: sum over k of Wq[n, k]
  float* row_absmax;         // int8 kind, or null: [M], receives max |out[m, :]| as stored (atomic maximum; zero before the launch)
  const void* ln_gamma;      // LN kernels: OutT[N], OutT[N], eps
  const void* ln_beta;
  float ln_eps;
  float2* ln_partials;       // LN kernels: [2 * N / 256 slots][ln_rows] {sum, sum of squares} of a row over 128 columns
  int* ln_counters;          // LN kernels: per 128-row block {warps that have published, warps that have read}; all zero between launches
  long long ln_rows;         // rows of the partials array (M rounded up to whole tiles)
  int epilogue;
  int staged;              // STORE_*: how the output tile leaves (BN >= 64)
  int split_k;             // CTAs per cluster sharing one tile (SK kernels), else 1
  int* status;
};

// One 16-byte group of output elements <-> floats: 8 values for the 16-bit types, 4 for fp32.
template <typename OutT> struct Per16 { static constexpr int value = 16 / (int)sizeof(OutT); };
template <typename OutT> __device__ __forceinline__ void unpack16(const uint4& q, float* f);
template <> __device__ __forceinline__ void unpack16<__half>(const uint4& q, float* f) {
  const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __half22float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
template <> __device__ __forceinline__ void unpack16<__nv_bfloat16>(const uint4& q, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
template <> __device__ __forceinline__ void unpack16<float>(const uint4& q, float* f) {
  f[0] = __uint_as_float(q.x); f[1] = __uint_as_float(q.y); f[2] = __uint_as_float(q.z); f[3] = __uint_as_float(q.w);
}
template <typename OutT> __device__ __forceinline__ uint4 pack16(const float* f);
template <> __device__ __forceinline__ uint4 pack16<__half>(const float* f) {
  uint4 q;
  __half2* h = reinterpret_cast<__half2*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
  return q;
}
template <> __device__ __forceinline__ uint4 pack16<__nv_bfloat16>(const float* f) {
  uint4 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return q;
}
template <> __device__ __forceinline__ uint4 pack16<float>(const float* f) {
  return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
}

// Instruction descriptor: accumulator format, operand formats, both operands K-major, N>>3, M>>4.
template <int KIND, int BN, bool TWO = false> __host__ __device__ constexpr uint32_t make_idesc() {
  return (KIND == KIND_I8 ? (2u << 4) | (1u << 7) | (1u << 10)                  // S32 accumulator, signed 8-bit A and B
          : KIND == KIND_TF32 ? (1u << 4) | (2u << 7) | (2u << 10)              // F32 accumulator, TF32 A and B
                              : (1u << 4) | ((uint32_t)KIND << 7) | ((uint32_t)KIND << 10))  // F32 accumulator, F16(0)/BF16(1)
         | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((TWO ? 2 * BM : BM) >> 4) << 24);
}

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 16-bit outputs use the hardware tanh approximation (its error is below their rounding step); fp32 outputs the full one.
template <typename OutT> __device__ __forceinline__ float tanh_out(float x) { return std::is_same<OutT, float>::value ? tanhf(x) : tanh_fast(x); }
template <typename OutT> __device__ __forceinline__ float gelu_out(float x) {
  if (std::is_same<OutT, float>::value) return gelu_tanh(x);  // the fp32 models' exact form
  const float hx = 0.5f * x;  // 0.5x(1 + tanh(0.79788456(x + 0.044715x^3))), regrouped to six operations
  return fmaf(hx, tanh_fast(x * fmaf(x * x, 0.7978845608028654f * 0.044715f, 0.7978845608028654f)), hx);
}

template <typename OutT> __device__ __forceinline__ void load32(const OutT* p, float (&f)[32]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    Vec8<OutT> v;
    v.load(p + i * 8);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[i * 8 + j] = v.v[j];
  }
}

// ---- the kernel -----------------------------------------------------------------------------------
// VAR selects an epilogue variant that costs registers, so that the plain kernels do not carry it:
//   VAR_PLAIN, VAR_TWO_PLANES (output written with a second plane, what a product drops of the first), VAR_TF32_PLANES (fp32 output rounded to tf32, and
//   what that dropped; as a choice at run time of the one before, 3 us of 30 at 527 x 3072 x 768), VAR_AFFINE (int8 with a per-tensor zero point),
//   VAR_WORDS (STORE_WORDS; carried by every kernel it cost packed fp16 batches 1 %: 4120 -> 4164 us, 4149 against 4159 without)
//   VAR_SPLIT (operands are fp32 as two scaled fp16 planes)
enum { VAR_PLAIN = 0, VAR_TWO_PLANES = 1, VAR_AFFINE = 2, VAR_WORDS = 3, VAR_TF32_PLANES = 4, VAR_SPLIT = 5 };

template <int BN, int KIND, typename OutT, bool TWO, bool SK, int VAR, bool LN = false>
__global__ void __launch_bounds__(Cfg<BN, TWO, SK>::THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
               const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
               const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmO2, const GemmParams p) {
  using P = Planes<BN, TWO, KIND, OutT, VAR>;
  using C = Cfg<BN, TWO, SK, P::A, P::B>;
  constexpr bool FUSED = P::shared;  // all products of a k-block from one slot
  static_assert(!SK || (BN == 32 && !TWO), "split-K runs on single-CTA 128 x 32 tiles");
  static_assert(!LN || (BN == 256 && !SK && VAR == VAR_PLAIN && sizeof(OutT) == 2), "the LayerNorm epilogue: 16-bit 256-column tiles");
  constexpr int IN_BYTES = (KIND == KIND_I8) ? 1 : (KIND == KIND_TF32 ? 4 : 2);
  constexpr int BK_ELEMS = BK_BYTES / IN_BYTES;
  constexpr uint32_t IDESC = make_idesc<KIND, BN, TWO>();
  constexpr int TILE_M = TWO ? 2 * BM : BM;                      // output rows per tile (per CTA pair when TWO)
  pdl_trigger();  // the next kernel in the stream may start its own set-up; it waits for this grid before touching memory
  const uint32_t rank = (TWO || SK) ? cluster_ctarank() : 0u;    // 0 = the CTA that issues the MMAs (TWO) / runs the epilogue (SK)
  const int group = SK ? p.split_k : (TWO ? 2 : 1);              // CTAs that share one tile
  const int tile0 = (int)blockIdx.x / group;
  const int tile_step = (int)gridDim.x / group;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t tiles = smem_u32(smem);
  uint8_t* staging = smem + C::STAGES * C::STAGE_BYTES;  // 1024-byte aligned: the tile area is a multiple of 1024
  uint32_t* reduce_buf = reinterpret_cast<uint32_t*>(staging + C::STAGING_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + C::STAGING_BYTES + C::REDUCE_BYTES);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (C::STAGES + s); };
  auto tfull_bar = [&](int a) { return bar0 + 8u * (2 * C::STAGES + a); };
  auto tempty_bar = [&](int a) { return bar0 + 8u * (2 * C::STAGES + 2 + a); };
  const uint32_t reduce_bar = bar0 + 8u * (2 * C::STAGES + 4);   // SK: the other CTAs' partial tiles have arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::STAGES + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 32) {  // the descriptors are kernel parameters: fetching them does not depend on the previous kernel
    prefetch_tensormap(&tmA0);
    prefetch_tensormap(&tmB0);
    if (p.npass > 1) {
      prefetch_tensormap(&tmA1);
      prefetch_tensormap(&tmB1);
    }
    if (p.staged == STORE_TMA) prefetch_tensormap(&tmO);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), C::PRODUCERS);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), C::ISSUERS);
      mbar_init(tempty_bar(a), TWO ? 16 : 8);  // one arrival per epilogue warp (of both CTAs when paired)
    }
    mbar_init(reduce_bar, (SK && group > 1) ? (uint32_t)(group - 1) * 4u : 1u);  // the other CTAs' four working warps
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    if (TWO) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                   "r"((uint32_t)C::TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tmem_alloc(smem_u32(tmem_slot), (uint32_t)C::TMEM_COLS);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (TWO || SK) cluster_sync_all();  // the peers' barriers are initialised before anything signals them remotely
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int num_m = (p.M + TILE_M - 1) / TILE_M, num_n = (p.N + BN - 1) / BN;
  const int num_tiles = num_m * num_n;
  const int num_kb = (p.K + BK_ELEMS - 1) / BK_ELEMS;   // k-blocks per pass
  const int total_kb = FUSED ? num_kb : num_kb * p.npass;
  // this CTA's share of a tile's k-blocks: all of them, or (split-K) one contiguous range per cluster rank
  const int kb_begin = SK ? (int)(((long long)total_kb * rank) / group) : 0;
  const int kb_end = SK ? (int)(((long long)total_kb * (rank + 1)) / group) : total_kb;
  // The first tile's weights start on their way to L2 while the previous kernel still runs. A prefetch into L2 is not a read:
  // should that kernel write the weights, the loads below (after the wait) see what it wrote.
  // With the bias and residual fetched ahead of the sums and one arrival per warp in the split-K exchange (below), one product
  // in a row of them, us: 128 x 768 x 768 5.5 -> 5.0, 1 x 768 x 768 5.0 -> 4.8, 128 x 768 x 3072 10.1 -> 9.4; whole passes, whose
  // weights are colder: BERT-base 1 x 17 476 -> 462, GPT-2 generation, one user, 24 steps, 14.3 -> 13.5 ms with the two issuers.
  // Where many rows of tiles share the weights, the first four send for them: asked for by every CTA they are 58 MB of requests to
  // L2 for a 2.3 MB matrix, fp16 8192 x 1000 x 768 14.1 us against 13.2, int8 11000 x 768 x 3072 23.5 against 22.1. (Sent for by
  // the first row of tiles alone, BERT-base fp16 8 x 99 takes 628 us against 622 to 624; not at all 629, generation 0.6 % more.)
  if (warp == 0 && lane == 0 && tile0 < min(num_tiles, 4 * num_n)) {
    const int n_row = (tile0 % num_n) * BN + (int)(TWO ? rank : 0u) * (BN / 2);
    int pass = kb_begin / num_kb, kk = kb_begin % num_kb;
    for (int kb = kb_begin; kb < min(kb_end, kb_begin + kPrefetchBlocks) && n_row < p.N; ++kb) {
      tma_prefetch_2d(((p.pass_b >> pass) & 1) ? &tmB1 : &tmB0, kk * BK_ELEMS, n_row);
      if (FUSED && p.pass_b) tma_prefetch_2d(&tmB1, kk * BK_ELEMS, n_row);
      if (++kk == num_kb) { kk = 0; ++pass; }
    }
  }
  pdl_wait();  // everything above ran in the shadow of the previous kernel; its results are visible from here on

  if (warp == 0 || (C::PRODUCERS == 2 && warp == 11)) {
    // ------------------------------------------------------------------ TMA producer(s)
    // One thread's wait, byte count and two loads take about 320 cycles a k-block, which is what paces tiles of up to 64
    // columns (a deeper ring changes nothing). With a warp per operand, us: 792 x 768 x 3072 fp16 13.0 -> 12.3, 128 x 2304 x 768
    // 5.3 -> 5.1, fp32 520 x 768 x 3072 56.2 -> 51.2. Tiles of 128 columns are slower that way (15.2 -> 15.6).
    const bool load_a = warp == 0, load_b = C::PRODUCERS == 1 || warp != 0;
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
        const int m_blk = tile / num_n, n_blk = tile % num_n;
        int pass = kb_begin / num_kb, kk = kb_begin % num_kb;
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag)) { ok = false; break; }
          const CUtensorMap* ma = ((p.pass_a >> pass) & 1) ? &tmA1 : &tmA0;
          const CUtensorMap* mb = ((p.pass_b >> pass) & 1) ? &tmB1 : &tmB0;
          const uint32_t a_dst = tiles + stage * C::STAGE_BYTES, b_dst = a_dst + (FUSED ? 2 : 1) * C::A_BYTES;
          const bool a2 = FUSED && p.pass_a != 0, b2 = FUSED && p.pass_b != 0;  // second planes in the same slot
          if (TWO) {
            // CTA 0's barrier counts the bytes of both CTAs; only CTA 0 arms it.
            if (rank == 0) mbar_expect_tx(full_bar(stage), 2u * (uint32_t)C::STAGE_BYTES);
            tma_load_2d_pair(a_dst, ma, full_bar(stage), kk * BK_ELEMS, m_blk * TILE_M + (int)rank * BM);
            tma_load_2d_pair(b_dst, mb, full_bar(stage), kk * BK_ELEMS, n_blk * BN + (int)rank * (BN / 2));
          } else {
            mbar_expect_tx(full_bar(stage), (load_a ? (uint32_t)(p.a_rows * BK_BYTES * (a2 ? 2 : 1)) : 0u) + (load_b ? (uint32_t)(C::B_BYTES * (b2 ? 2 : 1)) : 0u));
            if (load_a) tma_load_2d(a_dst, ma, full_bar(stage), kk * BK_ELEMS, m_blk * BM);
            if (load_b) tma_load_2d(b_dst, mb, full_bar(stage), kk * BK_ELEMS, n_blk * BN);
            if (load_a && a2) tma_load_2d(a_dst + C::A_BYTES, &tmA1, full_bar(stage), kk * BK_ELEMS, m_blk * BM);
            if (load_b && b2) tma_load_2d(b_dst + C::B_BYTES, &tmB1, full_bar(stage), kk * BK_ELEMS, n_blk * BN);
          }
          if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
          if (++kk == num_kb) { kk = 0; ++pass; }
        }
      }
      if (!ok) {
        // Gave up: give copies already in flight time to land (they take microseconds) before the CTA's
        // shared memory is released. A fixed, bounded delay; nothing is waited on.
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1 || (C::ISSUERS == 2 && warp == 10)) {
    // ------------------------------------------------------------------ MMA issuer(s)
    // A thread that has issued MMAs sees its next shared-memory read (the wait for the next slot) return only once they have
    // drained: 508 cycles per k-block at N <= 128, where the MMAs themselves need 128 to 256. So the narrow tiles have two
    // issuing warps: each takes every other k-block into its own accumulator, one's wait passes under the other's MMAs, and
    // the epilogue adds the two accumulators (the order of the sums is fixed by the shape). One issuer -> two, replayed from a
    // graph, us: 600 x 2304 x 768 fp16 9.7 -> 8.5, 792 x 768 x 3072 15.4 -> 12.9, 2048 x 768 x 3072 26.4 -> 21.8, 128 x 2304 x 768
    // 5.9 -> 5.4; fp32 (three products) 520 x 768 x 3072 68.7 -> 55.6. What is left there is the SM's share of L2 bandwidth
    // (24 KB a k-block at 64 bytes a cycle). The chains of additions are half as long, too: the tensor core truncates each partial
    // sum, and whole fp32 models come out at half their distance from 64 bits (4.9e-5 -> 2.4e-5 on 8 ragged sequences).
    const int issuer = (C::ISSUERS == 2 && warp == 10) ? 1 : 0;
    if (lane == 0 && (!TWO || rank == 0)) {
      uint32_t first_kb = 0;  // k-blocks of the tiles before this one: the ring position of the tile's first
      int acc_iter = 0;
      bool ok = true;
      // Descriptors differ only in the start-address field of their low word, so the loop below advances that
      // word with one add per MMA instead of rebuilding 64-bit descriptors (this single thread's instruction
      // stream is what paces the tensor core).
      const uint32_t a_lo0 = desc_lo(tiles);
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step, ++acc_iter, first_kb += (uint32_t)(kb_end - kb_begin)) {
        const int acc = acc_iter & 1;
        const uint32_t acc_phase = (uint32_t)(acc_iter >> 1) & 1u;
        int stage = (int)((first_kb + issuer) % C::STAGES);
        uint32_t phase = ((first_kb + issuer) / C::STAGES) & 1u;
        uint32_t a_lo = a_lo0 + (uint32_t)stage * (uint32_t)(C::STAGE_BYTES >> 4);
        if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)((acc * C::ISSUERS + issuer) * BN);
        uint32_t accumulate = 0;
        for (int kb = kb_begin + issuer; kb < kb_end; kb += C::ISSUERS) {
          // a slot whose previous use was the other issuer's: see there
          if (ring::wait_for_empty_first(C::STAGES, C::ISSUERS, kb_end - kb_begin, kb - kb_begin) &&
              !mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag)) { ok = false; break; }
          if (!mbar_wait(full_bar(stage), phase, abort_flag)) { ok = false; break; }
          const uint32_t b_lo = a_lo + (uint32_t)((FUSED ? 2 : 1) * C::A_BYTES >> 4);
          for (int pass = 0; pass < (FUSED ? p.npass : 1); ++pass) {
            const uint32_t a_at = a_lo + ((FUSED && ((p.pass_a >> pass) & 1)) ? (uint32_t)(C::A_BYTES >> 4) : 0u);
            const uint32_t b_at = b_lo + ((FUSED && ((p.pass_b >> pass) & 1)) ? (uint32_t)(C::B_BYTES >> 4) : 0u);
#pragma unroll
            for (int k = 0; k < BK_BYTES / UMMA_K_BYTES; ++k) {
              umma_ss<KIND, TWO>(d_tmem, a_at + (uint32_t)(k * (UMMA_K_BYTES >> 4)), b_at + (uint32_t)(k * (UMMA_K_BYTES >> 4)), IDESC, accumulate);
              accumulate = 1;
            }
          }
          // the slot is free (in both CTAs when paired) once these MMAs have read it
          if (TWO) tc_commit_pair(empty_bar(stage));
          else tc_commit(empty_bar(stage));
          a_lo += (uint32_t)(C::ISSUERS * (C::STAGE_BYTES >> 4));
          stage += C::ISSUERS;
          if (stage >= C::STAGES) { stage -= C::STAGES; phase ^= 1u; a_lo -= (uint32_t)(C::STAGES * (C::STAGE_BYTES >> 4)); }
        }
        if (ok) {  // accumulator complete: wake the epilogue warps (of both CTAs when paired)
          if (TWO) tc_commit_pair(tfull_bar(acc));
          else tc_commit(tfull_bar(acc));
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9)
    // Two warps share each TMEM lane quarter and split the tile's staged column chunks between them, so one warp's
    // TMEM / shared-memory / store latencies are covered by the other warp on the same scheduler.
    constexpr int EB = (int)sizeof(OutT);
    constexpr int CH = 128 / EB;                 // output columns of one staged chunk: a 128-byte row (64 or 32)
    constexpr int HALVES = CH / 32;              // 32-column TMEM loads per chunk
    constexpr int G16 = 32 * EB / 16;            // 16-byte groups per row of a 32-column half (4 or 8)
    constexpr int P16 = Per16<OutT>::value;      // elements per 16-byte group (8 or 4)
    constexpr int LO_N = (VAR == VAR_TWO_PLANES || VAR == VAR_TF32_PLANES) ? 8 : 1;  // 16-byte groups of a chunk's second plane kept in registers
    static_assert(VAR != VAR_AFFINE || KIND == KIND_I8, "the zero-point correction belongs to the int8 kind");
    const int quad = warp & 3;          // TMEM lanes [32*quad, 32*quad+32) are the ones this warp may read
    const int half = (warp - 2) >> 2;   // which half of the tile's column chunks this warp takes
    const OutT* bias = static_cast<const OutT*>(p.bias);
    const OutT* residual = static_cast<const OutT*>(p.residual);
    OutT* out = static_cast<OutT*>(p.out);
    const float w_scale = (KIND == KIND_I8) ? *p.w_scale : 1.0f;
    constexpr bool affine = (VAR == VAR_AFFINE);
    const float act_scale = affine ? p.act_qparams[0] : 1.0f;
    const int zero_point = affine ? (int)p.act_qparams[1] : 0;
    constexpr bool rounded = (VAR == VAR_TF32_PLANES), two_planes = (VAR == VAR_TWO_PLANES) || rounded;
    static_assert(!rounded || EB == 4, "planes as tf32 are fp32 words");
    constexpr bool split = P::split;
    static_assert(!split || EB == 4, "computed in fp32");
    const bool vec_ok = (p.ldo % 8 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) &&
                        ((reinterpret_cast<uintptr_t>(p.out_lo) & 15) == 0) &&
                        (!bias || (reinterpret_cast<uintptr_t>(bias) & 15) == 0) &&
                        (!residual || ((p.ldr % 8 == 0) && (reinterpret_cast<uintptr_t>(residual) & 15) == 0));
    const bool use_tma = (BN >= 64) && p.staged != STORE_DIRECT;
    uint8_t* buf = staging + (warp - 2) * 4096;  // this warp's [32 rows x 128 B] staging tile
    int acc_iter = 0;
    // Pulls a tile's residual rows towards L2 ahead of time, so the epilogue's loads do not each pay a DRAM
    // round trip: lane l touches the 128-byte lines of row l that the tile covers.
    auto prefetch_residual = [&](int t) {
      if (p.epilogue != TTB_EPI_BIAS_RESIDUAL || t >= num_tiles) return;
      const int r = (t / num_n) * TILE_M + (int)((TWO ? rank : 0u) * BM) + quad * 32 + lane, c0 = (t % num_n) * BN;
      if (r >= p.M) return;
      const OutT* rp = residual + (long long)r * p.ldr + c0;
#pragma unroll
      for (int c = 0; c < BN; c += CH)
        if (c0 + c < p.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + c));
    };
    // Coalesced fetch of a [32 rows x 128 bytes] residual block: 8 lanes per 128-byte row, 4 rows per instruction.
    auto load_residual = [&](uint4 (&dst)[8], int rb, int c0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int grow = rb + i * 4 + (lane >> 3), gcol = c0 + (lane & 7) * P16;
        dst[i] = (grow < p.M && gcol < p.N) ? __ldg(reinterpret_cast<const uint4*>(residual + (long long)grow * p.ldr + gcol))
                                            : make_uint4(0, 0, 0, 0);
      }
    };
    if (!SK) prefetch_residual(tile0);
    auto release_accumulator = [&](int a) {  // one arrival per epilogue warp on the MMA-issuing CTA's barrier
      if (TWO && rank != 0) mbar_arrive_remote(tempty_bar(a), 0);
      else mbar_arrive(tempty_bar(a));
    };
    // 32 columns of the tile's sums: one accumulator, or the even and the odd k-blocks' (a tile of one k-block has no odd one)
    const bool two_acc = C::ISSUERS == 2 && kb_end - kb_begin >= 2;
    auto load_sums = [&](uint32_t addr, uint32_t (&r)[32]) {
      tmem_ld32_issue(addr, r);
      if (two_acc) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // 16 columns at a time: 48 live words instead of 64
          uint32_t r1[16];
          tmem_ld16_issue(addr + (uint32_t)(BN + 16 * h), r1);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const uint32_t w = r[16 * h + j];
            r[16 * h + j] = (KIND == KIND_I8) ? (uint32_t)((int)w + (int)r1[j]) : __float_as_uint(__uint_as_float(w) + __uint_as_float(r1[j]));
          }
        }
      } else {
        tmem_ld_wait();
      }
    };
    // accumulator word -> value before bias: int8 dequantised (symmetric per row, or affine per tensor), else as it is
    auto dequant = [&](uint32_t word, float rs, int colsum) -> float {
      if (KIND != KIND_I8) return __uint_as_float(word);
      return (float)((int)word - zero_point * colsum) * rs;
    };
    if constexpr (LN) {
      // ---- bias + residual + LayerNorm. A warp owns 32 rows x 128 columns of the tile (two staged chunks). Pass 1 builds
      // the values (accumulator + bias + residual, rounded to OutT as the separate kernels would store them), keeps them
      // packed in registers, hands the accumulator back and publishes the rows' partial sums; pass 2 normalises with the
      // sums of the whole row and stores through the staging tile and TMA. The N-tiles of a row block are consecutive
      // tiles, so the CTAs that hold them work on them at the same time (the grid is persistent and wholly resident);
      // they meet through global memory: partial sums, then a counter per 128-row block that every warp raises after
      // publishing and waits on (bounded) before reading. A second counter tells the last reader to reset both.
      const OutT* gamma = static_cast<const OutT*>(p.ln_gamma);
      const OutT* beta = static_cast<const OutT*>(p.ln_beta);
      const int warps_per_block = num_n * 8;
      const float inv_n = 1.0f / (float)p.N;
      for (int tile = tile0; tile < num_tiles; tile += tile_step, ++acc_iter) {
        const int m_blk = tile / num_n, n_blk = tile % num_n;
        const int acc = acc_iter & 1;
        const uint32_t acc_phase = (uint32_t)(acc_iter >> 1) & 1u;
        const int row_block = m_blk * (TILE_M / BM) + (int)(TWO ? rank : 0u);  // which 128 rows of the matrix this CTA holds
        const int row_base = row_block * BM + quad * 32;
        const int c_beg = half * 2;
        uint4 res[8];
        load_residual(res, row_base, n_blk * BN + c_beg * CH);  // before the wait
        if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag)) break;
        tc_fence_after();
        prefetch_residual(tile + tile_step);
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * C::ISSUERS * BN);
        uint4 vp[2][2][4];  // [chunk][32-column half][16-byte group]: the values, packed
        float sum = 0.f, sq = 0.f;
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          const int cc = c_beg + ci;
          const int col0 = n_blk * BN + cc * CH;
          if (lane == 0) bulk_wait_read<0>();  // the staging tile may still be read by the previous tile's last store
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = i * 4 + (lane >> 3), ch = lane & 7;
            *reinterpret_cast<uint4*>(buf + r * 128 + ((ch ^ (r & 7)) << 4)) = res[i];
          }
          __syncwarp();
          if (ci == 0) load_residual(res, row_base, col0 + CH);  // the second chunk's rows travel during the first
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const int colh = col0 + hh * 32;
            uint4 bq[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) bq[g] = __ldg(reinterpret_cast<const uint4*>(bias + colh + g * 8));
            uint32_t r0[32];
            tmem_ld32_issue(taddr + (uint32_t)(cc * CH + hh * 32), r0);
            tmem_ld_wait();
            if (ci == 1 && hh == 1) {  // this warp's share of the accumulator is in registers: hand it back now
              tc_fence_before();
              __syncwarp();
              if (lane == 0) release_accumulator(acc);
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              float bb[8], q[8], v[8];
              unpack16<OutT>(bq[g], bb);
              unpack16<OutT>(*reinterpret_cast<const uint4*>(buf + lane * 128 + (((hh * 4 + g) ^ (lane & 7)) << 4)), q);
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r0[g * 8 + j]) + bb[j] + q[j];
              vp[ci][hh][g] = pack16<OutT>(v);
              unpack16<OutT>(vp[ci][hh][g], v);  // the statistics are those of the rounded values
#pragma unroll
              for (int j = 0; j < 8; ++j) { sum += v[j]; sq = fmaf(v[j], v[j], sq); }
            }
          }
          __syncwarp();  // every lane has read its residual row out of the staging tile before it is written again
        }
        {
          const long long prow = (long long)row_base + lane;
          p.ln_partials[(long long)(n_blk * 2 + half) * p.ln_rows + prow] = make_float2(sum, sq);
          __syncwarp();
          int* counters = p.ln_counters + 2 * row_block;
          bool arrived = true;
          if (lane == 0) {
            __threadfence();
            atomicAdd(counters, 1);
            const long long t0 = clock64();
            while (ld_acquire_gpu(counters) < warps_per_block) {
              if (*abort_flag || clock64() - t0 > kWaitCycles) {
                *abort_flag = 1;
                arrived = false;
                break;
              }
              __nanosleep(40);
            }
          }
          if (!__all_sync(0xffffffffu, arrived)) break;
          float tsum = 0.f, tsq = 0.f;
          for (int sl = 0; sl < 2 * num_n; ++sl) {
            const float2 part = __ldcg(p.ln_partials + (long long)sl * p.ln_rows + prow);
            tsum += part.x;
            tsq += part.y;
          }
          sum = tsum;
          sq = tsq;
          __syncwarp();
          if (lane == 0 && atomicAdd(counters + 1, 1) == warps_per_block - 1) {  // the last reader leaves the block's counters at zero
            counters[0] = 0;
            counters[1] = 0;
          }
        }
        const float mean = sum * inv_n;
        const float rstd = rsqrtf(fmaxf(sq * inv_n - mean * mean, 0.f) + p.ln_eps);
        const float shift = -mean * rstd;
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          const int col0 = n_blk * BN + (c_beg + ci) * CH;
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const int col = col0 + hh * 32 + g * 8;
              float v[8], gg[8], bb[8];
              unpack16<OutT>(vp[ci][hh][g], v);
              unpack16<OutT>(__ldg(reinterpret_cast<const uint4*>(gamma + col)), gg);
              unpack16<OutT>(__ldg(reinterpret_cast<const uint4*>(beta + col)), bb);
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] = fmaf(fmaf(v[j], rstd, shift), gg[j], bb[j]);
              *reinterpret_cast<uint4*>(buf + lane * 128 + (((hh * 4 + g) ^ (lane & 7)) << 4)) = pack16<OutT>(v);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmO, smem_u32(buf), col0, row_base);
            bulk_commit();
          }
        }
      }
      if (lane == 0) bulk_wait<0>();
      __syncwarp();
    } else {
    for (int tile = tile0; tile < num_tiles; tile += tile_step, ++acc_iter) {
      const int m_blk = tile / num_n, n_blk = tile % num_n;
      const int acc = acc_iter & 1;
      const uint32_t acc_phase = (uint32_t)(acc_iter >> 1) & 1u;
      const int row_base = m_blk * TILE_M + (int)((TWO ? rank : 0u) * BM) + quad * 32;
      const int row = row_base + lane;
      constexpr int kChunks = (BN >= CH) ? BN / CH : 1;
      constexpr int kPerWarp = (kChunks >= 2) ? kChunks / 2 : 1;
      // this warp's chunks of the tile: [c_beg, c_end), clipped to the columns that exist
      const int valid_chunks = min(kChunks, (p.N - n_blk * BN + CH - 1) / CH);
      const int c_beg = (kChunks >= 2) ? half * kPerWarp : 0;
      const int c_end = (kChunks >= 2 || half == 0) ? min(c_beg + kPerWarp, valid_chunks) : 0;
      const bool staged_work = use_tma && c_beg < c_end;
      uint4 res[8];
      if (staged_work && p.epilogue == TTB_EPI_BIAS_RESIDUAL) load_residual(res, row_base, n_blk * BN + c_beg * CH);  // before the wait
      // Narrow tiles (one 32-column chunk per row): bias and residual are fetched before the wait for the sums. Behind it they
      // would add their round trip to a kernel of 5 us.
      constexpr int QN = (BN == 32) ? 32 * EB / 16 : 1;
      uint4 bias_q[QN], res_q[QN];
      const bool fetched = BN == 32 && half == 0 && vec_ok && row < p.M && n_blk * BN + 32 <= p.N && !(SK && rank != 0);
      if (fetched) {
        if (split) asm volatile("prefetch.global.L1 [%0];" ::"l"(p.col_scale + n_blk * BN));  // (registers for them are not left)
        if (p.epilogue != TTB_EPI_NONE) {
          const uint4* bp = reinterpret_cast<const uint4*>(bias + n_blk * BN);
#pragma unroll
          for (int i = 0; i < QN; ++i) bias_q[i] = bp[i];
        }
        if (p.epilogue == TTB_EPI_BIAS_RESIDUAL) {
          const uint4* rp = reinterpret_cast<const uint4*>(residual + (long long)row * p.ldr + n_blk * BN);
#pragma unroll
          for (int i = 0; i < QN; ++i) res_q[i] = rp[i];
        }
      }
      const float rs = split ? (row < p.M ? p.row_scale[row] : 1.0f) : (KIND != KIND_I8) ? 1.0f : (affine ? act_scale * w_scale : (row < p.M ? p.row_scale[row] * w_scale : 1.0f));
      if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag)) break;
      tc_fence_after();
      if (!SK) prefetch_residual(tile + tile_step);  // the next tile's rows, a whole mainloop ahead
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * C::ISSUERS * BN);
      if (use_tma || half == 1) {
        if (!staged_work) {  // nothing to do for this warp on this tile: just hand the accumulator back
          tc_fence_before();
          __syncwarp();
          if (lane == 0) release_accumulator(acc);
          continue;
        }
        // ---- one 128-byte-wide chunk of output columns at a time: TMEM -> registers -> (bias, activation, residual) ->
        //      swizzled shared memory tile -> one TMA store per warp. Residual rows are fetched with coalesced 16-byte
        //      loads (8 lanes per 128-byte row) and handed over through the same tile.
        float row_max = 0.f;  // int8 kind with p.row_absmax: largest |value| this thread produced for its row in this tile
#pragma unroll 1
        for (int cc = c_beg; cc < c_end; ++cc) {
          const int col0 = n_blk * BN + cc * CH;
          // the TMA store that last read this warp's staging tile must have finished reading it
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
          if (p.epilogue == TTB_EPI_BIAS_RESIDUAL) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int r = i * 4 + (lane >> 3), ch = lane & 7;
              *reinterpret_cast<uint4*>(buf + r * 128 + ((ch ^ (r & 7)) << 4)) = res[i];
            }
            __syncwarp();
            // the next chunk's residual rows travel while this chunk is computed
            if (cc + 1 < c_end) load_residual(res, row_base, col0 + CH);
          }
          uint4 lo_pack[LO_N];  // two-plane outputs: the chunk's "lo" values, kept until the first store has read the tile
          // 32 columns at a time, to keep the live register set small
#pragma unroll
          for (int hh = 0; hh < HALVES; ++hh) {
            const int colh = col0 + hh * 32;
            // 16-bit outputs fetch the half's bias (4 groups) ahead of the TMEM wait; fp32 outputs (8 groups) fetch each
            // group where it is added, to stay within the register budget
            uint4 bq[(EB == 2) ? G16 : 1];
            if (EB == 2 && p.epilogue != TTB_EPI_NONE) {
#pragma unroll
              for (int g = 0; g < G16; ++g)
                bq[g % ((EB == 2) ? G16 : 1)] = (colh + g * P16 < p.N) ? __ldg(reinterpret_cast<const uint4*>(bias + colh + g * P16)) : make_uint4(0, 0, 0, 0);
            }
            uint32_t r0[32];
            load_sums(taddr + (uint32_t)(cc * CH + hh * 32), r0);
            if (hh == HALVES - 1 && cc == c_end - 1) {  // this warp's share of the accumulator is in registers: hand it back now
              tc_fence_before();
              __syncwarp();
              if (lane == 0) release_accumulator(acc);
            }
            float v[32];
            if (affine) {
#pragma unroll
              for (int g = 0; g < 8; ++g) {
                const int4 cs = (colh + g * 4 < p.N) ? __ldg(reinterpret_cast<const int4*>(p.col_sum + colh + g * 4)) : make_int4(0, 0, 0, 0);
                v[g * 4 + 0] = dequant(r0[g * 4 + 0], rs, cs.x);
                v[g * 4 + 1] = dequant(r0[g * 4 + 1], rs, cs.y);
                v[g * 4 + 2] = dequant(r0[g * 4 + 2], rs, cs.z);
                v[g * 4 + 3] = dequant(r0[g * 4 + 3], rs, cs.w);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = dequant(r0[j], rs, 0);
              if constexpr (split) {  // (one power of two after the other: their product may be out of range where the result is not)
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                  const float4 cs = (colh + g * 4 < p.N) ? __ldg(reinterpret_cast<const float4*>(p.col_scale + colh + g * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                  v[g * 4 + 0] = v[g * 4 + 0] * rs * cs.x;
                  v[g * 4 + 1] = v[g * 4 + 1] * rs * cs.y;
                  v[g * 4 + 2] = v[g * 4 + 2] * rs * cs.z;
                  v[g * 4 + 3] = v[g * 4 + 3] * rs * cs.w;
                }
              }
            }
            if (p.epilogue != TTB_EPI_NONE) {
#pragma unroll
              for (int g = 0; g < G16; ++g) {
                float bb[P16];
                if (EB == 2) unpack16<OutT>(bq[g % ((EB == 2) ? G16 : 1)], bb);
                else unpack16<OutT>((colh + g * P16 < p.N) ? __ldg(reinterpret_cast<const uint4*>(bias + colh + g * P16)) : make_uint4(0, 0, 0, 0), bb);
#pragma unroll
                for (int j = 0; j < P16; ++j) v[g * P16 + j] += bb[j];
              }
            }
            if (p.epilogue == TTB_EPI_BIAS_GELU) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = gelu_out<OutT>(v[j]);
            } else if (p.epilogue == TTB_EPI_BIAS_TANH) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = tanh_out<OutT>(v[j]);
            } else if (p.epilogue == TTB_EPI_BIAS_RESIDUAL) {
#pragma unroll
              for (int g = 0; g < G16; ++g) {
                float q[P16];
                unpack16<OutT>(*reinterpret_cast<const uint4*>(buf + lane * 128 + (((hh * G16 + g) ^ (lane & 7)) << 4)), q);
#pragma unroll
                for (int j = 0; j < P16; ++j) v[g * P16 + j] += q[j];
              }
            }
            if (KIND == KIND_I8 && p.row_absmax) {
#pragma unroll
              for (int j = 0; j < 32; ++j) row_max = fmaxf(row_max, fabsf(v[j]));
            }
#pragma unroll
            for (int g = 0; g < G16; ++g) {
              float first[P16];
#pragma unroll
              for (int j = 0; j < P16; ++j) first[j] = rounded ? tf32_hi(v[g * P16 + j]) : v[g * P16 + j];
              *reinterpret_cast<uint4*>(buf + lane * 128 + (((hh * G16 + g) ^ (lane & 7)) << 4)) = pack16<OutT>(first);
            }
            if (two_planes) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = rest_of<OutT>(v[j], rounded);
#pragma unroll
              for (int g = 0; g < G16; ++g) lo_pack[(hh * G16 + g) % LO_N] = pack16<OutT>(&v[g * P16]);
            }
          }
          if constexpr (VAR == VAR_WORDS) {
            // A row whose address is not a multiple of 4 (every other row of an odd 16-bit width) is shifted by half a word on
            // the way out, and its first and last elements go out alone: nothing beyond the row's own elements is written.
            __syncwarp();
            const int n_cols = min(CH, p.N - col0), n_rows = min(32, p.M - row_base);
            auto word = [&](int r) { return *reinterpret_cast<const uint32_t*>(buf + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4); };
            if (n_rows == 32 && n_cols == CH && EB == 2) {
              // whole chunks: eight rows in flight, at most one word and one half-word store a row
#pragma unroll
              for (int r0 = 0; r0 < 32; r0 += 8) {
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = word(r0 + i);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  uint16_t* dst = reinterpret_cast<uint16_t*>(out + (long long)(row_base + r0 + i) * p.ldo + col0);
                  if ((reinterpret_cast<uintptr_t>(dst) & 2) == 0) {
                    reinterpret_cast<uint32_t*>(dst)[lane] = w[i];
                  } else {
                    const uint32_t shifted = __funnelshift_r(w[i], __shfl_down_sync(0xffffffffu, w[i], 1), 16);  // elements 2 lane + 1, 2 lane + 2
                    if (lane < 31) *reinterpret_cast<uint32_t*>(dst + 2 * lane + 1) = shifted;
                    if (lane == 0 || lane == 31) dst[lane == 0 ? 0 : CH - 1] = (uint16_t)(lane == 0 ? w[i] : w[i] >> 16);
                  }
                }
              }
              continue;
            }
            for (int r = 0; r < n_rows; ++r) {
              OutT* dst = out + (long long)(row_base + r) * p.ldo + col0;
              const uint32_t w = word(r);
              if (EB == 4) {
                if (lane < n_cols) reinterpret_cast<uint32_t*>(dst)[lane] = w;
              } else if ((reinterpret_cast<uintptr_t>(dst) & 2) == 0) {
                if (2 * lane + 1 < n_cols) reinterpret_cast<uint32_t*>(dst)[lane] = w;
                else if (2 * lane < n_cols) reinterpret_cast<uint16_t*>(dst)[2 * lane] = (uint16_t)w;
              } else {
                const uint32_t shifted = __funnelshift_r(w, __shfl_down_sync(0xffffffffu, w, 1), 16);
                if (lane < 31 && 2 * lane + 2 < n_cols) *reinterpret_cast<uint32_t*>(dst + 2 * lane + 1) = shifted;
                else if (2 * lane + 1 < n_cols) reinterpret_cast<uint16_t*>(dst)[2 * lane + 1] = (uint16_t)shifted;
                if (lane == 0) reinterpret_cast<uint16_t*>(dst)[0] = (uint16_t)w;
              }
            }
            continue;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmO, smem_u32(buf), col0, row_base);
            bulk_commit();
          }
          if (two_planes) {  // second plane through the same staging tile, once the first store has read it
            if (lane == 0) bulk_wait_read<0>();
            __syncwarp();
#pragma unroll
            for (int g = 0; g < LO_N; ++g)
              *reinterpret_cast<uint4*>(buf + lane * 128 + ((g ^ (lane & 7)) << 4)) = lo_pack[g];
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmO2, smem_u32(buf), col0, row_base);
              bulk_commit();
            }
          }
        }
        // rounding to OutT is monotonic, so the maximum of the stored values is the rounded maximum; non-negative floats
        // order like their bit patterns
        if (KIND == KIND_I8 && p.row_absmax && row < p.M)
          atomicMax(reinterpret_cast<int*>(p.row_absmax + row), __float_as_int(to_f(from_f<OutT>(row_max))));
        continue;
      }
      // ---- direct path (narrow tiles or unaligned output): the first warp of each lane quarter walks the tile
      bool gave_up = false;
      float row_max = 0.f;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        load_sums(taddr + (uint32_t)(c * 32), r);
        const int col0 = n_blk * BN + c * 32;
        if (SK && group > 1) {
          // Split-K: ranks > 0 hand their partial tile to rank 0's shared memory ([slot][column][row] words, so a warp's
          // 32 rows of one column are one 128-byte line) and are done; rank 0 adds the slots in rank order.
          const int trow = quad * 32 + lane;
          if (rank != 0) {
            const uint32_t dst = map_to_rank(smem_u32(reduce_buf), 0) + (uint32_t)((((int)rank - 1) * BN * BM + trow) * 4);
#pragma unroll
            for (int j = 0; j < 32; ++j) st_cluster_f32(dst + (uint32_t)(j * BM * 4), __uint_as_float(r[j]));
            __syncwarp();  // orders the other lanes' stores before lane 0's release at cluster scope (which is cumulative)
            if (lane == 0) mbar_arrive_remote(reduce_bar, 0);  // one arrival per warp: 128 per CTA queued up on one barrier word
            continue;
          }
          if (!mbar_wait_cluster(reduce_bar, 0, abort_flag)) { gave_up = true; break; }
          for (int s = 0; s < group - 1; ++s) {
            const uint32_t* src = reduce_buf + s * BN * BM + trow;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (KIND == KIND_I8) r[j] = (uint32_t)((int)r[j] + (int)src[j * BM]);
              else r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(src[j * BM]));
            }
          }
        }
        if (row >= p.M || col0 >= p.N) continue;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = dequant(r[j], rs, (affine && col0 + j < p.N) ? p.col_sum[col0 + j] : 0);
        const bool full = vec_ok && (col0 + 32 <= p.N);
        if constexpr (split) {
          if (full) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 cs = reinterpret_cast<const float4*>(p.col_scale + col0)[i];
              v[i * 4 + 0] = v[i * 4 + 0] * rs * cs.x;
              v[i * 4 + 1] = v[i * 4 + 1] * rs * cs.y;
              v[i * 4 + 2] = v[i * 4 + 2] * rs * cs.z;
              v[i * 4 + 3] = v[i * 4 + 3] * rs * cs.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] * rs * (col0 + j < p.N ? p.col_scale[col0 + j] : 0.f);
          }
        }
        if (p.epilogue != TTB_EPI_NONE) {
          float b[32];
          if (BN == 32 && full) {
#pragma unroll
            for (int i = 0; i < QN; ++i) unpack16<OutT>(bias_q[i], b + i * P16);
          } else if (full) {
            load32<OutT>(bias + col0, b);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) b[j] = (col0 + j < p.N) ? to_f(bias[col0 + j]) : 0.f;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += b[j];
        }
        if (p.epilogue == TTB_EPI_BIAS_GELU) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = gelu_out<OutT>(v[j]);
        } else if (p.epilogue == TTB_EPI_BIAS_TANH) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = tanh_out<OutT>(v[j]);
        } else if (p.epilogue == TTB_EPI_BIAS_RESIDUAL) {
          const OutT* rp = residual + (long long)row * p.ldr + col0;
          float q[32];
          if (BN == 32 && full) {
#pragma unroll
            for (int i = 0; i < QN; ++i) unpack16<OutT>(res_q[i], q + i * P16);
          } else if (full) {
            load32<OutT>(rp, q);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) q[j] = (col0 + j < p.N) ? to_f(rp[j]) : 0.f;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += q[j];
        }
        if (KIND == KIND_I8 && p.row_absmax) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (col0 + j < p.N) row_max = fmaxf(row_max, fabsf(v[j]));
        }
#pragma unroll 1
        for (int plane = 0; plane < (two_planes ? 2 : 1); ++plane) {
          OutT* dstp = (plane == 0 ? out : static_cast<OutT*>(p.out_lo)) + (long long)row * p.ldo + col0;
          if (plane == 1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = rest_of<OutT>(v[j], rounded);
          }
          auto value = [&](float x) { return rounded && plane == 0 ? tf32_hi(x) : x; };
          if (full) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              Vec8<OutT> o;
#pragma unroll
              for (int j = 0; j < 8; ++j) o.v[j] = value(v[i * 8 + j]);
              o.store(dstp + i * 8);
            }
          } else if (BN == 32 && EB == 2 && col0 + 32 <= p.N) {
            // A whole chunk of a row that is not 16-byte aligned: words, shifted by half a word where the row is. Element by
            // element, 200 x 772 x 768 in fp16 takes 8.8 us, so 5.6; 300 x 130 x 1024 9.3, 5.9; 1024 x 65 x 768 8.7, 5.6.
            uint4 q4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) q4[i] = pack16<OutT>(&v[(i * 8) % 32]);
            const uint32_t w[16] = {q4[0].x, q4[0].y, q4[0].z, q4[0].w, q4[1].x, q4[1].y, q4[1].z, q4[1].w,
                                    q4[2].x, q4[2].y, q4[2].z, q4[2].w, q4[3].x, q4[3].y, q4[3].z, q4[3].w};
            if ((reinterpret_cast<uintptr_t>(dstp) & 2) == 0) {
#pragma unroll
              for (int j = 0; j < 16; ++j) reinterpret_cast<uint32_t*>(dstp)[j] = w[j];
            } else {
              uint16_t* d16 = reinterpret_cast<uint16_t*>(dstp);
              d16[0] = (uint16_t)w[0];
#pragma unroll
              for (int j = 0; j < 15; ++j) *reinterpret_cast<uint32_t*>(d16 + 2 * j + 1) = __funnelshift_r(w[j], w[j + 1], 16);
              d16[31] = (uint16_t)(w[15] >> 16);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) dstp[j] = from_f<OutT>(value(v[j]));
          }
        }
      }
      if (gave_up) break;
      if (KIND == KIND_I8 && p.row_absmax && row < p.M && !(SK && group > 1 && rank != 0))
        atomicMax(reinterpret_cast<int*>(p.row_absmax + row), __float_as_int(to_f(from_f<OutT>(row_max))));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) release_accumulator(acc);
    }
    // every TMA store issued by this warp must be complete before its shared memory goes away
    if (use_tma && lane == 0) bulk_wait<0>();
    __syncwarp();
    }
  }

  // ------------------------------------------------------------------ teardown (all roles reach this)
  tc_fence_before();
  __syncthreads();
  if (TWO || SK) cluster_sync_all();  // no CTA leaves while another may still read its shared memory or signal its barriers
  if (warp == 1) {
    tc_fence_after();
    if (TWO) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::TMEM_COLS) : "memory");
    else tmem_dealloc(tmem_base, (uint32_t)C::TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(p.status, (int)TTB_ERR_DEVICE_WAIT);
}

// ---- host side ------------------------------------------------------------------------------------
// Encoded tensor maps are a pure function of (address, shape, pitch, box, element type): weights keep theirs for the life
// of the model and the pool hands activations the same addresses step after step, so they are cached per process.
struct MapKey {
  const void* ptr;
  int64_t rows, k, ld;
  int box_rows, elem_kind;
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && rows == o.rows && k == o.k && ld == o.ld && box_rows == o.box_rows && elem_kind == o.elem_kind;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& m) const {
    size_t h = std::hash<const void*>()(m.ptr);
    auto mix = [&](uint64_t v) { h ^= std::hash<uint64_t>()(v) + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2); };
    mix((uint64_t)m.rows);
    mix((uint64_t)m.k);
    mix((uint64_t)m.ld);
    mix(((uint64_t)m.box_rows << 8) | (uint64_t)m.elem_kind);
    return h;
  }
};
std::mutex g_map_mu;
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_map_cache;

// 2-D row-major matrix [rows, k] with `ld` elements between rows; box = [box_rows, 128 bytes of k], 128-byte swizzle.
// Used for both operands (K-major tiles) and for the output (32-row x 128-byte store boxes).
// elem_kind: KIND_F16, KIND_BF16, KIND_I8 (one byte) or KIND_TF32 (fp32 words).
int make_map(ttb_ctx* ctx, CUtensorMap* map, int elem_kind, const void* ptr, int64_t rows, int64_t k, int64_t ld, int box_rows) {
  const MapKey key{ptr, rows, k, ld, box_rows, elem_kind};
  {
    std::lock_guard<std::mutex> g(g_map_mu);
    auto it = g_map_cache.find(key);
    if (it != g_map_cache.end()) {
      *map = it->second;
      return TTB_OK;
    }
  }
  const int es = elem_kind == KIND_I8 ? 1 : (elem_kind == KIND_TF32 ? 4 : 2);
  if (!encode_tile_map(map, ptr, es, elem_kind == KIND_BF16, (uint64_t)rows, (uint64_t)k, (uint64_t)ld, (uint32_t)box_rows))
    return fail(ctx, TTB_ERR_CUDA, "cuTensorMapEncodeTiled failed or is unavailable (rows=%lld k=%lld ld=%lld elem_bytes=%d)", (long long)rows,
                (long long)k, (long long)ld, es);
  std::lock_guard<std::mutex> g(g_map_mu);
  if (g_map_cache.size() >= 16384) g_map_cache.clear();
  g_map_cache.emplace(key, *map);
  return TTB_OK;
}

template <typename OutT> constexpr int out_kind() {
  return std::is_same<OutT, float>::value ? (int)KIND_TF32 : (std::is_same<OutT, __nv_bfloat16>::value ? (int)KIND_BF16 : (int)KIND_F16);
}

struct Operands {
  const void* A;   // [M, K], pitch lda
  const void* A2;  // second A plane or null
  int64_t lda;
  const void* W;   // [N, K] K-major
  const void* W2;  // second W plane or null
};

// Whether 16-byte stores can write the output's rows. The staged epilogue reads bias and residual one 16-byte group at a time, and
// a TMA store clips a row at 16-byte granularity: with a ragged N it writes zeros into the columns up to the next multiple of 16
// bytes. So a ragged N takes this route only without bias/residual and when the caller declared those columns scratch (p.staged on
// entry).
template <typename OutT> bool whole_rows(const GemmParams& p) {
  constexpr int EA = (int)sizeof(OutT) == 4 ? 4 : 8;  // output elements per 16 bytes
  const bool aligned16 = ((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.out_lo) | reinterpret_cast<uintptr_t>(p.bias) |
                           reinterpret_cast<uintptr_t>(p.residual) | reinterpret_cast<uintptr_t>(p.col_sum)) & 15) == 0;
  return aligned16 && p.ldo % EA == 0 && (p.N % EA == 0 || (p.epilogue == TTB_EPI_NONE && p.staged == STORE_TMA && !p.out_lo)) &&
         (!p.residual || p.ldr % EA == 0);
}

template <int BN, int KIND, typename OutT, bool TWO, bool SK, int VAR>
int launch_tc(ttb_ctx* ctx, const Operands& op, const GemmParams& p) {
  using P = Planes<BN, TWO, KIND, OutT, VAR>;
  using C = Cfg<BN, TWO, SK, P::A, P::B>;
  constexpr int TILE_M = TWO ? 2 * BM : BM;
  CUtensorMap tmA0, tmA1, tmB0, tmB1;
  // a few rows (decoding): a box of 32 or 64 rows, so that a slot is not filled up with zeros first
  const int a_rows = (TWO || p.M > 64) ? BM : (p.M > 32 ? 64 : 32);
  int s = make_map(ctx, &tmA0, KIND, op.A, p.M, p.K, op.lda, a_rows);
  if (s) return s;
  tmA1 = tmA0;
  if (op.A2 && (s = make_map(ctx, &tmA1, KIND, op.A2, p.M, p.K, op.lda, a_rows))) return s;
  s = make_map(ctx, &tmB0, KIND, op.W, p.N, p.K, p.K, TWO ? BN / 2 : BN);
  if (s) return s;
  tmB1 = tmB0;
  if (op.W2 && (s = make_map(ctx, &tmB1, KIND, op.W2, p.N, p.K, p.K, TWO ? BN / 2 : BN))) return s;
  GemmParams q = p;
  q.a_rows = a_rows;
  CUtensorMap tmO = tmA0, tmO2 = tmA0;  // placeholders when the direct-store epilogue is used
  const bool tma = BN >= 64 && whole_rows<OutT>(p);
  // Ragged or misaligned rows without bias, residual or second plane (a 50257-wide vocabulary): word stores.
  // 8192 x 50257 x 768 in fp16 into a contiguous tensor: 845 us, against about 560 into padded rows and 585 for the pass that
  // compacted them. What is left over the padded form are the partial 32-byte sectors at both ends of each 128 bytes.
  const bool words = BN >= 64 && !tma && p.epilogue == TTB_EPI_NONE && !p.out_lo && !P::split;
  if constexpr (VAR == VAR_PLAIN && BN >= 64) {
    if (words) return launch_tc<BN, KIND, OutT, TWO, SK, VAR_WORDS>(ctx, op, p);
  }
  q.staged = tma ? STORE_TMA : (VAR == VAR_WORDS ? STORE_WORDS : STORE_DIRECT);
  if (tma) {
    s = make_map(ctx, &tmO, out_kind<OutT>(), p.out, p.M, p.N, p.ldo, 32);
    if (s) return s;
    if (p.out_lo && (s = make_map(ctx, &tmO2, out_kind<OutT>(), p.out_lo, p.M, p.N, p.ldo, 32))) return s;
  }
  auto kern = gemm_tc_kernel<BN, KIND, OutT, TWO, SK, VAR>;
  static bool configured[64] = {};  // per instantiation and device
  static int max_clusters[64] = {};
  const int dev = ctx->device < 64 ? ctx->device : 63;
  if (ctx->device >= 64 || !configured[dev]) {
    TTB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    if (TWO) {
      cudaLaunchConfig_t probe = {};
      probe.gridDim = dim3(2 * (unsigned)ctx->sm_count);
      probe.blockDim = dim3(C::THREADS);
      probe.dynamicSmemBytes = C::SMEM_BYTES;
      cudaLaunchAttribute pa[1];
      pa[0].id = cudaLaunchAttributeClusterDimension;
      pa[0].val.clusterDim.x = 2;
      pa[0].val.clusterDim.y = 1;
      pa[0].val.clusterDim.z = 1;
      probe.attrs = pa;
      probe.numAttrs = 1;
      int n = 0;
      TTB_CUDA(ctx, cudaOccupancyMaxActiveClusters(&n, kern, &probe));
      max_clusters[dev] = n > 0 ? n : 1;
    }
    configured[dev] = true;
  }
  const int64_t num_tiles = ((p.M + TILE_M - 1) / TILE_M) * (int64_t)((p.N + BN - 1) / BN);
  if (!TWO && !SK) {
    const int grid = (int)(num_tiles < ctx->sm_count ? num_tiles : ctx->sm_count);
    cudaError_t e = launch_pdl(kern, dim3((unsigned)grid), dim3(C::THREADS), C::SMEM_BYTES, ctx->stream, tmA0, tmA1, tmB0, tmB1, tmO, tmO2, q);
    if (e != cudaSuccess) return fail(ctx, TTB_ERR_CUDA, "launch of gemm_tc failed: %s", cudaGetErrorString(e));
    return launched(ctx, "gemm_tc");
  }
  const int group = SK ? p.split_k : 2;
  const int clusters = SK ? (int)num_tiles : (int)(num_tiles < max_clusters[dev] ? num_tiles : max_clusters[dev]);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(group * clusters));
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)group;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tmA0, tmA1, tmB0, tmB1, tmO, tmO2, q);
  if (e != cudaSuccess) return fail(ctx, TTB_ERR_CUDA, "cluster launch of gemm_tc failed: %s", cudaGetErrorString(e));
  return launched(ctx, SK ? "gemm_tc_splitk" : "gemm_tc_pair");
}

// The GEMM whose epilogue is bias + residual + LayerNorm (N a multiple of 256, at most 1024), on the same persistent tile
// schedule as the plain kernels. Returns TTB_ERR_UNSUPPORTED (nothing launched) when its workspace cannot be had right now
// (it would have to grow while the stream is being captured); the caller then runs the product and the LayerNorm as two
// kernels.
constexpr size_t ln_ws_bytes(size_t rows) { return 2 * kLnMaxTiles * rows * sizeof(float2) + (rows / BM) * 2 * sizeof(int); }

int ensure_ln_workspace(ttb_ctx* ctx, size_t rows) {
  if (ctx->ln_ws && ctx->ln_ws_rows >= rows) return TTB_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return TTB_ERR_UNSUPPORTED;
  }
  size_t want = ctx->ln_ws_rows ? ctx->ln_ws_rows : 32768;
  while (want < rows) want *= 2;
  TTB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // nothing may still be using the old one
  if (ctx->ln_ws) cudaFree(ctx->ln_ws);
  ctx->ln_ws = nullptr;
  ctx->ln_ws_rows = 0;
  void* ws = nullptr;
  TTB_CUDA(ctx, cudaMalloc(&ws, ln_ws_bytes(want)));
  TTB_CUDA(ctx, cudaMemset(ws, 0, ln_ws_bytes(want)));
  ctx->ln_ws = ws;
  ctx->ln_ws_rows = want;
  return TTB_OK;
}

template <int KIND, typename OutT, bool TWO>
int launch_tc_ln(ttb_ctx* ctx, const Operands& op, const GemmParams& p) {
  using C = Cfg<256, TWO, false>;
  constexpr int BN = 256;
  constexpr int TILE_M = TWO ? 2 * BM : BM;
  const int64_t num_m = (p.M + TILE_M - 1) / TILE_M;
  const int num_n = p.N / BN;
  const size_t rows = (size_t)num_m * TILE_M;
  int s = ensure_ln_workspace(ctx, rows);
  if (s) return s;
  CUtensorMap tmA0, tmB0, tmO;
  if ((s = make_map(ctx, &tmA0, KIND, op.A, p.M, p.K, op.lda, BM))) return s;
  if ((s = make_map(ctx, &tmB0, KIND, op.W, p.N, p.K, p.K, TWO ? BN / 2 : BN))) return s;
  if ((s = make_map(ctx, &tmO, out_kind<OutT>(), p.out, p.M, p.N, p.ldo, 32))) return s;
  GemmParams q = p;
  q.staged = STORE_TMA;
  q.a_rows = BM;
  q.ln_partials = static_cast<float2*>(ctx->ln_ws);
  q.ln_rows = (long long)ctx->ln_ws_rows;
  q.ln_counters = reinterpret_cast<int*>(static_cast<char*>(ctx->ln_ws) + 2 * kLnMaxTiles * ctx->ln_ws_rows * sizeof(float2));
  auto kern = gemm_tc_kernel<256, KIND, OutT, TWO, false, VAR_PLAIN, true>;
  static int resident[64] = {};  // per instantiation and device: CTAs (single) or CTA pairs (TWO) the device holds at once
  const int dev = ctx->device < 64 ? ctx->device : 63;
  if (ctx->device >= 64 || resident[dev] == 0) {
    TTB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    int n = ctx->sm_count;
    if (TWO) {
      cudaLaunchConfig_t probe = {};
      probe.gridDim = dim3(2 * (unsigned)ctx->sm_count);
      probe.blockDim = dim3(kThreads);
      probe.dynamicSmemBytes = C::SMEM_BYTES;
      cudaLaunchAttribute pa[1];
      pa[0].id = cudaLaunchAttributeClusterDimension;
      pa[0].val.clusterDim.x = 2;
      pa[0].val.clusterDim.y = 1;
      pa[0].val.clusterDim.z = 1;
      probe.attrs = pa;
      probe.numAttrs = 1;
      TTB_CUDA(ctx, cudaOccupancyMaxActiveClusters(&n, kern, &probe));
    }
    resident[dev] = n > 0 ? n : 1;
  }
  // Every CTA must be resident: the CTAs that hold one row block wait for one another. Whole row blocks per round also keep
  // the N-tiles of a block in the same round.
  const int64_t num_tiles = num_m * num_n;
  int64_t units = num_tiles < resident[dev] ? num_tiles : (resident[dev] / num_n) * num_n;
  if (units < num_n) return TTB_ERR_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units * (TWO ? 2 : 1)));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (TWO) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 2;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tmA0, tmA0, tmB0, tmB0, tmO, tmO, q);
  if (e != cudaSuccess) return fail(ctx, TTB_ERR_CUDA, "launch of gemm_tc (LayerNorm epilogue) failed: %s", cudaGetErrorString(e));
  return launched(ctx, "gemm_tc_layernorm");
}

// TTB_GEMM_PAIR: 0 disables the two-CTA variant, 2 uses it for every shape with at least half a wave of pair tiles
// (measurement switches); unset = chosen by shape. TTB_GEMM_SPLITK=0 disables split-K.
int pair_mode() {
  static const int mode = [] {
    const char* e = getenv("TTB_GEMM_PAIR");
    return (e && e[0] == '0') ? 0 : ((e && e[0] == '2') ? 2 : 1);
  }();
  return mode;
}
// TTB_GEMM_SPLITK: 0 disables split-K, 2..6 caps the number of CTAs that share a tile (measurement switch).
int splitk_cap() {
  static const int cap = [] {
    const char* e = getenv("TTB_GEMM_SPLITK");
    if (!e || !e[0]) return kMaxSplit;
    const int v = atoi(e);
    return v <= 1 ? 1 : (v > kMaxSplit ? kMaxSplit : v);
  }();
  return cap;
}

// Clusters of `split` CTAs of the split-K kernel that can be resident on the device at once (cached per device and size).
template <int KIND, typename OutT, int VAR>
int max_resident_clusters(ttb_ctx* ctx, int split) {
  using P = Planes<32, false, KIND, OutT, VAR>;
  using C = Cfg<32, false, true, P::A, P::B>;
  static int cached[64][kMaxSplit + 1] = {};
  const int dev = ctx->device < 64 ? ctx->device : 63;
  if (ctx->device < 64 && cached[dev][split] != 0) return cached[dev][split] > 0 ? cached[dev][split] : 0;
  auto kern = gemm_tc_kernel<32, KIND, OutT, false, true, VAR>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t probe = {};
  probe.gridDim = dim3((unsigned)(split * ctx->sm_count));
  probe.blockDim = dim3(C::THREADS);
  probe.dynamicSmemBytes = C::SMEM_BYTES;
  cudaLaunchAttribute pa[1];
  pa[0].id = cudaLaunchAttributeClusterDimension;
  pa[0].val.clusterDim.x = (unsigned)split;
  pa[0].val.clusterDim.y = 1;
  pa[0].val.clusterDim.z = 1;
  probe.attrs = pa;
  probe.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &probe) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  if (ctx->device < 64) cached[dev][split] = n > 0 ? n : -1;
  return n;
}

// Which kernel runs a product: the tile's columns, the CTAs that share one (2 = a pair on 256 x 256, split_k = CTAs along K).
struct TilePlan {
  int columns, split_k;
  bool pair;
  int64_t tiles, slots;  // tiles of the product, and how many run at a time
};

// What a kernel is expected to take, in nanoseconds: `fixed` for the launch, the fill of its ring and its last epilogue, and for
// each wave of tiles over the chip its k-blocks or, where that takes longer, its epilogue. A k-block is 128 bytes of every row
// whatever the type, and costs the same; with two or three products issued from one slot it costs per_kb[1] or [2].
struct TileCost {
  int fixed;
  int per_kb[3];
  int epilogue[2];  // 16-bit rows; fp32 rows or two planes
  // Rows that no 16-byte store can write leave in words, one row after the other: `first` and `row` for each of them, up to the 32
  // that a warp has (from shared memory, wider tiles) or for all that the tile has (from registers, 32 columns).
  int first, row, most;
};
// Fitted to graph-replayed runs of every kernel on M = 1 .. 18424 by 18 pairs (N, K) from 128 x 128 to 4096 x 1024, 768 x 3072 and
// a vocabulary, in fp16, int8, bf16 as two products (16-bit, two-plane and fp32 outputs) and fp32 as three: 1914 shapes. The kernel
// chosen is on average 0.3 % slower than the best one; the widest tile that still gives every SM one would be 5 % slower.
// (Constants fitted to single products of BERT-base widths alone took the narrow tiles' shared slots to be cheaper than they are:
// bf16 4096 x 3072 x 768 37.7 us, 33.3 in pairs; fp32 4096 x 2304 x 768 63.3, 56.1.) fp32 as three products of fp16 planes, which came later, on M = 1 .. 6000 by 15
// pairs (N, K) from 256 x 256 to 1024 x 4096: on average 0.2 % slower than the best one, 8 to 10 % where pairs would just pay (3000 x 3072 x 768 36.4, 33.6 us in pairs).
constexpr TileCost kCostPair = {8900, {265, 0, 0}, {1050, 3700}, 500, 230, 32};
constexpr TileCost kCost256 = {5150, {385, 0, 0}, {2950, 6750}, 1000, 240, 32};
constexpr TileCost kCost128 = {2750, {255, 430, 520}, {2250, 3500}, 1200, 110, 32};
constexpr TileCost kCost64 = {2150, {230, 345, 430}, {1850, 1900}, 1200, 120, 32};
constexpr TileCost kCost32 = {2100, {200, 280, 405}, {1100, 1550}, 500, 13, 128};
constexpr int kCostSplit = 5650, kCostSplitCta = 280;  // instead of kCost32.fixed: a cluster launch and the exchange

// words: rows that no 16-byte store can write (ragged or misaligned).
template <int KIND, typename OutT, int VAR>
TilePlan choose_tile(ttb_ctx* ctx, int64_t M, int64_t N, int64_t K, int npass, bool words) {
  constexpr int IN_BYTES = (KIND == KIND_I8) ? 1 : (KIND == KIND_TF32 ? 4 : 2);
  constexpr bool fused = Planes<32, false, KIND, OutT, VAR>::shared;
  const int64_t sms = ctx->sm_count, num_m = (M + BM - 1) / BM;
  auto tiles = [&](int bn) { return num_m * ((N + bn - 1) / bn); };
  const int64_t pair_tiles = ((M + 2 * BM - 1) / (2 * BM)) * ((N + 255) / 256);
  const int64_t num_kb = (K * IN_BYTES + BK_BYTES - 1) / BK_BYTES;
  const int64_t wide_kb = num_kb * npass;                    // pairs and 256 columns: the products as passes over K
  const int64_t narrow_kb = fused ? num_kb : wide_kb;
  const int products = fused ? npass - 1 : 0;                // index of per_kb
  const int store = (sizeof(OutT) == 4 || VAR == VAR_TWO_PLANES) ? 1 : 0;
  auto epilogue = [&](const TileCost& c) -> int64_t {  // of an average tile: the last row of tiles may have few rows
    if (!words) return c.epilogue[store];
    const int64_t rest = M % BM, full = M / BM;
    return (full * (c.first + c.row * c.most) + (rest ? c.first + c.row * std::min<int64_t>(rest, c.most) : 0)) / num_m;
  };
  // Pairs lose where both the mainloop and the row of tiles are short (bias + residual epilogue: N = K = 768, M = 18424 25.7 us
  // single against 26.3 paired; N = K = 1024, M = 16384 37.1 against 35.8) and where a tile is bound by its epilogue (int8,
  // K = 768: 8000 x 3072 24.9 single, 27.5 paired).
  const int64_t k_bytes = K * IN_BYTES * npass;
  const bool pair_pays = k_bytes >= 4096 || (k_bytes >= 1536 && N >= 1536) || (k_bytes >= 2048 && N >= 1024);
  const TilePlan pair{256, 1, true, pair_tiles, sms / 2};
  if (pair_mode() == 2 && pair_tiles >= sms / 2) return pair;
  TilePlan best{};
  int64_t best_ns = INT64_MAX;
  auto consider = [&](const TilePlan& plan, int64_t fixed, const TileCost& c, int n_products, int64_t kb) {
    const int64_t waves = (plan.tiles + plan.slots - 1) / plan.slots;
    const int64_t ns = fixed + waves * std::max<int64_t>(c.per_kb[n_products] * kb, epilogue(c));
    if (ns < best_ns) { best = plan; best_ns = ns; }
  };
  if (pair_mode() && pair_pays) consider(pair, kCostPair.fixed, kCostPair, 0, wide_kb);
  consider({256, 1, false, tiles(256), sms}, kCost256.fixed, kCost256, 0, wide_kb);
  consider({128, 1, false, tiles(128), sms}, kCost128.fixed, kCost128, products, narrow_kb);
  consider({64, 1, false, tiles(64), sms}, kCost64.fixed, kCost64, products, narrow_kb);
  const int64_t t32 = tiles(32);
  consider({32, 1, false, t32, sms}, kCost32.fixed, kCost32, products, narrow_kb);
  auto splits = [&](int s) { return t32 * s <= sms && s <= narrow_kb / 2 && t32 <= max_resident_clusters<KIND, OutT, VAR>(ctx, s); };
  // Few 128 x 32 tiles: the CTAs of a cluster may share each tile's K range, two k-blocks or more each, so that the weights
  // stream through (nearly) all SMs instead of a few. At M = 128, K = 3072 (48 k-blocks): 15.6 us in one CTA per tile, 8.7 split
  // four ways. All clusters must be resident at once (one wave): how many the device holds depends on how they pack into its GPCs.
  for (int s = splitk_cap(); s >= 2; --s) {
    if (splits(s)) consider({32, s, false, t32, t32}, kCostSplit + kCostSplitCta * (s - 1), kCost32, products, (narrow_kb + s - 1) / s);
  }
  // fp32 as fp16 planes: where tf32 planes, with twice the k-blocks, pay for three CTAs along K and more, one less here, so that no accumulator adds up more
  // products than with those (the tensor core truncates each sum). us and error, tf32 / fp16 in one CTA / in three: 128 x 768 x 768 8.9, 8.3e-7 / 7.6, 1.5e-6 /
  // 8.0, 6.2e-7; 64 x 512 x 512 6.9, 6.0e-7 / 6.0, 1.1e-6 / 6.6, 5.2e-7. (For two tf32 CTAs and one of fp16 the errors are the same.)
  if constexpr (VAR == VAR_SPLIT) {
    int s = choose_tile<KIND_TF32, OutT, VAR_PLAIN>(ctx, M, N, K, npass, words).split_k - 1;
    if (s >= 2 && best.split_k < s) {
      while (s >= 2 && !splits(s)) --s;
      if (s >= 2 && best.split_k < s) return {32, s, false, t32, t32};
    }
  }
  return best;
}

template <int KIND, typename OutT, int VAR = VAR_PLAIN>
int pick_tile(ttb_ctx* ctx, const Operands& op, GemmParams& p) {
  const TilePlan plan = choose_tile<KIND, OutT, VAR>(ctx, p.M, p.N, p.K, p.npass, !whole_rows<OutT>(p));
  p.split_k = plan.split_k;
  if (plan.pair) return launch_tc<256, KIND, OutT, true, false, VAR>(ctx, op, p);
  if (plan.split_k > 1) return launch_tc<32, KIND, OutT, false, true, VAR>(ctx, op, p);
  switch (plan.columns) {
    case 256: return launch_tc<256, KIND, OutT, false, false, VAR>(ctx, op, p);
    case 128: return launch_tc<128, KIND, OutT, false, false, VAR>(ctx, op, p);
    case 64: return launch_tc<64, KIND, OutT, false, false, VAR>(ctx, op, p);
    default: return launch_tc<32, KIND, OutT, false, false, VAR>(ctx, op, p);
  }
}

int check_linear(ttb_ctx* ctx, const char* what, const void* A, const void* W, const void* bias, const void* residual,
                 int64_t M, int64_t N, int64_t K, int epilogue, const void* out, int64_t ldo, int k_align) {
  TTB_REQUIRE(ctx, M >= 0 && N > 0 && K > 0, "%s: bad shape M=%lld N=%lld K=%lld", what, (long long)M, (long long)N, (long long)K);
  TTB_REQUIRE(ctx, M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "%s: dimension too large", what);
  TTB_REQUIRE(ctx, epilogue >= TTB_EPI_NONE && epilogue <= TTB_EPI_BIAS_TANH, "%s: unknown epilogue %d", what, epilogue);
  if (M == 0) return TTB_OK;
  TTB_REQUIRE(ctx, A && W && out, "%s: null pointer", what);
  TTB_REQUIRE(ctx, epilogue == TTB_EPI_NONE || bias, "%s: epilogue %d needs a bias", what, epilogue);
  TTB_REQUIRE(ctx, epilogue != TTB_EPI_BIAS_RESIDUAL || residual, "%s: residual epilogue needs a residual", what);
  TTB_REQUIRE(ctx, K % k_align == 0, "%s: K=%lld must be a multiple of %d (16-byte TMA rows)", what, (long long)K, k_align);
  TTB_REQUIRE(ctx, ldo >= N, "%s: ldo < N", what);
  TTB_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) % 16 == 0, "%s: operands must be 16-byte aligned", what);
  return TTB_OK;
}

// Zero fill that takes part in programmatic dependent launch: it returns only after the kernel ahead of it has completed,
// so a kernel that waits for this one is ordered after that one too.
__global__ void __launch_bounds__(256) zero_floats_kernel(float* dst, int64_t n) {
  pdl_trigger();
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) dst[i] = 0.f;
}

int linear_int8_common(ttb_ctx* ctx, const char* what, int out_dtype, const int8_t* Aq, const float* row_scale, const float* act_qparams,
                       const int8_t* Wq, const float* w_scale, const int32_t* col_sum, const void* bias, const void* residual, int64_t ldr,
                       int64_t M, int64_t N, int64_t K, int epilogue, void* out, int64_t ldo, float* row_absmax = nullptr) {
  TTB_REQUIRE(ctx, out_dtype == TTB_F16 || out_dtype == TTB_BF16, "%s: output dtype must be F16 or BF16", what);
  int s = check_linear(ctx, what, Aq, Wq, bias, residual, M, N, K, epilogue, out, ldo, 16);
  if (s || M == 0) return s;
  TTB_REQUIRE(ctx, (row_scale || act_qparams) && w_scale, "%s: null scale pointer", what);
  TTB_REQUIRE(ctx, !act_qparams || col_sum, "%s: the affine form needs the weight's column sums", what);
  DeviceGuard g(ctx->device);
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.npass = 1;
  p.out = out; p.ldo = ldo; p.bias = bias; p.residual = residual; p.ldr = ldr;
  p.row_scale = row_scale; p.w_scale = w_scale; p.act_qparams = act_qparams; p.col_sum = col_sum;
  p.epilogue = epilogue; p.split_k = 1; p.status = ctx->d_status;
  if (row_absmax) {  // zero-filled by a kernel of its own, so that the launches stay one programmatic-dependency chain
    const int64_t n4 = (M + 3) / 4;
    launch_pdl(zero_floats_kernel, dim3((unsigned)std::min<int64_t>((n4 + 255) / 256, 1024)), dim3(256), 0, ctx->stream, row_absmax, M);
    p.row_absmax = row_absmax;
  }
  const Operands op{Aq, nullptr, K, Wq, nullptr};
  if (act_qparams) {
    if (out_dtype == TTB_F16) return pick_tile<KIND_I8, __half, VAR_AFFINE>(ctx, op, p);
    return pick_tile<KIND_I8, __nv_bfloat16, VAR_AFFINE>(ctx, op, p);
  }
  if (out_dtype == TTB_F16) return pick_tile<KIND_I8, __half>(ctx, op, p);
  return pick_tile<KIND_I8, __nv_bfloat16>(ctx, op, p);
}

// ---- weight re-layout -----------------------------------------------------------------------------
// dst[n, k] = convert(src[k, n])  (or src[n, k] when it is already [N,K])
template <typename S, typename D>
__global__ void __launch_bounds__(256)
prepack_kernel(const S* __restrict__ src, int src_is_nk, int K, int N, D* __restrict__ dst) {
  __shared__ float tile[32][33];
  const int k0 = blockIdx.x * 32, n0 = blockIdx.y * 32;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;  // 32 x 8
  if (src_is_nk) {
    for (int r = ty; r < 32; r += 8) {
      const int n = n0 + r, k = k0 + tx;
      if (n < N && k < K) dst[(int64_t)n * K + k] = from_f<D>(to_f(src[(int64_t)n * K + k]));
    }
    return;
  }
  for (int r = ty; r < 32; r += 8) {
    const int k = k0 + r, n = n0 + tx;
    tile[r][tx] = (k < K && n < N) ? to_f(src[(int64_t)k * N + n]) : 0.f;
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int n = n0 + r, k = k0 + tx;
    if (n < N && k < K) dst[(int64_t)n * K + k] = from_f<D>(tile[tx][r]);
  }
}

template <typename S>
__global__ void __launch_bounds__(256) absmax_kernel(const S* __restrict__ src, int64_t n, float* __restrict__ amax) {
  float m = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, fabsf(to_f(src[i])));
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(amax), __float_as_int(m));  // non-negative floats order as ints
}

__global__ void amax_to_scale_kernel(float* s) { *s = (*s > 0.f) ? *s / 127.0f : 1.0f; }

template <typename S>
__global__ void __launch_bounds__(256)
prepack_int8_kernel(const S* __restrict__ src, int src_is_nk, int K, int N, const float* __restrict__ scale, int8_t* __restrict__ dst) {
  const float sc = *scale;
  const int64_t n_el = (int64_t)K * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_el; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = i / K, k = i % K;  // destination order
    const float w = to_f(src_is_nk ? src[i] : src[k * N + n]);
    float q = rintf(w / sc);
    q = fminf(fmaxf(q, -127.f), 127.f);
    dst[i] = (int8_t)q;
  }
}

// torch's per-tensor symmetric qint8 rule (MinMaxObserver): scale = max|W| / 127.5, q = clamp(rint(W * (1 / scale)), -128, 127).
__global__ void amax_to_scale_torch_kernel(float* s) {
  const float sc = *s / 127.5f;
  *s = fmaxf(sc, 1.1920928955078125e-07f);
}
template <typename S>
__global__ void __launch_bounds__(256)
prepack_int8_torch_kernel(const S* __restrict__ src, int src_is_nk, int K, int N, const float* __restrict__ scale, int8_t* __restrict__ dst) {
  const float inv = 1.0f / *scale;
  const int64_t n_el = (int64_t)K * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_el; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = i / K, k = i % K;  // destination order
    const float w = to_f(src_is_nk ? src[i] : src[k * N + n]);
    dst[i] = (int8_t)fminf(fmaxf(rintf(w * inv), -128.f), 127.f);
  }
}
// col_sum[n] = sum over k of Wq[n, k]: one warp per output row.
__global__ void __launch_bounds__(256) int8_row_sum_kernel(const int8_t* __restrict__ wq, int K, int N, int32_t* __restrict__ col_sum) {
  const int n = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (n >= N) return;
  int acc = 0;
  for (int k = lane; k < K; k += 32) acc += wq[(int64_t)n * K + k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) col_sum[n] = acc;
}

// Rows of fp32 -> two fp16 planes of a row times the power of two that brings its largest magnitude below 2^15, and its inverse. Bound by latency, of
// activations between two products, and then by memory: a CTA has a row, a thread eight elements of it, which it reads once. us a launch, a warp a row and two
// reads / now: 128 rows of 768 2.5 / 1.5, of 3072 5.4 / 2.6; 527 rows 2.8 / 2.4, 5.8 / 3.1; 3000 rows 6.2 / 4.7, 21.5 / 9.3.
__global__ void __launch_bounds__(1024) split_f16_rows_kernel(const float* __restrict__ x, int64_t rows, int K, __half* __restrict__ hi, __half* __restrict__ lo,
                                                              float* __restrict__ scale) {
  __shared__ float part[2][32];
  pdl_trigger();
  pdl_wait();
  const int col = threadIdx.x * 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int turn = 0;  // (the next row's maxima are other words: warps may still read these)
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x, turn ^= 1) {
    Vec8<float> v{};
    if (col < K) v.load(x + row * K + col);
    float top = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) top = fmaxf(top, fabsf(v.v[j]));
    top = warp_max(top);
    if (lane == 0) part[turn][warp] = top;
    __syncthreads();
    top = warp_max(lane < warps ? part[turn][lane] : 0.f);
    float up;
    const float down = f16_planes_scale(top, &up);
    if (threadIdx.x == 0) scale[row] = down;
    if (col < K) {
      uint4 h, l;
      f16_planes8(v.v, up, &h, &l);
      *reinterpret_cast<uint4*>(hi + row * K + col) = h;
      *reinterpret_cast<uint4*>(lo + row * K + col) = l;
    }
  }
}

// The same for rows of any width and alignment, a warp a row.
__global__ void __launch_bounds__(256) split_f16_kernel(const float* __restrict__ x, int64_t rows, int K, __half* __restrict__ hi, __half* __restrict__ lo,
                                                        float* __restrict__ scale) {
  pdl_trigger();
  pdl_wait();
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float* src = x + row * K;
  float top = 0.f;
#pragma unroll 4
  for (int k = lane; k < K; k += 32) top = fmaxf(top, fabsf(src[k]));
  float up;
  const float down = f16_planes_scale(warp_max(top), &up);
  if (lane == 0) scale[row] = down;
  for (int k = lane; k < K; k += 32) {
    const float v = src[k] * up;
    const __half h = __float2half_rn(v);
    hi[row * K + k] = h;
    lo[row * K + k] = __float2half_rn(v - __half2float(h));
  }
}

// fp32 -> two tf32-representable planes: hi = x rounded to 10 mantissa bits, lo = (x - hi) rounded likewise. hi + lo
// is x to 2^-23, which is what three tf32 products recover.
__global__ void __launch_bounds__(256) split_tf32_kernel(const float* __restrict__ x, int64_t n, float* __restrict__ hi, float* __restrict__ lo) {
  pdl_trigger();
  pdl_wait();
  // x may alias hi (in-place split of a weight): each element is read before it is written, by the same thread
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += (int64_t)gridDim.x * blockDim.x * 4) {
    if (i + 4 <= n) {
      const float4 v = *reinterpret_cast<const float4*>(x + i);
      float4 h, l;
      h.x = round_tf32(v.x); h.y = round_tf32(v.y); h.z = round_tf32(v.z); h.w = round_tf32(v.w);
      l.x = round_tf32(v.x - h.x); l.y = round_tf32(v.y - h.y); l.z = round_tf32(v.z - h.z); l.w = round_tf32(v.w - h.w);
      *reinterpret_cast<float4*>(hi + i) = h;
      *reinterpret_cast<float4*>(lo + i) = l;
    } else {
      for (int64_t j = i; j < n; ++j) {
        const float v = x[j], h = round_tf32(v);
        hi[j] = h;
        lo[j] = round_tf32(v - h);
      }
    }
  }
}

}  // namespace

// =================================================================================================
extern "C" int ttb_linear_ex(ttb_ctx* ctx, const ttb_linear_args* a) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, a != nullptr, "linear_ex: null argument block");
  const int dt = a->dtype, odt = a->out_dtype;
  TTB_REQUIRE(ctx, dt == TTB_F16 || dt == TTB_BF16 || dt == TTB_F32, "linear_ex: operand dtype must be F16, BF16 or F32");
  TTB_REQUIRE(ctx, odt == dt || (odt == TTB_F32 && dt != TTB_F32), "linear_ex: the output is of the operand dtype, or F32 for 16-bit operands");
  TTB_REQUIRE(ctx, !a->W2 || (a->A2 && dt == TTB_F32), "linear_ex: a second weight plane belongs to the three-pass fp32 form (A, A2, W, W2)");
  TTB_REQUIRE(ctx, !a->out_lo || (odt == dt && dt != TTB_F16), "linear_ex: the second output plane exists for BF16 and F32 products only");
  const int pad_scratch = (a->epilogue & TTB_EPI_FLAG_ROW_PADDING_IS_SCRATCH) ? 1 : 0;
  const bool planes = (a->epilogue & TTB_EPI_FLAG_TF32_PLANES) != 0;
  TTB_REQUIRE(ctx, !planes || (dt == TTB_F32 && a->out_lo), "linear_ex: planes as tf32 belong to an F32 product with out_lo");
  const int epilogue = a->epilogue & ~(TTB_EPI_FLAG_ROW_PADDING_IS_SCRATCH | TTB_EPI_FLAG_TF32_PLANES);
  const int k_align = dt == TTB_F32 ? 4 : 8;
  int s = check_linear(ctx, "linear", a->A, a->W, a->bias, a->residual, a->M, a->N, a->K, epilogue, a->out, a->ldo, k_align);
  if (s || a->M == 0) return s;
  TTB_REQUIRE(ctx, a->lda >= a->K && a->lda % k_align == 0, "linear: lda must be >= K and a multiple of %d", k_align);
  TTB_REQUIRE(ctx, ((reinterpret_cast<uintptr_t>(a->A2) | reinterpret_cast<uintptr_t>(a->W2)) & 15) == 0, "linear: operands must be 16-byte aligned");
  DeviceGuard g(ctx->device);
  GemmParams p{};
  p.M = (int)a->M; p.N = (int)a->N; p.K = (int)a->K;
  p.npass = a->W2 ? 3 : (a->A2 ? 2 : 1);
  p.pass_a = a->A2 ? 2 : 0;   // passes: (A, W), (A2, W), (A, W2): bit 1 of pass_a, bit 2 of pass_b
  p.pass_b = a->W2 ? 4 : 0;
  p.out = a->out; p.ldo = a->ldo; p.out_lo = a->out_lo;
  p.bias = a->bias; p.residual = a->residual; p.ldr = a->ldr;
  p.epilogue = epilogue; p.staged = pad_scratch ? STORE_TMA : STORE_DIRECT; p.split_k = 1; p.status = ctx->d_status;
  const Operands op{a->A, a->A2, a->lda, a->W, a->W2};
  if (planes) return pick_tile<KIND_TF32, float, VAR_TF32_PLANES>(ctx, op, p);
  if (dt == TTB_F32) return a->out_lo ? pick_tile<KIND_TF32, float, VAR_TWO_PLANES>(ctx, op, p) : pick_tile<KIND_TF32, float>(ctx, op, p);
  if (dt == TTB_F16) return odt == TTB_F32 ? pick_tile<KIND_F16, float>(ctx, op, p) : pick_tile<KIND_F16, __half>(ctx, op, p);
  if (odt == TTB_F32) return pick_tile<KIND_BF16, float>(ctx, op, p);
  if (a->out_lo) return pick_tile<KIND_BF16, __nv_bfloat16, VAR_TWO_PLANES>(ctx, op, p);
  return pick_tile<KIND_BF16, __nv_bfloat16>(ctx, op, p);
}

extern "C" int ttb_linear_split(ttb_ctx* ctx, const ttb_linear_split_args* a) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, a != nullptr, "linear_split: null argument block");
  int s = check_linear(ctx, "linear_split", a->A, a->W, a->bias, a->residual, a->M, a->N, a->K, a->epilogue, a->out, a->ldo, 8);
  if (s || a->M == 0) return s;
  TTB_REQUIRE(ctx, a->A2 && a->W2 && a->row_scale && a->col_scale, "linear_split: null pointer");
  TTB_REQUIRE(ctx, a->lda >= a->K && a->lda % 8 == 0, "linear_split: lda must be >= K and a multiple of 8");
  TTB_REQUIRE(ctx, ((reinterpret_cast<uintptr_t>(a->A2) | reinterpret_cast<uintptr_t>(a->W2) | reinterpret_cast<uintptr_t>(a->col_scale)) & 15) == 0,
              "linear_split: operands must be 16-byte aligned");
  DeviceGuard g(ctx->device);
  GemmParams p{};
  p.M = (int)a->M; p.N = (int)a->N; p.K = (int)a->K;
  p.npass = 3;
  p.pass_a = 2;  // (A, W), (A2, W), (A, W2)
  p.pass_b = 4;
  p.out = a->out; p.ldo = a->ldo;
  p.bias = a->bias; p.residual = a->residual; p.ldr = a->ldr;
  p.row_scale = a->row_scale; p.col_scale = a->col_scale;
  p.epilogue = a->epilogue; p.staged = STORE_DIRECT; p.split_k = 1; p.status = ctx->d_status;
  const Operands op{a->A, a->A2, a->lda, a->W, a->W2};
  return pick_tile<KIND_F16, float, VAR_SPLIT>(ctx, op, p);
}

extern "C" int ttb_split_f16(ttb_ctx* ctx, const float* x, int64_t rows, int64_t K, void* hi, void* lo, float* scale) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, rows >= 0 && K > 0 && K < (1ll << 31) && rows < (1ll << 33), "split_f16: bad shape");
  if (rows == 0) return TTB_OK;
  TTB_REQUIRE(ctx, x && hi && lo && scale, "split_f16: null pointer");
  DeviceGuard g(ctx->device);
  const bool eights = K % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15) == 0;
  if (eights && K <= 8192)  // (what a CTA's threads hold at once)
    launch_pdl(split_f16_rows_kernel, dim3((unsigned)std::min<int64_t>(rows, 16 * (int64_t)ctx->sm_count)), dim3((unsigned)((K / 8 + 31) / 32 * 32)), 0, ctx->stream, x, rows,
               (int)K, (__half*)hi, (__half*)lo, scale);
  else
    launch_pdl(split_f16_kernel, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, ctx->stream, x, rows, (int)K, (__half*)hi, (__half*)lo, scale);
  return launched(ctx, "split_f16");
}

extern "C" int ttb_linear_plan(ttb_ctx* ctx, int dtype, int out_dtype, int products, int two_plane_out, int whole, int64_t M, int64_t N, int64_t K,
                               int64_t* plan) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, M > 0 && N > 0 && K > 0 && M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31), "linear_plan: bad shape");
  TTB_REQUIRE(ctx, plan != nullptr, "linear_plan: null pointer");
  DeviceGuard g(ctx->device);
  TilePlan t{};
  const bool words = !whole;
  if (dtype == TTB_F16 && out_dtype == TTB_F32 && products == 3) t = choose_tile<KIND_F16, float, VAR_SPLIT>(ctx, M, N, K, 3, words);  // fp32 as fp16 planes
  else if (dtype == TTB_F32 && out_dtype == TTB_F32 && products >= 1 && products <= 3) t = choose_tile<KIND_TF32, float, VAR_PLAIN>(ctx, M, N, K, products, words);
  else if (dtype == TTB_I8 && out_dtype == TTB_F16 && products == 1) t = choose_tile<KIND_I8, __half, VAR_PLAIN>(ctx, M, N, K, 1, words);
  else if (dtype == TTB_F16 && out_dtype == TTB_F16 && products == 1) t = choose_tile<KIND_F16, __half, VAR_PLAIN>(ctx, M, N, K, 1, words);
  else if (dtype == TTB_BF16 && out_dtype == TTB_F32 && (products == 1 || products == 2)) t = choose_tile<KIND_BF16, float, VAR_PLAIN>(ctx, M, N, K, products, words);
  else if (dtype == TTB_BF16 && out_dtype == TTB_BF16 && (products == 1 || products == 2))
    t = two_plane_out ? choose_tile<KIND_BF16, __nv_bfloat16, VAR_TWO_PLANES>(ctx, M, N, K, products, words)
                      : choose_tile<KIND_BF16, __nv_bfloat16, VAR_PLAIN>(ctx, M, N, K, products, words);
  else return fail(ctx, TTB_ERR_INVALID, "linear_plan: no such product");
  plan[0] = t.columns;
  plan[1] = t.pair ? 2 : 1;
  plan[2] = t.split_k;
  plan[3] = t.tiles;
  plan[4] = t.slots;
  return TTB_OK;
}

extern "C" int ttb_linear(ttb_ctx* ctx, int dtype, const void* A, int64_t lda, const void* Wp, const void* bias,
                          const void* residual, int64_t ldr, int64_t M, int64_t N, int64_t K, int epilogue, void* out,
                          int64_t ldo) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, dtype == TTB_F16 || dtype == TTB_BF16, "linear: dtype must be F16 or BF16 (ttb_linear_ex takes F32)");
  ttb_linear_args a{};
  a.dtype = dtype; a.out_dtype = dtype;
  a.A = A; a.lda = lda; a.W = Wp;
  a.bias = bias; a.residual = residual; a.ldr = ldr;
  a.M = M; a.N = N; a.K = K; a.epilogue = epilogue;
  a.out = out; a.ldo = ldo;
  return ttb_linear_ex(ctx, &a);
}

extern "C" int ttb_layernorm(ttb_ctx* ctx, int dtype, const void* in, void* out, const void* gamma, const void* beta, int64_t M, int64_t N,
                             float eps);

// TTB_GEMM_LN (read at every call): unset or 0 = the product and the LayerNorm run as two kernels; 1 = one kernel for Linears
// with a long mainloop (K >= 2048); 2 = one kernel whenever the shape allows. Off by default: the one-kernel form makes the
// CTAs that hold one row block wait for one another through global memory, which needs the whole grid resident at once.
// That holds for one context on a device, but two contexts running such kernels on one device at the same time could
// each hold SMs the other is waiting for (the waits are bounded: the calls would end with TTB_ERR_DEVICE_WAIT), and the
// measured gain is under one per cent of the benchmark step.
static int fused_ln_mode() {
  const char* e = getenv("TTB_GEMM_LN");
  return (e && e[0] >= '1' && e[0] <= '2') ? e[0] - '0' : 0;
}

extern "C" int ttb_linear_layernorm(ttb_ctx* ctx, int dtype, const void* A, int64_t lda, const void* Wp, const void* bias,
                                    const void* residual, int64_t ldr, const void* gamma, const void* beta, float eps, int64_t M, int64_t N,
                                    int64_t K, void* out, int64_t ldo) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, dtype == TTB_F16 || dtype == TTB_BF16, "linear_layernorm: dtype must be F16 or BF16");
  int s = check_linear(ctx, "linear_layernorm", A, Wp, bias, residual, M, N, K, TTB_EPI_BIAS_RESIDUAL, out, ldo, 8);
  if (s || M == 0) return s;
  TTB_REQUIRE(ctx, gamma && beta, "linear_layernorm: null LayerNorm parameters");
  TTB_REQUIRE(ctx, ldo == N, "linear_layernorm: the output rows must be dense (ldo == N)");
  TTB_REQUIRE(ctx, lda >= K && lda % 8 == 0, "linear_layernorm: lda must be >= K and a multiple of 8");
  const bool aligned = ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(Wp) | reinterpret_cast<uintptr_t>(bias) |
                         reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta) |
                         reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  // Below about a thousand rows the narrow-tile (and split-K) kernels plus the one-round-trip LayerNorm are faster than
  // N / 256 CTAs walking the whole K range.
  // and with a short mainloop (K < 2048) the kernel runs at the speed of its epilogue, which the exchange of row sums
  // lengthens by more than the separate LayerNorm costs (measured at M = 18424, N = 768: K = 768 40.2 us in one kernel
  // against 25.6 + 12.5; K = 3072 72.1 against 67.6 + 12.5).
  const int mode = fused_ln_mode();
  if (mode && aligned && N % 256 == 0 && N / 256 <= kLnMaxTiles && M >= 1024 && (K >= 2048 || mode == 2) && ldr % 8 == 0 && M < (1ll << 31) &&
      K < (1ll << 31)) {
    DeviceGuard g(ctx->device);
    GemmParams p{};
    p.M = (int)M; p.N = (int)N; p.K = (int)K; p.npass = 1;
    p.out = out; p.ldo = ldo; p.bias = bias; p.residual = residual; p.ldr = ldr;
    p.epilogue = TTB_EPI_BIAS_RESIDUAL; p.split_k = 1; p.status = ctx->d_status;
    p.ln_gamma = gamma; p.ln_beta = beta; p.ln_eps = eps;
    const Operands op{A, nullptr, lda, Wp, nullptr};
    // CTA pairs where the plain kernel would use them too: a long mainloop (see pick_tile)
    const bool pair = pair_mode() && K * 2 >= 4096 && ((M + 2 * BM - 1) / (2 * BM)) * (N / 256) >= ctx->sm_count / 2;
    if (dtype == TTB_F16) s = pair ? launch_tc_ln<KIND_F16, __half, true>(ctx, op, p) : launch_tc_ln<KIND_F16, __half, false>(ctx, op, p);
    else s = pair ? launch_tc_ln<KIND_BF16, __nv_bfloat16, true>(ctx, op, p) : launch_tc_ln<KIND_BF16, __nv_bfloat16, false>(ctx, op, p);
    if (s != TTB_ERR_UNSUPPORTED) return s;
  }
  s = ttb_linear(ctx, dtype, A, lda, Wp, bias, residual, ldr, M, N, K, TTB_EPI_BIAS_RESIDUAL, out, ldo);
  if (s) return s;
  return ttb_layernorm(ctx, dtype, out, out, gamma, beta, M, N, eps);
}

extern "C" int ttb_linear_int8(ttb_ctx* ctx, int out_dtype, const int8_t* Aq, const float* row_scale, const int8_t* Wq,
                               const float* w_scale, const void* bias, const void* residual, int64_t ldr, int64_t M,
                               int64_t N, int64_t K, int epilogue, void* out, int64_t ldo) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, M == 0 || row_scale != nullptr, "linear_int8: null scale pointer");
  return linear_int8_common(ctx, "linear_int8", out_dtype, Aq, row_scale, nullptr, Wq, w_scale, nullptr, bias, residual, ldr, M, N, K, epilogue, out,
                            ldo);
}

extern "C" int ttb_linear_int8_rowmax(ttb_ctx* ctx, int out_dtype, const int8_t* Aq, const float* row_scale, const int8_t* Wq,
                                      const float* w_scale, const void* bias, const void* residual, int64_t ldr, int64_t M, int64_t N,
                                      int64_t K, int epilogue, void* out, int64_t ldo, float* row_absmax) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, M == 0 || (row_scale != nullptr && row_absmax != nullptr), "linear_int8_rowmax: null scale or maximum pointer");
  return linear_int8_common(ctx, "linear_int8_rowmax", out_dtype, Aq, row_scale, nullptr, Wq, w_scale, nullptr, bias, residual, ldr, M, N, K, epilogue,
                            out, ldo, row_absmax);
}

extern "C" int ttb_linear_int8_affine(ttb_ctx* ctx, int out_dtype, const int8_t* Aq, const float* act_qparams, const int8_t* Wq,
                                      const float* w_scale, const int32_t* col_sum, const void* bias, const void* residual, int64_t ldr,
                                      int64_t M, int64_t N, int64_t K, int epilogue, void* out, int64_t ldo) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, M == 0 || (act_qparams != nullptr && col_sum != nullptr), "linear_int8_affine: null quantisation parameters");
  return linear_int8_common(ctx, "linear_int8_affine", out_dtype, Aq, nullptr, act_qparams, Wq, w_scale, col_sum, bias, residual, ldr, M, N, K,
                            epilogue, out, ldo);
}

extern "C" int ttb_prepack_weight(ttb_ctx* ctx, int src_dtype, const void* src, int src_is_nk, int64_t K, int64_t N,
                                  int dst_dtype, void* dst) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, K > 0 && N > 0 && K < (1ll << 31) && N < (1ll << 31), "prepack_weight: bad shape");
  TTB_REQUIRE(ctx, src && dst, "prepack_weight: null pointer");
  TTB_REQUIRE(ctx, dst_dtype == TTB_F16 || dst_dtype == TTB_BF16 || dst_dtype == TTB_F32, "prepack_weight: bad destination dtype");
  DeviceGuard g(ctx->device);
  dim3 grid((unsigned)((K + 31) / 32), (unsigned)((N + 31) / 32));
  TTB_REQUIRE(ctx, grid.y <= 65535, "prepack_weight: N too large");
#define PREPACK(S, D) prepack_kernel<S, D><<<grid, 256, 0, ctx->stream>>>((const S*)src, src_is_nk, (int)K, (int)N, (D*)dst)
  TTB_DISPATCH_FLOAT(ctx, src_dtype, S, {
    if (dst_dtype == TTB_F16) PREPACK(S, __half);
    else if (dst_dtype == TTB_BF16) PREPACK(S, __nv_bfloat16);
    else PREPACK(S, float);
  });
#undef PREPACK
  return launched(ctx, "prepack_weight");
}

extern "C" int ttb_prepack_weight_int8(ttb_ctx* ctx, int src_dtype, const void* src, int src_is_nk, int64_t K, int64_t N,
                                       int8_t* dst, float* scale_out) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, K > 0 && N > 0, "prepack_weight_int8: bad shape");
  TTB_REQUIRE(ctx, src && dst && scale_out, "prepack_weight_int8: null pointer");
  DeviceGuard g(ctx->device);
  TTB_CUDA(ctx, cudaMemsetAsync(scale_out, 0, sizeof(float), ctx->stream));
  const int64_t n = K * N;
  const int grid = (int)((n + 255) / 256 < (int64_t)ctx->sm_count * 8 ? (n + 255) / 256 : (int64_t)ctx->sm_count * 8);
  TTB_DISPATCH_FLOAT(ctx, src_dtype, S, {
    absmax_kernel<S><<<grid, 256, 0, ctx->stream>>>((const S*)src, n, scale_out);
    amax_to_scale_kernel<<<1, 1, 0, ctx->stream>>>(scale_out);
    prepack_int8_kernel<S><<<grid, 256, 0, ctx->stream>>>((const S*)src, src_is_nk, (int)K, (int)N, scale_out, dst);
  });
  ctx->launches.fetch_add(2);
  return launched(ctx, "prepack_weight_int8");
}

extern "C" int ttb_prepack_weight_int8_affine(ttb_ctx* ctx, int src_dtype, const void* src, int src_is_nk, int64_t K, int64_t N, int8_t* dst,
                                              float* scale_out, int32_t* col_sum_out) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, K > 0 && N > 0 && K < (1ll << 31) && N < (1ll << 31), "prepack_weight_int8_affine: bad shape");
  TTB_REQUIRE(ctx, src && dst && scale_out && col_sum_out, "prepack_weight_int8_affine: null pointer");
  DeviceGuard g(ctx->device);
  TTB_CUDA(ctx, cudaMemsetAsync(scale_out, 0, sizeof(float), ctx->stream));
  const int64_t n = K * N;
  const int grid = (int)((n + 255) / 256 < (int64_t)ctx->sm_count * 8 ? (n + 255) / 256 : (int64_t)ctx->sm_count * 8);
  TTB_DISPATCH_FLOAT(ctx, src_dtype, S, {
    absmax_kernel<S><<<grid, 256, 0, ctx->stream>>>((const S*)src, n, scale_out);
    amax_to_scale_torch_kernel<<<1, 1, 0, ctx->stream>>>(scale_out);
    prepack_int8_torch_kernel<S><<<grid, 256, 0, ctx->stream>>>((const S*)src, src_is_nk, (int)K, (int)N, scale_out, dst);
  });
  int8_row_sum_kernel<<<(unsigned)((N + 7) / 8), 256, 0, ctx->stream>>>(dst, (int)K, (int)N, col_sum_out);
  ctx->launches.fetch_add(3);
  return launched(ctx, "prepack_weight_int8_affine");
}

extern "C" int ttb_split_tf32(ttb_ctx* ctx, const float* x, int64_t n, float* hi, float* lo) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, n >= 0, "split_tf32: negative size");
  if (n == 0) return TTB_OK;
  TTB_REQUIRE(ctx, x && hi && lo, "split_tf32: null pointer");
  TTB_REQUIRE(ctx, ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15) == 0,
              "split_tf32: pointers must be 16-byte aligned");
  DeviceGuard g(ctx->device);
  const int64_t want = (n / 4 + 255) / 256 + 1;
  const int grid = (int)(want < (int64_t)ctx->sm_count * 16 ? want : (int64_t)ctx->sm_count * 16);
  launch_pdl(split_tf32_kernel, dim3(grid), dim3(256), 0, ctx->stream, x, n, hi, lo);
  return launched(ctx, "split_tf32");
}
