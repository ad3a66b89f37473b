// Self-attention of fp32 models over packed tokens, in one kernel (ttb_attention_f32).
//
// It takes the place of five (SplitAddBiasTransposeForScore, the score product, ApplyMaskAndSoftmax, the value product, TransposeForScore)
// that pad every sequence to the longest and write the scores out. Both products run on mma.sync m16n8k16 with every fp32 operand as two fp16 planes (three
// products, 22 bits of an element): on the CUDA cores, from shared memory, they were bound by its bandwidth (4 wavefronts a 16-byte read for
// 32 multiply-adds: 58 % of its peak, 8 us for 16 rows against 64 keys). A row of queries, keys or values is scaled by its own largest element, a row of
// probabilities, times their values' scales, by its own in each tile; the scales come out again in fp32. So a key that a row does not see leaves no trace in it, however
// large it is. (One scale for a tile of values was 7 % faster, and a hidden key of 1e9 made the others 6e-3 wrong.) The second planes are 2^11 times what the first ones
// leave, so that an element has all its bits down to 2^-28 of its row's largest. Softmax, sums and the outputs' accumulation from tile to tile are fp32. Of a tile's
// products the small ones are added up first, since the tensor core truncates the sum with every addition. Error against 64 bits, CUDA cores with fp32 operands / now:
// 128 keys 3.4e-7 / 2.2e-7, 512 keys 5.0e-7 / 2.4e-7; worst of all outputs, of its terms' magnitudes, with rows and dimensions up to 2^16 apart 1.3e-6 / 6.3e-7.
// A CTA of four warps has 16 WR query rows of one (sequence, head), and WK of its warps share a tile of 64 keys: few rows for few CTAs, since the keys' way and their
// conversion are then the time. us, 12 heads, CUDA cores / now: 8 sequences of up to 120 19.6 / 10.8, 1 x 128 15.4 / 9.8, 1 x 300 43 / 20.4, 1 x 512 71 / 31, 9 x 182 40 / 24,
// 6 x 512 149 / 82.
#include "ttb_common.cuh"

using namespace ttb;

namespace {

constexpr int kThreads = 128, kWarps = 4;
constexpr int D = 64;
constexpr int kKeys = 64;
constexpr int kPitch = 72;      // halves between the rows of a tile in shared memory: eight rows' sixteen bytes are in different banks
constexpr int kOutPitch = 68;   // floats between the rows of a warp's output, with {maximum, sum} behind the 64
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLoUp = 2048.f, kLoDown = 1.f / kLoUp;  // the second planes are multiplied by 2^11: see planes2

struct Tiles {
  __half k[2][kKeys * kPitch], v[2][kKeys * kPitch];  // hi, lo
  float k_scale[kKeys], v_scale[kKeys];
};
union Shared {
  Tiles t;
  float out[kWarps][16 * kOutPitch];
};

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two neighbouring elements as halves of the planes. The second plane is 2^11 times what the first has left, so that it has all its bits wherever
// the first has, down to 2^-28 of the row's largest; products with it are added up by themselves and divided by 2^11.
__device__ __forceinline__ void planes2(float x, float y, uint32_t* hi, uint32_t* lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn((x - f.x) * kLoUp, (y - f.y) * kLoUp);
  *hi = *reinterpret_cast<const uint32_t*>(&h);
  *lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Two magnitudes as far as their scales depend on them, in one word: fp32 numbers order like their upper halves do as whole numbers. (No number: none.)
__device__ __forceinline__ uint32_t pack_most(float a, float b) { return __byte_perm(__float_as_uint(fmaxf(a, 0.f)), __float_as_uint(fmaxf(b, 0.f)), 0x7632); }
__device__ __forceinline__ float first_of(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float second_of(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }

// ROUNDED: the output leaves as its two tf32 planes.
template <int WR, bool ROUNDED>
__global__ void __launch_bounds__(kThreads)
attention_f32_kernel(const float* __restrict__ qkv, const int32_t* __restrict__ cu, int heads, const float* __restrict__ mask, long long mask_batch,
                     long long mask_row, int causal, float scale, float* __restrict__ out, float* __restrict__ out_lo) {
  constexpr int WK = kWarps / WR, kRows = 16 * WR, kMine = kKeys / WK, NT = kMine / 8;  // keys of a tile for a warp, in eights
  __shared__ __align__(16) Shared sm;
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.z, h = blockIdx.y, q0 = blockIdx.x * kRows;
  const int begin = cu[b], len = cu[b + 1] - begin;
  if (q0 >= len) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wr = warp % WR, wk = warp / WR;
  const int H = heads * D;
  const long long pitch = 3ll * H;
  const float* base = qkv + (long long)begin * pitch + h * D;
  const int row0 = q0 + wr * 16 + g;  // of the thread's rows row0 and row0 + 8
  // the warp's queries as fragments
  uint32_t qh[4][4], ql[4][4];
  float q_scale[2];
  {
    float2 x[4][4];
    float top[2] = {0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = row0 + (e & 1) * 8;
        x[s][e] = row < len ? *reinterpret_cast<const float2*>(base + row * pitch + s * 16 + (e >> 1) * 8 + t * 2) : make_float2(0.f, 0.f);
        top[e & 1] = fmaxf(top[e & 1], fmaxf(fabsf(x[s][e].x), fabsf(x[s][e].y)));
      }
    float up[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], o));
      q_scale[r] = f16_planes_scale(top[r], &up[r]);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 4; ++e) planes2(x[s][e].x * up[e & 1], x[s][e].y * up[e & 1], &qh[s][e], &ql[s][e]);
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
  const int keys = causal ? min(len, q0 + kRows) : len;
  for (int j0 = 0; j0 < keys; j0 += kKeys) {
    // a thread's keys and values: four elements of rows (tid / 16), + 8, ...
    const int col = (tid & 15) * 4, first = tid >> 4;
    float4 k[8], v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      k[i] = v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j0 + first + i * 8 < keys) {
        const float* src = base + (j0 + first + i * 8) * pitch + H + col;
        k[i] = *reinterpret_cast<const float4*>(src);
        v[i] = *reinterpret_cast<const float4*>(src + H);
      }
    }
    __syncthreads();  // the tile before has been read
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t top = pack_most(fmaxf(fmaxf(fabsf(k[i].x), fabsf(k[i].y)), fmaxf(fabsf(k[i].z), fabsf(k[i].w))),
                               fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) top = __vmaxs2(top, __shfl_xor_sync(0xffffffffu, top, o));
      float k_up, v_up;
      const float k_down = f16_planes_scale(first_of(top), &k_up), v_down = f16_planes_scale(second_of(top), &v_up);
      const int r = first + i * 8;
      if (col == 0) {
        sm.t.k_scale[r] = k_down * scale;
        sm.t.v_scale[r] = v_down;
      }
      uint2 hi, lo;
      planes2(k[i].x * k_up, k[i].y * k_up, &hi.x, &lo.x);
      planes2(k[i].z * k_up, k[i].w * k_up, &hi.y, &lo.y);
      *reinterpret_cast<uint2*>(&sm.t.k[0][r * kPitch + col]) = hi;
      *reinterpret_cast<uint2*>(&sm.t.k[1][r * kPitch + col]) = lo;
      planes2(v[i].x * v_up, v[i].y * v_up, &hi.x, &lo.x);
      planes2(v[i].z * v_up, v[i].w * v_up, &hi.y, &lo.y);
      *reinterpret_cast<uint2*>(&sm.t.v[0][r * kPitch + col]) = hi;
      *reinterpret_cast<uint2*>(&sm.t.v[1][r * kPitch + col]) = lo;
    }
    __syncthreads();
    const int mine = wk * kMine;  // the warp's keys of the tile
    if (j0 + mine >= keys) continue;
    float s[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
    // the small products first: a sum is truncated with every one that is added to it
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
      const int at = (mine + n * 8 + (lane & 7) + (lane >> 4) * 8) * kPitch + ((lane >> 3) & 1) * 8;
      uint32_t kh[4][4];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        uint32_t kl[4];
        ldmatrix4(kh[d], &sm.t.k[0][at + d * 16]);
        ldmatrix4(kl, &sm.t.k[1][at + d * 16]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          mma16816(s[n + u], ql[d], kh[d][2 * u], kh[d][2 * u + 1]);
          mma16816(s[n + u], qh[d], kl[2 * u], kl[2 * u + 1]);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n + u][e] *= kLoDown;
#pragma unroll
      for (int d = 0; d < 4; ++d)
#pragma unroll
        for (int u = 0; u < 2; ++u) mma16816(s[n + u], qh[d], kh[d][2 * u], kh[d][2 * u + 1]);
    }
    float top[2] = {m[0], m[1]};
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int at = mine + n * 8 + t * 2 + (e & 1), j = j0 + at, i = row0 + (e >> 1) * 8;
        float x = s[n][e] * q_scale[e >> 1] * sm.t.k_scale[at];
        if (mask && i < len && j < len) x += mask[b * mask_batch + i * mask_row + j];
        if (j >= keys || (causal && j > i)) x = -INFINITY;
        s[n][e] = x;
        top[e >> 1] = fmaxf(top[e >> 1], x);
      }
    float keep[2], centre[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], o));
      centre[r] = top[r] == -INFINITY ? 0.f : top[r];
      keep[r] = exp2f((m[r] - centre[r]) * kLog2e);
      m[r] = top[r];
      l[r] *= keep[r];
    }
    // The probabilities, and those times the values' scales as planes, scaled by the largest of the row: a key that a row does not see leaves no
    // trace in it, however large its values.
    float most[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const float2 vs = *reinterpret_cast<const float2*>(&sm.t.v_scale[mine + n * 8 + t * 2]);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float x = expf(s[n][r * 2] - centre[r]), y = expf(s[n][r * 2 + 1] - centre[r]);
        l[r] += x + y;
        s[n][r * 2] = x * vs.x;
        s[n][r * 2 + 1] = y * vs.y;
        most[r] = fmaxf(most[r], fmaxf(s[n][r * 2], s[n][r * 2 + 1]));
      }
    }
    uint32_t both = pack_most(most[0], most[1]);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) both = __vmaxs2(both, __shfl_xor_sync(0xffffffffu, both, o));
    float p_up[2];
    const float factor[2] = {f16_planes_scale(first_of(both), &p_up[0]), f16_planes_scale(second_of(both), &p_up[1])};
    uint32_t ph[NT / 2][4], pl[NT / 2][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) planes2(s[n][r * 2] * p_up[r], s[n][r * 2 + 1] * p_up[r], &ph[n / 2][(n & 1) * 2 + r], &pl[n / 2][(n & 1) * 2 + r]);
#pragma unroll
    for (int d = 0; d < 4; ++d) {  // sixteen dimensions
      float o[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[u][e] = 0.f;
      uint32_t vh[NT / 2][4];
#pragma unroll
      for (int n = 0; n < NT / 2; ++n) {  // sixteen keys
        const int at = (mine + n * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * kPitch + d * 16 + (lane >> 4) * 8;
        uint32_t vl[4];
        ldmatrix4_trans(vh[n], &sm.t.v[0][at]);
        ldmatrix4_trans(vl, &sm.t.v[1][at]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          mma16816(o[u], pl[n], vh[n][2 * u], vh[n][2 * u + 1]);
          mma16816(o[u], ph[n], vl[2 * u], vl[2 * u + 1]);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[u][e] *= kLoDown;
#pragma unroll
      for (int n = 0; n < NT / 2; ++n)
#pragma unroll
        for (int u = 0; u < 2; ++u) mma16816(o[u], ph[n], vh[n][2 * u], vh[n][2 * u + 1]);
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[d * 2 + u][e] = fmaf(o[u][e], factor[e >> 1], acc[d * 2 + u][e] * keep[e >> 1]);
    }
  }
  __syncthreads();  // the last tile has been read: the warps' results take its place
  {
    float* mine = sm.out[warp];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], o);
      if (t == 0) *reinterpret_cast<float2*>(mine + (g + r * 8) * kOutPitch + D) = make_float2(m[r], l[r]);
#pragma unroll
      for (int n = 0; n < 8; ++n) *reinterpret_cast<float2*>(mine + (g + r * 8) * kOutPitch + n * 8 + t * 2) = make_float2(acc[n][r * 2], acc[n][r * 2 + 1]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < 2 * WR; ++n) {
    const int r = (n * kThreads + tid) >> 4, c = (tid & 15) * 4, i = q0 + r;
    if (i >= len) continue;
    // the warps that shared this row's keys, in their order
    float top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int w = 0; w < WK; ++w) top = fmaxf(top, sm.out[r / 16 + w * WR][(r & 15) * kOutPitch + D]);
    const float centre = top == -INFINITY ? 0.f : top;
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < WK; ++w) {
      const float* theirs = sm.out[r / 16 + w * WR] + (r & 15) * kOutPitch;
      const float f = exp2f((theirs[D] - centre) * kLog2e);
      const float4 x = *reinterpret_cast<const float4*>(theirs + c);
      sum = fmaf(theirs[D + 1], f, sum);
      y = make_float4(fmaf(x.x, f, y.x), fmaf(x.y, f, y.y), fmaf(x.z, f, y.z), fmaf(x.w, f, y.w));
    }
    const float inv = 1.0f / sum;
    y = make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv);
    const long long at = (long long)(begin + i) * H + h * D + c;
    *reinterpret_cast<float4*>(out + at) = ROUNDED ? make_float4(tf32_hi(y.x), tf32_hi(y.y), tf32_hi(y.z), tf32_hi(y.w)) : y;
    if (ROUNDED || out_lo) *reinterpret_cast<float4*>(out_lo + at) = make_float4(tf32_lo(y.x, ROUNDED), tf32_lo(y.y, ROUNDED), tf32_lo(y.z, ROUNDED), tf32_lo(y.w, ROUNDED));
  }
}

template <bool ROUNDED>
int attention_f32(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d, const float* mask,
                  int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, float* out, float* out_lo) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, d == D && heads > 0 && heads <= 65535 && B >= 0 && B <= 65535 && max_seqlen >= 0 && max_seqlen < (1 << 30), "attention_f32: bad shape");
  if (B == 0 || max_seqlen == 0) return TTB_OK;
  TTB_REQUIRE(ctx, qkv && cu_seqlens && out, "attention_f32: null pointer");
  TTB_REQUIRE(ctx, ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(out_lo)) & 15) == 0,
              "attention_f32: buffers must be 16-byte aligned");
  DeviceGuard g(ctx->device);
  auto blocks = [&](int rows) { return dim3((unsigned)((max_seqlen + rows - 1) / rows), (unsigned)heads, (unsigned)B); };
  auto ctas = [&](int64_t rows) { return B * heads * ((max_seqlen + rows - 1) / rows); };
#define ATTENTION_F32(WR)                                                                                                                                  \
  launch_pdl(attention_f32_kernel<WR, ROUNDED>, blocks(16 * WR), dim3(kThreads), 0, ctx->stream, qkv, cu_seqlens, (int)heads, mask, (long long)mask_batch_stride, \
             (long long)mask_row_stride, causal, scale, out, out_lo)
  // The most rows a CTA with which the chip is still full: us with 16, 32, 64 rows: 192 CTAs of 64 rows (384 of 32) 10.4, 12.4, 15.6; 324 (648) 36, 27.5, 23.1; 252
  // (504) 37.7, 32.8, 44.6; 96 (192) 28.6, 36, 44.7; 768 181, 128, 101.
  if (ctas(64) >= 2 * ctx->sm_count) ATTENTION_F32(4);
  else if (ctas(32) >= 3 * ctx->sm_count) ATTENTION_F32(2);
  else ATTENTION_F32(1);
#undef ATTENTION_F32
  return launched(ctx, "attention_f32");
}

}  // namespace

extern "C" int ttb_attention_f32(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d, const float* mask,
                                 int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, float* out, float* out_lo) {
  return attention_f32<false>(ctx, qkv, cu_seqlens, B, max_seqlen, heads, d, mask, mask_batch_stride, mask_row_stride, causal, scale, out, out_lo);
}

extern "C" int ttb_attention_f32_planes(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d,
                                        const float* mask, int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, float* hi, float* lo) {
  if (ctx && B > 0 && max_seqlen > 0) TTB_REQUIRE(ctx, lo, "attention_f32_planes: null pointer");
  return attention_f32<true>(ctx, qkv, cu_seqlens, B, max_seqlen, heads, d, mask, mask_batch_stride, mask_row_stride, causal, scale, hi, lo);
}
