// Self-attention of fp32 models over packed tokens, in one kernel (ttb_attention_f32).
//
// It takes the place of five (SplitAddBiasTransposeForScore, the score product, ApplyMaskAndSoftmax, the value product, TransposeForScore)
// that pad every sequence to the longest and write the scores out. Products and softmax stay in fp32 on the CUDA cores, as they were: scores that
// are rounded to a tensor-core format would cost accuracy, and at the sizes of fp32 requests the launches and the padding, not the
// arithmetic, were the time. A CTA has 8 R query rows of one (sequence, head) and goes over the keys in tiles of 64 with an online
// softmax; a thread computes R x 4 scores, then R x 4 outputs, from 16-byte reads of shared memory (rows of 68 floats: the lanes of a read
// hit different banks). BERT-base fp32, us a pass, with the planes below, against
// those five: 8 requests of 10 to 120 tokens 2591 -> 1730, 16 of 8 to 512 13283 -> 5670, 1 x 128 1187 -> 1084, 8 x 512 8826 -> 6050, 32 x 512 32363 ->
// 22300 (with the layer norms of few rows; its Linears are what is left); one layer's attention over 1 x 4096 tokens 2693 -> 1705. The output may leave as the two planes that the next product takes.
#include "ttb_common.cuh"

using namespace ttb;

namespace {

constexpr int kThreads = 128;
constexpr int D = 64;
constexpr int kKeys = 64;
constexpr int kPitch = 68;
constexpr float kLog2e = 1.4426950408889634f;

template <int R> constexpr int kSmem = (2 * 8 * R + 2 * kKeys) * kPitch * 4;

// What the planes of the output in fp16 take: of the rows that the queries, keys and values were computed from, what they were divided by, and the weights'
// statistics (ttb_split_f16), which bound the values and so their averages; the planes' own scale.
struct SplitOut {
  const float *row_scale, *stats;
  __half *hi, *lo;
  float* scale;
};
enum { OUT_VALUE = 0, OUT_TF32 = 1, OUT_F16 = 2 };

// OUT: the output leaves as it is, or as its two planes, in place of it. (As a choice at run time it cost 15 registers and 1.2 us of 18 at 527 rows.)
template <int R, int OUT>
__global__ void __launch_bounds__(kThreads)
attention_f32_kernel(const float* __restrict__ qkv, const int32_t* __restrict__ cu, int heads, const float* __restrict__ mask, long long mask_batch,
                     long long mask_row, int causal, float scale, float* __restrict__ out, float* __restrict__ out_lo, const SplitOut split) {
  constexpr bool ROUNDED = OUT == OUT_TF32;
  constexpr int kRows = 8 * R;
  extern __shared__ __align__(16) float smem[];
  float *qs = smem, *ps = qs + kRows * kPitch, *ks = ps + kRows * kPitch, *vs = ks + kKeys * kPitch;
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.z, h = blockIdx.y, q0 = blockIdx.x * kRows;
  const int begin = cu[b], len = cu[b + 1] - begin;
  if (q0 >= len) return;
  const int tid = threadIdx.x, kg = tid & 15, rg = tid >> 4;  // keys or dimensions, rows
  const int H = heads * D;
  const long long pitch = 3ll * H;
  const float* base = qkv + (long long)begin * pitch + h * D;
  for (int i = tid; i < kRows * 16; i += kThreads) {
    const int r = i >> 4, c = (i & 15) * 4;
    *reinterpret_cast<float4*>(qs + r * kPitch + c) =
        q0 + r < len ? *reinterpret_cast<const float4*>(base + (q0 + r) * pitch + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float m[R], l[R], acc[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[r][e] = 0.f;
  }
  const int keys = causal ? min(len, q0 + kRows) : len;
  for (int j0 = 0; j0 < keys; j0 += kKeys) {
    __syncthreads();  // the tile before has been read
    // four rows of keys and of values in flight per thread
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float4 k[4], v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (half * 4 + i) * 8 + rg;
        k[i] = v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j0 + r < keys) {
          const float* src = base + (j0 + r) * pitch + H + kg * 4;
          k[i] = *reinterpret_cast<const float4*>(src);
          v[i] = *reinterpret_cast<const float4*>(src + H);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (half * 4 + i) * 8 + rg;
        *reinterpret_cast<float4*>(ks + r * kPitch + kg * 4) = k[i];
        *reinterpret_cast<float4*>(vs + r * kPitch + kg * 4) = v[i];
      }
    }
    __syncthreads();
    // scores of rows rg * R .. and keys kg, kg + 16, ...
    float s[R][4];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[r][e] = 0.f;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 q[R], k[4];
#pragma unroll
      for (int r = 0; r < R; ++r) q[r] = *reinterpret_cast<const float4*>(qs + (rg * R + r) * kPitch + d);
#pragma unroll
      for (int e = 0; e < 4; ++e) k[e] = *reinterpret_cast<const float4*>(ks + (kg + 16 * e) * kPitch + d);
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[r][e] = fmaf(q[r].x, k[e].x, fmaf(q[r].y, k[e].y, fmaf(q[r].z, k[e].z, fmaf(q[r].w, k[e].w, s[r][e]))));
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = q0 + rg * R + r;
      float top = m[r];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = j0 + kg + 16 * e;
        s[r][e] *= scale;
        if (mask && i < len && j < len) s[r][e] += mask[b * mask_batch + i * mask_row + j];
        if (j >= keys || (causal && j > i)) s[r][e] = -INFINITY;
        top = fmaxf(top, s[r][e]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float centre = top == -INFINITY ? 0.f : top, keep = exp2f((m[r] - centre) * kLog2e);
      m[r] = top;
      l[r] *= keep;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[r][e] *= keep;
        const float p = expf(s[r][e] - centre);
        l[r] += p;  // this thread's keys; the sixteen threads' sums meet at the end
        ps[(rg * R + r) * kPitch + kg + 16 * e] = p;
      }
    }
    __syncwarp();  // a row's probabilities are written and read by one half-warp
    // outputs of rows rg * R .. and dimensions kg * 4 ..
    const int last = min(kKeys, (keys - j0 + 3) & ~3);
#pragma unroll 2
    for (int j = 0; j < last; j += 4) {
      float4 p[R], v[4];
#pragma unroll
      for (int r = 0; r < R; ++r) p[r] = *reinterpret_cast<const float4*>(ps + (rg * R + r) * kPitch + j);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float4*>(vs + (j + e) * kPitch + kg * 4);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        acc[r][0] = fmaf(p[r].x, v[0].x, fmaf(p[r].y, v[1].x, fmaf(p[r].z, v[2].x, fmaf(p[r].w, v[3].x, acc[r][0]))));
        acc[r][1] = fmaf(p[r].x, v[0].y, fmaf(p[r].y, v[1].y, fmaf(p[r].z, v[2].y, fmaf(p[r].w, v[3].y, acc[r][1]))));
        acc[r][2] = fmaf(p[r].x, v[0].z, fmaf(p[r].y, v[1].z, fmaf(p[r].z, v[2].z, fmaf(p[r].w, v[3].z, acc[r][2]))));
        acc[r][3] = fmaf(p[r].x, v[0].w, fmaf(p[r].y, v[1].w, fmaf(p[r].z, v[2].w, fmaf(p[r].w, v[3].w, acc[r][3]))));
      }
    }
    __syncwarp();
  }
  float up = 1.f;
  if constexpr (OUT == OUT_F16) {  // one scale for all heads and rows of the sequence: no value of it is beyond this bound
    float most = 0.f;
    for (int j = tid & 31; j < len; j += 32) most = fmaxf(most, split.row_scale[begin + j]);
    const float down = f16_planes_scale(warp_max(most) * 32768.f * split.stats[0] + split.stats[1], &up);
    if (h == 0 && tid < kRows && q0 + tid < len) split.scale[begin + q0 + tid] = down;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float sum = l[r];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const int i = q0 + rg * R + r;
    if (i >= len) continue;
    const float inv = 1.0f / sum;
    const float4 y = make_float4(acc[r][0] * inv, acc[r][1] * inv, acc[r][2] * inv, acc[r][3] * inv);
    const long long at = (long long)(begin + i) * H + h * D + kg * 4;
    if constexpr (OUT == OUT_F16) {
      const float v[4] = {y.x * up, y.y * up, y.z * up, y.w * up};
      __half2 hi[2], lo[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        hi[e] = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
        const float2 f = __half22float2(hi[e]);
        lo[e] = __floats2half2_rn(v[2 * e] - f.x, v[2 * e + 1] - f.y);
      }
      *reinterpret_cast<uint2*>(split.hi + at) = *reinterpret_cast<const uint2*>(hi);
      *reinterpret_cast<uint2*>(split.lo + at) = *reinterpret_cast<const uint2*>(lo);
      continue;
    }
    *reinterpret_cast<float4*>(out + at) = ROUNDED ? make_float4(tf32_hi(y.x), tf32_hi(y.y), tf32_hi(y.z), tf32_hi(y.w)) : y;
    if (ROUNDED || out_lo) *reinterpret_cast<float4*>(out_lo + at) = make_float4(tf32_lo(y.x, ROUNDED), tf32_lo(y.y, ROUNDED), tf32_lo(y.z, ROUNDED), tf32_lo(y.w, ROUNDED));
  }
}

template <int R, int OUT>
cudaError_t launch_f32(ttb_ctx* ctx, dim3 grid, const float* qkv, const int32_t* cu, int heads, const float* mask, int64_t mbs, int64_t mrs, int causal, float scale,
                       float* out, float* out_lo, const SplitOut& split) {
  cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<R, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem<R>);
  if (e != cudaSuccess) return e;
  return launch_pdl(attention_f32_kernel<R, OUT>, grid, dim3(kThreads), (size_t)kSmem<R>, ctx->stream, qkv, cu, heads, mask, (long long)mbs, (long long)mrs, causal, scale, out,
                    out_lo, split);
}

template <int OUT>
int attention_f32(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d, const float* mask,
                  int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, float* out, float* out_lo, const SplitOut& split = SplitOut()) {
  if (!ctx) return TTB_ERR_INVALID;
  TTB_REQUIRE(ctx, d == D && heads > 0 && heads <= 65535 && B >= 0 && B <= 65535 && max_seqlen >= 0 && max_seqlen < (1 << 30), "attention_f32: bad shape");
  if (B == 0 || max_seqlen == 0) return TTB_OK;
  TTB_REQUIRE(ctx, qkv && cu_seqlens && (out || OUT == OUT_F16), "attention_f32: null pointer");
  TTB_REQUIRE(ctx, ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(out_lo)) & 15) == 0,
              "attention_f32: buffers must be 16-byte aligned");
  DeviceGuard g(ctx->device);
  // 32 rows a CTA read a tile of keys half as often as 16; with few (sequence, head, rows) the chip has room for twice the CTAs
  const int64_t ctas = B * heads * ((max_seqlen + 31) / 32);
  if (ctas >= 2 * ctx->sm_count)
    TTB_CUDA(ctx, (launch_f32<4, OUT>(ctx, dim3((unsigned)((max_seqlen + 31) / 32), (unsigned)heads, (unsigned)B), qkv, cu_seqlens, (int)heads, mask, mask_batch_stride, mask_row_stride,
                                causal, scale, out, out_lo, split)));
  else
    TTB_CUDA(ctx, (launch_f32<2, OUT>(ctx, dim3((unsigned)((max_seqlen + 15) / 16), (unsigned)heads, (unsigned)B), qkv, cu_seqlens, (int)heads, mask, mask_batch_stride, mask_row_stride,
                                causal, scale, out, out_lo, split)));
  return launched(ctx, "attention_f32");
}

}  // namespace

extern "C" int ttb_attention_f32(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d, const float* mask,
                                 int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, float* out, float* out_lo) {
  return attention_f32<OUT_VALUE>(ctx, qkv, cu_seqlens, B, max_seqlen, heads, d, mask, mask_batch_stride, mask_row_stride, causal, scale, out, out_lo);
}

extern "C" int ttb_attention_f32_planes(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d,
                                        const float* mask, int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, float* hi, float* lo) {
  if (ctx && B > 0 && max_seqlen > 0) TTB_REQUIRE(ctx, lo, "attention_f32_planes: null pointer");
  return attention_f32<OUT_TF32>(ctx, qkv, cu_seqlens, B, max_seqlen, heads, d, mask, mask_batch_stride, mask_row_stride, causal, scale, hi, lo);
}

extern "C" int ttb_attention_f32_split(ttb_ctx* ctx, const float* qkv, const int32_t* cu_seqlens, int64_t B, int64_t max_seqlen, int64_t heads, int64_t d,
                                       const float* mask, int64_t mask_batch_stride, int64_t mask_row_stride, int causal, float scale, const float* row_scale,
                                       const float* stats, void* hi, void* lo, float* out_scale) {
  if (ctx && B > 0 && max_seqlen > 0)
    TTB_REQUIRE(ctx, row_scale && stats && hi && lo && out_scale && ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 7) == 0,
                "attention_f32_split: null or misaligned pointer");
  return attention_f32<OUT_F16>(ctx, qkv, cu_seqlens, B, max_seqlen, heads, d, mask, mask_batch_stride, mask_row_stride, causal, scale, nullptr, nullptr,
                                SplitOut{row_scale, stats, static_cast<__half*>(hi), static_cast<__half*>(lo), out_scale});
}
