// Softmax of fp32 score rows for a product that takes bf16 operands: every probability is written as the sum of two or
// three bf16 values (each the rounded remainder of the ones before).  Two keep 16 of its bits; three keep all 24, so that
// P V by three bf16 products takes the fp32 probability itself.
//
// The single-head attention of the video VAE has heads of 384, for which the library only has its fp32 fallback (two
// SIMT products and a softmax, 1.2 ms per 60 x 104 frame). With scores = Q K^T from the GEMM kernel (exact products of
// bf16 operands, fp32 accumulation) and [P_0 | P_1 | P_2] [V; V; V] as one product it is bound by writing and reading the
// scores. One CTA per row; the row is read three times, twice from L1 / L2.
#include "tt_common.cuh"

using namespace tt;

namespace {

__device__ __forceinline__ float block_reduce(float v, bool maximum, float* red) {
  v = maximum ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) t = maximum ? fmaxf(t, red[i]) : t + red[i];
  return t;
}

template <int PARTS>
__global__ void __launch_bounds__(256)
softmax_split_kernel(const float* __restrict__ s, bf16* __restrict__ p, int n, int np) {
  __shared__ float red[8];
  const float* row = s + (long long)blockIdx.x * np;
  bf16* out = p + (long long)blockIdx.x * PARTS * np;
  auto get = [&](int j, float (&v)[4]) {
    const float4 f = *reinterpret_cast<const float4*>(row + j);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  };
  float m = -INFINITY;
  for (int j = threadIdx.x * 4; j < np; j += 1024) {
    float v[4];
    get(j, v);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j + k < n) m = fmaxf(m, v[k]);
  }
  m = block_reduce(m, true, red);
  float sum = 0.f;
  for (int j = threadIdx.x * 4; j < np; j += 1024) {
    float v[4];
    get(j, v);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j + k < n) sum += expf(v[k] - m);
  }
  const float inv = 1.f / block_reduce(sum, false, red);
  for (int j = threadIdx.x * 4; j < np; j += 1024) {
    float v[4], h[4];
    get(j, v);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = j + k < n ? expf(v[k] - m) * inv : 0.f;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        h[k] = __bfloat162float(__float2bfloat16(v[k]));
        v[k] -= h[k];  // exact
      }
      *reinterpret_cast<uint2*>(out + (long long)i * np + j) = make_uint2(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]));
    }
  }
}

}  // namespace

// s: fp32 [rows, np], the first n columns are scores; p: bf16 [rows, parts, np], zero past column n
TT_API int tt_softmax_split(const float* s, void* p, long long rows, int n, int np, int parts, cudaStream_t stream) {
  TT_CHECK(rows > 0 && rows < (1ll << 31) && n > 0 && np >= n && np % 8 == 0 && (parts == 2 || parts == 3),
           "softmax_split: bad shape");
  TT_CHECK((((uintptr_t)s | (uintptr_t)p) & 15) == 0, "softmax_split: misaligned");
  auto kern = parts == 2 ? softmax_split_kernel<2> : softmax_split_kernel<3>;
  kern<<<(unsigned)rows, 256, 0, stream>>>(s, (bf16*)p, n, np);
  TT_LAUNCH_CHECK();
  return 0;
}
