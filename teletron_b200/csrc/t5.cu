// K-T5: the pointwise work of the umT5 text encoder, one pass over memory each.
//   tt_t5_add_norm   x (+ delta) and its T5 layer norm (RMS, no bias)
//   tt_t5_geglu      fc1 * gelu_tanh(gate)
//   tt_t5_bias       attention bias of one layer: relative-position embedding, lowest value where the key is masked
// Intermediate values are rounded to bf16 where the module chain rounds them.  The norm's fp32 sum runs in another order,
// so single roundings of its result differ; over the 24 layers of the full encoder the states are 2.16 % from fp64 either
// way, and as far from each other.
#include "tt_common.cuh"

using namespace tt;

namespace {

__device__ __forceinline__ void ld8(const bf16* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16(w[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 pk8(const float (&v)[8]) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
__device__ __forceinline__ float rnd(float x) { return __bfloat162float(__float2bfloat16(x)); }

// One row per CTA of 256 threads, VPT vectors of eight per thread: 6 us at 1,024 rows x 4,096 (nine ATen launches before,
// 34 us).
template <int VPT>
__global__ void __launch_bounds__(256)
t5_add_norm_kernel(const bf16* __restrict__ x, const bf16* __restrict__ delta, bf16* __restrict__ xo, bf16* __restrict__ y,
                   const bf16* __restrict__ w, int C, float eps) {
  __shared__ float red[8];
  const long long row = (long long)blockIdx.x * C;
  const int nvec = C >> 3;
  float v[VPT][8];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int i = threadIdx.x + k * 256;
    if (i < nvec) {
      ld8(x + row + i * 8, v[k]);
      if (delta) {
        float d[8];
        ld8(delta + row + i * 8, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[k][j] = rnd(v[k][j] + d[j]);
        *reinterpret_cast<uint4*>(xo + row + i * 8) = pk8(v[k]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += v[k][j] * v[k][j];
    }
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += red[i];
  const float r = rsqrtf(t / (float)C + eps);
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int i = threadIdx.x + k * 256;
    if (i < nvec) {
      float wv[8];
      ld8(w + i * 8, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[k][j] = rnd(v[k][j] * r) * wv[j];
      *reinterpret_cast<uint4*>(y + row + i * 8) = pk8(v[k]);
    }
  }
}

__device__ __forceinline__ float gelu_tanh_exact(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
}
__global__ void __launch_bounds__(256)
t5_geglu_kernel(const bf16* __restrict__ a, const bf16* __restrict__ g, bf16* __restrict__ y, long long nvec) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= nvec) return;
  float av[8], gv[8];
  ld8(a + i * 8, av);
  ld8(g + i * 8, gv);
#pragma unroll
  for (int j = 0; j < 8; ++j) av[j] *= rnd(gelu_tanh_exact(gv[j]));
  *reinterpret_cast<uint4*>(y + i * 8) = pk8(av);
}

// out[b, h, i, j] = keep[b, j] ? emb[bucket[j - i + n - 1], h] : lowest bf16.  A CTA handles eight query rows of one
// (b, h): the head's 2n - 1 position values and the key mask are staged in shared memory once.  Bound by the write: 35 us
// for 2 x 64 x 512 x 512, where gather, permuted copy, add and masked fill took 375 us.
__global__ void __launch_bounds__(256)
t5_bias_kernel(const bf16* __restrict__ emb, const int* __restrict__ bucket, const unsigned char* __restrict__ keep,
               bf16* __restrict__ out, int heads, int n) {
  extern __shared__ unsigned short vals[];  // [2n - 1] position values, then [n] flags
  const int h = blockIdx.y, b = blockIdx.z;
  unsigned short* msk = vals + 2 * n - 1;
  for (int i = threadIdx.x; i < 2 * n - 1; i += 256)
    vals[i] = *reinterpret_cast<const unsigned short*>(emb + (long long)bucket[i] * heads + h);
  for (int i = threadIdx.x; i < n; i += 256) msk[i] = keep ? keep[(long long)b * n + i] : 1;
  __syncthreads();
  const unsigned short lowest = 0xFF7F;
  const int r0 = blockIdx.x * 8;
  if ((n & 7) == 0) {
    const int per_row = n >> 3;
    for (int v = threadIdx.x; v < 8 * per_row; v += 256) {
      const int i = r0 + v / per_row, j = (v % per_row) * 8;
      if (i >= n) break;
      unsigned short u[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) u[k] = msk[j + k] ? vals[j + k - i + n - 1] : lowest;
      *reinterpret_cast<uint4*>(out + (((long long)b * heads + h) * n + i) * n + j) =
          make_uint4(u[0] | (uint32_t)u[1] << 16, u[2] | (uint32_t)u[3] << 16, u[4] | (uint32_t)u[5] << 16, u[6] | (uint32_t)u[7] << 16);
    }
  } else {
    for (int v = threadIdx.x; v < 8 * n; v += 256) {
      const int i = r0 + v / n, j = v % n;
      if (i >= n) break;
      reinterpret_cast<unsigned short*>(out)[(((long long)b * heads + h) * n + i) * n + j] = msk[j] ? vals[j - i + n - 1] : lowest;
    }
  }
}

}  // namespace

TT_API int tt_t5_add_norm(const void* x, const void* delta, void* x_out, void* y, const void* w, long long rows, int C,
                          float eps, cudaStream_t stream) {
  TT_CHECK(rows > 0 && rows < (1ll << 31) && C > 0 && C % 8 == 0 && C <= 8192, "t5_add_norm: bad shape");
  TT_CHECK((((uintptr_t)x | (uintptr_t)delta | (uintptr_t)x_out | (uintptr_t)y | (uintptr_t)w) & 15) == 0 &&
               (!delta || x_out), "t5_add_norm: bad pointers");
#define TT_T5(V) t5_add_norm_kernel<V><<<(unsigned)rows, 256, 0, stream>>>((const bf16*)x, (const bf16*)delta, (bf16*)x_out, (bf16*)y, (const bf16*)w, C, eps)
  if (C <= 2048) TT_T5(1);
  else if (C <= 4096) TT_T5(2);
  else TT_T5(4);
#undef TT_T5
  TT_LAUNCH_CHECK();
  return 0;
}

TT_API int tt_t5_geglu(const void* a, const void* g, void* y, long long n, cudaStream_t stream) {
  TT_CHECK(n > 0 && n % 8 == 0 && (((uintptr_t)a | (uintptr_t)g | (uintptr_t)y) & 15) == 0, "t5_geglu: bad arguments");
  t5_geglu_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, stream>>>((const bf16*)a, (const bf16*)g, (bf16*)y, n / 8);
  TT_LAUNCH_CHECK();
  return 0;
}

// bucket: int32 [2n - 1], row of `emb` [*, heads] for the distances j - i = 1 - n .. n - 1; keep: uint8 [B, n] or null
TT_API int tt_t5_bias(const void* emb, const int* bucket, const unsigned char* keep, void* out, int B, int heads, int n,
                      cudaStream_t stream) {
  TT_CHECK(B > 0 && B < 65536 && heads > 0 && heads < 65536 && n > 0 && n <= 8000 && ((uintptr_t)out & 15) == 0, "t5_bias: bad arguments");
  t5_bias_kernel<<<dim3((n + 7) / 8, heads, B), 256, (3 * n - 1) * 2, stream>>>((const bf16*)emb, bucket, keep, (bf16*)out, heads, n);
  TT_LAUNCH_CHECK();
  return 0;
}
