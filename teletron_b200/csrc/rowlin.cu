// K-ROWLIN: linear layers of one to four fp32 rows (timestep / guidance embedders, the modulation projections) with bf16
// weights, accumulated in fp32.
//
// Bound by reading the weights once: a 3072 -> 18432 projection is 113 MB.  Casting it to fp32 for a library call moved
// 113 + 2 x 226 MB and took 93 us; read as it is it takes the time of the 113 MB.
//   forward   y[b, n] = sum_k x[b, k] W[n, k] + bias[n]       a warp per two weight rows
//   dgrad     dx[b, k] = sum_n dy[b, n] W[n, k]               eight columns per thread, rows cut over CTAs, partial sums
//   wgrad     dW[n, k] (+)= sum_b dy[b, n] x[b, k]            into the fp32 gradient buffer or a bf16 gradient
#include "tt_common.cuh"

using namespace tt;

TT_API int tt_colsum_partials(const float* partial, float* out, int groups, int n, int width, int accumulate,
                              cudaStream_t stream);

namespace {

constexpr int RL_MAX = 4;

__device__ __forceinline__ void up8(const uint4& u, float (&v)[8]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16(w[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}
__device__ __forceinline__ void lf8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <int B>
__global__ void __launch_bounds__(256)
rowlin_fwd_kernel(const float* __restrict__ x, const bf16* __restrict__ w, const bf16* __restrict__ bias,
                  float* __restrict__ y, int N, int K) {
  const int lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 2;
  if (n0 >= N) return;
  const bool two = n0 + 1 < N;
  const bf16* w0 = w + (long long)n0 * K;
  const bf16* w1 = two ? w0 + K : w0;
  float acc[2][B];
#pragma unroll
  for (int b = 0; b < B; ++b) acc[0][b] = acc[1][b] = 0.f;
#pragma unroll 4
  for (int k = lane * 8; k < K; k += 256) {
    float a[8], c[8];
    up8(*reinterpret_cast<const uint4*>(w0 + k), a);
    up8(*reinterpret_cast<const uint4*>(w1 + k), c);
#pragma unroll
    for (int b = 0; b < B; ++b) {
      float v[8];
      lf8(x + (long long)b * K + k, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[0][b] += a[j] * v[j];
        acc[1][b] += c[j] * v[j];
      }
    }
  }
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const float s0 = warp_sum(acc[0][b]), s1 = warp_sum(acc[1][b]);
    if (lane == 0) {
      y[(long long)b * N + n0] = s0 + (bias ? __bfloat162float(bias[n0]) : 0.f);
      if (two) y[(long long)b * N + n0 + 1] = s1 + (bias ? __bfloat162float(bias[n0 + 1]) : 0.f);
    }
  }
}

// partial[chunk][b][k]; CTA (column block, chunk of weight rows)
template <int B>
__global__ void __launch_bounds__(256)
rowlin_dgrad_kernel(const float* __restrict__ dy, const bf16* __restrict__ w, float* __restrict__ partial, int N, int K,
                    int rows_per_chunk) {
  const int k = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (k >= K) return;
  const int n0 = blockIdx.y * rows_per_chunk, n1 = min(n0 + rows_per_chunk, N);
  float acc[B][8];
#pragma unroll
  for (int b = 0; b < B; ++b)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[b][j] = 0.f;
#pragma unroll 4
  for (int n = n0; n < n1; ++n) {
    float a[8];
    up8(*reinterpret_cast<const uint4*>(w + (long long)n * K + k), a);
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const float d = dy[(long long)b * N + n];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[b][j] += d * a[j];
    }
  }
#pragma unroll
  for (int b = 0; b < B; ++b) {
    float* p = partial + ((long long)blockIdx.y * B + b) * K + k;
    *reinterpret_cast<float4*>(p) = make_float4(acc[b][0], acc[b][1], acc[b][2], acc[b][3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(acc[b][4], acc[b][5], acc[b][6], acc[b][7]);
  }
}

template <int B, bool ACCUM>
__global__ void __launch_bounds__(256)
rowlin_wgrad_kernel(const float* __restrict__ dy, const float* __restrict__ x, void* __restrict__ dw, int N, int K) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const int kv = K >> 3;
  if (i >= (long long)N * kv) return;
  const int n = (int)(i / kv), k = (int)(i - (long long)n * kv) * 8;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int b = 0; b < B; ++b) {
    float v[8];
    lf8(x + (long long)b * K + k, v);
    const float d = dy[(long long)b * N + n];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] += d * v[j];
  }
  if (ACCUM) {
    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(dw) + (long long)n * K + k);
    float4 a = o[0], b = o[1];
    a.x += s[0]; a.y += s[1]; a.z += s[2]; a.w += s[3];
    b.x += s[4]; b.y += s[5]; b.z += s[6]; b.w += s[7];
    o[0] = a;
    o[1] = b;
  } else {
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(dw) + (long long)n * K + k) =
        make_uint4(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]), pack_bf16(s[4], s[5]), pack_bf16(s[6], s[7]));
  }
}

__global__ void __launch_bounds__(256)
rowlin_dbias_kernel(const float* __restrict__ dy, bf16* __restrict__ db, int B, int N) {
  const int n = blockIdx.x * 256 + threadIdx.x;
  if (n >= N) return;
  float s = 0.f;
  for (int b = 0; b < B; ++b) s += dy[(long long)b * N + n];
  db[n] = __float2bfloat16(s);
}

#define TT_ROWS(B, ...)                              \
  switch (B) {                                       \
    case 1: { constexpr int BB = 1; __VA_ARGS__; } break; \
    case 2: { constexpr int BB = 2; __VA_ARGS__; } break; \
    case 3: { constexpr int BB = 3; __VA_ARGS__; } break; \
    default: { constexpr int BB = 4; __VA_ARGS__; } break; \
  }

int check_rowlin(int B, int N, int K, const void* a, const void* b, const void* c) {
  TT_CHECK(B >= 1 && B <= RL_MAX && N > 0 && K > 0 && K % 8 == 0, "rowlin: bad shape %d x %d x %d", B, N, K);
  TT_CHECK((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0, "rowlin: misaligned operand");
  return 0;
}

}  // namespace

// x [B, K], y [B, N] dense fp32; w [N, K] dense bf16; bias bf16 [N] or null
TT_API int tt_rowlin_fwd(const float* x, const void* w, const void* bias, float* y, int B, int N, int K, cudaStream_t stream) {
  if (check_rowlin(B, N, K, x, w, nullptr)) return -1;
  TT_ROWS(B, rowlin_fwd_kernel<BB><<<(N + 15) / 16, 256, 0, stream>>>(x, (const bf16*)w, (const bf16*)bias, y, N, K));
  TT_LAUNCH_CHECK();
  return 0;
}

// The gradients that are wanted (null: not), as one call, since at small sizes the host's time for it is what counts: a
// 256 -> 1536 layer of one row takes 190 to 195 us forward and backward with a call per kernel, 166 us so, 156 to 167 by
// F.linear on fp32 copies.
//   dx [B, K] fp32, through partial: fp32 [chunks, B, K]
//   dw fp32 [N, K] that is added to (accumulate) or bf16 [N, K] that is written
//   db bf16 [N]
TT_API int tt_rowlin_bwd(const float* dy, const float* x, const void* w, float* partial, int chunks, float* dx, void* dw,
                         int accumulate, void* db, int B, int N, int K, cudaStream_t stream) {
  if (check_rowlin(B, N, K, x, w, dw) || check_rowlin(B, N, K, partial, nullptr, nullptr)) return -1;
  if (dx) {
    TT_CHECK(partial && chunks >= 1 && chunks <= 65535, "rowlin_bwd: bad chunk count");
    const dim3 grid((K / 8 + 255) / 256, chunks);
    TT_ROWS(B, rowlin_dgrad_kernel<BB><<<grid, 256, 0, stream>>>(dy, (const bf16*)w, partial, N, K, (N + chunks - 1) / chunks));
    TT_LAUNCH_CHECK();
    if (tt_colsum_partials(partial, dx, 1, chunks, B * K, 0, stream)) return -1;
  }
  if (dw) {
    const long long blocks = ((long long)N * (K / 8) + 255) / 256;
    TT_CHECK(blocks < (1ll << 31), "rowlin_bwd: too large");
    if (accumulate) TT_ROWS(B, (rowlin_wgrad_kernel<BB, true><<<(unsigned)blocks, 256, 0, stream>>>(dy, x, dw, N, K)))
    else TT_ROWS(B, (rowlin_wgrad_kernel<BB, false><<<(unsigned)blocks, 256, 0, stream>>>(dy, x, dw, N, K)))
    TT_LAUNCH_CHECK();
  }
  if (db) {
    rowlin_dbias_kernel<<<(N + 255) / 256, 256, 0, stream>>>(dy, (bf16*)db, B, N);
    TT_LAUNCH_CHECK();
  }
  return 0;
}
