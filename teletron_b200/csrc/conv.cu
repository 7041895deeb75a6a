// K-CONV3D: causal 3-D convolutions of the video VAE as an implicit GEMM on tcgen05 tensor cores, and the pointwise
// kernels around it (channel RMS norm + SiLU, layout changes, weight packing).
//
// Layout.  Activations are kept frame by frame in channel chunks of 16 bytes: [T][C / E][H][W][E] with E = 8 (bf16) or
// 4 (fp32, multiplied as TF32).  A TMA box of (w, h) pixels x KC chunks of one frame then lands in shared memory as KC
// planes of consecutive 16-byte pixels, which is the unswizzled K-major operand layout of tcgen05 (8 rows x 16 bytes
// per core matrix): the rows of an MMA are 8 pixels along w, groups of 8 rows step one pixel row down, and a spatial
// tap (dy, dx) is the same tile with its start address moved by (dy * box_w + dx) * 16 bytes.  One load of an
// 18 x 18 pixel box therefore feeds all nine taps of a 3 x 3 window.  At 96 channels a tap is 2 x 6 MMAs of 48 clocks: a
// fresh tile of 256 pixels per tap (49 KB) would need 85 B per clock and SM, the box (62 KB for nine taps) needs 12.  Padding is the zero fill of out-of-range box coordinates; frames
// before the first are not loaded and their taps are skipped.  A CTA owns 16 x 16 output pixels (two 128-row
// accumulators) x NT <= 192 output channels, so that every weight tile that comes from L2 is used twice.
//
// Weights are packed once per call into the order in which the B ring consumes them (tt_conv_pack), a contiguous
// cp.async.bulk per ring slot.  A stride-2 window is a 1-stride one over the four pixel phases of its input
// (tt_blk_move mode 1), each phase with its own taps.
//
// Roles (384 threads): warp 0 input boxes, warp 1 weight tiles, warps 2 and 3 MMA issue (one 128-row accumulator each;
// warp 2 also holds the tensor memory), warps 4..11 epilogue (bias, residual, store).  Every wait is bounded.
//
// What bounds it: the issuing threads.  An MMA is 48 to 96 clocks, and the wait, fence and commit around a weight tile cost
// one thread about as much as the tile's MMAs: with a single issuer halving its MMAs took away a fifth of the time, while
// loading no input, loading no weights, aligning every operand row or padding the weight planes changed nothing.  Two
// issuers hide each other's waits, and the loop over a weight tile is unrolled.
#include "tt_common.cuh"

using namespace tt;

namespace {

constexpr int CV_TW = 16, CV_TH = 16;  // output pixels of a tile
constexpr int CV_MAX_A = 4, CV_MAX_B = 8;
constexpr int CV_A_BYTES = 124416;     // input ring: two 18 x 18 boxes of 12 chunks
constexpr int CV_B_BYTES = 92160;      // weight ring: five tiles of 192 x 6 chunks
constexpr int CV_SMEM = CV_A_BYTES + CV_B_BYTES + 1024 + 256;
constexpr int CV_THREADS = 384;

struct ConvGroup {   // taps that read the same frame and channel range
  int dt, chunk0, n_taps;
  int off[9];        // pixel offset of each tap inside the box
};
struct ConvParams {
  int tiles_w, tiles_h, n_tiles, num_tiles;
  int T, H, W;                 // output frames and pixels
  int NT, KC, UC, n_cb;        // output channels per tile, chunks per input box, chunks per weight tile, boxes per group
  int box_w, plane;            // pixels per box row; bytes of one chunk plane of the box
  int a_bytes, a_slot, b_bytes, a_stages, b_stages;  // a_slot: a_bytes in steps of 128
  int n_groups, t_stride, t_off, pad;
  ConvGroup g[4];
  const uint8_t* B;
  long long b_tile_bytes;      // packed weights of one output-channel tile
  const float* bias;           // [N], fp32
  void* out;
  const void* res;             // residual in the output's layout, or null
  int C_out;                   // channels per output frame; channel n >= C_out goes to frame t * t_mul + n / C_out
  int t_mul;
  int planar;                  // 1: out is [C_real][T][H][W]
  int C_real;
  unsigned* status;
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ float round_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
template <bool F32>
__device__ __forceinline__ void umma_conv(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                          uint32_t idesc, uint32_t acc) {
  if constexpr (F32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\tmov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], ad, bd, %5, p;\n\t}" ::"r"(d),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\tmov.b64 ad, {%1, %2};\n\tmov.b64 bd, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %5, p;\n\t}" ::"r"(d),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc)
        : "memory");
  }
}
// STEPS consecutive 32-byte steps along K
template <bool F32, int STEPS>
__device__ __forceinline__ void umma_steps(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t a_step, uint32_t b_lo,
                                           uint32_t b_hi, uint32_t b_step, uint32_t idesc, uint32_t acc) {
#pragma unroll
  for (int k = 0; k < STEPS; ++k)
    umma_conv<F32>(d, a_lo + k * a_step, a_hi, b_lo + k * b_step, b_hi, idesc, k ? 1u : acc);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// the 16 bytes of chunk elements <-> floats
template <bool F32> struct Chunk;
template <> struct Chunk<false> {
  static constexpr int E = 8;
  static __device__ __forceinline__ void get(const uint4& u, float (&v)[8]) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16(w[j]);
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
    }
  }
  static __device__ __forceinline__ uint4 put(const float* v) {
    return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  }
};
template <> struct Chunk<true> {
  static constexpr int E = 4;
  static __device__ __forceinline__ void get(const uint4& u, float (&v)[4]) {
    v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
  }
  static __device__ __forceinline__ uint4 put(const float* v) {
    return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  }
};

struct TileAt { int nt, t, h0, w0; };
__device__ __forceinline__ TileAt conv_tile(const ConvParams& p, int tile) {
  // output-channel tiles of the same pixels next to each other, then frames: neighbours in time re-read the same
  // boxes while they are still in L2
  TileAt a;
  a.nt = tile % p.n_tiles;
  tile /= p.n_tiles;
  a.t = tile % p.T;
  tile /= p.T;
  a.w0 = (tile % p.tiles_w) * CV_TW;
  a.h0 = (tile / p.tiles_w) * CV_TH;
  return a;
}

template <bool F32>
__global__ void __launch_bounds__(CV_THREADS, 1)
conv_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ ConvParams p) {
  constexpr int E = Chunk<F32>::E;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + CV_A_BYTES;
  uint64_t* a_full = reinterpret_cast<uint64_t*>(smem + CV_A_BYTES + CV_B_BYTES);
  uint64_t* a_empty = a_full + CV_MAX_A;
  uint64_t* b_full = a_empty + CV_MAX_A;
  uint64_t* b_empty = b_full + CV_MAX_B;
  uint64_t* tfull = b_empty + CV_MAX_B;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_acc = p.NT <= 128 ? 2 : 1;  // accumulator buffers: 2 x 128 rows x NT columns each, 512 columns in all
  if (threadIdx.x == 0) {
    for (int i = 0; i < CV_MAX_A; ++i) { mbar_init(&a_full[i], 1); mbar_init(&a_empty[i], 2); }
    for (int i = 0; i < CV_MAX_B; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 2); }
    for (int i = 0; i < 2; ++i) { mbar_init(&tfull[i], 2); mbar_init(&tempty[i], 8); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) tma_prefetch_desc(&tmA);
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {  // ---------------------------------------------- input boxes
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
        const TileAt a = conv_tile(p, tile);
        for (int g = 0; g < p.n_groups && ok; ++g) {
          const int f = a.t * p.t_stride + p.g[g].dt + p.t_off;
          if (f < 0) continue;
          for (int cb = 0; cb < p.n_cb; ++cb) {
            if (!mbar_wait(&a_empty[s], ph ^ 1, abort_flag, p.status, TT_ST_TIMEOUT_PRODUCER)) { ok = false; break; }
            mbar_expect_tx(&a_full[s], p.a_bytes);
            tma_load_4d(sA + s * p.a_slot, &tmA, &a_full[s], (a.w0 - p.pad) * E, a.h0 - p.pad,
                        p.g[g].chunk0 + cb * p.KC, f);
            if (++s == p.a_stages) { s = 0; ph ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---------------------------------------------- weight tiles
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      const int per_box = p.KC / p.UC;
      for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
        const TileAt a = conv_tile(p, tile);
        const uint8_t* src = p.B + a.nt * p.b_tile_bytes;
        for (int g = 0; g < p.n_groups && ok; ++g) {
          const int units = p.n_cb * p.g[g].n_taps * per_box;
          if (a.t * p.t_stride + p.g[g].dt + p.t_off >= 0) {
            for (int u = 0; u < units; ++u) {
              if (!mbar_wait(&b_empty[s], ph ^ 1, abort_flag, p.status, TT_ST_TIMEOUT_PRODUCER + 1)) { ok = false; break; }
              mbar_expect_tx(&b_full[s], p.b_bytes);
              bulk_load(sB + s * p.b_bytes, src + (long long)u * p.b_bytes, p.b_bytes, &b_full[s]);
              if (++s == p.b_stages) { s = 0; ph ^= 1; }
            }
          }
          src += (long long)units * p.b_bytes;
        }
      }
    }
  } else if (warp < 4) {
    if (lane == 0) {  // ---------------------------------------------- MMA issue
      const int m = warp - 2;
      // bits 7..9 / 10..12: operand formats (1 = bf16, 2 = tf32); fp32 accumulate; both K-major
      const uint32_t fmt = F32 ? 2u : 1u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.NT >> 3) << 17) | (8u << 24);
      // unswizzled K-major descriptors: leading offset = next 16-byte chunk along K, stride offset = next 8 rows
      const uint32_t a_hi = (uint32_t)(p.box_w & 0x3FFF) | (1u << 14);  // box_w pixels of 16 bytes to the next row
      const uint32_t b_hi = 8u | (1u << 14);
      const uint32_t a_lbo = (uint32_t)(p.plane >> 4), b_lbo = (uint32_t)p.NT;
      const uint32_t a_top = a_lbo << 16, b_top = b_lbo << 16;
      const int per_box = p.KC / p.UC;
      int sa = 0, sb = 0, tcount = 0;
      uint32_t pa = 0, pb = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x, ++tcount) {
        const TileAt at = conv_tile(p, tile);
        const int buf = n_acc == 2 ? (tcount & 1) : 0;
        const uint32_t tph = n_acc == 2 ? ((tcount >> 1) & 1) : (tcount & 1);
        if (!mbar_wait(&tempty[buf], tph ^ 1, abort_flag, p.status, TT_ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + buf * 256 + m * p.NT;
        uint32_t acc = 0;
        for (int g = 0; g < p.n_groups && ok; ++g) {
          if (at.t * p.t_stride + p.g[g].dt + p.t_off < 0) continue;
          for (int cb = 0; cb < p.n_cb && ok; ++cb) {
            if (!mbar_wait(&a_full[sa], pa, abort_flag, p.status, TT_ST_TIMEOUT_MMA + 1)) { ok = false; break; }
            const uint32_t a0 = (smem_u32(sA + sa * p.a_slot) >> 4) + m * 8;
            for (int tap = 0; tap < p.g[g].n_taps && ok; ++tap) {
              uint32_t ax = a_top | (a0 + p.g[g].off[tap]);
              for (int u = 0; u < per_box; ++u) {
                if (!mbar_wait(&b_full[sb], pb, abort_flag, p.status, TT_ST_TIMEOUT_MMA + 2)) { ok = false; break; }
                tc_fence_after();
                const uint32_t bx = b_top | (smem_u32(sB + sb * p.b_bytes) >> 4);
                if (p.UC == 12) {
                  umma_steps<F32, 6>(d, ax, a_hi, 2 * a_lbo, bx, b_hi, 2 * b_lbo, idesc, acc);
                } else if (p.UC == 6) {
                  umma_steps<F32, 3>(d, ax, a_hi, 2 * a_lbo, bx, b_hi, 2 * b_lbo, idesc, acc);
                } else {
                  for (int k = 0; k < p.UC; k += 2)
                    umma_steps<F32, 1>(d, ax + k * a_lbo, a_hi, 0, bx + k * b_lbo, b_hi, 0, idesc, k ? 1u : acc);
                }
                acc = 1;
                ax += p.UC * a_lbo;
                tc_commit(&b_empty[sb]);
                if (++sb == p.b_stages) { sb = 0; pb ^= 1; }
              }
            }
            if (!ok) break;
            tc_commit(&a_empty[sa]);
            if (++sa == p.a_stages) { sa = 0; pa ^= 1; }
          }
        }
        if (ok) tc_commit(&tfull[buf]);
      }
    }
  } else if (warp >= 4) {  // ------------------------------------------- epilogue
    const int q = warp & 3, m = (warp - 4) >> 2;
    const long long hw = (long long)p.H * p.W;
    int tcount = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++tcount) {
      const TileAt at = conv_tile(p, tile);
      const int buf = n_acc == 2 ? (tcount & 1) : 0;
      const uint32_t tph = n_acc == 2 ? ((tcount >> 1) & 1) : (tcount & 1);
      if (!mbar_wait_warp(&tfull[buf], tph, abort_flag, p.status, TT_ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      const uint32_t tm = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256 + m * p.NT;
      const int h = at.h0 + q * 4 + (lane >> 3), w = at.w0 + m * 8 + (lane & 7);
      const bool in = h < p.H && w < p.W;
      const long long pix = (long long)h * p.W + w;
      const int n0 = at.nt * p.NT;
      for (int c = 0; c < p.NT; c += 16) {
        uint32_t r[16];
        tmem_ld16(tm + c, r);
        const int n = n0 + c;
        float v[16], b[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(&b[4 * j]) = *reinterpret_cast<const float4*>(p.bias + n + 4 * j);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + b[j];
        if (!in) {
        } else if (p.planar) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (n + j < p.C_real) {
              const long long i = ((long long)(n + j) * p.T + at.t) * hw + pix;
              if (F32) reinterpret_cast<float*>(p.out)[i] = v[j];
              else reinterpret_cast<bf16*>(p.out)[i] = __float2bfloat16(v[j]);
            }
          }
        } else {
          const int half = n / p.C_out;
          const long long base = ((long long)(at.t * p.t_mul + half) * (p.C_out / E) + (n - half * p.C_out) / E) * hw + pix;
          uint4* o = reinterpret_cast<uint4*>(p.out) + base;
#pragma unroll
          for (int k = 0; k < 16 / E; ++k) {
            if (p.res) {
              float rv[E];
              Chunk<F32>::get(reinterpret_cast<const uint4*>(p.res)[base + k * hw], rv);
#pragma unroll
              for (int j = 0; j < E; ++j) v[k * E + j] += rv[j];
            }
            o[k * hw] = Chunk<F32>::put(&v[k * E]);
          }
        }
        __syncwarp();  // tcgen05.ld is warp-collective
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
  }

  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies still in flight land before the shared memory goes away
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem_base, 512);
}

// ------------------------------------------------------------------ weight packing
// [N_real][C_real][taps_total] -> tiles in ring order: [n tile][group][box][tap][chunk][n][e].  Padding is zero.
struct PackParams {
  int N_real, C_real, taps_total, n_groups, NT, KC, n_cb, n_tiles;
  int n_taps[4];
  int tap_id[4][9];
};
template <bool F32>
__global__ void __launch_bounds__(256)
conv_pack_kernel(const void* __restrict__ src, const void* __restrict__ bias, void* __restrict__ dst, const PackParams p,
                 long long chunks_per_tile) {
  constexpr int E = Chunk<F32>::E;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;  // one 16-byte chunk of one output channel
  const long long total = chunks_per_tile * p.n_tiles * p.NT;
  if (i < p.n_tiles * p.NT) {  // the bias follows the weights, in fp32
    float b = 0.f;
    if (bias && i < p.N_real) b = F32 ? reinterpret_cast<const float*>(bias)[i] : __bfloat162float(reinterpret_cast<const bf16*>(bias)[i]);
    reinterpret_cast<float*>(reinterpret_cast<uint4*>(dst) + total)[i] = b;
  }
  if (i >= total) return;
  const int n = (int)(i % p.NT);
  long long r = i / p.NT;
  const int nt = (int)(r / chunks_per_tile);
  r -= nt * chunks_per_tile;
  int g = 0;
  while (g + 1 < p.n_groups && r >= (long long)p.n_cb * p.n_taps[g] * p.KC) r -= (long long)p.n_cb * p.n_taps[g++] * p.KC;
  const int k = (int)(r % p.KC);
  r /= p.KC;
  const int tap = (int)(r % p.n_taps[g]);
  const int cb = (int)(r / p.n_taps[g]);
  const int c0 = (cb * p.KC + k) * E, col = nt * p.NT + n;
  float v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    v[j] = 0.f;
    if (col < p.N_real && c0 + j < p.C_real) {
      const long long s = ((long long)col * p.C_real + c0 + j) * p.taps_total + p.tap_id[g][tap];
      v[j] = F32 ? round_tf32(reinterpret_cast<const float*>(src)[s]) : __bfloat162float(reinterpret_cast<const bf16*>(src)[s]);
    }
  }
  reinterpret_cast<uint4*>(dst)[i] = Chunk<F32>::put(v);
}

// ------------------------------------------------------------------ channel RMS norm + SiLU
// y = silu(x / max(|x|, 1e-12) * sqrt(C) * gamma), |x| over the channels of a pixel.  Bound by memory: one read, one
// write.  Four slices of a pixel's chunks per block column keep at most 24 chunks in registers; consecutive threads
// hold consecutive pixels, so every access is a full 512-byte row of a plane: 9 x 480 x 832 x 96 channels in 0.34 ms in bf16
// (4.0 TB/s; six ATen passes before), 0.44 ms in fp32 (6.2 TB/s).  In bf16 the exponential is the hardware's: with expf the
// pass takes 0.37 ms and the error against 64 bits is the same in all eight digits (1.6731514e-3 at 96 channels, the torch
// operators' 4.4e-3), because the result is rounded to bf16.
template <bool F32, int NCH>
__global__ void __launch_bounds__(256)
chan_norm_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, const void* __restrict__ gamma, long long hw,
                 int chunks, float scale, int act) {
  constexpr int E = Chunk<F32>::E;
  __shared__ float red[4][64];
  const int px = threadIdx.x & 63, sl = threadIdx.x >> 6;
  const long long pix = (long long)blockIdx.x * 64 + px;
  const long long base = (long long)blockIdx.y * chunks * hw + pix;
  const bool in = pix < hw;
  uint4 v[NCH];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    const int c = sl + 4 * k;
    v[k] = make_uint4(0, 0, 0, 0);
    if (in && c < chunks) v[k] = x[base + c * hw];
  }
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    float f[E];
    Chunk<F32>::get(v[k], f);
#pragma unroll
    for (int j = 0; j < E; ++j) ss += f[j] * f[j];
  }
  red[sl][px] = ss;
  __syncthreads();
  if (!in) return;
  const float nrm = sqrtf((red[0][px] + red[1][px]) + (red[2][px] + red[3][px]));
  const float inv = scale / (nrm < 1e-12f ? 1e-12f : nrm);  // a NaN stays one
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    const int c = sl + 4 * k;
    if (c < chunks) {
      float f[E], g[E];
      Chunk<F32>::get(v[k], f);
      Chunk<F32>::get(reinterpret_cast<const uint4*>(gamma)[c], g);
#pragma unroll
      for (int j = 0; j < E; ++j) {
        float t = f[j] * inv * g[j];
        if (act) t = t / (1.f + (F32 ? expf(-t) : __expf(-t)));  // see above
        f[j] = F32 ? round_tf32(t) : t;
      }
      y[base + c * hw] = Chunk<F32>::put(f);
    }
  }
}

// ------------------------------------------------------------------ layout changes (one thread per 16-byte chunk)
// [C][T][H][W] (any strides, in elements) -> chunks; channels past C are zero
template <bool F32>
__global__ void __launch_bounds__(256)
blk_from_planar_kernel(const void* __restrict__ src, uint4* __restrict__ dst, int C, int chunks, int T, int H, int W,
                       long long sc, long long st, long long sh, long long sw, int round) {
  constexpr int E = Chunk<F32>::E;
  const long long hw = (long long)H * W;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)T * chunks * hw) return;
  const long long pix = i % hw;
  const int c = (int)((i / hw) % chunks), t = (int)(i / hw / chunks);
  const long long o = t * st + (pix / W) * sh + (pix % W) * sw;
  float v[E];
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const int ch = c * E + j;
    v[j] = 0.f;
    if (ch < C) {
      v[j] = F32 ? reinterpret_cast<const float*>(src)[o + ch * sc] : __bfloat162float(reinterpret_cast<const bf16*>(src)[o + ch * sc]);
      if (F32 && round) v[j] = round_tf32(v[j]);
    }
  }
  dst[i] = Chunk<F32>::put(v);
}
// chunks -> dense [C][T][H][W]
template <bool F32>
__global__ void __launch_bounds__(256)
blk_to_planar_kernel(const uint4* __restrict__ src, void* __restrict__ dst, int chunks, int T, long long hw) {
  constexpr int E = Chunk<F32>::E;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)T * chunks * hw) return;
  const long long pix = i % hw;
  const int c = (int)((i / hw) % chunks), t = (int)(i / hw / chunks);
  float v[E];
  Chunk<F32>::get(src[i], v);
#pragma unroll
  for (int j = 0; j < E; ++j) {
    const long long o = ((long long)(c * E + j) * T + t) * hw + pix;
    if (F32) reinterpret_cast<float*>(dst)[o] = v[j];
    else reinterpret_cast<bf16*>(dst)[o] = __float2bfloat16(v[j]);
  }
}
// mode 0: nearest 2x enlargement [T][n][H][W] -> [T][n][2H][2W]
// mode 1: pixel phases [T][n][H][W] -> [T][4][n][(H+1)/2][(W+1)/2], zero outside
// mode 2: copy
// fp32 is rounded to TF32, so that the tensor cores' truncation does not bias the product
template <bool F32>
__global__ void __launch_bounds__(256)
blk_move_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int mode, long long planes, int n, int H, int W) {
  constexpr int E = Chunk<F32>::E;
  const int Ho = mode == 0 ? 2 * H : mode == 1 ? (H + 1) / 2 : H, Wo = mode == 0 ? 2 * W : mode == 1 ? (W + 1) / 2 : W;
  const long long hwo = (long long)Ho * Wo;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= planes * hwo) return;
  const long long pl = i / hwo;
  const int pix = (int)(i - pl * hwo), ho = pix / Wo, wo = pix - ho * Wo;
  long long sp = pl;
  int h = ho, w = wo;
  if (mode == 0) {
    h >>= 1;
    w >>= 1;
  } else if (mode == 1) {
    const long long t = pl / (4 * n);
    const int r = (int)(pl - t * 4 * n), phase = r / n;
    sp = t * n + (r - phase * n);
    h = 2 * ho + (phase >> 1);
    w = 2 * wo + (phase & 1);
  }
  uint4 u = make_uint4(0, 0, 0, 0);
  if (h < H && w < W) u = src[(sp * H + h) * W + w];
  if (F32) {
    float v[E];
    Chunk<F32>::get(u, v);
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = round_tf32(v[j]);
    u = Chunk<F32>::put(v);
  }
  dst[i] = u;
}

int largest_even_divisor(int n, int cap) {
  for (int d = cap < n ? cap : n; d >= 2; --d)
    if (n % d == 0 && d % 2 == 0) return d;
  return 0;
}
struct ConvShape { int NT, KC, UC, n_cb, n_tiles; };
// How a convolution of `chunks` input chunks (per tap) and N output channels (both padded) is cut: NT output channels per
// tile (two accumulators of 128 rows fit tensor memory twice up to 128, once up to 256 columns), boxes of up to 12
// chunks (62 KB, two in flight), weight tiles of at most 18 KB.
int conv_shape(int chunks, int N, int nt, ConvShape* s) {
  if (chunks < 2 || chunks % 2 || N < 16 || N % 16 || nt < 16 || nt > 192 || nt % 16 || N % nt) return -1;
  s->NT = nt;
  s->n_tiles = N / nt;
  s->KC = largest_even_divisor(chunks, 12);
  s->n_cb = chunks / s->KC;
  s->UC = largest_even_divisor(s->KC, CV_B_BYTES / 5 / (nt * 16));
  return s->KC && s->UC ? 0 : -1;
}
// kind 0: k_t x 3 x 3 pad 1; 1: k_t x 1 x 1; 2: 3 x 3 stride 2 over pixel phases
int conv_groups(int kind, int kt, int chunks, int box_w, ConvGroup* g, int tap_id[4][9]) {
  if (kind == 2) {
    for (int ph = 0; ph < 4; ++ph) {
      ConvGroup& q = g[ph];
      q.dt = 0; q.chunk0 = ph * chunks; q.n_taps = 0;
      for (int dy = ph >> 1; dy < 3; dy += 2)
        for (int dx = ph & 1; dx < 3; dx += 2) {
          tap_id[ph][q.n_taps] = dy * 3 + dx;
          q.off[q.n_taps++] = (dy >> 1) * box_w + (dx >> 1);
        }
    }
    return 4;
  }
  const int ks = kind == 0 ? 3 : 1;
  for (int t = 0; t < kt; ++t) {
    g[t].dt = t; g[t].chunk0 = 0; g[t].n_taps = ks * ks;
    for (int i = 0; i < ks * ks; ++i) {
      g[t].off[i] = (i / ks) * box_w + i % ks;
      tap_id[t][i] = t * ks * ks + i;
    }
  }
  return kt;
}

}  // namespace

// Output channels per tile for `frames` x H x W output pixels: the widest divisor of N whose waves over the SMs, times
// the cost of a wave, are fewest.  Measured with 384 channels, a wave of tiles wider than 96 takes 75 us, a wave of 96
// down to 16 takes 50 (the issue of an MMA bounds the narrow ones), so 96 pays where 192 would leave SMs idle:
// 3 x 30 x 52 pixels are 48 tiles of 192 (91.8 us) or 96 tiles of 96 (70.6 us); 5 x 120 x 208 take 604 and 772 us.
TT_API int tt_conv_tile_channels(int N, int frames, int H, int W, int sms) {
  if (N < 16 || N % 16 || frames < 1 || H < 1 || W < 1 || sms < 1) return -1;
  const long long pix = (long long)((W + CV_TW - 1) / CV_TW) * ((H + CV_TH - 1) / CV_TH) * frames;
  int best = -1;
  double cost = 0;
  for (int nt = 192; nt >= 16; nt -= 16) {
    if (N % nt) continue;
    const long long waves = (pix * (N / nt) + sms - 1) / sms;
    const double c = (double)waves * (nt > 96 ? 75 : 50);
    if (best < 0 || c < cost) { best = nt; cost = c; }
  }
  return best;
}

// Bytes of the packed weights and bias, or -1 when the shape is outside the kernel's domain (kt <= 4).
TT_API long long tt_conv_packed_bytes(int kind, int kt, int chunks, int N) {
  if (kind < 0 || kind > 2 || kt < 1 || kt > 4 || chunks < 2 || chunks % 2 || N < 16 || N % 16) return -1;
  return (long long)(kind == 2 ? 9 : (kind == 0 ? 9 : 1) * kt) * chunks * N * 16 + (long long)N * 4;
}

TT_API int tt_conv_pack(const void* w, const void* bias, int f32, int kind, int kt, int C_real, int N_real, int chunks,
                        int N, int nt, void* dst, cudaStream_t stream) {
  ConvShape s;
  TT_CHECK(tt_conv_packed_bytes(kind, kt, chunks, N) > 0 && !conv_shape(chunks, N, nt, &s), "conv_pack: bad shape");
  TT_CHECK(N_real <= N && C_real <= chunks * (f32 ? 4 : 8) && ((uintptr_t)dst & 15) == 0, "conv_pack: bad arguments");
  ConvGroup g[4];
  PackParams p;
  memset(&p, 0, sizeof(p));
  p.n_groups = conv_groups(kind, kt, chunks, 0, g, p.tap_id);
  p.N_real = N_real; p.C_real = C_real; p.NT = s.NT; p.KC = s.KC; p.n_cb = s.n_cb; p.n_tiles = s.n_tiles;
  for (int i = 0; i < p.n_groups; ++i) { p.n_taps[i] = g[i].n_taps; p.taps_total += g[i].n_taps; }
  const long long per_tile = (long long)p.taps_total * chunks, total = per_tile * N;
  const unsigned grid = (unsigned)((total + 255) / 256);
  if (f32) conv_pack_kernel<true><<<grid, 256, 0, stream>>>(w, bias, dst, p, per_tile);
  else conv_pack_kernel<false><<<grid, 256, 0, stream>>>(w, bias, dst, p, per_tile);
  TT_LAUNCH_CHECK();
  return 0;
}

// x: [T_in][x_chunks][H_in][W_in][E] (kind 2: x_chunks = 4 * chunks pixel phases).  Output frame t reads input frames
// t * t_stride + t_off + (0 .. kt - 1); frames below zero are zeros.  Output pixels H x W.
TT_API int tt_conv(const void* x, int f32, int kind, int kt, int T_in, int H_in, int W_in, int chunks, const void* packed,
                   int N, int nt, void* out, const void* res, int T, int H, int W, int t_stride, int t_off,
                   int C_out, int t_mul, int planar, int C_real, unsigned* status, cudaStream_t stream) {
  ConvShape s;
  TT_CHECK(kind >= 0 && kind <= 2 && kt >= 1 && kt <= 4 && (kind != 2 || kt == 1) && !conv_shape(chunks, N, nt, &s),
           "conv: bad shape kind=%d kt=%d chunks=%d N=%d", kind, kt, chunks, N);
  TT_CHECK(T > 0 && H > 0 && W > 0 && T_in > 0 && H_in > 0 && W_in > 0, "conv: empty input or output");
  TT_CHECK((long long)(T - 1) * t_stride + kt - 1 + t_off < T_in && kt - 1 + t_off >= 0, "conv: frames out of range");
  TT_CHECK((((uintptr_t)x | (uintptr_t)packed | (uintptr_t)out | (uintptr_t)res) & 15) == 0,
           "conv: operands must be 16-byte aligned");
  TT_CHECK(planar || (C_out > 0 && C_out % 16 == 0 && N % C_out == 0), "conv: bad output channel split");
  const int E = f32 ? 4 : 8;
  ConvParams p;
  memset(&p, 0, sizeof(p));
  const int halo = kind == 0 ? 2 : kind == 2 ? 1 : 0;
  p.box_w = CV_TW + halo;
  const int box_h = CV_TH + halo;
  p.plane = p.box_w * box_h * 16;
  p.pad = kind == 0 ? 1 : 0;
  int tap_id[4][9];
  p.n_groups = conv_groups(kind, kt, chunks, p.box_w, p.g, tap_id);
  p.NT = s.NT; p.KC = s.KC; p.UC = s.UC; p.n_cb = s.n_cb; p.n_tiles = s.n_tiles;
  p.a_bytes = p.plane * s.KC;
  p.a_slot = (p.a_bytes + 127) / 128 * 128;
  p.b_bytes = s.NT * s.UC * 16;
  p.a_stages = CV_A_BYTES / p.a_slot < CV_MAX_A ? CV_A_BYTES / p.a_slot : CV_MAX_A;
  p.b_stages = CV_B_BYTES / p.b_bytes < CV_MAX_B ? CV_B_BYTES / p.b_bytes : CV_MAX_B;
  TT_CHECK(p.a_stages >= 2 && p.b_stages >= 2, "conv: box does not fit");
  p.tiles_w = (W + CV_TW - 1) / CV_TW;
  p.tiles_h = (H + CV_TH - 1) / CV_TH;
  const long long tiles = (long long)p.tiles_w * p.tiles_h * T * s.n_tiles;
  TT_CHECK(tiles < (1ll << 30), "conv: too many tiles");
  p.num_tiles = (int)tiles;
  p.T = T; p.H = H; p.W = W;
  p.t_stride = t_stride; p.t_off = t_off;
  int taps = 0;
  for (int i = 0; i < p.n_groups; ++i) taps += p.g[i].n_taps;
  p.B = (const uint8_t*)packed;
  p.b_tile_bytes = (long long)taps * chunks * s.NT * 16;
  p.bias = reinterpret_cast<const float*>(p.B + p.b_tile_bytes * s.n_tiles);
  p.out = out; p.res = res;
  p.C_out = C_out; p.t_mul = t_mul; p.planar = planar; p.C_real = C_real; p.status = status;
  CUtensorMap tm;
  const int xc = kind == 2 ? 4 * chunks : chunks;
  uint64_t dims[4] = {(uint64_t)W_in * E, (uint64_t)H_in, (uint64_t)xc, (uint64_t)T_in};
  uint64_t str[3] = {(uint64_t)W_in * 16, (uint64_t)H_in * W_in * 16, (uint64_t)xc * H_in * W_in * 16};
  uint32_t box[4] = {(uint32_t)(p.box_w * E), (uint32_t)box_h, (uint32_t)s.KC, 1};
  if (tt_make_tmap(&tm, x, f32 ? 4 : 2, 4, dims, str, box, 0)) return -1;
  int dev = 0, sms = 0;
  TT_CUDA(cudaGetDevice(&dev));
  TT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid = p.num_tiles < sms ? p.num_tiles : sms;
  auto kern = f32 ? conv_kernel<true> : conv_kernel<false>;
  TT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CV_SMEM));
  kern<<<grid, CV_THREADS, CV_SMEM, stream>>>(tm, p);
  TT_LAUNCH_CHECK();
  return 0;
}

// gamma: [C] in the type of x
TT_API int tt_chan_norm(const void* x, void* y, const void* gamma, int f32, int frames, int chunks, long long hw,
                        int act, cudaStream_t stream) {
  TT_CHECK(frames > 0 && frames < 65536 && hw > 0 && chunks > 0 && chunks <= 96, "chan_norm: bad shape");
  TT_CHECK((((uintptr_t)x | (uintptr_t)y | (uintptr_t)gamma) & 15) == 0, "chan_norm: misaligned");
  const dim3 grid((unsigned)((hw + 63) / 64), frames);
  const float scale = sqrtf((float)(chunks * (f32 ? 4 : 8)));
#define TT_NORM(F, N) chan_norm_kernel<F, N><<<grid, 256, 0, stream>>>((const uint4*)x, (uint4*)y, gamma, hw, chunks, scale, act)
#define TT_NORM_N(N) (f32 ? TT_NORM(true, N) : TT_NORM(false, N))
  const int n = (chunks + 3) / 4;
  if (n <= 3) TT_NORM_N(3);
  else if (n <= 6) TT_NORM_N(6);
  else if (n <= 12) TT_NORM_N(12);
  else TT_NORM_N(24);
#undef TT_NORM_N
#undef TT_NORM
  TT_LAUNCH_CHECK();
  return 0;
}

TT_API int tt_blk_from_planar(const void* src, void* dst, int f32, int C, int chunks, int T, int H, int W, long long sc,
                              long long st, long long sh, long long sw, int round, cudaStream_t stream) {
  TT_CHECK(T > 0 && H > 0 && W > 0 && C <= chunks * (f32 ? 4 : 8) && ((uintptr_t)dst & 15) == 0, "blk_from_planar: bad arguments");
  const long long n = (long long)T * chunks * H * W;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (f32) blk_from_planar_kernel<true><<<grid, 256, 0, stream>>>(src, (uint4*)dst, C, chunks, T, H, W, sc, st, sh, sw, round);
  else blk_from_planar_kernel<false><<<grid, 256, 0, stream>>>(src, (uint4*)dst, C, chunks, T, H, W, sc, st, sh, sw, round);
  TT_LAUNCH_CHECK();
  return 0;
}

TT_API int tt_blk_to_planar(const void* src, void* dst, int f32, int chunks, int T, long long hw, cudaStream_t stream) {
  TT_CHECK(T > 0 && hw > 0 && chunks > 0 && ((uintptr_t)src & 15) == 0, "blk_to_planar: bad arguments");
  const unsigned grid = (unsigned)(((long long)T * chunks * hw + 255) / 256);
  if (f32) blk_to_planar_kernel<true><<<grid, 256, 0, stream>>>((const uint4*)src, dst, chunks, T, hw);
  else blk_to_planar_kernel<false><<<grid, 256, 0, stream>>>((const uint4*)src, dst, chunks, T, hw);
  TT_LAUNCH_CHECK();
  return 0;
}

TT_API int tt_blk_move(const void* src, void* dst, int f32, int mode, int T, int n, int H, int W, cudaStream_t stream) {
  TT_CHECK(mode >= 0 && mode <= 2 && T > 0 && n > 0 && H > 0 && W > 0, "blk_move: bad arguments");
  TT_CHECK((((uintptr_t)src | (uintptr_t)dst) & 15) == 0, "blk_move: misaligned");
  const long long planes = (long long)T * n * (mode == 1 ? 4 : 1);
  const long long hwo = mode == 0 ? 4ll * H * W : mode == 1 ? (long long)((H + 1) / 2) * ((W + 1) / 2) : (long long)H * W;
  TT_CHECK(hwo < (1ll << 31), "blk_move: frame too large");
  const unsigned grid = (unsigned)((planes * hwo + 255) / 256);
  if (f32) blk_move_kernel<true><<<grid, 256, 0, stream>>>((const uint4*)src, (uint4*)dst, mode, planes, n, H, W);
  else blk_move_kernel<false><<<grid, 256, 0, stream>>>((const uint4*)src, (uint4*)dst, mode, planes, n, H, W);
  TT_LAUNCH_CHECK();
  return 0;
}
