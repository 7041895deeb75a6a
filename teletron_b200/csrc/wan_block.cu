// K-WAN-BLOCK: the launches of one Wan DiT block without gradients (sampling, validation) as one native call.
//
// A block is sixteen kernels of a few microseconds at a small latent (256 tokens x 1536 channels), and issuing them one
// by one through the Python op layer costs the host more than the GPU needs to run them (41 ms of host time against
// 19 ms of kernels for the two passes of a 256-token sampling step).  Here Python hands over the addresses once per
// block and the launches follow each other from C++.  The kernels, their order and their arithmetic are those of the op
// layer; only the small fp32 conversions in front of them (modulation + timestep embedding, norm weights) are gathered
// into one kernel.
#include "tt_common.cuh"

using namespace tt;

TT_API int tt_adaln_fwd(const void* x, long long ldx, void* y, long long ldy, const float* mul, const float* add,
                        long long mod_ld, int plus_one, int rows, int C, int rows_per_batch, float eps, float* mean_out,
                        float* rstd_out, cudaStream_t stream);
TT_API int tt_rmsrope_fwd(const void* x, long long ldx, void* y, long long ldy, const float* w, const void* freqs,
                          int freq_rows, float* rstd, int rows, int C, int D, int per_head, float eps, cudaStream_t stream);
TT_API int tt_gemm_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* C,
                        long long ldc, int c_fp32, int M, int N, int K, const void* bias, int epi, const void* residual,
                        long long ldr, const float* gate, long long gate_ld, int rows_per_gate, void* aux_out, float alpha,
                        unsigned* status, int max_ctas, cudaStream_t stream);
TT_API int tt_gemm2_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* C,
                         long long ldc, int c_fp32, int M, int N, int K, const void* bias, int epi, const void* residual,
                         long long ldr, const float* gate, long long gate_ld, int rows_per_gate, void* aux_out, float alpha,
                         unsigned* status, cudaStream_t stream);
TT_API int tt_attn_fwd(const void* q, long long ldq, long long q_bs, const void* k, long long ldk, long long k_bs,
                       const void* v, long long ldv, long long v_bs, void* o, long long ldo, long long o_bs, float* lse,
                       const int* kv_lens, int B, int H, int Sq, int Skv, int D, float scale, unsigned* status,
                       cudaStream_t stream);

namespace {

// order of the parameter addresses; a weight is followed by its bias
enum Par : int { P_MOD, P_QKV_W, P_QKV_B, P_NQ, P_NK, P_O_W, P_O_B, P_N3_W, P_N3_B, P_CQ_W, P_CQ_B, P_KV_W, P_KV_B, P_CNQ,
                 P_CNK, P_CO_W, P_CO_B, P_F1_W, P_F1_B, P_F2_W, P_F2_B };

// small fp32 operands of the block: e [B][6][C] = modulation + t_mod, then six rows [C] of norm weights
struct PrepParams {
  const bf16* mod;
  const float* t_mod;
  const bf16* rows[6];
  float* out;
  int B, C;
};
__global__ void __launch_bounds__(256) wan_prep_kernel(const PrepParams p) {
  const int row = blockIdx.y, c = blockIdx.x * 256 + threadIdx.x;
  chain_release();
  chain_wait();
  if (c >= p.C) return;
  float v;
  if (row < 6 * p.B) v = __bfloat162float(p.mod[(row % 6) * p.C + c]) + p.t_mod[(long long)row * p.C + c];
  else v = __bfloat162float(p.rows[row - 6 * p.B][c]);
  p.out[(long long)row * p.C + c] = v;
}

struct Carver {
  uint8_t* base;
  long long off;
  void* take(long long bytes) {
    void* p = base ? base + off : nullptr;
    off += (bytes + 255) / 256 * 256;
    return p;
  }
};
struct Work {
  float *small, *lse;
  bf16 *h, *qkv, *q, *k, *a, *x1, *x2, *kv, *mid;
  long long bytes;
};
Work carve(uint8_t* base, int B, int S, int Lc, int C, int H, int F) {
  Carver c{base, 0};
  const long long R = (long long)B * S, Rc = (long long)B * Lc, Rk = R > Rc ? R : Rc;
  Work w;
  w.small = (float*)c.take((6ll * B + 6) * C * 4);
  w.lse = (float*)c.take((long long)B * H * S * 4);
  w.h = (bf16*)c.take(R * C * 2);
  w.q = (bf16*)c.take(R * C * 2);
  w.k = (bf16*)c.take(Rk * C * 2);
  w.a = (bf16*)c.take(R * C * 2);
  w.x1 = (bf16*)c.take(R * C * 2);
  w.x2 = (bf16*)c.take(R * C * 2);
  // qkv and kv are dead when the feed-forward's hidden rows are written
  const long long attn = R * 3 * C * 2 + 256 + Rc * 2 * C * 2, mid = R * F * 2;
  uint8_t* shared = (uint8_t*)c.take(attn > mid ? attn : mid);
  w.qkv = (bf16*)shared;
  w.kv = (bf16*)(shared + (R * 3 * C * 2 + 255) / 256 * 256);
  w.mid = (bf16*)shared;
  w.bytes = c.off;
  return w;
}

}  // namespace

TT_API long long tt_wan_block_workspace(int B, int S, int Lc, int C, int H, int F) {
  return carve(nullptr, B, S, Lc, C, H, F).bytes;
}

// x, out: bf16 [B * S, C]; ctx: bf16 [B * Lc, C]; t_mod: fp32 [B][6][C]; freqs: fp32 [freq_rows, 64, 2]; params: device
// addresses in the order of `Par`, all bf16 and dense.  pair: large products may take the CTA-pair kernel.
TT_API int tt_wan_block_fwd(const void* x, long long ldx, void* out, const void* ctx, const float* t_mod, const void* freqs,
                            int freq_rows, const long long* params, int B, int S, int Lc, int C, int H, int F, float eps,
                            int pair, void* workspace, unsigned* status, cudaStream_t stream) {
  TT_CHECK(B > 0 && S > 0 && Lc > 0 && C > 0 && H > 0 && C == H * 128 && F > 0 && F % 8 == 0, "wan_block: bad shape");
  TT_CHECK(6ll * B + 6 < 65536 && (long long)B * S < (1ll << 31) && (long long)B * Lc < (1ll << 31), "wan_block: too many rows");
  const Work w = carve((uint8_t*)workspace, B, S, Lc, C, H, F);
  const int R = B * S, Rc = B * Lc, D = 128;
  const float scale = (float)(1.0 / sqrt((double)D));
  auto par = [&](int i) { return reinterpret_cast<const bf16*>(params[i]); };
  PrepParams pp;
  pp.mod = par(P_MOD); pp.t_mod = t_mod; pp.out = w.small; pp.B = B; pp.C = C;
  const int rows6[6] = {P_NQ, P_NK, P_N3_W, P_N3_B, P_CNQ, P_CNK};
  for (int i = 0; i < 6; ++i) pp.rows[i] = par(rows6[i]);
  // Start-ups overlapped with the launch before.  A forward pass of eight 1536-wide blocks, without -> with, ms:
  //   256 tokens 1.76 -> 1.59, 1,024 2.54 -> 2.39, 3,072 3.49 -> 3.34, 6,144 6.71 -> 6.39;
  //   8,192 9.93 -> 9.98, 12,288 16.30 -> 16.35, 16,384 25.39 -> 25.56, 24,576 44.80 -> 45.02
  // so the line lies where it stops paying.  5120-wide blocks: within noise on both sides of it (+-3 %).
  const TTChain chain(R < 8192);
  TT_CUDA(tt_launch(wan_prep_kernel, dim3((C + 255) / 256, 6 * B + 6), dim3(256), 0, stream, 1, pp));
  TT_LAUNCH_CHECK();
  auto ev = [&](int i) { return w.small + (long long)i * C; };         // row i of sample 0; samples are 6 * C apart
  auto sm = [&](int i) { return w.small + (6ll * B + i) * C; };
  const long long e_ld = 6ll * C;
  auto gemm = [&](const void* a, long long lda, int wi, void* c, int M, int N, int K, int epi, const void* res, long long ldr,
                  const float* gate, long long gate_ld, int rpg) -> int {
    if (pair && M >= 256 && N >= 256) {
      const int rc = tt_gemm2_bf16(a, lda, 0, par(wi), K, 0, c, N, 0, M, N, K, par(wi + 1), epi, res, ldr, gate, gate_ld, rpg,
                                   nullptr, 1.f, status, stream);
      if (rc != -3) return rc;
    }
    return tt_gemm_bf16(a, lda, 0, par(wi), K, 0, c, N, 0, M, N, K, par(wi + 1), epi, res, ldr, gate, gate_ld, rpg, nullptr,
                        1.f, status, 0, stream);
  };
  const int NONE = 0, GELU = 1, GATE_RES = 2;
  const long long sc = (long long)S * C, lc2 = 2ll * Lc * C;
#define TT_RUN(call)        \
  do {                      \
    const int rc_ = (call); \
    if (rc_) return rc_;    \
  } while (0)
  // self-attention
  TT_RUN(tt_adaln_fwd(x, ldx, w.h, C, ev(1), ev(0), e_ld, 1, R, C, S, eps, nullptr, nullptr, stream));
  TT_RUN(gemm(w.h, C, P_QKV_W, w.qkv, R, 3 * C, C, NONE, nullptr, 0, nullptr, 0, 1));
  TT_RUN(tt_rmsrope_fwd(w.qkv, 3 * C, w.q, C, sm(0), freqs, freq_rows, nullptr, R, C, D, 0, eps, stream));
  TT_RUN(tt_rmsrope_fwd(w.qkv + C, 3 * C, w.k, C, sm(1), freqs, freq_rows, nullptr, R, C, D, 0, eps, stream));
  TT_RUN(tt_attn_fwd(w.q, C, sc, w.k, C, sc, w.qkv + 2 * C, 3 * C, 3 * sc, w.a, C, sc, w.lse, nullptr, B, H, S, S, D, scale,
                     status, stream));
  TT_RUN(gemm(w.a, C, P_O_W, w.x1, R, C, C, GATE_RES, x, ldx, ev(2), e_ld, S));
  // cross-attention
  TT_RUN(tt_adaln_fwd(w.x1, C, w.h, C, sm(2), sm(3), C, 0, R, C, R, eps, nullptr, nullptr, stream));
  TT_RUN(gemm(w.h, C, P_CQ_W, w.qkv, R, C, C, NONE, nullptr, 0, nullptr, 0, 1));
  TT_RUN(tt_rmsrope_fwd(w.qkv, C, w.q, C, sm(4), nullptr, 1, nullptr, R, C, D, 0, eps, stream));
  TT_RUN(gemm(ctx, C, P_KV_W, w.kv, Rc, 2 * C, C, NONE, nullptr, 0, nullptr, 0, 1));
  TT_RUN(tt_rmsrope_fwd(w.kv, 2 * C, w.k, C, sm(5), nullptr, 1, nullptr, Rc, C, D, 0, eps, stream));
  TT_RUN(tt_attn_fwd(w.q, C, sc, w.k, C, (long long)Lc * C, w.kv + C, 2 * C, lc2, w.a, C, sc, w.lse, nullptr, B, H, S, Lc, D,
                     scale, status, stream));
  TT_RUN(gemm(w.a, C, P_CO_W, w.x2, R, C, C, GATE_RES, w.x1, C, nullptr, 0, R));
  // feed-forward
  TT_RUN(tt_adaln_fwd(w.x2, C, w.h, C, ev(4), ev(3), e_ld, 1, R, C, S, eps, nullptr, nullptr, stream));
  TT_RUN(gemm(w.h, C, P_F1_W, w.mid, R, F, C, GELU, nullptr, 0, nullptr, 0, 1));
  TT_RUN(gemm(w.mid, F, P_F2_W, out, R, C, F, GATE_RES, w.x2, C, ev(5), e_ld, S));
#undef TT_RUN
  return 0;
}
