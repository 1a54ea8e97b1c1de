// BF16 / FP16 GEMM for sm_100a: the C ABI entry points over the kernel in gemm_core.cuh.
//
// Tensor-core bound: 2*M*N*K flops per launch.
#include "gemm_core.cuh"

extern "C" int wk_gemm_16bit(const wk_gemm16_args* g, void* stream) {
  using namespace wk;
  if (!g) return WK_E_ARG;
  const int m = g->m, n = g->n, k = g->k;
  if (m < 0 || n < 0 || k < 0 || m % 128 || n % 128 || k % 64) return WK_E_ARG;
  if (m == 0 || n == 0) return 0;
  if (k == 0) return WK_E_ARG;
  if (!g->a || !g->b || !g->out || !aligned16(g->a) || !aligned16(g->b) || !aligned16(g->out)) return WK_E_ARG;
  if (g->act < 0 || g->act > 2 || (g->act == ACT_DGELU && !g->pre_in)) return WK_E_ARG;
  if ((g->pre_out && !aligned16(g->pre_out)) || (g->pre_in && !aligned16(g->pre_in))) return WK_E_ARG;
  if (g->scale_b && g->scale_b_cols && !aligned16(g->scale_b)) return WK_E_ARG;
  if ((g->q_mx != nullptr) != (g->s_mx != nullptr) || (g->q_mx && !aligned16(g->q_mx))) return WK_E_ARG;
  if (g->cta_pair < 0 || g->cta_pair > 2 || g->group_m < 0) return WK_E_ARG;
  if (int unsupported = require_sm100()) return unsupported;
  GemmParams p = {};
  p.status = status_word();
  if (!p.status) return WK_E_CUDA;
  Epilogue& e = p.epi;
  e.scale_a = g->scale_a;
  e.scale_b = g->scale_b;
  e.scale_a_rows = g->scale_a_rows;
  e.scale_b_cols = g->scale_b_cols;
  e.accum = g->accum;
  e.act = g->act;
  e.out_f16 = g->f16;
  e.pre_out = g->pre_out;
  e.pre_in = g->pre_in;
  e.q_mx = static_cast<uint8_t*>(g->q_mx);
  e.s_mx = static_cast<uint8_t*>(g->s_mx);
  p.out = g->out;
  p.M = m;
  p.N = n;
  p.group_m = g->group_m ? g->group_m : 8;
  p.in_f16 = g->f16;
  p.a_trans = g->a_trans;
  p.b_trans = g->b_trans;
  return launch_gemm<KIND_16>(g->a, g->b, nullptr, nullptr, k, g->cta_pair, p, static_cast<cudaStream_t>(stream));
}

extern "C" int wk_gemm_bf16(const void* a, const void* b, void* out, int m, int n, int k, void* stream) {
  wk_gemm16_args g = {};
  g.a = a;
  g.b = b;
  g.out = out;
  g.m = m;
  g.n = n;
  g.k = k;
  return wk_gemm_16bit(&g, stream);
}
