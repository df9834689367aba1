// The layers of a prompt step, launched from native code.
//
// A prompt step of a model of pre-norm blocks (RMSNorm, grouped-query attention, gated feed-forward, no biases, bfloat16)
// launches eight kernels a layer.  From Python each launch costs 10 to 14 us, so that steps of up to some 300 tokens were
// as long as their 140 launches took.  Here the same launchers are called one after another through their addresses, with
// the same arguments; the products of more than 64 rows are the same calls of the library's GEMM as before, on the handle
// that torch keeps for the current stream.  Llama 1B sizes: four prompts of 150 to 260 tokens in portions beside single
// tokens 22.4 -> 16.1 ms; one of 333 tokens 1.99 -> 1.93 (1.8 of them the GPU's), the first of a new length 2.56 -> 2.00.
//
// Host code only: no kernels, no CUDA headers; the caller passes the addresses of the launchers.
#include <stddef.h>
#include <stdint.h>

extern "C" {

// y [T, N] = x [T, K] w [N, K]^T
typedef int (*GemmExFn)(void*, int, int, int, int, int, const void*, const void*, int, int, const void*, int, int, const void*,
                        void*, int, int, int, int);
typedef int (*SetMathModeFn)(void*, int);
typedef int (*AddRmsNormFn)(float*, const void*, int, const void*, int, void*, int, const int32_t*, int, int, float, void*);
typedef int (*RopeFn)(void*, int, const int32_t*, const int32_t*, const float*, const float*, void*, void*, int, int, int, int,
                      int, int, long long, int*, void*);
typedef int (*AttnDecodeFn)(int, const void*, int, const void*, const void*, const int32_t*, int, const int32_t*, float*, float*,
                            int, int*, void*, int, int, int, int, int, int, float, int, void*);
typedef int (*AttnPrefillFn)(int, const void*, int, const void*, const void*, const int32_t*, int, const int32_t*,
                             const int32_t*, const int32_t*, const int32_t*, void*, int, int, int, int, int, int, float, int,
                             int*, void*);
typedef int (*GemmTcFn)(const void*, int, const void*, void*, int, int, int, int, int, int*, int, int, void*);
typedef int (*GemmMidFn)(const void*, int, const void*, void*, int, int, int, int, int, float*, int, const void*, int, void*,
                         int, float*, int, const float*, int, int, float, int*, void*);
typedef int (*SwigluFn)(const void*, void*, int, int, int, void*);

struct RlPromptLayer {
  const void *w_qkv, *w_o, *w_gate_up, *w_down, *norm_mixer, *norm_ffn;
  void *kcache, *vcache;
  int* counters;
};

// What stays the same from step to step.
struct RlPromptPlan {
  GemmExFn gemm_ex;
  SetMathModeFn set_math_mode;
  AddRmsNormFn add_rmsnorm;
  RopeFn rope;
  AttnDecodeFn attn_decode;
  AttnPrefillFn attn_prefill;
  GemmTcFn gemm_tc;
  GemmMidFn gemm_mid;
  SwigluFn swiglu;
  const RlPromptLayer* layers;
  float* residual;                       // [max tokens, H]
  void *normed, *qkv, *attn, *mixer_out, *act, *gate_up, *ffn_out;
  void *hand_xw_a, *hand_xw_b;           // [128, H] (17 to 64 rows: a norm handed from product to product)
  float *hand_sums_a, *hand_sums_b;      // [128, hand_tiles]
  float *part_o, *part_ml;
  const float *cos, *sin;
  int *status, *tc_status;
  long long num_slots;
  float eps, scale;
  int32_t num_layers, H, I, hq, hkv, D, page_size, window, max_pos, sm_count, tc_min_rows, hand_tiles;
};

struct RlPromptStep {
  void *blas, *stream;
  const int32_t *positions, *slots, *block_table, *decode_info, *tile_seq, *tile_tok, *tile_rows;
  int32_t T, max_blocks, num_decode, decode_parts, num_tiles, decode_impl;
};

// The launchers, in the plan's order.
enum { kGemmEx, kSetMathMode, kAddRmsNorm, kRope, kAttnDecode, kAttnPrefill, kGemmTc, kGemmMid, kSwiglu };

// What has come of a step: the package's kernels launched, and the launcher that failed.
struct RlPromptCounts {
  int32_t launches, failed;
};

// Launches, or leaves the function with the launcher's error.
#define RL_TRY(launcher, call)      \
  do {                              \
    if (const int error = (call)) { \
      n->failed = launcher;         \
      return error;                 \
    }                               \
  } while (0)

static const int kBf16 = 1;

static int library_product(const RlPromptPlan* p, const RlPromptStep* s, const void* x, const void* w, void* y, int N, int K) {
  const float one = 1.f, zero = 0.f;
  const int r16 = 14, compute32 = 68, algo = 99;         // CUDA_R_16BF, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP
  return p->gemm_ex(s->blas, 1, 0, N, s->T, K, &one, w, r16, K, x, r16, K, &zero, y, r16, N, compute32, algo);
}

// Rotation, cache write and attention on the projected rows.
static int attend(const RlPromptPlan* p, const RlPromptStep* s, const RlPromptLayer& l, RlPromptCounts* n) {
  const int ld = (p->hq + 2 * p->hkv) * p->D, out_ld = p->hq * p->D;
  RL_TRY(kRope, p->rope(p->qkv, kBf16, s->positions, s->slots, p->cos, p->sin, l.kcache, l.vcache, s->T, p->hq, p->hkv, p->D,
                        p->page_size, p->max_pos, p->num_slots, p->status, s->stream));
  ++n->launches;
  if (s->num_decode > 0) {
    RL_TRY(kAttnDecode, p->attn_decode(kBf16, p->qkv, ld, l.kcache, l.vcache, s->block_table, s->max_blocks, s->decode_info,
                                       p->part_o, p->part_ml, s->decode_parts, l.counters, p->attn, out_ld, s->num_decode, p->hq,
                                       p->hkv, p->page_size, p->window, p->scale, s->decode_impl, s->stream));
    n->launches += 2;                                   // (the kernel and its merge, as the parts count them)
  }
  if (s->num_tiles > 0) {
    RL_TRY(kAttnPrefill, p->attn_prefill(kBf16, p->qkv, ld, l.kcache, l.vcache, s->block_table, s->max_blocks, s->tile_seq,
                                         s->tile_tok, s->tile_rows, s->positions, p->attn, out_ld, s->num_tiles, p->hq, p->hkv,
                                         p->page_size, p->window, p->scale, 0, p->tc_status, s->stream));
    ++n->launches;
  }
  return 0;
}

// More than 64 rows: the library's products; the last layer's output is left in ffn_out, not yet added to the stream.
static int many_rows(const RlPromptPlan* p, const RlPromptStep* s, RlPromptCounts* n) {
  const int q = p->hq * p->D, qkv = q + 2 * p->hkv * p->D, T = s->T;
  const void* pending = nullptr;
  for (int i = 0; i < p->num_layers; ++i) {
    const RlPromptLayer& l = p->layers[i];
    RL_TRY(kAddRmsNorm, p->add_rmsnorm(p->residual, pending, kBf16, l.norm_mixer, kBf16, p->normed, kBf16, nullptr, T, p->H, p->eps,
                                       s->stream));
    RL_TRY(kGemmEx, library_product(p, s, p->normed, l.w_qkv, p->qkv, qkv, p->H));
    if (const int e = attend(p, s, l, n)) return e;
    RL_TRY(kGemmEx, library_product(p, s, p->attn, l.w_o, p->mixer_out, p->H, q));
    RL_TRY(kAddRmsNorm, p->add_rmsnorm(p->residual, p->mixer_out, kBf16, l.norm_ffn, kBf16, p->normed, kBf16, nullptr, T, p->H,
                                       p->eps, s->stream));
    if (T >= p->tc_min_rows) {
      RL_TRY(kGemmTc, p->gemm_tc(p->normed, p->H, l.w_gate_up, p->act, p->I, 3, T, p->I, p->H, p->tc_status, p->sm_count, 0,
                                 s->stream));
    } else {
      RL_TRY(kGemmEx, library_product(p, s, p->normed, l.w_gate_up, p->gate_up, 2 * p->I, p->H));
      RL_TRY(kSwiglu, p->swiglu(p->gate_up, p->act, kBf16, T, p->I, s->stream));
    }
    RL_TRY(kGemmEx, library_product(p, s, p->act, l.w_down, p->ffn_out, p->H, p->I));
    n->launches += 3;
    pending = p->ffn_out;
  }
  return 0;
}

// 17 to 64 rows: tcgen05 products that add to the stream and hand the norms on; nothing is left to add.
static int few_rows(const RlPromptPlan* p, const RlPromptStep* s, RlPromptCounts* n) {
  const int q = p->hq * p->D, qkv = q + 2 * p->hkv * p->D, T = s->T, H = p->H, tiles = p->hand_tiles;
  RL_TRY(kAddRmsNorm, p->add_rmsnorm(p->residual, nullptr, kBf16, p->layers[0].norm_mixer, kBf16, p->normed, kBf16, nullptr, T, H,
                                     p->eps, s->stream));
  ++n->launches;
  for (int i = 0; i < p->num_layers; ++i) {
    const RlPromptLayer& l = p->layers[i];
    const void* x = i ? p->hand_xw_b : p->normed;
    const float* sums = i ? p->hand_sums_b : nullptr;
    RL_TRY(kGemmMid, p->gemm_mid(x, H, l.w_qkv, p->qkv, qkv, 0, T, qkv, H, nullptr, 0, nullptr, 0, nullptr, 0, nullptr, 0, sums,
                                 sums ? tiles : 0, sums ? tiles : 0, p->eps, p->tc_status, s->stream));
    if (const int e = attend(p, s, l, n)) return e;
    RL_TRY(kGemmMid, p->gemm_mid(p->attn, q, l.w_o, nullptr, 0, 2, T, H, q, p->residual, H, l.norm_ffn, 0, p->hand_xw_a, H,
                                 p->hand_sums_a, tiles, nullptr, 0, 0, 0.f, p->tc_status, s->stream));
    RL_TRY(kGemmMid, p->gemm_mid(p->hand_xw_a, H, l.w_gate_up, p->act, p->I, 3, T, p->I, H, nullptr, 0, nullptr, 0, nullptr, 0,
                                 nullptr, 0, p->hand_sums_a, tiles, tiles, p->eps, p->tc_status, s->stream));
    const bool more = i + 1 < p->num_layers;
    RL_TRY(kGemmMid, p->gemm_mid(p->act, p->I, l.w_down, nullptr, 0, 2, T, H, p->I, p->residual, H,
                                 more ? p->layers[i + 1].norm_mixer : nullptr, 0, more ? p->hand_xw_b : nullptr, more ? H : 0,
                                 more ? p->hand_sums_b : nullptr, more ? tiles : 0, nullptr, 0, 0, 0.f, p->tc_status, s->stream));
    n->launches += 4;
  }
  return 0;
}

// Launches all layers of the step.  Returns 0 or the error of the launcher n->failed (the first two: the library's status, the
// others: a CUDA error).
int rl_prompt_layers(const RlPromptPlan* p, const RlPromptStep* s, int few, RlPromptCounts* n) {
  n->launches = 0;
  if (few) return few_rows(p, s, n);
  const int keep_float32 = 16, default_math = 0;        // no reduced-precision sums of a split k (CUBLAS_MATH_DISALLOW_...)
  RL_TRY(kSetMathMode, p->set_math_mode(s->blas, keep_float32));
  const int e = many_rows(p, s, n), back = p->set_math_mode(s->blas, default_math);
  if (e) return e;
  RL_TRY(kSetMathMode, back);
  return 0;
}

}  // extern "C"
