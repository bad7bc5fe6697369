// The layers of a prompt step, launched from here: attention with a rotary encoding and a gated feed-forward between norms
// before and after (bfloat16), one run after the other.  No kernel of its own: the entry points that the parts call one
// by one, in the same order, with the same arguments, so that the results are the same bits.  What it saves is the host's
// time: from Python a launch and what stands around it take 17 us, more than most kernels of a short prompt; from here 4.
#include "common.cuh"

extern "C" {
int af_gemm_tc(void* out, int out_dtype, long long ldo, long long part_stride, const void* x, long long ldx, const void* w,
               long long ldw, long long n_w_rows, int M, int K, int gated, int act, int n_acc, float cap, int splits, int per_sm,
               int token_tile, int* err, cudaStream_t stream);
int af_rope_cache_write(void* qkv, int dtype, int row_stride, const float* parts, int n_parts, long long part_stride,
                        const int* positions, const int* seq_of_token, const int* slots, const int* len_after,
                        const float* inv_freq, const float* table, int n_tokens, int nq, int nkv, int hd, int rot_dim,
                        int pairing, void* kcache, void* vcache, const int* page_table, int max_pages, int ring_rows, int keep,
                        cudaStream_t stream);
int af_attn_prefill_tc(void* out, long long out_stride, const void* q, long long q_stride, const void* k, long long k_stride,
                       const void* v, long long v_stride, const int* seq_starts, int n_seqs, int n_tokens, int max_len, int nq,
                       int nkv, int hd, float scale, float cap, int window, int keep, const float* sinks, const float* gate,
                       long long gate_stride, int* err, cudaStream_t stream);
int af_add_rmsnorm(float* x, const void* a, int a_dtype, int n_parts, long long part_stride, const float* w_post, void* y,
                   int y_dtype, const float* w_next, int n_rows, int hidden, float eps_post, float eps_next, float offset,
                   cudaStream_t stream);
}

namespace {

// What a run has of its own, as the caller packs it.
struct PromptRun {
  const void *w_qkv, *w_o, *w_gu, *w_down;
  const float *n_post_mixer, *n_pre_ff, *n_post_ff, *n_next;      // n_next null: no run follows
  const float *inv_freq, *table;
  void *kcache, *vcache;
  const int* page_table;
  long long max_pages, ring_rows, window, keep;
  double eps_post_mixer, eps_pre_ff, eps_post_ff, eps_next, scale, cap;
};

// What all runs share.
struct PromptStep {
  float* x;                 // [T, H] the stream
  __nv_bfloat16 *h, *qkv, *ctx, *mid, *a;       // rows of H (holding the first run's input), (nq + 2 nkv) hd, nq hd, inter, H
  float* parts;             // split-K partial sums of one product
  const int *positions, *seq_of_token, *slots, *len_after, *seq_starts;
  int* err;
  long long T, H, nq, nkv, hd, rot_dim, pairing, inter, act, n_seqs, max_len;
  long long splits[3];              // of the products q k v, o, down
  double offset;
};

// One product into `out`, or into partial sums.
int prompt_product(const PromptStep& s, void* out, const void* x, const void* w, long long rows, int K, int splits, bool gated,
                   cudaStream_t stream) {
  const int M = (int)s.T, per_sm = 0;
  const long long N = gated ? rows / 2 : rows;
  if (splits > 1)
    return af_gemm_tc(s.parts, AF_F32, N, (long long)M * N, x, K, w, K, rows, M, K, 0, 0, 0, 0.f, splits, per_sm, 0, s.err, stream);
  return af_gemm_tc(out, AF_BF16, N, 0, x, K, w, K, rows, M, K, gated ? 1 : 0, (int)s.act, 0, 0.f, 1, per_sm, 0, s.err, stream);
}

}  // namespace

AF_EXPORT int af_prompt_layers_sizes(int which) { return which == 0 ? (int)sizeof(PromptRun) : (int)sizeof(PromptStep); }

AF_EXPORT int af_prompt_layers(const void* step, const void* runs, int n_runs, cudaStream_t stream) {
  const PromptStep& s = *static_cast<const PromptStep*>(step);
  const PromptRun* all = static_cast<const PromptRun*>(runs);
  AF_REQUIRE(s.T > 0 && s.T <= 0x7fffffff && s.nkv > 0 && s.nq % s.nkv == 0, "af_prompt_layers: bad sizes");
  const int T = (int)s.T, H = (int)s.H, nq = (int)s.nq, nkv = (int)s.nkv, hd = (int)s.hd, inter = (int)s.inter;
  const int W = (nq + 2 * nkv) * hd;
  const float offset = (float)s.offset;
  for (int i = 0; i < n_runs; ++i) {
    const PromptRun& r = all[i];
    int e = prompt_product(s, s.qkv, s.h, r.w_qkv, W, H, (int)s.splits[0], false, stream);
    if (e) return e;
    const bool joined = s.splits[0] > 1;
    e = af_rope_cache_write(s.qkv, AF_BF16, W, joined ? s.parts : nullptr, joined ? (int)s.splits[0] : 0,
                            joined ? (long long)T * W : 0, s.positions, s.seq_of_token, s.slots, s.len_after, r.inv_freq,
                            joined ? nullptr : r.table, T, nq, nkv, hd, (int)s.rot_dim, (int)s.pairing, r.kcache, r.vcache,
                            r.page_table, (int)r.max_pages, (int)r.ring_rows, (int)r.keep, stream);
    if (e) return e;
    e = af_attn_prefill_tc(s.ctx, (long long)nq * hd, s.qkv, W, s.qkv + nq * hd, W, s.qkv + (nq + nkv) * hd, W, s.seq_starts,
                           (int)s.n_seqs, T, (int)s.max_len, nq, nkv, hd, (float)r.scale, (float)r.cap, (int)r.window,
                           r.window ? (int)r.keep : 0, nullptr, nullptr, 0, s.err, stream);
    if (e) return e;
    e = prompt_product(s, s.a, s.ctx, r.w_o, H, nq * hd, (int)s.splits[1], false, stream);
    if (e) return e;
    auto add = [&](long long splits, const float* post, double eps_post, const float* next, double eps_next) {
      const bool sums = splits > 1;
      return af_add_rmsnorm(s.x, sums ? (const void*)s.parts : s.a, sums ? AF_F32 : AF_BF16, sums ? (int)splits : 1,
                            (long long)T * H, post, next ? s.h : nullptr, next ? AF_BF16 : AF_F32, next, T, H, (float)eps_post,
                            (float)eps_next, offset, stream);
    };
    e = add(s.splits[1], r.n_post_mixer, r.eps_post_mixer, r.n_pre_ff, r.eps_pre_ff);
    if (e) return e;
    e = prompt_product(s, s.mid, s.h, r.w_gu, 2ll * inter, H, 1, true, stream);
    if (e) return e;
    e = prompt_product(s, s.a, s.mid, r.w_down, H, inter, (int)s.splits[2], false, stream);
    if (e) return e;
    e = add(s.splits[2], r.n_post_ff, r.eps_post_ff, r.n_next, r.eps_next);
    if (e) return e;
  }
  return 0;
}
