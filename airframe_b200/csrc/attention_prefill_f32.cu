// Attention of prompts in 32 bits: every product and sum an fma in 32 bits, as in attention_plain.cu, but tiles of 16 queries of
// a head that share the keys and values they read.
//
// A warp that walks one query's keys (attention_plain.cu) reads every key and value row from L2 for that query alone and waits
// for the chain of loads, shuffles and exponentials behind every four keys.  Here a block of 16 warps holds 16 queries of a head in
// shared memory and walks the 64-key tiles they see:
//   scores   4 queries x 8 keys a thread, the head's elements dealt to 16 lanes whose sums meet by halving
//   softmax  a warp a query; maximum and sum are kept in 32 bits as in the other kernel
//   values   4 queries x dv / 32 columns a thread, a run of 16 keys four warps; the runs meet at the end
// The next tile's keys are copied (cp.async) under the softmax and the values' products, its values under the scores.
// Bound by latencies in the block with the most keys (eight warps with tiles of 8 x 8 issued an instruction every fifth cycle): 301 tokens, 8 heads of 256
// with 4 of keys: 73 -> 40 us.
//
// A query's result depends on its position in its sequence alone (tiles begin at multiples of 16 queries and of 64 keys of the
// sequence).  A key that a query does not see has no part in its sums at all (zero times an infinity would be NaN): tiles
// that not all four queries of a thread see whole go query by query.
#include "common.cuh"
#include "tma.cuh"

namespace {

constexpr int PT_Q = 16, PT_K = 64, PT_THREADS = 512;
constexpr int PT_SS = PT_K + 4;       // floats of a query's row of scores
constexpr int PT_PS = 36;             // floats of a key's row of weights: every weight twice, as the packed products take it

struct PtArgs {
  float* out;
  const float *q, *k, *v;
  long long out_stride, q_stride, k_stride, v_stride;
  const int* seq_starts;
  int n_seqs, least;                  // (shorter sequences are another kernel's)
  int nq, nkv, hd, dv;
  float scale, cap;
  int window, mask_kind, keep;
  const float *slopes, *sinks, *gate;
  long long gate_stride;
  int vec;                            // rows of whole 16-byte pieces
};

constexpr size_t pt_smem(int HD, int DV) {
  return (size_t)(PT_Q * HD + PT_K * HD + PT_K * DV + PT_Q * PT_SS + PT_K * PT_PS + 2 * PT_Q) * sizeof(float);
}

__device__ __forceinline__ void pt_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pt_both(float x) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
  return v;
}
__device__ __forceinline__ float2 pt_halves(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
// v[0 .. 2 N) summed over the lanes that differ in `bit`, which keep a half each: the upper one v[N ..].
template <int N>
__device__ __forceinline__ void pt_halve(float* v, int bit) {
  const bool up = threadIdx.x & bit;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float keep = up ? v[i + N] : v[i], give = up ? v[i] : v[i + N];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
  }
}
__device__ __forceinline__ int pt_first_visible(int pos, int size, int mask_kind) {
  if (size <= 0) return 0;
  return mask_kind == AF_MASK_CHUNK ? pos - pos % size : max(0, pos - size + 1);
}
__device__ __forceinline__ void pt_copy16(float* dst, const float* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void pt_copy4(float* dst, const float* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(on ? 4 : 0) : "memory");
}

// HD, DV: the head's and the values' sizes rounded up to 64, 128 or 256.
template <int HD, int DV>
__global__ void __launch_bounds__(PT_THREADS, 1)
attn_prefill_f32_kernel(PtArgs a) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float sm[];
  float *q_s = sm, *k_s = q_s + PT_Q * HD, *v_s = k_s + PT_K * HD, *s_s = v_s + PT_K * DV, *p_s = s_s + PT_Q * PT_SS,
        *corr_s = p_s + PT_K * PT_PS, *inv_s = corr_s + PT_Q;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, g = h / (a.nq / a.nkv);
  pdl_wait();
  a.q = pdl_fresh(a.q), a.k = pdl_fresh(a.k), a.v = pdl_fresh(a.v);
  // the block's sequence: tile blockIdx.x of those of all sequences of `least` tokens and more, one after the other.  (A block a tile of the
  // longest for every sequence left most of them without work, and each holds an SM: a sequence of 300 tokens among 100 of 3, 18 heads, a window of 64:
  // 100 us.)
  int first = 0, len = 0, tile = (int)blockIdx.x;
  for (int base = 0; base < a.n_seqs && len == 0; base += 32) {
    const int i = min(base + lane, a.n_seqs - 1), from = a.seq_starts[i], n = base + lane < a.n_seqs ? a.seq_starts[i + 1] - from : 0;
    const int mine = n >= a.least ? (n + PT_Q - 1) / PT_Q : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += up;
    }
    const unsigned behind = __ballot_sync(0xffffffffu, upto > tile);
    if (behind != 0) {
      const int of = __ffs(behind) - 1;
      first = __shfl_sync(0xffffffffu, from, of), len = __shfl_sync(0xffffffffu, n, of);
      tile -= __shfl_sync(0xffffffffu, upto - mine, of);
    } else {
      tile -= __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  if (len == 0) return;
  const int p0 = ((len + PT_Q - 1) / PT_Q - 1 - tile) * PT_Q, n_q = min(PT_Q, len - p0), last = p0 + n_q - 1;
  const int lo0 = pt_first_visible(p0, a.window, a.mask_kind);
  const float* kb = a.k + (size_t)first * a.k_stride + (size_t)g * a.hd;
  const float* vb = a.v + (size_t)first * a.v_stride + (size_t)g * a.dv;

  // `n` rows of `width` elements from row j0 on into rows of W; rows behind `end` are zeros
  auto load = [&](float* dst, int W, const float* src, long long stride, int width, int j0, int n, int end) {
    for (int r = warp; r < n; r += PT_THREADS / 32) {
      const bool on = j0 + r <= end;
      const float* row = src + (size_t)(on ? j0 + r : end) * stride;
      if (a.vec) {
        for (int c = lane * 4; c < width; c += 128) pt_copy16(dst + r * W + c, row + c, on);
      } else {
        for (int c = lane; c < width; c += 32) pt_copy4(dst + r * W + c, row + c, on);
      }
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  // the first tile from kt on that has a key in sight of some query
  auto next = [&](int kt) { return kt * PT_K >= a.keep ? max(kt, lo0 / PT_K) : kt; };

  // what lies behind the head's and the values' own sizes is never copied to: zeros
  if (a.hd < HD) {
    for (int i = tid; i < (PT_Q + PT_K) * HD; i += PT_THREADS) q_s[i] = 0.f;        // (queries and keys)
  }
  if (a.dv < DV) {
    for (int i = tid; i < PT_K * DV; i += PT_THREADS) v_s[i] = 0.f;
  }
  if (a.hd < HD || a.dv < DV) __syncthreads();
  int kt = next(0);
  load(q_s, HD, a.q + (size_t)first * a.q_stride + (size_t)h * a.hd, a.q_stride, a.hd, p0, PT_Q, last);
  load(k_s, HD, kb, a.k_stride, a.hd, kt * PT_K, PT_K, last);
  commit();
  load(v_s, DV, vb, a.v_stride, a.dv, kt * PT_K, PT_K, last);
  commit();

  // scores: 16 lanes a tile of 4 queries by 8 keys, lane `part` takes elements 4 part + 64 s
  const int part = tid & 15, tr = (tid >> 4 & 3) * 4, tk = (tid >> 6) * 8;
  // softmax: a warp a query, keys lane and lane + 32
  const int row = warp, pos = p0 + row;
  const int lo = pt_first_visible(pos, a.window, a.mask_kind);
  const float slope = a.slopes ? a.slopes[h] : 0.f;
  float m = a.sinks ? a.sinks[h] : -INFINITY;
  float l = lane == 0 && m > -INFINITY ? 1.f : 0.f;          // (this thread's part of the sum)
  // values: queries vr .. vr + 3, a run of 16 keys
  const int vr = (warp & 3) * 4, run = warp >> 2;
  constexpr int NP = DV / 64;                                // packed columns of a thread
  unsigned long long o[4][NP] = {};
  int lo_r[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) lo_r[r] = pt_first_visible(p0 + vr + r, a.window, a.mask_kind);
  // this thread's columns: DV 256 4 lane .. and 128 + 4 lane .., 128 4 lane .., 64 2 lane ..
  auto values = [&](int key, unsigned long long (&x)[NP]) {
    const float* src = v_s + key * DV;
    if constexpr (NP == 1) {
      x[0] = *reinterpret_cast<const unsigned long long*>(src + 2 * lane);
    } else {
#pragma unroll
      for (int e = 0; e < NP; e += 2) {
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(src + 64 * e + 4 * lane);
        x[e] = y.x, x[e + 1] = y.y;
      }
    }
  };

  while (kt * PT_K <= last) {
    const int nk = next(kt + 1);
    const bool more = nk * PT_K <= last;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                         // (the tile's keys are there)
    {
      unsigned long long acc[4][8] = {};
#pragma unroll 1
      for (int d = part * 4; d < HD; d += 64) {
        ulonglong2 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(q_s + (tr + i) * HD + d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(k_s + (tk + j) * HD + d);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            pt_fma2(acc[i][j], x[i].x, y.x);
            pt_fma2(acc[i][j], x[i].y, y.y);
          }
        }
      }
      float s[32];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 f = pt_halves(acc[i][j]);
          s[8 * i + j] = f.x + f.y;
        }
      pt_halve<16>(s, 8);
      pt_halve<8>(s, 4);
      pt_halve<4>(s, 2);
      pt_halve<2>(s, 1);                                     // lane `part` is left with values 2 part ..
      *reinterpret_cast<float2*>(s_s + (tr + (part >> 2)) * PT_SS + tk + (part & 3) * 2) = make_float2(s[0], s[1]);
    }
    __syncthreads();                                         // (scores are there, the keys are done with)
    if (more) load(k_s, HD, kb, a.k_stride, a.hd, nk * PT_K, PT_K, last);
    commit();
    {
      float s[2], top = m;
      bool sees[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = kt * PT_K + lane + 32 * e;
        sees[e] = j <= pos && (j >= lo || j < a.keep);
        s[e] = sees[e] ? softcap_f32(s_s[row * PT_SS + lane + 32 * e] * a.scale, a.cap) + slope * (float)(j - pos) : -INFINITY;
        top = fmaxf(top, s[e]);
      }
      top = warp_max(top);
      const float ref = top == -INFINITY ? 0.f : top;        // (no score above -inf yet: they weigh nothing)
      const float corr = expf(m - ref);
      m = top;
      l *= corr;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float w = sees[e] ? expf(s[e] - ref) : 0.f;
        l += w;
        *reinterpret_cast<float2*>(p_s + (lane + 32 * e) * PT_PS + 2 * row) = make_float2(w, w);
      }
      if (lane == 0) corr_s[row] = corr;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                         // (weights and values are there)
    {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const unsigned long long f = pt_both(corr_s[vr + r]);
#pragma unroll
        for (int e = 0; e < NP; ++e) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(o[r][e]) : "l"(f));
      }
      const int j0 = kt * PT_K + run * 16;
      const bool whole = j0 + 15 <= p0 + vr && (j0 >= lo_r[3] || j0 + 15 < a.keep);
      const float* w = p_s + run * 16 * PT_PS + 2 * vr;
      if (whole) {
#pragma unroll 2
        for (int n = 0; n < 16; ++n) {
          unsigned long long x[NP];
          values(run * 16 + n, x);
#pragma unroll
          for (int r = 0; r < 4; r += 2) {
            const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(w + n * PT_PS + 2 * r);
#pragma unroll
            for (int e = 0; e < NP; ++e) {
              pt_fma2(o[r][e], f.x, x[e]);
              pt_fma2(o[r + 1][e], f.y, x[e]);
            }
          }
        }
      } else {
#pragma unroll 1
        for (int n = 0; n < 16; ++n) {
          const int j = j0 + n;
          if (j > last) break;
          unsigned long long x[NP];
          values(run * 16 + n, x);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (j <= p0 + vr + r && (j >= lo_r[r] || j < a.keep)) {        // (the same for the whole warp)
              const unsigned long long f = *reinterpret_cast<const unsigned long long*>(w + n * PT_PS + 2 * r);
#pragma unroll
              for (int e = 0; e < NP; ++e) pt_fma2(o[r][e], f, x[e]);
            }
          }
        }
      }
    }
    __syncthreads();                                         // (weights and values are done with)
    if (more) load(v_s, DV, vb, a.v_stride, a.dv, nk * PT_K, PT_K, last);
    commit();
    kt = nk;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  l = warp_sum(l);
  if (lane == 0 && row < n_q) {
    const float factor = a.gate ? 1.f / (1.f + expf(-a.gate[(size_t)(first + pos) * a.gate_stride + h])) : 1.f;
    inv_s[row] = l > 0.f ? factor / l : 0.f;
  }
  // the runs' sums meet in the place of keys and values: [run][query][column]
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int e = 0; e < NP; ++e) {
      const int c = NP == 1 ? 2 * lane : 64 * (e & ~1) + 4 * lane + 2 * (e & 1);
      *reinterpret_cast<unsigned long long*>(k_s + (run * PT_Q + vr + r) * DV + c) = o[r][e];
    }
  __syncthreads();
  for (int r = warp; r < n_q; r += PT_THREADS / 32) {
    float* to = a.out + (size_t)(first + p0 + r) * a.out_stride + (size_t)h * a.dv;
    for (int c = lane; c < a.dv; c += 32) {
      float s = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) s += k_s[(e * PT_Q + r) * DV + c];
      to[c] = s * inv_s[r];
    }
  }
}

template <int HD, int DV>
int pt_launch(dim3 grid, const PtArgs& a, cudaStream_t stream) {
  static_assert(4 * PT_Q * DV <= PT_K * (HD + DV), "the runs' sums lie where keys and values did");
  static bool sized[AF_MAX_DEVICES];
  const int dev = af_current_device();
  if (dev < 0) return -1;
  if (af_first_on_device(sized, dev)) {
    const cudaError_t e = cudaFuncSetAttribute(attn_prefill_f32_kernel<HD, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pt_smem(HD, DV));
    if (e != cudaSuccess) return af_fail((int)e, "af_attn_prefill_f32: shared memory: %s", cudaGetErrorString(e));
  }
  af_launch(attn_prefill_f32_kernel<HD, DV>, grid, dim3(PT_THREADS), pt_smem(HD, DV), stream, a);
  AF_CHECK_LAUNCH("af_attn_prefill_f32");
}

}  // namespace

// Attention of the sequences of `least` tokens and more among n_seqs (rows seq_starts[i] .. seq_starts[i + 1] of n_rows; the longest has
// max_len) over the step's own keys and values, all float32; options as in af_attn_prefill_plain.  Keys and values of up to 256.
AF_EXPORT int af_attn_prefill_f32(float* out, long long out_stride, const float* q, long long q_stride, const float* k,
                                  long long k_stride, const float* v, long long v_stride, const int* seq_starts, int n_seqs,
                                  int n_rows, int max_len, int least, int nq, int nkv, int hd, int dv, float scale, float cap, int window,
                                  int mask_kind, int keep, const float* slopes, const float* sinks, const float* gate,
                                  long long gate_stride, cudaStream_t stream) {
  if (n_seqs == 0 || max_len < least) return 0;
  AF_REQUIRE(n_seqs > 0 && n_rows > 0 && max_len > 0 && least > 0 && nq > 0 && nq <= 65535 && nkv > 0 && nq % nkv == 0,
             "af_attn_prefill_f32: %d sequences of %d rows, heads %d, groups %d", n_seqs, n_rows, nq, nkv);
  AF_REQUIRE(hd > 0 && hd <= 256 && dv > 0 && dv <= 256, "af_attn_prefill_f32: key size %d or value size %d beyond 256", hd, dv);
  AF_REQUIRE(mask_kind == AF_MASK_WINDOW || mask_kind == AF_MASK_CHUNK, "af_attn_prefill_f32: mask kind %d", mask_kind);
  AF_REQUIRE(keep >= 0, "af_attn_prefill_f32: %d kept tokens", keep);
  const bool vec = (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) == 0 && ((q_stride | k_stride | v_stride | hd | dv) & 3) == 0;
  const PtArgs a{out, q, k, v, out_stride, q_stride, k_stride, v_stride, seq_starts, n_seqs, least, nq, nkv, hd, dv, scale, cap, window,
                 mask_kind, window > 0 ? keep : 0, slopes, sinks, gate, gate_stride, vec ? 1 : 0};
  // (no more tiles than these: a sequence's last may be short; those of max_len tokens each; a sequence of `least` tokens and more is one of n_rows / least)
  const long long longest = (max_len + PT_Q - 1) / PT_Q, seqs = n_seqs < n_rows / least ? n_seqs : n_rows / least;
  const long long most = n_rows / PT_Q + seqs < longest * seqs ? n_rows / PT_Q + seqs : longest * seqs;
  if (most == 0) return 0;
  const dim3 grid((unsigned)most, nq);
  const int HD = hd <= 64 ? 64 : hd <= 128 ? 128 : 256, DV = dv <= 64 ? 64 : dv <= 128 ? 128 : 256;
  if (DV == 256) return HD == 256 ? pt_launch<256, 256>(grid, a, stream) : pt_launch<128, 256>(grid, a, stream);
  if (HD == 256) return pt_launch<256, 128>(grid, a, stream);
  if (HD == 128 || DV == 128) return pt_launch<128, 128>(grid, a, stream);
  return pt_launch<64, 64>(grid, a, stream);
}
