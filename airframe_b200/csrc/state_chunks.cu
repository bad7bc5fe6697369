// Prompts of the matrix-valued states (recurrent.cu) in chunks of 32 tokens, every sum in true 32 bits: the generalized
// delta rule and linear attention with a decay per head.
//
// Token by token the recurrence is a chain of two reductions a token (690 ns each at 128 key channels) on a few warps.
// In chunks most of it needs no state and runs for all chunks side by side; what is left of the chain is two small products
// a chunk.  With G_t = w_1 .. w_t the decays' running product within a chunk (per key channel), S the state that enters
// it and p_t = S_(t-1)^T u_t what the delta rule takes out:
//   S_t = G_t S + sum over s <= t of (G_t / G_s) (k_s v_s^T - au_s p_s^T)
//   (I + A) P = (U . G_(t-1)) S + B V        A_ts = sum_c u_t au_s G_(t-1) / G_s,  B_ts the same with k_s   (s < t)
//   o_t = (r_t . G_t) S + C V - D P          C_ts = sum_c r_t k_s G_t / G_s, D_ts the same with au_s       (s <= t)
// so with W = (I + A)^-1 (U . G_(t-1)) and P0 = (I + A)^-1 B V a chunk is
//   P = P0 + W S,   o = (C V - D P0) + (r . G - D W) S,   S_out = G_end S + (k . G_end / G)^T V - (au . G_end / G)^T P.
// Linear attention is the same with A = B = D = 0.  Nothing is divided by a decay: G_t / G_s is the product
// w_(s+1) .. w_t itself, along a chain within 16 tokens, and across two groups of 16 as the product from s to its
// group's end times the product from the next group's start to t (all at most 1 where the decays are).
//
// The products are fma.rn.f32x2: operands and sums stay 32-bit, where pairs of bfloat16 (mma_pairs.cuh) would keep 16 to
// 17 bits.  2,048 tokens of 18 heads of 128: the delta rule 1,191 -> 391 us (with what stood in front of it), linear attention
// 628 -> 260 us.  Distance of the outputs from the recurrence in 64 bits (2-norm): 1.1e-7 (token by token 1.0e-7) and
// 5.8e-8 (9.3e-8).
#include "common.cuh"
#include "tma.cuh"

namespace {

constexpr int SC_C = 32;        // tokens of a chunk
constexpr int SC_N = 16;        // value columns of a walking block: 18 heads of 128 values are 144 blocks
constexpr int SC_PM = 36;       // floats of a row of A, B, C, D
constexpr int SC_RANK = 128;    // the largest rank of the decays' low-rank factor
constexpr int SC_LOW = 64;      // rows of it that lie in shared memory at a time

struct StateChunkArgs {
  const float *r, *k, *v;       // rows of H heads of dk (dv) values
  long long r_ts, k_ts, v_ts;
  // delta: removal logits, the low-rank row, biases, the second factor transposed [rank][H * dk]
  const float *a, *low;
  long long a_ts, low_ts;
  const float *a_bias, *w0, *w2t;
  int rank;
  float decay_scale, key_eps;
  const float* decay;           // linear attention: [H]
  int silu;                     // r, k and v through x sigmoid(x) as they are read
  float* blob;                  // [chunks * H][sc_blob]
  float* tiles;                 // [chunks * H][dv / SC_N][sc_tile]
  float* state;                 // [slots][H][dv][dk]
  float* out;                   // [tokens][H * dv], rows out_ts apart
  long long out_ts;
  const int *chunk_starts, *seq_first_chunk, *slots;   // of this launch's first chunk and sequence on
  int chunk0, n_chunks;         // this launch's chunks of the step (a sequence may begin before them and go on behind them)
  int H, dk, dv;
  int* err;
};

// Where a chunk's pieces lie, in memory as in the walking block's shared memory (floats; rows of dk + 4).  Delta rule:
// [W | r . G - D W | k . G_end / G | -au . G_end / G | G_end]; linear attention: [r . G | k . G_end / G | G_end in two
// parts, whose sum is right to 48 bits: its rounding would enter every chunk with the same sign].  A tile of value columns:
// [P0 (delta rule) | C V - D P0 | V], rows of SC_N.
__host__ __device__ constexpr int sc_blob(bool delta, int dk) { return (delta ? 4 : 2) * SC_C * (dk + 4) + (delta ? dk : 2 * dk); }
__host__ __device__ constexpr int sc_tile(bool delta) { return (delta ? 3 : 2) * SC_C * SC_N; }

__device__ __forceinline__ void sc_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long sc_both(float x) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(x));
  return v;
}
__device__ __forceinline__ float2 sc_halves(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ float4 sc_silu(float4 q) {
  q.x = q.x / (1.f + expf(-q.x)), q.y = q.y / (1.f + expf(-q.y));
  q.z = q.z / (1.f + expf(-q.z)), q.w = q.w / (1.f + expf(-q.w));
  return q;
}

// 32 sums over the warp's lanes at once: lane l ends with the sum of everybody's v[l].
__device__ __forceinline__ float sc_sum32(float* v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0];
}

// out[r0 + i][column] = sum over k <= r0 + i of m[k][r0 + i] x[k][column] for four rows i and up to eight columns of a lane
// (four from `col`, four from col + 64 where `second`): m lower triangular, transposed, rows of SC_PM.  No row meets a later
// token's values: zero times an infinity would be NaN.
__device__ __forceinline__ void sc_lower_rows(const float* m, int r0, const float* x, int ldx, bool second, float (&out)[4][8]) {
  unsigned long long acc[4][4] = {};
  auto step = [&](int k, int from) {               // rows from .. 3 of the four take token k's values
    const float4 f = *reinterpret_cast<const float4*>(m + k * SC_PM + r0);
    const unsigned long long fd[4] = {sc_both(f.x), sc_both(f.y), sc_both(f.z), sc_both(f.w)};
    const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(x + k * ldx);
    const ulonglong2 hi = second ? *reinterpret_cast<const ulonglong2*>(x + k * ldx + 64) : make_ulonglong2(0, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i < from) continue;
      sc_fma2(acc[i][0], fd[i], lo.x), sc_fma2(acc[i][1], fd[i], lo.y);
      sc_fma2(acc[i][2], fd[i], hi.x), sc_fma2(acc[i][3], fd[i], hi.y);
    }
  };
#pragma unroll 2
  for (int k = 0; k < r0; ++k) step(k, 0);
#pragma unroll
  for (int i = 0; i < 4; ++i) step(r0 + i, i);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = sc_halves(acc[i][j]);
      out[i][2 * j] = f.x, out[i][2 * j + 1] = f.y;
    }
}

// Four neighbours of a row of the product of two 32 x 32 matrices, a[row][k] b[k][col ..]: rows of SC_PM, or transposed
// (TA, TB), k from k0 to k1.
template <bool TA, bool TB>
__device__ __forceinline__ float4 sc_quad(const float* a, const float* b, int row, int col, int k0, int k1) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (int k = k0; k < k1; ++k) {
    const float x = TA ? a[k * SC_PM + row] : a[row * SC_PM + k];
    float4 y;
    if (TB) y = make_float4(b[col * SC_PM + k], b[(col + 1) * SC_PM + k], b[(col + 2) * SC_PM + k], b[(col + 3) * SC_PM + k]);
    else y = *reinterpret_cast<const float4*>(b + k * SC_PM + col);
    acc.x = fmaf(x, y.x, acc.x), acc.y = fmaf(x, y.y, acc.y), acc.z = fmaf(x, y.z, acc.z), acc.w = fmaf(x, y.w, acc.w);
  }
  return acc;
}
__device__ __forceinline__ void sc_put_column(float* m, int row, int col, float4 v) {      // m[col + i][row]
  m[col * SC_PM + row] = v.x, m[(col + 1) * SC_PM + row] = v.y, m[(col + 2) * SC_PM + row] = v.z, m[(col + 3) * SC_PM + row] = v.w;
}

// Shared memory of the delta rule's chunks: [k | a | decays], behind the cross products in the same place [five factors |
// values]; u, r; A, B, C, D; the first group's whole decays.
constexpr int SC_PX = 132;                         // floats of a token's row of values
constexpr int SC_FACTORS = 4 * SC_C * SC_PM + 16 * SC_PM;
__host__ __device__ constexpr int sc_front(int dk) {
  return 3 * SC_C * (dk + 4) > SC_FACTORS + SC_C * SC_PX ? 3 * SC_C * (dk + 4) : SC_FACTORS + SC_C * SC_PX;
}
constexpr size_t sc_delta_smem(int dk) { return ((size_t)sc_front(dk) + 2 * SC_C * (dk + 4) + 4 * SC_C * SC_PM + dk) * sizeof(float); }

// The delta rule's chunks: block (chunk, head), 256 threads; KP = the key size rounded up to 64 or 128.  Bound by its
// instructions; two blocks an SM cover each other's barriers.  The triangular system is inverted (32 x 32) and applied as
// products in rolled loops: solved a thread a column, straight through, the code of 4,000 instructions that a warp runs
// once was fetched slower than it ran (53,000 of a block's 140,000 cycles).
template <int KP>
__global__ void __launch_bounds__(256, 2)
delta_chunks_kernel(StateChunkArgs a) {
  pdl_launch_dependents();
  constexpr int NE = KP / 32, TT = SC_C * KP / 256;
  extern __shared__ __align__(16) float sm[];
  const int dk = a.dk, dv = a.dv, DP = dk + 4, quads = dk / 4;
  float *k_s = sm + sc_front(dk) - 3 * SC_C * DP, *a_s = k_s + SC_C * DP, *g_s = a_s + SC_C * DP, *u_s = g_s + SC_C * DP,
        *r_s = u_s + SC_C * DP;
  float *A_s = r_s + SC_C * DP, *B_s = A_s + SC_C * SC_PM, *C_s = B_s + SC_C * SC_PM, *D_s = C_s + SC_C * SC_PM;
  float* half_s = D_s + SC_C * SC_PM;             // [dk]: the first 16 tokens' whole product
  float* low_s = A_s;                             // [rank][SC_PM], before A .. D are made
  float* w2_s = g_s;                              // [SC_LOW][dk], before the decays and u are made
  float *T_t = sm, *DT_t = T_t + SC_C * SC_PM, *TB_t = DT_t + SC_C * SC_PM, *E_t = TB_t + SC_C * SC_PM, *X_s = E_t + SC_C * SC_PM;
  float* v_s = sm + SC_FACTORS;                   // [SC_C][SC_PX]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ch = blockIdx.x, h = blockIdx.y;
  const size_t unit = (size_t)ch * a.H + h, n = (size_t)a.H * dk;
  float* blob = a.blob + unit * sc_blob(true, dk);
  const int first = a.chunk_starts[ch], rows = a.chunk_starts[ch + 1] - first;
  auto fetch_low = [&](int l0) {                  // weights: the first rows before the wait for the projection
    const int count = min(SC_LOW, a.rank - l0) * quads;
    for (int i = tid; i < count; i += 256) {
      const int l = i / quads, c = (i - l * quads) * 4;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(w2_s + l * dk + c)),
                   "l"(a.w2t + (size_t)(l0 + l) * n + h * dk + c) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch_low(0);
  pdl_wait();
  a.r = pdl_fresh(a.r), a.k = pdl_fresh(a.k), a.v = pdl_fresh(a.v), a.a = pdl_fresh(a.a), a.low = pdl_fresh(a.low);
#pragma unroll 4
  for (int i = tid; i < SC_C * quads; i += 256) {
    const int t = i / quads, c = (i - t * quads) * 4;
    float4 rq = make_float4(0.f, 0.f, 0.f, 0.f), kq = rq, aq = rq;
    if (t < rows) {
      rq = *reinterpret_cast<const float4*>(a.r + (size_t)(first + t) * a.r_ts + h * dk + c);
      kq = *reinterpret_cast<const float4*>(a.k + (size_t)(first + t) * a.k_ts + h * dk + c);
      aq = *reinterpret_cast<const float4*>(a.a + (size_t)(first + t) * a.a_ts + h * dk + c);
    }
    *reinterpret_cast<float4*>(r_s + t * DP + c) = rq;
    *reinterpret_cast<float4*>(k_s + t * DP + c) = kq;
    *reinterpret_cast<float4*>(a_s + t * DP + c) = aq;
  }
#pragma unroll 4
  for (int i = tid; i < SC_C * a.rank; i += 256) {
    const int t = i / a.rank, l = i - t * a.rank;
    low_s[l * SC_PM + t] = t < rows ? tanhf(a.low[(size_t)(first + t) * a.low_ts + l]) : 0.f;
  }
  // ---- decays (a thread a channel of TT tokens: the second factor is read once for all of them), unit keys, removals
  {
    const int c = tid & (KP - 1), t0 = tid / KP * TT;
    float z[TT];
    const float z0 = c < dk ? a.w0[h * dk + c] : 0.f;
#pragma unroll
    for (int i = 0; i < TT; ++i) z[i] = z0;
    for (int l0 = 0; l0 < a.rank; l0 += SC_LOW) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      const int count = min(SC_LOW, a.rank - l0);
      if (c < dk) {
#pragma unroll 2
        for (int l = 0; l < count; ++l) {
          const float w = w2_s[l * dk + c];
          const float* lo = low_s + (l0 + l) * SC_PM + t0;
#pragma unroll
          for (int i = 0; i < TT; i += 4) {
            const float4 q = *reinterpret_cast<const float4*>(lo + i);
            z[i] = fmaf(q.x, w, z[i]), z[i + 1] = fmaf(q.y, w, z[i + 1]);
            z[i + 2] = fmaf(q.z, w, z[i + 2]), z[i + 3] = fmaf(q.w, w, z[i + 3]);
          }
        }
      }
      __syncthreads();                             // (these rows are read)
      if (l0 + SC_LOW < a.rank) fetch_low(l0 + SC_LOW);
    }
    if (c < dk) {
#pragma unroll 4
      for (int i = 0; i < TT; ++i)
        g_s[(t0 + i) * DP + c] = t0 + i < rows ? expf(-a.decay_scale * (1.f / (1.f + expf(-z[i])))) : 1.f;
    }
  }
  for (int i = tid; i < 4 * SC_C * SC_PM; i += 256) A_s[i] = 0.f;      // (what lies above the diagonals stays zero)
#pragma unroll 1
  for (int t = warp; t < SC_C; t += 8) {
    float x[NE], ss = 0.f;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int c = lane + 32 * e;
      x[e] = c < dk ? k_s[t * DP + c] : 0.f;
      ss = fmaf(x[e], x[e], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float nrm = sqrtf(ss + a.key_eps);
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int c = lane + 32 * e;
      if (c >= dk) continue;
      const float u = t < rows ? x[e] / nrm : 0.f;
      const float rm = 1.f / (1.f + expf(-(a_s[t * DP + c] + a.a_bias[h * dk + c])));
      u_s[t * DP + c] = u;
      a_s[t * DP + c] = rm * u;
    }
  }
  __syncthreads();
  // ---- the two groups by themselves: a warp takes a source token and walks the tokens behind it in its group
#pragma unroll 1
  for (int job = 0; job < 4; ++job) {
    const int base = (job >> 1) * 16, s = base + ((job & 1) ? 15 - warp : warp);
    float pk[NE], pa[NE], vk[32], va[32];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int c = lane + 32 * e;
      pk[e] = c < dk ? k_s[s * DP + c] : 0.f;
      pa[e] = c < dk ? a_s[s * DP + c] : 0.f;
    }
#pragma unroll
    for (int d = 0; d < 16; ++d) {
      float bk = 0.f, ba = 0.f, ck = 0.f, da = 0.f;
      if (s + d < base + 16) {
        const int at = (s + d) * DP + lane;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          if (lane + 32 * e >= dk) continue;
          if (d > 0) {
            const float u = u_s[at + 32 * e], g = g_s[at + 32 * e];
            bk = fmaf(u, pk[e], bk), ba = fmaf(u, pa[e], ba);
            pk[e] *= g, pa[e] *= g;
          }
          const float r = r_s[at + 32 * e];
          ck = fmaf(r, pk[e], ck), da = fmaf(r, pa[e], da);
        }
      }
      vk[2 * d] = bk, vk[2 * d + 1] = ck;
      va[2 * d] = ba, va[2 * d + 1] = da;
    }
    const float sk = sc_sum32(vk), sa = sc_sum32(va);
    const int t = s + (lane >> 1);
    if (t < base + 16) {
      if (lane & 1) C_s[t * SC_PM + s] = sk, D_s[t * SC_PM + s] = sa;
      else if (t > s) B_s[t * SC_PM + s] = sk, A_s[t * SC_PM + s] = sa;
    }
  }
  __syncthreads();
  // ---- running products, a thread a channel.  From the front (half the threads): u times what lies before it in its
  // group, r times that and its own decay.  From the back: keys and removals times what follows them in the chunk go out;
  // the first group's, times what follows in their group, stay in place.
  {
    const int c = tid & 127;
    if (c < dk) {
      float g[SC_C];
#pragma unroll
      for (int t = 0; t < SC_C; ++t) g[t] = g_s[t * DP + c];
      if (tid < 128) {
        float P = 1.f, half = 1.f;
#pragma unroll
        for (int t0 = 0; t0 < SC_C; t0 += 8) {
          float u[8], r[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) u[i] = u_s[(t0 + i) * DP + c], r[i] = r_s[(t0 + i) * DP + c];
          if (t0 == 16) half = P, P = 1.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            u_s[(t0 + i) * DP + c] = u[i] * P;
            P *= g[t0 + i];
            r_s[(t0 + i) * DP + c] = r[i] * P;
          }
        }
        half_s[c] = half;
        blob[4 * SC_C * DP + c] = half * P;
      } else {
        float *ko = blob + 2 * SC_C * DP + c, *ao = ko + SC_C * DP;
        float x = 1.f, second = 1.f;
#pragma unroll
        for (int s0 = SC_C - 8; s0 >= 0; s0 -= 8) {
          float k[8], q[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) k[i] = k_s[(s0 + i) * DP + c], q[i] = a_s[(s0 + i) * DP + c];
          if (s0 == 8) second = x, x = 1.f;
#pragma unroll
          for (int i = 7; i >= 0; --i) {
            const int s = s0 + i;
            const float kk = k[i] * x, aa = q[i] * x;
            ko[s * DP] = s < 16 ? kk * second : kk;
            ao[s * DP] = s < 16 ? -(aa * second) : -aa;
            if (s < 16) k_s[s * DP + c] = kk, a_s[s * DP + c] = aa;
            x *= g[s];
          }
        }
      }
    }
  }
  __syncthreads();
  // ---- the second group's tokens against the first group's: a thread a pair
  auto fetch_values = [&](int j0) {
    const int q4 = min(128, dv - j0) / 4;
#pragma unroll 4
    for (int i = tid; i < SC_C * q4; i += 256) {
      const int t = i / q4, c = (i - t * q4) * 4;
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < rows) q = *reinterpret_cast<const float4*>(a.v + (size_t)(first + t) * a.v_ts + (size_t)h * dv + j0 + c);
      *reinterpret_cast<float4*>(v_s + t * SC_PX + c) = q;
    }
  };
  {
    const int t = 16 + (tid >> 4), s = tid & 15;
    float aa = 0.f, bb = 0.f, cc = 0.f, dd = 0.f;
#pragma unroll 2
    for (int c = 0; c < dk; c += 4) {
      const float4 u = *reinterpret_cast<const float4*>(u_s + t * DP + c), r = *reinterpret_cast<const float4*>(r_s + t * DP + c);
      const float4 k = *reinterpret_cast<const float4*>(k_s + s * DP + c), x = *reinterpret_cast<const float4*>(a_s + s * DP + c);
      bb = fmaf(u.x, k.x, bb), aa = fmaf(u.x, x.x, aa), cc = fmaf(r.x, k.x, cc), dd = fmaf(r.x, x.x, dd);
      bb = fmaf(u.y, k.y, bb), aa = fmaf(u.y, x.y, aa), cc = fmaf(r.y, k.y, cc), dd = fmaf(r.y, x.y, dd);
      bb = fmaf(u.z, k.z, bb), aa = fmaf(u.z, x.z, aa), cc = fmaf(r.z, k.z, cc), dd = fmaf(r.z, x.z, dd);
      bb = fmaf(u.w, k.w, bb), aa = fmaf(u.w, x.w, aa), cc = fmaf(r.w, k.w, cc), dd = fmaf(r.w, x.w, dd);
    }
    A_s[t * SC_PM + s] = aa, B_s[t * SC_PM + s] = bb, C_s[t * SC_PM + s] = cc, D_s[t * SC_PM + s] = dd;
  }
  __syncthreads();                                 // (k, a and the decays are done with: factors and values lie in their place)
  fetch_values(0);
  for (int i = tid; i < 16 * quads; i += 256) {    // u . G of the second group from the chunk's start
    const int t = 16 + i / quads, c = (i % quads) * 4;
    float4 q = *reinterpret_cast<const float4*>(u_s + t * DP + c);
    const float4 f = *reinterpret_cast<const float4*>(half_s + c);
    *reinterpret_cast<float4*>(u_s + t * DP + c) = make_float4(q.x * f.x, q.y * f.y, q.z * f.z, q.w * f.w);
  }
  for (int i = tid; i < SC_C * SC_PM; i += 256) T_t[i] = 0.f;
  __syncthreads();
  // ---- T = (I + A)^-1, transposed: its diagonal blocks a thread a column, then T21 = -T22 A21 T11
  if (tid < 32) {
    const int base = (tid >> 4) * 16, col = tid & 15;
    float x[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const float* row = A_s + (base + t) * SC_PM + base;
      float x0 = t == col ? 1.f : 0.f, x1 = 0.f;
#pragma unroll
      for (int s = 0; s < t; s += 2) {
        x0 = fmaf(-row[s], x[s], x0);
        if (s + 1 < t) x1 = fmaf(-row[s + 1], x[s + 1], x1);
      }
      x[t] = x0 + x1;
    }
#pragma unroll
    for (int t = 0; t < 16; ++t) T_t[(base + col) * SC_PM + base + t] = x[t];
  }
  __syncthreads();
  const int qr = tid >> 3, qc = (tid & 7) * 4;     // a thread's four places of a 32 x 32 product
  if (tid < 64) {                                  // X = A21 T11
    const int row = tid >> 2, col = (tid & 3) * 4;
    *reinterpret_cast<float4*>(X_s + row * SC_PM + col) = sc_quad<false, true>(A_s + 16 * SC_PM, T_t, row, col, 0, 16);
  }
  __syncthreads();
  if (tid < 64) {
    const int row = tid >> 2, col = (tid & 3) * 4;
    const float4 q = sc_quad<true, false>(T_t + 16 * SC_PM + 16, X_s, row, col, 0, row + 1);
    sc_put_column(T_t, 16 + row, col, make_float4(-q.x, -q.y, -q.z, -q.w));
  }
  __syncthreads();
  {
    const float4 q = sc_quad<false, true>(D_s, T_t, qr, qc, 0, qr + 1);              // D T
    sc_put_column(DT_t, qr, qc, make_float4(-q.x, -q.y, -q.z, -q.w));
    sc_put_column(TB_t, qr, qc, sc_quad<true, false>(T_t, B_s, qr, qc, 0, qr + 1));  // T B
  }
  __syncthreads();
  {
    const float4 q = sc_quad<false, true>(D_s, TB_t, qr, qc, 0, qr + 1), c = *reinterpret_cast<const float4*>(C_s + qr * SC_PM + qc);
    sc_put_column(E_t, qr, qc, make_float4(c.x - q.x, c.y - q.y, c.z - q.z, c.w - q.w));   // C - D T B
  }
  __syncthreads();
  // ---- [W | r . G - D W] and [P0 | C V - D P0]: half a warp's lanes a matrix; four rows near the top of one factor and four
  // near the bottom of the other a warp, 36 products deep together
  const bool keys = lane < 16;
  const int col = (lane & 15) * 4;
  for (int j0 = 0; j0 < dv; j0 += 128) {
    if (j0 > 0) {
      __syncthreads();
      fetch_values(j0);
      __syncthreads();
    }
    const int width = keys ? (j0 == 0 ? dk : 0) : min(128, dv - j0);
    const bool second = col + 64 < width;
    const float* x = (keys ? u_s : v_s) + col;
    const int ldx = keys ? DP : SC_PX;
    if (col < width) {
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {
        const int r0 = part == 0 ? 4 * warp : 28 - 4 * warp;
        float o[4][8];
        sc_lower_rows(part == 0 ? (keys ? T_t : TB_t) : (keys ? DT_t : E_t), r0, x, ldx, second, o);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = r0 + i;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (q == 1 && !second) continue;
            const int c = col + 64 * q;
            float4 y = make_float4(o[i][4 * q], o[i][4 * q + 1], o[i][4 * q + 2], o[i][4 * q + 3]);
            if (keys) {
              if (part == 1) {
                const float4 r = *reinterpret_cast<const float4*>(r_s + t * DP + c);
                float4 f = make_float4(1.f, 1.f, 1.f, 1.f);
                if (t >= 16) f = *reinterpret_cast<const float4*>(half_s + c);
                y = make_float4(fmaf(r.x, f.x, y.x), fmaf(r.y, f.y, y.y), fmaf(r.z, f.z, y.z), fmaf(r.w, f.w, y.w));
              }
              *reinterpret_cast<float4*>(blob + (part * SC_C + t) * DP + c) = y;
            } else {
              const int j = j0 + c;
              float* tile = a.tiles + (unit * (dv / SC_N) + j / SC_N) * sc_tile(true) + t * SC_N + j % SC_N;
              *reinterpret_cast<float4*>(tile + part * SC_C * SC_N) = y;
              if (part == 0) *reinterpret_cast<float4*>(tile + 2 * SC_C * SC_N) = *reinterpret_cast<const float4*>(v_s + t * SC_PX + c);
            }
          }
        }
      }
    }
  }
}

constexpr size_t sc_decay_smem(int dk) {
  return ((size_t)2 * SC_C * (dk + 4) + SC_C * SC_PX + SC_C * SC_PM + SC_C + 4) * sizeof(float);
}

// Linear attention's chunks: block (chunk, head), 256 threads.  The decay's powers are worked out in 64 bits.
__global__ void __launch_bounds__(256)
decay_chunks_kernel(StateChunkArgs a) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float sm[];
  const int dk = a.dk, dv = a.dv, DP = dk + 4, quads = dk / 4;
  float *r_s = sm, *k_s = r_s + SC_C * DP, *v_s = k_s + SC_C * DP, *C_t = v_s + SC_C * SC_PX, *pw = C_t + SC_C * SC_PM;      // pw [SC_C + 2]: the last one what the whole decay's rounding left
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ch = blockIdx.x, h = blockIdx.y;
  const size_t unit = (size_t)ch * a.H + h;
  float* blob = a.blob + unit * sc_blob(false, dk);
  const int first = a.chunk_starts[ch], rows = a.chunk_starts[ch + 1] - first;
  if (tid <= SC_C) {
    const double d = (double)a.decay[h];
    double p = 1.0;
    for (int i = 0; i < tid; ++i) p *= d;
    pw[tid] = (float)p;
    if (tid == rows) pw[SC_C + 1] = (float)(p - (double)(float)p);
  }
  pdl_wait();
  a.r = pdl_fresh(a.r), a.k = pdl_fresh(a.k), a.v = pdl_fresh(a.v);
  __syncthreads();
  auto fetch_values = [&](int j0) {
    const int q4 = min(128, dv - j0) / 4;
#pragma unroll 4
    for (int i = tid; i < SC_C * q4; i += 256) {
      const int t = i / q4, c = (i - t * q4) * 4;
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < rows) q = *reinterpret_cast<const float4*>(a.v + (size_t)(first + t) * a.v_ts + (size_t)h * dv + j0 + c);
      *reinterpret_cast<float4*>(v_s + t * SC_PX + c) = a.silu ? sc_silu(q) : q;
    }
  };
#pragma unroll 4
  for (int i = tid; i < SC_C * quads; i += 256) {
    const int t = i / quads, c = (i - t * quads) * 4;
    float4 rq = make_float4(0.f, 0.f, 0.f, 0.f), kq = rq;
    float pk = 0.f;
    if (t < rows) {
      rq = *reinterpret_cast<const float4*>(a.r + (size_t)(first + t) * a.r_ts + h * dk + c);
      kq = *reinterpret_cast<const float4*>(a.k + (size_t)(first + t) * a.k_ts + h * dk + c);
      if (a.silu) rq = sc_silu(rq), kq = sc_silu(kq);
      pk = pw[rows - 1 - t];
    }
    *reinterpret_cast<float4*>(r_s + t * DP + c) = rq;
    *reinterpret_cast<float4*>(k_s + t * DP + c) = kq;
    const float pr = pw[t + 1];
    *reinterpret_cast<float4*>(blob + t * DP + c) = make_float4(rq.x * pr, rq.y * pr, rq.z * pr, rq.w * pr);
    *reinterpret_cast<float4*>(blob + (SC_C + t) * DP + c) = make_float4(kq.x * pk, kq.y * pk, kq.z * pk, kq.w * pk);
  }
  if (tid < dk) blob[2 * SC_C * DP + tid] = pw[rows], blob[2 * SC_C * DP + dk + tid] = pw[SC_C + 1];
  fetch_values(0);
  __syncthreads();
  {
    const int t = tid >> 4, s = tid & 15;          // pairs (t, s), (t, s + 16), (t + 16, s), (t + 16, s + 16)
    float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 2
    for (int c = 0; c < dk; c += 4) {
      float4 q[2], k[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        q[i] = *reinterpret_cast<const float4*>(r_s + (t + 16 * i) * DP + c);
        k[i] = *reinterpret_cast<const float4*>(k_s + (s + 16 * i) * DP + c);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          acc[i][e] = fmaf(q[i].w, k[e].w, fmaf(q[i].z, k[e].z, fmaf(q[i].y, k[e].y, fmaf(q[i].x, k[e].x, acc[i][e]))));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int tt = t + 16 * i, ss = s + 16 * e;
        C_t[ss * SC_PM + tt] = ss <= tt ? acc[i][e] * pw[tt - ss] : 0.f;
      }
  }
  __syncthreads();
  // ---- C V: four rows a warp, four columns a lane
  const int col = lane * 4, r0 = 4 * warp;
  for (int j0 = 0; j0 < dv; j0 += 128) {
    if (j0 > 0) {
      __syncthreads();
      fetch_values(j0);
      __syncthreads();
    }
    if (j0 + col < dv) {
      float o[4][8];
      sc_lower_rows(C_t, r0, v_s + col, SC_PX, false, o);
      const int j = j0 + col;
      float* tile = a.tiles + (unit * (dv / SC_N) + j / SC_N) * sc_tile(false) + r0 * SC_N + j % SC_N;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<float4*>(tile + i * SC_N) = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
        *reinterpret_cast<float4*>(tile + (SC_C + i) * SC_N) = *reinterpret_cast<const float4*>(v_s + (r0 + i) * SC_PX + col);
      }
    }
  }
}

// A contiguous piece from global to shared memory, counted by an mbarrier (16-byte aligned, a multiple of 16 bytes).
__device__ __forceinline__ void sc_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

constexpr size_t sc_walk_smem(bool delta, int dk) {
  return ((size_t)2 * (sc_blob(delta, dk) + sc_tile(delta)) + (delta ? 1 : 2) * SC_N * (dk + 4) + (delta ? SC_C * SC_N : 0)) * sizeof(float);
}

// v[0 .. 2 N) summed over the lanes that differ in `bit`, which keep a half each: the upper one v[N ..].
template <int N>
__device__ __forceinline__ void sc_halve(float* v, int bit) {
  const bool up = threadIdx.x & bit;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float keep = up ? v[i + N] : v[i], give = up ? v[i] : v[i + N];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
  }
}

// Eight rows of a chunk's matrix by four columns of the state, over the key channels: eight lanes take every eighth
// 16-byte piece, their sums meet by halving: lane `part` is left with row 4 b0 + 2 b1 + b2 of its bits.
__device__ __forceinline__ float4 sc_rows_times_state(const float* m, const float* st, int DP, int dk, int part) {
  unsigned long long acc[8][4] = {};
#pragma unroll 1
  for (int k = part * 4; k < dk; k += 32) {
    ulonglong2 y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const ulonglong2*>(st + j * DP + k);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(m + i * DP + k);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sc_fma2(acc[i][j], x.x, y[j].x);
        sc_fma2(acc[i][j], x.y, y[j].y);
      }
    }
  }
  __syncwarp();
  float s[32];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = sc_halves(acc[i][j]);
      s[i * 4 + j] = f.x + f.y;
    }
  sc_halve<16>(s, 1);
  sc_halve<8>(s, 2);
  sc_halve<4>(s, 4);
  return make_float4(s[0], s[1], s[2], s[3]);
}

// Eight key channels (pairs of two) by four value columns: one token's part of k^T v.
__device__ __forceinline__ void sc_outer(unsigned long long (&acc)[4][4], const float* k, const float* v) {
  const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(k), k1 = *reinterpret_cast<const ulonglong2*>(k + 4);
  const float4 f = *reinterpret_cast<const float4*>(v);
  const unsigned long long vd[4] = {sc_both(f.x), sc_both(f.y), sc_both(f.z), sc_both(f.w)};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sc_fma2(acc[j][0], k0.x, vd[j]), sc_fma2(acc[j][1], k0.y, vd[j]);
    sc_fma2(acc[j][2], k1.x, vd[j]), sc_fma2(acc[j][3], k1.y, vd[j]);
  }
}

// Block (SC_N value columns, head, sequence), eight warps, walks the sequence's chunks with its columns of the state in
// registers and, transposed to [column][key channel], in shared memory; the next chunk's pieces come by two bulk copies
// meanwhile.  Delta rule: all warps P and the outputs, a barrier, all warps the new state (four lanes share a tile of it and
// the tokens between them).  Linear attention: four warps the outputs, four the new state into the other of two places.
// Bound by the bytes that lanes load from shared memory (a 16-byte load takes four cycles of it, however many lanes read
// the same): tiles of 8 by 4 a lane, the rest of the lanes along the sum.  Tiles of 4 by 4 (and values stored twice for
// the packed products) took 227 us for 2,048 tokens of 18 heads of 128.
template <bool DELTA>
__global__ void __launch_bounds__(256)
state_walk_kernel(StateChunkArgs a) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float sm[];
  __shared__ uint64_t full[2];
  __shared__ int give_up_s;
  volatile int* give_up = &give_up_s;
  const int dk = a.dk, dv = a.dv, DP = dk + 4;
  const int blob_n = sc_blob(DELTA, dk), stage_n = blob_n + sc_tile(DELTA);
  float* s_T = sm + 2 * stage_n;                   // [1 or 2][SC_N][DP]
  float* p_s = s_T + SC_N * DP;                    // delta: [SC_C][SC_N]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, b = blockIdx.z, tiles = gridDim.x;
  const int j0 = blockIdx.x * SC_N;
  const int ch0 = max(a.seq_first_chunk[b] - a.chunk0, 0), ch1 = min(a.seq_first_chunk[b + 1] - a.chunk0, a.n_chunks);
  const int slot = a.slots[b];
  if (ch0 >= ch1) return;
  if (slot < 0) {                                  // (a padding row: zeros, and no state)
    pdl_wait();
    const int first = a.chunk_starts[ch0], count = (a.chunk_starts[ch1] - first) * (SC_N / 4);
    for (int i = tid; i < count; i += 256)
      *reinterpret_cast<float4*>(a.out + (size_t)(first + i / (SC_N / 4)) * a.out_ts + (size_t)h * dv + j0 + i % (SC_N / 4) * 4) =
          make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    give_up_s = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();
  auto load = [&](int ch, int which) {             // (one thread)
    float* sg = sm + which * stage_n;
    const size_t unit = (size_t)ch * a.H + h;
    mbar_expect_tx(&full[which], (uint32_t)stage_n * 4);
    sc_bulk(sg, a.blob + unit * blob_n, (uint32_t)blob_n * 4, &full[which]);
    sc_bulk(sg + blob_n, a.tiles + (unit * tiles + blockIdx.x) * sc_tile(DELTA), (uint32_t)sc_tile(DELTA) * 4, &full[which]);
  };
  if (tid == 0) load(ch0, 0);
  // this thread's piece of the state: eight key channels from c0 of COLS columns from col0
  constexpr int COLS = DELTA ? 1 : 2, SPLITS = 4 / COLS;
  const int cg = lane & 3, split = (lane >> 2) & (SPLITS - 1);
  const int group = DELTA ? warp * 2 + (lane >> 4) : (warp - 4) * 4 + (lane >> 3);
  const int c0 = group * 8, col0 = cg * 4 + (split & 1) * 2 + (DELTA ? split >> 1 : 0);
  const bool state_warp = group >= 0, mine = state_warp && c0 < dk;
  float* st = a.state + (((size_t)slot * a.H + h) * dv + j0) * dk;
  float4 S[COLS][2];
#pragma unroll
  for (int j = 0; j < COLS; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      S[j][e] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (mine) {
        S[j][e] = *reinterpret_cast<const float4*>(st + (size_t)(col0 + j) * dk + c0 + 4 * e);
        *reinterpret_cast<float4*>(s_T + (col0 + j) * DP + c0 + 4 * e) = S[j][e];
      }
    }
  const int part = lane & 7, ocg = lane >> 3;
  const int orow = 8 * warp + (part & 1) * 4 + (part & 2) + (part >> 2);
  bool ok = true;
  for (int ch = ch0; ch < ch1; ++ch) {
    const int i = ch - ch0, which = i & 1;
    mbar_wait(&full[which], (i >> 1) & 1, give_up);
    __syncthreads();                               // (the chunk's pieces and the state are there; the other stage is free)
    if (*give_up) {
      ok = false;
      break;
    }
    if (ch + 1 < ch1 && tid == 0) load(ch + 1, which ^ 1);
    const float *sg = sm + which * stage_n, *tile = sg + blob_n;
    const float* cur = s_T + (DELTA ? 0 : which * SC_N * DP);
    const int first = a.chunk_starts[ch], rows = a.chunk_starts[ch + 1] - first;
    if (DELTA || warp < 4) {                       // rows of [W | r . G - D W] (delta), of r . G, times the state
      float4 o = sc_rows_times_state(sg + 8 * warp * DP, cur + ocg * 4 * DP, DP, dk, part);
      const float4 o0 = *reinterpret_cast<const float4*>(tile + orow * SC_N + ocg * 4);
      o.x += o0.x, o.y += o0.y, o.z += o0.z, o.w += o0.w;
      if (DELTA && warp < 4) {
        *reinterpret_cast<float4*>(p_s + orow * SC_N + ocg * 4) = o;
      } else {
        const int row = DELTA ? orow - SC_C : orow;
        if (row < rows)
          *reinterpret_cast<float4*>(a.out + (size_t)(first + row) * a.out_ts + (size_t)h * dv + j0 + ocg * 4) = o;
      }
    }
    if (DELTA) __syncthreads();                    // (P is there, and nobody reads the old state any more)
    if (state_warp) {
      unsigned long long acc[4][4] = {};
      if (mine) {
        const float *kd = sg + (DELTA ? 2 : 1) * SC_C * DP + c0, *vs = tile + (DELTA ? 2 : 1) * SC_C * SC_N + cg * 4;
#pragma unroll 2
        for (int t = split; t < SC_C; t += SPLITS) {
          sc_outer(acc, kd + t * DP, vs + t * SC_N);
          if (DELTA) sc_outer(acc, kd + (SC_C + t) * DP, p_s + t * SC_N + cg * 4);
        }
      }
      __syncwarp();
      float v[32];                                 // [column][channel]
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = sc_halves(acc[j][e]);
          v[j * 8 + 2 * e] = f.x, v[j * 8 + 2 * e + 1] = f.y;
        }
      sc_halve<16>(v, 4);                          // the lanes of a tile keep their columns of it
      if (DELTA) sc_halve<8>(v, 8);
      if (mine) {
        const float* pe = sg + blob_n - (DELTA ? dk : 2 * dk) + c0;
        float* next = s_T + (DELTA ? 0 : (which ^ 1) * SC_N * DP);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float4 f = *reinterpret_cast<const float4*>(pe + 4 * e);
          const float4 f2 = DELTA ? f : *reinterpret_cast<const float4*>(pe + dk + 4 * e);
#pragma unroll
          for (int j = 0; j < COLS; ++j) {
            const float* add = v + j * 8 + 4 * e;
            float4 x = make_float4(add[0], add[1], add[2], add[3]);
            const float4 q = S[j][e];
            if (!DELTA) x = make_float4(fmaf(f2.x, q.x, x.x), fmaf(f2.y, q.y, x.y), fmaf(f2.z, q.z, x.z), fmaf(f2.w, q.w, x.w));
            S[j][e] = make_float4(fmaf(f.x, q.x, x.x), fmaf(f.y, q.y, x.y), fmaf(f.z, q.z, x.z), fmaf(f.w, q.w, x.w));
            *reinterpret_cast<float4*>(next + (col0 + j) * DP + c0 + 4 * e) = S[j][e];
          }
        }
      }
    }
  }
  if (!ok) {
    if (tid == 0) {
      grace_period();
      if (a.err) atomicExch(a.err, 1);
    }
    return;
  }
  if (mine) {
#pragma unroll
    for (int j = 0; j < COLS; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) *reinterpret_cast<float4*>(st + (size_t)(col0 + j) * dk + c0 + 4 * e) = S[j][e];
  }
}

template <typename K>
int sc_launch(K kernel, bool* flags, size_t most, size_t smem, dim3 grid, cudaStream_t stream, const StateChunkArgs& a) {
  const int dev = af_current_device();
  if (dev < 0) return -1;
  if (af_first_on_device(flags, dev)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return af_fail((int)e, "af_state_chunks: %s", cudaGetErrorString(e));
  }
  af_launch(kernel, grid, dim3(256), smem, stream, a);
  AF_COUNT_LAUNCH("af_state_chunks");
  return 0;
}

}  // namespace

AF_EXPORT int af_state_chunks_size() { return SC_C; }
AF_EXPORT int af_state_chunks_supported(int dk, int dv, int rank) {
  return dk >= 16 && dk <= 128 && dk % 16 == 0 && dv >= SC_N && dv % SC_N == 0 && rank <= SC_RANK ? 1 : 0;
}
// Floats of scratch a chunk and head: blob (which 0) and tiles (1).
AF_EXPORT long long af_state_chunks_scratch(int delta, int dk, int dv, int which) {
  return which == 0 ? sc_blob(delta != 0, dk) : (long long)(dv / SC_N) * sc_tile(delta != 0);
}

// A prefill step's recurrence over the n_chunks chunks from chunk0 on, which lie in n_seqs sequences; chunk_starts, slots and
// seq_first_chunk begin at the first of them (seq_first_chunk counts from the step's first chunk).  A sequence may be cut by
// the range: the next launch goes on from the state that this one leaves.  `delta`: the generalized delta rule from r, k, v,
// the removals' logits a, the low-rank rows `low` [rank] and their weights; else linear attention with a decay per head.
AF_EXPORT int af_state_chunks(int delta, float* out, long long out_ts, const float* r, long long r_ts, const float* k,
                              long long k_ts, const float* v, long long v_ts, const float* la, long long la_ts,
                              const float* low, long long low_ts, const float* a_bias, const float* w0, const float* w2t,
                              int rank, float decay_scale, float key_eps, const float* decay, int silu, float* state,
                              float* blob, float* tiles, const int* chunk_starts, const int* seq_first_chunk, const int* slots,
                              int chunk0, int n_chunks, int n_seqs, int H, int dk, int dv, int* err, cudaStream_t stream) {
  if (n_chunks == 0) return 0;
  AF_REQUIRE(af_state_chunks_supported(dk, dv, delta ? rank : 1), "af_state_chunks: heads of %d keys and %d values, rank %d", dk, dv, rank);
  AF_REQUIRE(chunk0 >= 0 && n_chunks > 0 && n_seqs > 0 && n_seqs < 65536 && H > 0 && H < 65536 && (!delta || rank > 0), "af_state_chunks: bad sizes");
  AF_REQUIRE(((r_ts | k_ts | v_ts | la_ts | out_ts) & 3) == 0 &&
                 (((uintptr_t)r | (uintptr_t)k | (uintptr_t)v | (uintptr_t)la | (uintptr_t)blob | (uintptr_t)tiles | (uintptr_t)out |
                   (uintptr_t)state | (uintptr_t)w2t) & 15) == 0,
             "af_state_chunks: rows of whole 16-byte pieces");
  StateChunkArgs a{r, k, v, r_ts, k_ts, v_ts, la, low, la_ts, low_ts, a_bias, w0, w2t, rank, decay_scale, key_eps, decay, silu,
                   blob, tiles, state, out, out_ts, chunk_starts, seq_first_chunk, slots, chunk0, n_chunks, H, dk, dv, err};
  static bool raised[5][AF_MAX_DEVICES];
  const dim3 chunks(n_chunks, H), walk(dv / SC_N, H, n_seqs);
  int e;
  if (delta) {
    e = dk <= 64 ? sc_launch(delta_chunks_kernel<64>, raised[0], sc_delta_smem(64), sc_delta_smem(dk), chunks, stream, a)
                 : sc_launch(delta_chunks_kernel<128>, raised[1], sc_delta_smem(128), sc_delta_smem(dk), chunks, stream, a);
    return e ? e : sc_launch(state_walk_kernel<true>, raised[2], sc_walk_smem(true, 128), sc_walk_smem(true, dk), walk, stream, a);
  }
  e = sc_launch(decay_chunks_kernel, raised[3], sc_decay_smem(128), sc_decay_smem(dk), chunks, stream, a);
  return e ? e : sc_launch(state_walk_kernel<false>, raised[4], sc_walk_smem(false, 128), sc_walk_smem(false, dk), walk, stream, a);
}
