// 32-bit matrix product out[M, N] = x[M, K] * w[N, K]^T for prompts, on the 5th-generation tensor cores.
//
// Every operand is taken apart into three bfloat16 parts: x = hi + mid + lo, each the nearest to what the parts before it leave.
// The remainders are exact and have a sign, so the three hold all 24 bits where 2^-110 <= |x| < 3.38e38 (bfloat16 ends at
// 2^-133: below, lo is off by up to 2^-134; above, hi is infinite: see the end).  Of the nine products of parts six are
// taken, from the smallest up: lo hi, hi lo, mid mid, mid hi, hi mid, hi hi; what is left out (mid lo, lo mid, lo lo) is at most
// 2^-24 of a product, of either sign (parts cut off instead of rounded leave out up to 2^-21, always of the product's sign).  The
// tensor cores' accumulator rounds towards zero, which over a long sum would drift: it holds 64 products of K at a time
// and the blocks' sums are added up in registers, in index order, by 32-bit additions that round to nearest.  Distance from
// the product in 64 bits (2-norm) for K of 64 to 9,216: normal values 7.7e-8 to 1.3e-7, where the chain of fmaf is 1.4e-7 to
// 1.7e-6 away; positive ones from 1 to 2 6.1e-8 to 7.6e-8 (on average -0.9 x 2^-24, the accumulator's), the chain 1.2e-7 to 1.5e-6.
//
// A block makes 128 features (weight rows: the MMA's A operand, TMEM lanes) by NT tokens.  The tokens' parts come from a
// small kernel and by TMA; the weights stay as they are in memory and are taken apart on their way into shared memory:
//   warps 0 .. 7   weights: global -> registers (a stage ahead) -> three swizzled tiles; the sums: TMEM -> registers
//   warp 8         TMEM, MMA issue (one lane)
//   warp 9         TMA (one lane)
// Two stages of 64 of K, two accumulators in turn.  Bound by the worker warps' instructions (taking a value apart, five and a
// half each) and, with 160 tokens, by shared memory (an MMA of 128 x 160 x 16 reads 9 KB of it in 80 cycles of products; the
// parts are written besides).  301 x 18432 x 2304: 132 us (194 TFLOP/s of 32-bit products), where the CUDA cores' kernel
// (gemm_plain.cu), which keeps the single tokens' and the small weights' products, takes 592; before the rare values left the way (182 us:
// a test a value, and the exact chain unrolled into the epilogue), weights were asked into L2 ahead, and TMEM was read
// 32 columns at a time.
//
// An output that is not finite is made again as a plain chain of fmaf (the parts of an infinity, and of a value that rounds to
// one, are NaN).
#include "umma.cuh"

namespace {

constexpr int FT_BM = 128, FT_BK = 64, FT_STAGES = 2;
constexpr int FT_AHEAD = 4;                                // K blocks between a weight's way into L2 and into registers
constexpr int FT_WORKERS = 256, FT_THREADS = FT_WORKERS + 64;
constexpr int FT_PART = FT_BM * FT_BK * 2;                 // bytes of a part of a weight tile

__host__ __device__ constexpr int ft_stage(int nt) { return 3 * FT_PART + 3 * nt * FT_BK * 2; }
__host__ __device__ constexpr int ft_smem(int nt) { return FT_STAGES * ft_stage(nt) + 1024; }

struct FtArgs {
  float* out;               // [M, N], rows ldo apart; with several splits [splits][M][N]
  long long ldo, split_stride;
  const float* x;
  long long ldx;
  const float* w;
  long long ldw;
  int M, N, K, part_rows;   // part_rows: rows between two parts of the tokens
  int kb_per_split;
  float cap;
  int* err;
};

// Two values into their parts, a pair of bfloat16 each (x below): rounded two at a time.
__device__ __forceinline__ uint32_t ft_nearest(float x, float y) {
  uint32_t p;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(y), "f"(x));
  return p;
}
__device__ __forceinline__ void ft_split2(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = ft_nearest(x, y);
  x -= __uint_as_float(hi << 16), y -= __uint_as_float(hi & 0xffff0000u);
  mid = ft_nearest(x, y);
  x -= __uint_as_float(mid << 16), y -= __uint_as_float(mid & 0xffff0000u);
  lo = ft_nearest(x, y);                                   // (what is not finite leaves NaN: its outputs are made again)
}

// Four values into three tiles of packed parts.
__device__ __forceinline__ void ft_split4(float4 v, uint2 (&p)[3]) {
  ft_split2(v.x, v.y, p[0].x, p[1].x, p[2].x);
  ft_split2(v.z, v.w, p[0].y, p[1].y, p[2].y);
}

// The tokens' parts: [3][rows][Kp] bfloat16, zeros from K on.
__global__ void __launch_bounds__(256)
f32_parts_kernel(uint2* __restrict__ parts, const float* __restrict__ x, long long ldx, int M, int K, int Kp) {
  pdl_launch_dependents();
  pdl_wait();
  x = pdl_fresh(x);
  const int k = (blockIdx.x * 256 + threadIdx.x) * 4, m = blockIdx.y;
  if (k >= Kp) return;
  uint2 p[3];
  ft_split4(k < K ? *reinterpret_cast<const float4*>(x + (size_t)m * ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f), p);
#pragma unroll
  for (int i = 0; i < 3; ++i) parts[(((size_t)i * M + m) * Kp + k) / 4] = p[i];
}

template <int NT>
__global__ void __launch_bounds__(FT_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, FtArgs a) {
  constexpr int HALF = NT / 2, STAGE = ft_stage(NT);
  constexpr uint32_t IDESC = umma_idesc(NT);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_w[FT_STAGES], full_x[FT_STAGES], empty[FT_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int give_up_s;
  volatile int* give_up = &give_up_s;
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total_kb = (a.K + FT_BK - 1) / FT_BK;
  const int kb0 = blockIdx.z * a.kb_per_split, count = min(a.kb_per_split, total_kb - kb0);
  const int n0 = blockIdx.x * FT_BM, m0 = blockIdx.y * NT;
  if (tid == 0) {
    for (int s = 0; s < FT_STAGES; ++s) {
      mbar_init(&full_w[s], FT_WORKERS / 32);
      mbar_init(&full_x[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], FT_WORKERS / 32);
    }
    give_up_s = 0;
    mbar_fence_init();
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;                       // the two accumulators: 256 columns apart

  if (warp < 8) {
    // a thread's 8 pieces of 16 bytes of a weight tile: rows tid / 16 + 16 i, values 4 (tid % 16) ..
    const int wr = tid >> 4, wk = (tid & 15) * 4;
    const float* src = a.w + (size_t)(n0 + wr) * a.ldw + wk;
    float4 q[8];
    auto fetch = [&](int kb) {
      const int k = (kb0 + kb) * FT_BK;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        q[i] = (n0 + wr + 16 * i < a.N && k + wk < a.K) ? *reinterpret_cast<const float4*>(src + (size_t)(16 * i) * a.ldw + k)
                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    // (and asked into L2 well ahead: a line a thread)
    const float* line = a.w + (size_t)(n0 + (tid >> 1)) * a.ldw + (tid & 1) * 32;
    auto ask = [&](int kb) {
      const int k = (kb0 + kb) * FT_BK;
      if (kb < count && n0 + (tid >> 1) < a.N && k + (tid & 1) * 32 < a.K) prefetch_l2(line + k);
    };
    const int quarter = warp & 3, col0 = (warp >> 2) * HALF;
    float acc[HALF];
#pragma unroll
    for (int j = 0; j < HALF; ++j) acc[j] = 0.f;
    bool ok = true;
    auto add_up = [&](int kb) {                            // K block kb's sums
      const int buf = kb & 1;
      if (!mbar_wait(&acc_full[buf], (kb >> 1) & 1, give_up)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tc_fence_after();
      const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + buf * 256 + col0;
#pragma unroll
      for (int c = 0; c < HALF; c += 32) {
        float v[32];
        tmem_ld16(at + c, v);
        if (c + 16 < HALF) tmem_ld16(at + c + 16, v + 16);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32 && c + j < HALF; ++j) acc[c + j] += v[j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    };
    fetch(0);                                              // (weights: they wait for nothing)
    for (int kb = 1; kb < FT_AHEAD; ++kb) ask(kb);
    pdl_wait();
    for (int kb = 0; kb < count && ok; ++kb) {
      const int s = kb % FT_STAGES;
      if (kb >= FT_STAGES && !mbar_wait(&empty[s], (kb / FT_STAGES - 1) & 1, give_up)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      unsigned char* st = tiles + (size_t)s * STAGE;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint2 p[3];
        ft_split4(q[i], p);
        const int r = wr + 16 * i;
        const uint32_t at = (uint32_t)(r * 128 + ((((tid & 15) >> 1) ^ (r & 7)) << 4) + (tid & 1) * 8);
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(st + e * FT_PART + at) = p[e];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_w[s]);
      if (kb + 1 < count) fetch(kb + 1);
      ask(kb + FT_AHEAD);
      if (kb > 0) add_up(kb - 1);
    }
    if (ok && count > 0) add_up(count - 1);
    const int f = n0 + quarter * 32 + lane;
    if (ok && f < a.N) {
      float* o = a.out + (size_t)blockIdx.z * a.split_stride + f;
      const int k0 = kb0 * FT_BK, k1 = min(a.K, k0 + count * FT_BK);
      bool again = a.cap > 0.f;
#pragma unroll
      for (int j = 0; j < HALF; ++j) {
        if (m0 + col0 + j < a.M) o[(size_t)(m0 + col0 + j) * a.ldo] = acc[j];
        again = again || !isfinite(acc[j]);
      }
      // what is seldom: in a rolled loop over what was just written (as straight code in the loop above it cost every
      // block 25 us of instruction fetches)
      if (again) {
#pragma unroll 1
        for (int m = m0 + col0; m < min(a.M, m0 + col0 + HALF); ++m) {
          float v = o[(size_t)m * a.ldo];
          if (!isfinite(v)) {
            const float *xr = a.x + (size_t)m * a.ldx, *wrow = a.w + (size_t)f * a.ldw;
            v = 0.f;
            for (int k = k0; k < k1 && !isnan(v); ++k) v = fmaf(xr[k], wrow[k], v);
          }
          o[(size_t)m * a.ldo] = softcap_f32(v, a.cap);
        }
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {
      for (int kb = 0; kb < count; ++kb) {
        const int s = kb % FT_STAGES, buf = kb & 1;
        const uint32_t ph = (kb / FT_STAGES) & 1;
        if (kb >= 2 && !mbar_wait(&acc_empty[buf], ((kb >> 1) - 1) & 1, give_up)) break;
        if (!mbar_wait(&full_x[s], ph, give_up) || !mbar_wait(&full_w[s], ph, give_up)) break;
        tc_fence_after();
        const uint32_t st = smem_u32(tiles + (size_t)s * STAGE), d = tmem + buf * 256;
        constexpr int WP[6] = {2, 0, 1, 1, 0, 0}, XP[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int e = 0; e < 6; ++e) {
          const uint64_t da = umma_desc(st + WP[e] * FT_PART), db = umma_desc(st + 3 * FT_PART + XP[e] * NT * FT_BK * 2);
#pragma unroll
          for (int k = 0; k < FT_BK / 16; ++k) umma_f16(d, da + 2 * k, db + 2 * k, IDESC, (e > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&empty[s]);
        umma_commit(&acc_full[buf]);
      }
    }
  } else if (lane == 0) {
    pdl_wait();
    for (int kb = 0; kb < count; ++kb) {
      const int s = kb % FT_STAGES;
      if (kb >= FT_STAGES && !mbar_wait(&empty[s], (kb / FT_STAGES - 1) & 1, give_up)) break;
      unsigned char* st = tiles + (size_t)s * STAGE + 3 * FT_PART;
      mbar_expect_tx(&full_x[s], 3 * NT * FT_BK * 2);
#pragma unroll
      for (int e = 0; e < 3; ++e)
        tma_load_2d(st + e * NT * FT_BK * 2, &map_x, (kb0 + kb) * FT_BK, e * a.part_rows + m0, &full_x[s]);
    }
    if (*give_up) grace_period();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0 && give_up_s && a.err) atomicExch(a.err, 1);
  if (warp == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// out = the splits' sums added in order.
__global__ void __launch_bounds__(256)
f32_join_kernel(float* __restrict__ out, long long ldo, const float* __restrict__ parts, int splits, int M, int N, float cap) {
  pdl_launch_dependents();
  pdl_wait();
  parts = pdl_fresh(parts);
  const int n = blockIdx.x * 256 + threadIdx.x, m = blockIdx.y;
  if (n >= N) return;
  float v = 0.f;
  for (int s = 0; s < splits; ++s) v += parts[((size_t)s * M + m) * N + n];
  out[(size_t)m * ldo + n] = softcap_f32(v, cap);
}

template <int NT>
int ft_launch(const CUtensorMap& map, const FtArgs& a, int splits, cudaStream_t stream) {
  static bool sized[AF_MAX_DEVICES];
  const int dev = af_current_device();
  if (dev < 0) return -1;
  if (af_first_on_device(sized, dev)) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, ft_smem(NT));
    if (e != cudaSuccess) return af_fail((int)e, "af_gemm_f32_tc: shared memory: %s", cudaGetErrorString(e));
  }
  const dim3 grid((a.N + FT_BM - 1) / FT_BM, (a.M + NT - 1) / NT, splits);
  AF_REQUIRE(grid.y <= 65535, "af_gemm_f32_tc: M %d too large", a.M);
  af_launch(gemm_f32_tc_kernel<NT>, grid, dim3(FT_THREADS), ft_smem(NT), stream, map, a);
  AF_COUNT_LAUNCH("af_gemm_f32_tc");
  return 0;
}

}  // namespace

// How many ranges K is cut into: as many as give the device a block an SM for tokens of one or two tiles (the number
// depends on the weight alone, so that a row's result does not change with the rows beside it), each of 512 of K at least.
AF_EXPORT int af_gemm_f32_tc_splits(int N, int K) {
  const int sms = af_sm_count(), tiles = (N + FT_BM - 1) / FT_BM, total = (K + FT_BK - 1) / FT_BK;
  if (sms <= 0) return -1;
  const int want = max(1, min(min(8, sms / (2 * tiles)), total / 8));
  const int per = (total + want - 1) / want;
  return (total + per - 1) / per;
}

// `parts`: 3 M (K rounded up to 64) bfloat16 values of scratch, 16-byte aligned; `sums`: [splits][M][N] floats where
// af_gemm_f32_tc_splits(N, K) > 1.  Rows of whole 16-byte pieces.  `cap` > 0 applies cap * tanh(v / cap).
AF_EXPORT int af_gemm_f32_tc(float* out, long long ldo, const float* x, long long ldx, const float* w, long long ldw, int M,
                             int N, int K, float cap, void* parts, float* sums, int* err, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  AF_REQUIRE(M > 0 && N > 0 && K > 0 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 &&
                 (((uintptr_t)x | (uintptr_t)w | (uintptr_t)parts) & 15) == 0 && M <= 65535,
             "af_gemm_f32_tc: rows of whole 16-byte pieces (M %d N %d K %d)", M, N, K);
  const int splits = af_gemm_f32_tc_splits(N, K);
  if (splits < 1) return -1;
  AF_REQUIRE(splits == 1 || sums != nullptr, "af_gemm_f32_tc: %d splits need scratch memory", splits);
  const int Kp = (K + FT_BK - 1) / FT_BK * FT_BK;
  af_launch(f32_parts_kernel, dim3((Kp / 4 + 255) / 256, M), dim3(256), 0, stream, (uint2*)parts, x, ldx, M, K, Kp);
  AF_COUNT_LAUNCH("af_gemm_f32_tc (parts)");
  // tokens in equal tiles of up to 160
  const int tiles = (M + 159) / 160, nt = ((M + tiles - 1) / tiles + 31) / 32 * 32;
  CUtensorMap map;
  if (int e = af_make_map_bf16(&map, parts, 3ll * M, Kp, Kp, nt)) return e;
  FtArgs a{splits > 1 ? sums : out, splits > 1 ? (long long)N : ldo, (long long)M * N, x, ldx, w, ldw, M, N, K, M,
           ((K + FT_BK - 1) / FT_BK + splits - 1) / splits, splits > 1 ? 0.f : cap, err};
  int e;
  switch (nt) {
    case 32: e = ft_launch<32>(map, a, splits, stream); break;
    case 64: e = ft_launch<64>(map, a, splits, stream); break;
    case 96: e = ft_launch<96>(map, a, splits, stream); break;
    case 128: e = ft_launch<128>(map, a, splits, stream); break;
    default: e = ft_launch<160>(map, a, splits, stream); break;
  }
  if (e || splits == 1) return e;
  af_launch(f32_join_kernel, dim3((N + 255) / 256, M), dim3(256), 0, stream, out, ldo, sums, splits, M, N, cap);
  AF_CHECK_LAUNCH("af_gemm_f32_tc (join)");
}
