// Plain matrix product out[M, N] = x[M, K] * w[N, K]^T on the CUDA cores with
// 32-bit multiply-adds and 32-bit accumulators (no tensor cores, no reduced
// precision mode).  Every output element adds its K products in index order,
// whatever M and N are, so a row's result does not depend on the batch it is
// in.  It is the 32-bit path's matrix product of few rows, of small and of
// unaligned sizes (gemm_f32_tc.cu takes the prompts') and the twin of the
// tensor-core kernels.
//
// float operands run the two gemm_f32 kernels (the reads from shared memory bound them for many rows, an output's chain
// over K for few);
// bfloat16 operands, which come here only where the tensor cores do not take the shape, run gemm_plain_kernel.
#include "common.cuh"

#define GP_BM 64
#define GP_BN 64
#define GP_BK 16

template <typename T, typename TO>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(TO* __restrict__ out, int ldo, const T* __restrict__ x, int ldx,
                  const T* __restrict__ w, int ldw, int M, int N, int K, float cap) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float xs[GP_BK][GP_BM + 1];
  __shared__ float ws[GP_BK][GP_BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, 4 x 4 outputs each
  const int m0 = blockIdx.y * GP_BM, n0 = blockIdx.x * GP_BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += GP_BK) {
    // 64 rows x 16 k per operand = 1024 elements, 4 per thread
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int idx = tid + e * 256;
      const int r = idx >> 4, kk = idx & 15;
      const int k = k0 + kk;
      const int m = m0 + r, n = n0 + r;
      xs[kk][r] = (m < M && k < K) ? to_f32(x[(size_t)m * ldx + k]) : 0.f;
      ws[kk][r] = (n < N && k < K) ? to_f32(w[(size_t)n * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GP_BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(softcap_f32(acc[i][j], cap));
    }
  }
}

// ---- float operands
// A block makes BM x BN outputs, a thread TM x TN of them; a warp's 4 x 8 threads lie side by side (neighbouring lanes
// share a column: 10 % fewer shared-memory accesses than neighbours that share a row), a thread's rows 4 and its columns
// 8 apart.  Both operands' tiles stay rows along K in shared memory, as cp.async brings them (ST stages; out-of-range
// rows and the tail of K arrive as zeros), and are read 16 bytes of K at a time: with rows 4 words longer than a
// multiple of 16 the 8 rows of a warp's read lie in different banks.  An output's chain of multiply-adds runs over K in
// order, as in the kernel above, bit for bit.  VEC: 16-byte copies (rows and pitches that allow them); else 4 bytes at a time.
template <int BM_, int BN_, int TM_, int TN_, int BK_, int ST_, int MINB_ = 1>
struct GpShape {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, BK = BK_, ST = ST_, MINB = MINB_;
  static constexpr int WX = BN / (8 * TN), WY = BM / (4 * TM), THREADS = 32 * WX * WY;
  static constexpr int PITCH = BK + 4, STAGE = (BM + BN) * PITCH;
  static constexpr int SMEM = STAGE * ST * 4;
};

__device__ __forceinline__ void gp_copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gp_copy4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// `rows` rows of BK values from src (row pitch ld), K values in a row of which k0 .. are wanted
template <int ROWS, int BK, int PITCH, int THREADS, bool VEC>
__device__ __forceinline__ void gp_tile(float* dst, const float* __restrict__ src, int ld, int row0, int rows, int k0,
                                        int K) {
  constexpr int STEP = VEC ? 4 : 1, PER_ROW = BK / STEP, N = ROWS * PER_ROW;
#pragma unroll
  for (int e = 0; e < (N + THREADS - 1) / THREADS; ++e) {
    const int i = threadIdx.x + e * THREADS;
    if (N % THREADS != 0 && i >= N) break;
    const int r = i / PER_ROW, k = i % PER_ROW * STEP;
    const bool in = row0 + r < rows && k0 + k < K;
    const float* from = src + (in ? (size_t)(row0 + r) * ld + k0 + k : 0);
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + r * PITCH + k);
    if (VEC) gp_copy16(to, from, in ? 4 * min(4, K - k0 - k) : 0);
    else gp_copy4(to, from, in ? 4 : 0);
  }
}

template <typename S, bool VEC, typename TO>
__global__ void __launch_bounds__(S::THREADS, S::MINB)
gemm_f32_kernel(TO* __restrict__ out, int ldo, const float* __restrict__ x, int ldx, const float* __restrict__ w,
                int ldw, int M, int N, int K, float cap) {
  extern __shared__ __align__(16) float gp_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ly = lane / 16 * 2 + lane % 2, lx = lane / 2 % 8;
  const int ry = warp / S::WX * (4 * S::TM) + ly, rx = warp % S::WX * (8 * S::TN) + lx;
  const int m0 = blockIdx.y * S::BM, n0 = blockIdx.x * S::BN;
  const int steps = (K + S::BK - 1) / S::BK;
  auto fetch = [&](int s) {
    if (s < steps) {
      float* t = gp_smem + s % S::ST * S::STAGE;
      gp_tile<S::BM, S::BK, S::PITCH, S::THREADS, VEC>(t, x, ldx, m0, M, s * S::BK, K);
      gp_tile<S::BN, S::BK, S::PITCH, S::THREADS, VEC>(t + S::BM * S::PITCH, w, ldw, n0, N, s * S::BK, K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < S::ST - 1; ++s) fetch(s);
  float acc[S::TM][S::TN];
#pragma unroll
  for (int i = 0; i < S::TM; ++i)
#pragma unroll
    for (int j = 0; j < S::TN; ++j) acc[i][j] = 0.f;

  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S::ST - 2) : "memory");
    __syncthreads();               // stage s is there, and everybody is done with the stage that is fetched into next
    fetch(s + S::ST - 1);
    const float* a = gp_smem + s % S::ST * S::STAGE + ry * S::PITCH;
    const float* b = gp_smem + s % S::ST * S::STAGE + (S::BM + rx) * S::PITCH;
#pragma unroll
    for (int k = 0; k < S::BK; k += 4) {
      float4 av[S::TM], bv[S::TN];
#pragma unroll
      for (int i = 0; i < S::TM; ++i) av[i] = *(const float4*)(a + i * 4 * S::PITCH + k);
#pragma unroll
      for (int j = 0; j < S::TN; ++j) bv[j] = *(const float4*)(b + j * 8 * S::PITCH + k);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < S::TM; ++i)
#pragma unroll
          for (int j = 0; j < S::TN; ++j)
            acc[i][j] = fmaf((&av[i].x)[e], (&bv[j].x)[e], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    const int m = m0 + ry + 4 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < S::TN; ++j) {
      const int n = n0 + rx + 8 * j;
      if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(softcap_f32(acc[i][j], cap));
    }
  }
}

// The same with two outputs a multiply-add instruction (fma.rn.f32x2: each half rounds as a single fmaf does): w's tile
// lies in pairs of rows, element by element in turn, so that a pair of columns is one 64-bit operand.
template <typename S, bool VEC>
__device__ __forceinline__ void gp_pair_load(float4 (&r)[2], const float* __restrict__ w, int ldw, int n0, int N, int k0, int K, int item) {
  const int p = item / (S::BK / 4), k = k0 + item % (S::BK / 4) * 4;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int n = n0 + 2 * p + h;
    r[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n < N) {
      const float* from = w + (size_t)n * ldw + k;
      if (VEC && k + 4 <= K) r[h] = *(const float4*)from;
      else
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (k + e < K) (&r[h].x)[e] = from[e];
    }
  }
}

template <typename S, bool VEC, typename TO>
__global__ void __launch_bounds__(S::THREADS, S::MINB)
gemm_f32_pair_kernel(TO* __restrict__ out, int ldo, const float* __restrict__ x, int ldx, const float* __restrict__ w,
                     int ldw, int M, int N, int K, float cap) {
  extern __shared__ __align__(16) float gp_smem[];
  pdl_launch_dependents();
  pdl_wait();
  constexpr int A_STAGE = S::BM * S::PITCH, BP = 2 * S::BK + 4, B_STAGE = S::BN / 2 * BP;
  constexpr int ITEMS = S::BN * S::BK / 8 / S::THREADS;
  static_assert(ITEMS * 8 * S::THREADS == S::BN * S::BK, "whole items");
  float* bs = gp_smem + S::ST * A_STAGE;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ly = lane / 16 * 2 + lane % 2, lx = lane / 2 % 8;
  const int ry = warp / S::WX * (4 * S::TM) + ly, rp = warp % S::WX * (4 * S::TN) + lx;
  const int m0 = blockIdx.y * S::BM, n0 = blockIdx.x * S::BN;
  const int steps = (K + S::BK - 1) / S::BK;
  auto fetch = [&](int s) {
    if (s < steps) gp_tile<S::BM, S::BK, S::PITCH, S::THREADS, VEC>(gp_smem + s % S::ST * A_STAGE, x, ldx, m0, M, s * S::BK, K);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float4 held[ITEMS][2];
  auto load = [&](int s) {
#pragma unroll
    for (int e = 0; e < ITEMS; ++e) gp_pair_load<S, VEC>(held[e], w, ldw, n0, N, s * S::BK, K, threadIdx.x + e * S::THREADS);
  };
  auto store = [&](int s) {
#pragma unroll
    for (int e = 0; e < ITEMS; ++e) {
      const int item = threadIdx.x + e * S::THREADS;
      float4* to = (float4*)(bs + s % 2 * B_STAGE + item / (S::BK / 4) * BP + item % (S::BK / 4) * 8);
      to[0] = make_float4(held[e][0].x, held[e][1].x, held[e][0].y, held[e][1].y);
      to[1] = make_float4(held[e][0].z, held[e][1].z, held[e][0].w, held[e][1].w);
    }
  };
  load(0);
#pragma unroll
  for (int s = 0; s < S::ST - 1; ++s) fetch(s);
  store(0);
  unsigned long long acc[S::TM][S::TN / 2];
#pragma unroll
  for (int i = 0; i < S::TM; ++i)
#pragma unroll
    for (int j = 0; j < S::TN / 2; ++j) acc[i][j] = 0ull;

  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S::ST - 2) : "memory");
    __syncthreads();               // stage s is there, and everybody is done with the stages that are filled next
    fetch(s + S::ST - 1);
    if (s + 1 < steps) load(s + 1);
    const float* a = gp_smem + s % S::ST * A_STAGE + ry * S::PITCH;
    const float* b = bs + s % 2 * B_STAGE + rp * BP;
#pragma unroll
    for (int k = 0; k < S::BK; k += 4) {
      float4 av[S::TM];
      ulonglong2 bv[S::TN / 2][2];
#pragma unroll
      for (int i = 0; i < S::TM; ++i) av[i] = *(const float4*)(a + i * 4 * S::PITCH + k);
#pragma unroll
      for (int j = 0; j < S::TN / 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) bv[j][h] = *(const ulonglong2*)(b + j * 8 * BP + 2 * k + 4 * h);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < S::TM; ++i) {
          unsigned long long aa;
          asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "r"(__float_as_uint((&av[i].x)[e])));
#pragma unroll
          for (int j = 0; j < S::TN / 2; ++j) {
            const unsigned long long bb = e & 1 ? bv[j][e / 2].y : bv[j][e / 2].x;
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(bb));
          }
        }
    }
    if (s + 1 < steps) store(s + 1);
  }
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    const int m = m0 + ry + 4 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < S::TN / 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = n0 + 2 * (rp + 8 * j) + h;
        const float v = __uint_as_float((unsigned)(acc[i][j] >> (32 * h)));
        if (n < N) out[(size_t)m * ldo + n] = from_f32<TO>(softcap_f32(v, cap));
      }
  }
}

template <typename S, bool VEC, typename TO>
static int gp_pair_launch(TO* out, int ldo, const float* x, int ldx, const float* w, int ldw, int M, int N, int K, float cap,
                     cudaStream_t stream) {
  static bool sized[AF_MAX_DEVICES];
  constexpr int SMEM = (S::ST * S::BM * S::PITCH + S::BN * (2 * S::BK + 4)) * 4;
  if (af_first_on_device(sized, af_current_device())) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_pair_kernel<S, VEC, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return af_fail((int)e, "af_gemm_plain: shared memory: %s", cudaGetErrorString(e));
  }
  const dim3 grid((N + S::BN - 1) / S::BN, (M + S::BM - 1) / S::BM);
  AF_REQUIRE(grid.y <= 65535, "af_gemm_plain: M %d too large", M);
  af_launch(gemm_f32_pair_kernel<S, VEC, TO>, grid, dim3(S::THREADS), SMEM, stream, out, ldo, x, ldx, w, ldw, M, N, K, cap);
  AF_CHECK_LAUNCH("af_gemm_plain");
}

template <typename S, bool VEC, typename TO>
static int gp_launch(TO* out, int ldo, const float* x, int ldx, const float* w, int ldw, int M, int N, int K, float cap,
                     cudaStream_t stream) {
  static bool sized[AF_MAX_DEVICES];
  if (af_first_on_device(sized, af_current_device())) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<S, VEC, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
    if (e != cudaSuccess) return af_fail((int)e, "af_gemm_plain: shared memory: %s", cudaGetErrorString(e));
  }
  const dim3 grid((N + S::BN - 1) / S::BN, (M + S::BM - 1) / S::BM);
  AF_REQUIRE(grid.y <= 65535, "af_gemm_plain: M %d too large", M);
  af_launch(gemm_f32_kernel<S, VEC, TO>, grid, dim3(S::THREADS), S::SMEM, stream, out, ldo, x, ldx, w, ldw, M, N, K, cap);
  AF_CHECK_LAUNCH("af_gemm_plain");
}

// Which shape.  A chain of K multiply-adds is the least an output takes, so a product of few tiles is bound by that chain
// and what stands beside it, and wants as many warps as it can get; one of many tiles by the reads from shared memory, and
// wants large tiles a thread.  Measured (us; N x K: 2304 x 9216, 2304 x 2048, 4096 x 2304, 18432 x 2304):
//   up to 4 rows, blocks of 16 columns and 7 stages in flight 45 / 10 / 14 / 46, of 32 columns 54 / 14 / 18 / 46: the
//     narrow ones while they all run at once (two an SM), else the wide ones, which read x half as often;
//   up to 8 rows 49 / 13 / 27 / 71; up to 16 rows 88 / 18 / 28 / 97 against 163 / 39 / 45 / 107 for 32 x 32 tiles, which
//     are better from two blocks of 16 x 16 an SM on (32 rows: 101 / 25 / 52 / 195 against 165 / 39 / 45 / 109);
//   301 rows: 32 x 32 tiles 431 / 99 / 179 / 695, 32 x 64 tiles 556 / 126 / 178 / 687 (from three and a half an SM on they
//     are the better ones), 64 x 128 tiles of pairs 773 / 170 / 320 / 581 (from four and a half an SM on: 44 TFLOP/s, where the
//     64 rows are not mostly empty: a tile takes 1.66 times as long as one of 32 x 64 for the same columns).
// So many rows come with the heads of decode steps (256000 x 2304: 17 to 32 rows 954 in tiles of 32 x 64 against 1,561, 33 to 64 rows
// 1,870 against 1,565) and with prompts that the tensor cores do not take (18432 x 2302, 301 rows: 827 / 647; 1000 x 1000, 8,192
// rows: 453 / 361).
// The kernel that all of these replace, 64 x 64 tiles fetched and then multiplied, took 1,297 us at 301 x 18432 x 2304
// (20 TFLOP/s) and 230 to 1,000 us for a few rows.
template <bool VEC, typename TO>
static int gp_choose(TO* out, int ldo, const float* x, int ldx, const float* w, int ldw, int M, int N, int K, float cap,
                     cudaStream_t stream) {
  const long long sms = af_sm_count();
  AF_REQUIRE(sms > 0, "af_gemm_plain: no device");
  auto tiles = [&](long long bm, long long bn) { return ((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
#define GP_ARGS out, ldo, x, ldx, w, ldw, M, N, K, cap, stream
  if (M <= 4) {
    if (tiles(4, 16) <= 2 * sms) return gp_launch<GpShape<4, 16, 1, 1, 128, 8>, VEC, TO>(GP_ARGS);
    return gp_launch<GpShape<4, 32, 1, 1, 64, 6>, VEC, TO>(GP_ARGS);
  }
  if (M <= 8) return gp_launch<GpShape<8, 16, 1, 1, 64, 4>, VEC, TO>(GP_ARGS);
  if (M <= 16 || tiles(16, 16) <= 2 * sms) return gp_launch<GpShape<16, 16, 2, 1, 128, 5>, VEC, TO>(GP_ARGS);
  if (2 * tiles(64, 128) >= 9 * sms && 5 * ((M + 63) / 64) <= 3 * ((M + 31) / 32)) return gp_pair_launch<GpShape<64, 128, 8, 8, 16, 3, 3>, VEC, TO>(GP_ARGS);
  if (2 * tiles(32, 64) >= 7 * sms) return gp_launch<GpShape<32, 64, 4, 4, 32, 4>, VEC, TO>(GP_ARGS);
  return gp_launch<GpShape<32, 32, 4, 4, 32, 4>, VEC, TO>(GP_ARGS);
#undef GP_ARGS
}

// `cap` > 0 applies cap * tanh(v / cap) to every output (the head's softcap).
AF_EXPORT int af_gemm_plain(void* out, int out_dtype, int ldo, const void* x, int ldx, const void* w,
                            int ldw, int dtype, int M, int N, int K, float cap, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  AF_REQUIRE(M > 0 && N > 0 && K > 0, "af_gemm_plain: bad sizes %d %d %d", M, N, K);
  if (dtype == AF_F32) {
    const bool vec = ldx % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
    AF_DISPATCH_DTYPE(out_dtype, TO,
                      return vec ? gp_choose<true, TO>((TO*)out, ldo, (const float*)x, ldx, (const float*)w, ldw, M, N, K, cap, stream)
                                 : gp_choose<false, TO>((TO*)out, ldo, (const float*)x, ldx, (const float*)w, ldw, M, N, K, cap, stream));
  }
  dim3 grid((N + GP_BN - 1) / GP_BN, (M + GP_BM - 1) / GP_BM);
  AF_REQUIRE(grid.y <= 65535, "af_gemm_plain: M %d too large", M);
  AF_REQUIRE(dtype == AF_BF16, "unsupported dtype code %d", dtype);
  AF_DISPATCH_DTYPE(out_dtype, TO,
                    af_launch(gemm_plain_kernel<__nv_bfloat16, TO>, dim3(grid), dim3(256), 0, stream, (TO*)out, ldo,
                              (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, ldw, M, N, K, cap));
  AF_CHECK_LAUNCH("af_gemm_plain");
}
