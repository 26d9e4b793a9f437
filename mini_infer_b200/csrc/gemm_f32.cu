// True 32-bit matrix product on CUDA cores:  C[M,N] = A[M,K] * W[N,K]^T
// (both operands K-contiguous, as linear layers store them).  No tensor cores, no
// reduced-precision mode.  Every output element is accumulated over k = 0..K-1 in that
// order with fused multiply-adds, whatever tile it falls in and whatever kernel and tile shape are
// chosen, so a row's result does not depend on which other rows share the call.
//
//   gemm_f32_rows_kernel   up to 32 rows (decode): bound by one reading of W
//   gemm_f32_tile_kernel   more rows, or operands without 16-byte rows: bound by the fused multiply-adds
#include "common.cuh"

MI_DEFINE_ERROR_API()

// ------------------------------------------------------------------------------------------
// Few rows.  A block owns 16 columns of the result (rows of W) and streams them, with the rows of A beside
// them, through a ring of shared-memory stages filled by cp.async; 16 x 4 threads, RM rows of A each.  One element's
// sum is a chain of K multiply-adds (4 cycles each: 4.3 us at K = 2048), so the columns have to be spread wide, 128
// blocks for N = 2048, and the ring deep.  The first stages of W are asked for before the wait for the kernel before.
// ------------------------------------------------------------------------------------------
#define RB_COLS 16
#define RB_K 64
#define RB_PITCH (RB_K + 4)      // floats per staged row: eight rows' 16-byte pieces touch every bank once
#define RB_STAGES 8
#define RB_MAX_ROWS 32

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = in ? 16 : 0;       // nothing read, zeros written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int RM>
__global__ void __launch_bounds__(64) gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                           float* __restrict__ C, int M, int N, int K, int lda, int ldw,
                                                           int ldc) {
  extern __shared__ __align__(16) float rsm[];
  constexpr int ROWS = 4 * RM;
  constexpr int STAGE = (RB_COLS + ROWS) * RB_PITCH;
  mi_pdl_launch_dependents();
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int n0 = blockIdx.x * RB_COLS;
  const int chunks = (K + RB_K - 1) / RB_K;
  auto load_w = [&](int kc) {
    float* dst = rsm + (kc % RB_STAGES) * STAGE;
    for (int i = tid; i < RB_COLS * (RB_K / 4); i += 64) {
      const int r = i / (RB_K / 4), c = (i % (RB_K / 4)) * 4, k = kc * RB_K + c;
      const bool in = n0 + r < N && k < K;
      cp_async16(dst + r * RB_PITCH + c, in ? W + (size_t)(n0 + r) * ldw + k : W, in);
    }
  };
  auto load_a = [&](int kc) {
    float* dst = rsm + (kc % RB_STAGES) * STAGE + RB_COLS * RB_PITCH;
    for (int i = tid; i < M * (RB_K / 4); i += 64) {
      const int r = i / (RB_K / 4), c = (i % (RB_K / 4)) * 4, k = kc * RB_K + c;
      const bool in = k < K;
      cp_async16(dst + r * RB_PITCH + c, in ? A + (size_t)r * lda + k : A, in);
    }
  };
  const int ahead = min(RB_STAGES - 1, chunks);
  for (int s = 0; s < ahead; ++s) load_w(s);      // weights depend on no kernel before this one
  mi_pdl_wait();
  for (int s = 0; s < RB_STAGES - 1; ++s) {
    if (s < chunks) load_a(s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");   // (W's first stages ride in the first group)
  }
  float acc[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) acc[i] = 0.f;
  for (int kc = 0; kc < chunks; ++kc) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(RB_STAGES - 2) : "memory");
    __syncthreads();               // stage kc is there, and stage kc - 1 is consumed
    const int next = kc + RB_STAGES - 1;
    if (next < chunks) {
      load_w(next);
      load_a(next);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* ws = rsm + (kc % RB_STAGES) * STAGE + tx * RB_PITCH;
    const float* as = rsm + (kc % RB_STAGES) * STAGE + (RB_COLS + ty * RM) * RB_PITCH;
#pragma unroll 8
    for (int k = 0; k < RB_K; k += 4) {
      const float4 w = *reinterpret_cast<const float4*>(ws + k);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(as + i * RB_PITCH + k);
        acc[i] = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, acc[i]))));
      }
    }
  }
  const int n = n0 + tx;
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = ty * RM + i;
    if (m < M && n < N) C[(size_t)m * ldc + n] = acc[i];
  }
}

// ------------------------------------------------------------------------------------------
// Many rows.  A BM x BN tile per block, TM x TN results per thread (two groups of four rows and of four columns,
// half a tile apart), k in steps of 16 through two shared-memory buffers: the next step's pieces come from global memory into
// registers while this one is multiplied.  The multiply-adds are the two-wide form, two columns at a time.
// ------------------------------------------------------------------------------------------
#define TB_K 16
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int lda, int ldw, int ldc) {
  mi_pdl_enter();   // inputs come from the kernels before this one
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr int GM = TM / 4, GN = TN / 4;                 // groups of four
  constexpr int PA = BM * (TB_K / 4) / THREADS, PW = BN * (TB_K / 4) / THREADS;   // 16-byte pieces per thread and step
  static_assert(PA * THREADS == BM * (TB_K / 4) && PW * THREADS == BN * (TB_K / 4), "whole pieces per thread");
  __shared__ __align__(16) float As[2][TB_K][BM + 4];
  __shared__ __align__(16) float Ws[2][TB_K][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  auto piece = [&](const float* p, int row, int rows, int ld, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= rows) return v;
    const float* src = p + (size_t)row * ld + k;
    if (VEC) {           // K % 4 == 0 and 16-byte rows
      if (k < K) v = *reinterpret_cast<const float4*>(src);
    } else {
      if (k < K) v.x = src[0];
      if (k + 1 < K) v.y = src[1];
      if (k + 2 < K) v.z = src[2];
      if (k + 3 < K) v.w = src[3];
    }
    return v;
  };
  float4 pa[PA], pw[PW];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int idx = tid + i * THREADS;
      pa[i] = piece(A, m0 + idx / (TB_K / 4), M, lda, k0 + (idx % (TB_K / 4)) * 4);
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int idx = tid + i * THREADS;
      pw[i] = piece(W, n0 + idx / (TB_K / 4), N, ldw, k0 + (idx % (TB_K / 4)) * 4);
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int idx = tid + i * THREADS, r = idx / (TB_K / 4), c = (idx % (TB_K / 4)) * 4;
      As[buf][c][r] = pa[i].x; As[buf][c + 1][r] = pa[i].y; As[buf][c + 2][r] = pa[i].z; As[buf][c + 3][r] = pa[i].w;
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int idx = tid + i * THREADS, r = idx / (TB_K / 4), c = (idx % (TB_K / 4)) * 4;
      Ws[buf][c][r] = pw[i].x; Ws[buf][c + 1][r] = pw[i].y; Ws[buf][c + 2][r] = pw[i].z; Ws[buf][c + 3][r] = pw[i].w;
    }
  };

  uint64_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;

  fetch(0);
  stage(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += TB_K) {
    const bool more = k0 + TB_K < K;
    if (more) fetch(k0 + TB_K);
#pragma unroll
    for (int k = 0; k < TB_K; ++k) {
      uint64_t w[TN / 2];
      float a[TM];
#pragma unroll
      for (int j = 0; j < GN; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[buf][k][j * (BN / GN) + tx * 4]);
        w[2 * j] = v.x;
        w[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < GM; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(&As[buf][k][i * (BM / GM) + ty * 4]);
        a[4 * i] = v.x; a[4 * i + 1] = v.y; a[4 * i + 2] = v.z; a[4 * i + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const uint64_t aa = pack2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, w[j]);
      }
    }
    if (more) stage(buf ^ 1);      // (that buffer was last read before the barrier of the step before)
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i / 4) * (BM / GM) + ty * 4 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const int n = n0 + (j / 2) * (BN / GN) + tx * 4 + (j & 1) * 2;
      float v0, v1;
      unpack2(acc[i][j], v0, v1);
      if (n < N) C[(size_t)m * ldc + n] = v0;
      if (n + 1 < N) C[(size_t)m * ldc + n + 1] = v1;
    }
  }
}

template <int BM, int BN, int TM, int TN>
static void launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                        int ldc, bool vec, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  constexpr int THREADS = (BM / TM) * (BN / TN);
  if (vec)
    MI_LAUNCH((gemm_f32_tile_kernel<BM, BN, TM, TN, true>), grid, THREADS, 0, stream, A, W, C, M, N, K, lda, ldw, ldc);
  else
    MI_LAUNCH((gemm_f32_tile_kernel<BM, BN, TM, TN, false>), grid, THREADS, 0, stream, A, W, C, M, N, K, lda, ldw, ldc);
}

template <int RM>
static cudaError_t launch_rows(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                               cudaStream_t stream) {
  const size_t smem = (size_t)RB_STAGES * (RB_COLS + 4 * RM) * RB_PITCH * sizeof(float);
  auto kern = gemm_f32_rows_kernel<RM>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return MI_LAUNCH(kern, (N + RB_COLS - 1) / RB_COLS, 64, smem, stream, A, W, C, M, N, K, lda, ldw, ldc);
}

// The time of a tile shape in units of multiply-adds: waves over the SMs times the tile, the smaller shapes marked
// down for what they read from shared memory per multiply-add.
static double tile_time(int M, int N, int bm, int bn, double weight) {
  const long long tiles = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
  return (double)((tiles + 147) / 148) * bm * bn * weight;
}

// Zero-padded K tails add exact zeros at the end of the sum, so they do not change it.
extern "C" int mi_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                           int ldw, int ldc, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) MI_REFUSE("gemm_f32: K must be positive, got %d", K);
  if (lda < K || ldw < K || ldc < N) MI_REFUSE("gemm_f32: leading dimensions too small");
  if ((M + 15) / 16 > 65535) MI_REFUSE("gemm_f32: too many rows (%d)", M);
  const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && mi_aligned(A, 16) && mi_aligned(W, 16);
  if (vec && M <= RB_MAX_ROWS) {
    const cudaError_t e = M <= 4    ? launch_rows<1>(A, W, C, M, N, K, lda, ldw, ldc, stream)
                          : M <= 8  ? launch_rows<2>(A, W, C, M, N, K, lda, ldw, ldc, stream)
                          : M <= 16 ? launch_rows<4>(A, W, C, M, N, K, lda, ldw, ldc, stream)
                                    : launch_rows<8>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (e != cudaSuccess) return (int)e;
    MI_RETURN_LAUNCH_STATUS();
  }
  const double big = tile_time(M, N, 128, 128, 1.0), wide = tile_time(M, N, 64, 128, 1.05),
               mid = tile_time(M, N, 64, 64, 1.25), small = tile_time(M, N, 32, 64, 1.6);
  if (big <= wide && big <= mid && big <= small)
    launch_tile<128, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
  else if (wide <= mid && wide <= small)
    launch_tile<64, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
  else if (mid <= small)
    launch_tile<64, 64, 4, 8>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
  else
    launch_tile<32, 64, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, stream);
  MI_RETURN_LAUNCH_STATUS();
}
