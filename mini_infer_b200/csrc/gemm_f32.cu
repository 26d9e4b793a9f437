// True 32-bit matrix product on CUDA cores:  C[M,N] = A[M,K] * W[N,K]^T
// (both operands K-contiguous, as linear layers store them).  No tensor cores, no
// reduced-precision mode.  Every output element is the sum, in this order, of four parts of k of equal length (a
// multiple of 32, the last one shorter), each accumulated from its first k on with fused multiply-adds, whatever kernel and
// tile it falls in, so a row's result does not depend on which other rows share the call.
//
//   gemm_f32_stream_kernel up to 4 rows of a wide result (decode): bound by one reading of W
//   gemm_f32_rows_kernel   up to 32 rows
//   gemm_f32_tile_kernel   more rows: bound by the fused multiply-adds
//   gemm_f32_any_kernel    operands without 16-byte rows
#include "bulk_copy.cuh"

MI_DEFINE_ERROR_API()
MI_DEFINE_STATUS_API(mi_gemm_f32_status)

#define PARTS 4
// where part p of k begins (a multiple of 32, so that a staged piece lies in one part)
__host__ __device__ __forceinline__ int part_begin(int K, int p) {
  const int len = ((K + PARTS - 1) / PARTS + 31) / 32 * 32;
  const int at = p * len;
  return at < K ? at : K;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = in ? 16 : 0;       // nothing read, zeros written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}
// the 64 threads of a part among themselves
__device__ __forceinline__ void part_barrier(int part) { asm volatile("bar.sync %0, 64;\n" ::"r"(part + 1) : "memory"); }

// ------------------------------------------------------------------------------------------
// Up to 4 rows.  What bounds it: the stream of W.  A block per SM owns N / 148 columns of the result (rows of W) over the
// whole of k, in tiles of up to 32 columns, a lane each; warps 0 to 3 have a part of k each, and warp 4 feeds them by TMA,
// 32 k of every part per stage, through a ring that is full of W before the wait for the kernel before and does not run
// empty between tiles.  Two rows, 32000 x 2048: 67 us in blocks of 16 columns whose ring starts anew with
// every block (the kernel below), 50 here (41 of bytes); a pass of two prompts of 131 tokens and
// four steps of a four-layer model of that width 3.58 -> 3.31 ms.  Behind the stream stand the reads of A from shared memory, RM of them beside
// one of W.
// ------------------------------------------------------------------------------------------
#define ST_K 32                     // k per part and stage: 128 bytes, one swizzle row
#define ST_COLS 32                  // most columns per tile
#define ST_MAX_ROWS 4
#define ST_MAX_STAGES 16
#define ST_THREADS (32 * (PARTS + 1))
#define ST_BUDGET (200 * 1024)

// LIMIT: polls of a copy's barrier before a warp gives up (0 in a test's instance).
template <int RM, int LIMIT>
__global__ void __launch_bounds__(ST_THREADS, 1)
gemm_f32_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, float* C,
                       int M, int N, int K, int ldc, int cols, int n_tiles, int stages, int w_constant) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[ST_MAX_STAGES], empty[ST_MAX_STAGES];
  __shared__ float sums[2][PARTS][RM][ST_COLS];
  __shared__ int give_up;
  // per stage and part a box of W (cols rows of 128 bytes) and one of A (M rows), each from a multiple of 1024 on
  const uint32_t w_bytes = (uint32_t)cols * ST_K * 4, a_bytes = (uint32_t)M * ST_K * 4;
  const uint32_t w_box = (w_bytes + 1023) & ~1023u, part_bytes = w_box + 1024, stage_bytes = PARTS * part_bytes;
  mi_pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = blockIdx.x * cols * n_tiles;
  const int tiles = min(n_tiles, (N - first + cols - 1) / cols);
  const int chunks = (part_begin(K, 1) + ST_K - 1) / ST_K;      // of the longest part; shorter ones read zeros from where they end
  volatile int* gu = &give_up;

  if (warp == PARTS) {
    if (lane < stages) {
      mbar_init(&full[lane], 2 * PARTS);       // the boxes of W and A
      mbar_init(&empty[lane], PARTS);
    }
    if (lane == 0) give_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    __syncwarp();
    asm volatile("bar.arrive 1, 160;\n" ::: "memory");
    const int units = tiles * chunks, first_turn = min(stages, units);
    const uint64_t policy = l2_policy_evict_first(), policy_a = l2_policy_evict_normal();
    // lane p: W's box of part p; lane PARTS + p: A's.  A chunk behind the end of its part is asked for at K (a multiple of 4
    // here): zeros.
    const int part = lane & (PARTS - 1), k0 = part_begin(K, part), k1 = part_begin(K, part + 1);
    auto load = [&](bool of_w, int st, int u) {
      const int tile = u / chunks, k = k0 + (u - tile * chunks) * ST_K, x = k < k1 ? k : K;
      unsigned char* dst = smem + (size_t)st * stage_bytes + part * part_bytes + (of_w ? 0u : w_box);
      mbar_expect_tx(&full[st], of_w ? w_bytes : a_bytes);
      tma_load_2d_hint(dst, of_w ? &map_w : &map_a, x, of_w ? first + tile * cols : 0, &full[st], of_w ? policy : policy_a);
    };
    if (!w_constant) mi_pdl_wait();
    if (lane < PARTS)
      for (int u = 0; u < first_turn; ++u) load(true, u, u);
    if (w_constant) mi_pdl_wait();
    if (lane >= PARTS && lane < 2 * PARTS)
      for (int u = 0; u < first_turn; ++u) load(false, u, u);
    __syncwarp();
    if (lane < 2 * PARTS) {
      int st = 0, round = 0;
      for (int u = first_turn; u < units; ++u) {
        if (!mbar_wait(&empty[st], round & 1, gu)) break;
        load(lane < PARTS, st, u);
        if (++st == stages) { st = 0; ++round; }
      }
    }
    return;
  }

  asm volatile("bar.sync 1, 160;\n" ::: "memory");      // the barriers are initialised
  mi_pdl_wait();                                        // the kernels before may read C
  const int row = min(lane, cols - 1), sw = row & 7;
  int st = 0, round = 0;
  // After a wait that ran out (ok) a warp computes no more but goes on waiting for every copy and handing its stage on, so that
  // none is under way when the block leaves; a copy that does not come then either (there) ends that too.
  bool ok = true, there = true;
  for (int tile = 0; tile < tiles; ++tile) {
    float acc[RM];
#pragma unroll
    for (int i = 0; i < RM; ++i) acc[i] = 0.f;
    for (int kc = 0; kc < chunks; ++kc) {
      if (there && !mbar_wait(&full[st], round & 1, gu, LIMIT)) {
        ok = false;
        there = mbar_drain(&full[st], round & 1);
      }
      if (ok) {
        const unsigned char* ws = smem + (size_t)st * stage_bytes + warp * part_bytes + row * 128;
        const unsigned char* as = smem + (size_t)st * stage_bytes + warp * part_bytes + w_box;
        float4 w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) w[c] = *reinterpret_cast<const float4*>(ws + ((c ^ sw) << 4));
#pragma unroll
        for (int c = 0; c < 8; ++c) {
#pragma unroll
          for (int i = 0; i < RM; ++i) {      // (rows beyond M: whatever lies behind the box; nothing stores them)
            const float4 a = *reinterpret_cast<const float4*>(as + i * 128 + ((c ^ i) << 4));
            acc[i] = fmaf(a.w, w[c].w, fmaf(a.z, w[c].z, fmaf(a.y, w[c].y, fmaf(a.x, w[c].x, acc[i]))));
          }
        }
      }
      __syncwarp();
      if (lane == 0 && there) mbar_arrive(&empty[st]);
      if (++st == stages) { st = 0; ++round; }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) sums[tile & 1][warp][i][lane] = acc[i];
    asm volatile("bar.sync 2, 128;\n" ::: "memory");     // (the next tile writes the other half)
    const int n = first + tile * cols + lane;
    if (ok && lane < cols && n < N) {
      for (int m = warp; m < M; m += PARTS) {
        float v = sums[tile & 1][0][m][lane];
#pragma unroll
        for (int p = 1; p < PARTS; ++p) v += sums[tile & 1][p][m][lane];
        C[(size_t)m * ldc + n] = v;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// Few rows.  A block owns 16 columns of the result (rows of W); 64 threads per part of k stream their part of
// them, with the rows of A beside it, through a ring of stages filled by cp.async, 16 x 4 threads, RM rows of A each.  One
// element's sum is a chain of K / 4 multiply-adds (4 cycles each: 1.1 us at K = 2048).  2 x 3072 x 2048 behind one another: 19 us with one part (a chain four times
// as long behind a ring four times as narrow), 322 us with 128 columns per block and no ring; 3.9 us of bytes.
// w_constant: no kernel before this one writes W, so that its first stages are asked for before the wait for that kernel.
// ------------------------------------------------------------------------------------------
#define RB_COLS 16
#define RB_K 32
#define RB_PITCH (RB_K + 4)      // floats per staged row: eight rows' 16-byte pieces touch every bank once
// Rows and tiles, us: N x K = 3072 x 2048 with 1 row 11 and 40, 16 18 and 36, 17 33 and 37, 32 38 and 37; 2048 x 3072 16 rows 25
// and 52, 32 29 and 53; 6144 x 2048 16 28 and 58, 17 49 and 57, 32 56 and 58; 32000 x 2048 8 81 and 121, 16 115 and 121, 17
// 222 and 121, 32 256 and 123 (a block's 16 columns then come round fourteen times, each with all rows).
#define RB_MAX_ROWS 32
#define RB_MAX_COLS 8192          // above 16 rows

template <int RM, int STAGES>
__global__ void __launch_bounds__(64 * PARTS) gemm_f32_rows_kernel(const float* A, const float* __restrict__ W,
                                                                   float* C, int M, int N, int K, int lda,
                                                                   int ldw, int ldc, int w_constant) {
  extern __shared__ __align__(16) float rsm[];
  constexpr int ROWS = 4 * RM;
  constexpr int STAGE = (RB_COLS + ROWS) * RB_PITCH;
  __shared__ float sums[PARTS - 1][ROWS][RB_COLS];
  mi_pdl_launch_dependents();
  const int part = threadIdx.x >> 6, tid = threadIdx.x & 63, tx = tid & 15, ty = tid >> 4;
  const int n0 = blockIdx.x * RB_COLS;
  const int k_begin = part_begin(K, part), k_end = part_begin(K, part + 1);
  const int chunks = (k_end - k_begin + RB_K - 1) / RB_K;
  float* ring = rsm + part * STAGES * STAGE;
  auto load_w = [&](int kc) {
    float* dst = ring + (kc % STAGES) * STAGE;
#pragma unroll
    for (int i = tid; i < RB_COLS * (RB_K / 4); i += 64) {
      const int r = i / (RB_K / 4), c = (i % (RB_K / 4)) * 4, k = k_begin + kc * RB_K + c;
      const bool in = n0 + r < N && k < k_end;
      cp_async16(dst + r * RB_PITCH + c, in ? W + (size_t)(n0 + r) * ldw + k : W, in);
    }
  };
  auto load_a = [&](int kc) {
    float* dst = ring + (kc % STAGES) * STAGE + RB_COLS * RB_PITCH;
    for (int i = tid; i < M * (RB_K / 4); i += 64) {
      const int r = i / (RB_K / 4), c = (i % (RB_K / 4)) * 4, k = k_begin + kc * RB_K + c;
      const bool in = k < k_end;
      cp_async16(dst + r * RB_PITCH + c, in ? A + (size_t)r * lda + k : A, in);
    }
  };
  const int ahead = min(STAGES - 1, chunks);
  if (!w_constant) mi_pdl_wait();
  for (int s = 0; s < ahead; ++s) load_w(s);
  if (w_constant) mi_pdl_wait();
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < chunks) load_a(s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");   // (W's first stages ride in the first group)
  }
  float acc[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) acc[i] = 0.f;
  for (int kc = 0; kc < chunks; ++kc) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    part_barrier(part);            // stage kc is there, and stage kc - 1 is consumed
    const int next = kc + STAGES - 1;
    if (next < chunks) {
      load_w(next);
      load_a(next);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* ws = ring + (kc % STAGES) * STAGE + tx * RB_PITCH;
    const float* as = ring + (kc % STAGES) * STAGE + (RB_COLS + ty * RM) * RB_PITCH;
    // a batch's pieces are read before its multiply-adds (each piece's chain alone would wait for it)
    constexpr int BATCH = RM <= 2 ? 8 : RM <= 4 ? 4 : 2;
#pragma unroll
    for (int k0 = 0; k0 < RB_K; k0 += 4 * BATCH) {
      float4 w[BATCH], a[BATCH][RM];
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        w[j] = *reinterpret_cast<const float4*>(ws + k0 + 4 * j);
#pragma unroll
        for (int i = 0; i < RM; ++i) a[j][i] = *reinterpret_cast<const float4*>(as + i * RB_PITCH + k0 + 4 * j);
      }
#pragma unroll
      for (int j = 0; j < BATCH; ++j)
#pragma unroll
        for (int i = 0; i < RM; ++i)
          acc[i] = fmaf(a[j][i].w, w[j].w, fmaf(a[j][i].z, w[j].z, fmaf(a[j][i].y, w[j].y, fmaf(a[j][i].x, w[j].x, acc[i]))));
    }
  }
  if (part) {
#pragma unroll
    for (int i = 0; i < RM; ++i) sums[part - 1][ty * RM + i][tx] = acc[i];
  }
  __syncthreads();
  if (part) return;
  const int n = n0 + tx;
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = ty * RM + i;
    float v = acc[i];
#pragma unroll
    for (int p = 0; p < PARTS - 1; ++p) v += sums[p][m][tx];
    if (m < M && n < N) C[(size_t)m * ldc + n] = v;
  }
}

// ------------------------------------------------------------------------------------------
// More rows.  An 8 TM x 64 tile per block and part of k: 64 threads per part, 8 x 8, TM x 8 results each (rows and
// columns 8 apart, so that a warp's reads of one operand are at most 128 different bytes), k in steps of 32 through two
// stages filled by cp.async, both operands as they lie in memory: a thread reads four k of its rows and columns.  The parts
// bring four times the warps of a tile to an SM, which a product of a few hundred rows needs: with one part a step of 16 k took
// 1400 cycles, most of it waiting (262 x 2048 x 2048: 148 us, now 63; 31 us of multiply-adds; 1024 x 6144 x 2048: 623 us, 358 of
// multiply-adds).  TM = 4: two blocks per SM; 2, 6 and 8 take 91, 94 and 114 us for the first and 913, 690 and 648 for the second.
// ------------------------------------------------------------------------------------------
#define TB_K 32
#define TB_PITCH (TB_K + 4)
#define TB_STAGES 2
#define TB_N 64

template <int TM>
__global__ void __launch_bounds__(64 * PARTS) gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                   float* __restrict__ C, int M, int N, int K, int lda,
                                                                   int ldw, int ldc) {
  extern __shared__ __align__(16) float tsm[];
  constexpr int BM = 8 * TM, STAGE = (BM + TB_N) * TB_PITCH;
  mi_pdl_enter();
  const int part = threadIdx.x >> 6, tid = threadIdx.x & 63, tx = tid & 7, ty = tid >> 3;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * TB_N;
  const int k_begin = part_begin(K, part), k_end = part_begin(K, part + 1);
  const int chunks = (k_end - k_begin + TB_K - 1) / TB_K;
  float* ring = tsm + part * TB_STAGES * STAGE;
  // this thread copies rows r0, r0 + 8, ... of A and of W, the four k from c on
  const int r0 = tid >> 3, c = (tid & 7) * 4;
  auto load = [&](int kc) {
    float* dst = ring + (kc & 1) * STAGE + r0 * TB_PITCH + c;
    const int k = k_begin + kc * TB_K + c;
    const bool k_in = k < k_end;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const bool in = k_in && m0 + r0 + 8 * i < M;
      cp_async16(dst + 8 * i * TB_PITCH, in ? A + (size_t)(m0 + r0 + 8 * i) * lda + k : A, in);
    }
#pragma unroll
    for (int j = 0; j < TB_N / 8; ++j) {
      const bool in = k_in && n0 + r0 + 8 * j < N;
      cp_async16(dst + (BM + 8 * j) * TB_PITCH, in ? W + (size_t)(n0 + r0 + 8 * j) * ldw + k : W, in);
    }
  };
  if (chunks > 0) load(0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  float acc[TM][8];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  for (int kc = 0; kc < chunks; ++kc) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    part_barrier(part);            // stage kc is there, and stage kc - 1 is consumed
    if (kc + 1 < chunks) load(kc + 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* as = ring + (kc & 1) * STAGE + ty * TB_PITCH;
    const float* ws = ring + (kc & 1) * STAGE + (BM + tx) * TB_PITCH;
#pragma unroll
    for (int k = 0; k < TB_K; k += 4) {
      float4 a[TM], w[8];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + 8 * i * TB_PITCH + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const float4*>(ws + 8 * j * TB_PITCH + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          acc[i][j] = fmaf(a[i].w, w[j].w, fmaf(a[i].z, w[j].z, fmaf(a[i].y, w[j].y, fmaf(a[i].x, w[j].x, acc[i][j]))));
    }
  }
  // the parts' sums, in the order of the parts, through the rings' memory
  __syncthreads();
  float* sums = tsm;               // [PARTS][BM][TB_N]
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sums[(part * BM + ty + 8 * i) * TB_N + tx + 8 * j] = acc[i][j];
  __syncthreads();
  for (int i = threadIdx.x; i < BM * TB_N; i += 64 * PARTS) {
    const int m = m0 + i / TB_N, n = n0 + i % TB_N;
    float v = sums[i];
#pragma unroll
    for (int p = 1; p < PARTS; ++p) v += sums[p * BM * TB_N + i];
    if (m < M && n < N) C[(size_t)m * ldc + n] = v;
  }
}

// ------------------------------------------------------------------------------------------
// Operands of any size and alignment: element by element through one stage, the parts one after the other.
// ------------------------------------------------------------------------------------------
#define AB_T 64
#define AB_K 16
__global__ void __launch_bounds__(256) gemm_f32_any_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                           float* __restrict__ C, int M, int N, int K, int lda, int ldw,
                                                           int ldc) {
  mi_pdl_enter();
  __shared__ float As[AB_K][AB_T + 4], Ws[AB_K][AB_T + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * AB_T, n0 = blockIdx.x * AB_T;
  float total[4][4], acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = 0.f;
  for (int p = 0; p < PARTS; ++p) {
    const int k_end = part_begin(K, p + 1);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int k0 = part_begin(K, p); k0 < k_end; k0 += AB_K) {
      __syncthreads();
      for (int idx = tid; idx < AB_T * AB_K; idx += 256) {
        const int r = idx / AB_K, c = idx % AB_K, k = k0 + c;
        As[c][r] = (m0 + r < M && k < k_end) ? A[(size_t)(m0 + r) * lda + k] : 0.f;
        Ws[c][r] = (n0 + r < N && k < k_end) ? W[(size_t)(n0 + r) * ldw + k] : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < AB_K; ++k) {
        float a[4], w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) total[i][j] = p ? total[i][j] + acc[i][j] : acc[i][j];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
      if (m < M && n < N) C[(size_t)m * ldc + n] = total[i][j];
    }
}

template <int RM, int STAGES>
static cudaError_t launch_rows(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                               int w_constant, cudaStream_t stream) {
  const size_t smem = (size_t)PARTS * STAGES * (RB_COLS + 4 * RM) * RB_PITCH * sizeof(float);
  auto kern = gemm_f32_rows_kernel<RM, STAGES>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return MI_LAUNCH(kern, (N + RB_COLS - 1) / RB_COLS, 64 * PARTS, smem, stream, A, W, C, M, N, K, lda, ldw, ldc,
                   w_constant);
}

template <int TM>
static cudaError_t launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                               cudaStream_t stream) {
  const size_t smem = (size_t)PARTS * TB_STAGES * (8 * TM + TB_N) * TB_PITCH * sizeof(float);
  auto kern = gemm_f32_tile_kernel<TM>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return MI_LAUNCH(kern, dim3((N + TB_N - 1) / TB_N, (M + 8 * TM - 1) / (8 * TM)), 64 * PARTS, smem, stream, A, W, C, M, N,
                   K, lda, ldw, ldc);
}

// A float32 matrix [rows, cols] with `ld` elements between rows, in boxes of box_rows x 32 with the 128-byte swizzle.
static bool make_map_f32(CUtensorMap* map, const float* base, int rows, int cols, long long ld, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {ST_K, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int RM, int LIMIT = SPIN_LIMIT>
static int launch_stream(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                         int w_constant, int sms, cudaStream_t stream) {
  const int tiles = (N + ST_COLS * sms - 1) / (ST_COLS * sms), per = sms * tiles, cols = (N + per - 1) / per;
  const int grid = (N + cols * tiles - 1) / (cols * tiles);
  const int chunks = (part_begin(K, 1) + ST_K - 1) / ST_K;
  const int stage_bytes = PARTS * (((cols * ST_K * 4 + 1023) & ~1023) + 1024);
  int stages = ST_BUDGET / stage_bytes;
  if (stages > ST_MAX_STAGES) stages = ST_MAX_STAGES;
  if (stages > chunks * tiles) stages = chunks * tiles;
  const size_t smem = (size_t)stages * stage_bytes + 1024;
  CUtensorMap map_w, map_a;
  if (!make_map_f32(&map_w, W, N, K, ldw, cols) || !make_map_f32(&map_a, A, M, K, lda, M))
    MI_REFUSE("gemm_f32: the driver refused a tensor map (M %d, N %d, K %d)", M, N, K);
  auto kern = gemm_f32_stream_kernel<RM, LIMIT>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  MI_LAUNCH(kern, grid, ST_THREADS, smem, stream, map_w, map_a, C, M, N, K, ldc, cols, tiles, stages, w_constant);
  return 0;
}

// Which of the two kernels takes up to 4 rows, from their times in us, streaming kernel and kernel for few rows, weights out of memory.
// A block per SM has few of its 32 lanes at work in narrow results, and three and four rows of A read from shared memory stand
// longer beside one of W:
//   rows, K       N = 256        1024         2048         4096         6144         8192         32000
//   1, 2048     7.5   6.7    7.9   6.8    7.9   9.7    8.0  10.5   14.2  17.3   14.8  21.0   48.4  66.5
//   2, 256      2.5   2.0    2.6   2.2    2.6   2.4    2.5   2.5    3.6   4.4    3.7   4.8    9.0  14.5
//   2, 2048     9.0   6.7    9.4   6.8    9.4   9.7    9.4  10.5   14.7  17.6   15.3  21.4   49.7  66.7
//   4, 1024     6.4   3.9    6.6   4.1    6.7   5.6    7.2   6.3   11.6  10.2   11.9  12.8   34.0  38.2
//   4, 4096    18.2  12.1   18.6  13.2   18.6  17.4   19.1  19.0   34.4  30.4   34.8  37.4    110   121
static bool takes_stream(int M, int N, int K) {
  if (M <= 2) return N >= 2048 && (long long)N * K >= 1 << 20;
  return M <= ST_MAX_ROWS && N >= 8192;
}

// w_constant: W is not written by any kernel that may still run (a loaded weight).  no_wait: the streaming kernel gives up
// at its first copy, as after a wait that ran out; C is then not to be trusted, and the status word says so.
// Zero-padded tails of a part add exact zeros at the end of its sum, so they do not change it.
extern "C" int mi_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                           int ldw, int ldc, int w_constant, int sms, int no_wait, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (sms <= 0) MI_REFUSE("gemm_f32: bad number of SMs %d", sms);
  if (K <= 0) MI_REFUSE("gemm_f32: K must be positive, got %d", K);
  if (lda < K || ldw < K || ldc < N) MI_REFUSE("gemm_f32: leading dimensions too small");
  if ((M + 15) / 16 > 65535) MI_REFUSE("gemm_f32: too many rows (%d)", M);
  const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && mi_aligned(A, 16) && mi_aligned(W, 16);
  cudaError_t e = cudaSuccess;
  if (!vec) {
    MI_LAUNCH((gemm_f32_any_kernel), dim3((N + AB_T - 1) / AB_T, (M + AB_T - 1) / AB_T), 256, 0, stream, A, W, C, M, N, K,
              lda, ldw, ldc);
  } else if (takes_stream(M, N, K)) {
    const int rc = no_wait  ? launch_stream<ST_MAX_ROWS, 0>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, sms, stream)
                   : M == 1 ? launch_stream<1>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, sms, stream)
                   : M == 2 ? launch_stream<2>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, sms, stream)
                            : launch_stream<4>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, sms, stream);
    if (rc) return rc;
  } else if (M <= 16 || (M <= RB_MAX_ROWS && N <= RB_MAX_COLS)) {
    e = M <= 4    ? launch_rows<1, 8>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, stream)
        : M <= 8  ? launch_rows<2, 6>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, stream)
        : M <= 16 ? launch_rows<4, 5>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, stream)
                  : launch_rows<8, 4>(A, W, C, M, N, K, lda, ldw, ldc, w_constant, stream);
  } else {
    e = launch_tile<4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  }
  if (e != cudaSuccess) return (int)e;
  MI_RETURN_LAUNCH_STATUS();
}
