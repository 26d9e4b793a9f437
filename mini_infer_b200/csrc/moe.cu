// Routed experts: every token goes through the `top` experts its router picks.
//
//   mi_moe_select     from the router logits z = W_r x (fp32, a matrix product): the `top` largest of a token
//                     (ties: the lower index; optionally among the experts of the best groups only) and
//                     their weights (the softmax over those alone, or their share of the softmax over all
//                     experts, times a factor, or their sigmoids times a factor, chosen with a correction
//                     added per expert) -> ids [M, top] int32, weights [M, top] fp32.  Where a token has fewer
//                     candidates than `top` (logits that are NaN or minus infinity) the others of its ids are
//                     valid ones and their weights NaN
//   mi_moe_plan       sorts the M*top (token, choice) entries by expert: perm[pos] = entry, inv[entry] =
//                     pos, offsets[E + 1], and the list of row tiles (expert, first row, rows) that the
//                     grouped products walk.  Nothing comes back to the host: the products are launched
//                     for the largest possible number of tiles and the surplus blocks leave at once.
//                     Tiles have 64 rows, or 8 for steps that bring an expert only a few rows.  An entry whose id
//                     is no expert's stands behind all others, in no tile, with inv = -1, and its token comes out NaN.
//   mi_moe_gate_up    act[pos, :] = glu(W_gate[e] x_token, W_up[e] x_token) for the entries of each expert
//   mi_moe_down       y[pos, :] = W_down[e] act[pos, :]   (fp32)
//   mi_moe_gather     xs[pos, :] = x[token of pos, :], for steps whose products are a library's grouped product
//   mi_moe_combine    out[t, :] = T(sum_k weight[t, k] * y[inv[t*top + k], :] + shared[t, :]), the shared
//                     expert's row optionally times sigmoid(gate[t])
//   mi_clamped_glu    the same activation for a dense expert: out = glu(gu[:, :I], gu[:, I:])
//
// glu(g, u) = g' * sigmoid(alpha * g') * (u' + offset), g' = min(g, limit), u' = clamp(u, -limit, limit).
// An infinite limit with alpha = 1 and offset = 0 is the plain silu(g) * u.
//
// Three products live here, all with fp32 accumulation, and none lets a row's result depend on which
// other rows share its tile: float32 on CUDA cores, k ascending (moe_gemm_kernel); bfloat16 tiles of 64
// rows on the tensor cores (mma.sync m16n8k16, moe_gemm_mma_kernel); bfloat16 tiles of 8 rows that
// stream an expert's weights (moe_rows_kernel on the tensor cores, moe_stream_kernel on CUDA cores in a kept order).  Large bfloat16 steps
// whose rows are whole 16-byte pieces go to the library's grouped product instead (the caller gathers
// the rows with mi_moe_gather and passes the experts' row ranges from the plan).
#include "common.cuh"

MI_DEFINE_ERROR_API()

__device__ __forceinline__ float mi_clamped_glu_value(float g, float u, float limit, float alpha, float offset) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g * (1.f / (1.f + expf(-alpha * g))) * (u + offset);
}

// ------------------------------------------------------------------------------------------ router
// The logits [M, E] (fp32) come from a matrix product; one warp per token picks the `top` largest
// choice scores (ties: the lower index).  Three ways to score and weigh.  mode 0: the choice score is
// the logit, the weights the softmax over the chosen logits alone.  mode 1: scores are the softmax over all
// experts (the logit orders alike); the chosen experts' scores are divided by their sum (+ 1e-20) and
// multiplied by `scale`.  mode 2: scores are sigmoid(logit), the choice score adds `correction[e]` (may be
// absent), the weights are the chosen experts' scores times `scale` (no division by their sum).  With n_groups > 1
// the experts lie in n_groups equal groups of neighbours and only experts of the `keep` best groups (ties:
// the lower index) can be chosen; a group counts as its best choice score (group_top2 = 0) or as the sum
// of its two best (group_top2 = 1).
#define ROUTE_MAX_PER_LANE 8
#define ROUTE_WARPS 4

// PER: experts (and groups) per lane, known to the compiler.  8 tokens of 32 experts in groups: 6.5 us with eight of them, 3.6 with
// one; of 64 experts 7.2, and 4.8 with two; 2048 tokens of 64 15.2 and 9.7.  More take eight: 96 experts 7.8, 128 8.5, 256
// 10.8 (an instance with four, for up to 128, was not measured).
template <int PER>
__global__ void __launch_bounds__(32 * ROUTE_WARPS)
moe_select_kernel(const float* __restrict__ logits, int stride, int* __restrict__ ids,
                  float* __restrict__ weights, int M, int E, int top, int mode, int n_groups,
                  int keep, float scale, const float* __restrict__ correction, int group_top2,
                  const float* __restrict__ bias) {
  // bias [E]: added to the logits before anything else; correction [E] (mode 2): to the choice scores alone
  mi_pdl_enter();
  __shared__ float choice_sh[ROUTE_WARPS][32 * PER];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * ROUTE_WARPS + warp;
  if (t >= M) return;
  const float* z = logits + (size_t)t * stride;
  float lg[PER];       // choice scores; minus infinity: out of the race
  float sc[PER];       // mode 2: the scores that become weights
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    lg[i] = e < E ? z[e] + (bias ? bias[e] : 0.f) : -INFINITY;
    sc[i] = 0.f;
    if (mode == 2 && e < E) {
      sc[i] = 1.f / (1.f + expf(-lg[i]));
      lg[i] = sc[i] + (correction ? correction[e] : 0.f);
    }
  }
  float zmax = -INFINITY, zsum = 0.f;
  if (mode == 1) {
#pragma unroll
    for (int i = 0; i < PER; ++i) zmax = fmaxf(zmax, lg[i]);
    zmax = mi_warp_max(zmax);
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) zsum += expf(lg[i] - zmax);
    zsum = mi_warp_sum(zsum);
  }
  if (n_groups > 1) {
    // group g's score sits with lane g % 32, place g / 32; the groups that stay: `keep` times the
    // best group that is still in; experts of the others are taken out
    const int per = E / n_groups;
    float* mine = choice_sh[warp];
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) mine[lane + 32 * i] = lg[i];
    __syncwarp();
    float gs[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int g = lane + 32 * i;
      gs[i] = -INFINITY;
      if (g < n_groups) {
        float b1 = -INFINITY, b2 = -INFINITY;
        for (int e = g * per; e < (g + 1) * per; ++e) {
          const float v = mine[e];
          if (v > b1) { b2 = b1; b1 = v; }
          else if (v > b2) b2 = v;
        }
        gs[i] = (group_top2 && per > 1) ? b1 + b2 : b1;
      }
    }
    unsigned kept_mask = 0u;             // bit i: this lane's group lane + 32 i stays
    for (int k = 0; k < keep; ++k) {
      float best = -INFINITY;
      int best_g = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int g = lane + 32 * i;
        if (g < n_groups && !((kept_mask >> i) & 1u) && (gs[i] > best || (gs[i] == best && g < best_g))) {
          best = gs[i];
          best_g = g;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int og = __shfl_xor_sync(0xffffffffu, best_g, o);
        if (ob > best || (ob == best && og < best_g)) {
          best = ob;
          best_g = og;
        }
      }
      if (best_g == 0x7fffffff) break;
      if ((best_g & 31) == lane) kept_mask |= 1u << (best_g >> 5);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      const int g = e < E ? e / per : 0;
      const unsigned owner_mask = __shfl_sync(0xffffffffu, kept_mask, g & 31);   // every lane takes part
      if (e < E && !((owner_mask >> (g >> 5)) & 1u)) lg[i] = -INFINITY;
    }
  }
  float my_val = 0.f, denom = 0.f, first = 0.f;
  int my_id = 0;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      if (e < E && (lg[i] > best || (lg[i] == best && e < best_e)) && lg[i] != -INFINITY) {
        best = lg[i];
        best_e = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
      if (ob > best || (ob == best && oe < best_e)) {
        best = ob;
        best_e = oe;
      }
    }
    const bool none = best_e >= E;       // no candidate is left
    if (none) best_e = k;
    float score = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (best_e == lane + 32 * i) {
        lg[i] = -INFINITY;   // taken
        score = sc[i];
      }
    if (k == 0) first = best;
    float p;
    if (mode == 2) p = __shfl_sync(0xffffffffu, score, best_e & 31);
    else p = mode == 1 ? expf(best - zmax) / zsum : expf(best - first);
    if (none) p = __int_as_float(0x7fc00000);
    denom += p;
    if (lane == k) {
      my_val = p;
      my_id = best_e;
    }
  }
  if (lane < top) {
    ids[(size_t)t * top + lane] = my_id;
    weights[(size_t)t * top + lane] = mode == 2 ? my_val * scale
                                    : mode == 1 ? my_val / (denom + 1e-20f) * scale : my_val / denom;
  }
}

extern "C" int mi_moe_select(const float* logits, int stride, int* ids, float* weights, int M, int E, int top,
                             int mode, int n_groups, int keep, float scale, const float* correction,
                             int group_top2, const float* bias, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (E <= 0 || E > 32 * ROUTE_MAX_PER_LANE) MI_REFUSE("moe: %d experts (1 to %d are taken)", E, 32 * ROUTE_MAX_PER_LANE);
  if (top <= 0 || top > E || top > 32) MI_REFUSE("moe: %d of %d experts per token", top, E);
  if (mode < 0 || mode > 2) MI_REFUSE("moe: unknown way %d to score the experts", mode);
  if (n_groups > 1) {
    if (E % n_groups) MI_REFUSE("moe: %d experts are no %d equal groups", E, n_groups);
    if (keep <= 0 || keep > n_groups) MI_REFUSE("moe: %d of %d groups kept", keep, n_groups);
    if (keep * (E / n_groups) < top) MI_REFUSE("moe: %d groups of %d experts cannot give %d experts", keep, E / n_groups, top);
  }
#define MI_SELECT(PER)                                                                                                    \
  MI_LAUNCH((moe_select_kernel<PER>), (M + ROUTE_WARPS - 1) / ROUTE_WARPS, 32 * ROUTE_WARPS, 0, stream, logits, stride, ids, \
            weights, M, E, top, mode, n_groups, keep, scale, correction, group_top2, bias)
  if (E <= 32) MI_SELECT(1);
  else if (E <= 64) MI_SELECT(2);
  else MI_SELECT(ROUTE_MAX_PER_LANE);
#undef MI_SELECT
  MI_RETURN_LAUNCH_STATUS();
}

// ------------------------------------------------------------------------------------------ plan
#define TILE_M 64
#define TILE_N 64
#define TILE_K 16

// plan layout (int32): [0] number of tiles, [1 .. E+1] offsets, then 3 ints per tile (expert, first row, rows)
__global__ void moe_plan_kernel(const int* __restrict__ ids, int n, int E, int* __restrict__ perm,
                                int* __restrict__ inv, int* __restrict__ plan, int tile_rows) {
  mi_pdl_enter();
  extern __shared__ int sh[];
  int* counts = sh;            // [E + 1]: the last one counts the ids that are no expert's
  int* cursor = sh + E + 1;    // [E + 1]
  auto expert = [&](int i) { const unsigned e = (unsigned)ids[i]; return e < (unsigned)E ? (int)e : E; };
  for (int e = threadIdx.x; e <= E; e += blockDim.x) counts[e] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&counts[expert(i)], 1);
  __syncthreads();
  // rows and tiles in front of every expert: a warp scan per 32 experts, carried on from one to the next by one warp
  if (threadIdx.x < 32) {
    int* offsets = plan + 1;
    int* tiles = plan + 2 + E;
    const int lane = threadIdx.x;
    int run = 0, nt = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int rows = e < E ? counts[e] : 0, own = (rows + tile_rows - 1) / tile_rows;
      int rs = rows, ts = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int r = __shfl_up_sync(0xffffffffu, rs, o), t = __shfl_up_sync(0xffffffffu, ts, o);
        if (lane >= o) {
          rs += r;
          ts += t;
        }
      }
      if (e < E) {
        const int first = run + rs - rows, at = nt + ts - own;
        offsets[e] = first;
        cursor[e] = first;
        for (int i = 0; i < own; ++i) {
          tiles[3 * (at + i)] = e;
          tiles[3 * (at + i) + 1] = first + i * tile_rows;
          tiles[3 * (at + i) + 2] = min(tile_rows, rows - i * tile_rows);
        }
      }
      run += __shfl_sync(0xffffffffu, rs, 31);
      nt += __shfl_sync(0xffffffffu, ts, 31);
    }
    if (lane == 0) {
      offsets[E] = run;
      cursor[E] = run;
      plan[0] = nt;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = expert(i), pos = atomicAdd(&cursor[e], 1);
    perm[pos] = i;
    inv[i] = e < E ? pos : -1;
  }
}

#define FEW_ROWS 8
// rows per tile: TILE_M for the tiled products, FEW_ROWS for the streaming ones (few rows per expert)
extern "C" int mi_moe_tile_rows(int few) { return few ? FEW_ROWS : TILE_M; }

extern "C" int mi_moe_plan(const int* ids, int n, int E, int* perm, int* inv, int* plan, int tile_rows,
                           cudaStream_t stream) {
  if (n <= 0) return 0;
  if (E <= 0 || E > 4096) MI_REFUSE("moe: %d experts", E);
  if (tile_rows != TILE_M && tile_rows != FEW_ROWS) MI_REFUSE("moe: tiles of %d rows", tile_rows);
  MI_LAUNCH((moe_plan_kernel), 1, 1024, 2 * (E + 1) * sizeof(int), stream, ids, n, E, perm, inv, plan, tile_rows);
  MI_RETURN_LAUNCH_STATUS();
}

// ------------------------------------------------------------------------------------------ grouped products
// A tile is TILE_M rows of one expert times TILE_N output columns; 256 threads, 4 x 4 outputs each.
// GATED: A rows are gathered (token = perm[pos] / top), two weight matrices, the activation in the
// epilogue, output in T.  Otherwise A rows are the sorted rows themselves and the output is fp32.
template <typename T, bool GATED>
__global__ void __launch_bounds__(256)
moe_gemm_kernel(const T* __restrict__ a, int a_stride, const T* __restrict__ w0, const T* __restrict__ w1,
                long long w_expert_stride, const int* __restrict__ perm, int top, const int* __restrict__ plan,
                int E, void* __restrict__ out_, int N, int K, float limit, float alpha, float offset) {
  mi_pdl_enter();
  const int tile = blockIdx.y;
  if (tile >= plan[0]) return;
  const int* td = plan + 2 + E + 3 * tile;
  const int e = td[0], row0 = td[1], rows = td[2];
  const int n0 = blockIdx.x * TILE_N;
  __shared__ float As[TILE_K][TILE_M + 4];
  __shared__ float B0[TILE_K][TILE_N + 4];
  __shared__ float B1[GATED ? TILE_K : 1][TILE_N + 4];
  __shared__ int arow[TILE_M];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  if (tid < TILE_M) {
    int r = -1;
    if (tid < rows) r = GATED ? perm[row0 + tid] / top : row0 + tid;
    arow[tid] = r;
  }
  const T* wb0 = w0 + (size_t)e * w_expert_stride;
  const T* wb1 = GATED ? w1 + (size_t)e * w_expert_stride : nullptr;
  float acc0[4][4], acc1[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc0[i][j] = acc1[i][j] = 0.f;
  __syncthreads();
  for (int k0 = 0; k0 < K; k0 += TILE_K) {
    // 64 x 16 elements of each operand: 4 per thread, k fastest
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int idx = tid + 256 * it;
      const int r = idx >> 4, kk = idx & 15;
      const int kg = k0 + kk;
      const int ar = arow[r];
      As[kk][r] = (ar >= 0 && kg < K) ? mi_to_float(a[(size_t)ar * a_stride + kg]) : 0.f;
      const int n = n0 + r;
      const bool ok = n < N && kg < K;
      B0[kk][r] = ok ? mi_to_float(wb0[(size_t)n * K + kg]) : 0.f;
      if (GATED) B1[kk][r] = ok ? mi_to_float(wb1[(size_t)n * K + kg]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TILE_K; ++kk) {
      float av[4], b0[4], b1[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b0[j] = B0[kk][tx * 4 + j];
        if (GATED) b1[j] = B1[kk][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc0[i][j] = fmaf(av[i], b0[j], acc0[i][j]);
          if (GATED) acc1[i][j] = fmaf(av[i], b1[j], acc1[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      if (GATED)
        reinterpret_cast<T*>(out_)[(size_t)(row0 + r) * N + n] =
            mi_from_float<T>(mi_clamped_glu_value(acc0[i][j], acc1[i][j], limit, alpha, offset));
      else
        reinterpret_cast<float*>(out_)[(size_t)(row0 + r) * N + n] = acc0[i][j];
    }
  }
}

// ------------------------------------------------------------------------------------------ the same on tensor cores
// bfloat16 only.  64 rows x 64 columns per block, k in steps of 32; four warps, each 32 x 32 of the
// tile as 2 x 4 mma.m16n8k16 tiles (twice that with two weight matrices).  Operands go through
// shared memory with rows of 40 elements, which makes the fragments' 32-bit reads conflict-free.
// Rows of 8 elements are fetched as one 16-byte load where k and the pointers allow it.
#define MMA_K 32
#define MMA_LD (MMA_K + 8)

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// 64 rows x 32 k of a row-major operand into shared memory; row pointers may be null (zero rows)
__device__ __forceinline__ void mma_stage(bf16 (*dst)[MMA_LD], const bf16* const* rowptr, int k0, int K, bool vec,
                                          int tid) {
  if (vec) {   // 64 rows x 4 chunks of 8 elements: 2 chunks per thread
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int idx = tid + 128 * it;
      const int r = idx >> 2, c8 = (idx & 3) << 3;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      const bf16* src = rowptr[r];
      if (src && k0 + c8 < K) v = *reinterpret_cast<const uint4*>(src + k0 + c8);   // K % 8 == 0: whole chunks
      *reinterpret_cast<uint4*>(&dst[r][c8]) = v;
    }
  } else {
    for (int idx = tid; idx < TILE_M * MMA_K; idx += 128) {
      const int r = idx / MMA_K, kk = idx - r * MMA_K;
      const bf16* src = rowptr[r];
      dst[r][kk] = (src && k0 + kk < K) ? src[k0 + kk] : __float2bfloat16_rn(0.f);
    }
  }
}

template <bool GATED>
__global__ void __launch_bounds__(128)
moe_gemm_mma_kernel(const bf16* __restrict__ a, int a_stride, const bf16* __restrict__ w0, const bf16* __restrict__ w1,
                    long long w_expert_stride, const int* __restrict__ perm, int top, const int* __restrict__ plan,
                    int E, void* __restrict__ out_, int N, int K, float limit, float alpha, float offset, int vec) {
  mi_pdl_enter();
  const int tile = blockIdx.y;
  if (tile >= plan[0]) return;
  const int* td = plan + 2 + E + 3 * tile;
  const int e = td[0], row0 = td[1], rows = td[2];
  const int n0 = blockIdx.x * TILE_N;
  __shared__ __align__(16) bf16 As[TILE_M][MMA_LD];
  __shared__ __align__(16) bf16 B0[TILE_N][MMA_LD];
  __shared__ __align__(16) bf16 B1[GATED ? TILE_N : 1][MMA_LD];
  __shared__ const bf16* aptr[TILE_M];
  __shared__ const bf16* b0ptr[TILE_N];
  __shared__ const bf16* b1ptr[TILE_N];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1, g = lane >> 2, t = lane & 3;
  const bf16* wb0 = w0 + (size_t)e * w_expert_stride;
  const bf16* wb1 = GATED ? w1 + (size_t)e * w_expert_stride : nullptr;
  if (tid < TILE_M) {
    const bf16* p = nullptr;
    if (tid < rows) p = a + (size_t)(GATED ? perm[row0 + tid] / top : row0 + tid) * a_stride;
    aptr[tid] = p;
    const int n = n0 + tid;
    b0ptr[tid] = n < N ? wb0 + (size_t)n * K : nullptr;
    b1ptr[tid] = (GATED && n < N) ? wb1 + (size_t)n * K : nullptr;
  }
  float acc0[2][4][4], acc1[GATED ? 2 : 1][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc0[i][j][c] = 0.f;
        if (GATED) acc1[i][j][c] = 0.f;
      }
  __syncthreads();
  for (int k0 = 0; k0 < K; k0 += MMA_K) {
    mma_stage(As, aptr, k0, K, vec != 0, tid);
    mma_stage(B0, b0ptr, k0, K, vec != 0, tid);
    if (GATED) mma_stage(B1, b1ptr, k0, K, vec != 0, tid);
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < MMA_K; ks += 16) {
      uint32_t af[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm * 32 + i * 16 + g;
        af[i][0] = *reinterpret_cast<const uint32_t*>(&As[r][ks + 2 * t]);
        af[i][1] = *reinterpret_cast<const uint32_t*>(&As[r + 8][ks + 2 * t]);
        af[i][2] = *reinterpret_cast<const uint32_t*>(&As[r][ks + 2 * t + 8]);
        af[i][3] = *reinterpret_cast<const uint32_t*>(&As[r + 8][ks + 2 * t + 8]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = wn * 32 + j * 8 + g;
        uint32_t bf[2];
        bf[0] = *reinterpret_cast<const uint32_t*>(&B0[n][ks + 2 * t]);
        bf[1] = *reinterpret_cast<const uint32_t*>(&B0[n][ks + 2 * t + 8]);
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_bf16(acc0[i][j], af[i], bf);
        if (GATED) {
          bf[0] = *reinterpret_cast<const uint32_t*>(&B1[n][ks + 2 * t]);
          bf[1] = *reinterpret_cast<const uint32_t*>(&B1[n][ks + 2 * t + 8]);
#pragma unroll
          for (int i = 0; i < 2; ++i) mma_bf16(acc1[i][j], af[i], bf);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int r = wm * 32 + i * 16 + g + (c >> 1) * 8;
        const int n = n0 + wn * 32 + j * 8 + 2 * t + (c & 1);
        if (r >= rows || n >= N) continue;
        if (GATED)
          reinterpret_cast<bf16*>(out_)[(size_t)(row0 + r) * N + n] =
              __float2bfloat16_rn(mi_clamped_glu_value(acc0[i][j][c], acc1[i][j][c], limit, alpha, offset));
        else
          reinterpret_cast<float*>(out_)[(size_t)(row0 + r) * N + n] = acc0[i][j][c];
      }
}

// whether rows of k elements starting at these pointers can be fetched in 16-byte pieces
static int mma_vec_ok(const void* a, long long a_stride, const void* w0, const void* w1, int K) {
  return K % 8 == 0 && a_stride % 8 == 0 && mi_aligned(a, 16) && mi_aligned(w0, 16) && (!w1 || mi_aligned(w1, 16));
}

// ------------------------------------------------------------------------------------------ few rows per expert
// A decode step brings an expert a handful of rows: the product is a stream of that expert's weights.  Tiles have at
// most FEW_ROWS rows.  A warp owns pairs of weight rows (gate and up of a column, or two columns of the plain product);
// lane l takes the 16-byte pieces of k at 8 l, 8 l + 256, ... of both, one fused multiply-add after the other, and the
// lanes' sums are added by butterfly.  That order is the result's, whatever rows share the tile.
//
// What bounds it is the stream of weights.  A warp's pairs are one list of pieces, fetched a batch ahead of the batch that
// is worked on, so that it does not stand still at the end of a column: a warp per pair without the batch ahead took 179 us
// for 630 MB (25 experts of 3 x 1024 x 4096), 0.54 of the copy bandwidth, and this takes 129 (2048 wide, 19 experts of
// 3 x 512 x 2048: 48 and 43).  It is run where a result's order of sums is kept from one version of these kernels to the next
// (`in_order` of the entry points); moe_rows_kernel below takes the other calls.
// bfloat16, k a multiple of 8, 16-byte aligned rows.
#define MS_WARPS 8
#define MS_UNITS 16       // a warp gets as many pairs as make up this many pieces of 256 k (8, 32: 139 and 124 us, 41 and 52)
__device__ __forceinline__ uint4 ms_load(const bf16* p, bool in) {       // weights: read once
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (in) asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void ms_unpack(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// the pairs [pair0, pair0 + n_pairs) of a warp for R rows of x, of which `rows` exist
template <bool GATED, int R>
__device__ __forceinline__ void moe_stream_pairs(const bf16* __restrict__ a, int a_stride, const bf16* __restrict__ w0,
                                                 const bf16* __restrict__ w1, const int* __restrict__ perm, int top, int row0,
                                                 int rows, void* __restrict__ out_, int N, int K, int pair0, int n_pairs,
                                                 float limit, float alpha, float offset) {
  constexpr int BATCH = R <= 4 ? 4 : 2;
  const int lane = threadIdx.x & 31;
  const int pieces = (K + 255) >> 8, units = n_pairs * pieces;
  const bf16* xr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = row0 + min(r, rows - 1);
    xr[r] = a + (size_t)(GATED ? perm[row] / top : row) * a_stride + lane * 8;
  }
  float acc0[R], acc1[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc0[r] = acc1[r] = 0.f;

  int l_pair = pair0, l_piece = 0;             // the next unit to be fetched
  auto fetch = [&](uint4 (&w)[BATCH][2]) {
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int k = l_piece * 256 + lane * 8;
      const bool in = l_pair < pair0 + n_pairs && k < K;
      const int n_a = GATED ? l_pair : 2 * l_pair, n_b = GATED ? l_pair : min(2 * l_pair + 1, N - 1);
      w[b][0] = ms_load(w0 + (size_t)n_a * K + k, in);
      w[b][1] = ms_load((GATED ? w1 : w0) + (size_t)n_b * K + k, in);
      if (++l_piece == pieces) {
        l_piece = 0;
        ++l_pair;
      }
    }
  };
  uint4 w[BATCH][2], next[BATCH][2];
  fetch(w);
  int pair = pair0, piece = 0;
#pragma unroll 1
  for (int u0 = 0; u0 < units; u0 += BATCH) {
    fetch(next);
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      if (u0 + b < units) {
        const int k = piece * 256 + lane * 8;
        float wa[8], wb[8];
        ms_unpack(w[b][0], wa);
        ms_unpack(w[b][1], wb);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float x[8];
          ms_unpack(k < K ? __ldg(reinterpret_cast<const uint4*>(xr[r] + piece * 256)) : make_uint4(0u, 0u, 0u, 0u), x);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            acc0[r] = fmaf(wa[i], x[i], acc0[r]);
            acc1[r] = fmaf(wb[i], x[i], acc1[r]);
          }
        }
        if (++piece == pieces) {               // the pair is done: a lane per row stores it
          float s0 = 0.f, s1 = 0.f;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float t0 = mi_warp_sum(acc0[r]), t1 = mi_warp_sum(acc1[r]);
            if (lane == r) {
              s0 = t0;
              s1 = t1;
            }
            acc0[r] = acc1[r] = 0.f;
          }
          if (lane < rows) {
            if (GATED) {
              reinterpret_cast<bf16*>(out_)[(size_t)(row0 + lane) * N + pair] =
                  __float2bfloat16_rn(mi_clamped_glu_value(s0, s1, limit, alpha, offset));
            } else {
              float* o = reinterpret_cast<float*>(out_) + (size_t)(row0 + lane) * N + 2 * pair;
              o[0] = s0;
              if (2 * pair + 1 < N) o[1] = s1;
            }
          }
          piece = 0;
          ++pair;
        }
      }
    }
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      w[b][0] = next[b][0];
      w[b][1] = next[b][1];
    }
  }
}

template <bool GATED>
__global__ void __launch_bounds__(32 * MS_WARPS, 2)
moe_stream_kernel(const bf16* __restrict__ a, int a_stride, const bf16* __restrict__ w0, const bf16* __restrict__ w1,
                  long long w_expert_stride, const int* __restrict__ perm, int top, const int* __restrict__ plan,
                  int E, void* __restrict__ out_, int N, int K, int pairs_per_warp, float limit, float alpha, float offset) {
  mi_pdl_enter();
  const int tile = blockIdx.y;
  if (tile >= plan[0]) return;
  const int* td = plan + 2 + E + 3 * tile;
  const int e = td[0], row0 = td[1], rows = td[2];
  const int n_all = GATED ? N : (N + 1) / 2, pair0 = (blockIdx.x * MS_WARPS + (threadIdx.x >> 5)) * pairs_per_warp;
  const int n_pairs = min(pairs_per_warp, n_all - pair0);
  if (n_pairs <= 0) return;
  const bf16* e0 = w0 + (size_t)e * w_expert_stride;
  const bf16* e1 = GATED ? w1 + (size_t)e * w_expert_stride : nullptr;
#define MI_GO(R) \
  moe_stream_pairs<GATED, R>(a, a_stride, e0, e1, perm, top, row0, rows, out_, N, K, pair0, n_pairs, limit, alpha, offset)
  if (rows <= 1) MI_GO(1);
  else if (rows <= 2) MI_GO(2);
  else if (rows <= 4) MI_GO(4);
  else MI_GO(8);
#undef MI_GO
}
// Pairs of weight rows per warp: MS_UNITS pieces, or fewer so that small products still fill the chip.
static int stream_pairs(int K, int n_pairs, int n_entries) {
  const int pieces = (K + 255) / 256;
  const long long fill = (long long)n_pairs * n_entries / (2 * 148 * MS_WARPS);
  const int most = pieces >= MS_UNITS ? 1 : MS_UNITS / pieces;
  return fill < 1 ? 1 : fill < most ? (int)fill : most;
}
static int stream_blocks(int n_pairs, int per_warp) { return (n_pairs + MS_WARPS * per_warp - 1) / (MS_WARPS * per_warp); }

// The same on the tensor cores.  The tile's rows are the N side of mma.sync.m16n8k16; a block owns 16 rows of both gated
// matrices (or 32 of the plain one), the M side, and its eight warps take the 64-wide pieces of k in turn and add up in
// shared memory.  A lane's fragments come straight from global memory, 16 bytes (8 consecutive k, taken as the k of two
// instructions in an order that is the same for both operands) at a time, two pieces of k, 16 loads, in flight.  What bounds
// it is the stream of weights; gate/up and down of 64 experts of 3 x 1024 x 4096, four each, here and by moe_stream_kernel:
// 8 tokens 114 and 129 us (102 of bytes), 32 tokens 224 and 320, 128 tokens 311 and 810.
// An instruction adds its 16 products to nothing; what it gives is added up pairwise in fp32, the warps' shares in fp64: the
// accumulator of a chain of instructions loses more than an fp32 addition does (distance from 64 bits at K = 512, 1024 and
// 2816: 8.6, 12.9 and 32.8e-8 as one chain, 5.0, 5.6 and 6.7e-8 so, 6.2, 7.0 and 8.5e-8 by fused multiply-adds), and the time
// is the same to one part in a hundred.  bfloat16, k a multiple of 8, 16-byte aligned rows.
#define MR_WARPS 8
#define MR_PIECE 64
#define MR_LEAST_K 256     // below, what an instruction cuts off its own sum is not made up: 4.1 against 3.9e-8 at K = 64
template <bool GATED>
__global__ void __launch_bounds__(32 * MR_WARPS, 2)
moe_rows_kernel(const bf16* __restrict__ a, int a_stride, const bf16* __restrict__ w0, const bf16* __restrict__ w1,
                long long w_expert_stride, const int* __restrict__ perm, int top, const int* __restrict__ plan,
                int E, void* __restrict__ out_, int N, int K, float limit, float alpha, float offset) {
  mi_pdl_enter();
  const int tile = blockIdx.y;
  if (tile >= plan[0]) return;
  const int* td = plan + 2 + E + 3 * tile;
  const int e = td[0], row0 = td[1], rows = td[2];
  __shared__ float shares[MR_WARPS][FEW_ROWS][32 + 4];      // [warp][row of x][row of either matrix]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  constexpr int COLS = GATED ? 16 : 32;                     // output columns of the block
  const int n0 = blockIdx.x * COLS;
  // rows g and g + 8 of the two halves: gate and up, or columns n0.. and n0 + 16..  (rows beyond N repeat the last one)
  const bf16* base[2] = {w0 + (size_t)e * w_expert_stride, (GATED ? w1 : w0) + (size_t)e * w_expert_stride};
  const bf16* wp[2][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      wp[h][r] = base[h] + (size_t)min(N - 1, n0 + (GATED ? 0 : 16 * h) + g + 8 * r) * K + q * 8;
  const bool has_x = g < rows;
  const bf16* xp = a + (size_t)(has_x ? (GATED ? perm[row0 + g] / top : row0 + g) : 0) * a_stride + q * 8;
  const int pieces = (K + MR_PIECE - 1) / MR_PIECE;
  float acc[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[h][i] = 0.f;
  for (int c = warp; c < pieces; c += 2 * MR_WARPS) {
    uint4 w[2][2][2][2], x[2][2];     // [piece][half of it][matrix][row]
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int k = (c + p * MR_WARPS) * MR_PIECE + s * 32;
        const bool in = k + q * 8 < K;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int r = 0; r < 2; ++r) w[p][s][h][r] = ms_load(wp[h][r] + k, in);
        x[p][s] = in && has_x ? __ldg(reinterpret_cast<const uint4*>(xp + k)) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float sum[2][4];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        float t[2][4];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const uint4 u = w[p][s][h][0], v = w[p][s][h][1], xx = x[p][s];
          const uint32_t a0[4] = {u.x, v.x, u.y, v.y}, b0[2] = {xx.x, xx.y};
          const uint32_t a1[4] = {u.z, v.z, u.w, v.w}, b1[2] = {xx.z, xx.w};
          float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
          mma_bf16(d0, a0, b0);
          mma_bf16(d1, a1, b1);
#pragma unroll
          for (int i = 0; i < 4; ++i) t[s][i] = d0[i] + d1[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[p][i] = t[0][i] + t[1][i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[h][i] += sum[0][i] + sum[1][i];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) shares[warp][2 * q + (i & 1)][16 * h + g + (i >> 1) * 8] = acc[h][i];
  __syncthreads();
  const int r = tid >> 5, j = tid & 31;       // a warp per row of x
  if (r >= rows) return;
  double all = 0.0;
#pragma unroll
  for (int s = 0; s < MR_WARPS; ++s) all += shares[s][r][j];
  const float v = (float)all;
  if (GATED) {
    const float up = __shfl_down_sync(0xffffffffu, v, 16);
    if (j < 16 && n0 + j < N)
      reinterpret_cast<bf16*>(out_)[(size_t)(row0 + r) * N + n0 + j] =
          __float2bfloat16_rn(mi_clamped_glu_value(v, up, limit, alpha, offset));
  } else if (n0 + j < N) {
    reinterpret_cast<float*>(out_)[(size_t)(row0 + r) * N + n0 + j] = v;
  }
}

static int max_tiles(int n_entries, int E, int tile_rows) { return (n_entries + tile_rows - 1) / tile_rows + E; }

extern "C" int mi_moe_gate_up(const void* x, int x_stride, const void* w_gate, const void* w_up,
                              long long w_expert_stride, const int* perm, int top, const int* plan, int E,
                              void* act, int n_entries, int ff, int H, float limit, float alpha, float offset,
                              int tile_rows, int in_order, int dtype, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (tile_rows == FEW_ROWS) {
    if (dtype != MI_DTYPE_BF16 || !mma_vec_ok(x, x_stride, w_gate, w_up, H))
      MI_REFUSE("moe: the streaming product takes bfloat16 rows of whole 16-byte pieces");
    const int per_warp = stream_pairs(H, ff, n_entries);
    const bool stream_it = in_order || H < MR_LEAST_K;
    dim3 g(stream_it ? stream_blocks(ff, per_warp) : (ff + 15) / 16, max_tiles(n_entries, E, FEW_ROWS));
    if (g.y > 65535) MI_REFUSE("moe: too many row tiles for one launch");
    if (stream_it)
      MI_LAUNCH_BEHIND((moe_stream_kernel<true>), g, 32 * MS_WARPS, 0, stream, (const bf16*)x, x_stride, (const bf16*)w_gate,
                (const bf16*)w_up, w_expert_stride, perm, top, plan, E, act, ff, H, per_warp, limit, alpha, offset);
    else
      MI_LAUNCH_BEHIND((moe_rows_kernel<true>), g, 32 * MR_WARPS, 0, stream, (const bf16*)x, x_stride, (const bf16*)w_gate,
                (const bf16*)w_up, w_expert_stride, perm, top, plan, E, act, ff, H, limit, alpha, offset);
    MI_RETURN_LAUNCH_STATUS();
  }
  dim3 grid((ff + TILE_N - 1) / TILE_N, max_tiles(n_entries, E, TILE_M));
  if (grid.y > 65535) MI_REFUSE("moe: too many row tiles for one launch");
  if (dtype == MI_DTYPE_F32)
    MI_LAUNCH((moe_gemm_kernel<float, true>), grid, 256, 0, stream, (const float*)x, x_stride, (const float*)w_gate,
              (const float*)w_up, w_expert_stride, perm, top, plan, E, act, ff, H, limit, alpha, offset);
  else if (dtype == MI_DTYPE_BF16)
    MI_LAUNCH((moe_gemm_mma_kernel<true>), grid, 128, 0, stream, (const bf16*)x, x_stride, (const bf16*)w_gate,
              (const bf16*)w_up, w_expert_stride, perm, top, plan, E, act, ff, H, limit, alpha, offset,
              mma_vec_ok(x, x_stride, w_gate, w_up, H));
  else
    MI_REFUSE("moe: unknown dtype %d", dtype);
  MI_RETURN_LAUNCH_STATUS();
}

extern "C" int mi_moe_down(const void* act, const void* w_down, long long w_expert_stride, const int* plan, int E,
                           float* y, int n_entries, int H, int ff, int tile_rows, int in_order, int dtype,
                           cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (tile_rows == FEW_ROWS) {
    if (dtype != MI_DTYPE_BF16 || !mma_vec_ok(act, ff, w_down, nullptr, ff))
      MI_REFUSE("moe: the streaming product takes bfloat16 rows of whole 16-byte pieces");
    const int per_warp = stream_pairs(ff, (H + 1) / 2, n_entries);
    const bool stream_it = in_order || ff < MR_LEAST_K;
    dim3 g(stream_it ? stream_blocks((H + 1) / 2, per_warp) : (H + 31) / 32, max_tiles(n_entries, E, FEW_ROWS));
    if (g.y > 65535) MI_REFUSE("moe: too many row tiles for one launch");
    if (stream_it)
      MI_LAUNCH_BEHIND((moe_stream_kernel<false>), g, 32 * MS_WARPS, 0, stream, (const bf16*)act, ff, (const bf16*)w_down,
                (const bf16*)nullptr, w_expert_stride, (const int*)nullptr, 1, plan, E, (void*)y, H, ff, per_warp, 0.f, 0.f, 0.f);
    else
      MI_LAUNCH_BEHIND((moe_rows_kernel<false>), g, 32 * MR_WARPS, 0, stream, (const bf16*)act, ff, (const bf16*)w_down,
                (const bf16*)nullptr, w_expert_stride, (const int*)nullptr, 1, plan, E, (void*)y, H, ff, 0.f, 0.f, 0.f);
    MI_RETURN_LAUNCH_STATUS();
  }
  dim3 grid((H + TILE_N - 1) / TILE_N, max_tiles(n_entries, E, TILE_M));
  if (grid.y > 65535) MI_REFUSE("moe: too many row tiles for one launch");
  if (dtype == MI_DTYPE_F32)
    MI_LAUNCH((moe_gemm_kernel<float, false>), grid, 256, 0, stream, (const float*)act, ff, (const float*)w_down,
              (const float*)nullptr, w_expert_stride, (const int*)nullptr, 1, plan, E, (void*)y, H, ff, 0.f, 0.f, 0.f);
  else if (dtype == MI_DTYPE_BF16)
    MI_LAUNCH((moe_gemm_mma_kernel<false>), grid, 128, 0, stream, (const bf16*)act, ff, (const bf16*)w_down,
              (const bf16*)nullptr, w_expert_stride, (const int*)nullptr, 1, plan, E, (void*)y, H, ff, 0.f, 0.f, 0.f,
              mma_vec_ok(act, ff, w_down, nullptr, ff));
  else
    MI_REFUSE("moe: unknown dtype %d", dtype);
  MI_RETURN_LAUNCH_STATUS();
}

// ------------------------------------------------------------------------------------------ gather, combine
// xs[pos, :] = x[perm[pos] / top, :]: an expert's rows side by side, for a library's grouped product
template <typename T>
__global__ void moe_gather_kernel(const T* __restrict__ x, int x_stride, const int* __restrict__ perm, int top,
                                  T* __restrict__ xs, int H, int vec) {
  mi_pdl_enter();
  const int pos = blockIdx.x;
  const T* src = x + (size_t)(perm[pos] / top) * x_stride;
  T* dst = xs + (size_t)pos * H;
  if (vec) {
    constexpr int EPC = 16 / (int)sizeof(T);
    for (int c = threadIdx.x * EPC; c < H; c += blockDim.x * EPC)
      *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
  } else {
    for (int c = threadIdx.x; c < H; c += blockDim.x) dst[c] = src[c];
  }
}

extern "C" int mi_moe_gather(const void* x, int x_stride, const int* perm, int top, void* xs, int n, int H, int dtype,
                             cudaStream_t stream) {
  if (n <= 0) return 0;
  const int es = dtype == MI_DTYPE_F32 ? 4 : 2;
  const int epc = 16 / es;
  const int vec = (H % epc == 0) && (x_stride % epc == 0) && mi_aligned(x, 16) && mi_aligned(xs, 16);
  if (dtype == MI_DTYPE_F32)
    MI_LAUNCH((moe_gather_kernel<float>), n, 128, 0, stream, (const float*)x, x_stride, perm, top, (float*)xs, H, vec);
  else if (dtype == MI_DTYPE_BF16)
    MI_LAUNCH((moe_gather_kernel<bf16>), n, 128, 0, stream, (const bf16*)x, x_stride, perm, top, (bf16*)xs, H, vec);
  else
    MI_REFUSE("moe: unknown dtype %d", dtype);
  MI_RETURN_LAUNCH_STATUS();
}

template <typename T, typename YT>
__global__ void moe_combine_kernel(const YT* __restrict__ y, const int* __restrict__ inv,
                                   const float* __restrict__ weights, const T* __restrict__ shared, int shared_stride,
                                   T* __restrict__ out, int H, int top, const float* __restrict__ shared_gate,
                                   int gate_stride) {
  mi_pdl_enter();
  const int t = blockIdx.x;
  // shared_gate: one fp32 number per token whose sigmoid multiplies the shared expert's output
  const float sg = (shared && shared_gate) ? 1.f / (1.f + expf(-shared_gate[(size_t)t * gate_stride])) : 1.f;
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float acc = 0.f;
    for (int k = 0; k < top; ++k) {
      const int row = inv[(size_t)t * top + k];
      acc = row < 0 ? __int_as_float(0x7fc00000) : fmaf(weights[(size_t)t * top + k], mi_to_float(y[(size_t)row * H + c]), acc);
    }
    if (shared) acc = fmaf(sg, mi_to_float(shared[(size_t)t * shared_stride + c]), acc);
    out[(size_t)t * H + c] = mi_from_float<T>(acc);
  }
}

// the same with four columns per access (sums in the same order)
template <typename T, typename YT>
__global__ void moe_combine4_kernel(const YT* __restrict__ y, const int* __restrict__ inv,
                                    const float* __restrict__ weights, const T* __restrict__ shared, int shared_stride,
                                    T* __restrict__ out, int H, int top, const float* __restrict__ shared_gate,
                                    int gate_stride) {
  mi_pdl_enter();
  __shared__ int rows[32];
  __shared__ float wts[32];
  const int t = blockIdx.x;
  if (threadIdx.x < top) {
    const int row = inv[(size_t)t * top + threadIdx.x];      // (a weight of NaN for an id that is no expert's)
    rows[threadIdx.x] = max(row, 0);
    wts[threadIdx.x] = row < 0 ? __int_as_float(0x7fc00000) : weights[(size_t)t * top + threadIdx.x];
  }
  const float sg = (shared && shared_gate) ? 1.f / (1.f + expf(-shared_gate[(size_t)t * gate_stride])) : 1.f;
  __syncthreads();
  for (int c = 4 * threadIdx.x; c < H; c += 4 * blockDim.x) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f}, f[4];
    for (int k0 = 0; k0 < top; k0 += 4) {              // four experts' pieces in flight
      Vec4<YT> v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k0 + u < top) v[u].load(y + (size_t)rows[k0 + u] * H + c);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k0 + u < top) {
          v[u].get(f);
          const float w = wts[k0 + u];
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i] = fmaf(w, f[i], acc[i]);
        }
    }
    if (shared) {
      Vec4<T> v;
      v.load(shared + (size_t)t * shared_stride + c);
      v.get(f);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] = fmaf(sg, f[i], acc[i]);
    }
    Vec4<T> o;
    o.set(acc);
    o.store(out + (size_t)t * H + c);
  }
}

// y_dtype: the experts' outputs are fp32 (own products) or in the compute dtype (a library's grouped product)
extern "C" int mi_moe_combine(const void* y, int y_dtype, const int* inv, const float* weights, const void* shared,
                              int shared_stride, void* out, int M, int H, int top, const float* shared_gate,
                              int gate_stride, int dtype, cudaStream_t stream) {
  if (M <= 0) return 0;
  const int threads = H >= 1024 ? 256 : 128;
  if (dtype == MI_DTYPE_BF16 && H % 4 == 0 && top <= 32 && mi_aligned(y, 16) && mi_aligned(out, 8) && mi_aligned(shared, 8) &&
      (!shared || shared_stride % 4 == 0) && (y_dtype == MI_DTYPE_F32 || y_dtype == MI_DTYPE_BF16)) {
    const int t4 = H >= 4096 ? 512 : (H >= 1024 ? 256 : 128);
    if (y_dtype == MI_DTYPE_F32)
      MI_LAUNCH((moe_combine4_kernel<bf16, float>), M, t4, 0, stream, (const float*)y, inv, weights, (const bf16*)shared,
                shared_stride, (bf16*)out, H, top, shared_gate, gate_stride);
    else
      MI_LAUNCH((moe_combine4_kernel<bf16, bf16>), M, t4, 0, stream, (const bf16*)y, inv, weights, (const bf16*)shared,
                shared_stride, (bf16*)out, H, top, shared_gate, gate_stride);
    MI_RETURN_LAUNCH_STATUS();
  }
  if (dtype == MI_DTYPE_F32 && y_dtype == MI_DTYPE_F32)
    MI_LAUNCH((moe_combine_kernel<float, float>), M, threads, 0, stream, (const float*)y, inv, weights,
              (const float*)shared, shared_stride, (float*)out, H, top, shared_gate, gate_stride);
  else if (dtype == MI_DTYPE_BF16 && y_dtype == MI_DTYPE_F32)
    MI_LAUNCH((moe_combine_kernel<bf16, float>), M, threads, 0, stream, (const float*)y, inv, weights,
              (const bf16*)shared, shared_stride, (bf16*)out, H, top, shared_gate, gate_stride);
  else if (dtype == MI_DTYPE_BF16 && y_dtype == MI_DTYPE_BF16)
    MI_LAUNCH((moe_combine_kernel<bf16, bf16>), M, threads, 0, stream, (const bf16*)y, inv, weights,
              (const bf16*)shared, shared_stride, (bf16*)out, H, top, shared_gate, gate_stride);
  else
    MI_REFUSE("moe: unsupported dtypes %d (activations) and %d (expert outputs)", dtype, y_dtype);
  MI_RETURN_LAUNCH_STATUS();
}

// ------------------------------------------------------------------------------------------ dense expert
template <typename T>
__global__ void clamped_glu_kernel(const T* __restrict__ gu, int stride, T* __restrict__ out, int M, int I,
                                   float limit, float alpha, float offset) {
  mi_pdl_enter();
  const size_t n = (size_t)M * I;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(idx / I), c = (int)(idx - (size_t)t * I);
    const float g = mi_to_float(gu[(size_t)t * stride + c]), u = mi_to_float(gu[(size_t)t * stride + I + c]);
    out[idx] = mi_from_float<T>(mi_clamped_glu_value(g, u, limit, alpha, offset));
  }
}

// the same with four outputs per access (grid: column groups x rows)
template <typename T>
__global__ void clamped_glu4_kernel(const T* __restrict__ gu, int stride, T* __restrict__ out, int M, int I,
                                    float limit, float alpha, float offset) {
  mi_pdl_enter();
  const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c >= I) return;
  for (int t = blockIdx.y; t < M; t += gridDim.y) {
    Vec4<T> a, b;
    a.load(gu + (size_t)t * stride + c);
    b.load(gu + (size_t)t * stride + I + c);
    float g[4], u[4];
    a.get(g);
    b.get(u);
#pragma unroll
    for (int i = 0; i < 4; ++i) g[i] = mi_clamped_glu_value(g[i], u[i], limit, alpha, offset);
    a.set(g);
    a.store(out + (size_t)t * I + c);
  }
}

extern "C" int mi_clamped_glu(const void* gu, int stride, void* out, int M, int I, float limit, float alpha,
                              float offset, int dtype, cudaStream_t stream) {
  if (M <= 0 || I <= 0) return 0;
  const size_t n = (size_t)M * I;
  if (dtype == MI_DTYPE_BF16 && I % 4 == 0 && stride % 4 == 0 && mi_aligned(gu, 8) && mi_aligned(out, 8)) {
    const dim3 grid((unsigned)((I / 4 + 127) / 128), (unsigned)(M < 16384 ? M : 16384));
    MI_LAUNCH((clamped_glu4_kernel<bf16>), grid, 128, 0, stream, (const bf16*)gu, stride, (bf16*)out, M, I, limit, alpha, offset);
    MI_RETURN_LAUNCH_STATUS();
  }
  const int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  if (dtype == MI_DTYPE_F32)
    MI_LAUNCH((clamped_glu_kernel<float>), blocks, 256, 0, stream, (const float*)gu, stride, (float*)out, M, I, limit, alpha, offset);
  else if (dtype == MI_DTYPE_BF16)
    MI_LAUNCH((clamped_glu_kernel<bf16>), blocks, 256, 0, stream, (const bf16*)gu, stride, (bf16*)out, M, I, limit, alpha, offset);
  else
    MI_REFUSE("moe: unknown dtype %d", dtype);
  MI_RETURN_LAUNCH_STATUS();
}
