// Gated linear attention over long portions in chunks of 64 tokens, as products instead of a walk.
//
// Per head S_t = diag(alpha_t) S_(t-1) + k_t v_t^T, o_t = S_t^T (q_t * q_scale) (see mi_gla_scan in recurrent.cu for the
// forms of alpha, k and v).  With D_t the product of the chunk's alphas up to and with t, and S the state the chunk begins
// with, per key channel:
//
//   o_t     = (q_t D_t)^T S + sum_(s <= t) P_ts v_s,     P_ts = sum_k q_t k_s D_t / D_s
//   S_end   = D_end S + sum_s (k_s D_end / D_s) v_s^T
//
//   gla_fold_kernel    per (request, chunk, head): sum_s (k_s prod_(r > s) alpha_r) v_s^T and D_end
//   gla_carry_kernel   per state element: the states the chunks begin with, one fused multiply-add per chunk
//   gla_out_kernel     per (request, chunk, head, 128 value columns): the two products of o
//
// Everything is fp32, on fused multiply-adds two columns wide; decays are products of alphas (never differences of
// logarithms) kept to twice that precision, so their error does not grow with how far a channel decays, and sums are taken in
// chains of 16.  Over 1000 tokens o and the state end 1.9 and 1.7e-7 from 64 bits with a decay per channel (2.0 and 1.8 by the
// walk), 1.8 and 1.8 with one per head (3.4 and 4.0), 1.2 and 0.8 with one per token (1.2 and 0.8); single products and one chain
// through all terms: 2.9 and 1.9, 8.0 and 10.0, 2.3 and 1.1.  What bounds it: 2 dk dv multiply-adds per
// token and head with the state and 32 (dk + dv) within the chunk, whose operands come out of shared
// memory 16 bytes at a time and 4 cycles a piece, so that about 0.2 of the fp32 rate is reached (15 TFLOP/s); the
// token-by-token walk does as many at 2.  Per 2000 tokens, walk and here: 4 heads of 128 x 256 824 and 110 us with a decay per
// channel, 752 and 92 with one per head; 32 heads of 128 x 128 1026 and 600, 870 and 459.  Inputs fetched 16 tokens ahead into
// registers: 194 for 176 us of folds, 329 for 307 of outputs; the halves of a chunk's decays one after the other instead of side
// by side: 814 for 588.  Where decays differ by channel the quotient D_t / D_s is taken as (q D_t) (k / D_s) if no
// channel of the chunk falls below 1e-20 (|log alpha| up to 0.72 per token on average); a chunk where one does multiplies
// its pairs' decays out one by one.
#include "common.cuh"

MI_DEFINE_ERROR_API()

#define GC_T 64                // tokens per chunk
#define GC_W 128               // key channels and value columns per tile
#define GC_PITCH (GC_W + 4)
#define GC_PP (GC_T + 4)       // row pitch of the pair weights
#define GC_SLAB 32             // rows of S or v staged at a time
// Terms per chain of additions; the chains' sums are added up.  Distance of o from 64 bits over 1000 tokens (a decay per channel,
// per head, per token) with one chain through all channels and keys, chains of 32, of 16 and of 8: 2.7, 2.1, 1.9, 1.9e-7; 2.9,
// 2.0, 1.9, 1.9e-7; 2.2, 1.4, 1.3, 1.3e-7 (by the walk 2.0, 3.4 and 1.2e-7), at 107, 107, 109 and 112 us.
#define GC_CHAIN 16
#define GC_THREADS 256
#define GC_SMALLEST 1e-20f     // leaves 1e18 on either side for k / D and q D before fp32 ends

struct GlaArgs {
  const void *q, *k, *v;
  int qk_stride, stride;
  const float* z;
  int z_stride;
  const float* z_bias;
  float inv_tau, q_scale;
  float* state;
  long long state_stride;
  const int *q_start, *q_len, *state_slot;
  float* o;
  int o_stride, n_requests, heads, dk, dv, extra_col, longer_than;
  float* scratch;              // per (chunk, head): D_end [dk], then [dk][dv]
  const float *head_decay, *tok_gates;
};

__device__ __forceinline__ float gc_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float gc_alpha(const GlaArgs& a, int head, size_t m, int ch) {
  if (a.tok_gates) return a.tok_gates[(m * a.heads + head) * 3];
  if (a.head_decay) return a.head_decay[head];
  const float zz = a.z[m * a.z_stride + head * a.dk + ch] + (a.z_bias ? a.z_bias[head * a.dk + ch] : 0.f);
  return expf(-gc_softplus(-zz) * a.inv_tau);        // sigmoid(zz)^(1/tau)
}
template <typename TQ>
__device__ __forceinline__ float gc_key(const GlaArgs& a, int head, size_t m, int ch) {
  const float k = mi_to_float(reinterpret_cast<const TQ*>(a.k)[m * a.qk_stride + head * a.dk + ch]);
  return a.tok_gates ? k * a.tok_gates[(m * a.heads + head) * 3 + 1] : k;
}
template <typename T>
__device__ __forceinline__ float gc_value(const GlaArgs& a, int head, size_t m, int j) {
  const int dv_in = a.dv - a.extra_col;
  return j < dv_in ? mi_to_float(reinterpret_cast<const T*>(a.v)[m * a.stride + head * dv_in + j]) : (j < a.dv ? 1.f : 0.f);
}
__device__ __forceinline__ float* gc_unit(const GlaArgs& a, int number, int head) {
  return a.scratch + ((size_t)number * a.heads + head) * ((size_t)a.dk + (size_t)a.dk * a.dv);
}

// The step's chunks are numbered through: request after request, those alone whose portion is longer than
// a.longer_than.  A block works out by itself where chunk `number`, or with `of_request` the number-th such request,
// lies (a scan over the requests' lengths, 256 at a time, below 1 us against some 80 of a block's work), so that grid
// and scratch are as large as the step's chunks are many and nothing comes from the host.  All threads of the block.
struct GcPlace { int req, chunk, first; };      // first: the number of the request's first chunk
__device__ __forceinline__ bool gc_find(const GlaArgs& a, int number, bool of_request, GcPlace& at) {
  __shared__ int found[3], totals[GC_THREADS / 32][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int chunks = 0, requests = 0;                 // in front of this turn's
  if (tid == 0) found[0] = -1;
  for (int r0 = 0; r0 < a.n_requests; r0 += GC_THREADS) {
    const int len = r0 + tid < a.n_requests ? a.q_len[r0 + tid] : 0;
    const int c = len > a.longer_than ? (len + GC_T - 1) / GC_T : 0, one = c > 0 ? 1 : 0;
    int cs = c, rs = one;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, cs, o), v = __shfl_up_sync(0xffffffffu, rs, o);
      if (lane >= o) {
        cs += u;
        rs += v;
      }
    }
    __syncthreads();
    if (lane == 31) {
      totals[warp][0] = cs;
      totals[warp][1] = rs;
    }
    __syncthreads();
    int cb = chunks + cs - c, rb = requests + rs - one;
#pragma unroll
    for (int w = 0; w < GC_THREADS / 32; ++w) {
      if (w < warp) {
        cb += totals[w][0];
        rb += totals[w][1];
      }
      chunks += totals[w][0];
      requests += totals[w][1];
    }
    if (one && (of_request ? rb == number : number >= cb && number < cb + c)) {
      found[0] = r0 + tid;
      found[1] = of_request ? 0 : number - cb;
      found[2] = cb;
    }
  }
  __syncthreads();
  at.req = found[0];
  at.chunk = found[1];
  at.first = found[2];
  return at.req >= 0;
}

__device__ __forceinline__ uint64_t gc_pack(float x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void gc_unpack(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void gc_mul2(uint64_t& d, uint64_t a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ void gc_add2(uint64_t& d, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ void gc_fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// A product of decays to twice fp32's precision: 64 roundings one after the other leave 2e-6, and all on one side where
// the decay is a fixed one, against one of a token's own in a walk.
struct GcDecay {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float a) {
    const float h = __fmul_rn(hi, a), l = fmaf(lo, a, fmaf(hi, a, -h));
    hi = __fadd_rn(h, l);
    lo = __fadd_rn(l, -__fadd_rn(hi, -h));
  }
  // x times the product, rounded once (an infinite x stays infinite: its remainder would be inf - inf)
  __device__ __forceinline__ float of(float x) const {
    const float h = __fmul_rn(x, hi);
    return isinf(h) ? h : __fadd_rn(h, fmaf(x, lo, fmaf(x, hi, -h)));
  }
};

// ------------------------------------------------------------------------------------------ the chunks' own part of S
template <typename TQ, typename T>
__global__ void __launch_bounds__(GC_THREADS) gla_fold_kernel(const GlaArgs a) {
  mi_pdl_enter();
  extern __shared__ __align__(16) float gsm[];
  float* ks = gsm;                              // [GC_T][GC_PITCH]
  float* vs = ks + GC_T * GC_PITCH;             // [GC_T][GC_PITCH]
  __shared__ float2 tail[GC_W];
  const int col_tiles = (a.dv + GC_W - 1) / GC_W;
  const int r0 = (blockIdx.z / col_tiles) * GC_W, j0 = (blockIdx.z % col_tiles) * GC_W, head = blockIdx.y;
  GcPlace at;
  if (!gc_find(a, blockIdx.x, false, at)) return;
  const int n = min(GC_T, a.q_len[at.req] - at.chunk * GC_T);
  const size_t m0 = (size_t)a.q_start[at.req] + (size_t)at.chunk * GC_T;
  const int tid = threadIdx.x, ch = tid & (GC_W - 1), half = tid >> 7;
  const bool mine = r0 + ch < a.dk;
  // k times the decays of the tokens behind it: 32 tokens per thread from the end, then the later half's whole decay
  GcDecay p;
#pragma unroll 8
  for (int t = half * 32 + 31; t >= half * 32; --t) {
    float kv = 0.f, al = 1.f;
    if (mine && t < n) {
      kv = gc_key<TQ>(a, head, m0 + t, r0 + ch);
      al = gc_alpha(a, head, m0 + t, r0 + ch);
    }
    ks[t * GC_PITCH + ch] = p.of(kv);
    p.times(al);
  }
  if (half == 1) tail[ch] = make_float2(p.hi, p.lo);
  for (int i = tid; i < GC_T * GC_W; i += GC_THREADS) {
    const int t = i >> 7, j = j0 + (i & (GC_W - 1));
    vs[t * GC_PITCH + (i & (GC_W - 1))] = t < n && j < a.dv ? gc_value<T>(a, head, m0 + t, j) : 0.f;
  }
  __syncthreads();
  float* unit = gc_unit(a, blockIdx.x, head);
  if (half == 0) {
    const float2 f = tail[ch];
    for (int t = 0; t < 32; ++t) ks[t * GC_PITCH + ch] *= f.x;
    if (j0 == 0 && mine) unit[r0 + ch] = (float)(((double)p.hi + p.lo) * ((double)f.x + f.y));
  }
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  uint64_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
#pragma unroll 4
  for (int t = 0; t < GC_T; ++t) {
    const float4 k0 = *reinterpret_cast<const float4*>(ks + t * GC_PITCH + ty * 4);
    const float4 k1 = *reinterpret_cast<const float4*>(ks + t * GC_PITCH + 64 + ty * 4);
    const ulonglong2 v0 = *reinterpret_cast<const ulonglong2*>(vs + t * GC_PITCH + tx * 4);
    const ulonglong2 v1 = *reinterpret_cast<const ulonglong2*>(vs + t * GC_PITCH + 64 + tx * 4);
    const float kk[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint64_t w = gc_pack(kk[i]);
      gc_fma2(acc[i][0], w, v0.x);
      gc_fma2(acc[i][1], w, v0.y);
      gc_fma2(acc[i][2], w, v1.x);
      gc_fma2(acc[i][3], w, v1.y);
    }
  }
  float* B = unit + a.dk;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = r0 + (i >> 2) * 64 + ty * 4 + (i & 3);
    if (row >= a.dk) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = j0 + (j >> 1) * 64 + tx * 4 + (j & 1) * 2;
      float x, y;
      gc_unpack(acc[i][j], x, y);
      if (col < a.dv) B[(size_t)row * a.dv + col] = x;
      if (col + 1 < a.dv) B[(size_t)row * a.dv + col + 1] = y;
    }
  }
}

// ------------------------------------------------------------------------------------------ the states in between
// One thread per state element; a chunk's place in the scratch receives the state that the chunk begins with.  The loads
// do not depend on the chain and run eight chunks ahead.
__global__ void __launch_bounds__(GC_THREADS) gla_carry_kernel(const GlaArgs a) {
  mi_pdl_enter();
  const int head = blockIdx.y;
  GcPlace at;
  if (!gc_find(a, blockIdx.z, true, at)) return;
  const long long e = (long long)blockIdx.x * GC_THREADS + threadIdx.x, elems = (long long)a.dk * a.dv;
  if (e >= elems) return;
  const int chunks = (a.q_len[at.req] + GC_T - 1) / GC_T;
  float* S = a.state + (size_t)a.state_slot[at.req] * a.state_stride + (size_t)head * elems + e;
  const size_t step = (size_t)a.heads * (a.dk + elems);
  float* unit = gc_unit(a, at.first, head);
  const float* A = unit + e / a.dv;
  float* B = unit + a.dk + e;
  float s = *S;
  for (int c0 = 0; c0 < chunks; c0 += 8) {
    float av[8], bv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool in = c0 + i < chunks;
      av[i] = in ? A[(c0 + i) * step] : 1.f;
      bv[i] = in ? B[(c0 + i) * step] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (c0 + i < chunks) {
        B[(c0 + i) * step] = s;
        s = fmaf(av[i], s, bv[i]);
      }
    }
  }
  *S = s;
}

// ------------------------------------------------------------------------------------------ the outputs
// acc[4][4] (rows 4 ty.., two columns each: 4 tx.. and 64 + 4 tx..) += rows [.][k] times mat [k][columns], `depth` of k,
// GC_CHAIN at most, as a sum of their own; with `own` four more k, row i taking the first i + 1 of them (a token's own key
// and those before it: what a later token brings must not reach it, not even as zero times an infinity)
struct GcNo { static constexpr bool value = false; };
struct GcYes { static constexpr bool value = true; };
__device__ __forceinline__ void gc_product(uint64_t (&acc)[4][4], const float* rows, int pitch, const float* mat, int depth,
                                           bool own, int tx) {
  uint64_t sum[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[i][j] = 0;
  auto four = [&](int k, auto triangle) {
    float4 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const float4*>(rows + i * pitch + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(mat + (k + kk) * GC_PITCH + tx * 4);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(mat + (k + kk) * GC_PITCH + 64 + tx * 4);
#pragma unroll
      for (int i = decltype(triangle)::value ? kk : 0; i < 4; ++i) {
        const uint64_t w = gc_pack(kk == 0 ? r[i].x : kk == 1 ? r[i].y : kk == 2 ? r[i].z : r[i].w);
        gc_fma2(sum[i][0], w, b0.x);
        gc_fma2(sum[i][1], w, b0.y);
        gc_fma2(sum[i][2], w, b1.x);
        gc_fma2(sum[i][3], w, b1.y);
      }
    }
  };
#pragma unroll 2
  for (int k = 0; k < depth; k += 4) four(k, GcNo());
  if (own) four(depth, GcYes());
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) gc_add2(acc[i][j], sum[i][j]);
}

// SCALAR: the decay is one number per token for all channels (tok_gates, head_decay).  Then it is left out of the products: the
// state's part of a token is multiplied by D_t behind them and a pair's weight by the product of the decays between its two
// tokens, so that no quotient is taken and no decay is too small.
template <typename TQ, typename T, bool SCALAR>
__global__ void __launch_bounds__(GC_THREADS, 2) gla_out_kernel(const GlaArgs a) {
  mi_pdl_enter();
  extern __shared__ __align__(16) float gsm[];
  float* qs = gsm;                              // [GC_T][GC_PITCH]  q D (SCALAR: q)
  float* ks = qs + GC_T * GC_PITCH;             // [GC_T][GC_PITCH]  k / D (SCALAR: k)
  float* slab = ks + GC_T * GC_PITCH;           // [GC_SLAB][GC_PITCH]
  float* ps = slab + GC_SLAB * GC_PITCH;        // [GC_T][GC_PP]
  __shared__ float tail[SCALAR ? 1 : GC_W], decay[SCALAR ? GC_T : 1], from_start[SCALAR ? GC_T : 1];
  const int j0 = blockIdx.z * GC_W, head = blockIdx.y;
  GcPlace at;
  if (!gc_find(a, blockIdx.x, false, at)) return;
  const int n = min(GC_T, a.q_len[at.req] - at.chunk * GC_T);
  const size_t m0 = (size_t)a.q_start[at.req] + (size_t)at.chunk * GC_T;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, ch = tid & (GC_W - 1), half = tid >> 7;
  const float* S = gc_unit(a, blockIdx.x, head) + a.dk;
  const TQ* q = reinterpret_cast<const TQ*>(a.q);

  uint64_t acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  for (int i = tid; i < GC_T * GC_PP; i += GC_THREADS) ps[i] = 0.f;
  if (SCALAR && tid < GC_T) decay[tid] = tid < n ? gc_alpha(a, head, m0 + tid, 0) : 1.f;

  for (int c0 = 0; c0 < a.dk; c0 += GC_W) {      // 128 key channels at a time
    const bool mine = c0 + ch < a.dk;
    if (c0) __syncthreads();
    bool quotient = true;
    if (SCALAR) {
#pragma unroll 8
      for (int t = half * 32; t < half * 32 + 32; ++t) {
        float qv = 0.f, kv = 0.f;
        if (mine && t < n) {
          qv = mi_to_float(q[(m0 + t) * a.qk_stride + head * a.dk + c0 + ch]) * a.q_scale;
          kv = gc_key<TQ>(a, head, m0 + t, c0 + ch);
        }
        qs[t * GC_PITCH + ch] = qv;
        ks[t * GC_PITCH + ch] = kv;
      }
    } else {
      // D of every token: 32 tokens per thread, then the earlier half's whole decay
      GcDecay p;
#pragma unroll 8
      for (int t = half * 32; t < half * 32 + 32; ++t) {
        if (mine && t < n) p.times(gc_alpha(a, head, m0 + t, c0 + ch));
        qs[t * GC_PITCH + ch] = p.hi;
      }
      if (half == 0) tail[ch] = p.hi;
      __syncthreads();
      const float f = half ? tail[ch] : 1.f;
      quotient = __syncthreads_and(p.hi * f >= GC_SMALLEST) != 0;
#pragma unroll 8
      for (int t = half * 32; t < half * 32 + 32; ++t) {
        float qv = 0.f, kv = 0.f;
        const float d = qs[t * GC_PITCH + ch] * f;
        if (mine && t < n) {
          qv = mi_to_float(q[(m0 + t) * a.qk_stride + head * a.dk + c0 + ch]) * a.q_scale;
          kv = gc_key<TQ>(a, head, m0 + t, c0 + ch);
        }
        qs[t * GC_PITCH + ch] = qv * d;
        ks[t * GC_PITCH + ch] = quotient ? kv / d : kv;
      }
    }
    __syncthreads();
    // the pairs' weights (a pair's weight counts from the key's token on), GC_CHAIN channels at a time
    if (quotient) {
      for (int k0 = 0; k0 < GC_W; k0 += GC_CHAIN) {
        float pair[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) pair[i][j] = 0.f;
#pragma unroll 2
        for (int k = k0; k < k0 + GC_CHAIN; k += 4) {
          float4 r[4], c[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const float4*>(qs + (ty * 4 + i) * GC_PITCH + k);
#pragma unroll
          for (int j = 0; j < 4; ++j) c[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * GC_PITCH + k);
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              pair[i][j] = fmaf(r[i].x, c[j].x, pair[i][j]);
              pair[i][j] = fmaf(r[i].y, c[j].y, pair[i][j]);
              pair[i][j] = fmaf(r[i].z, c[j].z, pair[i][j]);
              pair[i][j] = fmaf(r[i].w, c[j].w, pair[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int t = ty * 4 + i, s = tx + 16 * j;
            if (s <= t) ps[t * GC_PP + s] += pair[i][j];
          }
      }
    } else if (!SCALAR) {
      // A channel all but dies within the chunk: every key is carried on token by token, four threads per key with every
      // fourth 16 bytes of its channels, in registers; decays and then queries come out of shared memory, where all keys of
      // a warp read the same ones.  (A warp per key, each of its pairs anew from the gates: 32 heads of 128 x 128, 2000
      // tokens, 2652 us; 743 here; 600 where no channel dies, 1026 by the walk.)
      const int lane = tid & 31, key = tid >> 2, part = (tid & 3) * 4;
      float4 w[GC_W / 16];
#pragma unroll
      for (int i = 0; i < GC_W / 16; ++i) w[i] = *reinterpret_cast<const float4*>(ks + key * GC_PITCH + part + 16 * i);
      __syncthreads();
#pragma unroll 8
      for (int t = half * 32; t < half * 32 + 32; ++t) {
        const bool in = mine && t < n;
        qs[t * GC_PITCH + ch] = in ? gc_alpha(a, head, m0 + t, c0 + ch) : 1.f;
        ks[t * GC_PITCH + ch] = in ? mi_to_float(q[(m0 + t) * a.qk_stride + head * a.dk + c0 + ch]) * a.q_scale : 0.f;
      }
      __syncthreads();
      for (int t = key & ~7; t < n; ++t) {                    // (a warp's first key on)
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < GC_W / 16; ++i) {
          const float4 al = *reinterpret_cast<const float4*>(qs + t * GC_PITCH + part + 16 * i);
          const float4 qv = *reinterpret_cast<const float4*>(ks + t * GC_PITCH + part + 16 * i);
          if (t > key) {
            w[i].x *= al.x; w[i].y *= al.y; w[i].z *= al.z; w[i].w *= al.w;
          }
          sum = fmaf(qv.x, w[i].x, sum); sum = fmaf(qv.y, w[i].y, sum);
          sum = fmaf(qv.z, w[i].z, sum); sum = fmaf(qv.w, w[i].w, sum);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if ((lane & 3) == 0 && t >= key) ps[t * GC_PP + key] += sum;
      }
      __syncthreads();
      GcDecay d;                                              // q D, as the state's part reads it
      const float f = half ? tail[ch] : 1.f;
      for (int t = half * 32; t < half * 32 + 32; ++t) {
        d.times(qs[t * GC_PITCH + ch]);
        qs[t * GC_PITCH + ch] = ks[t * GC_PITCH + ch] * (d.hi * f);
      }
    }
    // what the state the chunk began with gives, 32 channels of it at a time
    const int depth = min(GC_W, a.dk - c0);
    for (int k0 = 0; k0 < depth; k0 += GC_SLAB) {
      __syncthreads();
      for (int i = tid; i < GC_SLAB * GC_W; i += GC_THREADS) {
        const int r = i >> 7, j = i & (GC_W - 1);
        slab[r * GC_PITCH + j] = (k0 + r < depth && j0 + j < a.dv) ? S[(size_t)(c0 + k0 + r) * a.dv + j0 + j] : 0.f;
      }
      __syncthreads();
      for (int u = 0; u < GC_SLAB; u += GC_CHAIN)
        gc_product(acc, qs + (ty * 4) * GC_PITCH + k0 + u, GC_PITCH, slab + u * GC_PITCH, GC_CHAIN, false, tx);
    }
  }
  if (SCALAR) {
    __syncthreads();
    if (tid <= GC_T) {       // thread s: the decays behind key s, thread 64: those from the chunk's beginning on
      GcDecay p;
      for (int t = tid < GC_T ? tid + 1 : 0; t < n; ++t) {
        p.times(decay[t]);
        if (tid < GC_T) ps[t * GC_PP + tid] *= p.hi;
        else from_start[t] = p.hi;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t d = gc_pack(ty * 4 + i < n ? from_start[ty * 4 + i] : 0.f);
#pragma unroll
      for (int j = 0; j < 4; ++j) gc_mul2(acc[i][j], d);
    }
  }
  // the chunk's own keys
  for (int s0 = 0; s0 < n; s0 += GC_SLAB) {
    __syncthreads();
    for (int i = tid; i < GC_SLAB * GC_W; i += GC_THREADS) {
      const int r = i >> 7, j = i & (GC_W - 1);
      slab[r * GC_PITCH + j] = (s0 + r < n && j0 + j < a.dv) ? gc_value<T>(a, head, m0 + s0 + r, j0 + j) : 0.f;
    }
    __syncthreads();
    for (int u = 0; u < GC_SLAB; u += GC_CHAIN) {
      const int before = ty * 4 - s0 - u;      // keys of this chain in front of the rows' own four
      if (before >= 0)
        gc_product(acc, ps + (ty * 4) * GC_PP + s0 + u, GC_PP, slab + u * GC_PITCH, min(GC_CHAIN, before), before < GC_CHAIN, tx);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty * 4 + i;
    if (t >= n) continue;
    float* dst = a.o + (m0 + t) * a.o_stride + head * a.dv;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = j0 + (j >> 1) * 64 + tx * 4 + (j & 1) * 2;
      float x, y;
      gc_unpack(acc[i][j], x, y);
      if (col < a.dv) dst[col] = x;
      if (col + 1 < a.dv) dst[col + 1] = y;
    }
  }
}

// ------------------------------------------------------------------------------------------ host

extern "C" int mi_gla_chunk_tokens() { return GC_T; }

// floats of scratch for this many chunks
extern "C" long long mi_gla_chunks_scratch(int total_chunks, int heads, int dk, int dv) {
  return (long long)total_chunks * heads * ((long long)dk + (long long)dk * dv);
}

template <typename TQ, typename T>
static cudaError_t gla_chunks_launch(const GlaArgs& a, int total_chunks, int n_long, cudaStream_t stream) {
  const int col_tiles = (a.dv + GC_W - 1) / GC_W, row_tiles = (a.dk + GC_W - 1) / GC_W;
  const size_t fold_smem = (size_t)2 * GC_T * GC_PITCH * sizeof(float);
  const size_t out_smem = ((size_t)(2 * GC_T + GC_SLAB) * GC_PITCH + (size_t)GC_T * GC_PP) * sizeof(float);
  auto fold = gla_fold_kernel<TQ, T>;
  auto out = a.tok_gates || a.head_decay ? gla_out_kernel<TQ, T, true> : gla_out_kernel<TQ, T, false>;
  cudaError_t e = cudaFuncSetAttribute(fold, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fold_smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(out, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
  if (e != cudaSuccess) return e;
  e = MI_LAUNCH(fold, dim3(total_chunks, a.heads, col_tiles * row_tiles), GC_THREADS, fold_smem, stream, a);
  if (e != cudaSuccess) return e;
  const long long elems = (long long)a.dk * a.dv;
  e = MI_LAUNCH(gla_carry_kernel, dim3((unsigned)((elems + GC_THREADS - 1) / GC_THREADS), a.heads, n_long), GC_THREADS, 0,
                stream, a);
  if (e != cudaSuccess) return e;
  return MI_LAUNCH(out, dim3(total_chunks, a.heads, col_tiles), GC_THREADS, out_smem, stream, a);
}

// The portions longer than `longer_than`; arguments as mi_gla_scan (recurrent.cu).  n_long: how many these are, total_chunks:
// how many chunks of 64 tokens they make together, scratch as mi_gla_chunks_scratch says.  Three launches.
extern "C" int mi_gla_chunks(const void* q, const void* k, int qk_stride, int qk_dtype, const void* v, int stride,
                             const float* z, int z_stride, const float* z_bias, float inv_tau, float q_scale, float* state,
                             long long state_stride, const int* q_start, const int* q_len, const int* state_slot, float* o,
                             int o_stride, int n_requests, int heads, int dk, int dv, float* scratch, int total_chunks, int n_long, int longer_than,
                             const float* head_decay, const float* tok_gates, int extra_col, int dtype,
                             cudaStream_t stream) {
  if (n_requests <= 0 || total_chunks <= 0 || n_long <= 0) return 0;
  if (!z && !head_decay && !tok_gates) MI_REFUSE("gla: neither decays per channel nor per head nor per token");
  if (extra_col != 0 && extra_col != 1) MI_REFUSE("gla: one extra column or none");
  if (dv - extra_col <= 0) MI_REFUSE("gla: no value columns");
  if (!scratch) MI_REFUSE("gla: chunks need scratch memory");
  if (dk <= 0 || dk > 256 || dv <= 0) MI_REFUSE("gla: key size %d must lie in [1, 256], value size %d above 0", dk, dv);
  if (heads > 65535 || n_long > 65535) MI_REFUSE("gla: too many heads or requests for one launch");
  const GlaArgs a = {q, k, v, qk_stride, stride, z, z_stride, z_bias, inv_tau, q_scale, state, state_stride, q_start, q_len,
                     state_slot, o, o_stride, n_requests, heads, dk, dv, extra_col, longer_than, scratch, head_decay, tok_gates};
  cudaError_t e;
  if (dtype == MI_DTYPE_BF16 && qk_dtype == MI_DTYPE_BF16) e = gla_chunks_launch<bf16, bf16>(a, total_chunks, n_long, stream);
  else if (dtype == MI_DTYPE_BF16 && qk_dtype == MI_DTYPE_F32) e = gla_chunks_launch<float, bf16>(a, total_chunks, n_long, stream);
  else MI_REFUSE("gla: dtypes %d (q, k) and %d (v) are not taken together in chunks", qk_dtype, dtype);
  if (e != cudaSuccess) return (int)e;
  MI_RETURN_LAUNCH_STATUS();
}
