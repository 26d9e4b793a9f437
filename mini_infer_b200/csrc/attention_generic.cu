// Attention over the paged key/value cache, any portion length, CUDA cores, fp32 math.
//
// This is the kernel of the 32-bit path and the plain twin of the tensor-core
// kernels.  One block takes 16 consecutive query tokens of one request and one query
// head, walks that request's keys in chunks of 32 (always cut at absolute multiples of
// 32, so a row's arithmetic never depends on what else is in the batch), and keeps an
// online softmax in fp32.  Keys and values are fetched through the block table; a
// query at absolute position p sees keys j with  max(0, p - window + 1) <= j <= p
// (window = 0: all keys up to p), and with chunk > 0 only those of its own chunk of positions,
// j >= (p / chunk) * chunk.  Keys and values may have different sizes per head (d for
// queries and keys, dv for values and the output); keys of any size that fits in shared memory
// and values up to 512 are taken, sizes that are no multiple of 4 element by element.
//
// `keep` > 0: beside its window a query also sees the first `keep` keys of the sequence; chunks between the two
// are not walked.  `softcap` > 0: a scaled score s becomes softcap tanh(s / softcap).
//
// Three optional extras.  `sinks` [nq]: the softmax's denominator also holds exp(sinks[h]), a
// score without a key or a value that is not scaled and counts once.  `slopes` [nq]: the scaled
// score of query i and key j is lowered by slopes[h] * (i - j).  `v_prefix`: there is no value
// cache; the value of a key is the first dv numbers of the key's own row (dv <= d).
//
// Layouts
//   q    [tokens, q_stride]   head h at columns [h*d, (h+1)*d)
//   out  [tokens, out_stride] head h at columns [h*dv, (h+1)*dv)
//   kcache [pages, nkv, page_size, d], vcache [pages, nkv, page_size, dv]: the page_size keys of
//                  a page lie together per key/value head; the 16-byte chunks of a row are permuted
//                  by the key's in-page offset (mi_swizzled in common.cuh; rows that are no whole
//                  number of chunks are not permuted, mi_swizzle_mask_rows)
//   block_table [rows, bt_stride] page ids; request b uses row table_rows[b] (row b when
//                  table_rows is null);  q_start / q_len / kv_len [requests]
//   tile_req / tile_tok0 [tiles]: request and first token (within the portion) of a tile
#include "common.cuh"

MI_DEFINE_ERROR_API()

#define BQ 16
#define BK 32
#define NTHREADS 128

// whether the instance for values of up to DMAX fetches these rows a chunk ahead (float32 rows of these sizes have
// attention_f32_kernel)
template <typename T, int DMAX>
__host__ __device__ __forceinline__ bool rows_ahead(int d, int dv, int v_prefix) {
  return sizeof(T) == 2 && DMAX <= 128 && d <= DMAX && (d & 3) == 0 && (dv & 3) == 0 && !v_prefix;
}

template <typename T, int DMAX>
__global__ void __launch_bounds__(NTHREADS)
attention_generic_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                         const T* __restrict__ kcache, const T* __restrict__ vcache,
                         const int* __restrict__ block_table, int bt_stride,
                         const int* __restrict__ table_rows, int page_size,
                         const int* __restrict__ q_start, const int* __restrict__ q_len,
                         const int* __restrict__ kv_len, const int* __restrict__ tile_req,
                         const int* __restrict__ tile_tok0, int nq, int nkv, int d, int dv, float scale,
                         int window, int chunk, const float* __restrict__ sinks, const float* __restrict__ slopes,
                         int v_prefix, int keep, float softcap) {
  mi_pdl_enter();   // inputs come from the kernels before this one
  extern __shared__ __align__(16) float smem[];
  float* Vs = smem;                       // [BK][dvp], dvp = dv rounded up to 4 (nothing with v_prefix)
  const int dvp = (dv + 3) & ~3;
  float* Qs = Vs + (v_prefix ? 0 : BK * dvp);   // [BQ][d]
  float* Ks = Qs + BQ * d;                // [BK][d + 1]
  float* Ss = Ks + BK * (d + 1);          // [BQ][BK]
  // With 16-byte pieces and heads of up to 128 the next chunk's rows come into registers while this one is worked on
  // (a chunk of 32 keys took 18 us when every one began with a round trip to the block table and one to its rows).
  constexpr int PRE = sizeof(T) == 2 && DMAX <= 128 ? DMAX / 16 : 0;
  const bool ahead = PRE > 0 && rows_ahead<T, DMAX>(d, dv, v_prefix);
  // per key row of the chunk at hand (and of the next): element offset / d (-1: none) and chunk permutation
  int* rowbase2 = reinterpret_cast<int*>(Ss + BQ * BK);  // [1 or 2][BK]
  int* rowswz2 = rowbase2 + (ahead ? 2 : 1) * BK;        // [1 or 2][BK]
  constexpr int EPC = 16 / (int)sizeof(T);
  const int swz_mask = mi_swizzle_mask_rows(d, (int)sizeof(T));
  const int swz_mask_v = mi_swizzle_mask_rows(dv, (int)sizeof(T));

  const int tid = threadIdx.x;
  const int tile = blockIdx.x / nq, h = blockIdx.x - tile * nq;   // all heads of a tile, then the next tile (the caller lists long tiles first)
  const int kvh = h / (nq / nkv);
  const int b = tile_req[tile], tok0 = tile_tok0[tile];
  const int ql = q_len[b], kl = kv_len[b], qs = q_start[b];
  const int trow = table_rows ? table_rows[b] : b;   // the request's row of the block table
  const int rows = min(BQ, ql - tok0);
  const int p0 = kl - ql + tok0;  // absolute position of the tile's first query
  const int j_end = p0 + rows;    // one past the last visible key
  int j_lo = window > 0 ? max(0, p0 - window + 1) : 0;   // the first row's bound is the lowest of the tile
  if (chunk > 0) j_lo = max(j_lo, (p0 / chunk) * chunk);
  const int dp = d + 1;
  const float* Vrows = v_prefix ? Ks : Vs;   // where the PV product finds a key's value, and its row pitch
  const int vpitch = v_prefix ? dp : dvp;
  const float slope = slopes ? slopes[h] : 0.f;

  for (int idx = tid; idx < BQ * d; idx += NTHREADS) {
    const int r = idx / d, k = idx - r * d;
    Qs[idx] = r < rows ? mi_to_float(q[(size_t)(qs + tok0 + r) * q_stride + h * d + k]) : 0.f;
  }

  const int r = tid >> 3, c = tid & 7;
  const int prow = p0 + r;
  int lo_r = window > 0 ? max(0, prow - window + 1) : 0;
  if (chunk > 0) lo_r = max(lo_r, (prow / chunk) * chunk);
  float m_i = -INFINITY, l_i = 0.f;
  float acc[DMAX / 8];
#pragma unroll
  for (int e = 0; e < DMAX / 8; ++e) acc[e] = 0.f;
  const int ne = (dv + 7) >> 3;

  const MiKeyWalk<true> walk(j_lo, keep, BK);
  const int n_chunks = walk.count(j_end, BK);
  auto locate = [&](int ci) {      // the rows of chunk ci, by the first 32 threads
    const int j = walk.chunk(ci) * BK + tid;
    int base = -1;
    if ((j >= j_lo || j < keep) && j < j_end) {
      const int page = block_table[(size_t)trow * bt_stride + j / page_size];
      base = (page * nkv + kvh) * page_size + j % page_size;
    }
    rowbase2[(ahead ? ci & 1 : 0) * BK + tid] = base;
    rowswz2[(ahead ? ci & 1 : 0) * BK + tid] = (j % page_size);
  };
  Vec4<T> kp[PRE > 0 ? PRE : 1], vp[PRE > 0 ? PRE : 1];
  auto piece = [&](Vec4<T>& to, const T* cache, int idx, int width, int mask, const int* base_of, const int* swz_of) {
    const int w4 = width >> 2, jj = idx / w4, k4 = (idx - jj * w4) << 2;
    const float none[4] = {0.f, 0.f, 0.f, 0.f};
    to.set(none);
    if (jj < BK && base_of[jj] >= 0)
      to.load(cache + (size_t)base_of[jj] * width + ((((k4 / EPC) ^ (swz_of[jj] & mask)) * EPC) + (k4 % EPC)));
  };
  auto fetch = [&](int ci) {
    const int *base_of = rowbase2 + (ci & 1) * BK, *swz_of = rowswz2 + (ci & 1) * BK;
#pragma unroll
    for (int i = 0; i < PRE; ++i) piece(kp[i], kcache, tid + i * NTHREADS, d, swz_mask, base_of, swz_of);
#pragma unroll
    for (int i = 0; i < PRE; ++i) piece(vp[i], vcache, tid + i * NTHREADS, dv, swz_mask_v, base_of, swz_of);
  };
  if (ahead && n_chunks > 0) {
    if (tid < BK) locate(0);
    __syncthreads();
    fetch(0);
  }
  for (int ci = 0; ci < n_chunks; ++ci) {
    const int j0 = walk.chunk(ci) * BK;
    const int *rowbase = rowbase2, *rowswz = rowswz2;      // (read by the loads below, not by those ahead)
    __syncthreads();  // previous chunk fully consumed (and Qs written, first time)
    if (tid < BK && !ahead) locate(ci);
    if (tid < BK && ahead && ci + 1 < n_chunks) locate(ci + 1);
    if (ahead) {
#pragma unroll
      for (int i = 0; i < PRE; ++i) {
        const int idx = tid + i * NTHREADS;
        float f[4];
        const int kj = idx / (d >> 2), vj = idx / (dv >> 2);
        if (kj < BK) {
          kp[i].get(f);
          float* kd = Ks + kj * dp + ((idx - kj * (d >> 2)) << 2);
          kd[0] = f[0]; kd[1] = f[1]; kd[2] = f[2]; kd[3] = f[3];
        }
        if (vj < BK) {
          vp[i].get(f);
          *reinterpret_cast<float4*>(Vs + vj * dvp + ((idx - vj * (dv >> 2)) << 2)) = make_float4(f[0], f[1], f[2], f[3]);
        }
      }
    }
    __syncthreads();
    if (ahead) {
      if (ci + 1 < n_chunks) fetch(ci + 1);
    } else {
    if ((d & 3) == 0) {
      const int d4 = d >> 2;
      for (int idx = tid; idx < BK * d4; idx += NTHREADS) {
        const int jj = idx / d4, k4 = (idx - jj * d4) << 2;
        const int base = rowbase[jj];
        float kf[4] = {0.f, 0.f, 0.f, 0.f};
        if (base >= 0) {
          const size_t off = (size_t)base * d + ((((k4 / EPC) ^ (rowswz[jj] & swz_mask)) * EPC) + (k4 % EPC));
          Vec4<T> kv;
          kv.load(kcache + off);
          kv.get(kf);
        }
        float* kd = Ks + jj * dp + k4;
        kd[0] = kf[0]; kd[1] = kf[1]; kd[2] = kf[2]; kd[3] = kf[3];
      }
    } else {
      for (int idx = tid; idx < BK * d; idx += NTHREADS) {
        const int jj = idx / d, k = idx - jj * d;
        const int base = rowbase[jj];
        Ks[jj * dp + k] = base >= 0 ? mi_to_float(kcache[(size_t)base * d + mi_swizzled(k, rowswz[jj], swz_mask, EPC)]) : 0.f;
      }
    }
    if (v_prefix) {
      // the values are the keys' own first columns, already in Ks
    } else if ((dv & 3) == 0) {
      const int d4 = dv >> 2;
      for (int idx = tid; idx < BK * d4; idx += NTHREADS) {
        const int jj = idx / d4, k4 = (idx - jj * d4) << 2;
        const int base = rowbase[jj];
        float vf[4] = {0.f, 0.f, 0.f, 0.f};
        if (base >= 0) {
          const size_t off = (size_t)base * dv + ((((k4 / EPC) ^ (rowswz[jj] & swz_mask_v)) * EPC) + (k4 % EPC));
          Vec4<T> vv;
          vv.load(vcache + off);
          vv.get(vf);
        }
        *reinterpret_cast<float4*>(Vs + jj * dvp + k4) = make_float4(vf[0], vf[1], vf[2], vf[3]);
      }
    } else {
      for (int idx = tid; idx < BK * dv; idx += NTHREADS) {
        const int jj = idx / dv, k = idx - jj * dv;
        const int base = rowbase[jj];
        Vs[jj * dvp + k] = base >= 0 ? mi_to_float(vcache[(size_t)base * dv + mi_swizzled(k, rowswz[jj], swz_mask_v, EPC)]) : 0.f;
      }
    }
    __syncthreads();
    }

    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const float* qrow = Qs + r * d;
#pragma unroll 8
    for (int k = 0; k < d; ++k) {
      const float qv = qrow[k];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) s[jj] = fmaf(qv, Ks[(c + 8 * jj) * dp + k], s[jj]);
    }
    float mx = -INFINITY;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const int j = j0 + c + 8 * jj;
      const bool ok = (r < rows) && (j <= prow) && (j >= lo_r || j < keep);
      const float raw = s[jj] * scale;
      s[jj] = ok ? (softcap > 0.f ? softcap * tanhf(raw / softcap) : raw) - slope * (float)(prow - j) : -INFINITY;
      mx = fmaxf(mx, s[jj]);
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    const float m_new = fmaxf(m_i, mx);
    float alpha = 1.f, psum = 0.f;
    float p[4] = {0.f, 0.f, 0.f, 0.f};
    if (m_new != -INFINITY) {
      alpha = expf(m_i - m_new);  // m_i = -inf gives 0
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        p[jj] = expf(s[jj] - m_new);  // masked entries give 0
        psum += p[jj];
      }
    }
    psum += __shfl_xor_sync(0xffffffffu, psum, 1);
    psum += __shfl_xor_sync(0xffffffffu, psum, 2);
    psum += __shfl_xor_sync(0xffffffffu, psum, 4);
    l_i = l_i * alpha + psum;
    m_i = m_new;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) Ss[r * BK + c + 8 * jj] = p[jj];
#pragma unroll
    for (int e = 0; e < DMAX / 8; ++e) acc[e] *= alpha;
    __syncthreads();
#pragma unroll 2
    for (int j = 0; j < BK; ++j) {
      const float pj = Ss[r * BK + j];
      const float* vrow = Vrows + j * vpitch + c;
#pragma unroll
      for (int e = 0; e < DMAX / 8; ++e)
        if (e < ne && c + 8 * e < dv) acc[e] = fmaf(pj, vrow[8 * e], acc[e]);
    }
  }
  if (sinks && r < rows) {
    // the sink joins the denominator once, on the scale of the larger of itself and the row's maximum
    const float sink = sinks[h];
    const float m_f = fmaxf(m_i, sink);
    const float keep = (m_i == -INFINITY) ? 0.f : expf(m_i - m_f);
    l_i = l_i * keep + expf(sink - m_f);
#pragma unroll
    for (int e = 0; e < DMAX / 8; ++e) acc[e] *= keep;
  }
  if (r < rows && l_i > 0.f) {
    const float inv = 1.f / l_i;
    T* orow = out + (size_t)(qs + tok0 + r) * out_stride + h * dv + c;
#pragma unroll
    for (int e = 0; e < DMAX / 8; ++e)
      if (e < ne && c + 8 * e < dv) orow[8 * e] = mi_from_float<T>(acc[e] * inv);
  }
}

// ------------------------------------------------------------------------------------------
// float32, keys and values of up to 128 in whole 16-byte pieces: the 32-bit path's kernel.
//
// What bounds it: for prompts the reads of shared memory (16 bytes a lane, 4 cycles a warp: 8 of them for 64 multiply-adds of
// the scores, 5 for 64 of the values), for single tokens the chain of a chunk (128 multiply-adds per score, then 32 per
// column).  So the four warps of a block (16 query tokens of one head) walk the keys side by side: warp w takes the chunks of
// 32 whose number is w modulo 4, with a running maximum, sum and output of its own, and the four are merged in the order of
// the warps.  Which warp adds what, and in which order, depends on a key's position alone, so a row has the same bits
// however the work is cut.  A warp copies its next keys (cp.async) while it works on the values, and the values while it
// works on the scores.  A tile of one token spreads keys and columns over all 32 lanes instead of 4 rows per lane; its
// sums run in the same order.  2 requests of 131 tokens, 16 heads over 4 of 128, in the kernel above and here: four
// launches for the prompts and 16 for single tokens 1.10 and 0.36 ms (here 50 and 10 us each).
// ------------------------------------------------------------------------------------------
#define F32_WARPS 4
#define F32_PPITCH 20        // floats per key of the weights (16 rows)

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool in) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(src), "r"(n) : "memory");
}

// the largest number of the lanes whose indices differ in the bits from lo to hi
__device__ __forceinline__ float lanes_max(float v, int lo, int hi) {
  for (int o = lo; o <= hi; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <int DMAX>
__global__ void __launch_bounds__(32 * F32_WARPS)
attention_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride,
                     const float* __restrict__ kcache, const float* __restrict__ vcache,
                     const int* __restrict__ block_table, int bt_stride, const int* __restrict__ table_rows, int page_size,
                     const int* __restrict__ q_start, const int* __restrict__ q_len, const int* __restrict__ kv_len,
                     const int* __restrict__ tile_req, const int* __restrict__ tile_tok0, int nq, int nkv, int d, int dv,
                     float scale, int window, int chunk, const float* __restrict__ sinks, const float* __restrict__ slopes,
                     int keep, float softcap) {
  mi_pdl_enter();   // inputs come from the kernels before this one
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kp = d + 4;                                  // pitch of query and key rows: eight rows touch every bank once
  float* Qs = smem;                                      // [BQ][kp]
  float* Ks = Qs + BQ * kp + warp * BK * (kp + dv);      // this warp's keys [BK][kp] ...
  float* Vs = Ks + BK * kp;                              // ... values [BK][dv] ...
  float* Ps = smem + BQ * kp + F32_WARPS * BK * (kp + dv) + warp * BK * F32_PPITCH;   // ... and weights [BK][16 rows]
  __shared__ float merge_m[F32_WARPS][BQ], merge_l[F32_WARPS][BQ];

  const int tile = blockIdx.x / nq, h = blockIdx.x - tile * nq;   // all heads of a tile, then the next tile (the caller lists long tiles first)
  const int kvh = h / (nq / nkv);
  const int b = tile_req[tile], tok0 = tile_tok0[tile];
  const int ql = q_len[b], kl = kv_len[b], qs = q_start[b];
  const int* table = block_table + (size_t)(table_rows ? table_rows[b] : b) * bt_stride;
  const int rows = min(BQ, ql - tok0);
  const int p0 = kl - ql + tok0, j_end = p0 + rows;      // the first query's position, one past the last visible key
  int j_lo = window > 0 ? max(0, p0 - window + 1) : 0;   // the first row's bound is the lowest of the tile
  if (chunk > 0) j_lo = max(j_lo, (p0 / chunk) * chunk);
  const float slope = slopes ? slopes[h] : 0.f;
  const MiKeyWalk<true> walk(j_lo, keep, BK);
  const int n_chunks = walk.count(j_end, BK);
  const int swz_k = mi_swizzle_mask_rows(d, 4), swz_v = mi_swizzle_mask_rows(dv, 4);

  // the rows of a chunk: lane j holds key j's row in the caches (-1: not visible to any query) and its offset in the page
  auto locate = [&](int c, int& base, int& off) {
    const int j = c * BK + lane;
    base = -1;
    off = j % page_size;
    if ((j >= j_lo || j < keep) && j < j_end) base = (table[j / page_size] * nkv + kvh) * page_size + off;
  };
  auto copy = [&](float* dst, int pitch, const float* cache, int width, int mask, int base, int off) {
    const int pieces = width >> 2;
    if (32 % pieces == 0) {          // a lane's piece is the same in every row
      const int step = 32 / pieces, piece = lane % pieces;
      int row = lane / pieces;
#pragma unroll 8
      for (int i = 0; i < pieces; ++i, row += step) {
        const int rb = __shfl_sync(0xffffffffu, base, row), ro = __shfl_sync(0xffffffffu, off, row);
        cp_async16_zfill(dst + row * pitch + piece * 4, cache + (size_t)max(rb, 0) * width + ((piece ^ (ro & mask)) << 2), rb >= 0);
      }
    } else {
      for (int i = lane; i < BK * pieces; i += 32) {       // (every lane takes as many turns: BK is 32)
        const int row = i / pieces, piece = i - row * pieces;
        const int rb = __shfl_sync(0xffffffffu, base, row), ro = __shfl_sync(0xffffffffu, off, row);
        cp_async16_zfill(dst + row * pitch + piece * 4, cache + (size_t)max(rb, 0) * width + ((piece ^ (ro & mask)) << 2), rb >= 0);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto next_of = [&](int i) {        // the first chunk of the walk from i on that is this warp's
    while (i < n_chunks && (walk.chunk(i) & (F32_WARPS - 1)) != warp) ++i;
    return i;
  };

  int ci = next_of(0), base = -1, off = 0;
  if (ci < n_chunks) {
    locate(walk.chunk(ci), base, off);
    copy(Ks, kp, kcache, d, swz_k, base, off);
    copy(Vs, dv, vcache, dv, swz_v, base, off);
  }
  for (int idx = tid; idx < (rows == 1 ? d : BQ * d); idx += 32 * F32_WARPS) {
    const int r = idx / d, k = idx - r * d;
    Qs[r * kp + k] = r < rows ? q[(size_t)(qs + tok0 + r) * q_stride + h * d + k] : 0.f;
  }
  __syncthreads();

  const int rg = lane >> 3, c8 = lane & 7;
  // many rows: row rg * 4 + i, keys c8 + 8 jj, columns c8 * 4 + 32 e ..; one row: key `lane`, columns lane * 4 ..
  constexpr int NE = DMAX / 32;
  float m_i[4], l_i[4], acc[4][NE * 4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_i[i] = -INFINITY;
    l_i[i] = 0.f;
#pragma unroll
    for (int e = 0; e < NE * 4; ++e) acc[i][e] = 0.f;
  }
  auto masked = [&](float s, int row, int j) {
    const int p = p0 + row;
    int lo = window > 0 ? max(0, p - window + 1) : 0;
    if (chunk > 0) lo = max(lo, (p / chunk) * chunk);
    // (every rounding is named: the two forms below must not contract it differently)
    float v = __fmul_rn(s, scale);
    if (softcap > 0.f) v = __fmul_rn(softcap, tanhf(v / softcap));
    return row < rows && j <= p && (j >= lo || j < keep) ? fmaf(-slope, (float)(p - j), v) : -INFINITY;
  };
  const bool one = rows == 1;

  while (ci < n_chunks) {
    const int j0 = walk.chunk(ci) * BK;
    const int cn = next_of(ci + 1);
    int base_n = -1, off_n = 0;
    if (cn < n_chunks) locate(walk.chunk(cn), base_n, off_n);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");       // the keys are there; the values may be under way
    __syncwarp();
    if (one) {
      float s = 0.f;
      const float4* kr = reinterpret_cast<const float4*>(Ks + lane * kp);
      const float4* qr = reinterpret_cast<const float4*>(Qs);
#pragma unroll 8
      for (int k = 0; k < (d >> 2); ++k) {
        const float4 kv = kr[k], qv = qr[k];
        s = fmaf(qv.w, kv.w, fmaf(qv.z, kv.z, fmaf(qv.y, kv.y, fmaf(qv.x, kv.x, s))));
      }
      s = masked(s, 0, j0 + lane);
      __syncwarp();
      if (cn < n_chunks) copy(Ks, kp, kcache, d, swz_k, base_n, off_n);
      else asm volatile("cp.async.commit_group;\n" ::: "memory");
      const float m_new = fmaxf(m_i[0], lanes_max(s, 1, 16));
      float alpha = 1.f, p = 0.f;
      if (m_new != -INFINITY) {
        alpha = expf(m_i[0] - m_new);
        p = expf(s - m_new);
      }
      Ps[lane] = p;
      p += __shfl_xor_sync(0xffffffffu, p, 8);
      p += __shfl_xor_sync(0xffffffffu, p, 16);
#pragma unroll
      for (int o = 1; o <= 4; o <<= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
      l_i[0] = fmaf(l_i[0], alpha, p);
      m_i[0] = m_new;
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[0][e] = __fmul_rn(acc[0][e], alpha);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");     // the values
      __syncwarp();
      if (lane * 4 < dv) {
#pragma unroll 8
        for (int j = 0; j < BK; ++j) {
          const float pj = Ps[j];
          const float4 v = *reinterpret_cast<const float4*>(Vs + j * dv + lane * 4);
          acc[0][0] = fmaf(pj, v.x, acc[0][0]);
          acc[0][1] = fmaf(pj, v.y, acc[0][1]);
          acc[0][2] = fmaf(pj, v.z, acc[0][2]);
          acc[0][3] = fmaf(pj, v.w, acc[0][3]);
        }
      }
    } else {
      float s[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) s[i][jj] = 0.f;
      if (rg * 4 < rows) {
        const float* qr = Qs + rg * 4 * kp;
        const float* kr = Ks + c8 * kp;
#pragma unroll 2
        for (int k = 0; k < d; k += 4) {
          float4 qv[4], kv[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(qr + i * kp + k);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) kv[jj] = *reinterpret_cast<const float4*>(kr + 8 * jj * kp + k);
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj)
              s[i][jj] = fmaf(qv[i].w, kv[jj].w, fmaf(qv[i].z, kv[jj].z, fmaf(qv[i].y, kv[jj].y, fmaf(qv[i].x, kv[jj].x, s[i][jj]))));
        }
      }
      __syncwarp();
      if (cn < n_chunks) copy(Ks, kp, kcache, d, swz_k, base_n, off_n);
      else asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float mx = -INFINITY;
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          s[i][jj] = masked(s[i][jj], rg * 4 + i, j0 + c8 + 8 * jj);
          mx = fmaxf(mx, s[i][jj]);
        }
        const float m_new = fmaxf(m_i[i], lanes_max(mx, 1, 4));
        float alpha = 1.f;
        if (m_new != -INFINITY) {
          alpha = expf(m_i[i] - m_new);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) s[i][jj] = expf(s[i][jj] - m_new);
        } else {
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) s[i][jj] = 0.f;
        }
        float psum = (s[i][0] + s[i][1]) + (s[i][2] + s[i][3]);      // (the order of one row's butterfly)
#pragma unroll
        for (int o = 1; o <= 4; o <<= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
        l_i[i] = fmaf(l_i[i], alpha, psum);
        m_i[i] = m_new;
#pragma unroll
        for (int e = 0; e < NE * 4; ++e) acc[i][e] = __fmul_rn(acc[i][e], alpha);
      }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        *reinterpret_cast<float4*>(Ps + (c8 + 8 * jj) * F32_PPITCH + rg * 4) = make_float4(s[0][jj], s[1][jj], s[2][jj], s[3][jj]);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");     // the values
      __syncwarp();
      if (rg * 4 < rows) {
#pragma unroll 4
        for (int j = 0; j < BK; ++j) {
          const float4 p = *reinterpret_cast<const float4*>(Ps + j * F32_PPITCH + rg * 4);
          const float pr[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
          for (int e = 0; e < NE; ++e) {
            if (c8 * 4 + 32 * e >= dv) continue;
            const float4 v = *reinterpret_cast<const float4*>(Vs + j * dv + c8 * 4 + 32 * e);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              acc[i][4 * e] = fmaf(pr[i], v.x, acc[i][4 * e]);
              acc[i][4 * e + 1] = fmaf(pr[i], v.y, acc[i][4 * e + 1]);
              acc[i][4 * e + 2] = fmaf(pr[i], v.z, acc[i][4 * e + 2]);
              acc[i][4 * e + 3] = fmaf(pr[i], v.w, acc[i][4 * e + 3]);
            }
          }
        }
      }
    }
    __syncwarp();
    if (cn < n_chunks) copy(Vs, dv, vcache, dv, swz_v, base_n, off_n);
    ci = cn;
  }

  // the warps' shares, over their own keys' memory, then row by row in the order of the warps
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncwarp();
  float* share = Ks;      // [rows][dv]
  if (one) {
    if (lane * 4 < dv) *reinterpret_cast<float4*>(share + lane * 4) = make_float4(acc[0][0], acc[0][1], acc[0][2], acc[0][3]);
    if (lane == 0) {
      merge_m[warp][0] = m_i[0];
      merge_l[warp][0] = l_i[0];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = rg * 4 + i;
#pragma unroll
      for (int e = 0; e < NE; ++e)
        if (c8 * 4 + 32 * e < dv)
          *reinterpret_cast<float4*>(share + row * dv + c8 * 4 + 32 * e) =
              make_float4(acc[i][4 * e], acc[i][4 * e + 1], acc[i][4 * e + 2], acc[i][4 * e + 3]);
      if (c8 == 0) {
        merge_m[warp][row] = m_i[i];
        merge_l[warp][row] = l_i[i];
      }
    }
  }
  __syncthreads();
  const float* shares = smem + BQ * kp;
  for (int idx = tid; idx < rows * dv; idx += 32 * F32_WARPS) {
    const int row = idx / dv, col = idx - row * dv;
    const float sink = sinks ? sinks[h] : -INFINITY;     // joins the denominator without a key or a value
    float m = sink;
#pragma unroll
    for (int w = 0; w < F32_WARPS; ++w) m = fmaxf(m, merge_m[w][row]);
    float l = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < F32_WARPS; ++w) {
      const float f = merge_m[w][row] == -INFINITY ? 0.f : expf(merge_m[w][row] - m);
      l = fmaf(merge_l[w][row], f, l);
      o = fmaf(shares[w * BK * (kp + dv) + row * dv + col], f, o);
    }
    if (sinks) l += expf(sink - m);
    if (l > 0.f) out[(size_t)(qs + tok0 + row) * out_stride + h * dv + col] = o * (1.f / l);
  }
}

template <int DMAX>
static int launch_f32(const void* q, int q_stride, void* out, int out_stride, const void* kcache, const void* vcache,
                      const int* block_table, int bt_stride, const int* table_rows, int page_size, const int* q_start,
                      const int* q_len, const int* kv_len, const int* tile_req, const int* tile_tok0, int n_tiles, int nq,
                      int nkv, int d, int dv, float scale, int window, int chunk, const float* sinks, const float* slopes,
                      int keep, float softcap, cudaStream_t stream) {
  const size_t smem = ((size_t)BQ * (d + 4) + (size_t)F32_WARPS * BK * (d + 4 + dv) + F32_WARPS * BK * F32_PPITCH) * sizeof(float);
  auto kern = attention_f32_kernel<DMAX>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  MI_LAUNCH((kern), (unsigned)(n_tiles * nq), 32 * F32_WARPS, smem, stream, (const float*)q, q_stride, (float*)out, out_stride,
            (const float*)kcache, (const float*)vcache, block_table, bt_stride, table_rows, page_size, q_start, q_len, kv_len,
            tile_req, tile_tok0, nq, nkv, d, dv, scale, window, chunk, sinks, slopes, keep, softcap);
  return 0;
}

template <typename T, int DMAX>
static int launch(const void* q, int q_stride, void* out, int out_stride, const void* kcache,
                  const void* vcache, const int* block_table, int bt_stride, const int* table_rows, int page_size,
                  const int* q_start, const int* q_len, const int* kv_len, const int* tile_req,
                  const int* tile_tok0, int n_tiles, int nq, int nkv, int d, int dv, float scale, int window,
                  int chunk, const float* sinks, const float* slopes, int v_prefix, int keep, float softcap,
                  cudaStream_t stream) {
  const size_t smem = ((v_prefix ? 0 : (size_t)BK * ((dv + 3) & ~3)) + (size_t)BQ * d + (size_t)BK * (d + 1) + BQ * BK) *
                          sizeof(float) + (rows_ahead<T, DMAX>(d, dv, v_prefix) ? 4 : 2) * BK * sizeof(int);
  auto kern = attention_generic_kernel<T, DMAX>;
  if (smem > 227 * 1024) return MI_REFUSED - 1;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid((unsigned)(n_tiles * nq));
  MI_LAUNCH((kern), grid, NTHREADS, smem, stream, (const T*)q, q_stride, (T*)out, out_stride, (const T*)kcache,
                                         (const T*)vcache, block_table, bt_stride, table_rows, page_size, q_start,
                                         q_len, kv_len, tile_req, tile_tok0, nq, nkv, d, dv, scale, window, chunk, sinks,
                                         slopes, v_prefix, keep, softcap);
  return 0;
}

extern "C" int mi_attention_generic_tile_tokens() { return BQ; }

extern "C" int mi_attention_generic_capped(const void* q, int q_stride, void* out, int out_stride,
                                           const void* kcache, const void* vcache, const int* block_table,
                                           int bt_stride, const int* table_rows, int page_size, const int* q_start,
                                           const int* q_len, const int* kv_len, const int* tile_req,
                                           const int* tile_tok0, int n_tiles, int nq, int nkv, int d, int dv,
                                           float scale, int window, int chunk, int keep, float softcap,
                                           const float* sinks, const float* slopes, int v_prefix, int dtype,
                                           cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (chunk < 0) MI_REFUSE("attention: bad chunk size %d", chunk);
  if (keep < 0 || (keep && chunk) || !(softcap >= 0.f)) MI_REFUSE("attention: bad kept keys %d or cap %f", keep, softcap);
  if (d <= 0 || d > 1024 || dv <= 0 || dv > 512)
    MI_REFUSE("attention: head sizes %d (keys, up to 1024) and %d (values, up to 512) are not taken", d, dv);
  if (v_prefix && dv > d) MI_REFUSE("attention: values of %d cannot be the first columns of keys of %d", dv, d);
  if (!v_prefix && !vcache) MI_REFUSE("attention: no value cache");
  if (nq <= 0 || nkv <= 0 || nq % nkv != 0)
    MI_REFUSE("attention: %d query heads cannot share %d key/value heads", nq, nkv);
  if ((long long)n_tiles * nq > 0x7fffffffLL) MI_REFUSE("attention: too many blocks for one launch");
  if (page_size <= 0 || window < 0) MI_REFUSE("attention: bad page size %d or window %d", page_size, window);
  if (!mi_aligned(kcache, 16) || !mi_aligned(vcache, 16)) MI_REFUSE("attention: cache must be 16-byte aligned");
  int rc;
  // One rule for every step of a model: its rows must not change kernels with the cutting.
  if (dtype == MI_DTYPE_F32 && !v_prefix && d <= 128 && dv <= 128 && d % 4 == 0 && dv % 4 == 0) {
#define MI_F32(DMAX)                                                                                                       \
  rc = launch_f32<DMAX>(q, q_stride, out, out_stride, kcache, vcache, block_table, bt_stride, table_rows, page_size, q_start, \
                        q_len, kv_len, tile_req, tile_tok0, n_tiles, nq, nkv, d, dv, scale, window, chunk, sinks, slopes, \
                        keep, softcap, stream)
    if (dv <= 64) MI_F32(64);
    else MI_F32(128);
#undef MI_F32
    if (rc) return rc;
    MI_RETURN_LAUNCH_STATUS();
  }
#define MI_GO(T, DMAX)                                                                              \
  rc = launch<T, DMAX>(q, q_stride, out, out_stride, kcache, vcache, block_table, bt_stride,        \
                       table_rows, page_size, q_start, q_len, kv_len, tile_req, tile_tok0, n_tiles, nq, nkv, d, dv, \
                       scale, window, chunk, sinks, slopes, v_prefix, keep, softcap, stream)
  if (dtype == MI_DTYPE_F32) {
    if (dv <= 64) MI_GO(float, 64);
    else if (dv <= 128) MI_GO(float, 128);
    else if (dv <= 256) MI_GO(float, 256);
    else MI_GO(float, 512);
  } else if (dtype == MI_DTYPE_BF16) {
    if (dv <= 64) MI_GO(bf16, 64);
    else if (dv <= 128) MI_GO(bf16, 128);
    else if (dv <= 256) MI_GO(bf16, 256);
    else MI_GO(bf16, 512);
  } else {
    MI_REFUSE("attention: unknown dtype %d", dtype);
  }
#undef MI_GO
  if (rc == MI_REFUSED - 1) MI_REFUSE("attention: keys of %d and values of %d do not fit in shared memory", d, dv);
  if (rc) return rc;
  MI_RETURN_LAUNCH_STATUS();
}

extern "C" int mi_attention_generic_masked(const void* q, int q_stride, void* out, int out_stride,
                                           const void* kcache, const void* vcache, const int* block_table,
                                           int bt_stride, const int* table_rows, int page_size, const int* q_start,
                                           const int* q_len, const int* kv_len, const int* tile_req,
                                           const int* tile_tok0, int n_tiles, int nq, int nkv, int d, int dv,
                                           float scale, int window, int chunk, const float* sinks,
                                           const float* slopes, int v_prefix, int dtype, cudaStream_t stream) {
  return mi_attention_generic_capped(q, q_stride, out, out_stride, kcache, vcache, block_table, bt_stride, table_rows,
                                     page_size, q_start, q_len, kv_len, tile_req, tile_tok0, n_tiles, nq, nkv, d, dv,
                                     scale, window, chunk, 0, 0.f, sinks, slopes, v_prefix, dtype, stream);
}

extern "C" int mi_attention_generic_ext(const void* q, int q_stride, void* out, int out_stride,
                                        const void* kcache, const void* vcache, const int* block_table,
                                        int bt_stride, const int* table_rows, int page_size, const int* q_start,
                                        const int* q_len, const int* kv_len, const int* tile_req,
                                        const int* tile_tok0, int n_tiles, int nq, int nkv, int d, int dv,
                                        float scale, int window, const float* sinks, const float* slopes,
                                        int v_prefix, int dtype, cudaStream_t stream) {
  return mi_attention_generic_masked(q, q_stride, out, out_stride, kcache, vcache, block_table, bt_stride, table_rows,
                                     page_size, q_start, q_len, kv_len, tile_req, tile_tok0, n_tiles, nq, nkv, d, dv,
                                     scale, window, 0, sinks, slopes, v_prefix, dtype, stream);
}

extern "C" int mi_attention_generic_kv(const void* q, int q_stride, void* out, int out_stride,
                                       const void* kcache, const void* vcache, const int* block_table,
                                       int bt_stride, const int* table_rows, int page_size, const int* q_start,
                                       const int* q_len, const int* kv_len, const int* tile_req,
                                       const int* tile_tok0, int n_tiles, int nq, int nkv, int d, int dv,
                                       float scale, int window, int dtype, cudaStream_t stream) {
  return mi_attention_generic_ext(q, q_stride, out, out_stride, kcache, vcache, block_table, bt_stride, table_rows,
                                  page_size, q_start, q_len, kv_len, tile_req, tile_tok0, n_tiles, nq, nkv, d, dv,
                                  scale, window, nullptr, nullptr, 0, dtype, stream);
}

// keys and values of one size, a multiple of 16 (what the tensor-core kernels take as well)
extern "C" int mi_attention_generic(const void* q, int q_stride, void* out, int out_stride,
                                    const void* kcache, const void* vcache, const int* block_table,
                                    int bt_stride, const int* table_rows, int page_size, const int* q_start,
                                    const int* q_len, const int* kv_len, const int* tile_req,
                                    const int* tile_tok0, int n_tiles, int nq, int nkv, int d,
                                    float scale, int window, int dtype, cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (d <= 0 || d % 16 != 0 || d > 256)
    MI_REFUSE("attention: head size %d is not a multiple of 16 in [16, 256]", d);
  return mi_attention_generic_kv(q, q_stride, out, out_stride, kcache, vcache, block_table, bt_stride, table_rows,
                                 page_size, q_start, q_len, kv_len, tile_req, tile_tok0, n_tiles, nq, nkv, d, d,
                                 scale, window, dtype, stream);
}
