// Layer norm over the fp32 residual stream, and the scaled token embedding that starts it.
//
//   mi_embedding_scaled   stream[t, :] = float(table[ids[t], :]) * scale          (fp32 out)
//   mi_add_layernorm      r = stream[src] + float(add1[src]) + float(add2[src])   (fp32)
//                         stream_out[i] = r                       (if given; may be the stream itself)
//                         out1[i] = T((r - mean) * rstd * w1 + b1)
//                         out2[i] = T((r - mean) * rstd * w2 + b2)   (if given: a second norm of the
//                                   same row, for layers whose two branches read the same stream)
//
// mean and variance are fp32, the variance is the mean of the squared deviations (two passes
// over the row, which is kept in shared memory).  One block per output row; src = rows[i] when a
// gather list is given, else i.  Gains and biases are fp32.
#include "common.cuh"

#include <initializer_list>

MI_DEFINE_ERROR_API()

template <typename T>
__global__ void embedding_scaled_kernel(const T* __restrict__ table, const int* __restrict__ ids,
                                        float* __restrict__ out, int H, int V, float scale) {
  mi_pdl_enter();
  const int t = blockIdx.x;
  const int id = ids[t];
  float* dst = out + (size_t)t * H;
  if ((unsigned)id >= (unsigned)V) {   // the step function validates ids; this keeps a fault visible
    for (int i = threadIdx.x; i < H; i += blockDim.x) dst[i] = __int_as_float(0x7fc00000);
    return;
  }
  const T* src = table + (size_t)id * H;
  if (H % 4 == 0) {                    // rows of whole aligned pieces (the host's tensors start aligned)
    for (int i = 4 * threadIdx.x; i < H; i += 4 * blockDim.x) {
      Vec4<T> a;
      float f[4];
      a.load(src + i);
      a.get(f);
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] *= scale;
      Vec4<float> o;
      o.set(f);
      o.store(dst + i);
    }
    return;
  }
  for (int i = threadIdx.x; i < H; i += blockDim.x) dst[i] = mi_to_float(src[i]) * scale;
}

extern "C" int mi_embedding_scaled(const void* table, const int* ids, float* out, int M, int H, int V,
                                   float scale, int dtype, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (H <= 0 || V <= 0) MI_REFUSE("embedding: bad sizes H=%d V=%d", H, V);
  if (!mi_aligned(table, 16) || !mi_aligned(out, 16)) MI_REFUSE("embedding: the table and the stream must be 16-byte aligned");
  const int threads = H >= 1024 ? 256 : 128;
  if (dtype == MI_DTYPE_F32)
    MI_LAUNCH((embedding_scaled_kernel<float>), M, threads, 0, stream, (const float*)table, ids, out, H, V, scale);
  else if (dtype == MI_DTYPE_BF16)
    MI_LAUNCH((embedding_scaled_kernel<bf16>), M, threads, 0, stream, (const bf16*)table, ids, out, H, V, scale);
  else
    MI_REFUSE("embedding: unknown dtype %d", dtype);
  MI_RETURN_LAUNCH_STATUS();
}

template <typename T>
__global__ void add_layernorm_kernel(const float* __restrict__ stream, const T* __restrict__ add1,
                                     const T* __restrict__ add2, float* __restrict__ stream_out,
                                     const int* __restrict__ rows, const float* __restrict__ w1,
                                     const float* __restrict__ b1, T* __restrict__ out1,
                                     const float* __restrict__ w2, const float* __restrict__ b2,
                                     T* __restrict__ out2, int H, float eps) {
  mi_pdl_enter();
  extern __shared__ float smem[];
  float* red = smem;        // 32 floats
  float* row = smem + 32;   // H floats
  const int i = blockIdx.x;
  const int src = rows ? rows[i] : i;
  const float* sr = stream + (size_t)src * H;
  const T* a1 = add1 ? add1 + (size_t)src * H : nullptr;
  const T* a2 = add2 ? add2 + (size_t)src * H : nullptr;
  float sum = 0.f;
  for (int k = threadIdx.x; k < H; k += blockDim.x) {
    float r = sr[k];
    if (a1) r += mi_to_float(a1[k]);
    if (a2) r += mi_to_float(a2[k]);
    row[k] = r;
    sum += r;
  }
  const float mean = mi_block_sum(sum, red) / (float)H;
  float sq = 0.f;
  for (int k = threadIdx.x; k < H; k += blockDim.x) {
    const float dlt = row[k] - mean;
    sq += dlt * dlt;
  }
  const float rstd = 1.f / sqrtf(mi_block_sum(sq, red) / (float)H + eps);
  float* so = stream_out ? stream_out + (size_t)i * H : nullptr;
  T* o1 = out1 + (size_t)i * H;
  T* o2 = out2 ? out2 + (size_t)i * H : nullptr;
  for (int k = threadIdx.x; k < H; k += blockDim.x) {
    const float r = row[k];
    const float n = (r - mean) * rstd;
    if (so) so[k] = r;
    o1[k] = mi_from_float<T>(n * w1[k] + b1[k]);
    if (o2) o2[k] = mi_from_float<T>(n * w2[k] + b2[k]);
  }
}

// The same bits for rows of whole aligned pieces of four that fit NV pieces a thread: the row stays on chip.  AHEAD: no
// kernel that may still run writes the gains and biases (a model's own), and they are asked for before the wait; without it 8 rows
// of 4096 with two norms 3.0 us become 3.4.  Every piece is read and written once, in one round trip.  The sums run in
// the order of the kernel above, a thread's elements blockDim apart: the row goes through shared memory for them.  8 rows of 4096 with two
// norms 6.0 us in the kernel above, 3.0 here (2.9 with the four of a piece added up first, which gives other bits); 2048 rows of
// 2048 17.6, 13.2 and 12.1 (10 of bytes).
template <typename T, int NV, bool AHEAD>
__global__ void __launch_bounds__(512, NV == 4 ? 1 : NV == 2 ? 2 : 3)
add_layernorm4_kernel(const float* stream, const T* add1, const T* add2, float* stream_out, const int* rows, const float* w1,
                      const float* b1, T* out1, const float* w2, const float* b2, T* out2, int H, float eps) {
  mi_pdl_launch_dependents();
  __shared__ float red[32];
  __shared__ __align__(16) float row[NV * 4 * 512];
  float g1[NV][4], c1[NV][4], g2[NV][4], c2[NV][4], r[4], f[4];
  Vec4<float> v;
  Vec4<T> a;
  auto gains = [&](int n) {
    const int k = 4 * (threadIdx.x + n * blockDim.x);
    if (k < H) {
      v.load(w1 + k); v.get(g1[n]);
      v.load(b1 + k); v.get(c1[n]);
      if (out2) {
        v.load(w2 + k); v.get(g2[n]);
        v.load(b2 + k); v.get(c2[n]);
      }
    }
  };
  if (AHEAD) {
#pragma unroll
    for (int n = 0; n < NV; ++n) gains(n);
  }
  mi_pdl_wait();
  const size_t i = blockIdx.x, src = rows ? rows[i] : i;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int k = 4 * (threadIdx.x + n * blockDim.x);
    if (k < H) {
      v.load(stream + src * H + k);
      v.get(r);
      if (add1) {
        a.load(add1 + src * H + k);
        a.get(f);
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] += f[e];
      }
      if (add2) {
        a.load(add2 + src * H + k);
        a.get(f);
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] += f[e];
      }
      v.set(r);
      v.store(row + k);
    }
  }
  __syncthreads();
  float own[NV * 4], sum = 0.f;
#pragma unroll
  for (int j = 0; j < NV * 4; ++j) {
    const int k = threadIdx.x + j * blockDim.x;
    own[j] = k < H ? row[k] : 0.f;
    sum += own[j];
  }
  const float mean = mi_block_sum(sum, red) / (float)H;
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < NV * 4; ++j)
    if (threadIdx.x + j * blockDim.x < H) {
      const float dlt = own[j] - mean;
      sq += dlt * dlt;
    }
  const float rstd = 1.f / sqrtf(mi_block_sum(sq, red) / (float)H + eps);
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int k = 4 * (threadIdx.x + n * blockDim.x);
    if (k >= H) continue;
    if (!AHEAD) gains(n);
    v.load(row + k);
    v.get(r);
    if (stream_out) v.store(stream_out + i * H + k);
    float y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f[e] = (r[e] - mean) * rstd;
      y[e] = f[e] * g1[n][e] + c1[n][e];
    }
    a.set(y);
    a.store(out1 + i * H + k);
    if (out2) {
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = f[e] * g2[n][e] + c2[n][e];
      a.set(y);
      a.store(out2 + i * H + k);
    }
  }
}

// w_constant: no kernel that may still run writes the gains and biases
extern "C" int mi_add_layernorm(const float* stream, const void* add1, const void* add2, float* stream_out,
                                const int* rows, const float* w1, const float* b1, void* out1,
                                const float* w2, const float* b2, void* out2, int M, int H, float eps, int w_constant,
                                int dtype, cudaStream_t stream_) {
  if (M <= 0) return 0;
  if (H <= 0) MI_REFUSE("layernorm: bad width %d", H);
  if (rows && stream_out == stream) MI_REFUSE("layernorm: a gathered norm cannot update the stream in place");
  const size_t smem = (32 + (size_t)H) * sizeof(float);
  if (smem > 200 * 1024) MI_REFUSE("layernorm: a row of %d floats does not fit in shared memory", H);
  const int threads = H >= 2048 ? 512 : (H >= 512 ? 256 : 128);
  bool pieces = H % 4 == 0 && H <= 16 * threads;
  for (const void* ptr : {(const void*)stream, add1, add2, (const void*)stream_out, (const void*)w1, (const void*)b1,
                          (const void*)out1, (const void*)w2, (const void*)b2, (const void*)out2})
    pieces = pieces && mi_aligned(ptr, 16);
  if (pieces) {
    const bool ahead = w_constant != 0;
#define MI_GO4(T, NV)                                                                                               \
  MI_LAUNCH((ahead ? add_layernorm4_kernel<T, NV, true> : add_layernorm4_kernel<T, NV, false>), M, threads, 0, stream_, \
            stream, (const T*)add1, (const T*)add2, stream_out, rows, w1, b1, (T*)out1, w2, b2, (T*)out2, H, eps)
#define MI_GO4_T(T)                          \
  if (H <= 4 * threads) MI_GO4(T, 1);        \
  else if (H <= 8 * threads) MI_GO4(T, 2);   \
  else MI_GO4(T, 4)
    if (dtype == MI_DTYPE_F32) {
      MI_GO4_T(float);
    } else if (dtype == MI_DTYPE_BF16) {
      MI_GO4_T(bf16);
    } else {
      MI_REFUSE("layernorm: unknown dtype %d", dtype);
    }
#undef MI_GO4_T
#undef MI_GO4
    MI_RETURN_LAUNCH_STATUS();
  }
#define MI_GO(T)                                                                                       \
  do {                                                                                                 \
    auto kern = add_layernorm_kernel<T>;                                                               \
    if (smem > 48 * 1024) {                                                                            \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e != cudaSuccess) return (int)e;                                                             \
    }                                                                                                  \
    MI_LAUNCH(kern, M, threads, smem, stream_, stream, (const T*)add1, (const T*)add2, stream_out, rows, w1, b1, \
              (T*)out1, w2, b2, (T*)out2, H, eps);                                                     \
  } while (0)
  if (dtype == MI_DTYPE_F32) MI_GO(float);
  else if (dtype == MI_DTYPE_BF16) MI_GO(bf16);
  else MI_REFUSE("layernorm: unknown dtype %d", dtype);
#undef MI_GO
  MI_RETURN_LAUNCH_STATUS();
}
