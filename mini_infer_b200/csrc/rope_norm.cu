// What stands around an attention whose queries and keys are rotated in the interleaved layout
// and then brought to unit root mean square, and whose heads are gated before the output
// projection.
//
//   mi_rope_norm_store   for every token and head: q and k are rotated on their first `rot` dimensions
//                        (dimension 2i pairs with 2i+1; the pair (u, v) at position p becomes
//                        (u cos a - v sin a, v cos a + u sin a), a = p * inv_freq[i]), then, with
//                        unit_norm, divided by sqrt(mean(x^2) + eps) over the head; q is written back
//                        in place, k and v go to their cache pages (k of size d, v of size dv).
//                        Angles, sines, cosines and the norm are fp32; each value is rounded once.
//   mi_gate_mul          out[t, c] = T(x[t, c] * act(g[t, c / per]) * scale), act = sigmoid or SiLU; per = 1: a
//                        gate per element, per = a head's size: one gate per head.
//
// q, k, v and the gate are column ranges of one packed projection [tokens, stride].
#include "heads_per_warp.cuh"

MI_DEFINE_ERROR_API()

// two neighbouring elements as one access
template <typename T>
struct PairBits { using type = uint32_t; };
template <>
struct PairBits<float> { using type = uint2; };
template <typename T>
__device__ __forceinline__ void load_pair(const T* p, float& u, float& v);
template <>
__device__ __forceinline__ void load_pair<float>(const float* p, float& u, float& v) {
  const float2 f = *reinterpret_cast<const float2*>(p);
  u = f.x;
  v = f.y;
}
template <>
__device__ __forceinline__ void load_pair<bf16>(const bf16* p, float& u, float& v) {
  const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
  u = f.x;
  v = f.y;
}
__device__ __forceinline__ void store_pair(float* p, float u, float v) { *reinterpret_cast<float2*>(p) = make_float2(u, v); }
__device__ __forceinline__ void store_pair(bf16* p, float u, float v) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(u, v);
}

// A warp takes heads of one token, lane l the pairs l, l + 32, ...: their angles are worked out once for all its heads.  VEC:
// every pair is one aligned access.  Bound by the round trips of a head, so the grid spreads a token's heads over as many blocks
// as fill the chip: 8 tokens of 32 + 8 + 8 heads of 128 17.5 us with a token per block, 5.3 so; 2048 tokens of 16 + 4 + 4
// heads 24 and 17 us.
template <typename T, bool VEC>
__global__ void __launch_bounds__(128)
rope_norm_store_kernel(T* __restrict__ qkv, int stride, int q_off, int k_off, int v_off,
                       const int* __restrict__ positions, const float* __restrict__ inv_freq,
                       const int* __restrict__ slots, T* __restrict__ kcache, T* __restrict__ vcache,
                       int nq, int nkv, int d, int dv, int rot, int unit_norm, float eps, int page_size,
                       int writes) {
  mi_pdl_enter();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const float pos = positions ? (float)positions[t] : 0.f;
  T* row = qkv + (size_t)t * stride;
  constexpr int EPC = 16 / (int)sizeof(T);
  const int slot = writes ? slots[t] : 0;
  const int page = slot / page_size, offset = slot - page * page_size;
  const int mk = mi_swizzle_mask_rows(d, (int)sizeof(T)), mv = mi_swizzle_mask_rows(dv, (int)sizeof(T));
  const int npairs = (d + 1) >> 1;
  // a lane keeps at most 4 pairs (d <= 256)
  float sn[4], cs[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = lane + 32 * j;
    sn[j] = 0.f;
    cs[j] = 1.f;
    if (p < npairs && 2 * p + 1 < rot) sincosf(pos * inv_freq[p], &sn[j], &cs[j]);
  }
  // heads 0..nq-1: queries; nq..nq+nkv-1: keys; then the values
  for (int h = blockIdx.y * nwarps + warp; h < nq + 2 * nkv; h += gridDim.y * nwarps) {
    if (h >= nq + nkv) {
      if (!writes) continue;
      const int kvh = h - nq - nkv;
      const T* src = row + v_off + kvh * dv;
      T* dst = vcache + ((size_t)(page * nkv + kvh) * page_size + offset) * dv;
      if (VEC) {
        using Bits = typename PairBits<T>::type;
        for (int k = 2 * lane; k < dv; k += 64)
          *reinterpret_cast<Bits*>(dst + mi_swizzled(k, offset, mv, EPC)) = *reinterpret_cast<const Bits*>(src + k);
      } else {
        for (int k = lane; k < dv; k += 32) dst[mi_swizzled(k, offset, mv, EPC)] = src[k];
      }
      continue;
    }
    const bool is_q = h < nq;
    T* x = is_q ? row + q_off + h * d : row + k_off + (h - nq) * d;
    if (!is_q && !writes && !unit_norm && rot == 0) continue;
    float ss = 0.f;
    float a0[4], a1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = lane + 32 * j;
      a0[j] = a1[j] = 0.f;
      if (p < npairs) {
        if (VEC) {
          load_pair<T>(x + 2 * p, a0[j], a1[j]);
        } else {
          a0[j] = mi_to_float(x[2 * p]);
          a1[j] = (2 * p + 1 < d) ? mi_to_float(x[2 * p + 1]) : 0.f;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = lane + 32 * j;
      if (p < npairs) {
        if (2 * p + 1 < rot) {
          float ru, rv;
          mi_rotate(a0[j], a1[j], sn[j], cs[j], ru, rv);
          a0[j] = ru;
          a1[j] = rv;
        }
        ss += a0[j] * a0[j] + a1[j] * a1[j];
      }
    }
    float mult = 1.f;
    if (unit_norm) {
      ss = mi_warp_sum(ss);
      mult = 1.f / sqrtf(ss / (float)d + eps);
    }
    T* kdst = nullptr;
    if (!is_q && writes) kdst = kcache + ((size_t)(page * nkv + (h - nq)) * page_size + offset) * d;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = lane + 32 * j;
      if (p < npairs) {
        if (VEC) {
          store_pair(x + 2 * p, a0[j] * mult, a1[j] * mult);
          if (kdst) store_pair(kdst + mi_swizzled(2 * p, offset, mk, EPC), a0[j] * mult, a1[j] * mult);
          continue;
        }
        const T u = mi_from_float<T>(a0[j] * mult), v = mi_from_float<T>(a1[j] * mult);
        x[2 * p] = u;
        if (2 * p + 1 < d) x[2 * p + 1] = v;
        if (kdst) {
          kdst[mi_swizzled(2 * p, offset, mk, EPC)] = u;
          if (2 * p + 1 < d) kdst[mi_swizzled(2 * p + 1, offset, mk, EPC)] = v;
        }
      }
    }
  }
}

extern "C" int mi_rope_norm_store(void* qkv, int stride, int q_off, int k_off, int v_off, const int* positions,
                                  const float* inv_freq, const int* slots, void* kcache, void* vcache, int M,
                                  int nq, int nkv, int d, int dv, int rot, int unit_norm, float eps,
                                  int page_size, int writes, int dtype, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (d <= 0 || d > 256 || dv <= 0 || dv > 256) MI_REFUSE("rope_norm: head sizes %d and %d must lie in [1, 256]", d, dv);
  if (rot < 0 || rot > d || (rot & 1)) MI_REFUSE("rope_norm: %d rotated dimensions of %d", rot, d);
  if (writes && (!slots || !kcache || !vcache || page_size <= 0)) MI_REFUSE("rope_norm: a cache write needs slots and pages");
  if (rot > 0 && (!positions || !inv_freq)) MI_REFUSE("rope_norm: a rotation needs positions and frequencies");
  const int size = dtype == MI_DTYPE_F32 ? 4 : 2, heads = nq + 2 * nkv;
  const bool vec = d % 2 == 0 && dv % 2 == 0 && stride % 2 == 0 && q_off % 2 == 0 && k_off % 2 == 0 && v_off % 2 == 0 &&
                   mi_aligned(qkv, 2 * size) && (!writes || (mi_aligned(kcache, 16) && mi_aligned(vcache, 16)));
  const int per_warp = heads_per_warp((long long)M * heads);
  const dim3 grid((unsigned)M, (unsigned)((heads + 4 * per_warp - 1) / (4 * per_warp)));
#define MI_GO(T, VEC)                                                                                                   \
  MI_LAUNCH((rope_norm_store_kernel<T, VEC>), grid, 128, 0, stream, (T*)qkv, stride, q_off, k_off, v_off, positions, inv_freq, \
            slots, (T*)kcache, (T*)vcache, nq, nkv, d, dv, rot, unit_norm, eps, page_size, writes)
  if (dtype == MI_DTYPE_F32) {
    if (vec) MI_GO(float, true);
    else MI_GO(float, false);
  } else if (dtype == MI_DTYPE_BF16) {
    if (vec) MI_GO(bf16, true);
    else MI_GO(bf16, false);
  } else {
    MI_REFUSE("rope_norm: unknown dtype %d", dtype);
  }
#undef MI_GO
  MI_RETURN_LAUNCH_STATUS();
}

// act: 1 sigmoid, 2 SiLU
template <typename T>
__global__ void gate_mul_kernel(const T* __restrict__ x, int x_stride, const T* __restrict__ g, int g_stride,
                                T* __restrict__ out, int out_stride, int M, int C, int act, float scale, int per) {
  mi_pdl_enter();
  const size_t n = (size_t)M * C;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(idx / C), c = (int)(idx - (size_t)t * C);
    float a = 1.f;                       // act 0: no gate, the factor alone
    if (act) {
      const float gv = mi_to_float(g[(size_t)t * g_stride + c / per]);
      const float sg = 1.f / (1.f + expf(-gv));
      a = act == 2 ? gv * sg : sg;
    }
    out[(size_t)t * out_stride + c] = mi_from_float<T>(mi_to_float(x[(size_t)t * x_stride + c]) * a * scale);
  }
}

// bfloat16, eight columns per thread: 16-byte accesses, one division by the row length for eight values.  2048 x 4096: 41 us
// element by element, 13 here (8 us of bytes).
__global__ void __launch_bounds__(256)
gate_mul8_kernel(const bf16* __restrict__ x, int x_stride, const bf16* __restrict__ g, int g_stride, bf16* __restrict__ out,
                 int out_stride, int M, int pieces, int act, float scale, int per) {
  mi_pdl_enter();
  const size_t n = (size_t)M * pieces;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(idx / pieces), c = (int)(idx - (size_t)t * pieces) * 8;
    const uint4 xv = *reinterpret_cast<const uint4*>(x + (size_t)t * x_stride + c);
    uint4 gv = make_uint4(0u, 0u, 0u, 0u);
    float one = 0.f;
    if (act && per == 1) gv = *reinterpret_cast<const uint4*>(g + (size_t)t * g_stride + c);
    else if (act) one = mi_to_float(g[(size_t)t * g_stride + c / per]);
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w}, gw[4] = {gv.x, gv.y, gv.z, gv.w};
    uint32_t r[4];
    auto gated = [&](float v, float z) {
      float a = 1.f;
      if (act) {
        const float sg = 1.f / (1.f + expf(-z));
        a = act == 2 ? z * sg : sg;
      }
      return v * a * scale;
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xw[j]));
      float2 z = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[j]));
      if (per != 1) z = make_float2(one, one);
      const __nv_bfloat162 o = __floats2bfloat162_rn(gated(f.x, z.x), gated(f.y, z.y));
      r[j] = *reinterpret_cast<const uint32_t*>(&o);
    }
    *reinterpret_cast<uint4*>(out + (size_t)t * out_stride + c) = make_uint4(r[0], r[1], r[2], r[3]);
  }
}

extern "C" int mi_gate_mul(const void* x, int x_stride, const void* g, int g_stride, void* out, int out_stride,
                           int M, int C, int act, float scale, int per, int dtype, cudaStream_t stream) {
  if (M <= 0 || C <= 0) return 0;
  if (per <= 0) MI_REFUSE("gate_mul: %d columns per gate", per);
  if (act < 0 || act > 2 || (act && !g)) MI_REFUSE("gate_mul: unknown activation %d, or no gate for it", act);
  const size_t n = (size_t)M * C;
  // rows of whole 16-byte pieces on all sides, a gate of their own for all eight columns or one for all of them
  if (dtype == MI_DTYPE_BF16 && C % 8 == 0 && x_stride % 8 == 0 && out_stride % 8 == 0 && mi_aligned(x, 16) && mi_aligned(out, 16) &&
      (!act || (per == 1 ? g_stride % 8 == 0 && mi_aligned(g, 16) : per % 8 == 0))) {
    const size_t n8 = n / 8;
    MI_LAUNCH((gate_mul8_kernel), (int)((n8 + 255) / 256 < 8192 ? (n8 + 255) / 256 : 8192), 256, 0, stream, (const bf16*)x, x_stride,
              (const bf16*)g, g_stride, (bf16*)out, out_stride, M, C / 8, act, scale, per);
    MI_RETURN_LAUNCH_STATUS();
  }
  const int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  if (dtype == MI_DTYPE_F32)
    MI_LAUNCH((gate_mul_kernel<float>), blocks, 256, 0, stream, (const float*)x, x_stride, (const float*)g, g_stride,
              (float*)out, out_stride, M, C, act, scale, per);
  else if (dtype == MI_DTYPE_BF16)
    MI_LAUNCH((gate_mul_kernel<bf16>), blocks, 256, 0, stream, (const bf16*)x, x_stride, (const bf16*)g, g_stride,
              (bf16*)out, out_stride, M, C, act, scale, per);
  else
    MI_REFUSE("gate_mul: unknown dtype %d", dtype);
  MI_RETURN_LAUNCH_STATUS();
}
