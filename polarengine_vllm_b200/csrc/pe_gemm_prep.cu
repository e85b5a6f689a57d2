// The passes around the tensor-core matmuls: activation preparation (gather, padding, FWHT-128, bf16, K order of the
// codes) and the sum of the partial results of a split K.
#include "pe_gemm.cuh"

namespace pe {

constexpr int kPrepThreads = 128;
constexpr int kPrepItems = kPrepThreads / 4;  // 128-blocks per CTA

// eight consecutive elements from `col` on, zero beyond `limit`
template <int XD>
struct Raw8 { uint4 w[XD == PE_F32 ? 2 : 1]; };
template <int XD>
__device__ __forceinline__ Raw8<XD> load8(const void* x, int64_t row_off, int col, int limit, bool vec) {
  Raw8<XD> r;
  constexpr int W = XD == PE_F32 ? 2 : 1;
  if (vec && col + 8 <= limit) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(x) + (row_off + col) * (XD == PE_F32 ? 4 : 2));
#pragma unroll
    for (int i = 0; i < W; ++i) r.w[i] = __ldg(src + i);
  } else {
    uint32_t u[4 * W] = {};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (col + i >= limit) continue;
      if (XD == PE_F32) u[i % (4 * W)] = static_cast<const uint32_t*>(x)[row_off + col + i];
      else u[i >> 1] |= (uint32_t)static_cast<const uint16_t*>(x)[row_off + col + i] << (16 * (i & 1));
    }
#pragma unroll
    for (int i = 0; i < W; ++i) r.w[i] = make_uint4(u[4 * i], u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]);
  }
  return r;
}
template <int XD>
__device__ __forceinline__ void unpack8(const Raw8<XD>& r, float f[8]) {
  if constexpr (XD == PE_F32) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      f[4 * i] = __uint_as_float(r.w[i].x); f[4 * i + 1] = __uint_as_float(r.w[i].y);
      f[4 * i + 2] = __uint_as_float(r.w[i].z); f[4 * i + 3] = __uint_as_float(r.w[i].w);
    }
  } else {
    const uint32_t u[4] = {r.w[0].x, r.w[0].y, r.w[0].z, r.w[0].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = XD == PE_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&u[i]))
                                    : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[i]));
      f[2 * i] = v.x; f[2 * i + 1] = v.y;
    }
  }
}

// Four lanes per 128-block.  Lane q holds k = 16 q .. 16 q + 15 and the same range + 64, as pairs (k, k + 64): five of
// the seven butterfly stages then stay in a lane's registers, two cross lanes, and for nibble codes the pairs leave in
// the order in which a code byte decodes.  (With one warp per block every stage but two was a shuffle, and the shuffles
// were what bounded the pass: 16384 rows of 1856 took 50 us, 28 us now.)
// Grouped launches: row m of the prepared matrix is row x_rows[m] of x, and only the first valid_rows[0] +
// valid_rows[1] rows exist (the rest of the list is undefined and is written as zeros).
// Or, with to_rows, row m of x goes to the rows to_rows[m * fanout ..] of the prepared matrix (negative: nowhere): a token
// of a mixture layer is rotated once for all of its experts (2048 tokens of 2688 to eight experts each: 37 us when every
// copy was rotated, 29 us now).
// With SILU rows are [gate | up] of `limit` columns each and the input is half(silu(gate)) * up, rounded as pe_silu_mul
// rounds (a launch and a trip through memory less per layer: 512 rows of 12288 took 8.5 us more).
template <int XD, bool SILU>
__global__ void __launch_bounds__(kPrepThreads) gemm_prep_kernel(const void* x, int raw, int64_t ld_x, int limit, __nv_bfloat16* xq, int M, int nb,
                                                                 int pair_layout, const int* x_rows, const int* valid_rows, const int* to_rows, int fanout, int* status) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // first: the matmul behind may then read what older kernels wrote at once
  asm volatile("griddepcontrol.launch_dependents;");
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;  // the matmul's status word (it follows in stream order)
  const int q = threadIdx.x & 3;
  const int64_t item = (int64_t)blockIdx.x * kPrepItems + (threadIdx.x >> 2);
  const bool on = item < (int64_t)M * nb;
  const int m = on ? (int)(item / nb) : 0, blk = on ? (int)(item - (int64_t)m * nb) : 0;
  const bool live = on && (!valid_rows || m < valid_rows[0] + valid_rows[1]);
  const int64_t row = live && x_rows ? x_rows[m] : m;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (ld_x & (XD == PE_F32 ? 3 : 7)) == 0 && (!SILU || (limit & 7) == 0);
  const int lim = live ? limit : 0, col = blk * kBlock + 16 * q;
  Raw8<XD> r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] = load8<XD>(x, row * ld_x, col + (i & 1) * 8 + (i >> 1) * 64, lim, vec);
  if constexpr (SILU) {
    Raw8<XD> up[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) up[i] = load8<XD>(x, row * ld_x + limit, col + (i & 1) * 8 + (i >> 1) * 64, lim, vec);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 *g = reinterpret_cast<__half2*>(&r[i].w[0]), *u = reinterpret_cast<__half2*>(&up[i].w[0]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(g[j]);
        g[j] = __hmul2(__floats2half2_rn(f.x / (1.f + expf(-f.x)), f.y / (1.f + expf(-f.y))), u[j]);
      }
    }
  }
  float2 p[16];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float lo[8], hi[8];
    unpack8<XD>(r[i], lo);
    unpack8<XD>(r[i + 2], hi);
#pragma unroll
    for (int j = 0; j < 8; ++j) p[8 * i + j] = make_float2(lo[j], hi[j]);
  }
  if (raw) {
    const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
    for (int s = 1; s < 16; s <<= 1)
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (!(j & s)) {
          const float2 a = p[j], b = p[j | s];
          p[j] = add2(a, b);
          p[j | s] = fma2(b, minus, a);
        }
#pragma unroll
    for (int s = 1; s <= 2; s <<= 1) {
      const float sg = (q & s) ? -1.f : 1.f;
      const float2 sign = make_float2(sg, sg);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, p[j].x, s), __shfl_xor_sync(0xffffffffu, p[j].y, s));
        p[j] = fma2(p[j], sign, o);
      }
    }
    const float sc = 0.08838834764831845f;  // 1 / sqrt(128)
    const float2 scale = make_float2(sc, sc);
#pragma unroll
    for (int j = 0; j < 16; ++j) p[j] = mul2(make_float2(p[j].x + p[j].y, p[j].x - p[j].y), scale);
  }
  if (!on) return;
  uint4 out[4];
  if (pair_layout) {  // positions 2 k, 2 k + 1 = elements k, k + 64
#pragma unroll
    for (int j = 0; j < 4; ++j)
      out[j] = make_uint4(pack_bf16(p[4 * j].x, p[4 * j].y), pack_bf16(p[4 * j + 1].x, p[4 * j + 1].y),
                          pack_bf16(p[4 * j + 2].x, p[4 * j + 2].y), pack_bf16(p[4 * j + 3].x, p[4 * j + 3].y));
  } else {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      out[j] = make_uint4(pack_bf16(p[8 * j].x, p[8 * j + 1].x), pack_bf16(p[8 * j + 2].x, p[8 * j + 3].x),
                          pack_bf16(p[8 * j + 4].x, p[8 * j + 5].x), pack_bf16(p[8 * j + 6].x, p[8 * j + 7].x));
      out[2 + j] = make_uint4(pack_bf16(p[8 * j].y, p[8 * j + 1].y), pack_bf16(p[8 * j + 2].y, p[8 * j + 3].y),
                              pack_bf16(p[8 * j + 4].y, p[8 * j + 5].y), pack_bf16(p[8 * j + 6].y, p[8 * j + 7].y));
    }
  }
  const int at0 = pair_layout ? 4 * q : 2 * q, at2 = pair_layout ? 4 * q + 2 : 8 + 2 * q;
  auto put = [&](int row_out) {
    uint4* dst = reinterpret_cast<uint4*>(xq + ((int64_t)row_out * nb + blk) * kBlock);
    dst[at0] = out[0]; dst[at0 + 1] = out[1];
    dst[at2] = out[2]; dst[at2 + 1] = out[3];
  };
  if (!to_rows) {
    put(m);
    return;
  }
  for (int j0 = 0; j0 < fanout; j0 += 8) {
    int to[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) to[j] = j0 + j < fanout ? __ldg(to_rows + (int64_t)m * fanout + j0 + j) : -1;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (to[j] >= 0) put(to[j]);
  }
}

int launch_gemm_prep(const void* x, int x_kind, int x_dtype, int64_t ld_x, int in_f, void* xq, int rows, int in_f_padded, int pair_layout,
                     const int* x_rows, const int* valid_rows, const int* to_rows, int fanout, int* status, cudaStream_t st) {
  const int nb = in_f_padded / kBlock;
  const int64_t blocks = ((int64_t)rows * nb + kPrepItems - 1) / kPrepItems;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  auto kfn = x_kind == PE_X_SILU_MUL ? gemm_prep_kernel<PE_F16, true>
             : x_dtype == PE_F32     ? gemm_prep_kernel<PE_F32, false>
             : x_dtype == PE_F16     ? gemm_prep_kernel<PE_F16, false>
                                     : gemm_prep_kernel<PE_BF16, false>;
  PE_CUDA_TRY(launch_pdl(kfn, dim3((unsigned)blocks), dim3(kPrepThreads), 0, st, x, x_kind != PE_X_ROTATED ? 1 : 0, ld_x,
                         x_kind != PE_X_ROTATED ? in_f : in_f_padded, static_cast<__nv_bfloat16*>(xq), rows, nb, pair_layout, x_rows, valid_rows, to_rows,
                         fanout, status));
  return PE_OK;
}

// Sum of the partial results of the K ranges, in their order (bit-reproducible), plus bias, to the output type.  Bounded
// by L2: four columns per thread and four ranges requested at once (one column and one range at a time left it waiting
// for each load: 512 x 4096 out of three ranges took 15 us, 5 us now).
template <bool VEC>
__global__ void __launch_bounds__(256) gemm_splitk_reduce_kernel(const float* part, int ksplit, int M, int N, const __half* bias, void* y, int y_dtype,
                                                                 int64_t ld_y) {
  pdl_enter();
  constexpr int W = VEC ? 4 : 1, U = 4;
  const int per_row = N / W;
  const int64_t total = (int64_t)M * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)M * per_row; i += (int64_t)gridDim.x * blockDim.x) {
    const int m = (int)(i / per_row), n = (int)(i - (int64_t)m * per_row) * W;
    const float* src = part + (int64_t)m * N + n;
    float s[W] = {};
    for (int k0 = 0; k0 < ksplit; k0 += U) {
      float v[U][W];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool on = k0 + u < ksplit;
        if constexpr (VEC) {
          const float4 f = on ? *reinterpret_cast<const float4*>(src + (k0 + u) * total) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[u][0] = f.x; v[u][1] = f.y; v[u][2] = f.z; v[u][3] = f.w;
        } else {
          v[u][0] = on ? src[(k0 + u) * total] : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int w = 0; w < W; ++w) s[w] += v[u][w];
    }
    if (bias) {
#pragma unroll
      for (int w = 0; w < W; ++w) s[w] += __half2float(bias[n + w]);
    }
    const int64_t o = (int64_t)m * ld_y + n;
    if constexpr (VEC) {
      if (y_dtype != PE_F32) {
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(y) + o) = y_dtype == PE_F16 ? make_uint2(pack_half2(s[0], s[1]), pack_half2(s[2], s[3]))
                                                                                    : make_uint2(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]));
        continue;
      }
    }
#pragma unroll
    for (int w = 0; w < W; ++w) store_from_float(y, y_dtype, o + w, s[w]);
  }
}

int launch_splitk_reduce(const float* part, int ksplit, int m, int n, const void* bias, void* y, int y_dtype, int64_t ld_y, int sms, cudaStream_t st) {
  // four columns at a time need whole, aligned groups of them in every row
  const bool vec = n % 4 == 0 && ld_y % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 7) == 0 && (reinterpret_cast<uintptr_t>(part) & 15) == 0;
  const int64_t items = (int64_t)m * (vec ? n / 4 : n), want = (items + 255) / 256, cap = (int64_t)sms * 8;
  auto kfn = vec ? gemm_splitk_reduce_kernel<true> : gemm_splitk_reduce_kernel<false>;
  PE_CUDA_TRY(launch_pdl(kfn, dim3((unsigned)(want < cap ? want : cap)), dim3(256), 0, st, part, ksplit, m, n, static_cast<const __half*>(bias), y,
                         y_dtype, ld_y));
  return PE_OK;
}

// ---- tensor maps ---------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// fp32 matrices [depth][height][width] one after the other, boxes of 32 x 32 x 1 with 128-byte swizzle
int encode_map_f32(CUtensorMap* map, const void* base, uint64_t width, uint64_t height, uint64_t depth, uint64_t row_bytes) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return PE_ERR_CUDA;
  const cuuint64_t dims[3] = {width, height, depth}, strides[2] = {row_bytes, row_bytes * height};
  const cuuint32_t box[3] = {32, 32, 1}, estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? PE_OK : PE_ERR_CUDA;
}

int encode_map_2d(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t width, uint64_t height, uint64_t row_bytes, uint32_t box_w,
                  uint32_t box_h, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return PE_ERR_CUDA;
  const cuuint64_t dims[2] = {width, height}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {box_w, box_h}, estr[2] = {1, 1};
  return enc(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? PE_OK : PE_ERR_CUDA;
}

}  // namespace pe
