// One-token matmul over the row-major layout that needs no scratch memory (pe_gemv_pro): column-owner kernel.
//
//   y[r] = sum_blk norm[r, blk] * sum_k ct[code[r, blk, k]] * xt[blk, k]   (+ bias[r])
//
// CTA c owns the weight rows [c N / G, (c+1) N / G): one contiguous region of the row-major code array and of the norm
// array, so nothing ever crosses CTAs and no scratch memory is needed.  An item is 8 or 16 weight rows x 128 bytes
// (8 lanes x 16 B per row, two or four rows per lane) and warp w owns the 128-byte column chunks w, w+16, ... of the
// CTA's rows, so a lane meets the same few activation slices over and over and keeps them in registers (16 fp16 pairs
// per chunk, at most CPW chunks), and the rows of a lane give the scheduler independent dependency chains.  Codes
// travel by 16-byte asynchronous copies into a lane-private ring.  The price is a reduction per row
// group -- three shuffles over the 8 lanes of a row -- and a sum over the 16 warps' column
// partials through shared memory, in warp order (bit-reproducible), after every pass of
// 256 rows.  Each warp rotates only the blocks it owns.
// Centroid lookup: register table (byte permutes) for layers with at most eight levels, lane-replicated shared-memory
// table otherwise.
#include "pe_gemv_decode.cuh"

namespace pe {

constexpr int kRowWarps = 16;
constexpr int kRowThreads = kRowWarps * 32;
constexpr int kItemBytes = 512;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

constexpr int kPassRows = 256;
constexpr int kPartStride = kRowWarps + 1;  // floats per row in the partial array (bank spread)

struct ColArgs {
  const uint8_t* codes; int64_t ld_codes;  // bytes
  const uint8_t* norms; int64_t ld_norms;  // bytes between rows of fp16 norms
  const float* ct; int n_levels;
  const void* x; int x_kind; int x_dtype; int in_f;
  void* y; int y_dtype;
  const __half* bias;
  int N, K, n_chunks;
  // activation prologue (PE_PRO_*): what turns `x` into the matmul input
  int pro;
  const void* delta; int delta_dtype;  // PE_PRO_ADD_RMSNORM: optional addend of the residual x (fp16 / fp32)
  const __half* norm_w;                // PE_PRO_ADD_RMSNORM: norm weight
  __half* resid_out;                   // PE_PRO_ADD_RMSNORM: the updated residual (written by CTA 0), may be null
  float eps;
};

// ---- activation prologues: the glue op in front of a projection, computed while its input is staged ----
// PE_PRO_ADD_RMSNORM  input = half(r * rsqrt(mean(r^2) + eps)) * w   with r = half(x + half(delta)), the rounding
//                     steps of pe_add_rmsnorm;  PE_PRO_SILU_MUL  input = half(silu(gate)) * up, those of pe_silu_mul.
// 4 consecutive elements starting at `col` (a multiple of 4), zero beyond in_f.
__device__ __forceinline__ void resid4(const ColArgs& p, int col, float r[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const __half*>(p.x) + col);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  r[0] = a.x; r[1] = a.y; r[2] = b.x; r[3] = b.y;
  if (p.delta) {
    float d[4];
    if (p.delta_dtype == PE_F32) {
      const float4 f = *reinterpret_cast<const float4*>(static_cast<const float*>(p.delta) + col);
      d[0] = f.x; d[1] = f.y; d[2] = f.z; d[3] = f.w;
    } else {
      const uint2 du = *reinterpret_cast<const uint2*>(static_cast<const __half*>(p.delta) + col);
      const float2 da = __half22float2(*reinterpret_cast<const __half2*>(&du.x)), db = __half22float2(*reinterpret_cast<const __half2*>(&du.y));
      d[0] = da.x; d[1] = da.y; d[2] = db.x; d[3] = db.y;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = __half2float(__float2half_rn(r[i] + __half2float(__float2half_rn(d[i]))));
  }
}

__device__ __forceinline__ void pro_load4(const ColArgs& p, int col, bool on, float scale, float v[4]) {
  v[0] = v[1] = v[2] = v[3] = 0.f;
  if (!on || col >= p.in_f) return;  // in_f is a multiple of 4 on this path
  if (p.pro == PE_PRO_ADD_RMSNORM) {
    float r[4];
    resid4(p, col, r);
    const uint2 wu = *reinterpret_cast<const uint2*>(p.norm_w + col);
    const __half2 n0 = __hmul2(__floats2half2_rn(r[0] * scale, r[1] * scale), *reinterpret_cast<const __half2*>(&wu.x));
    const __half2 n1 = __hmul2(__floats2half2_rn(r[2] * scale, r[3] * scale), *reinterpret_cast<const __half2*>(&wu.y));
    const float2 a = __half22float2(n0), b = __half22float2(n1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {  // PE_PRO_SILU_MUL: x = [gate (in_f) | up (in_f)]
    const uint2 g = *reinterpret_cast<const uint2*>(static_cast<const __half*>(p.x) + col);
    const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const __half*>(p.x) + p.in_f + col);
    const float2 g0 = __half22float2(*reinterpret_cast<const __half2*>(&g.x)), g1 = __half22float2(*reinterpret_cast<const __half2*>(&g.y));
    const __half2 s0 = __floats2half2_rn(g0.x / (1.f + expf(-g0.x)), g0.y / (1.f + expf(-g0.y)));
    const __half2 s1 = __floats2half2_rn(g1.x / (1.f + expf(-g1.x)), g1.y / (1.f + expf(-g1.y)));
    const float2 a = __half22float2(__hmul2(s0, *reinterpret_cast<const __half2*>(&u.x)));
    const float2 b = __half22float2(__hmul2(s1, *reinterpret_cast<const __half2*>(&u.y)));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// ring slot of one item: SUB sub-items of 4 rows x 128 bytes, then 4 bytes of norms per row, rounded to whole 128-byte lines
__host__ __device__ constexpr int col_stage_bytes(int sub) { return (sub * kItemBytes + sub * 16 + 127) & ~127; }

template <bool PACKED, bool REGTAB, int CPW, int DEPTH, int SUB>
__global__ void __launch_bounds__(kRowThreads, 1) gemv_cols_kernel(const ColArgs p) {
  constexpr int kColStage = col_stage_bytes(SUB);
  constexpr int kGroupRows = 4 * SUB;  // weight rows of one item
  static_assert(DEPTH % CPW == 0, "the ring holds whole row groups");
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ float pro_red[kRowWarps];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int rs = lane >> 3, pc = lane & 7;  // row of the sub-item, 16-byte piece of the chunk
  const int G = gridDim.x, cta = blockIdx.x;
  constexpr int kXPerChunk = PACKED ? 16 : 8;  // fp16 pairs a lane keeps per chunk
  constexpr int kRgDepth = DEPTH / CPW;        // row groups in flight per warp
  constexpr int kNormStep = PACKED ? 64 : 32;  // norm bytes between this warp's chunks

  const int r_beg = (int)((long long)p.N * cta / G), r_end = (int)((long long)p.N * (cta + 1) / G);
  const int n_rg = (r_end - r_beg + kGroupRows - 1) / kGroupRows;
  int cnt = (p.n_chunks - w + kRowWarps - 1) / kRowWarps;  // chunks w, w+16, ... of this warp
  cnt = cnt < 0 ? 0 : (cnt > CPW ? CPW : cnt);

  // The wait before the first read: codes, norms and table may be the output of a kernel that is still running (a layer just
  // loaded, arrays rewritten in place), and the launch in front may have let this one start before it.
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float ct_mine = 0.f;
  {
    const int e = PACKED ? (lane & 15) : (w + 16 * (lane & 15));
    if (e < p.n_levels) asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(ct_mine) : "l"(p.ct + e));
  }

  // shared memory: [table 32 KB unless REGTAB][rotation scratch][partials][ring]
  uint8_t* lut_g = smem;
  uint8_t* xw = smem + (REGTAB ? 0 : kLutBytes) + (size_t)w * (CPW * 512);
  float* part = reinterpret_cast<float*>(smem + (REGTAB ? 0 : kLutBytes) + (size_t)kRowWarps * CPW * 512);
  uint8_t* ring_g = reinterpret_cast<uint8_t*>(part) + kPassRows * kPartStride * 4 + (size_t)w * (DEPTH * kColStage);
  const uint32_t st_base = smem_u32(ring_g), st_end = st_base + DEPTH * kColStage;

  // ---- code stream.  An item is 4 SUB weight rows x 128 bytes: lane (rs, pc) copies its 16
  // bytes of rows rs, rs + 4, ... of the group.  The ring slot of item (row group rg, chunk
  // slot j) is (rg % kRgDepth) * CPW + j, so the refill issued after item (rg, j) is item
  // (rg + kRgDepth, j): same slot, same j, and the source is a running pointer plus a
  // compile-time offset.  One copy group per slot, empty for slots the warp does not
  // have, so the group count the math waits on is a constant.  Rows past the end of the
  // matrix are not fetched (their sums are never stored).
  const uint8_t* cptr_f = p.codes + (int64_t)(r_beg + rs) * p.ld_codes + (size_t)w * 128 + pc * 16;
  const uint8_t* nptr_f = p.norms + (int64_t)(r_beg + (lane & (kGroupRows - 1))) * p.ld_norms + (PACKED ? (size_t)w * 4 : (size_t)(w & ~1) * 2);
  const int64_t csub = 4 * p.ld_codes, cstep = kGroupRows * p.ld_codes, nstep = kGroupRows * p.ld_norms;
  int rg_f = 0;
  // sub-item s of the group being fetched covers rows r_beg + kGroupRows rg_f + 4 s .. + 3: skipped
  // as a whole beyond the CTA's rows, per row beyond the matrix
  int row_f = r_beg + rs;  // this lane's row in sub-item 0
  const uint32_t q_off = lane * 16;
  auto fetch_item = [&](uint32_t st, int j) {
    if (j < cnt && rg_f < n_rg) {
#pragma unroll
      for (int sb = 0; sb < SUB; ++sb)
        if (row_f + 4 * sb - rs < r_end && row_f + 4 * sb < p.N) cp_async16(st + sb * kItemBytes + q_off, cptr_f + sb * csub + j * 2048);
      if (lane < kGroupRows && row_f - rs + lane < p.N) cp_async4(st + SUB * kItemBytes + lane * 4, nptr_f + j * kNormStep);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto advance_fetch = [&]() {
    ++rg_f;
    cptr_f += cstep;
    nptr_f += nstep;
    row_f += kGroupRows;
  };
#pragma unroll
  for (int d = 0; d < kRgDepth; ++d) {
#pragma unroll
    for (int j = 0; j < CPW; ++j) fetch_item(st_base + (d * CPW + j) * kColStage, j);
    advance_fetch();
  }


  // ---- centroid table
  RegTable tb = {0, 0, 0, 0};
  if (PACKED && REGTAB) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t hb = __half_as_ushort(__float2half_rn(__shfl_sync(0xffffffffu, ct_mine, i)));
      if (i < 4) { tb.lo0 |= (hb & 0xff) << (8 * i); tb.hi0 |= (hb >> 8) << (8 * i); }
      else { tb.lo1 |= (hb & 0xff) << (8 * (i - 4)); tb.hi1 |= (hb >> 8) << (8 * (i - 4)); }
    }
  } else if (PACKED) {
    const float lo = __shfl_sync(0xffffffffu, ct_mine, w);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float hi = __shfl_sync(0xffffffffu, ct_mine, i);
      *reinterpret_cast<uint32_t*>(lut_g + (w + 16 * i) * 128 + lane * 4) = pack_half2(lo, hi);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float c = __shfl_sync(0xffffffffu, ct_mine, i);
      if (w + 16 * i < p.n_levels) *reinterpret_cast<uint32_t*>(lut_g + (w + 16 * i) * 128 + lane * 4) = pack_half2(c, c);
    }
  }
  const uint32_t lane_base = smem_u32(lut_g) + lane * 4;

  // ---- this warp's activation slices: load, rotate, bounce through the warp's scratch
  // into the item layout, keep in registers
  uint32_t xr[CPW][kXPerChunk];
  {
    const bool raw = p.x_kind == PE_X_RAW;
    const bool vec_ok = (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
    const int limit = raw ? p.in_f : p.K;
    constexpr int BPC = PACKED ? 2 : 1;  // quantization blocks per chunk
    float v[CPW * BPC][4];
    if (p.pro == PE_PRO_NONE) {
      // All loads are issued before any of them is used: the issue order is the program
      // order, so a conversion placed right behind its load would make every load wait for
      // the one before it (one memory round trip per block instead of one in total).
      Raw4 raw4[CPW * BPC];
#pragma unroll
      for (int u = 0; u < CPW * BPC; ++u) {
        const bool on = u / BPC < cnt;
        const int col = (on ? (w + 16 * (u / BPC)) * BPC + (u % BPC) : 0) * kBlock + lane * 4;
        raw4[u] = load4_raw(p.x, p.x_dtype, 0, col, on ? limit : 0, vec_ok);
      }
#pragma unroll
      for (int u = 0; u < CPW * BPC; ++u) cvt4(raw4[u], p.x_dtype, v[u]);
    } else {
      float scale = 1.f;
      if (p.pro == PE_PRO_ADD_RMSNORM) {
        // mean square of the updated residual over the whole row: every CTA computes it for itself (8 KB from
        // L2); CTA 0 also stores the updated residual for the launches that follow
        float ss = 0.f;
        for (int col = tid * 4; col < p.in_f; col += kRowThreads * 4) {
          float r[4];
          resid4(p, col, r);
          if (cta == 0 && p.resid_out)
            *reinterpret_cast<uint2*>(p.resid_out + col) = make_uint2(pack_half2(r[0], r[1]), pack_half2(r[2], r[3]));
          ss += r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3];
        }
        ss = warp_sum(ss);
        if (lane == 0) pro_red[w] = ss;
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (int i = 0; i < kRowWarps; ++i) tot += pro_red[i];
        scale = rsqrtf(tot / (float)p.in_f + p.eps);
      }
#pragma unroll
      for (int u = 0; u < CPW * BPC; ++u) {
        const bool on = u / BPC < cnt;
        const int col = (on ? (w + 16 * (u / BPC)) * BPC + (u % BPC) : 0) * kBlock + lane * 4;
        pro_load4(p, col, on, scale, v[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < CPW * BPC; ++u) {
      if (u / BPC < cnt) {  // warp-uniform
        if (raw) warp_fwht128(v[u], lane);
        uint8_t* dst = xw + (u / BPC) * 512 + (u % BPC) * 256;
        if (PACKED) {  // pairs (k, k+64), in pair order
          float o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = __shfl_xor_sync(0xffffffffu, v[u][i], 16);
          if (lane < 16)
            *reinterpret_cast<uint4*>(dst + lane * 16) = make_uint4(pack_half2(v[u][0], o[0]), pack_half2(v[u][1], o[1]),
                                                                    pack_half2(v[u][2], o[2]), pack_half2(v[u][3], o[3]));
        } else {
          *reinterpret_cast<uint2*>(dst + lane * 8) = make_uint2(pack_half2(v[u][0], v[u][1]), pack_half2(v[u][2], v[u][3]));
        }
      }
    }
    __syncwarp();
    const uint32_t xw_s = smem_u32(xw) + (PACKED ? (pc >> 2) * 256 + (pc & 3) * 64 : pc * 32);
#pragma unroll
    for (int j = 0; j < CPW; ++j) {
#pragma unroll
      for (int i = 0; i < kXPerChunk / 4; ++i) {
        uint4 t = make_uint4(0, 0, 0, 0);
        if (j < cnt) t = lds128(xw_s + j * 512 + i * 16);
        xr[j][4 * i + 0] = t.x; xr[j][4 * i + 1] = t.y; xr[j][4 * i + 2] = t.z; xr[j][4 * i + 3] = t.w;
      }
    }
  }
  if (!REGTAB) __syncthreads();  // the shared table has entries from every warp

  // ---- the item line, in passes of kPassRows rows
  const int n_warps_used = p.n_chunks < kRowWarps ? p.n_chunks : kRowWarps;
  const uint32_t norm_off = SUB * kItemBytes + rs * 4 + (PACKED ? (pc >> 2) * 2 : (w & 1) * 2);
  uint32_t st_rg = st_base;
  for (int rg0 = 0; rg0 < n_rg; rg0 += kPassRows / kGroupRows) {
    const int rg1 = n_rg < rg0 + kPassRows / kGroupRows ? n_rg : rg0 + kPassRows / kGroupRows;
    if (cnt > 0) {
      uint32_t part_s = smem_u32(part) + (rs * kPartStride + w) * 4;
      for (int rg = rg0; rg < rg1; ++rg) {
        const int rows_left = r_end - r_beg - kGroupRows * rg;  // sub-items beyond the CTA's rows were not fetched
        float acc[SUB];
#pragma unroll
        for (int sb = 0; sb < SUB; ++sb) acc[sb] = 0.f;
#pragma unroll
        for (int j = 0; j < CPW; ++j) {
          asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
          const uint32_t st = st_rg + j * kColStage;
          if (j < cnt) {
#pragma unroll
            for (int sb = 0; sb < SUB; ++sb) {
              if (4 * sb < rows_left) {  // warp-uniform
                const uint4 q = lds128(st + sb * kItemBytes + q_off);
                unsigned short nh;
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(nh) : "r"(st + norm_off + sb * 16));
                const float sdot = reg_dot<PACKED, REGTAB>(q, lane_base, tb, xr[j]);
                acc[sb] = fmaf(__half2float(__ushort_as_half(nh)), sdot, acc[sb]);
              }
            }
          }
          __syncwarp();  // every lane has read the slot before it is refilled
          fetch_item(st, j);
        }
        advance_fetch();
        st_rg += CPW * kColStage;
        if (st_rg == st_end) st_rg = st_base;
#pragma unroll
        for (int m = 1; m <= 4; m <<= 1) {
#pragma unroll
          for (int sb = 0; sb < SUB; ++sb) acc[sb] += __shfl_xor_sync(0xffffffffu, acc[sb], m);
        }
        if (pc == 0) {
#pragma unroll
          for (int sb = 0; sb < SUB; ++sb)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(part_s + sb * (4 * kPartStride * 4)), "f"(acc[sb]) : "memory");
        }
        part_s += kGroupRows * kPartStride * 4;
      }
    }
    __syncthreads();
    for (int r = tid; r < kGroupRows * (rg1 - rg0); r += kRowThreads) {
      const int row = r_beg + kGroupRows * rg0 + r;
      if (row < r_end) {
        float s = 0.f;
        for (int ww = 0; ww < n_warps_used; ++ww) s += part[r * kPartStride + ww];
        if (p.bias) s += __half2float(p.bias[row]);
        store_from_float(p.y, p.y_dtype, row, s);
      }
    }
    if (rg1 < n_rg) __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <bool PACKED, bool REGTAB, int CPW>
static int launch_cols(const ColArgs& a, int G, cudaStream_t st) {
  // Sub-items (4 rows each) per step = independent decode-multiply chains per lane.  Byte codes, whose
  // every weight is a table lookup of its own, gain from four (measured 0.3 us per launch on the
  // 4096-wide layers); nibble codes are as fast or faster with two and need fewer registers.
  constexpr int SUB = (!PACKED && CPW <= 3) ? 4 : 2;
  // items in flight per warp: 6 to 8 KB of codes
  constexpr int DEPTH = SUB == 4 ? (CPW == 3 ? 3 : 4) : (CPW == 4 ? 8 : 6);
  const unsigned dyn_bytes = (REGTAB ? 0u : (unsigned)kLutBytes) + kRowWarps * CPW * 512u + kPassRows * kPartStride * 4u +
                             kRowWarps * DEPTH * (unsigned)col_stage_bytes(SUB);
  auto kfn = gemv_cols_kernel<PACKED, REGTAB, CPW, DEPTH, SUB>;
  static thread_local bool configured[16] = {false};
  int dev = 0;
  PE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 16 || !configured[dev]) {
    PE_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_bytes));
    if (dev < 16) configured[dev] = true;
  }
  PE_CUDA_TRY(launch_pdl(kfn, dim3(G), dim3(kRowThreads), dyn_bytes, st, a));
  return PE_OK;
}

template <bool PACKED, bool REGTAB>
static int launch_cols_cpw(const ColArgs& a, int cpw, int G, cudaStream_t st) {
  switch (cpw) {
    case 1: return launch_cols<PACKED, REGTAB, 1>(a, G, st);
    case 2: return launch_cols<PACKED, REGTAB, 2>(a, G, st);
    case 3: return launch_cols<PACKED, REGTAB, 3>(a, G, st);
    case 4: return launch_cols<PACKED, REGTAB, 4>(a, G, st);
    default: return 1;
  }
}

struct ProArgs { int pro; const void* delta; int delta_dtype; const void* norm_w; void* resid_out; float eps; };

// batch 1: returns 1 if the shape is not this kernel's kind
static int gemv_cols_try(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                         const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype, int in_f, void* y,
                         int y_dtype, const void* bias, int out_f, int K, int sms, cudaStream_t stream,
                         const ProArgs* pro = nullptr) {
  const int64_t row_bytes = packed ? K / 2 : K;
  // norms are copied 4 bytes (two blocks) at a time: rows of norms must start 4-byte aligned and hold an even count
  if (row_bytes % 128 || (ld_norms & 1) || ((K / kBlock) & 1) || (reinterpret_cast<uintptr_t>(norms) & 3)) return 1;
  const int n_chunks = (int)(row_bytes / 128);
  const int cpw = (n_chunks + kRowWarps - 1) / kRowWarps;
  if (cpw > 4) return 1;
  // Small matrices (tensor-parallel shards) are latency bound: as many CTAs as there are groups of 8 rows, up to
  // one per SM.  Below 128 KB of codes the launch is all latency either way.
  const int G = out_f / 8 < sms ? out_f / 8 : sms;
  if (G < 1 || (long long)out_f * row_bytes < 131072) return 1;
  ColArgs a;
  a.codes = static_cast<const uint8_t*>(codes); a.ld_codes = ld_codes;
  a.norms = static_cast<const uint8_t*>(norms); a.ld_norms = ld_norms * 2;
  a.ct = ct_scaled; a.n_levels = n_levels;
  a.x = x; a.x_kind = x_kind; a.x_dtype = x_dtype; a.in_f = in_f;
  a.y = y; a.y_dtype = y_dtype;
  a.bias = static_cast<const __half*>(bias);
  a.N = out_f; a.K = K; a.n_chunks = n_chunks;
  a.pro = pro ? pro->pro : PE_PRO_NONE;
  a.delta = pro ? pro->delta : nullptr; a.delta_dtype = pro ? pro->delta_dtype : PE_F16;
  a.norm_w = pro ? static_cast<const __half*>(pro->norm_w) : nullptr;
  a.resid_out = pro ? static_cast<__half*>(pro->resid_out) : nullptr;
  a.eps = pro ? pro->eps : 0.f;
  if (packed && n_levels <= 8) return launch_cols_cpw<true, true>(a, cpw, G, stream);
  if (packed) return launch_cols_cpw<true, false>(a, cpw, G, stream);
  return launch_cols_cpw<false, false>(a, cpw, G, stream);
}

}  // namespace pe

// ---- batch-1 matmul with the glue op in front of it computed while the input is staged ----
// Checks of the operands that both layouts share.
static int pro_check(const float* ct_scaled, int n_levels, int packed, int prologue, const void* x, int in_f, const void* delta, int delta_dtype,
                     const void* norm_weight, const void* resid_out, const void* y, int y_dtype, int out_f, int in_f_padded) {
  if (!ct_scaled || !x || !y) return PE_ERR_ARG;
  if (prologue != PE_PRO_ADD_RMSNORM && prologue != PE_PRO_SILU_MUL) return PE_ERR_ARG;
  if (prologue == PE_PRO_ADD_RMSNORM && (!norm_weight || (delta && delta_dtype != PE_F16 && delta_dtype != PE_F32))) return PE_ERR_ARG;
  if (out_f < 1 || in_f < 4 || in_f > in_f_padded || y_dtype < PE_F32 || y_dtype > PE_BF16) return PE_ERR_ARG;
  if (n_levels < 2 || n_levels > 256 || (packed && n_levels > 16)) return PE_ERR_ARG;
  if (in_f_padded % pe::kBlock || in_f % 4) return PE_ERR_SHAPE;
  // the prologue reads its operands 8 or 16 bytes at a time
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(norm_weight) |
       reinterpret_cast<uintptr_t>(resid_out)) & 15)
    return PE_ERR_ALIGN;
  if (prologue == PE_PRO_SILU_MUL && (in_f % 8)) return PE_ERR_SHAPE;  // the `up` half starts in_f elements in: keep it 16-byte aligned
  return PE_OK;
}

extern "C" int pe_gemv_pro(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                           const float* ct_scaled, int n_levels, int prologue, const void* x, int in_f, const void* delta,
                           int delta_dtype, const void* norm_weight, void* resid_out, float eps, void* y, int y_dtype,
                           const void* bias, int out_f, int in_f_padded, void* stream) {
  using namespace pe;
  if (!codes || !norms) return PE_ERR_ARG;
  const int c = pro_check(ct_scaled, n_levels, packed, prologue, x, in_f, delta, delta_dtype, norm_weight, resid_out, y, y_dtype, out_f, in_f_padded);
  if (c != PE_OK) return c;
  if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15)) return PE_ERR_ALIGN;
  if (ld_codes < (packed ? in_f_padded / 2 : in_f_padded) || ld_norms < in_f_padded / kBlock) return PE_ERR_ARG;
  const int sms = sm_count();
  if (sms <= 0) return PE_ERR_CUDA;
  ProArgs pro = {prologue, delta, delta_dtype, norm_weight, resid_out, eps};
  const int r = gemv_cols_try(codes, packed, ld_codes, norms, ld_norms, ct_scaled, n_levels, x, PE_X_RAW, PE_F16, in_f, y, y_dtype,
                              bias, out_f, in_f_padded, sms, static_cast<cudaStream_t>(stream), &pro);
  return r == 1 ? PE_ERR_SHAPE : r;  // shapes the column-owner kernel does not take: the caller runs the separate launches
}

// The same over the bulk-copy kernel: the op is computed where the activations are prepared.
static int pro_bulk(pe::GemvBulkCall& q, int prologue, const float* ct_scaled, int n_levels, const void* x, int in_f, const void* delta, int delta_dtype,
                    const void* norm_weight, void* resid_out, float eps, void* y, int y_dtype, const void* bias, int out_f, int in_f_padded,
                    void* workspace, size_t workspace_bytes, void* stream) {
  using namespace pe;
  const int c = pro_check(ct_scaled, n_levels, q.packed, prologue, x, in_f, delta, delta_dtype, norm_weight, resid_out, y, y_dtype, out_f, in_f_padded);
  if (c != PE_OK) return c;
  if (reinterpret_cast<uintptr_t>(workspace) & 15) return PE_ERR_ALIGN;
  if (workspace_bytes < pe_gemv_scratch_bytes(1, in_f_padded)) return PE_ERR_WORKSPACE;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  q.ct_scaled = ct_scaled; q.n_levels = n_levels;
  q.x = x; q.x_kind = prologue == PE_PRO_SILU_MUL ? PE_X_SILU_MUL : PE_X_RAW; q.x_dtype = PE_F16; q.ld_x = 2 * (int64_t)in_f; q.in_f = in_f;
  q.y = y; q.y_dtype = y_dtype; q.ld_y = out_f; q.bias = bias;
  q.batch = 1; q.out_f = out_f; q.in_f_padded = in_f_padded;
  q.status = reinterpret_cast<int*>(ws + kGemvStatusBytes - 4);
  q.frags = ws + kGemvStatusBytes;
  q.pro = prologue == PE_PRO_ADD_RMSNORM ? prologue : PE_PRO_NONE;
  q.delta = delta; q.delta_dtype = delta_dtype; q.norm_w = norm_weight; q.resid_out = resid_out; q.eps = eps;
  return gemv_bulk_run(q, static_cast<cudaStream_t>(stream));
}

extern "C" int pe_gemv_pro_scratch(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms, const float* ct_scaled,
                                   int n_levels, int prologue, const void* x, int in_f, const void* delta, int delta_dtype, const void* norm_weight,
                                   void* resid_out, float eps, void* y, int y_dtype, const void* bias, int out_f, int in_f_padded, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  if (!codes || !norms || !workspace) return PE_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15)) return PE_ERR_ALIGN;
  if (ld_codes < (packed ? in_f_padded / 2 : in_f_padded) || ld_norms < in_f_padded / pe::kBlock) return PE_ERR_ARG;
  pe::GemvBulkCall q = {};
  q.codes = codes; q.packed = packed; q.ld_codes = ld_codes; q.norms = norms; q.ld_norms = ld_norms;
  return pro_bulk(q, prologue, ct_scaled, n_levels, x, in_f, delta, delta_dtype, norm_weight, resid_out, eps, y, y_dtype, bias, out_f, in_f_padded,
                  workspace, workspace_bytes, stream);
}

extern "C" int pe_gemv_pro_tiled(const void* tiles, int packed, const float* ct_scaled, int n_levels, int prologue, const void* x, int in_f,
                                 const void* delta, int delta_dtype, const void* norm_weight, void* resid_out, float eps, void* y,
                                 int y_dtype, const void* bias, int out_f, int in_f_padded, void* workspace, size_t workspace_bytes,
                                 void* stream) {
  if (!tiles || !workspace) return PE_ERR_ARG;
  if (reinterpret_cast<uintptr_t>(tiles) & 15) return PE_ERR_ALIGN;
  pe::GemvBulkCall q = {};
  q.tiles = tiles; q.packed = packed;
  return pro_bulk(q, prologue, ct_scaled, n_levels, x, in_f, delta, delta_dtype, norm_weight, resid_out, eps, y, y_dtype, bias, out_f, in_f_padded,
                  workspace, workspace_bytes, stream);
}
