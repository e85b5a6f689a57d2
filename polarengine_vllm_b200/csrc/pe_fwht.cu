// Stand-alone rotation and nibble-packing kernels (small, HBM-trivial).
#include "pe_common.cuh"

namespace pe {

// One warp per 128-block: pad, rotate (register + shuffle butterflies), convert, store.
__global__ void __launch_bounds__(256) fwht128_kernel(const void* x, int x_dtype, int64_t ld_x, void* out,
                                                      int out_dtype, int64_t ld_out, int batch, int in_f,
                                                      int nb) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t total = (int64_t)batch * nb;
  if (warp >= total) return;  // whole warps leave together
  const int m = (int)(warp / nb), blk = (int)(warp - (int64_t)m * nb);
  const bool vin = (ld_x % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
  float v[4];
  load4_as_float(x, x_dtype, (int64_t)m * ld_x, blk * kBlock + lane * 4, in_f, vin, v);
  warp_fwht128(v, lane);
  const int64_t o = (int64_t)m * ld_out + blk * kBlock + lane * 4;
  const bool vout = (ld_out % 4 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
  if (vout && out_dtype == PE_F32) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + o) = make_float4(v[0], v[1], v[2], v[3]);
  } else if (vout && out_dtype == PE_F16) {
    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(out) + o) = make_uint2(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) store_from_float(out, out_dtype, o + i, v[i]);
  }
}

// One thread per 16 output bytes: 16 codes of the first half, 16 of the second half.
__global__ void __launch_bounds__(256) pack_nibble_kernel(const int8_t* codes, uint8_t* packed, int64_t n_chunks) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_chunks) return;
  // chunk i covers packed bytes [16 i, 16 i + 16): block = i / 4, offset (i % 4) * 16 inside its 64 bytes
  const int64_t blk = i >> 2;
  const int off = (int)(i & 3) * 16;
  const uint4 lo = *reinterpret_cast<const uint4*>(codes + blk * kBlock + off);
  const uint4 hi = *reinterpret_cast<const uint4*>(codes + blk * kBlock + 64 + off);
  uint4 r;
  r.x = (lo.x & 0x0f0f0f0fu) | ((hi.x & 0x0f0f0f0fu) << 4);
  r.y = (lo.y & 0x0f0f0f0fu) | ((hi.y & 0x0f0f0f0fu) << 4);
  r.z = (lo.z & 0x0f0f0f0fu) | ((hi.z & 0x0f0f0f0fu) << 4);
  r.w = (lo.w & 0x0f0f0f0fu) | ((hi.w & 0x0f0f0f0fu) << 4);
  *reinterpret_cast<uint4*>(packed + i * 16) = r;
}

// ---- quantizer --------------------------------------------------------------------------------
// Zero-pad, L2 norm clamped at 1e-10, divide, rotate, scale by sqrt(128), nearest Lloyd-Max level by distance (first
// minimum wins, as the reference's argmin does), int8 code and fp16 norm out.  The butterfly rotation and the tree
// sum of squares round differently from the reference's matrix product and torch.norm, so a value that sits on a
// cell boundary to within fp32 rounding can land on the other side: a few codes per million differ from the CPU
// quantizer.
//
// fp32 weights (quantize_kernel): the launch is bound by instruction issue and the shared-memory port (two exchanges and two
// lookups per weight), not by memory (four bytes in, one out).  Four lanes share a 128-block, in four pieces of 8 consecutive values each: five
// of the seven butterfly stages stay in registers, a warp reads and writes whole sectors, the level is found with one
// table lookup and one comparison instead of a scan of all levels, the quotient is a product with the reciprocal and
// one correction, and fp32 arithmetic goes two values per instruction.  4096 x 12288, on 2 resident CTAs per SM
// with the next trip's loads in flight: to 4 bits 71 us, to 6 bits 75.

// Exact cell edges: the rotated unit-vector element v takes code j when j edges are below it.  edge[j] is the largest
// float that is still no farther from level j than from level j + 1 by the fp32 distances quant_dist() that a scan
// compares.  A uniform grid over [-1.06, 1.06] (elements of a unit vector) gives the edges below an element's cell; a
// cell holds at most one, so one comparison settles the code.
constexpr float kQuantRange = 1.06f;
__device__ __forceinline__ float quant_dist(float v, float level) { return fabsf(fmaf(v, 11.313708498984761f, -level)); }  // sqrt(128)
struct QuantTable {
  float edge[256];      // edge[n_levels - 1] = +inf
  uint8_t first[2048];  // edges in lower cells
  uint16_t cell[256];   // cell of each edge
};

// the sum with 1.5 * 2^23 has the cell in its low mantissa bits
__device__ __forceinline__ uint32_t quant_cell(float x, float scale, float magic, uint32_t mask) {
  return __float_as_uint(fmaf(x, scale, magic)) & mask;
}

// Returns whether the levels have to be scanned instead: not ascending, closer than fp32 distances or the grid
// resolve, or far outside the range of the values.
__device__ __forceinline__ bool build_quant_table(QuantTable& q, float* lv, const float* levels, int n, uint32_t cells, float scale, float magic) {
  const int tid = threadIdx.x;
  if (tid < n) lv[tid] = levels[tid];
  __syncthreads();
  bool bad = false;
  if (tid < n) {
    float e = __int_as_float(0x7f800000);
    if (tid + 1 < n) {
      const float lo = lv[tid], hi = lv[tid + 1];
      bad = !(hi - lo > 1e-4f && fabsf(lo) < 11.3f && fabsf(hi) < 11.3f);
      if (!bad) {  // halve [e, above] until the two are neighbours: `above` is nearer to hi, e is not
        const float m0 = 0.5f * (lo + hi) * 0.08838834764831845f, near_lo = m0 - 1e-6f, near_hi = m0 + 1e-6f;
        const bool lo_ok = !(quant_dist(near_lo, hi) < quant_dist(near_lo, lo)), hi_ok = quant_dist(near_hi, hi) < quant_dist(near_hi, lo);
        e = lo_ok ? near_lo : lo * 0.08838834764831845f;
        float above = hi_ok ? near_hi : hi * 0.08838834764831845f;
        for (int i = 0; i < 200; ++i) {
          const float m = 0.5f * (e + above);
          if (m == e || m == above) break;
          if (quant_dist(m, hi) < quant_dist(m, lo)) above = m;
          else e = m;
        }
        q.cell[tid] = (uint16_t)quant_cell(e, scale, magic, cells - 1);
      }
    }
    q.edge[tid] = e;
  }
  if (__syncthreads_or(bad)) return true;
  if (tid < n) {  // edge tid is the first one not below the cells from its lower neighbour's (exclusive) to its own
    const int c0 = tid ? q.cell[tid - 1] + 1 : 0, c1 = tid + 1 < n ? q.cell[tid] : (int)cells - 1;
    for (int c = c0; c <= c1; ++c) q.first[c] = (uint8_t)tid;
    bad = tid && tid + 1 < n && c0 > c1;
  }
  return __syncthreads_or(bad);
}

// 8 consecutive weights from column `col` of a row, zero from in_f on: the load and the conversion, so that the next
// trip's loads are in flight while this one's values are worked on
template <int W_DTYPE> struct Raw8 { uint4 q[W_DTYPE == PE_F32 ? 2 : 1]; };

template <int W_DTYPE>
__device__ __forceinline__ Raw8<W_DTYPE> load8_raw(const void* w, int64_t row_off, int col, int in_f, bool vec_ok) {
  constexpr int kSize = W_DTYPE == PE_F32 ? 4 : 2, kQuads = W_DTYPE == PE_F32 ? 2 : 1;
  Raw8<W_DTYPE> r;
  const uint8_t* src = static_cast<const uint8_t*>(w) + (row_off + col) * kSize;
  if (vec_ok && col + 8 <= in_f) {
#pragma unroll
    for (int i = 0; i < kQuads; ++i) r.q[i] = ldg_stream(src + 16 * i);
  } else {
    uint32_t u[4 * kQuads];
#pragma unroll
    for (int i = 0; i < 4 * kQuads; ++i) {
      if (W_DTYPE == PE_F32) {
        u[i] = col + i < in_f ? reinterpret_cast<const uint32_t*>(src)[i] : 0u;
      } else {
        const uint16_t* h = reinterpret_cast<const uint16_t*>(src);
        u[i] = (col + 2 * i < in_f ? h[2 * i] : 0u) | (col + 2 * i + 1 < in_f ? (uint32_t)h[2 * i + 1] << 16 : 0u);
      }
    }
#pragma unroll
    for (int i = 0; i < kQuads; ++i) r.q[i] = make_uint4(u[4 * i], u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]);
  }
  return r;
}

// ---- 16-bit weights: the rotation on the tensor cores ------------------------------------------------------------
// A value's index in its block is 8 a + j.  Lane (g, t) of a warp has the values of a = 2 t, 2 t + 1, 8 + 2 t and 9 + 2 t of block g
// (32 bytes at a time, so that a warp reads whole lines), which is what operand A of an m16n8k16 product wants of row g with
// k = a; rows 8 to 15 stay zero.  Products 2 j and 2 j + 1 are the two halves of the 16-point transform over a of the eight
// blocks' values j: 16-bit values times +-1, exact products, added in fp32 by the tensor core, which does not round every sum to
// the nearest as an addition does.  bf16 values are multiplied by +-2^-8 instead: 128 of the largest then stay finite, so that a
// finite block has no infinity or NaN among its rotated values however large they are (with +-1 the block of a sum past the
// largest fp32 number came out as NaN: norm 0, codes 0).  The lane gets back the same a of its own block, so that the
// eight-point transform over j, the norm and sixteen consecutive codes twice need no other lane but for one sum of four.
// (With the blocks as columns of the product the codes came out four blocks a lane: 59 us where this takes 55.)  The norm is that of
// the rotated values, which are divided by it afterwards: fewer roundings on the way than dividing first.  Codes that are not
// the nearest level in 64 bits, of 16.8 million: 16 at 4 bits, 31 at 6 (with the butterflies 15 and 35).
// What bounds it: the L1 data port, 76 % busy (a cycle per 32-byte sector that comes or goes, two look-ups a value), and the chain of
// a trip.  4096 x 12288 bf16 against the butterfly kernel: to 4 bits 62 -> 55 us, to 6 bits 67 -> 58.
template <int W_DTYPE>
__device__ __forceinline__ void mma_first(float2& d, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  float unused0, unused1;
  if (W_DTYPE == PE_F16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%9,%9,%9,%9};"
        : "=f"(d.x), "=f"(d.y), "=f"(unused0), "=f"(unused1) : "r"(a0), "r"(0), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%9,%9,%9,%9};"
        : "=f"(d.x), "=f"(d.y), "=f"(unused0), "=f"(unused1) : "r"(a0), "r"(0), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}

// Two CTAs an SM request the next trip's values ahead (116 registers); three do not (80).  FEW: at most 64 levels.
template <int W_DTYPE, int CTAS, bool FEW>
__global__ void __launch_bounds__(256, CTAS) quantize16_kernel(const void* w, int64_t ld_w, int64_t rows, int in_f, int nb,
                                                            const float* levels, int n_levels, int8_t* codes, int64_t ld_codes,
                                                            __half* norms, int64_t ld_norms, int vec_out) {
  __shared__ float lv[256];
  __shared__ QuantTable q;
  uint32_t cells = 64;  // as quantize_kernel
  while ((int)cells < 16 * n_levels && cells < 2048) cells *= 2;
  const float scale = (float)cells / (2.f * kQuantRange), magic = 12582912.f + (float)(cells / 2);
  const bool scan = build_quant_table(q, lv, levels, n_levels, cells, scale, magic);
  if (FEW && !scan) {  // up to 64 levels: four times the level, the byte offset of its edge
    for (int c = threadIdx.x; c < (int)cells; c += blockDim.x) q.first[c] *= 4;
    __syncthreads();
  }
  constexpr uint32_t kOne = FEW ? 4 : 1;
  auto edge_of = [&](uint32_t j) { return FEW ? *reinterpret_cast<const float*>(reinterpret_cast<const char*>(q.edge) + j) : q.edge[j]; };
  const uint32_t mask = cells - 1;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t n_warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const bool vin = (ld_w * 2) % 16 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0, vin32 = (ld_w * 2) % 32 == 0 && (reinterpret_cast<uintptr_t>(w) & 31) == 0;
  const int64_t first = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 8 + g;
  int64_t r = first / nb;
  int blk = (int)(first - r * nb);
  const int64_t step_r = n_warps * 8 / nb;
  const int step_b = (int)(n_warps * 8 - step_r * nb);
  // sign of H16: the parity of the bits that column n (g, g + 8) and index a (2 t, 2 t + 1 and 8 further on) share
  constexpr uint32_t one = W_DTYPE == PE_F16 ? 0x3c00u : 0x3b80u;  // 1, 2^-8
  constexpr float kBack = W_DTYPE == PE_F16 ? 1.f : 256.f;
  const uint32_t sign = (uint32_t)(__popc(g & 2 * t) & 1) << 15;
  const uint32_t h0 = one | sign | (one | (sign ^ ((uint32_t)(g & 1) << 15))) << 16, h1 = h0 ^ 0x80008000u;
  Raw8<W_DTYPE> raw[4];
  auto request = [&]() {  // block (r, blk) of the weight, zeros past its last row
    const int col = blk * kBlock + t * 16;
    if (vin32 && r < rows && (blk + 1) * kBlock <= in_f) {
      const uint16_t* src = static_cast<const uint16_t*>(w) + r * ld_w + col;
#pragma unroll
      for (int p = 0; p < 4; p += 2)
        asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(raw[p].q[0].x), "=r"(raw[p].q[0].y), "=r"(raw[p].q[0].z), "=r"(raw[p].q[0].w), "=r"(raw[p + 1].q[0].x),
                       "=r"(raw[p + 1].q[0].y), "=r"(raw[p + 1].q[0].z), "=r"(raw[p + 1].q[0].w) : "l"(src + 32 * p));
      return;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
      raw[p] = load8_raw<W_DTYPE>(w, r < rows ? r * ld_w : 0, col + (p >> 1) * 64 + (p & 1) * 8, r < rows ? in_f : 0, vin);
  };
  if (CTAS == 2) request();
  while (__any_sync(0xffffffffu, r < rows)) {
    if (CTAS != 2) request();
    const int64_t r_out = r;
    const int blk_out = blk;
    float2 v[8][2];  // values 8 (2 t + 8 h) + j (x) and 8 further on (y)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint32_t u[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) u[p] = j < 2 ? raw[p].q[0].x : j < 4 ? raw[p].q[0].y : j < 6 ? raw[p].q[0].z : raw[p].q[0].w;
      const uint32_t sel = j & 1 ? 0x7632 : 0x5410;
      const uint32_t x0 = __byte_perm(u[0], u[1], sel), x1 = __byte_perm(u[2], u[3], sel);
      mma_first<W_DTYPE>(v[j][0], x0, x1, h0, h0);
      mma_first<W_DTYPE>(v[j][1], x0, x1, h0, h1);
    }
    r += step_r;
    blk += step_b;
    if (blk >= nb) { blk -= nb; ++r; }
    if (CTAS == 2) request();
    const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (!(j & o))
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 a = v[j][h], b = v[j | o][h];
            v[j][h] = add2(a, b);
            v[j | o][h] = fma2(b, minus, a);
          }
    // the rotation keeps the norm: the squares of its results, sqrt(128) too large, sum to 128 times the block's
    const float s128 = 0.08838834764831845f * kBack;  // 1/sqrt(128)
    float2 squares = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) squares = fma2(v[j][h], v[j][h], squares);
    float sum = squares.x + squares.y;
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    float nrm = fmaxf(sqrtf(sum) * s128, 1e-10f), inv = __fdiv_rn(s128, nrm);
    // A norm whose square overflows, infinities, NaN: the norm and the codes of quantize_kernel, from the block itself.  The square of
    // the norm is infinite or NaN there; finite values become zero, a value that is not finite makes the whole block NaN.
    if (__any_sync(0xffffffffu, !(sum < 6.6461399789245794e35f))) {  // 128 * 2^128 / 2^16
      float own = 0.f, finite = 0.f;
#pragma unroll 1
      for (int i = 0; i < 32; ++i) {
        const int col = blk_out * kBlock + t * 32 + i;
        const uint16_t h = r_out < rows && col < in_f ? static_cast<const uint16_t*>(w)[r_out * ld_w + col] : (uint16_t)0;
        const float u = W_DTYPE == PE_F16 ? __half2float(__ushort_as_half(h)) : __uint_as_float((uint32_t)h << 16);
        own = fmaf(u, u, own);
        finite = fmaf(u, 0.f, finite);
      }
#pragma unroll
      for (int i = 1; i <= 2; i <<= 1) { own += __shfl_xor_sync(0xffffffffu, own, i); finite += __shfl_xor_sync(0xffffffffu, finite, i); }
      if (!(sum < 6.6461399789245794e35f)) {
        nrm = fmaxf(sqrtf(own), 1e-10f);
        inv = finite == 0.f ? __fdiv_rn(s128, nrm) : finite;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) v[j][h] = mul2(v[j][h], make_float2(inv, inv));
    uint32_t packed[2][2][2];  // half of the block, a, four codes each
#pragma unroll
    for (int i = 0; i < 8; ++i) packed[i >> 2][(i >> 1) & 1][i & 1] = 0;
    if (!scan) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 x = v[j][h], c = fma2(x, make_float2(scale, scale), make_float2(magic, magic));  // quant_cell of both
          const uint32_t jx = q.first[__float_as_uint(c.x) & mask], jy = q.first[__float_as_uint(c.y) & mask];
          uint32_t &px = packed[h][0][j >> 2], &py = packed[h][1][j >> 2];
          px += jx << (8 * (j & 3));
          py += jy << (8 * (j & 3));
          if (x.x > edge_of(jx)) px += kOne << (8 * (j & 3));
          if (x.y > edge_of(jy)) py += kOne << (8 * (j & 3));
        }
      if (FEW)
#pragma unroll
        for (int i = 0; i < 8; ++i) packed[i >> 2][(i >> 1) & 1][i & 1] >>= 2;
      if (inv != inv)  // a value that is not finite
#pragma unroll
        for (int i = 0; i < 8; ++i) packed[i >> 2][(i >> 1) & 1][i & 1] = 0;
    } else {
#pragma unroll 1
      for (int i = 0; i < 32; ++i) {
        float x = 0.f;
#pragma unroll
        for (int k = 0; k < 32; ++k)
          if (k == i) x = ((k >> 3) & 1) ? v[k & 7][k >> 4].y : v[k & 7][k >> 4].x;
        uint32_t best = 0;
        float bd = quant_dist(x, lv[0]);
        for (int j = 1; j < n_levels; ++j) {
          const float d = quant_dist(x, lv[j]);
          if (d < bd) { bd = d; best = j; }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k == i >> 2) packed[k >> 2][(k >> 1) & 1][k & 1] |= best << (8 * (i & 3));
      }
    }
    if (r_out < rows) {
      int8_t* dst = codes + r_out * ld_codes + blk_out * kBlock + t * 16;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 c = make_uint4(packed[h][0][0], packed[h][0][1], packed[h][1][0], packed[h][1][1]);
        if (vec_out) {
          *reinterpret_cast<uint4*>(dst + 64 * h) = c;
        } else {
          uint32_t* d = reinterpret_cast<uint32_t*>(dst + 64 * h);
          d[0] = c.x; d[1] = c.y; d[2] = c.z; d[3] = c.w;
        }
      }
      if (t == 0) norms[r_out * ld_norms + blk_out] = __float2half_rn(nrm);
    }
  }
}

__global__ void __launch_bounds__(256, 2) quantize_kernel(const void* w, int64_t ld_w, int64_t rows, int in_f, int nb,
                                                          const float* levels, int n_levels, int8_t* codes, int64_t ld_codes,
                                                          __half* norms, int64_t ld_norms, int vec_out) {
  __shared__ float lv[256];
  __shared__ QuantTable q;
  uint32_t cells = 64;  // at least 16 per level, which Lloyd-Max levels of every width need; 8 per level at 256
  while ((int)cells < 16 * n_levels && cells < 2048) cells *= 2;
  const float scale = (float)cells / (2.f * kQuantRange), magic = 12582912.f + (float)(cells / 2);
  const bool scan = build_quant_table(q, lv, levels, n_levels, cells, scale, magic);
  const uint32_t mask = cells - 1;
  const int lane = threadIdx.x & 31, part = lane & 3;
  const int64_t n_warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const bool vin = ld_w * 4 % 16 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  // block (row r, column block blk) of this lane, and how far one trip of the grid advances it
  const int64_t first = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 8 + (lane >> 2);
  int64_t r = first / nb;
  int blk = (int)(first - r * nb);
  const int64_t step_r = n_warps * 8 / nb;
  const int step_b = (int)(n_warps * 8 - step_r * nb);
  Raw8<PE_F32> raw[4];
  auto request = [&]() {  // block (r, blk) of the weight, zeros past its last row
#pragma unroll
    for (int p = 0; p < 4; ++p)
      raw[p] = load8_raw<PE_F32>(w, r < rows ? r * ld_w : 0, blk * kBlock + p * 32 + part * 8, r < rows ? in_f : 0, vin);
  };
  request();
  while (__any_sync(0xffffffffu, r < rows)) {
    const int64_t r_out = r;
    const int blk_out = blk;
    // element k of the block: bits 6..5 of k choose one of the lane's four pieces, bits 4..3 the lane, bits 2..0 the
    // place in the piece; v[4 * piece + i] holds places i and i + 4
    float2 v[16];
    float s[2];  // groups of four (places 0..3, 4..7), then a tree over the 32 groups, widest distance first
    {
      float u[4][8], g[4][2];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 x = raw[p].q[h];
          u[p][4 * h] = __uint_as_float(x.x); u[p][4 * h + 1] = __uint_as_float(x.y);
          u[p][4 * h + 2] = __uint_as_float(x.z); u[p][4 * h + 3] = __uint_as_float(x.w);
        }
      r += step_r;
      blk += step_b;
      if (blk >= nb) { blk -= nb; ++r; }
      request();
#pragma unroll
      for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          g[p][h] = u[p][4 * h] * u[p][4 * h] + u[p][4 * h + 1] * u[p][4 * h + 1] + u[p][4 * h + 2] * u[p][4 * h + 2] + u[p][4 * h + 3] * u[p][4 * h + 3];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * p + i] = make_float2(u[p][i], u[p][i + 4]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) s[h] = (g[0][h] + g[2][h]) + (g[1][h] + g[3][h]);
    }
#pragma unroll
    for (int m = 2; m >= 1; m >>= 1) {
#pragma unroll
      for (int h = 0; h < 2; ++h) s[h] += __shfl_xor_sync(0xffffffffu, s[h], m);
    }
    const float nrm = fmaxf(sqrtf(s[0] + s[1]), 1e-10f);
    // v / nrm: with y the rounded reciprocal and d = v * y, the remainder fma(-d, nrm, v) is exact and d + rem * y
    // is the rounded quotient (P. Markstein, IBM J. Res. Dev. 34, 1990) while nothing over- or underflows
    if (nrm > 1e-9f && nrm < 1e18f) {
      const float y = __frcp_rn(nrm);
      const float2 y2 = make_float2(y, y), n2 = make_float2(-nrm, -nrm);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 d = mul2(v[i], y2);
        v[i] = fma2(fma2(d, n2, v[i]), y2, d);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = make_float2(__fdiv_rn(v[i].x, nrm), __fdiv_rn(v[i].y, nrm));
    }
    // FWHT-128 in the order of the strides: 1, 2 between pairs, 4 inside them, 8, 16 between lanes, 32, 64 between pieces
    const float2 minus = make_float2(-1.f, -1.f);
    auto between_pairs = [&](int h) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (!(i & h)) {
          const float2 a = v[i], b = v[i | h];
          v[i] = add2(a, b);
          v[i | h] = fma2(b, minus, a);
        }
    };
    between_pairs(1);
    between_pairs(2);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = make_float2(v[i].x + v[i].y, v[i].x - v[i].y);
#pragma unroll
    for (int m = 1; m <= 2; m <<= 1) {
      const float sgn = (part & m) ? -1.f : 1.f;
      const float2 sgn2 = make_float2(sgn, sgn);
#pragma unroll
      for (int i = 0; i < 16; ++i)
        v[i] = fma2(sgn2, v[i], make_float2(__shfl_xor_sync(0xffffffffu, v[i].x, m), __shfl_xor_sync(0xffffffffu, v[i].y, m)));
    }
    between_pairs(4);
    between_pairs(8);
    const float s128 = 0.08838834764831845f;  // 1/sqrt(128)
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = mul2(v[i], make_float2(s128, s128));
    uint32_t packed[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) packed[i] = 0;
    if (!scan) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 c = fma2(v[i], make_float2(scale, scale), make_float2(magic, magic));  // quant_cell of both
        uint32_t jx = q.first[__float_as_uint(c.x) & mask], jy = q.first[__float_as_uint(c.y) & mask];
        jx += v[i].x > q.edge[jx];
        jy += v[i].y > q.edge[jy];
        packed[i >> 2 << 1] |= jx << (8 * (i & 3));
        packed[(i >> 2 << 1) + 1] |= jy << (8 * (i & 3));
      }
      if (v[0].x != v[0].x) {  // a NaN reaches the whole block
#pragma unroll
        for (int i = 0; i < 8; ++i) packed[i] = 0;
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < 32; ++i) {
        float x = 0.f;
#pragma unroll
        for (int k = 0; k < 32; ++k)
          if (k == i) x = (k & 4) ? v[(k >> 3) * 4 + (k & 3)].y : v[(k >> 3) * 4 + (k & 3)].x;
        uint32_t best = 0;
        float bd = quant_dist(x, lv[0]);
        for (int j = 1; j < n_levels; ++j) {
          const float d = quant_dist(x, lv[j]);
          if (d < bd) { bd = d; best = j; }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k == i >> 2) packed[k] |= best << (8 * (i & 3));
      }
    }
    if (r_out < rows) {
      int8_t* dst = codes + r_out * ld_codes + blk_out * kBlock + part * 8;
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        if (vec_out) {
          *reinterpret_cast<uint2*>(dst + p * 32) = make_uint2(packed[2 * p], packed[2 * p + 1]);
        } else {
          reinterpret_cast<uint32_t*>(dst + p * 32)[0] = packed[2 * p];
          reinterpret_cast<uint32_t*>(dst + p * 32)[1] = packed[2 * p + 1];
        }
      }
      if (part == 0) norms[r_out * ld_norms + blk_out] = __float2half_rn(nrm);
    }
  }
}

// Quantized embedding lookup: row ids[t] of the table is dequantised on the fly.
// One warp per (token, 128-block): centroid gather, inverse rotation (the rotation is its
// own inverse), block norm, cast.
__global__ void __launch_bounds__(256) embed_kernel(const uint8_t* codes, int packed, int64_t ld_codes, const __half* norms,
                                                    int64_t ld_norms, const float* ct, int n_levels, const int64_t* ids,
                                                    int64_t vocab, void* out, int out_dtype, int64_t ld_out, int tokens,
                                                    int hidden, int nb) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (warp >= (int64_t)tokens * nb) return;
  const int t = (int)(warp / nb), blk = (int)(warp - (int64_t)t * nb);
  int64_t row = ids[t];
  const bool ok = row >= 0 && row < vocab;  // out-of-range ids give a zero row
  if (!ok) row = 0;
  float v[4];
  if (packed) {
    // elements 4l..4l+3: low nibbles of bytes 4l.. for l < 16, high nibbles of bytes 4(l-16).. otherwise
    const uint32_t w = *reinterpret_cast<const uint32_t*>(codes + row * ld_codes + blk * 64 + (lane & 15) * 4);
    const uint32_t nib = (lane < 16 ? w : (w >> 4)) & 0x0f0f0f0fu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (nib >> (8 * i)) & 0xff;
      v[i] = c < n_levels ? __ldg(ct + c) : 0.f;
    }
  } else {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(codes + row * ld_codes + blk * kBlock + lane * 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (w >> (8 * i)) & 0xff;
      v[i] = c < n_levels ? __ldg(ct + c) : 0.f;
    }
  }
  warp_fwht128(v, lane);
  const float nrm = ok ? __half2float(norms[row * ld_norms + blk]) : 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int col = blk * kBlock + lane * 4 + i;
    if (col < hidden) store_from_float(out, out_dtype, (int64_t)t * ld_out + col, v[i] * nrm);
  }
}

}  // namespace pe

using namespace pe;

extern "C" int pe_embedding(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                            const float* ct_scaled, int n_levels, const int64_t* ids, int64_t vocab, void* out,
                            int out_dtype, int64_t ld_out, int tokens, int hidden, int hidden_padded, void* stream) {
  if (!codes || !norms || !ct_scaled || !ids || !out || tokens < 1 || hidden < 1 || vocab < 1) return PE_ERR_ARG;
  if (out_dtype < PE_F32 || out_dtype > PE_BF16 || n_levels < 2 || n_levels > 256 || (packed && n_levels > 16)) return PE_ERR_ARG;
  if (hidden_padded % kBlock || hidden > hidden_padded || hidden_padded - hidden >= kBlock) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(codes) & 3) || (ld_codes & 3)) return PE_ERR_ALIGN;
  if (ld_out < hidden) return PE_ERR_ARG;
  const int nb = hidden_padded / kBlock;
  const int64_t warps = (int64_t)tokens * nb;
  const int64_t blocks = (warps + 7) / 8;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  embed_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(codes), packed, ld_codes, static_cast<const __half*>(norms), ld_norms, ct_scaled, n_levels,
      ids, vocab, out, out_dtype, ld_out, tokens, hidden, nb);
  PE_CUDA_TRY(cudaGetLastError());
  return PE_OK;
}

extern "C" int pe_fwht128(const void* x, int x_dtype, int64_t ld_x, void* x_tf, int out_dtype, int64_t ld_out,
                          int batch, int in_f, int in_f_padded, void* stream) {
  if (!x || !x_tf || batch < 1 || in_f < 1) return PE_ERR_ARG;
  if (x_dtype < PE_F32 || x_dtype > PE_BF16 || out_dtype < PE_F32 || out_dtype > PE_BF16) return PE_ERR_ARG;
  if (in_f_padded % kBlock || in_f > in_f_padded || in_f_padded - in_f >= kBlock) return PE_ERR_SHAPE;
  if (ld_x < in_f || ld_out < in_f_padded) return PE_ERR_ARG;
  const int nb = in_f_padded / kBlock;
  const int64_t warps = (int64_t)batch * nb;
  const int64_t blocks = (warps + 7) / 8;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  fwht128_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, x_dtype, ld_x, x_tf, out_dtype,
                                                                                 ld_out, batch, in_f, nb);
  PE_CUDA_TRY(cudaGetLastError());
  return PE_OK;
}

extern "C" int pe_pack_nibble(const int8_t* codes, uint8_t* packed, int64_t out_f, int64_t in_f_padded, void* stream) {
  if (!codes || !packed || out_f < 1 || in_f_padded < 1) return PE_ERR_ARG;
  if (in_f_padded % kBlock) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(codes) & 15) || (reinterpret_cast<uintptr_t>(packed) & 15)) return PE_ERR_ALIGN;
  const int64_t n_chunks = out_f * (in_f_padded / 32);
  const int64_t blocks = (n_chunks + 255) / 256;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  pack_nibble_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(codes, packed, n_chunks);
  PE_CUDA_TRY(cudaGetLastError());
  return PE_OK;
}

extern "C" int pe_quantize(const void* weight, int w_dtype, int64_t ld_w, int64_t out_f, int in_f, int in_f_padded,
                           const float* levels, int n_levels, int8_t* codes, int64_t ld_codes, void* norms, int64_t ld_norms,
                           void* stream) {
  if (!weight || !levels || !codes || !norms || out_f < 1 || in_f < 1 || in_f > in_f_padded) return PE_ERR_ARG;
  if (w_dtype < PE_F32 || w_dtype > PE_BF16 || n_levels < 2 || n_levels > 256) return PE_ERR_ARG;
  if (in_f_padded % kBlock) return PE_ERR_SHAPE;
  if (ld_w < in_f || ld_codes < in_f_padded || ld_norms < in_f_padded / kBlock) return PE_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(codes) & 3) || (ld_codes & 3)) return PE_ERR_ALIGN;
  const int nb = in_f_padded / kBlock;
  const int64_t ctas = ((int64_t)out_f * nb + 63) / 64;  // a CTA takes 64 blocks per trip
  const int sms = sm_count();
  if (sms <= 0) return PE_ERR_CUDA;
  // the resident CTAs (two per SM, three for 16-bit weights of up to 16 levels); the level table is built once per CTA
  const bool wide = n_levels > 16;
  const long long per = w_dtype == PE_F32 || wide ? 2 : 3;
  const unsigned grid = (unsigned)(ctas < per * sms ? ctas : per * sms);
  // 4096 x 12288 bf16 with two / three CTAs an SM: to 4 bits 59 / 55 us, to 6 bits 58 / 60 us
#define PE_QUANTIZE16(W) (!wide ? quantize16_kernel<W, 3, true> : n_levels <= 64 ? quantize16_kernel<W, 2, true> : quantize16_kernel<W, 2, false>)
  auto kfn = w_dtype == PE_F32 ? quantize_kernel : w_dtype == PE_F16 ? PE_QUANTIZE16(PE_F16) : PE_QUANTIZE16(PE_BF16);
#undef PE_QUANTIZE16
  const int unit = w_dtype == PE_F32 ? 8 : 16, vec_out = reinterpret_cast<uintptr_t>(codes) % unit == 0 && ld_codes % unit == 0;
  kfn<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(weight, ld_w, out_f, in_f, nb, levels, n_levels, codes, ld_codes,
                                                           static_cast<__half*>(norms), ld_norms, vec_out);
  PE_CUDA_TRY(cudaGetLastError());
  return PE_OK;
}
