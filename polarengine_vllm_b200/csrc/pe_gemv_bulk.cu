// Decode-size quantized matmul (1..16 activation rows): bulk-copy kernel.
//
//   y[m, r] = sum_blk norm[r, blk] * sum_k ct[code[r, blk, k]] * xt[m, blk, k]   (+ bias[r])
//
// One persistent CTA per SM: sixteen math warps (fourteen where a warp takes three blocks), a copy warp, for row-major codes whose
// norms are no single copy a norm warp, and in launches whose CTAs have several passes one or two sum warps.  A stage of the shared-
// memory ring is one 16-row tile of the weight matrix by up to 32 quantization blocks.  The copy warp fills stages with bulk
// copies (of the row-major layout one or a few rows each, of the tiled layout of pe_retile, whose records are contiguous, one
// per stage).  Norms of row-major layers are a strided gather of halves: the norm warp loads them, two stages under way (with
// four its registers spill and 128 experts take 382 instead of 351 us), and stores them beside the codes.  Both warps start
// while the activations are prepared: the dependency wait of the programmatic launch is the math warps' alone
// (gemv_frags_kernel lets this kernel start once what it reads is there).  (Without a copy warp -- the last warp to finish with
// a stage refills it, 128 instead of 96 registers -- the refills came later and every warp had to track them: 4 us over four
// launches.  Norms loaded by the math warps at the head of every pass: 8 us.  There is one norm warp, not several taking stages
// in turn: a wait on a barrier's parity holds only for a waiter that took every earlier phase itself.)
//
// What bounds it: once the ring runs, the shared-memory port.  A warp takes blocks w and w + 16 of every stage or, where rows are
// short, blocks w, w + n and w + 2 n of every stage that falls to its group of n warps:
//  * centroid lookup: the table is replicated per lane at a spacing of 256 bytes per entry, so that ONE byte permute
//    forms the address (code byte in bits 8..15, lane * 4 below) and the load adds the table's constant address;
//    32 lanes with 32 different codes never meet on a bank.  A nibble layer indexes it with the whole byte and gets
//    the fp16 pair of both nibbles; a byte layer keeps (c, 0) and (0, c) in the two halves of an entry, and with up
//    to eight activation rows multiplies both without merging them (the tensor pipe has room, the integer pipe not);
//  * products on the tensor cores (mma.sync m16n8k16, weights as the 16-row A operand, activation rows as the eight
//    columns of B): 16 rows x 16 weights per instruction straight from the lookups' registers, which no descriptor-
//    based tensor-core operation offers (tcgen05 would need the decoded tile written to shared memory and read again);
//  * what a warp does for a tile besides its blocks (barriers, norms, handing its sums over) is about 100 instructions, as
//    many as one nibble block: 128 experts of 21 and 15 blocks, 64 tokens, took 177 us with no block multiplied and nothing
//    copied, 345 us in all.  So where rows are short (kGroupBlocks) a warp takes three blocks, fewer warps share a tile, and
//    the warps left form further groups that work on other tiles: 310 -> 262 us, one token 39.1 -> 37.0, 24576 x 1024 Q6 at
//    8 rows 11.1 -> 9.9.  (Whole rows per warp, activations read from shared memory for every block: 443 us.  22 warps of one
//    block: 341.  Q3 look-ups by byte permutes of register tables instead of loads: 352 to 362.)
//  * the sums of a pass: with all warps meeting at a barrier, adding and meeting again, 64 tokens of 128 experts took 345 us;
//    given to warps of their own, with two sets of partial sums so that the next pass runs meanwhile, 310 (four rows a lane and
//    one 16-byte load per warp's share; with a row a lane two sum warps did not keep up: 326).  24576 x 4096 at 8 rows
//    16.4 -> 15.8 us, 16 rows 25.2 -> 24.2.  The last pass of a CTA is added by all its warps.
//  * activations: a small launch in front (gemv_frags_kernel) pads, rotates and rounds them once and leaves them in
//    B-operand order in the workspace, so that a warp loads its own blocks with four coalesced reads each and keeps
//    them in registers.  Rotating inside this kernel was measured too (in registers, 16-point part by MMAs): its
//    straight-line code cost more in instruction fetches than the extra launch, 13 us over a layer's four launches.
//    The registers left over let the small launch's blocks be resident, waiting, while the launch before it still runs.
// Measured, row-major layout, a line of launches under a CUDA graph, weights from HBM (in brackets the tiled layout):
//   activation rows      1              8              16
//   6144 x 4096 Q5     9.2 (10.4)     9.2 (10.1)    11.2 (12.6) us
//   4096 x 4096 Q6     7.0  (7.5)     7.2  (8.0)     8.6  (9.4)
//   24576 x 4096 Q3   14.2 (15.1)    15.8 (15.5)    24.5 (23.2)
//   4096 x 12288 Q4    9.9 (10.6)    11.1 (11.7)    15.9 (15.9)
//   the four in turn  40.1 (42.9)    44.0 (46.3)    60.3 (61.6)
// Inside the ring's steady state the 24576 x 4096 launch moves 4.9 TB/s; the rest is the launch's own latency: about
// 3.5 us from the launch before it to the first product, 0.5 us from the last one to the stores.  Outside a line (launched
// eagerly, or with other kernels in between) the ring fills about 2 us later: the four in turn take 48.5 us for one row, 51.2 for 8.
//
// The tiles of all problems of a launch form one line that is cut into equal contiguous ranges, one per CTA; nothing
// crosses CTAs.  The partial sums that a tile's warps (all sixteen, or a group's) have of it go through shared memory and are added in
// warp order: bit-identical from run to run, and the same bits from either layout.
#include "pe_gemv_decode.cuh"
#include "pe_status.cuh"

namespace pe {

// Math warps.  Three blocks a warp (BPW) need the registers of a CTA of sixteen warps in all.
__host__ __device__ constexpr int bulk_warps(int bpw) { return bpw == 3 ? 14 : 16; }
__host__ __device__ constexpr int sum_warps(int bpw, bool passes) { return !passes ? 0 : bpw == 3 ? 1 : 2; }
// ... + the copy warp, the sum warps of launches of several passes, the norm warp: of row-major layers, with BPW 3 only where norms
// are no single copy, in an instance of its own (a seventeenth warp leaves 96 registers a thread, and 48 to 120 bytes spill)
__host__ __device__ constexpr int bulk_threads(int bpw, bool norm_warp, bool passes) {
  return (bulk_warps(bpw) + 1 + sum_warps(bpw, passes) + norm_warp) * 32;
}
constexpr int kGroupBlocks = 21;                      // blocks of a row, at most, where a warp takes three: two groups of seven warps (22 would take eight warps: one group)
constexpr int kTabAddr = 2048;                        // address of the centroid table in the shared window
constexpr int kTabReach = 255 * 256 + 256;            // bytes a lookup can reach from there, whatever the code byte is
constexpr int kBulkMaxStages = 8;
constexpr int kNormAhead = 1 << 18;                   // bytes of norms asked for ahead at most
constexpr unsigned kBulkSmemMax = 231424u;            // 227 KB minus the runtime's 1 KB

struct BulkArgs {
  const uint8_t* codes; int64_t ld_codes;  // row-major layout: bytes between rows
  const __half* norms; int64_t ld_norms;
  const uint8_t* tiles;                    // tiled layout
  const float* ct; int n_levels;
  const uint4* frags;                      // activations in B-operand order
  void* y; int y_dtype, y_vec; int64_t ld_y;  // y_vec: four rows from a multiple of 16 on are one store
  const __half* bias;
  int batch, N, nb;
  int n_chunk, chunk_blocks, n_stage;      // chunks of the K range, blocks of a full chunk
  int units;                               // 16-row tiles per problem
  int pass_rows;                           // rows whose partial sums shared memory holds (a multiple of 16)
  int part_stride;                         // floats between activation rows of the partial sums
  int part_rows;                           // activation rows the partial sums have room for
  int groups, group_warps;                 // three blocks a warp: groups of warps, warps of one
  int part_bufs, part_floats;              // sets of partial sums, floats of one
  int part_off, stage_off, stage_bytes;
  int row_stride, copy_rows;               // row-major layout: bytes between rows of a stage, weight rows per bulk copy
  int norm_stride;                         // row-major: bytes between the norms of two rows where a stage's come as one bulk copy, else 0
  int* status;
  // grouped launch: problem i multiplies rows grp[i].y .. + grp[i].z of the row list with matrix grp[i].x
  const int4* grp; int n_problems;
  int64_t codes_stride, norms_stride, tiles_stride;
};

// ---- barriers and bulk copies ---------------------------------------------------------------------------------
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded: after about half a second the status word is set and the wait gives up (the output is then undefined).
__device__ __noinline__ bool bar_wait_slow(uint32_t bar, uint32_t parity, int* status) {
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (bar_try(bar, parity)) return true;
    if (clock64() - t0 > (1ll << 30)) {
      record_timeout(status, PE_STATUS_SPLITK_TIMEOUT);
      return false;
    }
  }
}
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, int* status) {
  if (!bar_try(bar, parity)) bar_wait_slow(bar, parity, status);
}
// one lane of a converged warp: a bulk copy takes warp-uniform operands and issues fastest from a branch on this
__device__ __forceinline__ bool elect_lane() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <int WARPS>
__device__ __forceinline__ void math_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory"); }

// ---- tensor-core products -------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// centroid of byte E of a code word; OFF 128: the upper half of the entry
template <int E, int OFF>
__device__ __forceinline__ uint32_t centroid(uint32_t w, uint32_t lane4) {
  uint32_t a, v;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(lane4), "n"(0x7604 | (E << 4)));
  asm volatile("ld.shared.b32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kTabAddr + OFF));
  return v;
}

// One block: 16 weight rows x 128 weights x 8 NT activation rows.  pa, pb: this lane's bytes of rows g and g + 8.
// The k order of the products is the order of the code bytes: nibble byte i of the block (lane t holds 16 t .. 16 t + 15)
// is the pair (i, i + 64), byte codes are pairs of neighbours.
template <bool PACKED, int NT>
__device__ __forceinline__ void block_product(uint32_t pa, uint32_t pb, const uint32_t (&x)[NT][16], uint32_t lane4, float (&d)[NT][4]) {
  if (PACKED) {
    const uint4 qa = lds128(pa), qb = lds128(pb);
    const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t a0 = centroid<0, 0>(wa[i], lane4), b0 = centroid<0, 0>(wb[i], lane4), a1 = centroid<1, 0>(wa[i], lane4), b1 = centroid<1, 0>(wb[i], lane4);
      const uint32_t a2 = centroid<2, 0>(wa[i], lane4), b2 = centroid<2, 0>(wb[i], lane4), a3 = centroid<3, 0>(wa[i], lane4), b3 = centroid<3, 0>(wb[i], lane4);
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        if (i == 0) mma_f16_first(d[n], a0, b0, a1, b1, x[n][0], x[n][1]);
        else mma_f16(d[n], a0, b0, a1, b1, x[n][4 * i], x[n][4 * i + 1]);
        mma_f16(d[n], a2, b2, a3, b3, x[n][4 * i + 2], x[n][4 * i + 3]);
      }
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // halves of 64 weights
      const uint4 qa = lds128(pa + 64 * h), qb = lds128(pb + 64 * h);
      const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = 8 * h + 2 * i;
        const uint32_t a0 = centroid<0, 0>(wa[i], lane4), b0 = centroid<0, 0>(wb[i], lane4), a1 = centroid<2, 0>(wa[i], lane4), b1 = centroid<2, 0>(wb[i], lane4);
        const uint32_t a2 = centroid<1, 128>(wa[i], lane4), b2 = centroid<1, 128>(wb[i], lane4), a3 = centroid<3, 128>(wa[i], lane4), b3 = centroid<3, 128>(wb[i], lane4);
        if (NT == 1) {  // (c0, 0), (c2, 0) and (0, c1), (0, c3) against the same activations
          if (k == 0) mma_f16_first(d[0], a0, b0, a1, b1, x[0][k], x[0][k + 1]);
          else mma_f16(d[0], a0, b0, a1, b1, x[0][k], x[0][k + 1]);
          mma_f16(d[0], a2, b2, a3, b3, x[0][k], x[0][k + 1]);
        } else {
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            if (k == 0) mma_f16_first(d[n], a0 | a2, b0 | b2, a1 | a3, b1 | b3, x[n][k], x[n][k + 1]);
            else mma_f16(d[n], a0 | a2, b0 | b2, a1 | a3, b1 | b3, x[n][k], x[n][k + 1]);
          }
        }
      }
    }
  }
}

// ---- activations in B-operand order ------------------------------------------------------------------------------
// Fragments of one block and eight activation rows: four 16-byte pieces per lane, piece q of lane (g, t) holding the
// operands of MMAs 2 q and 2 q + 1 for activation row g: [problem][set of eight][block][q][lane].  One warp pads,
// rotates and stores one (row, block).
struct FragArgs {
  const void* x; int x_kind, x_dtype; int64_t ld_x; int in_f, nb, batch, sets;  // sets of eight rows per problem
  uint4* out;
  const int4* grp; const int32_t* x_rows;
  int in_line;
  // one row, fp16: the residual add and the norm in front of the projection (PE_PRO_ADD_RMSNORM)
  const void* delta; int delta_dtype; const __half* norm_w; __half* resid_out; float eps;
};
constexpr int kFragThreads = 128;

// Four consecutive fp16 / fp32 values as loaded, and their fp32 form; columns past in_f (a multiple of 4) are zero.
__device__ __forceinline__ Raw4 raw4(const void* base, int dtype, int col, int in_f) {
  Raw4 r = {{0u, 0u, 0u, 0u}};
  if (base && col < in_f) r = load4_raw(base, dtype, 0, col, in_f, true);
  return r;
}
// updated residual half(x + half(delta)) from the raw values
__device__ __forceinline__ void residual4(const FragArgs& p, const Raw4& x, const Raw4& d, float r[4]) {
  cvt4(x, PE_F16, r);
  if (p.delta) {
    float f[4];
    cvt4(d, p.delta_dtype, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = __half2float(__float2half_rn(r[i] + __half2float(__float2half_rn(f[i]))));
  }
}

template <bool PACKED, bool NORM>
__global__ void __launch_bounds__(kFragThreads) gemv_frags_kernel(const FragArgs p) {
  // The wait first: the matmul behind reads codes, norms and table before its own wait, which covers this launch only, so
  // what older kernels wrote (a layer just loaded, arrays rewritten in place) has to be visible before it may start.  In a
  // line of captured launches it was when the line began (line_holds), and the ring of the matmul fills while the launch in
  // front still runs: four launches for one row 48.5 us without, 40.2 us with.
  if (p.in_line) asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!p.in_line) asm volatile("griddepcontrol.launch_dependents;");
  const int lane = threadIdx.x & 31, job = blockIdx.x * (kFragThreads / 32) + (threadIdx.x >> 5);
  const int m = job / p.nb, b = job - m * p.nb, prob = blockIdx.y;
  if (!NORM && m >= p.batch) return;
  int64_t row = m;
  if (p.grp) {
    const int4 d = p.grp[prob];
    if (m >= d.z) return;
    row = p.x_rows ? p.x_rows[d.y + m] : d.y + m;
  }
  const bool vec_ok = (p.ld_x % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.x) & 15) == 0);
  float v[4];
  if (NORM) {  // PE_PRO_ADD_RMSNORM, one row
    // every block of threads sums the row's squares for itself (8 KB from L2, all loads of 4096 columns in flight
    // together); a warp stores the residual of its own 128 columns
    __shared__ float sums[kFragThreads / 32];
    const int col = b * kBlock + lane * 4;
    const Raw4 own_x = raw4(m == 0 ? p.x : nullptr, PE_F16, col, p.in_f), own_d = raw4(m == 0 ? p.delta : nullptr, p.delta_dtype, col, p.in_f),
               own_w = raw4(m == 0 ? p.norm_w : nullptr, PE_F16, col, p.in_f);
    constexpr int U = 8;
    float ss = 0.f;
    for (int c0 = threadIdx.x * 4; c0 < p.in_f; c0 += kFragThreads * 4 * U) {
      Raw4 x[U], d[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        x[u] = raw4(p.x, PE_F16, c0 + u * kFragThreads * 4, p.in_f);
        d[u] = raw4(p.delta, p.delta_dtype, c0 + u * kFragThreads * 4, p.in_f);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float r[4];
        residual4(p, x[u], d[u], r);
        ss += r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3];
      }
    }
#pragma unroll
    for (int i = 16; i >= 1; i >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, i);
    if (lane == 0) sums[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (m > 0) return;
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < kFragThreads / 32; ++i) ss += sums[i];
    const float scale = rsqrtf(ss / (float)p.in_f + p.eps);
    residual4(p, own_x, own_d, v);
    if (p.resid_out && col < p.in_f) *reinterpret_cast<uint2*>(p.resid_out + col) = make_uint2(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]));
    float wn[4];
    cvt4(own_w, PE_F16, wn);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __half2float(__hmul(__float2half_rn(v[i] * scale), __float2half_rn(wn[i])));
  } else {
    load4_as_float(p.x, p.x_dtype, row * p.ld_x, b * kBlock + lane * 4, p.x_kind == PE_X_ROTATED ? p.nb * kBlock : p.in_f, vec_ok, v);
  }
  if (p.x_kind == PE_X_SILU_MUL) {  // the row is [gate | up]: half(silu(gate)) * up, the rounding steps of pe_silu_mul
    float u[4];
    load4_as_float(p.x, p.x_dtype, row * p.ld_x + p.in_f, b * kBlock + lane * 4, p.in_f, vec_ok && p.in_f % 4 == 0, u);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __half2float(__hmul(__float2half_rn(v[i] / (1.f + expf(-v[i]))), __float2half_rn(u[i])));
  }
  if (p.x_kind != PE_X_ROTATED) warp_fwht128(v, lane);
  uint4* dst = p.out + ((size_t)(prob * p.sets + (m >> 3)) * p.nb + b) * 128;
  const int g = m & 7;
  if (PACKED) {  // nibble byte i of the block is the pair (i, i + 64); lane t of a row holds bytes 16 t .. 16 t + 15
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = __shfl_xor_sync(0xffffffffu, v[i], 16);
    if (lane < 16)
      dst[(lane & 3) * 32 + g * 4 + (lane >> 2)] = make_uint4(pack_half2(v[0], o[0]), pack_half2(v[1], o[1]), pack_half2(v[2], o[2]), pack_half2(v[3], o[3]));
  } else {       // neighbours; lane t holds codes 16 t .. 16 t + 15 of each half
    const int k = (lane < 16 ? 0 : 4) + (lane & 3);
    reinterpret_cast<uint2*>(dst + (k >> 1) * 32 + g * 4 + ((lane & 15) >> 2))[k & 1] = make_uint2(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]));
  }
}

// ---- the launch's line of units ---------------------------------------------------------------------------------
// A pass is a run of 16-row tiles of one problem whose partial sums fit in shared memory.  The copy, norm and math warps
// walk the same passes.
template <bool GROUPED>
struct Pass {
  int left;               // units of this CTA not yet passed
  int prob, off;          // problem, unit inside it
  int row0, rows;         // weight rows of this pass
  __device__ __forceinline__ void start(const BulkArgs& p, int beg, int n) {
    left = n;
    prob = GROUPED ? beg / p.units : 0;
    off = GROUPED ? beg - prob * p.units : beg;
  }
  __device__ __forceinline__ bool next(const BulkArgs& p) {  // false at the end; advances past the pass it describes
    if (left <= 0) return false;
    int n = min(p.pass_rows / 16, left);
    if (GROUPED) {
      if (off == p.units) { off = 0; ++prob; }
      n = min(n, p.units - off);
    }
    row0 = off * 16;
    rows = min(n * 16, p.N - row0);
    left -= n; off += n;
    return true;
  }
};

template <bool PACKED, int NT, int BPW, bool TILED, bool GROUPED, bool PASSES, bool NORM_WARP>
__global__ void __launch_bounds__(bulk_threads(BPW, NORM_WARP, PASSES), 1) gemv_bulk_kernel(const BulkArgs p) {
  extern __shared__ __align__(128) uint8_t smem[];  // no static shared memory: the window starts with it
  constexpr int kWarps = bulk_warps(BPW), kSumWarps = sum_warps(BPW, PASSES), kThreads = bulk_threads(BPW, NORM_WARP, PASSES);
  constexpr int kRowBytes = PACKED ? 64 : 128;           // codes of one row's block
  constexpr int kGroupWarps = kGroupBlocks / 3;
  constexpr int kRecBytes = kRowBytes * 16 + 32;         // tiled record: 16 rows of a block, then their norms
  const bool norms_copied = !TILED && (BPW == 3 ? !NORM_WARP : GROUPED) && p.norm_stride;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t full = sbase, empty = sbase + 8 * kBulkMaxStages;
  int& n_live = *reinterpret_cast<int*>(smem + 16 * kBulkMaxStages);
  const uint32_t part_full = sbase + 16 * kBulkMaxStages + 16, part_empty = part_full + 16;
  asm volatile("griddepcontrol.launch_dependents;");
  if (sbase > kTabAddr - 256) {  // the table's place is taken: never seen, the host sizes for any base below
    if (tid == 0) record_timeout(p.status, PE_STATUS_SPLITK_TIMEOUT);
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < p.n_stage; ++s) { bar_init(full + 8 * s, TILED || norms_copied ? 1 : 2); bar_init(empty + 8 * s, BPW == 3 ? p.group_warps : kWarps); }
    if (PASSES)
      for (int b = 0; b < 2; ++b) { bar_init(part_full + 8 * b, kWarps); bar_init(part_empty + 8 * b, kSumWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    n_live = 0;
  }
  __syncthreads();
  int line = p.units;
  if (GROUPED) {  // the problem list comes from the launch before this one
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = tid; i < p.n_problems; i += kThreads)
      if (p.grp[i].z > 0) atomicMax(&n_live, i + 1);
    __syncthreads();
    line = n_live * p.units;
  }
  Pass<GROUPED> ps;
  {
    const int q = line / (int)gridDim.x, r = line - q * (int)gridDim.x, cta = blockIdx.x;
    const int beg = cta * q + min(cta, r);
    ps.start(p, beg, q + (cta < r));
  }

  if (w == kWarps) {  // ---- copy warp
    const bool one = elect_lane();
    int s = 0;
    uint32_t ph = 1;
    while (ps.next(p)) {
      const uint8_t* codes = p.codes;
      const uint8_t* tiles = p.tiles;
      const __half* norms = p.norms;
      if (GROUPED) {
        const int4 d = p.grp[ps.prob];
        if (d.z <= 0) continue;
        codes += d.x * p.codes_stride;
        tiles += d.x * p.tiles_stride;
        norms += d.x * p.norms_stride;
      }
      for (int c = 0; c < p.n_chunk; ++c) {
        const int b0 = c * p.chunk_blocks, nblk = min(p.chunk_blocks, p.nb - b0);
        for (int r0 = 0; r0 < ps.rows; r0 += 16) {
          bar_wait(empty + 8 * s, ph, p.status);
          const uint32_t dst = sbase + p.stage_off + s * p.stage_bytes, bar = full + 8 * s;
          if (one) {
            if (TILED) {
              bar_expect(bar, nblk * kRecBytes);
              bulk_load(dst, tiles + ((int64_t)((ps.row0 + r0) >> 4) * p.nb + b0) * kRecBytes, nblk * kRecBytes, bar);
            } else {
              const int rows = min(16, ps.rows - r0);
              const uint8_t* src = codes + (int64_t)(ps.row0 + r0) * p.ld_codes + b0 * kRowBytes;
              bar_expect(bar, rows * (nblk * kRowBytes + (norms_copied ? p.norm_stride : 0)));
              if (norms_copied) bulk_load(dst + 16 * p.row_stride + 64, norms + (int64_t)(ps.row0 + r0) * p.nb, rows * p.norm_stride, bar);
              for (int r = 0; r < rows; r += p.copy_rows)
                bulk_load(dst + r * p.row_stride + (r >> 3) * 64, src + r * p.ld_codes, min(p.copy_rows, rows - r) * nblk * kRowBytes, bar);
            }
          }
          __syncwarp();
          if (++s == p.n_stage) { s = 0; ph ^= 1; }
        }
      }
    }
    return;
  }

  // The sums of a pass by warp `who` of `whos`: a lane adds the warps' shares of four rows of an activation row, in warp order.
  constexpr int kSlots = BPW == 3 ? kGroupWarps : kWarps;
  float* part = reinterpret_cast<float*>(smem + p.part_off);
  auto sum_pass = [&](const float* from, int batch, int y_row, int who, int whos) {
    const int quads = (ps.rows + 3) >> 2, slot = p.part_rows * p.part_stride;
    for (int e = who * 32 + lane; e < batch * quads; e += whos * 32) {
      const int m = e / quads, r = (e - m * quads) * 4;
      const float* q = from + m * p.part_stride + r;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < kSlots; ++i)
        if (BPW < 3 || i < p.group_warps) {
          const float4 v = *reinterpret_cast<const float4*>(q + i * slot);
          sum[0] += v.x; sum[1] += v.y; sum[2] += v.z; sum[3] += v.w;
        }
      const int row = ps.row0 + r, left = ps.rows - r;
      if (p.bias)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < left) sum[k] += __half2float(p.bias[row + k]);
      const int64_t at = (int64_t)(y_row + m) * p.ld_y + row;
      if (p.y_vec && left >= 4) {
        if (p.y_dtype == PE_F32) *reinterpret_cast<float4*>(static_cast<float*>(p.y) + at) = make_float4(sum[0], sum[1], sum[2], sum[3]);
        else if (p.y_dtype == PE_F16) *reinterpret_cast<uint2*>(static_cast<__half*>(p.y) + at) = make_uint2(pack_half2(sum[0], sum[1]), pack_half2(sum[2], sum[3]));
        else
          for (int k = 0; k < 4; ++k) store_from_float(p.y, PE_BF16, at + k, sum[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < left) store_from_float(p.y, p.y_dtype, at + k, sum[k]);
      }
    }
  };

  if (PASSES && w > kWarps && w <= kWarps + kSumWarps) {  // ---- sum warps: every pass but the CTA's last
    if (!GROUPED) asm volatile("griddepcontrol.wait;" ::: "memory");
    int b = 0, prob = -1, batch = p.batch, y_row = 0;
    uint32_t ph = 0;
    while (ps.next(p) && ps.left > 0) {
      if (GROUPED && ps.prob != prob) {
        const int4 d = p.grp[ps.prob];
        prob = ps.prob;
        batch = d.z < 8 * NT ? d.z : 8 * NT;
        y_row = d.y;
      }
      if (GROUPED && batch <= 0) continue;
      bar_wait(part_full + 8 * b, ph, p.status);
      sum_pass(part + b * p.part_floats, batch, y_row, w - kWarps - 1, kSumWarps);
      __syncwarp();
      if (lane == 0) bar_arrive(part_empty + 8 * b);
      if (++b == p.part_bufs) { b = 0; ph ^= 1; }
    }
    return;
  }

  if (NORM_WARP && w > kWarps && norms_copied) return;
  if (NORM_WARP && w > kWarps) {  // ---- norm warp: a stage's norms, the 16 rows of a block side by side
    constexpr int kPlaces = BPW == 1 ? 16 : 32, kLaneRows = 16 * kPlaces / 32;
    const int b = lane % kPlaces, r_lane = lane / kPlaces * kLaneRows, blocks = min(p.nb, p.chunk_blocks);
    const __half* norms = p.norms;
    int c = 0, r0 = 0;
    auto next_pass = [&]() {
      while (ps.next(p)) {
        if (GROUPED) {
          const int4 d = p.grp[ps.prob];
          if (d.z <= 0) continue;
          norms = p.norms + d.x * p.norms_stride;
        }
        // the whole pass on its way to L2 (of arrays with wide gaps between rows, its first part): a stage's loads then wait for
        // L2 and not for HBM
        const char* span = reinterpret_cast<const char*>(norms + (int64_t)ps.row0 * p.ld_norms);
        const int bytes = (int)min(((int64_t)(ps.rows - 1) * p.ld_norms + p.nb) * 2, (int64_t)kNormAhead);
        for (int o = lane * 128; o < bytes; o += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(span + o));
        return true;
      }
      return false;
    };
    auto next_stage = [&]() {
      r0 += 16;
      if (r0 < ps.rows) return true;
      r0 = 0;
      if (++c < p.n_chunk) return true;
      c = 0;
      return next_pass();
    };
    auto load = [&](unsigned short (&h)[kLaneRows]) {
      const int blk = c * p.chunk_blocks + b;
      const __half* src = norms + (int64_t)(ps.row0 + r0 + r_lane) * p.ld_norms + blk;
#pragma unroll
      for (int i = 0; i < kLaneRows; ++i) {
        h[i] = 0;
        if (b < blocks && blk < p.nb && r0 + r_lane + i < ps.rows) h[i] = __half_as_ushort(src[(int64_t)i * p.ld_norms]);
      }
    };
    int s = 0;
    uint32_t ph = 1;
    auto store = [&](const unsigned short (&h)[kLaneRows]) {
      bar_wait(empty + 8 * s, ph, p.status);
      if (b < blocks) {
        const uint32_t dst = sbase + p.stage_off + s * p.stage_bytes + 16 * p.row_stride + 64 + b * 32 + r_lane * 2;
#pragma unroll
        for (int q = 0; q < kLaneRows; q += 8)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + q * 2), "r"(h[q] | h[q + 1] << 16), "r"(h[q + 2] | h[q + 3] << 16),
                       "r"(h[q + 4] | h[q + 5] << 16), "r"(h[q + 6] | h[q + 7] << 16) : "memory");
      }
      __syncwarp();
      if (lane == 0) bar_arrive(full + 8 * s);
      if (++s == p.n_stage) { s = 0; ph ^= 1; }
    };
    unsigned short h0[kLaneRows], h1[kLaneRows];  // the loads of two stages under way
    bool more = next_pass();
    if (more) load(h0);
    while (more) {
      const bool second = next_stage();
      if (second) load(h1);
      store(h0);
      if (!second) break;
      more = next_stage();
      if (more) load(h0);
      store(h1);
    }
    return;
  }

  // ---- math warps: the table first (it needs nothing from the launch before this one)
  {
    uint8_t* tab = smem + (kTabAddr - sbase);
    const int entries = PACKED ? (p.n_levels <= 8 ? 128 : 256) : p.n_levels;
#pragma unroll 2
    for (int e = tid >> 3; e < entries; e += kWarps * 4) {
      uint32_t u;
      if (PACKED) {
        const int a = e & 15, b = e >> 4;
        u = pack_half2(a < p.n_levels ? __ldg(p.ct + a) : 0.f, b < p.n_levels ? __ldg(p.ct + b) : 0.f);
      } else {
        u = __half_as_ushort(__float2half_rn(__ldg(p.ct + e)));
      }
      *reinterpret_cast<uint4*>(tab + e * 256 + (tid & 7) * 16) = make_uint4(u, u, u, u);
      if (!PACKED) *reinterpret_cast<uint4*>(tab + e * 256 + 128 + (tid & 7) * 16) = make_uint4(u << 16, u << 16, u << 16, u << 16);
    }
  }
  bool more = ps.next(p);
  if (!GROUPED) asm volatile("griddepcontrol.wait;" ::: "memory");

  // Where this lane's codes and norms lie in a stage.  Its operand rows g and g + 8 are weight rows g and g + 8 of a tile's
  // records, and rows row_a and row_a + 4 of row-major stages: rows of those lie a multiple of 64 bytes apart, rows 0..7 and
  // 8..15 another 64 bytes, so that a quarter warp, which reads the rows of two neighbouring g, reads both halves of the banks.
  // Three blocks a warp: the warps form groups of group_warps, group q takes the tiles in stages q, q + groups, ...
  const int gw = BPW == 3 ? p.group_warps : kWarps, group = BPW == 3 ? w / gw : 0, wi = BPW == 3 ? w - group * gw : w;
  constexpr int kRowB = TILED ? 8 : 4;
  constexpr bool kPlain = PASSES || GROUPED;  // partial sums in the order of the rows
  constexpr int kPartB = kPlain ? kRowB : 8;
  const int row_a = TILED ? g : (g >> 1) + (g & 1) * 8;
  const uint32_t at_a = TILED ? wi * kRecBytes + g * kRowBytes + t * 16 : row_a * p.row_stride + (g & 1) * 64 + wi * kRowBytes + t * 16;
  const uint32_t at_b = at_a + kRowB * (TILED ? kRowBytes : p.row_stride);
  const uint32_t at_n = TILED ? wi * kRecBytes + 16 * kRowBytes + g * 2 : 16 * p.row_stride + 64 + (norms_copied ? wi * 2 + row_a * p.norm_stride : wi * 32 + row_a * 2);
  const int kStep = gw * (TILED ? kRecBytes : kRowBytes);
  const int norm_step = gw * (TILED ? kRecBytes : norms_copied ? 2 : 32), norm_b = kRowB * (norms_copied ? p.norm_stride : 2);
  const uint32_t lane4 = lane * 4;
  uint32_t x[BPW][NT][16];
  int x_prob = -1, group_rows = p.batch;
  int y_row = 0;

  auto load_x = [&](int prob, int c) {
    const uint4* src = p.frags + (size_t)(prob * NT * p.nb + c * p.chunk_blocks + wi) * 128 + lane;
    const int nblk = p.nb - c * p.chunk_blocks;
#pragma unroll
    for (int j = 0; j < BPW; ++j)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (wi + gw * j < nblk && n * 8 + g < (GROUPED ? group_rows : p.batch)) v = __ldcg(src + (n * p.nb + gw * j) * 128 + q * 32);
          x[j][n][4 * q] = v.x; x[j][n][4 * q + 1] = v.y; x[j][n][4 * q + 2] = v.z; x[j][n][4 * q + 3] = v.w;
        }
  };

  int s = 0, b = 0, turn = 0;
  uint32_t ph = 0, part_ph = 1;
  if (PASSES) math_sync<kWarps>();  // the table is there
  for (; more; more = ps.next(p)) {
    if (ps.prob != x_prob) {
      if (GROUPED) {
        const int4 d = p.grp[ps.prob];
        if (d.z <= 0) continue;
        group_rows = d.z < 8 * NT ? d.z : 8 * NT;
        y_row = d.y;
      }
      x_prob = ps.prob;
      if (p.n_chunk == 1) load_x(x_prob, 0);
    }
    if (PASSES) bar_wait(part_empty + 8 * b, part_ph, p.status);
    else math_sync<kWarps>();  // the table is there
    float* const sums = part + b * p.part_floats;
    for (int c = 0; c < p.n_chunk; ++c) {
      if (p.n_chunk > 1) load_x(x_prob, c);
      const int nblk = min(p.chunk_blocks, p.nb - c * p.chunk_blocks);
      for (int r0 = 0; r0 < ps.rows; r0 += 16) {
        if (BPW == 3) {
          const bool mine = turn == group;
          if (++turn == p.groups) turn = 0;
          if (!mine) {
            if (++s == p.n_stage) { s = 0; ph ^= 1; }
            continue;
          }
        }
        const uint32_t st = sbase + p.stage_off + s * p.stage_bytes;
        bar_wait(full + 8 * s, ph, p.status);
        float acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
#pragma unroll
        for (int j = 0; j < BPW; ++j) {
          const int blk = wi + gw * j;
          if (blk < nblk) {
            float d[NT][4];
            unsigned short ha, hb;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(ha) : "r"(st + at_n + j * norm_step));
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hb) : "r"(st + at_n + j * norm_step + norm_b));
            block_product<PACKED, NT>(st + at_a + j * kStep, st + at_b + j * kStep, x[j], lane4, d);
            const float fa = __half2float(__ushort_as_half(ha)), fb = __half2float(__ushort_as_half(hb));
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              acc[n][0] = fmaf(fa, d[n][0], acc[n][0]); acc[n][1] = fmaf(fa, d[n][1], acc[n][1]);
              acc[n][2] = fmaf(fb, d[n][2], acc[n][2]); acc[n][3] = fmaf(fb, d[n][3], acc[n][3]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(empty + 8 * s);
        if (++s == p.n_stage) { s = 0; ph ^= 1; }
        float* pp = sums + wi * p.part_rows * p.part_stride + r0 + (kPlain ? row_a : g);
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int m = n * 8 + 2 * t + e;
            if (m < (GROUPED ? group_rows : p.batch)) {
              float* q = pp + m * p.part_stride;
              if (c == 0) { q[0] = acc[n][e]; q[kPartB] = acc[n][2 + e]; }
              else { q[0] += acc[n][e]; q[kPartB] += acc[n][2 + e]; }
            }
          }
      }
    }
    if (!PASSES && GROUPED) {  // one set of sums: all warps add, and meet again before the next pass
      math_sync<kWarps>();
      sum_pass(sums, group_rows, y_row, w, kWarps);
      continue;
    }
    if (!PASSES) {  // few rows a CTA: a lane each
      math_sync<kWarps>();
      const int sets = (ps.rows + 31) >> 5;
      for (int e = w; e < sets * p.batch; e += kWarps) {
        const int m = sets == 1 ? e : e / sets, at = (e - m * sets) * 32 + lane;
        const int r = TILED ? at : (at & ~15) + ((at & 7) >> 1) + (at & 1) * 8 + ((at >> 1) & 4);  // the row that row_a put there
        if (r < ps.rows) {
          const float* q = sums + m * p.part_stride + at;
          float v[kWarps], sum = 0.f;
#pragma unroll
          for (int i = 0; i < kWarps; ++i) v[i] = q[i * p.part_rows * p.part_stride];
#pragma unroll
          for (int i = 0; i < kWarps; ++i) sum += v[i];
          const int row = ps.row0 + r;
          if (p.bias) sum += __half2float(p.bias[row]);
          store_from_float(p.y, p.y_dtype, (int64_t)m * p.ld_y + row, sum);
        }
      }
      continue;
    }
    if (ps.left == 0) {  // the last pass: nothing left to overlap, and all warps are faster than two
      math_sync<kWarps>();
      sum_pass(sums, GROUPED ? group_rows : p.batch, y_row, w, kWarps);
      break;
    }
    __syncwarp();
    if (lane == 0) bar_arrive(part_full + 8 * b);
    if (++b == p.part_bufs) { b = 0; part_ph ^= 1; }
  }
}

// ---- host side --------------------------------------------------------------------------------------------------
template <bool PACKED, int NT, int BPW, bool TILED, bool GROUPED, bool PASSES, bool NORM_WARP = !TILED && (BPW < 3)>
static int launch_bulk(BulkArgs& a, int sms, cudaStream_t st) {
  constexpr int kRowBytes = PACKED ? 64 : 128, kRecBytes = kRowBytes * 16 + 32;
  constexpr int kWarps = bulk_warps(BPW);
  a.chunk_blocks = kWarps * BPW;
  a.n_chunk = (a.nb + a.chunk_blocks - 1) / a.chunk_blocks;
  const int blocks = a.nb < a.chunk_blocks ? a.nb : a.chunk_blocks;  // of the largest stage
  a.units = (a.N + 15) / 16;
  const long long line = (long long)a.units * (a.grp ? a.n_problems : 1);
  if (line >= (1ll << 31)) return PE_ERR_LIMIT;
  const int G = (int)(line < sms ? line : sms);
  // Rows per pass: the sums of a pass meet at a barrier, and two sets of activation rows read their activations again for
  // every K range of a pass, so few and equal passes; but 64 rows of 8 activation rows are 34 KB of partial sums (of 16: 68 KB),
  // which the ring would rather have.  8 rows: 64 best of 32, 64, 96 and 176; 16 rows, 24576 x 4096: 35.9, 28.5 and 25.1 us for
  // 16, 32 and 64, 6144 x 4096: 14.1, 12.3 and 11.3 us.  Groups of few warps have room for 128 rows: 128 experts, 64 tokens,
  // 267 us against 276 with 64.
  a.part_rows = a.batch < 8 * NT ? a.batch : 8 * NT;
  const int cta_rows = (int)((line + G - 1) / G) * 16;
  const int entries = PACKED ? (a.n_levels <= 8 ? 128 : 256) : a.n_levels;
  // Three blocks a warp (short rows): as few warps a tile as hold it, as many tiles at a time as the warps make groups.
  a.group_warps = BPW == 3 ? (a.nb + 2) / 3 : kWarps;
  a.groups = kWarps / a.group_warps;
  a.part_off = kTabAddr + entries * 256;  // leaves room for the table wherever the window starts
  // Row-major stages: a copy of its own for every row of 2 KB or more; shorter rows that follow each other in memory share one
  // (a copy costs about 60 ns whatever its size: 128 experts of 21 and 15 blocks, rows of 1344 and 960 bytes, took 380 us with a
  // copy a row and 356 us with two or more rows in one; 24576 rows of 2 KB 14.3 us with a copy a row and 15.3 us with two).
  a.row_stride = blocks * kRowBytes;
  a.copy_rows = 1;
  if (a.n_chunk == 1 && a.ld_codes == a.row_stride)
    while (a.copy_rows < 8 && a.copy_rows * a.row_stride < 2048) a.copy_rows *= 2;
  a.stage_bytes = TILED ? (blocks * kRecBytes + 127) & ~127 : (16 * a.row_stride + 64 + blocks * 32 + 127) & ~127;
  // Stages a ring should have before a pass gets more rows: two for every group of warps; three beside two sets of sums
  // (32 experts of 32 blocks Q4, 4 rows: 80 us with two stages, 74 with 32-row passes; 64 of 20 blocks Q6, 8 rows: 162 with a stage a group,
  // 126 with two and 64-row passes).  Where no cap gives that many (32 blocks Q5: 160 us with 32 or 64 rows) the first that gives two.
  const int first_cap = BPW == 3 ? 128 : a.batch <= 2 ? 256 : 64;
  auto ring = [&](int cap) {
    const int passes = (cta_rows + cap - 1) / cap;
    a.pass_rows = GROUPED ? cap : ((cta_rows + passes - 1) / passes + 15) / 16 * 16;
    a.part_stride = a.pass_rows + 4;
    a.part_floats = a.group_warps * a.part_rows * a.part_stride;
    a.part_bufs = PASSES ? 2 : 1;
    a.stage_off = (a.part_off + a.part_bufs * a.part_floats * 4 + 127) & ~127;
    a.n_stage = a.stage_off < (int)kBulkSmemMax ? ((int)kBulkSmemMax - a.stage_off) / a.stage_bytes : 0;
    return a.n_stage;
  };
  int cap = first_cap;
  for (const int want = BPW == 3 ? 2 * a.groups : GROUPED && PASSES ? 3 : 2; cap >= 16 && ring(cap) < want;) cap /= 2;
  if (cap < 16)
    for (cap = first_cap; cap >= 16 && ring(cap) < 2;) cap /= 2;
  if (cap < 16) return PE_ERR_LIMIT;
  if (a.n_stage > kBulkMaxStages) a.n_stage = kBulkMaxStages;
  if (a.groups > a.n_stage) a.groups = a.n_stage;
  // Several passes: sums by warps of their own, where two sets of them leave a ring of three stages (15360 x 2560 Q5 at 16 rows
  // would have two, and takes 20.1 us that way, 18.7 with one set; 24576 x 4096 Q3 has three: 24.2 and 25.2 us; problems of 16
  // rows, 11.5 on average, 64 experts of 16 blocks Q5: 127 and 119 us, 32 of 32 blocks Q4: 142 and 134, 128 of 8 blocks Q3: 70 and 78).
  if (!PASSES && (GROUPED || a.pass_rows < cta_rows) && a.stage_off + a.part_floats * 4 + 3 * a.stage_bytes <= (int)kBulkSmemMax)
    return launch_bulk<PACKED, NT, BPW, TILED, GROUPED, true, NORM_WARP>(a, sms, st);
  a.n_stage -= a.n_stage % a.groups;  // a stage is one group's: a wait on a parity holds for a waiter that took every earlier phase
  unsigned dyn = a.stage_off + a.n_stage * a.stage_bytes;
  if (dyn < (unsigned)(kTabAddr + kTabReach)) dyn = kTabAddr + kTabReach;
  auto kfn = gemv_bulk_kernel<PACKED, NT, BPW, TILED, GROUPED, PASSES, NORM_WARP>;
  static thread_local unsigned configured[16] = {0};
  int dev = 0;
  PE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 16 || configured[dev] < dyn) {
    PE_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    if (dev < 16) configured[dev] = dyn;
  }
  PE_CUDA_TRY(launch_pdl(kfn, dim3(G), dim3(bulk_threads(BPW, NORM_WARP, PASSES)), dyn, st, a));
  return PE_OK;
}

template <bool PACKED, bool TILED, bool GROUPED>
static int launch_bulk_shape(BulkArgs& a, int sms, cudaStream_t st) {
  // Grouped launches, and others of short rows, meet new rows all the time, and the norm warp's sixteen loads a stage are what paces them: where the norms of
  // a tile follow each other and their bytes are whole 16s, they come as one more bulk copy (128 experts, 2688 -> 2 x 1856, 64
  // tokens: 354 and 349 us; one token 41.1 and 39.0).  Their rows then share banks where the block count is even, which the
  // long rows of a dense layer feel more than the loads (24576 x 4096 at 8 rows: 16.4 us by the norm warp, 17.0 copied).
  const bool three = a.batch <= 8 && a.nb <= kGroupBlocks && (GROUPED || ((a.N + 15) / 16 >= 6 * sms && (a.batch > 2 || a.nb > 16)));
  a.norm_stride = !TILED && (GROUPED || three) && a.nb <= 16 * (a.batch > 8 ? 1 : 2) && a.ld_norms == a.nb && (reinterpret_cast<uintptr_t>(a.norms) & 15) == 0 &&
                  a.norms_stride % 8 == 0 && (a.N % 16) * a.nb % 8 == 0 ? a.nb * 2 : 0;
  // Blocks per warp and stage: two when the row is longer than sixteen blocks.  Two sets of activation rows keep one:
  // their operands for two blocks spill (4096 x 12288 at 16 rows: 18.4 us with two, 15.9 with one).
  if (a.batch > 8) return launch_bulk<PACKED, 2, 1, TILED, GROUPED, false>(a, sms, st);
  // Three, and groups of warps, for rows of up to 21 blocks: always in grouped launches; in others where a CTA has six tiles or
  // more, for the groups to have several each (6400 x 2560 Q5 has 2.7: 7.9 us with two blocks a warp, 8.2 with three;
  // 10240 x 2048 Q3 4.3: 6.9 and 7.2; 15360 x 2560 Q3 6.5: 9.9 and 9.4), and for one or two activation rows only where one block a warp is
  // not enough (20480 x 1152 Q4, one row: 7.4 and 7.5; 15360 x 2560 Q3, one row: 9.1 and 8.8).
  // Norms with gaps, or that do not start or end on 16 bytes, are gathered by a norm warp there too (by the copy warp, between
  // its copies: 24576 x 2048 Q4 at 8 rows 17.1 us, 128 experts of 21 blocks at 4 rows 479, 64 of 11 blocks 100; now 12.9, 204 and 52, with
  // one copy 10.4, 147 and 32.5; two blocks a warp took 11.2, 208 and 44).  The order of the sums is the same.
  if (three)
    return TILED || a.norm_stride ? launch_bulk<PACKED, 1, 3, TILED, GROUPED, true>(a, sms, st) : launch_bulk<PACKED, 1, 3, TILED, GROUPED, true, !TILED>(a, sms, st);
  if constexpr (GROUPED) return launch_bulk<PACKED, 1, 2, TILED, GROUPED, true>(a, sms, st);
  else return a.nb > 16 ? launch_bulk<PACKED, 1, 2, TILED, GROUPED, false>(a, sms, st) : launch_bulk<PACKED, 1, 1, TILED, GROUPED, false>(a, sms, st);
}

template <bool PACKED, bool TILED>
static int launch_bulk_kind(BulkArgs& a, int sms, cudaStream_t st) {
  return a.grp ? launch_bulk_shape<PACKED, TILED, true>(a, sms, st) : launch_bulk_shape<PACKED, TILED, false>(a, sms, st);
}

PE_WAIT_STATUS_READER(gemv_wait_status)

size_t gemv_bulk_frag_bytes(int problems, int batch, int in_f_padded) {
  return (size_t)problems * (batch > 8 ? 2 : 1) * (in_f_padded / kBlock) * 2048;
}

int gemv_bulk_run(const GemvBulkCall& q, cudaStream_t st) {
  const int sms = sm_count();
  if (sms <= 0) return PE_ERR_CUDA;
  FragArgs f = {};
  f.x = q.x; f.x_kind = q.x_kind; f.x_dtype = q.x_dtype; f.ld_x = q.ld_x; f.in_f = q.in_f;
  f.nb = q.in_f_padded / kBlock; f.batch = q.batch; f.sets = q.batch > 8 ? 2 : 1;
  f.out = static_cast<uint4*>(q.frags);
  f.grp = static_cast<const int4*>(q.problems); f.x_rows = q.x_rows;
  f.delta = q.delta; f.delta_dtype = q.delta_dtype; f.norm_w = static_cast<const __half*>(q.norm_w);
  f.resid_out = static_cast<__half*>(q.resid_out); f.eps = q.eps;
  f.in_line = line_holds(st);
  const int warps = kFragThreads / 32;
  const dim3 grid((q.batch * f.nb + warps - 1) / warps, q.problems ? q.max_problems : 1);
  auto frags = q.pro == PE_PRO_ADD_RMSNORM ? (q.packed ? gemv_frags_kernel<true, true> : gemv_frags_kernel<false, true>)
                                           : (q.packed ? gemv_frags_kernel<true, false> : gemv_frags_kernel<false, false>);
  PE_CUDA_TRY(launch_pdl(frags, grid, dim3(kFragThreads), 0, st, f));
  BulkArgs a = {};
  a.codes = static_cast<const uint8_t*>(q.codes); a.ld_codes = q.ld_codes;
  a.norms = static_cast<const __half*>(q.norms); a.ld_norms = q.ld_norms;
  a.tiles = static_cast<const uint8_t*>(q.tiles);
  a.ct = q.ct_scaled; a.n_levels = q.n_levels;
  a.frags = f.out;
  a.y = q.y; a.y_dtype = q.y_dtype; a.ld_y = q.ld_y;
  a.y_vec = (reinterpret_cast<uintptr_t>(q.y) & 15) == 0 && q.ld_y % 4 == 0;
  a.bias = static_cast<const __half*>(q.bias);
  a.batch = q.batch; a.N = q.out_f; a.nb = f.nb;
  a.status = q.status;
  a.grp = f.grp; a.n_problems = q.max_problems;
  a.codes_stride = q.codes_stride; a.norms_stride = q.norms_stride; a.tiles_stride = q.tiles_stride;
  const int rc = q.packed ? (q.tiles ? launch_bulk_kind<true, true>(a, sms, st) : launch_bulk_kind<true, false>(a, sms, st))
                          : (q.tiles ? launch_bulk_kind<false, true>(a, sms, st) : launch_bulk_kind<false, false>(a, sms, st));
  if (rc == PE_OK && !f.in_line) line_extend(st);
  return rc;
}

}  // namespace pe
