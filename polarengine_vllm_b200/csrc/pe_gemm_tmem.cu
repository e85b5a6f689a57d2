// Quantized matmul on the tensor cores with the decoded weights in TENSOR MEMORY: up to 256 activation rows (and more,
// where many_rows_plan says so), and the
// grouped launches over the experts of a mixture layer.
//
//   Y[m, n] = sum_k X[m, k] * (ct[code[n, k]] * norm[n, k / 128])     (+ bias[n]; or silu(first half) * second half)
//
// The weight rows are the M = 128 side of tcgen05.mma and the activation rows its N side, so a tile costs what its
// tokens cost, rounded up to 16 instead of to 128 or 256.  A tile is 128 * halves weight rows (halves = 1 or 2) by up
// to 256 / halves (192 for two halves) tokens; both walk K in steps of 64.  Per CTA, one per SM, persistent:
//   * warp 0 copies the bf16 activations of a step;
//   * warp 2 copies raw codes, 128 weight rows x 128 K at a time;
//   * warps 8..23 decode.  Four groups of four warps; group g owns weight stage g.  A thread owns one weight row: it
//     reads the row's 64 codes, turns them into 32 bf16 pairs (byte permutes for up to eight levels, one table look-up
//     per code byte otherwise) times the block norm, and stores them with one tcgen05.st: operand A of the MMA is read
//     from tensor memory, so decoded weights take no shared-memory bandwidth at all, written or read;
//   * warps 1 and 3 issue the MMAs, accumulating in TMEM columns 0..383, weight stages in columns 384..511;
//   * warps 4..7 read finished accumulators back and store them, while the next tile is decoded.  A lane is a weight row,
//     so the stores of a token are consecutive.  Tiles whose accumulators fit 192 columns alternate between two sets.
//
// What bounds it: with up to about 100 tokens per tile the decode (13 instructions per 8 weights, near 60% of the issue
// slots), above that the MMAs and the issue of one after the other.  The form before had the weights in shared memory as
// the N = 256 side, padded tokens to 128 and drained accumulators with the decode warps: 16384 rows over 128 experts of
// 2688 -> 2 x 1856 took 492 us, 298 us now (343 us with the activation function, which was a pass of 36 us of its own).
//
// Every wait is bounded: on time-out a status code is recorded, all roles leave their loops, TMEM is released.
#include "pe_gemm_tmem.cuh"

namespace pe {

constexpr int kTmThreads = 768;
constexpr int kTmBarAddr = 1536;                // shared-window addresses: barriers,
constexpr int kTmTabAddr = 2048;                // the centroid table if there is one (256 B per entry: a byte permute forms the address),
constexpr int kTmTabBytes = 65536;              // activation stages behind it (their depth covers L2's latency: the longer ring without a
constexpr int kTmCAddr = 165888;                // table is worth a tenth), and code stages
constexpr int kTmCBytes = 65536;
constexpr int kTmEnd = kTmCAddr + kTmCBytes;
constexpr int kTmSmem = kTmEnd - 1024;          // the dynamic window starts at 1024; above it would not fit
constexpr int kTmMaxX = 8;                         // activation stages at most
constexpr int kTmAcc = 192;                        // columns of one accumulator set
constexpr int kTmW = 384;                          // first column of the weight stages, 32 columns each

struct TmUnit { int m0, rows, tn, n0, crow, expert, halves, kb0, kb1, split; };

__device__ __forceinline__ TmUnit tm_unit(const TmemGemmArgs& p, int unit) {
  TmUnit u;
  if (p.gtiles) {
    const int4 d = __ldg(p.gtiles + unit);
    u.m0 = d.x; u.rows = d.y; u.n0 = d.z; u.expert = d.w;
    u.crow = d.w * p.expert_codes + d.z;
    u.halves = p.up_row || d.z + 128 < p.N ? 2 : 1;
    u.kb0 = 0; u.kb1 = p.nb; u.split = 0;
  } else {
    const int tile = unit / p.ksplit;
    u.split = unit - tile * p.ksplit;
    u.m0 = (tile % p.tiles_m) * p.tok;
    u.rows = p.M - u.m0 < p.tok ? p.M - u.m0 : p.tok;
    u.n0 = (tile / p.tiles_m) * 128 * p.halves;
    u.expert = 0; u.crow = u.n0;
    u.halves = p.halves == 2 && u.n0 + 128 < p.N ? 2 : 1;
    u.kb0 = (int)((long long)u.split * p.nb / p.ksplit);
    u.kb1 = (int)((long long)(u.split + 1) * p.nb / p.ksplit);
  }
  u.tn = (u.rows + 15) & ~15;
  return u;
}

__device__ __forceinline__ void mma_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// table entry of code byte BYTE: its address is byte * 256 + lane * 4 (+ the table's), formed by one permute
template <int BYTE>
__device__ __forceinline__ uint32_t tab_ld(uint32_t word, uint32_t lane4) {
  uint32_t a, v;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(a) : "r"(word), "r"(lane4), "n"(0x7604 | (BYTE << 4)));
  asm volatile("ld.shared.b32 %0, [%1 + %2];" : "=r"(v) : "r"(a), "n"(kTmTabAddr));
  return v;
}
// 64 codes of a row (16-byte pieces) -> 32 bf16 pairs times the norm
template <bool PACKED, bool REGTAB>
__device__ __forceinline__ void decode64(const uint4* c, uint32_t n2, uint32_t lane4, const RegTable& tb, uint32_t (&o)[32]) {
#pragma unroll
  for (int i = 0; i < (PACKED ? 2 : 4); ++i) {
    const uint32_t w[4] = {c[i].x, c[i].y, c[i].z, c[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (PACKED) {
        uint32_t a[4];
        if (REGTAB) {
          reg_decode(w[j], tb, a);
        } else {
          a[0] = tab_ld<0>(w[j], lane4); a[1] = tab_ld<1>(w[j], lane4); a[2] = tab_ld<2>(w[j], lane4); a[3] = tab_ld<3>(w[j], lane4);
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) o[16 * i + 4 * j + b] = bf16x2_mul(a[b], n2);
      } else {
        o[8 * i + 2 * j] = bf16x2_mul(lo_hi16(tab_ld<0>(w[j], lane4), tab_ld<1>(w[j], lane4)), n2);
        o[8 * i + 2 * j + 1] = bf16x2_mul(lo_hi16(tab_ld<2>(w[j], lane4), tab_ld<3>(w[j], lane4)), n2);
      }
    }
  }
}

template <bool PACKED, bool REGTAB>
__global__ void __launch_bounds__(kTmThreads, 1)
gemm_tmem_kernel(const TmemGemmArgs p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap cmap) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kXAddr = kTmTabAddr + (REGTAB ? 0 : kTmTabBytes);
  constexpr int kCodeStage = PACKED ? 8192 : 16384, NC = kTmCBytes / kCodeStage / 2;  // two rings of NC code stages
  const uint32_t raw = smem_u32(smem_raw);
  if (raw > kTmBarAddr || raw < 1024) {  // the fixed addresses would leave the window
    if (threadIdx.x == 0) record_timeout(p.status, 12);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bars = kTmBarAddr;
  auto full_x = [&](int s) { return bars + 8 * s; };         // 8
  auto empty_x = [&](int s) { return bars + 64 + 8 * s; };   // 8
  auto full_c = [&](int s) { return bars + 128 + 8 * s; };   // 8
  auto empty_c = [&](int s) { return bars + 192 + 8 * s; };  // 8
  auto full_w = [&](int s) { return bars + 256 + 8 * s; };   // 4
  auto empty_w = [&](int s) { return bars + 288 + 8 * s; };  // 4
  auto acc_full = [&](int s) { return bars + 320 + 8 * s; };   // 2
  auto acc_empty = [&](int s) { return bars + 336 + 8 * s; };  // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (bars + 352 - raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + (bars + 356 - raw));
  const uint32_t sink = bars + 360, both_here = bars + 368;

  if (tid == 0) {
    for (int s = 0; s < p.nx; ++s) { mbar_init(full_x(s), 1); mbar_init(empty_x(s), 2); }
    for (int s = 0; s < 2 * NC; ++s) { mbar_init(full_c(s), 1); mbar_init(empty_c(s), 8); }  // two groups read a code stage
    for (int s = 0; s < 4; ++s) { mbar_init(full_w(s), 4); mbar_init(empty_w(s), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(acc_full(s), 2); mbar_init(acc_empty(s), 4); }
    mbar_init(both_here, 2);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (!REGTAB && warp >= 8) {  // one copy of the table per lane
    for (int e = warp - 8; e < (PACKED ? 256 : p.n_levels); e += 16) {
      uint32_t v;
      if (PACKED) {
        const int lo = e & 15, hi = e >> 4;
        v = pack_bf16(lo < p.n_levels ? p.ct[lo] : 0.f, hi < p.n_levels ? p.ct[hi] : 0.f);
      } else {
        v = pack_bf16(p.ct[e], p.ct[e]);
      }
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(kTmTabAddr + e * 256 + lane * 4), "r"(v) : "memory");
    }
  }
  if (warp == 3) {  // TMEM: all 512 columns, allocated and later freed by this warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // Codes, norms and table may be read at once: the preparation launch waited for whatever wrote them before it let this one start.
  // Its activations, the tile list and what an older launch may still read of the output wait for it.  (200 rows, 4096 x 4096 Q4:
  // 22.3 -> 20.9 us, 12288 x 4096 Q4 34.3 -> 33.1.)
  asm volatile("griddepcontrol.launch_dependents;");
  if (p.gtiles || warp == 0 || (warp >= 4 && warp < 8)) asm volatile("griddepcontrol.wait;" ::: "memory");

  const int n_units = p.gtiles ? *p.n_gtiles : p.tiles_m * p.tiles_n * p.ksplit;

  if (warp == 0) {
    // ---------------- activations ----------------
    const bool one = elect_one();
    int sx = 0, ph = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
      const TmUnit u = tm_unit(p, unit);
      const int copies = (u.tn + p.xbox - 1) / p.xbox;
      for (int ks = 2 * u.kb0; ks < 2 * u.kb1; ++ks) {
        ok = __all_sync(0xffffffffu, mbar_wait(empty_x(sx), ph ^ 1, abort_flag, p.status, 1));
        if (!ok) break;
        const uint32_t dst = kXAddr + sx * p.x_stage;
        if (one) {
          mbar_expect_tx(full_x(sx), copies * p.xbox * 128);
          for (int i = 0; i < copies; ++i) tma_load_2d(dst + i * p.xbox * 128, &xmap, ks * kStepK, u.m0 + i * p.xbox, full_x(sx));
        }
        __syncwarp();
        if (++sx == p.nx) { sx = 0; ph ^= 1; }
      }
    }
  } else if (warp == 2) {
    // ---------------- codes ----------------
    // Two rings: the blocks of the first half and those of the second (of a tile of one half: every other block), each
    // read by the two decode groups of its own.  (A wait on a barrier's parity is sound only when the waiter knows that
    // the phase before has passed, that is when it took every earlier stage of the ring itself.)
    const bool one = elect_one();
    int n[2] = {0, 0};
    bool ok = true;
    for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
      const TmUnit u = tm_unit(p, unit);
      for (int i = 0; i < (u.kb1 - u.kb0) * u.halves && ok; ++i) {
        const int c = i & 1, kb = u.kb0 + (u.halves == 2 ? i >> 1 : i), row = u.crow + (u.halves == 2 && c ? (p.up_row ? p.up_row : 128) : 0);
        const int at = c ? n[1]++ : n[0]++, sc = c * NC + at % NC;
        ok = __all_sync(0xffffffffu, mbar_wait(empty_c(sc), ((at / NC) & 1) ^ 1, abort_flag, p.status, 6));
        if (!ok) break;
        if (one) {
          mbar_expect_tx(full_c(sc), kCodeStage);
          tma_load_2d(kTmCAddr + sc * kCodeStage, &cmap, kb * (PACKED ? 64 : 128), row, full_c(sc));
        }
        __syncwarp();
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ---------------- MMA issuers: warp 1 for the first half of a tile, warp 3 for the second ----------------
    // A trip through a step -- two barriers, four MMAs, two commits -- is a serial chain that takes as long as the step's
    // decode or MMAs; one warp for both halves was what bounded the kernel.  The next barriers are asked about before the
    // MMAs of a step, so that the answer is there after them.  Tiles of one half: warp 1.
    if (elect_one()) {
      const int m = warp >> 1;
      int sx = 0, phx = 0;
      uint32_t phw = 0, phe = 0;  // one phase bit per pair of weight stages (s, s + 2); per accumulator set
      int next = 0;               // set of the next tile that needs one only
      bool ok = true;
      auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        return mbar_wait(bar, parity, abort_flag, p.status, code);
      };
      int phm = 0;
      auto meet = [&]() {
        mbar_arrive(both_here);
        const bool r = wait(both_here, phm, 13);
        phm ^= 1;
        return r;
      };
      for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
        const TmUnit u = tm_unit(p, unit);
        const bool both = u.halves * u.tn > kTmAcc;
        const int set = both ? 0 : next;
        if (!both) next ^= 1;
        ok = wait(acc_empty(set), ((phe >> set) & 1) ^ 1, 9);
        phe ^= 1u << set;
        if (ok && both) {
          ok = wait(acc_empty(1), ((phe >> 1) & 1) ^ 1, 9);
          phe ^= 2u;
        }
        if (!ok) break;
        const bool two = u.halves == 2;
        if (!two && !meet()) { ok = false; break; }  // both warps have taken every stage up to here
        if (!two && m == 1) {  // not this warp's: only its place in the rings moves on
          for (int i = 0; i < 2 * (u.kb1 - u.kb0); ++i) {
            if (++sx == p.nx) { sx = 0; phx ^= 1; }
            if (i & 1) phw ^= 1u << ((i >> 1) & 1);
          }
          ok = meet();
          continue;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + set * kTmAcc + m * u.tn;
        // D fp32, A and B bf16, both K-major, M = 128, N = tn
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(u.tn >> 3) << 17) | ((128u >> 4) << 24);
        auto issue = [&](int stage, uint32_t x, uint32_t acc) {
          const uint64_t db = smem_desc_sw128(x);
          const uint32_t a = tmem + kTmW + stage * 32;
#pragma unroll
          for (int kk = 0; kk < kStepK / 16; ++kk) mma_tmem_a(d, a + kk * 8, db + 2 * kk, idesc, kk > 0 ? 1u : acc);
          umma_commit(empty_w(stage));
        };
        int c = m;  // a block's weight stages: c and c + 2; of a tile of one half the two pairs take turns
        bool ready = false;
        for (int n = u.kb1 - u.kb0, i = 0; i < n && ok; ++i) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (!ready) ok = wait(full_x(sx), phx, 2) && wait(full_w(c + 2 * j), (phw >> c) & 1, 3);
            if (!ok) break;
            const uint32_t x = kXAddr + sx * p.x_stage, done_x = empty_x(sx), stage = c + 2 * j;
            if (++sx == p.nx) { sx = 0; phx ^= 1; }
            if (j == 1) {
              phw ^= two ? 3u : 1u << c;
              if (!two) c ^= 1;
            }
            ready = mbar_test(full_x(sx), phx) & mbar_test(full_w(c + 2 * (j ^ 1)), (phw >> c) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue(stage, x, i > 0 || j > 0);
            umma_commit(done_x);
            if (!two) umma_commit(done_x);  // the barrier counts both halves
          }
        }
        if (ok) {
          umma_commit(acc_full(set));
          if (!two) umma_commit(acc_full(set));
        }
        if (ok && !two) ok = meet();
      }
    }
  } else if (warp >= 8) {
    // ---------------- decode ----------------
    const int g = (warp - 8) >> 2, q = warp & 3, r = q * 32 + lane;
    const RegTable tb = REGTAB ? bf16_reg_table(p.ct, p.n_levels) : RegTable{0, 0, 0, 0};
    const uint32_t wdst = tmem + kTmW + g * 32 + ((uint32_t)(q * 32) << 16);
    const int xr = PACKED ? (r >> 1) & 3 : r & 7;  // 16-byte piece j of a row sits at j ^ xr (64- or 128-byte swizzle)
    // the group's sequence of (unit, block of K): every block of its half of two, every other block of one
    const int cls = g & 1, kh = g >> 1;
    int unit = blockIdx.x, kb = 0, ci = 0;
    TmUnit u = {};
    bool live = unit < n_units;
    const unsigned short* np = nullptr;  // norm of (this row, block kb); nullptr: the row does not exist
    auto enter = [&]() {                 // to the first block of this unit, or of the next that has one for this group
      while (live) {
        u = tm_unit(p, unit);
        kb = u.kb0 + (u.halves == 2 ? 0 : cls);
        if (kb < u.kb1) break;
        unit += gridDim.x;
        live = unit < n_units;
      }
      const int row = u.n0 + (u.halves == 2 && cls ? (p.up_row ? p.up_row : 128) : 0) + r, limit = p.up_row ? 2 * p.up_row : p.N;
      np = live && row < limit
               ? reinterpret_cast<const unsigned short*>(p.norms) + u.expert * p.expert_norms + (int64_t)row * p.ld_norms + kb
               : nullptr;
    };
    enter();
    unsigned short nf = np ? __ldg(np) : 0;
    int phw = 1;
    while (live) {
      const uint32_t n2 = pack_bf16(__half2float(__ushort_as_half(nf)), __half2float(__ushort_as_half(nf)));
      const int by = u.halves == 2 ? 1 : 2;
      kb += by;
      if (np) np += by;
      if (kb >= u.kb1) {
        unit += gridDim.x;
        live = unit < n_units;
        enter();
      }
      nf = np ? __ldg(np) : 0;  // on its way during the waits and the decode of this block
      const int sc = cls * NC + ci % NC, phc = (ci / NC) & 1;
      ++ci;
      if (!__all_sync(0xffffffffu, mbar_try(full_c(sc), phc))) {
        const bool ok = mbar_wait(full_c(sc), phc, abort_flag, p.status, 7);
        if (!__all_sync(0xffffffffu, ok)) break;  // leave together or not at all
      }
      constexpr int CW = PACKED ? 2 : 4;
      uint4 c[CW];
      const uint32_t src = kTmCAddr + sc * kCodeStage + r * (PACKED ? 64 : 128);
      uint32_t seen = 0;
#pragma unroll
      for (int i = 0; i < CW; ++i) {
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(c[i].x), "=r"(c[i].y), "=r"(c[i].z), "=r"(c[i].w) : "r"(src + (uint32_t)(((kh * CW + i) ^ xr) << 4)) : "memory");
      }
      // the stage goes back only after the loads have delivered (a store that consumes them stands between)
#pragma unroll
      for (int i = 0; i < CW; ++i) seen |= c[i].x | c[i].y | c[i].z | c[i].w;
      asm volatile("st.shared.u32 [%0], %1;" ::"r"(sink), "r"(seen) : "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_c(sc));
      uint32_t o[32];
      decode64<PACKED, REGTAB>(c, n2, lane * 4, tb, o);
      if (!__all_sync(0xffffffffu, mbar_try(empty_w(g), phw))) {
        const bool ok = mbar_wait(empty_w(g), phw, abort_flag, p.status, 4);
        if (!__all_sync(0xffffffffu, ok)) break;
      }
      phw ^= 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tmem_st32(wdst, o);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full_w(g));
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int q = warp & 3;
    uint32_t phf = 0;
    int next = 0;
    for (int unit = blockIdx.x; unit < n_units; unit += gridDim.x) {
      const TmUnit u = tm_unit(p, unit);
      const bool both = u.halves * u.tn > kTmAcc;
      const int set = both ? 0 : next;
      if (!both) next ^= 1;
      {
        const bool ok = mbar_wait(acc_full(set), (phf >> set) & 1, abort_flag, p.status, 5);
        if (!__all_sync(0xffffffffu, ok)) break;
      }
      phf ^= 1u << set;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t0 = tmem + set * kTmAcc + ((uint32_t)(q * 32) << 16);
      const int row0 = u.n0 + q * 32 + lane;
      if (p.up_row) {  // first half: gate, second half: up (the fast exponential and division: errors far below fp16's)
        const bool on = row0 < p.N;
        __half* dst = static_cast<__half*>(p.y) + (int64_t)u.m0 * p.ld_y + row0;
        for (int c = 0; c < u.tn; c += 16) {
          uint32_t a[16], b[16];
          tmem_ld16(t0 + c, a);
          tmem_ld16(t0 + u.tn + c, b);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j, dst += p.ld_y) {
            const float f = __uint_as_float(a[j]);
            if (on && c + j < u.rows) *dst = __float2half_rn(__fdividef(f, 1.f + __expf(-f)) * __uint_as_float(b[j]));
          }
        }
      } else {
        for (int h = 0; h < u.halves; ++h) {
          const int row = row0 + 128 * h;
          const bool on = row < p.N;
          const float bias = p.bias && on && p.ksplit == 1 ? __half2float(p.bias[row]) : 0.f;
          auto drain = [&](auto* dst, int64_t ld) {
            using T = typename std::remove_pointer<decltype(dst)>::type;
            dst += (int64_t)u.m0 * ld + row;
            for (int c = 0; c < u.tn; c += 32) {
              uint32_t a[32];
              tmem_ld32(t0 + h * u.tn + c, a);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 32; ++j, dst += ld) {
                const float f = __uint_as_float(a[j]) + bias;
                if (on && c + j < u.rows) {
                  if constexpr (sizeof(T) == 4) *dst = f;
                  else if constexpr (std::is_same<T, __half>::value) *dst = __float2half_rn(f);
                  else *dst = __float2bfloat16_rn(f);
                }
              }
            }
          };
          if (p.ksplit > 1) drain(p.part + (size_t)u.split * p.M * p.N, (int64_t)p.N);
          else if (p.y_dtype == PE_F32) drain(static_cast<float*>(p.y), p.ld_y);
          else if (p.y_dtype == PE_F16) drain(static_cast<__half*>(p.y), p.ld_y);
          else drain(static_cast<__nv_bfloat16*>(p.y), p.ld_y);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(acc_empty(set));
        if (both) mbar_arrive(acc_empty(1));
      }
    }
  }

  // ---------------- common exit ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag && tid == 0) {  // give copies that may still be in flight time to land
    const long long t0 = clock64();
    while (clock64() - t0 < 200000) {}
  }
  __syncthreads();
  if (warp == 3) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

int launch_gemm_tmem(TmemGemmArgs& a, const void* codes, int packed, int64_t ld_codes, int64_t code_rows, const void* xq, int64_t x_total, int units,
                     int sms, cudaStream_t st) {
  const bool regtab = packed && a.n_levels <= 8;
  const int x_bytes = kTmCAddr - kTmTabAddr - (regtab ? 0 : kTmTabBytes);
  a.nx = x_bytes / a.x_stage < kTmMaxX ? x_bytes / a.x_stage : kTmMaxX;
  CUtensorMap xmap, cmap;
  const int K = a.nb * kBlock;
  int rc = encode_map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, xq, K, x_total, (uint64_t)K * 2, kStepK, a.xbox,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (rc == PE_OK)
    rc = encode_map_2d(&cmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, codes, packed ? K / 2 : K, code_rows, ld_codes, packed ? 64 : 128, 128,
                       packed ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  if (rc != PE_OK) return rc;
  auto kfn = !packed ? gemm_tmem_kernel<false, false> : regtab ? gemm_tmem_kernel<true, true> : gemm_tmem_kernel<true, false>;
  PE_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTmSmem));
  PE_CUDA_TRY(launch_pdl(kfn, dim3((unsigned)(units < sms ? units : sms)), dim3(kTmThreads), kTmSmem, st, a, xmap, cmap));
  return PE_OK;
}

// Tile list of a grouped launch from the experts' row ranges (first, count): for every expert its activation tiles (as
// few as hold 192 rows each, of equal size to within one) x tiles_n weight tiles, the weight tiles of one activation
// tile adjacent, so that CTAs that run side by side share the activation tile in L2.  One block of 1024.
__global__ void __launch_bounds__(1024) gemm_tile_list_kernel(const int* expert_rows, int n_experts, int tiles_n, int tile_rows, int max_tiles,
                                                              int4* tiles, int* n_tiles) {
  __shared__ int4 span[1024];  // per expert: first row, rows, activation tiles, first tile
  __shared__ int warp_tot[32];
  pdl_enter();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = tid < n_experts ? expert_rows[2 * tid] : 0, cnt = tid < n_experts ? expert_rows[2 * tid + 1] : 0;
  const int mt = (cnt + kTmAcc - 1) / kTmAcc;
  int t = mt * tiles_n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, t, o);
    if (lane >= o) t += x;
  }
  if (lane == 31) warp_tot[warp] = t;
  __syncthreads();
  for (int w = 0; w < warp; ++w) t += warp_tot[w];
  span[tid] = make_int4(first, cnt, mt, t - mt * tiles_n);
  if (tid == 1023) *n_tiles = t < max_tiles ? t : max_tiles;
  __syncthreads();
  for (int e = warp; e < n_experts; e += 32) {
    const int4 s = span[e];
    for (int i = lane; i < s.z * tiles_n; i += 32) {
      const int a = i / tiles_n, n = i - a * tiles_n;
      const int r0 = (int)((long long)s.y * a / s.z), r1 = (int)((long long)s.y * (a + 1) / s.z);
      if (s.w + i < max_tiles) tiles[s.w + i] = make_int4(s.x + r0, r1 - r0, n * tile_rows, e);
    }
  }
}

PE_WAIT_STATUS_READER(gemm_tmem_wait_status)

}  // namespace pe

using namespace pe;

// ---- grouped launch: the experts of a mixture layer, prefill-size batches ----------------------------
// workspace: [status, 256 B][tile count, 256 B][tile list][bf16 activations rows x K]
static int grouped_max_tiles(int n_experts, int rows, int out_f) {
  return (n_experts + rows / kTmAcc) * ((out_f + 255) / 256 + 1);  // + 1: gate and up halves of 128 rows each
}

extern "C" size_t pe_gemm_grouped_workspace_bytes(int n_experts, int rows, int out_f, int in_f_padded) {
  if (n_experts < 1 || n_experts > 1024 || rows < 1 || out_f < 1 || in_f_padded < kBlock || in_f_padded % kBlock) return 0;
  const size_t list = ((size_t)grouped_max_tiles(n_experts, rows, out_f) * 16 + 255) & ~(size_t)255;
  return 512 + list + (size_t)rows * in_f_padded * 2;
}

static int grouped(const void* codes, int packed, int64_t ld_codes, int64_t codes_stride, const void* norms, int64_t ld_norms, int64_t norms_stride,
                   const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype, int64_t ld_x, int in_f, const int32_t* x_rows,
                   const int32_t* x_to, int n_x, int fanout, int silu_mul, void* y, int y_dtype, int64_t ld_y, const int32_t* expert_rows, int n_experts, int rows, int out_f,
                   int in_f_padded, void* workspace, size_t workspace_bytes, void* stream) {
  if (!codes || !norms || !ct_scaled || !x || !y || !expert_rows || !workspace) return PE_ERR_ARG;
  if (n_experts < 1 || rows < 1 || out_f < 1 || in_f < 1 || in_f > in_f_padded) return PE_ERR_ARG;
  if (n_experts > 1024) return PE_ERR_LIMIT;
  if (x_kind != PE_X_ROTATED && x_kind != PE_X_RAW) return PE_ERR_ARG;
  if (x_dtype < PE_F32 || x_dtype > PE_BF16 || y_dtype < PE_F32 || y_dtype > PE_BF16) return PE_ERR_ARG;
  if (n_levels < 2 || n_levels > 256 || (packed && n_levels > 16)) return PE_ERR_ARG;
  if (silu_mul && (out_f % 2 || y_dtype != PE_F16)) return PE_ERR_ARG;
  if (in_f_padded % kBlock) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15)) return PE_ERR_ALIGN;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return PE_ERR_ALIGN;
  // the experts' code matrices are addressed as one tall 2-D tensor: they must follow each other
  if (codes_stride != (int64_t)out_f * ld_codes) return PE_ERR_ARG;
  const int y_cols = silu_mul ? out_f / 2 : out_f;
  if (ld_codes < (packed ? in_f_padded / 2 : in_f_padded) || ld_norms < in_f_padded / kBlock) return PE_ERR_ARG;
  if (ld_x < (x_kind == PE_X_RAW ? in_f : in_f_padded) || ld_y < y_cols) return PE_ERR_ARG;
  if ((int64_t)n_experts * out_f > 0x7fffffff) return PE_ERR_LIMIT;
  const size_t need = pe_gemm_grouped_workspace_bytes(n_experts, rows, out_f, in_f_padded);
  if (need == 0) return PE_ERR_SHAPE;
  if (workspace_bytes < need) return PE_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int sms = sm_count();
  if (sms <= 0) return PE_ERR_CUDA;

  const int max_tiles = grouped_max_tiles(n_experts, rows, out_f);
  const size_t list_bytes = ((size_t)max_tiles * 16 + 255) & ~(size_t)255;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  int* status = reinterpret_cast<int*>(ws);
  int* n_tiles = reinterpret_cast<int*>(ws + 256);
  int4* tiles = reinterpret_cast<int4*>(ws + 512);
  void* xq = ws + 512 + list_bytes;
  const int tile_rows = silu_mul ? 128 : 256, tiles_n = (y_cols + tile_rows - 1) / tile_rows;
  PE_CUDA_TRY(launch_pdl(gemm_tile_list_kernel, dim3(1), dim3(1024), 0, st, expert_rows, n_experts, tiles_n, tile_rows, max_tiles, tiles, n_tiles));
  // (the preparation kernel clears the status word)
  const int rc = launch_gemm_prep(x, x_kind, x_dtype, ld_x, in_f, xq, x_to ? n_x : rows, in_f_padded, packed ? 1 : 0, x_rows,
                                  x_to ? nullptr : expert_rows + 2 * (n_experts - 1), x_to, fanout, status, st);
  if (rc != PE_OK) return rc;

  TmemGemmArgs a = {};
  a.norms = static_cast<const __half*>(norms); a.ld_norms = ld_norms; a.expert_norms = norms_stride;
  a.ct = ct_scaled; a.n_levels = n_levels;
  a.y = y; a.y_dtype = y_dtype; a.ld_y = ld_y;
  a.M = rows; a.N = y_cols; a.nb = in_f_padded / kBlock;
  a.ksplit = 1;
  a.xbox = 32; a.x_stage = kTmAcc * 128;
  a.gtiles = tiles; a.n_gtiles = n_tiles; a.expert_codes = out_f;
  a.up_row = silu_mul ? y_cols : 0;
  a.status = status;
  return launch_gemm_tmem(a, codes, packed, ld_codes, (int64_t)n_experts * out_f, xq, rows, max_tiles, sms, st);
}

extern "C" int pe_gemm_grouped(const void* codes, int packed, int64_t ld_codes, int64_t codes_stride, const void* norms,
                               int64_t ld_norms, int64_t norms_stride, const float* ct_scaled, int n_levels, const void* x,
                               int x_kind, int x_dtype, int64_t ld_x, int in_f, const int32_t* x_rows, void* y, int y_dtype,
                               int64_t ld_y, const int32_t* expert_rows, int n_experts, int rows, int out_f, int in_f_padded,
                               void* workspace, size_t workspace_bytes, void* stream) {
  return grouped(codes, packed, ld_codes, codes_stride, norms, ld_norms, norms_stride, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, x_rows, nullptr, 0, 0, 0, y,
                 y_dtype, ld_y, expert_rows, n_experts, rows, out_f, in_f_padded, workspace, workspace_bytes, stream);
}

extern "C" int pe_gemm_grouped_silu_mul(const void* codes, int packed, int64_t ld_codes, int64_t codes_stride, const void* norms,
                                        int64_t ld_norms, int64_t norms_stride, const float* ct_scaled, int n_levels, const void* x,
                                        int x_kind, int x_dtype, int64_t ld_x, int in_f, const int32_t* x_to, int n_x, int fanout, void* y,
                                        int64_t ld_y, const int32_t* expert_rows, int n_experts, int rows, int out_f, int in_f_padded,
                                        void* workspace, size_t workspace_bytes, void* stream) {
  if (!x_to || n_x < 1 || fanout < 1 || (int64_t)n_x * fanout > rows) return PE_ERR_ARG;
  return grouped(codes, packed, ld_codes, codes_stride, norms, ld_norms, norms_stride, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, nullptr, x_to, n_x, fanout, 1, y,
                 PE_F16, ld_y, expert_rows, n_experts, rows, out_f, in_f_padded, workspace, workspace_bytes, stream);
}
