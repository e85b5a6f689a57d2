// Prefill-size quantized matmul (many activation rows) on the 5th-generation tensor
// cores: tcgen05.mma with TMEM accumulators, TMA-staged activations, in-kernel dequant.
//
//   Y[m, n] = sum_k Xt[m, k] * (ct[code[n, k]] * norm[n, k / 128])        (+ bias[n])
//
// gemm_pair_kernel: more than 256 rows, where many_rows_plan does not prefer the tensor-memory kernel.  A cluster of two CTAs per 512 tokens x 256 weight rows, one cta_group::2 MMA
// per pair, each CTA decoding half of the weight tile.  (Up to 256 rows: pe_gemm_tmem.cu.)  It walks K in steps of 64:
//   * one thread issues TMA (cp.async.bulk.tensor.2d, 128-byte swizzle, no multicast) for the bf16
//     activation tiles and another for the raw code rows of the step;
//   * 16 decode warps turn code rows into a bf16 weight stage in the swizzled K-major layout the tensor
//     core reads (table look-up or byte permutes, times the block norm) -- the decoded weights never
//     touch HBM or L2.  The warps form groups that take alternate K steps, because one warp's trip through
//     a step (barrier round trips, proxy fence) lasts longer than the step's MMAs;
//   * one thread issues tcgen05.mma (bf16 in, fp32 accumulate in TMEM: two accumulators of 256 columns
//     = all 512) and hands stages back with tcgen05.commit;
//   * after the last step the decode warps read the accumulators back (tcgen05.ld), add the bias,
//     convert and store.
// The activations are prepared by a small kernel (pad + FWHT-128 for raw input, bf16, and for nibble
// layers the (k, k+64) pairing of the half-block layout so that one code byte decodes to two adjacent
// K elements).
//
// Every wait is bounded: on time-out the kernel records a status code in the first word
// of the workspace, all roles leave their loops, TMEM is released and the grid returns.
#include "pe_gemm_tmem.cuh"

namespace pe {

constexpr int kTileN = 256;          // weight rows per tile (UMMA N)
constexpr int kXTileBytes = 128 * kStepK * 2;        // 16 KB
constexpr int kDecodeThreads = 512;

struct GemmArgs {
  const __half* norms; int64_t ld_norms;
  const float* ct; int n_levels;
  void* y; int y_dtype; int64_t ld_y;
  const __half* bias;
  int M, N, K;
  int tiles_m, tiles_n;
  int lut_bytes;  // n_levels (256 for nibble pairs) x table stride
  int nc;         // code stages
  int full;       // tiles 0 .. full - 1 are computed whole, the others in ksplit K ranges each
  int ksplit;
  int col0;       // first column of the split tiles
  float* part;    // [ksplit][M][N - col0] fp32
  int y_tma;      // the output leaves through TMA stores (16-byte aligned rows)
  int part_tma;   // ... and so do the partials
  int* status;
};

// ---- paired form: two CTAs of a cluster share one tensor-core operation (cta_group::2) -----------------
// A pair owns 512 tokens x 256 weight rows.  Each CTA keeps ITS 128-token halves of the two 256-token
// accumulators in its own TMEM, stages its own activation tiles and decodes only 128 of the 256 weight
// rows: the tensor core of each SM reads that half from its own shared memory, so the decode work and the
// weight-operand traffic per SM are half of the single-CTA form (which is bound by them: with the decode
// and the activation copies switched off it still ran at three quarters of the dense-GEMM rate).
// The even CTA of the pair issues the MMAs.  It learns that the odd CTA's stages are full through
// arrivals on its own barriers (the byte count of both CTAs' activation copies, the decode warps'
// for the weight stages) and hands stages back with one tcgen05.commit per CTA.
constexpr int kPairWStages = 4;                      // 16 KB each: this CTA's 128 weight rows; one per decode group
constexpr int kPairCodeStages = 4;                   // one per decode group
constexpr int kPairLutStride = 64;                   // nibble layers: 16 copies of the 256-entry pair table (16 KB)
constexpr int kPairWTileBytes = 128 * kStepK * 2;
constexpr int kPairTileM = 512;
constexpr int kPairThreads = 64 + kDecodeThreads + 32;     // 19 warps: activation TMA, MMA, 16 decode/epilogue, code TMA
constexpr int kPairGroups = 4;                       // decode warp groups, one K step each.  A group owns weight stage g and
                                                     // code stage g: a parity wait is only sound while the waiter is
                                                     // less than two phases ahead of the barrier, which sharing a stage
                                                     // between groups does not guarantee
static_assert(kPairWStages == kPairGroups && kPairCodeStages == kPairGroups, "one stage of each ring per decode group");
constexpr int kPairGroupWarps = kDecodeThreads / 32 / kPairGroups;
constexpr uint32_t kIdescPair = (1u << 4) | (1u << 7) | (1u << 10) | ((kTileN >> 3) << 17) | ((256u >> 4) << 24);

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared-memory address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait on a barrier that CTAs of the cluster arrive on
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (mbar_try_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (mbar_try_cluster(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > kTimeoutCycles) {
      *abort_flag = 1;
      record_timeout(status, code);
      return false;
    }
  }
}
// TMA load of a CTA pair: the bytes land in THIS CTA's shared memory, the completion is counted on a barrier
// that may live in the other CTA of the pair (a mapped address).  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(cluster_bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void umma_pair_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0)
      : "memory");
}
// arrival on ONE barrier (of this CTA or, with a mapped address, of the other) once the MMAs issued so far are done
__device__ __forceinline__ void umma_pair_commit(uint32_t cluster_bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_bar) : "memory");
}

// table entry address: lut + byte * STRIDE + copy * 4
template <int BYTE, int STRIDE>
__device__ __forceinline__ uint32_t glut_s(uint32_t word, uint32_t lane_base) {
  uint32_t b, v;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(b) : "r"(word), "r"(0), "n"(0x4440 | BYTE));
  const uint32_t addr = b * (uint32_t)STRIDE + lane_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

template <bool PACKED>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const GemmArgs p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap cmap,
                 const __grid_constant__ CUtensorMap ymap, const __grid_constant__ CUtensorMap partmap) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023) & ~1023u;
  uint8_t* sm = smem_raw + (base - raw);
  // [X stages 4|3 x 32 KB][W stages 4 x 16 KB][table][code stages 4 x (128 rows x 32|64 B)][barriers]
  constexpr int kPairXStages = PACKED ? 4 : 3;  // byte codes need twice the code stages' room
  constexpr int kLutStride = PACKED ? kPairLutStride : 128;
  constexpr int kXStage = 2 * kXTileBytes;
  constexpr uint32_t kWOff = kPairXStages * kXStage;
  constexpr uint32_t kLutOff = kWOff + kPairWStages * kPairWTileBytes;
  constexpr int kCodeRow = PACKED ? 32 : 64;
  constexpr int kCodeStage = 128 * kCodeRow;
  const uint32_t c_off = kLutOff + p.lut_bytes;
  const uint32_t bar_off = c_off + p.nc * kCodeStage;
  const uint32_t lut_s = base + kLutOff;
  uint8_t* lut_g = sm + kLutOff;
  const uint32_t bars = base + bar_off;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + bar_off + 216);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + bar_off + 220);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  auto full_x = [&](int s) { return bars + 8 * s; };          // up to 4
  auto empty_x = [&](int s) { return bars + 32 + 8 * s; };    // up to 4
  auto full_w = [&](int s) { return bars + 64 + 8 * s; };     // 4 (used in the even CTA)
  auto empty_w = [&](int s) { return bars + 96 + 8 * s; };    // 4
  auto full_c = [&](int s) { return bars + 128 + 8 * s; };    // 4
  auto empty_c = [&](int s) { return bars + 160 + 8 * s; };   // 4
  const uint32_t acc_full = bars + 192;
  const uint32_t acc_empty = bars + 200;  // used in the even CTA: both CTAs have read the accumulators of a tile
  const uint32_t stg_free = bars + 208;   // the output staging (inside the weight stages) has been read by the TMA stores

  if (tid == 0) {
    // activation stage: one barrier in the even CTA counts the bytes of both CTAs' copies
    for (int s = 0; s < kPairXStages; ++s) { mbar_init(full_x(s), 1); mbar_init(empty_x(s), 1); }
    // weight stage: the decode warps of both CTAs
    for (int s = 0; s < kPairWStages; ++s) { mbar_init(full_w(s), 2 * kPairGroupWarps); mbar_init(empty_w(s), 1); }
    for (int s = 0; s < p.nc; ++s) { mbar_init(full_c(s), 1); mbar_init(empty_c(s), kPairGroupWarps); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 2 * (kDecodeThreads / 32));  // every decode warp of both CTAs, once per tile
    mbar_init(stg_free, kDecodeThreads / 32);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp >= 2 && warp < 18) {
    const int d = tid - 64;
    for (int e = d >> 5; e < (PACKED ? 256 : p.n_levels); e += kDecodeThreads / 32) {
      uint32_t v;
      if (PACKED) {
        const int lo = e & 15, hi = e >> 4;
        v = pack_bf16(lo < p.n_levels ? p.ct[lo] : 0.f, hi < p.n_levels ? p.ct[hi] : 0.f);
      } else {
        v = pack_bf16(p.ct[e], p.ct[e]);
      }
      if (lane * 4 < kLutStride) *reinterpret_cast<uint32_t*>(lut_g + e * kLutStride + lane * 4) = v;
    }
  }
  if (warp == 1) {  // one warp of EACH CTA of the pair allocates (all 512 columns) and later frees
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs exist before anybody arrives on them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // Codes, norms and table may be read at once: the preparation launch waited for whatever wrote them before it let this one start.
  // Its activations, and what an older launch may still read of the output, wait for it.
  asm volatile("griddepcontrol.launch_dependents;");
  if (warp == 0) asm volatile("griddepcontrol.wait;" ::: "memory");

  const int ksteps = p.K / kStepK;
  // A unit of work is a tile or, for the tiles of a last wave that would leave pairs idle, one of `ksplit` K ranges of a
  // tile (fp32 partials in the workspace, summed by a second kernel).  Whole tiles come first: split = -1.
  const int n_tiles = p.full + (p.tiles_m * p.tiles_n - p.full) * p.ksplit;
  auto unit_of = [&](int unit, int& split, int& ks0, int& ks1) {
    if (unit < p.full) { split = -1; ks0 = 0; ks1 = ksteps; return unit; }
    const int u = unit - p.full, tile = p.full + u / p.ksplit;
    split = u % p.ksplit;
    ks0 = (int)((long long)split * ksteps / p.ksplit);
    ks1 = (int)((long long)(split + 1) * ksteps / p.ksplit);
    return tile;
  };
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

  if (warp == 0) {
    // ---------------- TMA producer: this CTA's activation tiles ----------------
    // Both CTAs' copies complete on the even CTA's barrier, which expects the bytes of both.
    if (lane == 0) {
      const uint32_t lead = map_to_cta(bars, 0) - bars;
      int it = 0;
      for (int unit = pair; unit < n_tiles && !*abort_flag; unit += n_pairs) {
        int split, ks0, ks1;
        const int tile = unit_of(unit, split, ks0, ks1);
        const int m0 = (tile % p.tiles_m) * kPairTileM;
        const bool two = m0 + 256 < p.M;
        for (int ks = ks0; ks < ks1; ++ks, ++it) {
          const int sx = it % kPairXStages;
          if (!mbar_wait(empty_x(sx), ((it / kPairXStages) & 1) ^ 1, abort_flag, p.status, 1)) goto done_producer;
          if (leader) mbar_expect_tx(full_x(sx), 2 * (two ? 2 * kXTileBytes : kXTileBytes));
          tma_load_2d_pair(base + sx * kXStage, &xmap, ks * kStepK, m0 + (int)rank * 128, full_x(sx) + lead);
          if (two) tma_load_2d_pair(base + sx * kXStage + kXTileBytes, &xmap, ks * kStepK, m0 + 256 + (int)rank * 128, full_x(sx) + lead);
        }
      }
    done_producer:;
    }
  } else if (warp == 18) {
    // ---------------- TMA producer: this CTA's code rows (a thread of its own: it runs ahead of the activations) ----------------
    if (lane == 0) {
      int it = 0;
      for (int unit = pair; unit < n_tiles && !*abort_flag; unit += n_pairs) {
        int split, ks0, ks1;
        const int tile = unit_of(unit, split, ks0, ks1);
        const int n0 = (tile / p.tiles_m) * kTileN;
        for (int ks = ks0; ks < ks1; ++ks, ++it) {
          const int sc = it % p.nc;
          if (!mbar_wait(empty_c(sc), ((it / p.nc) & 1) ^ 1, abort_flag, p.status, 6)) goto done_codes;
          mbar_expect_tx(full_c(sc), kCodeStage);
          tma_load_2d(base + c_off + sc * kCodeStage, &cmap, ks * kCodeRow, n0 + (int)rank * 128, full_c(sc));
        }
      }
    done_codes:;
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {
      // ---------------- MMA issuer (even CTA) ----------------
      const uint32_t peer = map_to_cta(bars, 1) - bars;  // same barrier, odd CTA
      const uint32_t peer_acc_full = acc_full + peer;
      int it = 0, tcount = 0;
      for (int unit = pair; unit < n_tiles && !*abort_flag; unit += n_pairs, ++tcount) {
        int split, ks0, ks1;
        const int tile = unit_of(unit, split, ks0, ks1);
        const int m0 = (tile % p.tiles_m) * kPairTileM;
        const bool two = m0 + 256 < p.M;
        if (tcount > 0 && !mbar_wait_cluster(acc_empty, (tcount - 1) & 1, abort_flag, p.status, 9)) goto done_mma;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int ks = ks0; ks < ks1; ++ks, ++it) {
          const int sx = it % kPairXStages, sw = it % kPairWStages;
          if (!mbar_wait_cluster(full_x(sx), (it / kPairXStages) & 1, abort_flag, p.status, 2)) goto done_mma;
          if (!mbar_wait_cluster(full_w(sw), (it / kPairWStages) & 1, abort_flag, p.status, 3)) goto done_mma;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t xa = base + sx * kXStage, wb = base + kWOff + sw * kPairWTileBytes;
#pragma unroll
          for (int kk = 0; kk < kStepK / 16; ++kk) {
            const uint64_t db = smem_desc_sw128(wb + kk * 32);
            const uint32_t acc = (ks > ks0 || kk > 0) ? 1u : 0u;
            umma_pair_bf16(tmem, smem_desc_sw128(xa + kk * 32), db, kIdescPair, acc);
            if (two) umma_pair_bf16(tmem + 256, smem_desc_sw128(xa + kXTileBytes + kk * 32), db, kIdescPair, acc);
          }
          umma_pair_commit(empty_x(sx));
          umma_pair_commit(empty_x(sx) + peer);
          umma_pair_commit(empty_w(sw));
          umma_pair_commit(empty_w(sw) + peer);
        }
        umma_pair_commit(acc_full);
        umma_pair_commit(peer_acc_full);
      }
    done_mma:;
    }
  } else {
    // ---------------- decode + epilogue warps ----------------
    // A warp's trip through one K step is a chain of barrier round trips (codes full, weight stage empty,
    // proxy fence, arrival) that costs more than the MMAs of the step, however little it decodes.  So the 16
    // warps form four groups and group g takes the steps with it % 4 == g, a whole 128-row stage each
    // (thread = one weight row, all 64 K elements): four steps are in the decode pipeline at a time.
    const int d = tid - 64;
    const int r = d & 127, g = d >> 7;
    const bool regtab = PACKED && p.n_levels <= 8;  // nibble codes below 8: a valid byte-permute selector
    const RegTable tb = regtab ? bf16_reg_table(p.ct, p.n_levels) : RegTable{0, 0, 0, 0};
    // nibble layers: lanes l and l + 16 share a copy of the table (a two-way bank conflict when their
    // entries differ but have the same parity; the decode warps have the time)
    const uint32_t lane_base = lut_s + (uint32_t)(lane * 4 & (kLutStride - 1));
    const int q = warp & 3;
    const int grp = (warp - 2) >> 2;
    const int half = grp & 1;
    const int chalf = grp >> 1;
    const uint32_t wrow = (uint32_t)((r >> 3) * 1024 + (r & 7) * 128);
    const int sw7 = r & 7;
    const uint32_t lead = map_to_cta(bars, 0) - bars;
    int it = 0, tcount = 0, stg_phase = 0;
    for (int unit = pair; unit < n_tiles && !*abort_flag; unit += n_pairs, ++tcount) {
      int split, ks0, ks1;
      const int tile = unit_of(unit, split, ks0, ks1);
      const int m0 = (tile % p.tiles_m) * kPairTileM, n0 = (tile / p.tiles_m) * kTileN;
      const bool two = m0 + 256 < p.M;
      // where this unit's result goes: the output, or (K split) the fp32 partial of its K range
      const bool whole = split < 0;
      const int64_t part_ld = p.N - p.col0;
      void* const y_ptr = whole ? p.y : static_cast<void*>(p.part + (int64_t)split * p.M * part_ld - p.col0);
      const int y_dt = whole ? p.y_dtype : (int)PE_F32;
      const int64_t y_ld = whole ? p.ld_y : part_ld;
      const __half* const bias_ptr = whole ? p.bias : nullptr;
      const bool tma_out = whole ? p.y_tma : p.part_tma;
      int row = n0 + (int)rank * 128 + r;
      const bool row_ok = row < p.N;
      if (!row_ok) row = p.N - 1;
      const unsigned short* nrow = reinterpret_cast<const unsigned short*>(p.norms + (int64_t)row * p.ld_norms);
      bool dead = false;
      for (int ks = ks0; ks < ks1; ++ks, ++it) {
        if ((it & (kPairGroups - 1)) != g) continue;  // warp-uniform
        const float nf = row_ok ? __half2float(__ushort_as_half(__ldg(nrow + (ks >> 1)))) : 0.f;  // in flight across the waits
        const int sc = it % p.nc;
        {
          const bool ok = mbar_wait(full_c(sc), (it / p.nc) & 1, abort_flag, p.status, 7);
          if (!__all_sync(0xffffffffu, ok)) { dead = true; break; }
        }
        constexpr int CW = PACKED ? 2 : 4;  // 16-byte pieces of this row's codes
        uint4 c[CW];
        const uint8_t* csrc = sm + c_off + sc * kCodeStage + r * kCodeRow;
#pragma unroll
        for (int i = 0; i < CW; ++i) c[i] = *reinterpret_cast<const uint4*>(csrc + 16 * i);
        // The stage is handed back (and refilled at once by the code producer) only after the loads have
        // DELIVERED: a store that consumes every loaded register sits between them and the arrival.  Without
        // it rows of byte codes (64-byte row pitch, four-way bank conflicts) were overwritten before they were read.
        {
          uint32_t seen = 0;
#pragma unroll
          for (int i = 0; i < CW; ++i) seen |= c[i].x | c[i].y | c[i].z | c[i].w;
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(bars + 224), "r"(seen) : "memory");
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_c(sc));
        const uint32_t n2 = pack_bf16(nf, nf);
        const int sw = it % kPairWStages;
        {
          const bool ok = mbar_wait(empty_w(sw), ((it / kPairWStages) & 1) ^ 1, abort_flag, p.status, 4);
          if (!__all_sync(0xffffffffu, ok)) { dead = true; break; }
        }
        uint8_t* wt = sm + kWOff + sw * kPairWTileBytes + wrow;
#pragma unroll
        for (int i = 0; i < CW; ++i) {
          const uint32_t wq[4] = {c[i].x, c[i].y, c[i].z, c[i].w};
          if (PACKED) {  // one code byte -> two adjacent K elements; word j of piece i -> chunk 4 i + j
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t w = wq[j];
              uint4 o;
              if (regtab) {
                uint32_t a[4];
                reg_decode(w, tb, a);
                o.x = bf16x2_mul(a[0], n2); o.y = bf16x2_mul(a[1], n2); o.z = bf16x2_mul(a[2], n2); o.w = bf16x2_mul(a[3], n2);
              } else {
                o.x = bf16x2_mul(glut_s<0, kLutStride>(w, lane_base), n2);
                o.y = bf16x2_mul(glut_s<1, kLutStride>(w, lane_base), n2);
                o.z = bf16x2_mul(glut_s<2, kLutStride>(w, lane_base), n2);
                o.w = bf16x2_mul(glut_s<3, kLutStride>(w, lane_base), n2);
              }
              *reinterpret_cast<uint4*>(wt + (((4 * i + j) ^ sw7) << 4)) = o;
            }
          } else {       // one code byte -> one K element; words 2j, 2j+1 of piece i -> chunk 2 i + j
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint32_t wa = wq[2 * j], wb = wq[2 * j + 1];
              uint4 o;
              o.x = bf16x2_mul(lo_hi16(glut_s<0, kLutStride>(wa, lane_base), glut_s<1, kLutStride>(wa, lane_base)), n2);
              o.y = bf16x2_mul(lo_hi16(glut_s<2, kLutStride>(wa, lane_base), glut_s<3, kLutStride>(wa, lane_base)), n2);
              o.z = bf16x2_mul(lo_hi16(glut_s<0, kLutStride>(wb, lane_base), glut_s<1, kLutStride>(wb, lane_base)), n2);
              o.w = bf16x2_mul(lo_hi16(glut_s<2, kLutStride>(wb, lane_base), glut_s<3, kLutStride>(wb, lane_base)), n2);
              *reinterpret_cast<uint4*>(wt + (((2 * i + j) ^ sw7) << 4)) = o;
            }
          }
        }
        // visible to the tensor core of this SM, then one arrival per warp on the even CTA's barrier
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (leader) mbar_arrive(full_w(sw));
          else mbar_arrive_remote(full_w(sw) + lead);
        }
      }
      if (dead) break;
      // ---------------- epilogue: this CTA's 128 token rows of both accumulators ----------------
      asm volatile("griddepcontrol.wait;" ::: "memory");
      {
        const bool ok = mbar_wait_cluster(acc_full, tcount & 1, abort_flag, p.status, 5);
        if (!__all_sync(0xffffffffu, ok)) break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tma_out && y_dt == PE_F32) {
        // as below with 32 rows x 32 columns of fp32 (4 KB, 128-byte swizzle) per warp: the output, or the partial of a K range
        const uint32_t stg = base + kWOff + (uint32_t)(warp - 2) * 4096u;
        const int swz = lane & 7;
        if (half == 0 || two) {
          const int mrow0 = m0 + half * 256 + (int)rank * 128 + q * 32;
          const uint32_t trow = tmem + half * 256 + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
          for (int cc = chalf * 4; cc < chalf * 4 + 4; ++cc) {
            uint32_t rr[32];
            tmem_ld32(trow + cc * 32, rr);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int nb0 = n0 + cc * 32;
            if (bias_ptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (nb0 + j < p.N) rr[j] = __float_as_uint(__uint_as_float(rr[j]) + __half2float(bias_ptr[nb0 + j]));
            }
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the previous store has read the buffer
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(stg + (uint32_t)lane * 128u + (uint32_t)((j ^ swz) << 4)), "r"(rr[4 * j]),
                           "r"(rr[4 * j + 1]), "r"(rr[4 * j + 2]), "r"(rr[4 * j + 3]) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && mrow0 < p.M && nb0 < p.N) {
              asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                           ::"l"(whole ? &ymap : &partmap), "r"(stg), "r"(whole ? nb0 : nb0 - p.col0), "r"(mrow0), "r"(whole ? 0 : split) : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          }
        }
      } else if (tma_out) {
        // 16-bit output: every warp stages its 32 rows x 32 columns (2 KB, 64-byte swizzle) in its own piece of the
        // weight stages -- idle now: all MMAs are done and no warp decodes before the staging barrier below -- and one
        // lane sends it off as a TMA store, which writes whole 64-byte row pieces and clips at the matrix edges.
        // Per-lane 16-byte stores straight to global memory, 32 rows per instruction, took a quarter of the kernel.
        const uint32_t stg = base + kWOff + (uint32_t)(warp - 2) * 2048u + (uint32_t)lane * 64u;
        const int swz = (lane >> 1) & 3;
        if (half == 0 || two) {
          const int mrow0 = m0 + half * 256 + (int)rank * 128 + q * 32;
          const uint32_t trow = tmem + half * 256 + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
          for (int cc = chalf * 4; cc < chalf * 4 + 4; ++cc) {
            uint32_t rr[32];
            tmem_ld32(trow + cc * 32, rr);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int nb0 = n0 + cc * 32;
            uint32_t o[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float a = __uint_as_float(rr[2 * j]), b = __uint_as_float(rr[2 * j + 1]);
              if (p.bias) {
                if (nb0 + 2 * j < p.N) a += __half2float(p.bias[nb0 + 2 * j]);
                if (nb0 + 2 * j + 1 < p.N) b += __half2float(p.bias[nb0 + 2 * j + 1]);
              }
              o[j] = p.y_dtype == PE_F16 ? pack_half2(a, b) : pack_bf16(a, b);
            }
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the previous store has read the buffer
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(stg + (uint32_t)((j ^ swz) << 4)), "r"(o[4 * j]),
                           "r"(o[4 * j + 1]), "r"(o[4 * j + 2]), "r"(o[4 * j + 3]) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && mrow0 < p.M && nb0 < p.N) {
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                           ::"l"(&ymap), "r"(stg), "r"(nb0), "r"(mrow0) : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          }
        }
      } else {
      if (half == 0 || two) {
        const int m = m0 + half * 256 + (int)rank * 128 + q * 32 + lane;
        const uint32_t trow = tmem + half * 256 + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
        for (int cc = chalf * 4; cc < chalf * 4 + 4; ++cc) {
          uint32_t rr[32];
          tmem_ld32(trow + cc * 32, rr);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const int nb0 = n0 + cc * 32;
          if (m < p.M && nb0 < p.N) {
            const bool full = nb0 + 32 <= p.N && (y_ld % 8 == 0) && ((reinterpret_cast<uintptr_t>(y_ptr) & 15) == 0);
            if (full && y_dt != PE_F32) {
              uint32_t o[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                float a = __uint_as_float(rr[2 * j]), b = __uint_as_float(rr[2 * j + 1]);
                if (bias_ptr) { a += __half2float(bias_ptr[nb0 + 2 * j]); b += __half2float(bias_ptr[nb0 + 2 * j + 1]); }
                o[j] = y_dt == PE_F16 ? pack_half2(a, b) : pack_bf16(a, b);
              }
              uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(y_ptr) + (int64_t)m * y_ld + nb0);
#pragma unroll
              for (int j = 0; j < 4; ++j) dst[j] = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
            } else if (y_dt == PE_F32 && nb0 + 32 <= p.N && (y_ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(y_ptr) & 15) == 0)) {
              float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(y_ptr) + (int64_t)m * y_ld + nb0);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float4 v = make_float4(__uint_as_float(rr[4 * j]), __uint_as_float(rr[4 * j + 1]), __uint_as_float(rr[4 * j + 2]),
                                       __uint_as_float(rr[4 * j + 3]));
                if (bias_ptr) {
                  v.x += __half2float(bias_ptr[nb0 + 4 * j]); v.y += __half2float(bias_ptr[nb0 + 4 * j + 1]);
                  v.z += __half2float(bias_ptr[nb0 + 4 * j + 2]); v.w += __half2float(bias_ptr[nb0 + 4 * j + 3]);
                }
                dst[j] = v;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (nb0 + j < p.N) {
                  float a = __uint_as_float(rr[j]);
                  if (bias_ptr) a += __half2float(bias_ptr[nb0 + j]);
                  store_from_float(y_ptr, y_dt, (int64_t)m * y_ld + nb0 + j, a);
                }
              }
            }
          }
        }
      }
      }
      // the next tile's first MMA overwrites the accumulators: it waits for every decode warp of the pair
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (leader) mbar_arrive(acc_empty);
        else mbar_arrive_remote(acc_empty + lead);
      }
      if (tma_out) {
        // no warp writes a weight stage of the next tile before every warp's staging has been read
        if (lane == 0) {
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          mbar_arrive(stg_free);
        }
        const bool ok = mbar_wait(stg_free, stg_phase, abort_flag, p.status, 10);
        stg_phase ^= 1;
        if (!__all_sync(0xffffffffu, ok)) break;
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // stores complete before the CTA leaves
  }

  // ---------------- common exit: nobody leaves while the other CTA may still signal or read here ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag && tid == 0) {
    const long long t0 = clock64();
    while (clock64() - t0 < 200000) {}
  }
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

PE_WAIT_STATUS_READER(gemm_wait_status)

}  // namespace pe

using namespace pe;

// Up to 256 rows: one activation tile.  Tiles of 128 weight rows spread a small layer over more SMs and need fewer K
// ranges; with more of them than SMs, tiles of 256 rows read the activations half as often (their two accumulators and
// the weight stages leave room for 192 tokens).
static int small_halves(int m, int out_f, int sms) { return m <= 192 && (out_f + 127) / 128 > sms ? 2 : 1; }

// K ranges per tile: as many as there are idle SMs, at least two blocks each.
static int small_ksplit(int m, int out_f, int in_f_padded, int sms) {
  const int rows = 128 * small_halves(m, out_f, sms);
  int s = sms / ((out_f + rows - 1) / rows);
  const int nb = in_f_padded / kBlock;
  if (s > nb / 2) s = nb / 2;
  return s < 2 ? 1 : s;
}

// Whole and split tiles of a launch over pairs of CTAs.  Fewer tiles than pairs: as many K ranges as there are idle
// pairs, at least eight K steps each; two ranges from 40 steps on (1024 x 4096 rows, K 4096: 58.4 us whole, 48.6 us split; at
// K 2048 the fp32 partials and their sum cost what halving the tile saves, 34.0 against 35.4 us).  More: the tiles of the
// last, partly filled wave (rounded up to whole columns of tiles, so that the partials are one matrix) are split over all
// pairs where that saves 15 steps of a tile's time or more (600 x 13312 rows, K 2048: 16 saved, 63.2 against 59.5 us;
// 4096 x 12288, K 4096, 5.2 waves: 382 against 368 us).
struct PairPlan { int full, ksplit, col0; };
static PairPlan pair_plan(int tiles_m, int tiles_n, int ksteps, int sms) {
  const int tiles = tiles_m * tiles_n, pairs = sms / 2;
  if (tiles <= pairs) {
    int ks = pairs / tiles;
    if (ks > ksteps / 8) ks = ksteps / 8;
    if (ks == 2 && ksteps < 40) ks = 1;
    return ks < 2 ? PairPlan{tiles, 1, 0} : PairPlan{0, ks, 0};
  }
  const int cols = (tiles % pairs + tiles_m - 1) / tiles_m, rest = cols * tiles_m;
  int ks = rest ? pairs / rest : 1;
  if (ks > ksteps / 8) ks = ksteps / 8;
  if (ks < 2 || ksteps * (ks - 1) < 15 * ks) return {tiles, 1, 0};
  return {tiles - rest, ks, (tiles_n - cols) * kTileN};
}

// ---- more than 256 rows: which kernel, which tiles ----------------------------------------------------------------
// A pair of CTAs does the work of a full 512 x 256 tile in 0.69 us per 64 of K, the tensor-memory kernel that of its four 256 x 128
// tiles in 1.4 on two CTAs; but 512 x 256 is a coarse tile: rows are rounded up to 512, and a launch of a few hundred rows has less
// than one or just over one wave of them.  So the time of both is estimated, for every tiling that the tensor-memory kernel
// has, and the shorter one taken.  The constants are a fit to 590 launches of nine layer shapes at 24 to 2048 rows.  Over twelve
// shapes at 51 row counts to 2049 the estimated ratio of the two is 6 % off on average and 25 % at worst, and that worst is at short K,
// where the drain of the tiles, of which the estimate knows little, counts most (16384 x 1280 Q6 at 1280 rows: 0.94 estimated,
// 77.0 against 67.1 us); so a tiling has to be ahead by 10 % below K 2048 and by 5 % from there on, and by 10 % more above 1600 rows,
// where both have several waves (4096 x 12288 Q4 at 1856 rows: 0.93 estimated, 188 against 172 us).  What that picks of the launches
// measured is never slower than the pair kernel by more than the noise (2048 x 7168 Q6 at 1024 rows, 47.0 and 46.8 us); above
// 1600 rows it is 104 of 348, 17 % faster on average.  Not measured and not asked above 4096 rows.
// Pair / this, us, weights from HBM: 4096 x 4096 Q6 at 257 rows 30.2 / 23.7, 384: 32.1 / 28.0, 640: 45.7 / 32.9, 1024: 50.0 / 38.1; 24576 x
// 4096 Q3 at 257 rows 84.0 / 68.7, 640: 161.7 / 107.0; 4096 x 12288 Q4 at 257 rows 59.2 / 43.9, 384: 57.1 / 49.8, 640: 92.4 / 67.9; 12288 x 4096
// Q4 at 512 rows 57.7 / 47.5, 1700: 190 / 151; 2560 x 2560 Q5 at 512 rows 26.1 / 19.5, 1700: 43.2 / 28.7; 2048 x 7168 Q6 at 2112 rows 104.5 / 65.6.
//
// Order of the sums.  Both kernels multiply the same values and add them in the same order within a K range, so a tiling with the pair
// kernel's K ranges gives its bits.  Other K ranges are another order: as far from 64-bit arithmetic, but six decoder layers
// turn another order of q/k/v alone (6144 x 4096 Q5: one range for three) into 1.0 to 1.1 % of the logits.  Up to one row of pair tiles,
// another order is therefore taken only where a quarter of the time goes (0.76 by the estimate; q/k/v stays above that but at
// 432 rows, 0.7597).  What that leaves: q/k/v at 512 rows 41.1 us where 34.0 would do, 24576 x 4096 Q3 at 384 rows 95.6 (73.3), 2560 x 2560
// Q5 at 433 rows 25.1 (18.7; 432 rows, 0.746, take it), 2048 x 7168 Q6 at 384 rows 31.1 (23.1).
constexpr int kTmemMaxRows = 4096;

static PairPlan pair_plan_within(int m, int out_f, int in_f_padded, int sms, size_t part_bytes) {
  const int tiles_m = (m + kPairTileM - 1) / kPairTileM, tiles_n = (out_f + kTileN - 1) / kTileN;
  const PairPlan p = pair_plan(tiles_m, tiles_n, in_f_padded / kStepK, sms);
  return p.ksplit > 1 && (size_t)p.ksplit * m * (out_f - p.col0) * sizeof(float) > part_bytes ? PairPlan{tiles_m * tiles_n, 1, 0} : p;
}

static double pair_time_us(const PairPlan& p, int m, int out_f, int in_f_padded, int sms) {
  const int steps = in_f_padded / kStepK, pairs = sms / 2;
  double t = 7.8 + 1.26e-6 * m * in_f_padded;  // launch and preparation
  if (p.full) t += (p.full + pairs - 1) / pairs * (0.69 * steps + 7.1);
  if (p.ksplit > 1) t += (steps + p.ksplit - 1) / p.ksplit * 0.69 + 7.4 + 1.0e-6 * p.ksplit * m * (out_f - p.col0);
  return t;
}

// Does a cut of every tile's nb blocks into `ksplit` ranges give the ranges that p gives them?  (p's are ranges of half blocks.)
static bool same_ranges(const PairPlan& p, int ksplit, int nb) {
  if (ksplit != p.ksplit || (ksplit > 1 && p.full)) return false;
  for (int s = 1; s < ksplit; ++s)
    if (s * 2 * nb / ksplit != s * nb / ksplit * 2) return false;
  return true;
}

struct TmemPlan { int halves, tiles_m, tok, ksplit; };
static double tmem_time_us(const TmemPlan& p, int m, int out_f, int in_f_padded, int packed, int sms) {
  const int nb = in_f_padded / kBlock, tiles_n = (out_f + 128 * p.halves - 1) / (128 * p.halves);
  const int units = p.tiles_m * tiles_n * p.ksplit, waves = (units + sms - 1) / sms, steps = 2 * ((nb + p.ksplit - 1) / p.ksplit);
  // a step of 128 weight rows: MMAs, or the decode (of tiles of one half by two of the four groups at a time); or the bytes of a step
  double half = 127 + 0.92 * p.tok;
  if (!packed && half < 285) half = 285;
  if (p.halves == 1 && half < 259) half = 259;
  const double bytes = 128.0 * p.tok + p.halves * (packed ? 4096 : 8192), step = p.halves * half > bytes * 0.0108 ? p.halves * half : bytes * 0.0108;
  double unit = steps * step + 1740;  // ns
  if (p.halves * p.tok > 192) unit += 4.5 * p.tok * p.halves;  // the accumulators fill tensor memory: the drain is not hidden
  double t = 9.0 + 0.95e-6 * m * in_f_padded + waves * unit * 1e-3;
  if (p.ksplit > 1) t += 1.5 + 0.71e-6 * p.ksplit * m * out_f;
  return t;
}

// Shortest tiling of the tensor-memory kernel whose partials fit part_bytes; halves = 0: the pair kernel.
static TmemPlan many_rows_plan(int m, int out_f, int in_f_padded, int packed, int sms, size_t part_bytes) {
  TmemPlan best = {0, 0, 0, 1};
  if (m > kTmemMaxRows) return best;
  const int nb = in_f_padded / kBlock;
  const PairPlan pairs = pair_plan_within(m, out_f, in_f_padded, sms, part_bytes);
  const double pair = pair_time_us(pairs, m, out_f, in_f_padded, sms), margin = (in_f_padded < 2048 ? 0.9 : 0.95) - (m > 1600 ? 0.1 : 0);
  const double same = margin * pair, other = m <= kPairTileM ? 0.76 * pair : same;
  double least = same;
  for (int halves = 1; halves <= 2; ++halves) {
    const int most = halves == 1 ? 256 : 192, tiles_n = (out_f + 128 * halves - 1) / (128 * halves), first = (m + most - 1) / most;
    for (int tiles_m = first; tiles_m < first + 3; ++tiles_m) {
      TmemPlan p = {halves, tiles_m, ((m + tiles_m - 1) / tiles_m + 15) / 16 * 16, 1};
      p.tiles_m = (m + p.tok - 1) / p.tok;  // the rounded tiles may be one fewer: none is empty
      int idle = sms / (tiles_n * p.tiles_m);
      if (idle > nb / 2) idle = nb / 2;
      const int splits[3] = {1, idle, m <= kPairTileM ? pairs.ksplit : 1};  // whole, as many as there are idle SMs, as the pair kernel's
      for (int i = 0; i < 3; ++i) {
        p.ksplit = splits[i];
        if (i && (p.ksplit < 2 || (size_t)p.ksplit * m * out_f * sizeof(float) > part_bytes)) continue;
        const double t = tmem_time_us(p, m, out_f, in_f_padded, packed, sms);
        if (t < least && (t < other || same_ranges(pairs, p.ksplit, nb))) { least = t; best = p; }
      }
    }
  }
  return best;
}

// workspace: [status word, padded to 256 B][bf16 activations M x K]
extern "C" size_t pe_gemm_workspace_bytes(int m, int in_f_padded) {
  if (m < 1 || in_f_padded < kBlock || in_f_padded % kBlock) return 0;
  return 256 + (size_t)m * in_f_padded * 2;
}

// [the above][fp32 partials ksplit x M x N]: with this much room launches split K as they would like to
extern "C" size_t pe_gemm_workspace_bytes_splitk(int m, int out_f, int in_f_padded) {
  const size_t base = pe_gemm_workspace_bytes(m, in_f_padded);
  if (base == 0 || out_f < 1) return 0;
  const int sms = sm_count();
  if (sms < 2) return base;
  size_t floats = 0;
  auto want = [&](int ks, int cols) {
    const size_t f = ks > 1 ? (size_t)ks * m * cols : 0;
    if (f > floats) floats = f;
  };
  if (m <= 256) {
    want(small_ksplit(m, out_f, in_f_padded, sms), out_f);
  } else {
    const PairPlan p = pair_plan_within(m, out_f, in_f_padded, sms, ~(size_t)0);
    want(p.ksplit, out_f - p.col0);
    for (int packed = 0; packed < 2; ++packed) want(many_rows_plan(m, out_f, in_f_padded, packed, sms, ~(size_t)0).ksplit, out_f);
  }
  return floats ? ((base + 255) & ~(size_t)255) + floats * sizeof(float) : base;
}

extern "C" int pe_gemm(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                       const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype, int64_t ld_x,
                       int in_f, void* y, int y_dtype, int64_t ld_y, const void* bias, int m, int out_f, int in_f_padded,
                       void* workspace, size_t workspace_bytes, void* stream) {
  if (!codes || !norms || !ct_scaled || !x || !y || !workspace) return PE_ERR_ARG;
  if (m < 1 || out_f < 1 || in_f < 1 || in_f > in_f_padded) return PE_ERR_ARG;
  if (x_kind != PE_X_ROTATED && x_kind != PE_X_RAW && !(x_kind == PE_X_SILU_MUL && x_dtype == PE_F16)) return PE_ERR_ARG;
  if (x_dtype < PE_F32 || x_dtype > PE_BF16 || y_dtype < PE_F32 || y_dtype > PE_BF16) return PE_ERR_ARG;
  if (n_levels < 2 || n_levels > 256 || (packed && n_levels > 16)) return PE_ERR_ARG;
  if (in_f_padded % kBlock) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15)) return PE_ERR_ALIGN;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return PE_ERR_ALIGN;
  if (workspace_bytes < pe_gemm_workspace_bytes(m, in_f_padded)) return PE_ERR_WORKSPACE;
  if (ld_codes < (packed ? in_f_padded / 2 : in_f_padded) || ld_norms < in_f_padded / kBlock) return PE_ERR_ARG;
  if (ld_x < (x_kind == PE_X_RAW ? in_f : x_kind == PE_X_SILU_MUL ? 2 * (int64_t)in_f : in_f_padded) || ld_y < out_f) return PE_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int sms = sm_count();
  if (sms <= 0) return PE_ERR_CUDA;

  int* status = static_cast<int*>(workspace);
  uint8_t* xq = static_cast<uint8_t*>(workspace) + 256;
  int rc = launch_gemm_prep(x, x_kind, x_dtype, ld_x, in_f, xq, m, in_f_padded, packed ? 1 : 0, nullptr, nullptr, nullptr, 0, status, st);
  if (rc != PE_OK) return rc;
  // few tiles: split K when the caller's workspace has room for the partials
  const size_t part_off = (pe_gemm_workspace_bytes(m, in_f_padded) + 255) & ~(size_t)255;
  const size_t part_bytes = workspace_bytes > part_off ? workspace_bytes - part_off : 0;
  float* part = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + part_off);

  // Up to 256 rows: one tile of tokens of the tensor-memory kernel.  Above, as many_rows_plan says.
  TmemPlan plan = {small_halves(m, out_f, sms), 1, m, 1};
  if (m > 256) plan = many_rows_plan(m, out_f, in_f_padded, packed, sms, part_bytes);
  else plan.ksplit = small_ksplit(m, out_f, in_f_padded, sms);
  if ((size_t)plan.ksplit * m * out_f * sizeof(float) > part_bytes) plan.ksplit = 1;
  if (plan.halves) {
    TmemGemmArgs a = {};
    a.norms = static_cast<const __half*>(norms); a.ld_norms = ld_norms;
    a.ct = ct_scaled; a.n_levels = n_levels;
    a.y = y; a.y_dtype = y_dtype; a.ld_y = ld_y;
    a.bias = static_cast<const __half*>(bias);
    a.M = m; a.N = out_f; a.nb = in_f_padded / kBlock;
    a.halves = plan.halves;
    a.tiles_m = plan.tiles_m; a.tok = plan.tok;
    a.tiles_n = (out_f + 128 * a.halves - 1) / (128 * a.halves);
    a.ksplit = plan.ksplit;
    a.part = a.ksplit > 1 ? part : nullptr;
    a.xbox = (a.tok + 15) & ~15;
    a.x_stage = a.xbox * 128;
    a.status = status;
    rc = launch_gemm_tmem(a, codes, packed, ld_codes, out_f, xq, m, a.tiles_m * a.tiles_n * a.ksplit, sms, st);
    if (rc != PE_OK || a.ksplit == 1) return rc;
    return launch_splitk_reduce(part, a.ksplit, m, out_f, bias, y, y_dtype, ld_y, sms, st);
  }

  CUtensorMap map, pmap;
  const int code_row = packed ? 32 : 64;
  rc = encode_map_2d(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, xq, in_f_padded, m, (uint64_t)in_f_padded * 2, kStepK, 128, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (rc == PE_OK)  // codes as a 2-D byte tensor (row stride ld_codes), boxes of 128 rows x one K step
    rc = encode_map_2d(&pmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, codes, packed ? in_f_padded / 2 : in_f_padded, out_f, ld_codes, code_row, 128,
                       CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  CUtensorMap ymap = pmap;  // a valid map also when the kernel does not use it
  const bool y_tma = ld_y % (y_dtype == PE_F32 ? 4 : 8) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
  if (rc == PE_OK && y_tma && y_dtype == PE_F32)
    rc = encode_map_f32(&ymap, y, out_f, m, 1, (uint64_t)ld_y * 4);
  else if (rc == PE_OK && y_tma)
    rc = encode_map_2d(&ymap, CU_TENSOR_MAP_DATA_TYPE_UINT16, y, out_f, m, (uint64_t)ld_y * 2, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B,
                       CU_TENSOR_MAP_L2_PROMOTION_NONE);
  if (rc != PE_OK) return rc;

  GemmArgs a = {};
  a.norms = static_cast<const __half*>(norms); a.ld_norms = ld_norms;
  a.ct = ct_scaled; a.n_levels = n_levels;
  a.y = y; a.y_dtype = y_dtype; a.ld_y = ld_y;
  a.bias = static_cast<const __half*>(bias);
  a.M = m; a.N = out_f; a.K = in_f_padded;
  a.tiles_m = (m + kPairTileM - 1) / kPairTileM;
  a.tiles_n = (out_f + kTileN - 1) / kTileN;
  a.status = status;
  a.y_tma = y_tma ? 1 : 0;
  a.lut_bytes = packed ? 256 * kPairLutStride : n_levels * 128;
  a.nc = kPairCodeStages;
  const unsigned smem_bytes = (packed ? 4 : 3) * 2 * kXTileBytes + kPairWStages * kPairWTileBytes + a.lut_bytes + a.nc * 128 * code_row + 256 + 1024;
  const PairPlan pairs_of = pair_plan_within(m, out_f, in_f_padded, sms, part_bytes);
  const int tiles = a.tiles_m * a.tiles_n;
  a.full = pairs_of.full; a.ksplit = pairs_of.ksplit; a.col0 = pairs_of.col0;
  a.part = part;
  CUtensorMap partmap = ymap;
  a.part_tma = pairs_of.ksplit > 1 && (out_f - pairs_of.col0) % 4 == 0;
  if (a.part_tma && (rc = encode_map_f32(&partmap, part, out_f - pairs_of.col0, m, pairs_of.ksplit, (uint64_t)(out_f - pairs_of.col0) * 4)) != PE_OK) return rc;
  const int units = pairs_of.full + (tiles - pairs_of.full) * pairs_of.ksplit, pairs = units < sms / 2 ? units : sms / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  auto kfn = packed ? gemm_pair_kernel<true> : gemm_pair_kernel<false>;
  PE_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
  PE_CUDA_TRY(cudaLaunchKernelEx(&cfg, kfn, a, map, pmap, ymap, partmap));
  if (pairs_of.ksplit == 1) return PE_OK;
  const int c0 = pairs_of.col0;
  return launch_splitk_reduce(part, pairs_of.ksplit, m, out_f - c0, bias ? static_cast<const __half*>(bias) + c0 : nullptr,
                              static_cast<uint8_t*>(y) + (int64_t)c0 * (y_dtype == PE_F32 ? 4 : 2), y_dtype, ld_y, sms, st);
}
