// Glue ops of a decoder layer around the quantized projections: residual add + RMSNorm,
// rotary embedding + KV-cache write, SiLU * up.  They exist so that the end-to-end decode
// measurement is not dominated by dozens of tiny framework kernels; in a vLLM deployment
// the server's own fused ops play this role.  fp16 activations, fp32 arithmetic, results
// rounded where the op-by-op torch formulation rounds.
#include "pe_common.cuh"

namespace pe {

constexpr int kNormThreads = 256;
constexpr int kNormMaxIter = 8;  // hidden <= 256 threads x 8 elements x 8 iterations = 16384

// x[row] += half(delta[row]) (if delta), out[row] = half(x * rsqrt(mean(x^2) + eps)) * w.  One block per row, ITERS x 8
// elements per thread.  Bounded by memory latency: everything a row reads is requested before any of it is used.  (The
// store of the updated row between the loads of a loop kept the next iteration's loads behind it: 512 rows of 4096 with
// an fp32 delta took 9.4 us with the wait for the launch in front, 7.2 us now.)
template <int ITERS>
__global__ void __launch_bounds__(kNormThreads) add_rmsnorm_kernel(__half* x, const void* delta, int delta_dtype, const __half* w,
                                                                   __half* out, int hidden, float eps) {
  __shared__ float warp_sums[kNormThreads / 32];
  const int row = blockIdx.x, tid = threadIdx.x;
  pdl_enter();
  __half* xr = x + (int64_t)row * hidden;
  uint4 xv[ITERS], dv[ITERS][2], wv[ITERS];
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int col = (it * kNormThreads + tid) * 8;
    if (col >= hidden) continue;
    xv[it] = *reinterpret_cast<const uint4*>(xr + col);
    if (delta && delta_dtype == PE_F32) {
      const uint4* src = reinterpret_cast<const uint4*>(static_cast<const float*>(delta) + (int64_t)row * hidden + col);
      dv[it][0] = src[0];
      dv[it][1] = src[1];
    } else if (delta) {
      dv[it][0] = *reinterpret_cast<const uint4*>(static_cast<const __half*>(delta) + (int64_t)row * hidden + col);
    }
    wv[it] = *reinterpret_cast<const uint4*>(w + col);
  }
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int col = (it * kNormThreads + tid) * 8;
    if (col >= hidden) continue;
    __half2* h = reinterpret_cast<__half2*>(&xv[it]);
    if (delta) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        __half2 d;  // the delta is rounded to fp16 first, then added in fp16 (round to nearest of the exact sum)
        if (delta_dtype == PE_F32) {
          const float* f = reinterpret_cast<const float*>(dv[it]);
          d = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
        } else {
          d = reinterpret_cast<const __half2*>(dv[it])[i];
        }
        const float2 a = __half22float2(h[i]), c = __half22float2(d);
        h[i] = __floats2half2_rn(a.x + c.x, a.y + c.y);
      }
      *reinterpret_cast<uint4*>(xr + col) = xv[it];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      ss += f.x * f.x;
      ss += f.y * f.y;
    }
  }
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
  if ((tid & 31) == 0) warp_sums[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) tot += warp_sums[i];
  const float scale = rsqrtf(tot / (float)hidden + eps);
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const int col = (it * kNormThreads + tid) * 8;
    if (col >= hidden) continue;
    const __half2 *h = reinterpret_cast<const __half2*>(&xv[it]), *w2 = reinterpret_cast<const __half2*>(&wv[it]);
    uint4 o;
    __half2* o2 = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      o2[i] = __hmul2(__floats2half2_rn(f.x * scale, f.y * scale), w2[i]);
    }
    *reinterpret_cast<uint4*>(out + (int64_t)row * hidden + col) = o;
  }
}

// One block per token: the angles' sines and cosines once, then every head's pairs (j, j + d/2) (rotate-half form), two
// eight neighbouring pairs per thread and step where the rows are aligned for 16-byte accesses.  (A block per head
// computed them anew for every head, in blocks of two warps: 26 us for 512 tokens of 48 heads, 7.5 us with one block
// per token and two pairs per step.)
// Query heads go to q_out (head stride q_head, token stride q_tok, a sequence after the other); key heads (rotated) and value heads (copied)
// go into the caches (batch, hkv, max_len, d) at position base + token index.
constexpr int kRopeThreads = 256;
constexpr int kRopeMaxHalf = 1024;  // head_dim <= 2048

__global__ void __launch_bounds__(kRopeThreads) rope_cache_kernel(const __half* qkv, int64_t ld_qkv, const int64_t* pos_dev, int64_t pos_host, __half* q_out,
                                  __half* k_cache, __half* v_cache, int t, int hq, int hkv, int d, int max_len,
                                  float theta, int64_t q_head, int64_t q_tok) {
  __shared__ float cs[kRopeMaxHalf], sn[kRopeMaxHalf];
  const int tok = blockIdx.x, b = tok / t, i = tok - b * t;
  const int half_d = d >> 1;
  pdl_enter();
  const int64_t pos = (pos_dev ? *pos_dev : pos_host) + i;
  for (int j = threadIdx.x; j < half_d; j += kRopeThreads) {
    const float inv = 1.f / powf(theta, (float)(2 * j) / (float)d);
    const float ang = (float)pos * inv;
    cs[j] = cosf(ang); sn[j] = sinf(ang);
  }
  __syncthreads();
  const bool room = pos >= 0 && pos < max_len;
  const __half* row = qkv + (int64_t)tok * ld_qkv;
  auto head_dst = [&](int head) -> __half* {  // null: dropped
    if (head < hq) return q_out + (int64_t)b * hq * t * d + head * q_head + i * q_tok;
    const bool key = head < hq + hkv;
    return room ? (key ? k_cache : v_cache) + (((int64_t)b * hkv + (head - hq - (key ? 0 : hkv))) * max_len + pos) * d : nullptr;
  };
  const uintptr_t all = reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_cache) |
                        reinterpret_cast<uintptr_t>(v_cache);
  if ((half_d & 7) == 0 && (ld_qkv & 7) == 0 && (all & 15) == 0) {
    const int per_head = half_d >> 3;
    for (int e = threadIdx.x; e < (hq + 2 * hkv) * per_head; e += kRopeThreads) {
      const int head = e / per_head, j = (e - head * per_head) * 8;
      __half* dst = head_dst(head);
      if (!dst) continue;
      const __half* src = row + (int64_t)head * d;
      uint4 a = *reinterpret_cast<const uint4*>(src + j), c = *reinterpret_cast<const uint4*>(src + j + half_d);
      if (head < hq + hkv) {
        __half2 *h1 = reinterpret_cast<__half2*>(&a), *h2 = reinterpret_cast<__half2*>(&c);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 x1 = __half22float2(h1[k]), x2 = __half22float2(h2[k]);
          const float2 co = *reinterpret_cast<const float2*>(cs + j + 2 * k), si = *reinterpret_cast<const float2*>(sn + j + 2 * k);
          h1[k] = __floats2half2_rn(x1.x * co.x - x2.x * si.x, x1.y * co.y - x2.y * si.y);
          h2[k] = __floats2half2_rn(x2.x * co.x + x1.x * si.x, x2.y * co.y + x1.y * si.y);
        }
      }
      *reinterpret_cast<uint4*>(dst + j) = a;
      *reinterpret_cast<uint4*>(dst + j + half_d) = c;
    }
    return;
  }
  // pairs of neighbours where every row is aligned for them
  const bool two = (half_d & 1) == 0 && (ld_qkv & 1) == 0 && (all & 3) == 0;
  const int step = two ? 2 : 1, per_head = half_d / step, items = (hq + 2 * hkv) * per_head;
  for (int e = threadIdx.x; e < items; e += kRopeThreads) {
    const int head = e / per_head, j = (e - head * per_head) * step;
    __half* dst = head_dst(head);
    if (!dst) continue;
    const __half* src = row + (int64_t)head * d;
    if (two) {
      const __half2 h1 = *reinterpret_cast<const __half2*>(src + j), h2 = *reinterpret_cast<const __half2*>(src + j + half_d);
      __half2 o1 = h1, o2 = h2;
      if (head < hq + hkv) {
        const float2 x1 = __half22float2(h1), x2 = __half22float2(h2);
        o1 = __floats2half2_rn(x1.x * cs[j] - x2.x * sn[j], x1.y * cs[j + 1] - x2.y * sn[j + 1]);
        o2 = __floats2half2_rn(x2.x * cs[j] + x1.x * sn[j], x2.y * cs[j + 1] + x1.y * sn[j + 1]);
      }
      *reinterpret_cast<__half2*>(dst + j) = o1;
      *reinterpret_cast<__half2*>(dst + j + half_d) = o2;
    } else {
      __half o1 = src[j], o2 = src[j + half_d];
      if (head < hq + hkv) {
        const float x1 = __half2float(o1), x2 = __half2float(o2);
        o1 = __float2half_rn(x1 * cs[j] - x2 * sn[j]);
        o2 = __float2half_rn(x2 * cs[j] + x1 * sn[j]);
      }
      dst[j] = o1;
      dst[j + half_d] = o2;
    }
  }
}

// out[r, i] = half(silu(gate)) * up in fp16, gate = gu[r, i], up = gu[r, inter + i]; 8 elements per thread
__global__ void __launch_bounds__(256) silu_mul_kernel(const __half* gu, int64_t ld_gu, __half* out, int64_t ld_out, int inter,
                                                       int64_t n_vec) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  pdl_enter();
  if (idx >= n_vec) return;
  const int per_row = inter >> 3;
  const int64_t r = idx / per_row;
  const int col = (int)(idx - r * per_row) * 8;
  const uint4 g = *reinterpret_cast<const uint4*>(gu + r * ld_gu + col);
  const uint4 u = *reinterpret_cast<const uint4*>(gu + r * ld_gu + inter + col);
  const __half2* g2 = reinterpret_cast<const __half2*>(&g);
  const __half2* u2 = reinterpret_cast<const __half2*>(&u);
  uint4 o;
  __half2* o2 = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(g2[i]);
    const __half2 s = __floats2half2_rn(f.x / (1.f + expf(-f.x)), f.y / (1.f + expf(-f.y)));
    o2[i] = __hmul2(s, u2[i]);
  }
  *reinterpret_cast<uint4*>(out + r * ld_out + col) = o;
}


// Single-query attention over the KV cache for one decode step (grouped-query form), optionally with the
// rotary embedding and the KV-cache write of the new token folded in.
// A cluster of up to eight CTAs per (kv head, sequence): the G = hq / hkv query heads of a kv head share every K and V
// row; the cache positions 0 .. L-1 are cut into equal ranges, one per CTA, so that a one-sequence step still spreads.
// The launch is a chain of memory round trips (position -> rows -> merge), so the point is to have few of them:
//  * Half a warp owns a position: its lane l holds elements 8l .. 8l+7, a K or V row is one 16-byte load per lane, and
//    the K and V rows of five positions are requested together -- a CTA's share of a 640-token cache in one trip.
//    Per position G dot products (four shuffles each) and an online-softmax update.
//  * The 16 half-warps meet in shared memory, the CTAs of the cluster through distributed shared memory: CTA r
//    finishes its share of the outputs from the eight records, in rank order (bit-reproducible).  No scratch, no
//    tickets: the exchange through global memory that this replaces was a store, a fence, an atomic and a load, a
//    memory round trip each (decode step of one token at 513 positions, 8 kv heads: 19.4 us after the projection in
//    front of it, 7.2 us now).
//  * Fused form (qkv != null): q, k, v are the raw rows of the fused q/k/v projection.  Every half-warp rotates
//    the G queries for itself (rotate-half pairs (j, j + 64) live in lanes l and l + 8); the CTA whose range
//    holds the current position rotates the new key, writes key and value into the caches and uses its
//    registers for that position instead of reading the row back.
constexpr int kAttThreads = 256;
constexpr int kAttGroups = kAttThreads / 16;  // half-warps
constexpr int kAttMaxCluster = 8;             // the portable cluster size
constexpr int kAttMaxGroup = 8;
constexpr int kAttMaxSplits = 16;             // records per head that the scratch of the many-sequences kernel is sized for
constexpr int kAttInFlight = 5;               // positions whose K and V rows a half-warp requests together

struct AttArgs {
  const __half* q;      // (batch, hq, D) rotated queries, or null in the fused form
  const __half* qkv; int64_t ld_qkv;  // fused form: rows of (hq + 2 hkv) * D raw projection outputs
  __half* k_cache; __half* v_cache;   // (batch, hkv, max_len, D); written at the current position in the fused form
  const int64_t* pos_dev; int64_t pos_host;
  __half* out;          // (batch, hq * D)
  int hq, hkv, max_len;
  float scale, theta;
};

__device__ __forceinline__ void half8_to_float(const uint4& u, float f[8]) {
  const uint32_t h[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
    f[2 * i] = a.x; f[2 * i + 1] = a.y;
  }
}

// rotate-half rotary embedding of the 8 elements a lane holds (elements 8l..8l+7; the pair partner is 64 away,
// in lane l ^ 8), rounded to fp16 as pe_rope_cache stores them
__device__ __forceinline__ void rope8(float x[8], const float c[8], const float s[8], int l) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float o = __shfl_xor_sync(0xffffffffu, x[i], 8);
    const float r = l < 8 ? x[i] * c[i] - o * s[i] : x[i] * c[i] + o * s[i];
    x[i] = __half2float(__float2half_rn(r));
  }
}

// value at the same place of another CTA's shared memory
__device__ __forceinline__ float cluster_load(const float* p, int rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int D, int G>
__device__ __forceinline__ void attention_body(const AttArgs& p, float* att_smem) {
  static_assert(D == 128, "a row is 16 lanes x 8 elements");
  __shared__ float rope_c[D / 2], rope_s[D / 2];  // computed once per CTA
  const int tid = threadIdx.x, l = tid & 15, grp = tid >> 4;
  const int sp = blockIdx.x, splits = gridDim.x, kvh = blockIdx.y, b = blockIdx.z;  // the cluster is the x extent
  const bool fused = p.qkv != nullptr;
  float inv = 0.f;
  if (fused && tid < D / 2) inv = 1.f / powf(p.theta, (float)(2 * tid) / (float)D);
  pdl_enter();
  const int64_t pos = p.pos_dev ? *p.pos_dev : p.pos_host;
  uint4 qraw[G], kraw = make_uint4(0, 0, 0, 0), vnew = kraw;
  const __half* qrow = fused ? p.qkv + (int64_t)b * p.ld_qkv : p.q + (int64_t)b * p.hq * D;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const uint2* src = reinterpret_cast<const uint2*>(qrow + ((int64_t)kvh * G + g) * D + l * 8);
    const uint2 lo = src[0], hi = src[1];
    qraw[g] = make_uint4(lo.x, lo.y, hi.x, hi.y);
  }
  if (fused) {
    const uint2* ks = reinterpret_cast<const uint2*>(qrow + ((int64_t)p.hq + kvh) * D + l * 8);
    const uint2* vs = reinterpret_cast<const uint2*>(qrow + ((int64_t)p.hq + p.hkv + kvh) * D + l * 8);
    const uint2 k0 = ks[0], k1 = ks[1], v0 = vs[0], v1 = vs[1];
    kraw = make_uint4(k0.x, k0.y, k1.x, k1.y);
    vnew = make_uint4(v0.x, v0.y, v1.x, v1.y);
  }
  const int64_t len64 = pos + 1;  // the current token counts
  const int L = (int)(len64 < 1 ? 1 : (len64 > p.max_len ? p.max_len : len64));
  const int chunk = (L + splits - 1) / splits;
  const int p_lo = sp * chunk, p_hi = p_lo + chunk < L ? p_lo + chunk : L;
  __half* kb = p.k_cache + ((int64_t)b * p.hkv + kvh) * (int64_t)p.max_len * D + l * 8;
  __half* vb = p.v_cache + ((int64_t)b * p.hkv + kvh) * (int64_t)p.max_len * D + l * 8;
  const int cur = fused && pos >= 0 && pos < p.max_len ? (int)pos : -1;  // position whose K/V rows come from qkv

  constexpr int U = kAttInFlight;
  uint4 kr[U], vr[U];
  auto request = [&](int p0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int pp = p0 + u * kAttGroups;
      kr[u] = vr[u] = make_uint4(0, 0, 0, 0);
      if (pp < p_hi && pp != cur) {
        kr[u] = *reinterpret_cast<const uint4*>(kb + (int64_t)pp * D);
        vr[u] = *reinterpret_cast<const uint4*>(vb + (int64_t)pp * D);
      }
    }
  };
  request(p_lo + grp);  // the first rows travel while the queries are prepared

  float q[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) half8_to_float(qraw[g], q[g]);
  if (fused) {
    if (tid < D / 2) {
      const float ang = (float)pos * inv;
      rope_c[tid] = cosf(ang);
      rope_s[tid] = sinf(ang);
    }
    __syncthreads();
    float c[8], s[8], k[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      c[i] = rope_c[(l & 7) * 8 + i];
      s[i] = rope_s[(l & 7) * 8 + i];
    }
#pragma unroll
    for (int g = 0; g < G; ++g) rope8(q[g], c, s, l);
    half8_to_float(kraw, k);
    rope8(k, c, s, l);
    kraw = make_uint4(pack_half2(k[0], k[1]), pack_half2(k[2], k[3]), pack_half2(k[4], k[5]), pack_half2(k[6], k[7]));  // exact
    if (grp == 0 && cur >= p_lo && cur < p_hi) {  // this CTA owns the current position: half a warp fills the caches
      *reinterpret_cast<uint4*>(kb + (int64_t)cur * D) = kraw;
      *reinterpret_cast<uint4*>(vb + (int64_t)cur * D) = vnew;
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int i = 0; i < 8; ++i) q[g][i] *= p.scale;

  // ---- this half-warp's positions, online softmax
  float m[G], sum[G], acc[G][8];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY; sum[g] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[g][i] = 0.f;
  }
  for (int p0 = p_lo + grp; __any_sync(0xffffffffu, p0 < p_hi); p0 += kAttGroups * U) {
    if (p0 != p_lo + grp) request(p0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int pp = p0 + u * kAttGroups;
      if (!__any_sync(0xffffffffu, pp < p_hi)) break;  // whole warps take part in the shuffles
      float kf[8], vf[8], sc[G];
      half8_to_float(pp == cur ? kraw : kr[u], kf);
      half8_to_float(pp == cur ? vnew : vr[u], vf);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        sc[g] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) sc[g] = fmaf(q[g][i], kf[i], sc[g]);
      }
#pragma unroll
      for (int o = 8; o >= 1; o >>= 1) {
#pragma unroll
        for (int g = 0; g < G; ++g) sc[g] += __shfl_xor_sync(0xffffffffu, sc[g], o);
      }
      if (pp < p_hi) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float mn = fmaxf(m[g], sc[g]);
          const float corr = __expf(m[g] - mn), e = __expf(sc[g] - mn);
          m[g] = mn;
          sum[g] = sum[g] * corr + e;
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[g][i] = acc[g][i] * corr + e * vf[i];
        }
      }
    }
  }

  // ---- the half-warps meet: [group][G][D] weighted rows, [group][G] maxima and sums
  float* racc = att_smem;                         // kAttGroups * G * D
  float* rm = racc + kAttGroups * G * D;          // kAttGroups * G
  float* rl = rm + kAttGroups * G;                // kAttGroups * G
  float* rec = rl + kAttGroups * G;               // this CTA's record: [G][D] weighted rows, [G] maxima, [G] sums
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float* dst = racc + (grp * G + g) * D + l * 8;
    *reinterpret_cast<float4*>(dst) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
    if (l == 0) { rm[grp * G + g] = m[g]; rl[grp * G + g] = sum[g]; }
  }
  __syncthreads();
  __half* op = p.out + ((int64_t)b * p.hq + (int64_t)kvh * G) * D;
  for (int i = tid; i < G * D; i += kAttThreads) {
    const int g = i / D;
    float mx = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kAttGroups; ++w) mx = fmaxf(mx, rm[w * G + g]);
#pragma unroll
    for (int w = 0; w < kAttGroups; ++w) {
      const float f = rl[w * G + g] > 0.f ? __expf(rm[w * G + g] - mx) : 0.f;  // a half-warp without positions has no maximum
      num += racc[w * G * D + i] * f;
      den += rl[w * G + g] * f;
    }
    if (splits == 1) {
      op[i] = __float2half_rn(num / den);
    } else {
      rec[i] = num;
      if (i % D == 0) { rec[G * D + g] = mx; rec[G * D + G + g] = den; }
    }
  }
  if (splits == 1) return;
  cluster_sync();
  const int share = G * D / splits;  // outputs that this CTA finishes
  for (int i = sp * share + tid; i < (sp + 1) * share; i += kAttThreads) {
    const int g = i / D;
    float mv[kAttMaxCluster], lv[kAttMaxCluster], nv[kAttMaxCluster];
#pragma unroll
    for (int r = 0; r < kAttMaxCluster; ++r) {
      const int from = r < splits ? r : 0;
      mv[r] = cluster_load(rec + G * D + g, from);
      lv[r] = r < splits ? cluster_load(rec + G * D + G + g, from) : 0.f;
      nv[r] = cluster_load(rec + i, from);
    }
    float mx = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
    for (int r = 0; r < kAttMaxCluster; ++r) mx = fmaxf(mx, lv[r] > 0.f ? mv[r] : -INFINITY);
#pragma unroll
    for (int r = 0; r < kAttMaxCluster; ++r) {
      const float f = lv[r] > 0.f ? __expf(mv[r] - mx) : 0.f;  // an empty range has no maximum
      num += (lv[r] > 0.f ? nv[r] : 0.f) * f;
      den += lv[r] * f;
    }
    op[i] = __float2half_rn(num / den);
  }
  cluster_sync();  // the records stay until every CTA has read them
}

template <int D, int G>
__global__ void __launch_bounds__(kAttThreads) decode_attention_kernel(const AttArgs p) {
  extern __shared__ __align__(16) float att_smem[];
  attention_body<D, G>(p, att_smem);
}

// ---- many sequences: thread per cache position -------------------------------------------------------
// With dozens of (sequence, kv head) pairs the launch fills the SMs without cutting the cache finely, and the
// warp-per-position form above pays five shuffles per dot product for nothing.  Here a thread owns a cache
// position for the scores (the 16 16-byte pieces of its K row requested together, the full 128-wide dot per
// query head with the queries broadcast from shared memory), one warp per query head does the softmax, and
// the V rows are summed with thread = (position stride 16, 16-byte piece), eight rows in flight per thread.
// Same split / ticket / merge scheme and the same scratch layout.
constexpr int kAttWideThreads = 256;
constexpr int kAttWideMaxSplits = 8;

template <int D, int G>
__device__ __forceinline__ void attention_wide_body(const __half* q, const __half* kb, const __half* vb, __half* out_row, float* att_smem,
                                               int p_lo, int p_hi, int chunk_cap, float scale, int splits, float* part,
                                               unsigned* ticket) {
  static_assert(D == 128, "pieces and thread mapping are laid out for 128-wide heads");
  __shared__ float head_max[kAttMaxGroup], head_sum[kAttMaxGroup];
  __shared__ unsigned my_ticket;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int n = p_hi > p_lo ? p_hi - p_lo : 0;
  float* qs = att_smem;                 // [G][D]
  float* sc = qs + kAttMaxGroup * D;    // [G][chunk_cap]
  float* red = sc + G * chunk_cap;      // [16 position groups][G][D]
  for (int i = tid; i < G * D; i += kAttWideThreads) qs[i] = __half2float(q[i]) * scale;
  __syncthreads();
  for (int i = tid; i < n; i += kAttWideThreads) {
    uint4 u[D / 8];
    const uint4* row = reinterpret_cast<const uint4*>(kb + (int64_t)(p_lo + i) * D);
#pragma unroll
    for (int c = 0; c < D / 8; ++c) u[c] = row[c];
    float acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = 0.f;
#pragma unroll
    for (int c = 0; c < D / 8; ++c) {
      const __half2* h2 = reinterpret_cast<const __half2*>(&u[c]);
      float kf[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h2[j]);
        kf[2 * j] = f.x;
        kf[2 * j + 1] = f.y;
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 qa = *reinterpret_cast<const float4*>(qs + g * D + c * 8);
        const float4 qb = *reinterpret_cast<const float4*>(qs + g * D + c * 8 + 4);
        acc[g] += kf[0] * qa.x + kf[1] * qa.y + kf[2] * qa.z + kf[3] * qa.w + kf[4] * qb.x + kf[5] * qb.y + kf[6] * qb.z + kf[7] * qb.w;
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) sc[g * chunk_cap + i] = acc[g];
  }
  __syncthreads();
  if (w < G) {  // head w: maximum, exponentials (kept unnormalised), sum
    float* sh = sc + w * chunk_cap;
    float m = -INFINITY;
    for (int i = lane; i < n; i += 32) m = fmaxf(m, sh[i]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float sum = 0.f;
    for (int i = lane; i < n; i += 32) {
      const float e = __expf(sh[i] - m);
      sh[i] = e;
      sum += e;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) { head_max[w] = m; head_sum[w] = sum; }
  }
  __syncthreads();
  {
    const int ps = tid >> 4, piece = tid & 15;
    float acc[G][8];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[g][j] = 0.f;
    constexpr int U = 8;
    for (int i0 = ps; i0 < n; i0 += 16 * U) {
      uint4 u[U];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int i = i0 + 16 * j;
        u[j] = i < n ? *reinterpret_cast<const uint4*>(vb + (int64_t)(p_lo + i) * D + piece * 8) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int i = i0 + 16 * j;
        if (i < n) {
          const __half2* h2 = reinterpret_cast<const __half2*>(&u[j]);
          float vf[8];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float2 f = __half22float2(h2[c]);
            vf[2 * c] = f.x;
            vf[2 * c + 1] = f.y;
          }
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const float pr = sc[g * chunk_cap + i];
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[g][c] += pr * vf[c];
          }
        }
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float* dst = red + (ps * G + g) * D + piece * 8;
      *reinterpret_cast<float4*>(dst) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
    }
  }
  __syncthreads();
  if (splits == 1) {
    for (int i = tid; i < G * D; i += kAttWideThreads) {
      float v = 0.f;
#pragma unroll
      for (int gs = 0; gs < 16; ++gs) v += red[gs * G * D + i];
      out_row[i] = __float2half_rn(v / head_sum[i / D]);
    }
    return;
  }
  // this split's record: [G][D + 2] = weighted rows, maximum, sum
  for (int i = tid; i < G * D; i += kAttWideThreads) {
    float v = 0.f;
#pragma unroll
    for (int gs = 0; gs < 16; ++gs) v += red[gs * G * D + i];
    part[(i / D) * (D + 2) + (i % D)] = v;
  }
  if (tid < G) { part[tid * (D + 2) + D] = head_max[tid]; part[tid * (D + 2) + D + 1] = head_sum[tid]; }
  __threadfence();
  __syncthreads();
  if (tid == 0) my_ticket = atomicAdd(ticket, 1u);
  __syncthreads();
  if (my_ticket != (unsigned)(splits - 1)) return;
  __threadfence();
  const float* all = part - (size_t)blockIdx.z * G * (D + 2);  // record of split 0
  for (int i = tid; i < G * D; i += kAttWideThreads) {
    const int g = i / D, d = i % D;
    float mv[kAttWideMaxSplits], lv[kAttWideMaxSplits], nv[kAttWideMaxSplits];  // requested together: one memory round trip
#pragma unroll
    for (int s2 = 0; s2 < kAttWideMaxSplits; ++s2) {
      const float* rec = all + ((size_t)(s2 < splits ? s2 : 0) * G + g) * (D + 2);
      mv[s2] = __ldcg(rec + D);
      lv[s2] = s2 < splits ? __ldcg(rec + D + 1) : 0.f;
      nv[s2] = __ldcg(rec + d);
    }
    float m = -INFINITY;
#pragma unroll
    for (int s2 = 0; s2 < kAttWideMaxSplits; ++s2) m = fmaxf(m, lv[s2] > 0.f ? mv[s2] : -INFINITY);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int s2 = 0; s2 < kAttWideMaxSplits; ++s2) {
      const float f = lv[s2] > 0.f ? __expf(mv[s2] - m) : 0.f;  // an empty split has no maximum
      num += (lv[s2] > 0.f ? nv[s2] : 0.f) * f;
      den += lv[s2] * f;
    }
    out_row[i] = __float2half_rn(num / den);
  }
  if (tid == 0) *ticket = 0u;
}

template <int D>
__global__ void __launch_bounds__(kAttWideThreads) decode_attention_wide_kernel(const __half* q, const __half* k_cache, const __half* v_cache,
                                                                        const int64_t* pos_dev, int64_t pos_host, __half* out,
                                                                        int hq, int hkv, int max_len, float scale, float* parts,
                                                                        unsigned* tickets) {
  extern __shared__ __align__(16) float att_smem[];
  const int G = hq / hkv;
  const int kvh = blockIdx.x, b = blockIdx.y, sp = blockIdx.z, splits = gridDim.z;
  pdl_enter();
  const int64_t len64 = (pos_dev ? *pos_dev : pos_host) + 1;  // the current token is already in the cache
  const int L = (int)(len64 < 1 ? 1 : (len64 > max_len ? max_len : len64));
  // chunk_cap sizes the score rows in shared memory; a multiple of 4 keeps the float4 area behind them aligned
  const int chunk = (L + splits - 1) / splits, chunk_cap = ((max_len + splits - 1) / splits + 3) & ~3;
  const int p_lo = sp * chunk, p_hi = p_lo + chunk < L ? p_lo + chunk : L;
  const __half* qp = q + ((int64_t)b * hq + (int64_t)kvh * G) * D;
  const __half* kb = k_cache + ((int64_t)b * hkv + kvh) * (int64_t)max_len * D;
  const __half* vb = v_cache + ((int64_t)b * hkv + kvh) * (int64_t)max_len * D;
  __half* op = out + ((int64_t)b * hq + (int64_t)kvh * G) * D;
  const size_t head = (size_t)b * hkv + kvh;
  float* part = parts ? parts + (head * splits + sp) * G * (D + 2) : nullptr;
  unsigned* ticket = tickets ? tickets + head : nullptr;
  switch (G) {
    case 1: attention_wide_body<D, 1>(qp, kb, vb, op, att_smem, p_lo, p_hi, chunk_cap, scale, splits, part, ticket); break;
    case 2: attention_wide_body<D, 2>(qp, kb, vb, op, att_smem, p_lo, p_hi, chunk_cap, scale, splits, part, ticket); break;
    case 4: attention_wide_body<D, 4>(qp, kb, vb, op, att_smem, p_lo, p_hi, chunk_cap, scale, splits, part, ticket); break;
    case 8: attention_wide_body<D, 8>(qp, kb, vb, op, att_smem, p_lo, p_hi, chunk_cap, scale, splits, part, ticket); break;
    default: break;
  }
}

}  // namespace pe

using namespace pe;

extern "C" int pe_add_rmsnorm(void* x, const void* delta, int delta_dtype, const void* weight, void* out, int rows, int hidden,
                              float eps, void* stream) {
  if (!x || !weight || !out || rows < 1 || hidden < 8) return PE_ERR_ARG;
  if (delta && delta_dtype != PE_F32 && delta_dtype != PE_F16) return PE_ERR_ARG;
  if (hidden % 8 || hidden > kNormThreads * 8 * kNormMaxIter) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(weight) |
       reinterpret_cast<uintptr_t>(out)) & 15)
    return PE_ERR_ALIGN;
  const int iters = (hidden + 8 * kNormThreads - 1) / (8 * kNormThreads);
  auto kfn = iters == 1 ? add_rmsnorm_kernel<1> : iters == 2 ? add_rmsnorm_kernel<2> : add_rmsnorm_kernel<kNormMaxIter>;
  PE_CUDA_TRY(launch_pdl(kfn, dim3(rows), dim3(kNormThreads), 0, static_cast<cudaStream_t>(stream),
                         static_cast<__half*>(x), delta, delta_dtype, static_cast<const __half*>(weight), static_cast<__half*>(out),
                         hidden, eps));
  return PE_OK;
}

static int rope_cache(const void* qkv, int64_t ld_qkv, const int64_t* pos_dev, int64_t pos_host, void* q_out, void* k_cache, void* v_cache, int batch,
                      int t, int hq, int hkv, int head_dim, int max_len, float theta, bool token_major, void* stream) {
  if (!qkv || !q_out || !k_cache || !v_cache || batch < 1 || t < 1 || hq < 1 || hkv < 1 || max_len < 1) return PE_ERR_ARG;
  if (head_dim < 2 || head_dim > 2048 || (head_dim & 1)) return PE_ERR_SHAPE;
  if (ld_qkv < (int64_t)(hq + 2 * hkv) * head_dim) return PE_ERR_ARG;
  if ((int64_t)batch * t > 0x7fffffff || hq + 2 * hkv > 65535) return PE_ERR_LIMIT;
  PE_CUDA_TRY(launch_pdl(rope_cache_kernel, dim3((unsigned)(batch * t)), dim3(kRopeThreads), 0,
                         static_cast<cudaStream_t>(stream), static_cast<const __half*>(qkv), ld_qkv, pos_dev, pos_host,
                         static_cast<__half*>(q_out), static_cast<__half*>(k_cache), static_cast<__half*>(v_cache), t, hq, hkv,
                         head_dim, max_len, theta, token_major ? (int64_t)head_dim : (int64_t)t * head_dim,
                         token_major ? (int64_t)hq * head_dim : (int64_t)head_dim));
  return PE_OK;
}

extern "C" int pe_rope_cache(const void* qkv, int64_t ld_qkv, const int64_t* pos_dev, int64_t pos_host, void* q_out,
                             void* k_cache, void* v_cache, int batch, int t, int hq, int hkv, int head_dim, int max_len,
                             float theta, void* stream) {
  return rope_cache(qkv, ld_qkv, pos_dev, pos_host, q_out, k_cache, v_cache, batch, t, hq, hkv, head_dim, max_len, theta, false, stream);
}

extern "C" int pe_rope_cache_token_major(const void* qkv, int64_t ld_qkv, const int64_t* pos_dev, int64_t pos_host, void* q_out,
                                         void* k_cache, void* v_cache, int batch, int t, int hq, int hkv, int head_dim, int max_len,
                                         float theta, void* stream) {
  return rope_cache(qkv, ld_qkv, pos_dev, pos_host, q_out, k_cache, v_cache, batch, t, hq, hkv, head_dim, max_len, theta, true, stream);
}

extern "C" int pe_silu_mul(const void* gate_up, int64_t ld_gu, void* out, int64_t ld_out, int rows, int inter, void* stream) {
  if (!gate_up || !out || rows < 1 || inter < 8) return PE_ERR_ARG;
  if (inter % 8 || ld_gu % 8 || ld_out % 8) return PE_ERR_SHAPE;
  if (ld_gu < 2 * (int64_t)inter || ld_out < inter) return PE_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(out)) & 15) return PE_ERR_ALIGN;
  const int64_t n_vec = (int64_t)rows * (inter / 8);
  const int64_t blocks = (n_vec + 255) / 256;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  PE_CUDA_TRY(launch_pdl(silu_mul_kernel, dim3((unsigned)blocks), dim3(256), 0, static_cast<cudaStream_t>(stream),
                         static_cast<const __half*>(gate_up), ld_gu, static_cast<__half*>(out), ld_out, inter, n_vec));
  return PE_OK;
}

// scratch of the split form: [tickets: one counter per (sequence, kv head), 4 KB, zero before the first
// call and left zero][one record per (sequence, kv head, split, query head of the group)]
extern "C" size_t pe_decode_attention_workspace_bytes(int batch, int hq, int hkv, int head_dim) {
  if (batch < 1 || hq < 1 || hkv < 1 || head_dim != 128 || hq % hkv || (size_t)batch * hkv * 4 > 4096) return 0;
  return 4096 + (size_t)batch * hkv * kAttMaxSplits * (hq / hkv) * (head_dim + 2) * sizeof(float);
}

static int attention_launch(AttArgs a, int batch, int head_dim, void* stream) {
  if (!a.k_cache || !a.v_cache || !a.out || batch < 1 || a.hq < 1 || a.hkv < 1 || a.max_len < 1) return PE_ERR_ARG;
  if (head_dim != 128 || a.hq % a.hkv) return PE_ERR_SHAPE;
  const int G = a.hq / a.hkv;
  if (G != 1 && G != 2 && G != 4 && G != 8) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(a.k_cache) | reinterpret_cast<uintptr_t>(a.v_cache)) & 15) return PE_ERR_ALIGN;
  if (batch > 65535) return PE_ERR_LIMIT;
  // One cluster per (kv head, sequence): eight CTAs, fewer when the longest possible sequence has under 16 positions
  // for each of them, or when the heads alone fill the SMs twice over.
  const int sms = sm_count();
  if (sms <= 0) return PE_ERR_CUDA;
  int splits = kAttMaxCluster;
  while (splits > 1 && (a.max_len < 16 * splits || (int64_t)batch * a.hkv * splits > 4ll * sms)) splits /= 2;
  const size_t smem = ((size_t)kAttGroups * G * 128 + 2 * (size_t)kAttGroups * G + (size_t)G * 130) * sizeof(float);
  a.scale = 1.f / sqrtf((float)head_dim);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)splits, (unsigned)a.hkv, (unsigned)batch);
  cfg.blockDim = dim3(kAttThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)splits; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  auto kfn = G == 1 ? decode_attention_kernel<128, 1> : G == 2 ? decode_attention_kernel<128, 2>
             : G == 4 ? decode_attention_kernel<128, 4> : decode_attention_kernel<128, 8>;
  if (smem > 48 * 1024) {
    static thread_local bool configured[16] = {false};
    int dev = 0;
    PE_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 16 || !configured[dev]) {
      PE_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));  // G = 8 only
      if (dev < 16) configured[dev] = true;
    }
  }
  const bool line = line_holds(cfg.stream);
  PE_CUDA_TRY(cudaLaunchKernelEx(&cfg, kfn, a));
  if (line) line_extend(cfg.stream);
  return PE_OK;
}

extern "C" int pe_decode_attention(const void* q, const void* k_cache, const void* v_cache, const int64_t* pos_dev,
                                   int64_t pos_host, void* out, int batch, int hq, int hkv, int head_dim, int max_len,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  if (!q) return PE_ERR_ARG;
  if (reinterpret_cast<uintptr_t>(q) & 7) return PE_ERR_ALIGN;
  AttArgs a = {};
  a.q = static_cast<const __half*>(q);
  a.k_cache = static_cast<__half*>(const_cast<void*>(k_cache));
  a.v_cache = static_cast<__half*>(const_cast<void*>(v_cache));
  a.pos_dev = pos_dev; a.pos_host = pos_host;
  a.out = static_cast<__half*>(out);
  a.hq = hq; a.hkv = hkv; a.max_len = max_len;
  const int sms = sm_count();
  if (sms > 0 && batch >= 1 && hkv >= 1 && (int64_t)batch * hkv * 4 >= sms && head_dim == 128 && hq % hkv == 0 &&
      (hq / hkv == 1 || hq / hkv == 2 || hq / hkv == 4 || hq / hkv == 8) && k_cache && v_cache && out && max_len >= 1 &&
      batch <= 65535 && !((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15)) {
    // many (sequence, kv head) pairs: the thread-per-position kernel
    const int G = hq / hkv;
    int splits = 1;
    const size_t need = pe_decode_attention_workspace_bytes(batch, hq, hkv, head_dim);
    if (workspace && need && workspace_bytes >= need && !(reinterpret_cast<uintptr_t>(workspace) & 15)) {
      splits = sms / (hkv * batch);
      splits = splits < 1 ? 1 : (splits > kAttWideMaxSplits ? kAttWideMaxSplits : splits);
      if (max_len < 64 * splits) splits = max_len / 64 < 1 ? 1 : max_len / 64;
    }
    const int chunk_cap = ((max_len + splits - 1) / splits + 3) & ~3;  // as in the kernel
    const size_t smem = ((size_t)kAttMaxGroup * 128 + (size_t)G * chunk_cap + (size_t)16 * G * 128) * sizeof(float);
    if (smem <= 200 * 1024) {
      auto kfn = decode_attention_wide_kernel<128>;
      static thread_local size_t configured[16] = {0};
      int dev = 0;
      PE_CUDA_TRY(cudaGetDevice(&dev));
      if (smem > 48 * 1024 && (dev >= 16 || configured[dev] < smem)) {
        PE_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev < 16) configured[dev] = smem;
      }
      float* parts = splits > 1 ? reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + 4096) : nullptr;
      unsigned* tickets = splits > 1 ? static_cast<unsigned*>(workspace) : nullptr;
      PE_CUDA_TRY(launch_pdl(kfn, dim3((unsigned)hkv, (unsigned)batch, (unsigned)splits), dim3(kAttWideThreads), smem,
                             static_cast<cudaStream_t>(stream), static_cast<const __half*>(q), static_cast<const __half*>(k_cache),
                             static_cast<const __half*>(v_cache), pos_dev, pos_host, static_cast<__half*>(out), hq, hkv, max_len,
                             1.f / sqrtf((float)head_dim), parts, tickets));
      return PE_OK;
    }
  }
  return attention_launch(a, batch, head_dim, stream);
}

extern "C" int pe_rope_attention(const void* qkv, int64_t ld_qkv, const int64_t* pos_dev, int64_t pos_host, void* k_cache,
                                 void* v_cache, void* out, int batch, int hq, int hkv, int head_dim, int max_len, float theta,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  if (!qkv) return PE_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(qkv) & 7) || (ld_qkv & 3)) return PE_ERR_ALIGN;
  if (hq >= 1 && hkv >= 1 && ld_qkv < (int64_t)(hq + 2 * hkv) * head_dim) return PE_ERR_ARG;
  AttArgs a = {};
  a.qkv = static_cast<const __half*>(qkv); a.ld_qkv = ld_qkv;
  a.k_cache = static_cast<__half*>(k_cache);
  a.v_cache = static_cast<__half*>(v_cache);
  a.pos_dev = pos_dev; a.pos_host = pos_host;
  a.out = static_cast<__half*>(out);
  a.hq = hq; a.hkv = hkv; a.max_len = max_len;
  a.theta = theta;
  return attention_launch(a, batch, head_dim, stream);
}
