// Entry points of the decode-size quantized matmul (1..16 activation rows): argument checks, scratch layout, dispatch.
//
//   y[m, r] = sum_blk norm[r, blk] * sum_k ct[code[r, blk, k]] * xt[m, blk, k]   (+ bias[r])
//
// Every call goes to the bulk-copy kernel (pe_gemv_bulk.cu), whichever layout it has: a decoder layer's four launches for
// one row take 40.3 us on row-major arrays, 42.9 us on the tiled copy, and 52.0 us in the column-owner kernel
// (pe_gemv_cols.cu), which is left for pe_gemv_pro, whose callers give no scratch memory.
#include "pe_gemv_decode.cuh"

namespace pe {

// Scratch layout: [256 KB, last word: status (0 = ok)][activations in operand order], pe_gemv_scratch_bytes in all.
// pe_gemv_workspace_bytes is a bound that grows with the layer: it had room for fp32 partial sums of a K split that no kernel
// makes any more.  Callers planned with it and pe_gemv_noalloc refuses shapes by it, so it stays as it was.
constexpr size_t kCounterBytes = kGemvStatusBytes;
// limit on out_f, from the time when a launch kept one word per row tile there
constexpr int kMaxRowTiles = (int)(kCounterBytes / sizeof(unsigned)) - 1;
constexpr int kMaxSms = 256;

// fp32 partial sums of 16-row tiles for every part of the K range that `ctas` equal ranges of the layer can cut it into
static size_t partial_bytes(int batch, int N, int K, long long ctas) {
  const long long nb = K / kBlock, tiles = (N + 15) / 16, steps = (tiles + 15) / 16 * nb * 16;
  long long g = steps / 16;
  g = g < ctas ? (g < 1 ? 1 : g) : ctas;
  const long long per = steps / g;
  long long slots = (nb * 16 + per - 1) / per + 1;
  if (slots > g) slots = g;
  return (size_t)(tiles * slots * 16 * batch) * sizeof(float);
}

}  // namespace pe

using namespace pe;

extern "C" size_t pe_gemv_workspace_bytes(int batch, int out_f, int in_f_padded) {
  if (batch < 1 || batch > 16 || out_f < 1 || in_f_padded < kBlock || in_f_padded % kBlock) return 0;
  if ((out_f + 15) / 16 > kMaxRowTiles) return 0;
  const size_t part = partial_bytes(batch, out_f, in_f_padded, kMaxSms), frags = gemv_bulk_frag_bytes(1, batch, in_f_padded);
  return kCounterBytes + (part > frags ? part : frags);
}

extern "C" size_t pe_gemv_scratch_bytes(int batch, int in_f_padded) {
  if (batch < 1 || batch > 16 || in_f_padded < kBlock || in_f_padded % kBlock) return 0;
  return kCounterBytes + gemv_bulk_frag_bytes(1, batch, in_f_padded);
}

// Argument checks shared by every decode-size entry point.
static int gemv_check(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms, const void* tiles,
                      const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype, int64_t ld_x, int in_f,
                      void* y, int y_dtype, int64_t ld_y, int batch, int out_f, int in_f_padded) {
  if (!ct_scaled || !x || !y) return PE_ERR_ARG;
  if (!tiles && (!codes || !norms)) return PE_ERR_ARG;
  if (batch < 1 || out_f < 1 || in_f < 1 || in_f > in_f_padded) return PE_ERR_ARG;
  if (x_kind != PE_X_ROTATED && x_kind != PE_X_RAW) return PE_ERR_ARG;
  if (x_dtype < PE_F32 || x_dtype > PE_BF16 || y_dtype < PE_F32 || y_dtype > PE_BF16) return PE_ERR_ARG;
  if (n_levels < 2 || n_levels > 256 || (packed && n_levels > 16)) return PE_ERR_ARG;
  if (batch > 16 || in_f_padded % kBlock) return PE_ERR_SHAPE;
  if (tiles) {
    if (reinterpret_cast<uintptr_t>(tiles) & 15) return PE_ERR_ALIGN;
  } else {
    if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15)) return PE_ERR_ALIGN;
    if (ld_codes < (packed ? in_f_padded / 2 : in_f_padded) || ld_norms < in_f_padded / kBlock) return PE_ERR_ARG;
  }
  if (ld_x < (x_kind == PE_X_RAW ? in_f : in_f_padded) || ld_y < out_f) return PE_ERR_ARG;
  return PE_OK;
}

// Shared by every entry point: row-major codes + norms, or tiles.  Arguments checked.
static int gemv_dispatch(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms, const void* tiles,
                         const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype, int64_t ld_x, int in_f, void* y,
                         int y_dtype, int64_t ld_y, const void* bias, int batch, int out_f, int in_f_padded, void* workspace,
                         size_t workspace_bytes, void* stream) {
  if (!workspace) return PE_ERR_ARG;
  if ((out_f + 15) / 16 > kMaxRowTiles) return PE_ERR_LIMIT;
  if (workspace_bytes < pe_gemv_scratch_bytes(batch, in_f_padded)) return PE_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 15) return PE_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  GemvBulkCall q = {};
  q.codes = codes; q.packed = packed; q.ld_codes = ld_codes; q.norms = norms; q.ld_norms = ld_norms; q.tiles = tiles;
  q.ct_scaled = ct_scaled; q.n_levels = n_levels;
  q.x = x; q.x_kind = x_kind; q.x_dtype = x_dtype; q.ld_x = ld_x; q.in_f = in_f;
  q.y = y; q.y_dtype = y_dtype; q.ld_y = ld_y; q.bias = bias;
  q.batch = batch; q.out_f = out_f; q.in_f_padded = in_f_padded;
  q.status = reinterpret_cast<int*>(ws + kCounterBytes - 4);
  q.frags = ws + kCounterBytes;
  return gemv_bulk_run(q, st);
}

static int gemv_run(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                    const void* tiles, const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype,
                    int64_t ld_x, int in_f, void* y, int y_dtype, int64_t ld_y, const void* bias, int batch, int out_f,
                    int in_f_padded, void* workspace, size_t workspace_bytes, void* stream) {
  if (!workspace) return PE_ERR_ARG;
  const int c = gemv_check(codes, packed, ld_codes, norms, ld_norms, tiles, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, y,
                           y_dtype, ld_y, batch, out_f, in_f_padded);
  if (c != PE_OK) return c;
  return gemv_dispatch(codes, packed, ld_codes, norms, ld_norms, tiles, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, y, y_dtype, ld_y,
                       bias, batch, out_f, in_f_padded, workspace, workspace_bytes, stream);
}

// The row-major arrays stream as fast as the tiled copy (8 rows, a decoder layer's four launches: 44.7 and 47.0 us).
extern "C" int pe_gemv_small_batch_takes(int, int64_t, const void*, int64_t, int, int) { return 1; }

extern "C" int pe_gemv(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                       const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype, int64_t ld_x,
                       int in_f, void* y, int y_dtype, int64_t ld_y, const void* bias, int batch, int out_f,
                       int in_f_padded, void* workspace, size_t workspace_bytes, void* stream) {
  return gemv_run(codes, packed, ld_codes, norms, ld_norms, nullptr, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, y,
                  y_dtype, ld_y, bias, batch, out_f, in_f_padded, workspace, workspace_bytes, stream);
}

// Reads a status word back (and optionally clears it): waits for the stream, no allocation.
static int read_status_word(int* word, int clear, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int v = 0;
  PE_CUDA_TRY(cudaMemcpyAsync(&v, word, sizeof(int), cudaMemcpyDeviceToHost, st));
  PE_CUDA_TRY(cudaStreamSynchronize(st));
  if (clear && v != 0) PE_CUDA_TRY(cudaMemsetAsync(word, 0, sizeof(int), st));
  return v < 0 ? 0 : v;
}

extern "C" int pe_gemv_status(void* workspace, size_t workspace_bytes, int clear, void* stream) {
  if (!workspace || workspace_bytes < kCounterBytes) return PE_ERR_ARG;
  return read_status_word(reinterpret_cast<int*>(static_cast<uint8_t*>(workspace) + kCounterBytes - 4), clear, stream);
}

// ---- grouped launch: the experts of a mixture layer ------------------------------------
//
// `max_problems` problems of one shape share a launch.  Problem i is described on the device by (matrix index, first
// row, rows <= 16, 0): rows first .. first + rows - 1 of the row list `x_rows` (or of x itself when x_rows is NULL)
// times matrix `index` of a stack of matrices, written to the same rows of y.  Slots with rows <= 0 have no work, so
// the caller can size the launch for the worst case without knowing the routing.
namespace pe {
// last word: status.  The size, and with it the limit on problems x row tiles below, is that of a counter zone which is gone;
// both stay: callers size buffers and choose their path by them
constexpr size_t kGroupedZone = 4u << 20;
}  // namespace pe

extern "C" size_t pe_gemv_grouped_workspace_bytes(int max_problems, int out_f, int in_f_padded) {
  if (max_problems < 1 || out_f < 1 || in_f_padded < kBlock || in_f_padded % kBlock) return 0;
  // at most as many 16-row tiles (and one word per problem) over all problems as the zone has words
  if ((size_t)max_problems * (((size_t)((out_f + 15) / 16 + 1) * 4 + 255) & ~(size_t)255) > kGroupedZone) return 0;
  return kGroupedZone + gemv_bulk_frag_bytes(max_problems, 16, in_f_padded);
}

static int grouped_run(const void* codes, int packed, int64_t ld_codes, int64_t codes_stride, const void* norms, int64_t ld_norms,
                       int64_t norms_stride, const void* tiles, int64_t tiles_stride, const float* ct_scaled, int n_levels, const void* x,
                       int x_kind, int x_dtype, int64_t ld_x, int in_f, const int32_t* x_rows, void* y, int y_dtype, int64_t ld_y,
                       const int32_t* problems, int max_problems, int max_rows, int out_f, int in_f_padded, void* workspace,
                       size_t workspace_bytes, void* stream) {
  if ((!tiles && (!codes || !norms)) || !ct_scaled || !x || !y || !problems || !workspace) return PE_ERR_ARG;
  if (max_rows < 1 || max_rows > 16) return PE_ERR_ARG;
  if (max_problems < 1 || max_problems > 65535 || out_f < 1 || in_f < 1 || in_f > in_f_padded) return PE_ERR_ARG;
  if (x_kind != PE_X_ROTATED && x_kind != PE_X_RAW && x_kind != PE_X_SILU_MUL) return PE_ERR_ARG;
  if (x_dtype < PE_F32 || x_dtype > PE_BF16 || y_dtype < PE_F32 || y_dtype > PE_BF16) return PE_ERR_ARG;
  if (x_kind == PE_X_SILU_MUL && x_dtype != PE_F16) return PE_ERR_ARG;
  if (n_levels < 2 || n_levels > 256 || (packed && n_levels > 16)) return PE_ERR_ARG;
  if (in_f_padded % kBlock) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(problems) & 15) || (reinterpret_cast<uintptr_t>(workspace) & 15)) return PE_ERR_ALIGN;
  if (tiles) {
    if ((reinterpret_cast<uintptr_t>(tiles) & 15) || (tiles_stride & 15)) return PE_ERR_ALIGN;
  } else {
    if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15) || (codes_stride & 15)) return PE_ERR_ALIGN;
    if (ld_codes < (packed ? in_f_padded / 2 : in_f_padded) || ld_norms < in_f_padded / kBlock) return PE_ERR_ARG;
  }
  if (ld_x < (x_kind == PE_X_RAW ? in_f : x_kind == PE_X_SILU_MUL ? 2 * (int64_t)in_f : in_f_padded) || ld_y < out_f) return PE_ERR_ARG;
  const size_t need = pe_gemv_grouped_workspace_bytes(max_problems, out_f, in_f_padded);
  if (need == 0) return PE_ERR_LIMIT;
  if (workspace_bytes < need) return PE_ERR_WORKSPACE;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  GemvBulkCall q = {};
  q.codes = codes; q.packed = packed; q.ld_codes = ld_codes; q.norms = norms; q.ld_norms = ld_norms; q.tiles = tiles;
  q.ct_scaled = ct_scaled; q.n_levels = n_levels;
  q.x = x; q.x_kind = x_kind; q.x_dtype = x_dtype; q.ld_x = ld_x; q.in_f = in_f;
  q.y = y; q.y_dtype = y_dtype; q.ld_y = ld_y;
  q.batch = max_rows; q.out_f = out_f; q.in_f_padded = in_f_padded;
  q.status = reinterpret_cast<int*>(ws + kGroupedZone - 4);
  q.frags = ws + kGroupedZone;
  q.problems = problems; q.max_problems = max_problems; q.x_rows = x_rows;
  q.codes_stride = codes_stride; q.norms_stride = norms_stride; q.tiles_stride = tiles_stride;
  return gemv_bulk_run(q, static_cast<cudaStream_t>(stream));
}

extern "C" int pe_gemv_grouped(const void* codes, int packed, int64_t ld_codes, int64_t codes_stride, const void* norms,
                               int64_t ld_norms, int64_t norms_stride, const float* ct_scaled, int n_levels, const void* x,
                               int x_kind, int x_dtype, int64_t ld_x, int in_f, const int32_t* x_rows, void* y, int y_dtype,
                               int64_t ld_y, const int32_t* problems, int max_problems, int max_rows, int out_f,
                               int in_f_padded, void* workspace, size_t workspace_bytes, void* stream) {
  return grouped_run(codes, packed, ld_codes, codes_stride, norms, ld_norms, norms_stride, nullptr, 0, ct_scaled, n_levels, x, x_kind, x_dtype,
                     ld_x, in_f, x_rows, y, y_dtype, ld_y, problems, max_problems, max_rows, out_f, in_f_padded, workspace, workspace_bytes, stream);
}

extern "C" int pe_gemv_grouped_tiled(const void* tiles, int packed, int64_t tiles_stride, const float* ct_scaled, int n_levels, const void* x,
                                     int x_kind, int x_dtype, int64_t ld_x, int in_f, const int32_t* x_rows, void* y, int y_dtype,
                                     int64_t ld_y, const int32_t* problems, int max_problems, int max_rows, int out_f,
                                     int in_f_padded, void* workspace, size_t workspace_bytes, void* stream) {
  if (!tiles) return PE_ERR_ARG;
  return grouped_run(nullptr, packed, 0, 0, nullptr, 0, 0, tiles, tiles_stride, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, x_rows, y,
                     y_dtype, ld_y, problems, max_problems, max_rows, out_f, in_f_padded, workspace, workspace_bytes, stream);
}

// ---- tiled weight layout ---------------------------------------------------------
namespace pe {
// The codes of one 16-row tile and 128-block, 1 KB (2 KB for byte codes), followed by the 16 fp16 block norms; the
// blocks of a row tile follow each other.
template <bool PACKED> struct TileGeom {
  static constexpr int kCodeBytes = PACKED ? 1024 : 2048;
  static constexpr int kTileBytes = kCodeBytes + 32;
};
// one thread per 16-byte piece of the output
template <bool PACKED>
__global__ void __launch_bounds__(256) retile_kernel(const uint8_t* codes, int64_t ld_codes, const __half* norms,
                                                     int64_t ld_norms, uint8_t* out, int N, int nb, int64_t n_pieces) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pieces) return;
  constexpr int kPieces = TileGeom<PACKED>::kTileBytes / 16;   // 66 or 130
  constexpr int kRowBytes = PACKED ? 64 : 128;
  const int64_t tile = i / kPieces;
  const int piece = (int)(i - tile * kPieces);
  const int rt16 = (int)(tile / nb), b = (int)(tile - (int64_t)rt16 * nb);
  uint4 v = make_uint4(0, 0, 0, 0);
  if (piece < TileGeom<PACKED>::kCodeBytes / 16) {
    const int r = piece / (kRowBytes / 16), c = piece % (kRowBytes / 16);
    const int row = rt16 * 16 + r;
    if (row < N) v = *reinterpret_cast<const uint4*>(codes + (int64_t)row * ld_codes + b * kRowBytes + c * 16);
  } else {  // norms: rows 0..7 in the first piece, 8..15 in the second
    const int r0 = (piece - TileGeom<PACKED>::kCodeBytes / 16) * 8;
    unsigned short h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int row = rt16 * 16 + r0 + k;
      h[k] = row < N ? __half_as_ushort(norms[(int64_t)row * ld_norms + b]) : (unsigned short)0;
    }
    v = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
  }
  *reinterpret_cast<uint4*>(out + i * 16) = v;
}
}  // namespace pe

extern "C" size_t pe_retile_bytes(int packed, int64_t out_f, int64_t in_f_padded) {
  if (out_f < 1 || in_f_padded < kBlock || in_f_padded % kBlock) return 0;
  const size_t tile = packed ? TileGeom<true>::kTileBytes : TileGeom<false>::kTileBytes;
  return (size_t)((out_f + 15) / 16) * (size_t)(in_f_padded / kBlock) * tile;
}

extern "C" int pe_retile(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms, void* tiles,
                         int64_t out_f, int64_t in_f_padded, void* stream) {
  if (!codes || !norms || !tiles || out_f < 1 || out_f > 0x7fffffff) return PE_ERR_ARG;
  if (in_f_padded < kBlock || in_f_padded % kBlock) return PE_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(codes) & 15) || (ld_codes & 15) || (reinterpret_cast<uintptr_t>(tiles) & 15)) return PE_ERR_ALIGN;
  const int nb = (int)(in_f_padded / kBlock);
  const int64_t n_pieces = (int64_t)pe_retile_bytes(packed, out_f, in_f_padded) / 16;
  const int64_t blocks = (n_pieces + 255) / 256;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (packed)
    retile_kernel<true><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const uint8_t*>(codes), ld_codes,
                                                         static_cast<const __half*>(norms), ld_norms,
                                                         static_cast<uint8_t*>(tiles), (int)out_f, nb, n_pieces);
  else
    retile_kernel<false><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const uint8_t*>(codes), ld_codes,
                                                          static_cast<const __half*>(norms), ld_norms,
                                                          static_cast<uint8_t*>(tiles), (int)out_f, nb, n_pieces);
  PE_CUDA_TRY(cudaGetLastError());
  return PE_OK;
}

extern "C" int pe_gemv_tiled(const void* tiles, int packed, const float* ct_scaled, int n_levels, const void* x, int x_kind,
                             int x_dtype, int64_t ld_x, int in_f, void* y, int y_dtype, int64_t ld_y, const void* bias,
                             int batch, int out_f, int in_f_padded, void* workspace, size_t workspace_bytes, void* stream) {
  if (!tiles) return PE_ERR_ARG;
  return gemv_run(nullptr, packed, 0, nullptr, 0, tiles, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, y, y_dtype, ld_y,
                  bias, batch, out_f, in_f_padded, workspace, workspace_bytes, stream);
}

// ---- entry point for callers that cannot allocate device memory -------------------
//
// Some hosts of this library hand every byte of device memory to their own pool at
// start-up (an inference server sizes its KV cache from "whatever is free" and keeps
// it), so a cudaMalloc made later on behalf of one linear layer can fail, and the code
// that calls into the layer has no allocator of its own to ask.  For them the
// scratch lives inside the library image: a fixed array in device global memory that
// exists on every GPU that loads the library, from load until exit.
constexpr size_t kNoAllocScratchBytes = 8u << 20;  // 8 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// In host code the array's name only stands for the symbol; the device address has to
// be asked for, once per device, with that device current.
static void* g_noalloc_ptr[64] = {nullptr};

extern "C" size_t pe_gemv_noalloc_max_bytes(void) { return kNoAllocScratchBytes; }

// Device address of the array on the current device (looked up once per device).
static int noalloc_scratch(void** out) {
  int dev = 0;
  PE_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PE_ERR_LIMIT;
  if (!g_noalloc_ptr[dev]) {
    void* ptr = nullptr;
    PE_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    g_noalloc_ptr[dev] = ptr;
  }
  *out = g_noalloc_ptr[dev];
  return PE_OK;
}

extern "C" int pe_gemv_noalloc(const void* codes, int packed, int64_t ld_codes, const void* norms, int64_t ld_norms,
                               const float* ct_scaled, int n_levels, const void* x, int x_kind, int x_dtype,
                               int64_t ld_x, int in_f, void* y, int y_dtype, int64_t ld_y, const void* bias, int batch,
                               int out_f, int in_f_padded, void* stream) {
  const int c = gemv_check(codes, packed, ld_codes, norms, ld_norms, nullptr, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f,
                           y, y_dtype, ld_y, batch, out_f, in_f_padded);
  if (c != PE_OK) return c;
  const size_t need = pe_gemv_workspace_bytes(batch, out_f, in_f_padded);
  if (need == 0 || need > kNoAllocScratchBytes) return PE_ERR_LIMIT;  // shape needs more scratch than the built-in array holds
  void* ws = nullptr;
  const int r = noalloc_scratch(&ws);
  if (r != PE_OK) return r;
  return gemv_dispatch(codes, packed, ld_codes, norms, ld_norms, nullptr, ct_scaled, n_levels, x, x_kind, x_dtype, ld_x, in_f, y, y_dtype,
                       ld_y, bias, batch, out_f, in_f_padded, ws, kNoAllocScratchBytes, stream);
}

extern "C" int pe_gemv_noalloc_status(int clear, void* stream) {
  void* ws = nullptr;
  const int r = noalloc_scratch(&ws);
  if (r != PE_OK) return r;
  return read_status_word(reinterpret_cast<int*>(static_cast<uint8_t*>(ws) + kCounterBytes - 4), clear, stream);
}
