// Active-tile compaction: per-pixel masks as 64-bit tile words, ordered tile lists, and the
// dilated output-tile set of a convolution.
#include <stdio.h>
#include <string.h>
#include "mie_common.cuh"

namespace mie {
static thread_local char g_cuda_err[256] = "";
unsigned long long g_launch_count = 0;

void set_cuda_error(cudaError_t e) {
  snprintf(g_cuda_err, sizeof(g_cuda_err), "%s: %s", cudaGetErrorName(e), cudaGetErrorString(e));
}
}  // namespace mie

using namespace mie;

extern "C" int mie_version(void) { return 1; }

extern "C" const char *mie_status_string(int s) {
  switch (s) {
    case MIE_OK: return "ok";
    case MIE_EINVAL: return "invalid argument";
    case MIE_EALIGN: return "misaligned pointer or stride";
    case MIE_EUNSUPPORTED: return "unsupported combination";
    case MIE_ECUDA: return "CUDA runtime error";
    case MIE_ETOOBIG: return "size beyond capacity";
    default: return "unknown status";
  }
}

extern "C" const char *mie_last_cuda_error(void) { return g_cuda_err; }

// ---------------------------------------------------------------------------------------------
// mask words from a delta tensor or an explicit mask tensor: one warp per 8x8 tile
// ---------------------------------------------------------------------------------------------
// Any channel count, element by element (odd counts, strides or alignments).
template <typename T>
__global__ void __launch_bounds__(256) mask_words_kernel(const T *__restrict__ src, int64_t ps, int C, int N,
                                                         int H, int W, float thr, uint64_t *__restrict__ bits) {
  grid_dependency_wait();
  grid_dependency_trigger();
  const int TH = (H + 7) >> 3, TW = (W + 7) >> 3;
  const int ntiles = N * TH * TW;
  const int lane = threadIdx.x & 31;
  const int warps_per_grid = (gridDim.x * blockDim.x) >> 5;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntiles; t += warps_per_grid) {
    const int tx = t % TW, ty = (t / TW) % TH, n = t / (TW * TH);
    const int rows = min(8, H - ty * 8), cols = min(8, W - tx * 8);
    unsigned lo = 0, hi = 0;
    const int per_row = cols * C;
    const int total = rows * per_row;
    for (int i = lane; i < total; i += 32) {
      const int r = i / per_row, rem = i - r * per_row;
      const int px = rem / C, c = rem - px * C;
      const T v = src[((int64_t)(n * H + ty * 8 + r) * W + tx * 8 + px) * ps + c];
      bool a;
      if (sizeof(T) == 4 && thr >= 0.0f) a = fabsf((float)v) > thr;  // float source
      else a = v != (T)0;                                           // explicit mask source
      const int b = r * 8 + px;
      if (a) { if (b < 32) lo |= 1u << b; else hi |= 1u << (b - 32); }
    }
    lo = __reduce_or_sync(0xffffffffu, lo);
    hi = __reduce_or_sync(0xffffffffu, hi);
    if (lane == 0) bits[t] = ((uint64_t)hi << 32) | lo;
  }
}

// 16-byte pieces that lie inside one pixel each, `pieces` of them per pixel (16 bytes = 4 floats or int32, 16 mask bytes).
// A warp takes half a tile (32 pixels): the word half is one reduction.  Bound by HBM; what the first version spent its
// time on was two integer divisions per 16 bytes (46 MB of 32 channels: 33 us) -- here consecutive lanes take consecutive
// pieces of a row of eight pixels, and pixel and piece follow from a division by a loop invariant reciprocal.
template <bool FLOAT>
__global__ void __launch_bounds__(256) mask_words_vec_kernel(const uint4 *__restrict__ src, int64_t px_bytes, int pieces, unsigned recip, int N,
                                                             int H, int W, float thr, unsigned *__restrict__ bits32) {
  grid_dependency_wait();
  grid_dependency_trigger();
  const int TH = (H + 7) >> 3, TW = (W + 7) >> 3;
  const int halves = 2 * N * TH * TW;
  const int lane = threadIdx.x & 31;
  const int warps_per_grid = (gridDim.x * blockDim.x) >> 5;
  const int total = 32 * pieces;
  for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < halves; u += warps_per_grid) {
    const int t = u >> 1;
    const int tx = t % TW, ty = (t / TW) % TH, n = t / (TW * TH);
    const int y0 = ty * 8 + (u & 1) * 4, x0 = tx * 8;
    const char *base = reinterpret_cast<const char *>(src) + ((int64_t)(n * H + y0) * W + x0) * px_bytes;
    unsigned half = 0;
#pragma unroll 1
    for (int i0 = lane; i0 < total; i0 += 256) {
      uint4 v[8];
      int px[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {      // eight independent loads in flight
        const int i = i0 + 32 * j;
        px[j] = pieces == 1 ? i : (int)__umulhi((unsigned)i, recip);       // i / pieces
        v[j] = make_uint4(0u, 0u, 0u, 0u);
        if (i < total && y0 + (px[j] >> 3) < H && x0 + (px[j] & 7) < W)
          v[j] = *reinterpret_cast<const uint4 *>(base + ((int64_t)(px[j] >> 3) * W + (px[j] & 7)) * px_bytes + (i - px[j] * pieces) * 16);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        bool a;
        if (FLOAT)
          a = fabsf(__uint_as_float(v[j].x)) > thr || fabsf(__uint_as_float(v[j].y)) > thr || fabsf(__uint_as_float(v[j].z)) > thr ||
              fabsf(__uint_as_float(v[j].w)) > thr;
        else
          a = (v[j].x | v[j].y | v[j].z | v[j].w) != 0u;
        if (a) half |= 1u << px[j];
      }
    }
    half = __reduce_or_sync(0xffffffffu, half);
    if (lane == 0) bits32[u] = half;
  }
}

// Few channels: one thread per pixel, one warp per half tile, the ballot is the half word.
template <typename T>
__global__ void __launch_bounds__(256) mask_words_px_kernel(const T *__restrict__ src, int64_t ps, int C, int N, int H,
                                                            int W, float thr, unsigned *__restrict__ bits32) {
  grid_dependency_wait();
  grid_dependency_trigger();
  const int TH = (H + 7) >> 3, TW = (W + 7) >> 3;
  const int ntiles = N * TH * TW;
  const int lane = threadIdx.x & 31;
  for (int t = blockIdx.x * 4 + (threadIdx.x >> 6); t < ntiles; t += gridDim.x * 4) {
    const int p = threadIdx.x & 63;
    const int tx = t % TW, ty = (t / TW) % TH, n = t / (TW * TH);
    const int y = ty * 8 + (p >> 3), x = tx * 8 + (p & 7);
    bool a = false;
    if (y < H && x < W) {
      const T *px = src + ((int64_t)(n * H + y) * W + x) * ps;
      for (int c = 0; c < C; ++c) {
        const T v = px[c];
        if (sizeof(T) == 4 && thr >= 0.0f) a |= fabsf((float)v) > thr;
        else a |= (v != (T)0);
      }
    }
    const unsigned half = __ballot_sync(0xffffffffu, a);
    if (lane == 0) bits32[2 * (size_t)t + ((p >> 5) & 1)] = half;
  }
}

static int mask_grid(int ntiles) {
  int blocks = divup(ntiles, 8);
  int cap = MIE_SM_COUNT * 8;
  return blocks < cap ? (blocks > 0 ? blocks : 1) : cap;
}

// i / pieces = umulhi(i, ceil(2^32 / pieces)) for i < 32 * pieces + 256 while the error i * (pieces - 1) stays below 2^32
constexpr int MASK_MAX_PIECES = 4096;
static unsigned piece_reciprocal(int pieces) { return pieces == 1 ? 0u : (unsigned)(((1ull << 32) + pieces - 1) / pieces); }

extern "C" int mie_mask_from_delta(const float *delta, int64_t ps, int N, int C, int H, int W, float thr,
                                   uint64_t *bits, void *stream) {
  if (!delta || !bits || N <= 0 || C <= 0 || H <= 0 || W <= 0 || ps < C || !(thr >= 0.0f)) return MIE_EINVAL;
  const int ntiles = N * divup(H, 8) * divup(W, 8);
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = (C % 4 == 0) && (ps % 4 == 0) && aligned16(delta);
  if (C <= 16) {
    int blocks = divup(ntiles, 4);
    if (blocks > MIE_SM_COUNT * 8) blocks = MIE_SM_COUNT * 8;
    launch_chained(mask_words_px_kernel<float>, dim3(blocks), dim3(256), 0, st, delta, ps, C, N, H, W, thr, reinterpret_cast<unsigned *>(bits));
    return check_launch();
  }
  if (vec && C / 4 <= MASK_MAX_PIECES)
    launch_chained(mask_words_vec_kernel<true>, dim3(mask_grid(2 * ntiles)), dim3(256), 0, st, reinterpret_cast<const uint4 *>(delta), ps * 4, C / 4,
                   piece_reciprocal(C / 4), N, H, W, thr, reinterpret_cast<unsigned *>(bits));
  else launch_chained(mask_words_kernel<float>, dim3(mask_grid(ntiles)), dim3(256), 0, st, delta, ps, C, N, H, W, thr, bits);
  return check_launch();
}

extern "C" int mie_mask_from_mask(const void *mask, int elem_size, int64_t mps, int cm, int N, int H, int W,
                                  uint64_t *bits, void *stream) {
  if (!mask || !bits || N <= 0 || cm <= 0 || H <= 0 || W <= 0 || mps < cm) return MIE_EINVAL;
  const int ntiles = N * divup(H, 8) * divup(W, 8);
  cudaStream_t st = (cudaStream_t)stream;
  if (elem_size != 1 && elem_size != 4) return MIE_EUNSUPPORTED;
  const int pieces = cm * elem_size / 16;
  if (cm * elem_size % 16 == 0 && mps * elem_size % 16 == 0 && aligned16(mask) && pieces <= MASK_MAX_PIECES) {
    launch_chained(mask_words_vec_kernel<false>, dim3(mask_grid(2 * ntiles)), dim3(256), 0, st, (const uint4 *)mask, mps * elem_size, pieces,
                   piece_reciprocal(pieces), N, H, W, 0.0f, reinterpret_cast<unsigned *>(bits));
    return check_launch();
  }
  if (elem_size == 1)
    launch_chained(mask_words_kernel<uint8_t>, dim3(mask_grid(ntiles)), dim3(256), 0, st, (const uint8_t *)mask, mps, cm, N, H, W, -1.0f, bits);
  else
    launch_chained(mask_words_kernel<int32_t>, dim3(mask_grid(ntiles)), dim3(256), 0, st, (const int32_t *)mask, mps, cm, N, H, W, -1.0f, bits);
  return check_launch();
}

// ---------------------------------------------------------------------------------------------
// ordered compaction of non-zero words (warp ballot + block prefix)
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) tiles_compact_kernel(const uint64_t *__restrict__ bits, int ntiles,
                                                             int32_t *__restrict__ list, int32_t *__restrict__ counts) {
  grid_dependency_wait();
  grid_dependency_trigger();
  int n = block_ordered_compact([&](int i) { return bits[i] != 0ull; }, ntiles, list);
  if (threadIdx.x == 0) counts[0] = n;
}

extern "C" int mie_tiles_compact(const uint64_t *bits, int ntiles, int32_t *list, int32_t *counts, void *stream) {
  if (!bits || !list || !counts || ntiles <= 0) return MIE_EINVAL;
  launch_chained(tiles_compact_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, bits, ntiles, list, counts);
  return check_launch();
}

__global__ void mask_expand_kernel(const uint64_t *__restrict__ bits, int N, int H, int W, uint8_t *__restrict__ out) {
  const int TH = (H + 7) >> 3, TW = (W + 7) >> 3;
  const int64_t total = (int64_t)N * H * W;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % W), y = (int)((i / W) % H), n = (int)(i / ((int64_t)W * H));
    const uint64_t w = bits[((int64_t)n * TH + (y >> 3)) * TW + (x >> 3)];
    out[i] = (uint8_t)((w >> ((y & 7) * 8 + (x & 7))) & 1ull);
  }
}

extern "C" int mie_mask_expand(const uint64_t *bits, int N, int H, int W, uint8_t *bytes, void *stream) {
  if (!bits || !bytes || N <= 0 || H <= 0 || W <= 0) return MIE_EINVAL;
  const int64_t total = (int64_t)N * H * W;
  int blocks = (int)((total + 255) / 256);
  if (blocks > MIE_SM_COUNT * 16) blocks = MIE_SM_COUNT * 16;
  mask_expand_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(bits, N, H, W, bytes);
  return check_launch();
}

// ---------------------------------------------------------------------------------------------
// dilated output-tile set of a convolution, plus the stale list, in one launch
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) tiles_dilate_kernel(
    const uint64_t *__restrict__ in_bits, int N, int Hin, int Win, int Hout, int Wout, int k, int stride, int pad,
    const uint64_t *__restrict__ union_bits, uint64_t *__restrict__ out_bits, int32_t *__restrict__ list,
    int32_t *__restrict__ stale, int32_t *__restrict__ counts, uint8_t *__restrict__ flags) {
  grid_dependency_wait();
  grid_dependency_trigger();
  const int ntiles = N * ((Hout + 7) >> 3) * ((Wout + 7) >> 3);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < ntiles) flags[t] = dilate_flag(t, in_bits, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits);
  // the block that finishes last compacts both lists in ascending order
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(&counts[2], 1) == (int)gridDim.x - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // One chunk of consecutive tiles per thread: count it, scan the counts over the block, write it out.  (A sweep of the
  // whole block over 256 tiles at a time costs three barriers and a round trip per step: 38400 tiles took 75 us.)
  __shared__ int s_wa[8], s_wb[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int chunk = ((ntiles + 255) / 256 + 15) & ~15, lo = min((int)threadIdx.x * chunk, ntiles), hi = min(lo + chunk, ntiles);
  const bool vec = aligned16(flags);
  int ca = 0, cs = 0;
  auto sweep = [&](auto &&visit) {     // visit(first tile, flag bytes of four tiles)
    int i = lo;
    if (vec)
      for (; i + 16 <= hi; i += 16) {
        const uint4 f = __ldcg(reinterpret_cast<const uint4 *>(flags + i));
        visit(i, f.x); visit(i + 4, f.y); visit(i + 8, f.z); visit(i + 12, f.w);
      }
    for (; i < hi; ++i) visit(i, (unsigned)__ldcg(flags + i));
  };
  sweep([&](int, unsigned f) { ca += __popc(f & 0x01010101u); cs += __popc(f & 0x02020202u); });
  int ia = ca, is = cs;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, ia, d), b = __shfl_up_sync(0xffffffffu, is, d);
    if (lane >= d) { ia += a; is += b; }
  }
  if (lane == 31) { s_wa[warp] = ia; s_wb[warp] = is; }
  __syncthreads();
  int oa = ia - ca, os = is - cs, na = 0, ns = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) { oa += s_wa[w]; os += s_wb[w]; }
    na += s_wa[w];
    ns += s_wb[w];
  }
  sweep([&](int i, unsigned f) {
    for (int k = 0; f; ++k, f >>= 8) {
      if (f & 1u) list[oa++] = i + k;
      else if ((f & 2u) && stale) stale[os++] = i + k;
    }
  });
  if (threadIdx.x == 0) {
    counts[0] = na;
    counts[1] = stale ? ns : 0;
    counts[2] = 0;
  }
}

// The same for large fields, in blocks of 1024.
constexpr int DILATE_LARGE = 12288, DILATE_LARGE_THREADS = 1024;      // 9600 tiles: 10.3 us either way, 14400 12.8 and 11.3, 38400 40.3 and 18.8
__global__ void __launch_bounds__(DILATE_LARGE_THREADS) tiles_dilate_large_kernel(
    const uint64_t *__restrict__ in_bits, int N, int Hin, int Win, int Hout, int Wout, int k, int stride, int pad,
    const uint64_t *__restrict__ union_bits, uint64_t *__restrict__ out_bits, int32_t *__restrict__ list,
    int32_t *__restrict__ stale, int32_t *__restrict__ counts, uint8_t *__restrict__ flags) {
  grid_dependency_wait();
  grid_dependency_trigger();
  const int ntiles = N * ((Hout + 7) >> 3) * ((Wout + 7) >> 3);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < ntiles) flags[t] = dilate_flag(t, in_bits, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits);
  // the block that finishes last compacts both lists in ascending order
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(&counts[2], 1) == (int)gridDim.x - 1);
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // A run of consecutive tiles per warp, 128 at a time: count them, scan the counts over the block, write the tiles out.  Bound by
  // latency.  (38400 tiles: a sweep of the whole block over 256 tiles at a time took 75 us, a chunk of 150 tiles per thread of 256,
  // whose stores fall into 256 places, 40; this 19.)
  __shared__ int s_wa[DILATE_LARGE_THREADS / 32], s_wb[DILATE_LARGE_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = ((ntiles + DILATE_LARGE_THREADS / 32 - 1) / (DILATE_LARGE_THREADS / 32) + 127) & ~127, lo = min(warp * run, ntiles), hi = min(lo + run, ntiles);
  const bool vec = (reinterpret_cast<uintptr_t>(flags) & 3) == 0;
  auto four = [&](int i) {      // the flag bytes of tiles i .. i + 3
    if (vec && i + 4 <= hi) return __ldcg(reinterpret_cast<const unsigned *>(flags + i));
    unsigned f = 0;
    for (int k = 0; k < 4; ++k)
      if (i + k < hi) f |= (unsigned)__ldcg(flags + i + k) << (8 * k);
    return f;
  };
  int ca = 0, cs = 0;
#pragma unroll 4
  for (int i = lo + 4 * lane; i < hi; i += 128) {
    const unsigned f = four(i);
    ca += __popc(f & 0x01010101u);
    cs += __popc(f & 0x02020202u);
  }
  ca = __reduce_add_sync(0xffffffffu, ca);
  cs = __reduce_add_sync(0xffffffffu, cs);
  if (lane == 0) { s_wa[warp] = ca; s_wb[warp] = cs; }
  __syncthreads();
  int oa = 0, os = 0;
  int na = 0, ns = 0;
#pragma unroll
  for (int w = 0; w < DILATE_LARGE_THREADS / 32; ++w) {
    if (w == warp) { oa = na; os = ns; }
    na += s_wa[w];
    ns += s_wb[w];
  }
  unsigned next = lo + 4 * lane < hi ? four(lo + 4 * lane) : 0u;
  for (int base = lo; base < hi; base += 128) {
    const int i = base + 4 * lane;
    const unsigned f = next;
    next = i + 128 < hi ? four(i + 128) : 0u;
    const int mine = __popc(f & 0x01010101u) | __popc(f & 0x02020202u) << 16;
    int upto = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int below = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += below;
    }
    const int all = __shfl_sync(0xffffffffu, upto, 31);
    int at = oa + ((upto - mine) & 0xFFFF), as = os + ((upto - mine) >> 16);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned b = f >> (8 * k);
      if (b & 1u) list[at++] = i + k;
      else if ((b & 2u) && stale) stale[as++] = i + k;
    }
    oa += all & 0xFFFF;
    os += all >> 16;
  }
  if (threadIdx.x == 0) {
    counts[0] = na;
    counts[1] = stale ? ns : 0;
    counts[2] = 0;
  }
}

// Up to DILATE_SMALL_MAX tiles: one block keeps the flags in shared memory and compacts them itself -- no
// ticket, no fence, no round trip through global memory (the deeper levels of a UNet at batch 1 are this small;
// at 1452 tiles one block measured slower than the multi-block kernel).
constexpr int DILATE_SMALL_MAX = 512;

__global__ void __launch_bounds__(1024) tiles_dilate_small_kernel(
    const uint64_t *__restrict__ in_bits, int N, int Hin, int Win, int Hout, int Wout, int k, int stride, int pad,
    const uint64_t *__restrict__ union_bits, uint64_t *__restrict__ out_bits, int32_t *__restrict__ list,
    int32_t *__restrict__ stale, int32_t *__restrict__ counts) {
  grid_dependency_wait();
  grid_dependency_trigger();
  __shared__ uint8_t s_flags[DILATE_SMALL_MAX];
  const int ntiles = N * ((Hout + 7) >> 3) * ((Wout + 7) >> 3);
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
    s_flags[t] = dilate_flag(t, in_bits, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits);
  __syncthreads();
  int na, ns;
  block_ordered_compact2([&](int i) { return (int)s_flags[i]; }, ntiles, list, stale, &na, &ns);
  if (threadIdx.x == 0) {
    counts[0] = na;
    counts[1] = ns;
  }
}

int mie::dilate_check(const mie_tail_job &j) {
  if (!j.in_bits || !j.list || !j.counts || !j.flags || j.N <= 0 || j.Hin <= 0 || j.Win <= 0 || j.Hout <= 0 || j.Wout <= 0) return MIE_EINVAL;
  if (j.k < 1 || j.k > 7 || j.stride < 1 || j.stride > 2 || j.pad < 0 || j.pad > j.k) return MIE_EUNSUPPORTED;
  return j.out_bits && !j.stale ? MIE_EINVAL : MIE_OK;
}

extern "C" int mie_tiles_dilate(const uint64_t *in_bits, int N, int Hin, int Win, int Hout, int Wout, int k,
                                int stride, int pad, const uint64_t *union_bits, uint64_t *out_bits,
                                int32_t *list, int32_t *stale, int32_t *counts, uint8_t *flags, void *stream) {
  {
    const int s = dilate_check({in_bits, N, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits, list, stale, counts, flags});
    if (s != MIE_OK) return s;
  }
  const int ntiles = N * divup(Hout, 8) * divup(Wout, 8);
  if (ntiles <= DILATE_SMALL_MAX) {
    const int threads = ntiles <= 256 ? 256 : (ntiles <= 512 ? 512 : 1024);
    launch_chained(tiles_dilate_small_kernel, dim3(1), dim3(threads), 0, (cudaStream_t)stream, in_bits, N, Hin, Win, Hout, Wout, k, stride, pad,
                                                                       union_bits, out_bits, list, stale, counts);
    return check_launch();
  }
  if (ntiles >= DILATE_LARGE)
    launch_chained(tiles_dilate_large_kernel, dim3(divup(ntiles, DILATE_LARGE_THREADS)), dim3(DILATE_LARGE_THREADS), 0, (cudaStream_t)stream, 
      in_bits, N, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits, list, stale, counts, flags);
  else
    launch_chained(tiles_dilate_kernel, dim3(divup(ntiles, 256)), dim3(256), 0, (cudaStream_t)stream, 
      in_bits, N, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits, list, stale, counts, flags);
  return check_launch();
}
