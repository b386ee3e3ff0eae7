// What the CTA-pair convolution kernels share: taps and views of the reduction, cta_group::2 wrappers.
#pragma once
#include <cuda_fp16.h>
#include "mie_tc.cuh"

namespace mie {
namespace {

// The reduction of one channel chunk: for every view of the input a halo origin (relative to the tile's first pixel, in
// view pixels) and its taps, each an index into the filter and an offset into the halo in units of 128 bytes.
struct PairTaps {
  int nviews;
  int first[5];
  int x0[4], y0[4];
  unsigned char tap[49], off[49];
};

// Views and taps of a k x k filter with this stride and padding; *wp: halo extent (rows and columns) of a tile in a view.
// Stride 1: one view, the input itself.  Stride 2: four parity views (row parity * 2 + column parity).
static inline void pair_make_taps(int k, int stride, int pad, PairTaps *t, int *wp) {
  const int s = stride;
  int lo[2] = {0, 0}, span = k;                 // first offset of a parity, largest number of offsets of a parity
  if (s == 2) {
    int cnt[2] = {0, 0};
    for (int i = 0; i < k; ++i) {
      const int d = i - pad, par = d & 1, off = (d - par) / 2;
      if (!cnt[par]++) lo[par] = off;           // offsets ascend with i
    }
    span = cnt[0] > cnt[1] ? cnt[0] : cnt[1];
  }
  *wp = 8 + span - 1;
  t->nviews = s == 2 ? 4 : 1;
  int nt = 0;
  for (int v = 0; v < t->nviews; ++v) {
    const int py = v >> 1, px = v & 1;
    t->first[v] = nt;
    t->y0[v] = s == 2 ? lo[py] : -pad;
    t->x0[v] = s == 2 ? lo[px] : -pad;
    for (int ky = 0; ky < k; ++ky)
      for (int kx = 0; kx < k; ++kx) {
        const int dy = ky - pad, dx = kx - pad;
        if (s == 2 && ((dy & 1) != py || (dx & 1) != px)) continue;
        const int oy = s == 2 ? (dy - py) / 2 - lo[py] : ky, ox = s == 2 ? (dx - px) / 2 - lo[px] : kx;
        t->tap[nt] = (unsigned char)(ky * k + kx);
        t->off[nt] = (unsigned char)(oy * 2 * *wp + ox);
        ++nt;
      }
  }
  t->first[t->nviews] = nt;
}

__device__ __forceinline__ void tma_load_4d_pair(unsigned smem_addr, const CUtensorMap *map, unsigned bar_cluster_addr, int c0, int c1,
                                                 int c2, int c3) {
  // .cta_group::2: the barrier may lie in the other block of the pair
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_addr), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Up to four K-slices (8 channels = 32 bytes each) of one tap.  Called by a converged warp; the electing happens inside the
// asm block, next to the instructions it guards, so that the predicate stays uniform for the compiler.
__device__ __forceinline__ void pair_mma(unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc, unsigned accumulate,
                                         unsigned nks) {
  asm volatile(
      "{\n\t.reg .pred p, q, e, r1, r2, r3;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "setp.gt.and.u32 r1, %5, 1, e;\n\tsetp.gt.and.u32 r2, %5, 2, e;\n\tsetp.gt.and.u32 r3, %5, 3, e;\n\t"
      "add.u64 a1, %1, 2;\n\tadd.u64 a2, %1, 4;\n\tadd.u64 a3, %1, 6;\n\t"
      "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t"
      "@r1 tcgen05.mma.cta_group::2.kind::tf32 [%0], a1, b1, %3, q;\n\t"
      "@r2 tcgen05.mma.cta_group::2.kind::tf32 [%0], a2, b2, %3, q;\n\t"
      "@r3 tcgen05.mma.cta_group::2.kind::tf32 [%0], a3, b3, %3, q;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(nks)
      : "memory");
}
// Arrives on the barrier at the same offset in both blocks once the instructions issued so far have completed.
__device__ __forceinline__ void pair_commit(unsigned long long *bar) {
  asm volatile("{\n\t.reg .pred e;\n\t.reg .b16 m;\n\telect.sync _|e, 0xffffffff;\n\tmov.b16 m, 3;\n\t"
               "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(smem_u32(bar))
               : "memory");
}
// "This warp has read the accumulator": an arrival on a barrier of the other (or this) block of the pair.  What it orders is
// tensor memory (tcgen05.wait::ld and tcgen05.fence before it), no shared or global data; with release.cluster semantics the
// arrival first waits for every store of the warp to drain, about 1000 clocks per segment of conv_exact_kernel.
__device__ __forceinline__ void mbar_arrive_remote(unsigned cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void pair_cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

__device__ __forceinline__ void tma_store_slab(unsigned smem_addr, const CUtensorMap *map, int c0, int x, int y, int n) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_addr), "r"(c0), "r"(x), "r"(y), "r"(n) : "memory");
}

__device__ __forceinline__ void tma_add_slab(unsigned smem_addr, const CUtensorMap *map, int c0, int x, int y, int n) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_addr), "r"(c0), "r"(x), "r"(y), "r"(n) : "memory");
}

// Waits for three barriers at once (a barrier may be named twice): one round of their latency where three waits take three.
__device__ __forceinline__ bool mbar_wait3(unsigned b0, unsigned p0, unsigned b1, unsigned p1, unsigned b2, unsigned p2, volatile int *abort_flag, unsigned limit) {
  for (unsigned it = 0; it < limit; ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p, q, r;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 r, [%5], %6;\n\t"
        "and.pred p, p, q;\n\tand.pred p, p, r;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(b0), "r"(p0), "r"(b1), "r"(p1), "r"(b2), "r"(p2)
        : "memory");
    if (done) return true;
    if ((it & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// Taps of a reduction as the issuing warps read them.
struct PairTapTable {
  int first[5];
  int off[50];       // offset of the tap in the halo, in descriptor units
};

// What the two producer warps of a pair kernel walk through: items of four listed tiles and a column block, channel chunks, and
// per chunk `units` halos (the views of the input, in two parts where the kernel splits its operands).
struct PairWork {
  int item0, item_step, n_items, n_cblk, n_chunks, units;
  unsigned crank, limit;
  int withhold;      // self-test: load nothing
};
struct PairRing {
  unsigned long long *full, *empty;      // "operands are there" in the first block, "free" in each
  unsigned base, bytes, count;           // of a buffer
};

// Waits until the last uses of a ring's buffers are over: nothing may signal this block's barriers after it has left.  s and
// parity: the next buffer and the parity of its next release; first_lap: no buffer has been waited for yet.
__device__ __forceinline__ void pair_drain(const PairRing &r, unsigned s, unsigned parity, bool first_lap, bool ok, volatile int *abort_flag, unsigned limit) {
  for (int i = 0; i < (int)r.count && ok && !*abort_flag; ++i) {
    if (first_lap && (unsigned)i >= s) break;
    if (first_lap) ok = mbar_wait(&r.empty[i], 0u, abort_flag, limit);
    else {
      ok = mbar_wait(&r.empty[s], parity, abort_flag, limit);
      if (++s == r.count) { s = 0; parity ^= 1u; }
    }
  }
}

// Halo producer, one converged warp: one copy per halo row and tile, issued by one elected lane.  (With a row per lane the copies
// are issued one by one all the same, at several times the cost -- no uniform registers --, and paced every layer.)
// source(unit, view): the tensor map of a unit, and which view it is.  LOCAL: each block's own barrier counts its own bytes (the
// block works on the halo before the instructions read it); else the first block's barrier counts those of both.
template <bool LOCAL, typename Source>
__device__ __forceinline__ void pair_produce_halos(const PairWork &w, const PairRing &r, const PairTaps &t, int hp, unsigned row_bytes, const int32_t *lst,
                                                   int n_active, int ntiles_total, int TWo, int THo, int32_t *counts, volatile int *abort_flag,
                                                   Source source) {
  const unsigned leader = elect_one();
  unsigned s = 0, parity = 0;
  bool first_lap = true, ok = true;
  for (int item = w.item0; item < w.n_items && ok && !w.withhold; item += w.item_step) {
    const int e = 4 * (item / w.n_cblk) + 2 * (int)w.crank;
    int tx8[2], ty8[2], tn[2];
    bool have[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      int tile = __shfl_sync(0xffffffffu, e + i >= n_active ? -1 : LOCAL && !lst ? e + i : lst[e + i], 0);      // no list: every tile
      have[i] = e + i < n_active;
      // an entry outside the field is reported and skipped by the epilogue; here tile 0 stands in for it
      if (have[i] && (tile < 0 || tile >= ntiles_total)) {
        if (leader) atomicOr(&counts[3], MIE_ERR_BAD_TILE);
        tile = 0;
      }
      tx8[i] = have[i] ? (tile % TWo) * 8 : 0; ty8[i] = have[i] ? ((tile / TWo) % THo) * 8 : 0; tn[i] = have[i] ? tile / (TWo * THo) : 0;
    }
    const unsigned tx_bytes = (LOCAL ? (unsigned)have[0] + (unsigned)have[1] : (unsigned)min(4, n_active - 4 * (item / w.n_cblk))) * (unsigned)hp * row_bytes;
    for (int chunk = 0; chunk < w.n_chunks && ok; ++chunk)
      for (int u = 0; u < w.units; ++u) {
        if (!first_lap) ok = __all_sync(0xffffffffu, mbar_wait(&r.empty[s], parity, abort_flag, w.limit));
        if (!ok) break;
        const unsigned bar = LOCAL ? smem_u32(&r.full[s]) : mapa_shared(smem_u32(&r.full[s]), 0);
        if (leader) {
          if (LOCAL || w.crank == 0u)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&r.full[s])), "r"(tx_bytes) : "memory");
          int v;
          const CUtensorMap *map = source(u, v);
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (have[i]) {
              unsigned dst = r.base + s * r.bytes + (unsigned)i * row_bytes;
              const int x = tx8[i] + t.x0[v], y = ty8[i] + t.y0[v];
              for (int row = 0; row < hp; ++row, dst += 2u * row_bytes) {
                if (LOCAL) tma_load_4d_raw(dst, map, bar, chunk * 32, x, y + row, tn[i]);
                else tma_load_4d_pair(dst, map, bar, chunk * 32, x, y + row, tn[i]);
              }
            }
        }
        __syncwarp();
        if (++s == r.count) { s = 0; if (!first_lap) parity ^= 1u; first_lap = false; }
      }
  }
  if (!w.withhold) pair_drain(r, s, parity, first_lap, ok, abort_flag, w.limit);
}

// Filter producer, one converged warp: stages of `tps` taps.  view(unit): whose taps these are; bytes(unit): what a tap brings to
// both blocks; load(unit, tap, dst, bar, row, chunk): issues the copies of this block's part of a tap; row: of its column block's
// first filter row, row0 + column block * row_step.  A lane whose wait gave up stays with its warp until the end of the chunk,
// where they leave together: a vote for every stage took 0.6 % of an eight-stream 480x640 step.
template <typename View, typename Bytes, typename Load>
__device__ __forceinline__ void pair_produce_filter(const PairWork &w, const PairRing &r, const PairTaps &t, int tps, unsigned tap_bytes, int row0,
                                                    int row_step, volatile int *abort_flag, View view, Bytes bytes, Load load) {
  const unsigned leader = elect_one();
  unsigned s = 0, parity = 0, stage_addr = r.base;
  bool first_lap = true, ok = true;
  for (int item = w.item0; item < w.n_items && ok && !w.withhold; item += w.item_step) {
    const int row = row0 + (item % w.n_cblk) * row_step;
    for (int chunk = 0; chunk < w.n_chunks && ok; ++chunk) {
      for (int u = 0; u < w.units; ++u) {
        const int v = view(u), end = t.first[v + 1];
        for (int i = t.first[v]; i < end; i += tps) {
          if (!first_lap && ok) ok = mbar_wait(&r.empty[s], parity, abort_flag, w.limit);
          const int nt = min(tps, end - i);
          if (leader && ok) {
            if (w.crank == 0u)
              asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&r.full[s])), "r"((unsigned)nt * bytes(u)) : "memory");
            const unsigned bar = mapa_shared(smem_u32(&r.full[s]), 0);
            for (int k = 0; k < nt; ++k) load(u, (int)t.tap[i + k], stage_addr + (unsigned)k * tap_bytes, bar, row, chunk);
          }
          __syncwarp();
          stage_addr += r.bytes;
          if (++s == r.count) { s = 0; stage_addr = r.base; if (!first_lap) parity ^= 1u; first_lap = false; }
        }
      }
      ok = __all_sync(0xffffffffu, ok);
    }
  }
  if (!w.withhold) pair_drain(r, s, parity, first_lap, ok, abort_flag, w.limit);
}

// Barrier of the threads of an epilogue set (or of the splitting warps): whether all of them bring `ok`.
template <int THREADS = 128>
__device__ __forceinline__ bool set_all(int id, bool ok) {
  int r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %2, 0;\n\tbarrier.cta.red.and.pred q, %1, %3, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
               : "=r"(r) : "r"(id), "r"((int)ok), "n"(THREADS) : "memory");
  return r != 0;
}

// Shared-memory accesses by explicit address.  Through generic pointers (float4 * into the dynamic shared memory) the whole
// kernel was compiled such that an MMA took 85-117 clocks to issue instead of 40-65, even where the accesses never ran:
// decoder 0 / 2 of 8 streams 260x346 went from 184 / 416 us to 112 / 197 us with these two functions.
__device__ __forceinline__ float4 lds4(unsigned addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts4(unsigned addr, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}


// ---------------------------------------------------------------------------------------------------------------
// fp32 operands as two FP16 numbers each.  An operand v, scaled by a power of two s, is hi = fp16(s v) and lo = fp16(2^11 (s v - hi)),
// rounded to nearest: together they hold v to 2^-24, as two TF32 numbers do, but an instruction takes 16 of them where it takes 8
// TF32 numbers.  (A scaled FP16 split: Ootomo and Yokota, 2022.)  The input's scale is chosen for every halo in
// shared memory, so that its largest value lies in [2^14, 2^15): a value keeps its 24 bits down to 2^-28 of that, and an absolute
// step of 2^-49 of it below.  Halos for which that would not do -- an infinity, a NaN, values above 2^100, or above 2^14 beside
// values 2^-36 of it -- are marked (inverse scale NaN), and the epilogue computes their pixels with FP32 instructions.
// ---------------------------------------------------------------------------------------------------------------
constexpr unsigned SPLIT_RING = 16;      // inverse scales kept: more than halo buffers and segment accumulators in flight
constexpr float SPLIT_LO = 1.0f / 2048.0f;

// [D1] += A hi x [B hi | B lo], [D2] += A lo x B hi for up to two K-slices (16 channels = 32 bytes each).  A: rows of 128 bytes, 32 hi then
// 32 lo; B: rows of 64 bytes.  Called by a converged warp.
__device__ __forceinline__ void pair_mma_split(unsigned d1, unsigned d2, unsigned long long a_desc, unsigned long long b_desc, unsigned id1, unsigned id2,
                                               unsigned accumulate, unsigned nks) {
  asm volatile(
      "{\n\t.reg .pred p, q, e, r1;\n\t.reg .b64 a1, a2, a3, b1;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "setp.gt.and.u32 r1, %7, 1, e;\n\t"
      "add.u64 a1, %2, 2;\n\tadd.u64 a2, %2, 4;\n\tadd.u64 a3, %2, 6;\n\tadd.u64 b1, %3, 2;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %2, %3, %4, p;\n\t"
      "@r1 tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %4, q;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%1], a2, %3, %5, p;\n\t"
      "@r1 tcgen05.mma.cta_group::2.kind::f16 [%1], a3, b1, %5, q;\n\t}"
      ::"r"(d1), "r"(d2), "l"(a_desc), "l"(b_desc), "r"(id1), "r"(id2), "r"(accumulate), "r"(nks)
      : "memory");
}
// Instruction descriptor: FP16 operands, both K-major, FP32 accumulator, M = 256.
__device__ __forceinline__ unsigned make_idesc_f16_pair(int n) { return (1u << 4) | ((unsigned)(n >> 3) << 17) | (16u << 24); }
// Rows of 64 bytes, 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ unsigned long long make_smem_desc_64(unsigned smem_addr) {
  return (unsigned long long)((smem_addr & 0x3FFFFu) >> 4) | (unsigned long long)1 << 16 | (unsigned long long)(512 >> 4) << 32 |
         (unsigned long long)1 << 46 | (unsigned long long)4 << 61;
}

__device__ __forceinline__ void split_fp16(const float *v, float scale, float4 &hi, float4 &lo) {      // eight channels
  unsigned h[4], l[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = v[2 * j] * scale, b = v[2 * j + 1] * scale;
    const __half2 t = __floats2half2_rn(a, b);
    const float2 f = __half22float2(t);
    const __half2 u = __floats2half2_rn((a - f.x) * 2048.0f, (b - f.y) * 2048.0f);
    h[j] = *reinterpret_cast<const unsigned *>(&t);
    l[j] = *reinterpret_cast<const unsigned *>(&u);
  }
  hi = make_float4(__uint_as_float(h[0]), __uint_as_float(h[1]), __uint_as_float(h[2]), __uint_as_float(h[3]));
  lo = make_float4(__uint_as_float(l[0]), __uint_as_float(l[1]), __uint_as_float(l[2]), __uint_as_float(l[3]));
}

// The splitting warps (t: thread among theirs).  A halo lies in shared memory as `rows` rows of 128 bytes (32 fp32 channels of a
// pixel, 128-byte swizzle; [halo row][tile][halo column]) and is replaced in place by 64 bytes of hi and 64 bytes of lo.  A thread
// takes eight channels: it reads pieces 2 c and 2 c + 1 of a row and writes pieces c and 4 + c; the eight rows of a warp are dealt such that
// neighbouring lanes hold rows whose swizzles differ in bits 0 and 2, so that neither reads nor writes meet in a bank.
// What it costs: one read and one write of the halo through shared memory (400 clocks of its port for a 3x3 layer's 25 KB), and a
// chain of about 2200 clocks a unit (read 600, largest value of all warps 400, split and write 1100), beside the instructions of
// the unit before.
constexpr int SPLIT_WARPS = 8, SPLIT_PASS = 8 * SPLIT_WARPS;      // rows of a pass
constexpr int SPLIT_REGS = 288 / SPLIT_PASS + (288 % SPLIT_PASS != 0);      // passes held in registers: halos up to 12 x 12; larger ones (7x7) read the rest twice
struct SplitShared {
  float red[2][SPLIT_WARPS];
  unsigned least[SPLIT_WARPS];
  float inv[SPLIT_RING];                       // inverse scale of a unit's halo (NaN: marked) ...
  unsigned long long inv_full[SPLIT_RING];     // ... and that it is there
};
__device__ __forceinline__ float max3_abs(float a, float b, float c) {      // of magnitudes; a NaN stays
  float d;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Predicated accesses (no branch: the passes of a halo are one stretch of code that the compiler can interleave)
__device__ __forceinline__ float4 lds4_if(unsigned addr, bool on) {
  float4 v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
               "@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"((unsigned)on) : "memory");
  return v;
}
__device__ __forceinline__ void sts4_if(unsigned addr, float4 v, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n\t}"
               ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"((unsigned)on) : "memory");
}
// The smallest magnitude but zero of the rows in `live` that start at r0 and r1.
__device__ __noinline__ unsigned split_least(unsigned r0, unsigned r1, unsigned live) {
  unsigned least = 0x7FFFFFFFu;
  for (int it = 0; live >> it; ++it) {
    if (!(live >> it & 1u)) continue;
    const float4 a = lds4(r0 + (unsigned)(it * SPLIT_PASS * 128)), b = lds4(r1 + (unsigned)(it * SPLIT_PASS * 128));
    const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) { const unsigned u = __float_as_uint(x[j]) & 0x7FFFFFFFu; if (u) least = min(least, u); }
  }
  return least;
}
__device__ __forceinline__ void pair_split_halos(const PairWork &w, const PairRing &r, unsigned long long *ready, int rows, int wp, int n_active, int t,
                                                 SplitShared &sh, volatile int *abort_flag) {
  const int lane = t & 31, cw = t >> 5, c = lane & 3;
  const int row0 = cw * 8 + (int)((0x63724150u >> (4 * (lane >> 2))) & 7u);
  const int sw = row0 & 7, passes = (rows + SPLIT_PASS - 1) / SPLIT_PASS;
  const unsigned at = (unsigned)row0 * 128u, rd0 = at + (unsigned)((2 * c) ^ sw) * 16u, rd1 = at + (unsigned)((2 * c + 1) ^ sw) * 16u,
                 wr0 = at + (unsigned)(c ^ sw) * 16u, wr1 = at + (unsigned)((4 + c) ^ sw) * 16u;
  // which of the thread's rows hold input: of two tiles, or of the first alone (what lies in an absent tile's rows is none)
  unsigned both = 0, one = 0;
  for (int it = 0; it < passes; ++it)
    if (row0 + SPLIT_PASS * it < rows) { both |= 1u << it; if (!(((row0 + SPLIT_PASS * it) / wp) & 1)) one |= 1u << it; }
  unsigned s = 0, parity = 0, unit = 0;
  for (int item = w.item0; item < w.n_items; item += w.item_step) {
    const int tiles = n_active - 4 * (item / w.n_cblk) - 2 * (int)w.crank;
    const unsigned live = tiles >= 2 ? both : tiles == 1 ? one : 0u;
    for (int cu = 0; cu < w.n_chunks * w.units; ++cu, ++unit) {
      const bool ok = mbar_wait(&r.full[s], parity, abort_flag, w.limit);
      const unsigned base = r.base + s * r.bytes;
      auto read = [&](int it, float *v) {
        const float4 a = lds4_if(base + rd0 + (unsigned)(it * SPLIT_PASS * 128), live >> it & 1u), b = lds4_if(base + rd1 + (unsigned)(it * SPLIT_PASS * 128), live >> it & 1u);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      };
      auto largest = [](const float *v, float m) { return max3_abs(max3_abs(max3_abs(max3_abs(m, v[0], v[1]), v[2], v[3]), v[4], v[5]), v[6], v[7]); };
      float v[SPLIT_REGS][8], m = 0.0f;
#pragma unroll
      for (int it = 0; it < SPLIT_REGS; ++it) read(it, v[it]);
#pragma unroll
      for (int it = 0; it < SPLIT_REGS; ++it) m = largest(v[it], m);
#pragma unroll 1
      for (int it = SPLIT_REGS; it < passes; ++it) {
        float x[8];
        read(it, x);
        m = largest(x, m);
      }
      m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));      // (of non-negative floats, NaN above all)
      if (lane == 0) sh.red[unit & 1u][cw] = m;
      if (!set_all<32 * SPLIT_WARPS>(3, ok)) return;
      m = 0.0f;
#pragma unroll
      for (int i = 0; i < SPLIT_WARPS; i += 2) m = max3_abs(m, sh.red[unit & 1u][i], sh.red[unit & 1u][i + 1]);
      const unsigned mb = __float_as_uint(m);
      bool wide = false;
      if (mb >= 0x46800000u) {      // 2^14 or more: is it too much for what lies beside it?
        unsigned least = split_least(base + rd0, base + rd1, live);
        least = __reduce_min_sync(0xffffffffu, least);
        if (lane == 0) sh.least[cw] = least;
        set_all<32 * SPLIT_WARPS>(3, true);
#pragma unroll
        for (int i = 0; i < SPLIT_WARPS; ++i) least = min(least, sh.least[i]);
        wide = mb > 0x71800000u || (mb >> 23) - (least >> 23) > 36u;
      }
      const unsigned e = min(max(mb >> 23, 15u), 254u);
      const float scale = __uint_as_float((268u - e) << 23);
      if (t == 0) {
        sh.inv[unit % SPLIT_RING] = wide ? __uint_as_float(0x7FC00000u) : __uint_as_float((e - 14u) << 23);
        mbar_arrive(&sh.inv_full[unit % SPLIT_RING]);
      }
      auto write = [&](int it, const float *x) {
        float4 hi, lo;
        split_fp16(x, scale, hi, lo);
        sts4_if(base + wr0 + (unsigned)(it * SPLIT_PASS * 128), hi, live >> it & 1u);
        sts4_if(base + wr1 + (unsigned)(it * SPLIT_PASS * 128), lo, live >> it & 1u);
      };
#pragma unroll
      for (int it = 0; it < SPLIT_REGS; ++it) write(it, v[it]);
#pragma unroll 1
      for (int it = SPLIT_REGS; it < passes; ++it) {
        float x[8];
        read(it, x);
        __syncwarp();      // in place: the lanes of a row read before one of them writes
        write(it, x);
      }
      // The instructions read it through the asynchronous proxy.  What the arrival orders is this block's shared memory alone, so the
      // default (block) scope of its release is enough; with release.cluster it took 1300 clocks, as long as the splitting.
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&ready[s]), 0));
      if (++s == r.count) { s = 0; parity ^= 1u; }
    }
  }
}

}  // namespace
}  // namespace mie
