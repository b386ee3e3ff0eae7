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
// shared memory, so that its largest value lies in [2^15, 2^16) and does not round up to 2^16: a value is held to 2^-52 of that, which is 24
// bits down to 2^-27 of it and 22 at 2^-29.  A few values smaller than that but zero, in whatever unit, are taken out of the halo and
// listed, the halo's inverse scale gets a negative sign, and the epilogue multiplies them with FP32 instructions.  (Of normal values one halo
// in 8000 has one, in the dense pass and in steps alike.  The line lies where FireFlowNet's step is not slower for it: from 2^-27 on, with
// two such items a step, 336 us, from 2^-30 on 311, without 309; most of it is the fetching of instructions that are not at hand.)  Many such
// values stay in the parts, down to 16 bits; a halo in which that is not enough, because values 2^-36 of the largest are among them, is marked
// with a NaN, as are halos with an infinity, a NaN or values above 2^100, and the epilogue computes their pixels with FP32 instructions.  (To
// compute all halos with many small values so, as a network with closed gates makes them, takes a hundred times as long as the layer.)
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
// The same with every product that leaves 2^-35 of the largest: lo x [hi | lo], and where the channels are 16 at most (`third`) those of third
// parts, which lie where the second K-slice would be (input: of lo, filter: of hi; scaled like lo).  id: of N = 2 CB columns.
__device__ __forceinline__ void pair_mma_full(unsigned d1, unsigned d2, unsigned long long a_desc, unsigned long long b_desc, unsigned id, unsigned accumulate,
                                              unsigned nks, unsigned third) {
  asm volatile(
      "{\n\t.reg .pred p, q, e, r1, r3;\n\t.reg .b64 a1, a2, a3, b1;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "setp.gt.and.u32 r1, %6, 1, e;\n\t"
      "setp.ne.and.b32 r3, %7, 0, e;\n\t"
      "add.u64 a1, %2, 2;\n\tadd.u64 a2, %2, 4;\n\tadd.u64 a3, %2, 6;\n\tadd.u64 b1, %3, 2;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %2, %3, %4, p;\n\t"
      "@r1 tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %4, q;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%1], a2, %3, %4, p;\n\t"
      "@r1 tcgen05.mma.cta_group::2.kind::f16 [%1], a3, b1, %4, q;\n\t"
      "@r3 tcgen05.mma.cta_group::2.kind::f16 [%1], %2, b1, %4, q;\n\t"
      "@r3 tcgen05.mma.cta_group::2.kind::f16 [%1], a3, %3, %4, q;\n\t}"
      ::"r"(d1), "r"(d2), "l"(a_desc), "l"(b_desc), "r"(id), "r"(accumulate), "r"(nks), "r"(third)
      : "memory");
}
// Instruction descriptor: FP16 operands, both K-major, FP32 accumulator, M = 256.
__device__ __forceinline__ unsigned make_idesc_f16_pair(int n) { return (1u << 4) | ((unsigned)(n >> 3) << 17) | (16u << 24); }
// Rows of 64 bytes, 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ unsigned long long make_smem_desc_64(unsigned smem_addr) {
  return (unsigned long long)((smem_addr & 0x3FFFFu) >> 4) | (unsigned long long)1 << 16 | (unsigned long long)(512 >> 4) << 32 |
         (unsigned long long)1 << 46 | (unsigned long long)4 << 61;
}

// The exponent field that a largest magnitude (its bits) is scaled by; the scale and its inverse.
__device__ __forceinline__ unsigned split_exponent(unsigned m) { return min(max((m + 0x1000u) >> 23, 16u), 254u); }
__device__ __forceinline__ float split_scale(unsigned e) { return __uint_as_float((269u - e) << 23); }
__device__ __forceinline__ float split_inverse(unsigned e) { return __uint_as_float((e - 15u) << 23); }

// Two fp32 operations in an instruction.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
// Eight channels.  THIRD: also what two parts leave, scaled like lo (exact: two bits).
template <bool THIRD>
__device__ __forceinline__ void split_fp16(const float *v, float scale, float4 &hi, float4 &lo, float4 &third) {
  unsigned h[4], l[4], m[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = make_float2(v[2 * j], v[2 * j + 1]), a = mul2(x, make_float2(scale, scale));
    const __half2 t = __float22half2_rn(a);
    // (the scaling, by powers of two, and the differences are exact)
    const float2 f = __half22float2(__hneg2(t)), r = mul2(fma2(x, make_float2(scale, scale), f), make_float2(2048.0f, 2048.0f));
    const __half2 u = __float22half2_rn(r);
    h[j] = *reinterpret_cast<const unsigned *>(&t);
    l[j] = *reinterpret_cast<const unsigned *>(&u);
    if (THIRD) {
      const float2 g = __half22float2(u);
      const __half2 w = __floats2half2_rn(r.x - g.x, r.y - g.y);
      m[j] = *reinterpret_cast<const unsigned *>(&w);
    }
  }
  hi = make_float4(__uint_as_float(h[0]), __uint_as_float(h[1]), __uint_as_float(h[2]), __uint_as_float(h[3]));
  lo = make_float4(__uint_as_float(l[0]), __uint_as_float(l[1]), __uint_as_float(l[2]), __uint_as_float(l[3]));
  if (THIRD) third = make_float4(__uint_as_float(m[0]), __uint_as_float(m[1]), __uint_as_float(m[2]), __uint_as_float(m[3]));
}

// The splitting warps (t: thread among theirs).  A halo lies in shared memory as `rows` rows of 128 bytes (32 fp32 channels of a
// pixel, 128-byte swizzle; [halo row][tile][halo column]) and is replaced in place by 64 bytes of hi and 64 bytes of lo.  A thread
// takes eight channels: it reads pieces 2 c and 2 c + 1 of a row and writes pieces c and 4 + c; the eight rows of a warp are dealt such that
// neighbouring lanes hold rows whose swizzles differ in bits 0 and 2, so that neither reads nor writes meet in a bank.
// What it costs: one read and one write of the halo through shared memory (400 clocks of its port for a 3x3 layer's 25 KB), and a
// chain of about 2200 clocks a unit (read 600, largest and smallest value of all warps 400, split and write 1100), beside the
// instructions of the unit before.
constexpr int SPLIT_WARPS = 8, SPLIT_PASS = 8 * SPLIT_WARPS;      // rows of a pass
constexpr int SPLIT_REGS = 288 / SPLIT_PASS + (288 % SPLIT_PASS != 0);      // passes held in registers: halos up to 12 x 12; larger ones (7x7) read the rest twice
constexpr int SPLIT_BELOW = 29;      // binades below the largest value from which values are taken out, if they are few
constexpr int SPLIT_APART = 36;      // ... from which a halo with many such values is not split
constexpr int SPLIT_LISTED = 4;
struct SplitSmall {                          // values taken out, and where they stood: tile << 13 | halo row << 9 | halo column << 5 | channel
  float value[SPLIT_LISTED];
  unsigned short at[SPLIT_LISTED];           // (SPLIT_NONE behind the last one)
};
constexpr unsigned SPLIT_NONE = 0xFFFFu;
struct __align__(16) SplitShared {
  SplitSmall small[SPLIT_RING];              // of the units whose inverse scale is negative
  float red[2][SPLIT_WARPS];
  unsigned short least[2][SPLIT_WARPS];
  float inv[SPLIT_RING];                       // inverse scale of a unit's halo (negative: values were taken out; NaN: not split) ...
  unsigned long long inv_full[SPLIT_RING];     // ... and that it is there
  // the splitting warps' order to the one that takes values out: the halo, its exponent field | ring unit << 8 | tiles << 12 (~0: it may go)
  unsigned take_base, take;
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
// How many threads of the splitting warps bring `yes`.
__device__ __forceinline__ unsigned set_count(bool yes) {
  unsigned r;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.popc.u32 %0, 3, %2, p;\n\t}" : "=r"(r) : "r"((unsigned)yes), "n"(32 * SPLIT_WARPS) : "memory");
  return r;
}
// The splitting warps and the one that takes values out: an order is there, or carried out.
__device__ __forceinline__ void split_meet() { asm volatile("bar.sync 4, %0;" ::"n"(32 * SPLIT_WARPS + 32) : "memory"); }
// The warp that takes out of a halo the values below 2^-SPLIT_BELOW of its largest, but zero: lists them in ascending order and sets them to
// zero.  A warp of its own: as a branch of the splitting warps it cost FireFlowNet's step 3 % without being run (registers, and the
// instructions in between).
__device__ __forceinline__ void pair_take_out(SplitShared &sh, int rows, int wp, int lane) {
  for (;;) {
    split_meet();
    const unsigned order = sh.take, base = sh.take_base;
    if (order == ~0u) return;
    const int tiles = (int)(order >> 12);
    const float thr = __uint_as_float(((order & 255u) - SPLIT_BELOW) << 23);
    SplitSmall &list = sh.small[order >> 8 & 15u];
    const int piece = lane & 7;
    unsigned n = 0u;
#pragma unroll 1
    for (int r0 = 0; r0 < rows; r0 += 4) {
      const int row = r0 + (lane >> 3), line = row / wp;
      const bool live = row < rows && (line & 1) < tiles;
      const unsigned at = base + (unsigned)row * 128u + (unsigned)((piece ^ (row & 7)) << 4);
      const float4 v = lds4_if(at, live);
      float x[4] = {v.x, v.y, v.z, v.w};
      bool here = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool out = x[j] != 0.0f && fabsf(x[j]) < thr;
        const unsigned all = __ballot_sync(0xffffffffu, out), i = n + __popc(all & ((1u << lane) - 1u));
        if (out && i < (unsigned)SPLIT_LISTED) {
          list.value[i] = x[j];
          list.at[i] = (unsigned short)((line & 1) << 13 | (line >> 1) << 9 | (row - line * wp) << 5 | (4 * piece + j));
        }
        if (out) x[j] = 0.0f;
        here |= out;
        n += __popc(all);
      }
      sts4_if(at, make_float4(x[0], x[1], x[2], x[3]), here);
    }
    if (lane == 0 && n < (unsigned)SPLIT_LISTED) list.at[n] = (unsigned short)SPLIT_NONE;
    split_meet();
  }
}
// THIRD: of halos of 16 channels at most third parts too, in the place of the channels that do not exist (pair_mma_full).
template <int REGS, bool THIRD>
__device__ __forceinline__ void pair_split_halos_in(const PairWork &w, const PairRing &r, unsigned long long *ready, int rows, int wp, int n_active, int t,
                                                 SplitShared &sh, volatile int *abort_flag) {
  const int lane = t & 31, cw = t >> 5, passes = (rows + SPLIT_PASS - 1) / SPLIT_PASS;
  const int c = lane & 3, row0 = cw * 8 + (int)((0x63724150u >> (4 * (lane >> 2))) & 7u), sw = row0 & 7;
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
      // twice the smallest magnitude's bits less one: a zero is the largest number there is
      auto smallest = [](const float *v, unsigned m) {
        unsigned k[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) k[j] = 2u * __float_as_uint(v[j]) - 1u;
        return __vimin3_u32(__vimin3_u32(__vimin3_u32(__vimin3_u32(m, k[0], k[1]), k[2], k[3]), k[4], k[5]), k[6], k[7]);
      };
      float v[REGS][8], m = 0.0f;
      unsigned least = 0xFFFFFFFFu;
#pragma unroll
      for (int it = 0; it < REGS; ++it) read(it, v[it]);
#pragma unroll
      for (int it = 0; it < REGS; ++it) { m = largest(v[it], m); least = smallest(v[it], least); }
#pragma unroll 1
      for (int it = REGS; it < passes; ++it) {
        float x[8];
        read(it, x);
        m = largest(x, m);
        least = smallest(x, least);
      }
      m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));      // (of non-negative floats, NaN above all)
      least = __reduce_min_sync(0xffffffffu, least);
      if (lane == 0) { sh.red[unit & 1u][cw] = m; sh.least[unit & 1u][cw] = (unsigned short)(least >> 16); }
      if (!set_all<32 * SPLIT_WARPS>(3, ok)) return;
      m = 0.0f;
#pragma unroll
      for (int i = 0; i < SPLIT_WARPS; i += 2) m = max3_abs(m, sh.red[unit & 1u][i], sh.red[unit & 1u][i + 1]);
      const uint4 l = *reinterpret_cast<const uint4 *>(sh.least[unit & 1u]);      // (a power of two counts as the binade below, which does no harm)
      const unsigned l2 = __vminu2(__vminu2(l.x, l.y), __vminu2(l.z, l.w));
      least = min(l2 & 0xFFFFu, l2 >> 16) >> 8;
      const unsigned mb = __float_as_uint(m);
      const unsigned e = split_exponent(mb);
      const float scale = split_scale(e);
      float inv = split_inverse(e);
      if (mb > 0x71800000u) {
        inv = __uint_as_float(0x7FC00000u);
      } else if (__builtin_expect(mb && e > SPLIT_BELOW && least < e - SPLIT_BELOW, 0)) {
        // few enough for the list?
        const float thr = __uint_as_float((e - SPLIT_BELOW) << 23);
        unsigned few = 0u;
#pragma unroll 1
        for (int it = 0; it < passes; ++it) {
          float x[8];
          read(it, x);
#pragma unroll
          for (int j = 0; j < 8; ++j) few += x[j] != 0.0f && fabsf(x[j]) < thr;
        }
        if (set_count(few >= 1u) + set_count(few >= 2u) <= (unsigned)SPLIT_LISTED && !set_count(few >= 3u)) {
          if (t == 0) { sh.take_base = base; sh.take = e | (unit % SPLIT_RING) << 8 | (unsigned)tiles << 12; }
          split_meet();
          split_meet();
          inv = -inv;
        } else if (e - least > SPLIT_APART) {
          inv = __uint_as_float(0x7FC00000u);
        }
#pragma unroll
        for (int it = 0; it < REGS; ++it) read(it, v[it]);
      }
      if (t == 0) {
        sh.inv[unit % SPLIT_RING] = inv;
        mbar_arrive(&sh.inv_full[unit % SPLIT_RING]);
      }
      auto write = [&](int it, const float *x) {
        float4 hi, lo, third;
        split_fp16<THIRD>(x, scale, hi, lo, third);
        const unsigned by = (unsigned)(it * SPLIT_PASS * 128);
        sts4_if(base + wr0 + by, hi, live >> it & 1u);
        sts4_if(base + wr1 + by, lo, (!THIRD || c < 2) && live >> it & 1u);
        if (THIRD) sts4_if(base + at + (unsigned)(((6 + c) & 7) ^ sw) * 16u + by, third, c < 2 && live >> it & 1u);
      };
#pragma unroll
      for (int it = 0; it < REGS; ++it) write(it, v[it]);
#pragma unroll 1
      for (int it = REGS; it < passes; ++it) {
        float x[8];
        read(it, x);
        __syncwarp();      // in place: the lanes of a row read before one of them writes
        write(it, x);
      }
      // The instructions read it through the asynchronous proxy, also those that the other block issues: each block's rows are read by its own
      // SM's tensor core.  What the arrival orders is this block's shared memory alone, so the default (block) scope of its release is
      // enough; with release.cluster it took 1300 clocks, as long as the splitting.
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&ready[s]), 0));
      if (++s == r.count) { s = 0; parity ^= 1u; }
    }
  }
}
// By the passes that the halo takes: one that reads no row costs as many instructions as one that does (3x3: a fifth).
template <bool THIRD>
__device__ __forceinline__ void pair_split_halos(const PairWork &w, const PairRing &r, unsigned long long *ready, int rows, int wp, int n_active, int t,
                                                 SplitShared &sh, volatile int *abort_flag) {
  if (rows <= 3 * SPLIT_PASS) pair_split_halos_in<3, THIRD>(w, r, ready, rows, wp, n_active, t, sh, abort_flag);
  else if (rows <= 4 * SPLIT_PASS) pair_split_halos_in<4, THIRD>(w, r, ready, rows, wp, n_active, t, sh, abort_flag);
  else pair_split_halos_in<SPLIT_REGS, THIRD>(w, r, ready, rows, wp, n_active, t, sh, abort_flag);
  if (t == 0) sh.take = ~0u;      // (the splitting warps leave together, also where a wait gave up)
  split_meet();
}

}  // namespace
}  // namespace mie
