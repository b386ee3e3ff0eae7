// What the CTA-pair convolution kernels share: taps and views of the reduction, cta_group::2 wrappers.
#pragma once
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
// source(unit, view): the tensor map of a unit, and which view it is.
template <typename Source>
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
      int tile = __shfl_sync(0xffffffffu, e + i < n_active ? lst[e + i] : -1, 0);
      have[i] = e + i < n_active;
      // an entry outside the field is reported and skipped by the epilogue; here tile 0 stands in for it
      if (have[i] && (tile < 0 || tile >= ntiles_total)) {
        if (leader) atomicOr(&counts[3], MIE_ERR_BAD_TILE);
        tile = 0;
      }
      tx8[i] = have[i] ? (tile % TWo) * 8 : 0; ty8[i] = have[i] ? ((tile / TWo) % THo) * 8 : 0; tn[i] = have[i] ? tile / (TWo * THo) : 0;
    }
    const unsigned tx_bytes = (unsigned)min(4, n_active - 4 * (item / w.n_cblk)) * (unsigned)hp * row_bytes;   // both blocks
    for (int chunk = 0; chunk < w.n_chunks && ok; ++chunk)
      for (int u = 0; u < w.units; ++u) {
        if (!first_lap) ok = __all_sync(0xffffffffu, mbar_wait(&r.empty[s], parity, abort_flag, w.limit));
        if (!ok) break;
        const unsigned bar = mapa_shared(smem_u32(&r.full[s]), 0);
        if (leader) {
          if (w.crank == 0u)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&r.full[s])), "r"(tx_bytes) : "memory");
          int v;
          const CUtensorMap *map = source(u, v);
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (have[i]) {
              unsigned dst = r.base + s * r.bytes + (unsigned)i * row_bytes;
              const int x = tx8[i] + t.x0[v], y = ty8[i] + t.y0[v];
              for (int row = 0; row < hp; ++row, dst += 2u * row_bytes) tma_load_4d_pair(dst, map, bar, chunk * 32, x, y + row, tn[i]);
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

// Barrier of the 128 threads of an epilogue set: whether all of them bring `ok`.
__device__ __forceinline__ bool set_all(int id, bool ok) {
  int r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %2, 0;\n\tbarrier.cta.red.and.pred q, %1, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
               : "=r"(r) : "r"(id), "r"((int)ok) : "memory");
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

}  // namespace
}  // namespace mie
