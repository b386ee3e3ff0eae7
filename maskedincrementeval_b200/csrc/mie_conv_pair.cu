// Masked delta convolution on CTA pairs (tcgen05 cta_group::2, TF32 inputs, FP32 accumulation), k >= 3.
//
// A cluster of two thread blocks works on four active 8x8 output tiles: one tcgen05.mma of M = 256 covers the 2 x 2
// tiles, N = NB output channels, K = 8 of the reduction over (32-channel chunk, view, filter tap).  Each block holds the
// input of its own two tiles and HALF of the filter columns, and owns the accumulator rows of its two tiles.
//   A  The halo of the two tiles is fetched once per chunk as rows of 128 bytes per pixel (32 channels, 128-byte swizzle):
//      [halo row][tile][halo column][32 ch].  Eight neighbouring pixels are one 8-row group of the operand wherever the row
//      starts -- the swizzle is a function of the shared-memory address -- so a filter tap is an offset of the descriptor.
//      (With the un-swizzled layout this replaces the copy engine moved 16 bytes per step and set the pace of large layers.)
//      Stride 2 reads four parity views of the input, one halo buffer per view.
//   B  Filter taps stream through a ring, several per stage; each block fetches its half of the columns.
// Roles (384 threads): warp 0 halo producer (one row per lane), warp 1 filter producer, warp 2 MMA issuer of the first block
// (converged, one elected lane), warps 4..11 epilogue: two sets of four warps, one per quarter of the accumulator rows,
// take 32-channel slabs in turn (blocks of 32 channels: work items in turn).  A set's slab of the reservoir arrives by TMA
// while the MMAs run, a thread finishes one pixel of it in place, and TMA stores carry the new reservoir and the output
// delta away: with plain loads and stores a slab took 5-9 us, because the instructions' operand reads fill the shared
// memory port (next paragraph) and every load / store instruction queues behind them.
// Barriers that say "operands are there" live in the first block and count the bytes of both; barriers that say "free"
// and "accumulator complete" are signalled in both blocks by one multicast commit.
//
// What bounds it: an instruction reads 4 KB of A and NB / 2 rows of B from each block's shared memory at 128 bytes per
// clock, so it takes 39 / 43 / 64 / 128 clocks for N = 32 / 64 / 128 / 256 (measured with resident operands) where the
// tensor core itself needs 16 / 32 / 64 / 128: 156 / 172 / 256 / 512 clocks per tap and chunk of four K-slices.  The filter taps
// written by TMA share that port (20.5 / 24.6 / 32.8 / 49 KB per tap and chunk in all).  What a tap and chunk takes in the
// kernel is at pair_block_width().
#include "mie_pair.cuh"

using namespace mie;

namespace mie {
namespace {

constexpr int PAIR_THREADS = 384;
constexpr int PAIR_MAX_STAGES = 12;
constexpr int PAIR_MAX_HALOS = 4;
constexpr int PAIR_SLAB_BYTES = 128 * 128;    // 32 channels of the 128 pixels of a block, as two tiles of 64 rows of 128 bytes

struct PairParams {
  TcParams c;
  PairTaps t;
  int wp, hp;            // halo extent
  int halos;             // halo buffers
  int tps;               // taps per ring stage
  int slab_bufs;         // shared-memory slabs per epilogue set: output (+ reservoir (+ carry))
};

struct PairMaps {
  CUtensorMap in[4], w, out, res, emitted;
};

// 16 accumulator columns of this lane's row; two accumulators (taddr2 != taddr) are added.
__device__ __forceinline__ void tmem_ld16_pair(unsigned taddr, unsigned taddr2, float *v) {
  unsigned r[16], t[16];
#define MIE_LD16(R, A)                                                                                                                             \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"             \
               : "=r"(R[0]), "=r"(R[1]), "=r"(R[2]), "=r"(R[3]), "=r"(R[4]), "=r"(R[5]), "=r"(R[6]), "=r"(R[7]), "=r"(R[8]), "=r"(R[9]),           \
                 "=r"(R[10]), "=r"(R[11]), "=r"(R[12]), "=r"(R[13]), "=r"(R[14]), "=r"(R[15])                                                      \
               : "r"(A))
  MIE_LD16(r, taddr);
  if (taddr2 != taddr) {
    MIE_LD16(t, taddr2);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]) + __uint_as_float(t[i]);
  } else {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
  }
#undef MIE_LD16
}

__device__ __forceinline__ void tma_load_slab(unsigned smem_addr, const CUtensorMap *map, unsigned bar, int c0, int x, int y, int n) {
  tma_load_4d_raw(smem_addr, map, bar, c0, x, y, n);
}
// One pixel, 16 channels (quads h0 .. h0 + 3 of a slab): v, the accumulator values; xs / es / os, shared addresses of the pixel's rows of the
// reservoir, carry and output slabs (quad h of row r sits at h ^ (r & 7): the 128-byte swizzle of TMA).  Returns whether the
// group was sent: a thresholded layer sends it when any of its channels moved by more than the threshold.
template <int ACT, bool THR>
__device__ __forceinline__ bool pair_group(const TcParams &p, const float *v, unsigned xs, unsigned es, unsigned os, int sw, int h0, const float *addend, int nq) {
  float4 o[4];
  bool flag = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int h = h0 + i;
    float4 d = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    if (addend && h < nq) d = f4add(d, *reinterpret_cast<const float4 *>(addend + 4 * h));
    o[i] = d;
    if (ACT != MIE_ACT_NONE) {
      const float4 x = lds4(xs + ((h ^ sw) << 4)), xn = f4add(x, d);
      float4 b;
      if (THR && es) b = lds4(es + ((h ^ sw) << 4));
      else b = make_float4(tc_act<ACT>(p.act, x.x), tc_act<ACT>(p.act, x.y), tc_act<ACT>(p.act, x.z), tc_act<ACT>(p.act, x.w));
      o[i] = make_float4(tc_act<ACT>(p.act, xn.x) - b.x, tc_act<ACT>(p.act, xn.y) - b.y, tc_act<ACT>(p.act, xn.z) - b.z, tc_act<ACT>(p.act, xn.w) - b.w);
      sts4(xs + ((h ^ sw) << 4), xn);
    }
    const float thr = THR ? p.thr : 0.0f;
    flag |= fabsf(o[i].x) > thr || fabsf(o[i].y) > thr || fabsf(o[i].z) > thr || fabsf(o[i].w) > thr;
  }
  // Of a quad past the last channel the slabs hold zeros, and f(0) - 0 is not zero for a sigmoid that is measured against the carry.
  if (THR && __builtin_expect(nq - h0 < 4, 0)) {
    flag = false;
#pragma unroll
    for (int i = 0; i < 3; ++i) flag |= h0 + i < nq && (fabsf(o[i].x) > p.thr || fabsf(o[i].y) > p.thr || fabsf(o[i].z) > p.thr || fabsf(o[i].w) > p.thr);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) sts4(os + (((h0 + i) ^ sw) << 4), (THR && !flag) ? make_float4(0.f, 0.f, 0.f, 0.f) : o[i]);
  return flag;
}
template <bool THR>
__device__ __forceinline__ bool pair_group_act(const TcParams &p, const float *v, unsigned xs, unsigned es, unsigned os, int sw, int h0, const float *addend, int nq) {
  switch (p.act) {
    case MIE_ACT_RELU: return pair_group<MIE_ACT_RELU, THR>(p, v, xs, es, os, sw, h0, addend, nq);
    case MIE_ACT_SIGMOID:
    case MIE_ACT_TANH: return pair_group<MIE_ACT_SIGMOID, THR>(p, v, xs, es, os, sw, h0, addend, nq);
    default: return pair_group<MIE_ACT_NONE, THR>(p, v, xs, es, os, sw, h0, addend, nq);
  }
}

// The MMA issuer (first block of the pair, one converged warp).  Two accumulators take alternate taps.  (Two issuing warps
// with alternate stages measured slower: the ring then needs twice the slots for the same look-ahead.)
struct PairIssue {
  int item0, item_step, n_items, n_chunks, cin, NB, tps, nviews;
  unsigned nacc, tmem_base, a_base, b_base, row_bytes, halo_bytes, tap_bytes, stage_bytes, stages, halos, limit;
};
__device__ __forceinline__ void pair_issue(const PairIssue a, const PairTapTable &t, unsigned long long *b_full, unsigned long long *b_empty,
                                        unsigned long long *a_full, unsigned long long *a_empty, unsigned long long *acc_full,
                                        unsigned long long *acc_empty, volatile int *abort_flag) {
  unsigned idesc = make_idesc_tf32(a.NB);
  idesc = (idesc & ~(31u << 24)) | (16u << 24);                              // M = 256
  const unsigned long long b_tmpl = make_smem_desc(0), a_tmpl = make_smem_desc(0, a.row_bytes);   // 8-row groups: one halo row apart
  const unsigned long long b_hi = b_tmpl & 0xFFFFFFFF00000000ull, a_hi = a_tmpl & 0xFFFFFFFF00000000ull;
  const unsigned lo_flags = (unsigned)(b_tmpl & 0xFFFF0000ull);
  unsigned bs = 0, bpar = 0, as = 0, apar = 0, item_idx = 0, stage_addr = a.b_base;
  for (int item = a.item0; item < a.n_items; item += a.item_step, ++item_idx) {
    const unsigned buf = item_idx & 1u;
    if (item_idx >= 2 && !mbar_wait(&acc_empty[buf], ((item_idx >> 1) - 1) & 1u, abort_flag, a.limit)) return;
    tc_fence_after();
    const unsigned tmem_d = a.tmem_base + buf * a.nacc * (unsigned)a.NB;
    unsigned ntap = 0;
    for (int chunk = 0; chunk < a.n_chunks; ++chunk) {
      const unsigned nks = (unsigned)min(4, (a.cin - chunk * 32 + 7) >> 3);  // K-slices holding real channels
      for (int v = 0; v < a.nviews; ++v) {
        if (!mbar_wait(&a_full[as], apar, abort_flag, a.limit)) return;
        const unsigned halo = lo_flags | ((a.a_base + as * a.halo_bytes) >> 4);
        const int end = t.first[v + 1];
        for (int i = t.first[v]; i < end; i += a.tps) {
          const int nt = min(a.tps, end - i);
          unsigned b_lo = lo_flags | (stage_addr >> 4), off = (unsigned)t.off[i];
          if (!mbar_wait(&b_full[bs], bpar, abort_flag, a.limit)) return;
          tc_fence_after();
          for (int k = 0; k < nt; ++k, b_lo += a.tap_bytes >> 4, ++ntap) {
            const unsigned a_lo = halo + off;
            off = (unsigned)t.off[i + k + 1];     // the next tap's, while this one is issued (the table has a spare entry)
            pair_mma(tmem_d + (ntap & (a.nacc - 1u)) * (unsigned)a.NB, a_hi | a_lo, b_hi | b_lo, idesc, ntap >= a.nacc, nks);
          }
          pair_commit(&b_empty[bs]);
          stage_addr += a.stage_bytes;
          if (++bs == a.stages) { bs = 0; bpar ^= 1u; stage_addr = a.b_base; }
        }
        pair_commit(&a_empty[as]);
        if (++as == a.halos) { as = 0; apar ^= 1u; }
      }
    }
    pair_commit(&acc_full[buf]);
  }
}

// MODE 0: tile list from a launch before; PAIR_OWN: own tiles (see mie_tc.cuh); PAIR_HEAD: the first block makes the list.
// Separate instantiations: with the code of PAIR_HEAD compiled in, the list mode issued an MMA every 68-79 clocks instead of
// 34-50 (decoder 0 / 2 of 8 streams 260x346: 187 / 436 us against 115 / 220 us).
constexpr int PAIR_OWN = 1, PAIR_HEAD = 2;
template <int MODE>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
conv_pair_kernel(const PairParams P, const __grid_constant__ PairMaps maps) {
  constexpr bool OWN = MODE == PAIR_OWN;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // both blocks of a pair must lay out their shared memory alike: descriptors and barrier offsets are used in both
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const TcParams &p = P.c;
  const int NB = p.nb;
  const unsigned row_bytes = (unsigned)P.wp * 128u;                              // one halo row of one tile
  const unsigned halo_bytes = ((unsigned)P.hp * 2u * row_bytes + 1023u) & ~1023u;
  const unsigned tap_bytes = (unsigned)NB * 64u;                                 // this block's half of the columns of one tap
  const unsigned stage_bytes = tap_bytes * (unsigned)P.tps;
  __shared__ unsigned long long b_full[PAIR_MAX_STAGES], b_empty[PAIR_MAX_STAGES], a_full[PAIR_MAX_HALOS], a_empty[PAIR_MAX_HALOS],
      acc_full[2], acc_empty[2], slab_full[2];
  __shared__ OwnSharedT<OWN> s_own;
  __shared__ PairTapTable s_tap;
  __shared__ unsigned s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const unsigned crank = cluster_ctarank();
  const int bid = (int)(blockIdx.x >> 1), nblk = (int)(gridDim.x >> 1);          // clusters
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(&maps.in[0])) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(&maps.w)) : "memory");
  }
  const int THo = (p.hout + 7) >> 3, TWo = (p.wout + 7) >> 3;
  const int ntiles_total = p.n * THo * TWo;
  // Two item buffers; blocks of up to 128 channels have two accumulators in each, taken by alternate taps and added in the
  // epilogue: the tensor core truncates every time it adds to an accumulator, so half the additions mean half that bias.
  const unsigned nacc = NB <= 128 ? 2u : 1u;
  const unsigned tmem_cols = 2u * nacc * (unsigned)NB;                           // NB is a power of two >= 32

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < P.halos; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], NB == 32 ? 8 : 16); mbar_init(&slab_full[b], 1); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 3) {
    for (int i = lane; i < 50; i += 32) s_tap.off[i] = i < 49 ? (int)P.t.off[i] * 8 : 0;
    if (lane < 5) s_tap.first[lane] = P.t.first[lane];
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = s_tmem_base;
  pair_cluster_sync();    // neither block may signal the other's barriers before they exist

  // everything above touched no global memory: it may overlap the tail of the previous kernel in the stream
  grid_dependency_wait();
  grid_dependency_trigger();
  bool head_ok = true;
  if constexpr (MODE == PAIR_HEAD) {
    head_ok = run_head_job(p.head, p.spin_limit);
    if (tid == (int)blockDim.x - 1) count_head_job_passed(p.head);
  }
  const int n_cblk = p.cout_pad / NB;
  const bool own_multi = OWN && n_cblk > 1;      // several clusters finish a tile: its word goes through the scratch
  int item0 = bid, item_step = nblk, n_active;
  const int32_t *lst = p.list;
  if constexpr (OWN) {
    const int G = nblk / n_cblk, g = bid / n_cblk;
    own_scan(p.head.in_bits, p.head.Hin, p.head.Win, p.head.Hout, p.head.Wout, p.head.k, p.head.stride, p.head.pad, p.head.union_bits,
             (bid % n_cblk == 0 && crank == 0u) ? p.head.out_bits : nullptr, s_own, g < G ? g : 0x3fffffff, G, ntiles_total, false);
    lst = s_own.list;
    n_active = s_own.n_active;
    item0 = bid % n_cblk;
    item_step = n_cblk;
    if (!own_multi) {
      // the words this block alone will OR into: cleared by this block, so that nothing has to be ordered across the pair
      for (int i = tid; i < n_active; i += PAIR_THREADS)
        if (((i >> 1) & 1) == (int)crank) reinterpret_cast<unsigned long long *>(p.out_bits32)[lst[i]] = 0ull;
      __syncthreads();
    }
  } else {
    n_active = head_ok ? min(p.counts[0], p.max_tiles) : 0;
  }
  n_active = __shfl_sync(0xffffffffu, n_active, 0);     // uniform, for the compiler too
  const int n_items = ((n_active + 3) >> 2) * n_cblk;
  const int n_chunks = p.cin_pad >> 5;
  const unsigned b_base = smem_u32(smem);
  const unsigned a_base = b_base + (((unsigned)p.stages * stage_bytes + 1023u) & ~1023u);
  unsigned char *epi = smem + (a_base - b_base) + (size_t)P.halos * halo_bytes;   // slabs of the epilogue sets

  const PairWork work = {item0, item_step, n_items, n_cblk, n_chunks, P.t.nviews, crank, p.spin_limit, p.withhold_loads};
  if (warp == 0) {
    // =========================== halo producer ===========================
    const PairRing ring = {a_full, a_empty, a_base, halo_bytes, (unsigned)P.halos};
    pair_produce_halos<false>(work, ring, P.t, P.hp, row_bytes, lst, n_active, ntiles_total, TWo, THo, p.counts, &s_abort,
                       [&](int u, int &v) { v = u; return &maps.in[u]; });
  } else if (warp == 1) {
    // =========================== filter producer ===========================
    const PairRing ring = {b_full, b_empty, b_base, stage_bytes, (unsigned)p.stages};
    pair_produce_filter(work, ring, P.t, P.tps, tap_bytes, (int)crank * (NB >> 1), NB, &s_abort, [](int u) { return u; },
                        [&](int) { return 2u * tap_bytes; },
                        [&](int, int tap, unsigned dst, unsigned bar, int row, int chunk) { tma_load_4d_pair(dst, &maps.w, bar, 0, row, chunk, tap); });
  } else if (warp == 2) {
    if (crank == 0u) {
      PairIssue a;
      a.item0 = item0; a.item_step = item_step; a.n_items = n_items; a.n_chunks = n_chunks; a.cin = p.cin; a.NB = NB; a.nacc = nacc;
      a.tmem_base = tmem_base; a.a_base = a_base; a.b_base = b_base; a.row_bytes = row_bytes; a.halo_bytes = halo_bytes;
      a.tap_bytes = tap_bytes; a.stage_bytes = stage_bytes; a.stages = (unsigned)p.stages; a.halos = (unsigned)P.halos;
      a.tps = P.tps; a.nviews = P.t.nviews; a.limit = p.spin_limit;
      pair_issue(a, s_tap, b_full, b_empty, a_full, a_empty, acc_full, acc_empty, &s_abort);
    }
  } else if (warp >= 4) {
    // =========================== epilogue (warps 4..11) ===========================
    // Accumulator row m = 32q + lane is pixel row 2q + (lane >> 4), column lane & 7 of tile (lane >> 3) & 1.
    const int q = warp & 3, set = (warp - 4) >> 2;
    if constexpr (OWN) { if (bid % n_cblk == 0 && crank == 0u) tc_zero_stale_own(p, s_own, THo, TWo, tid - 128, PAIR_THREADS - 128); }
    else if (head_ok) tc_zero_stale(p, ntiles_total, THo, TWo, tid - 128, PAIR_THREADS - 128);
    const int n_slabs = NB >> 5;
    const bool thresholded = p.thr > 0.0f || p.emitted != nullptr, has_res = p.act != MIE_ACT_NONE;
    const int slot = (lane >> 3) & 1, prow = 2 * q + (lane >> 4), pcol = lane & 7, row = slot * 64 + prow * 8 + pcol;
    unsigned char *slab = epi + (size_t)set * P.slab_bufs * PAIR_SLAB_BYTES;       // output | reservoir | carry
    const unsigned slab_u32 = smem_u32(slab), os = slab_u32 + row * 128, xs = os + PAIR_SLAB_BYTES, es = p.emitted ? xs + PAIR_SLAB_BYTES : 0u;
    const bool chief = q == 0 && elect_one();          // issues the set's copies
    unsigned item_idx = 0, lap = 0;
    for (int item = item0; item < n_items; item += item_step, ++item_idx) {
      const int s0 = n_slabs == 1 ? 0 : set, ds = n_slabs == 1 ? 1 : 2;
      if (n_slabs == 1 && (int)(item_idx & 1u) != set) continue;
      const int quad = item / n_cblk, cb = item - quad * n_cblk;
      const unsigned buf = item_idx & 1u;
      int tile[2], tx[2], ty[2], tn[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int e = 4 * quad + 2 * (int)crank + s;
        int t = e < n_active ? lst[e] : -1;
        if (t < 0 || t >= ntiles_total) t = -1;
        tile[s] = t;
        tx[s] = (t >= 0) ? (t % TWo) * 8 : 0; ty[s] = (t >= 0) ? ((t / TWo) % THo) * 8 : 0; tn[s] = (t >= 0) ? t / (TWo * THo) : 0;
      }
      const bool valid = (slot ? tile[1] : tile[0]) >= 0 && (slot ? ty[1] : ty[0]) + prow < p.hout && (slot ? tx[1] : tx[0]) + pcol < p.wout;
      const int64_t pix = valid ? (int64_t)((slot ? tn[1] : tn[0]) * p.hout + (slot ? ty[1] : ty[0]) + prow) * p.wout + (slot ? tx[1] : tx[0]) + pcol : 0;
      bool sent = false, ok = true;
      for (int sl = s0; sl < n_slabs; sl += ds, ++lap) {
        const int co = cb * NB + sl * 32;
        if (chief) {
          // the stores of the previous slab have read shared memory; the loads of this one may overwrite it
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          const unsigned bar = smem_u32(&slab_full[set]), ntiles = (tile[0] >= 0) + (tile[1] >= 0);
          const unsigned bytes = (has_res && co < p.cout) ? ntiles * (PAIR_SLAB_BYTES / 2) * (p.emitted ? 2u : 1u) : 0u;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
          if (bytes)
#pragma unroll
            for (int s = 0; s < 2; ++s)
              if (tile[s] >= 0) {
                tma_load_slab(slab_u32 + PAIR_SLAB_BYTES + s * (PAIR_SLAB_BYTES / 2), &maps.res, bar, co, tx[s], ty[s], tn[s]);
                if (p.emitted) tma_load_slab(slab_u32 + 2 * PAIR_SLAB_BYTES + s * (PAIR_SLAB_BYTES / 2), &maps.emitted, bar, co, tx[s], ty[s], tn[s]);
              }
        }
        __syncwarp();
        // A wait that gives up does not leave the loop on its own: the four warps of the set meet at the barrier below in
        // every slab and leave together.
        if (sl == s0) {
          ok = mbar_wait(&acc_full[buf], (item_idx >> 1) & 1u, &s_abort, p.spin_limit);
          tc_fence_after();
        }
        ok = __all_sync(0xffffffffu, ok);
        if (ok) ok = mbar_wait(&slab_full[set], lap & 1u, &s_abort, p.spin_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
          const unsigned taddr = tmem_base + buf * nacc * (unsigned)NB + (unsigned)(sl * 32) + ((unsigned)(q * 32) << 16), acc2 = (nacc - 1u) * (unsigned)NB;
          const float *ad = (p.addend && valid) ? p.addend + pix * p.addend_ps + co : nullptr;
          const int nq = (p.cout - co) >> 2;      // channel quads of the slab that exist
#pragma unroll 1
          for (int h0 = 0; h0 < 8; h0 += 4) {
            float v[16];
            tmem_ld16_pair(taddr + 4 * h0, taddr + acc2 + 4 * h0, v);
            if (h0 == 4 && sl + ds >= n_slabs) {     // last read of this warp: hand the accumulator back
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&acc_empty[buf]), 0));
            }
            const bool f = thresholded ? pair_group_act<true>(p, v, xs, es, os, pcol, h0, ad, nq) : pair_group_act<false>(p, v, xs, es, os, pcol, h0, ad, nq);
            sent |= valid && f && co < p.cout;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the slabs, before the copy engine reads them
        }
        ok = set_all(1 + set, ok);
        if (!ok) break;
        if (chief && co < p.cout) {
#pragma unroll
          for (int s = 0; s < 2; ++s)
            if (tile[s] >= 0) {
              const unsigned half = s * (PAIR_SLAB_BYTES / 2);
              tma_store_slab(slab_u32 + half, &maps.out, co, tx[s], ty[s], tn[s]);
              if (has_res) tma_store_slab(slab_u32 + PAIR_SLAB_BYTES + half, &maps.res, co, tx[s], ty[s], tn[s]);
              if (p.emitted) tma_add_slab(slab_u32 + half, &maps.emitted, co, tx[s], ty[s], tn[s]);   // the carry advances by what was sent
            }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      if (!ok) break;
      // ballot bytes: [tile 0 row 2q][tile 1 row 2q][tile 0 row 2q+1][tile 1 row 2q+1]
      const unsigned bal = __ballot_sync(0xffffffffu, sent);
      const int ts = lane == 8 ? tile[1] : tile[0];
      if ((lane == 0 || lane == 8) && ts >= 0) {
        const unsigned rows = ((bal >> lane) & 0xFFu) | (((bal >> (16 + lane)) & 0xFFu) << 8);
        if (own_multi) own_contribute(p, ts, q >> 1, rows << ((q & 1) * 16), n_cblk * (n_slabs == 1 ? 4 : 8));
        else if (rows) atomicOr(p.out_bits32 + 2 * (size_t)ts + (q >> 1), rows << ((q & 1) * 16));
      }
    }
    if (chief) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  // ---- teardown ----
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    if (tid == 0) atomicOr(&p.counts[3], MIE_ERR_WAIT_EXPIRED);
    // copies and instructions that may still be in flight land before shared and tensor memory are released
    if (warp == 0) { const long long t0 = clock64(); while (clock64() - t0 < 2000000) { } }
    __syncthreads();
  }
  pair_cluster_sync();     // every wait above is bounded, so both blocks get here whatever happened
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
  run_tail_job(p.tail);
}

}  // namespace

// Output channels per pair: the width whose rounds of work items over the 74 clusters cost least.  Wide blocks are cheaper
// per column, small layers need the narrow ones to occupy the machine.  The costs are relative ones per tap and chunk, chosen
// on whole networks.  Measured by themselves (256 -> NB channels, every tile active, from a list, the slope from four to eight
// rounds, 1965 MHz), k = 3 / 5 / 7: 32 channels 212 / 187 / 178 clocks, 64 250 / 203 / 201, 128 398 / 329 / 349, 256 721 / 660 /
// 825.  Against the best width of each of 338 shapes (k 3 to 7, 64 and 256 -> 64 to 512 channels, 8 to 700 quads, from a list) the
// table's choice takes 1.02 times as long on average and 1.3 times at worst (one round of 256 channels at 45 quads, where 64 channels
// take three).  That sweep leaves out what one block per layer saves: its blocks find their own tiles without a dilation launch.
static int pair_block_width(const mie_conv_args *a) {
  static const struct { int nb, cost; } width[4] = {{256, 512}, {128, 270}, {64, 200}, {32, 164}};
  const int64_t quads = ((int64_t)a->max_tiles + 3) / 4, clusters = MIE_SM_COUNT / 2;
  int best = 32;
  int64_t best_cost = INT64_MAX;
  for (const auto &w : width) {
    if (a->cout_pad % w.nb) continue;
    const int64_t items = quads * (a->cout_pad / w.nb), cost = (items + clusters - 1) / clusters * w.cost;
    if (cost < best_cost) { best_cost = cost; best = w.nb; }
  }
  return best;
}

// Own-tiles mode: the groups of n_cblk clusters that share the tiles out, or 0 for the separate dilation launch.
// Not where several clusters finish a tile (kind 8, off by default): its word then goes through a scratch word and a
// ticket per epilogue warp, which costs more than the launch it saves (gates 0 / 1 / 2, one stream: 27.8 / 25.6 / 24.0 us
// against 23.6 / 23.1 / 22.2 us with the dilation launch).  Layers of 64 channels in two blocks keep the mode.
// A group's share of the tiles must fit the list in its shared memory.
static int pair_own_groups(const mie_conv_args *a, int n_cblk, int clusters, int64_t ntiles) {
  const int groups = clusters / n_cblk;
  const int64_t pairs = ((int64_t)a->max_tiles + 1) / 2;
  const int kind = n_cblk > 1 && a->cout_pad > 64 ? 8 : a->stride == 2 ? 1 : 4;
  return (g_opt_own_kernels & kind) && groups >= 1 && 2 * ((pairs + groups - 1) / groups) <= OWN_MAX && a->max_tiles == ntiles ? groups : 0;
}

// Host-side rule; tc_eligible() has already accepted the layer.
bool pair_takes(const mie_conv_args *a) { return a->k >= 3 && a->k <= 7; }

int launch_conv_pair(const mie_conv_args *a, cudaStream_t st) {
  PairParams P;
  memset(&P, 0, sizeof(P));
  TcParams &p = P.c;
  p.spin_limit = g_opt_spin_limit;
  p.withhold_loads = g_opt_withhold_loads;
  p.cin = a->cin; p.cout = a->cout; p.cout_pad = a->cout_pad;
  p.cin_pad = (a->cin + 31) / 32 * 32;
  p.n = a->n; p.hin = a->hin; p.win = a->win; p.hout = a->hout; p.wout = a->wout;
  p.k = a->k; p.stride = a->stride; p.pad = a->pad;
  p.list = a->list; p.stale = a->stale; p.counts = a->counts; p.max_tiles = a->max_tiles;
  p.out = a->out; p.out_ps = a->out_ps; p.out_bits32 = reinterpret_cast<unsigned int *>(a->out_bits);
  p.act = a->act; p.thr = a->thr; p.res = a->res; p.res_ps = a->res_ps;
  p.emitted = a->emitted; p.emitted_ps = a->emitted_ps; p.addend = a->addend; p.addend_ps = a->addend_ps;
  p.tail = tail_for_kernel(a->tail);
  p.head = tail_for_kernel(a->head);
  p.nb = pair_block_width(a);

  const int s = a->stride, k = a->k;
  pair_make_taps(k, s, a->pad, &P.t, &P.wp);
  P.hp = P.wp;

  // Shared memory: epilogue slabs, halo buffers, and the filter ring in what is left.  Taps per stage: enough that a stage
  // lasts several times the 120 clocks its barriers cost the issuer.
  P.slab_bufs = 1 + (a->act != MIE_ACT_NONE) + (a->emitted != nullptr);
  const int halo_bytes = (P.hp * 2 * P.wp * 128 + 1023) & ~1023;
  const int budget = 220 * 1024 - 2 * P.slab_bufs * PAIR_SLAB_BYTES;
  P.halos = PAIR_MAX_HALOS;
  while (P.halos > 2 && budget - P.halos * halo_bytes < 64 * 1024) --P.halos;
  int stage_bytes = 0;
  for (;; p.nb >>= 1) {      // (large halos beside three slabs per set leave little for the ring: narrower blocks then)
    P.tps = p.nb == 256 ? 1 : p.nb == 128 ? 3 : p.nb == 64 ? 5 : 9;
    while (P.tps > 1 && 3 * P.tps * p.nb * 64 > budget - P.halos * halo_bytes) --P.tps;
    stage_bytes = P.tps * p.nb * 64;
    p.stages = (budget - P.halos * halo_bytes) / stage_bytes;
    if (p.stages > PAIR_MAX_STAGES) p.stages = PAIR_MAX_STAGES;
    if (p.stages >= 2) break;
    if (p.nb == 32) return MIE_EUNSUPPORTED;
  }
  const size_t smem = (size_t)((p.stages * stage_bytes + 1023) & ~1023) + (size_t)P.halos * halo_bytes + 2 * P.slab_bufs * PAIR_SLAB_BYTES + 1024;

  PairMaps maps;
  memset(&maps, 0, sizeof(maps));
  const cuuint32_t box_in[4] = {32, (cuuint32_t)P.wp, 1, 1};
  for (int v = 0; v < P.t.nviews; ++v) {
    const int py = s == 2 ? v >> 1 : 0, px = s == 2 ? v & 1 : 0;
    const cuuint64_t dims[4] = {(cuuint64_t)a->cin, (cuuint64_t)((a->win - px + s - 1) / s), (cuuint64_t)((a->hin - py + s - 1) / s), (cuuint64_t)a->n};
    const cuuint64_t str[3] = {(cuuint64_t)a->in_ps * 4 * s, (cuuint64_t)a->win * a->in_ps * 4 * s, (cuuint64_t)a->hin * a->win * a->in_ps * 4};
    if (!tc_encode(&maps.in[v], 4, a->in + ((int64_t)py * a->win + px) * a->in_ps, dims, str, box_in, CU_TENSOR_MAP_SWIZZLE_128B)) return MIE_EINVAL;
  }
  {
    const cuuint64_t nch = (cuuint64_t)(p.cin_pad / 32);
    const cuuint64_t dims[4] = {32, (cuuint64_t)a->cout_pad, nch, (cuuint64_t)(k * k)};
    const cuuint64_t str[3] = {128, (cuuint64_t)a->cout_pad * 128, nch * a->cout_pad * 128};
    const cuuint32_t box_w[4] = {32, (cuuint32_t)(p.nb / 2), 1, 1};
    if (!tc_encode(&maps.w, 4, a->wpacked_tc, dims, str, box_w, CU_TENSOR_MAP_SWIZZLE_128B)) return MIE_EINVAL;
  }

  {
    // epilogue slabs: 32 channels of one tile; what lies outside the field is neither read nor written
    const cuuint32_t box[4] = {32, 8, 8, 1};
    auto slab_map = [&](CUtensorMap *m, const float *base, int64_t ps) {
      const cuuint64_t dims[4] = {(cuuint64_t)a->cout, (cuuint64_t)a->wout, (cuuint64_t)a->hout, (cuuint64_t)a->n};
      const cuuint64_t str[3] = {(cuuint64_t)ps * 4, (cuuint64_t)a->wout * ps * 4, (cuuint64_t)a->hout * a->wout * ps * 4};
      return tc_encode(m, 4, base, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    if (!slab_map(&maps.out, a->out, a->out_ps) || (a->act != MIE_ACT_NONE && !slab_map(&maps.res, a->res, a->res_ps)) ||
        (a->emitted && !slab_map(&maps.emitted, a->emitted, a->emitted_ps)))
      return MIE_EINVAL;
  }

  const int n_cblk = a->cout_pad / p.nb;
  const int64_t items = ((int64_t)a->max_tiles + 3) / 4 * n_cblk;
  int64_t clusters = items < MIE_SM_COUNT / 2 ? items : MIE_SM_COUNT / 2;
  if (a->own_tiles) {
    const int64_t ntiles = (int64_t)a->n * divup(a->hout, 8) * divup(a->wout, 8);
    const int groups = pair_own_groups(a, n_cblk, (int)clusters, ntiles);
    if (groups) {
      p.own = 1;
      p.head = *a->head;
      p.own_words = static_cast<unsigned long long *>(a->own_scratch);
      p.own_tickets = reinterpret_cast<int *>(static_cast<char *>(a->own_scratch) + 8 * ntiles);
      clusters = groups * n_cblk;
    } else {
      const mie_tail_job *h = a->head;
      const int r = mie_tiles_dilate(h->in_bits, h->N, h->Hin, h->Win, h->Hout, h->Wout, h->k, h->stride, h->pad, h->union_bits,
                                     h->out_bits, h->list, h->stale, h->counts, h->flags, st);
      if (r != MIE_OK) return r;
      p.head = mie_tail_job{};
    }
  }
  static int smem_set[3][MAX_DEVICES] = {{0}};
  auto launch = [&](auto kernel, int mode) {
    const int r = ensure_dynamic_smem(kernel, smem_set[mode], smem);
    if (r != MIE_OK) return r;
    launch_chained_cluster(kernel, dim3((unsigned)(2 * clusters)), dim3(PAIR_THREADS), smem, st, 2, P, maps);
    return check_launch();
  };
  if (p.own) return launch(conv_pair_kernel<PAIR_OWN>, PAIR_OWN);
  if (p.head.list) return launch(conv_pair_kernel<PAIR_HEAD>, PAIR_HEAD);
  return launch(conv_pair_kernel<0>, 0);
}

}  // namespace mie
