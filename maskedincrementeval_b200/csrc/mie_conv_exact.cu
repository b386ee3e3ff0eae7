// Dense evaluation (the refresh pass) in fp32 precision on the tensor cores, on CTA pairs like mie_conv_pair.cu.
//
// Every operand is two TF32 numbers, hi = round(v) and lo = round(v - hi) (round to nearest: together they hold v to 2^-24),
// and a product is hi*hi + hi*lo + lo*hi; the dropped lo*lo is 2^-24 of it.  The input comes as two fields (mie_split_exact),
// the filter as two arrays of rows.  Per filter tap two instructions per K-slice:
//     hi(input) x [hi(filter) | lo(filter)]  ->  N = 2 CB columns,      lo(input) x hi(filter)  ->  N = CB columns.
// (The split of an operand is that of Markidis et al., 2018; sums kept outside the tensor core because it truncates, that of
// Ootomo and Yokota, 2022.)
// What keeps the result at fp32 level is where the sums are rounded: the tensor core truncates each time it adds to an
// accumulator (1.7e-8 of the value per addition, always towards zero: 3e-5 after the 2400 additions of a 256-channel 5x5
// layer).  So the first product starts from zero again with every segment of two to five taps (exact_shape()) and the epilogue
// warps add the partial sums to registers, rounded to nearest, while the next segments run, low parts apart from high parts; the
// second product is 2^-12 of the first and stays in its accumulator for the whole work item.
// Error against a float64 convolution over that of the CUDA-core FP32 kernel: 0.68 to 0.95 for the first layers of the networks
// on their event inputs, 0.3 to 1.0 for normal and for rectified inputs from a reduction (cin * k * k) of 72 on.  It is larger only
// where few products meet, since the two parts leave 1e-7 of a value however short its sum: 1.2 to 1.6 for a reduction of 18, 1.1
// to 2.2 where isolated pixels are active and cin is below 48; and up to 1.4 where every product is positive.
// Epilogue: reservoir = conv + bias (+ addend), output = f(reservoir), every pixel of a listed tile marked.
#include "mie_pair.cuh"

using namespace mie;

namespace mie {
namespace {

constexpr int EXACT_THREADS = 384;
constexpr int EXACT_MAX_STAGES = 8;
constexpr int EXACT_MAX_HALOS = 4;

struct ExactParams {
  int cin, cout, cout_pad, n_chunks, n, hout, wout;
  const int32_t *list; int32_t *counts; int max_tiles;
  float *out; int64_t out_ps; unsigned int *out_bits32;
  int act; float *res; int64_t res_ps; const float *addend; int64_t addend_ps; const float *bias;
  int cb, stages, halos, tps, wp;   // tps: taps per ring stage
  int seg;     // taps per segment of the first product's sum
  unsigned spin_limit;
  int withhold_loads;      // self-test: the producers issue nothing, so the first wait runs out (MIE_OPT_TC_WITHHOLD_LOADS)
  mie_tail_job tail;
  PairTaps t;
};
struct ExactMaps {
  CUtensorMap hi[4], lo[4], w, out, res;
};

// acc[i] += column i (of n = 16 or 32) at taddr, + column i at taddr2: all loads in flight before the first addition
__device__ __forceinline__ void tmem_ld16_async(unsigned taddr, unsigned *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}
template <int N>
__device__ __forceinline__ void tmem_add(unsigned taddr, float *acc) {
  unsigned r[N];
#pragma unroll
  for (int g = 0; g < N; g += 16) tmem_ld16_async(taddr + g, r + g);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] += __uint_as_float(r[i]);
}

// Segment accumulators (2 CB columns each) beside the two item accumulators (CB each) in 512 columns: enough that the round
// trip of a segment to the epilogue and back does not hold up the issuer.
__host__ __device__ constexpr unsigned exact_segs(int cb) { return cb == 64 ? 3u : 6u; }

template <int CB>
__device__ __forceinline__ void exact_issue(const ExactParams &p, int bid, int nblk, int n_items, unsigned tmem_base, unsigned a_base, unsigned b_base,
    unsigned row_bytes, unsigned halo_bytes, unsigned tap_bytes, unsigned stage_bytes, unsigned long long *b_full, unsigned long long *b_empty,
    unsigned long long *a_full, unsigned long long *a_empty, unsigned long long *seg_full, unsigned long long *seg_empty, unsigned long long *item_full,
    unsigned long long *item_empty, volatile int *abort_flag) {
  constexpr unsigned NSEG = exact_segs(CB), item_col = NSEG * 2u * CB;
  const unsigned id0 = (make_idesc_tf32(0) & ~(31u << 24)) | (16u << 24);       // M = 256
  const unsigned id_hi = id0 | ((unsigned)(2 * CB >> 3) << 17), id_lo = id0 | ((unsigned)(CB >> 3) << 17);
  const unsigned long long b_tmpl = make_smem_desc(0), a_tmpl = make_smem_desc(0, row_bytes);
  const unsigned long long b_hi = b_tmpl & 0xFFFFFFFF00000000ull, a_hi = a_tmpl & 0xFFFFFFFF00000000ull;
  const unsigned lo_flags = (unsigned)(b_tmpl & 0xFFFF0000ull);
  const int nv = p.t.nviews;
  unsigned bs = 0, bpar = 0, as = 0, apar = 0, item_idx = 0, seg = 0, seg_par = 1, stage_addr = b_base;
#pragma unroll 1
  for (int item = bid; item < n_items; item += nblk, ++item_idx) {
    const unsigned buf = item_idx & 1u;
    if (item_idx >= 2 && !mbar_wait(&item_empty[buf], ((item_idx >> 1) - 1) & 1u, abort_flag, p.spin_limit)) return;
    unsigned started = 0;
#pragma unroll 1
    for (int chunk = 0; chunk < p.n_chunks; ++chunk) {
      const unsigned nks = (unsigned)min(4, (p.cin - chunk * 32 + 7) >> 3);
#pragma unroll 1
      for (int v = 0; v < nv; ++v) {
        if (!mbar_wait(&a_full[as], apar, abort_flag, p.spin_limit)) return;
        const unsigned halo = lo_flags | ((a_base + as * halo_bytes) >> 4);
        const int end = p.t.first[v + 1];
        int in_seg = 0;          // taps in the current segment
#pragma unroll 1
        for (int i = p.t.first[v]; i < end; i += p.tps) {
          const int nt = min(p.tps, end - i);
          unsigned b_lo = lo_flags | (stage_addr >> 4);
          if (!mbar_wait(&b_full[bs], bpar, abort_flag, p.spin_limit)) return;
          tc_fence_after();
#pragma unroll 1
          for (int k = 0; k < nt; ++k, b_lo += tap_bytes >> 4) {
            if (!in_seg) {
              if (!mbar_wait(&seg_empty[seg], seg_par, abort_flag, p.spin_limit)) return;
              tc_fence_after();
            }
            pair_mma(tmem_base + seg * (2u * CB), a_hi | (halo + ((unsigned)p.t.off[i + k] * 8u)), b_hi | b_lo, id_hi, (unsigned)in_seg, nks);
            if (++in_seg == p.seg || i + k + 1 == end) {
              pair_commit(&seg_full[seg]);
              in_seg = 0;
              if (++seg == NSEG) { seg = 0; seg_par ^= 1u; }
            }
          }
          pair_commit(&b_empty[bs]);
          stage_addr += stage_bytes;
          if (++bs == (unsigned)p.stages) { bs = 0; bpar ^= 1u; stage_addr = b_base; }
        }
        pair_commit(&a_empty[as]);
        if (++as == (unsigned)p.halos) { as = 0; apar ^= 1u; }
      }
#pragma unroll 1
      for (int v = 0; v < nv; ++v) {
        if (!mbar_wait(&a_full[as], apar, abort_flag, p.spin_limit)) return;
        const unsigned halo = lo_flags | ((a_base + as * halo_bytes) >> 4);
        const int end = p.t.first[v + 1];
#pragma unroll 1
        for (int i = p.t.first[v]; i < end; i += p.tps) {
          const int nt = min(p.tps, end - i);
          unsigned b_lo = lo_flags | (stage_addr >> 4);
          if (!mbar_wait(&b_full[bs], bpar, abort_flag, p.spin_limit)) return;
          tc_fence_after();
          const unsigned d = tmem_base + item_col + buf * CB;
#pragma unroll 1
          for (int k = 0; k < nt; ++k, b_lo += tap_bytes >> 4) {
            pair_mma(d, a_hi | (halo + ((unsigned)p.t.off[i + k] * 8u)), b_hi | b_lo, id_lo, started, nks);
            started = 1u;
          }
          pair_commit(&b_empty[bs]);
          stage_addr += stage_bytes;
          if (++bs == (unsigned)p.stages) { bs = 0; bpar ^= 1u; stage_addr = b_base; }
        }
        pair_commit(&a_empty[as]);
        if (++as == (unsigned)p.halos) { as = 0; apar ^= 1u; }
      }
    }
    pair_commit(&item_full[buf]);
  }
}

// HW: channels per epilogue set (CB = 2 HW channels per block)
template <int HW>
__global__ void __launch_bounds__(EXACT_THREADS, 1)
conv_exact_kernel(const ExactParams p, const __grid_constant__ ExactMaps maps) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int CB = 2 * HW;
  constexpr unsigned half_bytes = HW * 128u, tap_bytes = 2u * half_bytes;   // this block's rows of one tap: [hi | lo] of its half of the channels
  const unsigned row_bytes = (unsigned)p.wp * 128u;
  const unsigned halo_bytes = ((unsigned)p.wp * 2u * row_bytes + 1023u) & ~1023u;
  const unsigned stage_bytes = tap_bytes * (unsigned)p.tps;
  __shared__ unsigned long long b_full[EXACT_MAX_STAGES], b_empty[EXACT_MAX_STAGES], a_full[EXACT_MAX_HALOS], a_empty[EXACT_MAX_HALOS],
      seg_full[6], seg_empty[6], item_full[2], item_empty[2];
  __shared__ unsigned s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const unsigned crank = cluster_ctarank();
  const int bid = (int)(blockIdx.x >> 1), nblk = (int)(gridDim.x >> 1);
  const int THo = (p.hout + 7) >> 3, TWo = (p.wout + 7) >> 3;
  const int ntiles_total = p.n * THo * TWo;
  constexpr unsigned NSEG = exact_segs(CB), item_col = NSEG * 2u * CB, tmem_cols = 512u;

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < p.halos; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_empty[s], 1); }
    for (unsigned b = 0; b < NSEG; ++b) { mbar_init(&seg_full[b], 1); mbar_init(&seg_empty[b], 16); }
    for (int b = 0; b < 2; ++b) { mbar_init(&item_full[b], 1); mbar_init(&item_empty[b], 16); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = s_tmem_base;
  pair_cluster_sync();
  grid_dependency_wait();
  grid_dependency_trigger();

  const int n_active = __shfl_sync(0xffffffffu, min(p.counts[0], p.max_tiles), 0);
  const int n_cblk = p.cout_pad / CB, n_items = ((n_active + 3) >> 2) * n_cblk;
  const unsigned b_base = smem_u32(smem), a_base = b_base + (((unsigned)p.stages * stage_bytes + 1023u) & ~1023u);
  const int nv = p.t.nviews;

  // units of a chunk: the high parts of the views, then the low parts
  const PairWork work = {bid, nblk, n_items, n_cblk, p.n_chunks, 2 * nv, crank, p.spin_limit, p.withhold_loads};
  if (warp == 0) {
    // =========================== halo producer ===========================
    const PairRing ring = {a_full, a_empty, a_base, halo_bytes, (unsigned)p.halos};
    pair_produce_halos(work, ring, p.t, p.wp, row_bytes, p.list, n_active, ntiles_total, TWo, THo, p.counts, &s_abort, [&](int u, int &v) {
      v = u < nv ? u : u - nv;
      return u < nv ? &maps.hi[v] : &maps.lo[v];
    });
  } else if (warp == 1) {
    // =========================== filter producer: hi and lo rows beside the high part of the input, hi rows beside the low part ===========================
    const PairRing ring = {b_full, b_empty, b_base, stage_bytes, (unsigned)p.stages};
    pair_produce_filter(work, ring, p.t, p.tps, tap_bytes, (int)crank * HW, CB, &s_abort, [&](int u) { return u < nv ? u : u - nv; },
                        [&](int u) { return 2u * (u < nv ? tap_bytes : half_bytes); },
                        [&](int u, int tap, unsigned dst, unsigned bar, int row, int chunk) {
                          tma_load_4d_pair(dst, &maps.w, bar, 0, row, chunk, tap);
                          if (u < nv) tma_load_4d_pair(dst + half_bytes, &maps.w, bar, 0, p.cout_pad + row, chunk, tap);
                        });
  } else if (warp == 2) {
    // =========================== MMA issuer (first block of the pair) ===========================
    if (crank == 0u) {
      exact_issue<CB>(p, bid, nblk, n_items, tmem_base, a_base, b_base, row_bytes, halo_bytes, tap_bytes, stage_bytes, b_full, b_empty, a_full, a_empty, seg_full, seg_empty, item_full, item_empty, &s_abort);
    }
  } else if (warp >= 4) {
    // =========================== epilogue: set `set` takes channels [set * HW, set * HW + HW) of the block ===========================
    const int q = warp & 3, set = (warp - 4) >> 2;
    const int slot = (lane >> 3) & 1, prow = 2 * q + (lane >> 4), pcol = lane & 7;
    const unsigned lane_base = tmem_base + ((unsigned)(q * 32) << 16);
    int segs_per_chunk = 0;
    for (int v = 0; v < nv; ++v) segs_per_chunk += (p.t.first[v + 1] - p.t.first[v] + p.seg - 1) / p.seg;
    const int segs = segs_per_chunk * p.n_chunks;
    // slabs of this set: output, then reservoir; 128 rows of HW channels, 16-byte pieces swizzled as TMA does for rows of
    // 128 bytes (piece ^ (row & 7)) or 64 bytes (piece ^ (row / 2 & 3))
    constexpr unsigned SLAB = 128u * HW * 4u;
    const int row = slot * 64 + prow * 8 + pcol, sw = HW == 32 ? row & 7 : (row >> 1) & 3;
    const unsigned slab = a_base + (unsigned)p.halos * halo_bytes + (unsigned)set * (p.act != MIE_ACT_NONE ? 2u : 1u) * SLAB;
    const unsigned out_row = slab + (unsigned)row * (HW * 4u), res_row = out_row + SLAB;
    const bool chief = q == 0 && elect_one();
    unsigned item_idx = 0, seg = 0, seg_par = 0;
    bool ok = true;
    for (int item = bid; item < n_items && ok; item += nblk, ++item_idx) {
      const int quad = item / n_cblk, cb = item - quad * n_cblk;
      const unsigned buf = item_idx & 1u;
      const int e = 4 * quad + 2 * (int)crank + slot;
      int t = e < n_active ? p.list[e] : -1;
      if (t >= ntiles_total) t = -1;
      const int tx = (t >= 0) ? (t % TWo) * 8 : 0, ty = (t >= 0) ? ((t / TWo) % THo) * 8 : 0, n = (t >= 0) ? t / (TWo * THo) : 0;
      const bool valid = t >= 0 && ty + prow < p.hout && tx + pcol < p.wout;
      const int64_t pix = valid ? (int64_t)(n * p.hout + ty + prow) * p.wout + tx + pcol : 0;
      float acc[HW], low[HW];       // the low products are summed apart, so that the large sum is rounded once a segment
#pragma unroll
      for (int i = 0; i < HW; ++i) acc[i] = low[i] = 0.0f;
      for (int s = 0; s < segs; ++s) {
        if (!(ok = __all_sync(0xffffffffu, mbar_wait(&seg_full[seg], seg_par, &s_abort, p.spin_limit)))) break;
        tc_fence_after();
        const unsigned c = lane_base + seg * (2u * CB) + (unsigned)set * CB;     // [hi | lo] columns of this set's channels
        tmem_add<HW>(c, acc);
        tmem_add<HW>(c + HW, low);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&seg_empty[seg]), 0));
        if (++seg == NSEG) { seg = 0; seg_par ^= 1u; }
      }
      // a warp whose wait gave up goes on to the barrier of its set, where the four of them leave together
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&item_full[buf], (item_idx >> 1) & 1u, &s_abort, p.spin_limit));
      tc_fence_after();
      if (ok) tmem_add<HW>(lane_base + item_col + buf * CB + (unsigned)(set * HW), low);
#pragma unroll
      for (int i = 0; i < HW; ++i) acc[i] += low[i];
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&item_empty[buf]), 0));
      const int co = cb * CB + set * HW;
      // the slabs are free once the previous item's stores have read them
      if (chief) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      __syncwarp();
      ok = set_all(1 + set, ok);
      if (!ok) break;
#pragma unroll
      for (int h = 0; h < HW / 4; ++h) {
        const int c = co + 4 * h;
        float4 v = make_float4(acc[4 * h], acc[4 * h + 1], acc[4 * h + 2], acc[4 * h + 3]);
        if (p.bias && c < p.cout) v = f4add(v, make_float4(__ldg(p.bias + c), __ldg(p.bias + c + 1), __ldg(p.bias + c + 2), __ldg(p.bias + c + 3)));
        if (p.addend && valid && c < p.cout) v = f4add(v, *reinterpret_cast<const float4 *>(p.addend + pix * p.addend_ps + c));
        const unsigned at = (unsigned)(h ^ sw) << 4;
        if (p.act != MIE_ACT_NONE) {
          sts4(res_row + at, v);
          v = p.act == MIE_ACT_RELU ? make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f))
                                    : make_float4(tc_act_call(p.act, v.x), tc_act_call(p.act, v.y), tc_act_call(p.act, v.z), tc_act_call(p.act, v.w));
        }
        sts4(out_row + at, v);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
      if (chief && co < p.cout) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int es = 4 * quad + 2 * (int)crank + s, ts = es < n_active ? p.list[es] : -1;
          if (ts < 0 || ts >= ntiles_total) continue;
          const int x = (ts % TWo) * 8, y = ((ts / TWo) % THo) * 8, ns = ts / (TWo * THo);
          tma_store_slab(slab + s * (SLAB / 2), &maps.out, co, x, y, ns);
          if (p.act != MIE_ACT_NONE) tma_store_slab(slab + SLAB + s * (SLAB / 2), &maps.res, co, x, y, ns);
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      // every pixel written is marked; ballot bytes: [tile 0 row 2q][tile 1 row 2q][tile 0 row 2q+1][tile 1 row 2q+1]
      const unsigned bal = __ballot_sync(0xffffffffu, valid);
      if ((lane == 0 || lane == 8) && t >= 0) {
        const unsigned rows = ((bal >> lane) & 0xFFu) | (((bal >> (16 + lane)) & 0xFFu) << 8);
        if (rows) atomicOr(p.out_bits32 + 2 * (size_t)t + (q >> 1), rows << ((q & 1) * 16));
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
    if (warp == 0) { const long long t0 = clock64(); while (clock64() - t0 < 2000000) { } }
    __syncthreads();
  }
  pair_cluster_sync();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
  run_tail_job(p.tail);
}

}  // namespace

// How a launch divides its columns and its shared memory; `stages` < 2: no split of it fits.
struct ExactShape {
  PairTaps t;
  int wp, cb, tps, stages, halos, seg;
  size_t smem;
};
static ExactShape exact_shape(const mie_conv_args *a) {
  ExactShape h;
  pair_make_taps(a->k, a->stride, a->pad, &h.t, &h.wp);
  const int quads = divup(a->max_tiles, 4), clusters_max = MIE_SM_COUNT / 2;
  // 64 channels per block (144 clocks per K-slice and tap, both instructions) unless blocks of 32 (103) take fewer clocks over all
  // rounds: 256 -> 64 and 32 channels, the slope from four to eight rounds at 1965 MHz for k = 5 (k = 3: 159 and 113; k = 7: 178 and 105)
  h.cb = 32;
  if (a->cout_pad % 64 == 0 &&
      (int64_t)divup(quads * (a->cout_pad / 64), clusters_max) * 144 <= (int64_t)divup(quads * (a->cout_pad / 32), clusters_max) * 103)
    h.cb = 64;
  const int halo_bytes = (h.wp * 2 * h.wp * 128 + 1023) & ~1023, slab_bytes = 2 * (a->act != MIE_ACT_NONE ? 2 : 1) * 128 * (h.cb / 2) * 4;
  const int budget = 222 * 1024 - slab_bytes;
  // Fat stages: what the issuer and the producers spend per stage does not depend on its size.  Three of them where
  // halo buffers can be spared for that, else two; a 7x7 filter's halos beside the slabs of a wide block leave room for
  // two stages of three taps (still ahead of blocks of 32 channels with nine: 64 -> 64 on 2 x 256x336 366 against 436 us,
  // on 104x104 46 against 56).
  h.tps = h.cb == 32 ? 9 : 5;
  h.halos = EXACT_MAX_HALOS;
  while (h.halos > 2 && budget - h.halos * halo_bytes < 3 * h.tps * h.cb * 128) --h.halos;
  while (h.tps > 1 && budget - h.halos * halo_bytes < 2 * h.tps * h.cb * 128) --h.tps;
  const int stage_bytes = h.tps * h.cb * 128;
  h.stages = (budget - h.halos * halo_bytes) / stage_bytes;
  if (h.stages > EXACT_MAX_STAGES) h.stages = EXACT_MAX_STAGES;
  // A segment's truncation grows with its length, the FP32 kernel's rounding with the whole reduction: the longest segments that
  // keep the error below that kernel's for rectified inputs (segments of 2 / 3 / 5 taps: 288 products 0.83 / 1.13 / 1.62 of its
  // error, 576 0.63 / 0.85 / 1.21, 800 0.55 / 0.70 / 1.09, 1152 0.44 / 0.58 / 0.83).  Shorter ones cost time: a refresh of eight
  // E2Depth streams 480x640 takes 14.3 / 13.6 / 13.4 ms with one length for all layers.
  const int depth = a->cin * a->k * a->k;
  h.seg = depth < 400 ? 2 : depth < 1152 ? 3 : 5;
  h.smem = (size_t)((h.stages * stage_bytes + 1023) & ~1023) + (size_t)h.halos * halo_bytes + slab_bytes + 1024;
  return h;
}

bool exact_takes(const mie_conv_args *a) {
  // a field one pixel wide or high has no odd columns or rows: that parity view of stride 2 would be empty, and a tensor map
  // cannot say so
  if (a->stride == 2 && (a->hin == 1 || a->win == 1)) return false;
  return a->refresh && !a->head && a->wpacked_exact && a->in_lo && a->k >= 3 && a->k <= 7 && (a->k & 1) && (a->stride == 1 || a->stride == 2) && !a->in2 && !a->accum &&
         a->in_ps % 4 == 0 && aligned16(a->in) && aligned16(a->in_lo) && aligned16(a->wpacked_exact) && a->cout % 4 == 0 && a->out_ps % 4 == 0 &&
         aligned16(a->out) && (!a->res || (a->res_ps % 4 == 0 && aligned16(a->res))) && (!a->addend || (a->addend_ps % 4 == 0 && aligned16(a->addend))) &&
         a->cout_pad % 32 == 0 && exact_shape(a).stages >= 2;
}

int launch_conv_exact(const mie_conv_args *a, cudaStream_t st) {
  const ExactShape h = exact_shape(a);
  ExactParams p;
  memset(&p, 0, sizeof(p));
  p.spin_limit = g_opt_spin_limit;
  p.withhold_loads = g_opt_withhold_loads;
  p.cin = a->cin; p.cout = a->cout; p.cout_pad = a->cout_pad; p.n_chunks = divup(a->cin, 32);
  p.n = a->n; p.hout = a->hout; p.wout = a->wout;
  p.list = a->list; p.counts = a->counts; p.max_tiles = a->max_tiles;
  p.out = a->out; p.out_ps = a->out_ps; p.out_bits32 = reinterpret_cast<unsigned int *>(a->out_bits);
  p.act = a->act; p.res = a->res; p.res_ps = a->res_ps; p.addend = a->addend; p.addend_ps = a->addend_ps; p.bias = a->bias;
  p.tail = tail_for_kernel(a->tail);
  p.t = h.t; p.wp = h.wp; p.cb = h.cb; p.tps = h.tps; p.stages = h.stages; p.halos = h.halos; p.seg = h.seg;
  const size_t smem = h.smem;
  const int quads = divup(a->max_tiles, 4), clusters_max = MIE_SM_COUNT / 2;

  ExactMaps maps;
  memset(&maps, 0, sizeof(maps));
  const int s = a->stride;
  const cuuint32_t box_in[4] = {32, (cuuint32_t)p.wp, 1, 1};
  for (int v = 0; v < p.t.nviews; ++v) {
    const int py = s == 2 ? v >> 1 : 0, px = s == 2 ? v & 1 : 0;
    const cuuint64_t dims[4] = {(cuuint64_t)a->cin, (cuuint64_t)((a->win - px + s - 1) / s), (cuuint64_t)((a->hin - py + s - 1) / s), (cuuint64_t)a->n};
    const cuuint64_t str[3] = {(cuuint64_t)a->in_ps * 4 * s, (cuuint64_t)a->win * a->in_ps * 4 * s, (cuuint64_t)a->hin * a->win * a->in_ps * 4};
    const int64_t off = ((int64_t)py * a->win + px) * a->in_ps;
    if (!tc_encode(&maps.hi[v], 4, a->in + off, dims, str, box_in, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !tc_encode(&maps.lo[v], 4, a->in_lo + off, dims, str, box_in, CU_TENSOR_MAP_SWIZZLE_128B))
      return MIE_EINVAL;
  }
  {
    // [tap][chunk][hi rows | lo rows][32]
    const cuuint64_t rows = 2 * (cuuint64_t)a->cout_pad, nch = (cuuint64_t)p.n_chunks;
    const cuuint64_t dims[4] = {32, rows, nch, (cuuint64_t)(a->k * a->k)};
    const cuuint64_t str[3] = {128, rows * 128, nch * rows * 128};
    const cuuint32_t box_w[4] = {32, (cuuint32_t)(p.cb / 2), 1, 1};
    if (!tc_encode(&maps.w, 4, a->wpacked_exact, dims, str, box_w, CU_TENSOR_MAP_SWIZZLE_128B)) return MIE_EINVAL;
  }
  {
    // epilogue slabs: half a block's channels of one tile
    const cuuint32_t box[4] = {(cuuint32_t)(p.cb / 2), 8, 8, 1};
    const CUtensorMapSwizzle sw = p.cb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    auto slab_map = [&](CUtensorMap *m, const float *base, int64_t ps) {
      const cuuint64_t dims[4] = {(cuuint64_t)a->cout, (cuuint64_t)a->wout, (cuuint64_t)a->hout, (cuuint64_t)a->n};
      const cuuint64_t str[3] = {(cuuint64_t)ps * 4, (cuuint64_t)a->wout * ps * 4, (cuuint64_t)a->hout * a->wout * ps * 4};
      return tc_encode(m, 4, base, dims, str, box, sw);
    };
    if (!slab_map(&maps.out, a->out, a->out_ps) || (a->act != MIE_ACT_NONE && !slab_map(&maps.res, a->res, a->res_ps))) return MIE_EINVAL;
  }
  const int64_t items = (int64_t)quads * (a->cout_pad / p.cb);
  const int clusters = (int)(items < clusters_max ? items : clusters_max);
  static int smem_set[2][MAX_DEVICES] = {{0}};
  auto launch = [&](auto kernel, int i) {
    const int r = ensure_dynamic_smem(kernel, smem_set[i], smem);
    if (r != MIE_OK) return r;
    launch_chained_cluster(kernel, dim3((unsigned)(2 * clusters)), dim3(EXACT_THREADS), smem, st, 2, p, maps);
    return check_launch();
  };
  return p.cb == 64 ? launch(conv_exact_kernel<32>, 1) : launch(conv_exact_kernel<16>, 0);
}

// Round to nearest TF32 (10 mantissa bits).
__device__ __forceinline__ float round_tf32(float v) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}
// v as two TF32 numbers.  A finite v that would round up to infinity is truncated instead.  Infinity and NaN have no low part
// (inf - inf), and infinity times the low part of the other operand has any sign: they become the low part themselves, which
// meets nothing but the high part of the other operand, and give what fp32 gives.
__device__ __forceinline__ void split_two_tf32(float v, float &hi, float &lo) {
  if (!isfinite(v)) {
    hi = 0.0f;
    lo = isnan(v) ? __uint_as_float(0x7FC00000u) : v;     // (a NaN whose payload is in the bits that TF32 drops would read as infinity)
    return;
  }
  hi = round_tf32(v);
  if (isinf(hi)) hi = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
  lo = round_tf32(v - hi);
}

// hi = round(v), lo = round(v - hi): one pass over a dense field, a thread per four channels of a pixel.  HBM bound: one read
// and two writes at 5.6 to 6.0 TB/s on fields beyond the L2 (8 x 32 x 480x640: 167 us), 0.86 to 0.91 of a measured copy.
// counts (may be null): the work list of the convolution that reads the parts; none are made where it lists no tile.
__global__ void __launch_bounds__(256) split_exact_kernel(const float *__restrict__ in, int64_t in_ps, int C, int64_t pixels, float *__restrict__ hi,
                                                          float *__restrict__ lo, int64_t out_ps, int quads, int vec, const int32_t *counts) {
  grid_dependency_wait();
  grid_dependency_trigger();
  if (counts && counts[0] == 0) return;
  const int64_t total = pixels * quads;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t px = i / quads;
    const int c = (int)(i - px * quads) * 4;
    float v[4];
    if (vec) {
      const float4 x = *reinterpret_cast<const float4 *>(in + px * in_ps + c);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = c + j < C ? in[px * in_ps + c + j] : 0.0f;
    }
    float h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split_two_tf32(v[j], h[j], l[j]);
    *reinterpret_cast<float4 *>(hi + px * out_ps + c) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4 *>(lo + px * out_ps + c) = make_float4(l[0], l[1], l[2], l[3]);
  }
}

// [tap][chunk][hi: cout_pad rows | lo: cout_pad rows][32] <- w[cout][cin][ky][kx], zero padded
// (ihwo: the filter is stored [cin][ky][kx][cout] instead)
__global__ void pack_weights_exact_kernel(const float *__restrict__ w, int cout, int cin, int k, int nch, int cout_pad, float *__restrict__ wp, int64_t total,
                                          int ihwo) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int cl = (int)(i % 32);
    int64_t rest = i / 32;
    const int row = (int)(rest % (2 * cout_pad));
    rest /= 2 * cout_pad;
    const int ci = (int)(rest % nch) * 32 + cl, tap = (int)(rest / nch), co = row < cout_pad ? row : row - cout_pad;
    float v = 0.0f;
    if (co < cout && ci < cin) v = w[ihwo ? ((int64_t)ci * k * k + tap) * cout + co : ((int64_t)co * cin + ci) * k * k + tap];
    float h, l;
    split_two_tf32(v, h, l);
    wp[i] = row < cout_pad ? h : l;
  }
}

int pack_exact(const float *w, int cout, int cin, int k, int ihwo, float *wpacked, cudaStream_t st) {
  int64_t total;
  const int s = mie_conv_pack_dims_exact(cin, cout, k, &total);
  if (s != MIE_OK) return s;
  int64_t blocks = divup64(total, 256);
  if (blocks > MIE_SM_COUNT * 8) blocks = MIE_SM_COUNT * 8;
  pack_weights_exact_kernel<<<(unsigned)blocks, 256, 0, st>>>(w, cout, cin, k, divup(cin, 32), divup(cout, 32) * 32, wpacked, total, ihwo);
  return check_launch();
}

int split_exact(const float *in, int64_t in_ps, int C, int64_t pixels, float *hi, float *lo, int64_t out_ps, const int32_t *counts, cudaStream_t st) {
  if (!in || !hi || !lo || C <= 0 || pixels <= 0 || in_ps < C || out_ps < (C + 3) / 4 * 4 || out_ps % 4) return MIE_EINVAL;
  if (!aligned16(hi) || !aligned16(lo)) return MIE_EALIGN;
  const int quads = divup(C, 4), vec = C % 4 == 0 && in_ps % 4 == 0 && aligned16(in);
  int64_t blocks = divup64(pixels * quads, 256);
  if (blocks > MIE_SM_COUNT * 16) blocks = MIE_SM_COUNT * 16;
  launch_chained(split_exact_kernel, dim3((unsigned)blocks), dim3(256), 0, st, in, in_ps, C, pixels, hi, lo, out_ps, quads, vec, counts);
  return check_launch();
}

}  // namespace mie

extern "C" int mie_split_exact(const float *in, int64_t in_ps, int C, int64_t pixels, float *hi, float *lo, int64_t out_ps, void *stream) {
  return split_exact(in, in_ps, C, pixels, hi, lo, out_ps, nullptr, (cudaStream_t)stream);
}

extern "C" int mie_conv_pack_dims_exact(int cin, int cout, int k, int64_t *n_floats) {
  if (cin <= 0 || cout <= 0 || k <= 0 || !n_floats) return MIE_EINVAL;
  *n_floats = (int64_t)k * k * divup(cin, 32) * 2 * (divup(cout, 32) * 32) * 32;
  return MIE_OK;
}

extern "C" int mie_pack_conv_weights_exact(const float *w_oihw, int cout, int cin, int k, float *wpacked, void *stream) {
  if (!w_oihw || !wpacked) return MIE_EINVAL;
  return pack_exact(w_oihw, cout, cin, k, 0, wpacked, (cudaStream_t)stream);
}
