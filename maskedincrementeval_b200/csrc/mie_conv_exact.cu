// Convolutions in fp32 precision on the tensor cores, on CTA pairs like mie_conv_pair.cu: the dense evaluation (the refresh pass), and
// incremental steps of layers in split precision.
//
// Every operand is two FP16 numbers with a common power-of-two scale (mie_pair.cuh), together the fp32 value to 2^-24, and a
// product is hi*hi + hi*lo + lo*hi; the dropped lo*lo is 2^-24 of it.  The halo arrives as fp32 and is split in shared memory by
// eight warps of its block, in place; the filter is packed as two arrays of rows.  Per filter tap two instructions per
// K-slice of 16 channels:
//     hi(input) x [hi(filter) | lo(filter)]  ->  N = 2 CB columns,      lo(input) x hi(filter)  ->  N = CB columns.
// With two TF32 numbers per operand, which is what stood here before, an instruction takes 8 channels from the same 32 bytes,
// the input had to be split by a pass of its own (one read and two writes of every layer's input through HBM) and twice the operand
// bytes crossed L2: eight E2Depth streams 480x640 13.5 ms, with FP16 parts 9.2.
// (Splitting an operand: Markidis et al., 2018; scaled FP16 parts, and sums kept outside the tensor core because it truncates:
// Ootomo and Yokota, 2022.)
// What keeps the result at fp32 level is where the sums are rounded: the tensor core truncates each time it adds to an
// accumulator.  So the sums start from zero again with every segment of taps, which is a stage of the filter ring, and the epilogue
// warps add the segments to registers, rounded to nearest, while the next ones run.  Error against a float64 convolution over
// that of the CUDA-core FP32 kernel: 0.3 to 1.0 for normal and rectified inputs from a reduction (cin * k * k) of 72 on; larger only
// where few products meet, since the two parts leave 1e-7 of a value however short its sum: 1.2 to 1.5 for a reduction of 18, 1.0
// to 2.2 at isolated active pixels with cin below 32.
// What bounds it: operand reads and everything else that goes through shared memory (per tap and 32 channels, blocks of 64: 172 clocks
// of its port for the instructions, which take 214 in the tensor core, 32 for the filter arriving, 35 to 70 for the
// halo arriving and being split), then the epilogue's slabs on layers of few units (a chunk of a view) per item.
// Epilogue, dense: reservoir = conv + bias (+ addend), output = f(reservoir), every pixel of a tile marked.  A step: reservoir += conv
// (+ addend), output = the change of f(reservoir), threshold, carry and marks as in the other step kernels.
// What the parts do not hold (mie_pair.cuh) is multiplied with FP32 instructions, in functions that the ordinary course calls at most once an
// item and keeps no registers for.
#include <algorithm>
#include "mie_pair.cuh"

using namespace mie;

namespace mie {
namespace {

constexpr int EXACT_THREADS = 384 + 32 * SPLIT_WARPS;
constexpr int EXACT_MAX_STAGES = 8;
constexpr int EXACT_MAX_HALOS = 4;

struct ExactParams {
  const float *in; int64_t in_ps; int hin, win, k, stride, pad;      // read by the FP32 fallback only, like the filter below
  const float *fw; int64_t fw_tap, fw_ci; int fw_vec;                // filter entry (tap, ci, co) at fw[tap * fw_tap + ci * fw_ci + co]
  const float *winv;                                                 // inverse scale of every output channel's filter; NaN: not split
  int cin, cout, cout_pad, n_chunks, n, hout, wout;
  const int32_t *list; int32_t *counts; int max_tiles;               // list null (dense pass): every tile
  float *out; int64_t out_ps; unsigned int *out_bits32;
  int act; float *res; int64_t res_ps; const float *addend; int64_t addend_ps; const float *bias;
  int cb, stages, halos, wp;
  int tps;     // taps per ring stage, which is a segment of the sums
  int segs;    // segment accumulators
  unsigned spin_limit;
  int withhold_loads;      // self-test: the producers issue nothing, so the first wait runs out (MIE_OPT_TC_WITHHOLD_LOADS)
  int slab_bufs;           // shared-memory slabs per epilogue set: output (+ reservoir (+ carry))
  int slab_sets;           // ... and how many such buffers items take in turn (1 or 2)
  unsigned div_tw, div_th; // magic numbers for divisions by the field's tiles per row and rows of tiles; 0: plain division
  mie_tail_job tail;
  PairTaps t;
  TcParams c;              // a step: threshold, carry, stale tiles
};
struct ExactMaps {
  CUtensorMap in[4], w, out, res, emitted;
};

__device__ __forceinline__ void tmem_ld16_async(unsigned taddr, unsigned *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}
// hi + 2^-11 (mid + low + 2^-11 last): the products of a segment.
// FULL: the low parts are multiplied too (lo x lo), and in layers of up to 16 channels third parts, which hold what two leave of an operand,
// with the high ones (pair_mma_full).  The low accumulator then has N = 64 columns like the high one, and a segment a third more
// columns to read (64 -> 32 5x5 at 8 x 480x640, lo x lo alone: 874 us against 831), for 2^-24 of a product.  Taken by thin layers, where few
// products meet and the FP32 kernel is what they are measured against (16 -> 24 3x3, error of the change over that kernel's, 0.5 / 5 / 40 %
// active: without 1.21 / 1.01 / 0.96, with lo x lo 1.04 / 0.90 / 0.93, with third parts 0.73 / 0.72 / 0.80; a step on 97x131 15.8 us without these,
// 17.1 with).  Blocks of 32 channels only.
__device__ __forceinline__ float split_sum(unsigned hi, unsigned mid, unsigned low, unsigned last, bool full) {
  float v = __uint_as_float(mid) + __uint_as_float(low);
  if (full) v = fmaf(__uint_as_float(last), SPLIT_LO, v);
  return fmaf(v, SPLIT_LO, __uint_as_float(hi));
}
// acc[i] += inv * (the sum of a segment's products), 16 columns at a time
template <int N, bool FULL>
__device__ __forceinline__ void tmem_add_split(unsigned hi, unsigned mid, unsigned low, unsigned last, float inv, float *acc) {
#pragma unroll
  for (int g = 0; g < N; g += 16) {
    unsigned a[16], b[16], c[16], d[16];
    tmem_ld16_async(hi + g, a);
    tmem_ld16_async(mid + g, b);
    tmem_ld16_async(low + g, c);
    if (FULL) tmem_ld16_async(last + g, d);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[g + i] = fmaf(split_sum(a[i], b[i], c[i], FULL ? d[i] : 0u, FULL), inv, acc[g + i]);
  }
}

// Segment accumulators in 512 columns: [hi x hi | hi x lo] of either half of the channels, then lo x hi, or [lo x hi | lo x lo] like the first.
__host__ __device__ constexpr unsigned exact_cols(int cb, bool full) { return (full ? 4u : 3u) * (unsigned)cb; }
__host__ __device__ constexpr unsigned exact_segs(int cb, bool full) { return 512u / exact_cols(cb, full); }

// The MMA issuer.  A ring stage of the filter is a segment: one wait for its operands, its accumulator and (first stage) the
// halo together, one commit for both the filter producer and the epilogue.  The issuing warp is what paces the kernel: the
// instructions of a 3x3 chunk of 64 channels take 1930 clocks, a wait about 130 and a commit about 80 beside them.
struct ExactIssue {
  int item0, item_step, n_items, n_chunks, cin, tps, nviews;
  unsigned tmem_base, a_base, b_base, row_bytes, halo_bytes, stage_bytes, stages, halos, segs, limit;
};
template <int CB, bool ALT, bool FULL>
__device__ __forceinline__ void exact_issue(const ExactIssue a, const PairTapTable &t, unsigned long long *b_full, unsigned long long *done,
    unsigned long long *a_ready, unsigned long long *a_empty, unsigned long long *seg_empty, unsigned long long *item_full, volatile int *abort_flag) {
  constexpr unsigned tap_units = CB * 64 >> 4;
  const unsigned id_hi = make_idesc_f16_pair(2 * CB), id_lo = make_idesc_f16_pair(CB);
  const unsigned long long b_tmpl = make_smem_desc_64(0), a_tmpl = make_smem_desc(0, a.row_bytes);
  const unsigned long long b_hi = b_tmpl & 0xFFFFFFFF00000000ull, a_hi = a_tmpl & 0xFFFFFFFF00000000ull;
  const unsigned lo_flags = (unsigned)(b_tmpl & 0xFFFF0000ull);
  unsigned bs = 0, bpar = 0, as = 0, apar = 0, seg = 0, seg_par = 1, stage_addr = a.b_base, turn = 0;
#pragma unroll 1
  for (int item = a.item0; item < a.n_items; item += a.item_step) {
#pragma unroll 1
    for (int chunk = 0; chunk < a.n_chunks; ++chunk) {
      const unsigned nks = (unsigned)min(2, (a.cin - chunk * 32 + 15) >> 4);
#pragma unroll 1
      for (int v = 0; v < a.nviews; ++v) {
        const unsigned halo = lo_flags | ((a.a_base + as * a.halo_bytes) >> 4);
        const int end = t.first[v + 1];
        unsigned abar = smem_u32(&a_ready[as]), ap = apar;
#pragma unroll 1
        for (int i = t.first[v]; i < end; i += a.tps) {
          const int nt = min(a.tps, end - i);
          unsigned b_lo = lo_flags | (stage_addr >> 4), off = (unsigned)t.off[i];
          const unsigned d = a.tmem_base + seg * exact_cols(CB, FULL);
          const unsigned bbar = smem_u32(&b_full[bs]);
          if (!mbar_wait3(abar, ap, bbar, bpar, smem_u32(&seg_empty[seg]), seg_par, abort_flag, a.limit)) return;
          tc_fence_after();
          for (int k = 0; k < nt; ++k, b_lo += tap_units) {
            const unsigned a_lo = halo + off;
            off = (unsigned)t.off[i + k + 1];     // the next tap's, while this one is issued (the table has a spare entry)
            if (FULL) pair_mma_full(d, d + 2u * CB, a_hi | a_lo, b_hi | b_lo, id_hi, (unsigned)k, nks, (unsigned)(a.cin <= 16));
            else pair_mma_split(d, d + 2u * CB, a_hi | a_lo, b_hi | b_lo, id_hi, id_lo, (unsigned)k, nks);
          }
          pair_commit(&done[bs]);
          if (++seg == a.segs) { seg = 0; seg_par ^= 1u; }
          stage_addr += a.stage_bytes;
          if (++bs == a.stages) { bs = 0; bpar ^= 1u; stage_addr = a.b_base; }
          abar = smem_u32(&b_full[bs]); ap = bpar;      // further stages of the unit: the halo is there
        }
        pair_commit(&a_empty[as]);
        if (++as == a.halos) { as = 0; apar ^= 1u; }
      }
    }
    if (ALT) { pair_commit(&item_full[turn]); turn ^= 1u; }
  }
}

// ---- what two FP16 parts cannot hold, with FP32 instructions: out of line and on arrays in local memory, since what is run this seldom is
// paid in instructions that are fetched, and what it keeps in registers by everything else ----
// Adds to sums (HW channels from co on, in true units) the products of the values that were taken out of an item's unit cu (ring unit u), as
// far as this thread's pixel and the taps of the unit's view reach them.  Returns whether there were any; reach: only that.
template <int HW>
__device__ __noinline__ bool exact_small(const ExactParams &p, const SplitShared &sh, unsigned u, int cu, int co, float *sums, bool reach) {
  const SplitSmall &list = sh.small[u % SPLIT_RING];
  const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3, slot = (lane >> 3) & 1, prow = 2 * q + (lane >> 4), pcol = lane & 7;
  const int nv = p.t.nviews, view = cu % nv, chunk = cu / nv, odd_y = p.stride == 2 ? view >> 1 : 0, odd_x = p.stride == 2 ? view & 1 : 0;
  bool any = false;
#pragma unroll 1
  for (int i = 0; i < SPLIT_LISTED && list.at[i] != SPLIT_NONE; ++i) {
    const int at = list.at[i];
    // the tap that meets it at this pixel
    const int ky = p.stride * (p.t.y0[view] + (at >> 9 & 15) - prow) + odd_y + p.pad, kx = p.stride * (p.t.x0[view] + (at >> 5 & 15) - pcol) + odd_x + p.pad;
    if (at >> 13 != slot || ky < 0 || ky >= p.k || kx < 0 || kx >= p.k) continue;
    any = true;
    if (reach) continue;
    const float *w = p.fw + (ky * p.k + kx) * p.fw_tap + (32 * chunk + (at & 31)) * p.fw_ci + co;
#pragma unroll 4
    for (int c = 0; c < HW; ++c)
      if (co + c < p.cout) sums[c] += list.value[i] * __ldg(w + c);
  }
  return any;
}

// All channels of a pixel, where a halo or a channel's filter was not split: the same sums as the FP32 kernel's, padding multiplied as zeros
// like there.  Infinities, NaN, values above 2^100, many values far apart and filters with entries too far apart come to this.  Bounded by
// the latency of its loads, which the few KB of L1 beside the shared memory do not hold (64 -> 64 3x3 at 264x352, every halo: 3600 us, the FP32
// kernel 285, split 36).  which: a bit per channel that is wanted.
template <int HW>
__device__ __noinline__ void exact_fp32(const ExactParams &p, int n, int oy, int ox, int co, unsigned which, float *sums) {
  float acc[HW];
#pragma unroll
  for (int i = 0; i < HW; ++i) acc[i] = 0.0f;
#pragma unroll 1
  for (int tap = 0; tap < p.k * p.k; ++tap) {
    const int iy = oy * p.stride - p.pad + tap / p.k, ix = ox * p.stride - p.pad + tap % p.k;
    const bool in = iy >= 0 && iy < p.hin && ix >= 0 && ix < p.win;
    // (pixels are 16-byte aligned, a multiple of four channels apart; what lies behind the last channel is not used)
    const float4 *x = reinterpret_cast<const float4 *>(p.in + (in ? ((int64_t)(n * p.hin + iy) * p.win + ix) * p.in_ps : 0));
    const float *w = p.fw + tap * p.fw_tap + co;
    float4 next = __ldg(x);
#pragma unroll 1
    for (int c4 = 0; c4 < p.cin; c4 += 4) {
      const float4 now = next;
      if (c4 + 4 < p.cin) next = __ldg(++x);
#pragma unroll
      for (int j = 0; j < 4; ++j, w += p.fw_ci) {
        if (c4 + j >= p.cin) break;
        const float xv = !in ? 0.0f : j == 0 ? now.x : j == 1 ? now.y : j == 2 ? now.z : now.w;
#pragma unroll
        for (int h = 0; h < HW; h += 4) {
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (co + h < p.cout)
            f = p.fw_vec ? __ldg(reinterpret_cast<const float4 *>(w + h)) : make_float4(__ldg(w + h), __ldg(w + h + 1), __ldg(w + h + 2), __ldg(w + h + 3));
          acc[h] = fmaf(xv, f.x, acc[h]); acc[h + 1] = fmaf(xv, f.y, acc[h + 1]); acc[h + 2] = fmaf(xv, f.z, acc[h + 2]); acc[h + 3] = fmaf(xv, f.w, acc[h + 3]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < HW; ++i)
    if (which >> i & 1u) sums[i] = acc[i];
}

// A step's activation at one pixel: acc, the convolution's channels; the pixel's rows of the reservoir, output and carry slabs.  Groups of 16
// channels are sent when one of them moved by more than the threshold; returns whether one was.
struct ExactRow {
  unsigned res, out, em, sw;
};
template <int HW, int ACT>
__device__ __forceinline__ bool exact_step(const ExactParams &p, const float *acc, const ExactRow r, const float *addend, int co) {
  auto f = [&](float4 v) { return make_float4(tc_act<ACT>(p.act, v.x), tc_act<ACT>(p.act, v.y), tc_act<ACT>(p.act, v.z), tc_act<ACT>(p.act, v.w)); };
  bool sent = false;
#pragma unroll
  for (int g = 0; g < HW / 16; ++g) {
    float4 o[4], x[4];
    float top = 0.0f;
    auto at = [&](int i) { return (unsigned)(4 * g + i ^ (int)r.sw) << 4; };
    if (ACT != MIE_ACT_NONE)
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = lds4(r.res + at(i));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int h = 4 * g + i;
      o[i] = make_float4(acc[4 * h], acc[4 * h + 1], acc[4 * h + 2], acc[4 * h + 3]);
      if (addend && co + 4 * h < p.cout) o[i] = f4add(o[i], *reinterpret_cast<const float4 *>(addend + co + 4 * h));
      if (ACT != MIE_ACT_NONE) {
        const float4 b = p.c.emitted ? lds4(r.em + at(i)) : f(x[i]);
        x[i] = f4add(x[i], o[i]);
        const float4 y = f(x[i]);
        o[i] = make_float4(y.x - b.x, y.y - b.y, y.z - b.z, y.w - b.w);
        sts4(r.res + at(i), x[i]);
      }
      if (co + 4 * h < p.cout) top = fmaxf(top, fmaxf(fmaxf(fabsf(o[i].x), fabsf(o[i].y)), fmaxf(fabsf(o[i].z), fabsf(o[i].w))));
    }
    const bool flag = top > p.c.thr, withheld = (p.c.thr > 0.0f || p.c.emitted) && !flag;
#pragma unroll
    for (int i = 0; i < 4; ++i) sts4(r.out + at(i), withheld ? make_float4(0.f, 0.f, 0.f, 0.f) : o[i]);
    sent |= flag;
  }
  return sent;
}

// The same from tensor memory, where an item's one or two segments all are (c: columns of the first): eight channels at a time in a loop
// that the instruction cache holds.  As straight code over registers the epilogue of 32 channels ran at 20 clocks an instruction and
// set the pace of the whole kernel (8 x 32 -> 32 at 480x640: 574 us; two items in hand, still straight, 472).
// STEP false: the dense pass, out = f(reservoir = conv + bias).
__device__ __forceinline__ void tmem_ld8_async(unsigned taddr, unsigned *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
// eight columns of segment j of channels 8 g on, as in exact_finish
template <int HW, bool FULL>
struct ExactColumns {
  unsigned hi, mid, low, last;
  __device__ __forceinline__ ExactColumns(unsigned c, unsigned j, unsigned g) {
    const unsigned at = c + j * exact_cols(HW, FULL), ch = 8u * g;
    hi = at + ch / (HW / 2) * HW + ch % (HW / 2);
    mid = hi + HW / 2;
    low = FULL ? hi + 2u * HW : at + 2u * HW + ch;
    last = hi + 2u * HW + HW / 2;
  }
};
__device__ __forceinline__ void tmem_st8(unsigned taddr, const float *v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// An item (tile t of this thread, ring units unit .. unit + units - 1) of which the parts did not hold all, in front of exact_finish: its
// finished sums take the place of the first segment's high columns, the other columns become zero.  exact_finish then has no
// branch for it (a test and a call per four channels cost FireFlowNet's step 5 %, mostly in registers).  Called by a converged warp;
// returns whether any of its pixels was concerned.
template <int HW, bool FULL>
__device__ __noinline__ bool exact_rare_item(const ExactParams &p, const SplitShared &sh, unsigned c, unsigned n_seg, unsigned unit, int units, unsigned odd, int t, int co) {
  const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3, TWo = (p.wout + 7) >> 3, THo = (p.hout + 7) >> 3;
  const int n = t / (TWo * THo), oy = t / TWo % THo * 8 + 2 * q + (lane >> 4), ox = t % TWo * 8 + (lane & 7);
  const bool valid = t >= 0 && oy < p.hout && ox < p.wout;
  bool wide = odd != 0u, any = false;
#pragma unroll 1
  for (int cu = 0; cu < units; ++cu) {
    const float scale = sh.inv[(unit + (unsigned)cu) % SPLIT_RING];
    wide |= scale != scale;
    if (valid && scale < 0.0f) any |= exact_small<HW>(p, sh, unit + (unsigned)cu, cu, co, nullptr, true);
  }
  if (!__any_sync(0xffffffffu, wide || any)) return false;
  float sums[HW];
#pragma unroll 1
  for (unsigned g = 0; g < HW / 8; ++g) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll 1
    for (unsigned j = 0; j < n_seg; ++j) {
      const ExactColumns<HW, FULL> at(c, j, g);
      const float inv = fabsf(sh.inv[(unit + (n_seg == 2u ? j * (unsigned)units >> 1 : 0u)) % SPLIT_RING]);
      unsigned a[8], b[8], d[8], e[8];
      tmem_ld8_async(at.hi, a);
      tmem_ld8_async(at.mid, b);
      tmem_ld8_async(at.low, d);
      if (FULL) tmem_ld8_async(at.last, e);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(split_sum(a[i], b[i], d[i], FULL ? e[i] : 0u, FULL), inv, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sums[8 * g + i] = acc[i] * __ldg(p.winv + co + 8 * g + i);
  }
  unsigned which = odd;
  if (any)
#pragma unroll 1
    for (int cu = 0; cu < units; ++cu)
      if (sh.inv[(unit + (unsigned)cu) % SPLIT_RING] < 0.0f) exact_small<HW>(p, sh, unit + (unsigned)cu, cu, co, sums, false);
#pragma unroll 1
  for (int cu = 0; cu < units; ++cu)
    if (!(fabsf(sh.inv[(unit + (unsigned)cu) % SPLIT_RING]) > 0.0f)) which = ~0u;
  if (valid && which) exact_fp32<HW>(p, n, oy, ox, co, which, sums);
  __syncwarp();
#pragma unroll 1
  for (unsigned j = 0; j < n_seg; ++j)
#pragma unroll 1
    for (unsigned g = 0; g < HW / 8; ++g) {
      const ExactColumns<HW, FULL> at(c, j, g);
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = j ? 0.0f : sums[8 * g + i];
      tmem_st8(at.hi, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = 0.0f;
      tmem_st8(at.mid, v);
      tmem_st8(at.low, v);
      if (FULL) tmem_st8(at.last, v);
    }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  return true;
}

// scales: the channels' inverse scales, four at a time, scale_step apart.
template <int HW, bool STEP, bool FULL, int ACT>
__device__ __forceinline__ bool exact_finish(const ExactParams &p, unsigned c, unsigned n_seg, float inv0, float inv1, const float4 *scales, unsigned scale_step,
                                             const ExactRow r, const float4 *col, bool valid, int64_t pix, int co) {
  auto f = [&](float4 v) { return make_float4(tc_act<ACT>(p.act, v.x), tc_act<ACT>(p.act, v.y), tc_act<ACT>(p.act, v.z), tc_act<ACT>(p.act, v.w)); };
  const float *addend = p.addend && valid ? p.addend + pix * p.addend_ps + co : nullptr;
  const bool thresholded = STEP && (p.c.thr > 0.0f || p.c.emitted);
  bool sent = !STEP;
  float top = 0.0f;
#pragma unroll 1
  for (unsigned g = 0; g < HW / 8; ++g) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll 1
    for (unsigned j = 0; j < n_seg; ++j) {
      const ExactColumns<HW, FULL> at(c, j, g);
      const float inv = j ? inv1 : inv0;
      unsigned a[8], b[8], d[8], e[8];
      tmem_ld8_async(at.hi, a);
      tmem_ld8_async(at.mid, b);
      tmem_ld8_async(at.low, d);
      if (FULL) tmem_ld8_async(at.last, e);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(split_sum(a[i], b[i], d[i], FULL ? e[i] : 0u, FULL), inv, acc[i]);
    }
#pragma unroll
    for (unsigned i = 0; i < 2; ++i) {
      const unsigned h = 2u * g + i, at = (h ^ r.sw) << 4;
      const int ch = (int)(4u * h);
      const bool real = co + ch < p.cout;
      const float4 w = lds4(smem_u32(scales + h * scale_step));
      float4 v = make_float4(acc[4 * i] * w.x, acc[4 * i + 1] * w.y, acc[4 * i + 2] * w.z, acc[4 * i + 3] * w.w);
      if (!STEP && p.bias) v = f4add(v, lds4(smem_u32(col + HW / 4 + h)));
      if (addend && real) v = f4add(v, *reinterpret_cast<const float4 *>(addend + ch));
      if (!STEP) {
        if (ACT != MIE_ACT_NONE) sts4(r.res + at, v);
        v = f(v);
      } else if (ACT != MIE_ACT_NONE) {
        const float4 x = lds4(r.res + at), xn = f4add(x, v), b = p.c.emitted ? lds4(r.em + at) : f(x), y = f(xn);
        v = make_float4(y.x - b.x, y.y - b.y, y.z - b.z, y.w - b.w);
        sts4(r.res + at, xn);
      }
      sts4(r.out + at, v);
      if (STEP && real) top = fmaxf(top, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    if (STEP && (g & 1u)) {      // a group of 16 channels is complete
      const bool flag = top > p.c.thr;
      if (thresholded && !flag)
#pragma unroll
        for (unsigned i = 0; i < 4; ++i) sts4(r.out + (((2u * g - 2u + i) ^ r.sw) << 4), make_float4(0.f, 0.f, 0.f, 0.f));
      sent |= flag;
      top = 0.0f;
    }
  }
  return sent;
}

// HW: channels that a thread of the epilogue finishes.  ALT: the two sets of epilogue warps take items in turn (CB = HW channels per
// block), else halves of each item's channels (CB = 2 HW).  STEP: a step (incremental activation, threshold, carry) instead of the dense
// pass.
template <int HW, bool STEP, bool ALT, bool FULL>
__global__ void __launch_bounds__(EXACT_THREADS, 1)
conv_exact_kernel(const __grid_constant__ ExactParams p, const __grid_constant__ ExactMaps maps) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int CB = ALT ? HW : 2 * HW, HB = CB / 2;      // HB: filter rows of a tap in this block, of either part
  constexpr unsigned half_bytes = HB * 64u, tap_bytes = 2u * half_bytes;   // this block's rows of one tap: [hi | lo] of its half of the channels
  const unsigned row_bytes = (unsigned)p.wp * 128u;
  const unsigned halo_bytes = ((unsigned)p.wp * 2u * row_bytes + 1023u) & ~1023u;
  const unsigned stage_bytes = tap_bytes * (unsigned)p.tps;
  __shared__ unsigned long long b_full[EXACT_MAX_STAGES], done[EXACT_MAX_STAGES], a_full[EXACT_MAX_HALOS], a_ready[EXACT_MAX_HALOS],
      a_empty[EXACT_MAX_HALOS], seg_empty[5], slab_full[2][2], item_full[2];
  __shared__ SplitShared s_split;
  __shared__ PairTapTable s_tap;
  __shared__ float4 s_col[2][2][HW / 4];      // per epilogue set: inverse scales and biases of its channels
  __shared__ float4 s_one;
  __shared__ unsigned s_odd[2];               // ... and a bit for every channel whose filter was not split
  __shared__ unsigned s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const unsigned crank = cluster_ctarank();
  const int bid = (int)(blockIdx.x >> 1), nblk = (int)(gridDim.x >> 1);
  const int THo = (p.hout + 7) >> 3, TWo = (p.wout + 7) >> 3;
  const int ntiles_total = p.n * THo * TWo;
  constexpr unsigned tmem_cols = 512u;

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&b_full[s], 1); mbar_init(&done[s], 1); }
    for (int s = 0; s < p.halos; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_ready[s], 2 * SPLIT_WARPS); mbar_init(&a_empty[s], 1); }
    for (int b = 0; b < p.segs; ++b) mbar_init(&seg_empty[b], ALT ? 8 : 16);
    if (ALT) { mbar_init(&item_full[0], 1); mbar_init(&item_full[1], 1); }
    if (STEP)
      for (int b = 0; b < 4; ++b) mbar_init(&slab_full[b >> 1][b & 1], 2);
    for (unsigned u = 0; u < SPLIT_RING; ++u) mbar_init(&s_split.inv_full[u], 1);
    s_abort = 0;
    s_one = make_float4(1.f, 1.f, 1.f, 1.f);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 3) {
    for (int i = lane; i < 50; i += 32) s_tap.off[i] = i < 49 ? (int)p.t.off[i] * 8 : 0;
    if (lane < 5) s_tap.first[lane] = p.t.first[lane];
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

  const int n_cblk = p.cout_pad / CB;
  // (no list: every tile, and nothing to wait for)
  const int n_active = __shfl_sync(0xffffffffu, p.list ? min(p.counts[0], p.max_tiles) : ntiles_total, 0);     // uniform, for the compiler too
  const int n_items = ((n_active + 3) >> 2) * n_cblk;
  const unsigned b_base = smem_u32(smem), a_base = b_base + (((unsigned)p.stages * stage_bytes + 1023u) & ~1023u);
  const int nv = p.t.nviews;

  const PairWork work = {bid, nblk, n_items, n_cblk, p.n_chunks, nv, crank, p.spin_limit, p.withhold_loads};
  const PairRing halos = {a_full, a_empty, a_base, halo_bytes, (unsigned)p.halos};
  if (warp == 0) {
    // =========================== halo producer ===========================
    pair_produce_halos<true>(work, halos, p.t, p.wp, row_bytes, p.list, n_active, ntiles_total, TWo, THo, p.counts, &s_abort,
                             [&](int u, int &v) { v = u; return &maps.in[u]; });
  } else if (warp == 1) {
    // =========================== filter producer: hi and lo rows of a tap ===========================
    const PairRing ring = {b_full, done, b_base, stage_bytes, (unsigned)p.stages};
    pair_produce_filter(work, ring, p.t, p.tps, tap_bytes, (int)crank * HB, CB, &s_abort, [](int u) { return u; }, [&](int) { return 2u * tap_bytes; },
                        [&](int, int tap, unsigned dst, unsigned bar, int row, int chunk) {
                          tma_load_4d_pair(dst, &maps.w, bar, 0, row, chunk, tap);
                          tma_load_4d_pair(dst + half_bytes, &maps.w, bar, 0, p.cout_pad + row, chunk, tap);
                        });
  } else if (warp == 2) {
    // =========================== MMA issuer (first block of the pair) ===========================
    if (crank == 0u) {
      const ExactIssue a = {bid, nblk, n_items, p.n_chunks, p.cin, p.tps, nv, tmem_base, a_base, b_base, row_bytes, halo_bytes, stage_bytes, (unsigned)p.stages,
                            (unsigned)p.halos, (unsigned)p.segs, p.spin_limit};
      exact_issue<CB, ALT, FULL>(a, s_tap, b_full, done, a_ready, a_empty, seg_empty, item_full, &s_abort);
    }
  } else if (warp >= 12) {
    // =========================== halos as two FP16 parts ===========================
    if (FULL && p.cin <= 16) pair_split_halos<true>(work, halos, a_ready, 2 * p.wp * p.wp, p.wp, n_active, tid - 384, s_split, &s_abort);
    else pair_split_halos<false>(work, halos, a_ready, 2 * p.wp * p.wp, p.wp, n_active, tid - 384, s_split, &s_abort);
  } else if (warp == 3) {
    pair_take_out(s_split, 2 * p.wp * p.wp, p.wp, lane);
  } else if (warp >= 4) {
    // =========================== epilogue: set `set` takes channels [set * HW, set * HW + HW) of the block, or every other item ===========================
    const int q = warp & 3, set = (warp - 4) >> 2;
    const int slot = (lane >> 3) & 1, prow = 2 * q + (lane >> 4), pcol = lane & 7;
    const unsigned lane_base = tmem_base + ((unsigned)(q * 32) << 16);
    // slabs of this set: output, then reservoir; 128 rows of HW channels, 16-byte pieces swizzled as TMA does for rows of
    // 128 bytes (piece ^ (row & 7)) or 64 bytes (piece ^ (row / 2 & 3))
    constexpr unsigned SLAB = 128u * HW * 4u;
    const int row = slot * 64 + prow * 8 + pcol, sw = HW == 32 ? row & 7 : (row >> 1) & 3;
    // output | reservoir | carry, once or twice
    const unsigned set_bytes = (unsigned)p.slab_bufs * SLAB, slabs = a_base + (unsigned)p.halos * halo_bytes + (unsigned)(set * p.slab_sets) * set_bytes;
    // the copies of slot s are issued by lane 8 s (whose pixel lies in it) of warp s of the set
    const bool chief = q < 2 && lane == 8 * q, has_res = p.act != MIE_ACT_NONE;
    if constexpr (STEP) tc_zero_stale(p.c, ntiles_total, THo, TWo, tid - 128, 256);
    // units and segments of an item; with ALT a set skips the other one's
    const int units = p.n_chunks * nv;
    unsigned n_seg = 0;
    for (int v = 0; v < nv; ++v) n_seg += (unsigned)((p.t.first[v + 1] - p.t.first[v] + p.tps - 1) / p.tps);
    n_seg *= (unsigned)p.n_chunks;
    unsigned seg = ALT ? (unsigned)set * n_seg : 0u, stage = 0, stage_par = 0, unit = ALT ? (unsigned)(set * units) : 0u, item_idx = 0;
    bool ok = true;
    const int first = ALT ? bid + set * nblk : bid, step = ALT ? 2 * nblk : nblk;
    auto column = [&](int item) { return (n_cblk == 1 ? 0 : item % n_cblk) * CB + (ALT ? 0 : set * HW); };
    auto entry = [&](int item) {      // this lane's tile of an item
      const int e = 4 * (n_cblk == 1 ? item : item / n_cblk) + 2 * (int)crank + slot, t = item >= n_items || e >= n_active ? -1 : p.list ? p.list[e] : e;
      return t < ntiles_total ? t : -1;
    };
    auto place = [&](int t, int &x, int &y, int &n) {
      const int r = p.div_tw ? (int)__umulhi((unsigned)t, p.div_tw) : t / TWo;
      n = p.div_th ? (int)__umulhi((unsigned)r, p.div_th) : r / THo;
      x = (t - r * TWo) * 8; y = (r - n * THo) * 8;
    };
    auto buffer = [&](unsigned idx) { return slabs + (p.slab_sets == 2 ? idx & 1u : 0u) * set_bytes; };
    auto slab_bar = [&](unsigned idx) { return &slab_full[set][p.slab_sets == 2 ? idx & 1u : 0u]; };
    // a chief asks for its tile's state for item `idx`, once the stores that last used the buffer have read it
    auto fetch_state = [&](int item, int t, unsigned idx) {
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      const int co = column(item);
      const unsigned bar = smem_u32(slab_bar(idx)), at = buffer(idx) + SLAB + (unsigned)slot * (SLAB / 2);
      const unsigned bytes = has_res && co < p.cout && t >= 0 ? (SLAB / 2) * (p.c.emitted ? 2u : 1u) : 0u;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
      if (bytes) {
        int x, y, n;
        place(t, x, y, n);
        tma_load_4d_raw(at, &maps.res, bar, co, x, y, n);
        if (p.c.emitted) tma_load_4d_raw(at + SLAB, &maps.emitted, bar, co, x, y, n);
      }
    };
    // inverse scales and biases into shared memory, for behind the set's barrier
    auto keep_column = [&](int at_col, float col) {
      if (at_col < 2 * HW) reinterpret_cast<float *>(s_col[set][at_col / HW])[at_col % HW] = col;
      if (q == 0) {
        const unsigned odd = __ballot_sync(0xffffffffu, at_col < HW && col != col);
        if (lane == 0) s_odd[set] = odd;
      }
    };
    int listed = entry(first);
    if (STEP && chief && first < n_items) fetch_state(first, listed, 0u);
    __syncwarp();
    for (int item = first; item < n_items && ok; item += step, ++item_idx) {
      // What the end of the item needs from global memory is asked for here and first looked at behind the segments.  The end of an
      // item is what bounds layers of few units per item (32 -> 32 3x3: the nine taps take 1500 clocks, the end took 6500 with the
      // state asked for at the item's start, divisions, one thread for all copies, and a load and a store in turn).
      const int co = column(item), at_col = q * 32 + lane, t = listed;
      listed = entry(item + step);
      const float col = at_col < HW ? __ldg(p.winv + co + at_col) : (at_col < 2 * HW && p.bias && co + at_col - HW < p.cout) ? __ldg(p.bias + co + at_col - HW) : 0.0f;
      int tx = 0, ty = 0, n = 0;
      if (t >= 0) place(t, tx, ty, n);
      const bool valid = t >= 0 && ty + prow < p.hout && tx + pcol < p.wout;
      const int64_t pix = valid ? (int64_t)(n * p.hout + ty + prow) * p.wout + tx + pcol : 0;
      const unsigned slab = buffer(item_idx), out_row = slab + (unsigned)row * (HW * 4u), res_row = out_row + SLAB, em_row = res_row + SLAB;
      bool sent = false;
      if constexpr (!ALT) {
        float acc[HW];
        float lost[HW];
        bool wide = false, small = false;
#pragma unroll
        for (int i = 0; i < HW; ++i) acc[i] = 0.0f;
        for (int cu = 0; cu < units && ok; ++cu, ++unit) {
          const int v = nv == 1 ? 0 : cu % nv;
          if (!(ok = __all_sync(0xffffffffu, mbar_wait(&s_split.inv_full[unit % SPLIT_RING], (unit / SPLIT_RING) & 1u, &s_abort, p.spin_limit)))) break;
          const float scale = s_split.inv[unit % SPLIT_RING], inv = fabsf(scale);
          for (int left = p.t.first[v + 1] - p.t.first[v]; left > 0; left -= p.tps) {
            if (!(ok = __all_sync(0xffffffffu, mbar_wait(&done[stage], stage_par, &s_abort, p.spin_limit)))) break;
            tc_fence_after();
            // [hi | mid] columns of this set's channels, and [lo x hi | lo x lo] or lo x hi alone
            const unsigned c = lane_base + seg * exact_cols(CB, FULL), own = c + (unsigned)set * CB, low = c + 2u * CB + (unsigned)set * (FULL ? CB : HW);
            tmem_add_split<HW, FULL>(own, own + HW, low, low + HW, inv, acc);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&seg_empty[seg]), 0));
            if (++seg == (unsigned)p.segs) seg = 0;
            if (++stage == (unsigned)p.stages) { stage = 0; stage_par ^= 1u; }
          }
          if (__builtin_expect(!(scale > 0.0f), 0)) {
            wide |= scale != scale;
            if (scale < 0.0f && valid) {
              if (!small)
#pragma unroll 1
                for (int i = 0; i < HW; ++i) lost[i] = 0.0f;
              small = true;
              exact_small<HW>(p, s_split, unit, cu, co, lost, false);
            }
            __syncwarp();
          }
        }
        keep_column(at_col, col);
        // a warp whose wait gave up goes on to the barrier of its set, where the four of them leave together
        if (!STEP && chief) {      // the buffer is free once the stores of its last item have read it
          if (p.slab_sets == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        if (STEP) {
          if (chief && p.slab_sets == 2 && item + step < n_items) fetch_state(item + step, listed, item_idx + 1u);
          __syncwarp();
          if (ok) ok = mbar_wait(slab_bar(item_idx), (p.slab_sets == 2 ? item_idx >> 1 : item_idx) & 1u, &s_abort, p.spin_limit);
        }
        __syncwarp();
        ok = set_all(1 + set, ok);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < HW / 4; ++h) {
          const float4 f = lds4(smem_u32(&s_col[set][0][h]));
          acc[4 * h] *= f.x; acc[4 * h + 1] *= f.y; acc[4 * h + 2] *= f.z; acc[4 * h + 3] *= f.w;
        }
        const unsigned odd = s_odd[set];
        if (__builtin_expect(valid && (small || wide || odd), 0)) {
          float sums[HW];
#pragma unroll
          for (int i = 0; i < HW; ++i) sums[i] = small ? acc[i] + lost[i] : acc[i];
          if (wide || odd) exact_fp32<HW>(p, n, ty + prow, tx + pcol, co, wide ? ~0u : odd, sums);
#pragma unroll
          for (int i = 0; i < HW; ++i) acc[i] = sums[i];
        }
        sent = valid;
        if constexpr (!STEP) {
#pragma unroll
          for (int h = 0; h < HW / 4; ++h) {
            const int c = co + 4 * h;
            float4 v = make_float4(acc[4 * h], acc[4 * h + 1], acc[4 * h + 2], acc[4 * h + 3]);
            if (p.bias) v = f4add(v, lds4(smem_u32(&s_col[set][1][h])));
            if (p.addend && valid && c < p.cout) v = f4add(v, *reinterpret_cast<const float4 *>(p.addend + pix * p.addend_ps + c));
            const unsigned at = (unsigned)(h ^ sw) << 4;
            if (p.act != MIE_ACT_NONE) {
              sts4(res_row + at, v);
              v = p.act == MIE_ACT_RELU ? make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f))
                                        : make_float4(tc_act_call(p.act, v.x), tc_act_call(p.act, v.y), tc_act_call(p.act, v.z), tc_act_call(p.act, v.w));
            }
            sts4(out_row + at, v);
          }
        } else {
          // one stretch of code per activation: what is run once per item runs out of the instruction cache
          const ExactRow r = {res_row, out_row, em_row, (unsigned)sw};
          const float *ad = p.addend && valid ? p.addend + pix * p.addend_ps : nullptr;
          if (p.act == MIE_ACT_RELU) sent = exact_step<HW, MIE_ACT_RELU>(p, acc, r, ad, co);
          else if (p.act == MIE_ACT_NONE) sent = exact_step<HW, MIE_ACT_NONE>(p, acc, r, ad, co);
          else sent = exact_step<HW, MIE_ACT_SIGMOID>(p, acc, r, ad, co);
          sent = sent && valid;
        }
      } else {
        ok = __all_sync(0xffffffffu, mbar_wait(&item_full[set], item_idx & 1u, &s_abort, p.spin_limit));
        float inv[2];
        bool noted = false;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const unsigned u = unit + (n_seg == 2u ? (unsigned)(j * units) >> 1 : 0u);
          ok = __all_sync(0xffffffffu, ok && mbar_wait(&s_split.inv_full[u % SPLIT_RING], (u / SPLIT_RING) & 1u, &s_abort, p.spin_limit));
          const float scale = s_split.inv[u % SPLIT_RING];
          noted |= !(scale > 0.0f);
          inv[j] = fabsf(scale);
        }
        keep_column(at_col, col);
        // a warp whose wait gave up goes on to the barrier of its set, where the four of them leave together
        if (!STEP && chief) {      // the buffer is free once the stores of its last item have read it
          if (p.slab_sets == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        if (STEP) {
          if (chief && p.slab_sets == 2 && item + step < n_items) fetch_state(item + step, listed, item_idx + 1u);
          __syncwarp();
          if (ok) ok = mbar_wait(slab_bar(item_idx), (p.slab_sets == 2 ? item_idx >> 1 : item_idx) & 1u, &s_abort, p.spin_limit);
        }
        __syncwarp();
        ok = set_all(1 + set, ok);
        if (!ok) break;
        tc_fence_after();
        const ExactRow r = {res_row, out_row, em_row, (unsigned)sw};
        const unsigned c = lane_base + seg * exact_cols(CB, FULL);
        const float4 *scales = s_col[set][0];
        unsigned scale_step = 1u;
        const unsigned odd = s_odd[set];
        if (__builtin_expect(noted || odd, 0)) {
          if (exact_rare_item<HW, FULL>(p, s_split, c, n_seg, unit, units, odd, t, co)) {
            inv[0] = inv[1] = 1.0f;
            scales = &s_one; scale_step = 0u;
          }
        }
        const float4 *own = s_col[set][0];
        if (p.act == MIE_ACT_RELU) sent = exact_finish<HW, STEP, FULL, MIE_ACT_RELU>(p, c, n_seg, inv[0], inv[1], scales, scale_step, r, own, valid, pix, co);
        else if (p.act == MIE_ACT_NONE) sent = exact_finish<HW, STEP, FULL, MIE_ACT_NONE>(p, c, n_seg, inv[0], inv[1], scales, scale_step, r, own, valid, pix, co);
        else sent = exact_finish<HW, STEP, FULL, MIE_ACT_SIGMOID>(p, c, n_seg, inv[0], inv[1], scales, scale_step, r, own, valid, pix, co);
        sent = sent && valid;
        unit += 2u * (unsigned)units;
        tc_fence_before();
        __syncwarp();
        for (unsigned j = 0; j < n_seg; ++j)
          if (lane == 0) mbar_arrive_remote(mapa_shared(smem_u32(&seg_empty[seg + j]), 0));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
      if (chief) {
        if (co < p.cout && t >= 0) {
          const unsigned half = (unsigned)slot * (SLAB / 2);
          tma_store_slab(slab + half, &maps.out, co, tx, ty, n);
          if (has_res) tma_store_slab(slab + SLAB + half, &maps.res, co, tx, ty, n);
          if (STEP && p.c.emitted) tma_add_slab(slab + half, &maps.emitted, co, tx, ty, n);   // the carry advances by what was sent
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");      // (also without a copy: the waits count groups)
      }
      if (STEP && chief && p.slab_sets == 1 && item + step < n_items) fetch_state(item + step, listed, item_idx + 1u);
      __syncwarp();
      // the pixels sent (dense: every pixel written); ballot bytes: [tile 0 row 2q][tile 1 row 2q][tile 0 row 2q+1][tile 1 row 2q+1]
      const unsigned bal = __ballot_sync(0xffffffffu, sent);
      if ((lane == 0 || lane == 8) && t >= 0) {
        const unsigned rows = ((bal >> lane) & 0xFFu) | (((bal >> (16 + lane)) & 0xFFu) << 8);
        // (dense: every column block has the same rows to say, and says them whatever stood there)
        if (!STEP) reinterpret_cast<unsigned short *>(p.out_bits32)[4 * (size_t)t + q] = (unsigned short)rows;
        else if (rows) atomicOr(p.out_bits32 + 2 * (size_t)t + (q >> 1), rows << ((q & 1) * 16));
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

// Floats of a packed filter in front of its inverse scales.
static inline int64_t exact_scales_at(int cin, int cout_pad, int k) { return (int64_t)k * k * divup(cin, 32) * 2 * cout_pad * 16; }

// How a launch divides its columns and its shared memory; `stages` < 2: no split of it fits.
struct ExactShape {
  PairTaps t;
  int wp, cb, hw, tps, stages, halos, segs, slab_bufs, slab_sets;   // hw: channels of an epilogue thread
  bool alt, full;
  size_t smem;
};
static ExactShape exact_shape(const mie_conv_args *a) {
  ExactShape h;
  pair_make_taps(a->k, a->stride, a->pad, &h.t, &h.wp);
  const int quads = divup(a->max_tiles, 4), clusters_max = MIE_SM_COUNT / 2;
  // 64 channels per block unless blocks of 32, which take 0.75 of its time, need fewer rounds for it (5x5: 305 and 245 clocks per tap and
  // 32 channels, 3x3 430 and 300)
  h.cb = 32;
  h.full = !a->refresh && a->cin * a->k * a->k < 256;
  if (!h.full && a->cout_pad % 64 == 0 &&
      (int64_t)divup(quads * (a->cout_pad / 64), clusters_max) * 100 <= (int64_t)divup(quads * (a->cout_pad / 32), clusters_max) * 75)
    h.cb = 64;
  // Taps of a segment: its truncation grows with its additions, one per 16 channels and tap, the FP32 kernel's rounding with the whole
  // reduction.  Dense: the longest whose error is not above the FP32 kernel's, nor above that of the two TF32 parts that stood here, for
  // rectified inputs (segments of 3 / 5 / 9 taps over the FP32 kernel's error: 125 products 0.84 / 0.91 / 1.16, 288 0.75 / 0.99 / 1.68, 576
  // 0.53 / 0.70 / 1.22, 1152 0.40 / 0.52 / 0.88, 1600 0.36 / 0.47 / 0.71, 2304 0.29 / 0.36 / 0.60).  A step's result is a change, whose
  // error is a fraction of the state's, and its three blocks of TF32 channels were never summed in segments at all.
  const int depth = a->cin * a->k * a->k;
  const int most = !a->refresh ? 9 : depth < 100 ? 2 : depth < 400 ? (a->cin > 16 ? 3 : 5) : depth < 1600 ? 5 : 9;
  int taps = 0, n_seg = 0;
  for (int v = 0; v < h.t.nviews; ++v) taps = std::max(taps, h.t.first[v + 1] - h.t.first[v]);
  h.tps = divup(taps, divup(taps, most));
  for (int v = 0; v < h.t.nviews; ++v) n_seg += divup(h.t.first[v + 1] - h.t.first[v], h.tps);
  n_seg *= divup(a->cin, 32);
  // Items of one or two segments are bound by what follows them, a chain of about 7000 clocks: two of them are in hand at once then
  // (all segments of both in tensor memory).
  h.alt = h.cb == 32 && n_seg <= 2;
  h.hw = h.alt ? 32 : h.cb / 2;
  h.slab_bufs = 1 + (a->act != MIE_ACT_NONE) + (a->emitted != nullptr);
  // two buffers of slabs where they are small: the state of an item then arrives, and its results leave, while another is computed
  h.slab_sets = h.hw == 16 ? 2 : 1;
  const int halo_bytes = (h.wp * 2 * h.wp * 128 + 1023) & ~1023, slab_bytes = 2 * h.slab_sets * h.slab_bufs * 128 * h.hw * 4;
  const int budget = 222 * 1024 - slab_bytes;
  // Units of a single stage (3x3) need halo buffers more than stages: load, split and instructions of a unit are three links of a chain
  // (res 256 -> 256: three halos and two stages 144 us, two and three 157).  Longer ones need the filter ahead (64 -> 32 5x5: 787 us with
  // three halos and four stages, 939 with four and two).
  const int ring = h.tps == taps ? 2 : 3;
  h.halos = EXACT_MAX_HALOS;
  while (h.halos > 2 && budget - h.halos * halo_bytes < ring * h.tps * h.cb * 64) --h.halos;
  while (h.tps > 1 && budget - h.halos * halo_bytes < 2 * h.tps * h.cb * 64) --h.tps;
  const int stage_bytes = h.tps * h.cb * 64;
  h.stages = std::min((budget - h.halos * halo_bytes) / stage_bytes, EXACT_MAX_STAGES);
  // ... two items' worth with `alt`: an item's barrier is not signalled again before its set has looked at it
  h.segs = h.alt ? 2 * n_seg : std::min(h.stages, (int)exact_segs(h.cb, h.full));      // the epilogue learns of a segment from its stage's barrier
  h.smem = (size_t)((h.stages * stage_bytes + 1023) & ~1023) + (size_t)h.halos * halo_bytes + slab_bytes + 1024;
  return h;
}

// A dense evaluation (`refresh`), or a step of a layer in split precision, that the kernel takes.
bool exact_takes(const mie_conv_args *a) {
  // a field one pixel wide or high has no odd columns or rows: that parity view of stride 2 would be empty, and a tensor map
  // cannot say so
  if (a->stride == 2 && (a->hin == 1 || a->win == 1)) return false;
  if (a->refresh ? a->head != nullptr : (a->bias || ((a->thr > 0.0f || a->emitted) && !g_opt_tc_thresholded))) return false;
  return a->wpacked_exact && a->k >= 3 && a->k <= 7 && (a->k & 1) && (a->stride == 1 || a->stride == 2) && !a->in2 && !a->accum &&
         a->in_ps % 4 == 0 && aligned16(a->in) && aligned16(a->wpacked_exact) && a->cout % 4 == 0 && a->out_ps % 4 == 0 &&
         aligned16(a->out) && (!a->res || (a->res_ps % 4 == 0 && aligned16(a->res))) && (!a->addend || (a->addend_ps % 4 == 0 && aligned16(a->addend))) &&
         (!a->emitted || (a->emitted_ps % 4 == 0 && aligned16(a->emitted))) && a->cout_pad % 32 == 0 && exact_shape(a).stages >= 2;
}

// fw: the filter in fp32, entry (tap, ci, co) at fw[tap * fw_tap + ci * fw_ci + co]
int launch_conv_exact(const mie_conv_args *a, const float *fw, int64_t fw_tap, int64_t fw_ci, cudaStream_t st) {
  const ExactShape h = exact_shape(a);
  ExactParams p;
  memset(&p, 0, sizeof(p));
  p.spin_limit = g_opt_spin_limit;
  p.withhold_loads = g_opt_withhold_loads;
  p.in = a->in; p.in_ps = a->in_ps; p.hin = a->hin; p.win = a->win; p.k = a->k; p.stride = a->stride; p.pad = a->pad;
  p.fw = fw; p.fw_tap = fw_tap; p.fw_ci = fw_ci; p.fw_vec = aligned16(fw) && fw_tap % 4 == 0 && fw_ci % 4 == 0;
  p.cin = a->cin; p.cout = a->cout; p.cout_pad = a->cout_pad; p.n_chunks = divup(a->cin, 32);
  p.winv = a->wpacked_exact + exact_scales_at(a->cin, a->cout_pad, a->k);
  p.n = a->n; p.hout = a->hout; p.wout = a->wout;
  p.list = a->list; p.counts = a->counts; p.max_tiles = a->max_tiles;
  p.out = a->out; p.out_ps = a->out_ps; p.out_bits32 = reinterpret_cast<unsigned int *>(a->out_bits);
  p.act = a->act; p.res = a->res; p.res_ps = a->res_ps; p.addend = a->addend; p.addend_ps = a->addend_ps; p.bias = a->bias;
  p.tail = tail_for_kernel(a->tail);
  p.t = h.t; p.wp = h.wp; p.cb = h.cb; p.tps = h.tps; p.stages = h.stages; p.halos = h.halos; p.segs = h.segs; p.slab_bufs = h.slab_bufs; p.slab_sets = h.slab_sets;
  // n / d = high word of n * ceil(2^32 / d), exact while n * d < 2^32
  const unsigned tw = (unsigned)divup(a->wout, 8), th = (unsigned)divup(a->hout, 8);
  auto magic = [&](unsigned d) { return d > 1 && (uint64_t)a->n * tw * th * d < (1ull << 32) ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u; };
  p.div_tw = magic(tw); p.div_th = magic(th);
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
    if (!tc_encode(&maps.in[v], 4, a->in + ((int64_t)py * a->win + px) * a->in_ps, dims, str, box_in, CU_TENSOR_MAP_SWIZZLE_128B)) return MIE_EINVAL;
  }
  {
    // [tap][chunk][hi rows | lo rows][32 FP16 = 16 floats]
    const cuuint64_t rows = 2 * (cuuint64_t)a->cout_pad, nch = (cuuint64_t)p.n_chunks;
    const cuuint64_t dims[4] = {16, rows, nch, (cuuint64_t)(a->k * a->k)};
    const cuuint64_t str[3] = {64, rows * 64, nch * rows * 64};
    const cuuint32_t box_w[4] = {16, (cuuint32_t)(p.cb / 2), 1, 1};
    if (!tc_encode(&maps.w, 4, a->wpacked_exact, dims, str, box_w, CU_TENSOR_MAP_SWIZZLE_64B)) return MIE_EINVAL;
  }
  {
    // epilogue slabs: a set's channels of one tile
    const cuuint32_t box[4] = {(cuuint32_t)h.hw, 8, 8, 1};
    const CUtensorMapSwizzle sw = h.hw == 32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    auto slab_map = [&](CUtensorMap *m, const float *base, int64_t ps) {
      const cuuint64_t dims[4] = {(cuuint64_t)a->cout, (cuuint64_t)a->wout, (cuuint64_t)a->hout, (cuuint64_t)a->n};
      const cuuint64_t str[3] = {(cuuint64_t)ps * 4, (cuuint64_t)a->wout * ps * 4, (cuuint64_t)a->hout * a->wout * ps * 4};
      return tc_encode(m, 4, base, dims, str, box, sw);
    };
    if (!slab_map(&maps.out, a->out, a->out_ps) || (a->act != MIE_ACT_NONE && !slab_map(&maps.res, a->res, a->res_ps)) ||
        (a->emitted && !slab_map(&maps.emitted, a->emitted, a->emitted_ps)))
      return MIE_EINVAL;
  }
  const int n_cblk = a->cout_pad / p.cb;
  const int64_t items = (int64_t)quads * n_cblk;
  int clusters = (int)(items < clusters_max ? items : clusters_max);
  if (!a->refresh) {
    TcParams &c = p.c;
    c.thr = a->thr; c.emitted = a->emitted; c.stale = a->stale; c.counts = a->counts; c.max_tiles = a->max_tiles;
    c.out = a->out; c.out_ps = a->out_ps; c.cout = a->cout; c.hout = a->hout; c.wout = a->wout;
    if (a->head) {
      // (a kernel that finds its own tiles was slower here: FireFlowNet's six layers 368 us a step, with the launches 346)
      const mie_tail_job *j = a->head;
      const int r = mie_tiles_dilate(j->in_bits, j->N, j->Hin, j->Win, j->Hout, j->Wout, j->k, j->stride, j->pad, j->union_bits, j->out_bits, j->list, j->stale,
                                     j->counts, j->flags, st);
      if (r != MIE_OK) return r;
    }
  }
  static int smem_set[8][MAX_DEVICES] = {{0}};
  auto launch = [&](auto kernel, int i) {
    const int r = ensure_dynamic_smem(kernel, smem_set[i], smem);
    if (r != MIE_OK) return r;
    launch_chained_cluster(kernel, dim3((unsigned)(2 * clusters)), dim3(EXACT_THREADS), smem, st, 2, p, maps);
    return check_launch();
  };
  if (a->refresh)
    return h.alt ? launch(conv_exact_kernel<32, false, true, false>, 0) : h.cb == 64 ? launch(conv_exact_kernel<32, false, false, false>, 1)
                                                                                     : launch(conv_exact_kernel<16, false, false, false>, 2);
  if (h.full) return h.alt ? launch(conv_exact_kernel<32, true, true, true>, 6) : launch(conv_exact_kernel<16, true, false, true>, 7);
  return h.alt ? launch(conv_exact_kernel<32, true, true, false>, 3) : h.cb == 64 ? launch(conv_exact_kernel<32, true, false, false>, 4)
                                                                                  : launch(conv_exact_kernel<16, true, false, false>, 5);
}

// A field with a pixel stride or an address that TMA cannot read (5 bins of a voxel grid) as one it can: one read and one write.
// A thread per four channels of a pixel; counts (may be null): the work list of the convolution that reads the copy, nothing is
// copied where it lists no tile.  zero (may be null): a second field of that layout, cleared.
__global__ void __launch_bounds__(256) pad_field_kernel(const float *__restrict__ in, int64_t in_ps, int C, int64_t pixels, float *__restrict__ out,
                                                        float *__restrict__ zero, int64_t out_ps, int quads, int vec, const int32_t *counts) {
  grid_dependency_wait();
  grid_dependency_trigger();
  if (counts && counts[0] == 0) return;
  const int64_t total = pixels * quads;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t px = i / quads;
    const int c = (int)(i - px * quads) * 4;
    float4 v;
    if (vec) {
      v = *reinterpret_cast<const float4 *>(in + px * in_ps + c);
    } else {
      const float *x = in + px * in_ps + c;
      v = make_float4(x[0], c + 1 < C ? x[1] : 0.0f, c + 2 < C ? x[2] : 0.0f, c + 3 < C ? x[3] : 0.0f);
    }
    *reinterpret_cast<float4 *>(out + px * out_ps + c) = v;
    if (zero) *reinterpret_cast<float4 *>(zero + px * out_ps + c) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// [tap][chunk][hi: cout_pad rows | lo: cout_pad rows][32 FP16] <- w[cout][cin][ky][kx] (ihwo: stored [cin][ky][kx][cout]), zero padded, then
// cout_pad inverse scales.  A channel's scale puts its largest entry into [2^15, 2^16).  NaN for a channel whose entries two FP16 numbers
// cannot hold: infinities, NaN, or entries above 2^10 (2^100 in any case) beside entries 2^-36 of them; its outputs are computed
// with FP32 instructions.  Of the others an entry below 2^-27 of the largest is held to 2^-52 of that, which is 2^-42 of an input at most.
// (Such entries taken out, as the input's values are, cost 64 -> 64 3x3 at 264x352 67 us for 37 with one of them, and 440 with one input
// channel of them, which a trained network may well have.)  A block per NC channels, which it reads twice, the second time from the caches.
template <int NC>
__global__ void __launch_bounds__(512) pack_weights_exact_kernel(const float *__restrict__ w, int cout, int cin, int k, int nch, int cout_pad, float *__restrict__ wp,
                                                                 int64_t scales_at, int ihwo) {
  __shared__ unsigned s_max[NC], s_min[NC];
  const int kk = k * k, co0 = blockIdx.x * NC, n = cin * kk;
  if (threadIdx.x < NC) { s_max[threadIdx.x] = 0u; s_min[threadIdx.x] = 0x7FFFFFFFu; }
  __syncthreads();
  // neighbouring threads read neighbouring addresses: channels first where they are stored together
  const int c = ihwo ? (int)threadIdx.x % NC : 0, step = ihwo ? (int)blockDim.x / NC : (int)blockDim.x, first = ihwo ? (int)threadIdx.x / NC : (int)threadIdx.x;
  auto entry = [&](int i, int co) { return ihwo ? w[(int64_t)i * cout + co] : w[(int64_t)co * n + i]; };      // i = ci * kk + tap
  for (int cc = ihwo ? c : 0; cc < (ihwo ? c + 1 : NC); ++cc) {
    unsigned m = 0u, least = 0x7FFFFFFFu;
    if (co0 + cc < cout)
      for (int i = first; i < n; i += step) {
        const unsigned u = __float_as_uint(entry(i, co0 + cc)) & 0x7FFFFFFFu;
        m = max(m, u);
        if (u) least = min(least, u);
      }
    atomicMax(&s_max[cc], m);
    atomicMin(&s_min[cc], least);
  }
  __syncthreads();
  __half *out = reinterpret_cast<__half *>(wp);
  for (int cc = ihwo ? c : 0; cc < (ihwo ? c + 1 : NC); ++cc) {
    const unsigned m = s_max[cc], e = split_exponent(m);
    const float scale = split_scale(e);
    const int co = co0 + cc;
    if (first == 0 && co < cout_pad) {
      const bool wide = m > 0x71800000u || (m > 0x44800000u && (m >> 23) - (s_min[cc] >> 23) > 36u);
      wp[scales_at + co] = wide ? __uint_as_float(0x7FC00000u) : split_inverse(e);
    }
    for (int i = first; i < nch * 32 * kk; i += step) {
      const int ci = i / kk, tap = i - ci * kk;
      // (up to 16 channels: what two parts leave lies in the hi rows where 16 channels further on would be)
      const bool third = cin <= 16 && ci >= 16;
      const float v = co < cout && (third ? ci - 16 : ci) < cin ? entry(third ? i - 16 * kk : i, co) * scale : 0.0f;
      __half h = __float2half_rn(v);
      if (third) {
        const float r = (v - __half2float(h)) * 2048.0f;
        h = __float2half_rn(r - __half2float(__float2half_rn(r)));
      }
      const int64_t at = (((int64_t)tap * nch + (ci >> 5)) * 2 * cout_pad + co) * 32 + (ci & 31);
      out[at] = h;
      out[at + (int64_t)cout_pad * 32] = third ? __float2half_rn(0.0f) : __float2half_rn((v - __half2float(h)) * 2048.0f);
    }
  }
}

int pack_exact(const float *w, int cout, int cin, int k, int ihwo, float *wpacked, cudaStream_t st) {
  int64_t total;
  const int s = mie_conv_pack_dims_exact(cin, cout, k, &total);
  if (s != MIE_OK) return s;
  const int cout_pad = divup(cout, 32) * 32, nch = divup(cin, 32);
  const int64_t at = exact_scales_at(cin, cout_pad, k);
  if (ihwo) pack_weights_exact_kernel<4><<<cout_pad / 4, 512, 0, st>>>(w, cout, cin, k, nch, cout_pad, wpacked, at, 1);
  else pack_weights_exact_kernel<1><<<cout_pad, 512, 0, st>>>(w, cout, cin, k, nch, cout_pad, wpacked, at, 0);
  return check_launch();
}

int pad_field(const float *in, int64_t in_ps, int C, int64_t pixels, float *out, float *zero, int64_t out_ps, const int32_t *counts, cudaStream_t st) {
  if (!in || !out || C <= 0 || pixels <= 0 || in_ps < C || out_ps < (C + 3) / 4 * 4 || out_ps % 4) return MIE_EINVAL;
  if (!aligned16(out) || !aligned16(zero)) return MIE_EALIGN;
  const int quads = divup(C, 4), vec = C % 4 == 0 && in_ps % 4 == 0 && aligned16(in);
  int64_t blocks = divup64(pixels * quads, 256);
  if (blocks > MIE_SM_COUNT * 16) blocks = MIE_SM_COUNT * 16;
  launch_chained(pad_field_kernel, dim3((unsigned)blocks), dim3(256), 0, st, in, in_ps, C, pixels, out, zero, out_ps, quads, vec, counts);
  return check_launch();
}

}  // namespace mie

// (for callers of earlier versions)
extern "C" int mie_split_exact(const float *in, int64_t in_ps, int C, int64_t pixels, float *hi, float *lo, int64_t out_ps, void *stream) {
  if (!lo) return MIE_EINVAL;
  return pad_field(in, in_ps, C, pixels, hi, lo, out_ps, nullptr, (cudaStream_t)stream);
}

extern "C" int mie_pad_field(const float *in, int64_t in_ps, int C, int64_t pixels, float *out, int64_t out_ps, void *stream) {
  return pad_field(in, in_ps, C, pixels, out, nullptr, out_ps, nullptr, (cudaStream_t)stream);
}

extern "C" int mie_conv_pack_dims_exact(int cin, int cout, int k, int64_t *n_floats) {
  if (cin <= 0 || cout <= 0 || k <= 0 || !n_floats) return MIE_EINVAL;
  const int cout_pad = divup(cout, 32) * 32;
  *n_floats = exact_scales_at(cin, cout_pad, k) + cout_pad;
  return MIE_OK;
}

extern "C" int mie_pack_conv_weights_exact(const float *w_oihw, int cout, int cin, int k, float *wpacked, void *stream) {
  if (!w_oihw || !wpacked) return MIE_EINVAL;
  return pack_exact(w_oihw, cout, cin, k, 0, wpacked, (cudaStream_t)stream);
}
