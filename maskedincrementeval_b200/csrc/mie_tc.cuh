// What the tensor-core convolution kernels share (sm_100a): barriers, TMA and tcgen05 wrappers, operand descriptors, the
// activation of the epilogues, and the own-tiles mode.
#pragma once
#include <cuda.h>
#include <stdlib.h>
#include <string.h>
#include "mie_common.cuh"

namespace mie {

struct TcParams {
  int cin, cout, cout_pad, cin_pad;   // cin_pad: multiple of 32 (filter K extent)
  int n, hin, win, hout, wout, k, stride, pad;
  const int32_t *list; const int32_t *stale; int32_t *counts; int max_tiles;
  float *out; int64_t out_ps; unsigned int *out_bits32;
  int act; float thr;
  float *res; int64_t res_ps;
  float *emitted; int64_t emitted_ps;
  const float *addend; int64_t addend_ps;
  int nb;        // output channels per block (multiple of 16, <= 256)
  int stages;    // pipeline depth
  int tps;       // halo kernel: filter taps per pipeline stage (divides k*k)
  int issuers;   // halo kernel: 1 or 2 MMA-issuing warps (2: stages alternate, one accumulator each)
  unsigned spin_limit;   // iterations after which a barrier wait gives up (MIE_OPT_TC_SPIN_LIMIT)
  int withhold_loads;    // self-test: the producers issue nothing, so the first wait runs out (MIE_OPT_TC_WITHHOLD_LOADS)
  mie_tail_job tail;     // the next convolution's tile dilation, run by the last block (list == nullptr: none)
  mie_tail_job head;     // this convolution's own tile dilation, run by block 0 while the others wait (list == nullptr: none)
  int ksplit;            // halo kernel: CTAs of a cluster that share one work item, each reducing 1/ksplit of the
                         // input-channel chunks (1: no cluster)
  int own;               // every block finds the active tiles among those it owns itself (`head` describes the test);
                         // no global list is read
  unsigned long long *own_words;   // own mode, tiles that several blocks finish: the word under construction ...
  int *own_tickets;                // ... and how many epilogue warps have contributed to it (both zero between launches)
};

// ---- host side, defined in mie_conv_tc.cu ----
// A tensor map of fp32 elements (encoded once per set of arguments and host thread); false when the driver refuses it.
bool tc_encode(CUtensorMap *m, int rank, const void *base, const cuuint64_t *dims, const cuuint64_t *strides_bytes,
               const cuuint32_t *box, CUtensorMapSwizzle swizzle);
// The CTA-pair kernel (mie_conv_pair.cu).
bool pair_takes(const mie_conv_args *a);
int launch_conv_pair(const mie_conv_args *a, cudaStream_t st);
extern unsigned g_opt_spin_limit;   // MIE_OPT_TC_SPIN_LIMIT
extern int g_opt_tc_thresholded;    // MIE_OPT_TC_THRESHOLDED
extern int g_opt_withhold_loads;    // MIE_OPT_TC_WITHHOLD_LOADS
extern int g_opt_own_kernels;       // MIE_OPT_TC_OWN_KERNELS

// cudaFuncAttributeMaxDynamicSharedMemorySize is a per-device attribute of a kernel: the largest value set so far is
// remembered per device, so a process that drives several GPUs raises the limit on each of them.
constexpr int MAX_DEVICES = 64;
template <typename Kernel>
static inline int ensure_dynamic_smem(Kernel kernel, int *set_per_device, size_t smem) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { set_cuda_error(e); return MIE_ECUDA; }
  if (dev < 0 || dev >= MAX_DEVICES) return MIE_EUNSUPPORTED;
  if ((int)smem > set_per_device[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_cuda_error(e); return MIE_ECUDA; }
    set_per_device[dev] = (int)smem;
  }
  return MIE_OK;
}

namespace {

// -DMIE_TC_TRACE (debug builds only): conv_tc_kernel records SM-clock timestamps of its phases per block, read back
// through mie_debug_trace().  Compiled out of the product build.
#ifdef MIE_TC_TRACE
__device__ long long g_tc_trace[1024 * 16];
__device__ __forceinline__ long long trace_gtime() { long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }
#define TC_TRACE(slot) do { if (blockIdx.x < 1024) g_tc_trace[blockIdx.x * 16 + (slot)] = clock64(); } while (0)
#define TC_TRACE_G(slot) do { if (blockIdx.x < 1024) g_tc_trace[blockIdx.x * 16 + (slot)] = trace_gtime(); } while (0)
#define TC_TRACE_V(slot, v) do { if (blockIdx.x < 1024) g_tc_trace[blockIdx.x * 16 + (slot)] = (v); } while (0)
#else
#define TC_TRACE(slot) do { } while (0)
#define TC_TRACE_G(slot) do { } while (0)
#define TC_TRACE_V(slot, v) do { } while (0)
#endif

constexpr int TC_THREADS = 192;
constexpr int A_STAGE_BYTES = 128 * 128;  // 128 pixels x 32 channels x 4 B
constexpr unsigned SPIN_LIMIT = 1u << 20;   // default of TcParams::spin_limit

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait on a phase parity.  Returns false when the limit ran out or another role gave up.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, volatile int *abort_flag, unsigned limit) {
  const unsigned addr = smem_u32(bar);
  for (unsigned it = 0; it < limit; ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

__device__ __forceinline__ void tma_load_4d_raw(unsigned smem_addr, const CUtensorMap *map, unsigned bar_addr, int c0, int c1,
                                                int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_addr), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar_addr), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

__device__ __forceinline__ void tma_load_5d_raw(unsigned smem_addr, const CUtensorMap *map, unsigned bar_addr, int c0, int c1,
                                                int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_addr), "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar_addr), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, rows of 128 bytes,
// 8-row groups 1024 bytes apart.  Bits: [0,14) address>>4, [16,30) leading offset>>4 (unused for swizzled
// K-major), [32,46) stride offset>>4, [46,48) version = 1, [61,64) layout = 2 (128-byte swizzle).
__device__ __forceinline__ unsigned long long make_smem_desc(unsigned smem_addr, unsigned sbo_bytes = 1024) {
  unsigned long long d = 0;
  d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);
  d |= (unsigned long long)1 << 16;
  d |= (unsigned long long)(sbo_bytes >> 4) << 32;
  d |= (unsigned long long)1 << 46;
  d |= (unsigned long long)2 << 61;
  return d;
}

// Descriptor of a K-major operand stored WITHOUT swizzle: 8 rows x 16 bytes form one contiguous 128-byte core
// matrix; `lbo_bytes` is the distance between the two core matrices an MMA reads along K, `sbo_bytes` the distance
// between consecutive 8-row groups.  The start address only needs 16-byte alignment, which is what lets a filter
// tap be expressed as an address shift inside a resident halo tile.
__device__ __forceinline__ unsigned long long make_smem_desc_plain(unsigned smem_addr, unsigned lbo_bytes, unsigned sbo_bytes) {
  unsigned long long d = 0;
  d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);
  d |= (unsigned long long)(lbo_bytes >> 4) << 16;
  d |= (unsigned long long)(sbo_bytes >> 4) << 32;
  d |= (unsigned long long)1 << 46;
  return d;
}

// Instruction descriptor for kind::tf32, FP32 accumulator, both operands K-major, M = 128.
__device__ __forceinline__ unsigned make_idesc_tf32(int n) {
  unsigned d = 0;
  d |= 1u << 4;                 // accumulator format F32
  d |= 2u << 7;                 // A format TF32
  d |= 2u << 10;                // B format TF32
  d |= (unsigned)(n >> 3) << 17;
  d |= (unsigned)(128 >> 4) << 24;
  return d;
}

// The four K-slices of one stage (descriptor low words advance by 2 = 32 bytes), one predicate set-up.
__device__ __forceinline__ void umma_tf32_x4(unsigned leader, unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc,
                                             unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q, e;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "setp.ne.b32 e, %5, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "add.u64 a1, %1, 2;\n\tadd.u64 a2, %1, 4;\n\tadd.u64 a3, %1, 6;\n\t"
      "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], a1, b1, %3, q;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], a2, b2, %3, q;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], a3, b3, %3, q;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
// Same with a caller-given advance of the A descriptor per K-slice (in 16-byte units) and only the first `nks`
// (1..4) slices issued: a chunk that holds fewer than 32 real channels needs no MMA on its zero padding.
__device__ __forceinline__ void umma_tf32_step(unsigned leader, unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc,
                                               unsigned idesc, unsigned accumulate, unsigned long long a_step, unsigned nks) {
  asm volatile(
      "{\n\t.reg .pred p, q, e, r1, r2, r3;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "setp.ne.b32 e, %7, 0;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "setp.gt.and.u32 r1, %6, 1, e;\n\tsetp.gt.and.u32 r2, %6, 2, e;\n\tsetp.gt.and.u32 r3, %6, 3, e;\n\t"
      "add.u64 a1, %1, %5;\n\tadd.u64 a2, a1, %5;\n\tadd.u64 a3, a2, %5;\n\t"
      "add.u64 b1, %2, 2;\n\tadd.u64 b2, %2, 4;\n\tadd.u64 b3, %2, 6;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t"
      "@r1 tcgen05.mma.cta_group::1.kind::tf32 [%0], a1, b1, %3, q;\n\t"
      "@r2 tcgen05.mma.cta_group::1.kind::tf32 [%0], a2, b2, %3, q;\n\t"
      "@r3 tcgen05.mma.cta_group::1.kind::tf32 [%0], a3, b3, %3, q;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "l"(a_step), "r"(nks), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned leader, unsigned long long *bar) {
  asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
               "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)), "r"(leader)
               : "memory");
}
// 1 in one lane of a converged warp, 0 in the others.  The single-thread roles (MMA issue) run their loops with the whole
// warp and predicate only the tcgen05 instructions: inside `if (lane == 0)` the compiler cannot keep the descriptors in
// uniform registers, and an instruction then takes 77 clocks to issue whatever its size instead of the 40-64 of its operands.
__device__ __forceinline__ unsigned elect_one() {
  unsigned r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
// ---- thread-block cluster helpers (K-split variant of the halo kernel) ----
__device__ __forceinline__ unsigned cluster_ctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the address, in the cluster's shared window, of this CTA's shared-memory location `addr` inside CTA `rank`
__device__ __forceinline__ unsigned mapa_shared(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f4(unsigned cluster_addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(unsigned cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Every thread of every CTA of the cluster (whole warps: .aligned).  An execution barrier only: what it orders here is
// "barriers initialised (and made visible by fence.mbarrier_init) before any remote arrival" and "no CTA exits before
// the others are done with its shared memory" -- data is handed over through part_full, with its own release / acquire.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// mbar_wait whose acquire covers writes made by other CTAs of the cluster before their (release.cluster) arrivals
__device__ __forceinline__ bool mbar_wait_cluster(unsigned long long *bar, unsigned parity, volatile int *abort_flag, unsigned limit) {
  const unsigned addr = smem_u32(bar);
  for (unsigned it = 0; it < limit; ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ float4 f4add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// ReLU and "none" are inlined; sigmoid and tanh go through one shared out-of-line copy (ACT = MIE_ACT_SIGMOID stands
// for both): inlining 32 copies of expf / tanhf cost 180 registers and with them the third resident block.
__device__ __noinline__ float tc_act_call(int op, float x) { return act_apply(op, x); }
template <int ACT>
__device__ __forceinline__ float tc_act(int op, float x) {
  if (ACT == MIE_ACT_RELU) return fmaxf(x, 0.0f);
  if (ACT == MIE_ACT_NONE) return x;
  return tc_act_call(op, x);
}

struct TcMaps {
  CUtensorMap in[4];  // stride 1: [0] only; stride 2: [row parity * 2 + column parity]
  CUtensorMap w;
};

// Zeroes the stale tiles of the output field.  Run by the epilogue warps (`tid` = index within them, `nthreads` = how
// many they are) before their first accumulator arrives: the producer and the MMA issuer do not wait for it.
__device__ __forceinline__ void tc_zero_tile(const TcParams &p, int t, int THo, int TWo, int tid, int nthreads) {
  const int tx = t % TWo, ty = (t / TWo) % THo, n = t / (TWo * THo);
  for (int i = tid; i < 64 * p.cout; i += nthreads) {
    const int px = i / p.cout, c = i - px * p.cout;
    const int oy = ty * 8 + (px >> 3), ox = tx * 8 + (px & 7);
    if (oy < p.hout && ox < p.wout) p.out[((int64_t)(n * p.hout + oy) * p.wout + ox) * p.out_ps + c] = 0.0f;
  }
}
__device__ __forceinline__ void tc_zero_stale(const TcParams &p, int ntiles_total, int THo, int TWo, int tid, int nthreads) {
  const int n_stale = p.stale ? min(p.counts[1], p.max_tiles) : 0;
  for (int s = blockIdx.x; s < n_stale; s += gridDim.x) {
    const int t = p.stale[s];
    if (t < 0 || t >= ntiles_total) { if (tid == 0) atomicOr(&p.counts[3], MIE_ERR_BAD_TILE); continue; }
    tc_zero_tile(p, t, THo, TWo, tid, nthreads);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// "Own tiles" mode (mie_conv_args.own_tiles): the convolution needs no tile list from a launch before it.  The output
// tiles are dealt to the thread blocks in static pairs (2P, 2P+1), pair P to group P mod G, a group being the n_cblk
// blocks (or clusters) that finish the column blocks of the same pixels.  After the grid dependency wait every block
// tests the tiles of its group against the input words (dilate_flag: one round trip to L2, all loads in flight at once),
// compacts the active ones in ascending order into shared memory and pairs them up as work items; all blocks of a group
// arrive at the same list.  At full activity this spreads the work exactly as the global list does; at partial activity a
// block's share is what is active among its own tiles.  Stale tiles are zeroed by the one block of the group that also
// reads the previous word (column block 0, cluster rank 0).
// Tile words: a tile that a single block finishes is cleared by that block before its epilogue ORs the sent pixels in, as
// after a separate dilation.  A tile that several blocks finish cannot be cleared by one of them without racing the
// others' ORs; there the epilogue warps OR into a scratch word and draw a ticket, and the warp that draws the last ticket
// stores the finished word and leaves both scratch entries zero.
// ---------------------------------------------------------------------------------------------------------------
constexpr int OWN_MAX = 256;   // tiles one group can own; the host sends larger shares to the separate dilation launch

struct OwnShared {
  int list[OWN_MAX];           // active tiles from the front (ascending), stale tiles from the back
  int n_active, n_stale;
  uint8_t flags[OWN_MAX];
};
template <bool OWN> struct OwnSharedT : OwnShared {};
template <> struct OwnSharedT<false> { int list[1]; int n_active, n_stale; };

// Every thread of the block.  (Inlined: as a function of its own, called by all kernels, it made an E2Depth step 3 % slower.)
__device__ __forceinline__ void own_scan(const uint64_t *in_bits, int Hin, int Win, int Hout, int Wout, int k, int stride, int pad,
                                             const uint64_t *union_bits, uint64_t *out_bits /* null unless this block reads and
                                             clears the previous words */, OwnShared &sh, int g, int G, int ntiles_total, bool single) {
  const int SP = (ntiles_total + 1) >> 1;
  const int n_own = g < SP ? 2 * ((SP - g + G - 1) / G) : 0;
  for (int idx = threadIdx.x; idx < n_own; idx += blockDim.x) {
    const int t = 2 * (g + (idx >> 1) * G) + (idx & 1);
    sh.flags[idx] = t < ntiles_total ? dilate_flag(t, in_bits, Hin, Win, Hout, Wout, k, stride, pad, union_bits, out_bits, single)
                                     : (uint8_t)0;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int na = 0, ns = 0;
    const unsigned below = (1u << threadIdx.x) - 1u;
    for (int base = 0; base < n_own; base += 32) {
      const int idx = base + (int)threadIdx.x;
      const int f = idx < n_own ? sh.flags[idx] : 0;
      const unsigned ba = __ballot_sync(0xffffffffu, f == 1), bs = __ballot_sync(0xffffffffu, f == 2);
      const int t = 2 * (g + (idx >> 1) * G) + (idx & 1);
      if (f == 1) sh.list[na + __popc(ba & below)] = t;
      if (f == 2) sh.list[OWN_MAX - 1 - (ns + __popc(bs & below))] = t;
      na += __popc(ba);
      ns += __popc(bs);
    }
    if (threadIdx.x == 0) { sh.n_active = na; sh.n_stale = ns; }
  }
  __syncthreads();
}

__device__ __forceinline__ void tc_zero_stale_own(const TcParams &p, const OwnShared &sh, int THo, int TWo, int tid, int nthreads) {
  for (int s = 0; s < sh.n_stale; ++s) tc_zero_tile(p, sh.list[OWN_MAX - 1 - s], THo, TWo, tid, nthreads);
}

// One lane per (epilogue warp, tile): `v` = this warp's sent pixels, already shifted into 32-bit half `half32` of the
// tile word; `total` = warps that contribute to a tile over all blocks.
__device__ __forceinline__ void own_contribute(const TcParams &p, int t, int half32, unsigned v, int total) {
  if (v) atomicOr(reinterpret_cast<unsigned *>(p.own_words + t) + half32, v);
  __threadfence();
  if (atomicAdd(p.own_tickets + t, 1) == total - 1) {
    __threadfence();
    reinterpret_cast<unsigned long long *>(p.out_bits32)[t] = atomicExch(p.own_words + t, 0ull);
    p.own_tickets[t] = 0;
  }
}


}  // namespace
}  // namespace mie
