// Prefill attention for sm_100a: TMA-staged tiles, tcgen05 MMA with accumulators in tensor
// memory, online softmax in registers. Two kernels share the tile shapes, the shared-memory
// and tensor-memory layouts and the host code of this file:
//
//   prefill_kernel<D, MODE> (this file): the running-max modes - plain scores, generic score
//       mods, softcap with a large cap. One CTA per pair of query tiles, or two of one tile per SM.
//   prefill_bounded_kernel<D> (lf_prefill_bounded.cuh): softcap whose output range needs no
//       running max (the benchmark configurations). Persistent, one CTA per SM, or two of one tile slot.
//
// prefill_kernel: one CTA owns two consecutive 128-row query tiles of one (batch, q head) and
// walks the 64-key KV tiles that the skip range leaves (fully masked tiles are never loaded or
// multiplied). 384 threads (the narrow form, for one tile, has half of each role: see PrefillShape):
//   warps 0-3   softmax for query tile 0 (one thread per score row)
//   warps 4-7   softmax for query tile 1
//   warp  8     TMA producer: Q tiles once, then pairs of K/V tiles into a ring, in the order
//               the MMA warps consume them: {K(lo), K(lo+1)}, {V(lo), K(lo+2)}, {V(lo+1), ...
//   warp  9/10  MMA issuers (one thread each, one per query tile): S_t[buf] = Q_t K^T,
//               O_t += P_t V
//   warp  11    second producer of paged operands (idle otherwise)
//
// Tensor memory (512 columns x 128 lanes of 32 bit):
//   tile t, buffer b: S at column t*128 + b*64 (64 fp32 columns); P (bf16, two per column)
//   overwrites the first 32 columns of its S buffer.   O_t at column 256 + t*128 (D columns).
//
// S is double-buffered per query tile: QK^T of KV tile j+2 is issued right after PV of tile j,
// so the tensor pipe computes the next scores while the softmax warps work on the current
// ones; the only dependency left between the two sides is "PV(j) needs P(j)". The softmax warps
// rescale O_t in place when the running max moves by more than 2^8 (rare); "S(k+1) is ready"
// tells them that PV(k-1) is complete.
//
// Shared-memory tiles use the 128-byte swizzle that TMA writes and the MMA descriptors read:
// a [rows][D] bf16 tile is stored as D/64 blocks of [rows][64] (128-byte rows).
// No cluster launch and no multicast: every CTA fetches its own tiles; L2 provides the reuse
// between the CTAs of one kv head.
#include "lf_common.cuh"
#include "lf_skip_range.h"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <float.h>
#include <math.h>

#include <atomic>
#include <mutex>
#include <type_traits>

namespace lf {

constexpr int kTileQ = LF_PREFILL_TILE_Q;
constexpr int kTileK = LF_PREFILL_TILE_K;
static_assert(kTileQ == 128 && kTileK == 64, "the kernel is written for 128 x 64 tiles");
constexpr int kPrefillThreads = 12 * 32;  // 8 softmax, 1 producer, 2 MMA-issuer, 1 gather warp
constexpr int kMaxStages = 16;
constexpr uint32_t kStageBytesTotal = 8 * 2048;
// K/V ring depth in stages of two 64-key tiles: 4 x 32 KB at D=128, 8 x 16 KB at D=64 (which
// also keeps the CTA above half of the shared memory, so that two CTAs never compete for the 512
// tensor-memory columns). The narrow forms take 256 columns and less than half of the shared memory, but more
// than a third: two of them fit an SM, a third does not, nor one of them beside a CTA of the other forms.
template <int D>
struct StagesFor {
  static constexpr int value = D == 64 ? 8 : 4;
};
constexpr float kLog2eF = 1.4426950408889634f;
constexpr float kRescaleThreshold = 8.0f;  // log2 domain
// Largest row sum of a block that the fast pass accepts: 64 keys at the lazy rescale's 2^8, so that O
// stays as far inside fp32 as with it (at 2^40, values of 1e27 could overflow to infinity).
constexpr float kFastRowSum = 16384.f;  // 2^14
// tanh(x) by odd polynomial: x*(1 - x^2/3) up to |x| <= 0.125 (abs. error < 4.1e-6), degree 7
// up to |x| <= 0.4 (abs. error < 6e-6); MUFU tanh beyond.
constexpr float kTanhPoly1Limit = 0.125f;
constexpr float kTanhPoly3Limit = 0.4f;

constexpr int kModeNone = 0;     // logit2 = raw * c2
constexpr int kModeSoftcap = 1;  // logit2 = tanh(raw * a) * c2
constexpr int kModeGeneric = 2;  // logit2 = mods(raw * a) * c2
// Softcap whose output range is small enough (|c2| <= kBoundedMaxC2) that exp2(logit2) can be
// taken against the fixed reference 0 instead of a running row max: every P lies in
// [2^-80, 2^80], row sums and O stay far inside the fp32 range, and bf16 keeps the same relative
// precision at any magnitude. Without a running max the blocks of a row are independent, there
// is no O rescale, and a row can be split between two threads with no exchange but the final
// row sum.
constexpr int kModeBounded = 3;
constexpr float kBoundedMaxC2 = 80.f;
// logit2 = (raw * a + bias) * c2: the usual biased attention, a scale and an additive score bias with
// nothing behind it. (Any other chain around a bias is generic.)
constexpr int kModeBias = 4;

// Division by a divisor fixed at launch time: q = (mulhi(n, mul) + n) >> shift (Granlund &
// Montgomery's round-up method; exact for every 0 <= n < 2^31). The item decode of the
// persistent kernels runs on one warp that gets few issue slots; real divisions (a few dozen
// dependent instructions each) made it take thousands of clocks.
struct FastDiv {
  uint32_t mul, shift, d;
  static FastDiv make(int32_t divisor) {
    FastDiv f;
    f.d = static_cast<uint32_t>(divisor);
    f.shift = 0;
    while ((1u << f.shift) < f.d) ++f.shift;
    f.mul = static_cast<uint32_t>(((static_cast<uint64_t>(1) << 32) *
                                   ((static_cast<uint64_t>(1) << f.shift) - f.d)) / f.d + 1);
    return f;
  }
  __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const {
#ifdef __CUDA_ARCH__
    const uint32_t hi = __umulhi(n, mul);
#else
    const uint32_t hi = static_cast<uint32_t>((static_cast<uint64_t>(n) * mul) >> 32);
#endif
    return static_cast<uint32_t>((static_cast<uint64_t>(hi) + n) >> shift);
  }
};

struct PrefillParams {
  __nv_bfloat16* out;
  int64_t o_stride[3];
  int32_t Sq, Skv, Hq, group;
  int32_t mask_kind, window, causal_offset;
  int32_t n_qtiles;  // ceil(Sq / 128)
  float a;           // multiplies the raw dot product before the score function
  float c2;          // multiplies the score-function output; includes log2(e); > 0
  float qc[4];       // bounded mode: tanh polynomial in raw^2, scaled to give logit2 / raw
  float ylim[2];     // bounded mode: validity limits of the two polynomials, on raw^2
  ModChain mods;
  const __nv_bfloat16* bias;  // additive score bias [B, Hq, Sq, Skv] (bias and generic modes) or null
  int64_t bias_stride[3];
  int32_t bias_pos;           // the bias is added after this many ops of `mods`
  int32_t bias_sectors;       // bias rows are 32-byte aligned
  // Bias mode: bf16 [B, Hq, Sq, D] tensors added to Q and to the output, or null.
  const __nv_bfloat16* q_bias;
  const __nv_bfloat16* out_bias;
  int64_t qb_stride[3], ob_stride[3];
  int32_t* status;
  int32_t* dbg_ranges;
  // Persistent (bounded-mode) kernel only: the work queue.
  int32_t single;        // running-max kernel: one query tile per CTA instead of a pair
  int32_t n_pairs;       // query-tile pairs per head
  int32_t n_deferred;    // persistent kernels: lightest pairs of a head kept for the queue's end
  int32_t main_items;    // (n_pairs - n_deferred) * Hq * B: items ahead of the deferred ones
  // Divisors of the item decode. (prefill_kernel: div_main heads of a group, div_deferred tiles.)
  FastDiv div_main, div_deferred, div_hq, div_group;
  int32_t n_heads;       // Hq * B (prefill_kernel)
  int32_t n_items;       // n_pairs * Hq * B
  unsigned int* ticket;  // device counter, zero at launch
  int32_t sm_margin;     // SMs left without a CTA
  // Paged K and / or V (prefill_kernel only): pools [n_pages, page_size, Hkv, D] read through a
  // block table; bit 0 of `paged`: K, bit 1: V.
  int32_t paged;
  const __nv_bfloat16* k_pool;
  const __nv_bfloat16* v_pool;
  const int32_t* k_table;
  const int32_t* v_table;
  int64_t kp_stride[3], vp_stride[3];  // (page, slot, kv head)
  int64_t bt_stride;
  int32_t page_size, page_shift, n_pages;
  int32_t gather;  // paged operands come by TMA row gather: tmap_k / tmap_v are 2-D maps of the pools
  int32_t pe_steps;  // PE variant: 16-column steps of the second score product (D_pe / 16, rounded up)
};

// Barrier block at the start of shared memory.
struct __align__(8) PrefillBarriers {
  uint64_t q_full[2];
  uint64_t q_ready[2];     // query bias: it has been added to Q (one arrival per warp)
  uint64_t kv_full[kMaxStages];
  uint64_t kv_empty[kMaxStages];
  uint64_t s_full[2][2];   // [tile][buffer]  MMA -> softmax
  uint64_t p_full[2][2];   // [tile][buffer]  softmax -> MMA
  uint64_t pv_done[2];     // [tile] second-to-last PV done (running-max modes)
  uint64_t o_final[2];     // [tile] last PV done
  uint32_t tmem_base;
  uint32_t pad;
};

__device__ __forceinline__ void report_timeout(int32_t* status, int where) {
  if (status) atomicCAS(status, LF_DEV_OK, LF_DEV_TIMEOUT | (where << 8));
}

// An SM's 512 columns, by shared memory: never three narrow CTAs, nor one (of 96256 bytes at least) beside another form's.
constexpr bool keeps_tensor_memory(size_t smem, bool narrow) {
  return narrow ? smem >= 96256 && 3 * (smem + 1024) > 233472 : smem + 1024 + 96256 + 1024 > 233472;
}

// `PE`: scores are the sum of two products, Q K^T + Q_pe K_pe^T (the two-matmul form of the
// reference's MLA test, tests/test_attention.py:126-151: a "nope" part of width D and a rotary
// part of width D_pe <= 64). The second pair of operands rides along as one more 64-column
// swizzle block behind the D/64 blocks of every Q and K tile - TMA zero-fills the columns past
// D_pe - and the QK^T loop issues its k-steps after the others into the same accumulator. K tiles
// are then larger than V tiles; a ring slot has the size of a K tile.
template <int D, bool PE>
struct PrefillStages {
  static constexpr int value = PE ? (D == 64 ? 4 : 2) : StagesFor<D>::value;
};

// `NARROW`: one query tile per CTA and one slot, with half of an SM's registers, shared and tensor
// memory, so that two CTAs share an SM and the start and end of one lie under the blocks of the other.
template <int D, bool PE, bool NARROW>
struct PrefillShape {
  static constexpr int kSlots = NARROW ? 1 : 2;
  static constexpr int kThreads = NARROW ? 8 * 32 : kPrefillThreads;
  static constexpr int kStages = NARROW ? (D == 64 ? 4 : 2) : PrefillStages<D, PE>::value;
  // Output staging of the softmax warps (2 KB each), and row numbers of the gather warps behind it.
  static constexpr uint32_t kStaging = NARROW ? 4 * 2048 + 4096 : kStageBytesTotal;
  static constexpr uint32_t kTmemColumns = NARROW ? 256 : 512;
  static constexpr size_t kSmem = 1024 /*align slack*/ + 1024 /*barriers*/ + kStaging +
                                  static_cast<size_t>(kSlots) * kTileQ * (D + (PE ? 64 : 0)) * 2 +
                                  static_cast<size_t>(kStages) * 2 * kTileK * (D + (PE ? 64 : 0)) * 2;
};

template <int D, int MODE, bool PE, bool NARROW>
__global__ void __launch_bounds__(PrefillShape<D, PE, NARROW>::kThreads, NARROW ? 2 : 1)
    prefill_kernel(const __grid_constant__ CUtensorMap tmap_q,
                   const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v,
                   const __grid_constant__ CUtensorMap tmap_qpe,
                   const __grid_constant__ CUtensorMap tmap_kpe, const PrefillParams p) {
  using Shape = PrefillShape<D, PE, NARROW>;
  constexpr int kStages = Shape::kStages;
  constexpr int kBlocksD = D / 64;                    // 64-column swizzle blocks per tile row
  constexpr int kBlocksQK = kBlocksD + (PE ? 1 : 0);  // ... of a Q or K tile
  constexpr uint32_t kQBlockBytes = kTileQ * 128;     // one [128][64] bf16 block of Q
  constexpr uint32_t kQTileBytes = kQBlockBytes * kBlocksQK;
  constexpr uint32_t kKVBlockBytes = kTileK * 128;    // one [64][64] bf16 block of K or V
  constexpr uint32_t kVTileBytes = kKVBlockBytes * kBlocksD;
  constexpr uint32_t kKTileBytes = kKVBlockBytes * kBlocksQK;
  constexpr uint32_t kKVTileBytes = kKTileBytes;      // size of a ring slot (two per stage)
  constexpr uint32_t kIdescQK = make_idesc_bf16(128, kTileK, 0);
  constexpr uint32_t kIdescPV = make_idesc_bf16(128, D, 1);
  constexpr uint32_t kColO = Shape::kSlots * 128;
  constexpr int kSoftmaxWarps = Shape::kSlots * 4;
  constexpr int kProducerWarp = kSoftmaxWarps;
  constexpr int kMmaWarp0 = kSoftmaxWarps + 1;
  constexpr int kGatherWarp = kSoftmaxWarps + 3;

  pdl_trigger();
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
  PrefillBarriers* bars = reinterpret_cast<PrefillBarriers*>(smem);
  unsigned char* sStage = smem + 1024;  // 2 KB per softmax warp: output staging
  unsigned char* sQ = sStage + Shape::kStaging;
  unsigned char* sKV = sQ + Shape::kSlots * kQTileBytes;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // Heaviest query tiles first (causal work grows with the row index), over all the heads of a group
  // of heads, then the next group (see the launch).
  int pair, h, b;
  {
    const int r = static_cast<int>(p.div_main.div(blockIdx.x));
    const int chunk = static_cast<int>(p.div_deferred.div(r));
    const int hb = chunk * static_cast<int>(p.div_main.d) +
                   (static_cast<int>(blockIdx.x) - r * static_cast<int>(p.div_main.d));
    pair = (chunk + 1) * static_cast<int>(p.div_deferred.d) - 1 - r;
    if (hb >= p.n_heads) return;
    b = static_cast<int>(p.div_hq.div(hb));
    h = hb - b * p.Hq;
  }
  const int hkv = static_cast<int>(p.div_group.div(h));
  // (`single`: one query tile per CTA. Its key blocks alternate between the two slots, which have a
  // softmax warp group, S buffers and an O each and are merged at the end; chosen by the host.)
  const bool split = !NARROW && p.single;
  const int iq0 = NARROW || split ? pair : pair * 2;

  // (Scalars and selects: an array indexed with the warp's slot lies in local memory, and with nearly all of
  // the SM's memory taken as shared memory such a read goes to L2.)
  int lo0, hi0, lo1, hi1;
  skip_range(p.mask_kind, p.window, p.causal_offset, p.Sq, p.Skv, kTileQ, kTileK, iq0, &lo0, &hi0);
  skip_range(p.mask_kind, p.window, p.causal_offset, p.Sq, p.Skv, kTileQ, kTileK, iq0 + 1, &lo1,
             &hi1);
  const bool valid0 = iq0 * kTileQ < p.Sq, valid1 = !NARROW && !split && (iq0 + 1) * kTileQ < p.Sq;
  const bool work0 = valid0 && hi0 > lo0, work1 = valid1 && hi1 > lo1;
  auto lo_t = [&](int t) { return t ? lo1 : lo0; };
  auto hi_t = [&](int t) { return t ? hi1 : hi0; };
  auto tile_valid = [&](int t) { return t ? valid1 : valid0; };
  auto has_work = [&](int t) { return t ? work1 : work0; };
  int lo = 0, hi = 0;
  if (work0 && work1) {
    lo = min(lo0, lo1);
    hi = max(hi0, hi1);
  } else if (work0) {
    lo = lo0;
    hi = hi0;
  } else if (work1) {
    lo = lo1;
    hi = hi1;
  }

  // ---------------- setup ----------------
  // The producer warp sets the barriers up and requests Q and the first K tiles (of dense operands) before
  // the CTA meets: their latency then lies under the allocation of tensor memory (about 1000 clocks of
  // the 4700 from a CTA's start to its first scores).
  if (warp == kProducerWarp) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
      mbar_init(&bars->q_full[0], 1);
      mbar_init(&bars->q_full[1], 1);
      mbar_init(&bars->q_ready[0], split ? 8 : 4);
      mbar_init(&bars->q_ready[1], 4);
      for (int s = 0; s < kStages; ++s) {
        // (paged operands: one arrival of either gather warp, or one for the TMA part and one for the
        // warp's own copies)
        mbar_init(&bars->kv_full[s], p.paged ? 2 : 1);
        mbar_init(&bars->kv_empty[s], Shape::kSlots);
      }
      for (int t = 0; t < 2; ++t) {
        for (int bf = 0; bf < 2; ++bf) {
          mbar_init(&bars->s_full[t][bf], 1);
          mbar_init(&bars->p_full[t][bf], 4);
        }
        mbar_init(&bars->pv_done[t], 1);
        mbar_init(&bars->o_final[t], 1);
      }
      mbar_fence_init();
    }
    __syncwarp();
    pdl_wait();
    if (elect_one_sync()) {
#pragma unroll 1
      for (int t = 0; t < 2; ++t) {
        if (!has_work(t)) continue;
        mbar_arrive_expect_tx(&bars->q_full[t], kQTileBytes);
#pragma unroll
        for (int kb = 0; kb < kBlocksD; ++kb)
          tma_load_4d(sQ + t * kQTileBytes + kb * kQBlockBytes, &tmap_q, &bars->q_full[t], kb * 64,
                      (iq0 + t) * kTileQ, h, b);
        if constexpr (PE)
          tma_load_4d(sQ + t * kQTileBytes + kBlocksD * kQBlockBytes, &tmap_qpe, &bars->q_full[t], 0,
                      (iq0 + t) * kTileQ, h, b);
      }
      if (!p.paged && hi > lo) {
        const int n_k = lo + 1 < hi ? 2 : 1;
        mbar_arrive_expect_tx(&bars->kv_full[0], n_k * kKTileBytes);
#pragma unroll 1
        for (int i = 0; i < n_k; ++i) {
#pragma unroll
          for (int kb = 0; kb < kBlocksD; ++kb)
            tma_load_4d(sKV + i * kKVTileBytes + kb * kKVBlockBytes, &tmap_k, &bars->kv_full[0], kb * 64,
                        (lo + i) * kTileK, hkv, b);
          if constexpr (PE)
            tma_load_4d(sKV + i * kKVTileBytes + kBlocksD * kKVBlockBytes, &tmap_kpe, &bars->kv_full[0],
                        0, (lo + i) * kTileK, hkv, b);
        }
      }
    }
    __syncwarp();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_base, Shape::kTmemColumns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();  // (so far only the producer warp, which waited itself, has touched global memory)

  // Two CTAs of 256 threads have 128 registers per thread: 184 for the softmax warps, 72 for the others; 4 x 184 +
  // 4 x 72 = 8 x 128. setmaxnreg has to be one instruction for all warps of a warpgroup, so this one stands in front
  // of the dispatch of roles, on a condition that is the same in all four; the other is the first of the softmax
  // branch, which is that warpgroup's alone. (With both in front the compiler gives every warp 72: up to 1 KB spilled.)
  if constexpr (NARROW) {
    if (warp >= kSoftmaxWarps) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  }

  if ((warp == kProducerWarp || warp == kGatherWarp) && p.gather) {
    // ---------------- producer with a paged K and / or V, by TMA row gather ----------------
    // The two-level load of the reference (loopfuse/codegen.py:738-872: read tile_K table entries,
    // then gather the rows) as tile::gather4 loads of four rows x 64 columns, straight into the
    // 128-byte-swizzled tile; the pool is seen as a 2-D tensor of token rows, and tokens past Skv ask
    // for a row past its end (zeros). Two warps share the gathers of every tile: eight each, issued by
    // the elected lane. (Issued by the lanes that hold the row numbers, one diverged lane after the
    // other, a gather took ~200 clocks.) Next to the softmax warps these two get few issue slots, so
    // the look-up is done for eight tiles at a time: a token per lane and tile, its table entry
    // requested a window ahead, its checked row number left in shared memory. (Tile by tile the
    // look-up took 1500 clocks of a stage, as much as the gathers and more than the softmax.)
    // Nothing waits for the rows here, so the whole ring is in flight; the cp.async form below has
    // two stages in flight and a look-up in front of each.
    const bool elected = elect_one_sync();
    const int part = warp == kProducerWarp ? 0 : 1;
    const int n_rows = p.n_pages * p.page_size;
    constexpr int kWindow = 8;  // tiles
    // [K or V][tile of the window][32 tokens] of this warp, in the output staging of warps 4..7: their
    // tile is the last to finish, after the last gather. (`NARROW`: behind the staging.)
    int* const row_ids = reinterpret_cast<int*>(sStage + 4 * 2048) + part * (2 * kWindow * 32);
    static_assert(2 * 2 * kWindow * 32 * 4 <= 4 * 2048, "row numbers in the staging of four warps");
    auto page_of = [&](int t) { return p.page_shift >= 0 ? (t >> p.page_shift) : (t / p.page_size); };
    auto is_paged = [&](bool is_v) { return ((p.paged >> (is_v ? 1 : 0)) & 1) != 0; };
    const int t_end = min(p.Skv, hi * kTileK);
    // Token of this lane in tile j (each warp has half of the 64).
    auto token = [&](int j) { return j * kTileK + part * 32 + lane; };
    int entry_k[kWindow], entry_v[kWindow];  // table entries of the next window, not looked at
    auto request = [&](bool is_v, int w, int (&entry)[kWindow]) {
      const int32_t* table = (is_v ? p.v_table : p.k_table) + static_cast<int64_t>(b) * p.bt_stride;
#pragma unroll
      for (int e = 0; e < kWindow; ++e) {
        const int t = token(lo + w * kWindow + e);
        entry[e] = t < t_end ? table[page_of(t)] : 0;
      }
    };
    // Row numbers of window w from its entries, then the next window's request.
    auto look_up = [&](bool is_v, int w, int (&entry)[kWindow]) {
      __syncwarp();  // (the elected lane has read the last window's)
#pragma unroll
      for (int e = 0; e < kWindow; ++e) {
        const int t = token(lo + w * kWindow + e);
        int pg = entry[e];
        if (pg < 0 || pg >= p.n_pages) {
          if (p.status) atomicExch(p.status, LF_DEV_BAD_PAGE);
          pg = 0;
        }
        const int row = pg * p.page_size + (t - page_of(t) * p.page_size);
        row_ids[(is_v ? kWindow * 32 : 0) + e * 32 + lane] = t < t_end ? row : n_rows;
      }
      __syncwarp();
      request(is_v, w + 1, entry);
    };
    int n = 0;
    bool ok = true;
    // A stage is tile ja of K (or V, `first_is_v`) and tile jb of K (< 0: none).
    auto load_pair = [&](bool first_is_v, int ja, int jb) {
      if (!ok) return;
      if (first_is_v && is_paged(true) && (ja - lo) % kWindow == 0)
        look_up(true, (ja - lo) / kWindow, entry_v);
      if (!first_is_v && is_paged(false)) look_up(false, 0, entry_k);
      if (first_is_v && is_paged(false) && jb >= 0 && (jb - lo) % kWindow == 0)
        look_up(false, (jb - lo) / kWindow, entry_k);
      const int stage = n % kStages;
      const uint32_t parity = ((n / kStages) & 1) ^ 1;
      ++n;
      if (!mbar_wait(&bars->kv_empty[stage], parity)) {
        report_timeout(p.status, 1);
        ok = false;
        return;
      }
      if (elected) {
        auto bytes_of = [&](bool is_v) -> uint32_t {
          return is_paged(is_v) ? kKVTileBytes / 2 : part == 0 ? kKVTileBytes : 0u;
        };
        const uint32_t tx = bytes_of(first_is_v) + (jb >= 0 ? bytes_of(false) : 0u);
        if (tx) mbar_arrive_expect_tx(&bars->kv_full[stage], tx);
        else mbar_arrive(&bars->kv_full[stage]);
        auto load = [&](bool is_v, int j, unsigned char* dst) {
          const CUtensorMap* tma = is_v ? &tmap_v : &tmap_k;
          if (is_paged(is_v)) {
            const int4* ids = reinterpret_cast<const int4*>(
                row_ids + (is_v ? kWindow * 32 : 0) + ((j - lo) % kWindow) * 32);
            const int x = hkv * static_cast<int>(is_v ? p.vp_stride[2] : p.kp_stride[2]);
            const uint32_t d = smem_u32(dst);
#pragma unroll 8
            for (int i = 0; i < 8; ++i) {
              const int4 r = ids[i];
#pragma unroll
              for (int kb = 0; kb < kBlocksD; ++kb)
                tma_gather4(d + kb * kKVBlockBytes + (part * 8 + i) * 512, tma, &bars->kv_full[stage],
                            x + kb * 64, r.x, r.y, r.z, r.w);
            }
          } else if (part == 0) {
#pragma unroll
            for (int kb = 0; kb < kBlocksD; ++kb)
              tma_load_4d(dst + kb * kKVBlockBytes, tma, &bars->kv_full[stage], kb * 64, j * kTileK,
                          hkv, b);
          }
        };
        unsigned char* dst = sKV + stage * (2 * kKVTileBytes);
        load(first_is_v, ja, dst);
        if (jb >= 0) load(false, jb, dst + kKVTileBytes);
      }
    };
    if (hi > lo) {
      auto second = [&](int j) { return j < hi ? j : -1; };
      if (is_paged(false)) request(false, 0, entry_k);
      if (is_paged(true)) request(true, 0, entry_v);
      load_pair(false, lo, second(lo + 1));
      for (int j = lo; j < hi; ++j) load_pair(true, j, second(j + 2));
    }
  } else if (warp == kProducerWarp && p.paged) {
    // ---------------- producer with a paged K and / or V ----------------
    // The two-level load of the reference (loopfuse/codegen.py:738-872: read tile_K table
    // entries, then gather the rows) fused into the tile load: a dense operand still arrives by
    // TMA; a paged one is copied by the whole warp, row by row, with 16-byte cp.async straight
    // from the pool into the 128-byte-swizzled tile layout the MMA descriptors read (16-byte
    // piece c of row r of a 64-column block sits at piece c ^ (r & 7)). Rows past Skv are
    // zero-filled, like TMA does. Copies of up to kLag stages are in flight; a stage is
    // published (second arrival on its full barrier) when its copies have landed and a proxy
    // fence has made them visible to the tensor pipe.
    constexpr int kLag = 2;
    constexpr int kChunks = D / 8;            // 16-byte pieces per row
    constexpr int kRowsPerPass = 32 / kChunks;  // rows one pass of the warp covers
    const bool elected = elect_one_sync();
    int n = 0;
    int published = 0;  // stages whose copies have been published
    bool ok = true;
    auto page_of = [&](int t) { return p.page_shift >= 0 ? (t >> p.page_shift) : (t / p.page_size); };
    // Copy the 64 rows of KV tile j of a paged operand into `dst`.
    auto copy_tile = [&](bool is_v, int j, unsigned char* dst) {
      const __nv_bfloat16* pool = is_v ? p.v_pool : p.k_pool;
      const int32_t* table = (is_v ? p.v_table : p.k_table) + static_cast<int64_t>(b) * p.bt_stride;
      const int64_t* st = is_v ? p.vp_stride : p.kp_stride;
      // Lane l looks up the pages of rows l and l + 32; the others get them by shuffle.
      int64_t row_off[2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = j * kTileK + half * 32 + lane;
        row_off[half] = -1;
        if (t < p.Skv) {
          const int pg_idx = page_of(t);
          int32_t pg = table[pg_idx];
          if (pg < 0 || pg >= p.n_pages) {
            if (p.status) atomicExch(p.status, LF_DEV_BAD_PAGE);
            pg = 0;
          }
          row_off[half] = pg * st[0] + (t - pg_idx * p.page_size) * st[1] + hkv * st[2];
        }
      }
      const int c = lane % kChunks;
      const uint32_t dst_u32 = smem_u32(dst) + (c / 8) * kKVBlockBytes;
#pragma unroll
      for (int pass = 0; pass < kTileK / kRowsPerPass; ++pass) {
        const int r = pass * kRowsPerPass + lane / kChunks;
        const int64_t off_lo = __shfl_sync(0xffffffffu, row_off[0], r & 31);
        const int64_t off_hi = __shfl_sync(0xffffffffu, row_off[1], r & 31);
        const int64_t off = r < 32 ? off_lo : off_hi;
        const uint32_t d = dst_u32 + r * 128 + (((c & 7) ^ (r & 7)) << 4);
        const __nv_bfloat16* src = pool + (off >= 0 ? off : 0) + c * 8;
        const uint32_t nbytes = off >= 0 ? 16u : 0u;  // 0: the 16 bytes are zero-filled
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
                     "r"(nbytes)
                     : "memory");
      }
    };
    auto publish_up_to = [&](int upto) {  // publish stages [published, upto)
      if (published < upto) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0)
          for (int i = published; i < upto; ++i) mbar_arrive(&bars->kv_full[i % kStages]);
        published = upto;
      }
    };
    // ja: tile of `first_is_v ? V : K`; jb >= 0: a K tile in the second half of the stage.
    auto load_pair = [&](bool first_is_v, int ja, int jb) {
      if (!ok) return;
      const int stage = n % kStages;
      const uint32_t parity = ((n / kStages) & 1) ^ 1;
      if (!mbar_wait(&bars->kv_empty[stage], parity)) {
        report_timeout(p.status, 1);
        ok = false;
        return;
      }
      unsigned char* dst = sKV + stage * (2 * kKVTileBytes);
      const bool a_paged = (p.paged >> (first_is_v ? 1 : 0)) & 1;
      const bool b_paged = jb >= 0 && (p.paged & 1);
      if (elected) {
        const uint32_t tx = (a_paged ? 0u : kKVTileBytes) + ((jb >= 0 && !b_paged) ? kKVTileBytes : 0u);
        if (tx) mbar_arrive_expect_tx(&bars->kv_full[stage], tx);
        else mbar_arrive(&bars->kv_full[stage]);
        if (!a_paged) {
#pragma unroll
          for (int kb = 0; kb < kBlocksD; ++kb)
            tma_load_4d(dst + kb * kKVBlockBytes, first_is_v ? &tmap_v : &tmap_k,
                        &bars->kv_full[stage], kb * 64, ja * kTileK, hkv, b);
        }
        if (jb >= 0 && !b_paged) {
#pragma unroll
          for (int kb = 0; kb < kBlocksD; ++kb)
            tma_load_4d(dst + kKVTileBytes + kb * kKVBlockBytes, &tmap_k, &bars->kv_full[stage],
                        kb * 64, jb * kTileK, hkv, b);
        }
      }
      __syncwarp();
      if (a_paged) copy_tile(first_is_v, ja, dst);
      if (b_paged) copy_tile(false, jb, dst + kKVTileBytes);
      cp_async_commit();  // one group per stage, empty or not
      ++n;
      cp_async_wait<kLag>();  // the copies of every stage but the last kLag have landed
      publish_up_to(n - kLag);
    };
    if (hi > lo) {
      load_pair(false, lo, lo + 1 < hi ? lo + 1 : -1);
      for (int j = lo; j < hi; ++j) load_pair(true, j, j + 2 < hi ? j + 2 : -1);
    }
    cp_async_wait<0>();
    publish_up_to(n);
  } else if (warp == kProducerWarp) {
    // ---------------- TMA producer ----------------
    // The whole warp runs the loop and waits; the elected lane issues the copies (a warp that
    // has diverged into a single-lane branch gets few issue slots next to the softmax warps).
    {
      const bool elected = elect_one_sync();
      int n = 1;  // (stage 0 was requested above)
      bool ok = true;
      // A ring stage holds two 64-key tiles that the MMA warps need at the same time:
      // {K(lo), K(lo+1)} first, then {V(j), K(j+2)} for every j; one full / one empty barrier
      // per stage. `jb < 0` means the second half is not loaded (past the end of the range).
      auto load_pair = [&](int ja, int jb) {
        if (!ok) return;
        const int stage = n % kStages;
        const uint32_t parity = ((n / kStages) & 1) ^ 1;
        ++n;
        if (!mbar_wait(&bars->kv_empty[stage], parity)) {
          report_timeout(p.status, 1);
          ok = false;
          return;
        }
        if (elected) {
          mbar_arrive_expect_tx(&bars->kv_full[stage], kVTileBytes + (jb >= 0 ? kKTileBytes : 0u));
          unsigned char* dst = sKV + stage * (2 * kKVTileBytes);
#pragma unroll
          for (int kb = 0; kb < kBlocksD; ++kb)
            tma_load_4d(dst + kb * kKVBlockBytes, &tmap_v, &bars->kv_full[stage], kb * 64,
                        ja * kTileK, hkv, b);
          if (jb >= 0) {
#pragma unroll
            for (int kb = 0; kb < kBlocksD; ++kb)
              tma_load_4d(dst + kKVTileBytes + kb * kKVBlockBytes, &tmap_k,
                          &bars->kv_full[stage], kb * 64, jb * kTileK, hkv, b);
            if constexpr (PE)
              tma_load_4d(dst + kKVTileBytes + kBlocksD * kKVBlockBytes, &tmap_kpe,
                          &bars->kv_full[stage], 0, jb * kTileK, hkv, b);
          }
        }
        __syncwarp();
      };
      for (int j = lo; j < hi; ++j) load_pair(j, j + 2 < hi ? j + 2 : -1);
    }
  } else if (warp == kMmaWarp0 || (!NARROW && warp == kMmaWarp0 + 1)) {
    // (Two comparisons: as a range the two-slot form came out 0.1 us a launch slower, causal 4 x 8 x 593 D = 64
    // 9.01 -> 9.10 us.)
    // ---------------- MMA issuers: one warp per query tile ----------
    // Two issuing threads halve the per-instruction issue overhead; the tensor pipe serialises
    // the two independent streams. Both walk the same K/V ring and both release every stage
    // (kv_empty counts two arrivals), whether or not their tile used it.
    // The whole warp runs the loop (every lane waits on the barriers); the elected lane alone
    // issues MMAs and commits.
    if (hi > lo) {
      const int t = warp - kMmaWarp0;
      const int tq = split ? 0 : t;  // query tile of this slot
      const bool elected = elect_one_sync();
      bool ok = true;
      const bool own_q = MODE == kModeBias && p.q_bias != nullptr;
      if (has_work(tq) && !mbar_wait(own_q ? &bars->q_ready[tq] : &bars->q_full[tq], 0)) {
        report_timeout(p.status, 2);
        ok = false;
      }
      // Descriptors are built once; per MMA only the start-address field moves (in 16-byte
      // units, no carry out of the 14-bit field since shared memory ends below 256 KB).
      constexpr uint32_t kStageUnits = (2 * kKVTileBytes) >> 4;  // a stage is a pair of tiles
      constexpr uint32_t kHalfUnits = kKVTileBytes >> 4;
      const uint64_t qdesc = make_smem_desc_sw128(smem_u32(sQ) + tq * kQTileBytes, 16, 1024);
      const uint64_t kdesc0 = make_smem_desc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t vdesc0 = make_smem_desc_sw128(smem_u32(sKV), kKVBlockBytes, 1024);
      const uint32_t s_col = tmem_base + t * 128;
      const uint32_t o_col = tmem_base + kColO + t * 128;
      int n = 0;  // ring position, walks the same sequence as the producer

      auto active = [&](int j) {
        return split ? ((j - lo) & 1) == t : has_work(t) && j >= lo_t(t) && j < hi_t(t);
      };
      auto block_of = [&](int j) { return split ? (j - lo) >> 1 : j - lo_t(t); };  // of this slot
      auto wait_stage = [&](int where) -> int {  // next ring stage, waited full; -1 on time-out
        const int stage = n % kStages;
        const uint32_t parity = (n / kStages) & 1;
        ++n;
        if (!mbar_wait(&bars->kv_full[stage], parity)) {
          report_timeout(p.status, where);
          ok = false;
          return -1;
        }
        return stage;
      };
      // `half` selects the first or second tile of the stage.
      auto issue_qk = [&](int stage, int half, int j) {
        const int buf = block_of(j) & 1;
        const uint64_t kd = kdesc0 + static_cast<uint64_t>(stage * kStageUnits + half * kHalfUnits);
        const uint32_t d = s_col + buf * 64;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          mma_ss_if(elected, d,
                    qdesc + static_cast<uint64_t>((ks / 4) * (kQBlockBytes >> 4) + (ks % 4) * 2),
                    kd + static_cast<uint64_t>((ks / 4) * (kKVBlockBytes >> 4) + (ks % 4) * 2),
                    kIdescQK, ks > 0 ? 1u : 0u);
        }
        if constexpr (PE) {  // + Q_pe K_pe^T: the extra block of both tiles, same accumulator
          for (int ks = 0; ks < p.pe_steps; ++ks)
            mma_ss_if(elected, d,
                      qdesc + static_cast<uint64_t>(kBlocksD * (kQBlockBytes >> 4) + ks * 2),
                      kd + static_cast<uint64_t>(kBlocksD * (kKVBlockBytes >> 4) + ks * 2), kIdescQK,
                      1u);
        }
        tc_commit_if(elected, &bars->s_full[t][buf]);
      };
      auto issue_pv = [&](int stage, int kt) {
        const uint64_t vd = vdesc0 + static_cast<uint64_t>(stage * kStageUnits);
        const uint32_t a = s_col + (kt & 1) * 64;
#pragma unroll
        for (int ks = 0; ks < kTileK / 16; ++ks) {
          mma_ts_if(elected, o_col, a + ks * 8, vd + static_cast<uint64_t>(ks * (2048 >> 4)), kIdescPV,
                    (kt > 0 || ks > 0) ? 1u : 0u);
        }
      };

      // Prologue: scores of the first two KV tiles (one stage).
      {
        const int stage = ok ? wait_stage(3) : -1;
        if (stage >= 0) {
          tc_fence_after();
          if (active(lo)) issue_qk(stage, 0, lo);
          if (lo + 1 < hi && active(lo + 1)) issue_qk(stage, 1, lo + 1);
        }
        __syncwarp();  // (as below)
        tc_commit_if(elected && ok, &bars->kv_empty[0]);
      }
      const int nblk_t = split ? (hi - lo + 1 - t) >> 1 : has_work(t) ? hi_t(t) - lo_t(t) : 0;
      for (int j = lo; j < hi; ++j) {
        const int st = wait_stage(4);  // {V(j), K(j+2)}
        tc_fence_after();
        // (Split: K(j+2) is this slot's next block, not the one after it; its scores are made
        // while the softmax of block j runs. Its buffer was read by the slot's last PV.)
        if (split && st >= 0 && j + 2 < hi && active(j)) issue_qk(st, 1, j + 2);
        if (st >= 0 && active(j)) {
          const int kt = block_of(j);
          if (mbar_wait(&bars->p_full[t][kt & 1], (kt >> 1) & 1)) {
            tc_fence_after();
            issue_pv(st, kt);
            // Completion points the softmax warps may wait on: the second-to-last PV (for a
            // rescale in the last block) and the last PV (for the epilogue).
            tc_commit_if(elected && kt == nblk_t - 2, &bars->pv_done[t]);
            tc_commit_if(elected && kt == nblk_t - 1, &bars->o_final[t]);
          } else {
            report_timeout(p.status, 6 + t);
            ok = false;
          }
        }
        // The lanes meet once per step, before anything is issued that lets a barrier that they wait on in
        // this step complete its next phase (a lane left behind would then wait on a parity that has
        // flipped), and they leave together when a wait ran out.
        if (!__all_sync(0xffffffffu, ok)) break;
        if (!split && j + 2 < hi && active(j + 2)) issue_qk(st, 1, j + 2);
        tc_commit_if(elected, &bars->kv_empty[st]);
      }
    }
  } else if (warp < kSoftmaxWarps) {
    if constexpr (NARROW) asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    // ---------------- softmax warps ----------------
    const int t = warp >> 2;                 // slot of this warp group
    const int tq = split ? 0 : t;            // and its query tile
    const int row = (warp & 3) * 32 + lane;  // row inside the tile == tensor-memory lane
    const int grow = (iq0 + tq) * kTileQ + row;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_base = tmem_base + lane_addr + t * 128;
    const uint32_t o_addr = tmem_base + lane_addr + kColO + t * 128;

    if (p.dbg_ranges && tile_valid(t) && row == 0) {
      const int64_t idx = ((static_cast<int64_t>(b) * p.Hq + h) * p.n_qtiles + (iq0 + t)) * 2;
      p.dbg_ranges[idx] = lo_t(t);
      p.dbg_ranges[idx + 1] = hi_t(t);
    }

    if (has_work(tq)) {
      // Visible column interval of this row: [c_lo, c_hi].
      int c_hi = p.Skv - 1;
      int c_lo = 0;
      if (p.mask_kind != LF_MASK_NONE) c_hi = min(c_hi, grow + p.causal_offset);
      if (p.mask_kind == LF_MASK_CAUSAL_WINDOW)
        c_lo = max(0, grow + p.causal_offset - (p.window - 1));

      float m_used = -INFINITY;  // max the stored P and O are scaled by (log2 domain)
      float l_run = 0.f;
      bool ok = true;
      // Block k of this slot is block first + k * step of the tile.
      const int first = lo_t(tq) + (split ? t : 0), step = split ? 2 : 1;
      const int nblk = split ? (hi - lo + 1 - t) >> 1 : hi_t(t) - lo_t(t);
      // Bias mode: this row's 64 bias values of a block (128 contiguous bytes) are requested a block
      // ahead, so that their latency lies under the exp2 pass and the hand-shake; read when the
      // scores were there, they cost a round trip to HBM per block. (Rows past Sq read the last
      // row; both are clipped later. A block that crosses Skv is read value by value on the spot.)
      [[maybe_unused]] uint32_t bq[32];
      [[maybe_unused]] const __nv_bfloat16* brow =
          MODE == kModeBias ? p.bias + b * p.bias_stride[0] + h * p.bias_stride[1] +
                                  static_cast<int64_t>(min(grow, p.Sq - 1)) * p.bias_stride[2]
                            : nullptr;
      auto request_bias = [&](int k) {
        const int col = (first + k * step) * kTileK;
        if (k >= nblk || col + kTileK > p.Skv ||
            !LF_BOUNDS(col >= 0 && b * p.Hq + h < p.n_heads, p.status, 61))
          return;
        if (p.bias_sectors) {
#pragma unroll
          for (int i = 0; i < 4; ++i) ldg_stream_32(brow + col + i * 16, &bq[i * 8]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 v4 = *reinterpret_cast<const uint4*>(brow + col + i * 8);
            bq[4 * i] = v4.x; bq[4 * i + 1] = v4.y; bq[4 * i + 2] = v4.z; bq[4 * i + 3] = v4.w;
          }
        }
      };
      // O_t must hold every PV up to k-1 and none may be in flight. QK(k+1) is issued after PV(k-1), so
      // "S(k+1) is ready" implies it; in the last block there is no S(k+1) and the MMA warp commits
      // pv_done after the second-to-last PV instead.
      auto pvs_before_complete = [&](int k) {
        const bool last = k + 1 == nblk;
        uint64_t* bar = last ? &bars->pv_done[t] : &bars->s_full[t][(k + 1) & 1];
        if (!mbar_wait(bar, last ? 0u : (((k + 1) >> 1) & 1))) {
          report_timeout(p.status, 12 + t);
          return false;
        }
        tc_fence_after();
        return true;
      };
      auto rescale_o = [&](int c, float alpha) {
        uint32_t orr[32];
        tmem_ld_32x32b_x32(o_addr + c * 32, orr);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * alpha);
        tmem_st_32x32b_x32(o_addr + c * 32, orr);
      };
      auto publish_p = [&](int buf) {  // (one arrival per warp: those of all lanes queue up behind each other)
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full[t][buf]);
      };
      if constexpr (MODE == kModeBias) {
        request_bias(0);
        // The query bias: each thread adds its row (or half of it, when the slots share a tile) to the tile
        // in shared memory, one bf16 rounding as in the eager graph. (With passes of their own over Q in
        // front of the kernel and over the output behind it 4 x 8 x 1024, D = 64 takes 29.9 us on the
        // device instead of 28.9, and two more launches and allocations on the host.)
        if (p.q_bias) {
          constexpr int kPieces = D / 8;
          // (Rows past Sq keep their zeros: they vote on the warp's passes too.)
          const bool real = grow < p.Sq &&
                            LF_BOUNDS(grow >= 0 && b * p.Hq + h < p.n_heads, p.status, 62);
          const __nv_bfloat16* qb = p.q_bias + b * p.qb_stride[0] + h * p.qb_stride[1] +
                                    static_cast<int64_t>(grow) * p.qb_stride[2];
          const int first_piece = split ? t * (kPieces / 2) : 0;
          const int n_pieces = split ? kPieces / 2 : kPieces;
          uint4 add[kPieces];
#pragma unroll
          for (int i = 0; i < kPieces; ++i)
            if (real && i < n_pieces) add[i] = ldg_stream_16(qb + (first_piece + i) * 8);
          if (!mbar_wait(&bars->q_full[tq], 0)) {
            report_timeout(p.status, 16 + t);
            ok = false;
          }
#pragma unroll
          for (int i = 0; i < kPieces; ++i)
            if (real && i < n_pieces) {
              const int c = first_piece + i;
              uint4* piece = reinterpret_cast<uint4*>(sQ + tq * kQTileBytes + (c >> 3) * kQBlockBytes +
                                                      row * 128 + (((c & 7) ^ (row & 7)) << 4));
              *piece = add_bf16x8(*piece, add[i]);
            }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->q_ready[tq]);
        }
      }
      for (int k = 0; k < nblk && ok; ++k) {
        const int c0 = (first + k * step) * kTileK;
        const int buf = k & 1;
        const uint32_t s_addr = s_base + buf * 64;
        if (!mbar_wait(&bars->s_full[t][buf], (k >> 1) & 1)) {
          report_timeout(p.status, 8 + t);
          ok = false;
          break;
        }
        tc_fence_after();
        // Raw scores of this row: 64 fp32 values.
        uint32_t sr[2][32];
        tmem_ld_32x32b_x32(s_addr, sr[0]);
        tmem_ld_32x32b_x32(s_addr + 32, sr[1]);
        tmem_wait_ld();

        const int rel_lo = c_lo - c0;  // visible columns of this row inside the tile:
        const int rel_hi = c_hi - c0;  // [rel_lo, rel_hi]
        const bool masked = rel_lo > 0 || rel_hi < kTileK - 1;

        if constexpr (MODE == kModeBias) {
          if (c0 + kTileK > p.Skv) {
            const int whole = (p.Skv - c0) >> 3;  // 8-column groups; the next one crosses Skv
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (c0 + whole * 8 + e < p.Skv)
                w[e >> 1] |= static_cast<uint32_t>(__bfloat16_as_ushort(brow[c0 + whole * 8 + e]))
                             << ((e & 1) * 16);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              uint4 v4 = make_uint4(w[0], w[1], w[2], w[3]);  // (columns past Skv are masked)
              if (i < whole) v4 = *reinterpret_cast<const uint4*>(brow + c0 + i * 8);
              bq[4 * i] = v4.x; bq[4 * i + 1] = v4.y; bq[4 * i + 2] = v4.z; bq[4 * i + 3] = v4.w;
            }
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            uint32_t& s0 = sr[i >> 4][(2 * i) & 31];
            uint32_t& s1 = sr[i >> 4][(2 * i + 1) & 31];
            s0 = __float_as_uint(fmaf(__uint_as_float(s0), p.a, bf16lo_to_f32(bq[i])));
            s1 = __float_as_uint(fmaf(__uint_as_float(s1), p.a, bf16hi_to_f32(bq[i])));
          }
        }
        if constexpr (MODE == kModeGeneric) {
          // The chain is interpreted op by op over the row's 64 scores in registers: one
          // (warp-uniform) dispatch per op and block, not one per score - the reference compiles
          // a kernel per chain (loopfuse/codegen.py:454-998), an interpreter has to keep its
          // dispatch out of the element loop.
          auto each = [&](auto f) {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i)
                sr[c][i] = __float_as_uint(f(__uint_as_float(sr[c][i])));
          };
          auto run_mods = [&](int m_lo, int m_hi) {
#pragma unroll 1
            for (int m = m_lo; m < m_hi; ++m) {
              const float a = p.mods.arg[m];
              switch (p.mods.op[m]) {
                case LF_MOD_MUL: each([&](float x) { return x * a; }); break;
                case LF_MOD_ADD: each([&](float x) { return x + a; }); break;
                case LF_MOD_TANH: each([&](float x) { return tanhf(x); }); break;
                case LF_MOD_EXP: each([&](float x) { return __expf(x); }); break;
                case LF_MOD_EXP2: each([&](float x) { return exp2f(x); }); break;
                case LF_MOD_SIN: each([&](float x) { return sinf(x); }); break;
                case LF_MOD_COS: each([&](float x) { return cosf(x); }); break;
                case LF_MOD_RELU: each([&](float x) { return fmaxf(x, 0.f); }); break;
                case LF_MOD_SQUARE: each([&](float x) { return x * x; }); break;
                case LF_MOD_DIV: each([&](float x) { return x / a; }); break;
                default: break;
              }
            }
          };
          each([&](float x) { return x * p.a; });
          if (p.bias == nullptr) {
            run_mods(0, p.mods.n);
          } else {
            run_mods(0, p.bias_pos);
            // This row's 64 bias values of the block: 128 contiguous bytes, eight 16-byte loads
            // (rows past Sq read the last row, columns past Skv are not read: both are masked
            // or clipped later).
            const __nv_bfloat16* brow = p.bias + b * p.bias_stride[0] + h * p.bias_stride[1] +
                                        static_cast<int64_t>(min(grow, p.Sq - 1)) * p.bias_stride[2] +
                                        c0;
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i8 = 0; i8 < 4; ++i8) {
                const int cc = c * 32 + i8 * 8;
                uint32_t w[4] = {0u, 0u, 0u, 0u};
                if (c0 + cc + 8 <= p.Skv &&
                    LF_BOUNDS(c0 + cc >= 0 && b * p.Hq + h < p.n_heads,
                              p.status, 60)) {
                  const uint4 v4 = ldg_stream_16(brow + cc);
                  w[0] = v4.x; w[1] = v4.y; w[2] = v4.z; w[3] = v4.w;
                } else {
#pragma unroll
                  for (int e = 0; e < 8; ++e)
                    if (c0 + cc + e < p.Skv)
                      w[e >> 1] |= static_cast<uint32_t>(__bfloat16_as_ushort(brow[cc + e]))
                                   << ((e & 1) * 16);
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  const float bv = __uint_as_float((e & 1) ? (w[e >> 1] & 0xffff0000u)
                                                           : (w[e >> 1] << 16));
                  sr[c][i8 * 8 + e] = __float_as_uint(__uint_as_float(sr[c][i8 * 8 + e]) + bv);
                }
              }
            run_mods(p.bias_pos, p.mods.n);
          }
        }

        // Plain and biased scores, fast pass: where every row of the warp has a reference and sees the whole
        // block, P is taken against that reference without looking for the block's maximum first. P may then
        // exceed 1, which bf16 and fp32 hold as exactly as any other magnitude. The row sum of such a block
        // is taken over the bf16-rounded values that the PV product sees, so that numerator and denominator
        // carry the same rounding; against fp64 that is no worse than fp32 P (1.98e-3 against 2.02e-3,
        // causal 2 x 4 x 512).
        // Own-maximum pass, for the other blocks (a row's first, masked ones, and those whose fast row sum
        // passed kFastRowSum): masks set scores to -inf, the reference moves if the block's maximum asks for
        // it, and the row sum is taken over P in fp32.
        // Each pass exists once, and masks are a pass over the scores: waiting for instructions is the
        // largest stall of short calls (8 warps per issue, causal 2 x 4 x 512, cold). With one pass for both
        // kinds of blocks every block paid three votes instead of two: back to back 1 x 16 x 8192 D=64
        // 223 us against 209, 1 x 32 x 8192 D=128 529 against 518.
        if constexpr (MODE == kModeNone || MODE == kModeBias) {
          uint32_t pk[32];
          bool own_max = __any_sync(0xffffffffu, masked || m_used == -INFINITY);
          if (!own_max) {
            float fs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const float p0 = ex2_approx(fmaf(__uint_as_float(sr[c][i]), p.c2, -m_used));
                const float p1 = ex2_approx(fmaf(__uint_as_float(sr[c][i + 1]), p.c2, -m_used));
                const uint32_t pkv = pack_bf16x2(p0, p1);
                pk[c * 16 + (i >> 1)] = pkv;
                if ((i >> 1) & 1) add_bf16x2_to_f32(fs[2], fs[3], pkv);
                else add_bf16x2_to_f32(fs[0], fs[1], pkv);
              }
            const float sum = (fs[0] + fs[1]) + (fs[2] + fs[3]);
            own_max = __any_sync(0xffffffffu, !(sum <= kFastRowSum));
            if (!own_max) l_run += sum;
          }
          if (own_max) {
            if (__any_sync(0xffffffffu, masked)) {
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                // Bit i: column c * 32 + i is visible (shifts by 32 and more give 0). Comparing each column
                // with both bounds took three instructions per score: causal 2 x 4 x 512 D=64 7.24 ->
                // 6.99 us, 8 x 32 x 512 D=128 42.4 -> 40.8, biased 4 x 8 x 1024 29.3 -> 28.9.
                uint32_t seen, upto;
                asm("shl.b32 %0, 0xffffffff, %1;" : "=r"(seen) : "r"(max(rel_lo - c * 32, 0)));
                asm("shl.b32 %0, 0xfffffffe, %1;" : "=r"(upto) : "r"(max(rel_hi - c * 32, 0)));
                seen = rel_hi < c * 32 ? 0u : seen & ~upto;
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (!(seen & (1u << i))) sr[c][i] = 0xff800000u;  // -inf
              }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                mx[2 * c] = max3(mx[2 * c], __uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1]));
                mx[2 * c + 1] = max3(mx[2 * c + 1], __uint_as_float(sr[c][i + 2]),
                                     __uint_as_float(sr[c][i + 3]));
              }
            const float m_new =
                fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.c2);
            // Lazy rescale: move the reference only when it grew by more than 2^8.
            float alpha = 1.f;
            if (m_new > -INFINITY && (m_used == -INFINITY || m_new - m_used > kRescaleThreshold)) {
              alpha = ex2_approx(m_used - m_new);  // 0 when m_used is -inf
              m_used = m_new;
            }
            if (k > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
              if (!pvs_before_complete(k)) {
                ok = false;
                break;
              }
#pragma unroll 1
              for (int c = 0; c < D / 32; ++c) rescale_o(c, alpha);
            }
            const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
            float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const float p0 = ex2_approx(fmaf(__uint_as_float(sr[c][i]), p.c2, neg_m));
                const float p1 = ex2_approx(fmaf(__uint_as_float(sr[c][i + 1]), p.c2, neg_m));
                ps[(c * 2 + (i >> 1)) & 3] += p0;
                ps[(c * 2 + (i >> 1) + 2) & 3] += p1;
                pk[c * 16 + (i >> 1)] = pack_bf16x2(p0, p1);
              }
            l_run = fmaf(l_run, alpha, (ps[0] + ps[1]) + (ps[2] + ps[3]));
          }
          if constexpr (MODE == kModeBias) request_bias(k + 1);
          tmem_st_32x32b_x32(s_addr, pk);
          publish_p(buf);
        } else {
          // Pass 1: row max (and min, for the softcap range check), independent chains.
          float mxa[4], mna[4];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            mxa[2 * c] = mxa[2 * c + 1] = -INFINITY;
            mna[2 * c] = mna[2 * c + 1] = INFINITY;
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float v0 = __uint_as_float(sr[c][i]), v1 = __uint_as_float(sr[c][i + 1]);
              const float v2 = __uint_as_float(sr[c][i + 2]), v3 = __uint_as_float(sr[c][i + 3]);
              mxa[2 * c] = max3(mxa[2 * c], v0, v1);
              mxa[2 * c + 1] = max3(mxa[2 * c + 1], v2, v3);
              if constexpr (MODE == kModeSoftcap) {
                mna[2 * c] = min3(mna[2 * c], v0, v1);
                mna[2 * c + 1] = min3(mna[2 * c + 1], v2, v3);
              }
            }
          }
          const float mx_all = fmaxf(fmaxf(mxa[0], mxa[1]), fmaxf(mxa[2], mxa[3]));
          float mx_keep = mx_all;
          if (masked) {  // max over the visible columns only
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              mxa[c] = -INFINITY;
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const int cc = c * 32 + i;
                const float v = (cc >= rel_lo && cc <= rel_hi) ? __uint_as_float(sr[c][i]) : -INFINITY;
                mxa[c] = fmaxf(mxa[c], v);
              }
            }
            mx_keep = fmaxf(mxa[0], mxa[1]);
          }

          // The score function is monotonic for the plain and softcap modes, so the max of the
          // scores is the score of the max.
          float tmax = mx_keep;
          unsigned flags = 0;  // bit 0: |x| > poly-1 limit, bit 1: |x| > poly-3 limit, bit 2: rescale
          if constexpr (MODE == kModeSoftcap) {
            tmax = (mx_keep == -INFINITY) ? -INFINITY : tanh_approx(mx_keep * p.a);
            // Every |x| of the warp's rows decides (masked columns included: their raw scores
            // are ordinary finite numbers).
            const float mn_all = fminf(fminf(mna[0], mna[1]), fminf(mna[2], mna[3]));
            const float bound = fabsf(p.a) * fmaxf(fabsf(mx_all), fabsf(mn_all));
            flags = (bound > kTanhPoly1Limit ? 1u : 0u) | (bound > kTanhPoly3Limit ? 2u : 0u);
          }
          const float m_new = fmaxf(m_used, tmax * p.c2);

          // Lazy rescale: move the reference max only when it grew by more than 2^8.
          float alpha = 1.f;
          if (m_new > -INFINITY && (m_used == -INFINITY || m_new - m_used > kRescaleThreshold)) {
            flags |= 4u;
            alpha = ex2_approx(m_used - m_new);  // 0 when m_used is -inf
            m_used = m_new;
          }
          flags = __reduce_or_sync(0xffffffffu, flags);  // one vote for all warp-level decisions
          // 0: x*(1 - x^2/3), 1: degree-7 polynomial, 2: MUFU tanh
          const int tanh_path = (flags & 2u) ? 2 : ((flags & 1u) ? 1 : 0);
          if (k > 0 && (flags & 4u)) {
            if (!pvs_before_complete(k)) {
              ok = false;
              break;
            }
#pragma unroll
            for (int c = 0; c < D / 32; ++c) rescale_o(c, alpha);
          }
          const float m_safe = (m_used == -INFINITY) ? 0.f : m_used;

          // Pass 2: p = exp2(score * c2 - m). Plain fp32 instructions and every exp2 on MUFU: a packed
          // f32x2 multiply-add in front of exp2 made the plain pass slower (1 x 32 x 8192, D = 128, 853 ->
          // 896 thousand clocks; the short polynomial of the fixed-reference kernel, three of them per pair, gains by
          // it), and so did an FMA-pipe emulation of part of the exp2.
          const float neg_m = -m_safe;
          float ps[4] = {0.f, 0.f, 0.f, 0.f};
          uint32_t pk[32];
          auto finish_pair = [&](float z0, float z1, int c, int i, bool apply_mask) {
            if (apply_mask) {
              const int cc = c * 32 + i;
              if (cc < rel_lo || cc > rel_hi) z0 = -INFINITY;
              if (cc + 1 < rel_lo || cc + 1 > rel_hi) z1 = -INFINITY;
            }
            const float p0 = ex2_approx(z0), p1 = ex2_approx(z1);
            ps[(c * 2 + (i >> 1)) & 3] += p0;
            ps[(c * 2 + (i >> 1) + 2) & 3] += p1;
            pk[c * 16 + (i >> 1)] = pack_bf16x2(p0, p1);
          };
          if (MODE == kModeSoftcap && tanh_path < 2) {
            // tanh(x) = x*(1 + y*(-1/3 + y*(2/15 + y*(-17/315)))), y = x^2, x = a*raw; the powers
            // of a are folded into the coefficients so that the polynomial runs on raw^2.
            const float a2 = p.a * p.a;
            const float b1 = -a2 / 3.f;
            const float ac = p.a * p.c2;
            if (tanh_path == 0) {
              auto body = [&](bool apply_mask) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                  for (int i = 0; i < 32; i += 2) {
                    const float r0 = __uint_as_float(sr[c][i]), r1 = __uint_as_float(sr[c][i + 1]);
                    const float q0 = fmaf(r0 * r0, b1, 1.f), q1 = fmaf(r1 * r1, b1, 1.f);
                    finish_pair(fmaf(r0 * ac, q0, neg_m), fmaf(r1 * ac, q1, neg_m), c, i,
                                apply_mask);
                  }
              };
              if (masked) body(true); else body(false);
            } else {
              const float b2 = a2 * a2 * (2.f / 15.f);
              const float b3 = a2 * a2 * a2 * (-17.f / 315.f);
              auto body = [&](bool apply_mask) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                  for (int i = 0; i < 32; i += 2) {
                    const float r0 = __uint_as_float(sr[c][i]), r1 = __uint_as_float(sr[c][i + 1]);
                    const float y0 = r0 * r0, y1 = r1 * r1;
                    const float q0 = fmaf(fmaf(fmaf(y0, b3, b2), y0, b1), y0, 1.f);
                    const float q1 = fmaf(fmaf(fmaf(y1, b3, b2), y1, b1), y1, 1.f);
                    finish_pair(fmaf(r0 * ac, q0, neg_m), fmaf(r1 * ac, q1, neg_m), c, i,
                                apply_mask);
                  }
              };
              if (masked) body(true); else body(false);
            }
          } else if constexpr (MODE == kModeSoftcap) {
            auto body = [&](bool apply_mask) {
#pragma unroll
              for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  const float t0 = tanh_approx(__uint_as_float(sr[c][i]) * p.a);
                  const float t1 = tanh_approx(__uint_as_float(sr[c][i + 1]) * p.a);
                  finish_pair(fmaf(t0, p.c2, neg_m), fmaf(t1, p.c2, neg_m), c, i, apply_mask);
                }
            };
            if (masked) body(true); else body(false);
          } else {
            auto body = [&](bool apply_mask) {
#pragma unroll
              for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2)
                  finish_pair(fmaf(__uint_as_float(sr[c][i]), p.c2, neg_m),
                              fmaf(__uint_as_float(sr[c][i + 1]), p.c2, neg_m), c, i, apply_mask);
            };
            if (masked) body(true); else body(false);
          }
          const float psum = (ps[0] + ps[1]) + (ps[2] + ps[3]);
          l_run = l_run * alpha + psum;
          tmem_st_32x32b_x32(s_addr, pk);
          publish_p(buf);
        }
      }

      // Epilogue: O_t / l -> bf16 -> global (one row per thread).
      if (ok && nblk > 0) {
        if (!mbar_wait(&bars->o_final[t], 0)) {
          report_timeout(p.status, 10 + t);
          ok = false;
        }
      }
      // Split: the slots tell each other their reference and sum, and each finishes half of the
      // columns from both accumulators (the same tensor-memory lanes, so a warp reads the other
      // slot's directly). A slot without a block has sum 0 and an accumulator nobody wrote.
      float inv, w_own = 1.f, w_other = 0.f;
      bool two = false;  // the other slot has something to add
      if (split) {
        float2* ml = reinterpret_cast<float2*>(sStage);  // [slot][row]
        ml[t * 128 + row] = make_float2(m_used, l_run);
        tc_fence_before();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const float2 other = ml[(t ^ 1) * 128 + row];
        asm volatile("bar.sync 1, 256;" ::: "memory");  // (the staging buffers start there)
        two = hi - lo > 1;
        const float m_all = fmaxf(m_used, other.x);
        const float m_safe = m_all == -INFINITY ? 0.f : m_all;
        w_own = ex2_approx(m_used - m_safe);
        w_other = ex2_approx(other.x - m_safe);
        inv = 1.f / (l_run * w_own + other.y * w_other);
        w_own *= inv;
        w_other *= inv;
      } else {
        inv = 1.f / l_run;
      }
      const float out_scale = split ? 1.f : inv;
      if (ok) {
        tc_fence_after();
        // Each warp owns 32 rows. A 32-column chunk (64 bytes per row) goes through a swizzled
        // 2 KB buffer of the warp so that one store instruction writes eight 64-byte row
        // segments instead of thirty-two 16-byte pieces.
        unsigned char* stage = sStage + warp * 2048;
        __nv_bfloat16* obase = p.out + b * p.o_stride[0] + h * p.o_stride[1];
        const int row0 = (iq0 + tq) * kTileQ + (warp & 3) * 32;  // first global row of the warp
        const int c_first = split ? t * (D / 64) : 0, c_end = split ? (t + 1) * (D / 64) : D / 32;
        [[maybe_unused]] const __nv_bfloat16* ob =
            MODE == kModeBias && p.out_bias
                ? p.out_bias + b * p.ob_stride[0] + h * p.ob_stride[1] + (lane & 3) * 8
                : nullptr;
#pragma unroll 1
        for (int c = c_first; c < c_end; ++c) {
          uint32_t orr[32];
          // (The output bias of the four pieces that this thread stores, requested before they are made.)
          [[maybe_unused]] uint4 bias4[4];
          if constexpr (MODE == kModeBias) {
            if (ob && LF_BOUNDS(row0 >= 0 && b * p.Hq + h < p.n_heads && c * 32 + 32 <= D, p.status, 63)) {
#pragma unroll
              for (int rr = 0; rr < 4; ++rr)
                bias4[rr] = ldg_stream_16(
                    ob + static_cast<int64_t>(min(row0 + rr * 8 + (lane >> 2), p.Sq - 1)) *
                             p.ob_stride[2] + c * 32);
            }
          }
          if (!split) {
            tmem_ld_32x32b_x32(o_addr + c * 32, orr);
            tmem_wait_ld();
          } else {
            const uint32_t other_addr = o_addr + (t ? -128 : 128);
            if (two) {
              uint32_t oth[32];
              tmem_ld_32x32b_x32(o_addr + c * 32, orr);
              tmem_ld_32x32b_x32(other_addr + c * 32, oth);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i)
                orr[i] = __float_as_uint(__uint_as_float(orr[i]) * w_own +
                                         __uint_as_float(oth[i]) * w_other);
            } else {
              tmem_ld_32x32b_x32(tmem_base + lane_addr + kColO + c * 32, orr);  // slot 0 has it all
              tmem_wait_ld();
              const float w = t == 0 ? w_own : w_other;
#pragma unroll
              for (int i = 0; i < 32; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * w);
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // piece q of row r sits at position q ^ ((r >> 1) & 3)
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(orr[8 * q]) * out_scale,
                              __uint_as_float(orr[8 * q + 1]) * out_scale);
            w.y = pack_bf16x2(__uint_as_float(orr[8 * q + 2]) * out_scale,
                              __uint_as_float(orr[8 * q + 3]) * out_scale);
            w.z = pack_bf16x2(__uint_as_float(orr[8 * q + 4]) * out_scale,
                              __uint_as_float(orr[8 * q + 5]) * out_scale);
            w.w = pack_bf16x2(__uint_as_float(orr[8 * q + 6]) * out_scale,
                              __uint_as_float(orr[8 * q + 7]) * out_scale);
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) = w;
          }
          __syncwarp();
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) {
            const int r = rr * 8 + (lane >> 2);
            const int q = lane & 3;
            uint4 w = *reinterpret_cast<const uint4*>(stage + r * 64 + ((q ^ ((r >> 1) & 3)) << 4));
            if constexpr (MODE == kModeBias) {
              if (ob) w = add_bf16x8(w, bias4[rr]);
            }
            if (row0 + r < p.Sq)
              *reinterpret_cast<uint4*>(obase + static_cast<int64_t>(row0 + r) * p.o_stride[2] +
                                        c * 32 + q * 8) = w;
          }
          __syncwarp();
        }
      }
    } else if (tile_valid(t) && grow < p.Sq) {
      // No visible key at all for this tile: softmax of an all -inf row is NaN in the
      // eager computation, so the rows are written as NaN.
      __nv_bfloat16* orow = p.out + b * p.o_stride[0] + h * p.o_stride[1] +
                            static_cast<int64_t>(grow) * p.o_stride[2];
      const uint4 nan4 = {0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u};
#pragma unroll
      for (int c = 0; c < D; c += 8) *reinterpret_cast<uint4*>(orow + c) = nan4;
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Shape::kTmemColumns);
  }
}

}  // namespace lf

#include "lf_prefill_bounded.cuh"
#include "lf_prefill_wide.cuh"

namespace lf {

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000,
                                                     cudaEnableDefault, &qres);
    if (e == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    else
      set_cuda_error(e, "cudaGetDriverEntryPointByVersion(cuTensorMapEncodeTiled)");
  });
  return fn;
}

// Tensor map over a bf16 [B, H, S, D] tensor (innermost stride 1), box = [1, 1, box_rows,
// box_cols]; 128-byte swizzle for 64-column boxes (the K/V/Q loads, out-of-range rows read as
// zero), 64-byte swizzle for 32-column boxes (the output store of the persistent kernels).
static int encode_tile_map(CUtensorMap* map, const void* base, int B, int H, int S, int D,
                           const int64_t* stride /* b, h, s in elements */, int box_rows,
                           int box_cols) {
  auto fn = get_encode_fn();
  if (!fn) return LF_ERR_CUDA;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(S),
                        static_cast<cuuint64_t>(H), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(stride[2]) * 2,
                           static_cast<cuuint64_t>(stride[1]) * 2,
                           static_cast<cuuint64_t>(stride[0]) * 2};
  // A dimension of extent 1 may carry any stride; keep it a valid multiple of 16 bytes.
  for (int i = 0; i < 3; ++i)
    if (strides[i] == 0 || (strides[i] & 15)) {
      if (dims[i + 1] == 1)
        strides[i] = 16 * ((static_cast<cuuint64_t>(D) * 2 + 15) / 16);
      else
        return LF_ERR_ALIGNMENT;
    }
  cuuint32_t box[4] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows), 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
    return LF_ERR_CUDA;
  }
  return LF_OK;
}

// Tensor map over the token rows of a paged pool, for row gathers: `rows` rows of `cols` elements, box of
// one row x 64 columns (box_rows == 1 tells these from the maps above).
static int encode_gather_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols,
                             int64_t row_stride) {
  auto fn = get_encode_fn();
  if (!fn) return LF_ERR_CUDA;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_stride) * 2};
  cuuint32_t box[2] = {64, 1}, estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled(gather)");
    return LF_ERR_CUDA;
  }
  return LF_OK;
}

// Elements between the token rows of a pool [n_pages, page_size, Hkv, D] with strides (page, slot,
// kv head) when the pool is one 2-D tensor of rows that hold all heads; 0 when it is not.
static int64_t gather_row_stride(const int64_t* st, int n_pages, int page_size, int Hkv, int D) {
  const int64_t row = page_size == 1 ? st[0] : st[1];
  if (page_size > 1 && n_pages > 1 && st[0] != page_size * st[1]) return 0;
  if (row <= 0 || row % 8 || st[2] < 0 || (Hkv - 1) * st[2] + D > row) return 0;
  if (static_cast<int64_t>(n_pages) * page_size > 0x7fffff00ll || row > (1 << 30)) return 0;
  return row;
}

// Encoded tensor maps are kept in a small cache: a map depends only on (address, shape,
// strides, box), and serving loops call with the same buffers again and again. Direct-mapped,
// one mutex; a miss just encodes again, so the cache never changes a result. A CUtensorMap holds
// no reference to the memory it describes: an entry whose buffer was freed is harmless and is
// simply replaced when another key lands on its slot.
struct TileMapKey {
  const void* base;
  int32_t B, H, S, D, box_rows, box_cols;
  int64_t stride[3];
  bool operator==(const TileMapKey& o) const {
    return base == o.base && B == o.B && H == o.H && S == o.S && D == o.D &&
           box_rows == o.box_rows && box_cols == o.box_cols && stride[0] == o.stride[0] &&
           stride[1] == o.stride[1] && stride[2] == o.stride[2];
  }
};
struct TileMapEntry {
  bool valid = false;
  TileMapKey key;
  CUtensorMap map;
};
constexpr int kTileMapCacheSlots = 256;
static std::mutex g_tile_map_mutex;
static TileMapEntry g_tile_map_cache[kTileMapCacheSlots];
static std::atomic<uint64_t> g_tile_map_hits{0}, g_tile_map_misses{0};

static int make_tile_map(CUtensorMap* map, const void* base, int B, int H, int S, int D,
                         const int64_t* stride, int box_rows, int box_cols = 64) {
  TileMapKey key{base, B, H, S, D, box_rows, box_cols, {stride[0], stride[1], stride[2]}};
  uint64_t h = reinterpret_cast<uintptr_t>(base) * 0x9E3779B97F4A7C15ull;
  h ^= (static_cast<uint64_t>(S) << 32 | static_cast<uint32_t>(H)) * 0xC2B2AE3D27D4EB4Full;
  h ^= (static_cast<uint64_t>(B) << 40 | static_cast<uint64_t>(box_rows) << 16 |
        static_cast<uint64_t>(box_cols) << 8 | static_cast<uint64_t>(D)) * 0x165667B19E3779F9ull;
  h ^= static_cast<uint64_t>(stride[2]) * 0x27D4EB2F165667C5ull;
  const int slot = static_cast<int>((h >> 32) % kTileMapCacheSlots);
  {
    std::lock_guard<std::mutex> lock(g_tile_map_mutex);
    const TileMapEntry& e = g_tile_map_cache[slot];
    if (e.valid && e.key == key) {
      *map = e.map;
      g_tile_map_hits.fetch_add(1, std::memory_order_relaxed);
      return LF_OK;
    }
  }
  const int rc = box_rows == 1 ? encode_gather_map(map, base, S, D, stride[2])
                               : encode_tile_map(map, base, B, H, S, D, stride, box_rows, box_cols);
  if (rc != LF_OK) return rc;
  g_tile_map_misses.fetch_add(1, std::memory_order_relaxed);
  std::lock_guard<std::mutex> lock(g_tile_map_mutex);
  TileMapEntry& e = g_tile_map_cache[slot];
  e.key = key;
  e.map = *map;
  e.valid = true;
  return LF_OK;
}

// SMs of the current device (asked once per device); 0 after an error, which is recorded.
static int current_sm_count() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> counts[kMaxDevices];
  int dev = 0, n = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && dev < kMaxDevices) n = counts[dev].load(std::memory_order_relaxed);
  if (e == cudaSuccess && n == 0) {
    e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && dev < kMaxDevices) counts[dev].store(n, std::memory_order_relaxed);
  }
  if (e != cudaSuccess) {
    set_cuda_error(e, "number of SMs");
    return 0;
  }
  return n;
}

// How the prefill kernels deal the query tiles out.
enum class PrefillForm {
  kPairs = LF_FORM_PAIRS,    // two tiles of a head per CTA, one CTA per SM
  kSplit = LF_FORM_SPLIT,    // one tile per CTA, its key blocks split over the CTA's two slots
  kNarrow = LF_FORM_NARROW,  // one tile per CTA, two CTAs per SM
};

// Between one and two tiles per SM, with an SM for every pair: whether two CTAs per SM would place enough beside the
// longest tiles to be the slower form. A pair leaves the longest tile of an odd number alone on its SM; two tiles a
// head are no better off apart at D = 128. (From 1.2 tiles per SM on, and from 1.35 with five tiles a head or more, of
// which the first to share an SM are very light.)
static bool longest_tile_alone(int tiles, int64_t n_tiles, int D, int sm_count) {
  if (tiles == 2 ? D == 64 : tiles % 2 == 0) return false;
  return n_tiles * 20 >= sm_count * (tiles <= 3 ? 24ll : 27ll);
}

// One query tile per CTA, its key blocks split over the two slots:
//   - where all the tiles are resident at once, one per SM: half the steps of the longest tile (8
//     heads, 1024 queries, 8192 keys, D = 64: 111 -> 59 us);
//   - up to two tiles per SM, where the others would leave the short ones' SMs idle while the longest
//     runs: a pair of tiles takes as many steps as its longer tile has blocks; split tiles,
//     longest first, the mean load, half of the shortest tile, and about five steps for the start
//     and end of the second CTA of an SM (causal, 16 heads, 2048 keys, D = 64: pairs 34.9 us, narrow 27.9,
//     split 21.3; 7 tiles x 32 heads that see 3.4 to 4.1 thousand keys each, D = 128: pairs 64, split 75). With a
//     paged operand a step of split tiles gathers twice the rows: 1.4 steps.
// Two CTAs per SM (`can_narrow`: the kernel has that form): the start and end of a CTA, some 13 thousand clocks
// that pairs leave bare, lie under the other one's blocks, no slot is empty where a head has an odd number of
// tiles, and the issuing warps of two tiles no longer wait for one ring. Past two tiles per SM, back to back for half
// a second (causal; pairs -> narrow):
//   D = 64, any length: 8 x 32 x 512 34.0 -> 29.7 us, 8 x 32 x 1024 84.1 -> 76.5, 4 x 16 x 2048 68.4 -> 62.5, 1 x 16 x
//   8192 210 -> 194; paged 8 x 32 x 1024 100.4 -> 91.2, biased 8 x 16 x 512 38.1 -> 33.9.
//   D = 128 up to 24 blocks a tile: 8 x 64 x 100 23.1 -> 13.3, 8 x 32 x 640 59.0 -> 51.6, 8 x 32 x 1024 105.4 -> 101.7,
//   4 x 32 x 1536 103.5 -> 101.7, biased 4 x 16 x 1024 69.5 -> 64.4; windows of 64 to 1300 0.85 to 0.97 of pairs (also where
//   the last tile sees no key: the rule looks at that one alone). Further on the chip runs at its power limit and
//   K and V read once for both tiles count for more: chunks of 1024 with 4000 keys before them 158.8 -> 160.9,
//   1 x 32 x 8192 444.6 -> 453.7; but for heads of which pairs leave a good part of the slots empty. Three tiles a head
//   (a quarter empty): 456 tiles of 2500 / 4200 / 8200 keys 112 -> 99, 181 -> 161, 350 -> 305, 2592 of them 0.91 to 0.92 of
//   pairs, 444 0.90 to 1.00, but 384 of 1800 / 2500 / 4300 keys 51.8 -> 53.2, 68.4 -> 72.0, 114 -> 126 (paged, 2000:
//   65.0 -> 69.0; of 1200 and 8300 keys 0.95 to 1.01, biased 0.93 to 0.98). Five (a sixth): 680 tiles 1.02 to 1.06 of pairs, 1280 0.91 to
//   0.99, 2600 0.92 to 0.94. Seven: 0.95 to 1.05, nine 0.95 to 1.03, four 0.95 to 1.02.
// One tile a head (split -> narrow; 128 rows): 240 tiles of 64 keys 8.5 -> 4.4, of 4096 63.2 -> 57.5; D = 128 10.2 ->
// 5.8 and 94 -> 71; 592 tiles of 1024 keys 45.5 -> 34.4 and 67 -> 46. Between two and three tiles per SM split tiles
// take three rounds of half the steps against two of all, which is as good for plain scores (440 tiles, D = 128: 2048
// keys 76.9 -> 74.5, 4096 139.8 -> 142.8) and the better for biased ones, whose steps wait for their bias (320 tiles of 512
// keys the same, 1024 56.9 -> 59.3, 2048 98.5 -> 107.0; D = 128 65.3 -> 69.6 and 112.7 -> 125.4).
// Up to two tiles per SM (ratios are narrow / pairs):
//   - where pairs need a second round (three tiles of 384 rows x 96 heads, D = 128 15.4 -> 10.6 us, 2000 keys 57 -> 35;
//     D = 64 0.60 to 0.68) narrow;
//   - D = 64 and paged operands, otherwise: narrow (777 rows and 3319 keys before them, 32 heads, 58.0 -> 54.6, paged
//     4 x 8 x 1024 19.6 -> 18.8; 2 to 16 tiles a head 0.80 to 1.00), but for an odd number of short tiles a head: the
//     longest has an SM to itself as a pair, where narrow has to place others beside it (180 to 216 tiles, three a head, 6 blocks 1.04 to 1.08, 15 blocks 1.04 to 1.07, 53 blocks 1.00; five a head,
//     10 blocks 1.04; paged 1.00 to 1.07); two short paged tiles a head at D = 128 are no better (1.00 to 1.04);
//   - D = 128, dense: pairs (777 rows and 3319 keys 65.0 -> 65.4; two tiles a head 1.01 to 1.08, three 1.02 to 1.16).
static PrefillForm choose_form(const PrefillParams& p, int D, int B, int sm_count, bool can_narrow) {
  const int64_t n_tiles = static_cast<int64_t>(p.n_qtiles) * p.Hq * B;
  if (n_tiles <= sm_count) return PrefillForm::kSplit;
  int lo, hi;
  skip_range(p.mask_kind, p.window, p.causal_offset, p.Sq, p.Skv, kTileQ, kTileK, 0, &lo, &hi);
  const int shortest = hi - lo;
  skip_range(p.mask_kind, p.window, p.causal_offset, p.Sq, p.Skv, kTileQ, kTileK, p.n_qtiles - 1, &lo, &hi);
  const int longest = hi - lo;
  if (p.n_qtiles == 1) {
    const bool three_rounds = n_tiles > 2ll * sm_count && n_tiles <= 3ll * sm_count;
    const bool split = !can_narrow || (p.bias && three_rounds && longest >= 12);
    return split ? PrefillForm::kSplit : PrefillForm::kNarrow;
  }
  if (n_tiles <= 2ll * sm_count) {
    const double split = 0.25 * (shortest + longest) * static_cast<double>(n_tiles) / sm_count + 0.5 * shortest;
    if (split * (p.paged ? 1.4 : 1.0) + 5.0 < longest) return PrefillForm::kSplit;
    if (!can_narrow) return PrefillForm::kPairs;
    if ((p.n_qtiles + 1ll) / 2 * p.Hq * B > sm_count) return PrefillForm::kNarrow;
    if (D == 128 && !p.paged) return PrefillForm::kPairs;
    const bool alone = longest_tile_alone(p.n_qtiles, n_tiles, D, sm_count);
    return alone && longest <= 20 ? PrefillForm::kPairs : PrefillForm::kNarrow;
  }
  if (!can_narrow) return PrefillForm::kPairs;
  if (D == 64) return PrefillForm::kNarrow;
  // (2.2 to 3 tiles per SM: a second round of narrow CTAs that leaves most SMs half empty or empty)
  const bool half_round = n_tiles * 10 >= sm_count * 22ll && n_tiles < 3ll * sm_count;
  if (p.n_qtiles == 3 && half_round && longest > 20 && longest < 100 && !p.bias) return PrefillForm::kPairs;
  const bool empty_slots = p.n_qtiles == 3 || (p.n_qtiles == 5 && n_tiles > 6ll * sm_count);
  return longest <= 24 || empty_slots ? PrefillForm::kNarrow : PrefillForm::kPairs;
}

template <int D, int MODE, bool PE = false, bool NARROW = false>
static int launch_prefill(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                          const PrefillParams& p, int B, cudaStream_t st, PrefillForm form,
                          const CUtensorMap* mqpe = nullptr, const CUtensorMap* mkpe = nullptr) {
  using Shape = PrefillShape<D, PE, NARROW>;
  constexpr size_t smem = Shape::kSmem;
  static_assert(smem <= 232448 && (!NARROW || 2 * (smem + 1024) <= 233472), "shared memory of a CTA");
  static_assert(keeps_tensor_memory(smem, NARROW), "tensor memory of an SM");
  static thread_local int configured_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(prefill_kernel<D, MODE, PE, NARROW>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) {
      set_cuda_error(e, "cudaFuncSetAttribute(prefill_kernel)");
      return LF_ERR_CUDA;
    }
    configured_dev = dev;
  }
  const int pairs = (p.n_qtiles + 1) / 2;
  PrefillParams pp = p;
  pp.single = form != PrefillForm::kPairs;
  // Order of the CTAs: the heaviest tiles of a group of heads, then the next lighter ones, ..., then
  // the next group. With a head's tiles next to each other the last head's longest tile started
  // when the rest was nearly done (single launches of B=1 Hq=32 Hkv=8
  // S=8192 D=128, causal, at the full clock 535 -> 475 us, of B=4 Hq=16 S=2048 D=64 91 -> 78). A group is as many heads as keep their
  // K and V in half of L2, since its heads' tiles now read them at different times.
  const int tiles = pp.single ? p.n_qtiles : pairs;
  const int64_t heads = static_cast<int64_t>(p.Hq) * B;
  const int64_t kv_bytes = static_cast<int64_t>(p.Skv) * (D + (PE ? 64 : 0) + D) * 2;
  int64_t per_group = std::max<int64_t>(1, (64ll << 20) / kv_bytes) * p.group;
  const int64_t groups = (heads + per_group - 1) / per_group;
  per_group = ((heads + groups - 1) / groups + p.group - 1) / p.group * p.group;
  if (per_group * groups * tiles > 0x7fffffff) return LF_ERR_TOO_LARGE;
  pp.n_heads = static_cast<int32_t>(heads);
  pp.div_main = FastDiv::make(static_cast<int32_t>(per_group));
  pp.div_deferred = FastDiv::make(tiles);
  pp.div_hq = FastDiv::make(p.Hq);
  pp.div_group = FastDiv::make(p.group);
  const unsigned grid = static_cast<unsigned>(per_group * groups * tiles);
  // (without a second score product the two extra maps are never read)
  launch_pdl(prefill_kernel<D, MODE, PE, NARROW>, dim3(grid), Shape::kThreads, smem, st, mq, mk, mv,
             mqpe ? *mqpe : mq, mkpe ? *mkpe : mk, pp);
  return check_launch("prefill_kernel");
}

template <int D, int MODE>
static int launch_prefill_form(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                               const PrefillParams& p, int B, cudaStream_t st, PrefillForm form) {
  if constexpr (MODE == kModeNone || MODE == kModeBias)  // (form_of)
    if (form == PrefillForm::kNarrow) return launch_prefill<D, MODE, false, true>(mq, mk, mv, p, B, st, form);
  return launch_prefill<D, MODE>(mq, mk, mv, p, B, st, form);
}

// Ticket counters of the persistent kernel: a small ring in the library image, so that launching
// allocates nothing. A launch takes the next slot and zeroes it in stream order; launches that
// overlap on the GPU use different slots unless more than kTicketSlots are in flight.
constexpr int kTicketSlots = 256;
static __device__ unsigned int g_prefill_tickets[kTicketSlots];
static std::atomic<unsigned int> g_next_ticket_slot{0};

// Whether the fixed-reference kernel runs as two CTAs of one tile slot per SM (narrow) instead of one of two. The slots
// then no longer share a ring and an item's end, and a tile that has an SM to itself has all of it; but every tile
// fetches its own K and V. Both back to back for half a second, softcap 50 (two slots -> narrow):
//   D = 64: 8 x 32 x 1024 78.9 -> 76.9 us, 2 x 16 x 4096 142.0 -> 129.6, 2 x 4 x 512 14.5 -> 12.3, window 256, four heads
//   per kv head, 8 x 32 x 2048 87.7 -> 87.2, 1 x 8 x 2048 12.3 -> 10.3;
//   D = 128, no more tiles than SMs: 1 x 8 x 2048 38.4 -> 30.7, 2 x 8 x 1024 23.9 -> 19.1; unless a head has one tile, which
//   has an SM to itself in either form, where the deeper ring of the two-slot form holds its keys' latency better (8 to
//   148 tiles of 1000 keys 18.5 -> 19.3 to 22.6 -> 24.7, of 4000 52 -> 63, 148 of 8000 117 -> 146);
//   up to 10 blocks a tile: 8 x 64 x 256 30.7 -> 28.9, 8 x 32 x 512 41.9 -> 40.3, 8 x 16 x 600 32.7 -> 31.0; up to 16 and
//   four tiles per SM: 2 x 32 x 700 26.7 -> 24.5, 4 x 16 x 1024 35.8 -> 35.2; beyond, the chip's power limit decides and K
//   and V read once for two tiles win (8 x 32 x 1024 108.1 -> 109.1, 8 x 32 x 2048 338.7 -> 346.6, 1 x 8 x 8192 175.1 ->
//   180.0);
//   between one and two tiles per SM, at either head size: narrow where pairs need a second round (three tiles a head,
//   294 in all, D = 128 0.78, D = 64 over 3000 keys 0.63), two slots where an odd number of tiles leaves the longest one
//   alone (180 to 240 tiles, three a head 1.00 to 1.16; 200 to 240, five 1.00 to 1.12, seven 1.00 to 1.10), for seven causal
//   tiles a head also past 148 pairs, the light ones of which then take two turns under the longest (1.03), and for two
//   tiles a head at D = 128 (256 rows x 128 heads 12.4 against 13.1 us; 1.00 to 1.08);
//   D = 128 packed, up to four chunks per SM (1 x 8 x 2048, window 256 14.4 -> 12.3; 2 x 16 x 2048, window 1000
//   45.1 -> 43.2; 8 x 32 x 2048, window 256 121.3 -> 124.3).
static bool bounded_is_narrow(const PrefillParams& p, int D, int pack, int B, int sm_count) {
  if (p.sm_margin > 0) return false;  // (two CTAs per SM would spread over the SMs to be left free)
  if (D == 64 && pack > 1) return true;
  const int rows = kTileQ / pack;
  const int64_t heads = static_cast<int64_t>(p.Hq / pack) * B, n_tiles = (p.Sq + rows - 1) / rows * heads;
  const bool few = n_tiles <= 4ll * sm_count;
  if (pack > 1) return few;
  auto blocks = [&](int iq) {
    int lo, hi;
    skip_range(p.mask_kind, p.window, p.causal_offset, p.Sq, p.Skv, kTileQ, kTileK, iq, &lo, &hi);
    return hi - lo;
  };
  const int longest = blocks(p.n_qtiles - 1);
  if (p.n_qtiles > 1 && n_tiles > sm_count && n_tiles <= 2ll * sm_count) {
    const bool light = 2 * (blocks(1) + 5) <= longest + 5;  // (a CTA's start and end count as five blocks)
    if ((p.n_qtiles + 1ll) / 2 * heads > sm_count && !light) return true;
    if (longest_tile_alone(p.n_qtiles, n_tiles, D, sm_count)) return false;
  }
  if (D == 64) return true;
  if (p.n_qtiles == 1 && n_tiles <= sm_count) return false;
  return n_tiles <= sm_count || longest <= (few ? 16 : 10);
}

// The form of a call's kernel. Plain and biased scores have the narrow form of prefill_kernel. (Rows that the
// producer warp copies itself need three ring stages, which it has at D = 64.)
static PrefillForm form_of(const PrefillParams& p, int mode, bool has_pe, int D, int pack, int kv_tile, int B,
                           int sm_count) {
  if (mode == kModeBounded)
    return kv_tile != kWideK && bounded_is_narrow(p, D, pack, B, sm_count) ? PrefillForm::kNarrow
                                                                           : PrefillForm::kPairs;
  const bool can_narrow = (mode == kModeNone || mode == kModeBias) && !has_pe && (!p.paged || p.gather || D == 64);
  return choose_form(p, D, B, sm_count, can_narrow);
}

template <int D, int PACK = 1, bool NARROW = false>
static int launch_prefill_bounded(const CUtensorMap& mq, const CUtensorMap& mk,
                                  const CUtensorMap& mv, const CUtensorMap& mo, PrefillParams p,
                                  int B, cudaStream_t st, int sm_count) {
  using Shape = BoundedShape<D, PACK, NARROW>;
  constexpr size_t smem = Shape::kSmem;
  static_assert(smem <= 232448 && (!NARROW || 2 * (smem + 1024) <= 233472), "shared memory of a CTA");
  static_assert(keeps_tensor_memory(smem, NARROW), "tensor memory of an SM");
  static thread_local int configured_dev = -1;
  static thread_local unsigned int* tickets = nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(prefill_bounded_kernel<D, PACK, NARROW>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e == cudaSuccess)
      e = cudaGetSymbolAddress(reinterpret_cast<void**>(&tickets), g_prefill_tickets);
    if (e != cudaSuccess) {
      set_cuda_error(e, "prefill_bounded_kernel setup");
      return LF_ERR_CUDA;
    }
    configured_dev = dev;
  }
  // Packed layout: the query rows are walked in chunks of 128 / PACK (p.n_qtiles counts those) and an
  // item is a pair of chunks of one kv head, for all of its query heads at once.
  const int heads = PACK > 1 ? p.Hq / p.group : p.Hq;
  if (PACK > 1) p.n_qtiles = (p.Sq + kTileQ / PACK - 1) / (kTileQ / PACK);
  p.n_pairs = NARROW ? p.n_qtiles : (p.n_qtiles + 1) / 2;
  p.n_deferred = (p.mask_kind == LF_MASK_CAUSAL && p.Sq == p.Skv) ? p.n_pairs / 4 : 0;
  p.main_items = static_cast<int32_t>(static_cast<int64_t>(p.n_pairs - p.n_deferred) * heads * B);
  p.div_main = FastDiv::make(p.n_pairs - p.n_deferred);
  p.div_deferred = FastDiv::make(p.n_deferred > 0 ? p.n_deferred : 1);
  p.div_hq = FastDiv::make(heads);
  p.div_group = FastDiv::make(p.group);
  const int64_t n_items = static_cast<int64_t>(p.n_pairs) * heads * B;
  if (n_items > 0x7fffffff - 4096) return LF_ERR_TOO_LARGE;
  p.n_items = static_cast<int32_t>(n_items);
  p.ticket = tickets + g_next_ticket_slot.fetch_add(1) % kTicketSlots;
  cudaError_t e = cudaMemsetAsync(p.ticket, 0, sizeof(unsigned int), st);
  if (e != cudaSuccess) {
    set_cuda_error(e, "cudaMemsetAsync(ticket)");
    return LF_ERR_CUDA;
  }
  const int ctas = sm_count - p.sm_margin > 0 ? sm_count - p.sm_margin : 1;
  const int64_t slots = static_cast<int64_t>(ctas) * (NARROW ? 2 : 1);
  const int grid = static_cast<int>(n_items < slots ? n_items : slots);
  prefill_bounded_kernel<D, PACK, NARROW><<<grid, Shape::kThreads, smem, st>>>(mq, mk, mv, mo, p);
  return check_launch("prefill_bounded_kernel");
}

template <int D>
static int launch_prefill_bounded_form(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                                       const CUtensorMap& mo, const PrefillParams& p, int B, cudaStream_t st,
                                       int pack, PrefillForm form, int sm_count) {
  const bool narrow = form == PrefillForm::kNarrow;
  if (pack == 4)
    return narrow ? launch_prefill_bounded<D, 4, true>(mq, mk, mv, mo, p, B, st, sm_count)
                  : launch_prefill_bounded<D, 4>(mq, mk, mv, mo, p, B, st, sm_count);
  if (pack == 2)
    return narrow ? launch_prefill_bounded<D, 2, true>(mq, mk, mv, mo, p, B, st, sm_count)
                  : launch_prefill_bounded<D, 2>(mq, mk, mv, mo, p, B, st, sm_count);
  return narrow ? launch_prefill_bounded<D, 1, true>(mq, mk, mv, mo, p, B, st, sm_count)
                : launch_prefill_bounded<D>(mq, mk, mv, mo, p, B, st, sm_count);
}

template <int D>
static int launch_prefill_wide(const CUtensorMap& mq, const CUtensorMap& mk,
                               const CUtensorMap& mv, const CUtensorMap& mo, PrefillParams p,
                               int B, cudaStream_t st, int sm_count) {
  constexpr size_t kQTileBytes = static_cast<size_t>(kTileQ) * D * 2;
  constexpr size_t kKVTileBytes = static_cast<size_t>(kWideK) * D * 2;
  constexpr size_t smem = 1024 /*align slack*/ + 1024 /*barriers*/ + kBoundedStageBytes +
                          2 * kQTileBytes + WideRingFor<D>::value * kKVTileBytes;
  static thread_local int configured_dev = -1;
  static thread_local unsigned int* tickets = nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(prefill_wide_kernel<D>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e == cudaSuccess)
      e = cudaGetSymbolAddress(reinterpret_cast<void**>(&tickets), g_prefill_tickets);
    if (e != cudaSuccess) {
      set_cuda_error(e, "prefill_wide_kernel setup");
      return LF_ERR_CUDA;
    }
    configured_dev = dev;
  }
  p.n_pairs = (p.n_qtiles + 1) / 2;
  p.n_deferred = (p.mask_kind == LF_MASK_CAUSAL && p.Sq == p.Skv) ? p.n_pairs / 4 : 0;
  p.main_items = static_cast<int32_t>(static_cast<int64_t>(p.n_pairs - p.n_deferred) * p.Hq * B);
  p.div_main = FastDiv::make(p.n_pairs - p.n_deferred);
  p.div_deferred = FastDiv::make(p.n_deferred > 0 ? p.n_deferred : 1);
  p.div_hq = FastDiv::make(p.Hq);
  p.div_group = FastDiv::make(p.group);
  const int64_t n_items = static_cast<int64_t>(p.n_pairs) * p.Hq * B;
  if (n_items > 0x7fffffff - 4096) return LF_ERR_TOO_LARGE;
  p.n_items = static_cast<int32_t>(n_items);
  p.ticket = tickets + g_next_ticket_slot.fetch_add(1) % kTicketSlots;
  cudaError_t e = cudaMemsetAsync(p.ticket, 0, sizeof(unsigned int), st);
  if (e != cudaSuccess) {
    set_cuda_error(e, "cudaMemsetAsync(ticket)");
    return LF_ERR_CUDA;
  }
  const int ctas = sm_count - p.sm_margin > 0 ? sm_count - p.sm_margin : 1;
  const int grid = static_cast<int>(n_items < ctas ? n_items : ctas);
  prefill_wide_kernel<D><<<grid, kWideThreads, smem, st>>>(mq, mk, mv, mo, p);
  return check_launch("prefill_wide_kernel");
}

// KV tile of the kernel that serves these arguments. The bounded-softcap mode has two kernels:
// 64-key tiles (two S buffers per query tile, the default: the faster of the two on every
// configuration measured) and 128-key tiles (one S buffer, math-bound N=128 QK^T MMAs), which a
// caller can pin with kv_tile = 128. Every running-max kernel uses 64-key tiles.
static int choose_kv_tile(const LfPrefillArgs* a, int mode) {
  if (a->kv_tile != 0 && a->kv_tile != kTileK && a->kv_tile != kWideK) return LF_ERR_INVALID_ARG;
  if (mode != kModeBounded) return a->kv_tile == kWideK ? LF_ERR_UNSUPPORTED : kTileK;
  return a->kv_tile != 0 ? a->kv_tile : kTileK;
}

// What a call runs, for the queries.
struct PrefillChoice {
  int q_tile = 0;
  int sm_count = 0;  // in: of the device that is asked about; 0 = the current one, -1 = the form is not asked for
  int form = 0;
};

// `launch` == nullptr: only resolve the kernel choice and return its KV tile size.
static int prefill_impl(const LfPrefillArgs* a, void* const* launch, PrefillChoice* choice = nullptr,
                        const LfRowBias* rows = nullptr) {
  if (!a || !a->q || !a->k || !a->v || !a->out) return LF_ERR_INVALID_ARG;
  if (a->B <= 0 || a->Hq <= 0 || a->Hkv <= 0 || a->Sq <= 0 || a->Skv <= 0)
    return LF_ERR_INVALID_ARG;
  if (a->Hq % a->Hkv) return LF_ERR_INVALID_ARG;
  if (a->D != 64 && a->D != 128) return LF_ERR_UNSUPPORTED;
  if (a->n_mod < 0 || a->n_mod > LF_MAX_MODS) return LF_ERR_INVALID_ARG;
  if (a->mask_kind < LF_MASK_NONE || a->mask_kind > LF_MASK_CAUSAL_WINDOW)
    return LF_ERR_INVALID_ARG;
  if (a->mask_kind == LF_MASK_CAUSAL_WINDOW && a->window <= 0) return LF_ERR_INVALID_ARG;
  if (a->Hq > 65535 || a->B > 65535) return LF_ERR_TOO_LARGE;
  const void* ptrs[4] = {a->q, a->k, a->v, a->out};
  for (const void* ptr : ptrs)
    if (reinterpret_cast<uintptr_t>(ptr) & 15u) return LF_ERR_ALIGNMENT;
  for (int i = 0; i < 3; ++i)
    if (a->o_stride[i] % 8) return LF_ERR_ALIGNMENT;

  PrefillParams p;
  p.out = static_cast<__nv_bfloat16*>(a->out);
  for (int i = 0; i < 3; ++i) p.o_stride[i] = a->o_stride[i];
  p.Sq = a->Sq;
  p.Skv = a->Skv;
  p.Hq = a->Hq;
  p.group = a->Hq / a->Hkv;
  p.mask_kind = a->mask_kind;
  p.window = a->window;
  p.causal_offset = a->causal_offset;
  p.n_qtiles = (a->Sq + kTileQ - 1) / kTileQ;
  p.status = a->status;
  p.dbg_ranges = a->dbg_ranges;
  for (int i = 0; i < 4; ++i) p.qc[i] = 0.f;
  p.ylim[0] = p.ylim[1] = 0.f;
  p.single = 0;
  p.n_pairs = 0;
  p.n_deferred = 0;
  p.main_items = 0;
  p.div_main = p.div_deferred = p.div_hq = p.div_group = FastDiv::make(1);
  p.n_items = p.n_heads = 0;
  p.ticket = nullptr;
  if (a->sm_margin < 0) return LF_ERR_INVALID_ARG;
  p.sm_margin = a->sm_margin;
  // Paged operands: `k` / `v` is then a pool [n_pages, page_size, Hkv, D] with strides (page,
  // slot, kv head), read through its block table.
  p.paged = (a->k_block_table ? 1 : 0) | (a->v_block_table ? 2 : 0);
  p.k_pool = static_cast<const __nv_bfloat16*>(a->k);
  p.v_pool = static_cast<const __nv_bfloat16*>(a->v);
  p.k_table = a->k_block_table;
  p.v_table = a->v_block_table;
  for (int i = 0; i < 3; ++i) {
    p.kp_stride[i] = a->k_stride[i];
    p.vp_stride[i] = a->v_stride[i];
  }
  p.bt_stride = a->bt_stride;
  p.page_size = a->page_size;
  p.page_shift = -1;
  p.n_pages = a->n_pages;
  p.gather = 0;
  if (p.paged) {
    if (a->page_size <= 0 || a->n_pages <= 0) return LF_ERR_INVALID_ARG;
    if (a->bt_stride < (a->Skv + a->page_size - 1) / a->page_size) return LF_ERR_INVALID_ARG;
    for (int sh = 0; sh < 31; ++sh)
      if ((1 << sh) == a->page_size) p.page_shift = sh;
    for (int i = 0; i < 3; ++i)
      if (((p.paged & 1) && a->k_stride[i] % 8) || ((p.paged & 2) && a->v_stride[i] % 8))
        return LF_ERR_ALIGNMENT;
  }
  p.mods.n = 0;
  for (int i = 0; i < LF_MAX_MODS; ++i) {
    p.mods.op[i] = 0;
    p.mods.arg[i] = 0.f;
  }
  p.pe_steps = 0;
  const bool has_pe = a->q_pe != nullptr || a->k_pe != nullptr;
  if (has_pe) {
    if (!a->q_pe || !a->k_pe) return LF_ERR_INVALID_ARG;
    if (a->D_pe <= 0 || a->D_pe > 64 || a->D_pe % 8) return LF_ERR_UNSUPPORTED;
    if (p.paged || a->score_bias) return LF_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(a->q_pe) | reinterpret_cast<uintptr_t>(a->k_pe)) & 15u)
      return LF_ERR_ALIGNMENT;
    p.pe_steps = (a->D_pe + 15) / 16;
  }
  p.bias = static_cast<const __nv_bfloat16*>(a->score_bias);
  p.bias_pos = a->bias_pos;
  p.bias_sectors = reinterpret_cast<uintptr_t>(a->score_bias) % 32 == 0 &&
                   a->bias_stride[0] % 16 == 0 && a->bias_stride[1] % 16 == 0 &&
                   a->bias_stride[2] % 16 == 0;
  for (int i = 0; i < 3; ++i) p.bias_stride[i] = a->bias_stride[i];
  if (p.bias) {
    if (p.paged) return LF_ERR_UNSUPPORTED;
    if (a->bias_pos < 0 || a->bias_pos > a->n_mod) return LF_ERR_INVALID_ARG;
    if (reinterpret_cast<uintptr_t>(a->score_bias) & 15u) return LF_ERR_ALIGNMENT;
    for (int i = 0; i < 3; ++i)
      if (a->bias_stride[i] % 8) return LF_ERR_ALIGNMENT;
  }

  p.q_bias = p.out_bias = nullptr;
  for (int i = 0; i < 3; ++i) p.qb_stride[i] = p.ob_stride[i] = 0;
  if (rows) {
    p.q_bias = static_cast<const __nv_bfloat16*>(rows->q_bias);
    p.out_bias = static_cast<const __nv_bfloat16*>(rows->out_bias);
    if ((reinterpret_cast<uintptr_t>(rows->q_bias) | reinterpret_cast<uintptr_t>(rows->out_bias)) & 15u)
      return LF_ERR_ALIGNMENT;
    for (int i = 0; i < 3; ++i) {
      p.qb_stride[i] = rows->q_bias ? rows->q_bias_stride[i] : 0;
      p.ob_stride[i] = rows->out_bias ? rows->out_bias_stride[i] : 0;
      if (p.qb_stride[i] % 8 || p.ob_stride[i] % 8) return LF_ERR_ALIGNMENT;
    }
  }

  // Pick the score-function mode. Leading and trailing constant multipliers are folded into
  // `a` (before) and `c2` (after); c2 must stay positive for the max-before-scale shortcut.
  int mode = kModeGeneric;
  if (!p.bias) {  // (a score bias splits the chain: kModeBias below, or generic)
    int i = 0;
    float pre = a->scale;
    while (i < a->n_mod && (a->mod_op[i] == LF_MOD_MUL || a->mod_op[i] == LF_MOD_DIV)) {
      pre = a->mod_op[i] == LF_MOD_MUL ? pre * a->mod_arg[i] : pre / a->mod_arg[i];
      ++i;
    }
    if (i == a->n_mod) {
      if (pre > 0.f) {
        mode = kModeNone;
        p.a = 1.f;
        // (Subnormal factors are flushed on the device, and a masked score of -inf times 0 is NaN. The
        // smallest normal number is as near to such a factor as 0 is.)
        p.c2 = fmaxf(pre * kLog2eF, FLT_MIN);
      }
    } else if (a->mod_op[i] == LF_MOD_TANH) {
      int j = i + 1;
      float post = 1.f;
      while (j < a->n_mod && (a->mod_op[j] == LF_MOD_MUL || a->mod_op[j] == LF_MOD_DIV)) {
        post = a->mod_op[j] == LF_MOD_MUL ? post * a->mod_arg[j] : post / a->mod_arg[j];
        ++j;
      }
      if (j == a->n_mod && post > 0.f) {
        p.a = pre;
        p.c2 = post * kLog2eF;
        // |logit2| <= c2: small enough for the fixed softmax reference (the row sum of up to
        // 2^22 terms of at most 2^80 stays far below the fp32 limit).
        // (the fixed-reference kernels read dense K/V; a paged operand goes to the running-max
        // kernel, whose producer warp can gather)
        mode = (p.c2 <= kBoundedMaxC2 && a->Skv <= (1 << 22) && !p.paged) ? kModeBounded
                                                                           : kModeSoftcap;
        const float a2 = p.a * p.a, k0 = p.a * p.c2;
        p.qc[0] = k0;
        p.qc[1] = k0 * a2 * (-1.f / 3.f);
        p.qc[2] = k0 * a2 * a2 * (2.f / 15.f);
        p.qc[3] = k0 * a2 * a2 * a2 * (-17.f / 315.f);
        p.ylim[0] = kTanhPoly1Limit * kTanhPoly1Limit / a2;
        p.ylim[1] = kTanhPoly3Limit * kTanhPoly3Limit / a2;
      }
    }
  }
  if (p.bias && a->bias_pos == a->n_mod) {
    bool plain = true;  // a bias behind multipliers only
    float pre = a->scale;
    for (int i = 0; i < a->n_mod; ++i) {
      if (a->mod_op[i] == LF_MOD_MUL) pre *= a->mod_arg[i];
      else if (a->mod_op[i] == LF_MOD_DIV) pre /= a->mod_arg[i];
      else plain = false;
    }
    if (plain) {
      mode = kModeBias;
      p.a = pre;
      p.c2 = kLog2eF;
    }
  }
  {
    if (mode == kModeGeneric) {
      p.a = a->scale;
      p.c2 = kLog2eF;
      p.mods.n = a->n_mod;
      for (int m = 0; m < a->n_mod; ++m) {
        p.mods.op[m] = a->mod_op[m];
        p.mods.arg[m] = a->mod_arg[m];
      }
    }
  }

  if (has_pe) {
    // The two-product form runs in the plain running-max mode only (scale, then mask).
    if (mode != kModeNone)
      return LF_ERR_UNSUPPORTED;
  }
  if (rows && mode != kModeBias) return LF_ERR_UNSUPPORTED;
  const int kv_tile = choose_kv_tile(a, mode);
  if (kv_tile < 0) return kv_tile;
  // Two or four query heads per kv head under a window mask: the packed layout of the
  // fixed-reference kernel (128 / group query rows of each of the heads per tile slot).
  const int pack = (mode == kModeBounded && kv_tile != kWideK && (p.group == 2 || p.group == 4) &&
                    a->mask_kind == LF_MASK_CAUSAL_WINDOW) ? p.group : 1;
  const int64_t k_row = p.paged & 1 ? gather_row_stride(a->k_stride, a->n_pages, a->page_size, a->Hkv, a->D) : 1;
  const int64_t v_row = p.paged & 2 ? gather_row_stride(a->v_stride, a->n_pages, a->page_size, a->Hkv, a->D) : 1;
  p.gather = p.paged && k_row && v_row;
  auto form_on = [&](int sm_count) {
    return form_of(p, mode, has_pe, a->D, pack, kv_tile, a->B, sm_count);
  };
  if (launch == nullptr) {  // query only
    if (choice) {
      choice->q_tile = kTileQ / pack;
      if (choice->sm_count == 0 && (choice->sm_count = current_sm_count()) == 0) return LF_ERR_CUDA;
      if (choice->sm_count > 0) choice->form = static_cast<int>(form_on(choice->sm_count));
    }
    return kv_tile;
  }
  const int sm_count = current_sm_count();
  if (sm_count == 0) return LF_ERR_CUDA;
  const PrefillForm form = form_on(sm_count);

  CUtensorMap mq, mk, mv;
  int rc = make_tile_map(&mq, a->q, a->B, a->Hq, a->Sq, a->D, a->q_stride, kTileQ / pack);
  if (rc != LF_OK) return rc;
  auto pool_map = [&](CUtensorMap* m, const void* pool, int64_t row_stride, int64_t head_stride) {
    const int64_t st[3] = {0, 0, row_stride};
    return make_tile_map(m, pool, 0, 0, a->n_pages * a->page_size,
                         static_cast<int>((a->Hkv - 1) * head_stride + a->D), st, 1);
  };
  if (p.paged & 1) {
    mk = mq;  // (not used when the producer warp copies the rows of K itself)
    if (p.gather && (rc = pool_map(&mk, a->k, k_row, a->k_stride[2])) != LF_OK) return rc;
  } else {
    rc = make_tile_map(&mk, a->k, a->B, a->Hkv, a->Skv, a->D, a->k_stride, kv_tile);
    if (rc != LF_OK) return rc;
  }
  if (p.paged & 2) {
    mv = mq;
    if (p.gather && (rc = pool_map(&mv, a->v, v_row, a->v_stride[2])) != LF_OK) return rc;
  } else {
    rc = make_tile_map(&mv, a->v, a->B, a->Hkv, a->Skv, a->D, a->v_stride, kv_tile);
    if (rc != LF_OK) return rc;
  }

  CUtensorMap mo;  // output store boxes of the persistent kernels: 32 rows x 32 columns
  if (mode == kModeBounded) {
    rc = make_tile_map(&mo, a->out, a->B, a->Hq, a->Sq, a->D, a->o_stride, 32,
                       (pack > 1 && a->D == 128 && form != PrefillForm::kNarrow) ? 64 : 32);
    if (rc != LF_OK) return rc;
  }

  cudaStream_t st = static_cast<cudaStream_t>(*launch);
  if (has_pe) {
    // Boxes of 64 columns over tensors of D_pe columns: the columns past D_pe arrive as zeros.
    CUtensorMap mqpe, mkpe;
    rc = make_tile_map(&mqpe, a->q_pe, a->B, a->Hq, a->Sq, a->D_pe, a->qpe_stride, kTileQ);
    if (rc != LF_OK) return rc;
    rc = make_tile_map(&mkpe, a->k_pe, a->B, a->Hkv, a->Skv, a->D_pe, a->kpe_stride, kTileK);
    if (rc != LF_OK) return rc;
    if (a->D == 128)
      return launch_prefill<128, kModeNone, true>(mq, mk, mv, p, a->B, st, form, &mqpe, &mkpe);
    return launch_prefill<64, kModeNone, true>(mq, mk, mv, p, a->B, st, form, &mqpe, &mkpe);
  }
  if (a->D == 128) {
    if (mode == kModeNone) return launch_prefill_form<128, kModeNone>(mq, mk, mv, p, a->B, st, form);
    if (mode == kModeSoftcap) return launch_prefill_form<128, kModeSoftcap>(mq, mk, mv, p, a->B, st, form);
    if (mode == kModeBounded)
      return kv_tile == kWideK
               ? launch_prefill_wide<128>(mq, mk, mv, mo, p, a->B, st, sm_count)
               : launch_prefill_bounded_form<128>(mq, mk, mv, mo, p, a->B, st, pack, form, sm_count);
    if (mode == kModeBias) return launch_prefill_form<128, kModeBias>(mq, mk, mv, p, a->B, st, form);
    return launch_prefill_form<128, kModeGeneric>(mq, mk, mv, p, a->B, st, form);
  }
  if (mode == kModeNone) return launch_prefill_form<64, kModeNone>(mq, mk, mv, p, a->B, st, form);
  if (mode == kModeSoftcap) return launch_prefill_form<64, kModeSoftcap>(mq, mk, mv, p, a->B, st, form);
  if (mode == kModeBounded)
    return kv_tile == kWideK
               ? launch_prefill_wide<64>(mq, mk, mv, mo, p, a->B, st, sm_count)
               : launch_prefill_bounded_form<64>(mq, mk, mv, mo, p, a->B, st, pack, form, sm_count);
  if (mode == kModeBias) return launch_prefill_form<64, kModeBias>(mq, mk, mv, p, a->B, st, form);
  return launch_prefill_form<64, kModeGeneric>(mq, mk, mv, p, a->B, st, form);
}

}  // namespace lf

extern "C" {

int lf_prefill_bf16(const LfPrefillArgs* args, void* stream) {
  return lf::prefill_impl(args, &stream);
}

int lf_prefill_row_bias_bf16(const LfPrefillArgs* args, const LfRowBias* rows, void* stream) {
  if (!rows || (!rows->q_bias && !rows->out_bias)) return LF_ERR_INVALID_ARG;
  return lf::prefill_impl(args, &stream, nullptr, rows);
}

int lf_prefill_kv_tile(const LfPrefillArgs* args) { return lf::prefill_impl(args, nullptr); }

int lf_prefill_q_tile(const LfPrefillArgs* args) {
  lf::PrefillChoice choice;
  choice.sm_count = -1;
  const int rc = lf::prefill_impl(args, nullptr, &choice);
  return rc < 0 ? rc : choice.q_tile;
}

int lf_prefill_form(const LfPrefillArgs* args, int32_t sm_count) {
  if (sm_count < 0) return LF_ERR_INVALID_ARG;
  lf::PrefillChoice choice;
  choice.sm_count = sm_count;
  const int rc = lf::prefill_impl(args, nullptr, &choice);
  return rc < 0 ? rc : choice.form;
}

void lf_tile_map_cache_stats(uint64_t* hits, uint64_t* misses) {
  if (hits) *hits = lf::g_tile_map_hits.load();
  if (misses) *misses = lf::g_tile_map_misses.load();
}

void lf_skip_range(int32_t mask_kind, int32_t window, int32_t causal_offset, int32_t Sq,
                   int32_t Skv, int32_t tile_q, int32_t tile_k, int32_t iq, int32_t* lo,
                   int32_t* hi) {
  lf::skip_range(mask_kind, window, causal_offset, Sq, Skv, tile_q, tile_k, iq, lo, hi);
}

}  // extern "C"
