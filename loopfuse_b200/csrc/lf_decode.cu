// Decode attention for sm_100a: one query row per head, KV streamed once from HBM.
//
// Bandwidth-bound, so the work is laid out to keep many bytes in flight:
//   * a CTA owns one (batch, kv head, KV split); its warps take alternate 16-token groups of the
//     split, each group's K and V rows travelling global -> shared with 16-byte cp.async into a ring
//     private to the warp, so the bytes in flight do not cost registers;
//   * the G query heads that share the kv head are the M dimension of tensor-core products (see
//     decode_mma_kernel), softmax is online in the log2 domain;
//   * with splits > 1 the CTAs of a (batch, kv head) form a thread-block cluster and merge their
//     un-normalised partials (acc, max, sum) through distributed shared memory (log-sum-exp
//     combine); where they cannot (more splits than a cluster holds, grids of many waves, or a device
//     that cannot hold the cluster), each CTA writes its partial to the workspace and lf_combine
//     merges them;
//   * the paged variant stages its slice of the block table through shared memory, checks
//     every page id against the pool size (status word, clamped, never a trap) and turns
//     (page, slot) into row pointers.
#include "lf_common.cuh"

#include <cooperative_groups.h>
#include <math.h>

#include <mutex>
#include <type_traits>

namespace lf {

constexpr float kLog2e = 1.4426950408889634f;

struct DecodeParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  __nv_bfloat16* out;
  float* part_o;   // [units, splits, D]
  float* part_ml;  // [units, splits, 2]
  const int32_t* block_table;
  const int32_t* block_table_v;  // never null for the paged kernel (may equal block_table)
  int32_t* status;
  int64_t q_stride[3], o_stride[3], k_stride[3], v_stride[3];
  int64_t bt_stride;
  int32_t B, Hkv, Skv, splits, chunk;  // chunk = tokens per split
  int32_t page_size, page_shift, n_pages;  // page_shift >= 0 when page_size is 2^shift
  float scale;
  float cap;        // kModsSoftcap: logit2 = tanh(scale * dot) * cap (log2(e) included)
  int32_t cluster;  // the splits of a unit are one cluster and merge among themselves
  int32_t part_off; // ... through partials at this byte of shared memory (the same in all of them)
  ModChain mods;
};

// Score function of a decode kernel. Softcap has a form of its own: the interpreted chain is a
// switch per score and op, mostly instruction-cache misses in a launch of a few microseconds.
constexpr int kModsNone = 0, kModsSoftcap = 1, kModsGeneric = 2;

// Dot product (scaled by log2(e) * scale already when MODS == kModsNone) -> logit in the log2 domain.
template <int MODS>
__device__ __forceinline__ float decode_logit2(const DecodeParams& p, float d) {
  if constexpr (MODS == kModsSoftcap) return tanh_approx(d) * p.cap;
  else if constexpr (MODS == kModsGeneric) return apply_mods(p.mods, d) * kLog2e;
  else return d;
}

// Merge the partials of a unit's splits within their cluster. `mine` (shared memory of every CTA of
// the cluster, at the same offset): [G][D + 2] un-normalised output, max, sum. Each CTA finishes a
// slice of the G * D outputs. A launch less than the combine kernel, and no round trip of the
// partials through global memory (one sequence, 8 kv heads x 4, 8190 keys: 4.7 us for the combine).
template <int D>
__device__ __forceinline__ void merge_in_cluster(const DecodeParams& p, float* mine, int G, int b,
                                                 int kvh, int threads) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int rank = static_cast<int>(cluster.block_rank());
  constexpr int kStride = D + 2;
  for (int idx = rank * threads + threadIdx.x; idx < G * D; idx += p.splits * threads) {
    const int g = idx / D, c = idx - g * D;
    float m_all = -INFINITY;
    for (int r = 0; r < p.splits; ++r)
      m_all = fmaxf(m_all, cluster.map_shared_rank(mine, r)[g * kStride + D]);
    const float m_safe = (m_all == -INFINITY) ? 0.f : m_all;
    float l_all = 0.f, o = 0.f;
#pragma unroll 4
    for (int r = 0; r < p.splits; ++r) {
      const float* src = cluster.map_shared_rank(mine, r) + g * kStride;
      const float a = ex2_approx(src[D] - m_safe);
      l_all += src[D + 1] * a;
      o += src[c] * a;
    }
    __nv_bfloat16* op = p.out + b * p.o_stride[0] + kvh * p.o_stride[1] + g * p.o_stride[2];
    op[c] = __float2bfloat16_rn(o / l_all);
  }
  cluster.sync();  // (nobody leaves while its shared memory is being read)
}

// ---------------------------------------------------------------------------------------
// Decode on tensor cores (mma.sync m16n8k16, bf16 -> fp32).
//
// The G query rows of a kv head are rows 0..7 (zero-padded) of the 16-row M dimension of 16x8x16
// MMAs; rows 8..15 are padding in QK^T. The fragments come straight from the 16-byte pieces that were
// copied:
//
//   QK^T  8 tokens at a time. Lane (n = lane/4, c = lane%4) loads the 16-byte pieces
//         d = 32i + 8c .. +8 of token n's K row (i < D/32); the four 32-bit words of a piece
//         are exactly the B fragments of two MMAs (a dot product does not care in which order
//         the d's are visited as long as Q uses the same order, and Q is loaded with the same
//         pattern, row g = lane/4 instead of token n).
//   PV    16 tokens at a time. Lane (n, c) loads rows 2c, 2c+1, 2c+8, 2c+9 at d = 64h + 8n ..
//         +8; a byte permute of two rows gives the {V[2c][d], V[2c+1][d]} pairs the B fragment
//         wants; output column n of MMA (h, e) stands for d = 64h + 8n + e.
//   The fp32 score fragment of the QK MMAs has the layout of the bf16 A fragment of the PV
//   MMA, so P never leaves registers.
//   P enters the PV product as the sum of P_TERMS bf16, in rows that would be padding and at no extra
//   MMA: rows g take its rounding, rows 8 + g the rounding of the rest; with three (dense calls with
//   G <= 2, whose former FMA kernel had P in fp32) rows 2 + g, whose Q rows repeat rows g, what that
//   leaves. With one, P's rounding error is a fifth of the result's and depends on how the keys are
//   dealt out to warps and splits (the largest P of each is exactly 1); with two the result's error is
//   that of its own rounding. Against fp64, 1 x 8 x 4 heads, 8190 keys, softcap: 2.05e-3 in 31 splits,
//   2.08e-3 in 16, now 1.66e-3; 64 x 8 x 4, 2048 keys, paged: 2.22e-3 -> 1.66e-3 at 87.0 -> 86.7 us.
// A CTA is one (batch, kv head, KV split); its WARPS warps (launch_decode_shape says how many) take
// alternate 16-token groups (one page when page_size is 16) and are merged through shared memory.
// Against the FMA + shuffle form that dense calls with G <= 2 used (B200, D = 128): B=64 Hkv=32 2048 keys
// 318 -> 307 us, B=1 Hkv=32 4096 keys 20.3 -> 16.8 us, B=1 Hkv=4 G=2 16000 keys 27.9 -> 16.4 us, B=16
// Hkv=32 1000 keys 45.0 -> 46.3 us.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_16816_rows0to7(float& d0, float& d1, uint32_t a0, uint32_t a2,
                                                   uint32_t b0, uint32_t b1) {
  [[maybe_unused]] float unused2, unused3;  // rows 8..15 of the tile are padding
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %10, %11};"
      : "+f"(d0), "+f"(d1), "=f"(unused2), "=f"(unused3)
      : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.f), "f"(0.f));
}

// The same with all sixteen rows.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// STAGES: depth of a warp's ring in 16-token groups; STAGES - 1 are in flight.
template <int D, bool PAGED, int MODS, int WARPS, int STAGES, int P_TERMS>
__global__ void __launch_bounds__(WARPS * 32, (STAGES == 3 ? 8 : 12) / WARPS)
    decode_mma_kernel(const DecodeParams p, const int G) {
  pdl_wait();
  constexpr int KI = D / 32;  // 16-byte pieces of a K row per lane
  constexpr int VH = D / 64;  // 64-wide halves of a V row
  constexpr int NT = D / 8;   // output n-tiles (8 columns each)

  const int split = blockIdx.x;
  const int kvh = blockIdx.y;
  const int b = blockIdx.z;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;  // query row of this lane's score / output fragment; token index n
  const int c = lane & 3;

  const int t0 = split * p.chunk;
  const int t1 = min(p.Skv, t0 + p.chunk);

  extern __shared__ __align__(128) unsigned char smem_raw[];
  int32_t* s_pages_k = reinterpret_cast<int32_t*>(smem_raw);
  int32_t* s_pages_v = s_pages_k;
  int first_page = 0;
  size_t merge_off = 0;
  auto page_of = [&](int t) { return p.page_shift >= 0 ? (t >> p.page_shift) : (t / p.page_size); };
  if constexpr (PAGED) {
    int n_pages_local = 0;
    if (t1 > t0) {
      first_page = page_of(t0);
      n_pages_local = page_of(t1 - 1) - first_page + 1;
    }
    const bool two_tables = p.block_table_v != p.block_table;
    // The rings start on a 128-byte line: 16 bytes off it, a row's copy writes three lines instead of
    // two (192 units of 1200 keys 34.4 -> 25 us).
    const int pages_pad = (n_pages_local + 31) & ~31;
    if (two_tables) s_pages_v = s_pages_k + pages_pad;
    merge_off = static_cast<size_t>(pages_pad) * 4 * (two_tables ? 2 : 1);
    for (int which = 0; which < (two_tables ? 2 : 1); ++which) {
      const int32_t* bt = (which == 0 ? p.block_table : p.block_table_v) +
                          static_cast<int64_t>(b) * p.bt_stride + first_page;
      int32_t* dst = which == 0 ? s_pages_k : s_pages_v;
      for (int i = threadIdx.x; i < n_pages_local; i += (WARPS * 32)) {
        int32_t pg = bt[i];
        if (pg < 0 || pg >= p.n_pages) {
          if (p.status) atomicExch(p.status, LF_DEV_BAD_PAGE);
          pg = 0;
        }
        dst[i] = pg;
      }
    }
    __syncthreads();
  }
  float* s_merge = reinterpret_cast<float*>(smem_raw + merge_off);

  // Row pointers of token t for this lane's kv head.
  const __nv_bfloat16* kbase;
  const __nv_bfloat16* vbase;
  if constexpr (PAGED) {
    kbase = p.k + kvh * p.k_stride[2];
    vbase = p.v + kvh * p.v_stride[2];
  } else {
    kbase = p.k + b * p.k_stride[0] + kvh * p.k_stride[1];
    vbase = p.v + b * p.v_stride[0] + kvh * p.v_stride[1];
  }
  [[maybe_unused]] const int n_pages_staged =
      (PAGED && t1 > t0) ? page_of(t1 - 1) - first_page + 1 : 0;
  auto k_row = [&](int t) -> const __nv_bfloat16* {
    if (!LF_BOUNDS(t >= t0 && t < t1 && t < p.Skv, p.status, 42)) t = t0;
    if constexpr (PAGED) {
      const int pg_abs = page_of(t);
      const int slot = t - pg_abs * p.page_size;
      if (!LF_BOUNDS(pg_abs - first_page >= 0 && pg_abs - first_page < n_pages_staged,
                     p.status, 43))
        return kbase;
      return kbase + static_cast<int64_t>(s_pages_k[pg_abs - first_page]) * p.k_stride[0] +
             slot * p.k_stride[1];
    } else {
      return kbase + t * p.k_stride[2];
    }
  };
  auto v_row = [&](int t) -> const __nv_bfloat16* {
    if (!LF_BOUNDS(t >= t0 && t < t1 && t < p.Skv, p.status, 44)) t = t0;
    if constexpr (PAGED) {
      const int pg_abs = page_of(t);
      const int slot = t - pg_abs * p.page_size;
      if (!LF_BOUNDS(pg_abs - first_page >= 0 && pg_abs - first_page < n_pages_staged,
                     p.status, 45))
        return vbase;
      return vbase + static_cast<int64_t>(s_pages_v[pg_abs - first_page]) * p.v_stride[0] +
             slot * p.v_stride[1];
    } else {
      return vbase + t * p.v_stride[2];
    }
  };

  // Q fragments (rows g >= G are zero padding; three parts of P: rows 2 and 3 are rows 0 and 1 again).
  const int q_row = P_TERMS == 3 && g < 4 ? (g & 1) : g;
  auto chunk_of = [&](int i) { return 4 * i + c; };  // 16-byte piece of a row
  uint4 qr[KI];
#pragma unroll
  for (int i = 0; i < KI; ++i) {
    qr[i] = make_uint4(0u, 0u, 0u, 0u);
    if (q_row < G)
      qr[i] = *reinterpret_cast<const uint4*>(p.q + b * p.q_stride[0] + kvh * p.q_stride[1] +
                                              q_row * p.q_stride[2] + 8 * chunk_of(i));
  }
  const float smul = MODS != kModsNone ? p.scale : p.scale * kLog2e;

  float m_run = -INFINITY, l_run = 0.f;
  float o[NT][4];  // rows g, then rows 8 + g
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;

  // K/V rows travel global -> shared with 16-byte cp.async into a ring private to the warp
  // (STAGES groups of 16 tokens; STAGES-1 groups are in flight while one is consumed),
  // so the bytes in flight do not cost registers. The 16-byte piece j of row r sits at piece j ^ (r & 7):
  // fragment reads of eight different rows then hit distinct banks. (One 256-byte bulk copy per row is
  // an instruction per lane and group, but the SM takes them at 11 ns each: 64 units of 8190 keys 101
  // -> 190 us.)
  constexpr int CPR = D / 8;         // 16-byte pieces per row
  constexpr int RPI = 32 / CPR;      // rows that one instruction of the warp copies
  constexpr int kRowBytes = D * 2;
  constexpr int kStageBytes = 2 * 16 * kRowBytes;  // 16 K rows then 16 V rows
  const int t_last = t1 - 1;
  unsigned char* ring = smem_raw + merge_off + warp * (STAGES * kStageBytes);
  const int r0 = lane / CPR, j0 = lane % CPR;
  const uint32_t ring_u32 = smem_u32(ring) + r0 * kRowBytes;
  const int64_t ks = PAGED ? p.k_stride[1] : p.k_stride[2];
  const int64_t vs = PAGED ? p.v_stride[1] : p.v_stride[2];
  auto copy_group = [&](int tg, int stage) {
    if (tg < t1) {
      const uint32_t dst = ring_u32 + stage * kStageBytes;
      // A whole group that lies inside one page (always true for dense caches) has affine row
      // addresses: one table lookup per group instead of one per row.
      bool affine = tg + 15 <= t_last;
      if constexpr (PAGED) affine = affine && page_of(tg) == page_of(tg + 15);
      if (!LF_BOUNDS(stage >= 0 && stage < STAGES, p.status, 46)) {
      } else if (affine) {
        const __nv_bfloat16* kp = k_row(tg) + r0 * ks + 8 * j0;
        const __nv_bfloat16* vp = v_row(tg) + r0 * vs + 8 * j0;
#pragma unroll
        for (int q = 0; q < 16 / RPI; ++q) {
          const uint32_t to = dst + q * RPI * kRowBytes + ((j0 ^ ((r0 + q * RPI) & 7)) << 4);
          cp_async_16(to, kp);
          cp_async_16(to + 16 * kRowBytes, vp);
          kp += RPI * ks;
          vp += RPI * vs;
        }
      } else {
        // Rows that pages scatter: lane r < 16 finds K row r of the group, lane 16 + r V row r, and the
        // lanes that copy a row get its place by shuffle (416 units of 6443 one-token pages 300 -> 217 us
        // against every lane looking up every row that it copies). Rows past the end of the split
        // re-read its last token.
        const int tok = min(tg + (lane & 15), t_last);
        const int64_t off = lane < 16 ? k_row(tok) - kbase : v_row(tok) - vbase;
#pragma unroll
        for (int q = 0; q < 16 / RPI; ++q) {
          const int r = r0 + q * RPI;
          const uint32_t to = dst + q * RPI * kRowBytes + ((j0 ^ (r & 7)) << 4);
          cp_async_16(to, kbase + __shfl_sync(0xffffffffu, off, r) + 8 * j0);
          cp_async_16(to + 16 * kRowBytes, vbase + __shfl_sync(0xffffffffu, off, 16 + r) + 8 * j0);
        }
      }
    }
    cp_async_commit();
  };
  const int tg0 = t0 + warp * 16;
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) copy_group(tg0 + st * 16 * WARPS, st);

  int it = 0;
  for (int tg = tg0; tg < t1; tg += 16 * WARPS, ++it) {
    copy_group(tg + (STAGES - 1) * 16 * WARPS, (it + STAGES - 1) % STAGES);
    cp_async_wait<STAGES - 1>();
    __syncwarp();
    const unsigned char* stage = ring + (it % STAGES) * kStageBytes;
    // K: token n = g of each 8-token half; V: rows 2c, 2c+1, 2c+8, 2c+9 of the 16-token group.
    uint4 kr[2][KI];
#pragma unroll
    for (int s8 = 0; s8 < 2; ++s8)
#pragma unroll
      for (int i = 0; i < KI; ++i)
        kr[s8][i] =
            *reinterpret_cast<const uint4*>(stage + (8 * s8 + g) * kRowBytes + ((chunk_of(i) ^ g) << 4));

    // Scores of the two 8-token halves: this lane ends up with tokens 2c, 2c+1 of each.
    // (two accumulators each: half the chain of dependent MMAs)
    float sc[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, sc_b[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
    for (int s8 = 0; s8 < 2; ++s8)
#pragma unroll
      for (int i = 0; i < KI; ++i) {
        mma_16816_rows0to7(sc[s8][0], sc[s8][1], qr[i].x, qr[i].y, kr[s8][i].x, kr[s8][i].y);
        mma_16816_rows0to7(sc_b[s8][0], sc_b[s8][1], qr[i].z, qr[i].w, kr[s8][i].z, kr[s8][i].w);
      }
    float mx = -INFINITY;
#pragma unroll
    for (int s8 = 0; s8 < 2; ++s8)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float v = decode_logit2<MODS>(p, (sc[s8][e] + sc_b[s8][e]) * smul);
        if (tg + 8 * s8 + 2 * c + e >= t1) v = -INFINITY;
        sc[s8][e] = v;
        mx = fmaxf(mx, v);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx);
    const float m_safe = (m_new == -INFINITY) ? 0.f : m_new;
    if (__any_sync(0xffffffffu, m_new > m_run)) {  // (a new maximum becomes rare after a few groups)
      const float alpha = ex2_approx(m_run - m_safe);
      m_run = m_new;
      l_run *= alpha;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] *= alpha;
    }
    float pr[2][2];
    float psum = 0.f;
#pragma unroll
    for (int s8 = 0; s8 < 2; ++s8)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        pr[s8][e] = ex2_approx(sc[s8][e] - m_safe);
        psum += pr[s8][e];
      }
    l_run += psum;  // this lane's share; the quad is summed after the loop
    uint32_t pa0 = pack_bf16x2(pr[0][0], pr[0][1]);
    uint32_t pa2 = pack_bf16x2(pr[1][0], pr[1][1]);
    const float r0 = pr[0][0] - bf16lo_to_f32(pa0), r1 = pr[0][1] - bf16hi_to_f32(pa0);
    const float r2 = pr[1][0] - bf16lo_to_f32(pa2), r3 = pr[1][1] - bf16hi_to_f32(pa2);
    uint32_t pa1 = pack_bf16x2(r0, r1);
    uint32_t pa3 = pack_bf16x2(r2, r3);
    if constexpr (P_TERMS == 3) {
      if (g >= 2) {
        pa0 = pack_bf16x2(r0 - bf16lo_to_f32(pa1), r1 - bf16hi_to_f32(pa1));
        pa2 = pack_bf16x2(r2 - bf16lo_to_f32(pa3), r3 - bf16hi_to_f32(pa3));
        pa1 = pa3 = 0u;
      }
    }
#pragma unroll
    for (int h = 0; h < VH; ++h) {
      uint4 vq[4];
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int r = 2 * c + (r4 & 1) + 8 * (r4 >> 1);
        vq[r4] = *reinterpret_cast<const uint4*>(stage + (16 + r) * kRowBytes +
                                                 (((8 * h + g) ^ (r & 7)) << 4));
      }
      const uint32_t w0[4] = {vq[0].x, vq[0].y, vq[0].z, vq[0].w};
      const uint32_t w1[4] = {vq[1].x, vq[1].y, vq[1].z, vq[1].w};
      const uint32_t w2[4] = {vq[2].x, vq[2].y, vq[2].z, vq[2].w};
      const uint32_t w3[4] = {vq[3].x, vq[3].y, vq[3].z, vq[3].w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t sel = (e & 1) ? 0x7632u : 0x5410u;  // high or low halves of two words
        const uint32_t b0 = __byte_perm(w0[e >> 1], w1[e >> 1], sel);
        const uint32_t b1 = __byte_perm(w2[e >> 1], w3[e >> 1], sel);
        mma_16816(o[h * 8 + e], pa0, pa1, pa2, pa3, b0, b1);
      }
    }
    __syncwarp();  // every lane is done with this stage before it is refilled
  }
  cp_async_wait<0>();
  // (Not earlier: the next launch's CTAs would take the places that this one's leave as they come,
  // and crowd on some SMs: 512 units of 2048 keys take 8 % longer with the trigger at the top.)
  pdl_trigger();

  // Rows 8 + g (same lane), and with three parts rows 2 + g, hold the finer parts of row g.
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float fine = o[j][2 + e];
      if constexpr (P_TERMS == 3) fine += __shfl_down_sync(0xffffffffu, o[j][e], 8);
      // (a value row with an infinity: the parts of its weight have either sign or are zero)
      if (fabsf(o[j][e]) != INFINITY) o[j][e] += fine;
    }
  // Row sum over the quad (the four lanes of a row hold disjoint tokens).
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);

  // Merge the warps through shared memory: s_merge[warp][g][0..D) acc, then m, l. The merge
  // area reuses the rings, so every warp must have finished reading its last stage.
  constexpr int kStride = D + 2;
  __syncthreads();
  if (g < G) {
    float* dst = s_merge + (warp * G + g) * kStride;
#pragma unroll
    for (int h = 0; h < VH; ++h)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        dst[64 * h + 16 * c + e] = o[h * 8 + e][0];      // output column 2c   -> d = 64h+16c+e
        dst[64 * h + 16 * c + 8 + e] = o[h * 8 + e][1];  // output column 2c+1 -> d + 8
      }
    if (c == 0) {
      dst[D] = m_run;
      dst[D + 1] = l_run;
    }
  }
  __syncthreads();

  for (int idx = threadIdx.x; idx < G * D; idx += (WARPS * 32)) {
    const int gg = idx / D;
    const int cc = idx - gg * D;
    float m_all = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w)
      m_all = fmaxf(m_all, s_merge[(w * G + gg) * kStride + D]);
    const float m_safe = (m_all == -INFINITY) ? 0.f : m_all;
    float l_all = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float* src = s_merge + (w * G + gg) * kStride;
      const float a = ex2_approx(src[D] - m_safe);
      l_all += src[D + 1] * a;
      acc += src[cc] * a;
    }
    const int64_t unit = (static_cast<int64_t>(b) * p.Hkv + kvh) * G + gg;
    if (!LF_BOUNDS(gg < G && cc < D && b < p.B && kvh < p.Hkv && split < p.splits, p.status, 47))
      continue;
    if (p.cluster) {
      float* mine = reinterpret_cast<float*>(smem_raw + p.part_off) + gg * kStride;
      mine[cc] = acc;
      if (cc == 0) {
        mine[D] = m_all;
        mine[D + 1] = l_all;
      }
    } else if (p.splits == 1) {
      __nv_bfloat16* op = p.out + b * p.o_stride[0] + kvh * p.o_stride[1] + gg * p.o_stride[2];
      op[cc] = __float2bfloat16_rn(acc / l_all);
    } else {
      p.part_o[(unit * p.splits + split) * D + cc] = acc;
      if (cc == 0) {
        p.part_ml[(unit * p.splits + split) * 2] = m_all;
        p.part_ml[(unit * p.splits + split) * 2 + 1] = l_all;
      }
    }
  }
  if (p.cluster)
    merge_in_cluster<D>(p, reinterpret_cast<float*>(smem_raw + p.part_off), G, b, kvh, WARPS * 32);
}

// Log-sum-exp combine of split-KV partials: one warp per (batch, kv head, g) output row.
template <int D>
__global__ void __launch_bounds__(128)
    combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                   __nv_bfloat16* __restrict__ out, int64_t units, int32_t Hkv, int32_t G,
                   int32_t splits, int64_t os0, int64_t os1, int64_t os2) {
  pdl_trigger();
  pdl_wait();
  constexpr int EPL = D / 32;  // elements per lane
  const int64_t unit = static_cast<int64_t>(blockIdx.x) * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (unit >= units) return;
  // Lane s owns split s (at most 32 splits): one load round for all (max, sum) pairs, the
  // weights are then broadcast from their lanes while the partial rows stream in.
  const float* ml = part_ml + unit * splits * 2;
  float m_s = -INFINITY, l_s = 0.f;
  if (lane < splits) {
    const float2 v = *reinterpret_cast<const float2*>(ml + 2 * lane);
    m_s = v.x;
    l_s = v.y;
  }
  float m_all = m_s;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1)
    m_all = fmaxf(m_all, __shfl_xor_sync(0xffffffffu, m_all, off));
  const float m_safe = (m_all == -INFINITY) ? 0.f : m_all;
  const float w_s = ex2_approx(m_s - m_safe);
  float l_all = l_s * w_s;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) l_all += __shfl_xor_sync(0xffffffffu, l_all, off);
  float o[EPL];
#pragma unroll
  for (int e = 0; e < EPL; ++e) o[e] = 0.f;
  const float* src0 = part_o + unit * splits * D + lane * EPL;
  for (int s0 = 0; s0 < splits; s0 += 4) {
    float x[4][EPL];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int s = min(s0 + u, splits - 1);
      if constexpr (EPL == 4) {
        const float4 v = *reinterpret_cast<const float4*>(src0 + s * D);
        x[u][0] = v.x; x[u][1] = v.y; x[u][2] = v.z; x[u][3] = v.w;
      } else {
        const float2 v = *reinterpret_cast<const float2*>(src0 + s * D);
        x[u][0] = v.x; x[u][1] = v.y;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float a = (s0 + u < splits) ? __shfl_sync(0xffffffffu, w_s, (s0 + u) & 31) : 0.f;
#pragma unroll
      for (int e = 0; e < EPL; ++e) o[e] += x[u][e] * a;
    }
  }
  const float inv = 1.f / l_all;
  const int64_t g = unit % G;
  const int64_t h = (unit / G) % Hkv;
  const int64_t bb = unit / G / Hkv;
  __nv_bfloat16* op = out + bb * os0 + h * os1 + g * os2 + lane * EPL;
  if constexpr (EPL == 4) {
    uint2 w;
    w.x = pack_bf16x2(o[0] * inv, o[1] * inv);
    w.y = pack_bf16x2(o[2] * inv, o[3] * inv);
    *reinterpret_cast<uint2*>(op) = w;
  } else {
    *reinterpret_cast<uint32_t*>(op) = pack_bf16x2(o[0] * inv, o[1] * inv);
  }
}

// out[b, h, t, :] = pool[block_table[b, t / P], t % P, h, :]; one warp-row group per token.
template <int D>
__global__ void __launch_bounds__(256)
    paged_gather_kernel(const __nv_bfloat16* __restrict__ pool,
                        const int32_t* __restrict__ block_table, __nv_bfloat16* __restrict__ out,
                        int32_t B, int32_t Hkv, int32_t Skv, int32_t page_size, int32_t n_pages,
                        int64_t ps0, int64_t ps1, int64_t ps2, int64_t bt_stride,
                        int32_t* status) {
  constexpr int LPR = D / 8;
  const int64_t gid = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  const int64_t row = gid / LPR;
  const int col = static_cast<int>(gid % LPR);
  const int64_t total_rows = static_cast<int64_t>(B) * Hkv * Skv;
  if (row >= total_rows) return;
  const int t = static_cast<int>(row % Skv);
  const int h = static_cast<int>((row / Skv) % Hkv);
  const int b = static_cast<int>(row / Skv / Hkv);
  int32_t pg = block_table[b * bt_stride + t / page_size];
  if (pg < 0 || pg >= n_pages) {
    if (status) atomicExch(status, LF_DEV_BAD_PAGE);
    pg = 0;
  }
  const int slot = t % page_size;
  const uint4 x = *reinterpret_cast<const uint4*>(pool + pg * ps0 + slot * ps1 + h * ps2 + col * 8);
  *reinterpret_cast<uint4*>(out + row * D + col * 8) = x;
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
static int device_sm_count() {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev != cached_dev) {
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    cached_dev = dev;
  }
  return cached > 0 ? cached : 148;
}

static int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Shared memory the tensor-core kernel may spend on block-table slices (both tables), so that
// two CTAs (K/V rings of 96 KB each at D = 128) still fit on one SM.
constexpr size_t kMaxTableBytes = 16 * 1024;

static size_t table_smem_bytes(int chunk, int page_size) {
  // Room for the K table and a separate V table, each padded to 128 bytes.
  return 2 * (((static_cast<size_t>(chunk / page_size) + 2 + 31) & ~size_t(31)) * 4);
}

// Largest token chunk of one split whose block-table slice fits (paged caches only).
static int max_chunk_for_table(int page_size) {
  const int entries = static_cast<int>(kMaxTableBytes / 8) - 34;  // per table, minus padding
  const int64_t tokens = static_cast<int64_t>(entries) * page_size;
  return static_cast<int>(tokens > (1 << 30) ? (1 << 30) : tokens / 64 * 64);
}

constexpr int kMaxCluster = 16;  // (more than 8 CTAs: a non-portable cluster size)

// Split count for splits == 0. page_size: 0 for a dense cache, else the tokens per page. Powers of
// two only: clusters of other sizes are placed badly (16 x 8 units of 1001 keys took 18.5 us in twos,
// 22 in threes, 20 in fours, 33 in sixes; 8 x 4 units of 4000 keys 20.4 us in eights, 29 in nines).
static int choose_splits(int B, int Hkv, int Skv, int D, int page_size) {
  const int64_t units = static_cast<int64_t>(B) * Hkv;
  const int sms = device_sm_count();
  constexpr int kMinTokens = 120;  // per split: below, its start-up costs what the split saves
  // As many CTAs as one wave of one per SM takes. (Two per SM gain nothing over that: 64 units of 8190
  // keys 47 us in twos, 49 in fours, 49 in eights.) Sixteen-CTA clusters only where one fits in every
  // GPC: 16 units of 8190 keys 22.6 us in eights, 28.6 in sixteens.
  int s = 1;
  while (s < kMaxCluster && units * s * 2 <= sms && Skv / (s * 2) >= kMinTokens) s *= 2;
  // If that leaves 40 % of the SMs without work, four times as many smaller ones: 40 units of 8190
  // keys 39 us in twos, 37 in eights; of 3001 keys 24 and 20.
  if (units * s * 5 < 3ll * sms && s <= 4 && Skv / (s * 4) >= kMinTokens &&
      units * s * 4 >= 2ll * sms)
    s = s == 4 ? 8 : s * 4;
  // A dense grid of many waves gains from halves where the caches are long and rows are 256 bytes: its
  // last wave is shorter (D = 128, 2048 units of 2048 keys 309 -> 304 us, of 3000 445 -> 438, 1024 of 4000
  // 303 -> 300; of 1000 keys 170 -> 173 us; D = 64, 2048 of 2048 156 -> 161; paged 314 -> 322).
  if (page_size == 0 && D == 128 && units >= 6ll * sms + sms / 2 && Skv >= 2000) s = 2;
  if (page_size > 0) {
    // The block-table slice of a split must fit in shared memory (one-token pages at long
    // context): split further until it does.
    const int max_chunk = max_chunk_for_table(page_size);
    while (s < 32 && round_up((Skv + s - 1) / s, 16) > max_chunk) s = s < 16 ? s * 2 : s + 1;
  }
  return s;
}

// Splits whose partials go through the workspace when `splits` are asked for: chunks of 64 tokens, and
// none that is empty. Never more than were asked for, and what a workspace has to hold.
static int partial_chunk(int Skv, int splits) { return round_up((Skv + splits - 1) / splits, 64); }
static int partial_splits(int Skv, int splits) {
  const int chunk = partial_chunk(Skv, splits);
  return (Skv + chunk - 1) / chunk;
}

// Launch with the splits of a unit as a cluster, when p.cluster says so.
template <class Kernel, class... Args>
static cudaError_t launch_splits(Kernel kernel, const DecodeParams& p, int threads, size_t smem,
                                 cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.splits, p.Hkv, p.B);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (p.cluster) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = p.splits;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  // Large grids wait for the kernel before them to leave the SMs: their CTAs are then dealt out
  // evenly (512 units of 2048 keys take 2 % longer when they start between another launch's last ones).
  if (static_cast<int64_t>(p.splits) * p.Hkv * p.B <= 2ll * device_sm_count()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Per kernel, thread and device: shared memory beyond 48 KB and clusters beyond 8 CTAs are opted in to.
template <class Kernel>
static int configure_decode(Kernel kernel, int smem, int& configured_dev) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev == dev) return LF_OK;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) {
    set_cuda_error(e, "cudaFuncSetAttribute(decode kernel)");
    return LF_ERR_CUDA;
  }
  configured_dev = dev;
  return LF_OK;
}

// What launch_decode returns when the device cannot hold a cluster of a call's splits.
constexpr int kNoCluster = 1;

// Whether a cluster of `splits` CTAs can be resident at all. Sixteens of this size can on a whole B200,
// but not on every part of one (fewer SMs per GPC); the combine kernel serves the others. Asked
// once per kernel, thread and device for each cluster size, with the most shared memory it uses.
struct ClusterFit {
  int dev = -1;
  uint32_t known = 0, fits = 0;  // bit s: clusters of s
};
template <class Kernel>
static bool cluster_fits(Kernel kernel, int splits, int threads, size_t smem, ClusterFit& cache) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (cache.dev != dev) cache = ClusterFit{dev, 0, 0};
  const uint32_t bit = 1u << splits;
  if (!(cache.known & bit)) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    cache.known |= bit;
    if (n > 0) cache.fits |= bit;
  }
  return (cache.fits & bit) != 0;
}

static int launched(cudaError_t e, const char* where) {
  if (e == cudaSuccess) return check_launch(where);
  cudaGetLastError();
  set_cuda_error(e, where);
  return LF_ERR_CUDA;
}

// (`st` null: nothing is launched, only a cluster that cannot be is told.)
template <int D, bool PAGED, int MODS, int P_TERMS, int WARPS, int STAGES>
static int launch_decode_w(DecodeParams p, int G, const cudaStream_t* st, size_t table_bytes) {
  // page ids + the per-warp K/V rings (the warp-merge area and the partial reuse the rings)
  constexpr size_t ring = static_cast<size_t>(WARPS) * STAGES * 2 * 16 * D * 2;
  constexpr size_t max_merge = static_cast<size_t>(WARPS + 1) * 8 * (D + 2) * sizeof(float);
  static_assert(max_merge <= ring, "the warps' merge area lies in the rings");
  const size_t smem = table_bytes + ring;
  p.part_off = static_cast<int32_t>(table_bytes + WARPS * static_cast<size_t>(G) * (D + 2) * 4);
  static thread_local int configured_dev = -1;
  static thread_local ClusterFit fit;
  const auto kernel = decode_mma_kernel<D, PAGED, MODS, WARPS, STAGES, P_TERMS>;
  const int rc = configure_decode(kernel, 224 * 1024, configured_dev);
  if (rc != LF_OK) return st ? rc : kNoCluster;
  if (p.cluster && !cluster_fits(kernel, p.splits, WARPS * 32,
                                 ring + (PAGED ? kMaxTableBytes : 0), fit))
    return kNoCluster;
  if (!st) return LF_OK;
  return launched(launch_splits(kernel, p, WARPS * 32, smem, *st, p, G), "decode_mma_kernel");
}

template <int D, bool PAGED, int MODS, int P_TERMS>
static int launch_decode_shape(const DecodeParams& p, int G, const cudaStream_t* st,
                               size_t table_bytes) {
  const int64_t ctas = static_cast<int64_t>(p.splits) * p.Hkv * p.B;
  const int sms = device_sm_count();
  // Warps and ring depth, by how full the machine is (times: B200, D = 128, G = 4 paged):
  //   one CTA per SM at most: eight warps, since four do not keep up with HBM on their own (128 units
  //     of 8190 keys 96 -> 83 us), except that eights and sixteens of such CTAs find no place for their
  //     clusters (16 units of 8190 keys 23 us in eights of four warps, 29 of eight);
  //   otherwise four, two CTAs resident per SM (K/V rings of 96 KB each);
  //   up to three CTAs per SM: two-stage rings, so that they are all resident (320 units of 1001 keys
  //     35 -> 32 us);
  //   up to five: half-sized CTAs as well, six resident (640 units of 3001 keys 171 -> 150 us; 512 of
  //     2048 the same 87); at D = 64, where the rings are half as large, three stages of up to four.
  if (ctas * 10 <= 9ll * sms && p.splits <= 4)
    return launch_decode_w<D, PAGED, MODS, P_TERMS, 8, 3>(p, G, st, table_bytes);
  if (ctas <= 2ll * sms || ctas > (D == 128 ? 5ll : 4ll) * sms)
    return launch_decode_w<D, PAGED, MODS, P_TERMS, 4, 3>(p, G, st, table_bytes);
  if (ctas <= 3ll * sms)
    return launch_decode_w<D, PAGED, MODS, P_TERMS, 4, 2>(p, G, st, table_bytes);
  return launch_decode_w<D, PAGED, MODS, P_TERMS, 2, D == 128 ? 2 : 3>(p, G, st, table_bytes);
}

template <int D, bool PAGED>
static int launch_decode(const DecodeParams& p, int G, int mods, const cudaStream_t* st,
                         size_t table_bytes) {
  auto with_mods = [&](auto m) {
    constexpr int kMods = decltype(m)::value;
    if constexpr (!PAGED)
      if (G <= 2) return launch_decode_shape<D, PAGED, kMods, 3>(p, G, st, table_bytes);
    return launch_decode_shape<D, PAGED, kMods, 2>(p, G, st, table_bytes);
  };
  if (mods == kModsNone) return with_mods(std::integral_constant<int, kModsNone>{});
  if (mods == kModsSoftcap) return with_mods(std::integral_constant<int, kModsSoftcap>{});
  return with_mods(std::integral_constant<int, kModsGeneric>{});
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// `stream` == nullptr: only tell how many kernels the call launches.
static int decode_impl(const LfDecodeArgs* a, void* const* stream, bool paged) {
  if (!a || !a->q || !a->k || !a->v || !a->out) return LF_ERR_INVALID_ARG;
  if (a->B <= 0 || a->Hkv <= 0 || a->G <= 0 || a->Skv <= 0) return LF_ERR_INVALID_ARG;
  if (a->D != 64 && a->D != 128) return LF_ERR_UNSUPPORTED;
  if (a->G != 1 && a->G != 2 && a->G != 4 && a->G != 8) return LF_ERR_UNSUPPORTED;
  if (a->n_mod < 0 || a->n_mod > LF_MAX_MODS) return LF_ERR_INVALID_ARG;
  if (a->Hkv > 65535 || a->B > 65535) return LF_ERR_TOO_LARGE;
  if (!aligned16(a->q) || !aligned16(a->k) || !aligned16(a->v) || !aligned16(a->out))
    return LF_ERR_ALIGNMENT;
  for (int i = 0; i < 3; ++i) {
    if ((a->q_stride[i] % 8) || (a->k_stride[i] % 8) || (a->v_stride[i] % 8) ||
        (a->o_stride[i] % 4))
      return LF_ERR_ALIGNMENT;
  }
  if (paged) {
    if (!a->block_table || a->page_size <= 0 || a->n_pages <= 0) return LF_ERR_INVALID_ARG;
  }
  int splits = a->splits;
  if (splits < 0) return LF_ERR_INVALID_ARG;
  if (splits > 32) return LF_ERR_TOO_LARGE;
  if (splits == 0) splits = choose_splits(a->B, a->Hkv, a->Skv, a->D, paged ? a->page_size : 0);
  const int partials = partial_splits(a->Skv, splits);
  if (partials > 1) {
    const size_t need = lf_decode_workspace_bytes(a->B, a->Hkv, a->G, a->D, partials);
    if (!a->workspace || a->workspace_bytes < need) return LF_ERR_WORKSPACE;
    if (!aligned16(a->workspace)) return LF_ERR_ALIGNMENT;
  }

  DecodeParams p;
  p.q = static_cast<const __nv_bfloat16*>(a->q);
  p.k = static_cast<const __nv_bfloat16*>(a->k);
  p.v = static_cast<const __nv_bfloat16*>(a->v);
  p.out = static_cast<__nv_bfloat16*>(a->out);
  const int64_t units = static_cast<int64_t>(a->B) * a->Hkv * a->G;
  p.part_o = static_cast<float*>(a->workspace);
  p.part_ml = p.part_o ? p.part_o + units * partials * a->D : nullptr;
  p.block_table = a->block_table;
  p.block_table_v = a->block_table_v ? a->block_table_v : a->block_table;
  p.status = a->status;
  for (int i = 0; i < 3; ++i) {
    p.q_stride[i] = a->q_stride[i];
    p.o_stride[i] = a->o_stride[i];
    p.k_stride[i] = a->k_stride[i];
    p.v_stride[i] = a->v_stride[i];
  }
  p.bt_stride = a->bt_stride;
  p.B = a->B;
  p.Hkv = a->Hkv;
  p.Skv = a->Skv;
  p.page_size = paged ? a->page_size : 1;
  p.page_shift = -1;
  for (int sh = 0; sh < 31; ++sh)
    if ((1 << sh) == p.page_size) p.page_shift = sh;
  p.n_pages = paged ? a->n_pages : 0;
  p.scale = a->scale;
  p.mods.n = a->n_mod;
  for (int i = 0; i < LF_MAX_MODS; ++i) {
    p.mods.op[i] = i < a->n_mod ? a->mod_op[i] : 0;
    p.mods.arg[i] = i < a->n_mod ? a->mod_arg[i] : 0.f;
  }

  // A softcap chain, (MUL|DIV)* TANH (MUL|DIV)*, folds into two multipliers.
  int mods = a->n_mod > 0 ? kModsGeneric : kModsNone;
  p.cap = 0.f;
  p.part_off = 0;
  {
    int i = 0;
    float pre = a->scale, post = kLog2e;
    auto fold = [&](float& x) {
      for (; i < a->n_mod && (a->mod_op[i] == LF_MOD_MUL || a->mod_op[i] == LF_MOD_DIV); ++i)
        x = a->mod_op[i] == LF_MOD_MUL ? x * a->mod_arg[i] : x / a->mod_arg[i];
    };
    fold(pre);
    if (i < a->n_mod && a->mod_op[i] == LF_MOD_TANH) {
      ++i;
      fold(post);
      if (i == a->n_mod) {
        mods = kModsSoftcap;
        p.scale = pre;
        p.cap = post;
      }
    }
  }

  const cudaStream_t st = stream ? static_cast<cudaStream_t>(*stream) : nullptr;
  auto attempt = [&](bool cluster) -> int {
    // Tokens per split: a multiple of 16, so a split never starts in the middle of a warp's token batch.
    // Where the rounding leaves a cluster's last splits empty the count stays as it is; their partials
    // have weight zero. (Powers of two make the better clusters: over 70 sizes whose count a rounding to
    // 64 would trim, to 3, 6, 7 or 11..15, 6 % less time warm and 3 % cold.)
    p.cluster = cluster;
    p.splits = cluster ? splits : partials;
    p.chunk = cluster ? round_up((a->Skv + splits - 1) / splits, 16) : partial_chunk(a->Skv, splits);
    size_t table_bytes = 0;
    if (paged) {
      // A split's block-table slice lives in shared memory next to the K/V rings. The automatic
      // split count already keeps it small enough; an explicit count that does not is refused
      // (pass a larger `splits`, or 0).
      table_bytes = table_smem_bytes(p.chunk, p.page_size);
      if (table_bytes > kMaxTableBytes) return LF_ERR_TOO_LARGE;
    }
    if (!stream && !cluster) return LF_OK;
    const cudaStream_t* to = stream ? &st : nullptr;
    if (a->D == 128)
      return paged ? launch_decode<128, true>(p, a->G, mods, to, table_bytes)
                   : launch_decode<128, false>(p, a->G, mods, to, table_bytes);
    return paged ? launch_decode<64, true>(p, a->G, mods, to, table_bytes)
                 : launch_decode<64, false>(p, a->G, mods, to, table_bytes);
  };
  // The splits merge in their cluster where one holds them and the grid is about one wave; a grid
  // of many waves hides the combine kernel's time, and its CTAs need not be placed in groups. (In pairs:
  // 2048 units of 2048 keys, each call on other buffers, 313 -> 324 us; 3000 one-token pages 475 -> 510.)
  int rc = kNoCluster;
  if (splits > 1 && splits <= kMaxCluster &&
      static_cast<int64_t>(splits) * a->Hkv * a->B <= 8ll * device_sm_count())
    rc = attempt(true);
  if (rc == kNoCluster) rc = attempt(false);
  if (rc != LF_OK) return rc;
  const bool combine = p.splits > 1 && !p.cluster;
  if (!stream) return combine ? 2 : 1;
  if (combine)
    rc = lf_combine_f32(p.part_o, p.part_ml, a->out, a->B, a->Hkv, a->G, a->D, p.splits,
                        a->o_stride, *stream);
  return rc;
}

}  // namespace lf

extern "C" {

int lf_decode_auto_splits(int32_t B, int32_t Hkv, int32_t /*G*/, int32_t Skv, int32_t D,
                          int32_t page_size) {
  if (B <= 0 || Hkv <= 0 || Skv <= 0) return 1;
  return lf::choose_splits(B, Hkv, Skv, D, page_size > 0 ? page_size : 0);
}

size_t lf_decode_workspace_bytes(int32_t B, int32_t Hkv, int32_t G, int32_t D, int32_t splits) {
  if (splits <= 1) return 0;
  const size_t units = static_cast<size_t>(B) * Hkv * G;
  return units * splits * (static_cast<size_t>(D) + 2) * sizeof(float);
}

int lf_decode_bf16(const LfDecodeArgs* args, void* stream) {
  return lf::decode_impl(args, &stream, false);
}

int lf_decode_paged_bf16(const LfDecodeArgs* args, void* stream) {
  return lf::decode_impl(args, &stream, true);
}

int lf_decode_launches(const LfDecodeArgs* args, int32_t paged) {
  return lf::decode_impl(args, nullptr, paged != 0);
}

int lf_combine_f32(const float* part_o, const float* part_ml, void* out, int32_t B, int32_t Hkv,
                   int32_t G, int32_t D, int32_t splits, const int64_t* o_stride, void* stream) {
  if (!part_o || !part_ml || !out || !o_stride) return LF_ERR_INVALID_ARG;
  if (B <= 0 || Hkv <= 0 || G <= 0 || splits <= 0) return LF_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return LF_ERR_UNSUPPORTED;
  if (splits > 32) return LF_ERR_TOO_LARGE;  // one lane per split in the combine
  const int64_t units = static_cast<int64_t>(B) * Hkv * G;
  const unsigned blocks = static_cast<unsigned>((units + 3) / 4);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (D == 128)
    lf::launch_pdl(lf::combine_kernel<128>, dim3(blocks), 128, 0, st, part_o, part_ml,
                   static_cast<__nv_bfloat16*>(out), units, Hkv, G, splits, o_stride[0],
                   o_stride[1], o_stride[2]);
  else
    lf::launch_pdl(lf::combine_kernel<64>, dim3(blocks), 128, 0, st, part_o, part_ml,
                   static_cast<__nv_bfloat16*>(out), units, Hkv, G, splits, o_stride[0],
                   o_stride[1], o_stride[2]);
  return lf::check_launch("combine_kernel");
}

int lf_paged_gather_bf16(const void* pool, const int32_t* block_table, void* out, int32_t B,
                         int32_t Hkv, int32_t Skv, int32_t D, int32_t page_size, int32_t n_pages,
                         const int64_t* pool_stride, int64_t bt_stride, int32_t* status,
                         void* stream) {
  if (!pool || !block_table || !out || !pool_stride) return LF_ERR_INVALID_ARG;
  if (B <= 0 || Hkv <= 0 || Skv <= 0 || page_size <= 0 || n_pages <= 0)
    return LF_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return LF_ERR_UNSUPPORTED;
  if (!lf::aligned16(pool) || !lf::aligned16(out)) return LF_ERR_ALIGNMENT;
  for (int i = 0; i < 3; ++i)
    if (pool_stride[i] % 8) return LF_ERR_ALIGNMENT;
  const int64_t threads = static_cast<int64_t>(B) * Hkv * Skv * (D / 8);
  const unsigned blocks = static_cast<unsigned>((threads + 255) / 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (D == 128)
    lf::paged_gather_kernel<128><<<blocks, 256, 0, st>>>(
        static_cast<const __nv_bfloat16*>(pool), block_table, static_cast<__nv_bfloat16*>(out),
        B, Hkv, Skv, page_size, n_pages, pool_stride[0], pool_stride[1], pool_stride[2],
        bt_stride, status);
  else
    lf::paged_gather_kernel<64><<<blocks, 256, 0, st>>>(
        static_cast<const __nv_bfloat16*>(pool), block_table, static_cast<__nv_bfloat16*>(out),
        B, Hkv, Skv, page_size, n_pages, pool_stride[0], pool_stride[1], pool_stride[2],
        bt_stride, status);
  return lf::check_launch("paged_gather_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Decode without any allocation by the caller or the library.
//
// Some callers cannot call cudaMalloc or hand over a workspace at the point where they launch
// decode: a serving loop that has frozen its memory pool, a plugin running inside another
// runtime's callback where allocation is forbidden, or a host that only holds the input and
// output buffers it was given. For them the split-KV partials live in this fixed array, which
// is part of the library image: every GPU that loads the library holds these bytes until the
// process exits.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_static_scratch[LF_STATIC_SCRATCH_BYTES];

namespace lf {

constexpr int kMaxStaticDevices = 64;
static std::mutex g_static_mutex;
static void* g_static_scratch_addr[kMaxStaticDevices] = {};

// Device address of the scratch array on the current device. `g_static_scratch` itself is only
// a host-side handle in host code, so it is translated once per device (with that device
// current) and the translated pointer is what the kernels receive.
static int static_scratch_address(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_cuda_error(e, "cudaGetDevice");
    return LF_ERR_NO_DEVICE;
  }
  if (dev < 0 || dev >= kMaxStaticDevices) return LF_ERR_TOO_LARGE;
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_scratch_addr[dev]) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || !ptr) {
      set_cuda_error(e, "cudaGetSymbolAddress(g_static_scratch)");
      cudaGetLastError();
      return LF_ERR_CUDA;
    }
    g_static_scratch_addr[dev] = ptr;
  }
  *out = g_static_scratch_addr[dev];
  return LF_OK;
}

}  // namespace lf

extern "C" int lf_decode_bf16_static(const LfDecodeArgs* args, void* stream) {
  if (!args) return LF_ERR_INVALID_ARG;
  if (args->B <= 0 || args->Hkv <= 0 || args->G <= 0 || args->Skv <= 0)
    return LF_ERR_INVALID_ARG;
  int splits = args->splits;
  if (splits < 0) return LF_ERR_INVALID_ARG;
  if (splits > 32) splits = lf::partial_splits(args->Skv, splits);
  if (splits == 0) splits = lf::choose_splits(args->B, args->Hkv, args->Skv, args->D, 0);
  const size_t need = lf_decode_workspace_bytes(args->B, args->Hkv, args->G, args->D,
                                                lf::partial_splits(args->Skv, splits));
  if (need > static_cast<size_t>(LF_STATIC_SCRATCH_BYTES)) {
    if (args->splits != 0) return LF_ERR_TOO_LARGE;
    splits = 1;  // (the library's own count: without a split there are no partials)
  }
  void* scratch = nullptr;
  const int rc = lf::static_scratch_address(&scratch);
  if (rc != LF_OK) return rc;
  LfDecodeArgs local = *args;
  local.splits = splits;
  local.workspace = scratch;
  local.workspace_bytes = static_cast<size_t>(LF_STATIC_SCRATCH_BYTES);
  return lf::decode_impl(&local, &stream, false);
}
