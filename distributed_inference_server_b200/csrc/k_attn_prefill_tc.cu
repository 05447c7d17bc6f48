// k_attn_prefill_tc.cu -- causal prefill attention on the 5th-generation tensor cores:
// tcgen05.mma with S = Q K^T and the per-tile P V product accumulated in TMEM, K/V tiles staged by TMA.
// No reference counterpart (the reference has no tensor code at all).
//
// One CTA = (query block, kv head).  A query block is up to QT = 128 / G consecutive tokens of one sequence
// (G = query heads per kv head: 32 tokens for Llama-3-8B's 4:1 GQA, 16 for 70B's and TinyLlama's 8:1); its G heads x QT tokens
// are the 128 rows (= 128 TMEM lanes) of every MMA, row = head * QT + token, so K and V are fetched once per
// 128 query rows and the QK^T / PV products run at tcgen05 rate instead of through ldmatrix + mma.sync
// (k_attn_paged.cu).  Tensor- and exponential-bound: 4 * rows * keys * d flop and rows * keys exponentials per (block, kv head).
//
//   warp 0      TMA producer: 64-key K and V tiles (128B-swizzled boxes out of the page pool), two slots each
//   warp 1      the MMAs:  S_j = Q K_j^T   M128 N64 K16 x D/16  (A, B K-major, shared memory)
//                          O  += P_j V_j   M128 N=D K16 x 4     (A = P from TMEM, B = V MN-major)
//   warps 2-5   softmax of the even tiles, warps 6-9 of the odd ones, one thread per row: S_j from TMEM, causal mask, row maximum (no
//               shuffles: a thread owns a whole row); P_j = exp2(s - m) goes as packed bf16 back into S_j's own TMEM columns (no
//               shared-memory write, proxy fence or second read of it)
// TMEM per CTA: S0 | S1 64 columns each | O (D = 128: 128 columns; D = 64: one of 64 for each group) = 256; shared memory Q + 2 K + 2 V =
// 96 KB (D = 128): two CTAs per SM, so four softmax groups take turns on the exponentials (16 per clock and SM: 1024 clocks per 128 rows x
// 128 keys, beside 512 or 1024 of the tensor pipe).  O accumulates in TMEM.
//   D = 64   each group has an O and a reference of its own, the running maximum of its tiles: a row's largest weight is exactly 1 when it
//            is rounded to bf16, and O is rescaled behind the group's own P V, which the next S waits for anyway.  The two are joined at
//            the end.  With the lazy reference below the results were 3.5 % further from 64 bits than weights rounded under the row's own
//            maximum are, as the mma.sync kernel rounds them; so they are no further.
//   D = 128  no columns are left for a second O: the two groups share a row's reference m_ref, handed from tile to tile through shared
//            memory and raised only when a row's maximum exceeds it by more than 8 in the log2 domain (P <= 256, the reference cancels
//            in the final division by l), so O is rescaled on few tiles only (decided per warp, scaled per lane).
//
// Measured against what it replaced: heads of 64 (mma.sync), six prompts of 276 to 1900 tokens, 32 / 4 heads, 31.6 GFLOP: 165.1 -> 78.8
// us (with the lazy reference 74.0); heads of 128 (one softmax group per CTA, P through shared memory), six prompts of 437 to 3000
// tokens, 32 / 8 heads, 258 GFLOP: 362.4 -> 340.5 us.  With two CTAs on an SM a key tile takes each 1230 clocks (D = 64, lazy: 620 per
// tile and SM, 512 of them exponentials) or 1800 (D = 128: 900, 768 of them shared memory -- Q and K for S, V, and the tiles' arrival);
// a CTA's start and end take 5000 and 10000.
#include <cuda.h>

#include <cfloat>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "kernels.h"
#include "ptx.cuh"

namespace dis {

constexpr int kPfTile = 64;             // keys per tile
constexpr int kPfHalf = kPfTile * 128;  // one [64 keys][64 dims] block of K or V, 8 KB
constexpr int kPfTmemCols = 256;
constexpr float kPfLazy = 8.0f;

// V's descriptor (umma_lo_mn) is MN-major, 128B swizzle: element (mn, k) lives at (mn % 64) * 2 + (mn / 64) * LBO + (k % 8) * 128 +
// (k / 8) * SBO -- the [keys][dims] tile as TMA stores it, LBO the distance of its two 64-dim blocks.
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr int kPfThreads = 320;
constexpr int kPfQHalf = 128 * 128;  // one [128 rows][64 dims] block of Q, 16 KB

template <int D>
constexpr int pf_smem_bytes() { return (D / 64) * (kPfQHalf + 4 * kPfHalf) + 4 * 128 * 4 + 256; }

// Packed pairs: one issue slot for two lanes' worth of work
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// producer-consumer barriers of a pair of warps: one arrives, the other waits
__device__ __forceinline__ void named_sync_64(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void named_arrive_64(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// O's 32 columns from o_addr on, times f (a warp-collective read, scale and write back), eight at a time: it runs on few tiles, with the
// scores of the tile live.
__device__ __forceinline__ void rescale_32(uint32_t o_addr, float f) {
#pragma unroll
  for (int c = 0; c < 32; c += 8) {
    uint32_t v[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(o_addr + c)
                 : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(o_addr + c), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
  }
}

// Page numbers of a sequence for a warp that walks it: 32 at a time, one in each lane.  (A lookup per box in front of its TMA load took
// the producer 580 clocks a tile, an L2 latency.)
struct PageWindow {
  int first = -64, mine = 0;
  __device__ __forceinline__ int get(const int *pt, int i, int last) {  // i, last: the same in every lane
    if (i - first >= 32) {
      first = i;
      mine = pt[min(i + (int)(threadIdx.x & 31), last)];
    }
    return __shfl_sync(0xffffffffu, mine, i - first);
  }
};

template <int D, int G>
__global__ void __launch_bounds__(kPfThreads, 2)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap kv_map, long long row0, const uint16_t *__restrict__ q,
                        const int *__restrict__ page_table, int max_pages, const int *__restrict__ qb_tok0,
                        const int *__restrict__ qb_len, const int *__restrict__ qb_pos0, const int *__restrict__ qb_ptrow,
                        uint16_t *__restrict__ out, int n_heads, int n_kv, int page_shift) {
  constexpr int QT = 128 / G;
  constexpr int kHalves = D / 64;
  constexpr bool kOwn = 2 * kPfTile + 2 * D <= kPfTmemCols;  // an O and a softmax reference of each group's own
  constexpr uint32_t kSlot = kHalves * kPfHalf;  // one K or V tile
  extern __shared__ __align__(1024) uint8_t smem_al[];
  const uint32_t smem_base = smem_u32(smem_al);
  if (smem_base & 1023u) __trap();  // the 128B-swizzle atoms need 1024-byte alignment and there is no room for slack
  uint8_t *smem = smem_al;
  const uint32_t q_base = smem_base, k_base = q_base + kHalves * kPfQHalf, v_base = k_base + 2 * kSlot;
  const uint32_t bar_base = v_base + 2 * kSlot;
  auto k_full = [&](int w) { return bar_base + 8u * w; };
  auto k_empty = [&](int w) { return bar_base + 16u + 8u * w; };
  auto v_full = [&](int w) { return bar_base + 32u + 8u * w; };
  auto s_full = [&](int w) { return bar_base + 48u + 8u * w; };
  auto p_full = [&](int w) { return bar_base + 64u + 8u * w; };
  auto pv_done = [&](int w) { return bar_base + 80u + 8u * w; };
  const uint32_t q_full = bar_base + 96, tmem_slot = bar_base + 104;
  float *l_row = reinterpret_cast<float *>(smem + (bar_base - smem_base) + 256);  // [group][row]: at the end
  float *m_row = l_row + 256;  // one O: [row], the softmax reference, handed from tile to tile; two: [group][row], at the end

  // Later query blocks of a sequence have more key tiles: launch them first, so that the longest CTAs do not form the tail.  D = 64, whose passes of
  // more than a round stay here where histories are long: a block's kv heads one after the other, or the tail would be whole heads (one prompt of
  // 3000 tokens, 32 / 4 heads, 75.5 -> 63.6 us).
  const unsigned long long at = (unsigned long long)blockIdx.y * gridDim.x + blockIdx.x;
  const int qb = (int)(gridDim.x - 1 - (D == 64 ? at / n_kv : blockIdx.x)), kvh = D == 64 ? (int)(at % n_kv) : blockIdx.y;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&kv_map);
    for (int w = 0; w < 2; w++) {
      mbar_init(k_full(w), 1); mbar_init(k_empty(w), 1); mbar_init(v_full(w), 1); mbar_init(s_full(w), 1); mbar_init(pv_done(w), 1);
      mbar_init(p_full(w), 4);
    }
    mbar_init(q_full, 8);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) tmem_alloc<kPfTmemCols>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Only now, with the allocation done: a CTA of the next kernel that took its columns first would wait for this grid, and this CTA for
  // those columns.
  pdl_launch_dependents();
  pdl_wait();  // q and this chunk's K/V rows come from the previous kernels
  const int tok0 = qb_tok0[qb], len = qb_len[qb], pos0 = qb_pos0[qb];
  const int *pt = page_table + (size_t)qb_ptrow[qb] * max_pages;
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const uint32_t o_base = tmem_base + 2 * kPfTile;

  const int page_size = 1 << page_shift;
  const int box_rows = min(page_size, kPfTile);  // rows of the tensor map's box
  const int end = pos0 + len;                    // keys [0, end)
  const int n_tiles = (end + kPfTile - 1) / kPfTile;

  // Q is handed to the MMA warp by a barrier of its own: the key tiles are under way meanwhile
  if (warp >= 2) {  // Q tile: row = head * QT + token, K-major, 128B swizzle (rows of padding tokens are zero)
    const int row = (warp & 3) * 32 + lane, grp = (warp - 2) >> 2;
    const int hl = row / QT, t = row % QT;
    const uint4 *src = reinterpret_cast<const uint4 *>(q + ((size_t)(tok0 + t) * n_heads + kvh * G + hl) * D);
#pragma unroll
    for (int cc = 0; cc < D / 16; cc++) {
      const int c = grp * (D / 16) + cc;
      const uint4 v = t < len ? src[c] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t off = (uint32_t)(c >> 3) * kPfQHalf + (uint32_t)(row >> 3) * 1024 + (uint32_t)(row & 7) * 128 +
                           (uint32_t)(((c & 7) ^ (row & 7)) << 4);
      *reinterpret_cast<uint4 *>(smem + off) = v;
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(q_full);
  }

  if (warp == 0) {
    // ===== TMA producer: K_t as soon as S_{t-2} has read its slot, V_t as soon as P_{t-2} V_{t-2} has; one lane acts, all hold page numbers =====
    const int last_box = (end - 1) / box_rows * box_rows, last_page = last_box >> page_shift;
    PageWindow win[2];
    auto load = [&](int tile, bool is_v, PageWindow &pages) {
      const int w = tile & 1;
      const uint32_t full = is_v ? v_full(w) : k_full(w);
      if (tile >= 2) mbar_wait(is_v ? pv_done(w) : k_empty(w), (uint32_t)(tile / 2 - 1) & 1u);
      const uint32_t sbase = (is_v ? v_base : k_base) + w * kSlot;
      if (lane == 0) mbar_expect_tx(full, kSlot);
      for (int r = 0; r < kPfTile; r += box_rows) {
        // Boxes past the last key repeat the last one that holds a key: their scores are masked, and their values must be
        // finite because they are multiplied by a weight of zero.
        const int pos = min(tile * kPfTile + r, last_box);
        const long long page = pages.get(pt, pos >> page_shift, last_page);
        const long long krow = row0 + ((page * 2 + (is_v ? 1 : 0)) * n_kv + kvh) * page_size + (pos & (page_size - 1));
        if (lane == 0) {
#pragma unroll
          for (int hh = 0; hh < kHalves; hh++) tma_load_2d(sbase + hh * kPfHalf + r * 128, &kv_map, hh * 64, (int)krow, full, kEvictLast);
        }
      }
      __syncwarp();
    };
    for (int t = 0; t <= n_tiles; t++) {
      if (t < n_tiles) load(t, false, win[0]);
      if (t >= 1) load(t - 1, true, win[1]);
    }
  } else if (warp == 1 && n_tiles > 0) {  // (an empty block at position 0 has no tile to wait for)
    // ===== MMA issuer: the warp converged, one elected lane issues =====
    constexpr uint32_t idesc_s = umma_idesc<kPfTile>();
    constexpr uint32_t idesc_o = umma_idesc<D>() | (1u << 16);  // B (= V) MN-major
    const uint32_t q_lo = umma_lo(q_base), k_lo = umma_lo(k_base), v_lo = umma_lo_mn(v_base, kPfHalf);
    auto issue_s = [&](int j) {
      const uint32_t w = (uint32_t)j & 1u;
      mbar_wait(k_full(w), (uint32_t)(j >> 1) & 1u);
      tc_fence_after();
      if (elect_one()) {
        const uint32_t b = k_lo + w * (kSlot >> 4), d = tmem_base + w * kPfTile;
#pragma unroll
        for (uint32_t k = 0; k < D / 16; k++)
          umma_ss(d, q_lo + (k >> 2) * (kPfQHalf >> 4) + (k & 3) * 2, b + (k >> 2) * (kPfHalf >> 4) + (k & 3) * 2, idesc_s, k > 0 ? 1u : 0u);
        umma_commit(s_full(w));
        umma_commit(k_empty(w));
      }
      __syncwarp();
    };
    mbar_wait(q_full, 0);
    issue_s(0);
    if (n_tiles > 1) issue_s(1);
    for (int j = 0; j < n_tiles; j++) {
      const uint32_t w = (uint32_t)j & 1u;
      mbar_wait(v_full(w), (uint32_t)(j >> 1) & 1u);
      mbar_wait(p_full(w), (uint32_t)(j >> 1) & 1u);
      tc_fence_after();
      if (elect_one()) {
        const uint32_t b = v_lo + w * (kSlot >> 4), a = tmem_base + w * kPfTile;
#pragma unroll
        for (uint32_t k = 0; k < kPfTile / 16; k++)
          umma_ts(o_base + (kOwn ? w * D : 0), a + 8 * k, b + k * 128, idesc_o, k > 0 ? 1u : (uint32_t)(j > (kOwn ? 1 : 0)));
        umma_commit(pv_done(w));
      }
      __syncwarp();
      if (j + 2 < n_tiles) {
        mbar_wait(pv_done(w), (uint32_t)(j >> 1) & 1u);  // S_{j+2} overwrites the columns that P_j V_j reads
        issue_s(j + 2);
      }
    }
  } else if (warp >= 2 && n_tiles > 0) {
    // ===== softmax: group 0 takes the even tiles, group 1 the odd ones; one thread per row; O lives in TMEM =====
    const int quarter = warp & 3;  // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    const int grp = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const int hl = row / QT, t = row % QT;
    const int qp = pos0 + t;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + grp * kPfTile, o_addr = o_base + lane_off + (kOwn ? grp * D : 0);
    const int bar_in = 1 + 4 * grp + quarter, bar_out = 1 + 4 * (grp ^ 1) + quarter;  // hand-over of m_row to this group / to the other
    const float scale_log2 = rsqrtf((float)D) * 1.4426950408889634f;
    const float2 scale2 = make_float2(scale_log2, scale_log2);
    float m_ref = kOwn ? -FLT_MAX : -INFINITY, l_run = 0.f;  // (finite where a group's first tile may hide every key of a row)
    for (int j = grp; j < n_tiles; j += 2) {
      mbar_wait(s_full(grp), (uint32_t)(j >> 1) & 1u);
      tc_fence_after();
      uint32_t s[2][32];
      tmem_ld_32x32(s_addr, s[0]);
      tmem_ld_32x32(s_addr + 32, s[1]);
      tmem_ld_wait();
      const int rest = qp - j * kPfTile;  // keys 0 .. rest of the tile are visible
      if (rest < kPfTile - 1) {           // only the tiles that cross the diagonal need the causal mask
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int i = 0; i < 32; i++)
            if (32 * c + i > rest) s[c][i] = 0xff800000u;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; i++) mx4[i & 3] = max3(mx4[i & 3], __uint_as_float(s[0][i]), __uint_as_float(s[1][i]));
      const float mx = max3(mx4[0], mx4[1], fmaxf(mx4[2], mx4[3])) * scale_log2;  // scale > 0: it commutes with the maximum
      float m_now, f = 1.0f;
      bool rescale = false;
      if (kOwn) {
        // S_j was issued behind P_{j-2} V_{j-2}: this group's O is complete, and nobody else touches it
        m_now = fmaxf(m_ref, mx);
        rescale = j >= 2 && __any_sync(0xffffffffu, mx > m_ref);
        f = ex2_approx(m_ref - m_now);
      } else if (j == 0) {
        m_now = mx;  // finite: key 0 is visible to every query; O is first written by P_0 V_0 (accumulate off)
      } else {
        named_sync_64(bar_in);
        const float m_old = m_row[row];
        const bool need = mx > m_old + kPfLazy;
        m_now = need ? mx : m_old;
        if (__any_sync(0xffffffffu, need)) {  // tcgen05.ld / st are warp-collective: decide per warp, scale per lane
          // every P V so far must be in O; none follows before this tile's P is handed over
          mbar_wait(pv_done(grp ^ 1), (uint32_t)((j - 1) >> 1) & 1u);
          tc_fence_after();
          f = need ? ex2_approx(m_old - mx) : 1.0f;
#pragma unroll 1
          for (int c = 0; c < D; c += 32) rescale_32(o_addr + c, f);
          tmem_st_wait();
        }
      }
      if (!kOwn && j + 1 < n_tiles) {
        m_row[row] = m_now;
        named_arrive_64(bar_out);
      }
      l_run *= ex2_approx(m_ref - m_now);  // what this group has summed so far, under the reference of now (0 at its first tile)
      m_ref = m_now;
      const float2 neg_m = make_float2(-m_ref, -m_ref);
      float2 ps[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 2; c++) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float2 p = fma2(make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), scale2, neg_m);
          p.x = ex2_approx(p.x);
          p.y = ex2_approx(p.y);
          pk[i >> 1] = float2_to_bf16x2(p.x, p.y);
          // the sum takes the weights as P V takes them, rounded: a row that one key dominates keeps that key's weight at 1
          ps[(i >> 1) & 1] = add2(ps[(i >> 1) & 1], bf16x2_to_float2(pk[i >> 1]));
        }
        tmem_st_32x16(s_addr + 16 * c, pk);
      }
      if (kOwn && rescale) {
#pragma unroll
        for (int c = 0; c < D; c += 32) rescale_32(o_addr + c, f);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(grp));
      l_run += (ps[0].x + ps[0].y) + (ps[1].x + ps[1].y);
    }
    float inv, f0 = 1.f, f1 = 1.f;  // what the two groups' O are weighted with
    if (kOwn) {
      m_row[grp * 128 + row] = m_ref;
      l_row[grp * 128 + row] = l_run;
      asm volatile("bar.sync 9, 256;" ::: "memory");
      const float m0 = m_row[row], m1 = m_row[128 + row], m = fmaxf(m0, m1);
      f0 = ex2_approx(m0 - m);
      f1 = ex2_approx(m1 - m);
      inv = 1.0f / (l_row[row] * f0 + l_row[128 + row] * f1);
      f0 *= inv;
      f1 *= inv;
    } else {
      // the group of the last tile publishes the final reference; then each brings its sum to it
      if (grp == ((n_tiles - 1) & 1)) m_row[row] = m_ref;
      asm volatile("bar.sync 9, 256;" ::: "memory");
      l_row[grp * 128 + row] = l_run * ex2_approx(m_ref - m_row[row]);
      asm volatile("bar.sync 9, 256;" ::: "memory");
      inv = 1.0f / (l_row[row] + l_row[128 + row]);
    }
    mbar_wait(pv_done((n_tiles - 1) & 1), (uint32_t)((n_tiles - 1) >> 1) & 1u);
    tc_fence_after();
    uint4 *o = reinterpret_cast<uint4 *>(out + ((size_t)(tok0 + t) * n_heads + kvh * G + hl) * D);
#pragma unroll
    for (int cc = 0; cc < D / 2; cc += 32) {
      const int c = grp * (D / 2) + cc;
      uint32_t v[32];
      tmem_ld_32x32(o_base + lane_off + c, v);
      tmem_ld_wait();
      if (kOwn) {
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * f0);
        if (n_tiles > 1) {
          uint32_t u[32];
          tmem_ld_32x32(o_base + lane_off + D + c, u);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i++) v[i] = __float_as_uint(fmaf(__uint_as_float(u[i]), f1, __uint_as_float(v[i])));
        }
        inv = 1.f;
      }
      if (t < len) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          uint4 w;
          w.x = float2_to_bf16x2(__uint_as_float(v[i * 8 + 0]) * inv, __uint_as_float(v[i * 8 + 1]) * inv);
          w.y = float2_to_bf16x2(__uint_as_float(v[i * 8 + 2]) * inv, __uint_as_float(v[i * 8 + 3]) * inv);
          w.z = float2_to_bf16x2(__uint_as_float(v[i * 8 + 4]) * inv, __uint_as_float(v[i * 8 + 5]) * inv);
          w.w = float2_to_bf16x2(__uint_as_float(v[i * 8 + 6]) * inv, __uint_as_float(v[i * 8 + 7]) * inv);
          o[c / 8 + i] = w;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc<kPfTmemCols>(tmem_base);
}

// ---------------------------------------------------------------------------------------- two query blocks per CTA
// attn_prefill_pair_kernel: the form for passes that fill the GPU.  A CTA per SM stays, takes a pair of query blocks, and while it works on
// it asks the hardware for the next pair that no CTA has begun (cluster launch control: a dynamic schedule without a counter in memory).
// The two blocks, if they are of one sequence, share every K and V tile, and each has a softmax group, an O and a softmax reference of its own
// (D = 64: one of each for even and for odd tiles, as above and with the same bits): nothing is handed from group to group, S is
// double-buffered (2 x 2 x 64 columns, O 2 x 128), and the next pair's first tiles, scores and query rows are under way while the output of this
// one is read out.
//
//   warp 0       page numbers (32 at a time), K and V tiles of 64 keys into a ring of six, the list of passes
//   warps 1, 2   the MMAs of group 0 and 1, S two tiles ahead of P V
//   warp 3       query rows, two slots for each group
//   warps 4-11   softmax of the two groups, one thread per row; the running maxima of D = 64 and the lazy reference of D = 128 as above
//
// What bounds it, stamped per pair of 64-key tiles (D = 128): 1280 clocks of the tensor pipe (a product with N = 64 reads Q at shared memory's rate:
// 48 clocks where it computes 32) beside 1024 of exponentials; a group's own chain is 1800 (scores 200-400, maximum 250, exponentials 850-1100,
// hand-over).  A run of such passes draws 1000 W: 244 us cold, 281 under the power cap.  D = 64: the chain, 640 tensor, 1024 exponentials.
// Measured against the kernel above: heads of 128, six prompts of 437 to 3000 tokens, 32 / 8 heads: 335 -> 281 us (cold 312 -> 244); eight of up to
// 700: 39.5 -> 28.1; 64 / 8 heads, six of up to 1900: 202 -> 152; heads of 64, six of 276 to 1900 tokens, 32 / 4 heads: 76 -> 69.1.
// On the way: a page lookup in front of each TMA load cost 580 clocks a tile, one MMA warp for both groups 100 to 170 clocks per wait; tiles of 128 keys
// with one score buffer (a wait for S in every step) 335 us, four blocks per CTA for heads of 64 (96 registers, all in step) 79 to 84 us.
constexpr int kPpTile = kPfTile;             // keys per tile
constexpr int kPpThreads = 384;              // producer, 2 x MMA, query rows, 2 x 4 softmax warps
constexpr int kPpQSlots = 4, kPpDesc = 3;    // two query tiles for each group
constexpr int kPpRing = 6;                   // K and V tiles
template <int D>
constexpr int pp_smem_bytes() { return (D / 64) * (kPpQSlots * kPfQHalf + kPpRing * kPfHalf) + 1024; }

__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// O's 64 columns from o_addr on, times f, in one go
__device__ __forceinline__ void rescale_64(uint32_t o_addr, float f) {
  uint32_t v[2][32];
  tmem_ld_32x32(o_addr, v[0]);
  tmem_ld_32x32(o_addr + 32, v[1]);
  tmem_ld_wait();
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int i = 0; i < 32; i++) v[h][i] = __float_as_uint(__uint_as_float(v[h][i]) * f);
    tmem_st_32x32(o_addr + 32 * h, v[h]);
  }
}

// What one pass of a CTA works on: one or two query blocks of one sequence (the second's n is 0 where there is none)
struct PfPass {
  int n[2];                       // key tiles; -1: no pass follows
  int tok0[2], len[2], pos0[2];
  int kvh, pad;
};

// 16 bytes to shared memory, the part behind `bytes` of them zero
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Asks the hardware for a CTA of this grid that has not started yet; its index arrives in shared memory (Blackwell's cluster launch control).
__device__ __forceinline__ void clc_try_cancel(uint32_t resp, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(resp), "r"(bar) : "memory");
}
__device__ __forceinline__ bool clc_query(uint32_t resp, int &x) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t.reg .b32 y, z, w;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.b32 %0, 1, 0, p;\n\tmov.b32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, y, z, w}, h;\n\t}"
      : "=&r"(ok), "=&r"(x)
      : "r"(resp)
      : "memory");
  return ok != 0;
}

template <int D, int G>
__global__ void __launch_bounds__(kPpThreads, 1)
attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap kv_map, long long row0, const uint16_t *__restrict__ q,
                         const int *__restrict__ page_table, int max_pages, const int *__restrict__ qb_tok0,
                         const int *__restrict__ qb_len, const int *__restrict__ qb_pos0, const int *__restrict__ qb_ptrow,
                         uint16_t *__restrict__ out, int n_heads, int n_kv, int page_shift, int n_blocks) {
  constexpr int QT = 128 / G, kHalves = D / 64, kRing = kPpRing;
  constexpr uint32_t kQBytes = kHalves * kPfQHalf, kSlot = kHalves * kPfHalf;
  constexpr bool kOwn = D == 64;  // even and odd tiles each with an O and a reference of their own; D = 128: one of each, the reference lazy
  constexpr uint32_t kOCols = 128;  // columns of a group's O
  extern __shared__ __align__(1024) uint8_t smem_al[];
  const uint32_t smem_base = smem_u32(smem_al);
  if (smem_base & 1023u) __trap();  // the 128B-swizzle atoms need 1024-byte alignment and there is no room for slack
  const uint32_t q_base = smem_base, ring_base = q_base + kPpQSlots * kQBytes, bar_base = ring_base + kRing * kSlot;
  auto full = [&](uint32_t s) { return bar_base + 8u * s; };
  auto empty = [&](uint32_t s) { return bar_base + 64u + 8u * s; };
  auto q_full = [&](uint32_t s) { return bar_base + 128u + 8u * s; };
  auto q_empty = [&](uint32_t s) { return bar_base + 160u + 8u * s; };
  auto s_full = [&](uint32_t g, uint32_t w) { return bar_base + 192u + 16u * g + 8u * w; };
  auto p_full = [&](uint32_t g, uint32_t w) { return bar_base + 224u + 16u * g + 8u * w; };
  auto pv_done = [&](uint32_t g, uint32_t w) { return bar_base + 256u + 16u * g + 8u * w; };
  auto o_empty = [&](uint32_t g) { return bar_base + 288u + 8u * g; };
  auto d_full = [&](uint32_t s) { return bar_base + 304u + 8u * s; };
  auto d_empty = [&](uint32_t s) { return bar_base + 328u + 8u * s; };
  const uint32_t clc_bar = bar_base + 352u, clc_resp = bar_base + 368u, tmem_slot = bar_base + 384u;
  PfPass *desc = reinterpret_cast<PfPass *>(smem_al + (bar_base - smem_base) + 400);
  static_assert(400 + kPpDesc * sizeof(PfPass) <= 1024 && kRing <= 8, "barriers, passes");

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&kv_map);
    for (uint32_t i = 0; i < kRing; i++) { mbar_init(full(i), 1); mbar_init(empty(i), 2); }  // both groups read a tile
    for (uint32_t i = 0; i < kPpQSlots; i++) { mbar_init(q_full(i), 1); mbar_init(q_empty(i), 1); }
    for (uint32_t g = 0; g < 2; g++) {
      for (uint32_t w = 0; w < 2; w++) { mbar_init(s_full(g, w), 1); mbar_init(p_full(g, w), 4); mbar_init(pv_done(g, w), 1); }
      mbar_init(o_empty(g), 4);
    }
    for (uint32_t i = 0; i < kPpDesc; i++) { mbar_init(d_full(i), 1); mbar_init(d_empty(i), 11); }  // read by every warp but the producer
    mbar_init(clc_bar, 1);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // only now, with the allocation done: see attn_prefill_tc_kernel
  pdl_launch_dependents();
  pdl_wait();  // q and this chunk's K/V rows come from the previous kernels
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  const uint32_t s_base = tmem_base, o_base = tmem_base + 4 * kPpTile;  // S: two buffers for each group

  // every warp but the producer: the passes in turn
  uint32_t dk = 0;
  auto next_pass = [&] {
    const uint32_t s = dk % kPpDesc;
    mbar_wait(d_full(s), (dk / kPpDesc) & 1u);
    const PfPass p = desc[s];
    __syncwarp();
    if (lane == 0) mbar_arrive(d_empty(s));
    dk++;
    return p;
  };

  if (warp == 0) {
    // ===== producer: passes, key and value tiles; one lane acts, all hold page numbers =====
    const int page_size = 1 << page_shift, box_rows = min(page_size, 64);  // rows of the tensor map's box
    int x = blockIdx.x;
    uint32_t k = 0, dn = 0, asked = 0;
    auto push = [&](const PfPass &p) {
      const uint32_t s = dn % kPpDesc;
      if (dn >= kPpDesc) mbar_wait(d_empty(s), (dn / kPpDesc - 1) & 1u);
      if (lane == 0) {
        desc[s] = p;
        mbar_arrive(d_full(s));
      }
      __syncwarp();
      dn++;
    };
    auto ask = [&] {
      if (lane == 0) {
        fence_proxy_async();
        mbar_expect_tx(clc_bar, 16);
        clc_try_cancel(clc_resp, clc_bar);
      }
      __syncwarp();
    };
    for (;;) {
      // later query blocks of a sequence have more key tiles: first, so that the longest do not form the tail; the kv heads of a block
      // follow each other, or the tail would be one head's
      const int y = x % n_kv, b0 = 2 * ((n_blocks - 1) / 2 - x / n_kv), b1 = b0 + 1 < n_blocks ? b0 + 1 : b0;
      const int row[2] = {qb_ptrow[b0], qb_ptrow[b1]}, len[2] = {qb_len[b0], b1 > b0 ? qb_len[b1] : 0};
      const int pos0[2] = {qb_pos0[b0], qb_pos0[b1]}, tok0[2] = {qb_tok0[b0], qb_tok0[b1]};
      int n[2];
      for (int i = 0; i < 2; i++) n[i] = len[i] > 0 ? (pos0[i] + len[i] + kPpTile - 1) / kPpTile : 0;
      // blocks of different sequences share no tiles: one after the other
      const bool apart = row[0] != row[1] && n[0] > 0 && n[1] > 0;
      for (int pass = 0; pass < (apart ? 2 : 1); pass++) {
        PfPass p;
        int end = 0;
        for (int i = 0; i < 2; i++) {
          const bool in = !apart || i == pass;
          p.n[i] = in ? n[i] : 0;
          p.tok0[i] = tok0[i]; p.len[i] = len[i]; p.pos0[i] = pos0[i];
          if (p.n[i] > 0) end = max(end, pos0[i] + len[i]);
        }
        p.kvh = y;
        p.pad = 0;
        const int tiles = max(p.n[0], p.n[1]);
        const bool last_pass = pass == (apart ? 1 : 0);
        if (tiles > 0) push(p);
        const int *pt = page_table + (size_t)row[apart ? pass : (n[0] > 0 ? 0 : 1)] * max_pages;
        const int last_box = (end - 1) / box_rows * box_rows, last_page = last_box >> page_shift;
        PageWindow win[2];
        // K_0, K_1, V_0, K_2, V_1, ...: as the products take them
        for (int t = 0; t < 2 * tiles; t++, k++) {
          // the next pair is asked for as late as its answer still comes in time: one asked for early would wait here while others idle
          if (last_pass && t == max(2 * tiles - 4, 0)) ask();
          const bool is_v = t == 2 * tiles - 1 || (t > 0 && (t & 1) == 0);
          const int tile = t == 2 * tiles - 1 ? tiles - 1 : is_v ? t / 2 - 1 : (t + 1) / 2;
          const uint32_t s = k % kRing, bar = full(s), dst = ring_base + s * kSlot;
          if (k >= kRing) mbar_wait(empty(s), (k / kRing - 1) & 1u);
          if (lane == 0) mbar_expect_tx(bar, kSlot);
          for (int r = 0; r < kPpTile; r += box_rows) {
            // Boxes past the last key repeat the last one that holds a key: their scores are masked, and their values must be
            // finite because they are multiplied by a weight of zero.
            const int pos = min(tile * kPpTile + r, last_box);
            const long long page = is_v ? win[1].get(pt, pos >> page_shift, last_page) : win[0].get(pt, pos >> page_shift, last_page);
            const long long krow = row0 + ((page * 2 + (is_v ? 1 : 0)) * n_kv + y) * page_size + (pos & (page_size - 1));
            if (lane == 0) {
#pragma unroll
              for (int hh = 0; hh < kHalves; hh++) tma_load_2d(dst + hh * kPfHalf + r * 128, &kv_map, hh * 64, (int)krow, bar, kEvictLast);
            }
          }
          __syncwarp();
        }
        if (last_pass && tiles == 0) ask();
      }
      mbar_wait(clc_bar, asked & 1u);
      asked++;
      const bool more = clc_query(clc_resp, x);
      __syncwarp();
      if (!more) break;
    }
    PfPass p{};
    p.n[0] = p.n[1] = -1;
    push(p);
  } else if (warp < 3) {
    // ===== MMA issuers, a warp for each group: converged, one elected lane issues.  (One warp for both left the tensor pipe idle at each
    // of its waits.)  The group is a constant and the ring is walked in its order, so that little stands between a wait and its products. =====
    auto issuer = [&](auto group) {
      constexpr uint32_t g = decltype(group)::value;
      constexpr uint32_t idesc_s = umma_idesc<kPpTile>();
      constexpr uint32_t idesc_o = umma_idesc<D>() | (1u << 16);  // B (= V) MN-major
      const uint32_t q_lo = umma_lo(q_base) + 2 * g * (kQBytes >> 4), k_lo0 = umma_lo(ring_base), v_off = umma_lo_mn(ring_base, kPfHalf) - k_lo0;
      const uint32_t s_col = s_base + 2 * g * kPpTile, o_col = o_base + g * kOCols;
      uint32_t slot = 0, phase = 0, lo = k_lo0;                     // the ring's next tile
      uint32_t steps = 0, scores = 0, passes = 0, tiles_q = 0;      // the group's P V products, S products, passes, query tiles so far
      auto step_ring = [&] {
        lo += kSlot >> 4;
        if (++slot == kRing) { slot = 0; phase ^= 1u; lo = k_lo0; }
      };
      auto skip_tile = [&] {  // one that only the other group reads: its slot's phases are followed all the same
        mbar_wait(full(slot), phase);
        if (lane == 0) mbar_arrive(empty(slot));
        __syncwarp();
        step_ring();
      };
      auto issue_s = [&](bool first, bool last) {
        const uint32_t w = scores & 1u;
        if (first) mbar_wait(q_full(2 * g + (tiles_q & 1u)), (tiles_q >> 1) & 1u);
        mbar_wait(full(slot), phase);
        if (scores >= 2) mbar_wait(pv_done(g, w), ((scores >> 1) - 1) & 1u);  // S overwrites the columns that the P V two steps before it reads
        tc_fence_after();
        if (elect_one()) {
          const uint32_t qa = q_lo + (tiles_q & 1u) * (kQBytes >> 4), d = s_col + w * kPpTile;
#pragma unroll
          for (uint32_t k = 0; k < D / 16; k++)
            umma_ss(d, qa + (k >> 2) * (kPfQHalf >> 4) + (k & 3) * 2, lo + (k >> 2) * (kPfHalf >> 4) + (k & 3) * 2, idesc_s, k > 0 ? 1u : 0u);
          umma_commit(s_full(g, w));
          umma_commit(empty(slot));
          if (last) umma_commit(q_empty(2 * g + (tiles_q & 1u)));
        }
        __syncwarp();
        step_ring();
        scores++;
        tiles_q += last;
      };
      // Tiles come as K_0, K_1, V_0, K_2, V_1, ..., V_{tiles - 1}: S runs two steps ahead of P V, and on into the next pass, while this one's
      // output is read out.
      PfPass p = next_pass();
      int ahead = 0;  // scores of this pass issued during the one before
      while (p.n[0] >= 0) {
        const int n = p.n[g], tiles = max(p.n[0], p.n[1]);
        PfPass p2;
        int n2 = 0, ahead2 = 0;
        bool have2 = false;
        for (int j = ahead; j < min(tiles, 2); j++) {
          if (j < n) issue_s(j == 0, j == n - 1); else skip_tile();
        }
        for (int j = 0; j < tiles; j++) {
          if (j < n) {
            const uint32_t w = steps & 1u;
            mbar_wait(full(slot), phase);
            if (j == 0) {
              if (passes > 0) mbar_wait(o_empty(g), (passes - 1) & 1u);
              passes++;
            }
            mbar_wait(p_full(g, w), (steps >> 1) & 1u);
            tc_fence_after();
            if (elect_one()) {
              const uint32_t a = s_col + w * kPpTile, b = lo + v_off;
#pragma unroll
              for (uint32_t k = 0; k < kPpTile / 16; k++)
                umma_ts(o_col + (kOwn ? ((uint32_t)j & 1u) * D : 0u), a + 8 * k, b + k * 128, idesc_o, k > 0 ? 1u : (uint32_t)(j > (kOwn ? 1 : 0)));
              umma_commit(pv_done(g, w));
              umma_commit(empty(slot));
            }
            __syncwarp();
            step_ring();
            steps++;
          } else {
            skip_tile();
          }
          if (j + 2 < tiles) {
            if (j + 2 < n) issue_s(false, j + 2 == n - 1); else skip_tile();
          } else if (n > 0 && j == tiles - 1) {  // (every tile of this pass has been taken from the ring)
            p2 = next_pass();
            have2 = true;
            n2 = p2.n[g];
            for (; ahead2 < min(n2, 2); ahead2++) issue_s(ahead2 == 0, ahead2 == n2 - 1);
          }
        }
        if (!have2) p2 = next_pass();
        p = p2;
        ahead = ahead2;
      }
    };
    if (warp == 1) issuer(std::integral_constant<uint32_t, 0>{}); else issuer(std::integral_constant<uint32_t, 1>{});
  } else if (warp == 3) {
    // ===== query rows: row = head * QT + token, K-major, 128B swizzle (rows of padding tokens are zero) =====
    uint32_t qk[2] = {0u, 0u};
    for (PfPass p = next_pass(); p.n[0] >= 0; p = next_pass()) {
#pragma unroll
      for (int g = 0; g < 2; g++) {
        if (p.n[g] <= 0) continue;
        const uint32_t qi = qk[g]++, qs = 2 * g + (qi & 1u);
        if (qi >= 2) mbar_wait(q_empty(qs), ((qi >> 1) - 1) & 1u);
        const uint32_t dst = q_base + qs * kQBytes;
#pragma unroll 8
        for (int e = lane; e < 128 * (D / 8); e += 32) {
          const int row = e / (D / 8), c = e % (D / 8), hl = row / QT, t = row % QT;
          const bool in = t < p.len[g];
          const uint16_t *src = q + ((size_t)(p.tok0[g] + (in ? t : 0)) * n_heads + p.kvh * G + hl) * D + c * 8;
          cp_async_16(dst + (uint32_t)(c >> 3) * kPfQHalf + (uint32_t)(row >> 3) * 1024 + (uint32_t)(row & 7) * 128 + (uint32_t)(((c & 7) ^ (row & 7)) << 4), src, in ? 16 : 0);
        }
        cp_async_wait_all();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_full(qs));
      }
    }
  } else {
    // ===== softmax: group g has query tile g; one thread per row; O lives in TMEM =====
    const int quarter = warp & 3;  // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    const int g = (warp - 4) >> 2;
    const int row = quarter * 32 + lane, hl = row / QT, t = row % QT;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_addr0 = s_base + lane_off + 2 * g * kPpTile, o_addr = o_base + lane_off + g * kOCols;
    const float scale_log2 = rsqrtf((float)D) * 1.4426950408889634f;
    const float2 scale2 = make_float2(scale_log2, scale_log2);
    // The two warps of a quarter share an SM partition and its exponential unit, and left to themselves they run in step: both at the
    // exponentials (twice as long), then both at everything else.  So they take turns.
    const int my_turn = 1 + 4 * g + quarter, its_turn = 1 + 4 * (g ^ 1) + quarter;
    constexpr bool kTurns = D == 64;
    if (kTurns && g == 1) named_arrive_64(its_turn);
    const bool wide = (reinterpret_cast<uintptr_t>(out) & 31u) == 0;  // a row piece of 32 bytes is a whole sector
    uint32_t step = 0;
    for (PfPass p = next_pass(); p.n[0] >= 0; p = next_pass()) {
      const int n = g ? p.n[1] : p.n[0], tok0 = g ? p.tok0[1] : p.tok0[0], len = g ? p.len[1] : p.len[0], qp = (g ? p.pos0[1] : p.pos0[0]) + t;
      const int tiles = max(p.n[0], p.n[1]);
      float m_ref = kOwn ? -FLT_MAX : 0.f, l_run = 0.f;   // kOwn: of this tile's parity (finite where its first tile may hide every key of a row)
      float m_other = -FLT_MAX, l_other = 0.f;            // of the other parity
#pragma unroll 1
      for (int j = 0; j < n; j++, step++) {
        const uint32_t w = step & 1u, s_addr = s_addr0 + w * kPpTile;
        mbar_wait(s_full(g, w), (step >> 1) & 1u);
        tc_fence_after();
        uint32_t s[2][32];
        tmem_ld_32x32(s_addr, s[0]);
        tmem_ld_32x32(s_addr + 32, s[1]);
        tmem_ld_wait();
        const int rest = qp - j * kPpTile;  // keys 0 .. rest of the tile are visible
        if (rest < kPpTile - 1) {           // only the tiles that cross the diagonal need the causal mask
#pragma unroll
          for (int c = 0; c < 2; c++)
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (32 * c + i > rest) s[c][i] = 0xff800000u;
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; i++) mx4[i & 3] = max3(mx4[i & 3], __uint_as_float(s[0][i]), __uint_as_float(s[1][i]));
        const float mx = max3(mx4[0], mx4[1], fmaxf(mx4[2], mx4[3])) * scale_log2;  // scale > 0: it commutes with the maximum
        float f = 1.0f;
        bool rescale = false;
        if (kOwn) {
          const float m_now = fmaxf(m_ref, mx);
          rescale = j >= 2 && __any_sync(0xffffffffu, mx > m_ref);
          f = ex2_approx(m_ref - m_now);
          m_ref = m_now;
          l_run *= f;
        } else if (j == 0) {
          m_ref = mx;  // finite: key 0 is visible to every query; O is first written by P_0 V_0 (accumulate off)
        } else {
          const bool need = mx > m_ref + kPfLazy;
          rescale = __any_sync(0xffffffffu, need);  // tcgen05.ld / st are warp-collective: decide per warp, scale per lane
          if (need) {
            f = ex2_approx(m_ref - mx);
            m_ref = mx;
          }
        }
        if (kTurns) named_sync_64(my_turn);
        const float2 neg_m = make_float2(-m_ref, -m_ref);
        float2 ps[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float2 e = fma2(make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), scale2, neg_m);
            e.x = ex2_approx(e.x);
            e.y = ex2_approx(e.y);
            pk[i >> 1] = float2_to_bf16x2(e.x, e.y);
            // the sum takes the weights as P V takes them, rounded: a row that one key dominates keeps that key's weight at 1
            ps[(i >> 1) & 1] = add2(ps[(i >> 1) & 1], bf16x2_to_float2(pk[i >> 1]));
          }
          tmem_st_32x16(s_addr + 16 * c, pk);
        }
        if (kTurns) named_arrive_64(its_turn);
        if (rescale) {
          if (kOwn) {  // S was issued behind the P V of two tiles before: this parity's O is complete
            rescale_64(o_addr + ((uint32_t)j & 1u) * D, f);
          } else {  // behind the weights: the P V before this has had their time to end
            mbar_wait(pv_done(g, w ^ 1u), ((step - 1) >> 1) & 1u);
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < D; c += 64) rescale_64(o_addr + c, f);
            l_run *= f;
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(g, w));
        l_run += (ps[0].x + ps[0].y) + (ps[1].x + ps[1].y);
        if (kOwn) {
          const float m = m_ref, l = l_run;
          m_ref = m_other; l_run = l_other;
          m_other = m; l_other = l;
        }
      }
      if (kTurns)
        for (int j = max(n, 0); j < tiles; j++) {  // nothing to do while the other group works on
          named_sync_64(my_turn);
          named_arrive_64(its_turn);
        }
      if (n <= 0) continue;
      float inv, f0 = 1.f, f1 = 1.f;  // kOwn: what the even and the odd tiles' O are weighted with
      if (kOwn) {
        const bool last_odd = (n & 1) == 0;
        const float m0 = last_odd ? m_ref : m_other, m1 = last_odd ? m_other : m_ref, l0 = last_odd ? l_run : l_other, l1 = last_odd ? l_other : l_run;
        const float m = fmaxf(m0, m1);
        f0 = ex2_approx(m0 - m);
        f1 = ex2_approx(m1 - m);
        inv = 1.0f / (l0 * f0 + l1 * f1);
        f0 *= inv;
        f1 *= inv;
      } else {
        inv = 1.0f / l_run;
      }
      mbar_wait(pv_done(g, (step - 1) & 1u), ((step - 1) >> 1) & 1u);
      tc_fence_after();
      uint16_t *o = out + ((size_t)(tok0 + t) * n_heads + p.kvh * G + hl) * D;
#pragma unroll
      for (int c = 0; c < D; c += 64) {
        uint32_t v[2][32];
        tmem_ld_32x32(o_addr + c, v[0]);
        tmem_ld_32x32(o_addr + c + 32, v[1]);
        tmem_ld_wait();
        if (kOwn) {
#pragma unroll
          for (int i = 0; i < 64; i++) v[i >> 5][i & 31] = __float_as_uint(__uint_as_float(v[i >> 5][i & 31]) * f0);
          if (n > 1) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
              uint32_t u[32];
              tmem_ld_32x32(o_addr + D + 32 * h, u);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; i++) v[h][i] = __float_as_uint(fmaf(__uint_as_float(u[i]), f1, __uint_as_float(v[h][i])));
            }
          }
          inv = 1.f;
        }
        if (c == D - 64) {  // everything is in registers: the next pass may write O
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(o_empty(g));
        }
        if (t < len) {
          uint32_t r[32];
#pragma unroll
          for (int i = 0; i < 32; i++) r[i] = float2_to_bf16x2(__uint_as_float(v[i >> 4][(2 * i) & 31]) * inv, __uint_as_float(v[i >> 4][(2 * i + 1) & 31]) * inv);
          if (wide) {
#pragma unroll
            for (int i = 0; i < 32; i += 8)
              asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(o + (c + 2 * i)), "r"(r[i]), "r"(r[i + 1]), "r"(r[i + 2]), "r"(r[i + 3]), "r"(r[i + 4]), "r"(r[i + 5]), "r"(r[i + 6]), "r"(r[i + 7]) : "memory");
          } else {
#pragma unroll
            for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4 *>(o + c + 2 * i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
          }
        }
      }
    }
    if (kTurns && g == 0) named_sync_64(my_turn);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc<512>(tmem_base);
}

// DIS_ATTN_PREFILL=mma sends every geometry to the mma.sync kernel of k_attn_paged.cu (A/B runs).
static bool prefill_tc_enabled() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DIS_ATTN_PREFILL");
    v = e && !strcmp(e, "mma") ? 0 : 1;
  }
  return v != 0;
}

// Head sizes 128 and 64 with groups of 4 or 8 query heads per kv head.  Smaller groups stay on the mma.sync kernel: its blocks
// of 16 tokens would fill 16 or 32 of the 128 rows.
bool attn_prefill_uses_tc(int n_heads, int n_kv, int d) {
  if (n_kv <= 0 || n_heads % n_kv != 0) return false;
  const int G = n_heads / n_kv;
  return prefill_tc_enabled() && (d == 128 || d == 64) && (G == 4 || G == 8);
}

// q is read and out written 16 bytes at a time; rows of 64 or 128 bf16 keep the alignment of the first.
bool attn_prefill_tc_aligned(const uint16_t *q, const uint16_t *out) {
  return ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
}

// Most tokens a caller of the C ABI may put into one query block: 128 / G for heads of 128, 16 otherwise.
int attn_prefill_block_tokens(int n_heads, int n_kv, int d) {
  return d == 128 && attn_prefill_uses_tc(n_heads, n_kv, d) ? 128 / (n_heads / n_kv) : 16;
}
// The engine's own blocks: what the kernel takes.
int attn_prefill_full_block(int n_heads, int n_kv, int d) {
  return attn_prefill_uses_tc(n_heads, n_kv, d) ? 128 / (n_heads / n_kv) : 16;
}

template <class K, class... Args>
static cudaError_t prefill_tc_launch(K kern, dim3 grid, int threads, int smem, DeviceOnce &once, cudaStream_t st, const TmaMap &kv_map, Args... args) {
  DIS_CUDA_TRY(once.run([&] {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    return e;
  }));
  return launch_k(kern, grid, dim3(threads), (size_t)smem, st, *reinterpret_cast<const CUtensorMap *>(&kv_map), args...);
}

// A pair of blocks on an SM of its own pays where the GPU has more blocks than SMs to spread them on: us of one block per CTA / of pairs, by blocks
// times kv heads, heads of 128: 152 16.2 / 15.9, 208 12.9 / 13.6, 216 16.9 / 15.6, 304 25.8 / 24.8, 328 17.6 / 15.0, 560 39.5 / 30.4, 672 39.5 / 28.1.
// (Equal blocks that fill a little more than one round lose 5 to 14 %: 20 prompts of 33 tokens, 320, 10.8 / 12.0; blocks whose pairs are of two
// sequences likewise: 5 of 100 behind 700, 280, 22.0 / 25.4.)
// Heads of 64, whose single blocks run two to an SM with four softmax groups between them: 316 10.8 / 10.8, 320 27.6 / 35.4, and beyond that by the
// history that a block sees on average, up to which starts and ends weigh more: 80 prompts of 17 tokens 13.1 / 11.0, behind 700 35.2 / 41.2; ragged
// prompts (a quarter of the longest on average), eight to 700 tokens 20.9 / 19.9, six to 1900 69.2 / 66.4, three to 3333 134 / 140; one of 8000 364 / 405.
static bool prefill_in_pairs(int n_blocks, int n_kv, int d, long long mean_keys) {
  const long long n = (long long)n_blocks * n_kv;
  return n > (d == 128 ? 3 : 6) * kNumSMs / 2 && n < (1ll << 31) && (d == 128 || mean_keys <= 720);
}

// Same contract as launch_attn_prefill (k_attn_paged.cu) with query blocks of up to 128 / G tokens.
cudaError_t launch_attn_prefill_tc(const TmaMap &kv_map, long long row0, const uint16_t *q, const int *page_table,
                                   int max_pages, const int *qb_tok0, const int *qb_len, const int *qb_pos0,
                                   const int *qb_ptrow, uint16_t *out, int n_blocks, int n_heads, int n_kv, int d,
                                   int page_size, long long mean_keys, cudaStream_t st) {
  if (n_blocks <= 0) return cudaSuccess;
  if (n_kv <= 0 || n_heads % n_kv != 0 || n_kv > 65535) { set_last_error("attn_prefill_tc: bad head geometry"); return cudaErrorInvalidValue; }
  if (!attn_prefill_tc_aligned(q, out)) { set_last_error("attn_prefill_tc: q and out must start on 16 bytes"); return cudaErrorInvalidValue; }
  if (page_size < 8 || (page_size & (page_size - 1))) { set_last_error("attn_prefill_tc: page_size must be a power of two >= 8"); return cudaErrorInvalidValue; }
  int page_shift = 0;
  while ((1 << page_shift) < page_size) page_shift++;
  const int G = n_heads / n_kv;
#define DIS_PF_TC_CASE(DD, GG)                                                                                                   \
  if (d == DD && G == GG) {                                                                                                      \
    static DeviceOnce once, once_pair;                                                                                           \
    if (prefill_in_pairs(n_blocks, n_kv, DD, mean_keys))                                                                             \
      return prefill_tc_launch(attn_prefill_pair_kernel<DD, GG>, dim3((n_blocks + 1) / 2 * n_kv), kPpThreads, pp_smem_bytes<DD>(), once_pair, st, kv_map, \
                               row0, q, page_table, max_pages, qb_tok0, qb_len, qb_pos0, qb_ptrow, out, n_heads, n_kv, page_shift, n_blocks); \
    return prefill_tc_launch(attn_prefill_tc_kernel<DD, GG>, dim3(n_blocks, n_kv), kPfThreads, pf_smem_bytes<DD>(), once, st, kv_map, row0, q,        \
                             page_table, max_pages, qb_tok0, qb_len, qb_pos0, qb_ptrow, out, n_heads, n_kv, page_shift);        \
  }
  DIS_PF_TC_CASE(128, 4)
  DIS_PF_TC_CASE(128, 8)
  DIS_PF_TC_CASE(64, 4)
  DIS_PF_TC_CASE(64, 8)
#undef DIS_PF_TC_CASE
  set_last_error("attn_prefill_tc: head_dim must be 64 or 128 and the GQA group 4 or 8");
  return cudaErrorInvalidValue;
}

}  // namespace dis
