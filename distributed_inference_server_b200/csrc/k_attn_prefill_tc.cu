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

  // later query blocks of a sequence have more key tiles: launch them first, so that the longest CTAs do not form the tail
  const int qb = (int)gridDim.x - 1 - (int)blockIdx.x, kvh = blockIdx.y;
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
    // ===== TMA producer: K_t as soon as S_{t-2} has read its slot, V_t as soon as P_{t-2} V_{t-2} has =====
    if (lane == 0) {
      const int last_box = (end - 1) / box_rows * box_rows;
      auto load = [&](int tile, bool is_v) {
        const int w = tile & 1;
        const uint32_t full = is_v ? v_full(w) : k_full(w);
        if (tile >= 2) mbar_wait(is_v ? pv_done(w) : k_empty(w), (uint32_t)(tile / 2 - 1) & 1u);
        const uint32_t sbase = (is_v ? v_base : k_base) + w * kSlot;
        mbar_expect_tx(full, kSlot);
        for (int r = 0; r < kPfTile; r += box_rows) {
          // Boxes past the last key repeat the last one that holds a key: their scores are masked, and their values must be
          // finite because they are multiplied by a weight of zero.
          const int pos = min(tile * kPfTile + r, last_box);
          const long long page = pt[pos >> page_shift];
          const long long krow = row0 + ((page * 2 + (is_v ? 1 : 0)) * n_kv + kvh) * page_size + (pos & (page_size - 1));
#pragma unroll
          for (int hh = 0; hh < kHalves; hh++) tma_load_2d(sbase + hh * kPfHalf + r * 128, &kv_map, hh * 64, (int)krow, full, kEvictLast);
        }
      };
      for (int t = 0; t <= n_tiles; t++) {
        if (t < n_tiles) load(t, false);
        if (t >= 1) load(t - 1, true);
      }
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

template <class K>
static cudaError_t prefill_tc_launch(K kern, int threads, int smem, DeviceOnce &once, const TmaMap &kv_map, long long row0, const uint16_t *q,
                                     const int *page_table, int max_pages, const int *qb_tok0, const int *qb_len, const int *qb_pos0,
                                     const int *qb_ptrow, uint16_t *out, int n_blocks, int n_heads, int n_kv, int page_shift,
                                     cudaStream_t st) {
  DIS_CUDA_TRY(once.run([&] {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    return e;
  }));
  return launch_k(kern, dim3(n_blocks, n_kv), dim3(threads), (size_t)smem, st, *reinterpret_cast<const CUtensorMap *>(&kv_map), row0, q,
                  page_table, max_pages, qb_tok0, qb_len, qb_pos0, qb_ptrow, out, n_heads, n_kv, page_shift);
}

// Same contract as launch_attn_prefill (k_attn_paged.cu) with query blocks of up to 128 / G tokens.
cudaError_t launch_attn_prefill_tc(const TmaMap &kv_map, long long row0, const uint16_t *q, const int *page_table,
                                   int max_pages, const int *qb_tok0, const int *qb_len, const int *qb_pos0,
                                   const int *qb_ptrow, uint16_t *out, int n_blocks, int n_heads, int n_kv, int d,
                                   int page_size, cudaStream_t st) {
  if (n_blocks <= 0) return cudaSuccess;
  if (n_kv <= 0 || n_heads % n_kv != 0 || n_kv > 65535) { set_last_error("attn_prefill_tc: bad head geometry"); return cudaErrorInvalidValue; }
  if (!attn_prefill_tc_aligned(q, out)) { set_last_error("attn_prefill_tc: q and out must start on 16 bytes"); return cudaErrorInvalidValue; }
  if (page_size < 8 || (page_size & (page_size - 1))) { set_last_error("attn_prefill_tc: page_size must be a power of two >= 8"); return cudaErrorInvalidValue; }
  int page_shift = 0;
  while ((1 << page_shift) < page_size) page_shift++;
  const int G = n_heads / n_kv;
#define DIS_PF_TC_CASE(DD, GG, KERN, THREADS, SMEM)                                                                              \
  if (d == DD && G == GG) {                                                                                                      \
    static DeviceOnce once;                                                                                                      \
    return prefill_tc_launch(KERN, THREADS, SMEM, once, kv_map, row0, q, page_table, max_pages, qb_tok0, qb_len, qb_pos0, qb_ptrow, \
                             out, n_blocks, n_heads, n_kv, page_shift, st);                                                      \
  }
  DIS_PF_TC_CASE(128, 4, (attn_prefill_tc_kernel<128, 4>), kPfThreads, pf_smem_bytes<128>())
  DIS_PF_TC_CASE(128, 8, (attn_prefill_tc_kernel<128, 8>), kPfThreads, pf_smem_bytes<128>())
  DIS_PF_TC_CASE(64, 4, (attn_prefill_tc_kernel<64, 4>), kPfThreads, pf_smem_bytes<64>())
  DIS_PF_TC_CASE(64, 8, (attn_prefill_tc_kernel<64, 8>), kPfThreads, pf_smem_bytes<64>())
#undef DIS_PF_TC_CASE
  set_last_error("attn_prefill_tc: head_dim must be 64 or 128 and the GQA group 4 or 8");
  return cudaErrorInvalidValue;
}

}  // namespace dis
