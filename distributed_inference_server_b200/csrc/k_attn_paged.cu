// k_attn_paged.cu -- attention of single query tokens over a paged bf16 KV cache.
//
// One CTA handles one (query token, kv head, slice of the history) for all query heads of the GQA
// group, so K and V are read from HBM once per group; in ragged batches of long histories the CTAs of a
// cluster share the histories of up to eight tokens instead.  64-token K/V tiles are staged by TMA into
// 128B-swizzled shared memory through a 3-4 stage mbarrier ring (64-96 KB in flight per CTA, two
// or three CTAs per SM); K Q^T and V^T P^T run on mma.sync m16n8k16 (bf16 in, fp32 accumulate) with ldmatrix operand
// loads -- on CUDA cores the 4 FMA per KV byte of a 4:1 GQA group is issue-bound well below the HBM
// rate (measured: 56 us vs 5 us per layer at batch 32, ctx 512).  HBM-bound: algorithmic
// bytes = 2 (K,V) * ctx * n_kv * d * 2 B per query token (+ q and out, negligible).
//
// KV page pool layout, per layer: [page][2 (K,V)][n_kv][page_size][d] bf16 -- each (page, kv head)
// is one contiguous page_size*d block.
//
// With n_splits > 1 every slice writes (m, l, unnormalised o) to scratch and a combine pass merges
// them (flash-decoding); that keeps all 148 SMs busy at batch 1.
#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "../../include/dis_engine.h"
#include "kernels.h"
#include "ptx.cuh"

namespace dis {

constexpr int kAttnTile = 64;  // tokens per pipeline stage: 16 per warp of a group of four

template <int D>
struct AttnCfg {
  static constexpr int kHalves = D / 64;                                  // 128-byte column blocks per row
  static constexpr int kHalfBytes = kAttnTile * 128;                      // one [64 tokens][64 dims] block
  static constexpr int kStageBytes = 2 * kHalves * kHalfBytes;            // K tile + V tile, bf16
  static constexpr int kStages = D == 128 ? 3 : 4;                        // 96 KB / 64 KB -> two CTAs per SM
  static constexpr int kExtraBytes = 1024 + 128;                          // alignment slack + barriers
  static constexpr int kSmemBytes = kStages * kStageBytes + kExtraBytes;
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
// 2^x; results below 2^-126 are zero (as weights they are lost beside one of 1)
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// an 8x8 matrix of bf16 pairs transposed across the warp
__device__ __forceinline__ uint32_t movmatrix(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
// D(16x8, f32) += A(16x16, bf16, row) * B(16x8, bf16, col)
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// K/V tiles of 64 tokens arrive by TMA (a warp of its own, 128B-swizzled boxes of min(page,64) rows, mbarrier completion) into a 3-4 stage ring.
// A group of four warps takes a tile, each warp 16 of its 64 tokens, with an online-softmax state (m, l, O) of its own; the states are merged
// once at the end.  With two groups the tiles are taken in turn.
//
// What bounds it is HBM where the histories are alike; in a ragged batch the longest one, which a single CTA walks: the time of a tile
// in a warp is a chain of latencies (barrier, ldmatrix, MMAs, shuffles, exponential, MMAs).  Tokens are the MMAs' rows and the group's
// query heads (<= 8) their eight columns: S^T = K Q^T and O^T = V^T P^T fill the m16n8k16 shape, half the MMAs and half the accumulators (D / 2
// registers) of heads as 16 padded rows.  P^T is turned from accumulator to operand by movmatrix, and two accumulators halve S^T's chain of MMAs.
// From graphs, against heads as rows with weights in one half (32 / 8 heads of 128): 1 x 8000 keys 15.0 -> 14.7 us, 8 x 512 8.7 -> 8.5, 32 x 512
// 13.7 -> 13.9, 64 x 575 27.7 -> 28.4, 32 ragged ones of 500 to 6000 77.1 -> 74.9; heads of 64 (32 / 4): 32 x 512 9.1 -> 8.7, 64 x 2000 23.4 -> 24.4.
// Eight warps in two groups lose nearly everywhere (weights in one half: 8 x 512 9.4 us against 8.4, 32 x 512 14.6 / 13.8, 32 x 100 7.6 / 6.7: more to
// start, to merge and to keep resident); see attn_dispatch for where they stay.
//
// A weight goes into the V^T P^T product as two bf16, its upper half and the rest: rounded to one it was most of the error, the more so the fewer
// warps have a maximum (a weight of exactly 1) of their own.  Groups of up to four heads leave columns free, so a head has two: K Q^T forms its
// scores in both, and V^T P^T multiplies the halves in one product, to be added at the end.  Groups of eight take a second product (1 to 2 % of the
// time, 6 % where an SM has one CTA).  Error of 32 ragged histories against 64 bits, 2-norm: 1.91e-3 with one half and four warps, 1.87e-3 with
// eight, 1.66e-3 with two halves, which is the rounding of the output.
//
// A ragged batch in one wave is as slow as its longest history if every history has a CTA of its own.  So (kShared) the CTAs of a cluster lay
// the histories of up to eight tokens end to end and take equal shares; pieces of one history meet in the shared memory of the CTA that has its
// first: those 74.9 us are 53.8.  The cluster's start and end cost 2 to 3 us, the pieces as much again: attn_sharing_pays.  (Fetched one after the
// other, a load and a branch at a time, the pieces cost 5: 55.4.)
//
// Rows past the context inside a box hold stale (finite) cache contents and get probability 0; the
// engine zero-fills the pool once so that they can never be NaN.
// Decode steps fuse the RoPE + KV-write stage into this kernel (rope.qkv != nullptr): the CTA sums the split-K
// slices of the fused QKV projection for its query heads and -- if the new position falls in its split -- for
// its kv head, rotates q and k, writes the new K/V row to the page pool for later steps and patches it into
// the shared-memory tile that TMA fetched.  Because nothing but that one row depends on this step, the K/V
// stream is started BEFORE griddepcontrol.wait: attention's HBM traffic overlaps the QKV projection's tail.
struct AttnRope {
  const float *qkv;          // [S][T][(nh + 2 nkv) * d] fp32 split-K slices, or nullptr: q / pages are ready
  int n_partial;
  long long stride;
  const int *pos;            // [T]
  const float *cos_t, *sin_t;  // [max_ctx][d/2]
  uint16_t *kv_base;         // this layer's page pool
};

__device__ __forceinline__ float4 attn_sum_slices(const float *p, int n, long long stride) {
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int s = 0; s < n; s++) {
    const float4 v = *reinterpret_cast<const float4 *>(p + (size_t)s * stride);
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  return a;
}

// From another CTA's shared memory.  No memory clobber: several are in flight; they keep their order with the cluster barriers, which are volatile too.
__device__ __forceinline__ float2 ld_cluster2(const float2 *p, uint32_t rank) {
  uint32_t a;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 ld_cluster4(const float *p, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void attn_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

constexpr int kAttnMaxCluster = 8;  // the portable size

// kShared: a cluster's CTAs share the histories of as many tokens; otherwise a CTA has one slice of one history.  NG: groups of four computing warps
template <int D, int G, bool kShared, int NG>
__global__ void __launch_bounds__(NG * 128 + 32, 2)
attn_paged_kernel(const __grid_constant__ CUtensorMap kv_map, long long row0, const AttnRope rope, const uint16_t *__restrict__ q,
                  const int *__restrict__ page_table, int max_pages, const int *__restrict__ pt_row,
                  const int *__restrict__ ctx_len, uint16_t *__restrict__ out, float *__restrict__ scratch,
                  int n_splits, int T, int n_heads, int n_kv, int page_shift, int n_stages) {
  using Cfg = AttnCfg<D>;
  constexpr int kAttnThreads = NG * 128, kAttnWarps = NG * 4;  // those that compute
  static_assert(!kShared || NG == 1, "a shared history's stages are counted for one group");
  constexpr bool kTwice = G <= 4;  // a head has two columns: the weights' upper halves go through one, the rest through the other
  constexpr int KS = D / 16;  // k-steps of the K Q^T MMA, m-tiles of the V^T P^T MMA
  static_assert(kAttnWarps * G * D * 4 <= Cfg::kStageBytes, "the warps' states are merged in one stage");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // 128B swizzle atoms are 1024-byte aligned
  uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + n_stages * Cfg::kStageBytes;
  // A stage has a full barrier for each of the groups: tile i completes number i % (NG n_stages), whose phases then all belong to the
  // group that waits for it.  (With one per stage and three stages, a group that runs ahead would take the other group's phase for its own.)
  auto full_bar = [&](int tile) { return bar_base + 8u * (uint32_t)(tile % (NG * n_stages)); };
  auto empty_bar = [&](int s) { return bar_base + 64u + 8u * s; };

  const int kvh = blockIdx.y;
  const int rank = blockIdx.x, ranks = gridDim.x, per_cluster = kShared ? ranks / n_splits : 1;
  const int t0 = (int)blockIdx.z * per_cluster;
  const int count = kShared ? min(per_cluster, T - t0) : 1;
  const int h0 = kvh * G;  // first query head of this CTA (G = n_heads / n_kv)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tq = lane & 3;  // mma fragment coordinates

  __shared__ __align__(16) uint16_t s_q[G][D];
  __shared__ __align__(16) uint16_t s_kvnew[2][D];
  __shared__ float s_m[kAttnWarps][G], s_l[kAttnWarps][G];
  __shared__ __align__(16) float p_o[kShared ? 2 : 1][G][kShared ? D : 1];
  __shared__ float2 p_ml[2][G];  // pieces of a history: one begun by a CTA before, one that goes on in the next
  __shared__ int s_ctx[kAttnMaxCluster], s_row[kAttnMaxCluster];

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&kv_map);
    for (int s = 0; s < NG * n_stages; s++) mbar_init(full_bar(s), 1);
    for (int s = 0; s < n_stages; s++) mbar_init(empty_bar(s), 4);
    fence_barrier_init();
    fence_proxy_async();
  }
  pdl_launch_dependents();
  const bool fused = rope.qkv != nullptr;
  if (!fused) pdl_wait();  // q and this step's K/V rows come from the previous kernels
  int ctx_0 = 0, row_0 = 0;
  if (!kShared) {
    ctx_0 = ctx_len[t0];
    row_0 = pt_row[t0];
  } else if (threadIdx.x < (unsigned)count) {
    s_ctx[threadIdx.x] = ctx_len[t0 + threadIdx.x];
    s_row[threadIdx.x] = pt_row[t0 + threadIdx.x];
  }
  __syncthreads();

  const int page_size = 1 << page_shift;
  const int box_rows = min(page_size, kAttnTile);
  // ---- which tiles are this CTA's: [bound(rank), bound(rank + 1)) of the histories laid end to end
  auto tiles_of = [&](int i) { return max(1, ((kShared ? s_ctx[i] : ctx_0) + kAttnTile - 1) / kAttnTile); };
  int total = 0, most = 0;
  for (int i = 0; i < count; i++) {
    const int n = tiles_of(i);
    total += n;
    if (kShared) most = max(most, n);
  }
  // A history of its own for every n_splits CTAs, or equal shares of all where that is shorter by more than a piece's start and end cost
  const int share = kShared ? (total + ranks - 1) / ranks : 0;
  const bool level = kShared && most > (share + 2) * n_splits;
  const bool pieces = kShared && (level || n_splits > 1);  // (the same in every CTA of the cluster)
  auto bound = [&](int r) {
    if (!kShared) return min(total, r * ((total + n_splits - 1) / n_splits));
    if (level) return min(total, r * share);
    const int item = r / n_splits;
    int at = 0;
    for (int i = 0; i < min(item, count); i++) at += tiles_of(i);
    if (item >= count) return at;
    const int n = tiles_of(item);
    return at + min(n, (r % n_splits) * ((n + n_splits - 1) / n_splits));
  };
  const int lo = bound(rank), hi = bound(rank + 1);
  // f(history, first tile, end tile, tiles of the history) for every piece in [lo, hi); an empty history counts as a tile above, so that it has a
  // CTA, and as none here: nothing is fetched for it
  auto for_pieces = [&](auto f) {
    if constexpr (!kShared) {
      const bool some = ctx_0 > 0;
      f(0, some ? lo : 0, some ? hi : 0, some ? total : 0);  // (an empty slice writes an empty state)
    } else {
      for (int i = 0, at = 0; i < count && at < hi; i++) {
        const int n = tiles_of(i);
        const bool some = s_ctx[i] > 0;
        if (at + n > lo && hi > lo) f(i, some ? max(lo - at, 0) : 0, some ? min(hi - at, n) : 0, some ? n : 0);
        at += n;
      }
    }
  };

  // The last warp loads and does nothing else, the computing warps free a stage each for themselves: no barrier of the whole block per
  // tile (with one, the longest history of a ragged batch took 1.04 us per tile, without it 0.83).
  if (warp == kAttnWarps) {
    if (lane == 0) {
      int k = 0;  // stages handed out so far
      auto next_stage = [&] {
        const int stage = k % n_stages;
        if (k >= n_stages) mbar_wait(empty_bar(stage), (uint32_t)(k / n_stages - 1) & 1u);
        return stage;
      };
      for_pieces([&](int i, int a, int b, int n) {
        const int *pt = page_table + (size_t)(kShared ? s_row[i] : row_0) * max_pages;
        for (int tile = a; tile < b; tile++, k++) {
          // pool rows: [page][2 (K,V)][n_kv][page_size] of d elements each
          const uint32_t sbase = smem_base + next_stage() * Cfg::kStageBytes, bar = full_bar(k);
          mbar_expect_tx(bar, Cfg::kStageBytes);
          for (int r = 0; r < kAttnTile; r += box_rows) {
            const int pos = tile * kAttnTile + r;
            const long long page = pt[min(pos >> page_shift, max_pages - 1)];
            const long long krow = row0 + ((page * 2 + 0) * n_kv + kvh) * page_size + (pos & (page_size - 1));
            const long long vrow = krow + (long long)n_kv * page_size;
#pragma unroll
            for (int h = 0; h < Cfg::kHalves; h++) {
              tma_load_2d(sbase + h * Cfg::kHalfBytes + r * 128, &kv_map, h * 64, (int)krow, bar, kEvictFirst);
              tma_load_2d(sbase + (Cfg::kHalves + h) * Cfg::kHalfBytes + r * 128, &kv_map, h * 64, (int)vrow, bar, kEvictFirst);
            }
          }
        }
        if (kShared) {
          next_stage();  // one more, empty: the warps merge their states in it while the next piece's tiles are under way
          mbar_arrive(full_bar(k));
          k++;
        }
      });
    }
    __syncwarp();
    if (pieces) attn_cluster_sync();
    if (kShared) attn_cluster_sync();
    return;
  }
  auto sync_compute = [] { asm volatile("bar.sync 1, %0;" ::"n"(kAttnThreads) : "memory"); };  // the computing warps

  const float scale_log2 = rsqrtf((float)D) * 1.4426950408889634f;  // scores are kept in the log2 domain
  const int grp = warp >> 2, wtok = (warp & 3) * 16;                // this warp's token slice inside a tile
  const int mi = lane >> 3, mr = lane & 7;
  const int k_tok = wtok + (mi & 1) * 8 + mr, v_tok = wtok + (mi >> 1) * 8 + mr;  // the row whose address this lane gives ldmatrix
  if (fused) pdl_wait();  // the QKV projection's slices
  int k0 = 0, open = -1;  // stages consumed so far; the history whose first piece is here and goes on elsewhere
  for_pieces([&](int item, int a, int b, int n) {
    const int t = t0 + item, ctx = kShared ? s_ctx[item] : ctx_0;
    const int new_pos = ctx - 1;             // the position this decode step appends
    const bool owner = fused && b == n && b > a;  // the piece that holds it
    if (fused) {
      constexpr int HQ = D / 8;  // float4 rotate-half items per head
      const int nq = n_heads * D, nk = n_kv * D;
      const float *base = rope.qkv + (size_t)t * (nq + 2 * nk);
      const float *cs = rope.cos_t + (size_t)new_pos * (D / 2), *sn = rope.sin_t + (size_t)new_pos * (D / 2);
      for (int it = threadIdx.x; it < (G + 1) * HQ + D / 4; it += kAttnThreads) {
        if (it < (G + 1) * HQ) {
          const bool is_q = it < G * HQ;
          if (!is_q && !owner) continue;
          const int hh = is_q ? it / HQ : 0, i = (it % HQ) * 4;
          const int col = is_q ? (h0 + hh) * D + i : nq + kvh * D + i;
          const float4 va = attn_sum_slices(base + col, rope.n_partial, rope.stride);
          const float4 vb = attn_sum_slices(base + col + D / 2, rope.n_partial, rope.stride);
          const float4 c = *reinterpret_cast<const float4 *>(cs + i), sv = *reinterpret_cast<const float4 *>(sn + i);
          uint2 w0, w1;
          w0.x = float2_to_bf16x2(va.x * c.x - vb.x * sv.x, va.y * c.y - vb.y * sv.y);
          w0.y = float2_to_bf16x2(va.z * c.z - vb.z * sv.z, va.w * c.w - vb.w * sv.w);
          w1.x = float2_to_bf16x2(vb.x * c.x + va.x * sv.x, vb.y * c.y + va.y * sv.y);
          w1.y = float2_to_bf16x2(vb.z * c.z + va.z * sv.z, vb.w * c.w + va.w * sv.w);
          uint16_t *dst = is_q ? s_q[hh] : s_kvnew[0];
          *reinterpret_cast<uint2 *>(dst + i) = w0;
          *reinterpret_cast<uint2 *>(dst + D / 2 + i) = w1;
        } else if (owner) {
          const int i = (it - (G + 1) * HQ) * 4;
          const float4 v = attn_sum_slices(base + nq + nk + kvh * D + i, rope.n_partial, rope.stride);
          uint2 o;
          o.x = float2_to_bf16x2(v.x, v.y);
          o.y = float2_to_bf16x2(v.z, v.w);
          *reinterpret_cast<uint2 *>(s_kvnew[1] + i) = o;
        }
      }
      sync_compute();
      if (owner && threadIdx.x < 2 * (D / 8)) {  // the new row goes to the page pool for the steps to come
        const int kv = threadIdx.x / (D / 8), c = threadIdx.x % (D / 8);
        const long long page = page_table[(size_t)(kShared ? s_row[item] : row_0) * max_pages + (new_pos >> page_shift)];
        uint16_t *dst = rope.kv_base + ((((size_t)page * 2 + kv) * n_kv + kvh) * page_size + (new_pos & (page_size - 1))) * D + c * 8;
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(s_kvnew[kv] + c * 8);
      }
    }

    // ---- Q^T as the B operand: column g = head g; where the group leaves columns free, the next G repeat it (kTwice)
    uint32_t qb[KS][2];
#pragma unroll
    for (int ks = 0; ks < KS; ks++) {
      qb[ks][0] = 0u; qb[ks][1] = 0u;
      if (g < (kTwice ? 2 * G : G)) {
        const int hq = kTwice ? g % G : g;
        const uint16_t *qp = fused ? s_q[hq] + ks * 16 + tq * 2 : q + ((size_t)t * n_heads + h0 + hq) * D + ks * 16 + tq * 2;
        qb[ks][0] = *reinterpret_cast<const uint32_t *>(qp);
        qb[ks][1] = *reinterpret_cast<const uint32_t *>(qp + 8);
      }
    }

    float oacc[KS][4];  // O^T: dims 16 n + g (+ 8) of heads 2 tq (+ 1)
#pragma unroll
    for (int m = 0; m < KS; m++) { oacc[m][0] = 0.f; oacc[m][1] = 0.f; oacc[m][2] = 0.f; oacc[m][3] = 0.f; }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};  // heads 2 tq (+ 1); l_run: this thread's tokens (summed at the end)

    for (int tile = a + (NG > 1 ? grp : 0); tile < b; tile += NG) {
      const int k = k0 + tile - a, stage = k % n_stages;
      mbar_wait(full_bar(k), (uint32_t)(k / (NG * n_stages)) & 1u);
      const uint32_t ks_addr = smem_base + stage * Cfg::kStageBytes;
      const uint32_t vs_addr = ks_addr + Cfg::kHalves * Cfg::kHalfBytes;
      const int tile_len = min(kAttnTile, ctx - tile * kAttnTile);
      if (owner && tile == n - 1 && ((new_pos - tile * kAttnTile) >> 4) == (warp & 3)) {
        // the tile TMA fetched predates this step's K/V row: the warp that reads the row patches it in (same 128B swizzle as the TMA boxes)
        const int r = new_pos - tile * kAttnTile;
        if (lane < 2 * (D / 8)) {
          const int kv = lane / (D / 8), c = lane % (D / 8);
          const uint32_t dst = (kv ? vs_addr : ks_addr) + (c >> 3) * Cfg::kHalfBytes + r * 128 + (((c & 7) ^ (r & 7)) << 4);
          const uint4 v = *reinterpret_cast<const uint4 *>(s_kvnew[kv] + c * 8);
          asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
          fence_proxy_async();  // (a later tile may land in this stage)
        }
        __syncwarp();
      }
      if (wtok < tile_len) {  // warp-uniform (only a history's last tile is short)
        // ---- S^T = K Q^T for this warp's 16 tokens: tokens wtok + g (+ 8), heads 2 tq (+ 1); two accumulators halve the chain
        float sacc[2][4];
#pragma unroll
        for (int e = 0; e < 2; e++) { sacc[e][0] = 0.f; sacc[e][1] = 0.f; sacc[e][2] = 0.f; sacc[e][3] = 0.f; }
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
          const int c = ks * 2 + (mi >> 1);  // 16-byte chunk of the row
          uint32_t a0, a1, a2, a3;
          ldmatrix_x4(ks_addr + (c >> 3) * Cfg::kHalfBytes + k_tok * 128 + (((c & 7) ^ (k_tok & 7)) << 4), a0, a1, a2, a3);
          mma_bf16_16816(sacc[ks & 1], a0, a1, a2, a3, qb[ks][0], qb[ks][1]);
        }
        // ---- online softmax of the two heads
        const bool in0 = wtok + g < tile_len, in1 = wtok + g + 8 < tile_len;
        float p[4], corr[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          p[e] = in0 ? sacc[0][e] + sacc[1][e] : -INFINITY;
          p[2 + e] = in1 ? sacc[0][2 + e] + sacc[1][2 + e] : -INFINITY;
          float mx = fmaxf(p[e], p[2 + e]);
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
          const float m_new = fmaxf(m_run[e], mx * scale_log2);  // finite: token wtok is valid
          corr[e] = ex2_ftz(m_run[e] - m_new);      // 0 on the first tile
          m_run[e] = m_new;
          p[e] = ex2_ftz(fmaf(p[e], scale_log2, -m_new));
          p[2 + e] = ex2_ftz(fmaf(p[2 + e], scale_log2, -m_new));
        }
        l_run[0] = l_run[0] * corr[0] + (p[0] + p[2]);
        l_run[1] = l_run[1] * corr[1] + (p[1] + p[3]);
        const uint32_t p01 = float2_to_bf16x2(p[0], p[1]), p23 = float2_to_bf16x2(p[2], p[3]);
        const float2 r01 = bf16x2_to_float2(p01), r23 = bf16x2_to_float2(p23);
        const uint32_t q01 = float2_to_bf16x2(p[0] - r01.x, p[1] - r01.y), q23 = float2_to_bf16x2(p[2] - r23.x, p[3] - r23.y);
        // kTwice: columns G .. 2 G take the rest
        const bool rest = kTwice && tq * 2 >= G;
        const uint32_t pb0 = movmatrix(G == 1 ? (p01 & 0xffffu) | (q01 << 16) : rest ? q01 : p01), pb1 = movmatrix(G == 1 ? (p23 & 0xffffu) | (q23 << 16) : rest ? q23 : p23);
        const uint32_t pl0 = kTwice ? 0u : movmatrix(q01), pl1 = kTwice ? 0u : movmatrix(q23);
#pragma unroll
        for (int m = 0; m < KS; m++) { oacc[m][0] *= corr[0]; oacc[m][1] *= corr[1]; oacc[m][2] *= corr[0]; oacc[m][3] *= corr[1]; }
        // ---- O^T += V^T P^T : A = V^T by ldmatrix.trans of the [tokens][dims] tile
#pragma unroll
        for (int m = 0; m < KS; m++) {
          const int c = m * 2 + (mi & 1);
          uint32_t a0, a1, a2, a3;
          ldmatrix_x4_trans(vs_addr + (c >> 3) * Cfg::kHalfBytes + v_tok * 128 + (((c & 7) ^ (v_tok & 7)) << 4), a0, a1, a2, a3);
          mma_bf16_16816(oacc[m], a0, a1, a2, a3, pb0, pb1);
          if (!kTwice) mma_bf16_16816(oacc[m], a0, a1, a2, a3, pl0, pl1);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_bar(stage));
    }
    k0 += b - a;

    // ---- merge the warps' (m, l, O): [warps][G][D], a pair of heads 8 dims from the next (no bank twice).  Where a piece may follow, in the stage
    // that was handed out empty; where none does every load has been waited for, and behind the barrier any stage is free
    const int stage = kShared ? k0 % n_stages : 0;
    if (kShared) {
      mbar_wait(full_bar(k0), (uint32_t)(k0 / n_stages) & 1u);
      k0++;
    }
    sync_compute();
    if (kTwice) {
#pragma unroll
      for (int m = 0; m < KS; m++) {
        if (G == 1) {
          oacc[m][0] += oacc[m][1];
          oacc[m][2] += oacc[m][3];
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++) oacc[m][i] += __shfl_xor_sync(0xffffffffu, oacc[m][i], G / 2);
        }
      }
    }
    float *s_o = reinterpret_cast<float *>(smem + stage * Cfg::kStageBytes);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 4);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 8);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 16);
      const int hh = tq * 2 + e;
      if (hh < G) {
        float *o = s_o + (warp * G + hh) * D;
#pragma unroll
        for (int m = 0; m < KS; m++) { o[(m * 16 + g) ^ (tq * 8)] = oacc[m][e]; o[(m * 16 + 8 + g) ^ (tq * 8)] = oacc[m][2 + e]; }
        if (g == 0) { s_m[warp][hh] = m_run[e]; s_l[warp][hh] = l_run[e]; }
      }
    }
    sync_compute();
    const bool whole = kShared ? a == 0 && b == n : n_splits == 1;
    const int slot = a > 0 ? 0 : 1;
    if (kShared && !whole && slot == 1) open = item;
    for (int e = threadIdx.x; e < G * D; e += kAttnThreads) {
      const int hh = e / D, dd = e - hh * D;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < kAttnWarps; w++) M = fmaxf(M, s_m[w][hh]);
      float L = 0.f, o = 0.f;
#pragma unroll
      for (int w = 0; w < kAttnWarps; w++) {
        const float mw = s_m[w][hh];
        const float wgt = mw == -INFINITY ? 0.f : exp2f(mw - M);
        L += s_l[w][hh] * wgt;
        o += s_o[(w * G + hh) * D + (dd ^ ((hh >> 1) * 8))] * wgt;
      }
      const int h = h0 + hh;
      if (whole) {
        out[((size_t)t * n_heads + h) * D + dd] = float_to_bf16_bits(o / L);
      } else if constexpr (kShared) {
        p_o[slot][hh][dd] = o;
        if (dd == 0) p_ml[slot][hh] = make_float2(M, L);
      } else {
        // scratch: ml [T][n_heads][S][2] then o [T][n_heads][S][D]; m is in the log2 domain
        float *ml = scratch + (((size_t)t * n_heads + h) * n_splits + rank) * 2;
        float *op = scratch + (size_t)T * n_heads * n_splits * 2 + (((size_t)t * n_heads + h) * n_splits + rank) * D;
        op[dd] = o;
        if (dd == 0) { ml[0] = M; ml[1] = L; }
      }
    }
    if (kShared) {
      fence_proxy_async();  // (plain accesses to a stage that TMA will fill again)
      sync_compute();
      if (lane == 0) mbar_arrive(empty_bar(stage));
    }
  });
  // ---- pieces of one history in several CTAs: the CTA that holds its first piece reads the others' out of their shared memory
  if constexpr (kShared) {
    if (pieces) attn_cluster_sync();
    if (open >= 0) {
      int end = 0;
      for (int i = 0; i <= open; i++) end += tiles_of(i);
      int last = rank + 1;  // the CTAs rank + 1 .. last hold the rest
      while (bound(last + 1) < end) last++;
      for (int e = threadIdx.x * 4; e < G * D; e += kAttnThreads * 4) {
        const int hh = e / D, dd = e - hh * D;
        // all of them at once (the last one again where there are fewer): one after the other they took 0.2 us each
        float2 ml[kAttnMaxCluster];
        float4 po[kAttnMaxCluster];
        ml[0] = p_ml[1][hh];
        po[0] = *reinterpret_cast<const float4 *>(&p_o[1][hh][dd]);
#pragma unroll
        for (int r = 1; r < kAttnMaxCluster; r++) ml[r] = ld_cluster2(&p_ml[0][hh], (uint32_t)min(rank + r, last));
#pragma unroll
        for (int r = 1; r < kAttnMaxCluster; r++) po[r] = ld_cluster4(&p_o[0][hh][dd], (uint32_t)min(rank + r, last));
        float M = ml[0].x;
#pragma unroll
        for (int r = 1; r < kAttnMaxCluster; r++) M = fmaxf(M, ml[r].x);
        float L = 0.f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < kAttnMaxCluster; r++) {
          const float w = rank + r <= last ? exp2f(ml[r].x - M) : 0.f;  // every piece holds a visible key
          L = fmaf(ml[r].y, w, L);
          o.x = fmaf(po[r].x, w, o.x); o.y = fmaf(po[r].y, w, o.y); o.z = fmaf(po[r].z, w, o.z); o.w = fmaf(po[r].w, w, o.w);
        }
        uint16_t *to = out + ((size_t)(t0 + open) * n_heads + h0 + hh) * D + dd;  // (out may start on any element)
        to[0] = float_to_bf16_bits(o.x / L); to[1] = float_to_bf16_bits(o.y / L); to[2] = float_to_bf16_bits(o.z / L); to[3] = float_to_bf16_bits(o.w / L);
      }
    }
    // nobody leaves while its pieces are read; without pieces either, so that a cluster of the next launch finds eight places at once
    // (32 equal histories of 6000: 134 us where each CTA left by itself)
    attn_cluster_sync();
  }
}

// ---------------------------------------------------------------------------------------- prefill
// Attention of a BLOCK of up to 16 consecutive query tokens of one sequence.
// One CTA = (query block, kv head); warp w owns query head h0 + w: a 16-row MMA tile whose rows are the
// block's tokens.  All warps walk the same 64-token K/V tiles (TMA ring shared by the GQA group, so K/V
// are read once per 16 tokens x G heads), causal mask by position, online softmax per row, P in bf16.
template <int D, int G>
__global__ void __launch_bounds__(G * 32)
attn_prefill_kernel(const __grid_constant__ CUtensorMap kv_map, long long row0, const uint16_t *__restrict__ q,
                    const int *__restrict__ page_table, int max_pages, const int *__restrict__ qb_tok0,
                    const int *__restrict__ qb_len, const int *__restrict__ qb_pos0, const int *__restrict__ qb_ptrow,
                    uint16_t *__restrict__ out, int n_heads, int n_kv, int page_shift) {
  using Cfg = AttnCfg<D>;
  constexpr int KS = D / 16, NT = D / 8;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + Cfg::kStages * Cfg::kStageBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };

  const int qb = blockIdx.x, kvh = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tq = lane & 3;
  const int h = kvh * G + warp;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&kv_map);
    for (int s = 0; s < Cfg::kStages; s++) mbar_init(full_bar(s), 1);
    fence_barrier_init();
    fence_proxy_async();
  }
  pdl_launch_dependents();
  pdl_wait();
  __syncthreads();

  const int tok0 = qb_tok0[qb], len = qb_len[qb], pos0 = qb_pos0[qb];
  const int *pt = page_table + (size_t)qb_ptrow[qb] * max_pages;
  const int page_size = 1 << page_shift;
  const int box_rows = min(page_size, kAttnTile);
  const int end = pos0 + len;  // keys [0, end)
  const int n_tiles = (end + kAttnTile - 1) / kAttnTile;

  auto load_tile = [&](int tile, int stage) {  // one thread
    const int tile0 = tile * kAttnTile;
    const uint32_t sbase = smem_base + stage * Cfg::kStageBytes;
    mbar_expect_tx(full_bar(stage), Cfg::kStageBytes);
    for (int r = 0; r < kAttnTile; r += box_rows) {
      const int pos = tile0 + r;
      const long long page = pt[min(pos >> page_shift, max_pages - 1)];
      const long long krow = row0 + ((page * 2 + 0) * n_kv + kvh) * page_size + (pos & (page_size - 1));
      const long long vrow = krow + (long long)n_kv * page_size;
#pragma unroll
      for (int hh = 0; hh < Cfg::kHalves; hh++) {
        tma_load_2d(sbase + hh * Cfg::kHalfBytes + r * 128, &kv_map, hh * 64, (int)krow, full_bar(stage), kEvictLast);
        tma_load_2d(sbase + (Cfg::kHalves + hh) * Cfg::kHalfBytes + r * 128, &kv_map, hh * 64, (int)vrow, full_bar(stage), kEvictLast);
      }
    }
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < Cfg::kStages - 1; s++)
      if (s < n_tiles) load_tile(s, s);

  // ---- Q fragments: rows g and g+8 are tokens tok0+g, tok0+g+8 of head h
  uint32_t qa[KS][4];
  {
    const bool v0 = g < len, v1 = g + 8 < len;
    const uint16_t *q0 = q + ((size_t)(tok0 + g) * n_heads + h) * D + tq * 2;
    const uint16_t *q1 = q + ((size_t)(tok0 + g + 8) * n_heads + h) * D + tq * 2;
#pragma unroll
    for (int ks = 0; ks < KS; ks++) {
      qa[ks][0] = v0 ? *reinterpret_cast<const uint32_t *>(q0 + ks * 16) : 0u;
      qa[ks][1] = v1 ? *reinterpret_cast<const uint32_t *>(q1 + ks * 16) : 0u;
      qa[ks][2] = v0 ? *reinterpret_cast<const uint32_t *>(q0 + ks * 16 + 8) : 0u;
      qa[ks][3] = v1 ? *reinterpret_cast<const uint32_t *>(q1 + ks * 16 + 8) : 0u;
    }
  }
  const float scale_log2 = rsqrtf((float)D) * 1.4426950408889634f;
  float oacc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; n++) { oacc[n][0] = 0.f; oacc[n][1] = 0.f; oacc[n][2] = 0.f; oacc[n][3] = 0.f; }
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  const int qp0 = pos0 + g, qp1 = pos0 + g + 8;  // query positions of this thread's two rows

  for (int tile = 0; tile < n_tiles; tile++) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const int nt = tile + Cfg::kStages - 1;
      if (nt < n_tiles) load_tile(nt, nt % Cfg::kStages);
    }
    const int stage = tile % Cfg::kStages;
    mbar_wait(full_bar(stage), (uint32_t)(tile / Cfg::kStages) & 1u);
    const uint32_t ks_addr = smem_base + stage * Cfg::kStageBytes;
    const uint32_t vs_addr = ks_addr + Cfg::kHalves * Cfg::kHalfBytes;
    const int tile0 = tile * kAttnTile;

    // ---- S = Q K^T : 16 rows x 64 keys
    float sacc[8][4];
#pragma unroll
    for (int n = 0; n < 8; n++) { sacc[n][0] = 0.f; sacc[n][1] = 0.f; sacc[n][2] = 0.f; sacc[n][3] = 0.f; }
    {
      const int mi = lane >> 3, r = lane & 7;
#pragma unroll
      for (int ks = 0; ks < KS; ks++) {
        const int c = ks * 2 + (mi & 1);
#pragma unroll
        for (int np = 0; np < 4; np++) {  // n-tile pairs
          const int tok = np * 16 + (mi >> 1) * 8 + r;
          uint32_t b0, b1, b2, b3;
          ldmatrix_x4(ks_addr + (c >> 3) * Cfg::kHalfBytes + tok * 128 + (((c & 7) ^ (tok & 7)) << 4), b0, b1, b2, b3);
          mma_bf16_16816(sacc[2 * np], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
          mma_bf16_16816(sacc[2 * np + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
        }
      }
    }
    // ---- causal mask + online softmax (rows g and g+8)
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < 8; n++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int kp = tile0 + n * 8 + tq * 2 + e;
        const float v0 = kp <= qp0 ? sacc[n][e] * scale_log2 : -INFINITY;
        const float v1 = kp <= qp1 ? sacc[n][2 + e] * scale_log2 : -INFINITY;
        sacc[n][e] = v0; sacc[n][2 + e] = v1;
        mx0 = fmaxf(mx0, v0); mx1 = fmaxf(mx1, v1);
      }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
    // a row with nothing visible yet keeps m = -inf: use 0 as the reference so exp2(-inf - 0) = 0
    const float r0 = mn0 == -INFINITY ? 0.f : mn0, r1 = mn1 == -INFINITY ? 0.f : mn1;
    const float c0 = exp2f(m_run[0] - r0), c1 = exp2f(m_run[1] - r1);
    m_run[0] = mn0; m_run[1] = mn1;
    float ps0 = 0.f, ps1 = 0.f;
    uint32_t pa[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      const float a0 = exp2f(sacc[2 * kk][0] - r0), a1 = exp2f(sacc[2 * kk][1] - r0);
      const float b0 = exp2f(sacc[2 * kk][2] - r1), b1 = exp2f(sacc[2 * kk][3] - r1);
      const float c2 = exp2f(sacc[2 * kk + 1][0] - r0), c3 = exp2f(sacc[2 * kk + 1][1] - r0);
      const float d0 = exp2f(sacc[2 * kk + 1][2] - r1), d1 = exp2f(sacc[2 * kk + 1][3] - r1);
      ps0 += a0 + a1 + c2 + c3;
      ps1 += b0 + b1 + d0 + d1;
      pa[kk][0] = float2_to_bf16x2(a0, a1); pa[kk][1] = float2_to_bf16x2(b0, b1);
      pa[kk][2] = float2_to_bf16x2(c2, c3); pa[kk][3] = float2_to_bf16x2(d0, d1);
    }
    l_run[0] = l_run[0] * c0 + ps0;
    l_run[1] = l_run[1] * c1 + ps1;
#pragma unroll
    for (int n = 0; n < NT; n++) { oacc[n][0] *= c0; oacc[n][1] *= c0; oacc[n][2] *= c1; oacc[n][3] *= c1; }
    // ---- O += P V
    {
      const int mi = lane >> 3, r = lane & 7;
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        const int tok = kk * 16 + (mi & 1) * 8 + r;
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
          const int c = n + (mi >> 1);
          uint32_t b0, b1, b2, b3;
          ldmatrix_x4_trans(vs_addr + (c >> 3) * Cfg::kHalfBytes + tok * 128 + (((c & 7) ^ (tok & 7)) << 4), b0, b1, b2, b3);
          mma_bf16_16816(oacc[n], pa[kk][0], pa[kk][1], pa[kk][2], pa[kk][3], b0, b1);
          mma_bf16_16816(oacc[n + 1], pa[kk][0], pa[kk][1], pa[kk][2], pa[kk][3], b2, b3);
        }
      }
    }
  }
  // ---- normalise and store rows g, g+8
  l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], 1); l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], 2);
  l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], 1); l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], 2);
  const float i0 = 1.0f / l_run[0], i1 = 1.0f / l_run[1];
  if (g < len) {
    uint16_t *o = out + ((size_t)(tok0 + g) * n_heads + h) * D + tq * 2;
#pragma unroll
    for (int n = 0; n < NT; n++) *reinterpret_cast<uint32_t *>(o + n * 8) = float2_to_bf16x2(oacc[n][0] * i0, oacc[n][1] * i0);
  }
  if (g + 8 < len) {
    uint16_t *o = out + ((size_t)(tok0 + g + 8) * n_heads + h) * D + tq * 2;
#pragma unroll
    for (int n = 0; n < NT; n++) *reinterpret_cast<uint32_t *>(o + n * 8) = float2_to_bf16x2(oacc[n][2] * i1, oacc[n][3] * i1);
  }
}

template <int D>
__global__ void attn_combine_kernel(const float *__restrict__ scratch, uint16_t *__restrict__ out, int n_splits,
                                    int T, int n_heads) {
  const int t = blockIdx.y, h = blockIdx.x, dd = threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const float *ml = scratch + ((size_t)t * n_heads + h) * n_splits * 2;
  const float *op = scratch + (size_t)T * n_heads * n_splits * 2 + ((size_t)t * n_heads + h) * n_splits * D;
  float M = -INFINITY;
  for (int s = 0; s < n_splits; s++) M = fmaxf(M, ml[2 * s]);
  float L = 0.f, o = 0.f;
  for (int s = 0; s < n_splits; s++) {
    const float w = ml[2 * s] == -INFINITY ? 0.f : exp2f(ml[2 * s] - M);
    L += ml[2 * s + 1] * w;
    o += op[(size_t)s * D + dd] * w;
  }
  out[((size_t)t * n_heads + h) * D + dd] = float_to_bf16_bits(o / L);
}

// Whole histories can be shared as far as the clusters that have eight tokens run at once (33 of two CTAs per SM by the occupancy query of one
// B200): 36 of them in two rounds take 30.2 us where single CTAs take 23.8 (heads of 64, 72 histories of up to 2500).
constexpr int kAttnClusters = 32;
bool attn_may_share(int n_splits, int T, int n_kv) {
  const long long full = T >= kAttnMaxCluster ? (long long)(T / kAttnMaxCluster) * n_kv : ((long long)T * n_kv + kAttnMaxCluster - 1) / kAttnMaxCluster;
  return n_splits == 1 && T > 1 && full <= kAttnClusters && (long long)T * n_kv <= 2 * kNumSMs;
}
// A history's two to eight slices in one cluster, which joins them itself: no combine pass, but from graphs it takes longer (1 x 512 keys 6.2 -> 7.9 us, 8 x
// 512 8.5 -> 11.1, 8 x 2000 15.7 -> 18.3: a cluster starts and ends later than its CTAs alone).  A call of its own saves its caller a launch, 2 us.
static bool attn_may_join(int n_splits, int T, int n_kv) {
  const int per = kAttnMaxCluster / n_splits;
  return n_splits <= kAttnMaxCluster && (long long)((T + per - 1) / per) * n_kv <= kAttnClusters;
}
// Which takes longer, us: the longest history alone or the largest share of a cluster (0.8 us a tile of heads of 128, 0.5 of 64), the largest of the
// clusters that have to wait on top, neither less than the stream of all keys and values at 6.5 TB/s; sharing costs 6.  Of 29 ragged and 19 equal
// batches (heads of 128: 20 and 32 histories, of 64: 40 and 64; 100 to 7000 keys) it takes the slower form of two, by 3 and 7 %.
bool attn_sharing_pays(const int *ctx, int T, int n_kv, int d) {
  const int n = T < kAttnMaxCluster ? T : kAttnMaxCluster, at_once = std::max(1, kAttnClusters / n_kv);
  long long total = 0, most = 0, share = 0, later = 0;
  for (int t0 = 0, k = 0; t0 < T; t0 += n, k++) {
    long long sum = 0;
    for (int t = t0; t < std::min(t0 + n, T); t++) {
      const long long tiles = std::max(1, (ctx[t] + kAttnTile - 1) / kAttnTile);
      sum += tiles;
      most = std::max(most, tiles);
    }
    total += sum;
    long long &round = T >= kAttnMaxCluster && k >= at_once ? later : share;
    round = std::max(round, (sum + n - 1) / n);
  }
  const double tile = d == 128 ? 0.8 : 0.5, stream = (double)total * n_kv * (kAttnTile * d * 4) / 6.5e6;  // us
  return std::max((share + later) * tile, stream) + 6.0 < std::max(most * tile, stream);
}

size_t attn_scratch_elems(int T, int n_heads, int d, int n_splits) {
  if (n_splits <= 1) return 0;
  return (size_t)T * n_heads * n_splits * (2 + (size_t)d);
}

template <int D, int G, int NG, bool kShared>
static cudaError_t attn_launch(const TmaMap &kv_map, long long row0, const AttnRope &rope, const uint16_t *q, const int *page_table,
                               int max_pages, const int *pt_row, const int *ctx, uint16_t *out, float *scratch,
                               int n_splits, int T, int n_heads, int n_kv, int page_shift, cudaStream_t st) {
  auto kern = attn_paged_kernel<D, G, kShared, NG>;
  static DeviceOnce once;
  DIS_CUDA_TRY(once.run([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnCfg<D>::kSmemBytes); }));
  // ring depth: fewer stages leave shared memory for the NEXT kernel's CTAs to become resident (and prefetch their
  // weights) while this one is still streaming; DIS_ATTN_STAGES overrides (A/B runs), 2 <= stages <= AttnCfg::kStages
  static int stages = 0;
  if (stages == 0) {
    const char *e = getenv("DIS_ATTN_STAGES");
    stages = e ? atoi(e) : AttnCfg<D>::kStages;
    stages = stages < 2 ? 2 : (stages > AttnCfg<D>::kStages ? AttnCfg<D>::kStages : stages);
  }
  const int smem = stages * AttnCfg<D>::kStageBytes + AttnCfg<D>::kExtraBytes;
  const int per_cluster = kShared ? std::min(T, kAttnMaxCluster / n_splits) : 1, ranks = per_cluster * n_splits;
  DIS_CUDA_TRY(launch_k_cluster(kern, dim3(ranks, n_kv, (T + per_cluster - 1) / per_cluster), dim3(NG * 128 + 32), (size_t)smem, st, kShared ? ranks : 1,
                                *reinterpret_cast<const CUtensorMap *>(&kv_map), row0, rope, q, page_table, max_pages, pt_row, ctx, out,
                                scratch, n_splits, T, n_heads, n_kv, page_shift, stages));
  if (n_splits > 1 && !kShared)
    DIS_CUDA_TRY(launch_k(attn_combine_kernel<D>, dim3(n_heads, T), dim3(D), 0, st, (const float *)scratch, out, n_splits, T, n_heads));
  return cudaSuccess;
}

// The pool as a 2-D tensor of d-element rows, boxes of {64 dims, min(page_size, 64) rows}, 128B swizzle.
cudaError_t make_kv_map(TmaMap *out, const uint16_t *pool, long long total_rows, int d, int page_size) {
  return make_tma_map_2d(out, pool, (uint64_t)total_rows, (uint64_t)d, (uint32_t)(page_size < kAttnTile ? page_size : kAttnTile));
}

static cudaError_t attn_dispatch(const TmaMap &kv_map, long long row0, const AttnRope &rope, const uint16_t *q,
                                 const int *page_table, int max_pages, const int *pt_row, const int *ctx, uint16_t *out,
                                 float *scratch, int n_splits, int T, int n_heads, int n_kv, int d, int page_size,
                                 bool share, cudaStream_t st) {
  if (T <= 0) return cudaSuccess;
  if (n_kv <= 0 || n_heads % n_kv != 0) { set_last_error("attn_paged: n_heads must be a multiple of n_kv"); return cudaErrorInvalidValue; }
  if (n_splits < 1 || (n_splits > 1 && !scratch)) { set_last_error("attn_paged: n_splits > 1 needs scratch"); return cudaErrorInvalidValue; }
  if (T > 65535 || n_kv > 65535) { set_last_error("attn_paged: more than 65535 tokens or kv heads per launch"); return cudaErrorInvalidValue; }
  if (page_size < 8 || (page_size & (page_size - 1))) { set_last_error("attn_paged: page_size must be a power of two >= 8"); return cudaErrorInvalidValue; }
  int page_shift = 0;
  while ((1 << page_shift) < page_size) page_shift++;
  const int G = n_heads / n_kv;  // query heads per kv head, all handled by one CTA
  share = share && (n_splits > 1 ? attn_may_join(n_splits, T, n_kv) : attn_may_share(n_splits, T, n_kv));
  // Heads of 64: three CTAs of four computing warps fit an SM, or two of eight.  Just above three per SM the former leave most of a second round
  // empty, the latter fill theirs: 512 CTAs, 2500 keys 64.3 -> 55.3 us, 700 22.0 -> 20.2, 200 11.6 -> 11.7; 448 x 2500 58.2 -> 54.2 (200 keys 10.5 -> 11.1).
  // Elsewhere four warps are ahead: 304 x 700 12.1 against 17.8, 640 x 700 23.9 against 28.5, 1024 x 2500 103.8 against 110.1.
  const long long ctas = (long long)n_splits * T * n_kv;
  const bool two_groups = d == 64 && ctas > 3 * kNumSMs && ctas <= 4 * kNumSMs;
#define DIS_ATTN_GO(DD, GG, NG, SH) \
  attn_launch<DD, GG, NG, SH>(kv_map, row0, rope, q, page_table, max_pages, pt_row, ctx, out, scratch, n_splits, T, n_heads, n_kv, page_shift, st)
#define DIS_ATTN_CASE(DD, GG)                                               \
  if (d == DD && G == GG) {                                                 \
    if (share) return DIS_ATTN_GO(DD, GG, 1, true);                         \
    if constexpr (DD == 64) {                                               \
      if (two_groups) return DIS_ATTN_GO(DD, GG, 2, false);                 \
    }                                                                       \
    return DIS_ATTN_GO(DD, GG, 1, false);                                   \
  }
  DIS_ATTN_CASE(128, 8) DIS_ATTN_CASE(128, 4) DIS_ATTN_CASE(128, 2) DIS_ATTN_CASE(128, 1)
  DIS_ATTN_CASE(64, 8) DIS_ATTN_CASE(64, 4) DIS_ATTN_CASE(64, 2) DIS_ATTN_CASE(64, 1)
#undef DIS_ATTN_CASE
#undef DIS_ATTN_GO
  set_last_error("attn_paged: head_dim must be 64 or 128 and the GQA group 1, 2, 4 or 8");
  return cudaErrorInvalidValue;
}

static bool captured(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) == cudaSuccess) return cs != cudaStreamCaptureStatusNone;
  (void)cudaGetLastError();  // (another thread captures what the legacy stream would have to wait for: the launch says so)
  return true;
}
cudaError_t launch_attn_paged(const TmaMap &kv_map, long long row0, const uint16_t *q, const int *page_table,
                              int max_pages, const int *pt_row, const int *ctx, uint16_t *out, float *scratch,
                              int n_splits, int T, int n_heads, int n_kv, int d, int page_size, cudaStream_t st) {
  AttnRope none{};
  // The lengths are on the device; the page table's width bounds them, and from about these on a ragged batch gains (us, whole / shared; heads of 128, 32
  // histories of up to 1100 17.9 / 17.9, 1500 22.3 / 20.5, 2000 28.3 / 25.0, 7000 87.1 / 62.3, 20 of up to 1100 15.2 / 16.4, 1500 19.2 / 18.3; heads of
  // 64, 64 of up to 1100 13.1 / 14.5, 1500 16.4 / 16.0, 4500 39.1 / 27.1, 40 of up to 1500 14.6 / 15.5, 2000 18.2 / 16.9).  Where clusters have to wait,
  // those of the last tokens, it takes longer ones: 36 of up to 2500 33.8 / 33.7, 6000 74.1 / 57.9.  Equal histories lose: 32 x 2000 42.6 / 45.0, 32 x 6000
  // 115.1 / 119.7, heads of 64, 64 x 4000 43.0 / 45.1.
  const bool waits = (long long)((T + kAttnMaxCluster - 1) / kAttnMaxCluster) * n_kv > kAttnClusters && T >= kAttnMaxCluster;
  const long long keys = (long long)max_pages * page_size;
  bool share = keys > (waits ? 2560 : d == 128 ? 1280 : 1664);
  // Slices are joined in their cluster where the call is not captured and so short that its caller's time counts: up to 16 MB of keys and values
  if (n_splits > 1) share = T * keys * n_kv * d * 4 <= (16ll << 20) && !captured(st);
  return attn_dispatch(kv_map, row0, none, q, page_table, max_pages, pt_row, ctx, out, scratch, n_splits, T, n_heads, n_kv, d,
                       page_size, share, st);
}

// Decode step: RoPE + KV write of the step's new token (position ctx[t] - 1 == pos[t]) fused in.
cudaError_t launch_attn_decode_fused(const TmaMap &kv_map, long long row0, uint16_t *kv_layer_base, const float *qkv,
                                     int n_partial, long long partial_stride, const int *pos, const float *rope_cos,
                                     const float *rope_sin, const int *page_table, int max_pages, const int *pt_row,
                                     const int *ctx, uint16_t *out, float *scratch, int n_splits, int T, int n_heads,
                                     int n_kv, int d, int page_size, bool share, cudaStream_t st) {
  AttnRope r{qkv, n_partial, partial_stride, pos, rope_cos, rope_sin, kv_layer_base};
  return attn_dispatch(kv_map, row0, r, nullptr, page_table, max_pages, pt_row, ctx, out, scratch, n_splits, T, n_heads, n_kv, d,
                       page_size, share, st);
}

template <int D, int G>
static cudaError_t prefill_launch(const TmaMap &kv_map, long long row0, const uint16_t *q, const int *page_table,
                                  int max_pages, const int *qb_tok0, const int *qb_len, const int *qb_pos0,
                                  const int *qb_ptrow, uint16_t *out, int n_blocks, int n_heads, int n_kv,
                                  int page_shift, cudaStream_t st) {
  static DeviceOnce once;
  DIS_CUDA_TRY(once.run([&] { return cudaFuncSetAttribute(attn_prefill_kernel<D, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnCfg<D>::kSmemBytes); }));
  return launch_k(attn_prefill_kernel<D, G>, dim3(n_blocks, n_kv), dim3(G * 32), AttnCfg<D>::kSmemBytes, st,
                  *reinterpret_cast<const CUtensorMap *>(&kv_map), row0, q, page_table, max_pages, qb_tok0, qb_len, qb_pos0,
                  qb_ptrow, out, n_heads, n_kv, page_shift);
}

// Query blocks: block b covers tokens [qb_tok0[b], +qb_len[b]) of the flattened batch (qb_len <= 16), which are
// consecutive positions qb_pos0[b].. of the sequence whose page-table row is qb_ptrow[b].
cudaError_t launch_attn_prefill(const TmaMap &kv_map, long long row0, const uint16_t *q, const int *page_table,
                                int max_pages, const int *qb_tok0, const int *qb_len, const int *qb_pos0,
                                const int *qb_ptrow, uint16_t *out, int n_blocks, int n_heads, int n_kv, int d,
                                int page_size, cudaStream_t st) {
  if (n_blocks <= 0) return cudaSuccess;
  if (n_kv <= 0 || n_heads % n_kv != 0 || n_kv > 65535) { set_last_error("attn_prefill: bad head counts"); return cudaErrorInvalidValue; }
  if (page_size < 8 || (page_size & (page_size - 1))) { set_last_error("attn_prefill: page_size must be a power of two >= 8"); return cudaErrorInvalidValue; }
  int page_shift = 0;
  while ((1 << page_shift) < page_size) page_shift++;
  const int G = n_heads / n_kv;
#define DIS_PF_CASE(DD, GG)                                                                                        \
  if (d == DD && G == GG)                                                                                          \
    return prefill_launch<DD, GG>(kv_map, row0, q, page_table, max_pages, qb_tok0, qb_len, qb_pos0, qb_ptrow, out, \
                                  n_blocks, n_heads, n_kv, page_shift, st);
  DIS_PF_CASE(128, 8) DIS_PF_CASE(128, 4) DIS_PF_CASE(128, 2) DIS_PF_CASE(128, 1)
  DIS_PF_CASE(64, 8) DIS_PF_CASE(64, 4) DIS_PF_CASE(64, 2) DIS_PF_CASE(64, 1)
#undef DIS_PF_CASE
  set_last_error("attn_prefill: head_dim must be 64 or 128 and the GQA group 1, 2, 4 or 8");
  return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------------------------------
// dis_k_attn_paged_static: the split-KV attention above for hosts that must not allocate.
//
// Who needs it: a serving process that has already handed every free byte of HBM to its KV-page pool (this
// engine does exactly that with kv_mem_fraction) has nothing left for cudaMalloc to give, and a request
// loop that must stay free of cudaMalloc/cudaFree -- both synchronise the whole device and stall every
// other stream -- cannot afford the call even when memory is available.  Such a host still wants the
// split-KV path (it is what keeps all SMs busy at small batch), which needs room for the per-split
// (m, l, o) partials.  Here that room is a fixed array inside the library image instead of a buffer the
// caller provides.
namespace {
constexpr size_t kStaticScratchFloats = DIS_ATTN_STATIC_SCRATCH_FLOATS;
// Lives in every CUDA context that loads this library, from module load until the process exits.
static __device__ __align__(256) float g_attn_static_scratch[kStaticScratchFloats];

// In host code the array's name is only a handle for the runtime, not a device address: the address each
// device gave its own copy has to be asked for, once per device, while that device is current.
cudaError_t static_scratch_of_current_device(float **out) {
  static std::mutex mu;
  static float *ptrs[64] = {};
  int dev = -1;
  DIS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_last_error("attn_paged_static: device ordinal out of range"); return cudaErrorInvalidDevice; }
  std::lock_guard<std::mutex> lk(mu);
  if (!ptrs[dev]) {
    float *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_attn_static_scratch);
    if (e != cudaSuccess || !p) {
      set_last_error(std::string("attn_paged_static: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
      return e != cudaSuccess ? e : cudaErrorUnknown;
    }
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return cudaSuccess;
}
}  // namespace

}  // namespace dis

extern "C" DIS_API int dis_k_attn_paged_static(const uint16_t *q, const uint16_t *kv_pool, int64_t n_pages,
                                               const int32_t *page_table, int32_t max_pages, const int32_t *pt_row,
                                               const int32_t *ctx, uint16_t *out, int32_t n_splits, int32_t T,
                                               int32_t n_heads, int32_t n_kv, int32_t d, int32_t page_size, void *stream) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    dis::set_last_error("no CUDA device: there is no CPU fallback");
    return DIS_ERR_INFERENCE_FAILED;
  }
  if (T <= 0 || n_splits < 1) { dis::set_last_error("attn_paged_static: T and n_splits must be positive"); return DIS_ERR_INVALID_ARGUMENT; }
  const size_t need = dis::attn_scratch_elems(T, n_heads, d, n_splits);
  if (need > dis::kStaticScratchFloats) {
    dis::set_last_error("attn_paged_static: T*n_heads*n_splits*(2+d) = " + std::to_string(need) +
                        " floats of split-KV partials do not fit the built-in scratch of " +
                        std::to_string(dis::kStaticScratchFloats) + " floats (DIS_ATTN_STATIC_SCRATCH_FLOATS); use fewer "
                        "splits or tokens per call, or dis_k_attn_paged with your own buffer");
    return DIS_ERR_INVALID_ARGUMENT;
  }
  float *scratch = nullptr;
  if (dis::static_scratch_of_current_device(&scratch) != cudaSuccess) return DIS_ERR_INFERENCE_FAILED;
  dis::TmaMap map;  // encoded on the host stack; no device allocation
  if (dis::make_kv_map(&map, kv_pool, (long long)n_pages * 2 * n_kv * page_size, d, page_size) != cudaSuccess)
    return DIS_ERR_INFERENCE_FAILED;
  // Nothing in the scratch has to start at zero: every (m, l, o) slot the combine pass reads is written by a
  // split CTA of this same call first, so whatever the previous call left behind is never observed.
  const cudaError_t e = dis::launch_attn_paged(map, 0, q, page_table, max_pages, pt_row, ctx, out, n_splits > 1 ? scratch : nullptr,
                                               n_splits, T, n_heads, n_kv, d, page_size, static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? DIS_OK : DIS_ERR_INFERENCE_FAILED;
}
