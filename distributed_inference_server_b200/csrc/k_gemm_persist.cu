// k_gemm_persist.cu -- the projection GEMM for PROMPT-sized token counts, sm_100a: pairs of CTAs, one
// 256 x 256 tile per pair (tcgen05.mma cta_group::2).
//
// What bounds it: with one CTA per tile of 128 x 256 every k-block brings 48 KB into an SM for 512 clocks of tensor work, 96 bytes a
// clock where the L2 -> SM path carries about 64, and four epilogue warps drain a tile in 30000 clocks where a K of 1024 gives the
// tensor pipe 8000.  Here
//   * the two CTAs of a cluster share one tile of 256 tokens x 256 features: each brings its own 128 token rows (A) and half of the
//     feature rows (B), 32 KB per k-block, and the pair's MMA reads B from both;
//   * tokens are the MMA's rows (TMEM lanes) and features its columns, so an epilogue thread owns one token and consecutive features:
//     gate and up of a feature sit in the same lane (columns c and 128 + c) and nothing is exchanged, and a thread writes 32-byte
//     pieces of its row;
//   * eight epilogue warps, the accumulator double-buffered in TMEM (2 x 256 columns): tile i is drained while tile i + 1 runs;
//   * persistent: pair p walks tiles p, p + pairs, ...; the TMA ring (6 x 32 KB) never drains between tiles.
// Measured against the kernels it replaces (one CTA per 128 x 256 tile, persistent or not), us: gate-up 14336 x 4096, 8192 tokens
// 1517 -> 1257 (1.53 PFLOP/s), 5632 x 2048, 6554 tokens 370 -> 235, 4096 x 1024, 6554 tokens 264 -> 98; plain 4096 x 14336, 6554 tokens
// 578 -> 536, 6144 x 4096, 3000 tokens 116 -> 104, 6176 x 1024, 6554 tokens 152 -> 79.
//
//   warp 0      TMA producer of this CTA's operands; both CTAs' bytes complete on the first CTA's full barrier
//   warp 1      (first CTA) one elected lane issues the pair's MMAs; its commits reach both CTAs' barriers
//   warps 2-9   epilogue: warp % 4 picks 32 tokens, (warp - 2) / 4 the half of the columns
#include <cuda.h>

#include "kernels.h"
#include "ptx.cuh"

namespace dis {

namespace {

constexpr int kPairStages = 6;
constexpr int kPairOperand = 128 * kBK * 2;           // one CTA's A or B rows of a k-block, 16 KB
constexpr int kPairStage = 2 * kPairOperand;
constexpr int kPairSmem = kPairStages * kPairStage + 1024 + 256;
constexpr int kPairThreads = 320;
constexpr int kPairCols = 256;                        // accumulator columns of one tile

enum { kOutF32 = 0, kOutBf16 = 1, kOutRelu2 = 2, kOutGlu = 3 };

__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void *map, int c0, int c1, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void umma_ss_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
      : "memory");
}
// arrives at the same barrier of both CTAs once all MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t cluster_bar(uint32_t bar, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(bar), "r"(rank));
  return a;
}
// wait for a barrier that the other CTA of the pair arrives at: acquire at cluster scope
__device__ __forceinline__ void mbar_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok, polls = 0;
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (!ok && ++polls > (1u << 26)) __trap();  // as mbar_wait
  } while (!ok);
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 32 bytes to a 32-byte aligned address: a whole sector per lane
__device__ __forceinline__ void st_32(void *p, const uint32_t *v) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// BN: accumulator columns of a tile (256, 224 or 192; see pair_columns)
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld_32x32(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

template <int kOut, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, float *__restrict__ out_f32,
                 uint16_t *__restrict__ out_bf16, int T, int N, int K, int w_row0, int w_row_step, int tiles_n, int tiles_t, int t_fast,
                 int kb_per_split, int n_tiles, int act_kind, int ld_out, int wide) {
  constexpr int kTileN = kOut == kOutGlu ? BN / 2 : BN;  // output features of a tile
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + kPairStages * kPairStage;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };                              // (first CTA's are used)
  auto empty_bar = [&](int s) { return bar_base + 8u * (kPairStages + s); };
  auto acc_full = [&](uint32_t b) { return bar_base + 8u * (2 * kPairStages + b); };
  auto acc_empty = [&](uint32_t b) { return bar_base + 8u * (2 * kPairStages + 2 + b); };  // (first CTA's are used)
  const uint32_t tmem_slot = bar_base + 8u * (2 * kPairStages + 4);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
  const int num_kb = (K + kBK - 1) / kBK, tiles = tiles_n * tiles_t;
  // tile -> (split, feature tile, token tile).  The tiles in flight together should cover ALL tiles of the smaller operand (it stays in
  // L2 and is re-read every round) and only a few of the larger one (streamed from HBM once): token tile fastest when the weight
  // matrix is the larger operand.
  auto tile_n0 = [&](int tile) { const int i = tile % tiles; return (t_fast ? i / tiles_t : i % tiles_n) * kTileN; };
  auto tile_t0 = [&](int tile) { const int i = tile % tiles; return (t_fast ? i % tiles_t : i / tiles_n) * 256 + (int)rank * 128; };
  const uint64_t w_hint = t_fast ? kEvictFirst : kEvictLast, x_hint = t_fast ? kEvictLast : kEvictFirst;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&w_map);
    tma_prefetch_desc(&x_map);
    for (int s = 0; s < kPairStages; s++) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (uint32_t b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 16); }  // 8 epilogue warps of each CTA
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_slot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the other CTA's barriers and tensor memory are ready as well
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  pdl_launch_dependents();

  if (warp == 0) {
    // ===== TMA producer: one flat stream of (tile, k-block) stages =====
    if (lane == 0) {
      pdl_wait();  // activations come from the previous kernel
      int s = 0;
      uint32_t phase = 0;
      for (int tile = pair; tile < n_tiles; tile += pairs) {
        const int n0 = tile_n0(tile), t0 = tile_t0(tile), kb0 = tile / tiles * kb_per_split, kb1 = min(num_kb, kb0 + kb_per_split);
        const int wr = w_row0 + n0 + (int)rank * w_row_step;  // this CTA's half of the feature rows (gate-up: gate rows | up rows)
        for (int kb = kb0; kb < kb1; kb++) {
          mbar_wait(empty_bar(s), phase ^ 1u);  // passes on the first lap
          if (rank == 0) mbar_expect_tx(full_bar(s), 2 * kPairStage);
          const uint32_t bar = cluster_bar(full_bar(s), 0), a = smem_base + s * kPairStage;
          tma_load_2d_pair(a, &x_map, kb * kBK, t0, bar, x_hint);
          tma_load_2d_pair(a + kPairOperand, &w_map, kb * kBK, wr, bar, w_hint);
          if (++s == kPairStages) { s = 0; phase ^= 1u; }
        }
      }
      // The first CTA's commits still arrive at this CTA's barriers: wait for the last of every stage before the CTA may end.
      for (int i = 0; i < kPairStages; i++) {  // (a stage never filled passes at once)
        mbar_wait(empty_bar(s), phase ^ 1u);
        if (++s == kPairStages) { s = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer (first CTA; the warp converged, one elected lane issues): accumulator buffers alternate per tile =====
    if (rank == 0) {
      constexpr uint32_t idesc = (umma_idesc<BN>() & ~(31u << 24)) | (16u << 24);  // M 256: 128 rows of each CTA
      const uint32_t lo0 = umma_lo(smem_base);
      uint32_t lo = lo0, phase = 0, buf = 0, aphase = 0;
      int s = 0;
      for (int tile = pair; tile < n_tiles; tile += pairs) {
        const int kb0 = tile / tiles * kb_per_split, kb1 = min(num_kb, kb0 + kb_per_split);
        mbar_wait_cluster(acc_empty(buf), aphase ^ 1u);  // both epilogues have drained this buffer (passes on first use)
        tc_fence_after();
        const uint32_t acc = tmem_base + buf * kPairCols;
        for (int kb = kb0; kb < kb1; kb++) {
          mbar_wait_cluster(full_bar(s), phase);
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (uint32_t k = 0; k < kBK / 16; k++)
              umma_ss_pair(acc, lo + 2 * k, lo + (kPairOperand >> 4) + 2 * k, idesc, k > 0 ? 1u : (uint32_t)(kb > kb0));
            umma_commit_pair(empty_bar(s));                   // slot reusable in both CTAs once these MMAs have read it
            if (kb == kb1 - 1) umma_commit_pair(acc_full(buf));  // this tile's accumulator is complete
          }
          __syncwarp();
          lo += kPairStage >> 4;
          if (++s == kPairStages) { s = 0; phase ^= 1u; lo = lo0; }
        }
        aphase ^= buf;
        buf ^= 1u;
      }
    }
  } else {
    // ===== epilogue: TMEM -> registers -> global, one tile behind the MMAs =====
    const int quarter = warp & 3, half = (warp - 2) >> 2;  // a warp may only touch TMEM lanes [32 * (warp % 4), +32)
    uint32_t buf = 0, aphase = 0;
    const uint32_t empty0 = cluster_bar(acc_empty(0), 0), empty1 = cluster_bar(acc_empty(1), 0);
    bool waited = false;
    for (int tile = pair; tile < n_tiles; tile += pairs) {
      const int n0 = tile_n0(tile), t = tile_t0(tile) + quarter * 32 + lane;
      mbar_wait_cluster(acc_full(buf), aphase);
      tc_fence_after();
      if (!waited) { pdl_wait(); waited = true; }  // global writes only after every prerequisite grid has completed
      const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * kPairCols;
      // 32 columns at a time, or 16 where the tile's width asks for it; the first half of the warps takes the larger half of the chunks
      constexpr int CH = kTileN % 64 == 0 ? 32 : 16, kChunks = kTileN / CH, kFirst = (kChunks + 1) / 2;
      const int c1 = half ? kChunks : kFirst;
#pragma unroll 1
      for (int c = half ? kFirst : 0; c < c1; c++) {
        uint32_t v[CH];
        const int col = CH * c, n = n0 + col;
        tmem_ld_cols(acc + col, v);
        if (kOut == kOutGlu) {
          uint32_t u[CH];
          tmem_ld_cols(acc + kTileN + col, u);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < CH; i++) v[i] = __float_as_uint(gate_act_fast(act_kind, __uint_as_float(v[i])) * __uint_as_float(u[i]));
        } else {
          tmem_ld_wait();
        }
        if (c == c1 - 1) {  // everything of this buffer is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(buf ? empty1 : empty0);
        }
        if (kOut == kOutRelu2) {
#pragma unroll
          for (int i = 0; i < CH; i++) { const float r = fmaxf(__uint_as_float(v[i]), 0.f); v[i] = __float_as_uint(r * r); }
        }
        if (t >= T) continue;
        if (kOut == kOutF32) {
          float *o = out_f32 + ((size_t)(tile / tiles) * T + t) * N + n;
          if (wide && n + CH <= N) {
#pragma unroll
            for (int i = 0; i < CH; i += 8) st_32(o + i, v + i);
          } else {
#pragma unroll
            for (int i = 0; i < CH; i++)
              if (n + i < N) o[i] = __uint_as_float(v[i]);
          }
        } else {
          uint16_t *o = out_bf16 + (size_t)t * ld_out + n;
          if (wide && n + CH <= N) {
            uint32_t p[CH / 2];
#pragma unroll
            for (int i = 0; i < CH / 2; i++) p[i] = float2_to_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
#pragma unroll
            for (int i = 0; i < CH; i += 16) st_32(o + i, p + i / 2);
          } else {
#pragma unroll
            for (int i = 0; i < CH; i++)
              if (n + i < N) o[i] = float_to_bf16_bits(__uint_as_float(v[i]));
          }
        }
      }
      aphase ^= buf;
      buf ^= 1u;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the other's MMAs, commits or arrivals may still reach it
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
}

// Rounds of tiles of bn columns that the 74 pairs need.
long long pair_rounds(int T, int N, int split, bool dual, int bn) {
  const int feats = dual ? bn / 2 : bn;
  const long long tiles = (long long)((N + feats - 1) / feats) * ((T + 255) / 256) * split;
  return (tiles + kNumSMs / 2 - 1) / (kNumSMs / 2);
}
// Columns of a tile: the width whose rounds take the least time, a tile's being its columns plus what it costs at any width.  A last
// round that is nearly empty costs a whole one: gate-up of 1000 tokens, 14336 features: 448 tiles of 256 columns are 6.05 rounds
// (193.8 us), 512 of 224 are 6.92 (161.1 us); 8192 x 8192 features, 2000 tokens: 222.7 us against 178.6.
int pair_columns(int T, int N, int split, bool dual) {
  int best = 256;
  for (int bn : {224, 192})
    if (pair_rounds(T, N, split, dual, bn) * (bn + 32) < pair_rounds(T, N, split, dual, best) * (best + 32)) best = bn;
  return best;
}

template <int kOut, int BN>
cudaError_t pair_launch_bn(const TmaMap &w_map, const TmaMap &x_map, float *out, uint16_t *act, int T, int N, int K, int w_row0, int w_row_step,
                        int split, int act_kind, int ld_out, cudaStream_t st) {
  static DeviceOnce once;
  DIS_CUDA_TRY(once.run([&] { return cudaFuncSetAttribute(gemm_pair_kernel<kOut, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem); }));
  const int num_kb = (K + kBK - 1) / kBK, per = (num_kb + split - 1) / split;
  if ((num_kb + per - 1) / per != split) { set_last_error("gemm: split_k leaves an empty K slice; use gemm_pick_split_k"); return cudaErrorInvalidValue; }
  const int feats = kOut == kOutGlu ? BN / 2 : BN;
  const int tiles_n = (N + feats - 1) / feats, tiles_t = (T + 255) / 256;
  const long long n_tiles = (long long)tiles_n * tiles_t * split;
  if (n_tiles > (1 << 30)) { set_last_error("gemm: too many tiles"); return cudaErrorInvalidValue; }
  const int pairs = n_tiles < kNumSMs / 2 ? (int)n_tiles : kNumSMs / 2;
  const int t_fast = (long long)(kOut == kOutGlu ? 2 : 1) * N > (long long)T ? 1 : 0;  // weight rows vs token rows (same K)
  const uintptr_t at = kOut == kOutF32 ? (uintptr_t)out : (uintptr_t)act;
  const int wide = (at & 31u) == 0 && (kOut == kOutF32 ? N % 8 == 0 : ld_out % 16 == 0);  // every row piece starts on 32 bytes
  return launch_k(gemm_pair_kernel<kOut, BN>, dim3(2 * pairs), dim3(kPairThreads), (size_t)kPairSmem, st, *reinterpret_cast<const CUtensorMap *>(&w_map),
                  *reinterpret_cast<const CUtensorMap *>(&x_map), out, act, T, N, K, w_row0, w_row_step > 0 ? w_row_step : BN / 2, tiles_n, tiles_t, t_fast, per,
                  (int)n_tiles,
                  act_kind, ld_out, wide);
}
// w_row_step: from the first CTA's feature rows to the second's; 0: they follow each other
template <int kOut>
cudaError_t pair_launch(const TmaMap &w_map, const TmaMap &x_map, float *out, uint16_t *act, int T, int N, int K, int w_row0, int w_row_step,
                        int split, int act_kind, int ld_out, cudaStream_t st) {
  const int bn = pair_columns(T, N, split, kOut == kOutGlu);
  auto f = bn == 256 ? pair_launch_bn<kOut, 256> : bn == 224 ? pair_launch_bn<kOut, 224> : pair_launch_bn<kOut, 192>;
  return f(w_map, x_map, out, act, T, N, K, w_row0, w_row_step, split, act_kind, ld_out, st);
}

}  // namespace

// Which passes run in pairs.  Gate-up products (dual) from 129 tokens: the kernel for fewer (k_gemm_tcgen05.cu) walks its one tile per
// CTA at half the rate (14336 x 4096, 200 tokens: 78.2 us against 50.8; 4096 x 1024, 1000 tokens: 124 against 27).  Plain products from
// 1024 tokens always (4096 x 4096, 1300 tokens: 64.8 us there, 39.8 here; 512 x 512, 1024 tokens: 12.6 and 8.2).  Below that by what the
// two take behind their launch, in hundredths of a microsecond, fitted to 21 shapes from 512 x 512 to 8192 x 28672 at ten token counts
// each, weights from HBM: there 100 + 20 per k-block for every 148 CTAs of 128 x 128, here 320 + 33 per k-block for every round of 256
// columns, less 40.  The faster is taken within 2 % at 207 of the 210 points and within 8 % at the rest; counting rounds alone took the slower at
// 39 (us there / here: 2048 x 2048 in 8 slices, 200 tokens 9.9 / 11.0; 1024 x 5120 in 16, 200 tokens 10.4 / 11.4; while 3072 x 1024 in
// 4, 200 tokens 9.6 / 8.9; 4096 x 4096 in 2, 400 tokens 21.8 / 20.7; 4096 x 14336 in 4, 200 tokens 36.6 / 31.5).
bool gemm_use_persist(int T, int N, int K, int split, bool dual) {
  if (T <= 128) return false;
  if (dual || T >= 1024) return true;
  if (split < 1) return false;
  const long long kb = ((K + kBK - 1) / kBK + split - 1) / split;
  const long long ctas = (long long)((N + kBM - 1) / kBM) * ((T + 127) / 128) * split;
  const int bn = pair_columns(T, N, split, false);
  return (pair_rounds(T, N, split, false, bn) * bn * (320 + 33 * kb)) / 256 - 40 < (ctas + kNumSMs - 1) / kNumSMs * (100 + 20 * kb);
}

// w_map, x_map: 128-row boxes.  out[s][t][n] fp32, s the K slice.
cudaError_t launch_gemm_persist_partial(const TmaMap &w_map, const TmaMap &x_map, float *out, int T, int N, int K, int w_row0, int split,
                                        cudaStream_t st) {
  if (T <= 0) return cudaSuccess;
  if (split < 1) { set_last_error("gemm: split_k must be >= 1"); return cudaErrorInvalidValue; }
  return pair_launch<kOutF32>(w_map, x_map, out, nullptr, T, N, K, w_row0, 0, split, 0, N, st);
}

// The same product with the epilogue of an ungated unit: act[t][n] = bf16(relu(sum)^2).
cudaError_t launch_gemm_persist_relu2(const TmaMap &w_map, const TmaMap &x_map, uint16_t *act, int T, int N, int K, int w_row0, cudaStream_t st) {
  if (T <= 0) return cudaSuccess;
  if (!act) return cudaErrorInvalidValue;
  return pair_launch<kOutRelu2>(w_map, x_map, nullptr, act, T, N, K, w_row0, 0, 1, 0, N, st);
}

// The same product, its sums rounded to bf16 by the epilogue.
cudaError_t launch_gemm_persist_bf16(const TmaMap &w_map, const TmaMap &x_map, uint16_t *out, int T, int N, int K, int w_row0, cudaStream_t st) {
  if (T <= 0) return cudaSuccess;
  if (!out) return cudaErrorInvalidValue;
  return pair_launch<kOutBf16>(w_map, x_map, nullptr, out, T, N, K, w_row0, 0, 1, 0, N, st);
}

// w_map: 128-row boxes over the fused [2I][K] weight (gate rows, then up rows).  act[t][n] = bf16(act(gate) * up), act_kind 0 = silu,
// 1 = gelu_tanh.
cudaError_t launch_gemm_persist_glu(const TmaMap &w_map, const TmaMap &x_map, uint16_t *act, int T, int I, int K, int w_row0, int act_kind,
                                    cudaStream_t st, int ld_act) {
  if (T <= 0) return cudaSuccess;
  return pair_launch<kOutGlu>(w_map, x_map, nullptr, act, T, I, K, w_row0, I, 1, act_kind, ld_act > 0 ? ld_act : I, st);
}
cudaError_t launch_gemm_persist_silu(const TmaMap &w_map, const TmaMap &x_map, uint16_t *act, int T, int I, int K, int w_row0, cudaStream_t st) {
  return launch_gemm_persist_glu(w_map, x_map, act, T, I, K, w_row0, 0, st);
}

}  // namespace dis
