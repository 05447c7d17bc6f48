// k_sample.cu -- the sampler (argmax / temperature + nucleus) with a row spread over a cluster of eight CTAs.
// No reference counterpart; the sampling controls are InferenceParams (design.md:666-671), the definition of the draw is the
// oracle's: nucleus = {p >= tau}, tau the largest threshold whose kept mass reaches top_p, one uniform per (seed, step), first kept
// token in index order whose running mass exceeds u * kept.
//
// What bounds it: latency.  A row of 128256 logits is 513 KB; one CTA per row (sample_kernel in k_elementwise.cu, which stays
// for rows longer than kSampleClusterMaxV) walks it 30 to 40 times through one SM's L2 port, on as many SMs as there are rows: 701 us
// for 32 rows of 128256, three quarters of them sampled, against 42 us here.  Here the eight CTAs of a cluster read the row ONCE and keep it in
// registers (at most 16 float4 per thread); everything after that is arithmetic on registers.  The threshold search narrows 32-fold per
// round instead of halving: a thread adds each of its probabilities inside the current range to its own column of a [32][512] table
// (no atomics: the sums keep one order and a repeated call gives the same bits), the table's rows are summed per CTA, and the CTAs
// swap 32 partial masses through distributed shared memory -- six rounds cover the 2^30 bit patterns of floats up to 1.
#include "kernels.h"
#include "ptx.cuh"

namespace dis {

namespace {

constexpr int kCl = 8;          // CTAs per row: the portable cluster size
constexpr int kThr = 512;
constexpr int kWarps = kThr / 32;
constexpr int kBins = 32;       // thresholds per search round
constexpr int kBinsBytes = kBins * kThr * 4;

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_cluster(const float *p, uint32_t rank, float v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

struct Sh {
  float mine[kBins];                 // what this CTA gives away in an exchange
  float all[2][kCl][kBins];          // what every CTA gave; two halves in turn, so one exchange never overwrites what the last is read from
  float wv[kWarps];
  int wi[kWarps];
  int tok;
};

// mine[0..n) of every CTA of the cluster -> all[par][rank][0..n) in every CTA.
__device__ __forceinline__ void swap(Sh &s, int me, int n, int par) {
  __syncthreads();
  for (int i = threadIdx.x; i < n * kCl; i += kThr) st_cluster(&s.all[par][me][i % n], (uint32_t)(i / n), s.mine[i % n]);
  cluster_sync_all();
}

// Sum over the block, in a fixed order; every thread gets it.
__device__ __forceinline__ float sum_block(Sh &s, float v) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s.wv[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; w++) r += s.wv[w];
  return r;
}

// KV: float4 groups per thread.  Element (k, j) of a thread is index base + k * 128 + lane * 4 + j of the row: a warp owns a contiguous
// piece, warps and CTAs follow each other, so running masses go through (CTA, warp, k, lane, j) in index order.
template <int KV>
__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kThr, KV <= 8 ? 2 : 1)
sample_cluster_kernel(const float *__restrict__ logits, long long ld, int V, const float *__restrict__ temperature,
                      const float *__restrict__ top_p, const unsigned long long *__restrict__ seeds,
                      const unsigned long long *__restrict__ steps, uint32_t *__restrict__ out, int vocab_offset,
                      float *__restrict__ out_val, float *__restrict__ out_sumexp, float *__restrict__ out_logprob) {
  extern __shared__ float bins[];  // [kBins][kThr]: a column per thread
  __shared__ Sh s;
  const int t = blockIdx.x / kCl, me = (int)cluster_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int base = (me * kWarps + warp) * (KV * 128) + lane * 4;
  pdl_wait();
  pdl_launch_dependents();
  const float *row = logits + (size_t)t * ld;
  const float temp = temperature ? temperature[t] : 0.f;
  float v[KV][4];
  // 16-byte loads where every row starts on 16 bytes; elements behind the row's end read as -inf and never win, weigh or count
  const bool wide = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15u) == 0;
#pragma unroll
  for (int k = 0; k < KV; k++) {
    const int i = base + k * 128;
    if (wide && i + 3 < V) {
      const float4 f = *reinterpret_cast<const float4 *>(row + i);
      v[k][0] = f.x; v[k][1] = f.y; v[k][2] = f.z; v[k][3] = f.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) v[k][j] = i + j < V ? row[i + j] : -INFINITY;
    }
  }
  // ---- argmax, lowest index first
  float bv = -INFINITY;
  int bi = 0x7fffffff;
#pragma unroll
  for (int k = 0; k < KV; k++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (v[k][j] > bv) { bv = v[k][j]; bi = base + k * 128 + j; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  if (lane == 0) { s.wv[warp] = bv; s.wi[warp] = bi; }
  if (threadIdx.x == 0) s.tok = -1;
  cluster_sync_all();  // every CTA of the cluster is running: its shared memory may be written from now on
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kWarps; w++)
      if (s.wv[w] > bv || (s.wv[w] == bv && s.wi[w] < bi)) { bv = s.wv[w]; bi = s.wi[w]; }
    s.mine[0] = bv;
    s.mine[1] = __int_as_float(bi);
  }
  int par = 0;
  swap(s, me, 2, par);
  bv = s.all[par][0][0];
  bi = __float_as_int(s.all[par][0][1]);
#pragma unroll
  for (int r = 1; r < kCl; r++) {
    const float ov = s.all[par][r][0];
    const int oi = __float_as_int(s.all[par][r][1]);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  par ^= 1;
  // ---- sum of exp(z - max); a greedy row is done with it
  const bool greedy = temp <= 0.f;
  const float inv_t = greedy ? 1.f : 1.0f / temp;
  const float m = bv * inv_t;  // rounding keeps the order, so this is the largest z
  float se = 0.f;
  if (!greedy || out_sumexp || out_logprob) {
    float part = 0.f;
#pragma unroll
    for (int k = 0; k < KV; k++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        v[k][j] = expf(v[k][j] * inv_t - m);
        // an element behind the end of a row without a finite value is exp(-inf + inf): it must not make the sum NaN by itself
        if (base + k * 128 + j >= V) v[k][j] = 0.f;
        part += v[k][j];
      }
    part = sum_block(s, part);
    if (threadIdx.x == 0) s.mine[0] = part;
    swap(s, me, 1, par);
#pragma unroll
    for (int r = 0; r < kCl; r++) se += s.all[par][r][0];
    par ^= 1;
  }
  if (greedy) {
    if (me == 0 && threadIdx.x == 0) {
      out[t] = (uint32_t)(bi + vocab_offset);
      if (out_val) out_val[t] = bv;
      if (out_sumexp) out_sumexp[t] = se;
      if (out_logprob) out_logprob[t] = -logf(se);
    }
    return;
  }
  const float inv_z = 1.0f / se;
#pragma unroll
  for (int k = 0; k < KV; k++)
#pragma unroll
    for (int j = 0; j < 4; j++) v[k][j] *= inv_z;
  // ---- nucleus threshold: the largest bit pattern whose mass (the sum of all p at or above it) still reaches top_p
  const float tp = top_p ? top_p[t] : 1.0f;
  uint32_t tau = 0u;
  if (tp < 1.0f) {
    float above = 0.f;  // mass of everything at or above the current range's end
    for (int sh = 25; sh >= 0; sh -= 5) {
#pragma unroll
      for (int b = 0; b < kBins; b++) bins[b * kThr + threadIdx.x] = 0.f;
#pragma unroll
      for (int k = 0; k < KV; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t bits = __float_as_uint(v[k][j]);
          // the first round's last bin also takes NaN, whatever its sign (then the search ends at 0, as with any comparison that fails)
          const uint32_t b = sh == 25 ? min(bits >> 25, (uint32_t)(kBins - 1)) : (bits - tau) >> sh;
          if (bits >= tau && b < (uint32_t)kBins && v[k][j] != 0.f) bins[b * kThr + threadIdx.x] += v[k][j];
        }
      __syncthreads();
      // warp w sums rows 2 w and 2 w + 1 of the table
#pragma unroll
      for (int h = 0; h < kBins / kWarps; h++) {
        const int b = warp * (kBins / kWarps) + h;
        float x = 0.f;
#pragma unroll
        for (int i = 0; i < kThr / 32; i++) x += bins[b * kThr + i * 32 + lane];
        x = warp_sum(x);
        if (lane == 0) s.mine[b] = x;
      }
      swap(s, me, kBins, par);
      // every thread: lane j holds bin j's mass over the cluster, then the mass at or above threshold j
      float x = 0.f;
#pragma unroll
      for (int r = 0; r < kCl; r++) x += s.all[par][r][lane];
      par ^= 1;
      float suf = x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += n;
      }
      const uint32_t ok = __ballot_sync(0xffffffffu, above + suf >= tp) | 1u;  // threshold 0 holds by what the last round chose
      const int j = 31 - __clz(ok);
      const float next = __shfl_sync(0xffffffffu, suf, (j + 1) & 31);
      if (j < 31) above += next;
      tau += (uint32_t)j << sh;
    }
  }
  tau = max(tau, 1u);  // a weight of zero (a masked logit, an underflow) is never kept: no draw may return it
  // ---- draw: first kept token in index order whose running mass exceeds u * kept
  float local = 0.f;
#pragma unroll
  for (int k = 0; k < KV; k++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (__float_as_uint(v[k][j]) >= tau) local += v[k][j];
  local = warp_sum(local);
  __syncthreads();
  if (lane == 0) s.wv[warp] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    float x = 0.f;
    for (int w = 0; w < kWarps; w++) x += s.wv[w];
    s.mine[0] = x;
  }
  swap(s, me, 1, par);
  float kept = 0.f;
#pragma unroll
  for (int r = 0; r < kCl; r++) kept += s.all[par][r][0];
  const float target = hash_u01(mix64(seeds ? seeds[t] : 0ull, 0xC0FFEEull, steps ? steps[t] : 0ull)) * kept;
  int owner = -1;
  float start = 0.f, run = 0.f;
#pragma unroll
  for (int r = 0; r < kCl; r++) {
    const float x = s.all[par][r][0];
    if (owner < 0 && x > 0.f && target < run + x) { owner = r; start = run; }
    run += x;
  }
  if (owner < 0 ? me != 0 : me != owner) return;  // no exchange follows
  if (owner >= 0) {
    int w_own = -1, w_last = 0;
    float w_start = start, w_last_start = start, x = start;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      const float y = s.wv[w];
      if (y > 0.f) { w_last = w; w_last_start = x; }
      if (w_own < 0 && y > 0.f && target < x + y) { w_own = w; w_start = x; }
      x += y;
    }
    if (w_own < 0) { w_own = w_last; w_start = w_last_start; }  // rounding: the CTA's last kept piece
    if (warp == w_own) {
      float at = w_start;
      int tok = -1, last = -1;
#pragma unroll
      for (int k = 0; k < KV; k++) {
        float kp[4], mine = 0.f;
        bool in[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          in[j] = __float_as_uint(v[k][j]) >= tau && base + k * 128 + j < V;
          kp[j] = in[j] ? v[k][j] : 0.f;
          mine += kp[j];
        }
        float incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float n = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += n;
        }
        // a lane starts at the very number the lane before it ends with: were the two rounded apart, a token at the edge could gain
        // mass that is not its own
        const float before = __shfl_up_sync(0xffffffffu, incl, 1);
        float x2 = lane == 0 ? at : at + before;
        int first = 0x7fffffff, end = -1;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          x2 = j < 3 ? x2 + kp[j] : at + incl;
          if (in[j]) { end = base + k * 128 + j; if (x2 > target && first == 0x7fffffff) first = end; }
        }
        first = __reduce_min_sync(0xffffffffu, first);
        end = __reduce_max_sync(0xffffffffu, end);
        if (tok < 0 && first != 0x7fffffff) tok = first;
        if (end >= 0) last = end;
        at += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) s.tok = tok >= 0 ? tok : last;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int tok = s.tok >= 0 ? s.tok : bi;  // no interval (a row of NaN): the mode
    out[t] = (uint32_t)(tok + vocab_offset);
    const float at = tok < V ? row[tok] : NAN;  // (no index at all: every logit is -inf or NaN)
    if (out_val) out_val[t] = at;
    // log-probability of the drawn token under softmax(logits / temperature), before the nucleus cut
    if (out_logprob) out_logprob[t] = at * inv_t - m - logf(se);
  }
}

template <int KV>
cudaError_t go(const float *logits, long long ld, int T, int V, const float *temperature, const float *top_p,
               const unsigned long long *seeds, const unsigned long long *steps, uint32_t *out, int vocab_offset, float *out_val,
               float *out_sumexp, float *out_logprob, cudaStream_t st) {
  static DeviceOnce once;
  DIS_CUDA_TRY(once.run([&] { return cudaFuncSetAttribute(sample_cluster_kernel<KV>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBinsBytes); }));
  return launch_k(sample_cluster_kernel<KV>, dim3((unsigned)T * kCl), dim3(kThr), (size_t)kBinsBytes, st, logits, ld, V, temperature, top_p,
                  seeds, steps, out, vocab_offset, out_val, out_sumexp, out_logprob);
}

}  // namespace

// The smallest number of float4 per thread that holds the row.
cudaError_t launch_sample_cluster(const float *logits, long long ld, int T, int V, const float *temperature, const float *top_p,
                                  const unsigned long long *seeds, const unsigned long long *steps, uint32_t *out, int vocab_offset,
                                  float *out_val, float *out_sumexp, float *out_logprob, cudaStream_t st) {
  const int need = (V + kCl * kThr * 4 - 1) / (kCl * kThr * 4);
  auto f = need <= 1 ? go<1> : need <= 2 ? go<2> : need <= 4 ? go<4> : need <= 8 ? go<8> : go<16>;
  return f(logits, ld, T, V, temperature, top_p, seeds, steps, out, vocab_offset, out_val, out_sumexp, out_logprob, st);
}

}  // namespace dis
