// k_sample.cu -- the sampler (argmax / temperature + nucleus) with a row spread over a cluster of eight CTAs.
// No reference counterpart; the sampling controls are InferenceParams (design.md:666-671), the definition of the draw is the
// oracle's: nucleus = {p >= tau}, tau the largest threshold whose kept mass reaches top_p, one uniform per (seed, step), first kept
// token in index order whose running mass exceeds u * kept.
//
// What bounds it: latency.  A row of 128256 logits is 513 KB; one CTA per row (sample_kernel in k_elementwise.cu, which stays
// for rows longer than kSampleClusterMaxV) walks it 30 to 40 times through one SM's L2 port, on as many SMs as there are rows: 701 us
// for 32 rows of 128256, three quarters of them sampled, against 24.7 us here.  Here the eight CTAs of a cluster read the row ONCE and keep it in
// registers (at most 16 float4 per thread); everything after that is arithmetic on registers.  The nucleus threshold is found in four exchanges:
//   * the octave (exponent) it lies in: a thread adds each of its weights to its own column of a [32][512] table (no atomics: the sums
//     keep one order and a repeated call gives the same bits), the table's rows are summed per CTA and swapped through distributed shared
//     memory.  The total is the softmax's denominator, which needs no exchange of its own;
//   * its 23 mantissa bits, 8 + 8 + 7: within an octave every weight is a whole number of the same unit, so masses are exact sums of
//     24-bit integers and may be added by shared-memory atomics in any order; few weights take part, and a round costs a cluster barrier
//     and little else.  (Six rounds of the table, five bits each, took 4.5 us apiece: clearing and summing 64 KB.)
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
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster(const float *p, uint32_t rank, float v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

constexpr int kFine = 256;      // thresholds per round within an octave
constexpr int kFineRounds = 3;
static_assert(kFineRounds * kCl * 2 * kFine * 4 <= kBinsBytes, "the fine rounds' exchanges lie in the table");

struct Sh {
  float mine[kBins];                 // what this CTA gives away in an exchange
  float all[2][kCl][kBins];          // what every CTA gave; two halves in turn, so one exchange never overwrites what the last is read from
  float wv[kWarps];
  double wd[kWarps];
  int wi[kWarps];
  int tok;
  uint32_t fine[kFineRounds][2][kFine];  // a CTA's masses in the octave's unit: sums of the low 12 bits, of the high 12
  unsigned long long part[kFine / 32];
  int pick[kFineRounds];
  unsigned long long pick_above[kFineRounds];
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
  cluster_arrive();
  for (int i = threadIdx.x; i < kFineRounds * 2 * kFine; i += kThr) (&s.fine[0][0][0])[i] = 0u;
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
  cluster_wait();  // every CTA of the cluster is running: its shared memory may be written from now on
  __syncthreads();
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
  // ---- weights exp(z - max) and their sum; a greedy row is done with it
  const bool greedy = temp <= 0.f;
  const float tp = !greedy && top_p ? top_p[t] : 1.0f;
  const bool nucleus = tp < 1.0f;
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
    if (!nucleus) {
      part = sum_block(s, part);
      if (threadIdx.x == 0) s.mine[0] = part;
      swap(s, me, 1, par);
#pragma unroll
      for (int r = 0; r < kCl; r++) se += s.all[par][r][0];
      par ^= 1;
    }
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
  // ---- nucleus threshold: the largest bit pattern whose mass (the sum of all weights at or above it) still reaches top_p of the whole
  uint32_t tau = 0u;
  if (nucleus) {
    // The octave: bin b holds exponent low + b, bin 0 everything below as well (then the search goes on there: a nucleus that
    // reaches below 2^-30 of the largest weight).  The first search's last bin also takes NaN, whatever its sign: the sum is NaN then,
    // no threshold holds and everything is kept.
    float above = 0.f, goal = 0.f;
    int low = 96, top = 511, oct = 0;
    for (;;) {
#pragma unroll
      for (int b = 0; b < kBins; b++) bins[b * kThr + threadIdx.x] = 0.f;
#pragma unroll
      for (int k = 0; k < KV; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int e = (int)(__float_as_uint(v[k][j]) >> 23);
          if (e <= top && v[k][j] != 0.f) bins[min(max(e - low, 0), kBins - 1) * kThr + threadIdx.x] += v[k][j];
        }
      __syncthreads();
      // warp w sums rows 2 w and 2 w + 1 of the table
#pragma unroll
      for (int h = 0; h < kBins / kWarps; h++) {
        const int b = warp * (kBins / kWarps) + h;
        float x = 0.f;
#pragma unroll
        for (int i = 0; i < kThr / 128; i++) {
          const float4 f = *reinterpret_cast<const float4 *>(bins + b * kThr + i * 128 + lane * 4);
          x += (f.x + f.y) + (f.z + f.w);
        }
        x = warp_sum(x);
        if (lane == 0) s.mine[b] = x;
      }
      swap(s, me, kBins, par);
      // every thread: lane j holds bin j's mass over the cluster, then the mass at or above bin j
      float suf = 0.f;
#pragma unroll
      for (int r = 0; r < kCl; r++) suf += s.all[par][r][lane];
      par ^= 1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += n;
      }
      if (top == 511) {
        se = __shfl_sync(0xffffffffu, suf, 0);
        goal = tp * se;
      }
      const uint32_t ok = __ballot_sync(0xffffffffu, above + suf >= goal) | 1u;
      const int j = 31 - __clz(ok);
      const float next = __shfl_sync(0xffffffffu, suf, (j + 1) & 31);
      if (j < 31) above += next;
      oct = low + j;
      if (j > 0 || low == 0 || se != se) break;
      top = low;
      low = max(low - (kBins - 1), 0);
    }
    if (se == se) {
      // The mantissa.  The octave's unit is the spacing of its numbers; subnormal numbers share the first normal octave's.
      double need = ldexp((double)goal - (double)above, 150 - max(oct, 1));
      const uint32_t one = oct > 0 ? 0x800000u : 0u;
      uint32_t *area = reinterpret_cast<uint32_t *>(bins);  // [round][CTA][2][kFine]; every CTA has read its table
      uint32_t prefix = 0u;
#pragma unroll 1
      for (int round = 0; round < kFineRounds; round++) {
        const int sh = round == 0 ? 15 : round == 1 ? 7 : 0, bits_here = round == 2 ? 7 : 8;
        const uint32_t want = ((uint32_t)oct << (23 - sh - bits_here)) | prefix;  // what stands above this round's bits
#pragma unroll
        for (int k = 0; k < KV; k++)
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const uint32_t bits = __float_as_uint(v[k][j]);
            if (bits >> (sh + bits_here) == want && bits != 0u) {
              const uint32_t b = (bits >> sh) & ((1u << bits_here) - 1u), w = (bits & 0x7fffffu) | one;
              atomicAdd(&s.fine[round][0][b], w & 0xfffu);
              atomicAdd(&s.fine[round][1][b], w >> 12);
            }
          }
        __syncthreads();
        uint32_t *to = area + (size_t)(round * kCl + me) * (2 * kFine);
        for (int i = threadIdx.x; i < 2 * kFine; i += kThr) {
          const float x = __uint_as_float((&s.fine[round][0][0])[i]);
#pragma unroll
          for (int r = 0; r < kCl; r++) st_cluster(reinterpret_cast<const float *>(to + i), (uint32_t)r, x);
        }
        cluster_sync_all();
        unsigned long long mass = 0, suf = 0;
        if (threadIdx.x < kFine) {
          const uint32_t *from = area + (size_t)round * kCl * (2 * kFine) + threadIdx.x;
          uint32_t lo = 0, hi = 0;
#pragma unroll
          for (int r = 0; r < kCl; r++) { lo += from[r * 2 * kFine]; hi += from[r * 2 * kFine + kFine]; }
          mass = suf = ((unsigned long long)hi << 12) + lo;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long n = __shfl_down_sync(0xffffffffu, suf, o);
            if (lane + o < 32) suf += n;
          }
          if (lane == 0) s.part[warp] = suf;
        }
        __syncthreads();
        if (threadIdx.x < kFine) {
          for (int w = warp + 1; w < kFine / 32; w++) suf += s.part[w];
          // the largest threshold that holds (threshold 0 does, by what the last round chose): exactly one thread finds it
          if ((threadIdx.x == 0 || (double)suf >= need) && (threadIdx.x == kFine - 1 || !((double)(suf - mass) >= need))) {
            s.pick[round] = threadIdx.x;
            s.pick_above[round] = suf - mass;
          }
        }
        __syncthreads();
        prefix = (prefix << bits_here) | (uint32_t)s.pick[round];
        need -= (double)s.pick_above[round];
      }
      tau = ((uint32_t)oct << 23) | prefix;
    }
  }
  tau = max(tau, 1u);  // a weight of zero (a masked logit, an underflow) is never kept: no draw may return it
  // ---- draw: first kept token in index order whose running mass exceeds u * kept.  Positions on the scale of the whole mass are 64-bit
  // numbers (a thread's own sum and a chunk's scan are not): in 32 bits the scale's grain is that of a token of weight 10^-7.
  float local = 0.f;
#pragma unroll
  for (int k = 0; k < KV; k++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (__float_as_uint(v[k][j]) >= tau) local += v[k][j];
  double wsum = (double)local;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
  if (lane == 0) s.wd[warp] = wsum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0.;
    for (int w = 0; w < kWarps; w++) x += s.wd[w];
    s.mine[0] = __int_as_float(__double2loint(x));
    s.mine[1] = __int_as_float(__double2hiint(x));
  }
  swap(s, me, 2, par);
  auto cta_mass = [&](int r) { return __hiloint2double(__float_as_int(s.all[par][r][1]), __float_as_int(s.all[par][r][0])); };
  double kept = 0.;
#pragma unroll
  for (int r = 0; r < kCl; r++) kept += cta_mass(r);
  const double target = (double)hash_u01(mix64(seeds ? seeds[t] : 0ull, 0xC0FFEEull, steps ? steps[t] : 0ull)) * kept;
  int owner = -1;
  double start = 0., run = 0.;
#pragma unroll
  for (int r = 0; r < kCl; r++) {
    const double x = cta_mass(r);
    if (owner < 0 && x > 0. && target < run + x) { owner = r; start = run; }
    run += x;
  }
  if (owner < 0 ? me != 0 : me != owner) return;  // no exchange follows
  if (owner >= 0) {
    int w_own = -1, w_last = 0;
    double w_start = start, w_last_start = start, x = start;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      const double y = s.wd[w];
      if (y > 0.) { w_last = w; w_last_start = x; }
      if (w_own < 0 && y > 0. && target < x + y) { w_own = w; w_start = x; }
      x += y;
    }
    if (w_own < 0) { w_own = w_last; w_start = w_last_start; }  // rounding: the CTA's last kept piece
    if (warp == w_own) {
      double at = w_start;
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
        double x2 = lane == 0 ? at : at + (double)before;
        int first = 0x7fffffff, end = -1;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          x2 = j < 3 ? x2 + (double)kp[j] : at + (double)incl;
          if (in[j]) { end = base + k * 128 + j; if (x2 > target && first == 0x7fffffff) first = end; }
        }
        first = __reduce_min_sync(0xffffffffu, first);
        end = __reduce_max_sync(0xffffffffu, end);
        if (tok < 0 && first != 0x7fffffff) tok = first;
        if (end >= 0) last = end;
        at += (double)__shfl_sync(0xffffffffu, incl, 31);
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
