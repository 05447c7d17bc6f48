// ptx.cuh -- inline-PTX wrappers shared by the TMA-fed kernels: mbarrier, cp.async.bulk.tensor (TMA),
// programmatic dependent launch (griddepcontrol), and a launch helper that sets the PDL attribute.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace dis {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// A wait that never comes true (a TMA box that does not match the bytes the barrier expects, a lost arrive) would
// hang the GPU until a watchdog kills the process: after ~2^26 failed polls -- tens of seconds, no legitimate wait in
// these kernels is longer than milliseconds -- the kernel traps instead, which fails the launch with an error.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok, polls = 0;
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (!ok && ++polls > (1u << 26)) __trap();
  } while (!ok);
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tma_prefetch_desc(const void *map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
// 2-D tile load: coordinates {c0 = element offset along the contiguous dim, c1 = row}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void *map, int c0, int c1, uint32_t bar,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
// The same tile into L2 only.  L2 is where writes of running kernels meet reads, so what a kernel ahead still writes arrives there too.
__device__ __forceinline__ void tma_prefetch_2d(const void *map, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(c0), "r"(c1) : "memory");
}
constexpr uint64_t kEvictFirst = 0x12F0000000000000ull;  // stream-once data (weights)
constexpr uint64_t kEvictLast = 0x14F0000000000000ull;   // data every CTA re-reads (activations)


// ---- tcgen05 / TMEM ------------------------------------------------------------------------------
constexpr int kBM = 128;           // output features per GEMM tile (TMEM lanes)
constexpr int kBK = 64;            // bf16 per 128-byte swizzle row
constexpr int kGemmThreads = 192;  // warp 0 TMA, warp 1 MMA + TMEM alloc, warps 2-5 epilogue

template <int kCols>
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "n"(kCols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int kCols>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(kCols) : "memory");
}
// The issue path.  A batch of MMAs costs its issuing thread some twenty dependent instructions each when every descriptor is built
// from an address in front of it (measured with clock stamps: 140 clocks per MMA on a busy SM, against 32 to 64 that the MMA takes), so
// the descriptors' upper halves are a constant (SBO = 1024 bytes, version 1, 128B swizzle), the lower halves are built once and
// stepped by an add, and the issuing warp runs its loop converged, with one elected lane for the MMAs, so that these values stay in
// uniform registers.
// Shared-memory matrix descriptor, canonical 128B-swizzle layout (rows of 64 bf16 = 128 B, 8-row groups 1024 B apart):
// start >> 4 | LBO << 16 | SBO << 32 | version 1 << 46 | SW128 << 61.
constexpr uint32_t kUmmaDescHi = 64u | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t umma_lo(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFFu) | (1u << 16); }  // K-major
__device__ __forceinline__ uint32_t umma_lo_mn(uint32_t smem_addr, uint32_t lbo_bytes) { return ((smem_addr >> 4) & 0x3FFFu) | ((lbo_bytes >> 4) << 16); }
// D[tmem] (+)= A[smem] * B[smem]^T, bf16 x bf16 -> fp32
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
      : "memory");
}
// A from TMEM: 128 lanes x 16 bf16, two per column
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
      : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// mbarrier arrives once all MMAs issued so far by this thread have completed
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 lanes x 32 consecutive fp32 columns -> 32 registers per thread (thread = lane = accumulator row)
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Instruction descriptor: D=f32, A=B=bf16, both K-major, M=128, N=kN.
template <int kN>
__host__ __device__ constexpr uint32_t umma_idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// ---- programmatic dependent launch ------------------------------------------------------------
// A kernel launched with the PDL attribute may start while its predecessor in the stream is still
// running.  pdl_wait() blocks until every prerequisite grid has completed and its writes are
// visible: it must precede the first read of data a previous kernel produced and the first global
// write.  pdl_launch_dependents() lets the NEXT kernel in the stream begin its own prologue.
// Both are no-ops for a kernel launched without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Host: whether launches made through launch_k() on this thread carry the PDL attribute.
bool &pdl_enabled();
// Host: whether the weights of the products launched on this thread may be read before pdl_wait().  True for an engine, whose weights
// are written once; false for a call of the C ABI, whose weight may be what the kernel in front of it writes.
bool &pdl_weights_settled();

// cluster > 1: clusters of that many CTAs along x (kernels with __cluster_dims__ carry their own size)
template <class... KArgs, class... Args>
cudaError_t launch_k_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  cfg.attrs = at;
  if (pdl_enabled()) {
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[cfg.numAttrs++].val.clusterDim = {(unsigned)cluster, 1u, 1u};
  }
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <class... KArgs, class... Args>
cudaError_t launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  return launch_k_cluster(kern, grid, block, smem, st, 1, args...);
}

// Gate activation of the products' epilogues, whose result is rounded to bf16 at once: kind 0 = silu(g) = g sigmoid(g), kind 1 =
// gelu_tanh(g) = 0.5 g (1 + tanh y) = g sigmoid(2 y) with y = sqrt(2/pi) (g + 0.044715 g^3).  The approximate exponential and
// division are good to a few parts in 10^6 and keep the epilogue warp free of the exact division's branches.
__device__ __forceinline__ float gate_act_fast(int kind, float g) {
  const float z = kind == 1 ? 1.5957691216057308f * fmaf(0.044715f * g * g, g, g) : g;
  return __fdividef(g, 1.f + __expf(-z));
}

}  // namespace dis
