// Device helpers of the sequence-persistent LSTM kernels (lstm_seq.cu, lstm_seq_bwd.cu, lstm_bwd_wide.cu): bounded polling of hand-over
// counters in global memory, cluster-scope mbarrier operations, named-barrier reductions.
#pragma once
#include "tc_dev.cuh"

namespace {

constexpr uint32_t kPollLimit = 1u << 22;      // polls of a global counter before a CTA gives up (~ seconds)
constexpr uint32_t kSeqBufs = 4;               // TMEM accumulators (4 x 128 columns)
constexpr int SMEM_SEQ_BYTES = SMEM_BYTES + BM * 64 * 4;   // operand ring (3 x 64 KiB or 4 x 48 KiB) + a 64-column exchange buffer


__device__ __forceinline__ bool wait_counter(const uint32_t* p, uint32_t target) {
  for (uint32_t i = 0; i < kPollLimit; ++i) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v >= target) return true;
  }
  return false;
}
__device__ __forceinline__ uint32_t peek_counter(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void signal_counter(uint32_t* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
// mbarrier wait that also orders after arrivals from other CTAs of the cluster
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, uint32_t limit = kWaitLimit) {
  uint32_t done = 0;
  for (uint32_t it = 0; it < limit; ++it) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// arrive on the same barrier of CTA `rank` of this cluster
__device__ __forceinline__ void mbar_arrive_remote(uint64_t* bar, uint32_t rank) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(bar)), "r"(rank));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(ra) : "memory");
}
__device__ __forceinline__ uint32_t bar_and(uint32_t id, uint32_t count, bool pred) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.and.pred p, %2, %3, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(r) : "r"((uint32_t)pred), "r"(id), "r"(count) : "memory");
  return r;
}
// 16 columns of two accumulators
__device__ __forceinline__ void tmem_ld16x2(uint32_t t1, uint32_t t2, float* v1, float* v2) {
  uint32_t *r = reinterpret_cast<uint32_t*>(v1), *x = reinterpret_cast<uint32_t*>(v2);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
               "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]),
                 "=r"(x[7]), "=r"(x[8]), "=r"(x[9]), "=r"(x[10]), "=r"(x[11]), "=r"(x[12]), "=r"(x[13]), "=r"(x[14]), "=r"(x[15])
               : "r"(t1), "r"(t2)
               : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Four neighbouring values of a row of units, `left` of which are there (VEC: all, on 16 bytes)
template <bool VEC>
__device__ __forceinline__ float4 ldu(const float* p, uint32_t left) {
  if (VEC) return ld4(p);
  return make_float4(p[0], left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}
template <bool VEC>
__device__ __forceinline__ float4 ldu_cg(const float* p, uint32_t left) {   // (from L2)
  if (VEC) return __ldcg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldcg(p), left > 1 ? __ldcg(p + 1) : 0.f, left > 2 ? __ldcg(p + 2) : 0.f, left > 3 ? __ldcg(p + 3) : 0.f);
}
template <bool VEC>
__device__ __forceinline__ void stu(float* p, float4 v, uint32_t left) {
  if (VEC) { st4(p, v); return; }
  p[0] = v.x;
  if (left > 1) p[1] = v.y;
  if (left > 2) p[2] = v.z;
  if (left > 3) p[3] = v.w;
}
// The exchange buffer: columns of BM rows, quads of rows moved about so that the 16-byte stores of four neighbouring columns meet no bank twice.
__device__ __forceinline__ uint32_t park_at(uint32_t col, uint32_t quad) { return col * BM + 4 * (quad ^ (2 * (col & 3))); }
// v: four columns of this lane's row -> rows 4 (lane / 4) .. + 3 of column lane % 4.  (One 16-byte message to another CTA instead of four.)
__device__ __forceinline__ float4 transpose4(const float* v, uint32_t lane) {
  const bool o = lane & 1, h = lane & 2;
  float x = __shfl_xor_sync(0xffffffffu, o ? v[0] : v[1], 1), y = __shfl_xor_sync(0xffffffffu, o ? v[2] : v[3], 1);
  const float a0 = o ? x : v[0], a1 = o ? v[1] : x, b0 = o ? y : v[2], b1 = o ? v[3] : y;   // columns lane % 2 and 2 + lane % 2, two rows each
  x = __shfl_xor_sync(0xffffffffu, h ? a0 : b0, 2);
  y = __shfl_xor_sync(0xffffffffu, h ? a1 : b1, 2);
  return h ? make_float4(x, y, b0, b1) : make_float4(a0, a1, x, y);
}
// Messages to the shared memory of a CTA of the cluster that count towards an mbarrier beside their destination.  (Plain remote stores and an arrival
// that releases them took a round trip: the 32 KB of partial sums of a 128 x 64 tile were with their ranks 2.0 us after the last chain, this way 1.2.)
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void send4(uint32_t to, float4 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
               : "memory");
}

}  // namespace
