// Device-side building blocks shared by the Triadic GDN kernels (sm_100a only):
// mbarrier / TMA / tcgen05 wrappers in inline PTX, shared-memory operand layouts and their matrix descriptors.
//
// Reference counterpart: cute_triadic_gdn/kernels/sm100_tc.py:1-166 (the reference emits the same PTX
// instructions from its Python DSL); this file is an independent CUDA C++ formulation.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tgdn {

constexpr int CHUNK = 64;     // tokens per chunk
constexpr int HEAD = 128;     // key and value head dimension

// Device status word values (first failure wins).  A kernel that gives up on a wait records one of these and
// runs to its end without waiting again, so the launch always terminates and the context stays usable.
enum DeviceStatus : int {
  DEV_OK = 0,
  DEV_TIMEOUT_LOAD = 1,    // a TMA / bulk-copy transaction barrier did not complete in time
  DEV_TIMEOUT_MMA = 2,     // a tcgen05.commit barrier did not complete in time
  DEV_BAD_CHUNK_MAP = 3,   // a chunk-map entry pointed outside the token range
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------------------------------------
// mbarrier
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Non-blocking probe: unlike try_wait it never parks the warp, so a spinning waiter sees the flip within a few cycles.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Shared per-CTA control block of a kernel with bounded waits.
struct WaitCtl {
  volatile int* abort;   // shared-memory flag: once set, every wait of the CTA returns at once
  int* status;           // global status word
};

constexpr long long WAIT_LIMIT_CYCLES = 1ll << 31;   // about a second of SM clocks

// Wait for `parity` of `bar`; gives up after WAIT_LIMIT_CYCLES, records `code` and raises the CTA's abort flag.
// Spins on the non-parking probe, which sees the flip within a few cycles: for waits that are over as a rule when they begin.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const WaitCtl& ctl, int code,
                                          long long limit_cycles = WAIT_LIMIT_CYCLES) {
#pragma unroll 1
  for (int it = 0; it < 2048; ++it)
    if (mbar_test_wait(bar, parity)) return true;
  const long long start = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_test_wait(bar, parity)) return true;
    if ((it & 63u) == 0u) {
      if (*ctl.abort) return false;
      if (clock64() - start > limit_cycles) {
        *ctl.abort = 1;
        atomicCAS(ctl.status, DEV_OK, code);
        return false;
      }
    }
  }
}
// The same wait for a warp that has long to wait beside others that work: the probe parks the warp for at most PARK_NS.  A poll is an
// access to shared memory, and where that path is the bottleneck a dozen polling warps take a third of it (what each kernel gained, and
// lost where such a wait took the place of one that is over as a rule, stands in its file).
constexpr uint32_t PARK_NS = 200;
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      "selp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(PARK_NS)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_parked(uint64_t* bar, uint32_t parity, const WaitCtl& ctl, int code,
                                                 long long limit_cycles = WAIT_LIMIT_CYCLES) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0u) {
      if (*ctl.abort) return false;
      if (clock64() - start > limit_cycles) {
        *ctl.abort = 1;
        atomicCAS(ctl.status, DEV_OK, code);
        return false;
      }
    }
  }
}
// The parked wait of a whole warp: its lanes look together and have one outcome.  (A vote on what each lane's own wait returned would come on
// top of their loops: with the loads of the fused gradient kernel waiting that way, its backward took 0.5 % longer.)
__device__ __forceinline__ bool mbar_wait_parked_warp(uint64_t* bar, uint32_t parity, const WaitCtl& ctl, int code,
                                                      long long limit_cycles = WAIT_LIMIT_CYCLES) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long start = clock64();
  for (uint32_t it = 1;; ++it) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((it & 63u) == 0u) {
      if (__any_sync(0xffffffffu, *ctl.abort)) return false;
      if (__any_sync(0xffffffffu, clock64() - start > limit_cycles)) {
        *ctl.abort = 1;
        atomicCAS(ctl.status, DEV_OK, code);
        return false;
      }
    }
  }
}
// One verdict for warps that go through named barriers together: that of the thread which leads them.  A wait may be met for one warp and given
// up by another; whoever acts on its own outcome leaves the others at the next barrier for good.  `word` (shared) is free for the next
// verdict behind another barrier of the same warps.
template <int BARRIER, int THREADS>
__device__ __forceinline__ bool one_verdict(bool mine, bool leads, volatile int* word) {
  if (leads) *word = mine ? 1 : 0;
  asm volatile("bar.sync %0, %1;" ::"n"(BARRIER), "n"(THREADS) : "memory");
  return *word != 0;
}
__device__ __forceinline__ bool mbar_wait_spin(uint64_t* bar, uint32_t parity, const WaitCtl& ctl, int code) {
  return mbar_wait(bar, parity, ctl, code);
}

// ------------------------------------------------------------------------------------------------
// TMA (tensor-map tiles and plain bulk copies), completion on an mbarrier.  No multicast anywhere.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// Tile store shared -> global (bulk async-group completion).  The issuing thread commits the group and, before the
// shared-memory source may be overwritten, waits until the group's reads of shared memory are done.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(map), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3, int c4) {
  asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
               ::"l"(map), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
               : "memory");
}
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3, int c4) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_group_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// 1-D bulk copy shared -> global, in the thread's current bulk group; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_wait_group() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// 1-D bulk copy global -> shared; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Hints that pull a tile / a byte range into L2 ahead of the real load (no shared memory, no completion to wait for).
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];"
               ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void bulk_prefetch(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// Generic-proxy writes to shared memory -> visible to the async proxy (tcgen05.mma operands, bulk stores).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ------------------------------------------------------------------------------------------------
// tcgen05: tensor memory, MMA, commit, loads
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {   // one whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {     // one whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]; bf16 operands, f32 accumulator; issued by ONE thread.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive once on `bar` when every tcgen05.mma issued so far by this thread has completed.
// One lane of a fully active warp.  Tensor-core and TMA instructions are issued as "warp-uniform branch, then elected
// lane": their operands then stay warp-uniform values, which a branch on the thread index would not allow.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// tcgen05.ld 32x32b: lane L of the warp reads row (lane base + L); N consecutive f32 columns.  The lane base in
// `taddr` must be 32 * (warp index % 4).
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// N columns (multiple of 4) starting at taddr, in the widest pieces available; the caller waits with tmem_wait_ld().
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float* v) {
  static_assert(N % 4 == 0, "column count must be a multiple of 4");
  int done = 0;
#pragma unroll
  for (; done + 16 <= N; done += 16) tmem_ld16(taddr + done, v + done);
  if (N - done >= 8) { tmem_ld8(taddr + done, v + done); done += 8; }
  if (N - done >= 4) { tmem_ld4(taddr + done, v + done); }
}

// ------------------------------------------------------------------------------------------------
// Shared-memory operand layouts (bf16) and descriptors
//
// (1) SW128 tile: rows of 64 elements (128 bytes), 16-byte pieces XOR-swizzled with (row % 8); what a TMA tile load with
//     128-byte swizzle writes.  The tile base must be 1024-byte aligned.  Wider matrices are several such 64-column
//     blocks.  Read as K-major when the 64-element rows run along K, as MN-major when they run along M or N.
// (2) Plain image: 8x8 core matrices of 128 contiguous bytes; element (i, j) with j the direction that is contiguous
//     inside a 16-byte piece:  off = (i/8)*SI + (j/8)*SJ + (i%8)*16 + (j%8)*2.
//     K-major use (j = K):  SBO = SI, LBO = SJ.   MN-major use (j = M or N, i = K):  SBO = SJ, LBO = SI.
// ------------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint32_t sw128_off(uint32_t row, uint32_t col /* 0..63 */) {
  return row * 128u + ((((col >> 3) ^ row) & 7u) << 4) + ((col & 7u) << 1);
}
__host__ __device__ __forceinline__ uint32_t img_off(uint32_t i, uint32_t j, uint32_t SI, uint32_t SJ) {
  return (i >> 3) * SI + (j >> 3) * SJ + ((i & 7u) << 4) + ((j & 7u) << 1);
}

constexpr uint32_t LAYOUT_PLAIN = 0;
constexpr uint32_t LAYOUT_SW128 = 2;

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout) {
  uint64_t d = static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;                                   // descriptor version of this architecture
  d |= static_cast<uint64_t>(layout) << 61;
  return d;
}
__device__ __forceinline__ uint64_t desc_advance(uint64_t d, uint32_t bytes) { return d + (bytes >> 4); }

// kind::f16 instruction descriptor: bf16 A and B, f32 D.  major: 0 = K-major, 1 = MN-major.
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, int a_major, int b_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_major) << 15) |
         (static_cast<uint32_t>(b_major) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

// N floats from shared memory; 16-byte loads where N and the address allow, else 8-byte loads (N even) or one float
template <int N>
__device__ __forceinline__ void lds_part(const float* p, float* out) {
  if constexpr (N == 1) {
    out[0] = p[0];
  } else if constexpr (N % 4 == 0) {
#pragma unroll
    for (int j = 0; j < N / 4; ++j) {
      const float4 x = *(reinterpret_cast<const float4*>(p) + j);
      out[4 * j] = x.x; out[4 * j + 1] = x.y; out[4 * j + 2] = x.z; out[4 * j + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < N / 2; ++j) {
      const float2 x = *(reinterpret_cast<const float2*>(p) + j);
      out[2 * j] = x.x; out[2 * j + 1] = x.y;
    }
  }
}
// N floats from entry e0 on of row t of a dense table of E floats a row, where the lanes of a warp read a row each.  Rows of 32 and
// 64 bytes put every second or fourth lane on the same banks (sixteen wavefronts a load instead of four): there the lanes take the two
// 16-byte pieces in an order that depends on the row (ORDERED).
template <int E, int N, bool ORDERED = E == 8 || E == 16>
__device__ __forceinline__ void lds_row(const float* table, int t, int e0, float* out) {
  const float* p = table + t * E + e0;
  if constexpr (ORDERED && N == 8) {
    const bool swap = (t & (E == 8 ? 4 : 2)) != 0;
    const float4 x = *reinterpret_cast<const float4*>(p + (swap ? 4 : 0)), y = *reinterpret_cast<const float4*>(p + (swap ? 0 : 4));
    out[0] = swap ? y.x : x.x; out[1] = swap ? y.y : x.y; out[2] = swap ? y.z : x.z; out[3] = swap ? y.w : x.w;
    out[4] = swap ? x.x : y.x; out[5] = swap ? x.y : y.y; out[6] = swap ? x.z : y.z; out[7] = swap ? x.w : y.w;
  } else {
    lds_part<N>(p, out);
  }
}

// Two f32 fused multiply-adds in one instruction (each lane an ordinary fma): the epilogues of the recurrences are bound by
// instruction issue.
__device__ __forceinline__ void fma_pair(float& a0, float& a1, float f, float x0, float x1) {        // a += f * x
  const float2 r = __ffma2_rn(make_float2(f, f), make_float2(x0, x1), make_float2(a0, a1));
  a0 = r.x; a1 = r.y;
}
__device__ __forceinline__ void scale_add_pair(float& a0, float& a1, float f, float x0, float x1) {  // a = f * a + x
  const float2 r = __ffma2_rn(make_float2(f, f), make_float2(a0, a1), make_float2(x0, x1));
  a0 = r.x; a1 = r.y;
}

// ------------------------------------------------------------------------------------------------
// small helpers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);    // .x (low half, lower address) = lo
  return *reinterpret_cast<uint32_t*>(&p);
}
// Two bf16 products at once, each rounded to nearest: scaling a packed row by a packed factor costs one instruction per
// pair where unpacking, two f32 multiplies and a repack cost five.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ void st_shared_v4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

}  // namespace tgdn
