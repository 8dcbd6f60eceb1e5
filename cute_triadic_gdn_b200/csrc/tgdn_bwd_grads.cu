// State gradients and matrix gradients of the Triadic GDN backward in one kernel: everything behind the reverse recurrence.
//
// Persistent CTAs (one per SM) walk the (batch, chunk, head) items.  What the state-gradient kernel does with an item (tgdn_bwd_sg.cu:
// a stream of the saved states h through the tensor core, bound by HBM) and what the matrix-gradient kernel does with it
// (tgdn_bwd_mat.cu: a chain of five small product groups with sums over the slices between them, bound by latency) need each other
// only at the item's end, so they run side by side on warps of their own:
//   warps 0..7    "stream": per slice P_e = [dW ; dO] h_e^T from tensor memory: row sums against K, Q (da_e, dc_e) and the gate-weighted
//                 sum over the slices (f32, registers); at the end of the item dk, dq = that sum + the value-block images + G5
//   warps 8..15   "chain": gate tables, masks and their gradients, dA, dL, ... and dk2, dq2, dg, dbeta
//   warp 16       issues the products of the stream (P_e, traces, value-block images)
//   warp 17       loads: one ring of 16 KB stages through which dU, W, U, the half-slices of h (and G) and the value-block images pass,
//                 and the [dW;dO] tile
//   warp 18       loads [K;Q] and A, issues the chain's first products (G1, G2) and its last (G5)
// The formulas are those of the two kernels, value by value in the same order: the results are bitwise those of running them one after
// the other (dkq rounded to bf16 included), which tests/test_abi_gpu.py and tests/test_grads_gpu.py check.  What need not travel any more: dkq (32 KB an item there and
// back), da, dc, dd, and the second load of K, Q and dO: 518 KB of DRAM traffic an item at eight slices instead of 660.
//
// Tensor memory: the tiles P_e and, as the last one, the value-block sum in a double buffer (columns 0..255), G5 (256..383, before that G1
// in its first 64 columns and dA', Y, dp in turn in its last 64), traces h_e G_e^T (384..511, before that dPm' in the first 64 columns).
//
// What bounds it: the memory (518 KB an item at eight slices; 5.2 TB/s) and, close behind, the shared-memory path, which the chain's table
// rows, the stream's tensor-memory and K reads, the products' operands and the arriving tiles share; waiting warps park instead of
// polling for that reason (8192 items E8 939 -> 839 us when that was done).  us, state gradients + matrix gradients as two kernels -> this
// one: 8192 items E8 690 + 505 -> 811, with slow decays 845 + 501 -> 1205; 4096 items E1 148 + 200 -> 226, E4 238 + 225 -> 294.  Pulling tiles
// into L2 ahead of the ring, which helped the kernel of the states alone, costs 10 to 20 % here.  At eight, twelve and sixteen slices the
// chain does not fit its registers (-Xptxas -v: 48, 132 and 460 bytes of spill stores; 4 to 8 below): with this much
// shared memory in use a spilled value is a round trip to L2.
//
// Replaces cute_triadic_gdn/kernels/sm100_joint_state_grads.py:53-449, sm100_joint_bwd_parallel.py:80-405,
// sm90_joint_bwd_parallel.py:278-372 (mask_grad_kernel) and the reverse pass of sm90_joint_scan.py:21-80.
#include "tgdn_common.cuh"
#include "tgdn_host.h"
#include "tgdn_kernels.h"
#include "tgdn_mat.cuh"

namespace tgdn {

constexpr int GR_THREADS = 20 * 32;   // (warp 19 only completes its warpgroup)
// Registers a thread: 96 at launch (five warps on each quarter of an SM), then the two warpgroups of a role take what the last one gives
// back: 2 * 112 + 2 * 104 + 48 = 480 of 480 (40 for the service warps spilled 8 bytes more at one slice).
constexpr int GR_STREAM_REGS = 112, GR_CHAIN_REGS = 104, GR_SERVICE_REGS = 48;
static_assert(2 * GR_STREAM_REGS + 2 * GR_CHAIN_REGS + GR_SERVICE_REGS <= 5 * 96, "registers of the block");
template <int N> __device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr int TM_G5 = 256, TM_G1 = 256, TM_DA = 320, TM_Y = 320, TM_DPM = 384, TM_T = 384;

// f32 lower triangle of a 64x64 matrix as ten 16x16 blocks with rows 20 floats apart, blocks 336: neither a lane per row that writes
// 16-byte pieces nor a lane per column that reads floats meets a bank twice.
constexpr int TRI_FLOATS = 10 * 336;
__device__ __forceinline__ int tri_block(int bi, int bj) { return (bi * (bi + 1) / 2 + bj) * 336; }

// m[j] = <G, table row j> and acc += d[j] * table row j over eight rows of a dense table of E floats that a whole warp reads: eight
// independent sums, a piece of at most eight slices at a time (registers: several rows are on their way at once).
template <int E>
__device__ __forceinline__ void slice_dots(const GateVec<E>& G, const float* table, float (&m)[8]) {
  constexpr int PIECE = E <= 8 ? E : E / 2;
  float2 a[8];
#pragma unroll
  for (int e0 = 0; e0 < E; e0 += PIECE) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      GateVec<PIECE> row;
      row.load(table + j * E + e0);
#pragma unroll
      for (int i = 0; i < row.N; ++i) a[j] = e0 + i == 0 ? __fmul2_rn(G.p[0], row.p[0]) : __ffma2_rn(G.p[e0 / 2 + i], row.p[i], a[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) m[j] = E == 1 ? a[j].x : a[j].x + a[j].y;
}
template <int E>
__device__ __forceinline__ void slice_sums(GateVec<E>& acc, const float* table, const float (&d)[8]) {
  constexpr int PIECE = E <= 8 ? E : E / 2;
  asm volatile("" ::: "memory");                           // (or the compiler keeps the rows of the first pass)
#pragma unroll
  for (int e0 = 0; e0 < E; e0 += PIECE)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      GateVec<PIECE> row;
      row.load(table + j * E + e0);
#pragma unroll
      for (int i = 0; i < row.N; ++i) acc.p[e0 / 2 + i] = __ffma2_rn(make_float2(d[j], d[j]), row.p[i], acc.p[e0 / 2 + i]);
    }
}

// Eight columns of a row: m = <G, table row j>, d = column(j, m), acc += d * table row j.  Up to eight slices four rows are held from the dot to
// the sum; above, the registers do not suffice and they are read twice.
template <int E, typename F>
__device__ __forceinline__ void slice_columns(const GateVec<E>& G, GateVec<E>& acc, const float* table, F column) {
  if constexpr (E <= 8) {
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += 4) {
      GateVec<E> row[4];
      float d[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) row[j].load(table + (j0 + j) * E);
#pragma unroll
      for (int j = 0; j < 4; ++j) d[j] = column(j0 + j, G.dot(row[j]));
#pragma unroll
      for (int j = 0; j < 4; ++j) acc.add_scaled(d[j], row[j]);
    }
  } else {
    float m[8], d[8];
    slice_dots<E>(G, table, m);
#pragma unroll
    for (int j = 0; j < 8; ++j) d[j] = column(j, m[j]);
    slice_sums<E>(acc, table, d);
  }
}

template <int E>
struct GradsSmem {
  static constexpr int ES = E | 1;
  static constexpr int NS = E > 8 ? 3 : 4;      // ring stages
  uint8_t kq[32768];            // [K;Q] tile, 128B swizzle: two column halves of 128 rows x 64 columns
  uint8_t xt[32768];            // [dW;dO] tile
  uint8_t ring[NS][16384];
  uint8_t p5[16384];            // P = [dPkk ; X], 128 rows x 64 columns, 128B swizzle (read K-major and MN-major); then dk on its way out
  uint8_t dmp[16384];           // dmp, f32 triangle; then dq on its way out
  uint8_t ap[8192];             // A image (i = t, j = s), SI = 128, SJ = 1024
  union {
    uint8_t day[8192];          // dA image (i = t, j = s), SI = 128, SJ = 1024; then Y
    float dm[TRI_FLOATS];       // then dm
  } u;
  alignas(1024) uint8_t zero[2048];   // what the MN-major read of P finds for its rows 64..127
  uint8_t ident[3584];          // 16x16 identity in a 112x16 image of zeros, SI = 128, SJ = 1792: [I;0] of a K step is a window of it
  alignas(16) float hkv[64 * E], kxv[64 * E];   // as in the matrix-gradient kernel (kxv: its second table of that name)
  alignas(16) float qxv[64 * E];      // ... and, after the chain's join, half of c2 as [slice][row]
  float gc2[64 * ES], k2[64 * ES], q2[64 * ES];
  float r1[64 * ES], c1[64 * ES], r2[64 * ES], c2[64 * ES];     // r1: then dgc; c1: then dr * r
  float sums[128 * ES];         // row sums of the stream: da (negated sums) rows 0..63, dc rows 64..127
  float red[E * 4];             // per slice and 32-row block: partial trace of h_e G_e^T
  float browp[2][64], bcolp[2][64], beta[64];
  uint64_t full[NS], empty[NS], tiles_full, kq_full, kq_free, xt_full, xt_free, p_full[2], p_free[2], t_full, t_free, g12, g2read, g34, p_ready, g5_full,
      epi_free, stage_free, sums_free, sg_done;
  struct Place { int item, h, b, t0, rows; uint32_t traces; } place[4];   // of the CTA's item `it` in slot it % 4; item -1: the end
  uint64_t drained;             // all products issued are complete
  uint32_t tmem_base;
  int abort, drain_abort;
  int stream_go, chain_go;      // verdicts of the two roles: on to the item
  int steep;
};

template <int E>
__global__ void __launch_bounds__(GR_THREADS, 1)
grads_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q,
             const __grid_constant__ CUtensorMap map_dv, const __grid_constant__ CUtensorMap map_do,
             const __grid_constant__ CUtensorMap map_du, const __grid_constant__ CUtensorMap map_w,
             const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_a,
             const __grid_constant__ CUtensorMap map_dk, const __grid_constant__ CUtensorMap map_dq, GradsParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  using SM = GradsSmem<E>;
  SM& sm = *reinterpret_cast<SM*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int ES = SM::ES, NS = SM::NS;
  constexpr float LOG2E = 1.4426950408889634f;
  // The trace of an item's first slice: up to two slices it is a tile of the double buffer (T0_TILE) and need not wait until dPm' has left the
  // tensor memory that the other traces use; above, where the chain is what an item waits for, dU, W, U pass before that slice
  // (TILES_EARLY) so that the chain starts sooner, and its trace waits.  Time of the first way against the second, slow decays:
  // 4096 items E1 -9 %, E2 -9 %, E4 0; 8192 items E8 +6 %.
  constexpr bool T0_TILE = E <= 2, TILES_EARLY = !T0_TILE;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int warp_u = __shfl_sync(0xffffffffu, warp, 0);   // warp index as a warp-uniform value
  const int NVB = p.NV;
  const int n_items = p.B * p.NC * p.H;                    // fits (checked at the entry point)

  // The CTA's first item is its own index; the loading warp takes every further one from a counter and tells the others.  (Items cost what
  // their traces cost, and the SMs do not get equal shares of the memory: with items dealt out in advance the slowest CTA took 4 %
  // longer than the average at eight slices, 10 % with slow decays.)
  struct Walk { int item, h, b, t0, rows; };
  auto place = [&](Walk& w) {                              // false: an item without work
    const int n = w.item / p.H % p.NC;
    w.h = w.item % p.H;
    w.b = w.item / (p.H * p.NC);
    w.t0 = n * CHUNK;
    w.rows = CHUNK;
    if (p.cmap == nullptr) return true;
    w.t0 = p.cmap[n];
    w.rows = p.cmap[p.NC + n];
    if (w.rows <= 0) return false;                         // unused tail of the chunk map
    if (w.t0 >= 0 && w.rows <= CHUNK && w.t0 + w.rows <= p.T) return true;
    atomicCAS(p.status, DEV_OK, DEV_BAD_CHUNK_MAP);        // never follow a bad map entry
    return false;
  };

  if (tid == 0) {
    for (int i = 0; i < NS; ++i) { mbar_init(&sm.full[i], 1); mbar_init(&sm.empty[i], 1); }
    mbar_init(&sm.tiles_full, 3); mbar_init(&sm.kq_full, 1); mbar_init(&sm.kq_free, 9);
    mbar_init(&sm.xt_full, 1); mbar_init(&sm.xt_free, 18);
    for (int i = 0; i < 2; ++i) { mbar_init(&sm.p_full[i], 1); mbar_init(&sm.p_free[i], 8); }
    mbar_init(&sm.t_full, 1); mbar_init(&sm.t_free, 4);
    mbar_init(&sm.g12, 1); mbar_init(&sm.g2read, 4); mbar_init(&sm.g34, 1); mbar_init(&sm.p_ready, 8); mbar_init(&sm.g5_full, 1);
    mbar_init(&sm.epi_free, 8); mbar_init(&sm.stage_free, 1); mbar_init(&sm.sums_free, 8); mbar_init(&sm.sg_done, 8);
    mbar_init(&sm.drained, 3);
    mbar_fence_init();
    sm.abort = sm.drain_abort = 0;
    for (int i = 0; i < 4; ++i) sm.place[i].item = -1;
  }
  if (warp_u == 16) { tmem_alloc(&sm.tmem_base, 512); tmem_relinquish(); }
  for (int i = tid; i < (2048 + 3584) / 16; i += GR_THREADS) reinterpret_cast<uint4*>(sm.zero)[i] = make_uint4(0, 0, 0, 0);   // and ident
  for (int i = tid; i < 128 * ES; i += GR_THREADS) sm.sums[i] = 0.f;
  if (tid < E * 4) sm.red[tid] = 0.f;
  __syncthreads();                                         // the zeroed operand before its diagonal
  if (tid < 16) *reinterpret_cast<uint16_t*>(sm.ident + (tid >> 3) * 1792 + (48 + tid) * 16 + (tid & 7) * 2) = 0x3F80;   // bf16 1.0
  fence_async_smem();
  tc_fence_before();
  __syncthreads();                                         // barriers, operands and the tensor-memory address are visible
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);
  const uint32_t tmem_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  WaitCtl ctl{&sm.abort, p.status}, drain{&sm.drain_abort, p.status};
  auto seen = [&](uint64_t* bar, uint32_t parity, int code) { return mbar_wait_parked_warp(bar, parity, ctl, code); };
  // Where a wait gives up, every wait of the CTA that is not met returns at once, and each role ends: the loading warp asks for nothing more
  // and writes no further item record; a role goes on to an item only when its wait for the record was met (the stream and the
  // chain by one verdict for all their warps), so that no address comes from a record that was not written; an item that was begun is
  // gone through to its end.  Loads, stores and products in flight are waited for at the end of the warps that issued them.

  // Barriers, with one completion per item unless noted (so that the parity to wait for is the item's count; a wait for "free" before
  // the first use passes at once):
  //   full / empty[stage]  TMA -> issuer, tensor core -> loads; one per ring entry.  Entries of an item: per slice h, (G), h, (G); dU, W, U
  //                        behind (or before) the first slice; at the end the value-block images.  (dU, W, U have
  //                        another reader than the rest and complete tiles_full instead of full: a waiter that is early by a whole
  //                        round of the ring could not tell the phases of a stage apart.)
  //   kq_full, kq_free     [K;Q] and A; free: eight stream warps (last row sum taken) and G5 complete
  //   xt_full, xt_free     [dW;dO] and the item's place; free: the item's last P_e complete, G2, and all sixteen stream and chain warps have seen
  //                        xt_full (with one or two slices nothing else would keep the next item's from completing before they look)
  //   p_full / p_free[b]   tiles P_e, the first slice's trace (T0_TILE) and the value-block sum through the double buffer; free: eight stream warps
  //   t_full, t_free       other traces; free: the four stream warps that read it
  //   g12                  G1, G2 complete;   g2read: the four query-row warps hold dPm': traces may take its place
  //   g34                  G3, then G4 (two per item);   p_ready: the operand of G5 is written;   g5_full: G5
  //   epi_free             the stream warps have read all tiles of the item: the next G1, G2 may be issued
  //   stage_free           dk, dq have left shared memory: P and dmp may be written
  //   sg_done              da, dc, dd of the item are complete;   sums_free: they have been taken and zeroed
  if (warp < 8) {
    // ============================================ stream ============================================
    regs_up<GR_STREAM_REGS>();
    const int wg = warp >> 2;                              // half of the key axis
    const int row = (warp & 3) * 32 + lane;
    const bool krow = row < 64;
    const int t = row & 63;
    const uint32_t krow_smem = smem_u32(sm.kq) + wg * 16384 + row * 128;   // this thread's K (Q) row, its 64 columns
    uint32_t tq = 0, traces = 0;                           // tiles, traces read so far
    for (uint32_t it = 0;; ++it) {
      const typename SM::Place& pl = sm.place[it & 3];
      const bool known = seen(&sm.xt_full, it & 1, DEV_TIMEOUT_LOAD);   // (by all lanes, which xt_free says)
      const bool go = one_verdict<4, 256>(known && pl.item >= 0, tid == 0, &sm.stream_go);
      // the previous item's dk, dq have left shared memory (waited for behind the verdict: before it, everybody would wait for them;
      // us, a backward of 4096 items, E2 with slow decays: 703 -> 689)
      if (it > 0 && warp_u == 3 && elect_one()) {
        bulk_wait_group_read();
        mbar_arrive(&sm.stage_free);
      }
      __syncwarp();
      if (!go) break;
      if (lane == 0) mbar_arrive(&sm.xt_free);
      // this row's gate factors a = k2 exp(gc) (c = scale q2 exp(gc)) as the masks kernel stored them, zero behind a document's end; each
      // asked for a slice ahead
      const float* gates = p.gc + static_cast<int64_t>(pl.item) * gate_item_floats(E) + (krow ? 64 : 192) * E + t * E;
      float gate_next = __ldg(gates);
      const uint32_t fmask = pl.traces;
      const bool live = t < pl.rows;
      float acc[64];                                       // this row's gate-weighted sum over the slices, key columns wg*64 .. +64
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = 0.f;
      mbar_wait_parked(&sm.kq_full, it & 1, ctl, DEV_TIMEOUT_LOAD);
#pragma unroll 1
      for (int e = 0; e < E; ++e) {
        const float gate = krow ? -gate_next : gate_next;
        const bool trace = (fmask >> e) & 1u;
        if (e + 1 < E) gate_next = __ldg(gates + e + 1);
        mbar_wait_parked(&sm.p_full[tq & 1], (tq >> 1) & 1, ctl, DEV_TIMEOUT_MMA);
        tc_fence_after();
        {
          float2 a01 = make_float2(0.f, 0.f), a23 = make_float2(0.f, 0.f);   // row sum against the K (Q) row, four chains
          const uint32_t src = tmem_row + (tq & 1) * 128 + wg * 64;
          float pv[2][8];
          tmem_ld<8>(src, pv[0]);
#pragma unroll
          for (int c = 0; c < 8; ++c) {                    // eight columns at a time, the next piece travelling while this one is used
            uint32_t kw[4];
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(kw[0]), "=r"(kw[1]), "=r"(kw[2]), "=r"(kw[3]) : "r"(krow_smem + ((c ^ (t & 7)) << 4)));
            tmem_wait_ld();
            if (c + 1 < 8) tmem_ld<8>(src + (c + 1) * 8, pv[(c + 1) & 1]);
            const float* pc = pv[c & 1];
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
              const uint32_t w0 = kw[j >> 1], w1 = kw[(j >> 1) + 1];
              a01 = __ffma2_rn(make_float2(bf16_lo(w0), bf16_hi(w0)), make_float2(pc[j], pc[j + 1]), a01);
              a23 = __ffma2_rn(make_float2(bf16_lo(w1), bf16_hi(w1)), make_float2(pc[j + 2], pc[j + 3]), a23);
              fma_pair(acc[c * 8 + j], acc[c * 8 + j + 1], gate, pc[j], pc[j + 1]);
              fma_pair(acc[c * 8 + j + 2], acc[c * 8 + j + 3], gate, pc[j + 2], pc[j + 3]);
            }
          }
          tc_fence_before();                               // orders the reads of P_e before the products that will overwrite it
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.p_free[tq & 1]);
          ++tq;
          // the two key halves add to a zeroed entry: the same bits in either order
          const float rowsum = (a01.x + a01.y) + (a23.x + a23.y);
          if (e == 0) mbar_wait_parked(&sm.sums_free, (it & 1) ^ 1, ctl, DEV_TIMEOUT_MMA);
          if (live) atomicAdd(&sm.sums[row * ES + e], krow ? -rowsum : rowsum);
        }
        const bool in_tiles = T0_TILE && e == 0;
        if (trace && (wg == 0 || in_tiles)) {                // <h_e, G_e> = trace(h_e G_e^T): this warp's 32 diagonal elements
          mbar_wait_parked(in_tiles ? &sm.p_full[tq & 1] : &sm.t_full, (in_tiles ? tq >> 1 : traces) & 1, ctl, DEV_TIMEOUT_MMA);
          tc_fence_after();
          float dv[32];
          if (wg == 0) {
            tmem_ld<32>(tmem_row + (in_tiles ? (tq & 1) * 128 : TM_T) + (warp & 3) * 32, dv);
            tmem_wait_ld();
          }
          auto take_diagonal = [&]() {
            if (wg != 0) return;
            float d = 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) d = (lane == j) ? dv[j] : d;
            for (int o2 = 16; o2 > 0; o2 >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o2);
            if (lane == 0) sm.red[e * 4 + (warp & 3)] = d;
          };
          // (up to two slices the tile is handed back behind the sum: E1 -4 %, E2 -11 % against before it; above, before it: behind, E8 +2 %)
          if constexpr (T0_TILE) take_diagonal();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(in_tiles ? &sm.p_free[tq & 1] : &sm.t_free);
          if constexpr (!T0_TILE) take_diagonal();
          if (in_tiles) ++tq; else ++traces;
        }
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sm.kq_free);
        mbar_arrive(&sm.sg_done);
      }
      // ---- dk, dq: state part (the slices' sum + the value-block images, rounded) + G5 ----
      mbar_wait_parked(&sm.p_full[tq & 1], (tq >> 1) & 1, ctl, DEV_TIMEOUT_MMA);
      tc_fence_after();
      if (krow) {                                          // (the same for a whole warp)
        const uint32_t src = tmem_row + (tq & 1) * 128 + wg * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float blk[16];
          tmem_ld<16>(src + c * 16, blk);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c * 16 + j] += blk[j];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.p_free[tq & 1]);
      ++tq;
      mbar_wait_parked(&sm.g5_full, it & 1, ctl, DEV_TIMEOUT_MMA);
      tc_fence_after();
      const bool whole = pl.rows == CHUNK;
      // A whole chunk leaves by TMA: dk from the place of P, dq from that of dmp, a 64 x 64 tile per column half
      const uint32_t stage = smem_u32(krow ? sm.p5 : sm.dmp) + wg * 8192 + t * 128;
      __nv_bfloat16* dst = (krow ? p.dk : p.dq) + ((static_cast<int64_t>(pl.b) * p.TS + pl.t0 + t) * p.H + pl.h) * HEAD + wg * 64;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float g5[16];
        tmem_ld<16>(tmem_row + TM_G5 + wg * 64 + c * 16, g5);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j += 8) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const float* a = acc + c * 16 + j + i;
            w[i >> 1] = pack_bf16(g5[j + i] + (live ? round_bf16(a[0]) : 0.f), g5[j + i + 1] + (live ? round_bf16(a[1]) : 0.f));
          }
          if (whole) st_shared_v4(stage + (((2 * c + (j >> 3)) ^ (t & 7)) << 4), w[0], w[1], w[2], w[3]);
          else if (live) *reinterpret_cast<uint4*>(dst + c * 16 + j) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.epi_free);
      asm volatile("bar.sync 4, 256;" ::: "memory");
      if (whole && warp_u == 3 && elect_one()) {
        tma_store_4d(&map_dk, sm.p5, 0, pl.h, pl.t0, pl.b);
        tma_store_4d(&map_dk, sm.p5 + 8192, 64, pl.h, pl.t0, pl.b);
        tma_store_4d(&map_dq, sm.dmp, 0, pl.h, pl.t0, pl.b);
        tma_store_4d(&map_dq, sm.dmp + 8192, 64, pl.h, pl.t0, pl.b);
        bulk_commit_group();
      }
      __syncwarp();
    }
    if (warp_u == 3 && elect_one()) bulk_wait_group();
    __syncwarp();
  } else if (warp < 16) {
    // ============================================ chain ============================================
    regs_up<GR_CHAIN_REGS>();
    const int mw = warp_u - 8, mt = tid - 256;
    const int qh = mw >> 2;                                // column quarters 2 qh, 2 qh + 1
    const int r = (mw & 3) * 32 + lane;                    // tensor-memory lane = matrix row
    const bool krow = (mw & 3) < 2;
    const int t = r & 63;
    const int warp_tmin = (mw & 1) ? 32 : 0, warp_tmax = warp_tmin + 31;   // rows of this warp
    const int tb = t >> 4;                                 // this row's 16-row block
    const uint32_t p5 = smem_u32(sm.p5);
    float* dmp = reinterpret_cast<float*>(sm.dmp);
    float* dm = sm.u.dm;
    constexpr int GATE_ITERS = (64 * E + 255) / 256;
    auto chain_all = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    auto chain_half = [&]() {                              // the key-row warps, or the query-row warps
      if (krow) asm volatile("bar.sync 2, 128;" ::: "memory"); else asm volatile("bar.sync 3, 128;" ::: "memory");
    };
    auto zero_piece = [&](uint32_t rowbase, int rr, int piece) { st_shared_v4(rowbase + ((piece ^ (rr & 7)) << 4), 0u, 0u, 0u, 0u); };
    // All global values of an item are requested in one batch, from clamped (always valid) addresses, and masked when they are used.
    float gc_in[GATE_ITERS], k2_in[GATE_ITERS], q2_in[GATE_ITERS], beta_in;
    auto request_gates = [&](const typename SM::Place& w) {
      const int64_t tok = static_cast<int64_t>(w.b) * p.TS + w.t0;
      beta_in = __ldg(p.beta + (tok + min(mt & 63, w.rows - 1)) * p.H + w.h);
#pragma unroll
      for (int i = 0; i < GATE_ITERS; ++i) {
        const int idx = min(mt + i * 256, 64 * E - 1);
        const int64_t off = ((tok + min(idx / E, w.rows - 1)) * p.H + w.h) * E + idx % E;
        gc_in[i] = __ldg(p.gc + static_cast<int64_t>(w.item) * gate_item_floats(E) + idx);
        k2_in[i] = __ldg(p.k2 + off);
        q2_in[i] = __ldg(p.q2 + off);
      }
    };
    // the wait for an item's record, its gates asked for and the verdict on it; at its return sm.chain_go says whether there is such an item
    auto next_item = [&](uint32_t it) {
      const typename SM::Place& w = sm.place[it & 3];
      const bool go = seen(&sm.xt_full, it & 1, DEV_TIMEOUT_LOAD) && w.item >= 0;
      if (lane == 0) mbar_arrive(&sm.xt_free);
      if (go) request_gates(w);
      one_verdict<1, 256>(go, mt == 0, &sm.chain_go);
    };
    next_item(0);
    for (uint32_t it = 0; *static_cast<volatile int*>(&sm.chain_go) != 0; ++it) {
      const typename SM::Place& pl = sm.place[it & 3];
      const int rows = pl.rows;
      // ---- gate tables ----
#pragma unroll
      for (int i = 0; i < GATE_ITERS; ++i) {
        const int idx = mt + i * 256;
        if (idx < 64 * E) {
          const int o = idx / E * ES + idx % E;
          const bool ok = idx / E < rows;
          sm.gc2[o] = gc_in[i] * LOG2E;
          sm.k2[o] = ok ? k2_in[i] : 0.f;
          sm.q2[o] = ok ? q2_in[i] : 0.f;
        }
      }
      if (mt < 64) sm.beta[mt] = mt < rows ? beta_in : 0.f;
      if (mt == 0) sm.steep = 0;
      chain_all();
      // Hd[s][e] = exp2(gc[r0(s)][e] - gc[s][e]) * k2[s][e], Xd[t][e] = q2[t][e] exp2(gc[t][e] - gc[r0(t)][e]), r0 the first row of the
      // 16-row block (see the matrix-gradient kernel).  The direct path costs eight warps 13 k cycles an item more at eight slices, so that
      // rows behind a document's end, whose gc rises by roundings, must not choose it: ms of a backward, 2000 documents of three tokens,
      // eight slices, eight heads, with those rows 8.84, without 6.58.
#pragma unroll
      for (int i = 0; i < GATE_ITERS; ++i) {
        const int idx = mt + i * 256;
        if (idx < 64 * E) {
          const int rr = idx / E, e = idx % E, o = rr * ES + e;
          const float up = sm.gc2[(rr & ~15) * ES + e] - sm.gc2[o];
          if (rr < rows && (!(up <= 100.f) || up < 0.f || (rr > 0 && sm.gc2[o] > sm.gc2[o - ES]))) sm.steep = 1;
          sm.hkv[idx] = mexp2(up) * sm.k2[o];
          sm.qxv[idx] = sm.q2[o] * mexp2(-up);
          sm.kxv[idx] = sm.k2[o] * mexp2(sm.gc2[o] - sm.gc2[(rr & ~15) * ES + e]);
        }
      }
      chain_all();
      const bool fast = sm.steep == 0;                     // the same for the whole chain
      const float* gct = sm.gc2 + t * ES;
      GateVec<E> mine;                                     // query rows: c1; key rows: r2 (summed over this thread's quarters)
      mine.clear();
      float brow = 0.f;
      mbar_wait_parked(&sm.kq_full, it & 1, ctl, DEV_TIMEOUT_LOAD);   // (the A image is read by threads)
      mbar_wait_parked(&sm.g12, it & 1, ctl, DEV_TIMEOUT_MMA);
      tc_fence_after();
      mbar_wait_parked(&sm.stage_free, (it & 1) ^ 1, ctl, DEV_TIMEOUT_MMA);   // dk, dq of the previous item have left the places of P and dmp

      if (!krow) {
        // ---- query rows: X -> P (rows 64..127), dmp, r1 ----
        const float alive = (t < rows) ? 1.f : 0.f;
        const uint32_t prow = p5 + r * 128;
        // dPm' moves into the places of dmp first: traces want its tensor memory
        if (32 * qh <= warp_tmax) {
          float g[32];
          tmem_ld<32>(tmem_row + TM_DPM + 32 * qh, g);
          tmem_wait_ld();
#pragma unroll
          for (int qi = 0; qi < 2; ++qi) {
            if (2 * qh + qi > tb) continue;
            float4* dst = reinterpret_cast<float4*>(dmp + tri_block(tb, 2 * qh + qi) + (t & 15) * 20);
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[j] = make_float4(g[16 * qi + 4 * j], g[16 * qi + 4 * j + 1], g[16 * qi + 4 * j + 2], g[16 * qi + 4 * j + 3]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.g2read);
        GateVec<E> r1v;
        r1v.clear();
        if (32 * qh > warp_tmax) {                         // all columns behind the diagonal
#pragma unroll
          for (int j = 0; j < 4; ++j) zero_piece(prow, r, 4 * qh + j);
        } else {
#pragma unroll 1
          for (int qi = 0; qi < 2; ++qi) {
            const int q = 2 * qh + qi, s0 = 16 * q;
            GateVec<E> G, accr;
            G.clear(); accr.clear();
            if (fast) {
#pragma unroll
              for (int e = 0; e < E; ++e)                  // (rows above the block are masked below)
                G.set(e, sm.q2[t * ES + e] * mexp2(fminf(gct[e] - sm.gc2[s0 * ES + e], 0.f)));
            }
#pragma unroll 1
            for (int jb = 0; jb < 2; ++jb) {
              const int sb = s0 + 8 * jb;
              float pr[8], gr[8], x[8], d[8];
              tmem_ld<8>(tmem_row + TM_G1 + sb, pr);
              // (rows above the block have no entries, and none of its columns: they are masked)
              float4* mat = reinterpret_cast<float4*>(dmp + tri_block(tb, min(q, tb)) + (t & 15) * 20 + 8 * jb);
              *reinterpret_cast<float4*>(gr) = mat[0];
              *reinterpret_cast<float4*>(gr + 4) = mat[1];
              if (fast) {
                tmem_wait_ld();
                slice_columns<E>(G, accr, sm.hkv + sb * E, [&](int j, float mp) {
                  const float in = (sb + j <= t) ? p.scale * gr[j] : 0.f;
                  x[j] = in * mp;
                  return d[j] = alive * in * pr[j];
                });
              } else {
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const int s = sb + j;
                  x[j] = d[j] = 0.f;
                  if (s <= t) {
                    float mp = 0.f;
                    for (int e = 0; e < E; ++e) mp = fmaf(sm.q2[t * ES + e], mexp2(gct[e] - sm.gc2[s * ES + e]) * sm.k2[s * ES + e], mp);
                    x[j] = p.scale * mp * gr[j];
                    d[j] = alive * p.scale * pr[j] * gr[j];
#pragma unroll
                    for (int e = 0; e < E; ++e)
                      accr.set(e, fmaf(d[j], mexp2(gct[e] - sm.gc2[s * ES + e]) * sm.k2[s * ES + e], accr.get(e)));
                  }
                }
              }
              st_shared_v4(prow + (((2 * q + jb) ^ (r & 7)) << 4), pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
              if (q <= tb) {
                mat[0] = make_float4(d[0], d[1], d[2], d[3]);
                mat[1] = make_float4(d[4], d[5], d[6], d[7]);
              }
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
              const float f = fast ? mexp2(fminf(gct[e] - sm.gc2[s0 * ES + e], 0.f)) : 1.f;
              r1v.set(e, r1v.get(e) + __fmul_rn(f, accr.get(e)));
            }
          }
        }
        if (qh == 1) {
#pragma unroll
          for (int e = 0; e < E; ++e) sm.r1[t * ES + e] = r1v.get(e);
        }
        chain_half();                                      // dmp complete
        if (qh == 0) {
#pragma unroll
          for (int e = 0; e < E; ++e) sm.r1[t * ES + e] = r1v.get(e) + sm.r1[t * ES + e];
        }
        // ---- c1[s, e] = sum over t' of dmp[t', s] exp(gc[t'] - gc[s]) q2[t', e], s = this thread's row, t' in its quarters ----
#pragma unroll 1
        for (int qi = 0; qi < 2; ++qi) {
          const int q = 2 * qh + qi, s0 = 16 * q;
          if (s0 + 15 < warp_tmin) continue;
          GateVec<E> c1v;
          c1v.clear();
          const float* col = dmp + tri_block(q, min(tb, q)) + (t & 15);
          if (fast) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float dv = tb <= q ? col[j * 20] : 0.f;
              GateVec<E> qx;
              qx.load(sm.qxv + (s0 + j) * E);
              c1v.add_scaled(dv, qx);
            }
            if (s0 + 15 >= t) {
#pragma unroll
              for (int e = 0; e < E; ++e) c1v.set(e, __fmul_rn(c1v.get(e), mexp2(sm.gc2[s0 * ES + e] - gct[e])));
            }
          } else {
            for (int tt = max(t, s0); tt < s0 + 16; ++tt) {
              const float dv = col[(tt - s0) * 20];
#pragma unroll
              for (int e = 0; e < E; ++e)
                c1v.set(e, fmaf(dv * sm.q2[tt * ES + e], mexp2(sm.gc2[tt * ES + e] - gct[e]), c1v.get(e)));
            }
          }
#pragma unroll
          for (int e = 0; e < E; ++e) mine.set(e, mine.get(e) + c1v.get(e));
        }
        if (qh == 1) {
#pragma unroll
          for (int e = 0; e < E; ++e) sm.c1[t * ES + e] = mine.get(e);
        }
      } else {
        // ---- key rows: dA = dA' diag(beta) -> operand image; column sums of dA' * A ----
        const uint32_t arow = smem_u32(sm.ap) + (t >> 3) * 128 + (t & 7) * 16, dyrow = smem_u32(sm.u.day) + (t >> 3) * 128 + (t & 7) * 16;
#pragma unroll 1
        for (int qi = 0; qi < 2; ++qi) {
          const int q = 2 * qh + qi, s0 = 16 * q;
          float gr[16], prod[16];
          tmem_ld<16>(tmem_row + TM_DA + s0, gr);
          tmem_wait_ld();
#pragma unroll
          for (int jb = 0; jb < 2; ++jb) {
            uint32_t aw[4];
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(aw[0]), "=r"(aw[1]), "=r"(aw[2]), "=r"(aw[3]) : "r"(arow + (2 * q + jb) * 1024));
            const float4 b0 = *reinterpret_cast<const float4*>(sm.beta + s0 + jb * 8), b1 = *reinterpret_cast<const float4*>(sm.beta + s0 + jb * 8 + 4);
            const float bs[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            float dav[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const int j = jb * 8 + c;
              prod[j] = __fmul_rn(gr[j], (c & 1) ? bf16_hi(aw[c >> 1]) : bf16_lo(aw[c >> 1]));
              dav[c] = gr[j] * bs[c];
            }
            st_shared_v4(dyrow + (2 * q + jb) * 1024, pack_bf16(dav[0], dav[1]), pack_bf16(dav[2], dav[3]), pack_bf16(dav[4], dav[5]), pack_bf16(dav[6], dav[7]));
          }
          const float col = warp_sums16(prod, lane);
          if (!(lane & 1)) sm.bcolp[mw & 1][s0 + (lane >> 1)] = col;
        }
        fence_async_smem();
        tc_fence_before();
        chain_half();
        // ---- G3: Y = A^T dA ----
        if (mw == 0 && elect_one()) {
          tc_fence_after();
          const uint64_t da = make_desc(smem_u32(sm.ap), 128, 1024, LAYOUT_PLAIN);       // A^T, MN-major (rows past 63: don't care)
          const uint64_t db = make_desc(smem_u32(sm.u.day), 128, 1024, LAYOUT_PLAIN);    // dA (K = t, N = s), MN-major
          constexpr uint32_t idesc = make_idesc(128, 64, 1, 1);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_bf16(tmem + TM_Y, desc_advance(da, kk * 256), desc_advance(db, kk * 256), idesc, kk > 0);
          umma_commit(&sm.g34);
        }
        __syncwarp();                                      // the other lanes must not run ahead into a spin wait
        mbar_wait_parked(&sm.g34, 0, ctl, DEV_TIMEOUT_MMA);
        tc_fence_after();
        {
          float yr[32];
          tmem_ld<32>(tmem_row + TM_Y + 32 * qh, yr);
          tmem_wait_ld();
#pragma unroll
          for (int jb = 0; jb < 4; ++jb)
            st_shared_v4(dyrow + (4 * qh + jb) * 1024, pack_bf16(yr[jb * 8], yr[jb * 8 + 1]), pack_bf16(yr[jb * 8 + 2], yr[jb * 8 + 3]),
                         pack_bf16(yr[jb * 8 + 4], yr[jb * 8 + 5]), pack_bf16(yr[jb * 8 + 6], yr[jb * 8 + 7]));
        }
        fence_async_smem();
        tc_fence_before();
        chain_half();
        // ---- G4: dp = Y A^T ----
        if (mw == 0 && elect_one()) {
          tc_fence_after();
          const uint64_t da = make_desc(smem_u32(sm.u.day), 1024, 128, LAYOUT_PLAIN);    // Y, K-major
          const uint64_t db = make_desc(smem_u32(sm.ap), 1024, 128, LAYOUT_PLAIN);       // B[k][j] = A[j][k]: A rows as N, K-major
          constexpr uint32_t idesc = make_idesc(128, 64, 0, 0);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_bf16(tmem + TM_Y, desc_advance(da, kk * 2048), desc_advance(db, kk * 2048), idesc, kk > 0);
          umma_commit(&sm.g34);
        }
        __syncwarp();
        mbar_wait_parked(&sm.g34, 1, ctl, DEV_TIMEOUT_MMA);
        tc_fence_after();
        // ---- dL, dPkk -> P (rows 0..63), dm, r2, dbeta_row ----
        const uint32_t prow = p5 + t * 128;
        const float bt = sm.beta[t];
        if (32 * qh > warp_tmax) {
#pragma unroll
          for (int j = 0; j < 4; ++j) zero_piece(prow, t, 4 * qh + j);
        } else {
#pragma unroll 1
          for (int qi = 0; qi < 2; ++qi) {
            const int q = 2 * qh + qi, s0 = 16 * q;
            GateVec<E> G, accr;
            G.clear(); accr.clear();
            float bq = 0.f;
            if (fast) {
#pragma unroll
              for (int e = 0; e < E; ++e) G.set(e, sm.k2[t * ES + e] * mexp2(fminf(gct[e] - sm.gc2[s0 * ES + e], 0.f)));
            }
#pragma unroll 1
            for (int jb = 0; jb < 2; ++jb) {
              const int sb = s0 + 8 * jb;
              float pr[8], dpr[8], x[8], d[8];
              tmem_ld<8>(tmem_row + TM_G1 + sb, pr);
              tmem_ld<8>(tmem_row + TM_Y + sb, dpr);
              if (fast) {
                tmem_wait_ld();
                slice_columns<E>(G, accr, sm.hkv + sb * E, [&](int j, float m) {
                  const float dl = (sb + j < t) ? -dpr[j] : 0.f;
                  bq = fmaf(dl * pr[j], m, bq);
                  x[j] = bt * dl * m;                      // zero on and above the diagonal
                  return d[j] = bt * dl * pr[j];
                });
              } else {
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const int s = sb + j;
                  x[j] = d[j] = 0.f;
                  if (s < t) {
                    float m = 0.f;
                    for (int e = 0; e < E; ++e) m = fmaf(sm.k2[t * ES + e], mexp2(gct[e] - sm.gc2[s * ES + e]) * sm.k2[s * ES + e], m);
                    const float dl = -dpr[j];
                    bq = fmaf(dl * pr[j], m, bq);
                    d[j] = bt * dl * pr[j];
                    x[j] = bt * dl * m;
#pragma unroll
                    for (int e = 0; e < E; ++e)
                      accr.set(e, fmaf(d[j], mexp2(gct[e] - sm.gc2[s * ES + e]) * sm.k2[s * ES + e], accr.get(e)));
                  }
                }
              }
              st_shared_v4(prow + (((2 * q + jb) ^ (t & 7)) << 4), pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
              if (q <= tb) {
                float4* dst = reinterpret_cast<float4*>(dm + tri_block(tb, q) + (t & 15) * 20 + 8 * jb);
                dst[0] = make_float4(d[0], d[1], d[2], d[3]);
                dst[1] = make_float4(d[4], d[5], d[6], d[7]);
              }
            }
            brow += bq;
#pragma unroll
            for (int e = 0; e < E; ++e) {
              const float f = fast ? mexp2(fminf(gct[e] - sm.gc2[s0 * ES + e], 0.f)) : 1.f;
              mine.set(e, mine.get(e) + __fmul_rn(f, accr.get(e)));
            }
          }
        }
        if (qh == 1) {
#pragma unroll
          for (int e = 0; e < E; ++e) sm.r2[t * ES + e] = mine.get(e);
        }
        sm.browp[qh][t] = brow;
      }
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.p_ready);             // G5 may be issued
      chain_all();
      // the other halves of c1 and r2
      if (qh == 0) {
        float* tab = krow ? sm.r2 : sm.c1;
#pragma unroll
        for (int e = 0; e < E; ++e) tab[t * ES + e] = mine.get(e) + tab[t * ES + e];
      }
      // dr and the next item's gates: asked for here, used behind the column sums
      constexpr int NV_MAX = E <= 8 ? 4 : 8;
      float dr_in[GATE_ITERS][NV_MAX];
      auto request_dr = [&]() {
#pragma unroll
        for (int i = 0; i < GATE_ITERS; ++i)
#pragma unroll
          for (int v = 0; v < NV_MAX; ++v)
            dr_in[i][v] = __ldg(p.dr + (static_cast<int64_t>(pl.item) * NV_MAX + v) * (64 * E) + min(mt + i * 256, 64 * E - 1));
      };
      if (E <= 4) request_dr();                            // (above four slices their registers are wanted by the column sums)
      // ---- c2[s, e] = sum over t' > s of dm[t', s] exp(gc[t'] - gc[s]) k2[t', e]: row s = t, the t' of quarters 2 qh and 2 qh + 1, each
      //      in two sums of eight; the key-row thread takes half of the slices, the query-row thread the other ----
      {
        constexpr int EH = E > 1 ? E / 2 : 1;
        const int eo = krow ? 0 : E / 2;
        GateVec<EH> c2v;
        c2v.clear();
        if (E > 1 || krow) {
#pragma unroll 1
          for (int qi = 0; qi < 2; ++qi) {
            const int q = 2 * qh + qi, s0 = 16 * q;
            if (s0 + 15 <= warp_tmin) continue;            // (dm is zero on and above the diagonal)
            const float* col = dm + tri_block(q, min(tb, q)) + (t & 15);
            GateVec<EH> part[2];
            part[0].clear(); part[1].clear();
            if (fast) {
#pragma unroll
              for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int j = 8 * hh; j < 8 * hh + 8; ++j) {
                  const float dv = tb <= q ? col[j * 20] : 0.f;
                  GateVec<EH> kx;
                  kx.load(sm.kxv + (s0 + j) * E + eo);
                  part[hh].add_scaled(dv, kx);
                }
              if (s0 + 15 > t) {
#pragma unroll
                for (int e = 0; e < EH; ++e) {
                  const float f = mexp2(sm.gc2[s0 * ES + eo + e] - gct[eo + e]);
                  part[0].set(e, __fmul_rn(part[0].get(e), f));
                  part[1].set(e, __fmul_rn(part[1].get(e), f));
                }
              }
            } else {
#pragma unroll
              for (int hh = 0; hh < 2; ++hh)
                for (int tt = max(t + 1, s0 + 8 * hh); tt < s0 + 8 * hh + 8; ++tt) {
                  const float dv = col[(tt - s0) * 20];
#pragma unroll
                  for (int e = 0; e < EH; ++e)
                    part[hh].set(e, fmaf(dv * sm.k2[tt * ES + eo + e], mexp2(sm.gc2[tt * ES + eo + e] - gct[eo + e]), part[hh].get(e)));
                }
            }
#pragma unroll
            for (int e = 0; e < EH; ++e) c2v.set(e, c2v.get(e) + (part[0].get(e) + part[1].get(e)));
          }
          // quarters 0 + 1 in c2, quarters 2 + 3 in the place of the query decay table
#pragma unroll
          for (int e = 0; e < EH; ++e) {
            if (qh == 0) sm.c2[t * ES + eo + e] = c2v.get(e);
            else sm.qxv[(eo + e) * 64 + t] = c2v.get(e);
          }
        }
      }
      if (E > 4) request_dr();
      mbar_wait_parked(&sm.sg_done, it & 1, ctl, DEV_TIMEOUT_MMA);
      next_item(it + 1);
      // ---- gate gradients: one thread per (row, gate column) ----
      const int64_t tok = static_cast<int64_t>(pl.b) * p.TS + pl.t0;
#pragma unroll
      for (int i = 0; i < GATE_ITERS; ++i) {
        const int idx = mt + i * 256;
        if (idx < 64 * E) {
          const int rr = idx / E, e = idx % E, o = rr * ES + e;
          float drv = 0.f;                                 // summed over the value blocks in index order
#pragma unroll
          for (int v = 0; v < NV_MAX; ++v) drv += dr_in[i][v];
          const GateGrads gg = gate_gradients(sm.gc2[o], sm.gc2[63 * ES + e], sm.k2[o], sm.q2[o], p.scale, sm.sums[o], sm.sums[64 * ES + o], drv,
                                              sm.r1[o], sm.c1[o], sm.r2[o], sm.c2[o] + sm.qxv[e * 64 + rr]);
          if (rr < rows) {
            const int64_t off = ((tok + rr) * p.H + pl.h) * E + e;
            p.dk2[off] = gg.dk2;
            p.dq2[off] = gg.dq2;
          }
          sm.r1[o] = gg.dgc;
          sm.c1[o] = gg.drr;
          sm.sums[o] = sm.sums[64 * ES + o] = 0.f;         // the next item's sums start here
        }
      }
      if (mt < 64 && mt < rows) p.dbeta[(tok + mt) * p.H + pl.h] = (sm.bcolp[0][mt] + sm.bcolp[1][mt]) + (sm.browp[0][mt] + sm.browp[1][mt]);
      chain_all();
      for (int e = mw; e < E; e += 8) {                    // one warp per gate column
        float v1 = sm.r1[(63 - lane) * ES + e], v0 = sm.r1[(31 - lane) * ES + e];
        const float dd = (sm.red[e * 4] + sm.red[e * 4 + 1]) + (sm.red[e * 4 + 2] + sm.red[e * 4 + 3]);
        __syncwarp();
        if (lane < 4) sm.red[e * 4 + lane] = 0.f;
        reverse_scan(v1, v0, sm.c1[lane * ES + e] + sm.c1[(lane + 32) * ES + e], dd, mexp2(sm.gc2[63 * ES + e]), lane);
        sm.r1[(63 - lane) * ES + e] = v1;                  // leaves by rows, below: a column would write four bytes of every sector
        sm.r1[(31 - lane) * ES + e] = v0;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.sums_free);
      chain_all();
#pragma unroll
      for (int i = 0; i < GATE_ITERS; ++i) {
        const int idx = mt + i * 256, rr = idx / E, e = idx % E;
        if (rr < rows) p.dg[((tok + rr) * p.H + pl.h) * E + e] = sm.r1[rr * ES + e];
      }
    }
    if (mw == 0 && elect_one()) umma_commit(&sm.drained);
    __syncwarp();
  } else {
    regs_down<GR_SERVICE_REGS>();
    int st = 0;                                            // ring stage
    uint32_t sph = 0;                                      // loads: parity of the round; stream products: per stage, parity of its next filling
    auto next_stage = [&]() { st = st + 1 == NS ? 0 : st + 1; };
    auto skip_stages = [&](int n) { st = (st + n) % NS; };
    auto take_stage = [&]() {
      mbar_wait_parked(&sm.full[st], (sph >> st) & 1u, ctl, DEV_TIMEOUT_LOAD);
      sph ^= 1u << st;
      tc_fence_after();
    };
    // the slice before which dU, W, U pass: the second one, or (TILES_EARLY) the first when it has a trace
    auto place_of_tiles = [&](uint32_t fmask) { return TILES_EARLY && (fmask & 1u) ? 0 : 1; };
    constexpr uint32_t id_128 = make_idesc(128, 128, 0, 0), id_64 = make_idesc(128, 64, 0, 0);
    const uint32_t ring = smem_u32(sm.ring[0]);
    const uint64_t dxt = make_desc(smem_u32(sm.xt), 16, 1024, LAYOUT_SW128);
    const uint64_t dring = make_desc(ring, 2048, 128, LAYOUT_PLAIN);           // images of a stage, K = v (h, G) or t (value blocks)
    const uint64_t dring_sw = make_desc(ring, 16, 1024, LAYOUT_SW128);         // tiles
    if (warp_u == 16) {
      // ============================================ products of the stream ============================================
      uint32_t tq = 0, traces = 0;                         // tiles, traces issued so far
      auto free_tile = [&]() { mbar_wait_parked(&sm.p_free[tq & 1], ((tq >> 1) & 1) ^ 1, ctl, DEV_TIMEOUT_MMA); };
      for (uint32_t it = 0;; ++it) {
        if (!seen(&sm.xt_full, it & 1, DEV_TIMEOUT_LOAD) || sm.place[it & 3].item < 0) break;
        const uint32_t fmask = __shfl_sync(0xffffffffu, sm.place[it & 3].traces, 0);
        const int tiles_at = place_of_tiles(fmask);
        bool first_trace = true;
#pragma unroll 1
        for (int e = 0; e < E; ++e) {
          const bool trace = (fmask >> e) & 1u;
          if (e == tiles_at) skip_stages(3);
          const bool in_tiles = T0_TILE && e == 0;
          free_tile();
#pragma unroll
          for (int vh = 0; vh < 2; ++vh) {
            take_stage();
            const int sh = st;
            const uint64_t dh = desc_advance(dring, sh * 16384);
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)               // P_e (+)= [dW;dO][:, 64 value columns] h_e[:, those columns]^T
                umma_bf16(tmem + (tq & 1) * 128, desc_advance(dxt, vh * 16384 + kk * 32), desc_advance(dh, kk * 4096), id_128, (vh > 0 || kk > 0) ? 1u : 0u);
              if (!trace) umma_commit(&sm.empty[sh]);
              if (vh == 1) umma_commit(&sm.p_full[tq & 1]);
            }
            __syncwarp();
            next_stage();
            if (trace) {                                   // h_e G_e^T over the same value columns
              const uint32_t tile = in_tiles ? ((tq + 1) & 1) * 128 : TM_T;
              if (vh == 0 && in_tiles) {
                ++tq;
                free_tile();
                --tq;
              } else if (vh == 0) {
                if (first_trace) mbar_wait_parked(&sm.g2read, it & 1, ctl, DEV_TIMEOUT_MMA);
                first_trace = false;
                mbar_wait_parked(&sm.t_free, (traces & 1) ^ 1, ctl, DEV_TIMEOUT_MMA);
              }
              take_stage();
              const uint64_t dg = desc_advance(dring, st * 16384);
              if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                  umma_bf16(tmem + tile, desc_advance(dh, kk * 4096), desc_advance(dg, kk * 4096), id_128, (vh > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&sm.empty[sh]);
                umma_commit(&sm.empty[st]);
                if (vh == 1) umma_commit(in_tiles ? &sm.p_full[(tq + 1) & 1] : &sm.t_full);
              }
              __syncwarp();
              next_stage();
            }
          }
          tq += trace && in_tiles ? 2 : 1;
          traces += trace && !in_tiles ? 1u : 0u;
        }
        if (elect_one()) umma_commit(&sm.xt_free);
        __syncwarp();
        if (tiles_at == E) skip_stages(3);
        // ---- value-block images of the G part of dK, added up, transposed: += [I;0] P_u^T ----
        if (first_trace) mbar_wait_parked(&sm.g2read, it & 1, ctl, DEV_TIMEOUT_MMA);   // (not behind them: a waiter may not miss a phase)
        free_tile();
        const uint64_t did = make_desc(smem_u32(sm.ident), 1792, 128, LAYOUT_PLAIN);          // K = k
#pragma unroll 1
        for (int u = 0; u < NVB; ++u) {
          take_stage();
          if (elect_one()) {
            const uint64_t dpk = desc_advance(dring, st * 16384);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem + (tq & 1) * 128, desc_advance(did, (3 - kk) * 256), desc_advance(dpk, kk * 4096), id_128, (u > 0 || kk > 0) ? 1u : 0u);
            umma_commit(&sm.empty[st]);
            if (u == NVB - 1) umma_commit(&sm.p_full[tq & 1]);
          }
          __syncwarp();
          next_stage();
        }
        ++tq;
      }
      if (elect_one()) umma_commit(&sm.drained);
      __syncwarp();
    } else if (warp_u == 18) {
      // ============================================ products of the chain ============================================
      uint32_t kq_loads = 0;
      for (uint32_t it = 0;; ++it) {
        const typename SM::Place& pl = sm.place[it & 3];
        if (!seen(&sm.xt_full, it & 1, DEV_TIMEOUT_LOAD) || pl.item < 0) break;
        const uint32_t fmask = __shfl_sync(0xffffffffu, pl.traces, 0);
        const int before = place_of_tiles(fmask) * (2 + 2 * (fmask & 1u)), entries = 2 * E + 2 * __popc(fmask) + 3 + NVB;
        if (!seen(&sm.kq_free, (it & 1) ^ 1, DEV_TIMEOUT_LOAD)) break;
        ++kq_loads;
        if (elect_one()) {
          mbar_expect_tx(&sm.kq_full, 32768 + 8192);
          tma_load_4d(sm.kq, &map_k, &sm.kq_full, 0, pl.h, pl.t0, pl.b);
          tma_load_4d(sm.kq + 8192, &map_q, &sm.kq_full, 0, pl.h, pl.t0, pl.b);
          tma_load_4d(sm.kq + 16384, &map_k, &sm.kq_full, 64, pl.h, pl.t0, pl.b);
          tma_load_4d(sm.kq + 24576, &map_q, &sm.kq_full, 64, pl.h, pl.t0, pl.b);
          tma_load_5d(sm.ap, &map_a, &sm.kq_full, 0, 0, 0, 0, pl.item);
        }
        __syncwarp();
        // ---- G1 = [K;Q] K^T;  G2: dA' = dU W^T (rows 0..63), dPm' = dO U^T (rows 64..127) ----
        mbar_wait_parked(&sm.epi_free, (it & 1) ^ 1, ctl, DEV_TIMEOUT_MMA);
        if (!seen(&sm.kq_full, it & 1, DEV_TIMEOUT_LOAD)) break;
        tc_fence_after();
        const uint64_t dkq = make_desc(smem_u32(sm.kq), 16, 1024, LAYOUT_SW128);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint32_t off = (kk >> 2) * 16384 + (kk & 3) * 32;
            umma_bf16(tmem + TM_G1, desc_advance(dkq, off), desc_advance(dkq, off), id_64, kk > 0);
          }
        }
        __syncwarp();
        skip_stages(before);
        const int su = st;                                 // dU: its rows 64..127 are whatever lies behind it, in rows nobody reads
        next_stage();
        mbar_wait_parked(&sm.tiles_full, it & 1, ctl, DEV_TIMEOUT_LOAD);
        tc_fence_after();
        if (elect_one()) {
          const uint64_t du = desc_advance(dring_sw, su * 16384), dw = desc_advance(dring_sw, st * 16384);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint32_t off = (kk >> 2) * 8192 + (kk & 3) * 32;
            umma_bf16(tmem + TM_DA, desc_advance(du, off), desc_advance(dw, off), id_64, kk > 0);
          }
          umma_commit(&sm.empty[su]);
          umma_commit(&sm.empty[st]);
        }
        __syncwarp();
        next_stage();
        if (elect_one()) {
          const uint64_t du = desc_advance(dring_sw, st * 16384);   // U
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_bf16(tmem + TM_DPM, desc_advance(dxt, (kk >> 2) * 16384 + (kk & 3) * 32), desc_advance(du, (kk >> 2) * 8192 + (kk & 3) * 32), id_64, kk > 0);
          umma_commit(&sm.g12);
          umma_commit(&sm.empty[st]);
          umma_commit(&sm.xt_free);
        }
        __syncwarp();
        next_stage();
        skip_stages(entries - 3 - before);
        // ---- G5: [dK;dQ] = (P' + P'^T) [K;Q] with P' = [P, 0]: one tile, read K-major and (with zeros for its missing columns) MN-major ----
        mbar_wait_parked(&sm.p_ready, it & 1, ctl, DEV_TIMEOUT_MMA);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t p5 = smem_u32(sm.p5);
          const uint64_t da = make_desc(p5, 16, 1024, LAYOUT_SW128);
          const uint64_t db = make_desc(smem_u32(sm.kq), 16384, 1024, LAYOUT_SW128);       // (K = token rows, N = d), MN-major
          constexpr uint32_t idesc = make_idesc(128, 128, 0, 1), idesc_t = make_idesc(128, 128, 1, 1);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_bf16(tmem + TM_G5, desc_advance(da, kk * 32), desc_advance(db, kk * 2048), idesc, kk > 0);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint64_t dat = make_desc(p5 + kk * 2048, smem_u32(sm.zero) - (p5 + kk * 2048), 1024, LAYOUT_SW128);
            umma_bf16(tmem + TM_G5, dat, desc_advance(db, kk * 2048), idesc_t, true);
          }
          umma_commit(&sm.g5_full);
          umma_commit(&sm.kq_free);
        }
        __syncwarp();
      }
      mbar_wait_parked(&sm.kq_full, (kq_loads & 1) ^ 1, drain, DEV_TIMEOUT_LOAD);
      if (elect_one()) umma_commit(&sm.drained);
      __syncwarp();
    } else if (warp_u == 17) {
      // ============================================ loads ============================================
      bool open = true;                                    // false: a wait gave up, nothing more is asked for (an entry could meet the last
                                                           // one of its stage still on its way)
      uint32_t tiles = 0, tile_stages = 0;                 // tiles asked for, and their parity per stage
      auto open_stage = [&]() { return open = open && seen(&sm.empty[st], sph ^ 1u, DEV_TIMEOUT_LOAD); };
      auto filled = [&]() { next_stage(); sph ^= st == 0 ? 1u : 0u; };
      auto entry = [&](const uint8_t* src) {               // 16 KB of global memory -> the next stage
        if (!open_stage()) return;
        if (elect_one()) {
          mbar_expect_tx(&sm.full[st], 16384);
          bulk_load(sm.ring[st], src, 16384, &sm.full[st]);
        }
        __syncwarp();
        filled();
      };
      auto tile_entry = [&](const CUtensorMap* map, int crow) {   // a 64 x 128 tile of a chunk-layout tensor
        if (!open_stage()) return;
        ++tiles;
        tile_stages ^= 1u << st;
        if (elect_one()) {
          mbar_expect_tx(&sm.tiles_full, 16384);
          tma_load_4d(sm.ring[st], map, &sm.tiles_full, 0, 0, crow, 0);
          tma_load_4d(sm.ring[st] + 8192, map, &sm.tiles_full, 64, 0, crow, 0);
        }
        __syncwarp();
        filled();
      };
      // chunk decays of an item, one lane per slice: they decide per slice whether a trace is taken
      auto load_gl = [&](const Walk& w) {
        return (lane < E && w.item < n_items) ? __ldg(p.gc + static_cast<int64_t>(w.item) * gate_item_floats(E) + 63 * E + lane) : 0.f;
      };
      auto draw = [&]() {                                  // the whole warp: the next item with work, or one past the last
        Walk w;
        do {
          int drawn = lane == 0 ? atomicAdd(p.next_item, 1) : 0;
          w.item = min(static_cast<int>(gridDim.x) + __shfl_sync(0xffffffffu, drawn, 0), n_items);
          if (w.item == n_items || place(w)) return w;
          // (start T, no rows: the unused tail of the chunk map, up to half of it with many documents, and the end of the items of its one row.
          // Drawn one by one, each a round trip to the counter and one to the map, ahead of the last item's loads, they cost 0.14 of the 4.80 ms of
          // a backward of 2048 documents of one chunk, 16 heads, one slice.)
        } while (w.rows > 0 || w.t0 != p.T);
        w.item = n_items;
        return w;
      };
      Walk cur;
      cur.item = blockIdx.x;
      if (!place(cur)) cur = draw();
      float my_gl = load_gl(cur);
      uint32_t it = 0;                                     // item records written
      for (;; ++it) {
        Walk nxt = cur;
        if (cur.item < n_items) nxt = draw();
        const float next_gl = load_gl(nxt);                // asked for a whole item ahead
        const uint32_t fmask = __ballot_sync(0xffffffffu, lane < E && my_gl * LOG2E >= DD_MIN_LOG2_DECAY);
        if (!open || !seen(&sm.xt_free, (it & 1) ^ 1, DEV_TIMEOUT_LOAD)) break;
        const bool end = cur.item >= n_items;
        if (elect_one()) {
          typename SM::Place& pl = sm.place[it & 3];
          pl.item = end ? -1 : cur.item;
          pl.h = cur.h; pl.b = cur.b; pl.t0 = cur.t0; pl.rows = cur.rows; pl.traces = fmask;
          if (end) {
            mbar_arrive(&sm.xt_full);
          } else {
            mbar_expect_tx(&sm.xt_full, 32768);
            tma_load_4d(sm.xt, &map_dv, &sm.xt_full, 0, cur.h, cur.t0, cur.b);
            tma_load_4d(sm.xt + 8192, &map_do, &sm.xt_full, 0, cur.h, cur.t0, cur.b);
            tma_load_4d(sm.xt + 16384, &map_dv, &sm.xt_full, 64, cur.h, cur.t0, cur.b);
            tma_load_4d(sm.xt + 24576, &map_do, &sm.xt_full, 64, cur.h, cur.t0, cur.b);
          }
        }
        __syncwarp();
        if (end) { ++it; break; }
        // what threads load themselves -> L2: dr of this item, the gates of the next (the tiles and images come without: pulling those
        // ahead made the kernel 10 to 20 % slower)
        for (int l = lane; l < NVB * 2 * E; l += 32) prefetch_l2(p.dr + static_cast<int64_t>(cur.item) * NVB * (64 * E) + l * 32);
        if (nxt.item < n_items) {
          const float* gates = p.gc + static_cast<int64_t>(nxt.item) * gate_item_floats(E);
          for (int l = lane; l < 6 * E; l += 32) prefetch_l2(gates + (l < 4 * E ? l : l + 2 * E) * 32);
          for (int r = lane; r < nxt.rows; r += 32) {
            const int64_t ro = (static_cast<int64_t>(nxt.b) * p.TS + nxt.t0 + r) * p.H + nxt.h;
            prefetch_l2(p.k2 + ro * E);
            prefetch_l2(p.q2 + ro * E);
            if (E > 8) { prefetch_l2(p.k2 + ro * E + 8); prefetch_l2(p.q2 + ro * E + 8); }
            prefetch_l2(p.beta + ro);
          }
        }
        __syncwarp();
        const int tiles_at = place_of_tiles(fmask);
        const int64_t item = cur.item;
        const int crow = cur.item * 64;
        const uint8_t* h_item = reinterpret_cast<const uint8_t*>(p.h) + item * (static_cast<int64_t>(E) * 32768);
        const uint8_t* g_item = reinterpret_cast<const uint8_t*>(p.ds) + item * (static_cast<int64_t>(E) * 32768);
        const uint8_t* blocks = reinterpret_cast<const uint8_t*>(p.dkg) + item * (static_cast<int64_t>(NVB) * 16384);
        // One place in the code asks for entries and one for tiles: five roles' loops share an SM's instruction caches, and what this warp
        // executes between a free stage and the load into it is waited for.  us, a call in each place -> one: 4096 items E4 303 -> 294, with
        // slow decays 471 -> 440; 8192 items E8 827 -> 811, 1298 -> 1205; 2048 items E12 342 -> 352, 526 -> 485, E16 416 -> 402, 621 -> 577.
#pragma unroll 1
        for (int e = 0; e <= E; ++e) {                     // slices; at E the value-block images
          if (e == tiles_at) {
#pragma unroll 1
            for (int i = 0; i < 3; ++i) tile_entry(i == 0 ? &map_du : i == 1 ? &map_w : &map_u, crow);
          }
          const bool trace = e < E && ((fmask >> e) & 1u);
          const uint8_t* src = e < E ? h_item + e * 32768 : blocks;
          const int pieces = e == E ? NVB : trace ? 4 : 2;
#pragma unroll 1
          for (int i = 0; i < pieces; ++i) entry(!trace ? src + i * 16384 : (i & 1 ? g_item + e * 32768 : src) + (i >> 1) * 16384);
        }
        cur = nxt;
        my_gl = next_gl;
      }
      // what was asked for has arrived: the last phase of each barrier
      for (; tiles % 3 != 0; ++tiles)                      // (a set cut short: the arrivals that are missing)
        if (elect_one()) mbar_arrive(&sm.tiles_full);
#pragma unroll 1
      for (int i = 0; i < NS + 2; ++i) {
        const uint32_t phases = i < NS ? sph ^ (i < st ? 1u : 0u) ^ (tile_stages >> i) : i == NS ? tiles / 3 : it;
        mbar_wait_parked(i < NS ? &sm.full[i] : i == NS ? &sm.tiles_full : &sm.xt_full, (phases & 1) ^ 1, drain, DEV_TIMEOUT_LOAD);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp_u == 16) {
    mbar_wait_parked(&sm.drained, 0, drain, DEV_TIMEOUT_MMA);
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace tgdn

using namespace tgdn;

template <int E>
static int launch_grads(const CUtensorMap* m, const GradsParams& p, cudaStream_t s) {
  const int smem = static_cast<int>(sizeof(GradsSmem<E>)) + 1024;
  static_assert(sizeof(GradsSmem<E>) + 1024 <= 232448, "shared memory budget of one CTA exceeded");
  static bool configured[64] = {};
  if (const int rc = tgdn_dynamic_smem(reinterpret_cast<const void*>(grads_kernel<E>), smem, configured)) return rc;
  const long long items = static_cast<long long>(p.B) * p.NC * p.H;
  const int sms = tgdn_sm_count();
  grads_kernel<E><<<static_cast<int>(items < sms ? items : sms), GR_THREADS, smem, s>>>(m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7], m[8], m[9], p);
  return tgdn_cuda_error(cudaGetLastError());
}

int tgdn_bwd_grads_rows(const void* q, const void* k, const void* dO, const void* dV, const void* dU, const void* W, const void* U,
                        const void* AP, const void* h, const void* ds, const void* dkg, const float* k2, const float* q2,
                        const float* beta, const float* gc, const float* dr, float scale, const int32_t* chunk_map, int B, int T, int H,
                        int E, int NC, int row_tokens, int* next_item, void* dq, void* dk, float* dk2, float* dq2, float* dg, float* dbeta, void* stream) {
  if (!next_item || !q || !k || !dO || !dV || !dU || !W || !U || !AP || !h || !ds || !dkg || !k2 || !q2 || !beta || !gc || !dr || !dq || !dk || !dk2 ||
      !dq2 || !dg || !dbeta)
    return TGDN_ERR_NULL;
  int rc = tgdn_check_core_shape(B, T, H, E, NC, chunk_map != nullptr, row_tokens);
  if (rc) return rc;
  if ((reinterpret_cast<uintptr_t>(AP) | reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(ds) | reinterpret_cast<uintptr_t>(dkg) |
       reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(gc) | reinterpret_cast<uintptr_t>(dr)) & 15)
    return TGDN_ERR_ALIGN;
  const long long crows = static_cast<long long>(B) * NC * H * 64;
  if (crows > 0x7fffffffLL) return TGDN_ERR_SHAPE;          // item indices are 32-bit in the kernel
  CUtensorMap m[10];
  const void* token[4] = {k, q, dV, dO};
  const void* chunk[3] = {dU, W, U};
  for (int i = 0; i < 4; ++i)
    if ((rc = tgdn_make_token_map(&m[i], token[i], B, T, H, 64, 64, 1, row_tokens))) return rc;
  // chunk-layout tensors are plain (rows, 128) matrices: one batch row, one head
  for (int i = 0; i < 3; ++i)
    if ((rc = tgdn_make_token_map(&m[4 + i], chunk[i], 1, static_cast<int>(crows), 1, 64, 64, 1))) return rc;
  if ((rc = tgdn_make_a_half_map(&m[7], AP, crows / 64))) return rc;
  if ((rc = tgdn_make_token_map(&m[8], dk, B, T, H, 64, 64, 1, row_tokens))) return rc;
  if ((rc = tgdn_make_token_map(&m[9], dq, B, T, H, 64, 64, 1, row_tokens))) return rc;
  GradsParams p{static_cast<const __nv_bfloat16*>(AP), static_cast<const __nv_bfloat16*>(h), static_cast<const __nv_bfloat16*>(ds),
                static_cast<const __nv_bfloat16*>(dkg), k2, q2, beta, gc, dr, next_item, static_cast<__nv_bfloat16*>(dq),
                static_cast<__nv_bfloat16*>(dk), dk2, dq2, dg, dbeta, chunk_map, B, T, H, NC, HEAD / tgdn_value_block(E), row_tokens, scale,
                tgdn_status_word()};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (E) {
    case 1: return launch_grads<1>(m, p, s);
    case 2: return launch_grads<2>(m, p, s);
    case 4: return launch_grads<4>(m, p, s);
    case 8: return launch_grads<8>(m, p, s);
    case 12: return launch_grads<12>(m, p, s);
    case 16: return launch_grads<16>(m, p, s);
    default: return TGDN_ERR_SHAPE;
  }
}
