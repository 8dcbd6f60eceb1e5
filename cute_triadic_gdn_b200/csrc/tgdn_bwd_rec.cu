// Reverse chunk recurrence of the Triadic GDN backward.
//
// One CTA owns one (sequence, head, block of VC value columns) and walks the chunks from last to first with
// G_e = dL/dS_e[:, value block] (f32) in registers.  Per chunk, with dO, U the chunk's rows of the value block:
//   (a) KG = [K;Q] G                tcgen05 M=128, N=E*VC, K=128   (rows 0..63 are used)
//       Y  = Pm^T dO                tcgen05 M=128 (64 used), N=VC, K=64
//       dU = sum_e r_e*KG_e + Y ;   dr_e = sum_v U*KG_e  (per value block, summed later)
//   (c) Z  = A^T dU                 tcgen05 M=128 (64 used), N=VC, K=64
//       dW = beta*Z = dV ;  X = [-a_e*dW ; c_e*dO]
//   (p) P  = G Xu^T                 tcgen05 M=128 (key rows d), N=64 (tokens), K=E*VC     Xu_e = r_e*U
//       the value block's share of  sum_e (r_e*U) G_e^T, the part of dK that contracts the gradient state over the
//       value axis; it leaves as a bf16 operand image (16 KB) and the gradient kernel adds the blocks up
//   (d) dG = [K^T | Q^T] X          tcgen05 M=128, N=E*VC, K=128
//       G_e <- d_e G_e + dG_e ; bf16 copy -> operand of the next (a)
//
// Because (p) runs here, where G lives, the gradient state itself never has to travel: the reference writes it to HBM at
// every chunk (32 KB x E per chunk and head) and reads it back in its state-gradient kernel.  The one other consumer of
// G_e outside this kernel is dd_e = <h_e, G_e>, the gradient of the chunk decay d_e = exp(gL_e), which enters the result
// only as d_e*dd_e: slices whose chunk decay is below 2^-24 contribute less than one part in 10^7 of <h_e, G_e> and are
// skipped there (dd_e = 0); G_e is stored (ds) only for the slices of chunks whose decay is above that threshold.
//
// (p) is off the dependent chain of the chunk: it is issued behind (a) as soon as its operand Xu is built, runs while the
// epilogue of (a) occupies the threads, and is read out of tensor memory while (d) runs.
//
// The gate factors (a, r, c per row and slice, d per slice) were formed by the masks kernel and arrive with one bulk copy
// per chunk; every thread reads those of its own row from shared memory.  The gradient state can be handed in (dL/dS after the last token) and out (before the first), so
// that sequences can be processed in segments (tgdn_bwd_recurrent_state).
//
// Replaces cute_triadic_gdn/kernels/sm100_joint_bwd_recurrent.py:59-533 (rec_kernel) and the (r*U) G^T product of
// cute_triadic_gdn/kernels/sm100_joint_state_grads.py:373-378.  The operand X and the bf16 image of G share one buffer because they
// are never live at the same time.
//
// What bounds it: the dependent chain of a chunk (three MMA -> load -> epilogue round trips) over a shared-memory path that the
// products' operand reads and the operand images fill to two thirds.  Reverse recurrence, us, one lockstep CTA of four warpgroups
// that looked the chunk up when it began -> this version: B2 T8192 H32 E8 1241 -> 1092; B1 T32768 packed H8 E12 1132 -> 997;
// H16 E16 2497 -> 2414; B4 T4096 H16 E4 394 -> 285, E2 318 -> 226, E1 299 -> 202 (the last three with 64 value columns per CTA, then one block).
// Every copy operation costs the warp that issues it some sixty cycles and the chain waits for its last warp, so the images of dO and U,
// the A half and dU move with one operation each, whatever their width (22 -> 9 a chunk at E = 8); with that and the two-wide f32
// multiply-adds: E8 1095 -> 1075, E16 2418 -> 2395, E4 291 -> 275, E2 229 -> 209, E1 204 -> 178 us.  (Pulling later chunks into L2 by
// prefetch instructions made it 3 to 8 % slower: the loads are a chunk ahead already.)
// dV of a whole chunk leaves as a tile up to eight slices: us, 8192 items E8 1031 -> 1023, 4096 items E4 270 -> 255, E2 205 -> 194, E1 177 -> 171.
// One value block per chain in the 64-column CTA, with sums of its own, instead of one block of 64 columns (whose results depended on
// the width that the call picked): E4 254 -> 256, E2 193 -> 206, E1 172 -> 188, and four images are added up behind it again instead
// of two (in the state-gradient kernel of that time 217 -> 247, 164 -> 182, 137 -> 154); four slices on narrow blocks (2048 items), the chains' P in turn: 188 -> 193.
// Who waits for a product parks (the other chain's epilogue wants the shared-memory path that polls would take); the loads of a chunk are
// polled, being there already as a rule: us, all waits polled -> E8 1014 -> 987, E12 968 -> 929, E16 1208 -> 1176 (4096 items each),
// E4 256 -> 247; with the loads parked too E12 977.  (One polling warp and a named barrier for the rest: E8 1133.)
#include "tgdn_common.cuh"
#include "tgdn_host.h"
#include "tgdn_kernels.h"

namespace tgdn {

// The CTA is two independent CHAINS of two warpgroups, each owning half of the value columns of every slice: own MMAs, own barriers,
// own named barrier.  While one chain's threads are in an epilogue the tensor core works for the other one.  (One lockstep CTA of
// four warpgroups took 9.5 k cycles per chunk at E = 8, of which its products were in flight for 4.6 k and its epilogues ran for
// the other 4.9 k, neither overlapping the other.)  The chains share the chunk's tiles (two-stage ring; the last chain to hand a
// stage back refills it) and, at one block per CTA, two sums over all value columns: P and dr, which both chains read out together
// (below).  One and two slices on narrow blocks are one chain of four warpgroups: their products are so short that two of everything
// costs more than the overlap gives.
// P leaves rounded to bf16 per VALUE BLOCK of 32 columns (16 above eight slices) and dr is summed per block, so the block is part of
// the results, and the CTA's width must not be: the 64-column CTA (VC = 64, up to four slices, chosen by the number of sequences) is
// two blocks, one per chain, each with its own P and dr, formed from the same products in the same order as in a CTA of one block.
// What a sequence gets then does not depend on what runs beside it.  (At four slices the narrow CTA's two chains add into one P in
// turn, chain 0 first, which is the order of the wide CTA's single chain.)
// NSG = 2 (twelve and sixteen slices) splits the SLICES of a chain's columns over its two warpgroups: a thread then holds eight
// value columns of half the slices instead of four columns of all of them, which keeps the 16-byte accesses; the sum over all
// slices (dU) is completed through shared memory.
template <int THREADS>
__device__ __forceinline__ void rec_chain_sync(int chain) {
  asm volatile("bar.sync %0, %1;" ::"r"(chain + 1), "n"(THREADS) : "memory");
}

template <int E, int VC, int NCH, int NSG = 1>
struct RecCfg {
  static constexpr int NWG = 4, STAGES = 2;
  static constexpr int CHAIN_THREADS = NWG / NCH * 128;
  static constexpr int THREADS = NWG * 128;
  static constexpr int NCOLS = E * VC;
  static constexpr int NCG = NWG / NSG;           // column groups
  static constexpr int CW = VC / NCG;             // value columns per thread
  static constexpr int EL = E / NSG;              // slices per thread
  static constexpr int TPC = EL * CW;             // state columns per thread
  static constexpr int CC = NCOLS / NCH;          // state columns per chain
  static constexpr int CV = VC / NCH;             // value columns per chain
  static constexpr bool OWN = VC == 64;           // every chain is a value block of its own
  static constexpr int VBW = OWN ? CV : VC;       // width of a value block
  static constexpr bool IN_TURN = E == 4 && !OWN; // chain 1 adds its share of P to chain 0's
  static constexpr bool CROSS = NCH > 1 && !OWN;  // the chains share the sums over the block's columns
  static constexpr int YW = CV < 16 ? 16 : CV;    // columns of Y and Z (the smallest N of an M=128 MMA is 16)
  static_assert(CC % 16 == 0 && CC <= 256 && CV % 8 == 0, "columns of a chain's products");
  static_assert((NCH == 1 && NSG == 1) || NCH == 2, "slice groups are the two warpgroups of a chain");
  static_assert(!OWN || (NCH == 2 && NSG == 1 && CV == 32), "a wide CTA is two blocks of 32 columns");
  static_assert(CW == 8 || CW == 16, "value columns per thread");
  static constexpr int ES = E | 1;
  static_assert(NWG % NSG == 0 && E % NSG == 0 && (NSG == 1 || EL % 2 == 0), "slice groups split the slices evenly");
  static constexpr int TMEM_NEED = NCOLS + NCH * (2 * YW + 64);    // KG/dG, Y, Z, P
  static constexpr int TMEM_COLS = TMEM_NEED <= 64 ? 64 : TMEM_NEED <= 128 ? 128 : TMEM_NEED <= 256 ? 256 : 512;
  static constexpr int KQ_BYTES = 32768;
  static constexpr int A_BYTES = 8192;            // image (i = t, j = s), SI = 128, SJ = 1024: the A half of [A; Pm A]
  static constexpr int PM_BYTES = 8192;
  static constexpr int GX_BYTES = NCOLS * 256;    // image (i = row 0..127, j = n'), SI = 128, SJ = 2048
  static constexpr int XU_BYTES = NCOLS * 128;    // image (i = t, j = n'), SI = 128, SJ = 1024
  static constexpr int DO_BYTES = VC * 128;       // image (i = t, j = v), SI = 128, SJ = 1024
  static constexpr int DOB = (DO_BYTES + 1023) & ~1023;
  static constexpr int DRP_FLOATS = NCG * 64 * ES + (NSG > 1 ? 64 * VC : 0);   // dr partials per column group; partial dU of the other slice group
  // the gate factors of a chunk as the masks kernel stored them: a, r, c as 64 dense rows of E floats each, then d
  static constexpr int GT_BYTES = gate_factor_bytes(E);
  static constexpr int GT_STRIDE = (GT_BYTES + 127) & ~127;
  static constexpr int GF_R = 64 * E, GF_C = 128 * E, GF_D = 192 * E;   // float offsets of r, c, d behind a
  static constexpr int LIMIT = 232448;
  // Shared memory of a layout with `nb` copies of Pm and A (the gate factors have one per stage)
  static constexpr int layout_bytes(int nb) {
    const int xu = XU_BYTES < 8192 ? 8192 : XU_BYTES;
    const int upto_dt = STAGES * KQ_BYTES + GX_BYTES + nb * (PM_BYTES + A_BYTES) + xu + 2 * STAGES * DOB + DRP_FLOATS * 4;
    const int off_gt = (upto_dt + NCH * 128 + 127) & ~127;
    return off_gt + STAGES * (GT_STRIDE + (nb == 1 ? 1024 : 0)) + 256 + 1024;
  }
  // Pm and A get a second copy too where that fits.  Where it does not (eight and sixteen slices) they are single and requested
  // LATE, each on a barrier of its own, when both chains are done with it: Pm after the first products of the chunk, A after (c).
  // (So it is at four slices on 64 columns.)
  // Half a chunk lies between that and the next use by the chain that is ahead.
  static constexpr bool LATE = layout_bytes(2) > LIMIT;
  static constexpr int NB = LATE ? 1 : 2;
  static_assert(layout_bytes(NB) <= LIMIT, "shared memory budget of one CTA exceeded");
  static constexpr int OFF_KQ = 0;
  static constexpr int OFF_GX = OFF_KQ + STAGES * KQ_BYTES;
  // the 128-row descriptors over the 64-row Pm and A images read up to 8 KB past them: Pm is followed by A, A by Xu
  static constexpr int OFF_PM = OFF_GX + GX_BYTES;
  static constexpr int OFF_A = OFF_PM + NB * PM_BYTES;
  static constexpr int OFF_XU = OFF_A + NB * A_BYTES;
  // per stage: the dO rows of the value block, which TMA writes straight into the operand image of Y, and the U rows,
  // which TMA writes into the place where the operand image of dU is built later (every thread reads its piece of U
  // before it overwrites that very piece with dU)
  static constexpr int OFF_DO = OFF_XU + (XU_BYTES < 8192 ? 8192 : XU_BYTES);
  static constexpr int OFF_DU = OFF_DO + STAGES * DOB;
  static constexpr int OFF_DRP = OFF_DU + STAGES * DOB;
  static constexpr int OFF_DT = OFF_DRP + DRP_FLOATS * 4;     // per chain: exp(gL) of this chunk and the store flags of the next, 2 x 16 words
  static constexpr int OFF_GT = (OFF_DT + NCH * 128 + 127) & ~127;
  // per stage: the beta rows of the chunk for the four heads h & ~3 .. (TMA when H is a multiple of 4).  With LATE: at eight and sixteen
  // slices, whose chunks are bound by the L1 data path: a load per thread of a row of its own costs 32 wavefronts a warp (us, loads -> tile:
  // 8192 items E8 1055 -> 1031, packed E16 2297 -> 2278); elsewhere one more copy a chunk costs what that gives or a little more
  // (E12 1004 -> 1019, E2 205 -> 210).
  static constexpr int BT_BYTES = LATE ? 1024 : 0;
  static constexpr int OFF_BT = OFF_GT + STAGES * GT_STRIDE;
  static constexpr int OFF_CTRL = OFF_BT + STAGES * BT_BYTES;
  static constexpr int SMEM_BYTES = OFF_CTRL + 256 + 1024;
};

struct RecCtrl {
  uint64_t bar_load[2];      // K/Q tiles, dO and U rows, gate factors of a stage (and Pm, A where they have two copies)
  uint64_t bar_pm, bar_a;    // late scheme: Pm, A of the chunk
  uint64_t bar_ad[2];        // per chain: its (a), then its (d)
  uint64_t bar_mma[2];       // per chain: (c)
  uint64_t bar_xu[2];        // per chain: its key-row warps have written the operand Xu of (p), one arrival per warp
  uint64_t bar_ex[2];        // per chain: its share of P is complete and its dr partials are written (four key-row warps and a commit)
  uint64_t bar_turn;         // P of chain 0 is complete: chain 1 may add to it
  uint64_t bar_done;         // every warp has read its part of P and dr: the next chunk's may be written
  uint32_t released[2], released_pm, released_a;   // chains that are done with a stage, Pm, A (count up forever; a multiple of the chains = all)
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(RecCtrl) <= 256, "control block");

template <int E, int VC, int NCH, int NSG, bool PACKED>
__global__ void __launch_bounds__(512, 1)
rec_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q,
           const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_u,
           const __grid_constant__ CUtensorMap map_du, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_beta, const __grid_constant__ CUtensorMap map_dv, RecParams p) {
  using C = RecCfg<E, VC, NCH, NSG>;
  constexpr int REC_THREADS = C::THREADS, NWG = C::NWG, CT = C::CHAIN_THREADS, CC = C::CC, CV = C::CV, YW = C::YW;
  constexpr int NCOLS = C::NCOLS, CW = C::CW, TPC = C::TPC, ES = C::ES, NCG = C::NCG, EL = C::EL;
  constexpr int NV = HEAD / VC, NVB = HEAD / C::VBW;   // CTAs per head, value blocks per head
  constexpr bool CROSS = C::CROSS;
  constexpr bool DV_TILE = NSG == 1;                // (at twelve and sixteen slices the tile costs what it saves)
  constexpr bool TWO_WIDE = TPC * CW < 1024;        // the two-wide multiply-adds of (a) need register pairs: sixteen columns of four slices spill
                                                    // (and on packed rows they spill 36 bytes without)
  constexpr float LOG2E = 1.4426950408889634f;   // the decay threshold below is in the log2 domain
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* drp = reinterpret_cast<float*>(smem + C::OFF_DRP);
  float* dured = drp + NCG * 64 * ES;                                 // NSG > 1: [64 rows][VC] partial dU
  RecCtrl& ctrl = *reinterpret_cast<RecCtrl*>(smem + C::OFF_CTRL);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wg = warp >> 2;
  const int chain = wg / (NWG / NCH);
  const int cgp = NSG == 1 ? wg : chain;            // column group: value columns cgp*CW .. of the block
  const int sgp = NSG == 1 ? 0 : wg & 1;            // slice group: slices sgp*EL ..
  float* dtab = reinterpret_cast<float*>(smem + C::OFF_DT + chain * 128);        // [16] exp(gL_e)
  int* ftab = reinterpret_cast<int*>(smem + C::OFF_DT + chain * 128) + 16;       // [16] store G_e of the next chunk?
  const int e0 = sgp * EL;
  const int row = (warp & 3) * 32 + lane;
  const bool krow = row < 64;
  const int t = row & 63;

  const int vb = blockIdx.x % NV, h = (blockIdx.x / NV) % p.H, seq_rank = blockIdx.x / (NV * p.H);
  if (blockIdx.x == 0 && tid == 0 && p.zeroed != nullptr) *p.zeroed = 0;   // (before any early return)
  int b = seq_rank, first = 0, count = p.NC, seq = seq_rank;
  if constexpr (PACKED) {
    const int doc = p.cmap[2 * p.NC + seq_rank];
    if (doc < 0 || doc >= p.n_seq) return;
    b = 0;
    seq = doc;
    first = p.offsets[doc];
    count = p.offsets[doc + 1] - first;
    if (first < 0 || count <= 0 || first + count > p.NC) return;
  }

  if (tid == 0) {
    mbar_init(&ctrl.bar_load[0], 1);
    mbar_init(&ctrl.bar_load[1], 1);
    mbar_init(&ctrl.bar_pm, 1);
    mbar_init(&ctrl.bar_a, 1);
    for (int c = 0; c < 2; ++c) {
      mbar_init(&ctrl.bar_ad[c], 1);
      mbar_init(&ctrl.bar_mma[c], 1);
      mbar_init(&ctrl.bar_xu[c], 8 / NCH);            // its key-row warps
      mbar_init(&ctrl.bar_ex[c], 8 / NCH + 1);
      ctrl.released[c] = 0;
    }
    mbar_init(&ctrl.bar_turn, 1);
    mbar_init(&ctrl.bar_done, NWG * 4);
    ctrl.released_pm = ctrl.released_a = 0;
    mbar_fence_init();
    ctrl.abort = 0;
  }
  // Roles: the key-row warps (0, 1 of a warpgroup) build the operand of (p) under the first MMA group, so query-row warps of a chain
  // take the extra work: its warp 2 issues the MMAs, warp 3 its loads and stores, warp 7 reads the decays of the chunk below.
  constexpr int ISSUE_WARP = 2, COPY_WARP = 3;
  if (warp == 0) { tmem_alloc(&ctrl.tmem_base, C::TMEM_COLS); tmem_relinquish(); }
  // The gradient state after the last token: zero, or what a later segment of the same sequence handed over
  // (f32 [sequence][H][E][128 d][128 v]); its bf16 image is the operand of the first chunk's products.
  float G[TPC];
  if (p.g_in != nullptr) {
    static_assert(CW % 4 == 0 && TPC % 8 == 0, "state hand-off: whole 16-byte pieces per thread");
    const float* src = p.g_in + ((static_cast<int64_t>(seq) * p.H + h) * E + e0) * (HEAD * HEAD) + row * HEAD + vb * VC + cgp * CW;
#pragma unroll
    for (int e = 0; e < EL; ++e)
#pragma unroll
      for (int c = 0; c < CW; c += 4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(src + e * (HEAD * HEAD) + c));
        G[e * CW + c] = x.x; G[e * CW + c + 1] = x.y; G[e * CW + c + 2] = x.z; G[e * CW + c + 3] = x.w;
      }
    const uint32_t base = smem_u32(smem + C::OFF_GX) + (row >> 3) * 128 + (row & 7) * 16;
#pragma unroll
    for (int j = 0; j < TPC; j += 8)
      st_shared_v4(base + ((wg * TPC + j) >> 3) * 2048, pack_bf16(G[j], G[j + 1]), pack_bf16(G[j + 2], G[j + 3]),
                   pack_bf16(G[j + 4], G[j + 5]), pack_bf16(G[j + 6], G[j + 7]));
  } else {
#pragma unroll
    for (int j = 0; j < TPC; ++j) G[j] = 0.f;
    for (int i = tid; i < C::GX_BYTES / 16; i += REC_THREADS) reinterpret_cast<uint4*>(smem + C::OFF_GX)[i] = make_uint4(0, 0, 0, 0);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctrl.tmem_base, 0);
  const int warp_u = __shfl_sync(0xffffffffu, warp & (CT / 32 - 1), 0);   // warp index inside the chain as a warp-uniform value
  const uint32_t tmem_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  const uint32_t TM_C = chain * CC, TM_Y = NCOLS + chain * YW, TM_Z = NCOLS + (NCH + chain) * YW;   // this chain's accumulators
  constexpr uint32_t TM_P = NCOLS + 2 * NCH * YW;   // P of the chains, 64 columns each (IN_TURN: of both, the first 64)
  WaitCtl ctl{&ctrl.abort, p.status};

  auto chunk_info = [&](int i, int& t0, int& rows) {
    const int n = first + i;
    t0 = n * CHUNK;
    rows = CHUNK;
    if constexpr (!PACKED) return;                   // dense rows hold whole chunks
    t0 = p.cmap[n];
    rows = p.cmap[p.NC + n];
    if (t0 < 0 || rows < 0 || rows > CHUNK || t0 + rows > p.T) {
      atomicCAS(p.status, DEV_OK, DEV_BAD_CHUNK_MAP);
      t0 = 0; rows = 0;
    }
  };
  auto issue_pm = [&](int i, int nb, uint64_t* bar) {         // one thread: the Pm image of local chunk i -> copy nb
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    bulk_load(smem + C::OFF_PM + nb * C::PM_BYTES, p.Pm + item * (64 * 64), C::PM_BYTES, bar);
  };
  auto issue_a = [&](int i, int nb, uint64_t* bar) {          // one thread: the A half of [A;PmA] of local chunk i -> copy nb
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    tma_load_5d(smem + C::OFF_A + nb * C::A_BYTES, &map_a, bar, 0, 0, 0, 0, static_cast<int>(item));
  };
  auto issue_loads = [&](int i, int st) {           // one thread: the tiles of local chunk i that live in a stage
    int t0, rows;
    chunk_info(i, t0, rows);
    uint8_t* kq = smem + C::OFF_KQ + st * C::KQ_BYTES;
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    mbar_expect_tx(&ctrl.bar_load[st], C::KQ_BYTES + 2 * C::DO_BYTES + C::GT_BYTES + (C::LATE && p.beta_tma ? C::BT_BYTES : 0) + (C::LATE ? 0u : C::A_BYTES + C::PM_BYTES));
    if (C::LATE && p.beta_tma) tma_load_4d(smem + C::OFF_BT + st * C::BT_BYTES, &map_beta, &ctrl.bar_load[st], 0, h >> 2, t0, b);
    // (eight value columns x 64 rows = one 1 KB column block of the images)
    tma_load_5d(smem + C::OFF_DO + st * C::DOB, &map_do, &ctrl.bar_load[st], 0, t0, vb * (VC / 8), h, b);
    tma_load_5d(smem + C::OFF_DU + st * C::DOB, &map_u, &ctrl.bar_load[st], 0, static_cast<int>(item * 64), vb * (VC / 8), 0, 0);
    tma_load_4d(kq, &map_k, &ctrl.bar_load[st], 0, h, t0, b);
    tma_load_4d(kq + 8192, &map_q, &ctrl.bar_load[st], 0, h, t0, b);
    tma_load_4d(kq + 16384, &map_k, &ctrl.bar_load[st], 64, h, t0, b);
    tma_load_4d(kq + 24576, &map_q, &ctrl.bar_load[st], 64, h, t0, b);
    bulk_load(smem + C::OFF_GT + st * C::GT_STRIDE, p.gc + item * gate_item_floats(E) + 64 * E, C::GT_BYTES, &ctrl.bar_load[st]);
    if constexpr (!C::LATE) {
      issue_pm(i, st, &ctrl.bar_load[st]);
      issue_a(i, st, &ctrl.bar_load[st]);
    }
  };
  auto prefetch_rows = [&](int i) {                          // the first warpgroup: what threads load themselves, for a later chunk -> L2
    if (wg != 0 || (C::LATE && p.beta_tma)) return;
    int t0, rows;
    chunk_info(i, t0, rows);
    const int last = max(rows, 1) - 1;
    const int64_t ro = (static_cast<int64_t>(b) * p.TS + t0 + min(t, last)) * p.H + h;
    if (krow) prefetch_l2(p.beta + ro);
  };
  // This thread's piece of a row of an operand image (i = t, j = v) that TMA filled: CW value columns as raw bf16
  struct Piece { uint32_t w[CW / 2]; };
  auto image_piece = [&](const uint8_t* img) {
    const uint8_t* src = img + (t >> 3) * 128 + (t & 7) * 16 + cgp * (CW / 8) * 1024;
    Piece r;
#pragma unroll
    for (int c = 0; c < CW / 8; ++c) {
      const uint4 x = *reinterpret_cast<const uint4*>(src + c * 1024);
      r.w[4 * c] = x.x; r.w[4 * c + 1] = x.y; r.w[4 * c + 2] = x.z; r.w[4 * c + 3] = x.w;
    }
    return r;
  };
  // CW packed values -> 8-column blocks `stride` bytes apart, as they are or scaled by a factor in both halves of a packed pair: the
  // operand is bf16 either way, and the product of two bf16 values rounded once costs a fifth of the f32 route.
  auto store_packed = [&](uint32_t dst, uint32_t stride, const uint32_t* w) {
#pragma unroll
    for (int c = 0; c < CW / 2; c += 4) st_shared_v4(dst + (c >> 2) * stride, w[c], w[c + 1], w[c + 2], w[c + 3]);
  };
  auto store_scaled = [&](uint32_t dst, uint32_t stride, const uint32_t* w, float f) {
    const uint32_t ff = pack_bf16(f, f);
#pragma unroll
    for (int c = 0; c < CW / 2; c += 4)
      st_shared_v4(dst + (c >> 2) * stride, mul_bf16x2(w[c], ff), mul_bf16x2(w[c + 1], ff), mul_bf16x2(w[c + 2], ff), mul_bf16x2(w[c + 3], ff));
  };
  // G_e of one chunk boundary, for the slices the gradient kernel will ask for: slice e as [v/8][d][v%8]
  auto store_state = [&](int64_t item, const uint32_t* packed) {
    uint8_t* base = reinterpret_cast<uint8_t*>(p.ds) + item * (static_cast<int64_t>(E) * 32768);
#pragma unroll
    for (int e = 0; e < EL; ++e) {
      if (!ftab[e0 + e]) continue;
      uint8_t* dst = base + (e0 + e) * 32768 + ((vb * VC + cgp * CW) >> 3) * 2048 + row * 16;
#pragma unroll
      for (int c = 0; c < CW / 2; c += 4)
        *reinterpret_cast<uint4*>(dst + (c >> 2) * 2048) = make_uint4(packed[e * (CW / 2) + c], packed[e * (CW / 2) + c + 1],
                                                                      packed[e * (CW / 2) + c + 2], packed[e * (CW / 2) + c + 3]);
    }
  };
  auto decay_flag = [&](int64_t item, int e) {      // does d_e*dd_e of this chunk matter?  (same expression in the gradient kernel)
    return __ldg(p.gc + item * gate_item_floats(E) + 63 * E + e) * LOG2E >= DD_MIN_LOG2_DECAY ? 1 : 0;
  };

  if (chain == 0 && warp_u == COPY_WARP && elect_one()) {
    issue_loads(count - 1, 0);
    if (count > 1) issue_loads(count - 2, 1);
    if constexpr (C::LATE) {
      mbar_expect_tx(&ctrl.bar_pm, C::PM_BYTES);
      issue_pm(count - 1, 0, &ctrl.bar_pm);
      mbar_expect_tx(&ctrl.bar_a, C::A_BYTES);
      issue_a(count - 1, 0, &ctrl.bar_a);
    }
  }
  __syncwarp();
  if (count > 1) prefetch_rows(count - 2);
  {
    // the gradient state at the end of the last chunk (zero unless handed in)
    if ((tid & (CT - 1)) < E) ftab[tid & (CT - 1)] = decay_flag((static_cast<int64_t>(b) * p.NC + first + count - 1) * p.H + h, tid & (CT - 1));
    __syncthreads();
    uint32_t packed0[TPC / 2];
#pragma unroll
    for (int j = 0; j < TPC / 2; ++j) packed0[j] = pack_bf16(G[2 * j], G[2 * j + 1]);
    store_state((static_cast<int64_t>(b) * p.NC + first + count - 1) * p.H + h, packed0);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
  }

  // The chunk decays of the chunk below decide whether its gradient state is stored; they are read a whole chunk before they
  // are looked at (the warp that reads them must not arrive late at the chunk's first barrier).
  // (A query-row warp without any other role reads them: the key-row warps are the critical path of the chunk's first phase.)
  constexpr int FLAG_WARP = 7;
  const bool flag_lane = warp_u == FLAG_WARP && lane < E;
  auto decay_of = [&](int i) {                       // local chunk i, slice `lane` (lane < E)
    return __ldg(p.gc + ((static_cast<int64_t>(b) * p.NC + first + i) * p.H + h) * gate_item_floats(E) + 63 * E + lane);
  };
  float gl_below = (flag_lane && count > 1) ? decay_of(count - 2) : 0.f;
  int t0_next = 0, rows_next = CHUNK;                // packed rows: the chunk's place is looked up a chunk ahead
  if constexpr (PACKED) chunk_info(count - 1, t0_next, rows_next);
  for (int kstep = 0; kstep < count; ++kstep) {
    const int i = count - 1 - kstep;
    const int st = kstep & 1;
    uint8_t* kq = smem + C::OFF_KQ + st * C::KQ_BYTES;
    const int nbi = C::NB == 2 ? st : 0;             // which copy of Pm and A this chunk uses
    uint8_t* am = smem + C::OFF_A + nbi * C::A_BYTES;
    uint8_t* pm = smem + C::OFF_PM + nbi * C::PM_BYTES;
    uint8_t* doimg = smem + C::OFF_DO + st * C::DOB;     // dO rows of the value block: operand image of Y, by TMA
    uint8_t* duimg = smem + C::OFF_DU + st * C::DOB;     // U rows by TMA, later the operand image of dU

    // ---- (a) KG = [K;Q] G and Y = Pm^T dO -----------------------------------------------------------------------
    mbar_wait(&ctrl.bar_load[st], (kstep >> 1) & 1, ctl, DEV_TIMEOUT_LOAD);
    if (C::LATE && warp_u == ISSUE_WARP) mbar_wait(&ctrl.bar_pm, kstep & 1, ctl, DEV_TIMEOUT_LOAD);
    if (warp_u == ISSUE_WARP && elect_one()) {
      tc_fence_after();
      {
        const uint64_t da = make_desc(smem_u32(pm), 128, 1024, LAYOUT_PLAIN);       // Pm^T: MN-major over (i = t, j = s)
        const uint64_t db = make_desc(smem_u32(doimg) + chain * (CV / 8) * 1024, 128, 1024, LAYOUT_PLAIN);
        constexpr uint32_t idesc = make_idesc(128, YW, 1, 1);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16(tmem + TM_Y, desc_advance(da, kk * 256), desc_advance(db, kk * 256), idesc, kk > 0);
      }
      {
        const uint64_t da = make_desc(smem_u32(kq), 16, 1024, LAYOUT_SW128);
        const uint64_t db = make_desc(smem_u32(smem + C::OFF_GX) + TM_C / 8 * 2048, 128, 2048, LAYOUT_PLAIN);
        constexpr uint32_t idesc = make_idesc(128, CC, 0, 1);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_bf16(tmem + TM_C, desc_advance(da, (kk >> 2) * 16384 + (kk & 3) * 32), desc_advance(db, kk * 256), idesc, kk > 0);
        umma_commit(&ctrl.bar_ad[chain]);
      }
    }
    __syncwarp();                                    // the other lanes must not run ahead into a spin wait
    const float gl_use = gl_below;
    if (flag_lane && i > 1) gl_below = decay_of(i - 2);
    const int t0 = PACKED ? t0_next : (first + i) * CHUNK, rows = PACKED ? rows_next : CHUNK;
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    const int64_t tok = static_cast<int64_t>(b) * p.TS + t0;
    const bool live = t < rows;
    const int v0 = cgp * CW;                         // first value column of this thread inside the block

    if (warp_u == ISSUE_WARP) {
      // (p) P = G Xu^T goes out as soon as the key-row warps have built Xu (they do that first thing in this phase): it runs
      // behind (a), under the epilogue of (a), and nobody waits for it later.  (The previous chunk's P must have been read.)
      mbar_wait_parked(&ctrl.bar_xu[chain], kstep & 1, ctl, DEV_TIMEOUT_MMA);
      if (CROSS && kstep > 0) mbar_wait_parked(&ctrl.bar_done, (kstep - 1) & 1, ctl, DEV_TIMEOUT_MMA);
      const bool add = C::IN_TURN && chain == 1;
      if (add) mbar_wait(&ctrl.bar_turn, kstep & 1, ctl, DEV_TIMEOUT_MMA);
      if (elect_one()) {
        tc_fence_after();
        // A step of K = 16 is two column blocks: the same eight value columns of two slices (of one slice: the next eight columns).
        // With sixteen columns a thread the two lie two blocks apart; first all slices of the first eight columns, then of the others.
        constexpr int APART = CW == 16 && EL > 1 ? 2 : 1, EH = EL > 1 ? EL / 2 : 1;
        const uint64_t da = make_desc(smem_u32(smem + C::OFF_GX) + TM_C / 8 * 2048, APART * 2048, 128, LAYOUT_PLAIN);   // G: K-major over (i = d, j = n')
        const uint64_t db = make_desc(smem_u32(smem + C::OFF_XU) + TM_C / 8 * 1024, APART * 1024, 128, LAYOUT_PLAIN);   // Xu: K-major over (i = t, j = n')
        constexpr uint32_t idesc = make_idesc(128, 64, 0, 0);
        const uint32_t tm_p = tmem + TM_P + (C::IN_TURN ? 0 : chain * 64);
#pragma unroll
        for (int kk = 0; kk < CC / 16; ++kk) {
          const int blk = APART == 1 ? 2 * kk : kk / EL * (2 * EL) + kk % EL / EH + kk % EH * 4;
          umma_bf16(tm_p, desc_advance(da, blk * 2048), desc_advance(db, blk * 1024), idesc, add || kk > 0);
        }
        if (C::IN_TURN && chain == 0) umma_commit(&ctrl.bar_turn);
        umma_commit(&ctrl.bar_ex[chain]);
      }
      __syncwarp();
    }
    // This chain is done with the previous chunk's stage (its last store of dU has left the stage's buffer); the last chain to say
    // so refills it.
    if (kstep > 0 && warp_u == COPY_WARP && elect_one()) {
      if constexpr (!DV_TILE) bulk_wait_group_read();
      if (atomicAdd(&ctrl.released[st ^ 1], 1u) % NCH == NCH - 1 && kstep + 1 < count) issue_loads(i - 1, st ^ 1);
    }
    __syncwarp();
    // Under the MMA: this row's gate factors, and (K-row threads, which would otherwise only wait for the MMA) the operand
    // Xu of (p).
    float ga[EL];                                    // this thread's slices.  K rows: a_e = k2 exp(gc); Q rows: c_e = scale q2 exp(gc)
    float gr[EL];                                    // K rows: r_e = k2 exp(gL - gc)
    float bt = 0.f;
    {
      const float* gf = reinterpret_cast<const float*>(smem + C::OFF_GT + st * C::GT_STRIDE);
      lds_row<E, EL>(gf + (krow ? 0 : C::GF_C), t, e0, ga);
      if (krow) {
        lds_row<E, EL>(gf + C::GF_R, t, e0, gr);
        if (C::LATE && p.beta_tma) bt = reinterpret_cast<const float*>(smem + C::OFF_BT + st * C::BT_BYTES)[t * 4 + (h & 3)];
        else bt = __ldg(p.beta + (tok + min(t, max(rows, 1) - 1)) * p.H + h);   // masked where it is used, after (c): nothing here waits for it
        const Piece up = image_piece(duimg);
        // Xu_e = r_e * U -> operand image (i = t, j = n') of (p)
        const uint32_t base = smem_u32(smem + C::OFF_XU) + (t >> 3) * 128 + (t & 7) * 16;
#pragma unroll
        for (int e = 0; e < EL; ++e) {
          const int n0 = wg * TPC + e * CW;
          store_scaled(base + (n0 >> 3) * 1024, 1024, up.w, gr[e]);
        }
        fence_async_smem();                            // Xu is read by the tensor core: say so, one arrival per key-row warp
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctrl.bar_xu[chain]);
      } else {
#pragma unroll
        for (int e = 0; e < EL; ++e) gr[e] = 0.f;
      }
      if ((tid & (CT - 1)) < E) dtab[tid & (CT - 1)] = gf[C::GF_D + (tid & (CT - 1))];
      if (flag_lane && i > 0) {
        float glv = gl_use;
        asm volatile("" : "+f"(glv));                // the comparison stays here: nothing waits for the load before this point
        ftab[lane] = glv * LOG2E >= DD_MIN_LOG2_DECAY ? 1 : 0;   // read after the chunk's last barrier but one
      }
      if (kstep + 2 < count) prefetch_rows(i - 2);
    }
    mbar_wait_parked(&ctrl.bar_ad[chain], 0, ctl, DEV_TIMEOUT_MMA);      // (a) and (d) of every chunk: even and odd completions
    tc_fence_after();
    if constexpr (C::LATE) {                         // the chain's (a) has read Pm: when both have, the next chunk's copy is asked for
      if (warp_u == COPY_WARP && elect_one()) {
        if (atomicAdd(&ctrl.released_pm, 1u) % NCH == NCH - 1 && kstep + 1 < count) {
          mbar_expect_tx(&ctrl.bar_pm, C::PM_BYTES);
          issue_pm(i - 1, 0, &ctrl.bar_pm);
        }
      }
      __syncwarp();
    }
    float du[CW];                                    // K rows: dU of this thread's columns (NSG > 1: its slice group's part)
    if (krow) {
      float uv[CW];
      const Piece up = image_piece(duimg);
#pragma unroll
      for (int c = 0; c < CW; ++c) uv[c] = (c & 1) ? bf16_hi(up.w[c >> 1]) : bf16_lo(up.w[c >> 1]);
      constexpr int EP = (8 / CW) < 1 ? 1 : (8 / CW) < EL ? (8 / CW) : EL;   // slices per piece of eight columns
      constexpr int NP = EL / EP;
      float kg[2][EP * CW];
      if (CROSS && kstep > 0) mbar_wait_parked(&ctrl.bar_done, (kstep - 1) & 1, ctl, DEV_TIMEOUT_MMA);   // the previous chunk's dr partials have been read
      if (sgp == 0) {
        tmem_ld<CW>(tmem_row + TM_Y + (v0 - chain * CV), du);
      } else {
#pragma unroll
        for (int c = 0; c < CW; ++c) du[c] = 0.f;
      }
      tmem_ld<EP * CW>(tmem_row + wg * TPC, kg[0]);
#pragma unroll
      for (int pc = 0; pc < NP; ++pc) {                       // the next piece travels while this one is used
        tmem_wait_ld();
        if (pc + 1 < NP) tmem_ld<EP * CW>(tmem_row + wg * TPC + (pc + 1) * EP * CW, kg[(pc + 1) & 1]);
        const float* kp = kg[pc & 1];
#pragma unroll
        for (int ee = 0; ee < EP; ++ee) {
          // dr partials: the even and the odd columns of every eight apart, whatever the thread's width
          const float re = gr[pc * EP + ee];
          float part = 0.f;
#pragma unroll
          for (int c8 = 0; c8 < CW; c8 += 8) {
            float2 dot = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = c8; c < c8 + 8; c += 2) {
              const float k0 = kp[ee * CW + c], k1 = kp[ee * CW + c + 1];
              if constexpr (TWO_WIDE) {
                fma_pair(du[c], du[c + 1], re, k0, k1);
                dot = __ffma2_rn(make_float2(uv[c], uv[c + 1]), make_float2(k0, k1), dot);
              } else {
                du[c] = fmaf(re, k0, du[c]);
                du[c + 1] = fmaf(re, k1, du[c + 1]);
                dot.x = fmaf(uv[c], k0, dot.x);
                dot.y = fmaf(uv[c + 1], k1, dot.y);
              }
            }
            part = c8 == 0 ? dot.x + dot.y : part + (dot.x + dot.y);
          }
          drp[(cgp * 64 + t) * ES + e0 + pc * EP + ee] = part;
        }
      }
      if constexpr (NSG > 1) {
        static_assert(NSG <= 2 && (NSG == 1 || CW % 4 == 0), "the exchange below is written for two slice groups");
        if (sgp != 0) {
#pragma unroll
          for (int c = 0; c < CW; c += 4)
            *reinterpret_cast<float4*>(dured + t * VC + v0 + c) = make_float4(du[c], du[c + 1], du[c + 2], du[c + 3]);
        }
      }
    }
    if (krow) {                                      // this warp's dr partials are written (read by both chains, below)
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctrl.bar_ex[chain]);
    }
    if constexpr (NSG > 1) rec_chain_sync<CT>(chain);   // the other slice group's part of dU; every reader of the U piece is done
    if (krow && sgp == 0) {
      if constexpr (NSG > 1) {
#pragma unroll
        for (int c = 0; c < CW; c += 4) {
          const float4 x = *reinterpret_cast<const float4*>(dured + t * VC + v0 + c);
          du[c] += x.x; du[c + 1] += x.y; du[c + 2] += x.z; du[c + 3] += x.w;
        }
      }
      // dU replaces this thread's piece of U in the image; the image then leaves for global memory by a TMA store
      uint32_t dw[CW / 2];
#pragma unroll
      for (int c = 0; c < CW; c += 2) dw[c >> 1] = pack_bf16(du[c], du[c + 1]);
      store_packed(smem_u32(duimg) + cgp * (CW / 8) * 1024 + (t >> 3) * 128 + (t & 7) * 16, 1024, dw);
    }
    fence_async_smem();
    tc_fence_before();
    rec_chain_sync<CT>(chain);

    // ---- (c) Z = A^T dU -----------------------------------------------------------------------------------------
    if (C::LATE && warp_u == ISSUE_WARP) mbar_wait(&ctrl.bar_a, kstep & 1, ctl, DEV_TIMEOUT_LOAD);
    if (warp_u == ISSUE_WARP && elect_one()) {
      tc_fence_after();
      {
        const uint64_t da = make_desc(smem_u32(am), 128, 1024, LAYOUT_PLAIN);         // A^T: MN-major over (i = t, j = s)
        const uint64_t db = make_desc(smem_u32(duimg) + chain * (CV / 8) * 1024, 128, 1024, LAYOUT_PLAIN);
        constexpr uint32_t idesc = make_idesc(128, YW, 1, 1);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16(tmem + TM_Z, desc_advance(da, kk * 256), desc_advance(db, kk * 256), idesc, kk > 0);
        umma_commit(&ctrl.bar_mma[chain]);
      }
    }
    __syncwarp();                                    // the other lanes must not run ahead into a spin wait
    if (PACKED && i > 0) chunk_info(i - 1, t0_next, rows_next);
    if (warp_u == COPY_WARP && elect_one()) {                // dU (chunk layout) straight from its operand image
      tma_store_5d(&map_du, duimg + chain * (CV / 8) * 1024, 0, static_cast<int>(item * 64), (vb * VC + chain * CV) / 8, 0, 0);
      bulk_commit_group();
    }
    __syncwarp();
    mbar_wait_parked(&ctrl.bar_mma[chain], kstep & 1, ctl, DEV_TIMEOUT_MMA);
    tc_fence_after();
    if constexpr (C::LATE) {                         // the chain's (c) has read A
      if (warp_u == COPY_WARP && elect_one()) {
        if (atomicAdd(&ctrl.released_a, 1u) % NCH == NCH - 1 && kstep + 1 < count) {
          mbar_expect_tx(&ctrl.bar_a, C::A_BYTES);
          issue_a(i - 1, 0, &ctrl.bar_a);
        }
      }
      __syncwarp();
    }
    {
      uint32_t xw[CW / 2];
#pragma unroll
      for (int c = 0; c < CW / 2; ++c) xw[c] = 0u;   // K rows: dW; Q rows: dO; packed bf16, the form both leave in
      if (krow) {
        float z[CW];
        tmem_ld<CW>(tmem_row + TM_Z + (v0 - chain * CV), z);
        tmem_wait_ld();
        asm volatile("" : "+f"(bt));                   // first use of the beta load of phase (a)
        if (!live) bt = 0.f;
#pragma unroll
        for (int c = 0; c < CW; c += 2) xw[c >> 1] = pack_bf16(bt * z[c], bt * z[c + 1]);
        if (live && sgp == 0 && !(DV_TILE && rows == CHUNK)) {
          __nv_bfloat16* dst = p.dV + ((tok + t) * p.H + h) * HEAD + vb * VC + v0;
#pragma unroll
          for (int c = 0; c < CW / 2; c += 4) *reinterpret_cast<uint4*>(dst + 2 * c) = make_uint4(xw[c], xw[c + 1], xw[c + 2], xw[c + 3]);
        }
      } else if (live) {
        const Piece w = image_piece(doimg);
#pragma unroll
        for (int c = 0; c < CW / 2; ++c) xw[c] = w.w[c];
      }
      // (p) reads the image of G that X is about to replace
      mbar_wait_parked(&ctrl.bar_ex[chain], kstep & 1, ctl, DEV_TIMEOUT_MMA);
      // dV of a whole chunk leaves as an image from the place of Xu, which (p) has read (a row of its own per thread would cost 32
      // wavefronts a store; a chunk cut short by a document end may not leave as a tile)
      if (DV_TILE && krow && rows == CHUNK)
        store_packed(smem_u32(smem + C::OFF_XU) + (TM_C / 8 + (v0 - chain * CV) / 8) * 1024 + (t >> 3) * 128 + (t & 7) * 16, 1024, xw);
      // X image (i = row, j = n'): rows 0..63 -a_e*dW, rows 64..127 c_e*dO
      const uint32_t base = smem_u32(smem + C::OFF_GX) + (row >> 3) * 128 + (row & 7) * 16;
#pragma unroll
      for (int e = 0; e < EL; ++e) {
        const float f = krow ? -ga[e] : ga[e];
        const int n0 = wg * TPC + e * CW;
        store_scaled(base + (n0 >> 3) * 2048, 2048, xw, f);
      }
    }
    fence_async_smem();
    tc_fence_before();
    rec_chain_sync<CT>(chain);

    if (DV_TILE && warp_u == COPY_WARP && rows == CHUNK && elect_one()) {
      tma_store_5d(&map_dv, smem + C::OFF_XU + TM_C / 8 * 1024, 0, t0, (vb * VC + chain * CV) / 8, h, b);
      bulk_commit_group();
    }
    __syncwarp();
    // ---- (d) dG = [K^T | Q^T] X, G <- d G + dG ------------------------------------------------------------------
    if (warp_u == ISSUE_WARP && elect_one()) {
      tc_fence_after();
      const uint64_t da = make_desc(smem_u32(kq), 16384, 1024, LAYOUT_SW128);
      const uint64_t db = make_desc(smem_u32(smem + C::OFF_GX) + TM_C / 8 * 2048, 128, 2048, LAYOUT_PLAIN);
      constexpr uint32_t idesc = make_idesc(128, CC, 1, 1);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16(tmem + TM_C, desc_advance(da, kk * 2048), desc_advance(db, kk * 256), idesc, kk > 0);
      umma_commit(&ctrl.bar_ad[chain]);
    }
    __syncwarp();                                    // the other lanes must not run ahead into a spin wait
    // meanwhile: the two sums over all value columns of a block, of which each chain that shares one takes half of the tokens: P (128
    // key rows x 64 tokens, f32, the chains' shares added) -> bf16 operand image (i = d, j = t), SI = 128, SJ = 2048 (a warp's 16-byte
    // stores cover 512 contiguous bytes), and dr from the partials of the column groups in a fixed order.
    if (CROSS) mbar_wait_parked(&ctrl.bar_ex[chain ^ 1], kstep & 1, ctl, DEV_TIMEOUT_MMA);
    {
      tc_fence_after();
      const int64_t block = item * NVB + (C::OWN ? vb * 2 + chain : vb);
      uint8_t* dst = reinterpret_cast<uint8_t*>(p.dkg) + block * 16384 + row * 16;
      float* dr_out = p.dr + block * (64 * E);
      constexpr int TOKENS = C::OWN ? 32 : 16;       // of this warpgroup
      const int c0 = (C::OWN ? wg & 1 : wg) * TOKENS;
#pragma unroll
      for (int cc = 0; cc < TOKENS; cc += 16) {
        float pv[16], pw[16];
        tmem_ld<16>(tmem_row + TM_P + (C::OWN ? chain * 64 : 0) + c0 + cc, pv);
        if constexpr (CROSS && !C::IN_TURN) tmem_ld<16>(tmem_row + TM_P + 64 + c0 + cc, pw);
        if (cc == 0) {
          constexpr int ROWS = C::OWN ? 64 : 64 / NCH;
          for (int idx = tid & (CT - 1); idx < ROWS * E; idx += CT) {
            const int r = (C::OWN ? 0 : chain * ROWS) + idx / E, e = idx % E;
            const float* part = drp + r * ES + e;    // group w: 64 * ES floats further on
            float sum;
            if constexpr (C::OWN) sum = part[2 * chain * (64 * ES)] + part[(2 * chain + 1) * (64 * ES)];
            else if constexpr (E <= 4) sum = (part[0] + part[64 * ES]) + (part[2 * 64 * ES] + part[3 * 64 * ES]);   // as the wide CTA adds
            else {
              sum = part[0];
#pragma unroll
              for (int w = 1; w < NCG; ++w) sum += part[w * (64 * ES)];
            }
            dr_out[r * E + e] = sum;
          }
        }
        tmem_wait_ld();
        if constexpr (CROSS && !C::IN_TURN) {
#pragma unroll
          for (int j = 0; j < 16; ++j) pv[j] += pw[j];
        }
#pragma unroll
        for (int j = 0; j < 16; j += 8)
          *reinterpret_cast<uint4*>(dst + ((c0 + cc + j) >> 3) * 2048) =
              make_uint4(pack_bf16(pv[j], pv[j + 1]), pack_bf16(pv[j + 2], pv[j + 3]), pack_bf16(pv[j + 4], pv[j + 5]),
                         pack_bf16(pv[j + 6], pv[j + 7]));
      }
      if constexpr (CROSS) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctrl.bar_done);
      }
    }
    mbar_wait_parked(&ctrl.bar_ad[chain], 1, ctl, DEV_TIMEOUT_MMA);
    tc_fence_after();
    {
      constexpr int PIECE = TPC < 16 ? TPC : 16;
      const uint32_t base = smem_u32(smem + C::OFF_GX) + (row >> 3) * 128 + (row & 7) * 16;
      uint8_t* sbase = i > 0 ? reinterpret_cast<uint8_t*>(p.ds) + (item - p.H) * (static_cast<int64_t>(E) * 32768) : nullptr;
      const int vg = vb * VC + cgp * CW;
      float dg[2][PIECE];
      tmem_ld<PIECE>(tmem_row + wg * TPC, dg[0]);
#pragma unroll
      for (int j0 = 0; j0 < TPC; j0 += PIECE) {               // the next piece travels while this one is used
        tmem_wait_ld();
        if (j0 + PIECE < TPC) tmem_ld<PIECE>(tmem_row + wg * TPC + j0 + PIECE, dg[((j0 / PIECE) + 1) & 1]);
        const float* dp = dg[(j0 / PIECE) & 1];
        uint32_t packed[PIECE / 2];
#pragma unroll
        for (int j = 0; j < PIECE; j += 2) {
          scale_add_pair(G[j0 + j], G[j0 + j + 1], dtab[e0 + (j0 + j) / CW], dp[j], dp[j + 1]);
          packed[j / 2] = pack_bf16(G[j0 + j], G[j0 + j + 1]);
        }
        // operand image (i = d, j = n') of the next (a)
#pragma unroll
        for (int j = 0; j < PIECE; j += 8) {
          const int n0 = wg * TPC + j0 + j;
          st_shared_v4(base + (n0 >> 3) * 2048, packed[j / 2], packed[j / 2 + 1], packed[j / 2 + 2], packed[j / 2 + 3]);
        }
        // G_e at the end of the previous chunk, for the slices the gradient kernel will ask for: [v/8][d][v%8]
        if (sbase != nullptr) {
#pragma unroll
          for (int j = 0; j < PIECE; j += CW) {
            const int e = e0 + (j0 + j) / CW;
            if (!ftab[e]) continue;
            uint8_t* dst = sbase + e * 32768 + (vg >> 3) * 2048 + row * 16;
#pragma unroll
            for (int c = 0; c < (CW < PIECE ? CW : PIECE) / 2; c += 4)
              *reinterpret_cast<uint4*>(dst + (c >> 2) * 2048) = make_uint4(packed[j / 2 + c], packed[j / 2 + c + 1], packed[j / 2 + c + 2], packed[j / 2 + c + 3]);
          }
        }
      }
    }
    if (DV_TILE && warp_u == COPY_WARP && elect_one()) bulk_wait_group_read();   // dU and dV have left: their places take the next chunk's U and Xu
    fence_async_smem();
    tc_fence_before();
    rec_chain_sync<CT>(chain);
  }
  // dL/dS before the first token, for an earlier segment of the same sequence
  if (p.g_out != nullptr) {
    float* dst = p.g_out + ((static_cast<int64_t>(seq) * p.H + h) * E + e0) * (HEAD * HEAD) + row * HEAD + vb * VC + cgp * CW;
#pragma unroll
    for (int e = 0; e < EL; ++e)
#pragma unroll
      for (int c = 0; c < CW; c += 4)
        *reinterpret_cast<float4*>(dst + e * (HEAD * HEAD) + c) = make_float4(G[e * CW + c], G[e * CW + c + 1], G[e * CW + c + 2], G[e * CW + c + 3]);
  }
  if (warp_u == COPY_WARP && elect_one()) bulk_wait_group();   // the last store of dU reads shared memory of this CTA
  tc_fence_before();
  __syncthreads();                                           // both chains are done with tensor memory
  if (warp == 0) tmem_dealloc(tmem, C::TMEM_COLS);
}

}  // namespace tgdn

using namespace tgdn;

template <int E, int VC, int NCH, int NSG, bool PACKED>
static int launch_rec_rows(const CUtensorMap& mk, const CUtensorMap& mq,
                      const CUtensorMap& mdo, const CUtensorMap& mu, const CUtensorMap& mdu, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mdv, const RecParams& p, cudaStream_t s) {
  using C = RecCfg<E, VC, NCH, NSG>;
  static_assert(C::SMEM_BYTES <= 232448, "shared memory budget of one CTA exceeded");
  static bool configured[64] = {};
  if (const int rc = tgdn_dynamic_smem(reinterpret_cast<const void*>(rec_kernel<E, VC, NCH, NSG, PACKED>), C::SMEM_BYTES, configured)) return rc;
  rec_kernel<E, VC, NCH, NSG, PACKED><<<p.n_seq * p.H * (HEAD / VC), C::THREADS, C::SMEM_BYTES, s>>>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p);
  return tgdn_cuda_error(cudaGetLastError());
}
template <int E, int VC, int NCH, int NSG = 1>
static int launch_rec(const CUtensorMap& mk, const CUtensorMap& mq,
                      const CUtensorMap& mdo, const CUtensorMap& mu, const CUtensorMap& mdu, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mdv, const RecParams& p, cudaStream_t s) {
  return p.cmap != nullptr ? launch_rec_rows<E, VC, NCH, NSG, true>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s)
                           : launch_rec_rows<E, VC, NCH, NSG, false>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
}

// Two value blocks per CTA?  Up to four slices a CTA of 64 columns (two chains of 32) takes 1.3 to 1.35 times as long per chunk as one
// of 32 for twice the columns: it wins when it saves waves (one CTA per SM) by more than that.  us, narrow -> wide, B=4, T=4096, H=16
// (two waves or one): E = 1 289 -> 188, E = 2 306 -> 206, E = 4 378 -> 256.  On packed rows the host knows the number of documents but
// not their lengths, and where one document's chain sets the time the wide CTA's longer chunk loses: forward + backward, E = 1 / 2 / 4,
// sixteen documents of 1024 tokens, H=8: 505 / 562 / 655 -> 446 / 499 / 605; one of 8192 and eight of 1024: 834 / 920 / 1126 -> 906 /
// 994 / 1323.
static bool rec_wide(int E, long long sequences, int H) {
  if (E > 4) return false;
  const long long sms = tgdn_sm_count(), seqs = sequences * H;
  const long long narrow = (seqs * 4 + sms - 1) / sms, wide = (seqs * 2 + sms - 1) / sms;
  return wide * 7 < narrow * 5;
}

int tgdn_bwd_recurrent_rows(const void* q, const void* k, const void* dO, const float* k2, const float* q2, const float* beta,
                            const float* gc, const void* AP, const void* Pm, const void* U, float scale, const int32_t* doc_offsets,
                            const int32_t* chunk_map, int n_docs, int B, int T, int H, int E, int NC, int row_tokens, void* dV,
                            void* dU, void* ds, void* dkg, float* dr, const float* grad_state_in, float* grad_state_out,
                            void* stream, int* zeroed) {
  if ((reinterpret_cast<uintptr_t>(grad_state_in) | reinterpret_cast<uintptr_t>(grad_state_out)) & 15) return TGDN_ERR_ALIGN;
  if (!q || !k || !dO || !k2 || !q2 || !beta || !gc || !AP || !Pm || !U || !dV || !dU || !ds || !dkg || !dr) return TGDN_ERR_NULL;
  const bool packed = chunk_map != nullptr;
  if (packed && (!doc_offsets || n_docs < 1)) return TGDN_ERR_NULL;
  int rc = tgdn_check_core_shape(B, T, H, E, NC, packed, row_tokens);
  if (rc) return rc;
  if ((reinterpret_cast<uintptr_t>(dO) | reinterpret_cast<uintptr_t>(AP) | reinterpret_cast<uintptr_t>(Pm) |
       reinterpret_cast<uintptr_t>(U) | reinterpret_cast<uintptr_t>(dV) | reinterpret_cast<uintptr_t>(dU) |
       reinterpret_cast<uintptr_t>(ds) | reinterpret_cast<uintptr_t>(dkg) | reinterpret_cast<uintptr_t>(k2) |
       reinterpret_cast<uintptr_t>(q2) | reinterpret_cast<uintptr_t>(gc)) & 15)
    return TGDN_ERR_ALIGN;
  CUtensorMap mk, mq;
  if ((rc = tgdn_make_token_map(&mk, k, B, T, H, 64, 64, 1, row_tokens))) return rc;
  if ((rc = tgdn_make_token_map(&mq, q, B, T, H, 64, 64, 1, row_tokens))) return rc;
  // dO (token layout) and U, dU (chunk layout: item * 64 + t rows of 128 columns) as operand images of the value block
  const int64_t crows = static_cast<int64_t>(B) * NC * H * 64;
  if (crows > 0x7fffffffLL) return TGDN_ERR_SHAPE;
  CUtensorMap mdo, mu, mdu, mdv, ma, mb = mk;
  const int beta_tma = H % 4 == 0 && (reinterpret_cast<uintptr_t>(beta) & 15) == 0 ? 1 : 0;
  if (beta_tma && (rc = tgdn_make_gate_map(&mb, beta, B, T, H / 4, 4, row_tokens))) return rc;   // (B, T, H) read as (B, T, H/4, 4)
  const bool wide = rec_wide(E, packed ? n_docs : B, H);
  const int blocks = (wide ? 64 : tgdn_value_block(E)) / 8, share = E <= 2 && !wide ? blocks : blocks / 2;   // dU leaves by chain
  if ((rc = tgdn_make_image_map(&mdo, dO, B, T, H, blocks, row_tokens))) return rc;
  if ((rc = tgdn_make_image_map(&mu, U, 1, static_cast<int>(crows), 1, blocks))) return rc;
  if ((rc = tgdn_make_image_map(&mdu, dU, 1, static_cast<int>(crows), 1, share))) return rc;
  if ((rc = tgdn_make_image_map(&mdv, dV, B, T, H, share, row_tokens))) return rc;
  if ((rc = tgdn_make_a_half_map(&ma, AP, static_cast<long long>(B) * NC * H))) return rc;
  RecParams p{static_cast<const __nv_bfloat16*>(dO), k2, q2, beta, gc, static_cast<const __nv_bfloat16*>(AP),
              static_cast<const __nv_bfloat16*>(Pm), static_cast<const __nv_bfloat16*>(U),
              static_cast<__nv_bfloat16*>(dV), static_cast<__nv_bfloat16*>(dU), static_cast<__nv_bfloat16*>(ds),
              static_cast<__nv_bfloat16*>(dkg), dr, doc_offsets, chunk_map, B, T, H, NC, packed ? n_docs : B, row_tokens, scale,
              tgdn_status_word(), grad_state_in, grad_state_out, beta_tma, zeroed};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (E) {
    case 1:
      if (wide) return launch_rec<1, 64, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
      return launch_rec<1, 32, 1>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
    case 2:
      if (wide) return launch_rec<2, 64, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
      return launch_rec<2, 32, 1>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
    case 4:
      if (wide) return launch_rec<4, 64, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
      return launch_rec<4, 32, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
    // E = 8: 32 value columns per CTA measured 9% faster than two CTAs per SM of 16 columns each (5.26 -> 4.77 ms at B=8, T=8192, H=32,
    // before the chains), and the gradient kernel then adds four value-block images per item instead of eight.
    case 8: return launch_rec<8, 32, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
    case 12: return launch_rec<12, 16, 2, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
    case 16: return launch_rec<16, 16, 2, 2>(mk, mq, mdo, mu, mdu, ma, mb, mdv, p, s);
    default: return TGDN_ERR_SHAPE;
  }
}

extern "C" int tgdn_bwd_recurrent_state(const void* q, const void* k, const void* dO, const float* k2, const float* q2,
                                        const float* beta, const float* gc, const void* AP, const void* Pm, const void* U,
                                        float scale, const int32_t* doc_offsets, const int32_t* chunk_map, int n_docs, int B,
                                        int T, int H, int E, int NC, void* dV, void* dU, void* ds, void* dkg, float* dr,
                                        const float* grad_state_in, float* grad_state_out, void* stream) {
  return tgdn_bwd_recurrent_rows(q, k, dO, k2, q2, beta, gc, AP, Pm, U, scale, doc_offsets, chunk_map, n_docs, B, T, H, E, NC, T,
                                 dV, dU, ds, dkg, dr, grad_state_in, grad_state_out, stream);
}

extern "C" int tgdn_bwd_recurrent(const void* q, const void* k, const void* dO, const float* k2, const float* q2,
                                  const float* beta, const float* gc, const void* AP, const void* Pm, const void* U,
                                  float scale, const int32_t* doc_offsets, const int32_t* chunk_map, int n_docs, int B,
                                  int T, int H, int E, int NC, void* dV, void* dU, void* ds, void* dkg, float* dr,
                                  void* stream) {
  return tgdn_bwd_recurrent_state(q, k, dO, k2, q2, beta, gc, AP, Pm, U, scale, doc_offsets, chunk_map, n_docs, B, T, H, E, NC,
                                  dV, dU, ds, dkg, dr, nullptr, nullptr, stream);
}
