// Forward chunk recurrence of the Triadic GDN.
//
// One CTA owns one (sequence, head, block of VC value columns) and walks the sequence's 64-token chunks in order.  The
// block is split over NCH independent CHAINS of one or two warpgroups (a warpgroup = 128 threads = the 128 rows of [K;Q]); chain c
// owns CV value columns of every slice: its E state slices S_e[:, columns] (128 x CV each, f32) live in the registers of its
// threads.  Two warpgroups of a chain share its value columns (WV = 2) or, at twelve and sixteen slices, its slices (WS = 2).
// Per chunk a chain runs three dependent MMA groups of its own, with its own accumulators in tensor memory:
//   (1) R  = [K;Q] S          tcgen05, M=128, N=E*CW, K=128   rows 0..63: K S_e, rows 64..127: Q S_e
//       W  = V - sum_e a_e*R_e (K rows);   Oq = sum_e c_e*R_e (Q rows)
//   (2) [U;Oi] = [A;PmA] (beta*W)   tcgen05, M=128, N=16 (CW used), K=64
//       o  = Oq + Oi  ->  bf16;   Vn_e = r_e*U
//   (3) dS = K^T Vn           tcgen05, M=128, N=E*CW, K=64
//       S_e <- d_e S_e + dS_e  (registers), bf16 copy -> shared memory operand of the next (1) and saved state h
// with a = k2 exp(gc), r = k2 exp(gL-gc), c = scale q2 exp(gc), d = exp(gL).
//
// The chains of a CTA share only the chunk's tiles (K/Q, the [A;PmA] image, the gate factors, the value rows of the block
// and the beta rows), which arrive by TMA in a ring of STAGES stages; a stage is refilled by whichever chain is the last to
// hand it back, so no chain ever waits for another one except through that ring.  Everything else is private to a chain
// (its columns are independent of all other columns of the problem): its barrier is a named barrier of its own threads,
// its MMAs are issued by one of its own lanes and complete on its own mbarrier.  While one chain waits for its MMA or its tensor-memory load, the tensor core and the
// issue slots work for the others: the dependent chain of a chunk (three MMA -> load -> epilogue round trips) is what
// bounds this kernel, and the independent chains per SM are what hides it.  Next to it come instruction issue (hence the two-wide
// f32 multiply-adds) and the copy engine: it moves a row of a tile a cycle and writes 32 bytes a cycle, so o, W and U leave as
// tiles as wide as a chain, the state leaves by stores, and later chunks are pulled into L2 by the threads.
// us, before all three and after: 8192 items E8 850 -> 764, without saved state 717 -> 573; 4096 items E4 250 -> 209, 190 -> 160;
// E2 201 -> 152, 149 -> 129; E1 187 -> 133, 138 -> 111; packed E16 1658 -> 1663, 1450 -> 1264; E12 778 -> 745, 694 -> 569.
//
// The gate factors of a chunk (a, r, c per row and slice, d per slice) were formed by the masks kernel and arrive in the
// stage with one bulk copy; every thread reads those of its own row (K rows: a, r, beta; Q rows: c) right after its
// chain's MMA (1) went out.  Nothing couples the chains but the tile ring.  The key-row warps have the longer phases (two
// gate factors per slice, the operand images of beta*W and r_e*U), so the chain's extra roles sit on its query-row
// warps: one issues the MMAs and waits for them, one hands stages back and issues the loads.
//
// Replaces cute_triadic_gdn/kernels/sm100_joint_fwd.py:66-527 (fwd_kernel); math as cute_triadic_gdn/ops/gdn_joint.py:63-90.
// Column order inside a chain: n' = (w*E + e)*CW + c  <->  (slice e, value column w*CW + c of the chain).
#include "tgdn_common.cuh"
#include "tgdn_host.h"
#include "tgdn_kernels.h"

namespace tgdn {

template <int THREADS>
__device__ __forceinline__ void chain_sync(int chain) {     // the threads of one chain
  asm volatile("bar.sync %0, %1;" ::"r"(chain + 1), "n"(THREADS) : "memory");
}

// WS = 2 warpgroups share one chain and split its SLICES (warpgroup w of a chain owns slices w*E/WS ..): the chain's MMAs
// then have N = E*CW columns with CW = 8 columns per thread even at twelve and sixteen slices, where a warpgroup alone
// could hold only four columns of every slice in its registers; the sums over the slices (W, and the state part of o) are
// completed through shared memory.  WV = 2 warpgroups split the chain's value columns (CW per thread, CV per chain): nothing to
// exchange, and products of twice the width.
template <int E, int CW, int NCH, int WS, int WV, int STAGES>
struct FwdCfg {
  static constexpr int WPC = WS * WV;             // warpgroups per chain: WS share the slices, WV the value columns
  static constexpr int CHAIN_THREADS = WPC * 128;
  static constexpr int THREADS = NCH * CHAIN_THREADS;
  static constexpr int CV = CW * WV;              // value columns of a chain
  static constexpr int VC = CV * NCH;             // value columns of the CTA
  static constexpr int TPC = E * CV;              // state columns per chain
  static constexpr int ET = E / WS;               // slices per thread
  static constexpr int TPT = ET * CW;             // state columns per thread
  static constexpr int UW = CV < 16 ? 16 : CV;    // columns of the (2) accumulator (the smallest N of an M=128 MMA is 16)
  static constexpr int TW = TPC + UW;             // tensor-memory columns per chain
  static constexpr int TMEM_NEED = NCH * TW;
  static constexpr int TMEM_COLS = TMEM_NEED <= 32 ? 32 : TMEM_NEED <= 64 ? 64 : TMEM_NEED <= 128 ? 128 : TMEM_NEED <= 256 ? 256 : 512;
  // shared memory carve-up (bytes); the swizzled tiles are 1024-byte aligned
  static constexpr int KQ_BYTES = 32768;
  static constexpr int AP_BYTES = 16384;
  static constexpr int S_BYTES = TPC * 256;       // per chain: image (i = d, j = n'), SI = 128, SJ = 2048
  static constexpr int VN_BYTES = TPC * 128;      // per chain: image (i = t, j = n'), SI = 128, SJ = 1024
  static constexpr int BWI_BYTES = UW * 128;      // per chain: image (i = s, j = v), SI = 128, SJ = 1024
  // W on its way out: in the block that a chain of eight columns leaves unused, else behind the operand where that fits, else
  // (W_OWN false) in the place of the value rows, before o
  static constexpr int WST_OFF = CV == 8 ? 1024 : BWI_BYTES;
  static constexpr int bytes_with(int bw) {
    const int gt = (OFF_BW + NCH * bw + 127) & ~127;
    return gt + STAGES * (((gate_factor_bytes(E) + 127) & ~127) + VC * 128) + 512 + 128 + 1024;
  }
  static constexpr int OFF_KQ = 0;
  static constexpr int OFF_AP = OFF_KQ + STAGES * KQ_BYTES;
  static constexpr int OFF_S = OFF_AP + STAGES * AP_BYTES;
  static constexpr int OFF_VN = OFF_S + NCH * S_BYTES;
  static constexpr int OFF_BW = OFF_VN + NCH * VN_BYTES;
  static constexpr bool W_OWN = CV == 8 || bytes_with(BWI_BYTES + CV * 128) <= 232448;
  static constexpr int BW_BYTES = CV == 8 || !W_OWN ? BWI_BYTES : BWI_BYTES + CV * 128;
  // per stage: the gate factors of the chunk as the masks kernel stored them, a, r, c as 64 dense rows of E floats each,
  // then d (one bulk copy)
  static constexpr int GT_BYTES = gate_factor_bytes(E);
  static constexpr int GT_STRIDE = (GT_BYTES + 127) & ~127;
  static constexpr int GF_R = 64 * E, GF_C = 128 * E, GF_D = 192 * E;   // float offsets of r, c, d behind a
  static constexpr int OFF_GT = (OFF_BW + NCH * BW_BYTES + 127) & ~127;
  // per stage: the value rows of the CTA's columns, one tile of 64 rows x CV columns per chain, and the beta rows of the chunk for
  // the four heads h & ~3 .. (TMA when H is a multiple of 4)
  static constexpr int VBOX_BYTES = 64 * CV * 2;
  static constexpr int VT_BYTES = NCH * VBOX_BYTES;
  static constexpr int OFF_VT = (OFF_GT + STAGES * GT_STRIDE + 511) & ~511;
  static constexpr int OFF_BT = OFF_VT + STAGES * VT_BYTES;
  static constexpr bool TMA_BETA = OFF_BT + STAGES * 1024 + 128 + 1024 <= 232448;   // where the beta rows still fit
  static constexpr int BT_BYTES = TMA_BETA ? 1024 : 0;
  static constexpr int OFF_CTRL = OFF_BT + STAGES * BT_BYTES;
  static constexpr int SMEM_BYTES = OFF_CTRL + 128 + 1024;    // + control block + alignment slack
  static_assert(CV == 8 || CV == 16 || CV == 32, "rows of a value tile: 16 bytes or one of the swizzle widths");
  static_assert(CW == 8 || CW == 16, "a thread owns 8 or 16 value columns");
  static_assert(E % WS == 0 && (WS == 1 || ET % 2 == 0), "the slices split evenly over the chain's warpgroups");
  static_assert(TPC % 16 == 0 && TPC <= 256, "columns per chain: a multiple of 16 (MMA N)");
  static_assert(TPT % 16 == 0 && TPT <= 64, "columns per thread: a multiple of 16 (tensor-memory loads), at most 64 registers of state");
  static_assert(WS == 1 || VN_BYTES >= 2 * 64 * CW * 4, "the exchange of partial sums borrows the chain's Vn image");
};

// Byte offset of 16-byte piece k of row t in a tile of 64 rows of CV bf16 columns (V, o, W, U on their way in or out).  The pieces of
// rows of 32 and 64 bytes lie as the TMA swizzle of that width puts them, so that eight threads with a row each meet no bank twice.
// (A tile per chain, as wide as its columns allow: the copy engine spends its time per row, not per byte, and with rows of 16
// bytes the four tensors' rows were most of its work.)
template <int CV>
__device__ __forceinline__ int tile_piece(int t, int k) {
  return t * (CV * 2) + ((CV == 8 ? k : CV == 16 ? (k ^ ((t >> 2) & 1)) : (k ^ ((t >> 1) & 3))) << 4);
}

struct FwdCtrl {
  uint64_t bar_load[2];
  uint64_t bar_mma[4];
  uint32_t released[2];      // chains that have finished with the stage (counts up forever; a multiple of NCH = all)
  uint32_t tmem_base;
  int abort;
};

template <int E, int CW, int NCH, int WS, int WV, int STAGES, int MINB, bool PACKED, bool SAVE>
__global__ void __launch_bounds__(NCH * WS * WV * 128, MINB)
fwd_kernel(const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_beta,
           const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q,
           const __grid_constant__ CUtensorMap map_o, const __grid_constant__ CUtensorMap map_w,
           const __grid_constant__ CUtensorMap map_u, FwdParams p) {
  using C = FwdCfg<E, CW, NCH, WS, WV, STAGES>;
  constexpr int WPC = C::WPC, CV = C::CV, TPC = C::TPC, VC = C::VC, ET = C::ET, TPT = C::TPT, CT = C::CHAIN_THREADS;
  // Roles inside a chain: its key-row warps (0, 1) have the longer epilogues (gate factors r_e, the operand images of W
  // and of r_e U), so the query-row warps take the extra work: warp 2 issues the MMAs and waits for them, warp 3
  // hands stages back and issues the loads and stores.  (Every copy operation costs its warp some sixty cycles, whatever its size,
  // and the chain waits for its last warp: few and large ones.  Not on the warp that issues the MMAs: 15 % slower.)
  constexpr int ISSUE_WARP = 2, COPY_WARP = 3;
  const bool beta_tma = C::TMA_BETA && p.beta_tma;
  constexpr bool LATE_R = E >= 12;                   // read r_e after the epilogue of (1) (register pressure at many slices)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  FwdCtrl& ctrl = *reinterpret_cast<FwdCtrl*>(smem + C::OFF_CTRL);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chain = WPC == 1 ? (warp >> 2) : (warp >> 2) / WPC;   // WPC warpgroups form a chain
  const int sw = WS == 1 ? 0 : (warp >> 2) % WS;    // which share of the chain's slices this warpgroup owns
  const int wv = WV == 1 ? 0 : (warp >> 2) % WPC / WS;   // which share of its value columns
  const int e0 = sw * ET;                           // first slice of this thread
  const int col0 = wv * (E * CW) + sw * TPT;        // its first column among the chain's E*CV
  const int row = (warp & 3) * 32 + lane;           // tensor-memory lane = operand row
  const bool krow = row < 64;                       // rows 0..63 work on K rows (W, U, Vn), 64..127 on Q rows (o)
  const int t = row & 63;
  uint8_t* s_img = smem + C::OFF_S + chain * C::S_BYTES;
  uint8_t* vn_img = smem + C::OFF_VN + chain * C::VN_BYTES;
  uint8_t* bw_img = smem + C::OFF_BW + chain * C::BW_BYTES;

  // work item
  constexpr int NV = HEAD / VC;
  const int vb = blockIdx.x % NV, h = (blockIdx.x / NV) % p.H, seq_rank = blockIdx.x / (NV * p.H);
  int b = seq_rank, first = 0, count = p.NC, seq = seq_rank;
  if constexpr (PACKED) {
    const int doc = p.cmap[2 * p.NC + seq_rank];    // longest documents first
    if (doc < 0 || doc >= p.n_seq) return;
    b = 0;
    seq = doc;
    first = p.offsets[doc];
    count = p.offsets[doc + 1] - first;
    if (first < 0 || count <= 0 || first + count > p.NC) return;
  }
  const int v0c = vb * VC + chain * CV;             // first value column of this chain in the head
  const int v0g = v0c + wv * CW;                    // ... of this thread

  if (tid == 0) {
    mbar_init(&ctrl.bar_load[0], 1);
    mbar_init(&ctrl.bar_load[1], 1);
    for (int c = 0; c < 4; ++c) mbar_init(&ctrl.bar_mma[c], 1);
    mbar_fence_init();
    ctrl.released[0] = ctrl.released[1] = 0;
    ctrl.abort = 0;
  }
  if (warp == 0) { tmem_alloc(&ctrl.tmem_base, C::TMEM_COLS); tmem_relinquish(); }
  // state: zero, or the caller's initial state (f32 [seq][H][E][128 d][128 v])
  float S[TPT];
  if (p.s_in != nullptr) {
    const float* src = p.s_in + ((static_cast<int64_t>(seq) * p.H + h) * E + e0) * (HEAD * HEAD) + row * HEAD + v0g;
#pragma unroll
    for (int e = 0; e < ET; ++e)
#pragma unroll
      for (int c = 0; c < CW; c += 4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(src + e * (HEAD * HEAD) + c));
        S[e * CW + c] = x.x; S[e * CW + c + 1] = x.y; S[e * CW + c + 2] = x.z; S[e * CW + c + 3] = x.w;
      }
  } else {
#pragma unroll
    for (int j = 0; j < TPT; ++j) S[j] = 0.f;
  }
  // A chain of eight columns uses the first block of the (2) operand only.  The second starts as zeros and holds W on its way out; its
  // products land in columns that nobody reads.
  for (int i = (tid & (CT - 1)); i < C::BW_BYTES / 16; i += CT) reinterpret_cast<uint4*>(bw_img)[i] = make_uint4(0, 0, 0, 0);

  // Sixteen of this thread's state columns -> h of a chunk, slice e as [v / 8][d][v % 8].  A warp's 16-byte stores cover 512
  // contiguous bytes, and the threads store: the copy engine writes 32 bytes a cycle, which for the state alone (E * 8 KB per 32
  // value columns and chunk) was a third of the chunk, with o, W and U and the next loads queued behind it.  us, copies -> stores:
  // 8192 items E8 850 -> 760; 4096 items E4 250 -> 208, E2 201 -> 153, E1 187 -> 134.
  auto save_state = [&](int64_t item, int j0, const uint32_t* w) {
    uint8_t* dst = reinterpret_cast<uint8_t*>(p.h) + (item * E + e0) * 32768 + (v0g >> 3) * 2048 + row * 16;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<uint4*>(dst + (j0 + 8 * j) / CW * 32768 + (j0 + 8 * j) % CW / 8 * 2048) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
  };
  {
    const uint32_t base = smem_u32(s_img) + (row >> 3) * 128 + (row & 7) * 16;
#pragma unroll
    for (int j0 = 0; j0 < TPT; j0 += 16) {
      uint32_t packed[8];
#pragma unroll
      for (int j = 0; j < 16; j += 2) packed[j / 2] = pack_bf16(S[j0 + j], S[j0 + j + 1]);
      st_shared_v4(base + ((col0 + j0) >> 3) * 2048, packed[0], packed[1], packed[2], packed[3]);
      st_shared_v4(base + ((col0 + j0 + 8) >> 3) * 2048, packed[4], packed[5], packed[6], packed[7]);
      if (SAVE && p.h != nullptr) save_state((static_cast<int64_t>(b) * p.NC + first) * p.H + h, j0, packed);
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctrl.tmem_base, 0);
  const int cwarp_u = __shfl_sync(0xffffffffu, warp & (CT / 32 - 1), 0);   // warp index inside the chain as a warp-uniform value
  const uint32_t tmem_c = tmem + chain * C::TW;                  // this chain's columns: [0, TPC) R / dS, [TPC, TPC+UW) U / Oi
  const uint32_t tmem_row = tmem_c + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  WaitCtl ctl{&ctrl.abort, p.status};

  auto chunk_info = [&](int i, int& t0, int& rows) {
    const int n = first + i;
    t0 = n * CHUNK;
    rows = CHUNK;
    if constexpr (!PACKED) return;                  // dense rows hold whole chunks
    t0 = p.cmap[n];
    rows = p.cmap[p.NC + n];
    if (t0 < 0 || rows < 0 || rows > CHUNK || t0 + rows > p.T) {
      atomicCAS(p.status, DEV_OK, DEV_BAD_CHUNK_MAP);
      t0 = 0; rows = 0;
    }
  };
  auto issue_loads = [&](int i) {                   // one thread: K/Q tiles and the [A;PmA] image of local chunk i
    int t0, rows;
    chunk_info(i, t0, rows);
    const int st = i % STAGES;
    uint8_t* kq = smem + C::OFF_KQ + st * C::KQ_BYTES;
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    mbar_expect_tx(&ctrl.bar_load[st], C::KQ_BYTES + C::AP_BYTES + C::GT_BYTES + C::VT_BYTES + (beta_tma ? C::BT_BYTES : 0));
#pragma unroll
    for (int c = 0; c < NCH; ++c)
      tma_load_4d(smem + C::OFF_VT + st * C::VT_BYTES + c * C::VBOX_BYTES, &map_v, &ctrl.bar_load[st], vb * VC + c * CV, h, t0, b);
    if (beta_tma) tma_load_4d(smem + C::OFF_BT + st * C::BT_BYTES, &map_beta, &ctrl.bar_load[st], 0, h >> 2, t0, b);
    bulk_load(smem + C::OFF_GT + st * C::GT_STRIDE, p.gc + item * gate_item_floats(E) + 64 * E, C::GT_BYTES, &ctrl.bar_load[st]);
    tma_load_4d(kq, &map_k, &ctrl.bar_load[st], 0, h, t0, b);
    tma_load_4d(kq + 8192, &map_q, &ctrl.bar_load[st], 0, h, t0, b);
    tma_load_4d(kq + 16384, &map_k, &ctrl.bar_load[st], 64, h, t0, b);
    tma_load_4d(kq + 24576, &map_q, &ctrl.bar_load[st], 64, h, t0, b);
    bulk_load(smem + C::OFF_AP + st * C::AP_BYTES, p.AP + item * (128 * 64), C::AP_BYTES, &ctrl.bar_load[st]);
  };
  // The lines of a later chunk -> L2: tiles, images and gate factors by the key-row threads of the CTAs that share them, a part each;
  // one thread a line.  (A copy-engine prefetch of a tile occupies the engine like the load itself.)
  auto prefetch_chunk = [&](int i) {
    if (!krow) return;
    int t0, rows;
    chunk_info(i, t0, rows);
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    const int64_t tok = static_cast<int64_t>(b) * p.TS + t0;
    const int last = max(rows, 1) - 1;
    constexpr int LINES = 256 + 128 + (C::GT_BYTES + 127) / 128, SHARE = (LINES + NV - 1) / NV;
    static_assert(SHARE <= NCH * WPC * 64, "one line per key-row thread");
    const int idx = (warp >> 2) * 64 + t, line = vb * SHARE + idx;
    if (idx < SHARE && line < LINES) {
      const char* ptr;
      if (line < 256) {
        ptr = reinterpret_cast<const char*>(line < 128 ? p.k : p.q) + ((tok + min((line >> 1) & 63, last)) * p.H + h) * (HEAD * 2) + (line & 1) * 128;
      } else if (line < 384) {
        ptr = reinterpret_cast<const char*>(p.AP + item * (128 * 64)) + (line - 256) * 128;
      } else {
        ptr = reinterpret_cast<const char*>(p.gc + item * gate_item_floats(E) + 64 * E) + (line - 384) * 128;
      }
      prefetch_l2(ptr);
    }
    if (!beta_tma && chain == 0 && sw == 0 && wv == 0) prefetch_l2(p.beta + (tok + min(t, last)) * p.H + h);
  };
  // CW packed bf16 (CW/2 words) of one row -> 8-column blocks `stride` bytes apart
  auto store_packed = [&](uint32_t dst, uint32_t stride, const uint32_t* w) {
#pragma unroll
    for (int c = 0; c < CW / 2; c += 4) st_shared_v4(dst + (c >> 2) * stride, w[c], w[c + 1], w[c + 2], w[c + 3]);
  };

  if (tid == 0) {
    issue_loads(0);
    if (STAGES == 2 && count > 1) issue_loads(1);
  }
  uint32_t mma_phase = 0;
  int t0_next = 0, rows_next = CHUNK;               // packed rows: the chunk's place is looked up a chunk ahead
  if constexpr (PACKED) chunk_info(0, t0_next, rows_next);

  for (int i = 0; i < count; ++i) {
    const int st = i % STAGES;
    uint8_t* kq = smem + C::OFF_KQ + st * C::KQ_BYTES;
    uint8_t* ap = smem + C::OFF_AP + st * C::AP_BYTES;

    // ---- (1) R = [K;Q] S --------------------------------------------------------------------------------------
    // Every thread reads rows of the stage (gates, value row, beta) under the MMA, so every warp waits for the loads itself.
    // (The MMA completions below are waited for by the chain's issuing warp only: the others sleep in the chain's hardware
    // barrier, where they take no issue slots from the chains that are in an epilogue at that moment.  That warp parks: us, polled ->
    // parked, 4096 items E12 651 -> 636, E16 818 -> 813, 8192 items E8 745 -> 741.  The loads, which are there as a rule, are polled:
    // parked E16 852.)
    mbar_wait(&ctrl.bar_load[st], (i / STAGES) & 1, ctl, DEV_TIMEOUT_LOAD);
    if (cwarp_u == ISSUE_WARP && elect_one()) {
      tc_fence_after();
      const uint64_t da = make_desc(smem_u32(kq), 16, 1024, LAYOUT_SW128);
      const uint64_t db = make_desc(smem_u32(s_img), 128, 2048, LAYOUT_PLAIN);
      constexpr uint32_t idesc = make_idesc(128, TPC, 0, 1);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16(tmem_c, desc_advance(da, (kk >> 2) * 16384 + (kk & 3) * 32), desc_advance(db, kk * 256), idesc, kk > 0);
      umma_commit(&ctrl.bar_mma[chain]);
    }
    __syncwarp();                                    // the other lanes must not run ahead into a spin wait
    const int t0 = PACKED ? t0_next : (first + i) * CHUNK, rows = PACKED ? rows_next : CHUNK;
    const int64_t item = (static_cast<int64_t>(b) * p.NC + first + i) * p.H + h;
    const int64_t tok = static_cast<int64_t>(b) * p.TS + t0;
    const bool live = t < rows;
    const bool o_tile = rows == CHUNK;               // a chunk cut short by a document end cannot leave as a tile
    // The chain finished with the previous chunk's tiles when its third MMA group completed.  It says so now, under this
    // MMA, where its warps have time to spare; the last chain to say so refills that stage with the chunk STAGES ahead.
    // (o left from the stage's value rows, W and U from the place of beta*W: the stores must have read them.)
    if (cwarp_u == COPY_WARP && i > 0 && elect_one()) {
      bulk_wait_group_read();
      const uint32_t done = atomicAdd(&ctrl.released[(i - 1) % STAGES], 1u) + 1u;
      if (done % NCH == 0 && i - 1 + STAGES < count) issue_loads(i - 1 + STAGES);
    }
    __syncwarp();
    // Under the MMA: this row's gate factors, value row and beta from the stage.
    const float* gf = reinterpret_cast<const float*>(smem + C::OFF_GT + st * C::GT_STRIDE);
    float ga[ET];                                    // this thread's slices.  K rows: a_e = k2 exp(gc); Q rows: c_e = scale q2 exp(gc)
    float gr[ET];                                    // K rows: r_e = k2 exp(gL - gc)
    float bt = 0.f;
    // This chain's value rows in the stage (64 rows x CW columns per share): read here, then the place from which W and, after it, o
    // leave.  One 16-byte store per row into the tile and one TMA store replace a store per thread into a row of its own,
    // which cost 32 wavefronts of the L1 data path per warp (768 of about 4900 per chunk at E = 8).
    uint8_t* vbox = smem + C::OFF_VT + st * C::VT_BYTES + chain * C::VBOX_BYTES;
    auto put_row = [&](uint8_t* tile, const uint32_t* w) {   // this thread's columns of row t of a tile
#pragma unroll
      for (int c = 0; c < CW / 8; ++c)
        st_shared_v4(smem_u32(tile) + tile_piece<CV>(t, wv * (CW / 8) + c), w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
    };
    uint32_t vraw[CW / 2];
    if constexpr (WS > 1) {
#pragma unroll
      for (int c = 0; c < CW / 2; ++c) vraw[c] = 0u;
    }
    {
      // (at eight slices the selects of the ordered form cost the two chains more than its bank conflicts: 570 -> 622 us, 8192 items
      // without saved state; at sixteen it takes 1662 -> 1585 us, packed)
      lds_row<E, ET, E == 16>(gf + (krow ? 0 : C::GF_C), t, e0, ga);
      if (krow) {
        if constexpr (!LATE_R) lds_row<E, ET, E == 16>(gf + C::GF_R, t, e0, gr);
        if (sw == 0) {                               // the warpgroup that completes W: beta and the value row
          if (beta_tma) {
            bt = reinterpret_cast<const float*>(smem + C::OFF_BT + st * C::BT_BYTES)[t * 4 + (h & 3)];
          } else {
            bt = __ldg(p.beta + (tok + min(t, max(rows, 1) - 1)) * p.H + h);
          }
#pragma unroll
          for (int c = 0; c < CW / 2; c += 4)
            asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(vraw[c]), "=r"(vraw[c + 1]), "=r"(vraw[c + 2]), "=r"(vraw[c + 3]) : "r"(smem_u32(vbox) + tile_piece<CV>(t, wv * (CW / 8) + c / 4)));
        }
        if (!live) bt = 0.f;
      } else {
#pragma unroll
        for (int e = 0; e < ET; ++e) gr[e] = 0.f;
      }
      if (i + 2 < count) prefetch_chunk(i + 2);
    }
    if (cwarp_u == ISSUE_WARP) mbar_wait_parked(&ctrl.bar_mma[chain], mma_phase & 1, ctl, DEV_TIMEOUT_MMA);
    chain_sync<CT>(chain);
    ++mma_phase;
    tc_fence_after();

    float acc[CW];                                   // K rows: W (starts from V); Q rows: Oq
#pragma unroll
    for (int c = 0; c < CW; ++c) acc[c] = (krow && live && sw == 0) ? ((c & 1) ? bf16_hi(vraw[c >> 1]) : bf16_lo(vraw[c >> 1])) : 0.f;
    {
      // sixteen columns at a time, the next piece travelling while this one is used
      float rr[2][16];
      tmem_ld<16>(tmem_row + col0, rr[0]);
#pragma unroll
      for (int pc = 0; pc < TPT / 16; ++pc) {
        tmem_wait_ld();
        if (pc + 1 < TPT / 16) tmem_ld<16>(tmem_row + col0 + (pc + 1) * 16, rr[(pc + 1) & 1]);
        const float* rp = rr[pc & 1];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const int e = (pc * 16 + j) / CW, c = (pc * 16 + j) % CW;
          fma_pair(acc[c], acc[c + 1], krow ? -ga[e] : ga[e], rp[j], rp[j + 1]);
        }
      }
    }
    if constexpr (WS > 1) {
      // The sums over the slices are split over the chain's warpgroups: the first one completes W (K rows), the last one
      // the state part of o (Q rows); the others hand their partial sums over through shared memory (the chain's Vn image
      // is free between the last MMA of the previous chunk and the epilogue of (2)).
      static_assert(WS == 2 && WV == 1, "the exchange below is written for two warpgroups per chain");
      float* red = reinterpret_cast<float*>(vn_img) + (krow ? 0 : 64 * CW) + t * CW;
      const bool owner = krow ? (sw == 0) : (sw == WS - 1);
      if (!owner) {
#pragma unroll
        for (int c = 0; c < CW; c += 4) *reinterpret_cast<float4*>(red + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      }
      chain_sync<CT>(chain);
      if (owner) {
#pragma unroll
        for (int c = 0; c < CW; c += 4) {
          const float4 x = *reinterpret_cast<const float4*>(red + c);
          acc[c] += x.x; acc[c + 1] += x.y; acc[c + 2] += x.z; acc[c + 3] += x.w;
        }
      }
    }
    if (krow && sw == 0) {
      // beta*W -> operand image (i = s, j = v); W -> the value tile, to be saved (bf16)
      uint32_t w[CW / 2];
#pragma unroll
      for (int c = 0; c < CW; c += 2) w[c >> 1] = pack_bf16(bt * acc[c], bt * acc[c + 1]);
      store_packed(smem_u32(bw_img) + wv * (CW * 128) + t * 16, 1024, w);
      if (SAVE && p.W != nullptr) {
#pragma unroll
        for (int c = 0; c < CW; c += 2) w[c >> 1] = pack_bf16(acc[c], acc[c + 1]);
        put_row(C::W_OWN ? bw_img + C::WST_OFF : vbox, w);   // (the value row has been read by the same thread)
      }
    }
    fence_async_smem();
    tc_fence_before();
    chain_sync<CT>(chain);

    // ---- (2) [U;Oi] = [A;PmA] (beta W) ------------------------------------------------------------------------
    if (cwarp_u == ISSUE_WARP && elect_one()) {
      tc_fence_after();
      const uint64_t da = make_desc(smem_u32(ap), 2048, 128, LAYOUT_PLAIN);
      const uint64_t db = make_desc(smem_u32(bw_img), 128, 1024, LAYOUT_PLAIN);
      constexpr uint32_t idesc = make_idesc(128, C::UW, 0, 1);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16(tmem_c + TPC, desc_advance(da, kk * 4096), desc_advance(db, kk * 256), idesc, kk > 0);
      umma_commit(&ctrl.bar_mma[chain]);
    }
    __syncwarp();
    if (SAVE && p.W != nullptr && cwarp_u == COPY_WARP && elect_one()) {
      tma_store_4d(&map_w, C::W_OWN ? bw_img + C::WST_OFF : vbox, v0c, 0, static_cast<int>(item) * 64, 0);
      if constexpr (!C::W_OWN) {                     // o takes its place after this product
        bulk_commit_group();
        bulk_wait_group_read();
      }
    }
    __syncwarp();
    if (PACKED && i + 1 < count) chunk_info(i + 1, t0_next, rows_next);
    if constexpr (LATE_R) {                          // r_e only now, from the stage: sixteen registers fewer are live
      if (krow) lds_row<E, ET, E == 16>(gf + C::GF_R, t, e0, gr);   // through the epilogue of (1)
    }
    if (cwarp_u == ISSUE_WARP) mbar_wait_parked(&ctrl.bar_mma[chain], mma_phase & 1, ctl, DEV_TIMEOUT_MMA);
    chain_sync<CT>(chain);
    ++mma_phase;
    tc_fence_after();
    {
      float u[CW];
      tmem_ld<CW>(tmem_row + TPC + wv * CW, u);
      tmem_wait_ld();
      if (krow) {
        // U leaves as bf16 (the backward reads it back in that form); Vn_e = r_e * U is formed from the same packed row,
        // two products per instruction, and goes into the operand image (i = t, j = n'), this thread's slices
        uint32_t uw[CW / 2];
#pragma unroll
        for (int c = 0; c < CW; c += 2) uw[c >> 1] = pack_bf16(u[c], u[c + 1]);
        // (the operand beta*W has been read: its place takes U, which leaves from there by TMA)
        if (SAVE && p.U != nullptr && sw == 0) put_row(bw_img, uw);
        const uint32_t base = smem_u32(vn_img) + (t >> 3) * 128 + (t & 7) * 16;
#pragma unroll
        for (int e = 0; e < ET; ++e) {
          const uint32_t rr = pack_bf16(gr[e], gr[e]);
          const int n0 = col0 + e * CW;
#pragma unroll
          for (int c = 0; c < CW / 2; c += 4)
            st_shared_v4(base + ((n0 + 2 * c) >> 3) * 1024, mul_bf16x2(uw[c], rr), mul_bf16x2(uw[c + 1], rr), mul_bf16x2(uw[c + 2], rr),
                         mul_bf16x2(uw[c + 3], rr));
        }
      } else if (live && sw == WS - 1) {
        uint32_t ow[CW / 2];
#pragma unroll
        for (int c = 0; c < CW; c += 2) ow[c >> 1] = pack_bf16(acc[c] + u[c], acc[c + 1] + u[c + 1]);
        if (o_tile) {
          put_row(vbox, ow);
        } else {
          __nv_bfloat16* dst = p.o + ((tok + t) * p.H + h) * HEAD + v0g;
#pragma unroll
          for (int c = 0; c < CW / 2; c += 4) *reinterpret_cast<uint4*>(dst + 2 * c) = make_uint4(ow[c], ow[c + 1], ow[c + 2], ow[c + 3]);
        }
      }
    }
    fence_async_smem();
    tc_fence_before();
    chain_sync<CT>(chain);

    // ---- (3) dS = K^T Vn, S <- d S + dS -----------------------------------------------------------------------
    if (cwarp_u == ISSUE_WARP && elect_one()) {
      tc_fence_after();
      const uint64_t da = make_desc(smem_u32(kq), 16384, 1024, LAYOUT_SW128);
      const uint64_t db = make_desc(smem_u32(vn_img), 128, 1024, LAYOUT_PLAIN);
      constexpr uint32_t idesc = make_idesc(128, TPC, 1, 1);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16(tmem_c, desc_advance(da, kk * 2048), desc_advance(db, kk * 256), idesc, kk > 0);
      umma_commit(&ctrl.bar_mma[chain]);
    }
    __syncwarp();
    if (cwarp_u == COPY_WARP && elect_one()) {
      if (o_tile) tma_store_4d(&map_o, vbox, v0c, h, t0, b);
      if (SAVE && p.U != nullptr) tma_store_4d(&map_u, bw_img, v0c, 0, static_cast<int>(item) * 64, 0);
      bulk_commit_group();
    }
    __syncwarp();
    if (cwarp_u == ISSUE_WARP) mbar_wait_parked(&ctrl.bar_mma[chain], mma_phase & 1, ctl, DEV_TIMEOUT_MMA);
    chain_sync<CT>(chain);
    ++mma_phase;
    tc_fence_after();
    {
      float dch[ET];                                 // exp(gL) of this thread's slices
      lds_part<ET>(gf + C::GF_D + e0, dch);
      const uint32_t base = smem_u32(s_img) + (row >> 3) * 128 + (row & 7) * 16;
      float ds[2][16];
      tmem_ld<16>(tmem_row + col0, ds[0]);
#pragma unroll
      for (int pc = 0; pc < TPT / 16; ++pc) {
        const int j0 = pc * 16;
        tmem_wait_ld();
        if (pc + 1 < TPT / 16) tmem_ld<16>(tmem_row + col0 + j0 + 16, ds[(pc + 1) & 1]);
        const float* dp = ds[pc & 1];
        uint32_t packed[8];
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          scale_add_pair(S[j0 + j], S[j0 + j + 1], dch[(j0 + j) / CW], dp[j], dp[j + 1]);
          packed[j / 2] = pack_bf16(S[j0 + j], S[j0 + j + 1]);
        }
        // operand image (i = d, j = n') for the next chunk's (1)
        st_shared_v4(base + ((col0 + j0) >> 3) * 2048, packed[0], packed[1], packed[2], packed[3]);
        st_shared_v4(base + ((col0 + j0 + 8) >> 3) * 2048, packed[4], packed[5], packed[6], packed[7]);
        if (SAVE && p.h != nullptr && i + 1 < count) save_state(item + p.H, j0, packed);
      }
    }
    fence_async_smem();
    tc_fence_before();
    chain_sync<CT>(chain);
  }
  if (cwarp_u == COPY_WARP && elect_one()) bulk_wait_group();   // the last stores read shared memory of this CTA
  __syncwarp();
  // final state for the caller (f32, same form as the initial state)
  if (p.s_out != nullptr) {
    float* dst = p.s_out + ((static_cast<int64_t>(seq) * p.H + h) * E + e0) * (HEAD * HEAD) + row * HEAD + v0g;
#pragma unroll
    for (int e = 0; e < ET; ++e)
#pragma unroll
      for (int c = 0; c < CW; c += 4)
        *reinterpret_cast<float4*>(dst + e * (HEAD * HEAD) + c) = make_float4(S[e * CW + c], S[e * CW + c + 1], S[e * CW + c + 2], S[e * CW + c + 3]);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, C::TMEM_COLS);
}

}  // namespace tgdn

using namespace tgdn;

template <int E, int CW, int NCH, int WS, int WV, int STAGES, int MINB, bool PACKED, bool SAVE>
static int launch_fwd_rows(const CUtensorMap& mk, const CUtensorMap& mq, const void* v, const FwdParams& p, cudaStream_t s) {
  int rc;
  using C = FwdCfg<E, CW, NCH, WS, WV, STAGES>;
  static_assert(MINB == 1 || C::SMEM_BYTES <= 115712, "two CTAs per SM need at most 113 KB each");
  static_assert(C::SMEM_BYTES <= 232448, "shared memory budget of one CTA exceeded");
  static_assert(MINB * C::TMEM_COLS <= 512, "tensor memory budget of one SM exceeded");
  static bool configured[64] = {};
  if ((rc = tgdn_dynamic_smem(reinterpret_cast<const void*>(fwd_kernel<E, CW, NCH, WS, WV, STAGES, MINB, PACKED, SAVE>), C::SMEM_BYTES, configured)))
    return rc;
  CUtensorMap mv, mo, mb = mk, mw = mk, mu = mk;    // placeholders where a tensor is not loaded or stored by TMA
  if ((rc = tgdn_make_token_map(&mv, v, p.B, p.T, p.H, C::CV, 64, C::CV > 8, p.TS))) return rc;
  if ((rc = tgdn_make_token_map(&mo, p.o, p.B, p.T, p.H, C::CV, 64, C::CV > 8, p.TS))) return rc;
  if (C::TMA_BETA && p.beta_tma) {
    if ((rc = tgdn_make_gate_map(&mb, p.beta, p.B, p.T, p.H / 4, 4, p.TS))) return rc;    // (B, T, H) read as (B, T, H/4, 4)
  }
  // chunk-layout tensors are plain (rows, 128) matrices: one batch row, one head
  const int64_t crows = static_cast<int64_t>(p.B) * p.NC * p.H * 64;
  if ((p.W != nullptr || p.U != nullptr) && crows > 0x7fffffffLL) return TGDN_ERR_SHAPE;
  if (p.W != nullptr && (rc = tgdn_make_token_map(&mw, p.W, 1, static_cast<int>(crows), 1, C::CV, 64, C::CV > 8))) return rc;
  if (p.U != nullptr && (rc = tgdn_make_token_map(&mu, p.U, 1, static_cast<int>(crows), 1, C::CV, 64, C::CV > 8))) return rc;
  const int grid = p.n_seq * p.H * (HEAD / C::VC);
  fwd_kernel<E, CW, NCH, WS, WV, STAGES, MINB, PACKED, SAVE><<<grid, C::THREADS, C::SMEM_BYTES, s>>>(mv, mb, mk, mq, mo, mw, mu, p);
  return tgdn_cuda_error(cudaGetLastError());
}


template <int E, int CW, int NCH, int WS, int WV, int STAGES, int MINB, bool SAVE>
static int launch_fwd(const CUtensorMap& mk, const CUtensorMap& mq, const void* v, const FwdParams& p, cudaStream_t s) {
  return p.cmap != nullptr ? launch_fwd_rows<E, CW, NCH, WS, WV, STAGES, MINB, true, SAVE>(mk, mq, v, p, s)
                           : launch_fwd_rows<E, CW, NCH, WS, WV, STAGES, MINB, false, SAVE>(mk, mq, v, p, s);
}

int tgdn_fwd_rows(const void* q, const void* k, const void* v, const float* k2, const float* q2, const float* beta, const float* gc,
                  const void* AP, float scale, const int32_t* doc_offsets, const int32_t* chunk_map, int n_docs, int B, int T, int H,
                  int E, int NC, int row_tokens, void* o, void* W, void* U, void* h, const float* state_in, float* state_out,
                  void* stream) {
  if (!q || !k || !v || !k2 || !q2 || !beta || !gc || !AP || !o) return TGDN_ERR_NULL;
  const bool packed = chunk_map != nullptr;
  if (packed && (!doc_offsets || n_docs < 1)) return TGDN_ERR_NULL;
  int rc = tgdn_check_core_shape(B, T, H, E, NC, packed, row_tokens);
  if (rc) return rc;
  if ((reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(AP) |
       reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(U) | reinterpret_cast<uintptr_t>(h) |
       reinterpret_cast<uintptr_t>(k2) | reinterpret_cast<uintptr_t>(q2) | reinterpret_cast<uintptr_t>(gc) |
       reinterpret_cast<uintptr_t>(state_in) | reinterpret_cast<uintptr_t>(state_out)) & 15)
    return TGDN_ERR_ALIGN;
  CUtensorMap mk, mq;
  if ((rc = tgdn_make_token_map(&mk, k, B, T, H, 64, 64, 1, row_tokens))) return rc;
  if ((rc = tgdn_make_token_map(&mq, q, B, T, H, 64, 64, 1, row_tokens))) return rc;
  FwdParams p{static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k), k2, q2, beta, gc, static_cast<const __nv_bfloat16*>(AP),
              static_cast<__nv_bfloat16*>(o), static_cast<__nv_bfloat16*>(W), static_cast<__nv_bfloat16*>(U),
              static_cast<__nv_bfloat16*>(h), state_in, state_out, doc_offsets, chunk_map, B, T, H, NC,
              packed ? n_docs : B, row_tokens, scale, tgdn_status_word(),
              (H % 4 == 0 && (reinterpret_cast<uintptr_t>(beta) & 15) == 0) ? 1 : 0};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // Width of the value block, up to four slices.  One CTA per SM: the grid runs in whole waves.  A CTA of 64 columns takes 1.17 (one
  // slice), 1.12 (two) and 1.01 (four) times as long per chunk as one of 32, so it wins whenever it saves a wave (it then saves at
  // least a third of them); a grid that fills one wave either way keeps the narrow one.
  const long long sms = tgdn_sm_count(), seqs = static_cast<long long>(p.n_seq) * p.H;
  const long long narrow = (seqs * 4 + sms - 1) / sms, wide = (seqs * 2 + sms - 1) / sms;
  // Chains: two of two warpgroups (WV = 2, twice the columns per MMA) do better than four of one wherever the state is not saved,
  // and at one and two slices; at four and eight slices the state's stores want the four chains' finer interleaving.
  // us, four chains -> two: 8192 items E8 forward alone 618 -> 573, with saved state 764 -> 780; 4096 items E4 176 -> 160, 209 -> 220,
  // E2 135 -> 129, 156 -> 152, E1 127 -> 111, 152 -> 133.
  const bool save = W != nullptr || U != nullptr || h != nullptr;
#define TGDN_FWD(E, CW, NCH, WS, WV) \
  return save ? launch_fwd<E, CW, NCH, WS, WV, 2, 1, true>(mk, mq, v, p, s) : launch_fwd<E, CW, NCH, WS, WV, 2, 1, false>(mk, mq, v, p, s)
#define TGDN_FWD_BY_SAVE(E, CW) \
  return save ? launch_fwd<E, CW, 4, 1, 1, 2, 1, true>(mk, mq, v, p, s) : launch_fwd<E, CW, 2, 1, 2, 2, 1, false>(mk, mq, v, p, s)
  switch (E) {
    case 1:      // (its narrow block is two chains of 16 columns)
      if (wide < narrow) TGDN_FWD(1, 16, 2, 1, 2);
      TGDN_FWD(1, 16, 2, 1, 1);
    case 2:
      if (wide < narrow) TGDN_FWD(2, 16, 2, 1, 2);
      TGDN_FWD(2, 8, 2, 1, 2);
    case 4:
      if (wide < narrow) TGDN_FWD_BY_SAVE(4, 16);
      TGDN_FWD_BY_SAVE(4, 8);
    case 8: TGDN_FWD_BY_SAVE(8, 8);
    case 12: TGDN_FWD(12, 8, 2, 2, 1);
    case 16: TGDN_FWD(16, 8, 2, 2, 1);
    default: return TGDN_ERR_SHAPE;
  }
#undef TGDN_FWD
#undef TGDN_FWD_BY_SAVE
}

extern "C" int tgdn_fwd_state(const void* q, const void* k, const void* v, const float* k2, const float* q2,
                              const float* beta, const float* gc, const void* AP, float scale, const int32_t* doc_offsets,
                              const int32_t* chunk_map, int n_docs, int B, int T, int H, int E, int NC, void* o, void* W,
                              void* U, void* h, const float* state_in, float* state_out, void* stream) {
  return tgdn_fwd_rows(q, k, v, k2, q2, beta, gc, AP, scale, doc_offsets, chunk_map, n_docs, B, T, H, E, NC, T, o, W, U, h,
                       state_in, state_out, stream);
}

extern "C" int tgdn_fwd(const void* q, const void* k, const void* v, const float* k2, const float* q2, const float* beta,
                        const float* gc, const void* AP, float scale, const int32_t* doc_offsets,
                        const int32_t* chunk_map, int n_docs, int B, int T, int H, int E, int NC, void* o, void* W,
                        void* U, void* h, void* stream) {
  return tgdn_fwd_state(q, k, v, k2, q2, beta, gc, AP, scale, doc_offsets, chunk_map, n_docs, B, T, H, E, NC, o, W, U, h,
                        nullptr, nullptr, stream);
}
