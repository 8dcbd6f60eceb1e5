// Width-4 causal depthwise convolution with SiLU on the leading channels, forward and backward, and the same with the layer glue
// that follows it fused in (conv -> SiLU / softplus -> l2 norms -> q, k, v, k2, q2).
//
// Replaces the reference's Triton kernels cute_triadic_gdn/ops/conv_split_act.py:20-55 (_fwd_kernel) and :58-107 (_bwd_kernel).
//
// A warp walks a run of tokens of its channels with the three rows of the window (and, backward, the last three gradients and the
// weight gradient) in registers: each row is read once and nothing is computed twice but the three rows behind the end of a
// run.  Its rows arrive by TMA in a ring of its own (RING kernels: 128 channels per warp; what the tensor maps can describe) or
// by loads asked for a batch ahead (WALKERS: everything else).  The version before staged 32-token tiles per CTA, eight rows per
// warp: eleven rows computed for eight in the backward, a CTA barrier per tile, and padded copies of every tensor where the
// channel count was not a multiple of eight.  Measured at (1, 32768, 13056), of the HBM copy rate: backward 558 -> 424 us (70 ->
// 92%), forward 302 -> 300 us (87%; two transcendental operations per element are the co-limit); at (3, 1000, 1930), padded
// copies included, forward and backward 130 -> 27 us.
// The weight gradient is accumulated in f32 per run and the runs' partials are summed in a fixed order by a second small kernel.
#include <algorithm>
#include <mutex>

#include "tgdn_common.cuh"
#include "tgdn_host.h"
#include "tgdn_kernels.h"

namespace tgdn {

constexpr int CONV_W = 4;
constexpr int CONV_TOK = 32;           // granularity of the token groups that size the scratch of the public ABI

// ---- V channels of one row: raw bf16 words and f32 pairs -----------------------------------------------------------------
// The arithmetic runs on the two-wide f32 instructions (one instruction per pair, each lane an ordinary IEEE fma).
template <int V> struct RawRow;
template <> struct RawRow<4> { uint2 w; };
template <> struct RawRow<2> { uint32_t w; };
template <> struct RawRow<1> { unsigned short w; };
template <int V> struct Pairs { float2 p[(V + 1) / 2]; };

template <int V>
__device__ __forceinline__ RawRow<V> load_raw(const __nv_bfloat16* p) {      // streamed: not kept in L1
  RawRow<V> r;
  if constexpr (V == 4)
    asm volatile("ld.global.nc.L1::no_allocate.v2.b32 {%0,%1}, [%2];" : "=r"(r.w.x), "=r"(r.w.y) : "l"(p));
  else if constexpr (V == 2)
    asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(r.w) : "l"(p));
  else
    asm volatile("ld.global.nc.L1::no_allocate.b16 %0, [%1];" : "=h"(r.w) : "l"(p));
  return r;
}
template <int V>
__device__ __forceinline__ RawRow<V> zero_raw() {
  RawRow<V> r;
  if constexpr (V == 4) r.w = make_uint2(0u, 0u); else r.w = 0;
  return r;
}
template <int V>
__device__ __forceinline__ Pairs<V> unpack(const RawRow<V>& r) {
  Pairs<V> o;
  if constexpr (V == 4) {
    o.p[0] = make_float2(bf16_lo(r.w.x), bf16_hi(r.w.x));
    o.p[1] = make_float2(bf16_lo(r.w.y), bf16_hi(r.w.y));
  } else if constexpr (V == 2) {
    o.p[0] = make_float2(bf16_lo(r.w), bf16_hi(r.w));
  } else {
    o.p[0] = make_float2(bf16_lo(r.w), 0.f);
  }
  return o;
}
template <int V>
__device__ __forceinline__ Pairs<V> zero_pairs() {
  Pairs<V> o;
#pragma unroll
  for (int i = 0; i < (V + 1) / 2; ++i) o.p[i] = make_float2(0.f, 0.f);
  return o;
}
template <int V>
__device__ __forceinline__ void store_row(__nv_bfloat16* p, const Pairs<V>& a) {
  if constexpr (V == 4)
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(a.p[0].x, a.p[0].y), pack_bf16(a.p[1].x, a.p[1].y));
  else if constexpr (V == 2)
    *reinterpret_cast<uint32_t*>(p) = pack_bf16(a.p[0].x, a.p[0].y);
  else
    *p = __float2bfloat16_rn(a.p[0].x);
}

// The four taps of V channels as pairs, and the products with the window.
template <int V> struct Taps { float2 w[(V + 1) / 2][CONV_W]; };
template <int V>
__device__ __forceinline__ Taps<V> load_taps(const __nv_bfloat16* weight, int c0, bool live) {
  float f[V][CONV_W];
#pragma unroll
  for (int c = 0; c < V; ++c) {
    const uint2 u = live ? __ldg(reinterpret_cast<const uint2*>(weight + static_cast<int64_t>(c0 + c) * CONV_W)) : make_uint2(0u, 0u);
    f[c][0] = bf16_lo(u.x); f[c][1] = bf16_hi(u.x); f[c][2] = bf16_lo(u.y); f[c][3] = bf16_hi(u.y);
  }
  Taps<V> t;
#pragma unroll
  for (int i = 0; i < (V + 1) / 2; ++i)
#pragma unroll
    for (int j = 0; j < CONV_W; ++j) t.w[i][j] = make_float2(f[2 * i][j], 2 * i + 1 < V ? f[2 * i + (V > 1 ? 1 : 0)][j] : 0.f);
  return t;
}
// The window of a walk: x[t-1], x[t-2], x[t-3].
template <int V> struct Window {
  Pairs<V> m[3];
  __device__ __forceinline__ void push(const Pairs<V>& x0) { m[2] = m[1]; m[1] = m[0]; m[0] = x0; }
  __device__ __forceinline__ float2 conv(const Taps<V>& t, const Pairs<V>& x0, int i) const {
    float2 acc = __fmul2_rn(m[2].p[i], t.w[i][0]);
    acc = __ffma2_rn(m[1].p[i], t.w[i][1], acc);
    acc = __ffma2_rn(m[0].p[i], t.w[i][2], acc);
    return __ffma2_rn(x0.p[i], t.w[i][3], acc);
  }
};

// sigmoid with the fast exponential and the fast reciprocal: relative error of a few f32 ulps
__device__ __forceinline__ float fast_sigmoid(float y) { return __fdividef(1.f, 1.f + __expf(-y)); }
__device__ __forceinline__ float silu(float y) { return y * fast_sigmoid(y); }
// SiLU' of the bf16-rounded pre-activations of a pair, for the backward, where the result is rounded to bf16 after further
// products: the sigmoid comes from one tanh.approx (absolute error about 2^-11) instead of an exponential and a reciprocal.
__device__ __forceinline__ float2 silu_grad_pair(float2 pre) {
  const uint32_t r = pack_bf16(pre.x, pre.y);
  const float2 y = make_float2(bf16_lo(r), bf16_hi(r));
  const float2 h = __fmul2_rn(y, make_float2(0.5f, 0.5f));
  float2 th;
  asm("tanh.approx.f32 %0, %1;" : "=f"(th.x) : "f"(h.x));
  asm("tanh.approx.f32 %0, %1;" : "=f"(th.y) : "f"(h.y));
  const float2 half2 = make_float2(0.5f, 0.5f), one2 = make_float2(1.f, 1.f);
  const float2 s = __ffma2_rn(half2, th, half2);
  const float2 om = __ffma2_rn(s, make_float2(-1.f, -1.f), one2);
  return __fmul2_rn(s, __ffma2_rn(y, om, one2));
}

// The document of a token, and the next one's first token.
struct DocCursor {
  const int32_t* cu;
  int n_docs, d, start, next;
  __device__ __forceinline__ void init(const int32_t* cu_, int n_docs_, int t) {
    cu = cu_; n_docs = n_docs_; d = 0; start = 0; next = 0x7fffffff;
    if (cu == nullptr) return;
    int lo = 0, hi = n_docs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(cu + mid) <= t) lo = mid; else hi = mid - 1;
    }
    d = lo;
    start = __ldg(cu + d);
    set_next();
  }
  __device__ __forceinline__ void set_next() { next = (d + 1 < n_docs) ? __ldg(cu + d + 1) : 0x7fffffff; }
  __device__ __forceinline__ void advance(int t) {       // to the document of token t, which is not before the current one
    while (t >= next) { ++d; start = next; set_next(); }
  }
};

template <int V>
__device__ __forceinline__ void open_window(Window<V>& win, const __nv_bfloat16* col, int64_t stride, int t, int doc_start, bool live) {
#pragma unroll
  for (int j = 0; j < 3; ++j) win.m[j] = (live && t - 1 - j >= doc_start) ? unpack<V>(load_raw<V>(col + (t - 1 - j) * stride)) : zero_pairs<V>();
}

// Which channels of the warp pass through SiLU: 0 none, 1 all, 2 some.
__device__ __forceinline__ int act_kind(int c0, int channels, bool live, int act_channels) {
  if (__all_sync(0xffffffffu, !live || c0 + channels <= act_channels)) return 1;
  if (__all_sync(0xffffffffu, !live || c0 >= act_channels)) return 0;
  return 2;
}

// ---- per-warp TMA ring ---------------------------------------------------------------------------------------------------
// A warp that walks 128 channels (V = 4) of a run of tokens has its rows arrive by TMA, eight at a time, in a ring of its own:
// nothing couples the warps of a CTA, rows are read from shared memory at constant offsets (no address arithmetic per row),
// and three to six tiles per warp are in flight.  Rows past the end of a batch row arrive as zeros (the tensor map's fill).
constexpr int RING_ROWS = 8;
constexpr int RING_TILE = RING_ROWS * 256;       // bytes: 8 rows x 128 channels
constexpr int RING_WARPS = 4;                    // warps per CTA
constexpr int RING_FWD_STAGES = 6, RING_BWD_STAGES = 3;      // 12 KB per warp either way

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// TENSORS tiles per stage: x, and in the backward the gradient rows.
template <int TENSORS, int STAGES>
struct Ring {
  static constexpr int STAGE_BYTES = TENSORS * RING_TILE;
  static constexpr int WARP_BYTES = STAGES * STAGE_BYTES;
  uint8_t* buf;                                  // this warp's stages
  uint64_t* full;                                // and their barriers
  int k;                                         // tiles taken so far
  __device__ __forceinline__ void init(uint8_t* smem, uint64_t* bars) {
    const int warp = threadIdx.x >> 5;
    buf = smem + warp * WARP_BYTES;
    full = bars + warp * STAGES;
    k = 0;
    if ((threadIdx.x & 31) == 0) {
      for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
      mbar_fence_init();
    }
    __syncwarp();
  }
  __device__ __forceinline__ uint8_t* stage(int tile) const { return buf + tile % STAGES * STAGE_BYTES; }
  // issue(tile, stage, barrier): one lane sends off the loads of a tile
  template <typename F>
  __device__ __forceinline__ void open(int tiles, F issue) {
    if (elect_one()) {
      for (int i = 0; i < STAGES && i < tiles; ++i) {
        mbar_expect_tx(&full[i], STAGE_BYTES);
        issue(i, stage(i), &full[i]);
      }
    }
    __syncwarp();
  }
  __device__ __forceinline__ const uint8_t* wait(const WaitCtl& ctl) const {
    mbar_wait(&full[k % STAGES], (k / STAGES) & 1, ctl, DEV_TIMEOUT_LOAD);
    return stage(k) + (threadIdx.x & 31) * 8;    // this lane's four channels of row 0
  }
  template <typename F>
  __device__ __forceinline__ void release(int tiles, F issue) {       // every lane has read the tile
    __syncwarp();
    if (k + STAGES < tiles && elect_one()) {
      mbar_expect_tx(&full[k % STAGES], STAGE_BYTES);
      issue(k + STAGES, stage(k), &full[k % STAGES]);
    }
    __syncwarp();
    ++k;
  }
};
__device__ __forceinline__ RawRow<4> ring_row(const uint8_t* tile, int i) {
  RawRow<4> r;
  r.w = *reinterpret_cast<const uint2*>(tile + i * 256);
  return r;
}

// Sums of N = 4 or 8 values over the lanes of a warp, every lane gets all of them: halving exchanges (each step sends the half
// that the partner keeps), then one broadcast per value: 2N + 1 or 2N + 2 shuffles instead of 5N.
template <int N>
__device__ __forceinline__ void warp_sums(float (&v)[N]) {
  static_assert(N == 4 || N == 8, "four or eight values");
  const int lane = threadIdx.x & 31;
  int keep = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n >>= 1) {
    const bool up = (lane & keep) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], mine = up ? v[i + n] : v[i];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, send, keep);
    }
    keep >>= 1;
  }
  float s = v[0];
#pragma unroll
  for (; keep >= 1; keep >>= 1) s += __shfl_xor_sync(0xffffffffu, s, keep);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    int src = 0;
    if (N == 8) src = ((i >> 2) & 1) * 16 + ((i >> 1) & 1) * 8 + (i & 1) * 4;
    else src = ((i >> 1) & 1) * 16 + (i & 1) * 8;
    v[i] = __shfl_sync(0xffffffffu, s, src);
  }
}

// ---- ring kernels: channel counts that are multiples of eight ------------------------------------------------------------
struct RingArgs {
  const __nv_bfloat16* x;        // the three rows before a run; the rest arrives by TMA
  const __nv_bfloat16* weight;
  __nv_bfloat16* out;            // y or dx
  int64_t out_stride_b, out_stride_t;
  float* dw_partial;             // [B * runs][dw_channels][4], this launch's channels from dw_c0
  int dw_channels, dw_c0;
  const int32_t* cu;
  int n_docs, T, C, act_channels, units, runs, run;     // units of 128 channels; runs of `run` tokens
  int64_t stride_b, stride_t;
  // fused glue: the first 3 H units are the heads of q, k, v
  int H;
  float eps;
  __nv_bfloat16 *q, *k, *v;      // forward outputs (B, T, H, 128)
  int n_warps;
  int* status;
};
struct RingWork {
  int unit, run, b, lo, own, c0;
  bool live;
  __device__ __forceinline__ RingWork(const RingArgs& a, int wi) {
    unit = wi % a.units;
    run = wi / a.units % a.runs;
    b = wi / a.units / a.runs;
    lo = run * a.run;
    own = min(a.T, lo + a.run);
    c0 = unit * 128 + (threadIdx.x & 31) * 4;
    live = c0 < a.C;
  }
};

// Forward.  GLUE: a warp owns one head of q, k or v, so that the head's norm is a sum over its lanes.
template <bool GLUE, int ACT>
__device__ __forceinline__ void ring_fwd_walk(const CUtensorMap* map_x, const RingArgs& a, const RingWork& w, Ring<1, RING_FWD_STAGES>& ring,
                                              const WaitCtl& ctl) {
  const int tiles = (w.own - w.lo + RING_ROWS - 1) / RING_ROWS;
  const bool normed = GLUE && w.unit < 2 * a.H;
  auto issue = [&](int tile, uint8_t* dst, uint64_t* bar) { tma_load_3d(dst, map_x, bar, w.unit * 128, w.lo + tile * RING_ROWS, w.b); };
  ring.open(tiles, issue);
  const Taps<4> taps = load_taps<4>(a.weight, w.c0, w.live);
  DocCursor doc;
  doc.init(a.cu, a.n_docs, w.lo);
  doc.advance(w.lo);
  Window<4> win;
  open_window<4>(win, a.x + w.b * a.stride_b + (w.live ? w.c0 : 0), a.stride_t, w.lo, max(doc.start, 0), w.live);
  __nv_bfloat16* out;
  int64_t os;
  if constexpr (GLUE) {
    const int region = w.unit / a.H, head = w.unit % a.H;
    out = (region == 0 ? a.q : region == 1 ? a.k : a.v) + ((static_cast<int64_t>(w.b) * a.T + w.lo) * a.H + head) * HEAD + (threadIdx.x & 31) * 4;
    os = static_cast<int64_t>(a.H) * HEAD;
  } else {
    out = a.out + w.b * a.out_stride_b + w.lo * a.out_stride_t + w.c0;
    os = a.out_stride_t;
  }
  auto act_row = [&](const Pairs<4>& x0) {
    Pairs<4> s;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float2 acc = win.conv(taps, x0, p);
      if constexpr (ACT == 0) s.p[p] = acc;
      else if constexpr (ACT == 1) s.p[p] = make_float2(silu(acc.x), silu(acc.y));
      else s.p[p] = make_float2(w.c0 + 2 * p < a.act_channels ? silu(acc.x) : acc.x, w.c0 + 2 * p + 1 < a.act_channels ? silu(acc.y) : acc.y);
    }
    return s;
  };
  auto square = [&](const Pairs<4>& s) {
    const float2 q = __ffma2_rn(s.p[0], s.p[0], __fmul2_rn(s.p[1], s.p[1]));
    return q.x + q.y;
  };
  auto scaled = [&](const Pairs<4>& s, float r) {
    Pairs<4> o;
#pragma unroll
    for (int p = 0; p < 2; ++p) o.p[p] = __fmul2_rn(s.p[p], make_float2(r, r));
    return o;
  };
  for (int tile = 0; tile < tiles; ++tile) {
    const int t = w.lo + tile * RING_ROWS;
    const uint8_t* xt = ring.wait(ctl);
    if (t + RING_ROWS <= w.own && doc.next >= t + RING_ROWS) {     // every row is there and belongs to the window's document
      Pairs<4> s[RING_ROWS];
      float ss[RING_ROWS];
#pragma unroll
      for (int i = 0; i < RING_ROWS; ++i) {
        const Pairs<4> x0 = unpack<4>(ring_row(xt, i));
        s[i] = act_row(x0);
        if constexpr (GLUE) ss[i] = square(s[i]);
        win.push(x0);
        if (!GLUE) {
          if (w.live) store_row<4>(out, s[i]);
          out += os;
        }
      }
      if constexpr (GLUE) {
        if (normed) warp_sums<RING_ROWS>(ss);
#pragma unroll
        for (int i = 0; i < RING_ROWS; ++i) {
          store_row<4>(out, normed ? scaled(s[i], rsqrtf(ss[i] + a.eps)) : s[i]);
          out += os;
        }
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < RING_ROWS; ++i) {
        const int r = t + i;
        if (r >= w.own) break;
        if (r >= doc.next) {
          doc.advance(r);
#pragma unroll
          for (int j = 0; j < 3; ++j) win.m[j] = zero_pairs<4>();
        }
        const Pairs<4> x0 = unpack<4>(ring_row(xt, i));
        Pairs<4> s = act_row(x0);
        if (GLUE && normed) {
          float sums[4] = {square(s), 0.f, 0.f, 0.f};
          warp_sums<4>(sums);
          s = scaled(s, rsqrtf(sums[0] + a.eps));
        }
        if (w.live) store_row<4>(out, s);
        out += os;
        win.push(x0);
      }
    }
    ring.release(tiles, issue);
  }
}

template <bool GLUE>
__global__ void __launch_bounds__(RING_WARPS * 32, GLUE ? 5 : 6)
ring_fwd_kernel(const __grid_constant__ CUtensorMap map_x, RingArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bars[RING_WARPS * RING_FWD_STAGES];
  __shared__ int abort_s;
  if (threadIdx.x == 0) abort_s = 0;
  __syncthreads();
  const int wi = blockIdx.x * RING_WARPS + __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  if (wi >= a.n_warps) return;
  const RingWork w(a, wi);
  WaitCtl ctl{&abort_s, a.status};
  Ring<1, RING_FWD_STAGES> ring;
  ring.init(smem, bars);
  if constexpr (GLUE) {
    ring_fwd_walk<true, 1>(&map_x, a, w, ring, ctl);
  } else {
    const bool all = __all_sync(0xffffffffu, !w.live || w.c0 + 4 <= a.act_channels), none = __all_sync(0xffffffffu, !w.live || w.c0 >= a.act_channels);
    if (all) ring_fwd_walk<false, 1>(&map_x, a, w, ring, ctl);
    else if (none) ring_fwd_walk<false, 0>(&map_x, a, w, ring, ctl);
    else ring_fwd_walk<false, 2>(&map_x, a, w, ring, ctl);
  }
}

// Backward.  GLUE: the gradient rows are those of q, k, v (map_g: one map per region); the activations are formed again from the
// window, s = SiLU(pre), and
//   ds = r dy - r^3 <s, dy> s,   r = rsqrt(sum s^2 + eps)      (v: ds = dv),      dy' = ds SiLU'(pre)
// in one pass: x and the gradients are read once and dx written once.  (Two kernels, with the gradient of the convolution's
// output written and read in between, took 1.09 ms for the 12288 q, k, v channels
// of (1, 32768, 13056) where this one takes 0.58.)
// (Rows per reduction of the head norms: four rows take fewer shuffles each but hold s and SiLU' of four rows, 168 registers or
// spills: 595 to 790 us against 583.)
constexpr int GR = 2;
template <bool GLUE, int ACT>
__device__ __forceinline__ void ring_bwd_walk(const CUtensorMap* map_x, const CUtensorMap* map_g, const RingArgs& a, const RingWork& w,
                                              Ring<2, RING_BWD_STAGES>& ring, const WaitCtl& ctl, float2 (&dw)[2][CONV_W]) {
  const int tiles = (w.own + 3 - w.lo + RING_ROWS - 1) / RING_ROWS;
  const int head = GLUE ? w.unit % a.H : 0;
  const bool normed = GLUE && w.unit < 2 * a.H;
  auto issue = [&](int tile, uint8_t* dst, uint64_t* bar) {
    const int t = w.lo + tile * RING_ROWS;
    tma_load_3d(dst, map_x, bar, w.unit * 128, t, w.b);
    if constexpr (GLUE) tma_load_4d(dst + RING_TILE, map_g, bar, 0, head, t, w.b);
    else tma_load_3d(dst + RING_TILE, map_g, bar, w.unit * 128, t, w.b);
  };
  ring.open(tiles, issue);
  const Taps<4> taps = load_taps<4>(a.weight, w.c0, w.live);
  DocCursor doc;
  doc.init(a.cu, a.n_docs, w.lo);
  doc.advance(w.lo);
  Window<4> win, gw;                                     // x[t-1..t-3], dy'[t-1..t-3]
  open_window<4>(win, a.x + w.b * a.stride_b + (w.live ? w.c0 : 0), a.stride_t, w.lo, max(doc.start, 0), w.live);
#pragma unroll
  for (int j = 0; j < 3; ++j) gw.m[j] = zero_pairs<4>();
  int ds1 = 0x7fffffff, ds2 = 0x7fffffff;                // document starts of tokens t-1, t-2
  __nv_bfloat16* out = a.out + w.b * a.out_stride_b + (w.lo - 3) * a.out_stride_t + w.c0;   // row t - 3

  auto add_dw = [&](const Pairs<4>& gy, const Pairs<4>& x0) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      dw[p][0] = __ffma2_rn(gy.p[p], win.m[2].p[p], dw[p][0]);
      dw[p][1] = __ffma2_rn(gy.p[p], win.m[1].p[p], dw[p][1]);
      dw[p][2] = __ffma2_rn(gy.p[p], win.m[0].p[p], dw[p][2]);
      dw[p][3] = __ffma2_rn(gy.p[p], x0.p[p], dw[p][3]);
    }
  };
  // one row's pre-activation -> gradient factor: plain convolution
  auto plain_grad = [&](const Pairs<4>& x0, Pairs<4>& gy) {
    if constexpr (ACT != 0) {
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        float2 sg = silu_grad_pair(win.conv(taps, x0, p));
        if constexpr (ACT == 2) {
          sg.x = w.c0 + 2 * p < a.act_channels ? sg.x : 1.f;
          sg.y = w.c0 + 2 * p + 1 < a.act_channels ? sg.y : 1.f;
        }
        gy.p[p] = __fmul2_rn(gy.p[p], sg);
      }
    }
  };
  // s = SiLU(pre), sp = SiLU'(pre); this lane's shares of sum s^2 and <s, g>
  auto glue_act = [&](const Pairs<4>& x0, const Pairs<4>& g, Pairs<4>& s, Pairs<4>& sp, float& ss, float& dot) {
    float2 s2 = make_float2(0.f, 0.f), d2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float2 pre = win.conv(taps, x0, p);
      const float2 sig = make_float2(fast_sigmoid(pre.x), fast_sigmoid(pre.y));
      s.p[p] = __fmul2_rn(pre, sig);
      // sig (1 + pre (1 - sig)) = sig + s - s sig
      sp.p[p] = __ffma2_rn(s.p[p], __ffma2_rn(sig, make_float2(-1.f, -1.f), make_float2(1.f, 1.f)), sig);
      s2 = __ffma2_rn(s.p[p], s.p[p], s2);
      d2 = __ffma2_rn(s.p[p], g.p[p], d2);
    }
    ss = s2.x + s2.y;
    dot = d2.x + d2.y;
  };
  auto glue_grad = [&](Pairs<4>& gy, const Pairs<4>& s, const Pairs<4>& sp, float ss, float dot) {
    const float r = rsqrtf(ss + a.eps), f = -r * r * r * dot;
    const float2 r2 = make_float2(r, r), f2 = make_float2(f, f);
#pragma unroll
    for (int p = 0; p < 2; ++p) gy.p[p] = __fmul2_rn(__ffma2_rn(f2, s.p[p], __fmul2_rn(r2, gy.p[p])), sp.p[p]);
  };
  auto dx_row = [&](const Pairs<4>& g3, const Pairs<4>& g2, const Pairs<4>& g1, const Pairs<4>& g0) {
    Pairs<4> o;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      float2 acc = __fmul2_rn(g3.p[p], taps.w[p][3]);
      acc = __ffma2_rn(g2.p[p], taps.w[p][2], acc);
      acc = __ffma2_rn(g1.p[p], taps.w[p][1], acc);
      o.p[p] = __ffma2_rn(g0.p[p], taps.w[p][0], acc);
    }
    return o;
  };

  for (int tile = 0; tile < tiles; ++tile) {
    const int t = w.lo + tile * RING_ROWS;
    const uint8_t* xt = ring.wait(ctl);
    const uint8_t* gt = xt + RING_TILE;
    // Interior: every row is the warp's own and no document starts among the rows or the three before them.
    if (tile > 0 && t + RING_ROWS <= w.own && doc.next >= t + RING_ROWS && doc.start <= t - 3) {
      if constexpr (!GLUE) {
#pragma unroll
        for (int i = 0; i < RING_ROWS; ++i) {
          const Pairs<4> x0 = unpack<4>(ring_row(xt, i));
          Pairs<4> gy = unpack<4>(ring_row(gt, i));
          plain_grad(x0, gy);
          add_dw(gy, x0);
          const Pairs<4> o = dx_row(gw.m[2], gw.m[1], gw.m[0], gy);
          if (w.live) store_row<4>(out, o);
          out += a.out_stride_t;
          gw.push(gy);
          win.push(x0);
        }
      } else {
#pragma unroll
        for (int step = 0; step < RING_ROWS; step += GR) {
          Pairs<4> s[GR], sp[GR];
          float sums[2 * GR];
          const Window<4> keep = win;
#pragma unroll
          for (int i = 0; i < GR; ++i) {
            const Pairs<4> x0 = unpack<4>(ring_row(xt, step + i)), g = unpack<4>(ring_row(gt, step + i));
            glue_act(x0, g, s[i], sp[i], sums[i], sums[GR + i]);
            win.push(x0);
          }
          if (normed) warp_sums<2 * GR>(sums);
          win = keep;
#pragma unroll
          for (int i = 0; i < GR; ++i) {
            const Pairs<4> x0 = unpack<4>(ring_row(xt, step + i));
            Pairs<4> gy = unpack<4>(ring_row(gt, step + i));
            if (normed) {
              glue_grad(gy, s[i], sp[i], sums[i], sums[GR + i]);
            } else {
#pragma unroll
              for (int p = 0; p < 2; ++p) gy.p[p] = __fmul2_rn(gy.p[p], sp[i].p[p]);
            }
            add_dw(gy, x0);
            store_row<4>(out, dx_row(gw.m[2], gw.m[1], gw.m[0], gy));
            out += a.out_stride_t;
            gw.push(gy);
            win.push(x0);
          }
        }
      }
      ds1 = ds2 = doc.start;
    } else {
#pragma unroll 1
      for (int i = 0; i < RING_ROWS; ++i) {
        const int r = t + i;
        Pairs<4> x0 = zero_pairs<4>(), gy = zero_pairs<4>();
        int ds0 = 0x7fffffff;
        if (r < a.T && r < w.own + 3) {
          if (r >= doc.next) {                           // a document starts here
            doc.advance(r);
#pragma unroll
            for (int j = 0; j < 3; ++j) win.m[j] = zero_pairs<4>();
          }
          ds0 = doc.start;
          x0 = unpack<4>(ring_row(xt, i));
          gy = unpack<4>(ring_row(gt, i));
          if constexpr (!GLUE) {
            plain_grad(x0, gy);
          } else {
            Pairs<4> s, sp;
            float sums[4] = {0.f, 0.f, 0.f, 0.f};
            glue_act(x0, gy, s, sp, sums[0], sums[1]);
            if (normed) {
              warp_sums<4>(sums);
              glue_grad(gy, s, sp, sums[0], sums[1]);
            } else {
#pragma unroll
              for (int p = 0; p < 2; ++p) gy.p[p] = __fmul2_rn(gy.p[p], sp.p[p]);
            }
          }
          if (r < w.own) add_dw(gy, x0);                 // the weight gradient of a token belongs to one warp
        }
        const int u = r - 3;
        if (u >= w.lo && u < w.own && w.live) {          // gradients of later documents do not reach back
          const Pairs<4> z = zero_pairs<4>();
          store_row<4>(out, dx_row(gw.m[2], ds2 <= u ? gw.m[1] : z, ds1 <= u ? gw.m[0] : z, ds0 <= u ? gy : z));
        }
        out += a.out_stride_t;
        gw.push(gy);
        win.push(x0);
        ds2 = ds1;
        ds1 = ds0;
      }
    }
    ring.release(tiles, issue);
  }
}

template <bool GLUE>
__global__ void __launch_bounds__(RING_WARPS * 32, 4)
ring_bwd_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_g0,
                const __grid_constant__ CUtensorMap map_g1, const __grid_constant__ CUtensorMap map_g2, RingArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bars[RING_WARPS * RING_BWD_STAGES];
  __shared__ int abort_s;
  if (threadIdx.x == 0) abort_s = 0;
  __syncthreads();
  const int wi = blockIdx.x * RING_WARPS + __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  if (wi >= a.n_warps) return;
  const RingWork w(a, wi);
  WaitCtl ctl{&abort_s, a.status};
  Ring<2, RING_BWD_STAGES> ring;
  ring.init(smem, bars);
  float2 dw[2][CONV_W];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int j = 0; j < CONV_W; ++j) dw[p][j] = make_float2(0.f, 0.f);
  if constexpr (GLUE) {
    const int region = w.unit / a.H;
    ring_bwd_walk<true, 1>(&map_x, region == 0 ? &map_g0 : region == 1 ? &map_g1 : &map_g2, a, w, ring, ctl, dw);
  } else {
    const bool all = __all_sync(0xffffffffu, !w.live || w.c0 + 4 <= a.act_channels), none = __all_sync(0xffffffffu, !w.live || w.c0 >= a.act_channels);
    if (all) ring_bwd_walk<false, 1>(&map_x, &map_g0, a, w, ring, ctl, dw);
    else if (none) ring_bwd_walk<false, 0>(&map_x, &map_g0, a, w, ring, ctl, dw);
    else ring_bwd_walk<false, 2>(&map_x, &map_g0, a, w, ring, ctl, dw);
  }
  if (w.live) {                                          // the weight gradient of this run: 4 channels x 4 taps per lane
    float* out = a.dw_partial + ((static_cast<int64_t>(w.b) * a.runs + w.run) * a.dw_channels + a.dw_c0 + w.c0) * CONV_W;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      *reinterpret_cast<float4*>(out + 8 * p) = make_float4(dw[p][0].x, dw[p][1].x, dw[p][2].x, dw[p][3].x);
      *reinterpret_cast<float4*>(out + 8 * p + 4) = make_float4(dw[p][0].y, dw[p][1].y, dw[p][2].y, dw[p][3].y);
    }
  }
}


// ---- walkers: what the ring kernels cannot take (channel counts, strides or addresses that are no multiples of 16 bytes) --------
constexpr int CONV_WARPS = 8;          // sub-runs per CTA
constexpr int CONV_THREADS = CONV_WARPS * 32;
constexpr int WALK_ROWS = 4;           // rows per batch
// Rows of a walk in batches of U, the next batch asked for before the current one is used.  Addresses are clamped to the row
// `last` (always valid); what lies beyond the walk is masked by the caller.
template <int V, int U>
struct RowBatch {
  RawRow<V> r[U];
  __device__ __forceinline__ void load(const __nv_bfloat16* col, int64_t stride, int t, int last) {
    if (t + U - 1 <= last) {
      const __nv_bfloat16* p = col + t * stride;
#pragma unroll
      for (int i = 0; i < U; ++i) { r[i] = load_raw<V>(p); p += stride; }
    } else {
#pragma unroll
      for (int i = 0; i < U; ++i) r[i] = load_raw<V>(col + min(t + i, last) * stride);
    }
  }
};

struct ConvArgs {
  const __nv_bfloat16* x;
  const __nv_bfloat16* weight;
  const __nv_bfloat16* dy;       // backward
  __nv_bfloat16* out;            // y (forward) or dx (backward), contiguous (B, T, C)
  float* dw_partial;             // backward: [B * groups][C][4]
  const int32_t* cu;
  int n_docs, T, C, act_channels, run;      // run: tokens per CTA
  int64_t x_stride_b, x_stride_t, dy_stride_b, dy_stride_t;
};

// This warp's tokens [lo, hi) and channels.
template <int V>
struct Walk {
  int lo, hi, c0;
  bool live;
  __device__ __forceinline__ Walk(int T, int C, int run) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.y * run, sub = (run + CONV_WARPS - 1) / CONV_WARPS;
    lo = first + warp * sub;
    hi = min(T, min(lo + sub, first + run));
    c0 = (blockIdx.x * 32 + lane) * V;
    live = c0 < C;
  }
};

template <int V, int ACT>
__device__ __forceinline__ void conv_fwd_walk(const ConvArgs& a, const Walk<V>& w) {
  constexpr int P = (V + 1) / 2;
  const Taps<V> taps = load_taps<V>(a.weight, w.c0, w.live);
  const int64_t xs = a.x_stride_t, ys = a.C;
  const __nv_bfloat16* col = a.x + blockIdx.z * a.x_stride_b + (w.live ? w.c0 : 0);
  __nv_bfloat16* out = a.out + static_cast<int64_t>(blockIdx.z) * a.T * a.C + w.c0;
  DocCursor doc;
  doc.init(a.cu, a.n_docs, w.lo);
  for (int t = w.lo; t < w.hi;) {
    doc.advance(t);
    const int end = min(w.hi, doc.next);
    Window<V> win;
    RowBatch<V, WALK_ROWS> b0, b1;
    b0.load(col, xs, t, end - 1);
    open_window<V>(win, col, xs, t, max(doc.start, 0), w.live);
    auto rows = [&](const RowBatch<V, WALK_ROWS>& b) {
      __nv_bfloat16* y = out + t * ys;
      const int n = end - t;
#pragma unroll
      for (int i = 0; i < WALK_ROWS; ++i) {
        const Pairs<V> x0 = unpack<V>(b.r[i]);
        Pairs<V> o;
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const float2 acc = win.conv(taps, x0, p);
          if constexpr (ACT == 0) o.p[p] = acc;
          else if constexpr (ACT == 1) o.p[p] = make_float2(silu(acc.x), silu(acc.y));
          else o.p[p] = make_float2(w.c0 + 2 * p < a.act_channels ? silu(acc.x) : acc.x, w.c0 + 2 * p + 1 < a.act_channels ? silu(acc.y) : acc.y);
        }
        if (w.live && i < n) store_row<V>(y, o);
        y += ys;
        win.push(x0);
      }
      t += WALK_ROWS;
    };
    for (;;) {
      if (t + WALK_ROWS < end) b1.load(col, xs, t + WALK_ROWS, end - 1);
      rows(b0);
      if (t >= end) break;
      if (t + WALK_ROWS < end) b0.load(col, xs, t + WALK_ROWS, end - 1);
      rows(b1);
      if (t >= end) break;
    }
    t = end;
  }
}

template <int V>
__global__ void __launch_bounds__(CONV_THREADS, 3)
conv_fwd_kernel(ConvArgs a) {
  const Walk<V> w(a.T, a.C, a.run);
  if (w.lo >= w.hi) return;
  switch (act_kind(w.c0, V, w.live, a.act_channels)) {
    case 0: conv_fwd_walk<V, 0>(a, w); break;
    case 1: conv_fwd_walk<V, 1>(a, w); break;
    default: conv_fwd_walk<V, 2>(a, w); break;
  }
}

// Backward over the rows [lo, hi) of this warp: dx, and the weight gradient of these rows in `dw`.
//   dy'[t] = dy[t] SiLU'(pre[t])      dw[j] += dy'[t] x[t-3+j]      dx[u] = sum_j dy'[u+j] w[3-j]  over tokens of the same document
// A walk of one document's rows ends with the three gradients behind its own rows (which the next walk owns; zero past the end
// of the document).
template <int V, int ACT>
__device__ __forceinline__ void conv_bwd_walk(const ConvArgs& a, const Walk<V>& w, float2 (&dw)[(V + 1) / 2][CONV_W]) {
  constexpr int P = (V + 1) / 2;
  const Taps<V> taps = load_taps<V>(a.weight, w.c0, w.live);
  const int64_t xs = a.x_stride_t, gs = a.dy_stride_t, os = a.C;
  const __nv_bfloat16* col = a.x + blockIdx.z * a.x_stride_b + (w.live ? w.c0 : 0);
  const __nv_bfloat16* gcol = a.dy + blockIdx.z * a.dy_stride_b + (w.live ? w.c0 : 0);
  __nv_bfloat16* out = a.out + static_cast<int64_t>(blockIdx.z) * a.T * a.C + w.c0;
  DocCursor doc;
  doc.init(a.cu, a.n_docs, w.lo);
  for (int t = w.lo; t < w.hi;) {
    doc.advance(t);
    const int own = min(w.hi, doc.next), real = min(own + 3, min(doc.next, a.T)), first = t;
    Window<V> win, gw;                                   // gw: dy'[t-1], dy'[t-2], dy'[t-3]
    RowBatch<V, WALK_ROWS> x0b, g0b, x1b, g1b;
    x0b.load(col, xs, t, real - 1);
    g0b.load(gcol, gs, t, real - 1);
    open_window<V>(win, col, xs, t, max(doc.start, 0), w.live);
#pragma unroll
    for (int j = 0; j < 3; ++j) gw.m[j] = zero_pairs<V>();
    auto row = [&](const RawRow<V>& xr, const RawRow<V>& gr, int r, bool edge) {
      const Pairs<V> x0 = unpack<V>(xr);
      Pairs<V> gy = unpack<V>(gr);
      if constexpr (ACT != 0) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          float2 sg = silu_grad_pair(win.conv(taps, x0, p));
          if constexpr (ACT == 2) {
            sg.x = w.c0 + 2 * p < a.act_channels ? sg.x : 1.f;
            sg.y = w.c0 + 2 * p + 1 < a.act_channels ? sg.y : 1.f;
          }
          gy.p[p] = __fmul2_rn(gy.p[p], sg);
        }
      }
      if (edge && r >= real) gy = zero_pairs<V>();
      if (!edge || r < own) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          dw[p][0] = __ffma2_rn(gy.p[p], win.m[2].p[p], dw[p][0]);
          dw[p][1] = __ffma2_rn(gy.p[p], win.m[1].p[p], dw[p][1]);
          dw[p][2] = __ffma2_rn(gy.p[p], win.m[0].p[p], dw[p][2]);
          dw[p][3] = __ffma2_rn(gy.p[p], x0.p[p], dw[p][3]);
        }
      }
      if (w.live && r - 3 >= first && (!edge || r - 3 < own)) {
        Pairs<V> o;
#pragma unroll
        for (int p = 0; p < P; ++p) {
          float2 acc = __fmul2_rn(gw.m[2].p[p], taps.w[p][3]);
          acc = __ffma2_rn(gw.m[1].p[p], taps.w[p][2], acc);
          acc = __ffma2_rn(gw.m[0].p[p], taps.w[p][1], acc);
          o.p[p] = __ffma2_rn(gy.p[p], taps.w[p][0], acc);
        }
        store_row<V>(out + (r - 3) * os, o);
      }
      gw.push(gy);
      win.push(x0);
    };
    auto rows = [&](const RowBatch<V, WALK_ROWS>& xb, const RowBatch<V, WALK_ROWS>& gb) {
      if (t + WALK_ROWS <= own) {
#pragma unroll
        for (int i = 0; i < WALK_ROWS; ++i) row(xb.r[i], gb.r[i], t + i, false);
      } else {
#pragma unroll
        for (int i = 0; i < WALK_ROWS; ++i) row(xb.r[i], gb.r[i], t + i, true);
      }
      t += WALK_ROWS;
    };
    for (;;) {
      if (t + WALK_ROWS < real) {
        x1b.load(col, xs, t + WALK_ROWS, real - 1);
        g1b.load(gcol, gs, t + WALK_ROWS, real - 1);
      }
      rows(x0b, g0b);
      if (t >= own + 3) break;
      if (t + WALK_ROWS < real) {
        x0b.load(col, xs, t + WALK_ROWS, real - 1);
        g0b.load(gcol, gs, t + WALK_ROWS, real - 1);
      }
      rows(x1b, g1b);
      if (t >= own + 3) break;
    }
    t = own;
  }
}

// Sum of the warps' weight gradients in index order -> this CTA's partial.
template <int V>
__device__ __forceinline__ void reduce_dw(const float2 (&dw)[(V + 1) / 2][CONV_W], float* red, float* out, int channels, int cbase) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int c = 0; c < V; ++c) {
    float4 v;
    v.x = (c & 1) ? dw[c / 2][0].y : dw[c / 2][0].x;
    v.y = (c & 1) ? dw[c / 2][1].y : dw[c / 2][1].x;
    v.z = (c & 1) ? dw[c / 2][2].y : dw[c / 2][2].x;
    v.w = (c & 1) ? dw[c / 2][3].y : dw[c / 2][3].x;
    *reinterpret_cast<float4*>(red + (warp * 32 * V + lane * V + c) * CONV_W) = v;
  }
  __syncthreads();
  for (int e = tid; e < 32 * V * CONV_W; e += CONV_THREADS) {
    if (e / CONV_W >= channels) break;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < CONV_WARPS; ++w) s += red[w * 32 * V * CONV_W + e];
    out[static_cast<int64_t>(cbase) * CONV_W + e] = s;
  }
}

template <int V>
// (Three CTAs per SM leave the walk of single channels 80 registers: it spills 412 bytes.)
__global__ void __launch_bounds__(CONV_THREADS, V == 4 ? 2 : 3)
conv_bwd_kernel(ConvArgs a) {
  __shared__ __align__(16) float red[CONV_WARPS * 32 * V * CONV_W];
  const Walk<V> w(a.T, a.C, a.run);
  float2 dw[(V + 1) / 2][CONV_W];
#pragma unroll
  for (int p = 0; p < (V + 1) / 2; ++p)
#pragma unroll
    for (int j = 0; j < CONV_W; ++j) dw[p][j] = make_float2(0.f, 0.f);
  if (w.lo < w.hi) {
    switch (act_kind(w.c0, V, w.live, a.act_channels)) {
      case 0: conv_bwd_walk<V, 0>(a, w, dw); break;
      case 1: conv_bwd_walk<V, 1>(a, w, dw); break;
      default: conv_bwd_walk<V, 2>(a, w, dw); break;
    }
  }
  const int cbase = blockIdx.x * 32 * V;
  float* out = a.dw_partial + (static_cast<int64_t>(blockIdx.z) * gridDim.y + blockIdx.y) * (static_cast<int64_t>(a.C) * CONV_W);
  reduce_dw<V>(dw, red, out, a.C - cbase, cbase);
}

__global__ void conv_dw_reduce_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dw, int n_partial,
                                      int n_elem) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_elem) return;
  float acc = 0.f;
  for (int p = 0; p < n_partial; ++p) acc += partial[static_cast<int64_t>(p) * n_elem + i];
  dw[i] = __float2bfloat16_rn(acc);
}

}  // namespace tgdn

using namespace tgdn;

static int conv_check(const void* x, const void* weight, const void* y, const int32_t* cu, int n_docs, int B, int T,
                      int C, int64_t stride_b, int64_t stride_t) {
  if (!x || !weight || !y) return TGDN_ERR_NULL;
  if (B <= 0 || T <= 0 || C <= 0) return TGDN_ERR_SHAPE;
  if (cu && (B != 1 || n_docs < 1)) return TGDN_ERR_SHAPE;
  if (B > 65535) return TGDN_ERR_SHAPE;
  if (reinterpret_cast<uintptr_t>(weight) & 7) return TGDN_ERR_ALIGN;         // the four taps of a channel are one load
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 1) || stride_t < C) return TGDN_ERR_ALIGN;
  return 0;
}
// What the entry points of the public ABI ask for: whole 16-byte pieces.
static int conv_check_abi(const void* x, const void* weight, const void* y, const int32_t* cu, int n_docs, int B, int T,
                          int C, int64_t stride_b, int64_t stride_t) {
  const int rc = conv_check(x, weight, y, cu, n_docs, B, T, C, stride_b, stride_t);
  if (rc && rc != TGDN_ERR_ALIGN) return rc;
  if (C % 8) return TGDN_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(y)) & 15) return TGDN_ERR_ALIGN;
  return ((stride_b % 8) || (stride_t % 8) || stride_t < C) ? TGDN_ERR_ALIGN : 0;
}

// The ring kernels want what a tensor map wants: 16-byte aligned rows of whole 16-byte pieces (and 8-byte stores).
static bool ring_ok(int C, std::initializer_list<const void*> ptrs, std::initializer_list<int64_t> strides) {
  uintptr_t p = 0;
  int64_t s = C;
  for (const void* q : ptrs) p |= reinterpret_cast<uintptr_t>(q);
  for (int64_t q : strides) s |= q;
  return s % 8 == 0 && p % 16 == 0;
}
// Channels per lane of the walkers: 8-byte, 4-byte or 2-byte accesses.
static int walk_vec(int C, std::initializer_list<const void*> ptrs, std::initializer_list<int64_t> strides) {
  uintptr_t p = 0;
  int64_t s = C;
  for (const void* q : ptrs) p |= reinterpret_cast<uintptr_t>(q);
  for (int64_t q : strides) s |= q;
  if (s % 4 == 0 && p % 8 == 0) return 4;
  return (s % 2 == 0 && p % 4 == 0) ? 2 : 1;
}

// Runs per batch row of a ring kernel: as many warps as fill the chip `waves` times over with `per_sm` resident warps, runs of
// at least `least` tokens (a run loads three rows to open its window; the backward walks three more behind its end).
// Measured at (1, 32768, 13056), us: forward 23 runs 319, 46 310, 92 307, 164 299, 513 311; backward 23 runs 462, 46 452, 92 424,
// 164 431, 513 518 (each run leaves a weight-gradient partial); at (2, 4096, 4096) the forward falls from 42 (runs of 195) to 33
// (runs of 32), the backward is flat at 58 between runs of 195 and 63.
static int ring_runs(int B, int T, int units, int waves, int per_sm, int least) {
  const int64_t warps = static_cast<int64_t>(waves) * per_sm * tgdn_sm_count();
  int64_t runs = warps / (static_cast<int64_t>(units) * B);
  if (runs > T / least) runs = T / least;
  return static_cast<int>(runs < 1 ? 1 : runs);
}
static int fwd_runs(int B, int T, int units) { return ring_runs(B, T, units, 5, 24, 16); }
static int bwd_runs(int B, int T, int units) { return ring_runs(B, T, units, 4, 16, 48); }

// Token groups for which the caller of the public ABI has scratch: one f32 partial of C x 4 per group and batch row.
static int scratch_groups(int B, int T, int C) {
  const int n_tiles = (T + CONV_TOK - 1) / CONV_TOK;
  const int64_t columns = static_cast<int64_t>((C + 255) / 256) * B;
  int64_t g = static_cast<int64_t>(8) * tgdn_sm_count() / columns;                     // 148 on a B200 (and without a device)
  if (g > n_tiles / 8) g = n_tiles / 8;
  if (g < 1) g = 1;
  const int tpg = static_cast<int>((n_tiles + g - 1) / g);
  return (n_tiles + tpg - 1) / tpg;
}
static int64_t partial_bytes(int B, int groups, int C) { return static_cast<int64_t>(B) * groups * C * CONV_W * static_cast<int64_t>(sizeof(float)); }

// Scratch with which the backward runs best; tgdn_conv_bwd_scratch_bytes is the least.
int64_t tgdn_conv_bwd_best_scratch(int B, int T, int C) {
  if (B <= 0 || T <= 0 || C <= 0) return 0;                            // the entry points refuse these sizes
  return partial_bytes(B, std::max(scratch_groups(B, T, C), bwd_runs(B, T, (C + 127) / 128)), C);
}

static RingArgs ring_args(const void* x, const void* weight, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b,
                          int64_t stride_t, int runs) {
  RingArgs a{};
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.weight = static_cast<const __nv_bfloat16*>(weight);
  a.cu = cu; a.n_docs = n_docs; a.T = T; a.C = C;
  a.units = (C + 127) / 128;
  a.run = (T + runs - 1) / runs;
  a.runs = (T + a.run - 1) / a.run;
  a.stride_b = stride_b; a.stride_t = stride_t;
  a.out_stride_b = static_cast<int64_t>(T) * C; a.out_stride_t = C;
  a.dw_channels = C;
  a.n_warps = a.units * a.runs * B;
  a.status = tgdn_status_word();
  return a;
}
static unsigned ring_grid(const RingArgs& a) { return static_cast<unsigned>((a.n_warps + RING_WARPS - 1) / RING_WARPS); }
constexpr int RING_FWD_SMEM = RING_WARPS * RING_FWD_STAGES * RING_TILE, RING_BWD_SMEM = RING_WARPS * RING_BWD_STAGES * RING_TILE * 2;

template <bool GLUE>
static int ring_fwd_launch(const RingArgs& a, int B, cudaStream_t s) {
  CUtensorMap mx;
  int rc = tgdn_make_rows_map(&mx, a.x, a.C, a.T, B, a.stride_t, a.stride_b, 128, RING_ROWS);
  if (rc) return rc;
  static bool configured[64] = {};
  if ((rc = tgdn_dynamic_smem(reinterpret_cast<const void*>(ring_fwd_kernel<GLUE>), RING_FWD_SMEM, configured))) return rc;
  ring_fwd_kernel<GLUE><<<ring_grid(a), RING_WARPS * 32, RING_FWD_SMEM, s>>>(mx, a);
  return tgdn_cuda_error(cudaGetLastError());
}
template <bool GLUE>
static int ring_bwd_launch(const RingArgs& a, int B, const CUtensorMap* mg, cudaStream_t s) {
  CUtensorMap mx;
  int rc = tgdn_make_rows_map(&mx, a.x, a.C, a.T, B, a.stride_t, a.stride_b, 128, RING_ROWS);
  if (rc) return rc;
  static bool configured[64] = {};
  if ((rc = tgdn_dynamic_smem(reinterpret_cast<const void*>(ring_bwd_kernel<GLUE>), RING_BWD_SMEM, configured))) return rc;
  ring_bwd_kernel<GLUE><<<ring_grid(a), RING_WARPS * 32, RING_BWD_SMEM, s>>>(mx, mg[0], mg[GLUE ? 1 : 0], mg[GLUE ? 2 : 0], a);
  return tgdn_cuda_error(cudaGetLastError());
}
static int reduce_dw_launch(const float* partial, void* dw, int n_partial, int C, cudaStream_t s) {
  const int n_elem = C * CONV_W;
  conv_dw_reduce_kernel<<<(n_elem + 127) / 128, 128, 0, s>>>(partial, static_cast<__nv_bfloat16*>(dw), n_partial, n_elem);
  return tgdn_cuda_error(cudaGetLastError());
}

// Tokens per CTA of the walkers: sub-runs of at least 16 rows, a few waves of CTAs, and of at most 256 rows as long as the grid holds
// that many CTAs along the token axis (65535).
static int walk_run(int B, int T, int columns) {
  int64_t groups = static_cast<int64_t>(32) * tgdn_sm_count() / (static_cast<int64_t>(columns) * B);
  if (groups < 1) groups = 1;
  const int64_t run = (T + groups - 1) / groups;
  const int64_t longest = std::max<int64_t>(256 * CONV_WARPS, (static_cast<int64_t>(T) + 65534) / 65535);
  return static_cast<int>(std::min<int64_t>(std::max<int64_t>(run, 16 * CONV_WARPS), longest));
}
template <int V>
static dim3 walk_grid(int B, int C, int groups) { return dim3((C + 32 * V - 1) / (32 * V), groups, B); }

int tgdn_conv_fwd_any(const void* x, const void* weight, void* y, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b,
                      int64_t stride_t, int act_channels, void* stream) {
  int rc = conv_check(x, weight, y, cu, n_docs, B, T, C, stride_b, stride_t);
  if (rc) return rc;
  if (!tgdn_check_device()) return TGDN_ERR_DEVICE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (ring_ok(C, {x, y}, {stride_b, stride_t})) {
    RingArgs a = ring_args(x, weight, cu, n_docs, B, T, C, stride_b, stride_t, fwd_runs(B, T, (C + 127) / 128));
    a.out = static_cast<__nv_bfloat16*>(y);
    a.act_channels = act_channels;
    return ring_fwd_launch<false>(a, B, s);
  }
  ConvArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(weight), nullptr, static_cast<__nv_bfloat16*>(y), nullptr,
             cu, n_docs, T, C, act_channels, 0, stride_b, stride_t, 0, 0};
  const int V = walk_vec(C, {x, y}, {stride_b, stride_t});
  a.run = walk_run(B, T, (C + 32 * V - 1) / (32 * V));
  const int groups = (T + a.run - 1) / a.run;
  if (V == 4) conv_fwd_kernel<4><<<walk_grid<4>(B, C, groups), CONV_THREADS, 0, s>>>(a);
  else if (V == 2) conv_fwd_kernel<2><<<walk_grid<2>(B, C, groups), CONV_THREADS, 0, s>>>(a);
  else conv_fwd_kernel<1><<<walk_grid<1>(B, C, groups), CONV_THREADS, 0, s>>>(a);
  return tgdn_cuda_error(cudaGetLastError());
}

int tgdn_conv_bwd_any(const void* x, const void* weight, const void* dy, void* dx, void* dw, const int32_t* cu, int n_docs, int B, int T,
                      int C, int64_t stride_b, int64_t stride_t, int64_t dy_stride_b, int64_t dy_stride_t, int act_channels,
                      void* scratch, int64_t scratch_bytes, void* stream) {
  int rc = conv_check(x, weight, dx, cu, n_docs, B, T, C, stride_b, stride_t);
  if (rc) return rc;
  if (!dy || !dw) return TGDN_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(dy) & 1) || dy_stride_t < C) return TGDN_ERR_ALIGN;
  if (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15) || scratch_bytes < partial_bytes(B, scratch_groups(B, T, C), C)) return TGDN_ERR_SCRATCH;
  if (!tgdn_check_device()) return TGDN_ERR_DEVICE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int room = static_cast<int>(std::min<int64_t>(scratch_bytes / partial_bytes(B, 1, C), 1 << 20));
  if (ring_ok(C, {x, dy, dx}, {stride_b, stride_t, dy_stride_b, dy_stride_t})) {
    RingArgs a = ring_args(x, weight, cu, n_docs, B, T, C, stride_b, stride_t, std::min(room, bwd_runs(B, T, (C + 127) / 128)));
    a.out = static_cast<__nv_bfloat16*>(dx);
    a.act_channels = act_channels;
    a.dw_partial = static_cast<float*>(scratch);
    CUtensorMap mg;
    if ((rc = tgdn_make_rows_map(&mg, dy, C, T, B, dy_stride_t, dy_stride_b, 128, RING_ROWS))) return rc;
    if ((rc = ring_bwd_launch<false>(a, B, &mg, s))) return rc;
    return reduce_dw_launch(a.dw_partial, dw, B * a.runs, C, s);
  }
  ConvArgs a{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(weight), static_cast<const __nv_bfloat16*>(dy),
             static_cast<__nv_bfloat16*>(dx), static_cast<float*>(scratch), cu, n_docs, T, C, act_channels, 0, stride_b, stride_t,
             dy_stride_b, dy_stride_t};
  const int V = walk_vec(C, {x, dy, dx}, {stride_b, stride_t, dy_stride_b, dy_stride_t});
  int groups = std::min(room, (T + walk_run(B, T, (C + 32 * V - 1) / (32 * V)) - 1) / walk_run(B, T, (C + 32 * V - 1) / (32 * V)));
  a.run = (T + groups - 1) / groups;
  groups = (T + a.run - 1) / a.run;
  if (V == 4) conv_bwd_kernel<4><<<walk_grid<4>(B, C, groups), CONV_THREADS, 0, s>>>(a);
  else if (V == 2) conv_bwd_kernel<2><<<walk_grid<2>(B, C, groups), CONV_THREADS, 0, s>>>(a);
  else conv_bwd_kernel<1><<<walk_grid<1>(B, C, groups), CONV_THREADS, 0, s>>>(a);
  if ((rc = tgdn_cuda_error(cudaGetLastError()))) return rc;
  return reduce_dw_launch(a.dw_partial, dw, B * groups, C, s);
}

extern "C" int tgdn_conv_fwd(const void* x, const void* weight, void* y, const int32_t* cu_seqlens, int n_docs, int B,
                             int T, int C, int64_t stride_b, int64_t stride_t, int act_channels, void* stream) {
  const int rc = conv_check_abi(x, weight, y, cu_seqlens, n_docs, B, T, C, stride_b, stride_t);
  return rc ? rc : tgdn_conv_fwd_any(x, weight, y, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, act_channels, stream);
}

extern "C" int64_t tgdn_conv_bwd_scratch_bytes(int B, int T, int C) {
  if (B <= 0 || T <= 0 || C <= 0) return 0;
  return partial_bytes(B, scratch_groups(B, T, C), C);
}

extern "C" int tgdn_conv_bwd(const void* x, const void* weight, const void* dy, void* dx, void* dw,
                             const int32_t* cu_seqlens, int n_docs, int B, int T, int C, int64_t stride_b,
                             int64_t stride_t, int64_t dy_stride_b, int64_t dy_stride_t, int act_channels, void* scratch,
                             int64_t scratch_bytes, void* stream) {
  int rc = conv_check_abi(x, weight, dx, cu_seqlens, n_docs, B, T, C, stride_b, stride_t);
  if (rc) return rc;
  if (!dy || !dw) return TGDN_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(dy) & 15) || (dy_stride_b % 8) || (dy_stride_t % 8) || dy_stride_t < C) return TGDN_ERR_ALIGN;
  return tgdn_conv_bwd_any(x, weight, dy, dx, dw, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, dy_stride_b, dy_stride_t,
                           act_channels, scratch, scratch_bytes, stream);
}

// ---------------------------------------------------------------------------------------------------------------------
// tgdn_conv_bwd_static: the same backward, for hosts that may not allocate device memory.
//
// Some embedders load this library into a process whose device memory is owned by someone else: an inference server
// with a fixed arena, a plugin inside a framework that forbids cudaMalloc on its worker threads, a latency-critical loop
// in which an allocation (which can synchronise the whole device, or fail once memory is fragmented) is not acceptable.
// They can hand over inputs and outputs but have no pool to take the weight-gradient partials from.  For them the
// partials live in a fixed array that is part of the library image itself.
//
// The array costs TGDN_CONV_STATIC_SCRATCH_BYTES on every GPU that loads the library, until the process exits.
// Its device address is looked up once per device (cudaGetSymbolAddress, with that device current) on the first call
// made on that device; make that first call outside any stream capture.  The array is shared by every call on the
// device and keeps whatever the previous call left in it: this kernel overwrites every partial it later reads, so
// nothing has to be cleared, but two calls that overlap on the GPU (different streams) would corrupt each other.
// ---------------------------------------------------------------------------------------------------------------------
static __device__ __align__(256) float g_conv_static_scratch[TGDN_CONV_STATIC_SCRATCH_BYTES / sizeof(float)];

namespace {
constexpr int kMaxDevices = 64;
float* g_static_ptr[kMaxDevices] = {nullptr};
std::mutex g_static_mutex;

// Device address of the static scratch array on the current device (looked up once per device).
int conv_static_scratch(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return tgdn_cuda_error(e);
  if (dev < 0 || dev >= kMaxDevices) return TGDN_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (g_static_ptr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_conv_static_scratch);
    if (e != cudaSuccess) return tgdn_cuda_error(e);
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int tgdn_conv_bwd_static(const void* x, const void* weight, const void* dy, void* dx, void* dw,
                                    const int32_t* cu_seqlens, int n_docs, int B, int T, int C, int64_t stride_b,
                                    int64_t stride_t, int64_t dy_stride_b, int64_t dy_stride_t, int act_channels,
                                    void* stream) {
  int rc = conv_check_abi(x, weight, dx, cu_seqlens, n_docs, B, T, C, stride_b, stride_t);
  if (rc) return rc;
  if (!dy || !dw) return TGDN_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(dy) & 15) || (dy_stride_b % 8) || (dy_stride_t % 8) || dy_stride_t < C) return TGDN_ERR_ALIGN;
  if (tgdn_conv_bwd_scratch_bytes(B, T, C) > static_cast<int64_t>(TGDN_CONV_STATIC_SCRATCH_BYTES)) return TGDN_ERR_STATIC_LIMIT;
  float* scratch = nullptr;
  if ((rc = conv_static_scratch(&scratch))) return rc;
  // (the partials of a caller with the least scratch: the same runs, the same sums)
  return tgdn_conv_bwd_any(x, weight, dy, dx, dw, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, dy_stride_b, dy_stride_t,
                           act_channels, scratch, tgdn_conv_bwd_scratch_bytes(B, T, C), stream);
}


// ---- the layer glue ------------------------------------------------------------------------------------------------------
// x (B, T, C) with C = H (3*128 + 2E) channels laid out as [q: H x 128 | k: H x 128 | v: H x 128 | k2: H x E | q2: H x E] goes straight
// to the tensors the core takes:
//   q, k  = l2norm(SiLU(conv))   bf16 (B, T, H, 128)         v = SiLU(conv)   bf16 (B, T, H, 128)
//   k2, q2 = l2norm(softplus(conv))   f32 (B, T, H, E)        l2norm(s) = s * rsqrt(sum s^2 + eps)
// which the reference only describes (cute_triadic_gdn/ops/conv_split_act.py:3-5) and leaves to separate elementwise passes.
// q, k, v: the ring kernels above with GLUE.  k2, q2 (2E of 384 + 2E channels per head): the kernel below; its backward leaves the
// gradient of the convolution's output, compact, for a plain ring backward over those channels.
namespace tgdn {

// The gradient of the convolution's output at the q, k, v channels alone: ds = r dy - r^3 <s, dy> s, s = SiLU(conv).
__global__ void __launch_bounds__(RING_WARPS * 32, 4)
glue_norm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_g0,
                 const __grid_constant__ CUtensorMap map_g1, const __grid_constant__ CUtensorMap map_g2, RingArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bars[RING_WARPS * RING_BWD_STAGES];
  __shared__ int abort_s;
  if (threadIdx.x == 0) abort_s = 0;
  __syncthreads();
  const int wi = blockIdx.x * RING_WARPS + __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  if (wi >= a.n_warps) return;
  const RingWork w(a, wi);
  WaitCtl ctl{&abort_s, a.status};
  Ring<2, RING_BWD_STAGES> ring;
  ring.init(smem, bars);
  const int region = w.unit / a.H, head = w.unit % a.H, tiles = (w.own - w.lo + RING_ROWS - 1) / RING_ROWS;
  const CUtensorMap* map_g = region == 0 ? &map_g0 : region == 1 ? &map_g1 : &map_g2;
  auto issue = [&](int tile, uint8_t* dst, uint64_t* bar) {
    const int t = w.lo + tile * RING_ROWS;
    tma_load_3d(dst, &map_x, bar, w.unit * 128, t, w.b);
    tma_load_4d(dst + RING_TILE, map_g, bar, 0, head, t, w.b);
  };
  ring.open(tiles, issue);
  const Taps<4> taps = load_taps<4>(a.weight, w.c0, w.live);
  DocCursor doc;
  doc.init(a.cu, a.n_docs, w.lo);
  doc.advance(w.lo);
  Window<4> win;
  open_window<4>(win, a.x + w.b * a.stride_b + w.c0, a.stride_t, w.lo, max(doc.start, 0), true);
  __nv_bfloat16* out = a.out + (static_cast<int64_t>(w.b) * a.T + w.lo) * a.out_stride_t + w.c0;
  for (int tile = 0; tile < tiles; ++tile) {
    const uint8_t* xt = ring.wait(ctl);
    const int t = w.lo + tile * RING_ROWS;
#pragma unroll 4
    for (int i = 0; i < RING_ROWS; ++i) {
      if (t + i >= w.own) break;
      if (t + i >= doc.next) {
        doc.advance(t + i);
#pragma unroll
        for (int j = 0; j < 3; ++j) win.m[j] = zero_pairs<4>();
      }
      const Pairs<4> x0 = unpack<4>(ring_row(xt, i));
      Pairs<4> g = unpack<4>(ring_row(xt + RING_TILE, i)), s;
      if (region < 2) {
        float2 s2 = make_float2(0.f, 0.f), d2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float2 pre = win.conv(taps, x0, p);
          s.p[p] = make_float2(silu(pre.x), silu(pre.y));
          s2 = __ffma2_rn(s.p[p], s.p[p], s2);
          d2 = __ffma2_rn(s.p[p], g.p[p], d2);
        }
        float sums[4] = {s2.x + s2.y, d2.x + d2.y, 0.f, 0.f};
        warp_sums<4>(sums);
        const float r = rsqrtf(sums[0] + a.eps), f = -r * r * r * sums[1];
#pragma unroll
        for (int p = 0; p < 2; ++p) g.p[p] = __ffma2_rn(make_float2(f, f), s.p[p], __fmul2_rn(make_float2(r, r), g.p[p]));
      }
      store_row<4>(out, g);
      out += a.out_stride_t;
      win.push(x0);
    }
    ring.release(tiles, issue);
  }
}

struct GateArgs {
  const __nv_bfloat16* x;        // (B, T, C), element strides below
  const __nv_bfloat16* weight;
  const int32_t* cu;
  int n_docs, B, T, H, run, runs;
  int64_t stride_b, stride_t;
  float eps;
  float *k2, *q2;                // (B, T, H, E): outputs, or (backward) their gradients
  __nv_bfloat16* dy;             // backward: gradient at the gate channels, row t at dy + t * dy_stride_t (batch rows T of them apart)
  int64_t dy_stride_t;
  bool vec;                      // k2, q2 allow 16-byte accesses
};

// E consecutive bf16 / f32 in the widest pieces that E allows (the gate channels start at a multiple of E).
template <int E> struct GateRow { uint32_t w[(E + 1) / 2]; };
template <int E>
__device__ __forceinline__ GateRow<E> load_gate_row(const __nv_bfloat16* p) {
  GateRow<E> r;
  if constexpr (E % 4 == 0) {
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(p) + i);
      r.w[2 * i] = u.x; r.w[2 * i + 1] = u.y;
    }
  } else if constexpr (E == 2) {
    r.w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
  } else {
    r.w[0] = *reinterpret_cast<const unsigned short*>(p);
  }
  return r;
}

// One thread per (unit = k2 | q2 head, run of tokens): the window of its E channels stays in registers, the next row is asked for
// while the current one is used; neighbouring threads read neighbouring channels.  (One thread per token loaded every row
// four times and searched the document of every token: 97 us forward at (1, 32768) tokens, H = 32, E = 12.)
template <int E, bool BWD>
__global__ void __launch_bounds__(128)
glue_gate_kernel(GateArgs a) {
  const int units = 2 * a.H, idx = blockIdx.x * 128 + threadIdx.x;
  if (idx >= units * a.runs * a.B) return;
  const int u = idx % units, b = idx / units / a.runs, lo = idx / units % a.runs * a.run, hi = min(a.T, lo + a.run);
  const int head = u % a.H, c0 = 3 * a.H * HEAD + u * E;
  float w[E][CONV_W];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(a.weight + static_cast<int64_t>(c0 + e) * CONV_W));
    w[e][0] = bf16_lo(v.x); w[e][1] = bf16_hi(v.x); w[e][2] = bf16_lo(v.y); w[e][3] = bf16_hi(v.y);
  }
  const __nv_bfloat16* xb = a.x + b * a.stride_b + c0;
  DocCursor doc;
  doc.init(a.cu, a.n_docs, lo);
  doc.advance(lo);
  GateRow<E> m[3];                                       // x[t-1], x[t-2], x[t-3]
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    if (lo - 1 - j >= max(doc.start, 0)) {
      m[j] = load_gate_row<E>(xb + (lo - 1 - j) * a.stride_t);
    } else {
#pragma unroll
      for (int i = 0; i < (E + 1) / 2; ++i) m[j].w[i] = 0u;
    }
  }
  float* gp = (u < a.H ? a.k2 : a.q2) + ((static_cast<int64_t>(b) * a.T + lo) * a.H + head) * E;
  __nv_bfloat16* dyr = BWD ? a.dy + (static_cast<int64_t>(b) * a.T + lo) * a.dy_stride_t + u * E : nullptr;
  GateRow<E> next = load_gate_row<E>(xb + lo * a.stride_t);
  for (int t = lo; t < hi; ++t) {
    const GateRow<E> x0 = next;
    if (t + 1 < hi) next = load_gate_row<E>(xb + (t + 1) * a.stride_t);
    float g[E];
    if constexpr (BWD) {
#pragma unroll
      for (int e = 0; e < E; ++e) g[e] = gp[e];
    }
    if (t >= doc.next) {
      doc.advance(t);
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < (E + 1) / 2; ++i) m[j].w[i] = 0u;
    }
    auto at = [](const GateRow<E>& r, int e) { return (e & 1) ? bf16_hi(r.w[e / 2]) : bf16_lo(r.w[e / 2]); };
    float c[E], uu[E], ss = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      c[e] = fmaf(at(x0, e), w[e][3], fmaf(at(m[0], e), w[e][2], fmaf(at(m[1], e), w[e][1], at(m[2], e) * w[e][0])));
      uu[e] = c[e] > 15.f ? c[e] : __logf(1.f + __expf(c[e]));     // softplus; absolute error below 1e-7 at either end
      ss = fmaf(uu[e], uu[e], ss);
    }
    const float r = rsqrtf(ss + a.eps);
    if constexpr (!BWD) {
      if (E % 4 == 0 && a.vec) {
#pragma unroll
        for (int e = 0; e < E; e += 4) *reinterpret_cast<float4*>(gp + e) = make_float4(uu[e] * r, uu[e + 1] * r, uu[e + 2] * r, uu[e + 3] * r);
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) gp[e] = uu[e] * r;
      }
    } else {
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) dot = fmaf(uu[e], g[e], dot);
      const float f = -r * r * r * dot;
      float o[E];
#pragma unroll
      for (int e = 0; e < E; ++e) o[e] = fmaf(r, g[e], f * uu[e]) * fast_sigmoid(c[e]);     // d softplus = sigmoid
      if constexpr (E % 4 == 0) {
#pragma unroll
        for (int e = 0; e < E; e += 4) *reinterpret_cast<uint2*>(dyr + e) = make_uint2(pack_bf16(o[e], o[e + 1]), pack_bf16(o[e + 2], o[e + 3]));
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) dyr[e] = __float2bfloat16_rn(o[e]);
      }
      dyr += a.dy_stride_t;
    }
    gp += static_cast<int64_t>(a.H) * E;
    m[2] = m[1]; m[1] = m[0]; m[0] = x0;
  }
}

}  // namespace tgdn

using namespace tgdn;

static int glue_check(const void* x, const void* weight, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b,
                      int64_t stride_t, int H, int E, const void* q, const void* k, const void* v, const void* k2, const void* q2) {
  if (!q || !k || !v || !k2 || !q2) return TGDN_ERR_NULL;
  const int rc = conv_check_abi(x, weight, q, cu, n_docs, B, T, C, stride_b, stride_t);
  if (rc) return rc;
  if (H <= 0 || C != H * (3 * HEAD + 2 * E)) return TGDN_ERR_SHAPE;
  if (E != 1 && E != 2 && E != 4 && E != 8 && E != 12 && E != 16) return TGDN_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15) return TGDN_ERR_ALIGN;
  return tgdn_check_device() ? 0 : TGDN_ERR_DEVICE;
}
static RingArgs glue_args(const void* x, const void* weight, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b,
                          int64_t stride_t, int H, float eps, int runs) {
  RingArgs a = ring_args(x, weight, cu, n_docs, B, T, C, stride_b, stride_t, runs);
  a.units = 3 * H;                                       // one head of q, k or v each
  a.n_warps = a.units * a.runs * B;
  a.H = H;
  a.eps = eps;
  return a;
}
// Gate channels: runs of 32 tokens, shorter where that leaves the chip idle.
template <bool BWD>
static int gate_launch(const void* x, const void* weight, const int32_t* cu, int n_docs, int B, int T, int64_t stride_b, int64_t stride_t,
                       int H, int E, float eps, float* k2, float* q2, void* dy, int64_t dy_stride_t, cudaStream_t s) {
  GateArgs g{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(weight), cu, n_docs, B, T, H, 32, 0, stride_b, stride_t,
             eps, k2, q2, static_cast<__nv_bfloat16*>(dy), dy_stride_t, ((reinterpret_cast<uintptr_t>(k2) | reinterpret_cast<uintptr_t>(q2)) & 15) == 0};
  while (g.run > 8 && static_cast<int64_t>(2) * H * B * ((T + g.run - 1) / g.run) < static_cast<int64_t>(tgdn_sm_count()) * 256) g.run /= 2;
  g.runs = (T + g.run - 1) / g.run;
  const unsigned blocks = static_cast<unsigned>((static_cast<int64_t>(2) * H * B * g.runs + 127) / 128);
  switch (E) {
    case 1: glue_gate_kernel<1, BWD><<<blocks, 128, 0, s>>>(g); break;
    case 2: glue_gate_kernel<2, BWD><<<blocks, 128, 0, s>>>(g); break;
    case 4: glue_gate_kernel<4, BWD><<<blocks, 128, 0, s>>>(g); break;
    case 8: glue_gate_kernel<8, BWD><<<blocks, 128, 0, s>>>(g); break;
    case 12: glue_gate_kernel<12, BWD><<<blocks, 128, 0, s>>>(g); break;
    default: glue_gate_kernel<16, BWD><<<blocks, 128, 0, s>>>(g); break;
  }
  return tgdn_cuda_error(cudaGetLastError());
}

extern "C" int tgdn_glue_fwd(const void* x, const void* weight, const int32_t* cu_seqlens, int n_docs, int B, int T, int C,
                             int64_t stride_b, int64_t stride_t, int H, int E, float eps, void* q, void* k, void* v, float* k2,
                             float* q2, void* stream) {
  int rc = glue_check(x, weight, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, H, E, q, k, v, k2, q2);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RingArgs a = glue_args(x, weight, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, H, eps, fwd_runs(B, T, 3 * H));
  a.q = static_cast<__nv_bfloat16*>(q); a.k = static_cast<__nv_bfloat16*>(k); a.v = static_cast<__nv_bfloat16*>(v);
  if ((rc = ring_fwd_launch<true>(a, B, s))) return rc;
  return gate_launch<false>(x, weight, cu_seqlens, n_docs, B, T, stride_b, stride_t, H, E, eps, k2, q2, nullptr, 0, s);
}

static int glue_grad_maps(CUtensorMap* mg, const void* dq, const void* dk, const void* dv, int B, int T, int H) {
  const void* g[3] = {dq, dk, dv};
  for (int i = 0; i < 3; ++i)
    if (const int rc = tgdn_make_token_map(&mg[i], g[i], B, T, H, 128, RING_ROWS, 0)) return rc;
  return 0;
}

extern "C" int tgdn_glue_bwd_norm(const void* x, const void* weight, const int32_t* cu_seqlens, int n_docs, int B, int T, int C,
                                  int64_t stride_b, int64_t stride_t, int H, int E, float eps, const void* dq, const void* dk,
                                  const void* dv, const float* dk2, const float* dq2, void* dy, void* stream) {
  int rc = glue_check(x, weight, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, H, E, dq, dk, dv, dk2, dq2);
  if (rc) return rc;
  if (!dy) return TGDN_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(dy) & 15) return TGDN_ERR_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RingArgs a = glue_args(x, weight, cu_seqlens, n_docs, B, T, C, stride_b, stride_t, H, eps, fwd_runs(B, T, 3 * H));
  a.out = static_cast<__nv_bfloat16*>(dy);
  CUtensorMap mx, mg[3];
  if ((rc = glue_grad_maps(mg, dq, dk, dv, B, T, H))) return rc;
  if ((rc = tgdn_make_rows_map(&mx, x, C, T, B, stride_t, stride_b, 128, RING_ROWS))) return rc;
  static bool configured[64] = {};
  if ((rc = tgdn_dynamic_smem(reinterpret_cast<const void*>(glue_norm_kernel), RING_BWD_SMEM, configured))) return rc;
  glue_norm_kernel<<<ring_grid(a), RING_WARPS * 32, RING_BWD_SMEM, s>>>(mx, mg[0], mg[1], mg[2], a);
  if ((rc = tgdn_cuda_error(cudaGetLastError()))) return rc;
  return gate_launch<true>(x, weight, cu_seqlens, n_docs, B, T, stride_b, stride_t, H, E, eps, const_cast<float*>(dk2), const_cast<float*>(dq2),
                           static_cast<__nv_bfloat16*>(dy) + 3 * H * HEAD, C, s);
}

int tgdn_glue_bwd(const void* x, const void* weight, const int32_t* cu, int n_docs, int B, int T, int C, int64_t stride_b, int64_t stride_t,
                  int H, int E, float eps, const void* dq, const void* dk, const void* dv, const float* dk2, const float* dq2, void* dx,
                  void* dw, void* dy_gates, void* scratch, int64_t scratch_bytes, void* stream) {
  int rc = glue_check(x, weight, cu, n_docs, B, T, C, stride_b, stride_t, H, E, dq, dk, dv, dk2, dq2);
  if (rc) return rc;
  if (!dx || !dw || !dy_gates) return TGDN_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(dy_gates)) & 15) return TGDN_ERR_ALIGN;
  if (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15) || scratch_bytes < partial_bytes(B, 1, C)) return TGDN_ERR_SCRATCH;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int room = static_cast<int>(std::min<int64_t>(scratch_bytes / partial_bytes(B, 1, C), 1 << 20));
  // q, k, v channels
  RingArgs a = glue_args(x, weight, cu, n_docs, B, T, C, stride_b, stride_t, H, eps, std::min(room, bwd_runs(B, T, 3 * H)));
  a.out = static_cast<__nv_bfloat16*>(dx);
  a.dw_partial = static_cast<float*>(scratch);
  CUtensorMap mg[3];
  if ((rc = glue_grad_maps(mg, dq, dk, dv, B, T, H))) return rc;
  if ((rc = ring_bwd_launch<true>(a, B, mg, s))) return rc;
  // gate channels: the gradient of the convolution's output, then a plain backward over the same runs
  const int G = 2 * H * E, c0 = 3 * H * HEAD;
  if ((rc = gate_launch<true>(x, weight, cu, n_docs, B, T, stride_b, stride_t, H, E, eps, const_cast<float*>(dk2), const_cast<float*>(dq2),
                              dy_gates, G, s)))
    return rc;
  RingArgs g = ring_args(a.x + c0, a.weight + static_cast<int64_t>(c0) * CONV_W, cu, n_docs, B, T, G, stride_b, stride_t, a.runs);
  g.run = a.run; g.runs = a.runs; g.n_warps = g.units * g.runs * B;
  g.out = a.out + c0;
  g.out_stride_b = a.out_stride_b; g.out_stride_t = a.out_stride_t;
  g.dw_partial = a.dw_partial; g.dw_channels = C; g.dw_c0 = c0;
  if ((rc = tgdn_make_rows_map(&mg[0], dy_gates, G, T, B, G, static_cast<int64_t>(T) * G, 128, RING_ROWS))) return rc;
  if ((rc = ring_bwd_launch<false>(g, B, mg, s))) return rc;
  return reduce_dw_launch(a.dw_partial, dw, B * a.runs, C, s);
}
