// knj_stack.cu -- the resident decode stack (RMSNorm -> router -> top-k -> gate/up
// -> SiLU*up -> down -> ordered combine -> residual, layer after layer) for a decode
// batch of 1..64 tokens in ONE cooperative launch. The reference runs this loop on
// the host, one stage at a time (src/model/model.cpp:399-510 per layer, the device
// benches tools/bench/q4k_stream_ffn.hip:957-1313 between kernels).
//
// Why: a decode layer reads 21 MB (batch 1) to 340 MB (batch 64), 3 to 53 us of HBM
// time, but a chain of separate kernels pays a launch, a plan read and several
// dependent round trips per stage. Here the whole stack is one grid of one CTA per
// SM, and the four points per layer at which every CTA needs what the others
// produced (logits -> top-k, activations -> down, per-pair rows -> combine, layer
// output -> next layer) are grid barriers on a counter in global memory.
//
// Arithmetic. Logits and RMS statistics repeat moe_front_kernel's operation order
// exactly, so routing decisions are the same bits as the layer launches'. The expert
// projections run on the tile engine of knj_q4k_engine.cuh (exact integer products
// on the fp16 tensor cores, f32 results); the combine adds the k weighted rows of a
// token in ascending expert order from zero and the residual last, like
// combine_kernel and the CPU path (src/model/model.cpp:455-463, :652).
//
// Every wait is bounded: a barrier or a copy that does not complete within the
// limit sets the error word, every CTA that sees it returns, and
// knj_moe_stack_status reports KNJ_E_TIMEOUT. A copy is waited for by one warp,
// which raises the CTA's fail word; the next grid barrier turns that into the
// error word, whichever warp it was.
#include "knj_common.cuh"
#include "knj_q4k.h"
#include "knj_q4k_engine.cuh"
#include "knj_q6k_block.cuh"
#include "knj_topk.cuh"

#include <algorithm>
#include <type_traits>
#include <vector>

using namespace knj;

namespace {

constexpr int kMaxT = 64;  // tokens per step
constexpr int kThreads = q4e::kWarps * 32;
constexpr int kSplitMaxT = 16;  // batches up to this size may split a tile's K range over several warps
constexpr int kMaxSlices = 8;  // hidden <= 2048: the logits keep a router row in registers
constexpr int kMaxF6 = 1024;   // ffn of layers with Q6_K down matrices: as the prefill launch takes them, and as far as it is tested

struct LayerMaps {  // stay in global memory: the TMA unit reads them there
  CUtensorMap mg, mu, md;  // gate, up, down weights as TMA boxes of the projection phases
};
struct LayerDesc {  // copied to shared memory one layer ahead
  const void *x;
  void *out;
  const __nv_bfloat16 *Wr;
  const float *bias;
  const __nv_bfloat16 *norm_w;
  const uint8_t *w_down6;  // non-null: the layer's down matrices are Q6_K [E][H][F/256][210] (no TMA map for them)
  int32_t *tap_exp;
  float *tap_w;
  int64_t ldx, ldo;
  float eps;
  int residual, x_dtype, out_dtype;
};
static_assert(sizeof(LayerDesc) % 4 == 0, "copied by words");

struct StackParams {
  const LayerMaps *maps;
  const LayerDesc *layers;
  int n_layers, T, H, F, E, k;
  float *logits;       // [T][E]
  float *scales;       // [T] RMSNorm scale of the layer's rows
  float *act;          // [T*k][F]
  float *Y;            // [T*k][H]
  unsigned int *sync;  // [0] arrivals, [1] error word; both zero before the launch
  q4e::PhaseShape gu, dn;
  long long wait_cycles;  // limit of every wait inside the kernel
  int stall;              // test hook: added to the first barrier's target, which then cannot complete
  int stall_copy;         // test hook: w + 1 = the first copies of CTA 0's warp w never count as landed
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(unsigned *p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid barrier in two halves, so that work that does not depend on the other CTAs can sit between them.
// arrive: everything this CTA wrote so far is published. wait: all CTAs of the grid have arrived `target`
// times in total; false: a wait ran out, this one, one elsewhere in the grid, or that for a copy of any warp of this
// CTA (*fail, ordered by the CTA barrier of grid_arrive).
__device__ __forceinline__ void grid_arrive(unsigned *sync) {
  __syncthreads();
  if (threadIdx.x == 0) red_release(sync, 1u);  // cumulative: releases what the CTA barrier ordered before it
}
__device__ __forceinline__ bool grid_wait(unsigned *sync, volatile const int *fail, unsigned target, long long limit) {
  int ok = 1;
  if (threadIdx.x == 0) {
    const long long t0 = clock64();
    unsigned polls = 0;
    if (*fail) {
      atomicExch(sync + 1, 1u);
      ok = 0;
    }
    while (ok && ld_acquire(sync) < target) {
      if ((++polls & 63u) == 0u) {
        if (ld_acquire(sync + 1) != 0u) { ok = 0; break; }
        if (clock64() - t0 > limit) { atomicExch(sync + 1, 1u); ok = 0; break; }
      }
    }
  }
  return __syncthreads_and(ok) != 0;
}

// Shared-memory plan (byte offsets into the dynamic block).
struct Plan {
  uint32_t ring, panels, bars, sel_e, sel_w, mask, jbase, uexp, inv, pair, scale, ord, fail, desc, red, total;
};
__host__ __device__ inline Plan make_plan(const q4e::PhaseShape &gu, const q4e::PhaseShape &dn, int T, int k) {
  Plan pl;
  uint32_t o = 0;
  auto take = [&](size_t bytes) { const uint32_t at = o; o += (uint32_t)((bytes + 127) & ~(size_t)127); return at; };
  const size_t ring = max(q4e::phase_ring_bytes(gu.sbs, gu.stages), q4e::phase_ring_bytes(dn.sbs, dn.stages));
  const size_t panels = max(q4e::phase_panel_bytes(gu.nsb), q4e::phase_panel_bytes(dn.nsb));
  pl.ring = take(ring);
  pl.panels = take(panels);
  pl.bars = take((size_t)q4e::kWarps * q4e::kMaxStages * 8);
  pl.sel_e = take((size_t)T * k * 4);
  pl.sel_w = take((size_t)T * k * 4);
  pl.mask = take(256 * 8);
  pl.jbase = take(257 * 4);
  pl.uexp = take(256 * 4);
  pl.inv = take(q4e::kJobTok * 16 * 4);
  pl.pair = take(q4e::kJobTok * 4);
  pl.scale = take((size_t)T * 4);
  pl.ord = take((size_t)T * k);
  pl.fail = take(32);
  pl.desc = take(2 * sizeof(LayerDesc));
  // partial sums of warps that share a tile: only small batches have so few tiles that they do
  pl.red = T <= kSplitMaxT ? take((size_t)q4e::kWarps * 32 * sizeof(float4)) : 0;
  pl.total = o;
  return pl;
}

// Warps that take tiles in a Q6_K down phase: each needs a buffer for one whole tile, which lie in the ring and panel areas
// (the phase engine is idle) in front of the phase's own panel. Three superblocks a row (ffn 768) leave room for 14 warps at
// hidden 512 and 16 at hidden 2048, four for 11 and 12. 0: the areas do not hold a panel and one tile.
__host__ __device__ inline int down6_warps(const Plan &pl, int nsb) {
  const size_t room = pl.bars - pl.ring, panel = q6b::tile_panel_bytes(nsb);
  if (room < panel) return 0;
  const int fit = (int)((room - panel) / q6b::tile_bytes(nsb));
  return fit < q4e::kWarps ? fit : q4e::kWarps;
}

__device__ __forceinline__ void load8_bf16(const __nv_bfloat16 *p, float (&v)[8]) {
  const uint4 r = __ldg(reinterpret_cast<const uint4 *>(p));
  const uint32_t u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = __uint_as_float(u[j] << 16);
    v[2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
  }
}

#ifdef KNJ_TRACE
// Measurement build only: global-timer stamps of one CTA's stages in layer 1 (layer 0 of a one-layer stack).
__device__ unsigned long long g_stack_trace[16 * 160];
#define KNJ_STAMP(i) do { if (threadIdx.x == 0 && l == trace_layer) g_stack_trace[blockIdx.x * 16 + (i)] = global_timer_ns(); } while (0)
#else
#define KNJ_STAMP(i)
#endif

// Stage 1 of a layer for one CTA item: experts epi * eg .. + epi - 1 times tokens 8 tg .. 8 tg + 7; warp w takes
// expert w % epi and the token slot w / epi (epi / 2 tokens, at least one). epi = 8, 4, 2 or 1: fewer experts per
// item for smaller batches, so that the items still cover most of the grid. Row statistics and logits in moe_front_kernel's operation order (lane owns
// elements 256 sl + 8 lane + j, even/odd chains, warp_sum). The CTA first brings its eight router rows (times the
// norm weights, f32) and its token rows (as they are) into shared memory with every load in flight at once;
// scratch: 8 * H * 4 bytes for the router rows followed by 8 * H * 4 for the token rows.
__device__ __noinline__ void stage_logits(const StackParams &p, const LayerDesc &L, int epi, int eg, int tg, uint8_t *scratch,
                                          int l, int trace_layer) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int T = p.T, H = p.H, E = p.E, nslice = H / 256;
  const bool has_norm = L.norm_w != nullptr;
  float *wr_s = reinterpret_cast<float *>(scratch);
  uint8_t *rows_s = scratch + (size_t)8 * H * 4;
  const int esz = L.x_dtype == KNJ_DT_F32 ? 4 : 2, row_bytes = H * esz, cpr = row_bytes / 16;
  const int nt = min(8, T - tg * 8);
  // ---- loads first (router rows, norm weights, token rows), conversions after
  const int wchunks = epi * (H / 8);  // 16-byte pieces of the item's bf16 router rows
  constexpr int kPer = (8 * 256 * kMaxSlices / 8 + kThreads - 1) / kThreads;  // 4 pieces per thread at H = 2048
  uint4 wraw[kPer], nraw[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = threadIdx.x + q * kThreads;
    if (i < wchunks) {
      const int r = i / (H / 8), ch = i - r * (H / 8);
      const int ee = min(eg * epi + r, E - 1);
      wraw[q] = __ldg(reinterpret_cast<const uint4 *>(L.Wr + (size_t)ee * H + 8 * ch));
      if (has_norm) nraw[q] = __ldg(reinterpret_cast<const uint4 *>(L.norm_w + 8 * ch));
    }
  }
  // the token rows as asynchronous copies (through L2): all under way at once and no registers held (a loop of load and
  // store cost up to eight trips to L2)
  for (int i = threadIdx.x; i < nt * cpr; i += kThreads) {
    const int r = i / cpr, ch = i - r * cpr;
    const uint8_t *src = static_cast<const uint8_t *>(L.x) + (int64_t)(tg * 8 + r) * L.ldx * esz + 16 * ch;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(rows_s + (size_t)16 * i)), "l"(src) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int i = threadIdx.x + q * kThreads;
    if (i < wchunks) {
      const uint32_t w[4] = {wraw[q].x, wraw[q].y, wraw[q].z, wraw[q].w}, n[4] = {nraw[q].x, nraw[q].y, nraw[q].z, nraw[q].w};
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[2 * j] = __uint_as_float(w[j] << 16);
        v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        if (has_norm) {
          v[2 * j] *= __uint_as_float(n[j] << 16);
          v[2 * j + 1] *= __uint_as_float(n[j] & 0xffff0000u);
        }
      }
      *reinterpret_cast<float4 *>(wr_s + (size_t)8 * i) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4 *>(wr_s + (size_t)8 * i + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  KNJ_STAMP(11);
  const int es = warp % epi, tpw = max(1, epi / 2);
  const int e = eg * epi + es;
  const int t_first = tg * 8 + (warp / epi) * tpw, t_end = min(min(T, tg * 8 + 8), t_first + tpw);
  const float bias = (L.bias && e < E) ? L.bias[e] : 0.f;
  const float *wrow = wr_s + (size_t)es * H;
  // two tokens per pass over the router row: their chains are independent of each other
  for (int t = t_first; t < t_end; t += 2) {
    const bool second = t + 1 < t_end;
    float d0[2] = {0.f, 0.f}, d1[2] = {0.f, 0.f}, s0[2] = {0.f, 0.f}, s1[2] = {0.f, 0.f};
#pragma unroll
    for (int sl = 0; sl < kMaxSlices; ++sl) {
      if (sl < nslice) {
        const float4 wa = *reinterpret_cast<const float4 *>(wrow + 256 * sl + 8 * lane);
        const float4 wb = *reinterpret_cast<const float4 *>(wrow + 256 * sl + 8 * lane + 4);
        const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint8_t *row = rows_s + (size_t)(t + (second ? u : 0) - tg * 8) * row_bytes;
          float v[8];
          if (esz == 4) {
            const float4 a = *reinterpret_cast<const float4 *>(row + (256 * sl + 8 * lane) * 4);
            const float4 b = *reinterpret_cast<const float4 *>(row + (256 * sl + 8 * lane) * 4 + 16);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
          } else {
            const uint4 r = *reinterpret_cast<const uint4 *>(row + (256 * sl + 8 * lane) * 2);
            const uint32_t x4[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[2 * j] = __uint_as_float(x4[j] << 16);
              v[2 * j + 1] = __uint_as_float(x4[j] & 0xffff0000u);
            }
          }
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            d0[u] = fmaf(w[j], v[j], d0[u]);
            d1[u] = fmaf(w[j + 1], v[j + 1], d1[u]);
            s0[u] = fmaf(v[j], v[j], s0[u]);
            s1[u] = fmaf(v[j + 1], v[j + 1], s1[u]);
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 && !second) break;
      const float dot = warp_sum(d0[u] + d1[u]), ss = warp_sum(s0[u] + s1[u]);
      if (lane == 0) {
        const float scale = has_norm ? 1.0f / sqrtf(ss / (float)H + L.eps) : 1.0f;
        if (eg == 0 && es == 0) p.scales[t + u] = scale;
        if (e < E) p.logits[(size_t)(t + u) * E + e] = dot * scale + bias;
      }
    }
  }
}

// Stage 2 of a layer, by every CTA for itself: top-k of every token, the per-expert token sets (bit masks), the
// order of a token's slots for the weighted sum, and the job table of the projection stages.
__device__ __noinline__ void stage_plan(const StackParams &p, const LayerDesc &L, const Plan &pl, uint8_t *smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int T = p.T, E = p.E, k = p.k, P = T * k, c = blockIdx.x;
  int *sel_e = reinterpret_cast<int *>(smem + pl.sel_e);
  float *sel_w = reinterpret_cast<float *>(smem + pl.sel_w);
  unsigned long long *mask = reinterpret_cast<unsigned long long *>(smem + pl.mask);
  int *jbase = reinterpret_cast<int *>(smem + pl.jbase), *uexp = reinterpret_cast<int *>(smem + pl.uexp);
  float *scale_s = reinterpret_cast<float *>(smem + pl.scale);
  unsigned char *ord = smem + pl.ord;
    for (int t = threadIdx.x; t < T; t += kThreads) scale_s[t] = __ldcg(p.scales + t);
    for (int a = threadIdx.x; a < 256; a += kThreads) mask[a] = 0ull;
    auto select = [&](auto epl, auto group) {  // tokens warp, warp + 16, ...: `group` of them at a time
      constexpr int kEpl = decltype(epl)::value, kNt = decltype(group)::value;
#pragma unroll 1
      for (int t0 = warp; t0 < T; t0 += q4e::kWarps * kNt) {
        float v[kNt][kEpl], w[kNt];
        int e[kNt];
#pragma unroll
        for (int n = 0; n < kNt; ++n) topk_load<kEpl>(p.logits + (size_t)min(t0 + q4e::kWarps * n, T - 1) * E, E, lane, v[n]);
        warp_topk<kEpl, kNt>(v, E, k, lane, e, w);
#pragma unroll
        for (int n = 0; n < kNt; ++n) {
          const int t = t0 + q4e::kWarps * n;
          if (t < T && lane < k) {
            sel_e[t * k + lane] = e[n];
            sel_w[t * k + lane] = w[n];
            if (c == 0 && L.tap_exp) L.tap_exp[t * k + lane] = e[n];
            if (c == 0 && L.tap_w) L.tap_w[t * k + lane] = w[n];
          }
        }
      }
    };
    using std::integral_constant;
    // A token alone is latency (1.8 us), so a warp's tokens go together: two up to 32 tokens, four above (a layer of 64
    // tokens 2 us shorter than one after the other); a second and fourth token that do not exist repeat the last one.
    if (E > 128) select(integral_constant<int, kMaxEPerLane>{}, integral_constant<int, 1>{});
    else if (T <= q4e::kWarps) select(integral_constant<int, 4>{}, integral_constant<int, 1>{});
    else if (T <= 2 * q4e::kWarps) select(integral_constant<int, 4>{}, integral_constant<int, 2>{});
    else select(integral_constant<int, 4>{}, integral_constant<int, 4>{});
    __syncthreads();
    for (int pr = threadIdx.x; pr < P; pr += kThreads) {
      const int t = pr / k, e = sel_e[pr];
      atomicOr(&mask[e], 1ull << t);
      int r = 0;  // a token's slots in ascending expert order (the order of the weighted sum)
      for (int j = 0; j < k; ++j) r += sel_e[t * k + j] < e ? 1 : 0;
      ord[t * k + r] = (unsigned char)(pr - t * k);
    }
    __syncthreads();
    if (warp == 0) {
      int cnt[8], nact = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = 8 * lane + i;
        cnt[i] = e < E ? __popcll(mask[e]) : 0;
        nact += cnt[i] > 0 ? 1 : 0;
      }
      int incl = nact;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      int pos = incl - nact;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (cnt[i] > 0) {
          uexp[pos] = 8 * lane + i;
          jbase[pos] = (cnt[i] + q4e::kJobTok - 1) / q4e::kJobTok;
          ++pos;
        }
      for (int a = total + lane; a < 256; a += 32) {
        uexp[a] = -1;
        jbase[a] = 0;
      }
      __syncwarp();
      q4e::job_prefix(jbase, lane);
    }
    __syncthreads();

}

// Down phase of a layer whose down matrices are Q6_K: the CTA's run of the flat (job, 16-row tile) list, as in the Q4_K
// engine, with q6b's whole tiles: a warp copies a tile of its own (10 KB at ffn 768), multiplies it and asks for the next.
// The buffers lie in the ring area and the panel behind them; where sixteen do not fit fewer warps take tiles (down6_warps).
// Before, blocks of 64 rows were staged and reduced by the whole CTA, three CTA barriers each: 45 us on the mean and 60 to
// the last CTA at 8 tokens (51 experts, 66 MB, 10 us of HBM time), where the Q4_K phase takes 18; a layer of a stack of 48
// was 102 us and is 80.4, one with Q4_K down matrices 69.9.
__device__ __noinline__ void stage_down_q6k(const StackParams &p, const LayerDesc &L, const Plan &pl, uint8_t *smem, unsigned &parity_io,
                                            bool &ok_io) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int H = p.H, F = p.F, k = p.k, c = blockIdx.x, G = gridDim.x, tiles = p.dn.tiles, nsb = p.dn.nsb;
  const int *sel_e = reinterpret_cast<const int *>(smem + pl.sel_e);
  const unsigned long long *mask = reinterpret_cast<const unsigned long long *>(smem + pl.mask);
  const int *jbase = reinterpret_cast<const int *>(smem + pl.jbase), *uexp = reinterpret_cast<const int *>(smem + pl.uexp);
  float *inv = reinterpret_cast<float *>(smem + pl.inv);
  int *s_pair = reinterpret_cast<int *>(smem + pl.pair);
  volatile int *fail = reinterpret_cast<volatile int *>(smem + pl.fail);
  const uint32_t tb = (uint32_t)q6b::tile_bytes(nsb);
  const int nw = down6_warps(pl, nsb);
  uint8_t *buf = smem + pl.ring + (size_t)warp * tb, *panel = smem + pl.ring + (size_t)nw * tb;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + pl.bars) + warp * q4e::kMaxStages;
  static_assert(q6b::kTileTok == q4e::kJobTok, "one job table");
  const long long U = (long long)jbase[256] * tiles;
  const int u0 = (int)(U * c / G), u1 = (int)(U * (c + 1) / G);
  if (u0 >= u1) return;
  unsigned parity = parity_io;
  bool ok = ok_io;
  for (int job = u0 / tiles; job <= (u1 - 1) / tiles; ++job) {
    const int a = q4e::job_locate(jbase, job), e = uexp[a];
    const int r0 = max(u0, job * tiles), r1 = min(u1, (job + 1) * tiles);
    const uint8_t *src = L.w_down6 + ((size_t)e * H - (size_t)job * tiles * 16) * (tb / 16);
    auto issue = [&](int tile) {
      if (lane == 0 && ok) {
        fence_proxy_async();  // the buffer was read through the generic proxy
        mbar_expect_tx(bar, tb);
        bulk_g2s(buf, src + (size_t)tile * tb, tb, bar);
      }
    };
    int tile = warp < nw ? r0 + warp : r1;
    if (tile < r1) issue(tile);
    __syncthreads();  // the previous job's tiles are done with the panel
    // ---- the job's tokens: the (4 (job - first job of the expert))-th and following of the expert's set
    for (int item = warp; item < q4e::kJobTok * nsb; item += q4e::kWarps) {
      const int sb = item % nsb, tk = item / nsb, idx = (job - jbase[a]) * q4e::kJobTok + tk;
      unsigned long long m = mask[e];
      int pair = -1;
      if (idx < __popcll(m)) {
        for (int i = 0; i < idx; ++i) m &= m - 1ull;
        const int tok = __ffsll((long long)m) - 1;
        for (int j = 0; j < k; ++j) pair = sel_e[tok * k + j] == e ? tok * k + j : pair;
        float v[8];
        q4e::load8_f32(p.act, KNJ_DT_F32, (int64_t)pair * F + 256 * sb + 8 * lane, v);
        const float iv = q6b::tile_panel_convert(v, panel, sb, tk, lane);
        if (lane == 0) inv[tk * 16 + sb] = iv;
      }
      if (sb == 0 && lane == 0) s_pair[tk] = pair;
    }
    __syncthreads();
    for (; tile < r1; tile += nw) {
      if (ok && !mbar_wait_for(bar, parity & 1u, p.wait_cycles, fail)) ok = false;
      parity ^= 1u;
      float y0, y1;
      q6b::tile_mma(buf, panel, inv + t * 16, nsb, lane, y0, y1);  // whatever each lane's wait came to: as in run_phase
      __syncwarp();  // every lane is done with the buffer
      if (tile + nw < r1) issue(tile + nw);
      const int pair = s_pair[t];
      if (ok && pair >= 0) {
        float *y = p.Y + (size_t)pair * H + (tile - job * tiles) * 16 + g;
        y[0] = y0;
        y[8] = y1;
      }
    }
  }
  parity_io = parity;
  ok_io = ok;
  __syncthreads();  // the ring area returns to the projection phases
}

__global__ void __launch_bounds__(kThreads, 1) moe_stack_kernel(const StackParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int T = p.T, H = p.H, F = p.F, E = p.E, k = p.k;
  const int G = gridDim.x, c = blockIdx.x;
  const Plan pl = make_plan(p.gu, p.dn, T, k);
  int *sel_e = reinterpret_cast<int *>(smem + pl.sel_e);
  float *sel_w = reinterpret_cast<float *>(smem + pl.sel_w);
  unsigned long long *mask = reinterpret_cast<unsigned long long *>(smem + pl.mask);
  int *jbase = reinterpret_cast<int *>(smem + pl.jbase), *uexp = reinterpret_cast<int *>(smem + pl.uexp);
  float *scale_s = reinterpret_cast<float *>(smem + pl.scale);
  unsigned char *ord = smem + pl.ord;
  int *s_fail = reinterpret_cast<int *>(smem + pl.fail);
  q4e::PhaseSmem sm;
  sm.ring = smem + pl.ring;
  sm.panels = smem + pl.panels;
  sm.bars = reinterpret_cast<uint64_t *>(smem + pl.bars);
  sm.inv = reinterpret_cast<float *>(smem + pl.inv);
  sm.pair = reinterpret_cast<int *>(smem + pl.pair);
  sm.fail = s_fail;
  sm.red = reinterpret_cast<float4 *>(smem + pl.red);
  const q4e::JobTable jt{jbase, uexp};

  if (lane == 0)
    for (int s = 0; s < q4e::kMaxStages; ++s) mbar_init(&sm.bars[warp * q4e::kMaxStages + s], c == 0 && s == 0 && warp + 1 == p.stall_copy ? 2 : 1);
  if (threadIdx.x == 0) *s_fail = 0;
  mbar_init_fence();
  __syncthreads();

  unsigned arrivals = 0, parity = 0;
  bool ok = true;
  // logits: CTA c < n_eg * n_tg takes experts epi * eg .. + epi - 1 for tokens 8 tg .. 8 tg + 7
  const int n_tg = (T + 7) / 8;
  int epi = 8;
  while (epi > 1 && n_tg * ((E + epi / 2 - 1) / (epi / 2)) <= G) epi >>= 1;
  const int n_eg = (E + epi - 1) / epi;
  const bool has_item = c < n_eg * n_tg;
  const int eg = c % n_eg, tg = c / n_eg;

#ifdef KNJ_TRACE
  const int trace_layer = p.n_layers > 1 ? 1 : 0;
#endif
  // the layers' descriptions are read from shared memory; the next layer's arrives while the current one computes
  LayerDesc *descs = reinterpret_cast<LayerDesc *>(smem + pl.desc);
  auto stage_desc = [&](int l) {
    if (threadIdx.x < sizeof(LayerDesc) / 4)
      reinterpret_cast<uint32_t *>(&descs[l & 1])[threadIdx.x] = reinterpret_cast<const uint32_t *>(p.layers + l)[threadIdx.x];
  };
  stage_desc(0);
  __syncthreads();
  for (int l = 0; l < p.n_layers; ++l) {
    const LayerDesc &L = descs[l & 1];
    const LayerMaps &M = p.maps[l];
    const bool has_norm = L.norm_w != nullptr;
    if (l + 1 < p.n_layers) stage_desc(l + 1);  // published by the CTA barriers of this layer
    KNJ_STAMP(0);

    // ---- stage 1: row statistics and router logits
#ifdef KNJ_TRACE
    if (has_item) stage_logits(p, L, epi, eg, tg, smem + pl.ring, l, trace_layer);
#else
    if (has_item) stage_logits(p, L, epi, eg, tg, smem + pl.ring, l, 0);
#endif
    KNJ_STAMP(1);
    arrivals += G;
    grid_arrive(p.sync);
    if (!grid_wait(p.sync, s_fail, arrivals + (l == 0 ? (unsigned)p.stall : 0u), p.wait_cycles)) return;
    KNJ_STAMP(2);

    // ---- stage 2: top-k per token (every CTA for itself), the per-expert token sets, the job table
    stage_plan(p, L, pl, smem);

    // token slot tk of a job: the (4 (job - first job of the expert) + tk)-th token of the expert's set
    auto job_tok = [&](int job, int a, int tk, int &e_out) {
      const int e = uexp[a];
      unsigned long long m = mask[e];
      const int idx = (job - jbase[a]) * q4e::kJobTok + tk;
      e_out = e;
      if (idx >= __popcll(m)) return -1;
      for (int i = 0; i < idx; ++i) m &= m - 1ull;
      return __ffsll((long long)m) - 1;
    };
    auto pair_of = [&](int tok, int e) {
      int s = 0;
      for (int j = 0; j < k; ++j) s = sel_e[tok * k + j] == e ? j : s;
      return tok * k + s;
    };

    KNJ_STAMP(3);
    // ---- stage 3: gate, up, SiLU*up -> act
    {
      const long long U = (long long)jbase[256] * p.gu.tiles;
      const int u0 = (int)(U * c / G), u1 = (int)(U * (c + 1) / G);
      q4e::run_phase<true>(
          p.gu, sm, jt, u0, u1, T <= kSplitMaxT ? q4e::choose_ksplit(U, p.gu.nsb / p.gu.sbs, G) : 1, &M.mg, &M.mu, nullptr, nullptr, p.act, p.wait_cycles, parity, ok,
          [&](int job, int a, int tk, int &pair, int &row) {
            int e;
            const int tok = job_tok(job, a, tk, e);
            if (tok < 0) return false;
            pair = pair_of(tok, e);
            row = tok;
            return true;
          },
          [&](int row, int sb, int ln, float (&v)[8]) {
            q4e::load8_f32(L.x, L.x_dtype, (int64_t)row * L.ldx + 256 * sb + 8 * ln, v);
            if (has_norm) {
              float nw[8];
              load8_bf16(L.norm_w + 256 * sb + 8 * ln, nw);
              const float sc = scale_s[row];
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(__fmul_rn(v[j], sc), nw[j]);
            }
          });
    }
    KNJ_STAMP(4);
    arrivals += G;
    grid_arrive(p.sync);
    if (!grid_wait(p.sync, s_fail, arrivals, p.wait_cycles)) return;
    KNJ_STAMP(5);

    // ---- stage 4: down -> Y (one row per pair)
    if (L.w_down6) stage_down_q6k(p, L, pl, smem, parity, ok);
    else {
      const long long U = (long long)jbase[256] * p.dn.tiles;
      const int u0 = (int)(U * c / G), u1 = (int)(U * (c + 1) / G);
      q4e::run_phase<false>(
          p.dn, sm, jt, u0, u1, T <= kSplitMaxT ? q4e::choose_ksplit(U, p.dn.nsb / p.dn.sbs, G) : 1, &M.md, &M.md, p.Y, nullptr, nullptr, p.wait_cycles, parity, ok,
          [&](int job, int a, int tk, int &pair, int &row) {
            int e;
            const int tok = job_tok(job, a, tk, e);
            if (tok < 0) return false;
            pair = pair_of(tok, e);
            row = pair;
            return true;
          },
          [&](int row, int sb, int ln, float (&v)[8]) { q4e::load8_f32(p.act, KNJ_DT_F32, (int64_t)row * F + 256 * sb + 8 * ln, v); });
    }
    KNJ_STAMP(6);
    arrivals += G;
    grid_arrive(p.sync);
    if (!grid_wait(p.sync, s_fail, arrivals, p.wait_cycles)) return;
    KNJ_STAMP(7);

    // ---- stage 5: ordered weighted sum of a token's k rows, residual last, four columns per thread
    {
      const int H4 = H / 4, items = T * H4;
      for (int i = c * kThreads + threadIdx.x; i < items; i += G * kThreads) {
        const int t = i / H4, n = 4 * (i - t * H4);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < k; ++s) {
          const int pr = t * k + ord[t * k + s];
          const float w = sel_w[pr];
          const float4 y = __ldcg(reinterpret_cast<const float4 *>(p.Y + (size_t)pr * H + n));
          acc.x = __fadd_rn(acc.x, __fmul_rn(w, y.x));
          acc.y = __fadd_rn(acc.y, __fmul_rn(w, y.y));
          acc.z = __fadd_rn(acc.z, __fmul_rn(w, y.z));
          acc.w = __fadd_rn(acc.w, __fmul_rn(w, y.w));
        }
        if (L.residual) {
          float r[4];
          if (L.x_dtype == KNJ_DT_F32) {
            const float4 xv = __ldcg(reinterpret_cast<const float4 *>(static_cast<const float *>(L.x) + (int64_t)t * L.ldx + n));
            r[0] = xv.x; r[1] = xv.y; r[2] = xv.z; r[3] = xv.w;
          } else {
            const uint2 xv = __ldcg(reinterpret_cast<const uint2 *>(static_cast<const unsigned short *>(L.x) + (int64_t)t * L.ldx + n));
            r[0] = __uint_as_float(xv.x << 16); r[1] = __uint_as_float(xv.x & 0xffff0000u);
            r[2] = __uint_as_float(xv.y << 16); r[3] = __uint_as_float(xv.y & 0xffff0000u);
          }
          acc.x = __fadd_rn(r[0], acc.x); acc.y = __fadd_rn(r[1], acc.y);
          acc.z = __fadd_rn(r[2], acc.z); acc.w = __fadd_rn(r[3], acc.w);
        }
        if (L.out_dtype == KNJ_DT_F32) {
          *reinterpret_cast<float4 *>(static_cast<float *>(L.out) + (int64_t)t * L.ldo + n) = acc;
        } else {
          __nv_bfloat16 *o = static_cast<__nv_bfloat16 *>(L.out) + (int64_t)t * L.ldo + n;
          const __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
          *reinterpret_cast<uint2 *>(o) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
        }
      }
    }
    KNJ_STAMP(8);
    if (l + 1 < p.n_layers) {
      arrivals += G;
      grid_arrive(p.sync);
      if (!grid_wait(p.sync, s_fail, arrivals, p.wait_cycles)) return;
    }
    KNJ_STAMP(9);
  }
}

}  // namespace

namespace {
int g_force_big_stack = 0;  // measurement builds: run the tensor-core kernel for the smallest batches too
}

struct knj_moe_stack {
  SmallStack *small = nullptr;  // batches of at most kSmallStackMaxTokens run the scalar-FMA kernel instead
  StackParams p{};
  void *dev_block = nullptr;  // layer table, logits, scales, activations, per-pair rows, sync words
  size_t smem = 0;
  int grid = 0;
  int device = 0;
};

extern "C" {

int knj_moe_stack_create(const knj_moe_ffn_args *layers, int n_layers, knj_moe_stack **out) {
  KNJ_REQUIRE(layers && out && n_layers > 0, "knj_moe_stack_create: null argument or no layers");
  *out = nullptr;
  const knj_moe_ffn_args &a0 = layers[0];
  const int T = a0.n_tokens, H = a0.hidden, F = a0.ffn, E = a0.n_experts, k = a0.top_k;
  KNJ_REQUIRE(T >= 1 && T <= kMaxT, "knj_moe_stack_create: n_tokens=%d, this launch takes 1..%d", T, kMaxT);
  bool any_q6k = false;  // the scalar kernel of the smallest batches takes Q4_K down matrices only
  for (int l = 0; l < n_layers; ++l) any_q6k = any_q6k || layers[l].down_format == 1;
  if (T <= kSmallStackMaxTokens && !g_force_big_stack && !any_q6k) {
    SmallStack *sm = nullptr;
    const int rc = small_stack_create(layers, n_layers, &sm);
    if (rc) return rc;
    knj_moe_stack *st = new knj_moe_stack();
    st->small = sm;
    *out = st;
    return KNJ_OK;
  }
  KNJ_REQUIRE(H > 0 && H % 256 == 0 && H <= 256 * kMaxSlices, "knj_moe_stack_create: hidden=%d must be a multiple of 256, at most %d", H,
              256 * kMaxSlices);
  KNJ_REQUIRE(F > 0 && F % 256 == 0 && F <= 4096, "knj_moe_stack_create: ffn=%d must be a multiple of 256, at most 4096", F);
  KNJ_REQUIRE(!any_q6k || F <= kMaxF6, "knj_moe_stack_create: ffn=%d: layers with Q6_K down matrices are taken up to ffn %d", F, kMaxF6);
  KNJ_REQUIRE(k >= 1 && k <= 8 && k <= E && E <= 256, "knj_moe_stack_create: top_k=%d / n_experts=%d out of range", k, E);
  StackParams sp{};
  sp.gu.N = F; sp.gu.nsb = H / 256; sp.gu.sbs = (sp.gu.nsb % 2 == 0) ? 2 : 1; sp.gu.tiles = F / 8;
  sp.dn.N = H; sp.dn.nsb = F / 256; sp.dn.sbs = (sp.dn.nsb % 2 == 0) ? 2 : 1; sp.dn.tiles = H / 16;
  sp.gu.stages = sp.gu.sbs == 2 ? 2 : q4e::kMaxStages;
  sp.dn.stages = sp.dn.sbs == 2 ? 2 : q4e::kMaxStages;
  std::vector<LayerDesc> table(n_layers);
  std::vector<LayerMaps> maps(n_layers);
  for (int l = 0; l < n_layers; ++l) {
    const knj_moe_ffn_args &a = layers[l];
    KNJ_REQUIRE(a.n_tokens == T && a.hidden == H && a.ffn == F && a.n_experts == E && a.top_k == k,
                "knj_moe_stack_create: layer %d differs in shape from layer 0", l);
    KNJ_REQUIRE(a.x && a.out && a.w_router && a.w_gate && a.w_up && a.w_down, "knj_moe_stack_create: layer %d: null tensor pointer", l);
    KNJ_REQUIRE(a.down_format == 0 || a.down_format == 1, "knj_moe_stack_create: layer %d: unknown format of the down matrices", l);
    KNJ_REQUIRE(a.x_dtype == KNJ_DT_F32 || a.x_dtype == KNJ_DT_BF16, "knj_moe_stack_create: layer %d: x must be f32 or bf16", l);
    KNJ_REQUIRE(a.out_dtype == KNJ_DT_F32 || a.out_dtype == KNJ_DT_BF16, "knj_moe_stack_create: layer %d: out must be f32 or bf16", l);
    KNJ_REQUIRE(a.ldx >= H && a.ldo >= H && a.ldx % 8 == 0 && a.ldo % 4 == 0, "knj_moe_stack_create: layer %d: bad row strides", l);
    auto al16 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    KNJ_REQUIRE(al16(a.x) && al16(a.out) && al16(a.w_router) && al16(a.w_gate) && al16(a.w_up) && al16(a.w_down) &&
                    (!a.norm_w || al16(a.norm_w)),
                "knj_moe_stack_create: layer %d: x, out, router, norm and expert bases must be 16-byte aligned", l);
    KNJ_REQUIRE(a.x != a.out, "knj_moe_stack_create: layer %d: out must not alias x (other CTAs still read x)", l);
    LayerDesc &s = table[l];
    LayerMaps &m = maps[l];
    int rc = make_row_tensor_map(&m.mg, a.w_gate, (uint64_t)E * F, (uint32_t)sp.gu.nsb * KNJ_Q4K_BYTES, (uint32_t)sp.gu.sbs * KNJ_Q4K_BYTES, 8);
    if (!rc) rc = make_row_tensor_map(&m.mu, a.w_up, (uint64_t)E * F, (uint32_t)sp.gu.nsb * KNJ_Q4K_BYTES, (uint32_t)sp.gu.sbs * KNJ_Q4K_BYTES, 8);
    if (!rc && a.down_format == 0)
      rc = make_row_tensor_map(&m.md, a.w_down, (uint64_t)E * H, (uint32_t)sp.dn.nsb * KNJ_Q4K_BYTES, (uint32_t)sp.dn.sbs * KNJ_Q4K_BYTES, 16);
    if (rc) return rc;
    s.w_down6 = a.down_format == 1 ? a.w_down : nullptr;
    s.x = a.x;
    s.out = a.out;
    s.Wr = reinterpret_cast<const __nv_bfloat16 *>(a.w_router);
    s.bias = a.router_bias;
    s.norm_w = reinterpret_cast<const __nv_bfloat16 *>(a.norm_w);
    s.tap_exp = a.tap_pair_exp;
    s.tap_w = a.tap_pair_w;
    s.ldx = a.ldx;
    s.ldo = a.ldo;
    s.eps = a.rms_eps;
    s.residual = a.residual;
    s.x_dtype = a.x_dtype;
    s.out_dtype = a.out_dtype;
  }
  int device = 0;
  KNJ_CUDA(cudaGetDevice(&device));
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) {
    cudaGetLastError();
    set_error("knj_moe_stack_create: the device's properties cannot be read");
    return KNJ_E_RUNTIME;
  }
  // boxes in flight per warp: as many as the shared memory holds next to the panels
  auto total = [&]() { return (size_t)make_plan(sp.gu, sp.dn, T, k).total; };
  while (total() > (size_t)prop.sharedMemPerBlockOptin && (sp.gu.stages > 2 || sp.dn.stages > 2)) {
    if (q4e::phase_ring_bytes(sp.gu.sbs, sp.gu.stages) >= q4e::phase_ring_bytes(sp.dn.sbs, sp.dn.stages) && sp.gu.stages > 2) --sp.gu.stages;
    else if (sp.dn.stages > 2) --sp.dn.stages;
    else --sp.gu.stages;
  }
  const size_t smem = total();
  KNJ_REQUIRE(!any_q6k || down6_warps(make_plan(sp.gu, sp.dn, T, k), sp.dn.nsb) >= 1,
              "knj_moe_stack_create: ffn=%d leaves no room for a tile of the Q6_K down phase", F);
  if (!prop.cooperativeLaunch || smem > (size_t)prop.sharedMemPerBlockOptin) {
    set_error("knj_moe_stack_create: the device lacks cooperative launch or %zu bytes of shared memory per block", smem);
    return KNJ_E_REFUSE;
  }
  cudaError_t e = cudaFuncSetAttribute(moe_stack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, moe_stack_kernel, kThreads, smem);
  if (e != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    set_error("knj_moe_stack_create: the kernel does not fit an SM (%s)", cudaGetErrorString(e));
    return KNJ_E_RUNTIME;
  }
  knj_moe_stack *st = new knj_moe_stack();
  st->device = device;
  st->smem = smem;
  st->grid = sm_count();
  auto up256 = [](size_t n) { return (n + 255) & ~(size_t)255; };
  const size_t P = (size_t)T * k;
  const size_t off_desc = up256((size_t)n_layers * sizeof(LayerMaps));
  const size_t off_logits = off_desc + up256((size_t)n_layers * sizeof(LayerDesc));
  const size_t off_scales = off_logits + up256((size_t)T * E * 4);
  const size_t off_act = off_scales + up256((size_t)T * 4);
  const size_t off_y = off_act + up256(P * F * 4);
  const size_t off_sync = off_y + up256(P * H * 4);
  e = cudaMalloc(&st->dev_block, off_sync + 256);
  if (e == cudaSuccess) e = cudaMemcpy(st->dev_block, maps.data(), (size_t)n_layers * sizeof(LayerMaps), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(static_cast<char *>(st->dev_block) + off_desc, table.data(), (size_t)n_layers * sizeof(LayerDesc), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    if (st->dev_block) cudaFree(st->dev_block);
    delete st;
    cudaGetLastError();
    set_error("knj_moe_stack_create: device allocation failed (%s)", cudaGetErrorString(e));
    return KNJ_E_RUNTIME;
  }
  char *base = static_cast<char *>(st->dev_block);
  st->p = sp;
  st->p.maps = reinterpret_cast<const LayerMaps *>(base);
  st->p.layers = reinterpret_cast<const LayerDesc *>(base + off_desc);
  st->p.n_layers = n_layers;
  st->p.T = T; st->p.H = H; st->p.F = F; st->p.E = E; st->p.k = k;
  st->p.logits = reinterpret_cast<float *>(base + off_logits);
  st->p.scales = reinterpret_cast<float *>(base + off_scales);
  st->p.act = reinterpret_cast<float *>(base + off_act);
  st->p.Y = reinterpret_cast<float *>(base + off_y);
  st->p.sync = reinterpret_cast<unsigned int *>(base + off_sync);
  st->p.wait_cycles = kMaxWaitCycles;
  st->p.stall = 0;
  *out = st;
  return KNJ_OK;
}

int knj_moe_stack_decode_launch(knj_moe_stack *st, knj_stream_t s) {
  KNJ_REQUIRE(st && (st->small || st->dev_block), "knj_moe_stack_decode_launch: null stack");
  if (st->small) return small_stack_launch(st->small, s);
  KNJ_CUDA(cudaMemsetAsync(st->p.sync, 0, 8, as_stream(s)));
  void *args[] = {&st->p};
  KNJ_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(moe_stack_kernel), dim3(st->grid), dim3(kThreads), args,
                                       st->smem, as_stream(s)));
  return launch_status("moe_stack_kernel");
}

int knj_moe_stack_set_wait(knj_moe_stack *st, long long wait_cycles, int stall_first_barrier) {
  KNJ_REQUIRE(st, "knj_moe_stack_set_wait: null stack");
  st->p.wait_cycles = wait_cycles > 0 ? wait_cycles : kMaxWaitCycles;
  st->p.stall = stall_first_barrier > 0 ? stall_first_barrier : 0;
  if (st->small) small_stack_set_wait(st->small, st->p.wait_cycles, st->p.stall);
  return KNJ_OK;
}

int knj_moe_stack_test_stall_copy(knj_moe_stack *st, int warp) {
  KNJ_REQUIRE(st && !st->small && warp < q4e::kWarps, "knj_moe_stack_test_stall_copy: no such warp, or a stack without such copies");
  st->p.stall_copy = warp >= 0 ? warp + 1 : 0;
  return KNJ_OK;
}

int knj_moe_stack_status(knj_moe_stack *st, knj_stream_t s) {
  KNJ_REQUIRE(st && (st->small || st->dev_block), "knj_moe_stack_status: null stack");
  if (st->small) return small_stack_status(st->small, s);
  unsigned int words[2] = {0, 0};
  KNJ_CUDA(cudaMemcpyAsync(words, st->p.sync, 8, cudaMemcpyDeviceToHost, as_stream(s)));
  KNJ_CUDA(cudaStreamSynchronize(as_stream(s)));
  if (words[1] != 0) {
    set_error("knj_moe_stack: a bounded wait ran out of time (grid arrivals %u)", words[0]);
    return KNJ_E_TIMEOUT;
  }
  return KNJ_OK;
}

#ifdef KNJ_TRACE
int knj_trace_force_big_stack(int on) { g_force_big_stack = on; return 0; }
int knj_trace_stack(unsigned long long *host_out) {  // measurement build only: 160 CTAs x 16 stamps
  KNJ_CUDA(cudaMemcpyFromSymbol(host_out, g_stack_trace, sizeof(unsigned long long) * 16 * 160));
  return KNJ_OK;
}
#endif

void knj_moe_stack_destroy(knj_moe_stack *st) {
  if (!st) return;
  if (st->small) small_stack_destroy(st->small);
  if (st->dev_block) cudaFree(st->dev_block);
  delete st;
}

}  // extern "C"
