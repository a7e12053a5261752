// knj_q4k_mma.cu -- decode-class expert projections as stand-alone launches:
// gate+up+SiLU*up (tools/bench/q4k_moe_ffn.hip:164-241 knj_q4k_gateup fused with
// tools/bench/q4k_stream_ffn.hip:1021-1031), the single-matrix projection
// (tools/bench/q4k_stream_ffn.hip:834-882 knj_q4k_proj) and Model::matmul
// (src/model/model.cpp:326-380), all on the tile engine of knj_q4k_engine.cuh.
//
// One persistent CTA per SM, 16 independent warps. The work of a launch is the
// flat list (job, tile): a JOB is one active expert with up to 8 of its tokens (an
// expert with more tokens yields several jobs; its weights then come from L2 after
// the first), a tile is 16 weight rows. Every CTA takes an equal contiguous run of
// that list, one job at a time: the CTA converts the job's activation rows into a
// shared-memory panel once, then warp w takes every 16th tile of the run, walks its
// superblocks through its own ring of TMA boxes (filled `stages` boxes ahead, across
// tile boundaries) and stores the 16 x 8 results itself. No partial sums cross warps
// and nothing but weights and the panel is read in the inner loop.
#include "knj_common.cuh"
#include "knj_q4k.h"
#include "knj_q4k_engine.cuh"

using namespace knj;

namespace {

constexpr int kThreads = q4e::kWarps * 32;

struct ProjParams {
  const uint8_t *W0;  // gate (dual) or the single matrix
  const uint8_t *W1;  // up (dual) or null
  const void *X;      // activation rows
  int x_dtype;
  int64_t ldx;
  const int32_t *pair_idx;
  const int32_t *pair_cnt;
  const int32_t *row_map;  // pair -> activation row (null: pair / row_div)
  const int32_t *exp_list;
  const int32_t *n_active;
  float *out0;  // dual: G        single: Y
  float *out1;  // dual: U
  float *out2;  // dual: A = silu(G)*U
  int K, row_div;
  int n_experts;  // length of exp_list / pair_cnt
  int n_ident;    // rows of a dense product (IDENT)
  q4e::PhaseShape shape;
  int64_t idxStride;
  int *status;    // optional: set to 1 when a bounded wait gave up
  long long wait_cycles;   // limit of every wait inside the kernel
  int stall;      // test hook: the first box of CTA 0's first warp never counts as landed
  CUtensorMap map0, map1;  // TMA descriptors of W0 / W1: box = sbs superblocks x 8 (dual) or 16 rows
};

struct ProjSmem {
  size_t ring, panels, bars, red, total;
};
__host__ __device__ inline ProjSmem proj_smem(int nsb, int sbs, int stages) {
  ProjSmem m;
  m.ring = 0;
  m.panels = m.ring + q4e::phase_ring_bytes(sbs, stages);
  m.bars = m.panels + q4e::phase_panel_bytes(nsb);
  m.red = m.bars + (size_t)q4e::kWarps * q4e::kMaxStages * 8;
  m.total = m.red + (size_t)q4e::kWarps * 32 * sizeof(float4);
  return m;
}

#ifdef KNJ_TRACE
// Measurement build only: experiment modes (1: no arithmetic; 2: no weight copies; 3: no activation panels).
__device__ int g_trace_mode = 0;
#endif

// IDENT: one matrix and rows 0..n_ident-1 (a dense product); the plan's arrays are not read. PL = 1: rows of a 16-bit type,
// eight to a job (301 bf16 rows of a 2048 x 2048 matrix: 46.6 -> 31.1 us).
template <bool DUAL, bool IDENT, int PL>
__global__ void __launch_bounds__(kThreads, 1) q4k_proj_kernel(const __grid_constant__ ProjParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int s_jbase[257];
  __shared__ int s_uexp[256], s_ucnt[256];
  constexpr int kTok = q4e::job_tokens<PL>();
  __shared__ float s_inv[kTok * 16];
  __shared__ int s_pair[kTok];
  __shared__ int s_fail;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const ProjSmem lay = proj_smem(p.shape.nsb, p.shape.sbs, p.shape.stages);
  q4e::PhaseSmem sm;
  sm.ring = smem + lay.ring;
  sm.panels = smem + lay.panels;
  sm.bars = reinterpret_cast<uint64_t *>(smem + lay.bars);
  sm.red = reinterpret_cast<float4 *>(smem + lay.red);
  sm.inv = s_inv;
  sm.pair = s_pair;
  sm.fail = &s_fail;
  if (lane == 0)
    for (int s = 0; s < q4e::kMaxStages; ++s)
      mbar_init(&sm.bars[warp * q4e::kMaxStages + s], IDENT && p.stall && blockIdx.x == 0 && warp == 0 && s == 0 ? 2 : 1);
  if (threadIdx.x == 0) s_fail = 0;
  mbar_init_fence();
  grid_dep_wait();  // the plan and the activation rows come from earlier launches
  grid_dep_signal();

  // ---- the job table: jobs per active expert, exclusive prefix (every CTA derives the same table)
  const int n_act = IDENT ? 1 : min(p.n_active[0], 256);
  for (int a = threadIdx.x; a < 256; a += kThreads) {
    int c = 0, ex = -1;
    if (a < n_act) {
      ex = IDENT ? 0 : p.exp_list[a];
      c = IDENT ? p.n_ident : p.pair_cnt[ex];
    }
    s_uexp[a] = ex;
    s_ucnt[a] = c;
    s_jbase[a] = (c + kTok - 1) / kTok;
  }
  __syncthreads();
  if (warp == 0) q4e::job_prefix(s_jbase, lane);
  __syncthreads();

  const long long U = (long long)s_jbase[256] * p.shape.tiles;  // < 2^31 (checked by the launcher)
  const int u0 = (int)(U * blockIdx.x / gridDim.x), u1 = (int)(U * (blockIdx.x + 1) / gridDim.x);
  q4e::JobTable jt{s_jbase, s_uexp};
  unsigned parity = 0;
  bool ok = true;
  int tmode = 0;
#ifdef KNJ_TRACE
  tmode = g_trace_mode;
#endif
  q4e::run_phase<DUAL, PL>(
      p.shape, sm, jt, u0, u1, q4e::choose_ksplit(U, p.shape.nsb / p.shape.sbs, gridDim.x), &p.map0, &p.map1, p.out0, p.out1, p.out2, p.wait_cycles, parity, ok,
      [&](int job, int a, int tk, int &pair, int &row) {
        const int tok = (job - s_jbase[a]) * kTok + tk;
        if (tok >= s_ucnt[a]) return false;
        pair = IDENT ? tok : p.pair_idx[(size_t)s_uexp[a] * p.idxStride + tok];
        row = p.row_map ? p.row_map[pair] : pair / p.row_div;
        return true;
      },
      [&](int row, int sb, int ln, float (&v)[8]) { q4e::load8_f32(p.X, p.x_dtype, (int64_t)row * p.ldx + 256 * sb + 8 * ln, v); },
      tmode);
  if (!ok && p.status) atomicExch(p.status, 1);
  if (IDENT) {
    // A dense product has no status word: where a wait gave up, all outputs of this CTA's units become NaN, so that a
    // caller cannot take what the buffer held before for a result.
    __syncthreads();
    if (*sm.fail) {
      const int tiles = p.shape.tiles;
      for (long long i = threadIdx.x; i < (long long)(u1 - u0) * kTok * 16; i += kThreads) {
        const int u = u0 + (int)(i / (kTok * 16)), tk = (int)(i / 16) % kTok;
        const int tok = u / tiles * kTok + tk;
        if (tok < p.n_ident) p.out0[(size_t)tok * p.shape.N + u % tiles * 16 + (int)(i % 16)] = __int_as_float(0x7fffffff);
      }
    }
  }
}

long long g_decode_wait_cycles = kMaxWaitCycles;
thread_local int t_stall_dense = 0;  // knj_q4k_matmul_test_stall

template <bool DUAL, bool IDENT = false, int PL = 2>
int launch_proj(ProjParams p, int n_experts_max, cudaStream_t st) {
  const int nsb = p.K / KNJ_QK_K;
  KNJ_REQUIRE(nsb >= 1 && nsb <= 16, "q4k projection: rows of %d weights (at most 4096 are taken)", p.K);
  KNJ_REQUIRE((long long)n_experts_max * (p.idxStride / q4e::kJobTok + 1) * p.shape.tiles < (1ll << 31),
              "q4k projection: %d experts x %d tiles exceed the work index", n_experts_max, p.shape.tiles);
  p.n_experts = n_experts_max;
  p.shape.nsb = nsb;
  p.shape.sbs = (nsb % 2 == 0) ? 2 : 1;
  p.wait_cycles = g_decode_wait_cycles;
  {
    const uint64_t rows = (uint64_t)n_experts_max * p.shape.N;
    const uint32_t box = (uint32_t)p.shape.sbs * KNJ_Q4K_BYTES;
    int rc = make_row_tensor_map(&p.map0, p.W0, rows, (uint32_t)nsb * KNJ_Q4K_BYTES, box, DUAL ? 8 : 16);
    if (rc) return rc;
    if (DUAL) {
      rc = make_row_tensor_map(&p.map1, p.W1, rows, (uint32_t)nsb * KNJ_Q4K_BYTES, box, 8);
      if (rc) return rc;
    }
  }
  int dev = 0;
  KNJ_CUDA(cudaGetDevice(&dev));
  int smem_max = 0;
  KNJ_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t reserve = 6 * 1024;  // the kernel's static shared memory
  p.shape.stages = p.shape.sbs == 2 ? 2 : q4e::kMaxStages;  // four superblocks in flight per warp either way
  while (p.shape.stages > 2 && proj_smem(nsb, p.shape.sbs, p.shape.stages).total + reserve > (size_t)smem_max) --p.shape.stages;
  const size_t smem = proj_smem(nsb, p.shape.sbs, p.shape.stages).total;
  KNJ_REQUIRE(smem + reserve <= (size_t)smem_max, "q4k projection: rows of %d weights do not fit the shared memory", p.K);
  auto kern = q4k_proj_kernel<DUAL, IDENT, PL>;
  // opt in to the large dynamic shared memory once per device and instantiation
  // (kept out of later launches so they are plain stream work, capturable in a graph)
  static size_t opted[64] = {0};
  if (dev >= 0 && dev < 64 && opted[dev] < smem) {
    KNJ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    opted[dev] = smem;
  }
  KNJ_CUDA(launch_chain(kern, dim3((unsigned)sm_count()), dim3(kThreads), smem, st, p));
  return launch_status("q4k_proj_kernel");
}

int check_rows(const void *X, int dtype, int64_t ld, int K, const char *who) {
  KNJ_REQUIRE(dtype >= KNJ_DT_F32 && dtype <= KNJ_DT_F16, "%s: unknown activation dtype %d", who, dtype);
  const int64_t esz = dtype == KNJ_DT_F32 ? 4 : 2;
  KNJ_REQUIRE(aligned16(X) && ld >= K && (ld * esz) % 16 == 0, "%s: activation rows must be 16-byte aligned (ld=%lld)", who,
              (long long)ld);
  return KNJ_OK;
}

// y[m][n_out] = x . W^T with one matrix. The plan (pairs = rows 0..m-1) is derived in the kernel: a launch that wrote it
// to memory first, and a fill of y, were a third of a one-row product's time (768 x 2048: 22.7 -> 15.9 us; 301 rows of a
// 2048 x 2048 matrix 53.8 -> 46.9).
int dense_product(const uint8_t *W, int n_in, int n_out, const void *x, int x_dtype, int64_t ldx, int m, float *y, int64_t ldy,
                  knj_stream_t s) {
  KNJ_REQUIRE(W && x && y, "knj_q4k_matmul: null pointer");
  KNJ_REQUIRE(m > 0 && n_in > 0 && n_in % 256 == 0 && n_out > 0 && n_out % 16 == 0,
              "knj_q4k_matmul: needs n_in %% 256 == 0, n_out %% 16 == 0");
  KNJ_REQUIRE(ldy == n_out, "knj_q4k_matmul: y must be dense (ldy == n_out)");
  KNJ_REQUIRE(aligned16(W), "knj_q4k_matmul: W must be 16-byte aligned");
  const int rc = check_rows(x, x_dtype, ldx, n_in, "knj_q4k_matmul");
  if (rc) return rc;
  ProjParams p{};
  p.W0 = W; p.X = x; p.x_dtype = x_dtype; p.ldx = ldx; p.n_ident = m;
  p.out0 = y; p.shape.N = n_out; p.K = n_in; p.row_div = 1;
  p.shape.tiles = n_out / 16; p.idxStride = m; p.stall = t_stall_dense;
  // 16-bit rows hold in one plane of the panel (the other one would be all zeros), so twice as many can make a job: half the
  // unpacking, but also half the jobs to spread over 2368 warps. bf16, us, jobs of four / of eight, with the tiles of the
  // former and their superblocks in all: 16 x 768 x 2048 (192, 1.5 k) 7.4 / 8.1, 33 x 2048 x 1024 (1152, 4.6 k) 10.1 / 10.3,
  // 9 x 4096 x 4096 (768, 12 k) 20.3 / 15.3, 512 x 256 x 256 (2048, 2 k) 7.5 / 7.0, 64 x 2048 x 2048 (2048, 16 k) 18.3 / 16.2,
  // 512 x 4096 x 4096 229 / 132.
  const long long tiles4 = (long long)((m + 3) / 4) * p.shape.tiles;
  if (x_dtype != KNJ_DT_F32 && (tiles4 >= 2048 || tiles4 * (n_in / KNJ_QK_K) >= 8192)) return launch_proj<false, true, 1>(p, 1, as_stream(s));
  return launch_proj<false, true>(p, 1, as_stream(s));
}

}  // namespace

namespace knj {
long long decode_wait_cycles() { return g_decode_wait_cycles; }
}  // namespace knj

extern "C" {

#ifdef KNJ_TRACE
int knj_trace_proj(long long *, int mode) {  // measurement build only
  KNJ_CUDA(cudaMemcpyToSymbol(g_trace_mode, &mode, sizeof(mode)));
  return KNJ_OK;
}
int knj_trace_feed(int) { return 0; }
#endif

void knj_decode_wait_limit(long long cycles) { g_decode_wait_cycles = cycles > 0 ? cycles : kMaxWaitCycles; }

int knj_q4k_gateup_launch(const void *X, int x_dtype, int64_t ldx, const uint8_t *Wg, const uint8_t *Wu,
                          const int32_t *pair_idx, const int32_t *pair_cnt, const int32_t *pair_tok,
                          const int32_t *exp_list, const int32_t *n_active, float *G, float *U, float *A, int N, int K,
                          int rowBytes, int64_t idxStride, int n_experts, int top_k, int *status, knj_stream_t s) {
  KNJ_REQUIRE(X && Wg && Wu && pair_idx && pair_cnt && exp_list && n_active, "knj_q4k_gateup: null pointer");
  KNJ_REQUIRE(G || U || A, "knj_q4k_gateup: no output requested");
  KNJ_REQUIRE(K > 0 && K % 256 == 0 && rowBytes == K / 256 * KNJ_Q4K_BYTES,
              "knj_q4k_gateup: rowBytes=%d does not match K=%d", rowBytes, K);
  KNJ_REQUIRE(N > 0 && N % 8 == 0, "knj_q4k_gateup: N=%d must be a multiple of 8", N);
  KNJ_REQUIRE(aligned16(Wg) && aligned16(Wu), "knj_q4k_gateup: weights must be 16-byte aligned");
  KNJ_REQUIRE(n_experts > 0 && n_experts <= 256 && (pair_tok || top_k > 0), "knj_q4k_gateup: bad expert / top_k count");
  int rc = check_rows(X, x_dtype, ldx, K, "knj_q4k_gateup");
  if (rc) return rc;
  ProjParams p{};
  p.W0 = Wg; p.W1 = Wu; p.X = X; p.x_dtype = x_dtype; p.ldx = ldx;
  p.pair_idx = pair_idx; p.pair_cnt = pair_cnt; p.row_map = pair_tok; p.exp_list = exp_list; p.n_active = n_active;
  p.out0 = G; p.out1 = U; p.out2 = A;
  p.shape.N = N; p.K = K; p.row_div = top_k > 0 ? top_k : 1;
  p.shape.tiles = N / 8; p.idxStride = idxStride; p.status = status;
  return launch_proj<true>(p, n_experts, as_stream(s));
}

int knj_q4k_proj_launch(const void *A, int a_dtype, int64_t lda, const uint8_t *W, const int32_t *pair_idx,
                        const int32_t *pair_cnt, const int32_t *pair_row, const int32_t *exp_list, const int32_t *n_active,
                        float *Y, int N, int K, int rowBytes, int64_t idxStride, int n_experts, int *status,
                        knj_stream_t s) {
  KNJ_REQUIRE(A && W && pair_idx && pair_cnt && exp_list && n_active && Y, "knj_q4k_proj: null pointer");
  KNJ_REQUIRE(K > 0 && K % 256 == 0 && rowBytes == K / 256 * KNJ_Q4K_BYTES,
              "knj_q4k_proj: rowBytes=%d does not match K=%d", rowBytes, K);
  KNJ_REQUIRE(N > 0 && N % 16 == 0, "knj_q4k_proj: N=%d must be a multiple of 16", N);
  KNJ_REQUIRE(aligned16(W), "knj_q4k_proj: weights must be 16-byte aligned");
  KNJ_REQUIRE(n_experts > 0 && n_experts <= 256, "knj_q4k_proj: bad expert count");
  int rc = check_rows(A, a_dtype, lda, K, "knj_q4k_proj");
  if (rc) return rc;
  ProjParams p{};
  p.W0 = W; p.W1 = nullptr; p.X = A; p.x_dtype = a_dtype; p.ldx = lda;
  p.pair_idx = pair_idx; p.pair_cnt = pair_cnt; p.row_map = pair_row; p.exp_list = exp_list; p.n_active = n_active;
  p.out0 = Y; p.out1 = nullptr; p.out2 = nullptr;
  p.shape.N = N; p.K = K; p.row_div = 1;
  p.shape.tiles = N / 16; p.idxStride = idxStride; p.status = status;
  return launch_proj<false>(p, n_experts, as_stream(s));
}

void knj_q4k_matmul_test_stall(int on) { t_stall_dense = on & 1; }

size_t knj_q4k_matmul_workspace_bytes(int m, int n_in) {
  if (m <= 0 || n_in <= 0) return 0;
  // what callers have to bring (an identity pair list and counts; the kernel derives them and reads none)
  return (((size_t)m * 4 + 255) & ~(size_t)255) + 256;
}

int knj_q4k_matmul_launch(const uint8_t *W, int n_in, int n_out, const void *x, int x_dtype, int64_t ldx, int m,
                          float *y, int64_t ldy, void *workspace, size_t workspace_bytes, knj_stream_t s) {
  KNJ_REQUIRE(W && x && y, "knj_q4k_matmul: null pointer");
  KNJ_REQUIRE(m > 0 && n_in % 256 == 0 && n_out % 16 == 0, "knj_q4k_matmul: needs n_in %% 256 == 0, n_out %% 16 == 0");
  KNJ_REQUIRE(ldy == n_out, "knj_q4k_matmul: y must be dense (ldy == n_out)");
  if (!workspace || workspace_bytes < knj_q4k_matmul_workspace_bytes(m, n_in)) {
    set_error("knj_q4k_matmul: workspace of %zu bytes needed", knj_q4k_matmul_workspace_bytes(m, n_in));
    return KNJ_E_WORKSPACE;
  }
  KNJ_REQUIRE(aligned16(workspace), "knj_q4k_matmul: workspace must be 16-byte aligned");
  return dense_product(W, n_in, n_out, x, x_dtype, ldx, m, y, ldy, s);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of knj_q4k_matmul_launch.
//
// Who needs it: callers that must not allocate device memory at the point of
// the call and have no workspace to hand over -- code running inside a
// latency-critical serving loop whose memory pool is fully committed to the
// resident experts, plug-in hosts that are only given the input and output
// buffers, and callers that forbid allocator calls after start-up because an
// allocation can synchronise the device or fragment a tightly packed HBM budget.
//
// The product needs no scratch (the one-matrix plan is derived in the kernel),
// so calls may overlap. Problems whose workspace would exceed
// kNoAllocScratchBytes are refused with KNJ_E_WORKSPACE: a limit of this entry
// point and nothing more, kept so that what it refused it goes on refusing.
// ---------------------------------------------------------------------------
namespace {
constexpr size_t kNoAllocScratchBytes = (size_t)64 << 10;  // the workspace of 16,320 activation rows
}  // namespace

size_t knj_q4k_matmul_noalloc_max_scratch(void) { return kNoAllocScratchBytes; }

int knj_q4k_matmul_noalloc_launch(const uint8_t *W, int n_in, int n_out, const void *x, int x_dtype, int64_t ldx, int m,
                                  float *y, int64_t ldy, knj_stream_t s) {
  KNJ_REQUIRE(m > 0 && n_in > 0, "knj_q4k_matmul_noalloc: m and n_in must be positive");
  const size_t need = knj_q4k_matmul_workspace_bytes(m, n_in);
  if (need > kNoAllocScratchBytes) {
    set_error("knj_q4k_matmul_noalloc: m=%d rows of n_in=%d (a workspace of %zu bytes) are above this entry point's limit of %zu; "
              "use knj_q4k_matmul_launch with a caller workspace",
              m, n_in, need, kNoAllocScratchBytes);
    return KNJ_E_WORKSPACE;
  }
  return dense_product(W, n_in, n_out, x, x_dtype, ldx, m, y, ldy, s);
}

}  // extern "C"
