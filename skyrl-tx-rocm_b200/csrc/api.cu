// Host side of the C ABI: error reporting, TMA descriptor encoding and the
// operator entry points that chain the stage kernels on the caller's stream.
#include <stdarg.h>
#include <stdio.h>

#include <mutex>

#include "common.cuh"

namespace skyrl {

static thread_local char g_last_error[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
  return code;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  });
  return fn;
}

static int encode(CUtensorMap* map, CUtensorMapDataType dtype, int elem_bytes, uint32_t rank, const void* base,
                  const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return fail(SKYRL_ERR_DRIVER, "cuTensorMapEncodeTiled is not available from the CUDA driver");
  const cuuint32_t estr[3] = {1, 1, 1};
  const uint32_t width = box[0] * static_cast<uint32_t>(elem_bytes);  // the swizzle spans the box's inner extent
  const CUtensorMapSwizzle swizzle = width >= 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                     : width >= 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                   : CU_TENSOR_MAP_SWIZZLE_32B;
  CUresult r = fn(map, dtype, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(SKYRL_ERR_INVALID_ARGUMENT, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return SKYRL_OK;
}

int encode_tmap_2d(CUtensorMap* map, CUtensorMapDataType dtype, int elem_bytes, const void* base, uint64_t inner,
                   uint64_t outer, uint64_t row_pitch_bytes, uint32_t box_inner, uint32_t box_outer) {
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {row_pitch_bytes};
  const cuuint32_t box[2] = {box_inner, box_outer};
  return encode(map, dtype, elem_bytes, 2, base, dims, strides, box);
}

int encode_tmap_3d(CUtensorMap* map, CUtensorMapDataType dtype, int elem_bytes, const void* base, uint64_t d0,
                   uint64_t d1, uint64_t d2, uint64_t pitch1_bytes, uint64_t pitch2_bytes, uint32_t box0,
                   uint32_t box1, uint32_t box2) {
  const cuuint64_t dims[3] = {d0, d1, d2};
  const cuuint64_t strides[2] = {pitch1_bytes, pitch2_bytes};
  const cuuint32_t box[3] = {box0, box1, box2};
  return encode(map, dtype, elem_bytes, 3, base, dims, strides, box);
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cached[dev] = n;
  }
  return cached[dev];
}

// ---- workspace carving -------------------------------------------------------
static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

constexpr int MAX_CHUNKS = 16;
constexpr int SCHED_WORDS = ZERO_WORDS;  // room for four {claimed, finished} pairs of the GEMMs' dynamic tile scheduler

// Dense tiles of the sorted rows (tiles.cuh): tile i is rows 128 i ...; segments (tile, adapter) never number more than
// tiles + adapters.
static inline int dense_tiles(int rows) { return (rows + SKYRL_TILE_ROWS - 1) / SKYRL_TILE_ROWS; }
static inline size_t segment_slots(int m, int num_adapters) {
  return static_cast<size_t>(dense_tiles(m)) + (num_adapters > 0 ? num_adapters : 1);
}

struct Carver {
  unsigned char* base;
  size_t off = 0;
  explicit Carver(void* b) : base(static_cast<unsigned char*>(b)) {}
  template <typename T>
  T* take(size_t count) {
    off = align_up(off, 1024);
    T* p = base != nullptr ? reinterpret_cast<T*>(base + off) : nullptr;
    off += count * sizeof(T);
    return p;
  }
  size_t total() const { return align_up(off, 1024); }
};

// Batches of at most this many rows take the row-wise LoRA path (no adapter sort, one M tile).
constexpr int ROWS_PATH_MAX_M = SKYRL_TILE_ROWS;

struct RouteWs {
  int32_t* perm;
  int32_t* tiles;
  int32_t* seg_mask;
  int32_t* seg_adapter;
};
static RouteWs carve_route(Carver& c, int m, int num_adapters) {
  RouteWs r;
  r.perm = c.take<int32_t>(m);
  r.tiles = c.take<int32_t>(4 * static_cast<size_t>(dense_tiles(m)));
  r.seg_mask = c.take<int32_t>(4 * segment_slots(m, num_adapters));
  r.seg_adapter = c.take<int32_t>(segment_slots(m, num_adapters));
  return r;
}
// Tiles of sorted rows [row0, row0 + rows), row0 a multiple of 128; without routing they are computed, not listed.
static TileSource tile_source(const RouteWs& r, bool routed, int row0, int rows) {
  TileSource t = {};
  t.count = dense_tiles(rows);
  t.row0 = row0;
  t.row_end = row0 + rows;
  if (routed) {
    t.tiles = reinterpret_cast<const int4*>(r.tiles) + row0 / SKYRL_TILE_ROWS;
    t.seg_mask = reinterpret_cast<const int4*>(r.seg_mask);
    t.seg_adapter = r.seg_adapter;
  }
  return t;
}

struct LinearWs {
  RouteWs route;
  int8_t* xq;
  float* sx;
  uint16_t* xn;
  uint16_t* z_parts;  // bf16 [m, 6, 64]; the row-wise path keeps fp32 [m, 64] here instead
  int32_t* acc;       // int32 [m, n] accumulator, row-wise path only
  int32_t* sched;     // tile-claim counters of the GEMM launch (zeroed by the routing kernel, left at zero by the GEMM)
  size_t bytes;
};

static LinearWs carve_linear(void* ws, int m, int n, int k, int num_adapters) {
  Carver c(ws);
  LinearWs w;
  w.route = carve_route(c, m, num_adapters);
  w.sched = c.take<int32_t>(SCHED_WORDS);
  w.xq = c.take<int8_t>(static_cast<size_t>(m) * k);
  w.sx = c.take<float>(m);
  w.z_parts = c.take<uint16_t>(SKYRL_Z_PARTS * static_cast<size_t>(m) * SKYRL_LORA_RANK_PAD);
  if (m <= ROWS_PATH_MAX_M) {
    w.xn = nullptr;
    w.acc = c.take<int32_t>(static_cast<size_t>(m) * n * plan_gemm(m, n, k, SKYRL_EPI_ACC_I32, MAX_SPLIT_K_SLABS).k_splits);
  } else {
    w.xn = c.take<uint16_t>(static_cast<size_t>(m) * k);
    w.acc = nullptr;
  }
  w.bytes = c.total();
  return w;
}

struct MlpWs {
  RouteWs route;
  int8_t* xq;
  float* sx;
  uint16_t* xn;
  uint16_t* z_parts;
  uint16_t* h;
  int8_t* hq;
  float* sh;
  int32_t* acc;  // int32 [m, max(2I, H)] accumulator, row-wise path only
  float* h_amax; // fp32 [m]: absmax of every row of h, collected by the gate_up epilogue
  int32_t* sched; // tile-claim counters: words 0-1 gate_up GEMM, 2-3 down GEMM, 4-7 the same for odd chunks (zeroed by the routing kernel)
  size_t bytes;
};

static MlpWs carve_mlp(void* ws, int m, int hidden, int inter, int num_adapters) {
  Carver c(ws);
  MlpWs w;
  w.route = carve_route(c, m, num_adapters);
  w.sched = c.take<int32_t>(SCHED_WORDS);
  w.xq = c.take<int8_t>(static_cast<size_t>(m) * hidden);
  w.sx = c.take<float>(m);
  w.z_parts = c.take<uint16_t>(SKYRL_Z_PARTS * static_cast<size_t>(m) * SKYRL_LORA_RANK_PAD);
  w.h = c.take<uint16_t>(static_cast<size_t>(m) * inter);
  w.hq = c.take<int8_t>(static_cast<size_t>(m) * inter);
  w.sh = c.take<float>(m);
  w.xn = c.take<uint16_t>(static_cast<size_t>(m) * hidden);
  if (m <= ROWS_PATH_MAX_M) {
    const size_t gu = static_cast<size_t>(m) * 2 * inter *
                      plan_gemm(m, 2 * inter, hidden, SKYRL_EPI_ACC_I32, MAX_SPLIT_K_SLABS).k_splits;
    const size_t dn = static_cast<size_t>(m) * hidden *
                      plan_gemm(m, hidden, inter, SKYRL_EPI_ACC_I32, MAX_SPLIT_K_SLABS).k_splits;
    w.acc = c.take<int32_t>(gu > dn ? gu : dn);
  } else {
    w.acc = nullptr;
  }
  w.h_amax = c.take<float>(m);
  w.bytes = c.total();
  return w;
}

static int check_ws(const void* ws, size_t have, size_t need, const char* who) {
  if (ws == nullptr || (reinterpret_cast<uintptr_t>(ws) & 1023u) != 0)
    return fail(SKYRL_ERR_WORKSPACE, "%s: workspace must be non-null and 1024-byte aligned", who);
  if (have < need) return fail(SKYRL_ERR_WORKSPACE, "%s: workspace has %zu bytes, needs %zu", who, have, need);
  return SKYRL_OK;
}

// One W8A8 LoRA projection on rows that are already laid out as the GEMM wants them.
//   tensor-core route (m > 128): rows adapter-sorted, z planes from lora_a_proj, LoRA inside the GEMM epilogue
//   row-wise route (m <= 128): rows in token order; the GEMM leaves the int32 accumulator in global
//   memory (split over K when that fills the GPU better) and a row-wise kernel applies scales, LoRA,
//   the cast and the SwiGLU / residual step
struct Projection {
  const void* x;          // bf16 [m, k] source rows
  int64_t x_stride;
  const void* rms_delta;  // nullable
  float eps;
  const int32_t* gather;  // row gather for the quantiser (sorted route) or NULL
  bool keep_xn;           // sorted route: x must be re-laid out (gathered / normalised) for the projection MMA
  int m, n, k, rank, na;
  int q_row0, q_rows;     // sorted rows the quantiser stage covers (a chunk of the block, or all m rows)
  int list_row0;          // first sorted row of `src` (0, or the first row of the call's chunk)
  bool skip_quant;        // the quantiser stage of these rows already ran (its outputs are in xq / sx / z_parts)
  int gemm_variant;       // SKYRL_GEMM_VARIANT_* forced on the GEMM (0: the library chooses)
  bool two_step_rows;     // row-wise route: GEMM to an int32 accumulator in memory + finalize kernel (default)
  const float* known_amax;  // absmax of every source row, if the producer of x collected it (sorted route)
  float* zero_amax;         // quantiser stage: row absmax words it clears for the GEMM behind it (nullable)
  int32_t* zero_words;      // quantiser stage: scheduler words it clears where no routing kernel runs (nullable)
  float* row_amax;          // SwiGLU epilogue: collect the absmax of every output row here
  int cta_limit;
  void* const* scatter_bases;  // row scatter of the fp32 partial sums (see SkyrlW8A8GemmArgs) or NULL
  int scatter_row0, scatter_rows;

  const void* wq;
  const float* sw;
  const void* a_packed;
  const void* b_packed;
  const void* b_rows;     // dense [A, n, b_rows_rank] LoRA-B table for the row-wise route, or NULL
  int b_rows_rank;
  const float* scaling;
  const int32_t* ids;     // token-order adapter ids (row-wise route)
  int8_t* xq;
  float* sx;
  uint16_t* xn;
  uint16_t* z_parts;
  int32_t* acc;
  TileSource src;
  int epilogue;
  ColumnSplit split;      // linear epilogue: output columns dealt to several matrices (count 0: `out`)
  const int32_t* out_row_map;
  const void* residual;
  int64_t residual_stride;
  void* out;
  int64_t out_stride;
  int32_t* status;
  int32_t* sched;         // {claimed, finished} words of the GEMM launch inside the caller's workspace
  const void* prefetch;   // row-wise route: bytes the GEMM asks into L2 after its own loads (the next GEMM's weights)
  int64_t prefetch_bytes;
  void* ev_begin;
  void* ev_end;
};

// Quantiser stage of the sorted route for rows [q_row0, q_row0 + q_rows): RMSNorm + int8 codes + scales
// (+ the normalised bf16 rows the LoRA-A projection reads), then the LoRA-A projection of those rows.
static int run_quant_stage(const Projection& q, cudaStream_t stream) {
  const bool lora = q.rank > 0;
  const bool need_xn = lora && q.keep_xn;
  const int r0 = q.q_row0, rows = q.q_rows > 0 ? q.q_rows : q.m;
  int rc;
  // a gather reads rows perm[r0 ...] of x; without one the chunk's rows are rows r0 ... of x itself
  const unsigned char* xsrc = static_cast<const unsigned char*>(q.x) +
                              (q.gather != nullptr ? 0 : static_cast<size_t>(r0) * q.x_stride * 2);
  if (q.known_amax != nullptr && q.rms_delta == nullptr && q.gather == nullptr && !need_xn && q.x_stride == q.k) {
    // the rows' absmax came with them: one streaming pass
    if ((rc = launch_quant_stream(xsrc, q.known_amax + r0, rows, q.k, q.xq + static_cast<size_t>(r0) * q.k, q.sx + r0,
                                  stream)))
      return rc;
  } else if ((rc = launch_rms_quant(xsrc, q.x_stride, q.rms_delta, q.eps,
                                    q.gather != nullptr ? q.gather + r0 : nullptr, rows, q.k,
                                    q.xq + static_cast<size_t>(r0) * q.k, q.sx + r0,
                                    need_xn ? q.xn + static_cast<size_t>(r0) * q.k : nullptr, stream,
                                    q.zero_amax != nullptr ? q.zero_amax + r0 : nullptr, q.zero_words))) {
    return rc;
  }
  if (lora) {
    const void* xa = need_xn ? static_cast<const void*>(q.xn) : q.x;
    if ((rc = launch_lora_a_proj(xa, q.m, q.k, q.a_packed, q.scaling, q.na, q.rank, q.src, q.src.count, q.z_parts, q.status,
                                 stream, r0, r0 + rows, nullptr, 0, q.list_row0)))
      return rc;
  }
  return SKYRL_OK;
}

static int run_projection(const Projection& q, cudaStream_t stream) {
  const bool lora = q.rank > 0;
  const bool rows_path = q.m <= ROWS_PATH_MAX_M;
  int rc;
  SkyrlW8A8GemmArgs g = {};
  if (rows_path && lora && q.epilogue != SKYRL_EPI_ACC_I32) {
    float* z_rows = reinterpret_cast<float*>(q.z_parts);
    if ((rc = launch_rms_quant_rows(q.x, q.x_stride, q.rms_delta, q.eps, q.ids, q.na, q.a_packed, q.scaling, q.rank, q.m,
                                    q.k, q.xq, q.sx, z_rows, q.status, stream, true, q.keep_xn ? q.xn : nullptr)))
      return rc;
    const bool dense = q.b_rows != nullptr;
    const int brow = dense ? q.b_rows_rank : SKYRL_LORA_RANK_PAD;
    // timing events between the launches would cut the programmatic chain: use ordinary launches then
    const bool chain = q.ev_begin == nullptr && q.ev_end == nullptr;
    g.struct_size = sizeof(g);
    g.m = q.m;
    g.n = q.n;
    g.k = q.k;
    g.num_adapters = q.na;
    g.xq = q.xq;
    g.sx = q.sx;
    g.wq = q.wq;
    g.sw = q.sw;
    g.status = q.status;
    g.prefetch = q.prefetch;
    g.prefetch_bytes = q.prefetch_bytes;
    if (!q.two_step_rows) {
      // one kernel: the GEMM's epilogue warps evaluate the per-row LoRA term while the weights stream and apply
      // scales, LoRA, the cast and the SwiGLU / residual step from tensor memory
      g.epilogue = q.epilogue;
      g.rank = q.rank;
      g.z_rows = z_rows;
      g.row_adapter_ids = q.ids;
      g.lora_b_rows = dense ? q.b_rows : q.b_packed;
      g.lora_b_rows_rank = brow;
      g.residual = q.residual;
      g.residual_row_stride = q.residual_stride;
      g.out = q.out;
      g.out_row_stride = q.out_stride;
      if (q.ev_begin != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(q.ev_begin), stream);
      rc = launch_gemm(g, stream, chain, &q.src);
      if (q.ev_end != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(q.ev_end), stream);
      return rc;
    }
    // two steps (the default: faster at decode shapes): int32 accumulator to global memory, split over K when
    // that fills the GPU better, then a row-wise kernel run by a whole grid
    const int slabs = plan_gemm(q.m, q.n, q.k, SKYRL_EPI_ACC_I32, MAX_SPLIT_K_SLABS).k_splits;
    g.epilogue = SKYRL_EPI_ACC_I32;
    g.split_k_slabs = MAX_SPLIT_K_SLABS;
    g.rank = 0;
    g.out = q.acc;
    g.out_row_stride = q.n;
    if (q.ev_begin != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(q.ev_begin), stream);
    rc = launch_gemm(g, stream, chain, &q.src);
    if (q.ev_end != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(q.ev_end), stream);
    if (rc) return rc;
    return launch_finalize_rows(q.epilogue, q.acc, slabs, q.sx, q.sw, z_rows, q.ids, q.na,
                                dense ? q.b_rows : q.b_packed, static_cast<int64_t>(q.n) * brow, brow, q.rank, q.m, q.n,
                                q.residual, q.residual_stride, q.out, q.out_stride, q.status, stream, chain, q.split);
  }
  {
    if (!q.skip_quant && (rc = run_quant_stage(q, stream))) return rc;
    g.rank = q.rank;
    g.z_parts = lora ? q.z_parts : nullptr;
  }
  g.struct_size = sizeof(g);
  g.epilogue = q.epilogue;
  g.m = q.m;
  g.n = q.n;
  g.k = q.k;
  g.num_adapters = q.na;
  g.xq = q.xq;
  g.sx = q.sx;
  g.wq = q.wq;
  g.sw = q.sw;
  g.lora_b_packed = q.b_packed;
  if (lora && q.b_rows != nullptr) {
    g.lora_b_rows = q.b_rows;
    g.lora_b_rows_rank = q.b_rows_rank;
  }
  g.out_row_map = q.out_row_map;
  g.residual = q.residual;
  g.out = q.out;
  g.out_row_stride = q.out_stride;
  g.residual_row_stride = q.residual_stride;
  g.status = q.status;
  g.sched = q.sched;
  g.variant = q.gemm_variant;
  g.cta_limit = q.cta_limit;
  if (q.row_amax != nullptr && q.epilogue == SKYRL_EPI_SWIGLU) {
    if (q.skip_quant) {  // no quantiser stage in this call to clear it
      const int r0 = q.q_row0, rows = q.q_rows > 0 ? q.q_rows : q.m;
      cudaError_t e = cudaMemsetAsync(q.row_amax + r0, 0, static_cast<size_t>(rows) * sizeof(float), stream);
      if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "row_amax memset: %s", cudaGetErrorString(e));
    }
    g.row_amax = q.row_amax;
  }
  if (q.scatter_bases != nullptr && q.scatter_rows > 0) {
    for (int o = 0; o < 8; ++o) g.scatter_bases[o] = q.scatter_bases[o];
    g.scatter_row0 = q.scatter_row0;
    g.scatter_rows = q.scatter_rows;
  }
  if (q.ev_begin != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(q.ev_begin), stream);
  // Launched programmatically behind this call's own quantiser stage: what it touches before its wait (the tile list and
  // the claim counter) must come from at least two kernels back.  The routing kernel clears the counter, or the quantiser
  // with the LoRA-A projection behind it; without either the caller passes no counter (fixed stride).
  rc = launch_gemm(g, stream, !q.skip_quant && q.ev_begin == nullptr && q.ev_end == nullptr, &q.src,
                   q.split.count > 0 ? &q.split : nullptr);
  if (q.ev_end != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(q.ev_end), stream);
  return rc;
}

}  // namespace skyrl

using namespace skyrl;

extern "C" int skyrl_w8a8_abi_version(void) { return SKYRL_W8A8_ABI_VERSION; }
extern "C" const char* skyrl_w8a8_last_error(void) { return g_last_error; }

extern "C" int skyrl_w8a8_stream_capture_id(skyrl_stream_t stream, uint64_t* id) {
  if (id == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "stream_capture_id: id is null");
  cudaStreamCaptureStatus state = cudaStreamCaptureStatusNone;
  unsigned long long capture = 0;
  const cudaError_t e = cudaStreamGetCaptureInfo(static_cast<cudaStream_t>(stream), &state, &capture);
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "stream_capture_id: %s", cudaGetErrorString(e));
  *id = state == cudaStreamCaptureStatusActive ? capture : 0;
  return SKYRL_OK;
}

extern "C" size_t skyrl_w8a8_linear_workspace_bytes(int32_t m, int32_t n, int32_t k, int32_t num_adapters) {
  if (m <= 0 || n <= 0 || k <= 0) return 0;
  return carve_linear(nullptr, m, n, k, num_adapters).bytes;
}

extern "C" size_t skyrl_w8a8_mlp_workspace_bytes(int32_t m, int32_t hidden, int32_t inter, int32_t num_adapters) {
  if (m <= 0 || hidden <= 0 || inter <= 0) return 0;
  return carve_mlp(nullptr, m, hidden, inter, num_adapters).bytes;
}

static int linear_forward(const SkyrlW8A8LinearArgs* a, const ColumnSplit& split, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "linear: args is null");
  if (a->struct_size != sizeof(SkyrlW8A8LinearArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "linear: struct_size %u does not match ABI v%d (%zu)", a->struct_size,
                SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8LinearArgs));
  if (a->m <= 0 || a->n <= 0 || a->k <= 0) return fail(SKYRL_ERR_INVALID_ARGUMENT, "linear: non-positive shape");
  if (a->x == nullptr || a->wq == nullptr || a->sw == nullptr || a->out == nullptr || a->status == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "linear: null buffer");
  if (a->rank < 0 || a->rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_UNSUPPORTED, "linear: LoRA rank must be in [0, %d], got %d", SKYRL_LORA_RANK_PAD, a->rank);
  const bool lora = a->rank > 0;
  if (lora && (a->lora_a_packed == nullptr || a->lora_b_packed == nullptr || a->lora_scaling == nullptr ||
               a->num_adapters <= 0))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "linear: LoRA tables missing");
  if (a->adapter_ids != nullptr && a->num_adapters <= 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "linear: adapter ids given without adapters");
  const int na = a->num_adapters > 0 ? a->num_adapters : 1;
  const LinearWs w = carve_linear(a->workspace, a->m, a->n, a->k, na);
  int rc = check_ws(a->workspace, a->workspace_bytes, w.bytes, "linear");
  if (rc) return rc;
  const bool rows_path = a->m <= ROWS_PATH_MAX_M;
  const bool routed = a->adapter_ids != nullptr && !rows_path;

  if (routed && (rc = launch_route_dense(a->adapter_ids, a->m, na, w.route.perm, w.route.tiles, w.route.seg_mask,
                                         w.route.seg_adapter, a->status, stream, w.sched, SCHED_WORDS)))
    return rc;
  Projection q = {};
  q.x = a->x;
  q.x_stride = a->x_row_stride;
  q.rms_delta = a->rms_delta;
  q.eps = a->rms_eps;
  q.gather = routed ? w.route.perm : nullptr;
  q.keep_xn = routed || a->rms_delta != nullptr || a->x_row_stride != a->k;
  q.two_step_rows = (a->flags & SKYRL_LINEAR_FUSED_ROWS) == 0;
  q.gemm_variant = static_cast<int>((a->flags >> SKYRL_FLAGS_GEMM_VARIANT_SHIFT) & 7u);
  q.m = a->m;
  q.n = a->n;
  q.k = a->k;
  q.rank = a->rank;
  q.na = na;
  q.wq = a->wq;
  q.sw = a->sw;
  q.a_packed = a->lora_a_packed;
  q.b_packed = a->lora_b_packed;
  q.scaling = a->lora_scaling;
  q.ids = a->adapter_ids;
  q.xq = w.xq;
  q.sx = w.sx;
  q.xn = w.xn;
  q.z_parts = w.z_parts;
  q.acc = w.acc;
  q.b_rows = a->lora_b_rows;
  q.b_rows_rank = a->lora_b_rows_rank;
  q.src = tile_source(w.route, routed, 0, a->m);
  q.epilogue = a->epilogue;
  q.split = split;
  q.out_row_map = routed ? w.route.perm : nullptr;
  q.residual = a->residual;
  q.residual_stride = a->residual_row_stride;
  q.out = a->out;
  q.out_stride = a->out_row_stride;
  q.status = a->status;
  if (!rows_path && (routed || a->rank > 0)) q.sched = w.sched;
  if (!rows_path && !routed) q.zero_words = q.sched;
  q.ev_begin = a->timing_events[0];
  q.ev_end = a->timing_events[1];
  return run_projection(q, stream);
}

extern "C" int skyrl_w8a8_lora_forward_sm100_v1(const SkyrlW8A8LinearArgs* a, skyrl_stream_t stream) {
  return linear_forward(a, ColumnSplit{}, stream);
}

extern "C" int skyrl_w8a8_lora_forward_split_sm100_v1(const SkyrlW8A8LinearArgs* a, int32_t parts, const int32_t* part_cols,
                                                      void* const* outs, skyrl_stream_t stream) {
  if (a == nullptr || part_cols == nullptr || outs == nullptr || parts < 1 || parts > 4)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "split linear: one to four parts");
  if (a->struct_size != sizeof(SkyrlW8A8LinearArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "split linear: struct_size %u does not match", a->struct_size);
  ColumnSplit s = {};
  s.count = parts;
  for (int i = 0; i < parts; ++i) {
    if (part_cols[i] <= 0 || part_cols[i] % 32 != 0 || part_cols[i] > (1 << 24) || outs[i] == nullptr || !aligned16(outs[i]))
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "split linear: part %d needs a multiple of 32 columns and a 16-byte aligned output", i);
    s.off[i + 1] = s.off[i] + part_cols[i];
    s.base[i] = outs[i];
  }
  s.group = s.off[parts];
  if (a->epilogue != SKYRL_EPI_LINEAR || a->rank <= 0 || (a->flags & SKYRL_LINEAR_FUSED_ROWS) != 0 || a->n % s.group != 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "split linear: a linear with a LoRA term whose N is whole groups of the parts");
  return linear_forward(a, s, stream);
}

// ---- group-wise scales ---------------------------------------------------------
namespace skyrl {

struct GroupedWs {
  RouteWs route;
  int8_t* xq;
  float* sx;           // [groups, m]
  uint16_t* xn;
  uint16_t* z_parts;
  size_t bytes;
};

static GroupedWs carve_grouped(void* ws, int m, int k, int num_adapters, int group) {
  Carver c(ws);
  GroupedWs w;
  w.route = carve_route(c, m, num_adapters);
  w.xq = c.take<int8_t>(static_cast<size_t>(m) * k);
  w.sx = c.take<float>(static_cast<size_t>(m) * (k / group));
  w.xn = c.take<uint16_t>(static_cast<size_t>(m) * k);
  w.z_parts = c.take<uint16_t>(SKYRL_Z_PARTS * static_cast<size_t>(m) * SKYRL_LORA_RANK_PAD);
  w.bytes = c.total();
  return w;
}

}  // namespace skyrl

extern "C" size_t skyrl_w8a8_grouped_workspace_bytes(int32_t m, int32_t n, int32_t k, int32_t num_adapters,
                                                      int32_t group_size) {
  if (m <= 0 || n <= 0 || k <= 0 || group_size <= 0) return 0;
  return carve_grouped(nullptr, m, k, num_adapters, group_size).bytes;
}

extern "C" int skyrl_w8a8_lora_forward_grouped_sm100_v1(const SkyrlW8A8LinearArgs* a, int32_t group_size,
                                                         skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped linear: args is null");
  if (a->struct_size != sizeof(SkyrlW8A8LinearArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped linear: struct_size %u does not match ABI v%d (%zu)", a->struct_size,
                SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8LinearArgs));
  if (a->m <= 0 || a->n <= 0 || a->k <= 0) return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped linear: non-positive shape");
  if (group_size <= 0 || group_size % 32 != 0 || a->k % group_size != 0)
    return fail(SKYRL_ERR_UNSUPPORTED, "grouped linear: the group must be a multiple of 32 that divides K, got %d of %d", group_size, a->k);
  if (a->x == nullptr || a->wq == nullptr || a->sw == nullptr || a->out == nullptr || a->status == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped linear: null buffer");
  if (a->epilogue != SKYRL_EPI_LINEAR || a->rms_delta != nullptr || a->residual != nullptr)
    return fail(SKYRL_ERR_UNSUPPORTED, "grouped linear: plain linear epilogue only");
  if (a->rank < 0 || a->rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_UNSUPPORTED, "grouped linear: LoRA rank must be in [0, %d], got %d", SKYRL_LORA_RANK_PAD, a->rank);
  const bool lora = a->rank > 0;
  if (lora && (a->lora_a_packed == nullptr || a->lora_b_packed == nullptr || a->lora_scaling == nullptr || a->num_adapters <= 0))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped linear: LoRA tables missing");
  const int na = a->num_adapters > 0 ? a->num_adapters : 1;
  const GroupedWs w = carve_grouped(a->workspace, a->m, a->k, na, group_size);
  int rc = check_ws(a->workspace, a->workspace_bytes, w.bytes, "grouped linear");
  if (rc) return rc;
  // adapters in sorted order above one tile of rows, by masks over token order within one
  const bool routed = lora && a->adapter_ids != nullptr;
  if (routed && (rc = launch_route_dense(a->adapter_ids, a->m, na, w.route.perm, w.route.tiles, w.route.seg_mask,
                                         w.route.seg_adapter, a->status, stream, nullptr, 0)))
    return rc;
  const int32_t* perm = routed && a->m > SKYRL_TILE_ROWS ? w.route.perm : nullptr;
  const bool copy = lora && (perm != nullptr || a->x_row_stride != a->k);
  if ((rc = launch_group_quant(a->x, a->x_row_stride, perm, a->m, a->k, group_size, w.xq, w.sx, copy ? w.xn : nullptr, stream)))
    return rc;
  const TileSource src = tile_source(w.route, routed, 0, a->m);
  if (lora && (rc = launch_lora_a_proj(copy ? static_cast<const void*>(w.xn) : a->x, a->m, a->k, a->lora_a_packed,
                                       a->lora_scaling, na, a->rank, src, src.count, w.z_parts, a->status, stream)))
    return rc;
  GroupedGemmLaunch g = {};
  g.m = a->m;
  g.n = a->n;
  g.k = a->k;
  g.group = group_size;
  g.rank = a->rank;
  g.num_adapters = na;
  g.src = src;
  g.xq = w.xq;
  g.sx = w.sx;
  g.wq = a->wq;
  g.sw = a->sw;
  g.z_parts = w.z_parts;
  g.b_table = a->lora_b_rows != nullptr ? a->lora_b_rows : a->lora_b_packed;
  g.b_slots = a->lora_b_rows != nullptr ? a->lora_b_rows_rank : SKYRL_LORA_RANK_PAD;
  g.out_row_map = perm;
  g.out = a->out;
  g.out_stride = a->out_row_stride;
  g.status = a->status;
  return launch_grouped_gemm(g, stream);
}

// ---- training step -----------------------------------------------------------------
namespace skyrl {

struct TrainSaved {
  RouteWs route;
  int32_t* adapter_start;  // [A + 1]
  uint16_t* z_parts;       // s (x A) of the sorted rows
  size_t bytes;
};
static TrainSaved carve_train_saved(void* base, int m, int num_adapters) {
  Carver c(base);
  TrainSaved s;
  s.route = carve_route(c, m, num_adapters);
  s.adapter_start = c.take<int32_t>(num_adapters + 1);
  s.z_parts = c.take<uint16_t>(SKYRL_Z_PARTS * static_cast<size_t>(m) * SKYRL_LORA_RANK_PAD);
  s.bytes = c.total();
  return s;
}

// What a forward keeps may lie elsewhere by the time of the backward (a host that moves activations out and back), so it
// needs no more than the 16 bytes of its tensor map and its vector loads.
static int check_saved(const SkyrlW8A8TrainArgs* a, size_t need, const char* who) {
  if (a->saved == nullptr || !aligned16(a->saved))
    return fail(SKYRL_ERR_WORKSPACE, "%s: saved must be non-null and 16-byte aligned", who);
  if (a->saved_bytes < need) return fail(SKYRL_ERR_WORKSPACE, "%s: saved has %zu bytes, %zu needed", who, a->saved_bytes, need);
  return SKYRL_OK;
}

struct TrainWs {
  int32_t* sched;
  int8_t* xq;        // forward
  float* sx;
  uint16_t* rows;    // gathered rows of x (forward) or dy (backward)
  uint16_t* at;      // forward: tables in kernel layout
  uint16_t* bt;
  int8_t* q;         // backward: two planes
  float* s;
  uint16_t* zb;
  TrainSaved own;    // backward without `saved`
  size_t bytes;
};
static TrainWs carve_train(void* ws, int m, int n, int k, int rank, int num_adapters, bool backward) {
  Carver c(ws);
  TrainWs w = {};
  const size_t mm = static_cast<size_t>(m);
  w.sched = c.take<int32_t>(SCHED_WORDS);
  if (!backward) {
    w.xq = c.take<int8_t>(mm * k);
    w.sx = c.take<float>(mm);
    w.rows = c.take<uint16_t>(mm * k);
    w.at = c.take<uint16_t>(static_cast<size_t>(num_adapters) * rank * k);
    w.bt = c.take<uint16_t>(static_cast<size_t>(num_adapters) * n * ((rank + 7) / 8 * 8));
  } else {
    w.q = c.take<int8_t>(2 * mm * n);
    w.s = c.take<float>(2 * mm);
    w.rows = c.take<uint16_t>(mm * n);
    w.zb = c.take<uint16_t>(SKYRL_Z_PARTS * mm * SKYRL_LORA_RANK_PAD);
    c.off = align_up(c.off, 1024);
    w.own = carve_train_saved(c.base != nullptr ? c.base + c.off : nullptr, m, num_adapters);
    c.off += w.own.bytes;
  }
  w.bytes = c.total();
  return w;
}

static int check_train(const SkyrlW8A8TrainArgs* a, const char* who) {
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: args is null", who);
  if (a->struct_size != sizeof(SkyrlW8A8TrainArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: struct_size %u does not match ABI v%d (%zu)", who, a->struct_size,
                SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8TrainArgs));
  if (a->m <= 0 || a->n <= 0 || a->k <= 0 || a->n % 32 != 0 || a->k % 16 != 0 || a->n_logical <= 0 || a->n_logical > a->n)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: bad shape", who);
  if (a->wq == nullptr || a->sw == nullptr || a->status == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: null buffer", who);
  if (a->rank < 0 || a->rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_UNSUPPORTED, "%s: LoRA rank must be in [0, %d], got %d", who, SKYRL_LORA_RANK_PAD, a->rank);
  return SKYRL_OK;
}

}  // namespace skyrl

extern "C" size_t skyrl_w8a8_train_saved_bytes(int32_t m, int32_t num_adapters) {
  if (m <= 0) return 0;
  return carve_train_saved(nullptr, m, num_adapters > 0 ? num_adapters : 1).bytes;
}

extern "C" size_t skyrl_w8a8_train_workspace_bytes(int32_t m, int32_t n, int32_t k, int32_t rank, int32_t num_adapters,
                                                    int32_t backward) {
  if (m <= 0 || n <= 0 || k <= 0 || rank < 0) return 0;
  return carve_train(nullptr, m, n, k, rank, num_adapters > 0 ? num_adapters : 1, backward != 0).bytes;
}

extern "C" int skyrl_w8a8_train_forward_sm100_v1(const SkyrlW8A8TrainArgs* a, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int rc = check_train(a, "train_forward");
  if (rc) return rc;
  if (a->x == nullptr || a->y == nullptr || a->rank <= 0 || a->lora_a == nullptr || a->lora_b == nullptr ||
      a->lora_scaling == nullptr || a->num_adapters <= 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "train_forward: null buffer or LoRA tables missing");
  const int na = a->num_adapters;
  const TrainSaved sv = carve_train_saved(a->saved, a->m, na);
  const TrainWs w = carve_train(a->workspace, a->m, a->n, a->k, a->rank, na, false);
  if ((rc = check_saved(a, sv.bytes, "train_forward"))) return rc;
  if ((rc = check_ws(a->workspace, a->workspace_bytes, w.bytes, "train_forward"))) return rc;
  const bool routed = a->adapter_ids != nullptr;
  if ((rc = launch_train_tables(a->lora_a, a->lora_b, na, a->k, a->n_logical, a->n, a->rank, w.at, w.bt, stream))) return rc;
  if (routed && (rc = launch_route_dense(a->adapter_ids, a->m, na, sv.route.perm, sv.route.tiles, sv.route.seg_mask,
                                         sv.route.seg_adapter, a->status, stream, nullptr, 0, true, sv.adapter_start)))
    return rc;
  const int32_t* perm = routed ? sv.route.perm : nullptr;
  const bool copy = routed || a->x_row_stride != a->k;
  if ((rc = launch_rms_quant(a->x, a->x_row_stride, nullptr, 0.f, perm, a->m, a->k, w.xq, w.sx, copy ? w.rows : nullptr,
                             stream, nullptr, w.sched)))
    return rc;
  const TileSource src = tile_source(sv.route, routed, 0, a->m);
  if ((rc = launch_lora_a_proj(copy ? static_cast<const void*>(w.rows) : a->x, a->m, a->k, w.at, a->lora_scaling, na,
                               a->rank, src, src.count, sv.z_parts, a->status, stream, 0, -1, nullptr, 0, -1, a->rank)))
    return rc;
  SkyrlW8A8GemmArgs g = {};
  g.struct_size = sizeof(g);
  g.epilogue = SKYRL_EPI_LINEAR;
  g.m = a->m;
  g.n = a->n;
  g.k = a->k;
  g.rank = a->rank;
  g.num_adapters = na;
  g.xq = w.xq;
  g.sx = w.sx;
  g.wq = a->wq;
  g.sw = a->sw;
  g.z_parts = sv.z_parts;
  g.lora_b_packed = w.bt;
  g.lora_b_rows = w.bt;
  g.lora_b_rows_rank = (a->rank + 7) / 8 * 8;
  g.out_row_map = perm;
  g.out = a->y;
  g.out_row_stride = a->n;
  g.status = a->status;
  g.sched = w.sched;
  return launch_gemm(g, stream, true, &src);
}

extern "C" int skyrl_w8a8_train_backward_sm100_v1(const SkyrlW8A8TrainArgs* a, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int rc = check_train(a, "train_backward");
  if (rc) return rc;
  const bool grads = a->saved != nullptr;
  const bool lora = a->rank > 0;
  if (a->dy == nullptr || (a->dx == nullptr && !grads) ||
      (grads && (a->x == nullptr || a->da == nullptr || a->db == nullptr || !lora)))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "train_backward: null buffer");
  if (lora && (a->bwd_a == nullptr || a->bwd_b == nullptr || a->lora_scaling == nullptr || a->num_adapters <= 0))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "train_backward: LoRA tables missing");
  const int na = a->num_adapters > 0 ? a->num_adapters : 1;
  const TrainWs w = carve_train(a->workspace, a->m, a->n, a->k, a->rank, na, true);
  if ((rc = check_ws(a->workspace, a->workspace_bytes, w.bytes, "train_backward"))) return rc;
  TrainSaved sv = w.own;
  const bool routed = lora && a->adapter_ids != nullptr;
  if (grads) {
    sv = carve_train_saved(a->saved, a->m, na);
    if ((rc = check_saved(a, sv.bytes, "train_backward"))) return rc;
  } else if (routed && (rc = launch_route_dense(a->adapter_ids, a->m, na, sv.route.perm, sv.route.tiles, sv.route.seg_mask,
                                                sv.route.seg_adapter, a->status, stream, nullptr, 0, true, sv.adapter_start))) {
    return rc;
  }
  const int32_t* perm = routed ? sv.route.perm : nullptr;
  const TileSource src = tile_source(sv.route, routed, 0, a->m);
  const bool copy = lora && (routed || a->dy_row_stride != a->n);
  const size_t plane = static_cast<size_t>(a->m) * a->n;
  if ((rc = launch_grad_quant(a->dy, a->dy_row_stride, a->sw, perm, a->m, a->n, w.q, w.s, w.q + plane, w.s + a->m, stream,
                              copy ? w.rows : nullptr)))
    return rc;
  if (lora && (rc = launch_lora_a_proj(copy ? static_cast<const void*>(w.rows) : a->dy, a->m, a->n, a->bwd_a, a->lora_scaling,
                                       na, a->rank, src, src.count, w.zb, a->status, stream, 0, -1, nullptr, 0, -1,
                                       a->bwd_a_rows, a->bwd_a_cols)))
    return rc;
  if (a->dx != nullptr) {
    PlanesGemmLaunch g = {};
    g.m = a->m;
    g.n = a->k;
    g.k = a->n;
    g.rank = a->rank;
    g.num_adapters = na;
    g.src = src;
    g.q = w.q;
    g.s = w.s;
    g.wq = a->wq;
    g.z_parts = w.zb;
    g.b_table = a->bwd_b;
    g.b_slots = a->bwd_b_slots;
    g.out_row_map = perm;
    g.out = a->dx;
    g.out_stride = a->k;
    g.status = a->status;
    if ((rc = launch_planes_gemm(g, stream))) return rc;
  }
  if (!grads) return SKYRL_OK;
  LoraGradLaunch q = {};
  q.m = a->m;
  q.k = a->k;
  q.n = a->n;
  q.n_logical = a->n_logical;
  q.adapters = na;
  q.rank = a->rank;
  q.x = a->x;
  q.x_stride = a->x_row_stride;
  q.dy = a->dy;
  q.dy_stride = a->dy_row_stride;
  q.z = sv.z_parts;
  q.zb = w.zb;
  q.perm = perm;
  q.adapter_start = routed ? sv.adapter_start : nullptr;
  q.da = a->da;
  q.db = a->db;
  q.status = a->status;
  return launch_lora_grad(q, stream);
}

// One exported target per fused variant: thin wrappers that check what the variant needs and fix the epilogue.
extern "C" int skyrl_rms_gate_up_w8a8_lora_swiglu_sm100_v1(const SkyrlW8A8LinearArgs* a, skyrl_stream_t stream) {
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "rms_gate_up_swiglu: args is null");
  if (a->struct_size != sizeof(SkyrlW8A8LinearArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "rms_gate_up_swiglu: struct_size %u does not match ABI v%d (%zu)",
                a->struct_size, SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8LinearArgs));
  if (a->residual != nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "rms_gate_up_swiglu: takes no residual");
  if (a->n % 2 != 0) return fail(SKYRL_ERR_INVALID_ARGUMENT, "rms_gate_up_swiglu: n must count (gate, up) pairs");
  SkyrlW8A8LinearArgs b = *a;
  b.epilogue = SKYRL_EPI_SWIGLU;
  return skyrl_w8a8_lora_forward_sm100_v1(&b, stream);
}

extern "C" int skyrl_down_w8a8_lora_residual_sm100_v1(const SkyrlW8A8LinearArgs* a, skyrl_stream_t stream) {
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "down_residual: args is null");
  if (a->struct_size != sizeof(SkyrlW8A8LinearArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "down_residual: struct_size %u does not match ABI v%d (%zu)",
                a->struct_size, SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8LinearArgs));
  if (a->residual == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "down_residual: residual is null");
  if (a->rms_delta != nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "down_residual: takes no RMSNorm weights");
  SkyrlW8A8LinearArgs b = *a;
  b.epilogue = SKYRL_EPI_RESIDUAL;
  return skyrl_w8a8_lora_forward_sm100_v1(&b, stream);
}

namespace skyrl {

// What one MLP call works on: the carved workspace and the chunk of sorted rows with its tile list.
struct MlpPlan {
  MlpWs w;
  int na;
  bool rows_path, routed, chunked;
  const int32_t* perm;
  int chunk_rows, row0, rows;
  TileSource src;
};

static int plan_mlp(const SkyrlW8A8MlpArgs* a, const char* who, MlpPlan* pl) {
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: args is null", who);
  if (a->struct_size != sizeof(SkyrlW8A8MlpArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: struct_size %u does not match ABI v%d (%zu)", who, a->struct_size,
                SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8MlpArgs));
  if (a->m <= 0 || a->hidden <= 0 || a->inter <= 0) return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: non-positive shape", who);
  if (a->x == nullptr || a->gu_wq == nullptr || a->gu_sw == nullptr || a->dn_wq == nullptr || a->dn_sw == nullptr ||
      a->out == nullptr || a->status == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: null buffer", who);
  if (a->down_epilogue != SKYRL_EPI_RESIDUAL && a->down_epilogue != SKYRL_EPI_PARTIAL_F32 &&
      a->down_epilogue != SKYRL_EPI_LINEAR)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: down_epilogue must be RESIDUAL, LINEAR or PARTIAL_F32", who);
  if (a->rank < 0 || a->rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_UNSUPPORTED, "%s: LoRA rank must be in [0, %d], got %d", who, SKYRL_LORA_RANK_PAD, a->rank);
  const bool lora = a->rank > 0;
  if (lora && (a->gu_a_packed == nullptr || a->gu_b_packed == nullptr || a->gu_scaling == nullptr ||
               a->dn_a_packed == nullptr || a->dn_b_packed == nullptr || a->dn_scaling == nullptr ||
               a->num_adapters <= 0))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: LoRA tables missing", who);
  pl->na = a->num_adapters > 0 ? a->num_adapters : 1;
  pl->w = carve_mlp(a->workspace, a->m, a->hidden, a->inter, pl->na);
  int rc = check_ws(a->workspace, a->workspace_bytes, pl->w.bytes, who);
  if (rc) return rc;
  pl->rows_path = a->m <= ROWS_PATH_MAX_M;
  pl->routed = a->adapter_ids != nullptr && !pl->rows_path;
  pl->perm = pl->routed ? pl->w.route.perm : nullptr;
  pl->chunked = a->num_chunks > 1 && !pl->rows_path;
  if (pl->chunked && (a->num_chunks > MAX_CHUNKS || a->chunk_index < 0 || a->chunk_index >= a->num_chunks))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "%s: num_chunks must be <= %d and chunk_index inside it", who, MAX_CHUNKS);
  pl->chunk_rows = pl->chunked ? ((a->m + a->num_chunks - 1) / a->num_chunks + SKYRL_TILE_ROWS - 1) / SKYRL_TILE_ROWS *
                                     SKYRL_TILE_ROWS
                               : 0;
  pl->row0 = pl->chunked ? a->chunk_index * pl->chunk_rows : 0;
  pl->rows = pl->chunked ? (a->m - pl->row0 < pl->chunk_rows ? a->m - pl->row0 : pl->chunk_rows) : a->m;
  pl->src = tile_source(pl->w.route, pl->routed, pl->row0, pl->rows > 0 ? pl->rows : 0);
  return SKYRL_OK;
}

static int route_mlp(const SkyrlW8A8MlpArgs* a, const MlpPlan& pl, cudaStream_t stream) {
  if ((a->flags & SKYRL_MLP_REUSE_ROUTING) != 0 || !pl.routed) return SKYRL_OK;
  const RouteWs& r = pl.w.route;
  return launch_route_dense(a->adapter_ids, a->m, pl.na, r.perm, r.tiles, r.seg_mask, r.seg_adapter, a->status, stream,
                            pl.w.sched, SCHED_WORDS);
}

// front half: RMSNorm -> quant -> gate_up W8A8 LoRA -> SwiGLU; h keeps the row order of the GEMM
static Projection front_projection(const SkyrlW8A8MlpArgs* a, const MlpPlan& pl) {
  const MlpWs& w = pl.w;
  Projection q = {};
  q.x = a->x;
  q.x_stride = a->hidden;
  q.rms_delta = a->rms_delta;
  q.eps = a->rms_eps;
  q.gather = pl.perm;
  // small batches need no re-laid-out copy of x; they write one only when asked to (stage checks)
  q.keep_xn = pl.rows_path ? (a->flags & SKYRL_MLP_KEEP_NORMALIZED) != 0 : (pl.routed || a->rms_delta != nullptr);
  q.two_step_rows = (a->flags & SKYRL_MLP_FUSED_ROWS) == 0;
  q.gemm_variant = static_cast<int>((a->flags >> SKYRL_FLAGS_GEMM_VARIANT_SHIFT) & 7u);
  q.m = a->m;
  q.n = 2 * a->inter;
  q.k = a->hidden;
  q.rank = a->rank;
  q.na = pl.na;
  q.q_row0 = pl.row0;
  q.q_rows = pl.rows;
  q.list_row0 = pl.row0;
  q.cta_limit = a->gemm_cta_limit;
  q.wq = a->gu_wq;
  q.sw = a->gu_sw;
  q.a_packed = a->gu_a_packed;
  q.b_packed = a->gu_b_packed;
  q.scaling = a->gu_scaling;
  q.ids = a->adapter_ids;
  q.xq = w.xq;
  q.sx = w.sx;
  q.xn = w.xn;
  q.z_parts = w.z_parts;
  q.acc = w.acc;
  q.b_rows = a->gu_b_rows;
  q.b_rows_rank = a->b_rows_rank;
  q.src = pl.src;
  q.epilogue = SKYRL_EPI_SWIGLU;
  q.out_row_map = nullptr;
  q.out = w.h;
  q.out_stride = a->inter;
  q.status = a->status;
  // odd and even chunks claim tiles through counter pairs of their own, so that two chunks of one block may run
  // on two streams at the same time
  // (Without adapter ids no routing kernel runs to clear the words: a whole block's quantiser does, with the projection
  // between it and the GEMM; the chunks of a block without ids, and a block without LoRA, take their tiles with a fixed
  // stride.)
  if (pl.routed || (!pl.rows_path && !pl.chunked && a->rank > 0))
    q.sched = w.sched + (pl.chunked ? (a->chunk_index & 1) * 4 : 0);
  q.ev_begin = a->timing_events[0];
  q.ev_end = a->timing_events[1];
  return q;
}

}  // namespace skyrl

extern "C" int skyrl_w8a8_mlp_block_sm100_v1(const SkyrlW8A8MlpArgs* a, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  MlpPlan pl;
  int rc = plan_mlp(a, "mlp", &pl);
  if (rc) return rc;
  if (pl.rows <= 0) return SKYRL_OK;  // more chunks than rows: nothing to do for this one
  const bool prepared = (a->flags & SKYRL_MLP_INPUT_PREPARED) != 0;
  if (prepared && pl.rows_path)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "mlp: SKYRL_MLP_INPUT_PREPARED needs more than %d rows", ROWS_PATH_MAX_M);
  if ((rc = route_mlp(a, pl, stream))) return rc;
  const MlpWs& w = pl.w;

  Projection q = front_projection(a, pl);
  q.skip_quant = prepared;
  // sorted route: the gate_up epilogue collects the absmax of every row of h, so that quantising h is one
  // streaming pass (SKYRL_MLP_NO_ROW_AMAX keeps the two-pass quantiser; the two must agree bit for bit)
  const bool collect = !pl.rows_path && (a->flags & SKYRL_MLP_NO_ROW_AMAX) == 0;
  q.row_amax = collect ? w.h_amax : nullptr;
  q.zero_amax = q.row_amax;
  if (!pl.routed && !pl.rows_path && !pl.chunked) {
    if (prepared) q.sched = nullptr;  // the rows were prepared by a call of their own
    else q.zero_words = q.sched;
  }
  if (pl.rows_path && a->prefetch_down_bytes > 0) {
    // the down weights travel to L2 while the row-wise kernels behind gate_up run
    const int64_t dn_bytes = static_cast<int64_t>((a->inter + SKYRL_WEIGHT_KBLOCK - 1) / SKYRL_WEIGHT_KBLOCK) * a->hidden * SKYRL_WEIGHT_KBLOCK;
    q.prefetch = a->dn_wq;
    q.prefetch_bytes = (a->prefetch_down_bytes < dn_bytes ? a->prefetch_down_bytes : dn_bytes) / 16 * 16;
  }
  if ((rc = run_projection(q, stream))) return rc;

  // back half: quant(h) -> down W8A8 LoRA -> + residual, rows scattered back to token order
  q.skip_quant = false;
  q.row_amax = nullptr;
  q.zero_amax = nullptr;
  q.zero_words = nullptr;
  q.known_amax = collect ? w.h_amax : nullptr;
  q.x = w.h;
  q.x_stride = a->inter;
  q.rms_delta = nullptr;
  q.gather = nullptr;
  q.keep_xn = false;
  q.n = a->hidden;
  q.k = a->inter;
  q.wq = a->dn_wq;
  q.sw = a->dn_sw;
  q.a_packed = a->dn_a_packed;
  q.b_packed = a->dn_b_packed;
  q.b_rows = a->dn_b_rows;
  q.scaling = a->dn_scaling;
  q.xq = w.hq;
  q.sx = w.sh;
  if (q.sched != nullptr) q.sched += 2;
  q.prefetch = nullptr;
  q.prefetch_bytes = 0;
  if (pl.rows_path && a->prefetch_next != nullptr && a->prefetch_next_bytes > 0) {
    q.prefetch = a->prefetch_next;
    q.prefetch_bytes = a->prefetch_next_bytes;
  }
  q.epilogue = a->down_epilogue;
  q.out_row_map = a->down_epilogue == SKYRL_EPI_PARTIAL_F32 ? nullptr : pl.perm;
  q.residual = a->residual != nullptr ? a->residual : a->x;
  q.residual_stride = a->hidden;
  q.out = a->out;
  q.out_stride = a->hidden;
  if (a->tp_scatter_rows > 0) {
    if (a->down_epilogue != SKYRL_EPI_PARTIAL_F32 || pl.rows_path)
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "mlp: tp_scatter_rows needs down_epilogue PARTIAL_F32 and more than %d rows",
                  ROWS_PATH_MAX_M);
    q.scatter_bases = a->tp_scatter_bases;
    q.scatter_row0 = pl.row0;
    q.scatter_rows = a->tp_scatter_rows;
  }
  q.ev_begin = a->timing_events[2];
  q.ev_end = a->timing_events[3];
  return run_projection(q, stream);
}

extern "C" int skyrl_w8a8_mlp_tp_prepare_sm100_v1(const SkyrlW8A8MlpArgs* a, int32_t row_begin, int32_t row_count,
                                                   skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  MlpPlan pl;
  int rc = plan_mlp(a, "tp_prepare", &pl);
  if (rc) return rc;
  if (pl.rows_path)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_prepare: needs more than %d rows", ROWS_PATH_MAX_M);
  if (row_count <= 0 || row_begin < pl.row0 || row_begin + row_count > pl.row0 + pl.rows)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_prepare: rows [%d, %d) are not inside chunk rows [%d, %d)", row_begin,
                row_begin + row_count, pl.row0, pl.row0 + pl.rows);
  if ((rc = route_mlp(a, pl, stream))) return rc;
  Projection q = front_projection(a, pl);
  q.q_row0 = row_begin;
  q.q_rows = row_count;
  return run_quant_stage(q, stream);
}

extern "C" int skyrl_w8a8_mlp_workspace_regions(int32_t m, int32_t hidden, int32_t inter, int32_t num_adapters,
                                                 size_t* offsets) {
  if (m <= 0 || hidden <= 0 || inter <= 0 || offsets == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "workspace_regions: bad argument");
  unsigned char* const base = reinterpret_cast<unsigned char*>(static_cast<uintptr_t>(1024));
  const MlpWs w = carve_mlp(base, m, hidden, inter, num_adapters > 0 ? num_adapters : 1);
  offsets[0] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.xq) - base);
  offsets[1] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.sx) - base);
  offsets[2] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.z_parts) - base);
  return SKYRL_OK;
}

extern "C" int skyrl_w8a8_tp_signal_sm100_v1(int32_t* const* flags, int32_t count, int32_t value, skyrl_stream_t stream) {
  return launch_tp_signal(flags, count, value, static_cast<cudaStream_t>(stream));
}

extern "C" int skyrl_w8a8_tp_wait_sm100_v1(const int32_t* flags, int32_t count, int32_t value, int32_t* status,
                                            skyrl_stream_t stream) {
  return launch_tp_wait(flags, count, value, status, static_cast<cudaStream_t>(stream));
}

extern "C" int skyrl_w8a8_mlp_tp_exchange_sm100_v1(const SkyrlW8A8MlpArgs* blk, const SkyrlW8A8MlpArgs* next,
                                                    const SkyrlW8A8TpExchangeArgs* x, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (x == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: exchange args are null");
  if (x->struct_size != sizeof(SkyrlW8A8TpExchangeArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: struct_size %u does not match ABI v%d (%zu)", x->struct_size,
                SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8TpExchangeArgs));
  if (x->tp < 1 || x->tp > 8) return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: tp must be in [1, 8], got %d", x->tp);
  if (x->out == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: out is null");
  MlpPlan pl;
  int rc = plan_mlp(blk, "tp_exchange", &pl);
  if (rc) return rc;
  if (pl.rows_path) return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: needs more than %d rows", ROWS_PATH_MAX_M);
  if (x->row_count <= 0 || x->row_begin < 0 || x->row_begin + x->row_count > blk->m)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: rows [%d, %d) are outside [0, %d)", x->row_begin,
                x->row_begin + x->row_count, blk->m);
  TpExchangeLaunch e = {};
  e.tp = x->tp;
  for (int s = 0; s < x->tp; ++s) e.partial[s] = x->partials[s];
  e.row_begin = x->row_begin;
  e.row_count = x->row_count;
  e.hidden = blk->hidden;
  e.perm = pl.perm;
  e.residual = blk->residual != nullptr ? blk->residual : blk->x;
  e.out = x->out;
  e.out_sorted = (blk->flags & SKYRL_MLP_FINALIZE_SORTED) != 0;
  e.wait_flags = x->wait_flags;
  e.wait_value = x->wait_value;
  e.status = blk->status;
  if (static_cast<int64_t>(blk->m) * (blk->hidden >> 3) > 0x7fffffffLL)
    return fail(SKYRL_ERR_UNSUPPORTED, "tp_exchange: m * hidden / 8 must fit 31 bits");
  e.grid_ctas = x->grid_ctas;
  e.single_kernel = (x->flags & SKYRL_TP_EXCHANGE_SINGLE_KERNEL) != 0;
  e.multimem = (x->flags & SKYRL_TP_EXCHANGE_MULTIMEM) != 0;
  e.profile = (x->flags & SKYRL_TP_EXCHANGE_PROFILE) != 0;
  e.wide = (x->flags & SKYRL_TP_EXCHANGE_WIDE) != 0;
  MlpPlan np;
  const bool lora = next != nullptr && next->rank > 0;
  if (next != nullptr) {
    if ((rc = plan_mlp(next, "tp_exchange (next block)", &np))) return rc;
    if (next->m != blk->m || next->hidden != blk->hidden)
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: the next block has another shape");
    if (x->row_begin < np.row0 || x->row_begin + x->row_count > np.row0 + np.rows)
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: rows [%d, %d) are not inside the next block's chunk [%d, %d)",
                  x->row_begin, x->row_begin + x->row_count, np.row0, np.row0 + np.rows);
    unsigned char* const local = static_cast<unsigned char*>(next->workspace);
    const size_t off_xq = reinterpret_cast<unsigned char*>(np.w.xq) - local;
    const size_t off_sx = reinterpret_cast<unsigned char*>(np.w.sx) - local;
    e.quantize = true;
    e.delta = next->rms_delta;
    e.eps = next->rms_eps;
    e.xn = np.w.xn;  // the LoRA-A projection reads it; without LoRA it is still the scratch of the warp-per-row quantiser
    for (int r = 0; r < x->tp; ++r) {
      if (x->peer_workspaces[r] == nullptr || (reinterpret_cast<uintptr_t>(x->peer_workspaces[r]) & 1023u) != 0)
        return fail(SKYRL_ERR_WORKSPACE, "tp_exchange: workspace of rank %d is null or not 1024-byte aligned", r);
      unsigned char* const base = static_cast<unsigned char*>(x->peer_workspaces[r]);
      e.xq_dst[r] = reinterpret_cast<int8_t*>(base + off_xq);
      e.sx_dst[r] = reinterpret_cast<float*>(base + off_sx);
    }
  }
  if ((rc = launch_tp_exchange(e, stream))) return rc;
  if (lora) {
    // LoRA-A projection of the rows just normalised, its parts stored into every rank's workspace
    unsigned char* const local = static_cast<unsigned char*>(next->workspace);
    const size_t off_z = reinterpret_cast<unsigned char*>(np.w.z_parts) - local;
    void* extra[8];
    int extra_count = 0;
    for (int r = 0; r < x->tp; ++r) {
      void* dst = static_cast<unsigned char*>(x->peer_workspaces[r]) + off_z;
      if (dst != static_cast<void*>(np.w.z_parts)) extra[extra_count++] = dst;
    }
    if (extra_count > 7) return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_exchange: this rank's workspace is not among peer_workspaces");
    if ((rc = launch_lora_a_proj(np.w.xn, next->m, next->hidden, next->gu_a_packed, next->gu_scaling, np.na, next->rank,
                                 np.src, np.src.count, np.w.z_parts, next->status, stream, x->row_begin,
                                 x->row_begin + x->row_count, extra, extra_count, np.row0)))
      return rc;
  }
  bool any = false;
  for (int r = 0; r < x->tp; ++r) any = any || x->signal_flags[r] != nullptr;
  if (any) return launch_tp_signal(x->signal_flags, x->tp, x->signal_value, stream);
  return SKYRL_OK;
}

extern "C" int skyrl_w8a8_mlp_workspace_stage_regions(int32_t m, int32_t hidden, int32_t inter, int32_t num_adapters,
                                                       size_t* offsets) {
  if (m <= 0 || hidden <= 0 || inter <= 0 || offsets == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "workspace_stage_regions: bad argument");
  unsigned char* const base = reinterpret_cast<unsigned char*>(static_cast<uintptr_t>(1024));
  const MlpWs w = carve_mlp(base, m, hidden, inter, num_adapters > 0 ? num_adapters : 1);
  offsets[0] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.route.perm) - base);
  offsets[1] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.h) - base);
  offsets[2] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.hq) - base);
  offsets[3] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.sh) - base);
  offsets[4] = static_cast<size_t>(reinterpret_cast<unsigned char*>(w.xn) - base);
  return SKYRL_OK;
}

extern "C" int skyrl_w8a8_mlp_tp_unsort_sm100_v1(const SkyrlW8A8MlpArgs* a, const void* sorted_rows, void* out,
                                                  skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  MlpPlan pl;
  int rc = plan_mlp(a, "tp_unsort", &pl);
  if (rc) return rc;
  return launch_unsort_rows(sorted_rows, pl.perm, out, a->m, a->hidden, stream);
}

extern "C" int skyrl_w8a8_mlp_tp_finalize_sm100_v1(const SkyrlW8A8MlpArgs* a, const float* reduced, void* out,
                                                    int32_t row_begin, int32_t row_count, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (a == nullptr || reduced == nullptr || out == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_finalize: null argument");
  if (a->struct_size != sizeof(SkyrlW8A8MlpArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_finalize: struct_size does not match ABI v%d", SKYRL_W8A8_ABI_VERSION);
  if (a->m <= 0 || a->hidden <= 0 || a->hidden % 8 != 0 || row_begin < 0 || row_count <= 0 ||
      row_begin + row_count > a->m)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_finalize: bad shape or row range");
  const int na = a->num_adapters > 0 ? a->num_adapters : 1;
  const MlpWs w = carve_mlp(a->workspace, a->m, a->hidden, a->inter, na);
  int rc = check_ws(a->workspace, a->workspace_bytes, w.bytes, "tp_finalize");
  if (rc) return rc;
  const void* residual = a->residual != nullptr ? a->residual : a->x;
  const bool routed = a->adapter_ids != nullptr && a->m > ROWS_PATH_MAX_M;
  return launch_tp_finalize(reduced, routed ? w.route.perm : nullptr, residual, out, a->hidden, row_begin, row_count, stream,
                            (a->flags & SKYRL_MLP_FINALIZE_SORTED) != 0);
}

extern "C" int skyrl_w8a8_mlp_tp_finalize_slabs_sm100_v1(const SkyrlW8A8MlpArgs* a, const float* const* slabs,
                                                          int32_t num_slabs, void* out, int32_t row_begin,
                                                          int32_t row_count, skyrl_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (a == nullptr || slabs == nullptr || out == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_finalize_slabs: null argument");
  if (a->struct_size != sizeof(SkyrlW8A8MlpArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_finalize_slabs: struct_size does not match ABI v%d",
                SKYRL_W8A8_ABI_VERSION);
  if (a->m <= 0 || a->hidden <= 0 || a->hidden % 8 != 0 || row_begin < 0 || row_count <= 0 ||
      row_begin + row_count > a->m)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "tp_finalize_slabs: bad shape or row range");
  const int na = a->num_adapters > 0 ? a->num_adapters : 1;
  const MlpWs w = carve_mlp(a->workspace, a->m, a->hidden, a->inter, na);
  int rc = check_ws(a->workspace, a->workspace_bytes, w.bytes, "tp_finalize_slabs");
  if (rc) return rc;
  const void* residual = a->residual != nullptr ? a->residual : a->x;
  const bool routed = a->adapter_ids != nullptr && a->m > ROWS_PATH_MAX_M;
  return launch_tp_finalize_slabs(slabs, num_slabs, routed ? w.route.perm : nullptr, residual, out, a->hidden, row_begin,
                                  row_count, stream, (a->flags & SKYRL_MLP_FINALIZE_SORTED) != 0);
}

// ---------------------------------------------------------------------------
// W8A8 LoRA linear without a caller workspace: the scratch is a fixed array in
// this library's device image.  `g_noalloc_scratch` below is, in host code, only
// a handle for the symbol; the address kernels can use is looked up once per
// device with cudaGetSymbolAddress and cached.
// ---------------------------------------------------------------------------
// Beside the documented size there is room for what the segments of dense tiles take more than the two-adapter tile list
// they replaced (20 bytes a tile and 4 an adapter, at most 27 KB): whatever fitted before still does.
constexpr size_t NOALLOC_ARRAY_BYTES = SKYRL_NOALLOC_SCRATCH_BYTES + (64u << 10);
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_ARRAY_BYTES];

namespace skyrl {

static int noalloc_scratch(unsigned char** base, size_t* bytes) {
  static std::mutex mu;
  static unsigned char* cached[64] = {nullptr};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64)
    return fail(SKYRL_ERR_LAUNCH, "noalloc: no current CUDA device (%s)", cudaGetErrorString(e));
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);  // address of the array on the CURRENT device
    if (e != cudaSuccess || p == nullptr)
      return fail(SKYRL_ERR_LAUNCH, "noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    cached[dev] = static_cast<unsigned char*>(p);
  }
  // the operator carves its scratch on 1024-byte boundaries; the array is only 256-byte aligned
  const uintptr_t raw = reinterpret_cast<uintptr_t>(cached[dev]);
  const uintptr_t aligned = (raw + 1023u) & ~static_cast<uintptr_t>(1023u);
  *base = reinterpret_cast<unsigned char*>(aligned);
  *bytes = NOALLOC_ARRAY_BYTES - static_cast<size_t>(aligned - raw);
  return SKYRL_OK;
}

}  // namespace skyrl

extern "C" int skyrl_w8a8_lora_forward_noalloc_sm100_v1(const SkyrlW8A8LinearArgs* a, skyrl_stream_t stream_) {
  if (a == nullptr) return fail(SKYRL_ERR_INVALID_ARGUMENT, "noalloc linear: args is null");
  if (a->struct_size != sizeof(SkyrlW8A8LinearArgs))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "noalloc linear: struct_size %u does not match ABI v%d (%zu)",
                a->struct_size, SKYRL_W8A8_ABI_VERSION, sizeof(SkyrlW8A8LinearArgs));
  if (a->m <= 0 || a->n <= 0 || a->k <= 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "noalloc linear: non-positive shape");
  unsigned char* base = nullptr;
  size_t avail = 0;
  int rc = noalloc_scratch(&base, &avail);
  if (rc) return rc;
  const int na = a->num_adapters > 0 ? a->num_adapters : 1;
  const LinearWs w = carve_linear(base, a->m, a->n, a->k, na);
  if (w.bytes > avail)
    return fail(SKYRL_ERR_WORKSPACE,
                "noalloc linear: m=%d, n=%d, k=%d needs %zu bytes of scratch, the built-in array holds %zu "
                "(SKYRL_NOALLOC_SCRATCH_BYTES = %u); use skyrl_w8a8_lora_forward_sm100_v1 with a workspace",
                a->m, a->n, a->k, w.bytes, avail, SKYRL_NOALLOC_SCRATCH_BYTES);
  SkyrlW8A8LinearArgs b = *a;
  b.workspace = base;
  b.workspace_bytes = avail;
  return skyrl_w8a8_lora_forward_sm100_v1(&b, stream_);
}
