// LoRA-A projection on the tensor cores: for every 128-row tile of the
// adapter-sorted row space, z = s[a] * (x_tile @ A[a]) with a bf16 tcgen05 MMA
// (fp32 accumulator in TMEM, products of bf16 inputs are exact), written out as
// three bf16 parts (hi, mid, lo) that sum to the fp32 value exactly, so that the
// rank-r contraction of the GEMM epilogue sees z at full fp32 precision.  The parts of a row sit side by
// side, z_parts[row][part][64], so that a range of rows is one contiguous block (a rank of a
// tensor-parallel group computes a range and gathers the rest).  A row window [row_lo, row_hi) limits the rows
// written: tiles outside it are skipped, tiles that straddle its edge compute all their rows (rows of an MMA are
// independent, so whatever the unowned rows of x hold cannot reach an owned row) and store the owned ones.
//
// Bound by HBM at large batches (x streamed once through a TMA pipeline) and, at small ones, by the length of the K
// loop: one CTA pulls a 128-row tile at well under 100 GB/s, so seven tiles of K = 12288 took 63 us on seven SMs.
// The K range of a tile is therefore cut into up to eight slices (a function of K alone), which a cluster of up to
// eight CTAs shares whenever that many CTAs fit the GPU.  Every slice has tensor-memory columns of its own; the
// slices are added in order, through distributed shared memory where the cluster has several CTAs, so that a row's
// z depends neither on the batch around it nor on the cluster size (a row pushed through alone, or a chunk of a
// block, gives the bits of the whole launch).
//
// A tile of several adapters takes their tables side by side: one MMA of width adapters * rank per K step computes
// every row against every adapter of the group and the epilogue picks the row's own columns; groups beyond 128 table
// rows make another pass over the tile with the other rows' lanes disabled, on a cluster of its own (blockIdx.y) where
// the GPU has room for it.  The whole warp walks the issuing loop and elects a thread for the instruction alone: operands computed by one divergent thread cost the issue 144 cycles
// per MMA instead of 47.
//
// Reference arithmetic: `x.astype(f32) @ lora_a.astype(f32)`
// (skyrl/tx/kernels/quantized_lora.py:301) and the first ragged_dot of
// skyrl/tx/layers/lora.py:150; the per-adapter scaling of lora.py:155-156 is
// folded in here.
#include "common.cuh"
#include "ptx_sm100.cuh"
#include "tiles.cuh"

namespace skyrl {

constexpr int PROJ_BM = 128;
constexpr int PROJ_BK = 128;  // K values per stage: two swizzled 128-byte column blocks of x
constexpr int PROJ_HALF = 64;
constexpr int PROJ_TABLE_ROWS = 128;  // rank rows of LoRA-A per pass: 128 / rank16 adapters side by side
constexpr int PROJ_MAX_STAGES = 6;
constexpr int PROJ_X_BYTES = 2 * PROJ_BM * 128;
constexpr int PROJ_AREA_BYTES = 208 * 1024;
constexpr int PROJ_BAR_OFF = PROJ_AREA_BYTES;
constexpr int PROJ_SCALE_OFF = PROJ_BAR_OFF + 256;  // per row: scaling of its adapter, z slot (cluster form)
constexpr int PROJ_SMEM_BYTES = PROJ_SCALE_OFF + PROJ_BM * 8 + 1024;
constexpr int PROJ_THREADS = 192;
constexpr int PROJ_TMEM_COLS = 512;  // shared by the K slices of the CTA
constexpr int PROJ_Z_COLS = SKYRL_LORA_RANK_PAD;
constexpr int PROJ_Z_ROW = SKYRL_Z_PARTS * PROJ_Z_COLS;  // bf16 elements of one row of z_parts
constexpr int PROJ_MAX_SLICES = 8;

struct ProjParams {
  CUtensorMap tm_x;  // bf16 [M, K], box 64 x 128
  CUtensorMap tm_a;  // bf16 [A, 64, K], box 64 x rank16 x 1
  const float* scaling;
  TileSource src;
  __nv_bfloat16* z_parts[8];  // [m, 6, 64]: adapter slot 0 parts (hi, mid, lo), adapter slot 1 parts; the same rows
  int z_count;                // are written to every one of the z_count destinations (a tensor-parallel rank hands
                              // its rows to every peer's workspace with plain stores; one destination otherwise)
  int row_lo, row_hi;      // rows written
  int tile_base;           // cluster b looks at tile tile_base + b (a row window needs only the tiles that can overlap it)
  int32_t* status;
  int k;
  int slices;              // K slices of a tile, a power of two and a multiple of the cluster size
  int rank16;              // rank rounded up to 16: table rows per adapter, columns per adapter of the MMA
};

// N consecutive columns of one row of z: three bf16 parts that sum to the fp32 values exactly
template <int N>
__device__ __forceinline__ void proj_store(const ProjParams& p, int64_t row, int slot, int col, const float (&z)[N]) {
  uint32_t part[3][N / 2];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float h0 = round_bf16(z[2 * i]), h1 = round_bf16(z[2 * i + 1]);
    const float r0 = __fsub_rn(z[2 * i], h0), r1 = __fsub_rn(z[2 * i + 1], h1);  // exact
    const float m0 = round_bf16(r0), m1 = round_bf16(r1);
    part[0][i] = pack_bf16x2(h0, h1);
    part[1][i] = pack_bf16x2(m0, m1);
    part[2][i] = pack_bf16x2(__fsub_rn(r0, m0), __fsub_rn(r1, m1));  // <= 8 bits left: exact in bf16
  }
  const int64_t off = row * PROJ_Z_ROW + slot * 3 * PROJ_Z_COLS + col;
  for (int d = 0; d < p.z_count; ++d) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      __nv_bfloat16* dst = p.z_parts[d] + off + q * PROJ_Z_COLS;
      if (N >= 8) {
#pragma unroll
        for (int g = 0; g < N / 8; ++g)
          reinterpret_cast<uint4*>(dst)[g] =
              make_uint4(part[q][4 * g], part[q][4 * g + 1], part[q][4 * g + 2], part[q][4 * g + 3]);
      } else {
        *reinterpret_cast<uint2*>(dst) = make_uint2(part[q][0], part[q][1]);
      }
    }
  }
}

__global__ void __launch_bounds__(PROJ_THREADS, 1) lora_a_proj_kernel(const __grid_constant__ ProjParams p) {
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + PROJ_BAR_OFF);
  uint64_t* empty_bar = full_bar + PROJ_MAX_STAGES;
  uint64_t* acc_full = empty_bar + PROJ_MAX_STAGES;
  uint64_t* acc_free = acc_full + 1;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(acc_free + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  float* row_scale = reinterpret_cast<float*>(smem + PROJ_SCALE_OFF);
  int* row_slot = reinterpret_cast<int*>(row_scale + PROJ_BM);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int csize = static_cast<int>(cluster_size());
  const int crank = csize > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  pdl_wait();
  pdl_trigger();
  const int tile_index = static_cast<int>(blockIdx.x) / csize + p.tile_base;
  if (tile_index >= tile_count(p.src)) return;  // uniform for the cluster
  const int4 tile = tile_at(p.src, tile_index);
  if (tile.x >= p.row_hi || tile.x + tile.y <= p.row_lo) return;  // outside the row window, also uniform
  const int nseg = tile_segments(tile);
  const int group = min(nseg, PROJ_TABLE_ROWS / p.rank16);  // adapters per pass, at most eight
  const int seg_begin = static_cast<int>(blockIdx.y) * group, seg_step = static_cast<int>(gridDim.y) * group;
  if (seg_begin >= nseg) return;  // fewer adapters in this tile than the launch provided for, also uniform

  if (threadIdx.x == 0) {
    for (int s = 0; s < PROJ_MAX_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, PROJ_BM);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_ptr_smem, PROJ_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;

  const int kblocks = (p.k + PROJ_BK - 1) / PROJ_BK;
  const int own = p.slices / csize, slice0 = crank * own;  // this CTA's K slices; slices <= kblocks, so none is empty
  int slice_cols = 16;                                      // tensor-memory columns of a slice
  while (slice_cols < group * p.rank16) slice_cols <<= 1;
  const int per_phase = min(own, PROJ_TMEM_COLS / slice_cols);  // slices accumulated before the epilogue drains them
  const int phases = (own + per_phase - 1) / per_phase;         // 1 whenever the cluster has several CTAs
  const int table_bytes = p.rank16 * 128;
  const int stage_bytes = PROJ_X_BYTES + 2 * group * table_bytes;
  const int stages = min(PROJ_MAX_STAGES, PROJ_AREA_BYTES / stage_bytes);

  if (warp == 4) {
    if (lane == 0) {
      tma_prefetch_desc(&p.tm_x);
      tma_prefetch_desc(&p.tm_a);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int ph = 0; ph < phases && ok; ++ph) {
        const int kb0 = kblocks * (slice0 + ph * per_phase) / p.slices;
        const int kb1 = kblocks * (slice0 + min(own, (ph + 1) * per_phase)) / p.slices;
        for (int j0 = seg_begin; j0 < nseg && ok; j0 += seg_step) {
          const int cnt = min(group, nseg - j0);
          int adapter[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) adapter[j] = j < cnt ? segment_adapter(p.src, tile, j0 + j) : 0;
          for (int kb = kb0; kb < kb1; ++kb) {
            ok = mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER);
            if (!ok) break;
            unsigned char* sa = smem + stage * stage_bytes;
            mbar_expect_tx(&full_bar[stage], PROJ_X_BYTES + 2 * cnt * table_bytes);
            tma_load_2d(sa, &p.tm_x, kb * PROJ_BK, tile.x, &full_bar[stage]);
            tma_load_2d(sa + PROJ_X_BYTES / 2, &p.tm_x, kb * PROJ_BK + PROJ_HALF, tile.x, &full_bar[stage]);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (j >= cnt) break;
              tma_load_3d(sa + PROJ_X_BYTES + j * table_bytes, &p.tm_a, kb * PROJ_BK, 0, adapter[j], &full_bar[stage]);
              tma_load_3d(sa + PROJ_X_BYTES + (group + j) * table_bytes, &p.tm_a, kb * PROJ_BK + PROJ_HALF, 0, adapter[j],
                          &full_bar[stage]);
            }
            if (++stage == stages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
    }
  } else if (warp == 5) {
    const uint32_t smem_base = smem_u32(smem);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int ph = 0; ph < phases && ok; ++ph) {
      if (ph > 0) {
        ok = mbar_wait_warp(acc_free, (ph - 1) & 1u, abort_flag, p.status, STATUS_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after_sync();
      }
      const int sl0 = ph * per_phase, sl1 = min(own, sl0 + per_phase);
      for (int j0 = seg_begin; j0 < nseg && ok; j0 += seg_step) {
        const int cnt = min(group, nseg - j0);
        const uint32_t idesc = make_idesc(IDESC_D_F32, IDESC_BF16, IDESC_BF16, PROJ_BM, cnt * p.rank16);
        int4 off = make_int4(0, 0, 0, 0);
        if (nseg > group) {  // the lanes of the other passes keep what they hold
          for (int j = 0; j < cnt; ++j) {
            const int4 mk = segment_mask(p.src, tile, j0 + j);
            off.x |= mk.x; off.y |= mk.y; off.z |= mk.z; off.w |= mk.w;
          }
          off = make_int4(~off.x, ~off.y, ~off.z, ~off.w);
        }
        for (int sl = sl0; sl < sl1 && ok; ++sl) {
          const int kb0 = kblocks * (slice0 + sl) / p.slices, kb1 = kblocks * (slice0 + sl + 1) / p.slices;
          const uint32_t d = tmem_base + (sl - sl0) * slice_cols;
          for (int kb = kb0; kb < kb1; ++kb) {
            ok = mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.status, STATUS_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t sa = smem_base + stage * stage_bytes;
            if (elect_one()) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint64_t adesc = make_desc_sw128(sa + h * (PROJ_X_BYTES / 2));
                const uint64_t bdesc = make_desc_sw128(sa + PROJ_X_BYTES + h * group * table_bytes);
#pragma unroll
                for (int j = 0; j < PROJ_HALF / 16; ++j) {
                  const uint32_t accumulate = (kb > kb0 || h > 0 || j > 0) ? 1u : 0u;
                  if (nseg > group) mma_bf16_lanes(d, adesc + 2 * j, bdesc + 2 * j, idesc, accumulate, off);
                  else mma_bf16(d, adesc + 2 * j, bdesc + 2 * j, idesc, accumulate);
                }
              }
              mma_commit(&empty_bar[stage]);
            }
            __syncwarp();
            if (++stage == stages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (ok && elect_one()) mma_commit(acc_full);
      __syncwarp();
    }
  } else {
    const int r = warp * 32 + lane;
    // this row's segment: which columns of its pass, which adapter, which z slot
    int seg = 0;
#pragma unroll 8
    for (int j = 0; j < nseg; ++j) {
      const int4 mk = segment_mask(p.src, tile, j);
      const int word = warp == 0 ? mk.x : (warp == 1 ? mk.y : (warp == 2 ? mk.z : mk.w));
      if ((word >> lane) & 1) seg = j;
    }
    const int64_t row = tile.x + r;
    const bool row_valid = r < tile.y && row >= p.row_lo && row < p.row_hi &&
                           (seg / group) % static_cast<int>(gridDim.y) == static_cast<int>(blockIdx.y);
    const bool dense = tile_is_dense(tile);
    const int slot = segment_slot(tile, seg);
    const float s = __ldg(p.scaling + segment_adapter(p.src, tile, seg));
    row_scale[r] = s;
    row_slot[r] = row_valid ? slot : -1;
    const int col = seg % group;
    float* part = reinterpret_cast<float*>(smem);  // cluster form: [own][128][rank16 + 4] in the drained stages
    const int part_floats = PROJ_BM * (p.rank16 + 4);
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    float z[4][16];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc)
#pragma unroll
      for (int i = 0; i < 16; ++i) z[cc][i] = 0.f;
    bool ok = true;
    for (int ph = 0; ph < phases; ++ph) {
      ok = __all_sync(0xffffffffu, mbar_wait(acc_full, ph & 1u, abort_flag, p.status, STATUS_TIMEOUT_EPILOGUE));
      if (!ok) break;
      tc_fence_after_sync();
      const int cnt = min(own - ph * per_phase, per_phase);
      for (int sl = 0; sl < cnt; ++sl) {
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          if (cc * 16 >= p.rank16) break;
          float t[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) t[i] = 0.f;
          for (int g = 0; g < group; ++g) {
            if (!__any_sync(0xffffffffu, col == g)) continue;
            uint32_t v[16];
            tmem_ld16(lanes + sl * slice_cols + g * p.rank16 + cc * 16, v);
            tmem_wait_ld();
            if (col == g) {
#pragma unroll
              for (int i = 0; i < 16; ++i) t[i] = __uint_as_float(v[i]);
            }
          }
          if (csize > 1) {
            float4* dst = reinterpret_cast<float4*>(part + sl * part_floats + r * (p.rank16 + 4) + cc * 16);
#pragma unroll
            for (int g = 0; g < 4; ++g) dst[g] = make_float4(t[4 * g], t[4 * g + 1], t[4 * g + 2], t[4 * g + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) z[cc][i] = __fadd_rn(z[cc][i], t[i]);
          }
        }
      }
      tc_fence_before_sync();
      mbar_arrive(acc_free);
    }
    if (ok && csize == 1 && row_valid) {
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        if (cc * 16 >= p.rank16 && dense) break;  // nothing reads the columns past the rank
#pragma unroll
        for (int i = 0; i < 16; ++i) z[cc][i] = __fmul_rn(z[cc][i], s);
        proj_store<16>(p, row, slot, cc * 16, z[cc]);
      }
    }
    if (ok && !dense && nseg == 2 && row_valid && crank == 0) {  // two-slot lists: the slot that is not the row's is zero
      const float zero[16] = {};
      for (int cc = 0; cc < PROJ_Z_COLS / 16; ++cc) proj_store<16>(p, row, 1 - slot, cc * 16, zero);
    }
  }

  if (csize > 1) {
    __syncwarp();
    cluster_sync_all();  // every CTA's partial sums are in its shared memory
    if (warp < 4) {
      const int rows_per = PROJ_BM / csize, quads = p.rank16 / 4, pitch = p.rank16 + 4;
      const int all_quads = tile_is_dense(tile) ? quads : PROJ_Z_COLS / 4;
      for (int item = threadIdx.x; item < rows_per * all_quads; item += 128) {
        const int r = crank * rows_per + item / all_quads, q = item % all_quads;
        if (row_slot[r] < 0) continue;
        float z[4] = {0.f, 0.f, 0.f, 0.f};
        if (q < quads) {
          const uint32_t local = smem_u32(smem) + static_cast<uint32_t>((r * pitch + 4 * q) * 4);
          for (int c = 0; c < csize; ++c) {
            for (int sl = 0; sl < own; ++sl) {
              const float4 v = ld_cluster_float4(map_to_cta(local + sl * PROJ_BM * pitch * 4, c));
              z[0] = __fadd_rn(z[0], v.x);
              z[1] = __fadd_rn(z[1], v.y);
              z[2] = __fadd_rn(z[2], v.z);
              z[3] = __fadd_rn(z[3], v.w);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) z[i] = __fmul_rn(z[i], row_scale[r]);
        proj_store<4>(p, tile.x + r, row_slot[r], 4 * q, z);
      }
    }
    __syncwarp();
    cluster_sync_all();  // no CTA leaves while another reads its shared memory
  }
  if (p.z_count > 1) __threadfence_system();  // stores into other GPUs' memory are performed before the kernel ends

  __syncwarp();
  if (*abort_flag) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, PROJ_TMEM_COLS);
  }
}

// K slices of a tile (a function of K alone: it fixes the order of summation) and CTAs per tile: as many as fit the
// GPU beside the other tiles, each slice with at least two K blocks to hide its pipeline fill behind.
static int proj_slices(int k) {
  const int kblocks = (k + PROJ_BK - 1) / PROJ_BK;
  int s = PROJ_MAX_SLICES;
  while (s > 1 && kblocks < 2 * s) s >>= 1;
  return s;
}
static int proj_cluster(int m, int slices) {
  int sms = sm_count();
  if (sms <= 0) sms = 148;
  const int tiles = (m + PROJ_BM - 1) / PROJ_BM;
  int c = slices;
  while (c > 1 && tiles * c > sms) c >>= 1;
  return c;
}

int launch_lora_a_proj(const void* x, int m, int k, const void* a_packed, const float* scaling, int num_adapters,
                       int rank, const TileSource& src, int max_tiles, void* z_parts, int32_t* status,
                       cudaStream_t stream, int row_lo, int row_hi, void* const* extra_dests, int extra_count,
                       int list_row0, int table_rows, int table_k) {
  if (x == nullptr || a_packed == nullptr || scaling == nullptr || z_parts == nullptr || status == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: null buffer");
  if (m <= 0 || k <= 0 || num_adapters <= 0 || max_tiles <= 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: non-positive shape");
  if (k % 8 != 0) return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: K must be a multiple of 8, got %d", k);
  if (rank <= 0 || rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_UNSUPPORTED, "lora_a_proj: rank must be in [1, %d], got %d", SKYRL_LORA_RANK_PAD, rank);
  if (!aligned16(x) || !aligned16(a_packed) || !aligned16(z_parts) || !aligned16(src.tiles))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: buffers must be 16-byte aligned");
  if (x == z_parts) return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: aliased buffers");
  ProjParams p;
  p.rank16 = (rank + 15) / 16 * 16;
  int rc;
  if ((rc = encode_tmap_2d(&p.tm_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, k, m, static_cast<uint64_t>(k) * 2,
                           PROJ_HALF, PROJ_BM)))
    return rc;
  // table rows past the last, and columns past K where x is padded, read as zeros
  if (table_k <= 0) table_k = k;
  if (table_rows < rank || table_k % 8 != 0 || table_k > k)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: table of %d rows and %d columns", table_rows, table_k);
  if ((rc = encode_tmap_3d(&p.tm_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a_packed, table_k, table_rows, num_adapters,
                           static_cast<uint64_t>(table_k) * 2, static_cast<uint64_t>(table_k) * 2 * table_rows, PROJ_HALF,
                           p.rank16)))
    return rc;
  p.scaling = scaling;
  p.src = src;
  if (extra_count < 0 || extra_count > 7 || (extra_count > 0 && extra_dests == nullptr))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: at most 7 extra destinations");
  p.z_parts[0] = static_cast<__nv_bfloat16*>(z_parts);
  p.z_count = 1;
  for (int d = 0; d < extra_count; ++d) {
    if (extra_dests[d] == nullptr || !aligned16(extra_dests[d]))
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: extra destination %d is null or not 16-byte aligned", d);
    p.z_parts[p.z_count++] = static_cast<__nv_bfloat16*>(extra_dests[d]);
  }
  p.row_lo = row_lo;
  p.row_hi = row_hi < 0 ? m : row_hi;
  p.status = status;
  p.k = k;
  static bool attr_set[MAX_DEVICES] = {};
  cudaError_t e = ensure_dynamic_smem(lora_a_proj_kernel, PROJ_SMEM_BYTES, attr_set);
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "lora_a_proj attribute: %s", cudaGetErrorString(e));
  // The list starts at sorted row list_row0 (a whole block, or one row chunk of it) and its tiles are 128 rows each,
  // so a row window launches exactly the tiles it meets.  (Every CTA asks for most of an SM's shared memory: CTAs that
  // would only find out that they have nothing to do still queue for an SM beside a running GEMM.)
  int grid = src.num_tiles == nullptr ? src.count : max_tiles;
  p.tile_base = 0;
  if (src.num_tiles == nullptr && (p.row_lo > list_row0 || p.row_hi < m) && list_row0 >= 0 && p.row_lo >= list_row0 &&
      p.row_hi > p.row_lo) {
    p.tile_base = (p.row_lo - list_row0) / PROJ_BM;
    const int last = (p.row_hi - 1 - list_row0) / PROJ_BM;
    grid = (last < src.count - 1 ? last : src.count - 1) - p.tile_base + 1;
  }
  if (grid <= 0) return SKYRL_OK;
  p.slices = proj_slices(k);
  const int cluster = proj_cluster(m, p.slices);
  // A tile of more adapters than one pass takes: its passes on clusters of their own where the GPU has room for them (two
  // tiles of 32 adapters of rank 16 left 132 SMs idle and took three passes in a row: 36 us at K = 12288).
  int passes = 1;
  if (src.tiles != nullptr && src.num_tiles == nullptr) {
    const int most = num_adapters < PROJ_BM ? num_adapters : PROJ_BM, per_pass = PROJ_TABLE_ROWS / p.rank16;
    const int want = (most + per_pass - 1) / per_pass, room = sm_count() / (grid * cluster);
    passes = want < room ? want : (room > 1 ? room : 1);
  }
  e = launch_cluster_kernel(lora_a_proj_kernel, dim3(grid * cluster, passes), dim3(PROJ_THREADS), PROJ_SMEM_BYTES, stream, cluster, p);
  if (e == cudaSuccess) e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "lora_a_proj launch: %s", cudaGetErrorString(e));
  return SKYRL_OK;
}

}  // namespace skyrl

extern "C" int skyrl_lora_a_proj_sm100_v1(const void* x, int32_t m, int32_t k, const void* lora_a_packed,
                                          const float* lora_scaling, int32_t num_adapters, int32_t rank,
                                          const int32_t* tiles, const int32_t* num_tiles, int32_t max_tiles,
                                          void* z_parts, int32_t* status, skyrl_stream_t stream) {
  if (tiles == nullptr || num_tiles == nullptr)
    return skyrl::fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_a_proj: null buffer");
  const skyrl::TileSource src = {reinterpret_cast<const int4*>(tiles), nullptr, nullptr, num_tiles, 0, 0, m};
  return skyrl::launch_lora_a_proj(x, m, k, lora_a_packed, lora_scaling, num_adapters, rank, src, max_tiles, z_parts,
                                   status, static_cast<cudaStream_t>(stream));
}
