// Input gradient of the W8A8 LoRA linear in one GEMM launch:
//
//   dx[m, k] = bf16( f32(q1 . wq[k]) * s1[m] + f32(q2 . wq[k]) * s2[m]  +  zb[m, :] . A[a(m)][k, :] )
//
// q1, q2 are the two int8 planes of the scaled cotangent (grad_quant_kernel), wq the transposed packed weight, zb the
// cotangent's LoRA projection.  Both planes multiply the SAME weight tile, so a K stage holds two activation tiles and
// one weight tile and feeds two accumulators; the planes never meet in memory (two GEMM launches into fp32 slabs and a
// kernel that added and cast them moved 16 bytes per element of dx and took 445 us at 4096 x 4096 -> 12288, a fifth of
// it in the addition).  The sixteen epilogue warps read both accumulators into registers as one fp32 value per element;
// from then on the second accumulator's columns are free and take the LoRA term's MMAs, which are added on the way out.
//
// Bound by the tensor cores (two int8 MMAs per weight tile, the rate of one bf16 GEMM) plus the part of the epilogue
// that nothing hides: the accumulators of a 128 x 256 tile fill tensor memory.
#include "common.cuh"
#include "gemm_parts.cuh"
#include "ptx_sm100.cuh"
#include "tiles.cuh"

namespace skyrl {

constexpr int PL_EPI_WARPS = 16;
constexpr int PL_THREADS = (PL_EPI_WARPS + 2) * 32;  // + TMA producer, MMA issuer
constexpr int PL_AREA_BYTES = 216 * 1024;

template <int BN>
struct PlanesCfg {
  static constexpr int STAGE_BYTES = 2 * BM * BK + BN * BK;
  static constexpr int STAGES = PL_AREA_BYTES / STAGE_BYTES < 6 ? PL_AREA_BYTES / STAGE_BYTES : 6;
  static constexpr int BAR_OFF = STAGES * STAGE_BYTES;
  static constexpr int SMEM_BYTES = BAR_OFF + (2 * STAGES + 4) * 8 + 16 + 1024;
  static constexpr int TMEM_COLS = 2 * BN;
};

struct PlanesParams {
  CUtensorMap tm_xq;  // int8 [2 M, K]: plane 1, then plane 2; box 128 x 128
  CUtensorMap tm_w;
  CUtensorMap tm_z;
  CUtensorMap tm_b;
  TileSource src;
  LoraGeom lora;
  int rank_blocks;    // 0: no LoRA term
  const float* s;     // [2, m]
  const int32_t* out_row_map;
  __nv_bfloat16* out;
  int64_t out_stride;
  int32_t* status;
  int m, n, k;
};

template <int BN>
__global__ void __launch_bounds__(PL_THREADS, 1) w8a8_planes_gemm_kernel(const __grid_constant__ PlanesParams p) {
  using Cfg = PlanesCfg<BN>;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* tmem_full = empty_bar + Cfg::STAGES;
  uint64_t* tmem_empty = tmem_full + 1;   // both accumulators read
  uint64_t* acc2_free = tmem_empty + 1;   // the planes are in registers: the second accumulator takes the LoRA term
  uint64_t* lora_done = acc2_free + 1;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(lora_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(tmem_empty, PL_EPI_WARPS);
    mbar_init(acc2_free, PL_EPI_WARPS);
    mbar_init(lora_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == PL_EPI_WARPS + 1) {
    tmem_alloc(tmem_ptr_smem, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_wait();
  pdl_trigger();

  const int tm = tile_count(p.src);
  const int tn = (p.n + BN - 1) / BN;
  const int total = tm * tn;
  const int kblocks = (p.k + BK - 1) / BK;
  const bool lora = p.rank_blocks > 0;

  if (warp == PL_EPI_WARPS) {
    if (lane == 0) {
      tma_prefetch_desc(&p.tm_xq);
      tma_prefetch_desc(&p.tm_w);
      Pipe q = {smem, full_bar, empty_bar, Cfg::STAGES, Cfg::STAGE_BYTES, 0, 0u};
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const int4 tile = tile_at(p.src, t % tm);
        const int n0 = t / tm * BN;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = mbar_wait(&empty_bar[q.stage], q.phase ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER);
          if (!ok) break;
          unsigned char* sa = q.at();
          mbar_expect_tx(&full_bar[q.stage], Cfg::STAGE_BYTES);
          tma_load_2d(sa, &p.tm_xq, kb * BK, tile.x, &full_bar[q.stage]);
          tma_load_2d(sa + BM * BK, &p.tm_xq, kb * BK, tile.x + p.m, &full_bar[q.stage]);
          tma_load_3d(sa + 2 * BM * BK, &p.tm_w, 0, n0, kb, &full_bar[q.stage]);
          q.next();
        }
        if (ok && lora) ok = lora_load(p, q, tile, n0, abort_flag);
      }
    }
  } else if (warp == PL_EPI_WARPS + 1) {
    const uint32_t idesc = make_idesc(IDESC_D_S32, IDESC_S8, IDESC_S8, BM, BN);
    const uint32_t idesc_lora = make_idesc(IDESC_D_F32, IDESC_BF16, IDESC_BF16, BM, BN);
    const uint32_t smem_base = smem_u32(smem);
    Pipe q = {smem, full_bar, empty_bar, Cfg::STAGES, Cfg::STAGE_BYTES, 0, 0u};
    bool ok = true;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x, ++it) {
      ok = mbar_wait_warp(tmem_empty, (it & 1u) ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_MMA);
      if (!ok) break;
      tc_fence_after_sync();
      for (int kb = 0; kb < kblocks; ++kb) {
        ok = mbar_wait_warp(&full_bar[q.stage], q.phase, abort_flag, p.status, STATUS_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sa = smem_base + q.stage * Cfg::STAGE_BYTES;
        if (elect_one()) {
          const uint64_t a1 = make_desc_sw128(sa), a2 = make_desc_sw128(sa + BM * BK);
          const uint64_t b = make_desc_sw128(sa + 2 * BM * BK);
#pragma unroll
          for (int j = 0; j < BK / UMMA_K_I8; ++j) {
            const uint32_t accumulate = (kb != 0 || j != 0) ? 1u : 0u;
            mma_i8(tmem_base, a1 + 2 * j, b + 2 * j, idesc, accumulate);
            mma_i8(tmem_base + BN, a2 + 2 * j, b + 2 * j, idesc, accumulate);
          }
          mma_commit(&empty_bar[q.stage]);
        }
        __syncwarp();
        q.next();
      }
      if (!ok) break;
      if (elect_one()) mma_commit(tmem_full);
      __syncwarp();
      if (lora) {
        ok = lora_issue<true>(p, q, tile_at(p.src, t % tm), tmem_base + BN, idesc_lora, abort_flag, [&]() {
          return mbar_wait_warp(acc2_free, it & 1u, abort_flag, p.status, STATUS_TIMEOUT_LORA);
        });
        if (ok && elect_one()) mma_commit(lora_done);
        __syncwarp();
      }
    }
  } else {
    constexpr int COLS = BN / 4;  // four warps share a tensor-memory lane quadrant
    const int quad = warp & 3;
    const int col0 = (warp >> 2) * COLS;
    const int r = quad * 32 + lane;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + col0;
    bool ok = true;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x, ++it) {
      const int4 tile = tile_at(p.src, t % tm);
      const int n0 = t / tm * BN + col0;
      const bool row_valid = r < tile.y;
      const int srow = tile.x + (row_valid ? r : 0);
      const float s1 = __ldcg(p.s + srow), s2 = __ldcg(p.s + p.m + srow);
      const int64_t orow = p.out_row_map != nullptr ? __ldg(p.out_row_map + srow) : srow;
      ok = mbar_wait_warp(tmem_full, it & 1u, abort_flag, p.status, STATUS_TIMEOUT_EPILOGUE);
      if (!ok) break;
      tc_fence_after_sync();
      float f[COLS];
#pragma unroll
      for (int c = 0; c < COLS / 16; ++c) {
        uint32_t u[16], v[16];
        tmem_ld16(lanes + c * 16, u);
        tmem_ld16(lanes + BN + c * 16, v);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          f[c * 16 + i] = __fadd_rn(__fmul_rn(__int2float_rn(static_cast<int>(u[i])), s1),
                                    __fmul_rn(__int2float_rn(static_cast<int>(v[i])), s2));
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lora) {
        if (lane == 0) mbar_arrive(acc2_free);
        ok = mbar_wait_warp(lora_done, it & 1u, abort_flag, p.status, STATUS_TIMEOUT_LORA);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < COLS / 16; ++c) {
          uint32_t v[16];
          tmem_ld16(lanes + BN + c * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) f[c * 16 + i] = __fadd_rn(f[c * 16 + i], __uint_as_float(v[i]));
        }
        tc_fence_before_sync();
        __syncwarp();
      }
      if (lane == 0) mbar_arrive(tmem_empty);
      if (row_valid) {
        uint4* dst = reinterpret_cast<uint4*>(p.out + orow * p.out_stride + n0);
#pragma unroll
        for (int i = 0; i < COLS / 8; ++i) {
          if (n0 + i * 8 >= p.n) break;
          dst[i] = make_uint4(pack_bf16x2(f[8 * i], f[8 * i + 1]), pack_bf16x2(f[8 * i + 2], f[8 * i + 3]),
                              pack_bf16x2(f[8 * i + 4], f[8 * i + 5]), pack_bf16x2(f[8 * i + 6], f[8 * i + 7]));
        }
      }
    }
  }

  __syncwarp();
  if (*abort_flag) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == PL_EPI_WARPS + 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

template <int BN>
static int launch_planes_bn(const PlanesParams& p, int grid, cudaStream_t stream) {
  static bool attr_set[MAX_DEVICES] = {};
  auto kernel = w8a8_planes_gemm_kernel<BN>;
  cudaError_t e = ensure_dynamic_smem(kernel, PlanesCfg<BN>::SMEM_BYTES, attr_set);
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "planes gemm attribute: %s", cudaGetErrorString(e));
  e = launch_kernel(kernel, dim3(grid), dim3(PL_THREADS), PlanesCfg<BN>::SMEM_BYTES, stream, true, p);
  if (e == cudaSuccess) e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "planes gemm launch: %s", cudaGetErrorString(e));
  return SKYRL_OK;
}

int launch_planes_gemm(const PlanesGemmLaunch& a, cudaStream_t stream) {
  if (a.m <= 0 || a.n <= 0 || a.k <= 0 || a.n % 16 != 0 || a.k % 16 != 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "planes gemm: bad shape");
  if (!aligned16(a.q) || !aligned16(a.wq) || !aligned16(a.out) || a.out_stride < a.n || a.out_stride % 8 != 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "planes gemm: misaligned buffer or bad stride");
  const int sms = sm_count();
  if (sms <= 0) return fail(SKYRL_ERR_LAUNCH, "planes gemm: no CUDA device");
  // the widest column tile that still occupies most SMs (every narrower one reads the activation tiles again)
  const int tm = a.src.count;
  int bn = 256;
  while (bn > 64 && tm * ((a.n + bn - 1) / bn) * 4 < 3 * sms) bn >>= 1;
  PlanesParams p = {};
  int rc;
  if ((rc = encode_tmap_2d(&p.tm_xq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.q, a.k, 2 * static_cast<uint64_t>(a.m), a.k, BK, BM)))
    return rc;
  if ((rc = encode_tmap_3d(&p.tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.wq, BK, a.n, (a.k + BK - 1) / BK, BK,
                           static_cast<uint64_t>(a.n) * BK, BK, bn)))
    return rc;
  p.tm_z = p.tm_xq;
  p.tm_b = p.tm_xq;
  if (a.rank > 0) {
    if (a.z_parts == nullptr || a.b_table == nullptr || !aligned16(a.b_table) || a.b_slots < a.rank || a.b_slots % 8 != 0)
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "planes gemm: LoRA operands missing or misaligned");
    const uint32_t half = (a.rank <= 16 ? 32 : (a.rank <= 32 ? 64 : 128)) / 2;
    if ((rc = encode_tmap_3d(&p.tm_z, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.z_parts, SKYRL_LORA_RANK_PAD, SKYRL_Z_PARTS, a.m,
                             SKYRL_LORA_RANK_PAD * 2, SKYRL_Z_PARTS * SKYRL_LORA_RANK_PAD * 2, half, 1, BM)))
      return rc;
    if ((rc = encode_tmap_3d(&p.tm_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.b_table, a.b_slots, a.n, a.num_adapters,
                             static_cast<uint64_t>(a.b_slots) * 2, static_cast<uint64_t>(a.n) * a.b_slots * 2, half, bn)))
      return rc;
    const int stage = 2 * BM * BK + bn * BK;
    p.lora = lora_geom(a.rank, bn, stage, PL_AREA_BYTES / stage < 6 ? PL_AREA_BYTES / stage : 6);
  }
  p.src = a.src;
  p.rank_blocks = (a.rank + 15) / 16;
  p.s = a.s;
  p.out_row_map = a.out_row_map;
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.out_stride = a.out_stride;
  p.status = a.status;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  const int64_t total = static_cast<int64_t>(tm) * ((a.n + bn - 1) / bn);
  const int grid = static_cast<int>(total < sms ? total : sms);
  if (bn == 256) return launch_planes_bn<256>(p, grid, stream);
  if (bn == 128) return launch_planes_bn<128>(p, grid, stream);
  return launch_planes_bn<64>(p, grid, stream);
}

}  // namespace skyrl
