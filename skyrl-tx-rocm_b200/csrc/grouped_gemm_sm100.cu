// W8A8 LoRA linear on the reference's own storage: one weight scale per `group` values of K and one activation scale
// per row and group (skyrl/tx/kernels/quantized_lora.py:20-41, 199-254; the Pallas prototype's group is 64).
//
//   y[m, n] = bf16( sum_g (f32(acc_g[m, n]) * sx[g, m]) * sw[g, n]  +  z[m, :] . B[a(m)][n, :] )
//
// with the groups added in ascending order, as the reference's sum over the group axis does.  The int32 accumulator of
// a group covers `group` values of K only (two tcgen05.mma for group 64), so the work beside the tensor cores is what
// bounds this kernel: every accumulator element of every group is read from tensor memory, converted, scaled twice and
// added in fp32.  That takes one conversion and, as packed pairs (fp32x2), one and a half instructions an element;
// group 64 of a 128 x 128 tile costs 128 tensor-core cycles and about 360 issue cycles of the eight epilogue warps.
// Three accumulator buffers keep the tensor cores ahead of them.  The scales of a group's columns travel through a ring
// of small bulk copies of their own.  The LoRA term has tensor-memory columns of its own (the accumulators never are
// the sum it could be added to) and is added once, before the single cast.
//
// (ncu: the tensor pipe is busy 10 % of the time, ten warps issue on 42 % of the cycles, in dependent chains.)
// Before, every group was a launch of its own into an fp32 slab: 262 launches and 3.16 ms for 512 x 4096 -> 4096 at
// group 64; now four launches and 66 us, 48 of them in the GEMM.
#include "common.cuh"
#include "gemm_parts.cuh"
#include "ptx_sm100.cuh"
#include "quant_row.cuh"
#include "tiles.cuh"

namespace skyrl {

// ---- row quantiser: a scale per row and group ------------------------------------------------------------
// POW2: the vectors of a group are a power of two of neighbouring lanes (groups of 8 ... 256 values): one pass,
// shuffles only.  Otherwise a warp takes a whole group and reads it twice.
template <bool POW2>
__global__ void __launch_bounds__(QUANT_THREADS)
group_quant_kernel(const __nv_bfloat16* x, int64_t x_row_stride, const int32_t* row_map, int m, int k, int group_vecs,
                   int8_t* __restrict__ xq, float* __restrict__ sx, __nv_bfloat16* __restrict__ xn) {
  pdl_wait();
  pdl_trigger();
  const int row = blockIdx.x, lane = threadIdx.x & 31;
  const int64_t src_row = row_map != nullptr ? __ldcg(row_map + row) : row;
  const uint4* src = reinterpret_cast<const uint4*>(x + src_row * x_row_stride);
  uint2* dst = reinterpret_cast<uint2*>(xq + static_cast<int64_t>(row) * k);
  uint4* copy = xn != nullptr ? reinterpret_cast<uint4*>(xn + static_cast<int64_t>(row) * k) : nullptr;
  const int nvec = k >> 3;
  auto absmax = [](const uint4& u) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float a = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) a = fmaxf(a, fmaxf(fabsf(bf16_lo(w[j])), fabsf(bf16_hi(w[j]))));
    return a;
  };
  auto codes = [](const uint4& u, float scale, float rcp) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    int q[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      q[2 * j] = quant_code(bf16_lo(w[j]), scale, rcp);
      q[2 * j + 1] = quant_code(bf16_hi(w[j]), scale, rcp);
    }
    return make_uint2(pack_codes4(q[0], q[1], q[2], q[3]), pack_codes4(q[4], q[5], q[6], q[7]));
  };
  if (POW2) {
    for (int v0 = threadIdx.x & ~31; v0 < nvec; v0 += QUANT_THREADS) {
      const int v = v0 + lane;
      const uint4 u = v < nvec ? ld_stream16(src + v) : make_uint4(0u, 0u, 0u, 0u);
      float a = absmax(u);
      for (int o = 1; o < group_vecs; o <<= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
      const float scale = a > 0.f ? __fdiv_rn(a, 127.0f) : 1.0f;
      if (v < nvec) {
        dst[v] = codes(u, scale, quant_rcp(scale));
        if (copy != nullptr) copy[v] = u;
        if ((v & (group_vecs - 1)) == 0) sx[static_cast<int64_t>(v / group_vecs) * m + row] = scale;
      }
    }
  } else {
    for (int g = threadIdx.x >> 5; g * group_vecs < nvec; g += QUANT_THREADS / 32) {
      float a = 0.f;
      for (int i = lane; i < group_vecs; i += 32) a = fmaxf(a, absmax(ld_stream16(src + g * group_vecs + i)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
      const float scale = a > 0.f ? __fdiv_rn(a, 127.0f) : 1.0f;
      for (int i = lane; i < group_vecs; i += 32) {
        const uint4 u = ld_stream16(src + g * group_vecs + i);
        dst[g * group_vecs + i] = codes(u, scale, quant_rcp(scale));
        if (copy != nullptr) copy[g * group_vecs + i] = u;
      }
      if (lane == 0) sx[static_cast<int64_t>(g) * m + row] = scale;
    }
  }
}

int launch_group_quant(const void* x, int64_t x_row_stride, const int32_t* row_map, int m, int k, int group, void* xq,
                       float* sx, void* xn, cudaStream_t stream) {
  if (x == nullptr || xq == nullptr || sx == nullptr || m <= 0 || k <= 0 || group <= 0 || group % 8 != 0 || k % group != 0 ||
      x_row_stride < k || x_row_stride % 8 != 0 || !aligned16(x) || !aligned16(xq) || (xn != nullptr && !aligned16(xn)))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "group_quant: null or misaligned buffer, or bad shape");
  const int gv = group / 8;
  const bool pow2 = gv <= 32 && (gv & (gv - 1)) == 0;
  cudaError_t e = launch_kernel(pow2 ? group_quant_kernel<true> : group_quant_kernel<false>, dim3(m), dim3(QUANT_THREADS), 0,
                                stream, true, static_cast<const __nv_bfloat16*>(x), x_row_stride, row_map, m, k, gv,
                                static_cast<int8_t*>(xq), sx, static_cast<__nv_bfloat16*>(xn));
  if (e == cudaSuccess) e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "group_quant launch: %s", cudaGetErrorString(e));
  return SKYRL_OK;
}

// ---- GEMM --------------------------------------------------------------------------------------------------
constexpr int GRP_THREADS = 320;  // warps 0-3 and 6-9 epilogue, warp 4 TMA producer, warp 5 MMA issuer
constexpr int GRP_EPI_WARPS = 8;
constexpr int GRP_BUFS = 3;       // accumulator buffers of one group each
constexpr int GRP_SW_SLOTS = 8;   // groups whose column scales may be in flight
constexpr int GRP_STAGES = 6;

template <int BN>
struct GrpCfg {
  static constexpr int STAGE_BYTES = BM * BK + BN * BK;
  static constexpr int SW_OFF = GRP_STAGES * STAGE_BYTES;
  static constexpr int BAR_OFF = SW_OFF + GRP_SW_SLOTS * BN * 4;
  static constexpr int NUM_BARS = 2 * GRP_STAGES + 2 * GRP_BUFS + 2 * GRP_SW_SLOTS + 2;
  static constexpr int SMEM_BYTES = BAR_OFF + NUM_BARS * 8 + 16 + 1024;
  static constexpr int TMEM_COLS = 4 * BN;  // three accumulators and the LoRA term
};

struct GrpParams {
  CUtensorMap tm_xq;  // int8 [M, K], box 128 x 128
  CUtensorMap tm_w;   // int8 [K / 128, N, 128], box 128 x BN x 1
  CUtensorMap tm_z;
  CUtensorMap tm_b;
  TileSource src;
  LoraGeom lora;
  int rank_blocks;    // 0: no LoRA term
  const float* sx;    // [groups, m]
  const float* sw;    // [groups, n]
  const int32_t* out_row_map;
  __nv_bfloat16* out;
  int64_t out_stride;
  int32_t* status;
  int m, n, k, group;
  float one;          // 1.0f, see add_f32x2
};

__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f32x2_parts(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a + b as a * one + b, the same value, with a `one` the assembler cannot see through: a packed multiplication in front
// of a packed addition comes out of it as one fused operation, and the reference rounds the product (left alone, one
// bf16 result in 10^4 moved by a step)
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b, uint64_t one) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(one), "l"(b));
  return r;
}
// 16-byte multiples of global memory to shared memory, completing on `bar`
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <int BN>
__global__ void __launch_bounds__(GRP_THREADS, 1) w8a8_grouped_gemm_kernel(const __grid_constant__ GrpParams p) {
  using Cfg = GrpCfg<BN>;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* empty_bar = full_bar + GRP_STAGES;
  uint64_t* acc_full = empty_bar + GRP_STAGES;
  uint64_t* acc_empty = acc_full + GRP_BUFS;
  uint64_t* sw_full = acc_empty + GRP_BUFS;
  uint64_t* sw_empty = sw_full + GRP_SW_SLOTS;
  uint64_t* lora_full = sw_empty + GRP_SW_SLOTS;
  uint64_t* lora_empty = lora_full + 1;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(lora_empty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  float* sw_ring = reinterpret_cast<float*>(smem + Cfg::SW_OFF);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GRP_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < GRP_BUFS; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], GRP_EPI_WARPS);
    }
    for (int s = 0; s < GRP_SW_SLOTS; ++s) {
      mbar_init(&sw_full[s], 1);
      mbar_init(&sw_empty[s], GRP_EPI_WARPS);
    }
    mbar_init(lora_full, 1);
    mbar_init(lora_empty, GRP_EPI_WARPS);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_ptr_smem, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  const uint32_t lora_cols = tmem_base + GRP_BUFS * BN;
  pdl_wait();
  pdl_trigger();

  const int tm = tile_count(p.src);
  const int tn = (p.n + BN - 1) / BN;
  const int total = tm * tn;
  const int kblocks = (p.k + BK - 1) / BK;
  const int steps = (p.k + UMMA_K_I8 - 1) / UMMA_K_I8;  // 32-wide MMAs along K; a group is a whole number of them
  const int per_group = p.group / UMMA_K_I8;
  const int groups = p.k / p.group;
  const bool lora = p.rank_blocks > 0;

  if (warp == 4) {
    if (lane == 0) {
      tma_prefetch_desc(&p.tm_xq);
      tma_prefetch_desc(&p.tm_w);
      Pipe q = {smem, full_bar, empty_bar, GRP_STAGES, Cfg::STAGE_BYTES, 0, 0u};
      bool ok = true;
      uint32_t gi = 0;  // groups handed out so far, over all tiles
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        const int4 tile = tile_at(p.src, t % tm);
        const int n0 = t / tm * BN;
        const uint32_t sw_bytes = min(BN, p.n - n0) * 4;
        int g = 0;
        for (int kb = 0; kb < kblocks && ok; ++kb) {
          // the scales of the groups that begin inside this K block
          for (; ok && g < groups && g * per_group < (kb + 1) * (BK / UMMA_K_I8); ++g, ++gi) {
            const uint32_t slot = gi % GRP_SW_SLOTS;
            ok = mbar_wait(&sw_empty[slot], ((gi / GRP_SW_SLOTS) & 1u) ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER);
            if (!ok) break;
            mbar_expect_tx(&sw_full[slot], sw_bytes);
            bulk_load(sw_ring + slot * BN, p.sw + static_cast<int64_t>(g) * p.n + n0, sw_bytes, &sw_full[slot]);
          }
          if (!ok) break;
          ok = mbar_wait(&empty_bar[q.stage], q.phase ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER);
          if (!ok) break;
          unsigned char* sa = q.at();
          mbar_expect_tx(&full_bar[q.stage], Cfg::STAGE_BYTES);
          tma_load_2d(sa, &p.tm_xq, kb * BK, tile.x, &full_bar[q.stage]);
          tma_load_3d(sa + BM * BK, &p.tm_w, 0, n0, kb, &full_bar[q.stage]);
          q.next();
        }
        if (ok && lora) ok = lora_load(p, q, tile, n0, abort_flag);
      }
    }
  } else if (warp == 5) {
    const uint32_t idesc = make_idesc(IDESC_D_S32, IDESC_S8, IDESC_S8, BM, BN);
    const uint32_t idesc_lora = make_idesc(IDESC_D_F32, IDESC_BF16, IDESC_BF16, BM, BN);
    const uint32_t smem_base = smem_u32(smem);
    Pipe q = {smem, full_bar, empty_bar, GRP_STAGES, Cfg::STAGE_BYTES, 0, 0u};
    bool ok = true;
    uint32_t gi = 0, rounds = 0;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int in_group = 0;  // MMAs issued of the current group
      uint32_t d = tmem_base;
      for (int kb = 0; kb < kblocks && ok; ++kb) {
        ok = mbar_wait_warp(&full_bar[q.stage], q.phase, abort_flag, p.status, STATUS_TIMEOUT_MMA);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sa = smem_base + q.stage * Cfg::STAGE_BYTES;
        const uint64_t adesc = make_desc_sw128(sa), bdesc = make_desc_sw128(sa + BM * BK);
        for (int j = 0; j < BK / UMMA_K_I8; ++j) {
          if (kb * (BK / UMMA_K_I8) + j >= steps) break;
          if (in_group == 0) {
            const uint32_t buf = gi % GRP_BUFS;
            ok = mbar_wait_warp(&acc_empty[buf], ((gi / GRP_BUFS) & 1u) ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            d = tmem_base + buf * BN;
          }
          if (elect_one()) mma_i8(d, adesc + 2 * j, bdesc + 2 * j, idesc, in_group != 0 ? 1u : 0u);
          __syncwarp();
          if (++in_group == per_group) {
            if (elect_one()) mma_commit(&acc_full[gi % GRP_BUFS]);
            __syncwarp();
            in_group = 0;
            ++gi;
          }
        }
        if (!ok) break;
        if (elect_one()) mma_commit(&empty_bar[q.stage]);
        __syncwarp();
        q.next();
      }
      if (ok && lora) {
        ok = lora_issue<true>(p, q, tile_at(p.src, t % tm), lora_cols, idesc_lora, abort_flag, [&]() {
          return mbar_wait_warp(lora_empty, (rounds & 1u) ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_LORA);
        });
        if (ok && elect_one()) mma_commit(lora_full);
        __syncwarp();
        ++rounds;
      }
    }
  } else {
    constexpr int COLS = BN / 2;  // columns of this warp: two warps share a tensor-memory lane quadrant
    const int quad = warp & 3;
    const int col0 = warp < 4 ? 0 : COLS;
    const int r = quad * 32 + lane;
    const uint64_t one = f32x2(p.one, p.one);
    const uint32_t lanes = (static_cast<uint32_t>(quad * 32) << 16) + col0;
    bool ok = true;
    uint32_t gi = 0, rounds = 0;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const int4 tile = tile_at(p.src, t % tm);
      const int n0 = t / tm * BN + col0;
      const bool row_valid = r < tile.y;
      const float* sxp = p.sx + tile.x + (row_valid ? r : 0);
      uint64_t acc[COLS / 2];
#pragma unroll
      for (int i = 0; i < COLS / 2; ++i) acc[i] = 0ull;
      float sx_next = __ldcg(sxp);
      for (int g = 0; g < groups; ++g, ++gi) {
        const float sxr = sx_next;
        if (g + 1 < groups) sx_next = __ldcg(sxp + static_cast<int64_t>(g + 1) * p.m);
        const uint32_t buf = gi % GRP_BUFS, slot = gi % GRP_SW_SLOTS;
        ok = mbar_wait_warp(&sw_full[slot], (gi / GRP_SW_SLOTS) & 1u, abort_flag, p.status, STATUS_TIMEOUT_EPILOGUE) &&
             mbar_wait_warp(&acc_full[buf], (gi / GRP_BUFS) & 1u, abort_flag, p.status, STATUS_TIMEOUT_EPILOGUE);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t sx2 = f32x2(sxr, sxr);
        const float4* swv = reinterpret_cast<const float4*>(sw_ring + slot * BN + col0);
        uint32_t v[COLS / 16][16];
#pragma unroll
        for (int c = 0; c < COLS / 16; ++c) tmem_ld16(tmem_base + buf * BN + lanes + c * 16, v[c]);
        tmem_wait_ld();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);  // the values are in registers: the buffer is free
#pragma unroll
        for (int c = 0; c < COLS / 16; ++c) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 w = swv[c * 4 + i];
            const uint64_t a0 = f32x2(__int2float_rn(static_cast<int>(v[c][4 * i])), __int2float_rn(static_cast<int>(v[c][4 * i + 1])));
            const uint64_t a1 = f32x2(__int2float_rn(static_cast<int>(v[c][4 * i + 2])), __int2float_rn(static_cast<int>(v[c][4 * i + 3])));
            uint64_t& s0 = acc[c * 8 + 2 * i];
            uint64_t& s1 = acc[c * 8 + 2 * i + 1];
            s0 = add_f32x2(mul_f32x2(mul_f32x2(a0, sx2), f32x2(w.x, w.y)), s0, one);
            s1 = add_f32x2(mul_f32x2(mul_f32x2(a1, sx2), f32x2(w.z, w.w)), s1, one);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sw_empty[slot]);
      }
      if (!ok) break;
      if (lora) {
        ok = mbar_wait_warp(lora_full, rounds & 1u, abort_flag, p.status, STATUS_TIMEOUT_LORA);
        if (!ok) break;
        ++rounds;
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < COLS / 16; ++c) {
          uint32_t v[16];
          tmem_ld16(lora_cols + lanes + c * 16, v);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            acc[c * 8 + i] = add_f32x2(acc[c * 8 + i], f32x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), one);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(lora_empty);
      }
      if (row_valid) {
        const int64_t orow = p.out_row_map != nullptr ? __ldg(p.out_row_map + tile.x + r) : tile.x + r;
        uint4* dst = reinterpret_cast<uint4*>(p.out + orow * p.out_stride + n0);
#pragma unroll
        for (int i = 0; i < COLS / 8; ++i) {
          if (n0 + i * 8 >= p.n) break;
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float lo, hi;
            f32x2_parts(acc[i * 4 + j], lo, hi);
            o[j] = pack_bf16x2(lo, hi);
          }
          dst[i] = make_uint4(o[0], o[1], o[2], o[3]);
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
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

template <int BN>
static int launch_grouped_bn(const GrpParams& p, int grid, cudaStream_t stream) {
  static bool attr_set[MAX_DEVICES] = {};
  auto kernel = w8a8_grouped_gemm_kernel<BN>;
  cudaError_t e = ensure_dynamic_smem(kernel, GrpCfg<BN>::SMEM_BYTES, attr_set);
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "grouped gemm attribute: %s", cudaGetErrorString(e));
  e = launch_kernel(kernel, dim3(grid), dim3(GRP_THREADS), GrpCfg<BN>::SMEM_BYTES, stream, true, p);
  if (e == cudaSuccess) e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "grouped gemm launch: %s", cudaGetErrorString(e));
  return SKYRL_OK;
}

int launch_grouped_gemm(const GroupedGemmLaunch& a, cudaStream_t stream) {
  if (a.m <= 0 || a.n <= 0 || a.k <= 0 || a.n % 32 != 0 || a.k % 16 != 0 || a.group <= 0 || a.group % UMMA_K_I8 != 0 ||
      a.k % a.group != 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped gemm: bad shape (N %% 32, group %% 32 and K %% group must be 0)");
  if (!aligned16(a.xq) || !aligned16(a.wq) || !aligned16(a.sw) || !aligned16(a.out) || a.out_stride < a.n || a.out_stride % 8 != 0)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped gemm: misaligned buffer or bad stride");
  const int sms = sm_count();
  if (sms <= 0) return fail(SKYRL_ERR_LAUNCH, "grouped gemm: no CUDA device");
  // The widest tile whose tiles still occupy most SMs: the epilogue warps of an SM are the resource, so a half-empty GPU
  // costs more than the activation tiles that narrower tiles read again.
  const int tm = a.src.count;
  int bn = 128;
  while (bn > 32 && tm * ((a.n + bn - 1) / bn) * 4 < 3 * sms) bn >>= 1;
  GrpParams p = {};
  int rc;
  if ((rc = encode_tmap_2d(&p.tm_xq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.xq, a.k, a.m, a.k, BK, BM))) return rc;
  if ((rc = encode_tmap_3d(&p.tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.wq, BK, a.n, (a.k + BK - 1) / BK, BK,
                           static_cast<uint64_t>(a.n) * BK, BK, bn)))
    return rc;
  p.tm_z = p.tm_xq;
  p.tm_b = p.tm_xq;
  if (a.rank > 0) {
    if (a.z_parts == nullptr || a.b_table == nullptr || !aligned16(a.b_table) || a.b_slots < a.rank || a.b_slots % 8 != 0)
      return fail(SKYRL_ERR_INVALID_ARGUMENT, "grouped gemm: LoRA operands missing or misaligned");
    const uint32_t half = (a.rank <= 16 ? 32 : (a.rank <= 32 ? 64 : 128)) / 2;
    if ((rc = encode_tmap_3d(&p.tm_z, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.z_parts, SKYRL_LORA_RANK_PAD, SKYRL_Z_PARTS, a.m,
                             SKYRL_LORA_RANK_PAD * 2, SKYRL_Z_PARTS * SKYRL_LORA_RANK_PAD * 2, half, 1, BM)))
      return rc;
    if ((rc = encode_tmap_3d(&p.tm_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.b_table, a.b_slots, a.n, a.num_adapters,
                             static_cast<uint64_t>(a.b_slots) * 2, static_cast<uint64_t>(a.n) * a.b_slots * 2, half, bn)))
      return rc;
    p.lora = lora_geom(a.rank, bn, BM * BK + bn * BK, GRP_STAGES);
  }
  p.src = a.src;
  p.rank_blocks = (a.rank + 15) / 16;
  p.sx = a.sx;
  p.sw = a.sw;
  p.out_row_map = a.out_row_map;
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.out_stride = a.out_stride;
  p.status = a.status;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.group = a.group;
  p.one = 1.0f;
  const int64_t total = static_cast<int64_t>(tm) * ((a.n + bn - 1) / bn);
  const int grid = static_cast<int>(total < sms ? total : sms);
  if (bn == 128) return launch_grouped_bn<128>(p, grid, stream);
  if (bn == 64) return launch_grouped_bn<64>(p, grid, stream);
  return launch_grouped_bn<32>(p, grid, stream);
}

}  // namespace skyrl
