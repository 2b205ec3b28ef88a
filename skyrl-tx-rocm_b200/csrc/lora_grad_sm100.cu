// Parameter gradients of the LoRA tables and the table layouts of a training step.
//
//   dA[a][k, j] = sum over the rows i of adapter a of  x[i, k]  * zb[i, j]     zb = s (dy B^T)
//   dB[a][j, n] = sum over the rows i of adapter a of  dy[i, n] * z[i, j]      z  = s (x A)
//
// (skyrl/tx/kernels/quantized_lora.py:374-389, the scaling already inside z and zb).  Both are tall contractions over
// rows with a result of rank columns, so x and dy are read once and the floor is their bytes: one CTA takes 128 columns of
// x (or dy) and the rows of one adapter, multiplies 64 rows at a time on the tensor cores (both operands with the row
// as the slow index in shared memory, i.e. MN-major) and keeps the 128 x rank result in tensor memory.  z and zb are
// the bf16 parts the projection kernel leaves: the three parts sit side by side as one operand of 3 x rank columns and
// are added at the end, so the factor enters with its full fp32 value at the cost of one MMA.
//
// Rows are adapter-sorted through `perm`: the loads gather them (16-byte asynchronous copies, eight lanes per 128-byte
// row piece; the tensor-map gather delivers 512 bytes per 74 cycles and would bound the kernel), rows past the adapter's
// last are filled with zeros.  Where tables and blocks are too few for the GPU, a cluster shares the rows of a block and
// adds its partial sums in rank order through distributed shared memory.
//
// Before, a training step of eight adapters spent 150 launches of library matmuls, casts and additions here.  Now one launch,
// 197 us at 4096 rows, K 12288, N 4096, rank 32, 8 adapters, for 138 MB (21 us): no unit is near its limit (DRAM 9 %, issue
// 8 %), the loads of a stage wait for its row indices, and 1024 short CTAs pay fill and drain one after the other.
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace skyrl {

constexpr int LG_COLS = 128;     // columns of x or dy per CTA: accumulator lanes
constexpr int LG_ROWS = 64;      // rows per stage
constexpr int LG_STAGES = 4;
constexpr int LG_LAG = LG_STAGES - 1;
constexpr int LG_X_BYTES = LG_ROWS * LG_COLS * 2;
constexpr int LG_THREADS = 192;  // warps 0-3 load x, then drain; warp 4 loads z; warp 5 issues the MMAs
constexpr int LG_MAX_CLUSTER = 8;

struct LoraGradJob {
  const __nv_bfloat16* src;   // x or dy
  int64_t stride;
  int cols, blocks;           // columns (multiple of 8), blocks of 128
  int out_cols;               // columns of the result (dB of an N that is no multiple of 32 drops the padding)
  __nv_bfloat16* out;         // [A, cols, rank] or [A, rank, out_cols]
};
struct LoraGradParams {
  CUtensorMap tm_z[2];        // bf16 [m, 6, 64], box w / 2 x 1 x 64: zb for dA, z for dB
  LoraGradJob job[2];
  const int32_t* perm;           // NULL: rows as they are
  const int32_t* adapter_start;  // [A + 1]; NULL: one adapter, all rows
  int m, adapters, rank, w;
  int32_t* status;
};

template <int W>
struct LgCfg {
  static constexpr int Z_PLANE = LG_ROWS * W;
  static constexpr int STAGE_BYTES = LG_X_BYTES + 3 * Z_PLANE;
  static constexpr int BAR_OFF = LG_STAGES * STAGE_BYTES;
  static constexpr int SMEM_BYTES = BAR_OFF + (2 * LG_STAGES + 1) * 8 + 16 + 1024;
  static constexpr int N = 3 * (W / 2);
  static constexpr int TMEM_COLS = N <= 64 ? 64 : (N <= 128 ? 128 : 256);
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {  // bytes 0: zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// MN-major operand: rows of W bytes along M or N (swizzle of that width), 8-row groups of K 8 W bytes apart, the next
// W-byte column block `block` bytes away
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t smem_addr, uint32_t w, uint32_t block) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(block >> 4) << 16;
  d |= static_cast<uint64_t>(w >> 1) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(w == 128 ? 2 : (w == 64 ? 4 : 6)) << 61;
  return d;
}

template <int W>
__global__ void __launch_bounds__(LG_THREADS) lora_grad_kernel(const __grid_constant__ LoraGradParams p) {
  using Cfg = LgCfg<W>;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* empty_bar = full_bar + LG_STAGES;
  uint64_t* acc_full = empty_bar + LG_STAGES;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int csize = static_cast<int>(cluster_size());
  const int crank = csize > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  int unit = static_cast<int>(blockIdx.x) / csize;
  const int which = unit < p.adapters * p.job[0].blocks ? 0 : 1;
  if (which == 1) unit -= p.adapters * p.job[0].blocks;
  const LoraGradJob& job = p.job[which];
  const int adapter = unit / job.blocks, block = unit % job.blocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < LG_STAGES; ++s) {
      mbar_init(&full_bar[s], 128 + 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
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
  pdl_wait();
  pdl_trigger();

  const int first = p.adapter_start != nullptr ? __ldcg(p.adapter_start + adapter) : 0;
  const int last = p.adapter_start != nullptr ? __ldcg(p.adapter_start + adapter + 1) : p.m;
  // this CTA's share of the adapter's rows: whole stages
  const int stages_all = (last - first + LG_ROWS - 1) / LG_ROWS;
  const int per = (stages_all + csize - 1) / csize;
  const int r0 = min(last, first + crank * per * LG_ROWS), r1 = min(last, r0 + per * LG_ROWS);
  const int count = (r1 - r0 + LG_ROWS - 1) / LG_ROWS;

  if (warp < 4) {
    // ---- x: warp w loads rows 16 w ... 16 w + 15 of a stage, eight lanes per 128-byte piece of a row
    const int piece = lane & 7, sub = lane >> 3;
    const uint32_t smem_base = smem_u32(smem);
    bool ok = true;
    for (int i = 0; i < count; ++i) {
      const int stage = i % LG_STAGES;
      ok = mbar_wait_warp(&empty_bar[stage], ((i / LG_STAGES) & 1u) ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER);
      if (!ok) break;
      const uint32_t sa = smem_base + stage * Cfg::STAGE_BYTES;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int r = warp * 16 + g * 4 + sub;
        const int srow = r0 + i * LG_ROWS + r;
        const bool live = srow < r1;
        const int64_t row = live ? (p.perm != nullptr ? __ldcg(p.perm + srow) : srow) : 0;
        const __nv_bfloat16* src = job.src + row * job.stride;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int col = block * LG_COLS + h * 64 + piece * 8;
          const bool in = live && col < job.cols;
          cp_async16(sa + h * (LG_X_BYTES / 2) + r * 128 + ((piece ^ (r & 7)) << 4), in ? src + col : job.src, in ? 16u : 0u);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (i >= LG_LAG) {  // the copies of LG_LAG stages ago have landed: hand them to the tensor cores
        asm volatile("cp.async.wait_group %0;" ::"n"(LG_LAG) : "memory");
        fence_proxy_async_smem();
        mbar_arrive(&full_bar[(i - LG_LAG) % LG_STAGES]);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_proxy_async_smem();
    if (ok)
      for (int i = max(0, count - LG_LAG); i < count; ++i) mbar_arrive(&full_bar[i % LG_STAGES]);
  } else if (warp == 4) {
    if (lane == 0) {
      for (int i = 0; i < count; ++i) {
        const int stage = i % LG_STAGES;
        if (!mbar_wait(&empty_bar[stage], ((i / LG_STAGES) & 1u) ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER)) break;
        unsigned char* z = smem + stage * Cfg::STAGE_BYTES + LG_X_BYTES;
        mbar_expect_tx(&full_bar[stage], 3 * Cfg::Z_PLANE);
        for (int q = 0; q < 3; ++q)
          tma_load_3d(z + q * Cfg::Z_PLANE, &p.tm_z[which], 0, q, r0 + i * LG_ROWS, &full_bar[stage]);
      }
    }
  } else {
    const uint32_t idesc = make_idesc(IDESC_D_F32, IDESC_BF16, IDESC_BF16, LG_COLS, Cfg::N) | (1u << 15) | (1u << 16);
    const uint32_t smem_base = smem_u32(smem);
    bool ok = true;
    for (int i = 0; i < count; ++i) {
      const int stage = i % LG_STAGES;
      ok = mbar_wait_warp(&full_bar[stage], (i / LG_STAGES) & 1u, abort_flag, p.status, STATUS_TIMEOUT_MMA);
      if (!ok) break;
      const uint32_t sx = smem_base + stage * Cfg::STAGE_BYTES, sz = sx + LG_X_BYTES;
      const int valid = min(LG_ROWS, r1 - r0 - i * LG_ROWS);
      if (valid < LG_ROWS) {
        // the box also brought the first rows of the next adapter: they must not count
        uint4* z = reinterpret_cast<uint4*>(smem + stage * Cfg::STAGE_BYTES + LG_X_BYTES);
        for (int q = 0; q < 3; ++q)
          for (int v = valid * (W / 16) + lane; v < LG_ROWS * (W / 16); v += 32)
            z[q * (Cfg::Z_PLANE / 16) + v] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
        __syncwarp();
      }
      tc_fence_after_sync();
      if (elect_one()) {
        const uint64_t ad = make_desc_mn(sx, 128, LG_X_BYTES / 2), bd = make_desc_mn(sz, W, Cfg::Z_PLANE);
#pragma unroll
        for (int ks = 0; ks < LG_ROWS / 16; ++ks)
          mma_bf16(tmem_base, ad + ks * (16 * 128 / 16), bd + ks * (16 * W / 16), idesc, (i > 0 || ks > 0) ? 1u : 0u);
        mma_commit(&empty_bar[stage]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(acc_full);
    __syncwarp();
  }

  // ---- result: lane r of the accumulator is column block * 128 + r of x or dy
  const int rank16 = (p.rank + 15) / 16 * 16;
  float* part = reinterpret_cast<float*>(smem);  // cluster form: [128][rank16 + 4] in the drained stages
  const int pitch = rank16 + 4;
  bool ok = true;
  auto store = [&](int r, int j, float v) {
    const int c = block * LG_COLS + r;
    if (c >= job.out_cols || j >= p.rank) return;
    const int64_t at = which == 0 ? (static_cast<int64_t>(adapter) * job.cols + c) * p.rank + j
                                  : (static_cast<int64_t>(adapter) * p.rank + j) * job.out_cols + c;
    job.out[at] = __float2bfloat16_rn(v);
  };
  if (warp < 4) {
    const int r = warp * 32 + lane;
    if (count > 0) {
      ok = mbar_wait_warp(acc_full, 0u, abort_flag, p.status, STATUS_TIMEOUT_EPILOGUE);
      tc_fence_after_sync();
    }
    if (ok) {
      for (int cc = 0; cc < rank16 / 16; ++cc) {
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = 0.f;
        if (count > 0) {
          const uint32_t lanes = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + cc * 16;
          uint32_t hi[16], mid[16], lo[16];
          tmem_ld16(lanes, hi);
          tmem_ld16(lanes + W / 2, mid);
          tmem_ld16(lanes + W, lo);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i)
            f[i] = __fadd_rn(__fadd_rn(__uint_as_float(lo[i]), __uint_as_float(mid[i])), __uint_as_float(hi[i]));
        }
        if (csize > 1) {
          float4* dst = reinterpret_cast<float4*>(part + r * pitch + cc * 16);
#pragma unroll
          for (int g = 0; g < 4; ++g) dst[g] = make_float4(f[4 * g], f[4 * g + 1], f[4 * g + 2], f[4 * g + 3]);
        } else if (which == 0 && p.rank % 8 == 0) {
          const int c = block * LG_COLS + r;
          if (c < job.out_cols) {
            uint4* dst = reinterpret_cast<uint4*>(job.out + (static_cast<int64_t>(adapter) * job.cols + c) * p.rank + cc * 16);
#pragma unroll
            for (int g = 0; g < 2; ++g)
              if (cc * 16 + g * 8 < p.rank)
                dst[g] = make_uint4(pack_bf16x2(f[8 * g], f[8 * g + 1]), pack_bf16x2(f[8 * g + 2], f[8 * g + 3]),
                                    pack_bf16x2(f[8 * g + 4], f[8 * g + 5]), pack_bf16x2(f[8 * g + 6], f[8 * g + 7]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) store(r, cc * 16 + i, f[i]);
        }
      }
    }
  }
  if (csize > 1) {
    __syncwarp();
    cluster_sync_all();
    if (warp < 4) {
      const int rows_per = LG_COLS / csize, quads = rank16 / 4;
      for (int item = threadIdx.x; item < rows_per * quads; item += 128) {
        // neighbouring threads along the contiguous axis of the result
        const int r = crank * rows_per + (which == 0 ? item / quads : item % rows_per);
        const int q = which == 0 ? item % quads : item / rows_per;
        const uint32_t local = smem_u32(part) + static_cast<uint32_t>((r * pitch + 4 * q) * 4);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int c = 0; c < csize; ++c) {
          const float4 v = ld_cluster_float4(map_to_cta(local, c));
          s.x = __fadd_rn(s.x, v.x);
          s.y = __fadd_rn(s.y, v.y);
          s.z = __fadd_rn(s.z, v.z);
          s.w = __fadd_rn(s.w, v.w);
        }
        store(r, 4 * q, s.x);
        store(r, 4 * q + 1, s.y);
        store(r, 4 * q + 2, s.z);
        store(r, 4 * q + 3, s.w);
      }
    }
    __syncwarp();
    cluster_sync_all();
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

template <int W>
static int launch_lora_grad_w(const LoraGradParams& p, int units, int cluster, cudaStream_t stream) {
  static bool attr_set[MAX_DEVICES] = {};
  auto kernel = lora_grad_kernel<W>;
  cudaError_t e = ensure_dynamic_smem(kernel, LgCfg<W>::SMEM_BYTES, attr_set);
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "lora_grad attribute: %s", cudaGetErrorString(e));
  e = launch_cluster_kernel(kernel, dim3(units * cluster), dim3(LG_THREADS), LgCfg<W>::SMEM_BYTES, stream, cluster, p);
  if (e == cudaSuccess) e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "lora_grad launch: %s", cudaGetErrorString(e));
  return SKYRL_OK;
}

int launch_lora_grad(const LoraGradLaunch& a, cudaStream_t stream) {
  if (a.x == nullptr || a.dy == nullptr || a.z == nullptr || a.zb == nullptr || a.da == nullptr || a.db == nullptr ||
      a.status == nullptr || a.m <= 0 || a.k <= 0 || a.n <= 0 || a.adapters <= 0 || a.rank <= 0 || a.rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_grad: null buffer or bad shape");
  if (a.k % 8 != 0 || a.n % 8 != 0 || a.n_logical > a.n || !aligned16(a.x) || !aligned16(a.dy) || a.x_stride % 8 != 0 ||
      a.dy_stride % 8 != 0 || a.x_stride < a.k || a.dy_stride < a.n || !aligned16(a.da))
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_grad: rows must be 16-byte aligned");
  if (a.adapters > 1 && a.adapter_start == nullptr)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "lora_grad: row ranges of the adapters missing");
  LoraGradParams p = {};
  p.w = a.rank <= 16 ? 32 : (a.rank <= 32 ? 64 : 128);
  for (int j = 0; j < 2; ++j) {
    const int rc = encode_tmap_3d(&p.tm_z[j], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, j == 0 ? a.zb : a.z, SKYRL_LORA_RANK_PAD,
                                  SKYRL_Z_PARTS, a.m, SKYRL_LORA_RANK_PAD * 2, SKYRL_Z_PARTS * SKYRL_LORA_RANK_PAD * 2,
                                  p.w / 2, 1, LG_ROWS);
    if (rc) return rc;
  }
  p.job[0] = {static_cast<const __nv_bfloat16*>(a.x), a.x_stride, a.k, (a.k + LG_COLS - 1) / LG_COLS, a.k,
              static_cast<__nv_bfloat16*>(a.da)};
  p.job[1] = {static_cast<const __nv_bfloat16*>(a.dy), a.dy_stride, a.n, (a.n + LG_COLS - 1) / LG_COLS, a.n_logical,
              static_cast<__nv_bfloat16*>(a.db)};
  p.perm = a.perm;
  p.adapter_start = a.adapter_start;
  p.m = a.m;
  p.adapters = a.adapters;
  p.rank = a.rank;
  p.status = a.status;
  const int units = a.adapters * (p.job[0].blocks + p.job[1].blocks);
  // rows of a block shared by a cluster while that still fits the GPU once, each CTA with two stages or more of an
  // average adapter's rows
  int sms = sm_count();
  if (sms <= 0) sms = 148;
  int cluster = LG_MAX_CLUSTER;
  while (cluster > 1 && (units * cluster > 2 * sms || a.m / a.adapters < 2 * LG_ROWS * cluster)) cluster >>= 1;
  if (p.w == 32) return launch_lora_grad_w<32>(p, units, cluster, stream);
  if (p.w == 64) return launch_lora_grad_w<64>(p, units, cluster, stream);
  return launch_lora_grad_w<128>(p, units, cluster, stream);
}

// ---- table layouts of a training step ------------------------------------------------------------------------
// A [A, k, r] -> [A, r, k] (K-major operand of the projection) and B [A, r, n] -> [A, n_pad, rr] (operand of the GEMM's
// LoRA term, rank and columns zero-padded): the tables change at every optimizer step, so both are laid out by one
// launch.  A CTA turns 64 rows of K (or columns of N) of one adapter through shared memory.
__global__ void __launch_bounds__(256)
train_tables_kernel(const uint16_t* __restrict__ a, const uint16_t* __restrict__ b, int adapters, int k, int n, int n_pad,
                    int rank, int rr, uint16_t* __restrict__ at, uint16_t* __restrict__ bt, int a_blocks, int b_blocks) {
  __shared__ uint16_t tile[64][65];
  pdl_wait();
  pdl_trigger();
  int unit = blockIdx.x;
  if (unit < adapters * a_blocks) {
    const int ad = unit / a_blocks, k0 = unit % a_blocks * 64;
    const int rows = min(64, k - k0);
    const uint16_t* src = a + (static_cast<int64_t>(ad) * k + k0) * rank;
    for (int i = threadIdx.x; i < rows * rank; i += 256) tile[i / rank][i % rank] = src[i];
    __syncthreads();
    for (int i = threadIdx.x; i < rank * 64; i += 256) {
      const int j = i >> 6, c = i & 63;
      if (c < rows) at[(static_cast<int64_t>(ad) * rank + j) * k + k0 + c] = tile[c][j];
    }
  } else {
    unit -= adapters * a_blocks;
    const int ad = unit / b_blocks, n0 = unit % b_blocks * 64;
    for (int i = threadIdx.x; i < rr * 64; i += 256) {
      const int j = i >> 6, c = i & 63;
      tile[c][j] = (j < rank && n0 + c < n) ? b[(static_cast<int64_t>(ad) * rank + j) * n + n0 + c] : uint16_t(0);
    }
    __syncthreads();
    const int rows = min(64, n_pad - n0);
    uint16_t* dst = bt + (static_cast<int64_t>(ad) * n_pad + n0) * rr;
    for (int i = threadIdx.x; i < rows * rr; i += 256) dst[i] = tile[i / rr][i % rr];
  }
}

int launch_train_tables(const void* a, const void* b, int adapters, int k, int n, int n_pad, int rank, void* at, void* bt,
                        cudaStream_t stream) {
  if (a == nullptr || b == nullptr || at == nullptr || bt == nullptr || adapters <= 0 || k <= 0 || n <= 0 || n_pad < n ||
      rank <= 0 || rank > SKYRL_LORA_RANK_PAD)
    return fail(SKYRL_ERR_INVALID_ARGUMENT, "train_tables: null buffer or bad shape");
  const int a_blocks = (k + 63) / 64, b_blocks = (n_pad + 63) / 64;
  cudaError_t e = launch_kernel(train_tables_kernel, dim3(adapters * (a_blocks + b_blocks)), dim3(256), 0, stream, true,
                                static_cast<const uint16_t*>(a), static_cast<const uint16_t*>(b), adapters, k, n, n_pad, rank,
                                (rank + 7) / 8 * 8, static_cast<uint16_t*>(at), static_cast<uint16_t*>(bt), a_blocks, b_blocks);
  if (e == cudaSuccess) e = cudaPeekAtLastError();
  if (e != cudaSuccess) return fail(SKYRL_ERR_LAUNCH, "train_tables launch: %s", cudaGetErrorString(e));
  return SKYRL_OK;
}

}  // namespace skyrl
