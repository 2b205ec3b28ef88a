// What the tensor-core GEMM kernels share: tile geometry, the TMA pipeline cursor, and the LoRA operands of a tile.
// `P` is a kernel's parameter block with tensor maps tm_z and tm_b, the tile source `src`, the geometry `lora`,
// `rank_blocks` and the status word.
#pragma once

#include "ptx_sm100.cuh"
#include "tiles.cuh"

namespace skyrl {

constexpr int BM = 128;       // rows per tile == TMEM lanes
constexpr int BK = 128;       // int8 elements (bytes) of K per pipeline stage: one 128-byte swizzled row
constexpr int UMMA_K_I8 = 32; // K of one kind::i8 instruction

// The LoRA operands of one M tile x N tile travel through slots of the TMA pipeline, at the width of the rank
// (w = 32, 64 or 128 bytes per row for ranks up to 16, 32, 64, with the swizzle of that width).  They come in rounds:
// the three z planes of the tile's rows, then the LoRA-B tiles of its segments (adapters), several to a slot; a round
// never takes more slots than the pipeline has, so the slots of the planes can stay until its last MMA.
struct LoraGeom {
  int w;             // bytes per row of z and of a LoRA-B tile
  int z_plane;       // bytes of one plane: 128 rows
  int z_per_slot;    // planes per slot
  int b_tile;        // bytes of one adapter's LoRA-B tile
  int b_per_slot;    // adapters per slot
  int b_per_round;   // adapters per round
};
inline LoraGeom lora_geom(int rank, int b_rows, int stage_bytes, int stages) {
  LoraGeom g;
  g.w = rank <= 16 ? 32 : (rank <= 32 ? 64 : 128);
  g.z_plane = BM * g.w;
  g.z_per_slot = stage_bytes / g.z_plane < 3 ? stage_bytes / g.z_plane : 3;
  g.b_tile = b_rows * g.w;
  g.b_per_slot = stage_bytes / g.b_tile;
  g.b_per_round = (stages - (3 + g.z_per_slot - 1) / g.z_per_slot) * g.b_per_slot;
  return g;
}

// ---- LoRA operands of one tile through the TMA pipeline (one CTA per tile; see LoraGeom) ----------------
struct Pipe {
  unsigned char* smem;
  uint64_t* full;
  uint64_t* empty;
  int stages, bytes, stage;
  uint32_t phase;
  __device__ __forceinline__ void next() {
    if (++stage == stages) {
      stage = 0;
      phase ^= 1u;
    }
  }
  __device__ __forceinline__ unsigned char* at() const { return smem + stage * bytes; }
};

// A tile of many adapters (16 in each of two tiles for 256 rows over 32) would pay one round trip to memory per
// segment if its adapter and its row mask were read where they are used, between the waits: 17 segments added about 10 us
// to a tile's tail.  They are read ahead instead: eight adapters at a time by the producing thread, one segment's mask
// per lane by the issuing warp.
struct SegmentAdapters {
  int held[8];
  int first = -8;
  template <typename Fetch>
  __device__ __forceinline__ int at(int j, int nseg, Fetch fetch) {
    if (j >= first + 8) {
      first = j & ~7;
#pragma unroll
      for (int i = 0; i < 8; ++i) held[i] = first + i < nseg ? fetch(first + i) : 0;
    }
    return held[j & 7];
  }
};
__device__ __forceinline__ int4 shfl_int4(const int4& v, int lane) {
  return make_int4(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane),
                   __shfl_sync(0xffffffffu, v.z, lane), __shfl_sync(0xffffffffu, v.w, lane));
}

template <typename P>
__device__ __forceinline__ bool lora_load(const P& p, Pipe& q, const int4& tile, int n0, volatile int* abort_flag) {
  const LoraGeom& g = p.lora;
  const int nseg = tile_segments(tile);
  const bool dense = tile_is_dense(tile);
  SegmentAdapters adapters;
  for (int j = 0; j < nseg;) {
    const int slot = segment_slot(tile, j);
    for (int pl = 0; pl < 3; pl += g.z_per_slot) {  // lo, mid, hi: the smallest plane is added first
      if (!mbar_wait(&q.empty[q.stage], q.phase ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER)) return false;
      const int cnt = min(g.z_per_slot, 3 - pl);
      mbar_expect_tx(&q.full[q.stage], cnt * g.z_plane);
      for (int i = 0; i < cnt; ++i)
        tma_load_3d(q.at() + i * g.z_plane, &p.tm_z, 0, 3 * slot + 2 - (pl + i), tile.x, &q.full[q.stage]);
      q.next();
    }
    // a list of two slots keeps the second adapter's z elsewhere: every adapter is a round of its own
    for (int left = dense ? min(nseg - j, g.b_per_round) : 1; left > 0;) {
      const int cnt = min(g.b_per_slot, left);
      if (!mbar_wait(&q.empty[q.stage], q.phase ^ 1u, abort_flag, p.status, STATUS_TIMEOUT_PRODUCER)) return false;
      mbar_expect_tx(&q.full[q.stage], cnt * g.b_tile);
      for (int i = 0; i < cnt; ++i)
        tma_load_3d(q.at() + i * g.b_tile, &p.tm_b, 0, n0,
                    adapters.at(j + i, nseg, [&](int s) { return segment_adapter(p.src, tile, s); }), &q.full[q.stage]);
      q.next();
      j += cnt;
      left -= cnt;
    }
  }
  return true;
}

// Descriptors of the three z planes of a round whose first slot is `stage`.  Computed once: with a division per plane in
// front of every MMA an adapter cost the issuing warp 1400 cycles.
__device__ __forceinline__ void lora_plane_descs(const LoraGeom& g, uint32_t smem_base, int stage_bytes, int stages, int stage,
                                                 uint64_t (&zd)[3]) {
  int in_slot = 0;
#pragma unroll
  for (int plane = 0; plane < 3; ++plane) {
    zd[plane] = make_desc_width(smem_base + stage * stage_bytes + in_slot * g.z_plane, g.w);
    if (++in_slot == g.z_per_slot) {
      in_slot = 0;
      stage = stage + 1 == stages ? 0 : stage + 1;
    }
  }
}

// rank-r bf16 MMAs of one tile, accumulated onto the accumulator `d` the epilogue rewrote as fp32 (`ready` waits for
// that rewrite, once the first operands are there); every segment touches the lanes of its own rows only.  FRESH: `d` are
// columns of the LoRA term's own, whose first contribution overwrites.  Called by a whole warp, which elects a thread for
// the instructions.
template <bool FRESH = false, typename P, typename Ready>
__device__ __forceinline__ bool lora_issue(const P& p, Pipe& q, const int4& tile, uint32_t d, uint32_t idesc,
                                           volatile int* abort_flag, Ready ready) {
  const LoraGeom& g = p.lora;
  const int nseg = tile_segments(tile);
  const bool dense = tile_is_dense(tile);
  const int lane = static_cast<int>(threadIdx.x & 31u);
  int4 lane_mask = make_int4(0, 0, 0, 0);  // of segment (j & ~31) + lane
  int masks_from = -32;
  for (int j = 0; j < nseg;) {
    const int zstage0 = q.stage;
    const int zslots = (3 + g.z_per_slot - 1) / g.z_per_slot;
    for (int i = 0; i < zslots; ++i) {
      if (!mbar_wait_warp(&q.full[q.stage], q.phase, abort_flag, p.status, STATUS_TIMEOUT_LORA)) return false;
      q.next();
    }
    uint64_t zd[3];
    lora_plane_descs(g, smem_u32(q.smem), q.bytes, q.stages, zstage0, zd);
    const bool first = j == 0;
    bool started = false;
    for (int left = dense ? min(nseg - j, g.b_per_round) : 1; left > 0;) {
      const int cnt = min(g.b_per_slot, left);
      if (!mbar_wait_warp(&q.full[q.stage], q.phase, abort_flag, p.status, STATUS_TIMEOUT_LORA)) return false;
      if (first && !started && !ready()) return false;
      started = true;
      tc_fence_after_sync();
      uint64_t bd = make_desc_width(smem_u32(q.at()), g.w);
      for (int i = 0; i < cnt; ++i) {
        if (j + i >= masks_from + 32) {
          masks_from = (j + i) & ~31;
          lane_mask = segment_mask(p.src, tile, min(masks_from + lane, nseg - 1));
        }
        const int4 mk = shfl_int4(lane_mask, (j + i) & 31);
        const int4 off = make_int4(~mk.x, ~mk.y, ~mk.z, ~mk.w);
        if (elect_one()) {
#pragma unroll
          for (int plane = 0; plane < 3; ++plane)
            for (int kk = 0; kk < p.rank_blocks; ++kk)
              mma_bf16_lanes(d, zd[plane] + 2 * kk, bd + 2 * kk, idesc, FRESH && plane == 0 && kk == 0 ? 0u : 1u, off);
        }
        __syncwarp();
        bd += g.b_tile >> 4;  // the descriptor's address field counts 16 bytes
      }
      if (elect_one()) mma_commit(&q.empty[q.stage]);
      __syncwarp();
      q.next();
      j += cnt;
      left -= cnt;
    }
    if (elect_one()) {
      for (int i = 0; i < zslots; ++i) mma_commit(&q.empty[(zstage0 + i) % q.stages]);
    }
    __syncwarp();
  }
  return true;
}

}  // namespace skyrl
