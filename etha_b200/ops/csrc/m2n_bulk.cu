// TMA variant of the fast copy class: cp.async.bulk global -> shared -> global through a ring of stages.
//
// Two warps per CTA drive the copy engine.  The load warp walks the tiles (see TileSched: a CTA takes over the tiles of
// CTAs not launched yet), cuts them into stage-sized fills, computes the (at most one per matrix row) contiguous pieces of
// a fill in parallel, arms the stage's `full` barrier with the byte count and issues the pieces as untiled bulk loads; the
// store warp waits for the barrier and writes the same pieces out with bulk stores from shared memory, and hands the
// stage back (`empty`) once its stores have read it.  No cluster, no multicast.
//
// Loads always read this GPU's own memory; the stores go to local memory, to a peer's memory over NVLink
// (plain non-multicast bulk stores to the mapped peer address) or to several replicas one after the other
// (a Replicate fan-out: the stage is read from HBM once and stored once per destination).  Every address
// and size handed to the copy engine is a multiple of 16 bytes: the table packer admits only 16-byte units
// with 16-byte aligned bases and strides into this class.  A side that is contiguous over the whole fill is
// moved with ONE bulk copy per stage instead of one per matrix row.
// Waits on the barriers are bounded: after the limit the warp records an error word, drains its own stores
// and returns; the other warp runs into its own limit.  Tiles given up count as finished, and the error word keeps the
// flags back.
//
// 1 GiB on one GPU, read + written: contiguous 6.63 TB/s, 2 KiB rows out of 8 KiB ones 6.52, one source and four
// destinations 6.50 (one warp for both directions and a fixed stride of tiles: 6.00, 5.42, 5.67).  Six stages of 32 KiB,
// on a GPU where they gave 6.55 / 6.46 / 6.46: 12 x 16 KiB gives 6.48 / 6.19 / 6.46, 3 x 32 KiB 6.48 / 6.40 / 6.42.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>

#include "common.h"
#include "m2n_device.cuh"
#include "m2n_launch.h"

namespace {

#ifndef ETHA_BULK_STAGES
#define ETHA_BULK_STAGES 6
#endif
#ifndef ETHA_BULK_STAGE_KB
#define ETHA_BULK_STAGE_KB 32
#endif
constexpr int kStages = ETHA_BULK_STAGES;
constexpr uint32_t kStageBytes = ETHA_BULK_STAGE_KB * 1024;
constexpr uint32_t kMinRowBytes = 512;  // shortest matrix row the packer admits into this class
// store pieces (row fragments) per stage: a fill that starts and ends inside a row touches one row more than
// stage bytes / row bytes; the kernel still checks every fill against this bound before it issues anything
constexpr int kMaxPieces = kStageBytes / kMinRowBytes + 2;
constexpr uint32_t kWaitSpins = 1u << 22;

struct StageMeta {
  int64_t dof[kMaxPieces];  // byte offset of the piece inside every destination slice
  uint32_t off[kMaxPieces];
  uint32_t bytes[kMaxPieces];
  uint64_t dst[M2N_MAX_DST];
  uint32_t ndst;
  uint32_t npieces;  // 0: no fill follows
};

struct Ring {
  StageMeta meta[kStages];
  uint64_t full[kStages], empty[kStages];
  TileSched sched;
  M2NOp op;  // the load warp's copy of the op it works on
};

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// bounded wait of a whole warp
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  bool ready = false;
  for (uint32_t spin = 0; spin < kWaitSpins; ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) { ready = true; break; }
    if (spin > 64) __nanosleep(64);
  }
  return __all_sync(0xffffffffu, ready);
}
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(smem_dst)),
               "l"(gsrc), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_addr(smem_src)),
               "r"(bytes)
               : "memory");
}

// issue the loads of units [u0, u1) into a stage and record the matching stores; false (nothing issued) if the fill would
// need more store pieces than the stage's table holds
__device__ __forceinline__ bool issue_fill(const M2NOp& op, uint32_t u0, uint32_t u1, StageMeta& m, unsigned char* buf,
                                           uint64_t* full, uint32_t lane) {
  const bool rows = op.ndim != 0;
  const uint32_t inner = rows ? op.inner_units : 0xffffffffu;
  const uint32_t r0 = rows ? fast_div(u0, op.div_mul[M2N_MAX_DIMS], op.div_shr[M2N_MAX_DIMS]) : 0;
  const uint32_t r1 = rows ? fast_div(u1 - 1, op.div_mul[M2N_MAX_DIMS], op.div_shr[M2N_MAX_DIMS]) : 0;
  const uint32_t nrows = r1 - r0 + 1;
  const bool src_flat = !rows || op.src_stride[0] == (int64_t)inner * 16;
  const bool dst_flat = !rows || op.dst_stride[0] == (int64_t)inner * 16;
  const uint32_t n_store = dst_flat ? 1u : nrows;
  if (n_store > (uint32_t)kMaxPieces) return false;
  const char* src = reinterpret_cast<const char*>(op.src[0]);
  if (lane < op.ndst) m.dst[lane] = op.dst[lane];
  if (lane == 0) {
    m.npieces = n_store;
    m.ndst = op.ndst;
    if (dst_flat) m.dof[0] = (int64_t)u0 * 16, m.off[0] = 0, m.bytes[0] = (u1 - u0) * 16;
  }
  if (!dst_flat) {
    for (uint32_t k = lane; k < nrows; k += 32) {
      const uint32_t row = r0 + k, a = max(u0, row * inner), b = min(u1, (row + 1) * inner);
      m.dof[k] = (int64_t)(a - row * inner) * 16 + (int64_t)row * op.dst_stride[0];
      m.off[k] = (a - u0) * 16;
      m.bytes[k] = (b - a) * 16;
    }
  }
  __syncwarp();
  if (lane == 0) mbar_expect_tx(full, (u1 - u0) * 16);
  __syncwarp();
  if (src_flat) {
    if (lane == 0) bulk_load(buf, src + (int64_t)u0 * 16, (u1 - u0) * 16, full);
  } else {
    for (uint32_t k = lane; k < nrows; k += 32) {
      const uint32_t row = r0 + k, a = max(u0, row * inner), b = min(u1, (row + 1) * inner);
      bulk_load(buf + (a - u0) * 16, src + (int64_t)(a - row * inner) * 16 + (int64_t)row * op.src_stride[0], (b - a) * 16, full);
    }
  }
  return true;
}

__global__ void __launch_bounds__(64, 1)
m2n_bulk_kernel(const __grid_constant__ M2NLaunch args) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_done;
  unsigned char* stage_buf = smem;  // kStages * kStageBytes
  Ring& ring = *reinterpret_cast<Ring*>(smem + kStages * kStageBytes);
  const uint32_t lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    s_done = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ring.full[s], 1);
      mbar_init(&ring.empty[s], 1);
    }
  }
  sched_init(&ring.sched);
  after_previous_kernel();

  if (threadIdx.x < 32) {
    // ---- load warp --------------------------------------------------------------------------------------
    uint32_t tile = blockIdx.x, phase = 0, done = 0, fills = 0, begin = 1, end = 0;
    bool alive = true;
    const auto stage_free = [&]() {  // the stage of the next fill has been read by its previous stores
      return fills < (uint32_t)kStages || mbar_wait(&ring.empty[fills % kStages], (fills / kStages - 1) & 1);
    };
    while (alive) {
      if (lane == 0) sched_request(&ring.sched);
      if (tile < begin || tile >= end) {
        __syncwarp();
        const uint2 tiles = load_op(args, tile, &ring.op);
        begin = tiles.x, end = tiles.y;
        __syncwarp();
      }
      const M2NOp& op = ring.op;
      const uint32_t first = (tile - begin) * op.tile_units, limit = min(op.total_units, first + op.tile_units);
      for (uint32_t u = first; u < limit && alive; u += kStageBytes / 16) {
        const uint32_t s = fills % kStages;
        if (!stage_free()) {
          if (lane == 0) report(args, M2N_TIMEOUT);
          alive = false;
        } else if (!issue_fill(op, u, min(limit, u + kStageBytes / 16), ring.meta[s], stage_buf + (size_t)s * kStageBytes,
                               &ring.full[s], lane)) {
          if (lane == 0) report(args, M2N_BAD_OP);
          alive = false;
        } else {
          ++fills;
        }
      }
      ++done;  // run or given up: see `finish`
      const Take take = sched_take(&ring.sched, phase, tile, args);
      __syncwarp();
      if (gave_up(ring.sched.state, phase)) alive = false;
      phase ^= 1;
      if (!alive) done += take == kTile;  // taken over, but this CTA has stopped
      alive = alive && take == kTile;
    }
    if (stage_free() && lane == 0) {  // end mark
      ring.meta[fills % kStages].npieces = 0;
      mbar_arrive(&ring.full[fills % kStages]);
    }
    if (lane == 0) s_done = done;
  } else {
    // ---- store warp -------------------------------------------------------------------------------------
    for (uint32_t fill = 0;; ++fill) {
      const uint32_t s = fill % kStages;
      if (!mbar_wait(&ring.full[s], (fill / kStages) & 1)) {
        if (lane == 0) report(args, M2N_TIMEOUT);
        break;
      }
      const StageMeta& m = ring.meta[s];
      const uint32_t np = m.npieces;
      if (!np) break;
      const uint32_t n = np * m.ndst;
      for (uint32_t i = lane; i < n; i += 32) {  // piece k of destination j: the lanes walk the (destination, piece) pairs
        const uint32_t j = i / np, k = i - j * np;
        bulk_store(reinterpret_cast<char*>(m.dst[j]) + m.dof[k], stage_buf + (size_t)s * kStageBytes + m.off[k], m.bytes[k]);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      // the stage used one fill earlier may be refilled once its stores have read shared memory
      asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      __syncwarp();
      if (fill && lane == 0) mbar_arrive(&ring.empty[(fill - 1) % kStages]);
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  __syncthreads();
  finish(args, s_done);
}

}  // namespace

int m2n_launch_bulk(const M2NLaunch& args, uint32_t n_tiles, void* stream) {
  static bool configured[64] = {false};
  const size_t smem = (size_t)kStages * kStageBytes + sizeof(Ring);
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(m2n_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) {
      snprintf(etha_err_buf(), ETHA_ERR_LEN, "bulk kernel shared memory opt-in: %s", cudaGetErrorString(e));
      return -(int)e - 1000;
    }
    configured[dev] = true;
  }
  return m2n_launch(m2n_bulk_kernel, n_tiles, 64, smem, stream, args, "bulk");
}
