// Streaming class of the typed ops: dtype conversion and single-level Partial collapse of 2 or 4 sources over
// boxes that are one run or the rows of a matrix, in 8-element units (16-byte aligned on every side).
//
// One kernel instance per (source dtype, destination dtype, number of sources): no dtype or source-count
// branch is left inside the loop, the box arithmetic is the one-run / matrix-row form, and every load a thread
// needs for its `kUnits` units (all sources of all units, 128 bytes per thread) is issued before the first value
// is used, so that a Partial collapse whose other contributors live on peer GPUs keeps enough bytes in flight to
// cover the NVLink round trip.  Two 256-thread CTAs per SM (up to 128 registers per thread: no spills); tiles are taken
// dynamically (see TileSched).  1 GiB of bf16 results on one GPU, read + written: fp32 -> bf16 6.88 TB/s, two bf16 sources
// 6.90, four 6.76 (with fixed shares of 64 KiB tiles 6.57, 5.90 and 6.19).
// Arithmetic is the same as the general kernel's: fp32 accumulation in source order, "avg" divides by the
// number of sources, one rounding to the source dtype when the destination dtype differs, then conversion.
//
// Replaces, for these shapes, the reference's contiguous()/clone()/all_reduce/to() chain per chunk
// (src/etha/comm/ir.py:101-132).
#include <cuda_runtime.h>

#include <cstdio>

#include "common.h"
#include "m2n_device.cuh"
#include "m2n_launch.h"

namespace {

#ifndef ETHA_STREAM_THREADS
#define ETHA_STREAM_THREADS 256
#endif
#ifndef ETHA_STREAM_CTAS
#define ETHA_STREAM_CTAS 2
#endif
constexpr int kTypedThreads = ETHA_STREAM_THREADS;
constexpr int kTypedCtasPerSm = ETHA_STREAM_CTAS;

template <int SDT, int NSRC>
struct Plan {
  static constexpr int W = Elem<SDT>::W;                       // 16-byte words per unit and source
  static constexpr int kRaw = 8;                               // 16-byte words in flight per thread
  static constexpr int kUnits = (kRaw / (W * NSRC)) > 4 ? 4 : ((kRaw / (W * NSRC)) < 1 ? 1 : kRaw / (W * NSRC));
};

// U units of one thread, kTypedThreads apart, the first one `unit0`
template <int SDT, int DDT, int NSRC, int ND, int U>
__device__ __forceinline__ void stream_trip(const M2NOp& op, uint32_t unit0) {
  uint4 raw[U][NSRC][Elem<SDT>::W];
  int64_t dof[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    int64_t so;
    unit_offsets<ND>(op, unit0 + u * kTypedThreads, so, dof[u]);
#pragma unroll
    for (int i = 0; i < NSRC; ++i) Elem<SDT>::load_raw(reinterpret_cast<const char*>(op.src[i]) + so, raw[u][i]);
  }
  const int rop = op.red_op[0];
  const bool mc = op.flags & M2N_FLAG_MULTIMEM;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float acc[8];
    Elem<SDT>::decode(raw[u][0], acc);
    if constexpr (NSRC > 1) {
#pragma unroll
      for (int i = 1; i < NSRC; ++i) {
        float f[8];
        Elem<SDT>::decode(raw[u][i], f);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = reduce2(acc[k], f[k], rop);
      }
      if (rop == M2N_AVG) {
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = __fdiv_rn(acc[k], (float)NSRC);
      }
      if constexpr (SDT != DDT) {
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = round_through<SDT>(acc[k]);
      }
    }
    const int nd = op.ndst;
#pragma unroll 1
    for (int j = 0; j < nd; ++j) store8_to<DDT>(reinterpret_cast<char*>(op.dst[j]) + dof[u], acc, mc);
  }
}

template <int SDT, int DDT, int NSRC, int ND>
__device__ __forceinline__ void stream_tile(const M2NOp& op, uint32_t base, uint32_t limit) {
  constexpr int U = Plan<SDT, NSRC>::kUnits;
  uint32_t b = base;
#pragma unroll 1
  for (; b + kTypedThreads * U <= limit; b += kTypedThreads * U) stream_trip<SDT, DDT, NSRC, ND, U>(op, b + threadIdx.x);
#pragma unroll 1
  for (b += threadIdx.x; b < limit; b += kTypedThreads) stream_trip<SDT, DDT, NSRC, ND, 1>(op, b);
}

template <int SDT, int DDT, int NSRC>
__global__ void __launch_bounds__(kTypedThreads, kTypedCtasPerSm)
m2n_typed_kernel(const __grid_constant__ M2NLaunch args) {
  __shared__ M2NOp s_op;
  __shared__ TileSched s_sched;
  const uint32_t done = for_each_tile(&s_sched, &s_op, args, [&](const M2NOp& op, uint32_t base, uint32_t limit) {
    // the host only puts ops of this instance's key into the table; anything else is reported, not executed
    if (op.src_dtype != SDT || op.dst_dtype != DDT || op.nsrc != NSRC || op.unit_elems != 8 || op.ndim > 1) {
      if (threadIdx.x == 0) report(args, M2N_BAD_OP);
      return;
    }
    if (op.ndim == 0) stream_tile<SDT, DDT, NSRC, 0>(op, base, limit);
    else stream_tile<SDT, DDT, NSRC, 1>(op, base, limit);
  });
  finish(args, done);
}

// Collapses without an instance of their own (3 or 5 to 8 sources, two levels, the two 16-bit types mixed): one kernel per
// dtype pair, for one and for two levels.  The sources are read four at a time, all loads of the four issued before the
// first value is used, which is what the general kernel lacks: it reads one source after the other.  128 MiB per source on
// one GPU, TB/s read + written, general kernel -> here: sum of 3 bf16 2.4 -> 5.1, 8 bf16 3.9 -> 6.1, 8 fp32 2.9 -> 6.4, 2 x 2
// bf16 1.8 -> 4.5, 2 x 4 fp32 1.9 -> 5.6, maximum of 8 bf16 (bound by the comparisons) 3.2 -> 3.6.  Two CTAs per SM: three
// spill and reach 5.0, 6.0, 4.3, 3.5, 3.3.  Two levels keep a group and the total: those instances spill 52 to 108 bytes a thread at
// two CTAs as well.
constexpr int kSlots = 4;

template <int SDT, int DDT, bool TWO, int U>
__device__ __forceinline__ void collapse_trip(const M2NOp& op, uint32_t unit0) {
  int64_t so[U], dof[U];
#pragma unroll
  for (int u = 0; u < U; ++u) unit_offsets<1>(op, unit0 + u * kTypedThreads, so[u], dof[u]);
  const int n = op.nsrc, s0 = op.red_size[0], op0 = op.red_op[0];
  float acc[U][8], grp[U][8];
  int at = 0;  // sources in the open group of a two-level collapse
#pragma unroll 1
  for (int first = 0; first < n; first += kSlots) {
    uint4 raw[U][kSlots][Elem<SDT>::W];
#pragma unroll
    for (int i = 0; i < kSlots; ++i) {
      if (first + i < n) {
        const char* src = reinterpret_cast<const char*>(op.src[first + i]);
#pragma unroll
        for (int u = 0; u < U; ++u) Elem<SDT>::load_raw(src + so[u], raw[u][i]);
      }
    }
#pragma unroll
    for (int i = 0; i < kSlots; ++i) {
      if (first + i < n) {
        const bool closes = TWO && at + 1 == s0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float f[8];
          Elem<SDT>::decode(raw[u][i], f);
          if constexpr (!TWO) {
            if (i == 0 && first == 0) {
#pragma unroll
              for (int k = 0; k < 8; ++k) acc[u][k] = f[k];
            } else {
              reduce8(acc[u], f, op0);
            }
          } else {
            if (at == 0) {
#pragma unroll
              for (int k = 0; k < 8; ++k) grp[u][k] = f[k];
            } else {
              reduce8(grp[u], f, op0);
            }
            if (closes) {
              if (op0 == M2N_AVG) {
#pragma unroll
                for (int k = 0; k < 8; ++k) grp[u][k] = __fdiv_rn(grp[u][k], (float)s0);
              }
              if (first + i + 1 == s0) {
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[u][k] = grp[u][k];
              } else {
                reduce8(acc[u], grp[u], op.red_op[1]);
              }
            }
          }
        }
        if (TWO) at = closes ? 0 : at + 1;
      }
    }
  }
  const int groups = TWO ? op.red_size[1] : s0, last_op = TWO ? op.red_op[1] : op0;
  const bool mc = op.flags & M2N_FLAG_MULTIMEM;
  const int nd = op.ndst;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (last_op == M2N_AVG) {
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[u][k] = __fdiv_rn(acc[u][k], (float)groups);
    }
    if constexpr (SDT != DDT) {
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[u][k] = round_through<SDT>(acc[u][k]);
    }
#pragma unroll 1
    for (int j = 0; j < nd; ++j) store8_to<DDT>(reinterpret_cast<char*>(op.dst[j]) + dof[u], acc[u], mc);
  }
}

template <int SDT, int DDT, bool TWO>
__global__ void __launch_bounds__(kTypedThreads, kTypedCtasPerSm)
m2n_collapse_kernel(const __grid_constant__ M2NLaunch args) {
  __shared__ M2NOp s_op;
  __shared__ TileSched s_sched;
  const uint32_t done = for_each_tile(&s_sched, &s_op, args, [&](const M2NOp& op, uint32_t base, uint32_t limit) {
    if (op.mode != M2N_MODE_REDUCE || op.src_dtype != SDT || op.dst_dtype != DDT || op.unit_elems != 8 || op.ndim > 1 ||
        (op.red_size[1] > 1) != TWO) {
      if (threadIdx.x == 0) report(args, M2N_BAD_OP);
      return;
    }
    // a single run is a matrix of one row: its row index and its strides are 0
    constexpr int U = 8 / (kSlots * Elem<SDT>::W);  // eight 16-byte words in flight per thread
    uint32_t b = base;
#pragma unroll 1
    for (; b + kTypedThreads * U <= limit; b += kTypedThreads * U) collapse_trip<SDT, DDT, TWO, U>(op, b + threadIdx.x);
#pragma unroll 1
    for (b += threadIdx.x; b < limit; b += kTypedThreads) collapse_trip<SDT, DDT, TWO, 1>(op, b);
  });
  finish(args, done);
}

constexpr bool typed(int dt) { return dt == M2N_F32 || dt == M2N_BF16 || dt == M2N_F16; }

// combinations with a kernel instance: conversions between any two of fp32/bf16/fp16; collapses of 2 or 4
// sources whose destination dtype equals the source dtype or where one of the two is fp32
constexpr bool has_instance(int s, int d, int n) {
  if (!typed(s) || !typed(d)) return false;
  if (n == 1) return s != d;
  if (n != 2 && n != 4) return false;
  return s == d || s == M2N_F32 || d == M2N_F32;
}

template <int S, int D, int N>
int launch(const M2NLaunch& args, uint32_t grid, void* stream) {
  if constexpr (has_instance(S, D, N)) return m2n_launch(m2n_typed_kernel<S, D, N>, grid, kTypedThreads, 0, stream, args, "typed");
  else return m2n_no_instance("streaming", (S << 8) | (D << 4) | N);
}

}  // namespace

extern "C" {

// Key of the streaming instance that can run `op`: (src dtype << 8) | (dst dtype << 4) | sources, or 0 when the
// op has to stay in the general kernel.
int etha_op_stream_key(const M2NOp* op) {
  if (op->unit_elems != 8 || op->ndim > 1 || op->total_units == 0) return 0;
  if (op->mode == M2N_MODE_CVT) {
    if (op->nsrc != 1 || !has_instance(op->src_dtype, op->dst_dtype, 1)) return 0;
  } else if (op->mode == M2N_MODE_REDUCE) {
    if (op->red_size[1] != 1 || op->red_size[0] != op->nsrc || !has_instance(op->src_dtype, op->dst_dtype, op->nsrc)) return 0;
  } else {
    return 0;
  }
  return (op->src_dtype << 8) | (op->dst_dtype << 4) | op->nsrc;
}

// M2N_KEY_COLLAPSE | (two levels << 8) | (src dtype << 4) | dst dtype of the collapse instance that can run `op`, or 0
int etha_op_collapse_key(const M2NOp* op) {
  if (op->mode != M2N_MODE_REDUCE || op->unit_elems != 8 || op->ndim > 1 || op->total_units == 0) return 0;
  if (op->nsrc > 8 || op->red_size[0] * op->red_size[1] != op->nsrc) return 0;
  return M2N_KEY_COLLAPSE | ((op->red_size[1] > 1) << 8) | (op->src_dtype << 4) | op->dst_dtype;
}

}  // extern "C"

int m2n_launch_collapse(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream) {
#define CASE_N(S, D, N) \
  case (N << 8) | (S << 4) | D: return m2n_launch(m2n_collapse_kernel<S, D, N>, n_tiles, kTypedThreads, 0, stream, args, "collapse");
#define CASE(S, D) CASE_N(S, D, 0) CASE_N(S, D, 1)
  switch (key & 0xfff) {
    CASE(M2N_F32, M2N_F32) CASE(M2N_F32, M2N_BF16) CASE(M2N_F32, M2N_F16)
    CASE(M2N_BF16, M2N_F32) CASE(M2N_BF16, M2N_BF16) CASE(M2N_BF16, M2N_F16)
    CASE(M2N_F16, M2N_F32) CASE(M2N_F16, M2N_BF16) CASE(M2N_F16, M2N_F16)
    default: return m2n_no_instance("collapse", key);
  }
#undef CASE
#undef CASE_N
}

int m2n_launch_typed(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream) {
#define CASE_N(S, D, N) case (S << 8) | (D << 4) | N: return launch<S, D, N>(args, n_tiles, stream);
#define CASE(S, D) CASE_N(S, D, 1) CASE_N(S, D, 2) CASE_N(S, D, 4)
  switch (key) {
    CASE(M2N_F32, M2N_F32) CASE(M2N_F32, M2N_BF16) CASE(M2N_F32, M2N_F16)
    CASE(M2N_BF16, M2N_F32) CASE(M2N_BF16, M2N_BF16) CASE(M2N_BF16, M2N_F16)
    CASE(M2N_F16, M2N_F32) CASE(M2N_F16, M2N_BF16) CASE(M2N_F16, M2N_F16)
    default: return m2n_no_instance("streaming", key);
  }
#undef CASE
#undef CASE_N
}
