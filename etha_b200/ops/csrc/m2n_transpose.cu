// Transposing class: boxes whose unit-stride dimension differs on the two sides (a weight kept as [in, out] by one side
// and as [out, in] by the other), bit copies of 2- and 4-byte elements and conversions between fp32, bf16 and fp16.
//
// Bound by HBM if both sides are read and written in whole sectors; element by element in destination order, as the
// general kernel does it, every load touches a sector of its own.  A CTA moves blocks of 64 (destination-contiguous, "a") x
// 256 bytes (source-contiguous, "b") through shared memory: rows of the block are read along b in 16-byte words, each
// thread then collects 8 elements along a for one or two b and stores them as 16 (or 32) bytes; 8 neighbouring threads
// fill 128 (256) contiguous bytes.  The word at (a, w) of the block sits at w ^ 4 * (a / 8 % 8): the 16-byte writes keep
// their shape, and the 8 x 4 words that a warp collects at once lie in 32 different banks.
// A side that is not 16-byte aligned is moved element by element on that side; a block whose destination is not aligned
// is swizzled by w ^ a % 32 instead, since a warp then reads 32 consecutive a of one b.
// [16384, 8192] on one GPU, TB/s read + written, general kernel -> here: bf16 0.40 -> 5.0 to 5.3, fp32 0.79 -> 4.4, fp32 -> bf16
// 0.68 -> 4.1, bf16 with an odd width 0.44 -> 2.5, odd height 0.40 -> 1.8, both 0.44 -> 1.3 ([65536, 8192] bf16: 5.54, with 71 % of the
// issue slots busy and DRAM at 60 % of its peak); 16 wide (1/4 of a block's
// rows used) 0.47 -> 1.59, 8 wide 0.41 -> 0.82.  Five CTAs per SM: four give 5.06 and 4.22, six 4.51 and 4.20.
// At five (48 registers) every instance spills 32 to 64 bytes a thread; at four (64) five of the eight spill nothing, which does
// not make up for the loads in flight.
#include <cuda_runtime.h>

#include <cstdio>

#include "common.h"
#include "m2n_device.cuh"
#include "m2n_launch.h"

namespace {

constexpr int kThreads = 256;
constexpr int kA = M2N_TRANSPOSE_A;                 // block extent along a
constexpr int kRowBytes = M2N_TRANSPOSE_B_BYTES;    // block extent along b, in source bytes
constexpr int kRowWords = kRowBytes / 4;

template <int ES>
struct Uint;
template <>
struct Uint<2> { using T = uint16_t; };
template <>
struct Uint<4> { using T = uint32_t; };

// SDT / DDT: M2N_RAW means a bit copy of ES-byte elements
template <int SDT, int DDT, int ES>
__device__ __forceinline__ void block_move(const M2NOp& op, uint32_t block, uint32_t* tile) {
  using S = typename Uint<ES>::T;
  constexpr int ED = DDT == M2N_RAW ? ES : (DDT == M2N_F32 ? 4 : 2);
  using D = typename Uint<ED>::T;
  constexpr int kB = kRowBytes / ES;
  // block -> (other dims, block of b, block of a); a fastest
  const uint32_t da = op.tr_a, db = op.tr_b;
  const uint32_t na = (op.extent[da] + kA - 1) / kA, nb = (op.extent[db] + kB - 1) / kB;
  const uint32_t ia = block % na, rest = block / na, ib = rest % nb;
  uint32_t outer = rest / nb;
  int64_t so = 0, dof = 0;
#pragma unroll 1
  for (int d = op.ndim - 1; d >= 0; --d) {
    if (d == (int)da || d == (int)db) continue;
    const uint32_t q = outer / op.extent[d], i = outer - q * op.extent[d];
    so += (int64_t)i * op.src_stride[d];
    dof += (int64_t)i * op.dst_stride[d];
    outer = q;
  }
  const uint32_t a0 = ia * kA, b0 = ib * kB;
  const uint32_t an = min((uint32_t)kA, op.extent[da] - a0), bn = min((uint32_t)kB, op.extent[db] - b0);
  const int64_t sa = op.src_stride[da], dd = op.dst_stride[db];  // the strides that are not one element
  const char* src = reinterpret_cast<const char*>(op.src[0]) + so + (int64_t)a0 * sa + (int64_t)b0 * ES;
  dof += (int64_t)b0 * dd + (int64_t)a0 * ED;
  const bool wide_src = op.tr_flags & M2N_TR_SRC16, wide_dst = op.tr_flags & M2N_TR_DST16;
  const auto swz = [&](uint32_t a, uint32_t w) { return a * kRowWords + (wide_dst ? (w ^ ((a >> 3) & 7) * 4) : (w ^ (a & 31))); };

  // ---- source -> shared memory ----------------------------------------------------------------------
  if (wide_src) {
    constexpr int kPerRow = kRowBytes / 16, kTrips = kA * kPerRow / kThreads;
    uint4 v[kTrips];
#pragma unroll
    for (int t = 0; t < kTrips; ++t) {
      const uint32_t i = t * kThreads + threadIdx.x, a = i / kPerRow, x = i % kPerRow;
      // whole words of the row only (the row's end may lie inside a word: those elements are read one by one below)
      if (a < an && (x + 1) * (16 / ES) <= bn) v[t] = ld_stream<uint4>(src + (int64_t)a * sa + x * 16);
    }
#pragma unroll
    for (int t = 0; t < kTrips; ++t) {
      const uint32_t i = t * kThreads + threadIdx.x, a = i / kPerRow, x = i % kPerRow;
      if (a < an && (x + 1) * (16 / ES) <= bn) {
        if (wide_dst) {
          *reinterpret_cast<uint4*>(&tile[swz(a, 4 * x)]) = v[t];
        } else {
          tile[swz(a, 4 * x)] = v[t].x, tile[swz(a, 4 * x + 1)] = v[t].y;
          tile[swz(a, 4 * x + 2)] = v[t].z, tile[swz(a, 4 * x + 3)] = v[t].w;
        }
      }
    }
    const uint32_t done = bn / (16 / ES) * (16 / ES), left = bn - done;
    for (uint32_t i = threadIdx.x; i < an * left; i += kThreads) {
      const uint32_t a = i / left, b = done + i % left;
      reinterpret_cast<S*>(tile)[swz(a, b * ES / 4) * (4 / ES) + b % (4 / ES)] = ld_stream<S>(src + (int64_t)a * sa + b * ES);
    }
  } else {
    constexpr int kTrips = kA * kB / kThreads, kUnroll = 8;
#pragma unroll 1
    for (int t0 = 0; t0 < kTrips; t0 += kUnroll) {
      S v[kUnroll];
#pragma unroll
      for (int t = 0; t < kUnroll; ++t) {
        const uint32_t i = (t0 + t) * kThreads + threadIdx.x, a = i / kB, b = i % kB;
        if (a < an && b < bn) v[t] = ld_stream<S>(src + (int64_t)a * sa + b * ES);
      }
#pragma unroll
      for (int t = 0; t < kUnroll; ++t) {
        const uint32_t i = (t0 + t) * kThreads + threadIdx.x, a = i / kB, b = i % kB;
        if (a < an && b < bn) reinterpret_cast<S*>(tile)[swz(a, b * ES / 4) * (4 / ES) + b % (4 / ES)] = v[t];
      }
    }
  }
  __syncthreads();

  // ---- shared memory -> destination -----------------------------------------------------------------
  const int nd = op.ndst;
  const auto convert = [](S x) -> D {
    if constexpr (DDT == M2N_RAW) {
      return x;
    } else {
      float f;
      if constexpr (SDT == M2N_F32) f = __uint_as_float(x);
      else if constexpr (SDT == M2N_BF16) f = __uint_as_float((uint32_t)x << 16);
      else { __half h; *reinterpret_cast<uint16_t*>(&h) = x; f = __half2float(h); }
      if constexpr (DDT == M2N_F32) {
        return __float_as_uint(f);
      } else if constexpr (DDT == M2N_BF16) {
        const __nv_bfloat16 r = __float2bfloat16_rn(f);
        return *reinterpret_cast<const uint16_t*>(&r);
      } else {
        const __half r = __float2half_rn(f);
        return *reinterpret_cast<const uint16_t*>(&r);
      }
    }
  };
  if (wide_dst) {
    // a thread: 8 consecutive a, the 4 / ES b of one word; the 8 threads next to each other: consecutive a
    constexpr int kPer = 4 / ES, kTrips = (kA / 8) * kRowWords / kThreads;
#pragma unroll 1
    for (int t = 0; t < kTrips; ++t) {
      const uint32_t i = t * kThreads + threadIdx.x, g = i % (kA / 8), w = i / (kA / 8);
      if (g * 8 >= an || w * kPer >= bn) continue;
      uint32_t x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = tile[swz(g * 8 + k, w)];
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        const uint32_t b = w * kPer + p;
        if (b >= bn) continue;
        D y[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) y[k] = convert((S)(ES == 4 ? x[k] : (x[k] >> (16 * p))));
        const int64_t off = dof + (int64_t)b * dd + g * 8 * ED;
        if (g * 8 + 8 <= an) {
          uint4 z[ED / 2];
#pragma unroll
          for (int q = 0; q < ED / 2; ++q) {
            if constexpr (ED == 4) z[q] = make_uint4(y[4 * q], y[4 * q + 1], y[4 * q + 2], y[4 * q + 3]);
            else z[q] = make_uint4(y[0] | (uint32_t)y[1] << 16, y[2] | (uint32_t)y[3] << 16, y[4] | (uint32_t)y[5] << 16, y[6] | (uint32_t)y[7] << 16);
          }
#pragma unroll 1
          for (int j = 0; j < nd; ++j) {
#pragma unroll
            for (int q = 0; q < ED / 2; ++q) st_plain<uint4>(reinterpret_cast<char*>(op.dst[j]) + off + 16 * q, z[q]);
          }
        } else {
#pragma unroll 1
          for (int j = 0; j < nd; ++j) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (g * 8 + k < an) st_plain<D>(reinterpret_cast<char*>(op.dst[j]) + off + k * ED, y[k]);
          }
        }
      }
    }
  } else {
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < (uint32_t)(kA * kB); i += kThreads) {
      const uint32_t a = i % kA, b = i / kA;
      if (a >= an || b >= bn) continue;
      const D y = convert(reinterpret_cast<const S*>(tile)[swz(a, b * ES / 4) * (4 / ES) + b % (4 / ES)]);
      const int64_t off = dof + (int64_t)b * dd + a * ED;
      for (int j = 0; j < nd; ++j) st_plain<D>(reinterpret_cast<char*>(op.dst[j]) + off, y);
    }
  }
  __syncthreads();  // the block may be overwritten
}

template <int SDT, int DDT, int ES>
__global__ void __launch_bounds__(kThreads, 5)
m2n_transpose_kernel(const __grid_constant__ M2NLaunch args) {
  __shared__ M2NOp s_op;
  __shared__ TileSched s_sched;
  __shared__ __align__(16) uint32_t s_tile[kA * kRowWords];
  const uint32_t done = for_each_tile<true>(&s_sched, &s_op, args, [&](const M2NOp& op, uint32_t base, uint32_t limit) {
    // the host only puts ops of this instance into the table; anything else is reported, not executed
    if (!(op.tr_flags & M2N_TR) || (SDT == M2N_RAW ? (op.mode != M2N_MODE_RAW || op.unit_bytes_src != ES)
                                                   : (op.src_dtype != SDT || op.dst_dtype != DDT))) {
      if (threadIdx.x == 0) report(args, M2N_BAD_OP);
      return;
    }
    for (uint32_t b = base; b < limit; ++b) block_move<SDT, DDT, ES>(op, b, s_tile);
  });
  finish(args, done);
}

}  // namespace

extern "C" {

// M2N_KEY_TRANSPOSE | (source dtype << 4) | destination dtype; bit copies: element bytes << 8. 0: not of this class
int etha_op_transpose_key(const M2NOp* op) {
  if (!(op->tr_flags & M2N_TR)) return 0;
  if (op->mode == M2N_MODE_RAW) return M2N_KEY_TRANSPOSE | (op->unit_bytes_src << 8);
  return M2N_KEY_TRANSPOSE | (op->src_dtype << 4) | op->dst_dtype;
}

}  // extern "C"

int m2n_launch_transpose(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream) {
#define CASE(KEY, S, D, ES) \
  case KEY: return m2n_launch(m2n_transpose_kernel<S, D, ES>, n_tiles, kThreads, 0, stream, args, "transposing");
#define CVT(S, D, ES) CASE((S << 4) | D, S, D, ES)
  switch (key & 0xfff) {
    CASE(2 << 8, M2N_RAW, M2N_RAW, 2) CASE(4 << 8, M2N_RAW, M2N_RAW, 4)
    CVT(M2N_F32, M2N_BF16, 4) CVT(M2N_F32, M2N_F16, 4) CVT(M2N_BF16, M2N_F32, 2)
    CVT(M2N_BF16, M2N_F16, 2) CVT(M2N_F16, M2N_F32, 2) CVT(M2N_F16, M2N_BF16, 2)
    default: return m2n_no_instance("transposing", key);
  }
#undef CVT
#undef CASE
}
