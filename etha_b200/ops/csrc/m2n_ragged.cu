// Ragged class: boxes whose rows are long runs on both sides but start anywhere (odd vocabularies and widths, uneven
// shards, views), and boxes with two or more strided dims: bit copies, conversions and Partial collapses.
//
// Meant to be bound by HBM, and not quite: a bit copy of 801 of 1601 bf16 columns keeps the issue slots 56 % and L1 68 %
// busy and DRAM at 52 % of its peak.  The widest unit such a box divides into is one element, so one load and one
// store instruction per element would be issued.  Here a row is cut into chunks of 32 destination bytes (bit copies) or 8
// elements (typed ops) that start on a 16-byte boundary of the DESTINATION: a chunk is stored with 16-byte stores, and its
// source bytes, which start at any offset, are read as the aligned 16-byte words that hold them and shifted into place
// with funnel shifts.  Only the first and the last chunk of a row are partial; they are stored in pieces.  Only words that
// hold at least one byte of the row are read, so no read leaves the 16-byte granule of a valid byte (and with it the
// page); bytes next to the row are discarded.  Neighbouring chunks share a word, which the second reader finds in L1.
// Arithmetic of the typed ops is the general kernel's: fp32 accumulation in source order, "avg" divides by the group
// size, one rounding to the source dtype when the destination dtype differs, then conversion.
#include <cuda_runtime.h>

#include <cstdio>
#include <type_traits>

#include "common.h"
#include "m2n_device.cuh"
#include "m2n_launch.h"

namespace {

constexpr int kRaggedThreads = 256;
constexpr int kRawChunk = M2N_RAGGED_BYTES;

// CTAs per SM and chunks in flight per thread, as far as the registers go without spills.  Measured on one GPU (read +
// written): 131072 rows of 801 of 1601 bf16 columns 5.03 TB/s with 5 CTAs and two chunks (6 x 1: 4.80, 3 x 3: 3.87; chunks of 16 bytes: 4.63
// at best; 5.45 with 335000 rows; another GPU 4.8), the same columns fp32 -> bf16 5.6 (general kernel, element by element: 0.66 and 1.03).
template <int SDT, bool REDUCE>
constexpr int kRaggedCtas = SDT == M2N_RAW ? 5 : (REDUCE ? 2 : 3);
constexpr int kRaggedUnroll = 2;

__device__ __forceinline__ uint4 ld_word(const char* p) {  // aligned 16 bytes, kept in L1 for the neighbouring chunk
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(__cvta_generic_to_global(p)));
  return v;
}

// byte offsets of row `row` of the op in the source and the destination
__device__ __forceinline__ void row_offsets(const M2NOp& op, uint32_t row, int64_t& so, int64_t& dof) {
  so = dof = 0;
  const int nd = op.ndim;
  if (nd == 1) {
    so = (int64_t)row * op.src_stride[0];
    dof = (int64_t)row * op.dst_stride[0];
    return;
  }
#pragma unroll 1
  for (int d = nd - 1; d >= 0; --d) {
    const uint32_t q = d == 0 ? 0u : fast_div(row, op.div_mul[d], op.div_shr[d]);
    const uint32_t i = row - q * op.extent[d];
    so += (int64_t)i * op.src_stride[d];
    dof += (int64_t)i * op.dst_stride[d];
    row = q;
  }
}

// N bytes of a row, not aligned: the aligned words that hold them.  Words without a byte of the row are replaced by its
// nearest word, so that every load is unconditional and none leaves the row's words.
template <int N>
struct Window {
  static constexpr int W = N / 16 + 1;
  uint4 w[W];
  // `row`: first byte of the row, `first` / `last`: where its first and its last word start, relative to it, `off`: first
  // byte wanted
  __device__ __forceinline__ void load(const char* row, int first, int last, int off) {
    const int at = off - ((off - first) & 15);
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = ld_word(row + min(max(at + 16 * i, first), last));
  }
  // the N bytes, `k`: where the first one is in its word
  __device__ __forceinline__ void get(int k, uint32_t (&out)[N / 4]) const {
    uint32_t r[4 * W];
#pragma unroll
    for (int i = 0; i < W; ++i) r[4 * i] = w[i].x, r[4 * i + 1] = w[i].y, r[4 * i + 2] = w[i].z, r[4 * i + 3] = w[i].w;
    const bool two = k & 8, one = k & 4;
#pragma unroll
    for (int j = 0; j < 4 * W - 2; ++j) r[j] = two ? r[j + 2] : r[j];
#pragma unroll
    for (int j = 0; j < N / 4 + 1; ++j) r[j] = one ? r[j + 1] : r[j];
    const uint32_t bits = (k & 3) * 8;
#pragma unroll
    for (int j = 0; j < N / 4; ++j) out[j] = __funnelshift_r(r[j], r[j + 1], bits);
  }
};

// bytes [lo, hi) of the 16-byte aligned word at `p`
__device__ __forceinline__ void store_part(char* p, const uint32_t (&v)[4], int lo, int hi) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (4 * j >= lo && 4 * j + 4 <= hi) {
      st_plain<uint32_t>(p + 4 * j, v[j]);
    } else if (4 * j + 4 > lo && 4 * j < hi) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int b = 4 * j + 2 * h;
        if (b >= lo && b + 2 <= hi) {
          st_plain<uint16_t>(p + b, (uint16_t)(v[j] >> (16 * h)));
        } else {
          if (b >= lo && b < hi) st_plain<uint8_t>(p + b, (uint8_t)(v[j] >> (16 * h)));
          if (b + 1 >= lo && b + 1 < hi) st_plain<uint8_t>(p + b + 1, (uint8_t)(v[j] >> (16 * h + 8)));
        }
      }
    }
  }
}

__device__ __forceinline__ void store_word(char* p, const uint32_t (&v)[4], int lo, int hi) {
  if (lo <= 0 && hi >= 16) st_plain<uint4>(p, make_uint4(v[0], v[1], v[2], v[3]));
  else store_part(p, v, lo, hi);
}

// ---- bit copies -------------------------------------------------------------------------------------------------
template <int U>
__device__ __forceinline__ void raw_trip(const M2NOp& op, uint32_t chunk0) {
  Window<kRawChunk> win[U];
  int64_t dof[U];  // of the chunk's first byte
  int e0[U], k[U];
  const int row_bytes = (int)(op.inner_units * op.unit_bytes_dst);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t chunk = chunk0 + u * kRaggedThreads;
    const uint32_t row = fast_div(chunk, op.chunk_mul, op.chunk_shr);
    int64_t so;
    row_offsets(op, row, so, dof[u]);
    e0[u] = (int)((chunk - row * op.chunk_row) * kRawChunk) - (int)((uint32_t)(op.dst[0] + dof[u]) & 15);
    dof[u] += e0[u];
    const char* s = reinterpret_cast<const char*>(op.src[0]) + so;
    const int mis = (int)((uint32_t)(uint64_t)s & 15);
    win[u].load(s, -mis, ((mis + row_bytes - 1) & ~15) - mis, e0[u]);
    k[u] = (e0[u] + mis) & 15;
  }
  const int nd = op.ndst;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int lo = -e0[u], hi = row_bytes - e0[u];  // valid bytes of the chunk; none if hi <= 0
    uint32_t v[kRawChunk / 4];
    win[u].get(k[u], v);
#pragma unroll 1
    for (int j = 0; j < nd; ++j) {
      char* d = reinterpret_cast<char*>(op.dst[j]) + dof[u];
#pragma unroll
      for (int w = 0; w < kRawChunk; w += 16) {
        const uint32_t x[4] = {v[w / 4], v[w / 4 + 1], v[w / 4 + 2], v[w / 4 + 3]};
        store_word(d + w, x, lo - w, hi - w);
      }
    }
  }
}

// ---- typed ops --------------------------------------------------------------------------------------------------
template <int DT>
__device__ __forceinline__ void decode_words(const uint32_t (&r)[DT == M2N_F32 ? 8 : 4], float (&f)[8]) {
  if constexpr (DT == M2N_F32) {
    const uint4 a[2] = {make_uint4(r[0], r[1], r[2], r[3]), make_uint4(r[4], r[5], r[6], r[7])};
    Elem<DT>::decode(a, f);
  } else {
    const uint4 a[1] = {make_uint4(r[0], r[1], r[2], r[3])};
    Elem<DT>::decode(a, f);
  }
}

template <int SDT, int DDT, int U, bool REDUCE>
__device__ __forceinline__ void typed_trip(const M2NOp& op, uint32_t chunk0) {
  constexpr int ES = SDT == M2N_F32 ? 4 : 2, ED = DDT == M2N_F32 ? 4 : 2;
  int64_t so[U], dof[U];
  int e0[U];  // first element of the chunk, from the start of the row
  const int inner = (int)(op.inner_units * op.unit_elems);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t chunk = chunk0 + u * kRaggedThreads;
    const uint32_t row = fast_div(chunk, op.chunk_mul, op.chunk_shr);
    row_offsets(op, row, so[u], dof[u]);
    const int head = (int)((0 - (op.dst[0] + dof[u])) & 15) / ED;  // elements before the first 16-byte boundary
    e0[u] = (int)((chunk - row * op.chunk_row) * 8) - (head ? 8 - head : 0);
    dof[u] += (int64_t)e0[u] * ED;
  }
  float acc[U][8], grp[U][8];
  const int n = REDUCE ? op.nsrc : 1, s0 = op.red_size[0];
  const int op0 = op.red_op[0], op1 = op.red_op[1];
  int in_group = 0;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    Window<8 * ES> win[U];
    int k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const char* s = reinterpret_cast<const char*>(op.src[i]) + so[u];
      const int mis = (int)((uint32_t)(uint64_t)s & 15);
      win[u].load(s, -mis, ((mis + inner * ES - 1) & ~15) - mis, e0[u] * ES);
      k[u] = (e0[u] * ES + mis) & 15;
    }
    const bool closes = !REDUCE || in_group + 1 == s0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      uint32_t r[8 * ES / 4];
      win[u].get(k[u], r);
      float f[8];
      decode_words<SDT>(r, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if constexpr (!REDUCE) {
          acc[u][e] = f[e];
        } else {
          float g = in_group == 0 ? f[e] : reduce2(grp[u][e], f[e], op0);
          if (closes) {
            if (op0 == M2N_AVG) g = __fdiv_rn(g, (float)s0);
            acc[u][e] = i + 1 == s0 ? g : reduce2(acc[u][e], g, op1);
          }
          grp[u][e] = g;
        }
      }
    }
    in_group = closes ? 0 : in_group + 1;
  }
  const int s1 = op.red_size[1], nd = op.ndst;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int lo = -e0[u] * ED, hi = (inner - e0[u]) * ED;  // valid bytes of the chunk
    if constexpr (REDUCE) {
      if (op1 == M2N_AVG && s1 > 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[u][e] = __fdiv_rn(acc[u][e], (float)s1);
      }
      if constexpr (SDT != DDT) {
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[u][e] = round_through<SDT>(acc[u][e]);
      }
    }
    uint32_t v[2][4];
    if constexpr (DDT == M2N_F32) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e >> 2][e & 3] = __float_as_uint(acc[u][e]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) v[0][e] = Elem<DDT>::pack(acc[u][2 * e], acc[u][2 * e + 1]);
    }
#pragma unroll 1
    for (int j = 0; j < nd; ++j) {
      char* d = reinterpret_cast<char*>(op.dst[j]) + dof[u];
      store_word(d, v[0], lo, hi);
      if constexpr (DDT == M2N_F32) store_word(d + 16, v[1], lo - 16, hi - 16);
    }
  }
}

template <int SDT, int DDT, bool REDUCE>
__global__ void __launch_bounds__(kRaggedThreads, kRaggedCtas<SDT, REDUCE>)
m2n_ragged_kernel(const __grid_constant__ M2NLaunch args) {
  __shared__ M2NOp s_op;
  __shared__ TileSched s_sched;
  constexpr int U = kRaggedUnroll;
  constexpr int kMode = SDT == M2N_RAW ? M2N_MODE_RAW : (REDUCE ? M2N_MODE_REDUCE : M2N_MODE_CVT);
  const uint32_t done = for_each_tile<true>(&s_sched, &s_op, args, [&](const M2NOp& op, uint32_t base, uint32_t limit) {
    // the host only puts ops of this instance into the table; anything else is reported, not executed
    if (!op.chunks || op.mode != kMode || (SDT != M2N_RAW && (op.src_dtype != SDT || op.dst_dtype != DDT))) {
      if (threadIdx.x == 0) report(args, M2N_BAD_OP);
      return;
    }
    const auto trip = [&](auto units, uint32_t chunk0) {
      if constexpr (SDT == M2N_RAW) raw_trip<decltype(units)::value>(op, chunk0);
      else typed_trip<SDT, DDT, decltype(units)::value, REDUCE>(op, chunk0);
    };
    uint32_t b = base;
#pragma unroll 1
    for (; b + kRaggedThreads * U <= limit; b += kRaggedThreads * U) trip(std::integral_constant<int, U>(), b + threadIdx.x);
#pragma unroll 1
    for (b += threadIdx.x; b < limit; b += kRaggedThreads) trip(std::integral_constant<int, 1>(), b);
  });
  finish(args, done);
}

}  // namespace

extern "C" {

// M2N_KEY_RAGGED | (collapse << 8) | (source dtype << 4) | destination dtype (0 and 0: bit copy), or 0 when the op is not
// of this class
int etha_op_ragged_key(const M2NOp* op) {
  if (!op->chunks || op->tr_flags) return 0;
  if (op->mode == M2N_MODE_RAW) return M2N_KEY_RAGGED;
  return M2N_KEY_RAGGED | ((op->mode == M2N_MODE_REDUCE) << 8) | (op->src_dtype << 4) | op->dst_dtype;
}

}  // extern "C"

int m2n_launch_ragged(const M2NLaunch& args, int key, uint32_t n_tiles, void* stream) {
#define CASE(S, D, R) \
  case (R << 8) | (S << 4) | D: return m2n_launch(m2n_ragged_kernel<S, D, R>, n_tiles, kRaggedThreads, 0, stream, args, "ragged");
  switch (key & 0x1ff) {
    CASE(M2N_RAW, M2N_RAW, 0)
    CASE(M2N_F32, M2N_BF16, 0) CASE(M2N_F32, M2N_F16, 0) CASE(M2N_BF16, M2N_F32, 0)
    CASE(M2N_BF16, M2N_F16, 0) CASE(M2N_F16, M2N_F32, 0) CASE(M2N_F16, M2N_BF16, 0)
    CASE(M2N_F32, M2N_F32, 1) CASE(M2N_F32, M2N_BF16, 1) CASE(M2N_F32, M2N_F16, 1)
    CASE(M2N_BF16, M2N_F32, 1) CASE(M2N_BF16, M2N_BF16, 1) CASE(M2N_BF16, M2N_F16, 1)
    CASE(M2N_F16, M2N_F32, 1) CASE(M2N_F16, M2N_BF16, 1) CASE(M2N_F16, M2N_F16, 1)
    default: return m2n_no_instance("ragged", key);
  }
#undef CASE
}
