// sm_100a kernels of the M-to-N redistribution: strided gather -> (convert | reduce) -> strided
// scatter into local, peer or multicast memory, plus the release/acquire flag kernels.
//
// A launch walks a device-resident table of `M2NOp`s (see m2n.h).  The table is built
// once per registered batch and launched once per transfer, so a transfer costs no host work per
// chunk and no staging buffer: the producer GPU reads its own memory and stores straight into the
// consumers' slices over NVLink.  This replaces the reference's per-chunk slice/contiguous/cast/
// pack kernels and its NCCL send/recv/broadcast/all-reduce calls (src/etha/comm/ir.py:101-141,
// 229-310; src/etha/comm/transfer.py:20-41).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <type_traits>

#include "common.h"
#include "m2n_device.cuh"
#include "m2n_launch.h"

namespace {

// ---------------------------------------------------------------------------------------------
// tile bodies
// ---------------------------------------------------------------------------------------------
template <typename V, int UNROLL, int ND>
__device__ __forceinline__ void tile_raw(const M2NOp& op, uint32_t base, uint32_t limit) {
  V v[UNROLL];
  int64_t doff[UNROLL];
  bool ok[UNROLL];
  const char* src = reinterpret_cast<const char*>(op.src[0]);
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    uint32_t unit = base + u * blockDim.x + threadIdx.x;
    ok[u] = unit < limit;
    if (ok[u]) {
      int64_t so;
      unit_offsets<ND>(op, unit, so, doff[u]);
      v[u] = ld_stream<V>(src + so);
    }
  }
  const int nd = op.ndst;
  if constexpr (std::is_same<V, uint4>::value) {
    if (op.flags & M2N_FLAG_MULTIMEM) {
#pragma unroll
      for (int u = 0; u < UNROLL; ++u)
        if (ok[u]) st_multimem16(reinterpret_cast<char*>(op.dst[0]) + doff[u], v[u]);
      return;
    }
  }
  for (int j = 0; j < nd; ++j) {
    char* dst = reinterpret_cast<char*>(op.dst[j]);
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (ok[u]) st_plain<V>(dst + doff[u], v[u]);
  }
}

template <int SDT, int DDT, int UNROLL, int ND = -1>
__device__ __forceinline__ void tile_cvt8(const M2NOp& op, uint32_t base, uint32_t limit) {
  // all loads of the thread are issued before the first store, so UNROLL * 16..32 bytes are in flight per thread
  const char* src = reinterpret_cast<const char*>(op.src[0]);
  uint4 raw[UNROLL][Elem<SDT>::W];
  int64_t doff[UNROLL];
  bool ok[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    uint32_t unit = base + u * blockDim.x + threadIdx.x;
    ok[u] = unit < limit;
    if (ok[u]) {
      int64_t so;
      unit_offsets<ND>(op, unit, so, doff[u]);
      Elem<SDT>::load_raw(src + so, raw[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    if (ok[u]) {
      float f[8];
      Elem<SDT>::decode(raw[u], f);
      const bool mc = op.flags & M2N_FLAG_MULTIMEM;
      for (int j = 0; j < op.ndst; ++j) store8_to<DDT>(reinterpret_cast<char*>(op.dst[j]) + doff[u], f, mc);
    }
  }
}

// Single-level Partial collapse of exactly NSRC sources, 8 elements per unit: every source word of the unit is
// requested before the first one is used.
template <int SDT, int DDT, int NSRC, int ND = -1>
__device__ __forceinline__ void tile_reduce_flat(const M2NOp& op, uint32_t base, uint32_t limit, int unroll) {
  const int rop = op.red_op[0];
  for (int u = 0; u < unroll; ++u) {
    uint32_t unit = base + u * blockDim.x + threadIdx.x;
    if (unit >= limit) continue;
    int64_t so, dof;
    unit_offsets<ND>(op, unit, so, dof);
    uint4 raw[NSRC][Elem<SDT>::W];
#pragma unroll
    for (int i = 0; i < NSRC; ++i) Elem<SDT>::load_raw(reinterpret_cast<const char*>(op.src[i]) + so, raw[i]);
    float acc[8];
    Elem<SDT>::decode(raw[0], acc);
#pragma unroll
    for (int i = 1; i < NSRC; ++i) {
      float f[8];
      Elem<SDT>::decode(raw[i], f);
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
    const bool mc = op.flags & M2N_FLAG_MULTIMEM;
    for (int j = 0; j < op.ndst; ++j) store8_to<DDT>(reinterpret_cast<char*>(op.dst[j]) + dof, acc, mc);
  }
}

template <int SDT, int DDT, int UNROLL>
__device__ __forceinline__ void tile_cvt1(const M2NOp& op, uint32_t base, uint32_t limit) {
  const char* src = reinterpret_cast<const char*>(op.src[0]);
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    uint32_t unit = base + u * blockDim.x + threadIdx.x;
    if (unit < limit) {
      int64_t so, dof;
      unit_offsets(op, unit, so, dof);
      float f = Elem<SDT>::load1(src + so);
      for (int j = 0; j < op.ndst; ++j) Elem<DDT>::store1(reinterpret_cast<char*>(op.dst[j]) + dof, f);
    }
  }
}

// Partial collapse: level 0 groups of red_size[0] consecutive sources, then level 1 over the group results;
// fp32 accumulation in ascending source order, "avg" divides by the group size.  The collapsed value is
// rounded once to the SOURCE dtype (the dtype a Partial -> Replicate redistribution yields) and then converted
// to the destination dtype, so a two-way sum is bit-identical to an all-reduce in the source dtype.
template <int SDT, int DDT, int N>
__device__ __forceinline__ void tile_reduce(const M2NOp& op, uint32_t base, uint32_t limit, int unroll) {
  const int s0 = op.red_size[0], s1 = op.red_size[1];
  const int op0 = op.red_op[0], op1 = op.red_op[1];
  for (int u = 0; u < unroll; ++u) {
    uint32_t unit = base + u * blockDim.x + threadIdx.x;
    if (unit >= limit) continue;
    int64_t so, dof;
    unit_offsets(op, unit, so, dof);
    float acc[N];
    for (int g = 0; g < s1; ++g) {
      float a[N];
      for (int i = 0; i < s0; ++i) {
        const char* p = reinterpret_cast<const char*>(op.src[g * s0 + i]) + so;
        float f[N];
        if constexpr (N == 8) {
          Elem<SDT>::load8(p, f);
        } else {
          f[0] = Elem<SDT>::load1(p);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) a[k] = (i == 0) ? f[k] : reduce2(a[k], f[k], op0);
      }
      if (op0 == M2N_AVG) {
#pragma unroll
        for (int k = 0; k < N; ++k) a[k] = __fdiv_rn(a[k], (float)s0);
      }
#pragma unroll
      for (int k = 0; k < N; ++k) acc[k] = (g == 0) ? a[k] : reduce2(acc[k], a[k], op1);
    }
    if (op1 == M2N_AVG && s1 > 1) {
#pragma unroll
      for (int k = 0; k < N; ++k) acc[k] = __fdiv_rn(acc[k], (float)s1);
    }
    if constexpr (SDT != DDT) {
#pragma unroll
      for (int k = 0; k < N; ++k) acc[k] = round_through<SDT>(acc[k]);
    }
    for (int j = 0; j < op.ndst; ++j) {
      char* d = reinterpret_cast<char*>(op.dst[j]) + dof;
      if constexpr (N == 8) {
        store8_to<DDT>(d, acc, op.flags & M2N_FLAG_MULTIMEM);
      } else {
        Elem<DDT>::store1(d, acc[0]);
      }
    }
  }
}

// One out-of-line walker per (source dtype, destination dtype): each gets its own register allocation.
#ifndef ETHA_TYPED_UNROLL
#define ETHA_TYPED_UNROLL 4
#endif
#ifndef ETHA_GENERAL_CTAS
#define ETHA_GENERAL_CTAS 4
#endif
constexpr int kTypedUnroll = ETHA_TYPED_UNROLL;

template <int S, int D>
__device__ __noinline__ void walk_cvt(const M2NOp& op, uint32_t base, uint32_t limit) {
  const uint32_t step = blockDim.x * kTypedUnroll;
  if (op.unit_elems == 8) {
    // boxes that are one run or rows of a matrix (almost every weight) skip the generic index arithmetic
    if (op.ndim == 0) {
      for (uint32_t b = base; b < limit; b += step) tile_cvt8<S, D, kTypedUnroll, 0>(op, b, limit);
    } else if (op.ndim == 1) {
      for (uint32_t b = base; b < limit; b += step) tile_cvt8<S, D, kTypedUnroll, 1>(op, b, limit);
    } else {
      for (uint32_t b = base; b < limit; b += step) tile_cvt8<S, D, kTypedUnroll>(op, b, limit);
    }
  } else {
    for (uint32_t b = base; b < limit; b += step) tile_cvt1<S, D, kTypedUnroll>(op, b, limit);
  }
}

template <int S, int D>
__device__ __noinline__ void walk_red(const M2NOp& op, uint32_t base, uint32_t limit) {
  const bool vec = op.unit_elems == 8;
  const bool flat = vec && op.red_size[1] == 1;
  const uint32_t step = blockDim.x * 2;
  for (uint32_t b = base; b < limit; b += step) {
    if (flat && op.nsrc == 2 && op.ndim == 0) tile_reduce_flat<S, D, 2, 0>(op, b, limit, 2);
    else if (flat && op.nsrc == 2 && op.ndim == 1) tile_reduce_flat<S, D, 2, 1>(op, b, limit, 2);
    else if (flat && op.nsrc == 2) tile_reduce_flat<S, D, 2>(op, b, limit, 2);
    else if (flat && op.nsrc == 4) tile_reduce_flat<S, D, 4>(op, b, limit, 2);
    else if (flat && op.nsrc == 8) tile_reduce_flat<S, D, 8>(op, b, limit, 2);
    else if (vec) tile_reduce<S, D, 8>(op, b, limit, 2);
    else tile_reduce<S, D, 1>(op, b, limit, 2);
  }
}

__device__ __forceinline__ bool dispatch_typed(const M2NOp& op, uint32_t base, uint32_t limit) {
  const int key = (op.mode << 8) | (op.src_dtype << 4) | op.dst_dtype;
#define CASE_CVT(S, D) case (M2N_MODE_CVT << 8) | (S << 4) | D: walk_cvt<S, D>(op, base, limit); return true;
#define CASE_RED(S, D) case (M2N_MODE_REDUCE << 8) | (S << 4) | D: walk_red<S, D>(op, base, limit); return true;
  switch (key) {
    CASE_CVT(M2N_F32, M2N_BF16) CASE_CVT(M2N_F32, M2N_F16) CASE_CVT(M2N_BF16, M2N_F32) CASE_CVT(M2N_F16, M2N_F32)
    CASE_CVT(M2N_BF16, M2N_F16) CASE_CVT(M2N_F16, M2N_BF16)
    CASE_RED(M2N_F32, M2N_F32) CASE_RED(M2N_F32, M2N_BF16) CASE_RED(M2N_F32, M2N_F16) CASE_RED(M2N_BF16, M2N_BF16)
    CASE_RED(M2N_BF16, M2N_F32) CASE_RED(M2N_BF16, M2N_F16) CASE_RED(M2N_F16, M2N_F16) CASE_RED(M2N_F16, M2N_F32)
    CASE_RED(M2N_F16, M2N_BF16)
    default: return false;
  }
#undef CASE_CVT
#undef CASE_RED
}

// Fast class: 16-byte bit copies whose box is one run or rows of a matrix (the bulk of a weight sync).  Bound by HBM (or
// NVLink): 4 x 512 threads per SM at 32 registers, two 16-byte loads each before the first store, tiles of one such trip
// (16 KiB).  1 GiB on one GPU, read + written: contiguous 6.71 TB/s, 2 KiB rows out of 8 KiB ones 6.46, one source and four
// destinations 6.52 (2 x 512 threads with four loads and a fixed stride of 64 KiB tiles: 5.52, 5.79, 5.37).  With 76 bytes of
// spills per thread the same kernel falls to 5.97, so full trips carry no per-unit predicate.
constexpr int kFastThreads = 512;
constexpr int kFastCtas = 4;
constexpr int kFastUnroll = 2;

// U units of one thread, kFastThreads apart, the first one `unit0`: every load is issued before the first store
template <int ND, int U>
__device__ __forceinline__ void fast_trip(const M2NOp& op, uint32_t unit0) {
  uint4 v[U];
  int64_t dof[U];
  const char* src = reinterpret_cast<const char*>(op.src[0]);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    int64_t so;
    unit_offsets<ND, 16>(op, unit0 + u * kFastThreads, so, dof[u]);
    v[u] = ld_stream<uint4>(src + so);
  }
  if (op.flags & M2N_FLAG_MULTIMEM) {
#pragma unroll
    for (int u = 0; u < U; ++u) st_multimem16(reinterpret_cast<char*>(op.dst[0]) + dof[u], v[u]);
    return;
  }
  const int nd = op.ndst;
#pragma unroll 1
  for (int j = 0; j < nd; ++j) {
    char* dst = reinterpret_cast<char*>(op.dst[j]);
#pragma unroll
    for (int u = 0; u < U; ++u) st_plain<uint4>(dst + dof[u], v[u]);
  }
}

template <int ND>
__device__ __forceinline__ void fast_tile(const M2NOp& op, uint32_t base, uint32_t limit) {
  constexpr uint32_t step = kFastThreads * kFastUnroll;
  uint32_t b = base;
#pragma unroll 1
  for (; b + step <= limit; b += step) fast_trip<ND, kFastUnroll>(op, b + threadIdx.x);
#pragma unroll 1
  for (b += threadIdx.x; b < limit; b += kFastThreads) fast_trip<ND, 1>(op, b);
}

__global__ void __launch_bounds__(kFastThreads, kFastCtas)
m2n_fast_kernel(const __grid_constant__ M2NLaunch args) {
  __shared__ M2NOp s_op;
  __shared__ TileSched s_sched;
  const uint32_t done = for_each_tile(&s_sched, &s_op, args, [&](const M2NOp& op, uint32_t base, uint32_t limit) {
    if (op.ndim == 0) fast_tile<0>(op, base, limit);
    else fast_tile<1>(op, base, limit);
  });
  finish(args, done);
}

// General class: any other bit copy, converting copies and Partial collapses.
constexpr int kGeneralThreads = 256;
constexpr int kGenUnroll = 2;
template <typename V>
__device__ __noinline__ void walk_raw(const M2NOp& op, uint32_t base, uint32_t limit) {
  for (uint32_t b = base; b < limit; b += blockDim.x * kGenUnroll) tile_raw<V, kGenUnroll, -1>(op, b, limit);
}

__global__ void __launch_bounds__(kGeneralThreads, ETHA_GENERAL_CTAS)
m2n_general_kernel(const __grid_constant__ M2NLaunch args) {
  __shared__ M2NOp s_op;
  __shared__ TileSched s_sched;
  const uint32_t done = for_each_tile(&s_sched, &s_op, args, [&](const M2NOp& op, uint32_t base, uint32_t limit) {
    if (op.mode == M2N_MODE_RAW) {
      switch (op.unit_bytes_src) {
        case 16: walk_raw<uint4>(op, base, limit); break;
        case 8: walk_raw<uint2>(op, base, limit); break;
        case 4: walk_raw<uint32_t>(op, base, limit); break;
        case 2: walk_raw<uint16_t>(op, base, limit); break;
        default: walk_raw<uint8_t>(op, base, limit); break;
      }
    } else if (!dispatch_typed(op, base, limit)) {
      if (threadIdx.x == 0) report(args, M2N_BAD_OP);
    }
  });
  finish(args, done);
}

__global__ void set_flags_kernel(const uint64_t* __restrict__ signals, uint32_t n_signals, uint32_t epoch) {
  __threadfence_system();
  for (uint32_t i = threadIdx.x; i < n_signals; i += blockDim.x) {
    uint32_t* flag = reinterpret_cast<uint32_t*>(signals[i]);
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(epoch) : "memory");
  }
}

__device__ __forceinline__ bool flag_is_set(const uint32_t* flag, uint32_t epoch) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
  return (int32_t)(v - epoch) >= 0;
}

// Bounded acquire-wait by one warp.  A flag counts as set once it reached `epoch` (wrap-safe compare).  On timeout the
// kernel reports which flag was missing and returns; it never traps and never spins without a limit.  All flags share one
// deadline, however many of them a lane looks after.  It lets the
// next kernel of the stream start only when it has seen the flags: CTAs that are resident while it spins could keep a
// producer off this GPU.  What it costs when the flags are set already is latency only: the clock is read once a lane has
// missed one, and both status words go out in one store where their address allows it.
__global__ void __launch_bounds__(32)
wait_flags_kernel(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ which, uint32_t n, uint32_t epoch,
                  uint64_t timeout_ns, uint32_t* status) {
  after_previous_kernel();
  uint32_t missing = 0xffffffffu;
  bool late = false;
  for (uint32_t i = threadIdx.x; i < n; i += 32) late |= !flag_is_set(flags + which[i], epoch);
  if (__any_sync(0xffffffffu, late)) {
    uint64_t t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (uint32_t i = threadIdx.x; i < n; i += 32) {
      const uint32_t* flag = flags + which[i];
      bool ok = false;
      for (uint64_t it = 0; it < (1ull << 34); ++it) {
        ok = flag_is_set(flag, epoch);
        if (ok) break;
        if ((it & 63) == 0) {
          asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
          if (t - t0 > timeout_ns) break;
          if (it) __nanosleep(200);
        }
      }
      if (!ok) missing = min(missing, i);
    }
  }
  missing = __reduce_min_sync(0xffffffffu, missing);
  if (threadIdx.x == 0) {
    let_next_kernel_start();
    const uint32_t code = missing == 0xffffffffu ? M2N_OK : M2N_TIMEOUT;
    if ((reinterpret_cast<uint64_t>(status) & 7) == 0) {
      *reinterpret_cast<uint2*>(status) = make_uint2(code, missing);
    } else {
      status[1] = missing;
      __threadfence_system();
      status[0] = code;
    }
  }
}

inline int fail(cudaError_t e, const char* what) { return m2n_cuda_error(e, what); }

}  // namespace

int m2n_launch_copy(const M2NLaunch& args, bool general, uint32_t n_tiles, int ctas_per_sm, void* stream) {
  if (general) return m2n_launch(m2n_general_kernel, n_tiles, kGeneralThreads, 0, stream, args, "general");
  // a caller that asks for one CTA per SM (of the two that fill it by default) leaves half of each SM to other work:
  // shared memory that is never touched lets two of the four CTAs in
  const int smem = ctas_per_sm == 1 ? 76 * 1024 : 0;
  if (smem) {
    cudaError_t e = cudaFuncSetAttribute(m2n_fast_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(e, "fast kernel shared memory opt-in");
  }
  return m2n_launch(m2n_fast_kernel, n_tiles, kFastThreads, smem, stream, args, "fast");
}

extern "C" {

int etha_set_flags(const uint64_t* signals, uint32_t n_signals, uint32_t epoch, int device, void* stream) {
  const OnDevice on(device);
  if (on.error != cudaSuccess) return fail(on.error, "device of the launch");
  set_flags_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(signals, n_signals, epoch);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : fail(e, "set_flags launch");
}

int etha_wait_flags(const uint32_t* flags, const uint32_t* which, uint32_t n, uint32_t epoch, uint64_t timeout_ns,
                    uint32_t* status, int device, void* stream) {
  const OnDevice on(device);
  if (on.error != cudaSuccess) return fail(on.error, "device of the launch");
  cudaError_t e = m2n_launch_dependent(wait_flags_kernel, 1, 32, 0, stream, flags, which, n, epoch, timeout_ns, status);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess ? 0 : fail(e, "wait_flags launch");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------
// Allocation-free entry point (declared in no_alloc.h).  Same kernels as above; the op table, the tile
// prefix sums and the counters live in a resident array instead of caller-allocated device buffers.
// ---------------------------------------------------------------------------------------------------
#include <mutex>

#include "no_alloc.h"

namespace {

static_assert(sizeof(M2NOp) <= 320, "scratch layout assumes ops of at most 320 bytes");

// layout: [0,256) counters of the fast launch, [256,512) counters of the general launch,
//         [512,1280) tile_start of the fast class, [1280,2048) tile_start of the general class,
//         [2048, ...) ops: fast class first, general class after it
static __device__ __align__(256) unsigned char g_noalloc_scratch[ETHA_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices] = {nullptr};

// Host code must not use `g_noalloc_scratch` as an address: there it is only a stand-in for the symbol.
// The device address is queried once per device, with that device current.
int noalloc_setup(int dev, unsigned char** out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (dev < 0 || dev >= kMaxDevices) {
    snprintf(etha_err_buf(), ETHA_ERR_LEN, "device index %d out of range", dev);
    return -101;
  }
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) return fail(e, "cudaGetSymbolAddress(scratch)");
    g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}

}  // namespace

extern "C" int etha_m2n_run_noalloc(const M2NOpSpec* specs, uint32_t n_specs, int ctas_per_sm, void* stream) {
  if (!specs && n_specs) {
    snprintf(etha_err_buf(), ETHA_ERR_LEN, "null spec array");
    return -101;
  }
  if (n_specs > ETHA_NOALLOC_MAX_OPS) {
    snprintf(etha_err_buf(), ETHA_ERR_LEN, "%u ops requested, the allocation-free entry point takes at most %d per call",
             n_specs, ETHA_NOALLOC_MAX_OPS);
    return -100;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(e, "cudaGetDevice");
  // every call stages its tables from host arrays of the calling thread with asynchronous copies: recorded into a
  // stream capture they would be replayed later from whatever those arrays hold then, so a capturing stream is refused
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing((cudaStream_t)stream, &cap);
  if (e != cudaSuccess) return fail(e, "cudaStreamIsCapturing");
  if (cap != cudaStreamCaptureStatusNone) {
    snprintf(etha_err_buf(), ETHA_ERR_LEN, "the allocation-free entry point cannot be recorded into a stream capture");
    return -101;
  }
  unsigned char* scratch = nullptr;
  int rc = noalloc_setup(dev, &scratch);
  if (rc != 0) return rc;

  // host staging lives in thread-local storage: no heap allocation per call
  static thread_local M2NOp packed[2][ETHA_NOALLOC_MAX_OPS];
  static thread_local uint32_t tile_start[2][ETHA_NOALLOC_MAX_OPS + 1];
  uint32_t count[2] = {0, 0};
  for (uint32_t i = 0; i < n_specs; ++i) {
    M2NOp op;
    rc = etha_pack_op(&specs[i], &op, etha_err_buf(), ETHA_ERR_LEN);
    if (rc != 0) return rc;
    if (!etha_op_tiles(&op)) continue;
    const int c = etha_op_class(&op);
    packed[c][count[c]++] = op;
  }
  for (int c = 0; c < 2; ++c)
    if (etha_layout_tiles(packed[c], count[c], c, tile_start[c]) < 0) {
      snprintf(etha_err_buf(), ETHA_ERR_LEN, "too many tiles in one call");
      return -101;
    }
  cudaStream_t s = (cudaStream_t)stream;
  // counters must start at zero whatever the previous call left there
  e = cudaMemsetAsync(scratch, 0, 512, s);
  if (e != cudaSuccess) return fail(e, "cudaMemsetAsync(scratch counters)");
  if (ctas_per_sm <= 0) ctas_per_sm = 2;
  M2NOp* ops_dev = reinterpret_cast<M2NOp*>(scratch + 2048);
  for (int c = 0; c < 2; ++c) {
    if (!count[c]) continue;
    uint32_t* tiles_dev = reinterpret_cast<uint32_t*>(scratch + 512 + 768 * c);
    M2NOp* class_ops = ops_dev + (c == 0 ? 0 : count[0]);
    e = cudaMemcpyAsync(tiles_dev, tile_start[c], (count[c] + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return fail(e, "cudaMemcpyAsync(tile table)");
    e = cudaMemcpyAsync(class_ops, packed[c], count[c] * sizeof(M2NOp), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return fail(e, "cudaMemcpyAsync(op table)");
    const EthaLaunch launch = {c == 0 ? M2N_KEY_FAST : M2N_KEY_GENERAL, count[c], tile_start[c][count[c]], dev,
                               reinterpret_cast<uint64_t>(class_ops), reinterpret_cast<uint64_t>(tiles_dev)};
    rc = etha_run(&launch, 1, reinterpret_cast<uint32_t*>(scratch + 256 * c), nullptr, 0, 0, ctas_per_sm, s);
    if (rc != 0) return rc;
  }
  return 0;
}

extern "C" int etha_m2n_noalloc_status(uint32_t* status, void* stream) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(e, "cudaGetDevice");
  unsigned char* scratch = nullptr;
  int rc = noalloc_setup(dev, &scratch);
  if (rc != 0) return rc;
  uint32_t words[2] = {0, 0};
  e = cudaMemcpyAsync(&words[0], scratch + 4, 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&words[1], scratch + 256 + 4, 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return fail(e, "read scratch status");
  *status = words[0] ? words[0] : words[1];
  return 0;
}
