// Device helpers shared by the kernels of the M-to-N redistribution (sm_100a): streaming loads, multicast
// stores, box index arithmetic, typed 8-element vectors, the reduce step, completion signalling and the
// tile -> op lookup.  Everything is `static`/inline so that each translation unit gets its own copy.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "m2n.h"
#include "m2n_launch.h"

namespace {

// ---------------------------------------------------------------------------------------------
// memory access helpers
// ---------------------------------------------------------------------------------------------
// (plain loads, not the non-coherent ones: the sources may be written by the kernel before this one while this one is
// already resident, see `after_previous_kernel`; both kinds run at the same speed)
template <typename V>
__device__ __forceinline__ V ld_stream(const void* p);

template <>
__device__ __forceinline__ uint4 ld_stream<uint4>(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
template <>
__device__ __forceinline__ uint2 ld_stream<uint2>(const void* p) {
  uint2 v;
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
template <>
__device__ __forceinline__ uint32_t ld_stream<uint32_t>(const void* p) {
  uint32_t v;
  asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
template <>
__device__ __forceinline__ uint16_t ld_stream<uint16_t>(const void* p) {
  uint16_t v;
  asm volatile("ld.global.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
template <>
__device__ __forceinline__ uint8_t ld_stream<uint8_t>(const void* p) {
  uint32_t v;
  asm volatile("ld.global.L1::no_allocate.u8 %0, [%1];" : "=r"(v) : "l"(p));
  return (uint8_t)v;
}

// a thread that reads 32 contiguous bytes with two 16-byte loads touches every 32-byte sector twice: let the
// first load allocate the sector in L1 so that the second one does not go back to L2
__device__ __forceinline__ uint4 ld_keep(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// stores in the global state space: a plain `*p = v` could alias the op in shared memory, which would then be read again
// after every store
template <typename V>
__device__ __forceinline__ void st_plain(void* p, V v) {
  const size_t g = __cvta_generic_to_global(p);
  if constexpr (sizeof(V) == 16)
    asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(g), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
  else if constexpr (sizeof(V) == 8)
    asm volatile("st.global.v2.u32 [%0], {%1,%2};" ::"l"(g), "r"(v.x), "r"(v.y));
  else if constexpr (sizeof(V) == 4)
    asm volatile("st.global.u32 [%0], %1;" ::"l"(g), "r"((uint32_t)v));
  else if constexpr (sizeof(V) == 2)
    asm volatile("st.global.u16 [%0], %1;" ::"l"(g), "h"((uint16_t)v));
  else
    asm volatile("st.global.u8 [%0], %1;" ::"l"(g), "r"((uint32_t)v));
}

// one 16-byte store delivered by NVSwitch to every GPU bound to the multicast object
__device__ __forceinline__ void st_multimem16(void* p, uint4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

__host__ __device__ __forceinline__ uint32_t fast_div(uint32_t n, uint32_t mul, uint32_t shr) {
#ifdef __CUDA_ARCH__
  return mul ? (__umulhi(n, mul) >> shr) : n;  // mul == 0 encodes "divide by one"
#else
  return mul ? (uint32_t)(((uint64_t)n * mul) >> 32) >> shr : n;
#endif
}

// byte offsets of unit `unit` of the op inside the source and the destination box; BYTES: size of a unit on both sides
// where the kernel knows it.  A row can be longer than 4 GiB (28 bits of 16-byte units): bytes are 64 bits wide
// throughout.  The host runs the same code in etha_op_unit_offsets.
template <int ND = -1, int BYTES = 0>
__host__ __device__ __forceinline__ void unit_offsets(const M2NOp& op, uint32_t unit, int64_t& so, int64_t& dof) {
  const uint32_t bytes_src = BYTES ? BYTES : op.unit_bytes_src, bytes_dst = BYTES ? BYTES : op.unit_bytes_dst;
  if constexpr (ND == 0) {  // one contiguous run on both sides
    so = (int64_t)unit * bytes_src;
    dof = (int64_t)unit * bytes_dst;
    return;
  }
  uint32_t q = fast_div(unit, op.div_mul[M2N_MAX_DIMS], op.div_shr[M2N_MAX_DIMS]);
  uint32_t col = unit - q * op.inner_units;
  so = (int64_t)col * bytes_src;
  dof = (int64_t)col * bytes_dst;
  if constexpr (ND == 1) {  // rows of a matrix
    so += (int64_t)q * op.src_stride[0];
    dof += (int64_t)q * op.dst_stride[0];
    return;
  }
  const int nd = op.ndim;
#pragma unroll
  for (int d = M2N_MAX_DIMS - 1; d >= 0; --d) {
    if (d < nd) {
      uint32_t q2 = (d == 0) ? 0u : fast_div(q, op.div_mul[d], op.div_shr[d]);
      uint32_t i = q - q2 * op.extent[d];
      so += (int64_t)i * op.src_stride[d];
      dof += (int64_t)i * op.dst_stride[d];
      q = q2;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// typed element vectors (8 elements) for conversion and reduction
// ---------------------------------------------------------------------------------------------
template <int DT>
struct Elem;

template <>
struct Elem<M2N_F32> {
  static constexpr int W = 2;  // 16-byte words per 8 elements
  static __device__ __forceinline__ void load_raw(const char* p, uint4 (&r)[2]) {
    r[0] = ld_keep(p);
    r[1] = ld_keep(p + 16);
  }
  static __device__ __forceinline__ void decode(const uint4 (&r)[2], float (&f)[8]) {
    const uint4 a = r[0], b = r[1];
    f[0] = __uint_as_float(a.x), f[1] = __uint_as_float(a.y), f[2] = __uint_as_float(a.z), f[3] = __uint_as_float(a.w);
    f[4] = __uint_as_float(b.x), f[5] = __uint_as_float(b.y), f[6] = __uint_as_float(b.z), f[7] = __uint_as_float(b.w);
  }
  static __device__ __forceinline__ void load8(const char* p, float (&f)[8]) {
    uint4 r[2];
    load_raw(p, r);
    decode(r, f);
  }
  static __device__ __forceinline__ void store8(char* p, const float (&f)[8]) {
    st_plain<uint4>(p, make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3])));
    st_plain<uint4>(p + 16, make_uint4(__float_as_uint(f[4]), __float_as_uint(f[5]), __float_as_uint(f[6]), __float_as_uint(f[7])));
  }
  static __device__ __forceinline__ float load1(const char* p) { return __uint_as_float(ld_stream<uint32_t>(p)); }
  static __device__ __forceinline__ void store1(char* p, float f) { *reinterpret_cast<float*>(p) = f; }
};

template <>
struct Elem<M2N_BF16> {
  static __device__ __forceinline__ float up(uint32_t w, int hi) { return __uint_as_float(hi ? (w & 0xffff0000u) : (w << 16)); }
  static constexpr int W = 1;
  static __device__ __forceinline__ void load_raw(const char* p, uint4 (&r)[1]) { r[0] = ld_stream<uint4>(p); }
  static __device__ __forceinline__ void decode(const uint4 (&r)[1], float (&f)[8]) {
    const uint4 a = r[0];
    f[0] = up(a.x, 0), f[1] = up(a.x, 1), f[2] = up(a.y, 0), f[3] = up(a.y, 1);
    f[4] = up(a.z, 0), f[5] = up(a.z, 1), f[6] = up(a.w, 0), f[7] = up(a.w, 1);
  }
  static __device__ __forceinline__ void load8(const char* p, float (&f)[8]) {
    uint4 r[1];
    load_raw(p, r);
    decode(r, f);
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ void store8(char* p, const float (&f)[8]) {
    st_plain<uint4>(p, make_uint4(pack(f[0], f[1]), pack(f[2], f[3]), pack(f[4], f[5]), pack(f[6], f[7])));
  }
  static __device__ __forceinline__ float load1(const char* p) { return __uint_as_float((uint32_t)ld_stream<uint16_t>(p) << 16); }
  static __device__ __forceinline__ void store1(char* p, float f) { *reinterpret_cast<__nv_bfloat16*>(p) = __float2bfloat16_rn(f); }
};

template <>
struct Elem<M2N_F16> {
  static __device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi) {
    __half2 h = *reinterpret_cast<__half2*>(&w);
    float2 f = __half22float2(h);
    lo = f.x, hi = f.y;
  }
  static constexpr int W = 1;
  static __device__ __forceinline__ void load_raw(const char* p, uint4 (&r)[1]) { r[0] = ld_stream<uint4>(p); }
  static __device__ __forceinline__ void decode(const uint4 (&r)[1], float (&f)[8]) {
    const uint4 a = r[0];
    unpack(a.x, f[0], f[1]), unpack(a.y, f[2], f[3]), unpack(a.z, f[4], f[5]), unpack(a.w, f[6], f[7]);
  }
  static __device__ __forceinline__ void load8(const char* p, float (&f)[8]) {
    uint4 r[1];
    load_raw(p, r);
    decode(r, f);
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ void store8(char* p, const float (&f)[8]) {
    st_plain<uint4>(p, make_uint4(pack(f[0], f[1]), pack(f[2], f[3]), pack(f[4], f[5]), pack(f[6], f[7])));
  }
  static __device__ __forceinline__ float load1(const char* p) {
    uint16_t b = ld_stream<uint16_t>(p);
    return __half2float(*reinterpret_cast<__half*>(&b));
  }
  static __device__ __forceinline__ void store1(char* p, float f) { *reinterpret_cast<__half*>(p) = __float2half_rn(f); }
};

// store 8 converted elements either with plain stores or, for an NVLS destination, with multicast stores
template <int DDT>
__device__ __forceinline__ void store8_to(char* p, const float (&f)[8], bool multicast) {
  if (!multicast) {
    Elem<DDT>::store8(p, f);
    return;
  }
  if constexpr (DDT == M2N_F32) {
    st_multimem16(p, make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3])));
    st_multimem16(p + 16, make_uint4(__float_as_uint(f[4]), __float_as_uint(f[5]), __float_as_uint(f[6]), __float_as_uint(f[7])));
  } else {
    st_multimem16(p, make_uint4(Elem<DDT>::pack(f[0], f[1]), Elem<DDT>::pack(f[2], f[3]), Elem<DDT>::pack(f[4], f[5]),
                                Elem<DDT>::pack(f[6], f[7])));
  }
}

__device__ __forceinline__ float reduce2(float a, float b, int op) {
  switch (op) {
    case M2N_MAX: return (a != a) ? a : ((b != b) ? b : fmaxf(a, b));  // NaN propagates, like torch.maximum
    case M2N_MIN: return (a != a) ? a : ((b != b) ? b : fminf(a, b));
    case M2N_PROD: return a * b;
    default: return a + b;  // SUM and AVG
  }
}

// a[k] = reduce2(a[k], b[k], op), with one branch on the op
__device__ __forceinline__ void reduce8(float (&a)[8], const float (&b)[8], int op) {
  if (op == M2N_SUM || op == M2N_AVG) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] += b[k];
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = reduce2(a[k], b[k], op);
  }
}

template <int DT>
__device__ __forceinline__ float round_through(float x) {
  if constexpr (DT == M2N_BF16) return __bfloat162float(__float2bfloat16_rn(x));
  if constexpr (DT == M2N_F16) return __half2float(__float2half_rn(x));
  return x;
}

// ---------------------------------------------------------------------------------------------
// tile scheduling
// ---------------------------------------------------------------------------------------------
// The kernels are launched with one CTA per tile, and a CTA that has finished its tile takes over the tile of a CTA that
// has not been launched yet (cluster launch control), until none is left.  Why not a grid of resident CTAs with a
// fixed stride: SMs do not run equally fast, so fixed shares drift apart, the addresses in flight spread over many
// DRAM pages and the slowest SM sets the end.  A bare copy of 1 GiB with 16-byte units: fixed stride 5.7 to 6.0 TB/s (read
// + written) with any block size, unroll or cache hint; tiles taken in order as SMs become free 6.7 to 6.9; one read
// and four writes: 5.6 and 6.6.  Why not a counter in memory: the hardware's queue belongs to the launch, so two launches of one table (two
// streams, a graph) share no queue and nothing has to be reset.  Launches that signal share the table's count of finished
// tiles, though, and have to follow one another (see `finish`).  A CTA that takes tiles over pays its prologue (and the
// completion fence) once.
//
// `sync` is one 64-bit word to the kernels: finished tiles in the lower half, status bits in the upper one, so that the CTA
// whose add completes the launch learns from the same add whether any CTA has reported a failure.
__device__ __forceinline__ unsigned long long* sync_word(const M2NLaunch& args) {
  return reinterpret_cast<unsigned long long*>(args.sync);
}

__device__ __forceinline__ void report(const M2NLaunch& args, uint32_t status) {
  if (args.sync) atomicOr(sync_word(args), (unsigned long long)status << 32);
}

struct TileSched {
  uint4 handle;  // answer of try_cancel, written by the asynchronous proxy
  uint4 state;   // x, y: tiles of the op in `s_op`; z, w: a thread has given up in phase 0, 1 (read together once per tile)
  uint64_t bar;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void sched_init(TileSched* s) {
  if (threadIdx.x == 0) {
    s->state = make_uint4(1, 0, 0, 0);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s->bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}

// one thread asks for the next tile; the answer arrives while the CTA works on the present one
__device__ __forceinline__ void sched_request(TileSched* s) {
  const uint32_t bar = smem_addr(&s->bar);
  asm volatile("fence.proxy.async::generic.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cta.b64 _, [%0], 16;" ::"r"(bar) : "memory");
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_addr(&s->handle)),
               "r"(bar)
               : "memory");
}

enum Take { kNoTile, kTile, kNoAnswer };
constexpr uint32_t kAnswerSpins = 1u << 22;

// Every thread that asks waits for the answer, which names the next tile.  One that runs into the limit reports it, marks the
// queue, and waits once more: no answer should arrive in the shared memory of a CTA that has ended.  All threads see the mark after
// the barrier that the next request needs anyway, and stop together; a tile in the answer then counts as finished without being
// run.  A mark per phase: a thread that is quick to give up on the next answer does not change what a slow one still has to read.
// (With a voting barrier per tile instead, 1169.8 us for a sync that takes 1164.8; with the second wait in a place of its own, 5 more
// registers and 121 us for ragged conversions that take 112.)
__device__ __forceinline__ Take sched_take(TileSched* s, uint32_t phase, uint32_t& tile, const M2NLaunch& args) {
  const uint32_t bar = smem_addr(&s->bar);
  uint32_t ready = 0;
  for (uint32_t spin = 0; spin < 2 * kAnswerSpins && !ready; ++spin) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ready)
        : "r"(bar), "r"(phase)
        : "memory");
    if (spin == kAnswerSpins) {
      report(args, M2N_TIMEOUT);
      (phase ? s->state.w : s->state.z) = 1;
    }
  }
  if (!ready) return kNoAnswer;
  uint32_t more;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
      : "=r"(more), "=r"(tile)
      : "r"(smem_addr(&s->handle))
      : "memory");
  asm volatile("fence.proxy.async::generic.release.sync_restrict::shared::cta.cluster;" ::: "memory");
  return more ? kTile : kNoTile;
}

// whether a thread has given up in `phase`; the threads that asked have been synchronised since
__device__ __forceinline__ bool gave_up(const uint4& state, uint32_t phase) { return phase ? state.w : state.z; }

// one warp loads the op that owns `tile` (looked up 32 ways at a time) into shared memory; returns its tiles
__device__ __forceinline__ uint2 load_op(const M2NLaunch& args, uint32_t tile, M2NOp* s_op) {
  const uint32_t lane = threadIdx.x & 31;
  const M2NOp* op = &args.one;
  uint2 tiles = make_uint2(0, gridDim.x);
  if (args.ops) {
    uint32_t lo = 0, hi = args.n_ops;
    while (hi - lo > 1) {
      const uint32_t step = (hi - lo + 31) >> 5, i = lo + lane * step;
      const uint32_t below = __ballot_sync(0xffffffffu, i < hi && args.tile_start[i] <= tile);
      lo += (31 - __clz(below)) * step;
      hi = min(hi, lo + step);
    }
    op = args.ops + lo;
    tiles = make_uint2(args.tile_start[lo], args.tile_start[lo + 1]);
  }
  const uint4* g = reinterpret_cast<const uint4*>(op);
  uint4* d = reinterpret_cast<uint4*>(s_op);
  for (uint32_t i = lane; i < sizeof(M2NOp) / 16; i += 32) d[i] = g[i];
  return tiles;
}

// Make `s_op` the op that owns `tile`, whose first tile is returned; the CTA is synchronised since its last use and `state`
// read since then.  Tiles come in ascending order, so the op is nearly always the one already there.
__device__ __forceinline__ uint32_t sched_locate(TileSched* s, const uint4& state, const M2NLaunch& args, uint32_t tile, M2NOp* s_op) {
  if (tile >= state.x && tile < state.y) return state.x;
  __syncthreads();  // everybody has read the state
  if (threadIdx.x < 32) {
    const uint2 tiles = load_op(args, tile, s_op);
    if (threadIdx.x == 0) s->state.x = tiles.x, s->state.y = tiles.y;
  }
  __syncthreads();
  return s->state.x;
}

// Waits until the kernel before this one in the stream has finished and its writes are visible.  EVERY thread of EVERY kernel
// launched as a dependent passes here before it touches anything that is not its own launch's table: a kernel that
// finishes has then also outwaited all kernels before its predecessor.
__device__ __forceinline__ void after_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Lets the next kernel in the stream start its set-up once every CTA has come here (or ended).  One thread calls it, after a
// barrier of its CTA and a fence: a kernel that reads weights ahead of its own wait, because it takes them for
// constants, then still finds what this one has delivered.
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Walk over all tiles of the table: `body(op, first unit, one past the last unit)` runs with all threads of the CTA.
// Returns the number of tiles this CTA took.  CHUNKS: the tiles are counted in the op's chunks instead of its units.
template <bool CHUNKS = false, typename Body>
__device__ __forceinline__ uint32_t for_each_tile(TileSched* s, M2NOp* s_op, const M2NLaunch& args, Body&& body) {
  sched_init(s);
  uint32_t tile = blockIdx.x, taken = 1, phase = 0;
  Take take;
  uint4 state = s->state;
  do {
    if (threadIdx.x == 0) sched_request(s);
    const uint32_t first = sched_locate(s, state, args, tile, s_op);
    if (taken == 1) after_previous_kernel();
    const M2NOp& op = *s_op;
    const uint32_t base = (tile - first) * op.tile_units;
    body(op, base, min(CHUNKS ? op.chunks : op.total_units, base + op.tile_units));
    take = sched_take(s, phase, tile, args);
    __syncthreads();
    state = s->state;
    if (take != kTile) return taken;
    ++taken;
    if (gave_up(state, phase)) return taken;
    phase ^= 1;
  } while (true);
}

// The CTA that finishes the last tile publishes `epoch` to every flag with system-scope release ordering.  Each CTA
// releases its stores to this GPU only (fence + atomic add at GPU scope); the last one acquires all of them that way, and
// its system-scope release stores order them for the consumers too (release patterns are cumulative).  What a small table
// of 592 CTAs pays for its signal: 13 us with a system-scope fence in every CTA, 5 us with a GPU-scope one there and a
// system-scope fence before the release stores, 3 us as it stands.
// The count belongs to the table: two signalling launches of one table that overlap would complete each other's count and
// publish early.  They have to be ordered (one stream, or events); launches without signals do not touch it.
// `done` holds failed and abandoned tiles too, so that the count closes and the next launch starts at 0.  Nothing is
// published while the error word is set, in this launch or a later one: a flag never stands for data that was not
// delivered, and consumers run into their own limit.
__device__ __forceinline__ void finish(const M2NLaunch& args, uint32_t done) {
  __shared__ uint32_t s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    let_next_kernel_start();
  }
  if (!args.do_signal) return;
  if (threadIdx.x == 0) {
    const unsigned long long prev = atomicAdd(sync_word(args), (unsigned long long)done);
    const bool last = (uint32_t)prev + done == gridDim.x;
    if (last) args.sync[0] = 0;  // ready for the next launch on this stream
    s_last = last && (prev >> 32) == 0;
    __threadfence();
  }
  __syncthreads();
  if (s_last) {
    for (uint32_t i = threadIdx.x; i < args.n_signals; i += blockDim.x) {
      uint32_t* flag = reinterpret_cast<uint32_t*>(args.signals[i]);
      asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(args.epoch) : "memory");
    }
  }
}

}  // namespace
