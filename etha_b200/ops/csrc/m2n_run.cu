// Entry points that run launches: a table's list of them, and copies whose ops travel in the kernel arguments.
#include <cstring>

#include "m2n_device.cuh"
#include "m2n_launch.h"

extern "C" {

int etha_op_kernel_key(const M2NOp* op) {
  if (etha_op_class(op) == 0) return M2N_KEY_FAST;
  int key = etha_op_stream_key(op);
  if (!key) key = etha_op_collapse_key(op);
  if (!key) key = etha_op_ragged_key(op);
  if (!key) key = etha_op_transpose_key(op);
  return key ? key : M2N_KEY_GENERAL;
}

int etha_key_tile_class(int key) {
  switch (key >> 12) {
    case M2N_KEY_GENERAL >> 12: return 1;
    case M2N_KEY_RAGGED >> 12: return 2;
    case M2N_KEY_TRANSPOSE >> 12: return 3;
    default: return 0;
  }
}

void etha_op_unit_offsets(const M2NOp* op, uint32_t unit, int64_t* src, int64_t* dst) {
  if (etha_op_class(op) != 0) unit_offsets(*op, unit, *src, *dst);
  else if (op->ndim == 0) unit_offsets<0, 16>(*op, unit, *src, *dst);
  else unit_offsets<1, 16>(*op, unit, *src, *dst);
}

}  // extern "C"

namespace {

int run_one(const M2NLaunch& args, int key, uint32_t n_tiles, int ctas_per_sm, void* stream) {
  if (!n_tiles) return 0;
  switch (key >> 12) {
    case M2N_KEY_FAST >> 12: return m2n_launch_copy(args, false, n_tiles, ctas_per_sm, stream);
    case M2N_KEY_GENERAL >> 12: return m2n_launch_copy(args, true, n_tiles, ctas_per_sm, stream);
    case M2N_KEY_BULK >> 12: return m2n_launch_bulk(args, n_tiles, stream);
    case M2N_KEY_RAGGED >> 12: return m2n_launch_ragged(args, key, n_tiles, stream);
    case M2N_KEY_COLLAPSE >> 12: return m2n_launch_collapse(args, key, n_tiles, stream);
    case M2N_KEY_TRANSPOSE >> 12: return m2n_launch_transpose(args, key, n_tiles, stream);
    default: return m2n_launch_typed(args, key, n_tiles, stream);
  }
}

}  // namespace

extern "C" {

int etha_run(const EthaLaunch* launches, uint32_t n, uint32_t* sync, const uint64_t* signals, uint32_t n_signals, uint32_t epoch,
             int ctas_per_sm, void* stream) {
  M2NLaunch args;
  memset(&args, 0, sizeof(args));
  args.sync = sync;
  args.signals = signals;
  args.epoch = epoch;
  if (!n) return 0;
  const OnDevice on(launches[0].device);
  if (on.error != cudaSuccess) return m2n_cuda_error(on.error, "device of the launch");
  for (uint32_t i = 0; i < n; ++i) {
    const EthaLaunch& l = launches[i];
    args.ops = reinterpret_cast<const M2NOp*>(l.ops);
    args.tile_start = reinterpret_cast<const uint32_t*>(l.tiles);
    args.n_ops = l.n_ops;
    const bool signal = n_signals && i + 1 == n;  // the last kernel of the transfer publishes
    args.n_signals = signal ? n_signals : 0;
    args.do_signal = signal;
    const int rc = run_one(args, l.key, l.n_tiles, ctas_per_sm, stream);
    if (rc != 0) return rc;
  }
  return 0;
}

int etha_run_spec(const M2NOpSpec* spec, int device, void* stream) {
  M2NLaunch args;
  memset(&args, 0, sizeof(args));
  const int rc = etha_pack_op(spec, &args.one, nullptr, 0);
  if (rc != 0) return rc;
  if (!etha_op_tiles(&args.one)) return 0;
  const int key = etha_op_kernel_key(&args.one);
  uint32_t starts[2];
  const int64_t tiles = etha_layout_tiles(&args.one, 1, etha_key_tile_class(key), starts);
  if (tiles < 0) {
    snprintf(etha_err_buf(), ETHA_ERR_LEN, "too many tiles in one op");
    return -101;
  }
  args.n_ops = 1;
  const OnDevice on(device);
  if (on.error != cudaSuccess) return m2n_cuda_error(on.error, "device of the launch");
  return run_one(args, key, (uint32_t)tiles, 0, stream);
}

}  // extern "C"
