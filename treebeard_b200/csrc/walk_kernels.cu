// The general walk's variants, compiled apart from the other kernels (as walk_quant.cu).
#include "walk_kernels.cuh"

namespace tb {

namespace {
template <int REP, int TS> WalkKernel pick(int rpl, bool staged, bool cached, bool turn) {
  if (turn) return staged ? tb_walk_kernel<REP, TS, 1, true, true, true> : tb_walk_kernel<REP, TS, 1, false, true, true>;
  if (!cached) return staged ? tb_walk_kernel<REP, TS, 1, true, false> : tb_walk_kernel<REP, TS, 1, false, false>;
  if (rpl == 2) return staged ? tb_walk_kernel<REP, TS, 2, true, true> : tb_walk_kernel<REP, TS, 2, false, true>;
  return staged ? tb_walk_kernel<REP, TS, 1, true, true> : tb_walk_kernel<REP, TS, 1, false, true>;
}
template <int REP> WalkKernel pick_tile(int ts, int rpl, bool staged, bool cached, bool turn) {
  switch (ts) {
  case 1: return pick<REP, 1>(rpl, staged, cached, turn);
  case 2: return pick<REP, 2>(rpl, staged, cached, turn);
  case 3: return pick<REP, 3>(rpl, staged, cached, turn);
  default: return pick<REP, 4>(rpl, staged, cached, turn);
  }
}
} // namespace

WalkKernel walk_kernel(int representation, int tile_size, int rows_per_lane, bool staged, bool cached, bool turn) {
  switch (representation) { // (reorg: single nodes)
  case 0: return pick_tile<0>(tile_size, rows_per_lane, staged, cached, turn);
  case 1: return pick_tile<1>(tile_size, rows_per_lane, staged, cached, turn);
  default: return pick<2, 1>(rows_per_lane, staged, cached, turn);
  }
}

} // namespace tb
