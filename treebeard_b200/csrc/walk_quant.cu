// The walk over rounded keys of wide rows, compiled apart: its speed depends on where its code, and that of the exact
// re-walks it calls, come to lie, and an edit of any kernel compiled with it moved them: 262144 x 2000 took 1391 to 1438 us
// with one and the same kernel, and takes 1380 by itself.
#include "walk_quant.cuh"

namespace tb {

QuantKernel wide_quant_kernel(int depth, bool leaf_ids) {
  return depth == 8   ? (leaf_ids ? tb_walk_quant_kernel<8, true> : tb_walk_quant_kernel<8, false>)
         : depth == 6 ? (leaf_ids ? tb_walk_quant_kernel<6, true> : tb_walk_quant_kernel<6, false>)
                      : (leaf_ids ? tb_walk_quant_kernel<0, true> : tb_walk_quant_kernel<0, false>);
}

} // namespace tb
