// The walk over batches of rounded-key tiles, compiled apart (as walk_quant.cu).
#include "walk_quant_batch.cuh"

namespace tb {

QuantKernel batch_quant_kernel(int depth, bool leaf_ids, bool multi) {
  if (multi)
    return depth == 8 ? (leaf_ids ? tb_walk_quant_batch_kernel<8, true, true> : tb_walk_quant_batch_kernel<8, false, true>)
                      : (leaf_ids ? tb_walk_quant_batch_kernel<0, true, true> : tb_walk_quant_batch_kernel<0, false, true>);
  return depth == 8   ? (leaf_ids ? tb_walk_quant_batch_kernel<8, true, false> : tb_walk_quant_batch_kernel<8, false, false>)
         : depth == 6 ? (leaf_ids ? tb_walk_quant_batch_kernel<6, true, false> : tb_walk_quant_batch_kernel<6, false, false>)
                      : (leaf_ids ? tb_walk_quant_batch_kernel<0, true, false> : tb_walk_quant_batch_kernel<0, false, false>);
}

} // namespace tb
