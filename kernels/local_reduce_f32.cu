// fp32 reductions between buffers on this GPU (also with a 16-bit type between GPUs, whose roundings are kept).
#include "local_reduce.cuh"

namespace Al {
namespace internal {
namespace device {

bool local_reduce_f32(const LocalReduceParams& P, DType wire, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream) {
  const bool sum = op == ReductionOperator::sum || op == ReductionOperator::avg;
  if (sum && wire == DType::bf16) local_reduce_launch<float, __nv_bfloat16>(P, RedSum(), max_ctas, threads, stream);
  else if (sum && wire == DType::f16) local_reduce_launch<float, __half>(P, RedSum(), max_ctas, threads, stream);
  else if (sum && wire == DType::f32) local_reduce_launch<float, float>(P, RedSum(), max_ctas, threads, stream);
  else if (op == ReductionOperator::max && wire == DType::f32) local_reduce_launch<float, float>(P, RedMax(), max_ctas, threads, stream);
  else if (op == ReductionOperator::min && wire == DType::f32) local_reduce_launch<float, float>(P, RedMin(), max_ctas, threads, stream);
  else return false;
  return true;
}

bool launch_local_reduce(const LocalReduceParams& P, DType user, DType wire, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream) {
  if (user == DType::f32) return local_reduce_f32(P, wire, op, max_ctas, threads, stream);
  if (user != wire) return false;
  return local_reduce_16bit(P, user, op, max_ctas, threads, stream) || local_reduce_wide(P, user, op, max_ctas, threads, stream);
}

}  // namespace device
}  // namespace internal
}  // namespace Al
