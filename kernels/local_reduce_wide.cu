// fp64 and integer reductions between buffers on this GPU.
#include "local_reduce.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {
template <typename T>
bool run(const LocalReduceParams& P, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream) {
  switch (op) {
    case ReductionOperator::sum:
    case ReductionOperator::avg: local_reduce_launch<T, T>(P, RedSum(), max_ctas, threads, stream); return true;
    case ReductionOperator::max: local_reduce_launch<T, T>(P, RedMax(), max_ctas, threads, stream); return true;
    case ReductionOperator::min: local_reduce_launch<T, T>(P, RedMin(), max_ctas, threads, stream); return true;
    default: return false;
  }
}
}  // namespace

bool local_reduce_wide(const LocalReduceParams& P, DType dt, ReductionOperator op, int max_ctas, int threads, cudaStream_t stream) {
  if (dt == DType::f64) return run<double>(P, op, max_ctas, threads, stream);
  if (dt == DType::i32) return run<int32_t>(P, op, max_ctas, threads, stream);
  if (dt == DType::i64) return run<int64_t>(P, op, max_ctas, threads, stream);
  return false;
}

}  // namespace device
}  // namespace internal
}  // namespace Al
