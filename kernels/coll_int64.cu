// Collective kernel instantiations for 64-bit integers (operator chosen at run time).
#include "coll_launch.cuh"
namespace Al { namespace internal { namespace device {
void launch_coll_int64(const CollParams& P, DType dt, const LaunchCfg& cfg) {
  switch (dt) {
    case DType::i64: launch_int<long long>(P, cfg); break;
    case DType::u64: launch_int<unsigned long long>(P, cfg); break;
    default: throw_al_exception("not an integer datatype: ", dtype_name(dt));
  }
}
}}}
