// Collective kernel instantiations for 32-bit integers (operator chosen at run time).
#include "coll_launch.cuh"
namespace Al { namespace internal { namespace device {
void launch_coll_int32(const CollParams& P, DType dt, const LaunchCfg& cfg) {
  switch (dt) {
    case DType::i32: launch_int<int>(P, cfg); break;
    case DType::u32: launch_int<unsigned int>(P, cfg); break;
    default: throw_al_exception("not an integer datatype: ", dtype_name(dt));
  }
}
}}}
