// Collective kernel instantiations for 8-bit integers (operator chosen at run time).
#include "coll_launch.cuh"
namespace Al { namespace internal { namespace device {
void launch_coll_int8(const CollParams& P, DType dt, const LaunchCfg& cfg) {
  switch (dt) {
    case DType::i8: launch_int<signed char>(P, cfg); break;
    case DType::u8: launch_int<unsigned char>(P, cfg); break;
    default: throw_al_exception("not an integer datatype: ", dtype_name(dt));
  }
}
}}}
