// Collective kernel instantiations for 16-bit integers (operator chosen at run time).
#include "coll_launch.cuh"
namespace Al { namespace internal { namespace device {
void launch_coll_int16(const CollParams& P, DType dt, const LaunchCfg& cfg) {
  switch (dt) {
    case DType::i16: launch_int<short>(P, cfg); break;
    case DType::u16: launch_int<unsigned short>(P, cfg); break;
    default: throw_al_exception("not an integer datatype: ", dtype_name(dt));
  }
}
}}}
