// Collective kernel instantiations for integer elements (operator chosen at run time), dispatched to one file per width.
#include "coll_launch.cuh"
namespace Al { namespace internal { namespace device {
void launch_coll_int(const CollParams& P, DType dt, const LaunchCfg& cfg) {
  switch (dtype_size(dt)) {
    case 1: launch_coll_int8(P, dt, cfg); break;
    case 2: launch_coll_int16(P, dt, cfg); break;
    case 4: launch_coll_int32(P, dt, cfg); break;
    default: launch_coll_int64(P, dt, cfg); break;
  }
}
}}}
