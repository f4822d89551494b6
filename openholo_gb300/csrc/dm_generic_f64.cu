// Plan-driven depth-map passes, double.
#include "dm_generic_host.cuh"

namespace oh {
OH_DM_GENERIC(double)
}
