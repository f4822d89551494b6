// Plan-driven depth-map passes, float.
#include "dm_generic_host.cuh"

namespace oh {
OH_DM_GENERIC(float)
}
