// Plan-driven depth-map passes, two-float.
#include "dm_generic_host.cuh"

namespace oh {
OH_DM_GENERIC(ff)
}
