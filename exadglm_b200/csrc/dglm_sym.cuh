// Device code of the symmetry-adapted kernels for the units that use it (the
// single-mesh stages and the batches).
#pragma once

#include <cuda_runtime.h>

#include "dglm_common.cuh"
#include "dglm_ptx.cuh"
#include "dglm_ring.h"

namespace dglm {

#include "dglm_stage_sym.cuh"
#include "dglm_stage_sym_adv.cuh"

}  // namespace dglm
