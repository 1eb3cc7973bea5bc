// tb_bsc.h -- block-sparse plan internals shared with the batching layer.
#pragma once
#include <cstddef>

#include "../../include/talsh_b200.h"

namespace tb {

// Device bytes of a plan's operand and residue planes.
size_t bsc_plan_bytes(const tb_bsc_plan_t* plan);

}  // namespace tb
