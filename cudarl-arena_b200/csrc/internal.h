// internal.h -- what the facade classes use besides the C ABI; not visible outside the library.
#pragma once
#include "../../include/cudarl.h"

namespace cudarl {

struct SingleStep { int32_t x, y; float reward; bool done; };
// cudarl_step_actions (or cudarl_reset_all) of a context with one environment, with the environment's position: one launch, one wait.
int step_single(cudarl_ctx* ctx, bool reset, int32_t action, SingleStep* out);

}  // namespace cudarl
