// internal.h -- what the facade classes use besides the C ABI; not visible outside the library.
#pragma once
#include "../../include/cudarl.h"

namespace cudarl {

struct SingleStep { int32_t x, y; float reward; bool done; };
// cudarl_step_actions (or cudarl_reset_all) of a context with one environment, with the environment's position: one launch, one wait, and the
// caller's own work between the two.
int step_single_begin(cudarl_ctx* ctx, bool reset, int32_t action);
int step_single_end(cudarl_ctx* ctx, SingleStep* out);

}  // namespace cudarl
