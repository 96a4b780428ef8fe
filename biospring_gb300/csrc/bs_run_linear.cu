// bs_run_linear.cu -- k_run for one steric form.

#include "bs_run.cuh"

namespace bsg
{

const void *run_linear(int lanes, bool lean, int hold) { return run_form<BS_STERIC_LINEAR>(lanes, lean, hold); }

} // namespace bsg
