// bs_run_amber.cu -- k_run for one steric form.

#include "bs_run.cuh"

namespace bsg
{

const void *run_amber(int lanes, bool lean, int hold) { return run_form<BS_STERIC_LJ_12_6_AMBER>(lanes, lean, hold); }

} // namespace bsg
