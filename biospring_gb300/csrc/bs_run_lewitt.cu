// bs_run_lewitt.cu -- k_run for one steric form.

#include "bs_run.cuh"

namespace bsg
{

const void *run_lewitt(int lanes, bool lean, int hold) { return run_form<BS_STERIC_LJ_8_6_LEWITT>(lanes, lean, hold); }

} // namespace bsg
