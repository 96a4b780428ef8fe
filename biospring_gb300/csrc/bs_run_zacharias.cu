// bs_run_zacharias.cu -- k_run for one steric form.

#include "bs_run.cuh"

namespace bsg
{

const void *run_zacharias(int lanes, bool lean, int hold) { return run_form<BS_STERIC_LJ_8_6_ZACHARIAS>(lanes, lean, hold); }

} // namespace bsg
