// The force pass in 2 dimensions.
#include "pass_force.cuh"

template void launch_force<2>(armando_ctx*, const unsigned*, const StepArgs&);
