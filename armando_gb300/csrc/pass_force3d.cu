// The force pass in 3 dimensions.
#include "pass_force.cuh"

template void launch_force<3>(armando_ctx*, const unsigned*, const StepArgs&);
