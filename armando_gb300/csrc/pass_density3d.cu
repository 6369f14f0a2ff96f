// The density pass in 3 dimensions.
#include "pass_density.cuh"

template void launch_density<3>(armando_ctx*, const unsigned*, const StepArgs&);
