// The density pass in 2 dimensions.
#include "pass_density.cuh"

template void launch_density<2>(armando_ctx*, const unsigned*, const StepArgs&);
