// Poisson solve, float convolution.
#include <cmath>
#define IMPZ_POISSON_T float
#include "impz_poisson_impl.cuh"
