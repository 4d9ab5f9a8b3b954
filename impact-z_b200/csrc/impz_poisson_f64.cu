// Poisson solve, double convolution.
#include <cmath>
#define IMPZ_POISSON_T double
#include "impz_poisson_impl.cuh"
