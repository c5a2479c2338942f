// Two-factor passes for axis lengths 256.
#include "factor_instantiate.cuh"
WDM_FACTORS(256)
