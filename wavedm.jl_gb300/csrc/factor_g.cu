// Two-factor passes for axis lengths 512.
#include "factor_instantiate.cuh"
WDM_FACTORS(512)
