// Two-factor passes for axis lengths 96, 128.
#include "factor_instantiate.cuh"
WDM_FACTORS(96)
WDM_FACTORS(128)
