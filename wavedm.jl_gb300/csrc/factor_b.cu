// Two-factor passes for axis lengths 32, 48, 64.
#include "factor_instantiate.cuh"
WDM_FACTORS(32)
WDM_FACTORS(48)
WDM_FACTORS(64)
