// Two-factor passes for axis lengths 8, 12, 16, 24.
#include "factor_instantiate.cuh"
WDM_FACTORS(8)
WDM_FACTORS(12)
WDM_FACTORS(16)
WDM_FACTORS(24)
