// Two-factor passes for axis lengths 384.
#include "factor_instantiate.cuh"
WDM_FACTORS(384)
