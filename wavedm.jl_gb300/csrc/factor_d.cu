// Two-factor passes for axis lengths 192.
#include "factor_instantiate.cuh"
WDM_FACTORS(192)
