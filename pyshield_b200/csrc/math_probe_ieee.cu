// math_probe.cu's functions in a unit that keeps IEEE rounding.
#define SHIELD_IEEE
#define PROBE_MATH shield_probe_math_ieee
#include "math_probe.cu"
