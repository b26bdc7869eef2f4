#include "cb_march.cuh"
CB_MARCH_DEFINE(float)
