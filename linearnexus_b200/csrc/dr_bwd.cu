// Translation unit of the backward.
#include "dr_bwd.cuh"
