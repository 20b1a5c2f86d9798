#include "xstep.cuh"
template struct mlb::XUnit<128>;
