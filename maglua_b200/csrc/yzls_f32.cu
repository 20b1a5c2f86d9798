#include "yzls.cuh"
template struct mlb::YzUnit<float2>;
