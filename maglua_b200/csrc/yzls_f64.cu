#include "yzls.cuh"
template struct mlb::YzUnit<double2>;
