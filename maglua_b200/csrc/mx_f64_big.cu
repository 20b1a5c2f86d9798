#include "mx.cuh"
template struct mlb::MxUnit<double, true>;
