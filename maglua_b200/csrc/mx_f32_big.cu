#include "mx.cuh"
template struct mlb::MxUnit<float, true>;
