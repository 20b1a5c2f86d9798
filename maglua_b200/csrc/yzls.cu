// yzls.cu -- the sizes that the power-of-two (y,z) pass with the layer sum takes, and
// its dispatch by state precision (the pass: yzls.cuh).
#include "fftreg.cuh"
#include "kparams.h"
#include "launch.h"

#include <cuda_runtime.h>

#include <vector>

namespace mlb {

// place of each y frequency after the forward transform
template <int PY>
static void places(std::vector<int>& at)
{
    constexpr int T = fr::Split<PY>::T, E = fr::Split<PY>::E;
    at.resize(PY);
    for (int k = 0; k < PY; k++) at[k] = (k % E) * T + k / E;
}

bool yz_ls_plan(const ConvK& c, int rb, std::vector<int>& at)
{
    if (c.general || !(rb == 8 ? YzUnit<double2>::takes(c.Py, c.nz) : YzUnit<float2>::takes(c.Py, c.nz))) return false;
    switch (c.Py) {
    case 16: places<16>(at); break;
    case 32: places<32>(at); break;
    case 64: places<64>(at); break;
    case 128: places<128>(at); break;
    case 256: places<256>(at); break;
    case 512: places<512>(at); break;
    }
    return true;
}

cudaError_t launch_yz_ls(const ConvK& c, const FftLen L[3], const void* tw, void* spec, const void* tz, int rb,
                         cudaStream_t st)
{
    Prof pf("k_conv_yz", st);
    if (rb == 8)
        return YzUnit<double2>::pass(c, static_cast<const double2*>(tw) + L[1].tw_off, static_cast<double2*>(spec),
                                     static_cast<const double*>(tz), st);
    return YzUnit<float2>::pass(c, static_cast<const float2*>(tw) + L[1].tw_off, static_cast<float2*>(spec),
                                static_cast<const float*>(tz), st);
}

cudaError_t yz_ls_init()
{
    const cudaError_t e = YzUnit<float2>::init();
    return e != cudaSuccess ? e : YzUnit<double2>::init();
}

} // namespace mlb
