// gpufft-b200: the FP32 tile passes (gf_tile_pass.cuh).
#include "gf_tile_pass_launch.cuh"

namespace gfb
{
template <> int launch_tile_pass<float>(const PassArgs<float>& a, bool fwd, int LT, cudaStream_t s)
{
    return launch_tile_pass_t<float>(a, fwd, LT, s);
}
} // namespace gfb
