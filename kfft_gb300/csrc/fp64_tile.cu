// fp64_tile.cu -- the double build's IEEE arithmetic register tile, for the
// tiles its fixed-point kernels turn down (an infinity, a NaN, magnitudes
// near the ends of the exponent range).  One copy, linked to every kernel
// that needs it, compiled for 64 registers (it may spill: it hardly ever
// runs).
#include "fft_device.cuh"
#include "fx_tile.cuh"

namespace kfft {
#if !defined(KFFT_HALF_SCALAR)
__device__ __noinline__ void fp64_tile(const PassDesc& d, const PassExtra& x, uint32_t tile,
                                       unsigned char* smem) {
    vec2_t* sm = reinterpret_cast<vec2_t*>(smem);
    if (d.inv) tile_body_reg<true, false, false>(d, x, tile, sm);
    else tile_body_reg<false, false, false>(d, x, tile, sm);
}
#endif
}  // namespace kfft
