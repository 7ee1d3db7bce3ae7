// pass_fx.cu -- the double build's pass kernels in block fixed point: one
// kernel per power-of-two pass length (fx_spec.cuh) and one for every other
// register tile (fx_tile.cuh).  Built in parts (KFFT_FX_PART) that compile in
// parallel.
#include "fx_spec.cuh"

namespace kfft {
#if !defined(KFFT_HALF_SCALAR)

#ifndef KFFT_FX_PART
#define KFFT_FX_PART 0
#endif

using FxKernel = void (*)(PassDesc, PassExtra);

// Bound by integer issue and latency.  Two CTAs of 512 threads an SM (64
// registers): 256 x 4096 points forward + inverse 52.6 us, against 90 us with
// radix-16 stages at 128 registers and run-time lengths, and 213 us for the
// FP64 body, whose FP64 pipe was 72% busy.  The error against long double
// falls from 2.2e-16 to 0.6e-16 (geometric mean over 45 lengths).

template <uint32_t R>
__global__ void __launch_bounds__(kFxSpecThreads, 2) k_fx_spec(const __grid_constant__ PassDesc d,
                                                               const __grid_constant__ PassExtra x) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const FxLeft left = fx_spec_tile<R>(d, blockIdx.x, smem_raw);
    if (left != FX_NOTHING) fp64_tile(d, x, blockIdx.x, smem_raw, left);
}

#if KFFT_FX_PART == 0
#ifndef KFFT_FX_BLOCKS
#define KFFT_FX_BLOCKS 3
#endif
#ifndef KFFT_FX_WIDE_BLOCKS
#define KFFT_FX_WIDE_BLOCKS 2
#endif
// Run-time tiles: 256 threads, three CTAs an SM (80 registers; 16384 x 1000
// points 416 us, 502 with two CTAs, 408 with four, but 4096 x 4000 794 against
// 837); tiles whose exchange in one buffer takes more threads (above 2048
// points or so) two CTAs of up to 512 (4096 x 4000 494 us, 612 with one CTA of
// 128 registers, 794 with two buffers and 256 threads).
template <uint32_t T, int BLOCKS>
__global__ void __launch_bounds__(T, BLOCKS) k_pass_fx(const __grid_constant__ PassDesc d,
                                                       const __grid_constant__ PassExtra x) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double_tile(d, x, blockIdx.x, smem_raw);
}

// Passes of 2 and 4 points: in doubles, one butterfly a thread, straight from
// global memory to global memory.
template <bool INV>
__global__ void __launch_bounds__(kFxWideThreads) k_pass_short(const __grid_constant__ PassDesc d,
                                                             const __grid_constant__ PassExtra x) {
    const uint32_t lane0 = blockIdx.x * d.C, total = d.batch * d.lanes_j;
    if (d.R == 2) fused_pass<2, INV, STORE_ANY, false>(d, x.step[0], nullptr, nullptr, lane0, total, IO_GLOBAL, IO_GLOBAL);
    else fused_pass<4, INV, STORE_ANY, false>(d, x.step[0], nullptr, nullptr, lane0, total, IO_GLOBAL, IO_GLOBAL);
}

FxKernel fx_kernels_1(uint32_t spec);
FxKernel fx_kernels_2(uint32_t spec);
FxKernel fx_kernels_3(uint32_t spec);

void launch_pass_reg(const PassDesc& d, const PassExtra& x, cudaStream_t st) {
    struct Kernels {
        FxKernel f[13];
        cudaError_t error;
    };
    // one-time shared-memory limits (thread-safe; a failure is reported on every call)
    static const Kernels k = [] {
        Kernels v;
        v.error = cudaSuccess;
        for (uint32_t s = 0; s < 13; ++s) {
            v.f[s] = s < 4 ? nullptr : fx_kernels_1(s);
            if (s >= 4 && !v.f[s]) v.f[s] = fx_kernels_2(s);
            if (s >= 4 && !v.f[s]) v.f[s] = fx_kernels_3(s);
        }
        v.f[0] = k_pass_fx<kPassThreads, KFFT_FX_BLOCKS>;
        v.f[1] = k_pass_fx<kFxWideThreads, KFFT_FX_WIDE_BLOCKS>;
        for (FxKernel f : v.f) {
            if (!f) continue;
            const cudaError_t e = cudaFuncSetAttribute(
                (const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (e != cudaSuccess) {
                cudaGetLastError();
                v.error = e;
            }
        }
        return v;
    }();
    if (k.error != cudaSuccess) {
        note_cuda_error(k.error);
        return;
    }
    if (!d.fx && d.nrad == 1) {
        if (d.inv) k_pass_short<true><<<d.tiles, d.threads, 0, st>>>(d, x);
        else k_pass_short<false><<<d.tiles, d.threads, 0, st>>>(d, x);
    } else {
        k.f[d.spec ? d.spec : (d.threads > kPassThreads ? 1 : 0)]<<<d.tiles, d.threads, d.smem_bytes, st>>>(d, x);
    }
    note_cuda_error(cudaGetLastError());
    count_launch();
}
#elif KFFT_FX_PART == 1
FxKernel fx_kernels_1(uint32_t spec) {
    return spec == 4 ? k_fx_spec<16> : spec == 5 ? k_fx_spec<32> : spec == 6 ? k_fx_spec<64> : nullptr;
}
#elif KFFT_FX_PART == 2
FxKernel fx_kernels_2(uint32_t spec) {
    return spec == 7 ? k_fx_spec<128> : spec == 8 ? k_fx_spec<256> : spec == 9 ? k_fx_spec<512> : nullptr;
}
#else
FxKernel fx_kernels_3(uint32_t spec) {
    return spec == 10 ? k_fx_spec<1024> : spec == 11 ? k_fx_spec<2048> : spec == 12 ? k_fx_spec<4096> : nullptr;
}
#endif

#endif
}  // namespace kfft
