// fp64_tile.cu -- the double build's IEEE arithmetic register tiles, for the
// tiles its fixed-point kernels turn down (an infinity, a NaN, magnitudes
// near the ends of the exponent range, small parts that doubles keep apart
// from large ones) or for the lanes of a tile that are like that.  One copy,
// linked to every kernel that needs it, compiled for 64 registers.
#include "fft_device.cuh"
#include "fx_spec.cuh"

namespace kfft {
#if !defined(KFFT_HALF_SCALAR)

// The lanes' elements are read again.  Behind the rows of words one for what
// each lane holds and a bit an element that is near its lane's largest.
__device__ __noinline__ FxLeft fx_spec_look(const PassDesc& d, uint32_t R, uint32_t* words, uint32_t lane0,
                                            uint32_t total, int span) {
    constexpr int U = 4;  // loads in flight together
    const uint32_t log = d.spec, bits = (R + 31) / 32;
    uint32_t* holds = words + (kFxRows + 1) * d.C;
    uint32_t* big = holds + d.C;
    const bool lane_mode = d.load_mode == MODE_LANE;
    // rows of 32 elements or more, element by element: a warp has one lane's and
    // a word of bits (whole warps: C * R and the threads are multiples of 32)
    const bool by_warp = R >= 32 && !lane_mode;
    const uint32_t elems = d.pro_op == PRO_CHIRP ? 0u : d.C * R;  // (a chirp turns every element)
#pragma unroll 1
    for (uint32_t i0 = threadIdx.x; i0 < elems; i0 += U * blockDim.x) {
        double2 x[U];
        uint32_t at[U];  // the element's bit, lane by lane (none: past the last)
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = i0 + u * blockDim.x;
            const uint32_t r = lane_mode ? fdiv(i, d.div_C) : i & (R - 1);
            const uint32_t c = lane_mode ? i - r * d.C : i >> log;
            x[u] = {0.0, 0.0};
            at[u] = 0xffffffffu;
            if (i < elems) {
                at[u] = (c << log) + r;
                if (lane0 + c < total) {
                    uint32_t b, j;
                    fx_lane(d, lane0 + c, b, j);
                    uint32_t n = j + r * d.lanes_j;
                    if (d.pro_op == PRO_GATHER) n = __ldg(&d.pro_perm[n]);
                    x[u] = __ldcg(&d.in[uint64_t(b) * d.in_bs + uint64_t(n) * d.in_es]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (at[u] == 0xffffffffu) break;  // (whole warps)
            const uint32_t c = at[u] >> log, r = at[u] & (R - 1);
            const uint32_t from = fx_near(words[c], span);
            uint32_t f = fx_holds(x[u], from);
            const bool near = max(fx_mag(x[u].x), fx_mag(x[u].y)) >= from;
            if (by_warp) {
                f = __reduce_or_sync(0xffffffffu, f);
                const uint32_t w = __ballot_sync(0xffffffffu, near);
                if ((threadIdx.x & 31) == 0) {
                    if (f) atomicOr(&holds[c], f);
                    big[c * bits + r / 32] = w;
                }
            } else {
                if (f) atomicOr(&holds[c], f);
                if (near) atomicOr(&big[c * bits + r / 32], 1u << (r % 32));
            }
        }
    }
    __syncthreads();
    return fx_settle(d, words, holds, lane0, total, [&](uint32_t c) {
        const uint32_t* w = big + c * bits;
        for (uint32_t k = 0; k < bits; ++k) {
            // bit r with bit r + 1 (the first one behind the last)
            const uint32_t up = w[k + 1 < bits ? k + 1 : 0] & 1u;
            if (w[k] & ((w[k] >> 1) | up << (R < 32 ? R - 1 : 31))) return true;
        }
        return false;
    });
}

// The stages of fx_spec_tile in doubles: radix 8 with 8 points a thread, which
// fits the 64 registers of its kernels.  The run-time body with its stages of
// up to 16 spilled there and took, forward, with every tile in FP64, 145 us for
// 256 x 4096 points (105 before the fixed-point tiles), 380 (275) for 4096 x
// 1024 and 809 (577) for 16 x 2^18.  `only` as in fused_pass.
template <uint32_t R, uint32_t NS, bool INV>
__device__ __forceinline__ void fp64_spec_later(const PassDesc& d, double2* buf, uint32_t lane0,
                                                uint32_t total, const uint32_t* only) {
    constexpr int P = fx_spec_radix(R, NS);
    constexpr int G = 8 / P;
    constexpr uint32_t M = R / P, TWS = R / (NS * P);
    constexpr bool kLast = NS * P == R;
    const uint32_t items = d.C * M;
    const bool lane_mode = !only && kLast && d.store_mode == MODE_LANE;
    uint32_t c[G], jj[G];
    bool on[G];
    double2 v[G][P];
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t it = min(threadIdx.x + g * blockDim.x, items - 1);
        jj[g] = lane_mode ? fdiv(it, d.div_C) : it % M;
        c[g] = lane_mode ? it - jj[g] * d.C : it / M;
        on[g] = threadIdx.x + g * blockDim.x < items && (!only || only[c[g]]);
        if (!on[g]) continue;
        const double2* s = buf + c[g] * d.lane_stride;
#pragma unroll
        for (int q = 0; q < P; ++q) v[g][q] = s[pad(jj[g] + q * M)];
        apply_inner_twiddles<P>(v[g], d.tw_inner, (jj[g] % NS) * TWS);
        dft<P, INV>(v[g]);
    }
    if constexpr (!kLast) __syncthreads();
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (!on[g]) continue;
        const uint32_t ob = jj[g] % NS + (jj[g] / NS) * (NS * P);
        if constexpr (kLast) {
            if (lane0 + c[g] >= total) continue;
            uint32_t b, j;
            fx_lane(d, lane0 + c[g], b, j);
            fused_store<P>(d, b, j, ob, NS, v[g]);
        } else {
            double2* o = buf + c[g] * d.lane_stride;
#pragma unroll
            for (int q = 0; q < P; ++q) o[pad(ob + q * NS)] = v[g][q];
        }
    }
    if constexpr (!kLast) fp64_spec_later<R, NS * P, INV>(d, buf, lane0, total, only);
}

// The other lanes of a tile that leaves some, in fixed point.
template <uint32_t R>
__device__ __noinline__ void fx_spec_others(const PassDesc& d, uint32_t tile, unsigned char* smem) {
    __syncthreads();
    fx_spec_tile<R, true>(d, tile, smem);
    __syncthreads();
}

template <uint32_t R, bool INV>
__device__ __noinline__ void fp64_spec_tile(const PassDesc& d, uint32_t tile, unsigned char* smem,
                                            const uint32_t* only) {
    constexpr int P = fx_spec_radix(R, 1);
    constexpr int G = 8 / P;
    constexpr uint32_t M = R / P;
    const uint32_t total = d.batch * d.lanes_j, lane0 = tile * d.C, items = d.C * M;
    double2* buf = reinterpret_cast<double2*>(smem);
    const bool lane_mode = !only && d.load_mode == MODE_LANE;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t it = threadIdx.x + g * blockDim.x;
        if (it >= items) continue;
        const uint32_t jj = lane_mode ? fdiv(it, d.div_C) : it % M;
        const uint32_t c = lane_mode ? it - jj * d.C : it / M;
        if (only && !only[c]) continue;
        double2 v[P];
#pragma unroll
        for (int q = 0; q < P; ++q) v[q] = {0.0, 0.0};
        if (lane0 + c < total) {
            uint32_t b, j;
            fx_lane(d, lane0 + c, b, j);
            fused_load<P>(d, b, j, jj, M, v);
        }
        dft<P, INV>(v);
        double2* o = buf + c * d.lane_stride;
#pragma unroll
        for (int q = 0; q < P; ++q) o[pad(jj * P + q)] = v[q];
    }
    fp64_spec_later<R, P, INV>(d, buf, lane0, total, only);
}

template <uint32_t R>
__device__ __forceinline__ void fp64_spec(const PassDesc& d, uint32_t tile, unsigned char* smem,
                                          const uint32_t* only) {
    if (only) fx_spec_others<R>(d, tile, smem);
    if (d.inv) fp64_spec_tile<R, true>(d, tile, smem, only);
    else fp64_spec_tile<R, false>(d, tile, smem, only);
}

__device__ __noinline__ void fp64_tile(const PassDesc& d, const PassExtra& x, uint32_t tile,
                                       unsigned char* smem, FxLeft left) {
    // the lanes left over (in words behind the exchange buffers)
    const uint32_t* only = left == FX_SOME ? fx_left_row(d, smem) : nullptr;
    switch (d.spec) {
        case 4: fp64_spec<16>(d, tile, smem, only); return;
        case 5: fp64_spec<32>(d, tile, smem, only); return;
        case 6: fp64_spec<64>(d, tile, smem, only); return;
        case 7: fp64_spec<128>(d, tile, smem, only); return;
        case 8: fp64_spec<256>(d, tile, smem, only); return;
        case 9: fp64_spec<512>(d, tile, smem, only); return;
        case 10: fp64_spec<1024>(d, tile, smem, only); return;
        case 11: fp64_spec<2048>(d, tile, smem, only); return;
        case 12: fp64_spec<4096>(d, tile, smem, only); return;
        default: break;
    }
    vec2_t* sm = reinterpret_cast<vec2_t*>(smem);
    if (only) __syncthreads();  // (every thread has written the other lanes)
    if (d.inv) tile_body_reg<true, false, false>(d, x, tile, sm, only);
    else tile_body_reg<false, false, false>(d, x, tile, sm, only);
}
#endif
}  // namespace kfft
