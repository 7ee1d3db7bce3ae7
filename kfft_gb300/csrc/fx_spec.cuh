// fx_spec.cuh -- compile-time power-of-two tiles of the double build in fixed
// point: as fx_tile (fx_tile.cuh), with the pass length known to the
// compiler, radix-8 stages with 8 points a thread (64 registers a thread, 32
// warps an SM), the first stage fed from global memory and the last one
// written to it, and one exchange buffer.
#pragma once

#include "fx_tile.cuh"

#if !defined(KFFT_HALF_SCALAR)

namespace kfft {

// The radix of the stage that follows stages multiplying to NS: 8, then 4s
// (16 left: 4 and 4) or a 2.
constexpr int fx_spec_radix(uint32_t R, uint32_t NS) {
    const uint32_t rest = R / NS;
    return rest == 16 || rest == 4 ? 4 : (rest % 8 == 0 ? 8 : int(rest));
}

constexpr uint32_t kFxPad = 1u << kPadShift;  // slots between padding slots

// Sum of (2 - shift) over the stages from NS on: the change of a lane's
// exponent from the first stage's values to the last one's.
template <uint32_t R, uint32_t NS, int IDX>
__device__ __forceinline__ int fx_spec_shifts(const uint32_t* words, uint32_t C, uint32_t c) {
    if constexpr (NS == R) {
        return 0;
    } else {
        constexpr int P = fx_spec_radix(R, NS);
        return 2 - fx_norm(words[IDX * C + c], P) + fx_spec_shifts<R, NS * P, IDX + 1>(words, C, c);
    }
}

// One butterfly's outputs of the last stage through the epilogue (fx_write's
// element operations).
template <int P>
__device__ __forceinline__ void fx_spec_store(const PassDesc& d, uint32_t g, uint32_t ob, uint32_t ns,
                                              int eb, const cfx_t* v) {
    uint32_t b, j;
    fx_lane(d, g, b, j);
    const bool inv = d.inv != 0;
    const uint32_t op = d.epi_op;
    const bool table = op == EPI_MUL || op == EPI_CHIRP || op == EPI_RADER_FWD;
    const bool scaled = op == EPI_NONE || op == EPI_CHIRP;
    const int32_t sh = scaled ? d.fx_scale_h : 0, sl = d.fx_scale_l;
    const int e_out = eb + (scaled ? d.fx_scale_e : 0) + (sh ? 2 : 0) + (table ? 2 : 0) +
                      (table && op != EPI_CHIRP ? d.fx_epi_e : 0);
    const uint32_t blk = fdiv(j, d.div_Ns);
    const uint32_t k0 = blk * d.Ns * d.R + (j - blk * d.Ns) + ob * d.Ns, ks = ns * d.Ns;
    double2* out = d.out + uint64_t(b) * d.out_bs;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        const uint32_t k = k0 + q * ks;
        cfx_t u = inv ? cfx_t{v[q].y, v[q].x} : v[q];
        if (table) {
            if (op == EPI_CHIRP && k >= d.epi_bound) continue;
            if (op == EPI_RADER_FWD && k == 0) {
                store_elem(d, b, 0, double2{fx_to_double(u.x, eb), fx_to_double(u.y, eb)});
                continue;
            }
            u = fx_cmul(u, fx_tw_load(&d.fx_epi[k]), d.fx_one);
        }
        if (sh) {
            const FxLimbs x = fx_limbs(u.x), y = fx_limbs(u.y);
            u.x = fx_add_high(fx_mad(x.l, sh, fx_mul(x.h, sl)), fx_mul(x.h, sh), d.fx_one);
            u.y = fx_add_high(fx_mad(y.l, sh, fx_mul(y.h, sl)), fx_mul(y.h, sh), d.fx_one);
        }
        double2 r = {fx_to_double(u.x, e_out), fx_to_double(u.y, e_out)};
        double2* o = out;
        uint64_t at = uint64_t(k) * d.out_es;
        if (op == EPI_RADER_INV) {
            o = d.aux_out + uint64_t(b) * d.aux_out_bs;
            at = uint64_t(__ldg(&d.epi_perm[k])) * d.aux_out_es;
            r = cadd(r, d.aux_in[2 * uint64_t(b)]);
            if ((d.fx_scale_h | d.fx_scale_e) != 0) r = cscale(r, d.scale);  // scale != 1
            if (k == 0) o[0] = cscale(__ldcg(&d.aux_in[2 * uint64_t(b) + 1]), d.scale);
        } else if (op == EPI_MUL_OUT) {
            r = cscale(cmul(r, __ldcg(&d.epi_tab[uint64_t(b) * d.out_bs + at])), d.scale);
        }
        o[at] = r;
    }
}

// Writes a stage's outputs to the exchange buffer and their bits to `words`.
template <int P, int G, uint32_t R, uint32_t NS>
__device__ __forceinline__ void fx_spec_exchange(const PassDesc& d, cfx_t* buf, uint32_t* words,
                                                 const uint32_t* c, const uint32_t* jj,
                                                 cfx_t (*v)[P], bool lane_mode) {
    constexpr uint32_t M = R / P;
    const uint32_t items = d.C * M;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t it = threadIdx.x + g * blockDim.x;
        uint32_t b = it < items ? fx_bits<P>(v[g]) : 0u;
        if (it < items) {
            // padding keeps the P slots equally far apart where the distance is
            // whole pad periods, or all of them lie in one
            constexpr bool kLin = NS % kFxPad == 0 || (NS == 1 && kFxPad % P == 0);
            constexpr uint32_t kStep = NS + (NS >> kPadShift);
            const uint32_t ob = jj[g] % NS + (jj[g] / NS) * (NS * P);
            cfx_t* o = buf + c[g] * d.lane_stride + (kLin ? pad(ob) : 0u);
#pragma unroll
            for (int q = 0; q < P; ++q) o[kLin ? q * kStep : pad(ob + q * NS)] = v[g][q];
        }
        if (M % 32 == 0 && !lane_mode) {  // the warp's butterflies are all of one lane
            b = __reduce_or_sync(0xffffffffu, b);
            if ((threadIdx.x & 31) == 0 && b) atomicOr(&words[c[g]], b);
        } else if (it < items) {
            atomicOr(&words[c[g]], b);
        }
    }
}

// The stage after stages multiplying to NS > 1, and those after it.  OTHERS: the
// lanes left to the FP64 body are not stored.
template <uint32_t R, uint32_t NS, int IDX, bool OTHERS>
__device__ __forceinline__ void fx_spec_later(const PassDesc& d, cfx_t* buf, uint32_t* words,
                                              uint32_t lane0, uint32_t total) {
    constexpr int P = fx_spec_radix(R, NS);
    constexpr int G = 8 / P;
    constexpr uint32_t M = R / P, TWS = R / (NS * P);
    constexpr bool kLast = NS * P == R;
    const uint32_t items = d.C * M;
    const bool lane_mode = kLast && d.store_mode == MODE_LANE;
    uint32_t c[G], jj[G];
    cfx_t v[G][P];
    if constexpr (IDX > 1) __syncthreads();  // (behind the first stage the tile has one)
#pragma unroll
    for (int g = 0; g < G; ++g) {
        // threads past the last butterfly repeat it without storing
        const uint32_t it = min(threadIdx.x + g * blockDim.x, items - 1);
        if (lane_mode) {
            jj[g] = fdiv(it, d.div_C);
            c[g] = it - jj[g] * d.C;
        } else {
            c[g] = it / M;
            jj[g] = it % M;
        }
        {
            constexpr bool kLin = M % kFxPad == 0;
            constexpr uint32_t kStep = M + (M >> kPadShift);
            const cfx_t* s = buf + c[g] * d.lane_stride + (kLin ? pad(jj[g]) : 0u);
#pragma unroll
            for (int q = 0; q < P; ++q) v[g][q] = s[kLin ? q * kStep : pad(jj[g] + q * M)];
            const int sh = fx_norm(words[IDX * d.C + c[g]], P);
            if (sh >= 0) {
#pragma unroll
                for (int q = 0; q < P; ++q) v[g][q] = {v[g][q].x << sh, v[g][q].y << sh};
            } else {
#pragma unroll
                for (int q = 0; q < P; ++q) v[g][q] = {v[g][q].x >> -sh, v[g][q].y >> -sh};
            }
            const FxTw* tw = d.fx_inner;
            const uint32_t step = (jj[g] % NS) * TWS;
            v[g][0] = {v[g][0].x >> 2, v[g][0].y >> 2};
#pragma unroll
            for (int q = 1; q < P; ++q) v[g][q] = fx_cmul(v[g][q], fx_tw_load(&tw[q * step]), d.fx_one);
            fx_dft<P>(v[g], d.fx_one);
        }
    }
    if constexpr (kLast) {
        const bool pre = d.Ns > 1 || d.pro_op == PRO_CHIRP;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t it = threadIdx.x + g * blockDim.x;
            if (OTHERS && words[(kFxRows + 1) * d.C + c[g]]) continue;
            if (it < items && lane0 + c[g] < total) {
                constexpr int P0 = fx_spec_radix(R, 1);
                const int eb = fx_first_exp(words[c[g]], P0, pre) +
                               fx_spec_shifts<R, P0, 1>(words, d.C, c[g]);
                fx_spec_store<P>(d, lane0 + c[g], jj[g] % NS + (jj[g] / NS) * (NS * P), NS, eb, v[g]);
            }
        }
    } else {
        __syncthreads();
        fx_spec_exchange<P, G, R, NS>(d, buf, words + (IDX + 1) * d.C, c, jj, v, false);
        fx_spec_later<R, NS * P, IDX + 1, OTHERS>(d, buf, words, lane0, total);
    }
}

// The closer look at a tile of lanes of R points (a power of two) with one that
// may need the FP64 body (fx_beyond, fx_apart).  In fp64_tile.cu, out of the way
// of the other tiles' code (65536 x 64 points 48.1 us with it in line, 46.4 so;
// 320 x 8192 96.8 and 93.0).
__device__ FxLeft fx_spec_look(const PassDesc& d, uint32_t R, uint32_t* words, uint32_t lane0, uint32_t total,
                               int span);

// One tile (C * R <= 8 points a thread), and what of it is left for the FP64
// body: with anything left nothing is written, and the tile runs again as OTHERS
// (fx_left_row is set), which writes the other lanes.  (The fast form would pay
// for skipping lanes: 4096^2 both ways 1357 us, 1398 with the test at its stores.)
template <uint32_t R, bool OTHERS = false>
__device__ __forceinline__ FxLeft fx_spec_tile(const PassDesc& d, uint32_t tile, unsigned char* smem) {
    constexpr int P = fx_spec_radix(R, 1);
    constexpr int G = 8 / P;
    constexpr uint32_t M = R / P;
    const uint32_t total = d.batch * d.lanes_j;
    const uint32_t lane0 = tile * d.C;
    const uint32_t items = d.C * M;
    cfx_t* buf = reinterpret_cast<cfx_t*>(smem);
    uint32_t* words = reinterpret_cast<uint32_t*>(smem + d.fx_words);
    uint32_t* both = words + kFxRows * d.C;  // (fx_guard_row: at most four stages)
    for (uint32_t i = threadIdx.x; i < (kFxRows + (OTHERS ? 1 : fx_guard_rows(R))) * d.C; i += blockDim.x) words[i] = 0;
    const bool lane_mode = d.load_mode == MODE_LANE;
    uint32_t c[G], jj[G];
    double2 raw[G][P];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        // threads past the last butterfly repeat it without storing
        const uint32_t it = min(threadIdx.x + g * blockDim.x, items - 1);
        if (lane_mode) {
            jj[g] = fdiv(it, d.div_C);
            c[g] = it - jj[g] * d.C;
        } else {
            c[g] = it / M;
            jj[g] = it % M;
        }
#pragma unroll
        for (int q = 0; q < P; ++q) raw[g][q] = {0.0, 0.0};
        if (lane0 + c[g] < total) {
            uint32_t b, j;
            fx_lane(d, lane0 + c[g], b, j);
            const double2* p = d.in + uint64_t(b) * d.in_bs;
            const uint32_t n0 = j + jj[g] * d.lanes_j;
            if (d.pro_op == PRO_GATHER) {
#pragma unroll
                for (int q = 0; q < P; ++q)
                    raw[g][q] = __ldcg(&p[uint64_t(__ldg(&d.pro_perm[n0 + q * M * d.lanes_j])) * d.in_es]);
            } else {
                const uint32_t bound = d.pro_op == PRO_CHIRP ? d.pro_bound : 0xffffffffu;
                const uint64_t step = uint64_t(M) * d.lanes_j * d.in_es;
                p += uint64_t(n0) * d.in_es;
#pragma unroll
                for (int q = 0; q < P; ++q)
                    if (n0 + q * M * d.lanes_j < bound) raw[g][q] = __ldcg(&p[q * step]);
            }
        }
    }
    __syncthreads();  // the words are zero
#pragma unroll
    for (int g = 0; g < G; ++g) {
        // the largest magnitude word: of the negative values (the unsigned
        // maximum) and of the others (the signed one)
        uint32_t neg = 0, low = 0, m2 = 0;
        int pos = 0;
#pragma unroll
        for (int q = 0; q < P; ++q) {
            const int x = __double2hiint(raw[g][q].x), y = __double2hiint(raw[g][q].y);
            neg = __vimax3_u32(neg, uint32_t(x), uint32_t(y));
            pos = __vimax3_s32(pos, x, y);
            // (two elements of some butterflies show nearly every lane that stays)
            if (q == 0 || q == P / 2) m2 = max(m2, min(uint32_t(x) & 0x7fffffffu, uint32_t(y) & 0x7fffffffu));
            low |= uint32_t(__double2loint(raw[g][q].x)) | uint32_t(__double2loint(raw[g][q].y));
        }
        uint32_t m = max(neg & 0x7fffffffu, uint32_t(pos));
        if (m == 0 && low) m = 1;
        if (M % 32 == 0 && !lane_mode) {
            m = __reduce_max_sync(0xffffffffu, m);
            if ((threadIdx.x & 31) == 0 && m) atomicMax(&words[c[g]], m);
            if (jj[g] < 32) {  // (one warp of the lane)
                m2 = __reduce_max_sync(0xffffffffu, m2);
                if ((threadIdx.x & 31) == 0 && m2) atomicMax(&both[c[g]], m2);
            }
        } else {
            constexpr uint32_t kSome = M >= 16 ? 3 : (M >= 8 ? 1 : 0);  // (four butterflies or so)
            atomicMax(&words[c[g]], m);
            if ((jj[g] & kSome) == 0) atomicMax(&both[c[g]], m2);
        }
    }
    __syncthreads();
    const bool outer = d.Ns > 1, chirp = d.pro_op == PRO_CHIRP, inv = d.inv != 0;
    const int top = (outer || chirp ? 61 : 59) - fx_room(P);
    bool rare = false;
    cfx_t v[G][P];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        // (a chirp turns every element, so nothing stays apart)
        if constexpr (!OTHERS) {
            const uint32_t most = words[c[g]], near = fx_near(most, fx_span(P));
            bool look = !chirp && most != 0 && both[c[g]] < near;
            if (!lane_mode && __any_sync(0xffffffffu, look)) {
                // real values, the usual lanes without such an element: neighbouring
                // threads hold neighbouring elements
                uint32_t big = 0, im = 0;
#pragma unroll
                for (int q = 0; q < P; ++q) {
                    big |= uint32_t(fx_mag(raw[g][q].x) >= near) << q;
                    im |= fx_mag(raw[g][q].y) | uint32_t(__double2loint(raw[g][q].y));
                }
                if ((big & __shfl_xor_sync(0xffffffffu, big, 1)) && !im) look = false;
            }
            rare = rare || look || fx_beyond(most);
        }
        {
            const int field = int(words[c[g]] >> 20);
            const int emax = field ? field : 4096;  // a lane of zeros: everything shifts out
#pragma unroll
            for (int q = 0; q < P; ++q) {
                v[g][q] = {fx_from_double(raw[g][q].x, emax, top), fx_from_double(raw[g][q].y, emax, top)};
                if (inv) v[g][q] = {v[g][q].y, v[g][q].x};
            }
            if (outer || chirp) {
                uint32_t b, j;
                fx_lane(d, lane0 + c[g], b, j);
                if (outer) {
                    // W_N^(r k), r = jj + q M: the base times powers of the step
                    const uint32_t k = j - fdiv(j, d.div_Ns) * d.Ns;
                    FxTw t = fx_outer(d, uint32_t(uint64_t(jj[g]) * k * d.tw_mul));
                    const FxTw w = fx_outer(d, uint32_t(uint64_t(M) * k * d.tw_mul));
#pragma unroll
                    for (int q = 0; q < P; ++q) {
                        v[g][q] = fx_cmul(v[g][q], t, d.fx_one);
                        if (q + 1 < P) t = fx_tw_mul(t, w, d.fx_one);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < P; ++q) {
                        const uint32_t n = j + (jj[g] + q * M) * d.lanes_j;
                        if (n < d.pro_bound) v[g][q] = fx_cmul(v[g][q], fx_tw_load(&d.fx_pro[n]), d.fx_one);
                    }
                }
            }
            fx_dft<P>(v[g], d.fx_one);
        }
    }
    fx_spec_exchange<P, G, R, 1>(d, buf, words + d.C, c, jj, v, lane_mode);
    if (__builtin_expect(__syncthreads_or(rare), 0)) {
        const FxLeft left = fx_spec_look(d, R, words, lane0, total, fx_span(P));
        if (left != FX_NOTHING) return left;
    }
    fx_spec_later<R, P, 1, OTHERS>(d, buf, words, lane0, total);
    return FX_NOTHING;
}

}  // namespace kfft
#endif
