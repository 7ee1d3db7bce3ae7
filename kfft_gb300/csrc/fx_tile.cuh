// fx_tile.cuh -- the double build's register tile in 64-bit block fixed
// point (fx_math.cuh): the passes, descriptors, prologues and epilogues of
// tile_body_reg, with doubles read from and written to global memory and
// every butterfly between in integers.
//
// A tile is read element by element into shared memory, turned into integers
// there, run through its radix stages, and turned back into doubles on the
// way out.  Only the stages are instantiated per radix: the conversions,
// prologues and epilogues exist once, which keeps the kernel small.
//
// Scale of a lane (one length-R sub-FFT): once the tile is read, the largest
// exponent of each lane is known to all threads (an atomic maximum in shared
// memory and one barrier), and the inputs become integers against it.  Every
// stage but the first reads how many bits the lane's largest value really has
// (an OR of magnitude bits accumulated by the stage before) and shifts its
// inputs back up, so nothing is lost where a transform grows less than it
// might.
//
// An inverse transform is the forward one with the parts of every input and
// output swapped, so there is one body for both directions.
//
// Measured (forward, us): 4096 x 4000 points 494, against 987 with the inputs
// held in registers, radices at 128 registers and two exchange buffers;
// 16384 x 1000 417 against 566.  The FP64 body these tiles replace ran the
// uneven batch of 256 in 1672 us, they run it in 862.
//
// A lane that holds an infinity, a NaN, a magnitude from 2^768 on or nothing
// from 2^-767 on is left to the FP64 body, which treats them as IEEE arithmetic
// does (smaller values beside larger ones shift out), and so is one whose small
// parts doubles would keep apart from its large ones (fx_apart in fx_math.cuh):
// the lane, not its tile, so that what becomes of a sequence does not depend on
// those beside it.
//
// Telling the lanes costs up to 6% (65536 x 64 points 43.8 -> 46.4 us, 4096 x 1000
// 116 -> 119, uneven batch of 256 829 -> 862, 4096^2 both ways level); real values
// in the complex form, 4096 x 1000 points, take the closer look and 136; a tile
// that leaves after it has spent 10 to 15% of its FP64 time (256 x 4096 nearly
// real points 121 us, in FP64 from the start 106).
#pragma once

#include "fft_device.cuh"
#include "fx_math.cuh"

#if !defined(KFFT_HALF_SCALAR)

namespace kfft {

// a lane's largest exponent field outside this range goes to the FP64 body
constexpr uint32_t kFxExpLow = 256, kFxExpHigh = 1791;
__device__ __forceinline__ bool fx_beyond(uint32_t most) {
    return most != 0 && ((most >> 20) < kFxExpLow || (most >> 20) >= kFxExpHigh);
}

// What a fixed-point tile leaves to the FP64 body: nothing, the lanes named in
// fx_left_row, or all (nothing written).
enum FxLeft : uint32_t { FX_NOTHING = 0, FX_SOME = 1, FX_ALL = 2 };

__device__ __forceinline__ FxTw fx_tw_load(const FxTw* p) {
    const int4 v = __ldg(reinterpret_cast<const int4*>(p));
    return {v.x, v.y, v.z, v.w};
}

// The outer twiddle W_N^e from the two-level table.
__device__ __forceinline__ FxTw fx_outer(const PassDesc& d, uint32_t e) {
    return fx_tw_mul(fx_tw_load(&d.fx_hi[e >> d.tw_shift]),
                     fx_tw_load(&d.fx_lo[e & ((1u << d.tw_shift) - 1u)]), d.fx_one);
}

// A word whose highest bit b bounds P values by 2^(b + 32).
template <int P>
__device__ __forceinline__ uint32_t fx_bits(const cfx_t* v) {
    int hi = 0, lo = 0;
#pragma unroll
    for (int q = 0; q < P; ++q) {
        hi = __vimax3_s32(hi, int(v[q].x >> 32), int(v[q].y >> 32));
        lo = __vimin3_s32(lo, int(v[q].x >> 32), int(v[q].y >> 32));
    }
    return uint32_t(hi | (lo ^ (lo >> 31))) << 1;
}

// left shift (negative: right) of a stage of radix P whose lane has `bits`
__device__ __forceinline__ int fx_norm(uint32_t bits, int P) {
    return min(__clz(int(bits)), 31) - 1 - fx_room(P);
}

// the exponent (in fx_to_double's sense) of a lane's values after a first
// stage of radix P: `pre` for a chirp or outer twiddle before it
__device__ __forceinline__ int fx_first_exp(uint32_t emax_word, int P, bool pre) {
    int emax = int(emax_word >> 20);
    if (emax == 0) emax = 1023;  // a lane of zeros
    return emax - 1023 + 1085 + (pre ? 2 - 61 : -59) + fx_room(P);
}

// What the element loops need of one lane, worked out once per tile (shared
// memory): offsets of its first input and output, and the rest of its place.
struct __align__(16) FxLane {
    uint64_t in, out;  // element offsets of position 0
    uint32_t j;        // lane of the sequence: position r is input element j + r * lanes_j
    uint32_t k;        // position r is output element k + r * Ns
    uint32_t e;        // outer twiddle exponent per position
    uint32_t b;        // sequence; kFxDead past the last lane
};
static_assert(sizeof(FxLane) == kFxLaneBytes, "the planner sizes shared memory with it");
constexpr uint32_t kFxDead = 0xffffffffu;

// magnitude word of a part
__device__ __forceinline__ uint32_t fx_mag(double v) { return uint32_t(__double2hiint(v)) & 0x7fffffffu; }

__device__ __forceinline__ uint32_t fx_holds(double2 x, uint32_t near) {
    return fx_holds(fx_mag(x.x), fx_mag(x.y), x.x != 0.0, x.y != 0.0, near);
}

// first of the two rows of words behind the stages' ones: the largest of the
// elements' smaller parts (a lane where it is near the largest stays without a
// closer look), and what the lane holds (FX_HAS_RE ...)
__device__ __forceinline__ uint32_t fx_guard_row(const PassDesc& d) { return max(uint32_t(d.nrad), kFxRows); }

// the second of them, in the end: not zero for the lanes that FP64 has to do
__device__ __forceinline__ uint32_t* fx_left_row(const PassDesc& d, unsigned char* smem) {
    return reinterpret_cast<uint32_t*>(smem + d.fx_words) + (fx_guard_row(d) + 1) * d.C;
}

// Turns what the lanes hold into that; every thread gets the outcome.  pair(c):
// lane c has a pair that `holds` does not say.
template <class Pair>
__device__ __forceinline__ FxLeft fx_settle(const PassDesc& d, const uint32_t* words, uint32_t* holds,
                                            uint32_t lane0, uint32_t total, Pair pair) {
    bool some = false, all = true;
    for (uint32_t c = threadIdx.x; c < d.C; c += blockDim.x) {
        uint32_t f = holds[c];
        if (fx_apart(f) && pair(c)) f |= FX_PAIR;
        const bool left = fx_beyond(words[c]) || fx_apart(f);
        holds[c] = left;
        some = some || left;
        all = all && (left || lane0 + c >= total);
    }
    if (!__syncthreads_or(some)) return FX_NOTHING;
    return __syncthreads_and(all) ? FX_ALL : FX_SOME;
}

// sequence and lane index of lane g of a pass
__device__ __forceinline__ void fx_lane(const PassDesc& d, uint32_t g, uint32_t& b, uint32_t& j) {
    if (d.lanes_j == 1) {
        b = g;
        j = 0;
    } else if (d.order == ORDER_J) {
        b = fdiv(g, d.div_lanes_j);
        j = g - b * d.lanes_j;
    } else {
        j = fdiv(g, d.div_batch);
        b = g - j * d.batch;
    }
}

__device__ __forceinline__ void fx_lanes(const PassDesc& d, FxLane* lanes, uint32_t lane0,
                                         uint32_t total) {
    for (uint32_t c = threadIdx.x; c < d.C; c += blockDim.x) {
        FxLane l;
        l.b = kFxDead;
        l.in = l.out = 0;
        l.j = l.k = l.e = 0;
        if (lane0 + c < total) {
            fx_lane(d, lane0 + c, l.b, l.j);
            const uint32_t blk = fdiv(l.j, d.div_Ns), ko = l.j - blk * d.Ns;
            l.k = blk * d.Ns * d.R + ko;
            l.e = ko * d.tw_mul;
            l.in = uint64_t(l.b) * d.in_bs + uint64_t(l.j) * d.in_es;
            l.out = uint64_t(l.b) * d.out_bs + uint64_t(l.k) * d.out_es;
        }
        lanes[c] = l;
    }
}

// Walks a tile's elements (lane c, position r), thread by thread: lane-major
// (consecutive threads on consecutive lanes) or element-major.
struct FxWalk {
    uint32_t c, r, dc, dr;
    bool lane;
    __device__ __forceinline__ FxWalk(const PassDesc& d, bool lane_mode) : lane(lane_mode) {
        if (lane) {
            r = fdiv(threadIdx.x, d.div_C);
            c = threadIdx.x - r * d.C;
            dr = fdiv(blockDim.x, d.div_C);
            dc = blockDim.x - dr * d.C;
        } else {
            c = fdiv(threadIdx.x, d.div_R);
            r = threadIdx.x - c * d.R;
            dc = fdiv(blockDim.x, d.div_R);
            dr = blockDim.x - dc * d.R;
        }
    }
    __device__ __forceinline__ void next(const PassDesc& d) {
        c += dc;
        r += dr;
        if (lane) {
            if (c >= d.C) {
                c -= d.C;
                ++r;
            }
        } else if (r >= d.R) {
            r -= d.R;
            ++c;
        }
    }
};

// Reads the tile and leaves it in `buf` as integers (prologue and outer
// twiddle applied), unless all of it is for the FP64 body.  words[c] becomes the
// largest magnitude word of lane c.
__device__ __forceinline__ FxLeft fx_read(const PassDesc& d, cfx_t* buf, uint32_t* words,
                                          const FxLane* lanes, uint32_t lane0, uint32_t total) {
    const uint32_t elems = d.C * d.R;
    const bool lane_mode = d.load_mode == MODE_LANE;
    const uint64_t step = uint64_t(d.lanes_j) * d.in_es;
    constexpr int U = 4;  // loads in flight together
    uint32_t* both = words + fx_guard_row(d) * d.C;
    {
        // the raw doubles to shared memory, the largest of each lane to words,
        // the largest of the smaller parts to both
        FxWalk w(d, lane_mode);
        uint32_t most = 0, most2 = 0;  // one lane: kept to the end
        auto note = [&](uint32_t c, uint32_t m, uint32_t m2) {
            // a warp whose elements are all of one lane sends one maximum (32
            // atomics to one word take turns)
            if (!lane_mode && __all_sync(0xffffffffu, c == __shfl_sync(0xffffffffu, c, 0))) {
                m = __reduce_max_sync(0xffffffffu, m);
                m2 = __reduce_max_sync(0xffffffffu, m2);
                if (threadIdx.x & 31) return;
            }
            if (m) atomicMax(&words[c], m);
            if (m2) atomicMax(&both[c], m2);
        };
        // (every thread makes as many rounds: the warps vote in them)
#pragma unroll 1
        for (uint32_t base = 0; base < elems; base += U * blockDim.x) {
            const uint32_t i = base + threadIdx.x;
            double2 v[U];
            uint32_t c[U], at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u] = {0.0, 0.0};
                c[u] = w.c;
                at[u] = w.c * d.lane_stride + pad(w.r);
                if (i + u * blockDim.x < elems) {
                    const FxLane& l = lanes[w.c];
                    const uint32_t n = l.j + w.r * d.lanes_j;
                    if (l.b != kFxDead) {
                        if (d.pro_op == PRO_GATHER)
                            v[u] = __ldcg(&d.in[uint64_t(l.b) * d.in_bs + uint64_t(__ldg(&d.pro_perm[n])) * d.in_es]);
                        else if (d.pro_op != PRO_CHIRP || n < d.pro_bound)
                            v[u] = __ldcg(&d.in[l.in + w.r * step]);
                    }
                    w.next(d);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (base + u * blockDim.x >= elems) break;
                if (i + u * blockDim.x < elems) reinterpret_cast<double2*>(buf)[at[u]] = v[u];
                const uint32_t a = fx_mag(v[u].x), b = fx_mag(v[u].y);
                uint32_t m = max(a, b);
                if (m == 0 && (__double2loint(v[u].x) | __double2loint(v[u].y))) m = 1;
                if (d.C == 1) {
                    most = max(most, m);
                    most2 = max(most2, min(a, b));
                } else {
                    note(c[u], m, min(a, b));
                }
            }
        }
        if (d.C == 1) note(0, most, most2);
    }
    __syncthreads();
    // (a chirp turns every element, so nothing stays apart)
    const bool chirped = d.pro_op == PRO_CHIRP;
    const int span = fx_span(d.rad[0]);
    FxLeft left = FX_NOTHING;
    bool rare = false;
    for (uint32_t c = threadIdx.x; c < d.C; c += blockDim.x)
        rare = rare || fx_beyond(words[c]) || (!chirped && words[c] != 0 && both[c] < fx_near(words[c], span));
    if (__syncthreads_or(rare)) {
        uint32_t* holds = both + d.C;
        if (!chirped) {
            FxWalk w(d, false);
#pragma unroll 1
            for (uint32_t i = threadIdx.x; i < elems; i += blockDim.x, w.next(d)) {
                const double2* lane = reinterpret_cast<const double2*>(&buf[w.c * d.lane_stride]);
                const uint32_t near = fx_near(words[w.c], span), r1 = w.r + 1 == d.R ? 0 : w.r + 1;
                const double2 x = lane[pad(w.r)], y = lane[pad(r1)];
                uint32_t f = fx_holds(x, near);
                if (max(fx_mag(x.x), fx_mag(x.y)) >= near && max(fx_mag(y.x), fx_mag(y.y)) >= near) f |= FX_PAIR;
                if (f) atomicOr(&holds[w.c], f);
            }
            __syncthreads();
        }
        left = fx_settle(d, words, holds, lane0, total, [](uint32_t) { return false; });
        if (left == FX_ALL) return left;
    }
    // each thread its own elements again: integers against their lane's scale
    const bool outer = d.Ns > 1, chirp = chirped, inv = d.inv != 0;
    const int top = (outer || chirp ? 61 : 59) - fx_room(d.rad[0]);
    FxWalk w(d, lane_mode);
#pragma unroll 2
    for (uint32_t i = threadIdx.x; i < elems; i += blockDim.x) {
        cfx_t* p = &buf[w.c * d.lane_stride + pad(w.r)];
        const double2 x = *reinterpret_cast<const double2*>(p);
        const int field = int(words[w.c] >> 20);
        const int emax = field ? field : 4096;  // a lane of zeros: everything shifts out
        cfx_t v = {fx_from_double(x.x, emax, top), fx_from_double(x.y, emax, top)};
        if (inv) v = {v.y, v.x};
        if (outer) {
            v = fx_cmul(v, fx_outer(d, w.r * lanes[w.c].e), d.fx_one);
        } else if (chirp) {
            const uint32_t n = lanes[w.c].j + w.r * d.lanes_j;
            if (n < d.pro_bound) v = fx_cmul(v, fx_tw_load(&d.fx_pro[n]), d.fx_one);
        }
        *p = v;
        w.next(d);
    }
    return left;
}

// One stage of radix P, shared memory to shared memory (one buffer where
// d.inplace: at most one round of butterflies, a barrier between its reads
// and writes).
template <int P>
__device__ __forceinline__ void fx_stage(const PassDesc& d, const InnerStep& st, int p,
                                         const cfx_t* src, cfx_t* dst, uint32_t* words) {
    constexpr int G = int(fx_group(P));
    const uint32_t m = st.m, items = d.C * m;
    const bool last = p + 1 == d.nrad;
    const bool one_lane = (m & 31u) == 0;  // a warp's butterflies are all of one lane
#pragma unroll 1
    for (uint32_t base = 0; base < items; base += G * blockDim.x) {
        uint32_t c[G], ob[G];
        cfx_t v[G][P];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            // threads past the last butterfly repeat it without storing (a
            // branch around the loads and the butterfly makes the compiler
            // spill every radix's values around the barrier)
            const uint32_t it = min(base + g * blockDim.x + threadIdx.x, items - 1);
            c[g] = fdiv(it, st.div_m);
            const uint32_t jj = it - c[g] * m;
            const cfx_t* s = src + c[g] * d.lane_stride;
            ob[g] = jj * P;
#pragma unroll
            for (int q = 0; q < P; ++q) v[g][q] = s[pad(jj + q * m)];
            if (p > 0) {
                const int sh = fx_norm(words[p * d.C + c[g]], P);
                if (sh >= 0) {
#pragma unroll
                    for (int q = 0; q < P; ++q) v[g][q] = {v[g][q].x << sh, v[g][q].y << sh};
                } else {
#pragma unroll
                    for (int q = 0; q < P; ++q) v[g][q] = {v[g][q].x >> -sh, v[g][q].y >> -sh};
                }
                const uint32_t blk = fdiv(jj, st.div_ns);
                const uint32_t kk = jj - blk * st.ns;
                const FxTw* tw = d.fx_inner;
                const uint32_t step = kk * st.twstride;
                v[g][0] = {v[g][0].x >> 2, v[g][0].y >> 2};
#pragma unroll
                for (int q = 1; q < P; ++q)
                    v[g][q] = fx_cmul(v[g][q], fx_tw_load(&tw[q * step]), d.fx_one);
                ob[g] = blk * st.ns * P + kk;
            }
            fx_dft<P>(v[g], d.fx_one);
        }
        __syncthreads();
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const bool act = base + g * blockDim.x + threadIdx.x < items;
            uint32_t b = act ? fx_bits<P>(v[g]) : 0u;
            if (act) {
                cfx_t* o = dst + c[g] * d.lane_stride;
#pragma unroll
                for (int q = 0; q < P; ++q) o[pad(ob[g] + q * st.ns)] = v[g][q];
            }
            if (!last) {
                uint32_t* out_bits = words + (p + 1) * d.C;
                if (one_lane) {
                    b = __reduce_or_sync(0xffffffffu, b);
                    if ((threadIdx.x & 31) == 0 && b) atomicOr(&out_bits[c[g]], b);
                } else if (act) {
                    atomicOr(&out_bits[c[g]], b);
                }
            }
        }
    }
}

// The exponent of each lane's final values (in fx_to_double's sense) in
// words[c], from the exponent of its inputs and its stages' shifts.
__device__ __forceinline__ void fx_exponents(const PassDesc& d, uint32_t* words) {
    const bool pre = d.Ns > 1 || d.pro_op == PRO_CHIRP;
    for (uint32_t c = threadIdx.x; c < d.C; c += blockDim.x) {
        int eb = fx_first_exp(words[c], d.rad[0], pre);
        for (int i = 1; i < d.nrad; ++i) eb += 2 - fx_norm(words[i * d.C + c], d.rad[i]);
        words[c] = uint32_t(eb);
    }
}

// Writes the tile (but for the lanes in `skip`, if given) through the epilogue.
__device__ __forceinline__ void fx_write(const PassDesc& d, const cfx_t* buf, const uint32_t* words,
                                         const FxLane* lanes, const uint32_t* skip) {
    const uint32_t elems = d.C * d.R;
    const bool inv = d.inv != 0;
    const uint32_t op = d.epi_op;
    const bool table = op == EPI_MUL || op == EPI_CHIRP || op == EPI_RADER_FWD;
    // the scale: a power of two, times a factor where it is not one
    const bool scaled = op == EPI_NONE || op == EPI_CHIRP;
    const int32_t sh = scaled ? d.fx_scale_h : 0, sl = d.fx_scale_l;
    const int e_more = (scaled ? d.fx_scale_e : 0) + (sh ? 2 : 0) + (table ? 2 : 0) +
                       (table && op != EPI_CHIRP ? d.fx_epi_e : 0);
    const uint64_t step = uint64_t(d.Ns) * d.out_es;
    FxWalk w(d, d.store_mode == MODE_LANE);
#pragma unroll 2
    for (uint32_t i = threadIdx.x; i < elems; i += blockDim.x, w.next(d)) {
        const FxLane& l = lanes[w.c];
        if (l.b == kFxDead || (skip && skip[w.c])) continue;
        const uint32_t k = l.k + w.r * d.Ns;
        if (op == EPI_CHIRP && k >= d.epi_bound) continue;
        cfx_t u = buf[w.c * d.lane_stride + pad(w.r)];
        if (inv) u = {u.y, u.x};
        const int eb = int(words[w.c]);
        uint64_t at = l.out + w.r * step;
        double2* out = d.out;
        if (table) {
            if (op == EPI_RADER_FWD && k == 0) {
                // in doubles: bin 0 of the spectrum is far below the others, and
                // X_0 = x_0 + the sum of the others is saved with x_0
                store_elem(d, l.b, 0, double2{fx_to_double(u.x, eb), fx_to_double(u.y, eb)});
                continue;
            }
            u = fx_cmul(u, fx_tw_load(&d.fx_epi[k]), d.fx_one);
        }
        if (sh) {
            const FxLimbs x = fx_limbs(u.x), y = fx_limbs(u.y);
            u.x = fx_add_high(fx_mad(x.l, sh, fx_mul(x.h, sl)), fx_mul(x.h, sh), d.fx_one);
            u.y = fx_add_high(fx_mad(y.l, sh, fx_mul(y.h, sl)), fx_mul(y.h, sh), d.fx_one);
        }
        double2 r = {fx_to_double(u.x, eb + e_more), fx_to_double(u.y, eb + e_more)};
        if (op == EPI_RADER_INV) {
            out = d.aux_out + uint64_t(l.b) * d.aux_out_bs;
            at = uint64_t(__ldg(&d.epi_perm[k])) * d.aux_out_es;
            r = cadd(r, d.aux_in[2 * uint64_t(l.b)]);  // (a cached load: one value a sequence)
            if ((d.fx_scale_h | d.fx_scale_e) != 0) r = cscale(r, d.scale);  // scale != 1
            if (k == 0) out[0] = cscale(__ldcg(&d.aux_in[2 * uint64_t(l.b) + 1]), d.scale);
        } else if (op == EPI_MUL_OUT) {
            r = cscale(cmul(r, __ldcg(&d.epi_tab[at])), d.scale);
        }
        out[at] = r;
    }
}

// One tile of a pass in fixed point, and what of it is left for the FP64 body.
// Shared memory: the exchange buffers (one where d.inplace), at byte d.fx_words
// a row of words per stage and the guard's, and after them the lane table.
__device__ __forceinline__ FxLeft fx_tile(const PassDesc& d, const PassExtra& x, uint32_t tile,
                                          unsigned char* smem) {
    cfx_t* bufA = reinterpret_cast<cfx_t*>(smem);
    cfx_t* bufB = d.inplace ? bufA : bufA + d.C * d.lane_stride + 1;
    uint32_t* words = reinterpret_cast<uint32_t*>(smem + d.fx_words);
    FxLane* lanes = reinterpret_cast<FxLane*>(smem + d.fx_lanes);
    for (uint32_t i = threadIdx.x; i < (fx_guard_row(d) + 2) * d.C; i += blockDim.x) words[i] = 0;
    const uint32_t lane0 = tile * d.C, total = d.batch * d.lanes_j;
    fx_lanes(d, lanes, lane0, total);
    __syncthreads();
    const FxLeft left = fx_read(d, bufA, words, lanes, lane0, total);
    if (left == FX_ALL) return left;
    __syncthreads();
    cfx_t* src = bufA;
#pragma unroll 1
    for (int p = 0; p < d.nrad; ++p) {
        cfx_t* dst = src == bufA ? bufB : bufA;
        switch (d.rad[p]) {
#define KFFT_FX_CASE(P) \
    case P: fx_stage<P>(d, x.step[p], p, src, dst, words); break;
            KFFT_FX_CASE(2) KFFT_FX_CASE(3) KFFT_FX_CASE(4) KFFT_FX_CASE(5) KFFT_FX_CASE(6)
            KFFT_FX_CASE(7) KFFT_FX_CASE(8) KFFT_FX_CASE(9) KFFT_FX_CASE(10) KFFT_FX_CASE(11)
            KFFT_FX_CASE(12) KFFT_FX_CASE(13) KFFT_FX_CASE(14) KFFT_FX_CASE(15) KFFT_FX_CASE(16)
#undef KFFT_FX_CASE
            default: break;
        }
        if (p + 1 == d.nrad) fx_exponents(d, words);
        __syncthreads();
        src = dst;
    }
    fx_write(d, src, words, lanes, left == FX_SOME ? fx_left_row(d, smem) : nullptr);
    return left;
}

// The FP64 body (fp64_tile.cu) for what a fixed-point tile leaves.  (A
// compile-time tile stops before it stores anything; its other lanes run again
// first.)
__device__ void fp64_tile(const PassDesc& d, const PassExtra& x, uint32_t tile, unsigned char* smem,
                          FxLeft left);

// a register tile of the double build
__device__ __forceinline__ void double_tile(const PassDesc& d, const PassExtra& x, uint32_t tile,
                                            unsigned char* smem) {
    const FxLeft left = d.fx ? fx_tile(d, x, tile, smem) : FX_ALL;
    if (left != FX_NOTHING) fp64_tile(d, x, tile, smem, left);
}

}  // namespace kfft
#endif
