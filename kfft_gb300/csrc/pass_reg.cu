// pass_reg.cu -- the register-resident pass kernels of the FP32 build: the
// generic k_pass_reg, the compile-time power-of-two kernels and their
// launcher.  Built in parts (KFFT_REG_PART) that compile in parallel.
#include "fft_device.cuh"

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

#ifndef KFFT_REG_PART
#define KFFT_REG_PART 0
#endif

namespace kfft {

#if defined(KFFT_HALF_SCALAR)
using SpecKernel = void (*)(PassDesc);
using AsyncKernel = void (*)(PassDesc, uint32_t);
using BulkKernel = void (*)(PassDesc, uint32_t*, uint32_t);

enum SpecKind { SPEC_ONE_TILE = 0, SPEC_PIPE = 1 };

// the kernels of a pass of 2^spec points (null: none)
SpecKernel spec_kernel(uint32_t spec, int kind, bool inv);
AsyncKernel async_kernel(uint32_t spec, bool inv, bool plain);
BulkKernel bulk_kernel(uint32_t spec, bool inv, bool plain);

// FP32 power-of-two passes, one kernel per pass length R so each kernel holds
// only its own body (a small instruction footprint):
// * k_pass_bulk: whole contiguous sequences, a plain prologue and more tiles
//   than fit the GPU at once: a grid of resident CTAs, each running many tiles
//   with its next one on its way by a bulk copy (tile_loop_bulk);
// * k_pass_async: the same for full tiles of lanes in rows, the next tile on its
//   way by asynchronous copies (tile_loop_async);
// * k_pass_pipe: the same for other tiles, the next tile's loads in registers
//   (tile_loop_pipelined);
// * k_pass_spec: one tile per CTA otherwise.
#if KFFT_REG_PART == 1
template <uint32_t R, bool INV>
__global__ void __launch_bounds__(kPassThreads, 2) k_pass_pipe(const __grid_constant__ PassDesc d) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    tile_loop_pipelined<R, INV>(d, reinterpret_cast<vec2_t*>(smem_raw));
}

template <uint32_t R, bool INV>
__global__ void __launch_bounds__(kPassThreads, KFFT_REG_MINBLOCKS) k_pass_spec(
    const __grid_constant__ PassDesc d) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    vec2_t* sm = reinterpret_cast<vec2_t*>(smem_raw);
    tile_body_spec<R, INV>(d, blockIdx.x * d.C, d.batch * d.lanes_j, sm, sm + d.C * d.lane_stride + 1);
}

template <uint32_t R>
SpecKernel pick(int kind, bool inv) {
    if (kind == SPEC_PIPE) return inv ? k_pass_pipe<R, true> : k_pass_pipe<R, false>;
    return inv ? k_pass_spec<R, true> : k_pass_spec<R, false>;
}

SpecKernel spec_kernel(uint32_t spec, int kind, bool inv) {
    switch (spec) {
        case 4: return pick<16>(kind, inv);
        case 5: return pick<32>(kind, inv);
        case 6: return pick<64>(kind, inv);
        case 7: return pick<128>(kind, inv);
        case 8: return pick<256>(kind, inv);
        case 9: return pick<512>(kind, inv);
        case 10: return pick<1024>(kind, inv);
        case 11: return pick<2048>(kind, inv);
        case 12: return pick<4096>(kind, inv);
        default: return nullptr;
    }
}
#endif

#if KFFT_REG_PART == 2
template <uint32_t R, bool INV, int STORE>
__global__ void __launch_bounds__(kPassThreads, 3) k_pass_async(const __grid_constant__ PassDesc d,
                                                                uint32_t pairs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    tile_loop_async<R, INV, STORE>(d, pairs != 0, reinterpret_cast<vec2_t*>(smem_raw));
}

template <uint32_t R>
AsyncKernel pick_async(bool inv, bool plain) {
    if (plain) return inv ? k_pass_async<R, true, STORE_PLAIN> : k_pass_async<R, false, STORE_PLAIN>;
    return inv ? k_pass_async<R, true, STORE_PRODUCT> : k_pass_async<R, false, STORE_PRODUCT>;
}

AsyncKernel async_kernel(uint32_t spec, bool inv, bool plain) {
    switch (spec) {
        case 4: return pick_async<16>(inv, plain);
        case 5: return pick_async<32>(inv, plain);
        case 6: return pick_async<64>(inv, plain);
        case 7: return pick_async<128>(inv, plain);
        case 8: return pick_async<256>(inv, plain);
        case 9: return pick_async<512>(inv, plain);
        case 10: return pick_async<1024>(inv, plain);
        default: return nullptr;
    }
}
#endif

#if KFFT_REG_PART == 3
// Single-pass FP32 power-of-two batches of contiguous sequences: each tile's
// points arrive by one bulk copy (tile_loop_bulk).  One exchange buffer and 80
// registers, so three CTAs an SM: 4096 x 4096 points forward 63.6 us, 66 with
// two buffers and two CTAs (2048-point sequences 65.7 -> 60.5).
// `fail` is set when a copy's wait runs out (g_bulk_wait_failed).
template <uint32_t R, bool INV, int STORE>
__global__ void __launch_bounds__(kPassThreads, 3) k_pass_bulk(const __grid_constant__ PassDesc d,
                                                               uint32_t* fail, uint32_t max_polls) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    tile_loop_bulk<R, INV, STORE>(d, smem_raw, fail, max_polls);
}

template <uint32_t R>
BulkKernel pick_bulk(bool inv, bool plain) {
    if (plain) return inv ? k_pass_bulk<R, true, STORE_PLAIN> : k_pass_bulk<R, false, STORE_PLAIN>;
    return inv ? k_pass_bulk<R, true, STORE_PRODUCT> : k_pass_bulk<R, false, STORE_PRODUCT>;
}

BulkKernel bulk_kernel(uint32_t spec, bool inv, bool plain) {
    switch (spec) {
        case 4: return pick_bulk<16>(inv, plain);
        case 5: return pick_bulk<32>(inv, plain);
        case 6: return pick_bulk<64>(inv, plain);
        case 7: return pick_bulk<128>(inv, plain);
        case 8: return pick_bulk<256>(inv, plain);
        case 9: return pick_bulk<512>(inv, plain);
        case 10: return pick_bulk<1024>(inv, plain);
        case 11: return pick_bulk<2048>(inv, plain);
        case 12: return pick_bulk<4096>(inv, plain);
        default: return nullptr;
    }
}
#endif
#endif

#if KFFT_REG_PART == 0
#if defined(KFFT_HALF_SCALAR)
// The run-time tile: bound by instruction issue and latency (108 thread
// instructions a point for 10 x 10 x 10 before, at two instructions a clock).
// Apart from the tensor-core stage and the product stores, with the elements
// of a lane side by side in shared memory (no padding arithmetic), packed
// odd-radix sums and no spills it fits 64 registers, four CTAs an SM.  2^24
// points forward, us, before -> three CTAs -> four: length 1000 96 -> 79 -> 79,
// 1080 117 -> 76 -> 80, 2187 131 -> 114 -> 99, 3003 93 -> 81 -> 73, 59049
// 221 -> 200 -> 169; a 4160^2 convolution 597 -> 532 -> 478.
template <bool INV, int STORE, bool TC, int BLOCKS>
__global__ void __launch_bounds__(kPassThreads, BLOCKS) k_pass_reg(const __grid_constant__ PassDesc d,
                                                              const __grid_constant__ PassExtra x) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // power-of-two passes launch k_pass_bulk, k_pass_async, k_pass_pipe or
    // k_pass_spec instead
    tile_body_reg<INV, false, TC, STORE>(d, x, blockIdx.x, reinterpret_cast<vec2_t*>(smem_raw));
}

// Set when a bulk-copy wait of k_pass_bulk ran out (only a failed or very
// slow copy can cause it); the CTA then ends without finishing its tiles.
// One word per host-thread slot: a launch passes its thread's slot, and the
// thread's next synchronous completion (take_wait_failures) reads and clears
// it, so the failure becomes that call's return code.
__device__ uint32_t g_bulk_wait_failed[kWaitSlots];
#endif

namespace {
std::atomic<uint32_t> g_bulk_polls{kBulkMaxPolls};
std::atomic<int> g_slot_next{0};
thread_local bool t_bulk_launched = false;

#if defined(KFFT_HALF_SCALAR)
// device address of the failure flags (null: the lookup failed)
uint32_t* wait_flags() {
    static uint32_t* const p = [] {
        void* v = nullptr;
        if (cudaGetSymbolAddress(&v, g_bulk_wait_failed) != cudaSuccess) {
            cudaGetLastError();
            v = nullptr;
        }
        return static_cast<uint32_t*>(v);
    }();
    return p;
}
uint32_t bulk_wait_polls() { return g_bulk_polls.load(std::memory_order_relaxed); }
void note_bulk_launch() { t_bulk_launched = true; }

// Raises the dynamic shared-memory limit of a kernel once and caches its
// resident CTAs per SM for a shared-memory size (thread-safe).
int prepare(const void* f, uint32_t smem, uint32_t threads = kPassThreads) {
    static std::mutex mu;
    static std::map<std::pair<const void*, uint64_t>, int> cache;
    static std::map<const void*, bool> configured;
    std::lock_guard<std::mutex> lk(mu);
    if (!configured[f]) {
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) !=
            cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        configured[f] = true;
    }
    auto key = std::make_pair(f, (uint64_t(threads) << 32) | smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, int(threads), smem) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    cache[key] = n;
    return n;
}

int sm_count() {
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 1;
    }();
    return n;
}
#endif
}  // namespace

int wait_slot() {
    thread_local const int slot = g_slot_next.fetch_add(1) % kWaitSlots;
    return slot;
}

bool take_wait_failures(cudaStream_t st) {
#if defined(KFFT_HALF_SCALAR)
    if (!t_bulk_launched) return false;
    t_bulk_launched = false;
    static const uint32_t zero = 0;
    const size_t off = sizeof(uint32_t) * size_t(wait_slot());
    uint32_t v = 0;
    cudaMemcpyFromSymbolAsync(&v, g_bulk_wait_failed, sizeof(v), off, cudaMemcpyDeviceToHost, st);
    cudaMemcpyToSymbolAsync(g_bulk_wait_failed, &zero, sizeof(zero), off, cudaMemcpyHostToDevice,
                            st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        note_cuda_error(e);
        return true;
    }
    return v != 0;
#else
    (void)st;
    return false;
#endif
}

#if defined(KFFT_HALF_SCALAR)
void launch_pass_reg(const PassDesc& d, const PassExtra& x, cudaStream_t st) {
    // one-time shared-memory limit of the generic kernels (thread-safe; a
    // failure is reported on every call)
    static const cudaError_t configured = [] {
        for (const void* f :
             {(const void*)k_pass_reg<false, STORE_PLAIN, false, 4>, (const void*)k_pass_reg<true, STORE_PLAIN, false, 4>,
              (const void*)k_pass_reg<false, STORE_PRODUCT, false, 4>,
              (const void*)k_pass_reg<true, STORE_PRODUCT, false, 4>,
              (const void*)k_pass_reg<false, STORE_ANY, true, 3>, (const void*)k_pass_reg<true, STORE_ANY, true, 3>}) {
            cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 227 * 1024);
            if (e != cudaSuccess) {
                cudaGetLastError();
                return e;
            }
        }
        return cudaSuccess;
    }();
    if (configured != cudaSuccess) {
        note_cuda_error(configured);
        return;
    }
    if (d.spec && d.threads == kPassThreads) {
        const bool inv = d.inv != 0;
        // one pass over whole contiguous sequences, 16-byte aligned: the
        // tiles arrive by bulk copy
        const bool contiguous = d.lanes_j == 1 && d.order == ORDER_J && d.in_es == 1 &&
                                d.in_bs == d.R && (reinterpret_cast<uintptr_t>(d.in) & 15u) == 0;
        if (d.pro_op == PRO_NONE && contiguous) {
            BulkKernel f = bulk_kernel(d.spec, inv, d.epi_op == EPI_NONE);
            const uint32_t smem = 128 + (d.C * d.R + d.C * d.lane_stride + 1u) * uint32_t(sizeof(vec2_t));
            const int per_sm = f ? prepare((const void*)f, smem) : -1;
            const uint32_t grid = uint32_t(std::max(per_sm, 0)) * uint32_t(sm_count());
            uint32_t* fail = wait_flags();
            // from two full rounds on, 912 tiles.  (From where k_pass_pipe's two CTAs
            // an SM start a third round, 609 tiles, this kernel itself is no slower, us
            // there and here: 16 points 760 tiles 24.7, 20.6, 256 points 12.4, 10.4,
            // 4096 points level; but a synchronous call that has launched it asks for
            // failed waits behind it: the real 2D forward and inverse of 877 x 2500, whose
            // inverse has 626 tiles, 248 us with k_pass_pipe there, 265 with this.)
            if (fail && per_sm > 0 && d.tiles >= 2 * grid) {
                f<<<grid, kPassThreads, smem, st>>>(d, fail + wait_slot(), bulk_wait_polls());
                note_cuda_error(cudaGetLastError());
                note_bulk_launch();
                count_launch();
                return;
            }
        }
        // full tiles of lanes in rows (passes of up to 1024 points, so at
        // least four lanes): copied asynchronously, two lanes at a time where
        // they lie together on 16 bytes in every row
        if (d.pro_op == PRO_NONE && d.load_mode == MODE_LANE && d.C * d.R == kRegTile && d.C >= 4) {
            const bool rows_even = d.order == ORDER_J
                                       ? d.in_es == 1 && d.lanes_j % 2 == 0 && d.in_bs % 2 == 0
                                       : d.in_bs == 1 && d.in_es % 2 == 0 && d.batch % 2 == 0;
            const bool pairs = rows_even && (reinterpret_cast<uintptr_t>(d.in) & 15u) == 0;
            AsyncKernel f = async_kernel(d.spec, inv, d.epi_op == EPI_NONE);
            const uint32_t smem =
                (d.C * d.R + d.C * d.lane_stride + 1u) * uint32_t(sizeof(vec2_t));
            const int per_sm = f ? prepare((const void*)f, smem) : -1;
            const uint32_t grid = uint32_t(std::max(per_sm, 0)) * uint32_t(sm_count());
            // from 760 tiles on (us of k_pass_pipe and here: 2^20 points 768 tiles 44.8,
            // 39.1, 2^18 31.8, 30.9, 2^13 26.8, 23.1; at 704 tiles 2^18 28.8, 30.9)
            if (per_sm > 0 && 3 * d.tiles >= 5 * grid) {
                f<<<grid, kPassThreads, smem, st>>>(d, pairs ? 1u : 0u);
                note_cuda_error(cudaGetLastError());
                count_launch();
                return;
            }
        }
        if (d.pro_op == PRO_NONE) {
            SpecKernel f = spec_kernel(d.spec, SPEC_PIPE, inv);
            const int per_sm = f ? prepare((const void*)f, d.smem_bytes) : -1;
            const uint32_t grid = uint32_t(std::max(per_sm, 0)) * uint32_t(sm_count());
            if (per_sm > 0 && d.tiles >= 2 * grid) {
                f<<<grid, kPassThreads, d.smem_bytes, st>>>(d);
                note_cuda_error(cudaGetLastError());
                count_launch();
                return;
            }
        }
        SpecKernel f = spec_kernel(d.spec, SPEC_ONE_TILE, inv);
        if (f && prepare((const void*)f, d.smem_bytes) > 0) {
            f<<<d.tiles, kPassThreads, d.smem_bytes, st>>>(d);
            note_cuda_error(cudaGetLastError());
            count_launch();
            return;
        }
    }
    // the tensor-core stages, the plain store and the product stores each have
    // a kernel of their own (smaller, and no registers held for the others)
    void (*f)(PassDesc, PassExtra);
    if (d.tc) f = d.inv ? k_pass_reg<true, STORE_ANY, true, 3> : k_pass_reg<false, STORE_ANY, true, 3>;
    else if (d.epi_op == EPI_NONE) f = d.inv ? k_pass_reg<true, STORE_PLAIN, false, 4> : k_pass_reg<false, STORE_PLAIN, false, 4>;
    else f = d.inv ? k_pass_reg<true, STORE_PRODUCT, false, 4> : k_pass_reg<false, STORE_PRODUCT, false, 4>;
    f<<<d.tiles, d.threads, d.smem_bytes, st>>>(d, x);
    note_cuda_error(cudaGetLastError());
    count_launch();
}
#endif

#endif
}  // namespace kfft

#if KFFT_REG_PART == 0
extern "C" {
// Test hook: polls a bulk-copy wait makes before it gives up (0 restores the
// default of about a second).  Only a test that checks the failure path
// lowers it; see kfft_gb300.h.
KFFT_API void kfft_gb300_set_bulk_wait_polls(uint32_t polls) {
    kfft::g_bulk_polls.store(polls ? polls : kfft::kBulkMaxPolls);
}

// Synchronises `stream` and reports whether a bounded device wait of this
// thread's earlier asynchronous calls ran out (and clears the record).
KFFT_API int kfft_gb300_check_waits(void* stream) {
    const cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
        kfft::note_cuda_error(e);
        return -1;
    }
    return kfft::take_wait_failures(static_cast<cudaStream_t>(stream)) ? 1 : 0;
}
}  // extern "C"
#endif
