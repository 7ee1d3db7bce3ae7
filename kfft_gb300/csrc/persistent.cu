// persistent.cu -- the persistent work-queue kernel: one launch drains a
// queue of (pass, tile) items ordered by dependency level, with bounded waits
// on per-pass tile counters (a wait that gives up sets an error word).
#include "fft_device.cuh"
#include "fx_spec.cuh"

#include <mutex>

namespace kfft {

// resident CTAs per SM of the queue kernel (its tiles are capped at 2048
// points): four for FP32 (64 registers a thread), three for the double build
// (80 registers; 256 sequences of up to 2^18 points, as the tiles stood: 0.89
// ms, two CTAs 0.95, four 0.97; 0.86 now)
#ifndef KFFT_QUEUE_MINBLOCKS
#if defined(KFFT_HALF_SCALAR)
#define KFFT_QUEUE_MINBLOCKS 4
#else
#define KFFT_QUEUE_MINBLOCKS 3
#endif
#endif

// Publishes a finished item: the CTA's stores are ordered before one thread's
// by the barrier, and that thread publishes them all with one release add at
// GPU scope (the waiting CTA's acquire load pairs with it).  A thread of the
// last warp does it, so that thread 0 goes on to the next item's dependency
// meanwhile (512 sequences FP32 1412 -> 1354 us, 256 in double 852 -> 841).
__device__ __forceinline__ void publish_done(uint32_t* done) {
    __syncthreads();
    if (threadIdx.x == blockDim.x - 32) {
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(done), "r"(1u) : "memory");
    }
}

// Thread 0's dependency wait for item q (a bounded spin that sets the error
// word instead of hanging); the result goes to every thread through *s_ok.
__device__ __forceinline__ void item_wait(const QueueItem& q, const uint32_t* done,
                                          uint32_t* error, uint32_t max_polls, uint32_t* s_ok) {
    bool ok = true;
    if (q.dep >= 0) ok = wait_for(&done[q.dep], q.need, max_polls);
    if (!ok) atomicExch(error, 1u);
    *s_ok = ok ? 1u : 0u;
}

// Starts copying the descriptor and the stage table of pass `desc` into shared
// memory (8 bytes a thread and step).  One item ahead, so neither is waited
// for: 512 sequences FP32 1486 -> 1412 us against copying the descriptor when
// the item's turn came and reading the stage table from global memory.
__device__ __forceinline__ void stage_desc(const PassDesc* __restrict__ descs,
                                           const PassExtra* __restrict__ extras, uint32_t desc,
                                           PassDesc* s_desc, PassExtra* s_extra) {
    static_assert(sizeof(PassDesc) % 8 == 0 && sizeof(PassExtra) % 8 == 0, "copied 8 bytes at a time");
    constexpr uint32_t n0 = sizeof(PassDesc) / 8, n1 = sizeof(PassExtra) / 8;
    const char* g0 = reinterpret_cast<const char*>(&descs[desc]);
    const char* g1 = reinterpret_cast<const char*>(&extras[desc]);
    const uint32_t a0 = uint32_t(__cvta_generic_to_shared(s_desc));
    const uint32_t a1 = uint32_t(__cvta_generic_to_shared(s_extra));
    for (uint32_t i = threadIdx.x; i < n0 + n1; i += blockDim.x) {
        const bool first = i < n0;
        const char* g = first ? g0 + 8 * i : g1 + 8 * (i - n0);
        const uint32_t a = first ? a0 + 8 * i : a1 + 8 * (i - n0);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(g) : "memory");
    }
}

__device__ __forceinline__ void run_item(const PassDesc& d, const PassExtra& x, uint32_t tile,
                                         vec2_t* buf) {
#if !defined(KFFT_HALF_SCALAR)
    unsigned char* smem = reinterpret_cast<unsigned char*>(buf);
    FxLeft left = FX_ALL;
    if (d.fx) {
        switch (d.spec) {
            case 4: left = fx_spec_tile<16>(d, tile, smem); break;
            case 5: left = fx_spec_tile<32>(d, tile, smem); break;
            case 6: left = fx_spec_tile<64>(d, tile, smem); break;
            case 7: left = fx_spec_tile<128>(d, tile, smem); break;
            case 8: left = fx_spec_tile<256>(d, tile, smem); break;
            case 9: left = fx_spec_tile<512>(d, tile, smem); break;
            case 10: left = fx_spec_tile<1024>(d, tile, smem); break;
            case 11: left = fx_spec_tile<2048>(d, tile, smem); break;
            default: left = fx_tile(d, x, tile, smem); break;
        }
    }
    if (left != FX_NOTHING) fp64_tile(d, x, tile, smem, left);
#else
    if (d.inv) tile_body_reg<true, true, false>(d, x, tile, buf);
    else tile_body_reg<false, true, false>(d, x, tile, buf);
#endif
}

__global__ void __launch_bounds__(KFFT_QUEUE_THREADS, KFFT_QUEUE_MINBLOCKS) k_persistent(
    const PassDesc* __restrict__ descs, const PassExtra* __restrict__ extras,
    const QueueItem* __restrict__ items, uint32_t nitems, uint32_t* head, uint32_t* done,
    uint32_t* error, uint32_t max_polls) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_ok;
    __shared__ __align__(16) PassDesc s_desc[2];
    __shared__ __align__(16) PassExtra s_extra[2];
    vec2_t* buf = reinterpret_cast<vec2_t*>(smem_raw);
    // Items claimed two ahead, their records in a ring of three shared slots:
    // the current item, the next one (copied in during the previous item)
    // and the one after it (copied in during this item); the next item's
    // descriptor and stage table are copied in during this one too.  A CTA's
    // claims increase, so its current item is the earliest of its claims; the
    // earliest claimed and unfinished item of all then is some CTA's current
    // item, whose dependencies (earlier queue positions, all claimed) are
    // done: the queue cannot deadlock.
    constexpr uint32_t kEnd = 0xffffffffu;
    __shared__ __align__(16) QueueItem s_item[3];
    uint32_t claim = 0;  // thread 0: the queue position of the item after next
    if (threadIdx.x == 0) {
        const uint32_t a = atomicAdd(head, 1u);
        const uint32_t b = atomicAdd(head, 1u);
        s_item[0].desc = kEnd;
        s_item[1].desc = kEnd;
        if (a < nitems) s_item[0] = items[a];
        if (b < nitems) s_item[1] = items[b];
        claim = atomicAdd(head, 1u);
    }
    __syncthreads();
    uint32_t slot = 0, cur = 0;
    if (s_item[0].desc != kEnd) stage_desc(descs, extras, s_item[0].desc, &s_desc[0], &s_extra[0]);
    asm volatile("cp.async.wait_all;" ::: "memory");
    while (true) {
        const QueueItem q = s_item[slot];
        if (q.desc == kEnd) break;
        const uint32_t next = s_item[slot == 2 ? 0u : slot + 1u].desc;
        if (next != kEnd) stage_desc(descs, extras, next, &s_desc[cur ^ 1], &s_extra[cur ^ 1]);
        if (threadIdx.x == 0) {
            // the slot the previous item used (every thread read it before
            // the previous item's barriers) takes the record at `claim`
            const uint32_t s2 = slot == 0 ? 2u : slot - 1u;
            if (claim < nitems) {
                const uint32_t sa = uint32_t(__cvta_generic_to_shared(&s_item[s2]));
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(&items[claim])
                             : "memory");
            } else {
                s_item[s2].desc = kEnd;
            }
            item_wait(q, done, error, max_polls, &s_ok);
            claim = atomicAdd(head, 1u);
        }
        __syncthreads();
        if (s_ok) run_item(s_desc[cur], s_extra[cur], q.tile, buf);
        // the next item's record, descriptor and stage table have landed
        asm volatile("cp.async.wait_all;" ::: "memory");
        publish_done(&done[q.desc]);
        slot = slot == 2 ? 0u : slot + 1u;
        cur ^= 1u;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

bool launch_persistent(const PassDesc* descs, const void* extras,
                       const void* items, uint32_t nitems, uint32_t* head, uint32_t* done,
                       uint32_t* error, uint32_t smem_bytes, cudaStream_t st,
                       uint32_t max_polls) {
    // the kernel's shared-memory limit and occupancy, set up under a lock (several
    // host threads may record queues at once)
    static std::mutex mu;
    static int blocks_per_sm = -1;
    static uint32_t configured_smem = 0;
    static int sms = 0;
    uint32_t grid;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (configured_smem < smem_bytes) {
            cudaError_t e = cudaFuncSetAttribute(
                k_persistent, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes));
            if (e != cudaSuccess) {
                note_cuda_error(e);
                return false;
            }
            configured_smem = smem_bytes;
            blocks_per_sm = -1;
        }
        if (blocks_per_sm < 0) {
            int dev = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, k_persistent,
                                                          KFFT_QUEUE_THREADS, configured_smem);
            if (blocks_per_sm < 1) blocks_per_sm = 1;
        }
        grid = uint32_t(sms * blocks_per_sm);
    }
    if (grid > nitems) grid = nitems ? nitems : 1;
    k_persistent<<<grid, KFFT_QUEUE_THREADS, smem_bytes, st>>>(
        descs, static_cast<const PassExtra*>(extras), static_cast<const QueueItem*>(items),
        nitems, head, done, error, max_polls);
    note_cuda_error(cudaGetLastError());
    count_launch();
    return true;
}

}  // namespace kfft
