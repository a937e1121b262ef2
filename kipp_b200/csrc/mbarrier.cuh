// mbarrier waits with a limit.  Every wait of the tensor-core kernels (TMA arrivals, MMA
// commits, hand-overs between warps) goes through mbar_wait: it is bounded by time, not by
// polls (a poll may itself block for a while).  When the limit passes, or as soon as another
// thread of the CTA has given up, it sets the CTA's abort flag and returns false; the caller
// records that in a status word, drains what it has in flight, frees its tensor memory and
// returns, so that the context stays usable and the host learns of it.
#pragma once
#include <stdint.h>

constexpr long long KIPP_WAIT_LIMIT_CYCLES = 2000000000ll;   // about a second of SM clocks: a wait that long has failed

__device__ __forceinline__ uint32_t kipp_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool kipp_mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(kipp_smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool kipp_mbar_wait_limited(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                       long long limit_cycles) {
    if (kipp_mbar_try_wait(bar, parity)) return true;      // mostly the phase is complete already: no clock read
    const long long t0 = clock64();
    for (unsigned i = 0;; ++i) {
        if (kipp_mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 63u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > limit_cycles) break;
        }
    }
    *abort_flag = 1;
    return false;
}

// The end of a CTA of a cluster whose CTAs send into each other's shared memory (st.async, counted on the receiver's barrier
// `mail`).  A CTA that got what it waited for may leave, since nothing else is on its way to it.  One that gave up calls this with
// all its threads: it stays until every other thread of the cluster has left or come here too, which bounded waits make
// certain (barrier.cluster.wait waits for the threads that have not exited), and until what was sent has landed: a
// neighbour that was merely late still sends.  (One that gave up as well sends nothing: hence the limit.)
// (With an arrival by every thread on its way out, eight tokens of 8,100 keys took 3,518 us a step instead of 3,462; as a call ahead of
// the products' release of tensor memory 3,469, inline behind it 3,449.)
__device__ __forceinline__ void kipp_mail_drain(uint64_t* mail, long long limit_cycles) {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    int mine = 0;
    if (mail != nullptr) kipp_mbar_wait_limited(mail, 0, &mine, limit_cycles);
}
