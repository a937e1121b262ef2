// Probes of the bounded mbarrier wait (mbarrier.cuh), for the tests that make a wait run out
// without making any kernel of the engine fail: one CTA initialises a barrier that nothing
// ever arrives at, waits on it with a limit of `limit_cycles` SM clocks through the helper the
// tensor-core kernels use, and writes what the helper returned and how long it waited.  It
// allocates no tensor memory and starts no copy, so there is nothing to drain; it returns by
// itself when the limit has passed.
#include "common.cuh"
#include "mbarrier.cuh"

namespace {
__global__ void wait_probe_kernel(int* status, long long* waited, long long limit_cycles) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(kipp_smem_u32(&bar)), "r"(1));
    }
    __syncthreads();
    const long long t0 = clock64();
    const bool ok = kipp_mbar_wait_limited(&bar, 0, &abort_flag, limit_cycles);
    const long long dt = clock64() - t0;
    if (!ok) atomicMax(&status[1], 1);            // the word the tensor-core kernels set when a wait ran out
    if (threadIdx.x == 0) *waited = dt;
}
// The end of a cluster's CTA whose neighbour sends after it has given up (kipp_mail_drain): CTA 1 sends a word `late_cycles`
// after it started, CTA 0 waits for it for `limit_cycles`, sets the status word if that was too short, drains as the
// kernels do, and writes what then lies in its mailbox.  Both loops are bounded.
__global__ void mail_probe_kernel(int* status, int* landed, long long late_cycles, long long limit_cycles, int word) {
    __shared__ uint64_t bar;
    __shared__ int box, abort_flag;
    const int rank = blockIdx.x;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        box = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(kipp_smem_u32(&bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 4;" ::"r"(kipp_smem_u32(&bar)) : "memory");
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank == 1) {
        if (threadIdx.x == 0) {
            const long long t0 = clock64();
            while (clock64() - t0 < late_cycles) {}
            uint32_t to, at;
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(kipp_smem_u32(&box)));
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"(kipp_smem_u32(&bar)));
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(to), "r"(word), "r"(at) : "memory");
        }
        return;
    }
    if (!__syncthreads_and(kipp_mbar_wait_limited(&bar, 0, &abort_flag, limit_cycles))) {
        kipp_mail_drain(&bar, 100000000ll);
        if (threadIdx.x == 0) atomicMax(&status[1], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) *landed = *(volatile int*)&box;
}
}  // namespace

// The two limits are clamped to [0, 10 million] SM clocks (some 5 ms).
extern "C" int kipp_mail_probe(int* status, int* landed, long long late_cycles, long long limit_cycles, int word, void* stream) {
    if (status == nullptr || landed == nullptr) return KIPP_ERR_ARG;
    auto clamp = [](long long v) { return v < 0 ? 0ll : v > 10000000ll ? 10000000ll : v; };
    return kipp_launch_cluster(mail_probe_kernel, dim3(2), dim3(64), 0, (cudaStream_t)stream, dim3(2, 1, 1), status, landed, clamp(late_cycles),
                               clamp(limit_cycles), word);
}

// limit_cycles is clamped to [1 thousand, 100 million] SM clocks (at most some 50 ms).
extern "C" int kipp_wait_probe(int* status, long long* waited_cycles, long long limit_cycles, void* stream) {
    if (status == nullptr || waited_cycles == nullptr) return KIPP_ERR_ARG;
    if (limit_cycles < 1000) limit_cycles = 1000;
    if (limit_cycles > 100000000ll) limit_cycles = 100000000ll;
    wait_probe_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(status, waited_cycles, limit_cycles);
    return kipp_launch_status();
}
