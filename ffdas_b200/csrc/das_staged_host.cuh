// das_staged_host.cuh -- host helpers shared by the launchers of the staged kernels.
#pragma once

#include <atomic>
#include <cmath>

#include "core.h"
#include "das_problem.h"
#include "das_staged.cuh"

namespace ffdas {

template <typename Kernel>
inline ffdas_error_t prepare_kernel(Kernel kernel, size_t smem) {
    FFDAS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // all of the unified L1/shared array as shared memory: several CTAs per SM
    FFDAS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    (int)cudaSharedmemCarveoutMaxShared));
    return FFDAS_SUCCESS;
}

// Kernel attributes (dynamic shared memory above 48 KB, carveout) belong to a
// device: set them once for every device the process launches the kernel on.
template <auto Kernel>
inline ffdas_error_t prepare_once(size_t smem) {
    static std::atomic<unsigned long long> done{0ull};
    int dev = 0;
    FFDAS_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return FFDAS_SUCCESS;
    FFDAS_TRY(prepare_kernel(Kernel, smem));
    done.fetch_or(bit, std::memory_order_release);
    return FFDAS_SUCCESS;
}

// Channel slices (1 .. most) for `ctas` tiles on `sms` SMs that hold `resident`
// CTAs each: the fewest CTAs on the fullest SM per slice, 1.5 % a slice for the
// adds into the image, and less than a full residency hides less latency.
inline int balanced_slices(int64_t ctas, int sms, int resident, int most) {
    if (sms < 1) sms = 1;
    int best_n = 1;
    double best = 0.0;
    for (int n = 1; n == 1 || n <= most; n++) {
        const int64_t total = ctas * n, per = (total + sms - 1) / sms;
        const double full = (double)total / ((double)sms * resident);
        double cost = (double)per / n * (1.0 + 0.015 * n);
        if (full < 1.0) cost /= std::sqrt(full);
        if (n == 1 || cost < best * 0.97) {
            best = cost;
            best_n = n;
        }
        if (per >= 8 * resident) break;
    }
    return best_n;
}

// Defined in das_staged.cu.
staged_params base_params(ffdas_context &h, const das_problem &pb, const gather_params &gp);

}  // namespace ffdas
