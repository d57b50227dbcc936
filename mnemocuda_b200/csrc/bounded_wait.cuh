// A wait that ends: the loop around mbarrier tries of the tensor-core GEMMs, free of device code so that a host test can count its tries.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define MB200_INLINE __device__ __forceinline__
#else
#define MB200_INLINE inline
#endif

namespace mb200 {

constexpr uint32_t kWaitBudget = 1u << 16;  // tries; one that fails takes 4 us (measured, sm_100a), all of them 0.26 s
constexpr uint32_t kWaitBurst = 64;

// A wait that runs out raises the flag of its CTA, and from then on a wait of the CTA that is not satisfied at once returns after one more
// try. Nothing is checked where the first try succeeds; beyond it the flag is read before a try and looked at after it, once a burst (a check
// per step, a shared-memory load and a vote, cost an issuing warp 100 of its 400 cycles per chunk).
template <class Ready, class Pause>
MB200_INLINE void bounded_wait(Ready ready, Pause pause, volatile int *abort_flag)
{
    if (ready()) return;
    for (uint32_t i = 0; i < kWaitBudget / kWaitBurst; i++) {
        pause();
        const int raised = *abort_flag;
        if (ready() || raised) return;
#ifdef __CUDACC__
#pragma unroll 1
#endif
        for (uint32_t j = 1; j < kWaitBurst; j++) {
            pause();
            if (ready()) return;
        }
    }
    *abort_flag = 1;
}

}  // namespace mb200
