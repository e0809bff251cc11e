// Bounded mbarrier waits of the tensor-core kernels: a wait that runs out records why in the device status word,
// raises the CTA's abort flag and returns false.
#pragma once

#include "common.h"
#include "ptx_sm100.cuh"

namespace llmt_b200 {

// The template flag only marks barriers that the peer CTA of a pair also signals; those
// signals carry no generic-proxy data (ring entries arrive by st.async, operands by TMA,
// accumulators through tcgen05 fences), so the default CTA-scope acquire is enough.
template <bool CLUSTER = false>
__device__ __forceinline__ bool bounded_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                             DeviceStatus* st, int code, int detail, uint64_t limit_ns) {
    auto poll = [&]() { return ptx::mbar_try_wait(bar, parity); };
    if (poll()) return true;
    // The wall clock is slow to read: it is first looked at after 256 failed polls, so a wait
    // of ordinary length never touches it.
    uint64_t t0 = 0;
    uint32_t spins = 0;
    for (;;) {
        if (poll()) return true;
        if ((++spins & 255u) == 0u) {
            if (*abort_flag) return false;
            const uint64_t now = ptx::globaltimer_ns();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > limit_ns) {
                if (atomicCAS(&st->code, 0, code) == 0) {
                    st->detail = detail;
                    st->block = static_cast<int32_t>(blockIdx.x);
                }
                *abort_flag = 1;
                return false;
            }
        }
    }
}


// The same for a converged warp: every lane polls, so the warp stays converged and what it issues next may be
// issued by any of its lanes.
__device__ __forceinline__ bool bounded_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, DeviceStatus* st, int code,
                                                  int detail, uint64_t limit_ns) {
    if (__all_sync(0xffffffffu, ptx::mbar_try_wait(bar, parity))) return true;
    uint64_t t0 = 0;
    uint32_t spins = 0;
    for (;;) {
        if (__all_sync(0xffffffffu, ptx::mbar_try_wait(bar, parity))) return true;
        if ((++spins & 255u) == 0u) {
            int stop = 0;
            if ((threadIdx.x & 31) == 0) {
                if (*abort_flag) {
                    stop = 1;
                } else {
                    const uint64_t now = ptx::globaltimer_ns();
                    if (t0 == 0) {
                        t0 = now;
                    } else if (now - t0 > limit_ns) {
                        if (atomicCAS(&st->code, 0, code) == 0) {
                            st->detail = detail;
                            st->block = static_cast<int32_t>(blockIdx.x);
                        }
                        *abort_flag = 1;
                        stop = 1;
                    }
                }
            }
            if (__shfl_sync(0xffffffffu, stop, 0) != 0) return false;
        }
    }
}

}  // namespace llmt_b200
