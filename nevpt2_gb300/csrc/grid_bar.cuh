// Waits between the CTAs of cooperative kernels (all co-resident), bounded: a grid-wide
// barrier, and words that arrive where they are polled for.
#pragma once

namespace nvpt {
namespace s2 {

// Polls before a wait gives up: 1.9 s of a barrier's (0.45 us each, with back-off), 1.0 s of an
// exchange's (0.23 us, without: a column is a few polls).
constexpr unsigned kBarSpin = 1u << 22;

struct Bar {
    unsigned count, gen;
    int err;
};

// Arrival is an acq_rel add on the counter; the last CTA resets it and publishes
// the next generation with a release store; the others poll the generation with
// acquire loads.  Returns false if the wait timed out or another CTA reported an
// error.
__device__ __forceinline__ bool grid_bar(Bar *b, unsigned nblk, unsigned &gen, unsigned limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned g = gen;
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(&b->count) : "memory");
        if (old == nblk - 1) {
            asm volatile("st.relaxed.gpu.global.u32 [%0], 0;" ::"l"(&b->count) : "memory");
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&b->gen), "r"(g + 1) : "memory");
        } else {
            unsigned spins = 0, cur;
            for (;;) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(&b->gen) : "memory");
                if (cur != g) break;
                if (++spins > limit || *(volatile int *)&b->err) {
                    atomicExch(&b->err, 1);
                    ok = 0;
                    break;
                }
                if (spins > 64) __nanosleep(32);
            }
        }
        gen = g + 1;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// A double as a word that its reader polls for: kNoMsg until it has arrived.  A NaN of
// these very bits (payloads pass through FP64 arithmetic, and memory filled with 0xff
// bytes is one) becomes another NaN, or its readers would wait for good.
constexpr unsigned long long kNoMsg = ~0ull;
__device__ __forceinline__ void send_word(unsigned long long *to, double x) {
    unsigned long long w = (unsigned long long)__double_as_longlong(x);
    if (w == kNoMsg) w = 0x7ff8000000000000ull;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(to), "l"(w) : "memory");
}

}  // namespace s2
}  // namespace nvpt
