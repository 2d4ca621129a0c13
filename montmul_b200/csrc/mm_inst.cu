// Kernel instantiations of one transform length, n = 2^MM_M (the build compiles this file once
// per length so the lengths compile in parallel).
#include "mm_kernels.cuh"

#ifndef MM_M
#error "compile with -DMM_M=<log2 n>"
#endif

namespace mm {

#define MM_CAT2(a, b) a##b
#define MM_CAT(a, b) MM_CAT2(a, b)

template <int M, int NTA>
struct AltStep {
    static StepFn fn() { return step_kernel<M, NTA, alt_min_blocks_for(M)>; }
};
template <int M>
struct AltStep<M, 0> {
    static StepFn fn() { return nullptr; }
};

template <int M, int NTW>
struct WideStep {
    static StepFn fn() { return step_kernel<M, NTW, 512 / NTW, true>; }   // 128 registers a thread
};
template <int M>
struct WideStep<M, 0> {
    static StepFn fn() { return nullptr; }
};

KernelSet MM_CAT(kernels_m, MM_M)() {
    constexpr int NT = threads_for(MM_M), NTA = alt_threads_for(MM_M);
    constexpr int W0 = wide_threads_for(MM_M, 0), W1 = wide_threads_for(MM_M, 1);
    constexpr int NTM = W0 ? W0 : W1 ? W1 : NT;   // mul: one block, the widest shape
    return KernelSet{step_kernel<MM_M, NT>, AltStep<MM_M, NTA>::fn(), NTA,
                     {{WideStep<MM_M, W0>::fn(), W0}, {WideStep<MM_M, W1>::fn(), W1}}, mul_kernel<MM_M, NTM, (NTM != NT)>, NTM, setup_kernel<MM_M, NT>,
                     transform_kernel<MM_M, NT>, NT,
                     smem_bytes<MM_M>()};
}

}  // namespace mm
