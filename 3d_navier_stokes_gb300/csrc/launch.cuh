// launch.cuh — kernel launches with programmatic stream serialization.
#pragma once
#include <cuda_runtime.h>

namespace ns3d {

// Launch of a pass kernel with programmatic stream serialization: the launch itself
// overlaps the previous kernel's end, and the kernel waits for its results (pdl_begin).
// One RK4 step of 21 kernels, FP32: 32^3 67.6 -> 63.5 us, 64^3 75.7 -> 71.7 us, 128^3
// 206.9 -> 202.8 us; the closure's inference at 64^3 (five kernels) 97 -> 83 us.
template <typename A> struct ArgOf { using type = A; };
template <typename... KA> struct Launcher {
    void (*kernel)(KA...);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    void operator()(typename ArgOf<KA>::type... a) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, kernel, a...);
    }
};
template <typename... KA>
Launcher<KA...> pass(void (*kernel)(KA...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s) {
    Launcher<KA...> l{kernel, {}, {}};
    l.cfg.gridDim = grid;
    l.cfg.blockDim = dim3(threads);
    l.cfg.dynamicSmemBytes = smem;
    l.cfg.stream = s;
    return l;
}

}  // namespace ns3d
