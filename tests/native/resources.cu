// Kernels whose speed rests on keeping their state in registers
// (compiled by tests/test_kernel_resources.py for ptxas's report).
#include "../../kmertreecounter_b200/csrc/kc_kernels.cuh"

template __global__ void kc::count_routed<1>(kc::CountArgs);
template __global__ void kc::count_routed<2>(kc::CountArgs);
template __global__ void kc::count_routed<2, true>(kc::CountArgs);
