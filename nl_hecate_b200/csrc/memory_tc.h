// Entry points of the tensor-core memory-rule kernels (memory_tc.cu). Both return false when the
// shape, type of rule, options or alignment are outside what the kernels take; nothing is launched then.
#pragma once

#include "nlh_common.cuh"

namespace nlh {
namespace mtc {

// a.interval = tile length = distance of the stored states
bool forward(int rule, const FwdArgs& a, cudaStream_t st);
// T = tile length, mstep = floats between the stored states of consecutive tile starts
bool backward(int rule, const BwdArgs& a, int T, long long mstep, cudaStream_t st);
int timeout_flag();

}  // namespace mtc
}  // namespace nlh
