// Entry points of the tensor-core memory-rule kernels (memory_tc.cu). Both return false when the
// shape, type of rule, options or alignment are outside what the kernels take; nothing is launched then.
#pragma once

#include "nlh_common.cuh"

namespace nlh {
namespace mtc {

bool forward(int rule, const FwdArgs& a, cudaStream_t st);
bool backward(int rule, const BwdArgs& a, cudaStream_t st);
int timeout_flag();

}  // namespace mtc
}  // namespace nlh
