// The operator with its gradient: one autograd node around forward() and backward().
#pragma once
#include "gdr.h"

namespace fqla_host {

// Returns (o, final_state or nothing).  Without a differentiable input (or with gradients off)
// nothing is kept for a backward.
std::pair<at::Tensor, OptTensor> apply(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                       const at::Tensor& g, const at::Tensor& beta, double scale,
                                       const OptTensor& initial_state, const OptTensor& cu,
                                       Options opt);

}  // namespace fqla_host
