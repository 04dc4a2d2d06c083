// What the data gradient of a convolution does in its epilogue for the batch norm that produced the convolution's input
// z = act(batch_norm(y)): the gradient is stored with the ReLU's mask applied, and its sums go to dbeta and dgamma.  A pass
// of its own over the gradient and y cost 3.3 of 21.1 ms in a ResNet-50 step (batch 256).
#pragma once
extern "C" struct esgd_bn_grad {
  const void* y;          // bf16, like z
  const void* mask;       // a bit per element ([pixels][C / 8] bytes) as esgd_bn_fwd leaves it, or null: no ReLU
  const float* aux;       // mean [C], 1 / std [C]
  float* sums;            // dbeta [C], dgamma [C], zeroed by the caller
};
