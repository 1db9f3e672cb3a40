// What the op registration of _xpu_C and the native layer call (layer.cpp) share.
#pragma once

#include "shim.h"

namespace b200shim {

// The device's status word (pinned host memory, written by a grouped GEMM whose bounded wait ran
// out), and the check that turns it into the RuntimeError of the next call.
int32_t* device_status_word(int device);
void raise_if_timed_out(int32_t* word);

// How the library reads a weight tensor [experts, ...] of an N x K grouped GEMM (the format follows
// from dtypes and shapes); raises for what it does not take.
struct WeightDesc {
  b200moe_weight_format format;
  int group;          // int4: K elements per scale
  bool fp8, mxfp4, fp8_block;
};
WeightDesc describe_weights(const at::Tensor& w, const std::optional<at::Tensor>& scale, int64_t N, int64_t K,
                            int64_t num_experts, int64_t layout, at::ScalarType activation_dtype);

// Functions of the extension module: layer_plan, layer_run, layer_experts, workspace_clear.
PyMethodDef* layer_methods();

}  // namespace b200shim
