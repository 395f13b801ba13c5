// What the binding files share: the launchers of bindings.cpp that other files call on tensors.
#pragma once

#include <torch/extension.h>

#include "api.h"

torch::Tensor attn_err_word();   // device int32[4], set by bounded waits that expired
int bind_num_sms();              // SMs a persistent kernel may use
void bind_gemm(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& out, bool a_mn, bool b_mn, int64_t out_mode,
               int64_t splits = 0, int64_t tile_n = 0, bool b_is_old = false);
bool bind_gemm_swiglu(const torch::Tensor& x, const torch::Tensor& w, c10::optional<torch::Tensor> gu, torch::Tensor& act);
bool bind_gemm_swiglu_bwd(const torch::Tensor& dy, const torch::Tensor& w, const torch::Tensor& gu, torch::Tensor& dgu);
