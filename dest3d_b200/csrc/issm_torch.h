// Host-side operations over the C ABI shared by the two files of the torch extension (issm_torch.cpp: the operations
// themselves; issm_autograd.cpp: autograd functions over them).
#pragma once

#include <ATen/ATen.h>

#include <tuple>
#include <vector>

#include "../../include/issm_b200.h"

namespace issm_host {
using at::Tensor;
using OptTensor = c10::optional<Tensor>;

int dtype_code(at::ScalarType t);
void check_rc(int rc, const char* what);
void* stream_of(const Tensor& t);

std::tuple<Tensor, Tensor, Tensor, Tensor> fwd(const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk_size,
                                               const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, const OptTensor& initial_states,
                                               bool dt_softplus, double dt_min, double dt_max, bool reverse, int64_t path, bool want_final,
                                               bool save_states, const Tensor& status);
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> bwd(
    const Tensor& dout, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& out_x, int64_t chunk_size,
    const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, const OptTensor& initial_states, const OptTensor& dfinal_states, bool dt_softplus,
    double dt_min, double dt_max, bool reverse, int64_t path, const OptTensor& saved_states, const Tensor& status);
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> bi_fwd(
    const Tensor& x, const Tensor& xb, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, const Tensor& Bb, const Tensor& Cb,
    int64_t chunk_size, const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, const OptTensor& initial_states, bool dt_softplus,
    double dt_min, double dt_max, double scale, int64_t path, bool save_states, const Tensor& status);
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> bi_bwd(
    const Tensor& dout, const OptTensor& dfinal, const Tensor& x, const Tensor& xb, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C,
    const Tensor& Bb, const Tensor& Cb, const OptTensor& out_x, const OptTensor& out_xb, int64_t chunk_size, const OptTensor& D, const OptTensor& z,
    const OptTensor& dt_bias, const OptTensor& initial_states, bool dt_softplus, double dt_min, double dt_max, double scale, int64_t path,
    const OptTensor& saved_f, const OptTensor& saved_b, const Tensor& status);
std::tuple<Tensor, Tensor, Tensor> norm_fwd(const Tensor& x2, const OptTensor& z2, const Tensor& weight, const OptTensor& bias, double eps,
                                            int64_t group_size, bool norm_before_gate, bool is_rms);
std::tuple<Tensor, Tensor, Tensor, Tensor> norm_bwd(const Tensor& dy2, const Tensor& x2, const OptTensor& z2, const Tensor& weight, const OptTensor& bias,
                                                    const Tensor& rstd, const OptTensor& mean, double eps, int64_t group_size, bool norm_before_gate,
                                                    bool is_rms);
int64_t usable_slices(const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk, int64_t path, const Tensor& status,
                      int64_t slices);
std::vector<Tensor> sliced_fwd(const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk, const OptTensor& D,
                               const OptTensor& z, const OptTensor& dt_bias, const OptTensor& initial_states, bool dt_softplus, double dt_min, double dt_max,
                               bool reverse, int64_t path, int64_t slices, bool save, const Tensor& status);
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> sliced_bwd(
    const Tensor& dout, const OptTensor& dfinal, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& B, const Tensor& C, int64_t chunk,
    const OptTensor& D, const OptTensor& z, const OptTensor& dt_bias, const OptTensor& initial_states, bool dt_softplus, double dt_min, double dt_max,
    bool reverse, int64_t path, int64_t slices, const std::vector<Tensor>& kept, const Tensor& status);
}  // namespace issm_host
