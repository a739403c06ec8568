// Learned preconditioner model (cnn.cu): weights on the host (FP32 master copy, Adam state),
// BF16 real-form weights and activations on the device.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <complex>
#include <string>
#include <vector>

#include "gbc_kernels.h"

struct gbc_ctx;

namespace gbc {

struct Cnn {
  int hidden = 12;
  int nlayers = 4;
  // W[l][(d * cout + o) * cin + i], d = 0 self, 1 + 2 mu (+mu hop), 2 + 2 mu (-mu hop)
  std::vector<std::vector<std::complex<float>>> W;
  std::vector<std::vector<float>> m1, m2;  // Adam moments (re, im interleaved)
  long step = 0;
  bool dirty = true;
  int quit = -1;  // warp whose waits for the tensor cores give up at once (-1: none)

  __nv_bfloat16* dW[8] = {nullptr};     // real form, npad(cout) x kpad(cin) in core-matrix layout
  __nv_bfloat16* dWadj[8] = {nullptr};  // input-gradient form
  float* dG = nullptr;                  // real-form weight gradients, layer l at grad_offset(l)
  std::vector<float4*> act;             // activations per layer boundary, [batch][plane][V]
  float4* delta[2] = {nullptr, nullptr};
  float4* target = nullptr;             // training targets, as 4-channel activations
  double* norms = nullptr;              // |target_b|^2, then the loss
  int* errors = nullptr;                // waits for the tensor cores that gave up since the last check
  int act_batch = 0, train_batch = 0;
  float2* links = nullptr;              // FP32 links, planes [4 * 9][V] in even-odd order
  long links_version = -1;

  int cin(int l) const;
  int cout(int l) const;
  void init(int hidden, int layers, unsigned long long seed);
  void upload(cudaStream_t s);
  void ensure(gbc_ctx* c, int batch);
  void ensure_train(gbc_ctx* c, int batch);
  size_t grad_offset(int l) const;
  void forward(gbc_ctx* c, int batch);
  // forward + backward of sum_b |y_b - e_b|^2 / |e_b|^2 (odd sites; e in target, |e|^2 in norms);
  // gradients left in dG
  double loss_and_grad(gbc_ctx* c, int batch);
  void download_grad(cudaStream_t s, std::vector<std::vector<std::complex<float>>>& grad);
  void adam(const std::vector<std::vector<std::complex<float>>>& grad, double lr);
  bool save(const std::string& path) const;
  int load(const std::string& path);
  // waits for the stream and throws if a layer gave up waiting for the tensor cores since the last check
  void check_waits(cudaStream_t s);
  void release();
};

// (the caller runs net.check_waits before it relies on the result)
void cnn_apply_spinor(gbc_ctx* c, Cnn& net, const Spinor& in, const Spinor& out);
// norm2 (may be null): |f_b|^2 of each field over the odd sites, summed in FP64
void cnn_embed_canon(gbc_ctx* c, Cnn& net, int batch, const double* canon_dev, float4* act, double* norm2 = nullptr);
void cnn_extract_canon(gbc_ctx* c, Cnn& net, int batch, const float4* act, double* canon_dev);

}  // namespace gbc
