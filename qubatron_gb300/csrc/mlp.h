// Occluder-proposal network (mlp.cu): sizes, parameter layout and the
// device-side state a context keeps.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace qbc {
namespace mlp {

constexpr int kInUsed = 45;   // 9 features + 6-frequency sin/cos of the hit point
constexpr int kIn = 48;       // padded to a multiple of 16
constexpr int kHidden = 128;
constexpr int kOut = 3;       // proposed t along the shadow ray
constexpr int kGate = 3;      // output 3: logit of "the shadow ray is occluded before the hit"
constexpr int kOutUsed = 4;
constexpr int kOutPad = 16;
constexpr float kGateWeight = 0.05f;  // weight of the gate's cross-entropy in the loss

int64_t param_offset(int layer, bool bias);  // floats into the master array
int64_t param_count();
int64_t launches();  // kernels this thread has launched through the network so far

struct Net {
  float* master = nullptr;       // fp32 parameters (W1 b1 W2 b2 W3 b3 W4 b4, W as [out][in])
  __nv_bfloat16* wb = nullptr;   // bf16 copy used by the kernels (same layout)
  float* grad = nullptr;
  float* m = nullptr;            // Adam moments
  float* v = nullptr;
  float* partial = nullptr;      // weight gradients of each block of a gradient
  int sms = 0;
  int64_t step_count = 0;
  bool ready = false;
  unsigned* err = nullptr;       // device error word of the owning context

  int init(uint64_t seed, cudaStream_t s);
  int set(const float* host, cudaStream_t s);
  int get(float* host, cudaStream_t s) const;
  int sync_weights(cudaStream_t s);
  // loss (device float, mean over rows of 45 floats) and its parameter
  // gradient into grad
  int gradient(const float* X, const float* tlab, const int8_t* kind, int64_t rows, float* loss, cudaStream_t s);
  // one step of Adam on `rows` seeded picks of a training set of `samples`
  // bf16 rows of kIn; the step's loss to *loss (device)
  int train_step(const __nv_bfloat16* X, const float* tlab, const int8_t* kind, int64_t samples, uint64_t seed,
                 int64_t rows, float lr, float* loss, cudaStream_t s);
  // gradients of `rows` rows of src, by block, into partial
  template <class Src>
  int partials(const Src& src, int64_t rows, int* blocks, cudaStream_t s);
  void release();
};

}  // namespace mlp
}  // namespace qbc
