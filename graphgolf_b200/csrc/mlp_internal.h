// mlp_internal.h -- the proposal filter's network object and the enqueue
// helpers the annealing engine calls (all on a caller-given stream, usable
// inside a stream capture).  Not part of the public C ABI.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ggb {
namespace mlp {

constexpr int kFeatures = 32;
constexpr int kHidden = 256;
constexpr int kMaxTrainRows = 256;
// Packed FP32 parameters: W1 [256][32], b1 [256], W2 [256][256] (row n holds
// the weights into unit n), b2 [256], w3 [256], b3 [1].
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kHidden * kFeatures;
constexpr int kOffW2 = kOffB1 + kHidden;
constexpr int kOffB2 = kOffW2 + kHidden * kHidden;
constexpr int kOffW3 = kOffB2 + kHidden;
constexpr int kOffB3 = kOffW3 + kHidden;
constexpr int kParams = kOffB3 + 1;

struct AdamHyper {
  float lr, beta1, beta2, eps;
};

}  // namespace mlp
}  // namespace ggb

struct ggb_mlp {
  int max_rows = 0;
  ggb::mlp::AdamHyper hyper{};
  float* p = nullptr;          // FP32 master parameters
  float* g = nullptr;          // gradients of the last backward
  float* m1 = nullptr;         // Adam moments
  float* m2 = nullptr;
  int* step = nullptr;         // Adam step count (device)
  // W1 and W2 as BF16 in the tensor cores' shared-memory operand layout
  // (K-major, no swizzle: 8-row x 16-byte core matrices), staged by bulk copies
  __nv_bfloat16* W1u = nullptr;    // [256][32] tiled
  __nv_bfloat16* W2u = nullptr;    // [256][256] tiled
  // what a training step hands from its row pass to its weight pass, [kMaxTrainRows][256]
  __nv_bfloat16* H1 = nullptr;
  __nv_bfloat16* dZ2 = nullptr;
  __nv_bfloat16* dZ1 = nullptr;
  float* H2 = nullptr;
  float* dZ1f = nullptr;
  float* err = nullptr;        // [2][kMaxTrainRows]: dy, y - t
  float* loss = nullptr;
  // host-entry staging
  __nv_bfloat16* X = nullptr;      // [max_rows][32]
  float* xf = nullptr;             // [max_rows][32] as the caller gave them
  float* y = nullptr;              // [max_rows]
  float* t = nullptr;              // [kMaxTrainRows]
};

namespace ggb {

// y[0..rows) = network(X rows); rows % 16 == 0.
int mlp_forward(ggb_mlp* m, const __nv_bfloat16* X, int rows, float* y, cudaStream_t st);
// Loss and gradients of the mean squared error over B rows (B % 16 == 0,
// B <= 256) -- rows idx[0..B) of X, or 0..B-1 when idx is null -- into m->loss
// and m->g; with adam, one Adam step on them instead of writing m->g.
int mlp_step(ggb_mlp* m, const __nv_bfloat16* X, const int* idx, const float* t, int B, bool adam, cudaStream_t st);
// The training state (FP32 parameters, both Adam moments, the Adam step) as
// host bytes: its size, a copy out and a copy in (which also refreshes every
// BF16 copy of the weights).  Synchronous.
size_t mlp_state_bytes();
int mlp_save_state(ggb_mlp* m, void* host);
int mlp_load_state(ggb_mlp* m, const void* host);

}  // namespace ggb
