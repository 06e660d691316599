// What the kernels of the token-sequential recurrence share: their parameters, and the preprocessing of a
// decode step as device functions, so that the stand-alone preprocessing kernel and the fused decode step give the
// same bits.
#pragma once

#include "kda_common.cuh"

namespace kda {

struct ScanParams {
  const void* q; const void* k; const void* v; const void* g; const void* beta;
  int dt_q, dt_k, dt_v, dt_g, dt_beta;
  const float* h0;        // initial state / paged pool (may be null)
  float* ht;              // final state (may be null); the pool itself when paged
  void* out; int dt_out;
  const int32_t* cu_seqlens;     // null = dense [B, T]
  const int32_t* state_indices;  // null = sequence i uses row i
  int64_t slot_stride;           // elements between pool slots
  int num_slots;
  int nseq, T, H, K, V;
  float scale;
};

struct PrepDecodeParams {
  const void* x; const void* w; void* conv_state;          // [N, 3HD], [3HD, W], [slots, W-1, 3HD]
  const void* raw_gate; const float* A_log; const float* dt_bias;   // [N, H, D], [H], [H, D]
  void* q; void* k; void* v; float* g;                     // [N, H, D] each (q, k, v in the dtype of x)
  const int32_t* state_indices;                            // conv pool slots or NULL (slot = sequence)
  int dt, dt_gate, nseq, H, W, num_slots, act;
  float lower_bound, eps;
};

// Eight adjacent channels of the width-W convolution (raw: history rows, then the new token; wraw: their 8 W
// weights, element channel * W + tap) and the activation.
template <int W>
__device__ __forceinline__ void conv8(const uint4 (&raw)[W], const uint4 (&wraw)[W], int dt, int act, float (&y)[8]) {
  const unsigned short* wh = reinterpret_cast<const unsigned short*>(wraw);
#pragma unroll
  for (int i = 0; i < 8; ++i) y[i] = 0.f;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    float f[8];
    raw8_to_float(raw[j], dt, f);
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = fmaf(raw_to_float(wh[i * W + j], dt), f[i], y[i]);
  }
  if (act) {
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = y[i] / (1.f + expf(-y[i]));
  }
}
// 1 / ||y|| of a head whose 128 channels lie in 16 adjacent lanes, eight each (whole warps)
__device__ __forceinline__ float row_rnorm(const float (&y)[8], float eps) {
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) ss = fmaf(y[i], y[i], ss);
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  return rsqrtf(ss + eps);
}
// bounded log2 gate of one channel; a = exp(A_log)
__device__ __forceinline__ float decode_gate(float a, float raw, float bias, float lower_bound) {
  const float z = a * (raw + bias);
  return lower_bound / (1.f + expf(-z)) * kLog2e;
}

// The state-streaming kernel (kda_stream.cu).  A scan it can take: K = V = 128, 16-byte aligned states in and out.
bool stream_takes(const ScanParams& p);
int launch_stream(const ScanParams& p, cudaStream_t stream);
// The same with a wait that runs out (kda_selftest_bounded_stream).
int launch_stream_short(const ScanParams& p, int warp, int step, cudaStream_t stream);
// Whether a decode step of `states` (sequence, head) pairs runs in one launch: the vector form of the preprocessing and whole states
// by bulk copies.  address_bits: all addresses and the slot stride in bytes, or-ed together.  (Slots that overlap need no
// exception: as in the two launches, only states of the same call must not.)
inline bool decode_fuses(int64_t address_bits, int dtype, int64_t states, int width) {
  return dtype != KDA_F32 && width >= 2 && width <= 4 && (address_bits & 15) == 0 && states < (1 << 24);
}
int launch_fused_decode(const PrepDecodeParams& d, const ScanParams& p, cudaStream_t stream);
int stream_error_word();

}  // namespace kda
