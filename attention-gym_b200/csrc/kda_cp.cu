// Context-parallel boundary-state composition: h_out = M h_in + b per (sequence, head).
//
// A slice of a long sequence maps its entering state affinely to its leaving state; M [K, K] is the
// slice transition (kda_chunk_transition) and b [K, V] the leaving state for a zero entering state.
// Only h crosses GPUs; this kernel applies the local correction.  fp32 throughout: the product is
// tiny (K = V = 128 per head) and its rounding would otherwise accumulate along the rank chain.
// The reference has no context parallelism (docs/linear.md:220-222).
#include "kda_common.cuh"

namespace kda {

// Bound by the latency of its loads (4 MFLOP and 256 KB a head), and it stands in a chain: a CTA has 32 x 32 outputs, so that
// 32 heads fill the SMs, and asks for all of its rows of M and columns of h at once (up to 128 steps of K).  A thread adds two
// rows x four columns in the order of K.  32 heads, K = V = 128: 8.7 us, with tiles of 64 x 64 and slabs of 16 steps of K
// 19.  VEC: M and h are 16-byte aligned.
constexpr int kAffineSlab = 128;
template <bool VEC>
__global__ void __launch_bounds__(128, 4) state_affine_kernel(const float* __restrict__ M,
                                                           const float* __restrict__ hin,
                                                           const float* __restrict__ b,
                                                           float* __restrict__ hout, int K, int V,
                                                           int group, int64_t in_stride,
                                                           int64_t out_stride) {
  __shared__ __align__(16) float sM[32][kAffineSlab + 4];
  __shared__ __align__(16) float sH[kAffineSlab][32];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32, tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;
  // matrix blockIdx.z = (g, i) with i < group: inputs at g * in_stride + i, output at g * out_stride + i
  const int64_t n = (int64_t)(blockIdx.z / group) * in_stride + blockIdx.z % group;
  const int64_t no = (int64_t)(blockIdx.z / group) * out_stride + blockIdx.z % group;
  const float* Mn = M + n * K * K;
  const float* Hn = hin + n * K * V;
  auto copy = [](float* to, const float* from) {            // four values to shared memory, in flight together if VEC
    if (VEC) cp_async16(to, from, true);
    else *reinterpret_cast<float4*>(to) = make_float4(from[0], from[1], from[2], from[3]);
  };
  float4 bv[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
    bv[i] = *reinterpret_cast<const float4*>(b + n * K * V + (int64_t)(r0 + ty + 16 * i) * V + c0 + 4 * tx);
  float acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += kAffineSlab) {
    const int steps = min(kAffineSlab, K - k0);             // 64 or 128
    if (k0) __syncthreads();
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const int e = tid + 128 * l, mr = e >> 5, mk = 4 * (e & 31), hk = e >> 3, hc = 4 * (e & 7);
      if (mk < steps) copy(&sM[mr][mk], Mn + (int64_t)(r0 + mr) * K + k0 + mk);
      if (hk < steps) copy(&sH[hk][hc], Hn + (int64_t)(k0 + hk) * V + c0 + hc);
    }
    if (VEC) { cp_async_commit(); cp_async_wait<0>(); }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < steps; k += 4) {
      const float4 x0 = *reinterpret_cast<const float4*>(&sM[ty][k]), x1 = *reinterpret_cast<const float4*>(&sM[ty + 16][k]);
      const float a0[4] = {x0.x, x0.y, x0.z, x0.w}, a1[4] = {x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const float4 y = *reinterpret_cast<const float4*>(&sH[k + d][4 * tx]);
        const float hv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[0][j] = fmaf(a0[d], hv[j], acc[0][j]);
          acc[1][j] = fmaf(a1[d], hv[j], acc[1][j]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    *reinterpret_cast<float4*>(hout + no * K * V + (int64_t)(r0 + ty + 16 * i) * V + c0 + 4 * tx) =
        make_float4(acc[i][0] + bv[i].x, acc[i][1] + bv[i].y, acc[i][2] + bv[i].z, acc[i][3] + bv[i].w);
}

// `groups` x `group` products; the matrices of group g start at index g * in_stride (inputs) and
// g * out_stride (output).
int launch_state_affine(const float* M, const float* hin, const float* b, float* hout, int groups,
                        int group, int64_t in_stride, int64_t out_stride, int K, int V, cudaStream_t s) {
  if (groups <= 0 || group <= 0) return KDA_OK;
  dim3 grid(V / 32, K / 32, groups * group);
  if ((((uintptr_t)M | (uintptr_t)hin) & 15) == 0)
    state_affine_kernel<true><<<grid, 128, 0, s>>>(M, hin, b, hout, K, V, group, in_stride, out_stride);
  else
    state_affine_kernel<false><<<grid, 128, 0, s>>>(M, hin, b, hout, K, V, group, in_stride, out_stride);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

}  // namespace kda

extern "C" int kda_state_affine(const float* transition, const float* h_in, const float* b,
                                float* h_out, int count, int key_dim, int value_dim, void* stream) {
  if (!transition || !h_in || !b || !h_out || count < 0) return KDA_ERR_ARG;
  if (key_dim % 64 || value_dim % 64 || key_dim <= 0 || value_dim <= 0) return KDA_ERR_UNSUPPORTED;
  if (count == 0) return KDA_OK;
  return kda::launch_state_affine(transition, h_in, b, h_out, 1, count, 0, 0, key_dim, value_dim,
                                  (cudaStream_t)stream);
}
