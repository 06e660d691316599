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
                                                           float* __restrict__ hout, int K, int V) {
  __shared__ __align__(16) float sM[32][kAffineSlab + 4];
  __shared__ __align__(16) float sH[kAffineSlab][32];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32, tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;
  const int64_t n = blockIdx.z;
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
    *reinterpret_cast<float4*>(hout + n * K * V + (int64_t)(r0 + ty + 16 * i) * V + c0 + 4 * tx) =
        make_float4(acc[i][0] + bv[i].x, acc[i][1] + bv[i].y, acc[i][2] + bv[i].z, acc[i][3] + bv[i].w);
}

// The chain of such maps along the segments of a row, K = V = 128: h(s + 1) = M_s h(s) + b_s from the row's initial state (zero if
// NULL), every h(s) written to hin and the last one to fin (if given).  A column of h needs only the same column before it, so a
// CTA carries COLS columns of one head through all segments in one launch, without waiting for any other; the next M is on its
// way while one is multiplied.  A thread adds one or two rows x four columns in the order of K, as state_affine_kernel does.
// Bound by the chain: loads, 128 steps and two barriers a map on one SM.  32 heads, four maps: 28 us, as four launches of that
// kernel and the copy of the initial state 43; forward of 32768 tokens of 8 heads, eight maps, 475 us with launches, 370 with this
// kernel (375 with 32 columns per CTA for so few heads).
constexpr int kChainThreads = 512;
constexpr int kChainPitch = 132;
struct ChainParams {
  const float* M; const float* b;      // [rows, segs, heads, 128, 128]
  const float* h0;                     // [rows, heads, 128, 128] or NULL
  float* hin;                          // [rows, segs, heads, 128, 128]
  float* fin;                          // [rows, heads, 128, 128] or NULL
  int heads, segs;
};
template <int COLS>
__global__ void __launch_bounds__(kChainThreads) state_chain_kernel(const ChainParams p) {
  constexpr int Q = COLS / 4, R = COLS / 16, SLICES = 128 / COLS;      // column quads; rows per thread, 128 / R apart
  extern __shared__ __align__(16) float smem_chain[];
  float* const sH = smem_chain + 2 * 128 * kChainPitch;       // [128][COLS]
  const int tid = threadIdx.x, cq = 4 * (tid & (Q - 1)), r0 = tid / Q;
  const int c0 = COLS * (blockIdx.x % SLICES), item = blockIdx.x / SLICES;
  const int row = item / p.heads, head = item % p.heads;
  auto state = [&](int sg) { return ((int64_t)(row * (int64_t)p.segs + sg) * p.heads + head) * 16384; };
  auto fetch = [&](int sg) {
    const float* m = p.M + state(sg);
    float* to = smem_chain + (sg & 1) * 128 * kChainPitch;
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const int e = tid + kChainThreads * l;
      cp_async16(to + (e >> 5) * kChainPitch + 4 * (e & 31), m + 4 * e, true);
    }
    cp_async_commit();
  };
  const int maps = p.fin ? p.segs : p.segs - 1;
  if (maps > 0) fetch(0);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = r0 + 64 * i;
    const int64_t at = (int64_t)r * 128 + c0 + cq;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.h0) {                                               // (a caller's: it may start off a 16-byte address)
      const float* h = p.h0 + (int64_t)item * 16384 + at;
      x = make_float4(h[0], h[1], h[2], h[3]);
    }
    *reinterpret_cast<float4*>(sH + r * COLS + cq) = x;
    *reinterpret_cast<float4*>(p.hin + state(0) + at) = x;
  }
  for (int sg = 0; sg < maps; ++sg) {
    float4 bv[R], acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      bv[i] = *reinterpret_cast<const float4*>(p.b + state(sg) + (int64_t)(r0 + 64 * i) * 128 + c0 + cq);
      acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (sg + 1 < maps) { fetch(sg + 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();                                          // M_s and h(s) are in shared memory
    const float* m = smem_chain + (sg & 1) * 128 * kChainPitch + r0 * kChainPitch;
#pragma unroll 4
    for (int k = 0; k < 128; k += 4) {
      float a[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(m + 64 * i * kChainPitch + k);
        a[i][0] = x.x; a[i][1] = x.y; a[i][2] = x.z; a[i][3] = x.w;
      }
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const float4 y = *reinterpret_cast<const float4*>(sH + (k + d) * COLS + cq);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          acc[i].x = fmaf(a[i][d], y.x, acc[i].x); acc[i].y = fmaf(a[i][d], y.y, acc[i].y);
          acc[i].z = fmaf(a[i][d], y.z, acc[i].z); acc[i].w = fmaf(a[i][d], y.w, acc[i].w);
        }
      }
    }
    __syncthreads();                                          // h(s) and this buffer of M have been read
    float* to = sg + 1 < p.segs ? p.hin + state(sg + 1) : p.fin + (int64_t)item * 16384;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = r0 + 64 * i;
      const float4 x = make_float4(acc[i].x + bv[i].x, acc[i].y + bv[i].y, acc[i].z + bv[i].z, acc[i].w + bv[i].w);
      *reinterpret_cast<float4*>(sH + r * COLS + cq) = x;
      *reinterpret_cast<float4*>(to + (int64_t)r * 128 + c0 + cq) = x;
    }
  }
}

template <int COLS>
static int launch_chain(const ChainParams& p, int64_t chains, cudaStream_t s) {
  constexpr int smem = (2 * 128 * kChainPitch + 128 * COLS) * 4;
  if (chains * (128 / COLS) > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  if (cudaFuncSetAttribute(state_chain_kernel<COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return KDA_ERR_LAUNCH;
  state_chain_kernel<COLS><<<(unsigned)(chains * (128 / COLS)), kChainThreads, smem, s>>>(p);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

// One CTA fits an SM: 16 columns each while that leaves no CTA waiting, else 32.
int launch_state_chain(const float* M, const float* b, const float* h0, float* hin, float* fin, int rows, int heads, int segs,
                       cudaStream_t s) {
  if ((((uintptr_t)M | (uintptr_t)b | (uintptr_t)hin | (uintptr_t)fin) & 15) != 0) return KDA_ERR_ARG;
  const ChainParams p{M, b, h0, hin, fin, heads, segs};
  const int64_t chains = (int64_t)rows * heads;
  return chains * 8 <= device_sms() ? launch_chain<16>(p, chains, s) : launch_chain<32>(p, chains, s);
}

}  // namespace kda

extern "C" int kda_state_affine(const float* transition, const float* h_in, const float* b,
                                float* h_out, int count, int key_dim, int value_dim, void* stream) {
  if (!transition || !h_in || !b || !h_out || count < 0) return KDA_ERR_ARG;
  if (key_dim % 64 || value_dim % 64 || key_dim <= 0 || value_dim <= 0) return KDA_ERR_UNSUPPORTED;
  if (count == 0) return KDA_OK;
  if (!kda::aligned_to(16, b, h_out)) return KDA_ERR_ARG;
  dim3 grid(value_dim / 32, key_dim / 32, count);
  if ((((uintptr_t)transition | (uintptr_t)h_in) & 15) == 0)
    kda::state_affine_kernel<true><<<grid, 128, 0, (cudaStream_t)stream>>>(transition, h_in, b, h_out, key_dim, value_dim);
  else
    kda::state_affine_kernel<false><<<grid, 128, 0, (cudaStream_t)stream>>>(transition, h_in, b, h_out, key_dim, value_dim);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}
