// The decode step, one token per sequence and K = V = 128, as state streaming.
//
// Per (sequence, head) the kernel has to move the 64 KiB fp32 state in and out of HBM; the arithmetic of a token is
// small beside it.  One persistent CTA per SM moves whole states, which are contiguous, as single bulk copies through a
// ring of three shared-memory stages: one arriving, one being advanced, one leaving.
//
//   warp 16       one thread issues the copies, paced by a full / done mbarrier pair per stage
//   warps 17..22  three pairs bring the token operands.  A pair takes every third state of the CTA: it loads, converts
//                 (q scaled, 2^g, q.k) and publishes in one of eight operand slots, so that the microseconds a
//                 plain load takes beside the copies never reach the arithmetic.  In the fused decode step (W > 0)
//                 the pair computes the operands from the projections instead: short convolution over the paged
//                 history, activation, l2norm, gate
//   warps 0..15   warp (g, w) advances rows 32 w .. + 31 of columns 32 g .. + 31, a column per lane and rows in pairs for
//                 the packed arithmetic.  The two K-reductions cross the four warps of a column group through shared
//                 memory, one named barrier per state
//
// us per step of a captured graph, 32 heads, 1 / 37 / 256 sequences (of measured copy bandwidth at 256; the 78 MB of 37 sequences stay in
// L2 when one pool is advanced again and again, over four pools in turn the fused step takes 32): the fused step
// 6.6 / 21.8 / 189 (87 %), against 9.3 / 27.6 / 204 as two overlapping launches with q, k, v and the gate in memory between
// them; given operands 5.2 / 19.4 / 179 (91 %), against 5.7 / 22.6 / 191 with the states as 32-column slabs in four rings.
// Every wait is bounded.  One that runs out records code 64 and stops the CTA: the others look for that while they
// wait, the four warps of a column group decide together behind their barrier (a warp that left alone would leave them there),
// a state that was not advanced completely is never handed to the copying warp, and that warp waits for the loads it has
// issued before the shared memory goes back.
// (Several tokens per sequence on the same ring: one state at a time has 1.1 us a token, 48 sequences of 1 to 8 tokens 72
// against 58 us of the token scan.  Bulk-copied states under the token scan's layout, two persistent CTAs per SM: 80 us.)
#include "kda_recurrent.cuh"
#include "kda_sm100.cuh"
#include "kda_timing.cuh"

namespace kda {
namespace {

using namespace sm100;

constexpr int kStages = 3, kStateFloats = 128 * 128, kStateBytes = 4 * kStateFloats;
constexpr int kSlots = 8, kSlotFloats = 520;      // q (scaled) 128 | k 128 | 2^g 128 | v 128 | q.k | beta
constexpr int kPairs = 3;             // 23 warps: 80 registers a thread (72 from 24 on)
constexpr int kThreads = 32 * (16 + 1 + 2 * kPairs);
constexpr int kRedFloats = 4 * 2 * 2 * 4 * 32;    // [column group][token parity][two sums][four warps][32]
constexpr int kSmemBytes = kStages * kStateBytes + 4 * (kSlots * kSlotFloats + kRedFloats) + 256;
static_assert(kSmemBytes <= 232448, "shared memory of one CTA");

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}

// A bounded wait of the kernel: false if it ran out, or another warp of the CTA has given up meanwhile.
__device__ __forceinline__ bool wait_unless(uint64_t* bar, uint32_t parity, volatile int* abort, int limit) {
#pragma unroll 1
  for (int spin = 0; spin < limit; ++spin) {
    if (mbar_wait(bar, parity, 1)) return true;
    if ((spin & 63) == 63 && *abort) return false;
  }
  return false;
}
__device__ __forceinline__ void give_up(volatile int* abort, int* error) {
  *abort = 1;
  if (error) atomicExch(error, 64);
}

// pool slot of work item n = (sequence, head); < 0: padding (a non-positive or out of range index)
__device__ __forceinline__ int64_t slot_of(const ScanParams& p, int seq) {
  if (!p.state_indices) return seq;
  const int si = p.state_indices[seq];
  return si > 0 && si < p.num_slots ? si : -1;
}

// eight adjacent elements of an operand row as raw bits, and as floats
struct Raw8 { uint4 a, b; };
__device__ __forceinline__ void load8(const void* base, int dt, int64_t at, Raw8& r) {
  const int esz = dt == KDA_F32 ? 4 : 2;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(base) + at * esz;
  if ((reinterpret_cast<uintptr_t>(base) & 15) == 0) {      // (`at` is a multiple of 8)
    r.a = *reinterpret_cast<const uint4*>(src);
    if (dt == KDA_F32) r.b = *reinterpret_cast<const uint4*>(src + 16);
  } else {
    uint32_t x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = load_raw(base, dt, at + e);
    if (dt == KDA_F32) { r.a = make_uint4(x[0], x[1], x[2], x[3]); r.b = make_uint4(x[4], x[5], x[6], x[7]); }
    else r.a = make_uint4(x[0] | x[1] << 16, x[2] | x[3] << 16, x[4] | x[5] << 16, x[6] | x[7] << 16);
  }
}
__device__ __forceinline__ void to_floats(const Raw8& r, int dt, float (&x)[8]) {
  if (dt == KDA_F32) {
    x[0] = __uint_as_float(r.a.x); x[1] = __uint_as_float(r.a.y); x[2] = __uint_as_float(r.a.z); x[3] = __uint_as_float(r.a.w);
    x[4] = __uint_as_float(r.b.x); x[5] = __uint_as_float(r.b.y); x[6] = __uint_as_float(r.b.z); x[7] = __uint_as_float(r.b.w);
  } else {
    raw8_to_float(r.a, dt, x);
  }
}

// One warp of a pair puts its half of a token into an operand slot: warp 0 q (lanes 0..15) and k, warp 1 v and the gate.
__device__ __forceinline__ void publish(float* o, int half, int lane, float (&x)[8], float beta, float scale) {
  const int c0 = 8 * (lane & 15);
  float* dst = o + c0;
  if (half == 0) {
    if (lane < 16) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] *= scale;
    } else {
      dst += 128;
    }
    float dot = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) dot = fmaf(x[e], __shfl_down_sync(0xffffffffu, x[e], 16), dot);
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
    if (lane == 0) { o[512] = dot; o[513] = beta; }
  } else if (lane < 16) {
    dst += 384;
  } else {
    dst += 256;
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = exp2f(x[e]);
  }
  reinterpret_cast<float4*>(dst)[0] = make_float4(x[0], x[1], x[2], x[3]);
  reinterpret_cast<float4*>(dst)[1] = make_float4(x[4], x[5], x[6], x[7]);
}

// SHORT (the self-test): the waits of warp `warp` of CTA 0 have no polls from its state `step` on.
struct ShortWait { int warp, step; };
template <int W, bool SHORT = false>
__global__ void __launch_bounds__(kThreads, 1) kda_stream_kernel(const ScanParams p, const PrepDecodeParams d, int* error,
                                                                 const ShortWait short_wait) {
  extern __shared__ __align__(128) unsigned char sm[];
  float* ring = reinterpret_cast<float*>(sm);
  float* ops = ring + kStages * kStateFloats;
  float* s_red = ops + kSlots * kSlotFloats;
  uint64_t* full = reinterpret_cast<uint64_t*>(s_red + kRedFloats);      // [stage] the state has arrived
  uint64_t* done = full + kStages;                                       // [stage] it has been advanced
  uint64_t* op_full = done + kStages;                                    // [slot] the operands are there
  uint64_t* op_free = op_full + kSlots;                                  // [slot] they have been used
  volatile int* s_abort = reinterpret_cast<volatile int*>(op_free + kSlots);
  volatile int* s_stop = s_abort + 1;                                    // [column group][step parity] a warp's wait ran out
  static_assert(8 * (2 * kStages + 2 * kSlots) + 4 * (1 + 8) <= 256, "barriers");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int items = p.nseq * p.H, stride = (int)gridDim.x;
  const bool paged = p.state_indices != nullptr;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&done[s], 16); }
    for (int s = 0; s < kSlots; ++s) { mbar_init(&op_full[s], 2); mbar_init(&op_free[s], 16); }
    mbar_init_fence();
    *s_abort = 0;
  }
  if (tid < 8) s_stop[tid] = 0;
  __syncthreads();
  auto polls = [&](int step) {
    return SHORT && blockIdx.x == 0 && warp == short_wait.warp && step >= short_wait.step ? 0 : kSpinLimit;
  };
  if (warp == 16) {
    // ---- copies ------------------------------------------------------------------------------------------
    if (lane != 0) return;
    int64_t slot = 0;
    auto find = [&](int& n) -> bool {            // the next state that is not padding
      for (; n < items; n += stride)
        if ((slot = slot_of(p, n / p.H)) >= 0) return true;
      return false;
    };
    const int64_t pitch = paged ? p.slot_stride : (int64_t)p.H * kStateFloats;
    float* dst = paged ? const_cast<float*>(p.h0) : p.ht;
    int64_t off0 = 0, off1 = 0, off2 = 0;        // what the stages hold
    static_assert(kStages == 3, "three offsets");
    int n = blockIdx.x, loads = 0, st = 0;
    auto load = [&](int s) {
      const int64_t o = slot * pitch + (int64_t)(n % p.H) * kStateFloats;
      if (s == 0) off0 = o; else if (s == 1) off1 = o; else off2 = o;
      mbar_expect_tx(&full[s], kStateBytes);
      bulk_load(ring + s * kStateFloats, p.h0 + o, kStateBytes, &full[s]);
      ++loads;
      n += stride;
    };
    while (loads < kStages && find(n)) load(loads);
    uint32_t ph = 0;
    int stores = 0;
    for (; stores < loads; ++stores) {
      const bool more = find(n);                 // looked up before the wait
      if (!wait_unless(&done[st], ph, s_abort, polls(stores))) { give_up(s_abort, error); break; }
      bulk_store(dst + (st == 0 ? off0 : (st == 1 ? off1 : off2)), ring + st * kStateFloats, kStateBytes);
      tma_store_commit();
      if (more) {
        tma_store_wait_read();                   // the stage has been read: it takes the next state
        load(st);
      }
      if (++st == kStages) { st = 0; ph ^= 1; }
    }
    // (after a full run every load has been waited for) what is still on its way has to land in this CTA's shared memory
    for (int l = stores; l < loads; ++l) mbar_wait(&full[l % kStages], (l / kStages) & 1);
    tma_store_wait_read();
    return;
  }

  if (warp > 16) {
    // ---- operands ----------------------------------------------------------------------------------------
    const int pair = (warp - 17) >> 1, half = (warp - 17) & 1;
    // Part 0, 1, 2 = q, k, v of the lane's eight channels; the second half of warp 1 brings the gate.
    const int c16 = lane & 15;
    const bool gates = half == 1 && lane >= 16;
    int step = 0;
    for (int n = blockIdx.x; n < items; n += stride) {
      const int seq = n / p.H;
      float x[8], beta = 0.f;
      if constexpr (W == 0) {
        if (slot_of(p, seq) < 0) continue;
        if (step++ % kPairs != pair) continue;
        const void* base = half == 0 ? (lane < 16 ? p.q : p.k) : (lane < 16 ? p.v : p.g);
        const int dt = half == 0 ? (lane < 16 ? p.dt_q : p.dt_k) : (lane < 16 ? p.dt_v : p.dt_g);
        Raw8 raw;
        load8(base, dt, (int64_t)n * 128 + 8 * c16, raw);
        if (half == 0 && lane == 0) beta = load_as_float(p.beta, p.dt_beta, n);
        to_floats(raw, dt, x);
      } else {
        // The history of a (sequence, head) is advanced here and nowhere else.  A slot that only one of the two pools has:
        // the history moves alone, or the state sees zero operands and a unit decay.
        const int nvec = 3 * p.H * 16, part = half == 0 ? lane >> 4 : 2, head = n - seq * p.H, si = p.state_indices[seq];
        const bool live = si > 0 && si < p.num_slots, conv = si > 0 && si < d.num_slots;
        const bool mine = step % kPairs == pair;
        if (live) ++step;
        if (!mine || !(live || conv)) continue;
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = 0.f;
        if (live && half == 0 && lane == 0) beta = load_as_float(p.beta, p.dt_beta, n);
        if (conv && gates) {
          Raw8 raw;
          load8(d.raw_gate, d.dt_gate, (int64_t)n * 128 + 8 * c16, raw);
          const float4* bias = reinterpret_cast<const float4*>(d.dt_bias + head * 128 + 8 * c16);
          const float4 b0 = bias[0], b1 = bias[1];
          const float a = expf(d.A_log[head]);
          to_floats(raw, d.dt_gate, x);
          const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = decode_gate(a, x[e], bb[e], d.lower_bound);
        } else if (conv) {
          const int vec = part * p.H * 16 + head * 16 + c16;
          uint4* hist = reinterpret_cast<uint4*>(d.conv_state) + si * (int64_t)(W - 1) * nvec + vec;
          const uint4* wv = reinterpret_cast<const uint4*>(d.w) + (int64_t)vec * W;
          uint4 raw[W], wraw[W];
#pragma unroll
          for (int j = 0; j < W - 1; ++j) raw[j] = hist[(int64_t)j * nvec];
          raw[W - 1] = reinterpret_cast<const uint4*>(d.x)[(int64_t)seq * nvec + vec];
#pragma unroll
          for (int j = 0; j < W; ++j) wraw[j] = wv[j];
          conv8<W>(raw, wraw, d.dt, d.act, x);
#pragma unroll
          for (int j = 0; j < W - 1; ++j) hist[(int64_t)j * nvec] = raw[j + 1];      // shift left, append x
        }
        __syncwarp();
        const float r = row_rnorm(x, d.eps);
        if (!live) continue;
        if (!gates) {
          if (half == 0) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] *= r;
          }
          raw8_to_float(float8_to_raw(x, d.dt), d.dt, x);      // the rows the stand-alone preprocessing stores
        }
      }
      const int at = step - 1, slot = at % kSlots;
      if (!__all_sync(0xffffffffu, wait_unless(&op_free[slot], ((at / kSlots) & 1) ^ 1, s_abort, polls(at)))) {
        give_up(s_abort, error);
        return;
      }
      publish(ops + slot * kSlotFloats, half, lane, x, beta, p.scale);
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[slot]);
    }
    return;
  }

  // ---- arithmetic --------------------------------------------------------------------------------------------
  const int grp = warp >> 2, wj = warp & 3, col = 32 * grp + lane;
  float* red = s_red + grp * 512;
  int st = 0, step = 0;
  uint32_t ph = 0;
  for (int n = blockIdx.x; n < items; n += stride) {
    if (slot_of(p, n / p.H) < 0) {            // padding rows produce zero output and leave the pool untouched
      if (wj == 0) store_from_float(p.out, p.dt_out, (int64_t)n * 128 + col, 0.f);
      continue;
    }
    bool ready = wait_unless(&full[st], ph, s_abort, polls(step));
    float* S = ring + st * kStateFloats + 32 * wj * 128 + col;
    f32x2 s[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = pack2(S[2 * i * 128], S[(2 * i + 1) * 128]);
    const int slot = step % kSlots;
    ready = ready && wait_unless(&op_full[slot], (step / kSlots) & 1, s_abort, polls(step));
    volatile int* stop = s_stop + 2 * grp + (step & 1);      // (a warp that is a step ahead writes the other one)
    if (!ready) {
      give_up(s_abort, error);
      *stop = 1;
    }
    const float* o = ops + slot * kSlotFloats;
    const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(o + 32 * wj);
    const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(o + 128 + 32 * wj);
    const ulonglong2* d4 = reinterpret_cast<const ulonglong2*>(o + 256 + 32 * wj);
    f32x2 pk = 0, pq = 0;       // (zero bits: +0, +0) even rows in the low half, odd in the high
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const ulonglong2 dd = d4[i], kk = k4[i], qq = q4[i];
      s[2 * i] = mul2(s[2 * i], dd.x);
      s[2 * i + 1] = mul2(s[2 * i + 1], dd.y);
      pk = fma2(kk.x, s[2 * i], pk);
      pq = fma2(qq.x, s[2 * i], pq);
      pk = fma2(kk.y, s[2 * i + 1], pk);
      pq = fma2(qq.y, s[2 * i + 1], pq);
    }
    const float2 x = unpack2(pk), y = unpack2(pq);
    float* r = red + (step & 1) * 256 + lane;        // (the other parity may still be read)
    r[32 * wj] = x.x + x.y;
    r[128 + 32 * wj] = y.x + y.y;
    asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
    const float a = (r[0] + r[32]) + (r[64] + r[96]);
    const float delta = o[513] * (o[384 + col] - a);
    if (*stop) break;                                        // the whole group, and this state stays as it was
    if (wj == 0) {
      const float out = fmaf(o[512], delta, (r[128] + r[160]) + (r[192] + r[224]));
      store_from_float(p.out, p.dt_out, (int64_t)n * 128 + col, out);
    }
    const f32x2 delta2 = pack2(delta, delta);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const ulonglong2 kk = k4[i];
      const float2 u = unpack2(fma2(kk.x, delta2, s[2 * i])), v = unpack2(fma2(kk.y, delta2, s[2 * i + 1]));
      S[4 * i * 128] = u.x; S[(4 * i + 1) * 128] = u.y; S[(4 * i + 2) * 128] = v.x; S[(4 * i + 3) * 128] = v.y;
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&op_free[slot]);
      mbar_arrive(&done[st]);                           // 16 arrivals hand the state to the copying warp
    }
    ++step;
    if (++st == kStages) { st = 0; ph ^= 1; }
  }
}

__device__ int g_stream_error = 0;

template <int W, bool SHORT = false>
int launch(const ScanParams& p, const PrepDecodeParams& d, cudaStream_t stream, ShortWait short_wait = {}) {
  const int64_t items = (int64_t)p.nseq * p.H;
  if (items <= 0) return KDA_OK;
  int* error = nullptr;
  if (cudaGetSymbolAddress(reinterpret_cast<void**>(&error), g_stream_error) != cudaSuccess ||
      cudaFuncSetAttribute(kda_stream_kernel<W, SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess)
    return KDA_ERR_LAUNCH;
  const int sms = device_sms();
  StageScope timing(kStageRecurrent, stream);
  kda_stream_kernel<W, SHORT><<<(unsigned)(items < sms ? items : sms), kThreads, kSmemBytes, stream>>>(p, d, error, short_wait);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

}  // namespace

bool stream_takes(const ScanParams& p) {
  return p.K == 128 && p.V == 128 && p.h0 && (p.state_indices || p.ht) && p.nseq * (int64_t)p.H < (1 << 24) &&
         (((uintptr_t)p.h0 | (uintptr_t)p.ht) & 15) == 0 &&
         (!p.state_indices || (p.slot_stride % 4 == 0 && p.slot_stride >= (int64_t)p.H * kStateFloats));
}
int launch_stream(const ScanParams& p, cudaStream_t stream) { return launch<0>(p, PrepDecodeParams{}, stream); }

int launch_fused_decode(const PrepDecodeParams& d, const ScanParams& p, cudaStream_t stream) {
  if (d.W == 4) return launch<4>(p, d, stream);
  if (d.W == 3) return launch<3>(p, d, stream);
  return launch<2>(p, d, stream);
}

int launch_stream_short(const ScanParams& p, int warp, int step, cudaStream_t stream) {
  return launch<0, true>(p, PrepDecodeParams{}, stream, ShortWait{warp, step});
}

int stream_error_word() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_stream_error, sizeof(int)) != cudaSuccess) return -1;
  cudaMemcpyToSymbol(g_stream_error, &zero, sizeof(int));
  return v;
}

}  // namespace kda
