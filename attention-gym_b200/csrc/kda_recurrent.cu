// Token-sequential KDA recurrence: entry points, and the token scan (inference prefill, a few tokens per sequence,
// the fp32-accurate evaluation of chunk_kda).  One token per sequence at K = V = 128 is state streaming: kda_stream.cu.
//
// Replaces the reference's Triton scan `_kda_recurrent_fwd_kernel`
// (attn_gym/linear/kda/fwd/triton/recurrent.py:41-153).  Per token, per (sequence, head):
//     S <- diag(2^g) S ;  d = beta (v - S^T k) ;  S <- S + k d^T ;  o = scale S^T q
// The two K-reductions of a step (S^T k and S^T q, both taken on the decayed state) share one
// exchange:  o = scale (S_d^T q + (q.k) d).
#include <type_traits>

#include "kda_recurrent.cuh"
#include "kda_timing.cuh"

namespace kda {

// ------------------------------------------------------------------------------------------------
// Token scan.  Every computing warp owns 4 VC columns of the fp32 state and keeps them in registers for
// the whole scan: lane (lk = lane / 4, cv = lane % 4) holds VC adjacent columns and the key rows
// 4 (lk + 8 i) .. + 3, i < KR / 4, as pairs of rows for the packed fp32 arithmetic.  The K-reductions
// are three shuffles, so no token needs a barrier.  The CTA's warps share one (sequence, head): its
// operands are fetched TT tokens at a time, one tile ahead of their use (raw bits in registers), and
// published to shared memory as fp32 (q scaled, 2^g) with one barrier per tile.
//
// A long scan of few sequences is bound by the latency of one token: the dependent chain of decay, reduction, three shuffles
// and update.  So NP warps of their own fetch, publish and store (NP = 0: the computing warps do it), and up to K = 128 the next
// token's operands are read from shared memory before the shuffles.  T = 512, H = 4, K = V = 64: 114 us without moving warps, 79 with.
// A short scan of many sequences is bound by the state traffic and by how much of it two CTAs per SM
// can keep in flight: 48 sequences of 1 to 8 tokens, H = 32, K = V = 128 (212 MB): 58.9 us, with four of half the columns 57.6
// (60.9 and 59.5 over four pools in turn).  (Three CTAs of half the columns per lane: 74 us; asking the next CTA's state into L2: no change.)
// CUM: the gate is the cumulative one of chunk_kda; the per-token gate is its difference inside the
// 64-token chunks of a sequence.
// ------------------------------------------------------------------------------------------------
template <int KR, int VC, int NW, int NP, int TT, bool CUM, int MINB>
__global__ void __launch_bounds__(32 * (NW + NP), MINB) kda_scan_kernel(const ScanParams p) {
  constexpr int NT = 32 * (NP ? NP : NW);          // threads that fetch and publish operands
  constexpr int KP = 8 * KR, CT = 4 * VC * NW;
  constexpr int NE = TT * KP / NT;                 // operand elements per thread, array and tile
  constexpr int NV = (TT * CT + NT - 1) / NT;      // value and output elements per thread and tile
  constexpr int NR = KR / 4;
  constexpr bool kPrefetch = VC == 1 && KR <= 16 && NP > 0;
  static_assert(TT * KP % NT == 0 && TT <= 32, "tile split");
  __shared__ __align__(16) float s_q[2][TT][KP], s_k[2][TT][KP], s_d[2][TT][KP];
  __shared__ float s_v[2][TT][CT], s_o[2][TT][CT], s_beta[2][TT];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cv = lane & 3, lk = lane >> 2;
  const bool computes = warp < NW, moves = NP == 0 || warp >= NW;
  const int tid = NP ? (int)threadIdx.x - 32 * NW : (int)threadIdx.x;     // index among the moving threads
  const int K = p.K, V = p.V, H = p.H;
  const int vtiles = (V + CT - 1) / CT;
  const int vt = blockIdx.x % vtiles, sh = blockIdx.x / vtiles;
  const int head = sh % H, seq = sh / H;
  int64_t bos, eos;
  if (p.cu_seqlens) { bos = p.cu_seqlens[seq]; eos = p.cu_seqlens[seq + 1]; }
  else { bos = (int64_t)seq * p.T; eos = bos + p.T; }
  const int cta0 = vt * CT, wc = 4 * VC * warp + VC * cv, c0 = cta0 + wc;    // this lane's first column

  int64_t slot = seq;
  bool active = true;
  if (p.state_indices) {
    const int si = p.state_indices[seq];
    active = si > 0 && si < p.num_slots;   // non-positive (or out of range) slots are padding
    slot = si;
  }
  if (!active) {  // padding rows produce zero output and leave the pool untouched
    for (int64_t t = bos; t < eos; ++t)
      for (int c = cta0 + (int)threadIdx.x; c < min(cta0 + CT, V); c += 32 * (NW + NP))
        store_from_float(p.out, p.dt_out, (t * H + head) * V + c, 0.f);
    return;
  }
  const bool paged = p.state_indices != nullptr;
  const float* sin = p.h0 ? p.h0 + (paged ? slot * p.slot_stride : (int64_t)seq * H * K * V) +
                                (int64_t)head * K * V : nullptr;
  float* sout = paged ? const_cast<float*>(sin)
                      : (p.ht ? p.ht + ((int64_t)seq * H + head) * K * V : nullptr);

  // ---- operand tiles: raw bits in registers, published as fp32 ----------------------------------------
  // (a warp's elements of one n belong to one token, so tokens past the end cost it nothing)
  uint32_t rq[NE], rk[NE], rg[NE], rp[CUM ? NE : 1], rv[NV], rb = 0;
  auto bits = [](const void* base, int dt, int64_t at, int off) -> uint32_t {
    if (dt == KDA_F32) return (reinterpret_cast<const uint32_t*>(base) + at)[off];
    return (reinterpret_cast<const unsigned short*>(base) + at)[off];
  };
  auto fetch = [&](int64_t t0) {
    const int ntok = (int)min((int64_t)TT, eos - t0);
    const int64_t kbase = (t0 * H + head) * K, vbase = (t0 * H + head) * V + cta0;
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + n * NT, tok = e / KP, r = e % KP, off = tok * H * K + r;
      rq[n] = rk[n] = rg[n] = 0;
      if (CUM) rp[n] = 0;
      if (tok < ntok && r < K) {
        rq[n] = bits(p.q, p.dt_q, kbase, off);
        rk[n] = bits(p.k, p.dt_k, kbase, off);
        rg[n] = bits(p.g, p.dt_g, kbase, off);
        if (CUM && (((int)(t0 - bos) + tok) & (kChunk - 1)) != 0) rp[n] = bits(p.g, p.dt_g, kbase, off - H * K);
      }
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int e = tid + n * NT, tok = e / CT, c = e % CT;
      rv[n] = (tok < ntok && cta0 + c < V) ? bits(p.v, p.dt_v, vbase, tok * H * V + c) : 0;
    }
    if (tid < ntok) rb = bits(p.beta, p.dt_beta, t0 * H + head, tid * H);
  };
  auto publish = [&](int b, int ntok) {
#pragma unroll
    for (int n = 0; n < NE; ++n) {
      const int e = tid + n * NT, tok = e / KP, r = e % KP;
      if (NP || tok < ntok) {        // (a long scan's tiles are whole but for the last one)
        s_q[b][tok][r] = raw_to_float(rq[n], p.dt_q) * p.scale;
        s_k[b][tok][r] = raw_to_float(rk[n], p.dt_k);
        float g = raw_to_float(rg[n], p.dt_g);
        if (CUM) g -= raw_to_float(rp[n], p.dt_g);
        s_d[b][tok][r] = exp2f(g);
      }
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int e = tid + n * NT;
      if (e / CT < ntok) s_v[b][e / CT][e % CT] = raw_to_float(rv[n], p.dt_v);
    }
    if (tid < ntok) s_beta[b][tid] = raw_to_float(rb, p.dt_beta);
  };
  if (moves) fetch(bos);
  // ---- state slab: S[i][j] holds the rows 2 i, 2 i + 1 of this lane's list in column j -----------------------
  f32x2 S[KR / 2][VC];
  {
    float x[2][VC];
#pragma unroll
    for (int i = 0; i < KR; ++i) {
      const int r = 4 * (lk + 8 * (i >> 2)) + (i & 3);
      float (&xr)[VC] = x[i & 1];
#pragma unroll
      for (int j = 0; j < VC; ++j) xr[j] = 0.f;
      if (computes && sin && r < K) {
        if (VC > 1) {             // (V is a multiple of 4 then, and so is every column offset)
          if (c0 < V) {
            if (VC == 4) {
              const float4 f = *reinterpret_cast<const float4*>(sin + (int64_t)r * V + c0);
              xr[0] = f.x; xr[1 % VC] = f.y; xr[2 % VC] = f.z; xr[3 % VC] = f.w;
            } else {
              const float2 f = *reinterpret_cast<const float2*>(sin + (int64_t)r * V + c0);
              xr[0] = f.x; xr[1 % VC] = f.y;
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < VC; ++j)
            if (c0 + j < V) xr[j] = sin[(int64_t)r * V + c0 + j];
        }
      }
      if (i & 1) {
#pragma unroll
        for (int j = 0; j < VC; ++j) S[i >> 1][j] = pack2(x[0][j], x[1][j]);
      }
    }
  }

  auto flush = [&](int64_t t0, int b, int ntok) {      // the outputs of a tile
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int e = tid + n * NT, tok = e / CT, c = e % CT;
      if (tok < ntok && cta0 + c < V)
        store_from_float(p.out, p.dt_out, (t0 * H + head) * V + cta0 + (tok * H * V + c), s_o[b][tok][c]);
    }
  };
  if (moves) publish(0, (int)min((int64_t)TT, eos - bos));
  __syncthreads();
  int b = 0;
  for (int64_t t0 = bos; t0 < eos; t0 += TT, b ^= 1) {
    const bool more = t0 + TT < eos;
    const int ntok = more ? TT : (int)(eos - t0);
    if (moves && more) fetch(t0 + TT);
    if (NP && moves && t0 > bos) flush(t0 - TT, b ^ 1, TT);
    if (computes) {
    // The operands of a long scan's next token are read from shared memory between the two halves of
    // a step, where their latency hides behind the shuffles.
    f32x2 q[KR / 2], k[KR / 2], d[KR / 2];
    auto read = [&](int tok, f32x2 (&qd)[KR / 2], f32x2 (&kd)[KR / 2], f32x2 (&dd)[KR / 2]) {
      const ulonglong2* qs = reinterpret_cast<const ulonglong2*>(s_q[b][tok]) + lk;
      const ulonglong2* ks = reinterpret_cast<const ulonglong2*>(s_k[b][tok]) + lk;
      const ulonglong2* ds = reinterpret_cast<const ulonglong2*>(s_d[b][tok]) + lk;
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const ulonglong2 a = qs[8 * i], c = ks[8 * i], e = ds[8 * i];
        qd[2 * i] = a.x; qd[2 * i + 1] = a.y;
        kd[2 * i] = c.x; kd[2 * i + 1] = c.y;
        dd[2 * i] = e.x; dd[2 * i + 1] = e.y;
      }
    };
    if (kPrefetch) read(0, q, k, d);
#pragma unroll(kPrefetch ? 2 : 1)
    for (int tok = 0; tok < ntok; ++tok) {
      f32x2 pk[VC], pq[VC], pqk = 0;       // (zero bits: +0, +0) even rows in the low half, odd in the high
#pragma unroll
      for (int j = 0; j < VC; ++j) pk[j] = pq[j] = 0;
      const ulonglong2* ks = reinterpret_cast<const ulonglong2*>(s_k[b][tok]) + lk;
#pragma unroll
      for (int i = 0; i < KR / 2; ++i) {
        if (!kPrefetch && i % 2 == 0) {
          const ulonglong2 x = reinterpret_cast<const ulonglong2*>(s_q[b][tok])[lk + 4 * i], y = ks[4 * i],
                           z = reinterpret_cast<const ulonglong2*>(s_d[b][tok])[lk + 4 * i];
          q[i] = x.x; q[i + 1] = x.y; k[i] = y.x; k[i + 1] = y.y; d[i] = z.x; d[i + 1] = z.y;
        }
        pqk = fma2(q[i], k[i], pqk);
#pragma unroll
        for (int j = 0; j < VC; ++j) {
          S[i][j] = mul2(S[i][j], d[i]);
          pk[j] = fma2(k[i], S[i][j], pk[j]);
          pq[j] = fma2(q[i], S[i][j], pq[j]);
        }
      }
      float a[VC], o[VC];
      const float2 x = unpack2(pqk);
      float qk = x.x + x.y;
#pragma unroll
      for (int j = 0; j < VC; ++j) {
        const float2 y = unpack2(pk[j]), z = unpack2(pq[j]);
        a[j] = y.x + y.y;
        o[j] = z.x + z.y;
      }
      f32x2 qn[KR / 2], kn[KR / 2], dn[KR / 2];
      if (kPrefetch) read(tok + 1 < TT ? tok + 1 : tok, qn, kn, dn);
#pragma unroll
      for (int m = 4; m < 32; m <<= 1) {
#pragma unroll
        for (int j = 0; j < VC; ++j) {
          a[j] += __shfl_xor_sync(0xffffffffu, a[j], m);
          o[j] += __shfl_xor_sync(0xffffffffu, o[j], m);
        }
        qk += __shfl_xor_sync(0xffffffffu, qk, m);
      }
      const float bt = s_beta[b][tok];
      float mine = 0.f;                    // lane row lk < VC keeps column lk of its group
      f32x2 delta2[VC];
#pragma unroll
      for (int j = 0; j < VC; ++j) {
        const float delta = bt * (s_v[b][tok][wc + j] - a[j]);
        const float out = fmaf(qk, delta, o[j]);
        if (lk == j) mine = out;
        delta2[j] = pack2(delta, delta);
      }
#pragma unroll
      for (int i = 0; i < KR / 2; ++i) {
        if (!kPrefetch && i % 2 == 0) { const ulonglong2 y = ks[4 * i]; k[i] = y.x; k[i + 1] = y.y; }      // read again: fewer registers
#pragma unroll
        for (int j = 0; j < VC; ++j) S[i][j] = fma2(k[i], delta2[j], S[i][j]);
      }
      if (lk < VC) s_o[b][tok][wc + lk] = mine;
      if (kPrefetch) {
#pragma unroll
        for (int i = 0; i < KR / 2; ++i) { q[i] = qn[i]; k[i] = kn[i]; d[i] = dn[i]; }
      }
    }
    }
    if (moves && more) publish(b ^ 1, (int)min((int64_t)TT, eos - t0 - TT));   // those buffers were last read before the previous barrier
    __syncthreads();
    if (moves && (NP == 0 || !more)) flush(t0, b, ntok);
  }

  if (sout && computes) {
#pragma unroll
    for (int i = 0; i < KR; ++i) {
      const int r = 4 * (lk + 8 * (i >> 2)) + (i & 3);
      float x[VC];
#pragma unroll
      for (int j = 0; j < VC; ++j) {
        const float2 y = unpack2(S[i >> 1][j]);
        x[j] = (i & 1) ? y.y : y.x;
      }
      if (r < K) {
        if (VC > 1) {
          if (c0 < V) {
            if (VC == 4) *reinterpret_cast<float4*>(sout + (int64_t)r * V + c0) = make_float4(x[0], x[1 % VC], x[2 % VC], x[3 % VC]);
            else *reinterpret_cast<float2*>(sout + (int64_t)r * V + c0) = make_float2(x[0], x[1 % VC]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < VC; ++j)
            if (c0 + j < V) sout[(int64_t)r * V + c0 + j] = x[j];
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Token scan of few chains: four tokens at a time.  With D_i the product of the decays of a block's tokens 0 .. i and S
// the state that enters the block,
//     a_i = (k_i D_i)^T S + sum_{j < i} P_ij d_j,     P_ij = sum_kappa k_i k_j D_i / D_j,     d_i = beta_i (v_i - a_i)
//     o_i = (q_i D_i)^T S + sum_{j <= i} Q_ij d_j,    Q_ij = sum_kappa q_i k_j D_i / D_j
//     S  <- D_3 S + sum_j (k_j D_3 / D_j) d_j
// so the dot products with the state and their shuffles, most of a token's dependent chain, are taken once for
// four tokens, and what is left token by token are two scalar operations.  Everything that does not depend on the state
// (the scaled rows, the ten Q and six P, as products of decays: no division, no difference of logarithms) is made by four
// warps of their own, two channels per thread, one tile of blocks ahead, from operands fetched two tiles ahead.  A block that
// the sequence does not fill has zero rows and unit decays at its end.  The computing warps own four columns each: lane (lk = lane / 4, lane % 4) holds one column and the
// key rows 4 (lk + 8 i) .. + 3.  Bound by the chain from block to block (two dot products per token, three rounds of
// shuffles, four corrections, the update).  fp32, 4 chains, 512 tokens from the cumulative gate, us, one token at a time /
// blocks: K = V = 32 60 / 46, 64 80 / 50, 96 147 / 77, 128 147 / 78.  The error against 64 bits is the same; with one channel per
// thread (its products rounded before the sum) it was 3 to 8 % larger at gates that forget fast.  (The state is
// rounded five times a block instead of eight.)
// ------------------------------------------------------------------------------------------------
// Every operand is fp32.  (The same with a type test per operand and load, bf16 q, k and v: the moving warps took longer than the
// computing ones, and at K = V = 128 nothing was left of the gain: 32 chains of 100 tokens 53.7 us, one token at a time 52.1; 4 chains of
// 5 tokens 5.2 / 4.9.)
template <int KR, bool CUM>
__global__ void __launch_bounds__(256, 1) kda_block_scan_kernel(const ScanParams p) {
  constexpr int C = 4, KP = 8 * KR, NR = KR / 4, CT = 16;
  constexpr int LB = KP / 2, SW = (LB + 31) / 32;           // moving threads of a block (two channels each) and their warps
  constexpr int NB = 128 / LB, TT = C * NB;                 // blocks and tokens of a tile: 32, 16 or 8
  __shared__ __align__(16) float s_kt[2][TT][KP], s_qt[2][TT][KP], s_kn[2][TT][KP], s_dc[2][NB][KP];
  __shared__ __align__(16) float s_p[2][NB][SW][16], s_v[2][TT][CT], s_o[2][TT][CT], s_beta[2][TT];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cv = lane & 3, lk = lane >> 2;
  const bool moving = warp >= 4;
  const int tid = (int)threadIdx.x - 128;                   // index among the moving threads
  const int K = p.K, V = p.V, H = p.H;
  const int vtiles = (V + CT - 1) / CT;
  const int vt = blockIdx.x % vtiles, sh = blockIdx.x / vtiles;
  const int head = sh % H, seq = sh / H;
  int64_t bos, eos;
  if (p.cu_seqlens) { bos = p.cu_seqlens[seq]; eos = p.cu_seqlens[seq + 1]; }
  else { bos = (int64_t)seq * p.T; eos = bos + p.T; }
  const int cta0 = vt * CT, wc = 4 * warp + cv, c0 = cta0 + wc;       // this lane's column
  const bool paged = p.state_indices != nullptr;
  const int64_t slot = paged ? p.state_indices[seq] : seq;
  if (paged && (slot <= 0 || slot >= p.num_slots)) {   // padding: zero output, the pool untouched
    for (int64_t t = bos + (threadIdx.x >> 4); t < eos; t += 16) {
      const int c = cta0 + (threadIdx.x & 15);
      if (c < V) store_from_float(p.out, p.dt_out, (t * H + head) * V + c, 0.f);
    }
    return;
  }
  const float* sin = p.h0 ? p.h0 + (paged ? slot * p.slot_stride : slot * H * K * V) + (int64_t)head * K * V : nullptr;
  float* sout = paged ? const_cast<float*>(sin) : (p.ht ? p.ht + (slot * H + head) * K * V : nullptr);

  // ---- operand tiles: in registers, two tiles ahead; a moving thread owns two channels of one block ----
  // (one base address per operand and 32-bit offsets from it: with 64-bit index arithmetic the moving warps took longer than the
  // computing ones)
  const int blk0 = tid / LB, ch = 2 * (tid % LB), tok0 = C * blk0;       // (moving threads only)
  const bool in0 = ch < K, in1 = ch + 1 < K;
  float rq[C][2], rk[C][2], rg[C][2], rp[2], rv[TT * CT / 128], rb = 0.f;
  auto operand = [](const void* base, int64_t at) { return reinterpret_cast<const float*>(base) + at; };
  const int64_t kat = (bos * H + head) * K + (in0 ? ch : 0), vat = (bos * H + head) * V + cta0;
  const float *bq = operand(p.q, kat), *bk = operand(p.k, kat), *bg = operand(p.g, kat), *bv = operand(p.v, vat),
              *bb = operand(p.beta, bos * H + head);
  const uint32_t krow = (uint32_t)H * K, vrow = (uint32_t)H * V;      // (a tile of rows is well below 2^31 bytes)
  auto fetch = [&](int64_t t0) {
    const int ntok = (int)min((int64_t)TT, eos - t0);
    const int64_t kt = (t0 - bos) * krow, vt0 = (t0 - bos) * vrow, bt0 = (t0 - bos) * H;
    const float *q = bq + kt, *k = bk + kt, *g = bg + kt, *v = bv + vt0;
    // the gate before the block, unless the block starts a chunk (a block never straddles two)
    const bool before = CUM && tok0 < ntok && (((int)(t0 - bos) + tok0) & (kChunk - 1)) != 0;
    const float* gp = g - krow;
    rp[0] = before && in0 ? gp[tok0 * krow] : 0.f;
    rp[1] = before && in1 ? gp[tok0 * krow + 1] : 0.f;
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const bool live = tok0 + i < ntok;
      const uint32_t off = (uint32_t)(tok0 + i) * krow;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const bool in = live && (u ? in1 : in0);
        rq[i][u] = in ? q[off + u] : 0.f;
        rk[i][u] = in ? k[off + u] : 0.f;
        rg[i][u] = in ? g[off + u] : 0.f;
      }
    }
#pragma unroll
    for (int n = 0; n < TT * CT / 128; ++n) {
      const int e = tid + n * 128, tok = e / CT, c = e % CT;
      rv[n] = (tok < ntok && cta0 + c < V) ? v[(uint32_t)tok * vrow + c] : 0.f;
    }
    rb = tid < ntok ? bb[bt0 + (uint32_t)tid * H] : 0.f;
  };
  auto publish = [&](int b, int ntok) {
    float q[C][2], k[C][2], d[C][2], kt[C][2], qt[C][2], kn[C][2], dc[2], x[16];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int i = 0; i < C; ++i) {
        q[i][u] = rq[i][u] * p.scale;
        k[i][u] = rk[i][u];
        float g = rg[i][u];
        if (CUM) g -= i == 0 ? rp[u] : rg[i == 0 ? 0 : i - 1][u];
        d[i][u] = tok0 + i < ntok ? exp2f(g) : 1.f;
      }
      const float d01 = d[0][u] * d[1][u], d12 = d[1][u] * d[2][u], d23 = d[2][u] * d[3][u], d123 = d12 * d[3][u];
      const float D[C] = {d[0][u], d01, d01 * d[2][u], d01 * d23}, E[C] = {d123, d23, d[3][u], 1.f};
#pragma unroll
      for (int i = 0; i < C; ++i) {
        kt[i][u] = k[i][u] * D[i];
        qt[i][u] = q[i][u] * D[i];
        kn[i][u] = k[i][u] * E[i];
      }
      dc[u] = D[3];
      const float k0d1 = k[0][u] * d[1][u], k0d12 = k[0][u] * d12, k1d2 = k[1][u] * d[2][u];
      // P10 P20 P21 P30 P31 P32 | Q00 Q10 Q11 Q20 Q21 Q22 Q30 Q31 Q32 Q33 as (row, column) factors
      const float f[16] = {k[1][u], k[2][u], k[2][u], k[3][u], k[3][u], k[3][u], q[0][u], q[1][u],
                           q[1][u], q[2][u], q[2][u], q[2][u], q[3][u], q[3][u], q[3][u], q[3][u]};
      const float h[16] = {k0d1, k0d12, k1d2, kn[0][u], kn[1][u], kn[2][u], k[0][u], k0d1,
                           k[1][u], k0d12, k1d2, k[2][u], kn[0][u], kn[1][u], kn[2][u], k[3][u]};
#pragma unroll
      for (int e = 0; e < 16; ++e) x[e] = u == 0 ? f[e] * h[e] : fmaf(f[e], h[e], x[e]);
    }
#pragma unroll
    for (int i = 0; i < C; ++i) {
      *reinterpret_cast<float2*>(&s_kt[b][tok0 + i][ch]) = make_float2(kt[i][0], kt[i][1]);
      *reinterpret_cast<float2*>(&s_qt[b][tok0 + i][ch]) = make_float2(qt[i][0], qt[i][1]);
      *reinterpret_cast<float2*>(&s_kn[b][tok0 + i][ch]) = make_float2(kn[i][0], kn[i][1]);
    }
    *reinterpret_cast<float2*>(&s_dc[b][blk0][ch]) = make_float2(dc[0], dc[1]);
    // sums over the block's lanes: afterwards lane e of 16, or lanes 2 e and 2 e + 1 of a warp, hold the total of entry e
#pragma unroll
    for (int off = LB >= 32 ? 16 : 8, m = 8; m >= 1; off >>= 1, m >>= 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j < m) {
          const bool up = (lane & off) != 0;
          const float send = up ? x[j] : x[j + m], keep = up ? x[j + m] : x[j];
          x[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
    }
    if (LB >= 32) {
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
      if ((lane & 1) == 0) s_p[b][blk0][warp & (SW - 1)][lane >> 1] = x[0];
    } else {
      s_p[b][blk0][0][lane & 15] = x[0];
    }
#pragma unroll
    for (int n = 0; n < TT * CT / 128; ++n) {
      const int e = tid + n * 128;
      s_v[b][e / CT][e % CT] = rv[n];
    }
    if (tid < TT) s_beta[b][tid] = rb;
  };
  auto flush = [&](int64_t t0, int b, int ntok) {      // the outputs of a tile
#pragma unroll
    for (int n = 0; n < TT * CT / 128; ++n) {
      const int e = tid + n * 128, tok = e / CT, c = e % CT;
      if (tok < ntok && cta0 + c < V) store_from_float(p.out, p.dt_out, ((t0 + tok) * H + head) * V + cta0 + c, s_o[b][tok][c]);
    }
  };

  if (moving) fetch(bos);
  // ---- state: S[i] holds the rows 2 i, 2 i + 1 of this lane's list, rows 4 (lk + 8 i) .. + 3 ----------------
  f32x2 S[KR / 2];
  auto row = [&](int i) { return 4 * (lk + 8 * (i >> 2)) + (i & 3); };
#pragma unroll
  for (int i = 0; i < KR; i += 2) {
    const bool in = !moving && sin && c0 < V;
    const float x = in && row(i) < K ? sin[(int64_t)row(i) * V + c0] : 0.f;
    const float y = in && row(i + 1) < K ? sin[(int64_t)row(i + 1) * V + c0] : 0.f;
    S[i >> 1] = pack2(x, y);
  }
  if (moving) {
    publish(0, (int)min((int64_t)TT, eos - bos));
    if (bos + TT < eos) fetch(bos + TT);
  }
  __syncthreads();
  int b = 0;
  for (int64_t t0 = bos; t0 < eos; t0 += TT, b ^= 1) {
    const bool more = t0 + TT < eos;
    const int ntok = more ? TT : (int)(eos - t0);
    if (moving) {
      if (more) publish(b ^ 1, (int)min((int64_t)TT, eos - t0 - TT));
      if (t0 + 2 * TT < eos) fetch(t0 + 2 * TT);
      if (t0 > bos) flush(t0 - TT, b ^ 1, TT);
    } else {
      // a block of which `live` tokens exist (tail: fewer than C; its own copy, because the test costs 8 % of the chain)
      auto block = [&](int blk, auto partial, int live) {
        constexpr bool tail = decltype(partial)::value;
        const int tok0 = C * blk;
        f32x2 pa[C], po[C];
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const ulonglong2* kt = reinterpret_cast<const ulonglong2*>(s_kt[b][tok0 + i]) + lk;
          const ulonglong2* qt = reinterpret_cast<const ulonglong2*>(s_qt[b][tok0 + i]) + lk;
          pa[i] = po[i] = 0;         // (zero bits: +0, +0) even rows in the low half, odd in the high
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            const ulonglong2 x = kt[8 * r], y = qt[8 * r];
            pa[i] = fma2(x.x, S[2 * r], pa[i]);
            po[i] = fma2(y.x, S[2 * r], po[i]);
            pa[i] = fma2(x.y, S[2 * r + 1], pa[i]);
            po[i] = fma2(y.y, S[2 * r + 1], po[i]);
          }
        }
        float a[C], o[C];
#pragma unroll
        for (int i = 0; i < C; ++i) {
          const float2 x = unpack2(pa[i]), y = unpack2(po[i]);
          a[i] = x.x + x.y;
          o[i] = y.x + y.y;
        }
#pragma unroll
        for (int m = 4; m < 32; m <<= 1) {
#pragma unroll
          for (int i = 0; i < C; ++i) {
            a[i] += __shfl_xor_sync(0xffffffffu, a[i], m);
            o[i] += __shfl_xor_sync(0xffffffffu, o[i], m);
          }
        }
        float w[16];                 // the pairwise products
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          float4 x = *reinterpret_cast<const float4*>(&s_p[b][blk][0][e]);
#pragma unroll
          for (int u = 1; u < SW; ++u) {
            const float4 y = *reinterpret_cast<const float4*>(&s_p[b][blk][u][e]);
            x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
          }
          w[e] = x.x; w[e + 1] = x.y; w[e + 2] = x.z; w[e + 3] = x.w;
        }
        const float4 bt = *reinterpret_cast<const float4*>(&s_beta[b][tok0]);
        const float (*vv)[CT] = &s_v[b][tok0];
        const float e0 = bt.x * (vv[0][wc] - a[0]);
        const float e1 = bt.y * (vv[1][wc] - fmaf(w[0], e0, a[1]));
        const float e2 = bt.z * (vv[2][wc] - fmaf(w[2], e1, fmaf(w[1], e0, a[2])));
        const float e3 = bt.w * (vv[3][wc] - fmaf(w[5], e2, fmaf(w[4], e1, fmaf(w[3], e0, a[3]))));
        // (tokens past the end add nothing: their zero rows against an infinite state would give NaN)
        const float e[C] = {e0, tail && live < 2 ? 0.f : e1, tail && live < 3 ? 0.f : e2, tail ? 0.f : e3};
        {
          const ulonglong2* dc = reinterpret_cast<const ulonglong2*>(s_dc[b][blk]) + lk;
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            const ulonglong2 x = dc[8 * r];
            S[2 * r] = mul2(S[2 * r], x.x);
            S[2 * r + 1] = mul2(S[2 * r + 1], x.y);
          }
        }
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const ulonglong2* kn = reinterpret_cast<const ulonglong2*>(s_kn[b][tok0 + j]) + lk;
          const f32x2 ej = pack2(e[j], e[j]);
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            const ulonglong2 x = kn[8 * r];
            S[2 * r] = fma2(x.x, ej, S[2 * r]);
            S[2 * r + 1] = fma2(x.y, ej, S[2 * r + 1]);
          }
        }
        o[0] = fmaf(w[6], e0, o[0]);
        o[1] = fmaf(w[8], e1, fmaf(w[7], e0, o[1]));
        o[2] = fmaf(w[11], e2, fmaf(w[10], e1, fmaf(w[9], e0, o[2])));
        o[3] = fmaf(w[15], e3, fmaf(w[14], e2, fmaf(w[13], e1, fmaf(w[12], e0, o[3]))));
        if (lk < C) s_o[b][tok0 + lk][wc] = lk == 0 ? o[0] : (lk == 1 ? o[1] : (lk == 2 ? o[2] : o[3]));
      };
      for (int blk = 0; blk < ntok / C; ++blk) block(blk, std::false_type{}, C);
      if (ntok % C) block(ntok / C, std::true_type{}, ntok % C);
    }
    __syncthreads();
    if (moving && !more) flush(t0, b, ntok);
  }
  if (sout && !moving && c0 < V) {
#pragma unroll
    for (int i = 0; i < KR; ++i) {
      const float2 y = unpack2(S[i >> 1]);
      if (row(i) < K) sout[(int64_t)row(i) * V + c0] = (i & 1) ? y.y : y.x;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Token scan of a few tokens: bound by the state traffic and by the length of the prologue, so nothing is
// fetched ahead.  A CTA owns 32 state columns in registers: warp w holds the key rows w, w + 8, .., a lane one
// column, so that every row access is one 128-byte line whatever V is.  The two K-reductions cross the
// warps through shared memory, one CTA barrier before and one after.
// ------------------------------------------------------------------------------------------------
template <int KR>
__global__ void __launch_bounds__(256) kda_short_scan_kernel(const ScanParams p) {
  constexpr int NW = 8;
  __shared__ float s_q[2][8 * KR], s_k[2][8 * KR], s_d[2][8 * KR];
  __shared__ float s_red[2][2][NW][32], s_qk[2][NW], s_beta[2];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = p.K, V = p.V, H = p.H, vtiles = (V + 31) / 32;
  const int vt = blockIdx.x % vtiles, sh = blockIdx.x / vtiles;
  const int head = sh % H, seq = sh / H, c = 32 * vt + lane;
  int64_t bos, eos;
  if (p.cu_seqlens) { bos = p.cu_seqlens[seq]; eos = p.cu_seqlens[seq + 1]; }
  else { bos = (int64_t)seq * p.T; eos = bos + p.T; }
  const bool paged = p.state_indices != nullptr;
  const int64_t slot = paged ? p.state_indices[seq] : seq;
  if (paged && (slot <= 0 || slot >= p.num_slots)) {   // padding: zero output, the pool untouched
    if (warp == 0 && c < V)
      for (int64_t t = bos; t < eos; ++t) store_from_float(p.out, p.dt_out, (t * H + head) * V + c, 0.f);
    return;
  }
  const float* sin = p.h0 ? p.h0 + (paged ? slot * p.slot_stride : slot * H * K * V) + (int64_t)head * K * V : nullptr;
  float* sout = paged ? const_cast<float*>(sin) : (p.ht ? p.ht + (slot * H + head) * K * V : nullptr);

  float S[KR];
#pragma unroll
  for (int i = 0; i < KR; ++i) {
    const int r = i * NW + warp;
    S[i] = (sin && r < K && c < V) ? sin[(int64_t)r * V + c] : 0.f;
  }
  auto stage = [&](int64_t t, int b) {      // a token's operands: q scaled, k, 2^g, beta
    const int64_t base = (t * H + head) * K;
    for (int r = tid; r < K; r += 256) {
      s_q[b][r] = load_as_float(p.q, p.dt_q, base + r) * p.scale;
      s_k[b][r] = load_as_float(p.k, p.dt_k, base + r);
      s_d[b][r] = exp2f(load_as_float(p.g, p.dt_g, base + r));
    }
    if (tid == 0) s_beta[b] = load_as_float(p.beta, p.dt_beta, t * H + head);
  };
  if (bos < eos) stage(bos, 0);
  for (int64_t t = bos; t < eos; ++t) {
    const int b = (int)((t - bos) & 1);
    const float v = c < V ? load_as_float(p.v, p.dt_v, (t * H + head) * V + c) : 0.f;
    __syncthreads();                        // the token is staged; the step before has been read
    float pk = 0.f, pq = 0.f, pqk = 0.f;
#pragma unroll
    for (int i = 0; i < KR; ++i) {
      const int r = i * NW + warp;
      if (r < K) {
        S[i] *= s_d[b][r];
        pqk = fmaf(s_q[b][r], s_k[b][r], pqk);
        pk = fmaf(s_k[b][r], S[i], pk);
        pq = fmaf(s_q[b][r], S[i], pq);
      }
    }
    s_red[b][0][warp][lane] = pk;
    s_red[b][1][warp][lane] = pq;
    if (lane == 0) s_qk[b][warp] = pqk;
    if (t + 1 < eos) stage(t + 1, b ^ 1);   // overlaps the exchange
    __syncthreads();
    float qk = 0.f, a = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      qk += s_qk[b][w];
      a += s_red[b][0][w][lane];
      o += s_red[b][1][w][lane];
    }
    const float delta = s_beta[b] * (v - a);
    if (warp == 0 && c < V) store_from_float(p.out, p.dt_out, (t * H + head) * V + c, fmaf(qk, delta, o));
#pragma unroll
    for (int i = 0; i < KR; ++i) {
      const int r = i * NW + warp;
      if (r < K) S[i] = fmaf(s_k[b][r], delta, S[i]);
    }
  }
  if (sout && c < V) {
#pragma unroll
    for (int i = 0; i < KR; ++i) {
      const int r = i * NW + warp;
      if (r < K) sout[(int64_t)r * V + c] = S[i];
    }
  }
}

template <int KR>
static int launch_short_scan(const ScanParams& p, cudaStream_t stream) {
  const int64_t blocks = (int64_t)p.nseq * p.H * ((p.V + 31) / 32);
  if (blocks <= 0) return KDA_OK;
  if (blocks > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  StageScope timing(kStageRecurrent, stream);
  kda_short_scan_kernel<KR><<<(unsigned)blocks, 256, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    return 148;
  return sms;
}

template <int KR>
static int launch_block_scan(const ScanParams& p, bool cumulative, cudaStream_t stream) {
  const int64_t blocks = (int64_t)p.nseq * p.H * ((p.V + 15) / 16);
  if (blocks <= 0) return KDA_OK;
  if (blocks > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  StageScope timing(kStageRecurrent, stream);
  if (cumulative) kda_block_scan_kernel<KR, true><<<(unsigned)blocks, 256, 0, stream>>>(p);
  else kda_block_scan_kernel<KR, false><<<(unsigned)blocks, 256, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

template <int KR, int VC, int NW, int NP, int MINB>
static int launch_scan(const ScanParams& p, bool cumulative, cudaStream_t stream) {
  constexpr int CT = 4 * VC * NW, KP = 8 * KR;
  // 24 KiB of operands in two buffers (K = 128: 8 tokens, 4 or 2 where four or eight CTAs share an SM); the wide form also buffers its
  // columns of v and o
  constexpr int TT = KP <= 64 ? (VC > 1 ? 8 : 16) : (MINB <= 2 ? 1024 : 2048 / MINB) / KP;
  const int64_t blocks = (int64_t)p.nseq * p.H * ((p.V + CT - 1) / CT);
  if (blocks <= 0) return KDA_OK;
  if (blocks > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  StageScope timing(kStageRecurrent, stream);
  if (cumulative) kda_scan_kernel<KR, VC, NW, NP, TT, true, MINB><<<(unsigned)blocks, 32 * (NW + NP), 0, stream>>>(p);
  else kda_scan_kernel<KR, VC, NW, NP, TT, false, MINB><<<(unsigned)blocks, 32 * (NW + NP), 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

// Which form a scan takes; `slices` is the number of 16-column slices of all chains, `tokens` the average length (of a packed call the
// capacity of its buffer over its sequences: their lengths are on the device), a turn as many slices as there are SMs.  Figures in us, both sides of each line (K = V = 128 unless said otherwise).
// * narrow: one column per lane, 16 columns per CTA, the shortest chain from token to token; wide: four columns per lane, 16-byte state
//   accesses, sixteen warps per SM.  bf16 q, k and v, narrow / wide above one turn up to 8 tokens: 32 chains (256 slices) 7.4 / 4.4 at 2
//   tokens, 9.7 / 9.7 at 8; above two turns from there on: 32 chains 17.1 / 20.9 at 24, 123 / 183 at 256, 48 chains (384) 24.9 / 21.0 at 24.
//   K = V = 32: one turn up to 6 tokens, 96 chains (192 slices) 3.8 / 3.6 at 2, 4.5 / 4.9 at 8; three from 48 tokens on, 192 chains (384) 16.7 /
//   18.3 at 48, 65 / 86 at 256, 320 chains (640) 24 / 21 and 100 / 99.  These two and the unaligned form below add in the same order: from
//   three tokens a sequence on, a sequence of 16-bit rows has the same bits in every batch.
// * fp32 operands take blocks of four tokens where the above is narrow: 4 chains of 5 / 24 / 512 tokens 4.9 / 9.4 / 126 one at a time, 4.1 / 6.5 /
//   74 in blocks.  Not for K = 32 and less above one turn, except from the cumulative gate: 96 chains (192 slices) of 24 tokens 6.9 / 8.7,
//   cumulative 10.8 / 8.5.
// * blocks or wide: the time of blocks grows with every turn.  Blocks / wide, 2 to 8 tokens, wide above one turn: 16 chains (128 slices)
//   5.6 / 6.6 at 2 tokens, 32 chains 9.2 / 6.5 at 2, 10.1 / 10.0 at 8; up to 15 tokens above two.  Above three turns from 16 tokens
//   on: 48 chains (384) 14 / 16 at 16 tokens, 21 / 27 at 32, 56 chains (448) 17 / 16 and 26 / 27; four from 64 on: 72 chains (576)
//   45 / 50 at 64, 151 / 185 at 256, 76 chains (608) 55 / 49 and 187 / 185.  K = V = 32 above two turns, 192 chains (384) 11 / 8 at
//   16, 20 / 19 at 48; from 64 on above three: 192 chains 40 / 46 at 128, 224 chains (448) 51 / 46.
//   128 columns per CTA and two CTAs per SM, or 64 and four, where 128 would leave half of a CTA without columns: 128 / 64 columns
//   at V = 64, 1024 chains of 64 tokens, K = 64 172 / 100, K = 128 271 / 160; above V = 64 only if CTAs of 128 columns are more than
//   two per SM: K = 72, V = 132, 8 tokens, 256 chains 25.5 / 22.0, 64 chains 9.4 / 10.5.  K = V = 32 runs 32 columns and eight CTAs per SM:
//   2048 chains of 64 tokens 230 / 71.
//   K = 64, V = 128 keeps 128 columns: 64 would gain up to four turns (48 chains, 384 slices, 6.2 / 5.7 at 6 tokens, 25.1 / 24.1 at 48) and
//   lose above (80 chains, 640 slices, 6.2 / 6.7 and 25.4 / 28.9).  K over 64 also runs 64 columns for few tokens, where the states' way in and out is most of the time, so that more CTAs
//   move states while others compute: up to 4 tokens (2048 chains of 4 tokens 58.9 / 55.4, of 6 72.6 / 74.7), up to 8 on average where
//   lengths differ (48 sequences of 32 heads 54.3 / 50.6 at 4, 89.9 / 86.7 at 8, 104 / 108 at 12).
//   Up to 2 tokens 32 columns and eight CTAs: 64 columns / 32, 48 sequences 42.3 / 38.0 at 1, 45.3 / 43.0 at 2, 50.4 / 49.8 at 3, 51.6 /
//   52.7 at 4; 128 sequences 101.6 / 91.3 at 1, 105.8 / 100.8 at 2.  Not for V up to 64 (2048 chains of 2 20.0 / 20.7) and the cumulative
//   gate (39.6 / 43.7).
// * many: state rows that are not 16-byte aligned, more than two turns: one column per lane, but 32 per CTA and two CTAs
//   per SM.  K = 128, V = 130, one token at a time in 16 / 32 columns: 48 chains (432 slices) 15.8 / 10.1 at 3 tokens, 56 / 44 at
//   64 (blocks of four: 56 at 64 and 384 slices).
// * the short scan for one token, and where the forms above lose to it.  K = 128, V = 64, short / blocks / wide: 16 chains
//   4.4 / 5.4 / 4.8 at 1 token, 6.2 / 5.5 / 5.5 at 2; 48 chains (192 slices) 4.6 / 9.0 / 5.1 at 1, 7.9 / 8.9 / 6.1 at 3, 9.9 / 8.9 /
//   6.8 at 4.  V = 130, 2048 chains, short / many 117 / 130 at 1, 184 / 142 at 2.  K = 256, V = 128, short / one column per
//   lane: 128 chains 14.7 / 21.3 at 1, 19.2 / 23.2 at 2; 16 chains (128 slices) 11.2 / 9.1 at 2.
static int launch_scan_any(const ScanParams& p, bool cumulative, cudaStream_t s) {
  const int sms = device_sms();
  const int64_t slices = (int64_t)p.nseq * p.H * ((p.V + 15) / 16);
  const int64_t tokens = p.cu_seqlens && p.nseq > 0 ? p.T / p.nseq : p.T;      // per sequence, on average
  const bool aligned = (((uintptr_t)p.h0 | (uintptr_t)p.ht) & 15) == 0 && p.V % 4 == 0 && p.slot_stride % 4 == 0;
  const bool f32 = p.dt_q == KDA_F32 && p.dt_k == KDA_F32 && p.dt_v == KDA_F32 && p.dt_g == KDA_F32 && p.dt_beta == KDA_F32;
  const bool blocks = f32 && p.K <= 128 && !(p.K <= 32 && !cumulative && slices > sms);
  const int more = blocks ? (tokens >= 16 && p.K > 32) + (tokens >= 64) : p.K <= 32 && !cumulative && tokens >= 48;
  const int turns = tokens >= 2 && tokens <= (p.K <= 32 && !cumulative ? 6 : 8) ? 1 : 2 + more;
  const bool wide = aligned && p.K <= 128 && slices > (int64_t)turns * sms;
  const bool many = !aligned && p.K <= 128 && slices > 2 * sms;
  const int few = p.K > 128 ? (slices > 2 * sms ? 2 : 1) : (many || slices <= sms ? 1 : (p.K <= 32 ? 1 + f32 : 2 + f32));
  if (!wide && !cumulative && tokens <= few) {
    if (p.K <= 32) return launch_short_scan<4>(p, s);
    if (p.K <= 64) return launch_short_scan<8>(p, s);
    if (p.K <= 128) return launch_short_scan<16>(p, s);
    return launch_short_scan<32>(p, s);
  }
  if (p.K > 128) return launch_scan<32, 1, 4, 4, 2>(p, cumulative, s);
  if (wide) {
    const bool narrow = (p.V - 1) % 128 < 64 && (p.V <= 64 || (int64_t)p.nseq * p.H * ((p.V + 127) / 128) > 2 * sms);
    if (p.K <= 32) {
      if (p.V <= 32) return launch_scan<4, 4, 2, 0, 8>(p, cumulative, s);
      if (narrow) return launch_scan<4, 4, 4, 0, 4>(p, cumulative, s);
      return launch_scan<4, 4, 8, 0, 2>(p, cumulative, s);
    }
    if (p.K <= 64) {
      if (narrow) return launch_scan<8, 4, 4, 0, 4>(p, cumulative, s);
      return launch_scan<8, 4, 8, 0, 2>(p, cumulative, s);
    }
    if (tokens <= 2 && p.V > 64 && !cumulative) return launch_scan<16, 4, 2, 0, 8>(p, cumulative, s);
    if (narrow || tokens <= (p.cu_seqlens ? 8 : 4)) return launch_scan<16, 4, 4, 0, 4>(p, cumulative, s);
    return launch_scan<16, 4, 8, 0, 2>(p, cumulative, s);
  }
  if (many) {
    if (p.K <= 32) return launch_scan<4, 1, 8, 0, 2>(p, cumulative, s);
    if (p.K <= 64) return launch_scan<8, 1, 8, 0, 2>(p, cumulative, s);
    return launch_scan<16, 1, 8, 0, 2>(p, cumulative, s);
  }
  if (blocks) {
    if (p.K <= 32) return launch_block_scan<4>(p, cumulative, s);
    if (p.K <= 64) return launch_block_scan<8>(p, cumulative, s);
    return launch_block_scan<16>(p, cumulative, s);
  }
  if (p.K <= 32) return launch_scan<4, 1, 4, 4, 1>(p, cumulative, s);
  if (p.K <= 64) return launch_scan<8, 1, 4, 4, 1>(p, cumulative, s);
  return launch_scan<16, 1, 4, 4, 1>(p, cumulative, s);
}

static int launch_recurrent(const ScanParams& p, cudaStream_t s) {
  if (p.T == 1 && !p.cu_seqlens && stream_takes(p)) return launch_stream(p, s);
  return launch_scan_any(p, false, s);
}

}  // namespace kda

extern "C" int kda_recurrent_fwd(const void* q, const void* k, const void* v, const void* gate,
                                 const void* beta, int dt_q, int dt_k, int dt_v, int dt_gate,
                                 int dt_beta, const float* initial_state, float* final_state,
                                 void* out, int dt_out, const int32_t* cu_seqlens,
                                 const int32_t* state_indices, int64_t slot_stride, int num_slots,
                                 int nseq, int tokens_per_row, int heads, int key_dim,
                                 int value_dim, float scale, void* stream) {
  using namespace kda;
  if (!q || !k || !v || !gate || !beta || !out) return KDA_ERR_ARG;
  if (nseq < 0 || heads <= 0 || key_dim <= 0 || key_dim > 256 || value_dim <= 0)
    return KDA_ERR_ARG;
  if (state_indices && !initial_state) return KDA_ERR_ARG;
  ScanParams p;
  p.q = q; p.k = k; p.v = v; p.g = gate; p.beta = beta;
  p.dt_q = dt_q; p.dt_k = dt_k; p.dt_v = dt_v; p.dt_g = dt_gate; p.dt_beta = dt_beta;
  p.h0 = initial_state; p.ht = final_state; p.out = out; p.dt_out = dt_out;
  p.cu_seqlens = cu_seqlens; p.state_indices = state_indices;
  p.slot_stride = slot_stride; p.num_slots = num_slots;
  p.nseq = nseq; p.T = tokens_per_row; p.H = heads; p.K = key_dim; p.V = value_dim;
  p.scale = scale;
  return launch_recurrent(p, (cudaStream_t)stream);
}

extern "C" int64_t kda_decode_step_scratch_bytes(int64_t address_bits, int dtype, int nseq, int heads, int width) {
  const int64_t states = (int64_t)nseq * heads;
  return nseq <= 0 || heads <= 0 || kda::decode_fuses(address_bits, dtype, states, width)
             ? 0 : states * 128 * (3 * kda::dtype_size(dtype) + 4);
}

// One decode step: one launch where the vector form of the preprocessing applies; else preprocessing and state
// update one after the other, with q, k, v (dtype) and the gate (fp32), [nseq, heads, 128] each, in scratch between them.
extern "C" int kda_decode_step(const void* x, const void* conv_weight, void* conv_state, const int32_t* state_indices,
                               const void* raw_gate, int dt_gate, const float* A_log, const float* dt_bias,
                               const void* beta, int dt_beta, float* state_pool, int64_t slot_stride, void* scratch,
                               void* out, int dtype, int nseq, int heads, int width, int conv_slots, int state_slots,
                               int activation, float lower_bound, float eps, void* stream) {
  using namespace kda;
  if (!x || !conv_weight || !conv_state || !raw_gate || !A_log || !dt_bias || !state_indices || !beta || !state_pool || !out)
    return KDA_ERR_ARG;
  if (nseq < 0 || heads < 1 || width < 1 || width > 8 || conv_slots < 1) return KDA_ERR_ARG;
  if (nseq == 0) return KDA_OK;
  if ((int64_t)nseq * heads > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  ScanParams p{};
  p.beta = beta; p.dt_q = p.dt_k = p.dt_v = p.dt_out = dtype; p.dt_g = KDA_F32; p.dt_beta = dt_beta;
  p.h0 = state_pool; p.out = out; p.state_indices = state_indices;
  p.slot_stride = slot_stride; p.num_slots = state_slots;
  p.nseq = nseq; p.T = 1; p.H = heads; p.K = p.V = 128;
  p.scale = 0.08838834764831845f;  // 128^-0.5
  PrepDecodeParams d{};
  d.x = x; d.w = conv_weight; d.conv_state = conv_state; d.raw_gate = raw_gate; d.A_log = A_log; d.dt_bias = dt_bias;
  d.state_indices = state_indices; d.dt = dtype; d.dt_gate = dt_gate; d.nseq = nseq; d.H = heads; d.W = width;
  d.num_slots = conv_slots; d.act = activation; d.lower_bound = lower_bound; d.eps = eps;
  const uintptr_t bits = (uintptr_t)x | (uintptr_t)conv_weight | (uintptr_t)conv_state | (uintptr_t)dt_bias |
                         (uintptr_t)state_pool | (uintptr_t)(4 * slot_stride);
  if (decode_fuses((int64_t)bits, dtype, (int64_t)nseq * heads, width)) return launch_fused_decode(d, p, (cudaStream_t)stream);
  if (!scratch) return KDA_ERR_SCRATCH;
  const int64_t elems = (int64_t)nseq * heads * 128;
  unsigned char* q = reinterpret_cast<unsigned char*>(scratch);
  unsigned char* k = q + elems * dtype_size(dtype);
  unsigned char* v = k + elems * dtype_size(dtype);
  float* gate = reinterpret_cast<float*>(v + elems * dtype_size(dtype));
  const int rc = kda_decode_prep(x, conv_weight, conv_state, state_indices, raw_gate, dt_gate, A_log, dt_bias, q, k, v,
                                 gate, dtype, nseq, heads, 128, width, conv_slots, activation, lower_bound, eps, stream);
  if (rc != KDA_OK) return rc;
  p.q = q; p.k = k; p.v = v; p.g = gate;
  return launch_recurrent(p, (cudaStream_t)stream);
}

// The recurrence on the cumulative gate of chunk_kda (dense or packed, no paged pool).
extern "C" int kda_chunk_scan_fwd(const void* q, const void* k, const void* v, const void* cum_gate,
                                  const void* beta, int dt_q, int dt_k, int dt_v, int dt_gate, int dt_beta,
                                  const float* initial_state, float* final_state, void* out, int dt_out,
                                  const int32_t* cu_seqlens, int nseq, int tokens_per_row, int heads,
                                  int key_dim, int value_dim, float scale, void* stream) {
  using namespace kda;
  if (!q || !k || !v || !cum_gate || !beta || !out) return KDA_ERR_ARG;
  if (nseq < 0 || heads <= 0 || key_dim <= 0 || key_dim > 256 || value_dim <= 0) return KDA_ERR_ARG;
  ScanParams p{};
  p.q = q; p.k = k; p.v = v; p.g = cum_gate; p.beta = beta;
  p.dt_q = dt_q; p.dt_k = dt_k; p.dt_v = dt_v; p.dt_g = dt_gate; p.dt_beta = dt_beta;
  p.h0 = initial_state; p.ht = final_state; p.out = out; p.dt_out = dt_out;
  p.cu_seqlens = cu_seqlens; p.nseq = nseq; p.T = tokens_per_row; p.H = heads; p.K = key_dim; p.V = value_dim;
  p.scale = scale;
  return launch_scan_any(p, true, (cudaStream_t)stream);
}

// The state-streaming kernel on one token per state, in place, with one wait that runs out: from its state `step` on, warp `warp`
// of the first CTA does not wait (0..15 arithmetic, 16 copies, 17..22 operands).
extern "C" int kda_selftest_bounded_stream(const float* q, const float* k, const float* v, const float* gate, const float* beta,
                                           float* states, float* out, int nseq, int warp, int step, void* stream) {
  using namespace kda;
  if (!q || !k || !v || !gate || !beta || !states || !out || nseq < 1 || warp < 0 || warp > 22 || step < 0) return KDA_ERR_ARG;
  ScanParams p{};
  p.q = q; p.k = k; p.v = v; p.g = gate; p.beta = beta;
  p.dt_q = p.dt_k = p.dt_v = p.dt_g = p.dt_beta = p.dt_out = KDA_F32;
  p.h0 = states; p.ht = states; p.out = out;
  p.nseq = nseq; p.T = 1; p.H = 1; p.K = p.V = 128;
  p.slot_stride = 128 * 128;
  p.scale = 0.08838834764831845f;  // 128^-0.5
  return stream_takes(p) ? launch_stream_short(p, warp, step, (cudaStream_t)stream) : KDA_ERR_UNSUPPORTED;
}
