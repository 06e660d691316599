// Chunk-parallel half of the forward pass on tcgen05 tensor cores: per (chunk, head), one persistent
// kernel computes the gated pairwise products, the WY solve and the WY products
//
//   Aqk = scale tril(Q~ K~^T),  L = stril(diag(beta) K~ K~^T),  A = (I + L)^-1,
//   w = A (beta k 2^G),  u = A (beta v),  kg = k 2^{G_last - G},  qg = scale q 2^G
//
// (reference stages: fwd/triton/chunk_kda_fwd_intra_sub_chunk_forloop.py:66,
//  fwd/cute/chunk_kda_k3b_offdiag_cutedsl.py:177, fwd/cute/chunk_kda_k4b_inverse_cutedsl.py:188,
//  fwd/triton/recompute_w_u.py:257).
//
//   phase 0  TMA: G, q, k (requested while the previous item still runs, as their regions die).
//   phase 1  every (row, 8 channels) piece once: Qr = q 2^{G - R_b}, Kr = k 2^{G - R_b} (R_b = gate of
//            the first row of the 16-row block b of the row), the column operands
//            Kn_r = k 2^{R_r - G} for r >= b, the WY operand beta k 2^G (in place), and the results
//            kg, qg (straight from registers to memory).  Four exponentials per element; 2^{R_r - R_b}
//            comes from a small per-(block pair, channel) table.  (2^G as 2^{G - R_b} 2^{R_b} with the
//            second factor from a table rounds qg and beta k 2^G once more and saves nothing: 0.622 ms.)
//   phase 2  UMMA, M = 64 (the Qr, Kr rows of a pair of row blocks), N = 16 (r + 1) columns of Kn_r
//   phase 3  epilogue: masked, scaled Aqk tile (bf16); L in fp32; A = (I + L)^-1 by 16 x 16 blocks on
//            the CUDA cores in fp32; A as a bf16 operand tile and to memory (the tape)
//   phase 4  UMMA M = 64, N = 128:  w = A (beta k 2^G),  u = A (beta v);  epilogue; TMA stores.
//
// Two CTAs of 256 threads per SM, 113 KiB of shared memory and 256 tensor-memory columns each.  An item
// is a chain of short phases (load, gating, products, solve, products, store) that leaves every unit of
// the SM idle most of the time, so a second chain beside it is worth more than wider phases.  That it fits
// comes from the lifetimes: the gates move to registers and their tile becomes the Qr / Kr operand, v is
// fetched into the q tile when q is spent, and the solve, its operand tile and the result staging share
// the column-operand tiles.
// B = 8, T = 4096, H = 32: 0.602 ms = 4.5 TB/s of its 2564 B per unit, against 0.848 ms with one CTA of 512
// threads per SM and 230 KiB; one sequence of 1000 tokens, H = 32: 34 against 43 us.  (Two CTAs of 512
// threads with 64 registers: 0.75 ms, 30 % more instructions and more waiting at barriers.)  Issue slots and the
// shared-memory port are each half busy; the rest is the latency of the chain at four warps per scheduler.
//
// Gate rebasing and its range contract are those of the reference (fwd/triton/gate_fwd.py:619-631):
// exponents are clamped at 126, so masked entries cannot produce NaN.
// All barrier waits are bounded (error word + early exit instead of a hang).
#include "kda_common.cuh"
#include "kda_sm100.cuh"
#include "kda_timing.cuh"

namespace kda {
namespace {

using namespace sm100;

struct PrepParams {
  CUtensorMap tm_q, tm_k, tm_v, tm_g;                       // inputs
  CUtensorMap tm_w, tm_u;                                   // results staged in shared memory
  const float* beta;
  bf16* qg; bf16* kg; bf16* w; bf16* u; bf16* aqk; bf16* akk;
  float* rstd_q; float* rstd_k;    // NORM kernels: 1 / sqrt(sum x^2 + eps) of every q and k row, [tokens, H]
  float eps;
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;
  int* error;
  int nseq, H, total;          // total = chunk capacity x heads work items
  int64_t tokens;              // rows of the packed buffers
  float scale;
  long long* prof;             // debugging aid: phase timestamps of the 20th item of the first 64 CTAs
};

__device__ __forceinline__ void pr_mark(const PrepParams& p, int it, int slot) {
#ifdef KDA_PHASE_PROFILE
#ifndef KDA_PROFILE_THREAD
#define KDA_PROFILE_THREAD 0
#endif
  if (p.prof && it == 20 && threadIdx.x == KDA_PROFILE_THREAD && blockIdx.x < 64) {
    long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    p.prof[blockIdx.x * 32 + slot] = t;
  }
#endif
}

namespace pl {  // shared-memory layout (bytes); tiles that the tensor cores or TMA touch start on 1024-byte boundaries
constexpr int G = 0, QKR = G;              // [64 x 128] fp32 gates; once in registers, the Qr / Kr rows
constexpr int Q = 32768, V = Q;            // q, then v
constexpr int K = 49152;                   // k, then beta k 2^G in place
constexpr int KN = 65536;                  // column operands Kn_0 .. Kn_3; once multiplied:
constexpr int AQK = KN;                    //   Aqk tile
constexpr int LF = KN + 8192;              //   L blocks (fp32)
constexpr int XT = LF + 12800;             //   columns of A by block column, inner index contiguous (fp32)
constexpr int AT = KN + 32768;             //   A as a bf16 operand tile
constexpr int W = KN, U = KN + 16384;      //   after the last product: staging of w, u
constexpr int TAB = KN + 40960;            // per-channel tables of phase 1; then the diagonal blocks of A (fp32)
constexpr int AD = TAB;
constexpr int BETA = TAB + 5632, MISC = BETA + 512, OFFS = MISC + 128;      // beta: one copy per item parity
constexpr int kOffCache = 368;             // cu_seqlens / chunk_offsets entries kept in shared memory
constexpr int TOTAL = OFFS + 2 * 4 * kOffCache;
constexpr int BP = 20, BLK = 16 * BP;      // pitch and size of a 16 x 16 fp32 block (floats)
constexpr int TT = XT + 4 * 16 * (52 + 36 + 20);        //   columns of the right-hand sides, 48 x 20 floats
static_assert(TT + 4 * 48 * 20 <= AT && 4 * 4 * BLK <= BETA - AD && TOTAL <= 115712, "two CTAs per SM");
}  // namespace pl
namespace pt {  // tensor-memory columns
constexpr int kCols = 256;
constexpr int AQ = 0;                      // row block r: 16 (r + 1) columns from AQ + 8 r (r + 1); dead before w, u
constexpr int W = 0, U = 128;
}

constexpr int NT = 256;

__device__ __forceinline__ void ld_g8(const unsigned char* g, int row, int kappa0, float (&o)[8]) {
  // The eight lanes of a quarter-warp hold kappa0 = 0, 8, .., 56 (+64): two 32-float boxes, the same
  // four even chunks in each.  Lanes of the odd box fetch their second chunk first, so each 16-byte
  // load touches eight different chunks (no bank conflict).
  const unsigned char* base = g + (kappa0 >> 5) * 8192 + row * 128;
  const int c = (kappa0 & 31) >> 2, sw = row & 7, odd = (kappa0 >> 5) & 1;
  const float4 a = *reinterpret_cast<const float4*>(base + (((c + odd) ^ sw) << 4));
  const float4 b = *reinterpret_cast<const float4*>(base + (((c + 1 - odd) ^ sw) << 4));
  const float4 lo = odd ? b : a, hi = odd ? a : b;
  o[0] = lo.x; o[1] = lo.y; o[2] = lo.z; o[3] = lo.w; o[4] = hi.x; o[5] = hi.y; o[6] = hi.z; o[7] = hi.w;
}
__device__ __forceinline__ uint4 ld_raw8(const unsigned char* tile, int box_bytes, int row, int c16) {
  return *reinterpret_cast<const uint4*>(tile + (c16 >> 3) * box_bytes + sw128_chunk(row, c16 & 7));
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&o)[8]) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y; o[4] = c.x; o[5] = c.y; o[6] = d.x; o[7] = d.y;
}
__device__ __forceinline__ void pack8v(const float* x, uint4& o) {
  o.x = pack_bf16(x[0], x[1]); o.y = pack_bf16(x[2], x[3]);
  o.z = pack_bf16(x[4], x[5]); o.w = pack_bf16(x[6], x[7]);
}
// byte offset of Kn_r inside the KN region: the tiles have 16, 32, 48, 64 rows of 256 bytes
__device__ __forceinline__ int kn_off(int r) { return 4096 * (r * (r + 1) / 2); }
// position of block (r, c), c <= r, among the 16 x 16 blocks of a lower triangular matrix
__device__ __forceinline__ int blk_off(int r, int c) { return (r * (r + 1) / 2 + c) * pl::BLK; }
// the eight gates of one (row, 8 channels) piece as four pairs
__device__ __forceinline__ void ld_g8x2(const unsigned char* g, int row, int kappa0, f32x2 (&o)[4]) {
  float x[8];
  ld_g8(g, row, kappa0, x);
#pragma unroll
  for (int e = 0; e < 4; ++e) o[e] = pack2(x[2 * e], x[2 * e + 1]);
}
// a row of a per-channel table: the first four channels of every piece, then the other four
__device__ __forceinline__ void ld_tab8(const float* row, int c16, f32x2 (&o)[4]) {
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row + 4 * c16);
  const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(row + 64 + 4 * c16);
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
__device__ __forceinline__ uint32_t pack_pair(f32x2 x) {
  const float2 f = unpack2(x);
  return pack_bf16(f.x, f.y);
}
__device__ __forceinline__ f32x2 unpack_pair(uint32_t u) {
  const float2 f = unpack_bf16(u);
  return pack2(f.x, f.y);
}

// columns of block column c of A: floats from one to the next, and the byte offset of the first
__host__ __device__ constexpr int xt_pitch(int c) { return 52 - 16 * c; }
__host__ __device__ constexpr int xt_off(int c) { return pl::XT + 64 * (c > 0 ? 52 : 0) + 64 * (c > 1 ? 36 : 0); }

// Inner index k of a row or column of the solve lies at position 2 (k mod 8) + k / 8: a 16-byte vector holds two pairs
// (k, k + 8) for the packed arithmetic, which then sums the two halves of the inner index side by side.
__host__ __device__ constexpr int inner_pos(int k) { return 2 * (k & 7) + (k >> 3); }

// NC columns per lane of block column C of A = (I + L)^-1, from its diagonal block down: lane (i = lid / 2, lid & 1) holds
// row i of every block and NC adjacent columns; `part` is the warp's share of the block's columns.
template <int C, int NC>
__device__ __forceinline__ void solve_columns(unsigned char* sm, int part, int lid) {
  const float* Lf = reinterpret_cast<const float*>(sm + pl::LF);
  const float* Ad = reinterpret_cast<const float*>(sm + pl::AD);
  const int i = lid >> 1, pos = inner_pos(i), col0 = 2 * NC * part + NC * (lid & 1);
  float* x = reinterpret_cast<float*>(sm + xt_off(C)) + col0 * xt_pitch(C);     // [column][row - 16 C]
  float* t = reinterpret_cast<float*>(sm + pl::TT) + (16 * C + col0) * 20;      // [column][row of the block]
  auto dot = [&](const float* row, const float* cols, int pitch, f32x2 (&d)[NC]) {     // row . column, 16 inner indices, in halves
    ulonglong2 a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = *reinterpret_cast<const ulonglong2*>(row + 4 * k);
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      f32x2 s = 0;             // (zero bits: +0, +0)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(cols + j * pitch + 4 * k);
        s = fma2(a[k].x, b.x, s);
        s = fma2(a[k].y, b.y, s);
      }
      d[j] = s;
    }
  };
  f32x2 acc[4][NC];            // right-hand sides of the block rows below (only r > C are used)
#pragma unroll
  for (int m = C; m < 3; ++m) {            // X_m is known: its share of every right-hand side, then X_{m + 1}
    const float* xm = x + 16 * (m - C);
    f32x2 d[NC];
#pragma unroll
    for (int r = m + 1; r < 4; ++r) {
      dot(Lf + blk_off(r, m) + i * pl::BP, xm, xt_pitch(C), d);
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[r][j] = m == C ? d[j] : add2(acc[r][j], d[j]);
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const float2 h = unpack2(acc[m + 1][j]);
      t[j * 20 + pos] = h.x + h.y;
    }
    __syncwarp();
    float out[NC];
    dot(Ad + (m + 1) * pl::BLK + i * pl::BP, t, 20, d);
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const float2 h = unpack2(d[j]);
      out[j] = -(h.x + h.y);
      if (m + 1 < 3) x[j * xt_pitch(C) + 16 * (m + 1 - C) + pos] = out[j];
    }
#pragma unroll
    for (int j = 0; j < NC; j += 2) {
      const int c = col0 + j;
      *reinterpret_cast<uint32_t*>(sm + pl::AT + sw128_chunk(16 * (m + 1) + i, 2 * C + (c >> 3)) + 2 * (c & 7)) =
          pack_bf16(out[j], out[j + 1]);
    }
    __syncwarp();              // the column's next 16 rows are complete; the right-hand side has been read
  }
}

// NORM: q and k arrive unnormalised; every row is scaled to unit L2 norm (and rounded to bf16, as a
// separate l2norm launch would leave it) while its pieces pass through the registers of phase 1,
// and the two reciprocal norms are kept for the backward pass
// (reference stages: fwd/triton/l2norm_fwd.py:22, applied right before the core in
// examples/kda_training.py:412-421).
// The thread index, read anew: what a phase derives from it (lane, tile addresses) is then recomputed per
// item instead of being kept, or spilled, across the whole persistent loop.
__device__ __forceinline__ int fresh_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

template <bool NORM>
__global__ void __launch_bounds__(NT, 2) kda_prepare_tc_kernel(const __grid_constant__ PrepParams p) {
  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + pl::MISC);     // TMA: [0] G, [1] q and k, [2] v; UMMA: [3] pairwise, [4] w / u
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + pl::MISC + 64);
  volatile int* s_abort = reinterpret_cast<volatile int*>(sm + pl::MISC + 72);
  int* s_next = reinterpret_cast<int*>(sm + pl::MISC + 96);                // next item: token0 (two words), valid
  float* Lf = reinterpret_cast<float*>(sm + pl::LF);
  float* Ad = reinterpret_cast<float*>(sm + pl::AD);
  // rows: 0..3 R_b, 4..9 2^{R_r - R_b} for (r, b) = (1,0) (2,0) (3,0) (2,1) (3,1) (3,2), 10 G_last
  float* tab = reinterpret_cast<float*>(sm + pl::TAB);
  const unsigned char* sG = sm + pl::G;

  const int tid = threadIdx.x, warp = tid >> 5, lid = tid & 31;
  const int quad = warp & 3;                       // TMEM lane quadrant
  const int H = p.H;
  if ((saddr(sm) & 1023u) != 0) {                  // the tiles' swizzle needs an aligned base
    if (tid == 0 && p.error) atomicExch(p.error, 31);
    return;
  }

  // Work items are located by a binary search over the sequence offsets: from shared memory when
  // they fit (a chain of dependent global loads per item would sit on the critical path).
  int32_t* s_cu = reinterpret_cast<int32_t*>(sm + pl::OFFS);
  int32_t* s_co = s_cu + pl::kOffCache;
  const bool cached = p.nseq + 1 <= pl::kOffCache;
  if (cached)
    for (int i = tid; i <= p.nseq; i += NT) { s_cu[i] = p.cu_seqlens[i]; s_co[i] = p.chunk_offsets[i]; }
  const int32_t* cu_off = cached ? s_cu : p.cu_seqlens;
  const int32_t* ch_off = cached ? s_co : p.chunk_offsets;
  if (warp == 0) tmem_alloc(tmem_slot, pt::kCols);
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&bar[2], 1);
    mbar_init(&bar[3], 4);       // one arrival per issuing thread
    mbar_init(&bar[4], 2);
    mbar_init_fence();
    *s_abort = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tl = tmem + ((uint32_t)(32 * quad) << 16);

  auto load_gates = [&](int head, int64_t token0) {
    mbar_expect_tx(&bar[0], 32768);
    for (int b = 0; b < 4; ++b) tma_load_2d(sm + pl::G + b * 8192, &p.tm_g, head * 128 + 32 * b, (int)token0, &bar[0]);
  };
  auto load_qk = [&](int head, int64_t token0) {       // lanes 0..3 of a warp, one box each
    if (lid == 0) mbar_expect_tx(&bar[1], 32768);
    __syncwarp();
    const int b = lid >> 1, tx = head * 128 + 64 * b;
    if (lid < 4) {
      if (lid & 1) tma_load_2d(sm + pl::K + b * 8192, &p.tm_k, tx, (int)token0, &bar[1]);
      else tma_load_2d(sm + pl::Q + b * 8192, &p.tm_q, tx, (int)token0, &bar[1]);
    }
  };

  const f32x2 neg1 = pack2(-1.f, -1.f), scale2 = pack2(p.scale, p.scale);
  uint32_t ph = 0;
  int rc = 0, it = 0;
  bool pre = false;              // this item's loads were issued by the previous item
  ChunkWork cw_next{};
  int head_n = 0;
  for (int wi = blockIdx.x; wi < p.total; wi += gridDim.x) {
  const int head = pre ? head_n : wi % H;
  const ChunkWork cw = pre ? cw_next : locate_chunk(cu_off, ch_off, p.nseq, wi / H);
  if (cw.valid == 0) continue;               // capacity slot past the last active chunk
  if (!pre && !chunk_in_range(cw, p.tokens)) {     // (with pre the previous item checked it)
    if (tid == 0 && p.error) atomicExch(p.error, kOffsetsOutOfRange);
    continue;
  }
  const int valid = cw.valid;
  const int ty = (int)cw.token0, tx = head * 128;
  // No CTA barrier here: the tables were last read before barriers of the previous item, and beta (its copy
  // of the item before that) comes before the barrier that ends the table step.
  float* s_beta = reinterpret_cast<float*>(sm + pl::BETA) + 64 * (it & 1);
  if (!pre && tid < 64) s_beta[tid] = tid < valid ? p.beta[(cw.token0 + tid) * H + head] : 0.f;
  if (warp == 0 && !pre) {
    if (lid == 0) load_gates(head, cw.token0);
    load_qk(head, cw.token0);
  }
  // the next item is located by one thread while this item's tiles arrive (the search is a chain of
  // dependent loads); everybody reads the result after the barrier that ends the table step
  bool next_ok = false;
  if (tid == 160) {
    const int wn = wi + (int)gridDim.x;
    ChunkWork nx{};
    if (wn < p.total) nx = locate_chunk(cu_off, ch_off, p.nseq, wn / H);
    if (!chunk_in_range(nx, p.tokens)) {     // not prefetched; the item itself reports and skips
      nx.valid = 0;
    }
    s_next[0] = (int)(nx.token0 & 0xffffffffLL);
    s_next[1] = (int)(nx.token0 >> 32);
    s_next[2] = nx.valid;
    s_next[3] = wn % H;
  }
  auto body = [&]() -> int {
  const int tid = fresh_tid();
  pr_mark(p, it, 0);
  if (!mbar_wait(&bar[0], ph)) *s_abort = 1;
  pr_mark(p, it, 1);

  // ---- tables, and the gates into registers.  Rows >= valid of a partial tail chunk hold another
  //      sequence's tokens or unwritten memory: they read as q = k = 0 with the gate of the last row, so
  //      no later step needs a row guard.
  const int il = tid >> 4, c16 = tid & 15;         // row of each 16-row block, channel piece
  f32x2 g[4][4];
#pragma unroll
  for (int n = 0; n < 4; ++n) ld_g8x2(sG, min(16 * n + il, valid - 1), 8 * c16, g[n]);
  {
    const int ch = tid & 127, pos = ((ch >> 2) & 1) * 64 + (ch >> 3) * 4 + (ch & 3);
    auto gate = [&](int row) {
      row = min(row, valid - 1);
      return *reinterpret_cast<const float*>(sG + (ch >> 5) * 8192 + row * 128 +
                                             (((((ch & 31) >> 2) ^ (row & 7)) << 4) | ((ch & 3) << 2)));
    };
    float* t = tab + pos;
    const float r0 = gate(0), r1 = gate(16), r2 = gate(32), r3 = gate(48);
    if (tid < 128) {
      t[0] = r0; t[128] = r1; t[256] = r2; t[384] = r3;
      t[128 * 4] = fexp2(r1 - r0);
      t[128 * 10] = gate(63);
    } else {
      t[128 * 5] = fexp2(r2 - r0); t[128 * 6] = fexp2(r3 - r0);
      t[128 * 7] = fexp2(r2 - r1); t[128 * 8] = fexp2(r3 - r1); t[128 * 9] = fexp2(r3 - r2);
    }
  }
  if (tid == 192) tma_store_wait_read();     // the w, u staging tiles (over Kn) of the previous item have been read
  __syncthreads();
  pr_mark(p, it, 2);
  if (*s_abort) return 2;
  {   // the next item; its beta values travel straight to shared memory
    head_n = s_next[3];
    cw_next.token0 = (int64_t)(((uint64_t)(uint32_t)s_next[1] << 32) | (uint32_t)s_next[0]);
    cw_next.valid = s_next[2];
    next_ok = cw_next.valid > 0;        // 0 also when there is no further item
    if (tid < 64 && next_ok) {
      const bool in = tid < cw_next.valid;
      cp_async_4(reinterpret_cast<float*>(sm + pl::BETA) + 64 * ((it + 1) & 1) + tid,
                 p.beta + (in ? (cw_next.token0 + tid) * H + head_n : 0), in);
    }
  }
  pr_mark(p, it, 12);
  if (!mbar_wait(&bar[1], ph)) *s_abort = 1;
  pr_mark(p, it, 13);

  // ---- phase 1: one (row, 8 channels) piece of every row block per thread ---------------------------------
  {
    f32x2 gl[4];
    ld_tab8(tab + 128 * 10, c16, gl);
    const int64_t out0 = ((cw.token0 + il) * H + head) * 128 + 8 * c16;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = 16 * n + il;
      const bool in = i < valid;
      uint4 qw = ld_raw8(sm + pl::Q, 8192, i, c16), kw = ld_raw8(sm + pl::K, 8192, i, c16);
      if (!in) qw = kw = make_uint4(0, 0, 0, 0);
      if constexpr (NORM) {
        // the 16 lanes of a half-warp hold one row: sum of squares in the order of the stand-alone kernel (eight fused
        // multiply-adds per lane, then a butterfly over the lanes); after its first step lanes 0..7 go on with q, 8..15 with k
        // (five shuffles instead of eight; 40000 tokens, 32 heads: 10 us of 850)
        float qq[8], kk[8], sq = 0.f, sk = 0.f;
        unpack8(qw, qq);
        unpack8(kw, kk);
#pragma unroll
        for (int e = 0; e < 8; ++e) { sq = fmaf(qq[e], qq[e], sq); sk = fmaf(kk[e], kk[e], sk); }
        const bool upper = (c16 & 8) != 0;
        float ss = (upper ? sk : sq) + __shfl_xor_sync(0xffffffffu, upper ? sq : sk, 8);
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
        const float r = rsqrtf(ss + p.eps), other = __shfl_xor_sync(0xffffffffu, r, 8);
        if ((c16 & 7) == 0 && in) (upper ? p.rstd_k : p.rstd_q)[(cw.token0 + i) * H + head] = r;
        const float rq = upper ? other : r, rk = upper ? r : other;
        const f32x2 rq2 = pack2(rq, rq), rk2 = pack2(rk, rk);
        uint32_t* const qd[4] = {&qw.x, &qw.y, &qw.z, &qw.w}, * const kd[4] = {&kw.x, &kw.y, &kw.z, &kw.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {    // the bf16 rows are what every later step works with
          *qd[e] = pack_pair(mul2(pack2(qq[2 * e], qq[2 * e + 1]), rq2));
          *kd[e] = pack_pair(mul2(pack2(kk[2 * e], kk[2 * e + 1]), rk2));
        }
      }
      const uint32_t qu[4] = {qw.x, qw.y, qw.z, qw.w}, ku[4] = {kw.x, kw.y, kw.z, kw.w};
      f32x2 R[4], kk[4], ei[4];
      uint32_t qr[4], kr[4], qg[4], kt[4], kg[4], kn[4];
      const f32x2 bt2 = pack2(s_beta[i], s_beta[i]);
      ld_tab8(tab + 128 * n, c16, R);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack2(g[n][e]), d = unpack2(fma2(R[e], neg1, g[n][e])), l = unpack2(fma2(g[n][e], neg1, gl[e]));
        const f32x2 eg = pack2(fexp2(f.x), fexp2(f.y)), qq = unpack_pair(qu[e]);      // 2^{G_i}
        const f32x2 er = pack2(fexp2(d.x), fexp2(d.y));                               // 2^{G_i - R_b} <= 1
        ei[e] = pack2(fexp2(fminf(-d.x, 126.f)), fexp2(fminf(-d.y, 126.f)));          // 2^{R_b - G_i}
        kk[e] = unpack_pair(ku[e]);
        qr[e] = pack_pair(mul2(qq, er));
        kr[e] = pack_pair(mul2(kk[e], er));
        qg[e] = pack_pair(mul2(mul2(qq, eg), scale2));                                // scale q 2^G
        kt[e] = pack_pair(mul2(mul2(kk[e], eg), bt2));                                // beta k 2^G
        kg[e] = pack_pair(mul2(kk[e], pack2(fexp2(l.x), fexp2(l.y))));                // k 2^{G_last - G}
        kn[e] = pack_pair(mul2(kk[e], ei[e]));
      }
      const int so = (c16 >> 3) * 8192 + sw128_chunk(i, c16 & 7);
      *reinterpret_cast<uint4*>(sm + pl::K + so) = make_uint4(kt[0], kt[1], kt[2], kt[3]);
      // one row-operand tile for both sides: rows 32 b .. 32 b + 15 hold Qr of block b, the next 16 Kr
      const int ro = (c16 >> 3) * 16384 + sw128_chunk(32 * n + il, c16 & 7);
      *reinterpret_cast<uint4*>(sm + pl::QKR + ro) = make_uint4(qr[0], qr[1], qr[2], qr[3]);
      *reinterpret_cast<uint4*>(sm + pl::QKR + ro + 2048) = make_uint4(kr[0], kr[1], kr[2], kr[3]);
      if (in) {
        const int64_t o = out0 + (int64_t)(16 * n) * H * 128;
        *reinterpret_cast<uint4*>(p.qg + o) = make_uint4(qg[0], qg[1], qg[2], qg[3]);
        *reinterpret_cast<uint4*>(p.kg + o) = make_uint4(kg[0], kg[1], kg[2], kg[3]);
      }
      // column operands Kn_r[i] = k_i 2^{R_r - G_i} for the row blocks r >= b
#pragma unroll
      for (int rr = n; rr < 4; ++rr) {
        if (rr > n) {
          f32x2 T[4];                                                                 // 2^{R_r - R_b} <= 1
          ld_tab8(tab + 128 * (n == 0 ? 3 + rr : (n == 1 ? 5 + rr : 9)), c16, T);
#pragma unroll
          for (int e = 0; e < 4; ++e) kn[e] = pack_pair(mul2(kk[e], mul2(ei[e], T[e])));
        }
        *reinterpret_cast<uint4*>(sm + pl::KN + kn_off(rr) + (c16 >> 3) * (16 * (rr + 1) * 128) +
                                  sw128_chunk(i, c16 & 7)) = make_uint4(kn[0], kn[1], kn[2], kn[3]);
      }
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  pr_mark(p, it, 3);

  {
    const int tid = fresh_tid(), warp = tid >> 5, lid = tid & 31;
    // ---- phase 2: pairwise products, one issuing thread per row block (lane 0 of warps 0..3) ---------
    //   D_r[m][j] = sum_kappa QKR[m][kappa] Kn_r[j][kappa] over the 64 operand rows m of the row blocks
    //   (0, 1) or (2, 3); only the 32 rows of block r are read back
    if (lid == 0 && warp < 4) {
      tc_fence_after();
      const int r = warp;
      const uint32_t kn = saddr(sm + pl::KN + kn_off(r)), box = 16 * (r + 1) * 128;
      const uint32_t rows = saddr(sm + pl::QKR) + 8192 * (r >> 1);
      const uint32_t acc = tmem + pt::AQ + 8 * r * (r + 1);
      const uint32_t id = instr_desc(64, 16 * (r + 1), 0, 0);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) umma(acc, desc_kmajor(rows, ks, 16384), desc_kmajor(kn, ks, box), id, ks > 0);
      umma_commit(&bar[3]);
    }
    if (lid == 0 && warp == 4) {         // q is spent: v takes its place
      mbar_expect_tx(&bar[2], 16384);
      for (int b = 0; b < 2; ++b) tma_load_2d(sm + pl::V + b * 8192, &p.tm_v, tx + 64 * b, ty, &bar[2]);
    }
    __syncwarp();
    if (!mbar_wait(&bar[3], ph)) *s_abort = 1;
    tc_fence_after();
    pr_mark(p, it, 4);
    if (tid == 160 && next_ok) load_gates(head_n, cw_next.token0);     // over the Qr / Kr tile

  }
  {
    const int tid = fresh_tid(), warp = tid >> 5, lid = tid & 31, quad = warp & 3, wq = warp >> 2;
    // ---- phase 3a: lanes 0..15 of quadrants 0, 2 hold Aqk rows of the even and odd row blocks, those of
    //      quadrants 1, 3 the rows of P (M = 64 layout); one 16-column group at a time
    {
      const int odd = quad >> 1;
      for (int e = wq * (odd ? 3 : 2), end = e + (odd ? 3 : 2); e < end; ++e) {
        const int r = odd ? (e < 2 ? 1 : 3) : (e < 1 ? 0 : 2);
        const int c = odd ? (e < 2 ? e : e - 2) : (e < 1 ? 0 : e - 1);
        float a[16];
        tmem_ld16(tl + pt::AQ + 8 * r * (r + 1) + 16 * c, a);
        if (lid < 16) {
          const int i = 16 * r + lid, below = 16 * (r - c) + lid;      // column 16 c + jj is in row i's past if jj < below
          if (quad & 1) {
            const float bt = s_beta[i];
            float4* dst = reinterpret_cast<float4*>(Lf + blk_off(r, c) + lid * pl::BP);
            if (r == c) {
#pragma unroll
              for (int j = 0; j < 16; j += 4)
                dst[j >> 2] = make_float4(j < lid ? a[j] * bt : 0.f, j + 1 < lid ? a[j + 1] * bt : 0.f,
                                          j + 2 < lid ? a[j + 2] * bt : 0.f, j + 3 < lid ? a[j + 3] * bt : 0.f);
            } else {               // (every column is in the row's past) the inner order of the solve
#pragma unroll
              for (int j = 0; j < 8; j += 2) dst[j >> 1] = make_float4(a[j] * bt, a[j + 8] * bt, a[j + 1] * bt, a[j + 9] * bt);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = (j <= below && i < valid) ? a[j] * p.scale : 0.f;
            uint4 v;
            pack8v(a, v);
            *reinterpret_cast<uint4*>(sm + pl::AQK + sw128_chunk(i, 2 * c)) = v;
            pack8v(a + 8, v);
            *reinterpret_cast<uint4*>(sm + pl::AQK + sw128_chunk(i, 2 * c + 1)) = v;
          }
        }
      }
    }
  }
  __syncthreads();
  pr_mark(p, it, 5);
  if (*s_abort) return 3;

  // ---- phase 3b: A = (I + L)^-1 by 16 x 16 blocks, fp32 ---------------------------------------------------
  {
    const int tid = fresh_tid();
    if (tid < 64) {  // diagonal blocks: column c of block b by forward substitution
      const int b = tid >> 4, c = tid & 15;
      const float* L = Lf + blk_off(b, b);
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = (i == c) ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        float4 l[16];
#pragma unroll
        for (int i = j + 1; i < 16; ++i) l[i] = *reinterpret_cast<const float4*>(L + i * pl::BP + j);
#pragma unroll
        for (int i = j + 1; i < 16; ++i) x[i] = fmaf(-l[i].x, x[j], x[i]);
#pragma unroll
        for (int i = j + 2; i < 16; ++i) x[i] = fmaf(-l[i].y, x[j + 1], x[i]);
#pragma unroll
        for (int i = j + 3; i < 16; ++i) x[i] = fmaf(-l[i].z, x[j + 2], x[i]);
#pragma unroll
        for (int i = j + 4; i < 16; ++i) x[i] = fmaf(-l[i].w, x[j + 3], x[i]);
      }
      float* dst = Ad + b * pl::BLK + inner_pos(c);
#pragma unroll
      for (int i = 0; i < 16; ++i) dst[i * pl::BP] = x[i];
      if (b < 3) {
        float4* col = reinterpret_cast<float4*>(reinterpret_cast<float*>(sm + xt_off(b)) + c * xt_pitch(b));
#pragma unroll
        for (int i = 0; i < 4; ++i) col[i] = make_float4(x[2 * i], x[2 * i + 8], x[2 * i + 1], x[2 * i + 9]);
      }
    } else {         // meanwhile the Aqk tile leaves and v becomes beta v
      for (int idx = tid - 64; idx < valid * 8; idx += NT - 64) {
        const int r = idx >> 3, c = idx & 7;
        uint4 v = make_uint4(0, 0, 0, 0);
        if ((c >> 1) <= (r >> 4)) v = *reinterpret_cast<const uint4*>(sm + pl::AQK + sw128_chunk(r, c));
        *reinterpret_cast<uint4*>(p.aqk + ((cw.token0 + r) * H + head) * 64 + c * 8) = v;
      }
      if (!mbar_wait(&bar[2], ph)) *s_abort = 1;
      for (int idx = tid - 64; idx < 64 * 16; idx += NT - 64) {
        const int r = idx >> 4, c = idx & 15;
        uint4* cell = reinterpret_cast<uint4*>(sm + pl::V + (c >> 3) * 8192 + sw128_chunk(r, c & 7));
        uint4 v = make_uint4(0, 0, 0, 0);       // rows past the end of the sequence may hold NaN
        if (r < valid) {
          v = *cell;
          const f32x2 bt = pack2(s_beta[r], s_beta[r]);
          v.x = pack_pair(mul2(unpack_pair(v.x), bt)); v.y = pack_pair(mul2(unpack_pair(v.y), bt));
          v.z = pack_pair(mul2(unpack_pair(v.z), bt)); v.w = pack_pair(mul2(unpack_pair(v.w), bt));
        }
        *cell = v;
      }
    }
  }
  __syncthreads();
  pr_mark(p, it, 6);
  {
    const int tid = fresh_tid(), warp = tid >> 5, lid = tid & 31;
    // The blocks below the diagonal, column block by column block and without a CTA barrier: a warp takes its columns
    // of block column c through the block rows r > c,  T_r = sum_{c <= m < r} L[r][m] X_m,  X_r = -A[r][r] T_r.
    // Block column 0 is shared by four warps, 1 by two, 2 belongs to one: 9, 5 and 2 products of 16 x 16 by 4, 8 and 16
    // columns are about the same work.  Columns lie in shared memory with their inner index contiguous, as the rows of
    // L and A do, so both operands arrive as 16-byte vectors of pairs for the packed arithmetic.  The pairs are (k, k + 8):
    // measured against 64 bits (gates x 1, .02, .001 and nearly equal keys), the two halves side by side and the products
    // L[r][m] X_m added block by block have 0.77 to 0.99 of the rounding error of the products by distance; with pairs
    // (k, k + 1) it was up to 2.4 times that error, because between nearly equal keys neighbouring terms cancel.
    // (All six A[r][r] L[r][m] first and then the blocks by their distance from the diagonal: four more CTA
    // barriers; 0.622 ms for the whole kernel.)
    if (warp < 4) solve_columns<0, 2>(sm, warp, lid);
    else if (warp < 6) solve_columns<1, 4>(sm, warp - 4, lid);
    else if (warp == 6) solve_columns<2, 8>(sm, 0, lid);
    else {        // meanwhile the diagonal blocks, and zeros to their right, go into the operand tile: two rows per lane
      for (int r = lid; r < 64; r += 32) {
        const int b = r >> 4;
        const float4* src = reinterpret_cast<const float4*>(Ad + b * pl::BLK + (r & 15) * pl::BP);
        const float4 f0 = src[0], f1 = src[1], f2 = src[2], f3 = src[3];        // pairs (k, k + 8)
        *reinterpret_cast<uint4*>(sm + pl::AT + sw128_chunk(r, 2 * b)) =
            make_uint4(pack_bf16(f0.x, f0.z), pack_bf16(f1.x, f1.z), pack_bf16(f2.x, f2.z), pack_bf16(f3.x, f3.z));
        *reinterpret_cast<uint4*>(sm + pl::AT + sw128_chunk(r, 2 * b + 1)) =
            make_uint4(pack_bf16(f0.y, f0.w), pack_bf16(f1.y, f1.w), pack_bf16(f2.y, f2.w), pack_bf16(f3.y, f3.w));
        for (int c = 2 * b + 2; c < 8; ++c) *reinterpret_cast<uint4*>(sm + pl::AT + sw128_chunk(r, c)) = make_uint4(0, 0, 0, 0);
      }
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();

  pr_mark(p, it, 8);
  {
    const int tid = fresh_tid(), warp = tid >> 5, lid = tid & 31;
    // ---- phase 4: w = A (beta k 2^G) (thread 0), u = A (beta v) (thread 32) ------------------------------------
    if (lid == 0 && warp < 2) {
      tc_fence_after();
      const uint32_t at = saddr(sm + pl::AT);
      const uint32_t bop = saddr(sm + (warp == 0 ? pl::K : pl::V));
      const uint32_t id = instr_desc(64, 128, 0, 1);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        umma(tmem + (warp == 0 ? pt::W : pt::U), desc_kmajor(at, ks, 0), desc_mnmajor(bop, ks, 8192), id, ks > 0);
      umma_commit(&bar[4]);
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 2; ++n) {      // meanwhile A leaves
      const int idx = tid + n * NT, r = idx >> 3, c = idx & 7;
      const uint4 v = *reinterpret_cast<const uint4*>(sm + pl::AT + sw128_chunk(r, c));
      if (r < valid) *reinterpret_cast<uint4*>(p.akk + ((cw.token0 + r) * H + head) * 64 + c * 8) = v;
    }
    if (!mbar_wait(&bar[4], ph)) *s_abort = 1;
    tc_fence_after();
    pr_mark(p, it, 9);
    if (warp == 7 && next_ok) load_qk(head_n, cw_next.token0);         // the k and v tiles are dead

  }
  {
    const int tid = fresh_tid(), warp = tid >> 5, lid = tid & 31, quad = warp & 3, wq = warp >> 2;
    // ---- epilogue: rows i = 16 quad + lane (lanes 0..15), channels 64 wq .. 64 wq + 63 of w and u ----------
    {
      const int i = 16 * quad + lid;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float a[32];
        tmem_ld32(tl + (h < 2 ? pt::W : pt::U) + 64 * wq + 32 * (h & 1), a);
        if (lid < 16) {
#pragma unroll
          for (int qd = 0; qd < 4; ++qd) {
            uint4 v;
            pack8v(a + 8 * qd, v);
            *reinterpret_cast<uint4*>(sm + (h < 2 ? pl::W : pl::U) + wq * 8192 + sw128_chunk(i, 4 * (h & 1) + qd)) = v;
          }
        }
      }
    }
  }
  fence_async_smem();
  tc_fence_before();
  cp_async_wait_all();       // the next item's beta
  __syncthreads();
  pr_mark(p, it, 10);
  if (*s_abort) return 4;
  {
    const int tid = fresh_tid();
    if (valid == 64) {
      if (tid == 192) {
        for (int b = 0; b < 2; ++b) {
          tma_store_2d(&p.tm_w, sm + pl::W + b * 8192, tx + 64 * b, ty);
          tma_store_2d(&p.tm_u, sm + pl::U + b * 8192, tx + 64 * b, ty);
        }
        tma_store_commit();
      }
    } else {                 // partial chunk: rows < valid only, plain 16-byte stores
      for (int idx = tid; idx < valid * 16; idx += NT) {
        const int r = idx >> 4, ch = idx & 15;
        const int64_t gi = ((cw.token0 + r) * H + head) * 128 + ch * 8;
        const int so = (ch >> 3) * 8192 + sw128_chunk(r, ch & 7);
        *reinterpret_cast<uint4*>(p.w + gi) = *reinterpret_cast<const uint4*>(sm + pl::W + so);
        *reinterpret_cast<uint4*>(p.u + gi) = *reinterpret_cast<const uint4*>(sm + pl::U + so);
      }
    }
  }
  pr_mark(p, it, 11);
  return 0;
  };
  rc = body();
  if (rc) break;
  pre = next_ok;
  ph ^= 1;
  ++it;
  }  // work items
  if (tid == 192) tma_store_wait_read();    // staged tiles must outlive the bulk stores' reads
  if (rc && tid == 0 && p.error) atomicExch(p.error, 32 + rc);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_slot[0], pt::kCols);
}

static __device__ int g_prepare_error = 0;

}  // namespace

long long* debug_profile_buffer();

// pitch: elements from one token's row of q, k, v to the next one's
int launch_prepare_tc(const bf16* q, const bf16* k, const bf16* v, int64_t pitch, const float* g, const float* beta,
                      bf16* aqk, bf16* akk, bf16* w, bf16* u, bf16* kg, bf16* qg, float* rstd_q,
                      float* rstd_k, float eps, const int32_t* cu, const int32_t* co, int nseq, int H,
                      int64_t tokens, int chunks, cudaStream_t s) {
  if (chunks == 0) return KDA_OK;
  PrepParams p;
  const int64_t cols = (int64_t)H * 128;
  bool ok = make_tensor_map(&p.tm_q, q, tokens, cols, 64, false, pitch) &&
            make_tensor_map(&p.tm_k, k, tokens, cols, 64, false, pitch) &&
            make_tensor_map(&p.tm_v, v, tokens, cols, 64, false, pitch) && make_tensor_map(&p.tm_g, g, tokens, cols, 64, true) &&
            make_tensor_map(&p.tm_w, w, tokens, cols, 64) && make_tensor_map(&p.tm_u, u, tokens, cols, 64);
  // the other results are written with plain 16-byte stores
  if (!ok || (((uintptr_t)qg | (uintptr_t)kg | (uintptr_t)aqk | (uintptr_t)akk) & 15) != 0) return KDA_ERR_LAUNCH;
  p.beta = beta; p.qg = qg; p.kg = kg; p.w = w; p.u = u; p.aqk = aqk; p.akk = akk;
  p.rstd_q = rstd_q; p.rstd_k = rstd_k; p.eps = eps;
  if ((rstd_q == nullptr) != (rstd_k == nullptr)) return KDA_ERR_ARG;
  p.cu_seqlens = cu; p.chunk_offsets = co; p.nseq = nseq; p.H = H;
  p.total = chunks * H;
  p.tokens = tokens;
  p.scale = 0.08838834764831845f;  // 128^-0.5
  p.prof = debug_profile_buffer();
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1 ||
      cudaGetSymbolAddress(reinterpret_cast<void**>(&p.error), g_prepare_error) != cudaSuccess)
    return KDA_ERR_LAUNCH;
  const int smem = pl::TOTAL;
  auto kernel = rstd_q ? kda_prepare_tc_kernel<true> : kda_prepare_tc_kernel<false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared) != cudaSuccess)
    return KDA_ERR_LAUNCH;
  StageScope timing(kStagePrepare, s);
  kernel<<<(unsigned)(p.total < 2 * sms ? p.total : 2 * sms), NT, smem, s>>>(p);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

int prepare_tc_error_word() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_prepare_error, sizeof(int)) != cudaSuccess) return -1;
  cudaMemcpyToSymbol(g_prepare_error, &zero, sizeof(int));
  return v;
}

}  // namespace kda
