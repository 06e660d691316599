// Chunked KDA forward for K = V = 128, chunk = 64, bf16 operands, fp32 state and accumulation:
// entry points and orchestration.
//
// Two kernels replace the reference's seven forward launches
// (attn_gym/linear/kda/fwd/cute/chunk_kda_fwd.py:79-131):
//
//  prepare      per (chunk, head), tcgen05 (kda_prepare_tc.cu): the gated pairwise products, the WY
//               solve A = (I + stril(diag(beta) K~ K~^T))^-1, Aqk = scale tril(Q~ K~^T) and
//               w = A (beta k 2^G), u = A (beta v), kg = k 2^{G_last-G}, qg = scale q 2^G
//  state_fwd    per (sequence, head), serial over chunks with the fp32 state in tensor memory
//               (kda_state_tc.cu): v_new = u - w h;  o = qg h + Aqk v_new;
//               h <- diag(2^{G_last}) h + kg^T v_new
//
// The backward pass with recompute=True rebuilds w, u, kg, qg, h[c], v_new with the same two kernels
// (the tape they rewrite goes to scratch), so both modes give bit-identical results.
#include "kda_common.cuh"
#include "kda_timing.cuh"

namespace kda {

constexpr int D = 128;     // K = V
struct ChunkParams {
  const bf16* q; const bf16* k; const bf16* v; const float* g; const float* beta;
  int64_t pitch;                        // elements from one token's row of q, k, v to the next one's
  bf16* aqk; bf16* akk;                 // tape [N, H, 64]
  bf16* w; bf16* u; bf16* kg; bf16* qg;  // [N, H, 128]
  float* rstd_q; float* rstd_k; float eps;   // q / k arrive unnormalised when these are set
  const float* h0; float* ht;
  float* trans_out;                     // slice transition [nseq, H, 128, 128], or NULL
  const int32_t* limit_in; int32_t* limit_out;   // per (sequence, head) chunk limits of the state walk, or NULL
  bf16* o; bf16* h_out; bf16* vnew_out;
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;
  int nseq, H;
  float scale;
  int64_t tokens;   // rows of the token-major buffers (bounds of the TMA tensor maps)
  int chunks;       // chunk capacity: h_out holds chunks * H states (needed only with h_out)
};

int launch_prepare_tc(const bf16* q, const bf16* k, const bf16* v, int64_t pitch, const float* g, const float* beta,
                      bf16* aqk, bf16* akk, bf16* w, bf16* u, bf16* kg, bf16* qg, float* rstd_q,
                      float* rstd_k, float eps, const int32_t* cu, const int32_t* co, int nseq, int H,
                      int64_t tokens, int chunks, cudaStream_t s);
int launch_state_fwd_tc(const bf16* w, const bf16* u, const bf16* kg, const bf16* qg, const bf16* aqk,
                        const float* g, const float* h0, float* ht, float* trans_out,
                        const int32_t* limit_in, int32_t* limit_out, bf16* o, bf16* h_out,
                        bf16* vnew_out, const int32_t* cu, const int32_t* co, int nseq, int H,
                        int64_t tokens, int chunks, cudaStream_t s);

// forward: the whole chunk-parallel part (tape, w, u, kg, qg) in one tcgen05 kernel
int launch_prepare(const ChunkParams& p, int chunks, cudaStream_t s) {
  return launch_prepare_tc(p.q, p.k, p.v, p.pitch, p.g, p.beta, p.aqk, p.akk, p.w, p.u, p.kg, p.qg, p.rstd_q,
                           p.rstd_k, p.eps, p.cu_seqlens, p.chunk_offsets, p.nseq, p.H, p.tokens, chunks, s);
}
int launch_state_fwd(const ChunkParams& p, cudaStream_t s) {
  return launch_state_fwd_tc(p.w, p.u, p.kg, p.qg, p.aqk, p.g, p.h0, p.ht, p.trans_out, p.limit_in,
                             p.limit_out, p.o, p.h_out, p.vnew_out, p.cu_seqlens, p.chunk_offsets, p.nseq, p.H, p.tokens, p.chunks, s);
}

// Backward's recompute leg: w, u, kg, qg (and a scratch copy of the tape), then the chunk-entry states
// h[c] and v_new (no output, no final state).
int launch_recompute(const void* q, const void* k, const void* v, const float* g, const float* beta,
                     const void* aqk, const void* akk, const float* h0, void* w, void* u, void* kg,
                     void* qg, void* h_out, void* vnew_out, const int32_t* cu, const int32_t* co,
                     int nseq, int H, int chunks, int64_t tokens, cudaStream_t s) {
  ChunkParams p{};
  p.q = (const bf16*)q; p.k = (const bf16*)k; p.v = (const bf16*)v; p.g = g; p.beta = beta;
  p.pitch = (int64_t)H * 128;
  p.aqk = (bf16*)aqk; p.akk = (bf16*)akk;
  p.w = (bf16*)w; p.u = (bf16*)u; p.kg = (bf16*)kg; p.qg = (bf16*)qg;
  p.h0 = h0; p.ht = nullptr; p.o = nullptr;
  p.h_out = (bf16*)h_out; p.vnew_out = (bf16*)vnew_out;
  p.cu_seqlens = cu; p.chunk_offsets = co; p.nseq = nseq; p.H = H;
  p.scale = 0.08838834764831845f;
  p.tokens = tokens;
  p.chunks = chunks;
  int rc = launch_prepare(p, chunks, s);
  if (rc) return rc;
  return launch_state_fwd(p, s);
}

}  // namespace kda

using kda::bf16;

static int chunk_fwd_impl(bool keep, float* rstd_q, float* rstd_k, float eps, int64_t pitch, const void* q, const void* k,
                             const void* v, const float* cum_gate,
                             const float* beta, const float* initial_state, float* final_state,
                             void* out, void* aqk, void* akk, const int32_t* cu_seqlens,
                             const int32_t* chunk_offsets, int nseq, int64_t tokens, int heads,
                             int key_dim, int value_dim, int num_chunks, void* workspace,
                             int64_t workspace_bytes, void* stream) {
  if (!q || !k || !v || !cum_gate || !beta || !out || !aqk || !akk || !cu_seqlens ||
      !chunk_offsets || !workspace)
    return KDA_ERR_ARG;
  if (key_dim != 128 || value_dim != 128) return KDA_ERR_UNSUPPORTED;
  if (nseq < 1 || heads < 1 || tokens < 1 || num_chunks < 0) return KDA_ERR_ARG;
  if ((int64_t)nseq * heads * 8 > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  if (workspace_bytes < (keep ? kda_chunk_bwd_workspace_bytes(tokens, heads, num_chunks)
                              : kda_chunk_fwd_workspace_bytes(tokens, heads)))
    return KDA_ERR_ARG;
  if (((uintptr_t)workspace & 15) != 0) return KDA_ERR_ARG;
  kda::ChunkParams p{};
  const int64_t nd = tokens * heads * 128;
  bf16* ws = reinterpret_cast<bf16*>(workspace);
  p.q = (const bf16*)q; p.k = (const bf16*)k; p.v = (const bf16*)v; p.g = cum_gate; p.beta = beta;
  p.pitch = pitch;
  p.aqk = (bf16*)aqk; p.akk = (bf16*)akk;
  p.w = ws; p.u = ws + nd; p.kg = ws + 2 * nd; p.qg = ws + 3 * nd;
  p.rstd_q = rstd_q; p.rstd_k = rstd_k; p.eps = eps;
  p.h0 = initial_state; p.ht = final_state; p.o = (bf16*)out;
  // keep: the workspace has the backward layout (w, u, kg, qg, v_new, dv2, h, dh) and the state
  // walk also leaves v_new and the chunk-entry states there
  p.vnew_out = keep ? ws + 4 * nd : nullptr;
  p.h_out = keep ? ws + 6 * nd : nullptr;
  p.chunks = num_chunks;
  p.cu_seqlens = cu_seqlens; p.chunk_offsets = chunk_offsets; p.nseq = nseq; p.H = heads;
  p.scale = 0.08838834764831845f;  // 128^-0.5
  p.tokens = tokens;
  cudaStream_t s = (cudaStream_t)stream;
  int rc = kda::launch_prepare(p, num_chunks, s);
  if (rc) return rc;
  return kda::launch_state_fwd(p, s);
}

extern "C" int kda_chunk_fwd(const void* q, const void* k, const void* v, const float* cum_gate,
                             const float* beta, const float* initial_state, float* final_state,
                             void* out, void* aqk, void* akk, const int32_t* cu_seqlens,
                             const int32_t* chunk_offsets, int nseq, int64_t tokens, int heads,
                             int key_dim, int value_dim, int num_chunks, void* workspace,
                             int64_t workspace_bytes, void* stream) {
  return chunk_fwd_impl(false, nullptr, nullptr, 0.f, (int64_t)heads * 128, q, k, v, cum_gate, beta, initial_state, final_state,
                        out, aqk, akk, cu_seqlens, chunk_offsets, nseq, tokens, heads, key_dim, value_dim,
                        num_chunks, workspace, workspace_bytes, stream);
}

// kda_chunk_fwd / kda_chunk_fwd_save (keep != 0) for unnormalised q and k: every q and k row is scaled
// to unit L2 norm, x * rsqrt(sum x^2 + eps), inside the first kernel, and the reciprocal norms go to
// rstd_q / rstd_k (fp32 [tokens, heads]) for kda_chunk_bwd_qknorm_saved.
extern "C" int kda_chunk_fwd_qknorm(const void* q, const void* k, const void* v, const float* cum_gate,
                                    const float* beta, const float* initial_state, float* final_state,
                                    void* out, void* aqk, void* akk, float* rstd_q, float* rstd_k,
                                    float eps, const int32_t* cu_seqlens, const int32_t* chunk_offsets,
                                    int nseq, int64_t tokens, int heads, int key_dim, int value_dim,
                                    int num_chunks, void* workspace, int64_t workspace_bytes, int keep,
                                    void* stream) {
  if (!rstd_q || !rstd_k || !(eps >= 0.f)) return KDA_ERR_ARG;
  return chunk_fwd_impl(keep != 0, rstd_q, rstd_k, eps, (int64_t)heads * 128, q, k, v, cum_gate, beta, initial_state,
                        final_state, out, aqk, akk, cu_seqlens, chunk_offsets, nseq, tokens, heads,
                        key_dim, value_dim, num_chunks, workspace, workspace_bytes, stream);
}

extern "C" int kda_chunk_fwd_save(const void* q, const void* k, const void* v, const float* cum_gate,
                                  const float* beta, const float* initial_state, float* final_state,
                                  void* out, void* aqk, void* akk, const int32_t* cu_seqlens,
                                  const int32_t* chunk_offsets, int nseq, int64_t tokens, int heads,
                                  int key_dim, int value_dim, int num_chunks, void* saved,
                                  int64_t saved_bytes, void* stream) {
  return chunk_fwd_impl(true, nullptr, nullptr, 0.f, (int64_t)heads * 128, q, k, v, cum_gate, beta, initial_state, final_state,
                        out, aqk, akk, cu_seqlens, chunk_offsets, nseq, tokens, heads, key_dim, value_dim,
                        num_chunks, saved, saved_bytes, stream);
}

extern "C" int64_t kda_chunk_fwd_workspace_bytes(int64_t tokens, int heads) {
  return 4 * tokens * heads * 128 * (int64_t)sizeof(bf16);
}

// The two halves of kda_chunk_fwd as separate entry points: `prepare` is the chunk-parallel part
// (pairwise products, solve, w/u/kg/qg into the workspace), `state` the serial recurrence that
// consumes the workspace.  Context parallelism runs `prepare` once per slice and `state` several
// times (zero entering state, identity state for the slice transition, true entering state).
extern "C" int kda_chunk_fwd_prepare(const void* q, const void* k, const void* v,
                                     const float* cum_gate, const float* beta, void* aqk, void* akk,
                                     const int32_t* cu_seqlens, const int32_t* chunk_offsets,
                                     int nseq, int64_t tokens, int heads, int num_chunks,
                                     void* workspace, int64_t workspace_bytes, void* stream) {
  if (!q || !k || !v || !cum_gate || !beta || !aqk || !akk || !cu_seqlens || !chunk_offsets ||
      !workspace)
    return KDA_ERR_ARG;
  if (nseq < 1 || heads < 1 || tokens < 1 || num_chunks < 0) return KDA_ERR_ARG;
  if (workspace_bytes < kda_chunk_fwd_workspace_bytes(tokens, heads)) return KDA_ERR_ARG;
  kda::ChunkParams p{};
  const int64_t nd = tokens * heads * 128;
  bf16* ws = reinterpret_cast<bf16*>(workspace);
  p.q = (const bf16*)q; p.k = (const bf16*)k; p.v = (const bf16*)v; p.g = cum_gate; p.beta = beta;
  p.pitch = (int64_t)heads * 128;
  p.aqk = (bf16*)aqk; p.akk = (bf16*)akk;
  p.w = ws; p.u = ws + nd; p.kg = ws + 2 * nd; p.qg = ws + 3 * nd;
  p.cu_seqlens = cu_seqlens; p.chunk_offsets = chunk_offsets; p.nseq = nseq; p.H = heads;
  p.scale = 0.08838834764831845f;
  p.tokens = tokens;
  cudaStream_t s = (cudaStream_t)stream;
  return kda::launch_prepare(p, num_chunks, s);
}

// use_u == 0 runs the homogeneous recurrence (u = 0): with identity matrices as initial_state the
// final state is the slice transition M = prod_t (I - beta_t k_t k_t^T) diag(2^{g_t}), so that the
// state leaving the slice is M h_in + b.  out may be NULL.
extern "C" int kda_chunk_fwd_state(const float* cum_gate, const float* initial_state,
                                   float* final_state, void* out, const void* aqk,
                                   const int32_t* cu_seqlens, const int32_t* chunk_offsets, int nseq,
                                   int64_t tokens, int heads, void* workspace, int use_u,
                                   const int32_t* chunk_limit, void* stream) {
  if (!cum_gate || !aqk || !cu_seqlens || !chunk_offsets || !workspace) return KDA_ERR_ARG;
  if (nseq < 1 || heads < 1 || tokens < 1) return KDA_ERR_ARG;
  if ((int64_t)nseq * heads * 8 > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  kda::ChunkParams p{};
  const int64_t nd = tokens * heads * 128;
  bf16* ws = reinterpret_cast<bf16*>(workspace);
  p.g = cum_gate;
  p.aqk = (bf16*)aqk;
  p.w = ws; p.u = use_u ? ws + nd : nullptr; p.kg = ws + 2 * nd; p.qg = ws + 3 * nd;
  p.h0 = initial_state; p.ht = final_state; p.o = (bf16*)out;
  p.limit_in = chunk_limit;
  p.cu_seqlens = cu_seqlens; p.chunk_offsets = chunk_offsets; p.nseq = nseq; p.H = heads;
  p.tokens = tokens;
  return kda::launch_state_fwd(p, (cudaStream_t)stream);
}

// One launch for what a context-parallel rank needs before the boundary-state chain can pass through
// it: b = the state leaving the slice for a zero entering state, and M = the dense slice transition,
// so that the leaving state for any entering state is M h_in + b.  Half of the CTAs walk the chains
// with u from a zero state, the other half with u = 0 from an identity state.
extern "C" int kda_chunk_slice_map(const float* cum_gate, float* b_out, float* transition_out,
                                   void* out, int32_t* chunk_limit_out, const void* aqk,
                                   const int32_t* cu_seqlens,
                                   const int32_t* chunk_offsets, int nseq, int64_t tokens, int heads,
                                   void* workspace, void* stream) {
  if (!cum_gate || !b_out || !transition_out || !aqk || !cu_seqlens || !chunk_offsets || !workspace)
    return KDA_ERR_ARG;
  if (nseq < 1 || heads < 1 || tokens < 1) return KDA_ERR_ARG;
  if ((int64_t)nseq * heads * 8 > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  kda::ChunkParams p{};
  const int64_t nd = tokens * heads * 128;
  bf16* ws = reinterpret_cast<bf16*>(workspace);
  p.g = cum_gate;
  p.aqk = (bf16*)aqk;
  p.w = ws; p.u = ws + nd; p.kg = ws + 2 * nd; p.qg = ws + 3 * nd;
  p.ht = b_out; p.trans_out = transition_out;
  p.o = (bf16*)out; p.limit_out = chunk_limit_out;
  p.cu_seqlens = cu_seqlens; p.chunk_offsets = chunk_offsets; p.nseq = nseq; p.H = heads;
  p.tokens = tokens;
  return kda::launch_state_fwd(p, (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------------------
// Dense batches: `batch` rows of `tokens_per_row` tokens each.
//
// The offsets are built on the device from the two sizes.  When the batch has fewer (row, head)
// chains than half the SMs and the rows are long, every row is cut into segments of whole chunks
// that are walked in parallel, exactly as the ranks of a context-parallel chain would:
//   pass A  every segment from a zero state (outputs, b = its leaving state), and on further CTAs the
//           segment transition M together with the number of chunks after which it is exactly zero;
//   chain   h_in(s + 1) = M_s h_in(s) + b_s along each row (fp32, tiny);
//   pass B  every segment again with its true entering state, over the leading chunks that state
//           can still reach (all of them when the gates never forget completely).
// With gates that forget within a few chunks the serial walk shrinks by the number of segments;
// with gates that never forget it costs about what the unsegmented walk costs.  The results agree
// with the unsegmented walk to fp32 resolution of the state, not bit for bit.
// ------------------------------------------------------------------------------------------------
namespace kda {

int launch_state_chain(const float* M, const float* b, const float* h0, float* hin, float* fin, int rows, int heads, int segs,
                       cudaStream_t s);

static int g_row_segments = 0;   // 0 = choose; otherwise the forced number of segments per row (tests, tuning)

struct DensePlan {
  int segs;         // segments per row (1 = plain walk)
  int seg_chunks;   // chunks per segment (the last one of a row may be shorter)
  int row_chunks;
  int64_t count;    // batch * segs
};

static DensePlan plan_dense(int batch, int64_t tokens_per_row, int heads) {
  DensePlan pl;
  pl.row_chunks = (int)((tokens_per_row + kChunk - 1) / kChunk);
  int segs = 1;
  if (g_row_segments > 0) {
    segs = g_row_segments;
  } else {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t chains = (int64_t)batch * heads;
    if (chains * 2 <= sms) segs = (int)(sms / chains < 8 ? sms / chains : 8);
    if (segs > pl.row_chunks / 64) segs = pl.row_chunks / 64;     // at least 64 chunks per segment
  }
  if (segs > pl.row_chunks) segs = pl.row_chunks;
  if (segs < 1) segs = 1;
  pl.seg_chunks = (pl.row_chunks + segs - 1) / segs;
  pl.segs = (pl.row_chunks + pl.seg_chunks - 1) / pl.seg_chunks;
  pl.count = (int64_t)batch * pl.segs;
  return pl;
}

// sequence i = (row i / segs, segment i % segs)
__global__ void dense_offsets_kernel(int32_t* cu, int32_t* co, int count, int segs, int tokens_per_row,
                                     int row_chunks, int seg_chunks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > count) return;
  const int row = i / segs, s = i % segs;
  const int chunks = min(s * seg_chunks, row_chunks);
  cu[i] = row * tokens_per_row + min(chunks * kChunk, tokens_per_row);
  co[i] = row * row_chunks + chunks;
}

static int64_t align256(int64_t x) { return (x + 255) & ~(int64_t)255; }

struct DenseScratch {   // byte offsets from the start of the workspace
  int64_t cu, co, limit, b, trans, hin, end;      // end: the bytes the workspace needs
};
// What the dense forward keeps beside w, u, kg, qg: the offsets, and for rows in segments three fp32 states per
// (segment, head).  A forward that keeps its intermediates puts it where the backward pass will write dh[c], which
// the forward leaves alone, so the kept buffer does not grow: 32 KiB per (chunk, head) there against 192 KiB per
// segment of at least 64 chunks.  Otherwise (no kept buffer, or segments forced to be shorter) it is appended.
static DenseScratch dense_scratch(bool keep, int batch, int64_t tokens_per_row, int heads, const DensePlan& pl) {
  DenseScratch d{};
  const int64_t total = (int64_t)batch * tokens_per_row, chunks = (int64_t)batch * pl.row_chunks;
  const int64_t base = keep ? kda_chunk_bwd_workspace_bytes(total, heads, chunks)
                            : kda_chunk_fwd_workspace_bytes(total, heads);
  int64_t at = 0;
  d.cu = at; at = align256(at + (pl.count + 1) * 4);
  d.co = at; at = align256(at + (pl.count + 1) * 4);
  if (pl.segs > 1) {
    const int64_t states = pl.count * heads * (int64_t)D * D * 4;
    d.limit = at; at = align256(at + pl.count * heads * 4);
    d.b = at; at += states;
    d.trans = at; at += states;
    d.hin = at; at += states;
  }
  const int64_t hs = chunks * heads * (int64_t)D * D * 2;      // bytes of h[c], and of dh[c] behind it
  const bool inside = keep && at <= hs;
  const int64_t start = inside ? 6 * total * heads * (int64_t)D * 2 + hs : align256(base);
  for (int64_t* x : {&d.cu, &d.co, &d.limit, &d.b, &d.trans, &d.hin}) *x += start;
  d.end = inside ? base : start + at;
  return d;
}

}  // namespace kda

extern "C" int kda_set_row_segments(int segments) {
  if (segments < 0 || segments > 64) return KDA_ERR_ARG;
  kda::g_row_segments = segments;
  return KDA_OK;
}

extern "C" int64_t kda_chunk_fwd_dense_workspace_bytes(int batch, int64_t tokens_per_row, int heads,
                                                       int keep) {
  if (batch < 1 || tokens_per_row < 1 || heads < 1) return 0;
  return kda::dense_scratch(keep != 0, batch, tokens_per_row, heads, kda::plan_dense(batch, tokens_per_row, heads)).end;
}

static int chunk_fwd_dense_impl(bool keep, float* rstd_q, float* rstd_k, float eps, int64_t pitch, const void* q,
                                const void* k, const void* v, const float* cum_gate, const float* beta, const float* initial_state,
                                float* final_state, void* out, void* aqk, void* akk, int batch,
                                int64_t tokens_per_row, int heads, int key_dim, int value_dim,
                                void* workspace, int64_t workspace_bytes, void* stream) {
  if (!q || !k || !v || !cum_gate || !beta || !out || !aqk || !akk || !workspace) return KDA_ERR_ARG;
  if (key_dim != 128 || value_dim != 128) return KDA_ERR_UNSUPPORTED;
  if (batch < 1 || heads < 1 || tokens_per_row < 1) return KDA_ERR_ARG;
  const int64_t total = (int64_t)batch * tokens_per_row;
  if (total > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  const kda::DensePlan pl = kda::plan_dense(batch, tokens_per_row, heads);
  if (pl.count * heads * 8 > 0x7fffffffLL) return KDA_ERR_UNSUPPORTED;
  const int chunks = batch * pl.row_chunks;
  const kda::DenseScratch sc = kda::dense_scratch(keep, batch, tokens_per_row, heads, pl);
  if (workspace_bytes < sc.end || ((uintptr_t)workspace & 15) != 0) return KDA_ERR_ARG;
  unsigned char* scratch = reinterpret_cast<unsigned char*>(workspace);
  int32_t* cu = reinterpret_cast<int32_t*>(scratch + sc.cu);
  int32_t* co = reinterpret_cast<int32_t*>(scratch + sc.co);
  cudaStream_t s = (cudaStream_t)stream;
  const int count = (int)pl.count;
  kda::dense_offsets_kernel<<<(count + 256) / 256, 256, 0, s>>>(cu, co, count, pl.segs, (int)tokens_per_row,
                                                              pl.row_chunks, pl.seg_chunks);
  if (cudaGetLastError() != cudaSuccess) return KDA_ERR_LAUNCH;

  kda::ChunkParams p{};
  const int64_t nd = total * heads * 128;
  bf16* ws = reinterpret_cast<bf16*>(workspace);
  p.q = (const bf16*)q; p.k = (const bf16*)k; p.v = (const bf16*)v; p.g = cum_gate; p.beta = beta;
  p.pitch = pitch;
  p.aqk = (bf16*)aqk; p.akk = (bf16*)akk;
  p.w = ws; p.u = ws + nd; p.kg = ws + 2 * nd; p.qg = ws + 3 * nd;
  p.rstd_q = rstd_q; p.rstd_k = rstd_k; p.eps = eps;
  p.o = (bf16*)out;
  p.vnew_out = keep ? ws + 4 * nd : nullptr;
  p.h_out = keep ? ws + 6 * nd : nullptr;
  p.chunks = chunks;
  p.cu_seqlens = cu; p.chunk_offsets = co; p.nseq = count; p.H = heads;
  p.scale = 0.08838834764831845f;
  p.tokens = total;
  int rc = kda::launch_prepare(p, chunks, s);
  if (rc) return rc;
  if (pl.segs == 1) {
    p.h0 = initial_state; p.ht = final_state;
    return kda::launch_state_fwd(p, s);
  }
  // ---- pass A: zero-state walk of every segment + transitions with their measured reach
  float* b = reinterpret_cast<float*>(scratch + sc.b);
  float* trans = reinterpret_cast<float*>(scratch + sc.trans);
  float* hin = reinterpret_cast<float*>(scratch + sc.hin);
  int32_t* limit = reinterpret_cast<int32_t*>(scratch + sc.limit);
  if (cudaMemsetAsync(limit, 0, (size_t)count * heads * 4, s) != cudaSuccess) return KDA_ERR_LAUNCH;
  p.h0 = nullptr; p.ht = b; p.trans_out = trans; p.limit_out = limit;
  rc = kda::launch_state_fwd(p, s);
  if (rc) return rc;
  // ---- chain along each row: h_in(0) = the row's initial state, h_in(s + 1) = M_s h_in(s) + b_s
  rc = kda::launch_state_chain(trans, b, initial_state, hin, final_state, batch, heads, pl.segs, s);
  if (rc) return rc;
  // ---- pass B: the leading chunks of every segment with its true entering state
  p.h0 = hin; p.ht = nullptr; p.trans_out = nullptr; p.limit_out = nullptr; p.limit_in = limit;
  return kda::launch_state_fwd(p, s);
}

extern "C" int kda_chunk_fwd_dense(const void* q, const void* k, const void* v, const float* cum_gate,
                                   const float* beta, const float* initial_state, float* final_state,
                                   void* out, void* aqk, void* akk, int batch, int64_t tokens_per_row,
                                   int heads, int key_dim, int value_dim, void* workspace,
                                   int64_t workspace_bytes, void* stream) {
  return chunk_fwd_dense_impl(false, nullptr, nullptr, 0.f, (int64_t)heads * 128, q, k, v, cum_gate, beta, initial_state, final_state, out, aqk, akk,
                              batch, tokens_per_row, heads, key_dim, value_dim, workspace,
                              workspace_bytes, stream);
}

extern "C" int kda_chunk_fwd_dense_save(const void* q, const void* k, const void* v,
                                        const float* cum_gate, const float* beta,
                                        const float* initial_state, float* final_state, void* out,
                                        void* aqk, void* akk, int batch, int64_t tokens_per_row,
                                        int heads, int key_dim, int value_dim, void* saved,
                                        int64_t saved_bytes, void* stream) {
  return chunk_fwd_dense_impl(true, nullptr, nullptr, 0.f, (int64_t)heads * 128, q, k, v, cum_gate, beta, initial_state, final_state, out, aqk, akk,
                              batch, tokens_per_row, heads, key_dim, value_dim, saved, saved_bytes,
                              stream);
}

// The dense forward for unnormalised q and k (see kda_chunk_fwd_qknorm).  The walk of B = 1, T = 131072, H = 32: 3.35 ms as
// one packed sequence (2048 serial steps a chain), 1.23 ms in segments; T = 16384, H = 8: 479 and 142 us.
extern "C" int kda_chunk_fwd_dense_qknorm(const void* q, const void* k, const void* v, const float* cum_gate,
                                          const float* beta, const float* initial_state, float* final_state,
                                          void* out, void* aqk, void* akk, float* rstd_q, float* rstd_k, float eps,
                                          int batch, int64_t tokens_per_row, int heads, int key_dim, int value_dim,
                                          void* workspace, int64_t workspace_bytes, int keep, void* stream) {
  if (!rstd_q || !rstd_k || !(eps >= 0.f)) return KDA_ERR_ARG;
  return chunk_fwd_dense_impl(keep != 0, rstd_q, rstd_k, eps, (int64_t)heads * 128, q, k, v, cum_gate, beta, initial_state, final_state,
                              out, aqk, akk, batch, tokens_per_row, heads, key_dim, value_dim, workspace,
                              workspace_bytes, stream);
}

// ------------------------------------------------------------------------------------------------
// Rows of packed results that no sequence writes stay zero: the unused tail of a fixed-capacity buffer, which only the
// device knows.  Every block checks the offsets (a few KB that hit L2) and clears its share of the rows before the first and
// behind the last sequence; offsets that the chunk kernels would skip, because they leave the buffer or contradict one
// another, clear all rows.  (Filling the results first: 13.8 GB, 2.9 ms of a training step of 279046 tokens, H = 32.)
// ------------------------------------------------------------------------------------------------
namespace kda {
constexpr int kZeroBuffers = 8;
struct ZeroRowsParams {
  void* buffer[kZeroBuffers];
  int64_t row_bytes[kZeroBuffers];       // even
  int count, nseq, chunk;
  const int32_t* cu_seqlens; const int32_t* chunk_offsets;      // chunk_offsets may be null: not checked
  int64_t tokens;
};
__global__ void __launch_bounds__(256) zero_rows_kernel(const ZeroRowsParams p) {
  bool bad = p.nseq < 1;
  for (int i = threadIdx.x; i < p.nseq; i += 256) {
    const int64_t bos = p.cu_seqlens[i], eos = p.cu_seqlens[i + 1];
    bad |= bos < 0 || eos < bos || eos > p.tokens;
    if (p.chunk_offsets)
      bad |= p.chunk_offsets[i + 1] - (int64_t)p.chunk_offsets[i] != (eos - bos + p.chunk - 1) / p.chunk;
  }
  if (threadIdx.x == 0 && p.nseq > 0 && p.chunk_offsets) bad |= p.chunk_offsets[0] != 0;
  bad = __syncthreads_or(bad);
  const int64_t head = bad ? p.tokens : (int64_t)p.cu_seqlens[0], tail = bad ? p.tokens : (int64_t)p.cu_seqlens[p.nseq];
  const int64_t stride = (int64_t)gridDim.x * 256, me = (int64_t)blockIdx.x * 256 + threadIdx.x;
  for (int b = 0; b < p.count; ++b) {
    const uintptr_t base = reinterpret_cast<uintptr_t>(p.buffer[b]);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      // whole 16-byte words by all blocks, what is left at either end two bytes at a time by the first block
      const uintptr_t lo = base + (part ? tail : 0) * p.row_bytes[b], hi = base + (part ? p.tokens : head) * p.row_bytes[b];
      const uintptr_t first = min((lo + 15) & ~(uintptr_t)15, hi), last = max(hi & ~(uintptr_t)15, first);
      for (int64_t i = me; i < (int64_t)((last - first) / 16); i += stride)
        reinterpret_cast<uint4*>(first)[i] = make_uint4(0, 0, 0, 0);
      if (me < 16) {
        const uintptr_t at = me < 8 ? lo + me * 2 : last + (me - 8) * 2;
        if (at < (me < 8 ? first : hi)) *reinterpret_cast<uint16_t*>(at) = 0;
      }
    }
  }
}
}  // namespace kda

extern "C" int kda_zero_unused_rows(void* const* buffers, const int64_t* row_bytes, int count, const int32_t* cu_seqlens,
                                    const int32_t* chunk_offsets, int chunk_size, int nseq, int64_t tokens, void* stream) {
  if (!buffers || !row_bytes || (!cu_seqlens && nseq > 0) || chunk_size < 1 || count < 1 || tokens < 0) return KDA_ERR_ARG;
  if (count > kda::kZeroBuffers) return KDA_ERR_UNSUPPORTED;
  kda::ZeroRowsParams p{};
  for (int i = 0; i < count; ++i) {
    if (row_bytes[i] < 0 || row_bytes[i] % 2 || ((uintptr_t)buffers[i] & 1) != 0) return KDA_ERR_ARG;
    if (!buffers[i] && tokens * row_bytes[i] > 0) return KDA_ERR_ARG;
    p.buffer[i] = buffers[i];
    p.row_bytes[i] = row_bytes[i];
  }
  p.count = count; p.nseq = nseq; p.chunk = chunk_size; p.cu_seqlens = cu_seqlens; p.chunk_offsets = chunk_offsets; p.tokens = tokens;
  if (tokens == 0) return KDA_OK;
  kda::zero_rows_kernel<<<2 * kda::device_sms(), 256, 0, (cudaStream_t)stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}

// kda_chunk_fwd_qknorm (cu_seqlens given) or kda_chunk_fwd_dense_qknorm (cu_seqlens NULL: nseq rows of tokens / nseq
// tokens) on rows of [q | k | v], 3 * heads * 128 elements a token, as a projection or a convolution leaves them.
extern "C" int kda_chunk_fwd_qkv(const void* qkv, const float* cum_gate, const float* beta, const float* initial_state,
                                 float* final_state, void* out, void* aqk, void* akk, float* rstd_q, float* rstd_k,
                                 float eps, const int32_t* cu_seqlens, const int32_t* chunk_offsets, int nseq,
                                 int64_t tokens, int heads, int num_chunks, void* workspace, int64_t workspace_bytes,
                                 int keep, void* stream) {
  if (!qkv || !rstd_q || !rstd_k || !(eps >= 0.f) || nseq < 1 || heads < 1 || tokens < 1) return KDA_ERR_ARG;
  const int64_t width = (int64_t)heads * 128;
  const bf16 *q = (const bf16*)qkv, *k = q + width, *v = k + width;
  if (cu_seqlens)
    return chunk_fwd_impl(keep != 0, rstd_q, rstd_k, eps, 3 * width, q, k, v, cum_gate, beta, initial_state, final_state,
                          out, aqk, akk, cu_seqlens, chunk_offsets, nseq, tokens, heads, 128, 128, num_chunks, workspace,
                          workspace_bytes, stream);
  if (tokens % nseq) return KDA_ERR_ARG;
  return chunk_fwd_dense_impl(keep != 0, rstd_q, rstd_k, eps, 3 * width, q, k, v, cum_gate, beta, initial_state,
                              final_state, out, aqk, akk, nseq, tokens / nseq, heads, 128, 128, workspace,
                              workspace_bytes, stream);
}

// ------------------------------------------------------------------------------------------------
// Chunked forward for callers that must not allocate.
//
// Some hosts of this library cannot call cudaMalloc: a serving engine that has handed every free
// byte of the device to its own paged pool, or a plugin running under a runtime that forbids
// allocation once the model is loaded.  For them the w/u/kg/qg scratch of the forward lives in the
// file-scope device array below instead of a caller workspace.  CUDA loads device code lazily, so
// a GPU starts to hold the array (KDA_NOALLOC_SCRATCH_BYTES, until the process exits) when the first
// call on it looks the array's address up, not when the library is opened: that first call belongs
// in the host's start-up phase, before its own pool claims the rest of the device.
// ------------------------------------------------------------------------------------------------
namespace kda {
static __device__ __align__(256) unsigned char g_noalloc_scratch[KDA_NOALLOC_SCRATCH_BYTES];
static void* g_noalloc_ptr[64] = {nullptr};
}  // namespace kda

extern "C" int kda_chunk_fwd_noalloc(const void* q, const void* k, const void* v,
                                     const float* cum_gate, const float* beta,
                                     const float* initial_state, float* final_state, void* out,
                                     void* aqk, void* akk, const int32_t* cu_seqlens,
                                     const int32_t* chunk_offsets, int nseq, int64_t tokens,
                                     int heads, int key_dim, int value_dim, int num_chunks,
                                     void* stream) {
  if (tokens < 1 || heads < 1) return KDA_ERR_ARG;
  const int64_t need = kda_chunk_fwd_workspace_bytes(tokens, heads);
  if (need > (int64_t)KDA_NOALLOC_SCRATCH_BYTES) return KDA_ERR_SCRATCH;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return KDA_ERR_LAUNCH;
  // In host code the array's name is only a handle; the device address comes from the runtime,
  // once per device, with that device current.
  void* scratch = kda::g_noalloc_ptr[dev];
  if (!scratch) {
    if (cudaGetSymbolAddress(&scratch, kda::g_noalloc_scratch) != cudaSuccess || !scratch) {
      cudaGetLastError();   // leave no stale error behind for the next entry point's launch check
      return KDA_ERR_LAUNCH;
    }
    kda::g_noalloc_ptr[dev] = scratch;
  }
  // Nothing in the scratch has to start at zero: every row a kernel reads was written earlier in
  // the same call, rows past a sequence tail are masked on load.
  return kda_chunk_fwd(q, k, v, cum_gate, beta, initial_state, final_state, out, aqk, akk,
                       cu_seqlens, chunk_offsets, nseq, tokens, heads, key_dim, value_dim,
                       num_chunks, scratch, need, stream);
}

extern "C" int kda_dense_offsets(void* offsets, int batch, int tokens, void* stream) {
  if (!offsets || batch < 1 || tokens < 1) return KDA_ERR_ARG;
  int32_t* cu = reinterpret_cast<int32_t*>(offsets);
  const int row_chunks = (int)(((int64_t)tokens + kda::kChunk - 1) / kda::kChunk);
  kda::dense_offsets_kernel<<<(batch + 256) / 256, 256, 0, (cudaStream_t)stream>>>(cu, cu + batch + 1, batch, 1, tokens,
                                                                                 row_chunks, row_chunks);
  return cudaGetLastError() == cudaSuccess ? KDA_OK : KDA_ERR_LAUNCH;
}
