// hx_prefill.cuh -- kernels of the batched prefill (hx_prefill.cu): a chunk of tokens goes through every linear as ONE
// tcgen05 block-scaled GEMM (hx_gemm_dig.cu).
#pragma once
#include "hx_common.cuh"

#define HX_PF_TB 64                // tokens per chunk of the batched decode (its logits take vocab floats each), of a verify window and inside a tensor-parallel group
#define HX_PF_EARLY_SEQ 12         // see hx_pf_digits
#define HX_PF_MAX 1040             // tokens per chunk of a prompt: 40 groups of 26, so that 1024 tokens are one chunk and 2048 two.  A launch's ramp
                                   // and drain (about 6 us) are a twentieth of its work there; the chunk's buffers are 269 MB at the 8B shape

// Where the tokens of a chunk sit.  Prefill: consecutive positions of one sequence starting at *posp (device memory, so
// that captured launches can be replayed).  Batched decode: token t is at position pos_arr[t] of
// sequence seq_arr[t], whose KV cache starts seq_stride floats after the previous sequence's.
// With pos_arr == null and seqp != null the whole chunk belongs to sequence *seqp (prefill into one KV slot of a batch).
struct HxPfWhere { const int* posp; const int* pos_arr; const int* seq_arr; size_t seq_stride; const int* seqp; };

// Positions are read from device memory (*posp = position of the chunk's first token), so that a captured batch step can be
// replayed; chunks of a prompt are launched one by one.
// X[t][:] = emb[ids[*posp + t]][:] (+ wpe[*posp + t][:])
int hx_pf_embed(const int* ids, HxPfWhere wh, const float* emb, const float* wpe, float* X, int n_tok, int DM, cudaStream_t st);

// Digit columns of a chunk of activation vectors, in the B-cell layout of the digit-mode GEMM.
//   src [n_tok][ld] f32, K a multiple of four;
//   g != null: RMSNorm with gain g and eps first, or with b != null LayerNorm with gain g and bias b;
//   cells: K rounded up to 256 columns; per 256-column cell and group of hx_gemm_dig_group(n_tok) tokens HX_TC_DCELL bytes: row
//   16 (t / 2) + 2 d + t % 2 = digit d of the group's token t (eight base-13 digits, most significant first, as E2M1 codes), then the column scales;
//   early: the launch may overlap the end of the kernel before (prompts, and batch steps of up to HX_PF_EARLY_SEQ sequences);
//   scale[t]: x_n = scale[t] * column scale of the block * sum_d digit_d 13^(7-d)  (powers of two).
int hx_pf_digits(const float* src, int ld, int n_tok, int K, const float* g, const float* b, float eps, uint8_t* cells, float* scale, bool early, cudaStream_t st);

// Per token and head of a chunk: RMSNorm (gains qn_g / kn_g, may be null) + rotate_half RoPE at position *posp + t on
// q (in place) and k; k and v are written to the cache rows of their positions.
int hx_pf_qkpost(float* qkv, int ld, int n_tok, HxPfWhere wh, int NH, int NKV, int DH, const float* qn_g, const float* kn_g,
                  float eps, const float* cosT, const float* sinT, float* kc, float* vc, int cap, cudaStream_t st);

// Causal attention of a chunk over the cache: query t (position *posp + t) attends to positions 0 .. *posp + t.
// CTAs per (kv head, group of tokens, run of key tiles); the query heads of a kv head share its K and V rows, and so do
// the tokens of a group in a prefill chunk.  `part` (hx_pf_attn_scratch floats) and `tickets` (n_tok * NKV words, zero
// between launches) carry the runs' partial results; *err is raised when a bounded wait ran out.
size_t hx_pf_attn_scratch(int n_tok, int NH, int NKV, int DH);
bool hx_pf_head_dim(int DH);       // head sizes of the chunk kernels
int hx_pf_attn(const float* qkv, int ld, int n_tok, HxPfWhere wh, int NH, int NKV, int DH, const float* kc, const float* vc,
               int cap, float scale, float* ctx, int ld_ctx, float* part, unsigned* tickets, int* err, cudaStream_t st);

// The same on the tensor cores (hx_pf_attn_tc.cu), head_dim 128, one sequence: `pieces` holds hx_pf_attn_tc_bytes(ctx_len, NKV)
// bytes, ctx_len = position of the chunk's last token + 1.
size_t hx_pf_attn_tc_bytes(int ctx, int NKV);
bool hx_pf_attn_tc_takes(int NH, int NKV, int DH);
bool hx_pf_attn_tc_wanted(int n_tok, int ctx, int NH, int NKV);
int hx_pf_attn_tc(const float* qkv, int ld, int n_tok, HxPfWhere wh, int NH, int NKV, const float* kc, const float* vc, int cap, float scale,
                  float* ctx, int ld_ctx, uint8_t* pieces, int ctx_len, int* err, cudaStream_t st);

// *posp += n
int hx_pf_advance(int* posp, int n, cudaStream_t st);

// First maximum of logits[0..n): index to *tok and hist[pos + 1]; *pos_out = pos + 1.
void hx_pf_argmax(const float* logits, int n, int* tok, int* hist, int* pos_out, int pos, cudaStream_t st);
// per-row arg-max of logits [rows][ld] (n valid columns) -> next[row]; pos_arr[row] += 1 when given
// Tensor parallel: x[i] += sum over the ranks of part[i] (i < count), the ranks' values exchanged as (value, epoch)
// pairs through peer_areas[w] (rank r writes slot r of every peer; slots are area_pairs pairs apart).
void hx_pf_tp_reduce(const float* part, float* x, unsigned long long* const* peer_areas, int rank, int world, int count, size_t area_pairs,
                     unsigned ep, unsigned wait_limit, int* err, cudaStream_t st);
// Tensor parallel: per row the first maximum over the ranks' vocabulary slices (this rank's slice starts at vocab_off).
void hx_pf_tp_argmax_rows(const float* logits, int n, int ld, int rows, int vocab_off, unsigned long long* const* peer_areas, int rank, int world,
                          size_t area_pairs, unsigned ep, unsigned wait_limit, int* err, int* next, int* pos_arr, cudaStream_t st);
void hx_pf_top2_rows(const float* logits, int n, int ld, int rows, int* next, float* margin, cudaStream_t st);
void hx_pf_argmax_rows(const float* logits, int n, int ld, int rows, int* next, int* pos_arr, cudaStream_t st);
