// Argument block of the attention entry points (shared by the translation units that launch them).
#pragma once
#include "common.cuh"

struct AttnArgs {
    const bf16* q;            // [Tq, Hq, Dh]
    const bf16* k_cache;
    const bf16* v_cache;
    bf16* out;                // [Tq, Hq, Dh]
    const int* block_table;   // [B, max_pages]
    const int* kv_lens;       // [B] tokens in the cache for this sequence (including the new ones)
    const int* cu_q;          // [B + 1] query offsets (prefill); null for decode (one query per sequence)
    const float* sinks;       // [Hq] or null
    float* part_o;            // decode scratch [B, Hq, splits, Dh] (with `parts`: [parts, Hq, Dh])
    float* part_ml;           // decode scratch [B, Hq, splits, 2] ([parts, Hq, 2])
    float scale;
    float softcap;            // 0 = off
    int window;               // 0 = full causal
    int B, Hq, Hkv, Dh, page_size, max_pages, splits;
    // Prefill only.  Context parallelism runs the kernel once per KV shard and merges the partial results:
    const int* q_pos0;        // [B] cache position of each sequence's first query, or null = kv_len - q_len
    float* lse_out;           // [Tq, Hq] log-sum-exp of the scaled scores seen by this call (-inf if none), or null
    // Decode only: the output again as int8 groups of 32 with (scale, sum), the form the following
    // quantised projection reads, so that no separate quantise launch is needed.  Null = not wanted.
    int8_t* out_q;            // [B, Hq * Dh]
    float2* out_ds;           // [B, Hq * Dh / 32]
    // Set by the launcher, not the caller: per (sequence, KV head) arrival counters.  When present, the
    // CTA that finishes a head group last merges the split partials itself and no combine kernel runs.
    unsigned* ticket;
    // Decode: positions per split fixed by the caller (a multiple of 32), so that a CTA's range and its block-table
    // entries do not wait for the sequence length; 0 = derive it from the length (ceil(span / splits), rounded to 32).
    // Negative: derive it too, and where attn_decode_ring_kernel runs take parts of -split_len positions at least.
    int split_len;
    // Output gate: head h of query row t is multiplied by sigmoid(gate[t * gate_tok + h]) (t: packed query row; decode:
    // the sequence).  Null: none.
    const void* gate;
    long gate_tok;            // elements between query rows
    int gate_f32;
    int Dv;                   // value head size (0 = Dh): v_cache [slots, Hkv, Dv], out [Tq, Hq, Dv]
    // Elements between slots where the rows of a slot are not dense (attention_vd.cu and the 32-bit kernel): 0 = Hkv * Dh
    // and Hkv * Dv.  Multiples of 8.
    long k_ld, v_ld;
    // The forms below are served by attention_vd.cu and the 32-bit kernel.
    int keep_first;           // with a window: these first positions stay visible as well
    const float* slopes;      // [Hq] or null: slopes[h] * (query position - key position) is taken off the scaled score
    int gate_cols;            // 1: the gate has a value per output column, gate[t * gate_tok + h * Dv + d]
    int kv_scale;             // != 0: a row of k_cache is key and value at once (Dv = Dh; v_cache is not read), and the score of a
                              // key is multiplied by the f32 number that starts at element kv_scale of its row
    const float* log_r1;      // [Hq] or null: log_r1[h] ln(1 + log_r2[h] (query position - key position)) is taken off the score
    const float* log_r2;
    const float* sig_bias;    // [Hq] or null: no softmax; a visible key's weight is sigmoid(score + sig_bias[h])
    // Decode (attn_decode_ring_kernel): 1 = the launch just ahead on the stream waits for its own predecessor before it lets this one start, and
    // writes nothing of lengths, block table and cache but the rows of this step's tokens, each sequence's newest one: everything older
    // may be read while it ends.  0 = it may have written anything.
    int ahead;
    // Decode (attn_decode_ring_kernel): `plan` not null: the parts of all sequences are a list of `parts` places, in which a long sequence among short ones
    // has more of them than the `each` (at most) of the others, in place of `splits` parts each.  Of tsb_attn_plan for the same lengths and window: int4
    // {sequence (-1: none), which of its parts, how many it has, positions of one} for every place; then int4 {sequence (-1: none), first place, how many}
    // for the sequences of more than one, of which there are no more than attn_part_merges.
    int parts, each;
    const int4* plan;
};

// How the sequences of a merged step are cut: `total` positions of all of them over `room` parts are the length that a part should have, of whole rounds of the
// ring kernel's four warps and no less than `least`.  A sequence takes `each` parts, none below `least`, as it would alone; one whose parts would be longer
// than twice that length takes as many as it needs to meet it, at most the 64 that the merge takes.  All of them together have each B + room places at most:
// what is cut finer has less than one part beyond its share of room.
__host__ __device__ __forceinline__ int attn_part_merges(int parts, int each, int B) { return each > 1 || parts - B * each > B ? B : parts - B * each; }
__host__ __device__ __forceinline__ int attn_part_len(long total, int room, int least) {
    const int p = (int)((total + room - 1) / room);
    return ((p > least ? p : least) + 63) & ~63;
}
__host__ __device__ __forceinline__ int attn_part_count(int span, int length, int each, int least, int* per) {
    int p = ((span + each - 1) / each + 63) & ~63;
    if (p < least) p = least;
    if (p > 2 * length) {
        const int k = (span + length - 1) / length;
        p = k > 64 ? ((span + 63) / 64 + 63) & ~63 : ((span + k - 1) / k + 63) & ~63;
    }
    *per = p;
    return span > p ? (span + p - 1) / p : 1;
}

// Whether only the kernels for head sizes of their own know a form that these arguments ask for.
static inline bool attn_needs_vd(const AttnArgs& a) {
    return (a.Dv != 0 && a.Dv != a.Dh) || a.k_ld != 0 || a.v_ld != 0 || a.keep_first > 0 || a.slopes != nullptr || a.gate_cols || a.kv_scale ||
           a.log_r1 != nullptr || a.sig_bias != nullptr || (a.Dh != 64 && a.Dh != 128 && a.Dh != 256 && a.Dh != 512);
}

#ifdef __CUDACC__
// the gate of head h, or with gate_cols of its column d
__device__ __forceinline__ float attn_gate(const AttnArgs& a, long t, int h, int d = 0) {
    if (a.gate == nullptr) return 1.f;
    const long i = t * a.gate_tok + (a.gate_cols ? (long)h * a.Dv + d : h);
    const float g = a.gate_f32 ? reinterpret_cast<const float*>(a.gate)[i] : bf2f(reinterpret_cast<const bf16*>(a.gate)[i]);
    return 1.f / (1.f + __expf(-g));
}
__device__ __forceinline__ const float* attn_key_factor(const AttnArgs& a, long slot) {
    return reinterpret_cast<const float*>(a.k_cache + slot * a.k_ld + a.kv_scale);
}
#endif

// attention_vd.cu: key and value head sizes of their own (multiples of 16)
int tsb_attn_prefill_vd_launch(const AttnArgs& a, int max_q, cudaStream_t s);
int tsb_attn_decode_vd_launch(const AttnArgs& a, cudaStream_t s);         // the caller launches the combine

// attention_decode_mma.cu: the tensor-core split kernel for decode batches (head sizes 64 / 128, up to 16 query heads
// per KV head); the caller launches the combine unless `*merged` comes back true (splits merged by a thread-block cluster), with `a` as it comes back:
// without `parts` where the kernel that runs knows none.
bool tsb_attn_decode_mma_supported(const AttnArgs& a);
int tsb_attn_decode_mma_launch(AttnArgs& a, cudaStream_t s, bool* merged);
int tsb_attn_decode_mma_fp8_launch(const AttnArgs& a, cudaStream_t s);      // e4m3 pages; the caller launches the combine
