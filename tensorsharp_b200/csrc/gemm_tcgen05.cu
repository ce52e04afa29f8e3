// bf16 GEMM on the 5th-generation tensor cores:  Y[t, n] = sum_k X[t, k] * W[n, k]
//   (+ bias[n]) (+ residual[t, n]),  f32 accumulation in tensor memory.
//
// The problem is run "weights as the M operand": each CTA owns 128 rows of W (output
// features) and BN tokens, so that a small token count still fills the 128-lane MMA.  Up to 64
// tokens of bf16 weights (and the tensor-parallel forms) take the kernels below, GGUF blocks gemm_blocks.cu; plain and grouped products of more
// run on pairs of CTAs (gemm_bf16_pair_kernel).
//
//   warp 0    : TMA producer - W and X tiles (64-element K slabs, 128-byte swizzle) into a
//               STAGES-deep shared-memory ring, completion on mbarriers
//   warp 1    : allocates tensor memory, one thread issues tcgen05.mma (128 x BN x 16) and
//               commits each stage back to the producer
//   warps 2-5 : epilogue - tcgen05.ld the accumulator (lane = feature, column = token),
//               add bias / residual, store coalesced along the feature dimension
//
// Replaces in the reference: mul_mat_q + stream-k fixup + quantize_mmq_q8_1
// (ggml-cuda/mmq.cuh:3301, :3542, quantize.cu:51), mul_mat_f (mmf.cuh:25) and the cuBLAS
// fallback (ggml-cuda.cu:1361-1497): quantised weights are decoded once into an L2-resident
// bf16 scratch by tsb_gather_rows and consumed here.
#include <cudaTypedefs.h>
#include <mutex>
#include <cstdlib>
#include <type_traits>
#include "glu.cuh"
#include "tcgen05.cuh"
#include "tp_fused.cuh"

struct GemmEpi {
    void* out;              // [T, ldo]
    const float* bias;      // [N] or null
    const void* residual;   // same dtype / layout as out, or null
    long ldo;
    int T, N;               // valid tokens, valid features
    int out_f32;
    // Tensor-parallel prefill (tp_fused.cuh); both null for an ordinary GEMM.
    const TpSeq* rs;        // GEMM -> reduce-scatter: store the tile into the token owner's accumulator over NVLink
    const TpSeq* ag;        // all-gather -> GEMM: X is the gathered buffer; wait for the tile's shard to arrive
    int rs_rows;            // size * shard (host copy, for the grid)
    int tile_rot;           // token tiles are visited starting from this one (see tsb_gemm_bf16_tp)
    // Grouped mode (mixture of experts): W is a stack of matrices of N rows each, X holds the rows of all groups sorted
    // by group, and token tile y of the grid is described by groups[3 * y .. 3 * y + 2] = {matrix index or -1 for an
    // unused tile, first row, end row}.  The list is built on the device, so the host never learns the group sizes.
    const int* groups;
    // Split-K (one-tile-per-CTA kernel, few tiles and a long K: decode batches of 9 to 64 rows): blockIdx.z takes a
    // range of k-blocks and stores its raw partial tile into ws[z][t][n]; splitk_reduce_kernel adds the parts in order
    // with bias and residual.  Null for an ordinary launch.
    float* ws;
    int kb_per_split;
    // Gated pair kernel: W holds N / 2 gate rows and then N / 2 up rows, out [T, N / 2] = act(gate, up), bf16.
    int act;
};

// Epilogue of one thread for 16 consecutive tokens of its feature n: out[t, n] = acc + bias (+ residual[t, n]).
// The residual values are all requested before the first store: with the load and the store of one token back to back
// (the residual may be the output buffer itself, so the compiler keeps their order) every token would cost a full
// memory round trip, 16 in a row per chunk.  Each element is read and written by the same thread, so reading ahead is
// safe for an in-place residual too.
__device__ __forceinline__ void gemm_store16(const GemmEpi& ep, const uint32_t (&r)[16], int n, int t0, int t_end, float bias) {
    float res[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) res[j] = 0.f;
    if (ep.residual != nullptr) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int t = t0 + j;
            if (t < t_end) {
                const long o = (long)t * ep.ldo + n;
                res[j] = ep.out_f32 ? reinterpret_cast<const float*>(ep.residual)[o] : bf2f(reinterpret_cast<const bf16*>(ep.residual)[o]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int t = t0 + j;
        if (t < t_end) {
            const float v = __uint_as_float(r[j]) + bias + res[j];
            const long o = (long)t * ep.ldo + n;
            if (ep.out_f32) reinterpret_cast<float*>(ep.out)[o] = v;
            else reinterpret_cast<bf16*>(ep.out)[o] = f2bf(v);
        }
    }
}

template <int BN, int STAGES>
struct GemmSmem {
    static constexpr int A_BYTES = 128 * 64 * 2;
    static constexpr int B_BYTES = BN * 64 * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int BAR_OFF = STAGES * STAGE_BYTES;
    static constexpr int TOTAL = BAR_OFF + (2 * STAGES + 1) * 8 + 16 + 1024;  // + alignment slack
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(192) gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmW,
                                                        const __grid_constant__ CUtensorMap tmX, GemmEpi ep, int K,
                                                        int* status) {
    using L = GemmSmem<BN, STAGES>;
    constexpr int TMEM_COLS = BN < 32 ? 32 : BN;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_bar = empty_bar + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * 128;       // first feature (row of W)
    int n0 = (int)((blockIdx.y + (unsigned)ep.tile_rot) % gridDim.y) * BN;        // first token
    int t_end = ep.T;                      // tokens at or past this row are not stored
    int w_row0 = m0;                       // row of the (stacked) weight matrix where this tile's features start
    bool active = true;
    const int kb_all = (K + 63) / 64;
    const int kb_first = ep.ws != nullptr ? (int)blockIdx.z * ep.kb_per_split : 0;
    const int kblocks = ep.ws != nullptr ? min(kb_all - kb_first, ep.kb_per_split) : kb_all;     // this CTA's share (>= 1)

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full_bar[s], 1);
            tc::mbar_init(&empty_bar[s], 1);
        }
        tc::mbar_init(acc_bar, 1);
        tc::fence_barrier_init();
    }
    if (warp == 1) tc::tmem_alloc<TMEM_COLS>(tmem_slot);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();        // barrier set-up and the TMEM allocation above overlap the previous kernel's tail
    pdl_trigger();
    int group = 0;
    if (ep.groups != nullptr) {
        const int* gt = ep.groups + 3 * blockIdx.y;
        group = gt[0];
        active = group >= 0;
        n0 = gt[1];
        t_end = gt[2];
        w_row0 = group * ep.N + m0;
    }

    if (!active) {
        // an unused entry of the tile list: nothing to load, multiply or store
    } else if (warp == 0) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&tmW);
            tc::tma_prefetch_desc(&tmX);
            if (ep.ag != nullptr) {
                // the rows of this token tile come from one rank; its stores are complete once its
                // arrival counter here has reached the target left by the preceding gather kernel
                const TpSeq* g = ep.ag;
                const int owner = n0 / g->shard;
                if (owner < g->size && !tp_wait_counter(g->ag_arrive[g->rank] + owner, *g->ag_target))
                    atomicExch(status, 4);
            }
            for (int kb = 0; kb < kblocks; ++kb) {
                const int s = kb % STAGES;
                const uint32_t ph = (kb / STAGES) & 1;
                if (!tc::mbar_wait(&empty_bar[s], ph ^ 1)) { atomicExch(status, 1); break; }
                unsigned char* a = smem + s * L::STAGE_BYTES;
                tc::mbar_expect_tx(&full_bar[s], L::STAGE_BYTES);
                tc::tma_load_2d(a, &tmW, &full_bar[s], (kb_first + kb) * 64, w_row0);
                tc::tma_load_2d(a + L::A_BYTES, &tmX, &full_bar[s], (kb_first + kb) * 64, n0);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = tc::make_idesc_bf16(128, BN);
            bool ok = true;
            for (int kb = 0; kb < kblocks && ok; ++kb) {
                const int s = kb % STAGES;
                const uint32_t ph = (kb / STAGES) & 1;
                if (!tc::mbar_wait(&full_bar[s], ph)) { atomicExch(status, 2); ok = false; break; }
                tc::fence_after_sync();
                const uint32_t a = tc::smem_u32(smem + s * L::STAGE_BYTES);
                const uint64_t da = tc::make_desc_sw128(a), db = tc::make_desc_sw128(a + L::A_BYTES);
#pragma unroll
                for (int k = 0; k < 4; ++k) {   // 4 x (K = 16) per 64-element slab: +32 bytes = +2 descriptor units
                    tc::mma_f16_ss(tmem_base, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                }
                tc::mma_commit(&empty_bar[s]);
            }
            if (ok) tc::mma_commit(acc_bar);
        }
        __syncwarp();
    } else {
        const int q = warp & 3;                       // TMEM lane quadrant this warp may read
        if (tc::warp_wait(acc_bar, 0)) {
            tc::fence_after_sync();
            const int n = m0 + q * 32 + lane;             // feature owned by this thread
            const float bias = (ep.bias && n < ep.N && (ep.rs == nullptr || ep.rs->rank == 0)) ? ep.bias[(long)group * ep.N + n] : 0.f;
            bf16* rs_dst = nullptr;
            if (ep.rs != nullptr) {
                const TpSeq* g = ep.rs;
                const int owner = n0 / g->shard;                    // a token tile never straddles two shards
                if (owner < g->size)       // this rank's slot of the current accumulator, rebased to global token indices
                    rs_dst = g->acc[owner] + ((long)(*g->rs_phase & 1u) * g->size + g->rank) * g->shard * g->ld -
                             (long)owner * g->shard * g->ld;
            }
#pragma unroll 1
            for (int c = 0; c < BN / 16; ++c) {
                uint32_t r[16];
                tc::tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + c * 16, r);
                tc::tmem_ld_wait();
                if (rs_dst != nullptr) {
                    if (n < ep.N) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int t = n0 + c * 16 + j;
                            // a warp covers 32 consecutive features of one token: one 64-byte packet.  Rows
                            // past T are written too (zeros from the zero-filled X tile) so the owner
                            // never reads a stale slot row.
                            rs_dst[(long)t * ep.rs->ld + n] = f2bf(__uint_as_float(r[j]) + (t < ep.T ? bias : 0.f));
                        }
                    }
                } else if (ep.ws != nullptr) {
                    if (n < ep.N) {
                        float* part = ep.ws + (long)blockIdx.z * ep.T * ep.N;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int t = n0 + c * 16 + j;
                            if (t < ep.T) part[(long)t * ep.N + n] = __uint_as_float(r[j]);
                        }
                    }
                } else if (n < ep.N) {
                    gemm_store16(ep, r, n, n0 + c * 16, t_end, bias);
                }
            }
        } else {
            atomicExch(status, 3);
        }
        if (ep.rs != nullptr) __threadfence_system();               // reductions visible before the arrival below
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc<TMEM_COLS>(tmem_base);
    }
    if (ep.rs != nullptr && threadIdx.x == 0) {
        const TpSeq* g = ep.rs;
        const int owner = n0 / g->shard;
        if (owner < g->size) red_release_inc_sys(g->rs_arrive[owner]);
        const unsigned done = atomicAdd(g->ticket, 1u);
        if (done == gridDim.x * gridDim.y - 1) {
            // every owner receives (feature tiles) x (token tiles per shard) arrivals from each rank
            *g->ticket = 0;
            __threadfence();
            *g->rs_target += (unsigned)g->size * gridDim.x * (unsigned)(g->shard / BN);
        }
    }
}

// out[t, n] = sum over the splits (in order) of ws[z][t][n] + bias[n] + residual[t, n]
__global__ void __launch_bounds__(256) splitk_reduce_kernel(GemmEpi ep, int splits) {
    pdl_wait();
    pdl_trigger();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)ep.T * ep.N) return;
    const int t = (int)(i / ep.N), n = (int)(i % ep.N);
    float v = ep.bias ? ep.bias[n] : 0.f;
    for (int z = 0; z < splits; ++z) v += ep.ws[((long)z * ep.T + t) * ep.N + n];
    const long o = (long)t * ep.ldo + n;
    if (ep.out_f32) {
        if (ep.residual) v += reinterpret_cast<const float*>(ep.residual)[o];
        reinterpret_cast<float*>(ep.out)[o] = v;
    } else {
        if (ep.residual) v += bf2f(reinterpret_cast<const bf16*>(ep.residual)[o]);
        reinterpret_cast<bf16*>(ep.out)[o] = f2bf(v);
    }
}

// ------------------------------------------------------------------------------------------
// Persistent form of the tensor-parallel GEMMs: one CTA per SM walks the tiles
// (feature tile fastest, so CTAs that run together share a token slab in L2), the TMA producer keeps filling the
// shared-memory ring across tile boundaries, and tensor memory holds two accumulators: the epilogue warps drain tile i
// while the MMA warp already multiplies tile i + 1.  With short K (the gate / up and QKV projections) the epilogue is
// about half of a tile's time in the one-tile-per-CTA kernel above; here it disappears behind the next main loop.
// ------------------------------------------------------------------------------------------
template <int BN, int STAGES>
__global__ void __launch_bounds__(192) gemm_bf16_persistent_kernel(const __grid_constant__ CUtensorMap tmW,
                                                                   const __grid_constant__ CUtensorMap tmX, GemmEpi ep, int K,
                                                                   int m_tiles, int total_tiles, int* status) {
    using L = GemmSmem<BN, STAGES>;
    constexpr int TMEM_COLS = 2 * BN;
    static_assert(TMEM_COLS >= 32 && TMEM_COLS <= 512, "two accumulators must fit tensor memory");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;          // [2] accumulator complete (one commit by the MMA thread)
    uint64_t* acc_empty = acc_full + 2;               // [2] accumulator drained (one arrival per epilogue warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    // reduce-scatter epilogue: two buffers of 16 tokens x 128 features (bf16) in which the four epilogue warps turn
    // their feature-per-lane fragments into whole token rows, so that a peer store covers 256 contiguous bytes
    bf16* rs_stage = reinterpret_cast<bf16*>(smem + L::BAR_OFF + 256);      // past the barriers (at most 2 * 8 + 4 words) and the TMEM slot
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kblocks = (K + 63) / 64;
    const int n_tiles = total_tiles / m_tiles;
    // feature tile fastest: the CTAs that run together share one token slab
    auto tile_m = [&](int tile) { return tile % m_tiles; };
    auto tile_n = [&](int tile) { return tile / m_tiles; };
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full_bar[s], 1);
            tc::mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], 4);
        }
        tc::fence_barrier_init();
    }
    if (warp == 1) tc::tmem_alloc<TMEM_COLS>(tmem_slot);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&tmW);
            tc::tma_prefetch_desc(&tmX);
            long it = 0;                               // k-blocks issued so far, over all tiles of this CTA
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const int w_row0 = tile_m(tile) * 128, n0 = (int)((tile_n(tile) + (unsigned)ep.tile_rot) % n_tiles) * BN;
                if (ep.ag != nullptr) {
                    // the rows of this token tile come from one rank; its stores are complete once its arrival counter
                    // here has reached the target left by the preceding gather kernel
                    const TpSeq* g = ep.ag;
                    const int owner = n0 / g->shard;
                    if (owner < g->size && !tp_wait_counter(g->ag_arrive[g->rank] + owner, *g->ag_target)) atomicExch(status, 4);
                }
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = (int)(it % STAGES);
                    const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                    if (!tc::mbar_wait(&empty_bar[s], ph ^ 1)) { atomicExch(status, 1); ok = false; break; }
                    unsigned char* a = smem + s * L::STAGE_BYTES;
                    tc::mbar_expect_tx(&full_bar[s], L::STAGE_BYTES);
                    tc::tma_load_2d(a, &tmW, &full_bar[s], kb * 64, w_row0);
                    tc::tma_load_2d(a + L::A_BYTES, &tmX, &full_bar[s], kb * 64, n0);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = tc::make_idesc_bf16(128, BN);
            long it = 0;
            int j = 0;                                 // tiles done by this CTA
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const int buf = j & 1;
                const uint32_t aph = (uint32_t)(j >> 1) & 1u;
                if (!tc::mbar_wait(&acc_empty[buf], aph ^ 1)) { atomicExch(status, 5); ok = false; break; }
                tc::fence_after_sync();
                const uint32_t acc = tmem_base + (uint32_t)buf * BN;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = (int)(it % STAGES);
                    const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                    if (!tc::mbar_wait(&full_bar[s], ph)) { atomicExch(status, 2); ok = false; break; }
                    tc::fence_after_sync();
                    const uint32_t a = tc::smem_u32(smem + s * L::STAGE_BYTES);
                    const uint64_t da = tc::make_desc_sw128(a), db = tc::make_desc_sw128(a + L::A_BYTES);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tc::mma_f16_ss(acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                    tc::mma_commit(&empty_bar[s]);
                }
                if (ok) tc::mma_commit(&acc_full[buf]);
                ++j;
            }
        }
        __syncwarp();
    } else {
        const int q = warp & 3;
        int j = 0;
        for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
            const int n0 = (int)((tile_n(tile) + (unsigned)ep.tile_rot) % n_tiles) * BN;
            const int buf = j & 1;
            const uint32_t aph = (uint32_t)(j >> 1) & 1u;
            const int m0 = tile_m(tile) * 128;
            const int n = m0 + q * 32 + lane;
            if (!tc::warp_wait(&acc_full[buf], aph)) { atomicExch(status, 3); break; }
            tc::fence_after_sync();
            const float bias = (ep.bias && n < ep.N && (ep.rs == nullptr || ep.rs->rank == 0)) ? ep.bias[n] : 0.f;
            if (ep.rs == nullptr) {
#pragma unroll 1
                for (int c = 0; c < BN / 16; ++c) {
                    uint32_t r[16];
                    tc::tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * BN + c * 16, r);
                    tc::tmem_ld_wait();
                    if (n < ep.N) gemm_store16(ep, r, n, n0 + c * 16, ep.T, bias);
                }
                tc::fence_before_sync();              // this warp's reads of the accumulator are complete
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
            } else {
                // GEMM -> reduce-scatter: this rank's slot of the token owner's accumulator, over NVLink.  Rows past T
                // are written too (zeros from the zero-filled X tile) so the owner never reads a stale slot row.
                const TpSeq* g = ep.rs;
                const int owner = n0 / g->shard;                    // a token tile never straddles two shards
                bf16* rs_dst = nullptr;
                if (owner < g->size)
                    rs_dst = g->acc[owner] + ((long)(*g->rs_phase & 1u) * g->size + g->rank) * g->shard * g->ld -
                             (long)owner * g->shard * g->ld;
                const int et = threadIdx.x - 64;                    // 0..127 among the epilogue threads
#pragma unroll 1
                for (int c = 0; c < BN / 16; ++c) {
                    uint32_t r[16];
                    tc::tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * BN + c * 16, r);
                    tc::tmem_ld_wait();
                    bf16* st = rs_stage + (c & 1) * (16 * 128);
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj)
                        st[jj * 128 + q * 32 + lane] = f2bf(__uint_as_float(r[jj]) + (n0 + c * 16 + jj < ep.T ? bias : 0.f));
                    asm volatile("bar.sync 1, 128;" ::: "memory");  // the 16 x 128 chunk is complete
                    if (rs_dst != nullptr) {
                        // thread -> tokens et / 16 and et / 16 + 8, eight features: 16 threads cover one 256-byte row
#pragma unroll
                        for (int rr = 0; rr < 2; ++rr) {
                            const int tok = (et >> 4) + rr * 8, f0 = (et & 15) * 8;
                            const int nn = m0 + f0;
                            if (nn < ep.N) {                        // N is a multiple of 8 (checked by the host)
                                const uint4 v = *reinterpret_cast<const uint4*>(st + tok * 128 + f0);
                                *reinterpret_cast<uint4*>(rs_dst + (long)(n0 + c * 16 + tok) * g->ld + nn) = v;
                            }
                        }
                    }
                    // the other buffer is written next; this one again two chunks on, after the next barrier
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
                __threadfence_system();                             // this thread's peer stores are visible before the arrival
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (et == 0) {
                    if (owner < g->size) red_release_inc_sys(g->rs_arrive[owner]);
                    const unsigned done = atomicAdd(g->ticket, 1u);
                    if (done == (unsigned)total_tiles - 1u) {
                        // every owner receives (feature tiles) x (token tiles per shard) arrivals from each rank
                        *g->ticket = 0;
                        __threadfence();
                        *g->rs_target += (unsigned)g->size * (unsigned)m_tiles * (unsigned)(g->shard / BN);
                    }
                }
            }
            ++j;
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc<TMEM_COLS>(tmem_base);
    }
}

template <int BN, int STAGES>
static int launch_gemm_persistent(const CUtensorMap& tw, const CUtensorMap& tx, const GemmEpi& ep, int K, int sms, int* status,
                                  cudaStream_t s) {
    using L = GemmSmem<BN, STAGES>;
    constexpr int SMEM = L::TOTAL + 256 + 2 * 16 * 128 * 2;      // more barriers than the one-tile kernel + the reduce-scatter staging rows
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemm_bf16_persistent_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured = true;
    }
    // with a reduce-scatter epilogue the tiles also cover the padding rows of the last shard, so that every owner sees
    // the same number of arrivals
    const int t_cover = ep.rs != nullptr ? ep.rs_rows : ep.T;
    const int m_tiles = (ep.N + 127) / 128, n_tiles = (t_cover + BN - 1) / BN, total = m_tiles * n_tiles;
    const int grid = total < sms ? total : sms;
    TSB_CHECK_CUDA(tsb_launch(gemm_bf16_persistent_kernel<BN, STAGES>, dim3(grid), dim3(192), (size_t)SMEM, s, tw, tx, ep, K, m_tiles,
                              total, status));
    return TSB_OK;
}

// ------------------------------------------------------------------------------------------
// Pairs of CTAs (plain and grouped GEMMs of more than 64 tokens).  A 128 x 256 tile on one SM pulls 384 rows of a K slab
// for 512 cycles of products, 96 bytes a cycle from L2, and the kernel above settles where L2 delivers about 70.  Two SMs
// that share one 256 x bn tile (tcgen05.mma.cta_group::2) pull 128 + bn / 2 rows each for the same products: 64 bytes a
// cycle at bn = 256.  Each CTA loads its 128 features and its half of the tokens, the even CTA issues the products, each
// CTA keeps the accumulators of its own features in its own tensor memory (two buffers, epilogue under the next tile as
// above).  bn is any multiple of 16, so that the last wave can be filled (choose_pair_bn).
// Bound by the tensor pipe (busy 90 % of the time that an SM has work at 2048 x 19456 x 2560), on narrow shapes by the last wave.
// Measured (us; one CTA per SM as above, one-tile or persistent / this one): 65 x 2560 x 4096 21.1 / 19.2, 512 x 6144 x 2560 24.2 /
// 17.5, 2048 x 2560 x 4096 63.7 / 41.9, 2048 x 2560 x 9728 134 / 91, 4096 x 37984 x 2560 636 / 572; 2048 x (2 x 9728) x 2560 with
// SwiGLU 187 (and a kernel of its own for it) / 149.
// ------------------------------------------------------------------------------------------
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_STAGE_BYTES = 2 * 128 * 128;                  // 128 features and up to 128 tokens, 64 bf16 each
constexpr int PAIR_SMEM = PAIR_STAGES * PAIR_STAGE_BYTES + 256 + 1024;
constexpr int PAIR_GLU_SMEM = 4 * 2 * 16 * 32 * 4;               // two chunks of 16 tokens for each of four pairs of epilogue warps

// A barrier of the 64 threads that name `id`, which also tells each whether the predicate held for all of them.
__device__ __forceinline__ bool bar_all64(int id, bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, 64, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)ok), "r"(id) : "memory");
    return r != 0;
}

// GLU: the rows of a CTA's tile are 64 gate rows and the 64 up rows of the same features.  The warp that reads the gates of some
// features and tokens and the one that reads their up values give one another half of a chunk through shared memory and form the
// activation of eight tokens each, so the gated activation leaves the kernel and its two inputs, rounded to bf16 as a kernel of
// its own would have read them, never reach memory.
template <bool GLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320) gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmW,
                                                                                       const __grid_constant__ CUtensorMap tmX, GemmEpi ep, int K,
                                                                                       int bn, int m_tiles, int total_tiles, int m_group, int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + PAIR_STAGES * PAIR_STAGE_BYTES);      // the even CTA's count for both
    uint64_t* empty_bar = full_bar + PAIR_STAGES;
    uint64_t* acc_full = empty_bar + PAIR_STAGES;      // [2] accumulator complete
    uint64_t* acc_empty = acc_full + 2;                // [2] drained (one arrival per epilogue warp of both CTAs; the even CTA's)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    float* up_stage = reinterpret_cast<float*>(smem + PAIR_STAGES * PAIR_STAGE_BYTES + 256);
    constexpr int TILE_M = GLU ? 128 : 256;            // output features of a pair's tile
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)tc::cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int kblocks = (K + 63) / 64, n_tiles = total_tiles / m_tiles;
    // Tile order: groups of m_group feature tiles; inside a group feature tile fastest.  The pairs that run together share a
    // few weight tiles and a few token tiles, and a group's weights stay in L2 while the tokens pass by once.
    auto tile_mn = [&](int tile, int& m, int& n) {
        const int per = m_group * n_tiles, g = tile / per, r = tile - g * per, w = min(m_group, m_tiles - g * m_group);
        n = r / w;
        m = g * m_group + r - n * w;
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < PAIR_STAGES; ++s) {
            tc::mbar_init(&full_bar[s], 1);
            tc::mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], 16);
        }
        tc::fence_barrier_init();
    }
    // The tensor memory of a pair is allocated on both SMs at once, so neither CTA asks for it before the other one is there: asked
    // for while the peer's SM was still busy with the kernel ahead, the allocation never came back.
    __syncthreads();
    tc::cluster_sync();
    if (warp == 1) tc::tmem_alloc_pair<512>(tmem_slot);
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();                                // both CTAs have theirs, and barriers that the peer may arrive on
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&tmW);
            tc::tma_prefetch_desc(&tmX);
            const uint32_t half = (uint32_t)bn / 2;
            int it = 0;                                // k-blocks issued so far, over all tiles
            bool ok = true;
            for (int tile = pair; tile < total_tiles && ok; tile += pairs) {
                int m, n;
                tile_mn(tile, m, n);
                int w_row0 = m * TILE_M + rank * (TILE_M / 2), n0 = n * bn;
                if (ep.groups != nullptr) {
                    const int* gt = ep.groups + 3 * n;
                    if (gt[0] < 0) continue;
                    w_row0 += gt[0] * ep.N;
                    n0 = gt[1];
                }
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % PAIR_STAGES;
                    if (!tc::mbar_wait(&empty_bar[s], ((it / PAIR_STAGES) & 1) ^ 1)) { atomicExch(status, 1); ok = false; break; }
                    unsigned char* a = smem + s * PAIR_STAGE_BYTES;
                    if (rank == 0) tc::mbar_expect_tx(&full_bar[s], 2 * (128 + half) * 128);
                    const uint32_t bar = tc::map_to_rank(&full_bar[s], 0);
                    tc::tma_load_2d_pair(a, &tmW, bar, kb * 64, w_row0);
                    if (GLU) tc::tma_load_2d_pair(a + 64 * 128, &tmW, bar, kb * 64, w_row0 + ep.N / 2);
                    tc::tma_load_2d_pair(a + 128 * 128, &tmX, bar, kb * 64, n0 + rank * (int)half);
                }
            }
            // The pair leaves with no copy in flight, whichever wait gave up: the last slab of every stage, of both CTAs, has arrived.
            if (rank == 0)
                for (int i = max(0, it - PAIR_STAGES); i < it; ++i) tc::mbar_wait(&full_bar[i % PAIR_STAGES], (i / PAIR_STAGES) & 1);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = tc::make_idesc_bf16(256, bn);
            int it = 0, j = 0;                         // j: tiles done by this pair
            bool ok = true;
            for (int tile = pair; tile < total_tiles && ok; tile += pairs) {
                int m, n;
                tile_mn(tile, m, n);
                if (ep.groups != nullptr && ep.groups[3 * n] < 0) continue;
                const int buf = j & 1;
                if (!tc::mbar_wait(&acc_empty[buf], ((j >> 1) & 1) ^ 1)) { atomicExch(status, 5); ok = false; break; }
                tc::fence_after_sync();
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const int s = it % PAIR_STAGES;
                    if (!tc::mbar_wait(&full_bar[s], (it / PAIR_STAGES) & 1)) { atomicExch(status, 2); ok = false; break; }
                    tc::fence_after_sync();
                    const uint32_t a = tc::smem_u32(smem + s * PAIR_STAGE_BYTES);
                    const uint64_t da = tc::make_desc_sw128(a), db = tc::make_desc_sw128(a + 128 * 128);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tc::mma_f16_ss_pair(tmem_base + buf * 256, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                    tc::mma_commit_pair(&empty_bar[s]);
                }
                if (ok) tc::mma_commit_pair(&acc_full[buf]);
                ++j;
            }
        }
        __syncwarp();
    } else {
        // eight warps: two per quadrant of the accumulator's lanes, which take turns over chunks of 16 tokens
        const int q = warp & 3, turn = (warp - 2) >> 2;
        int j = 0;
        for (int tile = pair; tile < total_tiles; tile += pairs) {
            int m, n, t_end = ep.T, group = 0;
            tile_mn(tile, m, n);
            int n0 = n * bn;
            if (ep.groups != nullptr) {
                const int* gt = ep.groups + 3 * n;
                group = gt[0];
                if (group < 0) continue;
                n0 = gt[1];
                t_end = gt[2];
            }
            const int buf = j & 1, half = ep.N / 2;
            const int f = GLU ? m * 128 + rank * 64 + (q & 1) * 32 + lane : m * 256 + rank * 128 + q * 32 + lane;
            const bool mine = f < (GLU ? half : ep.N);
            const float bias = (ep.bias && mine) ? ep.bias[(long)group * ep.N + f + (GLU && q >= 2 ? half : 0)] : 0.f;
            const int cols = min(bn, t_end - n0);                  // tokens of this tile that exist
            if (GLU) {
                const int pr = turn * 2 + (q & 1);
                // Both warps of the pair go on, or both leave: one that gave up alone would leave the other at the barriers below.
                // The barrier also says that the place where this tile starts, which the tile before may have read last, was read.
                if (!bar_all64(pr + 1, tc::warp_wait(&acc_full[buf], (j >> 1) & 1))) { atomicExch(status, 3); break; }
                tc::fence_after_sync();
                auto chunks = [&](auto act) {
                    int side = 0;
#pragma unroll 1
                    for (int c = turn; c * 16 < cols; c += 2, side ^= 1) {
                        uint32_t r[16];
                        tc::tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * 256 + c * 16, r);
                        tc::tmem_ld_wait();
                        float v[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = bf2f(f2bf(__uint_as_float(r[i]) + bias));
                        float* st = up_stage + (pr * 2 + side) * (16 * 32) + lane;
#pragma unroll
                        for (int i = 0; i < 8; ++i) st[q < 2 ? (i + 8) * 32 : i * 32] = q < 2 ? v[i + 8] : v[i];
                        // both warps of the pair: the other half is there; and that of two chunks ago, in the same place, was read
                        asm volatile("bar.sync %0, 64;" ::"r"(pr + 1) : "memory");
                        const int left = cols - c * 16;
                        bf16* p = reinterpret_cast<bf16*>(ep.out) + (long)(n0 + c * 16 + (q < 2 ? 0 : 8)) * ep.ldo + f;
                        if (mine) {
#pragma unroll
                            for (int i = 0; i < 8; ++i, p += ep.ldo) {
                                const float other = st[q < 2 ? i * 32 : (i + 8) * 32], g = q < 2 ? v[i] : other, u = q < 2 ? other : v[i + 8];
                                if ((q < 2 ? i : i + 8) < left) *p = f2bf(act_glu(decltype(act)::value, g, u));
                            }
                        }
                    }
                };
                switch (ep.act) {
                case ACT_SWIGLU: chunks(std::integral_constant<int, ACT_SWIGLU>{}); break;
                case ACT_GEGLU_TANH: chunks(std::integral_constant<int, ACT_GEGLU_TANH>{}); break;
                case ACT_GEGLU_ERF: chunks(std::integral_constant<int, ACT_GEGLU_ERF>{}); break;
                default: chunks(std::integral_constant<int, ACT_SWIGLU_OAI>{}); break;
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive_cluster(tc::map_to_rank(&acc_empty[buf], 0));
                ++j;
                continue;
            }
            // the residual does not depend on the products: a chunk's values are requested one chunk ahead, the first
            // one's before the wait for the accumulator
            const long at = (long)n0 * ep.ldo + f;
            float res[16], next[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) res[i] = next[i] = 0.f;
            auto residual = [&](int c, float (&v)[16]) {
                const int left = cols - c * 16;
                if (ep.residual == nullptr || !mine || left <= 0) return;
                if (ep.out_f32) {
                    const float* p = reinterpret_cast<const float*>(ep.residual) + at + (long)(c * 16) * ep.ldo;
#pragma unroll
                    for (int i = 0; i < 16; ++i, p += ep.ldo)
                        if (i < left) v[i] = *p;
                } else {
                    const bf16* p = reinterpret_cast<const bf16*>(ep.residual) + at + (long)(c * 16) * ep.ldo;
#pragma unroll
                    for (int i = 0; i < 16; ++i, p += ep.ldo)
                        if (i < left) v[i] = bf2f(*p);
                }
            };
            residual(turn, res);
            if (!tc::warp_wait(&acc_full[buf], (j >> 1) & 1)) { atomicExch(status, 3); break; }
            tc::fence_after_sync();
#pragma unroll 1
            for (int c = turn; c * 16 < cols; c += 2) {
                residual(c + 2, next);
                uint32_t r[16];
                tc::tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * 256 + c * 16, r);
                tc::tmem_ld_wait();
                if (mine) {
                    const int left = cols - c * 16;
                    if (ep.out_f32) {
                        float* p = reinterpret_cast<float*>(ep.out) + at + (long)(c * 16) * ep.ldo;
#pragma unroll
                        for (int i = 0; i < 16; ++i, p += ep.ldo)
                            if (i < left) *p = __uint_as_float(r[i]) + bias + res[i];
                    } else {
                        bf16* p = reinterpret_cast<bf16*>(ep.out) + at + (long)(c * 16) * ep.ldo;
#pragma unroll
                        for (int i = 0; i < 16; ++i, p += ep.ldo)
                            if (i < left) *p = f2bf(__uint_as_float(r[i]) + bias + res[i]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) res[i] = next[i];
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_cluster(tc::map_to_rank(&acc_empty[buf], 0));
            ++j;
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();                                // neither CTA leaves while the other may still read or signal its memory
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc_pair<512>(tmem_base);
    }
    __syncwarp();
    tc::cluster_sync();                                // the tensor memory of a pair is given back by both CTAs: neither is gone before the other has done so
}

template <bool GLU>
static int launch_gemm_pair(const void* W, long ldw, long w_rows, const void* X, long ldx, long x_rows, const GemmEpi& ep, int K, int bn, int n_tiles,
                            int sms, int* status, cudaStream_t s) {
    constexpr int SMEM = PAIR_SMEM + (GLU ? PAIR_GLU_SMEM : 0);
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemm_bf16_pair_kernel<GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured = true;
    }
    CUtensorMap tw, tx;
    int rc = tsb_make_tmap_2d_bf16(&tw, W, (uint64_t)w_rows, (uint64_t)K, (uint64_t)ldw, GLU ? 64 : 128, 64);
    if (rc) return rc;
    rc = tsb_make_tmap_2d_bf16(&tx, X, (uint64_t)x_rows, (uint64_t)K, (uint64_t)ldx, (uint32_t)bn / 2, 64);
    if (rc) return rc;
    const int m_tiles = GLU ? (ep.N / 2 + 127) / 128 : (ep.N + 255) / 256, total = m_tiles * n_tiles, pairs = total < sms / 2 ? total : sms / 2;
    // groups of eight feature tiles, or all of them where the list of token tiles decides which matrix is read
    const int m_group = ep.groups != nullptr || m_tiles < 8 ? m_tiles : 8;
    TSB_CHECK_CUDA(tsb_launch(gemm_bf16_pair_kernel<GLU>, dim3(2 * pairs), dim3(320), (size_t)SMEM, s, tw, tx, ep, K, bn, m_tiles, total, m_group, status));
    return TSB_OK;
}

// Cycles per 64-element K slab of the slowest SM, from the products (4096 multiply-adds a cycle and SM) and the rows that it
// pulls from L2 (about 70 bytes a cycle when all SMs pull), for the tiles of the slowest SM or pair.
static double gemm_cost(long tiles, long units, int rows, int macs) {
    const double pull = rows * 128.0 / 70, mul = macs * 64.0 / 4096;
    return (double)((tiles + units - 1) / units) * (pull > mul ? pull : mul);
}
// Token tile of the pair kernel with the least cost, and that cost.  Small tiles fill the last wave, large ones re-read less.
static int choose_pair_bn(int T, int N, int sms) {
    int best = 0;
    double least = 1e30;
    for (int bn = 256; bn >= 32; bn -= 16) {
        const double c = gemm_cost((long)((N + 255) / 256) * ((T + bn - 1) / bn), sms / 2, 128 + bn / 2, 128 * bn);
        if (c < least * 0.999) least = c, best = bn;
    }
    return best;
}

// ------------------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
static std::once_flag g_encode_once;

static void resolve_encode() {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
        g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
}

// A tensor map over bf16 elements: `dims` and `box` innermost first, `strides_elems` of dimensions 1 .. rank - 1, the 128-byte swizzle.
int tsb_make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_elems, const uint32_t* box) {
    std::call_once(g_encode_once, resolve_encode);
    if (!g_encode) {
        tsb_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return TSB_ERR_CUDA;
    }
    TSB_CHECK_ARG(rank >= 2 && rank <= 3, "tensor map of rank %d", rank);
    TSB_CHECK_ARG((reinterpret_cast<uintptr_t>(base) & 15) == 0, "tensor map base %p is not 16-byte aligned", base);
    cuuint64_t gdim[3], gstride[2];
    cuuint32_t gbox[3], estr[3] = {1, 1, 1};
    for (int i = 0; i < rank; ++i) {
        gdim[i] = dims[i];
        gbox[i] = box[i];
        if (i + 1 < rank) {
            gstride[i] = strides_elems[i] * 2;
            TSB_CHECK_ARG(gstride[i] % 16 == 0, "tensor map row stride %llu elements is not a multiple of 16 bytes", (unsigned long long)strides_elems[i]);
        }
    }
    CUresult r = g_encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstride, gbox, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        tsb_set_error("cuTensorMapEncodeTiled failed with CUresult %d (inner dimensions %llu x %llu, box %u x %u)", (int)r,
                      (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1]);
        return TSB_ERR_CUDA;
    }
    return TSB_OK;
}

int tsb_make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t row_stride_elems,
                          uint32_t box_rows, uint32_t box_cols) {
    const uint64_t dims[2] = {cols, rows};
    const uint32_t box[2] = {box_cols, box_rows};
    return tsb_make_tmap_bf16(out, base, 2, dims, &row_stride_elems, box);
}

// A map over rows of bytes.  Boxes of 128 and of 64 bytes take the swizzle of their width, others none.
int tsb_make_tmap_bytes(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t box_bytes) {
    std::call_once(g_encode_once, resolve_encode);
    if (!g_encode) {
        tsb_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return TSB_ERR_CUDA;
    }
    TSB_CHECK_ARG((reinterpret_cast<uintptr_t>(base) & 15) == 0, "tensor map base %p is not 16-byte aligned", base);
    TSB_CHECK_ARG(row_bytes % 16 == 0 && box_bytes % 16 == 0 && box_bytes <= 256 && box_rows <= 256, "tensor map of rows of %llu bytes, box %u x %u",
                  (unsigned long long)row_bytes, box_rows, box_bytes);
    const cuuint64_t gdim[2] = {row_bytes, rows}, gstride[1] = {row_bytes};
    const cuuint32_t gbox[2] = {box_bytes, box_rows}, estr[2] = {1, 1};
    const CUtensorMapSwizzle sw = box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE;
    CUresult r = g_encode(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), gdim, gstride, gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        tsb_set_error("cuTensorMapEncodeTiled failed with CUresult %d (rows of %llu bytes, box %u x %u)", (int)r, (unsigned long long)row_bytes, box_rows, box_bytes);
        return TSB_ERR_CUDA;
    }
    return TSB_OK;
}

template <int BN, int STAGES>
static int launch_gemm(const CUtensorMap& tw, const CUtensorMap& tx, const GemmEpi& ep, int K, int* status,
                       cudaStream_t s) {
    using L = GemmSmem<BN, STAGES>;
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemm_bf16_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            L::TOTAL));
        configured = true;
    }
    // with a reduce-scatter epilogue the grid also covers the padding rows of the last shard, so
    // that every owner sees the same number of arrivals
    const int t_cover = ep.rs != nullptr ? ep.rs_rows : ep.T;
    const int kb_all = (K + 63) / 64;
    const int splits = ep.ws != nullptr ? (kb_all + ep.kb_per_split - 1) / ep.kb_per_split : 1;
    dim3 grid((ep.N + 127) / 128, (t_cover + BN - 1) / BN, splits);
    TSB_CHECK_CUDA(tsb_launch(gemm_bf16_kernel<BN, STAGES>, grid, dim3(192), (size_t)L::TOTAL, s, tw, tx, ep, K, status));
    if (ep.ws != nullptr) {
        const long n = (long)ep.T * ep.N;
        TSB_CHECK_CUDA(tsb_launch(splitk_reduce_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, s, ep, splits));
    }
    return TSB_OK;
}

// W: [N, K] bf16 row-major (ldw elements per row); X: [T, K] bf16 (ldx); out: [T, ldo].
// `status` is a device int the kernel sets non-zero if one of its bounded waits gave up.
static int gemm_bf16_impl(const void* W, long ldw, const void* X, long ldx, void* out, long ldo, int out_f32,
                          const float* bias, const void* residual, int T, int N, int K, const void* rs, const void* ag, int shard,
                          int size, int rank, int* status, void* stream, void* splitk_ws, long splitk_ws_bytes);

extern "C" int tsb_gemm_bf16(const void* W, long ldw, const void* X, long ldx, void* out, long ldo, int out_f32,
                             const float* bias, const void* residual, int T, int N, int K, int* status, void* stream) {
    return gemm_bf16_impl(W, ldw, X, ldx, out, ldo, out_f32, bias, residual, T, N, K, nullptr, nullptr, 0, 1, 0, status, stream,
                          nullptr, 0);
}

// The plain GEMM with a caller-provided float32 workspace, which lets launches with few tiles and a long K split K.
extern "C" int tsb_gemm_bf16_ws(const void* W, long ldw, const void* X, long ldx, void* out, long ldo, int out_f32,
                                const float* bias, const void* residual, int T, int N, int K, int* status, void* stream,
                                void* ws, long ws_bytes) {
    return gemm_bf16_impl(W, ldw, X, ldx, out, ldo, out_f32, bias, residual, T, N, K, nullptr, nullptr, 0, 1, 0, status, stream,
                          ws, ws_bytes);
}

extern "C" int tsb_gemm_bf16_tp(const void* W, long ldw, const void* X, long ldx, void* out, long ldo, int out_f32,
                                const float* bias, const void* residual, int T, int N, int K, const void* rs,
                                const void* ag, int shard, int size, int rank, int* status, void* stream) {
    return gemm_bf16_impl(W, ldw, X, ldx, out, ldo, out_f32, bias, residual, T, N, K, rs, ag, shard, size, rank, status, stream,
                          nullptr, 0);
}

// The GEMM with the tensor-parallel prefill hooks: `rs` (device TpSeq*) sends the result to the token
// owners' accumulators instead of `out`; `ag` makes the producer wait for X's shards.  `shard` and
// `size` repeat the descriptor's values for the host-side launch arithmetic; the token tile is
// 128 rows so that it divides the shard.
static int gemm_bf16_impl(const void* W, long ldw, const void* X, long ldx, void* out, long ldo, int out_f32,
                          const float* bias, const void* residual, int T, int N, int K, const void* rs, const void* ag, int shard,
                          int size, int rank, int* status, void* stream, void* splitk_ws, long splitk_ws_bytes) {
    TSB_CHECK_ARG(T >= 0 && N > 0 && K > 0, "gemm_bf16: bad shape T=%d N=%d K=%d", T, N, K);
    TSB_CHECK_ARG((!rs && !ag) || (shard > 0 && shard % 128 == 0 && size >= 1), "gemm_bf16: shard=%d must be a multiple of 128", shard);
    TSB_CHECK_ARG(!rs || !residual, "gemm_bf16: reduce-scatter mode takes no residual");
    TSB_CHECK_ARG(K % 8 == 0 && ldw % 8 == 0 && ldx % 8 == 0, "gemm_bf16: K, ldw, ldx must be multiples of 8");
    TSB_CHECK_ARG(status != nullptr, "gemm_bf16: status word is required");
    if (T == 0) return TSB_OK;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaStream_t s = (cudaStream_t)stream;
    // more than 64 tokens: pairs of CTAs.  Below, the weights are all there is to read, one SM per 128 of their rows (and K split
    // over CTAs) reads them with more SMs than pairs of 256 rows would.
    if (!rs && !ag && T > 64) {
        const int pair_bn = choose_pair_bn(T, N, sms);
        const GemmEpi ep{out, bias, residual, ldo, T, N, out_f32, nullptr, nullptr, 0, 0};
        return launch_gemm_pair<false>(W, ldw, N, X, ldx, T, ep, K, pair_bn, (T + pair_bn - 1) / pair_bn, sms, status, s);
    }
    int bn = T <= 32 ? 32 : 64;
    if (rs || ag) bn = shard % 256 == 0 ? 256 : 128;          // a token tile must not straddle two shards
    // Reduce-scatter epilogues stall on NVLink stores; with 128-token tiles and a 3-deep ring two
    // CTAs fit on an SM, so one CTA's epilogue overlaps the other's main loop.
    static const int rs_small = []() { const char* e = getenv("TSB_TP_RS_TILE"); return e ? atoi(e) : 256; }();
    const bool two_per_sm = rs && rs_small == 128;
    if (two_per_sm) bn = 128;
    CUtensorMap tw, tx;
    int rc = tsb_make_tmap_2d_bf16(&tw, W, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, 128, 64);
    if (rc) return rc;
    rc = tsb_make_tmap_2d_bf16(&tx, X, (uint64_t)T, (uint64_t)K, (uint64_t)ldx, (uint32_t)bn, 64);
    if (rc) return rc;
    // Visit order of the token tiles.  all-gather -> GEMM starts with this rank's own shard (already
    // here) so that waiting for remote shards overlaps useful work; GEMM -> reduce-scatter starts with
    // the next rank's shard and ends with its own, so remote owners receive their tiles first.
    int rot = 0;
    if (ag) rot = rank * (shard / bn);
    if (rs) rot = ((rank + 1) % size) * (shard / bn);
    GemmEpi ep{out, bias, residual, ldo, T, N, out_f32, (const TpSeq*)rs, (const TpSeq*)ag, shard * size, rot};
    // Few tiles and a long K (decode batches): split K over CTAs so that the weight stream uses the whole GPU.
    if (!rs && !ag && splitk_ws != nullptr && bn <= 64) {
        const int tiles = ((N + 127) / 128) * ((T + bn - 1) / bn), kb_all = (K + 63) / 64;
        int want = sms / (tiles > 0 ? tiles : 1);
        if (want > 8) want = 8;
        if (want > kb_all / 4) want = kb_all / 4;
        if (want >= 2 && (long)want * T * N * 4 <= splitk_ws_bytes) {
            ep.kb_per_split = (kb_all + want - 1) / want;
            ep.ws = (float*)splitk_ws;
        }
    }
    // tensor-parallel GEMMs with more tiles than SMs: the persistent kernel (epilogue of a tile under the next tile's main loop)
    static const int persist_mode = []() { const char* e = getenv("TSB_GEMM_PERSISTENT"); return e ? atoi(e) : 1; }();
    if ((rs || ag) && persist_mode != 0 && !two_per_sm && (!rs || N % 8 == 0)) {
        const long tiles = (long)((N + 127) / 128) * (((rs ? shard * size : T) + bn - 1) / bn);
        if (tiles > sms || persist_mode == 2)
            return bn == 256 ? launch_gemm_persistent<256, 4>(tw, tx, ep, K, sms, status, s)
                             : launch_gemm_persistent<128, 6>(tw, tx, ep, K, sms, status, s);
    }
    switch (bn) {
    case 32: return launch_gemm<32, 8>(tw, tx, ep, K, status, s);
    case 64: return launch_gemm<64, 8>(tw, tx, ep, K, status, s);
    case 128: return two_per_sm ? launch_gemm<128, 3>(tw, tx, ep, K, status, s) : launch_gemm<128, 6>(tw, tx, ep, K, status, s);
    default: return launch_gemm<256, 4>(tw, tx, ep, K, status, s);
    }
}

// Grouped GEMM over a stack of matrices (mixture-of-experts prefill): W [E * N, K] bf16, X [P, K] bf16 with the rows of
// each group contiguous, `groups` a device list of `n_tiles` entries {matrix index or -1, first row, end row} whose
// tiles hold at most `bn` rows (32, 64 or a multiple of 16 up to 256).  out [P, ldo]; bias [E, N] or null.  Rows that no tile covers are
// left as they are.  The host passes only upper bounds (P, n_tiles): the list itself is built by device code.
extern "C" int tsb_gemm_bf16_grouped(const void* W, long ldw, int E, const void* X, long ldx, void* out, long ldo, int out_f32,
                                     const float* bias, int P, int N, int K, const int* groups, int n_tiles, int bn,
                                     int* status, void* stream) {
    TSB_CHECK_ARG(P >= 0 && N > 0 && K > 0 && E > 0 && n_tiles >= 0, "gemm_bf16_grouped: bad shape P=%d N=%d K=%d E=%d", P, N, K, E);
    TSB_CHECK_ARG(K % 8 == 0 && ldw % 8 == 0 && ldx % 8 == 0, "gemm_bf16_grouped: K, ldw, ldx must be multiples of 8");
    TSB_CHECK_ARG(bn == 32 || bn == 64 || (bn > 64 && bn <= 256 && bn % 16 == 0), "gemm_bf16_grouped: tile of %d rows", bn);
    TSB_CHECK_ARG(status != nullptr && groups != nullptr, "gemm_bf16_grouped: status word and tile list are required");
    if (P == 0 || n_tiles == 0) return TSB_OK;
    if (bn > 64) {
        int dev = 0, sms = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        GemmEpi pe{out, bias, nullptr, ldo, n_tiles * bn, N, out_f32, nullptr, nullptr, 0, 0, groups};
        return launch_gemm_pair<false>(W, ldw, (long)E * N, X, ldx, P, pe, K, bn, n_tiles, sms, status, (cudaStream_t)stream);
    }
    CUtensorMap tw, tx;
    int rc = tsb_make_tmap_2d_bf16(&tw, W, (uint64_t)E * N, (uint64_t)K, (uint64_t)ldw, 128, 64);
    if (rc) return rc;
    rc = tsb_make_tmap_2d_bf16(&tx, X, (uint64_t)P, (uint64_t)K, (uint64_t)ldx, (uint32_t)bn, 64);
    if (rc) return rc;
    GemmEpi ep{out, bias, nullptr, ldo, n_tiles * bn, N, out_f32, nullptr, nullptr, 0, 0, groups};
    cudaStream_t s = (cudaStream_t)stream;
    return bn == 32 ? launch_gemm<32, 8>(tw, tx, ep, K, status, s) : launch_gemm<64, 8>(tw, tx, ep, K, status, s);
}

// The gated products act(X G^T + bg, X U^T + bu) in one kernel: W [2 F, K] holds the F gate rows and then the F up rows (grouped: of
// every matrix), bias likewise or null, out bf16 [T, ldo].  `groups` null: a plain product of T > 64 rows; else the tile list of
// tsb_gemm_bf16_grouped over E matrices (N = 2 F rows each, bn above 64).  act: one of the gated activations.
extern "C" int tsb_gemm_bf16_glu(const void* W, long ldw, int E, const void* X, long ldx, void* out, long ldo, const float* bias, int T, int N, int K,
                                 int act, const int* groups, int n_tiles, int bn, int* status, void* stream) {
    TSB_CHECK_ARG(T >= 0 && N > 0 && N % 2 == 0 && K > 0 && E > 0, "gemm_bf16_glu: bad shape T=%d N=%d K=%d", T, N, K);
    TSB_CHECK_ARG(K % 8 == 0 && ldw % 8 == 0 && ldx % 8 == 0, "gemm_bf16_glu: K, ldw, ldx must be multiples of 8");
    TSB_CHECK_ARG(act >= ACT_SWIGLU && act <= ACT_SWIGLU_OAI, "gemm_bf16_glu: activation %d is not gated", act);
    TSB_CHECK_ARG(status != nullptr && (groups == nullptr ? E == 1 : n_tiles >= 0 && bn > 64 && bn <= 256 && bn % 16 == 0), "gemm_bf16_glu: tiles of %d rows", bn);
    if (T == 0 || (groups != nullptr && n_tiles == 0)) return TSB_OK;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (groups == nullptr) bn = choose_pair_bn(T, N, sms), n_tiles = (T + bn - 1) / bn;
    GemmEpi ep{out, bias, nullptr, ldo, groups != nullptr ? n_tiles * bn : T, N, 0, nullptr, nullptr, 0, 0, groups};
    ep.act = act;
    return launch_gemm_pair<true>(W, ldw, (long)E * N, X, ldx, T, ep, K, bn, n_tiles, sms, status, (cudaStream_t)stream);
}
