// Prompt attention on the 5th-generation tensor cores: flash attention over the paged bf16 cache, causal, with window,
// sinks, soft cap and per-head gate, head sizes 64, 128 and 256.
//
// Rows.  The query heads that share a KV head are packed: a tile of 128 accumulator rows is 128 / G tokens times G heads
// (G: the largest power of two that divides Hq / Hkv, at most 16), so a short prompt still fills the 128 lanes and a tile's
// causal and window edges are a few tokens wide instead of 128.  In memory those rows are consecutive: one TMA box.
//
// Scores go through two TMEM buffers that take turns over the key tiles: the next tile's scores are computed while this
// one's go through the softmax.  The MMA warp issues
//     S(0) S(1) | PV(0) S(2) | PV(1) S(3) | ...        (key tile u: buffer u & 1)
// P replaces S in place as bf16 (the A operand of PV comes from TMEM), O stays in TMEM until the end.
//
//   warps 0 .. 3 : softmax, one thread per row; rescales O itself, after the exponentials of the tile, whenever the maximum of one
//                  of the warp's rows has grown.  (P is rounded to bf16.  Relative to the running maximum the largest weights
//                  lie at or just below 1, where that costs least; relative to an older one, which would spare most of the
//                  rescaling, the error of the result was up to a fifth larger.)
//   warp 4       : TMA producer, K and V rings
//   warp 5       : TMEM owner, zeroes the V rows past the end of the cache, issues the MMAs
//
// What bounds it: the softmax's exponentials and issue slots beside the products; at one CTA per SM also the CTA's start and
// end (barriers, TMEM, first loads, output).  With 64-key tiles a CTA needs half of the SM's tensor memory and less than half
// of its shared memory, so two CTAs cover each other's gaps; with 128-key tiles one CTA has fewer hand-overs per key.
// Measured (us; mma.sync kernel of attention.cu / 128-key tiles / 64-key tiles), causal, 32 / 8 heads of 128: 2048 tokens
// 254 / 63 / 51, 8192 tokens 3111 / 655 / 562 (978 TFLOP/s), 1024 tokens 88 / 23 / 26, 555 tokens on 6100 cached ones
// 360 / 80 / 113; 64 / 8 heads of 64, 8 x 1024 tokens 433 / 276 / 182, with a window of 128 179 / 204 / 106; 16 / 2 heads of
// 256, 8192 tokens 4530 / - / 620.
#include "attn_args.cuh"
#include "tcgen05.cuh"

int tsb_make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_elems, const uint32_t* box);

namespace {

using namespace tc;

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
                   "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                   "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                   "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// K-major rows are described by make_desc_sw128; this is the other case, V as [key][128 bytes of columns]: the columns are the
// contiguous dimension, 64-column chunks lie chunk_bytes apart, groups of eight keys 1024 bytes.
__device__ __forceinline__ uint64_t make_desc_mn_sw128(uint32_t smem_addr, uint32_t chunk_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)((chunk_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const bf162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

template <int DH, int BN, int KS>
struct PrefillSmem {
    static constexpr int Q_BYTES = 128 * DH * 2;
    static constexpr int KV_BYTES = BN * DH * 2;               // one tile of K or of V
    static constexpr int BAR_OFF = Q_BYTES + 2 * KS * KV_BYTES;
    static constexpr int TOTAL = BAR_OFF + 256 + 1024;         // barriers, alignment slack
    static constexpr int COLS = 2 * BN + DH;                  // S buffers at columns 0 and BN, O behind them
    static constexpr int TMEM = COLS <= 256 ? 256 : 512;
    static constexpr int PER_SM = TMEM == 256 && TOTAL <= 113 * 1024 ? 2 : 1;
};

struct PrefillGeom {
    int G;             // heads packed into a row tile
    int tiles;         // token tiles of the longest sequence
    int subheads;      // Hq / G
};

template <int DH, int BN, int KS>
__global__ void __launch_bounds__(192, PrefillSmem<DH, BN, KS>::PER_SM) attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                           const __grid_constant__ CUtensorMap tmV, AttnArgs a, PrefillGeom geo, int* status) {
    using L = PrefillSmem<DH, BN, KS>;
    constexpr int CH = DH / 64;                  // 128-byte column chunks of a row
    constexpr int SUB = BN / 64;                 // 64-row loads of a tile
    constexpr uint32_t O_COL = 2 * BN;
    static_assert(L::COLS <= 512, "tensor memory");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* sK = smem + L::Q_BYTES;
    unsigned char* sV = sK + KS * L::KV_BYTES;
    uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + KS;
    uint64_t* v_full = k_empty + KS;
    uint64_t* v_empty = v_full + KS;
    uint64_t* s_full = v_empty + KS;             // [2] scores in buffer s complete
    uint64_t* p_full = s_full + 2;               // [2] P written in their place (one arrival per softmax warp)
    uint64_t* o_full = p_full + 2;               // [2] PV of buffer s complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int W_LOAD = 4, W_MMA = 5;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < KS; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 4);
            mbar_init(&o_full[s], 1);
        }
        fence_barrier_init();
    }
    if (warp == W_MMA) tmem_alloc<L::TMEM>(tmem_slot);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_trigger();

    // token tiles from the last (most keys under a causal mask) to the first, over all heads and sequences at each step
    const int per = geo.subheads * a.B;
    const int tile = geo.tiles - 1 - (int)(blockIdx.x / per), sub = (int)(blockIdx.x % per);
    const int hb = sub % geo.subheads, b = sub / geo.subheads;
    const int G = geo.G, rows_tok = 128 / G, h0 = hb * G, hk = h0 / (a.Hq / a.Hkv);
    const int q0 = a.cu_q[b], qlen = a.cu_q[b + 1] - q0, kvlen = a.kv_lens[b];
    const int tok0 = tile * rows_tok;
    const bool active = tok0 < qlen;
    const int pos0 = kvlen - qlen;
    const int tok_last = min(tok0 + rows_tok, qlen) - 1;
    const int j_hi = pos0 + tok_last + 1, j_lo = a.window > 0 ? max(0, pos0 + tok0 - a.window + 1) : 0;
    const int t_lo = j_lo / BN, nt = active ? (j_hi + BN - 1) / BN - t_lo : 0;      // key tiles t_lo .. t_lo + nt - 1

    if (warp == W_LOAD) {
        if (active) {
            if (lane == 0) {
                tma_prefetch_desc(&tmQ);
                tma_prefetch_desc(&tmK);
                tma_prefetch_desc(&tmV);
                mbar_expect_tx(q_full, L::Q_BYTES);
                for (int c = 0; c < CH; ++c) tma_load_3d(smem + c * 16384, &tmQ, q_full, c * 64, h0, q0 + tok0);
            }
            const int* table = a.block_table + (long)b * a.max_pages;
            const int n_sub = (j_hi + 63) / 64;                                     // 64-slot runs that exist
            int base = -64, slot_of = 0;                                             // lane i: first slot of run base + i
            int loaded[2] = {0, 0};                                                  // tiles of K and of V requested
            bool ok = true;
            // K runs one tile ahead of V: two score tiles are computed before the first PV
            for (int i = 0; i <= nt && ok; ++i) {
                for (int kv = 0; kv < 2 && ok; ++kv) {                               // K of tile i, V of tile i - 1
                    const int t = i - kv;
                    if (t < 0 || t >= nt) continue;
                    const int s = t % KS, run = (t_lo + t) * SUB, valid = min(SUB, n_sub - run);
                    if (run < base || run + SUB > base + 32) {
                        base = kv == 0 ? max(0, run - SUB) : run;
                        const int j = (base + lane) * 64;
                        slot_of = base + lane < n_sub ? table[j / a.page_size] * a.page_size + j % a.page_size : 0;
                    }
                    if (lane == 0) ok = mbar_wait(kv ? &v_empty[s] : &k_empty[s], ((t / KS) & 1) ^ 1);
                    ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
                    if (!ok) {
                        if (lane == 0) atomicExch(status, 11);
                        break;
                    }
                    uint64_t* bar = kv ? &v_full[s] : &k_full[s];
                    unsigned char* dst = (kv ? sV : sK) + s * L::KV_BYTES;
                    if (lane == 0) mbar_expect_tx(bar, valid * CH * 8192);
                    if (kv) loaded[1] = t + 1;
                    else loaded[0] = t + 1;
#pragma unroll
                    for (int r = 0; r < SUB; ++r) {
                        const int row = __shfl_sync(0xffffffffu, slot_of, run + r - base);
                        if (lane == 0 && r < valid)
                            for (int c = 0; c < CH; ++c) tma_load_2d(dst + c * BN * 128 + r * 8192, kv ? &tmV : &tmK, bar, hk * DH + c * 64, row);
                    }
                }
            }
            // The CTA leaves with no copy in flight, whichever warp gave up: the last tile of every stage has arrived (where nothing
            // went wrong the products read it already).
            if (lane == 0) {
                mbar_wait(q_full, 0);
                for (int t = max(0, loaded[0] - KS); t < loaded[0]; ++t) mbar_wait(&k_full[t % KS], (t / KS) & 1);
                for (int t = max(0, loaded[1] - KS); t < loaded[1]; ++t) mbar_wait(&v_full[t % KS], (t / KS) & 1);
            }
        }
        __syncwarp();
    } else if (warp == W_MMA) {
        if (active) {
            constexpr uint32_t idesc_s = make_idesc_bf16(128, BN);
            constexpr uint32_t idesc_o = make_idesc_bf16(128, DH) | (1u << 16);     // B (= V) with its columns contiguous
            bool ok = warp_wait(q_full, 0);
            int err = ok ? 0 : 12;
            auto scores = [&](int u) {
                const int s = u % KS;
                if (!warp_wait(&k_full[s], (u / KS) & 1)) { ok = false; err = 13; return; }
                fence_after_sync();
                if (lane == 0) {
                    const uint32_t qa = smem_u32(smem), ka = smem_u32(sK + s * L::KV_BYTES);
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        const uint64_t dq = make_desc_sw128(qa + c * 16384), dk = make_desc_sw128(ka + c * BN * 128);
#pragma unroll
                        for (int k = 0; k < 4; ++k) mma_f16_ss(tmem + (u & 1) * BN, dq + 2 * k, dk + 2 * k, idesc_s, (c | k) != 0);
                    }
                    mma_commit(&s_full[u & 1]);
                    mma_commit(&k_empty[s]);
                }
                __syncwarp();
            };
            if (ok) scores(0);
            if (ok && nt > 1) scores(1);
            for (int u = 0; u < nt && ok; ++u) {
                const int s = u % KS;
                if (!warp_wait(&v_full[s], (u / KS) & 1)) { ok = false; err = 14; break; }
                const int valid = min(kvlen, (j_hi + 63) / 64 * 64) - (t_lo + u) * BN;
                if (valid < BN) {
                    // keys past the end of the cache and runs that were not loaded have P = 0, but whatever lies in their
                    // V rows must be finite
                    const int c16 = CH * 8, n = (BN - valid) * c16;
                    for (int i = lane; i < n; i += 32) {
                        const int row = valid + i / c16, c = i % c16;
                        *reinterpret_cast<uint4*>(sV + s * L::KV_BYTES + (c >> 3) * BN * 128 + row * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    fence_proxy_async();
                    __syncwarp();
                }
                if (!warp_wait(&p_full[u & 1], (u >> 1) & 1)) { ok = false; err = 15; break; }
                fence_after_sync();
                if (lane == 0) {
                    const uint32_t va = smem_u32(sV + s * L::KV_BYTES);
#pragma unroll
                    for (int k = 0; k < BN / 16; ++k)
                        mma_f16_ts(tmem + O_COL, tmem + (u & 1) * BN + k * 8, make_desc_mn_sw128(va + k * 2048, BN * 128), idesc_o, (u | k) != 0);
                    mma_commit(&o_full[u & 1]);
                    mma_commit(&v_empty[s]);
                }
                __syncwarp();
                if (u + 2 < nt) scores(u + 2);
            }
            if (!ok && lane == 0) atomicExch(status, err);
        }
        __syncwarp();
    } else if (active) {
        const int quad = warp;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        const uint32_t t_o = tmem + lanes + O_COL;
        const int row = quad * 32 + lane, tok = tok0 + row / G, h = h0 + row % G;
        const int qp = pos0 + tok, qp_first = pos0 + tok0 + quad * 32 / G, qp_last = qp_first + (31 / G);
        constexpr float LOG2E = 1.4426950408889634f;
        const float f = a.softcap > 0.f ? 1.f : a.scale, fl = f * LOG2E;
        float ref = -INFINITY, sum = 0.f;                // the running maximum (scaled, times log2 e) and the row sum
        bool ok = true;
        for (int i = 0; i < nt; ++i) {
            const int buf = i & 1;
            if (!(ok = warp_wait(&s_full[buf], (i >> 1) & 1))) break;
            fence_after_sync();
            const uint32_t t_s = tmem + lanes + buf * BN;
            float s[BN];
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) tmem_ld32(t_s + c * 32, reinterpret_cast<uint32_t*>(s) + c * 32);
            tmem_ld_wait();
            if (a.softcap > 0.f) {
                const float inv_cap = a.scale / a.softcap;
#pragma unroll
                for (int j = 0; j < BN; ++j) s[j] = a.softcap * tanhf(s[j] * inv_cap);
            }
            const int j0 = (t_lo + i) * BN;
            // only tiles that touch the diagonal, the end of the cache or the window's edge compare (uniform per warp)
            if (j0 + BN - 1 > qp_first || j0 + BN > kvlen || (a.window > 0 && j0 <= qp_last - a.window)) {
                const int hi = min(qp, kvlen - 1) - j0, lo = a.window > 0 ? qp - a.window + 1 - j0 : 0;
#pragma unroll
                for (int j = 0; j < BN; ++j) s[j] = j <= hi && j >= lo ? s[j] : -INFINITY;
            }
            float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < BN; j += 4) {
#pragma unroll
                for (int e = 0; e < 4; ++e) m[e] = fmaxf(m[e], s[j + e]);
            }
            const float top = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])) * fl;
            float corr = 1.f;
            if (top > ref) {
                if (ref != -INFINITY) corr = ex2(ref - top);
                ref = top;                               // (from -inf: nothing summed yet, O is zero or not yet written)
                sum *= corr;
            }
            const float neg = ref == -INFINITY ? 0.f : -ref;
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t p[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float x = ex2(fmaf(s[c * 32 + 2 * j], fl, neg)), y = ex2(fmaf(s[c * 32 + 2 * j + 1], fl, neg));
                    part[(2 * j) & 3] += x;
                    part[(2 * j + 1) & 3] += y;
                    p[j] = pack2(x, y);
                }
                tmem_st16(t_s + c * 16, p);
            }
            sum += (part[0] + part[1]) + (part[2] + part[3]);
            if (i > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                // S(i) was issued after PV(i - 2), so of the products only PV(i - 1) can be outstanding
                if (!(ok = warp_wait(&o_full[(i - 1) & 1], ((i - 1) >> 1) & 1))) break;
                fence_after_sync();
#pragma unroll 1
                for (int c = 0; c < DH / 32; ++c) {
                    uint32_t o[32];
                    tmem_ld32(t_o + c * 32, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
                    tmem_st16(t_o + c * 32, o);
                    tmem_st16(t_o + c * 32 + 16, o + 16);
                }
            }
            tmem_st_wait();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[buf]);
        }
        if (ok && (ok = warp_wait(&o_full[(nt - 1) & 1], ((nt - 1) >> 1) & 1))) {
            fence_after_sync();
            float inv = sum > 0.f ? 1.f / sum : 0.f;
            if (a.sinks != nullptr) {
                const float sk = a.sinks[h] * LOG2E, mn = fmaxf(ref, sk);
                const float oc = ref == -INFINITY ? 0.f : ex2(ref - mn), ll = sum * oc + ex2(sk - mn);
                inv = ll > 0.f ? oc / ll : 0.f;
            }
            const bool mine = tok < qlen;
            if (a.gate != nullptr && mine) inv *= attn_gate(a, q0 + tok, h);
            bf16* dst = a.out + ((long)(q0 + tok) * a.Hq + h) * DH;
#pragma unroll 1
            for (int c = 0; c < DH / 32; ++c) {
                uint32_t o[32];
                tmem_ld32(t_o + c * 32, o);
                tmem_ld_wait();
                if (mine) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint4 v;
                        v.x = pack2(__uint_as_float(o[8 * j]) * inv, __uint_as_float(o[8 * j + 1]) * inv);
                        v.y = pack2(__uint_as_float(o[8 * j + 2]) * inv, __uint_as_float(o[8 * j + 3]) * inv);
                        v.z = pack2(__uint_as_float(o[8 * j + 4]) * inv, __uint_as_float(o[8 * j + 5]) * inv);
                        v.w = pack2(__uint_as_float(o[8 * j + 6]) * inv, __uint_as_float(o[8 * j + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c * 32 + j * 8) = v;
                    }
                }
            }
        } else if (lane == 0) {
            atomicExch(status, 16);
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == W_MMA) {
        fence_after_sync();
        tmem_dealloc<L::TMEM>(tmem);
    }
}

template <int DH, int BN, int KS>
int launch(const AttnArgs& a, int G, int max_q, long q_rows, long cache_rows, int* status, cudaStream_t s) {
    using L = PrefillSmem<DH, BN, KS>;
    static_assert(L::TOTAL <= 227 * 1024, "shared memory");
    auto kernel = attn_prefill_tc_kernel<DH, BN, KS>;
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
        configured = true;
    }
    CUtensorMap tq, tk, tv;
    const uint64_t qd[3] = {(uint64_t)DH, (uint64_t)a.Hq, (uint64_t)q_rows}, qs[2] = {(uint64_t)DH, (uint64_t)a.Hq * DH};
    const uint32_t qb[3] = {64, (uint32_t)G, (uint32_t)(128 / G)};
    int rc = tsb_make_tmap_bf16(&tq, a.q, 3, qd, qs, qb);
    if (rc) return rc;
    const uint64_t kd[2] = {(uint64_t)a.Hkv * DH, (uint64_t)cache_rows}, ks[1] = {(uint64_t)a.Hkv * DH};
    const uint32_t kb[2] = {64, 64};
    rc = tsb_make_tmap_bf16(&tk, a.k_cache, 2, kd, ks, kb);
    if (rc) return rc;
    rc = tsb_make_tmap_bf16(&tv, a.v_cache, 2, kd, ks, kb);
    if (rc) return rc;
    const PrefillGeom geo{G, (max_q + 128 / G - 1) / (128 / G), a.Hq / G};
    TSB_CHECK_CUDA(tsb_launch(kernel, dim3((unsigned)(geo.tiles * geo.subheads * a.B)), dim3(192), (size_t)L::TOTAL, s, tq, tk, tv, a, geo, status));
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

// Heads packed into a row tile: the largest power of two that divides Hq / Hkv, at most 16.
int packed_heads(const AttnArgs& a) {
    int G = 1;
    while (G < 16 && (a.Hq / a.Hkv) % (2 * G) == 0) G *= 2;
    return G;
}
long prefill_ctas(const AttnArgs& a, int max_q_len) {
    const int G = packed_heads(a);
    return (long)((max_q_len + 128 / G - 1) / (128 / G)) * (a.Hq / G) * a.B;
}

}  // namespace

// Whether tsb_attn_prefill_tc takes these arguments: one head size of 64, 128 or 256 and no form beyond window, sinks, soft cap
// and a gate per head; pages of a multiple of 64 slots, which the 64-row loads never straddle; and q, the caches and out on
// 16 bytes, which tensor maps and the 16-byte stores ask for (tsb_attn_prefill stores four bytes at a time).
// Left to tsb_attn_prefill are also the smallest prompts, whose time is a CTA's start and end (barriers and tensor memory here),
// and small grids with a soft cap at head size 64, where its CTAs of 64 rows spread the tanh over more SMs.  Measured (us,
// mma.sync / here): head size 64, up to 64 slots: 8 / 1 heads, 1 to 16 prompts 4.1 .. 5.0 / 5.1 .. 5.5, 32 prompts 5.7 .. 6.8 /
// 5.1 .. 5.5; one KV head per query head, 6 or 16 of them, 1 to 32 prompts 4.1 .. 9.9 / 5.0 .. 10.6; 64 / 8 heads, 4 prompts 5.6 .. 6.8 /
// 5.2 .. 5.5.  Soft cap, head size 64: 38 CTAs 22.0 / 25.5, 64 CTAs 34 / 41, 72 CTAs 10.7 / 10.7, 80 CTAs 27.6 / 26.0, 128 CTAs
// 50 / 41; head size 128, 64 slots 7.9 / 8.2.
// And at head size 64 with one head per row tile, up to 128 slots, where a tile of 128 rows stands against tiles of 64: prompts of 65 to
// 128 tokens while those smaller tiles still have an SM each (6, 10, 14, 16 or 32 heads, 65 tokens, up to 64 CTAs here 5.1 .. 5.3 /
// 5.5 .. 5.9, 128 tokens 5.8 .. 6.0 / 5.7 .. 6.4; 80 CTAs 6.3 / 5.9, 112 CTAs 7.3 / 6.1), and more than two CTAs per SM of at most 64 tokens, half
// of each tile empty (10 tokens on 90: 256 CTAs 7.9 / 6.4, 320 CTAs 8.1 / 10.6, 448 CTAs 11.4 / 11.6, 1024 CTAs 18.1 / 22.1).
extern "C" int tsb_attn_prefill_tc_takes(const AttnArgs* args, int max_q_len, long cache_rows) {
    const AttnArgs& a = *args;
    const uintptr_t all = reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k_cache) | reinterpret_cast<uintptr_t>(a.v_cache) |
                          reinterpret_cast<uintptr_t>(a.out);
    if (attn_needs_vd(a) || (a.Dh != 64 && a.Dh != 128 && a.Dh != 256) || a.q_pos0 != nullptr || a.lse_out != nullptr || a.page_size <= 0 ||
        a.page_size % 64 != 0 || cache_rows < 64 || (all & 15) != 0 || a.Hkv <= 0 || a.Hq % a.Hkv != 0)
        return 0;
    const bool tiny = (long)a.max_pages * a.page_size <= 64, few = (long)a.Hq * a.B < 256;
    if (a.Dh == 64) {
        const long ctas = prefill_ctas(a, max_q_len);
        const bool single = packed_heads(a) == 1, two_pages = (long)a.max_pages * a.page_size <= 128;
        if ((tiny && (few || single)) || (a.softcap > 0.f && ctas < 72)) return 0;
        if (single && two_pages && (max_q_len > 64 ? ctas <= 74 : ctas > 296)) return 0;
    }
    return !(a.Dh == 128 && a.softcap > 0.f && tiny && few);
}

// Prompt attention on tcgen05.  `q_rows`: packed query rows of q and out; `cache_rows`: slots of the K and V caches;
// `status`: device word that a bounded wait which gave up sets.  Everything else as tsb_attn_prefill.
extern "C" int tsb_attn_prefill_tc(const AttnArgs* args, int max_q_len, long q_rows, long cache_rows, int* status, void* stream) {
    const AttnArgs& a = *args;
    TSB_CHECK_ARG(a.Hkv > 0 && a.Hq % a.Hkv == 0, "attn_prefill_tc: Hq=%d not a multiple of Hkv=%d", a.Hq, a.Hkv);
    TSB_CHECK_ARG(a.cu_q != nullptr && status != nullptr, "attn_prefill_tc: cu_q and the status word are required");
    TSB_CHECK_ARG(tsb_attn_prefill_tc_takes(args, max_q_len, cache_rows), "attn_prefill_tc: head size %d, pages of %d slots in a cache of %ld, a form or an alignment that tsb_attn_prefill serves",
                  a.Dh, a.page_size, cache_rows);
    if (a.B == 0 || max_q_len == 0 || q_rows == 0) return TSB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int G = packed_heads(a);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // 64-key tiles and two CTAs per SM once there are CTAs for that, else 128-key tiles (times of both at the top); at head
    // size 64 the smaller tiles are ahead down to one CTA per SM.  They are also ahead where a row sees few keys, so that half
    // of a larger tile would lie behind the mask, and with a soft cap, whose tanh two CTAs overlap with the products (us, 128 /
    // 64): 32 / 8 heads of 128, 130 tokens 7.9 / 7.2, 1024 tokens in a window of 128 18.8 / 11.8, 1024 tokens capped 54 / 49; 8 / 1
    // heads of 64, 130 tokens 7.4 / 6.8; equal at 300 keys (10.3 / 10.4).
    const long ctas = prefill_ctas(a, max_q_len), slots = (long)a.max_pages * a.page_size;
    const bool small = a.softcap > 0.f || (a.window > 0 && a.window < slots ? a.window : slots) <= 256;
    switch (a.Dh) {
    case 64: return small || ctas > sms ? launch<64, 64, 4>(a, G, max_q_len, q_rows, cache_rows, status, s) : launch<64, 128, 4>(a, G, max_q_len, q_rows, cache_rows, status, s);
    case 128: return small || ctas > 2 * sms ? launch<128, 64, 2>(a, G, max_q_len, q_rows, cache_rows, status, s) : launch<128, 128, 2>(a, G, max_q_len, q_rows, cache_rows, status, s);
    default: return launch<256, 64, 2>(a, G, max_q_len, q_rows, cache_rows, status, s);
    }
}
