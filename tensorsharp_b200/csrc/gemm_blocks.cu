// Products of up to 64 rows (dispatched from two or three) with weights in GGUF blocks, on the 5th-generation tensor cores:
//   Y[t, n] = sum_k X[t, k] * W[n, k]  (+ bias[n]) (+ residual[t, n]), or the gated activation of two row halves of W,
// and the same for tiles of up to 64 rows of the experts of a mixture (gemm_experts below).
//
// So few rows are bound by the bytes of the weights, so the blocks themselves are read (0.56 bytes a weight in Q4_K where a
// bf16 copy has two) and never leave the SM in another form: a warp decodes them in registers and stores the bf16 values to
// tensor memory, which is where tcgen05.mma takes its first operand (128 weight rows) from.  Shared memory carries the blocks and
// the activations only, and a weight is decoded once for all rows.
//
//   warp 0      TMA of the blocks: 128 rows x 256 (MXFP4: 128) values a stage; the first stages of a dense product ahead of the
//               dependency wait
//   warp 1      tensor memory, products: slots of two slabs of 64 values of K, A from tensor memory, X from shared memory
//   warp 2      TMA of X, one slot at a time
//   warps 3-10  decode: two sets of four warps take the slots in turn, a thread owns one weight row (one lane of tensor
//               memory); they are the epilogue too
// Bound by what decoding issues, not by the bytes.  The first three warps sleep between their polls, of five instructions each (tc::hold; polling as
// tc::mbar_wait does they took half of the issue slots; one warp for all three is too slow a chain).  They run with all their lanes and
// elect one for what a single thread issues: with a branch on the lane the products took 620 cycles a slab to issue.
// Two CTAs fit an SM.  Dense products split K over the CTAs of a cluster, which add their parts through distributed shared
// memory in the order of K: no workspace, no second kernel.  Expert tiles run persistent, two accumulators in turn.
//
// Values are those that tsb_gather_rows writes (f32 arithmetic, rounded to bf16 once; a Q4_K value's offset is rounded at 2^-24 of 128
// scales ahead of that); MXFP4 values are exact in bf16.
//
// Measured, us per launch in a row (the bf16 copy through gemm_bf16_kernel, with its split-K and activation kernels / this one): Q4_K, 16 rows,
// 6144 x 2560 11.0 / 8.5, 2560 x 4096 9.6 / 6.6, 2 x 9728 x 2560 with SwiGLU 31.7 / 17.8 (18.7 from memory), 2560 x 9728 13.7 / 11.0, 1024 x 2560 5.9 / 5.6; 64 rows 13.6 /
// 10.9, 11.5 / 8.6, 35.1 / 23.3, 15.7 / 13.3, 7.8 / 7.9; Q6_K, 16 rows, 32768 x 2560 32.3 / 22.9; Q8_0, 16 rows, 5376 x 21504 41.8 / 27.5.  A layer of 32
// MXFP4 experts of 2880 x 2880 with its routing (the int8 kernels of moe.cu / this one): 68 pairs 185 / 166, 256 254 / 194, 512 386 / 200, 1024 620 / 237.
#include <cudaTypedefs.h>
#include <mutex>
#include "glu.cuh"
#include "quant_blocks.cuh"
#include "tcgen05.cuh"

int tsb_make_tmap_bytes(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows, uint32_t box_bytes);

namespace {
using namespace tc;

struct BlockGemmArgs {
    void* out;                // [T, ldo] (experts: rows in expert order)
    const float* bias;        // [N] (experts: [E, N]) or null
    const void* residual;     // as out, or null
    const float* row_scale;   // experts: [rows] or null
    const uint8_t* scales;    // MXFP4: [rows][K / 32]
    const uint16_t* d;        // Q6_K: half [rows][K / 256]
    const int4* tiles;        // experts: {expert, first row, rows}
    const int* meta;          // experts: meta[0] = number of tiles
    long ldo;
    int T, N, n_out, K;       // N: weight rows of a matrix, n_out = N or (gated) N / 2
    int out_f32, act;
    int m_tiles, per;         // feature tiles; stages of a CTA's part of K (dense)
};

template <int TYPE> struct Blocks;
template <> struct Blocks<TSB_Q4_K> { static constexpr int SLABS = 4, BYTES = 128 * 144; };
template <> struct Blocks<TSB_Q6_K> { static constexpr int SLABS = 4, BYTES = 128 * (128 + 64 + 16); };
template <> struct Blocks<TSB_Q8_0> { static constexpr int SLABS = 4, BYTES = 128 * (256 + 16); };
template <> struct Blocks<TSB_MXFP4> { static constexpr int SLABS = 2, BYTES = 128 * 64; };

constexpr int BG_THREADS = 352;
constexpr int BG_SMEM = 113 * 1024;                     // of a CTA: two on an SM

template <int TYPE, int NT, bool GLU, bool EXPERTS>
struct Shape {
    static constexpr int SLABS = Blocks<TYPE>::SLABS, RAW = Blocks<TYPE>::BYTES, X = 2 * NT * 128;
    static constexpr int AS = NT == 64 ? 2 : 3;         // slots of A (64 columns each)
    static constexpr int XS = NT <= 32 ? 4 : TYPE == TSB_Q8_0 ? 2 : 3;                           // slots of X
    static constexpr int STAGE_OUT = GLU && EXPERTS ? 2 * 16 * 128 * 4 : 0;
    static constexpr int fixed(int strip) { return XS * X + STAGE_OUT + 2 * strip + 512 + 1024; }
    static_assert(2 * NT + AS * 64 <= 256, "tensor memory of two CTAs");
    // stages of blocks; `strip`: bytes of the scales of a tile (MXFP4)
    static constexpr int stages(int strip) {
        const int n = (BG_SMEM - fixed(strip)) / RAW;
        return n > 6 ? 6 : n;
    }
};

// ---- two f32 values in one register pair ----
__device__ __forceinline__ uint64_t pair(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint32_t round2(uint64_t v) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    const bf162 h = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Bytes become floats on both of the pipes that have an instruction for it, each with 64 lanes a cycle: a permutation (ALU) puts a
// byte into the mantissa of 128 or 2^15, a dot product with one (FMA) adds it to the bits of 2^23.  With permutations alone the ALU was
// the bound: 1120 cycles for four warps with a slab of Q4_K each, 820 with half of them.
__device__ __forceinline__ uint64_t bytes_128(uint32_t v, int i) {                       // 128 + byte (below 128)
    return pair(__uint_as_float(__byte_perm(v, 0x43000000u, 0x7044u | i << 8)), __uint_as_float(__byte_perm(v, 0x43000000u, 0x7044u | (i + 1) << 8)));
}
__device__ __forceinline__ uint64_t bytes_32768(uint32_t v, int i) {                     // 2^15 + byte
    return pair(__uint_as_float(__byte_perm(v, 0x47000000u, 0x7404u | i << 4)), __uint_as_float(__byte_perm(v, 0x47000000u, 0x7404u | (i + 1) << 4)));
}
__device__ __forceinline__ uint64_t bytes_less(uint32_t v, int i, float less) {          // byte - less, exact
    return add2(pair(__uint_as_float(__dp4a(v, 1u << (8 * i), 0x4B000000u)), __uint_as_float(__dp4a(v, 256u << (8 * i), 0x4B000000u))),
                pair(-8388608.f - less, -8388608.f - less));
}
__device__ __forceinline__ uint64_t signed_bytes(uint32_t v, int i) {
    return add2(pair(__int_as_float(__dp4a((int)v, 1 << (8 * i), 0x4B400000)), __int_as_float(__dp4a((int)v, 256 << (8 * i), 0x4B400000))),
                pair(-12582912.f, -12582912.f));                                         // 2^23 + 2^22
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
                   "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
                   "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ float ld_peer(const float* p, uint32_t rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_rank(p, rank)) : "memory");
    return v;
}
// A barrier of the 128 threads that name `id`, which also tells each whether the predicate held for all of them.
__device__ __forceinline__ bool bar_all128(int id, bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)ok), "r"(id) : "memory");
    return r != 0;
}

// ---- blocks of a stage: 128 rows (gated: 64 of each half), column s (stages) of the matrix ----
template <int TYPE, bool GLU>
__device__ __forceinline__ void load_blocks(unsigned char* raw, const CUtensorMap* m0, const CUtensorMap* m1, const CUtensorMap* m2, uint64_t* bar, int s,
                                            int row, int n_out) {
#pragma unroll
    for (int h = 0; h < (GLU ? 2 : 1); ++h) {
        const int r = row + h * n_out;
        if (TYPE == TSB_Q4_K) tma_load_2d(raw + h * 64 * 144, m0, bar, s * 144, r);
        if (TYPE == TSB_Q6_K) {
            tma_load_2d(raw + h * 64 * 128, m0, bar, s * 128, r);
            tma_load_2d(raw + 128 * 128 + h * 64 * 64, m1, bar, s * 64, r);
            tma_load_2d(raw + 128 * 192 + h * 64 * 16, m2, bar, s * 16, r);
        }
        if (TYPE == TSB_Q8_0) {
            tma_load_2d(raw + h * 64 * 128, m0, bar, s * 256, r);
            tma_load_2d(raw + 128 * 128 + h * 64 * 128, m0, bar, s * 256 + 128, r);
            tma_load_2d(raw + 128 * 256 + h * 64 * 16, m1, bar, s * 16, r);
        }
        if (TYPE == TSB_MXFP4) tma_load_2d(raw + h * 64 * 64, m0, bar, s * 64, r);
    }
}

// 64 values of row r of a stage (slab c of it) as 32 pairs of bf16.  `side`: the row's d of the block (Q6_K), its two scale
// bytes (MXFP4).
template <int TYPE>
__device__ __forceinline__ void decode_slab(const unsigned char* raw, int r, int c, uint32_t side, uint32_t (&o)[32]) {
    if constexpr (TYPE == TSB_Q4_K) {
        const unsigned char* b = raw + r * 144;
        const uint4 h = *reinterpret_cast<const uint4*>(b);
        // six-bit scales and offsets of the sub-blocks 2 c and 2 c + 1
        uint32_t s, m;
        if (c < 2) {
            s = (h.y >> (16 * c)) & 0x3F3Fu;
            m = (h.z >> (16 * c)) & 0x3F3Fu;
        } else {
            const int sh = 16 * (c - 2);
            const uint32_t lo = h.w >> sh;
            s = (lo & 0x0F0Fu) | (((h.y >> sh) >> 2) & 0x3030u);
            m = ((lo >> 4) & 0x0F0Fu) | (((h.z >> sh) >> 2) & 0x3030u);
        }
        const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(&h.x));
        const float s0 = dd.x * (float)(s & 255u), s1 = dd.x * (float)(s >> 8);
        const float m0 = -(dd.y * (float)(m & 255u)), m1 = -(dd.y * (float)(m >> 8)), c0 = fmaf(-128.f, s0, m0), c1 = fmaf(-128.f, s1, m1);
        const uint64_t S0 = pair(s0, s0), S1 = pair(s1, s1), M0 = pair(m0, m0), M1 = pair(m1, m1), C0 = pair(c0, c0), C1 = pair(c1, c1);
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const uint4 q4 = *reinterpret_cast<const uint4*>(b + 16 + c * 32 + v * 16);
            const uint32_t q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t lo = q[i] & 0x0F0F0F0Fu, hi = (q[i] >> 4) & 0x0F0F0F0Fu;
                o[v * 8 + i * 2] = round2(fma2(bytes_128(lo, 0), S0, C0));
                o[v * 8 + i * 2 + 1] = round2(fma2(bytes_less(lo, 2, 0.f), S0, M0));
                o[16 + v * 8 + i * 2] = round2(fma2(bytes_less(hi, 0, 0.f), S1, M1));
                o[16 + v * 8 + i * 2 + 1] = round2(fma2(bytes_128(hi, 2), S1, C1));
            }
        }
    } else if constexpr (TYPE == TSB_Q6_K) {
        const int n = c >> 1, kk = c & 1;                       // half of the block; which nibbles and bit pairs
        const float d = h2f_bits((uint16_t)side);
        const uint32_t sc = *reinterpret_cast<const uint32_t*>(raw + 128 * 192 + r * 16 + 8 * n + 4 * kk);
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const uint4 h4 = *reinterpret_cast<const uint4*>(raw + 128 * 128 + r * 64 + (((2 * n + v) ^ ((r >> 1) & 3)) << 4));
            const uint32_t hq[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint4 l4 = *reinterpret_cast<const uint4*>(raw + r * 128 + (((4 * n + 2 * e + v) ^ (r & 7)) << 4));
                const uint32_t lq[4] = {l4.x, l4.y, l4.z, l4.w};
                const float s = d * (float)(int8_t)(sc >> (16 * e + 8 * v));
                const uint64_t S = pair(s, s), M = pair(-160.f * s, -160.f * s);                // 128 + 32; exact: 19 bits of s
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t two = (hq[i] >> (4 * kk)) >> (2 * e);
                    const uint32_t q = ((lq[i] >> (4 * kk)) & 0x0F0F0F0Fu) | ((two * 16u) & 0x30303030u);
                    o[e * 16 + v * 8 + i * 2] = round2(i & 1 ? mul2(bytes_less(q, 0, 32.f), S) : fma2(bytes_128(q, 0), S, M));
                    o[e * 16 + v * 8 + i * 2 + 1] = round2(mul2(bytes_less(q, 2, 32.f), S));
                }
            }
        }
    } else if constexpr (TYPE == TSB_Q8_0) {
        const uint32_t d2 = *reinterpret_cast<const uint32_t*>(raw + 128 * 256 + r * 16 + c * 4);
        const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(&d2));
        const unsigned char* b = raw + (c >> 1) * (128 * 128) + r * 128;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const uint4 q4 = *reinterpret_cast<const uint4*>(b + ((((c & 1) * 4 + v) ^ (r & 7)) << 4));
            const uint32_t q[4] = {q4.x, q4.y, q4.z, q4.w};
            const float s = v < 2 ? dd.x : dd.y;
            const uint64_t S = pair(s, s), M = pair(-32896.f * s, -32896.f * s);          // 2^15 + 128; exact: 11 bits of s, 9 of the factor
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                o[v * 8 + i * 2] = round2(fma2(bytes_32768(q[i] ^ 0x80808080u, 0), S, M));
                o[v * 8 + i * 2 + 1] = round2(mul2(signed_bytes(q[i], 2), S));
            }
        }
    } else {
        // A code's sign at bit 15 and its three other bits at 8 .. 6 are a bf16 that is 2^-126 times the value, subnormal
        // ones too; times 2^(e - 1), in two steps where that is beyond bf16.
        const int e[2] = {(int)(side & 255u), (int)(side >> 8)};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t f = (uint32_t)min(e[u] + 126, 254) << 7;                           // 2^(min(e - 1, 127))
            const uint32_t ff = f | (f << 16);
            const bf162 scale = *reinterpret_cast<const bf162*>(&ff);
            const uint4 q4 = *reinterpret_cast<const uint4*>(raw + r * 64 + (((2 * c + u) ^ ((r >> 1) & 3)) << 4));
            const uint32_t q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t nib[2] = {q[i] & 0x0F0F0F0Fu, (q[i] >> 4) & 0x0F0F0F0Fu};
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t v = (__byte_perm(nib[n], 0, j ? 0x4342u : 0x4140u) * 0x1040u) & 0x81C081C0u;
                        const bf162 x = __hmul2(*reinterpret_cast<const bf162*>(&v), scale);
                        o[u * 16 + n * 8 + i * 2 + j] = *reinterpret_cast<const uint32_t*>(&x);
                    }
            }
        }
        if (__any_sync(0xffffffffu, e[0] > 128 || e[1] > 128)) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t g = (uint32_t)max(e[u] - 1, 127) << 7;                         // 2^(max(e - 128, 0))
                const uint32_t gg = g | (g << 16);
                const bf162 rest = *reinterpret_cast<const bf162*>(&gg);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const bf162 x = __hmul2(*reinterpret_cast<const bf162*>(&o[u * 16 + i]), rest);
                    o[u * 16 + i] = *reinterpret_cast<const uint32_t*>(&x);
                }
            }
        }
    }
}

template <int TYPE, int NT, bool GLU, bool EXPERTS>
__global__ void __launch_bounds__(BG_THREADS, 2) gemm_blocks_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
                                                                    const __grid_constant__ CUtensorMap tm2, const __grid_constant__ CUtensorMap tmX,
                                                                    BlockGemmArgs a, int stages, int strip, int splits, int* status) {
    using L = Shape<TYPE, NT, GLU, EXPERTS>;
    constexpr int SLABS = L::SLABS, AS = L::AS, XS = L::XS, ROWS = GLU ? 64 : 128;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* sX = smem_raw + (-smem_u32(smem_raw) & 1023u);         // an offset, not a cast: loads stay loads from shared memory
    unsigned char* ring = sX + XS * L::X;                                 // [stages][RAW]
    float* stage_out = reinterpret_cast<float*>(ring + stages * L::RAW);
    unsigned char* strips = ring + stages * L::RAW + L::STAGE_OUT;        // [2][strip]
    uint64_t* full = reinterpret_cast<uint64_t*>(strips + 2 * strip);     // [6]
    uint64_t* empty = full + 6;                                           // [6] one arrival per warp that reads a stage
    uint64_t* x_full = empty + 6;                                         // [4]
    uint64_t* x_empty = x_full + 4;                                       // [4] the products that read a slot of X have ended
    uint64_t* a_full = x_empty + 4;                                       // [3] one arrival per warp of a set
    uint64_t* a_empty = a_full + 3;                                       // [3] the products that read a slot of A have ended
    uint64_t* acc_full = a_empty + 3;                                     // [2]
    uint64_t* acc_empty = acc_full + 2;                                   // [2]
    uint64_t* s_full = acc_empty + 2;                                     // [2] scales of a tile
    uint64_t* s_empty = s_full + 2;                                       // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slabs_all = (a.K + 63) >> 6, stages_all = (slabs_all + SLABS - 1) / SLABS;
    constexpr int READERS = SLABS == 4 ? 8 : 4;                           // warps that read a stage
    const int rank = EXPERTS ? 0 : (int)blockIdx.x % splits;

    if (warp == 2 && lane < 4) tma_prefetch_desc(lane == 0 ? &tm0 : lane == 1 ? &tm1 : lane == 2 ? &tm2 : &tmX);
    if (threadIdx.x == 0) {
        for (int i = 0; i < 6; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], READERS);
        }
        for (int i = 0; i < XS; ++i) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], 1);
        }
        for (int i = 0; i < AS; ++i) {
            mbar_init(&a_full[i], 4);
            mbar_init(&a_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 4);
            mbar_init(&s_full[i], 1);
            mbar_init(&s_empty[i], 8);
        }
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<256>(tmem_slot);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + 2 * NT;

    // What there is to do: dense, one tile and a part of K; experts, every gridDim.x-th (tile of rows, feature tile).
    struct Unit { int m, group, row0, rows, first, n; };                  // first, n: stages
    auto unit = [&](int u) {
        Unit w;
        if (EXPERTS) {
            const int4 t = a.tiles[u / a.m_tiles];
            w.m = u % a.m_tiles, w.group = t.x, w.row0 = t.y, w.rows = t.z, w.first = 0, w.n = stages_all;
        } else {
            w.m = (int)blockIdx.x / splits, w.group = 0, w.row0 = 0, w.rows = a.T, w.first = rank * a.per;
            w.n = min(a.per, stages_all - w.first);
        }
        return w;
    };
    // the weights are nobody's output: a dense product asks for its first stages before it waits for the kernel ahead
    int early = 0;
    if (!EXPERTS && warp == 0) {
        const Unit w = unit(0);
        early = min(stages, w.n);
        if (elect_one())
            for (int i = 0; i < early; ++i) {
                mbar_expect_tx(&full[i], L::RAW);
                load_blocks<TYPE, GLU>(ring + i * L::RAW, &tm0, &tm1, &tm2, &full[i], w.first + i, w.m * ROWS, a.n_out);
            }
        __syncwarp();
    }
    // dense: only X, the residual and the output belong to the kernel ahead, so blocks are read and decoded while it ends
    if (EXPERTS || warp == 2) {
        pdl_wait();
        pdl_trigger();
    }
    const int units = EXPERTS ? a.meta[0] * a.m_tiles : 1, step = EXPERTS ? (int)gridDim.x : 1, first_unit = EXPERTS ? (int)blockIdx.x : 0;

    if (warp == 0) {
        int j = 0, it = 0, at = 0;
        uint32_t ph = 1;
        bool ok = true;
        for (int u = first_unit; u < units && ok; u += step, ++j) {
            const Unit w = unit(u);
            const int row = w.group * a.N + w.m * ROWS;
            if (TYPE == TSB_MXFP4) {
                const int kb = a.K >> 5, have = min(ROWS, a.n_out - w.m * ROWS);
                ok = hold<true>(&s_empty[j & 1], ((j >> 1) & 1) ^ 1);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(&s_full[j & 1], (GLU ? 2 : 1) * have * kb);
                    for (int h = 0; h < (GLU ? 2 : 1); ++h)
                        bulk_load(strips + (j & 1) * strip + h * 64 * kb, a.scales + (long)(row + h * a.n_out) * kb, have * kb, &s_full[j & 1]);
                }
                __syncwarp();
            }
            for (int s = 0; s < w.n; ++s, ++it) {
                if (it >= early) {
                    ok = ok && hold<true>(&empty[at], ph);
                    if (!ok) break;
                    if (elect_one()) {
                        mbar_expect_tx(&full[at], L::RAW);
                        load_blocks<TYPE, GLU>(ring + at * L::RAW, &tm0, &tm1, &tm2, &full[at], w.first + s, row, a.n_out);
                    }
                    __syncwarp();
                }
                if (++at == stages) at = 0, ph ^= 1;
            }
        }
        if (!ok && lane == 0) atomicExch(status, 1);
        // no copy is in flight when the CTA leaves, whichever wait gave up (unless it takes longer than a wait's limit)
        bool given_up = false;
        for (int i = max(0, it - stages); i < it; ++i) settle(&full[i % stages], (i / stages) & 1, given_up);
        if (TYPE == TSB_MXFP4)
            for (int i = max(0, j - 2); i < j; ++i) settle(&s_full[i & 1], (i >> 1) & 1, given_up);
    } else if (warp == 2) {
        int it = 0, at = 0;
        uint32_t ph = 1;
        bool ok = true;
        for (int u = first_unit; u < units && ok; u += step) {
            const Unit w = unit(u);
            const int k0 = w.first * SLABS, k1 = min(slabs_all, (w.first + w.n) * SLABS);
            for (int k = k0; k < k1; k += 2, ++it) {
                ok = hold<true>(&x_empty[at], ph);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(&x_full[at], k + 1 < k1 ? L::X : L::X / 2);
                    tma_load_2d(sX + at * L::X, &tmX, &x_full[at], k * 64, w.row0);
                    if (k + 1 < k1) tma_load_2d(sX + at * L::X + L::X / 2, &tmX, &x_full[at], k * 64 + 64, w.row0);
                }
                __syncwarp();
                if (++at == XS) at = 0, ph ^= 1;
            }
        }
        if (!ok && lane == 0) atomicExch(status, 1);
        bool given_up = false;
        for (int i = max(0, it - XS); i < it; ++i) settle(&x_full[i % XS], (i / XS) & 1, given_up);
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc_bf16(128, NT);
        const uint64_t dx = make_desc_sw128(smem_u32(sX));
        int at = 0, xat = 0, j = 0;
        uint32_t ph = 0, xph = 0;
        bool ok = true;
        for (int u = first_unit; u < units && ok; u += step, ++j) {
            const Unit w = unit(u);
            const int n = min(slabs_all, (w.first + w.n) * SLABS) - w.first * SLABS;
            const uint32_t acc = tmem + (j & 1) * NT;
            ok = hold(&acc_empty[j & 1], ((j >> 1) & 1) ^ 1);
            for (int k = 0; k < n; k += 2) {
                ok = ok && hold<true>(&a_full[at], ph) && hold(&x_full[xat], xph);
                if (!ok) break;
                fence_after_sync();
                if (elect_one()) {
                    const uint32_t as = tmem_a + at * 64;
                    const uint64_t xs = dx + (uint64_t)(xat * (L::X >> 4));
                    mma_ts(acc, as, xs, idesc, k != 0);
#pragma unroll
                    for (int i = 1; i < 4; ++i) mma_ts(acc, as + i * 8, xs + 2 * i, idesc, 1);
                    if (k + 1 < n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) mma_ts(acc, as + 32 + i * 8, xs + (L::X >> 5) + 2 * i, idesc, 1);
                    mma_commit(&a_empty[at]);
                    mma_commit(&x_empty[xat]);
                    if (k + 2 >= n) mma_commit(&acc_full[j & 1]);
                }
                __syncwarp();
                if (++at == AS) at = 0, ph ^= 1;
                if (++xat == XS) xat = 0, xph ^= 1;
            }
        }
        if (!ok && lane == 0) atomicExch(status, 2);
    } else {
        const int q = warp & 3, set = (warp - 3) >> 2, r = q * 32 + lane;
        const uint32_t quad = (uint32_t)(q * 32) << 16;
        const int kb = a.K >> 5;
        // Of the slots, and where a stage is one slot of the stages, every second one is this set's: its next places and their phases.
        constexpr int STEP = SLABS == 4 ? 1 : 2;
        int j = 0, turn = 0, my_stage = STEP == 2 ? set : 0, my_slot = set;
        uint32_t stage_ph = 0, slot_ph = 1;
        if (my_slot >= AS) my_slot -= AS, slot_ph ^= 1;
        bool ok = true;
        Unit before;
        // experts: the result of tile jj, by the set whose turn it is, while the other one goes on decoding
        auto result = [&](const Unit& w, int jj) {
            if ((jj & 1) != set) return;
            ok = ok && hold(&acc_full[jj & 1], (jj >> 1) & 1);
            if (!ok && lane == 0) atomicExch(status, 3);
            if (GLU) ok = bar_all128(1 + set, ok);
            if (!ok) return;
            fence_after_sync();
            const int f = w.m * ROWS + (GLU ? (q & 1) * 32 + lane : r);
            const bool mine = f < a.n_out;
            const float bias = a.bias && mine ? a.bias[(long)w.group * a.N + f + (GLU && q >= 2 ? a.n_out : 0)] : 0.f;
            float* so = stage_out + set * (16 * 128);
#pragma unroll 1
            for (int c = 0; c * 16 < w.rows; ++c) {
                uint32_t v[16];
                tmem_ld16(tmem + quad + (jj & 1) * NT + c * 16, v);
                tmem_ld_wait();
                if (GLU) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) so[i * 128 + r] = __uint_as_float(v[i]) + bias;
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
                    const int t0 = (q >> 1) * 8;                          // this thread: one feature, eight rows
                    if (mine)
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int t = c * 16 + t0 + i;
                            if (t < w.rows) {
                                const float g = so[(t0 + i) * 128 + (q & 1) * 32 + lane], up = so[(t0 + i) * 128 + 64 + (q & 1) * 32 + lane];
                                float y = act_glu(a.act, g, up);
                                if (a.row_scale) y *= a.row_scale[w.row0 + t];
                                const long at = (long)(w.row0 + t) * a.ldo + f;
                                if (a.out_f32) reinterpret_cast<float*>(a.out)[at] = y;
                                else reinterpret_cast<bf16*>(a.out)[at] = f2bf(y);
                            }
                        }
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
                } else if (mine) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int t = c * 16 + i;
                        if (t < w.rows) {
                            float y = __uint_as_float(v[i]) + bias;
                            if (a.act == ACT_RELU2) y = fmaxf(y, 0.f), y *= y;
                            else if (a.act == ACT_SILU) y = y / (1.f + __expf(-y));
                            if (a.row_scale) y *= a.row_scale[w.row0 + t];
                            const long at = (long)(w.row0 + t) * a.ldo + f;
                            if (a.out_f32) reinterpret_cast<float*>(a.out)[at] = y;
                            else reinterpret_cast<bf16*>(a.out)[at] = f2bf(y);
                        }
                    }
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[jj & 1]);
        };
        for (int u = first_unit; u < units; u += step, ++j) {
            const Unit w = unit(u);
            const int n = min(slabs_all, (w.first + w.n) * SLABS) - w.first * SLABS;
            const int wr = w.m * ROWS + (GLU ? (r < 64 ? min(r, a.n_out - 1 - w.m * ROWS) : a.n_out + min(r - 64, a.n_out - 1 - w.m * ROWS))
                                             : min(r, a.n_out - 1 - w.m * ROWS));
            const uint16_t* dp = TYPE == TSB_Q6_K ? a.d + (long)(w.group * a.N + wr) * (a.K >> 8) + w.first : nullptr;
            const unsigned char* sp = strips + (j & 1) * strip + (GLU && r >= 64 ? 64 * kb + (r - 64) * kb : r * kb);
            uint32_t side = TYPE == TSB_Q6_K ? dp[0] : 0;
            if (TYPE == TSB_MXFP4) ok = ok && hold(&s_full[j & 1], (j >> 1) & 1);
            bool first = true;
            for (int s = STEP == 2 ? turn ^ set : 0; s < w.n; s += STEP) {
                uint32_t ahead = 0;
                if (TYPE == TSB_Q6_K && s + 1 < w.n) ahead = dp[s + 1];
                const unsigned char* raw = ring + my_stage * L::RAW;
                ok = ok && hold(&full[my_stage], stage_ph);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = SLABS == 4 ? 2 * set + h : h;
                    if (TYPE == TSB_MXFP4) {
                        if (s * SLABS + c >= n) break;
                        const int u = 2 * (s * SLABS + c);
                        side = sp[u] | (u + 1 < kb ? (uint32_t)sp[u + 1] << 8 : 0u);
                    }
                    uint32_t o[32];
                    decode_slab<TYPE>(raw, r, c, side, o);
                    if (h == 0) {
                        ok = ok && hold(&a_empty[my_slot], slot_ph);
                        fence_after_sync();
                    }
                    if (ok) tmem_st32(tmem_a + quad + my_slot * 64 + h * 32, o);
                }
                tmem_st_wait();
                fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&empty[my_stage]);
                    if (ok) mbar_arrive(&a_full[my_slot]);
                }
                if (TYPE == TSB_Q6_K) side = ahead;
                my_stage += STEP;
                if (my_stage >= stages) my_stage -= stages, stage_ph ^= 1;
                my_slot += 2;
                if (my_slot >= AS) my_slot -= AS, slot_ph ^= 1;
                if (EXPERTS && first && j > 0) result(before, j - 1);
                first = false;
            }
            if (EXPERTS && first && j > 0) result(before, j - 1);         // no slot of this unit was this set's
            turn ^= w.n & 1;
            if (TYPE == TSB_MXFP4) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty[j & 1]);
            }
            before = w;
        }
        if (EXPERTS) {
            if (j > 0) result(before, j - 1);
        } else {
            // this CTA's part, [token][128 rows], over the ring (every copy has been read)
            ok = ok && hold(&acc_full[0], 0);
            if (!ok && lane == 0) atomicExch(status, 3);
            if (ok) {
                fence_after_sync();
                float* part = reinterpret_cast<float*>(ring);
#pragma unroll 1
                for (int c = set; c * 16 < a.T; c += 2) {
                    uint32_t v[16];
                    tmem_ld16(tmem + quad + c * 16, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) part[(c * 16 + i) * 128 + r] = __uint_as_float(v[i]);
                }
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (!EXPERTS) {
        pdl_wait();
        if (splits > 1) cluster_sync();
        const float* part = reinterpret_cast<const float*>(ring);
        const int m = (int)blockIdx.x / splits;
        for (int i = rank * BG_THREADS + threadIdx.x; i < a.T * ROWS; i += splits * BG_THREADS) {
            const int t = i / ROWS, f = i % ROWS, n = m * ROWS + f;
            if (n >= a.n_out) continue;
            float v = a.bias ? a.bias[n] : 0.f, up = GLU && a.bias ? a.bias[n + a.n_out] : 0.f;
            for (int z = 0; z < splits; ++z) {
                v += splits > 1 ? ld_peer(part + t * 128 + f, z) : part[t * 128 + f];
                if (GLU) up += splits > 1 ? ld_peer(part + t * 128 + 64 + f, z) : part[t * 128 + 64 + f];
            }
            const long at = (long)t * a.ldo + n;
            if (GLU) v = act_glu(a.act, v, up);
            else if (a.act == ACT_RELU2) v = fmaxf(v, 0.f), v *= v;
            else if (a.act == ACT_SILU) v = v / (1.f + __expf(-v));
            if (a.out_f32) {
                if (a.residual) v += reinterpret_cast<const float*>(a.residual)[at];
                reinterpret_cast<float*>(a.out)[at] = v;
            } else {
                if (a.residual) v += bf2f(reinterpret_cast<const bf16*>(a.residual)[at]);
                reinterpret_cast<bf16*>(a.out)[at] = f2bf(v);
            }
        }
        if (splits > 1) cluster_sync();                                   // a CTA's part stays until its peers have read it
    }
    if (warp == 1) {
        fence_after_sync();
        tmem_dealloc<256>(tmem);
    }
}

struct Launch {
    CUtensorMap m[3], x;
    BlockGemmArgs a;
    int strip, splits, grid;
    int* status;
    cudaStream_t s;
};

template <int TYPE, int NT, bool GLU, bool EXPERTS>
int launch(const Launch& l) {
    using L = Shape<TYPE, NT, GLU, EXPERTS>;
    const int stages = L::stages(l.strip);
    const size_t smem = (size_t)L::fixed(l.strip) + (size_t)stages * L::RAW;
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemm_blocks_kernel<TYPE, NT, GLU, EXPERTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, BG_SMEM));
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(l.grid);
    cfg.blockDim = dim3(BG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = l.s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = l.splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tsb_pdl_enabled() ? 2 : 1;
    TSB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_blocks_kernel<TYPE, NT, GLU, EXPERTS>, l.m[0], l.m[1], l.m[2], l.x, l.a, stages, l.strip, l.splits,
                                      l.status));
    return TSB_OK;
}

template <int TYPE, bool GLU>
int launch_dense(const Launch& l) {
    if (l.a.T <= 16) return launch<TYPE, 16, GLU, false>(l);
    if (l.a.T <= 32) return launch<TYPE, 32, GLU, false>(l);
    return launch<TYPE, 64, GLU, false>(l);
}

int sm_count() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Parts of K for `tiles` tiles of `n` stages: as many as the CTAs that run at once allow, up to a portable cluster.  Not seven: clusters of
// seven pack badly into the GPCs (20 tiles of 38 stages: six 11.6 us, seven 13.6, eight 12.0; 42 of 84: five 35.4, six 31.0).
int choose_splits(int tiles, int n, int sms) {
    for (int s = 8; s > 1; --s)
        if (s != 7 && s <= n && tiles * s <= 2 * sms) return s;
    return 1;
}
}  // namespace

// The maps of a weight's planes over `rows` rows, boxes of `box` rows.
static int block_maps(CUtensorMap* m, const void* const* p, int type, long rows, int K, int box) {
    int rc = TSB_OK;
    switch (type) {
    case TSB_Q4_K: rc = tsb_make_tmap_bytes(&m[0], p[0], rows, (uint64_t)(K / 256) * 144, box, 144); break;
    case TSB_Q6_K:
        rc = tsb_make_tmap_bytes(&m[0], p[0], rows, K / 2, box, 128);
        if (!rc) rc = tsb_make_tmap_bytes(&m[1], p[1], rows, K / 4, box, 64);
        if (!rc) rc = tsb_make_tmap_bytes(&m[2], p[2], rows, K / 16, box, 16);
        break;
    case TSB_Q8_0:
        rc = tsb_make_tmap_bytes(&m[0], p[0], rows, K, box, 128);
        if (!rc) rc = tsb_make_tmap_bytes(&m[1], p[1], rows, K / 16, box, 16);
        break;
    default: rc = tsb_make_tmap_bytes(&m[0], p[0], rows, K / 2, box, 64); break;
    }
    if (rc) return rc;
    if (type == TSB_Q4_K || type == TSB_MXFP4) m[1] = m[0];
    if (type != TSB_Q6_K) m[2] = m[0];
    return TSB_OK;
}

// Whether tsb_gemm_blocks takes a matrix: whole blocks of 256 values (the stages), planes that start on 16 bytes.
extern "C" int tsb_gemm_blocks_takes(int type, const void* p0, const void* p1, const void* p2, int N, int K, int act) {
    if ((type != TSB_Q4_K && type != TSB_Q6_K && type != TSB_Q8_0) || N <= 0 || K <= 0 || K % 256 != 0) return 0;
    if (act >= ACT_SWIGLU && act <= ACT_SWIGLU_OAI && N % 2 != 0) return 0;
    return ((reinterpret_cast<uintptr_t>(p0) | reinterpret_cast<uintptr_t>(p1) | reinterpret_cast<uintptr_t>(p2)) & 15) == 0;
}

// X [T, K] bf16 (ldx elements per row), 1 <= T <= 64; out [T, ldo] of N (gated: N / 2) columns, f32 or bf16; bias [N] or null;
// residual as out or null.  p0 .. p3: the planes of quant_blocks.cuh.
extern "C" int tsb_gemm_blocks(const void* p0, const void* p1, const void* p2, const void* p3, int type, int N, int K, const void* X, long ldx, int T,
                               void* out, long ldo, int out_f32, const float* bias, const void* residual, int act, int* status, void* stream) {
    TSB_CHECK_ARG(T >= 0 && T <= 64, "gemm_blocks: %d rows", T);
    TSB_CHECK_ARG(tsb_gemm_blocks_takes(type, p0, p1, p2, N, K, act), "gemm_blocks: weight type %d, N=%d K=%d", type, N, K);
    TSB_CHECK_ARG(ldx % 8 == 0 && status != nullptr, "gemm_blocks: ldx=%ld, or no status word", ldx);
    if (T == 0) return TSB_OK;
    const bool glu = act >= ACT_SWIGLU && act <= ACT_SWIGLU_OAI;
    const int rows = glu ? 64 : 128, nt = T <= 16 ? 16 : T <= 32 ? 32 : 64;
    Launch l = {};
    const void* p[3] = {p0, p1, p2};
    int rc = block_maps(l.m, p, type, N, K, rows);
    if (!rc) rc = tsb_make_tmap_2d_bf16(&l.x, X, (uint64_t)T, (uint64_t)K, (uint64_t)ldx, nt, 64);
    if (rc) return rc;
    BlockGemmArgs& a = l.a;
    a.out = out, a.bias = bias, a.residual = residual, a.d = (const uint16_t*)p3, a.ldo = ldo, a.T = T, a.N = N, a.n_out = glu ? N / 2 : N, a.K = K;
    a.out_f32 = out_f32, a.act = act;
    a.m_tiles = (a.n_out + rows - 1) / rows;
    const int n = K / 256;
    l.splits = choose_splits(a.m_tiles, n, sm_count());
    a.per = (n + l.splits - 1) / l.splits;
    l.splits = (n + a.per - 1) / a.per;
    l.grid = a.m_tiles * l.splits;
    l.status = status, l.s = (cudaStream_t)stream;
    switch (type) {
    case TSB_Q4_K: return glu ? launch_dense<TSB_Q4_K, true>(l) : launch_dense<TSB_Q4_K, false>(l);
    case TSB_Q6_K: return glu ? launch_dense<TSB_Q6_K, true>(l) : launch_dense<TSB_Q6_K, false>(l);
    default: return glu ? launch_dense<TSB_Q8_0, true>(l) : launch_dense<TSB_Q8_0, false>(l);
    }
}

template <bool GLU>
static int launch_experts(const Launch& l, int nt) {
    switch (nt) {
    case 16: return launch<TSB_MXFP4, 16, GLU, true>(l);
    case 32: return launch<TSB_MXFP4, 32, GLU, true>(l);
    default: return launch<TSB_MXFP4, 64, GLU, true>(l);
    }
}

// Most rows of a tile with which tsb_gemm_experts takes a stack of matrices (32 or 64; 0: not at all): MXFP4, scales of a tile in whole
// pieces of 16 bytes and few enough to lie beside three stages twice.
extern "C" int tsb_gemm_experts_takes(int type, int N, int K, int act) {
    const bool glu = act >= ACT_SWIGLU && act <= ACT_SWIGLU_OAI;
    if (type != TSB_MXFP4 || N <= 0 || K <= 0 || K % 32 != 0 || (glu && N % 2 != 0)) return 0;
    const long n_out = glu ? N / 2 : N, kb = K / 32;
    const int strip = (int)min(128 * kb, 1L << 20);
    if (n_out * kb % 16 != 0) return 0;
    return Shape<TSB_MXFP4, 64, true, true>::stages(strip) >= 3 ? 64 : Shape<TSB_MXFP4, 32, true, true>::stages(strip) >= 3 ? 32 : 0;
}

// The products of a mixture's experts: X [P, K] bf16 in expert order, `tiles` int4 {expert, first row, rows} with at most `tile_rows`
// (16, 32 or 64) rows each, meta[0] of them (at most max_tiles); out [P, ldo]; bias [E, N], row_scale [P] or null.
extern "C" int tsb_gemm_experts(const void* p0, const void* p1, int type, int N, int K, int E, const void* X, int P, void* out, long ldo, int out_f32,
                                const float* bias, const float* row_scale, const void* tiles, const int* meta, int max_tiles, int tile_rows, int act,
                                int* status, void* stream) {
    TSB_CHECK_ARG(tile_rows <= tsb_gemm_experts_takes(type, N, K, act), "gemm_experts: weight type %d, N=%d K=%d, tiles of %d rows", type, N, K, tile_rows);
    TSB_CHECK_ARG(((reinterpret_cast<uintptr_t>(p0) | reinterpret_cast<uintptr_t>(p1)) & 15) == 0, "gemm_experts: planes must start on 16 bytes");
    TSB_CHECK_ARG(tile_rows == 16 || tile_rows == 32 || tile_rows == 64, "gemm_experts: tiles of %d rows", tile_rows);
    TSB_CHECK_ARG(status != nullptr && E > 0 && P >= 0 && max_tiles >= 0, "gemm_experts: E=%d P=%d, or no status word", E, P);
    if (P == 0 || max_tiles == 0) return TSB_OK;
    const bool glu = act >= ACT_SWIGLU && act <= ACT_SWIGLU_OAI;
    const int rows = glu ? 64 : 128;
    Launch l = {};
    const void* p[3] = {p0, nullptr, nullptr};
    int rc = block_maps(l.m, p, type, (long)E * N, K, rows);
    if (!rc) rc = tsb_make_tmap_2d_bf16(&l.x, X, (uint64_t)P, (uint64_t)K, (uint64_t)K, tile_rows, 64);
    if (rc) return rc;
    BlockGemmArgs& a = l.a;
    a.out = out, a.bias = bias, a.row_scale = row_scale, a.scales = (const uint8_t*)p1, a.tiles = (const int4*)tiles, a.meta = meta, a.ldo = ldo;
    a.T = P, a.N = N, a.n_out = glu ? N / 2 : N, a.K = K, a.out_f32 = out_f32, a.act = act;
    a.m_tiles = (a.n_out + rows - 1) / rows;
    l.strip = 128 * (K / 32);
    l.splits = 1;
    l.grid = (int)min((long)max_tiles * a.m_tiles, 2L * sm_count());
    l.status = status, l.s = (cudaStream_t)stream;
    return glu ? launch_experts<true>(l, tile_rows) : launch_experts<false>(l, tile_rows);
}
