// Chunked prefill of the linear-attention layers: GatedDeltaNet from a layer's packed projections (the second half of this file), Mamba2, and first the kernel that
// carries a state over chunks whose operands are there already: Mamba2 takes it (with no correction, U_c = U0_c), and the delta rule where its own kernels are
// turned off and the chunk algebra runs as tensor ops.
//
// In the chunked (WY) form of the delta rule the work inside a chunk of 64 tokens is batched matrix algebra over
// (heads x chunks) that has no dependency between chunks (the decay mask, K K^T, the unit-triangular solve, Q K^T);
// what remains sequential is carrying the state S [Dv, Dk] of each head across the chunks:
//
//     U_c   = U0_c - W_c S^T                     [64, Dv]   the chunk's value updates, corrected by the state
//     O_c   = Qd_c S^T + P_c U_c                 [64, Dv]   outputs: state term + intra-chunk term
//     S    <- gamma_c S + U_c^T Kd_c             [Dv, Dk]
//
// The reference builds a ggml graph of about forty nodes per chunk for this
// (TensorSharp.GGML.Native/ggml_ops_gated_delta_net.cpp:178-615); as tensor ops it is three small batched products per
// chunk, launch-bound.  Here a CTA owns one head and a slice of 32 value dimensions, keeps its slice of S in shared
// memory for the whole prompt, and walks the chunks: the three products run on the tensor cores (mma.sync m16n8k8,
// tf32 operands, f32 accumulation; the state itself stays f32), the operands of the next chunk stream in with cp.async
// while the current one is multiplied (each operand buffer is refilled as soon as its product is done).
#include "common.cuh"
#include "tcgen05.cuh"

struct GdnCarryArgs {
    const float* U0;      // [Hv, nc, 64, Dv]
    const float* W;       // [Hv, nc, 64, Dk]
    const float* Qd;      // [Hv, nc, 64, Dk]
    const float* Kd;      // [Hv, nc, 64, Dk]
    const float* P;       // [Hv, nc, 64, 64]
    const float* gamma;   // [Hv, nc]
    float* state;         // [Hv, Dv, Dk], updated in place
    float* out;           // [Hv, nc, 64, Dv]
    int Hv, nc, Dk, Dv;
};

namespace {
constexpr int GC = 64;        // tokens per chunk
constexpr int DVS = 32;       // value dimensions per CTA

__device__ __forceinline__ uint32_t tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
__device__ __forceinline__ void cp_wait2() { asm volatile("cp.async.wait_group 2;"); }

// rows x cols f32 from global (row stride gs) into shared (row stride ss), 16 bytes per copy, all 256 threads
__device__ __forceinline__ void stage(float* dst, int ss, const float* src, int gs, int rows, int cols) {
    const int per = cols / 4;
    for (int i = threadIdx.x; i < rows * per; i += 256) {
        const int r = i / per, c = (i % per) * 4;
        cp16(dst + r * ss + c, src + (long)r * gs + c);
    }
}

// Shared-memory row strides (floats), chosen so that the fragment loads below touch 32 different banks:
// operands read as A[row g][k t] or B[n g][k t] want stride = 4 (mod 32); operands read as [k t][n g] want 8 (mod 32).
template <int DK> struct Lay {
    static constexpr int LW = DK + 4;      // W, Qd, S: [row][k]
    static constexpr int LK = DK + 8;      // Kd: [t][k] read as B[k = t][n = k]
    static constexpr int LP = GC + 4;      // P: [t][j]
    static constexpr int LU = DVS + 8;     // U: [j][v] read as B[k = j][n = v] and as A[m = v][k = j]
    static constexpr int floats = DVS * LW + 2 * GC * LW + GC * LK + GC * LP + GC * LU;
};
}  // namespace

// HASW = false: nothing to correct (W = 0, the Mamba2 form): U = U0, and neither W's tiles nor its product exist.
template <int DK, bool HASW>
__global__ void __launch_bounds__(256) gdn_chunk_carry_kernel(GdnCarryArgs a) {
    using L = Lay<DK>;
    extern __shared__ __align__(16) float sm[];
    float* sS = sm;                       // [DVS][LW]   state slice
    float* sW = sS + DVS * L::LW;         // [64][LW]
    float* sQ = sW + GC * L::LW;          // [64][LW]
    float* sK = sQ + GC * L::LW;          // [64][LK]
    float* sP = sK + GC * L::LK;          // [64][LP]
    float* sU = sP + GC * L::LP;          // [64][LU]
    const int h = blockIdx.y, dv0 = blockIdx.x * DVS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int Dv = a.Dv, nc = a.nc;
    float* Sg = a.state + ((long)h * Dv + dv0) * DK;
    const long hc = (long)h * nc;
    // prologue: the state slice and the first chunk's operands, in the commit order W | Qd + P | Kd kept below
    stage(sS, L::LW, Sg, DK, DVS, DK);
    if (HASW) stage(sW, L::LW, a.W + hc * GC * DK, DK, GC, DK);
    cp_commit();
    stage(sQ, L::LW, a.Qd + hc * GC * DK, DK, GC, DK);
    stage(sP, L::LP, a.P + hc * GC * GC, GC, GC, GC);
    cp_commit();
    stage(sK, L::LK, a.Kd + hc * GC * DK, DK, GC, DK);
    cp_commit();

    // tiles of the [64, 32] products: warp -> 16 rows (mt) x 16 columns (two n-tiles of 8)
    const int mt = warp >> 1, nb = (warp & 1) * 2;
    for (int c = 0; c < nc; ++c) {
        const long ch = hc + c;
        const bool more = c + 1 < nc;
        // U0 fragments straight from global (requested before the wait)
        float u[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float* p0 = a.U0 + (ch * GC + mt * 16 + g) * Dv + dv0 + (nb + j) * 8 + 2 * t;
            const float2 lo = *reinterpret_cast<const float2*>(p0), hi = *reinterpret_cast<const float2*>(p0 + 8L * Dv);
            u[j][0] = lo.x; u[j][1] = lo.y; u[j][2] = hi.x; u[j][3] = hi.y;
        }
        const float gam = a.gamma[ch];
        cp_wait2();                       // W of this chunk (and, for c = 0, the state) has landed
        __syncthreads();
        // ---- U = U0 - W S^T
        {
            float acc[2][4] = {};
#pragma unroll 4
            for (int k0 = 0; HASW && k0 < DK; k0 += 8) {
                uint32_t af[4];
                const float* ap = sW + (mt * 16 + g) * L::LW + k0 + t;
                af[0] = tf32(ap[0]); af[1] = tf32(ap[8 * L::LW]); af[2] = tf32(ap[4]); af[3] = tf32(ap[8 * L::LW + 4]);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float* bp = sS + ((nb + j) * 8 + g) * L::LW + k0 + t;
                    mma_tf32(acc[j], af, tf32(bp[0]), tf32(bp[4]));
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float* up = sU + (mt * 16 + g) * L::LU + (nb + j) * 8 + 2 * t;
                up[0] = u[j][0] - acc[j][0]; up[1] = u[j][1] - acc[j][1];
                up[8 * L::LU] = u[j][2] - acc[j][2]; up[8 * L::LU + 1] = u[j][3] - acc[j][3];
            }
        }
        __syncthreads();                  // U complete, W free
        if (more && HASW) stage(sW, L::LW, a.W + (ch + 1) * GC * DK, DK, GC, DK);
        cp_commit();
        cp_wait2();                       // Qd and P of this chunk
        __syncthreads();
        // ---- O = Qd S^T + P U
        {
            float acc[2][4] = {};
#pragma unroll 4
            for (int k0 = 0; k0 < DK; k0 += 8) {
                uint32_t af[4];
                const float* ap = sQ + (mt * 16 + g) * L::LW + k0 + t;
                af[0] = tf32(ap[0]); af[1] = tf32(ap[8 * L::LW]); af[2] = tf32(ap[4]); af[3] = tf32(ap[8 * L::LW + 4]);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float* bp = sS + ((nb + j) * 8 + g) * L::LW + k0 + t;
                    mma_tf32(acc[j], af, tf32(bp[0]), tf32(bp[4]));
                }
            }
#pragma unroll 4
            for (int k0 = 0; k0 < GC; k0 += 8) {
                uint32_t af[4];
                const float* ap = sP + (mt * 16 + g) * L::LP + k0 + t;
                af[0] = tf32(ap[0]); af[1] = tf32(ap[8 * L::LP]); af[2] = tf32(ap[4]); af[3] = tf32(ap[8 * L::LP + 4]);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float* bp = sU + (k0 + t) * L::LU + (nb + j) * 8 + g;
                    mma_tf32(acc[j], af, tf32(bp[0]), tf32(bp[4 * L::LU]));
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float* op = a.out + (ch * GC + mt * 16 + g) * Dv + dv0 + (nb + j) * 8 + 2 * t;
                *reinterpret_cast<float2*>(op) = make_float2(acc[j][0], acc[j][1]);
                *reinterpret_cast<float2*>(op + 8L * Dv) = make_float2(acc[j][2], acc[j][3]);
            }
        }
        __syncthreads();                  // Qd, P free; every read of the old state is done
        if (more) {
            stage(sQ, L::LW, a.Qd + (ch + 1) * GC * DK, DK, GC, DK);
            stage(sP, L::LP, a.P + (ch + 1) * GC * GC, GC, GC, GC);
        }
        cp_commit();
        cp_wait2();                       // Kd of this chunk
        __syncthreads();
        // ---- S = gamma S + U^T Kd: [32, DK] as 2 x (DK / 8) tiles, warp -> one 16-row half and DK / 32 column tiles
        {
            constexpr int NT = DK / 32;                   // n-tiles per warp
            const int m2 = warp & 1, n0 = (warp >> 1) * NT;
            float acc[NT][4];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const float* sp = sS + (m2 * 16 + g) * L::LW + (n0 + j) * 8 + 2 * t;
                acc[j][0] = gam * sp[0]; acc[j][1] = gam * sp[1];
                acc[j][2] = gam * sp[8 * L::LW]; acc[j][3] = gam * sp[8 * L::LW + 1];
            }
#pragma unroll 2
            for (int k0 = 0; k0 < GC; k0 += 8) {
                uint32_t af[4];                           // A[m = v][k = token] = U[token][v]
                const float* ap = sU + (k0 + t) * L::LU + m2 * 16 + g;
                af[0] = tf32(ap[0]); af[1] = tf32(ap[8]); af[2] = tf32(ap[4 * L::LU]); af[3] = tf32(ap[4 * L::LU + 8]);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const float* bp = sK + (k0 + t) * L::LK + (n0 + j) * 8 + g;
                    mma_tf32(acc[j], af, tf32(bp[0]), tf32(bp[4 * L::LK]));
                }
            }
            // each warp reads only the state rows and columns it writes, so no barrier between the read above and this
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                float* sp = sS + (m2 * 16 + g) * L::LW + (n0 + j) * 8 + 2 * t;
                sp[0] = acc[j][0]; sp[1] = acc[j][1];
                sp[8 * L::LW] = acc[j][2]; sp[8 * L::LW + 1] = acc[j][3];
            }
        }
        __syncthreads();                  // new state visible, Kd and U free
        if (more) stage(sK, L::LK, a.Kd + (ch + 1) * GC * DK, DK, GC, DK);
        cp_commit();
    }
    asm volatile("cp.async.wait_group 0;");
    for (int i = threadIdx.x; i < DVS * (DK / 4); i += 256) {
        const int r = i / (DK / 4), c4 = (i % (DK / 4)) * 4;
        *reinterpret_cast<float4*>(Sg + (long)r * DK + c4) = *reinterpret_cast<const float4*>(sS + r * L::LW + c4);
    }
}

template <int DK, bool HASW>
static int launch_carry_w(const GdnCarryArgs& a, cudaStream_t s) {
    const size_t smem = (size_t)Lay<DK>::floats * sizeof(float);
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gdn_chunk_carry_kernel<DK, HASW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = true;
    }
    gdn_chunk_carry_kernel<DK, HASW><<<dim3(a.Dv / DVS, a.Hv), 256, smem, s>>>(a);
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

template <int DK>
static int launch_carry(const GdnCarryArgs& a, cudaStream_t s) {
    return a.W != nullptr ? launch_carry_w<DK, true>(a, s) : launch_carry_w<DK, false>(a, s);
}

// One sequence: carries `state` through `nc` chunks of 64 tokens and writes the chunk outputs.
extern "C" int tsb_gdn_chunk_carry(const GdnCarryArgs* args, void* stream) {
    TSB_CHECK_ARG(args != nullptr, "gdn_chunk_carry: null arguments");
    const GdnCarryArgs& a = *args;
    TSB_CHECK_ARG(a.Hv > 0 && a.nc > 0, "gdn_chunk_carry: Hv=%d chunks=%d", a.Hv, a.nc);
    TSB_CHECK_ARG(a.Dv % DVS == 0 && a.Dv > 0, "gdn_chunk_carry: value head size %d is not a multiple of %d", a.Dv, DVS);
    switch (a.Dk) {
    case 64: return launch_carry<64>(a, (cudaStream_t)stream);
    case 128: return launch_carry<128>(a, (cudaStream_t)stream);
    default:
        tsb_set_error("gdn_chunk_carry: key head size %d unsupported (64, 128)", a.Dk);
        return TSB_ERR_UNSUPPORTED;
    }
}

// ==========================================================================================
// The delta rule from a layer's packed projections, in two kernels and an output norm.  With k, q the L2-normalised key / query rows
// (q also times Dv^-1/2), g the log-decay and b the write strength of each token, c_i the running sum of g inside a chunk of 64:
//     A[i][j]  = b_i (k_i . k_j) exp(c_i - c_j)        j <  i      (strictly lower triangular)
//     P[i][j]  =     (q_i . k_j) exp(c_i - c_j)        j <= i
//     T = (I + A)^-1                                   once per (value head, chunk): no dependency between chunks
// and then, chunk after chunk with the state S [Dv, Dk] of a head,
//     U = T (b v - b exp(c) k S^T),   O = exp(c) q S^T + P U,   S <- exp(c_last) S + (exp(c_last - c) U)^T k
// so that what the first kernel leaves in memory are two triangles of 64 x 64, four numbers per token, and once per key head the keys and
// queries as the second one reads them.  (It used to solve for T b v and T b exp(c) k, a column of 64 values per thread, and to write
// both and two scaled copies of q and k per value head.)  Tokens past a sequence's end are zero rows (b = 0, g = 0): they leave
// state and outputs untouched, so ragged batches share one launch.
// Measured, 8192 tokens, 16 key and 32 value heads of 128 (us): chunk kernel 994 -> 197, state kernel 612 -> 519, output norm 153 -> 92.
//
// Operands lie in slabs of eight columns, [slab][row][8]: the rows of a slab are contiguous 32 bytes, so a fragment is an 8-byte load per
// lane without bank conflicts (columns 2 t and 2 t + 1 stand for its k = t and t + 4, in both operands alike) and a whole matrix is one
// bulk copy.  Triangles keep the rows 16 p .. 63 of the slabs 2 p and 2 p + 1 only.
// ==========================================================================================
constexpr int TRI = 320 * 8;               // floats of a triangle
__device__ __forceinline__ int tri_at(int slab, int row) {             // of the row's eight columns, in rows of eight
    const int p = slab >> 1;
    return 128 * p - 16 * p * (p - 1) + (slab & 1) * (64 - 16 * p) + row - 16 * p;
}
struct GdnPrepArgs {
    const float* qkv; long qkv_s;          // [T, 2 Hk Dk + Hv Dv] rows: q heads | k heads | v heads
    const void* beta; const void* alpha; long ba_s; int ba_f32;      // [T, Hv]
    const float* dt_bias; const float* a_log;                        // [Hv]
    const int* cu_q;                       // [B + 1] first row of each sequence
    float* K; float* Q;                    // [B Hk, nc][Dk / 8][64][8] keys and queries as they are, rounded to tf32
    float* T; float* P;                    // [B Hv, nc]: two triangles (T and what tf32 leaves of it), one triangle, tf32
    float4* scale;                         // [B Hv, nc, 64]: of the query row, of the key row to the chunk's end, of the value, of the key row
    float* gamma;                          // [B Hv, nc]
    float* state; const long* slots;       // [slots, Hv, Dv, Dk] and a slot per sequence (scan)
    float* out;                            // [B Hv, nc, 64, Dv] (scan)
    int* status;                           // set where a bounded wait gave up
    int Hk, Hv, Dk, Dv, B, nc;
    float eps;
};

namespace {
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32(x);
    lo = tf32(x - __uint_as_float(hi));
}
__device__ __forceinline__ float ld_ba(const void* p, long i, int f32) {
    return f32 ? reinterpret_cast<const float*>(p)[i] : bf2f(reinterpret_cast<const bf16*>(p)[i]);
}
// 16 bytes, or zeros where there is no source
__device__ __forceinline__ void cp16_if(void* smem, const void* gmem, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(there ? 16 : 0));
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Fragments take the columns k0 + 2 t and k0 + 2 t + 1 as their k = t and t + 4 (of both operands alike), one 8-byte load for two values;
// row strides of 8 (mod 32) floats keep those free of conflicts.
template <int DK> struct PrepLay {
    static constexpr int LQ = DK + 8, LA = 68, LY = 36;
    static constexpr int fixed = 2 * GC * LQ + GC * LA + 32 * LY + 2 * GC;
};

// T21 = -T22 A21 T11 for the pairs of neighbouring N x N blocks on the diagonal, in place
template <int N>
__device__ __forceinline__ void combine(float* sA, float* sY) {
    constexpr int LA = PrepLay<128>::LA, LY = PrepLay<128>::LY, PER = 32 * N / 256;       // 64 / 2 N pairs of N x N results
    const int e0 = threadIdx.x * PER, pr = e0 / (N * N), i = (e0 / N) % N, j0 = e0 % N;
    float* D = sA + (pr * 2 * N) * LA + pr * 2 * N;                                       // T11; A21 below it, T22 beside that
    float y[PER];
#pragma unroll
    for (int c = 0; c < PER; ++c) y[c] = 0.f;
    for (int k = j0; k < N; ++k) {                                                        // T11 is lower triangular
        const float x = D[(N + i) * LA + k];
#pragma unroll
        for (int c = 0; c < PER; ++c) y[c] += x * D[k * LA + j0 + c];
    }
#pragma unroll
    for (int c = 0; c < PER; ++c) sY[(pr * N + i) * LY + j0 + c] = y[c];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < PER; ++c) y[c] = 0.f;
    for (int k = 0; k <= i; ++k) {
        const float x = D[(N + i) * LA + N + k];
#pragma unroll
        for (int c = 0; c < PER; ++c) y[c] -= x * sY[(pr * N + k) * LY + j0 + c];
    }
#pragma unroll
    for (int c = 0; c < PER; ++c) D[(N + i) * LA + j0 + c] = y[c];
    __syncthreads();
}
}  // namespace

// One CTA per (sequence, key head, chunk): the two Gram products once for all value heads of the key head, on the tensor cores with split
// tf32 operands (hi + lo parts, three products: f32-level accuracy in the matrix that is inverted), then per value head its decays and the
// inverse, in f32: blocks of 8 by substitution, three times T21 = -T22 A21 T11.
// Bound by latency (barriers between small steps); two CTAs share an SM.
template <int DK>
__global__ void __launch_bounds__(256, 2) gdn_chunk_prep_kernel(GdnPrepArgs a) {
    using L = PrepLay<DK>;
    constexpr int LQ = L::LQ, LA = L::LA;
    extern __shared__ __align__(16) float sm[];
    float* sK = sm;                        // [64][LQ]
    float* sQ = sK + GC * LQ;              // [64][LQ]
    float* sA = sQ + GC * LQ;              // [64][LA]
    float* sY = sA + GC * LA;              // [32][LY]
    float* kn = sY + 32 * L::LY;           // [64] 1 / |k|
    float* qn = kn + GC;                   // [64] Dv^-1/2 / |q|
    float* sc = qn + GC;                   // [value heads][64] running log-decay
    const int c = blockIdx.x, b = blockIdx.y / a.Hk, hk = blockIdx.y % a.Hk, R = (a.Hv - hk + a.Hk - 1) / a.Hk;
    float* sb = sc + R * GC;               // [value heads][64] write strength
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int row0 = a.cu_q[b], valid = max(0, min(GC, a.cu_q[b + 1] - row0 - c * GC));        // tokens of this chunk that exist
    const long tok0 = (long)row0 + (long)c * GC;
    for (int i = threadIdx.x; i < GC * (DK / 4); i += 256) {
        const int r = i / (DK / 4), col = (i % (DK / 4)) * 4;
        const float* src = a.qkv + (tok0 + (r < valid ? r : 0)) * a.qkv_s + hk * DK + col;
        const bool ok = r < valid;
        cp16_if(sQ + r * LQ + col, ok ? src : a.qkv, ok);
        cp16_if(sK + r * LQ + col, ok ? src + (long)a.Hk * DK : a.qkv, ok);
    }
    cp_commit();
    for (int h = warp; h < R; h += 8) {    // decays and strengths of a value head, and the running sum over the 64 tokens
        const int hv = hk + h * a.Hk;
        float x[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = lane + 32 * i;
            float gd = 0.f, be = 0.f;
            if (r < valid) {
                const float al = ld_ba(a.alpha, (tok0 + r) * a.ba_s + hv, a.ba_f32) + a.dt_bias[hv];
                gd = (al > 20.f ? al : log1pf(__expf(al))) * a.a_log[hv];
                be = 1.f / (1.f + __expf(-ld_ba(a.beta, (tok0 + r) * a.ba_s + hv, a.ba_f32)));
            }
            x[i] = gd;
            sb[h * GC + r] = be;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y0 = __shfl_up_sync(0xffffffffu, x[0], o), y1 = __shfl_up_sync(0xffffffffu, x[1], o);
            if (lane >= o) x[0] += y0, x[1] += y1;
        }
        x[1] += __shfl_sync(0xffffffffu, x[0], 31);
        sc[h * GC + lane] = x[0];
        sc[h * GC + lane + 32] = x[1];
    }
    cp_wait_all();
    __syncthreads();
    const float qscale = rsqrtf((float)a.Dv);
#pragma unroll 2
    for (int r = warp * 8; r < warp * 8 + 8; ++r) {
        float qs = 0.f, ks = 0.f;
#pragma unroll
        for (int i = 0; i < DK / 32; ++i) {
            const float x = sQ[r * LQ + lane + 32 * i], y = sK[r * LQ + lane + 32 * i];
            qs += x * x;
            ks += y * y;
        }
        qs = warp_sum(qs);
        ks = warp_sum(ks);
        if (lane == 0) {
            qn[r] = r < valid ? qscale * rsqrtf(qs + a.eps) : 0.f;
            kn[r] = r < valid ? rsqrtf(ks + a.eps) : 0.f;
        }
    }
    // ---- k k^T and q k^T, tiles of 16 x 8 on and below the diagonal: 8, 6, 4, 2 of the four row tiles, dealt to 3, 2, 2, 1 warps
    const int mt = warp < 3 ? 3 : warp < 5 ? 2 : warp < 7 ? 1 : 0;
    const int part = warp < 3 ? warp : warp < 5 ? warp - 3 : warp < 7 ? warp - 5 : 0;
    const int n0 = mt == 1 ? 2 * part : 3 * part, nt = min(mt == 1 || mt == 0 ? 2 : 3, 2 * (mt + 1) - n0);
    float kk[3][4] = {}, qk[3][4] = {};
#pragma unroll 2
    for (int k0 = 0; k0 < DK; k0 += 8) {
        uint32_t ah[4], al[4], qh[4], ql[4];
        const float2 ka = *reinterpret_cast<const float2*>(sK + (mt * 16 + g) * LQ + k0 + 2 * t), kb = *reinterpret_cast<const float2*>(sK + (mt * 16 + g + 8) * LQ + k0 + 2 * t);
        const float2 qa = *reinterpret_cast<const float2*>(sQ + (mt * 16 + g) * LQ + k0 + 2 * t), qb = *reinterpret_cast<const float2*>(sQ + (mt * 16 + g + 8) * LQ + k0 + 2 * t);
        split_tf32(ka.x, ah[0], al[0]); split_tf32(kb.x, ah[1], al[1]); split_tf32(ka.y, ah[2], al[2]); split_tf32(kb.y, ah[3], al[3]);
        split_tf32(qa.x, qh[0], ql[0]); split_tf32(qb.x, qh[1], ql[1]); split_tf32(qa.y, qh[2], ql[2]); split_tf32(qb.y, qh[3], ql[3]);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j >= nt) break;
            const float2 bv = *reinterpret_cast<const float2*>(sK + ((n0 + j) * 8 + g) * LQ + k0 + 2 * t);
            uint32_t b0h, b0l, b1h, b1l;
            split_tf32(bv.x, b0h, b0l);
            split_tf32(bv.y, b1h, b1l);
            mma_tf32(kk[j], al, b0h, b1h); mma_tf32(kk[j], ah, b0l, b1l); mma_tf32(kk[j], ah, b0h, b1h);
            mma_tf32(qk[j], ql, b0h, b1h); mma_tf32(qk[j], qh, b0l, b1l); mma_tf32(qk[j], qh, b0h, b1h);
        }
    }
    {                                      // keys and queries in slabs, rounded
        const long at = ((long)b * a.Hk + hk) * a.nc + c;
        uint4* Ko = reinterpret_cast<uint4*>(a.K + at * GC * DK);
        uint4* Qo = reinterpret_cast<uint4*>(a.Q + at * GC * DK);
        for (int i = threadIdx.x; i < GC * DK / 4; i += 256) {
            const int from = ((i >> 1) & 63) * LQ + (i >> 7) * 8 + (i & 1) * 4;
            const float4 x = *reinterpret_cast<const float4*>(sK + from), y = *reinterpret_cast<const float4*>(sQ + from);
            Ko[i] = make_uint4(tf32(x.x), tf32(x.y), tf32(x.z), tf32(x.w));
            Qo[i] = make_uint4(tf32(y.x), tf32(y.y), tf32(y.z), tf32(y.w));
        }
    }
    __syncthreads();                       // norms of all rows
    for (int h = 0; h < R; ++h) {
        const int hv = hk + h * a.Hk;
        const long ch = ((long)b * a.Hv + hv) * a.nc + c;
        const float* cs = sc + h * GC;
        const float* bs = sb + h * GC;
        uint32_t* Pg = reinterpret_cast<uint32_t*>(a.P + ch * TRI);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if (j >= nt) break;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = mt * 16 + g + e * 8, jj = (n0 + j) * 8 + 2 * t;
                const float ci = cs[i], m0 = jj <= i ? __expf(fminf(ci - cs[jj], 0.f)) * kn[jj] : 0.f;
                const float m1 = jj + 1 <= i ? __expf(fminf(ci - cs[jj + 1], 0.f)) * kn[jj + 1] : 0.f, bk = bs[i] * kn[i];
                *reinterpret_cast<uint2*>(Pg + tri_at(n0 + j, i) * 8 + 2 * t) = make_uint2(tf32(qk[j][2 * e] * m0 * qn[i]), tf32(qk[j][2 * e + 1] * m1 * qn[i]));
                sA[i * LA + jj] = jj < i ? kk[j][2 * e] * m0 * bk : 0.f;
                sA[i * LA + jj + 1] = jj + 1 < i ? kk[j][2 * e + 1] * m1 * bk : 0.f;
            }
        }
        if (threadIdx.x < GC) {
            const int r = threadIdx.x;
            const float dec = __expf(cs[r]);
            a.scale[ch * GC + r] = make_float4(qn[r] * dec, kn[r] * __expf(cs[GC - 1] - cs[r]), bs[r], bs[r] * dec * kn[r]);
            if (r == 0) a.gamma[ch] = __expf(cs[GC - 1]);
        }
        __syncthreads();
        if (threadIdx.x < 64) {            // the inverses of the eight 8 x 8 blocks, a column each thread
            float* D = sA + (threadIdx.x & ~7) * (LA + 1);
            const int j = threadIdx.x & 7;
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float acc = i == j ? 1.f : 0.f;
#pragma unroll
                for (int l = 0; l < i; ++l) acc -= D[i * LA + l] * x[l];
                x[i] = acc;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) D[i * LA + j] = x[i];
        }
        __syncthreads();
        combine<8>(sA, sY);
        combine<16>(sA, sY);
        combine<32>(sA, sY);
        uint4* Th = reinterpret_cast<uint4*>(a.T + ch * 2 * TRI);
        uint4* Tl = Th + TRI / 4;
        for (int i = threadIdx.x; i < GC * 16; i += 256) {
            const int slab = i >> 7, r = (i >> 1) & 63, q = i & 1;
            if (r < 16 * (slab >> 1)) continue;
            const float4 x = *reinterpret_cast<const float4*>(sA + r * LA + slab * 8 + q * 4);
            uint4 hi, lo;
            split_tf32(x.x, hi.x, lo.x); split_tf32(x.y, hi.y, lo.y); split_tf32(x.z, hi.z, lo.z); split_tf32(x.w, hi.w, lo.w);
            Th[tri_at(slab, r) * 2 + q] = hi;
            Tl[tri_at(slab, r) * 2 + q] = lo;
        }
        __syncthreads();                   // sA is free again
    }
}

namespace {
template <int DK> struct ScanLay {         // in floats; K, T, P and the rows' factors in two places
    static constexpr int LU = DVS + 4, LKU = DVS + 8;
    static constexpr int S = 0, K = S + DVS * DK, Q = K + 2 * GC * DK, T = Q + GC * DK, P = T + 4 * TRI, SC = P + 2 * TRI, RH = SC + 2 * GC * 4,
                         RL = RH + GC * LU, U = RL + GC * LU, KU = U + GC * LU, BAR = KU + GC * LKU, floats = BAR + 8;
};
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}
}  // namespace

// One CTA per (sequence, value head, 32 value dimensions), chunk after chunk.  The state stays in registers as the accumulators of its
// own update (f32) and goes to shared memory rounded to tf32, as the products with keys and queries read it; the product with T is made
// of split operands, as exact as the substitution that it replaces.  Sixteen warps:
//   1  keys (warps 0-7) and queries (8-15) times the state, R = b v - (b exp(c) k) S^T     2  U = T R     3  the state's update (0-7), O += P U (8-15)
// with one barrier behind each; the next chunk's operands arrive meanwhile by bulk copies.  Bound by what the fragment loads take from
// shared memory (step 1: 256 KB, 1850 of a chunk's 7200 cycles) and the latency of the chain; an SM takes 110 KB from L2 per chunk.  (With
// 256 threads, operands rounded and split where they are read and cp.async: 676 us.)
template <int DK>
__global__ void __launch_bounds__(512) gdn_chunk_scan_kernel(GdnPrepArgs a) {
    using L = ScanLay<DK>;
    constexpr int LU = L::LU, LKU = L::LKU, NB = DK / 64;                          // column tiles of the state of a warp (0-7)
    extern __shared__ __align__(128) float sm[];
    uint32_t* smu = reinterpret_cast<uint32_t*>(sm);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + L::BAR);                     // [2] K, T, P and factors, [2] Q
    const int bh = blockIdx.y, b = bh / a.Hv, h = bh % a.Hv, hk = h % a.Hk, dv0 = blockIdx.x * DVS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool keys = warp < 8;
    const int mt = (warp >> 1) & 3, n1 = (warp & 1) * 2;                           // step 1: row tile, first of two column tiles
    const int row0 = a.cu_q[b], len = a.cu_q[b + 1] - row0, nc = (len + GC - 1) / GC;
    const float* vg = a.qkv + (long)row0 * a.qkv_s + 2L * a.Hk * DK + (long)h * a.Dv + dv0;
    const long ch0 = (long)bh * a.nc, hk0 = ((long)b * a.Hk + hk) * a.nc;
    auto load = [&](int c) {
        const int side = c & 1;
        tc::mbar_expect_tx(&full[side], (GC * DK + 3 * TRI + GC * 4) * 4);
        bulk_load(sm + L::K + side * GC * DK, a.K + (hk0 + c) * GC * DK, GC * DK * 4, &full[side]);
        bulk_load(sm + L::T + side * 2 * TRI, a.T + (ch0 + c) * 2 * TRI, 2 * TRI * 4, &full[side]);
        bulk_load(sm + L::P + side * TRI, a.P + (ch0 + c) * TRI, TRI * 4, &full[side]);
        bulk_load(sm + L::SC + side * GC * 4, a.scale + (ch0 + c) * GC, GC * 16, &full[side]);
    };
    auto load_q = [&](int c) {
        tc::mbar_expect_tx(&full[2], GC * DK * 4);
        bulk_load(sm + L::Q, a.Q + (hk0 + c) * GC * DK, GC * DK * 4, &full[2]);
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; ++i) tc::mbar_init(&full[i], 1);
        tc::fence_barrier_init();
        if (nc > 0) {
            load(0);
            load_q(0);
        }
    }
    float2 v[2][2];
    auto values = [&](int c) {             // of the rows and columns of this thread's fragments
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = c * GC + mt * 16 + g + 8 * e;
#pragma unroll
            for (int n = 0; n < 2; ++n)
                v[n][e] = keys && r < len ? *reinterpret_cast<const float2*>(vg + (long)r * a.qkv_s + (n1 + n) * 8 + 2 * t) : make_float2(0.f, 0.f);
        }
    };
    values(0);
    float* Sg = a.state + ((a.slots[b] * a.Hv + h) * a.Dv + dv0) * (long)DK;
    float S[NB][2][4];                     // column tiles warp * NB .. of the slice, rows 0-15 and 16-31
    if (keys) {
#pragma unroll
        for (int n = 0; n < NB; ++n)
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = m * 16 + g + 8 * e;
                    const float2 x = *reinterpret_cast<const float2*>(Sg + (long)r * DK + (warp * NB + n) * 8 + 2 * t);
                    S[n][m][2 * e] = x.x, S[n][m][2 * e + 1] = x.y;
                    *reinterpret_cast<uint2*>(smu + L::S + ((warp * NB + n) * DVS + r) * 8 + 2 * t) = make_uint2(tf32(x.x), tf32(x.y));
                }
    }
    __syncthreads();
    int c = 0;
    for (; c < nc; ++c) {
        const int side = c & 1;
        const uint32_t* sK = smu + L::K + side * GC * DK;
        const uint32_t* sT = smu + L::T + side * 2 * TRI;
        const uint32_t* sP = smu + L::P + side * TRI;
        const float4* scale = reinterpret_cast<const float4*>(sm + L::SC) + side * GC;
        const float gam = a.gamma[ch0 + c];
        if (threadIdx.x == 0 && c + 1 < nc) load(c + 1);
        const bool ok = tc::mbar_wait(&full[side], (c >> 1) & 1) && tc::mbar_wait(&full[2], c & 1);
        // ---- 1: 16 key or query rows times 16 columns of the state
        float acc[2][4] = {};
        {
            const uint32_t* A = (keys ? sK : smu + L::Q) + (mt * 16 + g) * 8 + 2 * t;
            const uint32_t* B = smu + L::S + (n1 * 8 + g) * 8 + 2 * t;
#pragma unroll
            for (int k = 0; k < DK / 8; ++k) {
                const uint2 lo = *reinterpret_cast<const uint2*>(A + k * GC * 8), hi = *reinterpret_cast<const uint2*>(A + k * GC * 8 + 64);
                const uint2 b0 = *reinterpret_cast<const uint2*>(B + k * DVS * 8), b1 = *reinterpret_cast<const uint2*>(B + k * DVS * 8 + 64);
                const uint32_t af[4] = {lo.x, hi.x, lo.y, hi.y};
                mma_tf32(acc[0], af, b0.x, b0.y);
                mma_tf32(acc[1], af, b1.x, b1.y);
            }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = mt * 16 + g + 8 * e;
            const float4 s = scale[r];
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                if (keys) {
                    uint2 hi, lo;
                    split_tf32(s.z * v[n][e].x - s.w * acc[n][2 * e], hi.x, lo.x);
                    split_tf32(s.z * v[n][e].y - s.w * acc[n][2 * e + 1], hi.y, lo.y);
                    *reinterpret_cast<uint2*>(smu + L::RH + r * LU + (n1 + n) * 8 + 2 * t) = hi;
                    *reinterpret_cast<uint2*>(smu + L::RL + r * LU + (n1 + n) * 8 + 2 * t) = lo;
                } else acc[n][2 * e] *= s.x, acc[n][2 * e + 1] *= s.x;
            }
        }
        if (__syncthreads_or(!ok)) break;
        if (c + 1 < nc) {
            if (threadIdx.x == 0) load_q(c + 1);
            values(c + 1);
        }
        // ---- 2: U = T R, one tile of 16 x 8 per warp
        {
            const int m = warp >> 2, n = warp & 3;
            float u[3][4] = {};
            const uint32_t* B = smu + L::RH + 2 * t * LU + n * 8 + g;
#pragma unroll 4
            for (int k = 0; k < 2 * (m + 1); ++k) {
                const uint32_t* A = sT + (tri_at(k, m * 16 + g)) * 8 + 2 * t;
                const uint2 lo = *reinterpret_cast<const uint2*>(A), hi = *reinterpret_cast<const uint2*>(A + 64);
                const uint2 lol = *reinterpret_cast<const uint2*>(A + TRI), hil = *reinterpret_cast<const uint2*>(A + TRI + 64);
                const uint32_t ah[4] = {lo.x, hi.x, lo.y, hi.y}, al[4] = {lol.x, hil.x, lol.y, hil.y};
                const uint32_t b0h = B[k * 8 * LU], b1h = B[k * 8 * LU + LU], b0l = B[L::RL - L::RH + k * 8 * LU], b1l = B[L::RL - L::RH + k * 8 * LU + LU];
                mma_tf32(u[0], ah, b0h, b1h);
                mma_tf32(u[1], ah, b0l, b1l);
                mma_tf32(u[2], al, b0h, b1h);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = m * 16 + g + 8 * e;
                const float x = u[0][2 * e] + (u[1][2 * e] + u[2][2 * e]), y = u[0][2 * e + 1] + (u[1][2 * e + 1] + u[2][2 * e + 1]), ks = scale[r].y;
                *reinterpret_cast<uint2*>(smu + L::U + r * LU + n * 8 + 2 * t) = make_uint2(tf32(x), tf32(y));
                *reinterpret_cast<uint2*>(smu + L::KU + r * LKU + n * 8 + 2 * t) = make_uint2(tf32(ks * x), tf32(ks * y));
            }
        }
        __syncthreads();
        if (keys) {                        // ---- 3: S = gamma S + (ks U)^T K (tokens t and t + 4 of a slab of eight)
#pragma unroll
            for (int n = 0; n < NB; ++n)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[n][m][e] *= gam;
            const uint32_t* A = smu + L::KU + t * LKU + g;
            const uint32_t* B = sK + (warp * NB * GC + t) * 8 + g;
#pragma unroll 4
            for (int k0 = 0; k0 < GC; k0 += 8) {
                uint32_t af[2][4];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    af[m][0] = A[k0 * LKU + m * 16];
                    af[m][1] = A[k0 * LKU + m * 16 + 8];
                    af[m][2] = A[(k0 + 4) * LKU + m * 16];
                    af[m][3] = A[(k0 + 4) * LKU + m * 16 + 8];
                }
#pragma unroll
                for (int n = 0; n < NB; ++n) {
                    const uint32_t b0 = B[(n * GC + k0) * 8], b1 = B[(n * GC + k0 + 4) * 8];
                    mma_tf32(S[n][0], af[0], b0, b1);
                    mma_tf32(S[n][1], af[1], b0, b1);
                }
            }
#pragma unroll
            for (int n = 0; n < NB; ++n)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        *reinterpret_cast<uint2*>(smu + L::S + ((warp * NB + n) * DVS + m * 16 + g + 8 * e) * 8 + 2 * t) =
                            make_uint2(tf32(S[n][m][2 * e]), tf32(S[n][m][2 * e + 1]));
        } else {                           // ---- and O = O + P U
            const uint32_t* B = smu + L::U + 2 * t * LU + n1 * 8 + g;
#pragma unroll 4
            for (int k = 0; k < 2 * (mt + 1); ++k) {
                const uint32_t* A = sP + tri_at(k, mt * 16 + g) * 8 + 2 * t;
                const uint2 lo = *reinterpret_cast<const uint2*>(A), hi = *reinterpret_cast<const uint2*>(A + 64);
                const uint32_t af[4] = {lo.x, hi.x, lo.y, hi.y};
                mma_tf32(acc[0], af, B[k * 8 * LU], B[k * 8 * LU + LU]);
                mma_tf32(acc[1], af, B[k * 8 * LU + 8], B[k * 8 * LU + LU + 8]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float* op = a.out + ((ch0 + c) * GC + mt * 16 + g + 8 * e) * a.Dv + dv0 + n1 * 8 + 2 * t;
                *reinterpret_cast<float2*>(op) = make_float2(acc[0][2 * e], acc[0][2 * e + 1]);
                *reinterpret_cast<float2*>(op + 8) = make_float2(acc[1][2 * e], acc[1][2 * e + 1]);
            }
        }
        __syncthreads();
    }
    if (c < nc && threadIdx.x == 0) {      // a wait gave up: this chunk's copies and the next one's may be on their way, and land before the CTA leaves
        atomicExch(a.status, 6);           // (unless that takes longer than a wait's limit)
        bool given_up = false;
        tc::settle(&full[c & 1], (c >> 1) & 1, given_up);
        tc::settle(&full[2], c & 1, given_up);
        if (c + 1 < nc) tc::settle(&full[(c + 1) & 1], ((c + 1) >> 1) & 1, given_up);
    }
    if (keys) {
#pragma unroll
        for (int n = 0; n < NB; ++n)
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<float2*>(Sg + (long)(m * 16 + g + 8 * e) * DK + (warp * NB + n) * 8 + 2 * t) =
                        make_float2(S[n][m][2 * e], S[n][m][2 * e + 1]);
    }
}

// Gated output: core [B * Hv, nc, 64, Dv] -> out[t, h * Dv + d] = rmsnorm(core) * norm_w[d] * silu(z[t, h * Dv + d]) (bf16).
struct GdnFinishArgs {
    const float* core; const void* z; long z_s; int z_f32;
    const float* norm_w; const int* cu_q;
    bf16* out; long out_s;
    int Hv, Dv, B, nc;
    float eps;
};

// A lane holds V neighbouring columns of a row, four rows are asked for at a time.  Bound by memory: a row is read once and written once.
template <int V, typename Z>
__global__ void __launch_bounds__(256) gdn_chunk_finish_kernel(GdnFinishArgs a) {
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / a.Hv, h = bh % a.Hv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = a.cu_q[b], left = min(GC, a.cu_q[b + 1] - row0 - c * GC), Dv = a.Dv;
    const float* core = a.core + ((long)bh * a.nc + c) * GC * Dv;
    constexpr int IT = V == 4 ? 2 : 8;                         // of 32 V columns: Dv up to 256
    const int its = (Dv + 32 * V - 1) / (32 * V);
    for (int r0 = warp * 8; r0 < min(left, warp * 8 + 8); r0 += 4) {
        {
            float x[4][IT][V], z[4][IT][V];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < IT; ++k) {
                    const int d = (k * 32 + lane) * V;
#pragma unroll
                    for (int e = 0; e < V; ++e) x[i][k][e] = z[i][k][e] = 0.f;
                    if (k >= its || d >= Dv || r0 + i >= left) continue;
                    const long zi = ((long)row0 + c * GC + r0 + i) * a.z_s + (long)h * Dv + d;
                    const Z* zp = reinterpret_cast<const Z*>(a.z) + zi;
                    if (V == 4) {
                        const float4 y = *reinterpret_cast<const float4*>(core + (long)(r0 + i) * Dv + d);
                        x[i][k][0] = y.x, x[i][k][1 % V] = y.y, x[i][k][2 % V] = y.z, x[i][k][3 % V] = y.w;
                        if (sizeof(Z) == 4) {
                            const float4 w = *reinterpret_cast<const float4*>(zp);
                            z[i][k][0] = w.x, z[i][k][1 % V] = w.y, z[i][k][2 % V] = w.z, z[i][k][3 % V] = w.w;
                        } else {
                            const uint2 w = *reinterpret_cast<const uint2*>(zp);
                            const bf16* wb = reinterpret_cast<const bf16*>(&w);
#pragma unroll
                            for (int e = 0; e < V; ++e) z[i][k][e] = bf2f(wb[e]);
                        }
                    } else {
                        x[i][k][0] = core[(long)(r0 + i) * Dv + d];
                        z[i][k][0] = sizeof(Z) == 4 ? *reinterpret_cast<const float*>(zp) : bf2f(*reinterpret_cast<const bf16*>(zp));
                    }
                }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float ss = 0.f;
#pragma unroll
                for (int k = 0; k < IT; ++k)
#pragma unroll
                    for (int e = 0; e < V; ++e) ss += x[i][k][e] * x[i][k][e];
                const float rs = rsqrtf(warp_sum(ss) / (float)Dv + a.eps);
                if (r0 + i >= left) continue;
#pragma unroll
                for (int k = 0; k < IT; ++k) {
                    const int d = (k * 32 + lane) * V;
                    if (k >= its || d >= Dv) continue;
                    bf16 y[V];
#pragma unroll
                    for (int e = 0; e < V; ++e) y[e] = f2bf(x[i][k][e] * rs * a.norm_w[d + e] * (z[i][k][e] / (1.f + __expf(-z[i][k][e]))));
                    bf16* op = a.out + ((long)row0 + c * GC + r0 + i) * a.out_s + (long)h * Dv + d;
                    if (V == 4) *reinterpret_cast<uint2*>(op) = *reinterpret_cast<const uint2*>(y);
                    else *op = y[0];
                }
            }
        }
    }
}

template <int DK>
static int launch_prep(const GdnPrepArgs& a, cudaStream_t s) {
    const size_t smem = sizeof(float) * ((size_t)PrepLay<DK>::fixed + 2 * (size_t)((a.Hv + a.Hk - 1) / a.Hk) * GC);
    TSB_CHECK_ARG(smem <= 226 * 1024, "gdn_chunk_prep: %d value heads for %d key heads", a.Hv, a.Hk);
    static bool configured = false;
    if (!configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gdn_chunk_prep_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gdn_chunk_scan_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(ScanLay<DK>::floats * sizeof(float))));
        configured = true;
    }
    gdn_chunk_prep_kernel<DK><<<dim3(a.nc, a.B * a.Hk), 256, smem, s>>>(a);
    TSB_CHECK_LAUNCH();
    gdn_chunk_scan_kernel<DK><<<dim3(a.Dv / DVS, a.B * a.Hv), 512, ScanLay<DK>::floats * sizeof(float), s>>>(a);
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

// The chunk-parallel kernel and the one that carries the state, for a packed batch; `out` [B Hv, nc, 64, Dv], nc chunks of 64 for the longest sequence.
extern "C" int tsb_gdn_chunks(const GdnPrepArgs* args, void* stream) {
    TSB_CHECK_ARG(args != nullptr, "gdn_chunks: null arguments");
    const GdnPrepArgs& a = *args;
    TSB_CHECK_ARG(a.B > 0 && a.nc > 0 && a.Hv > 0 && a.Hk > 0, "gdn_chunks: B=%d chunks=%d heads=%d/%d", a.B, a.nc, a.Hk, a.Hv);
    TSB_CHECK_ARG(a.Dv % DVS == 0 && a.Dv > 0 && a.Dv <= 128, "gdn_chunks: value head size %d (multiples of 32 up to 128)", a.Dv);
    TSB_CHECK_ARG((long)a.B * a.Hv <= 65535 && (long)a.B * a.Hk <= 65535, "gdn_chunks: %d x %d sequence-heads exceed the grid", a.B, a.Hv);
    TSB_CHECK_ARG(a.status != nullptr, "gdn_chunks: status word is required");
    TSB_CHECK_ARG(a.qkv_s % 4 == 0 && (reinterpret_cast<uintptr_t>(a.qkv) & 15) == 0, "gdn_chunks: rows must start on 16 bytes");
    switch (a.Dk) {
    case 64: return launch_prep<64>(a, (cudaStream_t)stream);
    case 128: return launch_prep<128>(a, (cudaStream_t)stream);
    default:
        tsb_set_error("gdn_chunks: key head size %d unsupported (64, 128)", a.Dk);
        return TSB_ERR_UNSUPPORTED;
    }
}

// ------------------------------------------------------------------------------------------
// Mamba2 in chunked (state-space duality) form: the chunk-parallel part for one (sequence, head, chunk).  With
// d = softplus(dt + bias), log-decay c = cumsum(d * A) inside the chunk, inputs X = d * x, and the group's B / C rows:
//   U0 = X                       what a token writes
//   Qd = C * exp(c)              reads of the state entering the chunk
//   Kd = B * exp(c_last - c)     writes that survive to the chunk's end
//   P  = (C B^T) * exp(c_i - c_j) for j <= i, else 0        contributions inside the chunk
//   gamma = exp(c_last)
// which is exactly what gdn_chunk_carry_kernel consumes with W = 0: out = Qd S^T + P U0, S <- gamma S + U0^T Kd.
// Reference: the ssm_scan path of ggml (ggml-cuda/ssm-scan.cu) is a token-by-token scan; the chunked form is this
// framework's own.
// ------------------------------------------------------------------------------------------
struct MambaPrepArgs {
    const float* xbc; long xbc_s;          // [T, H Pd + 2 G N] rows: x heads | B groups | C groups
    const void* dt; long dt_s; int dt_f32; // [T, H]
    const float* dt_bias; const float* A;  // [H] (dt_bias may be null)
    const int* cu_q;                       // [B + 1]
    float* U0; float* Qd; float* Kd; float* P; float* gamma;
    int H, Pd, G, N, B, nc;
};

template <int DK>
__global__ void __launch_bounds__(256) mamba2_chunk_prep_kernel(MambaPrepArgs a) {
    constexpr int LQ = DK + 4;
    extern __shared__ __align__(16) float sm[];
    float* sK = sm;                        // [64][LQ] B rows
    float* sQ = sK + GC * LQ;              // [64][LQ] C rows
    float* sc = sQ + GC * LQ;              // [64] running log-decay
    float* sd = sc + GC;                   // [64] step size d
    const int c = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H, grp = h / (a.H / a.G);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = a.cu_q[b], len = a.cu_q[b + 1] - row0;
    const int valid = max(0, min(GC, len - c * GC));
    const long tok0 = (long)row0 + (long)c * GC;
    const long ch = (long)bh * a.nc + c;
    const int Pd = a.Pd;
    const long offB = (long)a.H * Pd + (long)grp * DK, offC = offB + (long)a.G * DK;
    for (int r = warp; r < GC; r += 8) {
        const bool ok = r < valid;
        const float* row = a.xbc + (tok0 + r) * a.xbc_s;
#pragma unroll
        for (int i = 0; i < DK / 32; ++i) {
            sK[r * LQ + lane + 32 * i] = ok ? row[offB + lane + 32 * i] : 0.f;
            sQ[r * LQ + lane + 32 * i] = ok ? row[offC + lane + 32 * i] : 0.f;
        }
        float d = 0.f;
        if (ok) {
            const long di = (tok0 + r) * a.dt_s + h;
            const float v = (a.dt_f32 ? reinterpret_cast<const float*>(a.dt)[di] : bf2f(reinterpret_cast<const bf16*>(a.dt)[di])) +
                            (a.dt_bias ? a.dt_bias[h] : 0.f);
            d = v > 20.f ? v : log1pf(__expf(v));
        }
        for (int e = lane; e < Pd; e += 32) a.U0[(ch * GC + r) * Pd + e] = ok ? row[(long)h * Pd + e] * d : 0.f;
        if (lane == 0) {
            sd[r] = d;
            sc[r] = d * a.A[h];
        }
    }
    __syncthreads();
    if (warp == 0) {                       // inclusive running sum over the 64 tokens
        float x0 = sc[lane], x1 = sc[lane + 32];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y0 = __shfl_up_sync(0xffffffffu, x0, o), y1 = __shfl_up_sync(0xffffffffu, x1, o);
            if (lane >= o) { x0 += y0; x1 += y1; }
        }
        x1 += __shfl_sync(0xffffffffu, x0, 31);
        sc[lane] = x0;
        sc[lane + 32] = x1;
    }
    __syncthreads();
    const float c_last = sc[GC - 1];
    // ---- C B^T: warp -> rows mt * 16 .. + 15, columns nq * 32 .. + 31 (split tf32: three products per term)
    {
        const int g = lane >> 2, t = lane & 3, mt = warp & 3, nq = warp >> 2;
        float qk[4][4] = {};
#pragma unroll 2
        for (int k0 = 0; k0 < DK; k0 += 8) {
            uint32_t qh[4], ql[4];
            const float* qp = sQ + (mt * 16 + g) * LQ + k0 + t;
            split_tf32(qp[0], qh[0], ql[0]); split_tf32(qp[8 * LQ], qh[1], ql[1]);
            split_tf32(qp[4], qh[2], ql[2]); split_tf32(qp[8 * LQ + 4], qh[3], ql[3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float* bp = sK + ((nq * 4 + j) * 8 + g) * LQ + k0 + t;
                uint32_t b0h, b0l, b1h, b1l;
                split_tf32(bp[0], b0h, b0l);
                split_tf32(bp[4], b1h, b1l);
                mma_tf32(qk[j], ql, b0h, b1h); mma_tf32(qk[j], qh, b0l, b1l); mma_tf32(qk[j], qh, b0h, b1h);
            }
        }
        float* Pg = a.P + ch * GC * GC;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = mt * 16 + g + (e >> 1) * 8, jj = (nq * 4 + j) * 8 + 2 * t + (e & 1);
                Pg[i * GC + jj] = jj <= i ? qk[j][e] * __expf(fminf(sc[i] - sc[jj], 0.f)) : 0.f;
            }
        }
    }
    for (int r = warp; r < GC; r += 8) {
        const float dec = __expf(sc[r]), tail = __expf(c_last - sc[r]);
#pragma unroll
        for (int i = 0; i < DK / 32; ++i) {
            const int d = lane + 32 * i;
            a.Kd[(ch * GC + r) * DK + d] = sK[r * LQ + d] * tail;
            a.Qd[(ch * GC + r) * DK + d] = sQ[r * LQ + d] * dec;
        }
    }
    if (threadIdx.x == 0) a.gamma[ch] = __expf(c_last);
}

template <int DK>
static int launch_mamba_prep(const MambaPrepArgs& a, cudaStream_t s) {
    const size_t smem = ((size_t)2 * GC * (DK + 4) + 2 * GC) * sizeof(float);
    static size_t configured = 0;
    if (smem > configured) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(mamba2_chunk_prep_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    mamba2_chunk_prep_kernel<DK><<<dim3(a.nc, a.B * a.H), 256, smem, s>>>(a);
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

extern "C" int tsb_mamba2_chunk_prep(const MambaPrepArgs* args, void* stream) {
    TSB_CHECK_ARG(args != nullptr, "mamba2_chunk_prep: null arguments");
    const MambaPrepArgs& a = *args;
    TSB_CHECK_ARG(a.B > 0 && a.nc > 0 && a.H > 0 && a.G > 0 && a.H % a.G == 0, "mamba2_chunk_prep: B=%d chunks=%d heads=%d groups=%d", a.B, a.nc,
                  a.H, a.G);
    TSB_CHECK_ARG(a.Pd > 0, "mamba2_chunk_prep: head size %d", a.Pd);
    TSB_CHECK_ARG((long)a.B * a.H <= 65535, "mamba2_chunk_prep: %d x %d sequence-heads exceed the grid", a.B, a.H);
    switch (a.N) {
    case 64: return launch_mamba_prep<64>(a, (cudaStream_t)stream);
    case 128: return launch_mamba_prep<128>(a, (cudaStream_t)stream);
    default:
        tsb_set_error("mamba2_chunk_prep: state size %d unsupported (64, 128)", a.N);
        return TSB_ERR_UNSUPPORTED;
    }
}

extern "C" int tsb_gdn_chunk_finish(const GdnFinishArgs* args, void* stream) {
    TSB_CHECK_ARG(args != nullptr, "gdn_chunk_finish: null arguments");
    const GdnFinishArgs& a = *args;
    TSB_CHECK_ARG(a.Dv > 0 && a.Dv <= 256 && a.B > 0 && a.nc > 0, "gdn_chunk_finish: Dv=%d B=%d chunks=%d", a.Dv, a.B, a.nc);
    TSB_CHECK_ARG((long)a.B * a.Hv <= 65535, "gdn_chunk_finish: %d x %d sequence-heads exceed the grid", a.B, a.Hv);
    // four columns at a time where every row of z and out starts on four of its own
    const uintptr_t zb = reinterpret_cast<uintptr_t>(a.z), ob = reinterpret_cast<uintptr_t>(a.out);
    const bool wide = a.Dv % 4 == 0 && a.z_s % 4 == 0 && a.out_s % 4 == 0 && zb % (a.z_f32 ? 16 : 8) == 0 && ob % 8 == 0;
    const dim3 grid(a.nc, a.B * a.Hv);
    cudaStream_t s = (cudaStream_t)stream;
    if (wide && a.z_f32) gdn_chunk_finish_kernel<4, float><<<grid, 256, 0, s>>>(a);
    else if (wide) gdn_chunk_finish_kernel<4, bf16><<<grid, 256, 0, s>>>(a);
    else if (a.z_f32) gdn_chunk_finish_kernel<1, float><<<grid, 256, 0, s>>>(a);
    else gdn_chunk_finish_kernel<1, bf16><<<grid, 256, 0, s>>>(a);
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}
