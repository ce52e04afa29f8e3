// Decode GEMV for Q4_K / Q5_K weights with a deep asynchronous row pipeline.
//
// The one-warp-per-row GEMV keeps two 16-byte loads per lane in flight; with rows of 1.4 KB (K = 2560)
// a warp's whole life is three such round trips, and the launch runs as four waves of short-lived
// CTAs: measured 17.7 us for the 28 MB gate/up matrix of a Qwen3-4B layer (4.3 us at the copy rate).
// Here a warp owns a contiguous range of row pairs and streams them through a ring of D row buffers
// in shared memory filled by cp.async (coalesced 16-byte copies of the row's contiguous GGUF blocks),
// so D - 1 whole rows per warp are in flight all the time (about 10 KB per warp, 150 KB per SM), the
// first rows are requested before the kernel waits for its predecessor, and the grid is one wave.
// The block arithmetic is the same comp_q45k as the plain kernel, fed from shared memory.
//
// Same contract as gemv_kernel without expert ids and without the tensor-parallel push: bias, gated
// activation over (row r, row r + N/2), ReLU^2, row scale, residual, f32 or bf16 output; M <= 4.
// Replaces mul_mat_vec_q + quantize_q8_1 of the reference (ggml-cuda/mmvq.cu:143) for these types.
#include <cstdlib>
#include "gemv_core.cuh"

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gsrc) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int M, bool GLU, bool Q5, int D>
__global__ void __launch_bounds__(128) gemv_stream_kernel(GemvArgs a, int ppw) {
    extern __shared__ uint4 stream_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int K = a.w.K, nb = K >> 8;
    constexpr int BLK16 = Q5 ? 11 : 9;                 // 16-byte chunks per 256-value block
    const int chunks = nb * BLK16;                     // per row
    uint4* ring = stream_smem + (long)warp * D * chunks;
    const int N = a.w.N, n_out = a.n_out;
    const int n_pairs = GLU ? n_out : (N + 1) / 2;
    const int p0 = (blockIdx.x * 4 + warp) * ppw, p1 = min(n_pairs, p0 + ppw);
    const int ntask = p1 > p0 ? 2 * (p1 - p0) : 0;

    auto task_row = [&](int i) -> int {                // weight row of task i, or -1
        const int pair = p0 + (i >> 1), which = i & 1;
        if (GLU) return which ? pair + n_out : pair;
        const int r = 2 * pair + which;
        return r < N ? r : -1;
    };
    auto issue = [&](int i) {
        if (i < ntask) {
            const int r = task_row(i);
            if (r >= 0) {
                const uint4* src = reinterpret_cast<const uint4*>(a.w.p0) + (long)r * chunks;
                uint4* dst = ring + (long)(i % D) * chunks;
                for (int c = lane; c < chunks; c += 32) cp_async16(dst + c, src + c);
            }
        }
        cp_async_commit();                             // one group per task, empty or not: the wait below counts groups
    };
#pragma unroll
    for (int i = 0; i < D - 1; ++i) issue(i);          // weights never change: requested before the dependency wait
    pdl_wait();
    pdl_trigger();

    float keep[M];                                     // gate result (GLU) while the up row is computed
#pragma unroll
    for (int m = 0; m < M; ++m) keep[m] = 0.f;
    const int mv = min(M, a.M);
    const int units = nb << 3;
    for (int i = 0; i < ntask; ++i) {
        issue(i + D - 1);
        cp_async_wait<D - 1>();
        __syncwarp();
        const int r = task_row(i);
        float acc[M];
#pragma unroll
        for (int m = 0; m < M; ++m) acc[m] = 0.f;
        if (r >= 0) {
            const uint4* st = ring + (long)(i % D) * chunks;
            for (int u = lane; u < units; u += 32) {
                const int b = u >> 3, uu = u & 7;
                WQ4K t;
                t.hdr = st[b * BLK16];
                if (Q5) {
                    t.hv = st[b * BLK16 + 1 + (uu & 1)];
                    t.qv = st[b * BLK16 + 3 + uu];
                } else {
                    t.qv = st[b * BLK16 + 1 + uu];
                }
                comp_q45k<M, Q5>(a.w, t, u, a.xq, a.xds, acc, mv);
            }
#pragma unroll
            for (int m = 0; m < M; ++m) acc[m] = warp_sum(acc[m]);
        }
        __syncwarp();                                  // every lane is done with this buffer before it is refilled
        if (GLU && !(i & 1)) {
#pragma unroll
            for (int m = 0; m < M; ++m) keep[m] = acc[m];
            continue;
        }
        if (lane != 0 || r < 0) continue;
        const int orow_col = GLU ? p0 + (i >> 1) : r;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            if (m >= mv) break;
            float v;
            if (GLU) {
                float g = keep[m], up = acc[m];
                if (a.bias) { g += a.bias[orow_col]; up += a.bias[orow_col + n_out]; }
                v = act_glu(a.act, g, up);
            } else {
                v = acc[m];
                if (a.bias) v += a.bias[orow_col];
                if (a.act == ACT_RELU2) { v = fmaxf(v, 0.f); v = v * v; }
            }
            if (a.row_scale) v *= a.row_scale[m];
            const long o = (long)m * n_out + orow_col;
            if (a.out_f32) {
                if (a.residual) v += reinterpret_cast<const float*>(a.residual)[o];
                reinterpret_cast<float*>(a.out)[o] = v;
            } else {
                if (a.residual) v += bf2f(reinterpret_cast<const bf16*>(a.residual)[o]);
                reinterpret_cast<bf16*>(a.out)[o] = f2bf(v);
            }
        }
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------------------------
// Single-token Q4_K, Q6_K and Q8_0: rows of a matrix in groups of R, 32 / R lanes to a row.
//
// At one activation row the bound is the bytes of the weights, and what kept the kernel from it was the
// instruction issue: with a row per warp and units of 32 values the Q4_K form spent 4.2 thread instructions
// a value (6.2 the Q6_K form, whose byte-wise subtraction alone is a fifth of that), issue slots 57 to 63 %
// busy at 40 % of the copy rate.  Here a unit is 64 values (a pair of Q4_K sub-blocks; 16 of each of the
// four bit planes of half a Q6_K block), so headers, scales and conversions are paid half as often; the
// activations of a lane's units are the same for every group and stay in registers; a unit's shared-memory
// offset is the first one's plus a constant; the sum over lanes takes 3 or 4 exchanges for R rows instead
// of 5 for one.  The high nibbles of Q4_K are multiplied where they stand (bytes times 16, shifted back once
// per unit, exactly); the offset 32 of Q6_K is the starting value of the integer sum, together with the bits
// that make the sum readable as a float.  All integer sums are exact, so R and the split change rounding only
// in the order of the float additions.
//
// Each warp streams its groups through a ring of D stages in shared memory (cp.async, the first D - 1 before
// the dependency wait: weights never change), so most of the matrix of a decode projection is on its way
// when the kernel starts.  KS = 4 (rows longer than 6144 values): the four warps of a CTA split every row by
// blocks and the partial sums meet in shared memory, one barrier per group.
// Measured (us, weights of several matrices in turn, before / after): 2 x 9728 x 2560 10.5 / 6.8, 2560 x 9728 7.3 / 4.7, Q6_K 7.3 / 6.3, 32768 x 2560
// Q6_K 24.0 / 13.4 (5.2 TB/s), 151936 x 2560 64.9 / 36.5, Q6_K 100 / 56; Q8_0, which has little to decode but kept two 16-byte loads a lane in flight:
// 2 x 21504 x 5376 44.7 / 40.1 (6.1 TB/s), 5376 x 21504 27.4 / 20.4, 5376 x 4096 7.0 / 5.3, 8192 x 5376 11.7 / 8.3.  What is left of the short ones is latency: activations through L2 after the
// wait, one group's arithmetic, the tail.  Three stages or two CTAs an SM measured slower, 128 registers (four CTAs) too: the units no longer overlap.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int dp4a_us(unsigned a, int b, int c) {      // unsigned bytes of a times signed bytes of b
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
constexpr int MAGIC_I = 0x4B400000;                                      // as a float 1.5 * 2^23: integers below 2^22 in magnitude added to these bits
constexpr float MAGIC_F = 12582912.f;                                    // are read back by one float subtraction
enum { ROWS_Q4, ROWS_Q6, ROWS_Q8 };
__host__ __device__ constexpr int rows_block_bytes(int ty) { return ty == ROWS_Q4 ? 144 : ty == ROWS_Q6 ? 210 : 272; }
constexpr int ROWS_D = 2, ROWS_PER_SM = 3;                             // stages of a warp, CTAs of an SM

// Blocks [first, end) of a row that a warp owns; even boundaries keep the 2-byte super-scales of Q6_K 4-byte aligned for cp.async
template <int TY, int KS>
__host__ __device__ __forceinline__ int rows_slice(int nb, int warp) {
    if (KS == 1) return warp ? nb : 0;
    return warp >= KS ? nb : TY == ROWS_Q6 ? ((nb * warp) / KS) & ~1 : (nb * warp) / KS;
}

// n chunks of 16 bytes (at most MOST, so that the loop unrolls to a compare and a copy each), lane by lane
template <int MOST>
__device__ __forceinline__ void rows_copy(uint8_t* dst, const uint8_t* src, int n, int lane) {
#pragma unroll
    for (int i = 0; i < (MOST + 31) / 32; ++i)
        if (lane + 32 * i < n) cp_async16(dst + 512 * i, src + 512 * i);
}

template <int TY, bool GLU, int R, int J, int KS>
__device__ __forceinline__ void rows_body(const GemvArgs& a, uint8_t* rows_smem, int stage_bytes, int n_groups, int block, int blocks) {
    __shared__ float part[2][4][R];
    constexpr bool Q4 = TY == ROWS_Q4, Q6 = TY == ROWS_Q6;
    constexpr int L = 32 / R, H = R / 2, D = ROWS_D;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = a.w.K >> 8;
    const int bs = rows_slice<TY, KS>(nb, KS == 1 ? 0 : warp), nblk = rows_slice<TY, KS>(nb, KS == 1 ? 1 : warp + 1) - bs;
    uint8_t* ring = rows_smem + (long)warp * D * stage_bytes;
    const int n_out = a.n_out;
    const int owner = KS == 1 ? block * 4 + warp : block, owners = KS == 1 ? blocks * 4 : blocks;
    const int t0 = (int)((long)n_groups * owner / owners), ntask = (int)((long)n_groups * (owner + 1) / owners) - t0;

    // n blocks (at most MOST) from block `sb` of the matrix to block `db` of a stage
    constexpr int MOST = (KS == 1 ? (GLU ? H : R) : 1) * (L / 4) * J;
    const int o_qh = R * nblk * 128, o_sc = R * nblk * 192, o_d = R * nblk * 208;
    // against bank conflicts: the low nibbles of Q6_K lie with chunks 2 and 3 of four exchanged in odd blocks, the bytes of Q8_0 with the four chunks of
    // a unit permuted by the unit's number
    const int swz = Q6 ? lane ^ ((lane >> 2) & 2) : lane ^ ((lane >> 3) & 3);
    auto copy = [&](uint8_t* st, int db, long sb, int n) {
        if (Q4) {
            rows_copy<MOST * 9>(st + (db * 9 + lane) * 16, a.w.p0 + sb * 144 + lane * 16, n * 9, lane);
        } else if (Q6) {
            rows_copy<MOST * 8>(st + (db * 8 + swz) * 16, a.w.p0 + sb * 128 + lane * 16, n * 8, lane);
            rows_copy<MOST * 4>(st + o_qh + (db * 4 + lane) * 16, a.w.p1 + sb * 64 + lane * 16, n * 4, lane);
            rows_copy<MOST>(st + o_sc + (db + lane) * 16, a.w.p2 + sb * 16 + lane * 16, n, lane);
            static_assert(MOST <= 64, "one word of super-scales a lane");
            if (lane < n / 2) cp_async4(st + o_d + db * 2 + lane * 4, a.w.p3 + sb * 2 + lane * 4);
        } else {
            rows_copy<MOST * 16>(st + (db * 16 + swz) * 16, a.w.p0 + sb * 256 + lane * 16, n * 16, lane);
            rows_copy<MOST>(st + R * nblk * 256 + (db + lane) * 16, a.w.p1 + sb * 16 + lane * 16, n, lane);
        }
    };
    auto issue = [&](int t, int slot) {
        if (t < ntask) {
            uint8_t* st = ring + slot * stage_bytes;
            const int r0 = (t0 + t) * (GLU ? H : R);                    // first row, or first gate row; rows past the end are not fetched
            const int nr = min(GLU ? H : R, n_out - r0);
#pragma unroll
            for (int half = 0; half < (GLU ? 2 : 1); ++half) {
                const long r = r0 + (half ? n_out : 0);
                if (KS == 1) {
                    copy(st, half * H * nblk, r * nb, nr * nb);
                } else {
#pragma unroll
                    for (int i = 0; i < (GLU ? H : R); ++i)
                        if (i < nr) copy(st, (half * H + i) * nblk, (r + i) * nb + bs, nblk);
                }
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < D - 1; ++i) issue(i, i);
    pdl_wait();
    pdl_trigger();
    if (ntask == 0) { cp_async_wait<0>(); return; }

    // what a lane keeps of the activations for all groups: unit u = l + L j of its row, four units to a block
    const int i_row = lane / L, l = lane % L;
    const int units = nblk << 2, bl0 = l >> 2;
    const int c4 = l & 3, hb = l & 1;
    int x[J][16];
    float f[J][4];
    int init[Q6 ? J : 1][4];
    const bool last_ok = l + L * (J - 1) < units;                        // J is chosen so that only the last unit can lie past the row's (slice's) end
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const bool ok = j < J - 1 || last_ok;
        const int b = bs + (ok ? bl0 + (L / 4) * j : 0);
        const int xoff = b * 256 + (Q6 ? 128 * (c4 >> 1) + 16 * hb : 64 * c4), step = Q6 ? 32 : 16;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int4 v = *reinterpret_cast<const int4*>(a.xq + xoff + step * k);
            x[j][4 * k] = v.x; x[j][4 * k + 1] = v.y; x[j][4 * k + 2] = v.z; x[j][4 * k + 3] = v.w;
        }
        if (Q6) {
            const float4 e0 = *reinterpret_cast<const float4*>(a.xds + b * 8 + 4 * (c4 >> 1)), e1 = *reinterpret_cast<const float4*>(a.xds + b * 8 + 4 * (c4 >> 1) + 2);
            f[j][0] = e0.x; f[j][1] = e0.z; f[j][2] = e1.x; f[j][3] = e1.z;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int s = 0;
#pragma unroll
                for (int w = 0; w < 4; ++w) s = __dp4a(x[j][4 * k + w], 0x01010101, s);
                init[j][k] = MAGIC_I - 32 * s;
            }
        } else {
            const float4 e = *reinterpret_cast<const float4*>(a.xds + b * 8 + 2 * c4);
            f[j][0] = e.x; f[j][1] = e.z; f[j][2] = e.y; f[j][3] = e.w;   // scales of the two sub-blocks, then their sums
        }
        if (!ok) f[j][0] = f[j][1] = f[j][2] = f[j][3] = 0.f;
    }
    const unsigned sh = 16u * (c4 & 1);                                  // Q4_K: which of the packed 6-bit fields
    const bool hi = c4 >= 2;
    const uint32_t m_lo = hi ? 0x0F0Fu : 0x3F3Fu, m_hi = hi ? 0x3030u : 0u;
    const unsigned shq = sh + (hi ? 4u : 0u);
    const uint32_t sel0 = 0x7540u | hb, sel1 = 0x7542u | hb;             // Q6_K: bytes hb and hb + 2 of a word of scales
    const int xr = ((l >> 1) + (KS == 1 ? 2 * ((GLU ? i_row % H : i_row) * nblk & 1) : 0)) & 3;   // Q8_0: what permutes the chunks of a lane's units (copies count rows of a run on)
    const int off0 = !Q4 && !Q6 ? (i_row * nblk + bl0) * 256 + 64 * c4 : Q6 ? (i_row * nblk + bl0) * 128 + (((4 * (c4 >> 1) + hb) ^ (2 * (bl0 & 1))) << 4) : (i_row * nblk + bl0) * 144;
    const int off1 = Q6 ? off0 ^ 32 : off0 + 16 + 32 * c4;
    const int off5 = R * nblk * 256 + (i_row * nblk + bl0) * 16 + 4 * c4;
    const int off2 = o_qh + (i_row * nblk + bl0) * 64 + 16 * c4, off3 = o_sc + (i_row * nblk + bl0) * 16 + 8 * (c4 >> 1), off4 = o_d + (i_row * nblk + bl0) * 2;

    int slot = 0, next = D - 1;
    for (int t = 0; t < ntask; ++t) {
        issue(t + D - 1, next);
        // what the result is joined with is on its way while the sums are formed
        const int orow = (t0 + t) * (GLU ? H : R) + (KS == 1 ? i_row : lane);
        const bool writes = a.push == nullptr && orow < n_out && (KS == 1 ? l == 0 && (!GLU || i_row < H) : warp == 0 && lane < (GLU ? H : R));
        float res = 0.f, b0 = 0.f, b1 = 0.f;
        if (writes) {
            if (a.residual) res = a.out_f32 ? reinterpret_cast<const float*>(a.residual)[orow] : bf2f(reinterpret_cast<const bf16*>(a.residual)[orow]);
            if (a.bias) { b0 = a.bias[orow]; if (GLU) b1 = a.bias[orow + n_out]; }
        }
        cp_async_wait<D - 1>();
        __syncwarp();
        const uint8_t* st = ring + slot * stage_bytes;
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int bj = j < J - 1 || last_ok ? (L / 4) * j : -bl0;                   // lanes past the row's end read its first block and add zero
            if (Q6) {
                const uint4 la = *reinterpret_cast<const uint4*>(st + off0 + bj * 128), lb = *reinterpret_cast<const uint4*>(st + off1 + bj * 128);
                const uint4 hv = *reinterpret_cast<const uint4*>(st + off2 + bj * 64);
                uint2 sc = *reinterpret_cast<const uint2*>(st + off3 + bj * 16);
                const float d = __half2float(*reinterpret_cast<const __half*>(st + off4 + bj * 2));
                const uint32_t A[4] = {la.x, la.y, la.z, la.w}, B[4] = {lb.x, lb.y, lb.z, lb.w}, V[4] = {hv.x, hv.y, hv.z, hv.w};
                int s[4] = {init[j][0], init[j][1], init[j][2], init[j][3]};
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    s[0] = __dp4a((int)((A[w] & 0x0F0F0F0Fu) | ((V[w] << 4) & 0x30303030u)), x[j][w], s[0]);
                    s[1] = __dp4a((int)((B[w] & 0x0F0F0F0Fu) | ((V[w] << 2) & 0x30303030u)), x[j][4 + w], s[1]);
                    s[2] = __dp4a((int)(((A[w] >> 4) & 0x0F0F0F0Fu) | (V[w] & 0x30303030u)), x[j][8 + w], s[2]);
                    s[3] = __dp4a((int)(((B[w] >> 4) & 0x0F0F0F0Fu) | ((V[w] >> 2) & 0x30303030u)), x[j][12 + w], s[3]);
                }
                sc.x ^= 0x80808080u;                                     // int8 scales as bytes 128 higher
                sc.y ^= 0x80808080u;
                const uint32_t sb[4] = {__byte_perm(sc.x, 0x4B000000u, sel0), __byte_perm(sc.x, 0x4B000000u, sel1),
                                        __byte_perm(sc.y, 0x4B000000u, sel0), __byte_perm(sc.y, 0x4B000000u, sel1)};
                float v = 0.f;
#pragma unroll
                for (int k = 0; k < 4; ++k) v += (__int_as_float(s[k]) - MAGIC_F) * (__uint_as_float(sb[k]) - 8388736.f) * f[j][k];
                acc += d * v;
            } else if (!Q4) {
                int s[2] = {MAGIC_I, MAGIC_I};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 q = *reinterpret_cast<const uint4*>(st + off0 + bj * 256 + ((k ^ xr) << 4));
                    s[k >> 1] = __dp4a((int)q.x, x[j][4 * k], s[k >> 1]);
                    s[k >> 1] = __dp4a((int)q.y, x[j][4 * k + 1], s[k >> 1]);
                    s[k >> 1] = __dp4a((int)q.z, x[j][4 * k + 2], s[k >> 1]);
                    s[k >> 1] = __dp4a((int)q.w, x[j][4 * k + 3], s[k >> 1]);
                }
                const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(st + off5 + bj * 16));
                acc += dd.x * f[j][0] * (__int_as_float(s[0]) - MAGIC_F) + dd.y * f[j][1] * (__int_as_float(s[1]) - MAGIC_F);
            } else {
                const uint4 hdr = *reinterpret_cast<const uint4*>(st + off0 + bj * 144);
                const uint4 qa = *reinterpret_cast<const uint4*>(st + off1 + bj * 144), qb = *reinterpret_cast<const uint4*>(st + off1 + bj * 144 + 16);
                const uint32_t q[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
                int s0 = 0, s1 = 0;
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    s0 = __dp4a((int)(q[w] & 0x0F0F0F0Fu), x[j][w], s0);
                    s1 = dp4a_us(q[w] & 0xF0F0F0F0u, x[j][8 + w], s1);   // sixteen times the sum
                }
                s1 >>= 4;
                // 6-bit scales and minimums of sub-blocks 2c and 2c + 1 as byte pairs: two encodings, one set of masks and shifts
                const uint32_t Y = hdr.y, Z = hdr.z;
                const uint32_t P = (((hi ? hdr.w : Y) >> sh) & m_lo) | ((Y >> (sh + 2)) & m_hi);
                const uint32_t Q = (((hi ? hdr.w : Z) >> shq) & m_lo) | ((Z >> (sh + 2)) & m_hi);
                const float p0 = __int_as_float(s0 * (int)(P & 0xFFu) + MAGIC_I) - MAGIC_F, p1 = __int_as_float(s1 * (int)(P >> 8) + MAGIC_I) - MAGIC_F;
                const float n0 = __uint_as_float(__byte_perm(Q, 0x4B000000u, 0x7540u)) - 8388608.f, n1 = __uint_as_float(__byte_perm(Q, 0x4B000000u, 0x7541u)) - 8388608.f;
                const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(&hdr.x));
                acc += dd.x * (p0 * f[j][0] + p1 * f[j][1]) - dd.y * (n0 * f[j][2] + n1 * f[j][3]);
            }
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        __syncwarp();                                                    // every lane is done with the stage before it is filled again
        slot = slot == D - 1 ? 0 : slot + 1;
        next = next == D - 1 ? 0 : next + 1;
        float up = 0.f;
        if (KS > 1) {
            if (l == 0) part[t & 1][warp][i_row] = acc;
            __syncthreads();
            if (warp != 0) continue;
            const float(*pt)[R] = part[t & 1];
            const int i = lane & (R - 1);
            acc = pt[0][i] + pt[1][i] + pt[2][i] + pt[3][i];
            if (GLU) up = __shfl_xor_sync(0xffffffffu, acc, H);
        } else if (GLU) {
            up = __shfl_xor_sync(0xffffffffu, acc, 16);
        }
        if (!GLU && a.push != nullptr) {
            // row-parallel projection of a tensor-parallel layer: lane q stores the sum, tagged with the exchange number, into rank q's mailbox
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float v = __shfl_sync(0xffffffffu, acc, KS == 1 ? i * L : i);
                const int r = (t0 + t) * R + i;
                if (r < n_out) gemv_push_store(a.push, lane, r, (a.bias && a.push->rank == 0) ? v + a.bias[r] : v);
            }
            continue;
        }
        if (!writes) continue;
        float v;
        if (GLU) {
            v = act_glu(a.act, acc + b0, up + b1);
        } else {
            v = acc + b0;
            if (a.act == ACT_RELU2) { v = fmaxf(v, 0.f); v = v * v; }
        }
        if (a.row_scale) v *= a.row_scale[0];
        v += res;
        if (a.out_f32) reinterpret_cast<float*>(a.out)[orow] = v;
        else reinterpret_cast<bf16*>(a.out)[orow] = f2bf(v);
    }
    cp_async_wait<0>();
}


template <int TY, bool GLU, int R, int J, int KS>
__global__ void __launch_bounds__(128, ROWS_PER_SM) gemv_rows_kernel(GemvArgs a, int stage_bytes, int n_groups) {
    extern __shared__ __align__(128) uint8_t rows_smem[];
    rows_body<TY, GLU, R, J, KS>(a, rows_smem, stage_bytes, n_groups, blockIdx.x, gridDim.x);
}

// Two or three matrices over the same activations (query, key and value rows of mixed types): each has the CTAs that its share of the bytes asks for.
// Q4_K 4096 + Q4_K 1024 + Q6_K 1024 rows of 2560 values in a decode step: 6.3 us with a row per warp and the general arithmetic, 4.3 so.
template <int J>
__global__ void __launch_bounds__(128, ROWS_PER_SM) gemv_rows_multi_kernel(GemvMultiArgs m, int stage_bytes, int end0, int end1) {
    extern __shared__ __align__(128) uint8_t rows_smem[];
    const int b = blockIdx.x, wi = b < end0 ? 0 : b < end1 ? 1 : 2, first = wi == 0 ? 0 : wi == 1 ? end0 : end1;
    const int blocks = (wi == 0 ? end0 : wi == 1 ? end1 : (int)gridDim.x) - first, row0 = wi ? m.row_end[wi - 1] : 0;
    GemvArgs a{};
    a.w = m.w[wi];
    a.xq = m.xq; a.xds = m.xds; a.M = 1; a.out_f32 = m.out_f32; a.n_out = a.w.N;
    a.out = m.out_f32 ? (void*)(reinterpret_cast<float*>(m.out) + row0) : (void*)(reinterpret_cast<bf16*>(m.out) + row0);
    const int n_groups = (a.n_out + 1) / 2;
    if (a.w.type == TSB_Q6_K) rows_body<ROWS_Q6, false, 2, J, 1>(a, rows_smem, stage_bytes, n_groups, b - first, blocks);
    else rows_body<ROWS_Q4, false, 2, J, 1>(a, rows_smem, stage_bytes, n_groups, b - first, blocks);
}

template <int J>
static int launch_rows_multi(const GemvMultiArgs& m, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemv_rows_multi_kernel<J>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr = true;
    }
    const int nb = m.w[0].K >> 8, stage_bytes = (2 * nb * 210 + 127) & ~127;
    const size_t smem = (size_t)stage_bytes * ROWS_D * 4;
    const int fit = (int)((226 * 1024) / (smem + 1024)), most = 148 * (fit < 1 ? 1 : fit > ROWS_PER_SM ? ROWS_PER_SM : fit);
    long bytes[3], sum = 0;
    for (int i = 0; i < 3; ++i) sum += bytes[i] = i < m.n_w ? (long)m.w[i].N * (m.w[i].type == TSB_Q6_K ? 210 : 144) : 0;
    int end[3], at = 0;
    for (int i = 0; i < 3; ++i) end[i] = at += i < m.n_w ? max(1, (int)(most * bytes[i] / sum)) : 0;
    TSB_CHECK_CUDA(tsb_launch(gemv_rows_multi_kernel<J>, dim3(end[2]), dim3(128), smem, s, m, stage_bytes, end[0], end[1]));
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

template <int TY, bool GLU, int R, int J, int KS>
static int launch_rows(const GemvArgs& a, int max_blocks, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemv_rows_kernel<TY, GLU, R, J, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr = true;
    }
    const int stage = R * max_blocks * rows_block_bytes(TY), stage_bytes = (stage + 127) & ~127;
    const size_t smem = (size_t)stage_bytes * ROWS_D * 4;
    const int n_groups = (a.n_out + (GLU ? R / 2 : R) - 1) / (GLU ? R / 2 : R);
    const int fit = (int)((226 * 1024) / (smem + 1024)), most = 148 * (fit < 1 ? 1 : fit > ROWS_PER_SM ? ROWS_PER_SM : fit);
    // fewer groups than warps: every SM takes its share all the same, a warp without a group ends at once
    const int need = KS == 1 ? (n_groups + 3) / 4 : n_groups, ctas = need < (KS == 1 ? 148 : most) ? need : most;
    TSB_CHECK_CUDA(tsb_launch(gemv_rows_kernel<TY, GLU, R, J, KS>, dim3(ctas), dim3(128), smem, s, a, stage_bytes, n_groups));
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

// Four rows to a warp where that leaves every warp a group of some length (and a lane's activations, 16 registers a unit, stay at six units), two otherwise:
// 2 x 9728 x 2560 6.8 us with four rows and 7.4 with two, 32768 x 2560 of Q6_K 13.4 and 14.2; 6144 x 2560 4.2 and 3.6, 2560 x 9728 5.5 and 4.7 (Q6_K
// 7.5 and 6.3).  Not where a second round of groups would have less than a fifth of the warps at work: behind a norm, us of four rows; two, 8192 x 2048 6.3; 5.5
// (Q6_K 7.8; 6.8, Q8_0 7.3; 6.2), 8448 x 3072 8.2; 6.5 (10.1; 8.2, 7.6; 7.4).  Rows longer than 6144 values are split over the CTA.
template <int TY, bool GLU>
static int launch_rows_any(const GemvArgs& a, cudaStream_t s) {
    const int nb = a.w.K >> 8;
#define TSB_ROWS(RV, JV, KSV) return launch_rows<TY, GLU, RV, JV, KSV>(a, mb, s)
    if (nb <= 24) {
        const int mb = nb;
        const int quads = (a.w.N + 3) / 4, warps = 148 * ROWS_PER_SM * 4;
        if (nb > 4 && nb <= 12 && quads >= warps && 5 * (quads - warps) > warps) {
            switch ((mb + 1) / 2) {
            case 3: TSB_ROWS(4, 3, 1);
            case 4: TSB_ROWS(4, 4, 1);
            case 5: TSB_ROWS(4, 5, 1);
            default: TSB_ROWS(4, 6, 1);
            }
        }
        switch ((mb + 3) / 4) {
        case 1: TSB_ROWS(2, 1, 1);
        case 2: TSB_ROWS(2, 2, 1);
        case 3: TSB_ROWS(2, 3, 1);
        case 4: TSB_ROWS(2, 4, 1);
        case 5: TSB_ROWS(2, 5, 1);
        default: TSB_ROWS(2, 6, 1);
        }
    }
    int mb = 0;
    for (int w = 0; w < 4; ++w) mb = max(mb, rows_slice<TY, 4>(nb, w + 1) - rows_slice<TY, 4>(nb, w));
    switch ((mb + 3) / 4) {                                              // slices of 7 to 16 blocks, of Q8_0 to 24
    case 2: TSB_ROWS(2, 2, 4);
    case 3: TSB_ROWS(2, 3, 4);
    case 4: TSB_ROWS(2, 4, 4);
    default: break;
    }
    if constexpr (TY == ROWS_Q8) {
        if ((mb + 3) / 4 == 5) TSB_ROWS(2, 5, 4);
        TSB_ROWS(2, 6, 4);
    }
    return TSB_ERR_UNSUPPORTED;
#undef TSB_ROWS
}

template <int M, bool GLU, bool Q5, int D>
static int launch_stream(const GemvArgs& a, int ppw, int ctas, size_t smem, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        TSB_CHECK_CUDA(cudaFuncSetAttribute(gemv_stream_kernel<M, GLU, Q5, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        attr = true;
    }
    TSB_CHECK_CUDA(tsb_launch(gemv_stream_kernel<M, GLU, Q5, D>, dim3(ctas), dim3(128), smem, s, a, ppw));
    TSB_CHECK_LAUNCH();
    return TSB_OK;
}

template <bool GLU, bool Q5, int D>
static int launch_stream_m(const GemvArgs& a, int ppw, int ctas, size_t smem, cudaStream_t s) {
    if (a.M <= 1) return launch_stream<1, GLU, Q5, D>(a, ppw, ctas, smem, s);
    if (a.M <= 2) return launch_stream<2, GLU, Q5, D>(a, ppw, ctas, smem, s);
    return launch_stream<4, GLU, Q5, D>(a, ppw, ctas, smem, s);
}

// Whether the row pipeline takes this GEMV (called by tsb_gemv_push before the plain launch): the single-token forms above.  The generic form
// (M <= 4, Q5_K, any row length) measured slower than the plain kernel inside the decode step and is kept behind TSB_GEMV_STREAM=2.
// TSB_GEMV_STREAM=0 turns the pipeline off altogether.
static int stream_mode() {
    static const int mode = []() { const char* e = getenv("TSB_GEMV_STREAM"); return e ? atoi(e) : 1; }();
    return mode;
}

// Whether a second round of groups would have less than a fifth of the warps at work, rows of up to 4096 values: such a matrix is twice the time of a group with
// most of the chip idle, and the row-per-warp kernel is the faster one for Q6_K and Q8_0.  Measured behind a norm, us of both (this pipeline; a row per
// warp): Q8_0 4096 x 4096 7.3; 6.5, gated 4096 x 1024 4.3; 3.7, gated 4096 x 2048 5.3; 4.3, Q6_K 4096 x 4096 7.8; 7.1; a second round that
// is half full Q8_0 5120 x 1024 4.3; 5.0, 5376 x 4096 pays.  (Q4_K 4096 x 4096 6.3; 6.4.)
static bool rows_second_round_idle(const GemvArgs& a, bool glu, int block_bytes) {
    const int nb = a.w.K >> 8, rows = 2;                                 // (four rows: launch_rows_any takes two in that case)
    if (nb > 16) return false;
    const size_t smem = (size_t)((rows * nb * block_bytes + 127) & ~127) * ROWS_D * 4;
    const int fit = (int)((226 * 1024) / (smem + 1024)), warps = 148 * 4 * (fit < 1 ? 1 : fit > ROWS_PER_SM ? ROWS_PER_SM : fit);
    const int per = glu ? rows / 2 : rows, groups = (a.n_out + per - 1) / per;
    return groups > warps && 5 * (groups - warps) <= warps;
}

static bool q6k_ok(const GemvArgs& a, bool glu) {
    const int nb = a.w.K >> 8;
    return a.w.type == TSB_Q6_K && !glu && a.M == 1 && nb >= 2 && nb % 2 == 0 && nb <= 64 && a.w.N >= 64 &&
           !rows_second_round_idle(a, glu, rows_block_bytes(ROWS_Q6));
}

static bool q8_ok(const GemvArgs& a, bool glu) {
    return a.w.type == TSB_Q8_0 && a.M == 1 && a.w.K % 256 == 0 && a.w.K <= 96 * 256 && a.w.N >= 64 &&
           ((reinterpret_cast<uintptr_t>(a.w.p0) | reinterpret_cast<uintptr_t>(a.w.p1)) & 15) == 0 && !rows_second_round_idle(a, glu, rows_block_bytes(ROWS_Q8));
}

static bool fast_ok(const GemvArgs& a) {
    const int nb = a.w.K >> 8;
    return a.w.type == TSB_Q4_K && a.M == 1 && nb >= 1 && nb * 8 <= 512 && a.w.N >= 64;
}

// One token, every matrix of the two types with rows of at most 24 blocks
bool tsb_gemv_rows_multi_eligible(const GemvMultiArgs& m) {
    const int nb = m.w[0].K >> 8;
    bool ok = stream_mode() != 0 && m.M == 1 && nb >= 1 && nb <= 24 && m.n_total >= 64;
    for (int i = 0; i < m.n_w; ++i) ok = ok && m.w[i].N > 0 && (m.w[i].type == TSB_Q4_K || (m.w[i].type == TSB_Q6_K && nb % 2 == 0));
    return ok;
}

int tsb_gemv_rows_multi_launch(const GemvMultiArgs& m, cudaStream_t s) {
    switch (((m.w[0].K >> 8) + 3) / 4) {
    case 1: return launch_rows_multi<1>(m, s);
    case 2: return launch_rows_multi<2>(m, s);
    case 3: return launch_rows_multi<3>(m, s);
    case 4: return launch_rows_multi<4>(m, s);
    case 5: return launch_rows_multi<5>(m, s);
    default: return launch_rows_multi<6>(m, s);
    }
}

bool tsb_gemv_stream_eligible(const GemvArgs& a) {
    const int mode = stream_mode();
    if (!mode || a.ids || a.M > 4 || a.M < 1) return false;
    const bool glu = a.act >= ACT_SWIGLU && a.act <= ACT_SWIGLU_OAI;
    if ((fast_ok(a) || q8_ok(a, glu)) && !(glu && a.push)) return true;
    if (q6k_ok(a, glu)) return true;
    if (a.push || mode < 2 || (a.w.type != TSB_Q4_K && a.w.type != TSB_Q5_K)) return false;
    const size_t rowbytes = (size_t)(a.w.K >> 8) * (a.w.type == TSB_Q5_K ? 176 : 144);
    return rowbytes * 4 * 4 <= 200 * 1024 && a.w.N >= 64;           // four warps x four buffers must fit
}

int tsb_gemv_stream_launch(const GemvArgs& a, bool glu, cudaStream_t s) {
    if (fast_ok(a)) return glu ? launch_rows_any<ROWS_Q4, true>(a, s) : launch_rows_any<ROWS_Q4, false>(a, s);
    if (q8_ok(a, glu)) return glu ? launch_rows_any<ROWS_Q8, true>(a, s) : launch_rows_any<ROWS_Q8, false>(a, s);
    if (q6k_ok(a, glu)) return launch_rows_any<ROWS_Q6, false>(a, s);
    const bool q5 = a.w.type == TSB_Q5_K;
    const size_t rowbytes = (size_t)(a.w.K >> 8) * (q5 ? 176 : 144);
    const size_t smem = rowbytes * 4 * 4;
    int per_sm = (int)((220 * 1024) / (smem + 1024));
    per_sm = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
    const int n_pairs = glu ? a.n_out : (a.w.N + 1) / 2;
    const int warps = 148 * per_sm * 4;
    const int ppw = (n_pairs + warps - 1) / warps;
    const int ctas = (n_pairs + 4 * ppw - 1) / (4 * ppw);
    if (glu) return q5 ? launch_stream_m<true, true, 4>(a, ppw, ctas, smem, s) : launch_stream_m<true, false, 4>(a, ppw, ctas, smem, s);
    return q5 ? launch_stream_m<false, true, 4>(a, ppw, ctas, smem, s) : launch_stream_m<false, false, 4>(a, ppw, ctas, smem, s);
}
