// Projections of small token batches (verification batches, short prompts), Q4_K and Q6_K weights, with mma.sync int8.
//
// The arithmetic is that of the decode kernels: exact integer sub-block dots, each scaled by the weights' scale and the
// activation group's, summed in fp32.  A sub-block of 32 (Q4_K) or 16 (Q6_K) weights is one MMA: 16 tokens (A: the int8
// activations) x 8 weight rows (B: the 4- or 6-bit values as they are).  Its accumulator starts at 1.5 * 2^23, so that its
// bits are that float plus the dot, and costs six packed operations for its 128 sums.  tcgen05 needs the weights' scales
// inside its f16 operand (tfr_gemm_tc.cuh): unpacking to it and a pipeline of barriers cost the same whatever the batch (2 900
// warp instructions per 96 rows x 64 weights x up to 128 tokens; here 860 for 16 tokens, 2 600 for 80), and there is no barrier
// here between a CTA's first weight and its last.
//
// A block's sums are joined to the row's once per block.  Relative error against float64, Gaussian values: Q4_K 1.9-2.2e-7
// for 512 to 27 648 inputs, Q6_K 0.8-1.15e-7 (dp4a 1.8-1.95e-7 and 0.7-1.0e-7); with one chain over a row's sub-blocks and
// terms cut off instead of rounded it was 3.3-4.5e-7 and 0.8-1.3e-7.
//
//   What bounds it: the chains of shared-memory read, MMA and sums, 80 cycles of a scheduler per MMA with five token tiles (11 008
//   gate and up rows of 2 048, a launch by itself: 20 us for 16 tokens, 31 for 48, 62 for 80; the tensor pipe is 10 to 16 %
//   busy, the schedulers issue in 34 to 36 % of the cycles).
#pragma once
#include "tfr_gemm_tc.cuh"

namespace tfr {

// ------------------------------------------------------------------ activations

// Image in global memory, in the order the MMAs' fragments are read: [token / 16][block of 256][7 KB]:
//   Q4_K   8 x 512 B    int8 A fragments of a sub-block (m16n8k32; lane's k: bytes 8 tq .. 8 tq + 7 of the 32)
//          8 x 128 B    d8 twice, of token g and of token g + 8 (g = lane / 4)
//          2 x 512 B    d8 * (sum of the group) as A fragments of m16n8k8, high and low tf32 term (split_tf32)
//   Q6_K  16 x 256 B    int8 A fragments of 16 values (m16n8k16)
//          8 x 128 B    d8 as above
//         16 x 128 B    start of the accumulators, twice for token g, twice for g + 8: 1.5 * 2^23 - 32 * (sum of the 16)
constexpr int MMA_BLOCK_BYTES = 7168, MMA_MAX_TILES = 5, MMA_MAX_TOKENS = 16 * MMA_MAX_TILES;
inline size_t mma_image_bytes(int K) { return (size_t)(2 * MMA_MAX_TILES) * (K / 256) * MMA_BLOCK_BYTES; }  // launches may round the tiles up

struct PrepMmaArgs {
    const float* x;      // [M][ldx]
    int ldx, K, M;
    const float* normw;  // RMSNorm weight or nullptr
    float eps;
    unsigned char* image;
    float* xn;           // optional [M][K]: the normalised vector (fp32-route rows read it)
    int q6;
};
constexpr int MMA_PREP_THREADS = 512;
constexpr int MMA_MAGIC = 0x4B400000;  // bits of 1.5 * 2^23

// One CTA per token, padding included (zeros): RMSNorm in the reference's reduction order, Q8 as in act_quantize4 with
// eight values per thread.
__global__ void __launch_bounds__(MMA_PREP_THREADS) k_prep_mma(PrepMmaArgs a) {
    extern __shared__ __align__(128) unsigned char mmap_smem[];
    float* xs = reinterpret_cast<float*>(mmap_smem);
    float* red = xs + xs_floats(a.K);
    const int m = blockIdx.x, tid = threadIdx.x, K = a.K, n8 = K >> 3;
    const bool live = m < a.M;
    griddep_wait();
    griddep_launch_dependents();
    const float* x = a.x + (size_t)(live ? m : 0) * a.ldx;
    float scale = 1.f;
    if (a.normw) {
        for (int i4 = tid; i4 < (K >> 2); i4 += MMA_PREP_THREADS)
            *reinterpret_cast<float4*>(xs + xs_idx(4 * i4)) = reinterpret_cast<const float4*>(x)[i4];
        __syncthreads();
        scale = rms_scale_staged(xs, K, a.eps, red);
    }
    unsigned char* tile = a.image + (size_t)(m >> 4) * (K >> 8) * MMA_BLOCK_BYTES;
    const int g = m & 7, up = (m >> 3) & 1;  // token g or g + 8 of its tile
    for (int i0 = 0; i0 < n8; i0 += MMA_PREP_THREADS) {
        const int i = i0 + tid;  // values 8 i .. 8 i + 7; four lanes share a 32-value group
        const bool on = i < n8;
        float v[8];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
            if (on && live) {
                u = a.normw ? *reinterpret_cast<const float4*>(xs + xs_idx(8 * i + 4 * h)) : reinterpret_cast<const float4*>(x)[2 * i + h];
                if (a.normw) {
                    const float4 w = reinterpret_cast<const float4*>(a.normw)[2 * i + h];
                    u.x = u.x * scale * w.x, u.y = u.y * scale * w.y, u.z = u.z * scale * w.z, u.w = u.w * scale * w.w;
                    if (a.xn) reinterpret_cast<float4*>(a.xn + (size_t)m * K)[2 * i + h] = u;
                }
            }
            v[4 * h] = u.x, v[4 * h + 1] = u.y, v[4 * h + 2] = u.z, v[4 * h + 3] = u.w;
        }
        float top = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) top = fmaxf(top, fabsf(v[k]));
        top = fmaxf(top, __shfl_xor_sync(TFR_FULL_MASK, top, 1));
        top = fmaxf(top, __shfl_xor_sync(TFR_FULL_MASK, top, 2));
        const float d = top * (1.0f / 127.0f);
        unsigned w[2] = {0u, 0u};
        int sum = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int q = top != 0.f ? (int)(signed char)__float2int_rn(v[k] / d) : 0;
            sum += q;
            w[k >> 2] |= (unsigned)(q & 0xff) << (8 * (k & 3));
        }
        const int s16 = sum + __shfl_xor_sync(TFR_FULL_MASK, sum, 1);
        const int s32 = s16 + __shfl_xor_sync(TFR_FULL_MASK, s16, 2);
        if (!on) continue;  // whole groups: n8 is a multiple of 32
        unsigned char* blk = tile + (size_t)(i >> 5) * MMA_BLOCK_BYTES;
        const int s = (i >> 2) & 7, tq = i & 3;
        if (a.q6) {
            const int c = (i >> 1) & 15;
            unsigned char* p = blk + c * 256 + (g * 4 + 2 * (i & 1)) * 8 + up * 4;
            *reinterpret_cast<unsigned*>(p) = w[0];
            *reinterpret_cast<unsigned*>(p + 8) = w[1];
            if ((i & 1) == 0) *reinterpret_cast<int2*>(blk + 5120 + c * 128 + g * 16 + up * 8) = make_int2(MMA_MAGIC - 32 * s16, MMA_MAGIC - 32 * s16);
        } else {
            unsigned char* p = blk + s * 512 + (g * 4 + tq) * 16 + up * 4;
            *reinterpret_cast<unsigned*>(p) = w[0];
            *reinterpret_cast<unsigned*>(p + 8) = w[1];
            if (tq == 0) {
                float* q = reinterpret_cast<float*>(blk + 5120 + (g * 4 + (s & 3)) * 16 + (s >> 2) * 8 + up * 4);
                split_tf32(d * (float)s32, q[0], q[128]);
            }
        }
        if (tq == 0) *reinterpret_cast<float2*>(blk + 4096 + s * 128 + g * 16 + up * 8) = make_float2(d, d);
    }
}

// ------------------------------------------------------------------ MMAs

// D = A B + C; C in registers of its own, so that a constant start is not copied in front of every MMA.
__device__ __forceinline__ int4 mma_u8_k32(const int4& a, unsigned b0, unsigned b1, const int4& c) {
    int4 d;
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d.x), "=r"(d.y), "=r"(d.z), "=r"(d.w)
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w));
    return d;
}
__device__ __forceinline__ int4 mma_u8_k16(const int2& a, unsigned b, const int4& c) {
    int4 d;
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
        : "=r"(d.x), "=r"(d.y), "=r"(d.z), "=r"(d.w)
        : "r"(a.x), "r"(a.y), "r"(b), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w));
    return d;
}
__device__ __forceinline__ float4 mma_tf32_k8(const float4& a, float b0, float b1, const float4& c) {
    float4 d;
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
        : "r"(__float_as_uint(a.x)), "r"(__float_as_uint(a.y)), "r"(__float_as_uint(a.z)), "r"(__float_as_uint(a.w)), "r"(__float_as_uint(b0)),
          "r"(__float_as_uint(b1)), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
    return d;
}
// Byte i of w as a float, exactly: the byte under the exponent that makes it 2^23 + byte.
__device__ __forceinline__ float mma_byte(unsigned w, int i) { return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440 + i)); }

// ------------------------------------------------------------------ the kernel

// CTA = a share of the weight rows, 16 (two MMA widths; ZIP: 8 gate and the same 8 up rows) at a time, x all tokens x a part
// of the k range whose activations fit shared memory.  Sixteen warps: `wpn` of them split the blocks of one 16-row strip,
// 16 / wpn strips side by side; a warp's words of its next block travel, from L2 where the CTA's first warps have sent for
// them, while it computes this one.  Per round of strips the warps' sums meet in shared memory (with the k range cut, those
// of the cluster's CTAs through distributed shared memory) and the threads share out the epilogue.
constexpr int MMA_THREADS = 512, MMA_WARPS = MMA_THREADS / 32;
constexpr size_t MMA_SMEM_MAX = 220 * 1024;

struct MmaArgs {
    const unsigned char* image;
    int M;
    Mat A1, A2;        // ZIP: the pair; otherwise A2 (optional) follows A1
    int strips1;       // 16-row strips of A1
    Share sh;          // strips over grid.x
    int id1, id2, zip, wpn, side;
    ChunkEpi epi;
    TokenState* st;
};

// The words of a block of weight row g = lane / 4 that this lane (tq = lane % 4) multiplies, and the row's scales.
struct MmaQ4 {
    uint2 w[4];
    int4 hdr;
    __device__ __forceinline__ void load(const Mat& m, int row, int b, int tq) {
        const int f = (int)mat_flat(m.nb, min(row, m.N - 1), b);
        const uint8_t* p = m.data + (size_t)(f >> 5) * Q4_TILE_BYTES + (f & 31) * 16;
        hdr = ldg_stream(p);
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = __ldg(reinterpret_cast<const uint2*>(p + (1 + 2 * j + (tq >> 1)) * 512 + (tq & 1) * 8));
    }
};
struct MmaQ6 {
    unsigned ql[2][2][2], qh[2][2];  // [half n][j & 1][is]; [n][is]
    int4 sc;
    float d;
    __device__ __forceinline__ void load(const Mat& m, int row, int b, int tq) {
        const int f = (int)mat_flat(m.nb, min(row, m.N - 1), b);
        const uint8_t* t = m.data + (size_t)(f >> 5) * Q6_TILE_BYTES;
        const uint8_t* p = t + (f & 31) * 16;
        sc = ldg_stream(p + 12 * 512);
        d = f16_to_f32(__ldg(reinterpret_cast<const unsigned short*>(t + Q6_PIECES * 512 + (f & 31) * 2)));
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int is = 0; is < 2; is++) {
                qh[n][is] = __ldg(reinterpret_cast<const unsigned*>(p + (8 + 2 * n + is) * 512 + tq * 4));
#pragma unroll
                for (int j = 0; j < 2; j++) ql[n][j][is] = __ldg(reinterpret_cast<const unsigned*>(p + (4 * n + 2 * j + is) * 512 + tq * 4));
            }
    }
};

template <class RAW, int MT>
__global__ void __launch_bounds__(MMA_THREADS, 1) k_gemm_mma(const MmaArgs a) {
    constexpr bool Q4 = sizeof(RAW) == sizeof(MmaQ4);
    constexpr bool AHEAD = MT <= 2;  // registers for the next block's words; more tokens hide the trip behind the other warps' work
    constexpr int SLOT = MT * 256 + 8;  // floats of a warp's sums, [token][16 rows], padded
    extern __shared__ __align__(128) unsigned char mma_smem[];
    __shared__ unsigned long long full;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
    const int S = gridDim.y, part = blockIdx.y, nb = a.A1.nb, b0 = nb * part / S, b1 = nb * (part + 1) / S, nbk = b1 - b0;
    const int m0 = blockIdx.z * MT * 16, M = min(MT * 16, a.M - m0);  // this CTA's tokens
    const int s0 = a.sh.begin(blockIdx.x), sn = a.sh.count(blockIdx.x), wpn = a.wpn, side = a.side;  // strips side by side
    unsigned char* acts = mma_smem;
    float* slots = reinterpret_cast<float*>(mma_smem + (size_t)MT * ((nb + S - 1) / S) * MMA_BLOCK_BYTES);  // the same place in a cluster's CTAs
    // strip s: its two matrices and first rows
    auto strip = [&](int s, Mat& ma, Mat& mb, int& r0, int& r1) {
        const bool second = !a.zip && s >= a.strips1;
        ma = second ? a.A2 : a.A1, mb = a.zip ? a.A2 : ma;
        r0 = a.zip ? 8 * s : 16 * (second ? s - a.strips1 : s), r1 = a.zip ? r0 : r0 + 8;
    };
    const int my = warp / wpn, kp = warp - my * wpn, c0 = b0 + nbk * kp / wpn, c1 = b0 + nbk * (kp + 1) / wpn;  // this warp's strip of a round, its blocks
    // The strips of a round on their way into L2, a round ahead of their use (more would push one another out again).
    auto ahead = [&](int round) {
        const int s = round * side + my;
        if (kp != 0 || lane >= 4 || s >= sn || my >= side) return;
        Mat ma, mb;
        int r0, r1;
        strip(s0 + s, ma, mb, r0, r1);
        const Mat& m = (lane & 2) ? mb : ma;
        const int row = ((lane & 2) ? r1 : r0) + ROW_GROUP * (lane & 1);
        if (row >= m.N) return;
        constexpr size_t TB = Q4 ? Q4_TILE_BYTES : Q6_TILE_BYTES;
        const size_t f = mat_flat(nb, row, 0), t0 = (f + ROW_GROUP * b0) >> 5, t1 = (f + ROW_GROUP * b1 + 31) >> 5;
        bulk_prefetch_l2(m.data + t0 * TB, (unsigned)((t1 - t0) * TB));
    };
    ahead(0);  // weights do not depend on earlier kernels
    if (tid == 0) {
        mbar_init(&full, 1);
        mbar_fence_init();
    }
    RAW raw[2];
    auto fetch = [&](int round, int b) {
        const int s = round * side + my;
        if (s >= sn || b >= c1 || my >= side) return;
        Mat ma, mb;
        int r0, r1;
        strip(s0 + s, ma, mb, r0, r1);
        raw[0].load(ma, r0 + g, b, tq);
        raw[1].load(mb, r1 + g, b, tq);
    };
    if (AHEAD) fetch(0, c0);
    __syncthreads();
    griddep_wait();
    griddep_launch_dependents();
    if (tid == 0) {
        mbar_expect_tx(&full, MT * nbk * MMA_BLOCK_BYTES);
        for (int t = 0; t < MT; t++)
            bulk_load(acts + (size_t)t * nbk * MMA_BLOCK_BYTES, a.image + ((size_t)(blockIdx.z * MT + t) * nb + b0) * MMA_BLOCK_BYTES, nbk * MMA_BLOCK_BYTES, &full);
    }
    const bool landed = __all_sync(TFR_FULL_MASK, mbar_wait(&full, 0));
    if (!landed && a.st) a.st->err = 2;
    const int rounds = (sn + side - 1) / side;
    for (int round = 0; round < rounds; round++) {
        const bool on = my < side && round * side + my < sn;
        ahead(round + 1);
        float2 acc[2][MT][2];  // [8 rows][token tile][token g, g + 8]: rows 2 tq, 2 tq + 1
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int t = 0; t < MT; t++) acc[n][t][0] = acc[n][t][1] = make_float2(0.f, 0.f);
        if (on && landed)
            for (int b = c0; b < c1; b++) {
                if (!AHEAD) fetch(round, b);
                const RAW cur[2] = {raw[0], raw[1]};
                if (AHEAD) {
                    if (b + 1 < c1) fetch(round, b + 1);
                    else fetch(round + 1, c0);
                }
                const unsigned char* blk = acts + (size_t)(b - b0) * MMA_BLOCK_BYTES;
                float2 sum[2][MT][2];  // of this block, without d: a chain over all sub-blocks of a row would round four times as coarsely
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int t = 0; t < MT; t++) sum[n][t][0] = sum[n][t][1] = make_float2(0.f, 0.f);
                // one sub-block of every token tile: B fragments and scales in, sums out; scale * dot is exact (below 2^24)
                auto step = [&](int t, int n, const int4& c, const float4& dd, const float2& sc) {
                    const float2 magic = make_float2(-12582912.f, -12582912.f), one = make_float2(1.f, 1.f);
                    const float2 f0 = fma_f32x2(make_float2(__int_as_float(c.x), __int_as_float(c.y)), one, magic);
                    const float2 f1 = fma_f32x2(make_float2(__int_as_float(c.z), __int_as_float(c.w)), one, magic);
                    sum[n][t][0] = fma_f32x2(mul_f32x2(f0, sc), make_float2(dd.x, dd.y), sum[n][t][0]);
                    sum[n][t][1] = fma_f32x2(mul_f32x2(f1, sc), make_float2(dd.z, dd.w), sum[n][t][1]);
                };
                auto join = [&](const float2 (&d)[2]) {
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int t = 0; t < MT; t++)
#pragma unroll
                            for (int i = 0; i < 2; i++) acc[n][t][i] = fma_f32x2(d[n], sum[n][t][i], acc[n][t][i]);
                };
                const int ra = 8 * tq, rb = ra + 4;  // lanes that hold rows 2 tq, 2 tq + 1
                if constexpr (Q4) {
                    float2 d[2], dm[2];
                    unsigned sa[2][2], sb[2][2];  // [8 rows][scales 0-3, 4-7] of the two rows
                    float bm[2][2];               // mins t and t + 4 of row g
#pragma unroll
                    for (int n = 0; n < 2; n++) {
                        const unsigned h0 = (unsigned)cur[n].hdr.x, h1 = (unsigned)cur[n].hdr.y, h2 = (unsigned)cur[n].hdr.z, h3 = (unsigned)cur[n].hdr.w;
                        const unsigned lo = h1 & 0x3f3f3f3fu, hi = (h3 & 0x0f0f0f0fu) | (((h1 >> 6) & 0x03030303u) << 4);
                        const unsigned mlo = h2 & 0x3f3f3f3fu, mhi = ((h3 >> 4) & 0x0f0f0f0fu) | (((h2 >> 6) & 0x03030303u) << 4);
                        bm[n][0] = (float)((mlo >> (8 * tq)) & 0xff), bm[n][1] = (float)((mhi >> (8 * tq)) & 0xff);
                        const unsigned da = __shfl_sync(TFR_FULL_MASK, h0, ra), db = __shfl_sync(TFR_FULL_MASK, h0, rb);
                        sa[n][0] = __shfl_sync(TFR_FULL_MASK, lo, ra), sb[n][0] = __shfl_sync(TFR_FULL_MASK, lo, rb);
                        sa[n][1] = __shfl_sync(TFR_FULL_MASK, hi, ra), sb[n][1] = __shfl_sync(TFR_FULL_MASK, hi, rb);
                        const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&da)), fb = __half22float2(*reinterpret_cast<const __half2*>(&db));
                        d[n] = make_float2(fa.x, fb.x), dm[n] = make_float2(-fa.y, -fb.y);
                    }
#pragma unroll
                    for (int s = 0; s < 8; s++) {
                        unsigned w0[2], w1[2];
                        float2 sc[2];
#pragma unroll
                        for (int n = 0; n < 2; n++) {
                            // high nibbles are multiplied as (nibble << 4): the exact factor leaves through the scale
                            const unsigned mask = (s & 1) ? 0xf0f0f0f0u : 0x0f0f0f0fu;
                            w0[n] = cur[n].w[s >> 1].x & mask, w1[n] = cur[n].w[s >> 1].y & mask;
                            const float k = (s & 1) ? 0.0625f : 1.f;
                            sc[n] = make_float2(k * (mma_byte(sa[n][s >> 2], s & 3) - 8388608.f), k * (mma_byte(sb[n][s >> 2], s & 3) - 8388608.f));
                        }
#pragma unroll
                        for (int t = 0; t < MT; t++) {
                            const unsigned char* p = blk + (size_t)t * nbk * MMA_BLOCK_BYTES;
                            const int4 A = *reinterpret_cast<const int4*>(p + s * 512 + lane * 16);
                            const float4 dd = *reinterpret_cast<const float4*>(p + 4096 + s * 128 + g * 16);
#pragma unroll
                            for (int n = 0; n < 2; n++) {
                                step(t, n, mma_u8_k32(A, w0[n], w1[n], make_int4(MMA_MAGIC, MMA_MAGIC, MMA_MAGIC, MMA_MAGIC)), dd, sc[n]);
                            }
                        }
                    }
                    // dmin * (mins x group sums): two tf32 terms of the sums, the mins are small integers.  The terms' sums stay
                    // apart, because the tensor core would truncate where they meet.
#pragma unroll
                    for (int t = 0; t < MT; t++) {
                        const unsigned char* p = blk + (size_t)t * nbk * MMA_BLOCK_BYTES + 5120 + lane * 16;
                        const float4 hi = *reinterpret_cast<const float4*>(p), lo = *reinterpret_cast<const float4*>(p + 512);
#pragma unroll
                        for (int n = 0; n < 2; n++) {
                            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), cl = mma_tf32_k8(lo, bm[n][0], bm[n][1], zero), ch = mma_tf32_k8(hi, bm[n][0], bm[n][1], zero);
                            acc[n][t][0] = fma_f32x2(dm[n], make_float2(ch.x, ch.y), fma_f32x2(dm[n], make_float2(cl.x, cl.y), acc[n][t][0]));
                            acc[n][t][1] = fma_f32x2(dm[n], make_float2(ch.z, ch.w), fma_f32x2(dm[n], make_float2(cl.z, cl.w), acc[n][t][1]));
                        }
                    }
                    join(d);
                } else {
                    float2 d[2];
                    unsigned sa[2][4], sb[2][4];  // scales + 128 of the two rows
#pragma unroll
                    for (int n = 0; n < 2; n++) {
                        d[n] = make_float2(__shfl_sync(TFR_FULL_MASK, cur[n].d, ra), __shfl_sync(TFR_FULL_MASK, cur[n].d, rb));
                        const unsigned sw[4] = {(unsigned)cur[n].sc.x, (unsigned)cur[n].sc.y, (unsigned)cur[n].sc.z, (unsigned)cur[n].sc.w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            sa[n][i] = __shfl_sync(TFR_FULL_MASK, sw[i] ^ 0x80808080u, ra);
                            sb[n][i] = __shfl_sync(TFR_FULL_MASK, sw[i] ^ 0x80808080u, rb);
                        }
                    }
#pragma unroll
                    for (int c16 = 0; c16 < 16; c16++) {
                        // group c = 8 h + 2 j + is (kernels/gemv.cu:302-337, as in block_dot)
                        const int h = c16 >> 3, j = (c16 >> 1) & 3, is = c16 & 1;
                        unsigned w[2];
                        float2 sc[2];
#pragma unroll
                        for (int n = 0; n < 2; n++) {
                            w[n] = ((cur[n].ql[h][j & 1][is] >> (4 * (j >> 1))) & 0x0f0f0f0fu) | (((cur[n].qh[h][is] >> (2 * j)) & 0x03030303u) << 4);
                            sc[n] = make_float2(mma_byte(sa[n][c16 >> 2], c16 & 3) - 8388736.f, mma_byte(sb[n][c16 >> 2], c16 & 3) - 8388736.f);
                        }
#pragma unroll
                        for (int t = 0; t < MT; t++) {
                            const unsigned char* p = blk + (size_t)t * nbk * MMA_BLOCK_BYTES;
                            const int2 A = *reinterpret_cast<const int2*>(p + c16 * 256 + lane * 8);
                            const float4 dd = *reinterpret_cast<const float4*>(p + 4096 + (c16 >> 1) * 128 + g * 16);
                            const int4 start = *reinterpret_cast<const int4*>(p + 5120 + c16 * 128 + g * 16);
#pragma unroll
                            for (int n = 0; n < 2; n++) {
                                step(t, n, mma_u8_k16(A, w[n], start), dd, sc[n]);
                            }
                        }
                    }
                    join(d);
                }
            }
        float* slot = slots + warp * SLOT;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int t = 0; t < MT; t++) {
                *reinterpret_cast<float2*>(slot + (t * 16 + g) * 16 + n * 8 + 2 * tq) = acc[n][t][0];
                *reinterpret_cast<float2*>(slot + (t * 16 + g + 8) * 16 + n * 8 + 2 * tq) = acc[n][t][1];
            }
        __syncthreads();
        // eight items (pairs of adjacent rows; ZIP: a gate and its up row) per strip, all tokens
        const int strips = min(side, sn - round * side), items = strips * 8;
        auto pair_at = [&](const float* base, int i) {
            return a.zip ? make_float2(base[i], base[8 + i]) : *reinterpret_cast<const float2*>(base + 2 * i);
        };
        if (S > 1) {
            for (int i = tid; i < strips * MT * 256; i += MMA_THREADS) {
                const int s = i / (MT * 256), e = i - s * (MT * 256);
                float* p = slots + s * wpn * SLOT + e;
                float v = p[0];
                for (int k = 1; k < wpn; k++) v += p[k * SLOT];
                p[0] = v;
            }
            cluster_sync_all();
        }
        for (int i = tid + part * MMA_THREADS; i < items * M; i += MMA_THREADS * S) {
            const int m = i / items, it = i - m * items, s = it >> 3;
            const float* base = slots + s * wpn * SLOT + m * 16;
            float2 v = make_float2(0.f, 0.f);
            if (S > 1) {
                const unsigned at0 = smem_u32(base + (a.zip ? it & 7 : 2 * (it & 7))), second = a.zip ? 32 : 4;
                float x[8], y[8];
#pragma unroll
                for (int p = 0; p < 8; p++) {
                    x[p] = y[p] = 0.f;
                    if (p < S) {
                        unsigned remote;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at0), "r"(p));
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[p]) : "r"(remote) : "memory");
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(y[p]) : "r"(remote + second) : "memory");
                    }
                }
#pragma unroll
                for (int p = 0; p < 8; p++) v.x += x[p], v.y += y[p];
            } else {
                v = pair_at(base, it & 7);
                for (int k = 1; k < wpn; k++) {
                    const float2 u = pair_at(base + k * SLOT, it & 7);
                    v.x += u.x, v.y += u.y;
                }
            }
            const int st = s0 + round * side + s;
            const bool second = !a.zip && st >= a.strips1;
            const int row = (a.zip ? 8 * st + (it & 7) : 16 * (second ? st - a.strips1 : st) + 2 * (it & 7));
            if (row < (second ? a.A2.N : a.A1.N)) ChunkEpiTok{&a.epi, m0 + m}.apply((second ? a.id2 : a.id1) + (a.zip ? row : row >> 1), v.x, v.y);
        }
        if (S > 1) cluster_sync_all();
        else __syncthreads();  // the slots are free
    }
}

// k parts (a power of two), or 0 where no cut makes the activations fit
inline int mma_parts(int nb, int mt) {
    for (int s = 1; s <= 8 && s <= nb; s *= 2)
        if ((size_t)mt * ((nb + s - 1) / s) * MMA_BLOCK_BYTES + (size_t)MMA_WARPS * (mt * 256 + 8) * 4 <= MMA_SMEM_MAX) return s;
    return 0;
}
template <class RAW, int MT>
inline cudaError_t launch_mma(cudaStream_t stream, int sms, MmaArgs& a, int strips, int S) {
    const int nb = a.A1.nb, z = (a.M + 16 * MT - 1) / (16 * MT), ctas = std::max(1, std::min(strips, cluster_ctas(k_gemm_mma<RAW, MT>, MMA_THREADS, S, sms) / (S * z))), nbk = (nb + S - 1) / S;
    a.sh = make_share(strips, ctas);
    const int most = a.sh.quot + (a.sh.rem ? 1 : 0);
    // warps per strip: rounds x (blocks of a warp x what a block costs + what a round costs)
    double best = 1e30;
    for (int w = 1; w <= std::min(MMA_WARPS, nbk); w++) {
        const int fit = MMA_WARPS / w, rounds = (most + fit - 1) / fit, side = (most + rounds - 1) / rounds;
        const double t = rounds * (((nbk + w - 1) / w) * (0.5 + 0.5 * MT) + 1.5 + 0.1 * w + (S > 1 ? 1.5 : 0));
        if (t < best) best = t, a.wpn = w, a.side = side;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas, S, z);
    cfg.blockDim = dim3(MMA_THREADS);
    cfg.dynamicSmemBytes = (size_t)MT * nbk * MMA_BLOCK_BYTES + (size_t)MMA_WARPS * (MT * 256 + 8) * 4;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = S;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = S > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_gemm_mma<RAW, MT>, (const MmaArgs)a);
}
// Token tiles of a CTA: all of them where their activations fit, else as even shares as do.
inline int mma_tiles(int nb, int M) {
    const int tiles = (M + 15) / 16;
    for (int z = 1; z <= tiles; z++)
        if (mma_parts(nb, (tiles + z - 1) / z) > 0) return (tiles + z - 1) / z;
    return 0;
}

// out = epilogue(W x) for the M <= 96 tokens of an image; jb: the second matrix of a gate/up pair or one that follows.
inline cudaError_t launch_gemm_mma(cudaStream_t stream, int sms, const unsigned char* image, int M, const RowJob& ja, const RowJob& jb,
                                   const ChunkEpi& epi, TokenState* st) {
    MmaArgs a{};
    a.image = image, a.M = M, a.A1 = ja.m, a.A2 = jb.m, a.id1 = ja.id_base, a.id2 = jb.id_base;
    a.zip = epi.kind == CEPI_SILU, a.epi = epi, a.st = st;
    const int rows = a.zip ? 8 : 16, mt = mma_tiles(ja.m.nb, M), S = mt ? mma_parts(ja.m.nb, mt) : 0;
    a.strips1 = (ja.m.N + rows - 1) / rows;
    const int strips = a.strips1 + (!a.zip && jb.m.data ? (jb.m.N + rows - 1) / rows : 0);
    if (S == 0) return cudaErrorInvalidValue;
    const bool q4 = ja.m.type == TFR_Q4_K;
    switch (mt) {
        case 1: return q4 ? launch_mma<MmaQ4, 1>(stream, sms, a, strips, S) : launch_mma<MmaQ6, 1>(stream, sms, a, strips, S);
        case 2: return q4 ? launch_mma<MmaQ4, 2>(stream, sms, a, strips, S) : launch_mma<MmaQ6, 2>(stream, sms, a, strips, S);
        case 3: return q4 ? launch_mma<MmaQ4, 3>(stream, sms, a, strips, S) : cudaErrorInvalidValue;
        case 4: return q4 ? launch_mma<MmaQ4, 4>(stream, sms, a, strips, S) : cudaErrorInvalidValue;
        case 5: return q4 ? launch_mma<MmaQ4, 5>(stream, sms, a, strips, S) : cudaErrorInvalidValue;
    }
    return cudaErrorInvalidValue;
}

}  // namespace tfr
