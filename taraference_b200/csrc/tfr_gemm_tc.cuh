// Projections of token batches on the fifth-generation tensor cores (tcgen05), Q4_K and Q6_K weights.
//
// What has to be computed is the decode arithmetic (kernels/gemv.cu:71-130, 302-337): integer sub-block dots of the
// 4- or 6-bit weights with the int8 activations, scaled per sub-block by the weight's 6- or 8-bit scale and the
// activation group's fp32 scale, scaled per 256-weight block by the block's fp16 d, minus (Q4_K) dmin times the scaled
// group sums.  An integer MMA would have to leave its accumulator after every 32 (Q4_K) or 16 (Q6_K) weights to meet the
// activation's scale, and on the way meet the weight's.  Here the weights' scales travel inside the f16 operand instead:
//
//   weights   scale * quant   an integer.  Q4_K: at most 63 * 15, exact in f16.  Q6_K: at most 128 * 32, so an f16 term and
//                             a residual of at most one unit (a second operand tile);
//   tokens    q8              an integer.
//
// The accumulator (fp32, in TMEM) runs over one group of 32 weights.  All products and their sum are integers below 2^24
// (4 096 * 127 * 32), so the tensor core's truncating additions lose nothing: it holds the exact dot that dp4a computes, and
// meets the group's d8 and the block's d in fp32 multiply-adds in registers, round to nearest.  (With d8 inside the operand, as
// two f16 terms, an accumulator could run over 128 weights, but truncated: 5-10e-7 against float64 where this has 1.75-2.1e-7,
// and groups far smaller than their token's largest lost their low terms among the f16 subnormals.)
//
// The min term of Q4_K, sum over a block's groups of m * (d8 * sum q8), is a tf32 product of 8 terms: m is exact, the group sums
// are two rounded terms whose products stay in accumulators of their own.
//
//   What bounds it: the schedulers and the chain through the two accumulators, about 1 400 cycles a stage of 96 rows x 128 tokens x
//   64 weights (the schedulers issue in half of the cycles, the tensor pipe is 13 % busy on Q4_K, 28 % on Q6_K; with no work left
//   in any role the waits alone take 860).  Gate and up rows of 2 048 inputs, 2 048 tokens: 768 us; 11 008 inputs to 2 048 rows: 341.
//   Tried: pairs of CTAs on one tile of rows (cta_group::2; an arrival at the other CTA takes 1 000 cycles: 1 011 us where one CTA
//   took 814), eight draining warps with 48 columns each (865 to 920 where sixteen took 817).
#pragma once
#include "tfr_chunk.cuh"

namespace tfr {

// ------------------------------------------------------------------ operand image of the activations

// Both operands lie in shared memory as K-major rows of 128 bytes with the 128-byte swizzle: 16-byte chunk c of row r at
// r * 128 + ((c ^ (r & 7)) << 4), 8-row atoms of 1 KB.  The activations are written to global memory in exactly that
// image, so a stage of a CTA's token tile is one run of bytes and travels as one untiled bulk copy:
//   [stage of 64 values][token / 8][1 KB atom]       f16
//   [pair of blocks][token / 8][1 KB atom]           group sums of a block as tf32: 8 high terms, 8 low terms; the second block
//   [stage][token][its two groups]                   d8
constexpr int TC_STAGE_K = 64;
__host__ __device__ inline int tc_pad_tokens(int M) { return (M + 7) & ~7; }  // whole atoms
__host__ __device__ inline size_t tc_sums_at(int K, int Mp) { return (size_t)(K / TC_STAGE_K) * Mp * 128; }
__host__ __device__ inline size_t tc_d8_at(int K, int Mp) { return tc_sums_at(K, Mp) + (size_t)((K / 256 + 1) / 2) * Mp * 128; }
__host__ __device__ inline size_t tc_image_bytes(int K, int M) {
    const int Mp = tc_pad_tokens(M);
    return tc_d8_at(K, Mp) + (size_t)(K / TC_STAGE_K) * Mp * 8;
}
// x as two tf32 terms, each rounded to nearest: 2^-24 of x is lost.  (The tensor core cuts off what does not fit: a high term cut
// off instead of rounded leaves a low term of 13 bits, of which it would drop two, always towards zero.)
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
    unsigned h, l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
    hi = __uint_as_float(h);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(x - hi));
    lo = __uint_as_float(l);
}
__device__ __forceinline__ unsigned tc_swz(int row, int chunk) { return (unsigned)(row * 128 + ((chunk ^ (row & 7)) << 4)); }

struct PrepTcArgs {
    const float* x;      // [M][ldx]
    int ldx, K, M;
    const float* normw;  // RMSNorm weight or nullptr
    float eps;
    unsigned char* image;
    float* xn;           // optional [M][K]: the normalised vector (fp32-route rows read it)
};

constexpr int TC_PREP_THREADS = 512;
inline size_t tc_prep_smem(int K) { return (xs_floats(K) + 272) * sizeof(float); }

// One CTA per token (padding tokens included: they become zeros).  RMSNorm in the reference's reduction order
// (rms_scale_staged), the Q8 quantiser of act_quantize4 with eight values per thread.
__global__ void __launch_bounds__(TC_PREP_THREADS) k_prep_tc(PrepTcArgs a) {
    extern __shared__ __align__(128) unsigned char tcp_smem[];
    float* xs = reinterpret_cast<float*>(tcp_smem);
    float* red = xs + xs_floats(a.K);
    const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, K = a.K, n8 = K >> 3, Mp = gridDim.x;
    const bool live = m < a.M;
    const int row = m & 7;
    griddep_wait();
    griddep_launch_dependents();
    const float* x = a.x + (size_t)(live ? m : 0) * a.ldx;
    float scale = 1.f;
    if (a.normw) {
        for (int i4 = tid; i4 < (K >> 2); i4 += TC_PREP_THREADS)
            *reinterpret_cast<float4*>(xs + xs_idx(4 * i4)) = reinterpret_cast<const float4*>(x)[i4];
        __syncthreads();
        scale = rms_scale_staged(xs, K, a.eps, red);
    }
    unsigned char* tok = a.image + (size_t)(m >> 3) * 1024;
    unsigned char* d8 = a.image + tc_d8_at(K, Mp) + (size_t)m * 8;
    for (int i0 = 0; i0 < n8; i0 += TC_PREP_THREADS) {
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
        float g = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) g = fmaxf(g, fabsf(v[k]));
        g = fmaxf(g, __shfl_xor_sync(TFR_FULL_MASK, g, 1));
        g = fmaxf(g, __shfl_xor_sync(TFR_FULL_MASK, g, 2));
        const float d = g * (1.0f / 127.0f);
        int sum = 0;
        unsigned q[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            int q0 = 0, q1 = 0;
            if (g != 0.f) {
                q0 = (int)(signed char)__float2int_rn(v[2 * k] / d);
                q1 = (int)(signed char)__float2int_rn(v[2 * k + 1] / d);
            }
            sum += q0 + q1;
            q[k] = pack_f16x2(__int2half_rn(q0), __int2half_rn(q1));
        }
        sum += __shfl_xor_sync(TFR_FULL_MASK, sum, 1);
        sum += __shfl_xor_sync(TFR_FULL_MASK, sum, 2);
        if (!on) continue;  // whole groups: n8 is a multiple of 32
        *reinterpret_cast<uint4*>(tok + (size_t)(i >> 3) * Mp * 128 + tc_swz(row, i & 7)) = make_uint4(q[0], q[1], q[2], q[3]);
        if ((i & 3) == 0) {
            const int grp = i >> 2, b = grp >> 3;
            float hi, lo;
            split_tf32(d * (float)sum, hi, lo);
            unsigned char* p = tok + tc_sums_at(K, Mp) + (size_t)(b >> 1) * Mp * 128;
            const int chunk = 4 * (b & 1) + ((grp >> 2) & 1), at = (grp & 3) * 4;
            *reinterpret_cast<float*>(p + tc_swz(row, chunk) + at) = hi;
            *reinterpret_cast<float*>(p + tc_swz(row, chunk + 2) + at) = lo;
            *reinterpret_cast<float*>(d8 + (size_t)(grp >> 1) * Mp * 8 + (grp & 1) * 4) = d;
        }
    }
}

// ------------------------------------------------------------------ tcgen05 primitives

__device__ __forceinline__ void tc_alloc(unsigned* slot, unsigned cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tc_dealloc(unsigned addr, unsigned cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// One thread of a converged warp, always the same.
__device__ __forceinline__ bool tc_elect() {
    unsigned p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// Barriers by their shared-memory address.  Arrives when the MMAs issued so far are done:
__device__ __forceinline__ void tc_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_arrive(unsigned bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// Shared-memory descriptor of a K-major operand with the 128-byte swizzle: start address, (unused) leading offset, 1 KB
// between 8-row atoms, version 1, swizzle mode 2.
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr) {
    return (unsigned long long)((addr & 0x3ffffu) >> 4) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: fp32 accumulator, K-major operands of type `ty` (0: f16, 2: tf32), m x n.
__device__ __forceinline__ unsigned tc_idesc(unsigned ty, unsigned m, unsigned n) { return (1u << 4) | (ty << 7) | (ty << 10) | ((n >> 3) << 17) | ((m >> 4) << 24); }
template <bool TF32>
__device__ __forceinline__ void tc_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
#define TFR_TC_MMA(form)                                                                                                    \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma.cta_group::1." form " [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), \
                 "l"(b), "r"(idesc), "r"(accumulate)                                                                         \
                 : "memory")
    if (TF32) TFR_TC_MMA("kind::tf32");
    else TFR_TC_MMA("kind::f16");
#undef TFR_TC_MMA
}
// Columns addr .. addr + W - 1 of this warp's 32 lanes; the values are there after tc_ld_wait.
template <int W>
__device__ __forceinline__ void tc_ld(float* v, unsigned addr) {
    static_assert(W == 8 || W == 16, "");
    if constexpr (W == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                     : "r"(addr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
                       "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
                     : "r"(addr));
}
// 24 columns of this warp's 32 lanes.
__device__ __forceinline__ void tc_ld24(float* v, unsigned addr) {
    tc_ld<16>(v, addr);
    tc_ld<8>(v + 16, addr + 16);
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float2 fma_f32x2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.ftz.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 mul_f32x2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.ftz.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// Bounded mbarrier wait of a pipeline: once one wait has run out, `dead` lets all others pass at once (the call is then
// reported as failed; what is computed meanwhile is not used).
__device__ __forceinline__ void tc_wait(unsigned bar, unsigned parity, volatile int* dead) {
    for (int i = 0; i < MBAR_POLL_LIMIT; i++) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return;
        if ((i & 63) == 63 && *dead) return;
    }
    *dead = 1;
}

// ------------------------------------------------------------------ weights: registers -> operand tile

// Two f16 integers 0 .. 255 out of bytes of w: the byte under an exponent that makes the f16 1024 + byte.
template <int PAIR>
__device__ __forceinline__ __half2 tc_bytes_1024(unsigned w) {
    const unsigned r = __byte_perm(w, 0x64646464u, PAIR ? 0x4342 : 0x4140);
    return *reinterpret_cast<const __half2*>(&r);
}
__device__ __forceinline__ unsigned tc_bits(__half2 h) { return *reinterpret_cast<const unsigned*>(&h); }

// Raw words of half g of a 256-weight block (two stages of 64 weights) that a thread turns into operand values.
struct RawQ4 {
    static constexpr int PLANES = 1;
    unsigned s0, s1, s2;  // scale words of the header
    unsigned n0, n1, n2;  // of the next block's
    unsigned w[2][8];     // 64 weights: [stage of the half]
    // Stage i of the half; the header with the first one, because its words are needed to the block's end.
    __device__ __forceinline__ void load_stage(int i, const uint8_t* data, int f, int g) {
        const uint8_t* p = data + (size_t)(f >> 5) * Q4_TILE_BYTES + (f & 31) * 16;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int4 v = ldg_stream(p + (1 + 2 * (2 * g + i) + h) * 512);
            w[i][4 * h] = v.x, w[i][4 * h + 1] = v.y, w[i][4 * h + 2] = v.z, w[i][4 * h + 3] = v.w;
        }
        if (i == 0) {
            const int4 hdr = ldg_stream(p);
            n0 = (unsigned)hdr.y, n1 = (unsigned)hdr.z, n2 = (unsigned)hdr.w;
        }
    }
    __device__ __forceinline__ void begin_block() { s0 = n0, s1 = n1, s2 = n2; }
    // The eight mins of a block as tf32 (the first 32 bytes of a row).
    __device__ __forceinline__ void store_mins(unsigned char* tile, int row) const {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned m = h ? ((s2 >> 4) & 0x0f0f0f0fu) | (((s1 >> 6) & 0x03030303u) << 4) : s1 & 0x3f3f3f3fu;
            *reinterpret_cast<float4*>(tile + tc_swz(row, h)) =
                make_float4(i2f_small((int)(m & 0xff)), i2f_small((int)((m >> 8) & 0xff)), i2f_small((int)((m >> 16) & 0xff)), i2f_small((int)(m >> 24)));
        }
    }
    // 64 weights of stage 2 g + i: low nibbles = sub-block 2 (2 g + i), high nibbles the next (kernels/common.cu:40-84)
    __device__ __forceinline__ void store(int i, unsigned char* tile, int row, int g, int) const {
        const unsigned sc4 = g == 0 ? s0 & 0x3f3f3f3fu : (s2 & 0x0f0f0f0fu) | (((s0 >> 6) & 0x03030303u) << 4);
        const __half2 bias = __half2half2(__ushort_as_half(0x6400)), m1024 = __half2half2(__ushort_as_half(0xe400));
        const unsigned sa = __byte_perm(sc4, 0x64646464u, i ? 0x4242 : 0x4040), sb = __byte_perm(sc4, 0x64646464u, i ? 0x4343 : 0x4141);
        const __half2 scl = __hsub2(*reinterpret_cast<const __half2*>(&sa), bias), sch = __hsub2(*reinterpret_cast<const __half2*>(&sb), bias);
        const __half2 ofl = __hmul2(scl, m1024), ofh = __hmul2(sch, m1024);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            unsigned lo[4], hi[4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const unsigned x = w[i][2 * c + k], l = x & 0x0f0f0f0fu, u = (x >> 4) & 0x0f0f0f0fu;
                // (1024 + q) * sc - 1024 * sc: both products below 2^16, the difference q * sc exact
                lo[2 * k] = tc_bits(__hfma2(tc_bytes_1024<0>(l), scl, ofl)), lo[2 * k + 1] = tc_bits(__hfma2(tc_bytes_1024<1>(l), scl, ofl));
                hi[2 * k] = tc_bits(__hfma2(tc_bytes_1024<0>(u), sch, ofh)), hi[2 * k + 1] = tc_bits(__hfma2(tc_bytes_1024<1>(u), sch, ofh));
            }
            *reinterpret_cast<uint4*>(tile + tc_swz(row, c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            *reinterpret_cast<uint4*>(tile + tc_swz(row, 4 + c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
};

struct RawQ6 {
    static constexpr int PLANES = 2;
    unsigned sc[2];  // the half's eight scales
    unsigned la[8], lb[8], hq[8];
    // Both stages of the half use the same words, in different bits: they come with the second.
    __device__ __forceinline__ void load_stage(int i, const uint8_t* data, int f, int g) {
        if (i == 0) return;
        const uint8_t* p = data + (size_t)(f >> 5) * Q6_TILE_BYTES + (f & 31) * 16;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int4 a = ldg_stream(p + (4 * g + h) * 512), b = ldg_stream(p + (4 * g + 2 + h) * 512), c = ldg_stream(p + (8 + 2 * g + h) * 512);
            la[4 * h] = a.x, la[4 * h + 1] = a.y, la[4 * h + 2] = a.z, la[4 * h + 3] = a.w;
            lb[4 * h] = b.x, lb[4 * h + 1] = b.y, lb[4 * h + 2] = b.z, lb[4 * h + 3] = b.w;
            hq[4 * h] = c.x, hq[4 * h + 1] = c.y, hq[4 * h + 2] = c.z, hq[4 * h + 3] = c.w;
        }
        const uint2 s = __ldg(reinterpret_cast<const uint2*>(p + 12 * 512 + 8 * g));
        sc[0] = s.x, sc[1] = s.y;
    }
    __device__ __forceinline__ void begin_block() {}
    // 64 weights of stage 2 g + i = runs j = 2 i, 2 i + 1 of half g (kernels/gemv.cu:302-337, as in block_dot):
    // scale * (q - 32) as its f16 rounding and the residual (0 or +-1: |scale * q| <= 4096)
    __device__ __forceinline__ void store(int i, unsigned char* tile, int row, int, int plane_bytes) const {
        const __half2 off = __half2half2(__ushort_as_half(0x6420));  // 1024 + 32
#pragma unroll
        for (int jl = 0; jl < 2; jl++) {
            const int j = 2 * i + jl;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int h = c >> 1;  // scale byte 2 j + h of the half
                const __half2 sch = __half2half2(__int2half_rn((int)(signed char)((sc[i] >> (8 * (2 * jl + h))) & 0xff)));
                unsigned hi[4], lo[4];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const unsigned nib = jl ? lb[2 * c + k] : la[2 * c + k];
                    const unsigned q = ((nib >> (4 * i)) & 0x0f0f0f0fu) | (((hq[2 * c + k] >> (2 * j)) & 0x03030303u) << 4);
                    const __half2 q0 = __hsub2(tc_bytes_1024<0>(q), off), q1 = __hsub2(tc_bytes_1024<1>(q), off);
                    const __half2 p0 = __hmul2(sch, q0), p1 = __hmul2(sch, q1);
                    hi[2 * k] = tc_bits(p0), hi[2 * k + 1] = tc_bits(p1);
                    lo[2 * k] = tc_bits(__hfma2(sch, q0, __hneg2(p0))), lo[2 * k + 1] = tc_bits(__hfma2(sch, q1, __hneg2(p1)));
                }
                *reinterpret_cast<uint4*>(tile + tc_swz(row, 4 * jl + c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(tile + plane_bytes + tc_swz(row, 4 * jl + c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
};

// ------------------------------------------------------------------ the kernel

// The tokens are the rows of the product (128 lanes of TMEM per CTA), the weight rows its columns: a thread that drains an
// accumulator has one token, whose d8 it holds in a register, and the columns' d come once a block.  (The other way round every
// d8 was a broadcast read of shared memory: 770 of 2 000 cycles a stage.)
//
// CTA = 128 tokens x a tile of 96 weight rows x a part of the k range, in stages of 64 weights (and one for the mins of a block).
// Lane 0 of warps 1 and 3 requests the tokens' operand as bulk copies, the unpacking warps turn weights into the other
// operand, lane 0 of warps 0 and 2 issues the MMAs, the sixteen warps behind drain the accumulators (two buffers in TMEM, each
// with the two groups of a stage side by side) into the block's and the row's sums they hold in registers (TMEM lanes
// 32 (w & 3) .., a quarter of the columns); every role runs ahead of the next as far as the rings allow.
//
// Gate / up pairs (ZIP) alternate the two matrices' rows in the tile, so that a thread holds a gate value beside its up value,
// as the two rows of a RoPE pair.  The k range is cut over the CTAs of a cluster (grid.y) where a matrix has too few rows to
// fill the chip, or so many blocks that a chain of additions over them would cost precision: the parts' sums meet through
// distributed shared memory, each CTA finishing its share of the columns.
constexpr int TC_C_WARPS = 4, TC_D_WARPS = 16, TC_MAX_STAGES = 8, TC_LANES = 128, TC_ROWS = 96, TC_COLSCALE_BYTES = TC_D_WARPS * 2 * (TC_ROWS / 4) * 4;
constexpr int TC_SUM_STRIDE = TC_ROWS / 2 + 1;  // float2 of a token's sums in the epilogue; odd, so that 16 tokens' pairs lie in 32 banks
constexpr size_t TC_SMEM_MAX = 225 * 1024;
// Unpacking warps, two threads per row, one for each half of its blocks (a warpgroup's registers change together: the last two
// idle; two threads on every stage paid the ring's price, 900 of 1 500 cycles, twice as often), and the registers of a
// thread of each role; what they add up to is what the launch has.
constexpr int TC_A_WARPS = 8, TC_A_BUSY = TC_ROWS / 16, TC_THREADS = 32 * (TC_C_WARPS + TC_A_WARPS + TC_D_WARPS), TC_LAUNCH_REGS = 72;
template <bool Q4>
struct TcRegs {
    static constexpr int C = 24, A = Q4 ? 48 : 64, D = Q4 ? 96 : 88;
    static_assert(32 * (TC_C_WARPS * C + TC_A_WARPS * A + TC_D_WARPS * D) <= TC_THREADS * TC_LAUNCH_REGS && TC_THREADS * TC_LAUNCH_REGS <= 65536,
                  "more registers than the launch has");
};
// Registers of a role: N of the LAUNCH a thread has.  Fewer must be given back, more asked for.
template <int N>
__device__ __forceinline__ void tc_regs() {
    static_assert(N % 8 == 0, "");
    if constexpr (N < TC_LAUNCH_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
    else if constexpr (N > TC_LAUNCH_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// Most blocks a CTA adds up one after the other.  The rounding of such a chain grows with the root of its length: Q6_K rows of 43
// and 108 blocks in one piece 1.30e-7 and 1.94e-7 against float64, in pieces of 22 and 27 1.04e-7 and 1.16e-7 (dp4a, which adds
// them as a tree, 0.93e-7 and 0.98e-7).
constexpr int TC_CHAIN = 27;

struct TcArgs {
    const unsigned char* image;
    int M, Mp;       // tokens, with padding
    Mat A1, A2;      // ZIP: the pair; otherwise A2 (optional) follows A1 in the grid
    int tiles1;      // row tiles of A1
    int id1, id2, zip, nst;
    int ahead;       // row tiles between a CTA and the one that takes its place (0: none does)
    ChunkEpi epi;
    TokenState* st;
};

// Position in a ring of n slots: slot, and the parity of the lap.
struct TcRing {
    int slot = 0;
    unsigned lap = 0;
    __device__ __forceinline__ void next(int n) {
        if (++slot == n) slot = 0, lap ^= 1;
    }
};

template <class RAW>
__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_tc(const TcArgs a) {
    constexpr bool Q4 = RAW::PLANES == 1;
    using Regs = TcRegs<Q4>;
    constexpr int NC = TC_ROWS / (TC_D_WARPS / 4);  // columns of a draining warp
    constexpr int SPB = Q4 ? 5 : 4;                 // stages of a block: four of weights, one of mins
    constexpr int T_BYTES = TC_LANES * 128, W_PLANE = TC_ROWS * 128, STAGE = T_BYTES + RAW::PLANES * W_PLANE;
    extern __shared__ __align__(128) unsigned char tc_smem_raw[];
    __shared__ unsigned long long bars[2 * TC_MAX_STAGES + 4];
    __shared__ unsigned tmem_slot;
    __shared__ int dead_s;
    volatile int* dead = &dead_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned full = smem_u32(bars), empty = full + 8 * TC_MAX_STAGES, accfull = empty + 8 * TC_MAX_STAGES, accempty = accfull + 16;
    const int S = gridDim.y, part = blockIdx.y;  // k parts
    const int n0 = blockIdx.z * TC_LANES, nt = min(TC_LANES, a.Mp - n0), nst = a.nst;  // this CTA's tokens
    const int tile = blockIdx.x;
    const bool second = !a.zip && a.A2.data != nullptr && tile >= a.tiles1;
    const Mat& A = second ? a.A2 : a.A1;
    const int nb = A.nb, K = A.K, N = A.N;
    const int row0 = (tile - (second ? a.tiles1 : 0)) * (a.zip ? TC_ROWS / 2 : TC_ROWS);
    const int b0 = nb * part / S, b1 = nb * (part + 1) / S;
    if (warp == 3) {
        // The rows this CTA unpacks start towards L2 at once, and so do those of the CTA that will follow on this SM: the registers
        // of the unpacking warps hold one block ahead, which covers an L2 hit but not a trip to memory.
        auto ahead = [&](const Mat& m, int row) {
            if (row >= m.N) return;
            const size_t f = mat_flat(nb, row, 0), t0 = (f + ROW_GROUP * b0) >> 5, t1 = (f + ROW_GROUP * b1 + 31) >> 5;
            constexpr size_t TB = Q4 ? Q4_TILE_BYTES : Q6_TILE_BYTES;
            bulk_prefetch_l2(m.data + t0 * TB, (unsigned)((t1 - t0) * TB));
        };
        for (int w = 0; w <= 1; w++) {
            if (w == 1 && a.ahead == 0) break;
            const int t = row0 + w * a.ahead * (a.zip ? TC_ROWS / 2 : TC_ROWS);
            if (lane < TC_ROWS / ROW_GROUP) {
                if (a.zip) ahead(lane & 1 ? a.A2 : A, t + (lane >> 1) * ROW_GROUP);
                else ahead(A, t + lane * ROW_GROUP);
            }
        }
    }
    const int stages = SPB * (b1 - b0);
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr unsigned ACC_COLS = 2 * TC_ROWS, TMEM_COLS = 512;  // the rows for a stage's first and second group, twice
    float* colscales = reinterpret_cast<float*>(smem + (size_t)nst * STAGE);  // d and -dmin of every draining warp's columns
    if (tid == 0) {
        for (int i = 0; i < nst; i++) {
            mbar_init(bars + i, TC_A_BUSY / 2 + 1);  // the warps that unpack a half and the tokens (with the bytes)
            mbar_init(bars + TC_MAX_STAGES + i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(bars + 2 * TC_MAX_STAGES + i, 1);
            mbar_init(bars + 2 * TC_MAX_STAGES + 2 + i, TC_D_WARPS);
        }
        dead_s = 0;
        mbar_fence_init();
    }
    if (warp == 0) tc_alloc(&tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_slot;

    if (warp < TC_C_WARPS) {
        tc_regs<Regs::C>();
        if ((warp & 1) == 0) {
            // Two issuing warps take turns by accumulator: with 28 warps at work a wait costs one 300 cycles even when there is
            // nothing to wait for.  The whole warp walks the loop and one thread of it issues: that way operands stand in uniform
            // registers.
            TcRing ring;
            const unsigned long long d0 = tc_desc(smem_u32(smem));
            const unsigned id = tc_idesc(0, TC_LANES, TC_ROWS), idm = tc_idesc(2, TC_LANES, TC_ROWS);
            const int buf = __shfl_sync(TFR_FULL_MASK, warp >> 1, 0);
            const unsigned acc = __shfl_sync(TFR_FULL_MASK, tmem, 0) + buf * ACC_COLS;
            if (buf) ring.next(nst);
            for (int j = buf; j < stages; j += 2) {
                tc_wait(full + 8 * ring.slot, ring.lap, dead);
                // what the unpacking warps stored becomes visible to the tensor core here, not where they store it: a
                // fence there waits for the warp's loads in flight, the next block's words (900 to 2 200 cycles a block)
                fence_proxy_async();
                const unsigned long long dt = d0 + ((ring.slot * STAGE) >> 4), dw = dt + (T_BYTES >> 4);
                if (j >= 2) tc_wait(accempty + 8 * buf, ((j >> 1) - 1) & 1, dead);  // last: nothing else stands behind the draining
                tc_fence_after();
                if (tc_elect()) {
                    if (Q4 && j % SPB == 4) {
                        // high terms of the group sums to the first columns, low terms to the second
                        const int odd = 4 * ((b0 + j / SPB) & 1);
                        tc_mma<true>(acc, dt + odd, dw, idm, 0);
                        tc_mma<true>(acc + TC_ROWS, dt + odd + 2, dw, idm, 0);
                    } else {
#pragma unroll
                        for (int kk = 0; kk < 4; kk++) {
                            tc_mma<false>(acc + (kk >> 1) * TC_ROWS, dt + 2 * kk, dw + 2 * kk, id, kk & 1);
                            if (!Q4) tc_mma<false>(acc + (kk >> 1) * TC_ROWS, dt + 2 * kk, dw + (W_PLANE >> 4) + 2 * kk, id, 1);
                        }
                    }
                    tc_commit(accfull + 8 * buf);
                    tc_commit(empty + 8 * ring.slot);
                }
                __syncwarp();
                ring.next(nst);
                ring.next(nst);
            }
        } else {
            // two threads take turns: a bulk request costs the one that makes it 300 to 560 cycles
            griddep_wait();  // the image comes from the previous kernel
            if (lane == 0) {
                TcRing ring;
                const size_t plane = (size_t)a.Mp * 128;
                const unsigned char* src = a.image + (size_t)n0 * 128;
                if (warp >> 1) ring.next(nst);
                for (int j = warp >> 1; j < stages; j += 2) {
                    const int b = b0 + j / SPB, s = j % SPB;
                    if (j >= nst) tc_wait(empty + 8 * ring.slot, ring.lap ^ 1, dead);
                    unsigned long long* bar = bars + ring.slot;
                    mbar_expect_tx(bar, nt * 128);
                    bulk_load(smem + ring.slot * STAGE, src + (s == 4 ? tc_sums_at(K, a.Mp) + (b >> 1) * plane : (4 * b + s) * plane), nt * 128, bar);
                    ring.next(nst);
                    ring.next(nst);
                }
            }
            __syncwarp();
        }
        griddep_launch_dependents();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * (TC_D_WARPS + TC_C_WARPS)) : "memory");  // the last accumulator has been read
        tc_fence_after();
        if (warp == 0) tc_dealloc(tmem, TMEM_COLS);
        if (S > 1) cluster_sync_all();
        if (S > 1) cluster_sync_all();
        return;
    }

    if (warp < TC_C_WARPS + TC_A_WARPS) {
        tc_regs<Regs::A>();
        const int ta = tid - 32 * TC_C_WARPS;
        griddep_launch_dependents();
        if (ta < 2 * TC_ROWS) {
            // three warps per half of the blocks, a thread per row; rows past the matrix repeat its last row
            const int g = ta >= TC_ROWS, row_l = ta - g * TC_ROWS;
            const uint8_t* wdata = (a.zip && (row_l & 1)) ? a.A2.data : A.data;
            const int f0 = (int)mat_flat(nb, min(row0 + (a.zip ? row_l >> 1 : row_l), N - 1), 0);
            RAW raw;
            raw.load_stage(0, wdata, f0 + ROW_GROUP * b0, g);  // weights do not depend on earlier kernels
            raw.load_stage(1, wdata, f0 + ROW_GROUP * b0, g);
            int slot = 0, j0 = 0;  // of the block's first stage
            unsigned lap = 0;
            // stage s of the block: its slot free, filled by `fill`, handed on
            auto stage = [&](int s, auto&& fill) {
                const bool wrap = slot + s >= nst;
                const int at = slot + s - (wrap ? nst : 0);
                if (j0 + s >= nst) tc_wait(empty + 8 * at, (lap ^ (wrap ? 1u : 0u)) ^ 1u, dead);
                fill(smem + at * STAGE + T_BYTES);
                __syncwarp();
                if (lane == 0) tc_arrive(full + 8 * at);
            };
            for (int b = b0; b < b1; b++) {
                raw.begin_block();
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    stage(2 * g + i, [&](unsigned char* t) { raw.store(i, t, row_l, g, W_PLANE); });
                    if (b + 1 < b1) raw.load_stage(i, wdata, f0 + ROW_GROUP * (b + 1), g);  // the words just used, of the next block
                }
                if constexpr (Q4)
                    if (g == (b & 1)) stage(4, [&](unsigned char* t) { raw.store_mins(t, row_l); });
                j0 += SPB, slot += SPB;
                if (slot >= nst) slot -= nst, lap ^= 1;
            }
        }
        if (S > 1) cluster_sync_all();
        if (S > 1) cluster_sync_all();
        return;
    }

    tc_regs<Regs::D>();
    const int dwarp = warp - TC_C_WARPS - TC_A_WARPS, quad = warp & 3, cg = dwarp >> 2, tok = quad * 32 + lane, m = n0 + tok;
    static_assert(NC == 24 && TC_COLSCALE_BYTES == TC_D_WARPS * 2 * NC * 4, "");
    float* colscale = colscales + dwarp * 2 * NC;
    float2 tot[NC / 2];  // of the token and its columns: over the row
#pragma unroll
    for (int i = 0; i < NC / 2; i++) tot[i] = make_float2(0.f, 0.f);
    {
        // lanes below NC hold a column's d, and dmin above it, a block ahead
        const int col = cg * NC + min(lane, NC - 1);
        const uint8_t* ddata = (a.zip && (col & 1)) ? a.A2.data : A.data;
        const int df = (int)mat_flat(nb, min(row0 + (a.zip ? col >> 1 : col), N - 1), 0);
        auto load_d = [&](int b) {
            const int f = df + ROW_GROUP * b;
            return Q4 ? __ldg(reinterpret_cast<const unsigned*>(ddata + (size_t)(f >> 5) * Q4_TILE_BYTES + (f & 31) * 16))
                      : (unsigned)__ldg(reinterpret_cast<const unsigned short*>(ddata + (size_t)(f >> 5) * Q6_TILE_BYTES + Q6_PIECES * 512 + (f & 31) * 2));
        };
        unsigned dnext = load_d(b0);
        griddep_launch_dependents();
        griddep_wait();  // nothing reaches an accumulator before the image is complete; residuals are then, too
        const unsigned lanes = tmem + ((unsigned)quad << 21) + cg * NC;
        float2 sum[NC / 2];  // of the block without its d
        // d8 of the token's groups, two stages ahead
        const float2* d8 = reinterpret_cast<const float2*>(a.image + tc_d8_at(K, a.Mp)) + (size_t)(4 * b0) * a.Mp + min(m, a.Mp - 1);
        const int d8_end = 4 * (b1 - b0);
        auto load_d8 = [&](int i) { return __ldcg(d8 + (size_t)min(i, d8_end - 1) * a.Mp); };  // L1 may hold the last image
        float2 knext[2] = {load_d8(0), load_d8(1)};
        int j = 0;
        float v[NC];
        // the two accumulators of stage j, one after the other: use(which)
        auto drain = [&](auto&& use) {
            const int buf = j & 1;
            tc_wait(accfull + 8 * buf, (j >> 1) & 1, dead);
            tc_fence_after();
#pragma unroll
            for (int g = 0; g < 2; g++) {
                tc_ld24(v, lanes + buf * ACC_COLS + g * TC_ROWS);
                tc_ld_wait();
                if (g == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc_arrive(accempty + 8 * buf);
                }
                use(g);
            }
            j++;
        };
        for (int b = b0; b < b1; b++) {
            if (lane < NC) {
                colscale[lane] = f16_to_f32((unsigned short)dnext);
                if (Q4) colscale[NC + lane] = -f16_to_f32((unsigned short)(dnext >> 16));
            }
            if (b + 1 < b1) dnext = load_d(b + 1);
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const float2 k = knext[s & 1];
                knext[s & 1] = load_d8(4 * (b - b0) + s + 2);
                drain([&](int g) {
                    const float kg = g ? k.y : k.x;
#pragma unroll
                    for (int i = 0; i < NC / 2; i++) {
                        const float2 t = make_float2(v[2 * i], v[2 * i + 1]);
                        sum[i] = s == 0 && g == 0 ? mul_f32x2(t, make_float2(kg, kg)) : fma_f32x2(t, make_float2(kg, kg), sum[i]);
                    }
                });
            }
            // the block's d * sums - dmin * mins, and once more rounded into the row's sum
            const float4* dc = reinterpret_cast<const float4*>(colscale);
#pragma unroll
            for (int i = 0; i < NC / 4; i++) {
                const float4 d = dc[i];
                sum[2 * i] = mul_f32x2(make_float2(d.x, d.y), sum[2 * i]), sum[2 * i + 1] = mul_f32x2(make_float2(d.z, d.w), sum[2 * i + 1]);
            }
            if constexpr (Q4)
                drain([&](int) {
#pragma unroll
                    for (int i = 0; i < NC / 4; i++) {
                        const float4 m = dc[NC / 4 + i];
                        sum[2 * i] = fma_f32x2(make_float2(m.x, m.y), make_float2(v[4 * i], v[4 * i + 1]), sum[2 * i]);
                        sum[2 * i + 1] = fma_f32x2(make_float2(m.z, m.w), make_float2(v[4 * i + 2], v[4 * i + 3]), sum[2 * i + 1]);
                    }
                });
#pragma unroll
            for (int i = 0; i < NC / 2; i++) tot[i] = fma_f32x2(make_float2(1.f, 1.f), sum[i], tot[i]);
            __syncwarp();  // the columns' scales have been read
        }
    }
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(32 * (TC_D_WARPS + TC_C_WARPS)) : "memory");

    // ---- epilogue.  A gate/up tile whose rows all exist leaves straight from the registers, twelve values of a token in three
    // stores (gate and up of 2 048 tokens 4 % faster than the other way).  All else goes as [token][pair of columns] through
    // shared memory (of the cluster's CTAs), then lanes along the columns: RoPE pairs, rows with residuals.  A thread's own token
    // and columns would touch 32 rows of the output with every access (a down projection of 2 048 tokens: 620 us).
    const int id_base = second ? a.id2 : a.id1;
    if (S == 1 && a.epi.kind == CEPI_SILU && row0 + TC_ROWS / 2 <= N && ((a.epi.ldo | (id_base + row0)) & 3) == 0 &&
        (reinterpret_cast<uintptr_t>(a.epi.out) & 15) == 0) {
        if (m < a.M) {
            float4* o = reinterpret_cast<float4*>(a.epi.out + (size_t)m * a.epi.ldo + id_base + row0 + cg * (NC / 2));
#pragma unroll
            for (int i = 0; i < NC / 2; i += 4) {
                float h[4];
#pragma unroll
                for (int q = 0; q < 4; q++) h[q] = (tot[i + q].x / (1.f + __expf(-tot[i + q].x))) * tot[i + q].y;  // as ChunkEpiTok::apply
                o[i / 4] = make_float4(h[0], h[1], h[2], h[3]);
            }
        }
        if (tid == 32 * (TC_C_WARPS + TC_A_WARPS) && dead_s && a.st) a.st->err = 2;
        return;
    }
    constexpr int PAIRS = TC_ROWS / 2, BATCH = 4;
    float2* mine = reinterpret_cast<float2*>(smem) + tok * TC_SUM_STRIDE + cg * (NC / 2);
#pragma unroll
    for (int i = 0; i < NC / 2; i++) mine[i] = tot[i];
    if (S > 1) cluster_sync_all();
    else asm volatile("bar.sync 2, %0;" ::"n"(32 * TC_D_WARPS) : "memory");
    const int td = tid - 32 * (TC_C_WARPS + TC_A_WARPS);
    const int t0 = TC_LANES * part / S, items = min(TC_LANES / S, a.M - n0 - t0) * PAIRS;  // S is a power of two
    const bool res = a.epi.kind == CEPI_STORE && a.epi.use_res == 2;
    ChunkEpi epi = a.epi;
    epi.use_res = 0;
    for (int k0 = td; k0 < items; k0 += BATCH * 32 * TC_D_WARPS) {
        // the parts' sums and the residuals of four items in flight together
        float2 v[BATCH], r[BATCH];
        int m[BATCH], id[BATCH];
#pragma unroll
        for (int q = 0; q < BATCH; q++) {
            const int k = k0 + q * 32 * TC_D_WARPS, t = t0 + k / PAIRS, pair = k % PAIRS;
            const int row = row0 + (a.zip ? pair : 2 * pair);
            const bool on = k < items && row < N;
            m[q] = n0 + t, id[q] = on ? id_base + (a.zip ? row : row >> 1) : -1;
            v[q] = r[q] = make_float2(0.f, 0.f);
            if (!on) continue;
            if (res) {
                const float* o = epi.out + (size_t)m[q] * epi.ldo + 2 * id[q];
                r[q].x = o[0];
                if (2 * id[q] + 1 < epi.n_rows) r[q].y = o[1];
            }
            const unsigned at = smem_u32(smem) + (t * TC_SUM_STRIDE + pair) * 8;
#pragma unroll
            for (int p = 0; p < 8; p++) {
                if (p >= S) break;
                float2 x;
                unsigned remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(p));
                asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(x.x), "=f"(x.y) : "r"(remote) : "memory");
                v[q].x += x.x, v[q].y += x.y;
            }
        }
#pragma unroll
        for (int q = 0; q < BATCH; q++)
            if (id[q] >= 0) ChunkEpiTok{&epi, m[q]}.apply(id[q], v[q].x + r[q].x, v[q].y + r[q].y);
    }
    if (tid == 32 * (TC_C_WARPS + TC_A_WARPS) && dead_s && a.st) a.st->err = 2;
    if (S > 1) cluster_sync_all();  // nobody leaves while others read its sums
}

// ------------------------------------------------------------------ rows on the fp32 activation route

// The Q6_K attn_v rows against the unquantised normalised vectors (kernels/gemv.cu:233-264), bit for bit what the decode
// kernel computes: a run of 16 products as one chain of multiply-adds, lane l summing runs l, l + 32, ... in order, then
// the warp's butterfly.  A warp unpacks the weights of its rows once, two rows to a packed multiply-add, and walks its
// tokens; the sums meet in a halving butterfly, the same tree as warp_sum, which leaves one row pair of one token per lane.
//   staged   more than 16 tokens: eight rows x eight tokens a warp, the warps of a CTA on different rows share the tokens'
//            vectors in shared memory.  Bound by multiply-adds and the reads that feed them (one 16-byte read per 16 packed
//            multiply-adds): 256 rows x 2 048 x 2 048 tokens 99 us; 161 with four rows, single multiply-adds and an integer
//            conversion per weight.
//   direct   up to 16 tokens: four rows x four tokens a warp, the warps of a CTA on different tokens, vectors straight
//            from L2: latency is all there is (nine tokens 6.5 us; eight CTAs of a staged form took 21).
constexpr int TCV_WARPS = 8, TCV_DIRECT_MAX = 16;

// tt: tokens per CTA (staged: as many of the TOK as fit shared memory)
template <int ROWS, int TOK, bool STAGED>
__global__ void __launch_bounds__(TCV_WARPS * 32, 1) k_rows_f32(Mat w, int id_base, const float* xn, int M, int tt, ChunkEpi epi) {
    extern __shared__ __align__(128) unsigned char tcv_smem_raw[];
    float* xs = reinterpret_cast<float*>(tcv_smem_raw);
    constexpr int U = STAGED ? 1 : 2, RP = ROWS / 2;  // runs per step, row pairs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, K = w.K, nb = w.nb, per_row = 16 * nb;
    const int row0 = (STAGED ? blockIdx.x * (blockDim.x >> 5) + warp : blockIdx.x) * ROWS;
    const int m0 = STAGED ? blockIdx.y * tt : warp * TOK, mt = min(STAGED ? tt : TOK, M - m0);
    const int xf = (int)xs_floats(K);
    float2 wt[U][RP][16], s[TOK * RP];  // rows 2 r, 2 r + 1; sums [token][row pair]
    // run 16 of a block's row as in q6k_run_weights_f32: d * scale * (q - 32), four bytes of q at a time
    auto unpack = [&](int i0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int run = min(i0 + 32 * u, per_row - 1), c = run & 15;
            const int n = c >> 3, j = (c >> 1) & 3, is = c & 1, nsh = 4 * (j >> 1), hsh = 2 * j;
#pragma unroll
            for (int r = 0; r < RP; r++) {
                unsigned ql[2][4], qh[2][4];
                float dsc[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const long long f = mat_flat(nb, min(row0 + 2 * r + i, w.N - 1), run >> 4);
                    const uint8_t* t = w.data + (f >> 5) * Q6_TILE_BYTES;
                    const uint8_t* p = t + (f & 31) * 16;
                    const int4 a = __ldg(reinterpret_cast<const int4*>(p + (4 * n + 2 * (j & 1) + is) * 512));
                    const int4 b = __ldg(reinterpret_cast<const int4*>(p + (8 + 2 * n + is) * 512));
                    ql[i][0] = a.x, ql[i][1] = a.y, ql[i][2] = a.z, ql[i][3] = a.w;
                    qh[i][0] = b.x, qh[i][1] = b.y, qh[i][2] = b.z, qh[i][3] = b.w;
                    const float sc = (float)(int)*reinterpret_cast<const signed char*>(p + 12 * 512 + 8 * n + is + 2 * j);
                    dsc[i] = f16_to_f32(__ldg(reinterpret_cast<const unsigned short*>(t + Q6_PIECES * 512 + (f & 31) * 2))) * sc;
                }
                const float2 d2 = make_float2(dsc[0], dsc[1]);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    unsigned q[2];
#pragma unroll
                    for (int i = 0; i < 2; i++) q[i] = ((ql[i][k] >> nsh) & 0x0f0f0f0fu) | (((qh[i][k] >> hsh) & 0x03030303u) << 4);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        // the byte under the exponent that makes it 2^23 + q, minus 2^23 + 32: exact
                        const float2 v = make_float2(__uint_as_float(__byte_perm(q[0], 0x4b000000u, 0x7440 + e)) - 8388640.f,
                                                     __uint_as_float(__byte_perm(q[1], 0x4b000000u, 0x7440 + e)) - 8388640.f);
                        wt[u][r][4 * k + e] = mul_f32x2(v, d2);
                    }
                }
            }
        }
    };
    unpack(lane);  // weights do not depend on earlier kernels
    griddep_wait();
    griddep_launch_dependents();
    if (STAGED) {
        const int n4 = K >> 2;
        for (int t = 0; t < mt; t++)
            for (int i4 = tid; i4 < n4; i4 += blockDim.x) cp_async16(xs + t * xf + xs_idx(4 * i4), xn + (size_t)(m0 + t) * K + 4 * i4, 16);
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
    }
    if (row0 >= w.N) return;
#pragma unroll
    for (int i = 0; i < TOK * RP; i++) s[i] = make_float2(0.f, 0.f);
    const float2 one = make_float2(1.f, 1.f);
    for (int i0 = lane; i0 < per_row; i0 += 32 * U) {
        if (i0 != lane) unpack(i0);
#pragma unroll
        for (int t = 0; t < TOK; t++) {
            if (t >= mt) break;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int run = i0 + 32 * u;
                if (run < per_row) {
                    const float4* x4 = reinterpret_cast<const float4*>(STAGED ? xs + t * xf + xs_idx(16 * run) : xn + (size_t)(m0 + t) * K + 16 * run);
                    float2 acc[RP];
#pragma unroll
                    for (int r = 0; r < RP; r++) acc[r] = make_float2(0.f, 0.f);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float4 x = x4[k];
                        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int e = 0; e < 4; e++)
#pragma unroll
                            for (int r = 0; r < RP; r++) acc[r] = fma_f32x2(wt[u][r][4 * k + e], make_float2(xv[e], xv[e]), acc[r]);
                    }
#pragma unroll
                    for (int r = 0; r < RP; r++) s[t * RP + r] = fma_f32x2(acc[r], one, s[t * RP + r]);
                }
            }
        }
    }
    int off = 16;
#pragma unroll
    for (int n = TOK * RP; n > 1; n >>= 1, off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            const float2 send = up ? s[i] : s[i + n / 2], keep = up ? s[i + n / 2] : s[i];
            s[i].x = keep.x + __shfl_xor_sync(TFR_FULL_MASK, send.x, off);
            s[i].y = keep.y + __shfl_xor_sync(TFR_FULL_MASK, send.y, off);
        }
    }
    for (; off > 0; off >>= 1) {
        s[0].x += __shfl_xor_sync(TFR_FULL_MASK, s[0].x, off);
        s[0].y += __shfl_xor_sync(TFR_FULL_MASK, s[0].y, off);
    }
    constexpr int SHARE = 32 / (TOK * RP);  // lanes with the same sums
    const int i = lane / SHARE, t = i / RP, row = row0 + 2 * (i % RP);
    if (lane % SHARE == 0 && t < mt && row < w.N) ChunkEpiTok{&epi, m0 + t}.apply(id_base + (row >> 1), s[0].x, s[0].y);
}
inline cudaError_t launch_rows_f32(cudaStream_t stream, int sms, const Mat& w, int id_base, const float* xn, int M, const ChunkEpi& epi) {
    if (M <= TCV_DIRECT_MAX)
        return launch_pdl(k_rows_f32<4, 4, false>, dim3((w.N + 3) / 4), dim3(32 * ((M + 3) / 4)), 0, stream, w, id_base, xn, M, 4, epi);
    const size_t per = xs_floats(w.K) * sizeof(float);
    const int tt = std::min(8, (int)(GEMV_SMEM_MAX / per));
    if (tt < 1) return cudaErrorInvalidValue;
    const int tiles = (M + tt - 1) / tt;
    int warps = TCV_WARPS;  // fewer per CTA while that brings more SMs to work
    while (warps > 2 && (w.N + 8 * warps - 1) / (8 * warps) * tiles < sms) warps /= 2;
    return launch_pdl(k_rows_f32<8, 8, true>, dim3((w.N + 8 * warps - 1) / (8 * warps), tiles), dim3(32 * warps), tt * per, stream, w, id_base, xn, M,
                      tt, epi);
}

// CTAs of a kernel, one to an SM, that the device runs at once in clusters of S along grid.y (GPCs hold whole clusters): the
// driver's answer, asked once per device, kernel type and S.  threads: of a CTA; it is taken to fill the shared memory.
template <class F>
inline int cluster_ctas(F* kernel, int threads, int S, int sms) {
    static std::atomic<int> known[16][4];
    if (S <= 1) return sms;
    int dev = 0, slot = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return S;
    while ((1 << slot) < S) slot++;
    std::atomic<int>& k = known[dev & 15][slot];
    if (dev < 16 && k.load() > 0) return k.load();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(64, S);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = 200 * 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = S;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = sms / (2 * S);  // no answer: count on half of the chip
    }
    const int ctas = std::max(1, n) * S;
    if (dev < 16) k.store(ctas);
    return ctas;
}

inline bool tc_type(int type) { return type == TFR_Q4_K || type == TFR_Q6_K; }

template <class RAW>
inline cudaError_t launch_tc(cudaStream_t stream, int sms, TcArgs& a, int row_tiles, int S) {
    constexpr int stage = TC_LANES * 128 + RAW::PLANES * TC_ROWS * 128;
    a.nst = std::min(TC_MAX_STAGES, (int)((TC_SMEM_MAX - 1024 - TC_COLSCALE_BYTES) / stage));
    static_assert((TC_SMEM_MAX - 1024 - TC_COLSCALE_BYTES) / stage >= 5, "the ring holds a block's stages");
    a.ahead = S == 1 && row_tiles > sms ? sms : 0;
    static_assert(TC_LANES * TC_SUM_STRIDE * 8 <= 2 * stage, "the epilogue's sums lie over the first stages");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(row_tiles, S, (a.M + TC_LANES - 1) / TC_LANES);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = (size_t)a.nst * stage + TC_COLSCALE_BYTES + 1024;
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
    return cudaLaunchKernelEx(&cfg, k_gemm_tc<RAW>, (const TcArgs)a);
}

// out = epilogue(W x) for the M tokens of an operand image; jb: the second matrix of a gate/up pair or one that follows.
inline cudaError_t launch_gemm_tc(cudaStream_t stream, int sms, const unsigned char* image, int M, const RowJob& ja,
                                  const RowJob& jb, const ChunkEpi& epi, TokenState* st) {
    TcArgs a{};
    a.image = image, a.M = M, a.Mp = tc_pad_tokens(M);
    a.A1 = ja.m, a.A2 = jb.m, a.id1 = ja.id_base, a.id2 = jb.id_base;
    a.zip = epi.kind == CEPI_SILU;
    a.epi = epi, a.st = st;
    const int rows = a.zip ? TC_ROWS / 2 : TC_ROWS;
    a.tiles1 = (ja.m.N + rows - 1) / rows;
    const int tiles = a.tiles1 + (!a.zip && jb.m.data ? (jb.m.N + rows - 1) / rows : 0), groups = (M + TC_LANES - 1) / TC_LANES;
    // the number of k parts with the shortest longest chain: waves of CTAs x (blocks x what a block takes + the ends), in units of
    // a quarter of a block (0.8 us)
    int S = 1;
    double best = 1e30;
    for (int s = 1; s <= 8 && s <= ja.m.nb; s *= 2) {
        if (s < 8 && (ja.m.nb + s - 1) / s > TC_CHAIN) continue;
        const int ctas = tiles * groups * s, at_once = cluster_ctas(k_gemm_tc<RawQ4>, TC_THREADS, s, sms);
        const double t = (double)((ctas + at_once - 1) / at_once) * (4.5 * ((ja.m.nb + s - 1) / s) + 6 + (s > 1 ? 3 : 0));
        if (t < best) best = t, S = s;
    }
    return ja.m.type == TFR_Q4_K ? launch_tc<RawQ4>(stream, sms, a, tiles, S) : launch_tc<RawQ6>(stream, sms, a, tiles, S);
}

}  // namespace tfr
