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
//   What bounds it: instructions, and the waits between the roles.  A block of 256 weights x 96 rows x 128 tokens takes 4 300
//   cycles; the schedulers issue in 57 % of them, the tensor pipe works in 21 (768 tokens).  Gate and up rows of 2 048 inputs,
//   2 048 tokens: 477 us (before: 744), without the unpacking 433, without the MMAs 385, without the multiply-adds 433, with none of
//   them and without the blocks' ends 212.  11 008 inputs to 2 048 rows: 281 us (before: 326).
//   What made the difference: waits looked at before their loop (tc_wait), one hand-over for both groups of a stage (532 us with one
//   for each), d and dmin from TMEM (tc_mma of ones), a CTA that goes on with the next tile, no register spills (local memory is an
//   L2 round trip where shared memory takes all of L1).  Tried on the way: eight draining warps with 48 or 64 columns each (532 us),
//   one issuing warp (534), pairs of CTAs on one tile of rows (an arrival at the other CTA takes 1 000 cycles).  A CTA's first rows
//   into L2 at its entry, as the ones that follow: launches of several token tiles up to 7 % faster, of one tile on Q4_K up to 5 %
//   slower, prompts as before (77 tokens 5 251 and 5 228 us, 2 048 tokens 45 098 and 45 123).
//   Fixed costs are higher than with one tile a CTA: launches of a few blocks a CTA on Q6_K take 0.7 to 1 us more (512 inputs to 2 048
//   rows, 40 tokens, 11.1 -> 12.0 us).
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

constexpr int TC_PREP_THREADS = 512;  // at most
// As many threads as share a token's values out evenly, and the 256 that rms_scale_staged wants (2 048 tokens of 2 048 values with a
// norm, half of whose 512 threads had nothing to do: 17.2 -> 14.9 us).
inline int tc_prep_threads(int K) {
    const int n8 = K / 8, passes = (n8 + TC_PREP_THREADS - 1) / TC_PREP_THREADS;
    return std::max(256, ((n8 + passes - 1) / passes + 31) & ~31);
}
inline size_t tc_prep_smem(int K) { return (xs_floats(K) + 272) * sizeof(float); }

// One CTA per token (padding tokens included: they become zeros).  RMSNorm in the reference's reduction order
// (rms_scale_staged), the Q8 quantiser of act_quantize4 with eight values per thread.
__global__ void __launch_bounds__(TC_PREP_THREADS) k_prep_tc(PrepTcArgs a) {
    extern __shared__ __align__(128) unsigned char tcp_smem[];
    float* xs = reinterpret_cast<float*>(tcp_smem);
    float* red = xs + xs_floats(a.K);
    const int m = blockIdx.x, tid = threadIdx.x, K = a.K, n8 = K >> 3, Mp = gridDim.x, nt = blockDim.x;
    const bool live = m < a.M;
    const int row = m & 7;
    griddep_wait();
    griddep_launch_dependents();
    const float* x = a.x + (size_t)(live ? m : 0) * a.ldx;
    float scale = 1.f;
    if (a.normw) {
        for (int i4 = tid; i4 < (K >> 2); i4 += nt)
            *reinterpret_cast<float4*>(xs + xs_idx(4 * i4)) = reinterpret_cast<const float4*>(x)[i4];
        __syncthreads();
        scale = rms_scale_staged(xs, K, a.eps, red);
    }
    unsigned char* tok = a.image + (size_t)(m >> 3) * 1024;
    unsigned char* d8 = a.image + tc_d8_at(K, Mp) + (size_t)m * 8;
    for (int i0 = 0; i0 < n8; i0 += nt) {
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
            const int at = (k & 1) + 4 * (k >> 1);  // values 0, 2, 1, 3 of every four: the order in which weights unpack
            int q0 = 0, q1 = 0;
            if (g != 0.f) {
                q0 = (int)(signed char)__float2int_rn(v[at] / d);
                q1 = (int)(signed char)__float2int_rn(v[at + 2] / d);
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
// The same for a K-major operand without swizzle, 32 bytes a row: cores of 8 rows x 16 bytes, 128 bytes apart along k, 256 along the rows.
__device__ __forceinline__ unsigned long long tc_desc_plain(unsigned addr) {
    return (unsigned long long)((addr & 0x3ffffu) >> 4) | ((unsigned long long)(128 >> 4) << 16) | ((unsigned long long)(256 >> 4) << 32) | (1ull << 46);
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
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
                     : "r"(addr));
}
// The same columns are stored; loads see them after tc_st_wait.
template <int W>
__device__ __forceinline__ void tc_st(unsigned addr, const float* v) {
    if constexpr (W == 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                     : "memory");
    else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
                     : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 16 or 24 columns.
template <int N>
__device__ __forceinline__ void tc_ldn(float* v, unsigned addr) {
#pragma unroll
    for (int c = 0; c + 16 <= N; c += 16) tc_ld<16>(v + c, addr + c);
    if constexpr (N % 16 == 8) tc_ld<8>(v + N - 8, addr + N - 8);
}
template <int N>
__device__ __forceinline__ void tc_stn(unsigned addr, const float* v) {
#pragma unroll
    for (int c = 0; c + 16 <= N; c += 16) tc_st<16>(addr + c, v + c);
    if constexpr (N % 16 == 8) tc_st<8>(addr + N - 8, v + N - 8);
}
// Waits for this warp's loads.  Uses of the values stay behind it if they are volatile assembly (fma_pair and the like); other uses
// take the second form, which costs moves.
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_ld_wait8(float* v) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7])::"memory");
}
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
// The same on pairs that stay in one 64-bit register: x * k + acc, x the two values of an accumulator.  Volatile: put off past the
// next load they would keep a third buffer of values alive.
__device__ __forceinline__ void fma_pair(unsigned long long& acc, const float* x, unsigned long long k) {
    asm volatile("{\n\t.reg .b64 x;\n\tmov.b64 x, {%1, %2};\n\tfma.rn.ftz.f32x2 %0, x, %3, %0;\n\t}" : "+l"(acc) : "f"(x[0]), "f"(x[1]), "l"(k));
}
__device__ __forceinline__ void fma_pair(unsigned long long& acc, const float* x, const float* y) {
    asm volatile("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%1, %2};\n\tmov.b64 y, {%3, %4};\n\tfma.rn.ftz.f32x2 %0, x, y, %0;\n\t}"
                 : "+l"(acc)
                 : "f"(x[0]), "f"(x[1]), "f"(y[0]), "f"(y[1]));
}
__device__ __forceinline__ void mul_pair(unsigned long long& acc, const float* x) {
    asm volatile("{\n\t.reg .b64 x;\n\tmov.b64 x, {%1, %2};\n\tmul.rn.ftz.f32x2 %0, x, %0;\n\t}" : "+l"(acc) : "f"(x[0]), "f"(x[1]));
}
__device__ __forceinline__ void add_pair(float* x, unsigned long long y) {
    asm volatile("{\n\t.reg .b64 x;\n\tmov.b64 x, {%0, %1};\n\tadd.rn.ftz.f32x2 x, x, %2;\n\tmov.b64 {%0, %1}, x;\n\t}" : "+f"(x[0]), "+f"(x[1]) : "l"(y));
}
__device__ __forceinline__ unsigned long long pair(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
// Bounded mbarrier wait of a pipeline: once one wait has run out, `dead` lets all others pass at once (the call is then
// reported as failed; what is computed meanwhile is not used).
__device__ __forceinline__ bool tc_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tc_wait_slow(unsigned bar, unsigned parity, volatile int* dead) {
    for (int i = 0; i < MBAR_POLL_LIMIT; i++) {
        if (tc_try(bar, parity)) return;
        if ((i & 63) == 63 && *dead) return;
    }
    *dead = 1;
}
// The first look stands before the loop: a wait that passes at once takes 67 cycles so, 142 as a pass through the loop.  Where
// it can, a role looks earlier (tc_try) and comes here with what it saw.
__device__ __forceinline__ void tc_wait(unsigned bar, unsigned parity, volatile int* dead, bool seen) {
    if (__builtin_expect(!seen, 0)) tc_wait_slow(bar, parity, dead);
}
// Roles that run ahead of the others leave the schedulers alone between looks.
__device__ __forceinline__ void tc_wait_idle(unsigned bar, unsigned parity, volatile int* dead) {
    if (__builtin_expect(tc_try(bar, parity), 1)) return;
    for (int i = 0; i < MBAR_POLL_LIMIT; i++) {
        __nanosleep(32);
        if (tc_try(bar, parity)) return;
        if ((i & 63) == 63 && *dead) return;
    }
    *dead = 1;
}
__device__ __forceinline__ void tc_wait(unsigned bar, unsigned parity, volatile int* dead) { tc_wait(bar, parity, dead, tc_try(bar, parity)); }

// ------------------------------------------------------------------ weights: registers -> operand tile

// 16 bytes to shared memory, by its own address: an aligned-up pointer would be a generic one.
__device__ __forceinline__ void sts16(unsigned addr, unsigned x, unsigned y, unsigned z, unsigned w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// A row of an operand tile: where its chunk 0 lies; chunk c is at this ^ (c << 4).
__device__ __forceinline__ unsigned tc_row_at(int row) { return (unsigned)(row * 128 + ((row & 7) << 4)); }

// Two f16 integers out of the bits `mask` of w: under the exponent that makes the f16 1024 + them.
__device__ __forceinline__ __half2 tc_bits_1024(unsigned w, unsigned mask) {
    const unsigned r = (w & mask) | 0x64006400u;
    return *reinterpret_cast<const __half2*>(&r);
}
// Out of bytes PAIR and PAIR + 2 of w.
template <int PAIR>
__device__ __forceinline__ __half2 tc_bytes_1024(unsigned w) {
    const unsigned r = __byte_perm(w, 0x64646464u, PAIR ? 0x4341 : 0x4240);
    return *reinterpret_cast<const __half2*>(&r);
}
__device__ __forceinline__ unsigned tc_bits(__half2 h) { return *reinterpret_cast<const unsigned*>(&h); }

// Raw words of half g of a 256-weight block (two stages of 64 weights) that a thread turns into operand values.
struct RawQ4 {
    static constexpr int PLANES = 1;
    unsigned dm, s0, s1, s2;  // header: d and dmin, scales
    unsigned nd, n0, n1, n2;  // of the next block's
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
            nd = (unsigned)hdr.x, n0 = (unsigned)hdr.y, n1 = (unsigned)hdr.z, n2 = (unsigned)hdr.w;
        }
    }
    __device__ __forceinline__ void begin_block() { dm = nd, s0 = n0, s1 = n1, s2 = n2; }
    // The eight mins of a block as tf32, 32 bytes; behind them d and -dmin, each the first of eight with zeros after it.
    __device__ __forceinline__ void store_mins(unsigned at) const {
        auto f = [](unsigned m, int i) { return __float_as_uint(i2f_small((int)((m >> (8 * i)) & 0xff))); };
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned m = h ? ((s2 >> 4) & 0x0f0f0f0fu) | (((s1 >> 6) & 0x03030303u) << 4) : s1 & 0x3f3f3f3fu;
            sts16(at ^ (h << 4), f(m, 0), f(m, 1), f(m, 2), f(m, 3));
            sts16(at ^ ((2 + 2 * h) << 4), __float_as_uint(h ? -f16_to_f32((unsigned short)(dm >> 16)) : f16_to_f32((unsigned short)dm)), 0, 0, 0);
            sts16(at ^ ((3 + 2 * h) << 4), 0, 0, 0, 0);
        }
    }
    // 64 weights of stage 2 g + i: low nibbles = sub-block 2 (2 g + i), high nibbles the next (kernels/common.cu:40-84)
    __device__ __forceinline__ void store(int i, unsigned at, int g, int) const {
        const unsigned sc4 = g == 0 ? s0 & 0x3f3f3f3fu : (s2 & 0x0f0f0f0fu) | (((s0 >> 6) & 0x03030303u) << 4);
        const __half2 bias = __half2half2(__ushort_as_half(0x6400)), m1024 = __half2half2(__ushort_as_half(0xe400));
        const unsigned sa = __byte_perm(sc4, 0x64646464u, i ? 0x4242 : 0x4040), sb = __byte_perm(sc4, 0x64646464u, i ? 0x4343 : 0x4141);
        const __half2 scl = __hsub2(*reinterpret_cast<const __half2*>(&sa), bias), sch = __hsub2(*reinterpret_cast<const __half2*>(&sb), bias);
        // (1024 + q) * sc - 1024 * sc, the high nibbles where they stand: (1024 + 16 q) * sc / 16 - 64 * sc.  Products below 2^16, sc / 16
        // and the difference q * sc exact
        const __half2 ofl = __hmul2(scl, m1024), sch16 = __hmul2(sch, __half2half2(__ushort_as_half(0x2c00))), ofh = __hmul2(sch16, m1024);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            unsigned lo[4], hi[4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const unsigned x = w[i][2 * c + k], y = x >> 8;
                lo[2 * k] = tc_bits(__hfma2(tc_bits_1024(x, 0x000f000fu), scl, ofl)), lo[2 * k + 1] = tc_bits(__hfma2(tc_bits_1024(y, 0x000f000fu), scl, ofl));
                hi[2 * k] = tc_bits(__hfma2(tc_bits_1024(x, 0x00f000f0u), sch16, ofh)), hi[2 * k + 1] = tc_bits(__hfma2(tc_bits_1024(y, 0x00f000f0u), sch16, ofh));
            }
            sts16(at ^ (c << 4), lo[0], lo[1], lo[2], lo[3]);
            sts16(at ^ ((4 + c) << 4), hi[0], hi[1], hi[2], hi[3]);
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
    __device__ __forceinline__ void store(int i, unsigned at, int, int plane_bytes) const {
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
                sts16(at ^ ((4 * jl + c) << 4), hi[0], hi[1], hi[2], hi[3]);
                sts16((at ^ ((4 * jl + c) << 4)) + plane_bytes, lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
};

// ------------------------------------------------------------------ the kernel

// The tokens are the rows of the product (128 lanes of TMEM per CTA), the weight rows its columns: a thread that drains an
// accumulator has one token, whose d8 it holds in a register, and the columns' d come once a block.  (The other way round every
// d8 was a broadcast read of shared memory: 770 of 2 000 cycles a stage.)
//
// A CTA stays on its SM and walks over items: 128 tokens x ROWS weight rows, in stages of 64 weights (and one for the mins of a
// block).  Lane 0 of warps 1 and 3 requests the tokens' operand as bulk copies, eight unpacking warps, a thread for each half of a
// row's blocks, turn weights into the other operand (two threads on every stage paid the ring's price twice as often), one thread of
// warps 0 and 2 issues the MMAs, sixteen warps drain the accumulators (two buffers in TMEM, each with the two groups of a stage side
// by side) into the block's sums in registers and those into the row's sums in TMEM (lanes 32 (w & 3) .., a quarter of the columns).
// Every role runs ahead of the next as far as the rings allow, over the end of an item too.
//
// A block's end needs d and dmin of every column in every lane.  They come as a product of their own: a column of ones times d is d,
// exactly, in every lane of an accumulator, and TMEM is read four times as fast as shared memory broadcasts.
//
// Gate / up pairs (ZIP) alternate the two matrices' rows in the tile, so that a thread holds a gate value beside its up value,
// as the two rows of a RoPE pair.  Where the items are too few to fill the chip, the k range is cut over the CTAs of a cluster
// (grid.y): the parts' sums meet through distributed shared memory, each CTA finishing its share of the tokens.
constexpr int TC_C_WARPS = 4, TC_A_WARPS = 8, TC_D_WARPS = 16, TC_MAX_STAGES = 12, TC_LANES = 128;
constexpr int TC_THREADS = 32 * (TC_C_WARPS + TC_A_WARPS + TC_D_WARPS), TC_LAUNCH_REGS = 72;
constexpr size_t TC_SMEM_MAX = 227 * 1024 - 512;  // less what the kernel declares itself
// Registers of a thread of each role; what they add up to is what the launch has.
constexpr int TC_REGS_C = 24, TC_REGS_A = 64, TC_REGS_D = 88;
static_assert(32 * (TC_C_WARPS * TC_REGS_C + TC_A_WARPS * TC_REGS_A + TC_D_WARPS * TC_REGS_D) <= TC_THREADS * TC_LAUNCH_REGS &&
                  TC_THREADS * TC_LAUNCH_REGS <= 65536,
              "more registers than the launch has");
// Registers of a role: N of the LAUNCH a thread has.  Fewer must be given back, more asked for.
template <int N>
__device__ __forceinline__ void tc_regs() {
    static_assert(N % 8 == 0, "");
    if constexpr (N < TC_LAUNCH_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
    else if constexpr (N > TC_LAUNCH_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// Most blocks a thread adds up one after the other.  The rounding of such a chain grows with the root of its length: Q6_K rows of 43
// and 108 blocks in one piece 1.30e-7 and 1.94e-7 against float64, in pieces of 22 and 27 1.04e-7 and 1.16e-7 (dp4a, which adds
// them as a tree, 0.93e-7 and 0.98e-7).
constexpr int TC_CHAIN = 27;

struct TcArgs {
    const unsigned char* image;
    int M, Mp;       // tokens, with padding
    Mat A1, A2;      // ZIP: the pair; otherwise A2 (optional) follows A1 in the grid
    int tiles1;      // row tiles of A1
    int items;       // row tiles x token tiles
    int groups;      // token tiles; an item's token tile is its index modulo this
    int id1, id2, zip;
    float2* park;    // sums of finished pieces of a chain (tc_park_bytes)
    ChunkEpi epi;
    TokenState* st;
};

constexpr int TC_ACCS = 4;  // accumulators in TMEM, two for a stage's groups, twice; behind them the sums of the rows

// Position in a ring of n slots: slot, and the parity of the lap.
struct TcRing {
    int slot = 0;
    unsigned lap = 0;
    __device__ __forceinline__ void next(int n) {
        if (++slot == n) slot = 0, lap ^= 1;
    }
};

// What a CTA works on.
template <int ROWS>
struct TcItem {
    int n0, nt, row0, N, id_base;
    bool second;
    const Mat* A;
    __device__ __forceinline__ TcItem(const TcArgs& a, int item) {
        const int tile = item / a.groups;
        n0 = (item - tile * a.groups) * TC_LANES, nt = min(TC_LANES, a.Mp - n0);
        second = !a.zip && a.A2.data != nullptr && tile >= a.tiles1;
        A = second ? &a.A2 : &a.A1;
        row0 = (tile - (second ? a.tiles1 : 0)) * (a.zip ? ROWS / 2 : ROWS);
        N = A->N, id_base = second ? a.id2 : a.id1;
    }
    // matrix and row of the tile's row r; rows past the matrix repeat its last row
    __device__ __forceinline__ const uint8_t* row(const TcArgs& a, int r, int& f) const {
        f = (int)mat_flat(A->nb, min(row0 + (a.zip ? r >> 1 : r), N - 1), 0);
        return (a.zip && (r & 1)) ? a.A2.data : A->data;
    }
};

template <bool Q4, int ROWS>
struct TcGeom {
    static constexpr int NC = ROWS / (TC_D_WARPS / 4);  // columns of a draining warp
    static constexpr int CH = 8;  // columns of a step at a block's end
    static constexpr int T_BYTES = TC_LANES * 128, W_PLANE = ROWS * 128, STAGE = T_BYTES + (Q4 ? 1 : 2) * W_PLANE;
    static constexpr int SUM_STRIDE = ROWS / 2 + 1;         // float2 of a token's sums when k parts meet; odd, so that 16 tokens' pairs lie in 32 banks
    static constexpr int OUT_PAIRS = 4;               // pairs of columns a warp turns from tokens to columns at a time
    static constexpr int WARP_BYTES = 32 * (OUT_PAIRS + 1) * 8 + (Q4 ? 0 : NC * 4);  // a draining warp's own: that, and on Q6_K its columns' d
    static constexpr int ONES_BYTES = Q4 ? TC_LANES * 32 : 0;  // a tf32 operand whose first column is ones, the others zero
    static constexpr int NST_MAX = (int)((TC_SMEM_MAX - 1024 - TC_D_WARPS * WARP_BYTES - ONES_BYTES) / STAGE);
    static constexpr int NST = NST_MAX < TC_MAX_STAGES ? NST_MAX : TC_MAX_STAGES;
    static constexpr size_t SMEM = (size_t)NST * STAGE + TC_D_WARPS * WARP_BYTES + ONES_BYTES + 1024;
    static_assert(ROWS % 32 == 0 && NC <= 32 && NC % CH == 0 && NC / 2 % OUT_PAIRS == 0, "whole warps of rows, a lane for every column, whole steps");
    static_assert(WARP_BYTES % 16 == 0 && (TC_ACCS + 1) * ROWS <= 512 && TC_LANES * SUM_STRIDE * 8 <= NST * STAGE, "");
};
constexpr size_t TC_PARK_BYTES = TC_LANES * 96 * 4;
// Most CTAs of a launch that cut chains: one an SM where the k range is in one part, three where parts of it are cut once more.
__host__ __device__ inline int tc_park_ctas(int parts, int sms) { return (parts > 1 ? 3 : 1) * sms; }
// Scratch for matrices of up to nb blocks a row, the sums of those CTAs (7.3 MB on 148 SMs for rows of 7 168 to 13 824 inputs, 21.8 MB
// for longer ones): rows short of two chains are whole ones or cut once, by the parts.
__host__ __device__ inline size_t tc_park_bytes(int nb, int sms) {
    return nb > 2 * TC_CHAIN ? tc_park_ctas(2, sms) * TC_PARK_BYTES : nb > TC_CHAIN ? tc_park_ctas(1, sms) * TC_PARK_BYTES : 0;
}

template <class RAW, int ROWS>
__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_tc(const __grid_constant__ TcArgs a) {
    constexpr bool Q4 = RAW::PLANES == 1;
    using G = TcGeom<Q4, ROWS>;
    constexpr int NC = G::NC, CH = G::CH;
    constexpr int SPB = Q4 ? 5 : 4;  // stages of a block: four of weights, one of mins
    constexpr int T_BYTES = G::T_BYTES, W_PLANE = G::W_PLANE, STAGE = G::STAGE, nst = G::NST;
    extern __shared__ __align__(128) unsigned char tc_smem_raw[];
    __shared__ unsigned long long bars[2 * TC_MAX_STAGES + 8];
    __shared__ unsigned tmem_slot;
    __shared__ int dead_s;
    volatile int* dead = &dead_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned full = smem_u32(bars), empty = full + 8 * TC_MAX_STAGES, accfull = empty + 8 * TC_MAX_STAGES, accempty = accfull + 32;
    const int S = gridDim.y, part = blockIdx.y;  // k parts
    const int nb = a.A1.nb, K = a.A1.K;
    const int b0 = nb * part / S, b1 = nb * (part + 1) / S;
    unsigned char* smem = tc_smem_raw + (-smem_u32(tc_smem_raw) & 1023u);
    if (tid == 0) {
        for (int i = 0; i < nst; i++) {
            mbar_init(bars + i, ROWS / 32 + 1);  // the warps that unpack a half and the tokens (with the bytes)
            mbar_init(bars + TC_MAX_STAGES + i, 2);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(bars + 2 * TC_MAX_STAGES + i, 1);
            mbar_init(bars + 2 * TC_MAX_STAGES + 4 + i, TC_D_WARPS);
        }
        dead_s = 0;
        mbar_fence_init();
    }
    if (Q4 && tid < 2 * TC_LANES) {
        // cores of even index hold the first half of eight rows
        const float4 z = make_float4(tid & 8 ? 0.f : 1.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(smem + (size_t)nst * STAGE + TC_D_WARPS * G::WARP_BYTES + tid * 16) = z;
    }
    fence_proxy_async();
    if (warp == 0) tc_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_slot;

    if (warp < TC_C_WARPS) {
        tc_regs<TC_REGS_C>();
        const int stages = SPB * (b1 - b0);
        if ((warp & 1) == 0) {
            // Two issuing warps take turns by stage, each with two accumulators of its own: a hand-over costs a warp some 200 cycles of
            // waiting and branching.  A block's mins are one stage to both: d and -dmin, and the mins' product.
            if (tc_elect()) {
                const int w = warp >> 1;
                TcRing ring;
                if (w) ring.next(nst);
                const unsigned base = smem_u32(smem) >> 4, dhi = (unsigned)(tc_desc(0) >> 32);
                const unsigned id = tc_idesc(0, TC_LANES, ROWS), idm = tc_idesc(2, TC_LANES, ROWS);
                auto desc = [&](unsigned at) { return ((unsigned long long)dhi << 32) | (at | (1u << 16)); };
                const unsigned acc0 = tmem + 2 * w * ROWS, af = accfull + 8 * w, ae = accempty + 8 * w;
                unsigned par = 1;     // of the accumulators' last reading; the first lap waits for none
                const int items = (a.items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
                // a stage's two accumulators: free, filled by mmas, handed on
                auto stage = [&](int step, int commits, auto&& mmas) {
                    const bool there = tc_try(full + 8 * ring.slot, ring.lap), free_ = tc_try(ae, par);
                    tc_wait(full + 8 * ring.slot, ring.lap, dead, there);
                    // what the unpacking warps stored becomes visible to the tensor core here, not where they store it: a
                    // fence there waits for the warp's loads in flight, the next block's words (900 to 2 200 cycles a block)
                    fence_proxy_async();
                    tc_wait(ae, par, dead, free_);
                    tc_fence_after();
#pragma unroll
                    for (int g = 0; g < 2; g++) mmas(g);
                    tc_commit(af);
                    par ^= 1;
                    for (int i = 0; i < commits; i++) tc_commit(empty + 8 * ring.slot);  // two a stage
                    for (int i = 0; i < step; i++) ring.next(nst);
                };
                for (int j = items * (b1 - b0), b = b0; j > 0; j--) {
#pragma unroll
                    for (int s = 0; s < 2; s++) {
                        const unsigned dt = base + ((ring.slot * STAGE) >> 4), dw = dt + (T_BYTES >> 4);
                        stage(Q4 && s == 1 && w ? 1 : 2, 2, [&](int g) {
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                const int kk = 2 * g + q;
                                tc_mma<false>(acc0 + g * ROWS, desc(dt + 2 * kk), desc(dw + 2 * kk), id, q);
                                if (!Q4) tc_mma<false>(acc0 + g * ROWS, desc(dt + 2 * kk), desc(dw + (W_PLANE >> 4) + 2 * kk), id, 1);
                            }
                        });
                    }
                    if constexpr (Q4) {
                        const unsigned dt = base + ((ring.slot * STAGE) >> 4) + 4 * (b & 1), dw = base + ((ring.slot * STAGE) >> 4) + (T_BYTES >> 4);
                        // d and -dmin of the columns in every lane; the mins' product with the high and with the low terms of the group sums
                        stage(w ? 2 : 1, 1, [&](int g) {
                            if (w) tc_mma<true>(acc0 + g * ROWS, desc(dt + 2 * g), desc(dw), idm, 0);
                            else tc_mma<true>(acc0 + g * ROWS, tc_desc_plain(smem_u32(smem) + nst * STAGE + TC_D_WARPS * G::WARP_BYTES), desc(dw + 2 + 2 * g), idm, 0);
                        });
                        if (++b == b1) b = b0;
                    }
                }
            }
            __syncwarp();
        } else {
            // two threads take turns: a bulk request costs the one that makes it 300 to 560 cycles
            griddep_wait();  // the image comes from the previous kernel
            if (lane == 0) {
                TcRing ring;
                const size_t plane = (size_t)a.Mp * 128;
                if (warp >> 1) ring.next(nst);
                int j = warp >> 1, lap = 0;
                for (int item = blockIdx.x; item < a.items; item += gridDim.x) {
                    const int n0 = (item % a.groups) * TC_LANES, nt = min(TC_LANES, a.Mp - n0);
                    const unsigned char* src = a.image + (size_t)n0 * 128;
                    for (; j < stages; j += 2) {
                        const int b = b0 + j / SPB, s = j % SPB;
                        if (lap) tc_wait_idle(empty + 8 * ring.slot, ring.lap ^ 1, dead);
                        if (*dead) break;
                        unsigned long long* bar = bars + ring.slot;
                        mbar_expect_tx(bar, nt * 128);
                        bulk_load(smem + ring.slot * STAGE, src + (s == 4 ? tc_sums_at(K, a.Mp) + (b >> 1) * plane : (4 * b + s) * plane), nt * 128, bar);
                        ring.next(nst);
                        ring.next(nst);
                        if (ring.lap) lap = 1;
                    }
                    j -= stages;
                }
            }
            __syncwarp();
        }
        if (*dead)  // after a wait that ran out: copies and MMAs in flight have this long to land before shared memory goes
            for (int i = 0; i < 100; i++) __nanosleep(1000);
        griddep_launch_dependents();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * (TC_D_WARPS + TC_C_WARPS)) : "memory");  // the last accumulator has been read
        tc_fence_after();
        if (warp == 0) tc_dealloc(tmem, 512);
        if (S > 1) cluster_sync_all();
        if (S > 1) cluster_sync_all();
        return;
    }

    if (warp < TC_C_WARPS + TC_A_WARPS) {
        tc_regs<TC_REGS_A>();
        const int ta = tid - 32 * TC_C_WARPS, g = ta >> 7, row_l = ta & 127;  // half of the blocks; row of the tile
        griddep_launch_dependents();
        if (row_l < ROWS) {
            const unsigned tile = smem_u32(smem) + T_BYTES + tc_row_at(row_l);  // the row in slot 0
            int slot = 0;  // of the block's first stage
            unsigned lap = 0;
            bool again = false;  // the ring has been round
            for (int item = blockIdx.x; item < a.items; item += gridDim.x) {
                const TcItem<ROWS> it(a, item);
                int f0;
                const uint8_t* wdata = it.row(a, row_l, f0);
                RAW raw;
                raw.load_stage(0, wdata, f0 + ROW_GROUP * b0, g);  // weights do not depend on earlier kernels
                raw.load_stage(1, wdata, f0 + ROW_GROUP * b0, g);
                // the rows of the CTA's next item start towards L2: the registers hold one block ahead, which covers an L2 hit but
                // not a trip to memory
                const int next = item + gridDim.x;
                if (next < a.items && next % a.groups == 0 && g == 0 && (row_l & 3) == 0) {
                    const TcItem<ROWS> in(a, next);
                    // one request a row group of each matrix
                    const int q = row_l >> 2, rows = a.zip ? ROWS / 2 : ROWS, rg = (a.zip ? q >> 1 : q) * ROW_GROUP;
                    if (rg < rows && in.row0 + rg < in.N) {
                        constexpr size_t TB = Q4 ? Q4_TILE_BYTES : Q6_TILE_BYTES;
                        const size_t f = mat_flat(nb, in.row0 + rg, 0), t0 = (f + ROW_GROUP * b0) >> 5, t1 = (f + ROW_GROUP * b1 + 31) >> 5;
                        bulk_prefetch_l2((a.zip && (q & 1) ? a.A2.data : in.A->data) + t0 * TB, (unsigned)((t1 - t0) * TB));
                    }
                }
                // stage s of the block: its slot free, filled by `fill`, handed on
                auto stage = [&](int s, auto&& fill) {
                    const bool wrap = slot + s >= nst;
                    const int at = slot + s - (wrap ? nst : 0);
                    if (again || wrap) tc_wait_idle(empty + 8 * at, (lap ^ (wrap ? 1u : 0u)) ^ 1u, dead);
                    fill(tile + at * STAGE);
                    __syncwarp();
                    if (lane == 0) tc_arrive(full + 8 * at);
                };
                for (int b = b0; b < b1; b++) {
                    raw.begin_block();
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        stage(2 * g + i, [&](unsigned t) { raw.store(i, t, g, W_PLANE); });
                        if (b + 1 < b1) raw.load_stage(i, wdata, f0 + ROW_GROUP * (b + 1), g);  // the words just used, of the next block
                    }
                    if constexpr (Q4)
                        if (g == (b & 1)) stage(4, [&](unsigned t) { raw.store_mins(t); });
                    slot += SPB;
                    if (slot >= nst) slot -= nst, lap ^= 1, again = true;
                }
            }
        }
        if (S > 1) cluster_sync_all();
        if (S > 1) cluster_sync_all();
        return;
    }

    tc_regs<TC_REGS_D>();
    const int dwarp = warp - TC_C_WARPS - TC_A_WARPS, td = tid - 32 * (TC_C_WARPS + TC_A_WARPS), quad = warp & 3, cg = dwarp >> 2, tok = quad * 32 + lane;
    unsigned char* own = smem + (size_t)nst * STAGE + dwarp * G::WARP_BYTES;
    float2* turn = reinterpret_cast<float2*>(own);
    float* colscale = reinterpret_cast<float*>(own + 32 * (G::OUT_PAIRS + 1) * 8);  // Q6_K: d of the warp's columns
    const unsigned lanes = tmem + ((unsigned)quad << 21) + cg * NC;
    const unsigned lanes_tot = lanes + TC_ACCS * ROWS;  // the row's sums of the token and its columns
    griddep_launch_dependents();
    griddep_wait();  // nothing reaches an accumulator before the image is complete; residuals are then, too
    const int pieces = (b1 - b0 + TC_CHAIN - 1) / TC_CHAIN;
    unsigned par = 0;  // of the buffers' first uses in a block; Q4_K uses them three times
    for (int item = blockIdx.x; item < a.items; item += gridDim.x) {
        // Q6_K: the lanes hold the columns' d, a block ahead
        int df;
        const uint8_t* dp;
        unsigned d8_at;
        {
            const TcItem<ROWS> it(a, item);
            d8_at = (unsigned)(4 * b0) * a.Mp + min(it.n0 + tok, a.Mp - 1);
            dp = it.row(a, cg * NC + min(lane, NC - 1), df);
        }
        float dnext;
        auto load_d = [&](int b) {
            const int f = df + ROW_GROUP * b;
            dnext = f16_to_f32(__ldg(reinterpret_cast<const unsigned short*>(dp + (size_t)(f >> 5) * Q6_TILE_BYTES + Q6_PIECES * 512 + (f & 31) * 2)));
        };
        if (!Q4) load_d(b0);
        // d8 of the token's groups, two stages ahead
        int d8_left = 4 * (b1 - b0);
        auto load_d8 = [&] {  // L1 may hold the last image
            const float2 k = __ldcg(reinterpret_cast<const float2*>(a.image + tc_d8_at(K, a.Mp)) + d8_at);
            if (--d8_left > 0) d8_at += a.Mp;
            return k;
        };
        float2 knext[2];
        knext[0] = load_d8(), knext[1] = load_d8();
        int piece = 1, cut = b0 + (b1 - b0) / pieces;
        auto clear = [&] {
            float z[NC];
#pragma unroll
            for (int i = 0; i < NC; i++) z[i] = 0.f;
            tc_stn<NC>(lanes_tot, z);
            tc_st_wait();
        };
        clear();
        for (int b = b0; b < b1; b++) {
            if (!Q4) {
                if (lane < NC) colscale[lane] = dnext;
                if (b + 1 < b1) load_d(b + 1);
            }
            // use k of the block of buffer `buf`
            auto wait_full = [&](int buf, int k) {
                tc_wait(accfull + 8 * buf, par ^ (k & 1), dead);
                tc_fence_after();
            };
            auto release = [&](int buf) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) tc_arrive(accempty + 8 * buf);
            };
            unsigned long long sum[NC / 2];  // of the block without its d
#pragma unroll
            for (int i = 0; i < NC / 2; i++) sum[i] = 0;
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const int buf = s & 1;
                const float2 k = knext[buf];
                knext[buf] = load_d8();
                float v[2][NC];
                wait_full(buf, s >> 1);
                tc_ldn<NC>(v[0], lanes + 2 * buf * ROWS);
                tc_ld_wait();
                tc_ldn<NC>(v[1], lanes + (2 * buf + 1) * ROWS);
                {
                    const unsigned long long kk = pair(k.x, k.x);
#pragma unroll
                    for (int i = 0; i < NC / 2; i++) fma_pair(sum[i], v[0] + 2 * i, kk);
                }
                tc_ld_wait();
                release(buf);
                {
                    const unsigned long long kk = pair(k.y, k.y);
#pragma unroll
                    for (int i = 0; i < NC / 2; i++) fma_pair(sum[i], v[1] + 2 * i, kk);
                }
            }
            // the block's d * sums - dmin * mins, and once more rounded into the row's sum
            tc_st_wait();  // of the block before
            if constexpr (Q4) {
                float w[4][CH];
                wait_full(0, 2);
#pragma unroll
                for (int c = 0; c < NC / CH; c++) {
                    tc_ld<CH>(w[0], lanes + c * CH);
                    tc_ld<CH>(w[1], lanes + ROWS + c * CH);
                    tc_ld<CH>(w[3], lanes_tot + c * CH);
                    if (c == 0) wait_full(1, 2);
                    tc_ld<CH>(w[2], lanes + 2 * ROWS + c * CH);
                    tc_ld_wait();
#pragma unroll
                    for (int i = 0; i < CH / 2; i++) {
                        mul_pair(sum[c * (CH / 2) + i], w[0] + 2 * i);
                        fma_pair(sum[c * (CH / 2) + i], w[1] + 2 * i, w[2] + 2 * i);
                    }
                    tc_ld<CH>(w[2], lanes + 3 * ROWS + c * CH);
                    tc_ld_wait();
                    if (c == NC / CH - 1) {
                        release(0);
                        release(1);
                    }
#pragma unroll
                    for (int i = 0; i < CH / 2; i++) {
                        fma_pair(sum[c * (CH / 2) + i], w[1] + 2 * i, w[2] + 2 * i);
                        add_pair(w[3] + 2 * i, sum[c * (CH / 2) + i]);
                    }
                    tc_st<CH>(lanes_tot + c * CH, w[3]);
                }
                par ^= 1;
            } else {
                __syncwarp();
                float v[NC];
                tc_ldn<NC>(v, lanes_tot);
                tc_ld_wait();
#pragma unroll
                for (int q = 0; q < NC / 4; q++) {
                    const float4 d = reinterpret_cast<const float4*>(colscale)[q];
                    mul_pair(sum[2 * q], &d.x), mul_pair(sum[2 * q + 1], &d.z);
                    add_pair(v + 4 * q, sum[2 * q]), add_pair(v + 4 * q + 2, sum[2 * q + 1]);
                }
                __syncwarp();  // the columns' scales have been read
                tc_stn<NC>(lanes_tot, v);
            }
            if (pieces > 1 && b + 1 == cut) {
                tc_st_wait();
                // a piece of the chain is done: its sums wait in memory (a thread's own 8 bytes beside its neighbours')
                const bool last = piece == pieces;
                float2* park = a.park + (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * (TC_PARK_BYTES / 8) + td;
                float v[NC];
                tc_ldn<NC>(v, lanes_tot);
                tc_ld_wait();
#pragma unroll
                for (int i = 0; i < NC / 2; i++) {
                    float2* p = park + i * (32 * TC_D_WARPS);
                    if (piece > 1) {
                        const float2 t = *p;
                        add_pair(v + 2 * i, pair(t.x, t.y));
                    }
                    if (!last) {
                        asm volatile("" : "+f"(v[2 * i]), "+f"(v[2 * i + 1]));
                        *p = make_float2(v[2 * i], v[2 * i + 1]);
                    }
                }
                if (last) {
                    tc_stn<NC>(lanes_tot, v);
                    tc_st_wait();
                } else {
                    clear();
                }
                piece++;
                cut = b0 + (b1 - b0) * piece / pieces;
            }
        }

        int again = item;  // looked up once more: it would cost registers in the loop
        asm volatile("" : "+r"(again));
        const TcItem<ROWS> it(a, again);
        const int m = it.n0 + tok;
        float2 tot[NC / 2];
        tc_st_wait();
#pragma unroll
        for (int c = 0; c < NC / 8; c++) {
            float v[8];
            tc_ld<8>(v, lanes_tot + 8 * c);
            tc_ld_wait8(v);
#pragma unroll
            for (int i = 0; i < 4; i++) tot[4 * c + i] = make_float2(v[2 * i], v[2 * i + 1]);
        }

        // ---- epilogue.  A gate/up tile whose rows all exist leaves straight from the registers (gate and up of 2 048 tokens 4 % faster
        // than the other way).  All else is turned first, so that lanes run along the columns: RoPE pairs, rows with residuals.  A thread's
        // own token and columns would touch 32 rows of the output with every access (a down projection of 2 048 tokens: 620 us).
        if (S > 1) {
            float2* mine = reinterpret_cast<float2*>(smem) + tok * G::SUM_STRIDE + cg * (NC / 2);
#pragma unroll
            for (int i = 0; i < NC / 2; i++) mine[i] = tot[i];
            break;  // one item a cluster
        }
        if (a.epi.kind == CEPI_SILU && it.row0 + ROWS / 2 <= it.N && ((a.epi.ldo | (it.id_base + it.row0)) & 3) == 0 &&
            (reinterpret_cast<uintptr_t>(a.epi.out) & 15) == 0) {
            if (m < a.M) {
                float4* o = reinterpret_cast<float4*>(a.epi.out + (size_t)m * a.epi.ldo + it.id_base + it.row0 + cg * (NC / 2));
#pragma unroll
                for (int i = 0; i < NC / 2; i += 4) {
                    float h[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) h[q] = (tot[i + q].x / (1.f + __expf(-tot[i + q].x))) * tot[i + q].y;  // as ChunkEpiTok::apply
                    o[i / 4] = make_float4(h[0], h[1], h[2], h[3]);
                }
            }
            continue;
        }
        constexpr int OP = G::OUT_PAIRS;
        const bool res = a.epi.kind == CEPI_STORE && a.epi.use_res == 2;
        ChunkEpi epi = a.epi;
        epi.use_res = 0;
#pragma unroll
        for (int c = 0; c < NC / 2; c += OP) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < OP; i++)
                turn[lane * (OP + 1) + i] = tot[c + i];
            __syncwarp();
            const int pl = lane & (OP - 1), pair = cg * (NC / 2) + c + pl;
            const int row = it.row0 + (a.zip ? pair : 2 * pair);
            const bool on = row < it.N;
            const int id = it.id_base + (a.zip ? row : row >> 1);
            float2 r[OP];
#pragma unroll
            for (int q = 0; q < OP; q++) {
                const int mt = it.n0 + quad * 32 + q * (32 / OP) + lane / OP;
                r[q] = make_float2(0.f, 0.f);
                if (res && on && mt < a.M) {
                    const float* o = epi.out + (size_t)mt * epi.ldo + 2 * id;
                    r[q].x = o[0];
                    if (2 * id + 1 < epi.n_rows) r[q].y = o[1];
                }
            }
#pragma unroll
            for (int q = 0; q < OP; q++) {
                const int t = q * (32 / OP) + lane / OP, mt = it.n0 + quad * 32 + t;
                const float2 x = turn[t * (OP + 1) + pl];
                if (on && mt < a.M) ChunkEpiTok{&epi, mt}.apply(id, x.x + r[q].x, x.y + r[q].y);
            }
        }
    }
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(32 * (TC_D_WARPS + TC_C_WARPS)) : "memory");
    if (td == 0 && dead_s && a.st) a.st->err = 2;
    if (S == 1) return;
    cluster_sync_all();
    {
        const TcItem<ROWS> it(a, blockIdx.x);
        constexpr int PAIRS = ROWS / 2, BATCH = 4;
        const int t0 = TC_LANES * part / S, items = min(TC_LANES / S, a.M - it.n0 - t0) * PAIRS;  // S is a power of two
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
                const int row = it.row0 + (a.zip ? pair : 2 * pair);
                const bool on = k < items && row < it.N;
                m[q] = it.n0 + t, id[q] = on ? it.id_base + (a.zip ? row : row >> 1) : -1;
                v[q] = r[q] = make_float2(0.f, 0.f);
                if (!on) continue;
                if (res) {
                    const float* o = epi.out + (size_t)m[q] * epi.ldo + 2 * id[q];
                    r[q].x = o[0];
                    if (2 * id[q] + 1 < epi.n_rows) r[q].y = o[1];
                }
                const unsigned at = smem_u32(smem) + (t * G::SUM_STRIDE + pair) * 8;
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
    }
    cluster_sync_all();  // nobody leaves while others read its sums
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

template <class RAW, int ROWS>
inline cudaError_t launch_tc(cudaStream_t stream, int sms, TcArgs& a, int S) {
    constexpr bool Q4 = RAW::PLANES == 1;
    using G = TcGeom<Q4, ROWS>;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(S > 1 ? a.items : std::min(a.items, sms), S);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = G::SMEM;
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
    return cudaLaunchKernelEx(&cfg, k_gemm_tc<RAW, ROWS>, (const TcArgs)a);
}

// out = epilogue(W x) for the M tokens of an operand image; jb: the second matrix of a gate/up pair or one that follows.
// park: tc_park_bytes.
inline cudaError_t launch_gemm_tc(cudaStream_t stream, int sms, const unsigned char* image, float2* park, int M, const RowJob& ja,
                                  const RowJob& jb, const ChunkEpi& epi, TokenState* st) {
    TcArgs a{};
    a.image = image, a.M = M, a.Mp = tc_pad_tokens(M);
    a.A1 = ja.m, a.A2 = jb.m, a.id1 = ja.id_base, a.id2 = jb.id_base;
    a.zip = epi.kind == CEPI_SILU;
    a.epi = epi, a.st = st, a.park = park;
    a.groups = (M + TC_LANES - 1) / TC_LANES;
    // Tile and number of k parts with the shortest longest chain: waves of CTAs x (blocks x what a block takes + the ends), in units of
    // 3.2 us.  Measured on Q6_K rows: 96 rows 2.4 us a block, 64 rows 1.95; ends 3 us, cut k ranges 3 more.  Q4_K has other stages and takes
    // what Q6_K takes (2 048 rows of 11 008 inputs, 500 and 2 048 tokens: 99.7 and 295 us, Q6_K 104 and 298).  All eight choices timed on
    // 14 matrices and pairs of both types, 2 048 to 27 648 inputs, at 66 to 2 048 tokens: the one taken is the fastest or within 7 % of it,
    // in 109 of 112 within 4 % (2 048 rows of 11 008 at 1 000 tokens 191 us in tiles of 64 rows, 179 in 96 and two parts).
    int S = 1, rows = 96;
    double best = 1e30;
    auto tiles = [&](int r, int& first) {
        const int per = a.zip ? r / 2 : r;
        first = (ja.m.N + per - 1) / per;
        return first + (!a.zip && jb.m.data ? (jb.m.N + per - 1) / per : 0);
    };
    for (int r : {96, 64})
        for (int s = 1; s <= 8 && s <= ja.m.nb; s *= 2) {
            int first;
            const int ctas = tiles(r, first) * a.groups * s, at_once = cluster_ctas(k_gemm_tc<RawQ4, 96>, TC_THREADS, s, sms);
            const int blocks = (ja.m.nb + s - 1) / s;
            if (s > 1 && blocks > TC_CHAIN && ctas > tc_park_ctas(s, sms)) continue;  // parked sums have no room
            const double t = (double)((ctas + at_once - 1) / at_once) * ((r == 96 ? 0.75 : 0.62) * blocks + 1 + (s > 1 ? 1 : 0));
            if (t < best) best = t, S = s, rows = r;
        }
    a.items = tiles(rows, a.tiles1) * a.groups;
    if (rows == 96) return ja.m.type == TFR_Q4_K ? launch_tc<RawQ4, 96>(stream, sms, a, S) : launch_tc<RawQ6, 96>(stream, sms, a, S);
    return ja.m.type == TFR_Q4_K ? launch_tc<RawQ4, 64>(stream, sms, a, S) : launch_tc<RawQ6, 64>(stream, sms, a, S);
}

}  // namespace tfr
