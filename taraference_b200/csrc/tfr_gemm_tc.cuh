// Projections of token batches on the fifth-generation tensor cores (tcgen05), Q4_K and Q6_K weights.
//
// What has to be computed is the decode arithmetic (kernels/gemv.cu:71-130, 302-337): integer sub-block dots of the
// 4- or 6-bit weights with the int8 activations, scaled per sub-block by the weight's 6- or 8-bit scale and the
// activation group's fp32 scale, scaled per 256-weight block by the block's fp16 d, minus (Q4_K) dmin times the scaled
// group sums.  An integer MMA would have to leave its accumulator after every 32 (Q4_K) or 16 (Q6_K) weights to meet the
// activation's scale, which binds the kernel to that scale arithmetic on CUDA cores (9 % of the tensor pipe, 90 us for
// the 22 016 x 2 048 gate/up pair and 64 tokens).  Here the scales travel inside the f16 operands instead:
//
//   A = scale * quant      an integer.  Q4_K: at most 63 * 15, exact in f16.  Q6_K: at most 128 * 32, so an f16 term and
//                          a residual of at most one unit (a second operand tile);
//   B = d8 * q8 * 2^s      as two f16 terms (22 bits; s per token puts the token's largest value at 2^9 .. 2^10, far from
//                          both ends of f16);
//
// the accumulator (fp32, in TMEM) runs over 64 weights and is then joined to the row's sum by fma(d, accumulator, sum) in
// registers, round to nearest.  The tensor core truncates as it adds: accumulators over whole 256-weight blocks left sums
// four times less accurate than fp32 sums of the integer dots (1e-6 of the largest logit against 2.5e-7), over 64 weights
// with the small products first they are as accurate.  The min
// term of Q4_K, sum over groups of dmin * m * (d8 * sum q8), is a product of its own with 1 / 32 of the depth, run as
// tf32 (two terms each; no range to fit) ahead of the blocks.
#pragma once
#include "tfr_chunk.cuh"

namespace tfr {

// ------------------------------------------------------------------ operand image of the activations

// Both operands lie in shared memory as K-major rows of 128 bytes with the 128-byte swizzle: 16-byte chunk c of row r at
// r * 128 + ((c ^ (r & 7)) << 4), 8-row atoms of 1 KB.  The activations are written to global memory in exactly that
// image, so a stage of a CTA's token tile is one run of bytes per plane and travels as one untiled bulk copy:
//   [stage][plane: high term, low term][token / 8][1 KB atom]
// stages 0 .. K/64 - 1 hold 64 values of f16 each, the next ceil(K / 1024) hold 32 group sums of tf32 each.
constexpr int TC_STAGE_K = 64;
__host__ __device__ inline int tc_min_stages(int K) { return (K + 1023) / 1024; }
// Padding tokens make MMA widths: multiples of 16 columns, of 32 for the two-CTA MMAs of larger batches.
__host__ __device__ inline int tc_pad_tokens(int M) { return M > 128 ? (M + 31) & ~31 : (M + 15) & ~15; }
__host__ __device__ inline size_t tc_image_bytes(int K, int M) {
    return (size_t)(K / TC_STAGE_K + tc_min_stages(K)) * tc_pad_tokens(M) * 256;
}
__host__ __device__ inline size_t tc_plane(int stage, int plane, int Mp) { return ((size_t)stage * 2 + plane) * Mp * 128; }
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
    float* tscale;       // [Mp]: 2^-s of every token
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
    float amax = 0.f;
    for (int i4 = tid; i4 < (K >> 2); i4 += TC_PREP_THREADS) {
        float4 v = live ? reinterpret_cast<const float4*>(x)[i4] : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(xs + xs_idx(4 * i4)) = v;
        amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    if (a.normw) {
        __syncthreads();
        const float scale = rms_scale_staged(xs, K, a.eps, red);
        amax = 0.f;
        for (int i4 = tid; i4 < (K >> 2); i4 += TC_PREP_THREADS) {
            float4 v = *reinterpret_cast<const float4*>(xs + xs_idx(4 * i4));
            const float4 w = reinterpret_cast<const float4*>(a.normw)[i4];
            v.x = v.x * scale * w.x;
            v.y = v.y * scale * w.y;
            v.z = v.z * scale * w.z;
            v.w = v.w * scale * w.w;
            *reinterpret_cast<float4*>(xs + xs_idx(4 * i4)) = v;
            if (a.xn && live) reinterpret_cast<float4*>(a.xn + (size_t)m * K)[i4] = v;
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        }
    }
    __syncthreads();  // red is free, the staged vector is final
    amax = warp_max(amax);
    if (lane == 0) red[tid >> 5] = amax;
    __syncthreads();
    if (tid < 32) {
        const float v = warp_max(tid < TC_PREP_THREADS / 32 ? red[tid] : 0.f);
        if (tid == 0) red[32] = v;
    }
    __syncthreads();
    amax = red[32];
    // 2^s with amax * 2^s in [2^9, 2^10): exponents outside +-100 are left alone (all zero, or no finite vector)
    int e = 0;
    if (amax > 1e-30f && amax < 1e30f) e = 9 - ((int)((__float_as_uint(amax) >> 23) & 0xff) - 127);
    const float up = __uint_as_float((unsigned)(127 + e) << 23);
    if (tid == 0) a.tscale[m] = __uint_as_float((unsigned)(127 - e) << 23);
    unsigned char* tok = a.image + (size_t)(m >> 3) * 1024;
    for (int i0 = 0; i0 < n8; i0 += TC_PREP_THREADS) {
        const int i = i0 + tid;  // values 8 i .. 8 i + 7; four lanes share a 32-value group
        const bool on = i < n8;
        float v[8];
        const float4 v0 = on ? *reinterpret_cast<const float4*>(xs + xs_idx(8 * i)) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v1 = on ? *reinterpret_cast<const float4*>(xs + xs_idx(8 * i + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = v0.x, v[1] = v0.y, v[2] = v0.z, v[3] = v0.w, v[4] = v1.x, v[5] = v1.y, v[6] = v1.z, v[7] = v1.w;
        float g = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) g = fmaxf(g, fabsf(v[k]));
        g = fmaxf(g, __shfl_xor_sync(TFR_FULL_MASK, g, 1));
        g = fmaxf(g, __shfl_xor_sync(TFR_FULL_MASK, g, 2));
        const float d = g * (1.0f / 127.0f), du = d * up;
        int sum = 0;
        unsigned hi[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            int q0 = 0, q1 = 0;
            if (g != 0.f) {
                q0 = (int)(signed char)__float2int_rn(v[2 * k] / d);
                q1 = (int)(signed char)__float2int_rn(v[2 * k + 1] / d);
            }
            sum += q0 + q1;
            const float f0 = (float)q0, f1 = (float)q1;
            const __half h0 = __float2half_rn(du * f0), h1 = __float2half_rn(du * f1);
            hi[k] = pack_f16x2(h0, h1);
            lo[k] = pack_f16x2(__float2half_rn(fmaf(du, f0, -__half2float(h0))), __float2half_rn(fmaf(du, f1, -__half2float(h1))));
        }
        sum += __shfl_xor_sync(TFR_FULL_MASK, sum, 1);
        sum += __shfl_xor_sync(TFR_FULL_MASK, sum, 2);
        if (!on) continue;  // whole groups: n8 is a multiple of 32
        const unsigned at = tc_swz(row, i & 7);
        *reinterpret_cast<uint4*>(tok + tc_plane(i >> 3, 0, Mp) + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(tok + tc_plane(i >> 3, 1, Mp) + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if ((i & 3) == 0) {
            const int grp = i >> 2;
            const float s = d * (float)sum * up, sh = __uint_as_float(__float_as_uint(s) & 0xffffe000u);
            const size_t o = tc_plane(K / TC_STAGE_K + (grp >> 5), 0, Mp) + tc_swz(row, (grp & 31) >> 2) + (grp & 3) * 4;
            *reinterpret_cast<float*>(tok + o) = sh;
            *reinterpret_cast<float*>(tok + o + (size_t)Mp * 128) = s - sh;
        }
    }
    // groups past the end of the last stage of sums
    for (int grp = K / 32 + tid; grp < 32 * tc_min_stages(K); grp += TC_PREP_THREADS) {
        const size_t o = tc_plane(K / TC_STAGE_K + (grp >> 5), 0, Mp) + tc_swz(row, (grp & 31) >> 2) + (grp & 3) * 4;
        *reinterpret_cast<float*>(tok + o) = 0.f;
        *reinterpret_cast<float*>(tok + o + (size_t)Mp * 128) = 0.f;
    }
}

// ------------------------------------------------------------------ tcgen05 primitives (CG: CTAs an MMA runs on)

template <int CG>
__device__ __forceinline__ void tc_alloc(unsigned* slot, unsigned cols) {
    if (CG == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
}
template <int CG>
__device__ __forceinline__ void tc_dealloc(unsigned addr, unsigned cols) {
    if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Arrives at the barrier when the MMAs issued so far are done; in both CTAs of a pair whose leader has cluster rank `lead`.
template <int CG>
__device__ __forceinline__ void tc_commit(unsigned long long* bar, int lead) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                     "h"((unsigned short)(3 << lead))
                     : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrives at the barrier at the same place in CTA `rank` of the cluster.
__device__ __forceinline__ void tc_arrive_at(unsigned long long* bar, int rank) {
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(rank));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// Shared-memory descriptor of a K-major operand with the 128-byte swizzle: start address, (unused) leading offset, 1 KB
// between 8-row atoms, version 1, swizzle mode 2.
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr) {
    return (unsigned long long)((addr & 0x3ffffu) >> 4) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: fp32 accumulator, K-major operands of type `ty` (0: f16, 2: tf32), m x n.
__device__ __forceinline__ unsigned tc_idesc(unsigned ty, unsigned m, unsigned n) { return (1u << 4) | (ty << 7) | (ty << 10) | ((n >> 3) << 17) | ((m >> 4) << 24); }
template <bool TF32, int CG>
__device__ __forceinline__ void tc_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
#define TFR_TC_MMA(form)                                                                                                    \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma." form " [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), \
                 "l"(b), "r"(idesc), "r"(accumulate)                                                                         \
                 : "memory")
    if (CG == 2) {
        if (TF32) TFR_TC_MMA("cta_group::2.kind::tf32");
        else TFR_TC_MMA("cta_group::2.kind::f16");
    } else {
        if (TF32) TFR_TC_MMA("cta_group::1.kind::tf32");
        else TFR_TC_MMA("cta_group::1.kind::f16");
    }
#undef TFR_TC_MMA
}
// Columns addr .. addr + W - 1 of this warp's 32 lanes; the values are there after tc_ld_wait.
template <int W>
__device__ __forceinline__ void tc_ld(float (&v)[W], unsigned addr) {
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
// reported as failed; what is computed meanwhile is not used).  CLUSTER: arrivals may come from another CTA.
template <bool CLUSTER>
__device__ __forceinline__ void tc_wait(unsigned long long* bar, unsigned parity, volatile int* dead) {
    for (int i = 0; i < MBAR_POLL_LIMIT; i++) {
        unsigned ok;
        if (CLUSTER)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok)
                         : "r"(smem_u32(bar)), "r"(parity)
                         : "memory");
        else
            ok = mbar_try_wait(bar, parity);
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

// Raw words of one 256-weight block that a thread turns into operand values: two threads share a row's block, thread h
// takes the 16 bytes of every 64 weights that start at byte 16 h.
struct RawQ4 {
    static constexpr int WPS = 4, PLANES = 1;
    unsigned s0, s2;  // of the header's three scale words, the two that hold the sub-block scales
    unsigned w[4][WPS];
    // What stage s alone uses; the header with the last one.
    __device__ __forceinline__ void load_stage(int s, const uint8_t* data, int f, int h) {
        const uint8_t* p = data + (size_t)(f >> 5) * Q4_TILE_BYTES + (f & 31) * 16;
        const int4 v = ldg_stream(p + (1 + 2 * s + h) * 512);
        w[s][0] = v.x, w[s][1] = v.y, w[s][2] = v.z, w[s][3] = v.w;
        if (s == 3) {
            const int4 hdr = ldg_stream(p);
            s0 = (unsigned)hdr.y, s2 = (unsigned)hdr.w;
        }
    }
    __device__ __forceinline__ void load(const uint8_t* data, int f, int h) {
#pragma unroll
        for (int s = 0; s < 4; s++) load_stage(s, data, f, h);
    }
    // 64 weights of stage s: low nibbles = sub-block 2 s, high nibbles = sub-block 2 s + 1 (kernels/common.cu:40-84)
    __device__ __forceinline__ void store(int s, unsigned char* tile, int row, int h, int) const {
        const unsigned sc4 = s < 2 ? s0 & 0x3f3f3f3fu : (s2 & 0x0f0f0f0fu) | (((s0 >> 6) & 0x03030303u) << 4);
        const __half2 bias = __half2half2(__ushort_as_half(0x6400)), m1024 = __half2half2(__ushort_as_half(0xe400));
        const unsigned sa = __byte_perm(sc4, 0x64646464u, (s & 1) ? 0x4242 : 0x4040), sb = __byte_perm(sc4, 0x64646464u, (s & 1) ? 0x4343 : 0x4141);
        const __half2 scl = __hsub2(*reinterpret_cast<const __half2*>(&sa), bias), sch = __hsub2(*reinterpret_cast<const __half2*>(&sb), bias);
        const __half2 ofl = __hmul2(scl, m1024), ofh = __hmul2(sch, m1024);
#pragma unroll
        for (int c = 0; c < WPS / 2; c++) {
            unsigned lo[4], hi[4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const unsigned x = w[s][2 * c + k], l = x & 0x0f0f0f0fu, u = (x >> 4) & 0x0f0f0f0fu;
                // (1024 + q) * sc - 1024 * sc: both products below 2^16, the difference q * sc exact
                lo[2 * k] = tc_bits(__hfma2(tc_bytes_1024<0>(l), scl, ofl)), lo[2 * k + 1] = tc_bits(__hfma2(tc_bytes_1024<1>(l), scl, ofl));
                hi[2 * k] = tc_bits(__hfma2(tc_bytes_1024<0>(u), sch, ofh)), hi[2 * k + 1] = tc_bits(__hfma2(tc_bytes_1024<1>(u), sch, ofh));
            }
            const int chunk = (WPS / 2) * h + c;
            *reinterpret_cast<uint4*>(tile + tc_swz(row, chunk)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            *reinterpret_cast<uint4*>(tile + tc_swz(row, 4 + chunk)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
    }
};

struct RawQ6 {
    static constexpr int WPS = 4, PLANES = 2;
    int4 sc;
    unsigned la[2][WPS], lb[2][WPS], hq[2][WPS];
    // What the stages up to s are the last to use: half n = s >> 1 after its second stage.
    __device__ __forceinline__ void load_stage(int s, const uint8_t* data, int f, int h) {
        if (!(s & 1)) return;
        const uint8_t* p = data + (size_t)(f >> 5) * Q6_TILE_BYTES + (f & 31) * 16;
        const int n = s >> 1;
        const int4 a = ldg_stream(p + (4 * n + h) * 512), b = ldg_stream(p + (4 * n + 2 + h) * 512), c = ldg_stream(p + (8 + 2 * n + h) * 512);
        la[n][0] = a.x, la[n][1] = a.y, la[n][2] = a.z, la[n][3] = a.w;
        lb[n][0] = b.x, lb[n][1] = b.y, lb[n][2] = b.z, lb[n][3] = b.w;
        hq[n][0] = c.x, hq[n][1] = c.y, hq[n][2] = c.z, hq[n][3] = c.w;
        if (s == 3) sc = ldg_stream(p + 12 * 512);
    }
    __device__ __forceinline__ void load(const uint8_t* data, int f, int h) {
        load_stage(1, data, f, h);
        load_stage(3, data, f, h);
    }
    // 64 weights of stage s = runs j = 2 (s & 1), + 1 of half n = s >> 1 (kernels/gemv.cu:302-337, as in block_dot):
    // scale * (q - 32) as its f16 rounding and the residual (0 or +-1: |scale * q| <= 4096)
    __device__ __forceinline__ void store(int s, unsigned char* tile, int row, int h, int plane_bytes) const {
        const int n = s >> 1;
        const __half2 off = __half2half2(__ushort_as_half(0x6420));  // 1024 + 32
#pragma unroll
        for (int jl = 0; jl < 2; jl++) {
            const int j = 2 * (s & 1) + jl;
            // scale byte 8 n + h + 2 j: word 2 n + (j >> 1), byte h + 2 (j & 1)
            const int word = n == 0 ? ((s & 1) ? sc.y : sc.x) : ((s & 1) ? sc.w : sc.z);
            const __half2 sch = __half2half2(__int2half_rn((int)(signed char)((word >> (8 * (h + 2 * jl))) & 0xff)));
#pragma unroll
            for (int c = 0; c < WPS / 2; c++) {
                unsigned hi[4], lo[4];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const unsigned nib = jl ? lb[n][2 * c + k] : la[n][2 * c + k];
                    const unsigned q = ((nib >> (4 * (s & 1))) & 0x0f0f0f0fu) | (((hq[n][2 * c + k] >> (2 * j)) & 0x03030303u) << 4);
                    const __half2 q0 = __hsub2(tc_bytes_1024<0>(q), off), q1 = __hsub2(tc_bytes_1024<1>(q), off);
                    const __half2 p0 = __hmul2(sch, q0), p1 = __hmul2(sch, q1);
                    hi[2 * k] = tc_bits(p0), hi[2 * k + 1] = tc_bits(p1);
                    lo[2 * k] = tc_bits(__hfma2(sch, q0, __hneg2(p0))), lo[2 * k + 1] = tc_bits(__hfma2(sch, q1, __hneg2(p1)));
                }
                const int chunk = 4 * jl + (WPS / 2) * h + c;
                *reinterpret_cast<uint4*>(tile + tc_swz(row, chunk)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(tile + plane_bytes + tc_swz(row, chunk)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
    }
};

// ------------------------------------------------------------------ the kernel

// CTA = 128 weight rows x a tile of tokens x a part of the k range, in stages of 64 weights: 16 KB of A per plane, and the
// tokens' two planes of B.  Warps 4-11 turn weights into A tiles, lanes of warp 1 request the B planes as bulk copies, lane
// 0 of warps 0 and 2 issues the MMAs, the warps behind drain the accumulators (two buffers in TMEM) into the row sums they
// hold in registers (TMEM lanes 32 (w & 3) .., a share of the tokens); every role runs ahead of the next as far as the
// rings allow.  (With all warps doing everything in turn a stage took 4 500 cycles.)  Two forms:
//
//   pair    batches of more than 128 tokens.  Two CTAs on adjacent row tiles share up to 256 tokens with cta_group::2
//           MMAs of 256 x 256 x 16: each holds its own rows of A and half of the tokens' B, which halves what B costs in
//           L2 reads and in shared-memory reads per MMA.  One CTA alone on 2 x 128 rows x 128 tokens ran at a third of it.
//   single  up to 128 tokens.  The high and the low terms of the tokens are columns of ONE MMA, so A is read once for both.
//
// Gate / up pairs (ZIP) alternate the two matrices' rows in the tile, so that a gate value meets its up value in the
// neighbouring lane, as the two rows of a RoPE pair do.  The k range is cut over the CTAs of a cluster (grid.y) where a
// matrix has too few rows to fill the chip: their sums meet through distributed shared memory, each CTA finishing its
// share of the tokens.
constexpr int TC_C_WARPS = 4, TC_A_WARPS = 8, TC_MAX_STAGES = 6;
constexpr size_t TC_SMEM_MAX = 225 * 1024;
enum { TC_PAIR, TC_SINGLE };
// Draining warps and the registers of a thread of each role (what they add up to is what the launch has).  Draining is a
// chain of TMEM loads (300 cycles for 16 columns, waited for one by one), so sixteen warps share the columns; the pairs on
// Q6_K matrices, whose third MMA leaves more time, keep eight and leave the registers to the unpacking.
template <int FORM, bool Q4>
struct TcRoles {
    static constexpr int D_WARPS = FORM == TC_PAIR && !Q4 ? 8 : 16, THREADS = 32 * (TC_C_WARPS + TC_A_WARPS + D_WARPS);
    static constexpr int LAUNCH_REGS = D_WARPS == 8 ? 96 : 72;
    static constexpr int C_REGS = D_WARPS == 8 ? 32 : 24, A_REGS = D_WARPS == 8 ? 64 : FORM == TC_PAIR ? 48 : 72,
                         D_REGS = D_WARPS == 8 ? 160 : FORM == TC_PAIR ? 96 : 80;
    static constexpr int NC = FORM == TC_PAIR ? 1024 / D_WARPS : 32;  // tokens of a draining warp
    static_assert(32 * (TC_C_WARPS * C_REGS + TC_A_WARPS * A_REGS + D_WARPS * D_REGS) <= THREADS * LAUNCH_REGS && THREADS * LAUNCH_REGS <= 65536,
                  "more registers than the launch has");
};
// Registers of a role: N of the LAUNCH a thread has.  Fewer must be given back, more asked for.
template <int N, int LAUNCH>
__device__ __forceinline__ void tc_regs() {
    static_assert(N % 8 == 0, "");
    if constexpr (N < LAUNCH) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
    else if constexpr (N > LAUNCH) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

struct TcArgs {
    const unsigned char* image;
    const float* tscale;
    int M, Mp, NT;   // tokens, with padding; tokens per tile
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

template <class RAW, int FORM>
__global__ void __launch_bounds__(TcRoles<FORM, RAW::PLANES == 1>::THREADS, 1) k_gemm_tc(const TcArgs a) {
    constexpr bool Q4 = RAW::PLANES == 1, PAIR = FORM == TC_PAIR;
    using Roles = TcRoles<FORM, Q4>;
    constexpr int TC_D_WARPS = Roles::D_WARPS, CGS = TC_D_WARPS / 4, NC = Roles::NC;  // column groups of NC tokens
    constexpr int CG = PAIR ? 2 : 1;  // CTAs of an MMA
    constexpr int DR = PAIR ? 2 : 1;  // stages an accumulator runs over
    extern __shared__ __align__(128) unsigned char tc_smem_raw[];
    __shared__ unsigned long long full[TC_MAX_STAGES], empty[TC_MAX_STAGES], accfull[2], accempty[2];
    __shared__ unsigned tmem_slot;
    __shared__ int dead_s;
    __shared__ float tscale_s[PAIR ? 256 : 128];
    volatile int* dead = &dead_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = gridDim.y, part = blockIdx.y;           // k parts
    const int pr = PAIR ? blockIdx.x & 1 : 0;             // this CTA of the pair; 0 leads
    const int lead = PAIR ? 2 * part : part;              // cluster rank of the pair's leader (single: of this CTA)
    const bool cluster = PAIR || S > 1;
    const int n0 = blockIdx.z * a.NT, nt = min(a.NT, a.Mp - n0), nst = a.nst;
    const int ntc = nt / CG, nc0 = n0 + pr * ntc;         // the tokens whose B this CTA holds
    const bool second = !a.zip && a.A2.data != nullptr && (int)blockIdx.x >= a.tiles1;
    const Mat& A = second ? a.A2 : a.A1;
    const int nb = A.nb, K = A.K, N = A.N;
    const int row0 = ((int)blockIdx.x - (second ? a.tiles1 : 0)) * (a.zip ? 64 : 128);
    const int b0 = nb * part / S, b1 = nb * (part + 1) / S;
    // stages of group sums come in two: the high terms of dmin * m with both of the sums' terms, its low terms with the high ones
    const int n_min = Q4 ? tc_min_stages(K) : 0, m0 = n_min * part / S, m1 = n_min * (part + 1) / S;
    if (warp == 3) {
        // The tile's weights start towards L2 at once, and so do those of the CTA that will follow on this SM: the registers
        // of the unpacking warps hold one block ahead, which covers an L2 hit but not a trip to memory.
        auto ahead = [&](const Mat& m, int group) {
            if (group * ROW_GROUP >= m.N) return;
            const size_t f = (size_t)group * ROW_GROUP * nb, t0 = (f + ROW_GROUP * b0) >> 5, t1 = (f + ROW_GROUP * b1 + 31) >> 5;
            constexpr size_t TB = Q4 ? Q4_TILE_BYTES : Q6_TILE_BYTES;
            bulk_prefetch_l2(m.data + t0 * TB, (unsigned)((t1 - t0) * TB));
        };
        for (int w = 0; w <= 1; w++) {
            const int row = row0 + w * a.ahead * (a.zip ? 64 : 128);
            if (w == 1 && a.ahead == 0) break;
            if (a.zip) ahead(lane & 1 ? a.A2 : A, row / ROW_GROUP + (lane >> 1));
            else ahead(A, row / ROW_GROUP + lane);
        }
    }
    const int min_stages = 2 * (m1 - m0), stages = min_stages + 4 * (b1 - b0);
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int A_SUB = RAW::PLANES * 16384;            // A of 64 weights: one 16 KB tile per plane
    const int b_plane = ntc * 128, stage_bytes = A_SUB + 2 * (a.NT / CG) * 128;
    constexpr unsigned ACC_COLS = (PAIR ? 1 : 2) * CGS * NC, TMEM_COLS = 2 * ACC_COLS;  // the tokens; single: high then low terms
    if (tid == 0) {
        for (int i = 0; i < nst; i++) {
            // every CTA's own A warps and B (with the bytes); the leader's also the word that the peer's are complete
            mbar_init(full + i, TC_A_WARPS + 1 + (PAIR && pr == 0));
            mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(accfull + i, 1);
            mbar_init(accempty + i, TC_D_WARPS + (PAIR && pr == 0));
        }
        dead_s = 0;
        mbar_fence_init();
    }
    if (warp == 0) tc_alloc<CG>(&tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    if (cluster) cluster_sync_all();  // the barriers of the cluster exist
    tc_fence_after();
    const unsigned tmem = tmem_slot;
    float* sums = reinterpret_cast<float*>(smem);  // S > 1: [token][128 rows], over the stages once every MMA has read them

    if (warp < TC_C_WARPS) {
        tc_regs<Roles::C_REGS, Roles::LAUNCH_REGS>();
        if ((warp & 1) == 0 && pr == 0) {
            // Two issuing threads take turns by accumulator: a wait costs one about 300 cycles even when there is nothing to
            // wait for, and the MMAs of a stage 650.
            if (lane == 0) {
                TcRing ring;
                const unsigned long long d0 = tc_desc(smem_u32(smem));
                for (int j = 0; j < stages; j++) {
                    const int r = j / DR, buf = r & 1;
                    if (buf != warp >> 1) {
                        ring.next(nst);
                        continue;
                    }
                    const bool fresh = j % DR == 0;
                    if (fresh && r >= 2) tc_wait<PAIR>(accempty + buf, ((r >> 1) - 1) & 1, dead);
                    tc_wait<PAIR>(full + ring.slot, ring.lap, dead);
                    // what the unpacking warps stored becomes visible to the tensor core here, not where they store it: a
                    // fence there waits for the warp's loads in flight, the next block's words (900 to 2 200 cycles a block)
                    fence_proxy_async();
                    tc_fence_after();
                    const unsigned acc = tmem + buf * ACC_COLS;
                    const unsigned long long da = d0 + ((ring.slot * stage_bytes) >> 4), db = da + (A_SUB >> 4);
                    if (Q4 && j < min_stages) {
                        const unsigned id = tc_idesc(2, 128 * CG, nt), id2 = tc_idesc(2, 128, 2 * nt);
                        const bool high = !(j & 1);
                        if (!PAIR && high) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) tc_mma<true, CG>(acc, da + 2 * kk, db + 2 * kk, id2, !fresh || kk > 0);
                        } else {
                            // the small products go first: the tensor core truncates as it adds, so what counts is how
                            // often it adds to the full sum
                            if (PAIR && high)
#pragma unroll
                                for (int kk = 0; kk < 4; kk++) tc_mma<true, CG>(acc, da + 2 * kk, db + (b_plane >> 4) + 2 * kk, id, !fresh || kk > 0);
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) tc_mma<true, CG>(acc, da + 2 * kk, db + 2 * kk, id, !fresh || (PAIR && high) || kk > 0);
                        }
                    } else {
                        const unsigned id = tc_idesc(0, 128 * CG, nt), id2 = tc_idesc(0, 128, 2 * nt);
                        if (PAIR) {
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) {
                                tc_mma<false, CG>(acc, da + 2 * kk, db + (b_plane >> 4) + 2 * kk, id, !fresh || kk > 0);
                                if (!Q4) tc_mma<false, CG>(acc, da + 1024 + 2 * kk, db + 2 * kk, id, 1);
                            }
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) tc_mma<false, CG>(acc, da + 2 * kk, db + 2 * kk, id, 1);
                        } else {
                            // Q6_K: the residuals of A touch the high columns alone and go first as well
                            if (!Q4) {
#pragma unroll
                                for (int kk = 0; kk < 4; kk++) tc_mma<false, CG>(acc, da + 1024 + 2 * kk, db + 2 * kk, id2, !fresh || kk > 0);
                            }
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) tc_mma<false, CG>(acc, da + 2 * kk, db + 2 * kk, id2, !Q4 || !fresh || kk > 0);
                        }
                    }
                    tc_commit<CG>(empty + ring.slot, lead);
                    if (j % DR == DR - 1) tc_commit<CG>(accfull + buf, lead);
                    ring.next(nst);
                }
            }
            __syncwarp();
        } else if (PAIR && (warp & 1) == 0) {
            // The second CTA of a pair passes its barriers' phases on to the leader's: one thread each, because an arrival at
            // another CTA that releases at cluster scope holds up the warp that makes it.
            if (lane == 0) {
                TcRing ring;
                if (warp == 0)
                    for (int j = 0; j < stages; j++) {
                        tc_wait<false>(full + ring.slot, ring.lap, dead);
                        fence_proxy_async();
                        tc_arrive_at(full + ring.slot, lead);
                        ring.next(nst);
                    }
                else
                    for (int r = 0; r < stages / DR - 2; r++) {
                        tc_wait<false>(accempty + (r & 1), (r >> 1) & 1, dead);
                        tc_arrive_at(accempty + (r & 1), lead);
                    }
            }
            __syncwarp();
        } else if (warp == 1) {
            griddep_wait();  // the image comes from the previous kernel
            TcRing ring;
            const size_t plane = (size_t)a.Mp * 128;
            const unsigned char* src = a.image + (size_t)nc0 * 128 + (lane & 1) * plane;
            for (int j = 0; j < stages; j++) {
                const bool mins = j < min_stages;
                // a lane per plane; the low terms of dmin * m meet the high plane alone
                const int image_stage = mins ? K / TC_STAGE_K + m0 + (j >> 1) : 4 * b0 + (j - min_stages);
                const int copies = mins && (j & 1) ? 1 : 2;
                if (j >= nst) tc_wait<false>(empty + ring.slot, ring.lap ^ 1, dead);
                if (lane == 0) mbar_expect_tx(full + ring.slot, copies * b_plane);
                __syncwarp();
                if (lane < copies)
                    bulk_load(smem + ring.slot * stage_bytes + A_SUB + lane * b_plane, src + (size_t)2 * image_stage * plane, b_plane, full + ring.slot);
                __syncwarp();
                ring.next(nst);
            }
        }
        griddep_launch_dependents();
        if (S > 1) cluster_sync_all();
        if (cluster) cluster_sync_all();
        else asm volatile("bar.sync 1, %0;" ::"n"(32 * (TC_D_WARPS + TC_C_WARPS)) : "memory");  // the last accumulator has been read
        tc_fence_after();
        if (warp == 0) tc_dealloc<CG>(tmem, TMEM_COLS);
        return;
    }

    if (warp < TC_C_WARPS + TC_A_WARPS) {
        tc_regs<Roles::A_REGS, Roles::LAUNCH_REGS>();
        // this thread's row of the tile and its half of the row's blocks; rows past the matrix repeat its last row
        const int wa = warp - TC_C_WARPS, row_l = (wa & 3) * 32 + lane, h = wa >> 2;
        const uint8_t* wdata = (a.zip && (row_l & 1)) ? a.A2.data : A.data;
        const int f0 = (int)mat_flat(nb, min(row0 + (a.zip ? row_l >> 1 : row_l), N - 1), 0);
        RAW raw;
        raw.load(wdata, f0 + ROW_GROUP * b0, h);  // weights do not depend on earlier kernels
        griddep_launch_dependents();
        TcRing ring;
        int j = 0;
        auto acquire = [&]() {
            if (j >= nst) tc_wait<false>(empty + ring.slot, ring.lap ^ 1, dead);
            return smem + ring.slot * stage_bytes;
        };
        auto publish = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(full + ring.slot);
            ring.next(nst);
            j++;
        };
        if constexpr (Q4) {
            for (int c = m0; c < m1; c++) {
                // groups of 32 weights 32 c .. 32 c + 31 = blocks 4 c .. 4 c + 3, two of them this thread's
                unsigned char* t = nullptr;
#pragma unroll 1
                for (int p = 0; p < 2; p++) {
                    t = acquire();
#pragma unroll 1
                    for (int i = 0; i < 2; i++) {
                        const int b = 4 * c + 2 * h + i, f = f0 + ROW_GROUP * min(b, nb - 1);
                        const int4 hdr = __ldg(reinterpret_cast<const int4*>(wdata + (size_t)(f >> 5) * Q4_TILE_BYTES + (f & 31) * 16));
                        const unsigned s1 = (unsigned)hdr.z, s2 = (unsigned)hdr.w;
                        const unsigned ml = s1 & 0x3f3f3f3fu, mh = ((s2 >> 4) & 0x0f0f0f0fu) | (((s1 >> 6) & 0x03030303u) << 4);
                        const float dmin = b < nb ? f16_to_f32((unsigned short)((unsigned)hdr.x >> 16)) : 0.f;
#pragma unroll
                        for (int half = 0; half < 2; half++) {
                            const unsigned mm = half ? mh : ml;
                            unsigned o[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const float v = dmin * i2f_small((int)((mm >> (8 * k)) & 0xff));
                                const unsigned top = __float_as_uint(v) & 0xffffe000u;
                                o[k] = p ? __float_as_uint(v - __uint_as_float(top)) : top;
                            }
                            *reinterpret_cast<uint4*>(t + tc_swz(row_l, 2 * (2 * h + i) + half)) = make_uint4(o[0], o[1], o[2], o[3]);
                        }
                    }
                    publish();
                }
            }
        }
        for (int b = b0; b < b1; b++) {
            unsigned char* t = nullptr;
#pragma unroll
            for (int s = 0; s < 4; s++) {
                t = acquire();
                raw.store(s, t, row_l, h, 16384);
                publish();
                if (b + 1 < b1) raw.load_stage(s, wdata, f0 + ROW_GROUP * (b + 1), h);  // the words just used, of the next block
            }
        }
        if (S > 1) cluster_sync_all();
        if (cluster) cluster_sync_all();
        return;
    }

    tc_regs<Roles::D_REGS, Roles::LAUNCH_REGS>();
    const int quad = warp & 3, cg = (warp - TC_C_WARPS - TC_A_WARPS) >> 2, row_d = quad * 32 + lane;
    float2 tot[NC / 2];  // token pairs: one packed multiply-add joins two accumulators to their sums
#pragma unroll
    for (int i = 0; i < NC / 2; i++) tot[i] = make_float2(0.f, 0.f);
    {
        const uint8_t* ddata = (a.zip && (row_d & 1)) ? a.A2.data : A.data;
        const int df = (int)mat_flat(nb, min(row0 + (a.zip ? row_d >> 1 : row_d), N - 1), 0);
        auto load_d = [&](int b) {
            const int f = df + ROW_GROUP * min(b, nb - 1);
            const uint8_t* p = ddata + (Q4 ? (size_t)(f >> 5) * Q4_TILE_BYTES + (f & 31) * 16
                                           : (size_t)(f >> 5) * Q6_TILE_BYTES + Q6_PIECES * 512 + (f & 31) * 2);
            return f16_to_f32(__ldg(reinterpret_cast<const unsigned short*>(p)));
        };
        float dnext = load_d(b0), dcur = -1.f;
        griddep_launch_dependents();
        griddep_wait();  // nothing reaches an accumulator before the image is complete; token scales and residuals are then, too
        const int td = tid - 32 * (TC_C_WARPS + TC_A_WARPS);
        if (td < nt) tscale_s[td] = n0 + td < a.M ? a.tscale[n0 + td] : 0.f;
        const int min_rounds = min_stages / DR;
        int left = min_rounds;  // rounds until the factor changes
        for (int r = 0; r < stages / DR; r++) {
            const bool minus = Q4 && r < min_rounds;
            if (left == 0) {
                dcur = dnext;
                dnext = load_d(b0 + (r - min_rounds) / (4 / DR) + 1);
                left = 4 / DR;
            }
            left--;
            const int buf = r & 1;
            tc_wait<false>(accfull + buf, (r >> 1) & 1, dead);
            tc_fence_after();
            const unsigned at = tmem + ((unsigned)quad << 21) + buf * ACC_COLS + cg * NC;
            // The truncations cost an accumulator, on average, about half (Q4_K) or three quarters (Q6_K) of a unit in its
            // last place (measured against float64); raising the factor by one unit in as many stages gives it back.
            const float f = (r & 3) < (Q4 ? 2 : 3) ? dcur * 1.00000012f : dcur;
            const float2 ff = make_float2(f, f);
            const bool low = !PAIR && !(minus && (r & 1));  // there are low columns
#pragma unroll
            for (int c = 0; c < NC; c += 16) {  // columns of a load
                if (cg * NC + c >= nt) break;
                float v[16], w[16];
                tc_ld<16>(v, at + c);
                if (low) tc_ld<16>(w, at + nt + c);
                tc_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; i++) tot[c / 2 + i] = fma_f32x2(ff, make_float2(v[2 * i], v[2 * i + 1]), tot[c / 2 + i]);
                if (low) {
#pragma unroll
                    for (int i = 0; i < 8; i++) tot[c / 2 + i] = fma_f32x2(ff, make_float2(w[2 * i], w[2 * i + 1]), tot[c / 2 + i]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty + buf);
        }
    }
    if (!cluster) asm volatile("bar.sync 1, %0;" ::"n"(32 * (TC_D_WARPS + TC_C_WARPS)) : "memory");
    else asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_D_WARPS) : "memory");  // the token scales

    // ---- epilogue
    auto total = [&](int i) { return (i & 1) ? tot[i >> 1].y : tot[i >> 1].x; };
    const int id_base = second ? a.id2 : a.id1;
    const int row = row0 + (a.zip ? row_d >> 1 : row_d);
    const bool odd = lane & 1, store = a.epi.kind == CEPI_STORE;
    ChunkEpi epi = a.epi;
    epi.bias = nullptr;  // added here, once per row
    const float bias = a.epi.bias && row < N ? a.epi.bias[2 * id_base + row] : 0.f;
    // items of two adjacent lanes (RoPE pairs, gate and up): id of the item and whether it exists
    const int item = id_base + (a.zip ? row : row >> 1);
    const bool item_on = a.zip ? row < N : (row & ~1) < N;
    if (S == 1) {
        const int t0 = n0 + cg * NC, tn = min(NC, min(nt, a.M - n0) - cg * NC);
#pragma unroll
        for (int i0 = 0; i0 < NC; i0 += 8) {
            if (i0 >= tn) break;
            // eight tokens' scales and residuals in flight together: a load behind each store would cost a trip to L2
            float v[8];
            {
                float ts[8], res[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const bool on = i0 + i < tn;
                    ts[i] = on ? tscale_s[cg * NC + i0 + i] : 0.f;
                    res[i] = on && store && epi.use_res == 2 && row < N ? epi.out[(size_t)(t0 + i0 + i) * epi.ldo + 2 * id_base + row] : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = total(i0 + i) * ts[i] + res[i] + bias;
            }
            if (store) {
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i0 + i < tn && row < N) epi.out[(size_t)(t0 + i0 + i) * epi.ldo + 2 * id_base + row] = v[i];
            } else {
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    // the even lane takes token i, the odd one token i + 1
                    const float got = __shfl_xor_sync(TFR_FULL_MASK, odd ? v[i] : v[i + 1], 1);
                    const int t = i0 + i + (odd ? 1 : 0);
                    if (t < tn && item_on) ChunkEpiTok{&epi, t0 + t}.apply(item, odd ? got : v[i], odd ? v[i + 1] : got);
                }
            }
        }
    } else {
        if (cg * NC < nt) {
#pragma unroll
            for (int i = 0; i < NC; i++)
                if (cg * NC + i < nt) sums[(cg * NC + i) * 128 + row_d] = total(i);
        }
        cluster_sync_all();
        const int per = (nt + S - 1) / S, c0 = part * per, cn = min(per, min(nt, a.M - n0) - c0);
        for (int c4 = c0 + cg; c4 < c0 + cn; c4 += 4 * CGS) {
            // four tokens' residuals and the parts' sums in flight together
            float res[4], v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = c4 + q * CGS;
                res[q] = c < c0 + cn && store && epi.use_res == 2 && row < N ? epi.out[(size_t)(n0 + c) * epi.ldo + 2 * id_base + row] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = min(c4 + q * CGS, c0 + cn - 1);
                const unsigned at0 = smem_u32(sums + c * 128 + row_d);
                float x[8];
#pragma unroll
                for (int p = 0; p < 8; p++) {
                    x[p] = 0.f;
                    if (p < S) {
                        unsigned remote;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at0), "r"(PAIR ? 2 * p + pr : p));
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[p]) : "r"(remote) : "memory");
                    }
                }
                v[q] = 0.f;
#pragma unroll
                for (int p = 0; p < 8; p++) v[q] += x[p];
                v[q] = v[q] * tscale_s[c] + res[q] + bias;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = c4 + q * CGS;
                if (c >= c0 + cn) break;
                if (store) {
                    if (row < N) epi.out[(size_t)(n0 + c) * epi.ldo + 2 * id_base + row] = v[q];
                } else {
                    const float got = __shfl_xor_sync(TFR_FULL_MASK, v[q], 1);
                    if (!odd && item_on) ChunkEpiTok{&epi, n0 + c}.apply(item, v[q], got);
                }
            }
        }
    }
    if (tid == 32 * (TC_C_WARPS + TC_A_WARPS) && dead_s && a.st) a.st->err = 2;
    if (cluster) cluster_sync_all();  // nobody leaves while others use its barriers, operands or sums
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

inline bool tc_type(int type) { return type == TFR_Q4_K || type == TFR_Q6_K; }

template <class RAW, int FORM>
inline cudaError_t launch_tc(cudaStream_t stream, int sms, TcArgs& a, int row_tiles, int S) {
    using Roles = TcRoles<FORM, RAW::PLANES == 1>;
    constexpr bool PAIR = FORM == TC_PAIR;
    const int stage = RAW::PLANES * 16384 + 2 * (a.NT / (PAIR ? 2 : 1)) * 128;
    a.nst = std::min(TC_MAX_STAGES, (int)((TC_SMEM_MAX - 1024) / stage));
    a.ahead = S == 1 && row_tiles > sms ? sms : 0;
    const size_t sums = S > 1 ? (size_t)a.NT * 512 : 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(PAIR ? (row_tiles + 1) & ~1 : row_tiles, S, (a.Mp + a.NT - 1) / a.NT);
    cfg.blockDim = dim3(Roles::THREADS);
    cfg.dynamicSmemBytes = std::max((size_t)a.nst * stage, sums) + 1024;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = PAIR ? 2 : 1;
    attr[1].val.clusterDim.y = S;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = PAIR || S > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_gemm_tc<RAW, FORM>, (const TcArgs)a);
}

// out = epilogue(W x) for the M tokens of an operand image; jb: the second matrix of a gate/up pair or one that follows.
inline cudaError_t launch_gemm_tc(cudaStream_t stream, int sms, const unsigned char* image, const float* tscale, int M, const RowJob& ja,
                                  const RowJob& jb, const ChunkEpi& epi, TokenState* st) {
    TcArgs a{};
    a.image = image, a.tscale = tscale, a.M = M, a.Mp = tc_pad_tokens(M);
    a.A1 = ja.m, a.A2 = jb.m, a.id1 = ja.id_base, a.id2 = jb.id_base;
    a.zip = epi.kind == CEPI_SILU;
    a.epi = epi, a.st = st;
    const bool q4 = ja.m.type == TFR_Q4_K;
    const int rows = a.zip ? 64 : 128;
    a.tiles1 = (ja.m.N + rows - 1) / rows;
    const int tiles = a.tiles1 + (!a.zip && jb.m.data ? (jb.m.N + rows - 1) / rows : 0);
    // CTAs the device runs at once by cluster size (GPCs hold whole clusters)
    auto fit = [&](int ctas) { return ctas <= 2 ? sms : ctas == 4 ? 132 : 112; };
    // the form and the number of k parts with the shortest longest chain: waves of CTAs x stages x what a stage takes, in
    // units of a 128-row, 128-token MMA stage
    auto plan = [&](int form, int& S, int& NT) {
        const bool pair = form == TC_PAIR;
        const int most = pair ? 256 : 128, tok_tiles = (a.Mp + most - 1) / most, unit = pair ? 32 : 16;
        NT = ((a.Mp + tok_tiles - 1) / tok_tiles + unit - 1) / unit * unit;
        double best = 1e30;
        for (int s = 1; s <= (pair ? 4 : 8) && s <= ja.m.nb; s *= 2) {
            const int ctas = (pair ? (tiles + 1) & ~1 : tiles) * tok_tiles * s, at_once = fit(pair ? 2 * s : s);
            const double stage = pair ? 0.4 + 1.2 * NT / 128 : 0.6 + 1.2 * NT / 128;
            const double t = (double)((ctas + at_once - 1) / at_once) * ((4.5 * ((ja.m.nb + s - 1) / s) * stage) + 6 + (s > 1 ? 3 : 0));
            if (t < best) best = t, S = s;
        }
        return best;
    };
    int S = 1, S2 = 1, NT2 = 0;
    const double single = plan(TC_SINGLE, S, a.NT);
    if (M > 128 && plan(TC_PAIR, S2, NT2) < single) {
        a.NT = NT2;
        return q4 ? launch_tc<RawQ4, TC_PAIR>(stream, sms, a, tiles, S2) : launch_tc<RawQ6, TC_PAIR>(stream, sms, a, tiles, S2);
    }
    return q4 ? launch_tc<RawQ4, TC_SINGLE>(stream, sms, a, tiles, S) : launch_tc<RawQ6, TC_SINGLE>(stream, sms, a, tiles, S);
}

}  // namespace tfr
