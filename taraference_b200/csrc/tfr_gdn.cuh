// Kernels of the hybrid (Qwen3.5-style) layers: the Gated-DeltaNet decode step and the
// per-head Q/K RMSNorm + partial RoPE + KV store of the gated full-attention layers.
//
// Reference: kernels/deltanet.cu:530-622 (conv + SiLU + split + L2), :628-728 (decay, delta rule,
// read-out, gated RMSNorm), :144-173 (Q|gate split), :189-235 (Q/K norm + partial RoPE),
// kernels/ops.cu:471-486 (f16 KV store).  The reference runs the mixer as two launches with Q, K, V
// bounced through global memory and walks the 128x128 state twice (decay pass, then update);
// here one CTA per V head does the conv for the 3 x 128 channels it needs, keeps its 64 KB
// state in registers and touches every state element exactly once (one load, one store).
#pragma once
#include "tfr_common.cuh"

namespace tfr {

constexpr int GDN_D = 128;        // state size per head (ssm.state_size of the supported models)
constexpr int GDN_PARTS = 4;      // row slabs of the state handled by different threads of a column
constexpr int GDN_THREADS = GDN_D * GDN_PARTS;
constexpr int GDN_MAX_KERNEL = 4;

struct GdnArgs {
    const float* proj;     // [channels | val_dim | n_v | n_v]: raw qkv, z gate, beta, alpha projections
    const float* conv_w;   // [channels][kernel], tap k of channel c at k + c * kernel (GGUF dims [kernel, channels])
    float* conv_ring;      // [kernel][channels]: slot (pos + ring_off) % kernel takes the current input
    float* state;          // [n_v][128][128] fp32; with a TokenState: its cache's arrays + the two offsets
    size_t conv_off, state_off;
    const float* ssm_a;    // [n_v], already -exp(A_log)
    const float* ssm_dt;   // [n_v]
    const float* norm_w;   // [128]
    float* out;            // [n_v * 128]: feeds the ssm_out projection
    int n_k, n_v, kernel;
    float eps;
    int slot;              // ring slot when st == nullptr
};

// The conv history is a ring indexed by position instead of the reference's shifted window
// (deltanet.cu:552-558): nothing moves, and the two V heads that share a K head can both read
// the Q/K history without racing against a shift.
// The sum over the history, and with the current input the channel's value.
__device__ __forceinline__ float gdn_conv_history(const GdnArgs& a, int c, int channels, int slot) {
    const int km1 = a.kernel - 1;
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < GDN_MAX_KERNEL - 1; k++) {
        if (k < km1) {
            int s = slot - km1 + k;
            s += s < 0 ? a.kernel : 0;
            acc += a.conv_w[(size_t)c * a.kernel + k] * a.conv_ring[(size_t)s * channels + c];
        }
    }
    return acc;
}
__device__ __forceinline__ float gdn_conv_value(const GdnArgs& a, int c, int channels, int slot, bool write, float acc, float w, float xt) {
    acc += w * xt;
    if (write) a.conv_ring[(size_t)slot * channels + c] = xt;
    return acc / (1.f + expf(-acc));
}

// Inside a token (st) the kernel before this one is the layer's projection, which writes neither the state nor the conv history
// and starts this kernel only behind its own wait, when what ran before it is complete (WaitsFirst): the state (64 KB a head) and all that does not come from the
// projection is asked for before the dependency wait and arrives under it (64 tokens in and 32 out on the hybrid 4B shape, with the
// same in k_qk_norm_rope_store: 46.33 -> 44.57 ms).  A stand-alone call may follow another one on the same state and waits first.
__global__ void __launch_bounds__(GDN_THREADS, 1) k_gdn_step(GdnArgs a, const TokenState* st) {
    int slot = a.slot, done = 0;
    if (st) {
        done = st->done;
        a.conv_ring = st->kv_conv + a.conv_off;
        a.state = st->kv_ssm + a.state_off;
        slot = (st->pos + st->ring_off) % a.kernel;
    }
    if (!st || done) {
        griddep_wait();
        griddep_launch_dependents();
        if (done) return;
    }
    constexpr int D = GDN_D, R = D / GDN_PARTS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.x, hk = h % a.n_k;
    const int key_dim = a.n_k * D, val_dim = a.n_v * D, channels = 2 * key_dim + val_dim;
    const int j = tid & (D - 1), part = tid >> 7;
    float* S = a.state + (size_t)h * D * D;

    __shared__ float sq[D], sk[D], sv[D], sz[D];
    __shared__ float red[GDN_PARTS][D];
    __shared__ float wred[16];
    __shared__ float sg, sb;

    // the state loads go out first; the conv and the norms run while they are in flight
    float s[R];
#pragma unroll
    for (int r = 0; r < R; r++) s[r] = __ldcs(S + (size_t)(part * R + r) * D + j);

    // part 0: Q channel j of K head hk, part 1: K channel, part 2: V channel j of head h; part 3: the z gate of output j
    const int c = part == 0 ? hk * D + j : part == 1 ? key_dim + hk * D + j : part == 2 ? 2 * key_dim + h * D + j : channels + h * D + j;
    float cv = 0.f, cw = 0.f;
    if (part < 3) {
        cv = gdn_conv_history(a, c, channels, slot);
        cw = a.conv_w[(size_t)c * a.kernel + a.kernel - 1];
    }
    const float nw = a.norm_w[j], dt = tid == 0 ? a.ssm_dt[h] : 0.f, decay = tid == 0 ? a.ssm_a[h] : 0.f;
    if (st) {
        griddep_wait();  // the projections come from the previous kernel
        griddep_launch_dependents();
    }
    const float xt = a.proj[c];
    if (tid == 0) {
        const float br = a.proj[channels + val_dim + h];
        sb = 1.f / (1.f + expf(-br));
        const float z = a.proj[channels + val_dim + a.n_v + h] + dt;
        const float sp = (z > 20.f) ? z : log1pf(expf(z));
        sg = expf(sp * decay);
    }
    if (part < 3) cv = gdn_conv_value(a, c, channels, slot, part == 2 || h < a.n_k, cv, cw, xt);
    else sz[j] = xt;
    // L2 norms of Q and K (sum of squares, deltanet.cu:598-620)
    const float sqr = warp_sum(part < 2 ? cv * cv : 0.f);
    if (lane == 0) wred[warp] = sqr;
    __syncthreads();
    if (part == 0) {
        const float inv = rsqrtf(wred[0] + wred[1] + wred[2] + wred[3] + a.eps);
        sq[j] = (cv * inv) * 0.08838834764f;  // 1/sqrt(128), deltanet.cu:668
    } else if (part == 1) {
        const float inv = rsqrtf(wred[4] + wred[5] + wred[6] + wred[7] + a.eps);
        sk[j] = cv * inv;
    } else if (part == 2) {
        sv[j] = cv;
    }
    __syncthreads();
    const float g = sg, b = sb;

    // decay and the memory read-out of this column slab
    float kv = 0.f;
#pragma unroll
    for (int r = 0; r < R; r++) {
        s[r] *= g;
        kv += s[r] * sk[part * R + r];
    }
    red[part][j] = kv;
    __syncthreads();
    const float delta = (sv[j] - (red[0][j] + red[1][j] + red[2][j] + red[3][j])) * b;
    __syncthreads();
    float o = 0.f;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float ki = sk[part * R + r];
        s[r] += ki * delta;
        __stcs(S + (size_t)(part * R + r) * D + j, s[r]);
        o += s[r] * sq[part * R + r];
    }
    red[part][j] = o;
    __syncthreads();
    // gated RMSNorm over the head's 128 outputs (deltanet.cu:703-727)
    float oj = 0.f;
    if (part == 0) oj = red[0][j] + red[1][j] + red[2][j] + red[3][j];
    const float ss = warp_sum(oj * oj);
    if (part == 0 && lane == 0) wred[8 + warp] = ss;
    __syncthreads();
    if (part == 0) {
        const float scale = rsqrtf((wred[8] + wred[9] + wred[10] + wred[11]) * (1.f / (float)D) + a.eps);
        const float gate = sz[j];
        const float silu = gate / (1.f + expf(-gate));
        a.out[h * D + j] = oj * scale * nw * silu;
    }
}

// ------------------------------------------------------------------ a batch of tokens through the mixer

// M tokens of a prompt.  What does not depend on the state runs over all tokens at once (k_gdn_chunk_conv: the conv and
// the L2 norms; k_gdn_chunk_norm: the gated RMSNorm); the recurrence itself (k_gdn_chunk_scan) keeps the state in
// registers and steps through the tokens without a barrier.  Every value is computed by the operations of k_gdn_step in
// the same order.
struct GdnChunkArgs {
    const float* proj;     // [M][ld]: raw qkv, z gate, beta, alpha projections
    int ld;
    const float* conv_w;
    float* conv_ring;      // slot (slot0 + m) % kernel takes token m
    float* state;          // [n_v][128][128]
    const float *ssm_a, *ssm_dt, *norm_w;
    float* mixed;          // [M][channels]: q (scaled), k, v after the conv
    float* gates;          // [M][n_v][2]: decay, write strength
    float* out;            // [M][n_v * 128]
    int M, n_k, n_v, kernel, slot0;
    float eps;
};

constexpr int GDN_CONV_TOKENS = 8;  // tokens of a CTA: a channel's four inputs slide through registers
// CTA = 128 channels (a head of Q, K or V) x 8 tokens.
__global__ void __launch_bounds__(GDN_D) k_gdn_chunk_conv(GdnChunkArgs a) {
    constexpr int T = GDN_CONV_TOKENS;
    __shared__ float wred[T][4];
    const int j = threadIdx.x, lane = j & 31, warp = j >> 5, grp = blockIdx.x, t0 = blockIdx.y * T, tn = min(T, a.M - t0);
    const int key_dim = a.n_k * GDN_D, val_dim = a.n_v * GDN_D, channels = 2 * key_dim + val_dim, c = grp * GDN_D + j, km1 = a.kernel - 1;
    float w[GDN_MAX_KERNEL], x[GDN_MAX_KERNEL - 1 + T];  // taps; inputs t0 - km1 ..
#pragma unroll
    for (int k = 0; k < GDN_MAX_KERNEL; k++) w[k] = k < a.kernel ? a.conv_w[(size_t)c * a.kernel + k] : 0.f;
    griddep_wait();
    griddep_launch_dependents();
#pragma unroll
    for (int i = 0; i < GDN_MAX_KERNEL - 1 + T; i++) {
        const int t = t0 - km1 + i;
        x[i] = i >= km1 + tn ? 0.f
               : t >= 0      ? a.proj[(size_t)t * a.ld + c]
                             : a.conv_ring[(size_t)((a.slot0 + t + a.kernel) % a.kernel) * channels + c];
    }
    float cv[T];
#pragma unroll
    for (int t = 0; t < T; t++) {
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < GDN_MAX_KERNEL; k++)
            if (k < a.kernel) acc += w[k] * x[t + k];
        cv[t] = acc / (1.f + expf(-acc));
    }
    if (grp < 2 * a.n_k) {
#pragma unroll
        for (int t = 0; t < T; t++) {
            const float s = warp_sum(cv[t] * cv[t]);
            if (lane == 0) wred[t][warp] = s;
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < T; t++) {
            cv[t] *= rsqrtf(wred[t][0] + wred[t][1] + wred[t][2] + wred[t][3] + a.eps);
            if (grp < a.n_k) cv[t] *= 0.08838834764f;
        }
    } else if (j < tn) {
        const int h = grp - 2 * a.n_k, m = t0 + j;
        const float* p = a.proj + (size_t)m * a.ld + channels + val_dim;
        const float z = p[a.n_v + h] + a.ssm_dt[h];
        const float sp = (z > 20.f) ? z : log1pf(expf(z));
        reinterpret_cast<float2*>(a.gates)[(size_t)m * a.n_v + h] = make_float2(expf(sp * a.ssm_a[h]), 1.f / (1.f + expf(-p[h])));
    }
#pragma unroll
    for (int t = 0; t < T; t++)
        if (t < tn) a.mixed[(size_t)(t0 + t) * channels + c] = cv[t];
}

// CTA = 32 columns of a head's state: four lanes share a column, 32 rows each, so a token costs a chain of 32
// multiply-adds and a few shuffles.  What bounds it is that chain (about 300 cycles a token); columns are spread over as
// many warps as it takes to have one on every scheduler of the chip.  The tokens' vectors arrive 16 tokens at a time.
constexpr int GDN_SCAN_THREADS = 128, GDN_SCAN_COLS = 32, GDN_SCAN_TOKENS = 16, GDN_SCAN_SLAB = 36;  // 32 rows + padding
__global__ void __launch_bounds__(GDN_SCAN_THREADS) k_gdn_chunk_scan(GdnChunkArgs a) {
    constexpr int D = GDN_D, R = D / GDN_PARTS, T = GDN_SCAN_TOKENS, SL = GDN_SCAN_SLAB;
    __shared__ __align__(16) float kq[2][T][2][GDN_PARTS * SL];
    __shared__ __align__(16) float vs[2][T][GDN_SCAN_COLS];
    __shared__ float2 gs[2][T];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.x, hk = h % a.n_k, col0 = blockIdx.y * GDN_SCAN_COLS;
    const int key_dim = a.n_k * D, channels = 2 * key_dim + a.n_v * D;
    const int jl = warp * 8 + (lane >> 2), j = col0 + jl, part = lane & 3;
    griddep_wait();
    griddep_launch_dependents();
    float* S = a.state + (size_t)h * D * D;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; r++) s[r] = S[(size_t)(part * R + r) * D + j];
    auto fetch = [&](int tile) {
        const int t0 = tile * T, tn = min(T, a.M - t0), buf = tile & 1;
        constexpr int PER = 2 * (D / 4) + GDN_SCAN_COLS / 4;  // 16-byte pieces of a token
        for (int i = tid; i < tn * PER; i += GDN_SCAN_THREADS) {
            const int t = i / PER, c = i - t * PER;
            const float* src = a.mixed + (size_t)(t0 + t) * channels;
            if (c < 2 * (D / 4)) {
                const int isq = c >= D / 4, e = 4 * (isq ? c - D / 4 : c);
                cp_async16(&kq[buf][t][isq][(e / R) * SL + e % R], src + (isq ? 0 : key_dim) + hk * D + e, 16);
            } else {
                const int e = 4 * (c - 2 * (D / 4));
                cp_async16(&vs[buf][t][e], src + 2 * key_dim + h * D + col0 + e, 16);
            }
        }
        if (tid < tn) gs[buf][tid] = reinterpret_cast<const float2*>(a.gates)[(size_t)(t0 + tid) * a.n_v + h];
        cp_async_commit();
    };
    const int tiles = (a.M + T - 1) / T;
    fetch(0);
    for (int tile = 0; tile < tiles; tile++) {
        const int buf = tile & 1, tn = min(T, a.M - tile * T);
        if (tile + 1 < tiles) fetch(tile + 1);
        if (tile + 1 < tiles) cp_async_wait_group<1>();
        else cp_async_wait_group<0>();
        __syncthreads();
        for (int t = 0; t < tn; t++) {
            const float4* k4 = reinterpret_cast<const float4*>(&kq[buf][t][0][part * SL]);
            const float4* q4 = reinterpret_cast<const float4*>(&kq[buf][t][1][part * SL]);
            const float2 gb = gs[buf][t];
            float k[R];
#pragma unroll
            for (int i = 0; i < R / 4; i++) {
                const float4 v = k4[i];
                k[4 * i] = v.x, k[4 * i + 1] = v.y, k[4 * i + 2] = v.z, k[4 * i + 3] = v.w;
            }
            float kv = 0.f;
#pragma unroll
            for (int r = 0; r < R; r++) {
                s[r] *= gb.x;
                kv += s[r] * k[r];
            }
            const int base = lane & ~3;
            const float mem = __shfl_sync(TFR_FULL_MASK, kv, base) + __shfl_sync(TFR_FULL_MASK, kv, base + 1) +
                              __shfl_sync(TFR_FULL_MASK, kv, base + 2) + __shfl_sync(TFR_FULL_MASK, kv, base + 3);
            const float delta = (vs[buf][t][jl] - mem) * gb.y;
            float o = 0.f;
#pragma unroll
            for (int i = 0; i < R / 4; i++) {
                const float4 q = q4[i];
                const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    s[4 * i + u] += k[4 * i + u] * delta;
                    o += s[4 * i + u] * qv[u];
                }
            }
            const float out = __shfl_sync(TFR_FULL_MASK, o, base) + __shfl_sync(TFR_FULL_MASK, o, base + 1) +
                              __shfl_sync(TFR_FULL_MASK, o, base + 2) + __shfl_sync(TFR_FULL_MASK, o, base + 3);
            if (part == 0) a.out[(size_t)(tile * T + t) * (a.n_v * D) + h * D + j] = out;
        }
        __syncthreads();  // the buffer is free
    }
#pragma unroll
    for (int r = 0; r < R; r++) S[(size_t)(part * R + r) * D + j] = s[r];
    // the last inputs of the head's channels become the conv history (the conv has read the one before)
    for (int t = max(0, a.M - a.kernel); t < a.M; t++) {
        const int what = tid >> 5;  // Q, K, V
        if (what < 3 && (what == 2 || h < a.n_k)) {
            const int c = (what == 0 ? 0 : what == 1 ? key_dim : 2 * key_dim) + h * D + col0 + lane;
            a.conv_ring[(size_t)((a.slot0 + t) % a.kernel) * channels + c] = a.proj[(size_t)t * a.ld + c];
        }
    }
}

// CTA = a head of a token: gated RMSNorm of the read-out, in place (deltanet.cu:703-727)
__global__ void __launch_bounds__(GDN_D) k_gdn_chunk_norm(GdnChunkArgs a) {
    __shared__ float wred[4];
    const int j = threadIdx.x, h = blockIdx.x, m = blockIdx.y, channels = (2 * a.n_k + a.n_v) * GDN_D;
    const float w = a.norm_w[j];
    griddep_wait();
    griddep_launch_dependents();
    float* o = a.out + (size_t)m * (a.n_v * GDN_D) + h * GDN_D + j;
    const float gate = a.proj[(size_t)m * a.ld + channels + h * GDN_D + j], oj = *o;
    const float ss = warp_sum(oj * oj);
    if ((j & 31) == 0) wred[j >> 5] = ss;
    __syncthreads();
    const float scale = rsqrtf((wred[0] + wred[1] + wred[2] + wred[3]) * (1.f / (float)GDN_D) + a.eps);
    *o = oj * scale * w * (gate / (1.f + expf(-gate)));
}

// out *= sigmoid(gate), the gated attention of a batch (deltanet.cu:176-186)
__global__ void __launch_bounds__(256) k_gate_rows(float* out, const float* gate, size_t n) {
    griddep_wait();
    griddep_launch_dependents();
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i < n) out[i] *= 1.f / (1.f + expf(-gate[i]));
}

// Gated full attention, between the raw projections and the attention kernel: one CTA per
// query head or KV head and token (grid.y; a decode step has one).  raw = [n_head x (Q_h | G_h) | K | V].
struct QkNormArgs {
    const float* raw;
    const float* q_norm;      // [hd] or nullptr (no norm)
    const float* k_norm;
    float* q_out;             // [n_head * hd]
    float* gate_out;          // [n_head * hd]
    unsigned short* kc;       // layer base [max_seq][n_kv * hd]; with a TokenState: its cache + kv_off
    unsigned short* vc;
    size_t kv_off;
    int n_head, n_kv, hd, n_rot;
    float theta, eps;
    int pos;                  // of the first token; used when st == nullptr
};

__global__ void __launch_bounds__(256) k_qk_norm_rope_store(QkNormArgs a, const TokenState* st) {
    // the state's words together and before the wait, as in k_gdn_step: the kernel before this one (WaitsFirst) does not write them
    int done = 0, pos0 = a.pos;
    if (st) {
        done = st->done, pos0 = st->pos;
        a.kc = st->kv_k + a.kv_off;
        a.vc = st->kv_v + a.kv_off;
    }
    griddep_wait();
    griddep_launch_dependents();
    if (done) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int head = blockIdx.x, hd = a.hd;
    const bool isq = head < a.n_head;
    const int hk = head - a.n_head;
    const int m = blockIdx.y, pos = pos0 + m;
    const int qn2 = 2 * a.n_head * hd, kvdim = a.n_kv * hd;
    const float* raw = a.raw + (size_t)m * (qn2 + 2 * kvdim);
    const float* src = isq ? raw + (size_t)head * 2 * hd : raw + qn2 + (size_t)hk * hd;
    const float* w = isq ? a.q_norm : a.k_norm;
    __shared__ float xs[256];
    __shared__ float wred[8];
    const float x = tid < hd ? src[tid] : 0.f;
    const float ss = warp_sum(x * x);
    if (lane == 0) wred[warp] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int i = 0; i < 8; i++) tot += wred[i];
    float y = x;
    if (w && tid < hd) y = x * rsqrtf(tot / (float)hd + a.eps) * w[tid];
    xs[tid] = y;
    __syncthreads();
    const int half = a.n_rot >> 1;
    if (tid < a.n_rot) {
        const int i = tid < half ? tid : tid - half;
        const float freq = powf(a.theta, -2.f * (float)i / (float)a.n_rot);
        const float ang = (float)pos * freq;
        const float c = cosf(ang), sn = sinf(ang);
        const float x0 = xs[i], x1 = xs[i + half];
        y = tid < half ? x0 * c - x1 * sn : x0 * sn + x1 * c;
    }
    if (tid >= hd) return;
    if (isq) {
        a.q_out[((size_t)m * a.n_head + head) * hd + tid] = y;
        a.gate_out[((size_t)m * a.n_head + head) * hd + tid] = src[hd + tid];
    } else {
        a.kc[(size_t)pos * kvdim + hk * hd + tid] = f32_to_f16_bits_ref(y);
        a.vc[(size_t)pos * kvdim + hk * hd + tid] = f32_to_f16_bits_ref(raw[qn2 + kvdim + hk * hd + tid]);
    }
}

}  // namespace tfr
