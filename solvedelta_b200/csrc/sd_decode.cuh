// Single-token recurrent step (T = 1, no gradient) of every (batch, head) stream: reads the FP32 cache (C, S), writes
// the updated one (the same buffers or others) and emits one output row.  The arithmetic is the token recurrence
// itself, in FP32.
//
// The step is state traffic (2 x 64 KiB read and written per stream at r = V = 128), so what counts is how many state
// loads are in flight and how few times the threads of a stream wait for one another.  A stream is a cluster of NS
// CTAs of 256 threads, each of which owns DP / NS rows of C and of S and holds them in REGISTERS for the whole step
// (thread = 4 columns of RW rows): no shared-memory copy of a state, every load issued before anything is waited for.
// With many streams NS is 1, and S waits in shared memory, each thread's elements in slots of its own (decode_split).
// The recurrence is arranged so that ONE exchange between the CTAs is enough.  With b = sigmoid(erase) k^,
//   delta_a = gamma (h_a - C_a . u^)                  needs row a of C only,
//   Cnew^T k^ = alpha (C^T k^) + u^ (delta . k^)      so its column sums run over the OLD C,
//   S^T(alpha e) and S^T(alpha chi), e = b - phi sb, chi = q^ - phi sq, phi = fs delta,
//                                                     are combinations of S^T(alpha b), S^T(alpha delta), S^T(alpha q^),
// so each CTA forms four partial column sums and three partial scalars from its own rows, the cluster adds them up
// through distributed shared memory, and the rows are updated in registers and stored.  What is per token and channel
// (norms, gates, conv) every warp works out for itself, four channels a lane: no block barrier for it.
// Upstream counterparts: _predictor_recurrent_kernel, _relative_recurrent_sources_kernel and the fused
// recurrent DPLR step (causallsso/ops/residual_frame/recurrent.py:33-98,188-327).
#pragma once
#include "sd_bf16.cuh"
#include "sd_common.cuh"
#include "sd_mixer.cuh"
#include "sd_token.cuh"

namespace sd {

struct DecodeParams {
    Geometry g;
    Operand u, h, q, k, v, er, wr, ld, gam;
    const float *Cin, *Sin;   // null: zero state
    float *C, *S;             // updated states; may be Cin / Sin (every CTA reads and writes its own rows only)
    void* y;
};

// The mixer glue of a cached single-token step, computed inside the decode kernel (k_decode_step<true>):
// q, k, v = SiLU(conv4) of the projection row against the carried three-token window, which is advanced in
// place (causallsso/model.py:146-164 at T = 1); log decay = -exp(A[h]) softplus(raw + bias) (model.py:383-390);
// geometry rate = sigmoid(raw + bias) (model.py:391-394).  The operands q, k, v, ld, gam of DecodeParams are
// then unused.
struct MixerDecode {
    const __nv_bfloat16* qkv;       // conv input of the token: [B] rows of D = 2 H r + H V channels (q | k | v)
    long long qkv_sb;               // elements between batch rows
    const float* conv_w;            // [D][4], tap 3 multiplies the current token
    __nv_bfloat16* conv_state;      // [B][D][3], oldest first; in/out
    const __nv_bfloat16* decay_raw; // [B][H*r]
    long long decay_sb;
    const float* log_rate;          // [H]
    const float* decay_bias;        // [H*r]
    const __nv_bfloat16* geom_raw;  // [B][H]
    long long geom_sb;
    const float* geom_bias;         // [H]
    // optional (norm_w != null): the sigmoid-gated RMSNorm of the output row (causallsso/ops/norm_gate.py:19-43)
    const float* norm_w;            // [V]
    float norm_eps;
    const __nv_bfloat16* gate;      // [B][H*V]
    long long gate_sb;
    // optional (decay_w / gate_w != null): the two small projections in front of the gates are taken here too,
    // raw = BF16(W hidden (+ bias)) with W [H*r][G] / [H*V][G] (causallsso/model.py:369-374); decay_raw / gate
    // above are then unused
    int G;
    const __nv_bfloat16 *decay_hidden, *decay_w;   // [B][G] (row stride dh_sb), [H*r][G]
    long long dh_sb;
    const __nv_bfloat16 *gate_hidden, *gate_w, *gate_b;   // [B][G], [H*V][G], [H*V] or null
    long long gh_sb;
    bool hid_vec;   // the two hidden rows are 8-byte aligned
};

__device__ __forceinline__ float warp_sum32(float v) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    return v;
}
// N sums over the warp at once: on return lane l holds the sum of v[l * N / 32] (N a power of two up to 32).  Each
// halving step sends half of the values across, so 8 sums take 9 shuffles instead of 40.
template <int N>
__device__ __forceinline__ float warp_sum_rows(float (&v)[N]) {
    const int lane = threadIdx.x & 31;
    int m = 16;
#pragma unroll
    for (int n = N / 2; n >= 1; n /= 2, m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < N / 2; ++i)
            if (i < n) {
                const float send = up ? v[i] : v[i + n];
                const float keep = up ? v[i + n] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
            }
    }
#pragma unroll
    for (; m > 0; m >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
    return v[0];
}

// Four consecutive FP32 elements of a row of `width`; zeros past it.
__device__ __forceinline__ float4 dec_load4(const float* row, int c0, int width, bool vec) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
        if (c0 < width) x = __ldcs(reinterpret_cast<const float4*>(row + c0));
    } else {
        if (c0 < width) x.x = row[c0];
        if (c0 + 1 < width) x.y = row[c0 + 1];
        if (c0 + 2 < width) x.z = row[c0 + 2];
        if (c0 + 3 < width) x.w = row[c0 + 3];
    }
    return x;
}
__device__ __forceinline__ void dec_store4(float* row, int c0, int width, bool vec, float4 x) {
    if (vec) {
        if (c0 < width) __stcs(reinterpret_cast<float4*>(row + c0), x);
    } else {
        if (c0 < width) row[c0] = x.x;
        if (c0 + 1 < width) row[c0 + 1] = x.y;
        if (c0 + 2 < width) row[c0 + 2] = x.z;
        if (c0 + 3 < width) row[c0 + 3] = x.w;
    }
}
// Four consecutive BF16 channels; `vec`: the row is 8-byte aligned and the width a multiple of four.
__device__ __forceinline__ void dec_bf4(const __nv_bfloat16* row, int c0, int width, bool vec, float (&x)[4]) {
    if (vec) {
        uint2 raw = make_uint2(0u, 0u);
        if (c0 < width) raw = *reinterpret_cast<const uint2*>(row + c0);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = c0 + e < width ? __bfloat162float(row[c0 + e]) : 0.f;
    }
}
// The value of channel a, held four channels a lane; a is uniform over the warp.
__device__ __forceinline__ float dec_channel(const float (&x)[4], int a) {
    const int e = a & 3;
    const float v = e == 0 ? x[0] : e == 1 ? x[1] : e == 2 ? x[2] : x[3];
    return __shfl_sync(0xffffffffu, v, a >> 2);
}

// One conv channel of the token: its carried window and taps, then the output, rounded to BF16 as the separate conv
// kernel stores it.
struct DecConv {
    __nv_bfloat16 window[3];   // oldest first; after `step` the advanced one
    float4 taps;
    __device__ __forceinline__ void load(const MixerDecode& m, int b, int D, int chn) {
        const __nv_bfloat16* st = m.conv_state + ((long long)b * D + chn) * 3;
        window[0] = st[0];
        window[1] = st[1];
        window[2] = st[2];
        taps = *reinterpret_cast<const float4*>(m.conv_w + (long long)chn * 4);
    }
    __device__ __forceinline__ float step(__nv_bfloat16 now) {
        const float z = taps.x * __bfloat162float(window[0]) + taps.y * __bfloat162float(window[1]) +
                        taps.z * __bfloat162float(window[2]) + taps.w * __bfloat162float(now);
        window[0] = window[1];
        window[1] = window[2];
        window[2] = now;
        return __bfloat162float(__float2bfloat16_rn(silu_f(z)));
    }
};

__device__ __forceinline__ void dec_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// FP32 value of the same shared-memory word in CTA `rank` of the cluster
__device__ __forceinline__ unsigned dec_remote(const void* p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(rank));
    return out;
}
__device__ __forceinline__ float dec_ld_remote(unsigned a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float2 dec_ld_remote2(unsigned a) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}

constexpr int DECODE_WARPS = 8;

// FULL: r = V = 128, every row aligned for the wide accesses, both states given.  Bounds and strides are then constants:
// the row loops are loads at immediate offsets, without a predicate or an address each, which is a third of the step
// (one CTA per stream: 55 -> 41 us at 768 streams; clusters of four: 6.6 -> 4.4 us at 8 streams).
template <bool MIXER, int NS, bool FULL>
__global__ void __launch_bounds__(DECODE_WARPS * 32, 2) k_decode_step(DecodeParams p, MixerDecode mix) {
    constexpr int WARPS = DECODE_WARPS, THREADS = WARPS * 32;
    constexpr int ROWS = DP / NS;            // state rows of this CTA
    constexpr int RW = ROWS / WARPS;         // ... of a warp
    constexpr int LPR = 32 / RW;             // lanes that hold a row's scalars after warp_sum_rows
    constexpr bool SSH = NS == 1;            // S in shared memory (each thread its own slots), not in registers
    constexpr int CONV_PER = (3 * DP + THREADS - 1) / THREADS;
    static_assert(RW >= 1 && THREADS >= 2 * DP, "at least one row per warp, one thread per two columns");
    __shared__ __align__(16) float s_part[WARPS][4][DP];       // per-warp column sums: C^T k^, S^T(alpha b | delta | q^)
    __shared__ __align__(16) float s_col[4][DP];               // ... of this CTA's rows (read by the cluster)
    __shared__ __align__(16) float s_own[3][ROWS];             // delta, alpha, output gate of this CTA's rows
    __shared__ __align__(16) float4 s_row[WARPS][RW];          // per-row factors of the column sums
    __shared__ float s_scw[WARPS][3], s_sc[3];                 // delta.delta, delta.u^, delta.k^
    __shared__ __align__(16) float s_all[7][DP];               // the sums over the cluster; delta, alpha, gate of every row
    __shared__ float s_sca[3];
    __shared__ __align__(16) float s_conv[MIXER ? 3 * DP : 4]; // q | k | v behind the conv

    int rank = 0;
    if (NS > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int s = blockIdx.x / NS, b = s / p.g.H, hh = s - b * p.g.H;
    const int r = FULL ? DP : p.g.r, V = FULL ? DP : p.g.V, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = lane * 4, row0 = rank * ROWS + warp * RW;
    const int my_row = row0 + lane / LPR;    // the row whose scalars this lane works out
    Chunk ch;
    ch.s = s; ch.c = 0; ch.b = b; ch.hh = hh; ch.t0 = 0; ch.nvalid = 1; ch.gi = s;
    ch.vm = 0ull; ch.rm = 0ull;

    // this warp's rows of both states, requested before anything else
    const bool vecC = FULL || ((r & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.Cin) | reinterpret_cast<uintptr_t>(p.C)) & 15) == 0);
    const bool vecS = FULL || ((V & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.Sin) | reinterpret_cast<uintptr_t>(p.S)) & 15) == 0);
    float4 Cv[RW], Sv[SSH ? 1 : RW];
#pragma unroll
    for (int j = 0; j < RW; ++j) {
        const int a = row0 + j;
        Cv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (FULL || (a < r && p.Cin != nullptr)) Cv[j] = dec_load4(p.Cin + ((long long)s * r + a) * r, c0, r, vecC);
    }
    extern __shared__ __align__(16) float4 s_state[];   // SSH: [RW][THREADS]
    if constexpr (SSH) {   // a thread reads only what it copied: no barrier
#pragma unroll
        for (int j = 0; j < RW; ++j) {
            const int a = row0 + j;
            const bool live = FULL || (a < r && c0 < V && p.Sin != nullptr);
            const float* row = p.Sin + ((long long)s * r + a) * V;
            if (vecS)
                cp16_zfill(s_state + j * THREADS + tid, live ? row + c0 : p.S, live);
            else
                s_state[j * THREADS + tid] = live ? dec_load4(row, c0, V, false) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        cp_commit();
    } else {
#pragma unroll
        for (int j = 0; j < RW; ++j) {
            const int a = row0 + j;
            Sv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (FULL || (a < r && p.Sin != nullptr)) Sv[j] = dec_load4(p.Sin + ((long long)s * r + a) * V, c0, V, vecS);
        }
    }
    auto state_s = [&](int j) {
        if constexpr (SSH) return s_state[j * THREADS + tid];
        else return Sv[j];
    };

    // the token's rows, four channels a lane
    const bool v4r = (r & 3) == 0, v4v = (V & 3) == 0;
    float u[4], k[4], q[4], bq[4], al[4] = {1.f, 1.f, 1.f, 1.f}, vv[4], wg[4], gamma, own_alpha = 1.f;
    const int D = 2 * p.g.H * r + p.g.H * V;
    const int live_v = FULL ? 4 : V - c0 < 4 ? (V - c0 < 0 ? 0 : V - c0) : 4;
    const bool fused_proj = MIXER && mix.decay_w != nullptr;
    // conv channels, one a thread: every CTA needs all of q and k for the norms
    DecConv conv[CONV_PER];
    auto channel = [&](int t) {   // slot t of q | k | v in s_conv -> conv channel, -1: none
        const int part = t / DP, c = t - part * DP;
        if (part > 2 || c >= (part == 2 ? V : r)) return -1;
        return part == 2 ? 2 * p.g.H * r + hh * V + c : part * p.g.H * r + hh * r + c;
    };
    uint2 wd[MIXER ? RW : 1], wgt[MIXER ? RW : 1];   // SSH: wgt after the first product, for want of registers
    if constexpr (MIXER) {
        // what the projection before this launch does not write is requested ahead of the wait for it: conv windows and
        // taps, and this CTA's rows of the two small projections (one row per warp and load)
#pragma unroll
        for (int n = 0; n < CONV_PER; ++n) {
            const int chn = channel(tid + n * THREADS);
            if (chn >= 0) conv[n].load(mix, b, D, chn);
        }
        const bool lg = fused_proj && c0 < mix.G;   // G is a multiple of 16
#pragma unroll
        for (int j = 0; j < RW; ++j) {
            const int a = row0 + j;
            wd[j] = wgt[j] = make_uint2(0u, 0u);
            if (lg && (FULL || a < r)) wd[j] = *reinterpret_cast<const uint2*>(mix.decay_w + (long long)(hh * r + a) * mix.G + c0);
            if (!SSH && lg && (FULL || a < V)) wgt[j] = *reinterpret_cast<const uint2*>(mix.gate_w + (long long)(hh * V + a) * mix.G + c0);
        }
        chain_wait();
        chain_release();
    }
    const float ha = FULL || my_row < r ? __bfloat162float(row_bf16(p.h, ch, 0)[my_row]) : 0.f;
    if constexpr (MIXER) {
#pragma unroll
        for (int n = 0; n < CONV_PER; ++n) {
            const int dst = tid + n * THREADS, chn = channel(dst);
            if (dst < 3 * DP) s_conv[dst] = chn >= 0 ? conv[n].step(mix.qkv[(long long)b * mix.qkv_sb + chn]) : 0.f;
        }
        if (fused_proj) {   // the two small projections
            float hdf[4], hgf[4], dd[RW], gg[RW];
            dec_bf4(mix.decay_hidden + (long long)b * mix.dh_sb, c0, mix.G, mix.hid_vec, hdf);
            dec_bf4(mix.gate_hidden + (long long)b * mix.gh_sb, c0, mix.G, mix.hid_vec, hgf);
            auto dot4 = [](uint2 w, const float (&x)[4]) {
                const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.x));
                const float2 c = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.y));
                return a.x * x[0] + a.y * x[1] + c.x * x[2] + c.y * x[3];
            };
#pragma unroll
            for (int j = 0; j < RW; ++j) dd[j] = dot4(wd[j], hdf);
            const float draw = warp_sum_rows<RW>(dd);
#pragma unroll
            for (int j = 0; j < RW; ++j) {
                const int a = row0 + j;
                if (SSH && c0 < mix.G && (FULL || a < V)) wgt[j] = *reinterpret_cast<const uint2*>(mix.gate_w + (long long)(hh * V + a) * mix.G + c0);
            }
#pragma unroll
            for (int j = 0; j < RW; ++j) gg[j] = dot4(wgt[j], hgf);
            const float graw = warp_sum_rows<RW>(gg);
            if (FULL || my_row < r) {
                const float z = __bfloat162float(__float2bfloat16_rn(draw)) + mix.decay_bias[hh * r + my_row];
                own_alpha = exp_ftz(-exp_ftz(mix.log_rate[hh]) * softplus_fast(z));
            }
            if (lane % LPR == 0) {
                const float bias = my_row < V && mix.gate_b != nullptr ? __bfloat162float(mix.gate_b[hh * V + my_row]) : 0.f;
                s_own[2][my_row - rank * ROWS] = __bfloat162float(__float2bfloat16_rn(graw + bias));
            }
        } else {
            const float rate = exp_ftz(mix.log_rate[hh]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (c0 + e < r) {
                    const int hc = hh * r + c0 + e;
                    const float z = __bfloat162float(mix.decay_raw[(long long)b * mix.decay_sb + hc]) + mix.decay_bias[hc];
                    al[e] = exp_ftz(-rate * softplus_fast(z));
                }
        }
        const float graw = __bfloat162float(mix.geom_raw[(long long)b * mix.geom_sb + hh]) + mix.geom_bias[hh];
        gamma = 1.f / (1.f + exp_ftz(-graw));
    } else {
        dec_bf4(row_bf16(p.k, ch, 0), c0, r, FULL || (p.k.vec && v4r), k);
        dec_bf4(row_bf16(p.q, ch, 0), c0, r, FULL || (p.q.vec && v4r), q);
        dec_bf4(row_bf16(p.v, ch, 0), c0, V, FULL || (p.v.vec && v4v), vv);
        const float4 l4 = dec_load4(row_f32(p.ld, ch, 0), c0, r, FULL || (p.ld.vec && v4r));
        al[0] = exp_ftz(l4.x); al[1] = exp_ftz(l4.y); al[2] = exp_ftz(l4.z); al[3] = exp_ftz(l4.w);
        gamma = *row_f32(p.gam, ch, 0);
    }
    dec_bf4(row_bf16(p.u, ch, 0), c0, r, FULL || (p.u.vec && v4r), u);
    dec_bf4(row_bf16(p.er, ch, 0), c0, r, FULL || (p.er.vec && v4r), bq);
    dec_bf4(row_bf16(p.wr, ch, 0), c0, V, FULL || (p.wr.vec && v4v), wg);
    if constexpr (MIXER) {
        __syncthreads();
        const float4 q4 = *reinterpret_cast<const float4*>(s_conv + c0), k4 = *reinterpret_cast<const float4*>(s_conv + DP + c0);
        const float4 v4 = *reinterpret_cast<const float4*>(s_conv + 2 * DP + c0);
        q[0] = q4.x; q[1] = q4.y; q[2] = q4.z; q[3] = q4.w;
        k[0] = k4.x; k[1] = k4.y; k[2] = k4.z; k[3] = k4.w;
        vv[0] = v4.x; vv[1] = v4.y; vv[2] = v4.z; vv[3] = v4.w;
    }
    // norms and the two dot products that only need them
    float sums[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        bq[e] = sigmoidf_(bq[e]) * k[e];
        sums[0] = fmaf(u[e], u[e], sums[0]);
        sums[1] = fmaf(k[e], k[e], sums[1]);
        sums[2] = fmaf(q[e], q[e], sums[2]);
        sums[3] = fmaf(u[e], bq[e], sums[3]);
        sums[4] = fmaf(u[e], q[e], sums[4]);
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) sums[n] = warp_sum32(sums[n]);
    const float rs_u = rsqrtf(sums[0] + 1e-24f), rs_k = rsqrtf(sums[1] + 1e-24f), rs_q = rsqrtf(sums[2] + 1e-24f);
    const float dot_ub = sums[3] * rs_u * rs_k, dot_uq = sums[4] * rs_u * rs_q;   // u^ . (sigma(e) k^),  u^ . q^
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        u[e] *= rs_u;
        k[e] *= rs_k;
        q[e] *= rs_q;
        bq[e] *= rs_k;
    }
    // residual of this warp's rows: one row per LPR lanes
    float delta;
    {
        float dots[RW];
#pragma unroll
        for (int j = 0; j < RW; ++j) dots[j] = Cv[j].x * u[0] + Cv[j].y * u[1] + Cv[j].z * u[2] + Cv[j].w * u[3];
        const float cu = warp_sum_rows<RW>(dots);
        delta = FULL || my_row < r ? gamma * (ha - cu) : 0.f;
        // the per-channel values of that row sit in lane row / 4
        const int src = my_row >> 2, el = my_row & 3;
        auto at_row = [&](const float (&x)[4]) {
            const float x0 = __shfl_sync(0xffffffffu, x[0], src), x1 = __shfl_sync(0xffffffffu, x[1], src);
            const float x2 = __shfl_sync(0xffffffffu, x[2], src), x3 = __shfl_sync(0xffffffffu, x[3], src);
            return el == 0 ? x0 : el == 1 ? x1 : el == 2 ? x2 : x3;
        };
        const float ua = at_row(u), ka = at_row(k), ba = at_row(bq), qa = at_row(q);
        if (!fused_proj) own_alpha = at_row(al);
        float sc[3] = {0.f, 0.f, 0.f};
        if (lane % LPR == 0) {
            s_row[warp][lane / LPR] = make_float4(ka, own_alpha * ba, own_alpha * delta, own_alpha * qa);
            s_own[0][my_row - rank * ROWS] = delta;
            s_own[1][my_row - rank * ROWS] = own_alpha;
            sc[0] = delta * delta;
            sc[1] = delta * ua;
            sc[2] = delta * ka;
        }
#pragma unroll
        for (int n = 0; n < 3; ++n)
#pragma unroll
            for (int m = 16; m >= LPR; m >>= 1) sc[n] += __shfl_xor_sync(0xffffffffu, sc[n], m);
        if (lane == 0) {
            s_scw[warp][0] = sc[0];
            s_scw[warp][1] = sc[1];
            s_scw[warp][2] = sc[2];
        }
    }
    __syncwarp();
    if constexpr (SSH) cp_wait<0>();
    {
        float part[4][4];
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[n][e] = 0.f;
#pragma unroll
        for (int j = 0; j < RW; ++j) {
            const float4 f = s_row[warp][j], sj = state_s(j);
            const float cv[4] = {Cv[j].x, Cv[j].y, Cv[j].z, Cv[j].w}, sv[4] = {sj.x, sj.y, sj.z, sj.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                part[0][e] = fmaf(cv[e], f.x, part[0][e]);
                part[1][e] = fmaf(sv[e], f.y, part[1][e]);
                part[2][e] = fmaf(sv[e], f.z, part[2][e]);
                part[3][e] = fmaf(sv[e], f.w, part[3][e]);
            }
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
            *reinterpret_cast<float4*>(&s_part[warp][n][c0]) = make_float4(part[n][0], part[n][1], part[n][2], part[n][3]);
    }
    __syncthreads();
    {   // sums over the warps, two columns of one of the four vectors a thread, then over the cluster
        const int n = tid >> 6, cc = (tid & 63) * 2;
        if (n < 4) {
            float2 t = make_float2(0.f, 0.f);
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const float2 x = *reinterpret_cast<const float2*>(&s_part[w][n][cc]);
                t.x += x.x;
                t.y += x.y;
            }
            *reinterpret_cast<float2*>((NS > 1 ? s_col[n] : s_all[n]) + cc) = t;
        }
        if (tid < 3) {
            float x = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) x += s_scw[w][tid];
            (NS > 1 ? s_sc : s_sca)[tid] = x;
        }
        if (NS > 1) {
            dec_cluster_sync();
            if (n < 4) {
                float2 t = make_float2(0.f, 0.f);
#pragma unroll
                for (int k2 = 0; k2 < NS; ++k2) {
                    const float2 x = dec_ld_remote2(dec_remote(&s_col[n][cc], k2));
                    t.x += x.x;
                    t.y += x.y;
                }
                *reinterpret_cast<float2*>(&s_all[n][cc]) = t;
            }
            if (tid < DP) {
                const int rk = tid / ROWS, jj = tid - rk * ROWS;
                s_all[4][tid] = dec_ld_remote(dec_remote(&s_own[0][jj], rk));
                if (fused_proj) {
                    s_all[5][tid] = dec_ld_remote(dec_remote(&s_own[1][jj], rk));
                    s_all[6][tid] = dec_ld_remote(dec_remote(&s_own[2][jj], rk));
                }
            } else if (tid < DP + 3) {
                float x = 0.f;
#pragma unroll
                for (int k2 = 0; k2 < NS; ++k2) x += dec_ld_remote(dec_remote(&s_sc[tid - DP], k2));
                s_sca[tid - DP] = x;
            }
        } else if (tid < DP) {
            s_all[4][tid] = s_own[0][tid];
            if (fused_proj) {
                s_all[5][tid] = s_own[1][tid];
                s_all[6][tid] = s_own[2][tid];
            }
        }
    }
    __syncthreads();
    // every CTA has read what it needs of its neighbours' shared memory once all have arrived here; the wait is at
    // the end of the kernel
    if (NS > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const float n2 = s_sca[0], fs = RHO * rsqrtf(RHO * RHO + n2), den = 1.f + fs * s_sca[1], sdk = s_sca[2];
    const float sb = dot_ub / den, sq = dot_uq / den;
    float d[4], w[4], y[4], gate[4], dchi = 0.f;
    {
        const float4 cc = *reinterpret_cast<const float4*>(&s_all[0][c0]), s1 = *reinterpret_cast<const float4*>(&s_all[1][c0]);
        const float4 s2 = *reinterpret_cast<const float4*>(&s_all[2][c0]), s3 = *reinterpret_cast<const float4*>(&s_all[3][c0]);
        const float4 dl = *reinterpret_cast<const float4*>(&s_all[4][c0]);
        const float ccf[4] = {cc.x, cc.y, cc.z, cc.w}, s1f[4] = {s1.x, s1.y, s1.z, s1.w}, s2f[4] = {s2.x, s2.y, s2.z, s2.w};
        const float s3f[4] = {s3.x, s3.y, s3.z, s3.w}, dlf[4] = {dl.x, dl.y, dl.z, dl.w};
        if (fused_proj) {
            const float4 a4 = *reinterpret_cast<const float4*>(&s_all[5][c0]), g4 = *reinterpret_cast<const float4*>(&s_all[6][c0]);
            al[0] = a4.x; al[1] = a4.y; al[2] = a4.z; al[3] = a4.w;
            gate[0] = g4.x; gate[1] = g4.y; gate[2] = g4.z; gate[3] = g4.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            d[e] = k[e] + fmaf(al[e], ccf[e], u[e] * sdk);   // zero past r: every factor is
            dchi = fmaf(d[e], q[e] - fs * dlf[e] * sq, dchi);
        }
        dchi = warp_sum32(dchi);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float fd = fs * s2f[e];
            w[e] = e < live_v ? sigmoidf_(wg[e]) * vv[e] - (s1f[e] - sb * fd) : 0.f;
            y[e] = (s3f[e] - sq * fd) + dchi * w[e];
        }
    }
#pragma unroll
    for (int j = 0; j < RW; ++j) {
        const int a = row0 + j;
        const float da = dec_channel(d, a), dl = s_own[0][warp * RW + j], aa = s_own[1][warp * RW + j];
        if (FULL || a < r) {
            const float4 cn = make_float4(fmaf(Cv[j].x, al[0], dl * u[0]), fmaf(Cv[j].y, al[1], dl * u[1]),
                                          fmaf(Cv[j].z, al[2], dl * u[2]), fmaf(Cv[j].w, al[3], dl * u[3]));
            const float4 sj = state_s(j);
            const float4 sn = make_float4(fmaf(aa, sj.x, da * w[0]), fmaf(aa, sj.y, da * w[1]),
                                          fmaf(aa, sj.z, da * w[2]), fmaf(aa, sj.w, da * w[3]));
            dec_store4(p.C + ((long long)s * r + a) * r, c0, r, vecC, cn);
            dec_store4(p.S + ((long long)s * r + a) * V, c0, V, vecS, sn);
        }
    }
    if (rank == 0) {
        if (warp == 0) {   // the output row
            float yv[4];   // rounded to BF16 as the operator returns it
#pragma unroll
            for (int e = 0; e < 4; ++e) yv[e] = e < live_v ? __bfloat162float(__float2bfloat16_rn(y[e])) : 0.f;
            if (MIXER && mix.norm_w != nullptr) {
                const float ss = warp_sum32(yv[0] * yv[0] + yv[1] * yv[1] + yv[2] * yv[2] + yv[3] * yv[3]);
                const float rstd = rsqrtf(ss / V + mix.norm_eps);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < live_v) {
                        const float g = fused_proj ? gate[e]
                                                   : __bfloat162float(mix.gate[(long long)b * mix.gate_sb + hh * V + c0 + e]);
                        yv[e] = yv[e] * rstd * mix.norm_w[c0 + e] * sigmoidf_(g);
                    }
            }
            __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.y) + (long long)s * V + c0;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (e < live_v) out[e] = __float2bfloat16_rn(yv[e]);
        }
        if (MIXER) {   // advance the conv windows: every thread of the cluster has read them before the exchange
#pragma unroll
            for (int n = 0; n < CONV_PER; ++n) {
                const int chn = channel(tid + n * THREADS);
                if (chn >= 0) {
                    __nv_bfloat16* st = mix.conv_state + ((long long)b * D + chn) * 3;
                    st[0] = conv[n].window[0];
                    st[1] = conv[n].window[1];
                    st[2] = conv[n].window[2];
                }
            }
        }
    }
    if (NS > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// CTAs per stream.  While a cluster of four per stream fits the device at two CTAs per SM (64 clusters do, 72 do not) the
// spread shortens every phase: 4.4 us a step at 8 streams and 6.0 us at 64, but 9.3 at 72.  Past that the redundant work of
// the cluster costs more than it hides, and a stream is one CTA of eight warps, two to an SM so that one's loads run
// under the other's arithmetic: S then waits in shared memory, since the registers of eight warps hold one state only.
// 7.9 us at 128 streams, 41 us at 768 (4.9 TB/s); one CTA of sixteen warps with both states in registers, one to an
// SM: 10.2 and 62 us; the same walking over the streams with the next states on their way: 69 us; the next CTA's
// states prefetched into L2: no gain.
inline int decode_split(int streams) { return streams <= 64 ? 4 : 1; }
constexpr size_t DECODE_STATE_BYTES = size_t(DP) * DP * sizeof(float);   // dynamic shared memory of the one-CTA form

}  // namespace sd
