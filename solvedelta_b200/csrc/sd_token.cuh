// Projections of a cached single-token step: y [M][N] = x [M][K] W^T (+ bias) for up to 32 rows, with the residual add
// and RMSNorm in front of it and SwiGLU behind it where the block has them.
//
// What bounds it: the weights, read once (15 MB for the fused projection of the 1024-wide model, 2.4 us at the measured
// HBM rate), and behind that the latency of one load, since a step is a chain of such launches.  So
// * two CTAs of eight warps per SM stay for the whole launch and walk over tiles of 16 columns (two groups of eight, a
//   quarter of K per warp) or, where that would leave SMs idle, of 8 columns (an eighth of K per warp); every lane keeps
//   the weight pieces of two steps (16 x 16 bytes) in flight, ahead of the products of the step before;
// * when the launch is chained to the kernel before it (programmatic dependent launch), the first two steps' requests go
//   out while that kernel still runs: only the activations wait for it;
// * the product runs on mma.sync m16n8k16 with the rows of x as the M side: the contraction index is permuted so that a
//   lane's 16-byte piece of a weight row is its B fragment of two instructions (k = 8 t + {0,1,2,3} and {4,5,6,7}), and
//   x, in shared memory, is read with the same permutation; an FMA per weight and row would bound it from 8 rows on;
// * up to sixteen rows the norm is taken by every CTA for itself on the way into shared memory, which removes a launch.
#pragma once
#include "sd_bf16.cuh"
#include "sd_common.cuh"
#include "sd_mixer.cuh"

namespace sd {

// A 16-byte load of data the kernel before may have written: coherent, and kept where it stands.
__device__ __forceinline__ uint4 load16_live(const __nv_bfloat16* p) {
    uint4 r;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}

constexpr int TOKEN_MAX_ROWS = 32;
constexpr int TOKEN_NORM_MAX_ROWS = 16;  // the fused norm: up to two rows per warp
constexpr int TOKEN_NORM_MAX_K = 2048;   // ... whose pieces sit in registers
constexpr size_t TOKEN_SMEM_MAX = 200 * 1024;   // of one CTA, beside the static part
constexpr int TOKEN_BATCH = 8;           // weight pieces per lane and step

struct TokenLinearParams {
    int M, N, K, swiglu;
    const __nv_bfloat16* x;
    long long x_stride;
    const __nv_bfloat16* W;      // [N][K]
    const __nv_bfloat16* bias;   // [N] or null
    __nv_bfloat16* y;
    long long y_stride;
    // fused residual add + RMSNorm (norm_w != null): the rows are RMSNorm(x + delta) * norm_w; the sum is stored
    const __nv_bfloat16* delta;  // rows x_stride apart, or null
    const float* norm_w;         // [K]
    float eps;
    __nv_bfloat16* sum;          // rows of K elements; unused without delta
};

// Row pitch of x in shared memory: 64 bytes off a multiple of 128, so that the eight 16-byte pieces that a quarter-warp
// reads (two rows, four consecutive pieces) fall into distinct banks.
__host__ __device__ constexpr int token_pitch(int K) { return (K + 63) / 64 * 64 + 32; }
inline size_t token_smem(int M, int K, bool norm) { return size_t(M) * token_pitch(K) * 2 + (norm ? size_t(K) * 4 : 0); }

// RG: groups of eight rows; CG: column groups of eight per CTA; NORM: 256-channel pieces of the widest row the fused norm
// takes (0: no norm).
template <int RG, int CG, int NORM>
__global__ void __launch_bounds__(256, RG <= 2 ? 2 : 1) k_token_linear(TokenLinearParams p) {
    constexpr int KS = 8 / CG;          // K slices
    constexpr int MT = (RG + 1) / 2;    // 16-row tiles
    static_assert(NORM == 0 || RG <= 2, "the fused norm takes up to two rows per warp");
    extern __shared__ __align__(16) unsigned char tok_smem[];
    const int pitch = token_pitch(p.K);
    __nv_bfloat16* s_x = reinterpret_cast<__nv_bfloat16*>(tok_smem);
    float* s_nw = reinterpret_cast<float*>(s_x + (size_t)p.M * pitch);
    __shared__ float s_red[2][8][RG * 8][9];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int cg = warp % CG, ks = warp / CG;
    const int outs = p.swiglu ? p.N / 2 : p.N;
    const int width = p.swiglu ? 8 : 8 * CG;   // output columns of a tile
    const int tiles = (outs + width - 1) / width;
    const int chunks = (p.K + 31) / 32, per = (chunks + KS - 1) / KS;
    const int begin = ks * per, end = begin + per < chunks ? begin + per : chunks;
    const int steps = (per + TOKEN_BATCH - 1) / TOKEN_BATCH;   // per tile, the same for every warp
    const int mine = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = mine * steps;

    auto request = [&](int item, uint4 (&wv)[TOKEN_BATCH]) {
        const int tile = blockIdx.x + item / steps * gridDim.x, base = begin + item % steps * TOKEN_BATCH;
        const int col = tile * width + (p.swiglu ? g : cg * 8 + g);
        const bool ok = item < total && col < outs;
        const __nv_bfloat16* w = p.W + (long long)(p.swiglu ? col + cg * outs : col) * p.K + t * 8;
#pragma unroll
        for (int i = 0; i < TOKEN_BATCH; ++i) {
            const int c = base + i;
            wv[i] = ok && c < end && c * 32 + t * 8 < p.K ? load16_pinned(w + c * 32) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    uint4 wa[TOKEN_BATCH], wb[TOKEN_BATCH];
    request(0, wa);
    request(1, wb);
    if constexpr (NORM > 0)
        for (int c = tid * 4; c < p.K; c += 1024) *reinterpret_cast<float4*>(s_nw + c) = *reinterpret_cast<const float4*>(p.norm_w + c);
    chain_wait();
    chain_release();

    if constexpr (NORM > 0) {
        // a warp takes every eighth row: sum, its mean square, the normalised row (the sum is rounded to BF16 first, as the separate
        // add stores it)
        __syncthreads();   // norm weights
#pragma unroll 1
        for (int m = warp; m < p.M; m += 8) {
            const __nv_bfloat16* x = p.x + m * p.x_stride;
            const __nv_bfloat16* d = p.delta != nullptr ? p.delta + m * p.x_stride : nullptr;
            uint4 xv[NORM], dv[NORM];
#pragma unroll
            for (int it = 0; it < NORM; ++it) {
                const int c0 = it * 256 + lane * 8;
                xv[it] = c0 < p.K ? load16_live(x + c0) : make_uint4(0u, 0u, 0u, 0u);
                dv[it] = c0 < p.K && d != nullptr ? load16_live(d + c0) : make_uint4(0u, 0u, 0u, 0u);
            }
            float ss = 0.f;
#pragma unroll
            for (int it = 0; it < NORM; ++it) {
                float a[8], b[8];
                norm_unpack8(xv[it], a);
                if (d != nullptr) {
                    norm_unpack8(dv[it], b);
                    __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&xv[it]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        o[e] = __floats2bfloat162_rn(a[2 * e] + b[2 * e], a[2 * e + 1] + b[2 * e + 1]);
                        const float2 f = __bfloat1622float2(o[e]);
                        a[2 * e] = f.x;
                        a[2 * e + 1] = f.y;
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) ss = fmaf(a[e], a[e], ss);
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
            const float rstd = rsqrtf(ss / p.K + p.eps);
#pragma unroll
            for (int it = 0; it < NORM; ++it) {
                const int c0 = it * 256 + lane * 8;
                if (c0 >= p.K) break;
                if (d != nullptr && blockIdx.x == 0) *reinterpret_cast<uint4*>(p.sum + (long long)m * p.K + c0) = xv[it];
                float a[8];
                norm_unpack8(xv[it], a);
                const float4 w0 = *reinterpret_cast<const float4*>(s_nw + c0), w1 = *reinterpret_cast<const float4*>(s_nw + c0 + 4);
                uint4 o;
                __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
                o2[0] = __floats2bfloat162_rn(a[0] * rstd * w0.x, a[1] * rstd * w0.y);
                o2[1] = __floats2bfloat162_rn(a[2] * rstd * w0.z, a[3] * rstd * w0.w);
                o2[2] = __floats2bfloat162_rn(a[4] * rstd * w1.x, a[5] * rstd * w1.y);
                o2[3] = __floats2bfloat162_rn(a[6] * rstd * w1.z, a[7] * rstd * w1.w);
                *reinterpret_cast<uint4*>(s_x + m * pitch + c0) = o;
            }
        }
    } else {
        const int pieces = p.K / 8;   // asynchronous copies: all of x in flight at once
        for (int idx = tid; idx < p.M * pieces; idx += 256) {
            const int m = idx / pieces, c0 = (idx - m * pieces) * 8;
            cp16(s_x + m * pitch + c0, p.x + m * p.x_stride + c0);
        }
        cp_commit();
        cp_wait<0>();
    }
    __syncthreads();

    float acc[MT][4];
    auto step = [&](int item, uint4 (&wv)[TOKEN_BATCH]) {
        const int st = item % steps, base = begin + st * TOKEN_BATCH;
        if (st == 0) {
#pragma unroll
            for (int a = 0; a < MT; ++a)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[a][e] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < TOKEN_BATCH; ++i) {
            const int k = (base + i) * 32 + t * 8;
            if (base + i < end) {   // warp-uniform; past K the weights are zero and x is not read
                uint4 xv[2 * MT];
#pragma unroll
                for (int rg = 0; rg < 2 * MT; ++rg) {
                    const int m = rg * 8 + g;
                    xv[rg] = rg < RG && m < p.M && k < p.K ? *reinterpret_cast<const uint4*>(s_x + m * pitch + k)
                                                           : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int a = 0; a < MT; ++a) {
                    const uint4 lo = xv[2 * a], hi = xv[2 * a + 1];
                    const uint32_t f0[4] = {lo.x, hi.x, lo.y, hi.y}, f1[4] = {lo.z, hi.z, lo.w, hi.w};
                    mma_bf16(acc[a], f0, wv[i].x, wv[i].y);
                    mma_bf16(acc[a], f1, wv[i].z, wv[i].w);
                }
            }
        }
        request(item + 2, wv);
        if (st != steps - 1) return;
        // last step of a tile: the K slices are added up through shared memory (two buffers in turn, so one barrier)
        const int tile_no = item / steps, buf = tile_no & 1;
#pragma unroll
        for (int a = 0; a < MT; ++a) {
            s_red[buf][warp][a * 16 + g][2 * t] = acc[a][0];
            s_red[buf][warp][a * 16 + g][2 * t + 1] = acc[a][1];
            if (2 * a + 1 < RG) {
                s_red[buf][warp][a * 16 + 8 + g][2 * t] = acc[a][2];
                s_red[buf][warp][a * 16 + 8 + g][2 * t + 1] = acc[a][3];
            }
        }
        __syncthreads();
        const int n0 = (blockIdx.x + tile_no * gridDim.x) * width;
        for (int idx = tid; idx < p.M * width; idx += 256) {
            const int m = idx / width, c = idx - m * width;
            if (n0 + c >= outs) continue;
            float v[CG];
#pragma unroll
            for (int j = 0; j < CG; ++j) {   // swiglu: both halves; otherwise only the group of column c is used
                v[j] = 0.f;
#pragma unroll
                for (int k = 0; k < KS; ++k) v[j] += s_red[buf][k * CG + j][m][c & 7];
            }
            float out = CG == 1 || c < 8 ? v[0] : v[CG - 1];
            if (p.bias != nullptr) out += __bfloat162float(p.bias[n0 + c]);
            if (p.swiglu) {
                // both halves rounded to BF16 first, as the separate projection stores them
                const float gate = __bfloat162float(__float2bfloat16_rn(out));
                const float up = v[CG - 1] + (p.bias != nullptr ? __bfloat162float(p.bias[n0 + c + outs]) : 0.f);
                out = silu_f(gate) * __bfloat162float(__float2bfloat16_rn(up));
            }
            p.y[m * p.y_stride + n0 + c] = __float2bfloat16_rn(out);
        }
    };
    for (int item = 0; item < total; item += 2) {
        step(item, wa);
        if (item + 1 < total) step(item + 1, wb);
    }
}

}  // namespace sd
