// The reverse chunk kernels of the fast chunks (sd_chunk_tc.cuh) on tcgen05; slow ones take their namesakes in
// sd_backward.cuh.  Operands are BF16 tiles of 64 channels (128-byte rows, 128-byte swizzle), which serve as K-major operands
// along their rows and as MN-major ones across them, so no panel is transposed.  Decay factors that vary along a row are left
// out of the contractions (G is referenced to the chunk start: rows carry exp(G), columns exp(-G)) and applied in the
// row passes, where the prefix row is read once.
#pragma once
#include "sd_backward.cuh"
#include "sd_chunk_tc.cuh"

namespace sd {

constexpr unsigned BF_TILE = CL * 128;    // [64 rows][64 channels]; a stack of two panels or a state has twice the rows

// byte offset of the 16-byte piece (8 channels) of a row in tiles TS bytes apart
template <unsigned TS>
__device__ __forceinline__ unsigned bf_off(int i, int piece) {
    return (piece >> 3) * TS + i * 128 + (((piece & 7) ^ (i & 7)) << 4);
}
// ... of four channels 4 lane ..
template <unsigned TS>
__device__ __forceinline__ unsigned bf_off4(int i, int lane) { return bf_off<TS>(i, lane >> 1) + ((lane & 1) << 3); }
__device__ __forceinline__ uint2 tile4(const unsigned char* sm, int i, int lane) {
    return *reinterpret_cast<const uint2*>(sm + bf_off4<BF_TILE>(i, lane));
}

// dense global panel or state -> tiles, asynchronously
template <int ROWS, unsigned TS>
__device__ __forceinline__ void async_tiles(unsigned char* sm, const bf16* g) {
#pragma unroll
    for (int k = 0; k < ROWS * 16 / NTHREADS; ++k) {
        const int idx = threadIdx.x + NTHREADS * k, i = idx >> 4, piece = idx & 15;
        cp16(sm + bf_off<TS>(i, piece), g + i * DP + piece * 8);
    }
}
__device__ __forceinline__ unsigned bf_idesc(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) | ((unsigned)(n >> 3) << 17) |
           ((128u >> 4) << 24);
}
__device__ __forceinline__ unsigned long long bf_desc(unsigned addr, unsigned lbo) { return tc_desc(addr, lbo, 1024) | (2ull << 61); }
// D[128][N] (+)= A B over K: an operand is K-major (tiles TS apart along the contraction) or MN-major (rows along the
// contraction, tiles TS apart across it)
template <int K, unsigned TSA, bool AMN, unsigned TSB, bool BMN>
__device__ __forceinline__ void mma_bf(unsigned d_tmem, unsigned a, unsigned b, int n, unsigned accumulate) {
    const unsigned id = bf_idesc(n, AMN, BMN);
    const unsigned long long da = bf_desc(a, AMN ? TSA : 16), db = bf_desc(b, BMN ? TSB : 16);
#pragma unroll
    for (int k = 0; k < K / 16; ++k)
        tb_mma_ss(d_tmem, da + (AMN ? k * 2048 : (k / 4) * TSA + (k % 4) * 32) / 16,
                  db + (BMN ? k * 2048 : (k / 4) * TSB + (k % 4) * 32) / 16, id, k > 0 ? 1u : accumulate);
}

// 16 accumulator columns of this thread's lane as two pieces of row i of a tiled panel
__device__ __forceinline__ void acc16_to_tiles(unsigned taddr, unsigned char* sm, int i, int piece) {
    float a[16];
    tc_ld16(taddr, a);
    tc_wait_ld();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = a[8 * h + e];
        *reinterpret_cast<uint4*>(sm + bf_off<BF_TILE>(i, piece + h)) = pack8_bf16(w);
    }
}

// Four channels of an output row [B,T,H,width], tokens `pitch` elements apart; exact zeros for a masked token
template <bool FAST, class CH>
__device__ __forceinline__ void store4_bf16(void* base, long long pitch, const Geometry& g, const CH& ch, int i, int c0,
                                            int width, const float (&x)[4]) {
    if (i >= ch.nvalid || c0 >= width) return;
    bf16* row = reinterpret_cast<bf16*>(base) + ((long long)ch.b * g.T + ch.t0 + i) * pitch + ch.hh * width + c0;
    uint2 raw = pack4_bf16(x);
    if (!ch.ok(i)) raw = make_uint2(0u, 0u);
    if (FAST || (width & 7) == 0) {
        *reinterpret_cast<uint2*>(row) = raw;
        return;
    }
    const unsigned short h[4] = {(unsigned short)raw.x, (unsigned short)(raw.x >> 16), (unsigned short)raw.y, (unsigned short)(raw.y >> 16)};
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (c0 + e < width) reinterpret_cast<unsigned short*>(row)[e] = h[e];
}

// ---------------------------------------------------------------------------
// k_exterior_pair_fast: the contractions of the exterior reverse step and the per-token reverse of the sources
// (k_exterior_pair_bwd).  With [dAqd; dAed] = tril / stril of [dy; dR] Z~^T:
//     [d chi; -d e] exp(-G) = [dy; dR] S^T + [dAqd; dAed] (d exp(-G))
//     ddp exp(G)            = [dAqd; dAed]^T [chi exp(G); -e exp(G)]            dDt = Z~ dS_end^T
// The stacked operands make it five contractions.  Shared memory (112 KB): [dy; dR] 32, Z~ 16, S 32, dS 32; then the stack
// [chi exp(G); -e exp(G)] in the first, the pair matrices and d exp(-G) in S, and the four results as BF16 panels where
// operands are dead.  What bounds it: the latency of a chunk's chain, two to an SM; the row pass is two fifths of it.  At
// 8 x 4096 tokens of 8 heads 430 us against 674 us of the block-centred kernel (one CTA per SM).
// Tensor memory: 0 the pair matrices, then dDt, then ddp; 128 [d chi; -d e].
constexpr unsigned XP_A = 0, XP_ZT = 32 * 1024, XP_S = 48 * 1024, XP_DS = 80 * 1024, XP_LAM = 112 * 1024;
constexpr unsigned XP_PAIR = XP_S, XP_DCOL = XP_S + 16 * 1024;                       // over S
constexpr unsigned XP_DCHI = XP_ZT, XP_DE = XP_DS + 16 * 1024, XP_DDT = XP_DS, XP_DDP = XP_A;
static_assert(XP_LAM + DP * 4 <= FAST_BAR_OFF, "tiles and table fit");

template <bool FAST, bool MASKED>
__device__ __forceinline__ void exterior_pair_fast(const BwdParams& p, const ChunkT<MASKED>& ch, FastCta& cta) {
    unsigned char* sm = cta.sm;
    const unsigned smem = tc_smem(sm);
    float* s_lam = reinterpret_cast<float*>(sm + XP_LAM);
    const int r = p.g.r, V = p.g.V, c0 = cta.lane * 4;
    int ph = 0;
    SD_PHASE_T(p.g, ch, ph);
    async_tiles<CL, 2 * BF_TILE>(sm + XP_A, bpanel_ptr(p.Dyf, ch.gi));
    async_tiles<CL, 2 * BF_TILE>(sm + XP_A + BF_TILE, bpanel_ptr(p.dR, ch.gi));
    async_tiles<CL, BF_TILE>(sm + XP_ZT, bpanel_ptr(p.Zt, ch.gi));
    cp_commit();
    async_tiles<DP, 2 * BF_TILE>(sm + XP_S, bstate_ptr(p.SCk, ch.gi));
    cp_commit();
    async_tiles<DP, 2 * BF_TILE>(sm + XP_DS, bstate_ptr(p.dSeCk, ch.gi));
    cp_commit();
    if (cta.tid < DP) s_lam[cta.tid] = p.Lam[ch.gi * DP + cta.tid];
    cp_wait<2>();
    cta.publish();
    if (cta.tid == 0) {
        tc_fence_after();
        mma_bf<DP, 2 * BF_TILE, false, BF_TILE, false>(cta.tmem, smem + XP_A, smem + XP_ZT, CL, 0u);
        tc_commit(cta.bar(0));
    }
    __syncwarp();
    SD_PHASE_T(p.g, ch, ph);
    // value side: dv = sigmoid(write) dR, d write_raw = dR v sigmoid'(write)
#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it) {
        const int i = cta.warp + 16 * it;
        float w[4], v[4], dr[4], dv[4];
        unpack4(load4_raw<FAST>(row_bf16(p.wr, ch, i), c0, V, p.wr.vec, ch.ok(i)), w);
        unpack4(load4_raw<FAST>(row_bf16(p.v, ch, i), c0, V, p.v.vec, ch.ok(i)), v);
        unpack4(*reinterpret_cast<const uint2*>(sm + XP_A + BF_TILE + bf_off4<2 * BF_TILE>(i, cta.lane)), dr);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float sw = sigmoidf_(w[e]);
            dv[e] = sw * dr[e];
            w[e] = dr[e] * v[e] * sw * (1.f - sw);
        }
        store4_bf16<FAST>(p.dv, p.pitch_v, p.g, ch, i, c0, V, dv);
        store4_bf16<FAST>(p.dwr, p.pitch_w, p.g, ch, i, c0, V, w);
    }
    cp_wait<1>();
    cta.publish();
    if (cta.tid == 32) {
        tc_fence_after();
        mma_bf<DP, 2 * BF_TILE, false, 2 * BF_TILE, false>(cta.tmem + 128, smem + XP_A, smem + XP_S, DP, 0u);
        tc_commit(cta.bar(1));
    }
    __syncwarp();
    SD_PHASE_T(p.g, ch, ph);
    cta.wait(0, 11);
    uint4 pair[2];   // this thread's 16 entries of a row of the stacked pair matrices, masked
    {
        float a[16];
        tc_ld16(cta.lanes() + 16 * cta.part, a);
        tc_wait_ld();
        const int i = (32 * cta.quarter + cta.lane) & (CL - 1), last = cta.quarter < 2 ? i : i - 1, j0 = 16 * cta.part;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = j0 + 8 * h + e <= last ? a[8 * h + e] : 0.f;
            pair[h] = pack8_bf16(w);
        }
    }
    cp_wait<0>();
    cta.publish();
    if (cta.tid == 64) {
        tc_fence_after();
        mma_bf<DP, BF_TILE, false, 2 * BF_TILE, false>(cta.tmem, smem + XP_ZT, smem + XP_DS, DP, 0u);
        tc_commit(cta.bar(2));
    }
    __syncwarp();
    {   // SdS[c] = sum_v S[c][v] dS_end[c][v]: four lanes per state row; odd rows take the pieces in the other order, so that
        // the eight lanes of an access touch all banks
        const int c = cta.tid >> 2, qt = cta.tid & 3;
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned off = bf_off<2 * BF_TILE>(c, 4 * (k ^ (c & 1)) + qt);
            float a[8], b[8];
            unpack8_bf16(*reinterpret_cast<const uint4*>(sm + XP_S + off), a);
            unpack8_bf16(*reinterpret_cast<const uint4*>(sm + XP_DS + off), b);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc = fmaf(a[e], b[e], acc);
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        if (qt == 0) p.SdS[ch.gi * DP + c] = acc;
    }
    cta.wait(1, 12);   // [dy; dR] and S are free of the second contraction
    __syncthreads();   // ... and S of the sums above
    async_tiles<CL, BF_TILE>(sm + XP_DCOL, bpanel_ptr(p.Dcol, ch.gi));
    cp_commit();
    async_tiles<CL, 2 * BF_TILE>(sm + XP_A, bpanel_ptr(p.Xg, ch.gi));
    async_tiles<CL, 2 * BF_TILE>(sm + XP_A + BF_TILE, bpanel_ptr(p.Ag, ch.gi));
    cp_commit();
    {
        const int i = 32 * cta.quarter + cta.lane;   // row of the stack, one tile of 64 tokens
        *reinterpret_cast<uint4*>(sm + XP_PAIR + bf_off<BF_TILE>(i, 2 * cta.part)) = pair[0];
        *reinterpret_cast<uint4*>(sm + XP_PAIR + bf_off<BF_TILE>(i, 2 * cta.part + 1)) = pair[1];
    }
    SD_PHASE_T(p.g, ch, ph);
    cta.wait(2, 13);
    const int row = 32 * cta.quarter + cta.lane;
    if (cta.quarter < 2) {   // dDt
#pragma unroll
        for (int h = 0; h < 2; ++h)
            acc16_to_tiles(cta.lanes() + 32 * cta.part + 16 * h, sm + XP_DDT, row, 4 * cta.part + 2 * h);
    }
    cp_wait<1>();
    cta.publish();
    if (cta.tid == 96) {
        tc_fence_after();
        mma_bf<CL, BF_TILE, false, BF_TILE, true>(cta.tmem + 128, smem + XP_PAIR, smem + XP_DCOL, DP, 1u);
        tc_commit(cta.bar(3));
    }
    __syncwarp();
    cp_wait<0>();
    cta.publish();
    if (cta.tid == 128) {
        tc_fence_after();
        mma_bf<DP, BF_TILE, true, 2 * BF_TILE, true>(cta.tmem, smem + XP_PAIR, smem + XP_A, DP, 0u);
        tc_commit(cta.bar(4));
    }
    __syncwarp();
    cta.wait(3, 14);
#pragma unroll
    for (int h = 0; h < 2; ++h)   // [d chi; -d e] exp(-G)
        acc16_to_tiles(cta.lanes() + 128 + 32 * cta.part + 16 * h, sm + (cta.quarter < 2 ? XP_DCHI : XP_DE), row & (CL - 1),
                       4 * cta.part + 2 * h);
    cta.wait(4, 15);
    if (cta.quarter < 2) {   // ddp exp(G)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            acc16_to_tiles(cta.lanes() + 32 * cta.part + 16 * h, sm + XP_DDP, row, 4 * cta.part + 2 * h);
    }
    tc_fence_before();
    __syncthreads();
    SD_PHASE_T(p.g, ch, ph);
    // ---- per-token reverse of the sources (sources_bwd_rows): every dot product of a row follows from ten sums ----
#pragma unroll 1
    for (int it = 0; it < FAST_PASSES; ++it) {
        const int i = cta.warp + 16 * it;
        const long long at = ch.gi * (CL * DP) + i * DP + c0;   // the same place in every panel
        const bool ok = ch.ok(i);
        const uint2 rk_ = load4_raw<FAST>(row_bf16(p.k, ch, i), c0, r, p.k.vec, ok);
        const uint2 rq_ = load4_raw<FAST>(row_bf16(p.q, ch, i), c0, r, p.q.vec, ok);
        const uint2 ru_ = load4_raw<FAST>(row_bf16(p.u, ch, i), c0, r, p.u.vec, ok);
        const uint2 re_ = load4_raw<FAST>(row_bf16(p.er, ch, i), c0, r, p.er.vec, ok);
        const float4 rg_ = ld_pinned16(p.Gp + at), rl_ = ld_pinned16(p.Delta + at), rd_ = ld_pinned16(p.Dprim + at);
        float dl[4], eg[4], ie[4], dd[4], xext[4];
        unpack4(rg_, eg);
        unpack4(rl_, dl);
        {
            float d[4], lam[4], ddt[4], dg[4];
            unpack4(rd_, d);
            unpack4(*reinterpret_cast<const float4*>(s_lam + c0), lam);
            unpack4(tile4(sm + XP_DDT, i, cta.lane), ddt);
            unpack4(tile4(sm + XP_DDP, i, cta.lane), dd);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ie[e] = exp_ftz(-eg[e]);
                eg[e] = exp_ftz(eg[e]);
                ddt[e] *= lam[e] * ie[e];
                dd[e] = fmaf(dd[e], ie[e], ddt[e]);
                xext[e] = ddt[e] * d[e];
                dg[e] = dd[e] * eg[e];
            }
            *reinterpret_cast<uint2*>(p.DG + at) = pack4_bf16(dg);
            *reinterpret_cast<uint2*>(p.Dd + at) = pack4_bf16(dd);
            *reinterpret_cast<uint2*>(p.Xext + at) = pack4_bf16(xext);
        }
        float k[4], q[4], u[4], se[4], dchi[4], de[4];
        unpack4(tile4(sm + XP_DCHI, i, cta.lane), dchi);
        unpack4(tile4(sm + XP_DE, i, cta.lane), de);
        unpack4(rk_, k);
        unpack4(rq_, q);
        unpack4(ru_, u);
        unpack4(re_, se);
        float s8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, s2[2] = {0.f, 0.f};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            se[e] = sigmoidf_(se[e]);
            dchi[e] *= eg[e];
            de[e] *= -eg[e];
            s8[0] = fmaf(k[e], k[e], s8[0]);
            s8[1] = fmaf(q[e], q[e], s8[1]);
            s8[2] = fmaf(u[e], u[e], s8[2]);
            s8[3] = fmaf(dl[e], dl[e], s8[3]);
            s8[4] = fmaf(u[e] * se[e], k[e], s8[4]);
            s8[5] = fmaf(u[e], q[e], s8[5]);
            s8[6] = fmaf(u[e], dl[e], s8[6]);
            s8[7] = fmaf(de[e], dl[e], s8[7]);
            s2[0] = fmaf(dchi[e], dl[e], s2[0]);
            s2[1] = fmaf(dchi[e], q[e], s2[1]);
        }
        row_sums32(s8);
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            s2[0] += __shfl_xor_sync(0xffffffffu, s2[0], m);
            s2[1] += __shfl_xor_sync(0xffffffffu, s2[1], m);
        }
        const float rk = rsqrtf(s8[0] + 1e-24f), rq = rsqrtf(s8[1] + 1e-24f), ru = rsqrtf(s8[2] + 1e-24f);
        const float n2 = RHO * RHO + s8[3], s = RHO * rsqrtf(n2);
        const float inv = 1.f / (1.f + s * ru * s8[6]);
        const float sb = ru * rk * s8[4] * inv, sq = ru * rq * s8[5] * inv;
        const float dsb = -s * s8[7] * inv, dsq = -s * s2[0] * inv;          // d(u^ . b) and d(u^ . q^)
        const float dden = -(dsb * sb + dsq * sq);
        const float coef = (dden * ru * s8[6] - sb * s8[7] - sq * s2[0]) * s / n2;   // (dphi . Delta) s / (rho^2 + |Delta|^2)
        const float dotq = rq * (s2[1] + dsq * ru * s8[5]);
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            k[e] *= rk; q[e] *= rq; u[e] *= ru;
            o[e] = (dchi[e] + dsq * u[e] - dotq * q[e]) * rq;
        }
        store4_bf16<FAST>(p.dq, p.pitch_q, p.g, ch, i, c0, r, o);
#pragma unroll
        for (int e = 0; e < 4; ++e)   // d(-d py + dd (d - k^)) with dd - py = exp(GL - G) dDt: the d terms collapse into xext
            o[e] = (q[e] - s * sq * dl[e]) * dchi[e] + (se[e] * k[e] - s * sb * dl[e]) * de[e] + xext[e] - dd[e] * k[e];
        *reinterpret_cast<uint2*>(p.dGPart + at) = pack4_bf16(o);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = s * (dden * u[e] - de[e] * sb - dchi[e] * sq) - coef * dl[e];
        *reinterpret_cast<uint2*>(p.dDelta + at) = pack4_bf16(o);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = dsb * se[e] * k[e] + dsq * q[e] + dden * s * dl[e];
        *reinterpret_cast<uint2*>(p.duPart + at) = pack4_bf16(o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            de[e] = fmaf(dsb, u[e], de[e]);   // d b
            o[e] = fmaf(se[e], de[e], dd[e]);
            de[e] *= k[e] * se[e] * (1.f - se[e]);
        }
        *reinterpret_cast<uint2*>(p.dkPart + at) = pack4_bf16(o);
        store4_bf16<FAST>(p.der, p.pitch_u, p.g, ch, i, c0, r, de);
    }
    SD_PHASE_T(p.g, ch, ph);
}

template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 2) k_exterior_pair_fast(BwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (leave_to_slow_kernel(p.Flags, FLAG_SLOW)) return;
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    exterior_pair_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}
// Both kinds of chunk in one launch, for calls that leave SMs empty anyway.
template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 1) k_exterior_pair_one(BwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (chunk_flags(p.Flags, blockIdx.x) & (FLAG_SLOW)) {
        chain_wait();
        chain_release();
        exterior_pair_blocks<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), fsm_raw);
        return;
    }
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    exterior_pair_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}

// ---------------------------------------------------------------------------
// FP32 accumulator columns 32 part .. of this warp's lanes (rows i) as pieces of an FP32 tiled panel
__device__ __forceinline__ void acc32_to_f32_tiles(const FastCta& cta, unsigned taddr, unsigned char* sm, int i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int col = 32 * cta.part + 16 * h;
        float a[16];
        tc_ld16(taddr + col, a);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(sm + f32_off<F32_TILE>(i, col + j)) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
    }
}

// ---------------------------------------------------------------------------
// k_primal_fast: reverse of the primal address and preparation of the dC scan (k_primal_bwd).  With DG = dd exp(G), Ucol =
// u^ exp(-G) and the stack [K^; DG]:
//     Aqk = tril(K^ Delta^T), dAqk = tril(DG Ucol^T)        t_u = exp(-G) (Aqk^T DG)
//     dk^ = dkPart + DG Ct + dAqk Delta                     dDelta_loc = dDelta + dAqk^T K^
//     P'' = (I+Lm)^-T dDelta_loc,  Q'' = (I+Lm)^-T Ubar,  Rneg = -gamma u^ exp(E)
// Shared memory (112 KB): the stack 32, Delta 16, the stacked pair matrices 16, Ucol then Ubar 16, Ct 32; the three results
// that leave FP32 take the stack, Delta with the pair matrices, and Ct; then the solve has its matrix in the stack's place
// and dDelta_loc in Ct's.  A warp takes four token rows in a row and requests all four before it uses one (391 -> 353 us
// against row by row).  At 8 x 4096 tokens of 8 heads 353 us against 559 us of the block-centred kernel.  Tensor memory: 0 and 64 the pair matrices, then t_u; 128 dk^, then dDelta.
constexpr unsigned PB_A = 0, PB_DL = 32 * 1024, PB_PP = 48 * 1024, PB_UC = 64 * 1024, PB_CT = 80 * 1024, PB_GAM = 112 * 1024;
constexpr unsigned PB_DK = PB_CT, PB_TU = PB_DL, PB_DD = PB_A, PB_RHS = PB_CT, PB_LM = PB_A;
static_assert(PB_GAM + CL * 4 <= FAST_BAR_OFF, "tiles and table fit");

template <bool FAST, bool MASKED>
__device__ __forceinline__ void primal_fast(const BwdParams& p, const ChunkT<MASKED>& ch, FastCta& cta) {
    unsigned char* sm = cta.sm;
    const unsigned smem = tc_smem(sm);
    float* s_gam = reinterpret_cast<float*>(sm + PB_GAM);
    const int r = p.g.r, c0 = cta.lane * 4;
    int ph = 0;
    SD_PHASE_T(p.g, ch, ph);
    async_tiles<CL, 2 * BF_TILE>(sm + PB_A + BF_TILE, bpanel_ptr(p.DG, ch.gi));
    cp_commit();
    async_tiles<DP, 2 * BF_TILE>(sm + PB_CT, bstate_ptr(p.CtCkB, ch.gi));
    cp_commit();
    load_gamma(p.gam, ch, s_gam);
    __syncthreads();
    uint2 ubar[FAST_PASSES], k_raw[FAST_PASSES];
    float rk[FAST_PASSES];
    const long long at0 = ch.gi * (CL * DP) + (4 * cta.warp) * DP + c0;   // rows 4 warp .. of every panel
    {   // k^ and Delta
        float4 dl[FAST_PASSES];
        const bf16* row = row_bf16(p.k, ch, 4 * cta.warp);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            k_raw[it] = load4_raw<FAST>(row + it * p.k.st, c0, r, p.k.vec, ch.ok(4 * cta.warp + it));
            dl[it] = ld_pinned16(p.Delta + at0 + it * DP);
        }
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4];
            unpack4(k_raw[it], x);
            rk[it] = fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3])));
        }
        row_sums32(rk);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = 4 * cta.warp + it;
            float x[4];
            unpack4(dl[it], x);
            *reinterpret_cast<uint2*>(sm + PB_DL + bf_off4<BF_TILE>(i, cta.lane)) = pack4_bf16(x);
            rk[it] = rsqrtf(rk[it] + 1e-24f);
            unpack4(k_raw[it], x);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] *= rk[it];
            const uint2 kh = pack4_bf16(x);
            *reinterpret_cast<uint2*>(sm + PB_A + bf_off4<2 * BF_TILE>(i, cta.lane)) = kh;
            *reinterpret_cast<uint2*>(p.Khat + at0 + it * DP) = kh;
        }
    }
    {   // u^: Ucol, Ubar, Rneg
        uint2 u[FAST_PASSES];
        float4 G[FAST_PASSES + 1];
        const bf16* row = row_bf16(p.u, ch, 4 * cta.warp);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            u[it] = load4_raw<FAST>(row + it * p.u.st, c0, r, p.u.vec, ch.ok(4 * cta.warp + it));
            G[it + 1] = ld_pinned16(p.Gp + at0 + it * DP);
        }
        G[0] = cta.warp > 0 ? ld_pinned16(p.Gp + at0 - DP) : make_float4(0.f, 0.f, 0.f, 0.f);   // E of a row is G of the one before
        float lam[4], ss[4];
        unpack4(*reinterpret_cast<const float4*>(p.Lam + ch.gi * DP + c0), lam);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4];
            unpack4(u[it], x);
            ss[it] = fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3])));
        }
        row_sums32(ss);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = 4 * cta.warp + it;
            float x[4], g[4], E[4], o[4];
            unpack4(u[it], x);
            unpack4(G[it + 1], g);
            unpack4(G[it], E);
            const float ru = rsqrtf(ss[it] + 1e-24f), gm = s_gam[i];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] *= ru;
                g[e] = x[e] * exp_ftz(-g[e]);
                o[e] = -gm * x[e] * exp_ftz(E[e]);
            }
            *reinterpret_cast<uint2*>(p.Rneg + at0 + it * DP) = pack4_bf16(o);
            *reinterpret_cast<uint2*>(sm + PB_UC + bf_off4<BF_TILE>(i, cta.lane)) = pack4_bf16(g);
#pragma unroll
            for (int e = 0; e < 4; ++e) g[e] *= lam[e];
            ubar[it] = pack4_bf16(g);
        }
    }
    cp_wait<1>();
    cta.publish();
    SD_PHASE_T(p.g, ch, ph);
    if (cta.tid == 0) {
        tc_fence_after();
        mma_bf<DP, 2 * BF_TILE, false, BF_TILE, false>(cta.tmem, smem + PB_A, smem + PB_DL, CL, 0u);
        mma_bf<DP, 2 * BF_TILE, false, BF_TILE, false>(cta.tmem + CL, smem + PB_A, smem + PB_UC, CL, 0u);
        tc_commit(cta.bar(0));
    }
    __syncwarp();
    cp_wait<0>();
    cta.publish();
    if (cta.tid == 32) {
        tc_fence_after();
        mma_bf<DP, 2 * BF_TILE, false, 2 * BF_TILE, true>(cta.tmem + 128, smem + PB_A, smem + PB_CT, DP, 0u);   // lanes 64 ..: DG Ct
    }
    __syncwarp();
    cta.wait(0, 11);
    const int row = 32 * cta.quarter + cta.lane;
    {   // lanes 0 .. 63: Aqk, lanes 64 .. 127: dAqk
        float a[16];
        tc_ld16(cta.lanes() + (cta.quarter < 2 ? 0 : CL) + 16 * cta.part, a);
        tc_wait_ld();
        const int i = row & (CL - 1), j0 = 16 * cta.part;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = j0 + 8 * h + e <= i ? a[8 * h + e] : 0.f;
            *reinterpret_cast<uint4*>(sm + PB_PP + bf_off<BF_TILE>(row, 2 * cta.part + h)) = pack8_bf16(w);
        }
    }
#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it)   // Ucol is free
        *reinterpret_cast<uint2*>(sm + PB_UC + bf_off4<BF_TILE>(4 * cta.warp + it, cta.lane)) = ubar[it];
    cta.publish();
    if (cta.tid == 32) {   // the thread that issued DG Ct: the sum goes on in order
        tc_fence_after();
        mma_bf<CL, BF_TILE, false, BF_TILE, true>(cta.tmem + 128, smem + PB_PP, smem + PB_DL, DP, 1u);   // + dAqk Delta
        tc_commit(cta.bar(2));
        mma_bf<CL, BF_TILE, true, 2 * BF_TILE, true>(cta.tmem, smem + PB_PP, smem + PB_A + BF_TILE, DP, 0u);   // Aqk^T DG
        tc_commit(cta.bar(3));
    }
    __syncwarp();
    SD_PHASE_T(p.g, ch, ph);
    cta.wait(2, 12);
    if (cta.quarter >= 2) acc32_to_f32_tiles(cta, cta.lanes() + 128, sm + PB_DK, row - CL);
    tc_fence_before();
    __syncthreads();
    if (cta.tid == 96) {
        tc_fence_after();
        mma_bf<CL, BF_TILE, true, 2 * BF_TILE, true>(cta.tmem + 128, smem + PB_PP + BF_TILE, smem + PB_A, DP, 0u);   // dAqk^T K^
        tc_commit(cta.bar(4));
    }
    __syncwarp();
    cta.wait(3, 13);
    cta.wait(4, 14);   // the operands are free: t_u takes the place of Delta and the pair matrices, dDelta that of the stack
    if (cta.quarter < 2) {
        acc32_to_f32_tiles(cta, cta.lanes(), sm + PB_TU, row);
        acc32_to_f32_tiles(cta, cta.lanes() + 128, sm + PB_DD, row);
    }
    __syncthreads();
    SD_PHASE_T(p.g, ch, ph);
    const auto piece = [&](unsigned base, int i) {
        return reinterpret_cast<const float4*>(sm + base + (cta.lane >> 3) * F32_TILE + i * 128 + (((cta.lane & 7) ^ (i & 7)) << 4));
    };
    uint2 rhs[FAST_PASSES];
    {   // dk^ and its norm reverse; a row of the solve's right-hand sides is only packed here, its place is still in use
        uint2 dkp[FAST_PASSES];
        float dot[FAST_PASSES];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            dkp[it] = ld_pinned8(p.dkPart + at0 + it * DP, true);
            rhs[it] = ld_pinned8(p.dDelta + at0 + it * DP, true);
        }
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4], y[4], k[4];
            unpack4(dkp[it], x);
            unpack4(*piece(PB_DK, 4 * cta.warp + it), y);
            unpack4(k_raw[it], k);
            dot[it] = fmaf(k[0], y[0] + x[0], fmaf(k[1], y[1] + x[1], fmaf(k[2], y[2] + x[2], k[3] * (y[3] + x[3]))));
        }
        row_sums32(dot);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = 4 * cta.warp + it;
            float x[4], y[4], k[4];
            unpack4(dkp[it], x);
            unpack4(*piece(PB_DK, i), y);
            unpack4(k_raw[it], k);
            const float along = dot[it] * rk[it] * rk[it];
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = (y[e] + x[e] - along * k[e]) * rk[it];
            store4_bf16<FAST>(p.dk, p.pitch_q, p.g, ch, i, c0, r, y);
            unpack4(rhs[it], x);
            unpack4(*piece(PB_DD, i), y);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] += x[e];
            rhs[it] = pack4_bf16(y);
        }
    }
    float4 N[2];   // (gamma N)^T, the matrix of the solve: two pieces a thread, as g2s_mat_transposed takes them
    {
        float4 G[FAST_PASSES];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) G[it] = ld_pinned16(p.Gp + at0 + it * DP);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int idx = cta.tid + NTHREADS * k;
            N[k] = ld_pinned16(mat_ptr(p.Npair, ch.gi) + (idx & (CL - 1)) * CL + ((idx >> 6) << 2));
        }
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4], y[4];
            unpack4(G[it], x);
            unpack4(*piece(PB_TU, 4 * cta.warp + it), y);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] *= exp_ftz(-x[e]);
            *reinterpret_cast<uint2*>(p.Tu + at0 + it * DP) = pack4_bf16(y);
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it)
        *reinterpret_cast<uint2*>(sm + PB_RHS + bf_off4<BF_TILE>(4 * cta.warp + it, cta.lane)) = rhs[it];
    float* s_lm = reinterpret_cast<float*>(sm + PB_LM);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int idx = cta.tid + NTHREADS * k, i = idx & (CL - 1);
        float x[4];
        unpack4(N[k], x);
#pragma unroll
        for (int e = 0; e < 4; ++e) s_lm[(((idx >> 6) << 2) + e) * LDA + i] = s_gam[i] * x[e];
    }
    __syncthreads();
    SD_PHASE_T(p.g, ch, ph);
    const int panel = cta.warp >> 3, cw = cta.warp & 7;
    unsigned char* tile = sm + (panel == 0 ? PB_RHS : PB_UC) + (cw >> 2) * BF_TILE;
    const int piece0 = (cw & 3) * 2;
    trisolve_blocked<true>(s_lm, 1.f, TileBF16{tile, piece0});
    SD_PHASE_T(p.g, ch, ph);
    bf16* out = (panel == 0 ? bpanel_ptr(p.Ppp, ch.gi) : bpanel_ptr(p.Qpp, ch.gi)) + 16 * cw;
#pragma unroll
    for (int it = 0; it < CL / 16; ++it) {   // 32 bytes of a row per lane pair
        const int i = it * 16 + (cta.lane >> 1), h = cta.lane & 1;
        *reinterpret_cast<uint4*>(out + i * DP + 8 * h) = *reinterpret_cast<const uint4*>(tile + i * 128 + (((piece0 + h) ^ (i & 7)) << 4));
    }
    SD_PHASE_T(p.g, ch, ph);
}

template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 2) k_primal_fast(BwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (leave_to_slow_kernel(p.Flags, FLAG_SLOW)) return;
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    primal_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}
// Both kinds of chunk in one launch, for calls that leave SMs empty anyway.
template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 1) k_primal_one(BwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (chunk_flags(p.Flags, blockIdx.x) & (FLAG_SLOW)) {
        chain_wait();
        chain_release();
        primal_blocks<FAST, MASKED, false>(p, chunk_of<MASKED>(p.g, blockIdx.x), fsm_raw);
        return;
    }
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    primal_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}

// ---------------------------------------------------------------------------
// k_predictor_close_fast: the end of the reverse pass (k_predictor_close_bwd).  With P = stril(dR Delta^T), Ucol = u^ exp(-G)
// and Rneg = -gamma u^ exp(E):
//     dUbar = Delta dC_end^T,   W = -gamma (dR Ct^T + P Ucol)  (= dU~ + t_i exp(-E)),   t_j = exp(-G) (P^T Rneg)
//     dgamma = (dR . Delta) / gamma   since Delta = gamma (h - U~ Ct - stril(N) Delta): no contraction, and neither h nor N
// (a chunk with a vanishing gamma takes the slow kernel, which evaluates the residual).  A warp takes four token rows in a
// row, last first, so that the suffix sums of d log_decay need one exchange between the warps.
// Shared memory (112 KB): Delta, then P, 16; dR 16; Ct 32, then W and t_j; dC 32, then Rneg and dUbar; Ucol 16, then the
// warps' sums.  At 8 x 4096 tokens of 8 heads 325 us against 635 us of the block-centred kernel, which evaluates the residual
// and three FP32 panels for the sums.  Tensor memory: 0 P, then W; 128 dUbar, then t_j; 0 again keeps what the row pass leaves for the end.
constexpr unsigned PC_DL = 0, PC_DR = 16 * 1024, PC_CT = 32 * 1024, PC_DC = 64 * 1024, PC_UC = 96 * 1024, PC_GAM = 112 * 1024;
constexpr unsigned PC_P = PC_DL, PC_W = PC_CT, PC_TJ = PC_CT + 16 * 1024, PC_RN = PC_DC, PC_DUB = PC_DC + 16 * 1024, PC_TOT = PC_UC;
constexpr unsigned PC_CDC = PC_GAM + CL * 4;
static_assert(PC_CDC + DP * 4 <= FAST_BAR_OFF, "tiles and tables fit");

template <bool FAST, bool MASKED>
__device__ __forceinline__ void predictor_close_fast(const BwdParams& p, const ChunkT<MASKED>& ch, FastCta& cta) {
    unsigned char* sm = cta.sm;
    const unsigned smem = tc_smem(sm);
    float *s_gam = reinterpret_cast<float*>(sm + PC_GAM), *s_cdc = reinterpret_cast<float*>(sm + PC_CDC);
    const int r = p.g.r, c0 = cta.lane * 4;
    int ph = 0;
    SD_PHASE_T(p.g, ch, ph);
    async_tiles<CL, BF_TILE>(sm + PC_DR, bpanel_ptr(p.dRr, ch.gi));
    cp_commit();
    async_tiles<DP, 2 * BF_TILE>(sm + PC_DC, bstate_ptr(p.dCeCk, ch.gi));
    async_tiles<DP, 2 * BF_TILE>(sm + PC_CT, bstate_ptr(p.CtCkB, ch.gi));
    cp_commit();
    load_gamma(p.gam, ch, s_gam);
    const long long at0 = ch.gi * (CL * DP) + (4 * cta.warp) * DP + c0;   // rows 4 warp .. of every panel
    {
        uint2 u[FAST_PASSES];
        float4 G[FAST_PASSES], dl[FAST_PASSES];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = 4 * cta.warp + it;
            dl[it] = ld_pinned16(p.Delta + at0 + it * DP);
            u[it] = load4_raw<FAST>(row_bf16(p.u, ch, i), c0, r, p.u.vec, ch.ok(i));
            G[it] = ld_pinned16(p.Gp + at0 + it * DP);
        }
        float ss[4];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4];
            unpack4(dl[it], x);
            *reinterpret_cast<uint2*>(sm + PC_DL + bf_off4<BF_TILE>(4 * cta.warp + it, cta.lane)) = pack4_bf16(x);
            unpack4(u[it], x);
            ss[it] = fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3])));
        }
        row_sums32(ss);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4], g[4];
            unpack4(u[it], x);
            unpack4(G[it], g);
            const float ru = rsqrtf(ss[it] + 1e-24f);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] *= ru * exp_ftz(-g[e]);
            *reinterpret_cast<uint2*>(sm + PC_UC + bf_off4<BF_TILE>(4 * cta.warp + it, cta.lane)) = pack4_bf16(x);
        }
        cp_wait<1>();
        cta.publish();
        if (cta.tid == 0) {
            tc_fence_after();
            mma_bf<DP, BF_TILE, false, BF_TILE, false>(cta.tmem, smem + PC_DR, smem + PC_DL, CL, 0u);
            tc_commit(cta.bar(0));
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {   // dgamma
            float x[4], y[4];
            unpack4(dl[it], x);
            unpack4(tile4(sm + PC_DR, 4 * cta.warp + it, cta.lane), y);
            ss[it] = fmaf(x[0], y[0], fmaf(x[1], y[1], fmaf(x[2], y[2], x[3] * y[3])));
        }
        row_sums32(ss);
        if (cta.lane < FAST_PASSES) {
            const int i = 4 * cta.warp + cta.lane;
            const float s = cta.lane == 0 ? ss[0] : cta.lane == 1 ? ss[1] : cta.lane == 2 ? ss[2] : ss[3];
            if (i < ch.nvalid)
                p.dgam[((long long)ch.b * p.g.T + ch.t0 + i) * p.g.H + ch.hh] = ch.ok(i) ? s / s_gam[i] : 0.f;
        }
    }
    SD_PHASE_T(p.g, ch, ph);
    cp_wait<0>();
    cta.publish();
    if (cta.tid == 32) {
        tc_fence_after();
        mma_bf<DP, BF_TILE, false, 2 * BF_TILE, false>(cta.tmem + 128, smem + PC_DL, smem + PC_DC, DP, 0u);
        tc_commit(cta.bar(1));
    }
    __syncwarp();
    {   // CdC[c] = sum_a Ct[c][a] dCt_end[c][a], as SdS in exterior_pair_fast
        const int c = cta.tid >> 2, qt = cta.tid & 3;
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned off = bf_off<2 * BF_TILE>(c, 4 * (k ^ (c & 1)) + qt);
            float a[8], b[8];
            unpack8_bf16(*reinterpret_cast<const uint4*>(sm + PC_CT + off), a);
            unpack8_bf16(*reinterpret_cast<const uint4*>(sm + PC_DC + off), b);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc = fmaf(a[e], b[e], acc);
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        if (qt == 0) s_cdc[c] = p.Lam[ch.gi * DP + c] * (p.SdS[ch.gi * DP + c] + acc);
    }
    cta.wait(0, 11);
    const int row = 32 * cta.quarter + cta.lane;
    uint4 pair[2];
    if (cta.quarter < 2) {   // P, strictly lower
        float a[16];
        tc_ld16(cta.lanes() + 16 * cta.part, a);
        tc_wait_ld();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = 16 * cta.part + 8 * h + e < row ? a[8 * h + e] : 0.f;
            pair[h] = pack8_bf16(w);
        }
    }
    tc_fence_before();
    __syncthreads();   // P is read, CdC is done
    if (cta.tid == 64) {
        tc_fence_after();
        mma_bf<DP, BF_TILE, false, 2 * BF_TILE, false>(cta.tmem, smem + PC_DR, smem + PC_CT, DP, 0u);
    }
    __syncwarp();
    cta.wait(1, 12);   // Delta and dC are free
    async_tiles<CL, BF_TILE>(sm + PC_RN, bpanel_ptr(p.Rneg, ch.gi));
    cp_commit();
    if (cta.quarter < 2) {
        *reinterpret_cast<uint4*>(sm + PC_P + bf_off<BF_TILE>(row, 2 * cta.part)) = pair[0];
        *reinterpret_cast<uint4*>(sm + PC_P + bf_off<BF_TILE>(row, 2 * cta.part + 1)) = pair[1];
#pragma unroll
        for (int h = 0; h < 2; ++h)   // dUbar
            acc16_to_tiles(cta.lanes() + 128 + 32 * cta.part + 16 * h, sm + PC_DUB, row, 4 * cta.part + 2 * h);
    }
    cp_wait<0>();
    cta.publish();
    if (cta.tid == 64) {   // the thread that issued dR Ct^T: the sum goes on in order
        tc_fence_after();
        mma_bf<CL, BF_TILE, false, BF_TILE, true>(cta.tmem, smem + PC_P, smem + PC_UC, DP, 1u);
        tc_commit(cta.bar(2));
        mma_bf<CL, BF_TILE, true, BF_TILE, true>(cta.tmem + 128, smem + PC_P, smem + PC_RN, DP, 0u);
        tc_commit(cta.bar(3));
    }
    __syncwarp();
    SD_PHASE_T(p.g, ch, ph);
    cta.wait(2, 13);
    if (cta.quarter < 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            acc16_to_tiles(cta.lanes() + 32 * cta.part + 16 * h, sm + PC_W, row, 4 * cta.part + 2 * h);
    }
    cta.wait(3, 14);
    if (cta.quarter < 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            acc16_to_tiles(cta.lanes() + 128 + 32 * cta.part + 16 * h, sm + PC_TJ, row, 4 * cta.part + 2 * h);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    SD_PHASE_T(p.g, ch, ph);
    float* s_tot = reinterpret_cast<float*>(sm + PC_TOT);   // [16 warps][DP] sums of dG
    float* s_x = s_tot + 16 * DP;                            // ... of X
    {
        float lam[4], run[4] = {0.f, 0.f, 0.f, 0.f}, X[4] = {0.f, 0.f, 0.f, 0.f};
        unpack4(*reinterpret_cast<const float4*>(p.Lam + ch.gi * DP + c0), lam);
#pragma unroll 1
        for (int it = FAST_PASSES - 1; it >= 0; --it) {
            const int i = 4 * cta.warp + it;
            const long long at = at0 + it * DP;
            const uint2 ru_ = load4_raw<FAST>(row_bf16(p.u, ch, i), c0, r, p.u.vec, ch.ok(i));
            const float4 rg_ = ld_pinned16(p.Gp + at), re_ = ld_pinned16(p.Gp + (i > 0 ? at - DP : at));
            const uint2 r1_ = ld_pinned8(p.duPart + at, true), r2_ = ld_pinned8(p.Tu + at, true);
            const uint2 r3_ = ld_pinned8(p.dGPart + at, true), r4_ = ld_pinned8(p.Xext + at, true);
            float u[4], ie[4], eE[4], duh[4], w[4], tj[4], dub[4], tu[4];
            unpack4(ru_, u);
            unpack4(rg_, ie);
            unpack4(re_, eE);
            unpack4(r1_, duh);
            unpack4(r2_, tu);
            unpack4(tile4(sm + PC_W, i, cta.lane), w);
            unpack4(tile4(sm + PC_TJ, i, cta.lane), tj);
            unpack4(tile4(sm + PC_DUB, i, cta.lane), dub);
            const float gm = s_gam[i];
            float ss[2] = {0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ie[e] = exp_ftz(-ie[e]);
                w[e] *= -gm * (i > 0 ? exp_ftz(eE[e]) : 1.f);   // (dU~ + t_i exp(-E)) exp(E)
                tj[e] *= ie[e];
                dub[e] *= lam[e] * ie[e];
                duh[e] += tu[e] + dub[e] + w[e] + tj[e];
                ss[0] = fmaf(u[e], u[e], ss[0]);
                ss[1] = fmaf(u[e], duh[e], ss[1]);
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) {
                ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], m);
                ss[1] += __shfl_xor_sync(0xffffffffu, ss[1], m);
            }
            const float rs = rsqrtf(ss[0] + 1e-24f), dot = ss[1] * rs * rs;
            float o[4], dgp[4], xe[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = (duh[e] - dot * u[e]) * rs;
            store4_bf16<FAST>(p.du, p.pitch_u, p.g, ch, i, c0, r, o);
            unpack4(tile4(sm + PC_DR, i, cta.lane), o);
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] *= gm;
            store4_bf16<FAST>(p.dh, p.pitch_u, p.g, ch, i, c0, r, o);
            unpack4(r3_, dgp);
            unpack4(r4_, xe);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                u[e] *= rs;
                const float dE = u[e] * w[e], x = xe[e] + dub[e] * u[e];
                X[e] += x;
                run[e] += dgp[e] - u[e] * tu[e] - x - u[e] * tj[e] + dE;   // dG, summed from the warp's last row on
                o[e] = run[e] - dE;
            }
            tc_st4(cta.lanes() + 16 * cta.part + 4 * it, o);
        }
        *reinterpret_cast<float4*>(s_tot + cta.warp * DP + c0) = pack4(run);
        *reinterpret_cast<float4*>(s_x + cta.warp * DP + c0) = pack4(X);
        tc_wait_st();
    }
    __syncthreads();
    SD_PHASE_T(p.g, ch, ph);
    if (cta.tid < DP) {   // end-of-chunk terms, then the sums of later warps
        float run = s_cdc[cta.tid];
#pragma unroll
        for (int w = 0; w < 16; ++w) run += s_x[w * DP + cta.tid];
#pragma unroll
        for (int w = 15; w >= 0; --w) {
            const float own = s_tot[w * DP + cta.tid];
            s_tot[w * DP + cta.tid] = run;
            run += own;
        }
    }
    __syncthreads();
    {
        float v[16], base[4];
        tc_ld16(cta.lanes() + 16 * cta.part, v);
        tc_wait_ld();
        unpack4(*reinterpret_cast<const float4*>(s_tot + cta.warp * DP + c0), base);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = 4 * cta.warp + it;
            if (i >= ch.nvalid) break;
            float* out = p.dld + (((long long)ch.b * p.g.T + ch.t0 + i) * p.g.H + ch.hh) * (long long)r + c0;
            const float z = ch.ok(i) ? 1.f : 0.f;
            if (FAST && (reinterpret_cast<uintptr_t>(p.dld) & 15) == 0) {
                if (c0 < r)
                    *reinterpret_cast<float4*>(out) = z != 0.f ? make_float4(v[4 * it] + base[0], v[4 * it + 1] + base[1], v[4 * it + 2] + base[2], v[4 * it + 3] + base[3])
                                                               : make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c0 + e < r) out[e] = z != 0.f ? v[4 * it + e] + base[e] : 0.f;
            }
        }
    }
    SD_PHASE_T(p.g, ch, ph);
}

template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 2) k_predictor_close_fast(BwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (leave_to_slow_kernel(p.Flags, FLAG_SLOW | FLAG_GAMMA)) return;
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    predictor_close_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}
// Both kinds of chunk in one launch, for calls that leave SMs empty anyway.
template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 1) k_predictor_close_one(BwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (chunk_flags(p.Flags, blockIdx.x) & (FLAG_SLOW | FLAG_GAMMA)) {
        chain_wait();
        chain_release();
        predictor_close_blocks<FAST, MASKED, false>(p, chunk_of<MASKED>(p.g, blockIdx.x), fsm_raw);
        return;
    }
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    predictor_close_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}

}  // namespace sd
