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
    if (leave_to_slow_kernel(p.Flags)) return;
    FastCta cta;
    fast_setup<!MASKED>(cta, fsm_raw, p.fault);
    exterior_pair_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}

}  // namespace sd
