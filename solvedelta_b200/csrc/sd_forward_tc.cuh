// k_primal_exterior_fast: primal address and exterior preparation of the fast chunks (sd_chunk_tc.cuh) on tcgen05; slow ones
// and the predictor-only entry take k_primal_exterior_fwd (sd_forward.cuh).
//
// With G referenced to the chunk start, Ubar = u^ exp(GL - G) (kept by k_prep_fwd) and lam = exp(GL):
//     D2 = lam (K^ Ct^T) + tril(K^ Delta^T) Ubar          d = k^ + exp(G - GL) D2
//     [Aqd; Aed] = tril / stril of [chi exp(G); -e exp(G)] (d exp(-G))^T
// All operands are TF32, rounded to nearest where they are written (the state by the scan).  Shared memory, three slots
// of 32 KB:  S0 K^;  S1 Delta, then Ubar;  S2 the state, 64 of its rows at a time, then d;  then S0 + S1 hold the stacked
// operand [chi exp(G); -e exp(G)] (128 rows: one contraction gives both pair matrices) and S2 d exp(-G) in place of d;
// then S0 z, S1 Aed and S2 -e exp(G), whose FP32 values wait in tensor memory meanwhile, for the solve.
//
// What bounds it: the latency of a chunk's chain (19 us alone on an SM) and, with two on an SM, shared-memory and
// global accesses (60 % of the load/store pipe's wavefronts; DRAM 3.4 TB/s).  At 8 x 4096 tokens of 8 heads 492 us against
// 838 us of the block-centred kernel; two chunks of 256 threads with 128 registers to an SM took 583 us, a next row kept in
// registers 600 us (spills), and prefetching the next task's panels into L2 40 us more.
// Tensor memory (256 columns): 0 D2, later the FP32 -e exp(G); 128 K^ Delta^T, later the pair matrices; 192 tril(K^ Delta^T).
#pragma once
#include "sd_chunk_tc.cuh"
#include "sd_forward.cuh"

namespace sd {

constexpr unsigned PE_D1 = 128, PE_A = 192, PE_PAIR = 128;
constexpr unsigned PE_SLOT = CL * DP * 4;
static_assert(3 * PE_SLOT + DP * 4 <= FAST_BAR_OFF, "slots and tables fit");
static_assert(CL * LDA * 4 <= PE_SLOT, "the pair matrix of the solve fits a slot");

struct SourceRow {   // what the per-token pass reads of a row from global memory, four channels
    uint2 k, q, u, er;
    float4 dl, g;
};

template <bool FAST, bool MASKED>
__device__ __forceinline__ void primal_exterior_fast(const FwdParams& p, const ChunkT<MASKED>& ch, FastCta& cta) {
    unsigned char *S0 = cta.sm, *S1 = S0 + PE_SLOT, *S2 = S1 + PE_SLOT;
    float* s_lam = reinterpret_cast<float*>(S2 + PE_SLOT);
    const int r = p.g.r, V = p.g.V;
    const int c0 = cta.lane * 4;
    const float *gDelta = panel_ptr(p.Delta, ch.gi), *gG = panel_ptr(p.Gp, ch.gi);
    const float* gCt = state_ptr(p.CtCk, ch.gi);
    const bool keep = p.Dprim != nullptr;   // kernel-uniform: a reverse pass will follow
    // rows by warp: the lane's four channels of row i, as a panel in global memory and as a piece of the tiles
    const auto piece = [&](int i, unsigned ts) { return (cta.lane >> 3) * ts + i * 128 + (((cta.lane & 7) ^ (i & 7)) << 4); };
    int ph = 0;
    SD_PHASE_T(p.g, ch, ph);

#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it) {
        const int i = cta.warp + 16 * it;
        cp16(S1 + piece(i, F32_TILE), gDelta + i * DP + c0);
    }
    cp_commit();
#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it) {
        const int i = cta.warp + 16 * it;
        cp16(S2 + piece(i, F32_TILE), gCt + i * DP + c0);
    }
    cp_commit();
    {   // k^
        uint2 raw[FAST_PASSES];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = cta.warp + 16 * it;
            raw[it] = load4_raw<FAST>(row_bf16(p.k, ch, i), c0, r, p.k.vec, ch.ok(i));
        }
        if (cta.tid < DP) s_lam[cta.tid] = p.Lam[ch.gi * DP + cta.tid];
        float ss[FAST_PASSES];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4];
            unpack4(raw[it], x);
            ss[it] = fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3])));
        }
        row_sums32(ss);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float x[4];
            unpack4(raw[it], x);
            const float rs = rsqrtf(ss[it] + 1e-24f);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] *= rs;
            *reinterpret_cast<float4*>(S0 + piece(cta.warp + 16 * it, F32_TILE)) = tf32_bits4(pack4(x));
        }
    }
    cp_wait<1>();
#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it) {   // Delta is also used in FP32: its copy here is rounded by the thread that landed it
        float4* q = reinterpret_cast<float4*>(S1 + piece(cta.warp + 16 * it, F32_TILE));
        *q = tf32_bits4(*q);
    }
    cta.publish();
    SD_PHASE_T(p.g, ch, ph);
    if (cta.tid == 0) {
        tc_fence_after();
        mma_tf32_kk<F32_TILE, F32_TILE>(cta.tmem + PE_D1, tc_smem(S0), tc_smem(S1), CL, 0u);
        tc_commit(cta.bar(0));
    }
    __syncwarp();
    cp_wait<0>();
    cta.publish();
    if (cta.tid == 32) {
        tc_fence_after();
        mma_tf32_kk<F32_TILE, F32_TILE>(cta.tmem, tc_smem(S0), tc_smem(S2), CL, 0u);
        tc_commit(cta.bar(1));
    }
    __syncwarp();
    cta.wait(0, 11);   // Delta is free: Ubar takes its slot
    {
        const float* gUbar = panel_ptr(p.Ubar, ch.gi);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = cta.warp + 16 * it;
            cp16(S1 + f32_mn_off(i, c0), gUbar + i * DP + c0);
        }
        cp_commit();
    }
    if (cta.quarter < 2) {   // tril(K^ Delta^T), rounded, back as an operand
        float a[16];
        tc_ld16(cta.lanes() + PE_D1 + 16 * cta.part, a);
        tc_wait_ld();
        const int i = 32 * cta.quarter + cta.lane;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            a[j] = 16 * cta.part + j <= i ? __uint_as_float(mma_tf32_bits(a[j])) : 0.f;
        tc_st16(cta.lanes() + PE_A + 16 * cta.part, a);
    }
    cta.wait(1, 12);   // the state's first rows are free
#pragma unroll
    for (int it = 0; it < FAST_PASSES; ++it) {
        const int i = cta.warp + 16 * it;
        cp16(S2 + piece(i, F32_TILE), gCt + (CL + i) * DP + c0);
    }
    cp_commit();
    const auto scale_by_lam = [&](int col) {
        float a[16];
        tc_ld16(cta.lanes() + col, a);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 l = *reinterpret_cast<const float4*>(s_lam + col + j);
            a[j] *= l.x; a[j + 1] *= l.y; a[j + 2] *= l.z; a[j + 3] *= l.w;
        }
        tc_st16(cta.lanes() + col, a);
        tc_wait_st();
    };
    if (cta.quarter < 2) scale_by_lam(16 * cta.part);
    cp_wait<0>();
    cta.publish();
    SD_PHASE_T(p.g, ch, ph);
    if (cta.tid == 64) {
        tc_fence_after();
        mma_tf32_kk<F32_TILE, F32_TILE>(cta.tmem + CL, tc_smem(S0), tc_smem(S2), CL, 0u);
        tc_commit(cta.bar(2));
    }
    __syncwarp();
    cta.wait(2, 13);
    if (cta.quarter < 2) scale_by_lam(CL + 16 * cta.part);
    cta.publish();
    if (cta.tid == 96) {
        tc_fence_after();
        const unsigned long long db = f32_mn_desc(tc_smem(S1));
#pragma unroll
        for (int k = 0; k < CL / 8; ++k)
            tc_mma_ta(cta.tmem, cta.tmem + PE_A + 8 * k, db + k * (1024 / 16), tc_idesc(DP) | (1u << 16), 1u);
        tc_commit(cta.bar(3));
    }
    __syncwarp();
    cta.wait(3, 14);
    if (cta.quarter < 2) {
        const int i = 32 * cta.quarter + cta.lane;
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
            const int col = 32 * cta.part + 16 * hc;
            float a[16];
            tc_ld16(cta.lanes() + col, a);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                *reinterpret_cast<float4*>(S2 + f32_off<F32_TILE>(i, col + j)) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    SD_PHASE_T(p.g, ch, ph);
    // ---- per-token pass: the sources (sources_fwd), all sums of a row in one reduction over the raw rows ----
    {
        float lam[4];
        unpack4(*reinterpret_cast<const float4*>(s_lam + c0), lam);
#pragma unroll 1
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = cta.warp + 16 * it;
            SourceRow row;
            {
                const bool ok = ch.ok(i);
                row.k = load4_raw<FAST>(row_bf16(p.k, ch, i), c0, r, p.k.vec, ok);
                row.q = load4_raw<FAST>(row_bf16(p.q, ch, i), c0, r, p.q.vec, ok);
                row.u = load4_raw<FAST>(row_bf16(p.u, ch, i), c0, r, p.u.vec, ok);
                row.er = load4_raw<FAST>(row_bf16(p.er, ch, i), c0, r, p.er.vec, ok);
                row.dl = ld_pinned16(gDelta + i * DP + c0);
                row.g = ld_pinned16(gG + i * DP + c0);
            }
            float k[4], q[4], dl[4], bk[4], sums[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            unpack4(row.k, k);
            unpack4(row.q, q);
            unpack4(row.er, bk);
            unpack4(row.dl, dl);
            {
                float u[4];
                unpack4(row.u, u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    bk[e] = sigmoidf_(bk[e]) * k[e];
                    sums[0] = fmaf(k[e], k[e], sums[0]);
                    sums[1] = fmaf(q[e], q[e], sums[1]);
                    sums[2] = fmaf(u[e], u[e], sums[2]);
                    sums[3] = fmaf(dl[e], dl[e], sums[3]);
                    sums[4] = fmaf(u[e], bk[e], sums[4]);
                    sums[5] = fmaf(u[e], q[e], sums[5]);
                    sums[6] = fmaf(u[e], dl[e], sums[6]);
                }
            }
            float d[4], eg[4], ie[4];
            float4* s_d = reinterpret_cast<float4*>(S2 + piece(i, F32_TILE));
            unpack4(*s_d, d);
            unpack4(row.g, eg);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ie[e] = exp_ftz(-eg[e]);
                eg[e] = exp_ftz(eg[e]);
                d[e] *= eg[e] * rcp_ftz(lam[e]);
            }
            row_sums32(sums);
            const float rk = rsqrtf(sums[0] + 1e-24f), rq = rsqrtf(sums[1] + 1e-24f), ru = rsqrtf(sums[2] + 1e-24f);
            const float sc = RHO * rsqrtf(RHO * RHO + sums[3]), den = 1.f + sc * ru * sums[6];
            const float sb = sc * (ru * rk * sums[4] / den), sq = sc * (ru * rq * sums[5] / den);
            float xg[4], ag[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                d[e] = fmaf(k[e], rk, d[e]);
                xg[e] = (q[e] * rq - dl[e] * sq) * eg[e];
                ag[e] = (dl[e] * sb - bk[e] * rk) * eg[e];
            }
            const long long at = ch.gi * (CL * DP) + i * DP + c0;   // the same place in every panel
            if (keep) *reinterpret_cast<float4*>(p.Dprim + at) = pack4(d);
#pragma unroll
            for (int e = 0; e < 4; ++e) d[e] *= ie[e];
            *reinterpret_cast<float4*>(S0 + piece(i, 2 * F32_TILE)) = tf32_bits4(pack4(xg));
            *reinterpret_cast<float4*>(S0 + piece(CL + i, 2 * F32_TILE)) = tf32_bits4(pack4(ag));
            *s_d = tf32_bits4(pack4(d));   // the elements this thread has read
            tc_st4(cta.lanes() + 16 * cta.part + 4 * it, ag);
            *reinterpret_cast<uint2*>(p.Xg + at) = pack4_bf16(xg);
            if (keep) {
                *reinterpret_cast<uint2*>(p.Ag + at) = pack4_bf16(ag);
                *reinterpret_cast<uint2*>(p.Dcol + at) = pack4_bf16(d);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) d[e] *= lam[e];
            if (keep) *reinterpret_cast<uint2*>(p.DtB + at) = pack4_bf16(d);
            // an operand of the state scan
            *reinterpret_cast<float4*>(p.Dt + at) = make_float4(round_tf32(d[0]), round_tf32(d[1]), round_tf32(d[2]), round_tf32(d[3]));
        }
        tc_wait_st();
    }
    cta.publish();
    SD_PHASE_T(p.g, ch, ph);
    if (cta.tid == 128) {
        tc_fence_after();
        mma_tf32_kk<2 * F32_TILE, F32_TILE>(cta.tmem + PE_PAIR, tc_smem(S0), tc_smem(S2), CL, 0u);
        tc_commit(cta.bar(4));
    }
    __syncwarp();
    {   // z = sigmoid(write) v, loaded behind the contraction
        uint2 wr[FAST_PASSES], v[FAST_PASSES];
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            const int i = cta.warp + 16 * it;
            wr[it] = load4_raw<FAST>(row_bf16(p.wr, ch, i), c0, V, p.wr.vec, ch.ok(i));
            v[it] = load4_raw<FAST>(row_bf16(p.v, ch, i), c0, V, p.v.vec, ch.ok(i));
        }
        cta.wait(4, 15);
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it) {
            float z[4], w[4];
            unpack4(v[it], z);
            unpack4(wr[it], w);
#pragma unroll
            for (int e = 0; e < 4; ++e) z[e] *= sigmoidf_(w[e]);
            *reinterpret_cast<float4*>(S0 + piece(cta.warp + 16 * it, F32_TILE)) = pack4(z);
        }
    }
    {
        float ag[16];
        tc_ld16(cta.lanes() + 16 * cta.part, ag);
        tc_wait_ld();
#pragma unroll
        for (int it = 0; it < FAST_PASSES; ++it)
            *reinterpret_cast<float4*>(S2 + piece(cta.warp + 16 * it, F32_TILE)) =
                make_float4(ag[4 * it], ag[4 * it + 1], ag[4 * it + 2], ag[4 * it + 3]);
    }
    float* s_aed = reinterpret_cast<float*>(S1);
    {
        float a[16];
        tc_ld16(cta.lanes() + PE_PAIR + 16 * cta.part, a);
        tc_wait_ld();
        const int i = (32 * cta.quarter + cta.lane) & (CL - 1), j0 = 16 * cta.part;
        if (cta.quarter < 2) {
            bf16* g = bmat_ptr(p.Aqd, ch.gi) + i * CL + j0;
#pragma unroll
            for (int j = 0; j < 16; j += 8) {
                float w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) w[e] = j0 + j + e <= i ? a[j + e] : 0.f;
                *reinterpret_cast<uint4*>(g + j) = pack8_bf16(w);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = j0 + j < i ? a[j] : 0.f;
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                *reinterpret_cast<float4*>(s_aed + i * LDA + j0 + j) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
            if (keep) {
                float* g = mat_ptr(p.Aed, ch.gi) + i * CL + j0;
#pragma unroll
                for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(g + j) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    SD_PHASE_T(p.g, ch, ph);
    const int panel = cta.warp >> 3, pt = (cta.warp >> 1) & 3;
    unsigned char* tile = (panel == 0 ? S2 : S0) + pt * F32_TILE;
    trisolve_blocked<false>(s_aed, -1.f, TileF32{tile, (cta.warp & 1) * 4});
    SD_PHASE_T(p.g, ch, ph);
    if (panel == 0)
        store_half_tile<true>(cta, panel_ptr(p.Wd, ch.gi) + 32 * pt, tile);   // a contraction operand of the state scan
    else
        store_half_tile<false>(cta, panel_ptr(p.Ud, ch.gi) + 32 * pt, tile);
    SD_PHASE_T(p.g, ch, ph);
}

template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 2) k_primal_exterior_fast(FwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (leave_to_slow_kernel(p.Flags, FLAG_SLOW)) return;
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    primal_exterior_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}
// Both kinds of chunk in one launch, for calls that leave SMs empty anyway.
template <bool FAST, bool MASKED>
__global__ void __launch_bounds__(NTHREADS, 1) k_primal_exterior_one(FwdParams p) {
    extern __shared__ __align__(1024) unsigned char fsm_raw[];
    if (chunk_flags(p.Flags, blockIdx.x) & (FLAG_SLOW)) {
        chain_wait();
        chain_release();
        primal_exterior_blocks<FAST, MASKED, false>(p, chunk_of<MASKED>(p.g, blockIdx.x), reinterpret_cast<float*>(fsm_raw));
        return;
    }
    FastCta cta;
    fast_setup(cta, fsm_raw, p.fault);
    primal_exterior_fast<FAST, MASKED>(p, chunk_of<MASKED>(p.g, blockIdx.x), cta);
    fast_teardown(cta);
}

}  // namespace sd
