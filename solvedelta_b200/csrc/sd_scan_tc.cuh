// The serial chunk-state scans on the fifth-generation tensor cores (tcgen05): C and S forward, dS and dC in reverse (at
// the end of this file).
//
//     X  = P + Q St ;  checkpoint St ;  St = diag(lam) St + R^T X
// for every chunk of a stream in order (the predictor state is carried transposed, St[c][a] = C[a][c], so that both C and
// S decay by rows; column slices never exchange data).  A CTA carries a 64-column slice of one stream's state, transposed, in tensor
// memory (lane = slice column c, column = state row p), and both contractions take their A operand from tensor memory:
//     X^T[c][tok] = sum_p St^T[c][p] Q[tok][p]      A = rounded state,  B = Q as it lies (K-major)
//     St^T[c][p] += sum_t X^T[c][tok] R[tok][p]     A = rounded X,      B = R as it lies (MN-major)
// (M = 128 of which 64 lanes are used), so neither the state nor X passes through shared memory and no panel is
// transposed.  Q and R land as tiles of 128-byte rows by TMA: Q with the 128-byte swizzle, R with its 32-byte-atom form,
// the one an MN-major TF32 operand takes.  The roles are split over the warps: one thread issues the loads two chunks
// ahead, one issues the contractions, and the 256 threads that own lanes 0..63 (32 state and 16 X columns each) round,
// decay, add P and store; mbarriers connect them, so no step has a CTA-wide barrier.  Checkpoints are stored behind the
// first contraction and X behind the second one.
//
// What bounds it: the chain of two contractions per chunk with their hand-overs.
//
// Segments.  With few streams the chain is long and most SMs are idle.  The recurrence is affine in St, so the chunks of
// a stream may be cut into segments: a first pass (TRANSFER) walks all segments but the last at once and gives each
// one's end state from zero and its transfer matrix (the end states from the identity's columns with P left out);
// k_scan_combine chains them in FP32 into the segments' entry states; the second pass is the scan itself with all
// segments at once.
//
// Operands are rounded to TF32 (round to nearest) before the tensor core, which would truncate, sees them: the state and
// X in registers here, Q and R by the kernels that write those panels.
//
// Every mbarrier wait is bounded: a wait that runs out raises the fault word the host reads back, the thread stops
// waiting for the rest of the launch, and the kernel still walks to its end and frees its tensor memory.
#pragma once
#include <cuda.h>   // CUtensorMap (types only: the encoder is reached through the runtime's driver entry point)

#include "sd_bf16.cuh"
#include "sd_common.cuh"

namespace sd {

constexpr int SCAN_NS = 64;   // state columns per CTA (2 CTAs per stream)

struct ScanParams {
    const float* P;    // [chunks][CL][DP]
    const float* Q;
    const float* R;
    const float* lam;  // [chunks][DP]
    float* X;          // out [chunks][CL][DP]            (FP32; or null when Xb is set)
    float* ck;         // out [chunks][DP][DP] state before the chunk's update (or null when ckb is set)
    bf16* Xb;          // BF16 alternatives for consumers that only feed BF16 contractions
    bf16* ckb;
    const float* init; // nullable: true-dimension state [S][rows][cols] (or transposed)
    float* fin;        // nullable
    int NC;            // chunks per stream
    int segs, seg_len; // segments a stream is cut into, and their chunks (the last one may be shorter)
    float* seg_state;  // [streams][segs - 1][2][DP][DP]: end states and transfer matrices, then entry states (segs > 1)
    int transposed_io; // init/fin hold the transpose (predictor state C[a][c])
    int nrows, ncols;  // true dims of the carried St: rows (<= DP), cols (<= DP)
};


constexpr unsigned TC_R_SBO = 512;          // bytes between the 4-row groups of an MN-major TF32 tile
constexpr int TC_WAIT_LIMIT = 1 << 20;    // polls of one mbarrier before the wait is given up

__device__ __forceinline__ unsigned tc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle: start address, leading and stride byte offsets in 16-byte units.
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((addr >> 4) & 0x3FFF) | ((unsigned long long)((lbo >> 4) & 0x3FFF) << 16) |
           ((unsigned long long)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// Instruction descriptor: FP32 accumulator, TF32 operands, both K-major, M = 128.
__device__ __forceinline__ unsigned tc_idesc(int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((unsigned)(n >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void tc_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Bounded wait on one phase of an mbarrier; false when the limit ran out.
__device__ __forceinline__ bool tc_wait(unsigned bar, unsigned parity) {
    for (int it = 0; it < TC_WAIT_LIMIT; ++it) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// 32 consecutive 32-bit tensor-memory columns of this thread's lane.
__device__ __forceinline__ void tc_ld32(unsigned taddr, float* r) {
    unsigned* u = reinterpret_cast<unsigned*>(r);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
          "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]),
          "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]),
          "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_st32(unsigned taddr, const float* r) {
    const unsigned* u = reinterpret_cast<const unsigned*>(r);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31};" ::"r"(u[0]),
        "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]),
        "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]), "r"(u[18]), "r"(u[19]),
        "r"(u[20]), "r"(u[21]), "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]), "r"(u[27]), "r"(u[28]),
        "r"(u[29]), "r"(u[30]), "r"(u[31]), "r"(taddr)
        : "memory");
}
// 16-column forms of the two moves above
__device__ __forceinline__ void tc_ld16(unsigned taddr, float* r) {
    unsigned* u = reinterpret_cast<unsigned*>(r);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
          "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_st16(unsigned taddr, const float* r) {
    const unsigned* u = reinterpret_cast<const unsigned*>(r);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(u[0]),
        "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]),
        "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(taddr)
        : "memory");
}
template <int N>
__device__ __forceinline__ void tc_ld(unsigned taddr, float* r) {
    static_assert(N == 16 || N == 32, "16 or 32 columns per move");
    if (N == 32) tc_ld32(taddr, r); else tc_ld16(taddr, r);
}
template <int N>
__device__ __forceinline__ void tc_st(unsigned taddr, const float* r) {
    static_assert(N == 16 || N == 32, "16 or 32 columns per move");
    if (N == 32) tc_st32(taddr, r); else tc_st16(taddr, r);
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float tc_round(float x) { return __uint_as_float(f2tf32(x)); }

// `N` rows of one column per thread as BF16, rows DP apart: neighbouring lanes swap halves of a row pair, so that each
// store moves two columns.
template <int N>
__device__ __forceinline__ void tc_store_pairs(bf16* rows, int c, int lane, const float (&v)[N]) {
    const bool odd = lane & 1;
    bf16* dst = rows + (c & ~1) + (odd ? DP : 0);
#pragma unroll
    for (int j = 0; j < N; j += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
        const __nv_bfloat162 w = odd ? __floats2bfloat162_rn(other, v[j + 1]) : __floats2bfloat162_rn(v[j], other);
        *reinterpret_cast<__nv_bfloat162*>(dst + j * DP) = w;
    }
}

// Profiling build only: thread 0 of the first CTA records the SM clock at the phase boundaries of its ninth step.
#ifdef SD_DIAGNOSTICS
#define TC_STAMP(k)                                                                              \
    do {                                                                                         \
        if (dbg != nullptr && blockIdx.x == 0 && tid == 0 && n == 8)                          \
            dbg[k] = clock64();                                                                  \
    } while (0)
#else
#define TC_STAMP(k) do { } while (0)
#endif

// The kernel's shared memory: a two-slot ring of the chunk's operands, every tile on a 1024-byte boundary.
constexpr int TC_THREADS = 512;
constexpr int TC_WORKERS = 256;            // threads that own tensor-memory lanes 0..63 (lane quarters 0 and 1)
constexpr int TC_SCOLS = DP / 4;           // state columns (rows p of St) per worker thread
constexpr int TC_XCOLS = CL / 4;           // tokens of X per worker thread
constexpr unsigned TC_PANEL_BYTES = CL * DP * 4;        // Q or R: four boxes of 32 channels
constexpr unsigned TC_BOX_BYTES = CL * 32 * 4;          // [64 tokens][32 channels], 128-byte rows
constexpr unsigned TC_P_BYTES = CL * SCAN_NS * 4;       // the CTA's columns of P, as they lie
constexpr unsigned TC_LAM_BYTES = DP * 4;
constexpr unsigned TC_SLOT_BYTES = 2 * TC_PANEL_BYTES + TC_P_BYTES;
constexpr size_t SCAN_TC_SMEM_BYTES = 2 * size_t(TC_SLOT_BYTES) + 2 * TC_LAM_BYTES + 1024;   // + room to align
// tensor-memory columns: the state, its rounded copy (operand), X, its rounded copy
constexpr unsigned TC_S_COL = 0, TC_SA_COL = 128, TC_X_COL = 256, TC_XA_COL = 320, TC_TMEM_COLS = 512;

// D[128][N] (+)= A[128][8] B[8][N] with A in tensor memory (lane = row, column = contraction index)
__device__ __forceinline__ void tc_mma_ta(unsigned d_tmem, unsigned a_tmem, unsigned long long db, unsigned idesc,
                                          unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_load_box(unsigned char* sm, const CUtensorMap* map, int col, int chunk, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            tc_smem(sm)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(col), "r"(0), "r"(chunk), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Rows p0.. of column c of a stream's carried state, from and to the caller's [rows][cols] (or transposed) layout.  The
// transposed layout holds a thread's rows side by side: 16-byte accesses when every row starts on such a boundary.
__device__ __forceinline__ void tc_init_state(const float* init, int s, int nrows, int ncols, int transposed, int p0, int c,
                                              float (&st)[TC_SCOLS]) {
#pragma unroll
    for (int j = 0; j < TC_SCOLS; ++j) st[j] = 0.f;
    if (init == nullptr || c >= ncols) return;
    const float* src = init + (long long)s * nrows * ncols;
    if (transposed && (nrows & 3) == 0 && (reinterpret_cast<uintptr_t>(init) & 15) == 0) {
#pragma unroll
        for (int j = 0; j < TC_SCOLS; j += 4)
            if (p0 + j < nrows) {
                const float4 v = *reinterpret_cast<const float4*>(src + (long long)c * nrows + p0 + j);
                st[j] = v.x; st[j + 1] = v.y; st[j + 2] = v.z; st[j + 3] = v.w;
            }
        return;
    }
#pragma unroll
    for (int j = 0; j < TC_SCOLS; ++j)
        if (p0 + j < nrows) st[j] = transposed ? src[(long long)c * nrows + p0 + j] : src[(long long)(p0 + j) * ncols + c];
}
__device__ __forceinline__ void tc_final_state(float* fin, int s, int nrows, int ncols, int transposed, int p0, int c,
                                               const float (&st)[TC_SCOLS]) {
    if (fin == nullptr || c >= ncols) return;
    float* dst = fin + (long long)s * nrows * ncols;
    if (transposed && (nrows & 3) == 0 && (reinterpret_cast<uintptr_t>(fin) & 15) == 0) {
#pragma unroll
        for (int j = 0; j < TC_SCOLS; j += 4)
            if (p0 + j < nrows)
                *reinterpret_cast<float4*>(dst + (long long)c * nrows + p0 + j) = make_float4(st[j], st[j + 1], st[j + 2], st[j + 3]);
        return;
    }
#pragma unroll
    for (int j = 0; j < TC_SCOLS; ++j)
        if (p0 + j < nrows) dst[transposed ? (long long)c * nrows + p0 + j : (long long)(p0 + j) * ncols + c] = st[j];
}

// TRANSFER: the pass that prepares a segmented scan (see ScanParams::segs): the CTA's slice starts from zero (the first
// segment: from the given state), or from a column block of the identity with P left out, and only its last state is
// stored.
template <bool TRANSFER>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_state_scan_tc(ScanParams p, const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap rmap,
                const __grid_constant__ CUtensorMap pmap, int* fault, long long* dbg) {
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    unsigned char* tsm = tsm_raw + ((1024u - (tc_smem(tsm_raw) & 1023u)) & 1023u);
    float* s_lam = reinterpret_cast<float*>(tsm + 2 * TC_SLOT_BYTES);   // [2][DP]
    __shared__ __align__(8) unsigned long long bars[8];
    __shared__ unsigned s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3, part = warp >> 2;

    // grid: (stream, segment, column slice); the transfer pass has no last segment and four slices
    int block = blockIdx.x;
    const int slices = TRANSFER ? 4 : DP / SCAN_NS, nseg = TRANSFER ? p.segs - 1 : p.segs;
    const int slice = block % slices;
    block /= slices;
    const int seg = block % nseg, s = block / nseg;
    const bool identity = TRANSFER && slice >= 2;
    if (identity && seg == 0) return;   // the first segment starts from a known state
    const int col0 = (slice & 1) * SCAN_NS;
    const int first = seg * p.seg_len, steps = p.NC - first < p.seg_len ? p.NC - first : p.seg_len;
    const long long base = (long long)s * p.NC + first;

    const unsigned full0 = tc_smem(&bars[0]), free0 = tc_smem(&bars[2]), bar_a = tc_smem(&bars[4]), bar_x = tc_smem(&bars[5]);
    const unsigned bar1 = tc_smem(&bars[6]), bar2 = tc_smem(&bars[7]);
    if (tid == 0) {
        for (int i = 0; i < 8; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(&bars[i])), "r"(i == 4 || i == 5 ? TC_WORKERS : 1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&s_tmem)), "r"(TC_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_wait();   // the set-up above overlaps the end of the kernel before
    chain_release();
    const unsigned tbase = s_tmem;
    bool alive = true;   // cleared by the first wait that runs out
    auto wait = [&](unsigned bar, int parity, int code) {
        if (alive && !tc_wait(bar, parity)) {
            alive = false;
            atomicExch(fault, code);
        }
    };

    if (warp == 2) {   // ---- loads: one elected thread, two chunks ahead
        if (lane == 0) {
            for (int n = 0; n < steps; ++n) {
                const int b = n & 1;
                if (n >= 2) wait(free0 + 8 * b, ((n >> 1) - 1) & 1, 5);
                unsigned char* slot = tsm + b * TC_SLOT_BYTES;
                const unsigned bar = full0 + 8 * b;
                const int chunk = (int)(base + n);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"(2 * TC_PANEL_BYTES + (identity ? 0u : TC_P_BYTES) + TC_LAM_BYTES)
                             : "memory");
#pragma unroll
                for (int i = 0; i < 4; ++i) tc_load_box(slot + i * TC_BOX_BYTES, &qmap, 32 * i, chunk, bar);
#pragma unroll
                for (int i = 0; i < 4; ++i) tc_load_box(slot + TC_PANEL_BYTES + i * TC_BOX_BYTES, &rmap, 32 * i, chunk, bar);
                if (!identity) tc_load_box(slot + 2 * TC_PANEL_BYTES, &pmap, col0, chunk, bar);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 tc_smem(s_lam + b * DP)),
                             "l"(p.lam + (long long)chunk * DP), "r"(TC_LAM_BYTES), "r"(bar)
                             : "memory");
            }
        }
        __syncwarp();
    } else if (warp == 3) {   // ---- contractions: one elected thread
        if (lane == 0) {
            const unsigned id1 = tc_idesc(CL), id2 = tc_idesc(DP) | (1u << 16);   // second one: B is MN-major
            for (int n = 0; n < steps; ++n) {
                const int b = n & 1;
                const unsigned sq = tc_smem(tsm + b * TC_SLOT_BYTES), sr = sq + TC_PANEL_BYTES;
                wait(full0 + 8 * b, (n >> 1) & 1, 3);
                wait(bar_a, n & 1, 8);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < DP / 8; ++k)   // X^T = S^T Q^T
                    tc_mma_ta(tbase + TC_X_COL, tbase + TC_SA_COL + 8 * k,
                              tc_desc(sq + (k / 4) * TC_BOX_BYTES + (k % 4) * 32, 16, 1024) | (2ull << 61), id1, k > 0);
                tc_commit(bar1);
                wait(bar_x, n & 1, 9);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < CL / 8; ++k)   // S^T += X^T R
                    tc_mma_ta(tbase + TC_S_COL, tbase + TC_XA_COL + 8 * k, tc_desc(sr + k * 1024, TC_BOX_BYTES, TC_R_SBO) | (1ull << 61),
                              id2, 1u);
                tc_commit(bar2);
                tc_commit(free0 + 8 * b);
            }
        }
        __syncwarp();
    } else if (quarter < 2) {   // ---- workers: lane = state column c
        const int c = col0 + quarter * 32 + lane, p0 = part * TC_SCOLS, x0 = part * TC_XCOLS;
        const unsigned t_lane = tbase + ((unsigned)(quarter * 32) << 16);
        float st[TC_SCOLS];
if (identity) {
#pragma unroll
            for (int j = 0; j < TC_SCOLS; ++j) st[j] = p0 + j == c ? 1.f : 0.f;
        } else if (seg > 0) {
#pragma unroll
            for (int j = 0; j < TC_SCOLS; ++j)
                st[j] = TRANSFER ? 0.f : p.seg_state[((long long)(s * (p.segs - 1) + seg - 1) * 2 * DP + p0 + j) * DP + c];
        } else {
            tc_init_state(p.init, s, p.nrows, p.ncols, p.transposed_io, p0, c, st);
        }
        for (int n = 0; n < steps; ++n) {
            const int b = n & 1;
            const long long gi = base + n;
            TC_STAMP(0);
            if (n > 0) {
                wait(bar2, (n - 1) & 1, 2);
                tc_fence_after();
                tc_ld<TC_SCOLS>(t_lane + TC_S_COL + p0, st);
                tc_wait_ld();
            }
            TC_STAMP(1);
            {   // operand of the first contraction
                float r[TC_SCOLS];
#pragma unroll
                for (int j = 0; j < TC_SCOLS; ++j) r[j] = tc_round(st[j]);
                tc_st<TC_SCOLS>(t_lane + TC_SA_COL + p0, r);
                tc_wait_st();
                tc_fence_before();
                tc_arrive(bar_a);
            }
            TC_STAMP(2);
            if (!TRANSFER) {   // checkpoints, behind the first contraction: 32 lanes = 32 consecutive columns
                if (p.ck != nullptr) {
                    float* ck = state_ptr(p.ck, gi) + p0 * DP + c;
#pragma unroll
                    for (int j = 0; j < TC_SCOLS; ++j) __stcs(ck + j * DP, tc_round(st[j]));   // only read as an operand
                }
                if (p.ckb != nullptr) tc_store_pairs<TC_SCOLS>(p.ckb + gi * (long long)(DP * DP) + p0 * DP, c, lane, st);
            }
            TC_STAMP(3);
            wait(full0 + 8 * b, (n >> 1) & 1, 4);   // decay and P of this chunk
#pragma unroll
            for (int j = 0; j < TC_SCOLS; j += 4) {
                const float4 l = *reinterpret_cast<const float4*>(s_lam + b * DP + p0 + j);
                st[j] *= l.x;
                st[j + 1] *= l.y;
                st[j + 2] *= l.z;
                st[j + 3] *= l.w;
            }
            tc_st<TC_SCOLS>(t_lane + TC_S_COL + p0, st);
            float pv[TC_XCOLS], x[TC_XCOLS];
            if (!identity) {
                const float* ps = reinterpret_cast<const float*>(tsm + b * TC_SLOT_BYTES + 2 * TC_PANEL_BYTES) + x0 * SCAN_NS + quarter * 32 + lane;
#pragma unroll
                for (int j = 0; j < TC_XCOLS; ++j) pv[j] = ps[j * SCAN_NS];
            }
            tc_wait_st();
            TC_STAMP(4);
            wait(bar1, n & 1, 1);
            tc_fence_after();
            TC_STAMP(5);
            tc_ld<TC_XCOLS>(t_lane + TC_X_COL + x0, x);
            tc_wait_ld();
            {
                float r[TC_XCOLS];
#pragma unroll
                for (int j = 0; j < TC_XCOLS; ++j) {
                    if (!identity) x[j] += pv[j];
                    r[j] = tc_round(x[j]);
                }
                tc_st<TC_XCOLS>(t_lane + TC_XA_COL + x0, r);
                tc_wait_st();
                tc_fence_before();
                tc_arrive(bar_x);
            }
            TC_STAMP(6);
            if (!TRANSFER) {   // behind the second contraction
                if (p.Xb != nullptr) {
                    tc_store_pairs<TC_XCOLS>(bpanel_ptr(p.Xb, gi) + x0 * DP, c, lane, x);
                } else {
                    float* xg = panel_ptr(p.X, gi) + x0 * DP + c;
#pragma unroll
                    for (int j = 0; j < TC_XCOLS; ++j) xg[j * DP] = x[j];
                }
            }
            TC_STAMP(7);
        }
        wait(bar2, (steps - 1) & 1, 2);
        tc_fence_after();
        tc_ld<TC_SCOLS>(t_lane + TC_S_COL + p0, st);
        tc_wait_ld();
        if (TRANSFER) {
            float* dst = p.seg_state + ((long long)((s * (p.segs - 1) + seg) * 2 + (identity ? 1 : 0)) * DP + p0) * DP + c;
#pragma unroll
            for (int j = 0; j < TC_SCOLS; ++j) dst[j * DP] = st[j];
        } else if (seg == p.segs - 1) {
            tc_final_state(p.fin, s, p.nrows, p.ncols, p.transposed_io, p0, c, st);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TC_TMEM_COLS));
}

// ---------------------------------------------------------------------------
// The two reverse scans (dS and dC), chunks last to first:
//     X = P + Q St ;  checkpoint St ;  St = diag(lam) St + R^T X + R2^T X2
// Same structure with BF16 panels and kind::f16 contractions (gradient tolerances admit BF16 operands; the state itself
// stays FP32).  All panels land with the 128-byte swizzle as tiles of 64 channels; X2, whose columns are the M side, is
// an MN-major A operand in shared memory (rows 64..127 of it alias what follows and feed lanes nobody reads).  The X2
// term does not wait for X: it is issued behind the first contraction as soon as the decayed state is back.
struct ScanParamsB {
    const bf16 *P, *Q, *R, *R2, *X2;   // [chunks][CL][DP]
    const float* lam;                  // [chunks][DP]
    bf16* X;                           // out [chunks][CL][DP]
    bf16* ck;                          // out [chunks][DP][DP]
    const float* init;
    float* fin;
    int NC;
    int segs, seg_len;                 // as in ScanParams; segment 0 holds the last chunks
    float* seg_state;
    int transposed_io, nrows, ncols;
};

constexpr unsigned TB_TILE_BYTES = CL * 64 * 2;         // [64 tokens][64 channels]
constexpr unsigned TB_Q = 0, TB_R = 2 * TB_TILE_BYTES, TB_R2 = 4 * TB_TILE_BYTES, TB_X2 = 6 * TB_TILE_BYTES, TB_P = 7 * TB_TILE_BYTES;
constexpr unsigned TB_SLOT_BYTES = 8 * TB_TILE_BYTES;   // X2 and P: the CTA's 64 columns
constexpr size_t SCAN_TB_SMEM_BYTES = 2 * size_t(TB_SLOT_BYTES) + 2 * TC_LAM_BYTES + 1024;
constexpr unsigned TB_SA_COL = 128, TB_X_COL = 192, TB_XA_COL = 256;   // BF16 operands: two elements a column

__device__ __forceinline__ void tb_mma_ta(unsigned d_tmem, unsigned a_tmem, unsigned long long db, unsigned idesc,
                                          unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tb_mma_ss(unsigned d_tmem, unsigned long long da, unsigned long long db, unsigned idesc,
                                          unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// N values as N / 2 packed tensor-memory columns
template <int N>
__device__ __forceinline__ void tb_st_packed(unsigned taddr, const float (&v)[N]) {
    float w[N / 2];
#pragma unroll
    for (int j = 0; j < N / 2; ++j) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        w[j] = __uint_as_float(*reinterpret_cast<const unsigned*>(&h));
    }
    if constexpr (N == 16) {
        const unsigned* u = reinterpret_cast<const unsigned*>(w);
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(u[0]), "r"(u[1]),
                     "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(taddr)
                     : "memory");
    } else {
        tc_st<N / 2>(taddr, w);
    }
}

template <bool TRANSFER>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_state_scan_b(ScanParamsB p, const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap rmap,
               const __grid_constant__ CUtensorMap r2map, const __grid_constant__ CUtensorMap x2map,
               const __grid_constant__ CUtensorMap pmap, int* fault) {
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    unsigned char* tsm = tsm_raw + ((1024u - (tc_smem(tsm_raw) & 1023u)) & 1023u);
    float* s_lam = reinterpret_cast<float*>(tsm + 2 * TB_SLOT_BYTES);   // [2][DP]
    __shared__ __align__(8) unsigned long long bars[9];
    __shared__ unsigned s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3, part = warp >> 2;

    int block = blockIdx.x;
    const int slices = TRANSFER ? 4 : DP / SCAN_NS, nseg = TRANSFER ? p.segs - 1 : p.segs;
    const int slice = block % slices;
    block /= slices;
    const int seg = block % nseg, s = block / nseg;
    const bool identity = TRANSFER && slice >= 2;
    if (identity && seg == 0) return;
    const int col0 = (slice & 1) * SCAN_NS;
    const int first = seg * p.seg_len, steps = p.NC - first < p.seg_len ? p.NC - first : p.seg_len;
    const long long last = (long long)s * p.NC + p.NC - 1 - first;   // chunk of step n: last - n

    const unsigned full0 = tc_smem(&bars[0]), free0 = tc_smem(&bars[2]), bar_a = tc_smem(&bars[4]), bar_x = tc_smem(&bars[5]);
    const unsigned bar1 = tc_smem(&bars[6]), bar2 = tc_smem(&bars[7]), bar_s = tc_smem(&bars[8]);
    if (tid == 0) {
        for (int i = 0; i < 9; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(&bars[i])),
                         "r"(i == 4 || i == 5 || i == 8 ? TC_WORKERS : 1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&s_tmem)), "r"(TC_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_wait();   // the set-up above overlaps the end of the kernel before
    chain_release();
    const unsigned tbase = s_tmem;
    bool alive = true;
    auto wait = [&](unsigned bar, int parity, int code) {
        if (alive && !tc_wait(bar, parity)) {
            alive = false;
            atomicExch(fault, code);
        }
    };

    if (warp == 2) {   // ---- loads
        if (lane == 0) {
            for (int n = 0; n < steps; ++n) {
                const int b = n & 1;
                if (n >= 2) wait(free0 + 8 * b, ((n >> 1) - 1) & 1, 5);
                unsigned char* slot = tsm + b * TB_SLOT_BYTES;
                const unsigned bar = full0 + 8 * b;
                const int chunk = (int)(last - n);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"((identity ? 4u : 8u) * TB_TILE_BYTES + TC_LAM_BYTES)
                             : "memory");
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    tc_load_box(slot + TB_Q + i * TB_TILE_BYTES, &qmap, 64 * i, chunk, bar);
                    tc_load_box(slot + TB_R + i * TB_TILE_BYTES, &rmap, 64 * i, chunk, bar);
                    if (!identity) tc_load_box(slot + TB_R2 + i * TB_TILE_BYTES, &r2map, 64 * i, chunk, bar);
                }
                if (!identity) {
                    tc_load_box(slot + TB_X2, &x2map, col0, chunk, bar);
                    tc_load_box(slot + TB_P, &pmap, col0, chunk, bar);
                }
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 tc_smem(s_lam + b * DP)),
                             "l"(p.lam + (long long)chunk * DP), "r"(TC_LAM_BYTES), "r"(bar)
                             : "memory");
            }
        }
        __syncwarp();
    } else if (warp == 3) {   // ---- contractions
        if (lane == 0) {
            // FP32 accumulator, BF16 operands, M = 128; K-major unless a major bit (15: A, 16: B) says otherwise
            const auto idesc = [](int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((128u >> 4) << 24); };
            const auto desc = [](unsigned addr, unsigned lbo) { return tc_desc(addr, lbo, 1024) | (2ull << 61); };
            const unsigned id1 = idesc(CL), id2 = idesc(DP) | (1u << 16), id3 = id2 | (1u << 15);
            for (int n = 0; n < steps; ++n) {
                const int b = n & 1;
                const unsigned slot = tc_smem(tsm + b * TB_SLOT_BYTES);
                wait(full0 + 8 * b, (n >> 1) & 1, 3);
                wait(bar_a, n & 1, 8);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < DP / 16; ++k)   // X^T = S^T Q^T
                    tb_mma_ta(tbase + TB_X_COL, tbase + TB_SA_COL + 8 * k, desc(slot + TB_Q + (k / 4) * TB_TILE_BYTES + (k % 4) * 32, 16), id1, k > 0);
                tc_commit(bar1);
                wait(bar_s, n & 1, 10);
                tc_fence_after();
                if (!identity) {
#pragma unroll
                    for (int k = 0; k < CL / 16; ++k)   // S^T += X2^T R2
                        tb_mma_ss(tbase + TC_S_COL, desc(slot + TB_X2 + k * 2048, TB_TILE_BYTES), desc(slot + TB_R2 + k * 2048, TB_TILE_BYTES), id3, 1u);
                }
                wait(bar_x, n & 1, 9);
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < CL / 16; ++k)   // S^T += X^T R
                    tb_mma_ta(tbase + TC_S_COL, tbase + TB_XA_COL + 8 * k, desc(slot + TB_R + k * 2048, TB_TILE_BYTES), id2, 1u);
                tc_commit(bar2);
                tc_commit(free0 + 8 * b);
            }
        }
        __syncwarp();
    } else if (quarter < 2) {   // ---- workers: lane = state column c
        const int cl = quarter * 32 + lane, c = col0 + cl, p0 = part * TC_SCOLS, x0 = part * TC_XCOLS;
        const unsigned t_lane = tbase + ((unsigned)(quarter * 32) << 16);
        float st[TC_SCOLS];
        if (identity) {
#pragma unroll
            for (int j = 0; j < TC_SCOLS; ++j) st[j] = p0 + j == c ? 1.f : 0.f;
        } else if (seg > 0) {
#pragma unroll
            for (int j = 0; j < TC_SCOLS; ++j)
                st[j] = TRANSFER ? 0.f : p.seg_state[((long long)(s * (p.segs - 1) + seg - 1) * 2 * DP + p0 + j) * DP + c];
        } else {
            tc_init_state(p.init, s, p.nrows, p.ncols, p.transposed_io, p0, c, st);
        }
        for (int n = 0; n < steps; ++n) {
            const int b = n & 1;
            const long long gi = last - n;
            if (n > 0) {
                wait(bar2, (n - 1) & 1, 2);
                tc_fence_after();
                tc_ld<TC_SCOLS>(t_lane + TC_S_COL + p0, st);
                tc_wait_ld();
            }
            tb_st_packed<TC_SCOLS>(t_lane + TB_SA_COL + p0 / 2, st);
            tc_wait_st();
            tc_fence_before();
            tc_arrive(bar_a);
            if (!TRANSFER) tc_store_pairs<TC_SCOLS>(p.ck + gi * (long long)(DP * DP) + p0 * DP, c, lane, st);
            wait(full0 + 8 * b, (n >> 1) & 1, 4);
#pragma unroll
            for (int j = 0; j < TC_SCOLS; j += 4) {
                const float4 l = *reinterpret_cast<const float4*>(s_lam + b * DP + p0 + j);
                st[j] *= l.x;
                st[j + 1] *= l.y;
                st[j + 2] *= l.z;
                st[j + 3] *= l.w;
            }
            tc_st<TC_SCOLS>(t_lane + TC_S_COL + p0, st);
            tc_wait_st();
            tc_fence_before();
            tc_arrive(bar_s);
            float x[TC_XCOLS], pv[TC_XCOLS];
            if (!identity) {   // P as TMA landed it: 16-byte piece (c / 8) of a row sits at piece (c / 8) ^ (row % 8)
                const unsigned char* ps = tsm + b * TB_SLOT_BYTES + TB_P + x0 * 128;
#pragma unroll
                for (int j = 0; j < TC_XCOLS; ++j)
                    pv[j] = __bfloat162float(*reinterpret_cast<const bf16*>(ps + j * 128 + ((((cl >> 3) ^ (j & 7)) << 4) | ((cl & 7) << 1))));
            }
            wait(bar1, n & 1, 1);
            tc_fence_after();
            tc_ld<TC_XCOLS>(t_lane + TB_X_COL + x0, x);
            tc_wait_ld();
            if (!identity) {
#pragma unroll
                for (int j = 0; j < TC_XCOLS; ++j) x[j] += pv[j];
            }
            tb_st_packed<TC_XCOLS>(t_lane + TB_XA_COL + x0 / 2, x);
            tc_wait_st();
            tc_fence_before();
            tc_arrive(bar_x);
            if (!TRANSFER) tc_store_pairs<TC_XCOLS>(bpanel_ptr(p.X, gi) + x0 * DP, c, lane, x);
        }
        wait(bar2, (steps - 1) & 1, 2);
        tc_fence_after();
        tc_ld<TC_SCOLS>(t_lane + TC_S_COL + p0, st);
        tc_wait_ld();
        if (TRANSFER) {
            float* dst = p.seg_state + ((long long)((s * (p.segs - 1) + seg) * 2 + (identity ? 1 : 0)) * DP + p0) * DP + c;
#pragma unroll
            for (int j = 0; j < TC_SCOLS; ++j) dst[j * DP] = st[j];
        } else if (seg == p.segs - 1) {
            tc_final_state(p.fin, s, p.nrows, p.ncols, p.transposed_io, p0, c, st);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TC_TMEM_COLS));
}

// Entry states of the segments of a segmented scan: E_g = local_g + transfer_g E_{g-1}, written over local_g, where
// (local, transfer) are the pairs the transfer pass stored.  FP32 throughout.  One CTA per stream and 8 columns (they
// never exchange data); the next transfer matrix streams into shared memory while the current one is multiplied, since
// the chain over segments would otherwise wait for memory at every link (5.8 us a segment against 1).
constexpr int COMBINE_COLS = 8, COMBINE_THREADS = 256, COMBINE_PITCH = DP + 4;
constexpr size_t COMBINE_SMEM = size_t(2) * DP * COMBINE_PITCH * 4 + DP * COMBINE_COLS * 4;
__global__ void __launch_bounds__(COMBINE_THREADS) k_scan_combine(float* seg_state, int segs) {
    chain_wait();
    chain_release();
    extern __shared__ __align__(16) float csm[];
    float* s_t = csm;                                   // [2][DP][COMBINE_PITCH]
    float* s_e = csm + 2 * DP * COMBINE_PITCH;          // [DP][COMBINE_COLS]
    const int col0 = (blockIdx.x % (DP / COMBINE_COLS)) * COMBINE_COLS, s = blockIdx.x / (DP / COMBINE_COLS);
    const int row = threadIdx.x >> 1, c0 = (threadIdx.x & 1) * 4;
    float* base = seg_state + (long long)s * (segs - 1) * 2 * DP * DP;
    auto issue = [&](int g) {
        if (g > 0 && g < segs - 1) {
            const float* t = base + ((long long)g * 2 + 1) * DP * DP;
            float* dst = s_t + (g & 1) * DP * COMBINE_PITCH;
            for (int idx = threadIdx.x; idx < DP * (DP / 4); idx += COMBINE_THREADS)
                cp16(dst + (idx >> 5) * COMBINE_PITCH + (idx & 31) * 4, t + idx * 4);
        }
        cp_commit();
    };
    issue(1);
    for (int g = 0; g < segs - 1; ++g) {
        float* local = base + (long long)g * 2 * DP * DP + row * DP + col0 + c0;
        float4 acc = *reinterpret_cast<const float4*>(local);
        if (g > 0) {
            issue(g + 1);
            cp_wait<1>();
            __syncthreads();
            const float* t = s_t + (g & 1) * DP * COMBINE_PITCH + row * COMBINE_PITCH;
#pragma unroll 8
            for (int k = 0; k < DP; k += 4) {
                const float4 w = *reinterpret_cast<const float4*>(t + k);
                const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 e = *reinterpret_cast<const float4*>(s_e + (k + i) * COMBINE_COLS + c0);
                    acc.x = fmaf(wv[i], e.x, acc.x);
                    acc.y = fmaf(wv[i], e.y, acc.y);
                    acc.z = fmaf(wv[i], e.z, acc.z);
                    acc.w = fmaf(wv[i], e.w, acc.w);
                }
            }
            *reinterpret_cast<float4*>(local) = acc;
        }
        __syncthreads();
        *reinterpret_cast<float4*>(s_e + row * COMBINE_COLS + c0) = acc;
        __syncthreads();
    }
}

}  // namespace sd
