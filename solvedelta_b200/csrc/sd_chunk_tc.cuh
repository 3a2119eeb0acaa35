// What the fast chunk kernels share: chunks whose contractions run on the fifth-generation tensor cores.
//
// Fast chunks.  A chunk that forgets at most FAST_CHUNK_NATS in every channel needs no block centring: with G the
// inclusive prefix of the log decay, every decay-weighted term exp(x_i - G_j) is the product of a row factor exp(x_i) <= 1
// and a column factor exp(-G_j) <= e^60, both far inside the range of FP32, TF32 and BF16 (which share their exponent),
// so a pair matrix is ONE contraction over all channels and a causal or anti-causal sum ONE contraction over all tokens,
// masked by a select.  Such chunks take tcgen05 in the kernels named *_fast; a chunk that forgets more, or holds a reset,
// takes the block-centred kernels (sd_decay.cuh), whose CTAs, one per SM, share the slow chunks of a launch.  The
// choice is made per chunk by k_prep_fwd, which stores it in the chunk's flag word: from what the chunk itself holds, so it
// does not depend on what else is in the call.
//
// A NaN or an infinity of one token reaches all tokens of its chunk, earlier ones too: in a causal sum over the chunk it meets
// the zeros of the mask, and zero times NaN is NaN.  (In the block-centred kernels the primal address of its own 16 tokens; y
// passes through such a sum, k_output_fwd_tc, after either.)  Nothing before its chunk is touched by it.
//
// A chunk is a chain of loads, contractions, row passes and a solve, each of which leaves most of an SM idle: what counts
// is the length of that chain and how many chains share the SM.  The fast kernels run one chunk a CTA of 16 warps, two CTAs
// to an SM (64 registers a thread, half of the shared and of the tensor memory each); with accumulators and the operands
// between two contractions in tensor memory the FP32 panels of a chunk fit a CTA's 113 KB.  Persistent CTAs were slower (the
// primal kernel 557 against 500 us at 4096 chunks: their row passes met more often).
#pragma once
#include "sd_decay.cuh"
#include "sd_scan_tc.cuh"

namespace sd {

constexpr float FAST_CHUNK_NATS = 60.f;
constexpr int FLAG_SLOW = 1;              // some channel's prefix leaves [-FAST_CHUNK_NATS, FAST_CHUNK_NATS]
constexpr int FLAG_GAMMA = 2;             // some valid token's geometry rate is below MIN_GAMMA
constexpr float MIN_GAMMA = 1e-20f;
constexpr int FAST_PASSES = CL / 16;      // row-wise passes: a warp takes a row, a lane four channels
constexpr int FAST_BARS = 8;
constexpr unsigned FAST_TMEM = 256;       // tensor-memory columns of a CTA
constexpr size_t FAST_SMEM = 113 * 1024;  // two CTAs per SM
constexpr size_t FAST_BAR_OFF = FAST_SMEM - (FAST_BARS + 1) * 8;
constexpr unsigned F32_TILE = CL * 128;   // [64 rows][32 channels] FP32, or [64 rows][64 channels] BF16: 128-byte rows

// The flags are read before a launch waits for the one before it.  They are two launches older or more: every launch of the
// sequence waits for its predecessor before it lets its successor begin, so k_prep_fwd has completed, with its writes performed,
// before any launch that reads flags begins; such a launch reads them once and holds no older copy.
// Nothing else is read before the wait.
__device__ __forceinline__ int chunk_flags(const unsigned char* flags, long long gi) { return __ldg(flags + gi); }

struct FastCta {
    int tid, warp, lane, quarter, part;   // quarter: the tensor-memory lanes of this warp, part: its quarter of the columns
    unsigned char* sm;
    unsigned tmem, bars;
    bool alive;
    int* fault;
    __device__ __forceinline__ unsigned bar(int i) const { return bars + 8 * i; }
    // every barrier is used once; a wait that runs out raises the fault word and ends all later ones
    __device__ __forceinline__ void wait(int i, int code) {
        bool done = alive && tc_wait(bar(i), 0);
        done = __all_sync(0xffffffffu, done);
        if (alive && !done && lane == 0) atomicExch(fault, code);
        alive = done;
        tc_fence_after();
    }
    __device__ __forceinline__ unsigned lanes() const { return tmem + ((unsigned)(quarter * 32) << 16); }
    // tensor-memory and shared-memory accesses of all threads are ordered before the contractions issued after this
    __device__ __forceinline__ void publish() const {
        tc_fence_before();
        tc_fence_async_smem();
        __syncthreads();
    }
};

// Tensor memory is allocated before the launch lets its successor start, so that a kernel that starts early can never hold
// what this one still waits for.  These kernels have no static shared memory: the dynamic part starts on the 1024-byte
// boundary that the swizzled tiles need (behind the 1 KB the system keeps), which is checked.
__device__ __forceinline__ void fast_setup(FastCta& cta, unsigned char* smem, int* fault) {
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + FAST_BAR_OFF);
    unsigned* s_tmem = reinterpret_cast<unsigned*>(bars + FAST_BARS);
    cta.tid = threadIdx.x;
    cta.warp = cta.tid >> 5;
    cta.lane = cta.tid & 31;
    cta.quarter = cta.warp & 3;
    cta.part = cta.warp >> 2;
    if (cta.tid == 0) {
        for (int i = 0; i < FAST_BARS; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&bars[i])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (cta.warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(s_tmem)), "r"(FAST_TMEM));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    cta.sm = smem;
    cta.tmem = *s_tmem;
    cta.bars = tc_smem(bars);
    cta.alive = (tc_smem(smem) & 1023u) == 0;   // else nothing here can be right: no waits, and the fault word says so
    cta.fault = fault;
    if (!cta.alive && cta.tid == 0) atomicExch(fault, 20);
    chain_wait();
    chain_release();
}
// True for a slow chunk, which another kernel does: the CTA only keeps its place in the chain of launches.  (The flags are
// older than the launch before.)
__device__ __forceinline__ bool leave_to_slow_kernel(const unsigned char* flags, int mask) {
    if (!(chunk_flags(flags, blockIdx.x) & mask)) return false;
    chain_wait();
    chain_release();
    return true;
}
__device__ __forceinline__ void fast_teardown(const FastCta& cta) {
    tc_fence_before();
    __syncthreads();
    if (cta.warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(cta.tmem), "r"(FAST_TMEM));
}

// The slow chunks of a launch, shared out over the CTAs by their rank, so that a CTA's share does not depend on where they
// lie.  A pass ranks 8192 flags, 16 a thread, and each CTA lists the chunks whose rank is its own (a few us; stepping through
// all slow chunks to find them took 0.12 us for each, 0.5 ms of a kernel with 4096).  Whether there are any is looked up while
// the launch before still runs (see chunk_flags): what stands between a wait and the end of a launch without slow chunks is
// waited for by all that follow (looked up behind the wait: 1024 tokens of 8 heads 267 -> 278 us forward and reverse).
// With every chunk slow, 8 x 4096 tokens of 8 heads take 3.84 ms forward and reverse, 3.72 in kernels of one CTA for each
// chunk: 4096 CTAs of a fast kernel take 28 us to come and go (8 us if it allocates no tensor memory).
constexpr int SLOW_PASS = NTHREADS * 16;
constexpr int SLOW_LIST = SLOW_PASS / 148 + 1;   // a share of a pass; grids of fewer CTAs have no more chunks than CTAs
template <int MASK, class F>
__device__ __forceinline__ void for_slow_chunks(const unsigned char* flags, int tasks, F f) {
    __shared__ unsigned short s_list[SLOW_LIST];
    __shared__ unsigned short s_count[NTHREADS / 32];
    unsigned any = 0;   // the flags are followed by zeros
#pragma unroll 1
    for (int t0 = 16 * threadIdx.x; t0 < tasks; t0 += SLOW_PASS) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(flags + t0));
        any |= w.x | w.y | w.z | w.w;
    }
    any = __syncthreads_or(any & (MASK * 0x01010101u));
    chain_wait();
    chain_release();
    if (any == 0) return;
    unsigned turn = blockIdx.x;   // this CTA's first rank among the slow chunks of the pass
#pragma unroll 1
    for (int base = 0; base < tasks; base += SLOW_PASS) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t0 = base + 16 * (int)threadIdx.x;
        unsigned slow = 0;   // bit i: flag t0 + i
        if (t0 < tasks) {
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(flags + t0));
            const unsigned words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if ((words[i >> 2] >> (8 * (i & 3))) & MASK) slow |= 1u << i;
        }
        const unsigned own = __popc(slow);
        unsigned upto = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned below = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= d) upto += below;
        }
        if (lane == 31) s_count[warp] = (unsigned short)upto;
        __syncthreads();
        unsigned rank = upto - own, total = 0;
#pragma unroll
        for (int w = 0; w < NTHREADS / 32; ++w) {
            const unsigned n = s_count[w];
            if (w < warp) rank += n;
            total += n;
        }
        // of at most 16 consecutive ranks, at most one is this CTA's: grids of fewer CTAs are not launched
        const unsigned k = rank > turn ? (rank - turn + gridDim.x - 1) / gridDim.x : 0, at = turn + k * gridDim.x - rank;
        if (at < own) {
            for (unsigned i = 0; i < at; ++i) slow &= slow - 1;
            s_list[k] = (unsigned short)(16 * threadIdx.x + __ffs(slow) - 1);
        }
        __syncthreads();
        const unsigned share = total > turn ? (total - turn - 1) / gridDim.x + 1 : 0;
#pragma unroll 1
        for (unsigned i = 0; i < share; ++i) {
            f(base + s_list[i]);
            __syncthreads();   // the next chunk's loads overwrite what this one reads
        }
        turn += share * gridDim.x - total;
    }
}

// Profiling build: thread 0 of the CTA that works on the chosen chunk records the SM clock (see SD_PHASE).
#ifdef SD_DIAGNOSTICS
#define SD_PHASE_T(g, ch, ph)                                                                                 \
    do {                                                                                                      \
        if ((g).dbg != nullptr && (int)(ch).gi == (g).dbg_block && threadIdx.x == 0 && (ph) < 16)             \
            (g).dbg[(ph)] = clock64();                                                                        \
        ++(ph);                                                                                               \
    } while (0)
#else
#define SD_PHASE_T(g, ch, ph) do { (void)(ph); } while (0)
#endif

// ---- operand tiles -----------------------------------------------------------
// K-major FP32 operand, 128-byte swizzle: tiles of 32 channels (TS bytes apart), 128-byte rows, 16-byte piece j of row i at
// piece j ^ (i mod 8).  The same tiles serve as plain panels: row-wise, lane-per-row and column accesses are all free of
// bank conflicts.
template <unsigned TS>
__device__ __forceinline__ unsigned f32_off(int i, int c) {
    return (c >> 5) * TS + i * 128 + ((((c >> 2) & 7) ^ (i & 7)) << 4) + ((c & 3) << 2);
}
// MN-major FP32 operand (the row is the contraction index): 128-byte swizzle of 32-byte atoms, atom j of row i at j ^ (i mod 4)
__device__ __forceinline__ unsigned f32_mn_off(int i, int c) {
    return (c >> 5) * F32_TILE + i * 128 + ((((c >> 3) & 3) ^ (i & 3)) << 5) + ((c & 7) << 2);
}
__device__ __forceinline__ float4 tf32_bits4(const float4& v) {   // rounded for a contraction, which cuts the low bits off
    return make_float4(__uint_as_float(mma_tf32_bits(v.x)), __uint_as_float(mma_tf32_bits(v.y)),
                       __uint_as_float(mma_tf32_bits(v.z)), __uint_as_float(mma_tf32_bits(v.w)));
}
__device__ __forceinline__ float4 pack4(const float (&x)[4]) { return make_float4(x[0], x[1], x[2], x[3]); }
__device__ __forceinline__ void unpack4(const float4& v, float (&x)[4]) { x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
__device__ __forceinline__ void unpack4(const uint2& raw, float (&x)[4]) {
    x[0] = __uint_as_float(raw.x << 16); x[1] = __uint_as_float(raw.x & 0xffff0000u);
    x[2] = __uint_as_float(raw.y << 16); x[3] = __uint_as_float(raw.y & 0xffff0000u);
}
__device__ __forceinline__ uint2 pack4_bf16(const float (&x)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x[0], x[1]), b = __floats2bfloat162_rn(x[2], x[3]);
    return make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}
// Loads that stay where they are written: a row pass requests all its rows before it uses one.  (Left to itself the compiler
// moves each load to its first use, which makes several memory latencies of one.)
__device__ __forceinline__ uint2 ld_pinned8(const void* p, bool ok) {   // zeros unless ok
    uint2 v;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t@p ld.global.v2.b32 {%0, %1}, [%2];\n\t}"
        : "=r"(v.x), "=r"(v.y)
        : "l"(p), "r"((unsigned)ok));
    return v;
}
__device__ __forceinline__ float4 ld_pinned16(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// Four channels of a BF16 row as they lie, zeros past the width and where the row is not `valid`
template <bool FAST>
__device__ __forceinline__ uint2 load4_raw(const bf16* row, int c0, int width, int vec, bool valid) {
    if (FAST) return ld_pinned8(row + c0, valid && c0 < width);
    uint2 raw = make_uint2(0u, 0u);
    if (!valid || c0 >= width) return raw;
    if (vec && c0 + 4 <= width) return *reinterpret_cast<const uint2*>(row + c0);
    const unsigned short* src = reinterpret_cast<const unsigned short*>(row) + c0;
    raw.x = src[0];
    if (c0 + 1 < width) raw.x |= (unsigned)src[1] << 16;
    if (c0 + 2 < width) raw.y = src[2];
    if (c0 + 3 < width) raw.y |= (unsigned)src[3] << 16;
    return raw;
}
// Sums over the 32 lanes of a row.  Three exchanges leave each lane with one of eight sums over a quarter of the lanes, two
// more complete it, and the sums are then fetched by lane: 9 shuffles and 8 fetches, where butterflies take 40.
__device__ __forceinline__ void row_sums32(float (&v)[8]) {
    const int lane = threadIdx.x & 31;
    float a[4], b[2];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const bool up = lane & 16;
        a[n] = (up ? v[n + 4] : v[n]) + __shfl_xor_sync(0xffffffffu, up ? v[n] : v[n + 4], 16);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const bool up = lane & 8;
        b[n] = (up ? a[n + 2] : a[n]) + __shfl_xor_sync(0xffffffffu, up ? a[n] : a[n + 2], 8);
    }
    const bool up = lane & 4;
    float c = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
#pragma unroll
    for (int n = 0; n < 8; ++n) v[n] = __shfl_sync(0xffffffffu, c, 4 * n);   // lanes 4 n .. hold sum n
}
__device__ __forceinline__ void row_sums32(float (&v)[4]) {
    const int lane = threadIdx.x & 31;
    float a[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        const bool up = lane & 16;
        a[n] = (up ? v[n + 2] : v[n]) + __shfl_xor_sync(0xffffffffu, up ? v[n] : v[n + 2], 16);
    }
    const bool up = lane & 8;
    float c = (up ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, up ? a[0] : a[1], 8);
    c += __shfl_xor_sync(0xffffffffu, c, 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
#pragma unroll
    for (int n = 0; n < 4; ++n) v[n] = __shfl_sync(0xffffffffu, c, 8 * n);
}
// ---- contractions (one thread issues) -------------------------------------------
__device__ __forceinline__ void tc_mma_ss(unsigned d_tmem, unsigned long long da, unsigned long long db, unsigned idesc,
                                          unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ unsigned long long f32_desc(unsigned addr) { return tc_desc(addr, 16, 1024) | (2ull << 61); }
__device__ __forceinline__ unsigned long long f32_mn_desc(unsigned addr) {
    return tc_desc(addr, F32_TILE, TC_R_SBO) | (1ull << 61);
}
// D[128][N] (+)= A[128][128] B[N][128]^T over K-major FP32 tiles; a descriptor counts addresses in 16-byte units
template <unsigned TSA, unsigned TSB>
__device__ __forceinline__ void mma_tf32_kk(unsigned d_tmem, unsigned a, unsigned b, int n, unsigned accumulate) {
    const unsigned id = tc_idesc(n);
    const unsigned long long da = f32_desc(a), db = f32_desc(b);
#pragma unroll
    for (int k = 0; k < DP / 8; ++k)
        tc_mma_ss(d_tmem, da + ((k / 4) * TSA + (k % 4) * 32) / 16, db + ((k / 4) * TSB + (k % 4) * 32) / 16, id,
                  k > 0 ? 1u : accumulate);
}

// ---- tensor memory, four columns at a time ---------------------------------------
__device__ __forceinline__ void tc_st4(unsigned taddr, const float (&r)[4]) {
    const unsigned* u = reinterpret_cast<const unsigned*>(r);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};" ::"r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]),
                 "r"(taddr)
                 : "memory");
}

// ---- unit-triangular solve (trisolve_blocked) --------------------------------------
// A warp's 16 right-hand-side columns in an FP32 tile: half of it, from 16-byte piece h4 on.  Columns modulo 16.
struct TileF32 {
    unsigned char* tile;
    int h4;
    __device__ __forceinline__ float* at(int i, int n) const {
        return reinterpret_cast<float*>(tile + i * 128 + (((h4 + ((n >> 2) & 3)) ^ (i & 7)) << 4) + ((n & 3) << 2));
    }
    __device__ __forceinline__ uint32_t operand(int k, int n) const { return mma_tf32_bits(*at(k, n)); }
    __device__ __forceinline__ float2 get2(int i, int n) const { return *reinterpret_cast<const float2*>(at(i, n)); }
    __device__ __forceinline__ void put2(int i, int n, float v0, float v1) const { *reinterpret_cast<float2*>(at(i, n)) = make_float2(v0, v1); }
};
// ... and in a BF16 tile: its pieces piece0 and piece0 + 1
struct TileBF16 {
    unsigned char* tile;
    int piece0;
    __device__ __forceinline__ bf16* at(int i, int n) const {
        return reinterpret_cast<bf16*>(tile + i * 128 + (((piece0 + ((n >> 3) & 1)) ^ (i & 7)) << 4) + ((n & 7) << 1));
    }
    __device__ __forceinline__ uint32_t operand(int k, int n) const { return __float_as_uint(__bfloat162float(*at(k, n))); }
    __device__ __forceinline__ float2 get2(int i, int n) const { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(at(i, n))); }
    __device__ __forceinline__ void put2(int i, int n, float v0, float v1) const {
        *reinterpret_cast<__nv_bfloat162*>(at(i, n)) = __floats2bfloat162_rn(v0, v1);
    }
};
// The warp's solved half tile to its 16 columns of a dense global panel.
template <bool TF32>
__device__ __forceinline__ void store_half_tile(const FastCta& cta, float* g, const unsigned char* tile) {
    const int j = (cta.warp & 1) * 4 + (cta.lane & 3);
#pragma unroll
    for (int it = 0; it < CL / 8; ++it) {
        const int i = it * 8 + (cta.lane >> 2);
        float4 v = *reinterpret_cast<const float4*>(tile + i * 128 + ((j ^ (i & 7)) << 4));
        if (TF32) v = make_float4(round_tf32(v.x), round_tf32(v.y), round_tf32(v.z), round_tf32(v.w));
        *reinterpret_cast<float4*>(g + i * DP + 4 * j) = v;
    }
}

}  // namespace sd
