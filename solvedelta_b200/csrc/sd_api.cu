// C ABI of the SolveDelta chunked recurrence for B200 (sm_100a).
// Declarations and the upstream interfaces they replace: include/solvedelta_b200.h
#include <cstdio>
#include <cstring>

#include "../../include/solvedelta_b200.h"
#include "sd_diagnostics.h"
#include "sd_backward.cuh"
#include "sd_backward_tc.cuh"
#include "sd_common.cuh"
#include "sd_decode.cuh"
#include "sd_forward.cuh"
#include "sd_forward_tc.cuh"
#include "sd_mixer.cuh"
#include "sd_scan_tc.cuh"
#include "sd_output_tc.cuh"
#include "sd_token.cuh"

namespace {

using namespace sd;

struct PanelDesc {
    const char* name;
    // FP32: 0 = panel [CL][DP], 1 = matrix [CL][CL], 2 = state [DP][DP], 3 = vector [DP]
    // BF16: 4 = panel, 5 = matrix, 6 = state
    int kind;
};

const PanelDesc kSaved[] = {{"Lam", 3}, {"Flags", 3}, {"G", 0}, {"Delta", 0}, {"Dprim", 0}, {"Zt", 4}, {"CtCk", 2}, {"CtCkB", 6}, {"SCk", 6},
                            {"N", 1}, {"Aed", 1}, {"Aqd", 5},
                            // BF16 source panels of the exterior, written once by the forward pass
                            {"Xg", 4}, {"Ag", 4}, {"Xr", 4}, {"Er", 4}, {"Dcol", 4}, {"DtB", 4}, {"Chi", 4}, {"Ee", 4}};
// what a call without gradients keeps of it: the panels that later forward kernels read
const PanelDesc kInfer[] = {{"Lam", 3}, {"Flags", 3}, {"G", 0}, {"Delta", 0}, {"Zt", 4}, {"CtCk", 2}, {"SCk", 6}, {"Aqd", 5}, {"Xg", 4}};
const PanelDesc kFwd[] = {{"Upd", 0}, {"Qc", 0}, {"Ubar", 0}, {"Wd", 0}, {"Ud", 0}, {"Dt", 0}};
const PanelDesc kBwd[] = {{"Pp", 4},     {"Qp", 4},     {"Dyf", 4},    {"dR", 4},     {"dSeCk", 6},
                          {"SdS", 3},    {"duPart", 4}, {"dkPart", 4}, {"dGPart", 4}, {"dDelta", 4}, {"DG", 4},
                          {"Xext", 4},   {"Dd", 4},     {"Tu", 4},   {"Khat", 4},   {"Ppp", 4},    {"Qpp", 4},    {"Rneg", 4},
                          {"dRr", 4},    {"dCeCk", 6}};

size_t kind_bytes(int kind) {
    switch (kind) {
        case 0: return size_t(CL) * DP * 4;
        case 1: return size_t(CL) * CL * 4;
        case 2: return size_t(DP) * DP * 4;
        case 3: return size_t(DP) * 4;
        case 4: return size_t(CL) * DP * 2;
        case 5: return size_t(CL) * CL * 2;
        default: return size_t(DP) * DP * 2;
    }
}

bool shape_ok(const sd_shape* s) {
    return s && s->B > 0 && s->T > 0 && s->H > 0 && s->r > 0 && s->V > 0;
}
bool shape_supported(const sd_shape* s) { return s->r <= DP && s->V <= DP; }

long long total_chunks(const sd_shape* s) {
    long long nc = (s->T + CL - 1) / CL;
    return nc * s->B * s->H;
}

template <size_t N>
size_t layout_bytes(const PanelDesc (&tab)[N], const sd_shape* s) {
    size_t chunks = (size_t)total_chunks(s), total = 0;
    for (size_t i = 0; i < N; ++i) {
        size_t bytes = kind_bytes(tab[i].kind) * chunks;
        total += (bytes + 255) & ~size_t(255);
    }
    return total;
}

template <size_t N>
bool layout_find(const PanelDesc (&tab)[N], const sd_shape* s, const char* name, size_t* off, size_t* bytes,
                 int* kind = nullptr) {
    size_t chunks = (size_t)total_chunks(s), total = 0;
    for (size_t i = 0; i < N; ++i) {
        size_t b = kind_bytes(tab[i].kind) * chunks;
        if (std::strcmp(tab[i].name, name) == 0) {
            *off = total;
            *bytes = b;
            if (kind) *kind = tab[i].kind;
            return true;
        }
        total += (b + 255) & ~size_t(255);
    }
    return false;
}

template <size_t N>
float* panel_at(const PanelDesc (&tab)[N], const sd_shape* s, void* base, const char* name) {
    size_t off = 0, bytes = 0;
    if (!layout_find(tab, s, name, &off, &bytes)) return nullptr;
    return reinterpret_cast<float*>(reinterpret_cast<char*>(base) + off);
}
template <size_t N>
bf16* bpanel_at(const PanelDesc (&tab)[N], const sd_shape* s, void* base, const char* name) {
    return reinterpret_cast<bf16*>(panel_at(tab, s, base, name));
}

Operand make_operand(const sd_operand& o, int elem_bytes) {
    Operand r;
    r.ptr = o.ptr;
    r.sb = o.stride_b;
    r.st = o.stride_t;
    r.sh = o.stride_h;
    const long long per16 = 16 / elem_bytes;
    r.vec = ((reinterpret_cast<uintptr_t>(o.ptr) & 15) == 0 && o.stride_b % per16 == 0 && o.stride_t % per16 == 0 &&
             o.stride_h % per16 == 0)
                ? 1
                : 0;
    return r;
}

#ifdef SD_DIAGNOSTICS
long long* g_dbg = nullptr;  // set by sd_debug_timeline (profiling build only)
#endif

// Fault word of the tensor-memory scan: a bounded mbarrier wait that ran out stores its code here
// (1 / 2: first / second contraction, 3: Q landed, 4: R and P landed, 5: R / P slot released);
// sd_device_fault reads it back, sd_device_fault_clear resets it.
__device__ int g_scan_fault_word = 0;
int* g_scan_fault_ptr[64] = {};
// cuTensorMapEncodeTiled is a driver function; it is reached through the runtime so that the library
// links against the runtime alone.
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                      const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                      CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TensorMapEncodeFn tensor_map_encoder() {
    static TensorMapEncodeFn encode = nullptr;
    if (encode == nullptr) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) == cudaSuccess &&
            found == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<TensorMapEncodeFn>(fn);
    }
    return encode;
}
// Tensor map of a [chunks][CL][DP] FP32 panel array: dimensions (DP, CL, chunks), box (`cols`, CL, 1).
bool make_row_map(CUtensorMap* map, const float* panels, long long chunks, int cols, CUtensorMapSwizzle swizzle) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (encode == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)DP, (cuuint64_t)CL, (cuuint64_t)chunks};
    const cuuint64_t strides[2] = {(cuuint64_t)DP * 4, (cuuint64_t)CL * DP * 4};
    const cuuint32_t box[3] = {(cuuint32_t)cols, (cuuint32_t)CL, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(panels), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of a [tasks][rows][cols] BF16 panel array for the output contraction: dimensions (cols, rows,
// tasks), box = 64 columns (128 bytes) x every row of one panel, 128-byte swizzle.
bool make_bpanel_map(CUtensorMap* map, const void* panels, long long tasks, int rows, int cols) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (encode == nullptr) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)tasks};
    const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)rows * cols * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)rows, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(panels), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The four maps of one output launch, cached per thread like the scan's.
struct OutputMaps {
    const void *xg, *aqd, *s, *zt;
    long long tasks;
    CUtensorMap xg_map, aqd_map, s_map, zt_map;
};
bool output_maps(const FwdParams& p, long long tasks, const OutputMaps** out) {
    constexpr int SLOTS = 4;
    thread_local OutputMaps cache[SLOTS] = {};
    thread_local int next = 0;
    for (int i = 0; i < SLOTS; ++i)
        if (cache[i].xg == p.Xg && cache[i].aqd == p.Aqd && cache[i].s == p.SCk && cache[i].zt == p.Zt &&
            cache[i].tasks == tasks && tasks != 0) {
            *out = &cache[i];
            return true;
        }
    OutputMaps& m = cache[next];
    next = (next + 1) % SLOTS;
    m.xg = nullptr;
    m.tasks = 0;
    if (!make_bpanel_map(&m.xg_map, p.Xg, tasks, CL, DP) || !make_bpanel_map(&m.aqd_map, p.Aqd, tasks, CL, CL) ||
        !make_bpanel_map(&m.s_map, p.SCk, tasks, DP, DP) || !make_bpanel_map(&m.zt_map, p.Zt, tasks, CL, DP))
        return false;
    m.xg = p.Xg; m.aqd = p.Aqd; m.s = p.SCk; m.zt = p.Zt; m.tasks = tasks;
    *out = &m;
    return true;
}

// The three tensor maps of one tensor-memory scan launch.  Encoding a map is a driver call; a thread that
// runs the same buffers again (a training loop on preallocated workspace, a replayed benchmark step) finds
// them in a small per-thread cache keyed on the panel pointers and the chunk count.
struct ScanMaps {
    const void *q, *r, *p;
    long long chunks;
    CUtensorMap qmap, rmap, pmap;
};
bool scan_maps(const ScanParams& sp, long long chunks, const ScanMaps** out) {
    constexpr int SLOTS = 4;
    thread_local ScanMaps cache[SLOTS] = {};
    thread_local int next = 0;
    for (int i = 0; i < SLOTS; ++i)
        if (cache[i].q == sp.Q && cache[i].r == sp.R && cache[i].p == sp.P && cache[i].chunks == chunks &&
            chunks != 0) {
            *out = &cache[i];
            return true;
        }
    ScanMaps& m = cache[next];
    next = (next + 1) % SLOTS;
    m.q = nullptr;
    m.chunks = 0;
    if (!make_row_map(&m.qmap, sp.Q, chunks, 32, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_row_map(&m.rmap, sp.R, chunks, 32, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B) ||
        !make_row_map(&m.pmap, sp.P, chunks, SCAN_NS, CU_TENSOR_MAP_SWIZZLE_NONE))
        return false;
    m.q = sp.Q; m.r = sp.R; m.p = sp.P; m.chunks = chunks;
    *out = &m;
    return true;
}

struct ScanBMaps {
    const void *q, *r, *r2, *x2, *p;
    long long chunks;
    CUtensorMap qmap, rmap, r2map, x2map, pmap;
};
bool scan_b_maps(const ScanParamsB& sp, long long chunks, const ScanBMaps** out) {
    constexpr int SLOTS = 4;
    thread_local ScanBMaps cache[SLOTS] = {};
    thread_local int next = 0;
    for (int i = 0; i < SLOTS; ++i)
        if (cache[i].q == sp.Q && cache[i].r == sp.R && cache[i].r2 == sp.R2 && cache[i].x2 == sp.X2 && cache[i].p == sp.P &&
            cache[i].chunks == chunks && chunks != 0) {
            *out = &cache[i];
            return true;
        }
    ScanBMaps& m = cache[next];
    next = (next + 1) % SLOTS;
    m.q = nullptr;
    m.chunks = 0;
    if (!make_bpanel_map(&m.qmap, sp.Q, chunks, CL, DP) || !make_bpanel_map(&m.rmap, sp.R, chunks, CL, DP) ||
        !make_bpanel_map(&m.r2map, sp.R2, chunks, CL, DP) || !make_bpanel_map(&m.x2map, sp.X2, chunks, CL, DP) ||
        !make_bpanel_map(&m.pmap, sp.P, chunks, CL, DP))
        return false;
    m.q = sp.Q; m.r = sp.R; m.r2 = sp.R2; m.x2 = sp.X2; m.p = sp.P; m.chunks = chunks;
    *out = &m;
    return true;
}

int* scan_fault_ptr() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    return g_scan_fault_ptr[dev];
}

// True when every strided operand admits 16-byte vector access and the head
// widths are multiples of eight: the kernels then use their branch-free loaders.
bool all_fast(const Operand* ops, int n, const sd_shape& s) {
    if ((s.r & 7) || (s.V & 7)) return false;
    for (int i = 0; i < n; ++i)
        if (!ops[i].vec) return false;
    return true;
}

Geometry make_geometry(const sd_shape& s) {
    Geometry g;
    g.B = s.B; g.T = s.T; g.H = s.H; g.r = s.r; g.V = s.V;
    g.NC = (s.T + CL - 1) / CL;
    g.valid = nullptr;
    g.reset = nullptr;
#ifdef SD_DIAGNOSTICS
    g.dbg = nullptr;
    g.dbg_block = 0;
#endif
    return g;
}

#ifdef SD_DIAGNOSTICS
// slot k of the diagnostic buffer belongs to the k-th launch of a step
void set_dbg(Geometry& g, int launch_index, int chunks) {
    g.dbg = g_dbg ? g_dbg + 16 * launch_index : nullptr;
    g.dbg_block = chunks > 300 ? chunks / 2 + 3 : 0;
}
long long* scan_dbg(int launch_index) { return g_dbg ? g_dbg + 16 * launch_index : nullptr; }
#else
inline void set_dbg(Geometry&, int, int) {}
inline long long* scan_dbg(int) { return nullptr; }
#endif

// A launch whose kernel may start while the one before it in the stream still runs (it waits for it itself).
cudaLaunchAttribute chained_launch() {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    return at;
}

// Launches a kernel of the operator's sequence, chained to the one before it unless it is the first of a call.
template <class... Params, class... Args>
void launch(void (*kernel)(Params...), long long grid, int threads, size_t smem, bool chained, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at = chained_launch();
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// How many segments to cut a scan into: the number with the least time by a model of what the launches were measured to
// take (us): 6.5 + steps x step for a scan or transfer pass while its CTAs fit the 148 SMs, a multiple of the steps past
// that, and 6 + 2.3 per product for the chaining in between.  A cut that gains less than a tenth is not made.  It is not
// made up to 64 chunks either: the rule depends on the number of streams, and a shard of a batch's streams is to give the
// bits of the whole batch at training lengths.  Past 24 streams the SMs are busy and nothing is cut.
constexpr float FWD_STEP_US = 2.2f, FWD_TRANSFER_US = 1.8f, BWD_STEP_US = 1.42f, BWD_TRANSFER_US = 1.18f;
int scan_segments(int streams, int NC, float step, float transfer_step) {
    constexpr int SMS = 148, MIN_CHUNKS = 64;
    if (NC <= MIN_CHUNKS) return 1;
    const auto waves = [](int ctas) { return (ctas + SMS - 1) / SMS; };
    const float whole = 6.5f + waves(2 * streams) * NC * step;
    float best = 0.9f * whole;
    int segs = 1;
    for (int g = 2; g <= NC && 2 * streams * (g - 1) <= 2 * SMS; ++g) {
        const int len = (NC + g - 1) / g;
        const float t = 13.f + len * (waves(streams * (4 * g - 6)) * transfer_step + waves(2 * streams * g) * step) + 6.f +
                        2.3f * (g - 2) * waves(streams * (DP / COMBINE_COLS));
        if (t < best) {
            best = t;
            segs = g;
        }
    }
    return segs;
}
// Cuts a scan into segments; `room`: scratch that is free while it runs, for the segment states.
template <class P>
void set_segments(P& sp, int streams, float step, float transfer_step, void* room, size_t room_bytes) {
    sp.segs = scan_segments(streams, sp.NC, step, transfer_step);
    while (sp.segs > 1 && size_t(streams) * (sp.segs - 1) * 2 * DP * DP * 4 > room_bytes) --sp.segs;
    sp.seg_len = (sp.NC + sp.segs - 1) / sp.segs;
    sp.segs = (sp.NC + sp.seg_len - 1) / sp.seg_len;   // no empty segment
    sp.seg_state = static_cast<float*>(room);
}
bool launch_scan_tc(ScanParams sp, int streams, void* room, size_t room_bytes, cudaStream_t stream, long long* dbg) {
    const ScanMaps* m = nullptr;
    if (!scan_maps(sp, (long long)streams * sp.NC, &m)) return false;
    set_segments(sp, streams, FWD_STEP_US, FWD_TRANSFER_US, room, room_bytes);
    if (sp.segs > 1) {
        launch(k_state_scan_tc<true>, streams * (sp.segs - 1) * 4, TC_THREADS, SCAN_TC_SMEM_BYTES, true, stream, sp,
               m->qmap, m->rmap, m->pmap, scan_fault_ptr(), nullptr);
        launch(k_scan_combine, streams * (DP / COMBINE_COLS), COMBINE_THREADS, COMBINE_SMEM, true, stream,
               sp.seg_state, sp.segs);
    }
    launch(k_state_scan_tc<false>, streams * sp.segs * (DP / SCAN_NS), TC_THREADS, SCAN_TC_SMEM_BYTES, true, stream, sp,
               m->qmap, m->rmap, m->pmap, scan_fault_ptr(), dbg);
    return true;
}
bool launch_scan_b(ScanParamsB sp, int streams, void* room, size_t room_bytes, cudaStream_t stream) {
    const ScanBMaps* m = nullptr;
    if (!scan_b_maps(sp, (long long)streams * sp.NC, &m)) return false;
    set_segments(sp, streams, BWD_STEP_US, BWD_TRANSFER_US, room, room_bytes);
    if (sp.segs > 1) {
        launch(k_state_scan_b<true>, streams * (sp.segs - 1) * 4, TC_THREADS, SCAN_TB_SMEM_BYTES, true, stream, sp,
               m->qmap, m->rmap, m->r2map, m->x2map, m->pmap, scan_fault_ptr());
        launch(k_scan_combine, streams * (DP / COMBINE_COLS), COMBINE_THREADS, COMBINE_SMEM, true, stream,
               sp.seg_state, sp.segs);
    }
    launch(k_state_scan_b<false>, streams * sp.segs * (DP / SCAN_NS), TC_THREADS, SCAN_TB_SMEM_BYTES, true, stream, sp,
               m->qmap, m->rmap, m->r2map, m->x2map, m->pmap, scan_fault_ptr());
    return true;
}

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Opt-in to large dynamic shared memory, once per device.  The flag array only
// caches that the (idempotent) attribute calls were made.
cudaError_t configure_kernels() {
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    if ((e = allow_smem(k_prep_fwd<true, false>, PREP_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_prep_fwd<false, false>, PREP_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_prep_fwd<true, true>, PREP_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_prep_fwd<false, true>, PREP_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_prep_fwd<false, true, true>, PREP_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_exterior_fwd<true, false>, PRIMAL_EXT_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_exterior_fwd<false, false>, PRIMAL_EXT_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_exterior_fwd<true, true>, PRIMAL_EXT_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_exterior_fwd<false, true>, PRIMAL_EXT_FWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_exterior_fwd<false, true, true>, PRIMAL_EXT_FWD_SMEM)) != cudaSuccess) return e;
#define SD_ALLOW_KINDS_OF(name, smem, F, M)                                                 \
    if ((e = allow_smem(name##_fast<F, M>, FAST_SMEM)) != cudaSuccess) return e;           \
    if ((e = allow_smem(name##_one<F, M>, smem)) != cudaSuccess) return e
#define SD_ALLOW_KINDS(name, smem)               \
    SD_ALLOW_KINDS_OF(name, smem, true, false);  \
    SD_ALLOW_KINDS_OF(name, smem, false, false); \
    SD_ALLOW_KINDS_OF(name, smem, true, true);   \
    SD_ALLOW_KINDS_OF(name, smem, false, true)
    SD_ALLOW_KINDS(k_primal_exterior, PRIMAL_EXT_FWD_SMEM);
    SD_ALLOW_KINDS(k_exterior_pair, EXT_PAIR_BWD_SMEM);
    SD_ALLOW_KINDS(k_primal, PRIMAL_BWD_SMEM);
    SD_ALLOW_KINDS(k_predictor_close, PRED_CLOSE_BWD_SMEM);
#undef SD_ALLOW_KINDS
#undef SD_ALLOW_KINDS_OF
    if ((e = allow_smem(k_state_scan_tc<false>, SCAN_TC_SMEM_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_state_scan_tc<true>, SCAN_TC_SMEM_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_output_fwd_tc<false>, OUTPUT_TC_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_output_fwd_tc<true>, OUTPUT_TC_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_decode_step<false, 1, false>, DECODE_STATE_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_decode_step<false, 1, true>, DECODE_STATE_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_decode_step<true, 1, false>, DECODE_STATE_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_decode_step<true, 1, true>, DECODE_STATE_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<2, 1, 4>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<2, 1, 8>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<2, 2, 4>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<2, 2, 8>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<1, 1, 4>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<1, 2, 4>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<1, 1, 8>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<1, 2, 8>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<1, 1, 0>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<1, 2, 0>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<2, 1, 0>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<2, 2, 0>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<4, 1, 0>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if ((e = allow_smem(k_token_linear<4, 2, 0>, TOKEN_SMEM_MAX)) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) {
        void* w = nullptr;
        if ((e = cudaGetSymbolAddress(&w, g_scan_fault_word)) != cudaSuccess) return e;
        g_scan_fault_ptr[dev] = static_cast<int*>(w);
    }
    if ((e = allow_smem(k_state_scan_b<false>, SCAN_TB_SMEM_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_state_scan_b<true>, SCAN_TB_SMEM_BYTES)) != cudaSuccess) return e;
    if ((e = allow_smem(k_scan_combine, COMBINE_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_prep_bwd<true, false>, EXT_PREP_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_prep_bwd<false, false>, EXT_PREP_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_prep_bwd<true, true>, EXT_PREP_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_prep_bwd<false, true>, EXT_PREP_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_pair_bwd<true, false>, EXT_PAIR_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_pair_bwd<false, false>, EXT_PAIR_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_pair_bwd<true, true>, EXT_PAIR_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_exterior_pair_bwd<false, true>, EXT_PAIR_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_bwd<true, false>, PRIMAL_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_bwd<false, false>, PRIMAL_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_bwd<true, true>, PRIMAL_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_bwd<false, true>, PRIMAL_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_primal_bwd<false, true, true>, PRIMAL_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_predictor_close_bwd<true, false>, PRED_CLOSE_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_predictor_close_bwd<false, false>, PRED_CLOSE_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_predictor_close_bwd<true, true>, PRED_CLOSE_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_predictor_close_bwd<false, true>, PRED_CLOSE_BWD_SMEM)) != cudaSuccess) return e;
    if ((e = allow_smem(k_predictor_close_bwd<false, true, true>, PRED_CLOSE_BWD_SMEM)) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev] = true;
    return cudaSuccess;
}

#ifdef SD_DIAGNOSTICS
// Launch recorder used by sd_profile_step only (profiling build; not thread safe).
struct LaunchRecorder {
    cudaEvent_t ev[40];
    int n;
};
LaunchRecorder* g_rec = nullptr;
inline void mark(cudaStream_t stream) {
    if (g_rec != nullptr && g_rec->n < 40) cudaEventRecord(g_rec->ev[g_rec->n++], stream);
}
#else
inline void mark(cudaStream_t) {}
#endif

#ifdef SD_DIAGNOSTICS
const char* const kLaunchNames[] = {
    "k_prep_fwd",          "k_state_scan[C]",     "k_primal_exterior_fwd", "k_state_scan[S]",
    "k_output_fwd_tc",     "k_exterior_prep_bwd", "k_state_scan_b[dS]",   "k_exterior_pair_bwd",
    "k_primal_bwd",        "k_state_scan_b[dC]",  "k_predictor_close_bwd"};
#endif

int launch_status() { return cudaGetLastError() == cudaSuccess ? SD_OK : SD_ERR_LAUNCH_FAILED; }

// One chunk kernel, instantiated for (vector-aligned operands?, token masks present?).
#define SD_LAUNCH_CHUNK(kernel, smem, chained)                                                          \
    do {                                                                                                \
        if (fast && !masked) launch(kernel<true, false>, chunks, NTHREADS, smem, chained, stream, p);   \
        else if (fast) launch(kernel<true, true>, chunks, NTHREADS, smem, chained, stream, p);          \
        else if (!masked) launch(kernel<false, false>, chunks, NTHREADS, smem, chained, stream, p);     \
        else launch(kernel<false, true>, chunks, NTHREADS, smem, chained, stream, p);                   \
    } while (0)

// The chunk kernels that come in two kinds (sd_chunk_tc.cuh).  Small calls have both kinds in one launch, NAME_one, with one CTA
// to an SM; beyond, slow chunks run with one CTA to an SM and fast ones with two, in two launches.
//   With gradients up to 32 chunks: such a call takes the host longer to issue (165 us forward and reverse) than the GPU to run,
// and four launches more cost it 9 us.  From 64 chunks on the GPU is what is waited for and the larger kernels are slower (64
// chunks 247 us of kernels against 229, 128 chunks 331 against 305, the same 195 at 32).
//   Without gradients up to 148 chunks, one to an SM: one launch less is 1 to 2 us of the call, more where few scan steps follow
// (two launches against one: 33 chunks 67 -> 65 us, 64 chunks 81 -> 70 and 95 -> 94, 128 chunks 108 -> 99 and 128 -> 127, 148
// chunks 98 -> 96).  In calls with gradients the same launch makes 1 x 1024 tokens 264 -> 272 us.
//   The slow kernel goes last, with masks too: the fast kernel starts while its predecessor ends, and the slow one may have
// nothing to do.  (Masked calls with the slow kernel first: 5 x 1531 tokens 893 us forward and reverse against 892; 881 if the
// fast CTAs then start without waiting for a predecessor whose results they read, which nothing documented allows.)
constexpr int ONE_LAUNCH_GRAD = 32, ONE_LAUNCH_NO_GRAD = 148;
#define SD_LAUNCH_KINDS_OF(name, slow_kernel, smem, limit, F, M)                                   \
    do {                                                                                           \
        if (chunks <= (limit)) {                                                                   \
            launch(name##_one<F, M>, chunks, NTHREADS, smem, true, stream, p);                     \
        } else {                                                                                   \
            launch(name##_fast<F, M>, chunks, NTHREADS, FAST_SMEM, true, stream, p);               \
            launch(slow_kernel<F, M>, chunks < 148 ? chunks : 148, NTHREADS, smem, true, stream, p, chunks); \
        }                                                                                          \
    } while (0)
#define SD_LAUNCH_KINDS(name, slow_kernel, smem, limit)                                            \
    do {                                                                                           \
        if (fast && !masked) SD_LAUNCH_KINDS_OF(name, slow_kernel, smem, limit, true, false);      \
        else if (fast) SD_LAUNCH_KINDS_OF(name, slow_kernel, smem, limit, true, true);             \
        else if (!masked) SD_LAUNCH_KINDS_OF(name, slow_kernel, smem, limit, false, false);        \
        else SD_LAUNCH_KINDS_OF(name, slow_kernel, smem, limit, false, true);                      \
    } while (0)
constexpr int KINDS_FORWARD = 1, KINDS_BACKWARD = 3;
int kind_launches(const sd_shape* s, int kinds) { return total_chunks(s) <= ONE_LAUNCH_GRAD ? 0 : kinds; }

bool operands_ok(const sd_operand* ops, int n) {
    for (int i = 0; i < n; ++i)
        if (ops[i].ptr == nullptr) return false;
    return true;
}

template <int RG, int CG, int NORM>
cudaError_t launch_token_linear(const TokenLinearParams& p, bool chained, cudaStream_t stream) {
    const int outs = p.swiglu ? p.N / 2 : p.N, width = p.swiglu ? 8 : 8 * CG, tiles = (outs + width - 1) / width;
    const size_t smem = token_smem(p.M, p.K, NORM > 0);
    const int resident = 148 * (RG <= 2 && smem <= TOKEN_SMEM_MAX / 2 ? 2 : 1);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles < resident ? tiles : resident));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at = chained_launch();
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_token_linear<RG, CG, NORM>, p);
}
template <int CG>
cudaError_t dispatch_token_linear(const TokenLinearParams& p, bool chained, cudaStream_t stream) {
    if (p.norm_w != nullptr && p.M <= 8)
        return p.K <= 1024 ? launch_token_linear<1, CG, 4>(p, chained, stream) : launch_token_linear<1, CG, 8>(p, chained, stream);
    if (p.norm_w != nullptr)
        return p.K <= 1024 ? launch_token_linear<2, CG, 4>(p, chained, stream) : launch_token_linear<2, CG, 8>(p, chained, stream);
    if (p.M <= 8) return launch_token_linear<1, CG, 0>(p, chained, stream);
    if (p.M <= 16) return launch_token_linear<2, CG, 0>(p, chained, stream);
    return launch_token_linear<4, CG, 0>(p, chained, stream);
}
int token_linear(const TokenLinearParams& p, bool chained, cudaStream_t stream) {
    // 16 columns a tile while that gives every SM one, else 8
    const cudaError_t e = p.swiglu || p.N >= 16 * 148 ? dispatch_token_linear<2>(p, chained, stream)
                                                      : dispatch_token_linear<1>(p, chained, stream);
    return e == cudaSuccess ? launch_status() : SD_ERR_LAUNCH_FAILED;
}

template <bool MIXER, int NS, bool FULL>
cudaError_t launch_decode_ns(const DecodeParams& p, const MixerDecode& m, int streams, bool chained, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(streams * NS));
    cfg.blockDim = dim3(DECODE_WARPS * 32);
    cfg.dynamicSmemBytes = NS == 1 ? DECODE_STATE_BYTES : 0;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (chained) at[n++] = chained_launch();
    if (NS > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = NS;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, k_decode_step<MIXER, NS, FULL>, p, m);
}
int add_rmsnorm(const sd_add_rmsnorm_args* a, bool chained, void* stream_) {
    if (!a || a->rows <= 0 || a->D <= 0 || !a->x || !a->weight || !a->normed || (a->delta && !a->sum))
        return SD_ERR_INVALID_ARGUMENT;
    if (a->rows > 0x7fffffffLL) return SD_ERR_UNSUPPORTED_SHAPE;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    AddNormParams p{};
    p.N = a->rows; p.D = a->D; p.eps = a->eps;
    p.x = reinterpret_cast<const __nv_bfloat16*>(a->x);
    p.delta = reinterpret_cast<const __nv_bfloat16*>(a->delta);
    p.w = a->weight;
    p.sum = reinterpret_cast<__nv_bfloat16*>(a->sum);
    p.normed = reinterpret_cast<__nv_bfloat16*>(a->normed);
    // few rows (single-token steps): a whole CTA per row finishes sooner than one warp per row
    if (addnorm_rows_ok(a->D) && (a->rows >= 1024 || !a->delta)) {
        dispatch_addnorm_rows(p, false, stream);
    } else {
        if (!a->delta) return SD_ERR_UNSUPPORTED_SHAPE;   // the norm alone is only built for the row kernels
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)a->rows);
        cfg.blockDim = dim3(256);
        cfg.stream = stream;
        cudaLaunchAttribute at = chained_launch();
        cfg.attrs = &at;
        cfg.numAttrs = chained ? 1 : 0;
        if (cudaLaunchKernelEx(&cfg, k_add_rmsnorm, p) != cudaSuccess) return SD_ERR_LAUNCH_FAILED;
    }
    return launch_status();
}

template <bool MIXER>
int launch_decode(const DecodeParams& p, const MixerDecode& m, int streams, bool chained, cudaStream_t stream) {
    if (configure_kernels() != cudaSuccess) return SD_ERR_NO_DEVICE;
    const uintptr_t states = reinterpret_cast<uintptr_t>(p.Cin) | reinterpret_cast<uintptr_t>(p.C) |
                             reinterpret_cast<uintptr_t>(p.Sin) | reinterpret_cast<uintptr_t>(p.S);
    // a full head with every row aligned: constant strides and no bounds (the operands q, k, v, ld of the mixer's step
    // are not read)
    const bool full = p.g.r == DP && p.g.V == DP && p.Cin != nullptr && p.Sin != nullptr && (states & 15) == 0 &&
                      p.u.vec && p.er.vec && p.wr.vec && (MIXER || (p.q.vec && p.k.vec && p.v.vec && p.ld.vec));
    const bool split = decode_split(streams) == 4;
    const cudaError_t e = full ? (split ? launch_decode_ns<MIXER, 4, true>(p, m, streams, chained, stream)
                                        : launch_decode_ns<MIXER, 1, true>(p, m, streams, chained, stream))
                               : (split ? launch_decode_ns<MIXER, 4, false>(p, m, streams, chained, stream)
                                        : launch_decode_ns<MIXER, 1, false>(p, m, streams, chained, stream));
    mark(stream);
    return e == cudaSuccess ? launch_status() : SD_ERR_LAUNCH_FAILED;
}

}  // namespace

extern "C" {

size_t sd_saved_bytes(const sd_shape* shape) {
    if (!shape_ok(shape) || !shape_supported(shape)) return 0;
    return layout_bytes(kSaved, shape);
}
size_t sd_inference_bytes(const sd_shape* shape) {
    if (!shape_ok(shape) || !shape_supported(shape)) return 0;
    return layout_bytes(kInfer, shape);
}
size_t sd_forward_scratch_bytes(const sd_shape* shape) {
    if (!shape_ok(shape) || !shape_supported(shape)) return 0;
    return layout_bytes(kFwd, shape);
}
size_t sd_backward_scratch_bytes(const sd_shape* shape) {
    if (!shape_ok(shape) || !shape_supported(shape)) return 0;
    return layout_bytes(kBwd, shape);
}

int sd_panel_info(const sd_shape* shape, int which, const char* name, size_t* offset, size_t* bytes) {
    if (!shape_ok(shape) || !name || !offset || !bytes) return SD_ERR_INVALID_ARGUMENT;
    if (!shape_supported(shape)) return SD_ERR_UNSUPPORTED_SHAPE;
    bool found = false;
    if (which == 0) found = layout_find(kSaved, shape, name, offset, bytes);
    if (which == 1) found = layout_find(kFwd, shape, name, offset, bytes);
    if (which == 2) found = layout_find(kBwd, shape, name, offset, bytes);
    return found ? SD_OK : SD_ERR_INVALID_ARGUMENT;
}

int sd_panel_kind(const sd_shape* shape, int which, const char* name) {
    if (!shape_ok(shape) || !name || !shape_supported(shape)) return SD_ERR_INVALID_ARGUMENT;
    size_t off = 0, bytes = 0;
    int kind = -1;
    bool found = false;
    if (which == 0) found = layout_find(kSaved, shape, name, &off, &bytes, &kind);
    if (which == 1) found = layout_find(kFwd, shape, name, &off, &bytes, &kind);
    if (which == 2) found = layout_find(kBwd, shape, name, &off, &bytes, &kind);
    return found ? kind : SD_ERR_INVALID_ARGUMENT;
}

// a scan that is cut into segments is three launches
int sd_forward_launches(const sd_shape* shape) {
    if (!shape_ok(shape)) return 0;
    return 5 + kind_launches(shape, KINDS_FORWARD) + (scan_segments(shape->B * shape->H, (shape->T + CL - 1) / CL, FWD_STEP_US, FWD_TRANSFER_US) > 1 ? 4 : 0);
}
int sd_backward_launches(const sd_shape* shape) {
    if (!shape_ok(shape)) return 0;
    return 6 + kind_launches(shape, KINDS_BACKWARD) + (scan_segments(shape->B * shape->H, (shape->T + CL - 1) / CL, BWD_STEP_US, BWD_TRANSFER_US) > 1 ? 4 : 0);
}
int sd_chunk_tokens(void) { return CL; }
int sd_version(void) { return 1; }

const char* sd_status_string(int status) {
    switch (status) {
        case SD_OK: return "ok";
        case SD_ERR_INVALID_ARGUMENT: return "invalid argument";
        case SD_ERR_UNSUPPORTED_SHAPE: return "unsupported shape (r and V must be in 1..128)";
        case SD_ERR_BUFFER_TOO_SMALL: return "saved or scratch buffer too small";
        case SD_ERR_LAUNCH_FAILED: return "CUDA launch failed";
        case SD_ERR_NO_DEVICE: return "no usable CUDA device";
        case SD_ERR_STATIC_WORKSPACE_EXCEEDED:
            return "shape needs more than SD_STATIC_WORKSPACE_BYTES of workspace: B*H*ceil(T/64) is too large for "
                   "sd_forward_static, use sd_forward with caller-provided buffers";
        default: return "unknown status";
    }
}

namespace {
// Non-null for the predictor-only entry points: the launch sequences stop after (forward) or start at
// (reverse) the predictor kernels, and the source / query rows are taken as unit vectors.
struct PredictorOnly {
    void *action, *update;                        // forward outputs, BF16 [B,T,H,r] contiguous
    const void *d_action, *d_update, *action_in;  // reverse inputs, same layout (the cotangents may be null)
};
int forward_impl(const sd_forward_args* a, void* stream_, const PredictorOnly* po, bool keep = true);
int backward_impl(const sd_backward_args* a, void* stream_, const PredictorOnly* po, int64_t qkv_pitch = 0, int64_t row_pitch = 0);
}  // namespace

int sd_forward(const sd_forward_args* a, void* stream_) { return forward_impl(a, stream_, nullptr); }
int sd_forward_inference(const sd_forward_args* a, void* stream_) { return forward_impl(a, stream_, nullptr, false); }
int sd_backward(const sd_backward_args* a, void* stream_) { return backward_impl(a, stream_, nullptr); }
int sd_backward_pitched(const sd_backward_args* a, int64_t qkv_pitch, int64_t row_pitch, void* stream_) {
    if (!a) return SD_ERR_INVALID_ARGUMENT;
    // the 16-byte stores need every row on such a boundary
    uintptr_t bits = 0;
    for (const void* q : {a->du, a->dh, a->dq, a->dkeys, a->dvalues, a->derase_raw, a->dwrite_raw}) bits |= reinterpret_cast<uintptr_t>(q);
    if ((bits & 15) != 0 || a->shape.r % 8 != 0 || a->shape.V % 8 != 0 || qkv_pitch % 8 != 0 || row_pitch % 8 != 0) return SD_ERR_UNSUPPORTED_SHAPE;
    const int64_t widest = (int64_t)a->shape.H * (a->shape.r > a->shape.V ? a->shape.r : a->shape.V);
    if (qkv_pitch < widest || row_pitch < widest) return SD_ERR_INVALID_ARGUMENT;
    return backward_impl(a, stream_, nullptr, qkv_pitch, row_pitch);
}

namespace {
int forward_impl(const sd_forward_args* a, void* stream_, const PredictorOnly* po, bool keep) {
    if (!a || !shape_ok(&a->shape)) return SD_ERR_INVALID_ARGUMENT;
    if (!shape_supported(&a->shape)) return SD_ERR_UNSUPPORTED_SHAPE;
    const sd_operand ops[] = {a->u, a->h, a->q, a->keys, a->values, a->erase_raw, a->write_raw, a->log_decay, a->gamma};
    if (!operands_ok(ops, 9) || !a->y || !a->saved || !a->scratch) return SD_ERR_INVALID_ARGUMENT;
    if (a->saved_bytes < (keep ? sd_saved_bytes(&a->shape) : sd_inference_bytes(&a->shape)) ||
        a->scratch_bytes < sd_forward_scratch_bytes(&a->shape))
        return SD_ERR_BUFFER_TOO_SMALL;
    if ((reinterpret_cast<uintptr_t>(a->saved) & 15) || (reinterpret_cast<uintptr_t>(a->scratch) & 15))
        return SD_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (configure_kernels() != cudaSuccess) return SD_ERR_NO_DEVICE;

    const sd_shape* s = &a->shape;
    FwdParams p;
    p.g = make_geometry(*s);
    p.g.valid = a->valid_mask;
    p.g.reset = a->reset_mask;
    p.u = make_operand(a->u, 2);
    p.h = make_operand(a->h, 2);
    p.q = make_operand(a->q, 2);
    p.k = make_operand(a->keys, 2);
    p.v = make_operand(a->values, 2);
    p.er = make_operand(a->erase_raw, 2);
    p.wr = make_operand(a->write_raw, 2);
    p.ld = make_operand(a->log_decay, 4);
    p.gam = make_operand(a->gamma, 4);
    p.Upd = panel_at(kFwd, s, a->scratch, "Upd");
    p.Qc = panel_at(kFwd, s, a->scratch, "Qc");
    p.Ubar = panel_at(kFwd, s, a->scratch, "Ubar");
    p.Wd = panel_at(kFwd, s, a->scratch, "Wd");
    p.Ud = panel_at(kFwd, s, a->scratch, "Ud");
    p.Dt = panel_at(kFwd, s, a->scratch, "Dt");
    const auto fp32 = [&](const char* name) {   // null where a call without gradients has no such panel
        return keep ? panel_at(kSaved, s, a->saved, name) : panel_at(kInfer, s, a->saved, name);
    };
    const auto half = [&](const char* name) { return reinterpret_cast<bf16*>(fp32(name)); };
    p.Xg = half("Xg"); p.Aqd = half("Aqd");
    p.Ag = half("Ag"); p.Xr = half("Xr"); p.Er = half("Er"); p.Dcol = half("Dcol"); p.DtB = half("DtB");
    p.Chi = half("Chi"); p.Ee = half("Ee");
    p.Npair = fp32("N"); p.Aed = fp32("Aed"); p.Dprim = fp32("Dprim");
    p.Lam = fp32("Lam"); p.Gp = fp32("G"); p.Delta = fp32("Delta"); p.CtCk = fp32("CtCk");
    p.Zt = half("Zt"); p.SCk = half("SCk");
    p.Flags = reinterpret_cast<unsigned char*>(fp32("Flags"));
    p.fault = scan_fault_ptr();
    if (p.fault == nullptr) return SD_ERR_LAUNCH_FAILED;
    p.y = a->y;
    p.action = po ? po->action : nullptr;
    p.update = po ? po->update : nullptr;

    const int chunks = (int)total_chunks(s);
    const int streams = s->B * s->H;
    const Operand fwd_ops[] = {p.u, p.h, p.q, p.k, p.v, p.er, p.wr, p.ld};
    const bool fast = all_fast(fwd_ops, 8, *s);
    const bool masked = a->valid_mask != nullptr || a->reset_mask != nullptr;

    // the segment states of a scan live in the panels of the other one: Wd, Ud, Dt (and Upd, Qc, Ubar) are neighbours in
    // the scratch, not yet written when the C scan runs (already read when the S scan runs)
    const size_t panel_bytes = kind_bytes(0) * (size_t)chunks;

    set_dbg(p.g, 0, chunks);
    if (po)   // the predictor-only instantiations: general operand layout, mask-aware (null masks are legal)
        k_prep_fwd<false, true, true><<<chunks, NTHREADS, PREP_FWD_SMEM, stream>>>(p);
    else
        SD_LAUNCH_CHUNK(k_prep_fwd, PREP_FWD_SMEM, false);
    mark(stream);
    {
        ScanParams sp{};
        sp.P = p.Upd; sp.Q = p.Qc; sp.R = p.Ubar;
        sp.lam = p.Lam; sp.X = p.Delta; sp.ck = p.CtCk; sp.Xb = nullptr;
        sp.ckb = half("CtCkB");
        sp.init = a->C0; sp.fin = a->C_T;
        sp.NC = p.g.NC; sp.transposed_io = 1; sp.nrows = s->r; sp.ncols = s->r;
        if (!launch_scan_tc(sp, streams, p.Wd, 3 * panel_bytes, stream, scan_dbg(1))) return SD_ERR_LAUNCH_FAILED;
        mark(stream);
    }
    set_dbg(p.g, 2, chunks);
    if (po) {
        k_primal_exterior_fwd<false, true, true><<<chunks, NTHREADS, PRIMAL_EXT_FWD_SMEM, stream>>>(p, chunks);
        return launch_status();   // the kernel stops after its primal half
    }
    SD_LAUNCH_KINDS(k_primal_exterior, k_primal_exterior_fwd, PRIMAL_EXT_FWD_SMEM, keep ? ONE_LAUNCH_GRAD : ONE_LAUNCH_NO_GRAD);
    mark(stream);
    {
        ScanParams sp{};
        sp.P = p.Ud; sp.Q = p.Wd; sp.R = p.Dt;
        sp.lam = p.Lam; sp.X = nullptr; sp.ck = nullptr; sp.Xb = p.Zt; sp.ckb = p.SCk;
        sp.init = a->S0; sp.fin = a->S_T;
        sp.NC = p.g.NC; sp.transposed_io = 0; sp.nrows = s->r; sp.ncols = s->V;
        if (!launch_scan_tc(sp, streams, p.Upd, 3 * panel_bytes, stream, scan_dbg(3))) return SD_ERR_LAUNCH_FAILED;
        mark(stream);
    }
    set_dbg(p.g, 4, chunks);
    {
        // the output contraction on tcgen05, its panels landed by tiled TMA loads
        const OutputMaps* m = nullptr;
        int* fault = scan_fault_ptr();
        if (fault == nullptr || !output_maps(p, total_chunks(s), &m)) return SD_ERR_LAUNCH_FAILED;
        if (masked)
            launch(k_output_fwd_tc<true>, chunks, OUT_TC_THREADS, OUTPUT_TC_SMEM, true, stream, p, m->xg_map, m->aqd_map,
                   m->s_map, m->zt_map, fault);
        else
            launch(k_output_fwd_tc<false>, chunks, OUT_TC_THREADS, OUTPUT_TC_SMEM, true, stream, p, m->xg_map, m->aqd_map,
                   m->s_map, m->zt_map, fault);
    }
    mark(stream);
    return launch_status();
}

int backward_impl(const sd_backward_args* a, void* stream_, const PredictorOnly* po, int64_t qkv_pitch, int64_t row_pitch) {
    if (!a || !shape_ok(&a->shape)) return SD_ERR_INVALID_ARGUMENT;
    if (!shape_supported(&a->shape)) return SD_ERR_UNSUPPORTED_SHAPE;
    const sd_operand ops[] = {a->u,         a->h,         a->q,         a->keys,  a->values,
                              a->erase_raw, a->write_raw, a->log_decay, a->gamma, a->dy};
    if (!operands_ok(ops, 10) || !a->saved || !a->scratch) return SD_ERR_INVALID_ARGUMENT;
    if (!a->du || !a->dh || !a->dq || !a->dkeys || !a->dvalues || !a->derase_raw || !a->dwrite_raw ||
        !a->dlog_decay || !a->dgamma)
        return SD_ERR_INVALID_ARGUMENT;
    if (a->saved_bytes < sd_saved_bytes(&a->shape) || a->scratch_bytes < sd_backward_scratch_bytes(&a->shape))
        return SD_ERR_BUFFER_TOO_SMALL;
    if ((reinterpret_cast<uintptr_t>(a->saved) & 15) || (reinterpret_cast<uintptr_t>(a->scratch) & 15))
        return SD_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    if (configure_kernels() != cudaSuccess) return SD_ERR_NO_DEVICE;

    const sd_shape* s = &a->shape;
    BwdParams p;
    p.g = make_geometry(*s);
    p.g.valid = a->valid_mask;
    p.g.reset = a->reset_mask;
    p.u = make_operand(a->u, 2);
    p.h = make_operand(a->h, 2);
    p.q = make_operand(a->q, 2);
    p.k = make_operand(a->keys, 2);
    p.v = make_operand(a->values, 2);
    p.er = make_operand(a->erase_raw, 2);
    p.wr = make_operand(a->write_raw, 2);
    p.ld = make_operand(a->log_decay, 4);
    p.gam = make_operand(a->gamma, 4);
    p.dy = make_operand(a->dy, 2);
    void* sv = const_cast<void*>(a->saved);
    p.Flags = reinterpret_cast<const unsigned char*>(panel_at(kSaved, s, sv, "Flags"));
    p.fault = scan_fault_ptr();
    if (p.fault == nullptr) return SD_ERR_LAUNCH_FAILED;
    p.Lam = panel_at(kSaved, s, sv, "Lam");
    p.Gp = panel_at(kSaved, s, sv, "G");
    p.Delta = panel_at(kSaved, s, sv, "Delta");
    p.Dprim = panel_at(kSaved, s, sv, "Dprim");
    p.Zt = bpanel_at(kSaved, s, sv, "Zt");
    p.CtCk = panel_at(kSaved, s, sv, "CtCk");
    p.CtCkB = bpanel_at(kSaved, s, sv, "CtCkB");
    p.SCk = bpanel_at(kSaved, s, sv, "SCk");
    p.Npair = panel_at(kSaved, s, sv, "N");
    p.Aed = panel_at(kSaved, s, sv, "Aed");
    p.Aqd = bpanel_at(kSaved, s, sv, "Aqd");
#define SD_BP(field) p.field = panel_at(kBwd, s, a->scratch, #field)
#define SD_BB(field) p.field = bpanel_at(kBwd, s, a->scratch, #field)
    SD_BB(Pp); SD_BB(Qp); SD_BB(Dyf); SD_BB(dR); SD_BB(dSeCk);
    p.Xg = bpanel_at(kSaved, s, sv, "Xg");
    p.Ag = bpanel_at(kSaved, s, sv, "Ag");
    p.Xr = bpanel_at(kSaved, s, sv, "Xr");
    p.Er = bpanel_at(kSaved, s, sv, "Er");
    p.Dcol = bpanel_at(kSaved, s, sv, "Dcol");
    p.DtB = bpanel_at(kSaved, s, sv, "DtB");
    p.Chi = bpanel_at(kSaved, s, sv, "Chi");
    p.Ee = bpanel_at(kSaved, s, sv, "Ee");
    SD_BB(DG); SD_BB(Dd); SD_BB(Tu); SD_BB(Khat);
    SD_BB(Ppp); SD_BB(Qpp); SD_BB(Rneg); SD_BB(dRr); SD_BB(dCeCk);
    SD_BB(duPart); SD_BB(dkPart); SD_BB(dGPart); SD_BB(dDelta); SD_BB(Xext); SD_BP(SdS);
#undef SD_BB
#undef SD_BP
    p.du = a->du; p.dh = a->dh; p.dq = a->dq; p.dk = a->dkeys; p.dv = a->dvalues;
    p.pitch_q = qkv_pitch ? qkv_pitch : (int64_t)s->H * s->r;
    p.pitch_v = qkv_pitch ? qkv_pitch : (int64_t)s->H * s->V;
    p.pitch_u = row_pitch ? row_pitch : (int64_t)s->H * s->r;
    p.pitch_w = row_pitch ? row_pitch : (int64_t)s->H * s->V;
    p.der = a->derase_raw; p.dwr = a->dwrite_raw; p.dld = a->dlog_decay; p.dgam = a->dgamma;

    const int chunks = (int)total_chunks(s);
    const int streams = s->B * s->H;
    // segment states: the dS scan's in duPart .. Xext (neighbours, not yet written), the dC scan's in Pp .. dR (already read)
    const size_t bpanel_bytes = kind_bytes(4) * (size_t)chunks;
    const Operand bwd_ops[] = {p.u, p.h, p.q, p.k, p.v, p.er, p.wr, p.ld, p.dy};
    const bool fast = all_fast(bwd_ops, 9, *s);
    const bool masked = a->valid_mask != nullptr || a->reset_mask != nullptr;

    if (po) {
        // cotangents of the frame action and of the update from the caller: contiguous [B,T,H,r] BF16
        auto dense = [&](const void* ptr) {
            sd_operand o;
            o.ptr = ptr;
            o.stride_h = s->r;
            o.stride_t = (int64_t)s->H * s->r;
            o.stride_b = (int64_t)s->T * s->H * s->r;
            Operand op = make_operand(o, 2);
            if (ptr == nullptr) op.vec = 0;
            return op;
        };
        const Operand dact = dense(po->d_action), dupd = dense(po->d_update), act = dense(po->action_in);
        if (masked)
            k_predictor_seed_bwd<true><<<chunks, NTHREADS, 0, stream>>>(p, dact, dupd, act);
        else
            k_predictor_seed_bwd<false><<<chunks, NTHREADS, 0, stream>>>(p, dact, dupd, act);
    } else {
    set_dbg(p.g, 5, chunks);
    SD_LAUNCH_CHUNK(k_exterior_prep_bwd, EXT_PREP_BWD_SMEM, false);
    mark(stream);
    {
        ScanParamsB sp{};
        sp.P = p.Pp; sp.Q = p.Qp; sp.R = p.Ag; sp.R2 = p.Xg; sp.X2 = p.Dyf;
        sp.lam = p.Lam; sp.X = p.dR; sp.ck = p.dSeCk;
        sp.init = a->dS_T; sp.fin = a->dS0;
        sp.NC = p.g.NC; sp.transposed_io = 0; sp.nrows = s->r; sp.ncols = s->V;
        if (!launch_scan_b(sp, streams, p.duPart, 6 * bpanel_bytes, stream)) return SD_ERR_LAUNCH_FAILED;
    mark(stream);
    }
    set_dbg(p.g, 7, chunks);
    SD_LAUNCH_KINDS(k_exterior_pair, k_exterior_pair_bwd, EXT_PAIR_BWD_SMEM, ONE_LAUNCH_GRAD);
    mark(stream);
    }
    set_dbg(p.g, 8, chunks);
    if (po)
        k_primal_bwd<false, true, true><<<chunks, NTHREADS, PRIMAL_BWD_SMEM, stream>>>(p, chunks);
    else
        SD_LAUNCH_KINDS(k_primal, k_primal_bwd, PRIMAL_BWD_SMEM, ONE_LAUNCH_GRAD);
    mark(stream);
    {
        ScanParamsB sp{};
        sp.P = p.Ppp; sp.Q = p.Qpp; sp.R = p.Rneg; sp.R2 = p.DG; sp.X2 = p.Khat;
        sp.lam = p.Lam; sp.X = p.dRr; sp.ck = p.dCeCk;
        sp.init = a->dC_T; sp.fin = a->dC0;
        sp.NC = p.g.NC; sp.transposed_io = 1; sp.nrows = s->r; sp.ncols = s->r;
        if (!launch_scan_b(sp, streams, p.Pp, 4 * bpanel_bytes, stream)) return SD_ERR_LAUNCH_FAILED;
    mark(stream);
    }
    set_dbg(p.g, 10, chunks);
    if (po)
        k_predictor_close_bwd<false, true, true><<<chunks, NTHREADS, PRED_CLOSE_BWD_SMEM, stream>>>(p, chunks);
    else
        SD_LAUNCH_KINDS(k_predictor_close, k_predictor_close_bwd, PRED_CLOSE_BWD_SMEM, ONE_LAUNCH_GRAD);
    mark(stream);
    return launch_status();
}
}  // namespace

// ---- predictor-only entry points ------------------------------------------------------------------
// The argument blocks of the full operator are reused: operands the predictor kernels never read
// (q, values, gate logits, y and their gradients) point at the query / at scratch outputs.
int sd_predictor_forward(const sd_predictor_forward_args* a, void* stream_) {
    if (!a || !a->frame_action || !a->update) return SD_ERR_INVALID_ARGUMENT;
    sd_forward_args f{};
    f.shape = a->shape;
    f.shape.V = a->shape.r;
    f.u = a->source; f.h = a->target; f.keys = a->query;
    f.q = f.values = f.erase_raw = f.write_raw = a->query;   // never read by the predictor kernels
    f.log_decay = a->log_decay; f.gamma = a->beta;
    f.C0 = a->C0; f.S0 = nullptr;
    f.y = a->frame_action; f.C_T = a->C_T; f.S_T = nullptr;
    f.saved = a->saved; f.saved_bytes = a->saved_bytes;
    f.scratch = a->scratch; f.scratch_bytes = a->scratch_bytes;
    f.valid_mask = a->valid_mask; f.reset_mask = a->reset_mask;
    PredictorOnly po{a->frame_action, a->update, nullptr, nullptr, nullptr};
    return forward_impl(&f, stream_, &po);
}

int sd_predictor_backward(const sd_predictor_backward_args* a, void* stream_) {
    if (!a || !a->frame_action || !a->dtarget || !a->dsource || !a->dquery || !a->dbeta || !a->dlog_decay)
        return SD_ERR_INVALID_ARGUMENT;
    sd_backward_args b{};
    b.shape = a->shape;
    b.shape.V = a->shape.r;
    b.u = a->source; b.h = a->target; b.keys = a->query;
    b.q = b.values = b.erase_raw = b.write_raw = b.dy = a->query;   // never read by the predictor kernels
    b.log_decay = a->log_decay; b.gamma = a->beta;
    b.dC_T = a->dC_T; b.dS_T = nullptr;
    b.saved = a->saved; b.saved_bytes = a->saved_bytes;
    b.scratch = a->scratch; b.scratch_bytes = a->scratch_bytes;
    b.du = a->dsource; b.dh = a->dtarget; b.dkeys = a->dquery;
    b.dq = b.dvalues = b.derase_raw = b.dwrite_raw = a->dquery;     // never written by the predictor kernels
    b.dlog_decay = a->dlog_decay; b.dgamma = a->dbeta;
    b.dC0 = a->dC0; b.dS0 = nullptr;
    b.valid_mask = a->valid_mask; b.reset_mask = a->reset_mask;
    PredictorOnly po{nullptr, nullptr, a->d_frame_action, a->d_update, a->frame_action};
    return backward_impl(&b, stream_, &po);
}

#ifdef SD_DIAGNOSTICS
void sd_debug_timeline(void* device_buffer) { g_dbg = reinterpret_cast<long long*>(device_buffer); }

static __global__ void k_debug_elementwise(int function, const float* x, float* y, long long count) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
        y[i] = function == 0 ? exp_ftz(x[i]) : function == 1 ? rcp_ftz(x[i]) : __uint_as_float(mma_tf32_bits(x[i]) & 0xffffe000u);
}
int sd_debug_elementwise(int function, const float* x, float* y, long long count, void* stream_) {
    if (function < 0 || function > 2 || !x || !y || count < 1) return SD_ERR_INVALID_ARGUMENT;
    k_debug_elementwise<<<256, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(function, x, y, count);
    return launch_status();
}
#endif

int sd_device_fault(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    int word = 0;
    if (cudaMemcpyFromSymbol(&word, g_scan_fault_word, sizeof(int)) != cudaSuccess) return -1;
    return word;
}

int sd_device_fault_clear(void) {
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    const int zero = 0;
    return cudaMemcpyToSymbol(g_scan_fault_word, &zero, sizeof(int)) == cudaSuccess ? 0 : -1;
}

#ifdef SD_DIAGNOSTICS
const char* sd_launch_name(int index) {
    const int n = (int)(sizeof(kLaunchNames) / sizeof(kLaunchNames[0]));
    return (index >= 0 && index < n) ? kLaunchNames[index] : "";
}

int sd_profile_step(const sd_forward_args* fwd, const sd_backward_args* bwd, void* stream_, float* ms,
                    int capacity, int* count) {
    if (!fwd || !ms || !count || capacity < 11) return SD_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    LaunchRecorder rec;
    rec.n = 0;
    for (int i = 0; i < 40; ++i)
        if (cudaEventCreate(&rec.ev[i]) != cudaSuccess) return SD_ERR_NO_DEVICE;
    cudaEventRecord(rec.ev[rec.n++], stream);
    g_rec = &rec;
    int status = sd_forward(fwd, stream_);
    if (status == SD_OK && bwd != nullptr) status = sd_backward(bwd, stream_);
    g_rec = nullptr;
    cudaError_t e = cudaStreamSynchronize(stream);
    *count = 0;
    if (status == SD_OK && e == cudaSuccess) {
        for (int i = 1; i < rec.n && i - 1 < capacity; ++i) {
            cudaEventElapsedTime(&ms[i - 1], rec.ev[i - 1], rec.ev[i]);
            *count = i;
        }
    }
    for (int i = 0; i < 40; ++i) cudaEventDestroy(rec.ev[i]);
    if (e != cudaSuccess) return SD_ERR_LAUNCH_FAILED;
    return status;
}

#endif  // SD_DIAGNOSTICS

// ---------------------------------------------------------------------------
// Forward pass on library-owned scratch, for hosts that must not allocate.
// The workspace of sd_forward (the `saved` and `scratch` regions) lives in one
// file-scope device array; its device address is looked up once per device.
static __device__ __align__(256) unsigned char g_static_workspace[SD_STATIC_WORKSPACE_BYTES];

int sd_forward_static(const sd_forward_args* a, void* stream_) {
    if (!a || !shape_ok(&a->shape)) return SD_ERR_INVALID_ARGUMENT;
    if (!shape_supported(&a->shape)) return SD_ERR_UNSUPPORTED_SHAPE;
    const size_t saved_bytes = sd_saved_bytes(&a->shape);
    const size_t scratch_bytes = sd_forward_scratch_bytes(&a->shape);
    if (saved_bytes + scratch_bytes > (size_t)SD_STATIC_WORKSPACE_BYTES) return SD_ERR_STATIC_WORKSPACE_EXCEEDED;
    // In host code the array's name is only a handle; kernels need the device
    // address, which differs per GPU.  Resolve it with that GPU current.
    static void* base_of_device[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SD_ERR_NO_DEVICE;
    if (base_of_device[dev] == nullptr) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_static_workspace) != cudaSuccess || ptr == nullptr) {
            cudaGetLastError();
            return SD_ERR_NO_DEVICE;
        }
        base_of_device[dev] = ptr;
    }
    sd_forward_args local = *a;
    local.saved = base_of_device[dev];
    local.saved_bytes = saved_bytes;
    local.scratch = static_cast<unsigned char*>(base_of_device[dev]) + saved_bytes;
    local.scratch_bytes = scratch_bytes;
    // Every panel of the workspace is written in full before any kernel reads
    // it, so nothing left by an earlier call has to be cleared.
    return sd_forward(&local, stream_);
}

// ---------------------------------------------------------------------------
// Mixer glue
namespace {
int conv_tiles(int T) { return (T + CONV_TT - 1) / CONV_TT; }
// Rows of a CTA of the gate's reverse kernel.  A thread walks its rows one load latency after the other, so they are
// halved while the CTAs do not reach every SM (1024 x 1024: 34 to 9 us).  More CTAs than that only add partial sums: at
// 16384 rows the kernel took 42 instead of 44 us and the sums 4 us more.
int gate_rows_per_block(int64_t rows) {
    int n = 64;
    while (n > 8 && rows / n < 148) n /= 2;
    return n;
}
constexpr int NORM_ROWS_PER_BLOCK = 256;
size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
}  // namespace

size_t sd_conv4_backward_scratch_bytes(int32_t B, int32_t T, int32_t D) {
    if (B <= 0 || T <= 0 || D <= 0) return 0;
    return align256(size_t(B) * conv_tiles(T) * D * 4 * sizeof(float));
}

// channel pairs can move as 4-byte accesses: even widths and strides, 4-byte aligned bases
static bool conv_pairs_ok(const ConvParams& p) {
    auto al = [](const void* q) { return q == nullptr || (reinterpret_cast<uintptr_t>(q) & 3) == 0; };
    return (p.D & 1) == 0 && (p.sb & 1) == 0 && (p.st & 1) == 0 && (p.dxt & 1) == 0 && al(p.x) && al(p.y) && al(p.dy) && al(p.dx);
}

int sd_conv4_silu_forward(const sd_conv4_forward_args* a, void* stream_) {
    if (!a || a->B <= 0 || a->T <= 0 || a->D <= 0 || !a->x || !a->weight || !a->y) return SD_ERR_INVALID_ARGUMENT;
    ConvParams p{};
    p.B = a->B; p.T = a->T; p.D = a->D;
    p.x = reinterpret_cast<const __nv_bfloat16*>(a->x);
    p.sb = a->x_stride_b; p.st = a->x_stride_t;
    p.w = a->weight;
    p.init = reinterpret_cast<const __nv_bfloat16*>(a->initial_state);
    p.y = reinterpret_cast<__nv_bfloat16*>(a->y);
    p.fin = reinterpret_cast<__nv_bfloat16*>(a->final_state);
    p.valid = a->valid_mask; p.reset = a->reset_mask;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    dim3 grid((a->D + 2 * CONV_THREADS - 1) / (2 * CONV_THREADS), conv_tiles(a->T), a->B);
    const bool masked = p.valid != nullptr || p.reset != nullptr;
    if (conv_pairs_ok(p)) {
        if (masked) k_conv4_silu_fwd_masked<true><<<grid, CONV_THREADS, 0, stream>>>(p);
        else k_conv4_silu_fwd<true><<<grid, CONV_THREADS, 0, stream>>>(p);
    } else {
        if (masked) k_conv4_silu_fwd_masked<false><<<grid, CONV_THREADS, 0, stream>>>(p);
        else k_conv4_silu_fwd<false><<<grid, CONV_THREADS, 0, stream>>>(p);
    }
    return launch_status();
}

int sd_conv4_silu_backward(const sd_conv4_backward_args* a, void* stream_) {
    return a ? sd_conv4_silu_backward_pitched(a, a->D, stream_) : SD_ERR_INVALID_ARGUMENT;
}
int sd_conv4_silu_backward_pitched(const sd_conv4_backward_args* a, int64_t dx_pitch, void* stream_) {
    if (!a || dx_pitch < a->D || a->B <= 0 || a->T <= 0 || a->D <= 0 || !a->x || !a->weight || !a->dy || !a->dx || !a->dweight ||
        !a->scratch)
        return SD_ERR_INVALID_ARGUMENT;
    if (a->scratch_bytes < sd_conv4_backward_scratch_bytes(a->B, a->T, a->D)) return SD_ERR_BUFFER_TOO_SMALL;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    ConvParams p{};
    p.B = a->B; p.T = a->T; p.D = a->D;
    p.x = reinterpret_cast<const __nv_bfloat16*>(a->x);
    p.sb = a->x_stride_b; p.st = a->x_stride_t;
    p.w = a->weight;
    p.init = reinterpret_cast<const __nv_bfloat16*>(a->initial_state);
    p.dy = reinterpret_cast<const __nv_bfloat16*>(a->dy);
    p.dx = reinterpret_cast<__nv_bfloat16*>(a->dx);
    p.dxt = dx_pitch;
    p.dinit = reinterpret_cast<__nv_bfloat16*>(a->dinitial_state);
    p.dw_part = reinterpret_cast<float*>(a->scratch);
    p.valid = a->valid_mask; p.reset = a->reset_mask;
    const int tiles = conv_tiles(a->T);
    dim3 grid((a->D + 2 * CONV_THREADS - 1) / (2 * CONV_THREADS), tiles, a->B);
    const bool masked = p.valid != nullptr || p.reset != nullptr;
    if (conv_pairs_ok(p)) {
        if (masked) k_conv4_silu_bwd_masked<true><<<grid, CONV_THREADS, 0, stream>>>(p);
        else k_conv4_silu_bwd<true><<<grid, CONV_THREADS, 0, stream>>>(p);
    } else {
        if (masked) k_conv4_silu_bwd_masked<false><<<grid, CONV_THREADS, 0, stream>>>(p);
        else k_conv4_silu_bwd<false><<<grid, CONV_THREADS, 0, stream>>>(p);
    }
    const long long n = (long long)a->D * 4;
    launch_column_sum(p.dw_part, a->B * tiles, n, a->dweight, stream);
    return launch_status();
}

size_t sd_kda_gate_backward_scratch_bytes(int64_t rows, int32_t H, int32_t r) {
    if (rows <= 0 || H <= 0 || r <= 0) return 0;
    const int per_block = gate_rows_per_block(rows);
    const size_t blocks = size_t((rows + per_block - 1) / per_block);
    return align256((2 * blocks + 1) * size_t(H) * r * sizeof(float));
}

int sd_kda_gate_forward(const sd_kda_gate_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->H <= 0 || a->r <= 0 || !a->raw || !a->log_rate || !a->bias || !a->log_decay)
        return SD_ERR_INVALID_ARGUMENT;
    GateParams p{};
    p.N = a->rows; p.H = a->H; p.r = a->r;
    p.raw = reinterpret_cast<const __nv_bfloat16*>(a->raw);
    p.A = a->log_rate; p.bias = a->bias; p.out = a->log_decay;
    const long long total = a->rows * a->H * a->r;
    const bool vec = (a->r & 7) == 0 && ((reinterpret_cast<uintptr_t>(a->raw) | reinterpret_cast<uintptr_t>(a->bias) |
                                          reinterpret_cast<uintptr_t>(a->log_decay)) & 15) == 0;
    long long blocks = (total + 256 * 8 - 1) / (256 * 8);
    if (blocks > 148 * 32) blocks = 148 * 32;
    if (vec)
        k_kda_gate_fwd_v8<<<(unsigned)(blocks ? blocks : 1), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    else
        k_kda_gate_fwd<<<(unsigned)(blocks ? blocks : 1), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

int sd_kda_gate_backward(const sd_kda_gate_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->H <= 0 || a->r <= 0 || !a->raw || !a->log_rate || !a->bias || !a->dlog_decay ||
        !a->draw || !a->dlog_rate || !a->dbias || !a->scratch)
        return SD_ERR_INVALID_ARGUMENT;
    const int HR = a->H * a->r;
    if (a->scratch_bytes < sd_kda_gate_backward_scratch_bytes(a->rows, a->H, a->r)) return SD_ERR_BUFFER_TOO_SMALL;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    const int per_block = gate_rows_per_block(a->rows), blocks = (int)((a->rows + per_block - 1) / per_block);
    GateParams p{};
    p.N = a->rows; p.H = a->H; p.r = a->r;
    p.raw = reinterpret_cast<const __nv_bfloat16*>(a->raw);
    p.A = a->log_rate; p.bias = a->bias; p.dout = a->dlog_decay;
    p.draw = reinterpret_cast<__nv_bfloat16*>(a->draw);
    p.dbias_part = reinterpret_cast<float*>(a->scratch);
    p.dA_part = p.dbias_part + (size_t)blocks * HR;
    float* dA_cols = p.dA_part + (size_t)blocks * HR;
    p.rows_per_block = per_block;
    const bool vec = (a->r & 7) == 0 &&
                     ((reinterpret_cast<uintptr_t>(a->raw) | reinterpret_cast<uintptr_t>(a->bias) |
                       reinterpret_cast<uintptr_t>(a->dlog_decay) | reinterpret_cast<uintptr_t>(a->draw)) & 15) == 0;
    if (vec) {
        int cgb = HR / 8;   // column groups per CTA: a power of two that divides 256, or 256
        if (cgb >= 256) cgb = 256;
        else { int q = 1; while (q * 2 <= cgb) q *= 2; cgb = q; }
        k_kda_gate_bwd_v8<<<dim3(blocks, (HR / 8 + cgb - 1) / cgb), 256, 0, stream>>>(p, cgb);
    } else {
        k_kda_gate_bwd<<<dim3(blocks, (HR + 255) / 256), 256, 0, stream>>>(p);
    }
    launch_column_sum(p.dbias_part, blocks, HR, a->dbias, stream);
    launch_column_sum(p.dA_part, blocks, HR, dA_cols, stream);
    k_group_sum<<<a->H, 32, 0, stream>>>(dA_cols, a->H, a->r, a->dlog_rate);
    return launch_status();
}

// rows of a CTA when they make less than one wave of three CTAs an SM: whole steps of 16, at least two
static int64_t norm_rows_few(int64_t rows) {
    const int64_t n = (rows + 148 * 3 - 1) / (148 * 3);
    return n > NORM_ROWS_PER_BLOCK ? NORM_ROWS_PER_BLOCK : n < 32 ? 32 : (n + 15) / 16 * 16;
}
size_t sd_norm_gate_backward_scratch_bytes(int64_t rows, int32_t V) {
    if (rows <= 0 || V <= 0) return 0;
    const size_t blocks = std::max(size_t((rows + NORM_ROWS_PER_BLOCK - 1) / NORM_ROWS_PER_BLOCK),
                                   size_t((rows + norm_rows_few(rows) - 1) / norm_rows_few(rows)));
    return align256(blocks * size_t(V) * sizeof(float));
}

int sd_norm_gate_forward(const sd_norm_gate_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->V <= 0 || !a->x || !a->gate || !a->weight || !a->y) return SD_ERR_INVALID_ARGUMENT;
    if (a->V > DP) return SD_ERR_UNSUPPORTED_SHAPE;
    NormParams p{};
    p.N = a->rows; p.V = a->V; p.eps = a->eps;
    p.x = reinterpret_cast<const __nv_bfloat16*>(a->x);
    p.gate = reinterpret_cast<const __nv_bfloat16*>(a->gate);
    p.w = a->weight;
    p.out = reinterpret_cast<__nv_bfloat16*>(a->y);
    long long blocks = (a->rows + 15) / 16;
    const long long wave = resident_ctas(k_norm_gate_fwd, 256, 0);   // one wave: a CTA carries its next rows
    if (blocks > wave) blocks = wave;
    k_norm_gate_fwd<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

int sd_norm_gate_backward(const sd_norm_gate_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->V <= 0 || !a->x || !a->gate || !a->weight || !a->dy || !a->dx || !a->dgate ||
        !a->dweight || !a->scratch)
        return SD_ERR_INVALID_ARGUMENT;
    if (a->V > DP) return SD_ERR_UNSUPPORTED_SHAPE;
    if (a->scratch_bytes < sd_norm_gate_backward_scratch_bytes(a->rows, a->V)) return SD_ERR_BUFFER_TOO_SMALL;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    // rows per CTA: NORM_ROWS_PER_BLOCK or more, stretched so that the grid is a whole number of waves of resident CTAs;
    // fewer when they would not fill one wave (the scratch is sized for both)
    long long rpb = NORM_ROWS_PER_BLOCK;
    {
        const long long wave = resident_ctas(k_norm_gate_bwd, 256, 0);
        const long long waves = a->rows / (wave * NORM_ROWS_PER_BLOCK);
        if (waves >= 1) rpb = ((a->rows + wave * waves - 1) / (wave * waves) + 15) / 16 * 16;
        if (rpb < NORM_ROWS_PER_BLOCK) rpb = NORM_ROWS_PER_BLOCK;
        if (waves < 1) rpb = norm_rows_few(a->rows);
    }
    const int blocks = (int)((a->rows + rpb - 1) / rpb);
    NormParams p{};
    p.N = a->rows; p.V = a->V; p.eps = a->eps;
    p.x = reinterpret_cast<const __nv_bfloat16*>(a->x);
    p.gate = reinterpret_cast<const __nv_bfloat16*>(a->gate);
    p.w = a->weight;
    p.dout = reinterpret_cast<const __nv_bfloat16*>(a->dy);
    p.dx = reinterpret_cast<__nv_bfloat16*>(a->dx);
    p.dgate = reinterpret_cast<__nv_bfloat16*>(a->dgate);
    p.dw_part = reinterpret_cast<float*>(a->scratch);
    p.rows_per_block = (int)rpb;
    k_norm_gate_bwd<<<blocks, 256, 0, stream>>>(p);
    launch_column_sum(p.dw_part, blocks, a->V, a->dweight, stream);
    return launch_status();
}

int sd_add_rmsnorm(const sd_add_rmsnorm_args* a, void* stream_) { return add_rmsnorm(a, false, stream_); }
int sd_add_rmsnorm_chained(const sd_add_rmsnorm_args* a, void* stream_) { return add_rmsnorm(a, true, stream_); }

size_t sd_add_rmsnorm_backward_scratch_bytes(int64_t rows, int32_t D) {
    if (rows <= 0 || D <= 0) return 0;
    return align256(size_t(addnorm_blocks(rows)) * size_t(D) * sizeof(float));
}

int sd_add_rmsnorm_backward(const sd_add_rmsnorm_backward_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->D <= 0 || !a->sum || !a->weight || !a->dnormed || !a->dx || !a->dweight || !a->scratch)
        return SD_ERR_INVALID_ARGUMENT;
    if (!addnorm_rows_ok(a->D)) return SD_ERR_UNSUPPORTED_SHAPE;
    if (a->scratch_bytes < sd_add_rmsnorm_backward_scratch_bytes(a->rows, a->D)) return SD_ERR_BUFFER_TOO_SMALL;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    AddNormParams p{};
    p.N = a->rows; p.D = a->D; p.eps = a->eps;
    p.sum = const_cast<__nv_bfloat16*>(reinterpret_cast<const __nv_bfloat16*>(a->sum));
    p.w = a->weight;
    p.dsum = reinterpret_cast<const __nv_bfloat16*>(a->dsum);
    p.dnormed = reinterpret_cast<const __nv_bfloat16*>(a->dnormed);
    p.dx = reinterpret_cast<__nv_bfloat16*>(a->dx);
    p.dw_part = reinterpret_cast<float*>(a->scratch);
    const unsigned blocks = dispatch_addnorm_rows(p, true, stream);
    launch_column_sum(p.dw_part, (int)blocks, a->D, a->dweight, stream);
    return launch_status();
}

static unsigned swiglu_blocks(const sd_swiglu_args* a) {
    long long blocks = (a->rows * ((a->I + 7) / 8) + 255) / 256;
    return (unsigned)(blocks > 148 * 32 ? 148 * 32 : blocks);
}

int sd_swiglu(const sd_swiglu_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->I <= 0 || !a->gate_value || !a->out) return SD_ERR_INVALID_ARGUMENT;
    SwigluParams p{};
    p.N = a->rows; p.I = a->I;
    p.in = reinterpret_cast<const __nv_bfloat16*>(a->gate_value);
    p.out = reinterpret_cast<__nv_bfloat16*>(a->out);
    k_swiglu<<<swiglu_blocks(a), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

int sd_swiglu_backward(const sd_swiglu_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->I <= 0 || !a->gate_value || !a->dout || !a->dgate_value) return SD_ERR_INVALID_ARGUMENT;
    SwigluParams p{};
    p.N = a->rows; p.I = a->I;
    p.in = reinterpret_cast<const __nv_bfloat16*>(a->gate_value);
    p.dout = reinterpret_cast<const __nv_bfloat16*>(a->dout);
    p.din = reinterpret_cast<__nv_bfloat16*>(a->dgate_value);
    k_swiglu_bwd<<<swiglu_blocks(a), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

int sd_cross_entropy_forward(const sd_cross_entropy_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->V <= 0 || !a->logits || !a->labels || !a->lse || !a->row_loss) return SD_ERR_INVALID_ARGUMENT;
    if (a->rows > 0x7fffffffLL) return SD_ERR_UNSUPPORTED_SHAPE;
    CrossEntropyParams p{};
    p.N = a->rows; p.V = a->V; p.ignore_index = a->ignore_index;
    p.logits = reinterpret_cast<const __nv_bfloat16*>(a->logits);
    p.labels = reinterpret_cast<const long long*>(a->labels);
    p.lse = a->lse; p.row_loss = a->row_loss;
    k_cross_entropy_fwd<<<(unsigned)a->rows, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

int sd_cross_entropy_backward(const sd_cross_entropy_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->V <= 0 || !a->logits || !a->labels || !a->lse || !a->coef || !a->dlogits)
        return SD_ERR_INVALID_ARGUMENT;
    if (a->rows > 0x7fffffffLL) return SD_ERR_UNSUPPORTED_SHAPE;
    CrossEntropyParams p{};
    p.N = a->rows; p.V = a->V; p.ignore_index = a->ignore_index;
    p.logits = reinterpret_cast<const __nv_bfloat16*>(a->logits);
    p.labels = reinterpret_cast<const long long*>(a->labels);
    p.lse = a->lse; p.coef = a->coef;
    p.dlogits = reinterpret_cast<__nv_bfloat16*>(a->dlogits);
    k_cross_entropy_bwd<<<(unsigned)a->rows, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

int sd_gemv(const sd_gemv_args* a, void* stream_) {
    if (!a || a->M <= 0 || a->N <= 0 || a->K <= 0 || !a->x || !a->weight || !a->y) return SD_ERR_INVALID_ARGUMENT;
    if (a->M > 4) return SD_ERR_UNSUPPORTED_SHAPE;
    sd_token_linear_args t{};
    t.M = a->M; t.N = a->N; t.K = a->K; t.swiglu = a->swiglu;
    t.x = a->x; t.x_stride = a->x_stride; t.weight = a->weight; t.bias = a->bias; t.y = a->y; t.y_stride = a->y_stride;
    return sd_token_linear(&t, stream_);
}

int sd_token_linear(const sd_token_linear_args* a, void* stream_) {
    if (!a || a->M <= 0 || a->N <= 0 || a->K <= 0 || !a->x || !a->weight || !a->y) return SD_ERR_INVALID_ARGUMENT;
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (a->M > TOKEN_MAX_ROWS || a->K % 8 != 0 || a->x_stride % 8 != 0 || (a->swiglu && a->N % 2 != 0) || !al(a->x) ||
        !al(a->weight))
        return SD_ERR_UNSUPPORTED_SHAPE;
    if (a->norm_weight != nullptr) {
        if (a->delta != nullptr && a->sum == nullptr) return SD_ERR_INVALID_ARGUMENT;
        if (a->M > TOKEN_NORM_MAX_ROWS || a->K > TOKEN_NORM_MAX_K || !al(a->norm_weight) || !al(a->delta) || !al(a->sum))
            return SD_ERR_UNSUPPORTED_SHAPE;
    }
    if (token_smem(a->M, a->K, a->norm_weight != nullptr) > TOKEN_SMEM_MAX) return SD_ERR_UNSUPPORTED_SHAPE;
    if (configure_kernels() != cudaSuccess) return SD_ERR_NO_DEVICE;
    TokenLinearParams p{};
    p.M = a->M; p.N = a->N; p.K = a->K; p.swiglu = a->swiglu ? 1 : 0;
    p.x = reinterpret_cast<const __nv_bfloat16*>(a->x); p.x_stride = a->x_stride;
    p.W = reinterpret_cast<const __nv_bfloat16*>(a->weight);
    p.bias = reinterpret_cast<const __nv_bfloat16*>(a->bias);
    p.y = reinterpret_cast<__nv_bfloat16*>(a->y); p.y_stride = a->y_stride;
    p.delta = a->norm_weight ? reinterpret_cast<const __nv_bfloat16*>(a->delta) : nullptr;
    p.norm_w = a->norm_weight; p.eps = a->norm_eps;
    p.sum = reinterpret_cast<__nv_bfloat16*>(a->sum);
    return token_linear(p, a->chained != 0, reinterpret_cast<cudaStream_t>(stream_));
}

int sd_pack_rows(const sd_pack_rows_args* a, void* stream_) {
    if (!a || a->rows <= 0 || a->pieces <= 0 || a->pieces > SD_PACK_MAX_PIECES || a->row_width <= 0 || !a->dst)
        return SD_ERR_INVALID_ARGUMENT;
    PackRowsParams p{};
    p.N = a->rows; p.pieces = a->pieces; p.row_width = a->row_width;
    p.dst = reinterpret_cast<__nv_bfloat16*>(a->dst);
    long long total = 0;
    for (int k = 0; k < a->pieces; ++k) {
        if (a->piece[k].width <= 0) return SD_ERR_INVALID_ARGUMENT;
        // 16-byte groups: widths in whole groups of eight channels, sources on 16-byte boundaries
        if (a->piece[k].width % 8 != 0 || (reinterpret_cast<uintptr_t>(a->piece[k].src) & 15) != 0)
            return SD_ERR_UNSUPPORTED_SHAPE;
        p.src[k] = reinterpret_cast<const __nv_bfloat16*>(a->piece[k].src);
        p.width[k] = a->piece[k].width;
        total += a->piece[k].width;
    }
    if (total > a->row_width) return SD_ERR_INVALID_ARGUMENT;
    if (a->row_width % 8 != 0 || (reinterpret_cast<uintptr_t>(a->dst) & 15) != 0) return SD_ERR_UNSUPPORTED_SHAPE;
    const unsigned gx = (unsigned)((a->row_width / 8 + 255) / 256);
    long long gy = (148 * 8 + gx - 1) / gx;
    if (gy > a->rows) gy = a->rows;
    k_pack_rows<<<dim3(gx, (unsigned)gy), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(p);
    return launch_status();
}

static int decode_impl(const sd_decode_args* a, const float* C_in, const float* S_in, void* stream_) {
    if (!a || !shape_ok(&a->shape) || a->shape.T != 1) return SD_ERR_INVALID_ARGUMENT;
    if (!shape_supported(&a->shape)) return SD_ERR_UNSUPPORTED_SHAPE;
    const sd_operand ops[] = {a->u, a->h, a->q, a->keys, a->values, a->erase_raw, a->write_raw, a->log_decay, a->gamma};
    if (!operands_ok(ops, 9) || !a->C || !a->S || !a->y) return SD_ERR_INVALID_ARGUMENT;
    DecodeParams p;
    p.g = make_geometry(a->shape);
    p.u = make_operand(a->u, 2);
    p.h = make_operand(a->h, 2);
    p.q = make_operand(a->q, 2);
    p.k = make_operand(a->keys, 2);
    p.v = make_operand(a->values, 2);
    p.er = make_operand(a->erase_raw, 2);
    p.wr = make_operand(a->write_raw, 2);
    p.ld = make_operand(a->log_decay, 4);
    p.gam = make_operand(a->gamma, 4);
    p.Cin = C_in;
    p.Sin = S_in;
    p.C = a->C;
    p.S = a->S;
    p.y = a->y;
    return launch_decode<false>(p, MixerDecode{}, a->shape.B * a->shape.H, false, reinterpret_cast<cudaStream_t>(stream_));
}

int sd_decode_step(const sd_decode_args* a, void* stream_) {
    return a ? decode_impl(a, a->C, a->S, stream_) : SD_ERR_INVALID_ARGUMENT;
}

int sd_decode_step_from(const sd_decode_args* a, const float* C_in, const float* S_in, void* stream_) {
    return decode_impl(a, C_in, S_in, stream_);
}

static int mixer_decode_impl(const sd_mixer_decode_args* a, bool chained, void* stream_) {
    if (!a || !shape_ok(&a->shape) || a->shape.T != 1) return SD_ERR_INVALID_ARGUMENT;
    if (!shape_supported(&a->shape)) return SD_ERR_UNSUPPORTED_SHAPE;
    const sd_operand ops[] = {a->u, a->h, a->erase_raw, a->write_raw};
    if (!operands_ok(ops, 4) || !a->C || !a->S || !a->y || !a->qkv || !a->conv_weight || !a->conv_state ||
        !a->log_rate || !a->decay_bias || !a->geometry_raw || !a->geometry_bias)
        return SD_ERR_INVALID_ARGUMENT;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
    DecodeParams p{};
    p.g = make_geometry(a->shape);
    p.u = make_operand(a->u, 2);
    p.h = make_operand(a->h, 2);
    p.er = make_operand(a->erase_raw, 2);
    p.wr = make_operand(a->write_raw, 2);
    p.q = p.k = p.v = p.u;       // unused by the fused instantiation
    p.ld = p.gam = p.u;
    p.Cin = p.C = a->C;
    p.Sin = p.S = a->S;
    p.y = a->y;
    MixerDecode m{};
    m.qkv = reinterpret_cast<const __nv_bfloat16*>(a->qkv);
    m.qkv_sb = a->qkv_stride_b;
    m.conv_w = a->conv_weight;
    m.conv_state = reinterpret_cast<__nv_bfloat16*>(a->conv_state);
    m.decay_raw = reinterpret_cast<const __nv_bfloat16*>(a->decay_raw);
    m.decay_sb = a->decay_stride_b;
    m.log_rate = a->log_rate;
    m.decay_bias = a->decay_bias;
    m.geom_raw = reinterpret_cast<const __nv_bfloat16*>(a->geometry_raw);
    m.geom_sb = a->geometry_stride_b;
    m.geom_bias = a->geometry_bias;
    m.norm_w = a->norm_weight;
    m.norm_eps = a->norm_eps;
    m.gate = reinterpret_cast<const __nv_bfloat16*>(a->output_gate);
    m.gate_sb = a->output_gate_stride_b;
    m.G = a->gate_rank;
    m.decay_hidden = reinterpret_cast<const __nv_bfloat16*>(a->decay_hidden);
    m.decay_w = reinterpret_cast<const __nv_bfloat16*>(a->decay_proj_weight);
    m.dh_sb = a->decay_hidden_stride_b;
    m.gate_hidden = reinterpret_cast<const __nv_bfloat16*>(a->gate_hidden);
    m.gate_w = reinterpret_cast<const __nv_bfloat16*>(a->gate_proj_weight);
    m.gate_b = reinterpret_cast<const __nv_bfloat16*>(a->gate_proj_bias);
    m.gh_sb = a->gate_hidden_stride_b;
    if ((m.decay_w != nullptr) != (m.gate_w != nullptr)) return SD_ERR_INVALID_ARGUMENT;   // both or neither
    if (m.decay_w != nullptr) {
        auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
        if (m.G <= 0 || m.G > DP || (m.G & 15) || !m.decay_hidden || !m.gate_hidden || !al(m.decay_w) || !al(m.gate_w))
            return SD_ERR_INVALID_ARGUMENT;
        if (m.norm_w == nullptr) return SD_ERR_INVALID_ARGUMENT;   // the fused gate projection feeds the fused norm
    } else if (m.decay_raw == nullptr) {
        return SD_ERR_INVALID_ARGUMENT;
    }
    if (m.norm_w != nullptr && m.gate == nullptr && m.gate_w == nullptr) return SD_ERR_INVALID_ARGUMENT;
    auto al8 = [](const void* q, long long stride) { return (reinterpret_cast<uintptr_t>(q) & 7) == 0 && (stride & 3) == 0; };
    m.hid_vec = al8(m.decay_hidden, m.dh_sb) && al8(m.gate_hidden, m.gh_sb);
    return launch_decode<true>(p, m, a->shape.B * a->shape.H, chained, stream);
}

int sd_mixer_decode_step(const sd_mixer_decode_args* a, void* stream_) { return mixer_decode_impl(a, false, stream_); }
int sd_mixer_decode_step_chained(const sd_mixer_decode_args* a, void* stream_) { return mixer_decode_impl(a, true, stream_); }

}  // extern "C"
