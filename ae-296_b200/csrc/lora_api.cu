// extern "C" entry points declared in include/b200_lora.h: argument checks and launches only.
#include <string.h>

#include <cstdlib>
#include <mutex>

#include "lora_common.cuh"

using namespace b200lora;

namespace {

thread_local char g_last_error[256] = "";

int cuda_fail(cudaError_t e) {
    strncpy(g_last_error, cudaGetErrorString(e), sizeof(g_last_error) - 1);
    return B200_LORA_ERR_CUDA;
}

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

// ---- tensor maps for the TMA kernels --------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
        tried = true;
    }
    return fn;
}

// 2-D map over a row-major 16-bit matrix [rows, inner] with row pitch `pitch` elements;
// cached per (base, shape, box)
bool tensor_map_2d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint32_t box_inner,
                   uint32_t box_rows, CUtensorMapSwizzle swizzle, uint64_t pitch = 0,
                   CUtensorMapL2promotion promote = CU_TENSOR_MAP_L2_PROMOTION_L2_256B) {
    if (pitch == 0) pitch = inner;
    // Encoded maps are kept in a hashed, 4-way set-associative table (4096 entries): an eager loop over
    // many layers presents a few hundred (base pointer, shape) keys per step, and a look-up touches one set.
    struct Entry { const void* base; uint64_t inner, rows, pitch; uint32_t bi, br; int sw; int promote; bool used; CUtensorMap map; };
    constexpr int kSets = 1024, kWays = 4;
    static Entry cache[kSets][kWays];
    static unsigned char victim[kSets];
    static std::mutex mu;
    uint64_t h = reinterpret_cast<uintptr_t>(base) >> 4;
    h = (h ^ (inner * 0x9E3779B97F4A7C15ull) ^ (rows * 0xC2B2AE3D27D4EB4Full) ^ (pitch << 21) ^ ((uint64_t)box_inner << 40) ^
         ((uint64_t)box_rows << 48) ^ ((uint64_t)swizzle << 56)) * 0xFF51AFD7ED558CCDull;
    const int set_idx = (int)((h >> 40) % kSets);
    Entry* set = cache[set_idx];
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < kWays; ++i) {
        const Entry& e = set[i];
        if (e.used && e.base == base && e.inner == inner && e.rows == rows && e.pitch == pitch && e.bi == box_inner &&
            e.br == box_rows && e.sw == (int)swizzle && e.promote == (int)promote) { *out = e.map; return true; }
    }
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    alignas(64) CUtensorMap m;
    cuuint64_t dims[2] = {inner, rows};
    cuuint64_t strides[1] = {pitch * 2};
    cuuint32_t box[2] = {box_inner, box_rows};
    cuuint32_t estr[2] = {1, 1};
    if (fn(&m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promote,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    int way = -1;
    for (int i = 0; i < kWays && way < 0; ++i)
        if (!set[i].used) way = i;
    if (way < 0) {                                          // a full set: its ways are replaced in turn
        way = victim[set_idx];
        victim[set_idx] = (unsigned char)((way + 1) % kWays);
    }
    Entry& e = set[way];
    e.base = base; e.inner = inner; e.rows = rows; e.pitch = pitch; e.bi = box_inner; e.br = box_rows; e.sw = (int)swizzle;
    e.promote = (int)promote;
    e.used = true; e.map = m;
    *out = m;
    return true;
}

// The tile kernels (tall runs) and the BGMV kernels (everything else) of one apply touch disjoint
// rows of y, v and the split-K partials, so they run as two chains: the tiles on a side stream
// that forks from the caller's stream and joins it again before the call returns.  Each chain is
// a string of short dependent launches whose start-up and tail leave SMs idle; the other chain's
// CTAs fill them.  One side stream per host thread and device, created on first use (outside
// stream capture: a first use inside a capture runs the two chains one after the other).
struct SideStream {
    cudaStream_t stream;
    cudaEvent_t fork, join;
    int state;                // 0 not tried, 1 ready, -1 unavailable
};
SideStream* side_stream(cudaStream_t caller) {
    static const bool serial = [] { const char* v = getenv("B200_LORA_SERIAL_TILES"); return v && v[0] == '1'; }();
    if (serial) return nullptr;
    thread_local SideStream side[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    SideStream& ss = side[dev];
    if (ss.state == 0) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(caller, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return nullptr;                                  // try again on a later call
        }
        const bool ok = cudaStreamCreateWithFlags(&ss.stream, cudaStreamNonBlocking) == cudaSuccess &&
                        cudaEventCreateWithFlags(&ss.fork, cudaEventDisableTiming) == cudaSuccess &&
                        cudaEventCreateWithFlags(&ss.join, cudaEventDisableTiming) == cudaSuccess;
        if (!ok) cudaGetLastError();
        ss.state = ok ? 1 : -1;
    }
    return ss.state == 1 ? &ss : nullptr;
}

// rows of an A pool viewed as a [rows, h_in] matrix
uint64_t pool_rows(const b200_lora_adapters* ad) {
    if (!ad->packed) return (uint64_t)ad->n_adapters * ad->n_layers * ad->r_pool;
    if (ad->total_rank > 0) return (uint64_t)ad->total_rank * ad->n_layers;
    return (uint64_t)ad->n_adapters * ad->n_layers * kMaxRank;       // upper bound
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_adapters(const b200_lora_adapters* ad) {
    if (!ad) return B200_LORA_ERR_NULL;
    if (ad->n_adapters < 1 || ad->n_layers < 1) return B200_LORA_ERR_DIM;
    if (ad->r_pool < 1 || ad->r_pool > kMaxRank) return B200_LORA_ERR_RANK;
    if (ad->packed) {
        if (!ad->cum_ranks || !ad->ranks) return B200_LORA_ERR_NULL;
    } else if (ad->r_pool % 8) {
        return B200_LORA_ERR_RANK;     // rows of the dense B pool must stay 16-byte aligned
    }
    return B200_LORA_OK;
}

// true when the TMA kernels may be used as far as ranks are concerned
bool fast_ranks(const b200_lora_adapters* ad) {
    const int r = ad->r_pool;
    const bool pow2 = (r == 8 || r == 16 || r == 32 || r == 64);
    if (!ad->packed && !ad->ranks) return pow2;
    return ad->ranks_pow2 != 0 && (ad->packed || pow2);
}

// Does the one-launch cluster kernel take this apply?  Yes while all its clusters (at most a segment per
// token, times the projections) run at once: each is a chain that is much longer than its bytes take, and a
// second round of clusters would pay the chain again, while the two streaming kernels only get longer.
// Microseconds per apply, two kernels / cluster kernel, distinct adapters, weights from HBM, graph replay; items =
// tokens x projections.  bgmv_cluster_limit() is the item count of the last column that is inside the rule:
//   h 4096, r 16 (3 CTAs an SM):  1 item 5.5 / 3.6   24 items 7.2 / 4.2   46 items 8.5 / 6.3   limit 48: 8.5 / 6.8   beyond, 64: 9.7 / 10.5
//   h 2048, r 64 (2 CTAs an SM):  1 item 6.1 / 4.7   24 items 8.6 / 6.3   31 items 9.4 / 7.2   limit 33: 9.5 / 8.4   beyond, 36: 10.2 / 11.7
//   h 4096, r 64 (1 CTA an SM):   1 item 6.8 / 5.0   12 items 9.1 / 6.4   13 items 9.3 / 6.6   limit 15: 9.7 / 6.9   beyond, 16: 10.4 / 11.9
// The limit is the right line at the other sizes too: h 4096, r 32 (33): 9.2 / 8.1; h 8192, r 16 (33): 9.4 / 8.8;
// h 5120, r 32 (15): 8.2 / 5.6; h 4096 to 1024, r 64 (15): 8.5 / 5.9; three projections, r 16 (48): 8.5 / 6.8; and with
// few adapters, whose clusters are fewer than the items (weights in L2): 8 tokens of one, h 1024 to 8192, r 64: 5.85 / 5.80;
// r 16: 5.2 / 4.2.
bool cluster_route(const ApplyParams& p, const b200_lora_adapters* ad, int io_dtype) {
    if (p.n_tokens > kClusterTokens) return false;                   // beyond any limit, and what the plan has room for
    const int other = B200_LORA_ONLY_SHRINK | B200_LORA_ONLY_EXPAND | B200_LORA_DELTA_THEN_ADD;
    if (!(p.flags & B200_LORA_NO_TENSOR) || (p.flags & other) || !fast_ranks(ad) || !bgmv_cluster_fits(p)) return false;
    // a cluster writes its y rows while others still read x: not when the two share memory
    for (int i = 0; i < p.n_proj; ++i)
        for (int j = 0; j < p.n_proj; ++j) {
            const ProjArgs &a = p.proj[i], &b = p.proj[j];
            const uintptr_t x0 = reinterpret_cast<uintptr_t>(a.x), y0 = reinterpret_cast<uintptr_t>(b.y);
            const uintptr_t x1 = x0 + 2 * ((uintptr_t)(p.n_tokens - 1) * a.ldx + a.h_in);
            const uintptr_t y1 = y0 + (p.y_f32 ? 4 : 2) * ((uintptr_t)(p.n_tokens - 1) * b.ldy + b.h_out);
            if (x0 < y1 && y0 < x1) return false;
        }
    return p.n_tokens * p.n_proj <= bgmv_cluster_limit(p, io_dtype);
}

// the workspace's sticky error word as a status code
int status_of_error_word(unsigned word) {
    if (word == 0u) return B200_LORA_OK;
    return word >= kErrPlanMismatch ? B200_LORA_ERR_DIM : B200_LORA_ERR_TIMEOUT;
}

PlanAdapters plan_adapters(const b200_lora_adapters* ad) {
    PlanAdapters pa;
    pa.ranks = ad->ranks;
    pa.cum_ranks = ad->packed ? reinterpret_cast<const long long*>(ad->cum_ranks) : nullptr;
    pa.scalings = ad->scalings;
    pa.scale = ad->scale;
    pa.r_pool = ad->r_pool;
    pa.n_adapters = ad->n_adapters;
    pa.ranks_pow2 = fast_ranks(ad) ? 1 : 0;
    return pa;
}

}  // namespace

// Scratch for b200_add_lora_bgmv_static: plan + workspace of the largest accepted call.  It
// lives in the library image, so every GPU that loads the library carries it until exit.
static __device__ __align__(256) unsigned char g_static_scratch[B200_LORA_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_mu;
void* g_static_ptr[64] = {nullptr};      // device address of the array, per device (guarded by the mutex)
size_t g_static_last_pb[64] = {0};       // plan bytes of the last static call, per device

// One-time set-up per device: in host code `g_static_scratch` is only a stand-in for the device
// array, so its device address has to be asked for, with that device current.
int static_scratch_address(void** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e);
    if (dev < 0 || dev >= 64) return B200_LORA_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e);
        g_static_ptr[dev] = ptr;
    }
    *out = g_static_ptr[dev];
    return B200_LORA_OK;
}
}  // namespace

extern "C" {

int b200_lora_arch(void) { return 100; }

const char* b200_lora_last_cuda_error(void) { return g_last_error; }

int b200_lora_stream_capture_id(void* stream, unsigned long long* id) {
    if (!id) return B200_LORA_ERR_NULL;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    unsigned long long cid = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(static_cast<cudaStream_t>(stream), &st, &cid);
    if (e != cudaSuccess) return cuda_fail(e);
    *id = st == cudaStreamCaptureStatusActive ? cid : 0ull;
    return B200_LORA_OK;
}

size_t b200_lora_plan_bytes(int32_t max_tokens, int32_t n_adapters) {
    if (max_tokens < 1 || n_adapters < 1) return 0;
    return plan_words(max_tokens, n_adapters) * 4;
}

static int plan_build(void* plan, size_t plan_bytes, int32_t max_tokens, const void* ids, int32_t ids_are_i64, int32_t n_tokens,
                      const b200_lora_adapters* adapters, void* clear, size_t clear_bytes, void* stream) {
    if (!plan || !ids) return B200_LORA_ERR_NULL;
    int rc = check_adapters(adapters);
    if (rc) return rc;
    if (n_tokens < 1 || n_tokens > max_tokens) return B200_LORA_ERR_DIM;
    const int cap = max_tokens;
    if (plan_bytes < b200_lora_plan_bytes(cap, adapters->n_adapters)) return B200_LORA_ERR_WORKSPACE;
    if (!aligned16(plan)) return B200_LORA_ERR_ALIGN;
    cudaError_t e = launch_plan_build(plan, cap, ids, ids_are_i64, n_tokens, plan_adapters(adapters), clear, clear_bytes,
                                      static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_plan_build(void* plan, size_t plan_bytes, int32_t max_tokens, const void* ids,
                         int32_t ids_are_i64, int32_t n_tokens, const b200_lora_adapters* adapters,
                         void* stream) {
    return plan_build(plan, plan_bytes, max_tokens, ids, ids_are_i64, n_tokens, adapters, nullptr, 0, stream);
}

static int plan_from_segments(void* plan, size_t plan_bytes, int32_t max_tokens, const int32_t* seg_starts, const int32_t* seg_adapter,
                              int32_t n_segs, int32_t n_tokens, int last_end_given, const b200_lora_adapters* adapters, void* stream) {
    if (!plan || !seg_starts || !seg_adapter) return B200_LORA_ERR_NULL;
    int rc = check_adapters(adapters);
    if (rc) return rc;
    if (n_tokens < 1 || n_tokens > max_tokens || n_segs < 1 || n_segs > n_tokens) return B200_LORA_ERR_DIM;
    const int cap = max_tokens;
    if (plan_bytes < b200_lora_plan_bytes(cap, adapters->n_adapters)) return B200_LORA_ERR_WORKSPACE;
    if (!aligned16(plan)) return B200_LORA_ERR_ALIGN;
    cudaError_t e = launch_plan_from_segments(plan, cap, seg_starts, seg_adapter, n_segs, n_tokens, last_end_given,
                                              plan_adapters(adapters), static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_plan_from_segments(void* plan, size_t plan_bytes, int32_t max_tokens,
                                 const int32_t* seg_starts, const int32_t* seg_adapter, int32_t n_segs,
                                 int32_t n_tokens, const b200_lora_adapters* adapters, void* stream) {
    return plan_from_segments(plan, plan_bytes, max_tokens, seg_starts, seg_adapter, n_segs, n_tokens, 1, adapters, stream);
}

int b200_lora_plan_from_requests(void* plan, size_t plan_bytes, int32_t max_tokens,
                                 const int32_t* start_loc, const int32_t* lora_ids, int32_t n_requests,
                                 int32_t n_tokens, const b200_lora_adapters* adapters, void* stream) {
    return plan_from_segments(plan, plan_bytes, max_tokens, start_loc, lora_ids, n_requests, n_tokens, 0, adapters, stream);
}

int b200_lora_plan_read(const void* plan, int32_t* perm, int32_t* seg_starts, int32_t* seg_adapter,
                        int32_t* n_segs, int32_t* n_tokens, void* stream) {
    if (!plan || !n_segs || !n_tokens) return B200_LORA_ERR_NULL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    PlanHeader h;
    cudaError_t e = cudaMemcpyAsync(&h, plan, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e);
    *n_segs = h.n_segs;
    *n_tokens = h.n_tokens;
    if (h.error == 1) return B200_LORA_ERR_ID_RANGE;
    if (h.error == 3) return B200_LORA_ERR_RANK;
    if (h.error) return B200_LORA_ERR_SEGMENTS;
    PlanView pv = plan_view(const_cast<void*>(plan), h.cap, h.n_adapters);
    if (perm) e = cudaMemcpyAsync(perm, pv.perm, 4 * (size_t)h.n_tokens, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && seg_starts)
        e = cudaMemcpyAsync(seg_starts, pv.seg_start, 4 * (size_t)(h.n_segs + 1), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && seg_adapter)
        e = cudaMemcpyAsync(seg_adapter, pv.seg_adapter, 4 * (size_t)h.n_segs, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

size_t b200_lora_workspace_bytes(int32_t max_tokens, int32_t n_proj, int32_t max_h_in) {
    if (max_tokens < 1 || n_proj < 1 || n_proj > kMaxProj || max_h_in < 8) return 0;
    return workspace_bytes(max_tokens, n_proj, max_h_in);
}

int b200_lora_workspace_init(void* workspace, size_t bytes, void* stream) {
    if (!workspace) return B200_LORA_ERR_NULL;
    if (bytes < sizeof(WorkspaceCtl)) return B200_LORA_ERR_WORKSPACE;
    cudaError_t e = cudaMemsetAsync(workspace, 0, bytes, static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

static bool tp_usable(const b200_lora_tp* tp) {
    if (tp->tp < 2 || tp->tp > B200_LORA_TP_MAX_RANKS || tp->rank < 0 || tp->rank >= tp->tp || tp->set_stride == 0) return false;
    for (int r = 0; r < tp->tp; ++r)
        if (!tp->landing[r][0] || !tp->landing[r][1] || !tp->flags[r]) return false;
    return true;
}

// One apply.  With `direct_ids` the plan buffer holds no plan: the cluster kernel works from the ids, or
// nothing is launched (B200_LORA_ERR_UNSUPPORTED).  With `tp` it is the tensor-parallel form: each chain (the tiles on the side stream,
// the BGMV kernels on the caller's) runs its shrink half, the exchange of its own rows of v over
// the ranks, and its expand half.
static int apply_core(const b200_lora_proj* projs, int32_t n_proj, const b200_lora_adapters* adapters,
                      const void* plan, int32_t max_tokens, int32_t n_tokens, int32_t layer, int32_t io_dtype,
                      int32_t y_dtype, int32_t flags, void* workspace, size_t workspace_bytes_, void* stream,
                      const b200_lora_tp* tp, int skip_arrival, const void* direct_ids = nullptr, int direct_i64 = 0) {
    if (!projs || !plan || !workspace) return B200_LORA_ERR_NULL;
    if (tp && !tp_usable(tp)) return B200_LORA_ERR_DIM;
    if (tp && (flags & (B200_LORA_ONLY_SHRINK | B200_LORA_ONLY_EXPAND))) return B200_LORA_ERR_DIM;
    int rc = check_adapters(adapters);
    if (rc) return rc;
    if (n_proj < 1 || n_proj > kMaxProj || max_tokens < 1 || n_tokens < 1 || n_tokens > max_tokens) return B200_LORA_ERR_DIM;
    if (io_dtype != B200_LORA_F16 && io_dtype != B200_LORA_BF16) return B200_LORA_ERR_DTYPE;
    if (y_dtype != io_dtype && y_dtype != B200_LORA_F32) return B200_LORA_ERR_DTYPE;
    if (layer < 0 || layer >= adapters->n_layers) return B200_LORA_ERR_LAYER;
    if (flags & B200_LORA_OVERWRITE) {
        if (tp || (flags & (B200_LORA_ONLY_SHRINK | B200_LORA_ONLY_EXPAND))) return B200_LORA_ERR_DIM;
        flags &= ~B200_LORA_DELTA_THEN_ADD;                 // the same on a y of zeros
    }
    if (!aligned16(plan) || !aligned16(workspace)) return B200_LORA_ERR_ALIGN;

    ApplyParams p;
    memset(&p, 0, sizeof(p));
    int max_h_in = 0;
    for (int i = 0; i < n_proj; ++i) {
        const b200_lora_proj& q = projs[i];
        if (!q.x || !q.y || !q.wa || !q.wb) return B200_LORA_ERR_NULL;
        if (q.h_in < 8 || q.h_out < 8 || (q.h_in % 8) || (q.h_out % 8)) return B200_LORA_ERR_DIM;
        if (q.ldx < q.h_in || q.ldy < q.h_out || (q.ldx % 8) || (q.ldy % 8)) return B200_LORA_ERR_DIM;
        if (!aligned16(q.x) || !aligned16(q.y) || !aligned16(q.wa) || !aligned16(q.wb)) return B200_LORA_ERR_ALIGN;
        ProjArgs& a = p.proj[i];
        a.x = q.x; a.y = q.y; a.wa = q.wa; a.wb = q.wb;
        a.ldx = q.ldx; a.ldy = q.ldy; a.h_in = q.h_in; a.h_out = q.h_out;
        a.n_super_in = (q.h_in + kSuper - 1) / kSuper;
        a.n_super_out = (q.h_out + kSuper - 1) / kSuper;
        p.total_super_in += a.n_super_in;
        p.total_super_out += a.n_super_out;
        if (q.h_in > max_h_in) max_h_in = q.h_in;
    }
    if (workspace_bytes_ < workspace_bytes(max_tokens, n_proj, max_h_in)) return B200_LORA_ERR_WORKSPACE;
    p.n_proj = n_proj;
    p.ranks = adapters->ranks;
    p.scalings = adapters->scalings;
    p.cum_ranks = reinterpret_cast<const long long*>(adapters->cum_ranks);
    p.n_adapters = adapters->n_adapters;
    p.n_layers = adapters->n_layers;
    p.r_pool = adapters->r_pool;
    p.packed = adapters->packed;
    p.scale = adapters->scale;
    p.layer = layer;
    p.flags = flags;
    p.y_f32 = (y_dtype == B200_LORA_F32);
    p.cap = max_tokens;
    p.n_tokens = n_tokens;
    p.plan = const_cast<void*>(plan);
    p.workspace = workspace;

    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int n_sm = sm_count();
    cudaError_t e = cudaSuccess;
    SideStream* side = nullptr;
    // a batch shorter than the shortest tall run has none: no tile launches, no side stream
    if (!sgmv_tiles_supported(p) || n_tokens < kTallMin) p.flags |= B200_LORA_NO_TENSOR;
    if (!tp && cluster_route(p, adapters, io_dtype)) {
        e = launch_bgmv_cluster(p, direct_ids, direct_i64, io_dtype, s);
        return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
    }
    if (direct_ids) return B200_LORA_ERR_UNSUPPORTED;       // every other route needs a plan
    bool fast = fast_ranks(adapters);
    // Dense pools of any other ranks take the TMA kernels' padded form, except where one half runs alone
    // or the ranks of a group exchange the intermediate (who adds up the split-K slots there works with
    // the adapters' own ranks).  32 layers of a 93-token decode step, ranks 8 to 64 in R = 64: 3316 us on the
    // general kernels, 943 us here.
    const bool padded = !fast && !adapters->packed && !tp && !(flags & (B200_LORA_ONLY_SHRINK | B200_LORA_ONLY_EXPAND));
    if (padded) { fast = true; p.flags &= ~B200_LORA_DELTA_THEN_ADD; }   // a flag that these pools do not have
    for (int i = 0; i < n_proj; ++i)
        // units are cut at multiples of 128 columns (the shrink kernel's weight box, the widest
        // per-warp column group of the expand kernel), so the last unit of a row may be partial
        if ((projs[i].h_in % 128) || (projs[i].h_out % 128) || projs[i].h_in > 8192) fast = false;
    CUtensorMap bmap[kMaxProj][4];
    if (fast) {
        if (padded) memset(bmap, 0, sizeof(bmap));
        for (int i = 0; i < n_proj && fast; ++i)
            for (int c = 0; c < 4 && fast; ++c) {
                const uint32_t rc = 8u << c;
                if (padded ? rc >= 2u * adapters->r_pool : !adapters->packed && rc != (uint32_t)adapters->r_pool) continue;    // dense pools have one rank
                if (padded) {
                    const uint64_t brows = (uint64_t)adapters->n_adapters * adapters->n_layers * projs[i].h_out;
                    fast = brows <= 0x7fffffffull &&        // box coordinates are 32-bit
                           tensor_map_2d(&bmap[i][c], projs[i].wb, (uint64_t)adapters->r_pool, brows, rc, 128,
                                         CU_TENSOR_MAP_SWIZZLE_NONE, 0, CU_TENSOR_MAP_L2_PROMOTION_NONE);
                }
                fast = fast && tensor_map_2d(&p.amap[i][c], projs[i].wa, (uint64_t)projs[i].h_in, pool_rows(adapters), 128, rc,
                                     CU_TENSOR_MAP_SWIZZLE_NONE);
            }
    }
    if (!fast && (p.flags & B200_LORA_OVERWRITE)) {         // the general kernels accumulate only
        const size_t es = p.y_f32 ? 4 : 2;
        for (int i = 0; i < n_proj && e == cudaSuccess; ++i)
            e = cudaMemset2DAsync(projs[i].y, (size_t)projs[i].ldy * es, 0, (size_t)projs[i].h_out * es, (size_t)n_tokens, s);
        if (e != cudaSuccess) return cuda_fail(e);
        p.flags &= ~B200_LORA_OVERWRITE;
    }
    if (!(p.flags & B200_LORA_NO_TENSOR)) {
        SgmvParams sp;
        memset(&sp, 0, sizeof(sp));
        bool ok = true;
        const uint64_t arows = pool_rows(adapters);
        for (int i = 0; i < n_proj && ok; ++i) {
            const b200_lora_proj& q = projs[i];
            ok = tensor_map_2d(&sp.xmap[i], q.x, (uint64_t)q.h_in, (uint64_t)n_tokens, 64, 128,
                               CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)q.ldx);
            if (ok && !p.y_f32)
                ok = tensor_map_2d(&sp.ymap[i], q.y, (uint64_t)q.h_out, (uint64_t)n_tokens, 64, 128,
                                   CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)q.ldy);
            for (int c = 0; c < 3 && ok; ++c) {
                const uint64_t rc = 16u << c;
                if (!adapters->packed && rc != (uint64_t)adapters->r_pool) continue;   // dense pools have one rank
                const uint64_t brows = arows * (uint64_t)q.h_out / rc;
                const CUtensorMapSwizzle sw = c == 0 ? CU_TENSOR_MAP_SWIZZLE_32B
                                            : c == 1 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
                ok = tensor_map_2d(&sp.bmap[i][c], q.wb, rc, brows, (uint32_t)rc, 128, sw) &&
                     tensor_map_2d(&sp.amap[i][c], q.wa, (uint64_t)q.h_in, arows, 64, (uint32_t)rc, CU_TENSOR_MAP_SWIZZLE_128B);
            }
        }
        if (!ok) p.flags |= B200_LORA_NO_TENSOR;        // no driver entry point: everything on the BGMV kernels
        else {
            side = side_stream(s);
            if (side && (cudaEventRecord(side->fork, s) != cudaSuccess ||
                         cudaStreamWaitEvent(side->stream, side->fork, 0) != cudaSuccess)) {
                cudaGetLastError();
                side = nullptr;
            }
            cudaStream_t ts = side ? side->stream : s;
            if (!tp) e = launch_sgmv_tiles(p, sp, io_dtype, n_sm, ts);
            else {
                ApplyParams h = p;
                h.flags = p.flags | B200_LORA_ONLY_SHRINK;
                e = launch_sgmv_tiles(h, sp, io_dtype, n_sm, ts);
                if (e == cudaSuccess) e = launch_tp_exchange_rows(tp, 1, true, false, p, 0, io_dtype, skip_arrival, n_sm, ts);
                h.flags = p.flags | B200_LORA_ONLY_EXPAND;
                if (e == cudaSuccess) e = launch_sgmv_tiles(h, sp, io_dtype, n_sm, ts);
            }
        }
    }
    auto bgmv = [&](const ApplyParams& q) { return fast ? launch_bgmv_tma(q, padded ? bmap : nullptr, io_dtype, n_sm, s) : launch_bgmv(q, io_dtype, n_sm, s); };
    if (e == cudaSuccess && !tp) e = bgmv(p);
    if (e == cudaSuccess && tp) {
        // the TMA shrink kernel leaves its split-K slots and the exchange adds them up; the general one leaves v
        ApplyParams h = p;
        h.flags = p.flags | B200_LORA_ONLY_SHRINK | (fast ? B200_LORA_KEEP_PARTIALS : 0);
        e = bgmv(h);
        if (e == cudaSuccess)
            e = launch_tp_exchange_rows(tp, 0, false, (p.flags & B200_LORA_NO_TENSOR) != 0, p, fast ? bgmv_tma_shrink_grid(n_sm) : 0,
                                        io_dtype, skip_arrival, n_sm, s);
        h.flags = p.flags | B200_LORA_ONLY_EXPAND;
        if (e == cudaSuccess) e = bgmv(h);
    }
    if (side) {                                             // the side stream always joins, also after a failed launch
        cudaError_t j = cudaEventRecord(side->join, side->stream);
        if (j == cudaSuccess) j = cudaStreamWaitEvent(s, side->join, 0);
        if (e == cudaSuccess) e = j;
    }
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_apply(const b200_lora_proj* projs, int32_t n_proj, const b200_lora_adapters* adapters,
                    const void* plan, int32_t max_tokens, int32_t n_tokens, int32_t layer, int32_t io_dtype,
                    int32_t y_dtype, int32_t flags, void* workspace, size_t workspace_bytes_, void* stream) {
    return apply_core(projs, n_proj, adapters, plan, max_tokens, n_tokens, layer, io_dtype, y_dtype, flags, workspace,
                      workspace_bytes_, stream, nullptr, 0);
}

int b200_lora_apply_tp(const b200_lora_proj* projs, int32_t n_proj, const b200_lora_adapters* adapters,
                       const void* plan, int32_t max_tokens, int32_t n_tokens, int32_t layer, int32_t io_dtype,
                       int32_t y_dtype, int32_t flags, void* workspace, size_t workspace_bytes_, const b200_lora_tp* tp,
                       int32_t skip_arrival, void* stream) {
    if (!tp) return B200_LORA_ERR_NULL;
    return apply_core(projs, n_proj, adapters, plan, max_tokens, n_tokens, layer, io_dtype, y_dtype, flags, workspace,
                      workspace_bytes_, stream, tp, skip_arrival);
}

int b200_lora_workspace_v_region(int32_t max_tokens, int32_t n_proj, size_t* offset_bytes, size_t* size_bytes) {
    if (!offset_bytes || !size_bytes) return B200_LORA_ERR_NULL;
    if (max_tokens < 1 || n_proj < 1 || n_proj > kMaxProj) return B200_LORA_ERR_DIM;
    // the view only does address arithmetic: run it on a fictitious 128-byte-aligned base
    WorkspaceView w = workspace_view(reinterpret_cast<void*>(uintptr_t(1) << 20), max_tokens, n_proj);
    *offset_bytes = reinterpret_cast<uintptr_t>(w.v) - (uintptr_t(1) << 20);
    *size_bytes = (size_t)n_proj * max_tokens * kMaxRank * 4;
    return B200_LORA_OK;
}

// ---- tensor-parallel exchange ---------------------------------------------------------------------
// one allocation: two sets of two landing buffers [tp + 1][n_proj][max_tokens][64] of 8-byte packets (value,
// exchange number), then per set the exchange counter and the CTA counter; everything 256-byte aligned
static size_t tp_landing_bytes(int32_t max_tokens, int32_t n_proj, int32_t tp) {
    return (((size_t)(tp + 1) * n_proj * max_tokens * kMaxRank * 8) + 255) & ~size_t(255);     // a slot per rank + one for owners' sums
}

size_t b200_lora_tp_bytes(int32_t max_tokens, int32_t n_proj, int32_t tp) {
    if (max_tokens < 1 || n_proj < 1 || n_proj > kMaxProj || tp < 2 || tp > B200_LORA_TP_MAX_RANKS) return 0;
    return 4 * tp_landing_bytes(max_tokens, n_proj, tp) + B200_LORA_TP_COUNTER_BYTES;
}

int b200_lora_tp_alloc(void** base, size_t bytes) {
    if (!base || bytes == 0) return B200_LORA_ERR_NULL;
    cudaError_t e = cudaMalloc(base, bytes);
    if (e == cudaSuccess) e = cudaMemset(*base, 0, bytes);
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_tp_free(void* base) {
    cudaError_t e = cudaFree(base);
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_tp_export(void* base, void* handle64) {
    if (!base || !handle64) return B200_LORA_ERR_NULL;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "handle size");
    cudaIpcMemHandle_t h;
    cudaError_t e = cudaIpcGetMemHandle(&h, base);
    if (e != cudaSuccess) return cuda_fail(e);
    memcpy(handle64, &h, 64);
    return B200_LORA_OK;
}

int b200_lora_tp_open(const void* handle64, void** mapped) {
    if (!handle64 || !mapped) return B200_LORA_ERR_NULL;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle64, 64);
    cudaError_t e = cudaIpcOpenMemHandle(mapped, h, cudaIpcMemLazyEnablePeerAccess);
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_tp_close(void* mapped) {
    cudaError_t e = cudaIpcCloseMemHandle(mapped);
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_tp_layout(b200_lora_tp* tp, int32_t r, void* base, int32_t max_tokens, int32_t n_proj) {
    if (!tp || !base) return B200_LORA_ERR_NULL;
    if (r < 0 || r >= B200_LORA_TP_MAX_RANKS || tp->tp < 2 || tp->tp > B200_LORA_TP_MAX_RANKS) return B200_LORA_ERR_DIM;
    const size_t lb = tp_landing_bytes(max_tokens, n_proj, tp->tp);
    char* b = static_cast<char*>(base);
    tp->landing[r][0] = b;
    tp->landing[r][1] = b + lb;
    tp->flags[r] = b + 4 * lb;
    tp->set_stride = 2 * lb;
    return B200_LORA_OK;
}

int b200_lora_tp_exchange(const b200_lora_tp* tp, void* workspace, int32_t max_tokens, int32_t n_tokens,
                          int32_t n_proj, int32_t skip_arrival, void* stream) {
    if (!tp || !workspace) return B200_LORA_ERR_NULL;
    if (tp->tp < 2 || tp->tp > B200_LORA_TP_MAX_RANKS || tp->rank < 0 || tp->rank >= tp->tp) return B200_LORA_ERR_DIM;
    if (max_tokens < 1 || n_tokens < 1 || n_tokens > max_tokens || n_proj < 1 || n_proj > kMaxProj) return B200_LORA_ERR_DIM;
    if (!tp_usable(tp)) return B200_LORA_ERR_NULL;
    cudaError_t e = launch_tp_exchange(tp, workspace, n_proj, max_tokens, n_tokens, skip_arrival, sm_count(),
                                       static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? B200_LORA_OK : cuda_fail(e);
}

int b200_lora_workspace_status(const void* workspace, void* stream) {
    if (!workspace) return B200_LORA_ERR_NULL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    WorkspaceCtl ctl;
    cudaError_t e = cudaMemcpyAsync(&ctl, workspace, sizeof(ctl), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e);
    return status_of_error_word(ctl.error);
}

size_t b200_add_lora_bgmv_workspace_bytes(int32_t n_tokens, int32_t n_adapters, int32_t h_in) {
    size_t pb = b200_lora_plan_bytes(n_tokens, n_adapters);
    size_t wb = b200_lora_workspace_bytes(n_tokens, 1, h_in);
    if (!pb || !wb) return 0;
    return ((pb + 255) & ~size_t(255)) + wb;
}

static int add_lora_bgmv(void* y, const void* x, const void* wa_T_all, const void* wb_T_all,
                       const void* indicies, int32_t indicies_are_i64, int32_t n_tokens,
                       int32_t h_in, int32_t h_out, int32_t n_adapters, int32_t n_layers, int32_t r,
                       int32_t layer_idx, float scale, int32_t dtype,
                       void* workspace, size_t workspace_bytes_, void* stream, bool plan_wanted) {
    if (!workspace) return B200_LORA_ERR_NULL;
    if (n_tokens < 1 || n_adapters < 1) return B200_LORA_ERR_DIM;
    if (workspace_bytes_ < b200_add_lora_bgmv_workspace_bytes(n_tokens, n_adapters, h_in)) return B200_LORA_ERR_WORKSPACE;
    b200_lora_adapters ad;
    memset(&ad, 0, sizeof(ad));
    ad.n_adapters = n_adapters; ad.n_layers = n_layers; ad.r_pool = r; ad.packed = 0; ad.scale = scale;
    size_t pb = (b200_lora_plan_bytes(n_tokens, n_adapters) + 255) & ~size_t(255);
    char* ws = static_cast<char*>(workspace) + pb;
    b200_lora_proj pj;
    pj.x = x; pj.y = y; pj.wa = wa_T_all; pj.wb = wb_T_all;
    pj.ldx = h_in; pj.ldy = h_out; pj.h_in = h_in; pj.h_out = h_out;
    // A few tokens whose plan nobody will read: no plan kernel (a one-token call: 12.3 us with it, 4.5 without).
    // Whatever stands against that, a refused argument included, is the longer way's to report.
    if (!plan_wanted && indicies && n_tokens <= kDirectTokens) {
        int rc = apply_core(&pj, 1, &ad, workspace, n_tokens, n_tokens, layer_idx, dtype, dtype, B200_LORA_NO_TENSOR, ws,
                            workspace_bytes_ - pb, stream, nullptr, 0, indicies, indicies_are_i64);
        if (rc == B200_LORA_OK || rc == B200_LORA_ERR_CUDA) return rc;
    }
    // Where the control words sit depends on this call's n_tokens and n_adapters, so a buffer that
    // served a call of another shape holds that call's records or partial sums there: clear them
    // (error word and arrival counters must start at zero) on every call.  The plan kernel does that on
    // its way (a memset node of its own in front of it cost a one-token call 2 us); where no plan is built, a memset.
    int rc = plan_build(workspace, pb, n_tokens, indicies, indicies_are_i64, n_tokens, &ad, ws, ws_ctl_bytes(n_tokens), stream);
    if (rc) {
        cudaError_t ce = cudaMemsetAsync(ws, 0, ws_ctl_bytes(n_tokens), static_cast<cudaStream_t>(stream));
        return ce == cudaSuccess ? rc : cuda_fail(ce);
    }
    return b200_lora_apply(&pj, 1, &ad, workspace, n_tokens, n_tokens, layer_idx, dtype, dtype, B200_LORA_NO_TENSOR, ws,
                           workspace_bytes_ - pb, stream);
}

int b200_add_lora_bgmv(void* y, const void* x, const void* wa_T_all, const void* wb_T_all,
                       const void* indicies, int32_t indicies_are_i64, int32_t n_tokens,
                       int32_t h_in, int32_t h_out, int32_t n_adapters, int32_t n_layers, int32_t r,
                       int32_t layer_idx, float scale, int32_t dtype,
                       void* workspace, size_t workspace_bytes_, void* stream) {
    return add_lora_bgmv(y, x, wa_T_all, wb_T_all, indicies, indicies_are_i64, n_tokens, h_in, h_out, n_adapters, n_layers, r,
                         layer_idx, scale, dtype, workspace, workspace_bytes_, stream, true);
}

// ---- allocation-free variant ---------------------------------------------------------------
int b200_add_lora_bgmv_static(void* y, const void* x, const void* wa_T_all, const void* wb_T_all,
                              const void* indicies, int32_t indicies_are_i64, int32_t n_tokens,
                              int32_t h_in, int32_t h_out, int32_t n_adapters, int32_t n_layers, int32_t r,
                              int32_t layer_idx, float scale, int32_t dtype, void* stream) {
    if (n_tokens < 1 || n_tokens > B200_LORA_STATIC_MAX_TOKENS || n_adapters < 1 ||
        n_adapters > B200_LORA_STATIC_MAX_ADAPTERS || h_in < 8 || h_in > B200_LORA_STATIC_MAX_H_IN)
        return B200_LORA_ERR_WORKSPACE;          // beyond what the static scratch was sized for
    const size_t need = b200_add_lora_bgmv_workspace_bytes(n_tokens, n_adapters, h_in);
    if (need == 0 || need > (size_t)B200_LORA_STATIC_SCRATCH_BYTES) return B200_LORA_ERR_WORKSPACE;

    void* scratch = nullptr;
    int rc = static_scratch_address(&scratch);       // the first call on a device looks the address up
    if (rc) return rc;
    // The array keeps whatever the previous call left.  A call of few tokens needs no plan and no workspace
    // (it only sets the two error words that the status call reads); a longer one rebuilds the plan in it, and the
    // plan kernel clears the control words (arrival counters, error word) of this call's layout.
    const size_t pb = (b200_lora_plan_bytes(n_tokens, n_adapters) + 255) & ~size_t(255);
    {
        std::lock_guard<std::mutex> lock(g_static_mu);
        int dev = 0;
        cudaGetDevice(&dev);
        g_static_last_pb[dev] = pb;              // where the last call's workspace part begins
    }
    return add_lora_bgmv(y, x, wa_T_all, wb_T_all, indicies, indicies_are_i64, n_tokens, h_in, h_out,
                         n_adapters, n_layers, r, layer_idx, scale, dtype, scratch,
                         (size_t)B200_LORA_STATIC_SCRATCH_BYTES, stream, false);
}

int b200_add_lora_bgmv_static_status(void* stream) {
    void* scratch = nullptr;
    int rc = static_scratch_address(&scratch);
    if (rc) return rc;
    size_t pb;
    {
        std::lock_guard<std::mutex> lock(g_static_mu);
        int dev = 0;
        cudaGetDevice(&dev);
        pb = g_static_last_pb[dev];
    }
    if (pb == 0) return B200_LORA_OK;            // no call yet on this device
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    PlanHeader h;
    WorkspaceCtl ctl;
    cudaError_t e = cudaMemcpyAsync(&h, scratch, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&ctl, static_cast<char*>(scratch) + pb, sizeof(ctl), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e);
    if (h.error == 1) return B200_LORA_ERR_ID_RANGE;
    if (h.error == 3) return B200_LORA_ERR_RANK;
    if (h.error) return B200_LORA_ERR_SEGMENTS;
    return status_of_error_word(ctl.error);
}

}  // extern "C"
