// Decode BGMV for a handful of tokens: one launch, one thread-block cluster per (work segment,
// projection) (sm_100a).
//
// A decode step of a few tokens moves a few hundred KB per apply, so its time is not the bytes but
// the chain: launch, plan, weights from HBM, shrink, hand-over, expand.  The two TMA kernels
// (lora_bgmv_tma.cu) pay that chain twice and hand over through split-K slots in global memory.
// Here the eight CTAs of a cluster share one segment: CTA c owns the c-th eighth of h_in and of
// h_out.  At its start it requests ALL the weights it will need (its A columns and its B rows) and,
// once the predecessor has ended, its x and y columns; then
//
//   shrink    partial v[ntok, r] over its columns            mma.sync m16n8k16, warps split rows x columns
//   exchange  the partial goes to all eight CTAs             st.shared::cluster, one cluster barrier
//   fold      v = sum of the eight partials, in CTA order    (bit-reproducible)
//   expand    y[:, its columns] += scale * v . B^T           hi + lo 16-bit halves of v in one MMA: they drop at most
//                                                            2^-17 of it (bf16), 2^-23 or 2^-25 absolute (fp16)
//
// What bounds it: that chain, 3.6 us for one token at h = 4096, r = 16 (two kernels: 5.5 us), of which
// the bytes are under 0.1.  The split in eight makes every copy short and keeps all of them in flight at
// once; the only global round trips are the plan record, and weights and activations together.  Nothing
// is written to global memory but y.  All loads are plain bulk copies of this GPU's memory (no
// tensor maps, no multicast); the A rows are stored 64 bytes apart modulo 128, which makes the
// fragment loads free of bank conflicts.
//
// Requirements (checked by the dispatch in lora_api.cu): ranks 8/16/32/64 with contiguous B blocks,
// widths that are multiples of 128, the slices of the pool's largest rank in shared memory, no tall
// runs on the tile kernels, x and y in different memory (a cluster writes its y columns while other
// clusters may still read x).
//
// Semantics: add_lora_bgmv(y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale) of the
// reference (lightllm/models/lora_gpu.py:138,150,162), pools as at :33-40.
#include <string.h>

#include <mutex>

#include "lora_common.cuh"
#include "lora_pipe.cuh"

namespace b200lora {

namespace {

constexpr int kCluster = 8;
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kVPitch = 72;                       // floats per token row of the folded intermediate
constexpr int kRedBytes = 8 * 8 * 20 * 4;         // largest for rank 16: 8 slices, rows of 20 floats
constexpr int kMaxSmem = 227 * 1024;

struct ClusterArgs {
    ProjArgs proj[kMaxProj];
    void* plan;
    void* workspace;
    int n_proj, n_adapters, n_layers, r_pool, packed, layer, flags, y_f32, cap, n_tokens;
    int r_cap;                 // largest rank the shared memory was sized for
    int kcols, jcols;          // widest slice of h_in and of h_out
    // DIRECT: the adapter of each token instead of a plan (one projection, dense pool of one rank)
    const void* ids;
    int ids_i64;
    float scale;
};

// Shared memory of one CTA: byte offsets of its parts.
struct Layout {
    int pitch, x, b, y, ypitch, red, vs, vt, bars, total;
};
__host__ __device__ inline Layout layout_of(int r_cap, int kcols, int jcols, int y_f32) {
    Layout l;
    l.pitch = kcols * 2 + 64;                              // A and x rows
    l.x = r_cap * l.pitch;
    l.b = l.x + 8 * l.pitch;
    l.y = l.b + jcols * r_cap * 2;
    l.ypitch = jcols * (y_f32 ? 4 : 2) + 32;
    l.red = l.y + 8 * l.ypitch;
    l.vs = l.red + kRedBytes;                              // cross-warp reduction: [slice][token][rank]
    l.vt = l.vs + kCluster * 8 * r_cap * 4;                // the eight partials: [cta][token][rank]
    l.bars = l.vt + 8 * kVPitch * 4;
    l.total = l.bars + 16;
    return l;
}
// the widest of eight slices cut at multiples of 128 columns
inline int widest_slice(int h) { return ((h / 128 + kCluster - 1) / kCluster) * 128; }

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned remote_smem(unsigned addr, unsigned cta) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, const float4& v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Weight rows are the M rows of the MMA (16 per block), the segment's tokens its N columns; the k
// index is permuted identically for both operands, so that a thread's fragment is one 16-byte chunk.
// The warps are R / 16 row blocks times slices of the CTA's columns; each leaves its partial in `red`.
template <typename T, int R>
__device__ __forceinline__ void cluster_shrink(const unsigned char* a, const unsigned char* x, int pitch, int ncol, float* red,
                                               int lane, int warp) {
    constexpr int MB = R >= 16 ? R / 16 : 1;
    constexpr int KSPLIT = kWarps / MB;
    constexpr int RP = R + 4;
    const int kslot = warp % KSPLIT, mblk = warp / KSPLIT;
    const int g = lane >> 2, t = lane & 3;
    const unsigned char* wrow = a + (mblk * 16 + g) * pitch + t * 16;
    const unsigned char* xrow = x + g * pitch + t * 16;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int col = kslot * 32; col < ncol; col += 2 * KSPLIT * 32) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = col + h * KSPLIT * 32;
            if (c < ncol) {
                const uint4 xb = *reinterpret_cast<const uint4*>(xrow + c * 2);
                const uint4 w = *reinterpret_cast<const uint4*>(wrow + c * 2);
                uint4 u = make_uint4(0u, 0u, 0u, 0u);
                if (R >= 16) u = *reinterpret_cast<const uint4*>(wrow + 8 * pitch + c * 2);      // rank 8 has no rows 8..15
                Mma<T>::run(acc[2 * h], w.x, u.x, w.y, u.y, xb.x, xb.y);
                Mma<T>::run(acc[2 * h + 1], w.z, u.z, w.w, u.w, xb.z, xb.w);
            }
        }
    }
    float* base = red + kslot * 8 * RP + mblk * 16 + g;
    base[(2 * t) * RP] = (acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]);
    base[(2 * t + 1) * RP] = (acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1]);
    if (R >= 16) {
        base[(2 * t) * RP + 8] = (acc[0][2] + acc[1][2]) + (acc[2][2] + acc[3][2]);
        base[(2 * t + 1) * RP + 8] = (acc[0][3] + acc[1][3]) + (acc[2][3] + acc[3][3]);
    }
}

// Sum over the warps' column slices, and the sum to every CTA of the cluster (slot `crank` there).
template <int R>
__device__ __forceinline__ void cluster_send(const float* red, unsigned vs, unsigned crank, int ntok, int tid) {
    constexpr int KSPLIT = R >= 16 ? kWarps / (R / 16) : kWarps;
    constexpr int RP = R + 4, Q = R / 4;                    // quads of a token
    for (int idx = tid; idx < 8 * Q * kCluster; idx += kThreads) {
        const int q = idx % (8 * Q), peer = idx / (8 * Q);
        const int tok = q / Q, k4 = (q % Q) * 4;
        if (tok >= ntok) continue;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < KSPLIT; ++w) {
            const float4 v = *reinterpret_cast<const float4*>(red + (w * 8 + tok) * RP + k4);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        st_cluster(remote_smem(vs + ((crank * 8 + tok) * R + k4) * 4, peer), s);
    }
}

// v = the eight partials in CTA order.
template <typename T, int R>
__device__ __forceinline__ void cluster_fold(const float* vs, float* vt, int ntok, bool mid_round, int tid) {
    constexpr int Q = R / 4;
    if (tid >= ntok * Q) return;
    const int tok = tid / Q, k4 = (tid % Q) * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < kCluster; ++c) {
        const float4 v = *reinterpret_cast<const float4*>(vs + (c * 8 + tok) * R + k4);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    if (mid_round) { s.x = Cvt<T>::round1(s.x); s.y = Cvt<T>::round1(s.y); s.z = Cvt<T>::round1(s.z); s.w = Cvt<T>::round1(s.w); }
    *reinterpret_cast<float4*>(vt + tok * kVPitch + k4) = s;
}

// The weight tile is the MMA's A operand: 16 output columns (M) by 16 rank indices (K, permuted so
// that a thread's fragments are wide loads).  Column 2q of N holds the hi half of token q's
// intermediate and column 2q+1 the lo half (tokens 0..3, then 4..7 with a second MMA: NG groups); thread (g, t)
// gets token t's products for columns g and g + 8, and lanes g and g ^ 1 swap one so that each owns two
// adjacent outputs.
//
// What bounds it: two warps a scheduler do not hide the chain of an MMA group (four dependent MMAs at rank 64, the
// swap, the store), so a warp works on two blocks of columns and both groups of tokens at once, with nothing but
// independent chains between the loads and the stores.  Five tokens of one adapter, 1024 to 8192 columns, rank 64, where
// a CTA has most to do, weights in L2: 6.6 us with a block at a time, 5.65 now (two kernels: 5.8); 4096 columns, rank 16:
// 3.5 and 3.2 (5.0).
template <typename T, int R, int NG>
__device__ __forceinline__ void expand_columns(const ClusterArgs& p, const ProjArgs& pj, float scale, const unsigned (&bf)[2][R == 64 ? 4 : R == 32 ? 2 : 1][2],
                                               const int (&row)[2], const unsigned char* b, const unsigned char* ysm, int ypitch, int j0,
                                               int njs, int lane, int warp) {
    constexpr int KS = R == 64 ? 4 : R == 32 ? 2 : 1;
    constexpr int kStep = kWarps * 16;
    const int g = lane >> 2, t = lane & 3;
    const bool overwrite = (p.flags & B200_LORA_OVERWRITE) != 0;      // y counts as zero
    const bool lo_half = (g & 1) != 0;
    for (int nb0 = warp * 16; nb0 < njs; nb0 += 2 * kStep) {
        const bool two = nb0 + kStep < njs;                // else the second block repeats the first and stores nothing
        unsigned a[2][KS][4];
        float acc[2][NG][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int nb = i == 1 && two ? nb0 + kStep : nb0;
            const unsigned char* w0 = b + (nb + g) * (R * 2);      // output column g of the block
            const unsigned char* w1 = w0 + 8 * (R * 2);            // output column g + 8
            if constexpr (R >= 32) {
#pragma unroll
                for (int c = 0; c < KS / 2; ++c) {
                    const uint4 r0 = *reinterpret_cast<const uint4*>(w0 + (t * (KS / 2) + c) * 16);
                    const uint4 r1 = *reinterpret_cast<const uint4*>(w1 + (t * (KS / 2) + c) * 16);
                    a[i][2 * c][0] = r0.x; a[i][2 * c][1] = r1.x; a[i][2 * c][2] = r0.y; a[i][2 * c][3] = r1.y;
                    a[i][2 * c + 1][0] = r0.z; a[i][2 * c + 1][1] = r1.z; a[i][2 * c + 1][2] = r0.w; a[i][2 * c + 1][3] = r1.w;
                }
            } else if constexpr (R == 16) {
                const uint2 r0 = *reinterpret_cast<const uint2*>(w0 + t * 8);
                const uint2 r1 = *reinterpret_cast<const uint2*>(w1 + t * 8);
                a[i][0][0] = r0.x; a[i][0][1] = r1.x; a[i][0][2] = r0.y; a[i][0][3] = r1.y;
            } else {
                a[i][0][0] = *reinterpret_cast<const unsigned*>(w0 + t * 4);
                a[i][0][1] = *reinterpret_cast<const unsigned*>(w1 + t * 4);
                a[i][0][2] = a[i][0][3] = 0u;
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int grp = 0; grp < NG; ++grp) acc[i][grp][0] = acc[i][grp][1] = acc[i][grp][2] = acc[i][grp][3] = 0.f;
#pragma unroll
        for (int k = 0; k < KS; ++k)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int grp = 0; grp < NG; ++grp)
                    Mma<T>::run(acc[i][grp], a[i][k][0], a[i][k][1], a[i][k][2], a[i][k][3], bf[grp][k][0], bf[grp][k][1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int jl = nb0 + i * kStep + (lo_half ? g + 7 : g);
#pragma unroll
            for (int grp = 0; grp < NG; ++grp) {
                const float c_lo = scale * (acc[i][grp][0] + acc[i][grp][1]);
                const float c_hi = scale * (acc[i][grp][2] + acc[i][grp][3]);
                const float got = __shfl_xor_sync(0xffffffffu, lo_half ? c_lo : c_hi, 4);
                const float d0 = lo_half ? got : c_lo, d1 = lo_half ? c_hi : got;
                if (row[grp] < 0 || (i == 1 && !two)) continue;
                const long long yoff = (long long)row[grp] * pj.ldy + j0 + jl;
                if (p.y_f32) {
                    float2 yv = overwrite ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(ysm + (t + 4 * grp) * ypitch + jl * 4);
                    yv.x += d0; yv.y += d1;
                    *reinterpret_cast<float2*>(reinterpret_cast<float*>(pj.y) + yoff) = yv;
                } else {
                    const unsigned yw = overwrite ? 0u : *reinterpret_cast<const unsigned*>(ysm + (t + 4 * grp) * ypitch + jl * 2);
                    float lo, hi;
                    if (Cvt<T>::is_bf16) {
                        lo = __uint_as_float(yw << 16); hi = __uint_as_float(yw & 0xffff0000u);
                    } else {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&yw));
                        lo = f.x; hi = f.y;
                    }
                    *reinterpret_cast<unsigned*>(reinterpret_cast<T*>(pj.y) + yoff) = Cvt<T>::pack2(lo + d0, hi + d1);
                }
            }
        }
    }
}

template <typename T, int R>
__device__ __forceinline__ void cluster_expand(const ClusterArgs& p, const ProjArgs& pj, const UnitRec& u, const unsigned char* b,
                                               const unsigned char* ysm, int ypitch, const float* vt, int j0, int njs, int lane, int warp) {
    constexpr int KS = R == 64 ? 4 : R == 32 ? 2 : 1;
    const int g = lane >> 2, t = lane & 3;
    const bool lo_half = (g & 1) != 0;
    unsigned bf[2][KS][2];
#pragma unroll
    for (int grp = 0; grp < 2; ++grp) {
#pragma unroll
        for (int k = 0; k < KS; ++k) bf[grp][k][0] = bf[grp][k][1] = 0u;
        const int q = (g >> 1) + 4 * grp;
        if (q >= u.ntok) continue;
        const float* v = vt + q * kVPitch + (R == 8 ? t * 2 : t * 4 * KS);
        if constexpr (R == 8) {
            const float2 v2 = *reinterpret_cast<const float2*>(v);
            bf[grp][0][0] = hl_pack<T>(v2.x, v2.y, lo_half);
        } else {
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                const float4 v4 = *reinterpret_cast<const float4*>(v + 4 * k);
                bf[grp][k][0] = hl_pack<T>(v4.x, v4.y, lo_half);
                bf[grp][k][1] = hl_pack<T>(v4.z, v4.w, lo_half);
            }
        }
    }
    int row[2];
#pragma unroll
    for (int grp = 0; grp < 2; ++grp) {
        const int q = t + 4 * grp;
        row[grp] = q < u.ntok ? u.tok[0] : -1;
#pragma unroll
        for (int i = 1; i < 8; ++i)
            if (q == i && q < u.ntok) row[grp] = u.tok[i];
    }
    __syncwarp();                                          // the MMAs are for whole warps
    if (u.ntok > 4) expand_columns<T, R, 2>(p, pj, u.scale, bf, row, b, ysm, ypitch, j0, njs, lane, warp);
    else expand_columns<T, R, 1>(p, pj, u.scale, bf, row, b, ysm, ypitch, j0, njs, lane, warp);
}

template <typename T, int R>
__device__ __forceinline__ void cluster_body(const ClusterArgs& p, const ProjArgs& pj, const UnitRec& u, unsigned char* smem, const Layout& l,
                                             unsigned crank, int ncol, int j0, int njs, unsigned* err, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    float* red = reinterpret_cast<float*>(smem + l.red);
    float* vs = reinterpret_cast<float*>(smem + l.vs);
    float* vt = reinterpret_cast<float*>(smem + l.vt);
    mbar_wait(smem_u32(smem + l.bars), 0, err, 5);
    __syncwarp();
    cluster_shrink<T, R>(smem, smem + l.x, l.pitch, ncol, red, lane, warp);
    __syncthreads();
    cluster_wait();                                        // every CTA of the cluster runs: its shared memory may be written
    cluster_send<R>(red, smem_u32(vs), crank, u.ntok, tid);
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                        // all eight partials have arrived; nothing remote follows
    cluster_fold<T, R>(vs, vt, u.ntok, (p.flags & B200_LORA_MID_ROUND) != 0, tid);
    __syncthreads();
    mbar_wait(smem_u32(smem + l.bars + 8), 0, err, 6);
    __syncwarp();
    cluster_expand<T, R>(p, pj, u, smem + l.b, smem + l.y, l.ypitch, vt, j0, njs, lane, warp);
}

// The work segments of a call that has no plan, for at most kDirectTokens tokens: token t heads one when it is
// the 1st, 9th, ... token of its adapter, and the segment is that token and the next seven of the adapter (a
// plan would cut in the same number of pieces and balance their lengths).  Every warp works it out from the
// ids.  Returns whether t heads a segment; `bad` when any id names no adapter.
__device__ __forceinline__ bool direct_segment(const ClusterArgs& p, int t, int lane, UnitRec& u, bool& bad) {
    int id[2];
    bool in[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        in[h] = i < p.n_tokens;
        id[h] = !in[h] ? -1 : p.ids_i64 ? (int)reinterpret_cast<const long long*>(p.ids)[i] : reinterpret_cast<const int*>(p.ids)[i];
    }
    bad = __ballot_sync(0xffffffffu, (in[0] && (id[0] < 0 || id[0] >= p.n_adapters)) || (in[1] && (id[1] < 0 || id[1] >= p.n_adapters))) != 0;
    const int a0 = __shfl_sync(0xffffffffu, id[0], t & 31), a1 = __shfl_sync(0xffffffffu, id[1], t & 31);
    const int a = t < 32 ? a0 : a1;
    unsigned long long m = __ballot_sync(0xffffffffu, in[0] && id[0] == a);
    m |= (unsigned long long)__ballot_sync(0xffffffffu, in[1] && id[1] == a) << 32;
    const int before = __popcll(m & ((1ull << t) - 1));
    m = m >> t << t;
    u.adapter = a; u.rank = p.r_pool; u.sub = 0; u.ntok = (short)min(8, __popcll(m)); u.scale = p.scale; u.wseg = t; u.start = t;
    u.cum_lo = u.cum_hi = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        u.tok[i] = m ? __ffsll((long long)m) - 1 : t;
        m &= m - 1;
    }
    return (before & 7) == 0;
}

template <typename T, bool DIRECT>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads) bgmv_cluster_kernel(const __grid_constant__ ClusterArgs p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned crank = cluster_rank();
    const int item = blockIdx.x / kCluster, seg = item / p.n_proj;      // seg < n_tokens <= cap
    cluster_arrive();
    const Layout l = layout_of(p.r_cap, p.kcols, p.jcols, p.y_f32);
    PlanView pv = plan_view(p.plan, p.cap, p.n_adapters);
    unsigned* err = &reinterpret_cast<WorkspaceCtl*>(p.workspace)->error;
    // header and segment record in one round trip (the record of a segment the plan does not have is not used; it is
    // inside every plan, seg < kClusterTokens)
    UnitRec u;
    PlanHeader hdr;
    bool heads = true;
    if constexpr (DIRECT) {
        pdl_wait_prior();                                  // the ids may come from the predecessor
        if (tid == 0) pdl_launch_dependents();
        bool bad;
        heads = direct_segment(p, seg, lane, u, bad);
        hdr.error = bad ? 1 : 0;
        hdr.cap = p.cap; hdr.n_tokens = hdr.n_wsegs = p.n_tokens;
        // What the status call reads.  All clusters start together, and a wait takes seconds to expire, so no
        // other CTA's record can be older than this.
        if (blockIdx.x == 0 && tid == 0) {
            pv.hdr->error = hdr.error;
            *err = 0u;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            reinterpret_cast<uint4*>(&u)[i] = __ldg(reinterpret_cast<const uint4*>(pv.seg_tab + (size_t)seg * 16) + i);
        hdr = *pv.hdr;
    }
    const unsigned bar_a = smem_u32(smem + l.bars), bar_b = bar_a + 8;
    if (tid == 0) {
        mbar_init(bar_a, 2);                               // weights, and x
        mbar_init(bar_b, 2);                               // weights, and y
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // the same decision in all CTAs of the cluster
    bool live = !hdr.error && seg < hdr.n_wsegs && heads;
    const bool rank_ok = (u.rank == 8 || u.rank == 16 || u.rank == 32 || u.rank == 64) && u.rank <= p.r_cap;
    const bool refused = hdr.error || hdr.cap != p.cap || hdr.n_tokens != p.n_tokens;      // the whole plan
    const bool bad_rank = !refused && live && !rank_ok;                                    // this segment
    if ((refused && !hdr.error) || bad_rank) {
        if (tid == 0) atomicMax(err, kErrPlanMismatch);
        live = false;
    }
    if (!live) {
        __syncwarp();                                      // the cluster barrier is for whole warps
        cluster_wait();                                    // pairs with the arrival above
        pdl_wait_prior();
        if (tid == 0) pdl_launch_dependents();
        // What nothing is applied to is cleared: the rows of the segment, or of a refused plan all rows (the
        // clusters are as many as rows times projections, and each clears one).
        if ((p.flags & B200_LORA_OVERWRITE) && (refused || bad_rank)) {
            const ProjArgs& pj = p.proj[item - seg * p.n_proj];
            const int es = p.y_f32 ? 4 : 2;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (refused ? i > 0 : i >= u.ntok) break;
                const int row = refused ? seg : u.tok[i];
                uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<char*>(pj.y) + (long long)row * pj.ldy * es);
                for (int q = (int)crank * kThreads + tid; q < pj.h_out * es / 16; q += kCluster * kThreads) dst[q] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        return;
    }
    const ProjArgs& pj = p.proj[item - seg * p.n_proj];
    const int r = u.rank;
    const int kb = pj.h_in / 128, jb = pj.h_out / 128;
    const int k0 = (int)crank * kb / kCluster * 128, ncol = ((int)crank + 1) * kb / kCluster * 128 - k0;
    const int j0 = (int)crank * jb / kCluster * 128, njs = ((int)crank + 1) * jb / kCluster * 128 - j0;
    const unsigned sbase = smem_u32(smem);
    if (warp == 0) {
        // the weights: no kernel that may still be running writes them
        const long long cum = ((long long)u.cum_hi << 32) | (unsigned)u.cum_lo;
        const long long row0 = p.packed ? (long long)p.n_layers * cum + (long long)p.layer * r
                                        : ((long long)u.adapter * p.n_layers + p.layer) * p.r_pool;
        if (lane == 0) { mbar_arrive_expect_tx(bar_a, r * ncol * 2); mbar_arrive_expect_tx(bar_b, njs * r * 2); }
        __syncwarp();
        const T* wa = reinterpret_cast<const T*>(pj.wa) + row0 * pj.h_in + k0;
        if (ncol > 0)
            for (int i = lane; i < r; i += 32) bulk_g2s(sbase + i * l.pitch, wa + (long long)i * pj.h_in, ncol * 2, bar_a);
        const unsigned char* wb = reinterpret_cast<const unsigned char*>(reinterpret_cast<const T*>(pj.wb) + row0 * pj.h_out + (long long)j0 * r);
        for (int o = lane * 4096; o < njs * r * 2; o += 32 * 4096)
            bulk_g2s(sbase + l.b + o, wb + o, min(4096, njs * r * 2 - o), bar_b);
    }
    pdl_wait_prior();
    if (tid == 0) pdl_launch_dependents();
    if (warp == 1) {
        const int y_size = p.y_f32 ? 4 : 2;
        const int y_bytes = p.flags & B200_LORA_OVERWRITE ? 0 : njs * y_size;
        if (lane == 0) { mbar_arrive_expect_tx(bar_a, u.ntok * ncol * 2); mbar_arrive_expect_tx(bar_b, u.ntok * y_bytes); }
        __syncwarp();
        const int q = lane & 7;
        int tok = u.tok[0];
#pragma unroll
        for (int i = 1; i < 8; ++i)
            if (q == i) tok = u.tok[i];
        if (q < u.ntok) {
            if (lane < 8 && ncol > 0)
                bulk_g2s(sbase + l.x + q * l.pitch, reinterpret_cast<const T*>(pj.x) + (long long)tok * pj.ldx + k0, ncol * 2, bar_a);
            else if (lane >= 8 && lane < 16 && y_bytes > 0)
                bulk_g2s(sbase + l.y + q * l.ypitch, reinterpret_cast<const char*>(pj.y) + ((long long)tok * pj.ldy + j0) * y_size, y_bytes, bar_b);
        }
        __syncwarp();
    }
    switch (r) {
        case 8:  cluster_body<T, 8>(p, pj, u, smem, l, crank, ncol, j0, njs, err, tid); break;
        case 16: cluster_body<T, 16>(p, pj, u, smem, l, crank, ncol, j0, njs, err, tid); break;
        case 32: cluster_body<T, 32>(p, pj, u, smem, l, crank, ncol, j0, njs, err, tid); break;
        default: cluster_body<T, 64>(p, pj, u, smem, l, crank, ncol, j0, njs, err, tid); break;
    }
}

// Clusters with `smem` bytes of shared memory per CTA that the current device runs at once (a question to
// the driver, asked once per device and size).  Also prepares the kernel for launches of that size.
template <typename T>
int resident_clusters(int smem) {
    struct Known { int dev, smem, n; };
    constexpr int kKnown = 32;
    static Known known[kKnown];
    static int n_known = 0;
    static std::mutex mu;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < (n_known < kKnown ? n_known : kKnown); ++i)
        if (known[i].dev == dev && known[i].smem == smem) return known[i].n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(bgmv_cluster_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess ||
        cudaFuncSetAttribute(bgmv_cluster_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, bgmv_cluster_kernel<T, false>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;                                             // the apply stays on the streaming kernels
    }
    known[n_known % kKnown] = Known{dev, smem, n};
    ++n_known;
    return n;
}

}  // namespace

bool bgmv_cluster_fits(const ApplyParams& p) {
    int kcols = 0, jcols = 0;
    for (int i = 0; i < p.n_proj; ++i) {
        if ((p.proj[i].h_in % 128) || (p.proj[i].h_out % 128)) return false;
        if (widest_slice(p.proj[i].h_in) > kcols) kcols = widest_slice(p.proj[i].h_in);
        if (widest_slice(p.proj[i].h_out) > jcols) jcols = widest_slice(p.proj[i].h_out);
    }
    if (kcols > 1024 || jcols > 1024) return false;
    const int smem = layout_of(pad_rank(p.r_pool), kcols, jcols, p.y_f32).total;
    return smem <= kMaxSmem;
}

int bgmv_cluster_limit(const ApplyParams& p, int io_dtype) {
    int kcols = 0, jcols = 0;
    for (int i = 0; i < p.n_proj; ++i) {
        if (widest_slice(p.proj[i].h_in) > kcols) kcols = widest_slice(p.proj[i].h_in);
        if (widest_slice(p.proj[i].h_out) > jcols) jcols = widest_slice(p.proj[i].h_out);
    }
    const int smem = layout_of(pad_rank(p.r_pool), kcols, jcols, p.y_f32).total;
    return io_dtype == B200_LORA_F16 ? resident_clusters<__half>(smem) : resident_clusters<__nv_bfloat16>(smem);
}

cudaError_t launch_bgmv_cluster(const ApplyParams& p, const void* ids, int ids_i64, int io_dtype, cudaStream_t s) {
    ClusterArgs a;
    memset(&a, 0, sizeof(a));
    a.r_cap = pad_rank(p.r_pool);
    for (int i = 0; i < p.n_proj; ++i) {
        a.proj[i] = p.proj[i];
        if (widest_slice(p.proj[i].h_in) > a.kcols) a.kcols = widest_slice(p.proj[i].h_in);
        if (widest_slice(p.proj[i].h_out) > a.jcols) a.jcols = widest_slice(p.proj[i].h_out);
    }
    a.plan = p.plan; a.workspace = p.workspace;
    a.n_proj = p.n_proj; a.n_adapters = p.n_adapters; a.n_layers = p.n_layers; a.r_pool = p.r_pool; a.packed = p.packed;
    a.layer = p.layer; a.flags = p.flags; a.y_f32 = p.y_f32; a.cap = p.cap; a.n_tokens = p.n_tokens;
    const int smem = layout_of(a.r_cap, a.kcols, a.jcols, a.y_f32).total;
    // a cluster per (work segment, projection); there are at most as many segments as tokens
    const int n = p.n_tokens * p.n_proj;
    a.ids = ids; a.ids_i64 = ids_i64; a.scale = p.scale;
    auto kernel = io_dtype == B200_LORA_F16 ? bgmv_cluster_kernel<__half, false> : bgmv_cluster_kernel<__nv_bfloat16, false>;
    if (ids) kernel = io_dtype == B200_LORA_F16 ? bgmv_cluster_kernel<__half, true> : bgmv_cluster_kernel<__nv_bfloat16, true>;
    return launch_pdl(kernel, dim3(n * kCluster), dim3(kThreads), smem, s, a);
}

}  // namespace b200lora
