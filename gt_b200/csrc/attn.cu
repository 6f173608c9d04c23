// Fused structure-masked sparse attention for sm_100a: SDDMM -> (clamp-)softmax -> SpMM in one pass over the CSR,
// forward and backward, nothing of size [E, H] or [E, H, d] is materialised.
//
// Work decomposition.  One warp owns one *segment* of a row (at most seg_edges consecutive CSR entries; rows longer
// than that -- hubs, the global token -- are cut and merged by a combine kernel: split-KV).  A feature row of H*D
// elements is cut into chunks of 8 elements (16 bytes of bf16); LPR = min(32, H*D/8) lanes cover one row, so a warp
// processes 32/LPR edges at once and every K / V row of an edge is fetched by one fully coalesced 16-byte-per-lane
// transaction.  A head occupies D/8 consecutive lanes; its dot product is finished with log2(D/8) shuffles.  Two edge
// groups are in flight per iteration (their K / V loads are issued before any arithmetic) to keep enough bytes
// outstanding per SM for HBM3e.  Why SIMT and not tcgen05 here: with ~20 edges per row the operation moves ~1 KB per
// edge and does ~1 KFLOP on it (1 FLOP/B against a machine balance of ~215 FLOP/B), so the kernel is bound by the
// gather traffic; a dense tile formulation would gather the same bytes and add >100x redundant MACs.
//
// The same kernels serve every layer kind: `row_map` + `accumulate` implement the compact-accumulate mode of the
// streamed layer (doubly-compressed row list, partials added in place into the reduce-scatter payload), and the
// `*_peers` tables let the forward fetch K / V rows straight from the owners' memory over NVLink (receiver-driven pull
// fused into the kernel: only the rows a tile references cross the switch).
//
// Semantics follow the operator specification in gt_b200/attention/ref.py (reference kernels:
// gt3d/gt3d/attention/triton_kernel.py:38-284, triton_tiled.py:157-479).
#include <algorithm>
#include <type_traits>

#include "attn_edge.cuh"
#include "common.cuh"
#include "kernels.h"

namespace gt {

namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kMaxTypesReg = 4;     // edge types whose gate / bias gradients are kept in registers
// edge groups in flight per warp (memory-level parallelism)
constexpr int kUnrollFwd = 2, kUnrollRow = 2, kUnrollCol = 2;

struct Lanes {
    int lpr;     // lanes per feature row
    int lph;     // lanes per head
    int epw;     // edges per warp iteration
    int sub;     // my edge slot
    int ll;      // my lane inside the row
};

__device__ __forceinline__ Lanes make_lanes(int HD, int D) {
    Lanes L;
    int nch = HD >> 3;
    L.lpr = nch < 32 ? nch : 32;
    L.lph = D >> 3;
    L.epw = 32 / L.lpr;
    int lane = threadIdx.x & 31;
    L.sub = lane / L.lpr;
    L.ll = lane - L.sub * L.lpr;
    return L;
}

__device__ __forceinline__ float head_sum(float v, int lph) {
    for (int o = lph >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(GT_FULL_MASK, v, o);
    return v;
}

__device__ __forceinline__ float safe_exp_diff(float a, float b) {   // exp(a - b) with exp(-inf - -inf) := 0
    return (a == -INFINITY) ? 0.f : __expf(a - b);
}

__device__ __forceinline__ int table_floats(const AttnCommon& c) {
    return (c.score == SCORE_GATED ? c.T * c.H * c.D : 0) + (c.score == SCORE_BIASED ? c.T * c.H : 0);
}

// shared-memory tables: gate [T, HD] and bias [T, H]
__device__ __forceinline__ void load_tables(const AttnCommon& c, float* s_gate, float* s_bias) {
    int HD = c.H * c.D;
    if (c.score == SCORE_GATED)
        for (int i = threadIdx.x; i < c.T * HD; i += blockDim.x) s_gate[i] = c.gate[i];
    if (c.score == SCORE_BIASED)
        for (int i = threadIdx.x; i < c.T * c.H; i += blockDim.x) s_bias[i] = c.bias[i];
    __syncthreads();
}

// Reduce-scatter fused into the forward epilogue: the finished partial row [acc | l] goes, as bf16, straight into the slot
// that the row's OWNER keeps for this rank (a[r, 0 : H*D] = acc, a[r, l_off : l_off + H] = l; 16-byte peer stores over NVLink),
// so the packed payload never exists in local memory and no separate collective moves it.  Called by all 32 lanes.
template <int CPL>
__device__ __forceinline__ void push_partial_row(const AttnFwdArgs& a, long long orow, const Lanes& L, int H, const int (&foff)[CPL],
                                                 const float (&acc)[CPL][8], const float (&l)[CPL]) {
    const int owner = (int)(orow / a.push_rows);
    const long long r = orow - (long long)owner * a.push_rows;
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.push_slot[owner]) + r * a.push_ld;
    const int lane = threadIdx.x & 31;
    const int Hp = (H + 7) & ~7;
    for (int g8 = 0; g8 < Hp; g8 += 8) {                 // the heads' l values are collected in lane 0, eight per 16-byte store
        float lv[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int chunk = (g8 + x) * L.lph;          // first 8-element chunk of head g8 + x
            const int src = chunk & 31, ci = chunk >> 5;
            float val = 0.f;
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                const float t = __shfl_sync(GT_FULL_MASK, l[i], src);
                if (i == ci) val = t;
            }
            lv[x] = (g8 + x) < H ? val : 0.f;
        }
        if (lane == 0) Vec8<__nv_bfloat16>::store(dst + a.push_l_off + g8, lv);
    }
    if (L.sub != 0) return;
#pragma unroll
    for (int i = 0; i < CPL; ++i) Vec8<__nv_bfloat16>::store(dst + foff[i], acc[i]);
}

// ------------------------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------------------------
template <typename T, int CPL, bool PEER>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, (CPL == 1 ? 6 : 3)) attn_fwd_kernel(AttnFwdArgs a) {
    extern __shared__ float smem[];
    const AttnCommon& c = a.c;
    const int H = c.H, D = c.D, HD = H * D;
    float* s_gate = smem;
    float* s_bias = smem + (c.score == SCORE_GATED ? c.T * HD : 0);
    load_tables(c, s_gate, s_bias);
    const Lanes L = make_lanes(HD, D);
    // row strides in elements (0 = dense rows of H*D): operands may be column slices of wider matrices, e.g. K | V | message
    const size_t ldq = c.ldq ? (size_t)c.ldq : (size_t)HD, ldk = c.ldk ? (size_t)c.ldk : (size_t)HD;
    const size_t ldr = c.ldr ? (size_t)c.ldr : (size_t)HD, ldo = c.ldo ? (size_t)c.ldo : (size_t)HD;
    (void)ldq; (void)ldk; (void)ldr; (void)ldo;
    const T* q = static_cast<const T*>(a.q);
    const T* kb = static_cast<const T*>(a.k);
    const T* vb = static_cast<const T*>(a.v);
    const bool softmax = c.norm == NORM_SOFTMAX;
    const bool head_writer = (L.ll & (L.lph - 1)) == 0;
    using Raw = typename Vec8<T>::Raw;
    constexpr int U = kUnrollFwd;
    int foff[CPL], head[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) { foff[i] = (L.ll + L.lpr * i) << 3; head[i] = foff[i] / D; }

    // persistent blocks: the tables are loaded once, warps stride over the segments
    const int n_warps = gridDim.x * kWarpsPerBlock;
    for (int seg = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); seg < c.plan.n_seg; seg += n_warps) {
        const int row = c.plan.seg_row[seg], beg = c.plan.seg_beg[seg], end = c.plan.seg_end[seg];
        const int slot = c.plan.seg_slot[seg];
        float qf[CPL][8], acc[CPL][8], l[CPL], m[CPL];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            Vec8<T>::load(q + (size_t)row * ldq + foff[i], qf[i]);
#pragma unroll
            for (int x = 0; x < 8; ++x) { qf[i][x] *= c.scale; acc[i][x] = 0.f; }
            l[i] = 0.f;
            m[i] = softmax ? -INFINITY : 0.f;
        }
        float qg[CPL][8];                 // q * scale * gate[type] of the type currently cached
        int gt_cached = -1;
        // indices of the first group; every iteration prefetches the next group's indices before it touches K / V
        int jn[U], tn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = beg + u * L.epw + L.sub;
            jn[u] = e < end ? c.idx[e] : -1;
            tn[u] = (e < end && c.etype) ? c.etype[e] : 0;
        }
        for (int base = beg; base < end; base += U * L.epw) {
            int j[U], t[U];
            Raw kr[U][CPL], vr[U][CPL];
#pragma unroll
            for (int u = 0; u < U; ++u) { j[u] = jn[u]; t[u] = tn[u]; }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (j[u] >= 0) {
                    const T* kp; const T* vp;
                    if (PEER) {
                        const int p = j[u] / a.rows_per_peer, r = j[u] - p * a.rows_per_peer;
                        kp = static_cast<const T*>(a.k_peers[p]) + (size_t)r * ldk;
                        vp = static_cast<const T*>(a.v_peers[p]) + (size_t)r * ldk;
                    } else {
                        kp = kb + (size_t)j[u] * ldk;
                        vp = vb + (size_t)j[u] * ldk;
                    }
#pragma unroll
                    for (int i = 0; i < CPL; ++i) { kr[u][i] = Vec8<T>::load_raw(kp + foff[i]); vr[u][i] = Vec8<T>::load_raw(vp + foff[i]); }
                } else {
#pragma unroll
                    for (int i = 0; i < CPL; ++i) { kr[u][i] = Vec8<T>::zero_raw(); vr[u][i] = Vec8<T>::zero_raw(); }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = base + (U + u) * L.epw + L.sub;
                jn[u] = e < end ? c.idx[e] : -1;
                tn[u] = (e < end && c.etype) ? c.etype[e] : 0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool ok = j[u] >= 0;
                if (c.score == SCORE_GATED && t[u] != gt_cached) {      // edges of a row are grouped by type: rare reload
                    gt_cached = t[u];
#pragma unroll
                    for (int i = 0; i < CPL; ++i) {
                        const float* g = s_gate + gt_cached * HD + foff[i];
#pragma unroll
                        for (int x = 0; x < 8; ++x) qg[i][x] = qf[i][x] * g[x];
                    }
                }
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    float kf[8], vf[8];
                    Vec8<T>::unpack(kr[u][i], kf);
                    float s = 0.f;
                    if (c.score == SCORE_GATED) {
#pragma unroll
                        for (int x = 0; x < 8; ++x) s = fmaf(qg[i][x], kf[x], s);
                    } else {
#pragma unroll
                        for (int x = 0; x < 8; ++x) s = fmaf(qf[i][x], kf[x], s);
                    }
                    s = head_sum(s, L.lph);
                    if (c.score == SCORE_BIASED) s += s_bias[t[u] * H + head[i]];
                    Vec8<T>::unpack(vr[u][i], vf);
                    if (softmax) {
                        const float mn = ok ? fmaxf(m[i], s) : m[i];
                        const float corr = safe_exp_diff(m[i], mn);
                        const float p = ok ? __expf(s - mn) : 0.f;
                        l[i] = l[i] * corr + p;
#pragma unroll
                        for (int x = 0; x < 8; ++x) acc[i][x] = fmaf(acc[i][x], corr, p * vf[x]);
                        m[i] = mn;
                    } else {
                        const float p = ok ? __expf(fminf(fmaxf(s, c.lo), c.hi)) : 0.f;
                        l[i] += p;
#pragma unroll
                        for (int x = 0; x < 8; ++x) acc[i][x] = fmaf(p, vf[x], acc[i][x]);
                    }
                }
            }
        }
        // merge the edge slots of the warp
        for (int off = L.lpr; off < 32; off <<= 1) {
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                const float mo = __shfl_xor_sync(GT_FULL_MASK, m[i], off);
                const float lo_ = __shfl_xor_sync(GT_FULL_MASK, l[i], off);
                float wa = 1.f, wb = 1.f;
                if (softmax) {
                    const float mn = fmaxf(m[i], mo);
                    wa = safe_exp_diff(m[i], mn);
                    wb = safe_exp_diff(mo, mn);
                    m[i] = mn;
                }
                l[i] = l[i] * wa + lo_ * wb;
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const float ao = __shfl_xor_sync(GT_FULL_MASK, acc[i][x], off);
                    acc[i][x] = acc[i][x] * wa + ao * wb;
                }
            }
        }
        if (a.push_n > 0 && slot < 0) {
            push_partial_row<CPL>(a, a.row_map ? a.row_map[row] : row, L, H, foff, acc, l);
            continue;
        }
        if (L.sub != 0) continue;
        if (slot < 0 && a.o != nullptr) {                // normalised output in the operand type
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                const float inv = softmax ? 1.f / (l[i] > 0.f ? l[i] : 1.f) : 1.f / (l[i] + a.eps);
#pragma unroll
                for (int x = 0; x < 8; ++x) acc[i][x] *= inv;
                Vec8<T>::store(static_cast<T*>(a.o) + (size_t)row * HD + foff[i], acc[i]);
                if (head_writer) {
                    a.l[(size_t)row * H + head[i]] = l[i];
                    if (a.m) a.m[(size_t)row * H + head[i]] = (m[i] == -INFINITY) ? 0.f : m[i];
                }
            }
        } else if (slot < 0) {
            const long long orow = a.row_map ? a.row_map[row] : row;
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                float* dst = a.acc + orow * a.acc_stride + foff[i];
                if (a.accumulate) {
                    float old[8];
                    Vec8<float>::load(dst, old);
#pragma unroll
                    for (int x = 0; x < 8; ++x) acc[i][x] += old[x];
                }
                Vec8<float>::store(dst, acc[i]);
                if (head_writer) {
                    float* lp = a.l + orow * a.l_stride + head[i];
                    *lp = a.accumulate ? *lp + l[i] : l[i];
                    if (a.m) a.m[orow * H + head[i]] = (m[i] == -INFINITY) ? 0.f : m[i];
                }
            }
        } else {
            float* sc = c.scratch + (size_t)slot * ((HD + 2 * H + 3) & ~3);
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                Vec8<float>::store(sc + foff[i], acc[i]);
                if (head_writer) { sc[HD + head[i]] = l[i]; sc[HD + H + head[i]] = m[i]; }
            }
        }
    }
}

// Sums over the slots [s0, s1) of four consecutive columns of a scratch area, by a block of (16, 8) threads: 64 columns, 8 thread rows
// striding over the slots, folded through shared memory in row order (the order of the sums is part of the result of a training step,
// so neither it nor the number of rows is changed lightly).  What bounds it is the latency of the chain of a hub row (the global token
// of 169 K nodes has 661 slots): eight loads are in flight per thread row.  With one 4-byte load at a time the three combines of an
// Exphormer layer (8 heads x 32) took 21 / 21 / 41 us.  The result is valid for threadIdx.y == 0.
constexpr int kSumX = 16, kSumY = 8;
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
template <typename F>
__device__ __forceinline__ float4 slots_sum(int s0, int s1, float4 (*sm)[kSumX], F load) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v = zero;
    for (int s = s0 + threadIdx.y; s < s1; s += 8 * kSumY) {
        float4 t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = s + k * kSumY < s1 ? load(s + k * kSumY) : zero;
#pragma unroll
        for (int k = 0; k < 8; ++k) v = add4(v, t[k]);
    }
    sm[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y == 0)
        for (int y = 1; y < kSumY; ++y) v = add4(v, sm[y][threadIdx.x]);
    return v;
}
template <typename T>
__device__ __forceinline__ void store4(T* p, float4 v) {
    p[0] = from_float<T>(v.x); p[1] = from_float<T>(v.y); p[2] = from_float<T>(v.z); p[3] = from_float<T>(v.w);
}

// Merge of the slots of a split row: grid (split rows, 64-column groups of acc), block (16, 8).  Softmax slots are rescaled to the
// common maximum of their head; clamp-exp slots add.
template <typename T>
__global__ void __launch_bounds__(kSumX * kSumY) attn_fwd_combine_kernel(AttnFwdArgs a) {
    __shared__ float4 sm[kSumY][kSumX];
    __shared__ float smx[kSumY][kSumX], sml[kSumY][kSumX];
    const AttnCommon& c = a.c;
    const int H = c.H, D = c.D, HD = H * D, W = (HD + 2 * H + 3) & ~3;     // slots are 16-byte aligned
    const int r = blockIdx.x, f = (blockIdx.y * kSumX + threadIdx.x) * 4, h = min(f, HD - 1) / D;
    const bool in = f < HD;
    const int row = c.plan.split_rows[r];
    const long long orow = a.row_map ? a.row_map[row] : row;
    const int s0 = c.plan.split_ptr[r], s1 = c.plan.split_ptr[r + 1];
    const float* base = c.scratch + (in ? f : 0);
    const float* lb = c.scratch + HD + h;
    const float* mb = lb + H;
    float mx = 0.f;
    if (c.norm == NORM_SOFTMAX) {
        mx = -INFINITY;
        for (int s = s0 + threadIdx.y; s < s1; s += 4 * kSumY)
#pragma unroll
            for (int k = 0; k < 4; ++k) mx = fmaxf(mx, mb[(size_t)min(s + k * kSumY, s1 - 1) * W]);
        smx[threadIdx.y][threadIdx.x] = mx;
        __syncthreads();
        for (int y = 0; y < kSumY; ++y) mx = fmaxf(mx, smx[y][threadIdx.x]);
        if (mx == -INFINITY) mx = 0.f;
    }
    float l = 0.f;
    const float4 acc = slots_sum(s0, s1, sm, [&](int s) {
        const float4 v = *reinterpret_cast<const float4*>(base + (size_t)s * W);
        const float w = c.norm == NORM_SOFTMAX ? __expf(mb[(size_t)s * W] - mx) : 1.f;
        l = fmaf(lb[(size_t)s * W], w, l);
        return make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
    });
    sml[threadIdx.y][threadIdx.x] = l;
    __syncthreads();
    if (threadIdx.y != 0 || !in) return;
    for (int y = 1; y < kSumY; ++y) l += sml[y][threadIdx.x];
    const bool first = f == h * D;
    if (a.push_n > 0) {                                  // split rows of the fused reduce-scatter: the merged row goes to its owner
        const int owner = (int)(orow / a.push_rows);
        __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.push_slot[owner]) + (orow - (long long)owner * a.push_rows) * a.push_ld;
        store4(dst + f, acc);
        if (first) dst[a.push_l_off + h] = __float2bfloat16(l);
        return;
    }
    if (a.o != nullptr) {
        const float inv = c.norm == NORM_SOFTMAX ? 1.f / (l > 0.f ? l : 1.f) : 1.f / (l + a.eps);
        store4(static_cast<T*>(a.o) + (size_t)row * HD + f, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
        if (first) {
            a.l[(size_t)row * H + h] = l;
            if (a.m) a.m[(size_t)row * H + h] = mx;
        }
        return;
    }
    float* dst = a.acc + orow * a.acc_stride + f;
    store4(dst, a.accumulate ? add4(make_float4(dst[0], dst[1], dst[2], dst[3]), acc) : acc);
    if (first) {
        float* lp = a.l + orow * a.l_stride + h;
        *lp = a.accumulate ? *lp + l : l;
        if (a.m) a.m[orow * H + h] = mx;
    }
}

// out[row] (+)= sum of the row's slots, columns [0, split) to out / out_f32 and [split, width) to out2 (dk | dv of the column pass)
template <typename T>
__global__ void __launch_bounds__(kSumX * kSumY) sum_slots_kernel(const SegPlan plan, const float* scratch, int width, int split, const int* row_map,
                                                                  T* out, T* out2, float* out_f32, int accumulate, long long ld) {
    __shared__ float4 sm[kSumY][kSumX];
    const int r = blockIdx.x, f = (blockIdx.y * kSumX + threadIdx.x) * 4;
    const int row = plan.split_rows[r];
    const long long orow = row_map ? row_map[row] : row;
    const float* base = scratch + (f < width ? f : 0);
    const float4 v = slots_sum(plan.split_ptr[r], plan.split_ptr[r + 1], sm,
                               [&](int s) { return *reinterpret_cast<const float4*>(base + (size_t)s * width); });
    if (threadIdx.y != 0 || f >= width) return;
    if (out_f32) {
        float* d = out_f32 + orow * ld + f;
        store4(d, accumulate ? add4(make_float4(d[0], d[1], d[2], d[3]), v) : v);
    } else if (f < split) {
        store4(out + orow * ld + f, v);
    } else {
        store4(out2 + orow * ld + f - split, v);
    }
}
dim3 sum_grid(int n_split, int width) { return dim3(n_split, (width + 4 * kSumX - 1) / (4 * kSumX)); }

// ------------------------------------------------------------------------------------------------------------------
// backward, row pass: dQ and the per-type gate / bias gradients
// ------------------------------------------------------------------------------------------------------------------
// Per row and edge type t the kernel accumulates A_t = sum_{edges of type t} ds_ij k_j.  Then dq_i = scale * sum_t g_t * A_t
// and the row's contribution to the gate gradient is q_i * scale * A_t: the per-edge work is one FMA set, and the per-type
// gradients are flushed to shared memory once per row instead of being carried in registers.
// End of a run of edges of one type in the row pass: dq += g_t * A, the gate gradient of the block += q * A, A = 0.
template <int CPL>
__device__ __forceinline__ void flush_type_run(const float* s_gate, float* s_dg, int t, int HD, const int (&foff)[CPL], const float (&qf)[CPL][8],
                                               float (&A)[CPL][8], float (&dqa)[CPL][8], bool want_dg) {
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const float* g = s_gate + t * HD + foff[i];
#pragma unroll
        for (int x = 0; x < 8; ++x) dqa[i][x] = fmaf(g[x], A[i][x], dqa[i][x]);
        if (want_dg) {
#pragma unroll
            for (int x = 0; x < 8; ++x) atomicAdd(&s_dg[t * HD + foff[i] + x], qf[i][x] * A[i][x]);
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) A[i][x] = 0.f;
    }
}

template <typename T, int CPL, bool GATED>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, (CPL == 1 ? 4 : 2)) attn_bwd_row_kernel(AttnBwdRowArgs a) {
    extern __shared__ float smem[];
    const AttnCommon& c = a.c;
    const int H = c.H, D = c.D, HD = H * D;
    float* s_gate = smem;
    float* s_bias = smem + (c.score == SCORE_GATED ? c.T * HD : 0);
    float* s_dg = s_bias + (c.score == SCORE_BIASED ? c.T * H : 0);      // [T, HD] or [T, H] block accumulators
    load_tables(c, s_gate, s_bias);
    const bool want_dg = GATED && a.dgate_part;
    const bool want_db = c.score == SCORE_BIASED && a.dbias_part;
    const int acc_n = want_dg ? c.T * HD : (want_db ? c.T * H : 0);
    for (int i = threadIdx.x; i < acc_n; i += blockDim.x) s_dg[i] = 0.f;
    __syncthreads();
    const Lanes L = make_lanes(HD, D);
    // row strides in elements (0 = dense rows of H*D): operands may be column slices of wider matrices, e.g. K | V | message
    const size_t ldq = c.ldq ? (size_t)c.ldq : (size_t)HD, ldk = c.ldk ? (size_t)c.ldk : (size_t)HD;
    const size_t ldr = c.ldr ? (size_t)c.ldr : (size_t)HD, ldo = c.ldo ? (size_t)c.ldo : (size_t)HD;
    (void)ldq; (void)ldk; (void)ldr; (void)ldo;
    const bool softmax = c.norm == NORM_SOFTMAX;
    const T* q = static_cast<const T*>(a.q);
    const T* kb = static_cast<const T*>(a.k);
    const T* vb = static_cast<const T*>(a.v);
    const T* rvb = static_cast<const T*>(a.row_vec);
    const bool head_writer = (L.ll & (L.lph - 1)) == 0;
    using Raw = typename Vec8<T>::Raw;
    constexpr int U = kUnrollRow;
    int foff[CPL], head[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) { foff[i] = (L.ll + L.lpr * i) << 3; head[i] = foff[i] / D; }

    const int n_warps = gridDim.x * kWarpsPerBlock;
    for (int seg = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); seg < c.plan.n_seg; seg += n_warps) {
        const int row = c.plan.seg_row[seg], beg = c.plan.seg_beg[seg], end = c.plan.seg_end[seg];
        const int slot = c.plan.seg_slot[seg];
        const long long srow = a.row_map ? a.row_map[row] : row;     // row of q / row_vec / stat / dq
        // A: sum of ds * k over the edges of the CURRENT type run (gated) or of the whole row; dqa: dq accumulated over finished runs
        float qf[CPL][8], rv[CPL][8], A[CPL][8], dqa[CPL][8], db[kMaxTypesReg][CPL], mrow[CPL], rb[CPL], ps[CPL];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            Vec8<T>::load(q + srow * ldq + foff[i], qf[i]);
            Vec8<T>::load(rvb + srow * ldr + foff[i], rv[i]);
            const float4 st = a.stat[srow * H + head[i]];
            mrow[i] = st.x; rb[i] = st.y; ps[i] = st.z;
#pragma unroll
            for (int x = 0; x < 8; ++x) qf[i][x] *= c.scale;
#pragma unroll
            for (int x = 0; x < 8; ++x) { A[i][x] = 0.f; dqa[i][x] = 0.f; }
#pragma unroll
            for (int tt = 0; tt < kMaxTypesReg; ++tt) db[tt][i] = 0.f;
        }
        float qg[CPL][8];
        int gt_cached = -1;
        const int n_it = (end - beg + U * L.epw - 1) / (U * L.epw);
        int jn[U], tn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = beg + u * L.epw + L.sub;
            jn[u] = e < end ? c.idx[e] : -1;
            tn[u] = (e < end && c.etype) ? c.etype[e] : 0;
        }
        for (int it = 0; it < n_it; ++it) {
            const int base = beg + it * U * L.epw;
            int j[U], t[U];
            Raw kr[U][CPL], vr[U][CPL];
#pragma unroll
            for (int u = 0; u < U; ++u) { j[u] = jn[u]; t[u] = tn[u]; }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (j[u] >= 0) {
#pragma unroll
                    for (int i = 0; i < CPL; ++i) {
                        kr[u][i] = Vec8<T>::load_raw(kb + (size_t)j[u] * ldk + foff[i]);
                        vr[u][i] = Vec8<T>::load_raw(vb + (size_t)j[u] * ldk + foff[i]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < CPL; ++i) { kr[u][i] = Vec8<T>::zero_raw(); vr[u][i] = Vec8<T>::zero_raw(); }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = base + (U + u) * L.epw + L.sub;
                jn[u] = e < end ? c.idx[e] : -1;
                tn[u] = (e < end && c.etype) ? c.etype[e] : 0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool ok = j[u] >= 0;
                if (GATED && ok && t[u] != gt_cached) {                 // edges of a row are grouped by type: a run ends (rare)
                    if (gt_cached >= 0) flush_type_run<CPL>(s_gate, s_dg, gt_cached, HD, foff, qf, A, dqa, want_dg);
                    gt_cached = t[u];
#pragma unroll
                    for (int i = 0; i < CPL; ++i) {
                        const float* g = s_gate + gt_cached * HD + foff[i];
#pragma unroll
                        for (int x = 0; x < 8; ++x) qg[i][x] = qf[i][x] * g[x];
                    }
                }
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    float kf[8], vf[8];
                    Vec8<T>::unpack(kr[u][i], kf);
                    Vec8<T>::unpack(vr[u][i], vf);
                    float s = 0.f, dp = 0.f;
                    if (GATED) {
#pragma unroll
                        for (int x = 0; x < 8; ++x) s = fmaf(qg[i][x], kf[x], s);
                    } else {
#pragma unroll
                        for (int x = 0; x < 8; ++x) s = fmaf(qf[i][x], kf[x], s);
                    }
#pragma unroll
                    for (int x = 0; x < 8; ++x) dp = fmaf(rv[i][x], vf[x], dp);
                    for (int o = L.lph >> 1; o > 0; o >>= 1) {
                        s += __shfl_xor_sync(GT_FULL_MASK, s, o);
                        dp += __shfl_xor_sync(GT_FULL_MASK, dp, o);
                    }
                    if (c.score == SCORE_BIASED) s += s_bias[t[u] * H + head[i]];
                    float p, mask = 1.f;
                    if (softmax) {
                        p = __expf(s - mrow[i]);
                    } else {
                        p = __expf(fminf(fmaxf(s, c.lo), c.hi));
                        mask = (s >= c.lo && s <= c.hi) ? 1.f : 0.f;
                    }
                    const float ds = ok ? p * ps[i] * (dp + rb[i]) * mask : 0.f;
#pragma unroll
                    for (int x = 0; x < 8; ++x) A[i][x] = fmaf(ds, kf[x], A[i][x]);
                    if (!GATED) {
                        if (want_db) {
#pragma unroll
                            for (int tt = 0; tt < kMaxTypesReg; ++tt)
                                if (t[u] == tt) db[tt][i] += ds;
                        }
                    }
                }
            }
        }
        if (GATED) {
            if (gt_cached >= 0) flush_type_run<CPL>(s_gate, s_dg, gt_cached, HD, foff, qf, A, dqa, want_dg);
        } else {
#pragma unroll
            for (int i = 0; i < CPL; ++i)
#pragma unroll
                for (int x = 0; x < 8; ++x) dqa[i][x] = A[i][x];
        }
        // merge the edge slots of the warp
        for (int off = L.lpr; off < 32; off <<= 1) {
#pragma unroll
            for (int i = 0; i < CPL; ++i)
#pragma unroll
                for (int x = 0; x < 8; ++x) dqa[i][x] += __shfl_xor_sync(GT_FULL_MASK, dqa[i][x], off);
            if (want_db) {
#pragma unroll
                for (int tt = 0; tt < kMaxTypesReg; ++tt)
#pragma unroll
                    for (int i = 0; i < CPL; ++i) db[tt][i] += __shfl_xor_sync(GT_FULL_MASK, db[tt][i], off);
            }
        }
        if (L.sub != 0) continue;
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            float dq[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) dq[x] = dqa[i][x];
            if (!GATED && want_db && head_writer) {
#pragma unroll
                for (int tt = 0; tt < kMaxTypesReg; ++tt)
                    if (tt < c.T) atomicAdd(&s_dg[tt * H + head[i]], db[tt][i]);
            }
#pragma unroll
            for (int x = 0; x < 8; ++x) dq[x] *= c.scale;
            if (slot >= 0) {
                Vec8<float>::store(c.scratch + (size_t)slot * HD + foff[i], dq);
            } else if (a.accumulate_dq) {
                float* dst = static_cast<float*>(a.dq) + srow * ldo + foff[i];
                float old[8];
                Vec8<float>::load(dst, old);
#pragma unroll
                for (int x = 0; x < 8; ++x) old[x] += dq[x];
                Vec8<float>::store(dst, old);
            } else {
                Vec8<T>::store(static_cast<T*>(a.dq) + srow * ldo + foff[i], dq);
            }
        }
    }
    __syncthreads();
    float* part = want_dg ? a.dgate_part + (size_t)blockIdx.x * acc_n : (want_db ? a.dbias_part + (size_t)blockIdx.x * acc_n : nullptr);
    for (int i = threadIdx.x; i < acc_n; i += blockDim.x) part[i] = s_dg[i];
}

// ------------------------------------------------------------------------------------------------------------------
// backward, column pass: dK, dV over the CSC (no atomics)
// ------------------------------------------------------------------------------------------------------------------
template <typename T, int CPL>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, (CPL == 1 ? 5 : 2)) attn_bwd_col_kernel(AttnBwdColArgs a) {
    extern __shared__ float smem[];
    const AttnCommon& c = a.c;
    const int H = c.H, D = c.D, HD = H * D;
    float* s_gate = smem;
    float* s_bias = smem + (c.score == SCORE_GATED ? c.T * HD : 0);
    load_tables(c, s_gate, s_bias);
    const Lanes L = make_lanes(HD, D);
    // row strides in elements (0 = dense rows of H*D): operands may be column slices of wider matrices, e.g. K | V | message
    const size_t ldq = c.ldq ? (size_t)c.ldq : (size_t)HD, ldk = c.ldk ? (size_t)c.ldk : (size_t)HD;
    const size_t ldr = c.ldr ? (size_t)c.ldr : (size_t)HD, ldo = c.ldo ? (size_t)c.ldo : (size_t)HD;
    (void)ldq; (void)ldk; (void)ldr; (void)ldo;
    const bool softmax = c.norm == NORM_SOFTMAX;
    const T* qb = static_cast<const T*>(a.q);
    const T* rvb = static_cast<const T*>(a.row_vec);
    using Raw = typename Vec8<T>::Raw;
    constexpr int U = kUnrollCol;
    int foff[CPL], head[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) { foff[i] = (L.ll + L.lpr * i) << 3; head[i] = foff[i] / D; }

    const int n_warps = gridDim.x * kWarpsPerBlock;
    for (int seg = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); seg < c.plan.n_seg; seg += n_warps) {
        const int colj = c.plan.seg_row[seg], beg = c.plan.seg_beg[seg], end = c.plan.seg_end[seg];
        const int slot = c.plan.seg_slot[seg];
        float kf[CPL][8], vf[CPL][8], dk[CPL][8], dv[CPL][8];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            Vec8<T>::load(static_cast<const T*>(a.k) + (size_t)colj * ldk + foff[i], kf[i]);
            Vec8<T>::load(static_cast<const T*>(a.v) + (size_t)colj * ldk + foff[i], vf[i]);
#pragma unroll
            for (int x = 0; x < 8; ++x) { dk[i][x] = 0.f; dv[i][x] = 0.f; }
        }
        float gc[CPL][8], kg[CPL][8];       // cached gate slice and k * gate of the type currently being walked
        int gt_cached = -1;
        const int n_it = (end - beg + U * L.epw - 1) / (U * L.epw);
        int rn[U], tn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = beg + u * L.epw + L.sub;
            rn[u] = e < end ? c.idx[e] : -1;
            tn[u] = (e < end && c.etype) ? c.etype[e] : 0;
        }
        for (int it = 0; it < n_it; ++it) {
            const int base = beg + it * U * L.epw;
            int r[U], t[U];
            Raw qr[U][CPL], rr[U][CPL];
            float4 st[U][CPL];
#pragma unroll
            for (int u = 0; u < U; ++u) { r[u] = rn[u]; t[u] = tn[u]; }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (r[u] >= 0) {
#pragma unroll
                    for (int i = 0; i < CPL; ++i) {
                        qr[u][i] = Vec8<T>::load_raw(qb + (size_t)r[u] * ldq + foff[i]);
                        rr[u][i] = Vec8<T>::load_raw(rvb + (size_t)r[u] * ldr + foff[i]);
                        st[u][i] = __ldg(a.stat + (size_t)r[u] * H + head[i]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < CPL; ++i) {
                        qr[u][i] = Vec8<T>::zero_raw(); rr[u][i] = Vec8<T>::zero_raw();
                        st[u][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = base + (U + u) * L.epw + L.sub;
                rn[u] = e < end ? c.idx[e] : -1;
                tn[u] = (e < end && c.etype) ? c.etype[e] : 0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool ok = r[u] >= 0;
                // CSR position of this entry, for the score gradients handed to the row pass (loaded ahead of the arithmetic)
                const int pe = (a.ds_out != nullptr && ok) ? a.pos[base + u * L.epw + L.sub] : 0;
                if (c.score == SCORE_GATED && t[u] != gt_cached) {      // a column's entries are grouped by type: rare reload
                    gt_cached = t[u];
#pragma unroll
                    for (int i = 0; i < CPL; ++i) {
                        const float* g = s_gate + gt_cached * HD + foff[i];
#pragma unroll
                        for (int x = 0; x < 8; ++x) { gc[i][x] = g[x]; kg[i][x] = kf[i][x] * g[x]; }
                    }
                }
#pragma unroll
                for (int i = 0; i < CPL; ++i) {
                    float qf[8], rv[8];
                    Vec8<T>::unpack(qr[u][i], qf);
                    Vec8<T>::unpack(rr[u][i], rv);
                    float s = 0.f, dp = 0.f;
                    if (c.score == SCORE_GATED) {
#pragma unroll
                        for (int x = 0; x < 8; ++x) s = fmaf(qf[x], kg[i][x], s);
                    } else {
#pragma unroll
                        for (int x = 0; x < 8; ++x) s = fmaf(qf[x], kf[i][x], s);
                    }
#pragma unroll
                    for (int x = 0; x < 8; ++x) dp = fmaf(rv[x], vf[i][x], dp);
                    for (int o = L.lph >> 1; o > 0; o >>= 1) {
                        s += __shfl_xor_sync(GT_FULL_MASK, s, o);
                        dp += __shfl_xor_sync(GT_FULL_MASK, dp, o);
                    }
                    s *= c.scale;
                    if (c.score == SCORE_BIASED) s += s_bias[t[u] * H + head[i]];
                    float p, mask = 1.f;
                    if (softmax) {
                        p = __expf(s - st[u][i].x);
                    } else {
                        p = __expf(fminf(fmaxf(s, c.lo), c.hi));
                        mask = (s >= c.lo && s <= c.hi) ? 1.f : 0.f;
                    }
                    const float P = ok ? p * st[u][i].z : 0.f;
                    const float ds0 = P * (dp + st[u][i].y) * mask;
                    const float ds = ds0 * c.scale;
                    if (a.ds_out != nullptr && ok && (foff[i] % D) == 0) a.ds_out[(size_t)pe * H + head[i]] = ds0;
#pragma unroll
                    for (int x = 0; x < 8; ++x) dv[i][x] = fmaf(P, rv[x], dv[i][x]);
                    if (c.score == SCORE_GATED) {
#pragma unroll
                        for (int x = 0; x < 8; ++x) dk[i][x] = fmaf(ds * qf[x], gc[i][x], dk[i][x]);
                    } else {
#pragma unroll
                        for (int x = 0; x < 8; ++x) dk[i][x] = fmaf(ds, qf[x], dk[i][x]);
                    }
                }
            }
        }
        for (int off = L.lpr; off < 32; off <<= 1)
#pragma unroll
            for (int i = 0; i < CPL; ++i)
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    dk[i][x] += __shfl_xor_sync(GT_FULL_MASK, dk[i][x], off);
                    dv[i][x] += __shfl_xor_sync(GT_FULL_MASK, dv[i][x], off);
                }
        if (L.sub != 0) continue;
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            if (slot >= 0) {
                Vec8<float>::store(c.scratch + (size_t)slot * 2 * HD + foff[i], dk[i]);
                Vec8<float>::store(c.scratch + (size_t)slot * 2 * HD + HD + foff[i], dv[i]);
            } else {
                Vec8<T>::store(static_cast<T*>(a.dk) + (size_t)colj * ldo + foff[i], dk[i]);
                Vec8<T>::store(static_cast<T*>(a.dv) + (size_t)colj * ldo + foff[i], dv[i]);
            }
        }
    }
}

// Row statistics of the normalised backward.  D / 8 lanes read a head's dO and o once (2 x 87 MB for 169 K nodes x 256 bf16): bound by
// that traffic.  As tensor operations (two casts, product, sum, reciprocal, stack) it took 0.70 ms of a 2.33 ms forward + backward.
template <typename T>
__global__ void attn_bwd_stat_kernel(const T* __restrict__ dout, const T* __restrict__ o, const float* __restrict__ l, const float* __restrict__ m,
                                     float4* __restrict__ stat, long long chunks, int lph, int softmax, float eps) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long end = (chunks + 31) / 32 * 32;                 // whole warps take part in the shuffles
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < end; i += stride) {
        float d = 0.f;
        if (i < chunks) {
            float a[8], b[8];
            Vec8<T>::load_nc(dout + i * 8, a);
            Vec8<T>::load_nc(o + i * 8, b);
#pragma unroll
            for (int x = 0; x < 8; ++x) d = fmaf(a[x], b[x], d);
        }
        d = head_sum(d, lph);
        if (i < chunks && i % lph == 0) {
            const long long r = i / lph;
            const float lv = l[r];
            stat[r] = make_float4(m ? m[r] : 0.f, -d, softmax ? 1.f / (lv > 0.f ? lv : 1.f) : 1.f / (lv + eps), 0.f);
        }
    }
}

// out[i] = sum_b part[b, i]: a block owns 32 columns, its thread rows stride over the partial blocks (coalesced 128-byte reads), the
// sums are folded through shared memory in a fixed order (deterministic).  Bound by the latency of a thread row's chain of loads (up to
// 1776 partial blocks): 32 thread rows with eight loads in flight each.  Eight rows with one load at a time took 21 us for 1776 x 768.
constexpr int kFoldRows = 32;
__global__ void __launch_bounds__(32 * kFoldRows) reduce_partials_kernel(const float* __restrict__ part, int n_blocks, int width, float* out, int accumulate) {
    __shared__ float sm[kFoldRows][33];
    const int i = blockIdx.x * 32 + threadIdx.x;
    float v = 0.f;
    if (i < width) {
        int b = threadIdx.y;
        for (; b + 7 * kFoldRows < n_blocks; b += 8 * kFoldRows) {
            float t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = __ldg(part + (size_t)(b + k * kFoldRows) * width + i);
#pragma unroll
            for (int k = 0; k < 8; ++k) v += t[k];
        }
        for (; b < n_blocks; b += kFoldRows) v += __ldg(part + (size_t)b * width + i);
    }
    sm[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y == 0 && i < width) {
        float t = 0.f;
#pragma unroll
        for (int y = 0; y < kFoldRows; ++y) t += sm[y][threadIdx.x];
        out[i] = accumulate ? out[i] + t : t;
    }
}

size_t table_bytes(const AttnCommon& c) {
    size_t n = 0;
    if (c.score == SCORE_GATED) n += (size_t)c.T * c.H * c.D;
    if (c.score == SCORE_BIASED) n += (size_t)c.T * c.H;
    return n * sizeof(float);
}

int cpl_of(int H, int D) { return (H * D / 8) > 32 ? (H * D / 8) / 32 : 1; }

template <typename K>
void set_smem(K kernel, size_t bytes) {
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

bool attn_shape_supported(int H, int D, int T) {
    int HD = H * D;
    if (D < 8 || (D & (D - 1)) || D > 256) return false;          // a head spans a power-of-two number of 8-chunks
    int nch = HD / 8;
    if (nch < 32) { if (nch & (nch - 1)) return false; }
    else if (nch != 32 && nch != 64) return false;                // H*D in {.., 256, 512}
    if (D / 8 > 32) return false;
    if (T > kMaxTypesReg) return false;                           // per-type gradients live in registers
    return true;
}

int attn_scratch_width_fwd(int H, int D) { return (H * D + 2 * H + 3) & ~3; }

int attn_bwd_row_blocks(int n_seg) {
    int want = (n_seg + kWarpsPerBlock - 1) / kWarpsPerBlock;
    int cap = 148 * 6;                  // one resident wave of the row pass
    return want < cap ? (want > 0 ? want : 1) : cap;
}

void attn_fwd(const AttnFwdArgs& a, cudaStream_t s) {
    const AttnCommon& c = a.c;
    if (c.plan.n_seg == 0) return;
    if (a.k_peers == nullptr && c.dtype == DT_BF16 && edge::fits(c)) {
        edge::fwd(a, s);
    } else {
        // fp32 operands (their ring of 64 KB a block leaves the edge kernels 12 warps per SM: 0.20 against 0.085 ms for 40 K nodes, 0.76 M
        // edges, 8 heads x 16), K / V rows in peer memory, or more gathered rows than the packed edge words address
        const int blocks = std::min((c.plan.n_seg + kWarpsPerBlock - 1) / kWarpsPerBlock, 148 * 24);
        const size_t sm = table_bytes(c);
        const bool peer = a.k_peers != nullptr;
        auto launch = [&](auto* kernel) {
            set_smem(kernel, sm);
            kernel<<<blocks, kWarpsPerBlock * 32, sm, s>>>(a);
        };
        const bool one = cpl_of(c.H, c.D) == 1;
        if (c.dtype == DT_BF16) {
            if (one) launch(peer ? attn_fwd_kernel<__nv_bfloat16, 1, true> : attn_fwd_kernel<__nv_bfloat16, 1, false>);
            else launch(peer ? attn_fwd_kernel<__nv_bfloat16, 2, true> : attn_fwd_kernel<__nv_bfloat16, 2, false>);
        } else {
            if (one) launch(peer ? attn_fwd_kernel<float, 1, true> : attn_fwd_kernel<float, 1, false>);
            else launch(peer ? attn_fwd_kernel<float, 2, true> : attn_fwd_kernel<float, 2, false>);
        }
    }
    if (c.plan.n_split > 0) {
        const dim3 grid = sum_grid(c.plan.n_split, c.H * c.D), block(kSumX, kSumY);
        if (c.dtype == DT_BF16) attn_fwd_combine_kernel<__nv_bfloat16><<<grid, block, 0, s>>>(a);
        else attn_fwd_combine_kernel<float><<<grid, block, 0, s>>>(a);
    }
}

void attn_bwd_row(const AttnBwdRowArgs& a_in, cudaStream_t s) {
    AttnBwdRowArgs a = a_in;
    const AttnCommon& c = a.c;
    if (c.plan.n_seg == 0) return;
    if (a.n_blocks <= 0) a.n_blocks = attn_bwd_row_blocks(c.plan.n_seg);
    const int HD = c.H * c.D;
    if (a.ds_in != nullptr && edge::fits(c)) {
        edge::row(a, s);                                 // the column pass ran first and left the score gradients
    } else {
        size_t sm = table_bytes(c);
        if (c.score == SCORE_GATED && a.dgate_part) sm += (size_t)c.T * HD * sizeof(float);
        if (c.score == SCORE_BIASED && a.dbias_part) sm += (size_t)c.T * c.H * sizeof(float);
        auto launch = [&](auto* kernel) {
            set_smem(kernel, sm);
            kernel<<<a.n_blocks, kWarpsPerBlock * 32, sm, s>>>(a);
        };
        const bool one = cpl_of(c.H, c.D) == 1, gated = c.score == SCORE_GATED;
        if (c.dtype == DT_BF16) {
            if (one) launch(gated ? attn_bwd_row_kernel<__nv_bfloat16, 1, true> : attn_bwd_row_kernel<__nv_bfloat16, 1, false>);
            else launch(gated ? attn_bwd_row_kernel<__nv_bfloat16, 2, true> : attn_bwd_row_kernel<__nv_bfloat16, 2, false>);
        } else {
            if (one) launch(gated ? attn_bwd_row_kernel<float, 1, true> : attn_bwd_row_kernel<float, 1, false>);
            else launch(gated ? attn_bwd_row_kernel<float, 2, true> : attn_bwd_row_kernel<float, 2, false>);
        }
    }
    if (c.plan.n_split > 0) {
        auto sum = [&](auto* out) {
            using T = std::remove_pointer_t<decltype(out)>;
            sum_slots_kernel<T><<<sum_grid(c.plan.n_split, HD), dim3(kSumX, kSumY), 0, s>>>(
                c.plan, c.scratch, HD, HD, a.row_map, out, nullptr, a.accumulate_dq ? static_cast<float*>(a.dq) : nullptr, a.accumulate_dq,
                c.ldo ? c.ldo : HD);
        };
        if (c.dtype == DT_BF16) sum(static_cast<__nv_bfloat16*>(a.dq));
        else sum(static_cast<float*>(a.dq));
    }
}

void attn_bwd_col(const AttnBwdColArgs& a, cudaStream_t s) {
    const AttnCommon& c = a.c;
    if (c.plan.n_seg == 0) return;
    const int HD = c.H * c.D;
    if (c.dtype == DT_BF16 && edge::fits(c)) {
        edge::col(a, s);
    } else {                                             // fp32 (see attn_fwd; 0.24 against 0.19 ms) or a very large row count
        const int blocks = std::min((c.plan.n_seg + kWarpsPerBlock - 1) / kWarpsPerBlock, 148 * 24);
        const size_t sm = table_bytes(c);
        auto launch = [&](auto* kernel) {
            set_smem(kernel, sm);
            kernel<<<blocks, kWarpsPerBlock * 32, sm, s>>>(a);
        };
        const bool one = cpl_of(c.H, c.D) == 1;
        if (c.dtype == DT_BF16) launch(one ? attn_bwd_col_kernel<__nv_bfloat16, 1> : attn_bwd_col_kernel<__nv_bfloat16, 2>);
        else launch(one ? attn_bwd_col_kernel<float, 1> : attn_bwd_col_kernel<float, 2>);
    }
    if (c.plan.n_split > 0) {
        auto sum = [&](auto* dk, auto* dv) {
            using T = std::remove_pointer_t<decltype(dk)>;
            sum_slots_kernel<T><<<sum_grid(c.plan.n_split, 2 * HD), dim3(kSumX, kSumY), 0, s>>>(c.plan, c.scratch, 2 * HD, HD, nullptr, dk, dv, nullptr,
                                                                                               0, c.ldo ? c.ldo : HD);
        };
        if (c.dtype == DT_BF16) sum(static_cast<__nv_bfloat16*>(a.dk), static_cast<__nv_bfloat16*>(a.dv));
        else sum(static_cast<float*>(a.dk), static_cast<float*>(a.dv));
    }
}

void attn_bwd_stat(int dtype, const void* dout, const void* o, const float* l, const float* m, void* stat, long long rows, int D, bool softmax, float eps,
                   cudaStream_t s) {
    if (rows <= 0) return;
    const long long chunks = rows * (D / 8);
    const int blocks = (int)std::min<long long>((chunks + 255) / 256, 148 * 16);
    if (dtype == DT_BF16)
        attn_bwd_stat_kernel<<<blocks, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(o), l, m,
                                                    static_cast<float4*>(stat), chunks, D / 8, softmax, eps);
    else
        attn_bwd_stat_kernel<<<blocks, 256, 0, s>>>(static_cast<const float*>(dout), static_cast<const float*>(o), l, m, static_cast<float4*>(stat), chunks,
                                                    D / 8, softmax, eps);
}

namespace {
KernelInfo info_of(const char* name, const void* kernel, size_t dyn_smem) {
    KernelInfo r{name, 0, 0, 0, (int)dyn_smem, 0};
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) { cudaGetLastError(); return r; }
    r.regs = fa.numRegs; r.local_bytes = (int)fa.localSizeBytes; r.static_smem = (int)fa.sharedSizeBytes;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r.blocks_per_sm, kernel, kWarpsPerBlock * 32, dyn_smem) != cudaSuccess) cudaGetLastError();
    return r;
}
}  // namespace

// Compiled resources of the attention kernels that serve bf16 operands with 8 heads of 32 and three edge types, and of the generic
// register kernels: registers per thread, local-memory bytes, shared memory and resident blocks per SM.  (The names are those that
// the kernel model's reports have always used for these passes.)
std::vector<KernelInfo> attn_kernel_info() {
    const size_t tbl = (size_t)3 * 256 * sizeof(float);
    std::vector<KernelInfo> v;
    AttnFwdArgs f{};
    AttnBwdColArgs cc{};
    AttnBwdRowArgs rr{};
    f.c.H = 8; f.c.D = 32; f.c.T = 3; f.c.score = SCORE_GATED; f.c.norm = NORM_CLAMPEXP; f.c.dtype = DT_BF16;
    cc.c = rr.c = f.c;
    float dummy = 0.f;
    rr.dgate_part = &dummy;
    v.push_back(info_of("fwd_ring_bf16_8x32", edge::fwd_8x32_bf16(), edge::fwd_smem(f)));
    v.push_back(info_of("fwd_regs_bf16", reinterpret_cast<const void*>(&attn_fwd_kernel<__nv_bfloat16, 1, false>), tbl));
    v.push_back(info_of("fwd_regs_fp32", reinterpret_cast<const void*>(&attn_fwd_kernel<float, 1, false>), tbl));
    v.push_back(info_of("row_ring_bf16_8x32", edge::row_8x32_bf16(), edge::row_smem(rr)));
    v.push_back(info_of("row_regs_bf16", reinterpret_cast<const void*>(&attn_bwd_row_kernel<__nv_bfloat16, 1, true>), 2 * tbl));
    v.push_back(info_of("col_ring_bf16_8x32", edge::col_8x32_bf16(), edge::col_smem(cc)));
    v.push_back(info_of("col_regs_bf16", reinterpret_cast<const void*>(&attn_bwd_col_kernel<__nv_bfloat16, 1>), tbl));
    return v;
}

void reduce_partials(const float* part, int n_blocks, int width, float* out, cudaStream_t s, int accumulate) {
    if (width <= 0) return;
    reduce_partials_kernel<<<(width + 31) / 32, dim3(32, kFoldRows), 0, s>>>(part, n_blocks, width, out, accumulate);
}

}  // namespace gt
