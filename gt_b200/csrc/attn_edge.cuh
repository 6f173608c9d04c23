// Edge-gather attention kernels (forward, column pass, row pass from stored score gradients).
//
// What bounds them: every edge moves one or two gathered feature rows of up to 512 bytes through the load path and does a few
// hundred multiply-adds on them, so the limits are the gather traffic and, long before that is reached, the number of warp
// instructions spent per edge.  The previous kernels (one 16-byte chunk per lane, a cp.async ring in shared memory, every lane of a
// head repeating the head's softmax arithmetic) issued 183 / 95 warp instructions per edge in the column / row pass (8 heads of 32,
// bf16) and ran at 60 % of the issue slots and 20 % of the L2 throughput.  Here:
//   * a lane owns 8 consecutive features (16 bytes of bf16); a feature row of up to 256 features is covered by LPR = H*D/8 lanes, a
//     warp walks one segment with 32 / LPR edges side by side, and 512 features are two independent halves of the heads (grid.y);
//   * the indices and types of 32 edges are fetched by one coalesced load and handed round by shuffles, the type only matters where it
//     changes (found once per 32 edges by a ballot), and everything that steers the loop is uniform over the warp;
//   * gathered rows go through a two-stage ring in shared memory (cp.async, a thread copies and reads only its own 16 bytes): the next
//     group of four edges per lane group is in flight while the current one is computed, also across the end of a segment;
//   * the dot products of four edges are finished by a transposing reduction, after which every lane of a head holds ONE edge's
//     score: exponential, clamp, statistics and score gradient are evaluated once per (edge, head) instead of once per lane;
//   * accumulations are packed pairs (fma.rn.f32x2): half the issue slots for the same fp32 arithmetic.
// Rows by direct loads into registers (no ring) needed 32 registers a group more and spilled or halved the warps in flight: 0.44 /
// 1.05 / 0.50 ms against 0.36 / 0.69 / 0.37 ms for the three passes (ring kernels replaced: 0.61 / 1.07 / 0.53) (169 K nodes, 4.03 M edges, 8 heads x 32).  A plain gather of the
// same rows runs at 12.4 TB/s when the operands are 174 MB (19 TB/s at 87 MB, 8 TB/s at 512 MB, measured with 512-byte rows), which
// puts the floor of the forward at 0.31 ms.
// The sums over the features of a head, over the edges of a segment and over the lane groups are taken in the same order as by the
// kernels these replace, so that clamp-exp training steps (heads of 32) continue bit for bit.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace gt {
namespace edge {

constexpr int kWarps = 4, kThreads = kWarps * 32;
constexpr int kU = 4;                              // edges per group (the transposing reduction works on four)
// Edges per group of the row pass (one gathered row each): with edge types, longer groups nearly always contain a change of the type
// and lose the path without tests (8 heads x 32, 4 M edges: 4 per group 0.39 ms, 8 per group 0.48 ms); without types 8 are better
// (4 heads x 32, 13.8 M edges: 0.40 against 0.45 ms).
__host__ __device__ constexpr int row_group(bool gated, int epw) { return gated || epw == 0 ? 4 : 8; }

// ---- host side ------------------------------------------------------------------------------------------------------------
void fwd(const AttnFwdArgs& a, cudaStream_t s);          // bf16
void col(const AttnBwdColArgs& a, cudaStream_t s);       // bf16
void row(const AttnBwdRowArgs& a, cudaStream_t s);       // needs a.ds_in
const void* fwd_8x32_bf16();                             // the instances of the common shape, for resource reports
const void* col_8x32_bf16();
const void* row_8x32_bf16();
// The packed edge word keeps 29 bits of index, and row offsets are 32-bit index x 32-bit row bytes.
inline bool fits(const AttnCommon& c) { return c.n_src <= (1ll << 29) && c.ldq < (1ll << 28) && c.ldk < (1ll << 28) && c.ldr < (1ll << 28); }
// compile-time lane layout of a launch: heads of 32 in rows of 256 (512: two halves) or 128, the common model shapes; 0 = any
inline int epw_code(const AttnCommon& c) { return c.D == 32 ? (c.H * c.D >= 256 ? 1 : (c.H * c.D == 128 ? 2 : 0)) : 0; }
inline int half_count(const AttnCommon& c) { return c.H * c.D > 256 ? c.H * c.D / 256 : 1; }
// Blocks of a pass that walks the segments with a stride of all warps; the segment order is balanced for 148 * 24 * 4 of them.
inline int grid_blocks(const AttnCommon& c, int cap) {
    const int want = (c.plan.n_seg + kWarps - 1) / kWarps;
    return want < cap ? want : cap;
}
// Shared-memory layout, in floats; every offset is a multiple of 4 floats (16 bytes).  The host sizes the launch and the kernels find
// their parts with the same functions: tables | gradient tables (row pass) | ring.
__host__ __device__ inline int slice_width(const AttnCommon& c) { return c.H * c.D > 256 ? 256 : c.H * c.D; }
__host__ __device__ inline int table_floats(const AttnCommon& c) {
    const int n = c.score == SCORE_GATED ? c.T * slice_width(c) : (c.score == SCORE_BIASED ? c.T * (slice_width(c) / c.D) : 0);
    return (n + 3) & ~3;
}
__host__ __device__ inline int grad_floats(const AttnBwdRowArgs& a) {
    if (a.c.score == SCORE_GATED) return a.dgate_part != nullptr ? kWarps * a.c.T * 256 : 0;
    return a.c.score == SCORE_BIASED && a.dbias_part != nullptr ? kThreads * a.c.T : 0;
}
__host__ __device__ inline int ring_floats(int dtype, int rows, int n) { return 2 * rows * n * kThreads * (dtype == DT_BF16 ? 4 : 8); }
inline size_t fwd_smem(const AttnFwdArgs& a) { return sizeof(float) * (size_t)(table_floats(a.c) + ring_floats(a.c.dtype, 2, kU)); }
inline size_t col_smem(const AttnBwdColArgs& a) { return sizeof(float) * (size_t)(table_floats(a.c) + ring_floats(a.c.dtype, 2, kU)); }
inline size_t row_smem(const AttnBwdRowArgs& a) {
    return sizeof(float) * (size_t)(table_floats(a.c) + grad_floats(a) + ring_floats(a.c.dtype, 1, row_group(a.c.score == SCORE_GATED, epw_code(a.c))));
}

// ---- device side ----------------------------------------------------------------------------------------------------------
constexpr uint32_t kIdxMask = 0x1fffffffu;         // packed edge word: bits 0..28 index, 29..30 edge type

using f2 = unsigned long long;                     // two packed fp32

__device__ __forceinline__ f2 pk(float lo, float hi) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ f2 pk1(float v) { return pk(v, v); }
__device__ __forceinline__ void upk(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// 8 features as loaded (4 registers of bf16, 8 of fp32) and as four packed fp32 pairs
template <typename T> struct Raw;
template <> struct Raw<__nv_bfloat16> {
    uint4 u;
    __device__ __forceinline__ void load(const void* p) {
        asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(p));
    }
    __device__ __forceinline__ void zero() { u = make_uint4(0u, 0u, 0u, 0u); }
    static __device__ __forceinline__ f2 two(uint32_t v) { return pk(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
    // asynchronous copy to the thread's own slot of a ring in shared memory (slot stride kThreads x 16 bytes); zeros if !ok
    static constexpr int kPieces = 1;
    static __device__ __forceinline__ void copy(uint32_t dst, const void* p) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
    }
    static __device__ __forceinline__ void copy(uint32_t dst, const void* p, bool ok) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p), "r"(ok ? 16 : 0) : "memory");
    }
    __device__ __forceinline__ void lds(uint32_t src) {
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(src) : "memory");
    }
    // the packed form is what stays in registers: without this the compiler keeps the converted copy of an earlier use alive
    __device__ __forceinline__ void opaque() { asm volatile("" : "+r"(u.x), "+r"(u.y), "+r"(u.z), "+r"(u.w)); }
    __device__ __forceinline__ void get(f2 (&f)[4]) const { f[0] = two(u.x); f[1] = two(u.y); f[2] = two(u.z); f[3] = two(u.w); }
};
template <> struct Raw<float> {
    f2 v[4];
    __device__ __forceinline__ void load(const void* p) {
        asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "l"(p));
        asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v[2]), "=l"(v[3]) : "l"(static_cast<const char*>(p) + 16));
    }
    __device__ __forceinline__ void zero() { v[0] = v[1] = v[2] = v[3] = 0ull; }
    static constexpr int kPieces = 2;
    static __device__ __forceinline__ void copy(uint32_t dst, const void* p) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + kThreads * 16), "l"(static_cast<const char*>(p) + 16) : "memory");
    }
    static __device__ __forceinline__ void copy(uint32_t dst, const void* p, bool ok) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p), "r"(ok ? 16 : 0) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + kThreads * 16), "l"(static_cast<const char*>(p) + 16), "r"(ok ? 16 : 0)
                     : "memory");
    }
    __device__ __forceinline__ void lds(uint32_t src) {
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(src) : "memory");
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[2]), "=l"(v[3]) : "r"(src + kThreads * 16) : "memory");
    }
    __device__ __forceinline__ void opaque() {}
    __device__ __forceinline__ void get(f2 (&f)[4]) const { f[0] = v[0]; f[1] = v[1]; f[2] = v[2]; f[3] = v[3]; }
};

__device__ __forceinline__ void store8(__nv_bfloat16* p, const f2 (&f)[4]) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) upk(f[i], x[2 * i], x[2 * i + 1]);
    Vec8<__nv_bfloat16>::store(p, x);
}
__device__ __forceinline__ void store8(float* p, const f2 (&f)[4]) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) upk(f[i], x[2 * i], x[2 * i + 1]);
    Vec8<float>::store(p, x);
}
__device__ __forceinline__ void add8(float* p, const f2 (&f)[4]) {
    float x[8], old[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) upk(f[i], x[2 * i], x[2 * i + 1]);
    Vec8<float>::load(p, old);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] += old[i];
    Vec8<float>::store(p, x);
}

// 8 fp32 of a lane in a shared-memory table of `lanes` x 8 values, kept as two planes of 4 per lane so that a warp's 16-byte accesses
// are free of bank conflicts (8 consecutive values per lane would double the cycles of every access)
__device__ __forceinline__ void lds8(const float* p, int lanes, f2 (&f)[4]) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + lanes * 4);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void sts8(float* p, int lanes, const f2 (&f)[4]) {
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(f[0], f[1]);
    *reinterpret_cast<ulonglong2*>(p + lanes * 4) = make_ulonglong2(f[2], f[3]);
}
// position of feature x of a row of 8 * lanes features in such a table
__device__ __forceinline__ int plane_at(int x, int lanes) { return ((x >> 2) & 1) * lanes * 4 + (x >> 3) * 4 + (x & 3); }

// sum over the 8 features in order (not as pairs: see the note on the order of sums above)
__device__ __forceinline__ float dot8(const f2 (&a)[4], const f2 (&b)[4]) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float x, y, u, v;
        upk(a[i], x, y);
        upk(b[i], u, v);
        s = fmaf(x, u, s);
        s = fmaf(y, v, s);
    }
    return s;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 shfl_xor2(f2 v, int o) { return __shfl_xor_sync(GT_FULL_MASK, v, o); }

// Transposing reduction over the LPH lanes of a head: pairs (0, 1) and (2, 3) of the four edges of a group are folded one after the
// other, so that edges are taken in order.  With LPH >= 4 lane ll ends with the sum of edge 2 (ll & 1) + (ll >> 1 & 1), with 2 lanes it
// has edges (ll & 1) and 2 + (ll & 1), with one lane all four: NV values per lane.  (Four lanes: first across distance 2, then 1.)
template <int LPH> struct Own { static constexpr int NV = LPH >= 4 ? 1 : (LPH == 2 ? 2 : 4); };
template <int LPH>
__device__ __forceinline__ int own_edge(int ll, int i) {
    return LPH >= 4 ? 2 * (ll & 1) + ((ll >> 1) & 1) : (LPH == 2 ? 2 * i + (ll & 1) : i);
}
// fold of a pair across `dist` lanes: lanes with that bit set keep the second value
__device__ __forceinline__ float fold(float x, float y, int ll, int dist) {
    const bool b = ll & dist;
    return (b ? y : x) + __shfl_xor_sync(GT_FULL_MASK, b ? x : y, dist);
}
template <int LPH>
__device__ __forceinline__ float fold_pair(float x, float y, int ll) { return fold(x, y, ll, LPH >= 4 ? 2 : 1); }
template <int LPH>
__device__ __forceinline__ float fold_last(float x, float y, int ll) {
    float v = fold(x, y, ll, 1);
#pragma unroll
    for (int o = 4; o < LPH; o <<= 1) v += __shfl_xor_sync(GT_FULL_MASK, v, o);       // lanes 4.. of a head repeat lanes 0..3
    return v;
}
// value of edge u from the lane of the head that keeps it
template <int LPH>
__device__ __forceinline__ float from_owner(const float (&o)[Own<LPH>::NV], int u) {
    if constexpr (LPH == 1) return o[u];
    else if constexpr (LPH == 2) return __shfl_sync(GT_FULL_MASK, o[u >> 1], u & 1, 2);
    else return __shfl_sync(GT_FULL_MASK, o[0], (u >> 1) | ((u & 1) << 1), 4);
}
template <int LPH>
__device__ __forceinline__ float owners_max(float v) {
    if constexpr (LPH >= 4) v = fmaxf(v, __shfl_xor_sync(GT_FULL_MASK, v, 2));
    if constexpr (LPH >= 2) v = fmaxf(v, __shfl_xor_sync(GT_FULL_MASK, v, 1));
    return v;
}

// base + index * row bytes as one widening multiply-add
__device__ __forceinline__ const char* row_ptr(const char* base, uint32_t j, uint32_t ld_bytes) { return base + (unsigned long long)j * ld_bytes; }

// Ring of two groups of N edges x ROWS gathered rows; every thread copies and reads only its own 8 features, so no barrier is needed.
template <typename T, int ROWS, int N>
struct Ring {
    static constexpr uint32_t kSlot = Raw<T>::kPieces * kThreads * 16, kStage = N * ROWS * kSlot;
    uint32_t base, at;               // this thread's first slot, offset of the stage of the group at the cursor
    __device__ __forceinline__ explicit Ring(const float* smem) : base((uint32_t)__cvta_generic_to_shared(smem) + threadIdx.x * 16), at(0u) {}
    __device__ __forceinline__ uint32_t slot(uint32_t stage, int u, int r) const { return base + stage + (u * ROWS + r) * kSlot; }
    __device__ __forceinline__ void flip() { at ^= kStage; }
    // rows b0 (and b1) + index * ld of the group at the cursor into the cursor's stage; slots behind the end of the segment get zeros
    template <typename K>
    __device__ __forceinline__ void issue(const K& k, const char* b0, uint32_t ld0, const char* b1, uint32_t ld1) const {
        if (k.whole()) {                                         // two loops: a test per copy would be predicated and issue both forms
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const uint32_t j = k.at(u) & kIdxMask;
                Raw<T>::copy(slot(at, u, 0), row_ptr(b0, j, ld0));
                if (ROWS == 2) Raw<T>::copy(slot(at, u, 1), row_ptr(b1, j, ld1));
            }
        } else {
#pragma unroll 1
            for (int u = 0; u < N; ++u) {
                const uint32_t j = k.at(u) & kIdxMask;
                Raw<T>::copy(slot(at, u, 0), row_ptr(b0, j, ld0), k.has(u));
                if (ROWS == 2) Raw<T>::copy(slot(at, u, 1), row_ptr(b1, j, ld1), k.has(u));
            }
        }
    }
    static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    static __device__ __forceinline__ void wait_previous() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
};

// Lane layout of a launch.  EPW: edges side by side in a warp (1 or 2 as a compile-time constant, 0 = any power of two up to 8).
template <int LPH, int EPW>
struct Lay {
    int lpr, ll, sub, epw, hg, head, foff, W, HL;
    __device__ __forceinline__ explicit Lay(const AttnCommon& c) {
        const int lane = threadIdx.x & 31;
        lpr = EPW ? 32 / EPW : min((c.H * c.D) >> 3, 32);
        epw = EPW ? EPW : 32 / lpr;
        ll = lane & (lpr - 1);
        sub = EPW == 1 ? 0 : lane / lpr;
        hg = blockIdx.y;
        W = lpr * 8;                               // features and heads handled by this block column
        HL = lpr / LPH;
        head = hg * HL + ll / LPH;
        foff = hg * W + ll * 8;
    }
};

// gate slice [T][W] (in planes) and bias slice [T][HL] of this block column
template <int LPH, int EPW>
__device__ __forceinline__ void load_tables(const AttnCommon& c, const Lay<LPH, EPW>& L, float* s_gate, float* s_bias, bool gated) {
    const int HD = c.H * c.D;
    if (gated)
        for (int i = threadIdx.x; i < c.T * L.W; i += kThreads)
            s_gate[(i / L.W) * L.W + plane_at(i % L.W, L.lpr)] = c.gate[(i / L.W) * HD + L.hg * L.W + i % L.W];
    else if (c.score == SCORE_BIASED)
        for (int i = threadIdx.x; i < c.T * L.HL; i += kThreads) s_bias[i] = c.bias[(i / L.HL) * c.H + L.hg * L.HL + i % L.HL];
    __syncthreads();
}

// Position of a warp in its list of segments: s, s + n_warps, s + 2 n_warps, ...  The edges of a segment are taken in chunks of 32 (one
// packed word per lane) and walked in groups of N per lane group; lane group `sub` takes the edges sub, sub + epw, ...  advance() only
// moves the position, so that a kernel starts the copies of the next group, also across the end of a segment, before it computes on
// the current one.  Descriptors are fetched two segments ahead and the first words one segment ahead.  All branches are uniform over
// the warp.  (Groups that never cross a change of the edge type cost 17 % padding and 40 instructions of bookkeeping per group; a
// segment per lane group instead of a segment per warp is 3 % faster at 4 heads x 32 but changes the order of the sums.)
enum Step : int { kDone = 0, kGroup = 1, kSegment = 2 };
// edge types of a group: bit u * epw of `starts` = the type changes at edge u of this lane group (never at its first edge)
template <int EPW>
struct Types {
    uint32_t starts, t0, t1;
    int epw;
    bool none;                       // no change in the group, for any lane group of the warp
    __device__ __forceinline__ int bit(int u) const { return u * (EPW ? EPW : epw); }
    __device__ __forceinline__ bool starts_at(int u) const { return (starts >> bit(u)) & 1u; }
    __device__ __forceinline__ int type(int u) const { return (int)((t0 >> bit(u)) & 1u) | (int)(((t1 >> bit(u)) & 1u) << 1); }
};
template <int LPH, bool GATED, int EPW, int N>
struct Cursor {
    const AttnCommon& c;
    const Lay<LPH, EPW>& L;
    const bool typed;
    const int n_warps;
    int s;                           // segment
    int row, beg, n, slot;           // its descriptor
    int done_row, done_slot;         // the segment that the last advance() finished
    int row1, beg1, n1, row2, beg2, n2;   // the next two
    uint32_t w, wnext, w1;           // words of this chunk, of the next chunk, of the next segment's first chunk
    int c0, p;                       // first edge of the chunk, position of the group in it
    uint32_t starts, t0, t1;         // types of the chunk (gated scores)

    __device__ __forceinline__ Cursor(const AttnCommon& c_, const Lay<LPH, EPW>& L_, bool typed_)
        : c(c_), L(L_), typed(typed_), n_warps((int)gridDim.x * kWarps) {
        // the shuffles here and in open() tell the compiler that the loop bounds are uniform over the warp
        s = __shfl_sync(GT_FULL_MASK, (int)blockIdx.x * kWarps + (int)(threadIdx.x >> 5), 0);
        fetch(s, row, beg, n);
        fetch(s + n_warps, row1, beg1, n1);
        fetch(s + 2 * n_warps, row2, beg2, n2);
        slot = s < c.plan.n_seg ? c.plan.seg_slot[s] : -1;
        w = word(beg, n, threadIdx.x & 31);
        w1 = word(beg1, n1, threadIdx.x & 31);
        open();
    }
    __device__ __forceinline__ int epw() const { return EPW ? EPW : L.epw; }
    __device__ __forceinline__ void fetch(int at, int& r, int& b, int& k) const {
        r = 0; b = 0; k = 0;
        if (at < c.plan.n_seg) { r = c.plan.seg_row[at]; b = c.plan.seg_beg[at]; k = c.plan.seg_end[at] - b; }
    }
    __device__ __forceinline__ uint32_t word(int b, int k, int e) const {          // 0 beyond the segment
        if (e >= k) return 0u;
        uint32_t x = (uint32_t)c.idx[b + e];
        if (typed) x |= (uint32_t)c.etype[b + e] << 29;
        return x;
    }
    __device__ __forceinline__ bool any() const { return s < c.plan.n_seg; }
    __device__ __forceinline__ bool mine() const { return L.sub < n; }             // this lane group has an edge in the segment
    __device__ __forceinline__ void open() {
        n = __shfl_sync(GT_FULL_MASK, n, 0);
        c0 = 0;
        chunk(0u);
    }
    __device__ __forceinline__ void chunk(uint32_t before) {     // before: words of the chunk before
        const int lane = threadIdx.x & 31;
        p = 0;
        if (c0 + 32 < n) wnext = word(beg, n, c0 + 32 + lane);
        if constexpr (GATED) {
            const int t = (int)(w >> 29);
            const int up = __shfl_sync(GT_FULL_MASK, t, lane - epw()), last = (int)(__shfl_sync(GT_FULL_MASK, before, lane - epw()) >> 29);
            const int prev = lane >= epw() ? up : (c0 > 0 ? last : t);
            starts = __ballot_sync(GT_FULL_MASK, c0 + lane < n && t != prev);
            t0 = __ballot_sync(GT_FULL_MASK, t & 1);
            t1 = __ballot_sync(GT_FULL_MASK, t & 2);
        }
    }
    __device__ __forceinline__ Types<EPW> types() const {
        const uint32_t here = (starts >> p) & (0xffffffffu >> (32 - N * epw()));
        return Types<EPW>{starts >> (p + L.sub), t0 >> (p + L.sub), t1 >> (p + L.sub), L.epw, here == 0u};
    }
    __device__ __forceinline__ int left() const { return n - c0 - p - L.sub; }     // edges from this lane group's first one to the end
    __device__ __forceinline__ bool has(int u) const { return u * epw() < left(); }
    __device__ __forceinline__ bool whole() const { return n - c0 - p >= N * epw(); }
    __device__ __forceinline__ uint32_t at(int u) const { return __shfl_sync(GT_FULL_MASK, w, p + L.sub + u * epw()); }
    __device__ __forceinline__ int edge(int u) const { return beg + c0 + p + L.sub + u * epw(); }
    __device__ __forceinline__ Step advance() {
        p += N * epw();
        if (p < 32 && c0 + p < n) return kGroup;
        c0 += 32;
        if (c0 < n) {
            const uint32_t before = w;
            w = wnext;
            chunk(before);
            return kGroup;
        }
        done_row = row; done_slot = slot;
        s += n_warps;
        if (s >= c.plan.n_seg) return kDone;
        row = row1; beg = beg1; n = n1; w = w1;
        row1 = row2; beg1 = beg2; n1 = n2;
        w1 = word(beg1, n1, threadIdx.x & 31);
        fetch(s + 2 * n_warps, row2, beg2, n2);
        slot = c.plan.seg_slot[s];
        open();
        return kSegment;
    }
};

// ------------------------------------------------------------------------------------------------------------------ forward
template <typename T, int LPH, bool GATED, bool SOFTMAX, int EPW>
__global__ void __launch_bounds__(kThreads, 6) fwd_kernel(AttnFwdArgs a) {
    extern __shared__ float smem[];
    const AttnCommon& c = a.c;
    const Lay<LPH, EPW> L(c);
    constexpr int NV = Own<LPH>::NV;
    const int H = c.H, HD = H * c.D;
    const bool biased = !GATED && c.score == SCORE_BIASED;
    const bool typed = (GATED || biased) && c.etype != nullptr;
    float* s_gate = smem;
    float* s_bias = smem;
    load_tables(c, L, s_gate, s_bias, GATED);
    const uint32_t ldk = (uint32_t)((c.ldk ? c.ldk : HD) * sizeof(T));
    const size_t ldq = (c.ldq ? c.ldq : HD);
    const char* kb = reinterpret_cast<const char*>(static_cast<const T*>(a.k) + L.foff);
    const char* vb = reinterpret_cast<const char*>(static_cast<const T*>(a.v) + L.foff);
    const T* qb = static_cast<const T*>(a.q) + L.foff;
    Cursor<LPH, GATED, EPW, kU> k(c, L, typed);
    if (!k.any()) return;
    Ring<T, 2, kU> ring(smem + table_floats(c));
    Raw<T> qr, qn;
    int tb[NV];                                                        // edge types of the lane's own edges (biased scores)
    qr.load(qb + (size_t)k.row * ldq);
    ring.issue(k, kb, ldk, vb, ldk);
    ring.commit();
    f2 qg[4], acc[4];                                                  // q * scale (* gate of the current run), sum of p v
    float l = 0.f, m = -INFINITY;
    auto regate = [&](int type) {
        qr.opaque();
        qr.get(qg);
#pragma unroll
        for (int i = 0; i < 4; ++i) qg[i] = mul2(qg[i], pk1(c.scale));
        if constexpr (GATED) {
            f2 gt[4];
            lds8(s_gate + type * L.W + L.ll * 4, L.lpr, gt);
#pragma unroll
            for (int i = 0; i < 4; ++i) qg[i] = mul2(qg[i], gt[i]);
        }
    };
    auto clear = [&]() {
        l = 0.f;
        m = -INFINITY;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = 0ull;
        regate(GATED ? k.types().type(0) : 0);
    };
    clear();
    for (;;) {
        // the group in flight becomes the current one; the next group's copies start before it is waited for
        const int left = k.left();
        const Types<EPW> ty = k.types();
        const uint32_t stage = ring.at;
        if (biased)
#pragma unroll
            for (int i = 0; i < NV; ++i) tb[i] = typed ? (int)(k.at(own_edge<LPH>(L.ll, i)) >> 29) : 0;
        const Step step = k.advance();
        ring.flip();
        if (step != kDone) ring.issue(k, kb, ldk, vb, ldk);
        ring.commit();
        if (step == kSegment) qn.load(qb + (size_t)k.row * ldq);
        ring.wait_previous();
        auto dot = [&](int u, auto tests) {
            if constexpr (GATED && tests.value) {
                if (ty.starts_at(u)) regate(ty.type(u));
            }
            Raw<T> x;
            f2 kf[4];
            x.lds(ring.slot(stage, u, 0));
            x.get(kf);
            return dot8(qg, kf);
        };
        float part[kU], sc[NV];
        if (!GATED || ty.none) {
#pragma unroll
            for (int u = 0; u < kU; ++u) part[u] = dot(u, std::false_type{});
        } else {
#pragma unroll
            for (int u = 0; u < kU; ++u) part[u] = dot(u, std::true_type{});
        }
        if constexpr (LPH == 1) {
#pragma unroll
            for (int u = 0; u < kU; ++u) sc[u] = part[u];
        } else {
            const float f0 = fold_pair<LPH>(part[0], part[1], L.ll), f1 = fold_pair<LPH>(part[2], part[3], L.ll);
            if constexpr (LPH == 2) { sc[0] = f0; sc[1] = f1; }
            else sc[0] = fold_last<LPH>(f0, f1, L.ll);
        }
        float mg = -INFINITY;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (biased) sc[i] += s_bias[tb[i] * L.HL + L.ll / LPH];
            const bool ok = own_edge<LPH>(L.ll, i) * k.epw() < left;
            if constexpr (SOFTMAX) {
                if (!ok) sc[i] = -INFINITY;
                mg = fmaxf(mg, sc[i]);
            } else {
                sc[i] = ok ? __expf(fminf(fmaxf(sc[i], c.lo), c.hi)) : 0.f;
            }
        }
        if constexpr (SOFTMAX) {
            const float mn = fmaxf(m, owners_max<LPH>(mg));
            const float ref = mn == -INFINITY ? 0.f : mn;
            const float corr = __expf(m - ref);
            m = mn;
            l *= corr;
            const f2 c2 = pk1(corr);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = mul2(acc[i], c2);
#pragma unroll
            for (int i = 0; i < NV; ++i) sc[i] = __expf(sc[i] - ref);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const float pu = from_owner<LPH>(sc, u);
            const f2 p2 = pk1(pu);
            l += pu;
            Raw<T> x;
            f2 vf[4];
            x.lds(ring.slot(stage, u, 1));
            x.get(vf);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] = fma2(p2, vf[i], acc[i]);
        }
        if (step == kGroup) continue;
        // the segment is through: merge the lane groups
        if constexpr (EPW != 1)
            for (int o = L.lpr; o < 32; o <<= 1) {
                float wa = 1.f, wb = 1.f;
                if constexpr (SOFTMAX) {
                    const float mo = __shfl_xor_sync(GT_FULL_MASK, m, o), mn = fmaxf(m, mo), ref = mn == -INFINITY ? 0.f : mn;
                    wa = __expf(m - ref);
                    wb = __expf(mo - ref);
                    m = mn;
                }
                l = l * wa + __shfl_xor_sync(GT_FULL_MASK, l, o) * wb;
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] = fma2(shfl_xor2(acc[i], o), pk1(wb), mul2(acc[i], pk1(wa)));
            }
        {
            const bool first = (L.ll & (LPH - 1)) == 0, writer = L.sub == 0;
            if (writer && k.done_slot >= 0) {
                float* sp = c.scratch + (size_t)k.done_slot * ((HD + 2 * H + 3) & ~3);
                store8(sp + L.foff, acc);
                if (first) { sp[HD + L.head] = l; sp[HD + H + L.head] = m; }
            }
            const bool whole = writer && k.done_slot < 0;                         // the segment is a whole row
            if (a.push_n > 0) {
                // reduce-scatter fused into the store: the finished row goes as bf16 into the slot that its owner keeps for this rank
                const long long orow = a.row_map ? a.row_map[k.done_row] : k.done_row;
                const int owner = (int)(orow / a.push_rows);
                __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.push_slot[owner]) + (orow - (long long)owner * a.push_rows) * a.push_ld;
                if (whole) store8(dst + L.foff, acc);
                if (L.HL % 8 == 0 || gridDim.y == 1) {                     // l of eight heads per 16-byte store; padding heads are zero
                    for (int h0 = 0; h0 < L.HL; h0 += 8) {
                        float lv[8];
    #pragma unroll
                        for (int x = 0; x < 8; ++x) {
                            const float t = __shfl_sync(GT_FULL_MASK, l, min((h0 + x) * LPH, L.lpr - 1));
                            lv[x] = h0 + x < L.HL ? t : 0.f;
                        }
                        if (whole && L.ll == 0) Vec8<__nv_bfloat16>::store(dst + a.push_l_off + L.hg * L.HL + h0, lv);
                    }
                } else if (whole && first) {
                    dst[a.push_l_off + L.head] = __float2bfloat16(l);
                }
            } else if (whole && a.o != nullptr) {                          // normalised output in the operand type
                const float inv = SOFTMAX ? 1.f / (l > 0.f ? l : 1.f) : 1.f / (l + a.eps);
    #pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] = mul2(acc[i], pk1(inv));
                store8(static_cast<T*>(a.o) + (size_t)k.done_row * HD + L.foff, acc);
                if (first) {
                    a.l[(size_t)k.done_row * H + L.head] = l;
                    if (a.m) a.m[(size_t)k.done_row * H + L.head] = m == -INFINITY ? 0.f : m;
                }
            } else if (whole) {
                const long long orow = a.row_map ? a.row_map[k.done_row] : k.done_row;
                float* dst = a.acc + orow * a.acc_stride + L.foff;
                if (a.accumulate) add8(dst, acc); else store8(dst, acc);
                if (first) {
                    float* lp = a.l + orow * a.l_stride + L.head;
                    *lp = a.accumulate ? *lp + l : l;
                    if (a.m) a.m[orow * H + L.head] = m == -INFINITY ? 0.f : m;
                }
            }
        }
        if (step == kDone) break;
        qr = qn;
        clear();
    }
}

// -------------------------------------------------------------------------------------------------------------- column pass
// dk_j = sum g_t (scale ds_ij q_i),  dv_j = sum P_ij dO_i, and the score gradient of every entry in CSR
// order for the row pass.
template <typename T, int LPH, bool GATED, bool SOFTMAX, int EPW>
__global__ void __launch_bounds__(kThreads, LPH == 1 ? 3 : 4) col_kernel(AttnBwdColArgs a) {
    extern __shared__ float smem[];
    const AttnCommon& c = a.c;
    const Lay<LPH, EPW> L(c);
    constexpr int NV = Own<LPH>::NV;
    const int H = c.H, HD = H * c.D;
    const bool biased = !GATED && c.score == SCORE_BIASED;
    const bool typed = (GATED || biased) && c.etype != nullptr;
    float* s_gate = smem;
    float* s_bias = smem;
    load_tables(c, L, s_gate, s_bias, GATED);
    const uint32_t ldq = (uint32_t)((c.ldq ? c.ldq : HD) * sizeof(T)), ldr = (uint32_t)((c.ldr ? c.ldr : HD) * sizeof(T));
    const size_t ldk = c.ldk ? c.ldk : HD, ldo = c.ldo ? c.ldo : HD;
    const char* qb = reinterpret_cast<const char*>(static_cast<const T*>(a.q) + L.foff);
    const char* rb = reinterpret_cast<const char*>(static_cast<const T*>(a.row_vec) + L.foff);
    const char* stb = reinterpret_cast<const char*>(a.stat + L.head);
    const uint32_t lds = (uint32_t)H * 16u;
    const T* kb = static_cast<const T*>(a.k) + L.foff;
    const T* vb = static_cast<const T*>(a.v) + L.foff;
    Cursor<LPH, GATED, EPW, kU> k(c, L, typed);
    if (!k.any()) return;
    Ring<T, 2, kU> ring(smem + table_floats(c));
    Raw<T> kr, vr, kn, vn;
    float4 stn[NV];                                 // row statistics, CSR position and edge type of the lane's own entries of the group in flight
    int posn[NV], tbn[NV];
    auto issue = [&]() {                            // q and row-vector rows of the group at the cursor, statistics of the own entries
        ring.issue(k, qb, ldq, rb, ldr);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int e = own_edge<LPH>(L.ll, i);
            const uint32_t wo = k.at(e);
            stn[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            posn[i] = 0;
            if (biased) tbn[i] = (int)(wo >> 29);
            if (k.has(e)) {
                stn[i] = __ldg(reinterpret_cast<const float4*>(row_ptr(stb, wo & kIdxMask, lds)));
                if (a.ds_out != nullptr) posn[i] = __ldg(a.pos + k.edge(e));
            }
        }
    };
    f2 kf[4], gc[4], dk[4], dv[4];                  // k (* gate of the current run), gate of the run that dk is at
    auto open = [&]() {                             // k / v row of the segment at the cursor
        kn.load(kb + (size_t)k.row * ldk);
        vn.load(vb + (size_t)k.row * ldk);
    };
    auto regate = [&](int type) {                   // kf = k (* gate[type])
        kr.opaque();
        kr.get(kf);
        if constexpr (GATED) {
            f2 gt[4];
            lds8(s_gate + type * L.W + L.ll * 4, L.lpr, gt);
#pragma unroll
            for (int i = 0; i < 4; ++i) kf[i] = mul2(kf[i], gt[i]);
        }
    };
    auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i) { dk[i] = dv[i] = 0ull; }
        kr = kn;
        vr = vn;
        const int type = GATED ? k.types().type(0) : 0;
        regate(type);
        if constexpr (GATED) lds8(s_gate + type * L.W + L.ll * 4, L.lpr, gc);
    };
    open();
    issue();
    ring.commit();
    clear();
    for (;;) {
        // the group in flight becomes the current one; the next group's copies start before it is waited for
        const int left = k.left();
        const Types<EPW> ty = k.types();
        const uint32_t stage = ring.at;
        float4 st[NV];
        int pos[NV], tb[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) { st[i] = stn[i]; pos[i] = posn[i]; tb[i] = tbn[i]; }
        const Step step = k.advance();
        ring.flip();
        if (step == kSegment) open();
        if (step != kDone) issue();
        ring.commit();
        ring.wait_previous();
        const bool plain = !GATED || ty.none;
        float sc[NV], dp[NV], P[NV], ds[NV];
        {
            f2 vf[4];
            vr.opaque();
            vr.get(vf);
            auto dots = [&](int u, float& x, float& y) {
                Raw<T> r;
                f2 f[4];
                r.lds(ring.slot(stage, u, 0));
                r.get(f);
                x = dot8(f, kf);
                r.lds(ring.slot(stage, u, 1));
                r.get(f);
                y = dot8(f, vf);
            };
            if constexpr (LPH == 1) {
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    if (GATED && ty.starts_at(u)) regate(ty.type(u));
                    dots(u, sc[u], dp[u]);
                }
            } else {
                float s0 = 0.f, d0 = 0.f, s1 = 0.f, d1 = 0.f;
#pragma unroll 1                                    // two entries at a time: all four in flight cost 40 registers more
                for (int u = 0; u < kU; u += 2) {
                    float x, dx, y, dy;
                    if (!GATED || plain) {
                        dots(u, x, dx);
                        dots(u + 1, y, dy);
                    } else {
                        if (ty.starts_at(u)) regate(ty.type(u));
                        dots(u, x, dx);
                        if (ty.starts_at(u + 1)) regate(ty.type(u + 1));
                        dots(u + 1, y, dy);
                    }
                    s0 = s1;
                    d0 = d1;
                    s1 = fold_pair<LPH>(x, y, L.ll);
                    d1 = fold_pair<LPH>(dx, dy, L.ll);
                }
                if constexpr (LPH == 2) {
                    sc[0] = s0; sc[1] = s1;
                    dp[0] = d0; dp[1] = d1;
                } else {
                    sc[0] = fold_last<LPH>(s0, s1, L.ll);
                    dp[0] = fold_last<LPH>(d0, d1, L.ll);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const bool ok = own_edge<LPH>(L.ll, i) * k.epw() < left;
            float x = sc[i] * c.scale;
            if (biased) x += s_bias[tb[i] * L.HL + L.ll / LPH];
            float pr, mask = 1.f;
            if constexpr (SOFTMAX) {
                pr = __expf(x - st[i].x);
            } else {
                pr = __expf(fminf(fmaxf(x, c.lo), c.hi));
                mask = (x >= c.lo && x <= c.hi) ? 1.f : 0.f;
            }
            P[i] = ok ? pr * st[i].z : 0.f;
            ds[i] = ok ? P[i] * (dp[i] + st[i].y) * mask : 0.f;
            if (a.ds_out != nullptr && ok && (LPH <= 4 || (L.ll & (LPH - 1)) < 4)) a.ds_out[(size_t)pos[i] * H + L.head] = ds[i];
        }
        auto add = [&](int u) {
            const f2 P2 = pk1(from_owner<LPH>(P, u)), d2 = pk1(from_owner<LPH>(ds, u) * c.scale);
            Raw<T> y;
            f2 x[4];
            y.lds(ring.slot(stage, u, 0));
            y.get(x);
#pragma unroll
            for (int i = 0; i < 4; ++i) dk[i] = GATED ? fma2(mul2(d2, x[i]), gc[i], dk[i]) : fma2(d2, x[i], dk[i]);
            y.lds(ring.slot(stage, u, 1));
            y.get(x);
#pragma unroll
            for (int i = 0; i < 4; ++i) dv[i] = fma2(P2, x[i], dv[i]);
        };
        if (plain) {
#pragma unroll
            for (int u = 0; u < kU; ++u) add(u);
        } else {
#pragma unroll (NV == 1 ? 1 : 4)
            for (int u = 0; u < kU; ++u) {
                if (ty.starts_at(u)) lds8(s_gate + ty.type(u) * L.W + L.ll * 4, L.lpr, gc);
                add(u);
            }
        }
        if (step == kGroup) continue;
        // the segment is through: merge the lane groups
        if constexpr (EPW != 1)
            for (int o = L.lpr; o < 32; o <<= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i) { dk[i] = add2(dk[i], shfl_xor2(dk[i], o)); dv[i] = add2(dv[i], shfl_xor2(dv[i], o)); }
        if (L.sub == 0) {
            if (k.done_slot >= 0) {
                float* sp = c.scratch + (size_t)k.done_slot * 2 * HD + L.foff;
                store8(sp, dk);
                store8(sp + HD, dv);
            } else {
                store8(static_cast<T*>(a.dk) + (size_t)k.done_row * ldo + L.foff, dk);
                store8(static_cast<T*>(a.dv) + (size_t)k.done_row * ldo + L.foff, dv);
            }
        }
        if (step == kDone) break;
        clear();
    }
}

// ----------------------------------------------------------------------------------------- row pass from stored score gradients
// dq_i = scale * sum_t g_t * A_t with A_t = sum_{edges of type t} ds_ij k_j: one gathered K row and H floats per edge.  The gate
// gradient (q * scale * A_t) is added per run of one type into a shared-memory table of the warp.
template <typename T, int LPH, bool GATED, int EPW>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 2 ? 6 : 4) row_kernel(AttnBwdRowArgs a) {
    extern __shared__ float smem[];
    const AttnCommon& c = a.c;
    const Lay<LPH, EPW> L(c);
    constexpr int NV = Own<LPH>::NV;
    constexpr int U = row_group(GATED, EPW);
    const int H = c.H, HD = H * c.D, lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
    const bool want_dg = GATED && a.dgate_part != nullptr;
    const bool want_db = !GATED && c.score == SCORE_BIASED && a.dbias_part != nullptr;
    const bool typed = (GATED || want_db) && c.etype != nullptr;
    float* s_gate = smem;                                              // [T][W]
    float* s_dg = smem + table_floats(c);                              // [warp][T][256] in planes (gated) or [thread][T] (biased)
    if (GATED) load_tables(c, L, s_gate, s_gate, true);
    float* my_dg = s_dg + (size_t)wrp * c.T * 256 + lane * 4;
    if (want_dg)
        for (int t = 0; t < c.T; ++t)
#pragma unroll
            for (int x = 0; x < 4; ++x) my_dg[t * 256 + x] = my_dg[t * 256 + 128 + x] = 0.f;
    float db[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t ldk = (uint32_t)((c.ldk ? c.ldk : HD) * sizeof(T));
    const size_t ldq = c.ldq ? c.ldq : HD, ldo = c.ldo ? c.ldo : HD;
    const char* kb = reinterpret_cast<const char*>(static_cast<const T*>(a.k) + L.foff);
    const T* qb = static_cast<const T*>(a.q) + L.foff;
    const float* dsb = a.ds_in + L.head;
    Cursor<LPH, GATED, EPW, U> k(c, L, typed);
    if (k.any()) {
        Ring<T, 1, U> ring(s_dg + grad_floats(a));
        Raw<T> qr, qn;
        float dsn[U / 4][NV];                       // score gradients of the lane's own edges of the group in flight
        auto issue = [&]() {                        // K rows of the group at the cursor, score gradients of the own edges
            ring.issue(k, kb, ldk, nullptr, 0u);
#pragma unroll
            for (int b = 0; b < U / 4; ++b)
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    const int e = 4 * b + own_edge<LPH>(L.ll, i);
                    dsn[b][i] = k.has(e) ? __ldg(dsb + (size_t)k.edge(e) * H) : 0.f;
                }
        };
        auto load_q = [&](Raw<T>& r) {
            r.zero();
            if (want_dg) r.load(qb + (a.row_map ? (long long)a.row_map[k.row] : (long long)k.row) * ldq);
        };
        f2 A[4], dq[4];                             // sum of ds k over the current run, dq of the finished runs
        auto flush = [&](int t) {                   // end of a run of type t: dq += g_t * A, gate gradient += q * scale * A
            f2 gt[4];
            lds8(s_gate + t * L.W + L.ll * 4, L.lpr, gt);
            if (want_dg) {
                f2 q0[4], sum[4];
                qr.get(q0);
                lds8(my_dg + t * 256, 32, sum);
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[i] = fma2(mul2(q0[i], pk1(c.scale)), A[i], sum[i]);
                sts8(my_dg + t * 256, 32, sum);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) { dq[i] = fma2(gt[i], A[i], dq[i]); A[i] = 0ull; }
        };
        load_q(qr);
        issue();
        ring.commit();
        int ta = 0;                                 // type of the run that A belongs to
        auto clear = [&]() {
#pragma unroll
            for (int i = 0; i < 4; ++i) A[i] = dq[i] = 0ull;
            if constexpr (GATED) {
                ta = k.mine() ? k.types().type(0) : -1;
            }
        };
        clear();
        for (;;) {
            // the group in flight becomes the current one; the next group's copies start before it is waited for
            const Types<EPW> ty = k.types();
            const uint32_t stage = ring.at;
            float ds[U / 4][NV];
#pragma unroll
            for (int b = 0; b < U / 4; ++b)
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    ds[b][i] = dsn[b][i];
                    if (want_db) {
                        const int t = typed ? (int)(k.at(4 * b + own_edge<LPH>(L.ll, i)) >> 29) : 0;
#pragma unroll
                        for (int tt = 0; tt < 4; ++tt)
                            if (t == tt) db[tt] += ds[b][i];
                    }
                }
            const Step step = k.advance();
            ring.flip();
            if (step != kDone) issue();
            ring.commit();
            if (step == kSegment) load_q(qn);
            ring.wait_previous();
            auto add = [&](int u) {
                const f2 d2 = pk1(from_owner<LPH>(ds[u / 4], u & 3));
                Raw<T> y;
                f2 kf[4];
                y.lds(ring.slot(stage, u, 0));
                y.get(kf);
#pragma unroll
                for (int i = 0; i < 4; ++i) A[i] = fma2(d2, kf[i], A[i]);
            };
            if (!GATED || ty.none) {
#pragma unroll
                for (int u = 0; u < U; ++u) add(u);
            } else {
#pragma unroll
                for (int b = 0; b < U / 4; ++b)
#pragma unroll (NV == 1 ? 1 : 4)
                    for (int u = 4 * b; u < 4 * b + 4; ++u) {
                        if (ty.starts_at(u)) {
                            flush(ta);
                            ta = ty.type(u);
                        }
                        add(u);
                    }
            }
            if (step == kGroup) continue;
            // the segment is through
            if constexpr (GATED) {
                if (ta >= 0) flush(ta);             // (a lane group without edges has no run)
#pragma unroll
                for (int i = 0; i < 4; ++i) A[i] = dq[i];
            }
            if constexpr (EPW != 1)                 // merge the lane groups
                for (int o = L.lpr; o < 32; o <<= 1)
#pragma unroll
                    for (int i = 0; i < 4; ++i) A[i] = add2(A[i], shfl_xor2(A[i], o));
            if (L.sub == 0) {
                const long long srow = a.row_map ? a.row_map[k.done_row] : k.done_row;
#pragma unroll
                for (int i = 0; i < 4; ++i) A[i] = mul2(A[i], pk1(c.scale));
                if (k.done_slot >= 0) store8(c.scratch + (size_t)k.done_slot * HD + L.foff, A);
                else if (a.accumulate_dq) add8(static_cast<float*>(a.dq) + srow * ldo + L.foff, A);
                else store8(static_cast<T*>(a.dq) + srow * ldo + L.foff, A);
            }
            if (step == kDone) break;
            qr = qn;
            clear();
        }
    }
    if (want_dg) {
        __syncthreads();
        float* part = a.dgate_part + (size_t)blockIdx.x * c.T * HD;
        for (int i = threadIdx.x; i < c.T * L.W; i += kThreads) {
            const int t = i / L.W, f = i - t * L.W;
            float v = 0.f;
            for (int x = 0; x < kWarps; ++x)
                for (int e = 0; e < L.epw; ++e) v += s_dg[((size_t)x * c.T + t) * 256 + plane_at(e * L.W + f, 32)];
            part[t * HD + L.hg * L.W + f] = v;
        }
    }
    if (want_db) {                                                     // lanes of a head that keep an edge each, folded in lane order
        for (int t = 0; t < c.T; ++t) s_dg[threadIdx.x * c.T + t] = (LPH <= 4 || (L.ll & (LPH - 1)) < 4) ? db[t & 3] : 0.f;
        __syncthreads();
        float* part = a.dbias_part + (size_t)blockIdx.x * c.T * H;
        for (int i = threadIdx.x; i < c.T * L.HL; i += kThreads) {
            const int t = i / L.HL, h = i - t * L.HL;
            float v = 0.f;
            for (int x = 0; x < kThreads / L.lpr; ++x)
                for (int k = 0; k < LPH; ++k) v += s_dg[(x * L.lpr + h * LPH + k) * c.T + t];
            part[t * H + L.hg * L.HL + h] = v;
        }
    }
}

}  // namespace edge
}  // namespace gt
