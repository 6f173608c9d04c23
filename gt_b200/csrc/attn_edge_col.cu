// Launch of the edge-gather column pass of the backward (csrc/attn_edge.cuh): one instance per operand type, lanes per head, score kind and norm.
#include "attn_edge.cuh"

namespace gt {
namespace edge {

namespace {
template <typename T, int LPH, bool GATED, bool SOFTMAX, int EPW>
void launch(const AttnBwdColArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    auto* k = col_kernel<T, LPH, GATED, SOFTMAX, EPW>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<grid, kThreads, smem, s>>>(a);
}

template <typename T, int LPH, bool GATED, bool SM>
void pick_width(const AttnBwdColArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    if constexpr (LPH == 4) {
        if (epw_code(a.c) == 1) return launch<T, LPH, GATED, SM, 1>(a, grid, smem, s);
        if (epw_code(a.c) == 2) return launch<T, LPH, GATED, SM, 2>(a, grid, smem, s);
    }
    launch<T, LPH, GATED, SM, 0>(a, grid, smem, s);
}
template <typename T, int LPH>
void pick_score(const AttnBwdColArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    const bool gated = a.c.score == SCORE_GATED;
    const bool sm = a.c.norm == NORM_SOFTMAX;
    if (gated && sm) pick_width<T, LPH, true, true>(a, grid, smem, s);
    else if (gated) pick_width<T, LPH, true, false>(a, grid, smem, s);
    else if (sm) pick_width<T, LPH, false, true>(a, grid, smem, s);
    else pick_width<T, LPH, false, false>(a, grid, smem, s);
}
template <typename T>
void pick_head(const AttnBwdColArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    switch (a.c.D >> 3) {
        case 1: pick_score<T, 1>(a, grid, smem, s); break;
        case 2: pick_score<T, 2>(a, grid, smem, s); break;
        case 4: pick_score<T, 4>(a, grid, smem, s); break;
        case 8: pick_score<T, 8>(a, grid, smem, s); break;
        case 16: pick_score<T, 16>(a, grid, smem, s); break;
        default: pick_score<T, 32>(a, grid, smem, s); break;
    }
}
}  // namespace

void col(const AttnBwdColArgs& a, cudaStream_t s) {
    const dim3 grid(grid_blocks(a.c, 148 * 24), half_count(a.c));
    const size_t smem = col_smem(a);
    pick_head<__nv_bfloat16>(a, grid, smem, s);
}
const void* col_8x32_bf16() { return reinterpret_cast<const void*>(&col_kernel<__nv_bfloat16, 4, true, false, 1>); }

}  // namespace edge
}  // namespace gt
