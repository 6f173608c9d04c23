// Launch of the edge-gather row pass of the backward (csrc/attn_edge.cuh): one instance per operand type, lanes per head, score kind.
#include "attn_edge.cuh"

namespace gt {
namespace edge {

namespace {
template <typename T, int LPH, bool GATED, int EPW>
void launch(const AttnBwdRowArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    auto* k = row_kernel<T, LPH, GATED, EPW>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<grid, kThreads, smem, s>>>(a);
}

template <typename T, int LPH, bool GATED>
void pick_width(const AttnBwdRowArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    if constexpr (LPH == 4) {
        if (epw_code(a.c) == 1) return launch<T, LPH, GATED, 1>(a, grid, smem, s);
        if (epw_code(a.c) == 2) return launch<T, LPH, GATED, 2>(a, grid, smem, s);
    }
    launch<T, LPH, GATED, 0>(a, grid, smem, s);
}
template <typename T, int LPH>
void pick_score(const AttnBwdRowArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
    const bool gated = a.c.score == SCORE_GATED;
    if (gated) pick_width<T, LPH, true>(a, grid, smem, s);
    else pick_width<T, LPH, false>(a, grid, smem, s);
}
template <typename T>
void pick_head(const AttnBwdRowArgs& a, dim3 grid, size_t smem, cudaStream_t s) {
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

void row(const AttnBwdRowArgs& a, cudaStream_t s) {
    const dim3 grid(a.n_blocks, half_count(a.c));            // dgate_part / dbias_part have one slice per block of grid.x
    const size_t smem = row_smem(a);
    if (a.c.dtype == DT_BF16) pick_head<__nv_bfloat16>(a, grid, smem, s);
    else pick_head<float>(a, grid, smem, s);
}
const void* row_8x32_bf16() { return reinterpret_cast<const void*>(&row_kernel<__nv_bfloat16, 4, true, 1>); }

}  // namespace edge
}  // namespace gt
