// Host dispatch of the tensor-core kernels of the frozen-M0 chunkwise rule (memory_tc.cuh).
#include "memory_tc.cuh"
#include "memory_tc.h"

namespace nlh {
namespace mtc {

static bool common_ok(int rule, int d, int tile, float clip, float mmax)
{
    return (rule == RULE_TITANS || rule == RULE_DELTA) && d == D && tile >= MIN_TILE && tile <= TMAX && !(clip > 0.0f) &&
           !m_norm_enabled(mmax);
}

template <int RULE>
static void launch_fwd(const FwdArgs& a, cudaStream_t st)
{
    cudaFuncSetAttribute(tile_fwd_kernel<RULE>, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
    tile_fwd_kernel<RULE><<<a.batch, NT, FWD_SMEM, st>>>(a, a.interval);
}
template <int RULE>
static void launch_bwd(const BwdArgs& a, cudaStream_t st)
{
    cudaFuncSetAttribute(tile_bwd_kernel<RULE>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM);
    tile_bwd_kernel<RULE><<<a.batch, NT, BWD_SMEM, st>>>(a, a.chunk);
}

bool forward(int rule, const FwdArgs& a, cudaStream_t st)
{
    if (!a.frozen || a.store_mode != STORE_CHUNK || a.seq_len <= 0 || !common_ok(rule, a.d, a.interval, a.error_clip, a.m_norm_max))
        return false;
    const bool al = aligned16(a.k) && aligned16(a.v) && aligned16(a.q) && aligned16(a.y) && aligned16(a.m_init) &&
                    aligned16(a.m_out) && (a.init_stride % 4 == 0) && (a.out_stride % 4 == 0) &&
                    (rule != RULE_TITANS || (a.s_init && a.s_out && aligned16(a.s_init) && aligned16(a.s_out)));
    if (!al) return false;
    if (rule == RULE_TITANS) launch_fwd<RULE_TITANS>(a, st);
    else launch_fwd<RULE_DELTA>(a, st);
    return true;
}

bool backward(int rule, const BwdArgs& a, cudaStream_t st)
{
    if (!a.frozen || a.t_end <= a.t_start || !common_ok(rule, a.d, a.chunk, a.error_clip, a.m_norm_max)) return false;
    const bool al = aligned16(a.k) && aligned16(a.v) && aligned16(a.q) && aligned16(a.d_y) && aligned16(a.d_k) &&
                    aligned16(a.d_v) && aligned16(a.d_q) && aligned16(a.m_traj) && (a.traj_stride % 4 == 0) &&
                    (rule != RULE_TITANS || a.s_traj) && aligned16(a.s_traj) && aligned16(a.d_m_seed) && aligned16(a.d_s_seed) &&
                    (a.atomic_out || (aligned16(a.d_m_out) && aligned16(a.d_s_out)));
    if (!al) return false;
    if (rule == RULE_TITANS) launch_bwd<RULE_TITANS>(a, st);
    else launch_bwd<RULE_DELTA>(a, st);
    return true;
}

int timeout_flag()
{
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_mtc_timeout, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

}  // namespace mtc
}  // namespace nlh
