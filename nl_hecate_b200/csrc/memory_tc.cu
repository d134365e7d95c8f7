// Host dispatch of the tensor-core memory-rule kernels (memory_tc.cuh).
#include "memory_tc.cuh"
#include "memory_tc.h"

namespace nlh {
namespace mtc {

static bool common_ok(int rule, int d, float clip, float mmax)
{
    return (rule == RULE_TITANS || rule == RULE_DELTA) && d == D && !(clip > 0.0f) && !m_norm_enabled(mmax);
}

template <int RULE, bool SOLVE>
static void launch_fwd(const FwdArgs& a, int T, cudaStream_t st)
{
    cudaFuncSetAttribute(tile_fwd_kernel<RULE, SOLVE>, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
    tile_fwd_kernel<RULE, SOLVE><<<a.batch, NT, FWD_SMEM, st>>>(a, T);
}
template <int RULE, bool SOLVE, bool SDER>
static void launch_bwd(const BwdArgs& a, int T, long long mstep, cudaStream_t st)
{
    cudaFuncSetAttribute(tile_bwd_kernel<RULE, SOLVE, SDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM);
    tile_bwd_kernel<RULE, SOLVE, SDER><<<a.batch, NT, BWD_SMEM, st>>>(a, T, mstep);
}

bool forward(int rule, const FwdArgs& a, cudaStream_t st)
{
    const int T = a.interval;
    if (!common_ok(rule, a.d, a.error_clip, a.m_norm_max) || T < MIN_TILE || T > TMAX || a.seq_len <= 0) return false;
    if (a.store_mode != STORE_CHUNK && a.store_mode != STORE_CKPT) return false;
    const bool al = aligned16(a.k) && aligned16(a.v) && aligned16(a.q) && aligned16(a.y) && aligned16(a.m_init) &&
                    aligned16(a.m_out) && (a.init_stride % 4 == 0) && (a.out_stride % 4 == 0) &&
                    (rule != RULE_TITANS || (a.s_init && a.s_out && aligned16(a.s_init) && aligned16(a.s_out)));
    if (!al) return false;
    const bool solve = !a.frozen;
    if (rule == RULE_TITANS) { if (solve) launch_fwd<RULE_TITANS, true>(a, T, st); else launch_fwd<RULE_TITANS, false>(a, T, st); }
    else { if (solve) launch_fwd<RULE_DELTA, true>(a, T, st); else launch_fwd<RULE_DELTA, false>(a, T, st); }
    return true;
}

bool backward(int rule, const BwdArgs& a, int T, long long mstep, cudaStream_t st)
{
    if (!common_ok(rule, a.d, a.error_clip, a.m_norm_max) || T < MIN_TILE || T > TMAX || a.t_end <= a.t_start) return false;
    const bool sder = rule == RULE_TITANS && a.s_traj == nullptr;
    if (sder && (mstep != (long long)T * DD || a.frozen)) return false;       // needs every M state
    const bool al = aligned16(a.k) && aligned16(a.v) && aligned16(a.q) && aligned16(a.d_y) && aligned16(a.d_k) &&
                    aligned16(a.d_v) && aligned16(a.d_q) && aligned16(a.m_traj) && (a.traj_stride % 4 == 0) &&
                    aligned16(a.s_traj) && aligned16(a.d_m_seed) && aligned16(a.d_s_seed) &&
                    (a.atomic_out || (aligned16(a.d_m_out) && aligned16(a.d_s_out)));
    if (!al) return false;
    const bool solve = !a.frozen;
    if (rule == RULE_TITANS) {
        if (sder) launch_bwd<RULE_TITANS, true, true>(a, T, mstep, st);
        else if (solve) launch_bwd<RULE_TITANS, true, false>(a, T, mstep, st);
        else launch_bwd<RULE_TITANS, false, false>(a, T, mstep, st);
    } else {
        if (solve) launch_bwd<RULE_DELTA, true, false>(a, T, mstep, st);
        else launch_bwd<RULE_DELTA, false, false>(a, T, mstep, st);
    }
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
