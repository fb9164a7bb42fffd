// seq_ssm.cuh -- arguments and segments of the state-space scan, shared by the recurrence (seq_ssm.cu) and the tile products (seq_ssm_tc.cu).
#pragma once
#include "seq_common.cuh"

namespace b200seq {

constexpr int SSM_TT = 16;     // tokens per staged tile
constexpr int SSM_SEG = 128;   // tokens per parallel segment
constexpr int SSM_WARPS = 8;
enum { SSM_DIRECT = 0, SSM_LOCAL = 1, SSM_FINAL = 2 };

struct SsmArgs {
    const float* proj;
    int64_t ldp;
    int z0, dt0;
    const float* xbc;
    int64_t ldx;
    const float *A_log, *Dp, *dt_bias;
    float* state;     // [slots][H][N][V]
    float* seg_state; // [segments][H][N][V]   (E after pass A, start state after pass B)
    float* seg_logdec;  // [segments][H]
    float* out;
    int H, V, N, G, NL, seg_len;
};

// segment `idx` of the step: entry, first token row, token count, whether it is the entry's first
__device__ __forceinline__ bool ssm_find_segment(const b200seq_step& st, int idx, int seg_len, int& e, int& row0, int& len) {
    int acc = 0;
    for (e = 0; e < st.B; ++e) {
        const int s0 = st.ent_start[e], n = st.ent_start[e + 1] - s0;
        const int ns = (n + seg_len - 1) / seg_len;
        if (idx < acc + ns) {
            const int local = idx - acc;
            row0 = s0 + local * seg_len;
            len = min(seg_len, n - local * seg_len);
            return true;
        }
        acc += ns;
    }
    return false;
}

// the tile products: passes A and C of long steps (one = false), or a step whose entries are one segment each (one = true; no pass B, no scratch)
cudaError_t launch_ssm_tiles_local(const SsmArgs& a, const b200seq_step& st, int segs, bool one, cudaStream_t cs);
cudaError_t launch_ssm_tiles_out(const SsmArgs& a, const b200seq_step& st, int segs, bool one, cudaStream_t cs);

}  // namespace b200seq
