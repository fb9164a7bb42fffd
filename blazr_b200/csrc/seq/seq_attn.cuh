// seq_attn.cuh -- what the attention kernels share: row lookup in the paged pool, the arguments of the attend step, its query tiles
#pragma once
#include "seq_common.cuh"

namespace b200seq {

__device__ __forceinline__ int64_t kv_row(const b200seq_step& st, int e, int pos, int* err) {
    const int b = pos / st.block_size;
    if (b >= st.max_blocks || pos < 0) {
        atomicOr(err, 1);
        return -1;
    }
    return (int64_t)st.block_table[(int64_t)e * st.max_blocks + b] * st.block_size + pos % st.block_size;
}

// pooled entry of block b (positions b * P .. b * P + P - 1) of a sequence: it lives in the page of the block's first position, at
// the block's rank among the blocks that start in that page
__device__ __forceinline__ int64_t pooled_row(const int32_t* bt, int bs, int P, int ppp, int b) {
    const int pg = (b * P) / bs;
    const int first = (pg * bs + P - 1) / P;
    return (int64_t)bt[pg] * ppp + (b - first);
}

struct AttnArgs {
    const float* qkvg;
    int64_t ld;
    const float *kpool, *vpool;
    const float *kpp, *vpp;   // pooled keys / values, pool > 0
    int pool, ppp;            // positions per pooled block; pooled entries per page
    int q_col, gate_col;
    int H, G, D, V, Rb, HB, QT, nsplit, share_kv;   // share_kv: V tiles reuse the K tile's shared memory (large heads: more blocks per SM)
    float scale;
    int chunk, window, gated;
    void* out;
    int out_dtype;
    float* part;   // [T][H][nsplit][V + 2] when nsplit > 1
    int* err;
    const float* sink;   // [H] or null: exp(sink[h]) joins the soft-max denominator of head h once; it has no key and no value
    const float* gate;   // gate logits [T][gld] (+ h)
    int64_t gld;
    int64_t kld, vld;    // floats per position in kpool / vpool (G * D and G * V, or the key row's width when the values lie inside the key rows)
    int ctx_rows;        // 1: kpool / vpool rows are the step's gathered context, entry after entry, position after position (no pages)
    int kd;              // floats of a key head that lie in kpool (at g * kd); the remaining D - kd come from krot, one part for all heads
    const float* krot;   // paged rows of krld floats (pointer already at the part's first column), or null
    int64_t krld;
    const float* head_scale;   // [H] or null: one more factor of head h's scores
    float softcap;             // > 0: score <- softcap * tanh(score / softcap)
    int keep_first;            // with a window: positions below this stay visible to all later positions
    int vdiv;                  // key head g reads value head g / vdiv
    int gate_elem;             // the gate has one logit per output element: gate[t * gld + h * V + c]
};

__device__ __forceinline__ bool attn_find_tile(const b200seq_step& st, int idx, int QT, int& e, int& t0, int& nq) {
    int acc = 0;
    for (e = 0; e < st.B; ++e) {
        const int s0 = st.ent_start[e], n = st.ent_start[e + 1] - s0;
        const int nt = (n + QT - 1) / QT;
        if (idx < acc + nt) {
            const int local = idx - acc;
            t0 = s0 + local * QT;
            nq = min(QT, n - local * QT);
            return true;
        }
        acc += nt;
    }
    return false;
}

// Attend step of many rows on the tensor cores (seq_attn_tc.cu).  max_keys bounds the keys one token sees; a.part holds part_floats.  Returns
// false when the step is not for that kernel (nothing is launched), else its status is in rc; a.nsplit is then what was used.
bool launch_attn_tc(AttnArgs& a, const b200seq_step& st, int max_keys, size_t part_floats, cudaStream_t cs, int& rc);

}  // namespace b200seq
