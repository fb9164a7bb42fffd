// seq_ssm.cu -- selective state-space recurrence (scalar decay per head, state N x V per head) over a flat mixed batch.
//
// One block per (tile of value columns, head, segment of tokens).  A value column's state (N floats) is spread over NL lanes
// (NL = 1, 2, 4 or 8, at most 32 floats per lane, so it stays in registers); a warp covers 32 / NL columns.  The tokens of a
// segment are walked in order; x, z, B, C, the step sizes and the decays of a tile of SSM_TT tokens are staged in shared memory
// with coalesced loads, the outputs of the tile leave through shared memory too.  Step sizes, decays and the state are f32.
//
// Short steps (T <= SSM_SEG: decode, small portions): one launch, a segment is an entry's whole portion, the state comes from and
// returns to the sequence's slot (read as zero for a new sequence).
// Long steps: every entry is cut into segments of SSM_SEG tokens that run in parallel, in three launches:
//   A  each segment runs the recurrence from a zero state -> its local end state E and the sum of its log-decays
//   B  per entry, in order: start[s] = S;  S = exp(sum log-decay of s) * S + E[s]   (elementwise; the last S goes to the slot)
//   C  each segment runs again from start[s] and writes the outputs
// which costs twice the arithmetic of the plain recurrence and removes the dependence on the portion's length.
// States of up to 128 x any multiple of 4 columns take passes A and C as products of tiles instead (below): the recurrence spends a multiply on the
// decay and one on the input for every multiply-add that counts, and walks its tokens one after another; pass B runs eight segments ahead.
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

// NPL: state floats per lane.  Lane -> (sub = lane / cpw, col = lane % cpw), cpw = 32 / NL; the lane holds n = sub * NPL + i.
template <int NPL, int MODE>
__global__ void __launch_bounds__(SSM_WARPS * 32) ssm_kernel(const SsmArgs a, const b200seq_step st) {
    extern __shared__ __align__(16) float sm[];
    const int H = a.H, V = a.V, N = a.N, NL = a.NL;
    const int cpw = 32 / NL, cols = SSM_WARPS * cpw;       // value columns of this block (NL, cpw, cols and NPL are powers of two)
    const int cols_shift = 31 - __clz(cols), npl_shift = 31 - __clz(NPL), nn_shift = npl_shift + (31 - __clz(NL));
    const int nstride = NPL + 4;                           // padded chunk of one sub-lane (conflict-free 16-byte reads)
    const int nrow = NL * nstride;
    float* Bs = sm;                          // [SSM_TT][nrow]
    float* Cs = Bs + SSM_TT * nrow;          // [SSM_TT][nrow]
    float* xs = Cs + SSM_TT * nrow;          // [SSM_TT][cols]   (outputs replace x)
    float* zs = xs + SSM_TT * cols;          // [SSM_TT][cols]
    float* dts = zs + SSM_TT * cols;         // [SSM_TT]
    float* dec = dts + SSM_TT;               // [SSM_TT]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane / cpw, cl = warp * cpw + lane % cpw;
    const int v0 = blockIdx.x * cols, v = v0 + cl;
    const int h = blockIdx.y;
    int e, row0, len;
    if (MODE == SSM_DIRECT) {
        e = blockIdx.z;
        row0 = st.ent_start[e];
        len = st.ent_start[e + 1] - row0;
    } else if (!ssm_find_segment(st, blockIdx.z, a.seg_len, e, row0, len)) {
        return;
    }
    const bool live = v < V;
    const int g = h / (H / a.G);
    const int inner = H * V;
    float S[NPL];
    const float* init = nullptr;
    if (MODE == SSM_DIRECT) init = st.ent_pos0[e] == 0 ? nullptr : a.state + ((int64_t)st.ent_slot[e] * H + h) * N * V;
    if (MODE == SSM_FINAL) init = a.seg_state + ((int64_t)blockIdx.z * H + h) * N * V;
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
        const int n = sub * NPL + i;
        S[i] = (init && live && n < N) ? init[(int64_t)n * V + v] : 0.f;
    }
    const float negA = -expf(a.A_log[h]);
    const float dtb = a.dt_bias[h], Dh = a.Dp[h];
    float logdec = 0.f;   // thread 0 only (pass A)
    for (int i0 = 0; i0 < len; i0 += SSM_TT) {
        const int nt = min(SSM_TT, len - i0);
        __syncthreads();
        for (int idx = tid; idx < (nt << nn_shift); idx += blockDim.x) {
            const int tt = idx >> nn_shift, n = idx & ((1 << nn_shift) - 1);
            const int at = tt * nrow + (n >> npl_shift) * nstride + (n & (NPL - 1));
            float b = 0.f, c = 0.f;
            if (n < N) {
                const float* r = a.xbc + (int64_t)(row0 + i0 + tt) * a.ldx + inner + (int64_t)g * N + n;
                b = r[0];
                if (MODE != SSM_LOCAL) c = r[(int64_t)a.G * N];
            }
            Bs[at] = b;
            Cs[at] = c;
        }
        for (int idx = tid; idx < (nt << cols_shift); idx += blockDim.x) {
            const int tt = idx >> cols_shift, c = idx & (cols - 1);
            const int64_t row = row0 + i0 + tt;
            const bool in = v0 + c < V;
            xs[idx] = in ? a.xbc[row * a.ldx + (int64_t)h * V + v0 + c] : 0.f;
            if (MODE != SSM_LOCAL) zs[idx] = in ? a.proj[row * a.ldp + a.z0 + (int64_t)h * V + v0 + c] : 0.f;
        }
        if (tid < nt) {
            const float dt = softplusf_acc(a.proj[(int64_t)(row0 + i0 + tid) * a.ldp + a.dt0 + h] + dtb);
            dts[tid] = dt;
            dec[tid] = expf(negA * dt);
        }
        __syncthreads();
        if (MODE == SSM_LOCAL && tid == 0)
            for (int tt = 0; tt < nt; ++tt) logdec += negA * dts[tt];
        for (int tt = 0; tt < nt; ++tt) {
            const float x = xs[tt * cols + cl];
            const float dA = dec[tt], dtx = dts[tt] * x;
            const float4* Bt = reinterpret_cast<const float4*>(Bs + tt * nrow + sub * nstride);
            const float4* Ct = reinterpret_cast<const float4*>(Cs + tt * nrow + sub * nstride);
            float y0 = 0.f, y1 = 0.f, y2 = 0.f, y3 = 0.f;
#pragma unroll
            for (int i = 0; i < NPL / 4; ++i) {
                const float4 b = Bt[i];
                S[4 * i] = fmaf(dA, S[4 * i], dtx * b.x);
                S[4 * i + 1] = fmaf(dA, S[4 * i + 1], dtx * b.y);
                S[4 * i + 2] = fmaf(dA, S[4 * i + 2], dtx * b.z);
                S[4 * i + 3] = fmaf(dA, S[4 * i + 3], dtx * b.w);
                if (MODE != SSM_LOCAL) {
                    const float4 c = Ct[i];
                    y0 = fmaf(S[4 * i], c.x, y0), y1 = fmaf(S[4 * i + 1], c.y, y1), y2 = fmaf(S[4 * i + 2], c.z, y2), y3 = fmaf(S[4 * i + 3], c.w, y3);
                }
            }
            if (MODE != SSM_LOCAL) {
                float y = (y0 + y1) + (y2 + y3);
                for (int o = cpw; o < 32; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                __syncwarp();
                if (sub == 0) xs[tt * cols + cl] = fmaf(Dh, x, y) * siluf_acc(zs[tt * cols + cl]);   // x of this token is consumed
            }
        }
        if (MODE != SSM_LOCAL) {
            __syncthreads();
            for (int idx = tid; idx < (nt << cols_shift); idx += blockDim.x) {
                const int tt = idx >> cols_shift, c = idx & (cols - 1);
                if (v0 + c < V) a.out[(int64_t)(row0 + i0 + tt) * inner + (int64_t)h * V + v0 + c] = xs[idx];
            }
        }
    }
    if (MODE == SSM_FINAL) return;
    float* dst = MODE == SSM_DIRECT ? a.state + ((int64_t)st.ent_slot[e] * H + h) * N * V : a.seg_state + ((int64_t)blockIdx.z * H + h) * N * V;
    if (live) {
#pragma unroll
        for (int i = 0; i < NPL; ++i) {
            const int n = sub * NPL + i;
            if (n < N) dst[(int64_t)n * V + v] = S[i];
        }
    }
    if (MODE == SSM_LOCAL && tid == 0 && blockIdx.x == 0) a.seg_logdec[(int64_t)blockIdx.z * H + h] = logdec;
}

// pass B: VW values (one thread) of an (entry, head, n, v); walks the entry's segments in order.  The loads of eight segments do not depend on one
// another and are issued together (one at a time, each behind the store before it: 791 us for 33 segments of 64 x 128 x 64, now bound by memory).
template <int VW>
__global__ void ssm_combine_kernel(const SsmArgs a, const b200seq_step st) {
    const int64_t per = (int64_t)a.H * a.N * a.V;
    const int64_t idx = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VW;
    const int e = blockIdx.y;
    if (idx >= per) return;
    const int h = (int)(idx / ((int64_t)a.N * a.V));
    int seg0 = 0;
    for (int i = 0; i < e; ++i) seg0 += (st.ent_start[i + 1] - st.ent_start[i] + a.seg_len - 1) / a.seg_len;
    const int ns = (st.ent_start[e + 1] - st.ent_start[e] + a.seg_len - 1) / a.seg_len;
    struct alignas(4 * VW) Vec {
        float f[VW];
    };
    Vec* slot = reinterpret_cast<Vec*>(a.state + (int64_t)st.ent_slot[e] * per + idx);
    Vec S{};
    if (st.ent_pos0[e] != 0) S = *slot;
    constexpr int AHEAD = 8;
    for (int s0 = 0; s0 < ns; s0 += AHEAD) {
        Vec E[AHEAD];
        float d[AHEAD];
        Vec* p = reinterpret_cast<Vec*>(a.seg_state + (int64_t)(seg0 + s0) * per + idx);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (s0 + i < ns) E[i] = *reinterpret_cast<const Vec*>(reinterpret_cast<const float*>(p) + i * per), d[i] = expf(a.seg_logdec[(int64_t)(seg0 + s0 + i) * a.H + h]);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (s0 + i < ns) {
                *reinterpret_cast<Vec*>(reinterpret_cast<float*>(p) + i * per) = S;
#pragma unroll
                for (int u = 0; u < VW; ++u) S.f[u] = fmaf(d[i], S.f[u], E[i].f[u]);
            }
    }
    *slot = S;
}

// ---- passes A and C as tile products -----------------------------------------------------------------------------------------------
// Over a segment of up to SSM_SEG tokens with step sizes dt and L_t the sum of the log-decays up to and including t:
//     E        = sum_s (dt_s exp(L_end - L_s)) B_s x_s^T                                                   [N x V]
//     y_t      = exp(L_t) C_t^T S_start + sum_(s <= t) (C_t . B_s) exp(L_t - L_s) dt_s x_s                  [V]
// f32 multiply-adds (packed pairs) on register tiles of 8 x 4 of a 128 x 64 result, operands staged in shared memory 32 deep.  Decays are
// exponentials of differences of the sums (never above 1), the sums kept as a float pair of the f64 running sum, so that a difference late in
// the segment is as exact as an early one.  C_t . B_s does not depend on the head: a block of pass C makes the 128 x 128 of them once and
// serves SSM_HB heads of the group; earlier tokens enter blockwise -- after 32 tokens the running rows are scaled to the new reference point -- and
// the tokens of a row's own 32 through a masked 32 x 32 block with exact decays.
// Every 32 terms are summed by themselves and then added: the rounding of a chain grows with its length.
// Bound by the f32 pipe (4096 tokens, 64 heads of 64, state 128: 13 GFLOP).
constexpr int ST_NT = 256, ST_K = 32, ST_V = 64, ST_P = SSM_SEG + 4;
constexpr int SSM_HB = 4;

__device__ __forceinline__ uint64_t ss_pk(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void ss_fma2(uint64_t& c, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint64_t ss_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2 ss_upk(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// dt and the running log-decay of the segment's tokens for head h (threads 0 .. 127); tokens beyond the segment: dt 0, the last sum
struct SegDecay {
    float dt[SSM_SEG], hi[SSM_SEG], lo[SSM_SEG];
    double part[4];
};
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 256;" ::"r"(1 + group) : "memory"); }   // ST_NT threads each
__device__ __forceinline__ bool group_any(int group, bool mine) {   // the same barrier; true for all when it is for one
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, %2, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((int)mine), "r"(1 + group) : "memory");
    return any != 0;
}
__device__ __forceinline__ void seg_decay(SegDecay& d, const SsmArgs& a, int h, int row0, int len, int t, int group) {
    const int lane = t & 31;
    double L = 0.0;
    if (t < SSM_SEG) {
        const float dt = t < len ? softplusf_acc(a.proj[(int64_t)(row0 + t) * a.ldp + a.dt0 + h] + a.dt_bias[h]) : 0.f;
        d.dt[t] = dt;
        const float ld = t < len ? -expf(a.A_log[h]) * dt : 0.f;
        L = ld < -200.f ? -200.0 : (double)ld;   // exp of either is 0 in f32; a sum of infinite terms would have no differences
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, L, o);
            if (lane >= o) L += u;
        }
        if (lane == 31) d.part[t >> 5] = L;
    }
    group_sync(group);
    if (t < SSM_SEG) {
        for (int w = 0; w < (t >> 5); ++w) L += d.part[w];
        const float hi = (float)L;
        d.hi[t] = hi, d.lo[t] = (float)(L - (double)hi);
    }
    group_sync(group);
}
// exp(L_t - L_s), t >= s (s = -1: from the segment's start)
__device__ __forceinline__ float seg_exp(const SegDecay& d, int t, int s) {
    return s < 0 ? expf(d.hi[t] + d.lo[t]) : expf((d.hi[t] - d.hi[s]) + (d.lo[t] - d.lo[s]));
}

// pass A: grid (V / 64, H, segments); thread (ty, tx) owns the state rows 4 ty + {0..3} (+ 64) and the columns 4 tx + {0..3}
template <int NR>   // state rows / 64: 1 or 2
__global__ void __launch_bounds__(ST_NT) ssm_tile_local_kernel(const SsmArgs a, const b200seq_step st) {
    __shared__ __align__(16) float Bs[ST_K][64 * NR], Xs[ST_K][ST_V];
    __shared__ SegDecay dec;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int h = blockIdx.y, v0 = blockIdx.x * ST_V, N = a.N, V = a.V, inner = a.H * V, g = h / (a.H / a.G);
    int e, row0, len;
    if (!ssm_find_segment(st, blockIdx.z, a.seg_len, e, row0, len)) return;
    seg_decay(dec, a, h, row0, len, tid, 0);
    uint64_t acc[2 * NR][4];
#pragma unroll
    for (int i = 0; i < 2 * NR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    const float* xb = a.xbc + (int64_t)h * V + v0;
    const float* bb = a.xbc + inner + (int64_t)g * N;
    float4 rb[2 * NR], rx[2];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i) {
            const int idx = tid + i * ST_NT, tt = idx / (16 * NR), c = idx % (16 * NR) * 4;
            rb[i] = t0 + tt < len && c < N ? ld4(bb + (int64_t)(row0 + t0 + tt) * a.ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = tid + i * ST_NT, tt = idx / 16, c = idx % 16 * 4;
            rx[i] = t0 + tt < len && v0 + c < V ? ld4(xb + (int64_t)(row0 + t0 + tt) * a.ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(0);
    for (int t0 = 0; t0 < len; t0 += ST_K) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i) {
            const int idx = tid + i * ST_NT;
            *reinterpret_cast<float4*>(&Bs[idx / (16 * NR)][idx % (16 * NR) * 4]) = rb[i];
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = tid + i * ST_NT, tt = idx / 16;
            const float w = dec.dt[t0 + tt] * seg_exp(dec, SSM_SEG - 1, t0 + tt);
            *reinterpret_cast<float4*>(&Xs[tt][idx % 16 * 4]) = make_float4(rx[i].x * w, rx[i].y * w, rx[i].z * w, rx[i].w * w);
        }
        __syncthreads();
        if (t0 + ST_K < len) fetch(t0 + ST_K);
        uint64_t sum[2 * NR][4];
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[i][j] = 0;
#pragma unroll 8
        for (int k = 0; k < ST_K; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(&Xs[k][4 * tx]);
            const uint64_t xx[4] = {ss_pk(x.x, x.x), ss_pk(x.y, x.y), ss_pk(x.z, x.z), ss_pk(x.w, x.w)};
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&Bs[k][64 * r + 4 * ty]);
#pragma unroll
                for (int j = 0; j < 4; ++j) ss_fma2(sum[2 * r][j], b.x, xx[j]), ss_fma2(sum[2 * r + 1][j], b.y, xx[j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = ss_add2(acc[i][j], sum[i][j]);
    }
    float* dst = a.seg_state + ((int64_t)blockIdx.z * a.H + h) * N * V + v0 + 4 * tx;
    if (v0 + 4 * tx < V) {
#pragma unroll
        for (int i = 0; i < 2 * NR; ++i) {
            const int n = 64 * (i >> 1) + 4 * ty + 2 * (i & 1);
            const float2 p0 = ss_upk(acc[i][0]), p1 = ss_upk(acc[i][1]), p2 = ss_upk(acc[i][2]), p3 = ss_upk(acc[i][3]);
            if (n < N) *reinterpret_cast<float4*>(dst + (int64_t)n * V) = make_float4(p0.x, p1.x, p2.x, p3.x);
            if (n + 1 < N) *reinterpret_cast<float4*>(dst + (int64_t)(n + 1) * V) = make_float4(p0.y, p1.y, p2.y, p3.y);
        }
    }
    if (tid == 0 && blockIdx.x == 0) a.seg_logdec[(int64_t)blockIdx.z * a.H + h] = dec.hi[SSM_SEG - 1] + dec.lo[SSM_SEG - 1];
}

// pass C: grid (V / 64, group x head blocks, segments), two groups of 256 threads that take every other head.  Token t of the segment sits at
// place 8 (t % 16) + t / 16 of a shared-memory row, so that the eight tokens ty + 16 i of a thread are two 16-byte loads, and the first 2 c of
// them belong to the first c blocks of 32 tokens.  With one group of 256 threads and each tile fetched when it was needed the pass took 649 us
// (4096 tokens, 64 heads of 64, state 128): two warps per scheduler waiting for loads and barriers.
struct TileGroup {
    float K[ST_K][ST_P];            // 32-deep tile of S, or of the block's dt x (columns 0 .. 63) beside the same decayed to the block's end (64 .. 127)
    float M[ST_K][ST_K + 4];        // the own block's masked weights [s][t]
    SegDecay dec;
};
struct TileOut {
    float Ct[128][ST_P];            // [n][token place]
    float Gt[SSM_SEG][ST_P];        // [s][token place]: C_t . B_s
    TileGroup grp[2];
};
__device__ __forceinline__ int tok_place(int t) { return 8 * (t & 15) + (t >> 4); }

__global__ void __launch_bounds__(2 * ST_NT) ssm_tile_out_kernel(const SsmArgs a, const b200seq_step st) {
    extern __shared__ __align__(16) unsigned char raw[];
    TileOut& sm = *reinterpret_cast<TileOut*>(raw);
    const int gi = threadIdx.x / ST_NT, tid = threadIdx.x % ST_NT, tx = tid & 15, ty = tid >> 4;
    TileGroup& sg = sm.grp[gi];
    const int N = a.N, V = a.V, H = a.H, v0 = blockIdx.x * ST_V, per = H / a.G, nb = (per + SSM_HB - 1) / SSM_HB;
    const int g = blockIdx.y / nb, h_first = g * per + (blockIdx.y % nb) * SSM_HB, h_end = min(h_first + SSM_HB, (g + 1) * per);
    const int inner = H * V, nq = (N + ST_K - 1) / ST_K;
    int e, row0, len;
    if (!ssm_find_segment(st, blockIdx.z, a.seg_len, e, row0, len)) return;
    const int nblk = (len + ST_K - 1) / ST_K;
    const float* bb = a.xbc + inner + (int64_t)g * N;
    const float* cb = bb + (int64_t)a.G * N;
    // tile i of head h: rows 32 i .. of the start state (i < nq), then the x rows of block i - nq
    float4 nx[2];
    auto fetch = [&](int h, int i) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int idx = tid + u * ST_NT, r = idx >> 4, c = (idx & 15) * 4;
            nx[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (h < h_end && v0 + c < V) {
                if (i < nq) {
                    if (i * ST_K + r < N) nx[u] = ld4(a.seg_state + (((int64_t)blockIdx.z * H + h) * N + i * ST_K + r) * V + v0 + c);
                } else if ((i - nq) * ST_K + r < len) {
                    nx[u] = ld4(a.xbc + (int64_t)(row0 + (i - nq) * ST_K + r) * a.ldx + (int64_t)h * V + v0 + c);
                }
            }
        }
    };
    fetch(h_first + gi, 0);
    // C, transposed (rows beyond the segment and n beyond the state are zero)
    for (int idx = threadIdx.x; idx < SSM_SEG * 32; idx += 2 * ST_NT) {
        const int t = (idx & 7) + 8 * (idx >> 8), n = ((idx >> 3) & 31) * 4, at = tok_place(t);
        const float4 c = t < len && n < N ? ld4(cb + (int64_t)(row0 + t) * a.ldx + n) : make_float4(0.f, 0.f, 0.f, 0.f);
        sm.Ct[n][at] = c.x, sm.Ct[n + 1][at] = c.y, sm.Ct[n + 2][at] = c.z, sm.Ct[n + 3][at] = c.w;
    }
    {   // C_t . B_s: a thread's 8 tokens x 4 columns s = 64 gi + 4 tx + {0..3}; the tokens of the first half see none of the second
        uint64_t acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0;
        for (int n0 = 0; n0 < N; n0 += ST_K) {
            __syncthreads();
            for (int idx = threadIdx.x; idx < SSM_SEG * 8; idx += 2 * ST_NT) {   // B's tile, transposed, in group 0's buffer
                const int s_ = idx >> 3, n = (idx & 7) * 4;
                const float4 b = s_ < len && n0 + n < N ? ld4(bb + (int64_t)(row0 + s_) * a.ldx + n0 + n) : make_float4(0.f, 0.f, 0.f, 0.f);
                sm.grp[0].K[n][s_] = b.x, sm.grp[0].K[n + 1][s_] = b.y, sm.grp[0].K[n + 2][s_] = b.z, sm.grp[0].K[n + 3][s_] = b.w;
            }
            __syncthreads();
            uint64_t sum[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[i][j] = 0;
#pragma unroll 8
            for (int k = 0; k < ST_K; ++k) {
                const float4 x = *reinterpret_cast<const float4*>(&sm.grp[0].K[k][64 * gi + 4 * tx]);
                const uint64_t xx[4] = {ss_pk(x.x, x.x), ss_pk(x.y, x.y), ss_pk(x.z, x.z), ss_pk(x.w, x.w)};
                const ulonglong2 c1 = *reinterpret_cast<const ulonglong2*>(&sm.Ct[n0 + k][8 * ty + 4]);
#pragma unroll
                for (int j = 0; j < 4; ++j) ss_fma2(sum[2][j], c1.x, xx[j]), ss_fma2(sum[3][j], c1.y, xx[j]);
                if (gi == 0) {
                    const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(&sm.Ct[n0 + k][8 * ty]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) ss_fma2(sum[0][j], c0.x, xx[j]), ss_fma2(sum[1][j], c0.y, xx[j]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = ss_add2(acc[i][j], sum[i][j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            *reinterpret_cast<ulonglong2*>(&sm.Gt[64 * gi + 4 * tx + j][8 * ty]) = make_ulonglong2(acc[0][j], acc[1][j]);
            *reinterpret_cast<ulonglong2*>(&sm.Gt[64 * gi + 4 * tx + j][8 * ty + 4]) = make_ulonglong2(acc[2][j], acc[3][j]);
        }
    }
    __syncthreads();   // Gt is complete, B's tile has been read
    for (int h = h_first + gi; h < h_end; h += 2) {
        seg_decay(sg.dec, a, h, row0, len, tid, gi);   // (its first barrier lies behind the head before's last use of dec: see the barrier at the loop's end)
        uint64_t acc[4][4];   // tokens ty + 16 (2 i, 2 i + 1), columns 4 tx + j
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0;
        for (int q = 0; q < nq; ++q) {   // C_t^T S_start
            if (q > 0) group_sync(gi);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int idx = tid + u * ST_NT;
                *reinterpret_cast<float4*>(&sg.K[idx >> 4][(idx & 15) * 4]) = nx[u];
            }
            group_sync(gi);
            fetch(h, q + 1);
            uint64_t sum[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[i][j] = 0;
#pragma unroll 8
            for (int k = 0; k < ST_K; ++k) {
                const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(&sm.Ct[q * ST_K + k][8 * ty]), c1 = *reinterpret_cast<const ulonglong2*>(&sm.Ct[q * ST_K + k][8 * ty + 4]);
                const float4 x = *reinterpret_cast<const float4*>(&sg.K[k][4 * tx]);
                const uint64_t xx[4] = {ss_pk(x.x, x.x), ss_pk(x.y, x.y), ss_pk(x.z, x.z), ss_pk(x.w, x.w)};
#pragma unroll
                for (int j = 0; j < 4; ++j) ss_fma2(sum[0][j], c0.x, xx[j]), ss_fma2(sum[1][j], c0.y, xx[j]), ss_fma2(sum[2][j], c1.x, xx[j]), ss_fma2(sum[3][j], c1.y, xx[j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = ss_add2(acc[i][j], sum[i][j]);
        }
        // rows are relative to the reference point r = 32 c - 1 (the segment's start for c = 0)
#pragma unroll
        for (int c = 0; c < SSM_SEG / ST_K; ++c) {
            const int s0 = c * ST_K;
            if (c < nblk) {
                group_sync(gi);
                bool odd = false;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int idx = tid + u * ST_NT, r = idx >> 4, col = (idx & 15) * 4;
                    const float w = sg.dec.dt[s0 + r], w2 = w * seg_exp(sg.dec, s0 + ST_K - 1, s0 + r);
                    const float4 k = make_float4(nx[u].x * w, nx[u].y * w, nx[u].z * w, nx[u].w * w);
                    odd |= !(isfinite(k.x) && isfinite(k.y) && isfinite(k.z) && isfinite(k.w));
                    *reinterpret_cast<float4*>(&sg.K[r][col]) = k;
                    *reinterpret_cast<float4*>(&sg.K[r][64 + col]) = make_float4(nx[u].x * w2, nx[u].y * w2, nx[u].z * w2, nx[u].w * w2);
                }
#pragma unroll
                for (int u = 0; u < ST_K * ST_K / ST_NT; ++u) {
                    const int idx = tid + u * ST_NT, s_ = idx >> 5, t = idx & 31;
                    sg.M[s_][t] = t >= s_ ? sm.Gt[s0 + s_][tok_place(s0 + t)] * seg_exp(sg.dec, s0 + t, s0 + s_) : 0.f;
                }
                odd = group_any(gi, odd);
                if (c + 1 < nblk) fetch(h, nq + c + 1);
                else fetch(h + 2, 0);
                {   // the block's own rows (tokens s0 + ty, s0 + 16 + ty) are finished: scale to the token, add the block's own part
                    const uint64_t ff = ss_pk(seg_exp(sg.dec, s0 + ty, s0 - 1), seg_exp(sg.dec, s0 + 16 + ty, s0 - 1));
                    uint64_t own[4] = {0, 0, 0, 0};
                    if (!odd) {
#pragma unroll 8
                        for (int k = 0; k < ST_K; ++k) {
                            const uint64_t m = ss_pk(sg.M[k][ty], sg.M[k][16 + ty]);
                            const float4 x = *reinterpret_cast<const float4*>(&sg.K[k][4 * tx]);
                            ss_fma2(own[0], m, ss_pk(x.x, x.x)), ss_fma2(own[1], m, ss_pk(x.y, x.y)), ss_fma2(own[2], m, ss_pk(x.z, x.z)), ss_fma2(own[3], m, ss_pk(x.w, x.w));
                        }
                    } else {   // a value that is not finite: a masked weight of zero does not keep it from earlier tokens, so each token's sum ends at its own
#pragma unroll 1
                        for (int k = 0; k <= 16 + ty; ++k) {
                            const float m0 = sg.M[k][ty], m1 = sg.M[k][16 + ty];
                            const float x[4] = {sg.K[k][4 * tx], sg.K[k][4 * tx + 1], sg.K[k][4 * tx + 2], sg.K[k][4 * tx + 3]};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 o = ss_upk(own[j]);
                                own[j] = ss_pk(k <= ty ? fmaf(m0, x[j], o.x) : o.x, fmaf(m1, x[j], o.y));
                            }
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint64_t r = own[j];
                        ss_fma2(r, acc[c][j], ff);
                        acc[c][j] = r;
                    }
                }
                if (c + 1 < nblk) {   // later rows: to the reference point at the block's end
                    const float f = seg_exp(sg.dec, s0 + ST_K - 1, s0 - 1);
                    const uint64_t ff = ss_pk(f, f);
                    uint64_t sum[4][4];
#pragma unroll
                    for (int i = c + 1; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) sum[i][j] = 0;
#pragma unroll 8
                    for (int k = 0; k < ST_K; ++k) {
                        const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(&sm.Gt[s0 + k][8 * ty]), c1 = *reinterpret_cast<const ulonglong2*>(&sm.Gt[s0 + k][8 * ty + 4]);
                        const uint64_t cc[4] = {c0.x, c0.y, c1.x, c1.y};
                        const float4 x = *reinterpret_cast<const float4*>(&sg.K[k][64 + 4 * tx]);
                        const uint64_t xx[4] = {ss_pk(x.x, x.x), ss_pk(x.y, x.y), ss_pk(x.z, x.z), ss_pk(x.w, x.w)};
#pragma unroll
                        for (int i = c + 1; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) ss_fma2(sum[i][j], cc[i], xx[j]);
                    }
#pragma unroll
                    for (int i = c + 1; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            ss_fma2(sum[i][j], acc[i][j], ff);
                            acc[i][j] = sum[i][j];
                        }
                }
            }
        }
        // + D x, times silu(z)
        const float Dh = a.Dp[h];
        const float* xb = a.xbc + (int64_t)h * V + v0;
        const float* zb = a.proj + a.z0 + (int64_t)h * V + v0;
        float* ob = a.out + (int64_t)h * V + v0;
        const int col = 4 * tx;
        if (v0 + col < V) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int t = ty + 16 * i;
                if (t >= len) break;
                const int64_t row = row0 + t;
                const float2 p0 = ss_upk(acc[i >> 1][0]), p1 = ss_upk(acc[i >> 1][1]), p2 = ss_upk(acc[i >> 1][2]), p3 = ss_upk(acc[i >> 1][3]);
                const float4 y = (i & 1) ? make_float4(p0.y, p1.y, p2.y, p3.y) : make_float4(p0.x, p1.x, p2.x, p3.x);
                const float4 x = ld4(xb + row * a.ldx + col), z = ld4(zb + row * a.ldp + col);
                *reinterpret_cast<float4*>(ob + row * inner + col) =
                    make_float4(fmaf(Dh, x.x, y.x) * siluf_acc(z.x), fmaf(Dh, x.y, y.y) * siluf_acc(z.y), fmaf(Dh, x.z, y.z) * siluf_acc(z.z), fmaf(Dh, x.w, y.w) * siluf_acc(z.w));
            }
        }
        group_sync(gi);   // the group is done with this head's K, M and dec
    }
}

template <int NPL, int MODE>
static cudaError_t ssm_launch(const SsmArgs& a, const b200seq_step& st, int nz, cudaStream_t cs) {
    const int cpw = 32 / a.NL, cols = SSM_WARPS * cpw;
    const size_t smem = ((size_t)2 * SSM_TT * a.NL * (NPL + 4) + 2 * SSM_TT * cols + 2 * SSM_TT + 4) * sizeof(float);
    dim3 grid((a.V + cols - 1) / cols, a.H, nz);
    ssm_kernel<NPL, MODE><<<grid, SSM_WARPS * 32, smem, cs>>>(a, st);
    return cudaGetLastError();
}

}  // namespace b200seq

using namespace b200seq;

extern "C" size_t b200seq_ssm_scratch_floats(int T, int B, int H, int V, int N) {
    if (T <= SSM_SEG) return 0;
    const size_t segs = (size_t)(T + SSM_SEG - 1) / SSM_SEG + (size_t)B;
    return segs * ((size_t)H * N * V + H);
}

extern "C" int b200seq_ssm_scan(const float* proj, int64_t ldp, int z0, int dt0, const float* xbc, int64_t ldx, const float* A_log, const float* Dp,
                                const float* dt_bias, float* state, const b200seq_step* st, int H, int V, int N, int G, float* out, float* scratch,
                                size_t scratch_floats, void* stream) {
    if (!proj || !xbc || !A_log || !Dp || !dt_bias || !state || !st || !out || H < 1 || V < 1 || N < 1 || G < 1 || H % G)
        return fail(B200SEQ_ERR_INVALID_ARG, "ssm_scan: bad arguments");
    if (N > 256) return fail(B200SEQ_ERR_UNSUPPORTED, "ssm_scan: state size %d > 256", N);
    if (st->B == 0 || st->T == 0) return 0;
    cudaStream_t cs = (cudaStream_t)stream;
    SsmArgs a{proj, ldp, z0, dt0, xbc, ldx, A_log, Dp, dt_bias, state, nullptr, nullptr, out, H, V, N, G, 1, SSM_SEG};
    const bool small = N <= 16;
    const int npl = small ? 16 : 32;
    while (a.NL * npl < N) a.NL *= 2;
    const size_t need = b200seq_ssm_scratch_floats(st->T, st->B, H, V, N);
    cudaError_t e;
    if (need == 0 || !scratch || scratch_floats < need) {   // one launch: every entry's portion in order
        e = small ? ssm_launch<16, SSM_DIRECT>(a, *st, st->B, cs) : ssm_launch<32, SSM_DIRECT>(a, *st, st->B, cs);
        if (e != cudaSuccess) return cuda_status(e, "ssm_scan");
        count_launch();
        return 0;
    }
    const int segs = (st->T + SSM_SEG - 1) / SSM_SEG + st->B;   // upper bound of the step's segment count
    a.seg_state = scratch;
    a.seg_logdec = scratch + (size_t)segs * H * N * V;
    // tile products: 16-byte rows everywhere and a state of 33 .. 128 rows (smaller ones leave the 64-row tiles mostly empty)
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool tiles = N > 32 && N <= 128 && N % 4 == 0 && V % 4 == 0 && ((ldp | ldx | z0) & 3) == 0 && al(proj) && al(xbc) && al(state) && al(out) && al(scratch);
    const int vt = (V + ST_V - 1) / ST_V;
    if (tiles) {
        if (N <= 64) ssm_tile_local_kernel<1><<<dim3(vt, H, segs), ST_NT, 0, cs>>>(a, *st);
        else ssm_tile_local_kernel<2><<<dim3(vt, H, segs), ST_NT, 0, cs>>>(a, *st);
        e = cudaGetLastError();
    } else {
        e = small ? ssm_launch<16, SSM_LOCAL>(a, *st, segs, cs) : ssm_launch<32, SSM_LOCAL>(a, *st, segs, cs);
    }
    if (e != cudaSuccess) return cuda_status(e, "ssm_scan local pass");
    const int64_t per = (int64_t)H * N * V;
    if (tiles) ssm_combine_kernel<4><<<dim3((unsigned)((per / 4 + 255) / 256), st->B), 256, 0, cs>>>(a, *st);
    else ssm_combine_kernel<1><<<dim3((unsigned)((per + 255) / 256), st->B), 256, 0, cs>>>(a, *st);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e, "ssm_scan combine pass");
    if (tiles) {
        static bool ready[16] = {false};
        int dev = 0;
        e = cudaGetDevice(&dev);
        if (e == cudaSuccess && (dev >= 16 || !ready[dev])) {
            e = cudaFuncSetAttribute(ssm_tile_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileOut));
            if (e == cudaSuccess && dev < 16) ready[dev] = true;
        }
        if (e == cudaSuccess) {
            ssm_tile_out_kernel<<<dim3(vt, G * ((H / G + SSM_HB - 1) / SSM_HB), segs), 2 * ST_NT, sizeof(TileOut), cs>>>(a, *st);
            e = cudaGetLastError();
        }
    } else {
        e = small ? ssm_launch<16, SSM_FINAL>(a, *st, segs, cs) : ssm_launch<32, SSM_FINAL>(a, *st, segs, cs);
    }
    if (e != cudaSuccess) return cuda_status(e, "ssm_scan final pass");
    count_launch(3);
    return 0;
}
