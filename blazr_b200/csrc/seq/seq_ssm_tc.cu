// seq_ssm_tc.cu -- passes A and C of the state-space scan (seq_ssm.cu) as products of tiles on the tensor cores, at 32-bit accuracy.
//
// Over a segment of up to SSM_SEG tokens with step sizes dt and L_t the sum of the log-decays up to and including t:
//     E        = sum_s B_s (dt_s exp(L_end - L_s) x_s)^T                                                     [N x V]   (pass A)
//     y_t      = exp(L_t) C_t^T S_start + sum_(s <= t) (C_t . B_s) exp(L_t - L_s) dt_s x_s                    [V]      (pass C)
// All four products are contractions of 128 x 128 by 128 x 64 (per head) or 128 (per group).  Every f32 operand is split into three bf16 parts and a
// product runs as six (tc_split.cuh).  The leading one (x1 y1) has accumulators of its own and the five small ones share another; they are added in
// registers.  Products of 8-bit parts leave room in 24 bits, so a short leading sum loses little to the tensor core's truncation, and what the small
// ones lose is 2^-8 of that.  Sums of values that have one sign more often than not grow with every step and drop bits of what they add: those of C . B
// are cut into steps of 16, the others into 32.  Error against 64 bits, 4096 tokens of 64 heads:
// outputs 1.14e-7, states 9.3e-8 (f32 multiply-add tiles: 1.14e-7, 8.8e-8; with one accumulator for each of the leading and the small products 1.6e-7).
// Decays are exponentials of differences of the sums (never above 1), the sums kept as a float pair of the f64 running sum, so that a difference late in
// the segment is as exact as an early one.
//
// A CTA has one segment, 64 value columns and some heads of one group, one after another: what depends on the group alone (B, C, C_t . B_s) is made once.
// 512 threads split, exponentiate and store; a warp of its own issues the products, which run beside the next step of that work:
//   pass A   x (dt exp) -> planes -> E = (B planes in TMEM) x (x planes);               beside it: the head before leaves
//   pass C   S planes -> C S;                          beside it: the head before leaves, the weights -> TMEM, dt x -> planes
//            weights x (x planes);                     beside it: exp(L) C S, the next head's S planes
// Weights above the diagonal are zeros (a block of 16 x 32 that lies there is not computed).
//
// Values without bf16 parts (infinities, NaN, beyond the bf16 range) leave a NaN in every sum that meets them, also in rows that do not see their token
// (0 x inf).  A head whose tile has a result that is not finite is made again token by token (recur_head), or by plain sums over the tokens (pass A).
// Every wait is bounded (tc_pair.cuh): one that runs out sets bit 1 of the library's error flags and the CTA leaves through the common exit.
#include "seq_ssm.cuh"
#include "tc_split.cuh"

namespace b200seq {

namespace {

using namespace tcsplit;

constexpr int TV = 64;                        // value columns of a tile
constexpr int TPL = 128 * 128;                // bytes of a plane: 128 rows of 64 bf16, 128-byte swizzle
constexpr int XPL = 3 * TPL;                  // a group's planes of x or S
constexpr int YLD = TV + 4;                   // floats of a row of results in shared memory (over the planes)
constexpr int MAX_HB = 8;                     // heads of a CTA
constexpr double LOG2E_D = 1.4426950408889634;

struct alignas(16) Decay {
    float dt[SSM_SEG];                             // step size
    float nhi[SSM_SEG], nlo[SSM_SEG];              // minus log2 of the decay from the segment's start, as a pair
    float w[SSM_SEG];                              // pass A: dt exp(L_end - L_t); pass C: exp(L_t)
    float in[SSM_SEG];                             // pass C: exp(L_t - L at the last token before t's block of 32)
    float from[3 * SSM_SEG];                       // pass C: [b][s] exp(L at the last token before block b + 1 - L_s), s before that block
    float end;                                     // sum of the log-decays of the whole segment
};
constexpr int WORKERS = 512, THREADS_SSM = WORKERS + 128;   // launched with 96 registers each; the workers take 112, the issuer's warpgroup keeps 32 (4 * 112 + 32 = 5 * 96)
struct Shared {
    double part[16];
    __align__(8) uint64_t bars[5];                 // products done (2), operands in place (2, one arrival per warp), the last one
    uint32_t tmem;
    int abort;
    int odd[2];
};

__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ bool worker_any(bool mine) {   // the same barrier; true for all when it is for one
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 1, 512, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((int)mine) : "memory");
    return any != 0;
}
// this thread's part of the operands (shared memory and TMEM) is in place, and what it read of the accumulators has been read
__device__ __forceinline__ void hand_over(uint32_t bar) {
    async_fence();
    fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) bar_arrive(bar);
}

// Decays of a segment for the heads h0 .. h1 - 1, four heads at a time (128 threads each, a thread = a token).  Tokens beyond the segment: dt 0, the last sum.
template <bool LOCAL>
__device__ __forceinline__ void seg_decays(Decay* dec, double* part, const SsmArgs& a, int row0, int len, int h0, int h1) {
    const int sub = threadIdx.x >> 7, t = threadIdx.x & 127, lane = t & 31;
    float raw[MAX_HB / 4];
#pragma unroll
    for (int i = 0; i < MAX_HB / 4; ++i) raw[i] = t < len && h0 + 4 * i + sub < h1 ? a.proj[(int64_t)(row0 + t) * a.ldp + a.dt0 + h0 + 4 * i + sub] : 0.f;
#pragma unroll
    for (int i = 0; i < MAX_HB / 4; ++i) {
        const int h = h0 + 4 * i + sub;
        if (h0 + 4 * i >= h1) break;
        const bool live = t < len && h < h1;
        const float dt = live ? softplusf_acc(raw[i] + a.dt_bias[h]) : 0.f;
        const float ld = live ? -expf(a.A_log[h]) * dt : 0.f;
        double L = ld < -200.f ? -200.0 : (double)ld;   // exp of either is 0 in f32; a sum of infinite terms would have no differences
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, L, o);
            if (lane >= o) L += u;
        }
        if (lane == 31) part[threadIdx.x >> 5] = L;
        worker_sync();
        const float within = (float)L;
        double end = 0.0, before[4];   // of the block of 32 tokens
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            before[w] = end;
            if (w < (t >> 5)) L += part[4 * sub + w];
            end += part[4 * sub + w];
        }
        if (h < h1) {
            Decay& d = dec[4 * i + sub];
            const double l2 = L * LOG2E_D;
            const float hi = (float)l2;
            d.dt[t] = dt, d.nhi[t] = -hi, d.nlo[t] = -(float)(l2 - (double)hi);
            d.w[t] = LOCAL ? dt * expf((float)(end - L)) : expf((float)L);
            if (!LOCAL) {
                d.in[t] = expf(within);
#pragma unroll
                for (int b = 0; b < 3; ++b)
                    if (t < 32 * (b + 1)) d.from[b * SSM_SEG + t] = expf((float)(before[b + 1] - L));
            }
            if (t == 0) d.end = (float)end;
        }
        worker_sync();
    }
}

// rows r0 + 32 i of four floats each, scaled -> the planes at U; rows from `rows` on (a multiple of 16) are not needed
template <class Scale>
__device__ __forceinline__ void stage_planes(uint32_t U, int rows, const float4 (&x)[4], Scale scale) {
    const int r0 = threadIdx.x >> 4, c = threadIdx.x & 15;
    uint32_t at = U + r0 * 128 + (((c >> 1) ^ (r0 & 7)) << 4) + ((c & 1) << 3);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (r0 + 32 * i < rows) {
            const float s = scale(r0 + 32 * i);
            uint32_t a1, a2, a3, b1, b2, b3;
            split2(x[i].x * s, x[i].y * s, a1, a2, a3);
            split2(x[i].z * s, x[i].w * s, b1, b2, b3);
            sts8(at, a1, b1), sts8(at + TPL, a2, b2), sts8(at + 2 * TPL, a3, b3);
        }
        at += 4096;
    }
}
// rows r0 + 32 i (below `rows`) of the 64 columns of a matrix; columns from V on are zero
__device__ __forceinline__ void load_rows(float4 (&x)[4], const float* base, int64_t ld, int rows, bool in) {
    const int r0 = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = in && r0 + 32 * i < rows ? ld4(base + (int64_t)(r0 + 32 * i) * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// tokens x states of B or C -> planes [token][n], 64 n to a block (three planes), by the 512 threads
__device__ __forceinline__ void stage_states(uint32_t dst, const float* src, int64_t ld, int len, int N) {
    const int r0 = threadIdx.x >> 5, c = threadIdx.x & 31, cc = c & 15;
    const uint32_t at = dst + (c >> 4) * XPL + r0 * 128 + (((cc >> 1) ^ (r0 & 7)) << 4) + ((cc & 1) << 3);
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = r0 + 16 * i;
        x[i] = t < len && 4 * c < N ? ld4(src + (int64_t)t * ld + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint32_t a1, a2, a3, b1, b2, b3;
        split2(x[i].x, x[i].y, a1, a2, a3);
        split2(x[i].z, x[i].w, b1, b2, b3);
        sts8(at + i * 2048, a1, b1), sts8(at + i * 2048 + TPL, a2, b2), sts8(at + i * 2048 + 2 * TPL, a3, b3);
    }
}

constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24);   // bf16 x bf16 -> f32, M = 128
constexpr uint32_t IDESC_G = IDESC | ((uint32_t)(SSM_SEG >> 3) << 17), IDESC_V = IDESC | (1u << 16) | ((uint32_t)(TV >> 3) << 17);   // (V: B is mn-major)

// the six products of one contraction, `steps` of 16 deep: issue(product, plane of A, plane of B, step); the last one is the leading product
template <class Issue>
__device__ __forceinline__ void six_products(int steps, Issue issue) {
    constexpr int PX[6] = {0, 2, 1, 0, 1, 0}, PY[6] = {2, 0, 1, 1, 0, 0};   // smallest first
#pragma unroll
    for (int pr = 0; pr < 6; ++pr)
#pragma unroll 1
        for (int kk = 0; kk < steps; ++kk) issue(pr, PX[pr], PY[pr], kk);
}

struct Segment {
    int e, row0, len;
};
// one: the entry's whole portion is the segment
__device__ __forceinline__ bool find(const SsmArgs& a, const b200seq_step& st, bool one, Segment& s) {
    if (!one) return ssm_find_segment(st, blockIdx.z, a.seg_len, s.e, s.row0, s.len);
    s.e = blockIdx.z, s.row0 = st.ent_start[s.e], s.len = st.ent_start[s.e + 1] - s.row0;
    return true;
}

__device__ __forceinline__ uint32_t enter(Shared& sh) {   // barriers and TMEM; all threads
    if (threadIdx.x == 0) {
        for (int i = 0; i < 5; ++i) bar_init(sa(&sh.bars[i]), i == 2 || i == 3 ? WORKERS / 32 : 1);
        sh.abort = 0, sh.odd[0] = sh.odd[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(sa(&sh.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    return sh.tmem;
}
__device__ __forceinline__ void leave(Shared& sh, uint32_t tmem, int* err) {
    fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        if (sh.abort && elect()) {   // what was issued reads shared memory and TMEM: wait for it (bounded) before the CTA goes
            const uint32_t last = sa(&sh.bars[4]);
            commit_one(last);
            const unsigned long long t0 = now_ns();
            while (!bar_try<false>(last, 0) && now_ns() - t0 < WAIT_NS) {}
            atomicOr(err, 2);
        }
        __syncwarp();
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// the accumulators of a product of 64 columns: the leading product in steps of 32, four of them, and the small ones
__device__ __forceinline__ uint32_t acc_of(uint32_t D, int pr, int kk) { return D + (pr == 5 ? 64 * (kk >> 1) : 256); }
__device__ __forceinline__ uint32_t acc_adds(int pr, int kk) { return pr == 5 ? (uint32_t)(kk & 1) : ((pr | kk) != 0 ? 1u : 0u); }
// acc += (or =) the five accumulators of 64 columns, the small products first; parts of the leading one that do not exist are left out
template <bool FRESH>
__device__ __forceinline__ void add_parts(float (&y)[16], uint32_t D, int steps) {
    float u[16];
    ld16(D + 256, u);
    ld_wait();
    float sum[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) sum[i] = u[i];
#pragma unroll
    for (int part = 0; part < 4; ++part) {
        if (2 * part >= steps) break;
        ld16(D + 64 * part, u);
        ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] += u[i];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = FRESH ? sum[i] : y[i] + sum[i];
}

// pass A: grid (V / 64, group x head blocks, segments).  TMEM: B^T planes (lane = n, column = token pair) 3 x 64, then the five accumulators
template <bool ONE>
__global__ void __launch_bounds__(THREADS_SSM, 1) ssm_tc_local_kernel(const __grid_constant__ SsmArgs a, const __grid_constant__ b200seq_step st, int hb, int* err) {
    extern __shared__ uint8_t raw[];
    __shared__ Shared sh;
    Segment s;
    if (!find(a, st, ONE, s)) return;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, q = warp & 3, wg = warp >> 2;
    const int N = a.N, V = a.V, H = a.H, v0 = blockIdx.x * TV, per = H / a.G, nb = (per + hb - 1) / hb, inner = H * V;
    const int g = blockIdx.y / nb, h_first = g * per + (blockIdx.y % nb) * hb, h_end = min(h_first + hb, (g + 1) * per);
    const int len = s.len, steps = (len + 15) >> 4;
    uint8_t* planes = raw + ((1024u - (sa(raw) & 1023u)) & 1023u);
    Decay* decs = reinterpret_cast<Decay*>(planes + 2 * XPL);
    const uint32_t U = sa(planes);
    volatile int* ab = &sh.abort;
    const uint32_t tmem = enter(sh), lanes = (uint32_t)(q * 32) << 16;
    const uint32_t done = sa(&sh.bars[0]), ready = sa(&sh.bars[2]);   // two each: even and odd heads
    if (warp >= WORKERS / 32) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == WORKERS / 32 && elect()) {
            for (int k = 0; k < h_end - h_first; ++k) {
                const int p = k & 1;
                if (!bar_wait<false>(ready + 8 * p, (k >> 1) & 1, ab)) break;
                fence_after();
                const uint64_t xd = desc_mn128(U + p * XPL, 0);
                six_products(steps, [&](int pr, int pa, int pb, int kk) {
                    mma_ts(acc_of(tmem + 192, pr, kk), tmem + pa * 64 + kk * 8, xd + (uint64_t)((pb * TPL + kk * 2048) / 16), IDESC_V, acc_adds(pr, kk));
                });
                commit_one(done + 8 * p);
            }
        }
        __syncwarp();
        leave(sh, tmem, err);
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const int n = q * 32 + lane, r0 = tid >> 4, c = (tid & 15) * 4;
    const bool in = v0 + c < V;
    const float* bb = a.xbc + (int64_t)s.row0 * a.ldx + inner + (int64_t)g * N;
    const float* xg = a.xbc + (int64_t)s.row0 * a.ldx + v0;
    float4 x[4];
    load_rows(x, xg + (int64_t)h_first * V, a.ldx, len, in);
    seg_decays<true>(decs, sh.part, a, s.row0, len, h_first, h_end);
    {   // B^T: 32 tokens per thread
        const int t0 = 32 * wg;
#pragma unroll 1
        for (int u = 0; u < 32; u += 16) {
            float b[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) b[i] = t0 + u + i < len && n < N ? bb[(int64_t)(t0 + u + i) * a.ldx + n] : 0.f;
            uint32_t p1[8], p2[8], p3[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) split2(b[2 * i], b[2 * i + 1], p1[i], p2[i], p3[i]);
            const uint32_t at = tmem + lanes + ((t0 + u) >> 1);
            st8(at, p1), st8(at + 64, p2), st8(at + 128, p3);
        }
        st_wait();
    }
    bool bad = false;
    float E[16];
    auto sums = [&](int h) {   // head h: its sums of this thread's state row n
        bad |= !bar_wait<false>(done + 8 * ((h - h_first) & 1), ((h - h_first) >> 1) & 1, ab);
        fence_after();
        add_parts<true>(E, tmem + lanes + 192 + 16 * wg, steps);
    };
    auto store = [&](int h) {   // -> the segment's state
        const int p = (h - h_first) & 1;
        const Decay& dec = decs[h - h_first];
        bool odd = false;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (steps == 0) E[i] = 0.f;
            odd |= !isfinite(E[i]);
        }
        if (__any_sync(0xffffffffu, odd)) {   // plain sums over the tokens
#pragma unroll
            for (int i = 0; i < 16; ++i) E[i] = 0.f;
            if (n < N) {
#pragma unroll 1
                for (int t = 0; t < len; ++t) {
                    const float b = bb[(int64_t)t * a.ldx + n], w = dec.w[t];
                    const float* xr = xg + (int64_t)t * a.ldx + (int64_t)h * V + 16 * wg;
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (v0 + 16 * wg + i < V) E[i] = fmaf(b, xr[i] * w, E[i]);
                }
            }
        }
        float* Y = reinterpret_cast<float*>(planes + p * XPL);   // the rows leave through shared memory (the planes have been read), 256 consecutive bytes at a time
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(&Y[n * YLD + 16 * wg + i]) = make_float4(E[i], E[i + 1], E[i + 2], E[i + 3]);
        worker_sync();
        float* dst = (ONE ? a.state + ((int64_t)st.ent_slot[s.e] * H + h) * N * V : a.seg_state + ((int64_t)blockIdx.z * H + h) * N * V) + v0 + c;
        const bool carried = ONE && st.ent_pos0[s.e] != 0;
        const float keep = carried ? expf(dec.end) : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + 32 * i;
            if (in && r < N) {
                float4 y = *reinterpret_cast<const float4*>(&Y[r * YLD + c]);
                float4* o = reinterpret_cast<float4*>(dst + (int64_t)r * V);
                if (carried) {
                    const float4 old = *o;
                    y.x = fmaf(keep, old.x, y.x), y.y = fmaf(keep, old.y, y.y), y.z = fmaf(keep, old.z, y.z), y.w = fmaf(keep, old.w, y.w);
                }
                *o = y;
            }
        }
        if (!ONE && tid == 0 && blockIdx.x == 0) a.seg_logdec[(int64_t)blockIdx.z * H + h] = dec.end;
    };
#pragma unroll 1
    for (int h = h_first; h < h_end; ++h) {
        const int p = (h - h_first) & 1;
        const Decay& dec = decs[h - h_first];
        stage_planes(U + p * XPL, 16 * steps, x, [&](int t) { return dec.w[t]; });
        if (h > h_first) sums(h - 1);
        hand_over(ready + 8 * p);
        if (h + 1 < h_end) load_rows(x, xg + (int64_t)(h + 1) * V, a.ldx, len, in);
        if (h > h_first) store(h - 1);
        if (worker_any(bad)) break;
    }
    if (!worker_any(bad)) {
        sums(h_end - 1);
        store(h_end - 1);
    }
    leave(sh, tmem, err);
}

// One head of a segment token by token, 64 value columns by 512 threads: thread = column, 16 states.  part: [8][64] floats of shared memory
__device__ __noinline__ void recur_head(const SsmArgs& a, int row0, int len, int g, int h, int v0, const float* init, float* part) {
    const int N = a.N, V = a.V, inner = a.H * V, vc = threadIdx.x & 63, sub = threadIdx.x >> 6, v = v0 + vc;
    const float negA = -expf(a.A_log[h]), Dh = a.Dp[h];
    float S[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) S[i] = init && v < V && sub * 16 + i < N ? init[(int64_t)(sub * 16 + i) * V + v] : 0.f;
    worker_sync();
#pragma unroll 1
    for (int t = 0; t < len; ++t) {
        const float* xr = a.xbc + (int64_t)(row0 + t) * a.ldx;
        const float* pr = a.proj + (int64_t)(row0 + t) * a.ldp;
        const float* b = xr + inner + (int64_t)g * N + sub * 16;
        const float dt = softplusf_acc(pr[a.dt0 + h] + a.dt_bias[h]), dA = expf(negA * dt), x = v < V ? xr[(int64_t)h * V + v] : 0.f, dtx = dt * x;
        float y = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (sub * 16 + i < N) {
                S[i] = fmaf(dA, S[i], dtx * b[i]);
                y = fmaf(S[i], b[(int64_t)a.G * N + i], y);
            }
        part[sub * 64 + vc] = y;
        worker_sync();
        if (sub == 0 && v < V) {
            y = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) y += part[i * 64 + vc];
            a.out[(int64_t)(row0 + t) * inner + (int64_t)h * V + v] = fmaf(Dh, x, y) * siluf_acc(pr[a.z0 + (int64_t)h * V + v]);
        }
        worker_sync();
    }
}

__device__ __forceinline__ float max_nan(float a, float b) {   // NaN if either is
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// 2^a and 2^b for arguments up to 0, NaN for NaN (what lies above is not used): to the nearest whole number by the addition of 1.5 2^23, then 1 + f q(f) with a
// polynomial of degree 5 (fitted by iterated weighted least squares on |f| <= 1/2: 2e-9 of the result), at half the instructions of two expf calls and
// closer to 64 bits than ex2.approx, whose errors alone made the outputs' 1.2e-7 to 1.4e-7
__device__ __forceinline__ uint64_t exp2_pair(uint64_t u) {
    float a, b;
    upk(u, a, b);
    u = pk(max_nan(a, -127.f), max_nan(b, -127.f));
    constexpr float MAGIC = 12582912.f;
    const uint64_t j = add2(u, pk(MAGIC, MAGIC)), f = fma2(add2(j, pk(-MAGIC, -MAGIC)), pk(-1.f, -1.f), u);
    uint64_t q = pk(0x1.41fbbcp-13f, 0x1.41fbbcp-13f);
    q = fma2(q, f, pk(0x1.5f3e52p-10f, 0x1.5f3e52p-10f));
    q = fma2(q, f, pk(0x1.3b2d4cp-7f, 0x1.3b2d4cp-7f));
    q = fma2(q, f, pk(0x1.c6aee8p-5f, 0x1.c6aee8p-5f));
    q = fma2(q, f, pk(0x1.ebfbdcp-3f, 0x1.ebfbdcp-3f));
    q = fma2(q, f, pk(0x1.62e430p-1f, 0x1.62e430p-1f));
    q = fma2(q, f, pk(1.f, 1.f));
    upk(j, a, b);
    return mul2(q, pk(__int_as_float((__float_as_int(a) << 23) + 0x3f800000), __int_as_float((__float_as_int(b) << 23) + 0x3f800000)));   // (2^-127: 0)
}

// pass C: grid (V / 64, group x head blocks, segments).  Shared memory: C's planes, S's planes, x's planes (at first the latter two hold B's).
// TMEM: five accumulators (the leading product in steps of 32, the small ones) for C S and then for the weights' product, three planes of weights; at
// first C . B, three times: the leading product's steps of 16, four at a time, then the small ones.
template <bool ONE>
__global__ void __launch_bounds__(THREADS_SSM, 1) ssm_tc_out_kernel(const __grid_constant__ SsmArgs a, const __grid_constant__ b200seq_step st, int hb, int* err) {
    extern __shared__ uint8_t raw[];
    __shared__ Shared sh;
    Segment s;
    if (!find(a, st, ONE, s) || s.len == 0) return;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, q = warp & 3, wg = warp >> 2;
    const int N = a.N, V = a.V, H = a.H, v0 = blockIdx.x * TV, per = H / a.G, nb = (per + hb - 1) / hb, inner = H * V;
    const int g = blockIdx.y / nb, h_first = g * per + (blockIdx.y % nb) * hb, h_end = min(h_first + hb, (g + 1) * per);
    const int len = s.len, nk = (N + 15) >> 4, steps = (len + 15) >> 4;
    uint8_t* base = raw + ((1024u - (sa(raw) & 1023u)) & 1023u);
    const uint32_t Cp = sa(base), Sp = Cp + 2 * XPL, Xp = Cp + 3 * XPL;
    float* Y = reinterpret_cast<float*>(base + 3 * XPL);
    Decay* decs = reinterpret_cast<Decay*>(base + 4 * XPL);
    volatile int* ab = &sh.abort;
    const uint32_t done_s = sa(&sh.bars[0]), done_x = sa(&sh.bars[1]), ready_s = sa(&sh.bars[2]), ready_x = sa(&sh.bars[3]);
    const uint32_t tmem = enter(sh), lanes = (uint32_t)(q * 32) << 16, W = tmem + 320;
    auto start_of = [&](int h) -> const float* {
        if (!ONE) return a.seg_state + ((int64_t)blockIdx.z * H + h) * N * V + v0;
        return st.ent_pos0[s.e] != 0 ? a.state + ((int64_t)st.ent_slot[s.e] * H + h) * N * V + v0 : nullptr;
    };
    const bool carried = start_of(h_first) != nullptr;
    if (warp >= WORKERS / 32) {
        // ===================== issuer =====================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == WORKERS / 32 && elect()) {
            const uint64_t cd = desc_k128(Cp), bd = desc_k128(Sp), sd = desc_mn128(Sp, 0), xd = desc_mn128(Xp, 0);
            auto groups = [&](int pr, int pa, int pb, int kk) {
                const uint64_t at = (uint64_t)((kk >> 2) * XPL / 16 + 2 * (kk & 3));
                mma_ss(pr == 5 ? tmem + 128 * (kk & 3) : tmem, cd + at + (uint64_t)(pa * TPL / 16), bd + at + (uint64_t)(pb * TPL / 16), IDESC_G, pr < 5 && (pr | kk) != 0 ? 1u : 0u);
            };
            bool ok = bar_wait<false>(ready_s, 0, ab);
            if (ok) {
                fence_after();
                for (int kk = 0; kk < min(nk, 4); ++kk) groups(5, 0, 0, kk);
                commit_one(done_s);
                ok = bar_wait<false>(ready_x, 0, ab);
            }
            if (ok) {
                fence_after();
                for (int kk = 4; kk < nk; ++kk) groups(5, 0, 0, kk);
                commit_one(done_x);
                ok = bar_wait<false>(ready_s, 1, ab);
            }
            if (ok) {
                fence_after();
                six_products(nk, [&](int pr, int pa, int pb, int kk) {
                    if (pr < 5) groups(pr, pa, pb, kk);
                });
                commit_one(done_s);
            }
            for (int k = 0; k < h_end - h_first && ok; ++k) {
                if (carried) {
                    ok = bar_wait<false>(ready_s, k & 1, ab);
                    if (!ok) break;
                    fence_after();
                    six_products(nk, [&](int pr, int pa, int pb, int kk) {
                        mma_ss(acc_of(tmem, pr, kk), cd + (uint64_t)(((kk >> 2) * XPL + pa * TPL) / 16 + 2 * (kk & 3)), sd + (uint64_t)((pb * TPL + kk * 2048) / 16), IDESC_V, acc_adds(pr, kk));
                    });
                    commit_one(done_s);
                }
                ok = bar_wait<false>(ready_x, (k + 1) & 1, ab);
                if (!ok) break;
                fence_after();
                six_products(steps, [&](int pr, int pa, int pb, int kk) {
                    mma_ts(acc_of(tmem, pr, kk), W + pa * 64 + kk * 8, xd + (uint64_t)((pb * TPL + kk * 2048) / 16), IDESC_V, acc_adds(pr, kk));
                });
                commit_one(done_x);
            }
        }
        __syncwarp();
        leave(sh, tmem, err);
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const int t = q * 32 + lane;                 // this thread's token in the products, and there its 16 columns from 16 wg on
    const int r0 = tid >> 4, c = (tid & 15) * 4; // its rows r0 + 32 i and columns of what is loaded and stored
    const bool in = v0 + c < V;
    const float* bb = a.xbc + (int64_t)s.row0 * a.ldx + inner + (int64_t)g * N;
    const float* xg = a.xbc + (int64_t)s.row0 * a.ldx + v0;
    const float* zg = a.proj + (int64_t)s.row0 * a.ldp + a.z0 + v0;
    bool bad = false;
    stage_states(Cp, bb + (int64_t)a.G * N, a.ldx, len, N);
    stage_states(Sp, bb, a.ldx, len, N);
    hand_over(ready_s);
    float4 R[4], x[4], z[4];   // R: what is staged next, S or x
    asm volatile("griddepcontrol.wait;" ::: "memory");   // what lies above needs the step's inputs only and runs beside the pass before; the states are complete from here on
    load_rows(R, start_of(h_first), V, carried ? N : 0, in);
    float G[32];   // C_t . B_s of the tokens s = 16 (4 j + wg) + i
    auto group_sums = [&](int part, bool fresh) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float u[16];
            ld16(tmem + lanes + 128 * part + 16 * (4 * j + wg), u);
            ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) G[16 * j + i] = fresh ? u[i] : G[16 * j + i] + u[i];
        }
    };
    bad |= !bar_wait<false>(done_s, 0, ab);
    fence_after();
    group_sums(0, true);
#pragma unroll 1
    for (int part = 1; part < 4 && part < nk; ++part) group_sums(part, false);
    hand_over(ready_x);
    bad |= !bar_wait<false>(done_x, 0, ab);
    fence_after();
#pragma unroll 1
    for (int part = 0; part + 4 < nk; ++part) group_sums(part, false);
    hand_over(ready_s);
    seg_decays<false>(decs, sh.part, a, s.row0, len, h_first, h_end);
    bad |= !bar_wait<false>(done_s, 1, ab);
    fence_after();
    group_sums(0, false);
    if (carried) {   // (each thread has seen the tensor core done with B's planes)
        stage_planes(Sp, 16 * nk, R, [](int) { return 1.f; });
        hand_over(ready_s);
    }
    load_rows(R, xg + (int64_t)h_first * V, a.ldx, len, in);
    float y[16];
#pragma unroll 1
    for (int h = h_first; h <= h_end; ++h) {
        // here: S's planes of this head are handed over, the results of the head before are in place
        const int k = h - h_first, p = k & 1;
        if (worker_any(bad)) break;
        const Decay& dec = decs[min(h, h_end - 1) - h_first];
        if (h > h_first) {   // the head before leaves
            const int hp = h - 1;
            if (sh.odd[p ^ 1]) {
                recur_head(a, s.row0, len, g, hp, v0, start_of(hp) ? start_of(hp) - v0 : nullptr, Y);
                worker_sync();
                if (tid == 0) sh.odd[p ^ 1] = 0;
            } else if (in) {
                const float Dh = a.Dp[hp];
                float* ob = a.out + (int64_t)s.row0 * inner + (int64_t)hp * V + v0 + c;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = r0 + 32 * i;
                    if (r < len) {
                        const float4 o = *reinterpret_cast<const float4*>(&Y[r * YLD + c]);
                        *reinterpret_cast<float4*>(ob + (int64_t)r * inner) = make_float4(fmaf(Dh, x[i].x, o.x) * siluf_acc(z[i].x), fmaf(Dh, x[i].y, o.y) * siluf_acc(z[i].y),
                                                                                          fmaf(Dh, x[i].z, o.z) * siluf_acc(z[i].z), fmaf(Dh, x[i].w, o.w) * siluf_acc(z[i].w));
                    }
                }
            }
            if (h == h_end) break;
        }
        load_rows(z, zg + (int64_t)h * V, a.ldp, len, in);
        {   // the weights exp(L_t - L_s) C_t . B_s -> TMEM
            const float thi = -dec.nhi[t], tlo = -dec.nlo[t], own = dec.in[t];
            const uint64_t minus1 = pk(-1.f, -1.f), thi2 = pk(thi, thi), tlo2 = pk(tlo, tlo);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int kk = 4 * j + wg, s0 = 16 * kk;
                if (kk >= steps) break;
                uint32_t p1[8], p2[8], p3[8];
                if (s0 > 32 * q + 31) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) p1[i] = p2[i] = p3[i] = 0;
                } else {
                    if (s0 < 32 * q) {   // all before the warp's 32 tokens: the decay in two parts, each made once
                        const uint64_t own2 = pk(own, own);
                        const float* from = dec.from + (q - 1) * SSM_SEG + s0;
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            float u, v;
                            upk(mul2(mul2(own2, *reinterpret_cast<const uint64_t*>(from + i)), pk(G[16 * j + i], G[16 * j + i + 1])), u, v);
                            cut2(u, v, minus1, p1[i >> 1], p2[i >> 1], p3[i >> 1]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            float u, v;
                            const uint64_t diff = add2(add2(thi2, *reinterpret_cast<const uint64_t*>(&dec.nhi[s0 + i])), add2(tlo2, *reinterpret_cast<const uint64_t*>(&dec.nlo[s0 + i])));
                            upk(mul2(exp2_pair(diff), pk(G[16 * j + i], G[16 * j + i + 1])), u, v);
                            u = s0 + i <= t ? u : 0.f, v = s0 + i + 1 <= t ? v : 0.f;
                            cut2(u, v, minus1, p1[i >> 1], p2[i >> 1], p3[i >> 1]);
                        }
                    }
                }
                const uint32_t at = W + lanes + 8 * kk;
                st8(at, p1), st8(at + 64, p2), st8(at + 128, p3);
            }
            st_wait();
        }
        worker_sync();   // the results of the head before have been read
        stage_planes(Xp, 16 * steps, R, [&](int r) { return dec.dt[r]; });
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = R[i];
        const bool more = h + 1 < h_end;
        if (more && carried) load_rows(R, start_of(h + 1), V, N, in);
        if (carried) {
            bad |= !bar_wait<false>(done_s, k & 1, ab);
            fence_after();
            add_parts<true>(y, tmem + lanes + 16 * wg, nk);
            const float f = dec.w[t];
#pragma unroll
            for (int i = 0; i < 16; ++i) y[i] *= f;
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) y[i] = 0.f;
        }
        hand_over(ready_x);
        if (more && carried) stage_planes(Sp, 16 * nk, R, [](int) { return 1.f; });   // (the tensor core is done with this head's S)
        if (more) load_rows(R, xg + (int64_t)(h + 1) * V, a.ldx, len, in);
        bad |= !bar_wait<false>(done_x, (k + 1) & 1, ab);
        fence_after();
        add_parts<false>(y, tmem + lanes + 16 * wg, steps);
        bool odd = false;
#pragma unroll
        for (int i = 0; i < 16; ++i) odd |= t < len && !isfinite(y[i]);
        if (odd) sh.odd[p] = 1;
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(&Y[t * YLD + 16 * wg + i]) = make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]);
        if (more && carried) hand_over(ready_s);
    }
    leave(sh, tmem, err);
}

// Heads per CTA: the least waves of (set-up + heads).  Setting up a CTA of pass C (B, C, C . B: 22 k cycles) costs as much as 1.4 heads (15 k each).
int heads_per_cta(const SsmArgs& a, int segs, int vt) {
    const int per = a.H / a.G, sms = pair_sms();
    int best = 1;
    double best_t = 0;
    for (int hb = per < MAX_HB ? per : MAX_HB; hb >= 1; --hb) {
        const int64_t ctas = (int64_t)vt * a.G * ((per + hb - 1) / hb) * segs;
        const double t = (double)((ctas + sms - 1) / sms) * (1.4 + hb);
        if (best_t == 0 || t < best_t) best = hb, best_t = t;
    }
    return best;
}

template <class Kernel>
cudaError_t run(Kernel kern, int smem, bool (&ready)[16], const SsmArgs& a, const b200seq_step& st, int segs, bool early, cudaStream_t cs) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 16 || !ready[dev]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev < 16) ready[dev] = true;
    }
    const int vt = (a.V + TV - 1) / TV, per = a.H / a.G;
    const int hb = heads_per_cta(a, st.T > SSM_SEG ? (st.T + SSM_SEG - 1) / SSM_SEG + st.B - 1 : segs, vt);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(vt, a.G * ((per + hb - 1) / hb), segs), cfg.blockDim = dim3(THREADS_SSM), cfg.dynamicSmemBytes = smem, cfg.stream = cs;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization, attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = early ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kern, a, st, hb, error_flag_dev());
    return e != cudaSuccess ? e : cudaGetLastError();
}

constexpr int SMEM_LOCAL = 136 * 1024;       // the planes of two heads; one CTA per SM: it takes all of TMEM
constexpr int SMEM_OUT = 4 * XPL + MAX_HB * (int)sizeof(Decay) + 1024;
static_assert(2 * XPL + MAX_HB * sizeof(Decay) + 1024 <= SMEM_LOCAL && 128 * YLD * 4 <= XPL, "results fit over the planes");

}  // namespace

cudaError_t launch_ssm_tiles_local(const SsmArgs& a, const b200seq_step& st, int segs, bool one, cudaStream_t cs) {
    static bool ready[2][16] = {};
    return one ? run(ssm_tc_local_kernel<true>, SMEM_LOCAL, ready[1], a, st, segs, false, cs) : run(ssm_tc_local_kernel<false>, SMEM_LOCAL, ready[0], a, st, segs, false, cs);
}
cudaError_t launch_ssm_tiles_out(const SsmArgs& a, const b200seq_step& st, int segs, bool one, cudaStream_t cs) {
    static bool ready[2][16] = {};
    return one ? run(ssm_tc_out_kernel<true>, SMEM_OUT, ready[1], a, st, segs, false, cs) : run(ssm_tc_out_kernel<false>, SMEM_OUT, ready[0], a, st, segs, true, cs);
}

}  // namespace b200seq
