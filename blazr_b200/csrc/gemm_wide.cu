// gemm_wide.cu -- dequant-GEMM of large steps (prompts): the weight is expanded ONCE per call, panel by panel, into f16 rows that the
// paired-SM GEMM (seq/tc_pair.cuh) reads by TMA.
//
// The fused kernel (gemm_impl.cuh) expands a weight tile again for every 256 token rows, in the same warps that feed the tensor pipe: at
// 2048 tokens that is eight times the expansion work, and the pipe was active for half of the time.  Here the expansion costs one pass
// (2 bytes per weight written to and read from L2) and runs beside the GEMM of the panel before:
//     stage x -> f16 rows;   [expand panel p -> buffer p % 2;   GEMM of panel p]  for all p
// as one chain of programmatic launches.  The GEMM of panel p lets the expansion of panel p + 1 start as soon as its own operands are
// complete; the expansion waits for that GEMM at its end, so buffer p % 2 is free again when panel p + 2 is expanded.
// Same operands (f16 roundings of weights and activations), the same order of k and the same cuts of it as the fused kernel: the same results, bit for bit.
#include "gemm_impl.cuh"
#include "seq/tc_pair.cuh"

namespace b200q {

// x[M, K] (f32 / f16 / bf16, columns gathered through perm) -> f16 rows [M][K_pad], clamped to the f16 range, zero beyond K; 8 columns per
// thread.  Bound by memory: 2048 x 4096 f32 9 us = 5.5 TB/s (the fused kernel's tile staging, two bytes per store: 37 us).
template <int DT, bool VEC>
__global__ void __launch_bounds__(256) stage_rows_kernel(const void* __restrict__ x, int64_t M, int64_t K, int64_t ldx, const int32_t* __restrict__ perm, int64_t K_pad,
                                                         __half* __restrict__ out) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, per = K_pad / 8;
    pdl_wait();   // x is written by the operator ahead in the stream; the buffers behind it are free
    pdl_launch_dependents();
    if (idx >= M * per) return;
    const int64_t m = idx / per, k = (idx - m * per) * 8;
    float v[8];
    if (VEC && k + 8 <= K) {
        if (DT == 0) {
            const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + m * ldx + k);
            const float4 a = p[0], b = p[1];
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
            const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(x) + m * ldx + k);
            const uint32_t wd[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (DT == 1) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&wd[j]));
                    v[2 * j] = f.x, v[2 * j + 1] = f.y;
                } else {
                    v[2 * j] = __uint_as_float(wd[j] << 16), v[2 * j + 1] = __uint_as_float(wd[j] & 0xFFFF0000u);
                }
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = k + j < K ? load_in(x, DT, m * ldx + (perm ? perm[k + j] : k + j)) : 0.0f;
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const __half2 h = __floats2half2_rn(fminf(fmaxf(v[2 * j], -65504.0f), 65504.0f), fminf(fmaxf(v[2 * j + 1], -65504.0f), 65504.0f));
        o[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(out + m * K_pad + k) = make_uint4(o[0], o[1], o[2], o[3]);
}

template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl_w(void (*kern)(KArgs...), int64_t blocks, int threads, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_stage_rows(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, const int32_t* perm, int64_t K_pad, void* rows, cudaStream_t st) {
    __half* out = reinterpret_cast<__half*>(rows);
    const int64_t es = x_dtype == 0 ? 4 : 2;
    const bool vec = !perm && ((uintptr_t)x & 15) == 0 && (ldx * es) % 16 == 0;
    const int64_t blocks = (M * (K_pad / 8) + 255) / 256;
#define STAGE_(DT, V) launch_pdl_w(stage_rows_kernel<DT, V>, blocks, 256, st, x, M, K, ldx, perm, K_pad, out)
    if (x_dtype == 0) return vec ? STAGE_(0, true) : STAGE_(0, false);
    if (x_dtype == 1) return vec ? STAGE_(1, true) : STAGE_(1, false);
    return vec ? STAGE_(2, true) : STAGE_(2, false);
#undef STAGE_
}

// y[m][n] = acc (+ bias); lanes hold 32 consecutive n
template <typename T>
struct EpiOut {
    T* y;
    int64_t ldy;
    const float* bias;
    int N, n0;   // columns of the whole weight; first one of this panel
    __device__ __forceinline__ void store(float (&v)[32], int n, int m, int m_end, int) const {
        n += n0;
        if (n >= N) return;
        const float b = bias ? bias[n] : 0.0f;
        T* o = y + (int64_t)m * ldy + n;
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (m + j < m_end) {
                const float f = v[j] + b;
                if constexpr (sizeof(T) == 4) o[(int64_t)j * ldy] = f;
                else if constexpr (std::is_same<T, __half>::value) o[(int64_t)j * ldy] = __float2half_rn(f);
                else o[(int64_t)j * ldy] = __float2bfloat16_rn(f);
            }
    }
};

// act[m][f] = f16(silu(gate) * up) of an interleaved weight: rows 8 i + 0 .. 3 of a tile are gates, 8 i + 4 .. 7 their ups (b200q_gate_up_row), in lanes
// four apart.  The gate's lane takes the first 16 tokens, the up's lane the others.  Same operations as swiglu_rows_kernel on the stored products, whose
// 134 MB (2048 tokens, 2 x 8192) are neither written nor read again: product and activation 102 + 32 us, now 99.
struct EpiGatedRows {
    static constexpr int WARPS = 16;   // (eight: two to a scheduler, whose divisions and shuffles took as long as a tile's products; a prompt of 2048 tokens 2 % longer)
    __half* act;
    int64_t ld;
    const float* bias;
    int N, n0;
    __device__ __forceinline__ void store(float (&v)[32], int n, int m, int m_end, int lane) const {
        n += n0;
        if (n >= N) return;      // (N % 128 == 0: the same for the whole warp)
        const float b = bias ? bias[n] : 0.0f;
        const bool up = (lane & 4) != 0;
        const int m0 = m + (up ? 16 : 0);
        __half* o = act + (int64_t)m0 * ld + (n >> 7) * 64 + ((n & 127) >> 3) * 4 + (n & 3);
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const float lo = v[j] + b, hi = v[16 + j] + b, got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, 4);
            const float g = up ? got : lo, u = up ? hi : got;
            const float a = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, det_expf(-g))), u);
            if (m0 + j < m_end) o[(int64_t)j * ld] = __float2half_rn(fminf(fmaxf(a, -65504.0f), 65504.0f));
        }
    }
};

struct WidePlan {
    int bt;            // token rows per tile
    int per, panels;   // weight tiles of 256 rows per panel (the last one has the rest)
    size_t x_bytes, buf_bytes;
    int nbuf, parts;   // parts: runs that K is cut into (one panel), as the fused kernel would
    size_t part_bytes; // their sums, f32 [parts][M][N]
    double us;         // estimated time
    size_t bytes() const { return x_bytes + nbuf * buf_bytes + part_bytes; }
};

// Panels of at most 64 MB of f16 weights, which L2 keeps; tile and panel sizes together are those with the least waves of tiles.  Nothing hides
// the expansion of the first panel, and every further one costs its launch chain, first slabs and last epilogues (measured: 9 us), so one panel
// is best up to that size.  A wave of tiles: tcpair::pick_bt.
static WidePlan wide_plan(const b200q_weight* w, int64_t M) {
    WidePlan p{};
    p.parts = gemm_k_splits(w, M);
    const int64_t pairs = w->num_sms / 2, NT = (w->T + 1) / 2, row_bytes = w->K_pad * 2;
    int64_t cap = (64ll << 20) / (256 * row_bytes);
    if (cap < 1) cap = 1;
    const int64_t panels = (NT + cap - 1) / cap;
    const int64_t least = panels > 1 ? (NT - 1) / panels + 1 : NT, most = panels > 1 ? cap : NT;
    for (int bt = tcpair::MAX_BT; bt >= 32; bt -= 32) {
        const int64_t MT = (M + bt - 1) / bt;
        const double wave = tcpair::wave_us(bt, w->K_pad / p.parts);
        for (int64_t per = most; per >= least; per--) {
            const int64_t full = NT / per, rest = NT - full * per;
            const double expand = (double)per * 256.0 * row_bytes * 1.5 / 5.0e6, gemm = (double)((per * MT * p.parts + pairs - 1) / pairs) * wave;
            const double last = (double)((rest * MT + pairs - 1) / pairs) * wave;
            const double us = expand + (double)(full - 1) * (gemm > expand ? gemm : expand) + gemm + last + 9.0 * (full + (rest > 0));
            if (p.bt == 0 || us < p.us) p.bt = bt, p.per = (int)per, p.panels = (int)(full + (rest > 0)), p.us = us;
        }
    }
    p.us += (double)M * w->K_pad * 6.0 / 5.0e6 + (p.parts > 1 ? 4.0 + (double)(p.parts + 1) * M * w->N * 4.0 / 4.0e6 : 0.0);
    p.part_bytes = p.parts > 1 ? (size_t)p.parts * M * w->N * sizeof(float) : 0;
    p.x_bytes = ((size_t)M * row_bytes + 1023) & ~(size_t)1023;
    p.buf_bytes = (size_t)p.per * 256 * row_bytes;
    p.nbuf = p.panels > 1 ? 2 : 1;
    return p;
}

// The fused kernel is the better one for fewer rows: it has no expansion pass, and up to 256 rows it expands a weight once too.  Its time is
// about (12 + 0.1 rows) us per wave of 128-row weight tiles at K = 4096 plus 4 us of staging and launch (measured from 136 to 4096 rows over the
// projections of hidden sizes 2048, 4096 and 8192; it cuts K when there are at most half as many tiles as SMs, which costs a pass over the partial
// sums, here as there).  Lines drawn from the same measurements: never below 512 rows; weights of several panels from 768 rows, with 14 % in hand
// (8192 x 8192, 800 rows: estimated 12 % faster, measured 3 % slower; 10240 x 8192, 300 to 640 rows: 10 to 25 % slower, 800: 8 to 14 % faster) and
// not where K is cut.  Cut products, fused / expanded, us, when the lines were drawn: 512 x 2048, 2048 rows 45.8 / 24.1; 1024 x 4096, 1280 rows 55.9 / 30.8; 1024 x 8192,
// 2048 rows 120 / 67; 4096 x 4096, 512 rows 49.0 / 47.0.
// The fused kernel's times are those from before all its warps stored results, and it would now be the better one above some of these lines (2048 x 8192, 2048 rows
// 76 / 84; 512 x 2048, 2048 rows 16 / 23).  They say what a step is expanded for where the paired kernel does not take it: gemm_pair_wins of gemm_pair.cu compares with today's
// times.  They alone decide a prompt's products with the expansion taken out of them, weights whose N is not a multiple of 256, products cut along K, and int4 weights
// with f32 results.  A caller who brings the smaller workspace has the fused kernel; all give the same bits.
static bool wide_wins(const b200q_weight* w, int64_t M, const WidePlan& p) {
    const int64_t mt = (M + 255) / 256, rows = ((M + mt - 1) / mt + 31) / 32 * 32, items = w->T * mt;
    const double wave = (12.0 + 0.1 * (double)rows) * (double)w->K_pad / 4096.0;
    if (p.parts > 1) {
        if (p.panels > 1 || (int64_t)p.parts * M > INT32_MAX / 2) return false;
        return p.us < 16.0 + (double)M * w->K_pad * 6.0 / 1.36e6 + wave / p.parts + (double)(p.parts + 1) * M * w->N * 4.0 / 4.0e6;
    }
    const double fused = 4.0 + (double)M * w->K_pad * 6.0 / 3.0e6 + (double)((items + w->num_sms - 1) / w->num_sms) * wave;
    return p.panels == 1 ? p.us < fused : M >= 768 && p.us * 1.14 < fused;
}

size_t gemm_wide_ws_bytes(const b200q_weight* w, int64_t M) {
    if (M < GEMM_WIDE_MIN_M || M > INT32_MAX / 2) return 0;
    const WidePlan p = wide_plan(w, M);
    return wide_wins(w, M, p) ? p.bytes() : 0;
}

// us of a whole call, not cut along K, runs of it back to back (fitted to 460 measured calls beside pair_us of gemm_pair.cu; the plan's own estimate above is a wave's
// relative one): every panel costs its launches, the longest panel's expansion is not hidden, and the products follow their waves.
double gemm_wide_us(const b200q_weight* w, int64_t M) {
    const WidePlan p = wide_plan(w, M);
    const int64_t pairs = w->num_sms / 2, NT = (w->T + 1) / 2, MT = (M + p.bt - 1) / p.bt, full = NT / p.per, rest = NT - full * p.per;
    const double waves = (double)(full * ((p.per * MT + pairs - 1) / pairs) + (rest * MT + pairs - 1) / pairs), rows = p.bt / 256.0, deep = (double)w->K_pad / 4096.0;
    const double panel = (double)p.per * 256.0 * (double)w->K_pad / 1e7, packed = (double)w->chunk_bytes / (TILE_ROWS * CHUNK_K);
    return -13.3 + 20.0 * p.panels + panel * (3.3 + 3.2 * packed) + waves * (2.3 * rows + deep * (1.25 + 28.1 * rows));
}

size_t gemm_wide_panel_bytes(const b200q_weight* w, int64_t M) { return gemm_wide_ws_bytes(w, M) ? wide_plan(w, M).buf_bytes : 0; }
bool gemm_wide_gated_ok(const b200q_weight* w, int64_t M) { return w->N % TILE_ROWS == 0 && gemm_wide_ws_bytes(w, M) && wide_plan(w, M).parts == 1; }

static cudaError_t dequant_f16_family(const b200q_weight* w, int tile0, int ntiles, __half* out, bool beside, cudaStream_t st) {
    switch (w->family) {
        case B200Q_FAM_Q4_K: return dequant_f16_launch<B200Q_FAM_Q4_K>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q6_K: return dequant_f16_launch<B200Q_FAM_Q6_K>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q8_0: return dequant_f16_launch<B200Q_FAM_Q8_0>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q5_K: return dequant_f16_launch<B200Q_FAM_Q5_K>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q4_1: return dequant_f16_launch<B200Q_FAM_Q4_1>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q5_1: return dequant_f16_launch<B200Q_FAM_Q5_1>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q2_K: return dequant_f16_launch<B200Q_FAM_Q2_K>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_Q3_K: return dequant_f16_launch<B200Q_FAM_Q3_K>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_IQ4_XS: return dequant_f16_launch<B200Q_FAM_IQ4_XS>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_TQ2_0: return dequant_f16_launch<B200Q_FAM_TQ2_0>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_I8S: return dequant_f16_launch<B200Q_FAM_I8S>(w, tile0, ntiles, out, beside, st);
        case B200Q_FAM_G4: return dequant_f16_launch<B200Q_FAM_G4>(w, tile0, ntiles, out, beside, st);
        default: return cudaErrorNotSupported;
    }
}

static int panel_tiles(const b200q_weight* w, const WidePlan& p, int nt0, int* nt) {   // weight tiles of 128 rows of the panel that starts at the pair nt0
    const int left = (int)((w->T + 1) / 2) - nt0;
    *nt = left < p.per ? left : p.per;
    return (int)(w->T - 2 * nt0 < 2 * *nt ? w->T - 2 * nt0 : 2 * *nt);
}

cudaError_t launch_expand(const b200q_weight* w, int64_t M, void* panel, bool beside, cudaStream_t st) {
    const WidePlan p = wide_plan(w, M);
    int nt;
    return dequant_f16_family(w, 0, panel_tiles(w, p, 0, &nt), reinterpret_cast<__half*>(panel), beside, st);
}

cudaError_t launch_gemm_wide(const b200q_weight* w, const void* x, int x_dtype, int64_t M, int64_t ldx, void* y, int y_dtype, int64_t ldy, uint8_t* ws, cudaStream_t st, const void* panel,
                             bool x_ready, void* act) {
    const WidePlan p = wide_plan(w, M);
    // Rows that are read in place need the expansion to be there already: one launched here would start beside the operator that makes the rows, which may
    // itself still wait for the product whose panel this one overwrites (staging waits for that operator first).
    const bool direct = x_ready && panel && x_dtype == 1 && !w->perm && w->K == w->K_pad && ((uintptr_t)x & 15) == 0 && ldx % 8 == 0;
    __half* staged = reinterpret_cast<__half*>(ws);
    const __half* xr = direct ? reinterpret_cast<const __half*>(x) : staged;
    const int64_t ldr = direct ? ldx : w->K_pad;
    cudaError_t e = direct ? cudaSuccess : launch_stage_rows(x, x_dtype, M, w->K, ldx, w->perm, w->K_pad, staged, st);
    int nt0 = 0;
    for (int i = 0; i < p.panels && e == cudaSuccess; i++) {
        int nt;
        const int ntiles = panel_tiles(w, p, nt0, &nt);
        __half* made = reinterpret_cast<__half*>(ws + p.x_bytes + (i & 1) * p.buf_bytes);
        const __half* buf = i == 0 && panel ? reinterpret_cast<const __half*>(panel) : made;
        if (buf == made) e = dequant_f16_family(w, 2 * nt0, ntiles, made, true, st);
        if (e != cudaSuccess) break;
        tcpair::Args a{};
        a.M = (int)M, a.N = ntiles * TILE_ROWS, a.K = (int)w->K_pad, a.E = 1, a.bt = p.bt, a.err = decode_error_dev(), a.err_bit = B200Q_DECODE_ERR_GEMM_WAIT;
        a.parts = p.parts;
        auto run = [&](const auto& epi) { return tcpair::launch(buf, a.N, w->K_pad, xr, ldr, a, epi, st, true); };
        const int n0 = nt0 * 256;
        if (p.parts > 1) {
            float* part = reinterpret_cast<float*>(ws + p.x_bytes + p.buf_bytes);
            e = tcpair::launch<true>(buf, a.N, w->K_pad, xr, ldr, a, EpiOut<float>{part, w->N, nullptr, (int)w->N, 0}, st, true);
            count_launch();
            return e != cudaSuccess ? e : launch_splitk_reduce(part, p.parts, M, w, y, y_dtype, ldy, st);
        }
        if (act) e = run(EpiGatedRows{(__half*)act, ldy, w->bias, (int)w->N, n0});
        else if (y_dtype == 0) e = run(EpiOut<float>{(float*)y, ldy, w->bias, (int)w->N, n0});
        else if (y_dtype == 1) e = run(EpiOut<__half>{(__half*)y, ldy, w->bias, (int)w->N, n0});
        else e = run(EpiOut<__nv_bfloat16>{(__nv_bfloat16*)y, ldy, w->bias, (int)w->N, n0});
        count_launch();
        nt0 += nt;
    }
    return e;
}

}  // namespace b200q
