// gemm_pair.cu -- host side of the paired dequant-GEMM (gemm_pair.cuh): which products take it, tile plan, launch.  The kernel is instantiated here for every
// format, apart from the decode kernels of inst_<format>.cu (with it among them a generated token was 2 % slower).
#include "gemm_pair.cuh"

namespace b200q {

struct PairPlan {
    int bt, nw, stages, w_stage_bytes, smem;
};

// Widths of a token tile: one wave of tiles of bt rows at K = 4096 against another (relative: what a call takes is pair_us)
static double pair_wave_us(int bt) { return 5.5 + 0.092 * bt; }

static int64_t pair_waves(const b200q_weight* w, int64_t M, int bt) {
    const int64_t pairs = tcpair::pair_sms() / 2;
    return ((w->T / 2) * ((M + bt - 1) / bt) + pairs - 1) / pairs;
}

static bool pair_plan(const b200q_weight* w, int64_t M, PairPlan* p) {
    double best = 0;
    p->bt = 0;
    for (int bt = tcpair::MAX_BT; bt >= 64; bt -= 16) {
        const double us = (double)pair_waves(w, M, bt) * pair_wave_us(bt);
        if (p->bt == 0 || us < best) p->bt = bt, best = us;
    }
    p->w_stage_bytes = (w->chunk_bytes + 127) & ~127;
    const int stage = p->bt * 64 + PG_A_BYTES, room = 227 * 1024 - PG_HDR - 1024;
    p->stages = (room - 2 * p->w_stage_bytes) / stage;
    if (p->stages > PG_MAX_STAGES) p->stages = PG_MAX_STAGES;
    if (p->stages < 4) return false;   // (an expanding warp holds two stages at a time)
    p->nw = (room - p->stages * stage) / p->w_stage_bytes;
    if (p->nw > PG_MAX_NW) p->nw = PG_MAX_NW;
    p->smem = PG_HDR + 1024 + p->stages * stage + p->nw * p->w_stage_bytes;
    return true;
}

// us of a whole call, runs of it back to back: this kernel and the fused one of gemm_tc.cu (the third way, an expansion ahead of the product: gemm_wide_us).  Fitted
// to 965 measured calls (twelve formats; 2560 to 28672 rows of weights, K 256 to 14336, 200 to 4096 tokens), off by 4 to 6 % (rms).  A wave of tiles takes
// a part for the weights, which the formats' expansion decides, and parts for its token rows, as waves of the chip and, power being what bounds them, as work.
struct FormatUs {
    double pair, fused;   // per wave of tiles at K = 4096
};
static FormatUs format_us(int family) {
    switch (family) {
        case B200Q_FAM_Q4_K: return {10.2, 5.4};
        case B200Q_FAM_Q6_K: return {11.3, 5.9};
        case B200Q_FAM_Q5_K: return {11.4, 6.7};
        case B200Q_FAM_Q4_1: return {9.2, 5.0};
        case B200Q_FAM_Q5_1: return {10.3, 6.1};
        case B200Q_FAM_Q2_K: return {8.8, 5.0};
        case B200Q_FAM_Q3_K: return {9.9, 5.4};
        case B200Q_FAM_IQ4_XS: return {16.0, 13.3};
        case B200Q_FAM_TQ2_0: return {7.2, 4.0};
        case B200Q_FAM_G4: return {8.9, 5.1};
        default: return {12.0, 6.3};   // Q8_0 (measured), I8S
    }
}
static double pair_us(const b200q_weight* w, int64_t M, int bt) {
    const double deep = (double)w->K_pad / 4096.0, rows = bt / 256.0, waves = (double)pair_waves(w, M, bt);
    const double work = (double)((w->T / 2) * ((M + bt - 1) / bt)) / (double)(tcpair::pair_sms() / 2);
    return 6.3 + 4.0 * waves * rows + deep * (waves * (format_us(w->family).pair + 4.7 * rows) + 14.1 * work * rows);
}
static double fused_us(const b200q_weight* w, int64_t M) {
    const int64_t mt = (M + 255) / 256, items = w->T * mt;
    const double deep = (double)w->K_pad / 4096.0, rows = (double)(((M + mt - 1) / mt + 31) / 32 * 32) / 256.0;
    const double waves = (double)((items + w->num_sms - 1) / w->num_sms), work = (double)items / (double)w->num_sms;
    return 2.8 + 6.7 * waves * rows + deep * (waves * (format_us(w->family).fused + 9.6 * rows) + 13.1 * work * rows);
}

// Which products take this kernel: those that the fused kernel does not cut along K (it then has fewer than half as many tiles as SMs) where the estimates put it
// ahead of the kernel that the caller's workspace would have otherwise, by what they are off for calls alike.  Measured (us, expanded / fused / this, f16 rows): Q6_K
// 14336 x 4096, 2048 rows 247 / 275 / 226, 900 rows 142 / 141 / 112, 700 rows - / 98 / 101, 520 rows - / 78 / 91; 8192 x 8192, 520 rows - / 91 / 97, 1536 rows 233 / 201 / 221;
// Q4_K 16384 x 2048, 700 rows - / 60 / 53; 2560 x 2048, 2048 rows 29.3 / 39.7 / 30.9; AWQ 6144 x 4096, 1536 rows 89 / 75 / 72; IQ4_XS 14336 x 4096, 2048 rows 245 / 325 / 255.
// (With one wave time
// for all formats and every product of 512 rows and two waves, 98 of 704 of these calls were slower than without this kernel, by up to 21 %; now
// none of 720 by more than 3 %.)  K of at most 1024: the expansion's second pass over the weight costs a call whose operands are not in L2 more than the loop shows (Q6_K
// 10240 x 1024, 785 rows 31.7 / 36.4 / 29.6 in a loop, 44 / 44 / 36 cold; IQ4_XS 30.9 / 43.2 / 33.7 and 42 / 50 / 42), so the line lies 12 % on this kernel's side.
bool gemm_pair_wins(const b200q_weight* w, int64_t M, bool expands) {
    PairPlan p;
    if (M < 192 || M > INT32_MAX / 2 || w->N % (2 * TILE_ROWS) != 0 || w->N > INT32_MAX || gemm_k_splits(w, M) > 1 || !pair_plan(w, M, &p)) return false;
    const double us = pair_us(w, M, p.bt);
    // (rows gathered through a permutation: 2.5 us a million values more to stage in rows than in the fused kernel's tiles; GPTQ 8192 x 8192, 520 rows - / 95 / 104)
    if (!expands) return us * 1.02 + (w->perm ? 2.5e-6 * (double)M * (double)w->K_pad : 0.0) < fused_us(w, M);
    return us * (w->K_pad <= 1024 && M <= 2048 ? 0.88 : 1.01) < gemm_wide_us(w, M);
}

static cudaError_t pair_family(int family, const PairParams& p, const CUtensorMap& mx, int ctas, int smem, cudaStream_t st) {
    switch (family) {
        case B200Q_FAM_Q4_K: return launch_pair_t<FmtQ4K>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q6_K: return launch_pair_t<FmtQ6K>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q8_0: return launch_pair_t<FmtQ8_0>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q5_K: return launch_pair_t<FmtQ5K>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q4_1: return launch_pair_t<FmtQ4_1>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q5_1: return launch_pair_t<FmtQ5_1>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q2_K: return launch_pair_t<FmtQ2K>(p, mx, ctas, smem, st);
        case B200Q_FAM_Q3_K: return launch_pair_t<FmtQ3K>(p, mx, ctas, smem, st);
        case B200Q_FAM_IQ4_XS: return launch_pair_t<FmtIQ4XS>(p, mx, ctas, smem, st);
        case B200Q_FAM_TQ2_0: return launch_pair_t<FmtTQ2_0>(p, mx, ctas, smem, st);
        case B200Q_FAM_I8S: return launch_pair_t<FmtI8S>(p, mx, ctas, smem, st);
        case B200Q_FAM_G4: return launch_pair_t<FmtG4>(p, mx, ctas, smem, st);
        default: return cudaErrorNotSupported;
    }
}

cudaError_t launch_gemm_pair(const b200q_weight* w, const void* x, int x_dtype, int64_t M, int64_t ldx, void* y, int y_dtype, int64_t ldy, uint8_t* ws, cudaStream_t st) {
    PairPlan pl;
    if (!pair_plan(w, M, &pl)) return cudaErrorNotSupported;
    const cudaError_t e = launch_stage_rows(x, x_dtype, M, w->K, ldx, w->perm, w->K_pad, ws, st);
    if (e != cudaSuccess) return e;
    CUtensorMap mx;
    if (!tcpair::make_map(&mx, ws, M, w->K_pad, w->K_pad, pl.bt / 2, false)) return cudaErrorInvalidValue;
    PairParams p{};
    p.w = w->data, p.bias = w->bias, p.y = y, p.ldy = ldy, p.y_dtype = y_dtype;
    p.M = (int)M, p.N = (int)w->N, p.KC = (int)w->KC;
    p.bt = pl.bt, p.MT = (int)((M + pl.bt - 1) / pl.bt), p.NT = (int)(w->T / 2);
    p.gpc = w->gpc, p.chunk_bytes = w->chunk_bytes, p.w_stage_bytes = pl.w_stage_bytes, p.nw = pl.nw, p.stages = pl.stages;
    p.err = decode_error_dev(), p.err_bit = B200Q_DECODE_ERR_GEMM_WAIT;
    int64_t ctas = 2 * (int64_t)p.MT * p.NT;
    if (ctas > tcpair::pair_sms()) ctas = tcpair::pair_sms();
    return pair_family(w->family, p, mx, (int)ctas, pl.smem, st);
}

}  // namespace b200q
