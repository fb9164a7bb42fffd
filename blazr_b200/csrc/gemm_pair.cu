// gemm_pair.cu -- host side of the paired dequant-GEMM (gemm_pair.cuh): which products take it, tile plan, launch.  The kernel is instantiated here for every
// format, apart from the decode kernels of inst_<format>.cu (with it among them a generated token was 2 % slower).
#include "gemm_pair.cuh"

namespace b200q {

struct PairPlan {
    int bt, nw, stages, w_stage_bytes, smem;
};

// Estimated time of one wave of tiles at K = 4096 (us, at the clock that a second of such products runs at): 29.5 for 256 token rows, 28 for 240, 23.6 for
// 176 measured; the fused kernel of gemm_tc.cu: 31 for 256, 22 to 24 for 192.
static double pair_wave_us(int bt) { return 5.5 + 0.092 * bt; }
static double fused_wave_us(int64_t rows) { return 0.125 * rows; }

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

// Which products take this kernel: those that the fused kernel does not cut along K (it then has fewer than half as many tiles as SMs), from 512 rows on where
// that kernel needs two waves and more, else where the estimates say so, with a launch of staged rows and a set-up that cost 4 us more here, and something in
// hand.  Measured in loops of seconds (us, expanded once by gemm_wide.cu / fused / this): Q6_K 14336 x 4096, 2048 rows 260 / 256 / 240, 1300 rows
// 193 / 167 / 153, 900 rows 148 / 136 / 112, 512 rows - / 68.5 / 65; Q4_K 16384 x 2048, 2048 rows 151 / 165 / 130, 1000 rows - / 89 / 72; 2048 x 8192, 1536 rows
// 70 / 64 / 61; 10240 x 8192, 1000 rows 224 / 183 / 162; Q8_0 6144 x 4096, 1800 rows 121 / 110 / 95; AWQ 6144 x 4096, 1531 rows 89 / 76 / 72; 57344 x 8192, 250
// rows - / 250 / 216; the fused kernel in one wave: Q8_0 6144 x 4096, 600 rows - / 34 / 36; GPTQ 4096 x 4096, 887 rows - / 33 / 34; Q4_K 8192 x 28672, 500 rows
// - / 215 / 227.  Where this one is taken and is the slower one it is so by 5 %: Q6_K 8192 x 8192, 520 rows - / 92 / 97; Q4_K
// 2560 x 2048, 2048 rows 28.7 / - / 30.1.
bool gemm_pair_wins(const b200q_weight* w, int64_t M) {
    PairPlan p;
    if (M < 192 || M > INT32_MAX / 2 || w->N % (2 * TILE_ROWS) != 0 || w->N > INT32_MAX || gemm_k_splits(w, M) > 1 || !pair_plan(w, M, &p)) return false;
    const int64_t mt = (M + 255) / 256, rows = ((M + mt - 1) / mt + 31) / 32 * 32, waves = (w->T * mt + w->num_sms - 1) / w->num_sms;
    if (M >= 512 && waves > 1) return true;
    const double deep = (double)w->K_pad / 4096.0;
    return ((double)pair_waves(w, M, p.bt) * pair_wave_us(p.bt) * deep + 4.0) * (waves > 1 ? 1.03 : 1.09) < (double)waves * fused_wave_us(rows) * deep;
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
