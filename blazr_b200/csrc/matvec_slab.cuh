// matvec_slab.cuh -- matvec of weights that fit the chip's shared memory: a CTA owns some ROWS over the whole of K.
//
// The stream-K kernel (matvec_impl.cuh) deals chunks of 128 rows x 256 k, so every tile of a small weight is shared by several CTAs, whose partial sums
// meet in L2: about 2 us behind the last product, in a launch that streams its weights in 1.5.  Here a CTA takes 8 to 128 rows (the least multiple of 8
// with which one CTA per SM covers the weight), brings all their bytes into shared memory at once -- the planes of every chunk, shortened to its rows -- and its 16 warps
// split the rows by eights and K between them; the warps' sums meet in shared memory.  No ring, no workspace, and the same terms summed in f64: the same
// bits.  The price is that 148 SMs rarely divide the rows: 4096 rows run on 128 CTAs of 32.
// Measured (a chain of calls with one row, us, stream-K / this kernel): Q4_K 2048 x 2048 3.95 / 3.15, 4096 x 4096 5.6 / 4.6, 6144 x 4096 6.6 / 5.5,
// 16384 x 2048 7.5 / 5.9; Q6_K 4096 x 4096 5.7 / 5.1; Q8_0 8192 x 2048 6.0 / 4.8; with four rows, bound by the dot products, 0 to 1.8 less.
#pragma once
#include "matvec_impl.cuh"

namespace b200q {

static_assert((1 + SLAB_MAX_KC) * 8 <= SLAB_HDR, "barriers: records, then one per k-chunk");
constexpr int SLAB_THREADS = MV_CONSUMER_WARPS * 32;

// bounded: copies that never arrive are reported, not waited for
__device__ __forceinline__ void slab_wait(uint32_t bar_sa, int* err) {
    for (int spin = 0; spin < (1 << 22); spin++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar_sa)
            : "memory");
        if (ok) return;
    }
    if (err) atomicOr(err, 2);
}

// rows [row0, row0 + rows) of the k-chunks warp, warp + 16, ... -> shared memory: the warp makes their barriers, a lane issues a copy (one plane's rows of
// one tile).  By one warp for all chunks the copies of a Q6_K slab (128 of them) left the SM one after another in 1.3 us.
template <class F>
__device__ __forceinline__ void slab_request(const uint8_t* w, int KC, int cb, int row0, int rows, int R, int gpc, uint8_t* dst, int stride, uint64_t* bars, int warp, int lane) {
    const uint64_t pol = policy_evict_first();
    const int t = row0 >> 7, r = row0 & 127, n0 = rows < 128 - r ? rows : 128 - r;   // (the rest lies in the next tile)
    const int pl = lane >> 1, n = lane & 1 ? rows - n0 : n0;
    int from = 0, to = 0, pb = 0;
#pragma unroll
    for (int q = 0; q < F::NPLANES; q++) {
        const int b = F::plane_bytes(q, gpc);
        if (q < pl) from += 128 * b, to += R * b;
        if (q == pl) pb = b;
    }
    if (lane & 1) to += n0 * pb, from += KC * cb;      // (rows from the next tile's first on)
    else from += r * pb;
    for (int kc = warp; kc < KC; kc += MV_CONSUMER_WARPS) {
        if (lane == 0) {
            mbar_init(&bars[kc], 1);
            fence_mbar_init();
            fence_proxy_async();
            mbar_arrive_expect_tx(&bars[kc], (uint32_t)(rows * (cb >> 7)));
        }
        __syncwarp();
        if (pl < F::NPLANES && n > 0) bulk_g2s_hint(dst + (size_t)kc * stride + to, w + ((size_t)t * KC + kc) * cb + from, (uint32_t)(n * pb), &bars[kc], pol);
    }
}

// this warp's share: rows 8 rg .. of the slab, chunks ks, ks + KS, ...
template <class F, int MB>
__device__ __forceinline__ void slab_math(uint32_t w_sa, int stride, int R, int gpc, uint32_t x_sa, int M, int KC, int rg, int ks, int KS, uint32_t bars_sa, int* err, int lane,
                                          double (&acc)[MV_STEPS][MB]) {
    const int g4 = lane >> 3, i = lane & 7;
    const FmtMeta meta{gpc};
    constexpr int NOFF = FmtNoff<F>::value;
    uint32_t uoff[NOFF];
    F::unit_offsets(8 * rg + g4, i, meta, uoff);
#pragma unroll
    for (int q = 0; q < NOFF; q++) {   // the planes ahead of this offset's have R rows instead of 128
        int ahead = 0;
#pragma unroll
        for (int pl = 0; pl < F::plane_of(q); pl++) ahead += F::plane_bytes(pl, gpc);
        uoff[q] = keep_in_reg(uoff[q] + w_sa - (uint32_t)(ahead * (TILE_ROWS - R)));
    }
    const uint32_t xq = keep_in_reg(x_sa + 32u * (uint32_t)i), xs = keep_in_reg(x_sa + 256u + 4u * (uint32_t)i);
    for (int kc = ks; kc < KC; kc += KS) {
        const uint32_t xo = (uint32_t)(kc * M) * ACT_REC_BYTES, wo = (uint32_t)(kc * stride);
        uint4 xa[MB], xb[MB];
        float dx[MB];
        int bsA[MB], bsB[MB];
#pragma unroll
        for (int m = 0; m < MB; m++) {
            xa[m] = lds128_sa(xq + xo + m * ACT_REC_BYTES);
            xb[m] = lds128_sa(xq + xo + m * ACT_REC_BYTES + 16);
            dx[m] = __uint_as_float(lds32_sa(xs + xo + m * ACT_REC_BYTES));
            const uint32_t bs = lds32_sa(xs + xo + m * ACT_REC_BYTES + 32);
            bsA[m] = (int)(int16_t)(bs & 0xFFFFu);
            bsB[m] = (int)(int16_t)(bs >> 16);
        }
        slab_wait(bars_sa + 8u * (uint32_t)kc, err);
#pragma unroll
        for (int s4 = 0; s4 < MV_STEPS; s4++) {
            Unit u;
            if (s4 == 0) F::template load_unit_at<0>(wo, uoff, i, u, meta);
            else F::template load_unit_at<1>(wo, uoff, i, u, meta);
#pragma unroll
            for (int m = 0; m < MB; m++) acc[s4][m] = unit_terms<F>(u, xa[m], xb[m], dx[m], bsA[m], bsB[m], acc[s4][m]);
        }
    }
}

// successor hint: this CTA's share (g of G) of the chunks that the next weight's CTAs take first, into L2 (one thread).
// matvec_kernel's producer has the same loop in line: through this function every one of its launches took 0.2 % longer.
__device__ __forceinline__ void prefetch_next(const MatvecParams& p, int64_t g, int64_t G) {
    for (int64_t ng = g; ng < p.next_G; ng += G) {
        const int64_t a0 = sk_begin(ng, p.next_C, p.next_G), a1 = sk_begin(ng + 1, p.next_C, p.next_G);
        const SkPlan np_ = sk_plan(a0, a1, p.next_KC);
        const int n = (int)(a1 - a0) < p.next_pf ? (int)(a1 - a0) : p.next_pf;
        for (int j = 0; j < n; j++)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.next_w + sk_chunk_at(np_, a0, j) * (int64_t)p.next_chunk_bytes), "r"(p.next_chunk_bytes) : "memory");
    }
}

// OUT_SWIGLU: gate|up rows interleaved per tile, a CTA has a whole tile (R = 128) and quantises its 64 activations.
// NEXT: the launch has a successor hint (a form of its own: as a branch it cost every launch 0.05 us)
template <class F, int MB, int PRO, int OUT, class F2 = F, bool NEXT = false>
__global__ void __launch_bounds__(SLAB_THREADS, 1) matvec_slab_kernel(const MatvecParams p) {
    constexpr bool DUAL = !std::is_same<F, F2>::value;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ double red[TILE_ROWS * MB];          // [k share][row][m]
    uint64_t* xbar = reinterpret_cast<uint64_t*>(smem);
    uint64_t* wbar = xbar + 1;
    uint8_t* xhat = smem + SLAB_HDR;                // records [kc][m]
    uint8_t* slab = xhat + p.xhat_bytes;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KC = (int)p.KC, R = p.slab_rows, g = (int)blockIdx.x;
    const bool second = DUAL && g >= p.slabs1;
    const int row0 = (second ? g - p.slabs1 : g) * R;                                           // in its weight
    const int cb = second ? p.cb2 : p.cb1, gpc = second ? p.gpc2 : p.gpc, stride = R * (cb >> 7);
    const int base = second ? p.T1 * TILE_ROWS : 0;                                             // output row of the weight's first
    const int N = second ? (int)p.N - base : (DUAL ? p.T1 * TILE_ROWS : (int)p.N);
    const int have = ((N + TILE_ROWS - 1) / TILE_ROWS) * TILE_ROWS - row0, rows = have < R ? have : R;
    if (PRO != PRO_FUSED || !p.late) pdl_launch_dependents();
    // the weights are static: requested before anything is waited for
    if (second) slab_request<F2>(p.w2, KC, cb, row0, rows, R, gpc, slab, stride, wbar, warp, lane);
    else slab_request<F>(p.w, KC, cb, row0, rows, R, gpc, slab, stride, wbar, warp, lane);
    if constexpr (NEXT)
        if (tid == SLAB_THREADS - 1) prefetch_next(p, g, gridDim.x);
    if (PRO == PRO_NONE && tid == 0) {
        mbar_init(xbar, 1);
        fence_mbar_init();
        fence_proxy_async();
    }
    __syncthreads();
    if constexpr (PRO == PRO_FUSED) {
        __shared__ double s_red[MV_CONSUMER_WARPS];
        switch (KC * CHUNK_K / (MV_CONSUMER_WARPS * 32)) {
            case 16: { float nw[16]; load_nw<16>(p.norm_w, tid, nw); pdl_wait(); norm_prologue<MB, 16>(p, xhat, nw, tid, warp, lane, g == 0, s_red); break; }
            case 8: { float nw[8]; load_nw<8>(p.norm_w, tid, nw); pdl_wait(); norm_prologue<MB, 8>(p, xhat, nw, tid, warp, lane, g == 0, s_red); break; }
            case 4: { float nw[4]; load_nw<4>(p.norm_w, tid, nw); pdl_wait(); norm_prologue<MB, 4>(p, xhat, nw, tid, warp, lane, g == 0, s_red); break; }
            case 2: { float nw[2]; load_nw<2>(p.norm_w, tid, nw); pdl_wait(); norm_prologue<MB, 2>(p, xhat, nw, tid, warp, lane, g == 0, s_red); break; }
            default: { float nw[1]; load_nw<1>(p.norm_w, tid, nw); pdl_wait(); norm_prologue<MB, 1>(p, xhat, nw, tid, warp, lane, g == 0, s_red); break; }
        }
        if (p.late) pdl_launch_dependents();
    } else {
        pdl_wait();   // y and the bias may still be in use by the preceding kernel before this point
        if constexpr (PRO == PRO_QUANT) {
            if (p.x_dtype == 0) quant_prologue_t<0>(p, xhat, KC, 0, warp, lane);
            else if (p.x_dtype == 1) quant_prologue_t<1>(p, xhat, KC, 0, warp, lane);
            else quant_prologue_t<2>(p, xhat, KC, 0, warp, lane);
        } else {
            if (tid == 0) {
                const uint32_t bytes = (uint32_t)(KC * p.M) * ACT_REC_BYTES;
                mbar_arrive_expect_tx(xbar, bytes);
                bulk_g2s(xhat, p.xq, bytes, xbar);
            }
            slab_wait(smem_u32(xbar), p.err);
        }
    }
    const int groups = R >> 3, KS = MV_CONSUMER_WARPS / groups, ks = warp / groups, rg = warp - ks * groups;
    double acc[MV_STEPS][MB];
#pragma unroll
    for (int s4 = 0; s4 < MV_STEPS; s4++)
#pragma unroll
        for (int m = 0; m < MB; m++) acc[s4][m] = 0.0;
    if (ks < KS) {
        if (second) slab_math<F2, MB>(smem_u32(slab), stride, R, gpc, smem_u32(xhat), p.M, KC, rg, ks, KS, smem_u32(wbar), p.err, lane, acc);
        else slab_math<F, MB>(smem_u32(slab), stride, R, gpc, smem_u32(xhat), p.M, KC, rg, ks, KS, smem_u32(wbar), p.err, lane, acc);
#pragma unroll
        for (int s4 = 0; s4 < MV_STEPS; s4++)
#pragma unroll
            for (int m = 0; m < MB; m++) {
                double v = acc[s4][m];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                if ((lane & 7) == 0) red[(ks * R + 8 * rg + 4 * s4 + (lane >> 3)) * MB + m] = v;
            }
    }
    named_bar_sync(4, MV_CONSUMER_WARPS * 32);
    if constexpr (OUT == OUT_SWIGLU) {
        __shared__ float sy[MB][TILE_ROWS];
        if (tid < TILE_ROWS * MB) {
            const int64_t n = row0 + tid / MB;
            sy[tid % MB][tid / MB] = (float)(red[tid] + ((p.bias && n < N) ? (double)p.bias[n] : 0.0));
        }
        named_bar_sync(4, MV_CONSUMER_WARPS * 32);
        if (warp < 2 * p.M) swiglu_block_epilogue(p, sy[warp >> 1], g, warp >> 1, warp & 1, lane);
        return;
    }
    if (tid < R * MB) {
        double sum = red[tid];
        for (int k = 1; k < KS; k++) sum += red[k * R * MB + tid];
        const int row = tid / MB, m = tid % MB;
        const int64_t n = row0 + row;
        if (n < N && m < p.M) store_out_d(p.y, p.y_dtype, (int64_t)m * p.ldy + base + n, sum + (p.bias ? (double)p.bias[n] : 0.0));
    }
}

template <class F, int MB, int PRO, int OUT = OUT_PLAIN, class F2 = F, bool NEXT = false>
static cudaError_t slab_launch_t(const MatvecParams& p, int grid, int smem, cudaStream_t st) {
    if constexpr (!NEXT && PRO != PRO_FUSED && std::is_same<F, F2>::value)
        if (p.next_pf > 0) return slab_launch_t<F, MB, PRO, OUT, F2, true>(p, grid, smem, st);
    static std::atomic<bool> configured[16];   // per device; racing first calls both set the attribute (idempotent): re-entrant
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 16 || !configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(matvec_slab_kernel<F, MB, PRO, OUT, F2, NEXT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 216 * 1024);
        if (e != cudaSuccess) return e;
        if (dev < 16) configured[dev].store(true, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(SLAB_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t le = cudaLaunchKernelEx(&cfg, matvec_slab_kernel<F, MB, PRO, OUT, F2, NEXT>, p);
    if (le != cudaSuccess) return le;
    count_launch();
    return cudaGetLastError();
}
template <class F, int MB, class F2 = F>
static cudaError_t slab_launch_pro(const MatvecParams& p, int grid, int smem, cudaStream_t st) {
    if constexpr (std::is_same<F, F2>::value) {
        if (p.xq_out) {
            if (p.pro == 1) return slab_launch_t<F, MB, PRO_FUSED, OUT_SWIGLU>(p, grid, smem, st);
            return p.pro == 0 ? slab_launch_t<F, MB, PRO_NONE, OUT_SWIGLU>(p, grid, smem, st) : cudaErrorInvalidValue;
        }
        if (p.pro == 3) return slab_launch_t<F, MB, PRO_QUANT>(p, grid, smem, st);
    }
    if (p.xq_out) return cudaErrorInvalidValue;
    if (p.pro == 1) return slab_launch_t<F, MB, PRO_FUSED, OUT_PLAIN, F2>(p, grid, smem, st);
    return p.pro == 0 ? slab_launch_t<F, MB, PRO_NONE, OUT_PLAIN, F2>(p, grid, smem, st) : cudaErrorInvalidValue;
}
template <class F, class F2 = F>
static cudaError_t slab_launch_f(const MatvecParams& p, int mb, int grid, int smem, cudaStream_t st) {
    switch (mb) {
        case 1: return slab_launch_pro<F, 1, F2>(p, grid, smem, st);
        case 2: return slab_launch_pro<F, 2, F2>(p, grid, smem, st);
        case 4: return slab_launch_pro<F, 4, F2>(p, grid, smem, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace b200q
