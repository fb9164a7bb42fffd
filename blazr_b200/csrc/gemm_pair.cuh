// gemm_pair.cuh -- dequant-GEMM on pairs of SMs: Y^T tile = W_tile[256 n x K] . X_tile[bt m x K]^T, the packed weight expanded inside the kernel.
//
// The paired GEMM of seq/tc_pair.cuh with another producer of its weight operand: where that kernel fetches f16 rows by TMA, sixteen warps of each CTA
// expand packed chunks (128 rows x 256 k, one bulk copy each) in registers and store f16 into the operand stage, in the 128-byte swizzle that the copy
// would have written.  So a prompt's weight is neither expanded in a pass of its own nor written to and read back from L2 (2 bytes per weight each way), a
// slab of 64 k costs an SM bt * 64 bytes of activations and 4.6 - 8.5 KB of packed weights, and the accumulator is double-buffered, so that an epilogue
// runs under the next tile's products.  A weight is expanded once per bt token rows, 16 of 28 warps doing nothing else.  Bound by power in long runs (the clock
// falls to 1.4 - 1.6 GHz; expansion and products together draw what the card may), by the expansion's latency per slab below about 200 rows a tile.  Measured, whole calls: Q6_K
// 14336 x 4096, 2048 f32 rows 265 us expanded ahead, 239 here (1.01 PFLOP/s), AWQ 6144 x 4096, 1531 rows 89 and 75; the product of rows expanded before takes 200 of the 265.
//
// Operands (f16 roundings of weights and activations), order of k and f32 accumulation are those of gemm_impl.cuh and gemm_wide.cu: the same results, bit for bit.
//
// Warp roles: 0 = activation tiles (TMA, both CTAs), 1 = MMA issuer (leader CTA), 2 = TMEM allocation, 3 = packed chunks, 4..11 = epilogue, 12..27 = expansion.
// Barriers: full[s] lives in the leader: the bytes of both CTAs' activation rows, one arrival per expanding warp of the leader's share of the stage and one for
// the whole of the peer's: its warps arrive on expanded[s] in their own CTA, and its warp 1, which has no products to issue, passes that on; empty[s] and
// acc_full are signalled in both CTAs by multicast tcgen05.commit; acc_empty lives in the leader; w_full / w_empty belong to the CTA's own chunk ring.
// Every wait is bounded (tcpair::bar_wait): one that runs out raises the abort flag, the roles leave their loops, copies in flight are waited for, TMEM is freed.
#pragma once
#include "gemm_impl.cuh"
#include "seq/tc_pair.cuh"

namespace b200q {

constexpr int PG_DQ_WARPS = 16, PG_EPI_WARPS = 8, PG_DQ_WARP0 = 4 + PG_EPI_WARPS;
constexpr int PG_THREADS = (PG_DQ_WARP0 + PG_DQ_WARPS) * 32;
constexpr int PG_MAX_STAGES = 6, PG_MAX_NW = 4, PG_HDR = 1024;
constexpr int PG_A_BYTES = TILE_ROWS * tcpair::BK * 2;

struct PairParams {
    const uint8_t* w;
    void* y;               // [M][ldy] of y_dtype
    const float* bias;
    int64_t ldy;
    int y_dtype;
    int M, N, KC;          // N a multiple of 256
    int bt, MT, NT;        // token rows per tile (a multiple of 16), token tiles, weight tiles of 256
    int gpc, chunk_bytes, w_stage_bytes, nw, stages;
    int* err;
    int err_bit;
};

// An arrival on another CTA's barrier that hands this CTA's shared memory over: what the thread has seen written there is ordered before it at cluster scope.
// The fence is restricted to shared memory: mbarrier.arrive.release.cluster also waits for all else that is on its way to memory (2.2 times the kernel's time).
__device__ __forceinline__ void arrive_cluster_shared(uint32_t bar) {
    asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void sts128_sa(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

template <class F>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PG_THREADS, 1) pair_dequant_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const PairParams p) {
    extern __shared__ uint8_t smem_raw[];
    using namespace tcpair;
    const int BT = p.bt, X_BYTES = BT / 2 * BK * 2, STAGE = PG_A_BYTES + X_BYTES, STAGES = p.stages;
    const uint32_t base = (sa(smem_raw) + 1023u) & ~1023u;
    const uint32_t full = base, empty = full + 8 * PG_MAX_STAGES, acc_full = empty + 8 * PG_MAX_STAGES, acc_empty = acc_full + 16, w_full = acc_empty + 16,
                   w_empty = w_full + 8 * PG_MAX_NW, expanded = w_empty + 8 * PG_MAX_NW;
    uint8_t* hdr = smem_raw + (base - sa(smem_raw));
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(hdr + 512);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(hdr + 520);
    const uint32_t stages = base + PG_HDR, chunks = stages + STAGES * STAGE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(rank));
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) bar_init(full + 8 * s, 2 + PG_DQ_WARPS / 2), bar_init(empty + 8 * s, 1), bar_init(expanded + 8 * s, PG_DQ_WARPS / 2);   // (half of a CTA's warps expand a stage)
        for (int b = 0; b < 2; ++b) bar_init(acc_full + 8 * b, 1), bar_init(acc_empty + 8 * b, 2 * PG_EPI_WARPS);
        for (int s = 0; s < p.nw; ++s) bar_init(w_full + 8 * s, 1), bar_init(w_empty + 8 * s, PG_DQ_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(tmem_ptr)), "n"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcpair::fence_before();
    __syncthreads();
    cluster_sync();   // the peer's barriers and TMEM exist
    tcpair::fence_after();
    const uint32_t tmem = *tmem_ptr;
    // packed weights depend on nothing: chunks and expansion start at once; the activation tiles and the epilogue wait for what is ahead in the stream
    pdl_launch_dependents();
    const int tiles = p.MT * p.NT, t0 = (int)blockIdx.x >> 1, stride = (int)gridDim.x >> 1, KC = p.KC;

    if (warp == 0) {
        if (elect()) {
            pdl_wait();
            const uint32_t full_l = map_leader(full);
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int t = t0; t < tiles && ok; t += stride) {
                const int xr = (t % p.MT) * BT + (int)rank * (BT / 2);
                for (int kb = 0; kb < 4 * KC; ++kb) {
                    ok = bar_wait(empty + 8 * s, ph, abort_flag);
                    if (!ok) break;
                    if (rank == 0) bar_expect(full + 8 * s, 2 * X_BYTES);
                    tma_pair(stages + s * STAGE + PG_A_BYTES, &map_x, kb * BK, xr, full_l + 8 * s);
                    if (++s == STAGES) s = 0, ph ^= 1u;
                }
            }
            // every slab issued has been consumed before the CTA's shared memory goes away (a stage never used passes at once; after an abort the waits give up)
            for (int i = 0; i < STAGES; ++i) {
                const unsigned long long since = now_ns();
                while (!bar_try(empty + 8 * s, ph) && now_ns() - since < WAIT_NS) {}
                if (++s == STAGES) s = 0, ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect()) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(BT >> 3) << 17) | ((uint32_t)(2 * ROWS >> 4) << 24);
            int s = 0, b = 0;
            uint32_t ph = 0, eph = 1;
            bool ok = true;
            for (int t = t0; t < tiles && ok; t += stride) {
                ok = bar_wait(acc_empty + 8 * b, eph, abort_flag);   // the epilogues of both CTAs have drained this buffer
                if (!ok) break;
                tcpair::fence_after();
                const uint32_t d = tmem + b * ACC_STRIDE;
                for (int kb = 0; kb < 4 * KC; ++kb) {
                    ok = bar_wait(full + 8 * s, ph, abort_flag);
                    if (!ok) break;
                    tcpair::fence_after();
                    const uint64_t da = desc_k128(stages + s * STAGE), db = desc_k128(stages + s * STAGE + PG_A_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) mma_pair(d, da + 2 * kk, db + 2 * kk, idesc, (kb | kk) != 0 ? 1u : 0u);
                    commit_pair(empty + 8 * s);
                    if (++s == STAGES) s = 0, ph ^= 1u;
                }
                if (ok) commit_pair(acc_full + 8 * b);
                b ^= 1;
                if (b == 0) eph ^= 1u;
            }
        } else if (rank != 0 && elect()) {
            // The peer's share of a stage, handed to the leader's products: its warps' stores are ordered before this thread by arrivals at CTA scope, and one arrival
            // at cluster scope passes all of them on (release is cumulative).  With a fence and an arrival of that kind in every expanding warp Q6_K 14336 x 4096 took 3 % longer
            // with 2048 rows and 6 % with 900 (AWQ 6144 x 4096, 1531 rows: 2 % less).
            const uint32_t full_l = map_leader(full);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = t0; t < tiles && ok; t += stride) {
                for (int kb = 0; kb < 4 * KC; ++kb) {
                    ok = bar_wait<false>(expanded + 8 * s, ph, abort_flag);
                    if (!ok) break;
                    arrive_cluster_shared(full_l + 8 * s);
                    if (++s == STAGES) s = 0, ph ^= 1u;
                }
            }
        }
    } else if (warp == 3) {
        if (elect()) {
            int s = 0;
            uint32_t ph = 1, issued = 0;
            bool ok = true;
            for (int t = t0; t < tiles && ok; t += stride) {
                const uint8_t* src = p.w + (size_t)(2 * (t / p.MT) + (int)rank) * KC * p.chunk_bytes;
                for (int kc = 0; kc < KC; ++kc) {
                    ok = bar_wait<false>(w_empty + 8 * s, ph, abort_flag);
                    if (!ok) break;
                    bar_expect(w_full + 8 * s, (uint32_t)p.chunk_bytes);
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(chunks + s * p.w_stage_bytes), "l"(src),
                                 "r"((uint32_t)p.chunk_bytes), "r"(w_full + 8 * s)
                                 : "memory");
                    src += p.chunk_bytes;
                    if (issued < (uint32_t)p.nw) ++issued;
                    if (++s == p.nw) s = 0, ph ^= 1u;
                }
            }
            // the last copy into every slot of the ring has landed (w_full: one phase behind the slot's next use)
            for (uint32_t i = 0; i < issued; ++i) {
                if (--s < 0) s = p.nw - 1, ph ^= 1u;
                const unsigned long long since = now_ns();
                while (!bar_try<false>(w_full + 8 * s, ph ^ 1u) && now_ns() - since < WAIT_NS) {}
            }
        }
    } else if (warp >= 4 && warp < PG_DQ_WARP0) {
        // ===================== epilogue: lane = weight row, columns = token rows =====================
        const int q = warp & 3, half = (warp - 4) >> 2;   // TMEM lane quarter; every other group of 32 columns
        const uint32_t drained = map_leader(acc_empty);
        int b = 0;
        uint32_t ph = 0;
        pdl_wait();   // y may still be read by what is ahead in the stream
        for (int t = t0; t < tiles; t += stride) {
            if (!__all_sync(0xffffffffu, bar_wait(acc_full + 8 * b, ph, abort_flag))) break;
            tcpair::fence_after();
            const int n = (t / p.MT) * 2 * ROWS + (int)rank * ROWS + q * 32 + lane, m0 = (t % p.MT) * BT, m_end = m0 + BT < p.M ? m0 + BT : p.M;
            const float bv = p.bias ? p.bias[n] : 0.0f;
            const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + b * ACC_STRIDE;
#pragma unroll 1
            for (int m = m0 + 32 * half; m < m_end; m += 64) {
                uint32_t v[32];
                ld32(ta + (m - m0), reinterpret_cast<float*>(v));
                ld_wait();
                const int nm = m_end - m;
                if (p.y_dtype == 0) store_cols<32>(reinterpret_cast<float*>(p.y) + m * p.ldy + n, p.ldy, v, bv, nm);
                else if (p.y_dtype == 1) store_cols<32>(reinterpret_cast<__half*>(p.y) + m * p.ldy + n, p.ldy, v, bv, nm);
                else store_cols<32>(reinterpret_cast<__nv_bfloat16*>(p.y) + m * p.ldy + n, p.ldy, v, bv, nm);
            }
            tcpair::fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive_cluster(drained + 8 * b);
            b ^= 1;
            if (b == 0) ph ^= 1u;
        }
    } else if (warp >= PG_DQ_WARP0) {
        // ===================== expansion: thread = weight row; a warp makes one of the two units (32 k) of every other slab =====================
        const int d = warp - PG_DQ_WARP0, q = d & 3, g = (d >> 2) & 1, grp = d >> 3, r = 32 * q + lane;
        const FmtMeta meta{p.gpc};
        const uint32_t made = rank == 0 ? full : expanded, row = stages + r * 128;
        uint32_t at[4];                             // the unit's four 16-byte pieces in a stage's row
#pragma unroll
        for (int c = 0; c < 4; ++c) at[c] = row + (uint32_t)(((4 * g + c) ^ (r & 7)) << 4);
        constexpr int NOFF = FmtNoff<F>::value;
        uint32_t uo[2][NOFF > 0 ? NOFF : 1];
        if constexpr (NOFF > 0) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                F::unit_offsets(r, 2 * (grp + 2 * j) + g, meta, uo[j]);
#pragma unroll
                for (int o = 0; o < NOFF; ++o) uo[j][o] += chunks;
            }
        }
        int s = grp, ws = 0;
        uint32_t ph = 1, wph = 0;
        bool ok = true;
        for (int t = t0; t < tiles && ok; t += stride) {
            for (int kc = 0; kc < KC; ++kc) {
                ok = __all_sync(0xffffffffu, bar_wait<false>(w_full + 8 * ws, wph, abort_flag));   // (the lanes leave together)
                if (!ok) break;
                Unit u[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if constexpr (NOFF > 0) F::template load_unit_at<0>((uint32_t)(ws * p.w_stage_bytes), uo[j], 2 * (grp + 2 * j) + g, u[j], meta);
                    else F::template load_unit<true>(hdr + (chunks - base) + (size_t)ws * p.w_stage_bytes, r, 2 * (grp + 2 * j) + g, u[j], meta);
                }
                // Both units are stored before one fence and their arrivals.  (The second stage is two slabs on: it is free once the slab STAGES - 2 before
                // this one is consumed, which waits for nothing of this warp's.)
                // The chunk's slot goes back with them: the copy that refills it writes through another proxy, which neither waits for loads that are in flight nor is
                // ordered behind them by an arrival.  The stores have the loaded values in them, and the fence is between the two proxies.  (Handed back behind the loads,
                // before their values were used, a slot was refilled under them: of 480 runs of Q8_0 4096 x 14336, 520 rows, 181 had wrong rows.)
                int s0 = s;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    uint32_t pk[16];
                    unit_to_f16<F::SIGNED, (NOFF > 0) && F::NIB, true>(u[j], pk);
                    ok = __all_sync(0xffffffffu, bar_wait<false>(empty + 8 * s, ph, abort_flag));   // the products that read this stage are done
                    if (!ok) break;
                    const uint32_t so = (uint32_t)(s * STAGE);
#pragma unroll
                    for (int c = 0; c < 4; ++c) sts128_sa(at[c] + so, pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                    if (j == 0) s0 = s;
                    else {
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_sa(w_empty + 8 * ws), mbar_arrive_sa(made + 8 * s0), mbar_arrive_sa(made + 8 * s);
                    }
                    if ((s += 2) >= STAGES) s -= STAGES, ph ^= 1u;
                }
                if (!ok) break;
                if (++ws == p.nw) ws = 0, wph ^= 1u;
            }
        }
    }
    __syncwarp();
    tcpair::fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.err) atomicOr(p.err, p.err_bit);
    cluster_sync();   // no CTA leaves while the peer may still signal its barriers or read its shared memory
    if (warp == 2) {
        tcpair::fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
    }
}

template <class F>
static cudaError_t launch_pair_t(const PairParams& p, const CUtensorMap& mx, int ctas, int smem, cudaStream_t st) {
    static std::atomic<bool> configured[16];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 16 || !configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(pair_dequant_gemm_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        if (dev < 16) configured[dev].store(true, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas), cfg.blockDim = dim3(PG_THREADS), cfg.dynamicSmemBytes = (size_t)smem, cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization, attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, pair_dequant_gemm_kernel<F>, mx, p);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}
}  // namespace b200q
