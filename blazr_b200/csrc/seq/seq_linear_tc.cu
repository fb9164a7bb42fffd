// seq_linear_tc.cu -- tensor-core path of the dense linear layer: y[M,N] (f32) = x[M,K] (bf16) . w[N,K]^T (bf16), f32 accumulation
// on the 5th-generation tensor cores (tcgen05.mma, accumulator in tensor memory).
//
// Ordinary and grouped products of 32 rows and more run on the paired-SM kernel of tc_pair.cuh (one tile of 256 weight rows per CTA pair,
// persistent; the epilogue functors and the choice of the token tile are below).  What follows describes the kernel that is kept for products of
// one weight per head and for banks of more experts than the paired kernel's shared memory lists.
//
// One CTA per 128 (n) x 128 (m) output tile.  The weight tile is the MMA's A operand (TMEM lane = n), the activation tile its B
// operand (TMEM column = m), so that in the epilogue the 32 threads of a warp hold 32 consecutive n of one token: coalesced stores.
// Both operands are K-major bf16 rows in global memory; TMA (cp.async.bulk.tensor.2d, 128-byte swizzle) brings 64-k slabs of both
// into a ring of shared-memory stages, rows and k beyond the matrices read as zero.  Warp 0 / lane 0 issues the copies, warp 1 /
// lane 0 the MMAs (4 per slab, K = 16 each); tcgen05.commit releases a stage and, after the last slab, publishes the accumulator
// to all 4 warps, which read it with tcgen05.ld.  The ring is 3 stages of 32 KB so that two CTAs share an SM and one's epilogue
// runs under the other's main loop.  The k order of every output element is fixed (ascending slabs), whatever M is.
//
// Optional epilogue EPI_GATED for a stacked gate|up weight whose rows alternate (gate j, up j): neighbouring lanes hold the pair,
// out[m][j] = act(gate, up) (clamped swish or tanh-gelu gate, seq_common.cuh) is written in the activation type and the [M, 2F]
// product never reaches memory.  EPI_PLAIN_ACT applies an activation of one argument (squared relu) to every output.
//
// Every wait is bounded: a wait that runs out sets bit 1 of the library's error flags and the CTA leaves through the common
// exit (its copies in flight are waited for, again bounded, and its tensor memory is freed).
#include <cuda.h>

#include <type_traits>

#include "seq_common.cuh"
#include "tc_pair.cuh"

namespace b200seq {

namespace {

constexpr int BM = 128, BN = 128, BK = 64, STAGES = 3;
constexpr int STAGE_BYTES = (BM + BN) * BK * 2;            // 32 KB: weight slab then activation slab
constexpr uint32_t WAIT_LIMIT = 1u << 24;                  // try_wait polls (each blocks for a while in hardware): seconds at most

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// false: the wait ran out (the caller leaves; nothing it waited for may be touched)
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023) == 1023 && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major operand, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

struct TcParams {
    float* y;
    void* act_out;
    int64_t ldy, ldo;
    int M, N, K, epi, out_dtype;
    ActParams act;
    int* err;
    const int32_t* offs;   // grouped form: [E + 1] first row of every group; rows of group e use the weight rows e * N .. e * N + N - 1
    int E;
    int heads;             // per-head form (blockIdx.z = head e): every row goes through every head's weight rows e * N .., reading the columns
    int silu_lo, silu_hi;  // EPI_NONE: the columns [silu_lo, silu_hi) pass silu
    int64_t ocol;          // e * K .. of its x row and writing the columns e * ocol .. of its output row
};
constexpr int EPI_NONE = 0, EPI_GATED = 1, EPI_PLAIN_ACT = 2;

__global__ void __launch_bounds__(128) linear_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const TcParams p) {
    chain_enter();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[STAGES], empty[STAGES], acc_full;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // token tiles vary fastest: the CTAs that run together share a few weight tiles and all activation tiles, which L2 holds, so the
    // weights cross HBM once instead of once per token tile
    const int n0 = blockIdx.y * BN;
    int m0 = blockIdx.x * BM, m_end = p.M, wrow0 = n0, xk0 = 0;
    int64_t oc0 = 0;
    if (p.heads) wrow0 = (int)blockIdx.z * p.N + n0, xk0 = (int)blockIdx.z * p.K, oc0 = (int64_t)blockIdx.z * p.ocol;
    if (p.offs) {   // grouped: blockIdx.x counts the row tiles of all groups in group order; a tile never crosses into the next group's rows
        __shared__ int grp[3];
        if (threadIdx.x == 0) {
            int acc = 0, e = 0;
            grp[2] = -1;
            for (; e < p.E; ++e) {
                const int b = p.offs[e], c = p.offs[e + 1] - b;
                const int nt = (c + BM - 1) / BM;
                if ((int)blockIdx.x < acc + nt) {
                    grp[0] = b + ((int)blockIdx.x - acc) * BM, grp[1] = b + c, grp[2] = e;
                    break;
                }
                acc += nt;
            }
        }
        __syncthreads();
        if (grp[2] < 0) return;   // more tiles were launched than the groups have (the bound does not know the group sizes)
        m0 = grp[0], m_end = grp[1], wrow0 = grp[2] * p.N + n0;
    }
    const int nk = (p.K + BK - 1) / BK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], 1);
        mbar_init(&acc_full, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(smem_u32(&tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    volatile int* ab = &abort_flag;

    if (warp == 0 && lane == 0) {
        int issued = 0;
        for (int kb = 0; kb < nk; ++kb, ++issued) {
            const int s = kb % STAGES;
            if (kb >= STAGES && !mbar_wait_bounded(&empty[s], ((kb / STAGES) - 1) & 1, ab)) break;
            mbar_expect_tx(&full[s], STAGE_BYTES);
            uint8_t* st = smem + (size_t)s * STAGE_BYTES;
            tma_load_2d(st, &map_w, kb * BK, wrow0, &full[s]);
            tma_load_2d(st + BN * BK * 2, &map_x, xk0 + kb * BK, m0, &full[s]);
        }
        if (*ab) {   // leave only when the copies already issued have landed (or the bounded wait gives up on them too)
            for (int kb = max(0, issued - STAGES); kb < issued; ++kb) {
                uint32_t i = 0;
                while (!mbar_try_wait(&full[kb % STAGES], (kb / STAGES) & 1) && ++i < WAIT_LIMIT) {}
            }
        }
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BM >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);   // bf16 x bf16 -> f32
        bool ok = true;
        for (int kb = 0; kb < nk && ok; ++kb) {
            const int s = kb % STAGES;
            ok = mbar_wait_bounded(&full[s], (kb / STAGES) & 1, ab);
            if (!ok) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + (size_t)s * STAGE_BYTES);
            const uint64_t da = make_desc(sa), db = make_desc(sa + BN * BK * 2);
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) tc_mma_ss(tmem, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), idesc, (kb | kk) != 0 ? 1u : 0u);
            tc_commit(&empty[s]);
        }
        if (ok) tc_commit(&acc_full);
    }
    __syncwarp();
    const bool have = mbar_wait_bounded(&acc_full, 0, ab);
    tc_fence_after();
    if (have) {
        const int n = n0 + warp * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < BM; c += 16) {
            if (m0 + c >= m_end) break;          // uniform across the CTA
            uint32_t r[16];
            tc_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, r);
            tc_wait_ld();
            if (p.epi == EPI_NONE) {
                if (n < p.N) {
                    if (n >= p.silu_lo && n < p.silu_hi) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(siluf_acc(__uint_as_float(r[j])));
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (m0 + c + j < m_end) p.y[(int64_t)(m0 + c + j) * p.ldy + oc0 + n] = __uint_as_float(r[j]);
                }
            } else if (p.epi == EPI_PLAIN_ACT) {
                if (n < p.N) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (m0 + c + j < m_end) store_act(p.act_out, p.out_dtype, (int64_t)(m0 + c + j) * p.ldo + oc0 + n, act_plain(p.act.kind, __uint_as_float(r[j])));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float mine = __uint_as_float(r[j]);
                    const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
                    if ((lane & 1) == 0 && n + 1 < p.N && m0 + c + j < m_end)
                        store_act(p.act_out, p.out_dtype, (int64_t)(m0 + c + j) * p.ldo + oc0 + (n >> 1), act_gated(p.act, mine, other));
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && abort_flag) atomicOr(p.err, 2);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem) : "memory");
}

// ---- epilogues of the paired-SM kernel (tc_pair.cuh): v[j] = acc[n][m + j] ----
// One instantiation per activation kind and output type: with the kind tested per value, every kind's code (divisions, erfc, tanh) was inlined for
// each of the 16 or 32 values and the epilogue warps waited for instructions.
template <bool SILU>
struct EpiF32 {
    float* y;
    int64_t ldy;
    int N, silu_lo, silu_hi;
    __device__ __forceinline__ void store(float (&v)[32], int n, int m, int m_end, int) const {
        if (n >= N) return;
        if (SILU && n >= silu_lo && n < silu_hi) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = siluf_acc(v[j]);
        }
        float* o = y + (int64_t)m * ldy + n;
        if (m + 32 <= m_end) {
#pragma unroll
            for (int j = 0; j < 32; ++j) o[(int64_t)j * ldy] = v[j];
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (m + j < m_end) o[(int64_t)j * ldy] = v[j];
        }
    }
};
template <int KIND, typename T>
struct EpiPlainAct {
    T* out;
    int64_t ldo;
    int N;
    __device__ __forceinline__ void store(float (&v)[32], int n, int m, int m_end, int) const {
        if (n >= N) return;
        T* o = out + (int64_t)m * ldo + n;
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (m + j < m_end) {
                const float r = act_plain(KIND, v[j]);
                if constexpr (sizeof(T) == 4) o[(int64_t)j * ldo] = r;
                else o[(int64_t)j * ldo] = __float2bfloat16_rn(r);
            }
    }
};
// Activations that leave as bf16 take the division without its branches (reciprocal approximation and one Newton step, 1 ulp of f32): the
// rounding call behind 1 / d kept the 16 activations of a lane from overlapping and made the epilogue, not the tensor pipe, the bound
// (4096 x 16384 x 2048: 326 us against 202 us of the plain product).  f32 outputs keep the rounded division.  A quarter of 1 + exp(-x) is formed,
// so that its reciprocal is a normal number as far as the exponential is finite; beyond, the sigmoid is 0.
__device__ __forceinline__ float sigmoid_nobranch(float x) {
    const float d = fmaf(0.25f, expf(fminf(-x, 88.7f)), 0.25f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = 0.25f * fmaf(r, fmaf(-d, r, 1.0f), r);
    return x < -88.7f ? 0.0f : r;
}
template <int KIND>
__device__ __forceinline__ float act_gated_nobranch(const ActParams& a, float gate, float up) {
    if (KIND == B200SEQ_ACT_GELU_TANH) return gate * sigmoid_nobranch(1.5957691216057308f * (gate + 0.044715f * gate * gate * gate)) * up;
    const float g = fminf(gate, a.limit);
    const float u = fminf(fmaxf(up, -a.limit), a.limit);
    return g * sigmoid_nobranch(a.alpha * g) * (u + a.shift);
}
// rows alternate (gate j, up j): an even lane holds the gates, the odd lane beside it the ups of the same 32 tokens.  They trade halves, so
// that the even lane computes tokens 0 .. 15 and the odd one 16 .. 31 (one activation per lane and token instead of one per lane pair).
// pack: bf16 output with 4-byte aligned pairs of columns -- lanes two apart trade again and store two columns at once
template <int KIND, typename T>
struct EpiGated {
    T* out;
    int64_t ldo;
    int N, pack;
    ActParams act;
    __device__ __forceinline__ void store(float (&v)[32], int n, int m, int m_end, int lane) const {
        constexpr bool BF16 = sizeof(T) == 2;
        const bool odd = lane & 1;
        ActParams a = act;
        a.kind = KIND;
        float r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float x = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 16], 1);
            const float g = odd ? x : v[j], u = odd ? v[j + 16] : x;
            r[j] = BF16 ? act_gated_nobranch<KIND>(a, g, u) : act_gated(a, g, u);
        }
        const int f = n >> 1, mt = m + (odd ? 16 : 0);
        if constexpr (BF16) {
            if (pack) {
                const bool hi = lane & 2;
                const int t0 = mt + (hi ? 8 : 0);
                T* o = out + (int64_t)t0 * ldo + (f & ~1);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float x = __shfl_xor_sync(0xffffffffu, hi ? r[j] : r[j + 8], 2);
                    const __nv_bfloat162 b = hi ? __floats2bfloat162_rn(x, r[j + 8]) : __floats2bfloat162_rn(r[j], x);
                    if (n < N && t0 + j < m_end) *reinterpret_cast<__nv_bfloat162*>(o + (int64_t)j * ldo) = b;
                }
                return;
            }
        }
        T* o = out + (int64_t)mt * ldo + f;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if ((n | 1) < N && mt + j < m_end) {
                if constexpr (BF16) o[(int64_t)j * ldo] = __float2bfloat16_rn(r[j]);
                else o[(int64_t)j * ldo] = r[j];
            }
    }
};

using tcpair::encode_fn;
using tcpair::make_map;

// Token rows per tile of the paired-SM kernel; 0: the product stays on the single-SM kernel (per-head products: K and N of one head)
int pick_tile(const TcParams& p) {
    const int64_t pairs = tcpair::pair_sms() / 2;
    if (p.heads || pairs < 1 || (p.offs && p.E > tcpair::MAX_GROUPS)) return 0;
    const int64_t NT = (p.N + 255) / 256;
    if (!p.offs) return tcpair::pick_bt(pairs, p.K, [&](int bt) { return (p.M + bt - 1) / bt * NT; });
    // Grouped: a group's last tile is half full on average, its rows are shared out evenly over its tiles, and few rows are a tile a group.  Of equal ones the
    // smallest: the less a stage holds, the more of them there are.
    int best = 0;
    double best_t = 0;
    for (int bt : {256, 192, 128, 64, 32}) {
        int64_t tiles = (p.M + bt / 2 * (int64_t)p.E + bt - 1) / bt;
        if (tiles < p.E) tiles = p.E;
        const int64_t width = p.M / tiles + 16 < bt ? p.M / tiles + 16 : bt;
        const double t = (double)((tiles * NT + pairs - 1) / pairs) * tcpair::wave_us((int)width, p.K);
        if (best == 0 || t <= best_t) best = bt, best_t = t;
    }
    return best;
}

template <class Epi>
cudaError_t launch_pair(int bt, const void* x, int64_t ldx, const void* w, const TcParams& p, const Epi& epi, cudaStream_t st) {
    tcpair::Args a{};
    a.M = p.M, a.N = p.N, a.K = p.K, a.offs = p.offs, a.E = p.offs ? p.E : 1, a.bf16 = 1, a.bt = bt, a.err = p.err, a.err_bit = 2;
    if (p.offs) return tcpair::launch<false, true>(w, (int64_t)p.E * p.N, p.K, x, ldx, a, epi, st, true);
    return tcpair::launch(w, p.N, p.K, x, ldx, a, epi, st, true);
}

int launch(const void* x, int64_t ldx, const void* w, TcParams p, cudaStream_t st) {
    CUtensorMap mw, mx;
    const int64_t wrows = p.offs ? (int64_t)p.E * p.N : (p.heads ? (int64_t)p.heads * p.N : p.N);
    p.err = error_flag_dev();
    if (const int tile = pick_tile(p)) {
        cudaError_t e = cudaErrorInvalidValue;
        auto typed = [&](auto* out) {
            using T = std::remove_pointer_t<decltype(out)>;
            const int pack = sizeof(T) == 2 && p.N % 4 == 0 && p.ldo % 2 == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0;
            switch (p.act.kind) {
                case B200SEQ_ACT_SWISH_CLAMP: return launch_pair(tile, x, ldx, w, p, EpiGated<B200SEQ_ACT_SWISH_CLAMP, T>{out, p.ldo, p.N, pack, p.act}, st);
                case B200SEQ_ACT_GELU_TANH: return launch_pair(tile, x, ldx, w, p, EpiGated<B200SEQ_ACT_GELU_TANH, T>{out, p.ldo, p.N, pack, p.act}, st);
                case B200SEQ_ACT_RELU2: return launch_pair(tile, x, ldx, w, p, EpiPlainAct<B200SEQ_ACT_RELU2, T>{out, p.ldo, p.N}, st);
                case B200SEQ_ACT_GELU_ERF: return launch_pair(tile, x, ldx, w, p, EpiPlainAct<B200SEQ_ACT_GELU_ERF, T>{out, p.ldo, p.N}, st);
                case B200SEQ_ACT_TANH: return launch_pair(tile, x, ldx, w, p, EpiPlainAct<B200SEQ_ACT_TANH, T>{out, p.ldo, p.N}, st);
                default: return launch_pair(tile, x, ldx, w, p, EpiPlainAct<B200SEQ_ACT_IDENT, T>{out, p.ldo, p.N}, st);
            }
        };
        if (p.epi == EPI_NONE) {
            if (p.silu_hi > p.silu_lo) e = launch_pair(tile, x, ldx, w, p, EpiF32<true>{p.y, p.ldy, p.N, p.silu_lo, p.silu_hi}, st);
            else e = launch_pair(tile, x, ldx, w, p, EpiF32<false>{p.y, p.ldy, p.N, 0, 0}, st);
        } else if (p.out_dtype == B200SEQ_F32) {
            e = typed(reinterpret_cast<float*>(p.act_out));
        } else {
            e = typed(reinterpret_cast<__nv_bfloat16*>(p.act_out));
        }
        if (e != cudaSuccess) return cuda_status(e, "linear tc pair");
        count_launch();
        return 0;
    }
    if (!make_map(&mw, w, wrows, p.K, p.K, 128, true) || !make_map(&mx, x, p.M, p.heads ? (int64_t)p.heads * p.K : p.K, ldx, 128, true))
        return fail(B200SEQ_ERR_CUDA, "linear: tensor map encoding failed");
    static bool attr_set = false;
    const int smem = STAGES * STAGE_BYTES + 1024;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(linear_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return cuda_status(e, "linear tc attribute");
        attr_set = true;
    }
    dim3 grid((p.M + BM - 1) / BM + (p.offs ? p.E : 0), (p.N + BN - 1) / BN, p.heads ? p.heads : 1);
    launch_chained(linear_tc_kernel, grid, 128, smem, st, mw, mx, p);
    SEQ_LAUNCH_CHECK("linear tc");
    return 0;
}

}  // namespace

bool linear_tc_usable(int x_dtype, int64_t ldx, int M, int N, int K, const void* x, const void* w) {
    (void)M, (void)N;
    return x_dtype == B200SEQ_BF16 && K % 8 == 0 && ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
           encode_fn() != nullptr;
}

int launch_linear_tc(const void* x, int64_t ldx, const void* w, int M, int N, int K, float* y, int64_t ldy, int silu_lo, int silu_hi, cudaStream_t st) {
    TcParams p{};
    p.silu_lo = silu_lo, p.silu_hi = silu_hi;
    p.y = y, p.ldy = ldy, p.M = M, p.N = N, p.K = K, p.epi = EPI_NONE;
    return launch(x, ldx, w, p, st);
}

// grouped form: rows [offs[e], offs[e + 1]) of x go through the weight w[e] ([E][N][K]); act_kind < 0: f32 product to out, else a plain activation
int launch_linear_tc_grouped(const void* x, int64_t ldx, const void* w, const int32_t* offs, int E, int rows, int N, int K, int act_kind, void* out, int out_dtype,
                             int64_t ldo, cudaStream_t st) {
    TcParams p{};
    p.M = rows, p.N = N, p.K = K, p.offs = offs, p.E = E;
    if (act_kind < 0) p.y = reinterpret_cast<float*>(out), p.ldy = ldo, p.epi = EPI_NONE;
    else p.act_out = out, p.ldo = ldo, p.out_dtype = out_dtype, p.epi = EPI_PLAIN_ACT, p.act = ActParams{act_kind, 0.f, 0.f, 0.f};
    return launch(x, ldx, w, p, st);
}

// per-head form: out[t][h * ocol + n] = sum_k x[t][h * K + k] * w[h][n][k]; act_kind < 0: f32 product, else a plain kind written in out_dtype
int launch_linear_tc_heads(const void* x, int64_t ldx, const void* w, int T, int H, int N, int K, int act_kind, void* out, int out_dtype, int64_t ldo, int64_t ocol,
                           cudaStream_t st) {
    TcParams p{};
    p.M = T, p.N = N, p.K = K, p.heads = H, p.ocol = ocol;
    if (act_kind < 0) p.y = reinterpret_cast<float*>(out), p.ldy = ldo, p.epi = EPI_NONE;
    else p.act_out = out, p.ldo = ldo, p.out_dtype = out_dtype, p.epi = EPI_PLAIN_ACT, p.act = ActParams{act_kind, 0.f, 0.f, 0.f};
    return launch(x, ldx, w, p, st);
}

// grouped form with any activation kind (gated kinds: the group's weight rows alternate gate / up, out has N / 2 columns)
int launch_linear_tc_grouped_act(const void* x, int64_t ldx, const void* w, const int32_t* offs, int E, int rows, int N, int K, const ActParams act, void* out,
                                 int out_dtype, int64_t ldo, cudaStream_t st) {
    TcParams p{};
    p.M = rows, p.N = N, p.K = K, p.offs = offs, p.E = E;
    p.act_out = out, p.ldo = ldo, p.out_dtype = out_dtype, p.epi = act_kind_gated(act.kind) ? EPI_GATED : EPI_PLAIN_ACT, p.act = act;
    return launch(x, ldx, w, p, st);
}

int launch_linear_tc_act(const void* x, int64_t ldx, const void* w, int M, int N, int K, const ActParams act, void* out, int out_dtype, int64_t ldo,
                         cudaStream_t st) {
    TcParams p{};
    p.act_out = out, p.ldo = ldo, p.out_dtype = out_dtype, p.M = M, p.N = N, p.K = K, p.epi = act_kind_gated(act.kind) ? EPI_GATED : EPI_PLAIN_ACT, p.act = act;
    return launch(x, ldx, w, p, st);
}

}  // namespace b200seq
