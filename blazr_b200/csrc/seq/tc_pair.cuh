// tc_pair.cuh -- dense 16-bit GEMM on pairs of SMs, shared by both libraries: acc[n][m] = sum_k w[n][k] x[m][k], f32 accumulation.
//
// Two CTAs of a cluster work on one tile of 256 weight rows x BT token rows (tcgen05.mma.cta_group::2, M = 256, N = BT, K = 16): each CTA
// holds its own 128 weight rows and HALF of the token rows in shared memory, so a 64-k slab costs 16 KB + BT * 64 bytes per SM where two
// single-SM 128 x 128 tiles would fetch 32 KB each for half the products.  TMEM lane = weight row, column = token: a warp's lanes hold
// 32 consecutive n of one token, the stores of the epilogue are coalesced.  Both operands are K-major 16-bit rows fetched by TMA
// (128-byte swizzle); rows and k outside the matrices read as zero.
//
// The kernel is persistent (one pair per two SMs, tiles dealt round-robin, token tiles fastest so that a weight tile is read from HBM
// once) and the accumulator is double-buffered in TMEM (2 x 256 columns): the epilogue warps drain tile i while the tensor cores run
// tile i + 1.  What bounds it is the tensor pipe; the single-SM kernel it replaces for large steps stalled on L2 -> SM traffic (512 bytes
// per 32 768 FLOPs against 1 024 per 131 072 here) and on a main loop that its epilogue interrupted.  Measured, 4096 tokens: 16384 x 2048 267 ->
// 198 us (1.39 PFLOP/s), with the gated activation 478 -> 201 us; 2048 x 8192 128 -> 100 us; 8192 x 1024 91 -> 61 us.
//
// Warp roles: 0 = TMA producer (both CTAs), 1 = MMA issuer (leader CTA only), 2 = TMEM allocation, 4 and on = epilogue.
// Barriers: full[s] lives in the leader and counts the bytes of both CTAs; empty[s] and acc_full are signalled in both CTAs by
// multicast tcgen05.commit; acc_empty lives in the leader and collects the epilogue warps of both CTAs.
// Every wait is bounded by a clock: one that runs out raises the abort flag, the role leaves its loop, and the CTA goes through the
// common exit (copies in flight waited for, TMEM freed).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

namespace tcpair {

constexpr int ROWS = 128;        // weight rows per CTA
constexpr int BK = 64;           // k per slab
// Warps of an epilogue: eight, or as many as it names itself (a multiple of four)
template <class Epi, class = void>
struct EpiWarps {
    static constexpr int value = 8;
};
template <class Epi>
struct EpiWarps<Epi, std::void_t<decltype(Epi::WARPS)>> {
    static constexpr int value = Epi::WARPS;
};
template <class Epi>
constexpr int THREADS = (4 + EpiWarps<Epi>::value) * 32;
constexpr int HDR = 1024;
constexpr int MAX_GROUPS = 1024;
constexpr unsigned long long WAIT_NS = 2000000000ull;

constexpr int MAX_BT = 256;
constexpr int ACC_STRIDE = MAX_BT;       // TMEM columns between the two accumulator buffers
constexpr int RING = 192 * 1024;         // bytes of operand stages
constexpr int MAX_STAGES = 9;
constexpr int SMEM = RING + HDR + 1024 + 2 * (MAX_GROUPS + 1) * 4;
constexpr int TMEM_COLS = 2 * ACC_STRIDE;
__host__ __device__ constexpr int stage_bytes(int bt) { return ROWS * BK * 2 + bt / 2 * BK * 2; }   // per CTA
__host__ __device__ constexpr int stage_count(int bt) { return RING / stage_bytes(bt) < MAX_STAGES ? RING / stage_bytes(bt) : MAX_STAGES; }

struct Args {
    int M, N, K;             // token rows, weight rows of one group, reduction length
    int bt;                  // token rows per tile: a multiple of 16, at most 256; grouped: the most that a tile has
    int MT, NT;              // token tiles (bound when grouped), weight tiles of 256
    int parts;               // PARTS (not grouped): K cut into this many runs of whole 256-k chunks, run i to the result rows i * M ..
    const int32_t* offs;     // grouped form: [E + 1] first token row of every group; group e uses the weight rows e * N ..
    int E;
    int bf16;                // operand type: 1 = bf16, 0 = f16
    int* err;                // device error word
    int err_bit;
};

__device__ __forceinline__ uint32_t sa(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t map_leader(uint32_t a) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive_cluster(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// CLUSTER: the arrivals may come from the other CTA of the pair (acquire at cluster scope; the CTA scope is the cheaper one)
template <bool CLUSTER = true>
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if (CLUSTER)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// false: the wait ran out, or another role of this CTA gave up
template <bool CLUSTER = true>
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (bar_try<CLUSTER>(bar, parity)) return true;
    unsigned long long t0 = 0;
    for (uint32_t i = 1;; ++i) {
        if (bar_try<CLUSTER>(bar, parity)) return true;
        if ((i & 255u) == 0) {
            if (*abort_flag) return false;
            const unsigned long long t = now_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > WAIT_NS) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}
// both CTAs' copies report to the leader's barrier (bar: its shared::cluster address)
__device__ __forceinline__ void tma_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map),
                 "r"(c0), "r"(c1), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar) {   // arrives on the same barrier of both CTAs when the MMAs issued so far are done
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// K-major operand, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t desc_k128(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void ld32(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Rows of a copy of token rows.  Grouped: 32, as many of them as the tile needs (a copy as long as the longest tile's 128 rows is an eighth too much for a tile
// of 176, and what bounds short products is 64 bytes a cycle from L2 to an SM), where they fill the longest tile's rows exactly; else all in one.
__host__ __device__ __forceinline__ int x_box(const Args& p) { return p.offs && p.bt % 64 == 0 ? 32 : p.bt / 2; }

struct Tile {
    int m0, m_end, wrow, n0;   // first token row, end of the tile's rows, first weight row in memory, first output column
    int bt;                    // columns of the tile: a multiple of 16, m_end - m0 or more
    int kb0, kb1, out;         // slabs of k; result row of token row 0
};

// slabs of k of tile t (PARTS: K is cut)
template <bool PARTS>
__device__ __forceinline__ void slabs_of(const Args& p, int MT, int t, int& kb0, int& kb1) {
    kb0 = 0, kb1 = (p.K + BK - 1) / BK;
    if (PARTS) {
        const int part = t / (MT * p.NT), chunks = p.K / (4 * BK);
        kb0 = 4 * (part * chunks / p.parts), kb1 = 4 * ((part + 1) * chunks / p.parts);
    }
}

// tile t of the step (token tiles fastest).  first, rows: grouped form, [E + 1] first token tile and first row of every group, in shared memory
template <bool PARTS, bool GROUPED>
__device__ __forceinline__ Tile tile_of(const Args& p, const int32_t* first, const int32_t* rows, int MT, int t) {
    Tile r;
    const int BT = p.bt;
    const int mt = t % MT;
    int nt = t / MT;
    r.out = 0;
    if (PARTS) {
        const int part = nt / p.NT;
        nt -= part * p.NT, r.out = part * p.M;
    }
    slabs_of<PARTS>(p, MT, t, r.kb0, r.kb1);
    r.n0 = nt * 2 * ROWS;
    r.wrow = r.n0;
    if constexpr (!GROUPED) {
        r.m0 = mt * BT, r.m_end = r.m0 + BT < p.M ? r.m0 + BT : p.M, r.bt = BT;
    } else {
        int lo = 0, hi = p.E;      // the last group whose first tile is <= mt (groups without rows have no tile)
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (first[mid] <= mt) lo = mid;
            else hi = mid;
        }
        // a group's rows are shared out evenly over its tiles: 32 groups of 512 rows, a few more or less, were 2 or 3 tiles of 256, a quarter of them padding
        const int t0 = first[lo], tiles = first[lo + 1] - t0, row0 = rows[lo], end = rows[lo + 1];
        r.bt = ((end - row0 + tiles - 1) / tiles + 15) & ~15;
        r.m0 = row0 + (mt - t0) * r.bt, r.m_end = r.m0 + r.bt < end ? r.m0 + r.bt : end;
        r.wrow += lo * p.N;
    }
    return r;
}

// Epi: struct with   __device__ void store(const float (&v)[32], int n, int m, int m_end, int lane) const
//   v[j] = acc[n][m + j] of this lane's n (n may be >= N: nothing is stored); all 32 lanes of a warp call it with the same m
// GROUPED is known when it is compiled: with a tile's width and copies read from memory in every product, what the elected threads pass to their instructions
// was no longer known to be uniform, and the product of 2048 x 2048 and 1303 rows took 15.0 us instead of 14.2.
template <class Epi, bool PARTS, bool GROUPED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS<Epi>, 1)
    pair_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Args p, const Epi epi) {
    extern __shared__ uint8_t smem_raw[];
    constexpr int EPI_WARPS = EpiWarps<Epi>::value;
    const int BT = p.bt, STAGE = stage_bytes(BT), STAGES = stage_count(BT);
    const uint32_t base = (sa(smem_raw) + 1023u) & ~1023u;
    const uint32_t full = base, empty = full + 8 * MAX_STAGES, acc_full = empty + 8 * MAX_STAGES, acc_empty = acc_full + 16;
    uint8_t* hdr = smem_raw + (base - sa(smem_raw));
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(hdr + 512);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(hdr + 520);
    int32_t* first = reinterpret_cast<int32_t*>(hdr + HDR + RING);
    int32_t* rows = first + MAX_GROUPS + 1;
    const uint32_t stages = base + HDR;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(rank));
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) bar_init(full + 8 * s, 1), bar_init(empty + 8 * s, 1);
        for (int b = 0; b < 2; ++b) bar_init(acc_full + 8 * b, 1), bar_init(acc_empty + 8 * b, 2 * EPI_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // programmatic launch: the operands (and what they were made from) are complete beyond this line, and what follows in the stream may start
    // (both are no-ops in a plain launch)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    int MT = p.MT;
    if (GROUPED && warp == 3) {   // first token tile of every group: an inclusive scan over the groups, 32 at a time
        int run = 0;
        for (int e0 = 0; e0 < p.E; e0 += 32) {
            const int e = e0 + lane, row = e < p.E ? p.offs[e] : 0, end = e < p.E ? p.offs[e + 1] : 0;
            if (e < p.E) rows[e] = row;
            if (e == p.E - 1) rows[p.E] = end;
            int n = (end - row + BT - 1) / BT;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, n, o);
                if (lane >= o) n += u;
            }
            if (e < p.E) first[e + 1] = run + n;
            run += __shfl_sync(0xffffffffu, n, 31);
        }
        if (lane == 0) first[0] = 0;
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(tmem_ptr)), "n"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    cluster_sync();   // the peer's barriers and TMEM exist
    fence_after();
    const uint32_t tmem = *tmem_ptr;
    if constexpr (GROUPED) MT = first[p.E];
    const int tiles = MT * p.NT * (PARTS ? p.parts : 1), stride = (int)gridDim.x >> 1;

    if (warp == 0) {
        if (elect()) {
            const uint32_t full_l = map_leader(full);
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            Tile next{};
            if (GROUPED && ((int)blockIdx.x >> 1) < tiles) next = tile_of<PARTS, GROUPED>(p, first, rows, MT, (int)blockIdx.x >> 1);
            for (int t = (int)blockIdx.x >> 1; t < tiles && ok; t += stride) {
                const Tile tl = GROUPED ? next : tile_of<PARTS, GROUPED>(p, first, rows, MT, t);
                const int box = x_box(p), half = GROUPED ? tl.bt / 2 : BT / 2, copies = GROUPED ? (half + box - 1) / box : 1;
                const int wr = tl.wrow + (int)rank * ROWS, xr = tl.m0 + (int)rank * half;
                for (int kb = tl.kb0; kb < tl.kb1; ++kb) {
                    ok = bar_wait(empty + 8 * s, ph, abort_flag);
                    if (!ok) break;
                    if (rank == 0) bar_expect(full + 8 * s, GROUPED ? 2 * (ROWS + copies * box) * BK * 2 : 2 * STAGE);
                    const uint32_t st = stages + s * STAGE;
                    tma_pair(st, &map_w, kb * BK, wr, full_l + 8 * s);
                    for (int i = 0; i < copies; ++i) tma_pair(st + (ROWS + i * box) * BK * 2, &map_x, kb * BK, xr + i * box, full_l + 8 * s);
                    if (++s == STAGES) s = 0, ph ^= 1u;
                    if (GROUPED && kb == tl.kb0 && t + stride < tiles) next = tile_of<PARTS, GROUPED>(p, first, rows, MT, t + stride);   // (looked up beside the copies)
                }
            }
            // every slab issued has been consumed before the CTA's shared memory goes away (a stage never used passes at once; after an
            // abort the waits give up)
            for (int i = 0; i < STAGES; ++i) {
                const unsigned long long t0 = now_ns();
                while (!bar_try(empty + 8 * s, ph) && now_ns() - t0 < WAIT_NS) {}
                if (++s == STAGES) s = 0, ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect()) {
            const uint32_t idesc0 = (1u << 4) | (p.bf16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(2 * ROWS >> 4) << 24);
            int s = 0, b = 0;
            uint32_t ph = 0, eph = 1;
            bool ok = true;
            Tile next{};
            if (GROUPED && ((int)blockIdx.x >> 1) < tiles) next = tile_of<PARTS, GROUPED>(p, first, rows, MT, (int)blockIdx.x >> 1);
            for (int t = (int)blockIdx.x >> 1; t < tiles && ok; t += stride) {
                ok = bar_wait(acc_empty + 8 * b, eph, abort_flag);   // the epilogues of both CTAs have drained this buffer
                if (!ok) break;
                fence_after();
                const uint32_t d = tmem + b * ACC_STRIDE;
                const uint32_t idesc = idesc0 | ((uint32_t)((GROUPED ? next.bt : BT) >> 3) << 17);
                int kb0, kb1;
                slabs_of<PARTS>(p, MT, t, kb0, kb1);
                const int nk = kb1 - kb0;
                for (int kb = 0; kb < nk; ++kb) {
                    ok = bar_wait(full + 8 * s, ph, abort_flag);
                    if (!ok) break;
                    fence_after();
                    const uint64_t da = desc_k128(stages + s * STAGE), db = desc_k128(stages + s * STAGE + ROWS * BK * 2);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) mma_pair(d, da + 2 * kk, db + 2 * kk, idesc, (kb | kk) != 0 ? 1u : 0u);
                    commit_pair(empty + 8 * s);
                    if (++s == STAGES) s = 0, ph ^= 1u;
                    if (GROUPED && kb == 0 && t + stride < tiles) next = tile_of<PARTS, GROUPED>(p, first, rows, MT, t + stride);
                }
                if (ok) commit_pair(acc_full + 8 * b);
                b ^= 1;
                if (b == 0) eph ^= 1u;
            }
        }
    } else if (warp >= 4) {
        const int q = warp & 3, share = (warp - 4) >> 2;    // TMEM lane quarter; one of every EPI_WARPS / 4 groups of 32 columns
        const uint32_t drained = map_leader(acc_empty);
        int b = 0;
        uint32_t ph = 0;
        for (int t = (int)blockIdx.x >> 1; t < tiles; t += stride) {
            const Tile tl = tile_of<PARTS, GROUPED>(p, first, rows, MT, t);
            if (!bar_wait(acc_full + 8 * b, ph, abort_flag)) break;
            fence_after();
            const int n = tl.n0 + (int)rank * ROWS + q * 32 + lane;
            const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + b * ACC_STRIDE;
#pragma unroll 1
            for (int c = share * 32; tl.m0 + c < tl.m_end; c += 8 * EPI_WARPS) {
                float v[32];
                ld32(ta + c, v);
                ld_wait();
                epi.store(v, n, tl.out + tl.m0 + c, tl.out + tl.m_end, lane);
            }
            fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive_cluster(drained + 8 * b);
            b ^= 1;
            if (b == 0) ph ^= 1u;
        }
    }
    __syncwarp();
    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.err) atomicOr(p.err, p.err_bit);
    cluster_sync();   // no CTA leaves while the peer may still signal its barriers or read its shared memory
    if (warp == 2) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
    }
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeFn>(f);
    }();
    return fn;
}

// rows x K 16-bit matrix with row stride ld elements; box = 64 k x box_rows rows, 128-byte swizzle, zero fill outside
inline bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t ld, int box_rows, bool bf16) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline int pair_sms() {   // SMs of the current device, rounded down to pairs
    static int sms[16] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev < 16 && sms[dev]) return sms[dev];
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    n &= ~1;
    if (dev < 16) sms[dev] = n;
    return n;
}

// Estimated time of one wave of tiles (us): per k a part for the weight rows and a part that grows with the token rows (measured at K = 4096:
// 25.4 us for 256 token rows, 14.2 us for 128), and a fixed part that keeps short products on wide tiles (32 experts of 512 rows, K = 1024:
// 236 us with 256 token rows, 249 us with 160).
inline double wave_us(int bt, int64_t K) { return (3.0 + 0.0875 * bt) * (double)K / 4096.0 + 0.6; }

// Token rows per tile: the size whose last wave is not nearly empty and whose rows are not padding.  tiles(bt): number of tiles of the step
template <class Tiles>
inline int pick_bt(int64_t pairs, int64_t K, Tiles tiles) {
    int best = MAX_BT;
    double best_t = 0;
    for (int bt = MAX_BT; bt >= 32; bt -= 16) {
        const double t = (double)((tiles(bt) + pairs - 1) / pairs) * wave_us(bt, K);
        if (bt == MAX_BT || t < best_t) best = bt, best_t = t;
    }
    return best;
}

// w: [w_rows][K] (row stride ldw), x: [p.M][K] (row stride ldx); p.bt is set, p.MT / p.NT are filled in here; PARTS: K cut into p.parts runs; GROUPED: p.offs
template <bool PARTS = false, bool GROUPED = false, class Epi>
cudaError_t launch(const void* w, int64_t w_rows, int64_t ldw, const void* x, int64_t ldx, Args p, const Epi& epi, cudaStream_t st, bool pdl = false) {
    CUtensorMap mw, mx;
    if (!make_map(&mw, w, w_rows, p.K, ldw, ROWS, p.bf16 != 0) || !make_map(&mx, x, p.M, p.K, ldx, x_box(p), p.bf16 != 0)) return cudaErrorInvalidValue;
    static bool ready[16] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 16 || !ready[dev]) {
        e = cudaFuncSetAttribute(pair_gemm_kernel<Epi, PARTS, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return e;
        if (dev < 16) ready[dev] = true;
    }
    p.MT = (p.M + p.bt - 1) / p.bt + (p.offs ? p.E : 0);
    p.NT = (p.N + 2 * ROWS - 1) / (2 * ROWS);
    int64_t ctas = 2 * (int64_t)p.MT * p.NT * (PARTS ? p.parts : 1);
    const int sms = pair_sms();
    if (ctas > sms) ctas = sms;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas), cfg.blockDim = dim3(THREADS<Epi>), cfg.dynamicSmemBytes = SMEM, cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization, attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = pdl ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, pair_gemm_kernel<Epi, PARTS, GROUPED>, mw, mx, p, epi);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace tcpair
