// seq_attn_tc.cu -- the attend step of prompt portions on the 5th-generation tensor cores, at 32-bit accuracy.
//
// The design asks for scores, weights and sums in 32 bits, so every f32 operand is split into three bf16 parts (x = x1 + x2 + x3, 24 bits) and
// a product runs as the six tcgen05.mma products that matter (x1y3, x3y1, x2y2, x1y2, x2y1, x1y1 -- smallest first, so that the tensor core's
// truncating f32 accumulation costs what the last product's few steps cost).  What is left out is below 2^-24 of the product.  The values of
// 64 keys at a time leave the tensor core and are summed over the key tiles by f32 adds in registers.  Error against 64 bits, 4096 tokens,
// heads of 64, chunks of 2048: see the test; no larger than that of the f32 multiply-add tiles (seq_attn.cu) that this replaces for steps
// of more than 16 tokens.
//
// One CTA works on MT tiles of 128 (token, query head) rows of one key head against tiles of 64 keys.  MT = 2 (heads up to 64): the two row
// tiles alternate, one in the soft-max while the other is in the tensor pipe; MT = 1 (heads up to 128): consecutive key tiles alternate.
//   warps 0 .. 4 MT - 1    soft-max: a thread owns a row -- its maximum, sum and value sums stay in registers, nothing is shuffled
//   next 4 warps           loaders: K and V rows through the block table, split into bf16 planes, 128-byte swizzled (K: k-major, V: mn-major)
//   last 4 warps           the first of them issues the MMAs
// Register split (setmaxnreg, per thread): launched with 128 (MT = 2) or 168 (MT = 1) for all; soft-max 184 / 240, loaders 104 / 120, issuer 40: the
// sums (2 * 184 + 104 + 40 = 4 * 128, 240 + 120 + 40 < 3 * 168) stay within what the block was launched with.
// TMEM: two slots of 96 columns (scores f32 [64], then the weights' three planes in the same columns), the value tile of every row tile,
// and the queries' planes (the A operand of the scores comes from TMEM: from shared memory its reads alone would take longer than the MMA).
// What bounds it: the tensor pipe, 6 x the products (D = V = 64: 1536 cycles per 128 x 64 scores), with the soft-max beside it at about 10
// instructions per score.
//
// Values that are not finite: an infinite key or value part makes the row NaN (inf - inf in the split), where a plain f32 product could still be inf.
// Every wait is bounded (tc_pair.cuh): one that runs out sets bit 1 of the library's error flags and the CTA leaves through the common exit.
#include "seq_attn.cuh"
#include "tc_pair.cuh"

namespace b200seq {

namespace {

using namespace tcpair;

constexpr int KT = 64;                       // keys per tile
constexpr int PLANE = KT * 128;              // bytes of one 64-key x 64-wide plane
constexpr int SLOT_COLS = 96;
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void commit_one(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
                 "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void ld16(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void async_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two values -> three packed bf16 pairs (low half = a)
__device__ __forceinline__ void split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(b), "f"(a));
    const float ra = a - __uint_as_float(p1 << 16), rb = b - __uint_as_float(p1 & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(rb), "f"(ra));
    const float sa_ = ra - __uint_as_float(p2 << 16), sb_ = rb - __uint_as_float(p2 & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p3) : "f"(sb_), "f"(sa_));
}
__device__ __forceinline__ void sts8(uint32_t addr, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory"); }
// mn-major operand, 128-byte swizzle: rows (k) of 128 bytes = 64 consecutive mn, 8-row groups 1024 bytes apart, the next 64 mn `lbo` bytes on
__device__ __forceinline__ uint64_t desc_mn128(uint32_t a, uint32_t lbo) {
    return (uint64_t)((a >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// the keys of one query tile, in the order they are walked: pooled blocks, kept first positions, then the positions from kbeg to hi
struct KeyTiles {
    int kbeg, hi, nbmax, npt, nfirst, nft, total;
};
__device__ __forceinline__ KeyTiles key_tiles(const AttnArgs& a, int p0, int hi) {
    KeyTiles k;
    k.kbeg = a.chunk > 0 ? (p0 / a.chunk) * a.chunk : 0;
    if (a.window > 0) k.kbeg = max(k.kbeg, p0 - a.window + 1);
    k.hi = hi;
    k.nbmax = (a.pool > 0 && hi - a.window + 1 > 0) ? (hi - a.window + 1) / a.pool : 0;
    k.npt = (k.nbmax + KT - 1) / KT;
    const int keep = (a.window > 0 && a.keep_first > 0) ? a.keep_first : 0;
    k.nfirst = min(keep, k.kbeg);
    k.nft = (k.nfirst + KT - 1) / KT;
    k.total = k.npt + k.nft + (hi - k.kbeg) / KT + 1;
    return k;
}

__device__ __forceinline__ int64_t pooled_slot(const int32_t* bt, int bs, int P, int ppp, int b) {
    const int pg = (b * P) / bs;
    return (int64_t)bt[pg] * ppp + (b - (pg * bs + P - 1) / P);
}

template <int MT, int VM>
__global__ void __launch_bounds__((4 * MT + 8) * 32, 1) attn_tc_kernel(const AttnArgs a, const b200seq_step st) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t tmem_base;
    __shared__ int abort_sh;
    __shared__ __align__(8) uint64_t bars[16];
    const uint32_t kv = (sa(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int D = a.D, V = a.V, H = a.H, G = a.G;
    const int KB = (D + 63) >> 6, VB = (V + 63) >> 6;
    const uint32_t kbytes = KB * 3 * PLANE, vbytes = VB * 3 * PLANE, stage = kbytes + vbytes;
    const uint32_t B0 = sa(bars);
    const uint32_t k_full = B0, k_free = B0 + 16, v_full = B0 + 32, v_free = B0 + 48, s_full = B0 + 64, p_ready = B0 + 80, o_full = B0 + 96;
    volatile int* ab = &abort_sh;
    int e, t0, nq;
    // the tiles with the most keys first: a causal step's last tiles see the most
    if (!attn_find_tile(st, (int)gridDim.x - 1 - (int)blockIdx.x, a.QT, e, t0, nq)) return;
    const int g = blockIdx.y / a.HB, hb = blockIdx.y - g * a.HB, R = H / G;
    const int h0 = g * R + hb * a.Rb, nh = min(a.Rb, R - hb * a.Rb);
    const int split = blockIdx.z;
    const int p0 = st.tok_pos[t0], hi = p0 + nq - 1, bs = st.block_size;
    const int32_t* bt = st.block_table + (int64_t)e * st.max_blocks;
    if (hi / bs >= st.max_blocks || p0 < 0) {
        if (threadIdx.x == 0) atomicOr(a.err, 1);
        return;
    }
    const KeyTiles kt = key_tiles(a, p0, hi);
    const int ntile = kt.total > split ? (kt.total - split + a.nsplit - 1) / a.nsplit : 0;   // tiles split, split + nsplit, ...
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            bar_init(k_full + 8 * i, 4), bar_init(k_free + 8 * i, 1), bar_init(v_full + 8 * i, 4), bar_init(v_free + 8 * i, 1);
            bar_init(s_full + 8 * i, 1), bar_init(p_ready + 8 * i, 4), bar_init(o_full + 8 * i, 1);
        }
        bar_init(B0 + 112, 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(sa(&tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_base;
    const uint32_t slot0 = tmem, o0 = tmem + 2 * SLOT_COLS, q0 = o0 + MT * VM;   // columns: slots | value tiles | query planes
    const int qplane = D >> 1, qtile = 3 * qplane;

    if (warp < 4 * MT) {
        // ===================== soft-max: thread == row =====================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MT == 2 ? 184 : 240));
        const int m = warp >> 2, q = warp & 3;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const int r = m * 128 + q * 32 + lane;
        const int tq = r / a.Rb, hr = r - tq * a.Rb;
        const bool live = tq < nq && hr < nh;
        {   // this row's query, split, to TMEM
            const float* src = a.qkvg + (int64_t)(t0 + tq) * a.ld + a.q_col + (int64_t)(h0 + hr) * D;
            const uint32_t qa = q0 + lanes + m * qtile;
            for (int d = 0; d < D; d += 16) {
                uint32_t p1[8], p2[8], p3[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 x = live ? ld4(src + d + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
                    split2(x.x, x.y, p1[2 * j], p2[2 * j], p3[2 * j]);
                    split2(x.z, x.w, p1[2 * j + 1], p2[2 * j + 1], p3[2 * j + 1]);
                }
                st8(qa + (d >> 1), p1), st8(qa + qplane + (d >> 1), p2), st8(qa + 2 * qplane + (d >> 1), p3);
            }
            st_wait();
            fence_before();
        }
        asm volatile("bar.sync 1, %0;" ::"n"((4 * MT + 1) * 32) : "memory");   // the queries are in place (with the MMA warp)
        int rlo = 0, rhi = 0x7fffffff, rnb = 0x7fffffff;   // rows without a token see everything and are not stored
        float rsc = a.scale;
        const int keep = (a.window > 0 && a.keep_first > 0) ? a.keep_first : 0;
        if (live) {
            const int p = p0 + tq;
            rlo = a.chunk > 0 ? (p / a.chunk) * a.chunk : 0;
            if (a.window > 0) rlo = max(rlo, p - a.window + 1);
            rhi = p;
            rnb = (a.pool > 0 && p - a.window + 1 > 0) ? (p - a.window + 1) / a.pool : 0;
            if (a.head_scale) rsc = a.scale * a.head_scale[h0 + hr];
        }
        float mx = -INFINITY, l = 0.f, acc[VM];
#pragma unroll
        for (int c = 0; c < VM; ++c) acc[c] = 0.f;
        bool ok = true;
        for (int j = 0; j < ntile && ok; ++j) {
            const int step = j * MT + m, slot = step & 1;
            const int tile = split + j * a.nsplit;
            const bool pooled = tile < kt.npt, first = !pooled && tile < kt.npt + kt.nft;
            const int k0 = pooled ? tile * KT : (first ? (tile - kt.npt) * KT : kt.kbeg + (tile - kt.npt - kt.nft) * KT);
            const bool whole = __all_sync(0xffffffffu, pooled ? k0 + KT <= rnb : (first ? k0 + KT <= kt.nfirst : (k0 >= rlo && k0 + KT - 1 <= rhi)));
            auto seen = [&](int kp) { return pooled ? kp < rnb : (first ? kp < kt.nfirst : ((kp >= rlo || kp < keep) && kp <= rhi)); };
            const uint32_t S = slot0 + lanes + slot * SLOT_COLS + 32;   // scores: columns 32 .. 95 of the slot
            ok = bar_wait(s_full + 8 * slot, (step >> 1) & 1, ab);
            if (!ok) break;
            fence_after();
            float v[32];
            // score of key c of this 32-key half, as the soft-max sees it
            auto shape = [&](int half) {
#pragma unroll
                for (int c = 0; c < 32; ++c) v[c] *= rsc;
                if (a.softcap > 0.f) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) v[c] = a.softcap * tanhf(v[c] / a.softcap);
                }
                if (!whole) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) v[c] = seen(k0 + 32 * half + c) ? v[c] : -INFINITY;
                }
            };
            float mn = mx;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                ld32(S + 32 * half, v);
                ld_wait();
                shape(half);
                float m0 = v[0], m1 = v[1];
#pragma unroll
                for (int c = 2; c < 32; c += 2) m0 = fmaxf(m0, v[c]), m1 = fmaxf(m1, v[c + 1]);
                mn = fmaxf(mn, fmaxf(m0, m1));
            }
            const float ms = mn == -INFINITY ? 0.f : mn;
            const float mb = ms * LOG2E;
            const float corr = ex2(fmaf(mx, LOG2E, -mb));   // 0 before the first visible key
            mx = mn;
            if (j > 0) {   // the value tile of the key tile before
                const int ps = (step - MT) & 1;
                ok = bar_wait(o_full + 8 * ps, ((step - MT) >> 1) & 1, ab);
                if (!ok) break;
                fence_after();
                const bool same = __all_sync(0xffffffffu, corr == 1.f);
#pragma unroll
                for (int c = 0; c < VM; c += 16) {
                    if (c >= V) break;
                    float o[16];
                    ld16(o0 + lanes + m * VM + c, o);
                    ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[c + i] += o[i];
                    if (!same) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[c + i] *= corr;
                    }
                }
            }
            float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
            for (int half = 0; half < 2; ++half) {   // the weights' planes: columns 48 half + 16 plane (over scores that are no longer needed)
                ld32(S + 32 * half, v);
                ld_wait();
                shape(half);
                uint32_t p1[16], p2[16], p3[16];
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    const float x = ex2(fmaf(v[c], LOG2E, -mb)), y = ex2(fmaf(v[c + 1], LOG2E, -mb));
                    sum0 += x, sum1 += y;
                    split2(x, y, p1[c >> 1], p2[c >> 1], p3[c >> 1]);
                }
                const uint32_t P = slot0 + lanes + slot * SLOT_COLS + 48 * half;
                st16(P, p1), st16(P + 16, p2), st16(P + 32, p3);
            }
            l = fmaf(l, corr, sum0 + sum1);
            st_wait();
            fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(p_ready + 8 * slot);
        }
        if (ok && ntile > 0) {
            const int step = (ntile - 1) * MT + m;
            ok = bar_wait(o_full + 8 * (step & 1), (step >> 1) & 1, ab);
            fence_after();
        }
        if (ok) {
            const int t = t0 + tq, h = h0 + hr;
            float f = 1.f;
            float* pp = nullptr;
            if (a.nsplit == 1) {
                float gate = 1.f, den = l, resc = 1.f;
                if (live && a.gated && !a.gate_elem) gate = sigmoidf_acc(a.gate[(int64_t)t * a.gld + h]);
                if (live && a.sink) {   // the sink's term, under the larger of the two maxima
                    const float sk = a.sink[h], mn = fmaxf(mx, sk);
                    resc = expf(mx - mn);
                    den = fmaf(l, resc, expf(sk - mn));
                }
                f = gate * resc / den;
            } else {
                pp = a.part + (((int64_t)t * H + h) * a.nsplit + split) * (V + 2);
                if (live) pp[0] = mx, pp[1] = l;
            }
#pragma unroll
            for (int c = 0; c < VM; c += 16) {
                if (c >= V) break;
                float o[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = 0.f;
                if (ntile > 0) {
                    ld16(o0 + lanes + m * VM + c, o);
                    ld_wait();
                }
                if (!live) continue;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float x = acc[c + i] + o[i];
                    if (pp) pp[2 + c + i] = x;
                    else o[i] = x * f * (a.gate_elem ? sigmoidf_acc(a.gate[(int64_t)t * a.gld + (int64_t)h * V + c + i]) : 1.f);
                }
                if (!pp) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) store_act4(a.out, a.out_dtype, ((int64_t)t * H + h) * V + c + i, make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]));
                }
            }
        }
    } else if (warp < 4 * MT + 4) {
        // ===================== loaders: 128 threads =====================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MT == 2 ? 104 : 120));
        const int lw = warp - 4 * MT;
        bool ok = true;
        for (int j = 0; j < ntile && ok; ++j) {
            const int s = j & 1;
            const uint32_t ph = ((j >> 1) & 1) ^ 1;
            const int tile = split + j * a.nsplit;
            const bool pooled = tile < kt.npt, first = !pooled && tile < kt.npt + kt.nft;
            const int k0 = pooled ? tile * KT : (first ? (tile - kt.npt) * KT : kt.kbeg + (tile - kt.npt - kt.nft) * KT);
            const int klim = pooled ? kt.nbmax - 1 : (first ? kt.nfirst - 1 : hi);
            // one operand: 16 lanes cover 64 floats of a key's row; `wide` blocks of 64
            auto bring = [&](bool is_v, int width, int wide, uint32_t dst, uint32_t bfull, uint32_t bfree) {
                const int per = 4 / wide * 2;                              // (rows per 8 half-warps) / blocks: 8 keys per pass (one block) or 4 (two)
                const int hw = lw * 2 + (lane >> 4), blk = wide == 2 ? hw & 1 : 0, rowi = wide == 2 ? hw >> 1 : hw;
                const int d = blk * 64 + (lane & 15) * 4;
#pragma unroll 1
                for (int part = 0; part < KT; part += 8 * per) {           // eight rows in flight per thread
                    float4 x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int kp = k0 + part + i * per + rowi;
                        x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (kp <= klim && d < width) {
                            const float* p;
                            if (pooled) p = is_v ? a.vpp + (pooled_slot(bt, bs, a.pool, a.ppp, kp) * G + g) * V : a.kpp + (pooled_slot(bt, bs, a.pool, a.ppp, kp) * G + g) * D;
                            else {
                                const int64_t prow = (int64_t)bt[kp / bs] * bs + kp % bs;
                                if (is_v) p = a.vpool + prow * a.vld + (int64_t)(g / a.vdiv) * V;
                                else p = a.kpool + prow * a.kld + (int64_t)g * D;
                            }
                            x[i] = ld4(p + d);
                        }
                    }
                    if (part == 0) ok = bar_wait(bfree + 8 * s, ph, ab);
                    if (!ok) return;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = part + i * per + rowi;
                        uint32_t a1, a2, a3, b1, b2, b3;
                        split2(x[i].x, x[i].y, a1, a2, a3);
                        split2(x[i].z, x[i].w, b1, b2, b3);
                        const uint32_t at = dst + blk * (3 * PLANE) + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4) + ((lane & 1) << 3);
                        sts8(at, a1, b1), sts8(at + PLANE, a2, b2), sts8(at + 2 * PLANE, a3, b3);
                    }
                }
                async_fence();
                __syncwarp();
                if (lane == 0) bar_arrive(bfull + 8 * s);
            };
            const uint32_t base = kv + s * stage;
            bring(false, D, KB, base, k_full, k_free);
            if (ok) bring(true, V, VB, base + kbytes, v_full, v_free);
        }
    } else {
        // ===================== MMA issuer =====================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 4 * MT + 4) asm volatile("bar.sync 1, %0;" ::"n"((4 * MT + 1) * 32) : "memory");
        if (warp == 4 * MT + 4 && elect()) {
            fence_after();
            const uint32_t ids = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(KT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
            const uint32_t ido = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(V >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // B is mn-major
            const int PX[6] = {0, 2, 1, 0, 1, 0}, PY[6] = {2, 0, 1, 1, 0, 0};   // smallest products first
            const int steps = ntile * MT;
            bool ok = true;
            auto scores = [&](int step) {
                const int j = step / MT, m = step - j * MT, s = j & 1, slot = step & 1;
                ok = bar_wait(k_full + 8 * s, (j >> 1) & 1, ab);
                if (!ok) return;
                fence_after();
                const uint32_t kb = kv + s * stage, d = slot0 + slot * SLOT_COLS + 32;
                uint32_t acc_ = 0;
#pragma unroll
                for (int pr = 0; pr < 6; ++pr)
                    for (int kk = 0; kk < D / 16; ++kk) {
                        const uint64_t b = desc_k128(kb + (kk >> 2) * (3 * PLANE) + PY[pr] * PLANE) + 2 * (kk & 3);
                        mma_ts(d, q0 + m * qtile + PX[pr] * qplane + kk * 8, b, ids, acc_);
                        acc_ = 1;
                    }
                commit_one(s_full + 8 * slot);
                if (m == MT - 1 && j + 2 < ntile) commit_one(k_free + 8 * s);   // (nobody waits for the last ones)
            };
            if (steps > 0) scores(0);
            for (int step = 0; step < steps && ok; ++step) {
                if (step + 1 < steps) {
                    if (step >= 1) {   // the other slot's weights have been read
                        ok = bar_wait(o_full + 8 * ((step - 1) & 1), ((step - 1) >> 1) & 1, ab);
                        if (!ok) break;
                    }
                    scores(step + 1);
                    if (!ok) break;
                }
                const int j = step / MT, m = step - j * MT, s = j & 1, slot = step & 1;
                ok = bar_wait(v_full + 8 * s, (j >> 1) & 1, ab) && bar_wait(p_ready + 8 * slot, (step >> 1) & 1, ab);
                if (!ok) break;
                fence_after();
                const uint32_t vb = kv + s * stage + kbytes, d = o0 + m * VM;
                uint32_t acc_ = 0;
#pragma unroll
                for (int pr = 0; pr < 6; ++pr)
#pragma unroll
                    for (int kk = 0; kk < KT / 16; ++kk) {
                        const uint64_t b = desc_mn128(vb + PY[pr] * PLANE + kk * 2048, 3 * PLANE);
                        mma_ts(d, slot0 + slot * SLOT_COLS + 48 * (kk >> 1) + 16 * PX[pr] + 8 * (kk & 1), b, ido, acc_);
                        acc_ = 1;
                    }
                commit_one(o_full + 8 * slot);
                if (m == MT - 1 && j + 2 < ntile) commit_one(v_free + 8 * s);
            }
            if (!ok) {   // what was issued reads shared memory and TMEM: wait for it (bounded) before the CTA goes
                commit_one(B0 + 112);
                const unsigned long long t0_ = now_ns();
                while (!bar_try(B0 + 112, 0) && now_ns() - t0_ < WAIT_NS) {}
            }
        }
        __syncwarp();
    }
    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && abort_sh) atomicOr(a.err, 2);
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

template <int MT, int VM>
cudaError_t run(const AttnArgs& a, const b200seq_step& st, dim3 grid, cudaStream_t cs) {
    const int KB = (a.D + 63) / 64, VB = (a.V + 63) / 64;
    int smem = 2 * (KB + VB) * 3 * PLANE + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;   // one CTA per SM: it takes all of TMEM
    static int ready[16] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 16 || ready[dev] < smem) {
        e = cudaFuncSetAttribute(attn_tc_kernel<MT, VM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev < 16) ready[dev] = smem;
    }
    attn_tc_kernel<MT, VM><<<grid, (4 * MT + 8) * 32, smem, cs>>>(a, st);
    return cudaGetLastError();
}

}  // namespace

// Steps of more than 16 tokens with whole 16-byte rows and head sizes up to 128 in steps of 16.  What stays on the f32 tiles of seq_attn.cu:
// decode steps (too few rows for a 128-row tile), keys that come in two parts or from gathered rows, odd head sizes, unaligned rows.
bool launch_attn_tc(AttnArgs& a, const b200seq_step& st, int max_keys, size_t part_floats, cudaStream_t cs, int& rc) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const int R = a.H / a.G;
    if (st.T <= 16 || a.D % 16 || a.V % 16 || a.D > 128 || a.V > 128 || a.ctx_rows || a.krot || a.kd != a.D || ((a.ld | a.kld | a.vld | a.q_col) & 3) || !al(a.qkvg) ||
        !al(a.kpool) || !al(a.vpool) || (a.pool > 0 && (!al(a.kpp) || !al(a.vpp))) || !al(a.out))
        return false;
    const int sms = tcpair::pair_sms();
    if (sms < 1) return false;
    const int64_t rows = (int64_t)st.T * a.H;
    // two row tiles per CTA where the heads are small enough and there are rows for it
    const int mt = a.D <= 64 && a.V <= 64 && rows >= 256ll * sms ? 2 : 1;
    const int RQ = 128 * mt;
    a.Rb = R < RQ ? R : RQ;
    a.HB = (R + a.Rb - 1) / a.Rb;
    a.QT = RQ / a.Rb;
    const int tiles = (st.T + a.QT - 1) / a.QT + st.B - (st.B == 1);   // upper bound of the step's query tiles (exact for one entry)
    const int64_t real = (int64_t)((st.T + a.QT - 1) / a.QT) * a.G * a.HB;
    int64_t ns = 1;
    if (2 * real <= sms) {   // too few tiles: deal the key tiles to several CTAs, at least four each
        ns = sms / real;
        const int64_t most = (max_keys / KT) / 4, fits = a.part ? (int64_t)(part_floats / ((size_t)st.T * a.H * (a.V + 2))) : 0;
        ns = ns < most ? ns : most;
        ns = ns < fits ? ns : fits;
        ns = ns > 32 ? 32 : (ns < 1 ? 1 : ns);
    }
    a.nsplit = (int)ns;
    const dim3 grid(tiles, a.G * a.HB, (unsigned)ns);
    cudaError_t e;
    if (mt == 2) e = run<2, 64>(a, st, grid, cs);
    else if (a.V <= 64) e = run<1, 64>(a, st, grid, cs);
    else e = run<1, 128>(a, st, grid, cs);
    if (e != cudaSuccess) {
        rc = cuda_status(e, "attn tc");
        return true;
    }
    count_launch();
    rc = 0;
    return true;
}

}  // namespace b200seq
