// seq_attn_tc.cu -- the attend step of prompt portions on the 5th-generation tensor cores, at 32-bit accuracy.
//
// The design asks for scores, weights and sums in 32 bits, so every f32 operand is split into three bf16 parts (x = x1 + x2 + x3, 24 bits) and
// a product runs as the six tcgen05.mma products that matter (x1y3, x3y1, x2y2, x1y2, x2y1, x1y1 -- smallest first, so that the tensor core's
// truncating f32 accumulation costs what the last product's few steps cost).  What is left out is below 2^-24 of the product.  The values of
// 64 keys at a time leave the tensor core and are summed over the key tiles by f32 adds in registers.  Error against 64 bits, 4096 tokens,
// heads of 64, chunks of 2048: 2.0e-7, that of the f32 multiply-add tiles (seq_attn.cu) that this replaces for steps of more than 16 tokens 3.9e-7.
//
// One CTA works on MT tiles of 128 (token, query head) rows of one key head against tiles of 64 keys.  MT = 2 (heads up to 64): the two row
// tiles alternate, one in the soft-max while the other is in the tensor pipe; MT = 1 (heads up to 128): consecutive key tiles alternate.
//   warps 0 .. 4 MT - 1    soft-max: a thread owns a row -- its maximum, sum and value sums stay in registers, nothing is shuffled
//   next 8 warps           loaders: K and V rows through the block table, split into bf16 planes, 128-byte swizzled (K: k-major, V: mn-major)
//   last 4 warps           the first of them issues the MMAs
// Register split (setmaxnreg, per thread): launched with 96 (MT = 2) or 128 (MT = 1) for all; soft-max 160 / 240, loaders 64 / 104, issuer 32 / 64:
// the sums (2 * 160 + 2 * 64 + 32 = 5 * 96, 240 + 2 * 104 + 64 = 4 * 128) are what the block was launched with.
// TMEM: two slots of 96 columns (scores f32 [64], then the weights' three planes in the same columns), the value tile of every row tile,
// and the queries' planes (the A operand of the scores comes from TMEM: from shared memory its reads alone would take longer than the MMA).
// What bounds it: the tensor pipe, 6 x the products (D = V = 64: 1536 cycles per 128 x 64 scores; a step takes 2 400, the difference being the
// hand-overs between a value product and the next scores of the same slot), with the soft-max beside it on the same schedulers.
//
// Values without such parts (infinities, NaN, beyond the bf16 range): a part that is not finite would reach rows that do not see its key (0 x inf)
// and make infinities NaN.  Any such part leaves a NaN in every row that meets it -- a key's in its scores, a value's in its column, whatever the weight --
// so a row that ends with a sum that is not finite is made again, by plain f32 sums over the keys it sees (plain_row).
// Every wait is bounded (tc_pair.cuh): one that runs out sets bit 1 of the library's error flags and the CTA leaves through the common exit.
#include "seq_attn.cuh"
#include "tc_split.cuh"

namespace b200seq {

namespace {

using namespace tcsplit;

constexpr int KT = 64;                       // keys per tile
constexpr int PLANE = KT * 128;              // bytes of one 64-key x 64-wide plane
constexpr int SLOT_COLS = 96;
constexpr float LOG2E = 1.4426950408889634f;

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

// One (token, query head) row by plain f32 sums over the keys it sees in the tiles of a split, maximum first, then weights and sums, as the f32 tiles have
// it (seq_attn.cu).  Called after the row's results are stored; out of line, so that nothing it needs is kept through the loops.
__device__ __noinline__ void plain_row(const AttnArgs& a, const b200seq_step& st, int e, int p0, int hi, int t, int h, int split) {
    const int D = a.D, V = a.V, G = a.G, g = h / (a.H / G), bs = st.block_size, p = st.tok_pos[t];
    const int32_t* bt = st.block_table + (int64_t)e * st.max_blocks;
    const KeyTiles kt = key_tiles(a, p0, hi);
    const int keep = (a.window > 0 && a.keep_first > 0) ? a.keep_first : 0;
    int lo = a.chunk > 0 ? (p / a.chunk) * a.chunk : 0;
    if (a.window > 0) lo = max(lo, p - a.window + 1);
    const int nb = (a.pool > 0 && p - a.window + 1 > 0) ? (p - a.window + 1) / a.pool : 0;
    const float sc = a.head_scale ? a.scale * a.head_scale[h] : a.scale;
    const float* q = a.qkvg + (int64_t)t * a.ld + a.q_col + (int64_t)h * D;
    float mx = -INFINITY, l = 0.f, f = 1.f;
    float* pp = a.nsplit > 1 ? a.part + (((int64_t)t * a.H + h) * a.nsplit + split) * (V + 2) : nullptr;
    for (int c = -16; c < V; c += 16) {   // first pass: the maximum; then 16 columns at a time (the first of them with the sum of the weights)
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        for (int tile = split; tile < kt.total; tile += a.nsplit) {
            const bool pooled = tile < kt.npt, first = !pooled && tile < kt.npt + kt.nft;
            const int k0 = pooled ? tile * KT : (first ? (tile - kt.npt) * KT : kt.kbeg + (tile - kt.npt - kt.nft) * KT);
            for (int kp = k0; kp < k0 + KT; ++kp) {
                if (!(pooled ? kp < nb : (first ? kp < kt.nfirst : (kp >= lo || kp < keep) && kp <= p))) continue;
                const int64_t row = pooled ? pooled_slot(bt, bs, a.pool, a.ppp, kp) : (int64_t)bt[kp / bs] * bs + kp % bs;
                const float* k = pooled ? a.kpp + (row * G + g) * D : a.kpool + row * a.kld + (int64_t)g * D;
                float s = 0.f;
#pragma unroll 4
                for (int d = 0; d < D; d += 4) {
                    const float4 x = ld4(q + d), y = ld4(k + d);
                    s = fmaf(x.x, y.x, s), s = fmaf(x.y, y.y, s), s = fmaf(x.z, y.z, s), s = fmaf(x.w, y.w, s);
                }
                s *= sc;
                if (s != s) return;   // the row is NaN, and so is what has been stored
                if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
                if (s == -INFINITY) continue;
                if (c < 0) {
                    mx = fmaxf(mx, s);
                    continue;
                }
                const float w = expf(s - mx), *v = (pooled ? a.vpp + (row * G + g) * V : a.vpool + row * a.vld + (int64_t)(g / a.vdiv) * V) + c;
                if (c == 0) l += w;
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[i] = fmaf(w, v[i], acc[i]);
            }
        }
        if (c < 0) continue;
        if (c == 0) {
            if (pp) {
                pp[0] = mx, pp[1] = l;
            } else {
                float gate = 1.f, den = l, resc = 1.f;
                if (a.gated && !a.gate_elem) gate = sigmoidf_acc(a.gate[(int64_t)t * a.gld + h]);
                if (a.sink) {
                    const float sk = a.sink[h], mn = fmaxf(mx, sk);
                    resc = expf(mx - mn);
                    den = fmaf(l, resc, expf(sk - mn));
                }
                f = gate * resc / den;
            }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (pp) pp[2 + c + i] = acc[i];
            else store_act(a.out, a.out_dtype, ((int64_t)t * a.H + h) * V + c + i, acc[i] * f * (a.gate_elem ? sigmoidf_acc(a.gate[(int64_t)t * a.gld + (int64_t)h * V + c + i]) : 1.f));
        }
    }
}

// DK: head size / 16, or 0 for a run-time one; CAP: scores are soft-capped.  The loops are kept short: with the soft-max in two unrolled passes,
// two copies of the loader and the issuer unrolled over four steps the kernel waited for instructions (ncu: no_instruction the largest stall,
// 0.21 instructions per cycle) and took 860 us where it now takes 206 (4096 tokens, 32 heads of 64, chunks of 2048; the f32 tiles: 1 656).
template <int MT, int VM, int DK, bool CAP>
__global__ void __launch_bounds__((4 * MT + 12) * 32, 1) attn_tc_kernel(const __grid_constant__ AttnArgs a, const __grid_constant__ b200seq_step st) {
    chain_enter();
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t tmem_base;
    __shared__ int abort_sh;
    __shared__ __align__(8) uint64_t bars[16];
    const uint32_t kv = (sa(smem_raw) + 1023u) & ~1023u;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // warp-uniform: the roles branch on it
    const int D = a.D, V = a.V, H = a.H, G = a.G;
    const int KB = (D + 63) >> 6, VB = (V + 63) >> 6;
    const uint32_t kbytes = KB * 3 * PLANE, vbytes = VB * 3 * PLANE, stage = kbytes + vbytes;
    const uint32_t B0 = sa(bars);
    const uint32_t k_full = B0, k_free = B0 + 16, v_full = B0 + 32, v_free = B0 + 48, s_full = B0 + 64, p_ready = B0 + 80, o_full = B0 + 96;
    volatile int* ab = &abort_sh;
    int e, t0, nq;
    // The tiles with the most keys first, for all heads at once, so that the last CTAs to start are short: a causal step's last tiles see the
    // most, in a step of chunks the last ones of every chunk.
    const int units = G * a.HB, n = (int)gridDim.x / units, r = (int)blockIdx.x / units, unit = (int)blockIdx.x - r * units;
    int tile_no = n - 1 - r;
    if (a.chunk > 0 && a.chunk % a.QT == 0 && a.chunk / a.QT < n) {
        const int per = a.chunk / a.QT, nc = (n + per - 1) / per, rem = n - (nc - 1) * per, longer = (per - rem) * (nc - 1);
        if (r < longer) tile_no = (r % (nc - 1)) * per + per - 1 - r / (nc - 1);
        else tile_no = ((r - longer) % nc) * per + rem - 1 - (r - longer) / nc;
    }
    if (!attn_find_tile(st, tile_no, a.QT, e, t0, nq)) return;
    const int g = unit / a.HB, hb = unit - g * a.HB, R = H / G;
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
            bar_init(k_full + 8 * i, 8), bar_init(k_free + 8 * i, 1), bar_init(v_full + 8 * i, 8), bar_init(v_free + 8 * i, 1);
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
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(MT == 2 ? 160 : 240));
        const int m = warp >> 2, q = warp & 3;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const int r = m * 128 + q * 32 + lane;
        const int tq = r / a.Rb, hr = r - tq * a.Rb;
        const bool live = tq < nq && hr < nh;
        int rlo = 0, rhi = 0x3fffffff, rnb = 0x3fffffff;   // rows without a token see everything and are not stored
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
        // soft-max in base 2 over raw scores: weight = 2^(c s - mb), mb = c max(s); the sign of the scale goes into the query.  With a soft cap
        // the scores are scaled and capped first (CAP) and c is log2 e alone.
        const float sgn = rsc < 0.f ? -1.f : 1.f;
        const float c = CAP ? LOG2E : fmaxf(fabsf(rsc) * LOG2E, 1e-37f);
        {   // this row's query, split, to TMEM
            const float* src = a.qkvg + (int64_t)(t0 + tq) * a.ld + a.q_col + (int64_t)(h0 + hr) * D;
            const uint32_t qa = q0 + lanes + m * qtile;
#pragma unroll 1
            for (int d = 0; d < D; d += 16) {
                float4 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = live ? ld4(src + d + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
                uint32_t p1[8], p2[8], p3[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    split2(x[j].x * sgn, x[j].y * sgn, p1[2 * j], p2[2 * j], p3[2 * j]);
                    split2(x[j].z * sgn, x[j].w * sgn, p1[2 * j + 1], p2[2 * j + 1], p3[2 * j + 1]);
                }
                st8(qa + (d >> 1), p1), st8(qa + qplane + (d >> 1), p2), st8(qa + 2 * qplane + (d >> 1), p3);
            }
            st_wait();
            fence_before();
        }
        asm volatile("bar.sync 1, %0;" ::"n"((4 * MT + 1) * 32) : "memory");   // the queries are in place (with the MMA warp)
        const uint64_t cc = pk(c, c), minus1 = pk(-1.f, -1.f);
        float mx = -INFINITY, mb = -INFINITY, l = 0.f;
        uint64_t acc[VM / 2];
#pragma unroll
        for (int i = 0; i < VM / 2; ++i) acc[i] = 0;
        bool ok = true;
        auto add_values = [&](int step) {   // acc += the value tile of a step
            ok = bar_wait<false>(o_full + 8 * (step & 1), (step >> 1) & 1, ab);
            if (!ok) return false;
            fence_after();
#pragma unroll
            for (int i = 0; i < VM; i += 32) {
                if (i >= V) break;
                float o[32];
                ld32(o0 + lanes + m * VM + i, o);     // (V = 16 or 48: the columns beyond are not used)
                ld_wait();
#pragma unroll
                for (int u = 0; u < 32; u += 2) acc[(i + u) >> 1] = add2(acc[(i + u) >> 1], pk(o[u], o[u + 1]));
            }
            fence_before();
            return true;
        };
#pragma unroll 1
        for (int j = 0; j < ntile && ok; ++j) {
            const int step = j * MT + m, slot = step & 1;
            const int tile = split + j * a.nsplit;
            const bool pooled = tile < kt.npt, first = !pooled && tile < kt.npt + kt.nft;
            const int k0 = pooled ? tile * KT : (first ? (tile - kt.npt) * KT : kt.kbeg + (tile - kt.npt - kt.nft) * KT);
            // visible keys of this row, relative to the tile: [lo, hi1) and, in the window's tiles, those below `kp`
            const int lo = pooled || first ? 0 : rlo - k0, hi1 = (pooled ? rnb : (first ? kt.nfirst : rhi + 1)) - k0, kp = pooled || first ? 0 : keep - k0;
            const bool whole = __all_sync(0xffffffffu, lo <= 0 && hi1 >= KT);
            const uint32_t S = slot0 + lanes + slot * SLOT_COLS + 32;   // scores: columns 32 .. 95 of the slot
            ok = bar_wait<false>(s_full + 8 * slot, (step >> 1) & 1, ab);
            if (!ok) break;
            fence_after();
            float v[KT];
            ld32(S, v);
            ld32(S + 32, v + 32);
            ld_wait();
            if (CAP) {
#pragma unroll
                for (int i = 0; i < KT; ++i) v[i] = a.softcap * tanhf(v[i] * fabsf(rsc) / a.softcap);
            }
            if (!whole) {
                auto below = [](int n) { return n <= 0 ? 0u : (n >= 32 ? 0xffffffffu : (1u << n) - 1u); };
                const uint32_t s0 = (below(hi1) & ~below(lo)) | (below(hi1) & below(kp)), s1 = (below(hi1 - 32) & ~below(lo - 32)) | (below(hi1 - 32) & below(kp - 32));
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    v[i] = (s0 >> i) & 1u ? v[i] : -INFINITY;
                    v[32 + i] = (s1 >> i) & 1u ? v[32 + i] : -INFINITY;
                }
            }
            float m0 = fmaxf(v[0], v[1]), m1 = fmaxf(v[2], v[3]);
#pragma unroll
            for (int i = 4; i < KT; i += 4) m0 = fmaxf(m0, fmaxf(v[i], v[i + 1])), m1 = fmaxf(m1, fmaxf(v[i + 2], v[i + 3]));
            mx = fmaxf(mx, fmaxf(m0, m1));
            const float mbn = mx * c;
            const float corr = mx == -INFINITY ? 1.f : ex2(mb - mbn);   // 0 at the first visible key
            mb = mbn;
            const float off = mx == -INFINITY ? 0.f : -mbn;
            const uint64_t off2 = pk(off, off);
            uint64_t sum = 0;
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {   // the weights' planes: columns 48 half + 16 plane (over the scores, which are in registers)
                uint32_t p1[8], p2[8], p3[8];
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    float x, y;
                    upk(fma2(pk(v[16 * q4 + i], v[16 * q4 + i + 1]), cc, off2), x, y);
                    x = ex2(x), y = ex2(y);
                    sum = add2(sum, pk(x, y));
                    cut2(x, y, minus1, p1[i >> 1], p2[i >> 1], p3[i >> 1]);
                }
                const uint32_t P = slot0 + lanes + slot * SLOT_COLS + 48 * (q4 >> 1) + 8 * (q4 & 1);
                st8(P, p1), st8(P + 16, p2), st8(P + 32, p3);
            }
            float sx, sy;
            upk(sum, sx, sy);
            l = fmaf(l, corr, sx + sy);
            const uint64_t corr2 = pk(corr, corr);
            const bool same = __all_sync(0xffffffffu, corr == 1.f);
            // MT = 1: the value tile of the key tile before, whose product ran beside this soft-max
            if (MT == 1 && j > 0 && !add_values(step - 1)) break;
            if (!same) {
#pragma unroll
                for (int i = 0; i < VM / 2; ++i) acc[i] = mul2(acc[i], corr2);
            }
            st_wait();
            fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(p_ready + 8 * slot);
            // MT = 2: this key tile's, while the next scores are made (the other row tile keeps the tensor pipe busy)
            if (MT == 2 && !add_values(step)) break;
        }
        if (!CAP && mx != -INFINITY) mx = mb / LOG2E;   // in the units of the scores, for the sink and the merge of key splits
        if (MT == 1 && ok && ntile > 0) add_values(ntile - 1);
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
            uint64_t odd = pk(l * 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < VM / 2; ++i)
                if (2 * i < V) odd = fma2(acc[i], 0, odd);
            float odd0, odd1;
            upk(odd, odd0, odd1);
#pragma unroll
            for (int cb = 0; cb < VM; cb += 16) {
                if (cb >= V) break;
                float o[16];
                if (!live) continue;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float x, x1;
                    upk(acc[(cb + i) >> 1], x, x1);
                    x = (i & 1) ? x1 : x;
                    if (pp) pp[2 + cb + i] = x;
                    else o[i] = x * f * (a.gate_elem ? sigmoidf_acc(a.gate[(int64_t)t * a.gld + (int64_t)h * V + cb + i]) : 1.f);
                }
                if (!pp) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) store_act4(a.out, a.out_dtype, ((int64_t)t * H + h) * V + cb + i, make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]));
                }
            }
            if (live && !(odd0 + odd1 == 0.f)) plain_row(a, st, e, p0, hi, t, h, split);   // a sum that is not finite
        }
    } else if (warp < 4 * MT + 8) {
        // ===================== loaders: 256 threads =====================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MT == 2 ? 64 : 104));
        // A unit is one operand's 64-wide block of a tile, or (two blocks wide) half of its keys: four 16-byte pieces per thread, 16 lanes to a
        // key's 64 floats.  The next unit's loads are in flight while this one is split and stored, and the page lookups run a tile ahead
        // (one key per lane, handed round by shuffles).
        const int lw = warp - 4 * MT, nu = KB + VB;
        const int hw = lw * 2 + (lane >> 4), c4 = lane & 15;
        const int shift = (bs & (bs - 1)) == 0 ? 31 - __clz(bs) : -1;
        struct TileAt {
            int k0, klim;
            bool pooled;
        };
        auto tile_at = [&](int j) {
            const int tile = split + j * a.nsplit;
            TileAt t;
            t.pooled = tile < kt.npt;
            const bool first = !t.pooled && tile < kt.npt + kt.nft;
            t.k0 = t.pooled ? tile * KT : (first ? (tile - kt.npt) * KT : kt.kbeg + (tile - kt.npt - kt.nft) * KT);
            t.klim = t.pooled ? kt.nbmax - 1 : (first ? kt.nfirst - 1 : hi);
            return t;
        };
        auto lookup = [&](const TileAt& t, int key) {       // pool row of a key of the tile (keys beyond the last one: a valid row, its values become zero)
            const int kp = min(t.k0 + key, t.klim);
            if (t.pooled) return (int)pooled_slot(bt, bs, a.pool, a.ppp, kp);
            return shift >= 0 ? bt[kp >> shift] * bs + (kp & (bs - 1)) : bt[kp / bs] * bs + kp % bs;
        };
        struct Piece {
            int row0, per, d;
            bool is_v;
        };
        auto piece = [&](int u) {
            Piece p;
            p.is_v = u >= KB;
            const int wide = p.is_v ? VB : KB, pu = p.is_v ? u - KB : u;
            p.per = wide == 2 ? 8 : 16;                      // keys per pass of the sixteen half-warps
            p.row0 = pu * 32 + (wide == 2 ? hw >> 1 : hw);
            p.d = (wide == 2 ? (hw & 1) * 64 : 0) + c4 * 4;
            return p;
        };
        auto fetch = [&](const TileAt& t, int u, int ra, int rb, float4 (&x)[4]) {
            const Piece p = piece(u);
            const int width = p.is_v ? V : D;
            const float* base = t.pooled ? (p.is_v ? a.vpp + (int64_t)g * V : a.kpp + (int64_t)g * D) : (p.is_v ? a.vpool + (int64_t)(g / a.vdiv) * V : a.kpool + (int64_t)g * D);
            const int64_t ld = t.pooled ? (int64_t)G * width : (p.is_v ? a.vld : a.kld);
            base += p.d < width ? p.d : 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = p.row0 + i * p.per;          // all keys of a warp in one pass lie in the same half
                const int row = __shfl_sync(0xffffffffu, key < 32 ? ra : rb, key & 31);
                x[i] = ld4(base + row * ld);
            }
        };
        TileAt t = tile_at(0), tn = t;
        int ra = 0, rb = 0, na = 0, nb = 0;
        float4 cur[4], nxt[4];
        if (ntile > 0) {
            ra = lookup(t, lane), rb = lookup(t, lane + 32);
            fetch(t, 0, ra, rb, nxt);
        }
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < ntile && ok; ++j) {
            const int s = j & 1;
            const bool more = j + 1 < ntile;
            if (more) tn = tile_at(j + 1), na = lookup(tn, lane), nb = lookup(tn, lane + 32);
#pragma unroll 1
            for (int u = 0; u < nu; ++u) {
#pragma unroll
                for (int i = 0; i < 4; ++i) cur[i] = nxt[i];
                const bool here = u + 1 < nu;
                if (here || more) fetch(here ? t : tn, here ? u + 1 : 0, here ? ra : na, here ? rb : nb, nxt);
                const Piece p = piece(u);
                const int width = p.is_v ? V : D;
                if (u == 0 || u == KB) {
                    ok = bar_wait<false>((p.is_v ? v_free : k_free) + 8 * s, ((j >> 1) & 1) ^ 1, ab);
                    if (!ok) break;
                }
                uint32_t at = kv + s * stage + (p.is_v ? kbytes : 0) + (p.d >> 6) * (3 * PLANE) + p.row0 * 128 + (((c4 >> 1) ^ (p.row0 & 7)) << 4) + ((c4 & 1) << 3);
                if (t.k0 + KT - 1 > t.klim || p.d >= width) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (t.k0 + p.row0 + i * p.per > t.klim || p.d >= width) cur[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {              // (the row's place in the swizzle is the same in every pass)
                    uint32_t a1, a2, a3, b1, b2, b3;
                    split2(cur[i].x, cur[i].y, a1, a2, a3);
                    split2(cur[i].z, cur[i].w, b1, b2, b3);
                    sts8(at, a1, b1), sts8(at + PLANE, a2, b2), sts8(at + 2 * PLANE, a3, b3);
                    at += p.per * 128;
                }
                if (u == KB - 1 || u == nu - 1) {
                    async_fence();
                    __syncwarp();
                    if (lane == 0) bar_arrive((p.is_v ? v_full : k_full) + 8 * s);
                }
            }
            t = tn, ra = na, rb = nb;
        }
    } else {
        // ===================== MMA issuer =====================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MT == 2 ? 32 : 64));
        if (warp == 4 * MT + 8) asm volatile("bar.sync 1, %0;" ::"n"((4 * MT + 1) * 32) : "memory");
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        if (warp == 4 * MT + 8 && elect()) {
            fence_after();
            constexpr uint32_t ids = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(KT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
            const uint32_t ido = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(V >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // B is mn-major
            constexpr uint32_t O0 = 2 * SLOT_COLS, Q0 = O0 + MT * VM;
            const int steps = ntile * MT, nkk = DK ? DK : D / 16;
            const uint32_t qp = DK ? DK * 8 : (uint32_t)qplane;
            bool ok = true;
            auto scores = [&](int step) {
                const int j = step / MT, s = j & 1, slot = step & 1, m = MT == 2 ? slot : 0;
                ok = bar_wait<false>(k_full + 8 * s, (j >> 1) & 1, ab);
                if (!ok) return;
                fence_after();
                const uint64_t kb = desc_k128(kv + s * stage);
                const uint32_t d = tm + slot * SLOT_COLS + 32, qa = tm + Q0 + m * 3 * qp;
#pragma unroll
                for (int pr = 0; pr < 6; ++pr) {
                    constexpr int PX[6] = {0, 2, 1, 0, 1, 0}, PY[6] = {2, 0, 1, 1, 0, 0};   // smallest products first
                    if (DK) {
#pragma unroll
                        for (int kk = 0; kk < DK; ++kk)
                            mma_ts(d, qa + PX[pr] * qp + kk * 8, kb + (uint64_t)(((kk >> 2) * (3 * PLANE) + PY[pr] * PLANE) / 16 + 2 * (kk & 3)), ids, (pr | kk) != 0 ? 1u : 0u);
                    } else {
#pragma unroll 1
                        for (int kk = 0; kk < nkk; ++kk)
                            mma_ts(d, qa + PX[pr] * qp + kk * 8, kb + (uint64_t)(((kk >> 2) * (3 * PLANE) + PY[pr] * PLANE) / 16 + 2 * (kk & 3)), ids, (pr | kk) != 0 ? 1u : 0u);
                    }
                }
                commit_one(s_full + 8 * slot);
                if ((MT == 1 || slot == 1) && j + 2 < ntile) commit_one(k_free + 8 * s);   // (nobody waits for the last ones)
            };
            if (steps > 0) scores(0);
#pragma unroll 1
            for (int step = 0; step < steps && ok; ++step) {
                if (step + 1 < steps) {
                    if (step >= 1) ok = bar_wait<false>(o_full + 8 * ((step + 1) & 1), ((step - 1) >> 1) & 1, ab);   // the other slot's weights have been read
                    if (ok) scores(step + 1);
                    if (!ok) break;
                }
                const int j = step / MT, s = j & 1, slot = step & 1, m = MT == 2 ? slot : 0;
                ok = bar_wait<false>(v_full + 8 * s, (j >> 1) & 1, ab) && bar_wait<false>(p_ready + 8 * slot, (step >> 1) & 1, ab);
                if (!ok) break;
                fence_after();
                const uint64_t vb = desc_mn128(kv + s * stage + kbytes, 3 * PLANE);
                const uint32_t d = tm + O0 + m * VM, pa = tm + slot * SLOT_COLS;
#pragma unroll
                for (int pr = 0; pr < 6; ++pr) {
                    constexpr int PX[6] = {0, 2, 1, 0, 1, 0}, PY[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
                    for (int kk = 0; kk < KT / 16; ++kk)
                        mma_ts(d, pa + 48 * (kk >> 1) + 16 * PX[pr] + 8 * (kk & 1), vb + (uint64_t)((PY[pr] * PLANE + kk * 2048) / 16), ido, (pr | kk) != 0 ? 1u : 0u);
                }
                commit_one(o_full + 8 * slot);
                if ((MT == 1 || slot == 1) && j + 2 < ntile) commit_one(v_free + 8 * s);
            }
            if (!ok) {   // what was issued reads shared memory and TMEM: wait for it (bounded) before the CTA goes
                commit_one(B0 + 112);
                const unsigned long long t0_ = now_ns();
                while (!bar_try<false>(B0 + 112, 0) && now_ns() - t0_ < WAIT_NS) {}
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

template <int MT, int VM, int DK, bool CAP>
cudaError_t run_cap(const AttnArgs& a, const b200seq_step& st, dim3 grid, cudaStream_t cs) {
    const int KB = (a.D + 63) / 64, VB = (a.V + 63) / 64;
    int smem = 2 * (KB + VB) * 3 * PLANE + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;   // one CTA per SM: it takes all of TMEM
    static int ready[16] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 16 || ready[dev] < smem) {
        e = cudaFuncSetAttribute(attn_tc_kernel<MT, VM, DK, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev < 16) ready[dev] = smem;
    }
    launch_chained(attn_tc_kernel<MT, VM, DK, CAP>, grid, (4 * MT + 12) * 32, smem, cs, a, st);
    return cudaGetLastError();
}

template <int MT, int VM, int DK>
cudaError_t run(const AttnArgs& a, const b200seq_step& st, dim3 grid, cudaStream_t cs) {
    return a.softcap > 0.f ? run_cap<MT, VM, 0, true>(a, st, grid, cs) : run_cap<MT, VM, DK, false>(a, st, grid, cs);
}

}  // namespace

// Which of the two kernels is the faster one for a step, from its row tiles and the keys a token may see.  Here a CTA has an SM to itself: about 15 us
// (33 with heads above 64) of set-up, load and store, whatever the rows it has, a little less where one wave is all, and 2.2 (3.3) us a key tile.  The f32 tiles (seq_attn.cu) are half or a
// quarter of the rows, two or three to an SM: a wave of them takes about 33 (37) us, 22 (29) where each has an SM, and 18 (21) us more for every
// further key tile of its share.  Merging key splits: 3 and 10 us.  Measured, us, f32 tiles / this kernel, 32 query heads of 8 key heads of 64 (of 128):
//   65 sequences of one token, 10 earlier ones   57 /  66 ( 73 / 130)      128 of them    110 / 164 (153 / 282)      40 of two tokens  34 /  42 ( 56 /  89)
//   65 of one token, 200 earlier ones           162 /  90 (263 / 177)      17, 1000       151 /  42 (256 /  97)      64, 2000         902 / 287 (1526 / 648)
//   one sequence, 100 tokens                     21 /  16 ( 29 /  29)      600 tokens     168 /  29 (227 /  62)      4 of 300, 100    182 /  44 (281 / 109)
bool tc_is_faster(const AttnArgs& f32, int64_t units, int64_t splits, int64_t f32_units, int key_tiles, int sms) {
    const bool big = f32.D > 64 || f32.V > 64;
    const auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
    const int64_t waves = up(units * splits, sms);
    const double set_up = waves == 1 ? (big ? 30.0 : 12.5) : (big ? 33.0 : 15.0);
    const double tc = (double)waves * (set_up + (big ? 3.3 : 2.2) * (double)up(key_tiles, splits)) + (splits > 1 ? 3.0 : 0.0);
    const int64_t blocks = f32_units * f32.nsplit, share = up(key_tiles, f32.nsplit), fit = (big ? 2 : 3) * (int64_t)sms;
    const double wave = (blocks <= sms ? (big ? 29.0 : 22.0) : (big ? 37.0 : 33.0)) + (big ? 21.0 : 18.0) * (double)(share - 1);
    return tc < (double)up(blocks, fit) * wave + (f32.nsplit > 1 ? 10.0 : 0.0);
}

// Steps of more than 16 tokens with whole 16-byte rows and head sizes up to 128 in steps of 16.  What stays on the f32 tiles of seq_attn.cu:
// steps of fewer tokens, keys that come in two parts or from gathered rows, odd head sizes, unaligned rows, up to 64 tokens that see no more than 128
// keys (whole call, 32 heads of 128, f32 tiles against this kernel: 48 tokens 41 / 45 us, 64 tokens 39 / 58) -- and what tc_is_faster leaves there.
bool launch_attn_tc(AttnArgs& a, const b200seq_step& st, int max_keys, size_t part_floats, cudaStream_t cs, int& rc) {
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const int R = a.H / a.G;
    if (st.T <= 16 || st.B < 1 || (st.T <= 64 && max_keys <= 128) || a.D % 16 || a.V % 16 || a.D > 128 || a.V > 128 || a.ctx_rows || a.krot || a.kd != a.D || ((a.ld | a.kld | a.vld | a.q_col) & 3) || !al(a.qkvg) ||
        !al(a.kpool) || !al(a.vpool) || (a.pool > 0 && (!al(a.kpp) || !al(a.vpp))) || !al(a.out))
        return false;
    const int sms = tcpair::pair_sms();
    if (sms < 1) return false;
    const int64_t rows = (int64_t)st.T * a.H;
    // two row tiles per CTA where the heads are small enough and there are rows for it
    const int mt = a.D <= 64 && a.V <= 64 && rows >= 256ll * sms ? 2 : 1;
    const int RQ = 128 * mt;
    const int Rb = R < RQ ? R : RQ, HB = (R + Rb - 1) / Rb, QT = RQ / Rb;
    const int tiles = (st.T + QT - 1) / QT + st.B - (st.B == 1);   // upper bound of the step's query tiles (exact for one entry)
    // (Counted over full tiles, 32 sequences of one token were one tile a key head instead of 32, and their keys were dealt to 16 CTAs each: 17 sequences
    // behind 1000 tokens 66 us, now 42; 64 behind 2000 579, now 287.)
    const int each = (st.T + st.B - 1) / st.B;
    auto units = [&](int qt, int hb) { return (int64_t)st.B * ((each + qt - 1) / qt) * a.G * hb; };   // row tiles, were all entries equally long: each has its own
    const int64_t real = units(QT, HB);
    int64_t ns = 1;
    if (2 * real <= sms) {   // too few tiles: deal the key tiles to several CTAs, at least four each
        ns = sms / real;
        const int64_t most = (max_keys / KT) / 4, fits = a.part ? (int64_t)(part_floats / ((size_t)st.T * a.H * (a.V + 2))) : 0;
        ns = ns < most ? ns : most;
        ns = ns < fits ? ns : fits;
        ns = ns > 32 ? 32 : (ns < 1 ? 1 : ns);
    }
    if (!tc_is_faster(a, real, ns, units(a.QT, a.HB), (max_keys + KT - 1) / KT, sms)) return false;
    a.Rb = Rb, a.HB = HB, a.QT = QT, a.nsplit = (int)ns;
    const dim3 grid((unsigned)(a.G * a.HB * tiles), 1, (unsigned)ns);   // (head blocks fastest; the second dimension would end at 65 535 tiles)
    cudaError_t e;
    if (mt == 2) e = a.D == 64 ? run<2, 64, 4>(a, st, grid, cs) : run<2, 64, 0>(a, st, grid, cs);
    else if (a.V <= 64) e = a.D == 64 ? run<1, 64, 4>(a, st, grid, cs) : run<1, 64, 0>(a, st, grid, cs);
    else e = a.D == 128 ? run<1, 128, 8>(a, st, grid, cs) : run<1, 128, 0>(a, st, grid, cs);
    if (e != cudaSuccess) {
        rc = cuda_status(e, "attn tc");
        return true;
    }
    count_launch();
    rc = 0;
    return true;
}

}  // namespace b200seq
