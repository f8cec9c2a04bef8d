// Prompts over paged keys and values in bf16 on tcgen05: scores and sums of values in tensor memory.
//
// A CTA owns 128 (token, head) rows of one key head and walks over their keys 64 at a time. Per 64 keys: 4 · dim / 64 products of 128 × 64 make the scores, two threads per
// row cap, mask and weigh them, 4 products of 128 × vdim add the weights' share of the values; the scores of the next 64 keys are made under the weights of these. Keys and
// values come by TMA, a page's rows are the rows of a tensor map; two of either are on their way.
//
// What bounds it is the chain of a step, about 1.3 µs in a CTA alone on its SM (256 dimensions: shared memory), of which the products are 0.7, and the sums' way through registers
// in steps that bring a new maximum; a short prompt's longest tiles are as long as the launch. The `mma.sync` kernel, which remains for small pages and short sequences (kv_prefill_fits), has four warps per
// SM at this size. µs, with it → here: 4096 tokens, 4 heads of 256 over one key head, capped 258 → 125; 1999 tokens, the same 133 → 69; 2048 tokens, 16 heads of 128 over 4,
// 130 → 60, the softmax's sums alone 92 → 41; keys that are the values, 32 heads of 128 over 16, four portions of 2048 tokens 2830 → 1083. Errors against 64-bit results are the same to
// four digits (scores of either spread, capped or not; 700 and 1999 tokens).
#include "paged_kv.cuh"

namespace oxk {

namespace {

constexpr int kRows = 128, kKeys = 64, kSoft = 256, kThreads = kSoft + 64;  // warps 0-7 softmax, 8 copies, 9 issues products
constexpr int kHalf = kKeys / 2;                                            // keys of a row per thread
constexpr unsigned kPanelQ = kRows * 128, kPanelKv = kKeys * 128;  // bytes: rows × 64 dimensions

struct PreP {
    alignas(64) unsigned char maps[2][128];  // keys, values: [rows of the pool, dim | vdim]
    KvP kv;
    int kp, vp;  // panels of 64 dimensions
};

// Rows of weights in tensor memory (two per column) × values, of which 64 stand side by side for a key.
__device__ __forceinline__ void umma_weights(unsigned d, unsigned a, unsigned long long b, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
        : "memory");
}
// Shared-memory matrix descriptor, 128-byte swizzle, 64 elements of the wide axis side by side: groups of eight keys 1 024 bytes apart, the next 64
// elements a panel further.
__device__ __forceinline__ unsigned long long umma_wide_desc(unsigned smem_byte_addr) {
    return (unsigned long long)((smem_byte_addr & 0x3FFFFu) >> 4) | ((unsigned long long)(kPanelKv >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tmem_ld32(unsigned (&v)[32], unsigned from) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
          "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
          "=r"(v[30]), "=r"(v[31])
        : "r"(from));
}
__device__ __forceinline__ void tmem_ld4(unsigned* v, unsigned from) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(from));
}
__device__ __forceinline__ void tmem_ld16(unsigned (&v)[16], unsigned from) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(from));
}
__device__ __forceinline__ void tmem_st16(unsigned to, const unsigned (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};\n" ::"r"(v[0]), "r"(v[1]), "r"(v[2]),
        "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(to)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// KEYS: keys are the values, scores have a factor per key and an addend by distance. LSE: no values; the softmax's sums are the result.
enum : int { FORM_PLAIN, FORM_CAPPED, FORM_KEYS };
template <int FORM, bool LSE> __global__ void __launch_bounds__(kThreads, 2) paged_kv_prefill_tc(const __grid_constant__ PreP pp) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const KvP& p = pp.kv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kp = pp.kp, vp = LSE ? 0 : pp.vp;
    constexpr bool KEYS = FORM == FORM_KEYS;
    constexpr int NS = KEYS ? 3 : 2;  // tiles on their way: keys that are values are kept until both products have read them
    const unsigned k_stage = kp * kPanelKv, v_stage = vp * kPanelKv;
    const unsigned sq0 = smem_u32(smem), sk = sq0 + kp * kPanelQ, sv = KEYS ? sk : sk + NS * k_stage, bars = sk + NS * k_stage + (KEYS ? 0 : NS * v_stage);
    // barriers: keys there, free (three each), values there, free, scores there, weights there, sums (two each)
    const unsigned k_full = bars, k_free = bars + 24, v_full = KEYS ? k_full : bars + 48, v_free = bars + 64, s_full = bars + 80, w_full = bars + 96, o_done = bars + 112;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + (bars + 128 - sq0));
    float* shared = reinterpret_cast<float*>(smem + (bars + 144 - sq0));  // [turn][half of the keys][row]: what the two threads of a row tell each other
    float *scale_s = shared + 4 * kRows, *bias_s = scale_s + NS * kKeys;  // KEYS: [tile][key], [head][distance]
    if (tid == 0) {
        for (int i = 0; i < 16; i++) mbar_init(bars + i * 8, i == 12 || i == 13 ? kSoft / 32 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_wait();
    const int rep = p.heads / p.kv_heads, tq = kRows / rep, g = blockIdx.y;
    int seq, first;
    // long rows first: the last tiles of a sequence see the most keys
    if (!locate_tile(p.seqs, p.n_seqs, (int)gridDim.x - 1 - (int)blockIdx.x, tq, &seq, &first)) return;
    const SeqRow sq = load_seq(p.seqs, seq);
    const int n_tok = min(tq, sq.len - first), pos0 = sq.past + first, last = pos0 + n_tok - 1;
    // Scores in two turns of 64 columns, weights in two of 32, sums. Up to 128 dimensions weights take their scores' place, so that two CTAs fit an SM.
    const bool apart = vp > 2;
    const unsigned cols = LSE ? 128 : apart ? 512 : 256;
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < kRows * kp * 8; i += kThreads) {
        const int r = i / (kp * 8), c = i % (kp * 8), tok = r / rep, h = g * rep + r % rep;
        const bool live = tok < n_tok && c * 8 < p.dim;
        const bf16* src = (const bf16*)p.q;
        cp_async16(sq0 + (c >> 3) * kPanelQ + r * 128 + (((c & 7) ^ (r & 7)) << 4), live ? src + ((long long)(sq.start + first + tok) * p.heads + h) * p.dim + c * 8 : src, live);
    }
    cp_async_commit();
    if constexpr (KEYS)
        if (p.bias)
            for (int i = tid; i < rep * p.nd; i += kThreads) bias_s[i] = p.bias[(long long)g * rep * p.nd + i] * kLog2e;
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads them
    before_sync();
    __syncthreads();
    after_sync();
    pdl_trigger();  // the tensor memory is taken: nothing that starts now can keep it from this CTA
    const unsigned tmem = *tmem_slot, t_weights = apart ? tmem + 128 : tmem, weights_turn = apart ? 32 : kKeys, t_sum = tmem + (apart ? 192 : 128);
    const int kt0 = first_key(p, pos0) / kKeys, n = last / kKeys + 1 - kt0;
    bool ok = true;
    // Waits until the products of tile i are in the sums. Tiles take turns at two barriers. Who has the scores of tile i knows the products of tile i - 2 and of all before it to be
    // done, so the barrier of tile i - 1 or i cannot be a round behind. (With one barrier for all tiles, parity alone takes the end of tile i - 2 for that of tile i while
    // tile i - 1 is open.)
    auto added = [&](int i) { return mbar_wait(o_done + (i & 1) * 8, (unsigned)(i >> 1) & 1); };

    if (warp == 8) {
        RingAt at;
        for (int i = 0; i < n && ok; i++) {
            const int j0 = (kt0 + i) * kKeys;
            const long long pg = page_of(p, seq, j0);
            const int row = (int)key_row(p, pg, g, j0);
            if (i >= NS && !mbar_wait(k_free + at.s * 8, at.parity ^ 1)) ok = false;
            if (elect_one() && ok) {
                mbar_expect_tx(k_full + at.s * 8, k_stage + (KEYS ? kKeys * 4 : 0));
                if constexpr (KEYS)  // a page's factors follow one another
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(scale_s + at.s * kKeys)),
                                 "l"(p.kscale + (pg << p.shift) + (j0 & ((1 << p.shift) - 1))), "r"(kKeys * 4), "r"(k_full + at.s * 8)
                                 : "memory");
                for (int c = 0; c < kp; c++) tma_load_2d(sk + at.s * k_stage + c * kPanelKv, pp.maps[0], c * 64, row, k_full + at.s * 8);
            }
            __syncwarp();
            if constexpr (!LSE && !KEYS) {
                if (i >= NS && ok && !mbar_wait(v_free + at.s * 8, at.parity ^ 1)) ok = false;
                if (elect_one() && ok) {
                    mbar_expect_tx(v_full + at.s * 8, v_stage);
                    for (int c = 0; c < vp; c++) tma_load_2d(sv + at.s * v_stage + c * kPanelKv, pp.maps[1], c * 64, row, v_full + at.s * 8);
                }
                __syncwarp();
            }
            ok = __all_sync(0xffffffffu, ok);
            at.next(NS);
        }
    } else if (warp == 9) {
        const unsigned base = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);  // bf16 × bf16 → f32, M 128
        const unsigned by_keys = base | ((kKeys >> 3) << 17), by_values = base | (1u << 16) | ((unsigned)(vp * 8) << 17);  // the values' wide axis is the result's
        const unsigned long long dq = umma_kmajor_desc(sq0), dk = umma_kmajor_desc(sk), dv = umma_wide_desc(sv);
        RingAt tile_ahead, ahead, tile, at;  // tiles, and turns of scores and weights
        auto scores = [&] {
            if (ok && !mbar_wait(k_full + tile_ahead.s * 8, tile_ahead.parity)) ok = false;
            after_sync();
            if (elect_one() && ok) {
                const unsigned long long k = dk + tile_ahead.s * (k_stage >> 4);
                for (int c = 0; c < kp; c++)
#pragma unroll
                    for (int e = 0; e < 4; e++) umma_bf16(tmem + ahead.s * kKeys, dq + c * (kPanelQ >> 4) + e * 2, k + c * (kPanelKv >> 4) + e * 2, by_keys, c > 0 || e > 0);
                if (!KEYS) umma_commit(k_free + tile_ahead.s * 8);
                umma_commit(s_full + ahead.s * 8);
            }
            __syncwarp();
            tile_ahead.next(NS);
            ahead.next(2);
        };
        scores();
        for (int i = 0; i < n; i++) {
            if (i + 1 < n) {
                // the other turn's scores were read by the threads that wrote its weights; where these have their place, products have to be done with them
                if (!LSE && !apart && i > 0 && ok && !added(i - 1)) ok = false;
                scores();
            }
            if (ok && !mbar_wait(w_full + at.s * 8, at.parity)) ok = false;
            if constexpr (!LSE) {
                if (ok && !mbar_wait(v_full + tile.s * 8, tile.parity)) ok = false;
                after_sync();
                if (elect_one() && ok) {
                    const unsigned long long v = dv + tile.s * (v_stage >> 4);
#pragma unroll
                    for (int e = 0; e < kKeys / 16; e++) umma_weights(t_sum, t_weights + at.s * weights_turn + e * 8, v + e * 128, by_values, i > 0 || e > 0);
                    umma_commit((KEYS ? k_free : v_free) + tile.s * 8);
                    umma_commit(o_done + at.s * 8);
                }
                __syncwarp();
            }
            tile.next(NS);
            at.next(2);
        }
    } else {
        // two threads per row, each with half of the keys
        const int r = tid & (kRows - 1), part = tid / kRows, tok = r / rep, head = g * rep + r % rep;
        const bool live = tok < n_tok;
        const int pos = live ? pos0 + tok : last, low = first_key(p, pos), last_low = first_key(p, last);  // rows without a token compute something harmless
        const float mul2 = p.mul2 * temp_of(p, head), cap2 = p.cap2;
        const unsigned lanes = (unsigned)((warp & 3) * 32) << 16;
        // what both threads of a row know: by the two warps that share its rows
        auto both = [&](int turn, float mine) {
            float* at = shared + turn * 2 * kRows + r;
            at[part * kRows] = mine;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
            return at[(part ^ 1) * kRows];
        };
        const float* bias = bias_s + r % rep * p.nd;
        float m = KEYS ? -INFINITY : kNoScore, l = 0.f, l2 = 0.f;  // KEYS: key 0 is there for every row
        RingAt at, tile;
        for (int i = 0; i < n; i++) {
            const int j0 = (kt0 + i) * kKeys, mine0 = j0 + part * kHalf;
            // Key e of this thread's half. LSE: four of every eight, so that the sums have the order of paged_kv_prefill's: of each two neighbouring keys of eight one after the other, the four sums in the end.
            auto key = [&](int e) { return LSE ? j0 + e / 4 * 8 + part * 4 + e % 4 : mine0 + e; };
            if (ok && !mbar_wait(s_full + at.s * 8, at.parity)) ok = false;
            if constexpr (KEYS)  // the factors
                if (ok && !mbar_wait(k_full + tile.s * 8, tile.parity)) ok = false;
            after_sync();
            float s[kHalf];
            {
                unsigned v[32];
                if constexpr (LSE) {
#pragma unroll
                    for (int n = 0; n < kHalf; n += 4) tmem_ld4(v + n, tmem + lanes + at.s * kKeys + n * 2 + part * 4);
                } else {
                    tmem_ld32(v, tmem + lanes + at.s * kKeys + part * kHalf);
                }
                tmem_ld_wait();
                if constexpr (KEYS) {
                    const float* f = scale_s + tile.s * kKeys + part * kHalf;
#pragma unroll
                    for (int e = 0; e < kHalf; e++) s[e] = __uint_as_float(v[e]) * f[e];
                    if (p.bias && pos0 - (j0 + kKeys - 1) >= p.nd - 1) {  // one addend per head for the whole tile
                        const float far = bias[p.nd - 1];
#pragma unroll
                        for (int e = 0; e < kHalf; e++) s[e] += far;
                    } else if (p.bias) {
#pragma unroll
                        for (int e = 0; e < kHalf; e++) s[e] += bias[min(max(pos - (mine0 + e), 0), p.nd - 1)];
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < kHalf; e++) {
                        const float x = __uint_as_float(v[e]) * mul2;
                        s[e] = FORM == FORM_CAPPED ? cap2 - __fdividef(2.f * cap2, 1.f + exp2f(x)) : x;
                    }
                }
            }
            if (j0 + kKeys - 1 > pos0 || j0 < last_low) {
#pragma unroll
                for (int e = 0; e < kHalf; e++)
                    if (key(e) > pos || key(e) < low) s[e] = -INFINITY;
            }
            float top = m;
#pragma unroll
            for (int e = 0; e < kHalf; e++) top = fmaxf(top, s[e]);
            top = fmaxf(top, both(i & 1, top));
            // Weights are taken against the maximum itself: the key that stands out weighs 1, which bf16 holds. (Against a maximum up to 2^8 behind it is rounded, though sums are
            // rarely taken anew then: 2048 tokens, 16 heads of 128 over 4, 51 µs against 60, but 1.85e-3 from 64-bit results against 1.65e-3 where single keys stand out, 2.08e-3
            // against 2.02e-3 where none do.) Both warps of a row see the same tops.
            if (__any_sync(0xffffffffu, top > m)) {
                const float keep = exp2f(m - top);
                m = top;
                l *= keep;
                l2 *= keep;
                if (!LSE && i > 0) {
                    if (ok && !added(i - 1)) ok = false;
                    after_sync();
#pragma unroll 1
                    for (int c = part * 16; c < vp * 64; c += 32) {
                        unsigned v[16];
                        tmem_ld16(v, t_sum + lanes + c);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; e++) v[e] = __float_as_uint(__uint_as_float(v[e]) * keep);
                        tmem_st16(t_sum + lanes + c, v);
                    }
                }
            }
            unsigned w[kHalf / 2];
#pragma unroll
            for (int e = 0; e < kHalf / 2; e++) {
                const float a = exp2f(s[2 * e] - m), b = exp2f(s[2 * e + 1] - m);
                if constexpr (LSE) (e & 1 ? l2 : l) = (e & 1 ? l2 : l) + a + b;
                else l += a + b;
                w[e] = pack_bf16(a, b);
            }
            if constexpr (!LSE) {
                // Where weights take their scores' place: both threads of the row have read these. Elsewhere: the products that read this turn's last weights were issued
                // before these scores.
                tmem_st16(t_weights + lanes + at.s * weights_turn + part * (kHalf / 2), w);
                if (j0 + kKeys - 1 > last) {  // what lies behind the last key may be no number, which a weight of 0 would not cancel
                    if (ok && !mbar_wait(v_full + tile.s * 8, tile.parity)) ok = false;
                    const int dead = j0 + kKeys - 1 - last;
                    for (int u = tid; u < dead * vp * 8; u += kSoft) {
                        const unsigned to = sv + tile.s * v_stage + (u >> 3) / dead * kPanelKv + (kKeys - dead + (u >> 3) % dead) * 128 + (u & 7) * 16;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(to), "r"(0) : "memory");
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                tmem_st_wait();
            }
            before_sync();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(w_full + at.s * 8) : "memory");
            tile.next(NS);
            at.next(2);
        }
        if (LSE) l += l2;
        l += both(n & 1, l);
        const long long token = sq.start + first + tok;
        if constexpr (LSE) {
            if (live && ok && part == 0) p.lse[token * p.heads + head] = m + log2f(l);
        } else {
            if (ok && !added(n - 1)) ok = false;
            after_sync();
            float f = 1.f / l;
            if (!KEYS && p.sink && live) {
                const float s = sink_of(p, head) * kLog2e, top = fmaxf(m, s), keep = exp2f(m - top);
                f = keep / (l * keep + exp2f(s - top));
            }
            if (KEYS) f *= p.out_scale;
            else if (live) f *= gate_of<bf16>(p, token, head);
            bf16* out = (bf16*)p.out + (token * p.heads + head) * p.vdim;
#pragma unroll 1
            for (int c = part * 32; c < vp * 64; c += 64) {
                unsigned v[32];
                tmem_ld32(v, t_sum + lanes + c);
                tmem_ld_wait();
                if (live && ok) {
#pragma unroll
                    for (int e = 0; e < 32; e += 8)
                        if (c + e < p.vdim) {
                            uint4 q;
                            q.x = pack_bf16(__uint_as_float(v[e]) * f, __uint_as_float(v[e + 1]) * f);
                            q.y = pack_bf16(__uint_as_float(v[e + 2]) * f, __uint_as_float(v[e + 3]) * f);
                            q.z = pack_bf16(__uint_as_float(v[e + 4]) * f, __uint_as_float(v[e + 5]) * f);
                            q.w = pack_bf16(__uint_as_float(v[e + 6]) * f, __uint_as_float(v[e + 7]) * f);
                            *reinterpret_cast<uint4*>(out + c + e) = q;
                        }
                }
                __syncwarp();
            }
        }
    }
    if (!ok && lane == 0) report(p.err, ERR_WAIT_TIMEOUT, p.node, (long long)blockIdx.x, (long long)warp);
    before_sync();
    __syncthreads();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

}  // namespace

static int prefill_smem(const KvP& kv, bool keys, bool lse) {
    const int kp = (kv.dim + 63) / 64, vp = (kv.vdim + 63) / 64, tiles = keys ? 3 : 2;
    return 1024 + kp * (int)(kPanelQ + tiles * kPanelKv) + (keys || lse ? 0 : vp * tiles * (int)kPanelKv) + 144 + 4 * kRows * 4 +
           (keys ? tiles * kKeys * 4 + kv.heads / kv.kv_heads * kv.nd * 4 : 0);
}

// Where no sequence has more keys than a tile there is nothing to overlap, and a tile of 128 rows is the emptier: the `mma.sync` kernel stays. µs of a step with it → here, keys and values:
// one prompt of 33 tokens, 16 heads of 128 over 4, 19.7 → 22.6; 64 prompts of 32, 8 heads of 64 over 8, 32.8 → 38.4; 64 sequences of 60 with two tokens more, 32 heads of 128 over 16,
// 40.7 → 49.6; keys that are the values, the same 52.0 → 64.8, prompts of 8, 8 heads of 64 over 8, 19.8 → 23.5. Up to twice a tile: 16 prompts of 128, 16 heads over 4, 49 → 38; one of 100, 4 heads of
// 256, 26.2 → 25.2; keys that are the values, where heads share none, 16 prompts of 128, 8 heads of 64, 31.2 → 36.4, so there twice a tile is the line. Of 160 tokens and more every
// form is faster here (16 heads of 128 over 4, 25.8 → 23.9; 260: 31.0 → 25.0).
bool kv_prefill_fits(const KvP& kv, const TRef& keys, const TRef* values, int64_t out_off) {
    const int64_t rows = (int64_t)kv.n_pages * kv.kv_heads << kv.shift, longest = (int64_t)kv.width << kv.shift;
    return longest > (values == &keys && kv.heads == kv.kv_heads ? 2 * kKeys : kKeys) && 1 << kv.shift >= kKeys && kv.dim % 8 == 0 && kv.dim <= 256 && kv.heads / kv.kv_heads <= kRows && rows < INT32_MAX && keys.buf.off % 16 == 0 &&
           (!values || (kv.vdim % 8 == 0 && kv.vdim <= 256 && values->buf.off % 16 == 0 && out_off % 16 == 0)) &&
           prefill_smem(kv, values == &keys, !values) <= 200 * 1024;
}

// `values` = &keys: the form whose keys are the values.
void emit_kv_prefill(Emitter& em, const KvP& kv, const TRef& keys, const TRef* values, std::initializer_list<std::pair<size_t, Buf>> ptrs, const char* label) {
    PreP p{};
    p.kv = kv;
    p.kp = (kv.dim + 63) / 64;
    p.vp = (kv.vdim + 63) / 64;
    const int64_t tq = kRows / (kv.heads / kv.kv_heads), rows = (int64_t)kv.n_pages * kv.kv_heads << kv.shift;
    void (*const k)(const PreP) = values == &keys   ? paged_kv_prefill_tc<FORM_KEYS, false>
                                  : kv.cap2 > 0.f ? (values ? paged_kv_prefill_tc<FORM_CAPPED, false> : paged_kv_prefill_tc<FORM_CAPPED, true>)
                                                  : (values ? paged_kv_prefill_tc<FORM_PLAIN, false> : paged_kv_prefill_tc<FORM_PLAIN, true>);
    ensure_max_dynamic_smem((const void*)k, 200 * 1024);
    LaunchRec& rec = em.launch(k, dim3((unsigned)((kv.rows + tq - 1) / tq + kv.n_seqs), (unsigned)kv.kv_heads), dim3(kThreads),
                               (unsigned)prefill_smem(kv, values == &keys, !values), p, {}, label, /*pdl=*/true);
    for (auto& pr : ptrs) rec.relocs.push_back(Reloc{(uint32_t)(offsetof(PreP, kv) + pr.first), pr.second});
    rec.tmaps.push_back(TmapReloc{(uint32_t)offsetof(PreP, maps), keys.buf, (uint64_t)kv.dim, (uint64_t)rows, (uint64_t)kv.dim * 2, 64u, (uint32_t)kKeys});
    if (values && values != &keys)
        rec.tmaps.push_back(TmapReloc{(uint32_t)offsetof(PreP, maps) + 128, values->buf, (uint64_t)kv.vdim, (uint64_t)rows, (uint64_t)kv.ldv * 2, 64u, (uint32_t)kKeys});
}

}  // namespace oxk
