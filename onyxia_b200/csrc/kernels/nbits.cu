// com.microsoft.MatMulNBits: y[m, n] = Σ_k a[m, k] · w[n, k] with
// w[n, k] = (q[n, k] − zp[n, k/bs]) · scale[n, k/bs] for 4-bit weights packed
// 32 to a 16-byte block (decomposition: crates/onyxia-ir/src/decomp.rs:615-663;
// lowering and wire layout: crates/onyxia-lower/src/rules.rs:890-940).
//
// Rounding follows the decomposition: each dequantised weight is rounded to
// the scales' dtype (exact here, see below), then to the activations' dtype if
// that differs, and the f32 dot product is rounded once to the activations'
// dtype on store. The interpreter accumulates in f64; f32 accumulation differs
// from it only by rounding.
//
// Generic path (`nbits_gemv_simt`, any float dtype mix; the f16 decode path is nbits_mma.cu): a warp owns two or four weight rows and takes 256 k
// per step, a lane eight of them: one word of nibbles per weight row, the matching activations in registers for all of them. Up to eight warps
// share the same weight rows and take the steps in turn. Algorithmic bytes per weight: 0.5 (nibbles) + 2/32 or 4/32
// (scale) = 0.5625 / 0.625 B.
#include "common.cuh"
#include "kernels.hpp"

namespace oxk {

struct NBitsGemvP {
    const void* a;        // [M, K] activations
    const unsigned* w;    // [N, n_blocks] 16-byte blocks of 32 nibbles
    const void* scales;   // [N, n_blocks]
    const unsigned char* zp;  // [N, n_blocks] packed nibbles, or null
    void* y;              // [M, N]
    long long m_first;    // first activation row of this launch
    long long m_total;
    long long k, n, n_blocks;
    int share;            // warps of a CTA that work on the same weight rows
};

// (q − zp)·scale rounded to the scales' dtype, then widened to f32. For f16
// scales the product is formed by one f16 multiply (single rounding); for f32
// scales by one f32 multiply. Both equal the interpreter's f64 product rounded
// once, because an integer of ≤ 5 bits times one scale is exact in f64.
template <int SDT> struct ScaleOps;
template <> struct ScaleOps<DT_F16> {
    using S = __half;
    static __device__ __forceinline__ S load(const void* p, long long i) { return ((const __half*)p)[i]; }
    static __device__ __forceinline__ float deq(int qmz, S s) { return __half2float(__hmul(__int2half_rn(qmz), s)); }
};
template <> struct ScaleOps<DT_F32> {
    using S = float;
    static __device__ __forceinline__ S load(const void* p, long long i) { return ((const float*)p)[i]; }
    static __device__ __forceinline__ float deq(int qmz, S s) { return (float)qmz * s; }
};

// Eight consecutive activations from k0 on as f32; zero beyond K.
template <int ADT> __device__ __forceinline__ void load_acts(const void* a, long long at, long long left, bool wide, float (&v)[8]) {
    if (wide && left >= 8) {
        if constexpr (ADT == DT_F32) {
            const float4 lo = *reinterpret_cast<const float4*>((const float*)a + at), hi = *reinterpret_cast<const float4*>((const float*)a + at + 4);
            v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
            v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        } else {
            const uint4 q = *reinterpret_cast<const uint4*>((const __half*)a + at);
            const unsigned u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[e]));
                v[2 * e] = f.x;
                v[2 * e + 1] = f.y;
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = e < left ? ld<ADT>(a, at + e) : 0.f;
    }
}

// MT activation rows (of blockIdx.y) share every weight read. These matrices are small (a 2-layer decoder holds 14 MB: they stay in L2), so
// what counts is the length of the chain: the first step's weights are read ahead of the grid dependency, every lane's loads of a step are
// in flight together, and sums over lanes fold several values at once. One token of that decoder: 29 launches, 360 → 160 µs against one warp per
// weight row that read its activations one by one (512 to 2048 by 512 to 2048: 14 → 2.5 µs a launch).
constexpr int kNbWarps = 8;
constexpr int nb_rows(int mt) { return mt == 8 ? 2 : 4; }  // weight rows of a warp
template <int ADT, int SDT, int MT> __global__ void __launch_bounds__(kNbWarps * 32, 2) nbits_gemv_simt(const NBitsGemvP p) {
    constexpr int kNbRows = nb_rows(MT), N = MT * kNbRows;
    __shared__ float red[kNbWarps][32];
    using SO = ScaleOps<SDT>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slice = warp % p.share;
    const long long row0 = ((long long)blockIdx.x * (kNbWarps / p.share) + warp / p.share) * kNbRows, m0 = p.m_first + (long long)blockIdx.y * MT;
    const int steps = row0 < p.n ? (int)((p.n_blocks + 7) / 8) : 0;
    const bool wide = p.k % (ADT == DT_F32 ? 4 : 8) == 0 && (reinterpret_cast<uintptr_t>(p.a) & 15) == 0;
    unsigned w[kNbRows];
    typename SO::S sc[kNbRows];
    int z[kNbRows];
    auto fetch_words = [&](int step) {
        const long long blk = (long long)step * 8 + (lane >> 2);
#pragma unroll
        for (int r = 0; r < kNbRows; r++)
            w[r] = step < steps && blk < p.n_blocks && row0 + r < p.n ? __ldg(p.w + ((row0 + r) * p.n_blocks + blk) * 4 + (lane & 3)) : 0x88888888u;
    };
    auto fetch_scales = [&](int step) {
        const long long blk = (long long)step * 8 + (lane >> 2);
#pragma unroll
        for (int r = 0; r < kNbRows; r++) {
            const bool live = step < steps && blk < p.n_blocks && row0 + r < p.n;
            const long long i = live ? (row0 + r) * p.n_blocks + blk : 0;
            sc[r] = SO::load(p.scales, i);
            z[r] = p.zp && live ? (p.zp[i >> 1] >> ((i & 1) * 4)) & 0xF : 8;
        }
    };
    pdl_trigger();
    fetch_words(slice);  // constants; scales and zero points may be another launch's results
    pdl_wait();
    fetch_scales(slice);
    float acc[N];
#pragma unroll
    for (int i = 0; i < N; i++) acc[i] = 0.f;
    for (int step = slice; step < steps; step += p.share) {
        const long long k0 = (long long)step * 256 + lane * 8, left = p.k - k0;
        float a[MT][8];
#pragma unroll
        for (int m = 0; m < MT; m++) {
            if (m0 + m < p.m_total) {
                load_acts<ADT>(p.a, (m0 + m) * p.k + k0, left, wide, a[m]);
            } else {
#pragma unroll
                for (int e = 0; e < 8; e++) a[m][e] = 0.f;
            }
        }
        unsigned now[kNbRows];
        typename SO::S s[kNbRows];
        int zero[kNbRows];
#pragma unroll
        for (int r = 0; r < kNbRows; r++) {
            now[r] = w[r];
            s[r] = sc[r];
            zero[r] = z[r];
        }
        fetch_words(step + p.share);
        fetch_scales(step + p.share);
#pragma unroll
        for (int r = 0; r < kNbRows; r++) {
            const bool live = row0 + r < p.n;
#pragma unroll
            for (int e = 0; e < 8; e++) {
                float wv = SO::deq((int)((now[r] >> (4 * e)) & 0xF) - zero[r], s[r]);
                if constexpr (ADT == DT_F16 && SDT == DT_F32) wv = __half2float(__float2half_rn(wv));
                if (e >= left || !live) wv = 0.f;  // the last block may be padding beyond K
#pragma unroll
                for (int m = 0; m < MT; m++) acc[m * kNbRows + r] = fmaf(a[m][e], wv, acc[m * kNbRows + r]);
            }
        }
    }
    // every step sends half of the values to the lanes that keep them: value m · kNbRows + r ends up in that lane
#pragma unroll
    for (int half = N / 2; half >= 1; half /= 2)
#pragma unroll
        for (int i = 0; i < half; i++) {
            const bool up = lane & half;
            const float give = up ? acc[i] : acc[i + half], keep = up ? acc[i + half] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    float sum = acc[0];
#pragma unroll
    for (int o = 16; o >= N; o /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (p.share > 1) {
        red[warp][lane] = sum;
        __syncthreads();
        if (slice) return;
        sum = 0.f;
        for (int i = 0; i < p.share; i++) sum += red[warp + i][lane];
    }
    const long long m = m0 + lane / kNbRows, row = row0 + lane % kNbRows;
    if (lane < N && m < p.m_total && row < p.n) st<ADT>(p.y, m * p.n + row, sum);
}

template <int ADT, int SDT> static void launch_gemv(Emitter& em, NBitsGemvP p, const TRef& a, const TRef& w,
                                                    const TRef& scales, const TRef* zp, const TRef& y) {
    const Buf zb = zp ? zp->buf : Buf{kSlotNull, 0};
    const int mt = p.m_total >= 5 ? 8 : p.m_total >= 3 ? 4 : (int)p.m_total;
    const long long units = (p.n + nb_rows(mt) - 1) / nb_rows(mt), steps = (p.n_blocks + 7) / 8;
    // warps per unit of weight rows: until there are 16 per SM, a step each at least
    p.share = 1;
    while (p.share < kNbWarps && units * p.share < 16LL * sm_count() && steps >= 2 * p.share) p.share *= 2;
    const int per_cta = kNbWarps / p.share;
    const auto k = mt == 1 ? nbits_gemv_simt<ADT, SDT, 1> : mt == 2 ? nbits_gemv_simt<ADT, SDT, 2> : mt == 4 ? nbits_gemv_simt<ADT, SDT, 4>
                                                                                                    : nbits_gemv_simt<ADT, SDT, 8>;
    for (long long passes = (p.m_total + mt - 1) / mt; passes > 0; passes -= 65535, p.m_first += 65535LL * mt)
        em.launch(k, dim3((unsigned)((units + per_cta - 1) / per_cta), (unsigned)std::min<long long>(passes, 65535)), dim3(kNbWarps * 32), 0, p,
                  {{&p.a, a.buf}, {&p.w, w.buf}, {&p.scales, scales.buf}, {&p.zp, zb}, {&p.y, y.buf}}, "nbits_gemv_simt", /*pdl=*/true);
}

void emit_matmul_nbits(Emitter& em, const NBitsDesc& d, const TRef& a, const TRef& w, const TRef& scales,
                       const TRef* zp, const TRef& y) {
    if (d.block_size != 32) throw std::runtime_error("nbits kernels need block_size 32");
    if (d.m == 0 || d.n == 0) return;
    if (d.tiled) {
        emit_matmul_nbits_stream(em, d, a, w, y);
        return;
    }
    if (d.interleaved) {
        emit_matmul_nbits_mma(em, d, a, w, scales, zp, y);
        return;
    }
    NBitsGemvP p{};
    p.m_total = d.m;
    p.k = d.k;
    p.n = d.n;
    p.n_blocks = d.n_blocks;
    if (d.act_dtype == DT_F16 && d.scale_dtype == DT_F16) launch_gemv<DT_F16, DT_F16>(em, p, a, w, scales, zp, y);
    else if (d.act_dtype == DT_F32 && d.scale_dtype == DT_F32) launch_gemv<DT_F32, DT_F32>(em, p, a, w, scales, zp, y);
    else if (d.act_dtype == DT_F16 && d.scale_dtype == DT_F32) launch_gemv<DT_F16, DT_F32>(em, p, a, w, scales, zp, y);
    else launch_gemv<DT_F32, DT_F16>(em, p, a, w, scales, zp, y);
}

}  // namespace oxk
