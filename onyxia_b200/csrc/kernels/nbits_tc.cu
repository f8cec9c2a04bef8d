// MatMulNBits for more than 8 activation rows (prefill, batched decode): a
// tcgen05 GEMM with the accumulator in tensor memory.
//
//   Yᵀ[n, m] = Σ_k W[n, k] · X[m, k],   W = round_f16((q − zp)·s) from the tile records
//
// The weights are the MMA's A operand (128 rows of W per CTA = 8 row tiles), the
// activations its B operand (MB = 16 … 256 rows of X per pass), so the weight
// stream is read once per MB activation rows. Per step of 128 k:
//   * eight producer warps each widen one tile record (the streaming GEMV's
//     nibble arithmetic, exact (q − zp)·s rounding) into the A panel in shared
//     memory — K-major, 128-byte rows, 128-byte swizzle; one of their threads asks the
//     TMA unit for the matching activation columns (two tiled loads of 64 k × MB rows
//     through a tensor map with the same swizzle, zero-filled outside the matrix), which
//     land in the B panel and complete the stage's barrier by byte count;
//   * one thread of a ninth warp issues eight tcgen05.mma (M 128 × N MB × K 16,
//     f16 inputs, f32 accumulation in TMEM) and commits them to the mbarrier that
//     frees the stage.
// Stages form a ring (full / empty mbarriers). After the last step the first four
// warps read the accumulator with tcgen05.ld (a warp reads the 32 TMEM lanes of
// its quarter), round to f16 and store Y, consecutive threads on consecutive n.
//
// Every wait is bounded; on expiry the kernel records ERR_WAIT_TIMEOUT, lets the
// remaining phases run out and frees its tensor memory before it exits.
//
// Accuracy: the tensor core adds into its f32 accumulator without rounding to nearest, so a long chain of
// MMAs drifts. Consecutive steps therefore rotate over up to four accumulators side by side in tensor
// memory, which the epilogue adds: chains a quarter as long, at no cost in the main loop.
//
// Split K: a matrix with few row blocks (or a few more than a whole wave of CTAs) would leave SMs idle,
// so the k range of the row blocks beyond the last whole wave (all of them when there is less than one
// wave) can be cut into `splits` pieces, each CTA writing its f32 partial
// accumulator to scratch; a second kernel adds the pieces in fixed order and rounds once.
//
// FLOPs 2·M·N·K; bytes as for the GEMV (0.5625 per weight) once per MB rows.
#include <cstdio>
#include <cstdlib>

#include "kernels.hpp"
#include "tc_util.cuh"

namespace oxk {

namespace {

constexpr int kProducerWarps = 8;         // warps that widen the weights (A panels), one per row tile
constexpr int kMmaWarp = kProducerWarps;  // the warp that issues the MMAs
constexpr int kThreadsTc = (kMmaWarp + 1) * 32;
constexpr int kTileWt = 1024, kTileSt = 128, kTileZt = 64;
constexpr int kPanelA = 128 * 128;  // bytes: 128 rows × 64 k of f16

struct TcP {
    alignas(64) unsigned char xmap[128];  // tensor map over the activations [M, K] (box 64 k × mb rows), when use_tma
    const __half* x;             // activations [M, K]
    const unsigned char* tiles;  // tile records, row tile by row tile
    __half* y[3];                // outputs per segment [M, seg_n]
    ErrWord* err;
    long long m0, m_total, k;
    long long seg_n[3];
    int seg_rt0[4];
    int n_seg, interleave2;      // interleave2: row tiles alternate between segment 0 and 1
    int k_tiles, row_tiles, mb, stages, tile_bytes, has_zp, node;
    int use_tma;                 // 0: K is not a multiple of 8 (or x is not 16-byte aligned) — plain loads
    int n_acc;                   // accumulators in tensor memory that the steps rotate over (1, 2 or 4)
    int n_full;                  // row blocks (CTAs) that take all of K; the blocks after them are cut along k
    int splits;                  // pieces of the k range of those tail blocks; > 1: partial sums go to `partial`
    float* partial;              // [splits][mb][n_pad] f32, rows counted from the first tail block
    long long n_pad;             // weight rows of the tail blocks (128 per block)
};

__device__ __forceinline__ unsigned s_addr(const void* p) { return smem_u32(p); }
__device__ __forceinline__ void bar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ unsigned and_or_tc(unsigned a, unsigned b, unsigned c) {
    unsigned d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ unsigned h2u_tc(__half2 h) { return *reinterpret_cast<unsigned*>(&h); }
__device__ __forceinline__ __half2 u2h_tc(unsigned u) { return *reinterpret_cast<__half2*>(&u); }
// One 32-bit word (8 interleaved nibbles) → 8 consecutive k as four f16 pairs.
__device__ __forceinline__ uint4 widen_tc(unsigned w, __half2 sub_lo, __half2 add_hi, __half2 s2) {
    const __half2 sixteenth = __float2half2_rn(0.0625f);
    const unsigned magic = 0x64006400u, m_lo = 0x000F000Fu, m_hi = 0x00F000F0u;
    const unsigned lo = and_or_tc(w, m_lo, magic), hi = and_or_tc(w, m_hi, magic);
    const unsigned w8 = w >> 8;
    const unsigned lo2 = and_or_tc(w8, m_lo, magic), hi2 = and_or_tc(w8, m_hi, magic);
    uint4 o;
    o.x = h2u_tc(__hmul2(__hsub2(u2h_tc(lo), sub_lo), s2));
    o.y = h2u_tc(__hmul2(__hfma2(u2h_tc(hi), sixteenth, add_hi), s2));
    o.z = h2u_tc(__hmul2(__hsub2(u2h_tc(lo2), sub_lo), s2));
    o.w = h2u_tc(__hmul2(__hfma2(u2h_tc(hi2), sixteenth, add_hi), s2));
    return o;
}

// f16 × f16 → f32, one CTA.
__device__ __forceinline__ void umma_f16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool accumulate) { umma_bf16(d, a, b, idesc, accumulate); }

__global__ void __launch_bounds__(kThreadsTc, 2) nbits_gemm_tc(const __grid_constant__ TcP p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the swizzle pattern repeats every 1 024 bytes: panels start on that boundary
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int mb = p.mb, S = p.stages;
    const int panel_b = mb * 128;                       // bytes of one 64-k activation panel
    const int stage_bytes = 2 * kPanelA + 2 * panel_b;  // A panels, then B panels
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + (size_t)S * stage_bytes);  // full[S], empty[S], done
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * S + 1);

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            // a stage is full when every producer warp has arrived, and so has the thread that posted the
            // activation bytes, and those bytes have landed
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_addr(bars + s)), "r"(kProducerWarps + 1) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s_addr(bars + S + s)) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s_addr(bars + 2 * S)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    int tmem_cols = 32;
    while (tmem_cols < mb * p.n_acc) tmem_cols <<= 1;
    if (warp == kMmaWarp) {  // the MMA warp owns the tensor-memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;
    pdl_trigger();  // the tensor memory is taken: what starts now may wait for it, but does not keep it from this kernel

    // CTAs 0 … n_full − 1 own a whole row block; the ones after them share the tail blocks, `splits` CTAs each
    const int tail_j = (int)blockIdx.x - p.n_full;
    const int block = tail_j < 0 ? (int)blockIdx.x : p.n_full + tail_j / p.splits;
    const int splits = tail_j < 0 ? 1 : p.splits, split = tail_j < 0 ? 0 : tail_j % p.splits;
    const int rt0 = block * 8;  // first row tile of this CTA
    const int kt_lo = (int)((long long)p.k_tiles * split / splits);  // this CTA's piece of the k range, in 128-k steps
    const int steps = (int)((long long)p.k_tiles * (split + 1) / splits) - kt_lo;
    bool ok = true;

    if (warp < kProducerWarps) {
        // ── producers: warp w widens row tile rt0 + w ──
        const int g = lane >> 2, t = lane & 3;
        const int rt = rt0 + warp;
        const bool rt_live = rt < p.row_tiles;
        const unsigned char* rec = p.tiles + (size_t)(rt_live ? rt : 0) * p.k_tiles * p.tile_bytes;
        // this warp's record of a step: two 16-byte words of nibbles per lane, the two rows' scales (and zero points)
        struct Rec {
            uint4 wl, wh;
            __half2 s2;
            uchar2 z;
        };
        auto fetch = [&](int i) {
            Rec r;
            r.wl = make_uint4(0, 0, 0, 0);
            r.wh = r.wl;
            r.s2 = __float2half2_rn(0.f);
            r.z = make_uchar2(8, 8);
            if (rt_live && i < steps) {
                const unsigned char* q = rec + (size_t)(kt_lo + i) * p.tile_bytes;
                r.wl = __ldg(reinterpret_cast<const uint4*>(q) + lane);
                r.wh = __ldg(reinterpret_cast<const uint4*>(q) + 32 + lane);
                r.s2 = *reinterpret_cast<const __half2*>(q + kTileWt + lane * 4);
                if (p.has_zp) r.z = *reinterpret_cast<const uchar2*>(q + kTileWt + kTileSt + lane * 2);
            }
            return r;
        };
        Rec next = fetch(0);  // weights are constants: may overlap the launches before this one
        pdl_wait();
        RingAt at;  // carried along: a division by the number of stages is a long chain
        for (int i = 0; i < steps; i++) {
            const unsigned s = at.s;
            if (i >= S && ok && !mbar_wait(s_addr(bars + S + s), at.parity ^ 1)) ok = false;
            at.next(S);
            unsigned char* stage = smem + (size_t)s * stage_bytes;
            ox_trace(p.err, 41);
            if (p.use_tma) {
                // B: activation rows m0 … m0 + mb, columns 128·i … + 128, as two 64-k panels
                if (tid == 0) {
                    const unsigned bar = s_addr(bars + s), dst = s_addr(stage + 2 * kPanelA);
                    const unsigned long long map = reinterpret_cast<unsigned long long>(&p.xmap);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(2u * (unsigned)panel_b) : "memory");
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                        "l"(map), "r"((kt_lo + i) * 128), "r"((int)p.m0), "r"(bar)
                        : "memory");
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                            dst + (unsigned)panel_b),
                        "l"(map), "r"((kt_lo + i) * 128 + 64), "r"((int)p.m0), "r"(bar)
                        : "memory");
                }
            } else {
                // plain loads, element by element: thread c fills chunk `c & 15` of rows (c >> 4) + 16·j
                const int ch = tid & 15, r0 = tid >> 4;
                unsigned char* bpan = stage + 2 * kPanelA;
                const long long k0 = (long long)(kt_lo + i) * 128 + ch * 8;
                const unsigned dst0 = s_addr(bpan + (ch >> 3) * panel_b + r0 * 128 + (((ch & 7) ^ (r0 & 7)) << 4));
                for (int j = 0; j * 16 < mb; j++) {
                    const long long row = p.m0 + r0 + 16 * j;
                    __half tmp[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) tmp[e] = (row < p.m_total && k0 + e < p.k) ? p.x[row * p.k + k0 + e] : __float2half(0.f);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst0 + j * 2048), "r"(reinterpret_cast<unsigned*>(tmp)[0]),
                                 "r"(reinterpret_cast<unsigned*>(tmp)[1]), "r"(reinterpret_cast<unsigned*>(tmp)[2]),
                                 "r"(reinterpret_cast<unsigned*>(tmp)[3])
                                 : "memory");
                }
                if (tid == 0) bar_arrive(s_addr(bars + s));  // stands for the byte-count arrival; the warp's own arrival below orders the stores
            }
            // A: rows 16·warp + g and + 8, k = 32·t + 8·m … + 8 of this 128-k step; the next record is already on its way
            const Rec cur = next;
            next = fetch(i + 1);
            const __half2 s2l = __low2half2(cur.s2), s2h = __high2half2(cur.s2);
            const float zl = (float)cur.z.x, zh = (float)cur.z.y;
            const __half2 subl = __float2half2_rn(1024.f + zl), subh = __float2half2_rn(1024.f + zh);
            const __half2 addl = __float2half2_rn(-64.f - zl), addh = __float2half2_rn(-64.f - zh);
            const unsigned wls[4] = {cur.wl.x, cur.wl.y, cur.wl.z, cur.wl.w}, whs[4] = {cur.wh.x, cur.wh.y, cur.wh.z, cur.wh.w};
            const int row_l = warp * 16 + g, row_h = row_l + 8;
            unsigned char* panel = stage + (t >> 1) * kPanelA;  // blocks 0,1 → first 64 k; 2,3 → second
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int chunk = (t & 1) * 4 + m;  // 16-byte chunk of the 128-byte row
                *reinterpret_cast<uint4*>(panel + row_l * 128 + ((chunk ^ (row_l & 7)) << 4)) = widen_tc(wls[m], subl, addl, s2l);
                *reinterpret_cast<uint4*>(panel + row_h * 128 + ((chunk ^ (row_h & 7)) << 4)) = widen_tc(whs[m], subh, addh, s2h);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // make the stores visible to the tensor core
            __syncwarp();
            if (lane == 0) bar_arrive(s_addr(bars + s));
            ox_trace(p.err, 43);
        }
    } else {
        // ── MMA issuer ──
        const unsigned idesc = (1u << 4) | ((unsigned)(mb >> 3) << 17) | (8u << 24);  // f16 × f16 → f32, K-major, N = mb, M = 128
        pdl_wait();
        RingAt at, acc;  // acc: the accumulator of a step
        const unsigned full = s_addr(bars), empty = full + S * 8, step16 = (unsigned)stage_bytes >> 4;
        const unsigned long long a0 = umma_kmajor_desc(s_addr(smem)), b0 = umma_kmajor_desc(s_addr(smem) + 2 * kPanelA);
        for (int i = 0; i < steps; i++) {
            if (ok && !mbar_wait(full + at.s * 8, at.parity)) ok = false;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the asynchronous copies landed through the generic proxy
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long da = a0 + at.s * step16, db = b0 + at.s * step16;  // descriptors count in 16 bytes
            const unsigned d = tmem + acc.s * (unsigned)mb;
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < 8; j++)  // the first step of each accumulator overwrites it
                    umma_f16(d, da + (j >> 2) * (kPanelA >> 4) + (j & 3) * 2, db + (j >> 2) * ((unsigned)panel_b >> 4) + (j & 3) * 2, idesc, i >= p.n_acc || j > 0);
                umma_commit(empty + at.s * 8);  // the stage is free once these MMAs have read it
                if (i == steps - 1) umma_commit(s_addr(bars + 2 * S));
            }
            __syncwarp();
            at.next(S);
            acc.next(p.n_acc);
        }
    }

    // ── epilogue: warps 0-3 read their quarter of the 128 accumulator lanes ──
    if (warp < 4) {
        if (ok && steps > 0 && !mbar_wait(s_addr(bars + 2 * S), 0)) ok = false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int row_in_cta = warp * 32 + lane;           // weight row = accumulator lane
        const int rtg = rt0 + (row_in_cta >> 4);
        int seg = 0;
        long long row;
        if (p.interleave2) {
            seg = rtg & 1;
            row = (long long)(rtg >> 1) * 16 + (row_in_cta & 15);
        } else {
            if (p.n_seg > 1 && rtg >= p.seg_rt0[1]) seg = 1;
            if (p.n_seg > 2 && rtg >= p.seg_rt0[2]) seg = 2;
            row = (long long)(rtg - p.seg_rt0[seg]) * 16 + (row_in_cta & 15);
        }
        const bool row_ok = rtg < p.row_tiles && row < p.seg_n[seg];
        __half* yout = p.y[seg];
        const int acc_used = min(p.n_acc, steps);
        for (int c0 = 0; c0 < mb; c0 += 16) {
            float sum[16];  // adding two to four f32 partial sums rounds to nearest: three roundings at 2^-24
#pragma unroll
            for (int j = 0; j < 16; j++) sum[j] = 0.f;
            for (int a = 0; a < acc_used; a++) {
                unsigned v[16];
                const unsigned addr = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(a * mb + c0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                      "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                    : "r"(addr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; j++) sum[j] += __uint_as_float(v[j]);
            }
            if (splits > 1) {
                float* part = p.partial + ((size_t)split * mb + c0) * p.n_pad + (size_t)(block - p.n_full) * 128 + row_in_cta;
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (ok && p.m0 + c0 + j < p.m_total) part[(size_t)j * p.n_pad] = sum[j];
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const long long mrow = p.m0 + c0 + j;
                    if (ok && row_ok && mrow < p.m_total) yout[mrow * p.seg_n[seg] + row] = __float2half_rn(sum[j]);
                }
            }
        }
    }
    if (!ok && lane == 0) report(p.err, ERR_WAIT_TIMEOUT, p.node, (long long)blockIdx.x, (long long)warp);

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
}

// Adds the pieces of a split-K pass in fixed order and stores the f16 outputs.
struct TcReduceP {
    const float* partial;
    __half* y[3];
    long long m0, m_total, n_pad;
    long long seg_n[3];
    int seg_rt0[4];
    int n_seg, interleave2, row_tiles, mb, splits;
    long long row0;  // first weight row (in stream order) of the tail blocks
};

// Adds the pieces of the row blocks that were cut along K, in piece order, in f64; one rounding. blockIdx.y is the
// activation row, a thread owns four consecutive weight rows (one 16-byte load per piece, the loads of four pieces in
// flight together).
__global__ void __launch_bounds__(256) nbits_gemm_reduce(const TcReduceP p) {
    pdl_enter();
    const int rows = (int)((long long)p.row_tiles * 16 - p.row0);  // a multiple of 16
    const int m = (int)blockIdx.y;
    const int rl = (int)(blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (rl >= rows) return;
    const float4* src = reinterpret_cast<const float4*>(p.partial + (size_t)m * p.n_pad + rl);
    const size_t piece = (size_t)p.mb * p.n_pad / 4;  // float4s between two pieces
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    int sp = 0;
    for (; sp + 4 <= p.splits; sp += 4) {
        const float4 a = src[(size_t)sp * piece], b = src[(size_t)(sp + 1) * piece], c = src[(size_t)(sp + 2) * piece], d = src[(size_t)(sp + 3) * piece];
        acc[0] = (((acc[0] + (double)a.x) + (double)b.x) + (double)c.x) + (double)d.x;
        acc[1] = (((acc[1] + (double)a.y) + (double)b.y) + (double)c.y) + (double)d.y;
        acc[2] = (((acc[2] + (double)a.z) + (double)b.z) + (double)c.z) + (double)d.z;
        acc[3] = (((acc[3] + (double)a.w) + (double)b.w) + (double)c.w) + (double)d.w;
    }
    for (; sp < p.splits; sp++) {
        const float4 a = src[(size_t)sp * piece];
        acc[0] += (double)a.x;
        acc[1] += (double)a.y;
        acc[2] += (double)a.z;
        acc[3] += (double)a.w;
    }
    const long long r = p.row0 + rl;
    const int rtg = (int)(r >> 4);
    int seg = 0;
    long long row;
    if (p.interleave2) {
        seg = rtg & 1;
        row = (long long)(rtg >> 1) * 16 + (r & 15);
    } else {
        if (p.n_seg > 1 && rtg >= p.seg_rt0[1]) seg = 1;
        if (p.n_seg > 2 && rtg >= p.seg_rt0[2]) seg = 2;
        row = (long long)(rtg - p.seg_rt0[seg]) * 16 + (r & 15);
    }
    __half* y = p.y[seg] + (size_t)(p.m0 + m) * p.seg_n[seg];
#pragma unroll
    for (int e = 0; e < 4; e++)
        if (row + e < p.seg_n[seg]) y[row + e] = __double2half(acc[e]);
}

// ───────────────────────────── many activation rows ─────────────────────────────
// nbits_gemm_tc widens a weight again for every 256 activation rows, which is what sets its pace (1.3 µs per 128 k and CTA). Where that costs
// more (wide_pays) the weights are widened once into scratch, as f16 rows that a plain tcgen05 GEMM takes by TMA.
struct WidenP {
    const unsigned char* tiles;  // of this panel
    __half* w;                   // [row tiles · 16][k_tiles · 128]
    int k_tiles, records, tile_bytes, has_zp;
};
// A warp widens one record: lane (g, t) rows g and g + 8 of block t, four 16-byte stores each.
__global__ void __launch_bounds__(256) nbits_widen(const WidenP p) {
    pdl_trigger();
    const int i = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (i >= p.records) {
        pdl_wait();
        return;
    }
    const unsigned char* q = p.tiles + (size_t)i * p.tile_bytes;
    const uint4 wl = __ldg(reinterpret_cast<const uint4*>(q) + lane), wh = __ldg(reinterpret_cast<const uint4*>(q) + 32 + lane);
    const __half2 s2 = *reinterpret_cast<const __half2*>(q + kTileWt + lane * 4);
    const uchar2 z = p.has_zp ? *reinterpret_cast<const uchar2*>(q + kTileWt + kTileSt + lane * 2) : make_uchar2(8, 8);
    const __half2 s2l = __low2half2(s2), s2h = __high2half2(s2);
    const float zl = (float)z.x, zh = (float)z.y;
    const __half2 subl = __float2half2_rn(1024.f + zl), subh = __float2half2_rn(1024.f + zh);
    const __half2 addl = __float2half2_rn(-64.f - zl), addh = __float2half2_rn(-64.f - zh);
    const unsigned wls[4] = {wl.x, wl.y, wl.z, wl.w}, whs[4] = {wh.x, wh.y, wh.z, wh.w};
    const int rt = i / p.k_tiles, kt = i - rt * p.k_tiles;
    const long long ld = (long long)p.k_tiles * 128;
    __half* to = p.w + ((long long)rt * 16 + g) * ld + kt * 128 + t * 32;
    pdl_wait();  // the panel before this one may still be read
#pragma unroll
    for (int m = 0; m < 4; m++) {
        *reinterpret_cast<uint4*>(to + m * 8) = widen_tc(wls[m], subl, addl, s2l);
        *reinterpret_cast<uint4*>(to + 8 * ld + m * 8) = widen_tc(whs[m], subh, addh, s2h);
    }
}

constexpr int kWideRows = 128, kWideWarps = 10, kWideThreads = kWideWarps * 32;  // warps 0-7 epilogue, 8 TMA, 9 MMA
constexpr int kWideStage = 2 * kPanelA, kWideStages = 6;                          // stage: 128 weight rows and 128 activation rows × 64 k
struct WideP {
    alignas(64) unsigned char maps[2][128];  // weights of the panel, activations
    __half* y[3];
    float* partial;              // apart: [pieces][m][n_pad]
    ErrWord* err;
    long long m, n_pad;
    long long seg_n[3];
    int seg_rt0[4];
    int n_seg, interleave2, row_tiles, rt_first;  // rt_first: the panel's first row tile
    int k_tiles, n_full, splits; // as in nbits_gemm_tc: row blocks before n_full take all of k, the others that many pieces
    int apart;                   // pieces are CTAs' work of their own; nbits_gemm_reduce adds them up
    int m_tiles, o_tiles, node;
    int y_odd;                   // rows of some result do not begin on four bytes
};
// Persistent CTAs, 128 weight rows × 128 activation rows per tile. Every sum is formed as nbits_gemm_tc forms it, bit for bit: 128-k steps go in
// turn into two accumulators, which are added in f32 (the tensor core adds without rounding to nearest: shorter chains), and the pieces
// of k are added in f64. A piece's accumulators are read, half of the columns per group of four warps, while the next piece runs in the other two.
// A result of one piece is an f32 value: it is rounded as such, without the way through f64, and two rows are stored at a time. With that and the rings' stage and parity
// carried along instead of divided out of a counter (both kernels), widening included, the same bits, µs: 2047 × 1152 × 13 824 107 → 84, 2047 × 6912 × 1152 59 → 50, 4096 × 5376 ×
// 5376 340 → 293, 512 × 1152 × 13 824 41 → 35; nbits_gemm_tc, which also takes its tensor memory and first weights before the launches in front of it end, 64 × 4096 × 5376
// 18.7 → 16.3, 64 × 5376 × 43 008 78 → 72, 16 × 5376 × 43 008 70 → 62. What is left in the wide kernel is the 32 KB that a step brings to an SM (64 bytes a cycle).
__global__ void __launch_bounds__(kWideThreads, 1) nbits_gemm_wide(const __grid_constant__ WideP p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + kWideStages * kWideStage);  // full, empty, finished[2], read[2]
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * kWideStages + 4);
    const unsigned full = s_addr(bars), empty = full + kWideStages * 8, finished = empty + kWideStages * 8, read = finished + 16;
    if (tid == 0) {
        for (int s = 0; s < 2 * kWideStages + 2; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + s * 8) : "memory");
        for (int s = 0; s < 2; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(read + s * 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(s_addr(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;
    pdl_trigger();
    pdl_wait();
    const int units = p.m_tiles * p.o_tiles * (p.apart ? p.splits : 1);  // activation tiles fastest, pieces slowest
    // a unit's tile and pieces; a piece's 128-k steps
    struct Unit {
        int m0, o0, pieces, from, to;
    };
    auto unit_of = [&](int u) {
        Unit q;
        const int rest = u / p.m_tiles, o = rest % p.o_tiles;
        q.m0 = u % p.m_tiles * kWideRows;
        q.o0 = o * 128;
        q.pieces = (p.rt_first >> 3) + o < p.n_full ? 1 : p.splits;
        q.from = p.apart ? rest / p.o_tiles : 0;
        q.to = p.apart ? q.from + 1 : q.pieces;
        return q;
    };
    auto first_step = [&](const Unit& q, int piece) { return (int)((long long)p.k_tiles * piece / q.pieces); };
    bool ok = true;
    if (warp == 8) {
        RingAt at;
        bool round = false;  // the ring's first round waits for nothing
        const unsigned data = s_addr(smem);
        for (int u = (int)blockIdx.x; u < units; u += (int)gridDim.x) {
            const Unit q = unit_of(u);
            const int lo = first_step(q, q.from) * 2, hi = first_step(q, q.to) * 2;  // 64-k steps; pieces follow one another
            for (int i = lo; i < hi; i++) {
                if (!__all_sync(0xffffffffu, !round || mbar_wait(empty + at.s * 8, at.parity ^ 1))) {
                    ok = false;
                    break;
                }
                const unsigned bar = full + at.s * 8, dst = data + at.s * kWideStage;
                if (elect_one()) {
                    mbar_expect_tx(bar, (unsigned)kWideStage);
                    tma_load_2d(dst, p.maps[0], i * 64, q.o0, bar);
                    tma_load_2d(dst + kPanelA, p.maps[1], i * 64, q.m0, bar);
                }
                __syncwarp();
                at.next(kWideStages);
                if (at.s == 0) round = true;
            }
            if (!__all_sync(0xffffffffu, ok)) break;
        }
        // every copy has landed before this CTA's shared memory can be given away
        for (unsigned n = 0; n < (round ? (unsigned)kWideStages : at.s); n++)
            if (!mbar_wait(full + n * 8, n < at.s ? at.parity : at.parity ^ 1)) ok = false;
    } else if (warp == 9) {
        const unsigned idesc = (1u << 4) | ((kWideRows >> 3) << 17) | (8u << 24);  // f16 × f16 → f32, M 128 × N 128
        RingAt at;
        bool ready = false;
        int j = 0;
        const unsigned long long a0 = umma_kmajor_desc(s_addr(smem)), b0 = umma_kmajor_desc(s_addr(smem) + kPanelA);
        for (int u = (int)blockIdx.x; u < units; u += (int)gridDim.x) {
            const Unit q = unit_of(u);
            for (int piece = q.from; piece < q.to; piece++, j++) {
                const int n = first_step(q, piece + 1) - first_step(q, piece);
                const unsigned d = tmem + (unsigned)((j & 1) * 2 * kWideRows);
                if (j >= 2 && ok && !mbar_wait(read + (j & 1) * 8, ((j >> 1) - 1) & 1)) ok = false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = 0; i < 2 * n; i++) {
                    if (ok && !ready && !mbar_wait(full + at.s * 8, at.parity)) ok = false;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned long long a = a0 + at.s * (kWideStage >> 4), b = b0 + at.s * (kWideStage >> 4);  // descriptors count in 16 bytes
                    const unsigned done = empty + at.s * 8, to = d + (unsigned)((i >> 1 & 1) * kWideRows);
                    at.next(kWideStages);
                    ready = mbar_test(full + at.s * 8, at.parity);  // the answer is there when the products have been issued
                    if (elect_one() && ok) {
#pragma unroll
                        for (int e = 0; e < 4; e++) umma_f16(to, a + e * 2, b + e * 2, idesc, i >= 4 || (i & 1) || e > 0);
                        umma_commit(done);
                    }
                    __syncwarp();
                }
                if (elect_one()) umma_commit(finished + (j & 1) * 8);
                __syncwarp();
            }
        }
    } else {
        constexpr int kCols = kWideRows / 2;
        const int lanes = (warp & 3) * 32, col0 = (warp >> 2) * kCols, odd = lane & 1;
        int j = 0;
        for (int u = (int)blockIdx.x; u < units; u += (int)gridDim.x) {
            const Unit q = unit_of(u);
            const long long m0 = q.m0 + col0;
            const int row_in_panel = q.o0 + lanes + lane, rtg = p.rt_first + (row_in_panel >> 4);
            int seg = 0;
            long long row;
            if (p.interleave2) {
                seg = rtg & 1;
                row = (long long)(rtg >> 1) * 16 + (row_in_panel & 15);
            } else {
                if (p.n_seg > 1 && rtg >= p.seg_rt0[1]) seg = 1;
                if (p.n_seg > 2 && rtg >= p.seg_rt0[2]) seg = 2;
                row = (long long)(rtg - p.seg_rt0[seg]) * 16 + (row_in_panel & 15);
            }
            const long long width = p.seg_n[seg];
            const bool row_ok = ok && rtg < p.row_tiles && row < width;
            const int there = (int)min((long long)kCols, p.m - m0);  // activation rows of these columns that exist
            // 16 columns of a piece: its two accumulators added in f32
            auto part_of = [&](int piece, int c, float (&part)[16]) {
                const int accs = min(2, first_step(q, piece + 1) - first_step(q, piece));
                const unsigned d = tmem + (unsigned)((j & 1) * 2 * kWideRows + col0 + c) + ((unsigned)lanes << 16);
#pragma unroll
                for (int e = 0; e < 16; e++) part[e] = 0.f;
                for (int a = 0; a < accs; a++) {
                    unsigned v[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                        : "r"(d + (unsigned)(a * kWideRows)));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 16; e++) part[e] += __uint_as_float(v[e]);
                }
            };
            auto piece_begin = [&] {
                if (ok && !mbar_wait(finished + (j & 1) * 8, (j >> 1) & 1)) ok = false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            };
            auto piece_end = [&] {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(read + (j & 1) * 8);
                j++;
            };
            // 16 columns as f16. Rows of neighbouring lanes are neighbours and of one segment: of two columns the even lane stores both rows of the first, the odd
            // lane of the second, where that is 32-bit aligned.
            auto store = [&](int c, const __half (&h)[16]) {
                if (!p.y_odd) {  // for all lanes alike: half of them may be of another segment
                    unsigned w[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const unsigned mine = __half_as_ushort(odd ? h[2 * e + 1] : h[2 * e]), got = __shfl_xor_sync(0xffffffffu, (unsigned)__half_as_ushort(odd ? h[2 * e] : h[2 * e + 1]), 1);
                        w[e] = odd ? got | mine << 16 : mine | got << 16;
                    }
                    __half* y = p.y[seg] + (m0 + c + odd) * width + (row & ~1ll);
#pragma unroll
                    for (int e = 0; e < 8; e++, y += 2 * width)
                        if (row_ok && c + 2 * e + odd < there) *reinterpret_cast<unsigned*>(y) = w[e];
                } else {
                    __half* y = p.y[seg] + (m0 + c) * width + row;
#pragma unroll
                    for (int e = 0; e < 16; e++, y += width)
                        if (row_ok && c + e < there) *y = h[e];
                }
                __syncwarp();
            };
            if (q.to - q.from == 1) {  // one piece: its f32 sums are the results, or the partial sums
                piece_begin();
#pragma unroll
                for (int c = 0; c < kCols; c += 16) {
                    float part[16];
                    part_of(q.from, c, part);
                    if (p.apart) {
                        float* to = p.partial + ((size_t)q.from * p.m + m0 + c) * p.n_pad + row_in_panel;
#pragma unroll
                        for (int e = 0; e < 16; e++, to += p.n_pad)
                            if (ok && c + e < there) *to = part[e];
                    } else {
                        __half h[16];
#pragma unroll
                        for (int e = 0; e < 16; e++) h[e] = __float2half_rn(part[e]);
                        store(c, h);
                    }
                }
                piece_end();
                continue;
            }
            double sum[kCols];
#pragma unroll
            for (int e = 0; e < kCols; e++) sum[e] = 0.0;
            for (int piece = q.from; piece < q.to; piece++) {
                piece_begin();
#pragma unroll
                for (int c = 0; c < kCols; c += 16) {
                    float part[16];
                    part_of(piece, c, part);
#pragma unroll
                    for (int e = 0; e < 16; e++) sum[c + e] += (double)part[e];
                }
                piece_end();
            }
#pragma unroll
            for (int c = 0; c < kCols; c += 16) {
                __half h[16];
#pragma unroll
                for (int e = 0; e < 16; e++) h[e] = __double2half(sum[c + e]);
                store(c, h);
            }
        }
    }
    if (!ok && lane == 0) report(p.err, ERR_WAIT_TIMEOUT, p.node, (long long)blockIdx.x, (long long)warp);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Row tiles of a panel: at most 64 MB of widened weights, which stay in L2 until the product reads them.
int panel_tiles(const TcP& t) { return (int)std::max<long long>(8, (64LL << 20) / ((long long)t.k_tiles * 128 * 32) / 8 * 8); }

// Few tiles: the pieces of k go to CTAs of their own where that, with the partial sums' trip (5 TB/s) and a second launch, is shorter.
bool pieces_apart(const TcP& t, long long m, int count) {
    const long long slots = sm_count(), ctas = (m + kWideRows - 1) / kWideRows * ((count + 7) / 8);
    const double step_us = 0.45;  // 128 k of a tile
    const double joined = (double)((ctas + slots - 1) / slots) * t.k_tiles * step_us;
    const double apart = (double)((ctas * t.splits + slots - 1) / slots) * ((double)t.k_tiles / t.splits * step_us + 1.0) + 3.0 +
                         (double)t.splits * m * ((count + 7) / 8 * 128) * 8.0 / 5e6;
    return t.splits > 1 && t.n_full == 0 && apart < joined;
}

// Whether the weights are widened once, for m rows whose launches of nbits_gemm_tc are `t`. Both sides as sums of what they do, fitted to 459 times of either by kernels that took 5 … 20 %
// longer than these. Against 267 times of either by these (30 sizes, k 512 … 21 504, 1024 … 43 008 weight rows, 257 … 4096 activation rows), with a tenth of margin: what is taken is at
// most 0.89 of nbits_gemm_tc; over all 0.600 of its time in the geometric mean, 0.588 with the better of the two at each size. What is not taken would be up to 28 % shorter, of large
// products above all (k 4096, 22 016 weight rows, 3000 rows: 837 and 604 µs), the wide kernel having gained more. nbits_gemm_tc → widened once, µs, at 257, 1024 and 4096 rows, in
// brackets what is not taken: k 1152, 13 824 weight rows 53 → 40, 112 → 62, 420 → 163; k 2560, 20 480: 99 → (111), 220 → (173), 836 → 468; k 5376, 5376: 61 → (61), 136 → (104),
// 485 → 271; k 5376, 43 008 (2047 rows for 4096): 281 → (346), 591 → (643), 1170 → (1109); k 6912, 1152: 49 → 37, 86 → 52, 314 → 90; k 21 504, 5376: 146 → (241), 296 → (383),
// 1147 → (1137).
bool wide_pays(const TcP& t, long long m) {
    const long long slots = sm_count(), grid = (t.row_tiles + 7) / 8, tail = grid - t.n_full;
    const double out_mb = (double)m * t.row_tiles * 32.0 / 1e6;
    const long long full = (t.n_full + slots - 1) / slots, cut = tail > 0 ? (tail * t.splits + slots - 1) / slots : 0;  // rounds of CTAs
    const double steps = (double)full * t.k_tiles + (double)cut * t.k_tiles / t.splits, sums_mb = t.splits > 1 ? (double)t.splits * t.mb * tail * 128 * 8.0 / 1e6 : 0.0;
    const double passes_us = (double)((m + t.mb - 1) / t.mb) * (3.65 + 1.036 * steps + 11.1 * (double)full + 6.5 * (double)cut + 0.12 * sums_mb) + 0.59 * out_mb;
    double wide_us = 5.5 + 0.38 * out_mb;
    for (int first = 0, size = panel_tiles(t); first < t.row_tiles; first += size) {
        const int count = std::min(size, t.row_tiles - first), pieces = pieces_apart(t, m, count) ? t.splits : 1;
        const long long o_tiles = (count + 7) / 8, rounds = ((m + kWideRows - 1) / kWideRows * o_tiles * pieces + slots - 1) / slots;
        wide_us += 2.5 * (pieces > 1 ? 3 : 2) + 0.69 * (double)rounds * t.k_tiles / pieces + 0.23 * (double)count * 16 * t.k_tiles * 128 * 2.5 / 1e6;
        if (pieces > 1) wide_us += 0.14 * (double)pieces * m * o_tiles * 128 * 8.0 / 1e6;
    }
    return wide_us < 0.9 * passes_us;
}

// `t`: the launch of nbits_gemm_tc for these rows (its pieces of k are kept). The activations come by tensor map alone: their offset in the
// buffer is checked by the caller, and buffers (arena granules, the pool's, a caller's whole tensors) begin on 256 bytes.
void emit_wide(Emitter& em, const NBitsGroup& gr, const TRef& x, const TRef& tiles, const TcP& t) {
    const Buf null{kSlotNull, 0};
    const long long ld = (long long)t.k_tiles * 128;
    const int per_panel = panel_tiles(t);
    const Buf wide = em.scratch((size_t)std::min(per_panel, (t.row_tiles + 7) / 8 * 8) * 16 * ld * 2);
    for (int first = 0; first < t.row_tiles; first += per_panel) {
        const int count = std::min(per_panel, t.row_tiles - first);
        WidenP a{};
        a.k_tiles = t.k_tiles;
        a.records = count * t.k_tiles;
        a.tile_bytes = t.tile_bytes;
        a.has_zp = t.has_zp;
        em.launch(nbits_widen, dim3((unsigned)((a.records + 7) / 8)), dim3(256), 0, a,
                  {{&a.tiles, tiles.buf.at((int64_t)first * t.k_tiles * t.tile_bytes)}, {&a.w, wide}}, "nbits_widen", /*pdl=*/true);
        WideP p{};
        p.m = gr.m;
        p.k_tiles = t.k_tiles;
        p.n_full = t.n_full;
        p.splits = t.splits;
        p.n_seg = t.n_seg;
        p.interleave2 = t.interleave2;
        p.row_tiles = t.row_tiles;
        p.rt_first = first;
        p.node = em.node;
        for (int i = 0; i < 3; i++) p.seg_n[i] = t.seg_n[i];
        for (int i = 0; i < 4; i++) p.seg_rt0[i] = t.seg_rt0[i];
        p.m_tiles = (int)((gr.m + kWideRows - 1) / kWideRows);
        for (int i = 0; i < gr.n_seg; i++) p.y_odd |= gr.y[i].buf.off % 4 != 0 || p.seg_n[i] % 2 != 0;
        p.o_tiles = (count + 7) / 8;
        p.n_pad = (long long)p.o_tiles * 128;
        const long long slots = sm_count(), ctas = (long long)p.m_tiles * p.o_tiles;
        p.apart = pieces_apart(t, gr.m, count);
        const Buf partial = p.apart ? em.scratch((size_t)p.splits * gr.m * p.n_pad * 4) : null;
        const size_t smem = kWideStages * kWideStage + 1024 + (2 * kWideStages + 4) * 8 + 16;
        ensure_max_dynamic_smem((const void*)nbits_gemm_wide, 220 * 1024);
        LaunchRec& rec = em.launch(nbits_gemm_wide, dim3((unsigned)std::min<long long>(slots, ctas * (p.apart ? p.splits : 1))), dim3(kWideThreads), (unsigned)smem, p,
                                   {{&p.err, Buf{kSlotErr, 0}}, {&p.partial, partial}, {&p.y[0], gr.y[0].buf}, {&p.y[1], gr.n_seg > 1 ? gr.y[1].buf : null},
                                    {&p.y[2], gr.n_seg > 2 ? gr.y[2].buf : null}},
                                   "nbits_gemm_wide", /*pdl=*/true);
        rec.tmaps.push_back(TmapReloc{(uint32_t)offsetof(WideP, maps), wide, (uint64_t)ld, (uint64_t)count * 16, (uint64_t)ld * 2, 64u, 128u});
        rec.tmaps.push_back(TmapReloc{(uint32_t)offsetof(WideP, maps) + 128, x.buf, (uint64_t)gr.k, (uint64_t)gr.m, (uint64_t)gr.k * 2, 64u, (uint32_t)kWideRows});
        if (p.apart) {
            TcReduceP q{};
            q.m_total = gr.m;
            q.n_pad = p.n_pad;
            q.n_seg = p.n_seg;
            q.interleave2 = p.interleave2;
            q.row_tiles = first + count;
            q.mb = (int)gr.m;
            q.splits = p.splits;
            q.row0 = (long long)first * 16;
            for (int i = 0; i < 3; i++) q.seg_n[i] = p.seg_n[i];
            for (int i = 0; i < 4; i++) q.seg_rt0[i] = p.seg_rt0[i];
            em.launch(nbits_gemm_reduce, dim3((unsigned)((count * 4 + 255) / 256), (unsigned)gr.m), dim3(256), 0, q,
                      {{&q.partial, partial}, {&q.y[0], gr.y[0].buf}, {&q.y[1], gr.n_seg > 1 ? gr.y[1].buf : null},
                       {&q.y[2], gr.n_seg > 2 ? gr.y[2].buf : null}},
                      "nbits_gemm_reduce", /*pdl=*/true);
        }
    }
}

}  // namespace

// The GEMM form of a MatMulNBits group (no prologue, no epilogue: the caller runs those as
// separate launches). `interleave2`: the stream alternates row tiles of segment 0 and 1.
void emit_nbits_gemm_tc(Emitter& em, const NBitsGroup& gr, const TRef& x, const TRef& tiles, bool interleave2) {
    if (gr.m == 0) return;
    TcP p{};
    p.m_total = gr.m;
    p.k = gr.k;
    p.k_tiles = (int)(((gr.k + 31) / 32 + 3) / 4);
    p.n_seg = gr.n_seg;
    p.interleave2 = interleave2 ? 1 : 0;
    int rt = 0;
    for (int i = 0; i < gr.n_seg; i++) {
        p.seg_n[i] = gr.seg_n[i];
        p.seg_rt0[i] = rt;
        rt += (int)((gr.seg_n[i] + 15) / 16);
    }
    p.seg_rt0[gr.n_seg] = rt;
    p.row_tiles = rt;
    p.has_zp = gr.has_zp ? 1 : 0;
    p.tile_bytes = kTileWt + kTileSt + (gr.has_zp ? kTileZt : 0);
    p.node = em.node;
    // activation rows per pass: the smallest MMA N that holds them all, at most 256
    int mb = 16;
    while (mb < gr.m && mb < 256) mb <<= 1;
    p.mb = mb;
    const size_t stage = 2 * (size_t)kPanelA + 2 * (size_t)mb * 128;
    // two CTAs per SM where two stages of each fit in half the shared memory, else one CTA with up to 4
    const size_t half_sm = 110 * 1024, whole_sm = 216 * 1024;
    p.stages = (int)std::min<size_t>(4, (2 * stage <= half_sm ? half_sm : whole_sm) / stage);
    if (p.stages < 2) p.stages = 2;
    p.n_acc = mb <= 128 ? 4 : 2;  // 512 columns of tensor memory per SM; two CTAs share it when mb ≤ 64
    p.use_tma = (gr.k % 8 == 0 && x.buf.off % 16 == 0) ? 1 : 0;
    const size_t smem = stage * p.stages + 1024 /*alignment slack*/ + (2 * p.stages + 1) * 8 + 16;
    ensure_max_dynamic_smem((const void*)nbits_gemm_tc, 220 * 1024);
    const Buf null{kSlotNull, 0};
    const unsigned grid = (unsigned)((p.row_tiles + 7) / 8);
    // Whole waves of row blocks take all of K. The blocks left over (all of them when there is less than one
    // wave) are cut into the number of pieces that minimises, in units of one 128-k step (≈ 1.3 µs),
    // waves × (steps per piece + about four steps of set-up and drain per CTA) + the second kernel's launch
    // and the partial sums' trip to memory and back; at least two steps per piece.
    const long long slots = (long long)sm_count() * (2 * stage <= half_sm ? 2 : 1);
    long long n_full = (long long)grid / slots * slots, tail = grid - n_full;
    if (tail * 10 >= slots * 6) {  // the last wave is well filled as it is
        n_full = grid;
        tail = 0;
    }
    int splits = 1;
    if (tail > 0) {
        double best = 1e300;
        for (int sp = 1; sp <= 8 && sp * 2 <= std::max(p.k_tiles, 2); sp++) {
            const long long waves = (tail * sp + slots - 1) / slots;
            double cost = (double)waves * ((double)p.k_tiles / sp + 4.0);
            if (sp > 1) cost += 2.5 + (double)sp * mb * (double)tail * 128 * 8.0 / 3.9e6;
            if (cost < best * 0.97) {  // a larger count has to earn its extra pass over the partial sums
                best = cost;
                splits = sp;
            }
        }
    }
    if (const char* e = std::getenv("ONYXIA_GEMM_SPLITS")) {  // diagnostics: every row block cut into that many pieces
        splits = std::max(1, std::min({std::atoi(e), 8, std::max(p.k_tiles, 1)}));
        n_full = 0;
        tail = grid;
    }
    if (splits == 1) {
        n_full = grid;
        tail = 0;
    }
    static const bool debug = std::getenv("ONYXIA_GEMM_DEBUG") != nullptr;  // diagnostics
    if (debug) std::fprintf(stderr, "nbits_gemm_tc: m %lld k_tiles %d grid %u mb %d: %d pieces over %lld of the row blocks\n", gr.m, p.k_tiles, grid, mb, splits, tail);
    p.n_full = (int)n_full;
    p.splits = splits;
    if (gr.m > 256 && gr.m < 65536 && gr.k % 8 == 0 && x.buf.off % 16 == 0 && wide_pays(p, gr.m)) return emit_wide(em, gr, x, tiles, p);
    p.n_pad = tail * 128;
    const Buf partial = splits > 1 ? em.scratch((size_t)splits * mb * p.n_pad * sizeof(float)) : null;
    for (long long m0 = 0; m0 < gr.m; m0 += mb) {
        p.m0 = m0;
        LaunchRec& rec = em.launch(nbits_gemm_tc, dim3((unsigned)(n_full + tail * splits)), dim3(kThreadsTc), (unsigned)smem, p,
                  {{&p.x, x.buf}, {&p.tiles, tiles.buf}, {&p.err, Buf{kSlotErr, 0}}, {&p.partial, partial}, {&p.y[0], gr.y[0].buf},
                   {&p.y[1], gr.n_seg > 1 ? gr.y[1].buf : null}, {&p.y[2], gr.n_seg > 2 ? gr.y[2].buf : null}},
                  "nbits_gemm_tc", /*pdl=*/true);
        if (p.use_tma)
            rec.tmaps.push_back(TmapReloc{(uint32_t)offsetof(TcP, xmap), x.buf, (uint64_t)gr.k, (uint64_t)gr.m, (uint64_t)gr.k * 2, 64u, (uint32_t)mb,
                                          (uint32_t)offsetof(TcP, use_tma)});
        if (splits > 1) {
            TcReduceP q{};
            q.m0 = m0;
            q.m_total = gr.m;
            q.n_pad = p.n_pad;
            q.n_seg = p.n_seg;
            q.interleave2 = p.interleave2;
            q.row_tiles = p.row_tiles;
            q.mb = mb;
            q.splits = splits;
            q.row0 = n_full * 128;
            for (int i = 0; i < 3; i++) q.seg_n[i] = p.seg_n[i];
            for (int i = 0; i < 4; i++) q.seg_rt0[i] = p.seg_rt0[i];
            const long long rows = (long long)p.row_tiles * 16 - q.row0, m_here = std::min<long long>(mb, gr.m - m0);
            em.launch(nbits_gemm_reduce, dim3((unsigned)((rows / 4 + 255) / 256), (unsigned)m_here), dim3(256), 0, q,
                      {{&q.partial, partial}, {&q.y[0], gr.y[0].buf}, {&q.y[1], gr.n_seg > 1 ? gr.y[1].buf : null},
                       {&q.y[2], gr.n_seg > 2 ? gr.y[2].buf : null}},
                      "nbits_gemm_reduce", /*pdl=*/true);
        }
    }
}

}  // namespace oxk
