// Dense products over unquantised weights, y = x · Wᵀ, and the residual norm in front of them.
//
//   linear_stream   up to 32 rows (decode): a warp reads 16 weight rows × 32 k straight into `mma.sync` A fragments (a dot
//                   product does not care in which order its k are visited, so a lane takes 16 consecutive bytes of
//                   a row), eight warps share a row tile's k. Weight loads run one batch ahead and start before the
//                   grid dependency resolves. For up to eight rows the residual norm that makes x runs as the
//                   prologue, in every CTA.
//   linear_flow     the same for large matrices (above eight rows where k is not long): more of their weights in flight, through shared memory.
//   linear_tc       more rows: tcgen05 GEMM. Weights are the MMA's A operand (128 rows), activations its B operand
//                   (32–256 rows), both loaded by TMA into 128-byte-swizzled stages; accumulator in tensor memory.
//                   Grids that would leave SMs idle are cut along k; `linear_reduce` adds the pieces in order.
//   linear_pair     products of many rows and groups of many rows (linear_pair.cu).
//   linear_rows_f32 f32 (true 32-bit), up to 32 rows and k of 512 and more: warps stream whole weight rows.
//   linear_f32      f32, more rows or shorter k: register-blocked tiles.
//   linear_simt     f32 of short k, and f32 and bf16 shapes whose rows are not 16-byte aligned.
//
// linear_tc, linear_pair, linear_f32 and linear_simt also run grouped: activation rows sorted by group, one weight matrix per group, the groups'
// row counts known on the device only. A CTA finds its group from the counts; the grid covers the most tiles
// that any counts can give.
//
// Bytes per launch: out · k · 2 once per 256 activation rows; FLOPs 2 · rows · out · k.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "linear.cuh"

namespace oxk {

namespace {

// ───────────────────────────── decode ───────────────────────────────────
constexpr int kStreamWarps = 8, kThreads = kStreamWarps * 32;

__device__ __forceinline__ uint4 ld_weights(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <bool YB> __device__ __forceinline__ float4 ld_y4(const void* y, long long i) {
    if constexpr (YB) {
        const uint2 v = *reinterpret_cast<const uint2*>((const bf16*)y + i);
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u));
    } else {
        return *reinterpret_cast<const float4*>((const float*)y + i);
    }
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
// Rows 0 … rows−1 of the residual norm into shared memory (bf16, `stride` elements per row); CTA 0 stores the residual
// and the low-precision copy. Eight warps; `per` of them work on one row. K is a multiple of 8.
template <bool YB> __device__ void norm_prologue(const LinP& p, bf16* xs, int stride, float* red) {
    const int rows = (int)p.rows, K = (int)p.k[0], warp = threadIdx.x >> 5;
    const int per = rows <= 1 ? 8 : rows <= 2 ? 4 : rows <= 4 ? 2 : 1;
    const int row = warp / per, t = ((warp % per) * 32 + (threadIdx.x & 31)) * 4, step = per * 128;
    const long long base = (long long)row * K, y0 = (long long)row * p.ny_ld;
    auto rstd_of = [&](float ss) {  // of this row, from every thread's share of the squares
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) red[warp] = ss;
        __syncthreads();
        float tot = 0.f;
        if (row < rows)
            for (int i = 0; i < per; i++) tot += red[row * per + i];
        return 1.f / sqrtf(tot / (float)K + p.eps);
    };
    float inner = p.y_scale;  // with `post`: one over the root mean square of y
    if (p.npost) {
        float ss = 0.f;
        if (row < rows) {
#pragma unroll 8
            for (int i = t; i < K; i += step) {
                const float4 v = ld_y4<YB>(p.ny, y0 + i);
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
        }
        inner = rstd_of(ss);
        __syncthreads();  // red is written again
    }
    auto normed = [&](int i) {  // what the mean square is taken of
        float4 v = ld_y4<YB>(p.ny, y0 + i);
        if (p.pre) {
            v = make_float4(v.x * inner, v.y * inner, v.z * inner, v.w * inner);
            if (p.npost) v = mul4(v, *reinterpret_cast<const float4*>(p.npost + i));
            if (p.nres) v = add4(v, *reinterpret_cast<const float4*>(p.nres + base + i));
            if (p.nadd) {
                const float4 r = p.add_bf16 ? ld_y4<true>(p.nadd, base + i) : ld_y4<false>(p.nadd, base + i);
                v = make_float4(fmaf(r.x, p.add_scale, v.x), fmaf(r.y, p.add_scale, v.y), fmaf(r.z, p.add_scale, v.z), fmaf(r.w, p.add_scale, v.w));
            }
            if (p.noffset) v = add4(v, *reinterpret_cast<const float4*>(p.noffset + i));
        }
        return v;
    };
    float ss = 0.f;
    if (row < rows) {
#pragma unroll 8
        for (int i = t; i < K; i += step) {
            const float4 v = normed(i);
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        }
    }
    const float rstd = rstd_of(ss);
    if (row < rows) {
#pragma unroll 4
        for (int i = t; i < K; i += step) {
            const float4 sum = normed(i), w = *reinterpret_cast<const float4*>(p.nw + i);
            float4 v = mul4(make_float4(sum.x * rstd, sum.y * rstd, sum.z * rstd, sum.w * rstd), w);
            if (p.ngain) v = mul4(v, *reinterpret_cast<const float4*>(p.ngain + i));
            if (p.ngate) v = mul4(v, ld_y4<true>(p.ngate, row * p.gate_ld + i));
            if (!p.pre && p.nres) v = add4(v, *reinterpret_cast<const float4*>(p.nres + base + i));
            const uint2 packed = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
            *reinterpret_cast<uint2*>(xs + (long long)row * stride + i) = packed;
            if (blockIdx.x == 0 && p.stream) *reinterpret_cast<float4*>(p.stream + base + i) = p.pre ? sum : v;
            if (blockIdx.x == 0 && p.low) *reinterpret_cast<uint2*>(p.low + base + i) = packed;
        }
    }
    __syncthreads();
}

// The same for a residual of several streams. Every CTA forms the norm's operand, and stores its share of the new streams.
template <bool YB> __device__ void streams_prologue(const LinP& p, bf16* xs, int stride, float* red) {
    const int rows = (int)p.rows, K = (int)p.k[0], S = p.streams, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = rows <= 1 ? 8 : rows <= 2 ? 4 : rows <= 4 ? 2 : 1;
    const int row = warp / per, t = ((warp % per) * 32 + lane) * 4, step = per * 128;
    const long long y0 = (long long)row * p.ny_ld, base = (long long)row * K;
    const float* res = p.nres + base * S;
    __shared__ float con[kMaxStreams * (kMaxStreams + 2)], take[kMaxStreams + 1];  // take: what the operand takes of every old stream and of y
    for (int i = threadIdx.x; i < S * (S + 2); i += kThreads) con[i] = p.connect[i];
    __syncthreads();
    const float *out = con + S * S, *in = out + S;
    if ((int)threadIdx.x <= S) {
        float a = 0.f;
        for (int u = 0; u < S; u++) a = fmaf(in[u], (int)threadIdx.x < S ? con[threadIdx.x * S + u] : out[u], a);
        take[threadIdx.x] = a;
    }
    float f1 = p.y_scale, f2 = 0.f;
    auto total_of = [&](float ss) {  // of this row
        ss = warp_sum(ss);
        __syncthreads();
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        float tot = 0.f;
        if (row < rows)
            for (int i = 0; i < per; i++) tot += red[row * per + i];
        return 1.f / sqrtf(tot / (float)K + p.eps);
    };
    auto squares = [&](const void* y, long long at) {
        float ss = 0.f;
        if (row < rows) {
#pragma unroll 4
            for (int i = t; i < K; i += step) {
                const float4 v = ld_y4<YB>(y, at + i);
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
        }
        return ss;
    };
    if (p.npost) f1 = total_of(squares(p.ny, y0));
    if (p.ny2) f2 = total_of(squares(p.ny2, base));
    __syncthreads();
    auto result = [&](int i) {  // y'
        float4 v = ld_y4<YB>(p.ny, y0 + i);
        v = make_float4(v.x * f1, v.y * f1, v.z * f1, v.w * f1);
        if (p.npost) v = mul4(v, *reinterpret_cast<const float4*>(p.npost + i));
        if (p.ny2) {
            const float4 o = ld_y4<YB>(p.ny2, base + i), w = *reinterpret_cast<const float4*>(p.npost2 + i);
            v = add4(v, make_float4(o.x * f2 * w.x, o.y * f2 * w.y, o.z * f2 * w.z, o.w * f2 * w.w));
        }
        return v;
    };
    auto plus = [](float4 a, float f, float4 b) { return make_float4(fmaf(f, b.x, a.x), fmaf(f, b.y, a.y), fmaf(f, b.z, a.z), fmaf(f, b.w, a.w)); };
    auto operand = [&](int i, float4 y) {
        float4 v = plus(make_float4(0.f, 0.f, 0.f, 0.f), take[S], y);
        if (p.nres)
#pragma unroll 4
            for (int r = 0; r < S; r++) v = plus(v, take[r], *reinterpret_cast<const float4*>(res + (long long)r * K + i));
        return v;
    };
    float ss = 0.f;
    if (row < rows)
#pragma unroll 2
        for (int i = t; i < K; i += step) {
            const float4 y = result(i), v = operand(i, y);
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            if (p.stream && (row + i / 128 * rows) % gridDim.x == blockIdx.x)  // (128 elements of a row: one warp)
                for (int u = 0; u < S; u++) {
                    float4 s = plus(make_float4(0.f, 0.f, 0.f, 0.f), out[u], y);
                    if (p.nres)
                        for (int r = 0; r < S; r++) s = plus(s, con[r * S + u], *reinterpret_cast<const float4*>(res + (long long)r * K + i));
                    *reinterpret_cast<float4*>(p.stream + base * S + (long long)u * K + i) = s;
                }
        }
    const float rstd = total_of(ss);
    if (row < rows) {
#pragma unroll 2
        for (int i = t; i < K; i += step) {
            const float4 u = operand(i, result(i)), w = *reinterpret_cast<const float4*>(p.nw + i);
            const uint2 packed = make_uint2(pack_bf16(u.x * rstd * w.x, u.y * rstd * w.y), pack_bf16(u.z * rstd * w.z, u.w * rstd * w.w));
            *reinterpret_cast<uint2*>(xs + (long long)row * stride + i) = packed;
            if (blockIdx.x == 0 && p.low) *reinterpret_cast<uint2*>(p.low + base + i) = packed;
        }
    }
    __syncthreads();
}

// The same for a norm of several runs of columns: a warp takes a row's run at a time.
template <bool YB> __device__ void groups_prologue(const LinP& p, bf16* xs, int stride) {
    const int rows = (int)p.rows, K = (int)p.k[0], G = p.norm_groups, size = K / G, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int unit = warp; unit < rows * G; unit += kThreads / 32) {
        const int row = unit / G, at = unit % G * size;
        const long long y0 = (long long)row * p.ny_ld + at;
        float ss = 0.f;
        for (int i = lane * 4; i < size; i += 128) {
            const float4 v = ld_y4<YB>(p.ny, y0 + i);
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        }
        const float rstd = 1.f / sqrtf(warp_sum(ss) / (float)size + p.eps);
        for (int i = lane * 4; i < size; i += 128) {
            float4 v = ld_y4<YB>(p.ny, y0 + i);
            v = mul4(make_float4(v.x * rstd, v.y * rstd, v.z * rstd, v.w * rstd), *reinterpret_cast<const float4*>(p.nw + at + i));
            if (p.ngate) v = mul4(v, ld_y4<true>(p.ngate, row * p.gate_ld + at + i));
            const uint2 packed = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
            *reinterpret_cast<uint2*>(xs + (long long)row * stride + at + i) = packed;
            if (blockIdx.x == 0 && p.low) *reinterpret_cast<uint2*>(p.low + (long long)row * K + at + i) = packed;
            if (blockIdx.x == 0 && p.stream) *reinterpret_cast<float4*>(p.stream + (long long)row * K + at + i) = v;
        }
    }
    __syncthreads();
}

// NT groups of eight activation rows
// NORM: what runs in front of the product
enum : int { PRO_NONE, PRO_NORM, PRO_STREAMS, PRO_GROUPS };
// BLOCKS: block-diagonal products; a row tile belongs to one block.
template <int NT, int NORM, bool BLOCKS> __global__ void __launch_bounds__(kStreamWarps * 32, 2) linear_stream(const __grid_constant__ LinP p) {
    constexpr int kBatch = NT == 4 ? 2 : 4;  // 32-k chunks a warp has in flight
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float red[kStreamWarps][16][NT * 8 + 1];
    __shared__ float norm_red[kStreamWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int c0 = (int)((p.k[0] + 31) / 32), c1 = (int)((p.k[1] + 31) / 32), chunks = c0 + c1;
    const int block_tiles = (int)((p.out + 15) / 16), tiles = BLOCKS ? block_tiles * p.blocks : block_tiles;
    const int per_tile = (chunks + kStreamWarps * kBatch - 1) / (kStreamWarps * kBatch);  // batches of a warp per row tile
    const int my_tiles = blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = my_tiles * per_tile;

    // chunk `c` of the joint k range → operand and first k of this lane
    auto where = [&](int c, int& op, long long& k) {
        op = c >= c0 ? 1 : 0;
        k = (long long)(op ? c - c0 : c) * 32 + t * 8;
        return c < chunks && k < p.k[op];
    };
    uint4 wl[kBatch], wh[kBatch];
    auto fetch = [&](int it) {
        const int tile = (int)blockIdx.x + (it / per_tile) * (int)gridDim.x;
        const int block = BLOCKS ? tile / block_tiles : 0;
        const long long r0 = (long long)(tile - block * block_tiles) * 16 + g, r1 = r0 + 8;
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int c = ((it % per_tile) * kBatch + j) * kStreamWarps + warp;
            int op;
            long long k;
            const bool live = it < total && where(c, op, k);
            const bf16* w = (const bf16*)p.w[live ? op : 0];
            if constexpr (BLOCKS) w += block * p.out * p.k[0];
            wl[j] = wh[j] = make_uint4(0, 0, 0, 0);
            if (live && r0 < p.out) wl[j] = ld_weights(w + r0 * p.k[op] + k);
            if (live && r1 < p.out) wh[j] = ld_weights(w + r1 * p.k[op] + k);
        }
    };
    pdl_trigger();
    fetch(0);
    pdl_wait();
    bf16* xs = reinterpret_cast<bf16*>(smem);
    const int stride = ((int)p.k[0] + 63) / 64 * 64 + 32;  // 64 bytes off a multiple of 128: conflict-free fragment loads
    if constexpr (NORM == PRO_NORM) {
        if (p.ny_bf16) norm_prologue<true>(p, xs, stride, norm_red);
        else norm_prologue<false>(p, xs, stride, norm_red);
    } else if constexpr (NORM == PRO_STREAMS) {
        if (p.ny_bf16) streams_prologue<true>(p, xs, stride, norm_red);
        else streams_prologue<false>(p, xs, stride, norm_red);
    } else if constexpr (NORM == PRO_GROUPS) {
        if (p.ny_bf16) groups_prologue<true>(p, xs, stride);
        else groups_prologue<false>(p, xs, stride);
    }
    float acc[NT][4];
    for (int it = 0; it < total; it++) {
        if (it % per_tile == 0) {
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[n][e] = 0.f;
        }
        uint4 a[kBatch], b[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            a[j] = wl[j];
            b[j] = wh[j];
        }
        uint4 xv[kBatch][NT];
        long long x0 = 0;
        if constexpr (BLOCKS) x0 = p.x_off + ((int)blockIdx.x + (it / per_tile) * (int)gridDim.x) / block_tiles * p.x_step;
#pragma unroll
        for (int j = 0; j < kBatch; j++) {
            const int c = ((it % per_tile) * kBatch + j) * kStreamWarps + warp;
            int op;
            long long k;
            const bool live = where(c, op, k);
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const long long row = n * 8 + g;
                xv[j][n] = make_uint4(0, 0, 0, 0);
                if (live && row < p.rows) {
                    if constexpr (NORM != PRO_NONE) xv[j][n] = *reinterpret_cast<const uint4*>(xs + row * stride + k);
                    else if constexpr (BLOCKS) xv[j][n] = *reinterpret_cast<const uint4*>((const bf16*)p.x[0] + row * p.ldx + x0 + k);
                    else xv[j][n] = *reinterpret_cast<const uint4*>((const bf16*)p.x[op] + row * p.k[op] + k);
                }
            }
        }
        fetch(it + 1);
#pragma unroll
        for (int j = 0; j < kBatch; j++)
#pragma unroll
            for (int n = 0; n < NT; n++) {
                mma_bf16(acc[n], a[j].x, b[j].x, a[j].y, b[j].y, xv[j][n].x, xv[j][n].y);
                mma_bf16(acc[n], a[j].z, b[j].z, a[j].w, b[j].w, xv[j][n].z, xv[j][n].w);
            }
        if (it % per_tile == per_tile - 1) {
#pragma unroll
            for (int n = 0; n < NT; n++) {
                red[warp][g][n * 8 + t * 2] = acc[n][0];
                red[warp][g][n * 8 + t * 2 + 1] = acc[n][1];
                red[warp][g + 8][n * 8 + t * 2] = acc[n][2];
                red[warp][g + 8][n * 8 + t * 2 + 1] = acc[n][3];
            }
            __syncthreads();
            long long tile = (long long)blockIdx.x + (it / per_tile) * (long long)gridDim.x, col0 = 0;  // col0: the block's first column
            if constexpr (BLOCKS) {
                col0 = tile / block_tiles * p.out;
                tile %= block_tiles;
            }
            auto total_of = [&](int r, int m) {
                float s = 0.f;
#pragma unroll
                for (int w = 0; w < kStreamWarps; w++) s += red[w][r][m];
                const long long o = tile * 16 + r;
                return s + (p.bias && o < p.out ? p.bias[col0 + o] : 0.f);
            };
            if constexpr (BLOCKS) {
                for (int i = tid; i < 16 * NT * 8; i += kStreamWarps * 32) {
                    const int r = i & 15, m = i >> 4;
                    const long long o = tile * 16 + r;
                    if (m < p.rows && o < p.out) put(p, m, p.ldy, col0 + o, activate(p, col0 + o, total_of(r, m)) * factor<bf16>(p, m, col0 + o));
                }
            } else if (p.glu) {
                for (int i = tid; i < 8 * NT * 8; i += kStreamWarps * 32) {
                    const int r = i & 7, m = i >> 3;
                    const long long o = tile * 8 + r;
                    if (m < p.rows && o < p.out / 2) put(p, m, p.out / 2, o, glu_value(p, total_of(2 * r, m), total_of(2 * r + 1, m)));
                }
            } else {
                for (int i = tid; i < 16 * NT * 8; i += kStreamWarps * 32) {
                    const int r = i & 15, m = i >> 4;
                    const long long o = tile * 16 + r;
                    if (m < p.rows && o < p.out) put(p, m, p.out, o, activate(p, o, total_of(r, m)));
                }
            }
            __syncthreads();
        }
    }
}

// The same for matrices of more than 19.4 MB (64 KB per CTA, two per SM): a warp's chunks pass through a ring in shared memory by 16-byte
// asynchronous copies, eight of them in flight instead of one batch of four between two waits. Every lane copies, and reads back, only the pieces
// of a chunk that are its own MMA fragments, so nothing but the lane's own copies has to be waited for. The ring is filled ahead of the grid
// dependency (activations behind it) and runs on across row tiles. Up to eight rows that no prologue makes travel with their weights: loaded a
// chunk ahead into registers, they held every chunk up by an L2 read (1 row × 21 504 × 5376 92 µs, now 50). The weights of the first eight chunks
// belong to the group of the first chunk's activations, so the first wait is for all of them; later ones are for a chunk each. 9 to 32 rows
// still come chunk by chunk from L2, which is why long k does not take this kernel (see its rule).
// 1 row: 5376 × 43 008 gated 123 → 77 µs (6.0 TB/s), 5376 × 16 896 56 → 34; 8 rows: 5376 × 32 768 62 (activations in registers: 92), 1152 × 32 768
// 31 → 22. Below that size the products are faster alone, too, but not behind one another: decode steps of small models took 3 % longer with it
// (13.8 against 13.4 ms for 48 steps of the 1b size, activations in registers).
constexpr int kRing = 8;  // 32-k chunks (1 KB) that a warp has in flight
constexpr int flow_slot(bool ring_x) { return ring_x ? 1536 : 1024; }  // bytes, with the chunk's activations (up to eight rows) or without
template <int NT, int NORM> __global__ void __launch_bounds__(kStreamWarps * 32, 2) linear_flow(const __grid_constant__ LinP p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float red[2][kStreamWarps][16][NT * 8 + 1];
    __shared__ float norm_red[kStreamWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int c0 = (int)((p.k[0] + 31) / 32), chunks = c0 + (int)((p.k[1] + 31) / 32);
    const int tiles = (int)((p.out + 15) / 16), per_tile = (chunks + kStreamWarps - 1) / kStreamWarps;  // chunks of a warp per row tile
    const int my_tiles = (int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    // the chunk that is asked for next: its number in the tile, and the row tile
    constexpr bool kRingX = NT == 1 && NORM == PRO_NONE;
    constexpr int kSlot = flow_slot(kRingX);
    unsigned char* slots = smem + warp * kRing * kSlot + lane * 16;
    const unsigned ring = smem_u32(slots);
    int f_at = warp, f_tile = (int)blockIdx.x, f_slot = 0, f_left = my_tiles * per_tile;
    auto fetch = [&](bool weights, bool acts) {
        if (f_left-- > 0) {
            const long long r0 = (long long)f_tile * 16 + g;
            const int op = f_at >= c0;
            const long long k = (long long)(op ? f_at - c0 : f_at) * 32 + t * 8, K = p.k[op];
            const bf16* w = (const bf16*)p.w[op] + r0 * K + k;
            const bool live = f_at < chunks && k < K;
            const unsigned to = ring + (unsigned)f_slot * kSlot;
            if (weights) {
                cp_async16(to, live && r0 < p.out ? w : (const bf16*)p.w[0], live && r0 < p.out);
                cp_async16(to + 512, live && r0 + 8 < p.out ? w + 8 * K : (const bf16*)p.w[0], live && r0 + 8 < p.out);
            }
            if (acts) {
                const bool met = live && g < p.rows;
                cp_async16(to + 1024, (const bf16*)p.x[met ? op : 0] + (met ? g * K + k : 0), met);
            }
            f_slot = f_slot + 1 == kRing ? 0 : f_slot + 1;
            f_at += kStreamWarps;
            if (f_at >= per_tile * kStreamWarps) {
                f_at = warp;
                f_tile += (int)gridDim.x;
            }
        }
        if (acts || !kRingX) cp_async_commit();
    };
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < kRing; i++) fetch(true, false);  // constants: ahead of the launches in front of this one
    pdl_wait();
    if constexpr (kRingX) {
        f_at = warp, f_tile = (int)blockIdx.x, f_slot = 0, f_left = my_tiles * per_tile;
#pragma unroll
        for (int i = 0; i < kRing; i++) fetch(false, true);
    }
    bf16* xs = reinterpret_cast<bf16*>(smem + kStreamWarps * kRing * kSlot);
    const int stride = ((int)p.k[0] + 63) / 64 * 64 + 32;  // 64 bytes off a multiple of 128: conflict-free fragment loads
    if constexpr (NORM == PRO_NORM) {
        if (p.ny_bf16) norm_prologue<true>(p, xs, stride, norm_red);
        else norm_prologue<false>(p, xs, stride, norm_red);
    } else if constexpr (NORM == PRO_STREAMS) {
        if (p.ny_bf16) streams_prologue<true>(p, xs, stride, norm_red);
        else streams_prologue<false>(p, xs, stride, norm_red);
    } else if constexpr (NORM == PRO_GROUPS) {
        if (p.ny_bf16) groups_prologue<true>(p, xs, stride);
        else groups_prologue<false>(p, xs, stride);
    }
    uint4 xv[NT];  // activations of a chunk, fetched one chunk ahead when they come from memory
    auto load_x = [&](int at) {
        const int op = at >= c0;
        const long long k = (long long)(op ? at - c0 : at) * 32 + t * 8;
        const bool live = at < chunks && k < p.k[op];
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const long long row = n * 8 + g;
            xv[n] = make_uint4(0, 0, 0, 0);
            if (live && row < p.rows) {
                if constexpr (NORM != PRO_NONE) xv[n] = *reinterpret_cast<const uint4*>(xs + row * stride + k);
                else xv[n] = *reinterpret_cast<const uint4*>((const bf16*)p.x[op] + row * p.k[op] + k);
            }
        }
    };
    int slot = 0;
    if (NORM == PRO_NONE && !kRingX && my_tiles > 0) load_x(warp);
    for (int done = 0; done < my_tiles; done++) {
        float acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[n][e] = 0.f;
        for (int i = 0; i < per_tile; i++) {
            cp_async_wait<kRing - 1>();
            const uint4 a = *reinterpret_cast<const uint4*>(slots + slot * kSlot), b = *reinterpret_cast<const uint4*>(slots + slot * kSlot + 512);
            if (kRingX) xv[0] = *reinterpret_cast<const uint4*>(slots + slot * kSlot + 1024);
            slot = slot + 1 == kRing ? 0 : slot + 1;
            if (NORM != PRO_NONE) load_x(i * kStreamWarps + warp);
            uint4 x[NT];
#pragma unroll
            for (int n = 0; n < NT; n++) x[n] = xv[n];
            if (NORM == PRO_NONE && !kRingX) {
                if (i + 1 < per_tile) load_x((i + 1) * kStreamWarps + warp);
                else if (done + 1 < my_tiles) load_x(warp);
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                mma_bf16(acc[n], a.x, b.x, a.y, b.y, x[n].x, x[n].y);
                mma_bf16(acc[n], a.z, b.z, a.w, b.w, x[n].z, x[n].w);
            }
            fetch(true, kRingX);  // into the slot that has just been read
        }
        const int half = done & 1;  // the other half is written before the next tile's meeting, which everybody comes to behind this tile's sums
#pragma unroll
        for (int n = 0; n < NT; n++) {
            red[half][warp][g][n * 8 + t * 2] = acc[n][0];
            red[half][warp][g][n * 8 + t * 2 + 1] = acc[n][1];
            red[half][warp][g + 8][n * 8 + t * 2] = acc[n][2];
            red[half][warp][g + 8][n * 8 + t * 2 + 1] = acc[n][3];
        }
        __syncthreads();
        const long long tile = (long long)blockIdx.x + done * (long long)gridDim.x;
        auto total_of = [&](int r, int m) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < kStreamWarps; w++) s += red[half][w][r][m];
            const long long o = tile * 16 + r;
            return s + (p.bias && o < p.out ? p.bias[o] : 0.f);
        };
        if (p.glu) {
            for (int i = tid; i < 8 * NT * 8; i += kThreads) {
                const int r = i & 7, m = i >> 3;
                const long long o = tile * 8 + r;
                if (m < p.rows && o < p.out / 2) put(p, m, p.out / 2, o, glu_value(p, total_of(2 * r, m), total_of(2 * r + 1, m)));
            }
        } else {
            for (int i = tid; i < 16 * NT * 8; i += kThreads) {
                const int r = i & 15, m = i >> 4;
                const long long o = tile * 16 + r;
                if (m < p.rows && o < p.out) put(p, m, p.out, o, activate(p, o, total_of(r, m)));
            }
        }
    }
}

// ───────────────────────────── tcgen05 GEMM ─────────────────────────────
constexpr int kTcThreads = 192;      // warps 0-3 epilogue, 4 TMA, 5 MMA
constexpr int kTcPanelA = 128 * 128; // bytes: 128 weight rows × 64 k

// A persistent CTA works through tiles (piece of k slowest, activation tiles fastest: they share a weight tile while it is in L2); loads and
// MMAs run on into the next tile while the epilogue of the last one empties the other of two accumulators. ONE: as many CTAs as tiles and pieces, which the
// grid's axes count; the loop's code is not there. 64 rows × 2560 × 5120 cut along k: 14.1 → 13.2 µs against the kernel that had no loop. Most products with more tiles than
// that belong to pairs of CTAs (linear_pair.cu); here remain those of few rows, of groups of few rows, and block-diagonal ones.
//
// The warps that copy and that issue products do their steps in few dependent instructions: stage and parity are carried along, descriptors advance by addition, the next
// stage's barrier is asked before this stage's products are issued. With the step counter divided and reduced by the number of stages (five runtime divisions a step) a
// step could not take less than 0.36 µs whatever its size: 400 × 5376 × 5376 42.8 → 33.5 µs, 1046 × 2560 × 4160 40.6 → 30.2, 512 × 1152 × 1152 11.8 → 8.5, 64 × 2560 × 4160
// with its reduction 12.5 → 11.3; 2048 × 5376 × 16 896, bound by what comes to an SM, 329 either way.
template <int EPI, bool ONE> __global__ void __launch_bounds__(kTcThreads) linear_tc(const __grid_constant__ LinP p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = p.nb, S = p.stages;
    const int stage_bytes = kTcPanelA + nb * 128;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + (size_t)S * stage_bytes);  // full[S], empty[S], finished[2], read[2]
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * S + 4);
    const unsigned finished = smem_u32(bars + 2 * S), read = finished + 16;
    pdl_trigger();
    int row_tiles = p.row_tiles, group = 0, group_row = 0, group_live = 0;
    if (p.groups) {  // the counts come from an earlier launch
        pdl_wait();
        if (!ONE) row_tiles = count_tiles(p, nb);
        else if (!locate_group(p, (int)blockIdx.x, nb, &group, &group_row, &group_live)) return;  // the grid covers the most tiles that any counts give
    }
    const int first = ONE ? 0 : (int)blockIdx.x, total = ONE ? 1 : row_tiles * p.out_tiles * p.splits;
    if (tid == 0) {
        for (int s = 0; s < 2 * S + 2; s++) mbar_init(smem_u32(bars + s), 1);
        for (int s = 0; s < 2; s++) mbar_init(read + s * 8, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    int cols = 32;
    while (cols < (ONE ? nb : 2 * nb)) cols <<= 1;
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;

    const int s0 = (int)((p.k[0] + 63) / 64), all = s0 + (int)((p.k[1] + 63) / 64);
    const int block_tiles = (int)((p.out + 127) / 128);
    struct Tile {
        int group = 0, n0, live, block, m0, piece, lo, steps;
    };
    auto tile_of = [&](int t) {  // by whole warps
        Tile q;
        int x = (int)blockIdx.x, y = (int)blockIdx.y;
        q.piece = (int)blockIdx.z;
        if (!ONE) {
            const int rest = t / row_tiles;
            x = t % row_tiles;
            y = rest % p.out_tiles;
            q.piece = rest / p.out_tiles;
        }
        q.n0 = x * nb;
        q.live = (int)min((long long)nb, p.rows - q.n0);
        if (p.groups) {
            if (!ONE) {
                locate_group(p, x, nb, &q.group, &q.n0, &q.live);
            } else {
                q.group = group;
                q.n0 = group_row;
                q.live = group_live;
            }
        }
        q.block = p.blocks > 1 ? y / block_tiles : 0;
        q.m0 = (y - q.block * block_tiles) * 128;
        q.lo = (int)((unsigned)(all * q.piece) / (unsigned)p.splits);
        q.steps = (int)((unsigned)(all * (q.piece + 1)) / (unsigned)p.splits) - q.lo;
        return q;
    };
    bool ok = true;

    if (warp == 4) {
        // Stage and parity are carried along: the divisions of a step counter took longer than the copies of the step.
        RingAt at;
        bool round = false;  // the ring's first round waits for nothing
        bool waited = p.groups != 0;
        const unsigned full = smem_u32(bars), empty = full + S * 8, data = smem_u32(smem);
        for (int t = first; t < total; t += (int)gridDim.x) {
            const Tile q = tile_of(t);
            const int w0 = (q.group + q.block) * (int)p.out + q.m0, x0 = (int)(p.x_off + q.block * p.x_step);
            auto load_w = [&](unsigned s, int i) {
                const int c = q.lo + i, op = c >= s0;
                mbar_expect_tx(full + s * 8, (unsigned)stage_bytes);
                tma_load_2d(data + s * stage_bytes, p.maps[op * 2 + 1], (op ? c - s0 : c) * 64, w0, full + s * 8);
            };
            auto load_x = [&](unsigned s, int i) {
                const int c = q.lo + i, op = c >= s0;
                tma_load_2d(data + s * stage_bytes + kTcPanelA, p.maps[op * 2], (op ? c - s0 : c) * 64 + x0, q.n0, full + s * 8);
            };
            int i = 0;
            if (!waited) {
                const int head = min(S, q.steps);
                if (elect_one())
                    for (int h = 0; h < head; h++) load_w(h, h);  // constants: may overlap the launches before this one
                __syncwarp();
                pdl_wait();
                for (; i < head; i++) {
                    if (elect_one()) load_x(i, i);
                    __syncwarp();
                    at.next(S);
                }
                round = head == S;
                waited = true;
            }
            for (; i < q.steps; i++) {
                if (!__all_sync(0xffffffffu, !round || mbar_wait(empty + at.s * 8, at.parity ^ 1))) {
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    load_w(at.s, i);
                    load_x(at.s, i);
                }
                __syncwarp();
                at.next(S);
                if (at.s == 0) round = true;
            }
            if (!__all_sync(0xffffffffu, ok)) break;
        }
        // every copy has landed before this CTA's shared memory can be given away
        for (unsigned n = 0; n < (round ? (unsigned)S : at.s); n++)
            if (!mbar_wait(full + n * 8, n < at.s ? at.parity : at.parity ^ 1)) ok = false;
    } else if (warp == 5) {
        pdl_wait();
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(nb >> 3) << 17) | (8u << 24);  // bf16 × bf16 → f32, M 128 × N nb
        RingAt at;
        bool ready = false;
        int j = 0;
        const unsigned full = smem_u32(bars), empty = full + S * 8, step16 = (unsigned)stage_bytes >> 4;
        const unsigned long long a0 = umma_kmajor_desc(smem_u32(smem)), b0 = umma_kmajor_desc(smem_u32(smem) + kTcPanelA);
        for (int t = first; t < total; t += (int)gridDim.x, j++) {
            const int piece = ONE ? (int)blockIdx.z : t / row_tiles / p.out_tiles, steps = (int)((unsigned)(all * (piece + 1)) / (unsigned)p.splits) - (int)((unsigned)(all * piece) / (unsigned)p.splits);
            const unsigned d = tmem + (unsigned)((j & 1) * nb);
            if (!ONE && j >= 2 && ok && !mbar_wait(read + (j & 1) * 8, ((j >> 1) - 1) & 1)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int i = 0; i < steps; i++) {
                if (ok && !ready && !mbar_wait(full + at.s * 8, at.parity)) ok = false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned long long a = a0 + at.s * step16, b = b0 + at.s * step16;  // descriptors count in 16 bytes
                const unsigned done = empty + at.s * 8;
                at.next(S);
                ready = mbar_test(full + at.s * 8, at.parity);  // the answer is there when the products have been issued
                if (elect_one() && ok) {
#pragma unroll
                    for (int e = 0; e < 4; e++) umma_bf16(d, a + e * 2, b + e * 2, idesc, i > 0 || e > 0);
                    umma_commit(done);
                }
                __syncwarp();
            }
            if (elect_one()) umma_commit(finished + (j & 1) * 8);
            __syncwarp();
        }
    } else {
        pdl_wait();
        int j = 0;
        for (int t = first; t < total; t += (int)gridDim.x, j++) {
            const Tile q = tile_of(t);
            if (ok && !mbar_wait(finished + (j & 1) * 8, (j >> 1) & 1)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const long long o = (long long)q.m0 + warp * 32 + lane;  // weight row = accumulator lane
            const long long n0 = q.n0, col0 = q.block * p.out;
            const float bias = p.bias && p.splits == 1 && o < p.out ? p.bias[col0 + o] : 0.f;
            const int live = q.live;
            const int f = EPI == EPI_ACT && col0 + o < p.act_end ? p.act[col0 + o >= p.act_split] : ACT_NONE;
            const unsigned d = tmem + (unsigned)((j & 1) * nb) + ((unsigned)(warp * 32) << 16);
            for (int c = 0; c < nb && c < live; c += 16) {
                unsigned v[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                      "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                    : "r"(d + (unsigned)c));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (p.splits > 1) {
                    float* part = p.partial + ((size_t)q.piece * p.rows + n0 + c) * p.ldy + col0 + o;
#pragma unroll
                    for (int e = 0; e < 16; e++)
                        if (ok && o < p.out && c + e < live) part[(size_t)e * p.ldy] = __uint_as_float(v[e]);
                } else if constexpr (EPI == EPI_GLU) {
                    // lanes 2i and 2i + 1 hold gate and up; of two activation rows the even lane finishes the first, the odd one
                    // the second
                    const int odd = lane & 1;
                    const long long width = p.out / 2, at = (n0 + c + odd) * width + (o >> 1);
                    const bool mine = ok && (o | 1) < p.out;
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        const float lo = __uint_as_float(v[e]) + bias, hi = __uint_as_float(v[e + 1]) + bias;
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
                        const float y = glu_value(p, odd ? got : lo, odd ? hi : got);
                        if (!mine || c + e + odd >= live) continue;
                        if (p.y_bf16) ((bf16*)p.y)[at + e * width] = __float2bfloat16_rn(y);
                        else ((float*)p.y)[at + e * width] = y;
                    }
                } else if (ok && o < p.out) {
                    float y[16];
#pragma unroll
                    for (int e = 0; e < 16; e++) y[e] = __uint_as_float(v[e]) + bias;
                    if constexpr (EPI == EPI_ACT) {
                        if (f == ACT_SOFTPLUS) {
#pragma unroll
                            for (int e = 0; e < 16; e++) y[e] = softplus_fast(y[e]);
                        } else if (f != ACT_NONE && p.y_bf16) {
#pragma unroll
                            for (int e = 0; e < 16; e++) y[e] = sigmoid_fast(y[e]) * (f == ACT_SILU ? y[e] : 1.f);
                        } else if (f != ACT_NONE) {
#pragma unroll
                            for (int e = 0; e < 16; e++) y[e] = sigmoid_f(y[e]) * (f == ACT_SILU ? y[e] : 1.f);
                        }
                        if (p.mul)
#pragma unroll
                            for (int e = 0; e < 16; e++)
                                if (c + e < live) y[e] *= factor<bf16>(p, n0 + c + e, col0 + o);
                    }
                    const long long at = (n0 + c) * p.ldy + col0 + o;
                    if (p.y_bf16) {
                        bf16* to = (bf16*)p.y + at;
#pragma unroll
                        for (int e = 0; e < 16; e++)
                            if (c + e < live) to[e * p.ldy] = __float2bfloat16_rn(y[e]);
                    } else {
                        float* to = (float*)p.y + at;
#pragma unroll
                        for (int e = 0; e < 16; e++)
                            if (c + e < live) to[e * p.ldy] = y[e];
                    }
                }
                __syncwarp();
            }
            if (ONE) break;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(read + (j & 1) * 8) : "memory");
        }
    }
    if (!ok && lane == 0) report(p.err, ERR_WAIT_TIMEOUT, p.node, (long long)blockIdx.x, (long long)warp);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

// Adds the pieces of a product that was cut along k, in piece order, with bias and gating. blockIdx.y is the activation
// row; V consecutive weight rows per thread (V = 4: out is a multiple of 4).
template <int V, typename T = bf16> __global__ void __launch_bounds__(256) linear_reduce(const __grid_constant__ LinP p) {
    pdl_enter();
    const long long row = blockIdx.y, o = ((long long)blockIdx.x * 256 + threadIdx.x) * V;
    if (o >= p.out) return;
    const size_t piece = (size_t)p.rows * p.out;
    const float* src = p.partial + row * p.out + o;
    float s[V];
#pragma unroll
    for (int e = 0; e < V; e++) s[e] = 0.f;
#pragma unroll 4
    for (int z = 0; z < p.splits; z++) {
        if constexpr (V == 4) {
            const float4 f = *reinterpret_cast<const float4*>(src + z * piece);
            s[0] += f.x;
            s[1] += f.y;
            s[2] += f.z;
            s[3] += f.w;
        } else {
#pragma unroll
            for (int e = 0; e < V; e++) s[e] += src[z * piece + e];
        }
    }
    if (p.bias)
#pragma unroll
        for (int e = 0; e < V; e++) s[e] += p.bias[o + e];
    if (!p.glu)
#pragma unroll
        for (int e = 0; e < V; e++) s[e] = activate(p, o + e, s[e]) * factor<T>(p, row, o + e);
    if (p.glu) {  // out is even, and so are o and V
#pragma unroll
        for (int e = 0; e < V; e += 2) put(p, row, p.out / 2, (o + e) / 2, glu_value(p, s[e], s[e + 1]));
    } else if (V == 4 && !p.y_bf16) {
        *reinterpret_cast<float4*>((float*)p.y + row * p.out + o) = make_float4(s[0], s[1 % V], s[2 % V], s[3 % V]);
    } else {
#pragma unroll
        for (int e = 0; e < V; e++)
            if (o + e < p.out) put(p, row, p.out, o + e, s[e]);
    }
}

// ───────────────────────────── 32-bit ───────────────────────────────────
__device__ __forceinline__ float4 ld4_f32(const float* p, bool wide) {
    return wide ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ float4 ld4_stream(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// Up to eight activation rows per blockIdx.y (M of them formed): bound by the weights' bytes. A warp owns R weight rows and takes 128
// consecutive k of each (512 bytes) per step, the next step's weights ahead of this step's sums; `nb` warps of a CTA share the same
// rows and take the steps in turn where there are few rows. Lanes keep sums of their own (chains 32 times shorter than one thread's),
// which fold over lanes at the end: value m · R + r ends up in lane m · R + r. Activations come through L1.
// 3 rows, k 1152, 13 824 weight rows (64 MB): 25 µs, 2.6 TB/s; k 6912, 1152 weight rows: 12 µs. One 64 × 64 tile per CTA (linear_simt), a
// grid of out / 64 CTAs that each walk all of k: 250 and 1175 µs.
template <int M, int R> __global__ void __launch_bounds__(kThreads, 2) linear_rows_f32(const __grid_constant__ LinP p) {
    constexpr int N = M * R;
    __shared__ float red[kStreamWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, share = p.nb, slice = warp % share;
    const int block_units = (int)((p.out + R - 1) / R);
    const long long unit = (long long)blockIdx.x * (kStreamWarps / share) + warp / share;
    const int block = p.blocks > 1 ? (int)(unit / block_units) : 0;
    const bool live = unit < (long long)block_units * p.blocks;
    const long long o0 = (unit - (long long)block * block_units) * R, w_at = block * p.out, x0 = p.x_off + block * p.x_step, row0 = (long long)blockIdx.y * 8;
    const int rows = (int)min((long long)M, p.rows - row0);
    const int c0 = (int)((p.k[0] + 127) / 128), chunks = live ? c0 + (int)((p.k[1] + 127) / 128) : 0;
    const bool wide = ((reinterpret_cast<uintptr_t>(p.x[0]) | reinterpret_cast<uintptr_t>(p.x[1])) & 15) == 0;
    float4 w[R];
    auto fetch = [&](int c) {
        const int op = c >= c0;
        const long long k = (long long)(op ? c - c0 : c) * 128 + lane * 4;
        const float* from = (const float*)p.w[op] + (w_at + o0) * p.k[op] + k;
#pragma unroll
        for (int r = 0; r < R; r++) w[r] = c < chunks && k < p.k[op] && o0 + r < p.out ? ld4_stream(from + r * p.k[op]) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    pdl_trigger();
    fetch(slice);  // constants: before the launches in front of this one are done
    pdl_wait();
    float acc[N];
#pragma unroll
    for (int i = 0; i < N; i++) acc[i] = 0.f;
    for (int c = slice; c < chunks; c += share) {
        const int op = c >= c0;
        const long long k = (long long)(op ? c - c0 : c) * 128 + lane * 4, ldx = p.ldx ? p.ldx : p.k[op];
        const float* from = (const float*)p.x[op] + row0 * ldx + x0 + k;
        float4 x[M], now[R];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = m < rows && k < p.k[op] ? ld4_f32(from + m * ldx, wide) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < R; r++) now[r] = w[r];
        fetch(c + share);
#pragma unroll
        for (int m = 0; m < M; m++)
#pragma unroll
            for (int r = 0; r < R; r++) {
                float& a = acc[m * R + r];
                a = fmaf(x[m].x, now[r].x, a);
                a = fmaf(x[m].y, now[r].y, a);
                a = fmaf(x[m].z, now[r].z, a);
                a = fmaf(x[m].w, now[r].w, a);
            }
    }
    // every step sends half of the values to the lanes that keep them; what is left of 32 / N lanes per value is added up
#pragma unroll
    for (int half = N / 2, o = N / 2; half >= 1; half /= 2, o /= 2)
#pragma unroll
        for (int i = 0; i < half; i++) {
            const bool up = lane & o;
            const float give = up ? acc[i] : acc[i + half], keep = up ? acc[i + half] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    float sum = acc[0];
#pragma unroll
    for (int o = 16; o >= N; o /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (share > 1) {
        red[warp][lane] = sum;
        __syncthreads();
        if (slice) return;
        sum = 0.f;
        for (int i = 0; i < share; i++) sum += red[warp + i][lane];
    }
    const int m = lane / R, r = lane % R;
    const long long o = o0 + r, row = row0 + m;
    const bool mine = live && lane < N && m < rows && o < p.out;
    if (p.bias && mine) sum += p.bias[w_at + o];
    if (p.glu) {
        const float up = __shfl_down_sync(0xffffffffu, sum, 1);
        if (mine && !(r & 1) && o + 1 < p.out) put(p, row, p.out / 2, o >> 1, glu_value(p, sum, up));
    } else if (mine) {
        put(p, row, p.ldy, w_at + o, activate(p, w_at + o, sum) * factor<float>(p, row, w_at + o));
    }
}

// More rows: 64 weight rows × 64 activation rows per CTA, 8 × 4 of them per thread, 16 k per step, the next step's operands in registers
// while this one's are multiplied; bound by the FMA pipe (12 shared-memory words per 32 FMAs). Small grids are cut along k (blockIdx.z),
// `linear_reduce` adds the pieces in order. k, ldx and x_off are multiples of 4. 303 rows: 31 – 33 TFLOP/s, 313 and 146 µs for the two sizes
// above (linear_simt, one scalar shared-memory read per two FMAs and no cut along k: 569 and 1046 µs).
constexpr int kF32Threads = 128;
// Its epilogue of 32 values per thread stands against few steps where k is short. linear_simt → linear_f32, µs: 40 rows × 64 weight rows, k 16: 7 → 15, k 64:
// 12 → 18, k 128: 19 → 21, k 192 (64 rows): 26 → 24, k 256: 32 → 27; 1000 × 4096, k 64: 40 → 46, k 192: 91 → 82.
static bool f32_pays(long long k) { return k >= 192; }
__global__ void __launch_bounds__(kF32Threads) linear_f32(const __grid_constant__ LinP p) {
    __shared__ __align__(16) float ws[2][16][68], xs[2][16][68];
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const int block_tiles = (int)((p.out + 63) / 64), block = p.blocks > 1 ? (int)blockIdx.x / block_tiles : 0;
    const long long m0 = (long long)((int)blockIdx.x - block * block_tiles) * 64, x0 = p.x_off + block * p.x_step, col0 = block * p.out;
    long long n0 = (long long)blockIdx.y * 64, rows = p.rows, w_at = col0;  // w_at: first row of the group's or block's weights
    pdl_enter();
    if (p.groups) {
        int group, row, live;
        if (!locate_group(p, (int)blockIdx.y, 64, &group, &row, &live)) return;
        n0 = row;
        rows = row + live;
        w_at = group * p.out;
    }
    const bool wide = ((reinterpret_cast<uintptr_t>(p.x[0]) | reinterpret_cast<uintptr_t>(p.x[1])) & 15) == 0;
    const int s0 = (int)((p.k[0] + 15) / 16), all = s0 + (int)((p.k[1] + 15) / 16);
    const int lo = (int)((long long)all * blockIdx.z / p.splits), hi = (int)((long long)all * (blockIdx.z + 1) / p.splits);
    const int lr = tid >> 2, lk = (tid & 3) * 4;  // this thread loads rows lr and lr + 32, four k
    float4 wv[2], xv[2];
    auto fetch = [&](int s) {
        const int op = s >= s0;
        const long long k = (long long)(op ? s - s0 : s) * 16 + lk, ldx = p.ldx ? p.ldx : p.k[op];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int r = lr + j * 32;
            const bool kl = s < hi && k < p.k[op];
            wv[j] = kl && m0 + r < p.out ? *reinterpret_cast<const float4*>((const float*)p.w[op] + (w_at + m0 + r) * p.k[op] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            xv[j] = kl && n0 + r < rows ? ld4_f32((const float*)p.x[op] + (n0 + r) * ldx + x0 + k, wide) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto keep = [&](int b) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int r = lr + j * 32;
            ws[b][lk][r] = wv[j].x;
            ws[b][lk + 1][r] = wv[j].y;
            ws[b][lk + 2][r] = wv[j].z;
            ws[b][lk + 3][r] = wv[j].w;
            xs[b][lk][r] = xv[j].x;
            xs[b][lk + 1][r] = xv[j].y;
            xs[b][lk + 2][r] = xv[j].z;
            xs[b][lk + 3][r] = xv[j].w;
        }
    };
    float acc[4][8] = {};  // [row][weight row: 4 tx …, 32 + 4 tx …]
    fetch(lo);
    keep(0);
    __syncthreads();
    for (int s = lo; s < hi; s++) {
        const int b = (s - lo) & 1;
        fetch(s + 1);
#pragma unroll
        for (int kk = 0; kk < 16; kk++) {
            const float4 a = *reinterpret_cast<const float4*>(&xs[b][kk][ty * 4]), u = *reinterpret_cast<const float4*>(&ws[b][kk][tx * 4]),
                         v = *reinterpret_cast<const float4*>(&ws[b][kk][32 + tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        keep(b ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const long long row = n0 + ty * 4 + i;
        if (row >= rows) continue;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const long long o = m0 + (j >> 2) * 32 + tx * 4 + (j & 3);
            if (o >= p.out) continue;
            if (p.splits > 1) {
                p.partial[((size_t)blockIdx.z * p.rows + row) * p.ldy + col0 + o] = acc[i][j];
                continue;
            }
            const float v = acc[i][j] + (p.bias ? p.bias[col0 + o] : 0.f);
            if (p.glu) {
                if (!(j & 1) && o + 1 < p.out) put(p, row, p.out / 2, o >> 1, glu_value(p, v, acc[i][(j + 1) & 7] + (p.bias ? p.bias[col0 + o + 1] : 0.f)));
            } else {
                put(p, row, p.ldy, col0 + o, activate(p, col0 + o, v) * factor<float>(p, row, col0 + o));
            }
        }
    }
}

// ───────────────────────────── any shape ────────────────────────────────
template <typename T> __global__ void __launch_bounds__(256) linear_simt(const __grid_constant__ LinP p) {
    __shared__ float xs[16][65], ws[16][65];
    pdl_enter();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int block_tiles = (int)((p.out + 63) / 64), block = p.blocks > 1 ? (int)blockIdx.x / block_tiles : 0;
    const long long m0 = (long long)((int)blockIdx.x - block * block_tiles) * 64, x0 = p.x_off + block * p.x_step, col0 = block * p.out;
    long long n0 = (long long)blockIdx.y * 64, rows = p.rows, w_at = col0;  // w_at: first row of the group's or block's weights
    if (p.groups) {
        int group, row, live;
        if (!locate_group(p, (int)blockIdx.y, 64, &group, &row, &live)) return;
        n0 = row;
        rows = row + live;
        w_at = group * p.out;
    }
    float acc[4][4] = {};  // [row][weight row]
    for (int op = 0; op < 2; op++) {
        const T *x = (const T*)p.x[op], *w = (const T*)p.w[op];
        const long long ldx = p.ldx ? p.ldx : p.k[op];
        for (long long k0 = 0; k0 < p.k[op]; k0 += 16) {
            for (int i = tid; i < 1024; i += 256) {
                const int kk = i & 15, r = i >> 4;
                const bool kl = k0 + kk < p.k[op];
                xs[kk][r] = kl && n0 + r < rows ? to_f(x[(n0 + r) * ldx + x0 + k0 + kk]) : 0.f;
                ws[kk][r] = kl && m0 + r < p.out ? to_f(w[(w_at + m0 + r) * p.k[op] + k0 + kk]) : 0.f;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < 16; kk++) {
                float a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    a[i] = xs[kk][ty * 4 + i];
                    b[i] = ws[kk][tx * 4 + i];
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const long long row = n0 + ty * 4 + i;
        if (row >= rows) continue;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const long long o = m0 + tx * 4 + j;
            v[j] = acc[i][j] + (p.bias && o < p.out ? p.bias[col0 + o] : 0.f);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const long long o = m0 + tx * 4 + j;
            if (p.glu) {
                if (!(j & 1) && o + 1 < p.out) put(p, row, p.out / 2, o >> 1, glu_value(p, v[j], v[j + 1]));
            } else if (o < p.out) {
                put(p, row, p.ldy, col0 + o, activate(p, col0 + o, v[j]) * factor<T>(p, row, col0 + o));
            }
        }
    }
}

// ───────────────────────────── residual norm ────────────────────────────
struct ResNormP {
    const void* y;
    const float *w, *gain, *res, *post, *offset;
    const void *gate, *add;
    float* stream;
    void* low;
    int* zero;
    long long rows, width, y_ld, gate_ld;
    float eps, y_scale, add_scale;
    int y_bf16, low_bf16, gate_bf16, add_bf16, pre, n_zero, groups;
};
// One CTA per row; V consecutive elements per load.
template <int V> struct Pack {
    float v[V];
};
template <int V> __device__ __forceinline__ Pack<V> ld_pack(const void* p, long long i, bool is_bf16) {
    Pack<V> o;
    if constexpr (V == 4) {
        const float4 f = is_bf16 ? ld_y4<true>(p, i) : ld_y4<false>(p, i);
        o.v[0] = f.x;
        o.v[1] = f.y;
        o.v[2] = f.z;
        o.v[3] = f.w;
    } else {
        o.v[0] = is_bf16 ? __bfloat162float(((const bf16*)p)[i]) : ((const float*)p)[i];
    }
    return o;
}
template <int V> __device__ __forceinline__ void st_pack(void* p, long long i, const Pack<V>& v, bool is_bf16) {
    if constexpr (V == 4) {
        if (is_bf16) *reinterpret_cast<uint2*>((bf16*)p + i) = make_uint2(pack_bf16(v.v[0], v.v[1]), pack_bf16(v.v[2], v.v[3]));
        else *reinterpret_cast<float4*>((float*)p + i) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
    } else {
        if (is_bf16) ((bf16*)p)[i] = __float2bfloat16_rn(v.v[0]);
        else ((float*)p)[i] = v.v[0];
    }
}
template <int V> __global__ void __launch_bounds__(256) residual_norm(const ResNormP p) {
    __shared__ float red[32];
    pdl_enter();
    const long long row = blockIdx.x, base = row * p.width;
    if (row == 0)
        for (int i = threadIdx.x; i < p.n_zero; i += 256) p.zero[i] = 0;
    const long long y0 = row * p.y_ld;
    auto rstd_of = [&](auto&& value) {
        float ss = 0.f;
#pragma unroll 4
        for (long long i = threadIdx.x * V; i < p.width; i += 256 * V) {
            const Pack<V> y = value(i);
#pragma unroll
            for (int e = 0; e < V; e++) ss = fmaf(y.v[e], y.v[e], ss);
        }
        return 1.f / sqrtf(block_sum(ss, red) / (float)p.width + p.eps);
    };
    const float inner = p.post ? rstd_of([&](long long i) { return ld_pack<V>(p.y, y0 + i, p.y_bf16); }) : p.y_scale;
    auto normed = [&](long long i) {  // what the mean square is taken of
        Pack<V> y = ld_pack<V>(p.y, y0 + i, p.y_bf16);
        auto plus = [&](const void* from, long long at, bool is_bf16, float scale) {
            const Pack<V> r = ld_pack<V>(from, at, is_bf16);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] = fmaf(r.v[e], scale, y.v[e]);
        };
        if (p.pre) {
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] *= inner;
            if (p.post) {
                const Pack<V> w = ld_pack<V>(p.post, i, false);
#pragma unroll
                for (int e = 0; e < V; e++) y.v[e] *= w.v[e];
            }
            if (p.res) plus(p.res, base + i, false, 1.f);
            if (p.add) plus(p.add, base + i, p.add_bf16, p.add_scale);
            if (p.offset) plus(p.offset, i, false, 1.f);
        }
        return y;
    };
    const float rstd = rstd_of(normed);
#pragma unroll 2
    for (long long i = threadIdx.x * V; i < p.width; i += 256 * V) {
        const Pack<V> sum = normed(i), w = ld_pack<V>(p.w, i, false);
        Pack<V> y;
#pragma unroll
        for (int e = 0; e < V; e++) y.v[e] = sum.v[e] * (rstd * w.v[e]);
        if (p.gain) {
            const Pack<V> g = ld_pack<V>(p.gain, i, false);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] *= g.v[e];
        }
        if (p.gate) {
            const Pack<V> g = ld_pack<V>(p.gate, row * p.gate_ld + i, p.gate_bf16);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] *= g.v[e];
        }
        if (!p.pre && p.res) {
            const Pack<V> r = ld_pack<V>(p.res, base + i, false);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] += r.v[e];
        }
        if (p.stream) st_pack<V>(p.stream, base + i, p.pre ? sum : y, false);
        if (p.low) st_pack<V>(p.low, base + i, y, p.low_bf16);
    }
}

// The same for rows of up to 1024 · R elements that are 16-byte aligned: a row is read once and stays in registers between the sums. (The kernel above reads y, the
// residual and what belongs to them again for every sum, each time a chain of loads behind a barrier: 64 × 2560 with two norms 7.6 µs of a step, 4096 × 1152 20.8.) The order of the
// sums is that of block_sum.
template <int R> __global__ void __launch_bounds__(256) residual_row(const ResNormP p) {
    __shared__ float red[2][8];
    pdl_enter();
    const long long row = blockIdx.x, base = row * p.width, y0 = row * p.y_ld;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (row == 0)
        for (int i = tid; i < p.n_zero; i += 256) p.zero[i] = 0;
    Pack<4> y[R], r[R], post[R], w[R];
    auto each = [&](auto&& f) {
#pragma unroll
        for (int k = 0; k < R; k++) {
            const long long i = (tid + k * 256) * 4;
            if (i < p.width) f(k, i);
        }
    };
    each([&](int k, long long i) { y[k] = ld_pack<4>(p.y, y0 + i, p.y_bf16); });
    if (p.res) each([&](int k, long long i) { r[k] = ld_pack<4>(p.res, base + i, false); });
    if (p.post) each([&](int k, long long i) { post[k] = ld_pack<4>(p.post, i, false); });
    each([&](int k, long long i) { w[k] = ld_pack<4>(p.w, i, false); });
    auto rstd_of = [&](int turn) {
        float ss = 0.f;
        each([&](int k, long long) {
#pragma unroll
            for (int e = 0; e < 4; e++) ss = fmaf(y[k].v[e], y[k].v[e], ss);
        });
        ss = warp_sum(ss);
        if (lane == 0) red[turn][warp] = ss;
        __syncthreads();
        const float* t = red[turn];
        return 1.f / sqrtf((((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7]))) / (float)p.width + p.eps);
    };
    const float inner = p.post ? rstd_of(0) : p.y_scale;
    if (p.pre)
        each([&](int k, long long i) {
#pragma unroll
            for (int e = 0; e < 4; e++) y[k].v[e] *= inner;
            if (p.post)
#pragma unroll
                for (int e = 0; e < 4; e++) y[k].v[e] *= post[k].v[e];
            if (p.res)
#pragma unroll
                for (int e = 0; e < 4; e++) y[k].v[e] = fmaf(r[k].v[e], 1.f, y[k].v[e]);
            if (p.add) {
                const Pack<4> a = ld_pack<4>(p.add, base + i, p.add_bf16);
#pragma unroll
                for (int e = 0; e < 4; e++) y[k].v[e] = fmaf(a.v[e], p.add_scale, y[k].v[e]);
            }
            if (p.offset) {
                const Pack<4> a = ld_pack<4>(p.offset, i, false);
#pragma unroll
                for (int e = 0; e < 4; e++) y[k].v[e] = fmaf(a.v[e], 1.f, y[k].v[e]);
            }
        });
    const float rstd = rstd_of(1);
    each([&](int k, long long i) {
        Pack<4> out;
#pragma unroll
        for (int e = 0; e < 4; e++) out.v[e] = y[k].v[e] * (rstd * w[k].v[e]);
        if (p.gain) {
            const Pack<4> g = ld_pack<4>(p.gain, i, false);
#pragma unroll
            for (int e = 0; e < 4; e++) out.v[e] *= g.v[e];
        }
        if (p.gate) {
            const Pack<4> g = ld_pack<4>(p.gate, row * p.gate_ld + i, p.gate_bf16);
#pragma unroll
            for (int e = 0; e < 4; e++) out.v[e] *= g.v[e];
        }
        if (!p.pre && p.res)
#pragma unroll
            for (int e = 0; e < 4; e++) out.v[e] += r[k].v[e];
        if (p.stream) st_pack<4>(p.stream, base + i, p.pre ? y[k] : out, false);
        if (p.low) st_pack<4>(p.low, base + i, out, p.low_bf16);
    });
}

// A residual of several streams: one CTA per row, the norm's operand in shared memory in between. S: the most streams.
struct StreamsP {
    const void *y, *y2;
    const float *w, *res, *post, *post2, *connect;
    float* stream;
    void* low;
    int* zero;
    long long width, y_ld;
    float eps, y_scale;
    int y_bf16, low_bf16, streams, n_zero;
};
template <int V, int S> __global__ void __launch_bounds__(256) streams_norm(const StreamsP p) {
    extern __shared__ __align__(16) float operand[];
    __shared__ float red[32], con[S * (S + 2)];
    pdl_trigger();
    const int n = p.streams, tid = threadIdx.x;
    for (int i = tid; i < n * (n + 2); i += 256) con[i] = p.connect[i];  // constants
    pdl_wait();
    const long long row = blockIdx.x, base = row * p.width, y0 = row * p.y_ld;
    if (row == 0)
        for (int i = tid; i < p.n_zero; i += 256) p.zero[i] = 0;
    auto factor_of = [&](const void* y, long long at) {
        float ss = 0.f;
#pragma unroll 4
        for (long long i = tid * V; i < p.width; i += 256 * V) {
            const Pack<V> v = ld_pack<V>(y, at + i, p.y_bf16);
#pragma unroll
            for (int e = 0; e < V; e++) ss = fmaf(v.v[e], v.v[e], ss);
        }
        return 1.f / sqrtf(block_sum(ss, red) / (float)p.width + p.eps);
    };
    const float f1 = p.post ? factor_of(p.y, y0) : p.y_scale, f2 = p.y2 ? factor_of(p.y2, base) : 0.f;
    __syncthreads();
    const float *out = con + n * n, *in = out + n;
    float ss = 0.f;
#pragma unroll 2
    for (long long i = tid * V; i < p.width; i += 256 * V) {
        Pack<V> y = ld_pack<V>(p.y, y0 + i, p.y_bf16), x[S], u;
        if (p.res)
#pragma unroll
            for (int r = 0; r < S; r++)
                if (r < n) x[r] = ld_pack<V>(p.res, base * n + r * p.width + i, false);
#pragma unroll
        for (int e = 0; e < V; e++) y.v[e] *= f1;
        if (p.post) {
            const Pack<V> w = ld_pack<V>(p.post, i, false);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] *= w.v[e];
        }
        if (p.y2) {
            const Pack<V> o = ld_pack<V>(p.y2, base + i, p.y_bf16), w = ld_pack<V>(p.post2, i, false);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] = fmaf(o.v[e] * f2, w.v[e], y.v[e]);
        }
#pragma unroll
        for (int e = 0; e < V; e++) u.v[e] = 0.f;
#pragma unroll
        for (int t = 0; t < S; t++) {
            if (t >= n) break;
            Pack<V> s;
#pragma unroll
            for (int e = 0; e < V; e++) s.v[e] = out[t] * y.v[e];
            if (p.res)
#pragma unroll
                for (int r = 0; r < S; r++)
                    if (r < n)
#pragma unroll
                        for (int e = 0; e < V; e++) s.v[e] = fmaf(con[r * n + t], x[r].v[e], s.v[e]);
#pragma unroll
            for (int e = 0; e < V; e++) u.v[e] = fmaf(in[t], s.v[e], u.v[e]);
            if (p.stream) st_pack<V>(p.stream, base * n + t * p.width + i, s, false);
        }
#pragma unroll
        for (int e = 0; e < V; e++) ss = fmaf(u.v[e], u.v[e], ss);
        st_pack<V>(operand, i, u, false);
    }
    const float rstd = 1.f / sqrtf(block_sum(ss, red) / (float)p.width + p.eps);
    if (!p.low) return;
#pragma unroll 4
    for (long long i = tid * V; i < p.width; i += 256 * V) {
        Pack<V> u = ld_pack<V>(operand, i, false);
        const Pack<V> w = ld_pack<V>(p.w, i, false);
#pragma unroll
        for (int e = 0; e < V; e++) u.v[e] *= rstd * w.v[e];
        st_pack<V>(p.low, base + i, u, p.low_bf16);
    }
}

// A norm of several runs of columns, times a gate: one warp per row and run.
template <int V> __global__ void __launch_bounds__(256) groups_norm(const ResNormP p) {
    pdl_enter();
    const int size = (int)p.width / p.groups, lane = threadIdx.x & 31;
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < p.n_zero; i += 256) p.zero[i] = 0;
    const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= p.rows * p.groups) return;
    const long long row = unit / p.groups, at = unit % p.groups * size, y0 = row * p.y_ld + at;
    float ss = 0.f;
#pragma unroll 4
    for (int i = lane * V; i < size; i += 32 * V) {
        const Pack<V> y = ld_pack<V>(p.y, y0 + i, p.y_bf16);
#pragma unroll
        for (int e = 0; e < V; e++) ss = fmaf(y.v[e], y.v[e], ss);
    }
    const float rstd = 1.f / sqrtf(warp_sum(ss) / (float)size + p.eps);
#pragma unroll 4
    for (int i = lane * V; i < size; i += 32 * V) {
        Pack<V> y = ld_pack<V>(p.y, y0 + i, p.y_bf16);
        const Pack<V> w = ld_pack<V>(p.w, at + i, false);
#pragma unroll
        for (int e = 0; e < V; e++) y.v[e] *= rstd * w.v[e];
        if (p.gate) {
            const Pack<V> g = ld_pack<V>(p.gate, row * p.gate_ld + at + i, p.gate_bf16);
#pragma unroll
            for (int e = 0; e < V; e++) y.v[e] *= g.v[e];
        }
        if (p.stream) st_pack<V>(p.stream, row * p.width + at + i, y, false);
        if (p.low) st_pack<V>(p.low, row * p.width + at + i, y, p.low_bf16);
    }
}

constexpr Buf kNull{kSlotNull, 0};
constexpr int64_t kFusedNormElements = 12288;
Buf buf_of(const TRef* t) { return t ? t->buf : kNull; }

}  // namespace

static void emit_streams_norm(Emitter& em, const ResidualNormDesc& d, const TRef* low, Buf zero, int n_zero) {
    StreamsP p{};
    p.width = d.w->numel();
    p.y_ld = d.y->shape[1];
    p.eps = (float)d.eps;
    p.y_scale = (float)d.y_scale;
    p.y_bf16 = d.y->dtype == DT_BF16;
    p.low_bf16 = low && low->dtype == DT_BF16;
    p.streams = (int)d.streams;
    p.n_zero = n_zero;
    bool wide = p.width % 4 == 0 && p.y_ld % 4 == 0 && d.y_off % 4 == 0;
    for (const TRef* t : {d.y, d.w, d.res, d.post, d.y2, d.post2, d.stream, low}) wide = wide && (!t || t->buf.off % 16 == 0);
    const auto k = wide ? (p.streams <= 2 ? streams_norm<4, 2> : p.streams <= 4 ? streams_norm<4, 4> : p.streams <= 8 ? streams_norm<4, 8> : streams_norm<1, kMaxStreams>)
                        : (p.streams <= 4 ? streams_norm<1, 4> : streams_norm<1, kMaxStreams>);
    const unsigned smem = (unsigned)p.width * 4;
    ensure_max_dynamic_smem((const void*)k, 200 * 1024);
    em.launch(k, dim3((unsigned)d.y->shape[0]), dim3(256), smem, p,
              {{&p.y, d.y->buf.at(d.y_off * (p.y_bf16 ? 2 : 4))}, {&p.y2, buf_of(d.y2)}, {&p.w, d.w->buf}, {&p.res, buf_of(d.res)}, {&p.post, buf_of(d.post)}, {&p.post2, buf_of(d.post2)},
               {&p.connect, d.connect->buf}, {&p.stream, buf_of(d.stream)}, {&p.low, buf_of(low)}, {&p.zero, n_zero ? zero : kNull}},
              "streams_norm", /*pdl=*/true);
}

void emit_residual_norm(Emitter& em, const ResidualNormDesc& d, const TRef* low, Buf zero, int n_zero) {
    ResNormP p{};
    p.width = d.w->numel();
    const long long rows = d.y->shape[0];
    if (rows == 0) return;
    if (d.streams > 0) return emit_streams_norm(em, d, low, zero, n_zero);
    p.rows = rows;
    p.groups = (int)d.groups;
    p.y_ld = d.y->shape[1];
    p.add_scale = (float)d.add_scale;
    p.add_bf16 = d.add && d.add->dtype == DT_BF16;
    p.eps = (float)d.eps;
    p.y_scale = (float)d.y_scale;
    p.pre = d.pre;
    p.y_bf16 = d.y->dtype == DT_BF16;
    p.low_bf16 = low && low->dtype == DT_BF16;
    p.n_zero = n_zero;
    bool wide = p.width % 4 == 0;  // every row is 16-byte aligned when the tensors are
    wide = wide && p.y_ld % 4 == 0 && d.y_off % 4 == 0;
    for (const TRef* t : {d.y, d.w, d.gain, d.res, d.post, d.add, d.offset, d.stream, low}) wide = wide && (!t || t->buf.off % 16 == 0);
    Buf gate = kNull;
    if (d.gate) {
        p.gate_bf16 = d.gate->dtype == DT_BF16;
        p.gate_ld = d.gate->shape[1];
        gate = d.gate->buf.at(d.gate_off * (p.gate_bf16 ? 2 : 4));
        wide = wide && p.gate_ld % 4 == 0 && d.gate_off % 4 == 0 && d.gate->buf.off % 16 == 0;
    }
    wide = wide && (p.width / d.groups) % 4 == 0;
    auto k = d.groups > 1 ? (wide ? groups_norm<4> : groups_norm<1>) : wide ? residual_norm<4> : residual_norm<1>;
    if (d.groups <= 1 && wide && p.width <= 6144) {  // 1024 elements per CTA and pack; more than six packs of four tensors do not fit the registers
        const auto of = [](long long n) -> void (*)(const ResNormP) {
            return n <= 1024 ? residual_row<1> : n <= 2048 ? residual_row<2> : n <= 3072 ? residual_row<3> : n <= 4096 ? residual_row<4> : residual_row<6>;
        };
        k = of(p.width);
    }
    em.launch(k, dim3((unsigned)(d.groups > 1 ? (rows * d.groups + 7) / 8 : rows)), dim3(256), 0, p,
              {{&p.y, d.y->buf.at(d.y_off * (p.y_bf16 ? 2 : 4))}, {&p.post, buf_of(d.post)}, {&p.add, buf_of(d.add)}, {&p.offset, buf_of(d.offset)}, {&p.w, d.w->buf}, {&p.gain, buf_of(d.gain)}, {&p.res, buf_of(d.res)}, {&p.gate, gate}, {&p.stream, buf_of(d.stream)},
               {&p.low, buf_of(low)}, {&p.zero, n_zero ? zero : kNull}},
              "residual_norm", /*pdl=*/true);
}

// Pieces of k that sums are cut into, whatever the kernel and the tile: results of a size have the same bits with all of them. The tensor core adds without rounding to nearest: a chain of
// n products of 64 k is about n · 6.7e-8 off, and pieces are added in f32. They are as many as a step of 0.36 … 0.45 µs makes worth it. By the costs of emit_linear others would often be
// faster, but fewer are further from 64-bit results (303 × 2560 × 2560 in f32: 2.7e-6 off in one chain, 6.0e-7 in five pieces; 512 × 21 504 × 5376 2.5e-5 and 7.9e-6).
static int pieces_of_k(long long rows, long long weight_tiles, long long steps, long long ldy) {
    double best = 1e300;
    int pieces = 1;
    for (int nb : {32, 64, 128, 256}) {
        if (nb > 32 && nb / 2 >= rows) break;
        const long long slots = (long long)sm_count() * (nb <= 128 ? 2 : 1), tiles = weight_tiles * ((rows + nb - 1) / nb);
        const double step = nb == 32 ? 0.36 : nb == 64 ? 0.38 : nb == 128 ? 0.42 : 0.45;
        for (int sp = 1; sp <= (rows < 65536 ? 16 : 1) && sp * 2 <= std::max<long long>(steps, 2); sp++) {
            double us = (double)((tiles * sp + slots - 1) / slots) * ((double)((steps + sp - 1) / sp) * step + (nb == 256 ? 10.0 : 7.0));
            if (sp > 1) us += 3.0 + (double)(sp + 1) * rows * ldy * 4.0 / 3e6;
            if (us < best * (sp > 1 ? 0.97 : 1.0)) {
                best = us;
                pieces = sp;
            }
        }
    }
    return pieces;
}

void emit_linear(Emitter& em, const LinearDesc& d, const TRef* x0, const TRef* x1, const TRef& w0, const TRef* w1, const TRef* bias,
                 const TRef& y, const ResidualNormDesc* norm, const TRef* low) {
    if (d.rows == 0) return;
    const bool tc_type = w0.dtype == DT_BF16;
    const bool blocks = d.blocks > 1 || d.x_off > 0 || d.mul || (x0 && x0->shape[1] != d.k[0]);
    const long long ldx = x0 ? x0->shape[1] : d.k[0];
    const bool aligned = d.k[0] % 8 == 0 && d.k[1] % 8 == 0 && (!blocks || (ldx % 8 == 0 && d.x_off % 8 == 0 && d.x_step % 8 == 0));
    const size_t norm_smem = (size_t)d.rows * ((d.k[0] + 63) / 64 * 64 + 32) * 2;
    const bool gate_fits = !norm || !norm->gate || (norm->gate->shape[1] % 4 == 0 && norm->gate_off % 4 == 0 && norm->gate->buf.off % 16 == 0);
    const bool y_fits = norm && norm->y->shape[1] % 4 == 0 && norm->y_off % 4 == 0;
    // every CTA of the product repeats the norm: beyond some elements a launch of its own is shorter
    const int pro = !norm ? PRO_NONE : norm->streams > 0 ? PRO_STREAMS : norm->groups > 1 ? PRO_GROUPS : PRO_NORM;
    const bool parts_fit = pro == PRO_GROUPS ? (d.k[0] / norm->groups) % 4 == 0 : pro != PRO_STREAMS || !norm->y2 || norm->y2->dtype == norm->y->dtype;
    const int64_t read = d.rows * d.k[0] * (pro == PRO_STREAMS ? (norm->streams + 1) / 2 : 1);
    const bool fuse_norm = norm && tc_type && aligned && gate_fits && y_fits && parts_fit && d.rows <= 8 && read <= kFusedNormElements;
    TRef made;
    if (norm && !fuse_norm) {
        made.dtype = w0.dtype;
        made.shape = {d.rows, d.k[0]};
        // in 32-bit the sum of a norm that is not followed by another operation is the operand itself
        const bool own = w0.dtype == DT_F32 && norm->stream && !norm->pre && !low;
        if (low) made.buf = low->buf;
        else made.buf = own ? norm->stream->buf : em.scratch((size_t)d.rows * d.k[0] * (tc_type ? 2 : 4));
        emit_residual_norm(em, *norm, own ? nullptr : &made);
        x0 = &made;
    }
    LinP p{};
    p.ldx = blocks ? ldx : 0;
    p.x_off = d.x_off;
    p.x_step = d.x_step;
    p.blocks = (int)d.blocks;
    p.ldy = d.blocks * d.out;
    p.mul_ld = d.mul ? d.mul->shape[1] : 0;
    const Buf mul = d.mul ? d.mul->buf.at(d.mul_off * (tc_type ? 2 : 4)) : kNull;
    p.rows = d.rows;
    p.out = d.out;
    p.k[0] = d.k[0];
    p.k[1] = d.k[1];
    p.y_bf16 = y.dtype == DT_BF16;
    p.fast = tc_type;
    p.glu = d.glu;
    p.alpha = d.alpha;
    p.limit = d.limit;
    p.shift = d.shift;
    p.act[0] = d.act[0];
    p.act[1] = d.act[1];
    p.act_split = d.act_split;
    p.act_end = d.act_end > 0 ? d.act_end : d.blocks * d.out;
    p.node = em.node;
    p.splits = 1;
    const Buf bx0 = fuse_norm ? kNull : x0->buf, bx1 = buf_of(x1), bw1 = buf_of(w1), bb = buf_of(bias);
    const auto reduce = [&](const Buf& partial) {  // of a product that was cut along k
        const bool wide = p.ldy % 4 == 0 && y.buf.off % 16 == 0;
        const int v = wide ? 4 : p.ldy % 2 == 0 ? 2 : 1;  // gating needs pairs; out is even then
        p.out = p.ldy;                                    // all blocks' columns
        const auto k = tc_type ? (wide ? linear_reduce<4> : v == 2 ? linear_reduce<2> : linear_reduce<1>)
                               : (wide ? linear_reduce<4, float> : v == 2 ? linear_reduce<2, float> : linear_reduce<1, float>);
        em.launch(k, dim3((unsigned)((p.out + 256 * v - 1) / (256 * v)), (unsigned)d.rows), dim3(256), 0, p,
                  {{&p.bias, bb}, {&p.y, y.buf}, {&p.mul, mul}, {&p.partial, partial}}, "linear_reduce", /*pdl=*/true);
    };
    const bool quads = d.k[0] % 4 == 0 && d.k[1] % 4 == 0 && p.ldx % 4 == 0 && d.x_off % 4 == 0 && d.x_step % 4 == 0 && w0.buf.off % 16 == 0 &&
                       (!w1 || w1->buf.off % 16 == 0);
    if (!tc_type && quads && d.rows <= 32 && d.k[0] + d.k[1] >= 512) {
        // Eight rows per pass over the weights. 32 rows (four passes) take the 83 µs of linear_f32's one tile of 64; a short k is few steps
        // of such a tile, and its sums are added in order.
        const int m = d.rows == 1 ? 1 : d.rows == 2 ? 2 : d.rows <= 4 ? 4 : 8;
        auto units = [&](int r) { return (d.out + r - 1) / r * d.blocks; };
        const bool eight = m < 8 && units(8) * kStreamWarps >= 16LL * sm_count();  // enough warps with eight weight rows each
        const int r = eight ? 8 : 4;
        const long long chunks = (d.k[0] + 127) / 128 + (d.k[1] + 127) / 128;
        // warps per unit: until there are 16 per SM, with at least two steps for each
        p.nb = 1;
        while (p.nb < kStreamWarps && units(r) * p.nb < 16LL * sm_count() && chunks >= 4 * p.nb) p.nb *= 2;
        const int per_cta = kStreamWarps / p.nb;
        const auto k = m == 1 ? (eight ? linear_rows_f32<1, 8> : linear_rows_f32<1, 4>) : m == 2 ? (eight ? linear_rows_f32<2, 8> : linear_rows_f32<2, 4>)
                     : m == 4 ? (eight ? linear_rows_f32<4, 8> : linear_rows_f32<4, 4>) : linear_rows_f32<8, 4>;
        em.launch(k, dim3((unsigned)((units(r) + per_cta - 1) / per_cta), (unsigned)((d.rows + 7) / 8)), dim3(kThreads), 0, p,
                  {{&p.mul, mul}, {&p.x[0], bx0}, {&p.x[1], bx1}, {&p.w[0], w0.buf}, {&p.w[1], bw1}, {&p.bias, bb}, {&p.y, y.buf}}, "linear_rows_f32", /*pdl=*/true);
        return;
    }
    if (!tc_type && quads && f32_pays(d.k[0] + d.k[1])) {
        const dim3 tiles((unsigned)((d.out + 63) / 64 * d.blocks), (unsigned)((d.rows + 63) / 64));
        const long long steps = (d.k[0] + 15) / 16 + (d.k[1] + 15) / 16, ctas = (long long)tiles.x * tiles.y;
        // five CTAs fit an SM; pieces of at least 16 steps until three per SM are there
        while (p.splits < 8 && ctas * p.splits < 3LL * sm_count() && steps >= 32LL * p.splits && d.rows < 65536) p.splits *= 2;
        const Buf partial = p.splits > 1 ? em.scratch((size_t)p.splits * d.rows * p.ldy * 4) : kNull;
        em.launch(linear_f32, dim3(tiles.x, tiles.y, (unsigned)p.splits), dim3(kF32Threads), 0, p,
                  {{&p.mul, mul}, {&p.x[0], bx0}, {&p.x[1], bx1}, {&p.w[0], w0.buf}, {&p.w[1], bw1}, {&p.bias, bb}, {&p.y, y.buf}, {&p.partial, partial}},
                  "linear_f32", /*pdl=*/true);
        if (p.splits > 1) reduce(partial);
        return;
    }
    if (!tc_type || !aligned) {
        const dim3 grid((unsigned)((d.out + 63) / 64 * d.blocks), (unsigned)((d.rows + 63) / 64));
        const auto k = tc_type ? linear_simt<bf16> : linear_simt<float>;
        em.launch(k, grid, dim3(256), 0, p, {{&p.mul, mul}, {&p.x[0], bx0}, {&p.x[1], bx1}, {&p.w[0], w0.buf}, {&p.w[1], bw1}, {&p.bias, bb}, {&p.y, y.buf}},
                  "linear_simt", /*pdl=*/true);
        return;
    }
    if (d.rows <= 32) {
        const long long tiles = (d.out + 15) / 16 * d.blocks;
        const dim3 grid((unsigned)std::min<long long>(tiles, 2 * sm_count()));
        const int nt = d.rows <= 8 ? 1 : d.rows <= 16 ? 2 : 4;
        // More than eight rows read their activations from L2 a chunk ahead, beside a first-level cache that the ring leaves little of: linear_stream
        // → linear_flow, µs, 16 rows: k 5376, 21 504 weight rows 102 → 66 (9 rows 78 → 64); k 6912, 8192: 41 → 37; k 9216, 8192: 53 → 54; k 12 288, 8192: 67 → 83;
        // k 16 896, 5376: 83 → 103. 32 rows: k 6912, 8192: 61 → 45; k 12 288, 8192: 98 → 98; k 14 336, 8192: 112 → 118.
        const bool flow = !blocks && d.out * (d.k[0] + d.k[1]) * 2 > 2LL * sm_count() * kStreamWarps * kRing * 1024 &&
                          (nt == 1 || d.k[0] + d.k[1] <= (nt == 2 ? 8192 : 12288));
        auto k = nt == 1 ? linear_stream<1, PRO_NONE, false> : nt == 2 ? linear_stream<2, PRO_NONE, false> : linear_stream<4, PRO_NONE, false>;
        if (blocks) k = nt == 1 ? linear_stream<1, PRO_NONE, true> : nt == 2 ? linear_stream<2, PRO_NONE, true> : linear_stream<4, PRO_NONE, true>;
        if (flow) k = nt == 1 ? linear_flow<1, PRO_NONE> : nt == 2 ? linear_flow<2, PRO_NONE> : linear_flow<4, PRO_NONE>;
        unsigned smem = flow ? kStreamWarps * kRing * flow_slot(nt == 1 && !fuse_norm) : 0;
        if (fuse_norm) {
            k = pro == PRO_STREAMS ? linear_stream<1, PRO_STREAMS, false> : pro == PRO_GROUPS ? linear_stream<1, PRO_GROUPS, false> : linear_stream<1, PRO_NORM, false>;
            if (flow) k = pro == PRO_STREAMS ? linear_flow<1, PRO_STREAMS> : pro == PRO_GROUPS ? linear_flow<1, PRO_GROUPS> : linear_flow<1, PRO_NORM>;
            p.streams = (int)norm->streams;
            p.norm_groups = (int)norm->groups;
            smem += (unsigned)norm_smem;
            p.eps = (float)norm->eps;
            p.ny_bf16 = norm->y->dtype == DT_BF16;
            p.y_scale = (float)norm->y_scale;
            p.pre = norm->pre;
            p.ny_ld = norm->y->shape[1];
            p.add_scale = (float)norm->add_scale;
            p.add_bf16 = norm->add && norm->add->dtype == DT_BF16;
            p.gate_ld = norm->gate ? norm->gate->shape[1] : 0;
        }
        ensure_max_dynamic_smem((const void*)k, 150 * 1024);
        em.launch(k, grid, dim3(kStreamWarps * 32), smem, p,
                  {{&p.x[0], bx0}, {&p.x[1], bx1}, {&p.w[0], w0.buf}, {&p.w[1], bw1}, {&p.bias, bb}, {&p.y, y.buf}, {&p.mul, mul},
                   {&p.npost, fuse_norm ? buf_of(norm->post) : kNull}, {&p.nadd, fuse_norm ? buf_of(norm->add) : kNull},
                   {&p.noffset, fuse_norm ? buf_of(norm->offset) : kNull}, {&p.connect, fuse_norm ? buf_of(norm->connect) : kNull},
                   {&p.ny2, fuse_norm ? buf_of(norm->y2) : kNull}, {&p.npost2, fuse_norm ? buf_of(norm->post2) : kNull},
                   {&p.ny, fuse_norm ? norm->y->buf.at(norm->y_off * (p.ny_bf16 ? 2 : 4)) : kNull}, {&p.nw, fuse_norm ? norm->w->buf : kNull},
                   {&p.ngain, fuse_norm ? buf_of(norm->gain) : kNull}, {&p.nres, fuse_norm ? buf_of(norm->res) : kNull},
                   {&p.ngate, fuse_norm && norm->gate ? norm->gate->buf.at(norm->gate_off * 2) : kNull},
                   {&p.stream, fuse_norm ? buf_of(norm->stream) : kNull}, {&p.low, fuse_norm ? buf_of(low) : kNull}},
                  flow ? "linear_flow" : "linear_stream", /*pdl=*/true);
        return;
    }
    // Which kernel and activation rows per tile: the choice with the smallest modelled time. A CTA alone on its SM has a step of 64 k in `one` µs,
    // waves of two (up to 128 rows) in `two`; epilogues grow with the tile. The
    // constants are fitted to 560 launches of 45 sizes (64 … 4096 rows, k 16 … 10 240, 1152 … 32 768 weight rows): of one of them (200 × 2560 × 4096, 10 %) is the choice
    // more than 3 % behind the best form.
    const long long mt = (d.out + 127) / 128 * d.blocks, steps = (d.k[0] + 63) / 64 + (d.k[1] + 63) / 64;
    p.splits = pieces_of_k(d.rows, mt, steps, p.ldy);
    const int sp = p.splits;
    double best = 1e300;
    for (int nb : {32, 64, 128, 256}) {
        if (nb > 32 && nb / 2 >= d.rows) break;
        const int resident = nb <= 128 ? 2 : 1;
        const long long tiles = mt * ((d.rows + nb - 1) / nb);
        const double one = nb == 32 ? 0.19 : nb == 64 ? 0.21 : nb == 128 ? 0.24 : 0.35, two = nb == 32 ? 0.21 : nb == 64 ? 0.285 : nb == 128 ? 0.4 : 0.34;
        const double epilogue = 5.8 * nb / 256;
        const long long waves = (tiles * sp + sm_count() * resident - 1) / (sm_count() * resident), piece = (steps + sp - 1) / sp;
        const double us = 4.1 + (tiles * sp <= sm_count() ? piece * one + 0.9 + epilogue : waves * (piece * two + 0.9 + epilogue / 2) + epilogue / 2);
        if (us < best) {
            best = us;
            p.nb = nb;
        }
    }
    // Pairs of CTAs, which do not cut k: a step is bound by the bytes that come to an SM, 128 weight rows and half a tile's activation rows. Any multiple of 16 rows, so that the last round
    // of tiles is as full as the others.
    bool pair = false;
    for (int nb = 256; nb >= 64 && !blocks && sp == 1; nb -= 16) {
        const double rounds = std::ceil((double)((d.rows + nb - 1) / nb * ((d.out + 255) / 256)) / (sm_count() / 2)), us = pair_us(rounds, steps, nb);
        if (us < best) {
            best = us;
            pair = true;
            p.nb = nb;
        }
    }
    if (const char* e = std::getenv("ONYXIA_LINEAR_TILE")) {  // diagnostics: "rows,pieces"; no pieces: pairs of CTAs
        int nb = 0, sp = 0;
        if (std::sscanf(e, "%d,%d", &nb, &sp) == 2 && (nb == 32 || nb == 64 || nb == 128 || nb == 256) && sp >= 1 && sp <= 16 && sp * 2 <= std::max<long long>(steps, 2)) {
            pair = false;
            p.nb = nb;
            p.splits = sp;
        } else if (!blocks && sp == 0 && nb >= 16 && nb <= 256 && nb % 16 == 0) {
            pair = true;
            p.nb = nb;
            p.splits = 1;
        }
    }
    auto add_maps = [&](LaunchRec& rec, uint32_t box) {
        auto add = [&](int i, const Buf& b, int64_t k, int64_t rows, uint32_t high) {
            rec.tmaps.push_back(TmapReloc{(uint32_t)(offsetof(LinP, maps) + 128 * i), b, (uint64_t)k, (uint64_t)rows, (uint64_t)k * 2, 64u, high});
        };
        add(0, bx0, blocks ? ldx : d.k[0], d.rows, box);
        add(1, w0.buf, d.k[0], d.blocks * d.out, 128u);
        if (d.k[1]) {
            add(2, bx1, d.k[1], d.rows, box);
            add(3, bw1, d.k[1], d.out, 128u);
        }
    };
    p.row_tiles = (int)((d.rows + p.nb - 1) / p.nb);
    if (pair) {
        p.out_tiles = (int)((d.out + 255) / 256);
        p.box = p.nb / 2;
        add_maps(launch_pair(em, p, d.glu ? EPI_GLU : d.act[0] || d.act[1] ? EPI_ACT : EPI_PLAIN,
                             {{&p.bias, bb}, {&p.y, y.buf}, {&p.mul, kNull}, {&p.err, Buf{kSlotErr, 0}}}, y.buf.off, "linear_pair"),
                 (uint32_t)p.box);
        return;
    }
    const size_t stage = kTcPanelA + (size_t)p.nb * 128;
    p.out_tiles = (int)mt;
    const long long tiles = mt * p.row_tiles * p.splits;
    if (tiles >= INT32_MAX) throw std::runtime_error("onyxia.Linear: too many tiles");
    const bool alone = tiles <= sm_count();  // one CTA per SM: all of its shared memory
    p.stages = (int)std::min<size_t>(8, (p.nb <= 128 && !alone ? 108 * 1024 : 208 * 1024) / stage);
    const size_t smem = stage * p.stages + 1024 + (2 * p.stages + 4) * 8 + 16;
    const long long slots = (long long)sm_count() * (p.nb <= 128 ? 2 : 1);
    const bool one = tiles <= slots;
    const bool act = d.act[0] || d.act[1] || d.mul;
    const auto kernel = one ? (d.glu ? linear_tc<EPI_GLU, true> : act ? linear_tc<EPI_ACT, true> : linear_tc<EPI_PLAIN, true>)
                            : (d.glu ? linear_tc<EPI_GLU, false> : act ? linear_tc<EPI_ACT, false> : linear_tc<EPI_PLAIN, false>);
    ensure_max_dynamic_smem((const void*)kernel, 220 * 1024);
    const Buf partial = p.splits > 1 ? em.scratch((size_t)p.splits * d.rows * p.ldy * 4) : kNull;
    LaunchRec& rec = em.launch(kernel, one ? dim3((unsigned)p.row_tiles, (unsigned)mt, (unsigned)p.splits) : dim3((unsigned)slots), dim3(kTcThreads), (unsigned)smem, p,
                               {{&p.bias, bb}, {&p.y, y.buf}, {&p.mul, mul}, {&p.partial, partial}, {&p.err, Buf{kSlotErr, 0}}}, "linear_tc", /*pdl=*/true);
    add_maps(rec, (uint32_t)p.nb);
    if (p.splits > 1) reduce(partial);
}

// One product per group of sorted rows.
void emit_grouped_linear(Emitter& em, const GroupedLinearDesc& d, const TRef& x, const TRef& w, const TRef& counts, const TRef& y) {
    if (d.rows == 0) return;
    LinP p{};
    p.rows = d.rows;
    p.out = d.out;
    p.ldy = d.out;
    p.blocks = 1;
    p.k[0] = d.k;
    p.y_bf16 = y.dtype == DT_BF16;
    p.glu = d.glu;
    p.alpha = d.alpha;
    p.limit = d.limit;
    p.shift = d.shift;
    p.node = em.node;
    p.splits = 1;
    p.groups = (int)d.groups;
    auto tiles_of = [&](int64_t size) { return std::min<int64_t>(d.rows / size + std::min(d.groups, d.rows), d.rows); };
    const bool tc_type = w.dtype == DT_BF16;
    if (!tc_type || d.k % 8 != 0) {
        const bool quads = !tc_type && d.k % 4 == 0 && w.buf.off % 16 == 0 && f32_pays(d.k);
        const auto k = quads ? linear_f32 : tc_type ? linear_simt<bf16> : linear_simt<float>;
        em.launch(k, dim3((unsigned)((d.out + 63) / 64), (unsigned)tiles_of(64)), dim3(quads ? kF32Threads : 256), 0, p,
                  {{&p.x[0], x.buf}, {&p.x[1], kNull}, {&p.w[0], w.buf}, {&p.w[1], kNull}, {&p.bias, kNull}, {&p.y, y.buf}, {&p.counts, counts.buf}},
                  "grouped_simt", /*pdl=*/true);
        return;
    }
    // Rows per tile: a group of so many rows that they spread over more than a tile is expected to fill whole tiles and half a one. The costs are those of
    // emit_linear; tiles of 32 rows may have four CTAs per SM below, which is not modelled. Of 16 groups, k 1152 → 3456 gated: pairs of CTAs from 100 rows per group on (160:
    // 45 → 36 µs, 1024: 143 → 114); k 1728 → 1152, from 250 (33 → 28; 160 rows would take 25 against 23); k 2560 → 4096 gated, from 62 (74 → 66).
    const long long mt = (d.out + 127) / 128, steps = (d.k + 63) / 64;
    const double met = (double)std::min(d.groups, d.rows), mean = (double)d.rows / met;
    auto parts = [&](double nb) { return mean + 2.0 * std::sqrt(mean) <= nb ? 1.0 : mean / nb + 0.5; };
    double best = 1e300;
    for (int nb : {32, 64, 128, 256}) {
        const double two = nb == 32 ? 0.21 : nb == 64 ? 0.285 : nb == 128 ? 0.4 : 0.34, epilogue = 5.8 * nb / 256;
        const double waves = std::ceil(met * parts(nb) * (double)mt / (double)(sm_count() * (nb <= 128 ? 2 : 1)));
        const double us = 4.1 + waves * ((double)steps * two + 0.9 + epilogue / 2) + epilogue / 2;
        if (us < best) {
            best = us;
            p.nb = nb;
        }
    }
    const double pair_rounds = std::max(1.0, met * parts(256) * (double)((d.out + 255) / 256) / (sm_count() / 2) + 0.5);
    bool pair = pair_us(pair_rounds, steps, mean / parts(256)) < best;
    if (pair) p.nb = 256;
    if (const char* e = std::getenv("ONYXIA_GROUPED_TILE")) {  // diagnostics: rows; below zero: pairs of CTAs
        const int nb = std::atoi(e);
        pair = nb < 0 && nb >= -256 && nb % 16 == 0;
        if (pair || nb == 32 || nb == 64 || nb == 128 || nb == 256) p.nb = std::abs(nb);
    }
    auto add_maps = [&](LaunchRec& rec, uint32_t box) {
        auto add = [&](int i, const Buf& b, int64_t rows, uint32_t high) {
            rec.tmaps.push_back(TmapReloc{(uint32_t)(offsetof(LinP, maps) + 128 * i), b, (uint64_t)d.k, (uint64_t)rows, (uint64_t)d.k * 2, 64u, high});
        };
        add(0, x.buf, d.rows, box);
        add(1, w.buf, d.groups * d.out, 128u);
    };
    if (pair) {
        p.out_tiles = (int)((d.out + 255) / 256);
        p.row_tiles = (int)tiles_of(p.nb);  // at most
        p.box = 32;
        add_maps(launch_pair(em, p, d.glu ? EPI_GLU : EPI_PLAIN,
                             {{&p.bias, kNull}, {&p.y, y.buf}, {&p.mul, kNull}, {&p.err, Buf{kSlotErr, 0}}, {&p.counts, counts.buf}}, y.buf.off, "grouped_pair"),
                 (uint32_t)p.box);
        return;
    }
    const size_t stage = kTcPanelA + (size_t)p.nb * 128;
    p.out_tiles = (int)mt;
    const long long tiles = tiles_of(p.nb) * mt;  // at most
    if (tiles >= INT32_MAX) throw std::runtime_error("grouped product: too many tiles");
    // Tiles of 32 rows are bound by the weights' bytes: where more are expected than two CTAs of five stages per SM take at once, four of two stages, so
    // that few are left for a second round.
    const double expected = std::max((double)std::min(d.groups, d.rows), (double)d.rows / p.nb + 0.5 * (double)std::min(d.groups, d.rows)) * (double)mt;
    const int resident = p.nb == 32 && expected > 2.0 * sm_count() ? 4 : p.nb <= 128 ? 2 : 1;
    // A CTA per tile where a group has few rows: what a persistent CTA spends on finding its tiles stands beside few, short ones.
    const bool one = d.rows < 64 * d.groups;
    p.stages = (int)std::min<size_t>(8, (resident == 4 ? 48 * 1024 : resident == 2 ? 108 * 1024 : 208 * 1024) / stage);
    const size_t smem = stage * p.stages + 1024 + (2 * p.stages + 4) * 8 + 16;
    const auto kernel = one ? (d.glu ? linear_tc<EPI_GLU, true> : linear_tc<EPI_PLAIN, true>) : (d.glu ? linear_tc<EPI_GLU, false> : linear_tc<EPI_PLAIN, false>);
    ensure_max_dynamic_smem((const void*)kernel, 220 * 1024);
    const dim3 grid = one ? dim3((unsigned)tiles_of(p.nb), (unsigned)mt) : dim3((unsigned)std::min<long long>(tiles, (long long)sm_count() * resident));
    LaunchRec& rec = em.launch(kernel, grid, dim3(kTcThreads), (unsigned)smem, p,
                               {{&p.bias, kNull}, {&p.y, y.buf}, {&p.partial, kNull}, {&p.err, Buf{kSlotErr, 0}}, {&p.counts, counts.buf}}, "grouped_tc",
                               /*pdl=*/true);
    add_maps(rec, (uint32_t)p.nb);
}

}  // namespace oxk
