// What the product kernels of linear.cu and linear_pair.cu share: their parameters, the group of a tile, gating and activations.
#pragma once
#include "tc_util.cuh"

namespace oxk {

struct LinP {
    alignas(64) unsigned char maps[4][128];  // x0, w0, x1, w1 (linear_tc)
    const void* x[2];
    const void* w[2];
    const float* bias;
    void* y;
    float* partial;
    ErrWord* err;
    // residual norm (linear_stream prologue)
    const void* ny;
    const float *nw, *ngain, *nres;
    const bf16* ngate;
    const float *npost, *noffset;
    const void* nadd;
    float* stream;
    bf16* low;
    long long gate_ld, ny_ld;
    float eps, y_scale, add_scale;
    int ny_bf16, pre, add_bf16, streams, norm_groups;
    const float *connect, *npost2;
    const void* ny2;
    long long rows, out, k[2];
    // block-diagonal products: x rows are ldx apart, block b reads its columns from x_off + b · x_step on; y rows are ldy apart
    const void* mul;
    long long ldx, x_off, x_step, ldy, mul_ld;
    int blocks;
    int y_bf16, fast, glu;  // fast: the operands are bf16
    float alpha, limit, shift;
    int act[2];           // functions of the columns before and from act_split on; none from act_end on
    long long act_split, act_end;
    int nb, stages, splits, node;  // linear_tc
    int row_tiles, out_tiles;      // tiles of activation rows (not grouped) and of weight rows
    int box, y_pairs;              // linear_pair: rows of one load of activations; results may be stored two columns at a time
    const int* counts;    // grouped: rows of every group
    int groups;
};

// Grouped: the `tile`-th tile of `size` rows, counted group by group → its group, first row and rows. Called by whole warps.
__device__ __forceinline__ bool locate_group(const LinP& p, int tile, int size, int* group, int* row, int* live) {
    const int lane = threadIdx.x & 31;
    int tiles = 0, rows = 0;
    for (int g0 = 0; g0 < p.groups; g0 += 32) {
        const int n = g0 + lane < p.groups ? p.counts[g0 + lane] : 0, mine = (n + size - 1) / size;
        int t_inc = mine, r_inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, t_inc, o), r = __shfl_up_sync(0xffffffffu, r_inc, o);
            if (lane >= o) {
                t_inc += t;
                r_inc += r;
            }
        }
        const unsigned hit = __ballot_sync(0xffffffffu, tiles + t_inc > tile);
        if (hit) {
            const int at = __ffs(hit) - 1;
            const int count = __shfl_sync(0xffffffffu, n, at);
            const int first = (tile - tiles - (__shfl_sync(0xffffffffu, t_inc, at) - __shfl_sync(0xffffffffu, mine, at))) * size;
            *group = g0 + at;
            *row = rows + __shfl_sync(0xffffffffu, r_inc, at) - count + first;
            *live = min(size, count - first);
            return true;
        }
        tiles += __shfl_sync(0xffffffffu, t_inc, 31);
        rows += __shfl_sync(0xffffffffu, r_inc, 31);
    }
    return false;
}

// Grouped: tiles of `size` rows over all groups. Called by whole warps.
__device__ __forceinline__ int count_tiles(const LinP& p, int size) {
    int tiles = 0;
    for (int g = threadIdx.x & 31; g < p.groups; g += 32) tiles += (p.counts[g] + size - 1) / size;
    return __reduce_add_sync(0xffffffffu, tiles);
}

__device__ __forceinline__ float glu_value(const LinP& p, float gate, float up) {
    const float g = fminf(gate, p.limit), u = fminf(fmaxf(up, -p.limit), p.limit);
    return g * (p.y_bf16 ? sigmoid_fast(p.alpha * g) : sigmoid_f(p.alpha * g)) * (u + p.shift);
}
// act: per column range
__device__ __forceinline__ float activate(const LinP& p, long long col, float v) {
    const int f = col < p.act_end ? p.act[col >= p.act_split] : ACT_NONE;
    if (f == ACT_NONE) return v;
    if (f == ACT_SOFTPLUS) return p.fast ? softplus_fast(v) : softplus_f(v);
    const float s = p.y_bf16 ? sigmoid_fast(v) : sigmoid_f(v);
    return f == ACT_SILU ? v * s : s;
}
// The factor of a block-diagonal product's result; the matrix has the weights' type.
template <typename T> __device__ __forceinline__ float factor(const LinP& p, long long row, long long col) {
    return p.mul ? to_f(((const T*)p.mul)[row * p.mul_ld + col]) : 1.f;
}
__device__ __forceinline__ void put(const LinP& p, long long row, long long width, long long col, float v) {
    if (p.y_bf16) ((bf16*)p.y)[row * width + col] = __float2bfloat16_rn(v);
    else ((float*)p.y)[row * width + col] = v;
}

// What an epilogue does: EPI_PLAIN bias only, EPI_GLU the gated unit, EPI_ACT functions of columns and factors. Kernels of their own: the
// paths of one are short enough to stay in the instruction cache.
enum : int { EPI_PLAIN, EPI_GLU, EPI_ACT };

// Pairs of CTAs on one tile (linear_pair.cu): the modelled µs of so many rounds of tiles, and the launch. `p` has its rows of a tile, its tiles and the rows of a load; the maps are the caller's.
double pair_us(double rounds, double steps, double nb);
LaunchRec& launch_pair(Emitter& em, LinP& p, int epi, std::initializer_list<std::pair<const void*, Buf>> ptrs, int64_t y_off, const char* label);

}  // namespace oxk
