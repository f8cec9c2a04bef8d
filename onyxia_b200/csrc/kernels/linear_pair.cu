// Dense and grouped products of many rows by pairs of CTAs: `tcgen05.mma.cta_group::2`, 256 weight rows × up to 256 activation rows per tile.
//
// What bounds a large product is the bytes that come to an SM: about 64 a cycle. linear_tc's two 128 × 128 tiles per SM need 64 KB for what its matrix unit does in 512
// cycles, a CTA of a pair 32 KB (its own 128 weight rows, half of the activation rows; the hardware reads the other half from its neighbour), which is as long as the
// products take. Persistent pairs, one per two SMs; a warp copies weights, one activations, one issues the products of both CTAs, eight empty one
// of two accumulators under the products of the next tile. A tile may have any multiple of 16 rows, so that rounds of tiles are even (emit_linear chooses).
//
// linear_tc at its best tile, k uncut → pairs, back to back with weights from memory, µs (TFLOP/s): 2048 × 5376 × 16 896 272 → 251 (1482), 2048 × 5376 × 43 008 gated 651 → 617
// (1536), 2048 × 21 504 × 5376 394 → 334 (1419), 2048 × 2560 × 20 480 gated 178 → 148 (1455), 2048 × 2560 × 2560 39 → 29 (929), 4096 × 1152 × 4608 44 → 34, 1999 × 1152 × 13 824
// gated 68 → 51, 1046 × 2560 × 4160 33 → 28; 16 groups of 1024 rows, 2560 → 4096 gated: 361 → 240. A large tile's steps take 700
// cycles of which products are 512 (the power limit at these rates); steps of 128 rows take 450, of 64 430: small tiles are bound by their weights' bytes.
#include <type_traits>

#include "linear.cuh"

namespace oxk {

namespace {

constexpr unsigned kPanelA = 128 * 128;  // bytes: a CTA's 128 weight rows × 64 k
constexpr int kPairEpilogue = 8;         // warps
constexpr int kPairThreads = 352;        // 0-7 epilogue, 8 copies weights, 9 issues MMAs, 10 copies activations
// Bytes of the ring, always asked for: with them no other kernel that holds tensor memory fits beside a CTA, so that neither waits for the other's.
constexpr int kPairRing = 208 * 1024;

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned in_cta(unsigned addr, unsigned rank) {  // the same place of another CTA's shared memory
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void arrive_cluster(unsigned bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One box into this CTA's shared memory, its bytes counted by a barrier of either CTA of the pair.
__device__ __forceinline__ void pair_load(unsigned dst, const void* map, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void pair_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
        : "memory");
}
// Arrives at the same barrier of both CTAs once the MMAs issued so far are done.
__device__ __forceinline__ void pair_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((unsigned short)3)
                 : "memory");
}

struct PairTile {
    int group = 0, n0 = 0, live = 0, n = 0, m = 0;  // rows n0 … n0 + live, n columns of the accumulator, 256 weight rows from 256 m on
};

// Grouped: rows of a group are cut into parts of one size, as few as hold at most p.nb rows each. All tiles of a group come one after the other: its
// activations are read again for every 256 weight rows, while they are in L2. (All groups' parts for the same weight rows first: 16 groups of 1024
// rows × 2560 × 4096 gated in 291 µs.)
__device__ __forceinline__ int group_tiles(const LinP& p) {  // by whole warps
    int tiles = 0;
    for (int g = threadIdx.x & 31; g < p.groups; g += 32) tiles += (p.counts[g] + p.nb - 1) / p.nb;
    return __reduce_add_sync(0xffffffffu, tiles);
}
__device__ __forceinline__ void find_group(const LinP& p, int tile, PairTile* q) {  // by whole warps
    const int lane = threadIdx.x & 31;
    int tiles = 0, rows = 0;
    for (int g0 = 0; g0 < p.groups; g0 += 32) {
        const int n = g0 + lane < p.groups ? p.counts[g0 + lane] : 0, mine = (n + p.nb - 1) / p.nb;
        int t_inc = mine * p.out_tiles, r_inc = n;
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
            const int count = __shfl_sync(0xffffffffu, n, at), parts = __shfl_sync(0xffffffffu, mine, at);
            const int inner = tile - tiles - (__shfl_sync(0xffffffffu, t_inc, at) - parts * p.out_tiles), part = inner % parts;
            const int size = ((count + parts - 1) / parts + 15) & ~15;
            q->group = g0 + at;
            q->m = inner / parts;
            q->n0 = rows + __shfl_sync(0xffffffffu, r_inc, at) - count + part * size;
            q->live = min(size, count - part * size);
            q->n = (q->live + 15) & ~15;
            return;
        }
        tiles += __shfl_sync(0xffffffffu, t_inc, 31);
        rows += __shfl_sync(0xffffffffu, r_inc, 31);
    }
}

template <int EPI, bool YB> __global__ void __launch_bounds__(kPairThreads, 1) linear_pair(const __grid_constant__ LinP p) {
    using T = std::conditional_t<YB, bf16, float>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the same offset in both CTAs of the pair: their windows are alike
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned rank = cluster_rank();
    const int S = p.stages, half = (p.nb / 2 + p.box - 1) / p.box * p.box;  // rows of an activation panel
    const unsigned stage_bytes = kPanelA + (unsigned)half * 128;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + (size_t)S * stage_bytes);  // full[S], empty[S], finished[2], read[2]
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * S + 4);
    const unsigned bar0 = smem_u32(bars), finished = smem_u32(bars + 2 * S), read = finished + 16;
    int row_tiles = p.row_tiles;
    if (p.groups) {  // the counts come from an earlier launch
        pdl_wait();
        row_tiles = group_tiles(p);
    }
    const int first = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1, total = row_tiles * p.out_tiles;
    if (tid == 0) {
        for (int s = 0; s < 2 * S + 2; s++) mbar_init(smem_u32(bars + s), 1);
        for (int s = 0; s < 2; s++) mbar_init(read + s * 8, 2 * kPairEpilogue);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;
    pdl_trigger();  // not before all of this kernel's tensor memory is taken: a later kernel must not hold any while it waits for this one

    const int s0 = (int)((p.k[0] + 63) / 64), steps = s0 + (int)((p.k[1] + 63) / 64);
    auto tile_of = [&](int t) {  // by whole warps
        PairTile q;
        if (p.groups) {
            find_group(p, t, &q);
        } else {
            q.m = t / row_tiles;
            q.n0 = t % row_tiles * p.nb;
            q.live = (int)min((long long)p.nb, p.rows - q.n0);
            q.n = (q.live + 15) & ~15;
        }
        return q;
    };
    bool ok = true;

    if (warp == 8 || warp == 10) {
        // One warp copies weights, one activations. Stage and parity are carried along: a division per step would be longer than the step's copies.
        const bool weights = warp == 8;
        RingAt at;
        int round = 0;  // of the ring: the first waits for nothing
        bool ready = false;
        const int box = p.box;
        const unsigned full0 = in_cta(bar0, 0), empty = bar0 + S * 8;  // the first CTA's barriers count both CTAs' bytes
        const unsigned data = smem_u32(smem) + (weights ? 0 : kPanelA), box_bytes = (unsigned)p.box * 128;
        if (!weights) pdl_wait();
        for (int t = first; t < total; t += pairs) {
            const PairTile q = tile_of(t);
            const int boxes = ((q.n >> 1) + box - 1) / box;
            const int y0 = weights ? q.group * (int)p.out + q.m * 256 + (int)rank * 128 : q.n0 + (int)rank * (q.n >> 1);
            const unsigned bytes = 2 * (kPanelA + (unsigned)boxes * box_bytes);
            for (int i = 0; i < steps; i++) {
                if (!__all_sync(0xffffffffu, !round || ready || mbar_wait(empty + at.s * 8, at.parity ^ 1))) {
                    ok = false;
                    break;
                }
                const int op = i >= s0, x = (op ? i - s0 : i) * 64;
                const unsigned to = data + at.s * stage_bytes, bar = full0 + at.s * 8, mine = bar0 + at.s * 8;
                at.next(S);
                if (at.s == 0) round = 1;
                ready = mbar_test(empty + at.s * 8, at.parity ^ 1);  // the answer is there when the copies have been issued
                if (elect_one()) {
                    if (weights) {
                        if (rank == 0) mbar_expect_tx(mine, bytes);
                        pair_load(to, p.maps[op * 2 + 1], x, y0, bar);
                    } else {
                        for (int b = 0; b < boxes; b++) pair_load(to + b * box_bytes, p.maps[op * 2], x, y0 + b * box, bar);
                    }
                }
                __syncwarp();
            }
            if (!__all_sync(0xffffffffu, ok)) break;
        }
        // every copy has landed before shared memory can be given away (the other CTA's as well: both meet below)
        if (rank == 0 && weights)
            for (unsigned n = 0; n < (round ? (unsigned)S : at.s); n++)
                if (!mbar_wait(bar0 + n * 8, n < at.s ? at.parity : at.parity ^ 1)) ok = false;
        if (weights) pdl_wait();
    } else if (warp == 9) {
        pdl_wait();
        if (rank == 0) {
            RingAt at;
            bool ready = false;
            int j = 0;
            const unsigned empty = bar0 + S * 8, step16 = stage_bytes >> 4;
            const unsigned long long a0 = umma_kmajor_desc(smem_u32(smem)), b0 = umma_kmajor_desc(smem_u32(smem) + kPanelA);
            for (int t = first; t < total; t += pairs, j++) {
                const PairTile q = tile_of(t);
                const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(q.n >> 3) << 17) | (16u << 24);  // bf16 × bf16 → f32, M 256 × N n
                const unsigned d = tmem + (unsigned)((j & 1) * 256);
                if (j >= 2 && ok && !mbar_wait(read + (j & 1) * 8, ((j >> 1) - 1) & 1)) ok = false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = 0; i < steps; i++) {
                    if (ok && !ready && !mbar_wait(bar0 + at.s * 8, at.parity)) ok = false;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned long long a = a0 + at.s * step16, b = b0 + at.s * step16;  // descriptors count in 16 bytes
                    const unsigned done = empty + at.s * 8;
                    at.next(S);
                    ready = mbar_test(bar0 + at.s * 8, at.parity);  // the answer is there when the products have been issued
                    if (elect_one() && ok) {
#pragma unroll
                        for (int e = 0; e < 4; e++) pair_mma(d, a + e * 2, b + e * 2, idesc, i > 0 || e > 0);
                        pair_commit(done);
                    }
                    __syncwarp();
                }
                if (elect_one()) pair_commit(finished + (j & 1) * 8);
                __syncwarp();
                ok = __all_sync(0xffffffffu, ok);
            }
        }
    } else {
        pdl_wait();
        const unsigned read0 = in_cta(read, 0);
        int j = 0;
        for (int t = first; t < total; t += pairs, j++) {
            const PairTile q = tile_of(t);
            if (ok && !mbar_wait(finished + (j & 1) * 8, (j >> 1) & 1)) ok = false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const long long o = (long long)q.m * 256 + rank * 128 + (warp & 3) * 32 + lane, n0 = q.n0;  // weight row = accumulator lane
            const bool mine = ok && o < p.out;
            const float bias = p.bias && o < p.out ? p.bias[o] : 0.f;
            const int live = q.live;
            const int f = EPI == EPI_ACT && o < p.act_end ? p.act[o >= p.act_split] : ACT_NONE;
            const unsigned d = tmem + (unsigned)((j & 1) * 256) + ((unsigned)((warp & 3) * 32) << 16);
            for (int c = (warp >> 2) * 32; c < live; c += 64) {
                __syncwarp();
                unsigned v[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
                    "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                      "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
                      "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
                      "=r"(v[30]), "=r"(v[31])
                    : "r"(d + (unsigned)c));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float y[32];
#pragma unroll
                for (int e = 0; e < 32; e++) y[e] = __uint_as_float(v[e]) + bias;
                const int odd = lane & 1, there = live - c;  // rows of this chunk that exist
                if constexpr (EPI == EPI_GLU) {
                    // lanes 2i and 2i + 1 hold gate and up; of two activation rows the even lane finishes the first, the odd one the second
                    const long long width = p.out / 2;
                    T* to = (T*)p.y + (n0 + c + odd) * width + (o >> 1);
                    float r[16];
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        const float got = __shfl_xor_sync(0xffffffffu, odd ? y[2 * e] : y[2 * e + 1], 1);
                        const float g = fminf(odd ? got : y[2 * e], p.limit), u = fminf(fmaxf(odd ? y[2 * e + 1] : got, -p.limit), p.limit);
                        r[e] = g * (YB ? sigmoid_fast(p.alpha * g) : sigmoid_f(p.alpha * g)) * (u + p.shift);
                    }
                    if (!ok || (o | 1) >= p.out) continue;
                    if (there >= 32) {
#pragma unroll
                        for (int e = 0; e < 16; e++, to += 2 * width) *to = from_f<T>(r[e]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 16; e++, to += 2 * width)
                            if (2 * e + odd < there) *to = from_f<T>(r[e]);
                    }
                } else {
                    if constexpr (EPI == EPI_ACT) {
                        if (f == ACT_SOFTPLUS) {
#pragma unroll
                            for (int e = 0; e < 32; e++) y[e] = softplus_fast(y[e]);
                        } else if (f != ACT_NONE) {
#pragma unroll
                            for (int e = 0; e < 32; e++) y[e] = (YB ? sigmoid_fast(y[e]) : sigmoid_f(y[e])) * (f == ACT_SILU ? y[e] : 1.f);
                        }
                        __syncwarp();
                    }
                    if (YB && p.y_pairs) {  // two columns of a row per lane: out is even
                        unsigned w[16];
#pragma unroll
                        for (int e = 0; e < 16; e++) {
                            const float got = __shfl_xor_sync(0xffffffffu, odd ? y[2 * e] : y[2 * e + 1], 1);
                            w[e] = odd ? pack_bf16(got, y[2 * e + 1]) : pack_bf16(y[2 * e], got);
                        }
                        if (!mine) continue;
                        T* to = (T*)p.y + (n0 + c + odd) * p.ldy + (o & ~1ll);
                        if (there >= 32) {
#pragma unroll
                            for (int e = 0; e < 16; e++, to += 2 * p.ldy) *reinterpret_cast<unsigned*>(to) = w[e];
                        } else {
#pragma unroll
                            for (int e = 0; e < 16; e++, to += 2 * p.ldy)
                                if (2 * e + odd < there) *reinterpret_cast<unsigned*>(to) = w[e];
                        }
                    } else if (mine) {
                        T* to = (T*)p.y + (n0 + c) * p.ldy + o;
#pragma unroll
                        for (int e = 0; e < 32; e++, to += p.ldy)
                            if (e < there) *to = from_f<T>(y[e]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_cluster(read0 + (j & 1) * 8);
        }
    }
    if (!ok) report(p.err, ERR_WAIT_TIMEOUT, p.node, (long long)blockIdx.x, (long long)warp);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

}  // namespace

// Fitted beside linear_tc's costs, see emit_linear.
double pair_us(double rounds, double steps, double nb) { return 5.2 + rounds * (steps * (256 + nb) * 0.00062 + 0.9); }

LaunchRec& launch_pair(Emitter& em, LinP& p, int epi, std::initializer_list<std::pair<const void*, Buf>> ptrs, int64_t y_off, const char* label) {
    const int half = (p.nb / 2 + p.box - 1) / p.box * p.box;
    const size_t stage = kPanelA + (size_t)half * 128;
    p.stages = (int)std::min<size_t>(8, kPairRing / stage);
    p.y_pairs = p.ldy % 2 == 0 && y_off % 4 == 0;
    if ((long long)p.row_tiles * p.out_tiles >= INT32_MAX) throw std::runtime_error("onyxia.Linear: too many tiles");
    void (*const kernel)(const LinP) = p.y_bf16 ? (epi == EPI_GLU ? linear_pair<EPI_GLU, true> : epi == EPI_ACT ? linear_pair<EPI_ACT, true> : linear_pair<EPI_PLAIN, true>)
                                         : (epi == EPI_GLU ? linear_pair<EPI_GLU, false> : epi == EPI_ACT ? linear_pair<EPI_ACT, false> : linear_pair<EPI_PLAIN, false>);
    const int smem = kPairRing + 2048;
    ensure_max_dynamic_smem((const void*)kernel, smem);
    LaunchRec& rec = em.launch(kernel, dim3((unsigned)(sm_count() / 2 * 2)), dim3(kPairThreads), (unsigned)smem, p, ptrs, label, /*pdl=*/true);
    rec.cluster = dim3(2, 1, 1);
    return rec;
}

}  // namespace oxk
