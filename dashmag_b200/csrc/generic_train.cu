// The generic training kernels: forward, delta, query gradient, key/value gradients.
//
// They take every call of the contract (f32 / bf16 / f16, any head dimension up to 256, any
// strides, every mask, Tq != Tk, queries that see no key) with plain f32 FMAs on the CUDA cores:
// this is the IEEE-f32 path (no TF32, crates/dash-contract/src/lib.rs:69) and the path of the
// shapes the tensor-core kernels do not take.  No T x T matrix is ever held; the backward
// recomputes the scores tile by tile from the saved log-sum-exp, and sums every gradient in a
// fixed order (no atomics), so its results are the same bits on every run.
//
// Work split: a block of eight warps owns 8 RPW rows (queries, or keys in the key/value gradient
// kernel), RPW to a warp; the other side streams through shared memory in tiles of 32, one row per
// lane, double-buffered: the next tile is on its way (16-byte asynchronous copies for f32 rows that allow
// them) while this one is worked on.  A lane forms the dot products of its tile row with the warp's rows - four
// features at a time, from rows whose stride is an odd number of 16-byte chunks, so that eight lanes
// meet all banks - the warp reduces the maxima with shuffles, and for the second product each lane
// owns the head dimensions `lane + 32 i`.
//
// RPW is four where the rows fill the GPU that way (a tile row read from shared memory then serves four
// products), two or one where they do not (rows_per_warp): small calls are bound by the length of a block's chain of
// tiles, not by throughput.  Where one would do and shared memory allows it the block takes its tiles two at a time (KS 2): a warp
// has two rows and every second tile, and the two warps of the same rows add their sums at the end - half the links in the chain, and
// half the reads of shared memory a product.  Blocks of a cluster share rows likewise, a run of the sweep each (SHARE: forward_cluster, dq_cluster,
// dkdv_cluster).  NI is the number of head dimensions a lane owns (2, 4, 8 for D up to 64, 128, 256).
// Two packed sequences of 384 tokens, four heads of 64, f32: the step 254 ->
// 61 us side by side (three kernels of 105-113 us each, most of it scalar copies with a division an element, one after
// another), and 57 with the tiles two at a time; 381 tokens, 3 / 1 heads of 96, 74 -> 55, 590 148 -> 103, 1478 of 64 345 -> 246
// (the sums of two halves are nearer to f64 than one: dk of that call 9.3e-7 -> 6.8e-7).
#include <algorithm>

#include "bwd_common.cuh"
#include "common.cuh"
#include "launch.h"

namespace dash {

constexpr int TILE = 32;      // streamed rows per tile (one per lane)
constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;

__host__ __device__ inline int padded_d(int d) { return (d + 3) & ~3; }
// Floats between two rows of a tile: whole 16-byte chunks, an odd number of them.
__host__ __device__ inline int tile_stride(int d) { return padded_d(d) % 8 == 0 ? padded_d(d) + 4 : padded_d(d); }

__device__ __forceinline__ void copy_async(float *dst, const void *src, bool valid, int bytes16) {
    const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if (bytes16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(valid ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
// All of this thread's copies, the resident rows' too: a block with nothing to sweep must not leave with them in flight.
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Copies rows [r0, r0 + rows) of one head into shared memory as f32, zero past `limit` and past d.  `vec`: every row of the
// source can be read 16 bytes at a time and d is whole 16-byte vectors (f32: asynchronously, complete after copies_wait).
template <typename T>
__device__ __forceinline__ void stage_rows(float *dst, int stride, const View4 &src, int b, int h, int r0, int rows, int limit, int d, bool vec) {
    const T *base = static_cast<const T *>(src.ptr) + (int64_t)b * src.sb + (int64_t)h * src.sh;
    if (vec) {
        constexpr int V = 16 / sizeof(T);
        const int per = d / V, total = rows * per;
        for (int i0 = threadIdx.x; i0 < total; i0 += 2 * THREADS) {
            uint4 raw[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = i0 + u * THREADS, r = i / per, c = (i - r * per) * V;
                const bool in = i < total, valid = in && r0 + r < limit;
                const T *from = base + (int64_t)(valid ? r0 + r : 0) * src.st + (valid ? c : 0);
                if constexpr (sizeof(T) == 4) {
                    if (in) copy_async(dst + r * stride + c, from, valid, 1);
                } else {
                    raw[u] = make_uint4(0, 0, 0, 0);
                    if (valid) raw[u] = *reinterpret_cast<const uint4 *>(from);
                }
            }
            if constexpr (sizeof(T) == 2) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = i0 + u * THREADS, r = i / per, c = (i - r * per) * V;
                    if (i >= total) continue;
                    const T *e = reinterpret_cast<const T *>(&raw[u]);
                    float4 *to = reinterpret_cast<float4 *>(dst + r * stride + c);
                    to[0] = make_float4(Num<T>::to_f32(e[0]), Num<T>::to_f32(e[1]), Num<T>::to_f32(e[2]), Num<T>::to_f32(e[3]));
                    to[1] = make_float4(Num<T>::to_f32(e[4]), Num<T>::to_f32(e[5]), Num<T>::to_f32(e[6]), Num<T>::to_f32(e[7]));
                }
            }
        }
        return;
    }
    const int dp = padded_d(d);
    for (int idx = threadIdx.x; idx < rows * dp; idx += THREADS) {
        const int r = idx / dp, c = idx - r * dp;
        float x = 0.f;
        if (r0 + r < limit && c < d) x = Num<T>::to_f32(base[(int64_t)(r0 + r) * src.st + (int64_t)c * src.sd]);
        dst[r * stride + c] = x;
    }
}

// dot[r] = sum_c rows[r][c] * tile_row[c]: the warp's rows as broadcast float4, four partial sums a row.
template <int RPW>
__device__ __forceinline__ void dots(const float *rows, int row_stride, const float *tile_row, int dp, float (&out)[RPW]) {
    float4 acc[RPW];
#pragma unroll
    for (int r = 0; r < RPW; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int c = 0; c < dp; c += 4) {
        const float4 t = *reinterpret_cast<const float4 *>(tile_row + c);
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const float4 x = *reinterpret_cast<const float4 *>(rows + r * row_stride + c);
            acc[r].x = fmaf(x.x, t.x, acc[r].x);
            acc[r].y = fmaf(x.y, t.y, acc[r].y);
            acc[r].z = fmaf(x.z, t.z, acc[r].z);
            acc[r].w = fmaf(x.w, t.w, acc[r].w);
        }
    }
#pragma unroll
    for (int r = 0; r < RPW; ++r) out[r] = (acc[r].x + acc[r].y) + (acc[r].z + acc[r].w);
}

// acc[r][i] += sum_j weight[j][r] * tile[j][lane + 32 i] over the tile's 32 rows.
template <int RPW, int NI>
__device__ __forceinline__ void accumulate(const float *weight, const float *tile, int stride, int dp, float (&acc)[RPW][NI]) {
    const int lane = threadIdx.x & 31;
    constexpr int JS = 4 / RPW;   // rows whose weights are one 16-byte read
#pragma unroll 8 / JS
    for (int j0 = 0; j0 < TILE; j0 += JS) {
        const float4 w4 = *reinterpret_cast<const float4 *>(weight + j0 * RPW);
        const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int jj = 0; jj < JS; ++jj)
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int c = lane + 32 * i;
                const float v = c < dp ? tile[(j0 + jj) * stride + c] : 0.f;
#pragma unroll
                for (int r = 0; r < RPW; ++r) acc[r][i] = fmaf(w[jj * RPW + r], v, acc[r][i]);
            }
    }
}

// A lane's weights for the warp's rows, in one store.
template <int RPW>
__device__ __forceinline__ void put_weights(float *weight, const float (&w)[RPW]) {
    const int lane = threadIdx.x & 31;
    if constexpr (RPW == 4) reinterpret_cast<float4 *>(weight)[lane] = make_float4(w[0], w[1], w[2], w[3]);
    else if constexpr (RPW == 2) reinterpret_cast<float2 *>(weight)[lane] = make_float2(w[0], w[1]);
    else weight[lane] = w[0];
}

// KS warps swept a step's KS tiles for the same rows: the sums of the first take the others' in order.  `box`: the tiles' shared memory.
template <int RPW, int NI, int KS>
__device__ __forceinline__ void gather_shares(float *box, float (&acc)[RPW][NI]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert((KS - 1) * (WARPS / KS) * RPW * NI * 32 <= 4 * KS * TILE * (NI > 2 ? 68 : 4), "the shares fit where the tiles were");
    __syncthreads();   // nobody reads the tiles (or the shares before) any more
    if (w >= WARPS / KS) {
#pragma unroll
        for (int r = 0; r < RPW; ++r)
#pragma unroll
            for (int i = 0; i < NI; ++i) box[(((w - WARPS / KS) * RPW + r) * NI + i) * 32 + lane] = acc[r][i];
    }
    __syncthreads();
    if (w < WARPS / KS) {
#pragma unroll
        for (int o = 1; o < KS; ++o)
#pragma unroll
            for (int r = 0; r < RPW; ++r)
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[r][i] += box[((((o - 1) * (WARPS / KS) + w) * RPW + r) * NI + i) * 32 + lane];
    }
}

// ---- the blocks of a cluster (forward) -----------------------------------------------------------
__device__ __forceinline__ int cluster_blocks() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r)); return (int)r; }
__device__ __forceinline__ int cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return (int)r; }
__device__ __forceinline__ void cluster_meet() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// What is in block `rank`'s shared memory where `mine` is in this one's.
__device__ __forceinline__ float cluster_read(const float *mine, int rank) {
    uint32_t at;
    float x;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(mine))), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(at) : "memory");
    return x;
}

// The sums of the cluster's first block take the others' in order, through the tiles' shared memory of each (from 32 features on).
template <int RPW, int NI, int KS>
__device__ __forceinline__ void gather_cluster(float *box, float (&acc)[RPW][NI], int csize, int crank) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert((WARPS / KS) * RPW * NI * 32 <= 4 * KS * TILE * (NI > 2 ? 68 : 36), "the shares fit where the tiles were");
    float *mine = box + w * RPW * NI * 32 + lane;
    __syncthreads();   // nobody reads the tiles (or the shares before) any more
    if (crank > 0 && w < WARPS / KS) {
#pragma unroll
        for (int r = 0; r < RPW; ++r)
#pragma unroll
            for (int i = 0; i < NI; ++i) mine[(r * NI + i) * 32] = acc[r][i];
    }
    cluster_meet();
    if (crank == 0 && w < WARPS / KS) {
        for (int o = 1; o < csize; ++o)
#pragma unroll
            for (int r = 0; r < RPW; ++r)
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[r][i] += cluster_read(mine + (r * NI + i) * 32, o);
    }
    cluster_meet();   // the others' shared memory stays until it has been read
}

// The block's first row, and what each of its rows sees: the queries' key intervals (warp 0 places them) and their union.
struct RowSpans {
    int lo[32], hi[32];
    int kmin, kmax;
};
__device__ __forceinline__ void place_rows(RowSpans &sp, const MaskArgs &m, int row0, int rows, int tq, int tk) {
    if (threadIdx.x < 32) {
        int lo, hi;
        row_bounds_warp(m, row0 + (int)threadIdx.x, tq, tk, lo, hi);
        if ((int)threadIdx.x >= rows) { lo = tk; hi = 0; }
        sp.lo[threadIdx.x] = lo;
        sp.hi[threadIdx.x] = hi;
        const int kmin = warp_min_i(hi > lo ? lo : tk), kmax = warp_max_i(hi > lo ? hi : 0);
        if (threadIdx.x == 0) { sp.kmin = kmin; sp.kmax = kmax; }
    }
}

// ---------------------------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------------------------
template <typename T, int RPW, int NI, int KS, bool SHARE>
__global__ void __launch_bounds__(THREADS) generic_forward_kernel(TrainArgs a, int vec) {
    extern __shared__ __align__(16) float smem[];
    constexpr int ROWS = WARPS * RPW / KS, STEP = TILE * KS;
    const int dp = padded_d(a.d), sp = tile_stride(a.d);
    float *qs = smem;                          // [ROWS][dp]
    float *kv = qs + ROWS * dp;                // [2 buffers][K, V][STEP][sp]
    float *ps = kv + 4 * STEP * sp;            // [8 warps][32 keys][RPW]
    __shared__ RowSpans rs;
    __shared__ int pad[2][STEP];               // key padding flags of the tile

    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wr = w % (WARPS / KS), sub = w / (WARPS / KS);   // the warp's rows; its tile of the step's KS
    const int csize = SHARE ? cluster_blocks() : 1, crank = SHARE ? cluster_rank() : 0;   // blocks that share the rows, each a run of their keys
    const int qt = (gridDim.x - 1 - blockIdx.x) / csize;  // long (late) causal rows first
    const int h = blockIdx.y, b = blockIdx.z;
    const int hk = h / (a.hq / a.hkv);
    const int row0 = qt * ROWS;

    stage_rows<T>(qs, dp, a.q, b, h, row0, ROWS, a.tq, a.d, vec);
    place_rows(rs, a.mask, row0, ROWS, a.tq, a.tk);
    __syncthreads();
    int kmin = rs.kmin, kmax = rs.kmax;
    if (a.mask.kind == 1) trim_padded(a.mask, b, kmin, kmax);

    int lo[RPW], hi[RPW];
    int wlo = a.tk, whi = 0;
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        lo[r] = rs.lo[wr * RPW + r];
        hi[r] = rs.hi[wr * RPW + r];
        if (hi[r] > lo[r]) { wlo = min(wlo, lo[r]); whi = max(whi, hi[r]); }
    }
    float m[RPW], l[RPW], acc[RPW][NI];   // l: this lane's share of the row's sum
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < NI; ++i) acc[r][i] = 0.f;
    }
    auto stage = [&](int k0, int buf) {
        stage_rows<T>(kv + (2 * buf) * STEP * sp, sp, a.k, b, hk, k0, STEP, a.tk, a.d, vec);
        stage_rows<T>(kv + (2 * buf + 1) * STEP * sp, sp, a.v, b, hk, k0, STEP, a.tk, a.d, vec);
        if (threadIdx.x < STEP) {
            const int key = k0 + threadIdx.x;
            pad[buf][threadIdx.x] = key >= a.tk || key_padded(a.mask, b, key) ? 1 : 0;
        }
    };
    int first = kmin / TILE * TILE;
    if (SHARE && kmax > kmin) {   // (tiles are whole, so only the last of the runs ends inside one)
        const int per = ((kmax - first + TILE - 1) / TILE + csize - 1) / csize * TILE;
        first += crank * per;
        kmax = min(kmax, first + per);
        whi = min(whi, kmax);
    }
    if (SHARE ? kmax > first : kmax > kmin) stage(first, 0);
    for (int k0 = first, buf = 0; k0 < kmax; k0 += STEP, buf ^= 1) {
        copies_wait();
        __syncthreads();   // the tile is whole, and every warp is done with the other buffer
        if (k0 + STEP < kmax) stage(k0 + STEP, buf ^ 1);
        const int t0 = k0 + sub * TILE;
        if (t0 + TILE <= wlo || t0 >= whi) continue;  // no row of this warp sees the tile
        const float *ks = kv + (2 * buf) * STEP * sp + sub * TILE * sp, *vs = ks + STEP * sp;

        float s[RPW];
        dots<RPW>(qs + wr * RPW * dp, dp, ks + lane * sp, dp, s);
        const int key = t0 + lane;
        const bool open = pad[buf][sub * TILE + lane] == 0;
        float *pw = ps + w * TILE * RPW, ps4[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const bool vis = open && key >= lo[r] && key < hi[r];
            const float sr = vis ? s[r] * a.scale : -INFINITY;
            const float mn = fmaxf(m[r], warp_max(sr));
            // No maximum yet: the weights are zero, but for a NaN - no maximum shows it, and it is a NaN of the row whatever else the
            // row sees, in this warp's tiles or in another's.
            float p = sr == sr ? 0.f : sr, alpha = 1.f;
            if (mn != -INFINITY) {
                alpha = expf(m[r] - mn);  // exp(-inf) = 0 on the first visible tile
                p = expf(sr - mn);
            }
            l[r] = l[r] * alpha + p;
#pragma unroll
            for (int i = 0; i < NI; ++i) acc[r][i] *= alpha;
            m[r] = mn;
            ps4[r] = p;
        }
        put_weights<RPW>(pw, ps4);
        __syncwarp();
        accumulate<RPW, NI>(pw, vs, sp, dp, acc);
        __syncwarp();
    }
    copies_wait();
    if constexpr (KS > 1) {
        // The warps that swept the other tiles hand over what they have, through the tiles' shared memory (4 STEP rows of at least
        // four floats).
        static_assert((KS - 1) * (WARPS / KS) * RPW * (NI + 2) * 32 <= 4 * STEP * (NI > 2 ? 68 : 4), "the shares fit where the tiles were");
        __syncthreads();
        auto box_of = [&](int s) { return kv + ((s - 1) * (WARPS / KS) + wr) * RPW * (NI + 2) * 32 + lane; };
        if (sub > 0) {
#pragma unroll
            for (int r = 0; r < RPW; ++r) {
                float *x = box_of(sub) + r * (NI + 2) * 32;
                x[0] = m[r];
                x[32] = l[r];
#pragma unroll
                for (int i = 0; i < NI; ++i) x[(2 + i) * 32] = acc[r][i];
            }
        }
        __syncthreads();
        if (sub > 0 && !SHARE) return;
#pragma unroll
        for (int o = 1; o < KS; ++o)
#pragma unroll
            for (int r = 0; r < RPW; ++r) {
                if (sub > 0) break;
                const float *x = box_of(o) + r * (NI + 2) * 32;
                const float mn = fmaxf(m[r], x[0]);
                const float mine = mn == -INFINITY ? 1.f : expf(m[r] - mn), theirs = mn == -INFINITY ? 1.f : expf(x[0] - mn);
                l[r] = l[r] * mine + x[32] * theirs;
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[r][i] = acc[r][i] * mine + x[(2 + i) * 32] * theirs;
                m[r] = mn;
            }
    }
    if constexpr (SHARE) {
        // The cluster's blocks hand over what they have in the same way, block after block in order, through the tiles' shared
        // memory of each; the first block finishes the rows.
        static_assert((WARPS / KS) * RPW * (NI + 2) * 32 <= 4 * STEP * (NI > 2 ? 68 : 36), "the shares fit where the tiles were, from 32 features on");
        float *box = kv + wr * RPW * (NI + 2) * 32 + lane;
        __syncthreads();   // no warp is at its last tile any more, nor at the shares above
        if (sub == 0 && crank > 0) {
#pragma unroll
            for (int r = 0; r < RPW; ++r) {
                float *x = box + r * (NI + 2) * 32;
                x[0] = m[r];
                x[32] = l[r];
#pragma unroll
                for (int i = 0; i < NI; ++i) x[(2 + i) * 32] = acc[r][i];
            }
        }
        cluster_meet();
        if (sub == 0 && crank == 0) {
            for (int o = 1; o < csize; ++o)
#pragma unroll
                for (int r = 0; r < RPW; ++r) {
                    const float *x = box + r * (NI + 2) * 32;
                    float theirs_acc[NI];
                    const float tm = cluster_read(x, o), tl = cluster_read(x + 32, o);
#pragma unroll
                    for (int i = 0; i < NI; ++i) theirs_acc[i] = cluster_read(x + (2 + i) * 32, o);
                    const float mn = fmaxf(m[r], tm);
                    const float mine = mn == -INFINITY ? 1.f : expf(m[r] - mn), theirs = mn == -INFINITY ? 1.f : expf(tm - mn);
                    l[r] = l[r] * mine + tl * theirs;
#pragma unroll
                    for (int i = 0; i < NI; ++i) acc[r][i] = acc[r][i] * mine + theirs_acc[i] * theirs;
                    m[r] = mn;
                }
        }
        cluster_meet();   // the others' shared memory stays until it has been read
        if (crank > 0 || sub > 0) return;
    }

    T *out = static_cast<T *>(a.out);
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int row = row0 + wr * RPW + r;
        const float sum = warp_sum(l[r]);
        if (row >= a.tq) continue;
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
        const int64_t base = (((int64_t)b * a.tq + row) * a.hq + h);
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int c = lane + 32 * i;
            if (c < a.d) out[base * a.d + c] = Num<T>::from_f32(acc[r][i] * inv);
        }
        if (lane == 0) a.lse[base] = sum > 0.f ? m[r] + logf(sum) : -INFINITY;
    }
}

// ---------------------------------------------------------------------------------------------
// delta = rowsum(dO * O), one warp per (batch, query, head); from the output as stored.
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(THREADS) generic_delta_kernel(TrainArgs a) {
    allow_beside();
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)a.b * a.tq * a.hq;
    int64_t row = (int64_t)blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);
    if (row < rows) {
        int h = (int)(row % a.hq);
        int64_t bt = row / a.hq;
        int t = (int)(bt % a.tq), b = (int)(bt / a.tq);
        float sum = 0.f;
        for (int c = lane; c < a.d; c += 32) sum = fmaf(load_f32<T>(a.dout, b, t, h, c), load_f32<T>(a.o, b, t, h, c), sum);
        sum = warp_sum(sum);
        if (lane == 0) a.delta[row] = sum;
    }
    end_beside();
}

// ---------------------------------------------------------------------------------------------
// dQ: each block of queries sweeps, in order, the key tiles it sees.
// ---------------------------------------------------------------------------------------------
// (Four rows a warp at D 128, shared: with more than 128 registers a thread a block would be alone on its multiprocessor.  One row a warp: 64
// registers, where ptxas left to itself takes 72 - 333 tokens in six, 8 / 2 heads of 80, backward 95 and 112 us.)
template <typename T, int RPW, int NI, int KS, bool SHARE>
__global__ void __launch_bounds__(THREADS, RPW == 4 && NI == 4 && SHARE ? 2 : RPW == 1 && NI == 4 ? 4 : 0) generic_dq_kernel(TrainArgs a, int vec) {
    extern __shared__ __align__(16) float smem[];
    constexpr int ROWS = WARPS * RPW / KS, STEP = TILE * KS;
    const int dp = padded_d(a.d), sp = tile_stride(a.d);
    float *qs = smem;                          // [ROWS][dp]
    float *gs = qs + ROWS * dp;                // [ROWS][dp]   dO
    float *kv = gs + ROWS * dp;                // [2 buffers][K, V][STEP][sp]
    float *ps = kv + 4 * STEP * sp;            // [8][32][RPW]  dS
    __shared__ RowSpans rs;
    __shared__ int pad[2][STEP];

    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wr = w % (WARPS / KS), sub = w / (WARPS / KS);
    const int csize = SHARE ? cluster_blocks() : 1, crank = SHARE ? cluster_rank() : 0;
    const int qt = (gridDim.x - 1 - blockIdx.x) / csize;
    const int h = blockIdx.y, b = blockIdx.z;
    const int hk = h / (a.hq / a.hkv);
    const int row0 = qt * ROWS;

    stage_rows<T>(qs, dp, a.q, b, h, row0, ROWS, a.tq, a.d, vec);
    stage_rows<T>(gs, dp, a.dout, b, h, row0, ROWS, a.tq, a.d, vec);
    place_rows(rs, a.mask, row0, ROWS, a.tq, a.tk);
    __syncthreads();
    int kmin = rs.kmin, kmax = rs.kmax;
    if (a.mask.kind == 1) trim_padded(a.mask, b, kmin, kmax);

    int lo[RPW], hi[RPW];
    float lse[RPW], delta[RPW];
    int wlo = a.tk, whi = 0;
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int row = row0 + wr * RPW + r;
        lo[r] = rs.lo[wr * RPW + r];
        hi[r] = rs.hi[wr * RPW + r];
        if (hi[r] > lo[r]) { wlo = min(wlo, lo[r]); whi = max(whi, hi[r]); }
        float x = INFINITY, dl = 0.f;
        if (row < a.tq) {
            const int64_t at = ((int64_t)b * a.tq + row) * a.hq + h;
            x = a.lse[at];
            dl = a.delta[at];
        }
        lse[r] = x == -INFINITY ? INFINITY : x;  // a query that saw no key: P = 0
        delta[r] = dl;
    }
    float acc[RPW][NI];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
        for (int i = 0; i < NI; ++i) acc[r][i] = 0.f;
    auto stage = [&](int k0, int buf) {
        stage_rows<T>(kv + (2 * buf) * STEP * sp, sp, a.k, b, hk, k0, STEP, a.tk, a.d, vec);
        stage_rows<T>(kv + (2 * buf + 1) * STEP * sp, sp, a.v, b, hk, k0, STEP, a.tk, a.d, vec);
        if (threadIdx.x < STEP) {
            const int key = k0 + threadIdx.x;
            pad[buf][threadIdx.x] = key >= a.tk || key_padded(a.mask, b, key) ? 1 : 0;
        }
    };
    int first = kmin / TILE * TILE;
    if (SHARE && kmax > kmin) {   // as in the forward
        const int per = ((kmax - first + TILE - 1) / TILE + csize - 1) / csize * TILE;
        first += crank * per;
        kmax = min(kmax, first + per);
        whi = min(whi, kmax);
    }
    if (SHARE ? kmax > first : kmax > kmin) stage(first, 0);
    for (int k0 = first, buf = 0; k0 < kmax; k0 += STEP, buf ^= 1) {
        copies_wait();
        __syncthreads();
        if (k0 + STEP < kmax) stage(k0 + STEP, buf ^ 1);
        const int t0 = k0 + sub * TILE;
        if (t0 + TILE <= wlo || t0 >= whi) continue;
        const float *ks = kv + (2 * buf) * STEP * sp + sub * TILE * sp, *vs = ks + STEP * sp;

        float s[RPW], dpv[RPW];
        dots<RPW>(qs + wr * RPW * dp, dp, ks + lane * sp, dp, s);
        dots<RPW>(gs + wr * RPW * dp, dp, vs + lane * sp, dp, dpv);
        const int key = t0 + lane;
        const bool open = pad[buf][sub * TILE + lane] == 0;
        float *pw = ps + w * TILE * RPW, ds4[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const bool vis = open && key >= lo[r] && key < hi[r];
            const float p = vis ? expf(s[r] * a.scale - lse[r]) : 0.f;
            ds4[r] = p * (dpv[r] - delta[r]);
        }
        put_weights<RPW>(pw, ds4);
        __syncwarp();
        accumulate<RPW, NI>(pw, ks, sp, dp, acc);
        __syncwarp();
    }
    copies_wait();
    if constexpr (KS > 1) gather_shares<RPW, NI, KS>(kv, acc);
    if constexpr (SHARE) gather_cluster<RPW, NI, KS>(kv, acc, csize, crank);

    T *dq = static_cast<T *>(a.dq);
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int row = row0 + wr * RPW + r;
        if (row >= a.tq || sub > 0 || crank > 0) continue;
        const int64_t base = (((int64_t)b * a.tq + row) * a.hq + h) * a.d;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int c = lane + 32 * i;
            if (c < a.d) dq[base + c] = Num<T>::from_f32(acc[r][i] * a.scale);
        }
    }
    end_beside();   // dkdv
}

// ---------------------------------------------------------------------------------------------
// dK, dV: each block of keys sweeps, in order, the query heads of its group and the query
// tiles that see it; a warp owns RPW keys, a lane one query of the tile.
// ---------------------------------------------------------------------------------------------
template <typename T, int RPW, int NI, int KS, bool SHARE>
__global__ void __launch_bounds__(THREADS) generic_dkdv_kernel(TrainArgs a, int vec) {
    extern __shared__ __align__(16) float smem[];
    constexpr int ROWS = WARPS * RPW / KS, STEP = TILE * KS;
    const int dp = padded_d(a.d), sp = tile_stride(a.d);
    float *ks = smem;                          // [ROWS][dp]
    float *vs = ks + ROWS * dp;                // [ROWS][dp]
    float *qg = vs + ROWS * dp;                // [2 buffers][Q, dO][STEP][sp]
    float *ps = qg + 4 * STEP * sp;            // [8][32][RPW]  P
    float *ds = ps + WARPS * TILE * RPW;       // [8][32][RPW]  dS
    __shared__ float lses[2][STEP], deltas[2][STEP];
    __shared__ int from[32], to[32];           // the queries that see each of the block's keys

    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wr = w % (WARPS / KS), sub = w / (WARPS / KS);
    const int csize = SHARE ? cluster_blocks() : 1, crank = SHARE ? cluster_rank() : 0;   // blocks that share the keys, each a run of the steps
    const int kt = blockIdx.x / csize, hk = blockIdx.y, b = blockIdx.z;
    const int group = a.hq / a.hkv;
    const int key0 = kt * ROWS;

    stage_rows<T>(ks, dp, a.k, b, hk, key0, ROWS, a.tk, a.d, vec);
    stage_rows<T>(vs, dp, a.v, b, hk, key0, ROWS, a.tk, a.d, vec);
    if (threadIdx.x < ROWS) {
        const int key = key0 + threadIdx.x;
        int qa = 0, qb = 0;
        if (key < a.tk && !key_padded(a.mask, b, key)) queries_of_key(a.mask, key, a.tq, a.tk, qa, qb);
        from[threadIdx.x] = qa;
        to[threadIdx.x] = qb;
    }
    // The queries that may see some key of the block: those that see none of them are masked key by key.
    int qfirst, qend;
    query_range(a.mask, key0, min(key0 + ROWS, a.tk), a.tq, a.tk, qfirst, qend);
    allow_beside();    // dq
    __syncthreads();
    int qa[RPW], qb[RPW];
    int wfrom = a.tq, wto = 0;
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        qa[r] = from[wr * RPW + r];
        qb[r] = to[wr * RPW + r];
        if (qb[r] > qa[r]) { wfrom = min(wfrom, qa[r]); wto = max(wto, qb[r]); }
    }
    float acck[RPW][NI], accv[RPW][NI];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
        for (int i = 0; i < NI; ++i) { acck[r][i] = 0.f; accv[r][i] = 0.f; }

    const int first = qfirst / TILE * TILE, tiles = qend > qfirst ? (qend - first + STEP - 1) / STEP : 0, all_steps = tiles * group;
    const int begin = all_steps * crank / csize, steps = all_steps * (crank + 1) / csize;   // this block's [begin, steps)
    auto stage = [&](int t, int buf) {
        const int h = hk * group + t / tiles, q0 = first + t % tiles * STEP;
        stage_rows<T>(qg + (2 * buf) * STEP * sp, sp, a.q, b, h, q0, STEP, a.tq, a.d, vec);
        stage_rows<T>(qg + (2 * buf + 1) * STEP * sp, sp, a.dout, b, h, q0, STEP, a.tq, a.d, vec);
        if (threadIdx.x < 2 * STEP) {
            const int row = q0 + (threadIdx.x & (STEP - 1));
            const bool in = row < a.tq;
            const int64_t at = ((int64_t)b * a.tq + (in ? row : 0)) * a.hq + h;
            if (threadIdx.x < STEP) copy_async(&lses[buf][threadIdx.x], a.lse + at, in, 0);
            else copy_async(&deltas[buf][threadIdx.x - STEP], a.delta + at, in, 0);
        }
    };
    if (steps > begin) stage(begin, begin & 1);
    for (int t = begin; t < steps; ++t) {
        const int buf = t & 1, q0 = first + t % tiles * STEP + sub * TILE;
        copies_wait();
        __syncthreads();
        if (t + 1 < steps) stage(t + 1, buf ^ 1);
        if (q0 + TILE <= wfrom || q0 >= wto) continue;   // no key of this warp is seen from the tile
        const float *qs = qg + (2 * buf) * STEP * sp + sub * TILE * sp, *gs = qs + STEP * sp;

        float s[RPW], dpv[RPW];
        dots<RPW>(ks + wr * RPW * dp, dp, qs + lane * sp, dp, s);
        dots<RPW>(vs + wr * RPW * dp, dp, gs + lane * sp, dp, dpv);
        const int row = q0 + lane;
        const float x = lses[buf][sub * TILE + lane], lse = x == -INFINITY ? INFINITY : x, delta = deltas[buf][sub * TILE + lane];
        float *pw = ps + w * TILE * RPW, *dw = ds + w * TILE * RPW, ps4[RPW], ds4[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const bool vis = row >= qa[r] && row < qb[r];
            const float p = vis ? expf(s[r] * a.scale - lse) : 0.f;
            ps4[r] = p;
            ds4[r] = p * (dpv[r] - delta);
        }
        put_weights<RPW>(pw, ps4);
        put_weights<RPW>(dw, ds4);
        __syncwarp();
        accumulate<RPW, NI>(pw, gs, sp, dp, accv);
        accumulate<RPW, NI>(dw, qs, sp, dp, acck);
        __syncwarp();
    }
    copies_wait();
    if constexpr (KS > 1) {
        gather_shares<RPW, NI, KS>(qg, acck);
        gather_shares<RPW, NI, KS>(qg, accv);
    }
    if constexpr (SHARE) {
        gather_cluster<RPW, NI, KS>(qg, acck, csize, crank);
        gather_cluster<RPW, NI, KS>(qg, accv, csize, crank);
    }

    T *dk = static_cast<T *>(a.dk), *dv = static_cast<T *>(a.dv);
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int key = key0 + wr * RPW + r;
        if (key >= a.tk || sub > 0 || crank > 0) continue;
        const int64_t base = (((int64_t)b * a.tk + key) * a.hkv + hk) * a.d;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int c = lane + 32 * i;
            if (c < a.d) {
                dk[base + c] = Num<T>::from_f32(acck[r][i] * a.scale);
                dv[base + c] = Num<T>::from_f32(accv[r][i]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------------

// Whether every row of the view can be read 16 bytes at a time.
template <typename T>
static bool rows_readable(const View4 &v, int d) {
    const int64_t per = 16 / sizeof(T);
    return v.sd == 1 && d % per == 0 && reinterpret_cast<uintptr_t>(v.ptr) % 16 == 0 && v.sb % per == 0 && v.st % per == 0 && v.sh % per == 0;
}

// `own`: tensors whose rows the block keeps; `probs`: arrays of a tile's weights.
// SHARED_ROWS in the place of the rows per warp: two rows a warp, and each pair of rows two warps' (KS 2).
constexpr int SHARED_ROWS = 0;
static int block_rows(int rpw) { return rpw == SHARED_ROWS ? WARPS : WARPS * rpw; }
static size_t generic_smem(int d, int rpw, int own, int probs) {
    const int each = rpw == SHARED_ROWS ? 2 : rpw, ks = rpw == SHARED_ROWS ? 2 : 1;
    return sizeof(float) * ((size_t)own * block_rows(rpw) * padded_d(d) + 4 * ks * TILE * tile_stride(d) + (size_t)probs * WARPS * TILE * each);
}

// Rows per warp: the fewest of one, two and four whose blocks all run at once - as many to a multiprocessor as its shared
// memory holds (a block also takes its static arrays and the kilobyte the system keeps for it), up to two and a half (beyond,
// the reads of shared memory that more rows would share are what it waits for) - else four.  Measured, f32, causal (rows per
// warp 1 | 2 | 4, us): forward of 130 tokens x 4 heads of 64 (68 | 36 | 20 blocks) 12 | 14 | 16; 300 x 8 of 128
// (304 | 152 | 80) 45 | 43 | 47; 1000 x 8 of 64 (1000 | 504 | 256) 190 | 127 | 125; 60 queries x 32 heads of 256 against 2060
// keys, one block to a multiprocessor (256 | 128 | 64) 672 | 362 | 501; 100 against 9100 (416 | 224 | 128) 4395 | 3153 | 2213;
// backward of 300 x 8 / 2 heads of 128 204 | 248 | 293 (the rule, which picks for each kernel: 184), of 1400 x 4 of 128
// 749 | 549 | 450, of 700 x 4 of 128 230 | 170 | 215.  It is not the best of the three everywhere: the forward of 700 x 4 of
// 128 takes one row a warp, 118 us, where four take 101; of 1000 x 8 / 2 of 96 four, 195, where two take 165.
// Shared rows sum in another order (even and odd tiles apart), so a slice of a call's heads or batch, which may take them where the call
// does not, can differ from it in the last bits.  What it would cost to keep them: every form with the two sums apart, 75 calls, f32,
// 0 to 3 % on average, but 4 heads of 128, 1500 tokens, 146 -> 205 us forward and 368 -> 420 backward, 8 of 96, 900 tokens, 111 -> 128
// and 214 -> 259 (the second set of sums in registers; in local memory 111 -> 133 and 214 -> 371); shared rows by the number of rows
// alone, 32 heads of 64, 200 tokens, backward 48 -> 65, 32 of 128 79 -> 138; without them 3 / 1 heads of 96, 590 tokens, 103 -> 148.
constexpr int64_t SMEM_PER_SM = 228 * 1024, SMEM_BESIDE = 2 * 1024;
static int rows_per_warp(int64_t rows, int64_t heads, int d, int own, int probs) {
    for (int rpw = 1; rpw < 4; rpw *= 2) {
        const int64_t blocks = (rows + WARPS * rpw - 1) / (WARPS * rpw) * heads;
        auto fit = [&](int r) { return SMEM_PER_SM / ((int64_t)generic_smem(d, r, own, probs) + SMEM_BESIDE); };
        if (blocks <= std::min<int64_t>(148 * fit(rpw), 370)) return rpw == 1 && d <= 128 && blocks <= 148 * fit(SHARED_ROWS) ? SHARED_ROWS : rpw;
    }
    return 4;
}

using GenericKernel = void (*)(TrainArgs, int);
static cudaError_t launch_generic(GenericKernel kernel, dim3 grid, size_t smem, cudaStream_t stream, bool beside, const TrainArgs &a, bool vec,
                                  unsigned cluster = 1) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_clusters(kernel, grid, THREADS, smem, stream, beside, cluster, a, (int)vec);
}
// The instance for the rows per warp and the head dimension.
#define GENERIC_PICK(kernel, T, rpw, d)                                                                                                \
    ((rpw) == 4 ? ((d) <= 64 ? kernel<T, 4, 2, 1, false> : (d) <= 128 ? kernel<T, 4, 4, 1, false> : kernel<T, 4, 8, 1, false>)         \
     : (rpw) == 2 ? ((d) <= 64 ? kernel<T, 2, 2, 1, false> : (d) <= 128 ? kernel<T, 2, 4, 1, false> : kernel<T, 2, 8, 1, false>)       \
     : (rpw) == 1 ? ((d) <= 64 ? kernel<T, 1, 2, 1, false> : (d) <= 128 ? kernel<T, 1, 4, 1, false> : kernel<T, 1, 8, 1, false>)       \
                  : ((d) <= 64 ? kernel<T, 2, 2, 2, false> : kernel<T, 2, 4, 2, false>))
#define GENERIC_PICK_SHARED(kernel, T, rpw, d)                                                                                         \
    ((rpw) == 4 ? ((d) <= 64 ? kernel<T, 4, 2, 1, true> : kernel<T, 4, 4, 1, true>) : (rpw) == 2 ? ((d) <= 64 ? kernel<T, 2, 2, 1, true> : kernel<T, 2, 4, 1, true>) \
     : (rpw) == 1 ? ((d) <= 64 ? kernel<T, 1, 2, 1, true> : kernel<T, 1, 4, 1, true>) : ((d) <= 64 ? kernel<T, 2, 2, 2, true> : kernel<T, 2, 4, 2, true>))

// Blocks of the cluster that shares a block's rows, each a run of what they sweep.  Small calls wait for the chain of a block's
// tiles, and where multiprocessors have room a second block halves it.  What it costs is the meeting (3 to 5 us with the first block's
// reads), and where multiprocessors have none the other blocks' time.  So by the blocks there are and the steps of a block's sweep:
// the more blocks, the longer the sweep.  Lines drawn from 2338 calls (f32 and bf16, 32 to 128 features, 60 to 4000 keys, packed, padded, plain,
// fewer queries than keys), each timed with one, two and four blocks, backward with each pair, and tried on 875 others, against one block: forward
// mean 1.07 times as fast, 13 calls slower by more than 3 %, the worst 0.89; backward 1.09, 9, 0.85.  (By sweeps of 190 keys and 400 blocks alone:
// the same means, 130 and 37 calls, the worst 0.36 and 0.65.)  us, one block | two | four, forward: 16 queries against 4000 keys, 32 / 8
// heads of 64, bf16, 64 blocks, 168 | 97 | 69; 450 tokens, 4 heads of 128, 228 blocks, 56 | 38 | 45; 384 in two, 4 heads of 64, 192 blocks, 16.6 | 16.6 | 20.7; 154, 2 heads of 128, 40 blocks, 10 | - | 20.
// Backward (one | dq's two | dkdv's two | both): 474, 3 / 1 heads of 80, 126 | 126 | 72 | 69; 649 in two, 2 / 1 of 80, 112 | 108 | 81 | 68; but 294, 4 of 64,
// whole rows, 43 | 43 | 61 | 48, and 161 queries against 294 keys, 39 | - | 51 | 46: dkdv's alone only where the keys' sweeps are a triangle.
// (`room`: blocks that fit at once.)  Below 32 features a tile has no room for a block's sums; above 128 a head's bits do not depend on
// the others, and a rule that does not look at them would cost the calls of many heads a few per cent.
static double block_steps(const TrainArgs &a, int64_t swept, int rpw) {
    const int64_t mean = a.mask.kind == 2 ? swept / std::max(a.mask.seqs, 1) : swept;
    return (double)std::min(mean, (int64_t)a.mask.left + a.mask.right + block_rows(rpw)) / (rpw == SHARED_ROWS ? 2 * TILE : TILE);
}
static bool shareable(const TrainArgs &a) { return a.d >= 32 && a.d <= 128; }
static int64_t room_for(const TrainArgs &a, int rpw, int own, int probs) { return 148 * (SMEM_PER_SM / ((int64_t)generic_smem(a.d, rpw, own, probs) + SMEM_BESIDE)); }
static unsigned forward_cluster(const TrainArgs &a, int rpw, int64_t blocks) {
    const int64_t room = room_for(a, rpw, 1, 1);
    const double steps = block_steps(a, a.tk, rpw);
    const bool causal = a.mask.right == 0;
    if (!shareable(a)) return 1;
    if (blocks * 4 <= room && ((blocks <= 37 && steps >= 3) || (blocks <= 74 && steps >= 4))) return 4;
    if (blocks * 2 > room) return causal && blocks <= 296 && steps >= 16 ? 2 : 1;
    if (blocks > 222) return causal && rpw < 4 && blocks <= 400 && steps >= 9 ? 2 : 1;
    return steps >= (rpw == 4 ? 9 : blocks > 148 ? 3 : 2.1) ? 2 : 1;
}
static unsigned dq_cluster(const TrainArgs &a, int rpw, int64_t blocks) {
    const bool roomy = rpw < 4 && blocks * 2 <= room_for(a, rpw, 2, 1);
    return shareable(a) && blocks <= 400 && block_steps(a, a.tk, rpw) >= (blocks <= 74 ? 3 : blocks <= 148 ? 6 : blocks <= 222 && roomy ? 3 : 9) ? 2 : 1;
}
static unsigned dkdv_cluster(const TrainArgs &a, int rpw, int64_t blocks, bool dq_shared) {
    const double steps = block_steps(a, a.tq, rpw) * (a.hq / a.hkv);   // a block sweeps its whole group
    if (!shareable(a)) return 1;
    if (blocks <= 37) return steps >= 1.5 ? 2 : 1;
    const bool triangle = a.mask.right == 0 && a.tq >= a.tk;
    if (blocks <= 148 && (dq_shared || triangle) && steps >= (blocks <= 74 ? 4 : 6)) return 2;
    return dq_shared && blocks <= 400 && steps >= 48 ? 2 : 1;
}

template <typename T>
static cudaError_t forward_t(const TrainArgs &a, cudaStream_t stream, int *launches) {
    const int rpw = rows_per_warp(a.tq, (int64_t)a.hq * a.b, a.d, 1, 1), rows = block_rows(rpw);
    const bool vec = rows_readable<T>(a.q, a.d) && rows_readable<T>(a.k, a.d) && rows_readable<T>(a.v, a.d);
    const int tiles = (a.tq + rows - 1) / rows;
    const unsigned cluster = forward_cluster(a, rpw, (int64_t)tiles * a.hq * a.b);
    *launches += 1;
    return launch_generic(cluster > 1 ? GENERIC_PICK_SHARED(generic_forward_kernel, T, rpw, a.d) : GENERIC_PICK(generic_forward_kernel, T, rpw, a.d), dim3(tiles * cluster, a.hq, a.b), generic_smem(a.d, rpw, 1, 1), stream, false, a,
                          vec, cluster);
}

template <typename T>
static cudaError_t backward_t(const TrainArgs &a, cudaStream_t stream, int *launches) {
    const bool vec = rows_readable<T>(a.q, a.d) && rows_readable<T>(a.k, a.d) && rows_readable<T>(a.v, a.d) && rows_readable<T>(a.dout, a.d);
    cudaError_t e;
    {
        const int64_t rows = (int64_t)a.b * a.tq * a.hq;
        const unsigned blocks = (unsigned)((rows + THREADS / 32 - 1) / (THREADS / 32));
        *launches += 1;
        generic_delta_kernel<T><<<blocks, THREADS, 0, stream>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const int q_rpw = rows_per_warp(a.tq, (int64_t)a.hq * a.b, a.d, 2, 1), q_rows = block_rows(q_rpw), q_tiles = (a.tq + q_rows - 1) / q_rows;
    const unsigned q_cluster = dq_cluster(a, q_rpw, (int64_t)q_tiles * a.hq * a.b);
    {
        const int rpw = rows_per_warp(a.tk, (int64_t)a.hkv * a.b, a.d, 2, 2), rows = block_rows(rpw);
        const int tiles = (a.tk + rows - 1) / rows;
        const unsigned cluster = dkdv_cluster(a, rpw, (int64_t)tiles * a.hkv * a.b, q_cluster > 1);
        *launches += 1;
        e = launch_generic(cluster > 1 ? GENERIC_PICK_SHARED(generic_dkdv_kernel, T, rpw, a.d) : GENERIC_PICK(generic_dkdv_kernel, T, rpw, a.d), dim3(tiles * cluster, a.hkv, a.b), generic_smem(a.d, rpw, 2, 2), stream,
                           false, a, vec, cluster);
        if (e != cudaSuccess) return e;
    }
    {   // beside dkdv.  (dkdv itself brought in under delta's end, to wait there, made the whole twice as slow: 1000 tokens, 4 / 2
        // heads of 64 327 against 213 us.)
        *launches += 1;
        return launch_generic(q_cluster > 1 ? GENERIC_PICK_SHARED(generic_dq_kernel, T, q_rpw, a.d) : GENERIC_PICK(generic_dq_kernel, T, q_rpw, a.d), dim3(q_tiles * q_cluster, a.hq, a.b), generic_smem(a.d, q_rpw, 2, 1), stream,
                              true, a, vec, q_cluster);
    }
}

// The same for 16-bit rows of D = 64, 128 or 256 elements that can be read 16 bytes at a time: D / 8
// lanes a row (at 128: sixteen lanes a row, two rows a warp), the row's bytes of each tensor in one
// request.
template <typename T, int D>
__global__ void __launch_bounds__(THREADS) delta_rows_kernel(TrainArgs a) {
    allow_beside();   // the key and value gradients' kernel, which waits for delta where it reads it
    constexpr int LPR = D / 8, RPW = 32 / LPR;   // lanes per row, rows per warp
    const int lane = threadIdx.x & 31, sub = lane % LPR;
    const int64_t rows = (int64_t)a.b * a.tq * a.hq;
    const int64_t row = ((int64_t)blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5)) * RPW + lane / LPR;
    float sum = 0.f;
    if (row < rows) {
        const int h = (int)(row % a.hq);
        const int64_t bt = row / a.hq;
        const int64_t t = bt % a.tq, b = bt / a.tq;
        const uint4 g = *reinterpret_cast<const uint4 *>(static_cast<const T *>(a.dout.ptr) + b * a.dout.sb + t * a.dout.st + h * a.dout.sh + sub * 8);
        const uint4 o = *reinterpret_cast<const uint4 *>(static_cast<const T *>(a.o.ptr) + b * a.o.sb + t * a.o.st + h * a.o.sh + sub * 8);
        const T *gv = reinterpret_cast<const T *>(&g), *ov = reinterpret_cast<const T *>(&o);
#pragma unroll
        for (int i = 0; i < 8; ++i) sum = fmaf(Num<T>::to_f32(gv[i]), Num<T>::to_f32(ov[i]), sum);
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (row < rows && sub == 0) a.delta[row] = sum;
    end_beside();
}

// Whether every row of the view starts on a 16-byte boundary and is contiguous.
static bool rows_16b(const View4 &v) {
    return v.sd == 1 && reinterpret_cast<uintptr_t>(v.ptr) % 16 == 0 && v.sb % 8 == 0 && v.st % 8 == 0 && v.sh % 8 == 0;
}

template <typename T>
static cudaError_t delta_t(const TrainArgs &a, cudaStream_t stream, int *launches, bool beside) {
    int64_t rows = (int64_t)a.b * a.tq * a.hq;
    if (sizeof(T) == 2 && (a.d == 64 || a.d == 128 || a.d == 256) && rows_16b(a.dout) && rows_16b(a.o)) {
        const int64_t per_block = (32 / (a.d / 8)) * (THREADS / 32);
        const unsigned blocks = (unsigned)((rows + per_block - 1) / per_block);
        *launches += 1;
        return launch_beside(a.d == 64 ? delta_rows_kernel<T, 64> : a.d == 128 ? delta_rows_kernel<T, 128> : delta_rows_kernel<T, 256>,
                             dim3(blocks), THREADS, 0, stream, beside, a);
    }
    unsigned blocks = (unsigned)((rows + THREADS / 32 - 1) / (THREADS / 32));
    *launches += 1;
    return launch_beside(generic_delta_kernel<T>, dim3(blocks), THREADS, 0, stream, beside, a);
}

// delta = rowsum(dO * O) alone, for the tensor-core backward.
cudaError_t launch_generic_delta(int dtype, const TrainArgs &a, cudaStream_t stream, int *launches, bool beside) {
    switch (dtype) {
        case 0: return delta_t<float>(a, stream, launches, beside);
        case 1: return delta_t<__nv_bfloat16>(a, stream, launches, beside);
        default: return delta_t<__half>(a, stream, launches, beside);
    }
}

cudaError_t launch_generic_forward(int dtype, const TrainArgs &a, cudaStream_t stream, int *launches) {
    switch (dtype) {
        case 0: return forward_t<float>(a, stream, launches);
        case 1: return forward_t<__nv_bfloat16>(a, stream, launches);
        default: return forward_t<__half>(a, stream, launches);
    }
}

cudaError_t launch_generic_backward(int dtype, const TrainArgs &a, cudaStream_t stream, int *launches) {
    switch (dtype) {
        case 0: return backward_t<float>(a, stream, launches);
        case 1: return backward_t<__nv_bfloat16>(a, stream, launches);
        default: return backward_t<__half>(a, stream, launches);
    }
}

}  // namespace dash
