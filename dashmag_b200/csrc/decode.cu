// The decoding step against a key-value cache: split-KV (flash-decoding) and an LSE merge.
//
// The step is a single scan of the cache, so it is bound by HBM bandwidth: the algorithmic bytes
// are (visible keys) x Hkv x D x element size x 2 (keys and values).  Layout of the work:
//
//   * the visible keys [first, len) of each sequence are cut into chunks of `chunk` keys; one WARP
//     owns one (chunk, key-value head) and all the query heads of that head's group, so that a
//     cache row is read once for the whole group; warps of a block take consecutive key-value
//     heads of the same chunk, so a block streams whole contiguous cache rows;
//   * D / 8 lanes share a key: each lane copies 16 bytes of the key row and 16 bytes of the value
//     row (bf16 / f16; two 16-byte vectors each for f32) - fully coalesced 128-bit accesses - and
//     owns eight head dimensions of the output; the copies are asynchronous, into a ring of
//     shared memory private to the lane, three steps of four keys ahead of the arithmetic;
//   * scores are reduced across the D / 8 lanes with shuffles, the softmax is kept online in f32
//     per query head, lane groups are merged with shuffles at the end, and each warp writes one
//     normalised partial output and its log-sum-exp;
//     (dash_attn_decode_append_rope: the pass also rotates the queries and the new key as it reads them, where it runs on the
//     tensor cores, below: a launch less);
//   * the merge kernel combines the partials of each (sequence, query head) by their log-sum-exp
//     and rounds to the queries' dtype.  Chunks past a sequence's length or before its window are
//     never touched.
//
// With 16-bit caches and two query heads or more per key-value head the pass runs on the tensor cores
// instead (decode_split_mma_kernel below): at that much arithmetic per cache row the FMA pipe, not HBM,
// bounds the pass above.  Groups of up to eight heads with more than 512 keys need neither chunks nor merge where
// their shares are short: the blocks of a cluster take a (sequence, key-value head) together (decode_cluster says which calls).
//
// Inputs the vector path cannot read (head dimension not 64 / 128 / 256, last stride not 1, rows
// not 16-byte aligned) go through a slower scalar kernel with the same arithmetic.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "launch.h"

namespace dash {

// DASH_ATTN_DECODE_CHUNK (read once) fixes the chunk for comparison runs, whose calls are then all in chunks; 0 and less: the planner's.
long long decode_fixed_chunk() {
    static const long long fixed = [] {
        const char *env = std::getenv("DASH_ATTN_DECODE_CHUNK");
        return env ? std::atoll(env) : 0LL;
    }();
    return fixed;
}

constexpr int DEC_WARPS = 4;    // warps per block, each with its own (chunk, key-value head)
constexpr int DEC_UNROLL = 4;   // keys per group of D / 8 lanes in one step
constexpr int DEC_STAGES = 4;   // steps of the per-lane ring (16-bit dtypes; two for f32)

template <typename T>
__device__ __forceinline__ void load8(const T *p, bool valid, float (&x)[8]);

template <>
__device__ __forceinline__ void load8<float>(const float *p, bool valid, float (&x)[8]) {
    float4 a = make_float4(0, 0, 0, 0), b = a;
    if (valid) {
        a = __ldg(reinterpret_cast<const float4 *>(p));
        b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
    }
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16 *p, bool valid, float (&x)[8]) {
    uint4 r = make_uint4(0, 0, 0, 0);
    if (valid) r = __ldg(reinterpret_cast<const uint4 *>(p));
    const unsigned u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[2 * i] = __uint_as_float(u[i] << 16);
        x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
}
template <>
__device__ __forceinline__ void load8<__half>(const __half *p, bool valid, float (&x)[8]) {
    uint4 r = make_uint4(0, 0, 0, 0);
    if (valid) r = __ldg(reinterpret_cast<const uint4 *>(p));
    const unsigned u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&u[i]));
        x[2 * i] = f.x;
        x[2 * i + 1] = f.y;
    }
}

// exp for the online softmax: the accurate one for f32 inputs, the fast one for 16-bit inputs,
// whose outputs round to 8 or 11 significant bits anyway.
template <typename T> __device__ __forceinline__ float soft_exp(float x) { return __expf(x); }
template <> __device__ __forceinline__ float soft_exp<float>(float x) { return expf(x); }
template <typename T> __device__ __forceinline__ float soft_log(float x) { return __logf(x); }
template <> __device__ __forceinline__ float soft_log<float>(float x) { return logf(x); }

// ---- 16-byte asynchronous copies, global -> this lane's slots of shared memory ------------------
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid) {
    // An invalid (out of range) key copies nothing and fills its slot with zeros.
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Eight values of T from this lane's own 16-byte slots.
template <typename T>
__device__ __forceinline__ void slot8(const uint4 *slot, float (&x)[8]);
template <>
__device__ __forceinline__ void slot8<float>(const uint4 *slot, float (&x)[8]) {
    const uint4 a = slot[0], b = slot[32];
    x[0] = __uint_as_float(a.x); x[1] = __uint_as_float(a.y); x[2] = __uint_as_float(a.z); x[3] = __uint_as_float(a.w);
    x[4] = __uint_as_float(b.x); x[5] = __uint_as_float(b.y); x[6] = __uint_as_float(b.z); x[7] = __uint_as_float(b.w);
}
template <>
__device__ __forceinline__ void slot8<__nv_bfloat16>(const uint4 *slot, float (&x)[8]) {
    const uint4 r = slot[0];
    const unsigned u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[2 * i] = __uint_as_float(u[i] << 16);
        x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
}
template <>
__device__ __forceinline__ void slot8<__half>(const uint4 *slot, float (&x)[8]) {
    const uint4 r = slot[0];
    const unsigned u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&u[i]));
        x[2 * i] = f.x;
        x[2 * i + 1] = f.y;
    }
}

// One warp per (chunk, key-value head, pass over GH query heads of the group).
//
// The cache rows reach the arithmetic through a ring of shared memory that is private to each
// lane: a lane copies, with 16-byte asynchronous copies, exactly the bytes it will later read
// itself, DEC_STAGES - 1 steps ahead (a step is DEC_UNROLL keys for each group of D / 8 lanes).
// The bytes in flight therefore cost shared memory, not registers, no lane ever waits for
// another, and a multiprocessor keeps three blocks of four such warps resident: twelve warps
// with three steps each on the way from HBM.
template <typename T, int D, int GH>
__global__ void __launch_bounds__(DEC_WARPS * 32) decode_split_kernel(DecodeArgs a) {
    allow_beside();   // the merge
    constexpr int LPK = D / 8;                    // lanes per key
    constexpr int KPW = 32 / LPK;                 // keys per warp in one load
    constexpr int VPK = sizeof(T) == 4 ? 2 : 1;   // 16-byte vectors per eight values
    constexpr int SLOTS = 2 * DEC_UNROLL * VPK;   // this lane's vectors per stage: K and V of DEC_UNROLL keys
    constexpr int NS = sizeof(T) == 4 ? 2 : DEC_STAGES;
    extern __shared__ uint4 ring[];               // [warp][stage][slot][lane]
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int group = a.hq / a.hkv;
    const int passes = (group + GH - 1) / GH;
    const int b = blockIdx.y;
    long long unit = (long long)blockIdx.x * DEC_WARPS + wib;
    const int hk = (int)(unit % a.hkv);
    unit /= a.hkv;
    const int pass = (int)(unit % passes);
    const long long split = unit / passes;
    if (split >= a.splits) return;

    int first, len;
    decode_range(a, b, first, len);
    const long long c0l = (long long)first + split * a.chunk;
    if (c0l >= len) return;
    const int c0 = (int)c0l, c1 = min(len, c0 + a.chunk);

    const int sub = lane / LPK, dl = lane % LPK;
    const int g0 = pass * GH;
    float q[GH][8], acc[GH][8], m[GH], l[GH];
#pragma unroll
    for (int g = 0; g < GH; ++g) {
        const bool live = g0 + g < group;
        const int h = hk * group + min(g0 + g, group - 1);
        const T *qp = static_cast<const T *>(a.q) + (int64_t)b * a.q_sb + (int64_t)h * a.q_sh + dl * 8;
        load8<T>(qp, live, q[g]);
        m[g] = -INFINITY;
        l[g] = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[g][c] = 0.f;
    }
    const T *kbase = static_cast<const T *>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)hk * a.k.sh + dl * 8;
    const T *vbase = static_cast<const T *>(a.v.ptr) + (int64_t)b * a.v.sb + (int64_t)hk * a.v.sh + dl * 8;
    // The appending step: the row at `pos` comes from the new rows, and the warp whose chunk holds
    // it (first pass only) also writes it into the cache.
    const int pos = decode_append_at(a, b);
    const T *knew = static_cast<const T *>(a.k_new) + ((int64_t)b * a.hkv + hk) * D + dl * 8;
    const T *vnew = static_cast<const T *>(a.v_new) + ((int64_t)b * a.hkv + hk) * D + dl * 8;
    if (pos >= c0 && pos < c1 && pass == 0 && sub == 0) {
#pragma unroll
        for (int x = 0; x < VPK; ++x) {
            reinterpret_cast<uint4 *>(const_cast<T *>(kbase) + (int64_t)pos * a.k.st)[x] = reinterpret_cast<const uint4 *>(knew)[x];
            reinterpret_cast<uint4 *>(const_cast<T *>(vbase) + (int64_t)pos * a.v.st)[x] = reinterpret_cast<const uint4 *>(vnew)[x];
        }
    }

    uint4 *mine = ring + (size_t)wib * NS * SLOTS * 32 + lane;
    const uint32_t mine_u32 = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
    constexpr int STEP_KEYS = KPW * DEC_UNROLL;
    const int iters = (c1 - c0 + STEP_KEYS - 1) / STEP_KEYS;

    auto issue = [&](int it) {
        if (it < iters) {
            const uint32_t dst = mine_u32 + (uint32_t)((it % NS) * SLOTS * 32 * 16);
#pragma unroll
            for (int u = 0; u < DEC_UNROLL; ++u) {
                const int key = c0 + it * STEP_KEYS + u * KPW + sub;
                const bool valid = key < c1;
                const T *kp = key == pos ? knew : kbase + (int64_t)(valid ? key : c0) * a.k.st;
                const T *vp = key == pos ? vnew : vbase + (int64_t)(valid ? key : c0) * a.v.st;
#pragma unroll
                for (int x = 0; x < VPK; ++x) {
                    cp_async16(dst + (uint32_t)(((2 * u) * VPK + x) * 32 * 16), reinterpret_cast<const char *>(kp) + 16 * x, valid);
                    cp_async16(dst + (uint32_t)(((2 * u + 1) * VPK + x) * 32 * 16), reinterpret_cast<const char *>(vp) + 16 * x, valid);
                }
            }
        }
        cp_async_commit();  // always, so that the group count stays in step with the iterations
    };

#pragma unroll
    for (int s = 0; s < NS - 1; ++s) issue(s);
    for (int it = 0; it < iters; ++it) {
        issue(it + NS - 1);
        cp_async_wait<NS - 1>();
        const uint4 *stage = mine + (size_t)(it % NS) * SLOTS * 32;
        const int key0 = c0 + it * STEP_KEYS + sub;
        float s[GH][DEC_UNROLL];
#pragma unroll
        for (int u = 0; u < DEC_UNROLL; ++u) {
            float kx[8];
            slot8<T>(stage + (2 * u) * VPK * 32, kx);
            const bool valid = key0 + u * KPW < c1;
#pragma unroll
            for (int g = 0; g < GH; ++g) {
                float d = 0.f;
#pragma unroll
                for (int c = 0; c < 8; ++c) d = fmaf(q[g][c], kx[c], d);
#pragma unroll
                for (int o = LPK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                s[g][u] = valid ? d * a.scale : -INFINITY;
            }
        }
        float corr[GH];
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            float mx = s[g][0];
#pragma unroll
            for (int u = 1; u < DEC_UNROLL; ++u) mx = fmaxf(mx, s[g][u]);
            const float mn = fmaxf(m[g], mx);
            const float base = mn == -INFINITY ? 0.f : mn;   // nothing seen yet: exponentiate against 0
            corr[g] = soft_exp<T>(m[g] - base);
            float sum = 0.f;
#pragma unroll
            for (int u = 0; u < DEC_UNROLL; ++u) {
                s[g][u] = soft_exp<T>(s[g][u] - base);
                sum += s[g][u];
            }
            l[g] = l[g] * corr[g] + sum;
            m[g] = mn;
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[g][c] *= corr[g];
        }
#pragma unroll
        for (int u = 0; u < DEC_UNROLL; ++u) {
            float vx[8];
            slot8<T>(stage + (2 * u + 1) * VPK * 32, vx);
#pragma unroll
            for (int g = 0; g < GH; ++g)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[g][c] = fmaf(s[g][u], vx[c], acc[g][c]);
        }
    }

    // Merge the lane groups (each saw different keys).
#pragma unroll
    for (int g = 0; g < GH; ++g) {
#pragma unroll
        for (int o = LPK; o < 32; o <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, m[g], o);
            const float lo = __shfl_xor_sync(0xffffffffu, l[g], o);
            const float mn = fmaxf(m[g], mo);
            const float wa = mn == -INFINITY ? 0.f : soft_exp<T>(m[g] - mn);
            const float wb = mn == -INFINITY ? 0.f : soft_exp<T>(mo - mn);
            l[g] = l[g] * wa + lo * wb;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float ao = __shfl_xor_sync(0xffffffffu, acc[g][c], o);
                acc[g][c] = acc[g][c] * wa + ao * wb;
            }
            m[g] = mn;
        }
        if (sub == 0 && g0 + g < group) {
            const int h = hk * group + g0 + g;
            const float inv = l[g] > 0.f ? 1.f / l[g] : 0.f;
            float *po = a.part_o + (((int64_t)b * a.hq + h) * a.splits + split) * D + dl * 8;
            reinterpret_cast<float4 *>(po)[0] = make_float4(acc[g][0] * inv, acc[g][1] * inv, acc[g][2] * inv, acc[g][3] * inv);
            reinterpret_cast<float4 *>(po)[1] = make_float4(acc[g][4] * inv, acc[g][5] * inv, acc[g][6] * inv, acc[g][7] * inv);
            if (dl == 0) a.part_lse[((int64_t)b * a.hq + h) * a.splits + split] = l[g] > 0.f ? m[g] + soft_log<T>(l[g]) : -INFINITY;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The split pass on the tensor cores (16-bit cache, head dimension 64, 128 or 256, groups of two heads or more)
// ---------------------------------------------------------------------------------------------
// With several query heads to a key-value head the scalar pass spends its time on FMA issue,
// not on HBM: a cache row of 512 bytes feeds 2048 multiply-adds.  Here warp-level MMAs (m16n8k16) do the products.  Groups of up to
// eight heads are the N dimension of the transposed products, S^T = K Q^T with the 16 keys of a tile as M, then O^T += V^T P^T
// with the features as M: half the MMAs, half the exponentials and half the accumulators of rows of sixteen heads, most of them
// not there.  (D 128, a group of four: 24 MMAs a tile and not 48.)  Larger groups (WIDE) are the M dimension, S = Q K^T with the
// 16 keys as two N tiles, then O += P V with P taken straight from the accumulator registers of S as the A operand: two column
// tiles of eight heads in the other form measured slower by a tenth, its 8 x 8 transposes and its maxima over eight lanes cost more.
// In chunks both forms sum in one order, so that a head's bits do not depend on how many others share its key-value head; that costs
// the narrow one at most 2 % (16 of 200 keys, 16 / 4 heads of 128, split and merge, 7.8 -> 7.9 us; with sixteen rows 8.6).
// One warp per (share of the keys, key-value head), with a ring of its own in shared memory: every lane copies 16-byte pieces of
// the tile's 16 key rows and 16 value rows asynchronously, two tiles ahead, into rows (256 bytes at D = 128) whose 16-byte chunks
// are XOR-swizzled by the row, and ldmatrix reads the fragments from there without bank conflicts (transposed for V).  What a warp
// waits for in a tile is its own chain, not memory (six stages for three change nothing, 0.8 us a tile where four warps are
// alone on a multiprocessor): all fragments are fetched in front of the products, V's under the softmax, no product follows
// the one it depends on, and a tile's copies go out from running addresses (0.5 us).  Split and merge, against
// heads as rows with each fragment fetched where it is used: 16 of 200 keys, 16 / 4 heads of 128, 9.0 -> 7.9 us, 64 of up to 16384, 32 / 8 of 64, 176 -> 166;
// groups of sixteen, 40 sequences of 20000, 56.2 -> 53.8.
//
// CLUSTER: the blocks of a cluster take one (sequence, key-value head) together, its tiles dealt evenly over their warps by the
// length the sequence really has, and meet in distributed shared memory: each block merges its warps' sums, hands every block of
// the cluster the outputs that block finishes, and finishes its own.  No partials in HBM, no merge kernel behind the pass (3.3 us
// of an 8 us step), no chunks past the lengths (figures at decode_cluster).
constexpr int DM_STAGES = 3;    // tiles of the per-warp ring
constexpr int DM_KEYS = 16;     // keys per tile

// The 8 x 8 matrix of 16-bit values held two a lane (row lane / 4, columns 2 (lane % 4), + 1), transposed.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}

template <typename T> struct MmaType;
template <> struct MmaType<__nv_bfloat16> {
    static constexpr bool NARROW = false;   // of exponents
    using Two = __nv_bfloat162;
    static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t *>(&v);
    }
    static __device__ __forceinline__ float lo(uint32_t u) { return __uint_as_float(u << 16); }
    static __device__ __forceinline__ float hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
};
template <> struct MmaType<__half> {
    static constexpr bool NARROW = true;
    using Two = __half2;
    static __device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t *>(&v);
    }
    static __device__ __forceinline__ float lo(uint32_t u) { return __low2float(*reinterpret_cast<const __half2 *>(&u)); }
    static __device__ __forceinline__ float hi(uint32_t u) { return __high2float(*reinterpret_cast<const __half2 *>(&u)); }
};
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// PARTS = 2 (head dimension 256): two neighbouring warps share a unit, each with D = 128 of the 256
// features - its half of the scores' sum over the features, which the two exchange through shared
// memory and add (in one order, so both hold the same bits), its half of Q, of every K and V row
// and of the output; the accumulators of a whole row of 256 would not fit a thread's registers.
//
// WARPS warps to a block: eight, or two where blocks of eight would leave multiprocessors without one (a block is a
// multiprocessor's worth of shared memory: 256 units of one sequence's 8 heads in blocks of eight are 32 blocks).  The warps
// resident at a time are the same.  Blocks of two up to sixteen warps a multiprocessor (at D 128 two waves of them, at D 64
// one), where they measured ahead (us, eight | two): one sequence of 300 keys with rotation and append, 12.2 | 10.1; 16 of up to 500, 16 / 4 heads,
// 10.2 | 8.8; 56 of up to 5136 with one head, 26.3 | 22.0; but 34 of up to 7657, 16 heads on one, 22.9 | 24.2, for which no rule was found.  Beyond,
// eight: its warps read neighbouring heads of the same keys at the same time (20 sequences of up to 8192, 32 / 2 heads, 23.0 | 26.1; 16 of up to 20000, 16
// on one, 22.0 | 24.1).  With heads as columns groups of four are ahead in twos there as well (64 of up to 4096, 8 heads, 92.3 | 88.4): the line
// was drawn before that.
//
// Two columns rotated in the dtype's own arithmetic, as rope_kernel does it (each product and the sum rounded once): `low` for
// the first half of the rotated features, whose partner enters with its sign turned.
template <typename T>
__device__ __forceinline__ uint32_t rotate_two(uint32_t x, uint32_t partner, uint32_t c, uint32_t s, bool low) {
    using P2 = typename MmaType<T>::Two;
    const P2 px = *reinterpret_cast<P2 *>(&x), pp = *reinterpret_cast<P2 *>(&partner), pc = *reinterpret_cast<P2 *>(&c), ps = *reinterpret_cast<P2 *>(&s);
    P2 r = __hadd2_rn(__hmul2_rn(px, pc), __hmul2_rn(low ? __hneg2(pp) : pp, ps));
    return *reinterpret_cast<uint32_t *>(&r);
}

// ---- the blocks of a cluster -------------------------------------------------------------------
constexpr int MAX_CLUSTER = 16, CLUSTER_WARPS = 4;
__device__ __forceinline__ uint32_t cluster_blocks() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// To the place that `mine` is in this block, in block `rank`.
__device__ __forceinline__ uint32_t cluster_address(const void *mine, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(mine))), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(void *mine, int rank, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_address(mine, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void cluster_store(void *mine, int rank, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(cluster_address(mine, rank)), "f"(v.x), "f"(v.y) : "memory");
}

template <typename T, int D, int PARTS, bool WIDE, int WARPS, bool ROPE, bool CLUSTER>
__global__ void __launch_bounds__(WARPS * 32) decode_split_mma_kernel(DecodeArgs a) {
    constexpr int DM_WARPS = WARPS;
    if constexpr (!CLUSTER) allow_beside();   // the merge
    constexpr int DFULL = D * PARTS;            // the head dimension; D is what one warp takes of it
    constexpr int ROWB = 2 * D;                 // bytes of a warp's part of a cache row: 256 at D = 128, 128 at D = 64
    constexpr int CH = D / 8;                   // its 16-byte chunks
    constexpr int DM_TILE = DM_KEYS * ROWB;     // bytes of a K (or V) tile of 16 rows
    extern __shared__ __align__(128) uint8_t dm_ring[];   // [warp][stage][K tile | V tile], then the warps' score exchange
    float *dm_exchange = reinterpret_cast<float *>(dm_ring + (size_t)DM_WARPS * DM_STAGES * 2 * DM_KEYS * ROWB);   // [warp][lane][8]
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int group = a.hq / a.hkv;
    const int b = blockIdx.y;
    const int csize = CLUSTER ? (int)cluster_blocks() : 1, crank = CLUSTER ? (int)cluster_rank() : 0;
    if constexpr (CLUSTER) cluster_arrive();   // (every block of the cluster runs before the first one's memory is written to)
    const long long unit = CLUSTER ? blockIdx.x / csize : ((long long)blockIdx.x * DM_WARPS + wib) / PARTS;
    const int part = wib % PARTS, d0 = part * D;   // this warp's features [d0, d0 + D)
    // A unit: eight query heads of a group, or sixteen (WIDE; a group of more takes several
    // units side by side, whose warps read the same chunk of the cache at the same time: once from
    // HBM, the rest from L2), a key-value head, a chunk.
    constexpr int HEADS = WIDE ? 16 : 8;
    static_assert(!(WIDE && CLUSTER), "sixteen heads meet in the merge");
    const int hblocks = (group + HEADS - 1) / HEADS;
    const int g_base = (int)(unit % hblocks) * HEADS;
    const int hk = (int)((unit / hblocks) % a.hkv);
    const long long split = CLUSTER ? 0 : unit / hblocks / a.hkv;
    if (!CLUSTER && split >= a.splits) return;
    int first, len;
    decode_range(a, b, first, len);
    int c0, c1;
    if constexpr (CLUSTER) {
        // The tiles of what the sequence really sees, dealt evenly over the cluster's warps in order; some may get none.
        constexpr int PER = DM_WARPS / PARTS;
        const int tiles = (max(len - first, 0) + DM_KEYS - 1) / DM_KEYS, shares = csize * PER, mine = crank * PER + wib / PARTS;
        c0 = first + (int)((long long)tiles * mine / shares) * DM_KEYS;
        c1 = min(len, first + (int)((long long)tiles * (mine + 1) / shares) * DM_KEYS);
    } else {
        const long long c0l = (long long)first + split * a.chunk;
        if (c0l >= len) return;
        c0 = (int)c0l;
        c1 = min(len, c0 + a.chunk);
    }
    const int iters = max(c1 - c0 + DM_KEYS - 1, 0) / DM_KEYS;

    const T *kbase = static_cast<const T *>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)hk * a.k.sh + d0;
    const T *vbase = static_cast<const T *>(a.v.ptr) + (int64_t)b * a.v.sb + (int64_t)hk * a.v.sh + d0;
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(dm_ring)) + (uint32_t)wib * DM_STAGES * 2 * DM_TILE;

    // This lane's pieces of a tile: chunk (lane % 16) of rows (lane / 16) + 2 j.
    const int cp_chunk = lane % CH, cp_row0 = lane / CH;
    constexpr int RPP = 32 / CH;                // rows the warp copies per pass
    // The appending step: the row at `pos` comes from the new rows, and the warp whose chunk holds it also writes it into the
    // cache, below.
    const int pos = decode_append_at(a, b);
    const T *knew = static_cast<const T *>(a.k_new) + ((int64_t)b * a.hkv + hk) * DFULL + d0;
    const T *vnew = static_cast<const T *>(a.v_new) + ((int64_t)b * a.hkv + hk) * DFULL + d0;
    const int pos_it = (pos >= c0 && pos < c1) ? (pos - c0) / DM_KEYS : -1;   // the tile of the new row, if this chunk holds it
    // (The rows of a lane differ from its first by whole multiples of a power of two above it, so their swizzles by one exclusive or.)
    const uint32_t to0 = ring + (uint32_t)(cp_row0 * ROWB), sw0 = (uint32_t)((cp_chunk ^ cp_row0) << 4);
    const int64_t k_hop = RPP * a.k.st, v_hop = RPP * a.v.st;
    auto issue = [&](int it) {
        if (it < iters) {
            const uint32_t dst = to0 + (uint32_t)(it % DM_STAGES) * 2 * DM_TILE;
            const int key0 = c0 + it * DM_KEYS + cp_row0;
            const T *kp = kbase + (int64_t)key0 * a.k.st + cp_chunk * 8, *vp = vbase + (int64_t)key0 * a.v.st + cp_chunk * 8;
            if (c0 + (it + 1) * DM_KEYS <= c1 && it != pos_it) {
#pragma unroll
                for (int j = 0; j < DM_KEYS / RPP; ++j) {
                    const uint32_t at = dst + (uint32_t)(RPP * j * ROWB) + (sw0 ^ (uint32_t)(((RPP * j) & 7) << 4));
                    cp_async16(at, kp);
                    cp_async16(at + DM_TILE, vp);
                    kp += k_hop;
                    vp += v_hop;
                }
            } else {   // keys past the last are zeros; the new row comes from where it was given
#pragma unroll
                for (int j = 0; j < DM_KEYS / RPP; ++j) {
                    const int key = key0 + RPP * j;
                    const bool valid = key < c1, fresh = key == pos;
                    const uint32_t at = dst + (uint32_t)(RPP * j * ROWB) + (sw0 ^ (uint32_t)(((RPP * j) & 7) << 4));
                    cp_async16(at, fresh ? knew + cp_chunk * 8 : valid ? kp + j * k_hop : kbase + (int64_t)c0 * a.k.st, valid);
                    cp_async16(at + DM_TILE, fresh ? vnew + cp_chunk * 8 : valid ? vp + j * v_hop : vbase + (int64_t)c0 * a.v.st, valid);
                }
            }
        }
        cp_async_commit();  // always, so that the group count stays in step with the tiles
    };

    const int g = lane >> 2, t = lane & 3;   // fragment coordinates
    // Q as the operand of every score MMA.  Eight heads: the B operand, per k-step features 16 ks + 2 t, + 1 and those eight further
    // on of head g.  Sixteen: the A operand [16 heads x 16 d], the same of heads g and g + 8.  Heads past the group are zero.
    uint32_t qa[D / 16][WIDE ? 4 : 2];
    const T *qg = static_cast<const T *>(a.q) + (int64_t)b * a.q_sb + (int64_t)(hk * group) * a.q_sh;
    constexpr int QH = WIDE ? 2 : 1;   // heads a lane holds: g, and g + 8
#pragma unroll
    for (int x = 0; x < QH; ++x) {
        const int head = g_base + g + 8 * x;
        const T *row = qg + (int64_t)min(head, group - 1) * a.q_sh + d0 + 2 * t;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
            for (int j = 0; j < 2; ++j) qa[ks][j * QH + x] = head < group ? *reinterpret_cast<const uint32_t *>(row + ks * 16 + 8 * j) : 0u;
    }
    // The first tiles are on their way before the rotation's tables are asked for: that trip to memory falls under theirs.
#pragma unroll
    for (int s = 0; s < DM_STAGES - 1; ++s) issue(s);
    // The rotation's row of the tables (no such row: every rotated feature is a NaN, as rope_kernel has it).
    const int half = a.rope_dim / 2;
    const T *cos_row = nullptr, *sin_row = nullptr;
    if constexpr (ROPE) {
        const int64_t at = a.rope_pos_bytes == 8 ? static_cast<const long long *>(a.rope_pos)[b] : static_cast<const int *>(a.rope_pos)[b];
        if (at >= 0 && at < a.rope_len) {
            cos_row = static_cast<const T *>(a.rope_cos) + at * a.rope_dim;
            sin_row = static_cast<const T *>(a.rope_sin) + at * a.rope_dim;
        }
#pragma unroll
        for (int x = 0; x < QH; ++x) {
            const int head = g_base + g + 8 * x;
            const T *row = qg + (int64_t)min(head, group - 1) * a.q_sh;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int c = d0 + ks * 16 + 8 * j + 2 * t;
                    if (c >= a.rope_dim || head >= group) continue;
                    const bool low = c < half;
                    const int other = low ? c + half : c - half;
                    uint32_t &q2 = qa[ks][j * QH + x];
                    q2 = cos_row ? rotate_two<T>(q2, *reinterpret_cast<const uint32_t *>(row + other), *reinterpret_cast<const uint32_t *>(cos_row + c),
                                                 *reinterpret_cast<const uint32_t *>(sin_row + c), low)
                                 : 0x7fff7fffu;   // a NaN in either dtype
                }
        }
    }
    // (D / 8 lanes the new key row, D / 8 the value row.)
    uint4 row_chunk = make_uint4(0, 0, 0, 0);   // lanes below CH: this lane's chunk of the new key row, rotated if the step rotates
    if (pos >= c0 && pos < c1 && lane < 2 * CH) {
        row_chunk = *reinterpret_cast<const uint4 *>((lane < CH ? knew : vnew) + cp_chunk * 8);
        const int c = d0 + cp_chunk * 8;
        if (ROPE && lane < CH && c < a.rope_dim) {
            const bool low = c < half;
            if (cos_row) {
                const uint4 o4 = *reinterpret_cast<const uint4 *>(knew - d0 + (low ? c + half : c - half));
                const uint4 cs = *reinterpret_cast<const uint4 *>(cos_row + c), sn = *reinterpret_cast<const uint4 *>(sin_row + c);
                row_chunk = make_uint4(rotate_two<T>(row_chunk.x, o4.x, cs.x, sn.x, low), rotate_two<T>(row_chunk.y, o4.y, cs.y, sn.y, low),
                                       rotate_two<T>(row_chunk.z, o4.z, cs.z, sn.z, low), rotate_two<T>(row_chunk.w, o4.w, cs.w, sn.w, low));
            } else {
                row_chunk = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
            }
        }
        if (g_base == 0) {
            T *dst = const_cast<T *>(lane < CH ? kbase + (int64_t)pos * a.k.st : vbase + (int64_t)pos * a.v.st) + cp_chunk * 8;
            *reinterpret_cast<uint4 *>(dst) = row_chunk;
        }
    }
    const float sl = a.scale * 1.4426950408889634f;   // scores are exponentiated in base 2
    // From one maximum to another, in clusters: the difference of the two offsets as the exponentials used them, each product rounded on
    // its own, so that what was summed against either shares one reference.
    auto between = [sl](float from, float to) { return exp2f(__fsub_rn(__fmul_rn(from, sl), __fmul_rn(to, sl))); };
    // The accumulator: eight heads have it transposed (rows are features, columns heads), sixteen as rows of heads.
    constexpr int ON = WIDE ? D / 8 : D / 16;
    float o[ON][4];
#pragma unroll
    for (int n = 0; n < ON; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    // This lane's two heads (2 t and 2 t + 1; of sixteen: g and g + 8); l is the lane's share of their sums.
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    // ldmatrix rows: lane -> (matrix lane / 8, row lane % 8)
    const int lm = lane >> 3, lr = lane & 7;

    for (int it = 0; it < iters; ++it) {
        __syncwarp();   // every lane is done with the stage about to be refilled
        issue(it + DM_STAGES - 1);
        cp_async_wait<DM_STAGES - 1>();
        __syncwarp();   // ... and sees the other lanes' pieces of this tile
        const uint32_t kt = ring + (uint32_t)(it % DM_STAGES) * 2 * DM_TILE, vt = kt + DM_TILE;
        const int key0 = c0 + it * DM_KEYS;
        if (ROPE && it == pos_it) {   // the new key arrived as it was given: the rotated row takes its place in the tile
            const int row = pos - key0;
            if (lane < CH) asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(kt + (uint32_t)(row * ROWB + ((cp_chunk ^ (row & 7)) << 4))),
                                        "r"(row_chunk.x), "r"(row_chunk.y), "r"(row_chunk.z), "r"(row_chunk.w) : "memory");
            __syncwarp();
        }

        float sc[WIDE ? 2 : 1][4] = {};
        uint32_t kf[D / 16][4], vf[D / 16][4];   // the tile's fragments
        if constexpr (WIDE) {
            // S[16 heads x 16 keys] as two N tiles of 8 keys.
#pragma unroll
            for (int ks = 0; ks < D / 16; ks += 2)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {   // b0, b1 of k-step ks, then of ks + 1
                    const int row = nt * 8 + lr;
                    ldmatrix_x4(kt + (uint32_t)(row * ROWB + (((2 * ks + lm) ^ (row & 7)) << 4)), kf[ks + nt]);
                }
#pragma unroll
            for (int ks = 0; ks < D / 16; ks += 2)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) MmaType<T>::mma(sc[nt], qa[ks + j], kf[ks + nt][2 * j], kf[ks + nt][2 * j + 1]);
        } else {
            // S transposed, [16 keys x 8 heads]; in clusters the even and the odd k-steps as two chains, in chunks one, as sixteen heads have it.
            float odd[4] = {};
            auto &second = CLUSTER ? odd : sc[0];
            const int row = (lm & 1) * 8 + lr;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)   // keys 0-7 and 8-15 of the k-step's first eight features, then of the others
                ldmatrix_x4(kt + (uint32_t)(row * ROWB + (((2 * ks + (lm >> 1)) ^ (row & 7)) << 4)), kf[ks]);
#pragma unroll
            for (int ks = 0; ks < D / 16; ks += 2) {
                MmaType<T>::mma(sc[0], kf[ks], qa[ks][0], qa[ks][1]);
                MmaType<T>::mma(second, kf[ks + 1], qa[ks + 1][0], qa[ks + 1][1]);
            }
            if constexpr (CLUSTER) {
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[0][e] += odd[e];
            }
        }
        // V's fragments are fetched under the softmax.
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
            if constexpr (WIDE) {   // b0, b1 of eight features, then of the next eight
                const int row = (lm & 1) * 8 + lr, chunk = 2 * n + (lm >> 1);
                ldmatrix_x4_trans(vt + (uint32_t)(row * ROWB + ((chunk ^ (row & 7)) << 4)), vf[n]);
            } else {                // features 0-7 and 8-15 of keys 0-7, then of keys 8-15
                const int row = (lm >> 1) * 8 + lr, chunk = 2 * n + (lm & 1);
                ldmatrix_x4_trans(vt + (uint32_t)(row * ROWB + ((chunk ^ (row & 7)) << 4)), vf[n]);
            }
        }
        if constexpr (PARTS == 2) {
            // The other half of the sum over the features is the neighbouring warp's: both write theirs, meet,
            // and add part 0's and part 1's in that order.
            constexpr int SN = WIDE ? 2 : 1;
            float *mine = dm_exchange + ((size_t)wib * 32 + lane) * 4 * SN, *other = dm_exchange + ((size_t)(wib ^ 1) * 32 + lane) * 4 * SN;
#pragma unroll
            for (int nt = 0; nt < SN; ++nt)
                *reinterpret_cast<float4 *>(mine + 4 * nt) = make_float4(sc[nt][0], sc[nt][1], sc[nt][2], sc[nt][3]);
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (wib >> 1)) : "memory");
#pragma unroll
            for (int nt = 0; nt < SN; ++nt) {
                const float4 o4 = *reinterpret_cast<const float4 *>(other + 4 * nt);
                const float theirs[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[nt][e] = part == 0 ? sc[nt][e] + theirs[e] : theirs[e] + sc[nt][e];
            }
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (wib >> 1)) : "memory");   // both have read before the next tile's are written
        }
        // Online softmax.  P goes to the tensor cores as the sum of two 16-bit values (what the rounding of the first
        // loses is the second), so that the products keep the f32 accuracy of the scalar pass.
        if constexpr (WIDE) {
            // Rows g (values 0, 1 of a tile) and g + 8 (values 2, 3); a tile's columns are keys key0 + 8 nt + 2 t + {0, 1}.
            if (key0 + DM_KEYS > c1) {
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (key0 + nt * 8 + 2 * t + (j & 1) >= c1) sc[nt][j] = -INFINITY;
            }
            uint32_t pa[4], pl[4];
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                float mx = fmaxf(fmaxf(sc[0][2 * rr], sc[0][2 * rr + 1]), fmaxf(sc[1][2 * rr], sc[1][2 * rr + 1]));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const float mn = fmaxf(m[rr], mx);
                if (__any_sync(0xffffffffu, mn > m[rr])) {
                    // The row's maximum grew (in some row of the warp): bring the sum and the accumulator along.
                    const float corr = mn == -INFINITY ? 1.f : exp2f((m[rr] - mn) * sl);   // exp2(-inf) = 0 for a first maximum
                    l[rr] *= corr;
#pragma unroll
                    for (int n = 0; n < ON; ++n) { o[n][2 * rr] *= corr; o[n][2 * rr + 1] *= corr; }
                    m[rr] = mn;
                }
                const float base = m[rr] == -INFINITY ? 0.f : __fmul_rn(m[rr], sl);
                const float p00 = exp2f(fmaf(sc[0][2 * rr], sl, -base)), p01 = exp2f(fmaf(sc[0][2 * rr + 1], sl, -base));
                const float p10 = exp2f(fmaf(sc[1][2 * rr], sl, -base)), p11 = exp2f(fmaf(sc[1][2 * rr + 1], sl, -base));
                l[rr] += (p00 + p01) + (p10 + p11);
                pa[rr] = MmaType<T>::pack(p00, p01);       // a0 / a1: keys 2t, 2t + 1
                pa[2 + rr] = MmaType<T>::pack(p10, p11);   // a2 / a3: keys 8 + 2t, 8 + 2t + 1
                pl[rr] = MmaType<T>::pack(p00 - MmaType<T>::lo(pa[rr]), p01 - MmaType<T>::hi(pa[rr]));
                pl[2 + rr] = MmaType<T>::pack(p10 - MmaType<T>::lo(pa[2 + rr]), p11 - MmaType<T>::hi(pa[2 + rr]));
            }
            // O[16 heads x D] += P[16 x 16 keys] V[16 keys x D]: one part of P over all features, then the other, so that no
            // product waits for the one before it.
#pragma unroll
            for (int n = 0; n < ON; ++n) MmaType<T>::mma(o[n], pa, vf[n / 2][2 * (n & 1)], vf[n / 2][2 * (n & 1) + 1]);
#pragma unroll
            for (int n = 0; n < ON; ++n) MmaType<T>::mma(o[n], pl, vf[n / 2][2 * (n & 1)], vf[n / 2][2 * (n & 1) + 1]);
        } else {
            // Heads 2 t (values 0 and 2: keys g and g + 8) and 2 t + 1 (values 1 and 3).
            if (key0 + DM_KEYS > c1) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (key0 + g + 8 * (j >> 1) >= c1) sc[0][j] = -INFINITY;
            }
            // A maximum moves in few tiles once some have been seen: a vote says whether one does in this, and only then the
            // lanes tell one another theirs and bring the sums and the accumulator along.
            const float mx0 = fmaxf(sc[0][0], sc[0][2]), mx1 = fmaxf(sc[0][1], sc[0][3]);
            if (__any_sync(0xffffffffu, mx0 > m[0] || mx1 > m[1])) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float mx = e == 0 ? mx0 : mx1;
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    const float mn = fmaxf(m[e], mx);
                    const float corr = mn == -INFINITY ? 1.f : CLUSTER ? between(m[e], mn) : exp2f((m[e] - mn) * sl);   // exp2(-inf) = 0 for a first maximum
                    l[e] *= corr;
#pragma unroll
                    for (int n = 0; n < ON; ++n) { o[n][e] *= corr; o[n][2 + e] *= corr; }
                    m[e] = mn;
                }
            }
            float p[4];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float base = m[e] == -INFINITY ? 0.f : __fmul_rn(m[e], sl);
                p[e] = exp2f(fmaf(sc[0][e], sl, -base));
                p[2 + e] = exp2f(fmaf(sc[0][2 + e], sl, -base));
            }
            // The lane's share of the sums: in clusters its own two keys; in chunks those of its pair of lanes (keys g and g ^ 1, then the two
            // eight further on), which is what a lane has of sixteen heads' rows: the sums are the same to the bit.
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if constexpr (CLUSTER) l[e] += p[e] + p[2 + e];
                else l[e] += (p[e] + __shfl_xor_sync(0xffffffffu, p[e], 4)) + (p[2 + e] + __shfl_xor_sync(0xffffffffu, p[2 + e], 4));
            }
            // A chunk's largest probability is 1 and has no error, and it is much of the chunk's sum; a cluster's shares go against one
            // maximum at the end and have fewer of them, and at bf16 a third part of P makes up for it, and more (8 of 2000 keys, 32 / 8 heads of
            // 128, error against f64 where the output is next to nothing: 6.3e-8 in chunks, 6.9e-8 with two parts, 2.4e-8 with three; under a window of 4096
            // keys, shares of 512, 5.3e-8, 5.8e-8, 3.2e-8).
            constexpr bool THIRD = CLUSTER && !MmaType<T>::NARROW;
            uint32_t pa[2], pl[2], pm[2];   // an 8 x 8 transpose each makes the accumulator's layout the B operand's
#pragma unroll
            for (int j = 0; j < 2; ++j) {   // keys 0 to 7 of the tile, then 8 to 15
                const uint32_t hi = MmaType<T>::pack(p[2 * j], p[2 * j + 1]);
                const float r0 = p[2 * j] - MmaType<T>::lo(hi), r1 = p[2 * j + 1] - MmaType<T>::hi(hi);
                const uint32_t low = MmaType<T>::pack(r0, r1);
                pa[j] = transpose_8x8(hi);
                pl[j] = transpose_8x8(low);
                if constexpr (THIRD) pm[j] = transpose_8x8(MmaType<T>::pack(r0 - MmaType<T>::lo(low), r1 - MmaType<T>::hi(low)));
            }
            // O[D x 8 heads] += V^T[D x 16 keys] P^T[16 keys x 8 heads]
#pragma unroll
            for (int n = 0; n < ON; ++n) MmaType<T>::mma(o[n], vf[n], pa[0], pa[1]);
#pragma unroll
            for (int n = 0; n < ON; ++n) MmaType<T>::mma(o[n], vf[n], pl[0], pl[1]);
            if constexpr (THIRD) {
#pragma unroll
                for (int n = 0; n < ON; ++n) MmaType<T>::mma(o[n], vf[n], pm[0], pm[1]);
            }
        }
    }
    cp_async_wait<0>();
    // Each head's sum over the lanes that share it.
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int x = WIDE ? 1 : CLUSTER ? 4 : 8; x < (WIDE ? 4 : 32); x *= 2) l[e] += __shfl_xor_sync(0xffffffffu, l[e], x);

    if constexpr (CLUSTER) {
        constexpr int PER = DM_WARPS / PARTS;
        float *const wide = reinterpret_cast<float *>(dm_ring);   // the warps' rings, from here on [PER][HEADS][DFULL]
        float *const box = dm_exchange + (PARTS == 2 ? (size_t)DM_WARPS * 32 * 4 : 0);   // [block][this block's outputs], HEADS DFULL floats and a piece a block
        float *const meets = box + HEADS * DFULL + 4 * MAX_CLUSTER;  // [block][HEADS][maximum, sum]
        float *const own = meets + MAX_CLUSTER * 2 * HEADS;         // [warp of PER][HEADS][maximum, sum]
        const int rows = min(HEADS, group - g_base), quads = rows * DFULL / 4;   // 16-byte pieces of the unit's output
        __syncthreads();   // nobody's ring is read any more
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int row = 2 * t + e;
            if (row < rows) {
                float *po = wide + ((size_t)(wib / PARTS) * HEADS + row) * DFULL + d0 + g;
#pragma unroll
                for (int n = 0; n < ON; ++n) {
                    po[n * 16] = o[n][e];
                    po[n * 16 + 8] = o[n][2 + e];
                }
                if (g == 0 && part == 0) *reinterpret_cast<float2 *>(own + ((wib / PARTS) * HEADS + row) * 2) = make_float2(m[e], l[e]);
            }
        }
        __syncthreads();
        // A part's weight against the maximum of all: where that is -inf nothing was seen (or nothing but NaN), and what is there
        // is kept as it is.
        auto weight = [&](float mine, float top) { return top == -INFINITY ? 1.f : between(mine, top); };
        cluster_wait();
        const int share = (quads + csize - 1) / csize;   // pieces a block finishes
        for (int i = threadIdx.x; i < quads; i += DM_WARPS * 32) {
            const int row = i / (DFULL / 4);
            float top = -INFINITY;
#pragma unroll
            for (int w = 0; w < PER; ++w) top = fmaxf(top, own[(w * HEADS + row) * 2]);
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < PER; ++w) {
                const float wt = weight(own[(w * HEADS + row) * 2], top);
                const float4 x = reinterpret_cast<const float4 *>(wide + (size_t)w * HEADS * DFULL)[i];
                sum.x = fmaf(wt, x.x, sum.x);
                sum.y = fmaf(wt, x.y, sum.y);
                sum.z = fmaf(wt, x.z, sum.z);
                sum.w = fmaf(wt, x.w, sum.w);
            }
            cluster_store(box + ((size_t)crank * share + i % share) * 4, i / share, sum);
        }
        for (int i = threadIdx.x; i < rows * csize; i += DM_WARPS * 32) {
            const int row = i % rows, to = i / rows;
            float top = -INFINITY, all = 0.f;
#pragma unroll
            for (int w = 0; w < PER; ++w) top = fmaxf(top, own[(w * HEADS + row) * 2]);
#pragma unroll
            for (int w = 0; w < PER; ++w) all = fmaf(weight(own[(w * HEADS + row) * 2], top), own[(w * HEADS + row) * 2 + 1], all);
            cluster_store(meets + (crank * HEADS + row) * 2, to, make_float2(top, all));
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        const int at = crank * share + (int)threadIdx.x;
        for (int i = at; i < min(quads, (crank + 1) * share); i += DM_WARPS * 32) {
            const int row = i / (DFULL / 4);
            float top = -INFINITY;
            for (int c = 0; c < csize; ++c) top = fmaxf(top, meets[(c * HEADS + row) * 2]);
            float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
            float den = 0.f;
#pragma unroll 4
            for (int c = 0; c < csize; ++c) {
                const float2 ml = *reinterpret_cast<const float2 *>(meets + (c * HEADS + row) * 2);
                const float4 x = *reinterpret_cast<const float4 *>(box + ((size_t)c * share + i - crank * share) * 4);
                const float wt = weight(ml.x, top);
                den = fmaf(wt, ml.y, den);
                num.x = fmaf(wt, x.x, num.x);
                num.y = fmaf(wt, x.y, num.y);
                num.z = fmaf(wt, x.z, num.z);
                num.w = fmaf(wt, x.w, num.w);
            }
            const float inv = den > 0.f ? 1.f / den : 0.f;
            const int64_t h = hk * group + g_base + row;
            uint2 two = make_uint2(MmaType<T>::pack(num.x * inv, num.y * inv), MmaType<T>::pack(num.z * inv, num.w * inv));
            reinterpret_cast<uint2 *>(static_cast<T *>(a.out) + ((int64_t)b * a.hq + h) * DFULL)[i % (DFULL / 4)] = two;
        }
        return;
    }
    // The normalised partial of each head and its log-sum-exp.
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int hg = g_base + (WIDE ? g + 8 * e : 2 * t + e);
        if (hg >= group) continue;
        const int64_t at = ((int64_t)b * a.hq + hk * group + hg) * a.splits + split;
        const float inv = l[e] > 0.f ? 1.f / l[e] : 0.f;
        float *po = a.part_o + at * DFULL + d0;
#pragma unroll
        for (int n = 0; n < ON; ++n) {
            if constexpr (WIDE) {
                *reinterpret_cast<float2 *>(po + n * 8 + 2 * t) = make_float2(o[n][2 * e] * inv, o[n][2 * e + 1] * inv);
            } else {
                po[n * 16 + g] = o[n][e] * inv;
                po[n * 16 + 8 + g] = o[n][2 + e] * inv;
            }
        }
        if ((WIDE ? t : g) == 0 && part == 0) a.part_lse[at] = l[e] > 0.f ? m[e] * a.scale + __logf(l[e]) : -INFINITY;
    }
}

// The same split for inputs the vector loads cannot take: one warp per (chunk, query head), a
// lane owning the head dimensions `lane + 32 i`, keys in order.
template <typename T>
__global__ void __launch_bounds__(DEC_WARPS * 32) decode_split_scalar_kernel(DecodeArgs a) {
    allow_beside();   // the merge
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.y;
    long long unit = (long long)blockIdx.x * DEC_WARPS + (threadIdx.x >> 5);
    const int h = (int)(unit % a.hq);
    const long long split = unit / a.hq;
    if (split >= a.splits) return;
    int first, len;
    decode_range(a, b, first, len);
    const long long c0l = (long long)first + split * a.chunk;
    if (c0l >= len) return;
    const int c0 = (int)c0l, c1 = min(len, c0 + a.chunk);
    const int hk = h / (a.hq / a.hkv);
    const int ni = (a.d + 31) / 32;
    float q[8], acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int c = lane + 32 * i;
        q[i] = (i < ni && c < a.d)
                   ? Num<T>::to_f32(static_cast<const T *>(a.q)[(int64_t)b * a.q_sb + (int64_t)h * a.q_sh + (int64_t)c * a.q_sd])
                   : 0.f;
        acc[i] = 0.f;
    }
    // The appending step: the row at `pos` comes from the new rows, and the warp of the group's
    // first head whose chunk holds it also writes it into the cache.
    const int pos = decode_append_at(a, b);
    const T *knew = static_cast<const T *>(a.k_new) + ((int64_t)b * a.hkv + hk) * a.d;
    const T *vnew = static_cast<const T *>(a.v_new) + ((int64_t)b * a.hkv + hk) * a.d;
    if (pos >= c0 && pos < c1 && h % (a.hq / a.hkv) == 0) {
        for (int c = lane; c < a.d; c += 32) {
            const_cast<T *>(static_cast<const T *>(a.k.ptr))[(int64_t)b * a.k.sb + (int64_t)pos * a.k.st + (int64_t)hk * a.k.sh + (int64_t)c * a.k.sd] = knew[c];
            const_cast<T *>(static_cast<const T *>(a.v.ptr))[(int64_t)b * a.v.sb + (int64_t)pos * a.v.st + (int64_t)hk * a.v.sh + (int64_t)c * a.v.sd] = vnew[c];
        }
    }
    float m = -INFINITY, l = 0.f;
    for (int key = c0; key < c1; ++key) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            int c = lane + 32 * i;
            if (i < ni && c < a.d) d = fmaf(q[i], key == pos ? Num<T>::to_f32(knew[c]) : load_f32<T>(a.k, b, key, hk, c), d);
        }
        const float s = warp_sum(d) * a.scale;
        const float mn = fmaxf(m, s);
        const float corr = expf(m - mn), p = expf(s - mn);
        l = l * corr + p;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            int c = lane + 32 * i;
            float v = (i < ni && c < a.d) ? (key == pos ? Num<T>::to_f32(vnew[c]) : load_f32<T>(a.v, b, key, hk, c)) : 0.f;
            acc[i] = fmaf(p, v, acc[i] * corr);
        }
        m = mn;
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    float *po = a.part_o + (((int64_t)b * a.hq + h) * a.splits + split) * a.d;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int c = lane + 32 * i;
        if (i < ni && c < a.d) po[c] = acc[i] * inv;
    }
    if (lane == 0) a.part_lse[((int64_t)b * a.hq + h) * a.splits + split] = l > 0.f ? m + logf(l) : -INFINITY;
}

// Merges the partials of one (sequence, query head) by their log-sum-exp: the weights once into
// shared memory, then every thread its head dimensions over the splits.
constexpr int MERGE_MAX = 1024;  // splits whose weights fit the shared array; more are folded in passes

constexpr int MERGE_EACH = 8;    // partials a thread asks for at once

template <typename T, int TH>
__global__ void __launch_bounds__(TH) decode_merge_kernel(DecodeArgs a) {
    __shared__ float w[MERGE_MAX];
    __shared__ float red[TH / 32];
    __shared__ float4 part[TH];
    __shared__ float dens[TH];
    wait_before();   // the split pass
    const int bh = blockIdx.x;
    const int b = bh / a.hq;
    int first, len;
    decode_range(a, b, first, len);
    const int n = (len - first + a.chunk - 1) / a.chunk;  // splits that hold keys
    T *out = static_cast<T *>(a.out) + (int64_t)bh * a.d;
    if (n <= 0) {
        for (int c = threadIdx.x; c < a.d; c += TH) out[c] = Num<T>::from_f32(0.f);
        return;
    }
    // Four head dimensions a thread (16-byte loads of the partials), the splits dealt over the TH / (d / 4) groups of threads,
    // whose sums meet in shared memory in group order.
    const int ct = max(a.d / 4, 1), groups = TH / ct;
    const int c4 = threadIdx.x % ct, sg = threadIdx.x / ct;
    auto finish = [&](float4 num, float den) {
        part[threadIdx.x] = num;
        dens[threadIdx.x] = den;
        __syncthreads();
        if (sg != 0) return;
        for (int g = 1; g < groups; ++g) {
            const float4 x = part[g * ct + c4];
            num.x += x.x; num.y += x.y; num.z += x.z; num.w += x.w;
            den += dens[g * ct + c4];
        }
        const float inv = den > 0.f ? 1.f / den : 0.f;
        T *o = out + 4 * c4;
        o[0] = Num<T>::from_f32(num.x * inv);
        o[1] = Num<T>::from_f32(num.y * inv);
        o[2] = Num<T>::from_f32(num.z * inv);
        o[3] = Num<T>::from_f32(num.w * inv);
    };
    const bool vec = a.d % 4 == 0;
    if (vec && n <= MERGE_EACH * groups) {
        // Few splits: a thread asks for its log-sum-exps and its partials at once and has the maximum worked out under their
        // flight, one trip to memory where the passes below take one for the maximum, one for the weights and one for
        // every four partials.
        const float *lse = a.part_lse + (int64_t)bh * a.splits;
        const float *po = a.part_o + (int64_t)bh * a.splits * a.d + 4 * c4;
        float own[MERGE_EACH];
        float4 x[MERGE_EACH];
#pragma unroll
        for (int e = 0; e < MERGE_EACH; ++e) {
            const int i = sg + e * groups;
            const bool in = sg < groups && i < n;
            own[e] = in ? lse[i] : -INFINITY;
            x[e] = in ? *reinterpret_cast<const float4 *>(po + (int64_t)i * a.d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float mx = own[0];
#pragma unroll
        for (int e = 1; e < MERGE_EACH; ++e) mx = fmaxf(mx, own[e]);
        mx = warp_max(mx);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
        __syncthreads();
        mx = red[0];
#pragma unroll
        for (int i = 1; i < TH / 32; ++i) mx = fmaxf(mx, red[i]);
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        float den = 0.f;
#pragma unroll
        for (int e = 0; e < MERGE_EACH; ++e) {
            if (sg + e * groups >= n) break;
            const float wi = expf(own[e] - mx);
            den += wi;
            num.x = fmaf(wi, x[e].x, num.x);
            num.y = fmaf(wi, x[e].y, num.y);
            num.z = fmaf(wi, x[e].z, num.z);
            num.w = fmaf(wi, x[e].w, num.w);
        }
        finish(num, den);
        return;
    }
    const float *lse = a.part_lse + (int64_t)bh * a.splits;
    const float *po = a.part_o + (int64_t)bh * a.splits * a.d;
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < n; i += TH) mx = fmaxf(mx, lse[i]);
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = red[0];
#pragma unroll
    for (int i = 1; i < TH / 32; ++i) mx = fmaxf(mx, red[i]);

    if (vec) {
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        float den = 0.f;
        for (int i0 = 0; i0 < n; i0 += MERGE_MAX) {
            const int m = min(MERGE_MAX, n - i0);
            __syncthreads();
            for (int i = threadIdx.x; i < m; i += TH) w[i] = expf(lse[i0 + i] - mx);
            __syncthreads();
            if (sg < groups) {
#pragma unroll 4
                for (int i = sg; i < m; i += groups) {
                    const float wi = w[i];
                    const float4 x = *reinterpret_cast<const float4 *>(po + (int64_t)(i0 + i) * a.d + 4 * c4);
                    den += wi;
                    num.x = fmaf(wi, x.x, num.x);
                    num.y = fmaf(wi, x.y, num.y);
                    num.z = fmaf(wi, x.z, num.z);
                    num.w = fmaf(wi, x.w, num.w);
                }
            }
        }
        finish(num, den);
        return;
    }
    float num[2] = {0.f, 0.f}, den = 0.f;  // a.d <= 256 <= 2 TH: two head dimensions per thread at most
    for (int i0 = 0; i0 < n; i0 += MERGE_MAX) {
        const int m = min(MERGE_MAX, n - i0);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += TH) w[i] = expf(lse[i0 + i] - mx);
        __syncthreads();
#pragma unroll 4
        for (int i = 0; i < m; ++i) {
            const float wi = w[i];
            den += wi;
            const float *row = po + (int64_t)(i0 + i) * a.d;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int c = threadIdx.x + TH * k;
                if (c < a.d) num[k] = fmaf(wi, row[c], num[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int c = threadIdx.x + TH * k;
        if (c < a.d) out[c] = Num<T>::from_f32(den > 0.f ? num[k] / den : 0.f);
    }
}

template <typename T, int D, int GH>
static cudaError_t split_vec_g(const DecodeArgs &a, dim3 grid, cudaStream_t stream) {
    constexpr int VPK = sizeof(T) == 4 ? 2 : 1, NS = sizeof(T) == 4 ? 2 : DEC_STAGES;
    constexpr size_t smem = (size_t)DEC_WARPS * NS * (2 * DEC_UNROLL * VPK) * 32 * 16;
    cudaError_t e = cudaFuncSetAttribute(decode_split_kernel<T, D, GH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    decode_split_kernel<T, D, GH><<<grid, DEC_WARPS * 32, smem, stream>>>(a);
    return cudaGetLastError();
}

template <typename T, int D>
static cudaError_t split_vec(const DecodeArgs &a, cudaStream_t stream) {
    const int group = a.hq / a.hkv;
    const int gh = group >= 4 ? 4 : (group >= 2 ? 2 : 1);
    const int passes = (group + gh - 1) / gh;
    const long long units = (long long)a.splits * a.hkv * passes;
    dim3 grid((unsigned)((units + DEC_WARPS - 1) / DEC_WARPS), a.b);
    if (gh == 4) return split_vec_g<T, D, 4>(a, grid, stream);
    if (gh == 2) return split_vec_g<T, D, 2>(a, grid, stream);
    return split_vec_g<T, D, 1>(a, grid, stream);
}

// Bytes of shared memory of a block of the tensor-core pass; `cluster`: with the boxes its cluster meets in (a share of the
// outputs is rounded up to a piece a block).
constexpr size_t mma_smem(int dfull, bool wide, int warps, bool cluster) {
    const int parts = dfull > 128 ? 2 : 1, d = dfull / parts;
    return (size_t)warps * DM_STAGES * 2 * DM_KEYS * 2 * d + (parts == 2 ? sizeof(float) * warps * 32 * (wide ? 8 : 4) : 0) +
           (cluster ? sizeof(float) * (8 * dfull + MAX_CLUSTER * 4 + (MAX_CLUSTER + (size_t)warps / parts) * 16) : 0);
}
// `warps`: of one sequence.
template <typename T, int DFULL, bool WIDE, int WARPS, bool CLUSTER>
static cudaError_t split_mma_w(const DecodeArgs &a, long long warps, int cluster, cudaStream_t stream) {
    constexpr int PARTS = DFULL > 128 ? 2 : 1, D = DFULL / PARTS;
    constexpr size_t smem = mma_smem(DFULL, WIDE, WARPS, CLUSTER);
    const auto kernel = a.rope_cos ? decode_split_mma_kernel<T, D, PARTS, WIDE, WARPS, true, CLUSTER> : decode_split_mma_kernel<T, D, PARTS, WIDE, WARPS, false, CLUSTER>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && cluster > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    return launch_clusters(kernel, dim3((unsigned)((warps + WARPS - 1) / WARPS), (unsigned)a.b), WARPS * 32, smem, stream, false, (unsigned)cluster, a);
}
// Blocks (of CLUSTER_WARPS warps) of the cluster that takes a key-value head of a sequence; 0: chunks, and the merge behind them.
// A cluster saves the merge and its launch, 3 to 5 us; what it costs is the chain of a warp's tiles (0.4 us a tile at D 64, 0.6 at 128,
// 0.7 at 256), which nobody else shortens: where one sequence is much longer than the others, or the last blocks start when the first have
// ended, the GPU waits for it, and chunks spread over all multiprocessors.  So: the blocks run at once, and the longest share that a sequence may
// give a warp (it may fill the cache) is short - five tiles where few blocks run, whose multiprocessors would stand idle beside them, more where
// they nearly fill the GPU; of several sizes the one with the shortest share.  Lengths given, blocks for 1.4 times to nearly twice the room still
// pay, in clusters of up to four with shares of 8 to 16 tiles: not all of them last.  (`room`: blocks that run at once, two of 104 KB to a multiprocessor and
// four at D 64, less what the clusters leave idle of GPU processing clusters; the runtime says 296, 296, 284, 264 and 224 for 1 to 16 blocks where
// nothing else runs, the lines lie a few clusters below.)
// Under a window of at most half the cache every longer sequence has the same share, and most chunks are empty: any number of blocks, priced
// in tiles - the longest share and eight tiles' time that a block costs, or the waves of that and half of it again.
// Chosen over 864 shapes (1 to 64 sequences, 530 to 32768 keys, D 64 to 256, groups of 2 to 8), each with whole caches and with lengths
// spread evenly, all short, a few long and one long, timed with chunks and with every size of cluster, and tried on 837 others with and without
// rotation and append, bf16 and f16: against chunks and merge with heads as rows the mean of those is 1.12 (whole), 1.17 (even), 1.25 (short), 1.18 (one
// long), 1.16 (a few long), the worst 0.94, under 0.97 in 5 of 3521.  (Clusters wherever a price that takes lengths at half the cache says so:
// 1.12, 1.20, 1.37, 1.13, 1.13, but under 0.97 in 237, the worst 0.52.)  1202 windows of 60 to 4096 keys: whole caches 1.93, even lengths 1.87, none slower.
// us, heads as rows | clusters wherever | now: 9 whole caches of 20576 keys, 16 / 4 heads of 128, 67 | 87 | 65; 18 of 6156, 8 / 2 of 256, 41 | 56 |
// 41; 23 of up to 32768, 32 / 8, one of them long, 59 | 123 | 57; 16 of up to 4096, one long, 19.5 | 24.9 | 16.0, evenly spread 35.5 | 30.7 | 31.4;
// 4 of up to 10006, evenly spread, 30.5 | 21.2 | 21.2, but 8 of up to 7537 42.2 | 31.5 | 39.4; one of 2947 with rotation and append 12.6 | 10.7 | 10.7.
// A share is at most 512 keys; at f16, whose P is sharper in two parts than bf16's, no longer than the chunk would be, or 192: one accumulator loses a
// little of each addition to a long sum, which shows there first (error against f64 where the output is next to nothing, 32 of 1000 keys, 32 / 8 heads
// of 128: 2.46e-8 in chunks of 128, 2.63e-8 in shares of 256, 2.14e-8 in shares of 128; 16 of 3000, 2.07e-8 in chunks, 2.02e-8 in shares of 192).
// Caches of at most 512 keys keep the two launches (tests/test_decode_rotates_gpu.py counts them): 16 of 200, 16 / 4 heads, 7.9 where a
// cluster takes 5.4.
static int decode_cluster(const DecodeArgs &a, bool narrow) {
    if (decode_fixed_chunk() > 0 || a.s <= 512) return 0;
    const int64_t units = (int64_t)a.hkv * a.b, shares = a.d > 128 ? CLUSTER_WARPS / 2 : CLUSTER_WARPS;
    const int64_t seen = std::min<int64_t>(a.s, (int64_t)a.left + 1), tiles = (seen + DM_KEYS - 1) / DM_KEYS, few = a.d == 128 ? 96 : 160;
    const bool window = 2 * seen <= a.s;
    const int64_t most_keys = narrow ? std::max(a.chunk, 192) : 512;
    int best = 0;
    double least = 0.;
    for (int c = 1; c <= MAX_CLUSTER; c *= 2) {
        const int64_t blocks = units * c, longest = (tiles + c * shares - 1) / (c * shares);
        const double full = blocks / ((c == 16 ? 128. : c == 8 ? 256. : c == 4 ? 272. : c == 2 ? 288. : 296.) * (a.d == 64 ? 2 : 1));   // of the room
        double cost = longest;
        if (longest * DM_KEYS > most_keys || (c == 16 && full > 1.)) continue;
        if (window) {
            if ((blocks < few && longest > 5) || (blocks < 192 && longest > 16)) continue;
            cost += 8.;
            if (full > 1.) cost *= full + 0.5;
        } else if (full <= 1.) {
            // (Clusters of sixteen leave half the multiprocessors without a block, which a cache that is not in L2 is read slower by.)
            const double most = a.d <= 128 ? 5. + 18. * full * full : 4. + 18. * full * full;
            if (longest > (c < 16 ? most : a.d <= 128 ? std::min(most, 12.) : 3. + full * full)) continue;
        } else {
            if (!a.lengths || full < 1.4 || full > 1.95 || c > 4 || a.d > 128 || longest < 8 || longest > 16) continue;
            cost += 64.;   // whatever runs at once first
        }
        if (best == 0 || cost < least) { best = c; least = cost; }
    }
    return best;
}
template <typename T, int DFULL>
static cudaError_t split_mma(const DecodeArgs &a, cudaStream_t stream, bool *merged) {
    const int group = a.hq / a.hkv;
    const bool wide = group > 8;
    // (A cluster stores its outputs eight bytes at a time, the merge one element: it takes any address.)
    const bool whole = reinterpret_cast<uintptr_t>(a.out) % 8 == 0;
    if (const int cluster = wide || !whole ? 0 : decode_cluster(a, MmaType<T>::NARROW)) {
        const long long warps = (long long)a.hkv * cluster * CLUSTER_WARPS;
        const cudaError_t e = split_mma_w<T, DFULL, false, CLUSTER_WARPS, true>(a, warps, cluster, stream);
        *merged = e == cudaSuccess;
        if (*merged) return e;
        cudaGetLastError();   // (a part of a GPU may have no room for such a cluster: the chunks go anywhere)
    }
    const long long warps = (long long)a.splits * a.hkv * (wide ? (group + 15) / 16 : 1) * (DFULL > 128 ? 2 : 1);   // of one sequence
    const bool few = warps * a.b < 148LL * 8 * 2;
    if (wide) return few ? split_mma_w<T, DFULL, true, 2, false>(a, warps, 1, stream) : split_mma_w<T, DFULL, true, 8, false>(a, warps, 1, stream);
    return few ? split_mma_w<T, DFULL, false, 2, false>(a, warps, 1, stream) : split_mma_w<T, DFULL, false, 8, false>(a, warps, 1, stream);
}
template <> cudaError_t split_mma<float, 128>(const DecodeArgs &, cudaStream_t, bool *) { return cudaErrorInvalidValue; }   // never taken: 16-bit caches only
template <> cudaError_t split_mma<float, 64>(const DecodeArgs &, cudaStream_t, bool *) { return cudaErrorInvalidValue; }
template <> cudaError_t split_mma<float, 256>(const DecodeArgs &, cudaStream_t, bool *) { return cudaErrorInvalidValue; }

// DASH_ATTN_DECODE_MMA=0 keeps the FMA pass (for comparison runs).
static bool decode_force_scalar_pass() {
    static const bool off = [] { const char *e = std::getenv("DASH_ATTN_DECODE_MMA"); return e && std::atoi(e) == 0; }();
    return off;
}

// (The tensor-core pass keeps maxima of scores that have not been scaled yet: a scale of zero or below would turn their order round, and
// what is not finite would meet their first -inf.  The FMA pass scales first.)
static bool decode_uses_mma(size_t elem, const DecodeArgs &a, bool vector_ok) {
    return vector_ok && elem == 2 && a.hq / a.hkv >= 2 && a.scale > 0.f && std::isfinite(a.scale) && !decode_force_scalar_pass();
}
bool decode_fuses_rope(int dtype, const DecodeArgs &a, bool vector_ok) {
    auto aligned = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    // Halves of whole 16-byte chunks: a pair's two columns then sit in chunks (and fragments) of their own.
    return dtype != 0 && decode_uses_mma(2, a, vector_ok) && a.rope_dim % 16 == 0 && aligned(a.rope_cos) && aligned(a.rope_sin);
}

template <typename T>
static cudaError_t decode_t(const DecodeArgs &a, bool vector_ok, cudaStream_t stream, int *launches) {
    cudaError_t e;
    const bool mma = decode_uses_mma(sizeof(T), a, vector_ok);
    bool merged = false;
    if (mma && a.d == 128) e = split_mma<T, 128>(a, stream, &merged);
    else if (mma && a.d == 64) e = split_mma<T, 64>(a, stream, &merged);
    else if (mma && a.d == 256) e = split_mma<T, 256>(a, stream, &merged);
    else if (vector_ok && a.d == 64) e = split_vec<T, 64>(a, stream);
    else if (vector_ok && a.d == 128) e = split_vec<T, 128>(a, stream);
    else if (vector_ok && a.d == 256) e = split_vec<T, 256>(a, stream);
    else {
        const long long units = (long long)a.splits * a.hq;
        dim3 grid((unsigned)((units + DEC_WARPS - 1) / DEC_WARPS), a.b);
        decode_split_scalar_kernel<T><<<grid, DEC_WARPS * 32, 0, stream>>>(a);
        e = cudaGetLastError();
    }
    *launches += 1;
    if (e != cudaSuccess || merged) return e;
    *launches += 1;
    // The merge comes in under the pass's end (us, after it | under it): 16 of up to 500 keys, 16 / 4 heads, 9.0 | 8.8; two of 8192, 8 on one, 9.5 | 8.9; eight
    // of 6144, 8 / 2 of 128, 14.8 | 14.3; 60 of up to 9557, 8 heads, 184.2 | 183.7.  (Its blocks gather on the multiprocessors the pass leaves first, and
    // a few calls lose by it: eight of 6144, 8 / 2 of 256, 22.6 | 23.0, one of up to 20000, 8 heads, 18.0 | 18.2.  Neither the parts' size nor the blocks'
    // number tells them apart.)
    // Threads of a merge block: 128, or where the blocks are at most two a multiprocessor the fewest (up to 512) with which every
    // partial is asked for at once.  (Threads 128 / 256 / 512: eight of 6144, 8 / 2 heads of 128, 15.7 / 14.3 / 15.3 us; one of up to 20000, 32 / 8, 20.0 / 18.5 / 18.2;
    // two of 8192, 8 on one, 10.6 / 9.5 / 8.9; eight of 6144, 8 / 2 of 256, 23.7 / 22.8 / 22.9; but 60 of up to 9557 on 1920 blocks 183.6 / 186.4 / 195.9, and 64 of up to
    // 4096 on 2048 92.5 / 96.3 / 105.8.)
    const int64_t blocks = (int64_t)a.b * a.hq;
    int threads = 128;
    if (blocks <= 2 * 148)
        while (threads < 512 && (int64_t)a.splits * std::max(a.d / 4, 1) > (int64_t)MERGE_EACH * threads) threads *= 2;
    const dim3 grid((unsigned)blocks);
    if (threads == 512) return launch_beside(decode_merge_kernel<T, 512>, grid, 512, 0, stream, true, a);
    if (threads == 256) return launch_beside(decode_merge_kernel<T, 256>, grid, 256, 0, stream, true, a);
    return launch_beside(decode_merge_kernel<T, 128>, grid, 128, 0, stream, true, a);
}

cudaError_t launch_decode(int dtype, const DecodeArgs &a, bool vector_ok, cudaStream_t stream, int *launches) {
    switch (dtype) {
        case 0: return decode_t<float>(a, vector_ok, stream, launches);
        case 1: return decode_t<__nv_bfloat16>(a, vector_ok, stream, launches);
        default: return decode_t<__half>(a, vector_ok, stream, launches);
    }
}

// ---------------------------------------------------------------------------------------------
// The decoding step with its scratch inside the library (dash_attn_decode_static)
// ---------------------------------------------------------------------------------------------
// Some callers hold nothing but the raw input and output buffers they were handed and have no way
// to produce a workspace: an FFI shim under a tensor runtime whose memory pool owns all device
// memory and is not reachable from C, or a serving loop that has promised not to allocate once it
// is running.  For them the partial outputs of the split pass live in this file-scope array
// instead of a caller-provided workspace.  Every GPU that loads the library reserves it until the
// process exits, so it is kept modest: 4 Mi floats (16 MiB).
//
// In host code the array's name is only a stand-in; its device address is asked for once per
// device (with that device current) and cached.  All calls share the array and it keeps whatever
// the last call left in it: nothing in it needs to start at zero, because the merge pass reads
// only the partials the split pass of the same call has just written - but two calls whose kernels
// overlap on the GPU (different streams, or different host threads without ordering) would write
// over each other's partials.
constexpr size_t DECODE_STATIC_FLOATS = size_t(4) << 20;
static __device__ __align__(256) float g_decode_static_scratch[DECODE_STATIC_FLOATS];

size_t decode_static_capacity_floats() { return DECODE_STATIC_FLOATS; }

// The device address of the static scratch on the current device; the first call on each device
// resolves it (and should therefore come before any stream capture begins).
cudaError_t decode_static_scratch(float **out) {
    constexpr int MAX_DEVICES = 64;
    static float *cache[MAX_DEVICES] = {};
    static std::mutex lock;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> guard(lock);
    if (!cache[dev]) {
        float *ptr = nullptr;
        e = cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_decode_static_scratch);
        if (e != cudaSuccess) return e;
        cache[dev] = ptr;
    }
    *out = cache[dev];
    return cudaSuccess;
}

}  // namespace dash
