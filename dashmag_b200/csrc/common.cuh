// Shared device-side pieces of the attention kernels: dtype conversion, strided tensor views, and
// the integer rule that says which keys a query sees.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace dash {

// ---------------------------------------------------------------------------------------------
// dtypes
// ---------------------------------------------------------------------------------------------
template <typename T> struct Num;
template <> struct Num<float> {
    static __device__ __forceinline__ float to_f32(float x) { return x; }
    static __device__ __forceinline__ float from_f32(float x) { return x; }
};
template <> struct Num<__nv_bfloat16> {
    static __device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
    static __device__ __forceinline__ __nv_bfloat16 from_f32(float x) { return __float2bfloat16_rn(x); }
};
template <> struct Num<__half> {
    static __device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }
    static __device__ __forceinline__ __half from_f32(float x) { return __float2half_rn(x); }
};

// A [batch, time, head, dim] view of caller-owned memory, strides in elements.
struct View4 {
    const void *ptr;
    int64_t sb, st, sh, sd;
};

template <typename T>
__device__ __forceinline__ float load_f32(const View4 &v, int64_t b, int64_t t, int64_t h, int64_t d) {
    return Num<T>::to_f32(static_cast<const T *>(v.ptr)[b * v.sb + t * v.st + h * v.sh + d * v.sd]);
}

// ---------------------------------------------------------------------------------------------
// Which keys a query sees
// ---------------------------------------------------------------------------------------------
// Every mask of the contract but key padding gives each query ONE interval of keys [lo, hi):
// the query's position is `row + Tk - Tq` (packed: `i + Lk - Lq` inside its own sequence) and it
// sees from `left` keys before that position to `right` after it
// (crates/dash-contract/src/attention.rs:33-54).  `left` and `right` arrive clamped to
// Tq + Tk + 1, which stands for "no bound" and keeps everything inside int32.
struct MaskArgs {
    int kind;              // 0 none, 1 key padding, 2 packed
    const void *kp;        // key padding [B,Tk]
    int kp_bytes;          // 1 or 4
    int64_t kp_sb, kp_st;  // element strides
    const void *cu_q;      // [seqs + 1]
    const void *cu_k;
    int seqs;
    int idx_bytes;         // 4 or 8
    int left, right;       // clamped reach; causal already folded into right = 0
};

__device__ __forceinline__ int load_index(const void *p, int bytes, int i) {
    if (bytes == 8) {
        long long v = static_cast<const long long *>(p)[i];
        v = v < -2147483647LL ? -2147483647LL : (v > 2147483647LL ? 2147483647LL : v);
        return static_cast<int>(v);
    }
    return static_cast<const int *>(p)[i];
}

// The last s with cu[s] <= pos over the non-decreasing offsets cu[0..seqs]: -1 before the first
// offset, `seqs` from the last one on (both: no sequence).
__device__ __forceinline__ int sequence_of(const void *cu, int bytes, int seqs, int pos) {
    int lo = 0, hi = seqs + 1;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (load_index(cu, bytes, mid) <= pos) lo = mid + 1; else hi = mid;
    }
    return lo - 1;
}

// The keys query `row` of packed sequence `s` sees, [lo, hi), or (tk, 0) when it sees none.
__device__ __forceinline__ void row_bounds_in_sequence(const MaskArgs &m, int s, int row, int tk, int &lo, int &hi) {
    lo = tk;
    hi = 0;
    if (s < 0 || s >= m.seqs) return;
    int q0 = load_index(m.cu_q, m.idx_bytes, s), q1 = load_index(m.cu_q, m.idx_bytes, s + 1);
    int k0 = load_index(m.cu_k, m.idx_bytes, s), k1 = load_index(m.cu_k, m.idx_bytes, s + 1);
    int lk = k1 - k0, lq = q1 - q0;
    int pos = row - q0 + lk - lq;
    int a = max(k0 + max(0, pos - m.left), 0);
    int c = min(k0 + min(lk, pos + m.right + 1), tk);
    if (c > a) { lo = a; hi = c; }
}

// The keys query `row` sees, [lo, hi), or (tk, 0) when it sees none or lies past the queries.
__device__ __forceinline__ void row_bounds(const MaskArgs &m, int row, int tq, int tk, int &lo, int &hi) {
    lo = tk;
    hi = 0;
    if (row < 0 || row >= tq) return;
    if (m.kind == 2) {
        row_bounds_in_sequence(m, sequence_of(m.cu_q, m.idx_bytes, m.seqs, row), row, tk, lo, hi);
    } else {
        int pos = row + tk - tq;
        int a = max(0, pos - m.left);
        int c = min(tk, pos + m.right + 1);
        if (c > a) { lo = a; hi = c; }
    }
}

// The same for the 32 rows of a (converged) warp at once.  A thread that places its row by itself walks
// the packed offsets by bisection - three or four DEPENDENT loads from global memory, some two thousand
// cycles of a block's set-up before its first tile load can be issued.  Here each lane fetches ONE pair of
// offsets (lane i: cu_q[i], cu_k[i]; batches of up to 31 sequences, else every lane falls back to
// row_bounds), the rows are placed by comparing against the lanes' values, and the four offsets of a row's
// sequence come by shuffle: one load latency instead of four.  All 32 lanes must call; results are
// identical to row_bounds.
__device__ __forceinline__ void row_bounds_warp(const MaskArgs &m, int row, int tq, int tk, int &lo, int &hi) {
    if (m.kind != 2 || m.seqs > 31) {
        row_bounds(m, row, tq, tk, lo, hi);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int cq = lane <= m.seqs ? load_index(m.cu_q, m.idx_bytes, lane) : 2147483647;
    const int ck = lane <= m.seqs ? load_index(m.cu_k, m.idx_bytes, lane) : 2147483647;
    int s = -1;   // the last s with cu_q[s] <= row: the offsets do not decrease, so it is a count
    for (int i = 0; i <= m.seqs; ++i) s += __shfl_sync(0xffffffffu, cq, i) <= row ? 1 : 0;
    const int sc = min(max(s, 0), 30);
    const int q0 = __shfl_sync(0xffffffffu, cq, sc), q1 = __shfl_sync(0xffffffffu, cq, sc + 1);
    const int k0 = __shfl_sync(0xffffffffu, ck, sc), k1 = __shfl_sync(0xffffffffu, ck, sc + 1);
    lo = tk;
    hi = 0;
    if (row < 0 || row >= tq || s < 0 || s >= m.seqs) return;
    const int lk = k1 - k0, lq = q1 - q0;
    const int pos = row - q0 + lk - lq;
    const int a = max(k0 + max(0, pos - m.left), 0);
    const int c = min(k0 + min(lk, pos + m.right + 1), tk);
    if (c > a) { lo = a; hi = c; }
}

__device__ __forceinline__ bool key_padded(const MaskArgs &m, int b, int key) {
    if (m.kind != 1) return false;
    int64_t at = (int64_t)b * m.kp_sb + (int64_t)key * m.kp_st;
    return m.kp_bytes == 4 ? static_cast<const int *>(m.kp)[at] != 0
                           : static_cast<const unsigned char *>(m.kp)[at] != 0;
}

// (declared below)
__device__ __forceinline__ int warp_max_i(int x);
__device__ __forceinline__ int warp_min_i(int x);

// A block's sweep [kmin, kmax) without the padded keys at its ends: right- and left-padded batches are swept no further
// than their tokens go.  All 32 lanes call and get one answer, the same in every warp; 256 flags a look, from either
// end, so that a sweep that is not padded there pays one trip to memory.  (kmax <= kmin: no key is left.)
// (By value, in and out: a reference would put the caller's arguments on the stack.)
static __device__ __noinline__ int2 trim_padded_span(const void *kp, int kp_bytes, int64_t sb, int64_t st, int b, int kmin, int kmax) {
    const int lane = threadIdx.x & 31;
    // A look's flags are all asked for before any is looked at (keys past the look's end: its last one again).
    auto look = [&](int from, int hop, bool (&shut)[8]) {
        int flag[8];
        if (kp_bytes == 4) {
#pragma unroll
            for (int i = 0; i < 8; ++i) flag[i] = static_cast<const int *>(kp)[(int64_t)b * sb + (int64_t)min(max(from + hop * (32 * i + lane), kmin), kmax - 1) * st];
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) flag[i] = static_cast<const unsigned char *>(kp)[(int64_t)b * sb + (int64_t)min(max(from + hop * (32 * i + lane), kmin), kmax - 1) * st];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) shut[i] = flag[i] != 0;
    };
    int last = -1;
    while (kmax > kmin && last < 0) {
        bool shut[8];
        look(kmax - 1, -1, shut);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int key = kmax - 1 - 32 * i - lane;
            if (key >= kmin && !shut[i]) last = max(last, key);
        }
        last = warp_max_i(last);
        kmax = last >= 0 ? last + 1 : kmax - 256;
    }
    int first = 2147483647;
    while (kmax > kmin && first == 2147483647) {
        bool shut[8];
        look(kmin, 1, shut);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int key = kmin + 32 * i + lane;
            if (key < kmax && !shut[i]) first = min(first, key);
        }
        first = warp_min_i(first);
        kmin = first != 2147483647 ? first : kmin + 256;
    }
    return kmax > kmin ? make_int2(kmin, kmax) : make_int2(0, 0);   // (nothing: no tile starts below the span's end)
}
__device__ __forceinline__ void trim_padded(const MaskArgs &m, int b, int &kmin, int &kmax) {
    const int2 span = trim_padded_span(m.kp, m.kp_bytes, m.kp_sb, m.kp_st, b, kmin, kmax);
    kmin = span.x;
    kmax = span.y;
}

// The keys of a batch element that are not padding, if they are one run - every right- or left-padded batch's are - and few enough that
// eight warps look at all of them at once: their first and last and how many there are, a warp's share each, to be met with the
// others'.  A sweep cut to the run has no flags to look at.  Asked for with the rows' intervals, in front of the block's first barrier,
// it costs a trip to memory beside theirs; trim_padded's looks come behind the barrier, one after the other (3000 to 4700 cycles of a
// block's 28 to 35 thousand, 16 x 509, 12 heads of 64; 7000 to 11000 while a look asked for one flag at a time), and the flags of
// every step 200 of its 2300.  That batch's forward 51.6 -> 44.1 us with whole looks, 39.4 with the run; 24 x 448, 12 / 4 heads, backward
// in fixed order 116.8 -> 102.7 -> 96.5.  (Longer masks: trim_padded.)
constexpr int OPEN_RUN_KEYS = 2048;
struct OpenRun { int first, last, count; };
__device__ __forceinline__ OpenRun open_run_share(const MaskArgs &m, int b, int tk, int warp) {
    constexpr int EACH = OPEN_RUN_KEYS / 256;
    const int lane = threadIdx.x & 31, base = warp * 32 + lane;
    int flag[EACH];
    if (m.kp_bytes == 4) {
#pragma unroll
        for (int i = 0; i < EACH; ++i) flag[i] = static_cast<const int *>(m.kp)[(int64_t)b * m.kp_sb + (int64_t)min(base + 256 * i, tk - 1) * m.kp_st];
    } else {
#pragma unroll
        for (int i = 0; i < EACH; ++i) flag[i] = static_cast<const unsigned char *>(m.kp)[(int64_t)b * m.kp_sb + (int64_t)min(base + 256 * i, tk - 1) * m.kp_st];
    }
    OpenRun r = {2147483647, -1, 0};
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int key = base + 256 * i;
        if (key < tk && flag[i] == 0) {
            r.first = min(r.first, key);
            r.last = max(r.last, key);
            r.count += 1;
        }
    }
    r.first = __reduce_min_sync(0xffffffffu, r.first);
    r.last = __reduce_max_sync(0xffffffffu, r.last);
    r.count = __reduce_add_sync(0xffffffffu, r.count);
    return r;
}
// The eight shares together, and the sweep [kmin, kmax) cut to the run; false (and nothing cut): there are holes.
__device__ __forceinline__ bool cut_to_open_run(const OpenRun (&shares)[8], OpenRun &run, int &kmin, int &kmax) {
    run = shares[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        run.first = min(run.first, shares[i].first);
        run.last = max(run.last, shares[i].last);
        run.count += shares[i].count;
    }
    if (run.count > 0 && run.count != run.last - run.first + 1) return false;
    kmin = max(kmin, run.first);
    kmax = min(kmax, run.last + 1);
    return true;
}

__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
__device__ __forceinline__ int warp_min_i(int x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = min(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ int warp_max_i(int x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// ---------------------------------------------------------------------------------------------
// Kernels of one call that run side by side
// ---------------------------------------------------------------------------------------------
// A kernel launched with launch_beside may start as soon as every block of the kernel in front of it
// has run allow_beside (or has left): its blocks take the multiprocessors that kernel's last wave leaves
// idle.  It must not touch what that kernel writes, and what both read was complete before either
// began.  Whatever comes next in the stream waits for the second kernel only, so that kernel's last block waits
// for the first before it leaves (end_beside; a no-op in an ordinary launch).
__device__ __forceinline__ void allow_beside() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void end_beside() {
    if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1)
        asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A kernel launched with launch_beside that does read what the kernel in front of it writes: its blocks are brought in
// under that kernel's end and wait here.
__device__ __forceinline__ void wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_clusters(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, bool beside, unsigned cluster, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    if (beside) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = cluster;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_beside(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, bool beside, A... args) {
    return launch_clusters(kernel, grid, threads, smem, stream, beside, 1u, args...);
}

// ---------------------------------------------------------------------------------------------
// Arguments of the generic kernels
// ---------------------------------------------------------------------------------------------
struct TrainArgs {
    int b, tq, tk, hq, hkv, d;
    float scale;
    View4 q, k, v, o, dout;     // o / dout: backward's inputs
    void *out;                  // forward: o (contiguous, q's dtype)
    float *lse;                 // forward: output; backward: input; contiguous [B,Tq,Hq]
    float *delta;               // backward scratch [B,Tq,Hq]
    void *dq, *dk, *dv;         // backward outputs, contiguous
    MaskArgs mask;
};

struct DecodeArgs {
    int b, s, hq, hkv, d;
    float scale;
    const void *q;
    int64_t q_sb, q_sh, q_sd;
    View4 k, v;
    const void *lengths;
    int len_bytes;
    int left;                   // clamped to s + 1 = no bound
    int chunk, splits;          // keys per split and splits per sequence
    float *part_o;              // [B,Hq,splits,D]
    float *part_lse;            // [B,Hq,splits]
    void *out;                  // [B,Hq,D]
    // The step that also appends: the new key and value rows [B,Hkv,D] (contiguous) go to
    // position lengths[b] of the cache, where the step already sees them.  Null otherwise.
    const void *k_new, *v_new;
    // The step that also rotates: the queries and the new key are rotated by the row of the tables [rope_len, rope_dim] at
    // rope_pos[b] as they are read (decode_fuses_rope says which calls).  rope_cos null otherwise.
    const void *rope_cos, *rope_sin, *rope_pos;
    int rope_dim, rope_pos_bytes;
    int64_t rope_len;
};

// Where the appending step writes sequence b's new row: its length before the step, or -1 when
// the step does not append or the cache is full.
__device__ __forceinline__ int decode_append_at(const DecodeArgs &a, int b) {
    if (!a.k_new || !a.lengths) return -1;
    const int len = max(load_index(a.lengths, a.len_bytes, b), 0);
    return len < a.s ? len : -1;
}

// The visible keys of sequence b in a decoding step: [first, len); the appended row counts.
__device__ __forceinline__ void decode_range(const DecodeArgs &a, int b, int &first, int &len) {
    len = a.s;
    if (a.lengths) len = min(max(load_index(a.lengths, a.len_bytes, b), 0) + (a.k_new ? 1 : 0), a.s);
    first = max(0, len - 1 - a.left);
    if (a.left > a.s) first = 0;
}

}  // namespace dash
