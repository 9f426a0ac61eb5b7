// Host side of the tcgen05 path: which calls it takes, the TMA tensor maps over the caller's
// tensors, and the launches.
#include "sm100.h"

#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "launch.h"
#include "sm100_kernels.h"

namespace dash {

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up through the runtime so that the library carries no
// link-time dependency on libcuda (it must load on machines without a driver).
EncodeTiled encoder() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    });
    return fn;
}

// Whether the current device is a compute-capability-10 part; -1 unknown, cached per device.
bool device_is_sm100() {
    static int cache[64];
    static std::once_flag once;
    std::call_once(once, [] { for (int &c : cache) c = -1; });
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return false; }
    if (cache[dev] < 0) {
        int major = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cache[dev] = major == 10 ? 1 : 0;
    }
    return cache[dev] == 1;
}

// The reference's in-place rule (crates/dash-ops/src/attention/cube.rs:428-461), which is also what
// a TMA tensor map needs: last stride 1, the others multiples of 16 bytes, base 16-byte aligned.
bool tma_strides(const int64_t *stride) {
    if (stride[3] != 1) return false;
    for (int i = 0; i < 3; ++i)
        if (stride[i] % 8 != 0 || stride[i] < 0) return false;
    return true;
}
bool tma_base(const void *ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0; }

// A [B, T, H, d] tensor of 16-bit elements (d = 64, 128 or 256) as a 4-D map (d, h, t, b) with boxes of
// 64 x heads x (rows / heads) x 1 and the 128-byte swizzle: each load brings 128 rows of 128 bytes, of one
// head, or of `heads` query heads of one group side by side (row = token * heads + head).
// (dtype DASH_ATTN_F32: the fused backward's accumulator, 32 f32 columns to a 128-byte box row.)
bool encode_uncached(CUtensorMap *map, int dtype, const void *ptr, int b, int t, int h, const int64_t *stride, int rows, int d, int heads) {
    EncodeTiled fn = encoder();
    if (!fn) return false;
    const bool f32 = dtype == DASH_ATTN_F32;
    auto bytes = [f32](int64_t elems) { return static_cast<cuuint64_t>(elems) * (f32 ? 4 : 2); };
    cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)h, (cuuint64_t)t, (cuuint64_t)b};
    // A dimension of extent 1 never moves: give it any legal stride.
    cuuint64_t strides[3] = {h > 1 ? bytes(stride[2]) : 256, t > 1 ? bytes(stride[1]) : 256, b > 1 ? bytes(stride[0]) : 256};
    for (cuuint64_t s : strides)
        if (s == 0 || s % 16 != 0 || s >= (1ull << 40)) return false;
    cuuint32_t box[4] = {f32 ? 32u : 64u, (cuuint32_t)heads, (cuuint32_t)(rows / heads), 1};
    cuuint32_t elem[4] = {1, 1, 1, 1};
    CUtensorMapDataType dt = f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : dtype == DASH_ATTN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = fn(map, dt, 4, const_cast<void *>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// A tensor map is a pure function of the address and the geometry it was encoded from, not of the
// bytes behind the address, and a training loop or a decoder calls with the same buffers step after
// step: the last maps are kept, keyed on everything the encoder reads, so that a repeated call costs
// a lookup instead of a trip through the driver per tensor (short calls are bound by exactly that
// host time, crates/dash-ops/src/attention.rs:123-127).
struct MapKey {
    const void *ptr;
    int dtype, b, t, h, rows, d, heads;
    int64_t s0, s1, s2;
    bool operator==(const MapKey &o) const {
        return ptr == o.ptr && dtype == o.dtype && b == o.b && t == o.t && h == o.h && rows == o.rows && d == o.d &&
               heads == o.heads && s0 == o.s0 && s1 == o.s1 && s2 == o.s2;
    }
};
struct MapSlot {
    MapKey key;
    CUtensorMap map;
    bool used;
};
constexpr int MAP_SLOTS = 64, MAP_WAYS = 4;
MapSlot g_maps[MAP_SLOTS];
unsigned g_map_turn[MAP_SLOTS / MAP_WAYS];
std::mutex g_map_mutex;
std::atomic<uint64_t> g_map_encodes{0};

bool encode(CUtensorMap *map, int dtype, const void *ptr, int b, int t, int h, const int64_t *stride, int rows = 128, int d = 128,
            int heads = 1) {
    const MapKey key{ptr, dtype, b, t, h, rows, d, heads, stride[0], stride[1], stride[2]};
    uint64_t x = reinterpret_cast<uintptr_t>(ptr) >> 4;
    x ^= (uint64_t)(unsigned)t * 0x9E3779B97F4A7C15ull + (uint64_t)(unsigned)h * 0xC2B2AE3D27D4EB4Full + (uint64_t)(unsigned)(rows + d + dtype + heads);
    x ^= x >> 29;
    const int set = (int)(x % (MAP_SLOTS / MAP_WAYS));
    {
        std::lock_guard<std::mutex> lock(g_map_mutex);
        for (int w = 0; w < MAP_WAYS; ++w) {
            const MapSlot &s = g_maps[set * MAP_WAYS + w];
            if (s.used && s.key == key) { *map = s.map; return true; }
        }
    }
    if (!encode_uncached(map, dtype, ptr, b, t, h, stride, rows, d, heads)) return false;
    g_map_encodes.fetch_add(1, std::memory_order_relaxed);
    std::lock_guard<std::mutex> lock(g_map_mutex);
    MapSlot &s = g_maps[set * MAP_WAYS + (g_map_turn[set]++ % MAP_WAYS)];
    s.key = key;
    s.map = *map;
    s.used = true;
    return true;
}

float resolved_scale(const dash_attn_params *p) {
    return p->has_scale ? p->scale : (float)(1.0 / std::sqrt((double)p->d));
}

// Query heads of one key-value group that share a tile of 128 query rows (row = token * 2^pack + head), as a
// power of two: the largest that divides the group, up to eight.  The rows of a tile sweep the union of their
// tokens' keys, so a tile of 128 tokens of one head pays, at the diagonal, at a window's edges and where two
// packed sequences meet, for up to 128 tokens' worth of keys its rows do not see; a tile of 128 / 2^pack
// tokens for that fraction of them, and a call of few queries fills its tiles with heads.  The keys are the
// same for every head of the group, so nothing is loaded more often.  (Eight: 16 tokens a tile, a quarter of
// the forward's sub-step; more would gain nothing.)  Side by side with tiles of 128 tokens: the training step of 8
// packed sequences, 16384 tokens, 32 / 8 heads, 1975 -> 1898 us; of 16 sequences, 65536 tokens, window 4096, 16 / 4
// heads, 5668 -> 5500 us; a prompt chunk of 500 against 7700 keys 131 -> 129 us.  Where the grid's second extent could not hold that many
// tiles of tokens, fewer heads.
int pack_log2(int group, int tq) {
    int p = 0;
    while (p < 3 && group % (2 << p) == 0 && ((int64_t)tq + (64 >> p) - 1) / (64 >> p) <= 65535) ++p;
    return p;
}

}  // namespace

uint64_t sm100_tensor_map_encodes() { return g_map_encodes.load(std::memory_order_relaxed); }

// What sm100_takes asks of a call's parameters (of its pointers and of the device: there).
static bool parameters_taken(const dash_attn_params *p, int backward, bool any_size) {
    if (backward && !tma_strides(p->do_stride)) return false;  // dO's base is checked at launch
    if (p->dtype != DASH_ATTN_BF16 && p->dtype != DASH_ATTN_F16) return false;
    // Head dimensions 64 and 256 only from 128 queries and 128 keys on: below that there is a single
    // partial tile of queries or of keys (one block per head), the tensor cores gain nothing, and the
    // generic kernels' f32 FMA sums keep the log-sum-exp within the one or two units in the last place
    // that the reference's records allow at those sizes.  (`any_size`, a switch for tests, lifts the
    // size rule, so that the records themselves can be run through the tensor-core kernels.)
    // At 256 the forward is the one-tile kernel and the backward the three passes of bwd256_sm100.cu.
    const bool big = any_size || (p->tq >= 128 && p->tk >= 128);
    if (p->d != 128 && !((p->d == 64 || p->d == 256) && big)) return false;
    const float scale = resolved_scale(p);
    if (!(scale > 0.f) || !std::isfinite(scale)) return false;  // the row maximum is taken before scaling
    if (!tma_strides(p->q_stride) || !tma_strides(p->k_stride) || !tma_strides(p->v_stride)) return false;
    return p->hq <= 65535 && p->b <= 65535;   // grid extents
}

bool sm100_takes(const dash_attn_params *p, const void *q, const void *k, const void *v, int backward, bool any_size) {
    if (!parameters_taken(p, backward, any_size)) return false;
    if (!q || !k || !v || !tma_base(q) || !tma_base(k) || !tma_base(v)) return false;
    if (!device_is_sm100() || !encoder()) return false;
    return true;
}

// Over how many blocks the forward splits the keys of a tile of queries.  A call of few queries - a chunk of a prompt
// against a long cache - has fewer tiles than the GPU has multiprocessors, each a long sweep: cut into runs of keys they
// fill it.  Estimated in steps of 64 keys (128 at D 256): a block's share of its sweep plus what a block costs however
// short its sweep (set-up, the first tiles' flight, the output: about six steps of the two-tile kernel, three of the
// other's, which are twice as long), times the waves of blocks; a split also pays for the merge's launch (five and three
// steps) and for the f32 rows of its parts, written and read at 2.3 TB/s (a step is 0.95 us, the other's 1.8).  Under
// causality tiles differ, the long ones first: waves are counted on the mean, the last wave, where it is not full, goes
// from the shortest towards the mean with its share of the multiprocessors, and the longest tile is a bound of its own.
// Packed batches, whose lengths the host does not know, are not split.
// At forced numbers of splits over 240 calls (130 to 5000 queries, D 64 to 256, 4 to 32 heads) the pick is never slower
// than the whole sweep.  With the parts unpriced, 3000 tokens of 12 / 4 heads of 128 were split in two, 65.7 us against 53.4;
// with the last wave as long as the others, 2380 queries against 6897 keys, 8 / 2 heads of 256 (150 blocks), in three, 143
// against 123.  (A chunk of 500 queries against 8200 keys, 32 / 8 heads, 64 tiles: the figures at fwd_merge.cu.)
int forward_splits(const dash_attn_params *p) {
    if (p->mask_kind == DASH_ATTN_MASK_PACKED || p->hkv <= 0 || p->tq <= 0) return 1;
    const bool one = p->d == 256;
    const int pack = pack_log2(p->hq / p->hkv, p->tq);
    const int64_t tokens = (one ? 128 : 256) >> pack, step = one ? 128 : 64, sms = 148;
    const int64_t tiles = (p->tq + tokens - 1) / tokens, blocks = tiles * (p->hq >> pack) * p->b;
    if (blocks >= 2 * sms) return 1;
    int64_t longest = p->tk, mean = p->tk, shortest = p->tk;
    // A side that reaches past every key is no bound (and must not be added to).
    const int64_t none = (int64_t)p->tq + p->tk + 1;
    auto side = [&](int64_t reach) { return p->has_window && reach >= 0 && reach < none ? reach : int64_t(-1); };
    const int64_t left = side(p->window_left), right = p->causal ? 0 : side(p->window_right);
    if (right >= 0) {   // query i sees keys up to i + tk - tq + right
        const int64_t last = std::min<int64_t>(p->tk, p->tk + right), first = std::min<int64_t>(p->tk, std::max<int64_t>(p->tk - p->tq + right + tokens, 0));
        longest = last;
        mean = (first + last) / 2;
        shortest = first;
    }
    if (left >= 0) {
        const int64_t reach = left + std::max<int64_t>(right, 0) + tokens;
        longest = std::min(longest, right < 0 ? p->tk : reach);
        mean = std::min(mean, longest);
        shortest = std::min(shortest, longest);
    }
    const int64_t l = (longest + step - 1) / step, m = (mean + step - 1) / step, n = (shortest + step - 1) / step, fixed = one ? 3 : 6;
    const double merge = one ? 3 : 5, part = (double)p->b * p->tq * p->hq * p->d * sizeof(float) / (one ? 4.1e6 : 2.2e6);
    auto cost = [&](int64_t s) {
        const int64_t full = blocks * s / sms, rest = blocks * s % sms, ms = (m + s - 1) / s, ns = (n + s - 1) / s;
        const double last = rest ? ns + (ms - ns) * ((double)rest / sms) + fixed : 0.;
        return std::max(full * (ms + fixed) + last, (double)((l + s - 1) / s + fixed)) + (s > 1 ? merge + s * part : 0.);
    };
    int best = 1;
    for (int s = 2; s <= 32 && l / s >= 2 && tiles * s <= 65535; ++s)
        if (cost(s) < 0.95 * cost(1) && cost(s) < cost(best)) best = s;
    return best;
}
static size_t split_rows(const dash_attn_params *p, int splits) { return (size_t)splits * p->b * p->tq * p->hq; }
static size_t split_lse_bytes(const dash_attn_params *p, int splits) { return (sizeof(float) * split_rows(p, splits) + 255) & ~size_t(255); }
static size_t split_bytes(const dash_attn_params *p, int splits) {
    return splits > 1 ? split_lse_bytes(p, splits) + sizeof(float) * split_rows(p, splits) * p->d : 0;
}
size_t sm100_forward_workspace(const dash_attn_params *p, bool any_size) {
    return parameters_taken(p, 0, any_size) ? split_bytes(p, forward_splits(p)) : 0;   // a call the generic kernels take is not split
}
// Whether two blocks share each unit (128 keys of a key-value head) of the key and value gradients, half its steps each (D 64 and
// 128; D 256 has a rule of its own).  A unit sweeps the queries of all heads of its group that see it, and with few units the
// longest sweep is the kernel's length; with two blocks to a unit it is half that, a second set-up and the meeting of the two.  The
// rule looks at no number of heads, so that a head slice of a packed batch keeps the whole call's bits: key blocks so few that
// with eight key-value heads (two, where groups are of eight) twice the units still start at once, and sweeps of five steps of
// 128 rows or more.  Backward, one block | two (us): 500 tokens, 16 / 4 heads of 128, 36.7 | 28.4, 32 / 8 39.2 | 30.9; 1000 in three,
// 32 / 8, 37.8 | 37.2, 16 / 8 24.9 | 26.8; 1152, 16 / 8, 42.6 | 36.0, 24 / 8 56.6 | 43.9; groups of eight, 8 / 1, 500 62.8 | 41.7, 4700 in two
// 350 | 188, 16 / 2 4700 505 | 274, 32 / 4 2400 267 | 158, 64 / 8 1800 216 | 197; heads of 64 the same.
// What the slices' bits cost: with more key-value heads the doubled blocks come in waves, and the pair loses what a line on the units
// (about 100) would keep - 32 / 16 heads, 500 tokens, 26.8 | 26.8, 1000 45.9 | 59.5, 1152 53.4 | 67.8; 64 / 32, 500, 37.0 | 49.3; 64 / 16,
// 500, 47.6 | 45.2, 1152 96.2 | 110; 64 / 8, 2400, 308 | 319, 4700 1145 | 1204, in four 411 | 441; 128 / 16, 4700 in four, 834 | 903.
constexpr int64_t PAIR_BLOCKS = 9, PAIR_BLOCKS_GROUP8 = 37, PAIR_ROWS = 5 * 128;
static bool backward_pairs(const dash_attn_params *p) {
    if (p->d != 64 && p->d != 128) return false;
    const int64_t blocks = (int64_t)p->b * ((p->tk + 127) / 128), group = p->hq / p->hkv;
    const int64_t none = (int64_t)p->tq + p->tk + 1;
    int64_t queries = p->mask_kind == DASH_ATTN_MASK_PACKED ? p->tq / std::max(p->cu_seqlens_q_len - 1, 1) : p->tq;
    if (p->has_window && p->window_left >= 0 && p->window_left < none && (p->causal || (p->window_right >= 0 && p->window_right < none)))
        queries = std::min(queries, p->window_left + (p->causal ? 0 : p->window_right) + 128);
    return queries * group >= PAIR_ROWS && group >= 2 && blocks <= (group >= 8 ? PAIR_BLOCKS_GROUP8 : PAIR_BLOCKS);
}
// Whether a call whose caller lets dQ be summed in any order takes the form that makes use of it, five products with dQ added by
// reductions in L2 (D 64, 128).  It shares the scores but not its
// units: the seven-product form fills what few units leave idle with dq's tiles, and at D 128 the reductions cost what the two products
// do.  Backward, 170 calls (us, seven products | five): D 64 packed, 16 / 4 heads, 4000 tokens, 128 units, 71 | 87, 8000, 252 units,
// 148 | 133, 30000 960 | 758; padded, 8 of 256, 12 / 4, 64 units, 24 | 25, 4 of 256, 12 / 12, 96 units, 19 | 17, 32 of 1000,
// 3072 units, 596 | 378.  D 128 packed, 1000 to 30000 tokens, 60 to 99.7 % of the speed; padded, 8 of 500, 12 / 12, 384 units,
// 77 | 81, 16 of 1000, 12 / 4, 512 units, 309 | 293, 32 of 1000, 1024 units, 603 | 507.
constexpr int64_t FIVE_UNITS_64 = 90, FIVE_UNITS_64_PACKED = 240, FIVE_UNITS_128 = 500;
static bool fused_backward(const dash_attn_params *p) {
    if (p->deterministic || (p->d != 64 && p->d != 128) || backward_pairs(p)) return false;
    const int64_t units = (int64_t)p->b * ((p->tk + 127) / 128) * p->hkv;
    const bool packed = p->mask_kind == DASH_ATTN_MASK_PACKED;
    return p->d == 64 ? units >= (packed ? FIVE_UNITS_64_PACKED : FIVE_UNITS_64) : !packed && units >= FIVE_UNITS_128;
}
static size_t dq_acc_bytes(const dash_attn_params *p) {
    return (sizeof(float) * (size_t)p->b * p->tq * p->hq * p->d + 255) & ~size_t(255);
}
size_t sm100_backward_workspace(const dash_attn_params *p) {
    return bwd_sm100_order_bytes(p->b, p->tk, p->hkv) + (fused_backward(p) ? dq_acc_bytes(p) : 0);
}

cudaError_t sm100_forward(const dash_attn_params *p, const TrainArgs &a, void *workspace, size_t workspace_bytes, cudaStream_t stream,
                          int *launches, std::string &err) {
    // The two-tile kernel shares every K / V tile between two query tiles; DASH_ATTN_FWD_TILES=1
    // keeps the one-tile kernel (for comparison runs).
    static const bool one_tile = [] { const char *e = std::getenv("DASH_ATTN_FWD_TILES"); return e && std::atoi(e) == 1; }();
    const int kv_rows = 128;
    CUtensorMap tq, tk, tv, to;
    const int64_t o_stride[4] = {(int64_t)p->tq * p->hq * p->d, (int64_t)p->hq * p->d, p->d, 1};   // the output is contiguous
    const int pack = pack_log2(p->hq / p->hkv, p->tq);
    if (!encode(&to, p->dtype, a.out, p->b, p->tq, p->hq, o_stride, 128, p->d, 1 << pack) ||
        !encode(&tq, p->dtype, a.q.ptr, p->b, p->tq, p->hq, p->q_stride, 128, p->d, 1 << pack) ||
        !encode(&tk, p->dtype, a.k.ptr, p->b, p->tk, p->hkv, p->k_stride, kv_rows, p->d) ||
        !encode(&tv, p->dtype, a.v.ptr, p->b, p->tk, p->hkv, p->v_stride, kv_rows, p->d)) {
        err = "attention: the driver refused a TMA tensor map over the inputs";
        return cudaSuccess;
    }
    Sm100FwdArgs f{};
    f.b = p->b; f.tq = p->tq; f.tk = p->tk; f.hq = p->hq; f.hkv = p->hkv; f.d = p->d;
    f.scale = a.scale;
    f.scale_log2 = a.scale * 1.4426950408889634f;
    f.out = a.out;
    f.lse = a.lse;
    f.mask = a.mask;
    f.pack = pack;
    // Without scratch for the parts (or with less than the query asks for) the keys stay in one block.
    const int splits = forward_splits(p);
    const bool split = splits > 1 && workspace && workspace_bytes >= split_bytes(p, splits) && reinterpret_cast<uintptr_t>(workspace) % 256 == 0 && !one_tile;
    f.splits = split ? splits : 1;
    if (split) {
        f.part_lse = static_cast<float *>(workspace);
        f.part_o = reinterpret_cast<float *>(static_cast<char *>(workspace) + split_lse_bytes(p, f.splits));
    }
    cudaError_t e = ((one_tile && p->d == 128) || p->d == 256) ? launch_fwd_sm100(p->dtype, tq, tk, tv, f, stream) : launch_fwd2_sm100(p->dtype, tq, tk, tv, to, f, stream);
    *launches += 1;
    if (e == cudaSuccess && split) {
        e = launch_fwd_merge(p->dtype, f, stream);
        *launches += 1;
    }
    return e;
}

// Units that need no launch order: one a multiprocessor, at D 256 (two passes, two blocks to a unit) a quarter of that.  Units shared by two
// blocks take the first line too, though 75 to 148 of them do not all start at once: of 90 such calls the order gained 2 % in three and
// cost up to 10 in the others (32 / 16 heads of 128, 700 tokens, 96 units, 41.1 us without, 45.2 with).
constexpr int AT_ONCE = 148, AT_ONCE_256 = 37;

cudaError_t sm100_backward(const dash_attn_params *p, const TrainArgs &a, void *workspace, cudaStream_t stream, int *launches,
                           bool *atomic, std::string &err) {
    const bool fused = fused_backward(p);
    *atomic = fused;
    Sm100BwdMaps m;
    float *dq_acc = fused ? reinterpret_cast<float *>(static_cast<char *>(workspace) + bwd_sm100_order_bytes(p->b, p->tk, p->hkv)) : nullptr;
    const void *q = a.q.ptr, *k = a.k.ptr, *v = a.v.ptr, *g = a.dout.ptr;
    const int64_t dq_stride[4] = {(int64_t)p->tq * p->hq * p->d, (int64_t)p->hq * p->d, p->d, 1};   // the gradients are contiguous
    const int pack = pack_log2(p->hq / p->hkv, p->tq), heads = 1 << pack;
    bool ok = encode(&m.dq128, p->dtype, a.dq, p->b, p->tq, p->hq, dq_stride, 128, p->d, heads) &&
              encode(&m.q128, p->dtype, q, p->b, p->tq, p->hq, p->q_stride, 128, p->d, heads) &&
              encode(&m.do128, p->dtype, g, p->b, p->tq, p->hq, p->do_stride, 128, p->d, heads) &&
              encode(&m.k128, p->dtype, k, p->b, p->tk, p->hkv, p->k_stride, 128, p->d) &&
              encode(&m.v128, p->dtype, v, p->b, p->tk, p->hkv, p->v_stride, 128, p->d);
    const int64_t dkv_stride[4] = {(int64_t)p->tk * p->hkv * p->d, (int64_t)p->hkv * p->d, p->d, 1};
    if (p->d != 256) ok = ok && encode(&m.dk128, p->dtype, a.dk, p->b, p->tk, p->hkv, dkv_stride, 128, p->d) &&
                          encode(&m.dv128, p->dtype, a.dv, p->b, p->tk, p->hkv, dkv_stride, 128, p->d);
    if (ok && fused) ok = encode(&m.dq_acc, DASH_ATTN_F32, dq_acc, p->b, p->tq, p->hq, dq_stride, 128, p->d, heads);
    else if (ok) m.dq_acc = m.dq128;   // not read
    if (!ok) {
        err = "attention_backward: the driver refused a TMA tensor map over the inputs";
        return cudaSuccess;
    }
    Sm100BwdArgs f{};
    f.b = p->b; f.tq = p->tq; f.tk = p->tk; f.hq = p->hq; f.hkv = p->hkv; f.d = p->d;
    f.scale = a.scale;
    f.scale_log2 = a.scale * 1.4426950408889634f;
    f.lse = a.lse;
    f.delta = a.delta;
    f.dq = a.dq; f.dk = a.dk; f.dv = a.dv;
    f.mask = a.mask;
    f.order = static_cast<int *>(workspace);
    f.dq_acc = dq_acc;
    f.pack = pack;
    f.pairs = backward_pairs(p) ? 1 : 0;
    // The plan's one block and delta run side by side; then dkdv, and dq beside its last waves (neither reads what
    // the other writes).
    cudaError_t e = launch_bwd_plan(f, p->d == 256 ? AT_ONCE_256 : AT_ONCE, stream, launches);
    if (e == cudaSuccess) e = launch_generic_delta(p->dtype, a, stream, launches, f.order != nullptr);
    if (e != cudaSuccess) return e;
    if (p->d == 256) return launch_bwd256_sm100(p->dtype, m, f, stream, launches);
    return launch_bwd_sm100(p->dtype, m, f, stream, launches);
}

}  // namespace dash
