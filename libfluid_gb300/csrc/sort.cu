// sort.cu -- stable LSD radix sort of (key, value) u32 pairs, one sweep per digit.
//
// Replaces the reference's single-threaded std::sort of ~80-byte particle records by
// z-index (include/fluid/oclsph.hpp:733-743).  Unlike std::sort this sort is stable:
// particles of one cell keep their previous relative order, so the sorted order (and
// every sum over it) is a deterministic function of the input.
//
// Per pass (8-bit digit): each CTA takes the next tile id from an atomic counter,
// ranks its 4096 keys (1024 in a short sort) with warp-level match_any (in index order, hence stable),
// publishes its per-digit counts, looks back over earlier tiles' published counts
// (decoupled look-back) to find where its keys start, and scatters.  The digits of all
// passes are counted before the first: by a kernel of their own, or by the one that makes
// the keys (digit_counts.cuh); each tile sums the counts of its pass itself.  Every
// look-back wait is bounded.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "digit_counts.cuh"
#include "fgb_device.cuh"
#include "fgb_internal.h"

namespace fgb {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Keys a thread takes.  A short sort waits for its few tiles' ranking, key after key: a pass
// over 4 k or 14 k keys takes 2 us less with 4 than with 16; from 64 k keys on they are equal,
// and for 1 M, where more tiles are more to look back over, 16 take 14 us and 4 take 19.
constexpr int kSortItems = 16, kShortItems = 4;
constexpr uint64_t kShortSort = 32768;  // keys below which a sort is short

constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagInclusive = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1u;

__global__ void __launch_bounds__(256) k_radix_histogram(const uint32_t *__restrict__ keys, uint32_t n,
                                                         int passes, uint32_t *__restrict__ hist) {
    __shared__ DigitCounts counts;
    counts.clear();
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        counts.add(keys[i], passes);
    __syncthreads();
    counts.give(hist, passes);
}

template <int kItems>
__global__ void __launch_bounds__(kSortThreads) k_onesweep(
    const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in,
    uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out, uint32_t n, int shift,
    const uint32_t *__restrict__ counts, uint32_t *status, uint32_t *tile_counter, uint32_t *err,
    LookbackCtl ctl) {
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_hist[kSortWarps][kRadix + 1];
    __shared__ uint32_t s_base[kRadix + 1];
    __shared__ uint32_t s_before[kSortWarps];

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
    for (int i = tid; i < kSortWarps * (kRadix + 1); i += kSortThreads) (&s_hist[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * (uint32_t)(kSortThreads * kItems) + (uint32_t)w * 32u * kItems;

    uint32_t k[kItems], v[kItems], rank[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        uint32_t idx = base + (uint32_t)i * 32u + (uint32_t)lane;
        bool ok = idx < n;
        k[i] = ok ? keys_in[idx] : 0u;
        v[i] = ok ? vals_in[idx] : 0u;
    }
    const uint32_t lt = lanemask_lt();
    // the keys with a digit below tid: the counts of the earlier digits
    uint32_t below = counts[tid];
    {
        const uint32_t own = below;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, below, o);
            if (lane >= o) below += y;
        }
        if (lane == 31) s_before[w] = below;
        below -= own;
    }
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        uint32_t idx = base + (uint32_t)i * 32u + (uint32_t)lane;
        uint32_t d = idx < n ? ((k[i] >> shift) & (kRadix - 1)) : (uint32_t)kRadix;
        uint32_t peers = __match_any_sync(0xffffffffu, d);
        uint32_t before = s_hist[w][d];
        __syncwarp();
        rank[i] = before + __popc(peers & lt);
        if ((peers & lt) == 0) s_hist[w][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();

    // tid == digit: tile count and the exclusive prefix over warps
    {
        const uint32_t d = (uint32_t)tid;
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < kSortWarps; ++ww) {
            uint32_t c = s_hist[ww][d];
            s_hist[ww][d] = run;
            run += c;
        }
        uint32_t *my = status + (size_t)tile * kRadix + d;
        // a skipped tile (fgb_test_lookback_fault only) publishes nothing
        const bool publish = tile != ctl.skip_tile;
        uint32_t excl = 0;
        if (tile == 0) {
            if (publish) st_relaxed(my, kFlagInclusive | run);
        } else {
            if (publish) st_relaxed(my, kFlagAggregate | run);
            int t = (int)tile - 1;
            uint32_t spins = 0;
            while (t >= 0) {
                uint32_t s = ld_relaxed(status + (size_t)t * kRadix + d);
                if ((s & ~kValueMask) == 0) {
                    // a timed-out wait keeps the partial prefix: a sum over a subset of
                    // the earlier tiles' counts, so every scatter index stays below n
                    if (++spins > ctl.spin_limit) {
                        raise_error(err, ERR_SORT_LOOKBACK);
                        break;
                    }
                    continue;
                }
                excl += s & kValueMask;
                if (s & kFlagInclusive) break;
                --t;
            }
            if (publish) st_relaxed(my, kFlagInclusive | (excl + run));
        }
        for (int ww = 0; ww < w; ++ww) below += s_before[ww];
        s_base[d] = below + excl;
    }
    __syncthreads();

#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        uint32_t idx = base + (uint32_t)i * 32u + (uint32_t)lane;
        if (idx < n) {
            uint32_t d = (k[i] >> shift) & (kRadix - 1);
            uint32_t pos = s_base[d] + s_hist[w][d] + rank[i];
            if (pos < n) {  // only a timed-out look-back can produce pos >= n
                keys_out[pos] = k[i];
                vals_out[pos] = v[i];
            } else {
                raise_error(err, ERR_SORT_LOOKBACK);
            }
        }
    }
}

struct SortLayout {
    size_t hist, counters, status, alt_keys, alt_vals, total;
    uint32_t tiles;
};

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

SortLayout sort_layout(uint64_t n, int items = kSortItems) {
    SortLayout L;
    const uint64_t tile = (uint64_t)kSortThreads * items;
    L.tiles = (uint32_t)((n + tile - 1) / tile);
    size_t o = 0;
    L.hist = o;
    o = align256(o + sizeof(uint32_t) * kMaxPasses * kRadix);
    L.counters = o;
    o = align256(o + sizeof(uint32_t) * kMaxPasses);
    L.status = o;
    o = align256(o + sizeof(uint32_t) * (size_t)kMaxPasses * (L.tiles ? L.tiles : 1) * kRadix);
    L.alt_keys = o;
    o = align256(o + sizeof(uint32_t) * (n ? n : 1));
    L.alt_vals = o;
    o = align256(o + sizeof(uint32_t) * (n ? n : 1));
    L.total = o;
    return L;
}

}  // namespace

namespace {
std::atomic<uint64_t> g_lookback{(uint64_t)kSpinLimit << 32 | 0xffffffffull};
}  // namespace

LookbackCtl lookback_ctl() {
    const uint64_t v = g_lookback.load(std::memory_order_relaxed);
    return LookbackCtl{(uint32_t)v, (uint32_t)(v >> 32)};
}

uint64_t radix_scratch_bytes(uint64_t n) { return sort_layout(n).total; }

uint64_t radix_scratch_bytes_short(uint64_t n) {
    return std::max(sort_layout(n).total, sort_layout(std::min(n, kShortSort), kShortItems).total);
}

// Whether a sort of n keys in a scratch of that size takes the short tiles.
static bool short_sort(uint64_t n, uint64_t scratch_bytes) {
    return n < kShortSort && scratch_bytes >= sort_layout(n, kShortItems).total;
}

int radix_passes(uint32_t key_bits) {
    int p = (int)((key_bits + kRadixBits - 1) / kRadixBits);
    return p < 1 ? 1 : p;
}

uint32_t *radix_state(uint64_t n, uint32_t key_bits, void *scratch, uint64_t scratch_bytes, uint64_t *words) {
    const SortLayout L = sort_layout(n, short_sort(n, scratch_bytes) ? kShortItems : kSortItems);
    *words = (L.status - L.counters) / sizeof(uint32_t) + (uint64_t)radix_passes(key_bits) * L.tiles * kRadix;
    return (uint32_t *)((char *)scratch + L.counters);
}

cudaError_t radix_sort_pairs(const uint32_t *keys_in, const uint32_t *vals_in, uint32_t *keys_out,
                             uint32_t *vals_out, uint64_t n, uint32_t key_bits, void *scratch,
                             uint64_t scratch_bytes, cudaStream_t stream, uint32_t *err,
                             uint64_t *launches, const uint32_t *counted) {
    if (n == 0) return cudaSuccess;
    if (key_bits > 32 || n > (uint64_t)kValueMask) return cudaErrorInvalidValue;
    const bool brief = short_sort(n, scratch_bytes);
    SortLayout L = sort_layout(n, brief ? kShortItems : kSortItems);
    if (scratch_bytes < L.total || scratch == nullptr) return cudaErrorInvalidValue;
    char *s = (char *)scratch;
    uint32_t *hist = (uint32_t *)(s + L.hist);
    uint32_t *counters = (uint32_t *)(s + L.counters);
    uint32_t *status = (uint32_t *)(s + L.status);
    uint32_t *alt_k = (uint32_t *)(s + L.alt_keys);
    uint32_t *alt_v = (uint32_t *)(s + L.alt_vals);
    const int passes = radix_passes(key_bits);
    const LookbackCtl ctl = lookback_ctl();
    if (!counted) {
        // hist, counters and the status words of every pass start at zero
        cudaError_t e = cudaMemsetAsync(s, 0, L.alt_keys, stream);
        if (e != cudaSuccess) return e;
        int blocks = (int)((n + 255) / 256);
        if (blocks > 1216) blocks = 1216;
        k_radix_histogram<<<blocks, 256, 0, stream>>>(keys_in, (uint32_t)n, passes, hist);
        counted = hist;
        if (launches) *launches += 1;
    }
    const uint32_t *src_k = keys_in, *src_v = vals_in;
    for (int p = 0; p < passes; ++p) {
        bool to_out = ((passes - 1 - p) % 2) == 0;
        uint32_t *dk = to_out ? keys_out : alt_k;
        uint32_t *dv = to_out ? vals_out : alt_v;
        auto kernel = brief ? k_onesweep<kShortItems> : k_onesweep<kSortItems>;
        kernel<<<L.tiles, kSortThreads, 0, stream>>>(
            src_k, src_v, dk, dv, (uint32_t)n, p * kRadixBits, counted + p * kRadix,
            status + (size_t)p * L.tiles * kRadix, counters + p, err, ctl);
        src_k = dk;
        src_v = dv;
    }
    if (launches) *launches += passes;
    return cudaGetLastError();
}

}  // namespace fgb

extern "C" {

uint64_t fgb_radix_sort_scratch_bytes(uint64_t n) {
    // one extra u32 at the end holds the device error flag of the standalone call
    return fgb::radix_scratch_bytes(n) + 256;
}

int fgb_radix_sort_pairs_u32(const uint32_t *d_keys_in, const uint32_t *d_vals_in, uint32_t *d_keys_out,
                             uint32_t *d_vals_out, uint64_t n, uint32_t key_bits, void *d_scratch,
                             uint64_t scratch_bytes, void *cuda_stream) {
    if (n && (!d_keys_in || !d_vals_in || !d_keys_out || !d_vals_out))
        return fgb::fail(FGB_ERR_INVALID, "radix sort: null pointer");
    if (key_bits == 0 || key_bits > 32) return fgb::fail(FGB_ERR_INVALID, "radix sort: key_bits must be 1..32");
    if (scratch_bytes < fgb_radix_sort_scratch_bytes(n))
        return fgb::fail(FGB_ERR_INVALID, "radix sort: scratch smaller than fgb_radix_sort_scratch_bytes(n)");
    uint64_t core = fgb::radix_scratch_bytes(n);
    uint32_t *err = (uint32_t *)((char *)d_scratch + core);
    cudaStream_t st = (cudaStream_t)cuda_stream;
    cudaError_t e = cudaMemsetAsync(err, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess)
        e = fgb::radix_sort_pairs(d_keys_in, d_vals_in, d_keys_out, d_vals_out, n, key_bits, d_scratch, core, st,
                                  err, nullptr, nullptr);
    if (e != cudaSuccess) return fgb::fail_cuda(e, "radix sort");
    return FGB_OK;
}

int fgb_radix_sort_error(const void *d_scratch, uint64_t n, void *cuda_stream, uint32_t *flags) {
    if (!d_scratch || !flags) return fgb::fail(FGB_ERR_INVALID, "radix sort error: null argument");
    return fgb::read_clear_flag((char *)d_scratch + fgb::radix_scratch_bytes(n), (cudaStream_t)cuda_stream, flags,
                                "radix sort error");
}

int fgb_test_lookback_fault(uint32_t skip_tile, uint32_t spin_limit) {
    if (skip_tile != 0xffffffffu && spin_limit == 0)
        return fgb::fail(FGB_ERR_INVALID, "lookback fault: a skipped tile needs a spin limit above 0");
    if (skip_tile == 0xffffffffu) spin_limit = fgb::kSpinLimit;
    fgb::g_lookback.store((uint64_t)spin_limit << 32 | skip_tile, std::memory_order_relaxed);
    return FGB_OK;
}
}
