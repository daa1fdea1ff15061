// mk_sort.cu — stable LSD onesweep radix sort of (63-bit key, 32-bit value).
//
// Replaces the reference's bitonic network (lbvh.wgsl:132-217, 54-77
// full-buffer passes per tick) with one histogram pass over the keys plus one
// single-pass "onesweep" scatter per 8-bit digit: each tile ranks its keys
// with warp match-any, publishes per-digit counts, and learns its global
// offsets by decoupled look-back over the preceding tiles.  Stability
// (equal keys keep input order) gives the reference's (code, index)
// tie-break when the values are collider indices in ascending order.
#include "mk_device.cuh"
#include "mk_internal.h"

#include <atomic>

namespace mk {

constexpr uint32_t kSortThreads = 256;
constexpr uint32_t kRadixBins = 256;
constexpr uint32_t kLookbackWindow = 16;   // predecessor tiles read per look-back round trip

// 30-bit digit look-back words: bits 30-31 status, 0-29 count.
constexpr uint32_t kDigitAggregate = 1u << 30;
constexpr uint32_t kDigitInclusive = 2u << 30;
constexpr uint32_t kDigitCountMask = (1u << 30) - 1;

// Digit counts of every pass over the keys, and the look-back words that the
// passes will use for this n cleared.  `s_hist` holds 8 x 256 words.
__device__ __forceinline__ void radix_histogram(const uint64_t* __restrict__ keys, uint32_t n, uint32_t passes,
                                                uint32_t* __restrict__ hist /* passes x 256 */,
                                                uint32_t* __restrict__ lookback, uint64_t lookback_pass_words,
                                                uint32_t tile_keys, uint32_t* s_hist) {
    const uint64_t used = (uint64_t)((n + tile_keys - 1) / tile_keys) * kRadixBins;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < used * passes;
         w += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t pass = w / used, off = w % used;
        lookback[pass * lookback_pass_words + off] = 0u;
    }
    for (uint32_t i = threadIdx.x; i < 8 * kRadixBins; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint64_t k = __ldcg(keys + i);
        for (uint32_t p = 0; p < passes; ++p) atomicAdd(&s_hist[p * kRadixBins + ((k >> (8 * p)) & 0xffu)], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < passes * kRadixBins; i += blockDim.x) {
        uint32_t v = s_hist[i];
        if (v) atomicAdd(&hist[i], v);
    }
}
__global__ void __launch_bounds__(kSortThreads)
k_radix_histogram(const uint64_t* __restrict__ keys, uint32_t n, uint32_t passes, uint32_t* __restrict__ hist,
                  uint32_t* __restrict__ lookback, uint64_t lookback_pass_words, uint32_t tile_keys) {
    __shared__ uint32_t s_hist[8 * kRadixBins];
    radix_histogram(keys, n, passes, hist, lookback, lookback_pass_words, tile_keys, s_hist);
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Ranks this warp's items by digit, item by item: lanes with the same digit
// are found by eight ballots (one per digit bit) under the valid-lane mask,
// and s_warp_row counts each digit over the warp's earlier items.  Digit
// kRadixBins marks an invalid item.
template <uint32_t kItems>
__device__ __forceinline__ void warp_rank(const uint32_t (&dig)[kItems], uint32_t (&rank)[kItems],
                                          uint32_t* s_warp_row, uint32_t lane) {
#pragma unroll
    for (uint32_t i = 0; i < kItems; ++i) {
        const uint32_t di = dig[i];
        const bool valid = di < kRadixBins;
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (uint32_t bit = 0; bit < 8; ++bit) {
            const uint32_t on = (di >> bit) & 1u;
            const uint32_t bal = __ballot_sync(0xffffffffu, on);
            peers &= on ? bal : ~bal;
        }
        const uint32_t leader = __ffs(peers) - 1;   // invalid lanes: unused
        uint32_t base = 0;
        if (valid && lane == leader) base = s_warp_row[di];
        base = __shfl_sync(0xffffffffu, base, valid ? leader : lane);
        rank[i] = base + __popc(peers & lanemask_lt());
        if (valid && lane == leader) s_warp_row[di] = base + __popc(peers);
        __syncwarp();
    }
}

// Up to kSmallSortKeys keys: each key's place is the number of keys before it,
// counted directly.  A block takes 32 keys, one per lane, and its warps split
// the other keys between them (read from shared memory, the whole warp the same
// word), so the work spreads over all SMs with one dependent step instead of a
// chain of radix passes in one CTA.  Ties go by input order (a stable sort).
// Measured on one B200 (the earlier one-CTA radix sort in brackets): 1,000 keys
// of 39 bits with values 6 us (12.3), 3,400 pair keys 12 us (22.0).  The
// n^2 compares of 4,096 keys are where the radix passes take over.
constexpr uint32_t kSmallSortKeys = 4096;
constexpr uint32_t kRankThreads = 512;
constexpr size_t kRankSmem = (size_t)kSmallSortKeys * 8;

// `s_keys` holds n keys (an even count), `s_place` 32 words.
__device__ __forceinline__ void rank_sort(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                          uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n,
                                          uint64_t mask, uint64_t* s_keys, uint32_t* s_place) {
    if (blockIdx.x * 32u >= n) return;
    const uint32_t lane = lane_id(), w = warp_id(), warps = blockDim.x >> 5;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) s_keys[i] = __ldcg(keys_in + i) & mask;
    if ((n & 1u) && threadIdx.x == 0) s_keys[n] = ~0ull;   // pads the last pair; an equal key comes before it
    for (uint32_t first = blockIdx.x * 32u; first < n; first += gridDim.x * 32u) {
        if (threadIdx.x < 32u) s_place[threadIdx.x] = 0u;
        __syncthreads();
        const uint32_t i = first + lane;
        const uint64_t key = i < n ? s_keys[i] : 0ull;
        // pairs [lo, hi) of this warp; the keys before i count when equal, those after do not
        const uint32_t pairs = (n + 1u) >> 1, per = (pairs + warps - 1u) / warps;
        const uint32_t lo = min(pairs, w * per), hi = min(pairs, lo + per);
        uint32_t count = 0;
#pragma unroll 8
        for (uint32_t q = lo; q < hi; ++q) {
            const ulonglong2 v = reinterpret_cast<const ulonglong2*>(s_keys)[q];
            count += (v.x < key || (v.x == key && 2u * q < i)) ? 1u : 0u;
            count += (v.y < key || (v.y == key && 2u * q + 1u < i)) ? 1u : 0u;
        }
        if (count) atomicAdd(s_place + lane, count);
        __syncthreads();
        if (w == 0 && i < n) {
            const uint32_t at = s_place[lane];
            keys_out[at] = __ldcg(keys_in + i);
            if (vals_out) vals_out[at] = __ldcg(vals_in + i);
        }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(kRankThreads)
k_rank_sort(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint64_t* __restrict__ keys_out,
            uint32_t* __restrict__ vals_out, uint32_t n, uint64_t mask) {
    __shared__ __align__(16) uint64_t s_keys[kSmallSortKeys];
    __shared__ uint32_t s_place[32];
    rank_sort(keys_in, vals_in, keys_out, vals_out, n, mask, s_keys, s_place);
}

// Shared-memory layout of a onesweep tile of kThreads x kItems keys: the
// reordered keys and values and one digit counter row per warp (dynamic
// shared memory: a 256 x 16 tile takes 56 KB).
template <uint32_t kThreads, uint32_t kItems>
struct SortTile {
    static constexpr uint32_t kTile = kThreads * kItems;
    static constexpr uint32_t kWarps = kThreads / 32;
    static constexpr size_t kValsOff = (size_t)kTile * 8;
    static constexpr size_t kWarpOff = kValsOff + (size_t)kTile * 4;
    static constexpr size_t kBytes = kWarpOff + (size_t)kWarps * kRadixBins * 4;
};

// One pass over n keys by the tiles that this block draws.
template <uint32_t kThreads, uint32_t kItems>
__device__ __forceinline__ void onesweep_pass(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                              uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                                              uint32_t n, uint32_t shift, const uint32_t* __restrict__ digit_hist,
                                              uint32_t* __restrict__ lookback, uint32_t* __restrict__ ticket,
                                              uint32_t* __restrict__ error_flags) {
    static_assert(kThreads >= kRadixBins && kThreads % 32 == 0, "one thread per digit at least");
    using L = SortTile<kThreads, kItems>;
    constexpr uint32_t kTile = L::kTile;
    constexpr uint32_t kWarps = L::kWarps;
    constexpr bool kPerDigit = kThreads == kSortThreads;   // how places are kept inside the result
    extern __shared__ __align__(16) unsigned char s_dyn[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_dyn);
    uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_dyn + L::kValsOff);
    uint32_t (*s_warp)[kRadixBins] = reinterpret_cast<uint32_t (*)[kRadixBins]>(s_dyn + L::kWarpOff);
    __shared__ uint32_t s_local_start[kRadixBins];
    __shared__ uint32_t s_global_base[kRadixBins];
    __shared__ uint32_t s_scan[33];
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_digit_offsets[kRadixBins];

    const uint32_t tiles = (n + kTile - 1) / kTile;
    if (blockIdx.x >= tiles) return;   // before taking a ticket (a grid sized for a capacity)
    const uint32_t lane = lane_id(), w = warp_id();
    const bool digit_thread = threadIdx.x < kRadixBins;
    const uint32_t d = threadIdx.x;   // the digit of a digit thread
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    const uint32_t hist_d = digit_thread ? __ldcg(digit_hist + d) : 0u;   // scanned while the first tile loads
    bool have_offsets = false;

    for (;;) {
        for (uint32_t i = threadIdx.x; i < kWarps * kRadixBins; i += kThreads) (&s_warp[0][0])[i] = 0;
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= tiles) break;
        const uint32_t tile_base = tile * kTile;

        // ---- load every item first (one memory round trip), warp-striped
        uint64_t k[kItems];
        uint32_t v[kItems];
        uint32_t rank[kItems];
        uint32_t dig[kItems];
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            const uint32_t idx = tile_base + w * 32 * kItems + i * 32 + lane;
            const bool valid = idx < n;
            k[i] = valid ? __ldcg(keys_in + idx) : 0ull;
            v[i] = (valid && vals_in) ? __ldcg(vals_in + idx) : 0u;
            dig[i] = valid ? (uint32_t)((k[i] >> shift) & 0xffu) : kRadixBins;
        }
        if (!have_offsets) {   // this pass's digit offsets: exclusive scan of its histogram
            uint32_t total_all;
            const uint32_t off = block_exclusive_scan(hist_d, s_scan, &total_all);
            if (digit_thread) s_digit_offsets[d] = off;
            have_offsets = true;
        }

        // ---- rank within each warp
        warp_rank<kItems>(dig, rank, s_warp[w], lane);
        __syncthreads();

        // ---- per digit: prefix over warps, tile count, tile-local start
        uint32_t count = 0;
        if (digit_thread) {
#pragma unroll 8
            for (uint32_t ww = 0; ww < kWarps; ++ww) {
                const uint32_t c = s_warp[ww][d];
                s_warp[ww][d] = count;
                count += c;
            }
        }
        uint32_t total;
        const uint32_t local_start = block_exclusive_scan(count, s_scan, &total);

        if (digit_thread) {
            s_local_start[d] = local_start;
            // ---- decoupled look-back for digit d (one thread per digit), reading a
            // window of kLookbackWindow predecessors per round trip: with every tile
            // starting at once, a one-word walk advances the inclusive prefixes by
            // about two tiles per L2 round trip, a window by kLookbackWindow + 1
            // (relaxed stores: a word carries its own status and count, and a
            // release store's fence costs about an L2 round trip per tile)
            uint32_t* lb = lookback + (size_t)tile * kRadixBins + d;
            uint32_t prefix = 0;
            if (tile == 0) {
                st_relaxed_u32(lb, kDigitInclusive | count);
            } else {
                st_relaxed_u32(lb, kDigitAggregate | count);
                int64_t t = (int64_t)tile - 1;
                uint32_t spins = 0;
                for (;;) {
                    uint32_t sw[kLookbackWindow];
#pragma unroll
                    for (uint32_t j = 0; j < kLookbackWindow; ++j)   // below tile 0: an inclusive 0
                        sw[j] = t >= (int64_t)j ? ld_relaxed_u32(lookback + (size_t)(t - j) * kRadixBins + d)
                                                : kDigitInclusive;
                    uint32_t advanced = 0;
                    bool stop = false, done = false;
#pragma unroll
                    for (uint32_t j = 0; j < kLookbackWindow; ++j) {   // nearest first, up to the first gap
                        const uint32_t status = sw[j] >> 30;
                        if (!stop) {
                            if (status == 0) {
                                stop = true;
                            } else {
                                prefix += sw[j] & kDigitCountMask;
                                ++advanced;
                                if (status == 2) stop = done = true;
                            }
                        }
                    }
                    if (done) break;
                    if (advanced == 0) {
                        if (++spins > kSpinLimit) {
                            if (error_flags) atomicOr(error_flags, MK_DEVICE_WAIT_TIMEOUT_FLAG);
                            break;
                        }
                        continue;
                    }
                    t -= advanced;
                }
                st_relaxed_u32(lb, kDigitInclusive | (prefix + count));
            }
            // Inside the result whatever the bins say: after a wait that gave up they may be of other keys.
            // The 8,192-key tile compares each place instead, which makes its stores faster (5M keys 540 -> 525 us)
            // and those of the smaller tiles slower (400k keys 0.2 us a pass).
            const uint32_t first = s_digit_offsets[d] + prefix;
            const bool inside = !kPerDigit || (first <= n && count <= n - first);
            s_global_base[d] = (inside ? first : 0u) - local_start;
        }
        __syncthreads();

        // ---- reorder through shared memory, then scatter by digit runs
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            if (dig[i] < kRadixBins) {
                const uint32_t r = s_local_start[dig[i]] + s_warp[w][dig[i]] + rank[i];
                s_keys[r] = k[i];
                if (vals_out) s_vals[r] = v[i];
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            const uint32_t j = threadIdx.x + i * kThreads;
            if (j < total) {
                const uint64_t kk = s_keys[j];
                const uint32_t dst = s_global_base[(uint32_t)((kk >> shift) & 0xffu)] + j;
                if (kPerDigit || dst < n) {
                    keys_out[dst] = kk;
                    if (vals_out) vals_out[dst] = s_vals[j];
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);   // every thread has read s_tile
    }
}

template <uint32_t kThreads, uint32_t kItems>
__global__ void __launch_bounds__(kThreads)
k_radix_onesweep(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                 uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n, uint32_t shift,
                 const uint32_t* __restrict__ digit_hist /* 256 */, uint32_t* __restrict__ lookback,
                 uint32_t* __restrict__ ticket, uint32_t* __restrict__ error_flags) {
    onesweep_pass<kThreads, kItems>(keys_in, vals_in, keys_out, vals_out, n, shift, digit_hist, lookback, ticket,
                                    error_flags);
}

// A whole sort of keys (no values) whose count is known on the device only, in
// one cooperative launch: small counts by rank, larger ones by the histogram
// and the passes with a grid barrier between them.  As launches of their own,
// the histogram and passes cost 2.5-3 us each on the ticks whose pairs the
// small sort takes (7 launches, about 16 us a tick).
template <uint32_t kThreads, uint32_t kItems>
__global__ void __launch_bounds__(kThreads)
k_sort_counted(const uint64_t* __restrict__ keys_in, uint64_t* __restrict__ tmp, uint64_t* __restrict__ keys_out,
               const uint32_t* __restrict__ n_ptr, uint32_t capacity, uint32_t passes, uint64_t mask,
               uint32_t* __restrict__ hist, uint32_t* __restrict__ lookback, uint64_t lookback_pass_words,
               uint32_t* __restrict__ tickets, uint32_t* __restrict__ barrier, uint32_t* __restrict__ error_flags) {
    using L = SortTile<kThreads, kItems>;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ uint32_t s_place[32];
    const uint32_t n = min(*n_ptr, capacity);   // a device count never exceeds the capacity
    if (n <= kSmallSortKeys) {
        rank_sort(keys_in, nullptr, keys_out, nullptr, n, mask, reinterpret_cast<uint64_t*>(s_dyn), s_place);
        return;
    }
    radix_histogram(keys_in, n, passes, hist, lookback, lookback_pass_words, L::kTile,
                    reinterpret_cast<uint32_t*>(s_dyn));
    const uint64_t* src = keys_in;
    for (uint32_t pass = 0; pass < passes; ++pass) {
        grid_barrier(barrier, error_flags, gridDim.x);
        uint64_t* dst = ((passes - 1 - pass) % 2) == 0 ? keys_out : tmp;   // the last pass writes keys_out
        onesweep_pass<kThreads, kItems>(src, nullptr, dst, nullptr, n, 8 * pass, hist + pass * kRadixBins,
                                        lookback + pass * lookback_pass_words, tickets + pass, error_flags);
        src = dst;
    }
}

uint32_t sort_passes(uint32_t key_bits) { return (key_bits + 7) / 8; }
// The key bits that the passes order by.
static uint64_t sort_mask(uint32_t passes) { return passes >= 8 ? ~0ull : (1ull << (8 * passes)) - 1ull; }

// Keys per thread of a 256-thread onesweep tile.  The pass is latency bound:
// its critical path is one tile's ranking (issue bound, so two tiles on one SM
// take twice as long) plus the look-back chain (one L2 round trip per
// kLookbackWindow tiles), so fewer, larger tiles win over spreading a sort
// across every SM.  Measured per pass on B200: 400k keys 12.9 us at 11 or 16 keys
// per thread (17.1 at 8); 1.6M 29.5 us at 11; 6.4M 82 us at 16.  Whole sorts of
// 63-bit keys with values at 4 / 6 / 8 / 11 / 16 keys per thread: 6,000 keys 73 / 72
// / 72 / 72 / 89 us; 20,000 101 / 84 / 77 / 72 / 89; 30,000 99 / 88 / 91 / 73 / 89;
// 65,000 121 / 91 / 111 / 89 / 91 (and alike for fewer bits).  Up to 16,384 keys,
// eight tiles of 8, a tick's broadphase is 1-2 us shorter with 8 than with 11 (10,000
// colliders 97 and 99 us), from there on longer (20,000 109 and 105, 65,000 144 and
// 125).  set_sort_items overrides the default (a tuning parameter).
// 32 names the 8,192-key tile of 512 threads x 16 keys (the same keys per 256
// threads as 32 keys each): half the tiles of the 4,096-key shape, so the
// look-back frontier, which advances a window of tiles per L2 round trip,
// covers twice the keys per round trip.
static uint32_t g_sort_items_override = 0;
bool valid_sort_items(uint32_t items) {
    return items == 2 || items == 4 || items == 6 || items == 8 || items == 11 || items == 16 || items == 32;
}
void set_sort_items(uint32_t items) { g_sort_items_override = items; }

// The pair-key sort's tile is fixed when the tick is captured (its key count
// is only known on the device).  The 8,192-key tile: on the 100,000-body
// start (14.0M pairs) the five passes take 0.32 ms less than with 2,048-key
// tiles, and ticks with 8k-40k pairs about 20 us more each (one B200).
static uint32_t g_pair_sort_items = 0;
constexpr uint32_t kPairSortItemsDefault = 32;
uint32_t pair_sort_items() { return valid_sort_items(g_pair_sort_items) ? g_pair_sort_items : kPairSortItemsDefault; }
void set_pair_sort_items(uint32_t items) { g_pair_sort_items = valid_sort_items(items) ? items : 0u; }
uint32_t sort_items_for(uint32_t n, int sm_count) {
    if (valid_sort_items(g_sort_items_override)) return g_sort_items_override;
    (void)sm_count;
    // above 2M keys the 8,192-key tile (standalone sort with values, one B200: 3.6M keys
    // 245 against 271 us at 16 keys per thread, 14M keys 817 against 868 us)
    return n <= (1u << 14) ? 8u : n <= (1u << 21) ? 11u : 32u;
}

// The histogram bins and tile tickets of a sort's scratch: the region that must
// be zero when the sort starts (launch_sort clears it unless told it is clear).
void sort_clear_region(void* scratch, uint32_t n, uint32_t key_bits, bool values, void** ptr, uint64_t* bytes) {
    const uint32_t passes = sort_passes(key_bits);
    char* p = (char*)scratch;
    p += align256((uint64_t)n * 8);
    p += align256((uint64_t)(values ? n : 0) * 4);
    *ptr = p;
    *bytes = align256((uint64_t)passes * kRadixBins * 4) + align256((uint64_t)passes * 4);
}

uint64_t sort_scratch_bytes(uint32_t n, uint32_t key_bits, bool values) {
    uint32_t passes = sort_passes(key_bits);
    uint64_t tiles = (n + 511) / 512;   // smallest tile: 512 keys
    uint64_t b = 0;
    b += align256((uint64_t)n * 8);                       // ping-pong keys
    b += align256((uint64_t)(values ? n : 0) * 4);        // ping-pong values
    b += align256((uint64_t)passes * kRadixBins * 4);     // histograms / offsets
    b += align256((uint64_t)passes * 4);                  // tile tickets
    b += align256((uint64_t)passes * (tiles ? tiles : 1) * kRadixBins * 4);   // look-back words
    return b;
}

// Shared memory of k_sort_counted: a tile, or the keys of a small sort.
template <uint32_t kThreads, uint32_t kItems>
constexpr size_t counted_smem() {
    return SortTile<kThreads, kItems>::kBytes > kRankSmem ? SortTile<kThreads, kItems>::kBytes : kRankSmem;
}

// Dynamic shared memory of every tile shape, set once per device (outside
// stream capture: the first sort on a device, or handle creation).
cudaError_t sort_prepare() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load() & bit) return cudaSuccess;
#define MK_SORT_ATTR(T, I)                                                                                    \
    if (e == cudaSuccess)                                                                                    \
        e = cudaFuncSetAttribute(k_radix_onesweep<T, I>, cudaFuncAttributeMaxDynamicSharedMemorySize,            \
                                 (int)SortTile<T, I>::kBytes);                                                   \
    if (e == cudaSuccess)                                                                                    \
        e = cudaFuncSetAttribute(k_sort_counted<T, I>, cudaFuncAttributeMaxDynamicSharedMemorySize,              \
                                 (int)counted_smem<T, I>());
    MK_SORT_ATTR(kSortThreads, 2)
    MK_SORT_ATTR(kSortThreads, 4)
    MK_SORT_ATTR(kSortThreads, 6)
    MK_SORT_ATTR(kSortThreads, 8)
    MK_SORT_ATTR(kSortThreads, 11)
    MK_SORT_ATTR(kSortThreads, 16)
    MK_SORT_ATTR(2 * kSortThreads, 16)
#undef MK_SORT_ATTR
    if (e == cudaSuccess) done.fetch_or(bit);
    return e;
}

// The buffers of a sort inside its scratch.
struct SortScratch {
    uint64_t* keys;
    uint32_t *vals, *hist, *tickets, *barrier, *lookback;
    uint64_t lookback_words;   // per pass
};
static SortScratch sort_scratch(void* scratch, uint32_t n, uint32_t passes, bool values) {
    char* p = (char*)scratch;
    SortScratch c;
    c.keys = (uint64_t*)p; p += align256((uint64_t)n * 8);
    c.vals = values ? (uint32_t*)p : nullptr; p += align256((uint64_t)(values ? n : 0) * 4);
    c.hist = (uint32_t*)p; p += align256((uint64_t)passes * kRadixBins * 4);
    c.tickets = (uint32_t*)p;
    c.barrier = c.tickets + 32;   // the tickets' 256 bytes hold at most 8 of them
    p += align256((uint64_t)passes * 4);
    c.lookback = (uint32_t*)p;
    c.lookback_words = (uint64_t)((n + 511) / 512) * kRadixBins;   // smallest tile: 512 keys
    return c;
}

// One pass over `n` keys whose bins are of other keys: every key has digit 200, the bins say digit 100, so the pass
// places all of them past the n words of `out`.  The 8,192-key tile above 65,536 keys.  `scratch` holds the bins, a ticket and the look-back words.
cudaError_t launch_stale_sort_pass(const uint64_t* keys, uint64_t* out, uint32_t n, uint32_t* scratch,
                                   uint32_t* error_flags, cudaStream_t stream) {
    cudaError_t e = sort_prepare();
    if (e != cudaSuccess) return e;
    auto pass = [&](auto* kernel, uint32_t threads, uint32_t items, size_t bytes) {
        kernel<<<(n + threads * items - 1) / (threads * items), threads, bytes, stream>>>(
            keys, nullptr, out, nullptr, n, 0u, scratch, scratch + 512, scratch + 256, error_flags);
    };
    if (n <= (1u << 16)) pass(k_radix_onesweep<kSortThreads, 8>, kSortThreads, 8, SortTile<kSortThreads, 8>::kBytes);
    else pass(k_radix_onesweep<2 * kSortThreads, 16>, 2 * kSortThreads, 16, SortTile<2 * kSortThreads, 16>::kBytes);
    return cudaGetLastError();
}

// Stream-ordered sort of n keys with values.
cudaError_t launch_sort(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out, uint32_t* vals_out,
                        uint32_t n, uint32_t key_bits, void* scratch, uint64_t scratch_bytes, uint32_t* error_flags,
                        cudaStream_t stream, int sm_count, uint32_t items_override, uint32_t ctas_per_sm,
                        bool precleared) {
    if (n == 0) return cudaSuccess;
    cudaError_t ep = sort_prepare();
    if (ep != cudaSuccess) return ep;
    uint32_t passes = sort_passes(key_bits);
    if (passes == 0 || passes > 8) return cudaErrorInvalidValue;
    const bool values = vals_in != nullptr;
    if (scratch_bytes < sort_scratch_bytes(n, key_bits, values)) return cudaErrorInvalidValue;
    if (n <= kSmallSortKeys) {
        k_rank_sort<<<(n + 31) / 32, kRankThreads, 0, stream>>>(keys_in, vals_in, keys_out, vals_out, n,
                                                                sort_mask(passes));
        return cudaGetLastError();
    }
    const uint32_t items = valid_sort_items(items_override) ? items_override : sort_items_for(n, sm_count);
    const uint32_t tile_keys = kSortThreads * items;
    const uint64_t tiles = (n + tile_keys - 1) / tile_keys;
    const SortScratch c = sort_scratch(scratch, n, passes, values);
    // histogram bins and tile tickets are cleared here; look-back words by the
    // histogram kernel, only as many as the count needs
    if (!precleared) {
        cudaError_t e = cudaMemsetAsync(c.hist, 0, (uint64_t)((char*)c.tickets - (char*)c.hist) + passes * 4, stream);
        if (e != cudaSuccess) return e;
    }
    // 1,024 keys per block while that fills the SMs no more than four deep: the histogram is a
    // short chain of loads and shared atomics, and its bins' global sums cost less than idle SMs
    // (402k keys 13.2 us with 4,096 keys per block, 9.1 with 2,048, 8.8 with 1,024)
    uint32_t hist_blocks = (uint32_t)std::min<uint64_t>((n + 1023) / 1024, (uint64_t)sm_count * 4);
    k_radix_histogram<<<hist_blocks, kSortThreads, 0, stream>>>(keys_in, n, passes, c.hist, c.lookback,
                                                                c.lookback_words, tile_keys);
    const uint32_t per_sm = ctas_per_sm ? ctas_per_sm : default_sort_ctas(items);
    const uint32_t grid = (uint32_t)std::min<uint64_t>(tiles, (uint64_t)sm_count * per_sm);
    // passes alternate between (tmp, out) so that the last pass writes `out`.
    const uint64_t* src_k = keys_in;
    const uint32_t* src_v = vals_in;
    for (uint32_t pass = 0; pass < passes; ++pass) {
        bool to_out = ((passes - 1 - pass) % 2) == 0;
        uint64_t* dk = to_out ? keys_out : c.keys;
        uint32_t* dv = values ? (to_out ? vals_out : c.vals) : nullptr;
        uint32_t* lb = c.lookback + pass * c.lookback_words;
        const uint32_t* offs = c.hist + pass * kRadixBins;
#define MK_SORT_PASS(T, I)                                                                                       \
    k_radix_onesweep<T, I><<<grid, T, SortTile<T, I>::kBytes, stream>>>(src_k, src_v, dk, dv, n, 8 * pass, offs, lb, \
                                                                        c.tickets + pass, error_flags)
        switch (items) {
            case 2: MK_SORT_PASS(kSortThreads, 2); break;
            case 4: MK_SORT_PASS(kSortThreads, 4); break;
            case 6: MK_SORT_PASS(kSortThreads, 6); break;
            case 8: MK_SORT_PASS(kSortThreads, 8); break;
            case 11: MK_SORT_PASS(kSortThreads, 11); break;
            case 32: MK_SORT_PASS(2 * kSortThreads, 16); break;
            default: MK_SORT_PASS(kSortThreads, 16); break;
        }
#undef MK_SORT_PASS
        src_k = dk;
        src_v = dv;
    }
    return cudaGetLastError();
}

template <uint32_t kThreads, uint32_t kItems>
static cudaError_t launch_counted(const uint64_t* keys_in, uint64_t* keys_out, uint32_t capacity, const uint32_t* n_dev,
                                  uint32_t passes, const SortScratch& c, uint32_t* error_flags, cudaStream_t stream,
                                  int sm_count) {
    constexpr size_t smem = counted_smem<kThreads, kItems>();
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sort_counted<kThreads, kItems>, kThreads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const uint64_t tiles = ((uint64_t)capacity + kThreads * kItems - 1) / (kThreads * kItems);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(std::max<uint64_t>(tiles, kSmallSortKeys / 32),
                                                                         (uint64_t)sm_count * per_sm)));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_sort_counted<kThreads, kItems>, keys_in, c.keys, keys_out, n_dev, capacity, passes,
                              sort_mask(passes), c.hist, c.lookback, c.lookback_words, c.tickets, c.barrier, error_flags);
}

// Stream-ordered sort of keys whose count is on the device (at most `capacity`);
// bins, tickets and the barrier word (sort_clear_region) are clear.
cudaError_t launch_sort_counted(const uint64_t* keys_in, uint64_t* keys_out, uint32_t capacity, const uint32_t* n_dev,
                                uint32_t key_bits, void* scratch, uint64_t scratch_bytes, uint32_t* error_flags,
                                cudaStream_t stream, int sm_count, uint32_t items) {
    cudaError_t ep = sort_prepare();
    if (ep != cudaSuccess) return ep;
    const uint32_t passes = sort_passes(key_bits);
    if (passes == 0 || passes > 8 || scratch_bytes < sort_scratch_bytes(capacity, key_bits, false))
        return cudaErrorInvalidValue;
    const SortScratch c = sort_scratch(scratch, capacity, passes, false);
#define MK_SORT_COUNTED(T, I) \
    return launch_counted<T, I>(keys_in, keys_out, capacity, n_dev, passes, c, error_flags, stream, sm_count)
    switch (items) {
        case 2: MK_SORT_COUNTED(kSortThreads, 2);
        case 4: MK_SORT_COUNTED(kSortThreads, 4);
        case 6: MK_SORT_COUNTED(kSortThreads, 6);
        case 8: MK_SORT_COUNTED(kSortThreads, 8);
        case 11: MK_SORT_COUNTED(kSortThreads, 11);
        case 32: MK_SORT_COUNTED(2 * kSortThreads, 16);
        default: MK_SORT_COUNTED(kSortThreads, 16);
    }
#undef MK_SORT_COUNTED
}

}  // namespace mk
