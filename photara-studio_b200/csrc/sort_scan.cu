// Hand-written device-wide scan and onesweep LSD radix sort (sm_100a).
//
// The reference calls CUB DeviceScan::InclusiveSum and
// DeviceRadixSort::SortPairs (third_party/splat_drender/src/pipeline.cu:231-311).
// Both are replaced here:
//  * scan: single-pass chained scan with decoupled look-back;
//  * sort: one histogram pass computing every digit histogram at once, then one
//    kernel per digit (the key bits cut into the fewest near-equal digits of at
//    most 9 bits; 8 for 64-bit keys) that ranks its tile stably (warp ballot
//    multisplit), stages it in shared memory in digit order, resolves its
//    global digit offsets by decoupled look-back over preceding tiles and
//    writes coalesced digit runs (Adinets & Merrill, "Onesweep", 2022).
// Every look-back spin is bounded by kSpinLimit; on timeout the kernel sets
// the device error word and proceeds, so a broken invariant reports an error
// instead of hanging the GPU.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace gsb {

// ------------------------------------------------------------------ scan --
static_assert(kScanTile == kBlock * kScanItems, "scan tile = block x items per thread");

// Exclusive scan of u32 `in` (read through `index` when given: in[index[k]])
// into `out`; total written to *total. status: one u64 per tile, zeroed;
// tile_counter zeroed. With `groups`, the running sum is also cut into groups
// of 2^group_shift: groups[b] = the first element whose exclusive sum is at
// least b << group_shift, for every b <= total >> group_shift below
// group_cap (elements of value 0 never start a group after the first).
__global__ void __launch_bounds__(kBlock) scan_kernel(int n, const unsigned* __restrict__ in,
                                                      const unsigned* __restrict__ index,
                                                      unsigned* __restrict__ out,
                                                      unsigned long long* __restrict__ status,
                                                      unsigned* __restrict__ tile_counter,
                                                      unsigned* __restrict__ total,
                                                      unsigned* __restrict__ err,
                                                      unsigned spin_limit,
                                                      unsigned* __restrict__ groups,
                                                      int group_shift, unsigned group_cap) {
    __shared__ unsigned s_tile;
    __shared__ unsigned s_warp[8];
    __shared__ unsigned long long s_prefix;
    if (threadIdx.x == 0)
        s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const unsigned tile = s_tile;
    const size_t base = size_t(tile) * kScanTile + size_t(threadIdx.x) * kScanItems;
    unsigned v[kScanItems];
    unsigned sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const size_t idx = base + k;
        v[k] = idx < size_t(n) ? in[index ? index[idx] : idx] : 0u;
        sum += v[k];
    }
    unsigned tile_sum;
    const unsigned excl = block_excl_scan256(sum, s_warp, tile_sum);
    if (threadIdx.x < 32) {
        const unsigned long long prefix =
            warp_lookback(status, tile, tile_sum, err, kDevLookbackTimeout, spin_limit);
        if (threadIdx.x == 0) {
            s_prefix = prefix;
            if (size_t(tile + 1) * kScanTile >= size_t(n))
                *total = unsigned(prefix + tile_sum);
        }
    }
    __syncthreads();
    unsigned run = unsigned(s_prefix) + excl;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const size_t idx = base + k;
        if (idx < size_t(n)) {
            out[idx] = run;
            if (groups) {
                // element idx + 1 starts every group whose first sum lies in
                // (run, run + v]
                if (idx == 0)
                    groups[0] = 0;
                const unsigned b_end = min((run + v[k]) >> group_shift, group_cap - 1u);
                for (unsigned b = (run >> group_shift) + 1; b <= b_end; ++b)
                    groups[b] = unsigned(idx + 1);
            }
        }
        run += v[k];
    }
}

// ------------------------------------------------------------------ sort --
constexpr int kSortItems = 12;
constexpr int kSortTile = kBlock * kSortItems; // 3072 keys per tile
constexpr int kWarpItems = 32 * kSortItems;    // 384 keys per warp
constexpr unsigned kStFlagAgg = 1u << 30;
constexpr unsigned kStFlagPre = 2u << 30;
constexpr unsigned kStMask = (1u << 30) - 1;

// Digit of `bits` bits starting at `shift`; bits above the sorted range never
// take part.
template <typename Key>
__device__ __forceinline__ unsigned digit_of(Key key, int shift, int bits) {
    return unsigned(key >> shift) & ((1u << bits) - 1u);
}

// All digit histograms in one read of the keys. hist: [passes][kMaxRadix], zeroed.
// Per-block shared-memory histograms with one shared atomic per key and pass
// (a block's keys spread over the bins, so conflicts are rare), flushed with
// one global atomic per non-empty bin. This replaced a ballot-per-bit warp
// aggregation that cost 8 ballots per key and pass (85 against 33 us for the
// 8.3M tile keys of a 1080p frame).
template <typename Key>
__global__ void __launch_bounds__(kBlock) radix_histogram_kernel(
    const Key* __restrict__ keys, const unsigned* __restrict__ count_ptr, int begin_bit,
    RadixPlan plan, unsigned* __restrict__ hist) {
    __shared__ unsigned s_hist[8][kMaxRadix];
    for (int k = threadIdx.x; k < 8 * kMaxRadix; k += kBlock)
        (&s_hist[0][0])[k] = 0;
    __syncthreads();
    const size_t n = *count_ptr;
    const size_t stride = size_t(gridDim.x) * kBlock;
#pragma unroll 4
    for (size_t i = size_t(blockIdx.x) * kBlock + threadIdx.x; i < n; i += stride) {
        const Key key = keys[i];
        for (int p = 0; p < plan.passes; ++p)
            atomicAdd(&s_hist[p][digit_of(key, begin_bit + plan.shift(p), plan.width(p))], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < plan.passes * kMaxRadix; k += kBlock) {
        const unsigned v = (&s_hist[0][0])[k];
        if (v)
            atomicAdd(&hist[k], v);
    }
}

// Exclusive block scans of two values per thread at once (256 threads);
// warp_tot holds 16 words. total: the block sum of the first.
__device__ __forceinline__ uint2 block_excl_scan256_pair(unsigned a, unsigned b,
                                                         unsigned* warp_tot, unsigned& total) {
    const unsigned ia = warp_incl_scan(a), ib = warp_incl_scan(b);
    const int w = threadIdx.x >> 5;
    if (lane_id() == 31) {
        warp_tot[w] = ia;
        warp_tot[8 + w] = ib;
    }
    __syncthreads();
    unsigned ba = 0, bb = 0, sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const unsigned ta = warp_tot[k], tb = warp_tot[8 + k];
        ba += k < w ? ta : 0u;
        bb += k < w ? tb : 0u;
        sum += ta;
    }
    total = sum;
    return make_uint2(ba + ia - a, bb + ib - b);
}

__device__ __forceinline__ void copy_async4(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(smem))),
                 "l"(gmem)
                 : "memory");
}

// One stable digit pass of kBits (<= 9) bits. hist: the pass's digit counts
// over all keys; status: [tiles][2^kBits] zeroed; tile_counter zeroed. A
// thread owns one digit (two neighbouring ones at 9 bits, whose status words
// it reads and writes as one 64-bit word): its counts over the warps, its
// look-back, its start in the output, which each tile works out from the digit
// counts itself. The tile is staged in digit order before the look-back, so
// its predecessors have that time to publish.
template <typename Key, int kBits>
__global__ void __launch_bounds__(kBlock, 4) onesweep_kernel(
    const Key* __restrict__ keys_in, const unsigned* __restrict__ vals_in,
    Key* __restrict__ keys_out, unsigned* __restrict__ vals_out,
    const unsigned* __restrict__ count_ptr, int shift, const unsigned* __restrict__ hist,
    unsigned* __restrict__ status, unsigned* __restrict__ tile_counter,
    unsigned* __restrict__ err, unsigned spin_limit) {
    constexpr int kDigits = 1 << kBits;
    constexpr int kOwn = kDigits > kBlock ? 2 : 1; // digits per thread
    __shared__ unsigned s_tile;
    __shared__ unsigned s_whist[8][kDigits]; // per-warp digit counts, then warp prefix
    __shared__ unsigned s_tprefix[kDigits];  // tile-local digit start
    __shared__ unsigned s_gbase[kDigits];    // global start of the digit run - its tile start
    __shared__ unsigned s_warp[16];
    __shared__ Key s_keys[kSortTile];
    __shared__ unsigned s_vals[kSortTile];

    const unsigned n = *count_ptr;
    const unsigned tiles = (n + kSortTile - 1) / kSortTile;
    if (threadIdx.x == 0)
        s_tile = atomicAdd(tile_counter, 1u);
    for (int k = threadIdx.x; k < 8 * kDigits; k += kBlock)
        (&s_whist[0][0])[k] = 0;
    __syncthreads();
    const unsigned tile = s_tile;
    if (tile >= tiles)
        return;
    const int warp = threadIdx.x >> 5;
    const unsigned lane = lane_id();
    // the thread's items: `first` + 32 k of the tile's `left` keys
    const unsigned first = unsigned(warp) * kWarpItems + lane;
    const unsigned left = n - tile * kSortTile;
    const Key* const kin = keys_in + size_t(tile) * kSortTile + first;
    const unsigned* const vin = vals_in + size_t(tile) * kSortTile + first;

    // Only the last tile is partial; full tiles skip the bounds tests.
    const bool full = left >= unsigned(kSortTile);
    Key key[kSortItems];
    unsigned rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k)
        key[k] = full || first + 32 * k < left ? kin[32 * k] : Key(~Key(0));
    const unsigned d0 = threadIdx.x * kOwn; // the thread's (first) digit
    const bool owner = d0 < unsigned(kDigits);
    unsigned total_of[kOwn];
#pragma unroll
    for (int o = 0; o < kOwn; ++o)
        total_of[o] = owner ? hist[d0 + o] : 0u;
    // Warp multisplit in index order (k-major, lane-minor == global order):
    // the lanes holding the same digit are found with one ballot per digit bit
    // (all items' ballots first, independent of the counters), then each
    // item's rank from the warp's running digit counts: every lane reads its
    // digit's count, then the group's first lane moves it on.
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const unsigned d = digit_of(key[k], shift, kBits);
        unsigned p = full ? 0xffffffffu : __ballot_sync(0xffffffffu, first + 32 * k < left);
#pragma unroll
        for (int b = 0; b < kBits; ++b) {
            const bool bit = (d >> b) & 1u;
            const unsigned vote = __ballot_sync(0xffffffffu, bit);
            p &= bit ? vote : ~vote;
        }
        rank[k] = p; // the lanes of the item's digit, until it is ranked below
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        unsigned* const c = &s_whist[warp][digit_of(key[k], shift, kBits)];
        const unsigned peers = rank[k];
        const unsigned below = __popc(peers & lanemask_lt());
        const unsigned prior = *c;
        __syncwarp();
        if (below == 0 && (full || first + 32 * k < left))
            *c = prior + __popc(peers);
        __syncwarp();
        rank[k] = prior + below;
    }
    __syncthreads();
    // The owned digits' warp prefixes and tile counts, published at once.
    unsigned cnt[kOwn];
    unsigned* const st = status + size_t(tile) * kDigits + d0;
    if (owner) {
#pragma unroll
        for (int o = 0; o < kOwn; ++o) {
            cnt[o] = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const unsigned c = s_whist[w][d0 + o];
                s_whist[w][d0 + o] = cnt[o];
                cnt[o] += c;
            }
        }
        const unsigned flag = tile == 0 ? kStFlagPre : kStFlagAgg;
        if constexpr (kOwn == 2)
            st_relaxed64(reinterpret_cast<unsigned long long*>(st),
                         (static_cast<unsigned long long>(flag | cnt[1]) << 32) | (flag | cnt[0]));
        else
            st_relaxed(st, flag | cnt[0]);
    } else {
#pragma unroll
        for (int o = 0; o < kOwn; ++o)
            cnt[o] = 0;
    }
    unsigned own_cnt = 0, own_total = 0;
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
        own_cnt += cnt[o];
        own_total += total_of[o];
    }
    unsigned tile_total;
    const uint2 at = block_excl_scan256_pair(own_cnt, own_total, s_warp, tile_total);
    if (owner) {
        s_tprefix[d0] = at.x;
        if constexpr (kOwn == 2)
            s_tprefix[d0 + 1] = at.x + cnt[0];
    }
    __syncthreads();
    // Stage the tile in digit order; the values go from global to shared memory
    // asynchronously, during the look-back. (The keys and ranks across the
    // ballots spill 36 to 72 bytes a thread at 64 registers.)
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        if (full || first + 32 * k < left) {
            const unsigned dk = digit_of(key[k], shift, kBits);
            const unsigned pos = s_tprefix[dk] + s_whist[warp][dk] + rank[k];
            s_keys[pos] = key[k];
            copy_async4(&s_vals[pos], vin + 32 * k);
        }
    }
    // Look-back over the preceding tiles' counts of the owned digits.
    if (owner) {
        unsigned excl[kOwn];
#pragma unroll
        for (int o = 0; o < kOwn; ++o)
            excl[o] = 0;
        if (tile > 0) {
            int pred = int(tile) - 1;
            unsigned spins = 0;
            while (pred >= 0) {
                unsigned s[kOwn];
                const unsigned* sp = status + size_t(pred) * kDigits + d0;
                if constexpr (kOwn == 2) {
                    // both words are written together
                    const unsigned long long v =
                        ld_relaxed64(reinterpret_cast<const unsigned long long*>(sp));
                    s[0] = unsigned(v);
                    s[1] = unsigned(v >> 32);
                } else {
                    s[0] = ld_relaxed(sp);
                }
                const unsigned flag = s[0] >> 30;
                if (flag == 0) {
                    if (++spins > spin_limit) {
                        atomicOr(err, kDevLookbackTimeout);
                        break;
                    }
                    continue;
                }
#pragma unroll
                for (int o = 0; o < kOwn; ++o)
                    excl[o] += s[o] & kStMask;
                if (flag == 2)
                    break;
                --pred;
            }
            if constexpr (kOwn == 2)
                st_relaxed64(reinterpret_cast<unsigned long long*>(st),
                             (static_cast<unsigned long long>(kStFlagPre | (excl[1] + cnt[1])) << 32) |
                                 (kStFlagPre | (excl[0] + cnt[0])));
            else
                st_relaxed(st, kStFlagPre | (excl[0] + cnt[0]));
        }
        s_gbase[d0] = at.y + excl[0] - at.x;
        if constexpr (kOwn == 2)
            s_gbase[d0 + 1] = at.y + total_of[0] + excl[1] - (at.x + cnt[0]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (unsigned pos = threadIdx.x; pos < tile_total; pos += kBlock) {
        const Key kk = s_keys[pos];
        const unsigned out = s_gbase[digit_of(kk, shift, kBits)] + pos;
        if (out < n) { // always true unless a look-back gave up (error word set)
            keys_out[out] = kk;
            vals_out[out] = s_vals[pos];
        }
    }
}

size_t scan_status_bytes(int n) {
    const size_t tiles = (size_t(n) + kScanTile - 1) / kScanTile;
    return tiles * sizeof(unsigned long long);
}

void launch_scan(cudaStream_t s, int n, const unsigned* in, const unsigned* index, unsigned* out,
                 unsigned long long* status, unsigned* tile_counter, unsigned* total,
                 unsigned* err, bool zeroed, unsigned* groups, int group_shift,
                 unsigned group_cap) {
    if (n <= 0)
        return;
    const int tiles = (n + kScanTile - 1) / kScanTile;
    if (!zeroed) {
        cudaMemsetAsync(status, 0, size_t(tiles) * sizeof(unsigned long long), s);
        cudaMemsetAsync(tile_counter, 0, sizeof(unsigned), s);
    }
    scan_kernel<<<tiles, kBlock, 0, s>>>(n, in, index, out, status, tile_counter, total, err,
                                         kSpinLimit, groups, group_shift, group_cap);
}

size_t sort_status_bytes(size_t count, const RadixPlan& plan) {
    const size_t tiles = (count + kSortTile - 1) / kSortTile;
    size_t digits = 0;
    for (int p = 0; p < plan.passes; ++p)
        digits += size_t(1) << plan.width(p);
    return tiles * digits * sizeof(unsigned);
}

size_t sort_status_bytes_max(size_t count, int bits) {
    size_t most = 0;
    for (int b = 1; b <= bits; ++b)
        most = std::max(most, sort_status_bytes(count, radix_plan(b)));
    return most;
}

int sort_tile_count(size_t count) { return int((count + kSortTile - 1) / kSortTile); }

// Sorts (keys, vals) of `count` elements (count also on device at count_dev)
// on bits [begin_bit, end_bit). Ping-pongs between the two buffers; returns
// the index (0 or 1) of the buffer holding the result.
template <typename Key>
int launch_radix_sort(cudaStream_t s, Key* keys[2], unsigned* vals[2], size_t count,
                      const unsigned* count_dev, int begin_bit, int end_bit, unsigned* hist,
                      unsigned* status, unsigned* tile_counters, unsigned* err,
                      bool hist_ready, bool zeroed) {
    const RadixPlan plan = sort_plan<Key>(end_bit - begin_bit);
    if (count <= 1 || plan.passes <= 0)
        return 0;
    const int tiles = sort_tile_count(count);
    if (!zeroed) {
        cudaMemsetAsync(status, 0, sort_status_bytes(count, plan), s);
        cudaMemsetAsync(tile_counters, 0, size_t(plan.passes) * sizeof(unsigned), s);
    }
    if (!hist_ready) {
        if (!zeroed)
            cudaMemsetAsync(hist, 0, size_t(plan.passes) * kMaxRadix * sizeof(unsigned), s);
        const int hist_blocks = min(tiles, 148 * 4);
        radix_histogram_kernel<Key>
            <<<hist_blocks, kBlock, 0, s>>>(keys[0], count_dev, begin_bit, plan, hist);
    }
    int cur = 0;
    for (int p = 0; p < plan.passes; ++p) {
        auto pass = [&](auto kernel) {
            kernel<<<tiles, kBlock, 0, s>>>(keys[cur], vals[cur], keys[cur ^ 1], vals[cur ^ 1],
                                            count_dev, begin_bit + plan.shift(p),
                                            hist + p * kMaxRadix, status, tile_counters + p, err,
                                            kSpinLimit);
        };
        switch (plan.width(p)) {
        case 1: pass(onesweep_kernel<Key, 1>); break;
        case 2: pass(onesweep_kernel<Key, 2>); break;
        case 3: pass(onesweep_kernel<Key, 3>); break;
        case 4: pass(onesweep_kernel<Key, 4>); break;
        case 5: pass(onesweep_kernel<Key, 5>); break;
        case 6: pass(onesweep_kernel<Key, 6>); break;
        case 7: pass(onesweep_kernel<Key, 7>); break;
        case 8: pass(onesweep_kernel<Key, 8>); break;
        default:
            if constexpr (sizeof(Key) == 4)
                pass(onesweep_kernel<Key, 9>);
            break;
        }
        status += size_t(tiles) << plan.width(p);
        cur ^= 1;
    }
    return cur;
}

namespace {
constexpr size_t align16(size_t v) { return (v + 15) / 16 * 16; }
} // namespace

size_t lookback_probe_bytes() {
    // counters, then the larger of the two probes' buffers: the scan's input,
    // output and two status words, or the sort's keys and values in and out,
    // two tiles of status words and the digit offsets
    const size_t scan = align16(2 * kScanTile * 4) * 2 + align16(2 * 8);
    const size_t sort = align16(2 * kSortTile * 4) * 4 + align16(2 * 256 * 4) + align16(256 * 4);
    return align16(16) + (scan > sort ? scan : sort);
}

// One block of the scan kernel (which == 0) or of an 8-bit onesweep pass
// (which == 1) over two tiles of zeros, with its tile counter starting at 1:
// the block takes tile 1, and tile 0 is never published, so its look-back
// waits for a predecessor that nothing sets until `spin_limit` re-reads have
// passed and then sets kDevLookbackTimeout in *err. Every access stays inside
// `scratch` (lookback_probe_bytes(), zeroed here): the input and output of
// both tiles and the status words of tiles 0 and 1.
void launch_lookback_probe(cudaStream_t s, int which, unsigned spin_limit, char* scratch,
                           unsigned* err) {
    cudaMemsetAsync(scratch, 0, lookback_probe_bytes(), s);
    char* p = scratch;
    auto take = [&](size_t bytes) {
        char* q = p;
        p += align16(bytes);
        return q;
    };
    unsigned* counter = reinterpret_cast<unsigned*>(take(16)); // [0] tile counter [1] count
    unsigned* count = counter + 1;                              // [2] scan total
    unsigned* total = counter + 2;
    // pageable host source: the copy is staged before cudaMemcpyAsync returns
    const unsigned init[2] = {1u, 2u * kSortTile};
    cudaMemcpyAsync(counter, init, sizeof(init), cudaMemcpyHostToDevice, s);
    if (which == 0) {
        unsigned* in = reinterpret_cast<unsigned*>(take(2 * kScanTile * 4));
        unsigned* out = reinterpret_cast<unsigned*>(take(2 * kScanTile * 4));
        auto* status = reinterpret_cast<unsigned long long*>(take(2 * 8));
        scan_kernel<<<1, kBlock, 0, s>>>(2 * kScanTile, in, nullptr, out, status, counter, total,
                                         err, spin_limit, nullptr, 0, 0u);
    } else {
        unsigned* keys_in = reinterpret_cast<unsigned*>(take(2 * kSortTile * 4));
        unsigned* vals_in = reinterpret_cast<unsigned*>(take(2 * kSortTile * 4));
        unsigned* keys_out = reinterpret_cast<unsigned*>(take(2 * kSortTile * 4));
        unsigned* vals_out = reinterpret_cast<unsigned*>(take(2 * kSortTile * 4));
        unsigned* status = reinterpret_cast<unsigned*>(take(2 * 256 * 4));
        unsigned* offsets = reinterpret_cast<unsigned*>(take(256 * 4));
        // every key is 0: the block's 3,072 keys go to output positions below
        // its tile's prefix (0 once the wait gives up), all inside [0, 6144)
        onesweep_kernel<unsigned, 8><<<1, kBlock, 0, s>>>(keys_in, vals_in, keys_out, vals_out,
                                                          count, 0, offsets, status, counter,
                                                          err, spin_limit);
    }
}

template int launch_radix_sort<unsigned>(cudaStream_t, unsigned* [2], unsigned* [2], size_t,
                                         const unsigned*, int, int, unsigned*, unsigned*,
                                         unsigned*, unsigned*, bool, bool);
template int launch_radix_sort<unsigned long long>(cudaStream_t, unsigned long long* [2],
                                                   unsigned* [2], size_t, const unsigned*, int,
                                                   int, unsigned*, unsigned*, unsigned*,
                                                   unsigned*, bool, bool);

} // namespace gsb
