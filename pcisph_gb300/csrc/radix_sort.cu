// radix_sort.cu -- stable LSD radix sort (see radix_sort.cuh).
#include "radix_sort.cuh"
#include "spare_memory.h"

#include <algorithm>

namespace pcisph {
namespace {

// The digit passes run 512 threads a block: with 256 (16 keys each) a tile's ranking was a chain of 16 warp matches at 8
// warps a block, and the sort latency-bound at every size. Before -> now, us (CUDA events): 3,000,001 random 32-bit keys
// 295 -> 184 (with the caller's two copies), a step's keys: 1,048,576 60 -> 48, 156,244 54 -> 32, 32,768 44 -> 22,
// 4,096 40 -> 12 (one launch). What bounds it: the scattered writes of the downsweep at 3M, launches and one tile's
// latency below 1M.
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kFusedTiles = 64;  // up to here a downsweep block sums the tile counts itself (157K keys: 29 against 33 us)

constexpr size_t align256(size_t b) { return radix_align256(b); }

// Exclusive scan in place over s[0..count) in shared memory; returns the total. All T threads call.
template <int T>
__device__ uint32_t block_exclusive_scan(uint32_t* s, int count, uint32_t* warp_tmp) {
    constexpr int W = T / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (count + T - 1) / T;
    const int beg = min(count, (int)threadIdx.x * per), end = min(count, beg + per);
    uint32_t sum = 0;
    for (int i = beg; i < end; ++i) sum += s[i];
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tmp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < W ? warp_tmp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < W) warp_tmp[lane] = w;
    }
    __syncthreads();
    uint32_t run = x - sum + (warp > 0 ? warp_tmp[warp - 1] : 0u);
    const uint32_t total = warp_tmp[W - 1];
    for (int i = beg; i < end; ++i) {
        uint32_t v = s[i];
        s[i] = run;
        run += v;
    }
    __syncthreads();
    return total;
}

// The lanes of the warp whose key has this lane's digit d (all lanes call; an invalid lane's result is not used). A match
// takes a step per distinct digit, the ballots one per bit: keys that come nearly sorted hold few digits a warp (1M
// keys, first pass: match 10% faster), others one per lane (3M random keys: ballots 20% faster).
__device__ __forceinline__ unsigned same_digit(uint32_t d, bool valid, int bits, bool by_ballot) {
    if (!by_ballot) return __match_any_sync(0xffffffffu, valid ? d : 0xffffffffu);
    unsigned peers = __ballot_sync(0xffffffffu, valid);
    for (int b = 0; b < bits; ++b) {
        const bool on = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        peers &= on ? m : ~m;
    }
    return peers;
}

// Stable ranks of a thread's keys among its warp's keys with the same digit, in element order; hist (zeroed, one per
// warp) ends as the warp's digit counts.
template <int ITEMS>
__device__ __forceinline__ void rank_digits(const uint32_t (&k)[ITEMS], unsigned short (&rank)[ITEMS], uint32_t valid_n,
                                            int shift, int bits, bool by_ballot, unsigned short* hist) {
    const uint32_t lane = threadIdx.x & 31u, mask = (1u << bits) - 1u;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const bool valid = it * 32u + lane < valid_n;
        const uint32_t d = (k[it] >> shift) & mask;
        const unsigned peers = same_digit(d, valid, bits, by_ballot);
        const unsigned lower = peers & ((1u << lane) - 1u);
        const unsigned short cur = hist[d];
        rank[it] = (unsigned short)(cur + __popc(lower));
        __syncwarp();
        if (valid && lower == 0u) hist[d] = (unsigned short)(cur + __popc(peers));
        __syncwarp();
    }
}

// Per-tile digit counts: digit-major counts[d * tiles + tile], or (fused) tile-major counts[tile << BITS | d].
template <int BITS, int ITEMS>
__global__ void __launch_bounds__(kThreads) k_upsweep(const uint32_t* __restrict__ keys, uint32_t n, int shift,
                                                      uint32_t* __restrict__ counts, uint32_t tiles, bool fused) {
    constexpr int RADIX = 1 << BITS;
    __shared__ uint32_t hist[RADIX];
    for (int d = threadIdx.x; d < RADIX; d += kThreads) hist[d] = 0;
    const size_t base = (size_t)blockIdx.x * (kThreads * ITEMS) + threadIdx.x;
    uint32_t k[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) k[i] = base + i * kThreads < n ? __ldg(&keys[base + i * kThreads]) : 0u;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (base + i * kThreads < n) atomicAdd(&hist[(k[i] >> shift) & (RADIX - 1)], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < RADIX; d += kThreads)
        counts[fused ? ((size_t)blockIdx.x << BITS) + d : (size_t)d * tiles + blockIdx.x] = hist[d];
}

// One warp per digit: exclusive scan of that digit's tile counts; the row total goes to totals[d].
constexpr int kScanWarps = 8;
__global__ void __launch_bounds__(kScanWarps * 32) k_scan_rows(uint32_t* __restrict__ counts, uint32_t tiles,
                                                               uint32_t* __restrict__ totals) {
    const uint32_t d = blockIdx.x * kScanWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    uint32_t* row = counts + (size_t)d * tiles;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < tiles; base += 128u) {
        uint32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t i = base + 4u * lane + u;
            v[u] = i < tiles ? row[i] : 0u;
        }
        const uint32_t sum = v[0] + v[1] + v[2] + v[3];
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        uint32_t run = carry + x - sum;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t i = base + 4u * lane + u;
            if (i < tiles) row[i] = run;
            run += v[u];
        }
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) totals[d] = carry;
}

// The warps' digit counts hist[w][d] become each warp's offset among the tile's keys of that digit, and start[d] the
// place of the tile's first key with digit d.
template <int T>
__device__ __forceinline__ void tile_digit_starts(unsigned short* hist, uint32_t* start, int radix, uint32_t* warp_tmp) {
    for (int d = threadIdx.x; d < radix; d += T) {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < T / 32; ++w) {
            const uint32_t c = hist[w * radix + d];
            hist[w * radix + d] = (unsigned short)run;
            run += c;
        }
        start[d] = run;
    }
    __syncthreads();
    block_exclusive_scan<T>(start, radix, warp_tmp);
}

// Stable rank within the tile, stage in digit order, write each digit run contiguously. offsets: the digit-major scan of
// the tile counts and its totals, or (fused) the tile-major counts themselves.
template <int BITS, int ITEMS>
__global__ void __launch_bounds__(kThreads) k_downsweep(const uint32_t* __restrict__ keys_in,
                                                        const uint32_t* __restrict__ vals_in,
                                                        uint32_t* __restrict__ keys_out,
                                                        uint32_t* __restrict__ vals_out, uint32_t n, int shift,
                                                        const uint32_t* __restrict__ offsets,
                                                        const uint32_t* __restrict__ totals, uint32_t tiles, bool fused,
                                                        bool by_ballot) {
    constexpr int RADIX = 1 << BITS;
    constexpr uint32_t MASK = RADIX - 1;
    constexpr uint32_t TILE = kThreads * ITEMS;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned short* whist = reinterpret_cast<unsigned short*>(smem);              // [kWarps][RADIX]
    uint32_t* local_start = reinterpret_cast<uint32_t*>(whist + kWarps * RADIX);  // [RADIX]
    uint32_t* gofs = local_start + RADIX;                                         // [RADIX]
    uint32_t* skeys = gofs + RADIX;                                               // [TILE]
    uint32_t* svals = skeys + TILE;                                               // [TILE]
    __shared__ uint32_t warp_tmp[kWarps];

    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const size_t tile_base = (size_t)blockIdx.x * TILE;
    const uint32_t tile_n = (uint32_t)min((size_t)TILE, (size_t)n - tile_base);
    const uint32_t first = warp * 32u * ITEMS;  // this warp's keys of the tile
    const uint32_t warp_n = tile_n > first ? tile_n - first : 0u;
    uint32_t k[ITEMS], v[ITEMS];
    unsigned short rk[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const size_t idx = tile_base + first + it * 32u + lane;
        const bool valid = idx < n;
        k[it] = valid ? __ldg(&keys_in[idx]) : 0u;
        v[it] = valid ? (vals_in ? __ldg(&vals_in[idx]) : (uint32_t)idx) : 0u;
    }
    for (int i = threadIdx.x; i < kWarps * RADIX / 2; i += kThreads) reinterpret_cast<uint32_t*>(whist)[i] = 0u;
    for (int d = threadIdx.x; d < RADIX; d += kThreads) {
        uint32_t before = 0, all = 0;  // keys with this digit in the tiles before this one, in all tiles
        if (fused) {
#pragma unroll 8
            for (uint32_t t = 0; t < tiles; ++t) {
                const uint32_t c = __ldg(&offsets[((size_t)t << BITS) + d]);
                all += c;
                before += t < blockIdx.x ? c : 0u;
            }
        } else {
            before = __ldg(&offsets[(size_t)d * tiles + blockIdx.x]);
            all = __ldg(&totals[d]);
        }
        local_start[d] = before;
        gofs[d] = all;
    }
    __syncthreads();
    unsigned short* my_hist = whist + warp * RADIX;
    rank_digits<ITEMS>(k, rk, warp_n, shift, BITS, by_ballot, my_hist);
    block_exclusive_scan<kThreads>(gofs, RADIX, warp_tmp);
    for (int d = threadIdx.x; d < RADIX; d += kThreads) gofs[d] += local_start[d];
    __syncthreads();
    tile_digit_starts<kThreads>(whist, local_start, RADIX, warp_tmp);
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        if (it * 32u + lane < warp_n) {
            const uint32_t d = (k[it] >> shift) & MASK;
            const uint32_t pos = local_start[d] + my_hist[d] + rk[it];
            skeys[pos] = k[it];
            svals[pos] = v[it];
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const uint32_t i = it * kThreads + threadIdx.x;
        if (i < tile_n) {
            const uint32_t key = skeys[i];
            const uint32_t d = (key >> shift) & MASK;
            const uint32_t o = gofs[d] + (i - local_start[d]);
            keys_out[o] = key;
            vals_out[o] = svals[i];
        }
    }
}

// All passes of a small sort in one block, in place: the keys stay in registers and shared memory between the passes.
template <int T, int ITEMS>
__global__ void __launch_bounds__(T) k_sort_block(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n,
                                                  int passes, int bits, bool identity, bool nearly_sorted) {
    constexpr uint32_t TILE = T * ITEMS;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* skeys = reinterpret_cast<uint32_t*>(smem);                            // [TILE]
    uint32_t* svals = skeys + TILE;                                                 // [TILE]
    uint32_t* start = svals + TILE;                                                 // [256]
    unsigned short* whist = reinterpret_cast<unsigned short*>(start + 256);         // [T / 32][1 << bits]
    __shared__ uint32_t warp_tmp[T / 32];
    const int radix = 1 << bits;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, first = warp * 32u * ITEMS;
    const uint32_t warp_n = n > first ? n - first : 0u;
    uint32_t k[ITEMS], v[ITEMS];
    unsigned short rk[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const uint32_t idx = first + it * 32u + lane;
        k[it] = idx < n ? keys[idx] : 0u;
        v[it] = idx < n ? (identity ? idx : vals[idx]) : 0u;
    }
    for (int pass = 0; pass < passes; ++pass) {
        const int shift = pass * bits;
        for (int i = threadIdx.x; i < T / 64 * radix; i += T) reinterpret_cast<uint32_t*>(whist)[i] = 0u;
        __syncthreads();
        unsigned short* my_hist = whist + warp * radix;
        rank_digits<ITEMS>(k, rk, warp_n, shift, bits, !(nearly_sorted && pass == 0), my_hist);
        __syncthreads();
        tile_digit_starts<T>(whist, start, radix, warp_tmp);
#pragma unroll
        for (int it = 0; it < ITEMS; ++it)
            if (it * 32u + lane < warp_n) {
                const uint32_t d = (k[it] >> shift) & (uint32_t)(radix - 1);
                const uint32_t pos = start[d] + my_hist[d] + rk[it];
                skeys[pos] = k[it];
                svals[pos] = v[it];
            }
        __syncthreads();
        if (pass + 1 < passes)
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                const uint32_t idx = first + it * 32u + lane;
                k[it] = idx < n ? skeys[idx] : 0u;
                v[it] = idx < n ? svals[idx] : 0u;
            }
    }
    for (uint32_t i = threadIdx.x; i < n; i += T) {
        keys[i] = skeys[i];
        vals[i] = svals[i];
    }
}
template <int T, int ITEMS>
constexpr size_t block_sort_smem() {
    return 2 * (size_t)T * ITEMS * 4 + 256 * 4 + (size_t)(T / 32) * 256 * 2;
}
constexpr uint32_t kSmallBlockSort = 4096u, kBlockSort = 8192u;
static_assert(block_sort_smem<512, 8>() <= 48 * 1024, "the small block sort runs without a raised limit");

template <int BITS, int ITEMS>
constexpr size_t downsweep_smem() {
    static_assert(ITEMS != 8 || kThreads * ITEMS == kRadixTile, "tile size of the scratch layout (radix_sort.cuh)");
    return (size_t)kWarps * (1 << BITS) * sizeof(unsigned short) + 2 * ((size_t)1 << BITS) * sizeof(uint32_t) +
           2 * (size_t)kThreads * ITEMS * sizeof(uint32_t);
}

struct Pass {
    const uint32_t *kin, *vin;
    uint32_t *kout, *vout, *counts, *totals;
    uint32_t n;
    int shift;
    bool by_ballot;
};

template <int BITS, int ITEMS>
cudaError_t run_pass(const Pass& p, cudaStream_t s, int* launches) {
    constexpr uint32_t TILE = kThreads * ITEMS;
    const uint32_t tiles = (uint32_t)(((size_t)p.n + TILE - 1) / TILE);
    const bool fused = tiles <= (uint32_t)kFusedTiles;
    k_upsweep<BITS, ITEMS><<<tiles, kThreads, 0, s>>>(p.kin, p.n, p.shift, p.counts, tiles, fused);
    if (!fused) k_scan_rows<<<(1 << BITS) / kScanWarps, kScanWarps * 32, 0, s>>>(p.counts, tiles, p.totals);
    k_downsweep<BITS, ITEMS><<<tiles, kThreads, downsweep_smem<BITS, ITEMS>(), s>>>(
        p.kin, p.vin, p.kout, p.vout, p.n, p.shift, p.counts, p.totals, tiles, fused, p.by_ballot);
    *launches += fused ? 2 : 3;
    return cudaGetLastError();
}
// Digits of 4 to 11 bits; 4 keys a thread up to 8 bits, 16 from 8 bits (sort() takes them only there)
template <int ITEMS>
cudaError_t dispatch_pass(int bits, const Pass& p, cudaStream_t s, int* launches) {
    if constexpr (ITEMS < 16) {
        switch (bits) {
            case 4: return run_pass<4, ITEMS>(p, s, launches);
            case 5: return run_pass<5, ITEMS>(p, s, launches);
            case 6: return run_pass<6, ITEMS>(p, s, launches);
            case 7: return run_pass<7, ITEMS>(p, s, launches);
            default: break;
        }
    }
    if (bits == 8) return run_pass<8, ITEMS>(p, s, launches);
    if constexpr (ITEMS > 4) {
        switch (bits) {
            case 9: return run_pass<9, ITEMS>(p, s, launches);
            case 10: return run_pass<10, ITEMS>(p, s, launches);
            case 11: return run_pass<11, ITEMS>(p, s, launches);
            default: break;
        }
    }
    return cudaErrorInvalidValue;
}

template <int BITS, int ITEMS>
cudaError_t configure_one() {
    constexpr size_t smem = downsweep_smem<BITS, ITEMS>();
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(k_downsweep<BITS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}
template <int BITS>
cudaError_t configure_width() {
    const cudaError_t e = configure_one<BITS, 8>(), f = configure_one<BITS, 16>();
    return e != cudaSuccess ? e : f;
}

}  // namespace

cudaError_t radix_configure_kernels(int digit_bits) {
    cudaError_t e = cudaFuncSetAttribute(k_sort_block<1024, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)block_sort_smem<1024, 8>());
    if (e == cudaSuccess && digit_bits >= 8) e = configure_width<8>();
    if (e == cudaSuccess && digit_bits >= 9) e = configure_width<9>();
    if (e == cudaSuccess && digit_bits >= 10) e = configure_width<10>();
    if (e == cudaSuccess && digit_bits >= 11) e = configure_width<11>();
    return e;
}

RadixSorter::~RadixSorter() {
    if (owns_ && scratch_) cudaFree(scratch_);
}

void RadixSorter::set_scratch(void* ptr, size_t bytes) {
    if (owns_ && scratch_) cudaFree(scratch_);
    scratch_ = ptr;
    scratch_cap_ = bytes;
    owns_ = false;
}

cudaError_t RadixSorter::sort(uint32_t* keys, uint32_t* values, size_t n, int bits, bool values_in_identity,
                              cudaStream_t stream, uint32_t** out_keys, uint32_t** out_values) {
    last_launches_ = 0;
    if (out_keys) *out_keys = keys;
    if (out_values) *out_values = values;
    if (n == 0) return cudaSuccess;
    if (n > 0xFFFFFFFFull) return cudaErrorInvalidValue;
    if (bits <= 0 || bits > 32) bits = 32;
    const int db = digit_bits_;
    if (db < 4 || db > 11) return cudaErrorInvalidValue;
    const size_t need = scratch_bytes(n, db);
    if (scratch_cap_ < need) {
        if (!owns_ && scratch_) return cudaErrorInvalidValue;  // caller scratch too small
        if (scratch_) cudaFree(scratch_);
        scratch_ = nullptr;
        scratch_cap_ = 0;
        cudaError_t e = host::device_malloc(&scratch_, need);
        if (e != cudaSuccess) return e;
        scratch_cap_ = need;
        owns_ = true;
    }
    const size_t tiles = (n + kRadixTile - 1) / kRadixTile;
    unsigned char* p = static_cast<unsigned char*>(scratch_);
    uint32_t* alt_k = reinterpret_cast<uint32_t*>(p);
    p += align256(n * sizeof(uint32_t));
    uint32_t* alt_v = reinterpret_cast<uint32_t*>(p);
    p += align256(n * sizeof(uint32_t));
    uint32_t* counts = reinterpret_cast<uint32_t*>(p);
    p += align256(((size_t)1 << db) * tiles * sizeof(uint32_t));
    uint32_t* totals = reinterpret_cast<uint32_t*>(p);

    // The step's own sorts (identity values) have keys below 2^bits: their digits are no wider than the passes need. A
    // caller's sort covers passes * digit_bits bits.
    const int passes = (bits + db - 1) / db;
    const int width = values_in_identity ? std::max(4, (bits + passes - 1) / passes) : db;
    if (n <= kSmallBlockSort || (n <= kBlockSort && !small_smem_)) {
        const int covered = std::min(32, passes * width);
        const int block_passes = (covered + 7) / 8, block_bits = (covered + block_passes - 1) / block_passes;
        if (n <= kSmallBlockSort)
            k_sort_block<512, 8><<<1, 512, block_sort_smem<512, 8>(), stream>>>(
                keys, values, (uint32_t)n, block_passes, block_bits, values_in_identity, nearly_sorted_);
        else
            k_sort_block<1024, 8><<<1, 1024, block_sort_smem<1024, 8>(), stream>>>(
                keys, values, (uint32_t)n, block_passes, block_bits, values_in_identity, nearly_sorted_);
        last_launches_ = 1;
        return cudaGetLastError();
    }
    // Keys a thread: 4 while the tiles are few (32,768 keys: 21 against 25 us with 8), where their counts fit the scratch,
    // 16 from 512K keys (1M: 43 against 45 us with 8; shared memory past the default limit).
    const bool few = n <= 65536 && width <= 8 && (2 * tiles << width) <= (tiles << db);
    const bool many = n >= (1u << 19) && width >= 8 && !small_smem_;
    uint32_t *sk = keys, *sv = values, *dk = alt_k, *dv = alt_v;
    for (int pass = 0; pass < passes; ++pass) {
        const Pass ps{sk, (pass == 0 && values_in_identity) ? nullptr : sv, dk, dv, counts, totals, (uint32_t)n,
                      pass * width, !(nearly_sorted_ && pass == 0)};
        const cudaError_t e = few    ? dispatch_pass<4>(width, ps, stream, &last_launches_)
                              : many ? dispatch_pass<16>(width, ps, stream, &last_launches_)
                                     : dispatch_pass<8>(width, ps, stream, &last_launches_);
        if (e != cudaSuccess) return e;
        std::swap(sk, dk);
        std::swap(sv, dv);
    }
    if (sk != keys) {
        if (out_keys && out_values) {
            *out_keys = sk;
            *out_values = sv;
        } else {
            cudaError_t e = cudaMemcpyAsync(keys, sk, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, stream);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(values, sv, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, stream);
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

}  // namespace pcisph
