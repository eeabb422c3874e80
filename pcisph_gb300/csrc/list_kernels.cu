// list_kernels.cu -- neighbour-list sweeps (kernel_variant 2), for one scene or a batch of scenes.
//
// The density sweep walks the reference's 27 buckets (grid_utils.cl:65-79) once per step and records,
// per particle and in walk order, two lists: every candidate j with |x_i - x_j| <= r_list = h (1 + skin),
// and the subset within h (plus a 1e-4 relative margin, far above rounding). The later sweeps of the step
// iterate a list instead of walking the buckets again: the sweeps at the current positions (normal,
// force, pressure force) the within-h list (~34 candidates), the pressure sweeps of the corrective
// iterations the skin list (~65-80), instead of the walk's ~210. Because a list keeps the walk order and
// drops only pairs that contribute exactly zero, the sums are the reference's sums in the reference's
// order.
//
// Exactness conditions, checked on the device:
//   - sweeps at the current positions x (normal, force, pressure force) need |x_i - x_j| <= h, always in
//     the within-h list;
//   - the pressure sweep measures distances between predicted positions x*. A pair with
//     |x*_i - x*_j| <= h has |x_i - x_j| <= h + |x*_i - x_i| + |x*_j - x_j|, so it is in both lists when
//     both displacements are at most half the skin. A particle whose displacement exceeds that ("fast")
//     flags its own bucket when it predicts x*. In a pressure sweep after any fast prediction, a particle
//     whose 27 buckets include a flagged one walks the buckets instead of using its list: every pair with a
//     fast particle j in i's walk (spatial neighbour or hash collision) is then summed by a walk. Flags
//     last for the rest of the step;
//   - in a step of moving lists (lists_move: many particles faster than half the skin per step) the skin lists are
//     built around y = x + v dt instead of x, and a prediction is fast when it strays half the skin from there;
//   - from the third pressure sweep of a step on, the sweeps read tight lists rebuilt at the second one's
//     predictions, as long as no prediction has moved past their margin from there (see the tight lists);
//   - a particle with more than list_cap (near_cap) candidates is marked (count > cap) and walks the
//     buckets in the sweeps that would use that list.
// Boundary particles (B > 0, single scene) are summed by walking the boundary buckets. The density sweep
// records per particle whether any boundary particle lies within r_list of x (b_near); boundary particles
// do not move, so a particle without one has only zero boundary terms in the pressure-force sweep (pairs
// within h of x) and, unless its prediction moved more than half the skin, in the pressure sweeps: those
// skip the boundary walk (27 bucket lookups and the hash-colliding boundary particles they hold).
//
// Parameter sources (list_kernels.cuh): OneScene passes one DevParams by value and the pressure kernel's
// last block decides the loop. SceneTable serves a batch: particle i belongs to scene scene_of[i], whose
// DevParams (own particle count, bucket count and base in the shared cell table, box, limits) and Control
// live in device tables. Scenes stay contiguous in the sorted arrays because each scene's keys occupy its
// own bucket range. k_batch_decide closes each iteration per scene; finished scenes skip the sweeps.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "list_kernels.cuh"
#include "pair_terms.cuh"
#include "sweep_device.cuh"

namespace pcisph {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kSms = 152u;  // of a GB300: launch shapes that fill it (results do not depend on them)
inline unsigned grid_for(uint32_t n) { return (n + kBlock - 1) / kBlock; }

// List layout: entries k = 8c .. 8c+7 of particle i (chunk c) are 32 contiguous bytes at uint4 offset
// 2 (c * stride + i); chunks are column-major over particles. A warp's 32 consecutive particles read
// chunk c as 1 KB of contiguous memory, and the builder writes whole 32-byte sectors.
__device__ __forceinline__ uint4* list_chunk(uint32_t* list, uint32_t i, uint32_t c, uint32_t stride) {
    return reinterpret_cast<uint4*>(list) + 2 * ((size_t)c * stride + i);
}

// One float4 of data that the step's kernels write: the read-only path, or (kCoherent) a plain load for data
// that other blocks of the same launch wrote before a grid barrier (the persistent loop), which the
// read-only path may serve stale.
template <bool kCoherent>
__device__ __forceinline__ float4 load_slot(const float4* p) {
    if constexpr (kCoherent) return *p;
    else return __ldg(p);
}

// A chunk's eight indices, as one 256-bit load: two 128-bit loads of a warp each touch every line of its 1 KB, and the
// sweeps are bound by the L1 data pipe. The lists are read once a sweep and written by earlier launches: through the
// read-only path, past L1 (which is left to the gathered particles; with .cs instead the within-h sweeps lost 8%, with
// evict-first lines the pressure sweep 0.6%). Pressure sweep, two 128-bit streaming loads -> this: 286,720 particles with
// boundary 42 -> 37 us, 1,048,576 135 -> 126, 8,388,608 1037 -> 957; pressure force at 1M 78.5 -> 77.3.
struct Chunk {
    uint32_t e[8];
};
__device__ __forceinline__ Chunk load_chunk(const uint4* p) {
    Chunk r;
    asm("ld.global.nc.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r.e[0]), "=r"(r.e[1]), "=r"(r.e[2]), "=r"(r.e[3]), "=r"(r.e[4]), "=r"(r.e[5]), "=r"(r.e[6]),
                   "=r"(r.e[7])
                 : "l"(p));
    return r;
}

__device__ __forceinline__ void store_chunk(uint4* p, const Chunk& r) {
    asm volatile("st.global.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"r"(r.e[0]), "r"(r.e[1]), "r"(r.e[2]),
                 "r"(r.e[3]), "r"(r.e[4]), "r"(r.e[5]), "r"(r.e[6]), "r"(r.e[7]), "l"(p)
                 : "memory");
}

// Call f(j) for the n listed neighbours of particle i in list order. The next chunk's indices are loaded
// while the current chunk's eight gathers are in flight, so the list stream and the gathers overlap.
template <class F>
__device__ __forceinline__ void for_each_listed(const uint32_t* __restrict__ list, uint32_t i, uint32_t n,
                                                uint32_t stride, F&& f) {
    const uint32_t chunks = (n + 7u) >> 3;
    if (!chunks) return;
    const uint4* p = list_chunk(const_cast<uint32_t*>(list), i, 0, stride);
    const size_t step = 2 * (size_t)stride;
    Chunk a = load_chunk(p);
#pragma unroll 1
    for (uint32_t c = 0; c < chunks; ++c) {
        Chunk next{};
        if (c + 1 < chunks) {
            p += step;
            next = load_chunk(p);
        }
        const uint32_t left = n - 8u * c;  // entries in this chunk: min(8, left)
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if ((uint32_t)u < left) f(a.e[u]);
        a = next;
    }
}

// The same where f has side effects that the compiler does not move loads across: a chunk's values first, then
// use(j, value(j)) for each; after each chunk, done().
template <class Value, class Use, class Done>
__device__ __forceinline__ void for_each_listed_ahead(const uint32_t* __restrict__ list, uint32_t i, uint32_t n,
                                                      uint32_t stride, Value&& value, Use&& use, Done&& done) {
    if (!n) return;
    const uint4* p = list_chunk(const_cast<uint32_t*>(list), i, 0, stride);
    Chunk a = load_chunk(p);
#pragma unroll 1
    for (uint32_t e = 0; e < n; e += 8u) {
        decltype(value(0u)) o[8];
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            if (e + u < n) o[u] = value(a.e[u]);
        Chunk next{};
        if (e + 8u < n) {
            p += 2 * (size_t)stride;
            next = load_chunk(p);
        }
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u)
            if (e + u < n) use(a.e[u], o[u]);
        done();
        a = next;
    }
}

// The same with the gathers of U chunks in flight before their first use (load(j), then use(value) in list order): for
// scenes of few warps, where nothing else covers a gather's latency.
template <int U, class Load, class Use>
__device__ __forceinline__ void for_each_listed_deep(const uint32_t* __restrict__ list, uint32_t i, uint32_t n,
                                                     uint32_t stride, Load&& load, Use&& use) {
    const uint4* p = list_chunk(const_cast<uint32_t*>(list), i, 0, stride);
    const size_t step = 2 * (size_t)stride;
    uint32_t j[8 * U];
    auto fetch = [&](uint32_t e) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e + 8u * u < n) {
                const Chunk a = load_chunk(p + u * step);
#pragma unroll
                for (int q = 0; q < 8; ++q) j[8 * u + q] = a.e[q];
            }
        p += U * step;
    };
    fetch(0u);
#pragma unroll 1
    for (uint32_t e = 0; e < n; e += 8u * U) {
        decltype(load(0u)) o[8 * U];
#pragma unroll
        for (uint32_t k = 0; k < 8u * U; ++k)
            if (e + k < n) o[k] = load(j[k]);
        fetch(e + 8u * U);
#pragma unroll
        for (uint32_t k = 0; k < 8u * U; ++k)
            if (e + k < n) use(o[k]);
    }
}

// ------------------------------------------------------------------ small scenes: eight lanes per particle
//
// A scene that fills less than a wave of threads is bound by each thread's chain of loads and sums (15 us a sweep from
// 4,096 to 32,768 particles). There eight lanes share a particle: lane q takes entry 8c + q of chunk c, so a chunk is one
// gather per lane instead of eight in a row, and the entries' terms are then summed in list order (the sum of the
// one-lane sweep: entries that contribute nothing add zero).

// The entries of this lane, chunk by chunk, in batches of U chunks whose gathers are in flight together: load(j) for
// the lane's entry, then sum(value, entry, valid) once per chunk by the whole warp. n: this particle's entries; most: the
// warp's largest n.
template <int L, int U, class Load, class Sum>
__device__ __forceinline__ void for_each_shared(const uint32_t* __restrict__ list, uint32_t i, uint32_t n, uint32_t most,
                                                uint32_t stride, uint32_t q, Load&& load, Sum&& sum) {
    const uint32_t* p = list + 8 * (size_t)i;
    auto entry = [&](uint32_t e) { return __ldcs(p + (e >> 3) * (8 * (size_t)stride) + (e & 7u)); };
    uint32_t j[U];
#pragma unroll
    for (int u = 0; u < U; ++u) j[u] = q + L * u < n ? entry(q + L * u) : 0u;
#pragma unroll 1
    for (uint32_t e = q; e - q < most; e += L * U) {
        decltype(load(0u)) o[U];
        uint32_t k[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (e + L * u < n) o[u] = load(j[u]);
            k[u] = j[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) j[u] = e + L * (U + u) < n ? entry(e + L * (U + u)) : 0u;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e - q + L * u < most) sum(o[u], k[u], e + L * u < n);
    }
}

// The lane's candidates of a walk over the buckets around c, eight at a time: use(j, valid) by the eight lanes (mask).
template <int L, class Use>
__device__ __forceinline__ void walk_shared(const uint2* __restrict__ cells, const Cell& c, const DevParams& P, uint32_t q,
                                            Use&& use) {
    for_each_bucket(cells, c, P, [&](uint2 r) {
        for (uint32_t j = r.x; j < r.y; j += L) use(j + q, j + q < r.y);
    });
}

// The L lanes that share this lane's particle.
template <int L>
__device__ __forceinline__ uint32_t lanes_mask() {
    return ((1u << L) - 1u) << (threadIdx.x & 31u & ~(L - 1u));
}

// acc plus the L lanes' terms in lane order.
template <int L>
__device__ __forceinline__ void add_lanes(float& acc, float term, uint32_t mask) {
#pragma unroll
    for (int k = 0; k < L; ++k) acc += __shfl_sync(mask, term, k, L);
}

// Vector terms of eight lanes, summed in lane order, one component per lane: lane q < 3 holds component q of the sum.
template <int L>
struct TermStage {
    float4 t[L];
};
template <int L>
__device__ __forceinline__ void add_lanes(float& acc, const PairTerm& term, TermStage<L>& s, uint32_t q, uint32_t mask) {
    s.t[q] = make_float4(term.x, term.y, term.z, term.k);
    __syncwarp(mask);
    const float* v = reinterpret_cast<const float*>(s.t) + (q < 3u ? q : 0u);
#pragma unroll
    for (int k = 0; k < L; ++k) acc = __fmaf_rn(v[4 * k], s.t[k].w, acc);
    __syncwarp(mask);
}

// Does any of the 27 buckets around c hold a fast particle this step?
__device__ __forceinline__ bool near_fast(const DevParams& P, const unsigned char* __restrict__ bucket_fast,
                                          const Cell& c) {
    bool any = false;
#pragma unroll 1
    for (int dz = -1; dz <= 1; ++dz) {
        const uint32_t z = c.z + (uint32_t)dz;
        const uint32_t hz = z * 83492791u, lz = 16u * (z & 63u);
#pragma unroll 1
        for (int dy = -1; dy <= 1; ++dy) {
            const uint32_t y = c.y + (uint32_t)dy;
            const uint32_t hyz = (y * 73856093u) ^ hz, lyz = 4u * (y & 63u) + lz;
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                const uint32_t x = c.x + (uint32_t)dx;
                const uint32_t v = (((x * 19349663u) ^ hyz) << 6) + (x & 63u) + lyz;
                any |= bucket_fast[P.bucket_base + mod_bk(v & 0x7FFFFFFFu, P)] != 0;
            }
        }
    }
    return any;
}

// ------------------------------------------------------------------ list builders: one warp per few particles
//
// A warp serves W consecutive particles, cell by cell (consecutive particles mostly share one). The candidates of a
// cell's 27 buckets, concatenated in walk order, sit in registers, 32 a round: every particle of the cell tests them
// without loading them again, and the hits of a round are appended in walk order by ballot. Tests run with all lanes
// busy, where a thread per particle walked with half of its lanes idle (buckets of unequal length, divergent appends),
// and a small scene has 4 to 16 times more warps in flight. Builder per launch (CUDA events), thread per particle -> this:
// 4,096 particles 72 -> 10 us, 32,768 96 -> 27, 156,244 138 -> 82, 1,048,576 649 -> 495, batch of 1.32M 815 -> 538;
// the boundary's fluid lists (103,736 boundary particles) 61 -> 37. What bounds it at 1M: issue (73% of the slots; of
// ~416 instructions a particle 145 are the tests, 90-120 the set-up of a cell's candidates, the rest the compaction
// into the two lists); 613 instructions a particle before, with 15 of 32 lanes active.
constexpr int kCellRounds = 10;   // candidate rounds in registers: 320, a full neighbourhood at rest density with its
                                  // hash collisions holds ~270 (9 rounds: 508 us at 1M, more cells take two passes;
                                  // 12: 614, fewer warps)
constexpr int kCellBlock = 128;   // 4 warps a block, 20 resident per SM (24 spill: 501 us)
constexpr uint32_t kAll = 0xffffffffu;

// ------------------------------------------------------------------ tight lists
//
// The first correction moves a prediction most (0.05 h and more), the later ones little: from the second prediction x*_2 on
// no particle of a collapsing column, a tank or a falling drop moves 0.035 h within a step of 7 iterations, and within one
// of 50 they pass that a few times. So the second pressure sweep of a step also writes, per particle and in walk order, the
// entries within h + 2 m of it (m = kTightMargin h; 40 of the skin list's 65 at rest density), and the later sweeps read
// those: 1,048,576 particles 126 us a sweep -> 82, 8,388,608 957 -> 544, 98,904 falling 21 -> 11; the building sweep costs
// 186, 1420 and 26. A step of 50 iterations of 8.4M particles 83.2 -> 68.2 ms, one of 6 at 1M 2060 -> 1990 us.
//
// Exact: a pair within h at later predictions, neither of which has moved more than m since, was within h + 2 m at the
// building. So the tight list of a particle that walked then holds every pair of its walk that comes within h; and that of
// one that read its skin list holds every such pair of the skin list, which is all of them unless the particle has to
// walk by the rules of the skin lists (fast predictions' flags or marks). It does walk where these say so, and did not in the
// building sweep. A fast prediction that was fast at the building, too, asks nobody again: there its partners within h + 2 m
// were marked (or all near its bucket flagged), and walked. Where others keep crossing half the skin, sweep after sweep asks the
// marks: a long loop builds the lists anew then, with the predictions flagged that came within m of it (99,768 / 150,000 /
// 186,000 particles that fall at 0.09 h a step, 50 iterations, before moving lists took them: 2500 / 2910 / 3540 us a step
// without, 2300 / 2510 / 3120 with). A particle with more than kTightCap entries walks in every sweep that would read them. One prediction
// out of reach (or NaN) puts the whole scene back on the skin lists, and from iteration kTightAgain on rebuilds: a building sweep in the loop (it stores entry by
// entry, 1670 us at 8.4M) pays from three sweeps that use it, which a loop of fewer iterations need not have left.
// Margins at 1M / 8.4M / a 98,904-particle drop, us a step: 0.02 2284 / 70510 / 1880, 0.03 1998 / 68148 / 1840, 0.04 2018 /
// 67244 / 1821.
//
// A list that held the pairs without asking again (every prediction flagged that came within m of half the skin) cost more than
// it spared wherever many did: 1,000,000 particles at 2 m/s 4480 us a step, 2770 now (3710 without tight lists); a tank at
// list_skin 0.1 1240, 750 now.
//
// A step of 3 iterations gains nothing (378 us of sweeps at 1M, 399 with them): the lists are built where the previous step
// took 4 or more. Batch of 32 scenes, 1.32M particles: 46.4 -> 44.6 ms for 16 steps (46.3 without that rule: its falling
// spheres walk in the building sweep, 456 us, for loops of 3).
//
// With per-particle skins (scenes with boundary particles) 1,048,576 fluid particles in a tank 2454 -> 2382 us a step, 279,936
// 862 -> 840. Eight lanes per particle: 4,096 particles at rest 159 -> 157 us, 8,000 violently jittered 985 -> 667.
//
// Skin lists narrower than this hold too few of the later pairs: the building sweep walks throughout, and every tight list is
// complete (list_skin 0.05, 4,096 particles 350 -> 183 us a step; from 0.08 on the lists are read, 140).
__device__ __forceinline__ bool tight_by_walks(const DevParams& P) { return P.skin_max_half < 1.05f * P.tight_margin; }
// The control fields that decide over the tight lists, loaded together: one thread decides at the end of a sweep, and small
// scenes wait for it.
struct TightState {
    unsigned next, stray, age, wait, backoff, iter, outrun, asked, early;
    int last;
    bool moves;
    unsigned long long fast, before, sweeps;
    __device__ __forceinline__ TightState(const DevParams& P, const Control* c)
        : next(tight_plan(c->tight_next)), stray(c->tight_stray), age(c->tight_age), wait(c->tight_wait), backoff(c->tight_backoff),
          iter(c->iter), outrun(c->tight_outrun), asked(c->tight_asked), early(c->tight_next & kTightEarly),
          last(c->iterations_last), moves(lists_move(P, c)), fast(c->fast_particles), before(c->fast_before),
          sweeps(c->tight_sweeps) {}
    __device__ __forceinline__ unsigned mode(const DevParams& P) const {
        if (next == kTightOff || (next == kTightUse && stray == 0u)) return next;
        const bool again = age != 0u && iter >= kTightAgain && (int)iter + 1 < P.max_iters;
        // many fast predictions of a scene that moving lists do not serve go apart (kTightShare); elsewhere they may go together
        const bool few = !P.moving_lists || moves || tight_by_walks(P) || P.fluid_count <= kSharedMax ||
                         fast - before <= P.fluid_count / kTightShare;
        return (next == kTightBuild || again) && few ? kTightBuild : kTightOff;
    }
};
// How this pressure sweep finds its neighbours (constant while it runs), and whether some prediction outran the lists that it
// reads.
struct ListState {
    unsigned mode;
    bool outrun;
};
template <bool kTight>
__device__ __forceinline__ ListState list_state(const DevParams& P, const Control* ctl, bool on) {
    const uint4 s = *reinterpret_cast<const uint4*>(&ctl->tight_next);  // next, stray, outrun, outrun since the building
    if (!kTight || !on) return ListState{kTightOff, s.z != 0u};
    unsigned mode = tight_plan(s.x);
    if (mode == kTightBuild || (mode == kTightUse && s.y != 0u)) mode = TightState(P, ctl).mode(P);
    return ListState{mode, (mode == kTightUse ? s.w : s.z) != 0u};
}
// After a pressure sweep (before the decision): what the next one does (returned, too). marks: the sweep took marks, not flags.
__device__ __forceinline__ unsigned tight_advance(const DevParams& P, Control* ctl, bool on, bool marks) {
    if (!on) return kTightOff;
    const TightState t(P, ctl);
    const unsigned m = t.mode(P);
    unsigned next = t.next | t.early;
    if (m == kTightUse) {
        ctl->tight_age = t.age + 1u;
        ctl->tight_sweeps = t.sweeps + 1ull;
        if (t.age != 0u && t.backoff != 0u) ctl->tight_backoff = 0;
        if (t.outrun != 0u && t.early == 0u) {
            ctl->tight_asked = t.asked + 1u;
            if (t.asked + 1u >= kTightAsked && t.last >= (int)(t.iter + kTightEarlyLeft)) {
                next = kTightBuild | kTightEarly;
            }
        }
    } else if (m == kTightBuild) {
        // built at once, after a stray: nothing was flagged early
        next = t.next == kTightUse ? kTightUse : kTightUse | t.early;
        ctl->tight_age = 0;
        ctl->tight_stray = 0;
        ctl->tight_marked = marks ? 1u : 0u;
        ctl->tight_outrun = 0;
    } else if (t.next != kTightOff) {  // left behind, or not built
        if (t.age == 0u) ctl->tight_wait = ctl->tight_backoff = min(2u * t.backoff + 1u, 63u);  // they served no sweep
        next = kTightOff;
    } else if (t.wait != 0u) {
        ctl->tight_wait = t.wait - 1u;
    } else if ((t.iter == 0u ? t.last == 0 || t.last >= kTightFrom : t.iter + 1u >= kTightAgain) && (int)t.iter + 2 < P.max_iters) {
        next = kTightBuild;
        ctl->tight_age = 0;
    }
    if (next != (t.next | t.early)) ctl->tight_next = next;
    ctl->fast_before = t.fast;
    return tight_plan(next);
}
// A lane's tight list in the making. kShared: two chunks staged in shared memory, a chunk written out when it is full (whole
// sectors; 188 us at 1M). Otherwise entry by entry: the sweeps of the loop, which seldom build, keep the L1 (16 KB of
// staging a block cost each of them 5 to 10%).
template <bool kShared>
struct TightWriter {
    uint32_t* list;
    uint32_t i, stride, n;
    uint32_t* column;  // kShared: the lane's column of [16][32]
    __device__ __forceinline__ TightWriter(uint32_t* list, uint32_t i, uint32_t stride, uint32_t* stage)
        : list(list), i(i), stride(stride), n(0), column(kShared ? stage + (threadIdx.x & 31u) : nullptr) {}
    __device__ __forceinline__ void add(uint32_t j) {
        if constexpr (kShared) column[(n & 15u) * 32u] = j;
        else if (n < kTightCap) reinterpret_cast<uint32_t*>(list_chunk(list, i, n >> 3, stride))[n & 7u] = j;
        ++n;
    }
    __device__ __forceinline__ void flush(uint32_t c) const {
        if constexpr (kShared) {
            if (c >= kTightCap / 8u) return;
            Chunk k;
#pragma unroll
            for (uint32_t u = 0; u < 8u; ++u) k.e[u] = column[((c & 1u) * 8u + u) * 32u];
            store_chunk(list_chunk(list, i, c, stride), k);
        }
    }
    __device__ __forceinline__ void finish() const {
        if (n & 7u) flush(n >> 3);
    }
};

constexpr unsigned long long kNoMarks = 1ull << 40;  // a round's count past any cap of the partner marks

// A warp's working set: the hits of one particle (index, |d|^2 bits), the cell's bucket offsets, the particles.
template <int W>
struct CellWarp {
    uint2 hit[kCellRounds * 32 + 32];  // 32 entries beyond the last hit: no distance (+inf)
    uint32_t delta[32];
    float4 target[W];  // x, y, z, list radius^2
};
// The density builder also stages each particle's near list: (index, poly6 term), in walk order.
template <int W>
struct DensityWarp : CellWarp<W> {
    uint2 near[W][kNearCap + 1];
};

__device__ __forceinline__ uint32_t lanes_below() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
// A shared store where a <= b, predicated (a branch costs the warp a reconvergence per round).
__device__ __forceinline__ void store_shared_le(float a, float b, uint32_t addr, uint32_t v0, uint32_t v1) {
    asm volatile("{ .reg .pred q; setp.le.f32 q, %0, %1; @q st.shared.v2.b32 [%2], {%3, %4}; }" ::"f"(a), "f"(b),
                 "r"(addr), "r"(v0), "r"(v1)
                 : "memory");
}

// The candidates of one cell: the 27 buckets in the reference's walk order (grid_utils.cl:68-69), one per lane.
// delta[k] turns a position in the concatenation into a particle index for the k-th bucket that is not empty.
struct CellWalk {
    uint32_t total;  // candidates of the cell
    uint32_t off;    // where this lane's bucket begins in the concatenation (kAll: empty, or no bucket)
    uint32_t rank;   // the last bucket begun before the next round
};
// The lanes' ranges concatenated in lane order.
__device__ __forceinline__ CellWalk concatenate(const uint2& r, uint32_t lane, uint32_t* delta) {
    const uint32_t len = r.y > r.x ? r.y - r.x : 0u;
    uint32_t incl = len;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, incl, o);
        if (lane >= o) incl += y;
    }
    CellWalk w;
    w.total = __shfl_sync(kAll, incl, 31);
    w.rank = kAll;
    const uint32_t filled = __ballot_sync(kAll, len != 0u);
    w.off = len ? incl - len : kAll;
    __syncwarp();  // the last reads of delta are done
    if (len) delta[__popc(filled & lanes_below())] = r.x - w.off;
    __syncwarp();
    return w;
}
__device__ __forceinline__ CellWalk begin_cell(const uint2* __restrict__ cells, const DevParams& P, uint32_t cx,
                                               uint32_t cy, uint32_t cz, uint32_t lane, uint32_t* delta) {
    uint2 r = make_uint2(0u, 0u);
    if (lane < 27u) {
        const uint32_t dz = lane / 9u, dy = (lane / 3u) % 3u, dx = lane % 3u;
        r = __ldg(&cells[P.bucket_base + hash_key(cx + dx - 1u, cy + dy - 1u, cz + dz - 1u, P)]);
    }
    return concatenate(r, lane, delta);
}

// The particle at position base + lane of the concatenation (kAll past its end); base goes up by 32 from 0.
__device__ __forceinline__ uint32_t next_candidate(CellWalk& w, uint32_t base, uint32_t lane, const uint32_t* delta) {
    // the buckets that begin in this round, as bits of their first position
    const uint32_t rel = w.off - base;
    const uint32_t begun = __reduce_or_sync(kAll, rel < 32u ? 1u << rel : 0u);
    const uint32_t f = base + lane, k = w.rank + __popc(begun & (2u * lanes_below() + 1u));
    w.rank += __popc(begun);
    return f < w.total ? f + delta[k & 31u] : kAll;
}

// The next kCellRounds rounds of candidates from position base: index and position, NaN beyond the last (no test
// accepts it). odd: some candidate has a coordinate that is not finite.
struct Candidates {
    uint32_t j[kCellRounds];
    float x[kCellRounds], y[kCellRounds], z[kCellRounds];
    uint32_t count;  // of these rounds
    bool odd;
};
template <class Place>
__device__ __forceinline__ void load_candidates(Candidates& c, CellWalk& w, uint32_t base, uint32_t lane,
                                                const uint32_t* delta, Place&& place) {
    const uint32_t at_or_below = 2u * lanes_below() + 1u;
    const float nan = __uint_as_float(0x7fffffffu);
    float zero = 0.f;  // stays 0 while every coordinate is finite
    c.count = min(w.total - base, (uint32_t)kCellRounds * 32u);
#pragma unroll
    for (int u = 0; u < kCellRounds; ++u) {
        // next_candidate, written out: as a call with its end test on the result the builder took 490 us at 1M, not 482
        const uint32_t rel = w.off - (base + u * 32u);
        const uint32_t begun = __reduce_or_sync(kAll, rel < 32u ? 1u << rel : 0u);
        const uint32_t f = base + u * 32u + lane;
        const uint32_t k = w.rank + __popc(begun & at_or_below);
        w.rank += __popc(begun);
        c.j[u] = 0u;
        c.x[u] = c.y[u] = c.z[u] = nan;
        if (f < w.total) {
            c.j[u] = f + delta[k & 31u];
            const float4 o = place(c.j[u]);
            c.x[u] = o.x;
            c.y[u] = o.y;
            c.z[u] = o.z;
            zero = __fmaf_rn(o.x, 0.f, __fmaf_rn(o.y, 0.f, __fmaf_rn(o.z, 0.f, zero)));
        }
    }
    c.odd = __any_sync(kAll, !(zero == 0.f));
}

// The candidates within sqrt(q.w) of q, into hit[] in walk order; returns their number (the whole warp calls, with
// the same q).
__device__ __forceinline__ uint32_t collect_hits(const Candidates& c, const float4& q, uint2* hit, uint32_t lane) {
    const uint32_t hit_addr = (uint32_t)__cvta_generic_to_shared(hit);
    const uint32_t below = lanes_below();
    uint32_t n = 0;
    __syncwarp();  // the last particle's hits have been read
#pragma unroll
    for (int u = 0; u < kCellRounds; ++u) {
        if (u < 6 || u * 32u < c.count) {
            const float r2 = dist2(q.x - c.x[u], q.y - c.y[u], q.z - c.z[u]);
            const uint32_t bits = __ballot_sync(kAll, r2 <= q.w);
            store_shared_le(r2, q.w, hit_addr + 8u * (n + __popc(bits & below)), c.j[u], __float_as_uint(r2));
            n += __popc(bits);
        }
    }
    hit[n + lane] = make_uint2(0u, 0x7f800000u);
    __syncwarp();
    return n;
}

// Is the distance of q from some candidate NaN (a rare path: some candidate is not finite)?
__device__ __forceinline__ bool nan_distance(const Candidates& c, const float4& q, uint32_t lane) {
    bool nan = false;
#pragma unroll
    for (int u = 0; u < kCellRounds; ++u) {
        const float r2 = dist2(q.x - c.x[u], q.y - c.y[u], q.z - c.z[u]);
        nan |= u * 32u + lane < c.count && r2 != r2;
    }
    return __any_sync(kAll, nan);
}

// Entry s of particle i's list.
__device__ __forceinline__ uint32_t* list_entry(uint32_t* list, uint32_t i, uint32_t s, uint32_t stride) {
    return list + 8 * ((size_t)(s >> 3) * stride + i) + (s & 7u);
}

// The fluid particles within r_list of each boundary particle at the step's start, in the order of the walk of
// pcisph.cl:212-263 with boundary_update = 1 (27 fluid buckets around the boundary particle's cell).
__global__ void __launch_bounds__(kCellBlock, 5) k_boundary_fluid_list(DevParams P, ListBuffers b) {
    constexpr int W = 8;
    __shared__ CellWarp<W> warps[kCellBlock / 32];
    CellWarp<W>& S = warps[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t k0 = (blockIdx.x * (kCellBlock / 32) + (threadIdx.x >> 5)) * W;
    if (k0 >= P.boundary_count) return;
    const uint32_t me = k0 + lane;
    const bool own = lane < W && me < P.boundary_count;
    const float4 xb = b.b_pos[own ? me : k0];
    const Cell c = cell_of(xb.x, xb.y, xb.z, P);
    if (lane < W) S.target[lane] = make_float4(xb.x, xb.y, xb.z, P.list_r2);
    uint32_t n_own = 0;
    uint32_t todo = __ballot_sync(kAll, own);
    while (todo) {
        const int lead = __ffs(todo) - 1;
        const uint32_t cx = __shfl_sync(kAll, c.x, lead), cy = __shfl_sync(kAll, c.y, lead),
                       cz = __shfl_sync(kAll, c.z, lead);
        const uint32_t group = __ballot_sync(kAll, c.x == cx && c.y == cy && c.z == cz) & todo;
        todo &= ~group;
        CellWalk w = begin_cell(b.cells, P, cx, cy, cz, lane, S.delta);
        for (uint32_t base = 0; base < w.total; base += kCellRounds * 32u) {
            Candidates cand;
            load_candidates(cand, w, base, lane, S.delta, [&](uint32_t j) { return __ldg(&b.pos[j]); });
            for (uint32_t g = group; g; g &= g - 1u) {
                const int t = __ffs(g) - 1;
                const uint32_t n = collect_hits(cand, S.target[t], S.hit, lane);
                const uint32_t n0 = __shfl_sync(kAll, n_own, t);
                for (uint32_t k = lane; k < n; k += 32u)
                    if (n0 + k < P.bfl_cap)
                        __stcs(list_entry(b.bfl, k0 + t, n0 + k, P.boundary_count), S.hit[k].x);
                if ((int)lane == t) n_own = n0 + n;
            }
        }
    }
    if (own) b.bfl_count[me] = n_own;
}

__global__ void __launch_bounds__(kBlock) k_boundary_cell_bounds(DevParams P, const float4* __restrict__ b_pos,
                                                                 int* __restrict__ bounds) {
    const uint32_t k = blockIdx.x * kBlock + threadIdx.x;
    if (k >= P.boundary_count) return;
    const float4 xb = b_pos[k];
    const Cell c = cell_of(xb.x, xb.y, xb.z, P);
    const int v[3] = {(int)c.x, (int)c.y, (int)c.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int lo = __reduce_min_sync(__activemask(), v[a]), hi = __reduce_max_sync(__activemask(), v[a]);
        if ((threadIdx.x & 31) == __ffs(__activemask()) - 1) {
            atomicMin(&bounds[a], lo);
            atomicMax(&bounds[3 + a], hi);
        }
    }
}

// Mark every cell within two cells (each axis) of boundary particle k's cell; the box org + [0, dim) holds
// them all (the boundary's cell bounds widened by two).
__global__ void __launch_bounds__(kBlock) k_boundary_zone(DevParams P, const float4* __restrict__ b_pos, int ox,
                                                          int oy, int oz, uint32_t nx, uint32_t ny,
                                                          unsigned char* __restrict__ zone) {
    const uint32_t k = blockIdx.x * kBlock + threadIdx.x;
    if (k >= P.boundary_count) return;
    const float4 xb = b_pos[k];
    const Cell c = cell_of(xb.x, xb.y, xb.z, P);
    const uint32_t x0 = (uint32_t)((int)c.x - ox) - 2u, y0 = (uint32_t)((int)c.y - oy) - 2u,
                   z0 = (uint32_t)((int)c.z - oz) - 2u;
#pragma unroll 1
    for (uint32_t dz = 0; dz < 5; ++dz)
#pragma unroll 1
        for (uint32_t dy = 0; dy < 5; ++dy)
#pragma unroll
            for (uint32_t dx = 0; dx < 5; ++dx)
                zone[((size_t)(z0 + dz) * ny + (y0 + dy)) * nx + (x0 + dx)] = 1;
}

// pcisph.cl:212-263 with boundary_update = 1 from boundary particle k's fluid list: a fluid particle not
// listed was farther than r_list from x_b at the step's start, so it is farther than h from x_b at its
// prediction unless it moved more than half the skin, which flags its bucket (then k walks).
template <bool kCoherent = false>
__device__ __forceinline__ void boundary_pressure_list_body(const DevParams& P, const Control* ctl,
                                                            const ListBuffers& b, uint32_t k) {
    if (k >= P.boundary_count) return;
    const float4 xb = b.b_pos[k];
    float acc = b.b_init[k];
    const uint32_t cnt = b.bfl_count[k];
    bool walk = cnt > P.bfl_cap;
    Cell c{0u, 0u, 0u};
    if (walk || ctl->lists_outrun != 0u) {
        c = cell_of(xb.x, xb.y, xb.z, P);
        walk = walk || near_fast(P, b.bucket_fast, c);
    }
    auto f = [&](uint32_t j) { boundary_density_term(xb, load_slot<kCoherent>(&b.pred[j]), P.h2, acc); };
    if (walk) for_each_neighbour(b.cells, c, P, f);
    else for_each_listed(b.bfl, k, cnt, P.boundary_count, f);
    boundary_pressure_finish(P, xb, acc, b.b_press, const_cast<float4*>(b.bpf), k);
}

__global__ void __launch_bounds__(kBlock) k_boundary_pressure_list(DevParams P, const Control* ctl, ListBuffers b) {
    boundary_pressure_list_body(P, ctl, b, blockIdx.x * kBlock + threadIdx.x);
}

// The skin lists of a step of moving lists (no work in any other step): the pairs of the walk (buckets around x) within
// r_list at y = x + v dt. A kernel of its own: inside the density sweep its registers slowed every step (1M: 495 -> 517
// us), as an early exit it costs 1-2 us. It also puts the round's count of fast predictions past any cap: no marks.
__global__ void __launch_bounds__(kCellBlock, 5) k_moving_lists(DevParams P, Control* ctl, ListBuffers b) {
    if (!lists_move(P, ctl)) return;
    constexpr int W = 8;
    __shared__ CellWarp<W> warps[kCellBlock / 32];
    CellWarp<W>& S = warps[threadIdx.x >> 5];
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->fast_n = kNoMarks;
    const uint32_t lane = threadIdx.x & 31u;
    auto place = [&](uint32_t j) { return moving_place(P, __ldg(&b.pos[j]), f3(__ldg(&b.vel[j]))); };
    for (uint32_t i0 = (blockIdx.x * (kCellBlock / 32) + (threadIdx.x >> 5)) * W; i0 < P.fluid_count;
         i0 += gridDim.x * (kCellBlock / 32) * W) {
        const uint32_t me = i0 + lane;
        const bool own = lane < W && me < P.fluid_count;
        const float4 xi = b.pos[own ? me : i0];
        const Cell c = cell_of(xi.x, xi.y, xi.z, P);
        if (lane < W) {
            S.target[lane] = moving_place(P, xi, f3(b.vel[own ? me : i0]));
            S.target[lane].w = P.list_r2;
        }
        uint32_t n_own = 0;
        uint32_t todo = __ballot_sync(kAll, own);
        while (todo) {
            const int lead = __ffs(todo) - 1;
            const uint32_t cx = __shfl_sync(kAll, c.x, lead), cy = __shfl_sync(kAll, c.y, lead),
                           cz = __shfl_sync(kAll, c.z, lead);
            const uint32_t group = __ballot_sync(kAll, c.x == cx && c.y == cy && c.z == cz) & todo;
            todo &= ~group;
            CellWalk w = begin_cell(b.cells, P, cx, cy, cz, lane, S.delta);
            for (uint32_t base = 0; base < w.total; base += kCellRounds * 32u) {
                Candidates cand;
                load_candidates(cand, w, base, lane, S.delta, place);
                for (uint32_t g = group; g; g &= g - 1u) {
                    const int t = __ffs(g) - 1;
                    const uint32_t n = collect_hits(cand, S.target[t], S.hit, lane);
                    const uint32_t n0 = __shfl_sync(kAll, n_own, t);
                    for (uint32_t k = lane; k < n; k += 32u)
                        if (n0 + k < P.list_cap) __stcs(list_entry(b.nbr, i0 + t, n0 + k, b.nbr_stride), S.hit[k].x);
                    if ((int)lane == t) n_own = n0 + n;
                }
            }
        }
        if (own) b.nbr_count[me] = n_own;
        __syncwarp();
    }
}

// Flags every bucket if the lists of the step are moving lists (see launch_distrust_moving_lists).
__global__ void __launch_bounds__(kBlock) k_distrust_moving_lists(DevParams P, Control* ctl, unsigned char* __restrict__ fast) {
    if (!lists_move(P, ctl)) return;
    const uint32_t k = blockIdx.x * kBlock + threadIdx.x;
    if (k < P.bucket_count) fast[k] = 1;
    if (k == 0) ctl->lists_outrun = 1u;
}

// pcisph.cl:65-92, and the neighbour lists of the step (see the list builders above). kBoundary: the scene has boundary
// particles (their walk is compiled out otherwise). A particle's density terms are staged in walk order and summed by
// one lane in that order: the sum of the walk, whose other terms are zero.
template <class PS, bool kBoundary, int W>
__global__ void __launch_bounds__(kCellBlock, 5) k_density_list(PS ps, ListBuffers b) {
    __shared__ DensityWarp<W> warps[kCellBlock / 32];
    DensityWarp<W>& S = warps[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u, below = lanes_below();
    const uint32_t i0 = (blockIdx.x * (kCellBlock / 32) + (threadIdx.x >> 5)) * W;
    const uint32_t N = ps.count();
    if (i0 >= N) return;
    const uint32_t me = i0 + lane;
    const bool own = lane < W && me < N;
    const DevParams& Pi = ps.params(own ? me : i0);
    const float4 xi = b.pos[own ? me : i0];  // xi.w: the particle's stored half skin
    const Cell c = cell_of(xi.x, xi.y, xi.z, Pi);
    const float sh = half_skin_of(Pi, xi.w);
    if (lane < W) S.target[lane] = make_float4(xi.x, xi.y, xi.z, particle_list_r2(Pi, sh));
    const uint32_t near_addr = (uint32_t)__cvta_generic_to_shared(&S.near[0][0]);
    const uint32_t stride = b.nbr_stride;
    // lane t < W: particle i0 + t's list lengths, the terms staged for it, their sum so far
    uint32_t n_own = 0, near_own = 0, staged = 0;
    float acc = 0.f;
    bool nan_own = false;  // some pair distance is NaN: so is the sum
    // where this lane stores the first of 32 entries of the skin list of particle i0
    uint32_t* const out0 = list_entry(b.nbr, i0, lane, stride);
    const size_t out_step = 32 * (size_t)stride;
    auto flush = [&](int t, uint32_t count) {
        __syncwarp();
        if ((int)lane == t)
            for (uint32_t k = 0; k < count; ++k) acc += __uint_as_float(S.near[t][k].y);
        __syncwarp();
    };
    uint32_t todo = __ballot_sync(kAll, own);
    // moving lists: k_moving_lists builds the skin lists, this pass at x only what lies within h of x
    const bool moving = !PS::kBatched && !kBoundary && lists_move(Pi, ps.control(0));
    if (moving && lane < W) S.target[lane].w = Pi.near_r2;
    while (todo) {
        const int lead = __ffs(todo) - 1;
        const DevParams& P = ps.params(i0 + lead);  // the same scene for the whole group: buckets do not overlap
        const uint32_t cx = __shfl_sync(kAll, c.x, lead), cy = __shfl_sync(kAll, c.y, lead),
                       cz = __shfl_sync(kAll, c.z, lead);
        bool same = c.x == cx && c.y == cy && c.z == cz;
        if (PS::kBatched) same = same && Pi.bucket_base == P.bucket_base;
        const uint32_t group = __ballot_sync(kAll, same) & todo;
        todo &= ~group;
        const float near_r2 = P.near_r2, h2 = P.h2;
        if (kBoundary && P.boundary_count) {
            // boundary particles within r_list, in walk order: the later sweeps read them from the boundary list
            // (all of them, or walk the boundary buckets when there are more than bnd_cap); a cell outside the
            // boundary zone has every boundary particle at least 2h away
            const bool in_zone = !b.b_zone || in_boundary_zone(b, Cell{cx, cy, cz});
            uint32_t nb_own = 0;
            if (in_zone) {
                CellWalk w = begin_cell(b.b_cells, P, cx, cy, cz, lane, S.delta);
                for (uint32_t base = 0; base < w.total; base += kCellRounds * 32u) {
                    Candidates cand;
                    load_candidates(cand, w, base, lane, S.delta, [&](uint32_t j) { return __ldg(&b.b_pos[j]); });
                    for (uint32_t g = group; g; g &= g - 1u) {
                        const int t = __ffs(g) - 1;
                        float4 q = S.target[t];
                        q.w = boundary_list_r2(P, __shfl_sync(kAll, sh, t));
                        if (cand.odd) nan_own |= nan_distance(cand, q, lane) && (int)lane == t;
                        const uint32_t n = collect_hits(cand, q, S.hit, lane);
                        const uint32_t n0 = __shfl_sync(kAll, nb_own, t);
                        uint32_t cnt = __shfl_sync(kAll, staged, t);
                        for (uint32_t k0 = 0; k0 < n; k0 += 32u) {
                            const uint32_t k = k0 + lane;
                            const uint2 e = S.hit[k];
                            const float r2 = __uint_as_float(e.y);
                            if (b.bnbr && k < n && n0 + k < P.bnd_cap)
                                __stcs(list_entry(b.bnbr, i0 + t, n0 + k, stride), e.x);
                            const uint32_t bits = __ballot_sync(kAll, r2 <= h2);
                            if (cnt + __popc(bits) > kNearCap) {
                                flush(t, cnt);
                                cnt = 0;
                            }
                            store_shared_le(r2, h2, near_addr + 8u * (t * (kNearCap + 1u) + cnt + __popc(bits & below)),
                                            e.x, __float_as_uint(poly6(r2, h2)));
                            cnt += __popc(bits);
                        }
                        if ((int)lane == t) {
                            nb_own = n0 + n;
                            staged = cnt;
                        }
                    }
                }
                for (uint32_t g = group; g; g &= g - 1u) {  // the staging area is for the fluid's near list from here
                    const int t = __ffs(g) - 1;
                    flush(t, __shfl_sync(kAll, staged, t));
                    if ((int)lane == t) staged = 0;
                }
            }
            if ((group >> lane) & 1u) {
                b.b_near[me] = nb_own ? 1 : 0;
                if (b.bnbr) b.bnbr_count[me] = nb_own;
            }
        }
        CellWalk w = begin_cell(b.cells, P, cx, cy, cz, lane, S.delta);
        for (uint32_t base = 0; base < w.total; base += kCellRounds * 32u) {
            Candidates cand;
            load_candidates(cand, w, base, lane, S.delta, [&](uint32_t j) { return __ldg(&b.pos[j]); });
            for (uint32_t g = group; g; g &= g - 1u) {
                const int t = __ffs(g) - 1;
                const float4 q = S.target[t];
                if (cand.odd) nan_own |= nan_distance(cand, q, lane) && (int)lane == t;
                const uint32_t n = collect_hits(cand, q, S.hit, lane);
                const uint32_t n0 = __shfl_sync(kAll, n_own, t);
                uint32_t cnt = __shfl_sync(kAll, staged, t);
                if (n0 != 0u && !moving)  // a cell of more than kCellRounds rounds: the list goes on
                    for (uint32_t k = lane; k < n; k += 32u)
                        if (n0 + k < P.list_cap) __stcs(list_entry(b.nbr, i0 + t, n0 + k, stride), S.hit[k].x);
                const uint32_t stored = n0 == 0u && !moving ? min(n, P.list_cap) : 0u;
                uint32_t* out = out0 + 8 * t;
                const uint32_t stage_addr = near_addr + 8u * t * (kNearCap + 1u);
                for (uint32_t k0 = 0; k0 < n; k0 += 32u) {
                    const uint2 e = S.hit[k0 + lane];
                    const float r2 = __uint_as_float(e.y);
                    if (k0 + lane < stored) __stcs(out, e.x);
                    out += out_step;
                    const uint32_t bits = __ballot_sync(kAll, r2 <= near_r2);
                    const uint32_t more = __popc(bits);
                    if (cnt + more > kNearCap) {
                        flush(t, cnt);
                        if ((int)lane == t) near_own += cnt;
                        cnt = 0;
                    }
                    const float dr = fmaxf(h2 - r2, 0.f);  // poly6 of a finite |d|^2
                    store_shared_le(r2, near_r2, stage_addr + 8u * (cnt + __popc(bits & below)), e.x,
                                    __float_as_uint(dr * dr * dr));
                    cnt += more;
                }
                if ((int)lane == t) {
                    n_own = n0 + n;  // > list_cap: this particle walks the buckets in the pressure sweeps
                    staged = cnt;
                }
            }
        }
    }
    near_own += staged;  // > near_cap: this particle walks the buckets in the sweeps at the current positions
    __syncwarp();
    if (own) {
        for (uint32_t k = 0; k < staged; ++k) acc += __uint_as_float(S.near[lane][k].y);
        if (nan_own) acc = __uint_as_float(0x7fffffffu);
        if (!moving) b.nbr_count[me] = n_own;
        b.near_count[me] = near_own;
        acc *= Pi.particle_mass * Pi.poly6_norm;
        b.rho[me] = acc;
        b.pr4[me] = make_float4(xi.x, xi.y, xi.z, acc);
    }
    // the near lists, chunk by chunk: the W particles' chunks are contiguous. A list that outran the staging area
    // (near_cap entries) is not read.
    const uint32_t longest = __reduce_max_sync(kAll, near_own <= kNearCap ? near_own : 0u);
    constexpr int kParts = (8 * W + 31) / 32;
    uint32_t len[kParts];
#pragma unroll
    for (int h = 0; h < kParts; ++h) {
        const uint32_t t = 4u * h + (lane >> 3);
        const uint32_t nn = __shfl_sync(kAll, near_own, t & 31u);
        len[h] = t < W && nn <= kNearCap ? nn : 0u;
    }
    uint32_t* out = b.near + 8 * (size_t)i0 + lane;
    for (uint32_t k = 0; k < longest; k += 8u) {
        const uint32_t e = k + (lane & 7u);
#pragma unroll
        for (int h = 0; h < kParts; ++h)
            if (e < len[h]) __stcs(out + 32 * h, S.near[4 * h + (lane >> 3)][e].x);
        out += 8 * (size_t)stride;
    }
}

// pcisph.cl:94-112
template <class PS, int DEEP = 1>
__global__ void __launch_bounds__(kBlock, DEEP == 1 ? 1 : 2) k_normal_list(PS ps, ListBuffers b) {
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= ps.count()) return;
    const DevParams& P = ps.params(i);
    const float4 xi = b.pr4[i];
    float3 n = make_float3(0.f, 0.f, 0.f);
    const uint32_t cnt = b.near_count[i];
    auto f = [&](uint32_t j) { normal_term(xi.x, xi.y, xi.z, __ldg(&b.pr4[j]), P.h2, n); };
    if (cnt > P.near_cap)
        for_each_neighbour(b.cells, cell_of(xi.x, xi.y, xi.z, P), P, f);
    else if constexpr (DEEP > 1)
        for_each_listed_deep<DEEP>(
            b.near, i, cnt, b.nbr_stride, [&](uint32_t j) { return __ldg(&b.pr4[j]); },
            [&](const float4& o) { normal_term(xi.x, xi.y, xi.z, o, P.h2, n); });
    else
        for_each_listed(b.near, i, cnt, b.nbr_stride, f);
    const float scale = P.h * P.particle_mass * P.poly6_d1_norm;
    b.normal[i] = make_float4(n.x * scale, n.y * scale, n.z * scale, 0.f);
}

// Partner marks of a prediction round (one scene). A pair of the reference's walk whose predictions are within h is in the
// skin list unless one of the two predictions is fast (moved more than half the skin), so the pressure sweep of particle
// i can use its list unless i is fast or some fast j has x*_j within h of x*_i while j is not in i's list. For every fast
// j, particle i is stamped with the round's number when |x_i - x_j| is beyond i's list radius (the builder's test, the
// same bits) and x*_j comes close enough, and j itself is stamped. Stamping more than needed only makes a particle walk,
// which gives the walk's sum. The round is the one the next pressure sweep reads (Control::round + 1); that sweep's last
// block closes it.
//
// Where the next sweep may build tight lists, partners count within h + 2 m. watch: it reads some.
__device__ __forceinline__ float marks_ahead(const DevParams& P, const Control* ctl, const ListBuffers& b, bool watch) {
    return b.tight && tight_plan(ctl->tight_next) != kTightOff && !watch ? 2.f * P.tight_margin : 0.f;
}
// Cell o of the 5 x 5 x 5 cells around x*_j's cell c0, if particles in it can be partners: a particle that is not fast
// lies within D = h + skin_max_half (< 2 cells, checked on the host) of such an x*_j, so its cell is among them, and its
// box comes within D of x*_j (with a margin for the divisions of cell_of). Within 2^14 cells of the origin the rounding of
// the box bounds and of cell_of's division is far below that margin; farther out (or saturated, or NaN) every cell counts.
__device__ __forceinline__ bool partner_cell(const DevParams& P, const float4& pj, const Cell& c0, uint32_t o, float ahead,
                                             Cell& c) {
    c = Cell{c0.x + o % 5u - 2u, c0.y + o / 5u % 5u - 2u, c0.z + o / 25u - 2u};
    auto inner = [](uint32_t v) { return v + 16384u < 32768u; };  // -2^14 < (int)v < 2^14, wrapping
    if (!(inner(c0.x) && inner(c0.y) && inner(c0.z))) return true;
    auto gap = [&](uint32_t v, float x) {  // distance from x to the cell along an axis
        const float lo = (float)(int)v * P.cell_size, hi = lo + P.cell_size;
        return fmaxf(fmaxf(lo - x, x - hi), 0.f);
    };
    const float gx = gap(c.x, pj.x), gy = gap(c.y, pj.y), gz = gap(c.z, pj.z);
    const float reach = P.h + P.skin_max_half + ahead + 0.01f * P.cell_size;
    return !(gx * gx + gy * gy + gz * gz > reach * reach);
}
__device__ __forceinline__ bool beyond_list(const DevParams& P, const float4& xi, const float4& xj) {
    return !(dist2(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z) <= particle_list_r2(P, half_skin_of(P, xi.w)));
}

// After a prediction round: a thread per (fast prediction that the round listed, cell). Close enough: |x*_i - x*_j| <= h
// (the pressure sweep's |d|^2, with d negated: the same bits). A round with more than mark_cap fast predictions stamps
// nothing (the sweep then uses the bucket flags), nor does a step of moving lists. Grid-stride over the items, 4 blocks an
// SM: a round of ~3,000 fast predictions at 1M takes 13 us (21 with one block an SM; 14 with a warp per prediction), a
// round without any 2.5.
constexpr unsigned kMarkBlocks = 4u * kSms;
__global__ void __launch_bounds__(kBlock) k_mark_partners(DevParams P, const Control* ctl, ListBuffers b) {
    const unsigned long long n = ctl->fast_n;
    if (n == 0 || n > P.mark_cap) return;
    const bool watch = b.tight && tight_plan(ctl->tight_next) == kTightUse && ctl->tight_stray == 0u;  // the next sweep reads tight lists
    if (watch && ctl->tight_outrun == 0u) return;  // and asks no marks
    const float ahead = marks_ahead(P, ctl, b, watch), far2 = ahead > 0.f ? P.tight_r2 : P.h2;
    const float threshold = built_threshold(P, ctl);
    const unsigned round = ctl->round + 1u;
    const unsigned long long items = n * 125ull;
    for (unsigned long long t = (unsigned long long)blockIdx.x * kBlock + threadIdx.x; t < items;
         t += (unsigned long long)gridDim.x * kBlock) {
        const uint32_t j = b.fast_list[t / 125ull];
        const uint32_t o = (uint32_t)(t % 125ull);
        const float4 pj = b.pred[j];
        const float4 xj = b.pos[j];
        float disp;
        if (watch && outruns<false>(P, ctl, xj, b.tight_ref[j], threshold, make_float3(0.f, 0.f, 0.f), disp)) continue;
        if (o == 62u) b.walk_stamp[j] = round;  // the centre cell's thread: j itself walks
        Cell c;
        if (!partner_cell(P, pj, cell_of(pj.x, pj.y, pj.z, P), o, ahead, c)) continue;
        const uint2 r = b.cells[P.bucket_base + hash_key(c.x, c.y, c.z, P)];
#pragma unroll 1
        for (uint32_t i0 = r.x; i0 < r.y; i0 += 4) {
            float4 pi[4], xi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u < r.y) {
                    pi[u] = b.pred[i0 + u];
                    xi[u] = b.pos[i0 + u];
                }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u < r.y && dist2(pj.x - pi[u].x, pj.y - pi[u].y, pj.z - pi[u].z) <= far2 &&
                    beyond_list(P, xi[u], xj))
                    b.walk_stamp[i0 + u] = round;
        }
    }
}

// The same by the warp that predicts, for the fast predictions set of its lanes' particles i (the whole warp calls). Close
// enough: |x_i - x*_j| <= D, which needs no other prediction of the round. It saves the launch after each round (4,096
// particles, 7 rounds: 182 -> 166 us a step). Larger scenes lose: the fast predictions of a warp follow one another (120K
// particles, up to 1 in 8 fast: pressure force 26 -> 108 us against 26 + 15 with the kernel).
__device__ __noinline__ void mark_partners_inline(const DevParams& P, Control* ctl, const ListBuffers& b, uint32_t i,
                                                  unsigned set, uint32_t* delta) {
    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long base = ~0ull;
    if (lane == 0 && *(volatile unsigned long long*)&ctl->fast_n <= P.mark_cap)
        base = atomicAdd(&ctl->fast_n, (unsigned long long)__popc(set));
    base = __shfl_sync(kAll, base, 0);
    if (base >= P.mark_cap) return;  // past the cap: the sweep takes the bucket flags
    __syncwarp();                    // the lanes' predictions are stored
    const unsigned round = ctl->round + 1u;
    const float ahead = marks_ahead(P, ctl, b, tight_plan(ctl->tight_next) == kTightUse);  // (else the sweep takes no marks)
    const float far = P.h + P.skin_max_half + ahead + 1e-4f * P.h;  // D, past the rounding of the distances
    for (; set; set &= set - 1u) {
        const uint32_t j = __shfl_sync(kAll, i, __ffs(set) - 1);
        const float4 pj = b.pred[j], xj = b.pos[j];
        const Cell c0 = cell_of(pj.x, pj.y, pj.z, P);
        if (lane == 0) b.walk_stamp[j] = round;
        uint2 r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t o = lane + 32u * q;
            Cell c;
            r[q] = make_uint2(0u, 0u);
            if (o < 125u && partner_cell(P, pj, c0, o, ahead, c)) r[q] = b.cells[P.bucket_base + hash_key(c.x, c.y, c.z, P)];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            CellWalk w = concatenate(r[q], lane, delta);
            for (uint32_t at = 0; at < w.total; at += 32u) {
                const uint32_t k = next_candidate(w, at, lane, delta);
                if (k == kAll) continue;
                const float4 x = b.pos[k];
                if (dist2(pj.x - x.x, pj.y - x.y, pj.z - x.z) <= far * far && beyond_list(P, x, xj))
                    b.walk_stamp[k] = round;
            }
        }
    }
}
template <class PS>
__device__ __forceinline__ void close_round(const PS& ps, const ListBuffers& b, uint32_t i, bool fast, uint32_t* delta) {
    if (PS::kBatched || !b.walk_stamp) return;
    const unsigned set = __ballot_sync(kAll, fast);
    if (set) mark_partners_inline(ps.params(0), ps.control(0), b, i, set, delta);
}

// The force sweep's epilogue from its three sums, and the first predict (pcisph.cl:175-193, F_p = 0); returns whether the
// prediction is fast.
template <class PS>
__device__ __forceinline__ bool finish_force(const PS& ps, const ListBuffers& b, const DevParams& P, uint32_t i,
                                             const float4& xi, const float3& vi, const float3& visc, const float3& coh,
                                             const float3& curv) {
    const float m = P.particle_mass;
    const float3 fo = other_force(m, P.gravity, visc, P.viscosity * m * P.visc_d2_norm, coh,
                                  -P.st_coeff * m * m * P.st_norm, curv, -P.st_coeff * m);
    b.f_other[i] = f4(fo, 0.f);
    b.press[i] = 0.f;
    const float3 v = vi + (fo / m) * P.dt;
    const float3 dx = v * P.dt;
    const float4 xs = make_float4(xi.x + dx.x, xi.y + dx.y, xi.z + dx.z, 0.f);
    b.pred[i] = xs;
    bool fast;
    const float disp = note_displacement<!PS::kBatched>(P, ps.control(i), b.bucket_fast, xi, xs, P.list_half_skin, vi, nullptr,
                                                        fast, PS::kBatched ? nullptr : b.fast_list, i);
    if (P.particle_skin) b.disp_max[i] = disp;
    return fast;
}

// pcisph.cl:121-173, then the first predict
template <class PS>
__global__ void __launch_bounds__(kBlock) k_force_list(PS ps, ListBuffers b) {
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= ps.count()) return;
    const DevParams& P = ps.params(i);
    const float4 xi = b.pr4[i];
    const float3 vi = f3(b.vel[i]);
    const float3 ni = f3(b.normal[i]);
    ForceAccum fa{make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
    const uint32_t cnt = b.near_count[i];
    auto f = [&](uint32_t j) {
        force_term(xi, vi, ni, __ldg(&b.pr4[j]), f3(__ldg(&b.vel[j])), f3(__ldg(&b.normal[j])), P, fa);
    };
    if (cnt <= P.near_cap) for_each_listed(b.near, i, cnt, b.nbr_stride, f);
    else for_each_neighbour(b.cells, cell_of(xi.x, xi.y, xi.z, P), P, f);
    finish_force(ps, b, P, i, xi, vi, fa.visc, fa.coh, fa.curv);
}

// The same two sweeps with eight lanes per particle (small scenes).
template <class PS, int L>
__global__ void __launch_bounds__(kBlock) k_normal_shared(PS ps, ListBuffers b) {
    const uint32_t t = blockIdx.x * kBlock + threadIdx.x, i0 = t / L, q = t % L;
    __shared__ TermStage<L> stage[kBlock / L];
    TermStage<L>& S = stage[threadIdx.x / L];
    const bool live = i0 < ps.count();
    const uint32_t i = live ? i0 : ps.count() - 1u;
    const DevParams& P = ps.params(i);
    const uint32_t mask = lanes_mask<L>();
    const float4 xi = b.pr4[i];
    const uint32_t cnt = b.near_count[i];
    const bool listed = cnt <= P.near_cap;
    const uint32_t n = listed ? cnt : 0u;
    float acc = 0.f;  // lane 0, 1, 2: x, y, z
    auto sum = [&](const float4& o, bool valid, uint32_t m) {
        PairTerm term{0.f, 0.f, 0.f, 0.f};
        if (valid) normal_pair(xi.x, xi.y, xi.z, o, P.h2, [&](const PairTerm& p) { term = p; });
        add_lanes(acc, term, S, q, m);
    };
    for_each_shared<L, 32 / L>(
        b.near, i, n, __reduce_max_sync(kAll, n), b.nbr_stride, q, [&](uint32_t j) { return __ldg(&b.pr4[j]); },
        [&](const float4& o, uint32_t, bool valid) { sum(o, valid, kAll); });
    if (!listed)
        walk_shared<L>(b.cells, cell_of(xi.x, xi.y, xi.z, P), P, q, [&](uint32_t j, bool valid) {
            float4 o = xi;
            if (valid) o = __ldg(&b.pr4[j]);
            sum(o, valid, mask);
        });
    acc *= P.h * P.particle_mass * P.poly6_d1_norm;
    const float y = __shfl_sync(mask, acc, 1, L), z = __shfl_sync(mask, acc, 2, L);
    if (live && q == 0) b.normal[i] = make_float4(acc, y, z, 0.f);
}

template <class PS, int L>
__global__ void __launch_bounds__(kBlock) k_force_shared(PS ps, ListBuffers b) {
    const uint32_t t = blockIdx.x * kBlock + threadIdx.x, i0 = t / L, q = t % L;
    __shared__ TermStage<L> stage[kBlock / L];
    TermStage<L>& S = stage[threadIdx.x / L];
    const bool live = i0 < ps.count();
    const uint32_t i = live ? i0 : ps.count() - 1u;
    const DevParams& P = ps.params(i);
    const uint32_t mask = lanes_mask<L>();
    const float4 xi = b.pr4[i];
    const float3 vi = f3(b.vel[i]), ni = f3(b.normal[i]);
    const uint32_t cnt = b.near_count[i];
    const bool listed = cnt <= P.near_cap;
    const uint32_t n = listed ? cnt : 0u;
    float visc = 0.f, coh = 0.f, curv = 0.f;  // lane 0, 1, 2: x, y, z
    struct ForceOperand {
        float4 x, v, n;
    };
    auto load = [&](uint32_t j) { return ForceOperand{__ldg(&b.pr4[j]), __ldg(&b.vel[j]), __ldg(&b.normal[j])}; };
    auto sum = [&](const ForceOperand& o, bool valid, uint32_t m) {
        const PairTerm none{0.f, 0.f, 0.f, 0.f};
        PairTerm a = none, c = none, d = none;
        if (valid)
            force_pair(
                xi, vi, ni, o.x, f3(o.v), f3(o.n), P, [&](const PairTerm& p) { a = p; },
                [&](const PairTerm& p, const PairTerm& r) {
                    c = p;
                    d = r;
                });
        add_lanes(visc, a, S, q, m);
        add_lanes(coh, c, S, q, m);
        add_lanes(curv, d, S, q, m);
    };
    for_each_shared<L, 16 / L>(b.near, i, n, __reduce_max_sync(kAll, n), b.nbr_stride, q, load,
                       [&](const ForceOperand& o, uint32_t, bool valid) { sum(o, valid, kAll); });
    if (!listed)
        walk_shared<L>(b.cells, cell_of(xi.x, xi.y, xi.z, P), P, q, [&](uint32_t j, bool valid) {
            ForceOperand o{xi, xi, xi};
            if (valid) o = load(j);
            sum(o, valid, mask);
        });
    auto all = [&](float v) {
        return make_float3(__shfl_sync(mask, v, 0, L), __shfl_sync(mask, v, 1, L), __shfl_sync(mask, v, 2, L));
    };
    const float3 sv = all(visc), sc = all(coh), su = all(curv);
    bool fast = false;
    if (live && q == 0) fast = finish_force(ps, b, P, i, xi, vi, sv, sc, su);
    __shared__ uint32_t delta[kBlock];
    close_round(ps, b, i, fast, delta + (threadIdx.x & ~31u));
}

// pcisph.cl:212-263 (boundary_update = 0); one scene: also the stop decision in the last block

// How one particle's pressure sweep finds its neighbours.
struct PressurePlan {
    uint32_t cnt, bcnt;              // entries of its skin list and of its boundary list
    bool walk;                       // the fluid buckets instead of the skin list
    bool walk_boundary, list_boundary;
    Cell c;                          // set where it walks
};
template <class PS>
__device__ __forceinline__ PressurePlan plan_pressure(const PS& ps, const ListBuffers& b, const DevParams& P,
                                                      const Control* ctl, uint32_t i, const float4& xi,
                                                      const float4& xp, const ListState& state) {
    PressurePlan p;
    const unsigned mode = state.mode;
    const bool all_lists_ok = !state.outrun;
    const uint32_t listed = mode == kTightUse ? b.tight_count[i] : b.nbr_count[i];
    const bool complete = mode == kTightUse && (listed & kTightWalked) != 0u;  // its tight list was built by a walk
    p.cnt = mode == kTightUse ? listed & ~kTightWalked : listed;
    const bool overflow = p.cnt > (mode == kTightUse ? kTightCap : P.list_cap);
    // self_fast: x* moved more than the particle's own half skin from x, so its lists (built for that
    // skin) may miss a pair: with per-particle skins it walks. Boundary terms: all zero unless a boundary
    // particle was within r_list of x, or x* moved past the half skin (boundary particles do not move);
    // within it, the boundary list (every boundary particle within r_list of x) holds every one that can
    // be within h of x*.
    bool self_fast = false;
    if (P.particle_skin || P.boundary_count) {
        const float dx = xp.x - xi.x, dy = xp.y - xi.y, dz = xp.z - xi.z;
        self_fast = sqrtf(dist2(dx, dy, dz)) > fast_threshold(P, half_skin_of(P, xi.w));
    }
    p.walk_boundary = p.list_boundary = false;
    p.bcnt = 0;
    if (P.boundary_count) {
        if (self_fast) {
            p.walk_boundary = true;
        } else if (b.b_near[i] != 0) {
            if (b.bnbr) p.bcnt = b.bnbr_count[i];
            p.list_boundary = b.bnbr && p.bcnt <= P.bnd_cap;
            p.walk_boundary = !p.list_boundary;
        }
    }
    p.c = Cell{0u, 0u, 0u};  // the cell (three IEEE divisions) only where a walk may need it
    const bool own_walk = overflow || (P.particle_skin && self_fast) || (mode == kTightBuild && tight_by_walks(P));
    if (complete || (mode == kTightUse && all_lists_ok && !own_walk)) {
        p.walk = overflow;
    } else {
        // partner marks of this round (one scene, after the marking kernel): the particles that may miss a
        // pair of their walk are stamped with the round's number; a round past the cap (or no marks) takes
        // the bucket flags: every particle near a fast one walks (marks by a predicting sweep that expected
        // tight lists to be read lack the predictions that were fast at their building)
        const unsigned long long fast_round = !PS::kBatched && b.walk_stamp ? ctl->fast_n : ~0ull;
        if (fast_round <= P.mark_cap && (mode == kTightUse || b.fast_list || !b.tight || tight_plan(ctl->tight_next) != kTightUse)) {
            p.walk = own_walk || (fast_round != 0 && b.walk_stamp[i] == ctl->round + 1u);
        } else {
            if (!all_lists_ok) p.c = cell_of(xi.x, xi.y, xi.z, P);
            p.walk = own_walk || (!all_lists_ok && near_fast(P, b.bucket_fast, p.c));
        }
    }
    if (p.walk || p.walk_boundary) p.c = cell_of(xi.x, xi.y, xi.z, P);
    return p;
}

// From a particle's density sum: its density variation (returned), pressure and packed operand.
template <class PS>
__device__ __forceinline__ float finish_pressure(const ListBuffers& b, const DevParams& P, Control* ctl, uint32_t i,
                                                 const float4& xi, float acc) {
    acc *= P.particle_mass * P.poly6_norm;
    if (!isfinite(acc)) atomicOr(&ctl->status, 2u);
    float dv = acc - P.rest_density;
    dv = 0.f < dv ? dv : 0.f;
    b.err[i] = dv;
    float p = b.press[i];
    if (dv != 0.f) {
        p += dv * P.delta;
        b.press[i] = p;
    }
    const float r = b.rho[i];
    b.pf4[i] = make_float4(xi.x, xi.y, xi.z, p / (r * r));
    if (PS::kBatched) warp_atomic_max(&ctl->max_err_bits, __float_as_uint(dv));
    return dv;
}

// The few particles of a warp that walk, after their boundary terms (acc). A walk by one lane takes the warp ~400 steps of one
// gather each, whatever its other lanes do; up to kFewWalkers are therefore served one after another by all 32 lanes (27
// bucket ranges at once, 32 candidates a round, ~9 rounds), and their terms summed in walk order by their own lane. Each costs
// ~500 instructions, a lane's share of a full warp's walk ~300: with more, each lane walks by itself (pressure_body).
// Pressure sweep with few hundred to few thousand fast predictions: 1M jittered block 158 -> 146 us, a 98,904-particle drop
// at 2.4 m/s 43 -> 31; from 6 to 32 the split makes no difference there.
constexpr int kFewWalkers = 12;
struct WalkStage {
    uint32_t delta[32];
    float term[96];
};
// With room to stage the tight lists of a warp's lanes (before its walkers are served, or by them).
union BuildStage {
    WalkStage walk;
    uint32_t tight[16 * 32];
};
template <bool kShared>
using Stage = std::conditional_t<kShared, BuildStage, WalkStage>;
__device__ __forceinline__ uint32_t* stage_tight(WalkStage&) { return nullptr; }
__device__ __forceinline__ uint32_t* stage_tight(BuildStage& s) { return s.tight; }
__device__ __forceinline__ WalkStage& stage_walk(WalkStage& s) { return s; }
__device__ __forceinline__ WalkStage& stage_walk(BuildStage& s) { return s.walk; }
template <class PS, bool kCoherent, bool kShared>
__device__ __forceinline__ float pressure_walkers(const PS& ps, const ListBuffers& b, uint32_t i, float acc,
                                               uint32_t walkers, bool build, Stage<kShared>& stage) {
    constexpr int U = 2;  // rounds with their gathers in flight
    WalkStage& S = stage_walk(stage);
    const uint32_t lane = threadIdx.x & 31u;
    const bool mine = (walkers >> lane) & 1u;
    const uint32_t first = __shfl_sync(kAll, i, __ffs(walkers) - 1);
    const uint32_t ii = mine ? i : first;  // a lane that does not walk stands in for the first that does
    const DevParams& P = ps.params(ii);
    const float4 xi = b.pos[ii];
    const float4 xp = b.pred[ii];
    const Cell c = cell_of(xi.x, xi.y, xi.z, P);
    const uint32_t below = lanes_below();
    for (uint32_t todo = walkers; todo; todo &= todo - 1u) {
        const int t = __ffs(todo) - 1;
        const DevParams& Q = ps.params(__shfl_sync(kAll, ii, t));
        const float x = __shfl_sync(kAll, xp.x, t), y = __shfl_sync(kAll, xp.y, t), z = __shfl_sync(kAll, xp.z, t);
        CellWalk w = begin_cell(b.cells, Q, __shfl_sync(kAll, c.x, t), __shfl_sync(kAll, c.y, t),
                                __shfl_sync(kAll, c.z, t), lane, S.delta);
        const uint32_t it = __shfl_sync(kAll, ii, t);
        const bool keep = __shfl_sync(kAll, (int)build, t) != 0;
        uint32_t n = 0, kept = 0;
        auto sum = [&] {  // the staged terms, by the walker's own lane
            __syncwarp();
            if ((int)lane == t)
                for (uint32_t k = 0; k < n; ++k) acc += S.term[k];
            n = 0;
            __syncwarp();
        };
        for (uint32_t base = 0; base < w.total; base += 32u * U) {
            float4 o[U];
            uint32_t js[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                js[u] = next_candidate(w, base + u * 32u, lane, S.delta);
                if (js[u] != kAll) o[u] = load_slot<kCoherent>(&b.pred[js[u]]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float term = 0.f;
                bool tight = false;
                if (base + u * 32u + lane < w.total) {
                    const float d2 = dist2(x - o[u].x, y - o[u].y, z - o[u].z);
                    term = poly6(d2, Q.h2);
                    tight = keep && !(d2 > Q.tight_r2);
                }
                const uint32_t set = __ballot_sync(kAll, tight);
                if (tight) {
                    const uint32_t e = kept + __popc(set & below);
                    if (e < kTightCap) reinterpret_cast<uint32_t*>(list_chunk(b.tight, it, e >> 3, b.nbr_stride))[e & 7u] = js[u];
                }
                kept += __popc(set);
                const uint32_t bits = __ballot_sync(kAll, term != 0.f);  // NaN counts
                if (n + __popc(bits) > 96u) sum();
                if (term != 0.f) S.term[n + __popc(bits & below)] = term;
                n += __popc(bits);
            }
        }
        sum();
        if (keep && (int)lane == t) b.tight_count[it] = kept | kTightWalked;
    }
    return mine ? finish_pressure<PS>(b, P, ps.control(ii), ii, xi, acc) : 0.f;
}

// A particle's fluid terms added to acc by its own lane, from its skin list (cnt entries) or a walk, building its tight
// list. (A chunk's distances before its entries are kept: 218 -> 186 us at 1M, the gathers in flight together.)
template <bool kCoherent, bool kShared>
__device__ __forceinline__ float build_tight_list(const ListBuffers& b, const DevParams& P, uint32_t i, const float4& xi,
                                                  const float4& xp, uint32_t cnt, float acc, bool walk, uint32_t* stage) {
    TightWriter<kShared> w(b.tight, i, b.nbr_stride, stage);
    uint32_t written = 0;  // entries at the last look
    auto away2 = [&](uint32_t j) {
        const float4 o = load_slot<kCoherent>(&b.pred[j]);
        return dist2(xp.x - o.x, xp.y - o.y, xp.z - o.z);
    };
    auto keep = [&](uint32_t j, float d2) {
        acc += poly6(d2, P.h2);
        if (!(d2 > P.tight_r2)) w.add(j);
    };
    auto flush = [&] {
        if ((written ^ w.n) & 8u) w.flush(written >> 3);
        written = w.n;
    };
    if (walk)
        for_each_neighbour(b.cells, cell_of(xi.x, xi.y, xi.z, P), P, [&](uint32_t j) {
            keep(j, away2(j));
            flush();
        });
    else for_each_listed_ahead(b.nbr, i, cnt, b.nbr_stride, away2, keep, flush);
    w.finish();
    b.tight_count[i] = w.n | (walk ? kTightWalked : 0u);
    return acc;
}
// One particle's pressure sweep; returns its density variation (0 when skipped or out of range). The whole warp calls;
// stage: its WalkStage. The decisions are plan_pressure's (a struct returned to this form slowed it: 286,720 particles with
// boundary 42.5 -> 48.7 us), and kTightSkin's for a batch.
//
// Where more than kFewWalkers lanes of a warp walk, each does so by itself, here and not in pressure_walkers: with that walk
// there, as a function whose parameters lie in memory or inlined at 48 registers, a sweep in which most particles walk took
// 1.2 to 2.2 times as long. us a step with most predictions fast, without walks by warps / so / now: 110,592 particles 677 /
// 811 / 636, 1,000,000 3620 / 5270 / 3990, 16 batched scenes of 65,000 9690 / 12780 / 10670.
//
// kFew: few walkers of a warp go to pressure_walkers (or each walks by itself, too). kTight: the launch may have tight lists.
template <class PS, bool kCoherent, bool kFew, bool kShared, bool kTight = true>
__device__ __forceinline__ float pressure_body(const PS& ps, const ListBuffers& b, uint32_t i, Stage<kShared>& stage) {
    float dv = 0.f, acc = 0.f;
    bool walk = false, build = false, tight = false;
    uint32_t cnt = 0;
    float4 xi{}, xp{};
    const bool live = i < ps.count() && !ps.skip_pressure(i);
    const DevParams& P = ps.params(live ? i : 0u);
    Control* ctl = ps.control(live ? i : 0u);
    if (live) {
        xi = b.pos[i];
        xp = b.pred[i];
        const ListState state = list_state<kTight>(P, ctl, b.tight != nullptr);
        const unsigned mode = state.mode;
        const bool all_lists_ok = !state.outrun;
        build = mode == kTightBuild;
        tight = mode == kTightUse;
        cnt = tight ? b.tight_count[i] : b.nbr_count[i];
        const bool complete = tight && (cnt & kTightWalked) != 0u;  // its tight list was built by a walk
        if (tight) cnt &= ~kTightWalked;
        if (PS::kBatched && tight && cnt == kTightSkin) {
            cnt = b.nbr_count[i];
            tight = false;
        }
        const bool overflow = cnt > (tight ? kTightCap : P.list_cap);
        // self_fast: x* moved more than the particle's own half skin from x, so its lists (built for that
        // skin) may miss a pair: with per-particle skins it walks. Boundary terms: all zero unless a boundary
        // particle was within r_list of x, or x* moved past the half skin (boundary particles do not move);
        // within it, the boundary list (every boundary particle within r_list of x) holds every one that can
        // be within h of x*.
        bool self_fast = false;
        if (P.particle_skin || P.boundary_count) {
            const float dx = xp.x - xi.x, dy = xp.y - xi.y, dz = xp.z - xi.z;
            self_fast = sqrtf(dist2(dx, dy, dz)) > fast_threshold(P, half_skin_of(P, xi.w));
        }
        bool walk_boundary = false, list_boundary = false;
        uint32_t bcnt = 0;
        if (P.boundary_count) {
            if (self_fast) {
                walk_boundary = true;
            } else if (b.b_near[i] != 0) {
                if (b.bnbr) bcnt = b.bnbr_count[i];
                list_boundary = b.bnbr && bcnt <= P.bnd_cap;
                walk_boundary = !list_boundary;
            }
        }
        Cell c{0u, 0u, 0u};  // the cell (three IEEE divisions) only where a walk may need it
        const bool own_walk = overflow || (P.particle_skin && self_fast) || (build && tight_by_walks(P));
        if (complete || (tight && all_lists_ok && !own_walk)) {
            walk = overflow;
        } else {  // by marks or flags (see plan_pressure)
            const unsigned long long fast_round = !PS::kBatched && b.walk_stamp ? ctl->fast_n : ~0ull;
            if (fast_round <= P.mark_cap) {
                walk = own_walk || (fast_round != 0 && b.walk_stamp[i] == ctl->round + 1u);
            } else {
                if (!all_lists_ok) c = cell_of(xi.x, xi.y, xi.z, P);
                walk = own_walk || (!all_lists_ok && near_fast(P, b.bucket_fast, c));
            }
        }
        if (walk_boundary) c = cell_of(xi.x, xi.y, xi.z, P);
        auto fb = [&](uint32_t j) { acc += density_term(xp.x, xp.y, xp.z, __ldg(&b.b_pos[j]), P.h2); };
        if (walk_boundary) for_each_neighbour(b.b_cells, c, P, fb);
        else if (list_boundary) for_each_listed(b.bnbr, i, bcnt, b.nbr_stride, fb);
        if (build) {
            b.tight_ref[i] = xp;
            if (PS::kBatched && cnt > b.tight_below) {
                b.tight_count[i] = walk ? kTightCap + 1u : kTightSkin;
                build = false;
            }
        }
    }
    const auto load = [&](uint32_t j) { return load_slot<kCoherent>(&b.pred[j]); };
    const auto by_lane = [&] {  // this lane's walk
        if (build) {
            acc = build_tight_list<kCoherent, kShared>(b, P, i, xi, xp, cnt, acc, true, stage_tight(stage));
        } else {
            const Cell c = cell_of(xi.x, xi.y, xi.z, P);
            auto use = [&](uint32_t, const float4& o) { acc += density_term(xp.x, xp.y, xp.z, o, P.h2); };
            // a batch walks with two gathers in flight (terms still added in walk order): its walkers are latency-bound
            // (256 batched scenes, 9.8M particles, over 500 steps: 26.8 -> 25.8 s); one scene walks plainly (8M
            // particles all walking: 3.0 ms per sweep, 3.6 with the prefetch)
            if constexpr (PS::kBatched) for_each_neighbour_prefetched(b.cells, c, P, load, use);
            else for_each_neighbour(b.cells, c, P, [&](uint32_t j) { use(j, load(j)); });
        }
        dv = finish_pressure<PS>(b, P, ctl, i, xi, acc);
    };
    if (live && !walk) {
        if (build) acc = build_tight_list<kCoherent, kShared>(b, P, i, xi, xp, cnt, acc, false, stage_tight(stage));
        else
            for_each_listed(tight ? b.tight : b.nbr, i, cnt, b.nbr_stride,
                            [&](uint32_t j) { acc += density_term(xp.x, xp.y, xp.z, load(j), P.h2); });
        dv = finish_pressure<PS>(b, P, ctl, i, xi, acc);
    } else if (!kFew && walk) {
        by_lane();
    }
    if constexpr (kFew) {
        const uint32_t walkers = __ballot_sync(kAll, walk);
        if (__popc(walkers) > kFewWalkers) {
            if (walk) by_lane();
        } else if (walkers) {
            __syncwarp();  // the stage changes hands
            const float w = pressure_walkers<PS, kCoherent, kShared>(ps, b, i, acc, walkers, build, stage);
            if (walk) dv = w;
        }
    }
    return dv;
}

// The same with eight lanes per particle, lane q; returned to each of them.
template <class PS, int L>
__device__ __forceinline__ float pressure_shared(const PS& ps, const ListBuffers& b, uint32_t i0, uint32_t q) {
    const bool live = i0 < ps.count() && !ps.skip_pressure(i0);
    const uint32_t i = i0 < ps.count() ? i0 : ps.count() - 1u;
    const uint32_t mask = lanes_mask<L>();
    const DevParams& P = ps.params(i);
    Control* ctl = ps.control(i);
    const float4 xi = b.pos[i];
    const float4 xp = b.pred[i];
    PressurePlan p{};
    const ListState state = list_state<true>(P, ctl, b.tight != nullptr);
    const unsigned mode = state.mode;
    if (live) p = plan_pressure(ps, b, P, ctl, i, xi, xp, state);
    float acc = 0.f;
    auto sum = [&](const float4& o, bool valid, uint32_t m) {
        add_lanes<L>(acc, valid ? density_term(xp.x, xp.y, xp.z, o, P.h2) : 0.f, m);
    };
    auto walk = [&](const uint2* cells, const float4* src) {
        walk_shared<L>(cells, p.c, P, q, [&](uint32_t j, bool valid) {
            float4 o = xp;
            if (valid) o = __ldg(&src[j]);
            sum(o, valid, mask);
        });
    };
    if (P.boundary_count) {
        const uint32_t n = p.list_boundary ? p.bcnt : 0u;
        for_each_shared<L, 32 / L>(
            b.bnbr, i, n, __reduce_max_sync(kAll, n), b.nbr_stride, q, [&](uint32_t j) { return __ldg(&b.b_pos[j]); },
            [&](const float4& o, uint32_t, bool valid) { sum(o, valid, kAll); });
        if (p.walk_boundary) walk(b.b_cells, b.b_pos);
    }
    const uint32_t n = live && !p.walk ? p.cnt : 0u;
    const uint32_t most = __reduce_max_sync(kAll, n);
    auto load = [&](uint32_t j) { return __ldg(&b.pred[j]); };
    if (mode == kTightBuild) {
        uint32_t kept = 0;
        auto keep = [&](const float4& o, uint32_t j, bool valid, uint32_t m) {
            const float d2 = dist2(xp.x - o.x, xp.y - o.y, xp.z - o.z);
            add_lanes<L>(acc, valid ? poly6(d2, P.h2) : 0.f, m);
            const bool in = valid && !(d2 > P.tight_r2);
            const uint32_t set = __ballot_sync(m, in) & mask, e = kept + __popc(set & lanes_below());
            if (in && e < kTightCap) reinterpret_cast<uint32_t*>(list_chunk(b.tight, i, e >> 3, b.nbr_stride))[e & 7u] = j;
            kept += __popc(set);
        };
        for_each_shared<L, 32 / L>(b.nbr, i, n, most, b.nbr_stride, q, load,
                                   [&](const float4& o, uint32_t j, bool valid) { keep(o, j, valid, kAll); });
        if (p.walk)
            walk_shared<L>(b.cells, p.c, P, q, [&](uint32_t j, bool valid) {
                float4 o = xp;
                if (valid) o = load(j);
                keep(o, j, valid, mask);
            });
        if (live && q == 0) {
            b.tight_count[i] = kept | (p.walk ? kTightWalked : 0u);
            b.tight_ref[i] = xp;
        }
    } else {
        for_each_shared<L, 32 / L>(mode == kTightUse ? b.tight : b.nbr, i, n, most, b.nbr_stride, q, load,
                                   [&](const float4& o, uint32_t, bool valid) { sum(o, valid, kAll); });
        if (p.walk) walk(b.cells, b.pred);
    }
    float dv = 0.f;
    if (live && q == 0) dv = finish_pressure<PS>(b, P, ctl, i, xi, acc);
    return dv;
}

// BS: threads per block (128, 256 or 512; the autotuner's choice for one scene)
// kThreads: resident threads per SM, 1024 at 64 registers or 1280 at 48 (see launch_pressure_list)
template <class PS, int BS = kBlock, int LANES = 1, bool kFew = true, bool kShared = false, int kThreads = 1024>
__global__ void __launch_bounds__(BS, LANES > 1 ? 1 : kThreads / BS) k_pressure_list(PS ps, ListBuffers b) {
    const uint32_t t = blockIdx.x * BS + threadIdx.x;
    float dv;
    __shared__ Stage<kShared> stage[LANES == 1 ? BS / 32 : 1];
    if constexpr (LANES == 1) dv = pressure_body<PS, false, kFew, kShared>(ps, b, t, stage[threadIdx.x >> 5]);
    else dv = pressure_shared<PS, LANES>(ps, b, t / LANES, t % LANES);
    if (PS::kBatched) return;
    // one scene: block max of dv, the last block decides (dv >= 0: bit patterns order like values)
    const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(dv));
    __shared__ unsigned warp_max[BS / 32];
    __shared__ bool is_last;
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = bits;
    __syncthreads();
    Control* ctl = ps.control(0);
    if (threadIdx.x == 0) {
        unsigned m = 0;
#pragma unroll
        for (int w = 0; w < BS / 32; ++w) m = max(m, warp_max[w]);
        atomicMax(&ctl->max_err_bits, m);
        __threadfence();
        is_last = atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (is_last && threadIdx.x == 0) {
        __threadfence();
        const DevParams& P = ps.params(0);
        const bool marks = b.walk_stamp && ctl->fast_n <= P.mark_cap, moves = lists_move(P, ctl);
        const unsigned round = ctl->round;
        const unsigned next = tight_advance(P, ctl, b.tight != nullptr, marks);
        if (b.walk_stamp) {  // close the prediction round of the partner marks: the next one starts empty
            ctl->round = round + 1u;
            // no marks with moving lists, nor where nobody needs them
            ctl->fast_n = moves || (next != kTightOff && tight_by_walks(P)) ? kNoMarks : 0ull;
        }
        ctl->max_err_bits = atomicAdd(&ctl->max_err_bits, 0u);  // see every block's contribution
        decide(ps.params(0), ctl);
    }
}

// pcisph.cl:265-300, then predict (pcisph.cl:175-193) or integrate with optional walls
// After the pressure-force sum f: predict (mode 0 before the decision, 1) or integrate (mode 0 after it, 2) with
// optional walls. Returns whether a prediction is fast.
template <class PS>
__device__ __forceinline__ bool finish_pressure_force(const PS& ps, const ListBuffers& b, const DevParams& P,
                                                      Control* ctl, uint32_t i, const float4& xi, const float3& f,
                                                      int mode) {
    const float m = P.particle_mass;
    const float scale = -P.spiky_d1_norm * m * m;
    const float3 fp = make_float3(f.x * scale, f.y * scale, f.z * scale);
    b.f_press[i] = f4(fp, 0.f);
    const bool integrate = mode == 0 ? (ctl->done != 0u) : mode == 2;
    const unsigned plan = b.tight ? ctl->tight_next : kTightOff;
    const bool watch = tight_plan(plan) == kTightUse;
    float4 r = xi;
    if (watch) r = b.tight_ref[i];  // with the loads below, not after them
    const float3 a = (f3(b.f_other[i]) + fp) / m;
    const float3 vi = f3(b.vel[i]);
    float3 v = vi + a * P.dt;
    const float3 dx = v * P.dt;
    float3 x = make_float3(xi.x + dx.x, xi.y + dx.y, xi.z + dx.z);
    if (!integrate) {
        const float4 xs = f4(x, 0.f);
        b.pred[i] = xs;
        bool fast;
        const float threshold = plan == (kTightBuild | kTightEarly) ? P.list_half_skin - P.tight_margin : P.list_half_skin;
        const float disp = note_displacement<!PS::kBatched>(P, ctl, b.bucket_fast, xi, xs, threshold, vi, watch ? &r : nullptr,
                                                            fast, PS::kBatched ? nullptr : b.fast_list, i);
        if (watch) {
            if (!(sqrtf(dist2(xs.x - r.x, xs.y - r.y, xs.z - r.z)) <= P.tight_reach) && ctl->tight_stray == 0u)
                ctl->tight_stray = 1u;  // NaN strays
        }
        if (P.particle_skin) b.disp_max[i] = fmaxf(b.disp_max[i], disp);
        return fast;
    }
    if (P.walls) {
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            float* xs = ax == 0 ? &x.x : ax == 1 ? &x.y : &x.z;
            float* vs = ax == 0 ? &v.x : ax == 1 ? &v.y : &v.z;
            if (*xs < P.box_lo[ax]) {
                *xs = P.box_lo[ax];
                if (*vs < 0.f) *vs = -P.restitution * *vs;
            } else if (*xs > P.box_hi[ax]) {
                *xs = P.box_hi[ax];
                if (*vs > 0.f) *vs = -P.restitution * *vs;
            }
        }
    }
    if constexpr (!PS::kBatched) {
        if (lists_move(P, ctl)) {
            float disp;
            const unsigned set = __ballot_sync(__activemask(), outruns<true>(P, ctl, xi, f4(x, 0.f), P.list_half_skin, vi, disp));
            if (set && (int)(threadIdx.x & 31u) == __ffs(set) - 1) atomicAdd(&ctl->strays, (unsigned)__popc(set));
        }
    }
    const uint32_t o = b.out_index ? b.out_index[i] : i;  // working order -> sorted order
    b.state_pos[o] = f4(x, 0.f);
    b.state_vel[o] = f4(v, 0.f);
    if (P.particle_skin)  // the next step's half skin: twice this step's largest predicted displacement
        b.state_skin[o] = fminf(fmaxf(P.skin_factor * b.disp_max[i] + P.skin_add, P.skin_min_half), P.skin_max_half);
    return false;
}

// One particle's pressure-force sweep.
template <class PS, bool kCoherent = false, int DEEP = 1>
__device__ __forceinline__ void pressure_force_body(const PS& ps, const ListBuffers& b, uint32_t i, int mode) {
    if (i >= ps.count() || ps.skip_force(i)) return;
    const DevParams& P = ps.params(i);
    Control* ctl = ps.control(i);
    const float4 xi = b.pf4[i];
    float3 f = make_float3(0.f, 0.f, 0.f);
    const uint32_t cnt = b.near_count[i];
    // boundary terms at x (within h): all zero unless a boundary particle was within r_list of x; the
    // boundary list holds every one within r_list (terms beyond h are zero)
    const bool near_b = P.boundary_count && b.b_near[i] != 0;
    const uint32_t bcnt = near_b && b.bnbr ? b.bnbr_count[i] : 0u;
    const bool list_boundary = near_b && b.bnbr && bcnt <= P.bnd_cap;
    const bool walk_boundary = near_b && !list_boundary;
    Cell c{0u, 0u, 0u};
    if (cnt > P.near_cap || walk_boundary) c = cell_of(xi.x, xi.y, xi.z, P);
    auto fb = [&](uint32_t j) { pressure_force_term(xi, load_slot<kCoherent>(&b.bpf[j]), P.h, P.h2, f); };
    if (walk_boundary) for_each_neighbour(b.b_cells, c, P, fb);
    else if (list_boundary) for_each_listed(b.bnbr, i, bcnt, b.nbr_stride, fb);
    auto body = [&](uint32_t j) { pressure_force_term(xi, load_slot<kCoherent>(&b.pf4[j]), P.h, P.h2, f); };
    if (cnt > P.near_cap) {
        for_each_neighbour(b.cells, c, P, body);
    } else if constexpr (DEEP > 1) {
        for_each_listed_deep<DEEP>(
            b.near, i, cnt, b.nbr_stride, [&](uint32_t j) { return load_slot<kCoherent>(&b.pf4[j]); },
            [&](const float4& o) { pressure_force_term(xi, o, P.h, P.h2, f); });
    } else {
        for_each_listed(b.near, i, cnt, b.nbr_stride, body);
    }
    finish_pressure_force(ps, b, P, ctl, i, xi, f, mode);
}

// The same with eight lanes per particle, lane q; lane 0 returns whether the prediction is fast.
template <class PS, int L>
__device__ __forceinline__ bool pressure_force_shared(const PS& ps, const ListBuffers& b, uint32_t i0, uint32_t q,
                                                      TermStage<L>& S, int mode) {
    const bool live = i0 < ps.count() && !ps.skip_force(i0);
    const uint32_t i = i0 < ps.count() ? i0 : ps.count() - 1u;
    const uint32_t mask = lanes_mask<L>();
    const DevParams& P = ps.params(i);
    const float4 xi = b.pf4[i];
    float acc = 0.f;  // lane 0, 1, 2: x, y, z
    auto sum = [&](const float4& o, bool valid, uint32_t m) {
        PairTerm term{0.f, 0.f, 0.f, 0.f};
        if (valid) pressure_force_pair(xi, o, P.h, P.h2, [&](const PairTerm& t) { term = t; });
        add_lanes(acc, term, S, q, m);
    };
    auto walk = [&](const uint2* cells, const float4* src) {
        walk_shared<L>(cells, cell_of(xi.x, xi.y, xi.z, P), P, q, [&](uint32_t j, bool valid) {
            float4 o = xi;
            if (valid) o = __ldg(&src[j]);
            sum(o, valid, mask);
        });
    };
    if (P.boundary_count) {
        const bool near_b = live && b.b_near[i] != 0;
        const uint32_t bcnt = near_b && b.bnbr ? b.bnbr_count[i] : 0u;
        const bool listed = b.bnbr && bcnt <= P.bnd_cap;
        const uint32_t n = listed ? bcnt : 0u;
        for_each_shared<L, 32 / L>(
            b.bnbr, i, n, __reduce_max_sync(kAll, n), b.nbr_stride, q, [&](uint32_t j) { return __ldg(&b.bpf[j]); },
            [&](const float4& o, uint32_t, bool valid) { sum(o, valid, kAll); });
        if (near_b && !listed) walk(b.b_cells, b.bpf);
    }
    const uint32_t cnt = live ? b.near_count[i] : 0u;
    const uint32_t n = cnt <= P.near_cap ? cnt : 0u;
    for_each_shared<L, 32 / L>(
        b.near, i, n, __reduce_max_sync(kAll, n), b.nbr_stride, q, [&](uint32_t j) { return __ldg(&b.pf4[j]); },
        [&](const float4& o, uint32_t, bool valid) { sum(o, valid, kAll); });
    if (cnt > P.near_cap) walk(b.cells, b.pf4);
    const float y = __shfl_sync(mask, acc, 1, L), z = __shfl_sync(mask, acc, 2, L);
    if (live && q == 0) return finish_pressure_force(ps, b, P, ps.control(i), i, xi, make_float3(acc, y, z), mode);
    return false;
}

template <class PS, int BS = kBlock, int LANES = 1, int DEEP = 1>
// (at most 40 registers: 48 resident warps per SM; 48 registers measured 10% slower at 1M)
__global__ void __launch_bounds__(BS, LANES > 1 ? 1 : DEEP == 1 ? 1536 / BS : 512 / BS) k_pressure_force_list(PS ps, ListBuffers b, int mode,
                                                            cudaGraphConditionalHandle cond, int use_cond) {
    const uint32_t i = blockIdx.x * BS + threadIdx.x;
    if (!PS::kBatched && use_cond && i == 0) {
        // continue the graph's while loop unless the step is done; the counter bounds it on its own
        Control* ctl = ps.control(0);
        const unsigned g = ++ctl->guard_iters;
        const bool stop = ctl->done != 0u || g >= (unsigned)ps.params(0).max_iters;
        cudaGraphSetConditional(cond, stop ? 0u : 1u);
    }
    if constexpr (LANES == 1) {
        pressure_force_body<PS, false, DEEP>(ps, b, i, mode);
    } else {
        __shared__ TermStage<LANES> stage[BS / LANES];
        const bool fast =
            pressure_force_shared<PS, LANES>(ps, b, i / LANES, i % LANES, stage[threadIdx.x / LANES], mode);
        __shared__ uint32_t delta[BS];
        close_round(ps, b, i / LANES, fast, delta + (threadIdx.x & ~31u));
    }
}

// The corrective loop of one step as one cooperative launch (every block resident, grid-stride over the
// particles): pressure sweep, grid barrier, the loop decision in block 0 (one scene, or every scene of a
// batch with its own convergence flags), grid barrier, pressure-force sweep, grid barrier; until no scene
// iterates, at most max_iters times. Same sweeps and decisions as the graph's while loop, so the same bits.
// Every thread takes every barrier: the bodies return to the loop, never out of the kernel.
// The form of few registers throughout (48, a batch 64: 5 or 4 blocks per SM): what the graph's sweeps gain by walks served by
// a whole warp and by tight lists costs this kernel, whose registers are the largest of its parts', more than half of its warps
// (103 and 123 registers, 2 blocks: 1,000,000 particles at rest 2334 -> 2990 us a step, 16 scenes of 65,000 3119 -> 3610).
template <class PS>
__global__ void __launch_bounds__(kBlock, PS::kBatched ? 4 : 5) k_corrective_loop(PS ps, ListBuffers b, Control* loop, int max_iters) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    const uint32_t stride = gridDim.x * kBlock;
    const uint32_t rounds = (ps.count() + stride - 1) / stride;
    __shared__ int running;
    __shared__ WalkStage unused;
    for (int it = 0; it < max_iters; ++it) {
        if constexpr (!PS::kBatched) {  // boundary pressures at the predicted positions (read by the force)
            const DevParams& P = ps.params(0);
            for (uint32_t k = blockIdx.x * kBlock + threadIdx.x; k < P.boundary_count; k += stride)
                boundary_pressure_list_body<true>(P, ps.control(0), b, k);
        }
        unsigned local = 0;
        for (uint32_t r = 0; r < rounds; ++r)
            local = max(local, __float_as_uint(
                                   pressure_body<PS, true, false, false, false>(
                                       ps, b, r * stride + blockIdx.x * kBlock + threadIdx.x, unused)));
        if (!PS::kBatched) {  // batched scenes reduced per scene inside the body
            const unsigned m = __reduce_max_sync(0xffffffffu, local);
            if ((threadIdx.x & 31) == 0 && m) atomicMax(&ps.control(0)->max_err_bits, m);
        }
        grid.sync();
        if (blockIdx.x == 0) {
            if (threadIdx.x == 0) running = 0;
            __syncthreads();
            if constexpr (!PS::kBatched) {
                if (threadIdx.x == 0) {
                    Control* c = ps.control(0);
                    decide(ps.params(0), c);
                    running = c->done ? 0 : 1;
                }
            } else {
                for (uint32_t sc = threadIdx.x; sc < ps.n_scenes; sc += blockDim.x) {
                    Control* c = &ps.ctls[sc];
                    if (c->done) {
                        c->finished = 1;
                        continue;
                    }
                    decide(ps.table[sc], c);
                    if (!c->done) atomicOr(&running, 1);
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                loop->guard_iters += 1;
                if (PS::kBatched) loop->total_iters += 1;
                loop->any_running = running ? 1u : 0u;
            }
        }
        grid.sync();
        for (uint32_t r = 0; r < rounds; ++r)
            pressure_force_body<PS, true>(ps, b, r * stride + blockIdx.x * kBlock + threadIdx.x, 0);
        grid.sync();
        if (*reinterpret_cast<volatile unsigned*>(&loop->any_running) == 0u) break;
    }
}

// Batch: close one corrective iteration per scene (one thread per scene) and set the graph's loop
// condition: continue while some scene iterates. A scene decided done here is integrated by the
// pressure-force sweep that follows; the next call marks it finished. Every scene is done by its
// max_iters, so the loop ends; the guard bounds it by the largest max_iters on its own.
__global__ void k_batch_decide(const DevParams* __restrict__ table, Control* ctls, uint32_t n_scenes, bool tight, Control* batch,
                               int max_iters, cudaGraphConditionalHandle cond, int use_cond) {
    __shared__ int running;
    if (threadIdx.x == 0) running = 0;
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < n_scenes; s += blockDim.x) {
        Control* c = &ctls[s];
        if (c->done) {
            c->finished = 1;
            continue;
        }
        tight_advance(table[s], c, tight, false);
        decide(table[s], c);
        if (!c->done) atomicOr(&running, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned g = ++batch->guard_iters;
        batch->total_iters += 1;
        const bool more = running != 0 && g < (unsigned)max_iters;
        batch->any_running = more ? 1u : 0u;
        if (use_cond) cudaGraphSetConditional(cond, more ? 1u : 0u);
    }
}

// Batch step start: per-scene iteration state.
// Per scene, before a step: reset the step's control fields. A scene with an adaptive skin takes the
// smallest skin level that at most 1 in skin_outrun_ratio of the previous step's predictions outran (the
// largest if none), from that step's counts, and writes its list radius into the scene table; the builder
// and the sweeps of this step read it there. Results do not depend on the choice.
__global__ void k_batch_begin(DevParams* table, Control* ctls, uint32_t n_scenes, Control* batch) {
    for (uint32_t s = threadIdx.x; s < n_scenes; s += blockDim.x) {
        Control* c = &ctls[s];
        DevParams* P = &table[s];
        if (P->adaptive_skin) {
            int level = 0;
            if (c->steps) {
                const unsigned long long preds =
                    (unsigned long long)P->fluid_count * (unsigned long long)max(c->iterations_last, 1);
                level = kSkinLevels - 1;
                for (int k = kSkinLevels - 1; k >= 0; --k)
                    if (c->over_level[k] * (unsigned long long)P->skin_outrun_ratio <= preds) level = k;
            }
            c->skin_level = (unsigned)level;
            set_list_skin(P, skin_level_value(level));
            for (int k = 0; k < kSkinLevels; ++k) c->over_level[k] = 0;
        }
        c->iter = 0;
        c->done = 0;
        c->finished = 0;
        c->max_err_bits = 0;
        c->fast_at_begin = c->fast_particles;
        c->lists_outrun = 0;
        c->tight_next = kTightOff;
        c->tight_stray = 0;
        c->tight_age = 0;
        c->tight_outrun = 0;
        c->tight_asked = 0;
        c->fast_before = c->fast_particles;
        c->status = 0;
    }
    if (threadIdx.x == 0) {
        batch->guard_iters = 0;
        batch->any_running = 1;
        batch->status = 0;  // the reorder flags an out-of-range sorted index here
    }
}

__global__ void __launch_bounds__(kBlock) k_scene_of(const uint32_t* __restrict__ offsets, uint32_t n_scenes,
                                                     uint32_t n, uint16_t* __restrict__ scene_of) {
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= n) return;
    uint32_t lo = 0, hi = n_scenes;  // largest s with offsets[s] <= i
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (offsets[mid] <= i) lo = mid;
        else hi = mid;
    }
    scene_of[i] = (uint16_t)lo;
}

// sort_utils.cl:12-23 per scene, offset into the scene's bucket range of the shared table
__global__ void __launch_bounds__(kBlock) k_hash_scenes(SceneTable ps, const float4* __restrict__ pos,
                                                        uint32_t* __restrict__ keys) {
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= ps.count()) return;
    const DevParams& P = ps.params(i);
    const float4 p = pos[i];
    const Cell c = cell_of(p.x, p.y, p.z, P);
    keys[i] = P.bucket_base + hash_key(c.x, c.y, c.z, P);
}

}  // namespace

namespace {
inline unsigned grid_cells(uint32_t n, int w) {
    const uint32_t per = (kCellBlock / 32) * (uint32_t)w;
    return (n + per - 1) / per;
}
template <class PS>
void launch_density(const PS& ps, uint32_t n, bool boundary, const ListBuffers& b, cudaStream_t s) {
    auto go = [&](auto w) {
        constexpr int W = decltype(w)::value;
        if constexpr (!PS::kBatched)
            if (boundary) {
                k_density_list<PS, true, W><<<grid_cells(n, W), kCellBlock, 0, s>>>(ps, b);
                return;
            }
        k_density_list<PS, false, W><<<grid_cells(n, W), kCellBlock, 0, s>>>(ps, b);
    };
    // Fewer particles per warp where warps are few: 4,096 particles take 12 us with 8, 10 with 2 (32,768: 28 / 27 / 32 us
    // with 8 / 4 / 2, and 8 scenes at once 7% less time each with 8); from there on the set-up of a cell per warp costs more than it spreads (156,244 particles
    // 82 / 95 / 129 us, 1,048,576 495 / 605 / 845).
    if (n <= 8192u) go(std::integral_constant<int, 2>{});
    else if (n <= 16384u) go(std::integral_constant<int, 4>{});
    else go(std::integral_constant<int, 8>{});
}
}  // namespace

void launch_density_list(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    launch_density(OneScene{P, ctl}, P.fluid_count, P.boundary_count != 0, b, s);
}
// Scenes of few threads, us per launch (CUDA events; about 5 of them the events' own) by one lane / two chunks in flight /
// eight lanes per particle:
//   particles   pressure             pressure force       normal               force
//   4,096       15.2 / 15.7 / 11.3   14.2 / 10.1 / 8.0    14.7 / 10.4 / 8.5    19.0 / 18.9 / 11.4
//   8,000       14.4 / 15.8 / 11.8   14.4 / 10.2 / 10.1   15.0 / 11.0 / 10.1   19.5 / 19.4 / 14.6
//   15,625      14.8 / 15.4 / 13.3   15.3 / 10.7 / 12.2   15.0 / 10.9 / 12.7   19.2 / 20.2 / 22.2
//   32,768      14.8 / 16.8 / 19.0   15.2 / 12.1 / 16.2   14.5 / 10.7 / 16.2   19.2 /  -   / 33
//   64,000      19.5 / 21.0 / 29.8   16.2 / 16.3 / 26.4   15.1 / 16.2 / 25
constexpr int kLanes = 8;
constexpr uint32_t kDeepMax = 49152u;   // two chunks in flight, pressure force and normal
// Past 2M particles the default block of the corrective sweeps, 256, stands for 128 threads (8.4M: pressure force 614 -> 588
// us, pressure 663 -> 658; equal at 1M).
constexpr uint32_t kLargeScene = 1u << 21;
int sweep_block_used(uint32_t n, int block) {
    if (n <= kSharedMax) return 0;
    return block == kBlock && n > kLargeScene ? 128 : block;
}

void launch_moving_lists(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    const unsigned blocks = std::min(grid_cells(P.fluid_count, 8), 5u * kSms);
    if (P.fluid_count) k_moving_lists<<<blocks, kCellBlock, 0, s>>>(P, ctl, b);
}

void launch_distrust_moving_lists(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    k_distrust_moving_lists<<<grid_for(P.bucket_count), kBlock, 0, s>>>(P, ctl, b.bucket_fast);
}

void launch_normal_list(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    const uint32_t n = P.fluid_count;
    if (n <= kSharedMax) k_normal_shared<OneScene, kLanes><<<grid_for(n * kLanes), kBlock, 0, s>>>(OneScene{P, ctl}, b);
    else if (n <= kDeepMax) k_normal_list<OneScene, 2><<<grid_for(n), kBlock, 0, s>>>(OneScene{P, ctl}, b);
    else k_normal_list<<<grid_for(n), kBlock, 0, s>>>(OneScene{P, ctl}, b);
}
void launch_force_list(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    const uint32_t n = P.fluid_count;
    if (n <= kSharedMax) k_force_shared<OneScene, kLanes><<<grid_for(n * kLanes), kBlock, 0, s>>>(OneScene{P, ctl}, b);
    else k_force_list<<<grid_for(n), kBlock, 0, s>>>(OneScene{P, ctl}, b);
}
void launch_pressure_list(const DevParams& P, Control* ctl, const ListBuffers& b, int block, bool builds,
                          cudaStream_t s) {
    const OneScene ps{P, ctl};
    const uint32_t n = P.fluid_count;
    auto go = [&](auto bs, auto shared) {
        constexpr int BS = decltype(bs)::value;
        constexpr bool S = decltype(shared)::value;
        const unsigned blocks = (n + BS - 1) / BS;
        // 64 registers a thread (4 blocks of 256 per SM) against 48 (5 blocks), us per launch over the sweeps of a step (skin,
        // building and tight): 200,704 particles 35.5 / 36.8, 287,496 37.5 / 42.4, 405,224 52.5 / 55.8, 592,704 67.0 / 70.9,
        // 1,048,576 112.3 / 113.5, 2.6M equal (few walkers in a function of their own then; inlined, a step of 200,000 to
        // 2,000,000 takes 0.4 to 0.7% less). 48 where they hold a scene in one wave that 64 just miss (156,244: 27.6 / 23.9;
        // the building sweep 43 / 37). Past 2M every lane walks by itself, which needs none of the spills of the other form
        // (skin list, before the lists were read past L1: 8.4M 1050 -> 1036).
        if (n > kLargeScene) k_pressure_list<OneScene, BS, 1, false, S, 1280><<<blocks, BS, 0, s>>>(ps, b);
        else if (n > 1024u * kSms && n <= 1280u * kSms) k_pressure_list<OneScene, BS, 1, true, S, 1280><<<blocks, BS, 0, s>>>(ps, b);
        else k_pressure_list<OneScene, BS, 1, true, S><<<blocks, BS, 0, s>>>(ps, b);
    };
    if (n <= kSharedMax) k_pressure_list<OneScene, kBlock, kLanes><<<grid_for(n * kLanes), kBlock, 0, s>>>(ps, b);
    else if (builds && b.tight) go(std::integral_constant<int, 128>{}, std::true_type{});
    else if (sweep_block_used(n, block) == 128) go(std::integral_constant<int, 128>{}, std::false_type{});
    else if (block == 512) go(std::integral_constant<int, 512>{}, std::false_type{});
    else go(std::integral_constant<int, kBlock>{}, std::false_type{});
}
bool marks_inline(uint32_t n) { return n <= kSharedMax; }
void launch_mark_partners(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    k_mark_partners<<<kMarkBlocks, kBlock, 0, s>>>(P, ctl, b);
}
void launch_pressure_force_list(const DevParams& P, Control* ctl, const ListBuffers& b, int mode,
                                cudaGraphConditionalHandle cond, bool use_cond, int block, cudaStream_t s) {
    const OneScene ps{P, ctl};
    const uint32_t n = P.fluid_count;
    const int uc = use_cond ? 1 : 0;
    if (n <= kSharedMax)
        k_pressure_force_list<OneScene, kBlock, kLanes><<<grid_for(n * kLanes), kBlock, 0, s>>>(ps, b, mode, cond, uc);
    else if (n <= kDeepMax)
        k_pressure_force_list<OneScene, 128, 1, 2><<<(n + 127) / 128, 128, 0, s>>>(ps, b, mode, cond, uc);
    else if (sweep_block_used(n, block) == 128)
        k_pressure_force_list<OneScene, 128><<<(n + 127) / 128, 128, 0, s>>>(ps, b, mode, cond, uc);
    else if (block == 512) k_pressure_force_list<OneScene, 512><<<(n + 511) / 512, 512, 0, s>>>(ps, b, mode, cond, uc);
    else k_pressure_force_list<OneScene, kBlock><<<grid_for(n), kBlock, 0, s>>>(ps, b, mode, cond, uc);
}

namespace {
template <class PS>
cudaError_t launch_loop(const PS& ps, uint32_t n, const ListBuffers& b, Control* loop, int max_iters, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    int dev = 0, sms = 0, per_sm = 0, coop = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_corrective_loop<PS>, kBlock, 0);
    if (e != cudaSuccess) return e;
    if (!coop || per_sm < 1) return cudaErrorNotSupported;
    const unsigned blocks = std::min<unsigned>((unsigned)(sms * per_sm), grid_for(n));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kBlock);
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_corrective_loop<PS>, ps, b, loop, max_iters);
}
}  // namespace

cudaError_t launch_corrective_loop(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    return launch_loop(OneScene{P, ctl}, P.fluid_count, b, ctl, P.max_iters, s);
}
cudaError_t launch_corrective_loop_scenes(const SceneTable& t, const ListBuffers& b, Control* batch, int max_iters,
                                          cudaStream_t s) {
    return launch_loop(t, t.n, b, batch, max_iters, s);
}

void launch_boundary_cell_bounds(const DevParams& P, const float4* b_pos, int* bounds, cudaStream_t s) {
    if (P.boundary_count) k_boundary_cell_bounds<<<grid_for(P.boundary_count), kBlock, 0, s>>>(P, b_pos, bounds);
}
void launch_boundary_zone(const DevParams& P, const float4* b_pos, const int* org, const uint32_t* dim,
                          unsigned char* zone, cudaStream_t s) {
    if (P.boundary_count)
        k_boundary_zone<<<grid_for(P.boundary_count), kBlock, 0, s>>>(P, b_pos, org[0], org[1], org[2], dim[0],
                                                                      dim[1], zone);
}
void launch_boundary_fluid_list(const DevParams& P, const ListBuffers& b, cudaStream_t s) {
    if (P.boundary_count) k_boundary_fluid_list<<<grid_cells(P.boundary_count, 8), kCellBlock, 0, s>>>(P, b);
}
void launch_boundary_pressure_list(const DevParams& P, Control* ctl, const ListBuffers& b, cudaStream_t s) {
    if (P.boundary_count) k_boundary_pressure_list<<<grid_for(P.boundary_count), kBlock, 0, s>>>(P, ctl, b);
}
void launch_batch_begin(DevParams* table, Control* ctls, uint32_t n_scenes, Control* batch, cudaStream_t s) {
    k_batch_begin<<<1, 256, 0, s>>>(table, ctls, n_scenes, batch);
}
void launch_scene_of(const uint32_t* offsets, uint32_t n_scenes, uint32_t n, uint16_t* scene_of, cudaStream_t s) {
    if (n) k_scene_of<<<grid_for(n), kBlock, 0, s>>>(offsets, n_scenes, n, scene_of);
}
void launch_hash_scenes(const SceneTable& t, const float4* pos, uint32_t* keys, cudaStream_t s) {
    if (t.n) k_hash_scenes<<<grid_for(t.n), kBlock, 0, s>>>(t, pos, keys);
}
void launch_density_scenes(const SceneTable& t, const ListBuffers& b, cudaStream_t s) {
    if (t.n) launch_density(t, t.n, false, b, s);  // no boundary in a batch
}
void launch_normal_scenes(const SceneTable& t, const ListBuffers& b, cudaStream_t s) {
    if (t.n) k_normal_list<<<grid_for(t.n), kBlock, 0, s>>>(t, b);
}
void launch_force_scenes(const SceneTable& t, const ListBuffers& b, cudaStream_t s) {
    if (t.n) k_force_list<<<grid_for(t.n), kBlock, 0, s>>>(t, b);
}
void launch_pressure_scenes(const SceneTable& t, const ListBuffers& b, bool builds, cudaStream_t s) {
    if (!t.n) return;
    if (builds && b.tight)
        k_pressure_list<SceneTable, 128, 1, true, true><<<(t.n + 127) / 128, 128, 0, s>>>(t, b);
    else k_pressure_list<<<grid_for(t.n), kBlock, 0, s>>>(t, b);
}
void launch_pressure_force_scenes(const SceneTable& t, const ListBuffers& b, cudaStream_t s) {
    if (t.n) k_pressure_force_list<<<grid_for(t.n), kBlock, 0, s>>>(t, b, 0, 0, 0);
}
void launch_batch_decide(const SceneTable& t, const ListBuffers& b, Control* batch, int max_iters, cudaGraphConditionalHandle cond,
                         bool use_cond, cudaStream_t s) {
    k_batch_decide<<<1, 256, 0, s>>>(t.table, t.ctls, t.n_scenes, b.tight != nullptr, batch, max_iters, cond, use_cond ? 1 : 0);
}

}  // namespace pcisph
