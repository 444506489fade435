// Kernels of the GB300 pairwise box-intersection pipeline.
//
//   k_count    boxes -> per-cell counts                (src/pbig/pbig.cu:174-221)
//   k_scan     counts -> cell starts + cell work lists (host thrust scan, pbig.cu:1497-1505,
//              and the job list of sched_phase, pbig.cu:1586-1688)
//   k_scatter  boxes -> cell entry lists               (d_mapping, pbig.cu:321-427)
//   k_pairs    per-cell all-pairs test with the reference-cell rule and compacted output
//              (d_matching + prefix_scan, pbig.cu:429-543, 562-603, 641-932), with tile tasks for
//              cells too big for shared memory         (sched_phase's 256-row jobs)
//
// Box records are the reference's RectInfo (rect.h): 2*D+1 unsigned words.
// Cell ids follow the reference linearisation gid = (k*nrc + j)*nrc + i.
// An entry stores the box index, three "starts here" bits -- bit d is set
// when the box's minimum along axis d lies in this cell -- and the box's part
// of the cell in 15-bit terms ("entries" below). The reference-cell rule of
// calcRightToWrite (pbig.cu:579-603) -- a pair is reported in the cell holding
// the minimum corner of the two boxes' intersection -- is then exactly
// (flags_a | flags_b) == 7: along each axis max(min_a, min_b) falls in this
// cell iff one of the two minima does (both boxes cover the cell).
#include "kernels.cuh"

#include <cstdio>

namespace pbig {

#define FULL_MASK 0xffffffffu

__host__ __device__ __forceinline__ unsigned long long mn64(unsigned long long a, unsigned long long b) {
    return a < b ? a : b;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(FULL_MASK, v, o);
        if (lane_id() >= o) v += t;
    }
    return v;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

// kernels take their sizes from device memory when p.dyn is set
__device__ __forceinline__ Params resolve(const Params& in) {
    Params p = in;
    if (p.dyn) {
        p.nboxes = p.dyn->nboxes;
        p.ncells = p.dyn->ncells;
        p.nscenes = p.dyn->nscenes;
        p.open |= p.dyn->open;
    }
    return p;
}

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// the query's clock: a kernel's first block notes when it starts
__device__ __forceinline__ void stamp(const Params& p, int k) {
    if (blockIdx.x == 0 && threadIdx.x == 0) p.ctr->stamp[k] = now_ns();
}

// the run counters to page-locked host memory (one thread; the counters were
// changed through L2 by other blocks)
__device__ __forceinline__ void ctr_to_host(const Ctr* ctr, Ctr* host) {
    constexpr uint32_t kWords = sizeof(Ctr) / sizeof(unsigned long long);
    static_assert(sizeof(Ctr) % sizeof(unsigned long long) == 0, "run counters in 8-byte words");
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(ctr);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(host);
    unsigned long long w[kWords];
#pragma unroll
    for (uint32_t k = 0; k < kWords; k++) w[k] = __ldcg(src + k);
#pragma unroll
    for (uint32_t k = 0; k < kWords; k++) dst[k] = w[k];
    __threadfence_system();
}

// at the end of a query's last kernel (p.ctr_host set): its last block to
// finish hands the run counters to the host, so no copy follows the kernel
__device__ __forceinline__ void query_end(const Params& p) {
    if (!p.ctr_host) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&p.ctr->done, 1u) == gridDim.x - 1) {
            __threadfence();
            p.ctr->stamp[kStampEnd] = now_ns();
            __threadfence();
            ctr_to_host(p.ctr, p.ctr_host);
        }
    }
}

// (where the last two kernels run beside each other)
__global__ void k_query_end(Params p) { query_end(p); }

// the last scene s in [lo, hi) with scene_box_off[s] <= gi
__device__ __forceinline__ uint32_t search_scene(const Params& p, uint64_t gi, uint32_t lo, uint32_t hi) {
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (p.scene_box_off[mid] <= gi) lo = mid;
        else hi = mid;
    }
    return lo;
}

// scene of global box gi: with the scene table (scene of every 256th box)
// the search covers only the scenes that start inside gi's 256-box block
constexpr uint32_t kSceneTableShift = 8;
__device__ __forceinline__ uint32_t find_scene(const Params& p, uint64_t gi) {
    if (p.nscenes <= 1) return 0;
    if (p.scene_table) {
        const uint64_t b = gi >> kSceneTableShift;
        const uint32_t s0 = p.scene_table[b];
        const uint32_t s1 = ((b + 1) << kSceneTableShift) < p.nboxes ? p.scene_table[b + 1] : p.nscenes - 1;
        return search_scene(p, gi, s0, s1 + 1);
    }
    return search_scene(p, gi, 0, p.nscenes);
}

__global__ void k_scene_table(Params pin) {
    chain_wait();
    const Params p = resolve(pin);
    const uint64_t n = (p.nboxes + (1u << kSceneTableShift) - 1) >> kSceneTableShift;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < n; b += (uint64_t)gridDim.x * blockDim.x)
        p.scene_table[b] = p.nscenes <= 1 ? 0u : search_scene(p, b << kSceneTableShift, 0, p.nscenes);
}

// ---------------------------------------------------------------------------
// per-scene cell sizes of a batched query: one warp per scene runs the host
// tuner's analytic model (tune_impl with T = E^2 / 2C) on the rows
// a + floor(k * n / m), k < m = min(n, 64), of the scene [a, a + n). Every
// sum is of integers (exact in any order), so the choice equals the host
// model's on the same rows. The sizes are counted one after the other in
// integers and weighed side by side, a lane a size: double precision runs at a
// sixty-fourth of the rate, and with all of it in every lane, eight scenes to
// an SM, the kernel took 40 us; now 12.
// ---------------------------------------------------------------------------
constexpr uint32_t kTuneRows = 64;

__device__ __forceinline__ uint32_t nrc_dev(uint32_t range, int s) {
    return (uint32_t)(((uint64_t)range + (1ull << s) - 1) >> s);
}

// one warp: the cell shift of the scene of n boxes at row a (grids of at
// most max_cells cells)
__device__ __forceinline__ SceneTune tune_scene_warp(const uint32_t* boxes, uint64_t a, uint64_t n, int dims,
                                                     uint32_t range, double max_cells) {
    const uint32_t lane = lane_id();
    const uint32_t W = 2 * (uint32_t)dims + 1;
    {
        const uint64_t m = n < kTuneRows ? n : kTuneRows;
        uint32_t lo[2][3] = {{0, 0, 0}, {0, 0, 0}}, hi[2][3] = {{0, 0, 0}, {0, 0, 0}};
        bool ok[2] = {false, false};
        uint64_t ext = 0, good = 0;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint64_t k = lane + 32u * j;
            if (k >= m) continue;
            const uint32_t* b = boxes + (a + k * n / m) * W;
            bool v = true;
            for (int d = 0; d < dims; d++) {
                lo[j][d] = b[2 * d];
                hi[j][d] = b[2 * d + 1];
                v = v && lo[j][d] <= hi[j][d] && hi[j][d] < range;
            }
            ok[j] = v;
            if (v) {
                for (int d = 0; d < dims; d++) ext += (uint64_t)(hi[j][d] - lo[j][d]) + 1;
                good++;
            }
        }
        ext = warp_sum_u64(ext);
        good = warp_sum_u64(good);
        SceneTune best{0u, 0u, 0.0};
        if (m == 0) {
            uint32_t s = 31;
            while (s > 0 && nrc_dev(range, (int)s - 1) <= 1) s--;
            best.shift = s;
        } else {
            const int s0 = tune_s0(ext, (good ? good : 1) * (uint64_t)dims);
            const double scale = (double)n / (double)m;
            const int s_win = s0 + 3 < 31 ? s0 + 3 : 31;
            best.shift = 32u;
            // the window, then every coarser size if none of it qualifies
            for (int pass = 0; pass < 2 && best.shift == 32u; pass++) {
                const int first = pass ? s_win + 1 : s0 - 2 > 0 ? s0 - 2 : 0, last = pass ? 31 : s_win;
                uint32_t entries = 0;  // lane s - first: the sample's at shift s
                bool fits = false;
                for (int s = first; s <= last; s++) {
                    uint32_t e = 0;
                    bool huge = false;  // (without one, 64 boxes of less than 2^26 cells: below 2^32)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        if (!ok[j]) continue;
                        uint64_t c = 1;
                        for (int d = 0; d < dims; d++) c = c >= (1ull << 26) ? c : c * ((uint64_t)((hi[j][d] >> s) - (lo[j][d] >> s)) + 1);
                        huge = huge || c >= (1ull << 26);
                        e += (uint32_t)c;
                    }
                    e = __reduce_add_sync(FULL_MASK, e);
                    huge = __any_sync(FULL_MASK, huge);
                    if ((int)lane == s - first) {
                        entries = e;
                        fits = !huge && e <= 64u * (uint32_t)m;
                    }
                }
                const double C = tune_cells(nrc_dev(range, min(first + (int)lane, 31)), dims);
                double E = 0.0;
                unsigned long long cost = ~0ull;  // (positive doubles are in the order of their bits)
                if (fits && C <= max_cells && (!pass || C <= fmax(4096.0, 64.0 * (double)n))) {
                    E = tune_mul((double)entries, scale);
                    cost = (unsigned long long)__double_as_longlong(tune_cost(C, E, tune_mul(E, E) / tune_mul(2.0, C)));
                }
                uint32_t l = lane;  // of the least cost, the finest on a tie
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    const unsigned long long k = __shfl_xor_sync(FULL_MASK, cost, o);
                    const uint32_t kl = __shfl_xor_sync(FULL_MASK, l, o);
                    if (k < cost || (k == cost && kl < l)) {
                        cost = k;
                        l = kl;
                    }
                }
                if (cost != ~0ull) {
                    best.shift = (uint32_t)first + l;
                    best.est_entries = __shfl_sync(FULL_MASK, E, l);
                }
            }
            if (best.shift == 32u) {  // the coarsest grid that is not a single cell
                uint32_t s = 31;
                while (s > 0 && nrc_dev(range, (int)s - 1) <= 1) s--;
                best.shift = s;
                best.est_entries = (double)n;
            }
        }
        return best;
    }
}

__global__ void k_tune_scenes(const uint32_t* boxes, const unsigned long long* offs, uint32_t nsc, int dims,
                              uint32_t range, SceneTune* out) {
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t sc = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; sc < nsc; sc += nw) {
        const uint64_t a = offs[sc];
        const SceneTune best = tune_scene_warp(boxes, a, offs[sc + 1] > a ? offs[sc + 1] - a : 0, dims, range, 4.0e9);
        if (lane_id() == 0) out[sc] = best;
    }
}

// ---------------------------------------------------------------------------
// the cell size of a single-scene query: block b of kTuneBlocks weighs the
// candidates s0 - 2 + b, + kTuneBlocks, ... (s0 = log2 of the sample's mean
// extent) with the cost model on a strided sample: C cells, E entries, and T tests. A cell holds
// about E/m entries for every box whose lower corner lies in it (m boxes in
// the sample), so T is (E/m)^2 times the pairs of sampled corners that share a
// cell (counted in a shared-memory hash table), times (n/m)^2, since a pair
// survives sampling with probability (m/n)^2. The last block to finish takes
// the cheapest, the finest on a tie, and writes the query's tables.
//
// Latency is all that counts here, so one thread does the arithmetic in double
// precision (its rate is a sixty-fourth: 30 us with every thread at it) and
// the others count in integers. Counting every cell of the sampled boxes
// took 40 us when they were dealt out evenly over the threads, and 115 to 300
// us with a thread per box, which waited for its largest. On the host the
// sample's way there and back took 20 us or more, and a scene not seen before
// two milliseconds of hashing; scenes were recognised by size and mean extent,
// and one taken for another could run at a cell size that made it ten times
// slower.
// ---------------------------------------------------------------------------
constexpr int kTuneThreads = 1024;
constexpr uint32_t kTuneBlocks = 8;          // s0 - 2 .. s0 + 5; coarser sizes are dealt out over the blocks
constexpr uint32_t kTuneSlots = 8192;        // hash table {cell + 1, corners}, twice the sample
constexpr int kTunePer = (int)(kTuneSample / kTuneThreads);
constexpr size_t kTuneSmem = kTuneSlots * 2 * sizeof(uint32_t);
static_assert(kTuneSlots == 2 * kTuneSample && kTuneThreads == 1024, "tuner table and sums");
static_assert((1 + 3 * kTuneBlocks) * sizeof(unsigned long long) < kTuneScratchBytes, "tuner scratch, launch_least_shift's word at its end");

// a box's coordinates, wherever its row begins, in two or three 16-byte loads
// (every row is a line or two of its own, and each load instruction looks all
// of a warp's lines up: with a load per word the sample alone took 12 us). Rows
// [0, n) of the array at `rows`; one whose 16 bytes reach out of it is read word
// by word.
template <int D>
__device__ __forceinline__ void load_row(const uint32_t* rows, uint64_t n, uint64_t i, uint32_t (&v)[2 * D]) {
    constexpr uint32_t W = 2 * D + 1;
    const uint32_t* b = rows + i * W;
    const uint32_t o = (uint32_t)((uint64_t)b >> 2) & 3u;
    if ((i == 0 || i + 1 == n) && row_loads((uint64_t)b, 2 * D, (uint64_t)rows, (uint64_t)(rows + n * W)).count == 0u) {
#pragma unroll
        for (int k = 0; k < 2 * D; k++) v[k] = __ldg(b + k);
        return;
    }
    const uint4* q = reinterpret_cast<const uint4*>(b - o);
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    const uint4 q0 = __ldg(q), q1 = o + 2 * D > 4 ? __ldg(q + 1) : z, q2 = o + 2 * D > 8 ? __ldg(q + 2) : z;
    uint32_t w[11] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z};
    if (o & 1u) {
#pragma unroll
        for (int k = 0; k < 10; k++) w[k] = w[k + 1];
    }
#pragma unroll
    for (int k = 0; k < 2 * D; k++) v[k] = o & 2u ? w[k + 2] : w[k];
}

struct TuneShared {
    uint32_t part[2][kTuneThreads / 32];
    int s0;
};

// two sums over the block, each below 2^32 (every thread gets them)
__device__ __forceinline__ uint2 block_sums(TuneShared& s, uint32_t x, uint32_t y) {
    x = __reduce_add_sync(FULL_MASK, x);
    y = __reduce_add_sync(FULL_MASK, y);
    __syncthreads();
    if (lane_id() == 0) {
        s.part[0][threadIdx.x >> 5] = x;
        s.part[1][threadIdx.x >> 5] = y;
    }
    __syncthreads();
    return make_uint2(__reduce_add_sync(FULL_MASK, s.part[0][lane_id()]),
                      __reduce_add_sync(FULL_MASK, s.part[1][lane_id()]));
}

// cells of the grid at shift sh, ~0 for 2^32 per two axes or more (beyond every limit here)
template <int D>
__device__ __forceinline__ uint64_t tune_grid(uint32_t range, uint32_t sh) {
    const uint64_t nrc = nrc_dev(range, (int)sh);
    return nrc >= 65536ull ? ~0ull : D == 3 ? nrc * nrc * nrc : nrc * nrc;
}

// this thread's part of the sample's entries at cell shift sh. (A box of too many
// cells counts for 2^19: the sample may have 2^18 at most.)
template <int D>
__device__ __forceinline__ uint32_t tune_entries(const uint32_t (&lo)[kTunePer][D], const uint32_t (&hi)[kTunePer][D],
                                                 const bool (&ok)[kTunePer], uint32_t sh) {
    uint32_t e = 0;
#pragma unroll
    for (int j = 0; j < kTunePer; j++) {
        if (!ok[j]) continue;
        unsigned long long c = 1;
#pragma unroll
        for (int d = 0; d < D; d++) {
            const unsigned long long k = (hi[j][d] >> sh) - (lo[j][d] >> sh) + 1;
            c = c >= (1ull << 26) ? c : c * k;
        }
        e += (uint32_t)(c < (1ull << 19) ? c : (1ull << 19));
    }
    return e;
}

// the sample's pairs of corners in a cell at cell shift sh (grids of less than 2^32 cells)
template <int D>
__device__ uint32_t tune_pairs(TuneShared& s, uint32_t* key, const uint32_t (&lo)[kTunePer][D], const bool (&ok)[kTunePer],
                               uint32_t range, uint32_t sh) {
    const uint32_t t = threadIdx.x, nrc = nrc_dev(range, (int)sh);
    uint32_t* cnt = key + kTuneSlots;
    for (uint32_t i = t; i < kTuneSlots / 2; i += kTuneThreads) reinterpret_cast<uint4*>(key)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    uint32_t found = 0;  // < 2^23
#pragma unroll
    for (int j = 0; j < kTunePer; j++) {
        if (!ok[j]) continue;
        const uint32_t z = D == 3 ? lo[j][D - 1] >> sh : 0u;
        const uint32_t id = (z * nrc + (lo[j][1] >> sh)) * nrc + (lo[j][0] >> sh) + 1u;  // (C < 2^32)
        uint32_t h = (id * 0x9e3779b1u) >> 19;
        for (uint32_t probe = 0; probe < kTuneSlots; probe++, h = (h + 1) & (kTuneSlots - 1)) {
            const uint32_t old = atomicCAS(&key[h], 0u, id);
            if (old != 0u && old != id) continue;
            found += atomicAdd(&cnt[h], 1u);  // a new member pairs with every earlier one
            break;
        }
    }
    static_assert(kTuneSlots == 1u << 13, "13 bits of the hash");
    return block_sums(s, found, 0u).x;
}

// the cost model (one thread): C cells, the sample's counts, m of n boxes. Of
// a red/blue query's tests those of one colour are left out.
__device__ double tune_cost_query(uint64_t C, uint32_t entries, uint32_t pairs, uint32_t m, uint64_t n, bool bip, double& E) {
    const double per_box = (double)entries / (double)m, f = per_box * ((double)n / (double)m);
    E = per_box * (double)n;
    return kQueryCell * (double)C + kQueryEntry * E + (bip ? 0.5 : 1.0) * kQueryTest * ((double)pairs * f * f);
}

// the finest cell shift at which every valid box covers less than 2^26 cells
// (the tuner's sample can miss the box that does not; of queries that met one)
template <int D>
__global__ void __launch_bounds__(256) k_least_shift(TuneArgs a, unsigned int* least) {
    constexpr uint32_t W = 2 * D + 1;
    uint32_t s = 0;  // at which all of this thread's boxes so far fit
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < a.n; g += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t* b = g < a.n_red ? a.red + g * W : a.blue + (g - a.n_red) * W;
        uint32_t lo[D], hi[D];
        bool valid = true;
#pragma unroll
        for (int d = 0; d < D; d++) {
            lo[d] = __ldg(b + 2 * d);
            hi[d] = __ldg(b + 2 * d + 1);
            valid = valid && lo[d] <= hi[d] && hi[d] < a.range;
        }
        while (valid && s < 31u) {
            unsigned long long c = 1;
#pragma unroll
            for (int d = 0; d < D; d++) {
                const unsigned long long k = (hi[d] >> s) - (lo[d] >> s) + 1ull;
                c = c >= (1ull << 26) ? c : c * k;
            }
            if (c < (1ull << 26)) break;
            s++;
        }
    }
    s = __reduce_max_sync(FULL_MASK, s);
    if (lane_id() == 0 && s) atomicMax(least, s);
}

template <int D>
__global__ void __launch_bounds__(kTuneThreads, 1) k_tune_query(Params p, TuneArgs a) {
    extern __shared__ __align__(16) uint32_t table[];
    __shared__ TuneShared s;
    const uint32_t t = threadIdx.x;
    chain_wait();
    const unsigned long long began = now_ns();
    uint32_t shift = a.shift;
    double est = (double)a.n;
    if (a.shift == kTuneShift) {
        const uint32_t m = (uint32_t)mn64(a.n, kTuneSample);
        uint32_t lo[kTunePer][D], hi[kTunePer][D];
        bool ok[kTunePer];
        unsigned long long ext = 0;
        uint32_t good = 0;
#pragma unroll
        for (int j = 0; j < kTunePer; j++) {
            const uint32_t k = t + (uint32_t)j * kTuneThreads;
            ok[j] = k < m;
            static_assert(kTuneSample == 1u << 12, "row k * n / m of a full sample");
            const uint64_t g = !ok[j] ? 0ull : a.n > kTuneSample ? (uint64_t)k * a.n >> 12 : k;
            const bool red = g < a.n_red;
            uint32_t v[2 * D] = {};
            if (ok[j]) load_row<D>(red ? a.red : a.blue, red ? a.n_red : a.n - a.n_red, red ? g : g - a.n_red, v);
#pragma unroll
            for (int d = 0; d < D; d++) {
                lo[j][d] = v[2 * d];
                hi[j][d] = v[2 * d + 1];
            }
#pragma unroll
            for (int d = 0; d < D; d++) ok[j] = ok[j] && lo[j][d] <= hi[j][d] && hi[j][d] < a.range;
            if (ok[j]) {
#pragma unroll
                for (int d = 0; d < D; d++) ext += (unsigned long long)(hi[j][d] - lo[j][d]) + 1;
                good++;
            }
        }
        // (ext: up to 2^46 over the block, in three sums)
        const uint2 lo_mid = block_sums(s, (uint32_t)ext & 0xffffu, (uint32_t)(ext >> 16) & 0xffffu);
        const uint2 top = block_sums(s, (uint32_t)(ext >> 32), good);
        ext = ((unsigned long long)top.x << 32) + ((unsigned long long)lo_mid.y << 16) + lo_mid.x;
        if (t == 0) {
            const unsigned long long mean = ext / ((top.y ? top.y : 1u) * (unsigned long long)D);
            s.s0 = mean < 2ull ? 0 : 63 - __clzll((long long)mean);
        }
        __syncthreads();
        const int s0 = s.s0, s_lo = s0 - 2 > 0 ? s0 - 2 : 0, s_win = s0 + 3 < 31 ? s0 + 3 : 31;
        // s0 + 4 and s0 + 5 (of boxes of two sizes the mean says little) where s0 + 3
        // makes at most 64 cells a box
        const int s_far = tune_grid<D>(a.range, (uint32_t)s_win) <= 64 * a.n ? (s0 + 5 < 31 ? s0 + 5 : 31) : s_win;
        const int mine = s_lo + (int)blockIdx.x;
        const uint32_t first = block_sums(s, tune_entries<D>(lo, hi, ok, (uint32_t)min(mine, 31)), 0u).x;
        // Coarser ones up to a single cell, on grids in proportion to the boxes, where
        // none of those qualifies (boxes too sparse in their range, or a few huge ones
        // among them; the coarsest decides, for cells and entries only fall, and a block
        // whose own size does need not ask it), and where s0 + 3 makes more cells than
        // that: on 300 000 boxes of side 2048 in a range of 2^24 it makes 2^30, where
        // 2^18 are a few microseconds' work. (Small queries, which run in one launch on
        // coarse grids of their own if they can, stay with s0 + 3.)
        const bool none = !(mine <= s_far && tune_grid<D>(a.range, (uint32_t)mine) <= a.max_cells && first <= 64u * m) &&
                          (tune_grid<D>(a.range, (uint32_t)s_far) > a.max_cells ||
                           block_sums(s, tune_entries<D>(lo, hi, ok, (uint32_t)s_far), 0u).x > 64u * m);
        const bool coarser = none || (a.n > kFusedMaxBoxes && tune_grid<D>(a.range, (uint32_t)s_win) > 64 * a.n);
        const int s_one = a.range <= 1u ? 0 : min(32 - __clz((int)(a.range - 1u)), 31);  // the first of a single cell
        const int last = coarser ? max(s_one, s_far) : s_far;
        const uint64_t far = mn64(a.max_cells, a.n * 64 > 4096 ? a.n * 64 : 4096);
        unsigned long long best = ~0ull;  // (thread 0: the bits of the least cost, which are in its order; the finest on a tie)
        for (int w = mine; w <= last && m > 0; w += (int)kTuneBlocks) {
            if (tune_grid<D>(a.range, (uint32_t)w) > (w > s_far ? far : a.max_cells)) continue;
            const uint32_t e = w == mine ? first : block_sums(s, tune_entries<D>(lo, hi, ok, (uint32_t)w), 0u).x;
            if (e > 64u * m) continue;
            const uint32_t pairs = tune_pairs<D>(s, table, lo, ok, a.range, (uint32_t)w);
            if (t == 0) {
                double E;
                const unsigned long long cost = (unsigned long long)__double_as_longlong(
                    tune_cost_query(tune_grid<D>(a.range, (uint32_t)w), e, pairs, m, a.n, a.bip, E));
                if (cost < best) {
                    best = cost;
                    shift = (uint32_t)w;
                    est = E;
                }
            }
        }
        if (t == 0) {
            unsigned long long* mine3 = a.scratch + 1 + 3 * blockIdx.x;
            mine3[0] = best;
            mine3[1] = (unsigned long long)__double_as_longlong(est);
            mine3[2] = shift;
            shift = kTuneShift;
            __threadfence();
            if (atomicAdd(a.scratch, 1ull) == gridDim.x - 1) {
                __threadfence();
                unsigned long long all[kTuneBlocks][3];
#pragma unroll
                for (uint32_t b = 0; b < kTuneBlocks; b++)
#pragma unroll
                    for (int k = 0; k < 3; k++) all[b][k] = __ldcg(a.scratch + 1 + 3 * b + k);
                best = ~0ull;
#pragma unroll
                for (uint32_t b = 0; b < kTuneBlocks; b++) {
                    if (all[b][0] < best || (all[b][0] == best && (uint32_t)all[b][2] < shift)) {
                        best = all[b][0];
                        est = __longlong_as_double((long long)all[b][1]);
                        shift = (uint32_t)all[b][2];
                    }
                }
                if (best == ~0ull) {  // the coarsest grid that is not a single cell
                    shift = 31;
                    while (shift > 0 && nrc_dev(a.range, (int)shift - 1) <= 1) shift--;
                    est = (double)a.n;
                }
            }
        }
        if (t != 0 || shift == kTuneShift) return;  // (another block writes the tables)
        if (a.least) shift = max(shift, __ldcg(a.least));
    }
    if (t != 0) return;
    if (a.shift == kTuneShift) a.scratch[0] = 0;
    const uint32_t nrc = nrc_dev(a.range, (int)shift);
    const uint64_t C = D == 3 ? (uint64_t)nrc * nrc * nrc : (uint64_t)nrc * nrc;
    const uint32_t n_scenes = a.bip ? 2u : 1u;
    a.scenes[0] = Scene{0u, (uint32_t)(a.bip ? a.n_red : a.n), shift, nrc, 0ull, a.range, 0u};
    a.box_off[0] = 0u;
    a.box_off[n_scenes] = (uint32_t)a.n;
    if (a.bip) {
        a.scenes[1] = Scene{(uint32_t)a.n_red, (uint32_t)(a.n - a.n_red), shift, nrc, 0ull, a.range, 0u};
        a.box_off[1] = (uint32_t)a.n_red;
    }
    const bool room = C <= a.room_cells;
    *a.dims = RunDims{room ? a.n : 0ull, room ? C : 0ull, n_scenes, shift >= kOpenShift ? 1u : 0u};
    Ctr c{};
    if (!room) c.err = kErrGridRoom;
    c.cells = C;
    c.shift = shift;
    c.est_entries = (unsigned long long)fmin(est, 1e18);
    c.stamp[kStampStart] = began;
    *p.ctr = c;
}

// ---------------------------------------------------------------------------
// count / scatter: one thread per box, boxes staged through shared memory with
// 16-byte vector loads; the cells of the 32 boxes of a warp are enumerated
// cooperatively (lane q handles cell q of the warp's concatenated cell list),
// so a box spanning many cells does not stall its warp.
// ---------------------------------------------------------------------------
constexpr int kBoxThreads = 256;

__device__ __forceinline__ void copy_words(const uint32_t* src, uint32_t* dst, uint32_t nwords) {
    if ((((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) && (nwords & 3u) == 0) {
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
        uint4* d4 = reinterpret_cast<uint4*>(dst);
        for (uint32_t k = threadIdx.x; k < nwords / 4; k += blockDim.x) d4[k] = __ldg(s4 + k);
    } else {
        for (uint32_t k = threadIdx.x; k < nwords; k += blockDim.x) dst[k] = __ldg(src + k);
    }
}

// a tile of boxes into shared memory: boxes [0, split) at red, the rest at blue
template <int D>
__device__ __forceinline__ void stage_two(const uint32_t* red, const uint32_t* blue, uint64_t split, uint64_t b0,
                                          uint32_t nb, uint32_t* sbox) {
    constexpr uint32_t W = 2 * D + 1;
    if (b0 + nb <= split || b0 >= split) {
        copy_words(b0 < split ? red + b0 * W : blue + (b0 - split) * W, sbox, nb * W);
    } else {  // the tile straddles red and blue
        const uint64_t sw = split * W;
        for (uint32_t k = threadIdx.x; k < nb * W; k += blockDim.x) {
            const uint64_t gw = b0 * W + k;
            sbox[k] = gw < sw ? __ldg(red + gw) : __ldg(blue + (gw - sw));
        }
    }
}

template <int D>
__device__ __forceinline__ void stage_boxes(const Params& p, uint64_t b0, uint32_t nb, uint32_t* sbox) {
    if (p.blue) stage_two<D>(p.boxes, p.blue, p.split, b0, nb, sbox);
    else copy_words(p.boxes + b0 * (2 * D + 1), sbox, nb * (2 * D + 1));
}

// the coordinates of box id, red and blue in one array or two
template <int D>
__device__ __forceinline__ const uint32_t* box_row(const uint32_t* boxes, const uint32_t* blue, uint32_t split, uint32_t id) {
    return blue && id >= split ? blue + (uint64_t)(id - split) * (2 * D + 1) : boxes + (uint64_t)id * (2 * D + 1);
}

// the count's upload: a tile of boxes from page-locked host memory into
// shared memory (the host link is the bound, so the count's own work hides
// under it), then on to the device copy
template <int D>
__device__ __forceinline__ void stage_upload(const Params& p, uint64_t b0, uint32_t nb, uint32_t* sbox) {
    constexpr uint32_t W = 2 * D + 1;
    stage_two<D>(p.up_red, p.up_blue, p.up_split, b0, nb, sbox);
    __syncthreads();
    uint32_t* dst = p.box_copy + b0 * W;
    if (((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) && ((nb * W) & 3u) == 0) {
        const uint4* s4 = reinterpret_cast<const uint4*>(sbox);
        uint4* d4 = reinterpret_cast<uint4*>(dst);
        for (uint32_t k = threadIdx.x; k < nb * W / 4; k += blockDim.x) d4[k] = s4[k];
    } else {
        for (uint32_t k = threadIdx.x; k < nb * W; k += blockDim.x) dst[k] = sbox[k];
    }
}

// n / d (d >= 1) by a multiply-high with the divisor's multiplier m =
// magic_of(d) = ceil(2^32 / d) (0 for d = 1): for n < 2^31 the estimate is
// exact or one too large, which one compare fixes
__device__ __forceinline__ uint32_t magic_of(uint32_t d) { return d > 1u ? 0xffffffffu / d + 1u : 0u; }
__device__ __forceinline__ uint32_t div_magic(uint32_t n, uint32_t d, uint32_t m) {
    if (m == 0u) return n;
    const uint32_t q = __umulhi(n, m);
    return q * d > n ? q - 1u : q;
}

// ---- entries -----------------------------------------------------------------
// An entry is 16 bytes: a word per axis with the box's part of the cell, then
// {start bits << 29 | box index}. Both corners are counted from the cell's
// first coordinate and scaled to 1..32765; a lower corner before the cell is 0
// and an upper one beyond it 32766, so for two boxes of the cell lower <= upper
// holds for the scaled corners whenever it holds for the real ones, and is the
// same unless both fall into the cell and are scaled to one value (cells of
// 2^kOpenShift or wider only). The high half of the word is the lower corner,
// the low half 32767 minus the upper one: a row's lower corner plus a column's
// low half is at most 32767 iff that side of the boxes overlaps, and never
// carries out of 16 bits. An empty entry's first word, 32768 in the low half,
// overlaps nothing.
//
// The pair kernels read the entries of a cell one after the other and never
// the boxes (only to settle scaled corners that compare equal). With 4-byte
// entries that named the boxes, fetching them took 0.26 of the 0.42 ms of the
// medium-cell kernel on the clustered 4M-box scene, 0.29 of 0.39 ms on two
// million red and blue boxes and 0.69 of 0.94 ms on 512 scenes: a random
// 28-byte read per entry.
constexpr uint32_t kTermSpan = 32765u;
constexpr uint32_t kTermBeyond = 32767u - (kTermSpan + 1u);  // low half of a box that ends beyond the cell
constexpr uint32_t kTermEmpty = 32768u;
__device__ __forceinline__ uint4 entry_empty() { return make_uint4(kTermEmpty, 0u, 0u, 0u); }

// x of [0, 2^s) scaled: floor(x * 32765 / 2^s)
__device__ __forceinline__ uint32_t term_scale(uint32_t x, uint32_t s) {
    return __umulhi(x << (31u - s), 2u * kTermSpan);
}
__device__ __forceinline__ uint32_t term_word(uint32_t lo, uint32_t hi) {
    return ((lo + 1u) << 16) | (32766u - hi);
}
// a box's word in one of its cells, from that of a cell it lies in whole
__device__ __forceinline__ uint32_t term_cut(uint32_t w, bool starts, bool ends) {
    return (starts ? w & 0xffff0000u : 0u) | (ends ? w & 0xffffu : kTermBeyond);
}

// a box's cells: cnt of them, sx along x and sy along y, from cell `base` of a
// grid of nrc cells per axis; none of an invalid box
struct BoxCells {
    uint32_t cnt = 0, sx = 1, sy = 1, nrc = 0;
    uint64_t base = 0;
};
// b: the box's row in shared memory (TERMS: it becomes the box's terms, one
// word per axis); REPORT: an invalid box is counted
template <int D, bool TERMS, bool REPORT>
__device__ __forceinline__ BoxCells box_cells(const Params& p, uint32_t* b, uint64_t gi) {
    BoxCells c;
    const Scene sc = p.scenes[find_scene(p, gi)];
    uint32_t err = 0;
#pragma unroll
    for (int d = 0; d < D; d++) {
        if (b[2 * d] >= sc.range || b[2 * d + 1] >= sc.range) err |= kErrRange;
        if (b[2 * d] > b[2 * d + 1]) err |= kErrInverted;
    }
    if (b[2 * D] != (uint32_t)(gi - sc.box_off)) err |= kErrRid;
    if (gi > kIdMask) err |= kErrIndex;
    if (!err) {
        const uint32_t sh = sc.shift;
        const uint32_t lo0 = b[0] >> sh, lo1 = b[2] >> sh, lo2 = D == 3 ? (b[4] >> sh) : 0u;
        const uint32_t sx = (b[1] >> sh) - lo0 + 1, sy = (b[3] >> sh) - lo1 + 1;
        const uint32_t sz = D == 3 ? (b[5] >> sh) - lo2 + 1 : 1u;
        const uint64_t c64 = (uint64_t)sx * sy * sz;
        if (c64 >= (1ull << 26)) {
            err |= kErrCellOvf;
        } else {
            c.cnt = (uint32_t)c64;
            c.sx = sx;
            c.sy = sy;
            c.nrc = sc.nrc;
            c.base = sc.cell_off + ((uint64_t)lo2 * c.nrc + lo1) * c.nrc + lo0;
            if (TERMS) {
                const uint32_t low = (1u << sh) - 1u;
#pragma unroll
                for (int d = 0; d < D; d++)
                    b[d] = term_word(term_scale(b[2 * d] & low, sh), term_scale(b[2 * d + 1] & low, sh));
            }
        }
    }
    if (err && REPORT) {
        atomicOr(&p.ctr->err, err);
        atomicAdd(&p.ctr->bad, 1u);
    }
    return c;
}

// (scatter: the boxes' rows in sbox are overwritten)
template <int D, bool SCATTER, bool MERGED>
__device__ __forceinline__ void enumerate_cells(const Params& p, uint32_t* sbox, uint64_t b0, uint32_t nb) {
    constexpr uint32_t W = 2 * D + 1;
    const uint32_t t = threadIdx.x, lane = t & 31u;
    BoxCells c;
    if (t < nb) c = box_cells<D, SCATTER && !MERGED, !SCATTER>(p, sbox + t * W, b0 + t);
    const uint32_t cnt = c.cnt, sx = c.sx, sy = c.sy, nrc = c.nrc;
    const uint64_t base = c.base;
    if (SCATTER) __syncwarp();
    const uint32_t incl = warp_incl_scan(cnt);
    const uint32_t total = __shfl_sync(FULL_MASK, incl, 31);
    const uint32_t excl = incl - cnt;
    const uint64_t wbox0 = b0 + (t & ~31u);
    const uint32_t mx = magic_of(sx), my = magic_of(sy);  // one division per box, none per cell
    for (uint32_t q0 = 0; q0 < total; q0 += 32) {
        const uint32_t q = q0 + lane;
        uint32_t o = 0;  // owner lane: number of lanes whose inclusive count <= q
#pragma unroll
        for (uint32_t step = 16; step; step >>= 1) {
            const uint32_t v = __shfl_sync(FULL_MASK, incl, o + step - 1);
            if (v <= q) o += step;
        }
        const uint32_t o_excl = __shfl_sync(FULL_MASK, excl, o);
        const uint32_t o_sx = __shfl_sync(FULL_MASK, sx, o);
        const uint32_t o_sy = __shfl_sync(FULL_MASK, sy, o);
        const uint32_t o_nrc = __shfl_sync(FULL_MASK, nrc, o);
        const uint64_t o_base = __shfl_sync(FULL_MASK, base, o);
        const uint32_t o_mx = __shfl_sync(FULL_MASK, mx, o);
        const uint32_t o_my = __shfl_sync(FULL_MASK, my, o);
        const uint32_t o_cnt = SCATTER ? __shfl_sync(FULL_MASK, cnt, o) : 0u;
        if (q < total) {
            const uint32_t lq = q - o_excl;  // < 2^26
            const uint32_t rr = div_magic(lq, o_sx, o_mx), i = lq - rr * o_sx;
            const uint32_t k = div_magic(rr, o_sy, o_my), j = rr - k * o_sy;
            uint64_t gid = o_base + ((uint64_t)k * o_nrc + j) * o_nrc + i;
            uint32_t f = (i == 0 ? 1u : 0u) | (j == 0 ? 2u : 0u) | ((D == 2 || k == 0) ? 4u : 0u);
            bool take = true;
            uint4 rec = make_uint4(0u, 0u, 0u, 0u);
            const uint32_t* ob = sbox + ((t & ~31u) + o) * W;
            if constexpr (SCATTER && !MERGED) {
                rec.x = term_cut(ob[0], i == 0, i + 1 == o_sx);
                rec.y = term_cut(ob[1], j == 0, j + 1 == o_sy);
                // (the last layer: its cells are the last sx*sy)
                if (D == 3) rec.z = term_cut(ob[2], k == 0, lq + o_sx * o_sy >= o_cnt);
            }
            if (MERGED) {
                // merged mode: a cell of a merged block stands for the block's
                // root, and a box enters the block once, at the minimum corner of
                // (box range x block) -- the first-visit rule of d_postcounting,
                // pbig.cu:223-318; "starts here" is then per axis "the box's
                // first cell is inside the block"
                const uint32_t m = p.merged[gid];
                if (m != kUnmerged) {
                    const uint64_t nr = o_nrc;
                    const uint32_t ci = (uint32_t)(gid % nr), cj = (uint32_t)((gid / nr) % nr);
                    const uint32_t ck = D == 3 ? (uint32_t)(gid / (nr * nr)) : 0u;
                    const uint32_t lx = ci - i, ly = cj - j, lz = ck - k;
                    const uint32_t rx = (uint32_t)(m % nr), ry = (uint32_t)((m / nr) % nr);
                    const uint32_t rz = D == 3 ? (uint32_t)(m / (nr * nr)) : 0u;
                    take = ci == max(lx, rx) && cj == max(ly, ry) && ck == max(lz, rz);
                    gid = m;
                    f = (lx >= rx ? 1u : 0u) | (ly >= ry ? 2u : 0u) | ((D == 2 || lz >= rz) ? 4u : 0u);
                }
                if (SCATTER && take) {  // the box's part of the block (or of an unmerged cell)
                    const uint64_t nr = o_nrc, ext = m != kUnmerged ? p.merged_ext[m] : (1ull << 42 | 1ull << 21 | 1ull);
                    const uint32_t sh = p.scenes[0].shift;  // (one grid in merged mode)
                    uint32_t root[3] = {(uint32_t)(gid % nr), (uint32_t)((gid / nr) % nr), (uint32_t)(gid / (nr * nr))};
                    uint32_t w[3] = {0u, 0u, 0u};
#pragma unroll
                    for (int d = 0; d < D; d++) {
                        const uint64_t len = (ext >> (21 * d) & 0x1fffffull) << sh, at = (uint64_t)root[d] << sh;
                        const uint64_t lo = ob[2 * d] - at, hi = ob[2 * d + 1] - at;  // (lo wraps where it is cut)
                        w[d] = term_cut(term_word((uint32_t)((lo < len ? lo : 0u) * kTermSpan / len),
                                                  (uint32_t)((hi < len ? hi : 0u) * kTermSpan / len)),
                                        lo < len, hi < len);
                    }
                    rec.x = w[0];
                    rec.y = w[1];
                    rec.z = w[2];
                }
            }
            if (!take) {
            } else if (SCATTER) {
                // after the scan a cell's counter holds its end: counting it
                // down hands out the cell's slots (and leaves its start)
                const uint64_t pos = (uint64_t)(atomicSub(&p.counts[gid], 1u) - 1u);
                rec.w = (f << kIdBits) | (uint32_t)(wbox0 + o);
                if (pos < p.entry_cap) p.entries[pos] = rec;
                else atomicOr(&p.ctr->err, kErrEntryOvf);
            } else {
                atomicAdd(&p.counts[gid], 1u);
            }
        }
    }
}

// counts = 0 before a pass (the scatter leaves every cell's start there), and
// the scan's tile records
__global__ void k_zero_counts(Params pin) {
    chain_wait();
    const Params p = resolve(pin);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.ctr->stamp[kStampCount] = now_ns();
        if (p.ctr->stamp[kStampStart] == 0ull) p.ctr->stamp[kStampStart] = p.ctr->stamp[kStampCount];
    }
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n4 = p.ncells / 4;
    uint4* c4 = reinterpret_cast<uint4*>(p.counts);
    for (uint64_t i = t; i < n4; i += stride) c4[i] = make_uint4(0, 0, 0, 0);
    for (uint64_t i = 4 * n4 + t; i < p.ncells; i += stride) p.counts[i] = 0;
    const uint64_t r4 = scan_tiles(p.ncells) * (kTileRecBytes / 16);
    uint4* s4 = reinterpret_cast<uint4*>(p.tile_state);
    for (uint64_t i = t; i < r4; i += stride) s4[i] = make_uint4(0, 0, 0, 0);
}

// tiles of kBoxThreads boxes: blk, blk + nblk, ...
template <int D, bool SCATTER, bool MERGED>
__device__ __forceinline__ void box_pass(const Params& p, uint32_t* sbox, uint64_t blk, uint64_t nblk) {
    for (uint64_t b0 = blk * kBoxThreads; b0 < p.nboxes; b0 += nblk * kBoxThreads) {
        const uint32_t nb = (uint32_t)mn64(kBoxThreads, p.nboxes - b0);
        if (!SCATTER && p.box_copy) stage_upload<D>(p, b0, nb, sbox);
        else stage_boxes<D>(p, b0, nb, sbox);
        __syncthreads();
        enumerate_cells<D, SCATTER, MERGED>(p, sbox, b0, nb);
        __syncthreads();
    }
}

template <int D, bool MERGED>
__global__ void __launch_bounds__(kBoxThreads) k_count(Params pin) {
    __shared__ __align__(16) uint32_t sbox[kBoxThreads * (2 * D + 1)];
    chain_wait();
    box_pass<D, false, MERGED>(resolve(pin), sbox, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// expand: cells larger than kBigMax get tile tasks {cell, row tile r, column
// tiles [x0,x1)} with 32-box tiles, x >= r, at most 8 column tiles a task.
// ---------------------------------------------------------------------------
constexpr uint32_t kTaskCols = 8;

// the size of a work list (kNumLists: the tile tasks) that a pass reads.
// FRESH: one-launch queries, where the counters change while the kernel runs;
// they are read past L1 once, together, before the passes (a read in each pass
// was half a microsecond each time). The separate kernels read them plainly.
template <bool FRESH>
__device__ __forceinline__ uint32_t list_size(const Params& p, int k) {
    if (FRESH) return p.list_sizes[k];
    return k < kNumLists ? p.ctr->n_list[k] : p.ctr->need_tasks;
}

// tile tasks of the last k row tiles of a cell: ceil(i / kTaskCols), i = 1 .. k
__device__ __forceinline__ uint32_t tile_tasks(uint32_t k) {
    const uint32_t a = k / kTaskCols, b = k % kTaskCols;
    return (a + 1) * (a * (kTaskCols / 2) + b);
}
constexpr uint32_t kMostRows = 1u << 17;  // (2^30 tasks; cells of more boxes ask for more than there can be)

// huge cells i0, i0 + stride, ..., a warp each and its lanes a row tile: a
// thread to a cell took 0.6 ms to write the 25 000 tasks of one of 20 000 boxes,
// 1.06 ms the query; with a warp it takes 0.51.
// (pl: the kernel's own parameters, as in scan_chunk)
__device__ __forceinline__ void expand_cells(const Params& p, const Params& pl, uint32_t huge, uint32_t i0, uint32_t stride) {
    const uint32_t nh = (uint32_t)mn64(huge, pl.list_cap[kListHuge]);
    for (uint32_t i = i0; i < nh; i += stride) {
        const uint2 sn = p.lists[pl.list_off[kListHuge] + i];
        const uint32_t R = (sn.y + 31) >> 5, cap = (uint32_t)mn64(p.task_cap, 0x7fffffffu);
        const uint32_t cnt = R <= kMostRows ? tile_tasks(R) : 0x7fffffffu;
        uint32_t b = 0;
        if (lane_id() == 0) {
            b = atomicAdd(&p.ctr->need_tasks, cnt);
            if ((uint64_t)b + cnt > cap) atomicOr(&p.ctr->err, kErrTaskOvf);
        }
        b = __shfl_sync(FULL_MASK, b, 0);
        if (b >= cap || R > kMostRows) continue;
        for (uint32_t r = lane_id(); r < R; r += 32) {
            uint32_t k = b + cnt - tile_tasks(R - r);
            for (uint32_t x0 = r; x0 < R && k < cap; x0 += kTaskCols, k++) p.tasks[k] = make_uint4(sn.x, sn.y, r, x0);
        }
    }
}

template <int D, bool MERGED>
__global__ void __launch_bounds__(kBoxThreads) k_scatter(Params pin) {
    __shared__ __align__(16) uint32_t sbox[kBoxThreads * (2 * D + 1)];
    chain_wait();
    stamp(pin, kStampScatter);
    box_pass<D, true, MERGED>(resolve(pin), sbox, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// scan: counts -> cell starts and the work lists of the pair kernels, in
// two launches without inter-block waits.
//
// A tile is 4096 cells, a chunk 512 of them; every warp works on whole
// chunks with no block barrier, so the loads of all resident warps are in
// flight together. Tile records (64 bytes, zeroed before the scan) collect
// per-chunk entry sums and per-tile totals.
//
//   k_scan_reduce  chunk entry total (stored per chunk, added to the tile);
//                  two chunks per warp iteration, so eight 16-byte loads
//                  per lane are in flight together. The last block to
//                  finish turns the tile entry totals into exclusive
//                  prefixes; the entry total goes to the counters.
//   k_scan_cells   the same chunks again: starts from the tile prefix, the
//                  tile's earlier chunks and a warp scan; every cell of two
//                  or more boxes goes to its work list, a chunk reserving
//                  its places with one atomic per list (list order is free);
//                  each warp sums the work statistics of its cells (pair
//                  tests, numCompPairs, 256-row jobs, largest cell) and adds
//                  them to the counters once.
//
// Lane l of a warp owns the 4 cells at 4l of each of the chunk's 4 rows of
// 128 cells, so each 16-byte load or store of a warp covers 512 contiguous
// bytes. The work list of a cell of n >= 2 boxes is 2..4, 5..8, 9..16,
// 17..32, 33..128, 129..512 or more boxes; per-lane list counts travel
// packed in 10-bit fields (a chunk has at most 512 cells per list).
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanPerThread = 16;
constexpr int kScanChunk = 32 * kScanPerThread;              // cells per warp item
constexpr int kScanChunks = 8;                               // chunks per tile
constexpr int kScanTile = kScanChunk * kScanChunks;

struct TileRec {                         // 64 bytes per tile
    unsigned long long sum;              // entries; exclusive prefix after k_scan_reduce
    uint32_t chunk[kScanChunks];         // entries per chunk
    uint32_t pad[6];
};
static_assert(sizeof(TileRec) == kTileRecBytes && kScanTile == kTileCells, "tile record layout");

static_assert(kMedMax == 128 && kBigMax == 512, "list bounds are powers of two (the class map's buckets)");
// the work list of a cell of n >= 2 boxes under the class map
__device__ __forceinline__ uint32_t class_of(uint32_t n, unsigned long long map) {
    const uint32_t lg = 32u - __clz(n - 1u);  // ceil(log2 n) for n >= 2
    return (uint32_t)(map >> (4u * min(lg, 15u))) & 15u;
}

__device__ __forceinline__ unsigned long long warp_incl_scan64(unsigned long long v) {
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(FULL_MASK, v, o);
        if (lane_id() >= o) v += t;
    }
    return v;
}

// cell r*128 + 4*lane of chunk `chunk`, chunks of Q rows of 128 cells
template <int Q = 4>
__device__ __forceinline__ uint64_t chunk_cell(uint64_t chunk, int r) {
    return chunk * (128u * Q) + (uint64_t)r * 128 + lane_id() * 4;
}

// the 4*Q counts of this lane's cells of the chunk (zeros past the end);
// PAST_L1: counts written by other blocks of the same launch
template <int Q = 4, bool PAST_L1 = false>
__device__ __forceinline__ void scan_load(const Params& p, uint64_t chunk, uint32_t (&v)[4 * Q]) {
    const bool full = chunk * (128u * Q) + 128u * Q <= p.ncells;
#pragma unroll
    for (int r = 0; r < Q; r++) {
        const uint64_t c = chunk_cell<Q>(chunk, r);
        if (full) {
            const uint4* a = reinterpret_cast<const uint4*>(p.counts + c);
            const uint4 q = PAST_L1 ? __ldcg(a) : *a;
            v[4 * r] = q.x; v[4 * r + 1] = q.y; v[4 * r + 2] = q.z; v[4 * r + 3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[4 * r + k] = c + k < p.ncells ? (PAST_L1 ? __ldcg(p.counts + c + k) : p.counts[c + k]) : 0u;
        }
    }
}

__device__ __forceinline__ void reduce_chunk(TileRec* rec, uint64_t ch, const uint32_t v[kScanPerThread]) {
    const uint32_t lane = lane_id();
    uint32_t lsum = 0;  // < 2^32 while the entry total is
#pragma unroll
    for (int k = 0; k < kScanPerThread; k++) lsum += v[k];
    lsum = __reduce_add_sync(FULL_MASK, lsum);
    TileRec& r = rec[ch / kScanChunks];
    if (lane == 0) {
        r.chunk[ch % kScanChunks] = lsum;
        if (lsum) atomicAdd(&r.sum, (unsigned long long)lsum);
    }
}

// tile entry totals -> exclusive prefixes; the entry total goes to the
// counters. Run by one block of kReduceThreads threads, kPrefixPer tiles per
// thread per round (4096 tiles in two rounds).
constexpr int kReduceThreads = kScanThreads;
constexpr int kPrefixPer = 8;
__device__ __forceinline__ void scan_prefix_block(const Params& p) {
    __shared__ unsigned long long s_part[kReduceThreads / 32];
    __shared__ unsigned long long s_carry;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint64_t tiles = (p.ncells + kScanTile - 1) / kScanTile;
    TileRec* rec = reinterpret_cast<TileRec*>(p.tile_state);
    if (t == 0) s_carry = 0;
    // rounds of kPrefixPer tiles per thread: all loads of a round in flight
    // together; the records were written through L2 by other blocks (read
    // past L1)
    for (uint64_t r0 = 0; r0 < tiles; r0 += kPrefixPer * kReduceThreads) {
        unsigned long long x[kPrefixPer], sx = 0;
#pragma unroll
        for (int k = 0; k < kPrefixPer; k++) {
            const uint64_t i = r0 + kPrefixPer * (uint64_t)t + k;
            x[k] = i < tiles ? __ldcg(&rec[i].sum) : 0ull;
            sx += x[k];
        }
        const unsigned long long ix = warp_incl_scan64(sx);
        if (lane == 31) s_part[warp] = ix;
        __syncthreads();
        unsigned long long wo = s_carry, tot = 0;
        for (int w = 0; w < kReduceThreads / 32; w++) {
            const unsigned long long a = s_part[w];
            if (w < (int)warp) wo += a;
            tot += a;
        }
        unsigned long long run = wo + (ix - sx);
#pragma unroll
        for (int k = 0; k < kPrefixPer; k++) {
            const uint64_t i = r0 + kPrefixPer * (uint64_t)t + k;
            if (i < tiles) rec[i].sum = run;
            run += x[k];
        }
        __syncthreads();
        if (t == 0) s_carry += tot;
        __syncthreads();
    }
    if (t == 0) {
        p.ctr->entries = s_carry;
        if (s_carry >= (1ull << 32)) atomicOr(&p.ctr->err, kErrEntryOvf);
    }
}

// the last block to finish (a ticket taken after a fence, no waiting) runs
// the tile prefix, so no separate launch is needed for it
__global__ void __launch_bounds__(kReduceThreads, 4) k_scan_reduce(Params pin) {
    __shared__ uint32_t s_last;
    chain_wait();
    const Params p = resolve(pin);
    stamp(p, kStampScan);
    const uint32_t warp = threadIdx.x >> 5;
    const uint64_t chunks = (p.ncells + kScanChunk - 1) / kScanChunk;
    TileRec* rec = reinterpret_cast<TileRec*>(p.tile_state);
    const uint64_t nw = (uint64_t)gridDim.x * (kReduceThreads / 32);
    for (uint64_t ch = 2 * ((uint64_t)blockIdx.x * (kReduceThreads / 32) + warp); ch < chunks; ch += 2 * nw) {
        uint32_t v[kScanPerThread], w[kScanPerThread];
        scan_load(p, ch, v);
        const bool two = ch + 1 < chunks;
        if (two) scan_load(p, ch + 1, w);
        reduce_chunk(rec, ch, v);
        if (two) reduce_chunk(rec, ch + 1, w);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&p.ctr->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (s_last == 0u) return;
    __threadfence();
    scan_prefix_block(p);
    if (threadIdx.x == 0) p.ctr->ticket = 0;  // the next scan needs no reset
}

// ---- bulk asynchronous copies (global -> shared) completing on an mbarrier
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// arm the barrier for `bytes` and copy them (16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned long long* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the phase of parity `parity`; false when it gave up
constexpr uint32_t kBulkWaitLimit = 1u << 20;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity) {
    for (uint32_t i = 0; i < kBulkWaitLimit; i++)
        if (mbar_test(bar, parity)) return true;
    return false;
}

// the cells of chunk ch (counts v; `base` entries before the chunk): each
// non-empty cell's end (start + count) into its counter (an empty cell's is
// never read: the scatter and the work lists touch cells with entries only,
// and skipping those stores, most of a fine grid, saves the scatter the
// write-backs of their lines), each cell of two or more boxes into its work
// list (one atomic per list and chunk), and the work statistics into ws
struct ScanStats {
    unsigned long long tests = 0;
    uint32_t half = 0, jobs = 0, max = 0;
};

// (pl: the kernel's own parameters, for the list tables: indexing a local
// copy of Params with a run-time list number would move it to local memory)
template <int Q = 4>
__device__ __forceinline__ void scan_chunk(const Params& p, const Params& pl, uint64_t ch, bool full,
                                           const uint32_t (&v)[4 * Q], unsigned long long base, ScanStats& ws) {
    constexpr int kPer = 4 * Q;
    const uint32_t lane = lane_id();
    const unsigned long long cmap = p.class_map ? p.class_map : kClassMapDefault;
    uint32_t big = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) big |= v[k] >> 1;
    // row scans: the cells of row q before this lane's, and rows < q whole
    uint32_t st[kPer];
    unsigned long long wtot = 0;
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const uint32_t rs = v[4 * q] + v[4 * q + 1] + v[4 * q + 2] + v[4 * q + 3];
        const uint32_t inc = warp_incl_scan(rs);  // < 2^32 while the entry total is
        unsigned long long run = base + wtot + (inc - rs);
        wtot += __shfl_sync(FULL_MASK, inc, 31);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            st[4 * q + k] = (uint32_t)run;
            run += v[4 * q + k];
        }
        // a non-empty cell's counter becomes its end (start + count), in place
        const uint64_t c = chunk_cell<Q>(ch, q);
        if (full) {
            if (rs != 0u)
                *reinterpret_cast<uint4*>(p.counts + c) = make_uint4(
                    st[4 * q] + v[4 * q], st[4 * q + 1] + v[4 * q + 1], st[4 * q + 2] + v[4 * q + 2], st[4 * q + 3] + v[4 * q + 3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (c + k < p.ncells && v[4 * q + k] != 0u) p.counts[c + k] = st[4 * q + k] + v[4 * q + k];
        }
    }
    if (__any_sync(FULL_MASK, big != 0)) {
        // per-lane list counts: lists 0..5 in 10-bit fields of pk, list 6 in pk6
        unsigned long long pk = 0;
        uint32_t pk6 = 0;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            if (v[k] >= 2u) {
                const uint32_t c = class_of(v[k], cmap);
                if (c < 6u) pk += 1ull << (10u * c);
                else pk6 += 1u;
            }
        }
        const unsigned long long pinc = warp_incl_scan64(pk);
        const uint32_t p6inc = warp_incl_scan(pk6);
        unsigned long long pk_excl = pinc - pk;
        uint32_t pk6_excl = p6inc - pk6;
        // lane c < 7: this chunk's first place in list c
        const unsigned long long ptot = __shfl_sync(FULL_MASK, pinc, 31);
        const uint32_t p6tot = __shfl_sync(FULL_MASK, p6inc, 31);
        uint32_t lbase = 0;
        if (lane < kNumLists) {
            const uint32_t x = lane < 6u ? (uint32_t)(ptot >> (10u * lane)) & 1023u : p6tot;
            if (x) lbase = atomicAdd(&p.ctr->n_list[lane], x);
        }
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const uint32_t c = v[k] >= 2u ? class_of(v[k], cmap) : 0u;
            const uint32_t b = __shfl_sync(FULL_MASK, lbase, c);
            if (v[k] >= 2u) {
                uint32_t rk;
                if (c < 6u) {
                    rk = (uint32_t)(pk_excl >> (10u * c)) & 1023u;
                    pk_excl += 1ull << (10u * c);
                } else {
                    rk = pk6_excl++;
                }
                const uint64_t idx = (uint64_t)b + rk;
                const uint32_t key = p.records ? (uint32_t)(chunk_cell<Q>(ch, k >> 2) + (k & 3)) : st[k];
                if (idx < pl.list_cap[c]) p.lists[pl.list_off[c] + idx] = make_uint2(key, v[k]);
                ws.tests += (unsigned long long)v[k] * (v[k] - 1u) / 2u;
                ws.half += v[k] >> 1;  // n*n/2 = n(n-1)/2 + n/2, rounded down
                ws.jobs += (v[k] + 255u) >> 8;
                ws.max = max(ws.max, v[k]);
            }
        }
    }
}

// the work statistics of a warp's cells (pair tests, and the reference's
// numCompPairs, 256-row jobs and largest cell) into the counters
__device__ __forceinline__ void scan_stats_flush(const Params& p, const ScanStats& st) {
    const unsigned long long tests = warp_sum_u64(st.tests);
    const unsigned long long half = warp_sum_u64(st.half), jobs = warp_sum_u64(st.jobs);
    const uint32_t mx = __reduce_max_sync(FULL_MASK, st.max);
    if (lane_id() == 0 && mx) {
        atomicAdd(&p.ctr->tests, tests);
        atomicAdd(&p.ctr->comp_pairs, tests + half);
        atomicAdd(&p.ctr->jobs, jobs);
        atomicMax(&p.ctr->max_cell, mx);
    }
}

// k_scan_cells: each warp keeps its next chunk's counts in flight as a bulk
// copy into one of two shared-memory buffers while it works on the current
// one. A partial chunk (only the grid's last) is read with plain loads.
__global__ void __launch_bounds__(kScanThreads, 4) k_scan_cells(Params pin) {
    __shared__ __align__(128) uint32_t s_buf[kScanThreads / 32][2][kScanChunk];
    __shared__ __align__(8) unsigned long long s_bar[kScanThreads / 32][2];
    chain_wait();
    const Params p = resolve(pin);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint64_t chunks = (p.ncells + kScanChunk - 1) / kScanChunk;
    const uint64_t full_chunks = p.ncells / kScanChunk;
    const TileRec* rec = reinterpret_cast<const TileRec*>(p.tile_state);
    const uint64_t nw = (uint64_t)gridDim.x * (kScanThreads / 32);
    const uint64_t first = (uint64_t)blockIdx.x * (kScanThreads / 32) + warp;
    if (lane == 0) {
        mbar_init(&s_bar[warp][0], 1);
        mbar_init(&s_bar[warp][1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    auto issue = [&](uint64_t i) {  // chunk i of this warp into buffer i & 1
        const uint64_t ch = first + i * nw;
        if (lane == 0 && ch < full_chunks)
            bulk_load(s_buf[warp][i & 1], p.counts + ch * kScanChunk, kScanChunk * 4, &s_bar[warp][i & 1]);
    };
    issue(0);
    issue(1);
    ScanStats stats;
    for (uint64_t i = 0;; i++) {
        const uint64_t ch = first + i * nw;
        if (ch >= chunks) break;
        uint32_t v[kScanPerThread];
        if (ch < full_chunks) {
            if (!mbar_wait(&s_bar[warp][i & 1], (uint32_t)(i >> 1) & 1u)) {
                // give up: report, wait (bounded) for the copy still in flight, stop
                if (lane == 0) atomicOr(&p.ctr->err, kErrWait);
                mbar_wait(&s_bar[warp][i & 1], (uint32_t)(i >> 1) & 1u);
                if (first + (i + 1) * nw < full_chunks)
                    mbar_wait(&s_bar[warp][(i + 1) & 1], (uint32_t)((i + 1) >> 1) & 1u);
                return;
            }
            const uint32_t* b = s_buf[warp][i & 1];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint4 x = *reinterpret_cast<const uint4*>(b + q * 128 + lane * 4);
                v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
            }
            __syncwarp();
            // the buffer's reads are done: it can take the chunk after next
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(i + 2);
        } else {
            scan_load(p, ch, v);
        }
        const TileRec& r = rec[ch / kScanChunks];
        const uint32_t ci = (uint32_t)(ch % kScanChunks);
        // entries before this chunk: tile prefix + the tile's earlier chunks
        unsigned long long base = lane == 0 ? r.sum : 0ull;
        if (lane > 0 && lane <= ci) base = r.chunk[lane - 1];
        base = warp_sum_u64(base);
        scan_chunk(p, pin, ch, ch < full_chunks, v, base, stats);
    }
    scan_stats_flush(p, stats);
}

// ---------------------------------------------------------------------------
// pair test
//
// Three kernels:
//   k_pairs_small  cells of 2..32 boxes, 32/WG cells per warp item
//   k_pairs_med    cells of 33..kMedMax boxes, one cell per warp item,
//                  staged whole in the warp's shared memory
//   k_pairs_block  cells of kMedMax+1..kBigMax boxes staged whole by a
//                  team of four warps, and 32x32 tile tasks of larger cells
// Warps test and compact independently; each has a shared-memory buffer of
// pairs that it flushes to the pair array with one global reservation.
// Cells above the small ones are tested tile by tile (32 rows x 32 columns,
// "tiles" below).
// ---------------------------------------------------------------------------
constexpr int kPairThreads = 256;
constexpr int kPairWarps = kPairThreads / 32;
constexpr uint32_t kWarpOut = 256;          // per-warp output buffer (pairs), small cells
constexpr uint32_t kMedOut = 512;           // per-warp output buffer (pairs), other cells: above the
                                            // typical output of one emission step, so it rarely spills
constexpr uint32_t kSmallSlots = 64;        // per-warp staging, small cells (each cell twice in a row)


// ---- output: warp-private buffer ------------------------------------------
struct WarpOut {
    uint2* buf;    // candidate order: {row entry, column entry}, flag bits and all
    uint32_t n;    // warp-uniform fill
    uint32_t cap;  // buffer capacity (pairs)
    unsigned long long hits = 0;  // record mode: pairs written by this lane
};

// a buffered word as it is reported: the entries' start bits off, the
// smaller index first, the blue index counted from the first blue box.
// (Done here, by full warps, rather than in the emission loops, where on
// average half the lanes are idle.) Record words are written as they are.
template <bool BIP, bool REC>
__device__ __forceinline__ uint2 out_pair(const Params& p, uint2 w) {
    if (REC) return w;
    const uint32_t a = w.x & kIdMask, b = w.y & kIdMask;
    return make_uint2(min(a, b), BIP ? max(a, b) - p.split : max(a, b));
}

// copy n pairs (8-byte words) from shared memory to p.out[base, base + n):
// a lane stores 16-byte units laid on the destination's 128-byte lines, so a
// warp store covers whole lines and only the first and last line of a run
// are partial. The pair array may be page-locked host memory, where partial
// lines cost a large share of the link's write bandwidth.
template <bool BIP, bool REC>
__device__ __forceinline__ void store_run(const Params& p, unsigned long long base, const uint2* src, uint32_t n) {
    const uint32_t lane = lane_id();
    if (base + n > p.out_cap) {
        for (uint32_t k = lane; k < n; k += 32) {
            const unsigned long long g = base + k;
            if (g < p.out_cap) p.out[g] = out_pair<BIP, REC>(p, src[k]);
            else atomicOr(&p.ctr->err, kErrOutOvf);
        }
        return;
    }
    // pairs of base's line before base (the pair array is 8-byte aligned)
    const uint32_t lead = (uint32_t)(((reinterpret_cast<uintptr_t>(p.out) >> 3) + base) & 15u);
    const uint32_t units = (lead + n + 1) >> 1;
    uint2* dst = p.out + base;
    for (uint32_t u = lane; u < units; u += 32) {
        const int r = 2 * (int)u - (int)lead;  // first pair of the unit, relative to base
        if (r >= 0 && r + 1 < (int)n) {
            const uint2 a = out_pair<BIP, REC>(p, src[r]), b = out_pair<BIP, REC>(p, src[r + 1]);
            *reinterpret_cast<uint4*>(dst + r) = make_uint4(a.x, a.y, b.x, b.y);
        } else {
            if (r >= 0 && r < (int)n) dst[r] = out_pair<BIP, REC>(p, src[r]);
            if (r + 1 >= 0 && r + 1 < (int)n) dst[r + 1] = out_pair<BIP, REC>(p, src[r + 1]);
        }
    }
}

template <bool BIP, bool REC>
__device__ __forceinline__ void wflush(const Params& p, WarpOut& o) {
    if (o.n == 0) return;
    const uint32_t lane = lane_id();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&p.ctr->pairs, (unsigned long long)o.n);
    base = __shfl_sync(FULL_MASK, base, 0);
    __syncwarp();
    store_run<BIP, REC>(p, base, o.buf, o.n);
    __syncwarp();
    o.n = 0;
}

// compaction of the set bits of two masks (ranks from one warp scan of the
// per-lane popcounts) into the warp buffer, or straight to the pair array
// when the batch is larger than the buffer. pa, pb: the entry (or box index)
// of a bit's column; row: this lane's own.
template <bool BIP, class PA, class PB>
__device__ __forceinline__ void wemit(const Params& p, WarpOut& o, uint32_t ma, PA pa, uint32_t mb, PB pb,
                                      uint32_t row) {
    const uint32_t lane = lane_id();
    const uint32_t k = __popc(ma) + __popc(mb);
    const uint32_t incl = warp_incl_scan(k);
    const uint32_t total = __shfl_sync(FULL_MASK, incl, 31);
    if (total == 0) return;
    bool direct = false;
    unsigned long long gbase = 0;
    if (o.n + total > o.cap) {
        wflush<BIP, false>(p, o);
        if (total > o.cap) {
            direct = true;
            if (lane == 0) gbase = atomicAdd(&p.ctr->pairs, (unsigned long long)total);
            gbase = __shfl_sync(FULL_MASK, gbase, 0);
        }
    }
    uint32_t w = incl - k;
    if (!direct) {  // (warp-uniform: the loops below carry no per-pair branch)
        uint2* dst = o.buf + o.n + w;
        while (ma) {
            const uint32_t bit = 31u - __clz(ma);  // highest set bit first
            ma ^= 1u << bit;
            *dst++ = make_uint2(row, pa(bit));
        }
        while (mb) {
            const uint32_t bit = 31u - __clz(mb);
            mb ^= 1u << bit;
            *dst++ = make_uint2(row, pb(bit));
        }
        __syncwarp();
        o.n += total;
        return;
    }
    auto put = [&](uint32_t q) {
        const unsigned long long g = gbase + w;
        if (g < p.out_cap) p.out[g] = out_pair<BIP, false>(p, make_uint2(row, q));
        else atomicOr(&p.ctr->err, kErrOutOvf);
        w++;
    };
    while (ma) {
        const uint32_t bit = __ffs(ma) - 1;
        ma &= ma - 1;
        put(pa(bit));
    }
    while (mb) {
        const uint32_t bit = __ffs(mb) - 1;
        mb &= mb - 1;
        put(pb(bit));
    }
    __syncwarp();
}

// ---- record mode: the reference's Rice stream ------------------------------
// (RICE_COMPRESSION with 8-byte OTYPE: writer src/pbig/pbig.cu:788-920, reader
// src/pbig/decode.cc:38-131). A block is the header {UNUSED, cell id} followed
// by records; a record is one row box's hits in one 256-column tile of the
// cell: byte 0 row tile (row >> 8), byte 1 column tile, bytes 2-3 the row's
// index in its tile, bytes 4-5 the hit count, then one byte per hit (the
// column's index in its tile), padded to 8 bytes. Rows and columns are
// indices into the cell's entry list. Here a block is written per emission
// step (a cell may have several blocks, as the reference's cells of several
// jobs do), and a record covers one 32-column tile or the diagonal sweep.
constexpr unsigned long long kRiceUnused = 0x0fffff11ull;  // UNUSED, the block marker

__device__ __forceinline__ uint32_t rec_words(uint32_t hits) { return hits ? (6u + hits + 7u) >> 3 : 0u; }

// one record: `row` and the columns loc(bit) of the set bits of m (all in one
// 256-column tile) into dst, or nowhere when `keep` is false
template <class L>
__device__ __forceinline__ void rec_write(unsigned long long* dst, bool keep, uint32_t row, uint32_t m, L loc) {
    const uint32_t nh = __popc(m);
    unsigned long long word = (unsigned long long)(row >> 8) | ((unsigned long long)(loc(__ffs(m) - 1) >> 8) << 8) |
                              ((unsigned long long)(row & 255u) << 16) | ((unsigned long long)nh << 32);
    uint32_t byte = 6, wi = 0;
    while (m) {
        const uint32_t b = __ffs(m) - 1;
        m &= m - 1;
        word |= (unsigned long long)(loc(b) & 255u) << (8 * byte);
        if (++byte == 8) {
            if (keep) dst[wi] = word;
            wi++;
            word = 0;
            byte = 0;
        }
    }
    if (byte && keep) dst[wi] = word;
}

// warp step: lane records for ma (columns la) and mb (columns lb), one block
// header per cell before its first record; gmask: the lanes of this lane's
// cell (the whole warp, or a lane group of the small-cell kernel)
template <class LA, class LB>
__device__ __forceinline__ void remit(const Params& p, WarpOut& o, uint32_t ma, LA la, uint32_t mb, LB lb,
                                      uint32_t row, uint32_t gid, uint32_t gmask) {
    const uint32_t lane = lane_id();
    const uint32_t wa = rec_words(__popc(ma)), wb = rec_words(__popc(mb));
    const uint32_t gany = __ballot_sync(FULL_MASK, (wa | wb) != 0u) & gmask;
    const bool hdr = gany != 0u && lane == (uint32_t)(__ffs(gany) - 1);
    const uint32_t k = wa + wb + (hdr ? 2u : 0u);
    const uint32_t incl = warp_incl_scan(k);
    const uint32_t total = __shfl_sync(FULL_MASK, incl, 31);
    if (total == 0) return;
    o.hits += __popc(ma) + __popc(mb);
    bool direct = false;
    unsigned long long gbase = 0;
    if (o.n + total > o.cap) {
        wflush<false, true>(p, o);
        if (total > o.cap) {
            direct = true;
            if (lane == 0) gbase = atomicAdd(&p.ctr->pairs, (unsigned long long)total);
            gbase = __shfl_sync(FULL_MASK, gbase, 0);
        }
    }
    const bool keep = !direct || gbase + total <= p.out_cap;
    if (direct && !keep && lane == 0) atomicOr(&p.ctr->err, kErrOutOvf);
    unsigned long long* dst = direct ? reinterpret_cast<unsigned long long*>(p.out) + gbase
                                     : reinterpret_cast<unsigned long long*>(o.buf + o.n);
    uint32_t w = incl - k;
    if (hdr && keep) {
        dst[w] = kRiceUnused;
        dst[w + 1] = gid;
    }
    if (hdr) w += 2;
    if (wa) rec_write(dst + w, keep, row, ma, la);
    if (wb) rec_write(dst + w + wa, keep, row, mb, lb);
    __syncwarp();
    if (!direct) o.n += total;
}

// ---- small cells ------------------------------------------------------------
// lane group g (WG lanes) holds cell item*G+g of the class list, lane r its
// entry r; the circular half sweep runs inside the group: lane l < n tests
// its box against boxes l+1 .. l+floor(n/2) (mod n), lanes past n/2 one fewer
// when n is even (the BALANCE=1 sweep of d_matching, pbig.cu:804-825), so each
// unordered pair is tested once. The group's cell is staged twice in a row, so
// partner r+d needs no wrap. A row is its entry with each word's halves
// swapped: row plus column holds the two sides of an axis, so the boxes
// overlap iff the largest sums of both halves are below 32768 -- a u16x2
// add-max per axis. The
// reference-cell and red/blue rules are applied once per cell from ballots.

// the hits of `mask` (bit d: partner slot i + d) that hold on the whole coordinates
template <int D>
__device__ __noinline__ uint32_t small_exact(const uint32_t* boxes, const uint32_t* blue, uint32_t split,
                                             uint64_t nboxes, const uint4* s, uint32_t i, uint32_t mask) {
    uint32_t keep = 0;
    while (mask) {
        const uint32_t d = __ffs(mask) - 1;
        mask &= mask - 1;
        const uint32_t a = s[i].w & kIdMask, b = s[i + d].w & kIdMask;
        if (a >= nboxes || b >= nboxes) continue;  // cannot happen with a consistent grid
        const uint32_t *x = box_row<D>(boxes, blue, split, a), *y = box_row<D>(boxes, blue, split, b);
        bool hit = true;
#pragma unroll
        for (int k = 0; k < D; k++)
            hit = hit && __ldg(x + 2 * k) <= __ldg(y + 2 * k + 1) && __ldg(y + 2 * k) <= __ldg(x + 2 * k + 1);
        keep |= (hit ? 1u : 0u) << d;
    }
    return keep;
}

template <int D, int WG, bool BIP, bool REC, bool FRESH = false>
__device__ __forceinline__ void small_items(const Params& p, uint4* s, WarpOut& o, int list, uint64_t first,
                                            uint64_t stride) {
    constexpr uint32_t G = 32 / WG;
    const uint32_t lane = lane_id(), g = lane / WG, r = lane % WG, gb = g * (2 * WG);
    const uint64_t nl = mn64(list_size<FRESH>(p, list), p.list_cap[list]);
    const uint64_t nitems = (nl + G - 1) / G;
    // a batch's warp takes items next to each other, so that its pairs leave it
    // in long runs of one scene (4 % slower here than every stride-th item, and
    // less than half the time in the grouping)
    const uint64_t per = (nitems + stride - 1) / stride;
    const uint64_t step = p.scene_table ? 1 : stride, end = p.scene_table ? mn64((first + 1) * per, nitems) : nitems;
    for (uint64_t item = p.scene_table ? first * per : first; item < end; item += step) {
        const uint64_t ci = item * G + g;
        uint32_t n = 0, gid = 0, start = 0;
        if (ci < nl) {
            const uint2 sn = p.lists[p.list_off[list] + ci];
            gid = sn.x;  // record mode: the list holds the cell id; its start is in the counters after the scatter
            start = REC ? (gid < p.ncells ? p.counts[gid] : 0xffffffffu) : sn.x;
            n = sn.y;
            if (n > WG || (uint64_t)start + n > p.entry_cap) n = 0;  // inconsistent grid: skip
        }
        const uint4 me = r < n ? p.entries[start + r] : entry_empty();
        __syncwarp();  // (the last item's slots are read)
        if (r < n) {
            s[gb + r] = me;
            s[gb + n + r] = me;
        }
        __syncwarp();
        const uint32_t nelm = r < n ? (r < (n >> 1) ? (n >> 1) : ((n - 1) >> 1)) : 0u;
        const uint32_t dlim = __reduce_max_sync(FULL_MASK, nelm);
        // bit j: group lane j is a partner the rules exclude
        const uint32_t sh = WG == 32 ? 0u : g * WG;
        const uint32_t nm = n >= 32u ? FULL_MASK : ((1u << n) - 1u);
        const bool f0 = ((me.w >> kIdBits) & 1u) == 0u, f1 = ((me.w >> (kIdBits + 1)) & 1u) == 0u;
        const bool f2 = ((me.w >> (kIdBits + 2)) & 1u) == 0u;
        const uint32_t m0 = (__ballot_sync(FULL_MASK, f0) >> sh) & nm;
        const uint32_t m1 = (__ballot_sync(FULL_MASK, f1) >> sh) & nm;
        const uint32_t m2 = (__ballot_sync(FULL_MASK, f2) >> sh) & nm;
        uint32_t deny = (f0 ? m0 : 0u) | (f1 ? m1 : 0u) | (f2 ? m2 : 0u);
        if (BIP) {
            const bool is_red = (me.w & kIdMask) < p.split;
            const uint32_t red = (__ballot_sync(FULL_MASK, is_red) >> sh) & nm;
            deny |= is_red ? red : (~red & nm);
        }
        // bit d: partner (r + d) mod n
        uint32_t rot = 0;
        if (r < n) rot = n >= 32u ? __funnelshift_r(deny, deny, r) : (((deny >> r) | (deny << (n - r))) & nm);
        const uint32_t rx = __byte_perm(me.x, 0u, 0x1032), ry = __byte_perm(me.y, 0u, 0x1032);
        const uint32_t rz = __byte_perm(me.z, 0u, 0x1032);
        uint32_t miss = 0, top = 0;
#pragma unroll
        for (uint32_t d = 1; d <= WG / 2; d++) {
            if (d > dlim) break;
            const uint4 c = s[gb + r + d];
            uint32_t m = __viaddmax_u16x2(ry, c.y, rx + c.x);
            if (D == 3) m = __viaddmax_u16x2(rz, c.z, m);
            m = __vmaxu2(m, __byte_perm(m, 0u, 0x1032));
            top = __vmaxs2(top, m);
            miss |= (m >> 31) << d;
        }
        uint32_t mask = ~miss & ~rot & ((2u << nelm) - 2u);
        // a largest sum of 32767 may be two corners of one scaled value
        if (p.open && top == 0x7fff7fffu && mask) mask = small_exact<D>(p.boxes, p.blue, p.split, p.nboxes, s, gb + r, mask);
        __syncwarp();
        if constexpr (REC) {
            auto ploc = [&](uint32_t d) {
                uint32_t pr = r + d;
                if (pr >= n) pr -= n;
                return pr;
            };
            const uint32_t gmask = WG == 32 ? FULL_MASK : (((1u << WG) - 1u) << (g * WG));
            remit(p, o, mask, ploc, 0u, ploc, r, gid, gmask);
        } else {
            auto pid = [&](uint32_t d) { return s[gb + r + d].w; };
            wemit<BIP>(p, o, mask, pid, 0u, pid, me.w);
        }
    }
}

// hits of a warp's records, added to the query's pair count
__device__ __forceinline__ void rec_hits(const Params& p, const WarpOut& o) {
    const unsigned long long h = warp_sum_u64(o.hits);
    if (lane_id() == 0 && h) atomicAdd(&p.ctr->rec_pairs, h);
}

// the four small-cell lists, warp gw of nw; per-warp staging of kSmallSlots
// entries in s and an output buffer of kWarpOut pairs
template <int D, bool BIP, bool REC, bool FRESH = false>
__device__ __forceinline__ void small_pass(const Params& p, uint4* s, uint2* s_out, uint64_t gw, uint64_t nw) {
    WarpOut o{s_out, 0, kWarpOut};
    // classes interleaved over the warps so every warp gets a similar mix
    small_items<D, 32, BIP, REC, FRESH>(p, s, o, 3, gw, nw);
    small_items<D, 16, BIP, REC, FRESH>(p, s, o, 2, (gw + nw / 4) % nw, nw);
    small_items<D, 8, BIP, REC, FRESH>(p, s, o, 1, (gw + nw / 2) % nw, nw);
    small_items<D, 4, BIP, REC, FRESH>(p, s, o, 0, (gw + 3 * nw / 4) % nw, nw);
    wflush<BIP, REC>(p, o);
    if (REC) rec_hits(p, o);
}

// (with the tile tasks of huge cells, which the block kernel takes: a launch of
// their own took 4 to 6 us, and in the scatter they cost it registers that its
// blocks need to fill the SMs: 89 us became 108 on 4 million points)
template <int D, bool BIP, bool REC = false>
__global__ void __launch_bounds__(kPairThreads, 5) k_pairs_small(Params pin) {
    chain_wait();
    const Params p = resolve(pin);
    stamp(p, kStampSmall);
    const uint32_t huge = p.ctr->n_list[kListHuge];  // (there by the time it is needed)
    __shared__ uint4 s_slot[kPairWarps][kSmallSlots];
    __shared__ uint2 s_out[kPairWarps][kWarpOut];
    const uint32_t warp = threadIdx.x >> 5;
    small_pass<D, BIP, REC>(p, s_slot[warp], s_out[warp], (uint64_t)blockIdx.x * kPairWarps + warp,
                            (uint64_t)gridDim.x * kPairWarps);
    expand_cells(p, pin, huge, blockIdx.x * kPairWarps + warp, gridDim.x * kPairWarps);
}

// ---- tiles ------------------------------------------------------------------
// Cells above the small ones are tested tile by tile, 32 rows against 32
// columns, staged in shared memory as pairs of columns: a word holds one term
// of two boxes, so an add, five u16x2 add-max instructions and two shared
// loads test two columns. The kernels are bound by these instructions (the
// integer pipe issues one of them every other clock; the plain add has a
// second pipe). With 32-bit terms of one column the shared loads alone would
// allow 20 tests/ns per SM, and a sweep with a partner of its own per lane 10;
// a tile against itself is therefore swept whole and masked, rather than in a
// half sweep.
//
// Slot 8b + g of a tile is that bit of the masks and holds box 4g + b; column
// pair j holds the boxes 2j and 2j + 1. So the signs of two pairs, spread over
// bytes by one prmt, go to bit g of every byte, and the columns of a partial
// tile end with group ceil(n/4).
//
// Cells of 2^15 or wider: a sum of exactly 32767 may be two corners that share
// a scaled value, which leaves the test open when no other sum is larger. The
// sweep keeps the largest signed value it saw (32767 is the largest there is),
// and a tile that met one is tested again on the whole coordinates (about 1 %
// of the tiles of random boxes). A box ties with itself where one of its sides
// is shorter than a scaled step, so of points every tile that meets itself did.
// One-launch queries, whose tiles nearly all meet themselves, look at such a
// tile again without those sums first: 262 144 points 106 -> 84 us, 100 000 66
// -> 62. (In the kernels of large queries it gained nothing on points, and
// their registers spilled: the crowded 4M-box scene took 1 % longer.)
//
// Red/blue queries stage the two colours apart, so their tiles are red rows
// against blue columns (or the other way, whichever takes fewer steps), and a
// cell of one colour costs no more than reading its entries.
constexpr uint32_t kMedTiles = kMedMax / 32 + 1;   // (+ 1: two colours, each rounded up to whole tiles)
constexpr uint32_t kBigTiles = kBigMax / 32 + 1;
constexpr uint32_t kHugeTiles = 3;                 // a row tile and two column tiles
constexpr uint32_t kTileBytes = 16 * (sizeof(uint4) + sizeof(uint2)) + 32 * sizeof(uint32_t);

struct Tiles {
    uint4* xy;      // 16 per tile: {x1, x0, y1, y0} terms of a column pair, the second column in the high halves
    uint2* z;       // 16 per tile: {z1, z0}
    uint32_t* raw;  // 32 per tile: the entries' last words (start bits << 29 | box index)
    __device__ __forceinline__ Tiles(unsigned char* m, uint32_t tiles)
        : xy(reinterpret_cast<uint4*>(m)), z(reinterpret_cast<uint2*>(xy + 16 * tiles)),
          raw(reinterpret_cast<uint32_t*>(z + 16 * tiles)) {}
};

// box e of a tile <-> its slot
__device__ __forceinline__ uint32_t tile_slot(uint32_t e) { return ((e & 3u) << 3) | (e >> 2); }
__device__ __forceinline__ uint32_t tile_box(uint32_t s) { return ((s & 7u) << 2) | (s >> 3); }
__device__ __forceinline__ uint32_t tile_fill(uint32_t n, uint32_t x) { return min(32u, n - 32u * x); }

// column pair j of tile x: entries a and b
template <int D>
__device__ __forceinline__ void tile_put_pair(const Tiles& t, uint32_t x, uint32_t j, const uint4& a, const uint4& b) {
    t.xy[16 * x + j] = make_uint4(__byte_perm(a.x, b.x, 0x5410), __byte_perm(a.x, b.x, 0x7632),
                                  __byte_perm(a.y, b.y, 0x5410), __byte_perm(a.y, b.y, 0x7632));
    if (D == 3) t.z[16 * x + j] = make_uint2(__byte_perm(a.z, b.z, 0x5410), __byte_perm(a.z, b.z, 0x7632));
    const uint32_t s = 32 * x + tile_slot(2 * j);
    t.raw[s] = a.w;
    t.raw[s + 8] = b.w;
}

// one entry into slot `slot` of tile x
template <int D>
__device__ __forceinline__ void tile_put(const Tiles& t, uint32_t x, uint32_t slot, const uint4& e) {
    const uint32_t box = tile_box(slot), j = 16 * x + (box >> 1);
    unsigned short* a = reinterpret_cast<unsigned short*>(t.xy + j) + (box & 1u);
    a[0] = (unsigned short)e.x;
    a[2] = (unsigned short)(e.x >> 16);
    a[4] = (unsigned short)e.y;
    a[6] = (unsigned short)(e.y >> 16);
    if (D == 3) {
        unsigned short* b = reinterpret_cast<unsigned short*>(t.z + j) + (box & 1u);
        b[0] = (unsigned short)e.z;
        b[2] = (unsigned short)(e.z >> 16);
    }
    t.raw[32 * x + slot] = e.w;
}

// empty slots of a group's last tile (red/blue: the slots are filled one by one)
template <int D>
__device__ __forceinline__ void tile_clear_rest(const Tiles& t, uint32_t tile, uint32_t n) {
    const uint32_t slot = lane_id();
    if ((n & 31u) != 0u && tile_box(slot) >= (n & 31u)) tile_put<D>(t, tile, slot, entry_empty());
}

__device__ __forceinline__ uint4 entry_at(const Params& p, uint32_t start, uint32_t e, uint32_t n) {
    return e < n ? p.entries[start + e] : entry_empty();
}

// a row: this lane's slot of a tile, each term in both halves of its word,
// and a full mask per axis that it does not start on
template <int D>
struct Row {
    uint32_t t[2 * D];
    uint32_t raw, f0, f1, f2;
};
template <int D>
__device__ __forceinline__ Row<D> tile_row(const Tiles& t, uint32_t x) {
    const uint32_t lane = lane_id(), box = tile_box(lane), sel = box & 1u ? 0x3232u : 0x1010u;
    const uint4 a = t.xy[16 * x + (box >> 1)];
    Row<D> r;
    r.t[0] = __byte_perm(a.y, 0u, sel);  // (a row's lower corner meets the columns' upper ones)
    r.t[1] = __byte_perm(a.x, 0u, sel);
    r.t[2] = __byte_perm(a.w, 0u, sel);
    r.t[3] = __byte_perm(a.z, 0u, sel);
    if (D == 3) {
        const uint2 z = t.z[16 * x + (box >> 1)];
        r.t[2 * D - 2] = __byte_perm(z.y, 0u, sel);
        r.t[2 * D - 1] = __byte_perm(z.x, 0u, sel);
    }
    r.raw = t.raw[32 * x + lane];
    r.f0 = (r.raw >> kIdBits) & 1u ? 0u : ~0u;
    r.f1 = (r.raw >> (kIdBits + 1)) & 1u ? 0u : ~0u;
    r.f2 = (r.raw >> (kIdBits + 2)) & 1u ? 0u : ~0u;
    return r;
}

template <int D>
__device__ __forceinline__ uint32_t tile_pair(const Tiles& t, const Row<D>& r, uint32_t i) {
    const uint4 c = t.xy[i];
    uint32_t m = __viaddmax_u16x2(r.t[1], c.y, r.t[0] + c.x);  // (the halves of the plain add carry nothing)
    m = __viaddmax_u16x2(r.t[2], c.z, m);
    m = __viaddmax_u16x2(r.t[3], c.w, m);
    if (D == 3) {
        const uint2 z = t.z[i];
        m = __viaddmax_u16x2(r.t[2 * D - 2], z.x, m);
        m = __viaddmax_u16x2(r.t[2 * D - 1], z.y, m);
    }
    return m;
}
// column pairs i and i + 1: a miss sets the bit `bits` has in its byte
template <int D>
__device__ __forceinline__ void tile_group(const Tiles& t, const Row<D>& r, uint32_t i, uint32_t bits, uint32_t& miss,
                                           uint32_t& top) {
    const uint32_t m = tile_pair<D>(t, r, i), n = tile_pair<D>(t, r, i + 1);
    uint32_t signs;  // a byte per half: all its sign bit
    asm("prmt.b32 %0, %1, %2, 0xfdb9;" : "=r"(signs) : "r"(m), "r"(n));
    top = __vimax3_s16x2(top, m, n);
    miss |= signs & bits;
}

// the same tile on the whole coordinates: the column boxes pass from lane to
// lane (rare, so it reads the boxes rather than keep them staged)
template <int D>
__device__ __noinline__ uint32_t tile_exact(const uint32_t* boxes, const uint32_t* blue, uint32_t split,
                                            uint64_t nboxes, uint32_t row, uint32_t col, uint32_t rows, uint32_t cols) {
    const uint32_t e = tile_box(lane_id());
    const uint32_t ri = row & kIdMask, ci = col & kIdMask;
    uint32_t a[2 * D], b[2 * D];
    const bool rv = e < rows && ri < nboxes, cv = e < cols && ci < nboxes;
#pragma unroll
    for (int k = 0; k < 2 * D; k++) {
        a[k] = rv ? __ldg(box_row<D>(boxes, blue, split, ri) + k) : 0u;
        b[k] = cv ? __ldg(box_row<D>(boxes, blue, split, ci) + k) : 0u;
    }
    uint32_t mask = 0;
    for (uint32_t j = 0; j < 32; j++) {
        bool hit = true;
#pragma unroll
        for (int d = 0; d < D; d++)
            hit = hit & (a[2 * d] <= __shfl_sync(FULL_MASK, b[2 * d + 1], j)) &
                  (__shfl_sync(FULL_MASK, b[2 * d], j) <= a[2 * d + 1]);
        mask |= (hit ? 1u : 0u) << j;
    }
    const uint32_t there = __ballot_sync(FULL_MASK, cv);
    return rv ? mask & there : 0u;
}

// the bits of the slots of groups `groups` .. 7
__device__ __forceinline__ uint32_t tile_beyond(uint32_t groups) { return ((0xffu << groups) & 0xffu) * 0x01010101u; }

__device__ __forceinline__ bool tile_tied(uint32_t top) {
    const uint32_t low = top ^ 0x7fff7fffu;  // a zero half: a sum of 32767 was the largest of its pair
    return __any_sync(FULL_MASK, ((low - 0x00010001u) & ~low & 0x80008000u) != 0u);
}

// the largest sums of a tile against itself without those of a box with itself
template <int D>
__device__ __forceinline__ uint32_t tile_others(const Tiles& t, const Row<D>& r, uint32_t x, uint32_t cols) {
    const uint32_t lane = lane_id(), own = 0x8000u << (2u * (lane & 8u));  // this lane's box: its half of a pair
    uint32_t top = 0;
#pragma unroll 1
    for (uint32_t g = 0; 4u * g < cols; g++) {
        uint32_t m = tile_pair<D>(t, r, 16 * x + 2 * g), n = tile_pair<D>(t, r, 16 * x + 2 * g + 1);
        if (g == (lane & 7u)) {
            m |= lane < 16u ? own : 0u;
            n |= lane < 16u ? 0u : own;
        }
        top = __vimax3_s16x2(top, m, n);
    }
    return top;
}

// row tile against column tile x of `cols` boxes: bit s set iff this lane's
// box and slot s overlap and the reference-cell rule reports them here. OWN:
// ties of boxes with themselves are looked for where the tiles are one (self).
template <int D, bool OWN>
__device__ __forceinline__ uint32_t tile_hits(const Params& p, const Tiles& t, const Row<D>& r, uint32_t rows,
                                              uint32_t x, uint32_t cols, bool self) {
    uint32_t miss = 0, top = 0;
    if (cols > 24u) {
#pragma unroll
        for (uint32_t g = 0; g < 8; g++) tile_group<D>(t, r, 16 * x + 2 * g, 0x01010101u << g, miss, top);
    } else {
        const uint32_t groups = ((cols + 7u) >> 3) * 2u;
        uint32_t bits = 0x01010101u;
        for (uint32_t g = 0; g < groups; g += 2, bits <<= 2) {
            tile_group<D>(t, r, 16 * x + 2 * g, bits, miss, top);
            tile_group<D>(t, r, 16 * x + 2 * g + 2, bits << 1, miss, top);
        }
        miss |= tile_beyond(groups);
    }
    const uint32_t raw = t.raw[32 * x + lane_id()];
    uint32_t mask = ~miss;
    if (p.open && tile_tied(top) && (!OWN || !self || tile_tied(tile_others<D>(t, r, x, cols))))
        mask = tile_exact<D>(p.boxes, p.blue, p.split, p.nboxes, r.raw, raw, rows, cols);
    const uint32_t m0 = __ballot_sync(FULL_MASK, ((raw >> kIdBits) & 1u) == 0u);
    const uint32_t m1 = __ballot_sync(FULL_MASK, ((raw >> (kIdBits + 1)) & 1u) == 0u);
    const uint32_t m2 = __ballot_sync(FULL_MASK, ((raw >> (kIdBits + 2)) & 1u) == 0u);
    return mask & ~((m0 & r.f0) | (m1 & r.f1) | (m2 & r.f2));
}

// the slots after this lane's, for a tile against itself
__device__ __forceinline__ uint32_t after_lane() { return 0xfffffffeu << lane_id(); }

// The pairs of a row tile with column tiles a and b (their entries' last words
// at ca and cb, by slot) into the warp buffer. A lane writes the pairs of its
// own row, a pair a step, if there are at most kRowHits of them; the warp
// writes a longer row together, a lane a column of each tile. Rows differ: a
// step has 102 pairs on two million red and blue boxes, and 22 in its longest
// row; in the crowded 4M-box scene 131 and 17, in the clustered one 55 and 7.
// Big cells of the three with every row its lane's: 261, 887 and 450 us; with
// rows above 12 written together 232, 794 and 407, above 9 230, 811 and 407,
// above 16 236, 793 and 415.
constexpr uint32_t kRowHits = 12;

// More pairs than the buffer holds, straight to the pair array: a lane a column
// of each tile, so that a store covers its row's pairs one after the other. (A
// lane a row, each store's pairs were up to 512 bytes apart: 84 million pairs of
// 20 000 boxes in one cell took 2780 us, now 1060.) k: the
// lane's pairs, `at` of the total before them.
template <bool BIP>
__device__ __forceinline__ void row_store(const Params& p, uint32_t ma, const uint32_t* ca, uint32_t mb, const uint32_t* cb,
                                       uint32_t row, uint32_t k, uint32_t at, uint32_t total) {
    const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&p.ctr->pairs, (unsigned long long)total);
    base = __shfl_sync(FULL_MASK, base, 0);
    if (base + total > p.out_cap && lane == 0) atomicOr(&p.ctr->err, kErrOutOvf);
    const uint32_t va = ca[lane], vb = cb[lane];
    for (uint32_t rows = __ballot_sync(FULL_MASK, k != 0u); rows; rows &= rows - 1) {
        const uint32_t l = __ffs(rows) - 1;
        const uint32_t a = __shfl_sync(FULL_MASK, ma, l), b = __shfl_sync(FULL_MASK, mb, l);
        const uint32_t r = __shfl_sync(FULL_MASK, row, l);
        const unsigned long long g = base + __shfl_sync(FULL_MASK, at, l);
        const unsigned long long ga = g + __popc(a & below), gb = g + __popc(a) + __popc(b & below);
        if (((a >> lane) & 1u) && ga < p.out_cap) p.out[ga] = out_pair<BIP, false>(p, make_uint2(r, va));
        if (((b >> lane) & 1u) && gb < p.out_cap) p.out[gb] = out_pair<BIP, false>(p, make_uint2(r, vb));
    }
    __syncwarp();
}

template <bool BIP>
__device__ __forceinline__ void row_emit(const Params& p, WarpOut& o, uint32_t ma, const uint32_t* ca, uint32_t mb,
                                         const uint32_t* cb, uint32_t row) {
    const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
    const uint32_t k = __popc(ma) + __popc(mb);
    const uint32_t incl = warp_incl_scan(k);
    const uint32_t total = __shfl_sync(FULL_MASK, incl, 31);
    if (total == 0) return;
    if (o.n + total > o.cap) {
        wflush<BIP, false>(p, o);
        if (total > o.cap) {  // past the buffer: every row by the whole warp
            row_store<BIP>(p, ma, ca, mb, cb, row, k, incl - k, total);
            return;
        }
    }
    const uint32_t first = o.n + incl - k;
    uint32_t longer = __ballot_sync(FULL_MASK, k > kRowHits);
    if (k <= kRowHits) {
        uint2* dst = o.buf + first;
        for (uint32_t m = ma; m;) {
            const uint32_t bit = 31u - __clz(m);  // highest set bit first
            m ^= 1u << bit;
            *dst++ = make_uint2(row, ca[bit]);
        }
        for (uint32_t m = mb; m;) {
            const uint32_t bit = 31u - __clz(m);
            m ^= 1u << bit;
            *dst++ = make_uint2(row, cb[bit]);
        }
    }
    if (longer) {
        const uint32_t va = ca[lane], vb = cb[lane];
        do {
            const uint32_t l = 31u - __clz(longer);
            longer ^= 1u << l;
            const uint32_t a = __shfl_sync(FULL_MASK, ma, l), b = __shfl_sync(FULL_MASK, mb, l);
            const uint32_t r = __shfl_sync(FULL_MASK, row, l);
            uint2* dst = o.buf + __shfl_sync(FULL_MASK, first, l);
            if ((a >> lane) & 1u) dst[__popc(a & below)] = make_uint2(r, va);
            if ((b >> lane) & 1u) dst[__popc(a) + __popc(b & below)] = make_uint2(r, vb);
        } while (longer);
    }
    __syncwarp();
    o.n += total;
}

// the pairs of one or two column tiles of a row tile; gid and the tiles'
// first box in the cell are for record mode
template <bool BIP, bool REC>
__device__ __forceinline__ void tile_emit(const Params& p, const Tiles& t, WarpOut& o, uint32_t row, uint32_t ma,
                                          uint32_t xa, uint32_t mb, uint32_t xb, uint32_t row0, uint32_t col0a,
                                          uint32_t col0b, uint32_t gid) {
    if constexpr (REC) {
        remit(p, o, ma, [&](uint32_t b) { return col0a + tile_box(b); }, mb,
              [&](uint32_t b) { return col0b + tile_box(b); }, row0 + tile_box(lane_id()), gid, FULL_MASK);
    } else {
        row_emit<BIP>(p, o, ma, t.raw + 32 * xa, mb, t.raw + 32 * xb, row);
    }
}

// A staged cell's rows and columns as tiles: self queries have n boxes in
// tiles 0, 1, ...; red/blue queries the red boxes in tiles 0, 1, ... and the
// blue ones in the last tile, the one before, ...
struct CellTiles {
    uint32_t rows, cols;  // boxes
    int row0, row_step, col0, col_step;
    __device__ __forceinline__ uint32_t row_tiles() const { return (rows + 31u) >> 5; }
    __device__ __forceinline__ uint32_t col_tiles() const { return (cols + 31u) >> 5; }
    __device__ __forceinline__ uint32_t row_tile(uint32_t r) const { return (uint32_t)(row0 + row_step * (int)r); }
    __device__ __forceinline__ uint32_t col_tile(uint32_t x) const { return (uint32_t)(col0 + col_step * (int)x); }
};
// red/blue: the colour whose tiles make fewer steps (whole row tiles, quarters of column tiles) is the columns
__device__ __forceinline__ CellTiles cell_tiles_bip(uint32_t red, uint32_t blue, uint32_t tiles) {
    const int last = (int)tiles - 1;
    if (((red + 31u) >> 5) * ((blue + 7u) >> 3) <= ((blue + 31u) >> 5) * ((red + 7u) >> 3))
        return CellTiles{red, blue, 0, 1, last, -1};
    return CellTiles{blue, red, last, -1, 0, 1};
}

// a red/blue entry into its colour's tiles: box rank e of its colour
template <int D>
__device__ __forceinline__ void tile_put_colour(const Tiles& t, uint32_t tiles, bool is_red, uint32_t e, const uint4& w) {
    tile_put<D>(t, is_red ? e >> 5 : tiles - 1 - (e >> 5), tile_slot(e & 31u), w);
}

// row tile r of a staged cell against its column tiles from x (self: from r),
// `count` of them at most, two per emission step
template <int D, bool BIP, bool REC, bool OWN>
__device__ __forceinline__ void row_sweep(const Params& p, const Tiles& t, WarpOut& o, const CellTiles& c, uint32_t r,
                                          uint32_t x, uint32_t count, uint32_t gid) {
    const uint32_t rows = tile_fill(c.rows, r), end = min(c.col_tiles(), x + count);
    const Row<D> row = tile_row<D>(t, c.row_tile(r));
    for (; x < end; x += 2) {
        const uint32_t xa = c.col_tile(x);
        uint32_t ma = tile_hits<D, OWN && !BIP>(p, t, row, rows, xa, tile_fill(c.cols, x), x == r);
        if (!BIP && x == r) ma &= after_lane();
        uint32_t mb = 0, xb = xa;
        if (x + 1 < end) {
            xb = c.col_tile(x + 1);
            mb = tile_hits<D, false>(p, t, row, rows, xb, tile_fill(c.cols, x + 1), false);
        }
        tile_emit<BIP, REC>(p, t, o, row.raw, ma, xa, mb, xb, 32 * r, 32 * x, 32 * (x + 1), gid);
    }
}

// ---- medium cells: one per warp item, staged whole ---------------------------
// the medium-cell list, warp gw of nw (the one-launch kernel: items in a
// fixed stride; the medium-cell kernel: every warp takes items from one
// counter); wsm: the warp's kMedWarpBytes of shared memory (tiles, then the
// output buffer)
constexpr uint32_t kMedWarpBytes = kMedTiles * kTileBytes + kMedOut * sizeof(uint2);

template <int D, bool BIP, bool REC, bool FRESH = false>
__device__ __forceinline__ void med_pass(const Params& p, unsigned char* wsm, uint64_t gw, uint64_t nw) {
    const uint32_t lane = lane_id();
    const Tiles t(wsm, kMedTiles);
    WarpOut o{reinterpret_cast<uint2*>(wsm + kMedTiles * kTileBytes), 0, kMedOut};
    const uint64_t nl = mn64(list_size<FRESH>(p, kListMed), p.list_cap[kListMed]);
    auto cell = [&](uint64_t item) {
        const uint2 sn = p.lists[p.list_off[kListMed] + item];
        const uint32_t gid = sn.x;  // record mode: the cell id (its start is in the counters)
        const uint32_t start = REC ? (gid < p.ncells ? p.counts[gid] : 0xffffffffu) : sn.x;
        const uint32_t n = sn.y;
        if (n > kMedMax || (uint64_t)start + n > p.entry_cap) return;  // inconsistent grid: skip
        CellTiles c{n, n, 0, 1, 0, 1};
        if (!BIP) {  // a lane takes one column pair of each two tiles (all loads in flight together)
            constexpr uint32_t kPer = kMedMax / 64;
            uint4 a[kPer], b[kPer];
#pragma unroll
            for (uint32_t k = 0; k < kPer; k++) {
                a[k] = entry_at(p, start, 64 * k + 2 * lane, n);
                b[k] = entry_at(p, start, 64 * k + 2 * lane + 1, n);
            }
#pragma unroll
            for (uint32_t k = 0; k < kPer; k++)
                if (64 * k < n) tile_put_pair<D>(t, 2 * k + (lane >> 4), lane & 15u, a[k], b[k]);
        } else {
            constexpr uint32_t kPer = kMedMax / 32;
            uint4 w[kPer];
            uint32_t reds[kPer], red = 0;
#pragma unroll
            for (uint32_t k = 0; k < kPer; k++) w[k] = entry_at(p, start, 32 * k + lane, n);
#pragma unroll
            for (uint32_t k = 0; k < kPer; k++) {
                reds[k] = __ballot_sync(FULL_MASK, 32 * k + lane < n && (w[k].w & kIdMask) < p.split);
                red += __popc(reds[k]);
            }
            if (red == 0u || red == n) return;  // one colour: no pair
            uint32_t r0 = 0, b0 = 0;  // boxes of each colour before chunk k
#pragma unroll
            for (uint32_t k = 0; k < kPer; k++) {
                const uint32_t left = n > 32 * k ? min(32u, n - 32 * k) : 0u;
                const uint32_t rr = __popc(reds[k] & ((1u << lane) - 1u));
                const bool is_red = (reds[k] >> lane) & 1u;
                if (lane < left) tile_put_colour<D>(t, kMedTiles, is_red, is_red ? r0 + rr : b0 + (lane - rr), w[k]);
                r0 += __popc(reds[k]);
                b0 += left - __popc(reds[k]);
            }
            tile_clear_rest<D>(t, (red - 1) >> 5, red);
            tile_clear_rest<D>(t, kMedTiles - 1 - ((n - red - 1) >> 5), n - red);
            c = cell_tiles_bip(red, n - red, kMedTiles);
        }
        __syncwarp();
        const uint32_t R = c.row_tiles();
        for (uint32_t r = 0; r < R; r++) row_sweep<D, BIP, REC, FRESH>(p, t, o, c, r, BIP ? 0u : r, ~0u >> 1, gid);
        __syncwarp();
    };
    // items taken from a counter, so warps whose cells were larger end no
    // later than the others (with one cell at a time 0.444 ms on the clustered
    // 4M-box scene when this was tried, against 0.499 ms for a fixed stride
    // over the list), of a batch 16 at a time and fewer as the list ends, so
    // that its pairs leave the warp in long runs of one scene (512 scenes 0.58
    // ms here, with one at a time 0.56, with 15 to the end 0.60; the grouping
    // takes 0.17 ms instead of 0.27). A one-launch query's warps take one or
    // two cells each: there the counter's round trip costs more than the
    // balance gains.
    if constexpr (FRESH) {
        for (uint64_t item = gw; item < nl; item += nw) cell(item);
    } else {
        uint32_t run = 0;
        uint64_t item = 0;
        for (;;) {
            run = p.scene_table ? max((uint32_t)mn64((nl - item) / (4 * nw), 16), 1u) : 1u;
            if (lane == 0) item = atomicAdd(&p.ctr->med_next, run);
            item = __shfl_sync(FULL_MASK, item, 0);
            if (item >= nl) break;
            for (const uint64_t end = mn64(item + run, nl); item < end; item++) cell(item);
        }
    }
    wflush<BIP, REC>(p, o);
    if (REC) rec_hits(p, o);
}

template <int D, bool BIP, bool REC = false>
__global__ void __launch_bounds__(kPairThreads, 4) k_pairs_med(Params pin) {
    chain_wait();
    const Params p = resolve(pin);
    stamp(p, kStampMed);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t warp = threadIdx.x >> 5;
    med_pass<D, BIP, REC>(p, smem_raw + warp * kMedWarpBytes, (uint64_t)blockIdx.x * kPairWarps + warp,
                          (uint64_t)gridDim.x * kPairWarps);
}

// ---- big cells (staged by a team of warps) and huge cells (tile tasks) -------
// A team of four warps stages a big cell and shares its tiles. Small teams, so
// that those waiting for a cell's entries or for their last warp are few among
// the eight on an SM: with teams of eight warps, three an SM, half the issue
// slots were empty (1.10 ms for the cells of 129..512 boxes of the crowded
// 4M-box scene, against 0.78 ms).
constexpr int kTeamWarps = 4;
constexpr int kTeamThreads = 32 * kTeamWarps;

struct TeamSmem {
    uint4 tiles[kBigTiles * kTileBytes / sizeof(uint4)];  // a big cell's; huge cells: kHugeTiles per warp
    uint2 out[kTeamWarps][kMedOut];
    uint2 cell;          // the team's cell {start, n}; n = 0: none is left
    uint32_t red, blue;  // red/blue: boxes of each colour placed so far
    uint32_t next_unit;
    uint32_t pad[3];
};
static_assert(kTeamWarps * kHugeTiles <= kBigTiles, "huge cells' tiles in a big cell's");

// a barrier of the team: the block, or (SUB) a quarter of the one-launch kernel's
template <bool SUB>
__device__ __forceinline__ void team_sync() {
    if constexpr (SUB) asm volatile("bar.sync %0, %1;" ::"r"(1u + threadIdx.x / kTeamThreads), "n"(kTeamThreads) : "memory");
    else __syncthreads();
}

// one big cell: staged by the team's threads, then its warps take units of a
// row tile and up to two column tiles from a counter. s.next_unit and the
// colour counts are zero at the start.
template <int D, bool BIP, bool REC, bool SUB>
__device__ __forceinline__ void big_cell(const Params& p, TeamSmem& s, WarpOut& o, uint2 sn) {
    const uint32_t lane = lane_id(), tid = threadIdx.x % kTeamThreads, warp = tid >> 5;
    const Tiles t(reinterpret_cast<unsigned char*>(s.tiles), kBigTiles);
    const uint32_t gid = sn.x, n = sn.y;  // record mode: the list holds the cell id, its start is in the counters
    const uint32_t start = REC ? (gid < p.ncells ? p.counts[gid] : 0xffffffffu) : sn.x;
    if (n > kBigMax || (uint64_t)start + n > p.entry_cap) return;  // inconsistent grid: skip (the whole team)
    CellTiles c{n, n, 0, 1, 0, 1};
    if (!BIP) {
        constexpr uint32_t kPer = kBigMax / 2 / kTeamThreads;
        uint4 a[kPer], b[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            const uint32_t q = tid + kTeamThreads * k;  // column pair
            a[k] = entry_at(p, start, 2 * q, n);
            b[k] = entry_at(p, start, 2 * q + 1, n);
        }
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            const uint32_t q = tid + kTeamThreads * k;
            if (32 * (q >> 4) < n) tile_put_pair<D>(t, q >> 4, q & 15u, a[k], b[k]);
        }
        team_sync<SUB>();
    } else {
        constexpr uint32_t kPer = kBigMax / kTeamThreads;
        uint4 w[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) w[k] = entry_at(p, start, tid + kTeamThreads * k, n);
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            const uint32_t first = 32 * (warp + kTeamWarps * k);  // this warp's 32 entries
            if (first >= n) continue;
            const uint32_t left = min(32u, n - first);
            const bool is_red = lane < left && (w[k].w & kIdMask) < p.split;
            const uint32_t reds = __ballot_sync(FULL_MASK, is_red), nr = __popc(reds);
            uint32_t r0 = 0, b0 = 0;
            if (lane == 0) {
                r0 = atomicAdd(&s.red, nr);
                b0 = atomicAdd(&s.blue, left - nr);
            }
            r0 = __shfl_sync(FULL_MASK, r0, 0);
            b0 = __shfl_sync(FULL_MASK, b0, 0);
            const uint32_t rr = __popc(reds & ((1u << lane) - 1u));
            if (lane < left) tile_put_colour<D>(t, kBigTiles, is_red, is_red ? r0 + rr : b0 + (lane - rr), w[k]);
        }
        team_sync<SUB>();
        const uint32_t red = s.red;
        if (red == 0u || red == n) return;  // one colour: no pair
        if (warp == 0) tile_clear_rest<D>(t, (red - 1) >> 5, red);
        if (warp == 1) tile_clear_rest<D>(t, kBigTiles - 1 - ((n - red - 1) >> 5), n - red);
        c = cell_tiles_bip(red, n - red, kBigTiles);
        team_sync<SUB>();
    }
    // units in the order of their row tiles: row r's first unit is `before`
    const uint32_t R = c.row_tiles(), X = c.col_tiles();
    uint32_t r = 0, before = 0;
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(&s.next_unit, 1u);
        u = __shfl_sync(FULL_MASK, u, 0);
        uint32_t units;
        while (r < R && u >= before + (units = (X - (BIP ? 0u : r) + 1u) >> 1)) {
            before += units;
            r++;
        }
        if (r >= R) break;
        row_sweep<D, BIP, REC, SUB>(p, t, o, c, r, (BIP ? 0u : r) + 2 * (u - before), 2, gid);
    }
}

// huge cells: one tile task {start, n, r, x0} per warp; the row tile and two
// column tiles at a time staged in the warp's own tiles
template <int D, bool BIP, bool REC>
__device__ __forceinline__ void huge_item(const Params& p, const Tiles& t, WarpOut& o, const uint4& tk) {
    const uint32_t lane = lane_id();
    const uint32_t gid = tk.x;  // record mode: the cell id; its start is in the counters
    const uint32_t start = REC ? (gid < p.ncells ? p.counts[gid] : 0xffffffffu) : tk.x;
    const uint32_t n = tk.y, r = tk.z, x0 = tk.w;
    if (REC && n >= 65536u) {  // beyond the record format (u8 row tile)
        if (lane == 0) atomicOr(&p.ctr->err, kErrRecCell);
        return;
    }
    const uint32_t R = (n + 31) >> 5;
    const uint32_t x1 = min(x0 + kTaskCols, R);
    if ((uint64_t)start + n > p.entry_cap || r >= R || x0 >= R) return;
    const uint32_t rows = tile_fill(n, r), j = lane & 15u;
    if (lane < 16u)
        tile_put_pair<D>(t, 0, j, entry_at(p, start, 32 * r + 2 * j, n), entry_at(p, start, 32 * r + 2 * j + 1, n));
    __syncwarp();
    const Row<D> row = tile_row<D>(t, 0);
    for (uint32_t x = x0; x < x1; x += 2) {
        const uint32_t e = 32 * x + 2 * lane, end = min(n, 32 * x1);
        __syncwarp();  // (the last columns are read)
        tile_put_pair<D>(t, 1 + (lane >> 4), j, entry_at(p, start, e, end), entry_at(p, start, e + 1, end));
        __syncwarp();
        uint32_t m[2] = {0u, 0u};
#pragma unroll
        for (uint32_t k = 0; k < 2; k++) {
            if (x + k >= x1) continue;
            m[k] = tile_hits<D, false>(p, t, row, rows, 1 + k, tile_fill(n, x + k), false);
            if (x + k == r) m[k] &= after_lane();
            if (BIP) {
                const uint32_t red = __ballot_sync(FULL_MASK, (t.raw[32 * (1 + k) + lane] & kIdMask) < p.split);
                m[k] &= (row.raw & kIdMask) < p.split ? ~red : red;
            }
        }
        tile_emit<BIP, REC>(p, t, o, row.raw, m[0], 1, m[1], 2, 32 * r, 32 * x, 32 * (x + 1), gid);
    }
    __syncwarp();
}

// big cells, then the tile tasks of huge cells: team `team` of nteam. Big
// cells are taken from a counter (the one-launch kernel: in a fixed stride),
// the next one while the team is at work on its own.
template <int D, bool BIP, bool REC, bool FRESH = false, bool SUB = false>
__device__ __forceinline__ void team_pass(const Params& p, TeamSmem& s, uint64_t team, uint64_t nteam) {
    const uint32_t tid = threadIdx.x % kTeamThreads, warp = tid >> 5;
    WarpOut o{s.out[warp], 0, kMedOut};
    const uint64_t nb = mn64(list_size<FRESH>(p, kListBig), p.list_cap[kListBig]);
    const uint64_t nt = mn64(list_size<FRESH>(p, kNumLists), p.task_cap);
    uint64_t item = team;
    auto fetch = [&]() {
        if (!FRESH) item = atomicAdd(&p.ctr->big_next, 1u);
        const uint2 sn = item < nb ? p.lists[p.list_off[kListBig] + item] : make_uint2(0u, 0u);
        item += nteam;
        return sn;
    };
    uint2 next = make_uint2(0u, 0u);
    if (nb > 0) {  // (uniform)
        if (tid == 0) next = fetch();
        for (;;) {
            if (tid == 0) {
                s.cell = next;
                s.red = s.blue = s.next_unit = 0u;
            }
            team_sync<SUB>();
            const uint2 sn = s.cell;
            if (sn.y == 0u) break;
            if (tid == 0) next = fetch();
            big_cell<D, BIP, REC, SUB>(p, s, o, sn);
            team_sync<SUB>();
        }
    }
    const Tiles t(reinterpret_cast<unsigned char*>(s.tiles) + warp * kHugeTiles * kTileBytes, kHugeTiles);
    for (uint64_t i = team * kTeamWarps + warp; i < nt; i += nteam * kTeamWarps) huge_item<D, BIP, REC>(p, t, o, p.tasks[i]);
    wflush<BIP, REC>(p, o);
    if (REC) rec_hits(p, o);
}

template <int D, bool BIP, bool REC = false>
__global__ void __launch_bounds__(kTeamThreads, 8) k_pairs_block(Params pin) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    chain_wait();
    const Params p = resolve(pin);
    stamp(p, kStampBlock);
    team_pass<D, BIP, REC>(p, *reinterpret_cast<TeamSmem*>(smem_raw), blockIdx.x, gridDim.x);
    query_end(p);
}

// record mode, after the pair kernels: the entries' box indices, which the
// record decoder reads (the reference's Recs array)
__global__ void k_strip_entries(Params pin) {
    const Params p = resolve(pin);
    const uint64_t n = mn64(p.ctr->entries, p.entry_cap);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p.recs[i] = p.entries[i].w & kIdMask;
}

// ---------------------------------------------------------------------------
// group pairs by scene (batched queries): a pair's scene is the scene of its
// first box; pairs are written to their scene's range with scene-local ids.
//
// As one pass of a radix sort by scene: each block counts a run of the pairs
// per scene in shared memory (k_scene_hist, which keeps the block's counts and
// adds them to the scenes' totals) and, once the totals are offsets, reserves
// its part of every scene it met with one atomic and places its pairs from
// shared-memory counters (k_group_by_scene). Pairs come out of the pair kernels
// in runs of one scene, so each warp takes a run of its own and keeps the
// bounds of the scene it is in: a lookup, five loads one after the other, is
// made where the scene changes only. With a lookup per warp step 512 scenes of
// 18.4 M pairs took 470 us, with one per pair 288 us, and with the warps adding
// to the scenes' totals themselves 326 us (eight scenes of 1.3 M pairs, all on
// a few counters' heels, 79 us). More than kGroupScenes scenes still do that:
// their counters do not fit the shared memory, and are many.
// ---------------------------------------------------------------------------
constexpr int kGroupThreads = 512;
constexpr int kGroupAhead = 4;            // warp steps of pairs loaded together
constexpr uint32_t kGroupScenes = 8192;   // 12 bytes of counters each: two blocks an SM
constexpr size_t kGroupBytes = sizeof(unsigned long long) + sizeof(uint32_t);

// the scene a warp is in: its boxes [lo, hi)
struct SceneRun {
    uint32_t scene = 0, lo = 0, hi = 0;
};

// warp step over the boxes gi of the valid lanes: each scene among them, with
// the lanes that have it; change() where it is not the one before
template <class C, class F>
__device__ __forceinline__ void warp_by_scene(const Params& p, SceneRun& run, uint32_t gi, bool valid, C change, F lanes) {
    uint32_t left = __ballot_sync(FULL_MASK, valid);
    while (left) {
        uint32_t mine = __ballot_sync(FULL_MASK, gi >= run.lo && gi < run.hi) & left;
        if (mine == 0u) {  // another scene: that of the first lane left
            const uint32_t x = __shfl_sync(FULL_MASK, gi, __ffs(left) - 1);
            const uint32_t s = find_scene(p, x);
            change(s);
            run.scene = s;
            run.lo = p.scene_box_off[s];
            run.hi = p.scene_box_off[s + 1];
            mine = __ballot_sync(FULL_MASK, gi >= run.lo && gi < run.hi) & left;
            if (mine == 0u) return;  // (cannot happen: every box has its scene)
        }
        lanes(mine);
        left &= ~mine;
    }
}

// step(pair, whether the lane has one) over this warp's run of the pairs, a
// few steps' loads in flight together
template <class F>
__device__ __forceinline__ void group_pairs(const Params& p, F step) {
    const unsigned long long n = mn64(__ldcg(&p.ctr->pairs), p.out_cap);
    const unsigned long long warps = (unsigned long long)gridDim.x * (kGroupThreads / 32);
    const unsigned long long per = ((n + 31) / 32 + warps - 1) / warps * 32;
    const unsigned long long first = per * ((unsigned long long)blockIdx.x * (kGroupThreads / 32) + (threadIdx.x >> 5));
    const unsigned long long end = first + per < n ? first + per : n;
    for (unsigned long long i = first; i < end; i += 32 * kGroupAhead) {
        uint2 pr[kGroupAhead];
#pragma unroll
        for (int k = 0; k < kGroupAhead; k++) {
            const unsigned long long at = i + 32 * k + lane_id();
            pr[k] = at < end ? p.out[at] : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int k = 0; k < kGroupAhead; k++) step(pr[k], i + 32 * k + lane_id() < end);
    }
}

// LOCAL: the block's counters are in shared memory
template <bool LOCAL>
__global__ void __launch_bounds__(kGroupThreads, 2) k_scene_hist(Params pin, unsigned long long* hist, uint32_t* block_counts) {
    extern __shared__ unsigned long long group_smem[];
    chain_wait();
    const Params p = resolve(pin);
    stamp(p, kStampGroup);
    const uint32_t lane = lane_id();
    uint32_t* counts = reinterpret_cast<uint32_t*>(group_smem);
    if constexpr (LOCAL) {
        for (uint32_t s = threadIdx.x; s < p.nscenes; s += kGroupThreads) counts[s] = 0u;
        __syncthreads();
    }
    SceneRun run;
    uint32_t have = 0;  // pairs of the scene the warp is in, not yet added to its counter
    const auto add = [&](uint32_t) {
        if (lane == 0 && have) {
            if constexpr (LOCAL) atomicAdd(&counts[run.scene], have);
            else atomicAdd(&hist[run.scene], (unsigned long long)have);
        }
        have = 0;
    };
    group_pairs(p, [&](uint2 pr, bool valid) {
        warp_by_scene(p, run, pr.x, valid, add, [&](uint32_t mine) { have += __popc(mine); });
    });
    add(0u);
    if constexpr (LOCAL) {
        __syncthreads();
        for (uint32_t s = threadIdx.x; s < p.nscenes; s += kGroupThreads) {
            const uint32_t c = counts[s];
            block_counts[(uint64_t)blockIdx.x * p.nscenes + s] = c;
            if (c) atomicAdd(&hist[s], (unsigned long long)c);
        }
    }
}

template <bool LOCAL>
__global__ void __launch_bounds__(kGroupThreads, 2) k_group_by_scene(Params pin, const unsigned long long* scene_pair_off,
                                                                     unsigned long long* scene_cursor,
                                                                     const uint32_t* block_counts, uint2* dst) {
    extern __shared__ unsigned long long group_smem[];  // a scene's part of dst for this block, then its pairs so far
    chain_wait();
    const Params p = resolve(pin);
    const uint32_t lane = lane_id();
    uint32_t* placed = reinterpret_cast<uint32_t*>(group_smem + p.nscenes);
    if constexpr (LOCAL) {
        for (uint32_t s = threadIdx.x; s < p.nscenes; s += kGroupThreads) {
            const uint32_t c = block_counts[(uint64_t)blockIdx.x * p.nscenes + s];
            if (c) group_smem[s] = scene_pair_off[s] + atomicAdd(&scene_cursor[s], (unsigned long long)c);
            placed[s] = 0u;
        }
        __syncthreads();
    }
    SceneRun run;
    uint2* part = dst;  // of the scene the warp is in
    const auto change = [&](uint32_t s) { part = dst + (LOCAL ? group_smem[s] : scene_pair_off[s]); };
    group_pairs(p, [&](uint2 pr, bool valid) {
        warp_by_scene(p, run, pr.x, valid, change, [&](uint32_t mine) {
            const uint32_t leader = __ffs(mine) - 1;
            unsigned long long at = 0;
            if constexpr (LOCAL) {
                uint32_t k = 0;
                if (lane == leader) k = atomicAdd(&placed[run.scene], (uint32_t)__popc(mine));
                at = __shfl_sync(FULL_MASK, k, leader);
            } else {
                if (lane == leader) at = atomicAdd(&scene_cursor[run.scene], (unsigned long long)__popc(mine));
                at = __shfl_sync(FULL_MASK, at, leader);
            }
            if ((mine >> lane) & 1u)
                part[at + __popc(mine & ((1u << lane) - 1u))] = make_uint2(pr.x - run.lo, pr.y - run.lo);
        });
    });
    query_end(p);
}

// exclusive scan of the per-scene pair counts: off[s] = sum of hist[< s],
// off[nscenes] = total, also to page-locked host memory; one block, 1024
// threads, chunks of 1024 scenes
__global__ void __launch_bounds__(1024) k_scene_offsets(Params pin, const unsigned long long* hist,
                                                        unsigned long long* off, unsigned long long* off_host) {
    chain_wait();
    const Params p = resolve(pin);
    __shared__ unsigned long long s_w[32];
    __shared__ unsigned long long s_carry;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    if (t == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t c0 = 0; c0 <= p.nscenes; c0 += 1024) {
        const uint32_t i = c0 + t;
        const unsigned long long v = i < p.nscenes ? hist[i] : 0ull;
        unsigned long long x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(FULL_MASK, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31) s_w[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned long long w = s_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(FULL_MASK, w, o);
                if (lane >= (uint32_t)o) w += y;
            }
            s_w[lane] = w;
        }
        __syncthreads();
        const unsigned long long incl = x + (warp ? s_w[warp - 1] : 0ull) + s_carry;
        if (i <= p.nscenes) {
            off[i] = incl - v;
            off_host[i] = incl - v;
        }
        __syncthreads();
        if (t == 1023) s_carry = incl;
        __syncthreads();
    }
}


// ---------------------------------------------------------------------------
// queries of a few thousand boxes: every pair of 32x32 tiles of the boxes,
// rows in registers, columns in the warp's shared memory, whole coordinates --
// no grid, no phases to wait for. 1024 boxes take 3.5 us here and took 22 us in
// the one-launch kernel, most of it latency between its grid barriers. An invalid box (its
// row then overlaps nothing) is reported by the tile of its row or column
// against itself (red/blue: by the first tile that it is in).
// ---------------------------------------------------------------------------
template <int D>
struct WholeBox {
    uint32_t lo[D], hi[D];
};
template <int D>
__device__ __forceinline__ WholeBox<D> whole_box(const Params& p, const uint32_t* boxes, uint32_t i, uint32_t n, bool report) {
    WholeBox<D> b;
    uint32_t err = 0;
    if (i < n) {
        const uint32_t* r = boxes + (uint64_t)i * (2 * D + 1);
#pragma unroll
        for (int d = 0; d < D; d++) {
            b.lo[d] = __ldg(r + 2 * d);
            b.hi[d] = __ldg(r + 2 * d + 1);
        }
        if (__ldg(r + 2 * D) != i) err |= kErrRid;
#pragma unroll
        for (int d = 0; d < D; d++) {
            if (b.lo[d] >= p.max_range || b.hi[d] >= p.max_range) err |= kErrRange;
            if (b.lo[d] > b.hi[d]) err |= kErrInverted;
        }
        if (err && report) {
            atomicOr(&p.ctr->err, err);
            atomicAdd(&p.ctr->bad, 1u);
        }
    }
    if (i >= n || err) {
#pragma unroll
        for (int d = 0; d < D; d++) {
            b.lo[d] = 0xffffffffu;
            b.hi[d] = 0u;
        }
    }
    return b;
}

constexpr uint32_t kAllOut = 256;  // per-warp output buffer (pairs)

template <int D, bool BIP>
__global__ void __launch_bounds__(kPairThreads) k_all_pairs(Params p, Ctr* ctr_next) {
    __shared__ uint4 s_xy[kPairWarps][32];
    __shared__ uint2 s_z[kPairWarps][32];
    __shared__ uint2 s_out[kPairWarps][kAllOut];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.ctr->stamp[kStampStart] = now_ns();
        *ctr_next = Ctr{};
    }
    uint4* xy = s_xy[warp];
    uint2* zz = s_z[warp];
    WarpOut o{s_out[warp], 0, kAllOut};
    const uint32_t n = (uint32_t)p.nboxes, rows = BIP ? p.split : n, cols = BIP ? n - p.split : n;
    const uint32_t* blue = BIP ? (p.blue ? p.blue : p.boxes + (uint64_t)p.split * (2 * D + 1)) : p.boxes;
    const uint32_t first = BIP ? p.split : 0u;  // index of the first column
    const uint32_t R = (rows + 31) >> 5, X = (cols + 31) >> 5;
    // self: the triangle of tiles x >= r folded into rows of F + 1, F = R
    // rounded up to an even number: row k and row F - 1 - k together
    const uint32_t F = (R + 1) & ~1u;
    const uint32_t tasks = BIP ? R * X : F / 2 * (F + 1);
    for (uint32_t task = blockIdx.x * kPairWarps + warp; task < tasks; task += gridDim.x * kPairWarps) {
        uint32_t r, x;
        if (BIP) {
            r = task / X;
            x = task - r * X;
        } else {
            const uint32_t k = task / (F + 1), c = task - k * (F + 1);
            r = c > k ? k : F - 1 - k;
            x = c > k ? c - 1 : F - 1 - c;
            if (r >= R || x >= R) continue;
        }
        const WholeBox<D> me = whole_box<D>(p, p.boxes, 32 * r + lane, rows, BIP ? x == 0 : x == r);
        const WholeBox<D> col = whole_box<D>(p, blue, 32 * x + lane, cols, BIP && r == 0);
        __syncwarp();  // (the last columns are read)
        xy[lane] = make_uint4(col.lo[0], col.hi[0], col.lo[1], col.hi[1]);
        if (D == 3) zz[lane] = make_uint2(col.lo[D - 1], col.hi[D - 1]);
        __syncwarp();
        uint32_t mask = 0;
#pragma unroll
        for (uint32_t j = 0; j < 32; j++) {
            const uint4 c = xy[j];
            bool hit = me.lo[0] <= c.y && c.x <= me.hi[0] && me.lo[1] <= c.w && c.z <= me.hi[1];
            if (D == 3) {
                const uint2 z = zz[j];
                hit = hit && me.lo[D - 1] <= z.y && z.x <= me.hi[D - 1];
            }
            mask |= (hit ? 1u : 0u) << j;
        }
        if (!BIP && x == r) mask &= after_lane();
        const auto id = [&](uint32_t b) { return first + 32 * x + b; };
        wemit<BIP>(p, o, mask, id, 0u, id, 32 * r + lane);
    }
    if (BIP && (R == 0 || X == 0)) {  // one colour: its boxes are still checked
        const uint32_t count = R ? rows : cols;
        for (uint32_t i = blockIdx.x * kPairThreads + threadIdx.x; i < count; i += gridDim.x * kPairThreads)
            whole_box<D>(p, R ? p.boxes : blue, i, count, true);
    }
    wflush<BIP, false>(p, o);
    query_end(p);
}

// ---------------------------------------------------------------------------
// one-launch queries of small scenes: a cooperative launch whose blocks run
// the whole pipeline, phase after phase, separated by grid barriers
//   P0   every block: the cell size (warp 0 runs the tuner's model on 64
//        sampled boxes: the same choice in every block) and the scene in
//        shared memory; block 0 the chosen grid for the host and the next
//        launch's zeroed run counters; the counters are zeroed first only
//        when they may hold anything else (one more barrier)
//   P1   count
//   P2   entry totals of chunks -- a small grid's (128-cell chunks)
//        computed by every block itself, a larger one's (512-cell chunks) by
//        all blocks (one more barrier) -- then the chunk prefixes in shared
//        memory, and each warp's chunks' cell ends, work lists, statistics;
//        a small grid's cell ends go to a buffer of their own, since other
//        blocks may still be reading the counters
//   P3   expand and scatter
//   P4   small, medium and block pair passes; the grid's counters zeroed for
//        the next launch; the last block to finish copies the run counters
//        to the host
// Data written in one phase and read in a later one is read past L1. A
// barrier's wait is bounded: a block that gives up sets kErrWait and leaves,
// and the others give up at their next barrier.
// ---------------------------------------------------------------------------
constexpr uint32_t kFusedThreads = 2 * kPairThreads;
constexpr uint32_t kFusedWarps = kFusedThreads / 32;
constexpr uint32_t kFusedChunks = (uint32_t)(kFusedMaxCells / kScanChunk);
constexpr uint32_t kFusedLocalCells = 8192;  // grids of up to 8192 cells: 128-cell chunks, totals per block
constexpr uint32_t kFusedLeave = 32;  // no cell shift: the query is left to the regular pipeline
constexpr uint32_t kGridWaitLimit = 1u << 20;  // polls of 64 ns or more: the wait ends after a second at most
constexpr uint32_t kSmallWarpBytes = kSmallSlots * sizeof(uint4) + kWarpOut * sizeof(uint2);
static_assert(kFusedChunks % kFusedThreads == 0, "chunk prefixes per thread");

// barrier number k of this launch (k counts the barriers passed so far)
__device__ __forceinline__ bool grid_barrier(const FusedArgs& a, uint32_t k) {
    __shared__ uint32_t s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        const uint32_t target = (k + 1) * gridDim.x;
        uint32_t ok = 0;
        for (uint32_t i = 0; i < kGridWaitLimit; i++) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
            if ((int32_t)(v - a.bar_base) >= (int32_t)target) {
                ok = 1;
                break;
            }
            if (i >= 64) __nanosleep(64);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0u;
}

// The count and the scatter of a one-launch query. A block takes an even part
// of the boxes (at most kFusedThreads at a time) and deals their cells out over
// all its threads, so that a warp whose boxes cover hundreds of cells each does
// not keep the next barrier waiting: on 50 000 red and blue boxes, one in a
// hundred of them large, the last warp of the scatter came 16 us after the
// first (50 us the kernel, 33 with the cells dealt out). A part that is one tile
// stays in shared memory from the count to the scatter.
struct DealtTile {
    uint32_t* rows;  // the boxes' rows, then terms
    uint4* box;      // {first cell, cells along x | along y << 16, and their multipliers}
    uint32_t* ends;  // cells of the boxes up to and with this one
    uint32_t* warp;  // [kFusedThreads / 32]
};
constexpr uint32_t kDealtBytes = kFusedThreads * (7 * sizeof(uint32_t) + sizeof(uint4) + sizeof(uint32_t)) + kFusedWarps * sizeof(uint32_t);
__device__ __forceinline__ DealtTile dealt_tile(unsigned char* m) {
    DealtTile s;
    s.box = reinterpret_cast<uint4*>(m);
    s.rows = reinterpret_cast<uint32_t*>(s.box + kFusedThreads);
    s.ends = s.rows + 7 * kFusedThreads;
    s.warp = s.ends + kFusedThreads;
    return s;
}

// boxes [b0, b0 + nb) into the tile; their cells in all
template <int D, bool REPORT>
__device__ __forceinline__ uint32_t deal_boxes(const Params& p, const DealtTile& s, uint64_t b0, uint32_t nb) {
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    __syncthreads();  // (the last tile is read)
    stage_boxes<D>(p, b0, nb, s.rows);
    __syncthreads();
    BoxCells c;
    if (t < nb) c = box_cells<D, true, REPORT>(p, s.rows + t * (2 * D + 1), b0 + t);
    // (grids of at most 2^20 cells: cells, and cells per axis, in 32 and 16 bits)
    s.box[t] = make_uint4((uint32_t)c.base, c.sx | c.sy << 16, magic_of(c.sx), magic_of(c.sy));
    const uint32_t incl = warp_incl_scan(c.cnt);
    if (lane == 31) s.warp[warp] = incl;
    __syncthreads();
    const uint32_t w = lane < kFusedWarps ? s.warp[lane] : 0u, upto = warp_incl_scan(w);
    s.ends[t] = incl + __shfl_sync(FULL_MASK, upto - w, warp);
    __syncthreads();
    return __shfl_sync(FULL_MASK, upto, 31);
}

template <int D, bool SCATTER>
__device__ __forceinline__ void deal_cells(const Params& p, const DealtTile& s, uint64_t b0, uint32_t total, uint32_t nrc) {
    for (uint32_t e = threadIdx.x; e < total; e += kFusedThreads) {
        uint32_t o = 0;  // the box: the first whose end lies beyond e
#pragma unroll
        for (uint32_t step = kFusedThreads / 2; step; step >>= 1)
            if (s.ends[o + step - 1] <= e) o += step;
        const uint32_t lq = e - (o ? s.ends[o - 1] : 0u), cnt = s.ends[o] - (o ? s.ends[o - 1] : 0u);
        const uint4 b = s.box[o];
        const uint32_t sx = b.y & 0xffffu, sy = b.y >> 16;
        const uint32_t rr = div_magic(lq, sx, b.z), i = lq - rr * sx;
        const uint32_t k = div_magic(rr, sy, b.w), j = rr - k * sy;
        const uint32_t gid = b.x + (k * nrc + j) * nrc + i;
        if (SCATTER) {
            const uint32_t* ob = s.rows + o * (2 * D + 1);
            const uint32_t f = (i == 0 ? 1u : 0u) | (j == 0 ? 2u : 0u) | ((D == 2 || k == 0) ? 4u : 0u);
            const uint4 rec = make_uint4(term_cut(ob[0], i == 0, i + 1 == sx), term_cut(ob[1], j == 0, j + 1 == sy),
                                         D == 3 ? term_cut(ob[2], k == 0, lq + sx * sy >= cnt) : 0u,
                                         (f << kIdBits) | (uint32_t)(b0 + o));
            const uint32_t pos = atomicSub(&p.counts[gid], 1u) - 1u;
            if (pos < p.entry_cap) p.entries[pos] = rec;
            else atomicOr(&p.ctr->err, kErrEntryOvf);
        } else {
            atomicAdd(&p.counts[gid], 1u);
        }
    }
}

// the one-launch queries' cost model for one scene of n boxes at row 0, with T =
// E^2 / 2C on 64 sampled boxes, in single precision over exact integer sums: the
// one-launch path cannot wait for double-precision divisions. Grids of at most
// max_cells cells, so a box covers at most max_cells cells and every per-box
// product fits 32 bits.
template <int dims, bool BIP>
__device__ __forceinline__ uint32_t tune_scene_fast(const Params& p, uint32_t range, uint64_t max_cells, uint32_t warps) {
    const uint32_t lane = lane_id();
    const uint64_t n = p.nboxes;
    const uint64_t m = n < kTuneRows ? n : kTuneRows;
    uint32_t lo[2][3] = {{0, 0, 0}, {0, 0, 0}}, hi[2][3] = {{0, 0, 0}, {0, 0, 0}};
    bool ok[2] = {false, false};
    unsigned long long ext = 0, good = 0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const uint64_t k = lane + 32u * j;
        if (k >= m) continue;
        const uint32_t* b = box_row<dims>(p.boxes, p.blue, p.split, (uint32_t)(k * n / m));
        bool v = true;
        for (int d = 0; d < dims; d++) {
            lo[j][d] = __ldg(b + 2 * d);
            hi[j][d] = __ldg(b + 2 * d + 1);
            v = v && lo[j][d] <= hi[j][d] && hi[j][d] < range;
        }
        ok[j] = v;
        if (v) {
            for (int d = 0; d < dims; d++) ext += (unsigned long long)(hi[j][d] - lo[j][d]) + 1;
            good++;
        }
    }
    ext = warp_sum_u64(ext);
    good = warp_sum_u64(good);
    // s0 = floor(log2(mean extent)), 0 below 2
    const unsigned long long mean = ext / ((good ? good : 1ull) * (unsigned long long)dims);
    const int s0 = mean < 2 ? 0 : 63 - __clzll(mean);
    const int s_win = s0 + 3 < 31 ? s0 + 3 : 31;
    // red and blue boxes too sparse in their range for these grids: the regular
    // pipeline's, unless it took a coarser grid itself
    if (BIP && tune_grid<dims>(range, (uint32_t)s_win) > max_cells && tune_grid<dims>(range, (uint32_t)s_win) <= kQueryMaxCells)
        return kFusedLeave;
    const float scale = (float)n / (float)(m ? m : 1);
    const uint64_t far_cap = n * 64 > 4096 ? n * 64 : 4096;
    uint32_t best = 0xffffffffu;
    // the window, then every coarser size if none of it qualifies: entries counted
    // in integers, size after size, and weighed side by side, a lane a size
    for (int pass = 0; pass < 2 && best == 0xffffffffu && m > 0; pass++) {
        const int first = pass ? s_win + 1 : s0 - 2 > 0 ? s0 - 2 : 0, last = pass ? 31 : s_win;
        const uint64_t limit = pass ? mn64(max_cells, far_cap) : max_cells;
        uint32_t entries = 0xffffffffu;  // lane s - first: the sample's at shift s, if it qualifies
        for (int s = first; s <= last; s++) {
            if (tune_grid<dims>(range, (uint32_t)s) > limit) continue;
            uint32_t e = 0;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                if (!ok[j]) continue;
                uint32_t c = 1;
                for (int d = 0; d < dims; d++) c *= (hi[j][d] >> s) - (lo[j][d] >> s) + 1;
                e += c;  // <= 2 * max_cells
            }
            e = __reduce_add_sync(FULL_MASK, e);
            if ((int)lane == s - first && e <= 64u * (uint32_t)m) entries = e;
            if (nrc_dev(range, s) <= 1u) break;  // (coarser ones are this cell again)
        }
        uint32_t bits = 0x7f800000u;  // of the cost (positive floats are in the order of their bits)
        if (entries != 0xffffffffu) {
            const uint64_t C = tune_grid<dims>(range, (uint32_t)first + lane);
            const float E = (float)entries * scale, Cf = (float)C;
            const float T = E * E / (2.0f * Cf);
            // (fewer cells than warps leave warps idle: 30 000 boxes of one
            // density took 35 us on 512 cells and 26 us on 4096)
            const float l = E / Cf, l3 = l * l * l;
            // (a cell of l boxes has about l^2 / 16384 tile tasks, a warp's each)
            const float units = Cf * fmaxf(1.0f, l * l * (1.0f / 16384.0f));
            const float idle = (float)warps > units ? (float)warps / units : 1.0f;
            bits = __float_as_uint((C > kFusedLocalCells ? (float)kFusedGrid : 0.0f) + (float)kQueryCell * Cf + (float)kQueryEntry * E +
                                   (float)kFusedCell * Cf * (l3 / (l3 + (float)kFusedShare)) +
                                   (BIP ? 0.5f : 1.0f) * (float)kFusedTest * idle * T);
        }
        const uint32_t least = __reduce_min_sync(FULL_MASK, bits);
        // (the finest on a tie)
        if (least < 0x7f800000u) best = (uint32_t)first + __ffs(__ballot_sync(FULL_MASK, bits == least)) - 1u;
    }
    if (best == 0xffffffffu) {  // the coarsest grid that is not a single cell
        uint32_t s = 31;
        while (s > 0 && nrc_dev(range, (int)s - 1) <= 1) s--;
        best = s;
    }
    return best;
}

template <int D, bool BIP>
__global__ void __launch_bounds__(kFusedThreads, 1) k_fused(Params pin, FusedArgs a) {
    Params p = pin;  // the grid's size is set below
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_shift;
    __shared__ Scene s_scene[2];
    __shared__ uint32_t s_off[3];
    __shared__ unsigned long long s_wsum[kFusedWarps];
    __shared__ uint32_t s_csum[kFusedLocalCells / 128];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint64_t blk = blockIdx.x, nblk = gridDim.x;
    const uint64_t gw = blk * kFusedWarps + warp, nw = nblk * kFusedWarps;
    const uint64_t gt = blk * kFusedThreads + t, nt = nblk * kFusedThreads;
    const uint32_t range = p.max_range;
    uint32_t nbar = 0;
    if (blk == 0 && t == 0) p.ctr->t_start = now_ns();
#define FUSED_BARRIER()                                        \
    if (!grid_barrier(a, nbar++)) {                            \
        if (t == 0) atomicOr(&p.ctr->err, (unsigned)kErrWait); \
        return;                                                \
    }
    // P0
    if (warp == 0) {
        uint32_t sh = a.shift;
        if (sh == kFusedTune) sh = tune_scene_fast<D, BIP>(p, range, kFusedMaxCells, (uint32_t)nw);
        if (lane == 0) s_shift = sh;
    }
    __syncthreads();
    const bool leave = BIP && s_shift == kFusedLeave;  // (the same in every block)
    const uint32_t shift = leave ? 0u : s_shift, nrc = leave ? 0u : nrc_dev(range, (int)shift);
    p.ncells = D == 3 ? (uint64_t)nrc * nrc * nrc : (uint64_t)nrc * nrc;
    if (t == 0) {
        const uint32_t red = BIP ? p.split : (uint32_t)p.nboxes;
        s_scene[0] = Scene{0u, red, shift, nrc, 0ull, range, 0u};
        s_off[0] = 0u;
        s_off[1] = red;
        if (BIP) {
            s_scene[1] = Scene{red, (uint32_t)p.nboxes - red, shift, nrc, 0ull, range, 0u};
            s_off[2] = (uint32_t)p.nboxes;
        }
    }
    if (blk == 0 && t == 0) {
        *a.ctr_next = Ctr{};
        p.ctr->cells = p.ncells;
        p.ctr->shift = shift;
        if (leave) atomicOr(&p.ctr->err, (unsigned)kErrGridRoom);
    }
    __syncthreads();
    p.open = shift >= kOpenShift ? 1u : 0u;
    p.scenes = s_scene;  // the count and the scatter read the scenes from shared memory
    p.scene_box_off = s_off;
    unsigned long long total = 0;
    bool fits = false;
    if (!leave) {
    if (a.zero_cells) {
        uint4* c4 = reinterpret_cast<uint4*>(p.counts);
        for (uint64_t i = gt; i < a.zero_cells / 4; i += nt) c4[i] = make_uint4(0u, 0u, 0u, 0u);
        for (uint64_t i = 4 * (a.zero_cells / 4) + gt; i < a.zero_cells; i += nt) p.counts[i] = 0u;
        FUSED_BARRIER()
    }
    // P1: count
    const DealtTile tile = dealt_tile(smem_raw);
    const uint64_t part = ((p.nboxes + nblk - 1) / nblk + 3) & ~3ull;  // (parts begin at multiples of 16 bytes)
    const uint64_t part0 = mn64(blk * part, p.nboxes), part1 = mn64(part0 + part, p.nboxes);
    uint32_t dealt = 0;
    for (uint64_t b0 = part0; b0 < part1; b0 += kFusedThreads) {
        dealt = deal_boxes<D, true>(p, tile, b0, (uint32_t)mn64(kFusedThreads, part1 - b0));
        deal_cells<D, false>(p, tile, b0, dealt, nrc);
    }
    FUSED_BARRIER()
    // P2: chunk entry totals and prefixes, then the cells
    uint32_t* pre = reinterpret_cast<uint32_t*>(smem_raw + kDealtBytes);  // (the tile stays)
    if (p.ncells <= kFusedLocalCells) {
        const uint32_t nch = (uint32_t)((p.ncells + 127) / 128);
        for (uint32_t ch = warp; ch < nch; ch += kFusedWarps) {
            uint32_t v[4];
            scan_load<1, true>(p, ch, v);
            s_csum[ch] = __reduce_add_sync(FULL_MASK, v[0] + v[1] + v[2] + v[3]);  // < 2^32 (at most 2^25)
        }
        __syncthreads();
        if (t == 0) {
            unsigned long long run = 0;
            for (uint32_t ch = 0; ch < nch; ch++) {
                pre[ch] = (uint32_t)run;  // < entry_cap when it is used
                run += s_csum[ch];
            }
            s_wsum[0] = run;
        }
        __syncthreads();
        total = s_wsum[0];
        fits = total <= p.entry_cap;
        if (fits) {
            // the cell ends go to a buffer of their own: other blocks may
            // still be summing the counters
            Params pe = p;
            pe.counts = a.ends;
            ScanStats ws;
            const uint64_t full = p.ncells / 128;
            for (uint64_t ch = gw; ch < nch; ch += nw) {
                uint32_t v[4];
                scan_load<1, true>(p, ch, v);
                scan_chunk<1>(pe, pin, ch, ch < full, v, pre[ch], ws);
            }
            scan_stats_flush(p, ws);
        }
    } else {
        const uint64_t nch = (p.ncells + kScanChunk - 1) / kScanChunk;
        for (uint64_t ch = gw; ch < nch; ch += nw) {
            uint32_t v[kScanPerThread];
            scan_load<4, true>(p, ch, v);
            uint32_t sum = 0;  // < 2^32: a chunk holds at most 512 cells of at most kFusedMaxBoxes entries
#pragma unroll
            for (int k = 0; k < kScanPerThread; k++) sum += v[k];
            sum = __reduce_add_sync(FULL_MASK, sum);
            if (lane == 0) a.chunk_sum[ch] = sum;
        }
        FUSED_BARRIER()
        constexpr uint32_t kPer = kFusedChunks / kFusedThreads;
        uint32_t x[kPer];
        unsigned long long sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            const uint64_t i = (uint64_t)t * kPer + k;
            x[k] = i < nch ? __ldcg(a.chunk_sum + i) : 0u;
            sum += x[k];
        }
        const unsigned long long incl = warp_incl_scan64(sum);
        if (lane == 31) s_wsum[warp] = incl;
        __syncthreads();
        unsigned long long run = incl - sum;
#pragma unroll
        for (uint32_t w = 0; w < kFusedWarps; w++) {
            if (w < warp) run += s_wsum[w];
            total += s_wsum[w];
        }
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            const uint64_t i = (uint64_t)t * kPer + k;
            if (i < nch) pre[i] = (uint32_t)run;  // < entry_cap when it is used
            run += x[k];
        }
        __syncthreads();
        fits = total <= p.entry_cap;
        if (fits) {
            ScanStats ws;
            const uint64_t full = p.ncells / kScanChunk;
            for (uint64_t ch = gw; ch < nch; ch += nw) {
                uint32_t v[kScanPerThread];
                scan_load<4, true>(p, ch, v);
                scan_chunk(p, pin, ch, ch < full, v, pre[ch], ws);
            }
            scan_stats_flush(p, ws);
        }
    }
    if (blk == 0 && t == 0) {
        p.ctr->entries = total;
        if (!fits) atomicOr(&p.ctr->err, (unsigned)kErrEntryOvf);
    }
    FUSED_BARRIER()
    // P3: tile tasks of huge cells, scatter (against the cell ends)
    if (fits) {
        expand_cells(p, pin, __ldcg(&p.ctr->n_list[kListHuge]), (uint32_t)gw, (uint32_t)nw);
        Params pe = p;
        if (p.ncells <= kFusedLocalCells) pe.counts = a.ends;
        for (uint64_t b0 = part0; b0 < part1; b0 += kFusedThreads) {
            if (part > kFusedThreads) dealt = deal_boxes<D, false>(pe, tile, b0, (uint32_t)mn64(kFusedThreads, part1 - b0));
            deal_cells<D, true>(pe, tile, b0, dealt, nrc);
        }
    }
    FUSED_BARRIER()
    }
#undef FUSED_BARRIER
    // P4: the counters zeroed for the next launch (the pair passes read the
    // work lists, not the counters), then the pairs
    {
        uint4* c4 = reinterpret_cast<uint4*>(p.counts);
        for (uint64_t i = gt; i < p.ncells / 4; i += nt) c4[i] = make_uint4(0u, 0u, 0u, 0u);
        for (uint64_t i = 4 * (p.ncells / 4) + gt; i < p.ncells; i += nt) p.counts[i] = 0u;
    }
    __shared__ uint32_t s_sizes[kNumLists + 1];
    p.list_sizes = s_sizes;
    if (t <= (uint32_t)kNumLists)
        s_sizes[t] = __ldcg(t < (uint32_t)kNumLists ? &p.ctr->n_list[t] : &p.ctr->need_tasks);
    __syncthreads();  // (the sizes are there and the tile is read)
    if (fits) {
        uint4* ws = reinterpret_cast<uint4*>(smem_raw + warp * kSmallWarpBytes);
        small_pass<D, BIP, false, true>(p, ws, reinterpret_cast<uint2*>(ws + kSmallSlots), gw, nw);
        __syncthreads();
        med_pass<D, BIP, false, true>(p, smem_raw + warp * kMedWarpBytes, gw, nw);
        __syncthreads();
        constexpr uint32_t kTeams = kFusedThreads / kTeamThreads;
        team_pass<D, BIP, false, true, true>(p, reinterpret_cast<TeamSmem*>(smem_raw)[t / kTeamThreads],
                                               blk * kTeams + t / kTeamThreads, nblk * kTeams);
    }
    // the last block to finish copies the run counters to the host (one
    // more arrival per block on the barriers' count)
    __syncthreads();
    if (t == 0) {
        __threadfence();
        uint32_t old;
        asm volatile("atom.acq_rel.gpu.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.bar) : "memory");
        if ((int32_t)(old - a.bar_base) == (int32_t)((nbar + 1) * nblk - 1)) {
            __threadfence();
            ctr_to_host(p.ctr, a.ctr_host);
            a.ctr_host->barriers = nbar + 1;
            a.ctr_host->t_end = now_ns();
            __threadfence_system();
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static int g_blocks_small = 1, g_blocks_med = 1, g_blocks_block = 1;
static int g_sm_count = 0;

static size_t med_smem() { return (size_t)kPairWarps * kMedWarpBytes; }

template <int D, bool B, bool R = false>
static cudaError_t init_variant() {
    cudaError_t e = cudaFuncSetAttribute(k_pairs_med<D, B, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)med_smem());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_pairs_block<D, B, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TeamSmem));
    return e;
}

static int g_fused_blocks = 0;

static size_t fused_smem() {
    size_t b = (size_t)kFusedWarps * kMedWarpBytes;
    const size_t team = sizeof(TeamSmem) * (kFusedThreads / kTeamThreads);
    b = b > team ? b : team;
    b = b > (size_t)kFusedWarps * kSmallWarpBytes ? b : (size_t)kFusedWarps * kSmallWarpBytes;
    b = b > kDealtBytes + (size_t)kFusedChunks * 4 ? b : kDealtBytes + (size_t)kFusedChunks * 4;
    return b;
}

int fused_blocks() { return g_fused_blocks; }

cudaError_t launch_all_pairs(const Params& p, Ctr* ctr_next, int dims, cudaStream_t st) {
    const uint64_t red = p.split == kNoSplit ? p.nboxes : p.split, blue = p.nboxes - (p.split == kNoSplit ? 0 : p.split);
    const uint64_t R = (red + 31) / 32, X = (blue + 31) / 32;
    const uint64_t tiles = p.split == kNoSplit ? R * (R + 1) / 2 : R * X, cap = (uint64_t)(g_sm_count > 0 ? g_sm_count : 152) * 2;
    const uint64_t b = (tiles + kPairWarps - 1) / kPairWarps;
    const unsigned g = (unsigned)(b < cap ? (b ? b : 1) : cap);
    if (p.split != kNoSplit) {
        if (dims == 2) k_all_pairs<2, true><<<g, kPairThreads, 0, st>>>(p, ctr_next);
        else k_all_pairs<3, true><<<g, kPairThreads, 0, st>>>(p, ctr_next);
    } else {
        if (dims == 2) k_all_pairs<2, false><<<g, kPairThreads, 0, st>>>(p, ctr_next);
        else k_all_pairs<3, false><<<g, kPairThreads, 0, st>>>(p, ctr_next);
    }
    return cudaGetLastError();
}

template <int D, bool B>
static cudaError_t launch_fused_t(const Params& p, const FusedArgs& a, cudaStream_t st) {
    Params pp = p;
    FusedArgs aa = a;
    void* args[] = {&pp, &aa};
    return cudaLaunchCooperativeKernel((const void*)k_fused<D, B>, dim3((unsigned)g_fused_blocks), dim3(kFusedThreads),
                                      args, fused_smem(), st);
}

cudaError_t launch_fused(const Params& p, const FusedArgs& a, int dims, cudaStream_t st) {
    if (g_fused_blocks <= 0) return cudaErrorNotSupported;
    if (p.split != kNoSplit) return dims == 2 ? launch_fused_t<2, true>(p, a, st) : launch_fused_t<3, true>(p, a, st);
    return dims == 2 ? launch_fused_t<2, false>(p, a, st) : launch_fused_t<3, false>(p, a, st);
}

template <int D, bool B>
static cudaError_t init_fused() {
    return cudaFuncSetAttribute(k_fused<D, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem());
}

cudaError_t kernels_init() {
    cudaError_t e;
    {
        int dev = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    }
    if ((e = init_variant<2, false>()) != cudaSuccess) return e;
    if ((e = init_variant<3, false>()) != cudaSuccess) return e;
    if ((e = init_variant<2, true>()) != cudaSuccess) return e;
    if ((e = init_variant<3, true>()) != cudaSuccess) return e;
    if ((e = init_variant<2, false, true>()) != cudaSuccess) return e;
    if ((e = init_variant<3, false, true>()) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_scene_hist<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kGroupScenes * sizeof(uint32_t)))) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_group_by_scene<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kGroupScenes * kGroupBytes))) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_tune_query<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTuneSmem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_tune_query<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTuneSmem)) != cudaSuccess) return e;
    int nb = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pairs_small<3, false>, kPairThreads, 0)) != cudaSuccess) return e;
    g_blocks_small = nb > 0 ? nb : 1;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pairs_med<3, false>, kPairThreads, med_smem())) != cudaSuccess) return e;
    g_blocks_med = nb > 0 ? nb : 1;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pairs_block<3, false>, kTeamThreads, sizeof(TeamSmem))) != cudaSuccess) return e;
    g_blocks_block = nb > 0 ? nb : 1;
    // one-launch queries: one block per SM, all resident (cooperative launch)
    if ((e = init_fused<2, false>()) != cudaSuccess) return e;
    if ((e = init_fused<3, false>()) != cudaSuccess) return e;
    if ((e = init_fused<2, true>()) != cudaSuccess) return e;
    if ((e = init_fused<3, true>()) != cudaSuccess) return e;
    {
        int dev = 0, coop = 0, nf = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return e;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nf, k_fused<3, true>, kFusedThreads, fused_smem())) !=
            cudaSuccess)
            return e;
        g_fused_blocks = coop && nf >= 1 ? g_sm_count : 0;
    }
    return cudaSuccess;
}

uint64_t scene_table_entries(uint64_t nboxes) { return (nboxes >> kSceneTableShift) + 2; }

cudaError_t launch_scene_table(const Params& p, cudaStream_t st) {
    const uint64_t n = scene_table_entries(p.nboxes);
    const uint64_t cap = (uint64_t)(g_sm_count > 0 ? g_sm_count : 152) * 4;
    const uint64_t g = (n + 255) / 256;
    k_scene_table<<<(unsigned)(g < cap ? g : cap), 256, 0, st>>>(p);
    return cudaGetLastError();
}

static unsigned box_grid(uint64_t nboxes) {
    const uint64_t nb = (nboxes + kBoxThreads - 1) / kBoxThreads;
    const uint64_t cap = (uint64_t)(g_sm_count > 0 ? g_sm_count : 152) * 8;
    return (unsigned)(nb < cap ? nb : cap);
}

cudaError_t launch_count(const Params& p, int dims, cudaStream_t st, bool chained, bool after_kernel) {
    const unsigned sms = (unsigned)(g_sm_count > 0 ? g_sm_count : 152), g = box_grid(p.nboxes);
    cudaError_t e = launch_after(chained && after_kernel, k_zero_counts, sms * 4, 512, 0, st, p);
    if (e != cudaSuccess || g == 0) return e;
    auto* k = p.merged ? (dims == 2 ? k_count<2, true> : k_count<3, true>) : (dims == 2 ? k_count<2, false> : k_count<3, false>);
    return launch_after(chained, k, g, kBoxThreads, 0, st, p);
}

cudaError_t launch_scatter(const Params& p, int dims, cudaStream_t st, bool chained) {
    const unsigned g = box_grid(p.nboxes);
    if (g == 0) return cudaSuccess;
    auto* k = p.merged ? (dims == 2 ? k_scatter<2, true> : k_scatter<3, true>)
                       : (dims == 2 ? k_scatter<2, false> : k_scatter<3, false>);
    return launch_after(chained, k, g, kBoxThreads, 0, st, p);
}

cudaError_t launch_scan(const Params& p, cudaStream_t st, bool chained) {
    const uint64_t chunks = (p.ncells + kScanChunk - 1) / kScanChunk;
    const uint64_t blocks = (chunks + kScanThreads / 32 - 1) / (kScanThreads / 32);
    const uint64_t sms = (uint64_t)(g_sm_count > 0 ? g_sm_count : 152);
    const uint64_t cap = sms * 4;  // resident: 4 blocks per SM
    const unsigned g = (unsigned)(blocks < cap ? (blocks ? blocks : 1) : cap);
    // reduce: two chunks per warp item, 4 resident blocks per SM
    const uint64_t rblocks = (chunks + 2 * (kReduceThreads / 32) - 1) / (2 * (kReduceThreads / 32));
    const unsigned g2 = (unsigned)(rblocks < cap ? (rblocks ? rblocks : 1) : cap);
    const cudaError_t e = launch_after(chained, k_scan_reduce, g2, kReduceThreads, 0, st, p);
    return e != cudaSuccess ? e : launch_after(chained, k_scan_cells, g, kScanThreads, 0, st, p);
}

cudaError_t launch_least_shift(const TuneArgs& a, int dims, unsigned int* least, cudaStream_t st) {
    const uint64_t blocks = (a.n + 255) / 256, cap = (uint64_t)(g_sm_count > 0 ? g_sm_count : 152) * 8;
    const unsigned g = (unsigned)(blocks < cap ? (blocks ? blocks : 1) : cap);
    if (dims == 2) k_least_shift<2><<<g, 256, 0, st>>>(a, least);
    else k_least_shift<3><<<g, 256, 0, st>>>(a, least);
    return cudaGetLastError();
}

cudaError_t launch_tune_query(const Params& p, const TuneArgs& a, int dims, cudaStream_t st) {
    const unsigned blocks = a.shift == kTuneShift ? kTuneBlocks : 1u;
    if (dims == 2) k_tune_query<2><<<blocks, kTuneThreads, kTuneSmem, st>>>(p, a);
    else k_tune_query<3><<<blocks, kTuneThreads, kTuneSmem, st>>>(p, a);
    return cudaGetLastError();
}

cudaError_t launch_tune_scenes(const uint32_t* boxes, const unsigned long long* offs, uint32_t nscenes, int dims,
                               uint32_t range, SceneTune* out, cudaStream_t st) {
    if (nscenes == 0) return cudaSuccess;
    const uint64_t cap = (uint64_t)(g_sm_count > 0 ? g_sm_count : 152) * 32;  // a warp per block: scenes on SMs of their own
    k_tune_scenes<<<(unsigned)(nscenes < cap ? nscenes : cap), 32, 0, st>>>(boxes, offs, nscenes, dims, range, out);
    return cudaGetLastError();
}

template <int D, bool B, bool R = false>
static cudaError_t launch_pairs_t(const Params& p, int sm_count, cudaStream_t st, const PairOverlap* ov, bool chained) {
    if (ov && !R && ov->side_sms > 0 && ov->side_sms < sm_count) {
        cudaError_t e;
        Params q = p;
        q.ctr_host = nullptr;  // the query ends behind both streams
        if ((e = cudaEventRecord(ov->fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(ov->side, ov->fork, 0)) != cudaSuccess) return e;
        k_pairs_small<D, B, R><<<ov->side_sms * g_blocks_small, kPairThreads, 0, ov->side>>>(q);
        k_pairs_block<D, B, R><<<ov->side_sms * g_blocks_block, kTeamThreads, sizeof(TeamSmem), ov->side>>>(q);
        k_pairs_med<D, B, R><<<(sm_count - ov->side_sms) * g_blocks_med, kPairThreads, med_smem(), st>>>(q);
        if ((e = cudaEventRecord(ov->join, ov->side)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(st, ov->join, 0)) != cudaSuccess) return e;
        k_query_end<<<1, 32, 0, st>>>(p);
        return cudaGetLastError();
    }
    cudaError_t e = launch_after(chained, k_pairs_small<D, B, R>, sm_count * g_blocks_small, kPairThreads, 0, st, p);
    if (e == cudaSuccess)
        e = launch_after(chained, k_pairs_med<D, B, R>, sm_count * g_blocks_med, kPairThreads, med_smem(), st, p);
    if (e == cudaSuccess)
        e = launch_after(chained, k_pairs_block<D, B, R>, sm_count * g_blocks_block, kTeamThreads, sizeof(TeamSmem), st, p);
    if (e != cudaSuccess) return e;
    if (R) k_strip_entries<<<(unsigned)(sm_count * 4), 512, 0, st>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_pairs(const Params& p, int dims, int sm_count, cudaStream_t st, const PairOverlap* ov, bool chained) {
    const bool bip = p.split != kNoSplit;
    if (p.records) {  // record mode: self queries
        if (bip) return cudaErrorInvalidValue;
        return dims == 2 ? launch_pairs_t<2, false, true>(p, sm_count, st, ov, chained)
                         : launch_pairs_t<3, false, true>(p, sm_count, st, ov, chained);
    }
    if (dims == 2) return bip ? launch_pairs_t<2, true>(p, sm_count, st, ov, chained) : launch_pairs_t<2, false>(p, sm_count, st, ov, chained);
    return bip ? launch_pairs_t<3, true>(p, sm_count, st, ov, chained) : launch_pairs_t<3, false>(p, sm_count, st, ov, chained);
}

static unsigned group_blocks() { return (unsigned)((g_sm_count > 0 ? g_sm_count : 152) * 2); }

size_t group_count_bytes(uint32_t nscenes) {
    return nscenes <= kGroupScenes ? (size_t)group_blocks() * nscenes * sizeof(uint32_t) : 0;
}

cudaError_t launch_group_by_scene(const Params& p, const GroupArgs& g, cudaStream_t st, bool chained) {
    // the pair count is read on the device; the scenes may be fewer than p.nscenes
    const bool local = p.nscenes <= kGroupScenes;
    const size_t n = local ? p.nscenes : 0;
    const unsigned blocks = group_blocks();
    cudaError_t e = launch_after(chained, local ? k_scene_hist<true> : k_scene_hist<false>, blocks, kGroupThreads,
                                 n * sizeof(uint32_t), st, p, g.hist, local ? g.block_counts : nullptr);
    if (e == cudaSuccess)
        e = launch_after<Params, const unsigned long long*, unsigned long long*, unsigned long long*>(
            chained, k_scene_offsets, 1, 1024, 0, st, p, g.hist, g.off, g.off_host);
    if (e != cudaSuccess) return e;
    Params q = p;
    q.ctr_host = g.ctr_host;  // the query ends here
    return launch_after<Params, const unsigned long long*, unsigned long long*, const uint32_t*, uint2*>(
        chained, local ? k_group_by_scene<true> : k_group_by_scene<false>, blocks, kGroupThreads, n * kGroupBytes, st, q, g.off,
        g.cursor, local ? g.block_counts : nullptr, g.dst);
}

}  // namespace pbig
