// Resident scenes and incremental updates (pbig2_scene_*).
//
// A scene keeps its boxes, a grid and its full pair list on the device. The
// grid gives every cell a capacity above its count (slack), so that moving a
// few boxes re-bins only those boxes: their entries become tombstones in the
// cells they leave and go into the slack of the cells they enter. The pairs
// that moved boxes have after the move are found by testing each against the
// entries of its own cells (those they had before are the full list's, or
// without one are found in the same way) with the same closed-interval test
// and reference-cell rule as the full query (src/pbig/pbig.cu:562-603); a pair
// of two moved boxes is reported once, from the box with the smaller index.
// The full list follows as (old list minus every pair touching a moved box)
// plus the pairs after.
// Every slot of the grid holds the box's coordinates next to its index (32
// bytes), so testing a cell reads it contiguously with no gather, and a new
// entry first takes a tombstone of its cell. A cell whose slack runs out
// rebuilds the grid from the current boxes.
#include <cstdio>
#include <cstring>
#include <vector>

#include "engine.h"

namespace pbig {

constexpr uint32_t kDead = 0xffffffffu;

struct alignas(16) ResCtr {
    unsigned int err;                // kErr* bits
    unsigned int overflow;           // a cell ran out of slack
    unsigned long long rem;          // pairs of the moved boxes before the move (may exceed capacity)
    unsigned long long add;          // and after it (may exceed capacity)
    unsigned long long full;         // pairs of the full list after the move
    unsigned int done;               // blocks of the last kernel that finished
    unsigned int wide;               // a box covers more cells than it may (k_res_count)
    unsigned long long sum;          // slots of the cells (k_res_caps)
};

struct ResGrid {
    const uint32_t* boxes;
    uint64_t nboxes;
    uint32_t shift, nrc, range;
    uint64_t ncells, nslots;
    uint32_t* start;     // [ncells + 1] capacity region of each cell
    uint32_t* used;      // [ncells] slots used (live entries and tombstones)
    uint4* entries;      // two per slot: {x0, x1, y0, y1}, {z0, z1, start bits << 29 | box index (kDead: free), 0}
    ResCtr* ctr;
};

// slack of a cell of n boxes
__host__ __device__ __forceinline__ uint32_t res_cap(uint32_t n) { return n + (n >> 1) + 4u; }
// the starts are 32-bit words, the last of them the number of slots
constexpr uint64_t kMaxSlots = 0xffffffffull;

__device__ __forceinline__ void res_sum(unsigned long long* sum, unsigned long long x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31u) == 0 && x) atomicAdd(sum, x);
}

template <int D>
__device__ __forceinline__ void res_range(const uint32_t* b, uint32_t sh, uint32_t lo[3], uint32_t hi[3]) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] = d < D ? b[2 * d] >> sh : 0u;
        hi[d] = d < D ? b[2 * d + 1] >> sh : 0u;
    }
}

__device__ __forceinline__ uint64_t res_gid(const ResGrid& g, uint32_t i, uint32_t j, uint32_t k) {
    return ((uint64_t)k * g.nrc + j) * g.nrc + i;
}

// one thread per box: count its cells, unless they are more than `widest` (ctr->wide)
template <int D>
__global__ void k_res_count(ResGrid g, uint32_t* cnt, uint32_t widest) {
    constexpr int W = 2 * D + 1;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < g.nboxes; t += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t lo[3], hi[3];
        res_range<D>(g.boxes + t * W, g.shift, lo, hi);
        uint64_t c = 1;  // (at most the grid's cells: below 2^32)
        for (int d = 0; d < D; d++) c *= (uint64_t)(hi[d] - lo[d]) + 1;
        if (c > widest) {
            atomicOr(&g.ctr->wide, 1u);
            continue;
        }
        for (uint32_t k = lo[2]; k <= hi[2]; k++)
            for (uint32_t j = lo[1]; j <= hi[1]; j++)
                for (uint32_t i = lo[0]; i <= hi[0]; i++) atomicAdd(&cnt[res_gid(g, i, j, k)], 1u);
    }
}

__global__ void k_res_caps(const uint32_t* cnt, uint32_t* cap, uint64_t ncells, ResCtr* ctr) {
    unsigned long long sum = 0;
    for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t x = res_cap(cnt[c]);
        cap[c] = x;
        sum += x;
    }
    res_sum(&ctr->sum, sum);
}

// ends (in place of the capacities, after the scan) -> starts; used = 0
__global__ void k_res_starts(const uint32_t* cnt, const uint32_t* ends, ResGrid g) {
    for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < g.ncells; c += (uint64_t)gridDim.x * blockDim.x) {
        g.start[c] = ends[c] - res_cap(cnt[c]);
        g.used[c] = 0;
        if (c == g.ncells - 1) g.start[g.ncells] = ends[c];
    }
}

// the slot pair of a box in one cell
template <int D>
__device__ __forceinline__ void res_slot(const uint32_t* b, uint32_t idw, uint4& e0, uint4& e1) {
    e0 = make_uint4(b[0], b[1], b[2], b[3]);
    e1 = make_uint4(D == 3 ? b[4] : 0u, D == 3 ? b[5] : 0u, idw, 0u);
}

// build: every box (one thread each) appended to its cells (and nothing outside
// the slots, whatever the scan made of the starts)
template <int D>
__global__ void k_res_fill(ResGrid g) {
    constexpr int W = 2 * D + 1;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < g.nboxes; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t* b = g.boxes + t * W;
        uint32_t lo[3], hi[3];
        res_range<D>(b, g.shift, lo, hi);
        for (uint32_t kk = lo[2]; kk <= hi[2]; kk++)
            for (uint32_t j = lo[1]; j <= hi[1]; j++)
                for (uint32_t i = lo[0]; i <= hi[0]; i++) {
                    const uint64_t c = res_gid(g, i, j, kk);
                    const uint32_t f = (i == lo[0] ? 1u : 0u) | (j == lo[1] ? 2u : 0u) | (kk == lo[2] ? 4u : 0u);
                    const uint32_t slot = atomicAdd(&g.used[c], 1u);
                    if (slot < g.start[c + 1] - g.start[c] && (uint64_t)g.start[c] + slot < g.nslots) {
                        uint4 e0, e1;
                        res_slot<D>(b, (f << kIdBits) | (uint32_t)t, e0, e1);
                        g.entries[2 * (uint64_t)(g.start[c] + slot)] = e0;
                        g.entries[2 * (uint64_t)(g.start[c] + slot) + 1] = e1;
                    } else {
                        atomicOr(&g.ctr->overflow, 1u);
                    }
                }
    }
}

__device__ __forceinline__ bool res_moved(const uint32_t* bits, uint32_t id) { return (bits[id >> 5] >> (id & 31u)) & 1u; }

// ---------------------------------------------------------------------------
// A move is four kernels and one wait: check and mark; entries that stay in
// their cells or leave them, beside the split of the full list into the pairs
// that stay and the pairs these boxes had; insertion; pairs after. (Without a
// full list the pairs before are found as those after are, in a kernel of
// their own.)
// Each looks at the counters of the ones before it and does nothing where
// those found an error, a buffer too small or a cell without slack: the host
// reads the counters once, at the end, and repeats what is missing with more
// room. The kernels are chained (chain_wait). Nine kernels with five waits, the
// pairs before by a query, took 234 us for 10 485 of a million boxes, 120 of
// them in kernels; these took 80 and 53, on the finer grid (build_first) 70, and
// chained 63.
struct Move {
    ResGrid g;
    const uint32_t* idx;  // [k] listed boxes
    uint32_t* nb;         // [k] their new rows; once they have moved, their old ones
    uint64_t k;
    uint32_t* moved;      // one bit per box of the scene
    uint2* rem;
    uint2* add;
    uint64_t rem_cap, add_cap;
    const uint2* old_full;  // (null: no full list is kept)
    uint2* full;            // room for nold + add_cap pairs
    uint64_t nold;
    ResCtr* host;           // page-locked: the counters after the last kernel
};

// (blocks of 4 warps, 10 to an SM, each lane two slots in flight: a move of
// 10 485 of a million boxes 87 us; 8 warps, 4 blocks and four slots 90; 2
// warps, 16 blocks and four slots 89)
constexpr int kResThreads = 128;
constexpr int kResBlocks = 10;
constexpr int kResPer = 2;
constexpr int kResWarps = kResThreads / 32;
constexpr uint32_t kResBuf = 256;  // pairs per warp buffer

// What the kernels before found, in one load of 16 bytes that the L1 keeps
// (nothing else changes these words while a kernel depends on them): with
// three loads from the L2 in every warp, the line they share took 31 000
// requests a kernel and 12 of the last kernel's 33 us.
struct MoveState {
    bool bad, no_slack;
    uint64_t rem;
};
__device__ __forceinline__ MoveState move_state(const Move& m) {
    const uint4 w = *reinterpret_cast<const uint4*>(m.g.ctr);
    return MoveState{w.x != 0u, w.y != 0u, (uint64_t)w.w << 32 | w.z};
}

// validate the new records (rid = listed index < n, coordinates < range,
// min <= max) and mark the listed boxes; an index listed twice is an error
template <int D>
__global__ void k_move_check(Move m) {
    constexpr int W = 2 * D + 1;
    chain_wait();
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m.k; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t* b = m.nb + t * W;
        const uint32_t id = m.idx[t];
        uint32_t err = 0;
        if (id >= m.g.nboxes || b[2 * D] != id) err |= kErrRid;
#pragma unroll
        for (int d = 0; d < D; d++) {
            if (b[2 * d] >= m.g.range || b[2 * d + 1] >= m.g.range) err |= kErrRange;
            if (b[2 * d] > b[2 * d + 1]) err |= kErrInverted;
        }
        if (id < m.g.nboxes) {
            const uint32_t bit = 1u << (id & 31u);
            if (atomicOr(&m.moved[id >> 5], bit) & bit) err |= kErrIndex;
        }
        if (err) atomicOr(&m.g.ctr->err, err);
    }
}

// A warp walks the cells of its box 32 at a time, a lane a cell, and their
// slots as one list: the starts and counts of all cells are one load and the
// slots of small cells share the next one. With a loop over the cells each
// waited for the last: 10 485 boxes of 1.7 cells and 54 slots a cell took 31
// us to test, 17 to remove and 22 to insert.
struct ResRun {
    bool in;         // this lane has a cell
    uint32_t c;      // this lane's cell
    uint32_t f;      // its start bits
    uint32_t s0, cap, n;
    uint32_t ends;   // slots of the cells up to and with this one
    uint32_t total;  // of all
    uint32_t top;    // half of the lanes with a cell, rounded up to a power of two (0: one cell)
};
__device__ __forceinline__ uint32_t res_ncells(const uint32_t lo[3], const uint32_t hi[3]) {
    return (hi[0] - lo[0] + 1u) * (hi[1] - lo[1] + 1u) * (hi[2] - lo[2] + 1u);  // (at most the grid's cells, < 2^32)
}
__device__ __forceinline__ bool res_inside(const uint32_t c[3], const uint32_t lo[3], const uint32_t hi[3]) {
    return c[0] >= lo[0] && c[0] <= hi[0] && c[1] >= lo[1] && c[1] <= hi[1] && c[2] >= lo[2] && c[2] <= hi[2];
}
// SKIP: without the cells in [lo0, hi0]
template <bool SKIP>
__device__ __forceinline__ ResRun res_run(const ResGrid& g, const uint32_t lo[3], const uint32_t hi[3], uint32_t q, uint32_t nq,
                                          const uint32_t* lo0 = nullptr, const uint32_t* hi0 = nullptr) {
    ResRun r{};
    if (q < nq) {
        const uint32_t sx = hi[0] - lo[0] + 1u, sy = hi[1] - lo[1] + 1u;
        const uint32_t rr = q / sx, i = q - rr * sx, k = rr / sy, j = rr - k * sy;
        const uint32_t at[3] = {lo[0] + i, lo[1] + j, lo[2] + k};
        if (!SKIP || !res_inside(at, lo0, hi0)) {
            r.in = true;
            r.c = (uint32_t)res_gid(g, at[0], at[1], at[2]);
            r.f = (i == 0 ? 1u : 0u) | (j == 0 ? 2u : 0u) | (k == 0 ? 4u : 0u);
            r.s0 = g.start[r.c];
            r.cap = g.start[r.c + 1] - r.s0;
            r.n = min(g.used[r.c], r.cap);
        }
    }
    r.ends = r.n;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, r.ends, o);
        if ((threadIdx.x & 31u) >= o) r.ends += x;
    }
    r.total = __shfl_sync(0xffffffffu, r.ends, 31);
    const uint32_t cells = min(nq - (q - (threadIdx.x & 31u)), 32u);
    r.top = cells > 1 ? 1u << (31 - __clz(cells - 1)) : 0u;
    return r;
}
// lane that owns slot e < total of the run's list (the first whose end lies
// beyond it), and the slot's place in the grid
__device__ __forceinline__ uint32_t res_owner(const ResRun& r, uint32_t e, uint64_t& slot) {
    uint32_t o = 0;
    for (uint32_t step = r.top; step; step >>= 1) {
        const uint32_t v = __shfl_sync(0xffffffffu, r.ends, o + step - 1);
        if (v <= e) o += step;
    }
    slot = __shfl_sync(0xffffffffu, r.s0 + r.n - r.ends, o) + e;
    return o;
}

// pairs of the listed boxes' warps on their way to one or two lists: per-warp
// buffers in shared memory; at the end a block's rest takes one reservation
struct ResOut {
    uint2 buf[kResWarps][kResBuf];
    uint32_t n[kResWarps], sum;
    unsigned long long at[2];
};
struct ResDst {
    uint2* list;
    uint64_t cap;
    unsigned long long* ctr;
    uint2* also;              // the full list (null: none), which takes the pairs too
    uint64_t also_cap;
    unsigned long long* also_ctr;
};
__device__ __forceinline__ void res_put(const ResDst& d, const uint2* buf, uint32_t n, unsigned long long at,
                                        unsigned long long at2) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t q = lane; q < n; q += 32) {
        if (at + q < d.cap) d.list[at + q] = buf[q];
        if (at2 + q < d.also_cap) d.also[at2 + q] = buf[q];
    }
}
__device__ __forceinline__ void res_flush(const ResDst& d, const uint2* buf, uint32_t n) {
    unsigned long long at = 0, at2 = 0;
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) {
        at = atomicAdd(d.ctr, (unsigned long long)n);
        if (d.also) at2 = atomicAdd(d.also_ctr, (unsigned long long)n);
    }
    res_put(d, buf, n, __shfl_sync(0xffffffffu, at, 0), __shfl_sync(0xffffffffu, at2, 0));
    __syncwarp();
}

// one warp per listed box m: every pair (m, o) of the box with another box o
// that shares a cell with it, reported in the cell of the minimum corner of
// their intersection; a pair of two listed boxes is reported from the smaller
// index
template <int D>
__device__ __forceinline__ void res_query(const Move& mv, const ResDst& dst, uint32_t block, uint32_t nblocks, ResOut& s) {
    constexpr int W = 2 * D + 1;
    const ResGrid& g = mv.g;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint2* buf = s.buf[warp];
    uint32_t nbuf = 0;
    for (uint64_t t = (uint64_t)block * kResWarps + warp; t < mv.k; t += (uint64_t)nblocks * kResWarps) {
        const uint32_t m = mv.idx[t];
        const uint32_t* bm = g.boxes + (uint64_t)m * W;
        uint32_t a[6];
#pragma unroll
        for (int d = 0; d < 6; d++) a[d] = d < 2 * D ? bm[d] : 0u;
        uint32_t lo[3], hi[3];
        res_range<D>(a, g.shift, lo, hi);
        const uint32_t nq = res_ncells(lo, hi);
        for (uint32_t q0 = 0; q0 < nq; q0 += 32) {
            const ResRun r = res_run<false>(g, lo, hi, q0 + lane, nq);
            // two slot pairs per lane in flight together
            for (uint32_t e0 = 0; e0 < r.total; e0 += 32 * kResPer) {
                uint4 c0[kResPer], c1[kResPer];
                uint32_t f[kResPer];
#pragma unroll
                for (int u = 0; u < kResPer; u++) {
                    const uint32_t e = e0 + 32 * u + lane;
                    uint64_t sl;
                    const uint32_t o = res_owner(r, min(e, r.total - 1u), sl);
                    f[u] = __shfl_sync(0xffffffffu, r.f, o);
                    c1[u].z = kDead;
                    if (e < r.total) {
                        c0[u] = g.entries[2 * sl];
                        c1[u] = g.entries[2 * sl + 1];
                    }
                }
                bool part[kResPer];
                uint32_t listed[kResPer];  // (of a hit with a smaller index; the loads together)
#pragma unroll
                for (int u = 0; u < kResPer; u++) {
                    const uint32_t v = c1[u].z, o = v & kIdMask;
                    bool hit = v != kDead && o != m && ((f[u] | (v >> kIdBits)) == 7u);
                    if (hit) {
                        hit = a[0] <= c0[u].y && c0[u].x <= a[1] && a[2] <= c0[u].w && c0[u].z <= a[3];
                        if (D == 3) hit = hit && a[4] <= c1[u].y && c1[u].x <= a[5];
                    }
                    part[u] = hit;
                    listed[u] = hit && o < m ? mv.moved[o >> 5] : 0u;
                }
#pragma unroll
                for (int u = 0; u < kResPer; u++) {
                    const uint32_t o = c1[u].z & kIdMask;
                    const bool hit = part[u] && !((listed[u] >> (o & 31u)) & 1u);
                    const uint32_t hm = __ballot_sync(0xffffffffu, hit);
                    if (nbuf + __popc(hm) > kResBuf) {
                        res_flush(dst, buf, nbuf);
                        nbuf = 0;
                    }
                    if (hit) buf[nbuf + __popc(hm & ((1u << lane) - 1u))] = make_uint2(min(m, o), max(m, o));
                    nbuf += __popc(hm);
                }
            }
        }
    }
    if (lane == 0) s.n[warp] = nbuf;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
        for (int w = 0; w < kResWarps; w++) {
            const uint32_t x = s.n[w];
            s.n[w] = sum;
            sum += x;
        }
        s.sum = sum;
    }
    __syncwarp();
    if (warp == 0 && lane < 2) {  // (both counters at once)
        unsigned long long* c = lane ? dst.also_ctr : dst.ctr;
        s.at[lane] = c ? atomicAdd(c, (unsigned long long)s.sum) : 0ull;
    }
    __syncthreads();
    res_put(dst, buf, nbuf, s.at[0] + s.n[warp], s.at[1] + s.n[warp]);
}

// the old list's pairs without a moved box go to the new one, the others are
// the pairs that the moved boxes had: each thread takes 4 pairs (two 16-byte
// loads), one reservation per block, round and list
constexpr int kFilterPer = 4;
static_assert(kResThreads * kFilterPer < 1 << 16, "two counts in a word");
__device__ __forceinline__ void res_split(const Move& m, uint32_t block, uint32_t nblocks, uint32_t* s_w,
                                          unsigned long long* s_at) {
    const uint2* in = m.old_full;
    const uint64_t n = m.nold;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint64_t round = (uint64_t)kResThreads * kFilterPer;
    for (uint64_t b0 = (uint64_t)block * round; b0 < n; b0 += (uint64_t)nblocks * round) {
        const uint64_t i0 = b0 + (uint64_t)t * kFilterPer;
        uint2 pr[kFilterPer];
        uint32_t keep = 0, drop = 0;
        if (i0 + kFilterPer <= n) {
            const uint4* q = reinterpret_cast<const uint4*>(in + i0);
            const uint4 a = q[0], b = q[1];
            pr[0] = make_uint2(a.x, a.y); pr[1] = make_uint2(a.z, a.w);
            pr[2] = make_uint2(b.x, b.y); pr[3] = make_uint2(b.z, b.w);
        } else {
#pragma unroll
            for (int k = 0; k < kFilterPer; k++) pr[k] = i0 + k < n ? in[i0 + k] : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int k = 0; k < kFilterPer; k++) {
            const bool moved = res_moved(m.moved, pr[k].x) | res_moved(m.moved, pr[k].y);
            if (i0 + k < n) (moved ? drop : keep) |= 1u << k;
        }
        const uint32_t cnt = __popc(keep) | __popc(drop) << 16;
        uint32_t incl = cnt;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        uint32_t before = 0, tot = 0;  // of the block's warps
        for (uint32_t w = 0; w < kResWarps; w++) {
            if (w == warp) before = tot;
            tot += s_w[w];
        }
        if (t < 2) {
            const uint32_t sum = t ? tot >> 16 : tot & 0xffffu;
            s_at[t] = sum ? atomicAdd(t ? &m.g.ctr->rem : &m.g.ctr->full, (unsigned long long)sum) : 0ull;
        }
        __syncthreads();
        before += incl - cnt;
        uint64_t pos = s_at[0] + (before & 0xffffu), rpos = s_at[1] + (before >> 16);
#pragma unroll
        for (int k = 0; k < kFilterPer; k++) {
            if (keep & (1u << k)) m.full[pos++] = pr[k];
            if (drop & (1u << k)) {
                if (rpos < m.rem_cap) m.rem[rpos] = pr[k];
                rpos++;
            }
        }
        __syncthreads();
    }
}

// one warp per listed box: its entries take the new coordinates where the cell
// is one of the box's new ones too, and become tombstones elsewhere
template <int D>
__device__ __forceinline__ void res_remove(const Move& m, uint32_t block, uint32_t nblocks) {
    constexpr int W = 2 * D + 1;
    const ResGrid& g = m.g;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t t = (uint64_t)block * kResWarps + (threadIdx.x >> 5); t < m.k; t += (uint64_t)nblocks * kResWarps) {
        const uint32_t id = m.idx[t];
        const uint32_t* b = m.nb + t * W;
        uint32_t lo[3], hi[3], lo1[3], hi1[3];
        res_range<D>(g.boxes + (uint64_t)id * W, g.shift, lo, hi);
        res_range<D>(b, g.shift, lo1, hi1);
        const uint32_t nq = res_ncells(lo, hi);
        for (uint32_t q0 = 0; q0 < nq; q0 += 32) {
            const ResRun r = res_run<false>(g, lo, hi, q0 + lane, nq);
            for (uint32_t e0 = 0; e0 < r.total; e0 += 128) {
                uint32_t v[4], c[4];
                uint64_t sl[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t e = e0 + 32 * u + lane;
                    c[u] = __shfl_sync(0xffffffffu, r.c, res_owner(r, min(e, r.total - 1u), sl[u]));
                    v[u] = e < r.total ? g.entries[2 * sl[u] + 1].z : kDead;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (v[u] == kDead || (v[u] & kIdMask) != id) continue;
                    const uint32_t cy = c[u] / g.nrc, cz = cy / g.nrc;
                    const uint32_t at[3] = {c[u] - cy * g.nrc, cy - cz * g.nrc, cz};
                    if (res_inside(at, lo1, hi1)) {
                        const uint32_t f = (at[0] == lo1[0] ? 1u : 0u) | (at[1] == lo1[1] ? 2u : 0u) | (at[2] == lo1[2] ? 4u : 0u);
                        uint4 a0, a1;
                        res_slot<D>(b, (f << kIdBits) | id, a0, a1);
                        g.entries[2 * sl[u]] = a0;
                        g.entries[2 * sl[u] + 1] = a1;
                    } else {
                        g.entries[2 * sl[u] + 1].z = kDead;
                    }
                }
            }
        }
    }
}

// the first `rblocks` blocks move the listed boxes' entries, the others
// split the full list beside them
template <int D>
__global__ void __launch_bounds__(kResThreads) k_move_out(Move m, uint32_t rblocks) {
    __shared__ uint32_t s_w[kResWarps];
    __shared__ unsigned long long s_at[2];
    chain_wait();
    // (with a full list, the pairs before are being counted here)
    const MoveState c = move_state(m);
    if (c.bad || (!m.full && c.rem > m.rem_cap)) return;
    if (blockIdx.x < rblocks) res_remove<D>(m, blockIdx.x, rblocks);
    else res_split(m, blockIdx.x - rblocks, gridDim.x - rblocks, s_w, s_at);
}

// pairs of the listed boxes before the move, where there is no full list to take them from
template <int D>
__global__ void __launch_bounds__(kResThreads, kResBlocks) k_move_before(Move m) {
    __shared__ ResOut s;
    chain_wait();
    if (move_state(m).bad) return;
    res_query<D>(m, ResDst{m.rem, m.rem_cap, &m.g.ctr->rem, nullptr, 0, nullptr}, blockIdx.x, gridDim.x, s);
}

// one warp per listed box; in each of its cells that it was not in before it
// takes a tombstone (claimed with a compare-and-swap on the index word, by the
// first lane that sees one of the cell's) or else appends; the box takes its
// new coordinates. Boxes that stay in their cells, as most do that move less
// than a cell's edge, are done there: inserting all anew took 22 us of a move
// of 10 485 boxes, this 12.
template <int D>
__global__ void __launch_bounds__(kResThreads) k_move_in(Move m, uint32_t* boxes) {
    constexpr int W = 2 * D + 1;
    chain_wait();
    const MoveState c = move_state(m);
    if (c.bad || c.rem > m.rem_cap) return;
    const ResGrid& g = m.g;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t t = (uint64_t)blockIdx.x * kResWarps + (threadIdx.x >> 5); t < m.k; t += (uint64_t)gridDim.x * kResWarps) {
        const uint32_t id = m.idx[t];
        const uint32_t* b = m.nb + t * W;
        uint32_t a[6];
#pragma unroll
        for (int d = 0; d < 6; d++) a[d] = d < 2 * D ? b[d] : 0u;
        uint32_t lo[3], hi[3], lo0[3], hi0[3];
        res_range<D>(boxes + (uint64_t)id * W, g.shift, lo0, hi0);
        res_range<D>(a, g.shift, lo, hi);
        __syncwarp();  // (every lane has read the old coordinates)
        if (lane < W) {  // (the old row stays at hand: k_move_back)
            uint32_t &now = boxes[(uint64_t)id * W + lane], &then = m.nb[t * W + lane];
            const uint32_t w = now;
            now = then;
            then = w;
        }
        auto put = [&](uint64_t slot, uint32_t idw) {
            uint4 e0, e1;
            res_slot<D>(a, idw, e0, e1);
            g.entries[2 * slot] = e0;
            g.entries[2 * slot + 1] = e1;
        };
        const uint32_t nq = res_ncells(lo, hi);
        for (uint32_t q0 = 0; q0 < nq; q0 += 32) {
            const ResRun r = res_run<true>(g, lo, hi, q0 + lane, nq, lo0, hi0);
            const uint32_t all = __ballot_sync(0xffffffffu, r.in);
            uint32_t have = 0;  // cells of the run that took a slot (the same in every lane)
            for (uint32_t e0 = 0; e0 < r.total && have != all; e0 += 128) {
                uint32_t v[4], o[4];
                uint64_t sl[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t e = e0 + 32 * u + lane;
                    o[u] = res_owner(r, min(e, r.total - 1u), sl[u]);
                    v[u] = e < r.total ? g.entries[2 * sl[u] + 1].z : 0u;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t f = __shfl_sync(0xffffffffu, r.f, o[u]);
                    bool mine = v[u] == kDead;
                    while (true) {
                        mine = mine && !((have >> o[u]) & 1u);
                        if (!__any_sync(0xffffffffu, mine)) break;
                        // one lane of each cell tries (lanes with nothing to take stand apart)
                        const uint32_t peers = __match_any_sync(0xffffffffu, mine ? o[u] : 32u + lane);
                        bool won = false;
                        if (mine && lane == __ffs(peers) - 1u) {
                            const uint32_t idw = (f << kIdBits) | id;
                            won = atomicCAS(&g.entries[2 * sl[u] + 1].z, kDead, idw) == kDead;
                            if (won) put(sl[u], idw);
                            mine = false;
                        }
                        have |= __reduce_or_sync(0xffffffffu, won ? 1u << o[u] : 0u);
                    }
                }
            }
            if (((all & ~have) >> lane) & 1u) {  // no tombstone: append
                const uint32_t sl = atomicAdd(&g.used[r.c], 1u);
                if (sl < r.cap) put((uint64_t)r.s0 + sl, (r.f << kIdBits) | id);
                else atomicOr(&g.ctr->overflow, 1u);
            }
        }
    }
}

// the rows that k_move_in left at hand, back in their places
template <int D>
__global__ void k_move_back(Move m, uint32_t* boxes) {
    constexpr int W = 2 * D + 1;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < m.k * W; w += (uint64_t)gridDim.x * blockDim.x)
        boxes[(uint64_t)m.idx[w / W] * W + w % W] = m.nb[w];
}

// pairs of the listed boxes after the move, to the list of added pairs and
// behind the filtered full list; the last block hands the counters to the host
template <int D>
__global__ void __launch_bounds__(kResThreads, kResBlocks) k_move_after(Move m) {
    __shared__ ResOut s;
    ResCtr* c = m.g.ctr;
    chain_wait();
    const MoveState before = move_state(m);
    if (!before.bad && !before.no_slack && before.rem <= m.rem_cap)
        res_query<D>(m, ResDst{m.add, m.add_cap, &c->add, m.full, m.full ? m.nold + m.add_cap : 0,
                                    m.full ? &c->full : nullptr}, blockIdx.x, gridDim.x, s);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&c->done, 1u) == gridDim.x - 1u) {
            ResCtr h;
            h.err = __ldcg(&c->err);
            h.overflow = __ldcg(&c->overflow);
            h.rem = __ldcg(&c->rem);
            h.add = __ldcg(&c->add);
            h.full = __ldcg(&c->full);
            h.done = h.wide = 0;
            h.sum = 0;
            *m.host = h;
            __threadfence_system();
        }
    }
}

}  // namespace pbig

using namespace pbig;

struct pbig2_scene {
    pbig2_ctx* ctx = nullptr;
    int dims = 3;
    uint32_t range = 0, shift = 0, nrc = 0;
    uint64_t n = 0, ncells = 0, nslots = 0;
    DevBuf boxes, entries, idx, nb;
    DevBuf cells;  // of the grid: starts, slots used; while it is built: counts, capacities, the scan's state and counters
    DevBuf rctr;  // ResCtr, then one bit per box: listed by the move
    DevBuf full[2], rem, add;
    int cur = 0;  // full[cur] holds the current list
    bool stale = false;     // a move that failed half-way left the grid: it is built anew before the next one
    bool lost = false;      // a CUDA error struck while the boxes were moving
    bool keep_full = true;  // maintain the full pair list on every move
    bool automatic = false; // the cell size is the engine's choice
    uint64_t nfull = 0, nrem = 0, nadd = 0;

    template <class F>
    void each_buffer(F f) {
        for (DevBuf* b : {&boxes, &entries, &cells, &rctr, &idx, &nb, &full[0], &full[1], &rem, &add}) f(*b);
    }
    // `cells`: four arrays of a word per cell and one more, then the scan's tile
    // records, counters and (unused) lists; one allocation, for they are all large
    // and are taken each time a scene is made
    size_t cell_pitch() const { return ((ncells + 1) * 4 + 255) & ~size_t(255); }
    size_t scan_at() const { return 4 * cell_pitch(); }
    size_t ctr_at() const { return scan_at() + ((scan_state_bytes(ncells) + 255) & ~size_t(255)); }
    size_t cells_bytes() const { return ctr_at() + ((sizeof(Ctr) + 255) & ~size_t(255)) + 256; }
    unsigned char* cell_bytes(size_t at) { return cells.as<unsigned char>() + at; }
    uint32_t* cell_words(int k) { return reinterpret_cast<uint32_t*>(cell_bytes(k * cell_pitch())); }
    size_t rctr_bytes() const { return sizeof(ResCtr) + ((n + 31) / 32) * 4; }
    ResGrid grid() {
        ResGrid g{};
        g.boxes = boxes.as<uint32_t>();
        g.nboxes = n;
        g.shift = shift;
        g.nrc = nrc;
        g.range = range;
        g.ncells = ncells;
        g.nslots = nslots;
        g.start = cell_words(0);
        g.used = cell_words(1);
        g.entries = entries.as<uint4>();
        g.ctr = rctr.as<ResCtr>();
        return g;
    }
};

namespace {

#define SCK(expr)                                                                                      \
    do {                                                                                               \
        cudaError_t _e = (expr);                                                                       \
        if (_e != cudaSuccess) {                                                                       \
            char _m[256];                                                                              \
            snprintf(_m, sizeof _m, "%s: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
            return api_fail(_e == cudaErrorMemoryAllocation ? PBIG2_ENOMEM : PBIG2_ECUDA, _m);        \
        }                                                                                              \
    } while (0)

constexpr char kLost[] = "the scene was lost to a CUDA error in a move";

unsigned grid_for(uint64_t items, unsigned per_block, int sms) {
    uint64_t b = (items + per_block - 1) / per_block;
    const uint64_t cap = (uint64_t)(sms > 0 ? sms : 152) * 16;
    if (b > cap) b = cap;
    return (unsigned)(b ? b : 1);
}

ResCtr read_ctr(pbig2_scene* s, cudaStream_t st, cudaError_t* e) {
    ResCtr h{};
    *e = cudaMemcpyAsync(&h, s->rctr.p, sizeof h, cudaMemcpyDeviceToHost, st);
    if (*e == cudaSuccess) *e = cudaStreamSynchronize(st);
    return h;
}

void set_shift(pbig2_scene* s, uint32_t shift) {
    s->shift = shift;
    s->nrc = nrc_for(s->range, shift);
    s->ncells = grid_cells(s->range, shift, s->dims);
}

// the grid of the scene's current boxes: counts, capacities with slack,
// starts (the engine's scan), then every box inserted. The slots are summed in
// 64 bits before anything is placed by them: 2^32 or more are refused, and so is
// a box of more than `widest` cells.
int build_grid(pbig2_scene* s, cudaStream_t st, uint32_t widest = 0xffffffffu) {
    const int sms = s->ctx->sm_count;
    if (pbig2_scene_slots(s->ncells, 0) + s->n > kMaxSlots)  // (every box has an entry)
        return api_fail(PBIG2_ECAPACITY, "resident grid: 2^32 slots or more");
    SCK(s->cells.ensure(s->cells_bytes(), false, st));
    uint32_t *cnt = s->cell_words(2), *cap = s->cell_words(3);
    SCK(cudaMemsetAsync(cnt, 0, s->ncells * 4, st));
    SCK(cudaMemsetAsync(s->rctr.p, 0, sizeof(ResCtr), st));
    ResGrid g = s->grid();
    if (s->dims == 2) k_res_count<2><<<grid_for(s->n, 256, sms), 256, 0, st>>>(g, cnt, widest);
    else k_res_count<3><<<grid_for(s->n, 256, sms), 256, 0, st>>>(g, cnt, widest);
    SCK(cudaGetLastError());
    k_res_caps<<<grid_for(s->ncells, 256, sms), 256, 0, st>>>(cnt, cap, s->ncells, g.ctr);
    SCK(cudaGetLastError());
    cudaError_t e;
    ResCtr h = read_ctr(s, st, &e);
    SCK(e);
    if (h.wide || h.sum > kMaxSlots) return api_fail(PBIG2_ECAPACITY, "resident grid: 2^32 slots or more, or a box too wide for it");
    s->nslots = h.sum;
    SCK(s->entries.ensure(s->nslots * 32 + 32, false, st));
    g = s->grid();
    // exclusive scan of the capacities with the engine's scan kernels (the
    // cell ends replace the capacities in place; no work lists)
    Params p{};
    p.counts = cap;
    p.ncells = s->ncells;
    p.tile_state = reinterpret_cast<unsigned long long*>(s->cell_bytes(s->scan_at()));
    p.ctr = reinterpret_cast<Ctr*>(s->cell_bytes(s->ctr_at()));
    p.lists = reinterpret_cast<uint2*>(s->cell_bytes(s->cells_bytes() - 256));
    SCK(cudaMemsetAsync(p.tile_state, 0, s->ctr_at() - s->scan_at() + sizeof(Ctr), st));  // (and p.ctr behind it)
    SCK(launch_scan(p, st));
    k_res_starts<<<grid_for(s->ncells, 256, sms), 256, 0, st>>>(cnt, cap, g);
    SCK(cudaGetLastError());
    // free slots hold no tombstone of an older grid: one that a box is about to
    // be appended to must not be claimed by another box of the same move
    SCK(cudaMemsetAsync(s->entries.p, 0, s->nslots * 32, st));
    if (s->dims == 2) k_res_fill<2><<<grid_for(s->n, 256, sms), 256, 0, st>>>(g);
    else k_res_fill<3><<<grid_for(s->n, 256, sms), 256, 0, st>>>(g);
    SCK(cudaGetLastError());
    h = read_ctr(s, st, &e);
    SCK(e);
    if (h.overflow) return api_fail(PBIG2_ECUDA, "resident grid: a cell overflowed its own count");
    return PBIG2_OK;
}

// with an automatic cell size, on coarser grids until the slots can be numbered
// and there is memory for them
int build(pbig2_scene* s, cudaStream_t st) {
    int rc = build_grid(s, st);
    while ((rc == PBIG2_ECAPACITY || rc == PBIG2_ENOMEM) && s->automatic && s->ncells > 1 && s->shift < 31) {
        for (DevBuf* b : {&s->cells, &s->entries}) b->release();
        set_shift(s, s->shift + 1);
        rc = build_grid(s, st);
    }
    return rc;
}

// With an automatic cell size the scene's grid is one size finer than the
// query's, where that makes at most 4 cells a box, no box covers more than 512
// and it fits: a move tests the moved boxes against whole cells, while the query
// tests each pair of a cell once. Moves of 1 % of a million boxes of one density
// 81 us on the query's grid, 70 on the finer one and 69 on the next; of 65 536
// boxes 52 and 46; of the clustered 4M-box scene 716, 568 and 621.
int build_first(pbig2_scene* s, cudaStream_t st) {
    if (s->automatic && s->shift > 0 && grid_cells(s->range, s->shift - 1, s->dims) <= 4 * s->n) {
        set_shift(s, s->shift - 1);
        const int rc = build_grid(s, st, 512);
        if (rc != PBIG2_ECAPACITY && rc != PBIG2_ENOMEM) return rc;
        for (DevBuf* b : {&s->cells, &s->entries}) b->release();
        set_shift(s, s->shift + 1);
    }
    return build(s, st);
}

// room for `need` pairs in a buffer that keeps its first `have`: a move that
// is refused leaves the lists of the last one as they were
cudaError_t room_for(DevBuf& buf, uint64_t need, uint64_t have, cudaStream_t st) {
    if (need * 8 <= buf.bytes) return cudaSuccess;
    DevBuf grown;
    grown.most = buf.most;
    cudaError_t e = grown.ensure(need * 8, false, st);
    if (e == cudaSuccess && have) {
        e = cudaMemcpyAsync(grown.p, buf.p, have * 8, cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) {
        grown.release();
        return e;
    }
    buf.release();
    buf = grown;
    return cudaSuccess;
}

enum MovePart : unsigned { kMoveAll = 0, kMoveRest = 1 };  // the rest: once the boxes are moved

template <int D>
cudaError_t launch_move(pbig2_scene* s, const Move& m, MovePart part, cudaStream_t st) {
    const int sms = s->ctx->sm_count;
    const unsigned gw = grid_for(m.k, kResWarps, sms), r = part == kMoveAll ? gw : 0u;
    const unsigned f = m.nold ? grid_for(m.nold, kResThreads * kFilterPer, sms) : 0u;
    const bool all = part == kMoveAll;
    cudaError_t e = cudaSuccess;
    if (all) e = launch_after(false, k_move_check<D>, grid_for(m.k, 256, sms), 256, 0, st, m);
    if (e == cudaSuccess && all && !m.full) e = launch_after(true, k_move_before<D>, gw, kResThreads, 0, st, m);
    if (e == cudaSuccess && r + f) e = launch_after(all, k_move_out<D>, r + f, kResThreads, 0, st, m, (uint32_t)r);
    if (e == cudaSuccess && all) e = launch_after(true, k_move_in<D>, gw, kResThreads, 0, st, m, s->boxes.as<uint32_t>());
    return e != cudaSuccess ? e : launch_after(all || r + f, k_move_after<D>, gw, kResThreads, 0, st, m);
}

// The passes of a move until the pairs before and after it fit their lists.
// `part`: whether the boxes have moved. A move that fails once its kernels have
// run leaves `stale` set.
int move_passes(pbig2_scene* s, Move& m, uint64_t guess, ResCtr& h, MovePart& part, cudaStream_t st) {
    const int nxt = s->cur ^ 1;
    for (int attempt = 0;; attempt++) {
        m.rem = s->rem.as<uint2>();
        m.add = s->add.as<uint2>();
        m.rem_cap = s->rem.bytes / 8;
        m.add_cap = s->add.bytes / 8;
        if (s->keep_full) {
            // (the list that a larger one of these replaces is the one before the last)
            SCK(s->full[nxt].ensure((s->nfull + (part == kMoveAll ? guess : h.add)) * 8 + 16, false, st));
            const uint64_t room = s->full[nxt].bytes / 8 - s->nfull;
            if (m.add_cap > room) m.add_cap = room;
            m.old_full = s->full[s->cur].as<uint2>();
            m.full = s->full[nxt].as<uint2>();
            m.nold = s->nfull;
        }
        s->stale = true;
        SCK(s->dims == 2 ? launch_move<2>(s, m, part, st) : launch_move<3>(s, m, part, st));
        SCK(cudaStreamSynchronize(st));
        h = *m.host;
        if (h.err) {
            s->stale = false;  // nothing was touched
            return api_fail(PBIG2_EINVAL, h.err == kErrIndex
                                              ? "a box is listed twice"
                                              : "moved boxes must keep rid = their index, coordinates < range and min <= max");
        }
        const bool more_rem = h.rem > m.rem_cap, more_add = !more_rem && !h.overflow && h.add > m.add_cap;
        if (!more_rem && !h.overflow && !more_add) break;
        if (attempt == 4) return api_fail(PBIG2_ENOMEM, "pair buffer retries exhausted");
        ResCtr again{};
        if (more_rem) {  // the boxes have their old coordinates
            s->nrem = 0;
            SCK(s->rem.ensure(h.rem * 8 + h.rem / 4, false, st));
        } else {
            if (!m.full) again.rem = h.rem;
            part = kMoveRest;
            if (h.overflow) {  // a cell ran out of slack
                const int rc = build(s, st);
                if (rc) return rc;
                m.g = s->grid();
                h.add = guess;
            } else {
                s->nadd = 0;
                SCK(s->add.ensure(h.add * 8 + h.add / 4, false, st));
            }
        }
        // (the check marks the boxes again, or they stay marked)
        if (more_rem) SCK(cudaMemsetAsync(s->rctr.p, 0, s->rctr_bytes(), st));
        else SCK(cudaMemcpyAsync(s->rctr.p, &again, sizeof again, cudaMemcpyHostToDevice, st));
    }
    return PBIG2_OK;
}

// What is left of a move that failed on the way, for want of memory: the boxes
// have their old rows again, so that the full list is theirs, and the grid is
// built anew before the next move. After a CUDA error the scene is lost.
int take_back(pbig2_scene* s, const Move& m, MovePart part, int rc, cudaStream_t st) {
    s->nrem = s->nadd = 0;
    if (rc == PBIG2_ECUDA) {
        s->lost = true;
        return rc;
    }
    if (part == kMoveAll) return rc;  // the boxes had not moved
    const unsigned g = grid_for(m.k, 256, s->ctx->sm_count);
    if (s->dims == 2) k_move_back<2><<<g, 256, 0, st>>>(m, s->boxes.as<uint32_t>());
    else k_move_back<3><<<g, 256, 0, st>>>(m, s->boxes.as<uint32_t>());
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) s->lost = true;
    return rc;
}

}  // namespace

extern "C" {

PBIG2_API uint64_t pbig2_scene_slots(uint64_t ncells, uint64_t entries) {
    const unsigned __int128 s = (unsigned __int128)entries + entries / 2 + (unsigned __int128)ncells * res_cap(0);
    return s > ~0ull ? ~0ull : (uint64_t)s;
}

PBIG2_API int pbig2_scene_create(pbig2_ctx* c, const uint32_t* boxes, uint64_t n, uint32_t dims, uint32_t range,
                                 uint32_t cell_shift, int boxes_loc, uint32_t flags, pbig2_scene** out,
                                 uint64_t* npairs) {
    if (!c || !out || !npairs || (dims != 2 && dims != 3) || range == 0 || (n && !boxes))
        return api_fail(PBIG2_EINVAL, "bad arguments");
    *out = nullptr;
    *npairs = 0;
    if (n == 0 || n > (uint64_t)kIdMask + 1) return api_fail(PBIG2_EINVAL, "a scene holds 1 .. 2^29 boxes");
    // the full query first: its pairs, its cell size, and the input checks
    uint64_t np = 0;
    c->want_grid = true;
    int rc = pbig2_self_intersect(c, boxes, n, dims, range, cell_shift, boxes_loc, nullptr, &np);
    c->want_grid = false;
    if (rc != PBIG2_OK) return rc == PBIG2_EINPUT ? api_fail(PBIG2_EINPUT, "a scene's boxes must all be valid") : rc;
    pbig2_stats st{};
    pbig2_get_stats(c, &st);
    pbig2_scene* s = new pbig2_scene();
    s->ctx = c;
    s->each_buffer([c](DevBuf& b) { b.most = &c->max_buffer; });
    s->dims = (int)dims;
    s->range = range;
    s->n = n;
    s->automatic = cell_shift == PBIG2_AUTO;
    set_shift(s, st.cell_shift);  // below 2^32 cells: the query above ran on this grid
    cudaStream_t sm = c->own_stream;
    const int W = 2 * (int)dims + 1;
    auto bail = [&](int code) {
        pbig2_scene_destroy(s);
        return code;
    };
    if (s->boxes.ensure(n * W * 4 + 16, false, sm) != cudaSuccess ||
        s->rctr.ensure(s->rctr_bytes(), false, sm) != cudaSuccess ||
        s->full[0].ensure(np * 8 + 16, false, sm) != cudaSuccess)
        return bail(api_fail(PBIG2_ENOMEM, "scene allocation failed"));
    if (cudaMemcpyAsync(s->boxes.p, boxes, n * W * 4, cudaMemcpyDefault, sm) != cudaSuccess)
        return bail(api_fail(PBIG2_ECUDA, "copying the scene's boxes failed"));
    if (np && pbig2_copy_pairs(c, s->full[0].as<uint32_t>(), 0, np, PBIG2_DEVICE, sm) != PBIG2_OK) return bail(PBIG2_ECUDA);
    s->nfull = np;
    s->keep_full = (flags & PBIG2_SCENE_DELTA_ONLY) == 0;
    rc = build_first(s, sm);
    if (rc != PBIG2_OK) return bail(rc);
    *out = s;
    *npairs = np;
    return PBIG2_OK;
}

PBIG2_API int pbig2_scene_destroy(pbig2_scene* s) {
    if (!s) return PBIG2_OK;
    s->each_buffer([](DevBuf& b) { b.release(); });
    delete s;
    return PBIG2_OK;
}

PBIG2_API int pbig2_scene_move(pbig2_scene* s, const uint32_t* idx, uint64_t k, const uint32_t* new_boxes, int loc,
                               uint64_t* n_removed, uint64_t* n_added) {
    if (!s || !n_removed || !n_added || (k && (!idx || !new_boxes))) return api_fail(PBIG2_EINVAL, "bad arguments");
    *n_removed = *n_added = 0;
    if (k == 0) {
        s->nrem = s->nadd = 0;
        return PBIG2_OK;
    }
    if (k > s->n) return api_fail(PBIG2_EINVAL, "more moved boxes than the scene holds");
    if (s->lost) return api_fail(PBIG2_ECUDA, kLost);
    SCK(cudaSetDevice(s->ctx->device));
    cudaStream_t st = s->ctx->own_stream;
    const int W = 2 * s->dims + 1;
    (void)loc;  // copies below read host or device memory alike
    static_assert(sizeof(ResCtr) <= sizeof(Ctr), "a move's counters in the page-locked block of a query's");
    SCK(s->ctx->h_ctr.ensure(sizeof(Ctr)));
    SCK(s->idx.ensure(k * 4 + 16, false, st));
    SCK(s->nb.ensure(k * W * 4 + 16, false, st));
    if (s->stale) {
        const int rc = build(s, st);
        if (rc) return rc;
        s->stale = false;
    }
    SCK(cudaMemsetAsync(s->rctr.p, 0, s->rctr_bytes(), st));
    SCK(cudaMemcpyAsync(s->idx.p, idx, k * 4, cudaMemcpyDefault, st));
    SCK(cudaMemcpyAsync(s->nb.p, new_boxes, k * W * 4, cudaMemcpyDefault, st));
    // twice the pairs that k boxes have on average, if the full list is of
    // some use as a measure; a move that needs more repeats from there
    const uint64_t mean = (uint64_t)(4.0 * (double)s->nfull * ((double)k / (double)s->n));
    const uint64_t guess = 1024 + (mean < s->nfull ? mean : s->nfull);
    SCK(room_for(s->rem, guess, s->nrem, st));
    SCK(room_for(s->add, guess, s->nadd, st));
    Move m{};
    m.g = s->grid();
    m.idx = s->idx.as<uint32_t>();
    m.nb = s->nb.as<uint32_t>();
    m.k = k;
    m.moved = reinterpret_cast<uint32_t*>(s->rctr.as<ResCtr>() + 1);
    m.host = static_cast<ResCtr*>(s->ctx->h_ctr.p);
    ResCtr h{};
    MovePart part = kMoveAll;
    const int rc = move_passes(s, m, guess, h, part, st);
    if (rc) return s->stale ? take_back(s, m, part, rc, st) : rc;
    s->stale = false;
    if (s->keep_full) {
        s->cur ^= 1;
        s->nfull = h.full;
    }
    *n_removed = s->nrem = h.rem;
    *n_added = s->nadd = h.add;
    return PBIG2_OK;
}

PBIG2_API int pbig2_scene_delta(pbig2_scene* s, const uint32_t** removed, uint64_t* n_removed, const uint32_t** added,
                                uint64_t* n_added) {
    if (!s || !removed || !n_removed || !added || !n_added) return api_fail(PBIG2_EINVAL, "bad arguments");
    if (s->lost) return api_fail(PBIG2_ECUDA, kLost);
    *removed = s->rem.as<uint32_t>();
    *n_removed = s->nrem;
    *added = s->add.as<uint32_t>();
    *n_added = s->nadd;
    return PBIG2_OK;
}

PBIG2_API int pbig2_scene_pairs(pbig2_scene* s, const uint32_t** pairs, uint64_t* npairs) {
    if (!s || !pairs || !npairs) return api_fail(PBIG2_EINVAL, "bad arguments");
    if (!s->keep_full) return api_fail(PBIG2_EINVAL, "the scene keeps no full pair list (PBIG2_SCENE_DELTA_ONLY)");
    if (s->lost) return api_fail(PBIG2_ECUDA, kLost);
    *pairs = s->full[s->cur].as<uint32_t>();
    *npairs = s->nfull;
    return PBIG2_OK;
}

PBIG2_API int pbig2_scene_copy(pbig2_scene* s, int which, uint32_t* dst, uint64_t count) {
    if (!s || (count && !dst) || which < 0 || which > 2) return api_fail(PBIG2_EINVAL, "bad arguments");
    if (which == 0 && !s->keep_full) return api_fail(PBIG2_EINVAL, "the scene keeps no full pair list (PBIG2_SCENE_DELTA_ONLY)");
    if (s->lost) return api_fail(PBIG2_ECUDA, kLost);
    const uint64_t have = which == 0 ? s->nfull : which == 1 ? s->nrem : s->nadd;
    if (count > have) return api_fail(PBIG2_EINVAL, "more pairs asked for than the list holds");
    if (count == 0) return PBIG2_OK;
    const void* src = which == 0 ? s->full[s->cur].p : which == 1 ? s->rem.p : s->add.p;
    SCK(cudaSetDevice(s->ctx->device));
    SCK(cudaMemcpyAsync(dst, src, count * 8, cudaMemcpyDefault, s->ctx->own_stream));
    SCK(cudaStreamSynchronize(s->ctx->own_stream));
    return PBIG2_OK;
}

PBIG2_API int pbig2_scene_boxes(pbig2_scene* s, const uint32_t** boxes, uint64_t* n) {
    if (!s || !boxes || !n) return api_fail(PBIG2_EINVAL, "bad arguments");
    if (s->lost) return api_fail(PBIG2_ECUDA, kLost);
    *boxes = s->boxes.as<uint32_t>();
    *n = s->n;
    return PBIG2_OK;
}

}  // extern "C"
