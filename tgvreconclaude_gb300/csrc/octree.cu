// Stages 2 and 3 on the GPU: the k-way merge of sorted cube lists (the
// reference's kway_merge, src/merge.cpp:7-97) and the 2:1 balance
// (balance_octree, src/balance.cpp:60-150).
//
// Merge.  The code-sorted inputs are merged pairwise, neighbours first, in
// ceil(log2 k) stable passes, so equal codes keep input order (the reference's
// heap leaves the order of equal codes from different inputs to
// std::priority_queue; the two agree whenever no code occurs in more than one
// input).  An input that is not sorted is found by the first pass; all inputs
// are then concatenated in order and stably radix-sorted by code.  Runs of
// consecutive equal (code, depth) collapse into one cube whose r_c is the run's
// float sum in order divided by its length (merge.cpp:64-88).
//
// Balance.  The reference processes a FIFO of cells one at a time, and each
// cell's decisions read the cell sets as the cells before it left them.  The
// kernels reproduce that order exactly.  A window of pending FIFO entries is
// evaluated in parallel: every (entry, face) slot that can add a bridge computes
// its proposal against the sets at the window start plus the bridges that slots
// before it propose, and the evaluation repeats until the proposals stop
// changing.  A slot's result depends only on slots before it, so the fixed
// point is the sequential result, and a prefix of slots that did not change
// is already exact (used to bound the repetitions).  The accepted bridges are
// appended to the FIFO in slot order, which is the reference's push order.
//
// Presence is tested per exact (depth, code) cell; the output table is keyed
// like the reference's dc_key, depth << 60 | (code & (2^60 - 1)) in 64-bit
// arithmetic (balance.cpp:57-59), so the output drops the code's top three
// bits and folds depths 16..21 onto 0..5, as the reference's does.  Input
// cubes must be valid cells (depth 0..21, code aligned to its depth's grid).
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"
#include "fileio.h"

namespace tgvg {
namespace {

constexpr uint64_t DC_MASK = 0x0fffffffffffffffull;
constexpr unsigned long long CELL_EMPTY = 0ull;   // cell keys are never 0
constexpr unsigned long long DC_EMPTY = ~0ull;    // no aligned cell has this output key
constexpr int64_t WINDOW = int64_t(1) << 22;      // FIFO entries evaluated together
constexpr int MAX_ROUNDS = 24;                    // evaluations of one window before a prefix is committed

inline unsigned grid_of(int64_t n, int t) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

// Locational key of an aligned cell: its depth-d index under a marker bit 3d.
__host__ __device__ __forceinline__ uint64_t cell_key(uint64_t code, int d) {
    return (code >> (3 * (21 - d))) | (1ull << (3 * d));
}
// The reference's output-table key (balance.cpp:57-59).
__host__ __device__ __forceinline__ uint64_t dc_key(int d, uint64_t code) {
    return ((uint64_t)(uint32_t)d << 60) | (code & DC_MASK);
}

// Insert-only open-addressing key set, linear probing, power-of-two capacity.
struct KeySet {
    unsigned long long* keys;
    uint64_t mask;
    unsigned long long empty;
};
__device__ __forceinline__ long long set_slot(const KeySet& s, uint64_t k) {
    uint64_t i = mix64(k) & s.mask;
    for (uint64_t p = 0; p <= s.mask; ++p) {
        const unsigned long long v = s.keys[i];
        if (v == k) return (long long)i;
        if (v == s.empty) return -1;
        i = (i + 1) & s.mask;
    }
    return -1;
}
__device__ __forceinline__ long long set_insert(const KeySet& s, uint64_t k) {
    uint64_t i = mix64(k) & s.mask;
    for (uint64_t p = 0; p <= s.mask; ++p) {
        const unsigned long long prev = atomicCAS(s.keys + i, s.empty, (unsigned long long)k);
        if (prev == s.empty || prev == k) return (long long)i;
        i = (i + 1) & s.mask;
    }
    return -1;  // full: the host sizes every set to at most half load
}

struct Cell {
    unsigned long long code;
    int depth;
    int pad;
};

// ---------------------------------------------------------------- merge ---

__global__ void k_merge_keys(int64_t n, const tgvg_cube* __restrict__ c, unsigned long long* __restrict__ key,
                             long long* __restrict__ idx) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = ((unsigned long long)c[i].hi << 32) | c[i].lo;
    idx[i] = i;
}

__global__ void k_merge_gather(int64_t n, const tgvg_cube* __restrict__ c, const long long* __restrict__ sidx,
                               tgvg_cube* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = c[sidx[i]];
}

// One stable pairwise merge pass (merge path): run [a, b) with run [b, e) of
// src into dst[a..e), for every pair of a pass in one launch.  A block makes
// MERGE_TILE consecutive outputs of one pair: two warps find how many of them,
// and of those before them, come from the first run (a 32-way search along the
// tile's diagonal), both segments go to shared memory, each thread merges
// MERGE_ITEMS of them from its own diagonal, and the tile is written in order.
// Equal codes: the first run's come first.
//
// Bound by bytes: 16 read and 16 written per cube and pass, whole records, so
// nothing is gathered afterwards; what it reaches, 3.1 TB/s, is set by the
// shared-memory merge.  2,048 outputs a block keep five to six blocks on an SM
// (37 KB each), which covers the searches' latency.  16 lists of 400,000 cubes:
// four passes of 63-66 us where a radix sort of (code, index) pairs took 680 us
// with its keys, and its indices were gathered by the two kernels after it.
constexpr int MERGE_THREADS = 256, MERGE_ITEMS = 8, MERGE_TILE = MERGE_THREADS * MERGE_ITEMS;
// a spare record after every eight: threads whose records lie eight apart meet different banks
__device__ __forceinline__ int merge_at(int i) { return i + (i >> 3); }
struct MergePair {
    int a, b, e;  // the two runs
    int tile;     // the pair's first tile in the pass
};
__device__ __forceinline__ unsigned long long code_of(const uint4& c) { return ((unsigned long long)c.x << 32) | c.y; }

// How many of the first d outputs come from the first run (whole warp).
__device__ __forceinline__ int merge_split(const uint4* __restrict__ A, int na, const uint4* __restrict__ B, int nb,
                                           int d, int lane) {
    int lo = max(0, d - nb), hi = min(d, na);
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32;
        const int x = lo + lane * step + step - 1;
        const bool first = x < hi && code_of(__ldg(A + x)) <= code_of(__ldg(B + (d - 1 - x)));
        const int t = __popc(__ballot_sync(0xffffffffu, first));
        lo = min(hi, lo + t * step);
        hi = min(hi, lo + step - 1);
    }
    return lo;
}

// bad (first pass only): set when a run is not sorted by code.
__global__ void __launch_bounds__(MERGE_THREADS) k_merge_pass(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                            const MergePair* __restrict__ pairs, int npairs,
                                                            int* __restrict__ bad) {
    __shared__ uint4 s[MERGE_TILE + MERGE_TILE / 8];
    __shared__ int s_cut[2];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int lo = 0, hi = npairs - 1;  // last pair that starts at or before this tile
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&pairs[mid].tile) <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const MergePair pr = pairs[lo];
    const uint4 *A = src + pr.a, *B = src + pr.b;
    const int na = pr.b - pr.a, nb = pr.e - pr.b;
    const int d0 = ((int)blockIdx.x - pr.tile) * MERGE_TILE, cnt = min(MERGE_TILE, na + nb - d0), d1 = d0 + cnt;
    if (warp < 2) {
        const int x = merge_split(A, na, B, nb, warp ? d1 : d0, lane);
        if (lane == 0) s_cut[warp] = x;
    }
    __syncthreads();
    const int a0 = s_cut[0], a1 = s_cut[1], b0 = d0 - a0, b1 = d1 - a1;
    if (a1 < a0 || b1 < b0) {  // only where a run is not sorted; the output is not used
        if (bad && t == 0) atomicOr(bad, 1);
        return;
    }
    const int ca = a1 - a0, cb = b1 - b0;
    bool off = false;
    for (int i = t; i < cnt; i += MERGE_THREADS) {
        const bool in_a = i < ca;
        const uint4* p = in_a ? A + a0 + i : B + b0 + (i - ca);
        const uint4 v = __ldg(p);
        s[merge_at(i)] = v;
        if (bad && (in_a ? a0 + i + 1 < na : b0 + (i - ca) + 1 < nb)) off |= code_of(v) > code_of(__ldg(p + 1));
    }
    if (bad && off) atomicOr(bad, 1);
    __syncthreads();
    // this thread's diagonal inside the tile
    const int d = min(t * MERGE_ITEMS, cnt);
    int x = max(0, d - cb);
    for (int h = min(d, ca); x < h;) {
        const int mid = (x + h) >> 1;
        if (code_of(s[merge_at(mid)]) <= code_of(s[merge_at(ca + d - 1 - mid)])) x = mid + 1; else h = mid;
    }
    int y = d - x;
    // the heads of both runs stay in registers; a taken one is replaced by the next record
    // (reads past a run's end meet the other run or the spare record and are not used)
    uint4 r[MERGE_ITEMS], ha = s[merge_at(min(x, MERGE_TILE - 1))], hb = s[merge_at(min(ca + y, MERGE_TILE - 1))];
#pragma unroll
    for (int k = 0; k < MERGE_ITEMS; ++k) {
        if (d + k >= cnt) break;
        const bool first = y >= cb || (x < ca && code_of(ha) <= code_of(hb));
        r[k] = first ? ha : hb;
        x += first;
        y += !first;
        const uint4 h = s[merge_at(min(first ? x : ca + y, MERGE_TILE - 1))];
        if (first) ha = h; else hb = h;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MERGE_ITEMS; ++k)
        if (d + k < cnt) s[merge_at(d + k)] = r[k];
    __syncthreads();
    uint4* out = dst + pr.a + d0;
    for (int i = t; i < cnt; i += MERGE_THREADS) out[i] = s[merge_at(i)];
}

__device__ __forceinline__ bool same_cell(const uint4& a, const uint4& b) {
    return a.x == b.x && a.y == b.y && a.w == b.w;
}

// Runs of equal (code, depth): per tile their number ...
constexpr int RUN_THREADS = 256, RUN_TILE = 2048;
__global__ void __launch_bounds__(RUN_THREADS) k_run_count(int64_t n, const uint4* __restrict__ c, int* __restrict__ sums) {
    __shared__ int ws[RUN_THREADS / 32];
    const int64_t base = (int64_t)blockIdx.x * RUN_TILE;
    int cnt = 0;
    for (int k = threadIdx.x; k < RUN_TILE; k += RUN_THREADS) {
        const int64_t i = base + k;
        if (i < n) cnt += i == 0 || !same_cell(__ldg(c + i), __ldg(c + i - 1));
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int w = 0; w < RUN_THREADS / 32; ++w) s += ws[w];
        sums[blockIdx.x] = s;
    }
}

// ... and, after a scan of those numbers, one cube per run: the reference's
// pending-cube accumulation (merge.cpp:64-88).  A run's sum is a serial chain by
// definition.  One thread takes a short run out of the tile in shared memory; a
// run of RUN_SHORT cubes or more
// (a coarse cell that thousands of pixels fall into) is left for a whole warp,
// which loads 128 records ahead of the chain, so it advances at the latency of an
// add and not of a load.  6.4 M cubes in 1.6 M runs: 325 us (a thread per run,
// gathering) -> 99 us; with runs of more than 6 cubes left to warps 156 us.
constexpr int RUN_SHORT = 41;  // 1 + a multiple of 4: four records are read at a time
__global__ void __launch_bounds__(RUN_THREADS) k_run_emit(int64_t n, const uint4* __restrict__ c,
                                                        const int* __restrict__ sums, uint4* __restrict__ out) {
    __shared__ uint4 s[RUN_TILE + RUN_SHORT];  // the record before the tile, the tile, RUN_SHORT - 1 after it
    __shared__ int ws[RUN_THREADS / 32];
    __shared__ int s_long, s_off[RUN_TILE / RUN_SHORT + 1], s_out[RUN_TILE / RUN_SHORT + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * RUN_TILE;
    int at = sums[blockIdx.x];
    if (threadIdx.x == 0) s_long = 0;
    for (int k = threadIdx.x; k < RUN_TILE + RUN_SHORT; k += RUN_THREADS) {
        const int64_t i = base + k - 1;
        if (i >= 0 && i < n) s[k] = __ldg(c + i);
    }
    __syncthreads();
    for (int k0 = 0; k0 < RUN_TILE; k0 += RUN_THREADS) {
        const int x = k0 + (int)threadIdx.x + 1;  // the record's place in s
        const int64_t i = base + x - 1;
        uint4 p = make_uint4(0, 0, 0, 0);
        bool start = false;
        if (i < n) {
            p = s[x];
            start = i == 0 || !same_cell(p, s[x - 1]);
        }
        const unsigned m = __ballot_sync(0xffffffffu, start);
        if (lane == 0) ws[w] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int q = 0; q < RUN_THREADS / 32; ++q) {
            if (q < w) before += ws[q];
            all += ws[q];
        }
        if (start) {
            const int o = at + before + __popc(m & ((1u << lane) - 1u));
            float sum = __uint_as_float(p.z);
            int cnt = 1;
            bool more = true;
            while (more && cnt < RUN_SHORT) {
                uint4 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = s[x + cnt + q];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    more = more && i + cnt < n && same_cell(v[q], p);
                    if (more) { sum = fadd(sum, __uint_as_float(v[q].z)); ++cnt; }
                }
            }
            // at RUN_SHORT the run may end here or go on: the warp's loop settles it
            if (!more) {
                out[o] = make_uint4(p.x, p.y, __float_as_uint(fdiv(sum, (float)cnt)), p.w);
            } else {  // at least RUN_SHORT cubes: starts lie that far apart, so there is room
                const int q = atomicAdd(&s_long, 1);
                s_off[q] = x - 1;
                s_out[q] = o;
            }
        }
        at += all;
        __syncthreads();
    }
    for (int q = w; q < s_long; q += RUN_THREADS / 32) {
        const int64_t i = base + s_off[q];
        const uint4 p = __ldg(c + i);
        float sum = __uint_as_float(p.z);
        uint32_t cnt = 1;
        auto load = [&](int64_t j) {
            return j < n ? __ldg(c + j) : make_uint4(~p.x, p.y, 0, p.w);  // past the end: another cell
        };
        uint4 v[4];
        int64_t j = i + 1 + lane;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = load(j + 32 * e);
        for (bool more = true; more; j += 128) {
            uint4 nx[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) nx[e] = load(j + 128 + 32 * e);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned in = __ballot_sync(0xffffffffu, same_cell(v[e], p));
                const int len = more ? (in == 0xffffffffu ? 32 : __ffs(~in) - 1) : 0;
                if (len == 32) {
#pragma unroll
                    for (int r = 0; r < 32; ++r) sum = fadd(sum, __uint_as_float(__shfl_sync(0xffffffffu, v[e].z, r)));
                } else {
                    for (int r = 0; r < len; ++r) sum = fadd(sum, __uint_as_float(__shfl_sync(0xffffffffu, v[e].z, r)));
                    more = false;
                }
                cnt += len;
                v[e] = nx[e];
            }
        }
        if (lane == 0) out[s_out[q]] = make_uint4(p.x, p.y, __float_as_uint(fdiv(sum, (float)cnt)), p.w);
    }
}

// -------------------------------------------------------------- balance ---

// Validity of the input cells: depth 0..21 and a code on its depth's grid.
__global__ void k_bal_check(int64_t n, const tgvg_cube* __restrict__ c, int* __restrict__ bad) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int d = c[i].depth;
    const uint64_t code = ((uint64_t)c[i].hi << 32) | c[i].lo;
    if (d < 0 || d > 21 || (code >> 63) != 0 || ancestor_key(code, d) != code) atomicOr(bad, 1);
}

__global__ void k_bal_seed(int64_t n, const tgvg_cube* __restrict__ c, Cell* __restrict__ q,
                           unsigned long long* __restrict__ dck, long long* __restrict__ dci) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t code = ((uint64_t)c[i].hi << 32) | c[i].lo;
    q[i] = Cell{code, c[i].depth, 0};
    dck[i] = dc_key(c[i].depth, code);
    dci[i] = i;
}

// Insert FIFO entries [0, t) into the cell set and the output-key set.
__global__ void k_bal_insert(int64_t t0, int64_t t, const Cell* __restrict__ q, KeySet cells, KeySet dcs) {
    const int64_t i = t0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= t) return;
    const Cell c = q[i];
    set_insert(cells, cell_key(c.code, c.depth));
    set_insert(dcs, dc_key(c.depth, c.code));
}

// One window of the FIFO.  A slot (entry, face) of the reference's queue loop
// (balance.cpp:82-121) adds the parent-depth cell `par` of its face neighbour `nb`
// when neither nb nor par is present, some coarser ancestor of nb is, and par's
// output key is new.  Sets only grow, so a slot for which nb, par or the output
// key is present at the window's start never adds anything and is left out for
// good; what remains (the live slots, a few per cent) is decided in rounds
// against the bridges that earlier live slots add.  Everything about a live
// slot that the rounds need is fixed for the window and worked out once: whether
// a coarser ancestor is present at the start, and where nb, par and par's output
// key lie in tables that hold the live slots' cells and keys.  A round then only
// claims and reads 32-bit numbers at known places, in two launches.
// (Evaluating all slots again from their codes in every round and hashing every
// proposal into fresh tables took 1.2 M cubes in 7 windows 3.1 ms of kernels; the
// live slots 1.0 ms, 0.27 of it the one look at every slot.  A reset, a launch that
// wrote the winners' cells and the two launches left: a call 2.49 -> 2.38 ms.)
constexpr int SLOT_TILE = 2048, SLOT_THREADS = 256;
constexpr unsigned SLOT_NONE = ~0u;

// The face neighbour of slot `me`, or NO_KEY where the slot never adds a bridge.
__device__ __forceinline__ uint64_t slot_nb(const Cell& c, int f) {
    return c.depth >= 2 ? face_key(c.code, f, c.depth) : NO_KEY;
}

// Live slots of the window: one bit each, and their number per tile.
__global__ void __launch_bounds__(SLOT_THREADS) k_bal_first(int64_t h, int64_t m, const Cell* __restrict__ q, KeySet cells,
                                                          KeySet dcs, unsigned* __restrict__ mask, int* __restrict__ sums) {
    __shared__ int ws[SLOT_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int cnt = 0;
    for (int k = 0; k < SLOT_TILE; k += SLOT_THREADS) {
        const int64_t me = (int64_t)blockIdx.x * SLOT_TILE + k + threadIdx.x;
        bool live = false;
        if (me < m) {
            const Cell c = q[h + me / 6];
            const uint64_t nb = slot_nb(c, (int)(me % 6));
            if (nb != NO_KEY && set_slot(cells, cell_key(nb, c.depth)) < 0) {
                const uint64_t par = ancestor_key(nb, c.depth - 1);
                live = set_slot(cells, cell_key(par, c.depth - 1)) < 0 && set_slot(dcs, dc_key(c.depth - 1, par)) < 0;
            }
        }
        const unsigned b = __ballot_sync(0xffffffffu, live);
        if (lane == 0) mask[((int64_t)blockIdx.x * SLOT_TILE + k) / 32 + w] = b;
        cnt += __popc(b);
    }
    if (lane == 0) ws[w] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int x = 0; x < SLOT_THREADS / 32; ++x) s += ws[x];
        sums[blockIdx.x] = s;
    }
}

// The live slots in slot order.
struct Live {
    unsigned* slot;
    unsigned long long* par;  // the cell the slot would add, at depth - 1
    int* nb_at;    // entry of nb among the live cells, -1: none of them
    int* cell_at;  // entry of par
    int* key_at;   // entry of par's output key
    int* cell_key;  // per entry of the cells: its output key's entry
    uint8_t* coarse;  // a coarser ancestor of nb is present at the window's start
    uint8_t* prop;    // the slot proposes its bridge
};

__global__ void __launch_bounds__(SLOT_THREADS) k_bal_live(int64_t h, const Cell* __restrict__ q, KeySet cells,
                                                         const unsigned* __restrict__ mask, const int* __restrict__ sums,
                                                         Live L) {
    constexpr int NW = SLOT_TILE / 32;
    __shared__ unsigned s_mask[NW];
    __shared__ int s_at[NW];
    const int t = threadIdx.x, lane = t & 31;
    if (t < NW) s_mask[t] = mask[(int64_t)blockIdx.x * NW + t];
    __syncthreads();
    if (t < 32) {  // ranks of the tile's words: two per lane
        const int a = __popc(s_mask[2 * t]), b = __popc(s_mask[2 * t + 1]);
        int x = a + b;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        s_at[2 * t] = x - a - b;
        s_at[2 * t + 1] = x - b;
    }
    __syncthreads();
    const int base = sums[blockIdx.x];
    for (int k = 0; k < SLOT_TILE; k += SLOT_THREADS) {
        const int word = (k + t) / 32;
        const unsigned bits = s_mask[word];
        if (!(bits >> lane & 1)) continue;
        const int l = base + s_at[word] + __popc(bits & ((1u << lane) - 1u));
        const unsigned me = blockIdx.x * (unsigned)SLOT_TILE + k + t;
        const Cell c = q[h + me / 6];
        const uint64_t nb = slot_nb(c, (int)(me % 6));
        bool coarse = false;
        for (int d = c.depth - 2; d >= 0 && !coarse; --d) coarse = set_slot(cells, cell_key(ancestor_key(nb, d), d)) >= 0;
        L.slot[l] = me;
        L.par[l] = ancestor_key(nb, c.depth - 1);
        L.coarse[l] = L.prop[l] = coarse;
    }
}

__global__ void k_bal_tables(int nl, int64_t h, const Cell* __restrict__ q, KeySet wcell, KeySet wdc, Live L) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const int d = q[h + L.slot[l] / 6].depth - 1;
    L.cell_at[l] = (int)set_insert(wcell, cell_key(L.par[l], d));
    L.key_at[l] = (int)set_insert(wdc, dc_key(d, L.par[l]));
    L.cell_key[L.cell_at[l]] = L.key_at[l];  // the same from every slot with this cell
}

__global__ void k_bal_nb(int nl, int64_t h, const Cell* __restrict__ q, KeySet wcell, Live L) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const unsigned me = L.slot[l];
    const Cell c = q[h + me / 6];
    L.nb_at[l] = (int)set_slot(wcell, cell_key(slot_nb(c, (int)(me % 6)), c.depth));
}

// A round: proposals of one output key compete for it and the earliest live slot
// wins (the reference's emplace succeeds for the first one only).  An entry holds
// the winner's number in the live list below the round's tag; later rounds have
// smaller tags, so nothing is reset between rounds.
constexpr int TAG_SHIFT = 27;  // 6 WINDOW slots and 24 rounds fit in 32 bits
static_assert(6 * WINDOW <= (int64_t(1) << TAG_SHIFT) && MAX_ROUNDS < (1 << (32 - TAG_SHIFT)) - 1, "tags");
__host__ __device__ __forceinline__ unsigned round_tag(int round) { return unsigned(MAX_ROUNDS - round) << TAG_SHIFT; }

__global__ void k_bal_claim(int nl, Live L, unsigned* __restrict__ winner, unsigned tag) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < nl && L.prop[l]) atomicMin(winner + L.key_at[l], tag | (unsigned)l);
}

// Whether a live slot before l adds the cell at entry e: the winner of its key adds this very cell.
__device__ __forceinline__ bool added_before(const Live& L, const unsigned* __restrict__ winner, unsigned tag, int e, int l) {
    const unsigned w = winner[L.cell_key[e]] - tag;  // below 1 << TAG_SHIFT only with this round's tag
    return w < (unsigned)l && L.cell_at[w] == e;
}

// ... and every live slot is evaluated again against the earlier ones.
__global__ void k_bal_again(int nl, int64_t h, const Cell* __restrict__ q, KeySet wcell,
                            const unsigned* __restrict__ winner, unsigned tag, Live L, unsigned* __restrict__ first_change) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const unsigned me = L.slot[l];
    const int nb_at = L.nb_at[l];
    bool p = !(nb_at >= 0 && added_before(L, winner, tag, nb_at, l)) && !added_before(L, winner, tag, L.cell_at[l], l);
    if (p && !L.coarse[l]) {
        const Cell c = q[h + me / 6];
        const uint64_t nb = slot_nb(c, (int)(me % 6));
        p = false;
        for (int d = c.depth - 2; d >= 0 && !p; --d) {
            const long long e = set_slot(wcell, cell_key(ancestor_key(nb, d), d));
            p = e >= 0 && added_before(L, winner, tag, (int)e, l);
        }
    }
    if (p != (L.prop[l] != 0)) {
        L.prop[l] = p;
        atomicMin(first_change, me);
    }
}

// The bridges that the round's winners add.  Slots below the first change are
// exact; with `limit` only whole entries of them are taken.
__global__ void k_bal_accept(int nl, Live L, const unsigned* __restrict__ winner, unsigned tag,
                             const unsigned* __restrict__ first_change, bool limit, int* __restrict__ acc) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const unsigned change = *first_change;
    acc[l] = L.prop[l] && winner[L.key_at[l]] == (tag | (unsigned)l) &&
             !(limit && change != SLOT_NONE && L.slot[l] >= change / 6 * 6);
}

// Append the accepted bridges to the FIFO, in slot order.
__global__ void k_bal_append(int nl, int64_t h, int64_t t, const Cell* __restrict__ qin, Cell* __restrict__ qout, Live L,
                             const int* __restrict__ acc, const int* __restrict__ apos) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl || !acc[l]) return;
    qout[t + apos[l]] = Cell{L.par[l], qin[h + L.slot[l] / 6].depth - 1, 0};
}

// Output cubes: the input cells averaged per output key in input order
// (balance.cpp:66-75), then the bridges with r_c = r_root / 2^depth (:113).
__global__ void k_bal_starts(int64_t n, const unsigned long long* __restrict__ skey, int* __restrict__ start) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) start[i] = i == 0 || skey[i] != skey[i - 1];
}

__global__ void k_bal_avg(int64_t n, const unsigned long long* __restrict__ skey, const long long* __restrict__ sidx,
                          const tgvg_cube* __restrict__ c, const int* __restrict__ start, const int* __restrict__ pos,
                          unsigned long long* __restrict__ okey, float* __restrict__ orc) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !start[i]) return;
    float sum = 0.0f;
    uint32_t cnt = 0;
    for (int64_t j = i; j < n && (j == i || !start[j]); ++j) {
        sum = fadd(sum, c[sidx[j]].r_c);
        ++cnt;
    }
    const uint64_t k = skey[i];
    okey[pos[i]] = ((k & DC_MASK) << 4) | (k >> 60);
    orc[pos[i]] = fdiv(sum, (float)cnt);
}

__global__ void k_bal_bridges(int64_t nb, const Cell* __restrict__ q, float r_root, int64_t off,
                              unsigned long long* __restrict__ okey, float* __restrict__ orc) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    const Cell c = q[i];
    const uint64_t k = dc_key(c.depth, c.code);
    okey[off + i] = ((k & DC_MASK) << 4) | (k >> 60);
    orc[off + i] = fdiv(r_root, (float)(1u << c.depth));
}

__global__ void k_bal_emit(int64_t n, const unsigned long long* __restrict__ skey, const int* __restrict__ sidx,
                           const float* __restrict__ rc, tgvg_cube* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t k = skey[i];
    const uint64_t code = k >> 4;
    out[i] = tgvg_cube{(uint32_t)(code >> 32), (uint32_t)code, rc[sidx[i]], (int32_t)(k & 15)};
}

__global__ void k_iota(int64_t n, int* __restrict__ v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (int)i;
}

uint64_t pow2_at_least(uint64_t x) {
    uint64_t c = 1024;
    while (c < x) c <<= 1;
    return c;
}

// Device memory of one merge or balance run.  Blocks come from and go back to
// the context's cache of such blocks (tgvg_ctx::ws_get / ws_put: at most
// ws_limit() bytes between calls, given back by tgvg_trim and before one of the
// context's own allocations fails): a merge
// made 9 and a balance about 30 cudaMalloc / cudaFree pairs per call, 0.9 ms of a
// 2.8 ms merge and 4 ms of an 8.4 ms balance.  All uses of a block are on the
// context's stream, so a block may be handed on while kernels still use it.
struct Dev {
    tgvg_ctx* ctx;
    std::vector<void*> ptrs;
    explicit Dev(tgvg_ctx* c) : ctx(c) {}
    ~Dev() {
        for (void* p : ptrs) ctx->ws_put(p);
    }
    template <class T>
    T* get(size_t count) {
        void* p = ctx->ws_get(std::max<size_t>(count, 1) * sizeof(T));
        if (p) ptrs.push_back(p);
        return (T*)p;
    }
    void release(void* p) {
        auto it = std::find(ptrs.begin(), ptrs.end(), p);
        if (it != ptrs.end()) {
            ctx->ws_put(p);
            ptrs.erase(it);
        }
    }
};

// Results go to `vec` (resized) when given, else to `out` when it has room
// (cap), else TGVG_ERR_LIMIT; *count receives their number.
int merge_dev(tgvg_ctx* ctx, const tgvg_cube* const* in, const int64_t* counts, int k, std::vector<tgvg_cube>* vec,
              tgvg_cube* out, int64_t cap, int64_t* count) {
    int64_t n = 0;
    for (int s = 0; s < k; ++s) n += counts[s];
    *count = 0;
    if (vec) vec->clear();
    if (n == 0) return TGVG_OK;
    if (n > (int64_t(1) << 31) - 1) return ctx->fail(TGVG_ERR_LIMIT, "more than 2^31 - 1 cubes");
    cudaStream_t st = ctx->stream;
    Dev D(ctx);
    auto* cat = D.get<tgvg_cube>(n);
    auto* oth = D.get<tgvg_cube>(n);
    const int64_t ntiles = (n + RUN_TILE - 1) / RUN_TILE;
    auto* sums = D.get<int>(ntiles + 2);  // [ntiles] total, [ntiles + 1] an input is not sorted
    if (!cat || !oth || !sums) return ctx->fail(TGVG_ERR_NOMEM, "merge buffers");
    auto upload = [&]() -> int {
        int64_t off = 0;
        for (int s = 0; s < k; ++s) {
            if (counts[s])
                TGVG_CK(ctx, cudaMemcpyAsync(cat + off, in[s], sizeof(tgvg_cube) * counts[s], cudaMemcpyHostToDevice, st));
            off += counts[s];
        }
        return TGVG_OK;
    };
    int rc = upload();
    if (rc) return rc;
    // The passes: runs of the concatenation, joined two by two until one is left
    // (a single input still takes one pass, which checks that it is sorted).
    std::vector<int> runs_at;  // run starts, then n
    {
        int64_t off = 0;
        for (int s = 0; s < k; ++s) {
            if (counts[s]) runs_at.push_back((int)off);
            off += counts[s];
        }
        runs_at.push_back((int)n);
    }
    std::vector<MergePair> table;
    struct Pass { int first, pairs, tiles; };
    std::vector<Pass> passes;
    do {
        Pass ps{(int)table.size(), 0, 0};
        std::vector<int> next;
        for (size_t r = 0; r + 1 < runs_at.size(); r += 2) {
            const int a = runs_at[r], b = runs_at[r + 1], e = r + 2 < runs_at.size() ? runs_at[r + 2] : b;
            table.push_back({a, b, e, ps.tiles});
            ps.tiles += (int)(((int64_t)e - a + MERGE_TILE - 1) / MERGE_TILE);
            ++ps.pairs;
            next.push_back(a);
        }
        next.push_back((int)n);
        runs_at.swap(next);
        passes.push_back(ps);
    } while (runs_at.size() > 2);
    auto* d_table = D.get<MergePair>(table.size());
    if (!d_table) return ctx->fail(TGVG_ERR_NOMEM, "merge buffers");
    TGVG_CK(ctx, cudaMemcpyAsync(d_table, table.data(), sizeof(MergePair) * table.size(), cudaMemcpyHostToDevice, st));
    int* bad = sums + ntiles + 1;
    TGVG_CK(ctx, cudaMemsetAsync(bad, 0, sizeof(int), st));
    for (size_t q = 0; q < passes.size(); ++q) {
        k_merge_pass<<<(unsigned)passes[q].tiles, MERGE_THREADS, 0, st>>>(
            reinterpret_cast<const uint4*>(cat), reinterpret_cast<uint4*>(oth), d_table + passes[q].first,
            passes[q].pairs, q == 0 ? bad : nullptr);
        TGVG_LAUNCHED(ctx);
        std::swap(cat, oth);
    }
    auto count_runs = [&](int64_t* total, bool* unsorted) -> int {
        k_run_count<<<(unsigned)ntiles, RUN_THREADS, 0, st>>>(n, reinterpret_cast<const uint4*>(cat), sums);
        TGVG_LAUNCHED(ctx);
        const int src = scan_tile_sums(ctx, sums, (int)ntiles);
        if (src) return src;
        int h[2] = {0, 0};
        TGVG_CK(ctx, cudaMemcpyAsync(h, sums + ntiles, sizeof(h), cudaMemcpyDeviceToHost, st));
        TGVG_CK(ctx, cudaStreamSynchronize(st));
        *total = h[0];
        *unsorted = h[1] != 0;
        return TGVG_OK;
    };
    int64_t runs = 0;
    bool unsorted = false;
    if ((rc = count_runs(&runs, &unsorted))) return rc;
    if (unsorted) {  // stable radix sort of the concatenation
        if ((rc = upload())) return rc;
        auto* key = D.get<unsigned long long>(n);
        auto* skey = D.get<unsigned long long>(n);
        auto* idx = D.get<long long>(n);
        auto* sidx = D.get<long long>(n);
        if (!key || !skey || !idx || !sidx) return ctx->fail(TGVG_ERR_NOMEM, "merge buffers");
        k_merge_keys<<<grid_of(n, 256), 256, 0, st>>>(n, cat, key, idx);
        TGVG_LAUNCHED(ctx);
        size_t tb = 0;
        TGVG_CK(ctx, cub::DeviceRadixSort::SortPairs(nullptr, tb, key, skey, idx, sidx, (int)n, 0, 63, st));
        void* tmp = D.get<char>(tb);
        if (!tmp) return ctx->fail(TGVG_ERR_NOMEM, "merge sort buffer");
        TGVG_CK(ctx, cub::DeviceRadixSort::SortPairs(tmp, tb, key, skey, idx, sidx, (int)n, 0, 63, st));
        k_merge_gather<<<grid_of(n, 256), 256, 0, st>>>(n, cat, sidx, oth);
        TGVG_LAUNCHED(ctx);
        std::swap(cat, oth);
        if ((rc = count_runs(&runs, &unsorted))) return rc;
    }
    tgvg_cube* res = oth;  // at most n runs
    k_run_emit<<<(unsigned)ntiles, RUN_THREADS, 0, st>>>(n, reinterpret_cast<const uint4*>(cat), sums,
                                                        reinterpret_cast<uint4*>(res));
    TGVG_LAUNCHED(ctx);
    *count = runs;
    if (vec) {
        vec->resize(size_t(runs));
        out = vec->data();
    } else if (!out) {
        return TGVG_OK;
    } else if (cap < runs) {
        return TGVG_ERR_LIMIT;
    }
    TGVG_CK(ctx, cudaMemcpyAsync(out, res, sizeof(tgvg_cube) * runs, cudaMemcpyDeviceToHost, st));
    TGVG_CK(ctx, cudaStreamSynchronize(st));
    return TGVG_OK;
}

struct BalanceSets {
    unsigned long long* cell_keys = nullptr;
    unsigned long long* dc_keys = nullptr;
    uint64_t cap = 0;
    KeySet cells() const { return KeySet{cell_keys, cap - 1, CELL_EMPTY}; }
    KeySet dcs() const { return KeySet{dc_keys, cap - 1, DC_EMPTY}; }
};

// Results as merge_dev's.
int balance_dev(tgvg_ctx* ctx, const tgvg_cube* cubes, int64_t n, float r_root, std::vector<tgvg_cube>* vec,
                tgvg_cube* out, int64_t cap, int64_t* count) {
    *count = 0;
    if (vec) vec->clear();
    if (n == 0) return TGVG_OK;
    if (n > (int64_t(1) << 30)) return ctx->fail(TGVG_ERR_LIMIT, "more than 2^30 cubes");
    cudaStream_t st = ctx->stream;
    Dev D(ctx);
    auto* c = D.get<tgvg_cube>(n);
    auto* bad = D.get<int>(1);
    if (!c || !bad) return ctx->fail(TGVG_ERR_NOMEM, "balance buffers");
    TGVG_CK(ctx, cudaMemcpyAsync(c, cubes, sizeof(tgvg_cube) * n, cudaMemcpyHostToDevice, st));
    TGVG_CK(ctx, cudaMemsetAsync(bad, 0, sizeof(int), st));
    k_bal_check<<<grid_of(n, 256), 256, 0, st>>>(n, c, bad);
    TGVG_LAUNCHED(ctx);
    int hbad = 0;
    TGVG_CK(ctx, cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
    TGVG_CK(ctx, cudaStreamSynchronize(st));
    if (hbad) return ctx->fail(TGVG_ERR_INVALID, "balance input holds a cube whose depth is outside 0..21 or "
                                                 "whose code is not on its depth's grid");

    // FIFO (grows), the two sets (rebuilt larger when half full), output keys of the inputs.
    int64_t qcap = std::max<int64_t>(2 * n, 4096);
    Cell* q = D.get<Cell>(qcap);
    auto* dck = D.get<unsigned long long>(n);
    auto* sdck = D.get<unsigned long long>(n);
    auto* dci = D.get<long long>(n);
    auto* sdci = D.get<long long>(n);
    if (!q || !dck || !sdck || !dci || !sdci) return ctx->fail(TGVG_ERR_NOMEM, "balance buffers");
    k_bal_seed<<<grid_of(n, 256), 256, 0, st>>>(n, c, q, dck, dci);
    TGVG_LAUNCHED(ctx);
    BalanceSets S;
    auto build_sets = [&](uint64_t cap, int64_t t) -> int {
        if (S.cell_keys) D.release(S.cell_keys);
        if (S.dc_keys) D.release(S.dc_keys);
        S.cap = cap;
        S.cell_keys = D.get<unsigned long long>(cap);
        S.dc_keys = D.get<unsigned long long>(cap);
        if (!S.cell_keys || !S.dc_keys) return ctx->fail(TGVG_ERR_NOMEM, "balance sets");
        TGVG_CK(ctx, cudaMemsetAsync(S.cell_keys, 0x00, sizeof(unsigned long long) * cap, st));
        TGVG_CK(ctx, cudaMemsetAsync(S.dc_keys, 0xff, sizeof(unsigned long long) * cap, st));
        k_bal_insert<<<grid_of(t, 256), 256, 0, st>>>(0, t, q, S.cells(), S.dcs());
        TGVG_LAUNCHED(ctx);
        return TGVG_OK;
    };
    int rc = build_sets(pow2_at_least(4 * uint64_t(n)), n);
    if (rc) return rc;

    int64_t h = 0, t = n;
    while (h < t) {
        const int64_t wn = std::min<int64_t>(t - h, WINDOW);
        const int64_t m = 6 * wn, tiles = (m + SLOT_TILE - 1) / SLOT_TILE;
        Dev W(ctx);  // this window's scratch
        auto* mask = W.get<unsigned>(tiles * (SLOT_TILE / 32));
        auto* sums = W.get<int>(tiles + 1);
        if (!mask || !sums) return ctx->fail(TGVG_ERR_NOMEM, "balance window buffers");
        k_bal_first<<<(unsigned)tiles, SLOT_THREADS, 0, st>>>(h, m, q, S.cells(), S.dcs(), mask, sums);
        TGVG_LAUNCHED(ctx);
        if ((rc = scan_tile_sums(ctx, sums, (int)tiles))) return rc;
        int nl = 0;
        TGVG_CK(ctx, cudaMemcpyAsync(&nl, sums + tiles, sizeof(int), cudaMemcpyDeviceToHost, st));
        TGVG_CK(ctx, cudaStreamSynchronize(st));
        if (nl == 0) {
            h += wn;
            continue;
        }
        const uint64_t wc = pow2_at_least(2 * uint64_t(nl));
        Live L{W.get<unsigned>(nl), W.get<unsigned long long>(nl), W.get<int>(nl), W.get<int>(nl), W.get<int>(nl),
               W.get<int>(wc), W.get<uint8_t>(nl), W.get<uint8_t>(nl)};
        auto* wcell = W.get<unsigned long long>(wc);
        auto* wdc = W.get<unsigned long long>(wc);
        auto* winner = W.get<unsigned>(wc + MAX_ROUNDS);  // per key entry; then each round's first change
        auto* acc = W.get<int>(nl);
        auto* apos = W.get<int>(nl);
        const int64_t nsum = scan_sums_len(nl);
        auto* asum = W.get<int>(nsum);
        if (!L.slot || !L.par || !L.nb_at || !L.cell_at || !L.key_at || !L.cell_key || !L.coarse || !L.prop || !wcell || !wdc || !winner ||
            !acc || !apos || !asum)
            return ctx->fail(TGVG_ERR_NOMEM, "balance window buffers");
        unsigned* first = winner + wc;
        const KeySet kcell{wcell, wc - 1, CELL_EMPTY}, kdc{wdc, wc - 1, DC_EMPTY};
        TGVG_CK(ctx, cudaMemsetAsync(wcell, 0x00, sizeof(unsigned long long) * wc, st));
        TGVG_CK(ctx, cudaMemsetAsync(wdc, 0xff, sizeof(unsigned long long) * wc, st));
        TGVG_CK(ctx, cudaMemsetAsync(winner, 0xff, sizeof(unsigned) * (wc + MAX_ROUNDS), st));
        k_bal_live<<<(unsigned)tiles, SLOT_THREADS, 0, st>>>(h, q, S.cells(), mask, sums, L);
        TGVG_LAUNCHED(ctx);
        const unsigned lg = grid_of(nl, 256);
        k_bal_tables<<<lg, 256, 0, st>>>(nl, h, q, kcell, kdc, L);
        TGVG_LAUNCHED(ctx);
        k_bal_nb<<<lg, 256, 0, st>>>(nl, h, q, kcell, L);
        TGVG_LAUNCHED(ctx);
        // Rounds in batches, the host looking at the end of each: a round after
        // the proposals settled changes nothing.
        int rounds = 0, na = 0;
        unsigned change = SLOT_NONE;
        for (int batch = 3; rounds < MAX_ROUNDS; batch *= 2) {
            const int upto = std::min(MAX_ROUNDS, rounds + batch);
            for (; rounds < upto; ++rounds) {
                k_bal_claim<<<lg, 256, 0, st>>>(nl, L, winner, round_tag(rounds));
                TGVG_LAUNCHED(ctx);
                k_bal_again<<<lg, 256, 0, st>>>(nl, h, q, kcell, winner, round_tag(rounds), L, first + rounds);
                TGVG_LAUNCHED(ctx);
            }
            // (at the last round allowed, what lies below the first change is committed)
            k_bal_accept<<<lg, 256, 0, st>>>(nl, L, winner, round_tag(rounds - 1), first + rounds - 1,
                                             rounds == MAX_ROUNDS, acc);
            TGVG_LAUNCHED(ctx);
            if ((rc = scan_exclusive_async(ctx, acc, nl, apos, asum))) return rc;
            TGVG_CK(ctx, cudaMemcpyAsync(&change, first + rounds - 1, sizeof(change), cudaMemcpyDeviceToHost, st));
            TGVG_CK(ctx, cudaMemcpyAsync(&na, asum + nsum - 1, sizeof(na), cudaMemcpyDeviceToHost, st));
            TGVG_CK(ctx, cudaStreamSynchronize(st));
            if (change == SLOT_NONE) break;  // settled: the sequential result
        }
        const int64_t done = change == SLOT_NONE ? wn : int64_t(change / 6);  // FIFO entries finished in this window
        if (na > 0) {
            Cell* qout = q;
            const int64_t ncap = std::max<int64_t>(2 * qcap, t + na);
            if (t + na > qcap) {  // grow the FIFO, keeping its contents
                qout = D.get<Cell>(ncap);
                if (!qout) return ctx->fail(TGVG_ERR_NOMEM, "balance queue");
                TGVG_CK(ctx, cudaMemcpyAsync(qout, q, sizeof(Cell) * t, cudaMemcpyDeviceToDevice, st));
            }
            k_bal_append<<<lg, 256, 0, st>>>(nl, h, t, q, qout, L, acc, apos);
            TGVG_LAUNCHED(ctx);
            if (qout != q) {
                D.release(q);
                q = qout;
                qcap = ncap;
            }
            if (uint64_t(t + na) * 2 > S.cap) {
                rc = build_sets(pow2_at_least(4 * uint64_t(t + na)), t + na);
                if (rc) return rc;
            } else {
                k_bal_insert<<<grid_of(na, 256), 256, 0, st>>>(t, t + na, q, S.cells(), S.dcs());
                TGVG_LAUNCHED(ctx);
            }
        }
        h += done;
        t += na;
    }

    // Output: averaged input keys, then the bridges, sorted by (code, depth).
    size_t tb = 0;
    TGVG_CK(ctx, cub::DeviceRadixSort::SortPairs(nullptr, tb, dck, sdck, dci, sdci, (int)n, 0, 64, st));
    void* tmp = D.get<char>(tb);
    if (!tmp) return ctx->fail(TGVG_ERR_NOMEM, "balance sort buffer");
    TGVG_CK(ctx, cub::DeviceRadixSort::SortPairs(tmp, tb, dck, sdck, dci, sdci, (int)n, 0, 64, st));
    auto* start = D.get<int>(n);
    auto* spos = D.get<int>(n);
    if (!start || !spos) return ctx->fail(TGVG_ERR_NOMEM, "balance buffers");
    k_bal_starts<<<grid_of(n, 256), 256, 0, st>>>(n, sdck, start);
    TGVG_LAUNCHED(ctx);
    int64_t nu = 0;
    rc = scan_exclusive(ctx, start, n, spos, &nu);
    if (rc) return rc;
    const int64_t nb = t - n, no = nu + nb;
    auto* okey = D.get<unsigned long long>(no);
    auto* sokey = D.get<unsigned long long>(no);
    auto* orc = D.get<float>(no);
    auto* oidx = D.get<int>(no);
    auto* soidx = D.get<int>(no);
    auto* res = D.get<tgvg_cube>(no);
    if (!okey || !sokey || !orc || !oidx || !soidx || !res) return ctx->fail(TGVG_ERR_NOMEM, "balance output");
    k_bal_avg<<<grid_of(n, 256), 256, 0, st>>>(n, sdck, sdci, c, start, spos, okey, orc);
    TGVG_LAUNCHED(ctx);
    if (nb > 0) {
        k_bal_bridges<<<grid_of(nb, 256), 256, 0, st>>>(nb, q + n, r_root, nu, okey, orc);
        TGVG_LAUNCHED(ctx);
    }
    k_iota<<<grid_of(no, 256), 256, 0, st>>>(no, oidx);
    TGVG_LAUNCHED(ctx);
    tb = 0;
    TGVG_CK(ctx, cub::DeviceRadixSort::SortPairs(nullptr, tb, okey, sokey, oidx, soidx, (int)no, 0, 64, st));
    void* tmp2 = D.get<char>(tb);
    if (!tmp2) return ctx->fail(TGVG_ERR_NOMEM, "balance sort buffer");
    TGVG_CK(ctx, cub::DeviceRadixSort::SortPairs(tmp2, tb, okey, sokey, oidx, soidx, (int)no, 0, 64, st));
    k_bal_emit<<<grid_of(no, 256), 256, 0, st>>>(no, sokey, soidx, orc, res);
    TGVG_LAUNCHED(ctx);
    *count = no;
    if (vec) {
        vec->resize(size_t(no));
        out = vec->data();
    } else if (!out) {
        return TGVG_OK;
    } else if (cap < no) {
        return TGVG_ERR_LIMIT;
    }
    TGVG_CK(ctx, cudaMemcpyAsync(out, res, sizeof(tgvg_cube) * no, cudaMemcpyDeviceToHost, st));
    TGVG_CK(ctx, cudaStreamSynchronize(st));
    return TGVG_OK;
}

int write_cube_file(const char* path, float r_root, const std::vector<tgvg_cube>& cubes) {
    char hdr[16] = {'T', 'G', 'V', '1'};
    const uint32_t ver = 1, cnt = uint32_t(cubes.size());
    std::memcpy(hdr + 4, &ver, 4);
    std::memcpy(hdr + 8, &r_root, 4);
    std::memcpy(hdr + 12, &cnt, 4);
    return fileio::write_file(path, hdr, 16, cubes.data(), sizeof(tgvg_cube) * cubes.size());
}

}  // namespace
}  // namespace tgvg

using namespace tgvg;

extern "C" int tgvg_merge_cubes(tgvg_ctx* ctx, const tgvg_cube* const* arrays, const int64_t* counts, int32_t k,
                                tgvg_cube* out, int64_t cap, int64_t* count) {
    if (!ctx || !count || k < 0 || (k > 0 && (!arrays || !counts))) return TGVG_ERR_INVALID;
    for (int s = 0; s < k; ++s)
        if (counts[s] < 0 || (counts[s] > 0 && !arrays[s])) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    return merge_dev(ctx, arrays, counts, k, nullptr, out, cap, count);
}

extern "C" int tgvg_kway_merge(tgvg_ctx* ctx, const char* const* in_paths, int32_t k, const char* out_path) {
    if (!ctx || k < 0 || (k > 0 && !in_paths) || !out_path) return TGVG_ERR_INVALID;
    std::vector<std::vector<tgvg_cube>> ins(size_t(std::max(k, 0)));
    float r_root = 0.0f;
    for (int s = 0; s < k; ++s) {
        // merge.cpp:30-40 reads each stream's cubes until the file ends
        std::vector<char> b;
        int rc = fileio::read_file(in_paths[s], b);
        if (rc) return ctx->fail(rc, std::string("Cannot open: ") + (in_paths[s] ? in_paths[s] : ""));
        if (b.size() < 16 || std::memcmp(b.data(), "TGV1", 4) != 0)
            return ctx->fail(TGVG_ERR_FORMAT, std::string("Bad magic: ") + in_paths[s]);
        if (s == 0) std::memcpy(&r_root, b.data() + 8, 4);
        const size_t nc = (b.size() - 16) / sizeof(tgvg_cube);
        ins[s].resize(nc);
        if (nc) std::memcpy(ins[s].data(), b.data() + 16, nc * sizeof(tgvg_cube));
    }
    std::vector<const tgvg_cube*> ptr;
    std::vector<int64_t> cnt;
    for (auto& v : ins) {
        ptr.push_back(v.data());
        cnt.push_back(int64_t(v.size()));
    }
    std::vector<tgvg_cube> res;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        int64_t nres = 0;
        const int rc = merge_dev(ctx, ptr.data(), cnt.data(), k, &res, nullptr, 0, &nres);
        if (rc) return rc;
    }
    const int rc = write_cube_file(out_path, r_root, res);
    return rc ? ctx->fail(rc, std::string("Cannot open output: ") + out_path) : TGVG_OK;
}

extern "C" int tgvg_balance_cubes(tgvg_ctx* ctx, const tgvg_cube* cubes, int64_t n, float r_root, tgvg_cube* out,
                                  int64_t cap, int64_t* count) {
    if (!ctx || !count || n < 0 || (n > 0 && !cubes)) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    return balance_dev(ctx, cubes, n, r_root, nullptr, out, cap, count);
}

extern "C" int tgvg_balance_octree(tgvg_ctx* ctx, const char* in_path, const char* out_path) {
    if (!ctx || !in_path || !out_path) return TGVG_ERR_INVALID;
    std::vector<tgvg_cube> cubes;
    float r_root = 0.0f;
    int rc = fileio::load_cube_file(in_path, cubes, &r_root);
    if (rc) return ctx->fail(rc, std::string(rc == TGVG_ERR_IO ? "Cannot open cube file: " : "Bad magic in cube file: ") +
                                     in_path);
    std::vector<tgvg_cube> res;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        int64_t nres = 0;
        rc = balance_dev(ctx, cubes.data(), int64_t(cubes.size()), r_root, &res, nullptr, 0, &nres);
        if (rc) return rc;
    }
    rc = write_cube_file(out_path, r_root, res);
    return rc ? ctx->fail(rc, std::string("Cannot open output: ") + out_path) : TGVG_OK;
}
