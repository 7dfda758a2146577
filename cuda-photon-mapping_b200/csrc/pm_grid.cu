// pm_grid.cu -- photon grid build.
//
// Reference: CudaPhotonMapping/PhotonGrid.cu:41-218 (analyze_density,
// count_photons_per_cell, prescan_per_cell_counts, assign_photons_to_cells).
// The reference scatters with an atomic per-cell offset, so the order inside a
// cell changes from run to run.  Here the order inside a cell is defined: by
// sub-cell (each cell split S x S x S, S chosen for the gather) and then by
// trace order, which makes the sorted arrays a pure function of the photon
// list; cell_starts / cell_sizes are the reference's exactly.  Pipeline (one stream, no host round trip except the
// re-grid decision the reference also takes on the host):
//   k_count_cells  per-cell counts of both candidate grids (the desired
//                  resolution and the re-grid one) and their largest counts
//                  (shared-memory counters + k_count_max when both grids fit)
//                  -> host decides on the re-grid and on S
//   k_cell_rank (many cells: k_cell_flags + scan_u32)   rank of each cell among those that hold photons
//   k_key_count    key = rank * S^3 + sub-cell per photon + key counts
//   scan_u32       exclusive scan of key counts (decoupled look-back)
//   k_key_starts   key_starts of all sub-cells; cell_starts, cell_sizes
//   LSD radix sort of the keys, <= 9 bits per pass, carrying the photon index:
//     k_radix_count    digit counts of every block's run of keys
//     k_radix_offsets  their prefixes over the blocks
//     k_radix_pass     stable in-tile ranks (per-bit ballots) + scatter
//     (up to 1.8M keys: k_radix_hist once, then k_radix_pass alone, its tiles
//     looking back over each other)
//   k_grid_gather  sorted photon index -> (pos, id), dir, power in slot order
#include <cmath>
#include <algorithm>
#include "pm_grid.cuh"
#include "pm_scan.cuh"
#include "pm_device.cuh"

namespace pm {

namespace {

// 512 threads of 8 keys per tile (3 blocks, 48 warps per SM): the ranking and
// staging phases are latency bound, so resident warps pay (256 x 16 keys, 32
// warps: 7 % more for the grid build of 10M photons; 256 x 8: 4 %).
// RADIX_THREADS >= RADIX_MAX_BINS (one thread per digit).
constexpr int RADIX_THREADS = 512;
constexpr int RADIX_ITEMS = 8;
constexpr int RADIX_TILE = RADIX_THREADS * RADIX_ITEMS;
constexpr int RADIX_WARPS = RADIX_THREADS / 32;
constexpr int RADIX_MAX_BITS = 9;
constexpr int RADIX_MAX_BINS = 1 << RADIX_MAX_BITS;
static_assert(RADIX_THREADS >= RADIX_MAX_BINS, "one thread per digit");
constexpr int RADIX_MAX_PASSES = 4;    // 32-bit keys, <= 9 bits each
// Blocks of a pass, all resident (3 per SM by shared memory): up to as many tiles
// one tile each, beyond that each block takes a run of consecutive tiles.
constexpr int RADIX_BLOCKS = 3 * 148;

struct GridGeom {
    float mnx, mny, mnz;
    int gx, gy, gz;
    float cell;
    float inv;        // 1 / cell
};

// The sub-cell index along one axis: with u = (p - min) / cell in IEEE float, the
// truncated u selects the cell (clamped to the grid) and its fractional part the
// sub-cell, together trunc(u S) clamped to [0, g S) (u S and u - cell are exact).
// The product with 1 / cell differs from u by under 2e-7 u, so the division is
// made only where that product lies near an integer that decides (not one at or
// beyond the ends, where walls are).  Counting pass of 10M photons (six
// quotients each) 0.124 -> 0.083 ms.
__device__ __noinline__ int exact_index(float d, float cell, float S) { return (int)((d / cell) * S); }   // (a call: not hoisted)
template <int LOG_S>
__device__ __forceinline__ int sub_index(float p, float mn, float cell, float inv, int log_s, int g) {
    const int sh = LOG_S >= 0 ? LOG_S : log_s;
    const float S = (float)(1 << sh);
    const float d = p - mn, w = d * inv * S;
    const float r = rintf(w);
    const int last = (g << sh) - 1;
    int i = (int)w;
    if (fabsf(w - r) <= 1e-5f + 4e-7f * w && r >= 1.f && r <= (float)last) i = exact_index(d, cell, S);
    return min(max(i, 0), last);
}

__device__ __forceinline__ uint32_t cell_of(const GridGeom& g, float px, float py, float pz) {
    const int x = sub_index<0>(px, g.mnx, g.cell, g.inv, 0, g.gx);
    const int y = sub_index<0>(py, g.mny, g.cell, g.inv, 0, g.gy);
    const int z = sub_index<0>(pz, g.mnz, g.cell, g.inv, 0, g.gz);
    return (uint32_t)(x + y * g.gx + z * g.gx * g.gy);
}

// Shared-memory variant of k_count_cells for grids whose cells fit in shared
// memory as 16-bit counters (two per 32-bit word; a block counts at most
// COUNT_CHUNK <= 65535 photons, so a half-word never carries into its
// neighbour).  Photons land on a few thousand hot surface cells, so global
// atomics on the cell counters contend; here each block adds into its own
// copy and flushes its non-zero counters once.
constexpr int COUNT_THREADS = 1024;
constexpr int COUNT_CHUNK = 65535;
constexpr int COUNT_SMEM_WORDS = 56 * 1024;   // 224 KB: 114,688 16-bit counters

// Photons [blockIdx.x * chunk, ... + chunk) (chunk <= COUNT_CHUNK, so no
// 16-bit counter can overflow).
__global__ void __launch_bounds__(COUNT_THREADS)
k_count_cells_smem(const float* __restrict__ pos, int64_t n, int64_t chunk, GridGeom ga, GridGeom gb, int two,
                   int cells_a, int cells_b, uint32_t* __restrict__ ca, uint32_t* __restrict__ cb) {
    extern __shared__ uint32_t h16[];
    const int words_a = (cells_a + 1) >> 1, words = words_a + (two ? (cells_b + 1) >> 1 : 0);
    for (int i = threadIdx.x; i < words; i += COUNT_THREADS) h16[i] = 0u;
    __syncthreads();
    const int64_t first = (int64_t)blockIdx.x * chunk;
    const int64_t last = min(first + chunk, n);
    for (int64_t i = first + threadIdx.x; i < last; i += COUNT_THREADS) {
        const float* p = pos + 3 * i;
        const float x = p[0], y = p[1], z = p[2];
        const uint32_t c = cell_of(ga, x, y, z);
        atomicAdd(&h16[c >> 1], 1u << (16 * (c & 1u)));
        if (two) {
            const uint32_t c2 = cell_of(gb, x, y, z);
            atomicAdd(&h16[words_a + (c2 >> 1)], 1u << (16 * (c2 & 1u)));
        }
    }
    __syncthreads();
    for (int w = threadIdx.x; w < words; w += COUNT_THREADS) {
        const uint32_t v = h16[w];
        if (!v) continue;
        const bool in_a = w < words_a;
        uint32_t* dst = in_a ? ca : cb;
        const int cell = 2 * (in_a ? w : w - words_a);
        if (v & 0xffffu) atomicAdd(dst + cell, v & 0xffffu);
        if (v >> 16) atomicAdd(dst + cell + 1, v >> 16);
    }
}

// largest counts of the two count arrays: mx[0] (a), mx[1] (b); cells that hold
// photons: mx[2], mx[3]
__global__ void k_count_max(const uint32_t* __restrict__ ca, int64_t na, const uint32_t* __restrict__ cb, int64_t nb,
                            uint32_t* mx) {
    uint32_t ma = 0u, mb = 0u, fa = 0u, fb = 0u;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < na; i += stride) {
        const uint32_t c = ca[i];
        ma = max(ma, c);
        fa += c ? 1u : 0u;
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += stride) {
        const uint32_t c = cb[i];
        mb = max(mb, c);
        fb += c ? 1u : 0u;
    }
    fa = __reduce_add_sync(0xffffffffu, fa);
    fb = __reduce_add_sync(0xffffffffu, fb);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ma = max(ma, __shfl_xor_sync(0xffffffffu, ma, o));
        mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (ma) atomicMax(mx, ma);
        if (mb) atomicMax(mx + 1, mb);
        if (fa) atomicAdd(mx + 2, fa);
        if (fb) atomicAdd(mx + 3, fb);
    }
}

// photon counts of grid a and (when two) grid b
__global__ void k_count_cells(const float* __restrict__ pos, int64_t n, GridGeom ga, GridGeom gb, int two,
                              uint32_t* __restrict__ ca, uint32_t* __restrict__ cb) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* p = pos + 3 * i;
    const float x = p[0], y = p[1], z = p[2];
    atomicAdd(ca + cell_of(ga, x, y, z), 1u);
    if (two) atomicAdd(cb + cell_of(gb, x, y, z), 1u);
}

// cell and sub-cell of a photon; sub-cell key = cell * S^3 + sub-cell
__device__ __forceinline__ uint32_t sub_cell_of(const GridGeom& g, int sh, const float* p, uint32_t& cell) {
    const int x = sub_index<-1>(p[0], g.mnx, g.cell, g.inv, sh, g.gx);
    const int y = sub_index<-1>(p[1], g.mny, g.cell, g.inv, sh, g.gy);
    const int z = sub_index<-1>(p[2], g.mnz, g.cell, g.inv, sh, g.gz);
    const int m = (1 << sh) - 1;
    cell = (uint32_t)((x >> sh) + (y >> sh) * g.gx + (z >> sh) * g.gx * g.gy);
    return (uint32_t)((x & m) + (((y & m) + ((z & m) << sh)) << sh));
}

// The photons lie on surfaces, in a tenth of the cells: sort keys count only the
// cells that hold photons (rank[cell]), which keeps the order, shortens the keys
// by three or four bits and the count array by as much.
// One block: ranks of up to RANK_CELLS cells in one launch (beyond: flags + scan).
constexpr int RANK_THREADS = 1024;
constexpr int64_t RANK_CELLS = 8 * RANK_THREADS;   // 50K cells: 22 us, flags + scan 13
__global__ void __launch_bounds__(RANK_THREADS)
k_cell_rank(const uint32_t* __restrict__ counts, int cells, uint32_t* __restrict__ rank) {
    __shared__ uint32_t wsum[RANK_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t before = 0u;   // cells with photons before this round of RANK_THREADS
    for (int c0 = 0; c0 < cells; c0 += RANK_THREADS) {
        const int c = c0 + (int)threadIdx.x;
        const bool full = c < cells && counts[c] != 0u;
        const unsigned m = __ballot_sync(0xffffffffu, full);
        if (lane == 0) wsum[warp] = (uint32_t)__popc(m);
        __syncthreads();
        const uint32_t w = wsum[lane];
        const uint32_t off = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
        if (c < cells) rank[c] = before + off + (uint32_t)__popc(m & lanemask_lt());
        before += __reduce_add_sync(0xffffffffu, w);
        __syncthreads();
    }
}

__global__ void k_cell_flags(const uint32_t* __restrict__ counts, int64_t cells, uint32_t* __restrict__ flags) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < cells) flags[c] = counts[c] ? 1u : 0u;
}

__global__ void k_key_count(const float* __restrict__ pos, int64_t n, GridGeom g, int sh, const uint32_t* __restrict__ rank,
                            uint32_t* __restrict__ key, uint32_t* __restrict__ counts) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t cell;
    const uint32_t s = sub_cell_of(g, sh, pos + 3 * i, cell);
    const uint32_t k = (__ldg(rank + cell) << (3 * sh)) + s;
    key[i] = k;
    atomicAdd(counts + k, 1u);
}

// key_starts of all sub-cells from the starts of those whose cell holds photons
// (starts[rank * S^3 + sub-cell], the total last); cell_starts and cell_sizes
// (which may be counts itself).
// PER = 4 keys per thread (S > 1: of one cell), one 16-byte store; bound by the 4
// bytes written per sub-cell (25.9M: 0.033 ms, one key per thread 0.099).
template <int PER>
__global__ void k_key_starts(const uint32_t* __restrict__ rank, const uint32_t* counts, const uint32_t* __restrict__ starts,
                             int64_t keys, int sh, uint32_t* __restrict__ key_starts, uint32_t* __restrict__ cell_starts,
                             uint32_t* cell_sizes) {
    const int64_t k = PER * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= keys) return;
    const int64_t c = k >> (3 * sh);
    const uint32_t s = (uint32_t)k & ((1u << (3 * sh)) - 1u), n = counts[c];
    const uint32_t* from = starts + ((size_t)rank[c] << (3 * sh));
    if (PER == 4) {
        const uint4 v = n ? *reinterpret_cast<const uint4*>(from + s) : make_uint4(from[0], from[0], from[0], from[0]);
        *reinterpret_cast<uint4*>(key_starts + k) = v;
    } else {
        key_starts[k] = from[0];
    }
    if (s == 0u) {
        cell_starts[c] = from[0];
        if (cell_sizes != counts) cell_sizes[c] = n;
    }
    if (k + PER == keys) key_starts[keys] = from[n ? 1u << (3 * sh) : 0u];   // the total
}

__device__ __forceinline__ int find_range(const int64_t* __restrict__ off, int n, int64_t v) {
    int lo = 0, hi = n - 1;   // last i with off[i] <= v
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= v) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Several instances in one key space: photon p of instance i's region (the
// first min(cap, filled) of its slots are photons) gets key key0 + its
// sub-cell key in the instance's grid; other slots get `sentinel`.
__global__ void k_key_count_multi(const float* __restrict__ pos, int64_t n, const GridInstDev* __restrict__ tab,
                                  const int64_t* __restrict__ ph_off, int ninst, const int64_t* __restrict__ filled,
                                  uint32_t sentinel, uint32_t* __restrict__ key, uint32_t* __restrict__ counts) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int i = find_range(ph_off, ninst, p);
    const GridInstDev t = tab[i];
    const int64_t local = p - t.ph0;
    uint32_t k = sentinel;
    if (local < min(t.cap, filled[i])) {
        GridGeom g;
        g.mnx = t.mn[0]; g.mny = t.mn[1]; g.mnz = t.mn[2];
        g.gx = t.gx; g.gy = t.gy; g.gz = t.gz; g.cell = t.cell;
        g.inv = 1.0f / t.cell;
        const int sh = __ffs(t.S) - 1;
        uint32_t cell;
        const uint32_t s = sub_cell_of(g, sh, pos + 3 * p, cell);
        k = (uint32_t)t.key0 + (cell << (3 * sh)) + s;
    }
    key[p] = k;
    atomicAdd(counts + k, 1u);
}

// per global cell: the instance-relative start and size of its photons
__global__ void k_cells_multi(int64_t cells, const GridInstDev* __restrict__ tab, const int64_t* __restrict__ cell_off,
                              int ninst, const uint32_t* __restrict__ key_starts, uint32_t* __restrict__ starts,
                              uint32_t* __restrict__ sizes) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const int i = find_range(cell_off, ninst, c);
    const GridInstDev t = tab[i];
    const int64_t S3 = (int64_t)t.S * t.S * t.S;
    const int64_t lc = c - t.cell0;
    const uint32_t base = key_starts[t.key0];
    const uint32_t a = key_starts[t.key0 + lc * S3], b = key_starts[t.key0 + (lc + 1) * S3];
    starts[c] = a - base;
    sizes[c] = b - a;
}

// Digit histograms of all passes in one read of the keys: hist[p][digit].
__global__ void __launch_bounds__(RADIX_THREADS)
k_radix_hist(const uint32_t* __restrict__ keys, int64_t n, int width, int passes, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[RADIX_MAX_PASSES][RADIX_MAX_BINS];
    const int tid = threadIdx.x, bins = 1 << width;
    for (int i = tid; i < RADIX_MAX_PASSES * RADIX_MAX_BINS; i += RADIX_THREADS) (&h[0][0])[i] = 0u;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * RADIX_THREADS;
    for (int64_t i = (int64_t)blockIdx.x * RADIX_THREADS + tid; i < n; i += stride) {
        const uint32_t k = keys[i];
        for (int p = 0; p < passes; p++) atomicAdd(&h[p][(k >> (width * p)) & (uint32_t)(bins - 1)], 1u);
    }
    __syncthreads();
    for (int p = 0; p < passes; p++)
        for (int b = tid; b < bins; b += RADIX_THREADS)
            if (h[p][b]) atomicAdd(hist + p * RADIX_MAX_BINS + b, h[p][b]);
}

// exclusive scan over the block's RADIX_THREADS values
__device__ __forceinline__ uint32_t radix_block_scan(uint32_t v, uint32_t* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t off = incl - v;
    for (int w = 0; w < warp; w++) off += wsum[w];
    return off;
}

// One radix pass: a stable scatter by one digit.
//
// Few keys (one tile per block, all blocks resident): the tiles find their
// places themselves (one-sweep radix sort: Adinets & Merrill, "Onesweep", 2022,
// over the decoupled look-back of Merrill & Garland, 2016).  Tiles take dynamic
// ids; each publishes its count of every digit in one word (state, count), later
// the count of it and all tiles before, and one thread per digit adds the words of
// the tiles before its own up to the first of the second kind, four at a time.
// The words of pass p have states 2p + 1 and 2p + 2, so those of earlier passes
// read as not yet there and the array is cleared once per sort.  Every wait is
// bounded (ST_TIMEOUT; the tile then writes nothing).
// Many keys: each block scatters a run of consecutive tiles, whose digits' places
// k_radix_count and k_radix_offsets have found.
//
// Bound by the latency of the in-tile ranking (0.5 of the issue slots).  Against
// a histogram per tile, a scan over all (digit, tile) and a scatter of single
// tiles: a pass over 10M keys 0.17 -> 0.13 ms (grid build 1.00 -> 0.96), grid build
// of 100K photons 0.108 -> 0.096 ms, of 100M 14.8 -> 14.0.
//
// A warp owns 256 consecutive keys and walks
// them 32 at a time in order; equal digits inside a step are ranked by lane
// (the lanes of a digit found by one ballot per digit bit: grid build 1.14 ->
// 1.10 ms against __match_any_sync), across steps by a per-warp running
// count, across warps by a
// prefix over the warps' counts.  The tile is then staged in shared memory in
// digit order, so that consecutive threads write consecutive slots of each
// digit's output run (coalesced) instead of one scattered word per key.
// vals_in == null means vals = index.
struct RadixSmem {
    uint32_t wh[RADIX_WARPS][RADIX_MAX_BINS];   // per-warp digit counts, then warp offsets
    uint32_t dbase[RADIX_MAX_BINS];             // global start of the tile's run of each digit
    uint32_t lbase[RADIX_MAX_BINS];             // start of each digit inside the staged tile
    uint32_t wsum[RADIX_WARPS];
    int tile, failed;
    uint32_t key[RADIX_TILE];
    uint32_t val[RADIX_TILE];
};

// the look-back's words: a state in the top 4 bits, a count below
constexpr int WORD_SHIFT = 28;
static_assert((int64_t)RADIX_BLOCKS * RADIX_TILE < ((int64_t)1 << WORD_SHIFT), "a count fits");

// Digit counts of every block's run of keys, counts[block][digit].
__global__ void __launch_bounds__(RADIX_THREADS)
k_radix_count(const uint32_t* __restrict__ keys, int64_t n, int64_t run, int shift, int bins, uint32_t* __restrict__ counts) {
    __shared__ uint32_t h[RADIX_MAX_BINS];
    const int tid = threadIdx.x;
    for (int b = tid; b < bins; b += RADIX_THREADS) h[b] = 0u;
    __syncthreads();
    const int64_t first = (int64_t)blockIdx.x * run, last = min(first + run, n);
#pragma unroll 4
    for (int64_t i = first + tid; i < last; i += RADIX_THREADS) atomicAdd(&h[(keys[i] >> shift) & (uint32_t)(bins - 1)], 1u);
    __syncthreads();
    for (int b = tid; b < bins; b += RADIX_THREADS) counts[(int64_t)blockIdx.x * bins + b] = h[b];
}

// One block per digit: counts[.][digit] becomes its exclusive prefix over the
// blocks, totals[digit] its sum.
__global__ void __launch_bounds__(RADIX_THREADS)
k_radix_offsets(uint32_t* __restrict__ counts, int blocks, int bins, uint32_t* __restrict__ totals) {
    __shared__ uint32_t wsum[RADIX_WARPS];
    static_assert(RADIX_BLOCKS <= RADIX_THREADS, "one block of counts per thread");
    uint32_t* c = counts + (int64_t)threadIdx.x * bins + blockIdx.x;
    const bool in = (int)threadIdx.x < blocks;
    const uint32_t v = in ? *c : 0u;
    const uint32_t e = radix_block_scan(v, wsum);
    if (in) *c = e;
    if ((int)threadIdx.x == blocks - 1) totals[blockIdx.x] = e + v;
}

// RUNS: block i scatters the run of keys [i * run, ...) tile by tile, counts[i]
// its digits' prefixes over the blocks, hist the digits' totals.  Else one tile,
// whose digits' prefixes come from the look-back.
template <bool RUNS>
__global__ void __launch_bounds__(RADIX_THREADS, 3)   // 3 blocks per SM: the shared-memory limit
k_radix_pass(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, int64_t n, int64_t run, int width,
             int pass, const uint32_t* __restrict__ hist, uint32_t* __restrict__ words, unsigned* __restrict__ tile_counter,
             uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, unsigned* status) {
    extern __shared__ __align__(16) unsigned char radix_smem[];
    RadixSmem& R = *reinterpret_cast<RadixSmem*>(radix_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, bins = 1 << width, shift = width * pass, bits = width;
    const uint32_t dm = (uint32_t)bins - 1u;
    const unsigned part = 2u * pass + 1u, whole = part + 1u;
    const int b = tid;   // one thread per digit
    int tile = 0, tile_end = 1;
    uint32_t dnext = 0;  // RUNS: global start of the next tile's run of digit b
    if (RUNS) {
        tile = (int)(blockIdx.x * (run / RADIX_TILE));
        tile_end = (int)min((int64_t)tile + run / RADIX_TILE, (n + RADIX_TILE - 1) / RADIX_TILE);
        dnext = radix_block_scan(b < bins ? hist[b] : 0u, R.wsum);
        if (b < bins) dnext += words[(int64_t)blockIdx.x * bins + b];
        __syncthreads();
    } else {
        if (tid == 0) {
            R.tile = (int)atomicAdd(tile_counter, 1u);
            R.failed = 0;
        }
        __syncthreads();
        tile = R.tile;
        tile_end = tile + 1;
    }
    for (; tile < tile_end; tile++) {
        for (int i = tid; i < RADIX_WARPS * RADIX_MAX_BINS; i += RADIX_THREADS) (&R.wh[0][0])[i] = 0u;
        __syncthreads();
        const int64_t tbase = (int64_t)tile * RADIX_TILE;
        const int64_t wbase = tbase + (int64_t)warp * (32 * RADIX_ITEMS);
        const int tcount = (int)min((int64_t)RADIX_TILE, n - tbase);
        uint32_t k[RADIX_ITEMS], v[RADIX_ITEMS], r[RADIX_ITEMS];
#pragma unroll
        for (int j = 0; j < RADIX_ITEMS; j++) {
            int64_t gi = wbase + j * 32 + lane;
            bool valid = gi < n;
            unsigned vm = __ballot_sync(0xffffffffu, valid);
            k[j] = valid ? keys_in[gi] : 0u;
            v[j] = valid ? (vals_in ? vals_in[gi] : (uint32_t)gi) : 0u;
            r[j] = 0u;
            // lanes holding the same digit: one ballot per digit bit (independent
            // instructions, where a match has one long latency)
            const uint32_t d = (k[j] >> shift) & dm;
            unsigned peers = vm;
#pragma unroll
            for (int b = 0; b < RADIX_MAX_BITS; b++) {
                if (b < bits) {
                    const unsigned on = __ballot_sync(0xffffffffu, (d >> b) & 1u);
                    peers &= ((d >> b) & 1u) ? on : ~on;
                }
            }
            const int leader = valid ? __ffs(peers) - 1 : lane;
            uint32_t old = 0u;
            if (valid && lane == leader) {
                old = R.wh[warp][d];
                R.wh[warp][d] = old + (uint32_t)__popc(peers);
            }
            // (the whole warp: a shuffle per group of equal digits runs the groups one after another)
            old = __shfl_sync(0xffffffffu, old, leader);
            r[j] = old + (uint32_t)__popc(peers & lanemask_lt());
            __syncwarp();   // the next step's leader of a digit may be another lane: it reads this step's count
        }
        __syncthreads();
        // exclusive prefix of each digit over warps; the tile's count
        uint32_t total = 0;
        if (b < bins) {
#pragma unroll
            for (int w = 0; w < RADIX_WARPS; w++) {
                const uint32_t c = R.wh[w][b];
                R.wh[w][b] = total;
                total += c;
            }
        }
        if (RUNS) {
            if (b < bins) R.dbase[b] = dnext;
            dnext += total;
        } else if (tile == 0) {
            const uint32_t base = radix_block_scan(b < bins ? hist[b] : 0u, R.wsum);
            if (b < bins) {
                ((volatile uint32_t*)words)[b] = whole << WORD_SHIFT | (base + total);
                R.dbase[b] = base;
            }
            __syncthreads();
        } else if (b < bins) {
            ((volatile uint32_t*)words)[tile * bins + b] = part << WORD_SHIFT | total;
        }
        const uint32_t lb = radix_block_scan(total, R.wsum);
        if (b < bins) R.lbase[b] = lb;
        __syncthreads();
        // stage the tile in digit order
#pragma unroll
        for (int j = 0; j < RADIX_ITEMS; j++) {
            int64_t gi = wbase + j * 32 + lane;
            if (gi < n) {
                const uint32_t d = (k[j] >> shift) & dm;
                const uint32_t lp = R.lbase[d] + R.wh[warp][d] + r[j];
                R.key[lp] = k[j];
                R.val[lp] = v[j];
            }
        }
        if (!RUNS && tile != 0 && b < bins) {
            uint32_t sum = 0;   // keys of lower digits, and of b in the tiles before
            long long polls = 0;
            bool found = false;
            for (int t = tile - 1; !found;) {
                uint32_t w[4];
#pragma unroll
                for (int u = 0; u < 4; u++) w[u] = t - u >= 0 ? ((volatile uint32_t*)words)[(t - u) * bins + b] : 0u;
                int seen = 0;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned st = w[u] >> WORD_SHIFT;
                    if (found || seen != u || (st != part && st != whole)) continue;
                    sum += w[u] & ((1u << WORD_SHIFT) - 1u);
                    seen++;
                    found = st == whole;
                }
                t -= seen;
                if (seen == 0 && ++polls > SCAN_SPIN_LIMIT) {
                    raise_status(status, ST_TIMEOUT);
                    R.failed = 1;
                    break;
                }
            }
            ((volatile uint32_t*)words)[tile * bins + b] = whole << WORD_SHIFT | (sum + total);
            R.dbase[b] = sum;
        }
        __syncthreads();
        if (!RUNS && R.failed) return;
        // write out: slot i of the staged tile goes to dbase[d] + (i - lbase[d])
        for (int i = tid; i < tcount; i += RADIX_THREADS) {
            const uint32_t kk = R.key[i];
            const uint32_t d = (kk >> shift) & dm;
            const uint32_t p = R.dbase[d] + ((uint32_t)i - R.lbase[d]);
            if (keys_out) keys_out[p] = kk;
            vals_out[p] = R.val[i];
        }
        __syncthreads();
    }
}

// pw == nullptr: every photon has power pw0 (a traced map), so the power is
// written without a random read of the source list (gpow == nullptr: not
// written at all).  rec != nullptr: the
// photon's position and direction are read as one 32-byte record (one DRAM
// sector) instead of two 12-byte pieces of the position and direction arrays.
__global__ void k_grid_gather(const uint32_t* __restrict__ order, int64_t n, const float* __restrict__ pos,
                              const float* __restrict__ dir, const float4* __restrict__ rec,
                              const float* __restrict__ pw, float3 pw0, float4* __restrict__ gpos,
                              float* __restrict__ gdir, float* __restrict__ gpow, unsigned* status) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t s = order[j];
    if ((int64_t)s >= n) { raise_status(status, ST_BAD_INPUT); return; }
    float3 pp, dd;
    if (rec) {
        const float4 a = __ldg(rec + 2 * (int64_t)s), b = __ldg(rec + 2 * (int64_t)s + 1);
        pp = make_float3(a.x, a.y, a.z);
        dd = make_float3(b.x, b.y, b.z);
    } else {
        const float* p = pos + 3 * (int64_t)s;
        const float* d = dir + 3 * (int64_t)s;
        pp = make_float3(p[0], p[1], p[2]);
        dd = make_float3(d[0], d[1], d[2]);
    }
    gpos[j] = make_float4(pp.x, pp.y, pp.z, __uint_as_float(s));
    gdir[3 * j] = dd.x; gdir[3 * j + 1] = dd.y; gdir[3 * j + 2] = dd.z;
    if (!gpow) return;
    float3 w = pw0;
    if (pw) {
        const float* q = pw + 3 * (int64_t)s;
        w = make_float3(q[0], q[1], q[2]);
    }
    gpow[3 * j] = w.x; gpow[3 * j + 1] = w.y; gpow[3 * j + 2] = w.z;
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void grid_dims(const float aabb[6], int64_t n, int desired, int dims[3], float* cell) {
    float sx = std::fabs(aabb[3] - aabb[0]);
    float sy = std::fabs(aabb[4] - aabb[1]);
    float sz = std::fabs(aabb[5] - aabb[2]);
    int N = (int)((n + desired - 1) / desired);
    float volume = sx * sy * sz;
    float c = std::cbrt(volume / N);
    dims[0] = (int)std::ceil(sx / c);
    dims[1] = (int)std::ceil(sy / c);
    dims[2] = (int)std::ceil(sz / c);
    *cell = c;
}

void grid_scratch_sizes(int64_t n, int64_t max_keys, size_t* hist_elems, size_t* scan_ws_bytes) {
    *hist_elems = radix_hist_elems(n);
    *scan_ws_bytes = scan_workspace_bytes(max_keys + 1);
}

int grid_auto_subdiv(uint32_t max_count, int k_hint) {
    double per = (double)max_count / (2.0 * std::max(k_hint, 1));
    int S = 1;
    while (S < 8 && (double)(2 * S) * (2 * S) <= per) S *= 2;
    return S;
}

cudaError_t grid_count(GridBuffers& B, const float aabb[6], int desired, int regrid_mult, int regrid_div,
                       GridPlan* plan, cudaStream_t st) {
    cudaError_t e;
    const int64_t n = B.n;
    GridPlan pa{}, pb{};
    grid_dims(aabb, n, desired, pa.dims, &pa.cell);
    pa.cells = (int64_t)pa.dims[0] * pa.dims[1] * pa.dims[2];
    const int want_b = std::max(desired / regrid_div, 1);
    const bool two = want_b != desired;
    grid_dims(aabb, n, want_b, pb.dims, &pb.cell);
    pb.cells = (int64_t)pb.dims[0] * pb.dims[1] * pb.dims[2];
    auto geom = [&](const GridPlan& p) {
        GridGeom g;
        g.mnx = aabb[0]; g.mny = aabb[1]; g.mnz = aabb[2];
        g.gx = p.dims[0]; g.gy = p.dims[1]; g.gz = p.dims[2]; g.cell = p.cell;
        g.inv = 1.0f / p.cell;
        return g;
    };
    if ((e = cudaMemsetAsync(B.cell_sizes, 0, (size_t)pa.cells * 4, st)) != cudaSuccess) return e;
    if (two && (e = cudaMemsetAsync(B.counts2, 0, (size_t)pb.cells * 4, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(B.small, 0, 16, st)) != cudaSuccess) return e;
    int launches = 0;
    const int64_t smem_words = (pa.cells + 1) / 2 + (two ? (pb.cells + 1) / 2 : 0);
    if (n > 0 && smem_words <= COUNT_SMEM_WORDS) {
        const int smem = (int)smem_words * 4;
        if ((e = cudaFuncSetAttribute(k_count_cells_smem, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
            return e;
        // one block per SM at this shared-memory size: whole waves of equal chunks
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const int64_t least = blocks_for(n, COUNT_CHUNK);
        const int64_t nblk = (least + sms - 1) / sms * sms;
        const int64_t chunk = (n + nblk - 1) / nblk;
        k_count_cells_smem<<<(unsigned)blocks_for(n, (int)chunk), COUNT_THREADS, smem, st>>>(
            B.pos, n, chunk, geom(pa), geom(pb), two ? 1 : 0, (int)pa.cells, (int)pb.cells, B.cell_sizes, B.counts2);
    } else if (n > 0) {
        k_count_cells<<<blocks_for(n, 256), 256, 0, st>>>(B.pos, n, geom(pa), geom(pb), two ? 1 : 0, B.cell_sizes,
                                                            B.counts2);
    }
    if (n > 0) {
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        k_count_max<<<std::min<int64_t>(blocks_for(std::max(pa.cells, pb.cells), 256), 296), 256, 0, st>>>(
            B.cell_sizes, pa.cells, B.counts2, two ? pb.cells : 0, B.small);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        launches = 2;
    }
    uint32_t stack_mx[4] = {0u, 0u, 0u, 0u};
    uint32_t* mx = B.host_words ? B.host_words : stack_mx;
    if ((e = cudaMemcpyAsync(mx, B.small, 16, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    pa.max_count = mx[0];
    pb.max_count = two ? mx[1] : mx[0];
    pa.full_cells = mx[2];
    pb.full_cells = two ? mx[3] : mx[2];
    pa.counts = B.cell_sizes;
    pb.counts = two ? B.counts2 : B.cell_sizes;
    // the reference rebuilds at the finer resolution when a cell is overfull
    *plan = (mx[0] > (uint32_t)(regrid_mult * desired)) ? pb : pa;
    plan->launches = launches;
    return cudaSuccess;
}

cudaError_t grid_sort(GridBuffers& B, const float aabb[6], GridPlan& plan, int S, cudaStream_t st) {
    cudaError_t e;
    const int64_t n = B.n;
    const int64_t cells = plan.cells;
    const int sh = S == 8 ? 3 : S == 4 ? 2 : S == 2 ? 1 : 0;
    const int64_t keys = cells << (3 * sh);
    const int64_t full_keys = std::max<int64_t>(plan.full_cells, 1) << (3 * sh);   // keys of cells that hold photons
    GridGeom g;
    g.mnx = aabb[0]; g.mny = aabb[1]; g.mnz = aabb[2];
    g.gx = plan.dims[0]; g.gy = plan.dims[1]; g.gz = plan.dims[2]; g.cell = plan.cell;
    g.inv = 1.0f / plan.cell;
    if (cells <= RANK_CELLS) {
        k_cell_rank<<<1, RANK_THREADS, 0, st>>>(plan.counts, (int)cells, B.rank);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    } else {
        k_cell_flags<<<blocks_for(cells, 256), 256, 0, st>>>(plan.counts, cells, B.rank);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = scan_u32(B.rank, B.rank, cells, 0, nullptr, B.scan_ws, B.status, st)) != cudaSuccess) return e;
        plan.launches++;
    }
    if ((e = cudaMemsetAsync(B.key_counts, 0, (size_t)full_keys * 4, st)) != cudaSuccess) return e;
    if (n > 0) {
        k_key_count<<<blocks_for(n, 256), 256, 0, st>>>(B.pos, n, g, sh, B.rank, B.cid, B.key_counts);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        plan.launches++;
    }
    if ((e = scan_u32(B.key_counts, B.key_counts, full_keys, 0, B.key_counts + full_keys, B.scan_ws, B.status, st)) != cudaSuccess)
        return e;
    if (sh > 0)
        k_key_starts<4><<<blocks_for(keys / 4, 256), 256, 0, st>>>(B.rank, plan.counts, B.key_counts, keys, sh, B.key_starts,
                                                                  B.cell_starts, B.cell_sizes);
    else
        k_key_starts<1><<<blocks_for(keys, 256), 256, 0, st>>>(B.rank, plan.counts, B.key_counts, keys, sh, B.key_starts,
                                                              B.cell_starts, B.cell_sizes);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    plan.launches += 3;
    if (n == 0) return cudaSuccess;

    int launches = 0;
    e = radix_and_gather(B, n, full_keys, &launches, st);
    plan.launches += launches;
    return e;
}

// per-pass digit totals, tile counters, and a word per (block, digit)
size_t radix_hist_elems(int64_t n) {
    const int64_t tiles = std::min<int64_t>(std::max<int64_t>(1, (n + RADIX_TILE - 1) / RADIX_TILE), RADIX_BLOCKS);
    return RADIX_MAX_PASSES * RADIX_MAX_BINS + RADIX_MAX_PASSES + RADIX_MAX_BINS * (size_t)tiles;
}

// Stable LSD radix sort of n keys below 2^key_bits, digits of equal width <= 9 bits.
// Up to RADIX_BLOCKS tiles (1.8M keys) a pass is one launch, its tiles looking
// back over each other; beyond, three launches (counts, offsets, scatter): with
// more tiles than resident blocks each wave of them starts together and most of
// the look-back is waiting (10M keys: 0.23 ms a pass).
cudaError_t radix_sort_u32(const RadixBuffers& B, const uint32_t* keys_in, const uint32_t* vals_in, int64_t n,
                           int key_bits, bool want_keys, const uint32_t** keys_sorted, const uint32_t** vals_sorted,
                           int* launches, cudaStream_t st) {
    cudaError_t e;
    const int bits = std::min(std::max(key_bits, 1), 32);
    const int passes = (bits + RADIX_MAX_BITS - 1) / RADIX_MAX_BITS;
    const int width = (bits + passes - 1) / passes, bins = 1 << width;
    const int64_t tiles = (n + RADIX_TILE - 1) / RADIX_TILE;
    const bool runs = tiles > RADIX_BLOCKS;
    const int64_t run = (runs ? (tiles + RADIX_BLOCKS - 1) / RADIX_BLOCKS : 1) * RADIX_TILE;
    const int blocks = (int)((n + run - 1) / run);
    uint32_t* hist = B.hist;
    unsigned* counters = hist + RADIX_MAX_PASSES * RADIX_MAX_BINS;
    uint32_t* words = counters + RADIX_MAX_PASSES;
    auto kernel = runs ? k_radix_pass<true> : k_radix_pass<false>;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RadixSmem))) != cudaSuccess)
        return e;
    if (!runs) {
        const size_t clear = RADIX_MAX_PASSES * RADIX_MAX_BINS + RADIX_MAX_PASSES + (size_t)blocks * bins;
        if ((e = cudaMemsetAsync(hist, 0, clear * 4, st)) != cudaSuccess) return e;
        k_radix_hist<<<blocks, RADIX_THREADS, 0, st>>>(keys_in, n, width, passes, hist);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *launches += 1;
    }
    const uint32_t* kin = keys_in;
    const uint32_t* vin = vals_in;
    for (int p = 0; p < passes; p++) {
        const bool last = p == passes - 1;
        uint32_t* kout = (last && !want_keys) ? nullptr : B.keys[p & 1];
        uint32_t* vout = B.vals[p & 1];
        uint32_t* h = hist + p * RADIX_MAX_BINS;
        if (runs) {
            k_radix_count<<<blocks, RADIX_THREADS, 0, st>>>(kin, n, run, width * p, bins, words);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            k_radix_offsets<<<bins, RADIX_THREADS, 0, st>>>(words, blocks, bins, h);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            *launches += 2;
        }
        kernel<<<blocks, RADIX_THREADS, sizeof(RadixSmem), st>>>(kin, vin, n, run, width, p, h, words, counters + p, kout, vout,
                                                                 B.status);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *launches += 1;
        kin = kout;
        vin = vout;
    }
    if (keys_sorted) *keys_sorted = kin;
    if (vals_sorted) *vals_sorted = vin;
    return cudaSuccess;
}

// LSD radix sort of B.cid (keys < key_space, stable), carrying the photon
// index; then the sorted records.
cudaError_t radix_and_gather(GridBuffers& B, int64_t n, int64_t key_space, int* launches, cudaStream_t st) {
    int bits = 1;
    while (bits < 32 && ((uint64_t)1 << bits) < (uint64_t)key_space) bits++;
    RadixBuffers RB{{B.keys[0], B.keys[1]}, {B.vals[0], B.vals[1]}, B.hist, B.status};
    const uint32_t* order = nullptr;
    cudaError_t e = radix_sort_u32(RB, B.cid, nullptr, n, bits, false, nullptr, &order, launches, st);
    if (e != cudaSuccess) return e;
    k_grid_gather<<<blocks_for(n, 256), 256, 0, st>>>(
        order, n, B.pos, B.dir, B.rec, B.uniform_pow ? nullptr : B.pow,
        make_float3(B.pow_value[0], B.pow_value[1], B.pow_value[2]), B.gpos, B.gdir,
        B.uniform_pow && B.defer_pow ? nullptr : B.gpow, B.status);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t grid_multi(GridBuffers& B, const GridMulti& M, int* launches, cudaStream_t st) {
    cudaError_t e;
    const int64_t n = B.n;
    const int64_t key_space = M.total_keys + 1;           // + the sentinel of empty slots
    if ((e = cudaMemsetAsync(B.key_counts, 0, (size_t)key_space * 4, st)) != cudaSuccess) return e;
    if (n > 0) {
        k_key_count_multi<<<blocks_for(n, 256), 256, 0, st>>>(B.pos, n, M.tab, M.ph_off, M.ninst, M.filled,
                                                             (uint32_t)M.total_keys, B.cid, B.key_counts);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *launches += 1;
    }
    if ((e = scan_u32(B.key_counts, B.key_starts, key_space, 0, B.key_starts + key_space, B.scan_ws, B.status, st)) !=
        cudaSuccess)
        return e;
    k_cells_multi<<<blocks_for(M.total_cells, 256), 256, 0, st>>>(M.total_cells, M.tab, M.cell_off, M.ninst,
                                                                  B.key_starts, B.cell_starts, B.cell_sizes);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *launches += 2;
    if (n == 0) return cudaSuccess;
    return radix_and_gather(B, n, key_space, launches, st);
}

}  // namespace pm
