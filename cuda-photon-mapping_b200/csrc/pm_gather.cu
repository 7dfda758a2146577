// pm_gather.cu -- kNN photon gather + radiance estimate.
//
// Reference: CudaPhotonMapping/PhotonGrid.cu:222-284 (cube of cells of half
// width ceil(r / cell) around the query's cell, distance test <= r),
// PhotonMaxHeap.cuh:43-127 (bounded max-heap of k), Raytracer.cuh:110-138
// (Gaussian-filtered density estimate over the selected photons).
//
// Selection rule: the k photons with the smallest (distance, source id) pairs
// among those with distance <= r.  This is the reference heap's set whenever no
// two candidates tie at the k-th distance; on ties it is deterministic (the
// reference's heap keeps whichever the sift order leaves).  Distances are the
// reference's length(p - q) in IEEE float, so the sets are bit-exact.
//
// One warp per query.  Photons are stored by (cell, sub-cell); the warp scans
// the query's sub-cell and its 26 neighbours, then, with k candidates found,
// the rest of the sub-cells that the bound on the k-th distance reaches, within
// the reference's cube of cells.  With fewer than k it scans the sphere that
// should hold them, a larger one until it does or the radius is covered.  Runs of photons with
// consecutive slots are queued and scanned as one list, one photon per lane
// (one 16-byte load each); a photon whose squared distance is within the bound
// goes to a per-warp shared-memory store (squared distance, slot) by ballot and
// is counted in a 64-bin histogram of squared distance, from which the bound
// tightens.  Rounded roots order like the squared distances up to ties, so
// roots and source ids are looked at only where the k-th distance ties.
//
// The estimate sums the k photons in one order, whatever was scanned when: the
// 27 sub-cells around the query first, (z, y, x) order, then the others in
// (z, y, x) order if those 27 hold k photons within r, else by shells of equal
// Chebyshev distance (shell_index).
//
// What bounds it: instructions and the latency of the reads that each round of
// 32 photons waits for (from L1 / L2): 1,417 warp instructions a query at 0.56 of
// the issue slots for the 137K requests (k 64) of a 640 x 360 frame of 4M photons.
// Against a store of 64-bit (distance, id) keys with a root per candidate, sub-cells
// tested one by one and the set-up by the whole warp (2,233 at 0.70 there): 3.03 ->
// 1.91 ms for the 1.23M queries (k 64) of the 10M-photon 1080p frame; k 128 on 2M
// photons 2.12 -> 1.27 ms, k 200 on 30M photons 7.0 -> 5.4 ms, k 32 on 500K photons
// 2.03 -> 1.27 ms.
// Loops are not unrolled and the scan is there once: with three unrolled copies
// the kernel waited for its instructions (2.6 of 10 stall cycles per issue,
// 2.78 ms).  A dense caustic (60,000 photons in 27 sub-cells) makes single
// queries of 1 ms; a loop of its own for long runs made every other query 7 %
// slower.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>
#include "pm_gather.cuh"
#include "pm_device.cuh"
#include "pm_div.h"

namespace pm {

namespace {

constexpr int WARPS = 8;   // warps per block

constexpr int NB = 64;      // squared-distance histogram bins over [0, the first bound]
constexpr int QCAP = 96;    // queued photon runs per warp (one round appends at most 64 to fewer than 32)

template <int UCAP>
struct WarpStore {
    uint2 ent[UCAP];          // candidates in scan order: squared distance bits, sorted slot
    uint32_t dh[NB];          // histogram of the store's squared distances
    uint32_t qa[QCAP];        // queued runs of consecutive slots: first slot, length
    uint32_t qc[QCAP];
    uint32_t sel[32];
    int box[8];               // the box of rows being scanned: x0, x1, y0, rows along y, z0, runs per row; [7]: overflow's count
};

// A query as the set-up (one thread per query) leaves it for its warp.
struct Staged {
    float qx, qy, qz;
    float lim2;               // first bound on the squared distance: the density guess or r2
    int X0, Y0, Z0;           // its sub-cell
    int flags;                // Q_* | instance << 8
    float block2;             // squared distance to the nearest face of the 27 sub-cells with sub-cells behind it
    float bscale;             // NB / lim2
};
constexpr float BLOCK_MARGIN = 1.f + 2e-5f;   // of squared bounds over box distances: above their rounding
enum { Q_ACTIVE = 1, Q_GUESSED = 2, Q_WIDE = 4 };

// Shared memory of a block of NW warps: its queries and each warp's store.
template <int UCAP, int NW>
struct BlockSmem {
    WarpStore<UCAP> st[NW];
    Staged q[32 * NW];
    int next;                 // the block's next query
    unsigned long long first; // queue position of its first query (persistent kernels)
};

// Cell / sub-cell of a point: the quotient (p - min) / cell selects the cell
// (clamped, CudaPhotonMapping/PhotonGrid.cu:10-23); its fractional part the sub-cell.
__device__ __forceinline__ void locate(float p, float mn, float cell, int g, int S, int& c, int& s) {
    float u = (p - mn) / cell;
    c = min(max((int)u, 0), g - 1);
    float f = u - (float)c;
    s = min(max((int)(f * (float)S), 0), S - 1);
}

// distance from q to the slab [lo, hi] along one axis; an open side (photons
// clamped into a boundary cell from outside the grid) is at infinity
__device__ __forceinline__ float axis_gap(float q, float lo, float hi, bool open_lo, bool open_hi) {
    float a = open_lo ? 0.f : lo - q;
    float b = open_hi ? 0.f : q - hi;
    return fmax3(a, b, 0.f);
}

// Place of the sub-cell at offset (dx, dy, dz) in its shell at Chebyshev distance
// R: the two full z faces (y, x order), then the perimeter of each inner z layer.
__device__ __forceinline__ uint32_t shell_index(int dx, int dy, int dz, int R) {
    const int side = 2 * R + 1, e = side - 1, x = dx + R, y = dy + R;
    if (dz == -R) return (uint32_t)(y * side + x);
    if (dz == R) return (uint32_t)(side * side + y * side + x);
    int p;
    if (y == 0 && x < e) p = x;
    else if (x == e && y < e) p = e + y;
    else if (y == e && x > 0) p = 3 * e - x;
    else p = 4 * e - y;
    return (uint32_t)(2 * side * side + (dz + R - 1) * 4 * e + p);
}

// key of the sub-cell at global sub-cell coordinates (sh = log2 S)
__device__ __forceinline__ uint32_t sub_key(const GatherGrid& G, int X, int Y, int Z, int sh) {
    const int S = 1 << sh;
    const uint32_t cell = (uint32_t)((X >> sh) + (Y >> sh) * G.gx + (Z >> sh) * G.gx * G.gy);
    return (cell << (3 * sh)) + (uint32_t)((X & (S - 1)) + (((Y & (S - 1)) + ((Z & (S - 1)) << sh)) << sh));
}

__device__ __forceinline__ uint32_t lanemask_le() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_le;" : "=r"(m));
    return m;
}
__device__ __forceinline__ float rcp(float x) { return __fdividef(1.f, x); }   // estimates only
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// 1 << s, 0 for s >= 32 (PTX shl clamps the shift amount)
__device__ __forceinline__ uint32_t bit_or_zero(uint32_t s) {
    uint32_t r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(s));
    return r;
}

// ascending bitonic sort of keys[0, n) by one warp (the form whose comparisons
// all ascend, so that n need not be a power of two: what lies past the end
// would be larger than all)
__device__ __noinline__ void warp_sort_keys(unsigned long long* keys, int n, int lane) {
    __syncwarp();
#pragma unroll 1
    for (int size = 2; size < 2 * n; size <<= 1)
#pragma unroll 1
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const int flip = stride == size >> 1 ? size - 1 : stride;
#pragma unroll 1
            for (int e = lane; e < n; e += 32) {
                const int o = e ^ flip;
                if (o > e && o < n) {
                    const unsigned long long a = keys[e], b = keys[o];
                    if (a > b) { keys[e] = b; keys[o] = a; }
                }
            }
            __syncwarp();
        }
}

// the need-th smallest (1-based) of the lanes' first `got` values (others: any larger or equal value)
__device__ __forceinline__ uint32_t nth_of_lanes(uint32_t mine, int got, uint32_t need, int lane) {
    uint32_t below = 0, same = 0;
#pragma unroll 1
    for (int j = 0; j < got; j++) {
        const uint32_t o = __shfl_sync(0xffffffffu, mine, j);
        below += o < mine ? 1u : 0u;
        same += o == mine ? 1u : 0u;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, lane < got && below < need && need <= below + same);
    __syncwarp();
    return __shfl_sync(0xffffffffu, mine, __ffs(hit) - 1);
}

// (out of line: resolve_ties is called where registers are short)
__device__ __noinline__ uint32_t nth_tie(const uint32_t* sel, int ties, uint32_t need, int lane) {
    return nth_of_lanes(lane < ties ? sel[lane] : 0xffffffffu, ties, need, lane);
}

// Of w kept candidates more than k remain: some lie so close behind the
// k-th squared distance that their rounded distances may tie with its own.
// Order is (distance, source index): drop the largest.  Rare.
__device__ __noinline__ int resolve_ties(uint2* ent, uint32_t* sel, const float4* gpos, int w, int k, float sk, int lane) {
    const float dk = sqrtf(sk);
    int below = 0, ties = 0;
#pragma unroll 1
    for (int base = 0; base < w; base += 32) {
        const int i = base + lane;
        const float d = i < w ? sqrtf(__uint_as_float(ent[i].x)) : INFINITY;
        const unsigned m = __ballot_sync(0xffffffffu, i < w && d == dk);
        const int pos = ties + __popc(m & lanemask_lt());
        if (i < w && d == dk && pos < 32) sel[pos] = __float_as_uint(gpos[ent[i].y].w);
        below += __popc(__ballot_sync(0xffffffffu, d < dk));
        ties += __popc(m);
    }
    __syncwarp();
    const int need = k - below;   // ties that stay, smallest source index first
    uint32_t id_max = 0xffffffffu;
    if (ties > need && ties <= 32) {
        id_max = nth_tie(sel, ties, (uint32_t)need, lane);
    } else if (ties > need) {
        id_max = 0u;              // the need-th smallest index among the ties
#pragma unroll 1
        for (int bit = 31; bit >= 0; bit--) {
            const uint32_t t = id_max | 1u << bit;
            int c = 0;
#pragma unroll 1
            for (int base = 0; base < w; base += 32) {
                const int i = base + lane;
                const bool tie = i < w && sqrtf(__uint_as_float(ent[i].x)) == dk;
                c += __popc(__ballot_sync(0xffffffffu, tie && __float_as_uint(gpos[ent[i].y].w) < t));
            }
            if (c < need) id_max = t;
        }
    }
    int out = 0;
#pragma unroll 1
    for (int base = 0; base < w; base += 32) {
        const int i = base + lane;
        const uint2 e = i < w ? ent[i] : make_uint2(0u, 0u);
        const float d = sqrtf(__uint_as_float(e.x));
        const bool keep = i < w && (d < dk || (d == dk && __float_as_uint(gpos[e.y].w) <= id_max));
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        __syncwarp();
        if (keep) ent[out + __popc(m & lanemask_lt())] = e;
        out += __popc(m);
        __syncwarp();
    }
    return out;
}

// bin | before << 8 | count << 20 of the histogram bin that holds the k-th
// smallest squared distance (before: candidates in lower bins)
__device__ __forceinline__ uint32_t find_bin(const uint32_t* dh, int k, int lane) {
    const uint2 c = reinterpret_cast<const uint2*>(dh)[lane];
    const uint32_t sum = c.x + c.y;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t excl = incl - sum;
    const bool second = excl + c.x < (uint32_t)k;
    const uint32_t pack = (uint32_t)(2 * lane + (second ? 1 : 0)) | (second ? excl + c.x : excl) << 8 |
                          (second ? c.y : c.x) << 20;
    const unsigned own = __ballot_sync(0xffffffffu, excl < (uint32_t)k && (uint32_t)k <= incl);
    return __shfl_sync(0xffffffffu, pack, own ? __ffs(own) - 1 : 0);
}

// The keys (bits of squared distances) of the store in [lo, hi], at most 32, to sel;
// returns the need-th smallest of them.
template <int UCAP>
__device__ __forceinline__ uint32_t pick_s(WarpStore<UCAP>& U, int n, uint32_t lo, uint32_t hi, uint32_t need, int lane) {
    int got = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
        const int i = base + lane;
        const uint32_t sb = i < n ? U.ent[i].x : 0u;
        const bool m = i < n && sb >= lo && sb <= hi;
        const unsigned bm = __ballot_sync(0xffffffffu, m);
        if (m) U.sel[got + __popc(bm & lanemask_lt())] = sb;
        got += __popc(bm);
    }
    __syncwarp();
    return nth_of_lanes(lane < got ? U.sel[lane] : 0xffffffffu, got, need, lane);
}

// The need-th smallest key of the store's histogram bin `bin`, which holds more than
// 32 (a histogram over [0, r^2] in a dense place): the bin's range of keys is cut
// into 64 bins of its own, in dh, until at most 32 share one.  Bit by bit over
// the whole store it took up to 31 passes instead of about three: frame with a
// caustic map 4.49 -> 4.29 ms, 2,027 queries at k 200 among clusters 1.99 -> 1.43.
template <int UCAP>
__device__ __noinline__ float kth_of_full_bin(WarpStore<UCAP>& U, int n, uint32_t need, uint32_t bin, float bscale,
                                              int lane) {
    uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
        const uint32_t sb = U.ent[i].x;
        if (min((uint32_t)(__uint_as_float(sb) * bscale), (uint32_t)(NB - 1)) == bin) { lo = min(lo, sb); hi = max(hi, sb); }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
#pragma unroll 1
    while (lo != hi) {
        const int shift = max(26 - __clz(hi - lo), 0);
        __syncwarp();
        reinterpret_cast<uint2*>(U.dh)[lane] = make_uint2(0u, 0u);
        __syncwarp();
#pragma unroll 1
        for (int i = lane; i < n; i += 32) {
            const uint32_t sb = U.ent[i].x;
            if (sb >= lo && sb <= hi) atomicAdd(&U.dh[(sb - lo) >> shift], 1u);
        }
        __syncwarp();
        const uint32_t f = find_bin(U.dh, (int)need, lane);
        lo += (f & 255u) << shift;
        hi = min(hi, lo + (1u << shift) - 1u);
        need -= f >> 8 & 4095u;
        if (f >> 20 <= 32u) return __uint_as_float(pick_s<UCAP>(U, n, lo, hi, need, lane));
    }
    return __uint_as_float(lo);
}

// The k-th smallest squared distance of the store (n > k; found: find_bin's answer
// for it): the keys of the bin that holds it are ranked against each other.
template <int UCAP>
__device__ __forceinline__ float kth_s(WarpStore<UCAP>& U, int n, int k, uint32_t found, float bscale, int lane) {
    const uint32_t bin = found & 255u, before = found >> 8 & 4095u, cnt = found >> 20;
    const uint32_t need = (uint32_t)k - before;   // 1-based rank inside the bin
    if (cnt > 32u) return kth_of_full_bin<UCAP>(U, n, need, bin, bscale, lane);
    int got = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
        const int i = base + lane;
        const uint32_t sb = i < n ? U.ent[i].x : 0x7f800000u;
        const bool m = i < n && min((uint32_t)(__uint_as_float(sb) * bscale), (uint32_t)(NB - 1)) == bin;
        const unsigned bm = __ballot_sync(0xffffffffu, m);
        if (m) U.sel[got + __popc(bm & lanemask_lt())] = sb;
        got += __popc(bm);
    }
    __syncwarp();
    return __uint_as_float(nth_of_lanes(lane < got ? U.sel[lane] : 0xffffffffu, got, need, lane));
}

// Keep the k best of the store's n > k candidates, in their order, and with them
// (ties: up to this many) those that tie with the k-th; returns the k-th squared
// distance and in n what is kept.
template <int UCAP>
__device__ __forceinline__ float cut_store(WarpStore<UCAP>& U, const float4* gpos, int& n, int k, uint32_t found,
                                            float bscale, int ties, int lane) {
    const float sk = kth_s<UCAP>(U, n, k, found, bscale, lane);
    // beyond the k-th by less than the rounding of a root: kept for resolve_ties
    const float hi = sk * (1.f + 5e-7f);
    int w = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
        const int i = base + lane;
        const uint2 e = i < n ? U.ent[i] : make_uint2(0u, 0u);
        const bool keep = i < n && __uint_as_float(e.x) <= hi;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        __syncwarp();
        if (keep) U.ent[w + __popc(m & lanemask_lt())] = e;
        w += __popc(m);
    }
    __syncwarp();
    n = w;
    if (w > k + ties) n = resolve_ties(U.ent, U.sel, gpos, w, k, sk, lane);
    return sk;
}

// The store is full (n > k): keep its k best, and ties with the k-th that leave a
// third of the rest free, count them again; returns their bound, and in box[7] how
// many they are.
template <int UCAP>
__device__ __noinline__ float overflow(WarpStore<UCAP>& U, const float4* gpos, int n, int k, float bscale, int lane) {
    __syncwarp();
    const uint32_t found = find_bin(U.dh, k, lane);
    const float d = sqrtf(cut_store<UCAP>(U, gpos, n, k, found, bscale, (UCAP - 32 - k) * 2 / 3, lane));
    reinterpret_cast<uint2*>(U.dh)[lane] = make_uint2(0u, 0u);
    if (lane == 0) U.box[7] = n;
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < n; i += 32)
        atomicAdd(&U.dh[min((uint32_t)(__uint_as_float(U.ent[i].x) * bscale), (uint32_t)(NB - 1))], 1u);
    __syncwarp();
    return d * d * 1.000001f;
}

// A first bound on squared distances, x raised by at most a thousandth so that it
// is the largest square with its rounded root: distances are compared as
// rounded roots, and of photons that share one either all are within the bound
// or none.  The root d has 12 bits, so d * d is exact, and the squares beyond it
// that round to d end before d * d + d ulp(d): at the next float where d's
// mantissa is below sqrt(2) (an even exponent of d * d), at d * d itself elsewhere.
__device__ __forceinline__ float tie_bound(float x) {
    const float d = __uint_as_float((__float_as_uint(sqrt_approx(x)) + 0xfffu) & ~0xfffu);
    const uint32_t s = __float_as_uint(d * d);
    return __uint_as_float(s + (s >> 23 & 1u));   // (beyond the largest float: NaN, which fminf drops)
}

// the cells of the reference's cube around cell (cx, cy, cz)
struct Cube {
    int x0, y0, z0, x1, y1, z1;
};
__device__ __forceinline__ Cube cube_of(const GatherGrid& G, const GatherReach& E, int cx, int cy, int cz) {
    return Cube{max(0, cx - E.rc), max(0, cy - E.rc), max(0, cz - E.rc), min(G.gx - 1, cx + E.rc),
                min(G.gy - 1, cy + E.rc), min(G.gz - 1, cz + E.rc)};
}

// The set-up of one query: by one thread (by the query's own warp it took a fifth
// of the query's instructions), or, WARP, by all lanes of a warp where a block
// has no more queries than warps and only the latency counts (one thread's nine
// dependent rows take 9,500 cycles, more than the rest of a query that finds few
// photons).
//
// Density guess of the bound on the k-th distance: the N photons of the 27
// sub-cells around the query, spread over a plane through them (area 9 sc^2),
// give about G.guess x k photons within g = 3 sc sqrt(G.guess k / (pi N)).
// The guess filters which candidates enter the store, and a sub-cell whose
// padded box lies farther than g is not scanned at all; when fewer than k
// photons lie within g, the query starts again with larger bounds, up to r, so the
// answer is unchanged.
template <bool WARP = false>
__device__ __forceinline__ void stage_query(const GatherGrid& G, const GatherReach& E, Staged& s, V3 q, int k,
                                            int flags) {
    int cx, cy, cz, sx, sy, sz;
    locate(q.x, G.mn[0], G.cell, G.gx, G.S, cx, sx);
    locate(q.y, G.mn[1], G.cell, G.gy, G.S, cy, sy);
    locate(q.z, G.mn[2], G.cell, G.gz, G.S, cz, sz);
    const int S = G.S, sh = E.sh;
    const float sc = E.sc, r2 = E.r2;
    const Cube C = cube_of(G, E, cx, cy, cz);
    const int X0 = (cx << sh) + sx, Y0 = (cy << sh) + sy, Z0 = (cz << sh) + sz;
    const int lx = C.x0 << sh, ly = C.y0 << sh, lz = C.z0 << sh;
    const int hx = (C.x1 << sh) + S - 1, hy = (C.y1 << sh) + S - 1, hz = (C.z1 << sh) + S - 1;
    uint32_t N = 0u;
    const int xl = max(X0 - 1, lx), xr = min(X0 + 1, hx);
    const bool cut = S > 1 && (xl >> sh) != (xr >> sh);   // the row crosses into the next cell
    auto row = [&](int dy, int dz) -> uint32_t {   // photons of three sub-cells along x
        const int Y = Y0 + dy, Z = Z0 + dz;
        if (xl > xr || Y < ly || Y > hy || Z < lz || Z > hz) return 0u;
        if (!cut) return __ldg(G.key_starts + sub_key(G, xr, Y, Z, sh) + 1) - __ldg(G.key_starts + sub_key(G, xl, Y, Z, sh));
        const int xm = (xr >> sh) << sh;
        return __ldg(G.key_starts + sub_key(G, xm - 1, Y, Z, sh) + 1) - __ldg(G.key_starts + sub_key(G, xl, Y, Z, sh)) +
               __ldg(G.key_starts + sub_key(G, xr, Y, Z, sh) + 1) - __ldg(G.key_starts + sub_key(G, xm, Y, Z, sh));
    };
    if (WARP) {
        const int lane = threadIdx.x & 31;
        N = __reduce_add_sync(0xffffffffu, lane < 9 ? row(lane % 3 - 1, lane / 3 - 1) : 0u);
        if (lane != 0) return;
    } else {
#pragma unroll 1
        for (int dz = -1; dz <= 1; dz++)
#pragma unroll
            for (int dy = -1; dy <= 1; dy++) N += row(dy, dz);
    }
    auto face = [&](float p, float mn, int X, int lo, int hi) {
        const float a = X - 1 > lo ? p - (mn + (X - 1) * sc) : INFINITY, b = X + 1 < hi ? mn + (X + 2) * sc - p : INFINITY;
        return fminf(a, b);
    };
    const float f = fminf(fminf(face(q.x, G.mn[0], X0, lx, hx), face(q.y, G.mn[1], Y0, ly, hy)),
                          face(q.z, G.mn[2], Z0, lz, hz)) - E.pad;
    const float block2 = f > 0.f ? f * f : 0.f;
    s.block2 = block2;
    // A query outside the grid (its sub-cell is then the nearest one): spheres are
    // taken that much larger, and the guess says nothing.
    auto beyond = [&](float p, float mn, int g) { return fmax3(mn - p, p - (mn + (float)g * G.cell), 0.f); };
    const float ox = beyond(q.x, G.mn[0], G.gx), oy = beyond(q.y, G.mn[1], G.gy), oz = beyond(q.z, G.mn[2], G.gz);
    const float out2 = ox * ox + oy * oy + oz * oz;
    const bool outside = out2 > 0.25f * sc * sc;
    auto bound = [&](float x) {
        const float t = sqrt_approx(out2) + sqrt_approx(x);
        return fminf(r2, tie_bound(outside ? t * t : x));
    };
    s.lim2 = N >= (uint32_t)k ? bound(outside ? 27.f * sc * sc : E.ring2) : r2;
    if (G.guess > 0.f && N > (uint32_t)k && !outside) {   // else too few photons in the block to gain anything
        const float g2 = tie_bound(9.f * sc * sc * (G.guess * (float)k) / (3.14159265f * (float)N));
        if (g2 < r2) {
            s.lim2 = g2;
            flags |= Q_GUESSED;
        }
    } else if (N < (uint32_t)k && !(r2 * BLOCK_MARGIN < block2)) {
        // fewer than k in the block and more of r's sphere beyond it: the
        // sphere of the guess, of at most eight sub-cells (a larger one that reaches
        // a dense place meets its photons far side first, and the store overflows
        // dozens of times), at once that of r where it hardly leaves the
        // block.  Where none of r's sphere lies beyond, the 27 sub-cells in the
        // walk's own order, bound r, answer the query: as a growing sphere, its
        // answer ordered afterwards, 61,779 requests of the small room (k 100)
        // took 0.174 ms instead of 0.143.
        const float per = G.guess > 0.f ? G.guess : GATHER_GUESS;
        if (r2 > 4.f * sc * sc)
            s.lim2 = bound(fminf(9.f * sc * sc * (per * (float)k) / (3.14159265f * (float)N), 64.f * sc * sc));
        flags |= Q_WIDE;
    }
    s.qx = q.x; s.qy = q.y; s.qz = q.z;
    s.X0 = X0; s.Y0 = Y0; s.Z0 = Z0;
    s.flags = flags;
    s.bscale = (float)NB / s.lim2;
}

// The bound with which a walk goes on that found n < k photons within lim2 (below r2).
// A sphere (wide): a larger one, from the grid's diagonal on r's at once.  The 27
// sub-cells: once a larger bound, unless so few were found that the count says
// nothing here, then all of theirs, then all within r.  (r at once: every photon of
// the 27 goes through the store, and the histogram over [0, r2] bounds nothing where r
// spans many sub-cells.  1,021 queries at k 16 62 -> 51 us, 100,003 at k 200
// 1.77 -> 1.60 ms; at a radius of 100 boxes 2.2 ms for 20,000, now 0.2.  Larger ones
// until one holds: each scans a dense sub-cell again, 273 queries at k 8 0.6 -> 1.2 ms.)
// Out of line, as the other rare parts are: the walk then takes fewer registers
// and instruction lines (30M photons, k 200: 5.57 -> 5.41 ms).
__device__ __noinline__ float next_bound(float lim2, int n, int k, bool wide, bool once, float r2, float ring2, float far2) {
    const float per = __fdividef(1.f, (float)max(n, 1));
    float x;
    if (wide) x = lim2 >= far2 ? r2 : lim2 * fminf(4.f, fmaxf(2.f, 1.5f * GATHER_GUESS * (float)k * per));
    else if (lim2 >= 0.99f * ring2) x = r2;
    else if (once || 4 * n + 4 < k) x = ring2;
    else x = fminf(ring2, lim2 * (GATHER_GUESS * (float)k + 4.f) * per);
    return x < r2 ? fminf(r2, tie_bound(x)) : r2;
}

// Sub-cells [range_low, range_high] along an axis hold every photon within
// reach of f (both in sub-cell units), clamped to [lo, hi].  Taken wide: a
// sub-cell too many costs time only, its photons fail the distance test.
__device__ __forceinline__ int range_low(float f, float reach, int lo, int hi) {
    return (int)fminf(fmaxf(floorf(f - reach - fabsf(f) * 1e-6f), (float)lo), (float)hi);
}
__device__ __forceinline__ int range_high(float f, float reach, int lo, int hi) {
    return (int)fminf(fmaxf(floorf(f + reach + fabsf(f) * 1e-6f), (float)lo), (float)hi);
}

// Ascending sort of keys[0, n), n <= 32 NR, one warp, NR keys per lane in
// registers (bitonic).
template <int NR>
__device__ __noinline__ void sort_u32(uint32_t* keys, int n, int lane) {
    uint32_t v[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) v[r] = 32 * r + lane < n ? keys[32 * r + lane] : 0xffffffffu;
#pragma unroll
    for (int size = 2; size <= 32 * NR; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride >= 32; stride >>= 1)
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const int o = r ^ (stride >> 5);
                if (o > r) {
                    const uint32_t lo = min(v[r], v[o]), hi = max(v[r], v[o]);
                    const bool up = ((32 * r) & size) == 0;
                    v[r] = up ? lo : hi;
                    v[o] = up ? hi : lo;
                }
            }
#pragma unroll 1
        for (int stride = min(size >> 1, 16); stride > 0; stride >>= 1)
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], stride);
                const bool up = ((32 * r + lane) & size) == 0, lower = (lane & stride) == 0;
                v[r] = up == lower ? min(v[r], o) : max(v[r], o);
            }
    }
#pragma unroll
    for (int r = 0; r < NR; r++)
        if (32 * r + lane < n) keys[32 * r + lane] = v[r];
    __syncwarp();
}

// The store's cnt candidates, found block by block, into the shells' order: to
// the store's upper half, by keys (sub-cell's place in the walk of shells, scan
// order; cnt <= k <= UCAP / 2; inside a sub-cell the scan order is the slots').
template <int UCAP>
__device__ __forceinline__ void shells_order(const GatherGrid& G, const GatherReach& E, WarpStore<UCAP>& U, const Staged& s,
                                          int cnt, int lane) {
    __syncwarp();
    uint2* out = U.ent + UCAP / 2;
    unsigned long long* key = reinterpret_cast<unsigned long long*>(out);
    uint32_t* key32 = reinterpret_cast<uint32_t*>(out);
    // pass 0: 24-bit places (shells up to 127); pass 1, when one does not fit: 64-bit keys
    int wide = 0;
#pragma unroll 1
    for (; wide < 2; wide++) {
        bool fits = true;
#pragma unroll 1
        for (int e = lane; e < cnt; e += 32) {
            const float4 p = __ldg(G.gpos + U.ent[e].y);
            int cx, cy, cz, ux, uy, uz;
            locate(p.x, G.mn[0], G.cell, G.gx, G.S, cx, ux);
            locate(p.y, G.mn[1], G.cell, G.gy, G.S, cy, uy);
            locate(p.z, G.mn[2], G.cell, G.gz, G.S, cz, uz);
            const int dx = (cx << E.sh) + ux - s.X0, dy = (cy << E.sh) + uy - s.Y0, dz = (cz << E.sh) + uz - s.Z0;
            const int R = max(max(abs(dx), abs(dy)), abs(dz));
            const uint32_t t = R <= 1 ? (uint32_t)(9 * (dz + 1) + 3 * (dy + 1) + dx + 1) : shell_index(dx, dy, dz, R);
            if (wide) {
                key[e] = ((unsigned long long)(R <= 1 ? 0 : R) << 32 | t) << 10 | (unsigned long long)e;
            } else {
                const uint32_t inside = R <= 1 ? 0u : (uint32_t)((2 * R - 1) * (2 * R - 1) * (2 * R - 1));
                key32[e] = (inside + t) << 8 | (uint32_t)e;
                fits = fits && R <= 127;
            }
        }
        __syncwarp();
        if (wide) {
            warp_sort_keys(key, cnt, lane);
        } else if (__all_sync(0xffffffffu, fits)) {
            if (cnt <= 32) {   // one key per lane: its rank by comparing it with the others
                const uint32_t v = lane < cnt ? key32[lane] : 0u;
                const uint2 x = U.ent[lane];
                int rank = 0;
#pragma unroll 1
                for (int e = 0; e < cnt; e++) rank += (int)(__shfl_sync(0xffffffffu, v, e) < v);
                __syncwarp();
                if (lane < cnt) out[rank] = x;
                __syncwarp();
                return;
            }
            if (cnt <= 64) sort_u32<2>(key32, cnt, lane);
            else if (cnt <= 128) sort_u32<4>(key32, cnt, lane);
            else sort_u32<8>(key32, cnt, lane);
            break;
        }
    }
    uint2 v[8];   // cnt <= 256
#pragma unroll
    for (int r = 0; r < 8; r++)
        if (32 * r + lane < cnt)
            v[r] = U.ent[wide ? (int)(key[32 * r + lane] & 1023ull) : (int)(key32[32 * r + lane] & 255u)];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 8; r++)
        if (32 * r + lane < cnt) out[32 * r + lane] = v[r];
    __syncwarp();
}

// The ids of the answer's entries (cnt <= k <= UCAP / 2, in one half of the store)
// by ascending (distance, id).  The entries are put into NB bins of equal width
// over [0, rk] in the other half (the bin of a distance grows with it, and equal
// distances share one); an entry's place is its bin's first one plus the entries
// of its bin that come before it.  A bitonic sort of the 64-bit keys in shared
// memory took 36 passes at k 200 (photons set, grid, 100,003 queries with ids
// at k 200: 2.15 ms, now 1.77).
template <int UCAP>
__device__ __noinline__ void write_ids(WarpStore<UCAP>& U, const float4* gpos, const uint2* ent, int cnt, int k, float rk,
                                       uint32_t* ids, int lane) {
    unsigned long long* key = reinterpret_cast<unsigned long long*>(U.ent);
    unsigned long long* out = key;
    (ent == U.ent ? out : key) += UCAP / 2;
    const float scale = (float)NB / rk;   // (rk 0: all in bin 0 or NB - 1 alike)
    auto bin = [&](unsigned long long x) {
        return min((int)(__uint_as_float((uint32_t)(x >> 32)) * scale), NB - 1);
    };
    __syncwarp();
    reinterpret_cast<uint2*>(U.dh)[lane] = make_uint2(0u, 0u);
    __syncwarp();
#pragma unroll 1
    for (int e = lane; e < cnt; e += 32) {
        const uint2 x = ent[e];
        const unsigned long long v = (unsigned long long)__float_as_uint(sqrtf(__uint_as_float(x.x))) << 32 |
                                     __float_as_uint(__ldg(&gpos[x.y].w));
        key[e] = v;
        atomicAdd(&U.dh[bin(v)], 1u);
    }
    __syncwarp();
    const uint2 c = reinterpret_cast<uint2*>(U.dh)[lane];
    uint32_t incl = c.x + c.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    reinterpret_cast<uint2*>(U.dh)[lane] = make_uint2(incl - c.x - c.y, incl - c.y);
    __syncwarp();
#pragma unroll 1
    for (int e = lane; e < cnt; e += 32) {
        const unsigned long long v = key[e];
        out[atomicAdd(&U.dh[bin(v)], 1u)] = v;   // dh: from a bin's first place to the next bin's
    }
    __syncwarp();
#pragma unroll 1
    for (int e = lane; e < k; e += 32) {
        if (e >= cnt) {
            ids[e] = 0xffffffffu;
            continue;
        }
        const unsigned long long v = out[e];
        const int b = bin(v);
        const int lo = b > 0 ? (int)U.dh[b - 1] : 0, hi = (int)U.dh[b];
        int place = lo;
#pragma unroll 1
        for (int q = lo; q < hi; q++) place += (int)(out[q] < v);
        ids[place] = (uint32_t)v;
    }
    __syncwarp();
}

// What a warp scans: the query's sub-cell and its 26 neighbours; the rest of a
// bound's sphere; or (too few in the 27) a whole sphere that grows until it holds
// k or reaches r, by its sub-cells or, from 4 sub-cells on, by its cells unless
// those hold more than COARSE_MAX photons.
enum { M_RING = 0, M_REST = 1, M_WIDE = 2 };
constexpr uint32_t COARSE_MAX = 1536;

// one staged query (one warp): the k nearest photons within r and the estimate
// (UNI: G.pow_uniform is honoured; the batch kernel reads the power array
// instead.  Its G and E are its instance's in global memory, read where they are
// used: copied to registers per query, the 16-instance gather took 16.3 ms
// instead of 13.7.  inv_norm: 1 / (1 - exp(-1.953)))
template <int UCAP, bool UNI = true>
__device__ __forceinline__ void gather_query(const GatherGrid& G, const GatherReach& E, WarpStore<UCAP>& U,
                                             const Staged& s, int64_t i, const float* __restrict__ pnrm, int k,
                                             int require_full, const GatherOut& O, float inv_norm, int lane) {
    int n = 0;                 // candidates in the store
    int qn = 0;                // queued runs
    float lim2 = s.lim2;       // a candidate enters when its squared distance <= lim2 (<= E.r2)
    float bscale = s.bscale;   // histogram bin of d2 = min(NB - 1, (int)(d2 * bscale))
    uint32_t found = 0u;       // find_bin's answer for a store of `fn`
    int fn = -1;               // (-1: none; -2: none, and a larger bound was tried in the 27)
    int mode = s.flags & Q_WIDE ? M_WIDE : M_RING, base = 0, total = 27;
    bool coarse = false;       // M_WIDE: rows of cells, not of sub-cells
    bool plan = mode == M_WIDE;   // the box of rows is still to be set
    const float m2 = BLOCK_MARGIN;
    reinterpret_cast<uint2*>(U.dh)[lane] = make_uint2(0u, 0u);
    __syncwarp();
    coarse = plan && lim2 > 16.f * E.sc * E.sc && E.sh > 0;
#pragma unroll 1
    while (true) {
        const int sh = coarse ? 0 : E.sh;               // log2 of the units per cell
        const float unit = coarse ? G.cell : E.sc;
        if (plan) {
            // The box, in units, that the sphere of squared radius lim2 can
            // reach inside the cube.  One lane per (row of units along x, cell the
            // row crosses): the sub-cells of a row inside one cell have
            // consecutive keys, so their photons are one run of slots (two where
            // the 27 sub-cells cut the row), and so have all cells of a row.
            plan = false;
            const float inv = coarse ? 1.f / G.cell : E.inv_sc;
            const int X0 = s.X0 >> (E.sh - sh), Y0 = s.Y0 >> (E.sh - sh), Z0 = s.Z0 >> (E.sh - sh);
            const Cube C = cube_of(G, E, X0 >> sh, Y0 >> sh, Z0 >> sh);
            const float reach = (sqrt_approx(lim2 * m2) * (1.f + 1e-5f) + E.pad) * inv + 0.01f;
            const float fx = (s.qx - G.mn[0]) * inv, fy = (s.qy - G.mn[1]) * inv, fz = (s.qz - G.mn[2]) * inv;
            const int x0 = range_low(fx, reach, C.x0 << sh, X0), x1 = range_high(fx, reach, X0, ((C.x1 + 1) << sh) - 1);
            const int y0 = range_low(fy, reach, C.y0 << sh, Y0), y1 = range_high(fy, reach, Y0, ((C.y1 + 1) << sh) - 1);
            const int z0 = range_low(fz, reach, C.z0 << sh, Z0), z1 = range_high(fz, reach, Z0, ((C.z1 + 1) << sh) - 1);
            if (mode == M_REST && x0 >= X0 - 1 && x1 <= X0 + 1 && y0 >= Y0 - 1 && y1 <= Y0 + 1 && z0 >= Z0 - 1 && z1 <= Z0 + 1)
                break;
            const int runs = sh == 0 ? 1 : (x1 >> sh) - (x0 >> sh) + 1;
            const int ny = y1 - y0 + 1;
            total = ny * (z1 - z0 + 1) * runs;
            base = 0;
            if (coarse && total > 64) {
                coarse = false;
                plan = true;
                continue;
            }
            __syncwarp();
            if (lane == 0) {
                U.box[0] = x0; U.box[1] = x1; U.box[2] = y0; U.box[3] = ny; U.box[4] = z0; U.box[5] = runs;
            }
            __syncwarp();
        }
        // ---- up to 32 (M_REST: 64) runs of photons, one or two per lane
        uint32_t a = 0u, b = 0u, a2 = 0u, b2 = 0u;
        const int t = base + lane;
        if (mode == M_RING) {
            const int t3 = t / 3, t9 = t3 / 3;
            const int X = s.X0 + t - 3 * t3 - 1, Y = s.Y0 + t3 - 3 * t9 - 1, Z = s.Z0 + t9 - 1;
            const Cube C = cube_of(G, E, s.X0 >> sh, s.Y0 >> sh, s.Z0 >> sh);
            const int cx = X >> sh, cy = Y >> sh, cz = Z >> sh;
            if (t < total && cx >= C.x0 && cx <= C.x1 && cy >= C.y0 && cy <= C.y1 && cz >= C.z0 && cz <= C.z1) {
                const float gx = axis_gap(s.qx, G.mn[0] + X * E.sc - E.pad, G.mn[0] + (X + 1) * E.sc + E.pad, X == 0,
                                          X == (G.gx << sh) - 1);
                const float gy = axis_gap(s.qy, G.mn[1] + Y * E.sc - E.pad, G.mn[1] + (Y + 1) * E.sc + E.pad, Y == 0,
                                          Y == (G.gy << sh) - 1);
                const float gz = axis_gap(s.qz, G.mn[2] + Z * E.sc - E.pad, G.mn[2] + (Z + 1) * E.sc + E.pad, Z == 0,
                                          Z == (G.gz << sh) - 1);
                if (gx * gx + gy * gy + gz * gz <= lim2 * m2) {
                    const uint32_t key = sub_key(G, X, Y, Z, sh);
                    a = __ldg(G.key_starts + key);
                    b = __ldg(G.key_starts + key + 1);
                }
            }
        } else {
            // Rows in (z, y) order and runs in x order: the photons come in
            // (z, y, x) order of their sub-cells (M_REST; M_WIDE sorts).
            const int x0 = U.box[0], x1 = U.box[1], y0 = U.box[2], ny = U.box[3], z0 = U.box[4], runs = U.box[5];
            const int row = runs == 1 ? t : small_div(t, runs, rcp((float)runs)), run = t - row * runs;
            const int iz = small_div(row, ny, rcp((float)ny));
            const int Y = y0 + row - iz * ny, Z = z0 + iz;
            const float gy = axis_gap(s.qy, G.mn[1] + Y * unit - E.pad, G.mn[1] + (Y + 1) * unit + E.pad, Y == 0,
                                      Y == (G.gy << sh) - 1);
            const float gz = axis_gap(s.qz, G.mn[2] + Z * unit - E.pad, G.mn[2] + (Z + 1) * unit + E.pad, Z == 0,
                                      Z == (G.gz << sh) - 1);
            const float rem = lim2 * m2 - gy * gy - gz * gz;
            if (t < total && rem >= 0.f) {
                const float inv = coarse ? rcp(G.cell) : E.inv_sc;
                const float fx = (s.qx - G.mn[0]) * inv;
                const float rx = (sqrt_approx(rem) * (1.f + 1e-5f) + E.pad) * inv + 0.01f;
                int xa = range_low(fx, rx, x0, x1), xb = range_high(fx, rx, x0, x1);
                if (sh == 0) {
                    const uint32_t* ks = G.key_starts + ((size_t)((Y + Z * G.gy) * G.gx + xa) << (3 * E.sh));
                    a = __ldg(ks);
                    b = __ldg(ks + ((size_t)(xb + 1 - xa) << (3 * E.sh)));
                    if (mode == M_REST && abs(Y - s.Y0) <= 1 && abs(Z - s.Z0) <= 1) {   // (sub-cells: S = 1)
                        b2 = b;
                        b = __ldg(ks + (min(max(s.X0 - 1, xa), xb + 1) - xa));
                        a2 = __ldg(ks + (min(max(s.X0 + 2, xa), xb + 1) - xa));
                    }
                } else {
                    const int c = (x0 >> sh) + run;
                    xa = max(xa, c << sh);
                    xb = min(xb, ((c + 1) << sh) - 1);
                    if (xa <= xb) {
                        const uint32_t* ks = G.key_starts + sub_key(G, xa, Y, Z, sh);
                        a = __ldg(ks);
                        b = __ldg(ks + (xb + 1 - xa));
                        if (mode == M_REST && abs(Y - s.Y0) <= 1 && abs(Z - s.Z0) <= 1) {
                            b2 = b;
                            b = __ldg(ks + (min(max(s.X0 - 1, xa), xb + 1) - xa));
                            a2 = __ldg(ks + (min(max(s.X0 + 2, xa), xb + 1) - xa));
                        }
                    }
                }
            }
        }
        base += 32;
        const bool end = base >= total;
        {
            const unsigned m1 = __ballot_sync(0xffffffffu, b > a), mb = __ballot_sync(0xffffffffu, b2 > a2);
            int pos = qn + __popc(m1 & lanemask_lt()) + __popc(mb & lanemask_lt());
            if (b > a) { U.qa[pos] = a; U.qc[pos] = b - a; pos++; }
            if (b2 > a2) { U.qa[pos] = a2; U.qc[pos] = b2 - a2; }
            qn += __popc(m1) + __popc(mb);
            __syncwarp();
        }
        if (!end && (qn < 32 || coarse)) continue;
        if (coarse) {   // at most 64 runs: too many photons in them?
            uint32_t sum = 0u;
            for (int e = lane; e < qn; e += 32) sum += min(U.qc[e], COARSE_MAX + 1u);
            if (__reduce_add_sync(0xffffffffu, sum) > COARSE_MAX) {
                coarse = false;
                plan = true;
                qn = 0;
                continue;
            }
        }
        // ---- the photons of 32 queued runs at a time as one list, one photon
        // per lane: list entry o lies in the last run that starts at or before
        // it (the runs that started before this round of 32 plus those that
        // start in it at or before this lane; runs are not empty)
#pragma unroll 1
        for (int q0 = 0; q0 < qn; q0 += 32) {
            uint32_t ra = 0u, c = 0u;
            if (q0 + lane < qn) { ra = U.qa[q0 + lane]; c = U.qc[q0 + lane]; }
            uint32_t incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t photons = __shfl_sync(0xffffffffu, incl, 31);
            const uint32_t excl = q0 + lane < qn ? incl - c : 0xffffffffu;
            const uint32_t delta = ra - excl;
            const V3 q = v3(s.qx, s.qy, s.qz);
            auto enter = [&](float d2, uint32_t j) {   // the lanes whose photon is within lim2
                const bool ok = d2 <= lim2;
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                if (ok) {
                    U.ent[n + __popc(m & lanemask_lt())] = make_uint2(__float_as_uint(d2), j);
                    atomicAdd(&U.dh[min((uint32_t)(d2 * bscale), (uint32_t)(NB - 1))], 1u);
                }
                n += __popc(m);
                if (n > UCAP - 32) {
                    lim2 = fminf(lim2, overflow<UCAP>(U, G.gpos, n, k, bscale, lane));
                    n = U.box[7];
                    fn = min(fn, -1);
                }
            };
            int before = -1;
#pragma unroll 1
            for (uint32_t p0 = 0; p0 < photons; p0 += 32) {
                const uint32_t starts = __reduce_or_sync(0xffffffffu, bit_or_zero(excl - p0));
                const uint32_t o = min(p0 + lane, photons - 1);   // lanes past the end read the last photon, unused
                const uint32_t j = __shfl_sync(0xffffffffu, delta, before + __popc(starts & lanemask_le())) + o;
                before += __popc(starts);
                const float4 p = __ldg(G.gpos + j);
                const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                // (NaN: within no bound; infinity is within that of r = inf)
                enter(p0 + lane < photons ? d2 : __int_as_float(0x7fffffff), j);
            }
        }
        qn = 0;
        __syncwarp();
        if (!end) continue;

        // ---- what next
        if (mode == M_REST) break;
        plan = true;
        if (n >= k) {
            if (mode == M_WIDE) break;
            found = find_bin(U.dh, k, lane);
            fn = n;
            // the k-th lies in that bin: its upper edge (with a margin over the rounding of d2 * bscale) bounds it
            if (bscale < 1e30f) lim2 = fminf(lim2, __fdividef((float)((found & 255u) + 1u), bscale) * m2);
            if (lim2 * m2 < s.block2) break;
            mode = M_REST;
            continue;
        }
        if (lim2 == E.r2) {           // all within r is found ...
            if (mode == M_WIDE || lim2 * m2 < s.block2) break;
            mode = M_WIDE;            // ... in the 27 sub-cells, which hold k: r hardly leaves them
        } else {
            lim2 = next_bound(lim2, n, k, mode == M_WIDE, fn == -2, E.r2, E.ring2, E.far2);
            plan = mode == M_WIDE;
            fn = -2;
        }
        coarse = plan && lim2 > 16.f * E.sc * E.sc && E.sh > 0;
        bscale = __fdividef((float)NB, lim2);
        n = 0;
        base = 0;
        reinterpret_cast<uint2*>(U.dh)[lane] = make_uint2(0u, 0u);
        __syncwarp();
    }
    const bool sorted = mode != M_WIDE;   // the store is in the estimate's order

    float smax;   // the largest squared distance of the answer
    if (n > k) {
        if (fn != n) found = find_bin(U.dh, k, lane);
        smax = cut_store<UCAP>(U, G.gpos, n, k, found, bscale, 0, lane);
    } else {
        uint32_t m = 0u;
#pragma unroll 1
        for (int e = lane; e < n; e += 32) m = max(m, U.ent[e].x);
        smax = __uint_as_float(__reduce_max_sync(0xffffffffu, m));
    }
    const int cnt = n;
    const float rk = sqrtf(smax);
    uint2* ent = U.ent;
    if (!sorted && cnt > 0) {
        shells_order<UCAP>(G, E, U, s, cnt, lane);
        ent += UCAP / 2;
    }
    __syncwarp();

    // estimate (Raytracer.cuh:110-138): lanes take entries, then a fixed-order
    // reduction.  The filter's two divisions (by 2 r_k^2 and by its norm) are
    // multiplications by reciprocals taken once per query (the estimate
    // changes by float rounding only); a map of uniform power takes each
    // photon's power from the grid parameters instead of loading it (the same
    // products and sums, so a traced map and the same photons given as a list
    // give the same bits).
    V3 res = v3(0.f, 0.f, 0.f);
    const V3 nrm = ld3(pnrm);
    if (cnt > 0 && !(require_full && cnt != k)) {
        const float alpha = 1.818f, beta = 1.953f;
        const float fr = rk * rk;
        const float inv_2fr = 1.f / (2.f * fr);
        const bool uni = UNI && G.pow_uniform;
        const V3 pwu = UNI ? v3(G.pw[0], G.pw[1], G.pw[2]) : v3(0.f, 0.f, 0.f);
        // the channels of a white light's map are one sum
        const bool white = uni && pwu.x == pwu.y && pwu.x == pwu.z;
        auto filter = [&](uint32_t d2) {
            const float d = sqrtf(__uint_as_float(d2));
            return alpha * (1.f - (1.f - expf(-beta * d * d * inv_2fr)) * inv_norm);
        };
#pragma unroll 1
        for (int e0 = 0; e0 < cnt; e0 += 64) {
            const int ea = e0 + lane, eb = ea + 32;
            bool va = ea < cnt, vb = eb < cnt;
            const uint2 xa = va ? ent[ea] : make_uint2(0u, 0u), xb = vb ? ent[eb] : make_uint2(0u, 0u);
            const V3 pda = va ? ld3(G.gdir + 3 * (size_t)xa.y) : v3(0.f, 0.f, 0.f);
            const V3 pdb = vb ? ld3(G.gdir + 3 * (size_t)xb.y) : v3(0.f, 0.f, 0.f);
            va = va && vdot(nrm, vneg(pda)) > 0;
            vb = vb && vdot(nrm, vneg(pdb)) > 0;
            const float fa = filter(xa.x), fb = filter(xb.x);
            if (white) {
                if (va) res.x += pwu.x * fa;
                if (vb) res.x += pwu.x * fb;
            } else {
                if (va) res = vadd(res, vscale(uni ? pwu : ld3(G.gpow + 3 * (size_t)xa.y), fa));
                if (vb) res = vadd(res, vscale(uni ? pwu : ld3(G.gpow + 3 * (size_t)xb.y), fb));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) res.x += __shfl_xor_sync(0xffffffffu, res.x, o);
        if (white) {
            res.y = res.z = res.x;
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                res.y += __shfl_xor_sync(0xffffffffu, res.y, o);
                res.z += __shfl_xor_sync(0xffffffffu, res.z, o);
            }
        }
        float common = 1.f / (3.14159265358979f * (rk * rk) * 1);
        res = vscale(res, common);
    }
    if (lane == 0) {
        st3(O.rad + 3 * i, res);
        if (O.cnt) O.cnt[i] = cnt;
        if (O.rk) O.rk[i] = rk;
    }
    if (O.ids) {
        write_ids<UCAP>(U, G.gpos, ent, cnt, k, rk, O.ids + i * k, lane);
    }
    __syncwarp();
}

__device__ __forceinline__ void gather_zero(int64_t i, int k, const GatherOut& O, int lane) {
    if (lane == 0) {
        st3(O.rad + 3 * i, v3(0.f, 0.f, 0.f));
        if (O.cnt) O.cnt[i] = 0;
        if (O.rk) O.rk[i] = 0.f;
    }
    if (O.ids) for (int e = lane; e < k; e += 32) O.ids[i * k + e] = 0xffffffffu;
}

__device__ __forceinline__ float filter_norm() { return 1.f / (1.f - expf(-1.953f)); }

// record qi of Q: its index, position and whether it asks for this map
__device__ __forceinline__ int64_t record_of(const GatherQueries& Q, int64_t qi) {
    return Q.idx ? (int64_t)__ldg(Q.idx + qi) : qi;
}
__device__ __forceinline__ bool load_query(const GatherQueries& Q, int64_t i, V3& q) {
    if (Q.pos3) {
        q = ld3(Q.pos3 + 3 * i);
        return true;
    }
    q = xyz(Q.pos4[i]);
    return (__float_as_uint(Q.nrm4[i].w) & Q.flag_mask) != 0u;
}
__device__ __forceinline__ const float* normal_of(const GatherQueries& Q, int64_t i) {
    return Q.pos3 ? Q.nrm3 + 3 * i : reinterpret_cast<const float*>(Q.nrm4 + i);
}

// Queries 0 .. cnt - 1 of a block (cnt <= its threads).  Each thread sets one
// query up (FEW: each warp), then the warps take them in order: neighbouring queries (the frame's
// come in Morton order) run at the same time on an SM and share its L1 (32
// consecutive queries per warp instead: 0.5 ms more for the 10M-photon frame).
// FEW: no more queries than warps.
template <int UCAP, int NW, bool FEW = false, class Stage, class Answer>
__device__ __forceinline__ void block_queries(BlockSmem<UCAP, NW>& M, int cnt, const Stage& stage, const Answer& answer) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) M.next = 0;
    const int own = FEW ? (int)threadIdx.x >> 5 : (int)threadIdx.x;
    if (own < cnt) stage(own);
    __syncthreads();
#pragma unroll 1
    while (true) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&M.next, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= cnt) break;
        answer(t);
    }
}

template <int UCAP, bool FEW = false>
__device__ __forceinline__ void gather_block(const GatherGrid& G, const GatherReach& E, BlockSmem<UCAP, WARPS>& M,
                                             const GatherQueries& Q, int64_t q0, int cnt, int k, int require_full,
                                             const GatherOut& O, float inv_norm) {
    const int lane = threadIdx.x & 31;
    WarpStore<UCAP>& U = M.st[threadIdx.x >> 5];
    block_queries<UCAP, WARPS, FEW>(
        M, cnt,
        [&](int t) {
            V3 q;
            const bool active = load_query(Q, record_of(Q, q0 + t), q) && k > 0;
            if (active) stage_query<FEW>(G, E, M.q[t], q, k, Q_ACTIVE);
            else M.q[t].flags = 0;
        },
        [&](int t) {
            const int64_t i = record_of(Q, q0 + t);
            if (M.q[t].flags & Q_ACTIVE)
                gather_query<UCAP>(G, E, U, M.q[t], i, normal_of(Q, i), k, require_full, O, inv_norm, lane);
            else
                gather_zero(i, k, O, lane);
        });
}

// FEW: launched with one query per warp (per == WARPS)
template <int UCAP, bool FEW>
__global__ void __launch_bounds__(WARPS * 32, 4)
k_gather(GatherGrid G, GatherReach E, GatherQueries Q, int k, int require_full, GatherOut O, int per) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int64_t q0 = (int64_t)blockIdx.x * per;
    gather_block<UCAP, FEW>(G, E, *reinterpret_cast<BlockSmem<UCAP, WARPS>*>(smem_raw), Q, q0,
                            (int)min((int64_t)per, Q.n - q0), k, require_full, O, filter_norm());
}

// Queries a block takes at a time from n, for `blocks` resident ones: one per
// thread, fewer where the blocks would not get 16 turns (the last ones end
// together; 4 turns: 0.07 ms more at 547K queries), but two per warp while
// there are enough (the set-up of one alone costs a ninth at 62K queries).
__host__ __device__ __forceinline__ int block_chunk(int64_t n, int64_t blocks, int warps) {
    const int64_t c = n / (16 * blocks) / warps * warps, least = n >= 4 * blocks * warps ? 2 * warps : warps;
    return (int)(c < least ? least : c > 32 * warps ? 32 * warps : c);
}

// Listed queries, persistent: blocks take list positions from *queue until
// min(*n_dev, Q.n) is reached (a device-side count, so no host round trip
// sits between the list's producer and this launch); position qi answers
// record Q.idx[qi].
template <int UCAP>
__global__ void __launch_bounds__(WARPS * 32, 4)
k_gather_listed(GatherGrid G, GatherReach E, GatherQueries Q, const unsigned long long* __restrict__ n_dev,
                unsigned long long* __restrict__ queue, int k, GatherOut O) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BlockSmem<UCAP, WARPS>& M = *reinterpret_cast<BlockSmem<UCAP, WARPS>*>(smem_raw);
    const int64_t n = (int64_t)min(*n_dev, (unsigned long long)Q.n);
    const int per = block_chunk(n, gridDim.x, WARPS);
    const float inv_norm = filter_norm();
#pragma unroll 1
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) M.first = atomicAdd(queue, (unsigned long long)per);
        __syncthreads();
        const int64_t q0 = (int64_t)M.first;
        if (q0 >= n) break;
        gather_block<UCAP>(G, E, M, Q, q0, (int)min((int64_t)per, n - q0), k, 0, O, inv_norm);
    }
}

template <int UCAP>
cudaError_t launch_listed(const GatherGrid& G, const GatherQueries& Q, const unsigned long long* n_dev,
                          unsigned long long* queue, float r, int k, const GatherOut& O, int sm_count,
                          cudaStream_t st) {
    const size_t smem = sizeof(BlockSmem<UCAP, WARPS>);
    cudaError_t e = cudaFuncSetAttribute(k_gather_listed<UCAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gather_listed<UCAP>, WARPS * 32, smem)) != cudaSuccess)
        return e;
    const int64_t need = (Q.n + WARPS - 1) / WARPS;
    const unsigned grid = (unsigned)std::min<int64_t>(need, (int64_t)std::max(per_sm, 1) * std::max(sm_count, 1));
    k_gather_listed<UCAP><<<grid, WARPS * 32, smem, st>>>(G, gather_reach(G, r), Q, n_dev, queue, k, O);
    return cudaGetLastError();
}

__device__ __forceinline__ int find_instance_px(const int64_t* __restrict__ off, int ninst, int64_t g) {
    int lo = 0, hi = ninst - 1;   // last i with off[i] <= g
#pragma unroll 1
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Requests of several instances, one persistent work queue: blocks take
// request indices from *queue until *n_req (the eye
// pass's device counter of this class) is reached.  Request q belongs to the
// instance of its pixel (c.w bits, a global pixel index in [px_off[i],
// px_off[i+1])) and is answered with that instance's grid, r and k.  The eye
// pass puts every request in its class's range, so an instance of another
// store class never appears here; the check guards the store size.
template <int UCAP, int NW>
__global__ void __launch_bounds__(NW * 32, 32 / NW)
k_gather_multi(const GatherInstDev* __restrict__ tab, const int64_t* __restrict__ px_off, int ninst,
               GatherQueries Q, const float4* __restrict__ rec_c, const unsigned long long* __restrict__ n_req,
               unsigned long long* __restrict__ queue, int cls, GatherOut O) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BlockSmem<UCAP, NW>& M = *reinterpret_cast<BlockSmem<UCAP, NW>*>(smem_raw);
    const int lane = threadIdx.x & 31;
    WarpStore<UCAP>& U = M.st[threadIdx.x >> 5];
    const int64_t n = (int64_t)min(*n_req, (unsigned long long)Q.n);
    const int per = block_chunk(n, gridDim.x, NW);
    const float inv_norm = filter_norm();
#pragma unroll 1
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) M.first = atomicAdd(queue, (unsigned long long)per);
        __syncthreads();
        const int64_t q0 = (int64_t)M.first;
        if (q0 >= n) break;
        block_queries(
            M, (int)min((int64_t)per, n - q0),
            [&](int t) {
                const int64_t i = q0 + t;
                const int inst = find_instance_px(px_off, ninst, (int64_t)__float_as_uint(rec_c[i].w));
                const GatherInstDev& T = tab[inst];
                V3 q;
                const bool active = load_query(Q, i, q) && T.k > 0;
                const int tag = inst << 8;
                if (T.cls != cls) M.q[t].flags = -1;
                else if (active) stage_query(T.G, T.E, M.q[t], q, T.k, Q_ACTIVE | tag);
                else M.q[t].flags = tag;
            },
            [&](int t) {
                const int flags = M.q[t].flags;
                if (flags < 0) return;
                if (flags & Q_ACTIVE) {
                    const GatherInstDev& T = tab[flags >> 8];
                    gather_query<UCAP, false>(T.G, T.E, U, M.q[t], q0 + t, normal_of(Q, q0 + t), T.k, 0, O, inv_norm, lane);
                } else {
                    gather_zero(q0 + t, 0, O, lane);
                }
            });
    }
}

template <int UCAP>
cudaError_t launch(const GatherGrid& G, const GatherQueries& Q, float r, int k, int require_full, const GatherOut& O,
                   cudaStream_t st) {
    const size_t smem = sizeof(BlockSmem<UCAP, WARPS>);
    const int per = block_chunk(Q.n, 4 * 148, WARPS);
    const auto kernel = per == WARPS ? k_gather<UCAP, true> : k_gather<UCAP, false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const unsigned blocks = (unsigned)((Q.n + per - 1) / per);
    kernel<<<blocks, WARPS * 32, smem, st>>>(G, gather_reach(G, r), Q, k, require_full, O, per);
    return cudaGetLastError();
}

}  // namespace

template <int UCAP, int NW>
cudaError_t launch_multi(const GatherInstDev* tab, const int64_t* px_off, int ninst, const GatherQueries& Q,
                         const float4* rec_c, const unsigned long long* n_req, unsigned long long* queue, int cls,
                         const GatherOut& O, int sm_count, cudaStream_t st) {
    const size_t smem = sizeof(BlockSmem<UCAP, NW>);
    cudaError_t e = cudaFuncSetAttribute(k_gather_multi<UCAP, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gather_multi<UCAP, NW>, NW * 32, smem)) != cudaSuccess)
        return e;
    k_gather_multi<UCAP, NW><<<(unsigned)(std::max(per_sm, 1) * sm_count), NW * 32, smem, st>>>(
        tab, px_off, ninst, Q, rec_c, n_req, queue, cls, O);
    return cudaGetLastError();
}

cudaError_t gather_multi(const GatherInstDev* tab, const int64_t* px_off, int ninst, const GatherQueries& Q,
                         const float4* rec_c, const unsigned long long* n_req, int64_t split,
                         unsigned long long* queues, const GatherOut& O, int warps, const int max_k[2], int sm_count,
                         cudaStream_t st) {
    if (Q.n <= 0) return cudaSuccess;
    if (split < 0 || split > Q.n || O.ids || O.cnt || O.rk || Q.idx) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(queues, 0, 16, st);
    if (e != cudaSuccess) return e;
    // class 0: [0, split); class 1: the records from split on, indexed from 0
    GatherQueries Q0 = Q, Q1 = Q;
    Q0.n = split;
    Q1.n = Q.n - split;
    Q1.pos4 = Q.pos4 + split;
    Q1.nrm4 = Q.nrm4 + split;
    GatherOut O1 = O;
    O1.rad = O.rad + 3 * split;
    const float4* c1 = rec_c + split;
    auto one = [&](auto ucap, const GatherQueries& q, const float4* c, int cls, const GatherOut& o) {
        constexpr int U = decltype(ucap)::value;
        return warps == 4 ? launch_multi<U, 4>(tab, px_off, ninst, q, c, n_req + cls, queues + cls, cls, o, sm_count, st)
                          : launch_multi<U, 8>(tab, px_off, ninst, q, c, n_req + cls, queues + cls, cls, o, sm_count, st);
    };
    using std::integral_constant;
    if (Q0.n > 0) {
        e = max_k[0] <= 64 ? one(integral_constant<int, 192>(), Q0, rec_c, 0, O)
                           : one(integral_constant<int, 256>(), Q0, rec_c, 0, O);
        if (e != cudaSuccess) return e;
    }
    if (Q1.n > 0)
        e = max_k[1] <= 160 ? one(integral_constant<int, 352>(), Q1, c1, 1, O1)
                            : one(integral_constant<int, 512>(), Q1, c1, 1, O1);
    return e;
}

GatherReach gather_reach(const GatherGrid& G, float r) {
    GatherReach E{};
    E.r = r;
    if (!(r >= 0.f)) {
        E.r2 = -1.f;                // no distance is <= a negative radius or NaN
    } else if (std::isinf(r)) {
        E.r2 = r;
    } else {
        float s = std::min(r * r, FLT_MAX);
        while (std::sqrt(s) > r) s = std::nextafter(s, 0.f);
        while (s < FLT_MAX && std::sqrt(std::nextafter(s, INFINITY)) <= r) s = std::nextafter(s, INFINITY);
        E.r2 = s;
    }
    const float c = std::ceil(r / G.cell);
    E.rc = c != c ? 0 : (int)std::min(std::max(c, -1e9f), 1e9f);
    E.sh = 0;
#pragma unroll 1
    while ((1 << E.sh) < G.S) E.sh++;
    E.sc = G.cell / (float)G.S;
    E.inv_sc = 1.f / E.sc;
    E.ring2 = 12.5f * E.sc * E.sc;   // 3 (2 sc)^2 and a margin
    E.far2 = G.cell * G.cell * ((float)G.gx * (float)G.gx + (float)G.gy * (float)G.gy + (float)G.gz * (float)G.gz);
    E.pad = G.cell * 1e-4f;
    return E;
}

int gather_class(int k) { return k <= 96 ? 0 : 1; }

cudaError_t gather_listed(const GatherGrid& G, const GatherQueries& Q, const unsigned long long* n_dev,
                          unsigned long long* queue, float r, int k, const GatherOut& O, int sm_count,
                          cudaStream_t st) {
    if (Q.n <= 0) return cudaSuccess;
    if (!Q.idx || !Q.pos4 || !Q.nrm4) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(queue, 0, 8, st);
    if (e != cudaSuccess) return e;
    if (k <= 64) return launch_listed<192>(G, Q, n_dev, queue, r, k, O, sm_count, st);
    if (k <= 96) return launch_listed<256>(G, Q, n_dev, queue, r, k, O, sm_count, st);
    if (k <= 160) return launch_listed<352>(G, Q, n_dev, queue, r, k, O, sm_count, st);
    if (k <= 256) return launch_listed<512>(G, Q, n_dev, queue, r, k, O, sm_count, st);
    return cudaErrorInvalidValue;
}

// Store sizes: at least 2 k (the shells' order needs the upper half) and room for
// the guess's 1.6 k candidates, no more: shared memory the store does not take
// is L1 for the photons (k 128: 352 entries instead of 512 1.65 -> 1.53 ms; k 64:
// 192 instead of 256 2.29 -> 2.23 ms).
cudaError_t gather(const GatherGrid& G, const GatherQueries& Q, float r, int k, int require_full,
                   const GatherOut& O, unsigned* status, cudaStream_t st) {
    (void)status;
    if (Q.n <= 0) return cudaSuccess;
    if (k <= 64) return launch<192>(G, Q, r, k, require_full, O, st);
    if (k <= 96) return launch<256>(G, Q, r, k, require_full, O, st);
    if (k <= 160) return launch<352>(G, Q, r, k, require_full, O, st);
    if (k <= 256) return launch<512>(G, Q, r, k, require_full, O, st);
    return cudaErrorInvalidValue;
}

}  // namespace pm
