// Tree construction without chain walks: basins, saddles, sorted chains.
//
// The merging build (dcf_build.cu) zips the sorted root paths of neighbouring tiles
// node by node, so its time grows with the depth of the tree: on float images, whose
// levels are nearly all distinct, root paths run through a large part of the image.
// Here the same tree comes out of a fixed number of passes plus one radix sort,
// whatever its depth.
//
// Pixels are ordered by (order key, index): x is above y when it comes later.  A flat
// zone is then a chain of its pixels that ends at its lowest index, which is the level
// root of the canonical form.
//
//   k_basins    every pixel points to its highest neighbour if that is above it, else
//               it is a peak and starts a basin; pointers are followed inside the tile.
//               A pixel whose higher neighbours fall into several groups that do not
//               touch each other around it is a saddle: it emits one edge (x, y) for
//               each group but the one it points into.  Higher neighbours that touch
//               are joined above x by pixels that emit (or imply) their own edges, so
//               these edges alone keep which pixels are joined at every threshold.
//   k_basin_ids every pixel's basin.
//   k_saddles, k_saddles_tail  Boruvka rounds over the basins: every component c takes its highest
//               edge; s(c) is that edge's lower pixel.  Components joined in a round
//               become one component of the next.
//   k_chain     a pixel x of basin b belongs to the chain of the first component c on
//               b's path of components with x above s(c).  Above s(c) nothing outside
//               c is joined to c, and at or below the s() of the parts that formed c
//               all of c's remaining pixels hang on one path: a chain is a path of the
//               tree, sorted by the pixel order, and its lowest pixel's parent is s(c).
//   radix sort  of the pixels by (chain, key), stable, so ties stay in index order.
//   k_order .. k_parents  canonical parents straight from the sorted order: the pixels of
//               a run of equal keys take its first, lowest pixel, that one the run below
//               it or, at the chain's end, the node of s(c).
//
// What bounds it, on images beyond a few megapixels: in k_basins, k_chain and the sort's
// first pass instructions (4096^2 u16: 64 to 67% of the issue slots with half the warps
// resident, DRAM at 8 to 35%), in the other passes the latency of shared memory, gathers
// and stores out of order (DRAM at 17 to 48%).  Below about a megapixel the latency of some
// 20 kernels and of the grid barriers in k_saddles.  Build alone (without node list
// and attributes) on GB300 against the merging build:
//   1447 x 1083 f32, 8-connected                     0.32 ms   200 ms
//   128 x 120 x 112 f32, 6-connected                 0.25 ms   141 ms
//   192 f32 cutouts of 64..1024 px (22.8 Mpx)         2.4 ms   546 ms
//   150 x 139 x 90 u16 min tree, 26-connected        0.24 ms  15.7 ms
//   2001 x 1997 u16, both trees                      0.72 ms  17.4 ms
//   8190 x 8211 u16 min tree                          5.1 ms  30.1 ms
//   16384 x 16384 u16 max tree                       19.8 ms  35.4 ms
//   1024 x 1024 u8, 4-connected                      0.17 ms  0.61 ms
//   96 x 80 u8                                       0.08 ms  0.49 ms
// Images made of ties alone: 4096 x 4096 u8 of one value 1.14 against 1.24 ms with
// attributes, a checkerboard 11.1 against 18.6.
#include "dcf_around.h"
#include "dcf_kernels.cuh"

namespace dcf {

using u64 = unsigned long long;

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
// Basin and component numbers as they stand in the pointer arrays: a value below zero
// is final (the number in the low 31 bits), anything else points further on.
constexpr int FINAL = (int)0x80000000u;
constexpr int FINAL_NONE = -1;  // a component with no parent
__device__ __forceinline__ int final_id(int v) { return v & 0x7FFFFFFF; }
// a pixel's final label: its basin, and a mark on the pixels that chains hang on
constexpr int LABEL_HUNG = 1 << 30;
__device__ __forceinline__ int basin_of(int v) { return v & 0x3FFFFFFF; }

// Pixel x in the order of the edge weights: key, index, and three bits that tell
// the edges of one pixel apart (at most seven: eight groups around a pixel).  Indices
// stay below 2^29.
__device__ __forceinline__ u64 edge_weight(uint32_t key, int x, int j)
{
    return ((u64)key << 32) | ((unsigned)x << 3) | (unsigned)j;
}
__device__ __forceinline__ int weight_pixel(u64 w) { return (int)((unsigned)w >> 3); }

// counters of one build, zeroed at its start
enum ForestCtr : int { FC_NEXT = 0, FC_EDGES0, FC_EDGES1, FC_BARRIER, FC_CHAINS, FC_SPARE, FC_LOW, FC_LIST, FC_ROUND, FC_TICKET, FC_COUNT = FC_TICKET + 8 };

template <typename T> struct KeyBits { static constexpr int bits = 32; };
template <> struct KeyBits<uint8_t> { static constexpr int bits = 8; };
template <> struct KeyBits<uint16_t> { static constexpr int bits = 16; };

// ---------------------------------------------------------------------------
// basins and saddle edges of one tile
// ---------------------------------------------------------------------------
constexpr int BASIN_THREADS = 256, BASIN_PIX = 2048, BASIN_PER = BASIN_PIX / BASIN_THREADS;
template <int CONN> struct BasinTile {
    static constexpr bool flat = CONN == 4 || CONN == 8;
    static constexpr int X = flat ? BASIN_TILE_X : 16, Y = flat ? BASIN_TILE_Y : 16, Z = flat ? 1 : 8;
    static constexpr int SX = X + 2, SY = Y + 2, SZ = flat ? 1 : Z + 2;
    static constexpr int CELLS = SX * SY * SZ;
};
static_assert(BASIN_TILE_X * BASIN_TILE_Y == BASIN_PIX, "tile size");

template <typename T, bool MIN, int CONN, bool BATCH>
__global__ void __launch_bounds__(BASIN_THREADS)
k_basins(const T *__restrict__ img, Geom g, const BatchImg *__restrict__ imgs, const BatchTile *__restrict__ tiles,
         const unsigned *kmax, float *__restrict__ gval, int *__restrict__ label,
         u64 *__restrict__ ew, int2 *__restrict__ eab, unsigned *ctr, unsigned ecap, unsigned *err)
{
    after_previous();
    using BT = BasinTile<CONN>;
    __shared__ uint32_t sk[BT::CELLS];
    __shared__ int snext[BASIN_PIX];
    __shared__ unsigned s_warp[BASIN_THREADS / 32];
    __shared__ unsigned s_base[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float gmax = MIN ? key_to_level(*kmax) : 0.0f;
    long long off = 0;
    int W = g.W, H = g.H, x0, y0, z0 = 0;
    if (BATCH) {
        const BatchTile tl = tiles[blockIdx.x];
        const BatchImg im = imgs[tl.img];
        off = im.off;
        W = im.W;
        H = im.H;
        x0 = tl.x0;
        y0 = tl.y0;
    } else {
        // rows of tiles, of all slices, counted over grid.y and grid.z: each holds 65535 only
        // (a 1-D grid, with a division for the place: a call on 16384^2 u16 28.06 ms, this 28.00)
        const unsigned row = blockIdx.y + gridDim.y * blockIdx.z, rows = (H + BT::Y - 1) / BT::Y;
        const unsigned slice = BT::flat ? 0u : row / rows;
        x0 = (int)blockIdx.x * BT::X;
        y0 = (int)(row - slice * rows) * BT::Y;
        z0 = (int)slice * BT::Z;
        if (BT::flat ? y0 >= H : z0 >= g.D) return;  // beyond the last row: the whole block
    }
    const int D = BT::flat ? 1 : g.D;
    const long long WH = (long long)W * H;
    for (int i = tid; i < BT::CELLS; i += BASIN_THREADS) {
        const int cx = i % BT::SX, cy = i / BT::SX % BT::SY, cz = BT::flat ? 1 : i / (BT::SX * BT::SY);
        const int x = x0 + cx - 1, y = y0 + cy - 1, z = z0 + cz - 1;
        uint32_t k = 0;
        if (x >= 0 && x < W && y >= 0 && y < H && z >= 0 && z < D) {
            const long long p = off + z * WH + (long long)y * W + x;
            const float lv = level_of<T, MIN>(img[p], gmax);
            k = max(order_key(lv), 1u);  // only a NaN's key can be 0
            if (cx >= 1 && cx <= BT::X && cy >= 1 && cy <= BT::Y && (BT::flat || (cz >= 1 && cz <= BT::Z))) gval[p] = lv;
        }
        sk[i] = k;
    }
    __syncthreads();
    constexpr int SXY = BT::SX * BT::SY;
    unsigned reps[BASIN_PER];
    int leave[BASIN_PER];  // a pointer that leaves the tile (cube bit), 13 = peak, -1 = stays inside or no pixel
    unsigned n = 0;        // peaks, and edges << 16
#pragma unroll
    for (int j = 0; j < BASIN_PER; j++) {
        const int i = tid + j * BASIN_THREADS;
        const int lx = i % BT::X, ly = i / BT::X % BT::Y, lz = i / (BT::X * BT::Y);
        const bool in = x0 + lx < W && y0 + ly < H && z0 + lz < D;
        reps[j] = 0;
        leave[j] = -1;
        int next = i;
        if (in) {
            int up;
            look_around<CONN>(sk + (lx + 1) + (ly + 1) * BT::SX + (BT::flat ? 0 : (lz + 1) * SXY), BT::SX, SXY, up,
                              reps[j]);
            const int tx = lx + up % 3 - 1, ty = ly + up / 3 % 3 - 1, tz = lz + up / 9 - 1;
            if (up == 13 || tx < 0 || tx >= BT::X || ty < 0 || ty >= BT::Y || tz < 0 || tz >= BT::Z) leave[j] = up;
            else next = tx + ty * BT::X + tz * BT::X * BT::Y;
            n += (up == 13 ? 1u : 0u) + ((unsigned)__popc(reps[j]) << 16);
        }
        snext[i] = next;
    }
    // exclusive scan of the counts over the block, one pair of atomics per tile
    unsigned inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();  // also: snext complete
    unsigned before = inc - n, total = 0;
    for (int w = 0; w < BASIN_THREADS / 32; w++) {
        if (w < warp) before += s_warp[w];
        total += s_warp[w];
    }
    if (tid == 0) {
        s_base[0] = atomicAdd(ctr + FC_NEXT, total & 0xFFFFu);
        s_base[1] = atomicAdd(ctr + FC_EDGES0, total >> 16);
        if (s_base[1] + (total >> 16) > ecap) raise_error(err, DEVERR_CAPACITY);
    }
    // follow the pointers inside the tile: concurrent doubling in place, a pointer read
    // while its owner moves it is the old or the new one, both on the way up
    for (int round = 0; round < 12; round++) {
        int moved = 0;
#pragma unroll
        for (int j = 0; j < BASIN_PER; j++) {
            const int i = tid + j * BASIN_THREADS;
            const int a = ((volatile int *)snext)[i], b = ((volatile int *)snext)[a];
            if (b != a) {
                ((volatile int *)snext)[i] = b;
                moved = 1;
            }
        }
        if (!__syncthreads_or(moved)) break;
    }
    // The ends of the pointers get their values: a peak its basin number, a pixel whose
    // pointer leaves the tile that neighbour's index.  They go where the keys were read
    // from, once every thread is past the keys.
    __syncthreads();
    int id = (int)(s_base[0] + (before & 0xFFFFu));
    unsigned at = s_base[1] + (before >> 16);
#pragma unroll
    for (int j = 0; j < BASIN_PER; j++) {
        const int i = tid + j * BASIN_THREADS;
        const int lx = i % BT::X, ly = i / BT::X % BT::Y, lz = i / (BT::X * BT::Y);
        const long long p = off + (z0 + lz) * WH + (long long)(y0 + ly) * W + (x0 + lx);
        unsigned m = reps[j];
        if (m) {
            const uint32_t k = sk[(lx + 1) + (ly + 1) * BT::SX + (BT::flat ? 0 : (lz + 1) * SXY)];
            for (int e = 0; m; e++, at++) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                if (at < ecap) {
                    ew[at] = edge_weight(k, (int)p, e);
                    eab[at].x = (int)(p + (b % 3 - 1) + (long long)(b / 3 % 3 - 1) * W + (b / 9 - 1) * WH);
                }
            }
        }
        const int up = leave[j];
        if (up == 13) leave[j] = FINAL | id++;
        else if (up >= 0) leave[j] = (int)(p + (up % 3 - 1) + (long long)(up / 3 % 3 - 1) * W + (up / 9 - 1) * WH);
        else leave[j] = 0;
    }
    __syncthreads();  // keys are read no more
    int *sval = (int *)sk;
#pragma unroll
    for (int j = 0; j < BASIN_PER; j++) sval[tid + j * BASIN_THREADS] = leave[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < BASIN_PER; j++) {
        const int i = tid + j * BASIN_THREADS;
        const int lx = i % BT::X, ly = i / BT::X % BT::Y, lz = i / (BT::X * BT::Y);
        if (x0 + lx < W && y0 + ly < H && z0 + lz < D)
            label[off + (z0 + lz) * WH + (long long)(y0 + ly) * W + (x0 + lx)] = sval[snext[i]];
    }
}

// Follows a pointer forest from v (path halving); returns the final value.  A halving
// CAS expects the pointer it read, so it cannot replace a final value.
__device__ __forceinline__ int follow(int *ptr, long long stride, int v, long long bound, unsigned *err)
{
    int j = __ldcg(ptr + v * stride);
    for (long long it = 0; it < bound; it++) {
        if (j < 0) return j;
        const int jj = __ldcg(ptr + j * stride);
        if (jj < 0) return jj;
        atomicCAS(ptr + v * stride, j, jj);
        v = jj;
        j = __ldcg(ptr + v * stride);
    }
    raise_error(err, DEVERR_WALK_BOUND);
    return FINAL_NONE;
}

// label becomes every pixel's basin (final values)
__global__ void k_basin_ids(int *label, long long n, unsigned *err)
{
    after_previous();
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
        const int j = __ldcg(label + p);
        if (j < 0) continue;
        const int jj = __ldcg(label + j);
        label[p] = jj < 0 ? jj : follow(label, 1, jj, n + 1, err);
    }
}

// ---------------------------------------------------------------------------
// Boruvka rounds over the basins, in one cooperative kernel
// ---------------------------------------------------------------------------
// Barrier of a whole cooperative grid on a counter that only grows; false when the
// wait ran out (an error bit is set and the caller returns).
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned &phase, unsigned *err)
{
    __shared__ int s_ok;
    __syncthreads();
    phase++;
    if (threadIdx.x == 0) {
        const unsigned target = phase * gridDim.x;
        __threadfence();
        unsigned seen = atomicAdd(bar, 1u) + 1u;
        int tries = 0;
        while (seen < target && tries < (1 << 22)) {
            __nanosleep(20);
            seen = *(volatile unsigned *)bar;
            tries++;
        }
        __threadfence();
        s_ok = seen >= target;
        if (seen < target) raise_error(err, DEVERR_WAIT_BOUND);
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ void take_best(Comp *comp, int c, u64 w)
{
    // a look first: most edges of a large component are below its best already
    if (__ldcg(&comp[c].best) < w) atomicMax(&comp[c].best, w);
}

// Appends an edge between two components (every lane of a warp calls it) and offers
// it to both as their highest.
__device__ __forceinline__ void push_edge(bool valid, u64 w, int a, int b, u64 *ew, int2 *eab, unsigned *count,
                                          Comp *comp)
{
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, valid);
    if (!m) return;
    unsigned base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(count, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    if (!valid) return;
    const unsigned i = base + __popc(m & ((1u << lane) - 1u));
    ew[i] = w;
    eab[i] = make_int2(a, b);
    take_best(comp, a, w);
    take_best(comp, b, w);
}

// Marks the pixels that components lo .. hi - 1 hang on.  Components without pixels of
// their own are no chains, so a marked pixel may have nothing hanging on it; telling them
// apart cost more (a flag per component that every pixel of a long chain looks at).
__device__ __forceinline__ void mark_hung(const Comp *comp, unsigned lo, unsigned hi, int *label, long long t,
                                          long long stride)
{
    for (long long c = lo + t; c < hi; c += stride) {
        const u64 s = __ldcg(&comp[c].best);
        if (s) atomicOr(label + weight_pixel(s), LABEL_HUNG);
    }
}

constexpr int SADDLE_THREADS = 512;
constexpr int CHAIN_THREADS = 1024, CHAIN_PER = 4, SORT_PASSES = 8;  // 32 key bits and at most 30 of a component number
constexpr unsigned TAIL_COMPS = 4096, TAIL_EDGES = 8192;  // 16-bit local numbers, 160 KB of shared memory
constexpr int TAIL_THREADS = 1024;
constexpr size_t TAIL_SMEM = TAIL_EDGES * 12 + TAIL_COMPS * 16;

__global__ void __launch_bounds__(SADDLE_THREADS)
k_saddles(int *label, long long npix, u64 *ew0, int2 *eab0, u64 *ew1, int2 *eab1, Comp *comp,
          unsigned *ctr, unsigned ecap, long long max_rounds, unsigned *err)
{
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    unsigned phase = 0;
    unsigned lo = 0, hi = __ldcg(ctr + FC_NEXT);  // the components of this round
    unsigned ne = min(__ldcg(ctr + FC_EDGES0), ecap);
    for (long long c = t0; c < hi; c += stride) {
        comp[c].best = 0ull;
        comp[c].par = FINAL_NONE;
    }
    if (!grid_barrier(ctr + FC_BARRIER, phase, err)) return;
    // from pixels to basins
    for (long long base = t0 - lane; base < ne; base += stride) {
        bool valid = base + lane < ne;
        u64 w = 0;
        int a = 0, b = 0;
        if (valid) {
            w = __ldcg(ew0 + base + lane);
            a = basin_of(__ldcg(label + weight_pixel(w)));
            b = basin_of(__ldcg(label + __ldcg(&eab0[base + lane].x)));
            valid = a != b;
        }
        push_edge(valid, w, a, b, ew1, eab1, ctr + FC_EDGES1, comp);
    }
    int cur = 1;
    long long round = 0;
    for (;; round++) {
        if (!grid_barrier(ctr + FC_BARRIER, phase, err)) return;
        u64 *ew = cur ? ew1 : ew0, *ewn = cur ? ew0 : ew1;
        int2 *eab = cur ? eab1 : eab0, *eabn = cur ? eab0 : eab1;
        ne = __ldcg(ctr + (cur ? FC_EDGES1 : FC_EDGES0));
        if (ne <= TAIL_EDGES && hi - lo <= TAIL_COMPS) break;  // k_saddles_tail
        if (round >= max_rounds) {
            if (t0 == 0) raise_error(err, DEVERR_MERGE_BOUND);
            break;
        }
        // the one edge that is a component's highest names the other side
        for (long long i = t0; i < ne; i += stride) {
            const u64 w = __ldcg(ew + i);
            const int2 ab = __ldcg(eab + i);
            if (__ldcg(&comp[ab.x].best) == w) comp[ab.x].hook = ab.y;
            if (__ldcg(&comp[ab.y].best) == w) comp[ab.y].hook = ab.x;
        }
        if (!grid_barrier(ctr + FC_BARRIER, phase, err)) return;
        if (t0 == 0) ctr[cur ? FC_EDGES0 : FC_EDGES1] = 0;  // the next list
        // Hooks lead along rising edges to the one pair that chose each other; the
        // smaller of the two numbers the new component.
        for (long long base = (long long)lo + t0 - lane; base < hi; base += stride) {
            const long long c = base + lane;
            const bool live = c < hi && __ldcg(&comp[c].best) != 0ull;
            int h = 0;
            bool root = false;
            if (live) {
                h = __ldcg(&comp[c].hook);
                root = c < h && __ldcg(&comp[h].hook) == (int)c;
            }
            const unsigned m = __ballot_sync(0xffffffffu, root);
            unsigned id = 0;
            if (m) {
                if (lane == __ffs(m) - 1) id = atomicAdd(ctr + FC_NEXT, (unsigned)__popc(m));
                id = __shfl_sync(0xffffffffu, id, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
            }
            if (root) {
                comp[id].best = 0ull;
                comp[id].par = FINAL_NONE;
                comp[c].par = FINAL | (int)id;
            } else if (live) {
                comp[c].par = h;
            }
        }
        if (!grid_barrier(ctr + FC_BARRIER, phase, err)) return;
        for (long long c = (long long)lo + t0; c < hi; c += stride)
            if (__ldcg(&comp[c].par) >= 0) {
                const int v = follow(&comp[0].par, sizeof(Comp) / sizeof(int), (int)c, npix + 1, err);
                ((volatile Comp *)comp)[c].par = v;
            }
        if (!grid_barrier(ctr + FC_BARRIER, phase, err)) return;
        for (long long base = t0 - lane; base < ne; base += stride) {
            bool valid = base + lane < ne;
            u64 w = 0;
            int a = 0, b = 0;
            if (valid) {
                w = __ldcg(ew + base + lane);
                const int2 ab = __ldcg(eab + base + lane);
                a = final_id(__ldcg(&comp[ab.x].par));
                b = final_id(__ldcg(&comp[ab.y].par));
                valid = a != b;
            }
            push_edge(valid, w, a, b, ewn, eabn, ctr + (cur ? FC_EDGES0 : FC_EDGES1), comp);
        }
        lo = hi;
        hi = __ldcg(ctr + FC_NEXT);
        cur ^= 1;
    }
    if (t0 == 0) {
        ctr[FC_LOW] = lo;
        ctr[FC_LIST] = (unsigned)cur;
        ctr[FC_ROUND] = (unsigned)round;
    }
    mark_hung(comp, 0, lo, label, t0, stride);
}

// The last rounds, once at most TAIL_COMPS components and TAIL_EDGES edges are left: one
// block in shared memory, where a round costs a microsecond or two instead of four grid
// barriers and their L2 round trips (about 10 us).  Local numbers: component c is
// lo + c, and a round's new components follow the ones before.
__global__ void __launch_bounds__(TAIL_THREADS, 1)
k_saddles_tail(int *label, const u64 *__restrict__ ew0, const int2 *__restrict__ eab0, const u64 *__restrict__ ew1,
               const int2 *__restrict__ eab1, Comp *comp, unsigned *ctr, unsigned raw, long long max_rounds,
               unsigned *err)
{
    after_previous();
    extern __shared__ u64 tail_smem[];
    u64 *w = tail_smem, *best = w + TAIL_EDGES;
    unsigned *ab = (unsigned *)(best + TAIL_COMPS);  // ends, 16 bits each
    int *hook = (int *)(ab + TAIL_EDGES), *par = hook + TAIL_COMPS;
    __shared__ unsigned s_edges, s_next;
    const int tid = threadIdx.x;
    // zeroes without k_saddles
    const bool one = ctr[FC_LIST] != 0;
    unsigned lo = ctr[FC_LOW], nc = ctr[FC_NEXT] - lo, ne = ctr[one ? FC_EDGES1 : FC_EDGES0];
    const unsigned first = lo;
    long long round = ctr[FC_ROUND];
    if (raw) {  // from pixels to basins, here
        ne = min(ne, raw);
        if (tid == 0) s_edges = 0;
        __syncthreads();
        for (unsigned i = tid; i < ne; i += TAIL_THREADS) {
            const u64 x = ew0[i];
            const unsigned a = (unsigned)basin_of(label[weight_pixel(x)]), b = (unsigned)basin_of(label[eab0[i].x]);
            if (a == b) continue;
            const unsigned at = atomicAdd(&s_edges, 1u);
            w[at] = x;
            ab[at] = a | (b << 16);
        }
        __syncthreads();
        ne = s_edges;
        __syncthreads();
    }
    if (ne > TAIL_EDGES || nc > TAIL_COMPS) ne = 0;  // the grid gave up (an error is raised)
    for (unsigned i = tid; i < ne && !raw; i += TAIL_THREADS) {
        const int2 e = one ? eab1[i] : eab0[i];
        w[i] = one ? ew1[i] : ew0[i];
        ab[i] = (unsigned)(e.x - (int)lo) | ((unsigned)(e.y - (int)lo) << 16);
    }
    while (ne > 0 && round < max_rounds) {
        for (unsigned c = tid; c < nc; c += TAIL_THREADS) best[c] = 0ull;
        if (tid == 0) s_edges = s_next = 0;
        __syncthreads();
        for (unsigned i = tid; i < ne; i += TAIL_THREADS) {
            const u64 x = w[i];
            const unsigned a = ab[i] & 0xFFFFu, b = ab[i] >> 16;
            if (((volatile u64 *)best)[a] < x) atomicMax(best + a, x);
            if (((volatile u64 *)best)[b] < x) atomicMax(best + b, x);
        }
        __syncthreads();
        for (unsigned i = tid; i < ne; i += TAIL_THREADS) {
            const u64 x = w[i];
            const unsigned a = ab[i] & 0xFFFFu, b = ab[i] >> 16;
            if (best[a] == x) hook[a] = (int)b;
            if (best[b] == x) hook[b] = (int)a;
        }
        __syncthreads();
        // as in k_saddles: the pair that chose each other numbers the new component
        for (unsigned c = tid; c < nc; c += TAIL_THREADS) {
            if (!best[c]) {
                par[c] = FINAL_NONE;
                continue;
            }
            const int h = hook[c];
            par[c] = (int)c < h && hook[h] == (int)c ? FINAL | (int)atomicAdd(&s_next, 1u) : h;
        }
        __syncthreads();
        for (unsigned c = tid; c < nc; c += TAIL_THREADS) {
            volatile int *p = par;
            int v = p[c];
            for (int it = 0; v >= 0 && it < TAIL_COMPS; it++) {
                const int up = p[v];
                if (up >= 0) p[c] = up;  // only shortens its own way; the final value comes below
                v = up;
            }
            hook[c] = v;
        }
        __syncthreads();
        const unsigned hi = lo + nc;
        for (unsigned c = tid; c < nc; c += TAIL_THREADS) {
            const int v = hook[c];
            comp[lo + c].best = best[c];
            comp[lo + c].par = v == FINAL_NONE ? FINAL_NONE : FINAL | (int)(hi + (unsigned)final_id(v));
        }
        // edges that still join two components, in place: a thread's edges leave its
        // registers once every thread has read its own
        u64 kw[TAIL_EDGES / TAIL_THREADS];
        unsigned kab[TAIL_EDGES / TAIL_THREADS];
#pragma unroll
        for (int j = 0; j < TAIL_EDGES / TAIL_THREADS; j++) {
            const unsigned i = tid + j * TAIL_THREADS;
            kab[j] = 0u;
            if (i < ne) {
                kw[j] = w[i];
                kab[j] = (unsigned)final_id(hook[ab[i] & 0xFFFFu]) | ((unsigned)final_id(hook[ab[i] >> 16]) << 16);
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < TAIL_EDGES / TAIL_THREADS; j++)
            if ((kab[j] & 0xFFFFu) != (kab[j] >> 16)) {
                const unsigned at = atomicAdd(&s_edges, 1u);
                w[at] = kw[j];
                ab[at] = kab[j];
            }
        __syncthreads();
        ne = s_edges;
        nc = s_next;
        lo = hi;
        round++;
        __syncthreads();
    }
    if (ne > 0 && tid == 0) raise_error(err, DEVERR_MERGE_BOUND);
    for (unsigned c = tid; c < nc; c += TAIL_THREADS) {  // whole trees: nothing above
        comp[lo + c].best = 0ull;
        comp[lo + c].par = FINAL_NONE;
    }
    if (tid == 0) ctr[FC_NEXT] = lo + nc;
    __syncthreads();
    mark_hung(comp, first, lo, label, tid, TAIL_THREADS);
}

// ---------------------------------------------------------------------------
// chains
// ---------------------------------------------------------------------------
// the chain of the pixel with weight x: first component on its basin's way with x above
// the pixel it hangs on
__device__ __forceinline__ unsigned chain_of(u64 x, unsigned c, const Comp *__restrict__ comp, unsigned nc)
{
    for (int step = 0; step < 64 && c < nc; step++) {
        const int4 v = __ldg((const int4 *)(comp + c));
        const u64 s = ((u64)(unsigned)v.y << 32) | (unsigned)v.x;
        if (x > (s & ~7ull) || v.z == FINAL_NONE) break;
        c = (unsigned)final_id(v.z);
    }
    return c;
}

__device__ __forceinline__ int sort_passes(int key_bits, const unsigned *ctr)
{
    const unsigned nc = ctr[FC_NEXT];
    const int cb = nc > 1 ? 32 - __clz(nc - 1) : 0;
    return (key_bits + cb + 7) / 8;
}

// Sort keys (chain, key), and how often every digit of every sort pass occurs.  The way to a
// pixel's chain is a chain of dependent loads, so a thread takes four pixels at a time, a step
// of each in turn, as many as the deepest of a warp's pixels needs.  Instructions take 67% of
// the issue slots (4096^2 u16, half the warps, DRAM at 20%), and one large block an SM does as
// well as more and flushes its counts once (with copies of the counts by lane the
// same).  One pixel at a time and eight blocks of 256 an SM took 26 us at 1447 x 1083 f32 and
// 19 at 1024^2 u8; now 23 and 14 (four at a time with those blocks: 22 and 18; 8190 x 8211 u16
// 637, now 583; eight at a time 28 and 14, 608).
template <int KB>
__global__ void __launch_bounds__(CHAIN_THREADS) k_chain(const int *__restrict__ label, const float *__restrict__ gval,
                                                         long long n, const Comp *__restrict__ comp,
                                                         const unsigned *__restrict__ ctr, u64 *__restrict__ skey,
                                                         unsigned *totals)
{
    after_previous();
    __shared__ unsigned hist[SORT_PASSES * 256];
    const int passes = sort_passes(KB, ctr);
    for (int i = threadIdx.x; i < passes * 256; i += CHAIN_THREADS) hist[i] = 0;
    __syncthreads();
    const unsigned nc = ctr[FC_NEXT];
    constexpr int TILE = CHAIN_THREADS * CHAIN_PER;
    for (long long first = blockIdx.x * (long long)TILE + threadIdx.x; first < n; first += (long long)gridDim.x * TILE) {
        unsigned c[CHAIN_PER];
        u64 x[CHAIN_PER];
        uint32_t k[CHAIN_PER];
#pragma unroll
        for (int j = 0; j < CHAIN_PER; j++) {
            const long long p = first + j * CHAIN_THREADS;
            const float lv = p < n ? gval[p] : 0.0f;
            const uint32_t key = max(order_key(lv), 1u);
            c[j] = p < n ? (unsigned)basin_of(label[p]) : ~0u;
            x[j] = edge_weight(key, (int)p, 0);
            k[j] = KB == 32 ? key : (uint32_t)lv;
        }
        // chain_of, one step of all at a time
        unsigned open = (1u << CHAIN_PER) - 1u;
        for (int step = 0; step < 64 && open; step++) {
            int4 v[CHAIN_PER];
#pragma unroll
            for (int j = 0; j < CHAIN_PER; j++)
                if ((open >> j) & 1u && c[j] < nc) v[j] = __ldg((const int4 *)(comp + c[j]));
                else open &= ~(1u << j);
#pragma unroll
            for (int j = 0; j < CHAIN_PER; j++) {
                if (!((open >> j) & 1u)) continue;
                const u64 s = ((u64)(unsigned)v[j].y << 32) | (unsigned)v[j].x;
                if (x[j] > (s & ~7ull) || v[j].z == FINAL_NONE) open &= ~(1u << j);
                else c[j] = (unsigned)final_id(v[j].z);
            }
        }
#pragma unroll
        for (int j = 0; j < CHAIN_PER; j++) {
            const long long p = first + j * CHAIN_THREADS;
            if (p >= n) continue;
            const u64 key = ((u64)c[j] << KB) | k[j];
            skey[p] = key;
            for (int d = 0; d < passes; d++) atomicAdd(hist + d * 256 + ((unsigned)(key >> (8 * d)) & 255u), 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += CHAIN_THREADS)
        if (hist[i]) atomicAdd(totals + i, hist[i]);
}

// per chain: the chain it hangs on, and that one's count of them; the number of chains
__global__ void k_chain_up(const int *__restrict__ attach, const int *__restrict__ label,
                           const float *__restrict__ gval, const Comp *__restrict__ comp, const unsigned *__restrict__ ctr, int *__restrict__ up,
                           int *kids, unsigned *nchains)
{
    after_previous();
    const unsigned n = ctr[FC_CHAINS], nc = ctr[FC_NEXT];
    if (blockIdx.x == 0 && threadIdx.x == 0) *nchains = n;
    for (unsigned o = blockIdx.x * blockDim.x + threadIdx.x; o < n; o += gridDim.x * blockDim.x) {
        const int s = attach[o];
        int q = NONE;
        if (s != NONE) {
            const uint32_t k = max(order_key(gval[s]), 1u);
            const unsigned c = chain_of(edge_weight(k, s, 0), (unsigned)basin_of(label[s]), comp, nc);
            if (c < nc) q = comp[c].hook;  // its number, from k_chain_tables
        }
        up[o] = q;
        if (q != NONE) atomicAdd(kids + q, 1);
    }
}

// ---------------------------------------------------------------------------
// radix sort of (key, index), eight bits and one kernel a pass.  Blocks take the tiles
// of the input in order (tickets); a tile publishes its digit counts, then the running
// counts once it knows them from the tiles before it, and looks back over what those
// have published so far.  The number of passes follows from the number of components,
// which only the device knows: passes beyond it return at once, and the data is in
// buffer (passes & 1).  Before: a kernel for the counts of all blocks, one for their
// prefix sums, then the scatter, 8 bytes a pixel and two launches a pass more
// (16384^2 u16, five passes: 8.8 ms, from 11.9).
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 256, RS_PER = 16, RS_BLOCK = RS_THREADS * RS_PER, RS_WARPS = RS_THREADS / 32;
// a tile's published word per digit: none, its own count, or the count up to and with it
constexpr unsigned RS_OWN = 1u << 30, RS_UPTO = 2u << 30, RS_VALUE = RS_OWN - 1u;

constexpr size_t RS_SMEM = RS_BLOCK * 12 + RS_WARPS * 256 * 2;  // with 16-bit counts four blocks fit an SM

// Lanes whose digit is this lane's, by one vote per bit.  __match_any_sync takes a step
// per distinct value: dearer for the low key bytes, which are nearly all distinct (268 M
// pixels, first pass: 3.1 ms with it, 2.1 with votes), cheaper for the highest key byte
// and the chain numbers, of which a warp holds a few (second pass 1.5 against 1.9).
__device__ __forceinline__ unsigned same_digit(unsigned d, unsigned active)
{
    unsigned m = active;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const unsigned v = __ballot_sync(0xffffffffu, (d >> b) & 1u);
        m &= (d >> b) & 1u ? v : ~v;
    }
    return m;
}

// the first pass (iin null) takes the pixels in order, with the mark of their label
__global__ void __launch_bounds__(RS_THREADS, 4) k_rs_scatter(const u64 *__restrict__ kin, const int *__restrict__ iin,
                                                              const int *__restrict__ label,
                                                              u64 *__restrict__ kout, int *__restrict__ iout,
                                                              long long n, int pass, int key_bits, unsigned *ctr,
                                                              unsigned *state, unsigned *state_next,
                                                              const unsigned *__restrict__ totals, unsigned *err)
{
    after_previous();
    if (pass >= sort_passes(key_bits, ctr)) return;
    extern __shared__ u64 rs_smem[];
    u64 *skey = rs_smem;
    int *sidx = (int *)(skey + RS_BLOCK);
    unsigned short(*cnt)[256] = (unsigned short(*)[256])(sidx + RS_BLOCK);  // per warp and digit
    __shared__ unsigned s_warp[RS_WARPS], s_warp2[RS_WARPS], s_tile;
    __shared__ unsigned gpos[256];  // where the digit's items of this tile go, less their place in the tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < RS_WARPS * 128; i += RS_THREADS) ((unsigned *)cnt)[i] = 0;
    if (tid == 0) s_tile = atomicAdd(ctr + FC_TICKET + pass, 1u);
    __syncthreads();
    const unsigned tile = s_tile;
    const long long first = tile * (long long)RS_BLOCK;
    const int shift = 8 * pass;
    const int here = (int)min((long long)RS_BLOCK, n - first);
    // a warp takes 32 * RS_PER consecutive items, 32 at a time, so ranks keep the order
    const int mine0 = warp * 32 * RS_PER + lane;
    u64 k[RS_PER];
#pragma unroll
    for (int j = 0; j < RS_PER; j++) k[j] = mine0 + j * 32 < here ? kin[first + mine0 + j * 32] : ~0ull;
    unsigned rank[RS_PER / 2];  // two 16-bit ranks a word
    const bool votes = shift + 8 < key_bits;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_PER; j++) {
        const bool valid = mine0 + j * 32 < here;
        const unsigned d = (unsigned)(k[j] >> shift) & 255u;
        const unsigned same = votes ? same_digit(d, __ballot_sync(0xffffffffu, valid))
                                    : __match_any_sync(0xffffffffu, valid ? d : 256u);
        unsigned c = 0;
        if (valid) c = cnt[warp][d];
        __syncwarp();
        if (valid && lane == __ffs(same) - 1) cnt[warp][d] = (unsigned short)(c + __popc(same));
        __syncwarp();
        const unsigned r = c + __popc(same & ((1u << lane) - 1u));
        if (j & 1) rank[j / 2] |= r << 16;
        else rank[j / 2] = r;
    }
    __syncthreads();
    // thread = digit: prefix over the warps, then over the digits (the tile's and all tiles')
    unsigned mine = 0, start, start2;
    {
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) {
            const unsigned c = cnt[w][tid];
            cnt[w][tid] = (unsigned short)mine;
            mine += c;
        }
        ((volatile unsigned *)state)[(size_t)tile * 256 + tid] = (tile ? RS_OWN : RS_UPTO) | mine;
        state_next[(size_t)tile * 256 + tid] = 0u;  // for the next pass; nobody reads it in this one
        const unsigned all = totals[tid];
        unsigned inc = mine, inc2 = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, inc, o), t2 = __shfl_up_sync(0xffffffffu, inc2, o);
            if (lane >= o) {
                inc += t;
                inc2 += t2;
            }
        }
        if (lane == 31) {
            s_warp[warp] = inc;
            s_warp2[warp] = inc2;
        }
        __syncthreads();
        start = inc - mine;
        start2 = inc2 - all;
        for (int w = 0; w < warp; w++) {
            start += s_warp[w];
            start2 += s_warp2[w];
        }
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) cnt[w][tid] = (unsigned short)(cnt[w][tid] + start);
    }
    __syncthreads();
    // Keys to their places, then the indices on their way while the counts of the tiles
    // before are collected: keys and indices in registers at once would leave room for
    // fewer blocks.
#pragma unroll
    for (int j = 0; j < RS_PER; j++) {
        const unsigned at = (unsigned)cnt[warp][(unsigned)(k[j] >> shift) & 255u] + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
        if (mine0 + j * 32 < here) skey[at] = k[j];
        rank[j / 2] = j & 1 ? (rank[j / 2] & 0xFFFFu) | (at << 16) : (rank[j / 2] & 0xFFFF0000u) | at;
    }
    int ix[RS_PER];
#pragma unroll
    for (int j = 0; j < RS_PER; j++) {
        const int i = mine0 + j * 32;
        ix[j] = i < here ? (iin ? iin : label)[first + i] : 0;
    }
    // Counts of this digit in the tiles before, four at a look.  Tickets are drawn in order,
    // so every tile waited for runs or has run; the limit is for the case that it never
    // publishes.
    unsigned before = 0;
    if (tile) {
        const volatile unsigned *st = (const volatile unsigned *)state + tid;
        int tries = 0;
        bool done = false;
        for (long long t = (long long)tile - 1; !done;) {  // tile 0 publishes RS_UPTO
            unsigned v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = st[(t >= q ? t - q : 0) * 256];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (done || !(v[q] & (RS_OWN | RS_UPTO))) break;
                before += v[q] & RS_VALUE;
                done = (v[q] & RS_UPTO) != 0u;
                t--;
            }
            if (!done && ++tries > (1 << 22)) {
                raise_error(err, DEVERR_WAIT_BOUND);
                break;
            }
            if (t < 0) break;
        }
        ((volatile unsigned *)state)[(size_t)tile * 256 + tid] = RS_UPTO | ((before + mine) & RS_VALUE);
    }
#pragma unroll
    for (int j = 0; j < RS_PER; j++) {
        const int i = mine0 + j * 32;
        if (i < here)
            sidx[(rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu] =
                iin ? ix[j] : (int)((unsigned)(first + i) | (ix[j] & LABEL_HUNG ? ORDER_HUNG : 0u));
    }
    gpos[tid] = start2 + before - start;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_PER; j++) {
        const int i = tid + j * RS_THREADS;
        if (i < here) {
            const u64 kk = skey[i];
            const unsigned to = gpos[(unsigned)(kk >> shift) & 255u] + i;
            if (to >= n) continue;  // only after a wait that gave up
            kout[to] = kk;
            iout[to] = sidx[i];
        }
    }
}

// ---------------------------------------------------------------------------
// parents from the sorted chains
// ---------------------------------------------------------------------------
// A run of equal keys in a chain is (part of) a node; its first, lowest pixel is the
// node's level root, unless the run is the chain's lowest and the pixel the chain hangs
// on has the same key: then the node goes on in that pixel's chain.
constexpr int LINK_THREADS = 256, LINK_BLOCK = CHAIN_BLOCK, LINK_PER = LINK_BLOCK / LINK_THREADS;

// the order entries, and per block of them: the last start of a run and of a chain (0:
// none) and the number of chains that start
template <int KB>
__global__ void __launch_bounds__(LINK_THREADS) k_order(const u64 *__restrict__ k0, const u64 *__restrict__ k1,
                                                        const int *__restrict__ i0, const int *__restrict__ i1,
                                                        long long n, const Comp *__restrict__ comp,
                                                        const unsigned *__restrict__ ctr, int *__restrict__ order,
                                                        unsigned *last_run, unsigned *last_chain, unsigned *chains)
{
    after_previous();
    const bool odd = sort_passes(KB, ctr) & 1;
    const u64 *key = odd ? k1 : k0;
    const int *idx = odd ? i1 : i0;
    __shared__ unsigned s_run, s_chain, s_chains;
    if (threadIdx.x == 0) s_run = s_chain = s_chains = 0;
    __syncthreads();
    const long long first = blockIdx.x * (long long)LINK_BLOCK;
    unsigned run = 0, low = 0, count = 0;
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) {
        const long long i = first + threadIdx.x + j * LINK_THREADS;
        if (i >= n) continue;
        const u64 k = key[i], kp = i > 0 ? key[i - 1] : 0ull;
        const bool start = i == 0 || k != kp, lowest = i == 0 || (k >> KB) != (kp >> KB);
        bool root = start;
        if (lowest) {
            const uint32_t part = (uint32_t)(k & (KB == 32 ? 0xFFFFFFFFull : ((1ull << (KB & 31)) - 1)));
            const uint32_t okey = KB == 32 ? part : order_key((float)part);
            root = (uint32_t)(comp[k >> KB].best >> 32) != okey;
            low = (unsigned)i;
            count++;
        }
        if (start) run = (unsigned)i;
        const unsigned at = (unsigned)idx[i];
        // (beyond the image only after a wait of the sort that gave up)
        order[i] = (int)(min(at & ORDER_PIXEL, (unsigned)n - 1u) | (at & ORDER_HUNG) | (root ? ORDER_ROOT : 0u) |
                         (lowest ? ORDER_START : 0u));
    }
    run = __reduce_max_sync(0xffffffffu, run);
    low = __reduce_max_sync(0xffffffffu, low);
    count = __reduce_add_sync(0xffffffffu, count);
    if ((threadIdx.x & 31) == 0) {
        if (run) atomicMax(&s_run, run);
        if (low) atomicMax(&s_chain, low);
        if (count) atomicAdd(&s_chains, count);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        last_run[blockIdx.x] = s_run;
        last_chain[blockIdx.x] = s_chain;
        chains[blockIdx.x] = s_chains;
    }
}

// Exclusive running maximum of a and b and running sum of c, in place, over the entries
// of one group per block (SCAN_GROUP entries); what the group passes on goes to t*[group].
constexpr int SCAN_GROUP = 8192;
__global__ void __launch_bounds__(1024) k_scan3(unsigned *a, unsigned *b, unsigned *c, int n, unsigned *ta,
                                                unsigned *tb, unsigned *tc)
{
    after_previous();
    __shared__ unsigned s_a[32], s_b[32], s_c[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lo = blockIdx.x * SCAN_GROUP, hi = min(n, lo + SCAN_GROUP);
    unsigned ra = 0, rb = 0, rc = 0;
    for (int base = lo; base < hi; base += 1024) {
        const int i = base + threadIdx.x;
        const bool in = i < hi;
        unsigned va = in ? a[i] : 0, vb = in ? b[i] : 0, vc = in ? c[i] : 0;
        const unsigned own = vc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned x = __shfl_up_sync(0xffffffffu, va, o), y = __shfl_up_sync(0xffffffffu, vb, o),
                           z = __shfl_up_sync(0xffffffffu, vc, o);
            if (lane >= o) {
                va = max(va, x);
                vb = max(vb, y);
                vc += z;
            }
        }
        if (lane == 31) {
            s_a[warp] = va;
            s_b[warp] = vb;
            s_c[warp] = vc;
        }
        unsigned ea = __shfl_up_sync(0xffffffffu, va, 1), eb = __shfl_up_sync(0xffffffffu, vb, 1);
        if (lane == 0) ea = eb = 0;
        __syncthreads();
        unsigned wa = s_a[lane], wb = s_b[lane], wc = s_c[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned x = __shfl_up_sync(0xffffffffu, wa, o), y = __shfl_up_sync(0xffffffffu, wb, o),
                           z = __shfl_up_sync(0xffffffffu, wc, o);
            if (lane >= o) {
                wa = max(wa, x);
                wb = max(wb, y);
                wc += z;
            }
        }
        const int from = warp ? warp - 1 : 0;
        const unsigned pa = __shfl_sync(0xffffffffu, wa, from), pb = __shfl_sync(0xffffffffu, wb, from),
                       pc = __shfl_sync(0xffffffffu, wc, from);
        if (in) {
            a[i] = max(ra, warp ? max(pa, ea) : ea);
            b[i] = max(rb, warp ? max(pb, eb) : eb);
            c[i] = rc + (warp ? pc : 0u) + vc - own;
        }
        ra = max(ra, __shfl_sync(0xffffffffu, wa, 31));
        rb = max(rb, __shfl_sync(0xffffffffu, wb, 31));
        rc += __shfl_sync(0xffffffffu, wc, 31);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        ta[blockIdx.x] = ra;
        tb[blockIdx.x] = rb;
        tc[blockIdx.x] = rc;
    }
}

// several groups: the sums that reach a group, added to its entries
__global__ void __launch_bounds__(1024) k_scan3_add(unsigned *a, unsigned *b, unsigned *c, int n,
                                                    const unsigned *__restrict__ ta, const unsigned *__restrict__ tb,
                                                    const unsigned *__restrict__ tc)
{
    after_previous();
    const unsigned pa = ta[blockIdx.x], pb = tb[blockIdx.x], pc = tc[blockIdx.x];
    const int lo = blockIdx.x * SCAN_GROUP, hi = min(n, lo + SCAN_GROUP);
    for (int i = lo + threadIdx.x; i < hi; i += 1024) {
        a[i] = max(a[i], pa);
        b[i] = max(b[i], pb);
        c[i] += pc;
    }
}

// What a thread of the passes over the order sees: each warp takes 32 * LINK_PER
// consecutive entries, 32 at a time; `run` and `chain` are the positions where the run
// and the chain of the entry before the warp's next 32 start, `number` the chains that
// start before them.
struct OrderWalk {
    unsigned e[LINK_PER];
    unsigned runs[LINK_PER], lows[LINK_PER];  // lanes where a run, a chain starts
    long long first;                          // the warp's first position
    unsigned run, chain, number;

    // GROUPS: blocks of the order per CTA, each by LINK_THREADS threads of it
    template <int GROUPS = 1>
    __device__ __forceinline__ void begin(const int *__restrict__ order, long long n, const unsigned *__restrict__ last_run,
                                          const unsigned *__restrict__ last_chain, const unsigned *__restrict__ chains)
    {
        constexpr int WARPS = LINK_THREADS / 32;
        __shared__ unsigned s_run[GROUPS * WARPS], s_chain[GROUPS * WARPS], s_num[GROUPS * WARPS];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp / WARPS;
        const long long block = blockIdx.x * (long long)GROUPS + group;
        first = block * LINK_BLOCK + (warp - group * WARPS) * (32 * LINK_PER);
        unsigned r = 0, c = 0, m = 0;
#pragma unroll
        for (int j = 0; j < LINK_PER; j++) {
            const long long i = first + j * 32 + lane;
            e[j] = i < n ? (unsigned)order[i] : 0u;
            runs[j] = __ballot_sync(0xffffffffu, (e[j] & (ORDER_ROOT | ORDER_START)) != 0u);
            lows[j] = __ballot_sync(0xffffffffu, (e[j] & ORDER_START) != 0u);
            if (runs[j]) r = (unsigned)first + j * 32 + 31 - __clz(runs[j]);
            if (lows[j]) c = (unsigned)first + j * 32 + 31 - __clz(lows[j]);
            m += __popc(lows[j]);
        }
        if (lane == 0) {
            s_run[warp] = r;
            s_chain[warp] = c;
            s_num[warp] = m;
        }
        __syncthreads();
        const bool in = GROUPS == 1 || block * LINK_BLOCK < n;
        run = in ? last_run[block] : 0u;
        chain = in ? last_chain[block] : 0u;
        number = in ? chains[block] : 0u;
        for (int w = group * WARPS; w < warp; w++) {
            run = max(run, s_run[w]);
            chain = max(chain, s_chain[w]);
            number += s_num[w];
        }
    }
    // for entry j of this lane: starts of its run and chain, of the run below it (equal
    // to its own unless it starts one), and the number of its chain
    __device__ __forceinline__ void at(int j, unsigned &own, unsigned &below, unsigned &low, int &num) const
    {
        const unsigned base = (unsigned)first + j * 32, lane = threadIdx.x & 31, le = 0xFFFFFFFFu >> (31 - lane);
        const unsigned m = runs[j] & le, b = runs[j] & (le >> 1), c = lows[j] & le;
        own = m ? base + 31 - __clz(m) : run;
        below = b ? base + 31 - __clz(b) : run;
        low = c ? base + 31 - __clz(c) : chain;
        num = (int)(number + __popc(c)) - 1;
    }
    __device__ __forceinline__ void next(int j)
    {
        const unsigned base = (unsigned)first + j * 32;
        if (runs[j]) run = base + 31 - __clz(runs[j]);
        if (lows[j]) chain = base + 31 - __clz(lows[j]);
        number += __popc(lows[j]);
    }
};

// The chains get their numbers and what they hang on; a pixel that chains hang on gets
// the first pixel of its run (in its parent entry, for k_chain_roots).  Three dependent loads
// an entry: those of a thread's eight entries are in flight together (1447 x 1083 f32 31 to 9
// us, 1024^2 u8 18 to 8).
template <int KB>
__global__ void __launch_bounds__(LINK_THREADS) k_chain_tables(const int *__restrict__ order, long long n,
                                                               const u64 *__restrict__ k0, const u64 *__restrict__ k1,
                                                               Comp *comp, const unsigned *__restrict__ ctr,
                                                               const unsigned *__restrict__ last_run,
                                                               const unsigned *__restrict__ last_chain,
                                                               const unsigned *__restrict__ chains, int *attach,
                                                               int *kids, int *bottom, int *parent)
{
    after_previous();
    const u64 *key = sort_passes(KB, ctr) & 1 ? k1 : k0;
    OrderWalk w;
    w.begin(order, n, last_run, last_chain, chains);
    const int lane = threadIdx.x & 31;
    // every load of the eight entries before the first store
    unsigned c[LINK_PER];
    u64 s[LINK_PER];
    int num[LINK_PER], run[LINK_PER];
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) c[j] = w.e[j] & ORDER_START ? (unsigned)(key[w.first + j * 32 + lane] >> KB) : 0u;
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) {
        unsigned own, below, low;
        w.at(j, own, below, low, num[j]);
        run[j] = w.e[j] & ORDER_HUNG ? order[own] & (int)ORDER_PIXEL : 0;
        w.next(j);
    }
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) s[j] = w.e[j] & ORDER_START ? comp[c[j]].best : 0ull;
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) {
        const unsigned e = w.e[j];
        if (e & ORDER_START) {
            comp[c[j]].hook = num[j];
            attach[num[j]] = s[j] ? weight_pixel(s[j]) : NONE;
            kids[num[j]] = 0;
            // its lowest pixel; negative when that is no level root
            bottom[num[j]] = e & ORDER_ROOT ? (int)(e & ORDER_PIXEL) : (int)~(e & ORDER_PIXEL);
        }
        if (e & ORDER_HUNG) parent[e & ORDER_PIXEL] = run[j];
    }
}

// Per chain: level root of its lowest run (node), and the parent entry of its lowest
// pixel.  Chains nest only as deep as there were rounds, so the loops are short.
__global__ void k_chain_roots(const unsigned *__restrict__ ctr, const int *__restrict__ attach,
                              const int *__restrict__ up, const int *__restrict__ bottom,
                              const int *__restrict__ parent, int *__restrict__ node, int *__restrict__ entry)
{
    after_previous();
    const unsigned n = ctr[FC_CHAINS];
    // level root of the node of the pixel that chain o hangs on
    auto above = [&](int o) {
        for (int step = 0; step < 64; step++) {
            const int s = attach[o], q = up[o];
            if (s == NONE || q == NONE) return NONE;
            const int h = parent[s], b = bottom[q];
            if (b >= 0 || h != (int)~b) return h;
            o = q;  // the lowest run of q, whose node goes on above
        }
        return NONE;
    };
    for (unsigned o = blockIdx.x * blockDim.x + threadIdx.x; o < n; o += gridDim.x * blockDim.x) {
        const int b = bottom[o], r = above((int)o);
        entry[o] = r;
        node[o] = b >= 0 ? b : r;
    }
}

// Canonical parents; a level root's entry is marked (parent_mark), so that the root flags
// can be written in pixel order instead of scattered like the parents.
__global__ void __launch_bounds__(LINK_THREADS) k_parents(const int *__restrict__ order, long long n,
                                                          const unsigned *__restrict__ last_run,
                                                          const unsigned *__restrict__ last_chain,
                                                          const unsigned *__restrict__ chains,
                                                          const int *__restrict__ node, const int *__restrict__ entry,
                                                          int *__restrict__ parent)
{
    after_previous();
    OrderWalk w;
    w.begin(order, n, last_run, last_chain, chains);
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) {
        const unsigned e = w.e[j];
        unsigned own, below, low;
        int num;
        w.at(j, own, below, low, num);
        if (w.first + j * 32 + lane < n) {
            const int q = e & ORDER_START ? entry[num] : below == low ? node[num] : order[below] & (int)ORDER_PIXEL;
            parent[e & ORDER_PIXEL] = e & ORDER_ROOT ? parent_mark(q) : q;
        }
        w.next(j);
    }
}

// The same for large images.  In the order of the sorted chains the entries' pixels lie all
// over the image, and once the parents no longer fit the L2 each is a partial write to
// memory of its own.  The entries go to buckets of neighbouring pixels first (k_parents_split:
// of known sizes, as every pixel occurs once; sorted within the block, so that a bucket's
// share is written in one piece), and from there to their places, a few buckets at a time
// (k_parents_fill).
constexpr int SPLIT_GROUPS = 2, SPLIT_THREADS = SPLIT_GROUPS * LINK_THREADS, SPLIT_BLOCK = SPLIT_GROUPS * LINK_BLOCK;
constexpr int SPLIT_BUCKETS = 512;
// Link kernels of noise images, k_parents against these two: 2896^2 u16 0.25 and 0.29 ms,
// 4096^2 0.51 and 0.59, 5800^2 1.45 and 1.25, 8192^2 3.6 and 2.7, 16384^2 18.0 and 13.2
// (smooth 16384^2 u16 7.1 and 4.6, the build's largest scatter).
constexpr long long SPLIT_FROM = 1LL << 25;

__global__ void __launch_bounds__(SPLIT_THREADS) k_parents_split(const int *__restrict__ order, long long n,
                                                                 const unsigned *__restrict__ last_run,
                                                                 const unsigned *__restrict__ last_chain,
                                                                 const unsigned *__restrict__ chains,
                                                                 const int *__restrict__ node, const int *__restrict__ entry,
                                                                 int shift, unsigned *filled, uint2 *__restrict__ pairs)
{
    after_previous();
    __shared__ uint2 s_pair[SPLIT_BLOCK];
    __shared__ unsigned s_count[SPLIT_BUCKETS], s_to[SPLIT_BUCKETS], s_warp[SPLIT_THREADS / 32];
    static_assert(SPLIT_BUCKETS == SPLIT_THREADS, "a thread per bucket");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    s_count[tid] = 0u;
    OrderWalk w;
    w.begin<SPLIT_GROUPS>(order, n, last_run, last_chain, chains);
    unsigned pixel[LINK_PER], value[LINK_PER], rank[LINK_PER];
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) {
        const unsigned e = w.e[j];
        unsigned own, below, low;
        int num;
        w.at(j, own, below, low, num);
        pixel[j] = ~0u;
        if (w.first + j * 32 + lane < n) {
            const int q = e & ORDER_START ? entry[num] : below == low ? node[num] : order[below] & (int)ORDER_PIXEL;
            pixel[j] = e & ORDER_PIXEL;
            value[j] = (unsigned)(e & ORDER_ROOT ? parent_mark(q) : q);
        }
        w.next(j);
    }
#pragma unroll
    for (int j = 0; j < LINK_PER; j++)
        if (pixel[j] != ~0u) rank[j] = atomicAdd(s_count + (pixel[j] >> shift), 1u);
    __syncthreads();
    const unsigned mine = s_count[tid];
    unsigned inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    const unsigned at = mine ? ((unsigned)tid << shift) + atomicAdd(filled + tid, mine) : 0u;
    __syncthreads();
    unsigned start = inc - mine;
    for (int v = 0; v < warp; v++) start += s_warp[v];
    s_count[tid] = start;
    s_to[tid] = at - start;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < LINK_PER; j++)
        if (pixel[j] != ~0u) s_pair[s_count[pixel[j] >> shift] + rank[j]] = make_uint2(pixel[j], value[j]);
    __syncthreads();
    const int here = (int)min((long long)SPLIT_BLOCK, n - blockIdx.x * (long long)SPLIT_BLOCK);
#pragma unroll
    for (int j = 0; j < LINK_PER; j++) {
        const int i = tid + j * SPLIT_THREADS;
        if (i >= here) continue;
        const uint2 p = s_pair[i];
        const unsigned to = s_to[p.x >> shift] + (unsigned)i;
        if (to < n) pairs[to] = p;
    }
}

__global__ void __launch_bounds__(256) k_parents_fill(const uint2 *__restrict__ pairs, long long n, int *__restrict__ parent)
{
    after_previous();
    const long long first = blockIdx.x * 1024LL + threadIdx.x;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (first + j * 256 < n) {
            const uint2 p = pairs[first + j * 256];
            if (p.x < n) parent[p.x] = (int)p.y;  // anything else only after a wait that gave up
        }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t up256(size_t b) { return (b + 255) / 256 * 256; }

long long forest_edge_cap(int conn, long long n)
{
    // 2-D: the groups beyond the first around all pixels number at most peaks + pits.
    // 3-D has no such bound; a build that needs more falls back to the merging build.
    return conn == 4 || conn == 8 ? n + 64 : 2 * n + 64;
}

static long long rs_blocks(long long n) { return (n + RS_BLOCK - 1) / RS_BLOCK; }

static long long scan_groups(long long n) { return (chain_blocks(n) + SCAN_GROUP - 1) / SCAN_GROUP; }

ForestWork forest_carve(void *mem, int conn, long long n, long long basin_cap, size_t *bytes)
{
    ForestWork w;
    char *m = (char *)mem;
    auto take = [&](size_t b) { char *p = m; m += up256(b); return p; };
    // zeroed at the start of a build, in one piece: counters, digit totals, the published
    // counts of the node list and of the first sort pass
    w.ctr = (unsigned *)take(FC_COUNT * 4);
    w.totals = (unsigned *)take(4 * 256 * SORT_PASSES);
    w.filled = (unsigned *)take(4 * SPLIT_BUCKETS);
    w.nodes_state = (unsigned *)take(marked_nodes_bytes(n));
    for (int k = 0; k < 2; k++) {
        w.state[k] = (unsigned *)take(4 * 256 * (size_t)rs_blocks(n));
        if (k == 0) w.zero_bytes = (size_t)(m - (char *)mem);
    }
    w.label = (int *)take(4 * (size_t)n);
    w.comp = (Comp *)take(sizeof(Comp) * 2 * (size_t)basin_cap);
    w.last_run = (unsigned *)take(4 * (size_t)chain_blocks(n));
    w.last_chain = (unsigned *)take(4 * (size_t)chain_blocks(n));
    w.group = (unsigned *)take(4 * 3 * (size_t)scan_groups(n));
    const size_t chain_cap = (size_t)forest_chain_cap(n, basin_cap);
    w.attach = (int *)take(4 * chain_cap);
    w.up = (int *)take(4 * chain_cap);
    w.kids = (int *)take(4 * chain_cap);
    w.bottom = (int *)take(4 * chain_cap);
    w.node = (int *)take(4 * chain_cap);
    w.entry = (int *)take(4 * chain_cap);
    // the edges and the sort are never alive together
    char *shared = m;
    const long long ecap = forest_edge_cap(conn, n);
    for (int k = 0; k < 2; k++) w.ew[k] = (u64 *)take(8 * (size_t)ecap);
    for (int k = 0; k < 2; k++) w.eab[k] = (int2 *)take(8 * (size_t)ecap);
    char *end = m;
    m = shared;
    for (int k = 0; k < 2; k++) w.skey[k] = (u64 *)take(8 * (size_t)n);
    for (int k = 0; k < 2; k++) w.sidx[k] = (int *)take(4 * (size_t)n);
    if (m > end) end = m;
    w.ecap = ecap;
    if (bytes) *bytes = (size_t)(end - (char *)mem);
    return w;
}

cudaError_t basin_opt_in()
{
    const cudaError_t e = cudaFuncSetAttribute(k_saddles_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TAIL_SMEM);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_rs_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RS_SMEM);
}

template <int KB>
static void after_basins(const ForestWork &w, const ChainOrder &c, const float *gval, long long n, long long comp_cap, long long max_rounds,
                         int *parent, unsigned *err, int sm, cudaStream_t s)
{
    prof_begin(P_SADDLES, s);
    launch_next(k_basin_ids, grid_for(n, 256, sm), 256, 0, s, w.label, n, err);
    {
        // Every block more is one more arrival at each of four barriers a round, so a block
        // has 32 pixels a thread and an SM one block: 1447 x 1083 f32 57 us, 1531 x 997 u8 26,
        // 8190 x 8211 u16 115, against 65, 28 and 122 with 16 pixels and two blocks (64 pixels:
        // 62 us at the first, 128: 83).
        const long long want = n / (SADDLE_THREADS * 32) + 1;
        const int nb = (int)(want < sm ? want : sm);
        int *label = w.label;
        u64 *ew0 = w.ew[0], *ew1 = w.ew[1];
        int2 *ab0 = w.eab[0], *ab1 = w.eab[1];
        Comp *comp = w.comp;
        unsigned *ctr = w.ctr;
        unsigned ecap = (unsigned)w.ecap;
        void *args[] = {&label, &n, &ew0, &ab0, &ew1, &ab1, &comp, &ctr, &ecap, &max_rounds, &err};
        // Images whose edges and basins fit the tail's shared memory whatever they hold (2-D:
        // up to 8128 pixels) go there directly: a cooperative launch and its barriers less, about
        // 10 us of the 129 that a call on 96 x 80 u8 took.
        const bool raw = ecap <= TAIL_EDGES && 2 * TAIL_COMPS >= (unsigned long long)comp_cap;
        if (!raw && may_launch())
            note_launch(cudaLaunchCooperativeKernel((const void *)k_saddles, dim3(nb), dim3(SADDLE_THREADS), args, 0, s));
        launch_next(k_saddles_tail, 1, TAIL_THREADS, TAIL_SMEM, s, label, ew0, ab0, ew1, ab1, comp, ctr,
                    raw ? ecap : 0u, max_rounds, err);
    }
    {
        const long long want = n / (CHAIN_THREADS * CHAIN_PER) + 1, cap = sm;  // one histogram flush per block
        launch_next(k_chain<KB>, (int)(want < cap ? want : cap), CHAIN_THREADS, 0, s, w.label, gval, n, w.comp, w.ctr,
                    w.skey[0], w.totals);
    }
    const int cb_blocks = grid_for(comp_cap, 256, sm);
    prof_end(P_SADDLES, s);
    prof_begin(P_SORT, s);
    int cb = 0;
    while ((1LL << cb) < comp_cap) cb++;
    const int passes = (KB + cb + 7) / 8, nblk = (int)rs_blocks(n);
    for (int pass = 0; pass < passes; pass++) {
        const u64 *kin = w.skey[pass & 1];
        const int *iin = pass ? w.sidx[pass & 1] : nullptr;
        launch_next(k_rs_scatter, nblk, RS_THREADS, RS_SMEM, s, kin, iin, w.label, w.skey[(pass + 1) & 1],
                    w.sidx[(pass + 1) & 1], n, pass, KB, w.ctr, w.state[pass & 1], w.state[(pass + 1) & 1],
                    w.totals + 256 * pass, err);
    }
    prof_end(P_SORT, s);
    prof_begin(P_LINK, s);
    const int lb = (int)chain_blocks(n), groups = (int)scan_groups(n);
    unsigned *ga = w.group, *gb = ga + groups, *gc = gb + groups, *total = w.ctr + FC_CHAINS, *none = w.ctr + FC_SPARE;
    launch_next(k_order<KB>, lb, LINK_THREADS, 0, s, w.skey[0], w.skey[1], w.sidx[0], w.sidx[1], n, w.comp, w.ctr,
                c.order, w.last_run, w.last_chain, c.first);
    if (groups == 1) {
        launch_next(k_scan3, 1, 1024, 0, s, w.last_run, w.last_chain, c.first, lb, none, none, total);
    } else {
        launch_next(k_scan3, groups, 1024, 0, s, w.last_run, w.last_chain, c.first, lb, ga, gb, gc);
        launch_next(k_scan3, 1, 1024, 0, s, ga, gb, gc, groups, none, none, total);
        launch_next(k_scan3_add, groups, 1024, 0, s, w.last_run, w.last_chain, c.first, lb, ga, gb, gc);
    }
    launch_next(k_chain_tables<KB>, lb, LINK_THREADS, 0, s, c.order, n, w.skey[0], w.skey[1], w.comp, w.ctr,
                w.last_run, w.last_chain, c.first, w.attach, w.kids, w.bottom, parent);
    launch_next(k_chain_up, cb_blocks, 256, 0, s, w.attach, w.label, gval, w.comp, w.ctr, w.up, w.kids, c.nchains);
    launch_next(k_chain_roots, cb_blocks, 256, 0, s, w.ctr, w.attach, w.up, w.bottom, parent, w.node, w.entry);
    if (n >= SPLIT_FROM) {
        int shift = 16;
        while (((n - 1) >> shift) >= SPLIT_BUCKETS) shift++;
        uint2 *pairs = (uint2 *)w.skey[0];  // nothing reads the keys any more
        launch_next(k_parents_split, (unsigned)((n + SPLIT_BLOCK - 1) / SPLIT_BLOCK), SPLIT_THREADS, 0, s, c.order, n,
                    w.last_run, w.last_chain, c.first, w.node, w.entry, shift, w.filled, pairs);
        launch_next(k_parents_fill, (unsigned)((n + 1023) / 1024), 256, 0, s, pairs, n, parent);
    } else {
        launch_next(k_parents, lb, LINK_THREADS, 0, s, c.order, n, w.last_run, w.last_chain, c.first, w.node, w.entry,
                    parent);
    }
    prof_end(P_LINK, s);
}

template <typename T, bool MIN, int CONN, bool BATCH>
static void basins(const ForestArgs &a, cudaStream_t s)
{
    using BT = BasinTile<CONN>;
    auto tiles = [](int side, int tile) { return (unsigned)((side + tile - 1) / tile); };
    const unsigned rows = tiles(a.g.H, BT::Y) * tiles(a.g.D, BT::Z), ny = rows < 65535u ? rows : 65535u;
    const dim3 grid = BATCH ? dim3(a.ntiles) : dim3(tiles(a.g.W, BT::X), ny, (rows + ny - 1) / ny);
    launch_next(k_basins<T, MIN, CONN, BATCH>, grid, BASIN_THREADS, 0, s, (const T *)a.img, a.g, a.imgs, a.tiles,
                a.kmax, a.gval, a.w.label, a.w.ew[0], a.w.eab[0], a.w.ctr, (unsigned)a.w.ecap, a.err);
}

template <typename T, bool MIN>
static void forest_t(const ForestArgs &a, cudaStream_t s)
{
    prof_begin(P_BASINS, s);
    if constexpr (!MIN) {
        if (a.tiles) {
            if (a.g.conn == 4) basins<T, false, 4, true>(a, s);
            else basins<T, false, 8, true>(a, s);
        }
    }
    if (!a.tiles) {
        switch (a.g.conn) {
        case 4: basins<T, MIN, 4, false>(a, s); break;
        case 8: basins<T, MIN, 8, false>(a, s); break;
        case 6: basins<T, MIN, 6, false>(a, s); break;
        default: basins<T, MIN, 26, false>(a, s); break;
        }
    }
    prof_end(P_BASINS, s);
    if (a.input_read) cudaEventRecord(a.input_read, s);
    ChainOrder c = a.c;
    c.n = a.g.N;
    c.attach = a.w.attach;
    c.up = a.w.up;
    c.kids = a.w.kids;
    after_basins<KeyBits<T>::bits>(a.w, c, a.gval, a.g.N, 2 * a.basin_cap, a.g.merge_bound > 0 ? a.g.merge_bound : 64,
                                   a.parent, a.err, a.sm_count, s);
}

void launch_forest(const ForestArgs &a, cudaStream_t s)
{
    switch (a.dtype * 2 + (a.tree_min ? 1 : 0)) {
    case 0: forest_t<uint8_t, false>(a, s); break;
    case 1: forest_t<uint8_t, true>(a, s); break;
    case 2: forest_t<uint16_t, false>(a, s); break;
    case 3: forest_t<uint16_t, true>(a, s); break;
    case 4: forest_t<uint32_t, false>(a, s); break;
    case 5: forest_t<uint32_t, true>(a, s); break;
    case 6: forest_t<float, false>(a, s); break;
    default: forest_t<float, true>(a, s); break;
    }
}

}  // namespace dcf
