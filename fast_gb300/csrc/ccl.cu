// 6-connected component labelling of a uint8 volume on the GPU, numbered as
// the reference numbers them (fastlib/src/cuda/VolumeCCL.cu:381-620
// VolumeCCL_Label, :753-818 VolumeCCL_BoundaryLabels;
// fastlib/src/volume/VolumeSegmentation.cpp:14-64):
//
//   * foreground = voxels whose value differs from `background`;
//   * label 0 = background; components are numbered 1..K in increasing order
//     of their smallest linear index (x fastest); num_labels = K + 1;
//   * boundary[d * num_labels + l] = 1 when label l > 0 has a voxel on face d
//     (Dir order: X_POS is x = nx-1, X_NEG is x = 0, ...); row 6 is the AND of
//     rows 0..5.
//
// The reference gets that numbering from span labels merged by atomicMin and a
// scan over root spans.  Here it comes from a union-find over x-runs whose
// links always point from a larger to a smaller linear index, so the root of
// every tree is its component's minimum index; roots are then ranked by a
// two-level scan in linear-index order.  Passes:
//   1. bricks: one block per 64 x 8 x 8 brick holds its rows as 64-bit words
//      and joins their runs in shared memory.  A run's node is named by its
//      row and start in the brick, which order as linear indices do, so the
//      local root is the run with the smallest index.  Kept in global memory:
//      the words, every run's local root (16 bits, at slot start / 2 of its
//      row: runs start at least two voxels apart) and which runs are local
//      roots;
//   2. merge: the joins across brick faces, between local roots; Rem's union
//      with splicing, lock-free (compare-and-swap), on parents kept at the
//      local roots' places of the label array;
//   3. flatten: every local root that is a global root counts itself in its
//      chunk of voxels and sets its bit of a root bitmap, every other one is
//      pointed straight at its root;
//   4. scan the chunk counts;
//   5. rank: one block per chunk numbers the chunk's roots from the bitmap;
//   6. relabel: a brick fetches the labels of its local roots, then writes
//      every voxel's (0 on the background);
//   7. face bitmaps, 8. the all-faces AND.
// Every loop terminates: a find follows strictly decreasing indices, and a
// failed link continues from a strictly smaller index.
//
// Joining voxels in global memory was bound by dependent loads: most joins
// are inside a brick, where shared memory answers in a few dozen cycles, and
// about one in five is left for pass 2.  768 x 700 x 720 spheres: 5.92 ms of
// kernels -> 1.30 (pass 1 0.57, issue bound; pass 2 0.25; pass 6 0.37, 4.2 TB/s
// of labels); 1024^3 17.3 -> 3.7 ms.  Scratch is 76 bytes per 64-voxel word of
// a row plus a bit per voxel: 1.3 bytes per voxel at multiples of 64, at most
// 2.5 above 64 (a parent per voxel: 4.1).  A row of less than 64 voxels keeps
// 12 + 2 ceil(nx / 2) bytes: 1.3 per voxel at 63, 2.0 at 14, 5.5 and 7.1 at 3
// and 2.  A volume one voxel wide is labelled as its y-z plane (the same
// indices and neighbours): 1 x 6000 x 5000 takes 1.1 ms instead of 4.3, and 1.3
// bytes per voxel instead of 14.  30 M voxels 2, 3, 8 and 33 wide: 2.1, 1.6,
// 0.93 and 0.45 ms (5.8, 4.6, 3.0 and 1.5 with a parent per voxel).
#include <cuda_runtime.h>
#include <stdint.h>

#include "ccl_faces.h"
#include "fasttau.h"
#include "tau_errors.h"

namespace ft {
namespace {

constexpr int kChunk = 32768;      // voxels per block in the ranking pass
constexpr int kRankThreads = 256;  // each takes kRankWords root-bitmap words (32 voxels)
constexpr int kRankWords = 4;
static_assert(kChunk == kRankThreads * kRankWords * 32, "a rank block covers one chunk");

// Bricks: 64 voxels (one word) x RY x RZ rows.
constexpr int RY = 8, RZ = 8, ROWS = RY * RZ;
constexpr int kSlots = 32;          // runs of a word at most: slot = start / 2
constexpr int kBrickThreads = 128;
static_assert(RY == 8 && RZ == 8, "three join steps in y and in z");

// Geometry of a labelling and its scratch arrays.
struct Ccl {
    int nx, ny, nz;
    int wx, by, bz;    // words per row, bricks in y and z
    int slots;         // slots kept per word
    uint8_t bg;
    const uint8_t *mask;
    uint64_t *bits;    // [z][y][word]: foreground
    uint16_t *local;   // [z][y][word][slot]: local root, row * 64 + start
    uint32_t *roots;   // [z][y][word]: slots that are local roots
    uint32_t *par;     // the label array: parents at the local roots' places
    uint32_t *cnt, *root_bits;
    int64_t zero_words;  // cnt and root_bits, from cnt on: zeroed by pass 1

    __device__ int64_t word(int y, int z, int w) const { return ((int64_t)z * ny + y) * wx + w; }
    __device__ uint32_t voxel(int x, int y, int z) const
    {
        return (uint32_t)x + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
    }
};

// First bits of the word's runs.
__device__ __forceinline__ uint64_t run_starts(uint64_t w) { return w & ~(w << 1); }

// Start of the run that holds bit b of half h (0: bits 0..31) of a word.
__device__ __forceinline__ int run_start(uint64_t starts, int h, int b)
{
    const uint32_t lo = (uint32_t)starts, hi = (uint32_t)(starts >> 32);
    const uint32_t upto = 0xFFFFFFFFu >> (31 - b);
    const uint32_t m = (h ? hi : lo) & upto;
    return m ? 32 * h + 31 - __clz((int)m) : 31 - __clz((int)lo);
}

// Start bit of the run in a slot.
__device__ __forceinline__ int slot_start(uint64_t starts, int slot)
{
    return 2 * slot + (int)((starts >> (2 * slot + 1)) & 1);
}

// Parent reads during the merge and flatten passes go through L1
// (ld.global.ca): a read may return a stale parent written earlier in the
// same pass by another SM, which is harmless.  Every value ever stored is a
// pointer to a smaller index of the same component, so a walk that follows
// stale pointers still ends at a root.  A stale "root" is caught by the
// linking compare-and-swap, whose old value the union continues from.  The next
// pass, after the kernel boundary, sees the final values.  The root of a
// large component is read by most finds; through L2 alone that one line
// would serialise them.
__device__ __forceinline__ uint32_t ld_par(const uint32_t *p, uint32_t i) { return __ldca(p + i); }

// Root of a's tree (no writes).
__device__ __forceinline__ uint32_t find_root(const uint32_t *par, uint32_t a)
{
    uint32_t p = ld_par(par, a);
    while (p != a) {
        a = p;
        p = ld_par(par, a);
    }
    return a;
}

// Joins the trees of x and y: Rem's union with splicing, concurrent form
// (links by compare-and-swap).  The node whose parent is larger moves up;
// before it does, its parent is swung to the other node's (smaller) parent,
// so paths shorten as unions proceed; the walk stops as soon as both nodes
// have the same parent, which for two voxels already in one component
// usually happens well below the root.  Invariants: a parent never exceeds
// its node (so a root is its tree's smallest index) and every stored parent
// is a local root, which the flatten and relabel passes rely on.  A link or splice that loses a race
// only fails its compare-and-swap; a failed link hands back the node's
// current parent, so a stale read cannot make the loop spin, and every
// step moves a node to a strictly smaller index.
__device__ void unite(uint32_t *par, uint32_t x, uint32_t y)
{
    uint32_t px = ld_par(par, x), py = ld_par(par, y);
    for (;;) {
        if (px == py) return;
        if (px < py) {
            uint32_t t = x;
            x = y;
            y = t;
            t = px;
            px = py;
            py = t;
        }
        // px > py
        if (x == px) {  // x is a root: hang it under y's parent
            const uint32_t old = atomicCAS(par + x, x, py);
            if (old == x) return;
            px = old;  // x got a parent meanwhile
            continue;
        }
        atomicCAS(par + x, px, py);  // splice; losing the race is harmless
        x = px;
        px = ld_par(par, x);
    }
}

// Place of a node in the brick's shared array: row and slot, the slot XORed
// with the row.  Threads take a row each, and where the rows look alike (plates
// across x) they go to the same slot at once, which without it is one bank for
// all of them: alternating planes across x, 384^3, 1.10 -> 0.44 ms in pass 1.
__device__ __forceinline__ uint32_t node_at(uint32_t v) { return v >> 1 ^ (v >> 6 & 31u); }

// Root of a run of the brick; every second node on the way is pointed at its
// grandparent (a plain store: it may undo a concurrent shortening, never a
// link, since only roots are linked).
__device__ __forceinline__ uint32_t find_local(volatile uint32_t *par, uint32_t u)
{
    uint32_t p = par[node_at(u)];
    while (p != u) {
        const uint32_t g = par[node_at(p)];
        if (g != p) par[node_at(u)] = g;
        u = p;
        p = g;
    }
    return u;
}

// Joins two runs of the brick: the larger root is hung under the smaller; a
// root that got a parent meanwhile is followed up.
__device__ __forceinline__ void join_local(uint32_t *par, uint32_t u, uint32_t v)
{
    for (;;) {
        u = find_local(par, u);
        v = find_local(par, v);
        if (u == v) return;
        if (u < v) {
            const uint32_t t = u;
            u = v;
            v = t;
        }
        const uint32_t old = atomicCAS(par + node_at(u), u, v);
        if (old == u) return;
        u = old;
    }
}

// Pass 1: one brick per block.
__global__ void __launch_bounds__(kBrickThreads) ccl_bricks(Ccl A)
{
    __shared__ uint64_t s_bits[ROWS];
    __shared__ uint32_t s_par[ROWS * kSlots];  // parents, at node_at
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t b = blockIdx.x;
    const int w = (int)(b % A.wx);
    const int y0 = (int)(b / A.wx % A.by) * RY, z0 = (int)(b / A.wx / A.by) * RZ;
    const int x0 = w * 64;

    for (int64_t k = b * kBrickThreads + tid; k < A.zero_words; k += (int64_t)gridDim.x * kBrickThreads) A.cnt[k] = 0u;

    // A warp takes consecutive rows; all its loads are in flight together.
    constexpr int PER = ROWS / (kBrickThreads / 32), U = 8;
    const bool in0 = x0 + lane < A.nx, in1 = x0 + 32 + lane < A.nx;
#pragma unroll
    for (int k0 = 0; k0 < PER; k0 += U) {
        uint8_t m[U][2];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = warp * PER + k0 + u;
            const int y = y0 + r % RY, z = z0 + r / RY;
            const uint8_t *row = A.mask + ((int64_t)z * A.ny + y) * A.nx + x0 + lane;
            const bool in = y < A.ny && z < A.nz;
            m[u][0] = in && in0 ? __ldg(row) : A.bg;
            m[u][1] = in && in1 ? __ldg(row + 32) : A.bg;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t lo = __ballot_sync(0xFFFFFFFFu, m[u][0] != A.bg);
            const uint32_t hi = __ballot_sync(0xFFFFFFFFu, m[u][1] != A.bg);
            if (lane == 0) s_bits[warp * PER + k0 + u] = (uint64_t)hi << 32 | lo;
        }
    }
    __syncthreads();
    if (tid < ROWS) {
        for (uint64_t o = run_starts(s_bits[tid]); o; o &= o - 1) {
            const uint32_t v = (uint32_t)(tid * 64 + __ffsll((long long)o) - 1);
            s_par[node_at(v)] = v;
        }
    }
    __syncthreads();

    // Joins of neighbouring rows, one per stretch of voxels that both have, in
    // six steps: rows 1, 3, 5, 7 of every plane with the row before, then 2
    // and 6, then 4, then the planes likewise.  A step joins pairs of groups
    // that nothing else touches, so trees stay shallow and links rarely race.
    // A thread takes a quarter of a word, so the later steps leave whole warps
    // out: most words hold one or two stretches.  (All rows at once, a thread per
    // row, made chains as long as the brick and retried links: 35 us for one
    // brick; as many pieces of a row as there are threads, 14,800 instructions
    // per brick.)
#pragma unroll 1
    for (int step = 0; step < 6; step++) {
        const int lvl = step % 3;         // lowest set bit of the row (plane) number
        const int n = ROWS >> (lvl + 1);  // rows in this step
        if (tid < 4 * n) {
            const int q = tid % n, piece = tid / n, h = piece >> 1;
            int r, to;
            if (step < 3) {
                const int per = RY >> (lvl + 1);
                r = q / per * RY + ((2 * (q % per) + 1) << lvl);
                to = r - 1;
            } else {
                r = ((2 * (q / RY) + 1) << lvl) * RY + q % RY;
                to = r - RY;
            }
            const uint64_t a = s_bits[r], c = s_bits[to];
            const uint64_t both = run_starts(a & c), sa = run_starts(a), sc = run_starts(c);
            const uint32_t half = (uint32_t)(h ? both >> 32 : both) & (piece & 1 ? 0xFFFF0000u : 0x0000FFFFu);
            for (uint32_t o = half; o; o &= o - 1) {
                const int bit = __ffs((int)o) - 1;
                join_local(s_par, (uint32_t)(r * 64 + run_start(sa, h, bit)),
                           (uint32_t)(to * 64 + run_start(sc, h, bit)));
            }
        }
        __syncthreads();
    }

    if (tid < ROWS) {
        const int y = y0 + tid % RY, z = z0 + tid / RY;
        if (y < A.ny && z < A.nz) {
            const int64_t at = A.word(y, z, w);
            const uint64_t bits = s_bits[tid];
            uint32_t roots = 0;
            for (uint64_t o = run_starts(bits); o; o &= o - 1) {
                const int start = __ffsll((long long)o) - 1;
                const uint32_t u = (uint32_t)(tid * 64 + start);
                uint32_t v = u, p;
                while ((p = s_par[node_at(v)]) != v) v = p;
                A.local[at * A.slots + (start >> 1)] = (uint16_t)v;
                if (u == v) {
                    roots |= 1u << (start >> 1);
                    const uint32_t i = A.voxel(x0 + start, y, z);
                    A.par[i] = i;
                }
            }
            A.bits[at] = bits;
            A.roots[at] = roots;
        }
    }
}

// Linear index of the local root of the run that starts at bit `start` of a word.
__device__ __forceinline__ uint32_t local_root(const Ccl &A, int y, int z, int w, int start)
{
    const uint32_t v = A.local[A.word(y, z, w) * A.slots + (start >> 1)];
    const int r = (int)(v >> 6);
    return A.voxel(w * 64 + (int)(v & 63u), y / RY * RY + r % RY, z / RZ * RZ + r / RY);
}

// Pass 2: joins across brick faces.  Tasks: every word with a word to its
// left, every quarter word of the rows that begin a brick in y, and in z.
__global__ void __launch_bounds__(256) ccl_merge(Ccl A, int64_t tasks_x, int64_t tasks_y, int64_t tasks_z)
{
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < tasks_x) {
        const int w = 1 + (int)(t % (A.wx - 1));
        t /= A.wx - 1;
        const int y = (int)(t % A.ny), z = (int)(t / A.ny);
        const uint64_t a = A.bits[A.word(y, z, w)], c = A.bits[A.word(y, z, w - 1)];
        if ((a & 1) && (c >> 63))
            unite(A.par, local_root(A, y, z, w, 0), local_root(A, y, z, w - 1, run_start(run_starts(c), 1, 31)));
        return;
    }
    t -= tasks_x;
    int w, y, z, ty, tz;
    const int piece = (int)(t & 3), h = piece >> 1;
    t >>= 2;
    if (t < tasks_y) {
        w = (int)(t % A.wx);
        t /= A.wx;
        y = RY * (1 + (int)(t % (A.by - 1)));
        z = (int)(t / (A.by - 1));
        ty = y - 1;
        tz = z;
    } else {
        t -= tasks_y;
        if (t >= tasks_z) return;
        w = (int)(t % A.wx);
        t /= A.wx;
        y = (int)(t % A.ny);
        z = RZ * (1 + (int)(t / A.ny));
        ty = y;
        tz = z - 1;
    }
    const uint64_t a = A.bits[A.word(y, z, w)], c = A.bits[A.word(ty, tz, w)];
    const uint64_t sa = run_starts(a), sc = run_starts(c);
    uint32_t u0 = 0, v0 = 0;
    bool any = false;
    const uint64_t both = run_starts(a & c);
    const uint32_t mine = (uint32_t)(h ? both >> 32 : both) & (piece & 1 ? 0xFFFF0000u : 0x0000FFFFu);
    for (uint32_t o = mine; o; o &= o - 1) {
        const int bit = __ffs((int)o) - 1;
        const uint32_t u = local_root(A, y, z, w, run_start(sa, h, bit));
        const uint32_t v = local_root(A, ty, tz, w, run_start(sc, h, bit));
        if (any && u == u0 && v == v0) continue;  // the pair just joined
        unite(A.par, u, v);
        u0 = u;
        v0 = v;
        any = true;
    }
}

// Pass 3: local roots.  A global root (its own parent) counts itself in its
// chunk and sets its bit in the root bitmap; another gets its root as parent.
__global__ void __launch_bounds__(256) ccl_flatten(Ccl A, int64_t words)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= words) return;
    uint32_t m = A.roots[t];
    if (!m) return;
    const uint64_t starts = run_starts(A.bits[t]);
    const uint32_t row = (uint32_t)(t / A.wx) * (uint32_t)A.nx + (uint32_t)(t % A.wx) * 64u;
    for (; m; m &= m - 1) {
        const uint32_t i = row + (uint32_t)slot_start(starts, __ffs((int)m) - 1);
        const uint32_t p = ld_par(A.par, i);
        if (p == i) {
            atomicAdd(A.cnt + i / (uint32_t)kChunk, 1u);
            atomicOr(A.root_bits + (i >> 5), 1u << (i & 31u));
        } else {
            const uint32_t r = find_root(A.par, p);
            if (r != p) A.par[i] = r;
        }
    }
}

// Exclusive block scan of one value per thread (kRankThreads threads).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *s_warp, uint32_t &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t s = lane < kRankThreads / 32 ? s_warp[lane] : 0u;
        uint32_t si = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, si, o);
            if (lane >= o) si += t;
        }
        if (lane < kRankThreads / 32) s_warp[lane] = si - s;  // exclusive warp offsets
        if (lane == kRankThreads / 32 - 1) s_warp[kRankThreads / 32] = si;
    }
    __syncthreads();
    total = s_warp[kRankThreads / 32];
    return s_warp[w] + inc - v;
}

// Pass 4: exclusive scan of the chunk counts in place (one block of 1024
// threads, each summing a contiguous slice); cnt[nchunks] = number of roots.
__global__ void __launch_bounds__(1024) ccl_scan_chunks(uint32_t *cnt, uint32_t nchunks)
{
    __shared__ uint32_t s[1024];
    const uint32_t per = (nchunks + 1023u) / 1024u;
    const uint32_t a = threadIdx.x * per, b = min(a + per, nchunks);
    uint32_t sum = 0;
    for (uint32_t k = a; k < b; k++) sum += cnt[k];
    s[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {  // Hillis-Steele inclusive scan
        const uint32_t t = threadIdx.x >= (unsigned)o ? s[threadIdx.x - o] : 0u;
        __syncthreads();
        s[threadIdx.x] += t;
        __syncthreads();
    }
    uint32_t run = s[threadIdx.x] - sum;
    for (uint32_t k = a; k < b; k++) {
        const uint32_t c = cnt[k];
        cnt[k] = run;
        run += c;
    }
    if (threadIdx.x == 1023) cnt[nchunks] = s[1023];
}

// Pass 5: label of every root = 1 + its rank.  One block per chunk,
// kRankWords neighbouring bitmap words per thread.
__global__ void __launch_bounds__(kRankThreads) ccl_rank(const uint32_t *__restrict__ root_bits,
                                                         const uint32_t *__restrict__ chunk_off, uint32_t *labels)
{
    __shared__ uint32_t s_warp[kRankThreads / 32 + 1];
    const uint32_t w = (blockIdx.x * (uint32_t)kRankThreads + threadIdx.x) * kRankWords;
    uint32_t bits[kRankWords], mine = 0;
#pragma unroll
    for (int k = 0; k < kRankWords; k++) {
        bits[k] = root_bits[w + k];
        mine += (uint32_t)__popc(bits[k]);
    }
    uint32_t total;
    uint32_t r = chunk_off[blockIdx.x] + block_exclusive_scan(mine, s_warp, total) + 1u;
#pragma unroll
    for (int k = 0; k < kRankWords; k++) {
        while (bits[k]) {
            labels[(w + k) * 32u + (uint32_t)(__ffs((int)bits[k]) - 1)] = r++;
            bits[k] &= bits[k] - 1u;
        }
    }
}

// Pass 6: labels, in place of the parents.  A local root's place holds its
// label if it is a global root (pass 5), else its root's index.  A block
// reads its own local roots before it writes, and other blocks read only the
// places of global roots, where a block writes the label that is already
// there.  Reads go through L1: one component can own most of the volume, and
// every brick fetches its root's label.
__global__ void __launch_bounds__(kBrickThreads) ccl_relabel(Ccl A)
{
    __shared__ uint64_t s_bits[ROWS];
    __shared__ uint32_t s_label[ROWS * kSlots];  // of the local roots, then of every run, at node_at
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t b = blockIdx.x;
    const int w = (int)(b % A.wx);
    const int y0 = (int)(b / A.wx % A.by) * RY, z0 = (int)(b / A.wx / A.by) * RZ;
    const int x0 = w * 64;
    const int ry = tid % RY, rz = tid / RY;
    const bool mine = tid < ROWS && y0 + ry < A.ny && z0 + rz < A.nz;  // a row per thread
    int64_t at = 0;
    uint64_t starts = 0;
    if (mine) {
        at = A.word(y0 + ry, z0 + rz, w);
        const uint64_t bits = __ldg(A.bits + at);
        s_bits[tid] = bits;
        starts = run_starts(bits);
        for (uint32_t m = __ldg(A.roots + at); m; m &= m - 1) {
            const int slot = __ffs((int)m) - 1;
            const uint32_t i = A.voxel(x0 + slot_start(starts, slot), y0 + ry, z0 + rz);
            const bool root = (__ldg(A.root_bits + (i >> 5)) >> (i & 31u)) & 1u;
            uint32_t v = ld_par(A.par, i);
            if (!root) v = ld_par(A.par, v);
            s_label[tid * kSlots + (slot ^ (tid & 31))] = v;
        }
    }
    __syncthreads();
    // A run that is no local root takes its root's label (roots' entries are
    // not written here).
    for (uint64_t o = starts; o; o &= o - 1) {
        const int start = __ffsll((long long)o) - 1;
        const uint32_t v = __ldg(A.local + at * A.slots + (start >> 1));
        if (v != (uint32_t)(tid * 64 + start)) s_label[node_at((uint32_t)(tid * 64 + start))] = s_label[node_at(v)];
    }
    __syncthreads();
    constexpr int PER = ROWS / (kBrickThreads / 32);
    const uint32_t upto = 0xFFFFFFFFu >> (31 - lane);
    const bool in0 = x0 + lane < A.nx, in1 = x0 + 32 + lane < A.nx;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int r = warp * PER + k, y = y0 + r % RY, z = z0 + r / RY;
        if (y >= A.ny || z >= A.nz) continue;
        const uint64_t row = s_bits[r], st = run_starts(row);
        const uint32_t *lab = s_label + r * kSlots;
        uint32_t *out = A.par + (A.voxel(x0, y, z) + (uint32_t)lane);
        const uint32_t lo = (uint32_t)row, hi = (uint32_t)(row >> 32);
        const uint32_t slo = (uint32_t)st, shi = (uint32_t)(st >> 32);
        // slot = start / 2; a run of the high half may start in the low one
        const int s0 = (31 - __clz((int)(slo & upto))) >> 1;
        const uint32_t mh = shi & upto;
        const int s1 = (mh ? 63 - __clz((int)mh) : 31 - __clz((int)slo)) >> 1;
        if (in0) out[0] = (lo >> lane) & 1u ? lab[s0 ^ (r & 31)] : 0u;
        if (in1) out[32] = (hi >> lane) & 1u ? lab[s1 ^ (r & 31)] : 0u;
    }
}

// A voxel of the six faces, its face (Dir order) and linear index.  Face d is
// flattened over the two secondary axes; faces are concatenated in d order.
__device__ __forceinline__ uint32_t face_voxel(int64_t t, int nx, int ny, int nz, int &d)
{
    const int64_t fxy = (int64_t)nx * ny, fxz = (int64_t)nx * nz, fyz = (int64_t)ny * nz;
    const int64_t sizes[3] = {fyz, fxz, fxy};  // face area by primary axis
    d = 0;
    while (t >= sizes[d >> 1]) {
        t -= sizes[d >> 1];
        d++;
    }
    const bool pos = (d & 1) == 0;  // X_POS, Y_POS, Z_POS: the last plane
    int x, y, z;
    if (d < 2) { x = pos ? nx - 1 : 0; y = (int)(t % ny); z = (int)(t / ny); }
    else if (d < 4) { y = pos ? ny - 1 : 0; x = (int)(t % nx); z = (int)(t / nx); }
    else { z = pos ? nz - 1 : 0; x = (int)(t % nx); y = (int)(t / nx); }
    return (uint32_t)x + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
}

// Pass 7: the six face bitmaps.
__global__ void ccl_faces(const uint32_t *labels, int nx, int ny, int nz, uint32_t num_labels, uint8_t *bnd)
{
    const int64_t total = 2 * ((int64_t)ny * nz + (int64_t)nx * nz + (int64_t)nx * ny);
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        int d;
        const uint32_t l = labels[face_voxel(t, nx, ny, nz, d)];
        if (l > 0) bnd[(size_t)d * num_labels + l] = 1;
    }
}

// The faces each label touches as one byte per label, bit d = face d (label
// 0 touches none): what the area pass reads, made where it is read instead of
// through the face bitmaps and the host.
__global__ void ccl_face_bits(const uint32_t *__restrict__ labels, int nx, int ny, int nz, uint32_t *bits)
{
    const int64_t total = 2 * ((int64_t)ny * nz + (int64_t)nx * nz + (int64_t)nx * ny);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; t0 < total; t0 += stride) {
        int d = 0;
        const uint32_t l = t0 + lane < total ? labels[face_voxel(t0 + lane, nx, ny, nz, d)] : 0u;
        // One lane per label and face: one component can own most of a face.
        const unsigned same = __match_any_sync(0xFFFFFFFFu, (unsigned long long)l << 3 | (unsigned)d);
        if (l == 0 || lane != __ffs((int)same) - 1) continue;
        const uint32_t bit = 1u << (8 * (l & 3u) + d);
        // a stale read only repeats the atomic
        if (!(*(volatile uint32_t *)(bits + (l >> 2)) & bit)) atomicOr(bits + (l >> 2), bit);
    }
}

// Pass 8: row 6 = AND of rows 0..5.
__global__ void ccl_all_faces(uint32_t num_labels, uint8_t *bnd)
{
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < num_labels; l += gridDim.x * blockDim.x) {
        uint8_t all = 1;
        for (int d = 0; d < 6; d++) all &= bnd[(size_t)d * num_labels + l];
        bnd[(size_t)6 * num_labels + l] = all;
    }
}

#define CK(expr)                                                                                        \
    do {                                                                                                \
        cudaError_t e_ = (expr);                                                                        \
        if (e_ != cudaSuccess) return ft_fail(FAST_CUDA_ERROR, "%s: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

int check_dims(int64_t nx, int64_t ny, int64_t nz)
{
    if (nx <= 0 || ny <= 0 || nz <= 0) return ft_fail(FAST_BAD_ARG, "dimensions must be positive");
    if (nx > INT32_MAX || ny > INT32_MAX || nz > INT32_MAX) return ft_fail(FAST_BAD_ARG, "dimension too large");
    const double n = (double)nx * (double)ny * (double)nz;
    if (n >= 4294967295.0) return ft_fail(FAST_BAD_ARG, "labelling is limited to 4294967294 voxels");
    return FAST_OK;
}

// Geometry and scratch plan of a labelling; `base` null: sizes only.
// Returns the scratch bytes: 8 + 2 x slots + 4 per 64-voxel word, one bit per
// voxel and one count per chunk (1.2 bytes per voxel of a wide volume), and
// with `copy` (the mask lies in the labels' memory, which pass 1 writes while
// other blocks still read the mask) the mask.
size_t plan(Ccl &A, char *base, bool copy)
{
    const size_t words = (size_t)A.wx * A.ny * A.nz;
    const size_t n = (size_t)A.nx * A.ny * A.nz;
    const size_t nchunks = (n + kChunk - 1) / kChunk;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off += (bytes + 255) / 256 * 256;
        return p;
    };
    A.bits = (uint64_t *)take(words * 8);
    A.local = (uint16_t *)take(words * A.slots * 2);
    A.roots = (uint32_t *)take(words * 4);
    const size_t zero_off = off;
    A.cnt = (uint32_t *)take((nchunks + 1) * 4);
    A.root_bits = (uint32_t *)take(nchunks * (kChunk / 32) * 4);
    A.zero_words = (int64_t)((off - zero_off) / 4);
    if (copy) A.mask = (uint8_t *)take(n);
    return off;
}

// Labels of A.mask into A.par (device, N uint32) on `st`; scratch planned.
int label_device(const Ccl &A, uint32_t *num_labels, cudaStream_t st)
{
    const size_t n = (size_t)A.nx * A.ny * A.nz;
    const uint32_t nchunks = (uint32_t)((n + kChunk - 1) / kChunk);
    const int64_t words = (int64_t)A.wx * A.ny * A.nz;
    const int64_t bricks = (int64_t)A.wx * A.by * A.bz;
    ccl_bricks<<<(unsigned)bricks, kBrickThreads, 0, st>>>(A);
    const int64_t tx = (int64_t)(A.wx - 1) * A.ny * A.nz, ty = (int64_t)A.wx * (A.by - 1) * A.nz,
                  tz = (int64_t)A.wx * A.ny * (A.bz - 1);
    const int64_t tasks = tx + 4 * (ty + tz);
    if (tasks > 0) ccl_merge<<<(unsigned)((tasks + 255) / 256), 256, 0, st>>>(A, tx, ty, tz);
    ccl_flatten<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(A, words);
    ccl_scan_chunks<<<1, 1024, 0, st>>>(A.cnt, nchunks);
    ccl_rank<<<nchunks, kRankThreads, 0, st>>>(A.root_bits, A.cnt, A.par);
    ccl_relabel<<<(unsigned)bricks, kBrickThreads, 0, st>>>(A);
    CK(cudaGetLastError());
    uint32_t roots = 0;
    CK(cudaMemcpyAsync(&roots, A.cnt + nchunks, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    *num_labels = roots + 1u;
    return FAST_OK;
}

// Face bitmaps of device labels into the host buffer `boundary`.
int boundary_device(const uint32_t *d_labels, int64_t nx, int64_t ny, int64_t nz, uint32_t num_labels,
                    uint8_t *boundary, cudaStream_t st)
{
    const size_t bytes = (size_t)7 * num_labels;
    uint8_t *d_bnd = nullptr;
    CK(cudaMallocAsync((void **)&d_bnd, bytes, st));
    cudaError_t e = cudaMemsetAsync(d_bnd, 0, bytes, st);
    if (e == cudaSuccess) {
        ccl_faces<<<1024, 256, 0, st>>>(d_labels, (int)nx, (int)ny, (int)nz, num_labels, d_bnd);
        ccl_all_faces<<<(num_labels + 255) / 256 < 4096 ? (num_labels + 255) / 256 : 4096, 256, 0, st>>>(
            num_labels, d_bnd);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(boundary, d_bnd, bytes, cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(d_bnd, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return ft_fail(FAST_CUDA_ERROR, "boundary labels: %s", cudaGetErrorString(e));
    return FAST_OK;
}

int label_common(const uint8_t *d_mask, int64_t nx, int64_t ny, int64_t nz, uint8_t bg, uint32_t *d_labels,
                 uint32_t *num_labels, uint8_t *boundary, uint64_t boundary_cap, cudaStream_t st)
{
    int dev = 0;
    CK(cudaGetDevice(&dev));
    ft_retain_pool_memory(dev);
    Ccl A = {};
    A.nx = (int)(nx > 1 ? nx : ny);
    A.ny = (int)(nx > 1 ? ny : nz);
    A.nz = (int)(nx > 1 ? nz : 1);
    A.wx = (int)(((int64_t)A.nx + 63) / 64);
    A.by = (int)(((int64_t)A.ny + RY - 1) / RY);
    A.bz = (int)(((int64_t)A.nz + RZ - 1) / RZ);
    A.slots = A.nx >= 64 ? kSlots : (A.nx + 1) / 2;
    A.bg = bg;
    A.mask = d_mask;
    A.par = d_labels;
    const size_t n = (size_t)(nx * ny * nz);
    const uintptr_t m0 = (uintptr_t)d_mask, l0 = (uintptr_t)d_labels;
    const bool copy = m0 < l0 + 4 * n && l0 < m0 + n;
    const size_t need = plan(A, nullptr, copy);
    char *scratch = nullptr;
    cudaError_t e = cudaMallocAsync((void **)&scratch, need, st);
    if (e != cudaSuccess) return ft_fail(FAST_NOMEM, "labelling scratch: %s", cudaGetErrorString(e));
    plan(A, scratch, copy);
    int s = FAST_OK;
    if (copy) {
        e = cudaMemcpyAsync((void *)A.mask, d_mask, n, cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) s = ft_fail(FAST_CUDA_ERROR, "labelling mask: %s", cudaGetErrorString(e));
    }
    if (s == FAST_OK) s = label_device(A, num_labels, st);
    cudaFreeAsync(scratch, st);
    if (s == FAST_OK && boundary) {
        if (boundary_cap < (uint64_t)7 * *num_labels)
            s = ft_fail(FAST_BAD_ARG, "boundary buffer holds %llu bytes, 7 x %u needed",
                        (unsigned long long)boundary_cap, *num_labels);
        else
            s = boundary_device(d_labels, nx, ny, nz, *num_labels, boundary, st);
    }
    return s;
}

}  // namespace
}  // namespace ft

using namespace ft;

cudaError_t ft_label_faces(const uint32_t *d_labels, int64_t nx, int64_t ny, int64_t nz, uint32_t *d_bits,
                           cudaStream_t st)
{
    ccl_face_bits<<<1024, 256, 0, st>>>(d_labels, (int)nx, (int)ny, (int)nz, d_bits);
    return cudaGetLastError();
}

extern "C" {

FAST_API int fast_ccl_label_device(const uint8_t *d_mask, int64_t nx, int64_t ny, int64_t nz, uint8_t background,
                                   uint32_t *d_labels, uint32_t *num_labels, uint8_t *boundary,
                                   uint64_t boundary_cap, void *stream)
{
    ft_clear_error();
    if (!d_mask || !d_labels || !num_labels) return ft_fail(FAST_BAD_ARG, "null argument");
    int s = check_dims(nx, ny, nz);
    if (s != FAST_OK) return s;
    cudaStream_t st = (cudaStream_t)stream;
    s = label_common(d_mask, nx, ny, nz, background, d_labels, num_labels, boundary, boundary_cap, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (s == FAST_OK && e != cudaSuccess) s = ft_fail(FAST_CUDA_ERROR, "labelling: %s", cudaGetErrorString(e));
    return s;
}

FAST_API int fast_ccl_boundary_device(const uint32_t *d_labels, int64_t nx, int64_t ny, int64_t nz,
                                      uint32_t num_labels, uint8_t *boundary, void *stream)
{
    ft_clear_error();
    if (!d_labels || !boundary || num_labels == 0) return ft_fail(FAST_BAD_ARG, "null argument or no labels");
    const int s = check_dims(nx, ny, nz);
    if (s != FAST_OK) return s;
    return boundary_device(d_labels, nx, ny, nz, num_labels, boundary, (cudaStream_t)stream);
}

FAST_API int fast_ccl_label(const uint8_t *mask, int64_t nx, int64_t ny, int64_t nz, uint8_t background,
                            uint32_t *labels, uint32_t *num_labels, uint8_t *boundary, uint64_t boundary_cap)
{
    ft_clear_error();
    if (!mask) return ft_fail(FAST_NO_HOST_DATA, "mask must be allocated");
    if (!num_labels) return ft_fail(FAST_BAD_ARG, "num_labels is NULL");
    int s = check_dims(nx, ny, nz);
    if (s != FAST_OK) return s;
    const size_t n = (size_t)(nx * ny * nz);
    cudaStream_t st = nullptr;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    uint8_t *d_mask = nullptr;
    uint32_t *d_labels = nullptr;
    cudaError_t e = cudaMallocAsync((void **)&d_mask, n, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&d_labels, n * 4, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_mask, mask, n, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) {
        s = ft_fail(FAST_NOMEM, "labelling buffers: %s", cudaGetErrorString(e));
    } else {
        s = label_common(d_mask, nx, ny, nz, background, d_labels, num_labels, boundary, boundary_cap, st);
        if (s == FAST_OK && labels) {
            e = cudaMemcpyAsync(labels, d_labels, n * 4, cudaMemcpyDeviceToHost, st);
            if (e != cudaSuccess) s = ft_fail(FAST_CUDA_ERROR, "labels download: %s", cudaGetErrorString(e));
        }
    }
    if (d_mask) cudaFreeAsync(d_mask, st);
    if (d_labels) cudaFreeAsync(d_labels, st);
    e = cudaStreamSynchronize(st);
    if (s == FAST_OK && e != cudaSuccess) s = ft_fail(FAST_CUDA_ERROR, "labelling: %s", cudaGetErrorString(e));
    cudaStreamDestroy(st);
    return s;
}

}  // extern "C"
