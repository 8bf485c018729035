// Reactive area density ("alpha"): the marching-cubes area of a binary
// volume's 0.5 iso-surface (getReactiveAreaDensity, fastlib/src/volume/
// VolumeMeasures.cpp:294-301; getVolumeArea, fastlib/src/volume/
// VolumeSurface.cpp:10-36; the per-cell kernel ___generateTrianglesSurfaceArea,
// fastlib/src/cuda/VolumeSurface.cu:198-262) and its per-direction form over
// the pore space connected to each face (getReactiveAreaDensityTensor,
// VolumeMeasures.cpp:303-335, on generateBoundaryConnectedVolume,
// fastlib/src/volume/VolumeSegmentation.cpp:66-90).
//
// What the reference computes, restated:
//   * one cell per voxel position (i, j, k) in [0, n)^3; its corners are the
//     grid points (i..i+1, j..j+1, k..k+1);
//   * a grid point's value is the volume's texture read there: normalized
//     coordinates, linear filtering, clamp addressing, uint8 read as v/255
//     (fastlib/src/utility/DataPtr.cpp:565-595).  At the grid point g/n the
//     filter weights are 1/2, so the value is the mean of the 2x2x2 voxels
//     (g-1..g per axis, clamped to the volume): a multiple of 1/8 for a
//     0/255 volume;
//   * a corner is "below" when its value < isovalue (getCubeIndex); vertices
//     are interpolated on the cut edges, vertex = p0 + t (p1 - p0),
//     t = (iso - f0) / (f1 - f0); positions are in normalized units,
//     p = (i/nx, j/ny, k/nz) + corner offsets of 1/n per axis;
//   * triangle area = |(v1 - v0) x (v2 - v0)| / 2 in float, summed per cell
//     in double, then over all cells.
//
// The engine evaluates all of it in one pass over the volume and, for the
// per-direction form, over the CCL labels at the same time.  A block owns a
// brick of 62 x 16 x up to 16 cells and holds the voxels it needs as bits, 64
// along x in a word, one word array per field (bit set: the voxel's pore
// component touches face d; the seventh field: the voxel is solid).  Corner
// counts are sums of eight bits, done for 63 corners at once with word-wide
// adders, and so are the comparison with the isovalue and the test of which
// cells the surface cuts: a few instructions per 62 cells.  Only cut cells go
// further, compacted into a queue.  Fields that are equal over the brick (the
// face-connected pores, nearly everywhere) share their triangles.  Reductions
// are per block then in a fixed order, so results are run-to-run identical.
//
// The triangulation table is generated at compile time, not copied: for each of the 256
// corner patterns the cut edges of every cube face are joined in pairs (on a
// face with four cut edges, the two "below" corners are kept apart), the
// pairs close into loops, and each loop is fanned from its first edge.  Two
// cells sharing a face join that face's cut edges the same way, so the
// surface is closed.  The reference uses a fixed published table; on cells
// where the loop is not planar, or a face is ambiguous, its triangles and so
// its area differ slightly from these.
//
// The reference's texture unit quantises filter weights to 1/256; at the
// grid points the weights are 1/2 (exact) whenever 1/n is exact (n a power of
// two) and within 1/512 of 1/2 otherwise.  The engine uses exactly 1/2.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ccl_faces.h"
#include "fasttau.h"
#include "tau_errors.h"

namespace {

constexpr int NT = 256;
constexpr int BX = 62, BY = 16, BZ = 16;  // cells of a brick (z: at most)
constexpr int VY = BY + 2;                // voxel rows of a brick's plane
constexpr int VROWS = VY * (BZ + 2);      // voxel rows of a brick, 64 bits each
constexpr int CROWS = (BY + 1) * (BZ + 1);  // rows of grid points
static_assert(BY * BZ <= NT, "one row of cells per thread");
constexpr int kMaxTri = 5;
constexpr int kFields = 7;               // six face-connected pore fields + the solid field

struct McTable {
    uint8_t ntri[256];
    uint8_t edge[256][3 * kMaxTri];
};

// Corner c of a cell sits at offset (c&1 ^ c>>1&1, c>>1&1, c>>2) in the
// reference's order: 0 (0,0,0) 1 (1,0,0) 2 (1,1,0) 3 (0,1,0), 4..7 the same at
// z + 1.  Edge e joins corners kEdgeA[e] and kEdgeB[e] (the vertexInterp
// order of the per-cell kernel).
constexpr int kEdgeA[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3};
constexpr int kEdgeB[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
constexpr int kFaces[6][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {0, 1, 5, 4}, {3, 2, 6, 7}, {0, 3, 7, 4}, {1, 2, 6, 5}};

constexpr int edge_between(int a, int b)
{
    for (int e = 0; e < 12; e++)
        if ((kEdgeA[e] == a && kEdgeB[e] == b) || (kEdgeA[e] == b && kEdgeB[e] == a)) return e;
    return -1;
}

constexpr McTable build_table()
{
    McTable T{};
    for (int cs = 0; cs < 256; cs++) {
        int nb[12][2] = {}, deg[12] = {};
        for (int fi = 0; fi < 6; fi++) {
            const int *f = kFaces[fi];
            int E[4] = {}, pair[4] = {};
            bool cut[4] = {}, below[4] = {};
            int ncut = 0, npair = 0;
            for (int q = 0; q < 4; q++) {
                E[q] = edge_between(f[q], f[(q + 1) & 3]);
                below[q] = (cs >> f[q]) & 1;
            }
            for (int q = 0; q < 4; q++) {
                cut[q] = below[q] != below[(q + 1) & 3];
                ncut += cut[q];
            }
            if (ncut == 2) {
                for (int q = 0; q < 4; q++)
                    if (cut[q]) pair[npair++] = E[q];
            } else if (ncut == 4) {
                const int first = below[0] ? 3 : 0;  // corners 0 and 2 below: cut around each; else around 1 and 3
                for (int q = 0; q < 4; q++) pair[npair++] = E[(first + q) & 3];
            }
            for (int q = 0; q < npair; q += 2) {
                nb[pair[q]][deg[pair[q]]++] = pair[q + 1];
                nb[pair[q + 1]][deg[pair[q + 1]]++] = pair[q];
            }
        }
        bool seen[12] = {};
        int nt = 0;
        for (int e = 0; e < 12; e++) {
            if (deg[e] == 0 || seen[e]) continue;
            int loop[12] = {}, len = 0, prev = e, cur = nb[e][0] < nb[e][1] ? nb[e][0] : nb[e][1];
            loop[len++] = e;
            seen[e] = true;
            while (cur != e) {
                loop[len++] = cur;
                seen[cur] = true;
                const int next = nb[cur][0] == prev ? nb[cur][1] : nb[cur][0];
                prev = cur;
                cur = next;
            }
            for (int q = 1; q + 1 < len; q++) {
                T.edge[cs][3 * nt + 0] = (uint8_t)loop[0];
                T.edge[cs][3 * nt + 1] = (uint8_t)loop[q];
                T.edge[cs][3 * nt + 2] = (uint8_t)loop[q + 1];
                nt++;
            }
        }
        T.ntri[cs] = (uint8_t)nt;
    }
    return T;
}

// The same by corner pattern in one word, as fans: the edges of a loop's
// vertices in order, 4 bits each, kRestart before every further loop, and 0
// bits from the end on (a loop's 12 edges and 3 restarts fit 60 bits; the
// number of entries is in bits 60..63).
using PackedCase = uint64_t;
constexpr int kRestart = 15;
struct PackedTable {
    PackedCase at[256];
};

constexpr PackedTable pack_table(const McTable &T)
{
    PackedTable P{};
    for (int cs = 0; cs < 256; cs++) {
        int n = 0;
        for (int t = 0; t < T.ntri[cs]; t++) {
            const uint8_t *e = &T.edge[cs][3 * t];
            const bool more = t > 0 && e[0] == e[-3] && e[1] == e[-1];
            if (!more) {
                if (t > 0) P.at[cs] |= (PackedCase)kRestart << (4 * n++);
                P.at[cs] |= (PackedCase)e[0] << (4 * n++);
                P.at[cs] |= (PackedCase)e[1] << (4 * n++);
            }
            P.at[cs] |= (PackedCase)e[2] << (4 * n++);
        }
        P.at[cs] |= (PackedCase)n << 60;
    }
    return P;
}

// What a vertex on an edge needs: the corners' counts to pick (a byte
// selector over the counts of the even then the odd corners), the direction
// along each axis from its first corner (1, -1, or 0 across the edge) and
// all-ones where that corner is the cell's high one.
struct alignas(16) EdgeInfo {
    float dir[3];
    uint32_t pick;
    uint32_t high[3];
    uint32_t pad;
};
struct EdgeTable {
    EdgeInfo at[12];
};

constexpr EdgeTable make_edges()
{
    EdgeTable E{};
    for (int e = 0; e < 12; e++) {
        const int c[2] = {kEdgeA[e], kEdgeB[e]};
        int at[2][3] = {};
        for (int k = 0; k < 2; k++) {
            at[k][0] = (c[k] & 1) ^ ((c[k] >> 1) & 1);
            at[k][1] = (c[k] >> 1) & 1;
            at[k][2] = c[k] >> 2;
        }
        for (int a = 0; a < 3; a++) {
            E.at[e].dir[a] = (float)(at[1][a] - at[0][a]);
            E.at[e].high[a] = at[0][a] ? 0xffffffffu : 0u;
        }
        // bytes 0..3: corners 0, 2, 4, 6; bytes 4..7: corners 1, 3, 5, 7;
        // byte 0 of the result: the second corner, byte 1: the first
        auto byte_of = [](int q) { return (uint32_t)((q & 1) * 4 + q / 2); };
        E.at[e].pick = byte_of(c[1]) | byte_of(c[0]) << 4;
    }
    return E;
}

constexpr McTable kTable = build_table();
__device__ const McTable d_table = kTable;
__device__ const PackedTable d_cases = pack_table(kTable);
__device__ const EdgeTable d_edges = make_edges();

struct AlphaArgs {
    const uint8_t *mask;
    const uint32_t *labels;      // nullptr: the solid field alone
    const uint8_t *label_bits;   // per label: bit d = touches face d
    double *partials;            // [kFields][blocks]
    uint32_t *bad;               // set when a voxel is neither 0 nor 255
    int nx, ny, nz, zc, tiles_x, tiles_y;
    int64_t nblocks;
    float iso, vx, vy, vz;       // isovalue, voxel size 1/n per axis
    int thr;                     // corner below <=> count < thr (count = 8 x value)
};

// kEdgeA / kEdgeB packed one nibble per edge, for device code.
__device__ __forceinline__ int edge_a(int e) { return (int)((0x321076543210ULL >> (4 * e)) & 15u); }
__device__ __forceinline__ int edge_b(int e) { return (int)((0x765447650321ULL >> (4 * e)) & 15u); }

__device__ __forceinline__ float lerp1(float a, float b, float t) { return __fadd_rn(a, __fmul_rn(t, __fsub_rn(b, a))); }

// What a cell's vertices are made of: its low corner, high corner XOR low
// corner (as bits) and high - low along each axis, and its corner counts, a
// byte each, corners 0, 2, 4, 6 and 1, 3, 5, 7.
struct Cell {
    uint32_t p[3], x[3];
    float d[3];
    uint32_t even, odd;
};

// t by the counts n0, n1 at an edge's two ends sits at n0 * 256 + n1, the
// two bytes that a byte permute picks from the cell's counts.
constexpr int kTSize = 8 * 256 + 9;

// The vertex on an edge, in float arithmetic as the reference's helpers
// (lerp, cross, length) write it, with no fused multiply-add, so that every
// cell's area is reproducible: p0 + t (p1 - p0) per axis, where p1 - p0 is
// plus or minus high - low along the edge and 0 across it.
__device__ __forceinline__ float3 vertex(const Cell &C, const float *t_of, const EdgeInfo *edges, int e)
{
    const uint4 a = *reinterpret_cast<const uint4 *>(&edges[e].dir[0]);
    const uint4 b = *reinterpret_cast<const uint4 *>(&edges[e].high[0]);
    const float t = t_of[__byte_perm(C.even, C.odd, a.w) & 0xffffu];
    auto axis = [&](int k, uint32_t dir, uint32_t high) {
        return __fadd_rn(__uint_as_float(C.p[k] ^ (C.x[k] & high)), __fmul_rn(__fmul_rn(t, __uint_as_float(dir)), C.d[k]));
    };
    return make_float3(axis(0, a.x, b.x), axis(1, a.y, b.y), axis(2, a.z, b.z));
}

__device__ __forceinline__ float triangle_area(const float3 &v0, const float3 &v1, const float3 &v2)
{
    const float ax = __fsub_rn(v1.x, v0.x), ay = __fsub_rn(v1.y, v0.y), az = __fsub_rn(v1.z, v0.z);
    const float bx = __fsub_rn(v2.x, v0.x), by = __fsub_rn(v2.y, v0.y), bz = __fsub_rn(v2.z, v0.z);
    const float cx = __fsub_rn(__fmul_rn(ay, bz), __fmul_rn(az, by));
    const float cy = __fsub_rn(__fmul_rn(az, bx), __fmul_rn(ax, bz));
    const float cz = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
    const float d = __fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz));
    return __fmul_rn(__fsqrt_rn(d), 0.5f);
}

// Full adder of three words: sum and carry.
__device__ __forceinline__ uint64_t maj3(uint64_t a, uint64_t b, uint64_t c) { return (a & b) | (c & (a | b)); }

// Counts over two neighbouring voxels along x then y, bit c of word b the bit
// 2^b of the count at grid point c.
struct Sum2x2 {
    uint64_t b0, b1, b2;
};

__device__ __forceinline__ Sum2x2 sum2x2(uint64_t u, uint64_t v)
{
    const uint64_t u0 = u ^ (u >> 1), u1 = u & (u >> 1), v0 = v ^ (v >> 1), v1 = v & (v >> 1);
    const uint64_t k = u0 & v0;
    return Sum2x2{u0 ^ v0, u1 ^ v1 ^ k, maj3(u1, v1, k)};
}

// Grid points whose count over both planes is below thr (1..8).
__device__ __forceinline__ uint64_t below_word(const Sum2x2 &a, const Sum2x2 &b, int thr)
{
    const uint64_t t0 = a.b0 ^ b.b0, k0 = a.b0 & b.b0;
    const uint64_t t1 = a.b1 ^ b.b1 ^ k0, k1 = maj3(a.b1, b.b1, k0);
    const uint64_t t2 = a.b2 ^ b.b2 ^ k1, t3 = maj3(a.b2, b.b2, k1);
    uint64_t lt = (thr & 1) ? ~t0 : 0ull;
    lt = (thr & 2) ? (~t1 | lt) : (~t1 & lt);
    lt = (thr & 4) ? (~t2 | lt) : (~t2 & lt);
    return (thr & 8) ? (~t3 | lt) : (~t3 & lt);
}

// Counts at the eight corners of the cell in row (j, k) whose low corner is
// grid point c: three bits of each of the nine voxel rows around it.
__device__ __forceinline__ uint32_t cell_counts(const uint64_t *v, int j, int k, int c)
{
    uint32_t p[3][2];
#pragma unroll
    for (int dz = 0; dz < 3; dz++) {
        uint32_t x[3];
#pragma unroll
        for (int dy = 0; dy < 3; dy++) {
            const uint32_t b = (uint32_t)(v[(k + dz) * VY + j + dy] >> c) & 7u;
            // sums of bits 0, 1 (low nibble) and 1, 2 (high nibble)
            x[dy] = __byte_perm(0x12110100u, 0x22211110u, b);
        }
        p[dz][0] = x[0] + x[1];
        p[dz][1] = x[1] + x[2];
    }
    auto swap = [](uint32_t g) { return ((g & 15u) << 4) | (g >> 4); };  // corners 2, 3 run against x
    return (p[0][0] + p[1][0]) | swap(p[0][1] + p[1][1]) << 8 | (p[1][0] + p[2][0]) << 16 |
           swap(p[1][1] + p[2][1]) << 24;
}

// Corner pattern of eight counts: bit q set when count q < thr (1..8).
__device__ __forceinline__ int cube_of(uint32_t cnt, int thr)
{
    uint32_t m = (~(cnt + (uint32_t)(8 - thr) * 0x11111111u) >> 3) & 0x11111111u;
    m = (m | m >> 3) & 0x03030303u;
    m = (m | m >> 6) & 0x000f000fu;
    return (int)((m | m >> 12) & 0xffu);
}

constexpr int QCAP = 4096;  // cells in the queue at once

// The cut cells go through a shared queue so that all lanes have one: about
// one cell in seven of a porous volume is cut.  Queue positions come from a
// block-wide scan and item q is done by thread q mod NT, so every sum has a
// fixed order.  A cell's triangles are fans: a thread keeps the fan's first
// and last vertex and makes one new vertex per triangle.  Areas add in double
// at every level, which keeps the FP64 pipe half busy beside the other
// instructions (512^3, seven fields, with the labelling: 1.86 ms, and 1.87 with
// float pairs, or with the conversion done in integer instructions).
//
// Bound by instruction issue (384^3: 80 % of the slots busy, DRAM 7 %); most
// of it is the cut cells' vertices and areas.  Against summing every cell's
// corners as one 4-bit lane per field and queueing triangles: 512^3 spheres
// 7.40 -> 1.03 ms for the seven fields, 1024^3 58.6 -> 8.3; 200 x 181 x 190
// one field 146 -> 69 us.  U rows in flight hide the loads; more cost
// registers and so blocks per SM: five fit by their shared memory, and the
// bound keeps the registers of the seven-field pass to 46 (it took 57, and
// 4 % more time at 512^3, when left to the compiler).
template <bool LABELS>
__global__ void __launch_bounds__(NT, 5) alpha_kernel(AlphaArgs A)
{
    constexpr int NF = LABELS ? kFields : 1;
    __shared__ uint64_t s_v[NF][VROWS];
    __shared__ uint64_t s_below[CROWS];
    __shared__ PackedCase s_tab[256];
    __shared__ float s_t[kTSize];
    __shared__ EdgeInfo s_edge[12];
    __shared__ uint16_t s_q[QCAP];  // c | row << 6
    __shared__ int s_warp[NT / 32];
    __shared__ double s_red[NT / 32];
    __shared__ uint32_t s_differ;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tiles_xy = A.tiles_x * A.tiles_y;
    const int bz = blockIdx.x / tiles_xy;
    const int rem = blockIdx.x - bz * tiles_xy;
    const int by = rem / A.tiles_x, bx = rem - by * A.tiles_x;
    const int i0 = bx * BX, j0 = by * BY, k0 = bz * A.zc;
    const int nzc = min(A.zc, A.nz - k0);
    s_tab[tid] = d_cases.at[tid];
    if (tid < 81) {
        const float fa = __fmul_rn((float)(tid / 9), 0.125f), fb = __fmul_rn((float)(tid % 9), 0.125f);
        s_t[tid / 9 * 256 + tid % 9] = __fdiv_rn(__fsub_rn(A.iso, fa), __fsub_rn(fb, fa));
    } else if (tid >= 128 && tid < 128 + 24) {
        reinterpret_cast<uint4 *>(s_edge)[tid - 128] = reinterpret_cast<const uint4 *>(d_edges.at)[tid - 128];
    }
    if (tid == 0) s_differ = 0;

    // Voxel rows as bits: one warp per row, bit b = the voxel at x = i0 - 1 + b
    // (clamped to the volume, as y and z).
    const int rows = VY * (nzc + 2);
    // The clamps are on the offset from the voxel before the brick: on the
    // longest axes the coordinate itself leaves 32 bits before a clamp.
    auto clamped = [](int plus, int at, int n) { return min(max(plus, at == 0 ? 1 : 0), n - at); };
    const int x0 = i0 - 1 + clamped(lane, i0, A.nx), x1 = i0 - 1 + clamped(32 + lane, i0, A.nx);
    bool bad = false;
    constexpr int U = LABELS ? 3 : 6;  // rows in flight per warp
    for (int r0 = warp; r0 < rows; r0 += (NT / 32) * U) {
        uint32_t m[U][2], l[U][2];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = min(r0 + u * (NT / 32), rows - 1);
            const int zz = r / VY, yy = r - zz * VY;
            const int gz = k0 - 1 + clamped(zz, k0, A.nz), gy = j0 - 1 + clamped(yy, j0, A.ny);
            const int64_t base = ((int64_t)gz * A.ny + gy) * A.nx;
            m[u][0] = __ldg(A.mask + base + x0);
            m[u][1] = __ldg(A.mask + base + x1);
            if (LABELS) {
                l[u][0] = __ldg(A.labels + base + x0);
                l[u][1] = __ldg(A.labels + base + x1);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = min(r0 + u * (NT / 32), rows - 1);
#pragma unroll
            for (int h = 0; h < 2; h++) bad |= m[u][h] != 0 && m[u][h] != 255;
            const uint32_t s0 = __ballot_sync(0xffffffffu, m[u][0] != 0), s1 = __ballot_sync(0xffffffffu, m[u][1] != 0);
            uint32_t w0 = s0, w1 = s1;
            if (LABELS) {
                const uint32_t c0 = __ldg(A.label_bits + l[u][0]), c1 = __ldg(A.label_bits + l[u][1]);
                // Nearly every row's labelled voxels belong to components that
                // touch the same faces: one ballot then serves all of them.
                const uint32_t q = __reduce_or_sync(0xffffffffu, c0 | c1);
                if (__all_sync(0xffffffffu, (c0 == 0 || c0 == q) && (c1 == 0 || c1 == q))) {
                    const uint32_t b0 = __ballot_sync(0xffffffffu, c0 != 0), b1 = __ballot_sync(0xffffffffu, c1 != 0);
                    if (lane < kFields - 1) {
                        w0 = (q >> lane) & 1u ? b0 : 0u;
                        w1 = (q >> lane) & 1u ? b1 : 0u;
                    }
                } else {
#pragma unroll
                    for (int f = 0; f < kFields - 1; f++) {
                        const uint32_t b0 = __ballot_sync(0xffffffffu, (c0 >> f) & 1u);
                        const uint32_t b1 = __ballot_sync(0xffffffffu, (c1 >> f) & 1u);
                        if (lane == f) {
                            w0 = b0;
                            w1 = b1;
                        }
                    }
                }
            }
            if (lane < NF) s_v[lane][r] = (uint64_t)w1 << 32 | w0;
        }
    }
    if (bad) *A.bad = 1;
    __syncthreads();

    // Fields equal to an earlier one over the whole brick.
    if (LABELS) {
        uint32_t differ = 0;  // bit of (f, g), f < g
        for (int r = tid; r < rows; r += NT) {
            uint64_t w[kFields];
#pragma unroll
            for (int f = 0; f < kFields; f++) w[f] = s_v[LABELS ? f : 0][r];
            int bit = 0;
#pragma unroll
            for (int g = 1; g < kFields; g++)
#pragma unroll
                for (int f = 0; f < g; f++, bit++) differ |= (uint32_t)(w[f] != w[g]) << bit;
        }
        differ = __reduce_or_sync(0xffffffffu, differ);
        if (lane == 0) atomicOr(&s_differ, differ);
        __syncthreads();
    }
    const uint32_t differ = s_differ;
    const int bit0[kFields] = {0, 0, 1, 3, 6, 10, 15};  // first bit of the pairs (., g)

    for (int f = 0; f < NF; f++) {
        bool dup = false;
        for (int e = 0; e < f; e++) dup |= !((differ >> (bit0[f] + e)) & 1u);
        if (dup) continue;
        const uint64_t *v = s_v[f];
        for (int r = tid; r < (BY + 1) * (nzc + 1); r += NT) {
            const int z = r / (BY + 1), y = r - z * (BY + 1);
            const uint64_t *q = v + z * VY + y;
            s_below[r] = below_word(sum2x2(q[0], q[1]), sum2x2(q[VY], q[VY + 1]), A.thr);
        }
        __syncthreads();
        // One row of cells per thread: those with corners on both sides.
        const int k = tid / BY, j = tid - k * BY;
        uint64_t cut = 0;
        if (k < nzc && j < A.ny - j0) {
            const int nc = min(BX, A.nx - i0);
            uint64_t any = 0, all = ~0ull;
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const uint64_t w = s_below[(k + (h >> 1)) * (BY + 1) + j + (h & 1)];
                any |= w | w >> 1;
                all &= w & w >> 1;
            }
            cut = any & ~all & ((1ull << nc) - 1);
        }
        const int mine = __popcll(cut);
        int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        int at = inc - mine, total = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++) {
            const int t = s_warp[w];
            at += w < warp ? t : 0;
            total += t;
        }
        double acc = 0.0;
        for (int base = 0; base < total; base += QCAP) {
            while (cut && at < base + QCAP) {
                const int c = __ffsll((long long)cut) - 1;
                cut &= cut - 1;
                s_q[at - base] = (uint16_t)(c | tid << 6);
                at++;
            }
            __syncthreads();
            const int n = min(total - base, QCAP);
            for (int q = tid; q < n; q += NT) {
                const int it = s_q[q], c = it & 63, row = it >> 6;
                const int ck = row / BY, cj = row - ck * BY;
                const uint32_t cnt = cell_counts(v, cj, ck, c);
                Cell C;
                C.even = cnt & 0x0f0f0f0fu;
                C.odd = (cnt >> 4) & 0x0f0f0f0fu;
                const float lo[3] = {__fmul_rn(A.vx, (float)(i0 + c)), __fmul_rn(A.vy, (float)(j0 + cj)),
                                     __fmul_rn(A.vz, (float)(k0 + ck))};
                const float size[3] = {A.vx, A.vy, A.vz};
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    const float hi = __fadd_rn(lo[a], size[a]);
                    C.p[a] = __float_as_uint(lo[a]);
                    C.x[a] = __float_as_uint(lo[a]) ^ __float_as_uint(hi);
                    C.d[a] = __fsub_rn(hi, lo[a]);
                }
                PackedCase pc = s_tab[cube_of(cnt, A.thr)];
                int left = (int)(pc >> 60) - 2;
                float3 v0 = vertex(C, s_t, s_edge, (int)pc & 15), v2 = vertex(C, s_t, s_edge, (int)(pc >> 4) & 15);
                pc >>= 8;
                for (; left > 0; left--, pc >>= 4) {
                    int e = (int)pc & 15;
                    if (e == kRestart) {
                        v0 = vertex(C, s_t, s_edge, (int)(pc >> 4) & 15);
                        v2 = vertex(C, s_t, s_edge, (int)(pc >> 8) & 15);
                        pc >>= 12;
                        left -= 3;
                        e = (int)pc & 15;
                    }
                    const float3 v1 = v2;
                    v2 = vertex(C, s_t, s_edge, e);
                    acc += (double)triangle_area(v0, v1, v2);
                }
            }
            __syncthreads();
        }
        // The brick's sum, in a fixed order.
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (lane == 0) s_red[warp] = acc;
        __syncthreads();
        if (tid < NF) {  // to every field of the group
            bool same = tid == f;
            if (tid > f) same = !((differ >> (bit0[tid] + f)) & 1u);
            if (same) {
                double sum = 0.0;
                for (int w = 0; w < NT / 32; w++) sum += s_red[w];
                A.partials[(size_t)tid * A.nblocks + blockIdx.x] = sum;
            }
        }
    }
}

// One block per field sums its per-block partials in a fixed order.
constexpr int NSUM = 1024;
__global__ void __launch_bounds__(NSUM) alpha_sum_kernel(const double *partials, int nblocks, double *out)
{
    __shared__ double s[NSUM];
    const double *p = partials + (size_t)blockIdx.x * nblocks;
    double v = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < nblocks; b += NSUM) v += p[b];
    s[threadIdx.x] = v;
    __syncthreads();
    for (int w = NSUM / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = s[0];
}

int check_args(int64_t nx, int64_t ny, int64_t nz, float iso)
{
    if (nx <= 0 || ny <= 0 || nz <= 0) return ft_fail(FAST_BAD_ARG, "dimensions must be positive");
    if (nx > INT32_MAX || ny > INT32_MAX || nz > INT32_MAX) return ft_fail(FAST_BAD_ARG, "dimension too large");
    if (iso != iso) return ft_fail(FAST_BAD_ARG, "isovalue is NaN");
    return FAST_OK;
}

// The whole area pass on device data; out[kFields] (host) gets the sums.
int area_device(const uint8_t *d_mask, const uint32_t *d_labels, const uint8_t *d_bits, int64_t nx, int64_t ny,
                int64_t nz, float iso, double *out, cudaStream_t st)
{
    AlphaArgs A;
    memset(&A, 0, sizeof(A));
    A.mask = d_mask;
    A.labels = d_labels;
    A.label_bits = d_bits;
    A.nx = (int)nx;
    A.ny = (int)ny;
    A.nz = (int)nz;
    A.tiles_x = (int)((nx + BX - 1) / BX);
    A.tiles_y = (int)((ny + BY - 1) / BY);
    // Bricks 16 cells deep, halved while the grid has fewer than 6 blocks per
    // SM.  Of 2, 3, 4, 6, 8 and 12 at eleven sizes from 48^3 to 256^3, one field
    // and the tensor call, each of the others is 10 % or more behind somewhere
    // (2: 239 against 210 us at 97 x 300 x 150; 3 and 4: 283 against 252 at 190 x
    // 181 x 200, both tensors; 8 and 12: 79 against 70 at 160^3, one field), 6 at
    // 128^3 with one field alone (67 against 60 at 3).
    int sms = 152, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t xy = (int64_t)A.tiles_x * A.tiles_y;
    int zc = BZ;
    while (zc > 1 && xy * ((nz + zc - 1) / zc) < 6LL * sms) zc /= 2;
    const int64_t nblocks = xy * ((nz + zc - 1) / zc);
    if (nblocks > INT32_MAX) return ft_fail(FAST_BAD_ARG, "volume too large for one area pass");
    A.zc = zc;
    A.nblocks = nblocks;
    A.iso = iso;
    A.vx = 1.0f / (float)nx;
    A.vy = 1.0f / (float)ny;
    A.vz = 1.0f / (float)nz;
    A.thr = 9;
    for (int c = 8; c >= 0; c--)
        if ((float)c * 0.125f >= iso) A.thr = c;
    const bool none = A.thr < 1 || A.thr > 8;  // no corner, or every corner, is below: no surface
    if (none) A.thr = 8;

    const size_t part_bytes = (size_t)nblocks * kFields * sizeof(double);
    char *scratch = nullptr;
    const size_t need = part_bytes + 256 + kFields * sizeof(double) + 256 + 16;
    cudaError_t e = cudaMallocAsync((void **)&scratch, need, st);
    if (e != cudaSuccess) return ft_fail(FAST_NOMEM, "area scratch: %s", cudaGetErrorString(e));
    double *d_part = (double *)scratch;
    double *d_out = (double *)((char *)d_part + part_bytes + 256);
    uint32_t *d_bad = (uint32_t *)((char *)d_out + kFields * sizeof(double) + 256);
    A.partials = d_part;
    A.bad = d_bad;
    double h_out[kFields];
    uint32_t h_bad = 0;
    e = cudaMemsetAsync(d_bad, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess) {
        if (d_labels)
            alpha_kernel<true><<<(unsigned)nblocks, NT, 0, st>>>(A);
        else
            alpha_kernel<false><<<(unsigned)nblocks, NT, 0, st>>>(A);
        alpha_sum_kernel<<<d_labels ? kFields : 1, NSUM, 0, st>>>(d_part, (int)nblocks, d_out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_out, d_out, sizeof(h_out), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_bad, d_bad, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(scratch, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return ft_fail(FAST_CUDA_ERROR, "area pass: %s", cudaGetErrorString(e));
    if (h_bad) return ft_fail(FAST_BAD_TYPE, "the volume must hold 0 and 255 only");
    for (int f = 0; f < (d_labels ? kFields : 1); f++) out[f] = none ? 0.0 : h_out[f];
    return FAST_OK;
}

// getVolumeCCL(mask, 255) on the device, then the seven-field pass.
int tensor_device(const uint8_t *d_mask, int64_t nx, int64_t ny, int64_t nz, float iso, double *tensor,
                  double *area_solid, cudaStream_t st)
{
    if ((double)nx * ny * nz >= 4294967295.0) return ft_fail(FAST_BAD_ARG, "labelling is limited to 4294967294 voxels");
    const size_t n = (size_t)(nx * ny * nz);
    uint32_t *d_labels = nullptr;
    cudaError_t e = cudaMallocAsync((void **)&d_labels, n * 4, st);
    if (e != cudaSuccess) return ft_fail(FAST_NOMEM, "labels: %s", cudaGetErrorString(e));
    uint32_t num_labels = 0;
    int s = fast_ccl_label_device(d_mask, nx, ny, nz, 255, d_labels, &num_labels, nullptr, 0, st);
    uint8_t *d_bits = nullptr;
    if (s == FAST_OK) {
        const size_t words = ((size_t)num_labels + 3) / 4;
        e = cudaMallocAsync((void **)&d_bits, words * 4, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(d_bits, 0, words * 4, st);
        if (e == cudaSuccess) e = ft_label_faces(d_labels, nx, ny, nz, (uint32_t *)d_bits, st);
        if (e != cudaSuccess) s = ft_fail(FAST_CUDA_ERROR, "label bits: %s", cudaGetErrorString(e));
    }
    double out[kFields];
    if (s == FAST_OK) s = area_device(d_mask, d_labels, d_bits, nx, ny, nz, iso, out, st);
    if (d_bits) cudaFreeAsync(d_bits, st);
    cudaFreeAsync(d_labels, st);
    cudaStreamSynchronize(st);
    if (s != FAST_OK) return s;
    for (int d = 0; d < 6; d++) tensor[d] = out[d];
    if (area_solid) *area_solid = out[6];
    return FAST_OK;
}

// Host mask -> device copy on a private stream, then `body`.
template <class F>
int with_device_mask(const uint8_t *mask, int64_t nx, int64_t ny, int64_t nz, F body)
{
    const size_t n = (size_t)(nx * ny * nz);
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) return ft_fail(FAST_CUDA_ERROR, "stream: %s", cudaGetErrorString(e));
    uint8_t *d = nullptr;
    int s;
    e = cudaMallocAsync((void **)&d, n, st);
    if (e != cudaSuccess) {
        s = ft_fail(FAST_NOMEM, "mask copy: %s", cudaGetErrorString(e));
    } else {
        e = cudaMemcpyAsync(d, mask, n, cudaMemcpyHostToDevice, st);
        s = e == cudaSuccess ? body(d, st) : ft_fail(FAST_CUDA_ERROR, "mask upload: %s", cudaGetErrorString(e));
        cudaFreeAsync(d, st);
    }
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return s;
}

// ---------------------------------------------------------------------------
// Mesh export: the triangles themselves (getVolumeAreaMesh, fastlib/src/
// volume/VolumeSurface.cpp:38-68, ___generateTriangles in fastlib/src/cuda/
// VolumeSurface.cu:264-357).  Field = voxel != 0, corner values and cut
// vertices as for the area; positions in the reference's mesh frame: a voxel
// is dx = 1/max(n) wide on every axis and the grid is centred on the origin,
// p = (dx i - dx n / 2, ...); one face normal per triangle,
// normalize((v1 - v0) x (v2 - v0)).  Two passes with a fixed order: blocks
// of 256 cells count their triangles, the host scans the block totals, and
// each block writes its cells' triangles in cell order (12 floats each: three
// vertices, then the normal).
// ---------------------------------------------------------------------------
constexpr int kMeshBlock = 256;

struct MeshArgs {
    const uint8_t *mask;
    int nx, ny, nz, thr;
    float iso, vx, vy, vz, dx;
};

__device__ __forceinline__ uint32_t mesh_counts(const MeshArgs &A, int64_t cell, int &cube, int &i, int &j, int &k)
{
    i = (int)(cell % A.nx);
    j = (int)((cell / A.nx) % A.ny);
    k = (int)(cell / ((int64_t)A.nx * A.ny));
    uint32_t cnt = 0;
    cube = 0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const int ox = (c & 1) ^ ((c >> 1) & 1), oy = (c >> 1) & 1, oz = c >> 2;
        int n = 0;
        for (int dz = -1; dz <= 0; dz++)
            for (int dy = -1; dy <= 0; dy++)
                for (int dxx = -1; dxx <= 0; dxx++) {
                    int gx = i + ox + dxx, gy = j + oy + dy, gz = k + oz + dz;
                    gx = gx < 0 ? 0 : (gx >= A.nx ? A.nx - 1 : gx);
                    gy = gy < 0 ? 0 : (gy >= A.ny ? A.ny - 1 : gy);
                    gz = gz < 0 ? 0 : (gz >= A.nz ? A.nz - 1 : gz);
                    n += A.mask[((int64_t)gz * A.ny + gy) * A.nx + gx] != 0;
                }
        cnt |= (uint32_t)n << (4 * c);
        cube |= (n < A.thr) << c;
    }
    return cnt;
}

__global__ void __launch_bounds__(kMeshBlock) mesh_count_kernel(MeshArgs A, int64_t ncell, uint32_t *block_tri)
{
    __shared__ uint32_t s[kMeshBlock];
    const int64_t cell = (int64_t)blockIdx.x * kMeshBlock + threadIdx.x;
    uint32_t nt = 0;
    if (cell < ncell) {
        int cube, i, j, k;
        mesh_counts(A, cell, cube, i, j, k);
        nt = d_table.ntri[cube];
    }
    s[threadIdx.x] = nt;
    __syncthreads();
    for (int w = kMeshBlock / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_tri[blockIdx.x] = s[0];
}

__global__ void __launch_bounds__(kMeshBlock) mesh_emit_kernel(MeshArgs A, int64_t ncell, const uint64_t *block_off,
                                                               float *out)
{
    __shared__ uint32_t s[kMeshBlock];
    const int64_t cell = (int64_t)blockIdx.x * kMeshBlock + threadIdx.x;
    int cube = 0, i = 0, j = 0, k = 0;
    uint32_t cnt = 0, nt = 0;
    if (cell < ncell) {
        cnt = mesh_counts(A, cell, cube, i, j, k);
        nt = d_table.ntri[cube];
    }
    // exclusive scan of the counts in cell order (Hillis-Steele over the block)
    s[threadIdx.x] = nt;
    __syncthreads();
    for (int o = 1; o < kMeshBlock; o <<= 1) {
        const uint32_t v = threadIdx.x >= o ? s[threadIdx.x - o] : 0u;
        __syncthreads();
        s[threadIdx.x] += v;
        __syncthreads();
    }
    const uint64_t base = block_off[blockIdx.x] + s[threadIdx.x] - nt;
    if (nt == 0) return;
    // positions in the mesh frame (VolumeSurface.cu:291-297)
    const float px = __fsub_rn(__fmul_rn(A.dx, (float)i), __fmul_rn(0.5f, __fmul_rn(A.dx, (float)A.nx)));
    const float py = __fsub_rn(__fmul_rn(A.dx, (float)j), __fmul_rn(0.5f, __fmul_rn(A.dx, (float)A.ny)));
    const float pz = __fsub_rn(__fmul_rn(A.dx, (float)k), __fmul_rn(0.5f, __fmul_rn(A.dx, (float)A.nz)));
    const float qx = __fadd_rn(px, A.dx), qy = __fadd_rn(py, A.dx), qz = __fadd_rn(pz, A.dx);
    for (uint32_t t = 0; t < nt; t++) {
        float v[3][3];
        for (int q = 0; q < 3; q++) {
            const int e = d_table.edge[cube][3 * t + q];
            const int ca = edge_a(e), cb = edge_b(e);
            const float fa = __fmul_rn((float)((cnt >> (4 * ca)) & 15u), 0.125f);
            const float fb = __fmul_rn((float)((cnt >> (4 * cb)) & 15u), 0.125f);
            const float x0 = ((ca & 1) ^ ((ca >> 1) & 1)) ? qx : px, y0 = ((ca >> 1) & 1) ? qy : py, z0 = (ca >> 2) ? qz : pz;
            const float x1 = ((cb & 1) ^ ((cb >> 1) & 1)) ? qx : px, y1 = ((cb >> 1) & 1) ? qy : py, z1 = (cb >> 2) ? qz : pz;
            if (fa == fb) {
                v[q][0] = x0; v[q][1] = y0; v[q][2] = z0;
            } else {
                const float tt = __fdiv_rn(__fsub_rn(A.iso, fa), __fsub_rn(fb, fa));
                v[q][0] = lerp1(x0, x1, tt);
                v[q][1] = lerp1(y0, y1, tt);
                v[q][2] = lerp1(z0, z1, tt);
            }
        }
        const float ax = __fsub_rn(v[1][0], v[0][0]), ay = __fsub_rn(v[1][1], v[0][1]), az = __fsub_rn(v[1][2], v[0][2]);
        const float bx = __fsub_rn(v[2][0], v[0][0]), by = __fsub_rn(v[2][1], v[0][1]), bz = __fsub_rn(v[2][2], v[0][2]);
        const float cx = __fsub_rn(__fmul_rn(ay, bz), __fmul_rn(az, by));
        const float cy = __fsub_rn(__fmul_rn(az, bx), __fmul_rn(ax, bz));
        const float cz = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
        const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz)));
        const float inv = len > 0.f ? __fdiv_rn(1.0f, len) : 0.f;
        float *o = out + (base + t) * 12;
        for (int q = 0; q < 3; q++)
            for (int a = 0; a < 3; a++) o[3 * q + a] = v[q][a];
        o[9] = __fmul_rn(cx, inv);
        o[10] = __fmul_rn(cy, inv);
        o[11] = __fmul_rn(cz, inv);
    }
}

int mesh_device(const uint8_t *d_mask, int64_t nx, int64_t ny, int64_t nz, float iso, float *out, uint64_t capacity,
                uint64_t *ntri, cudaStream_t st)
{
    const int64_t ncell = nx * ny * nz;
    const int64_t nblocks = (ncell + kMeshBlock - 1) / kMeshBlock;
    if (nblocks > INT32_MAX) return ft_fail(FAST_BAD_ARG, "volume too large for the mesh export");
    MeshArgs A;
    A.mask = d_mask;
    A.nx = (int)nx;
    A.ny = (int)ny;
    A.nz = (int)nz;
    A.iso = iso;
    A.thr = 9;
    for (int c = 8; c >= 0; c--)
        if ((float)c * 0.125f >= iso) A.thr = c;
    const int64_t maxdim = std::max(nx, std::max(ny, nz));
    A.dx = 1.0f / (float)maxdim;
    char *scratch = nullptr;
    const size_t need = (size_t)nblocks * 4 + 256 + (size_t)nblocks * 8;
    cudaError_t e = cudaMallocAsync((void **)&scratch, need, st);
    if (e != cudaSuccess) return ft_fail(FAST_NOMEM, "mesh scratch: %s", cudaGetErrorString(e));
    uint32_t *d_cnt = (uint32_t *)scratch;
    uint64_t *d_off = (uint64_t *)((char *)d_cnt + ((size_t)nblocks * 4 + 255) / 256 * 256);
    std::vector<uint32_t> cnt((size_t)nblocks);
    std::vector<uint64_t> off((size_t)nblocks);
    int s = FAST_OK;
    mesh_count_kernel<<<(unsigned)nblocks, kMeshBlock, 0, st>>>(A, ncell, d_cnt);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(cnt.data(), d_cnt, (size_t)nblocks * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    uint64_t total = 0;
    if (e == cudaSuccess) {
        for (int64_t b = 0; b < nblocks; b++) {
            off[(size_t)b] = total;
            total += cnt[(size_t)b];
        }
        *ntri = total;
        if (out && total > capacity)
            s = ft_fail(FAST_BAD_ARG, "mesh buffer holds %llu triangles, %llu needed", (unsigned long long)capacity,
                        (unsigned long long)total);
        if (out && s == FAST_OK && total > 0) {
            float *d_out = nullptr;
            e = cudaMallocAsync((void **)&d_out, (size_t)total * 12 * sizeof(float), st);
            if (e != cudaSuccess) {
                s = ft_fail(FAST_NOMEM, "mesh triangles: %s", cudaGetErrorString(e));
            } else {
                e = cudaMemcpyAsync(d_off, off.data(), (size_t)nblocks * 8, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) {
                    mesh_emit_kernel<<<(unsigned)nblocks, kMeshBlock, 0, st>>>(A, ncell, d_off, d_out);
                    e = cudaGetLastError();
                }
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(out, d_out, (size_t)total * 12 * sizeof(float), cudaMemcpyDeviceToHost, st);
                cudaFreeAsync(d_out, st);
            }
        }
    }
    cudaFreeAsync(scratch, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    if (s == FAST_OK && e != cudaSuccess) s = ft_fail(FAST_CUDA_ERROR, "mesh: %s", cudaGetErrorString(e));
    return s;
}

}  // namespace

extern "C" {

FAST_API int fast_reactive_area_mesh(const uint8_t *mask, int64_t nx, int64_t ny, int64_t nz, float isovalue,
                                     float *triangles, uint64_t capacity, uint64_t *ntri)
{
    ft_clear_error();
    if (!mask) return ft_fail(FAST_NO_HOST_DATA, "mask is NULL");
    if (!ntri) return ft_fail(FAST_BAD_ARG, "ntri is NULL");
    int s = check_args(nx, ny, nz, isovalue);
    if (s != FAST_OK) return s;
    return with_device_mask(mask, nx, ny, nz, [&](const uint8_t *d, cudaStream_t st) {
        return mesh_device(d, nx, ny, nz, isovalue, triangles, capacity, ntri, st);
    });
}


FAST_API int fast_reactive_area_device(const uint8_t *d_mask, int64_t nx, int64_t ny, int64_t nz, float isovalue,
                                       double *area, void *stream)
{
    ft_clear_error();
    if (!d_mask) return ft_fail(FAST_NO_HOST_DATA, "mask is NULL");
    if (!area) return ft_fail(FAST_BAD_ARG, "area is NULL");
    int s = check_args(nx, ny, nz, isovalue);
    if (s != FAST_OK) return s;
    return area_device(d_mask, nullptr, nullptr, nx, ny, nz, isovalue, area, (cudaStream_t)stream);
}

FAST_API int fast_reactive_area(const uint8_t *mask, int64_t nx, int64_t ny, int64_t nz, float isovalue, double *area)
{
    ft_clear_error();
    if (!mask) return ft_fail(FAST_NO_HOST_DATA, "mask is NULL");
    if (!area) return ft_fail(FAST_BAD_ARG, "area is NULL");
    int s = check_args(nx, ny, nz, isovalue);
    if (s != FAST_OK) return s;
    return with_device_mask(mask, nx, ny, nz, [&](const uint8_t *d, cudaStream_t st) {
        return area_device(d, nullptr, nullptr, nx, ny, nz, isovalue, area, st);
    });
}

FAST_API int fast_reactive_area_tensor_device(const uint8_t *d_mask, int64_t nx, int64_t ny, int64_t nz,
                                              float isovalue, double *tensor, double *area_solid, void *stream)
{
    ft_clear_error();
    if (!d_mask) return ft_fail(FAST_NO_HOST_DATA, "mask is NULL");
    if (!tensor) return ft_fail(FAST_BAD_ARG, "tensor is NULL");
    int s = check_args(nx, ny, nz, isovalue);
    if (s != FAST_OK) return s;
    return tensor_device(d_mask, nx, ny, nz, isovalue, tensor, area_solid, (cudaStream_t)stream);
}

FAST_API int fast_reactive_area_tensor(const uint8_t *mask, int64_t nx, int64_t ny, int64_t nz, float isovalue,
                                       double *tensor, double *area_solid)
{
    ft_clear_error();
    if (!mask) return ft_fail(FAST_NO_HOST_DATA, "mask is NULL");
    if (!tensor) return ft_fail(FAST_BAD_ARG, "tensor is NULL");
    int s = check_args(nx, ny, nz, isovalue);
    if (s != FAST_OK) return s;
    return with_device_mask(mask, nx, ny, nz, [&](const uint8_t *d, cudaStream_t st) {
        return tensor_device(d, nx, ny, nz, isovalue, tensor, area_solid, st);
    });
}

}  // extern "C"
