// CG of small F64 and F32 volumes in one kernel: every tile of the launch is a
// block of a cooperative launch that keeps its part of p, r and q in shared
// memory and iterates; a right-hand side's blocks wait for one another's
// partial sums where the sweeps have a kernel boundary.
//
// What bounds small volumes is not their voxels: of the 8 us of a sweep of a
// 28 x 24 x 20 volume, two are the tile's planes, the rest the launch, the
// block's start (its job, tables, scalars, tensor maps) and the finisher's
// chain (count the block in, fetch the partial sums, update the scalars).
// Here the start is paid once per launch, every block sums all partial sums
// and updates its own copy of the scalars, and between two exchanges a block
// reads from global memory only the residual around its tile.  In F64 the
// pointwise updates and the stencil then run at the FP64 pipe's rate.
//
// Arithmetic, tiles and summation order are those of OpCG1 and PwCG2: a solve
// has the same bits either way (the serving context runs the sweeps).  Every
// spin is bounded (2 s); a block that gives up marks its right-hand side FAULT
// and leaves.
//
// us per iteration of the two sweeps (replayed from a graph) -> here: F64 20.3
// -> 13.6 at 40^3, 25.3 -> 18.0 at 64^3, 42.4 -> 34.9 at 80^3; F32 15.8 -> 11.2 at
// 64^3, 22.2 -> 14.2 for twelve times 32^3.  At 64^3 (128 blocks of four
// planes) 8.4 of the 18.0 are the FP64 pipe's (2.1 us a plane), the rest
// the two exchanges and the residual around the tile.
// Two blocks on an SM hold six planes each in F64 and twelve in F32, one
// alone about twice that: larger volumes stay with the sweeps.
#pragma once
#include <cstddef>

#include "tau_launch.h"
#include "tau_pointwise.cuh"

namespace ft {
inline namespace FT_TILES {

constexpr int kBoxW = TX + 2;  // codes of a plane's box: columns -1 .. TX

// Shared memory of a tile of zc planes: p with halo, r and q, codes with halo.
template <typename T>
__host__ __device__ constexpr size_t resident_smem(int zc)
{
    return (size_t)(zc + 2) * HY * PW * sizeof(T) + 2 * (size_t)zc * TX * TY * sizeof(T) + (size_t)(zc + 2) * HY * kBoxW + 16;
}

// A tile's partial sums of a step, each with the iteration it belongs to: 16
// bytes read and written as one, so the sums need no barrier beside them (with
// a counter to wait on and the sums read after it: 13.9 against 13.6 us per
// iteration at 40^3 in F64, 11.8 against 11.2 at 64^3 and 15.0 against 14.2 for
// twelve times 32^3 in F32).  A block has read all of an iteration's step 1 when it writes its step 2, and
// the reverse, so a slot is never overwritten unread.
constexpr int kSlots = 3;  // p.q; |r|^2, r.z
static_assert(kSlots * sizeof(ulonglong2) == kResidentSlotBytes);

__device__ __forceinline__ void slot_write(ulonglong2 *s, double v, uint64_t epoch)
{
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.release.gpu.global.b128 [%0], t; }" ::"l"(s),
                 "l"(__double_as_longlong(v)), "l"(epoch)
                 : "memory");
}

// The value of a slot once it has the epoch; false after kWaitLimitNs.
__device__ __forceinline__ bool slot_read(const ulonglong2 *s, uint64_t epoch, double &v)
{
    uint64_t t0 = 0;
    for (int n = 0;; n++) {
        uint64_t bits, e;
        asm volatile("{ .reg .b128 t; ld.acquire.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                     : "=l"(bits), "=l"(e)
                     : "l"(s)
                     : "memory");
        v = __longlong_as_double((long long)bits);
        if (e == epoch) return true;
        if ((n & 63) == 63) {
            const uint64_t now = global_timer_ns();
            if (!t0) t0 = now;
            else if (now - t0 > kWaitLimitNs) return false;
        }
    }
}

// Publishes the block's partial sums v of `epoch` and waits for those of all
// of the right-hand side's blocks: their totals, in sum_partials' order.  What
// the blocks wrote before is visible then.  false: one did not come in time
// (silent: test-hook builds, a block that publishes nothing).
template <int NV, typename V>
__device__ __forceinline__ bool exchange(const V (&v)[NV], ulonglong2 *slots, int64_t local, int64_t ntiles,
                                         uint64_t epoch, double (&tot)[NV], double *s_red, double *s_val, int *s_ok,
                                         bool silent)
{
    __shared__ double s_tot[NV];
    const int tid = threadIdx.x;
    block_sum_store<NV, V>(v, s_tot, s_red);
    if (tid < NV && !silent) slot_write(slots + local * kSlots + tid, s_tot[tid], epoch);
    for (int e = tid; e < NV * (int)ntiles; e += NTHREADS)  // a slot per thread: no two waits in a row
        if (!slot_read(slots + (e / NV) * kSlots + e % NV, epoch, s_val[e])) *s_ok = 0;
    __syncthreads();
    double a[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) a[k] = 0.0;
    for (int t = tid; t < (int)ntiles; t += NTHREADS) {
#pragma unroll
        for (int k = 0; k < NV; k++) a[k] += s_val[t * NV + k];
    }
    block_sum_store<NV, double>(a, s_tot, s_red, ntiles < NTHREADS ? (int)ntiles : NTHREADS);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = s_tot[k];
    return *s_ok != 0;
}

// p = p beta + r / diag with the roundings that the compiler gives OpCG1 (a
// served solve runs the sweeps and equals the same solve alone).  Keeping
// r / diag from step 2 would save an operation, 4 % here, but the rounding it
// needs costs the FP64 sweep 2 % at 100^3.
template <typename T>
__device__ __forceinline__ T cg_direction(T p, T beta, T r, T inv)
{
    if constexpr (sizeof(T) == 8) return __fma_rn(r, inv, __dmul_rn(p, beta));
    else return __fmaf_rn(r, inv, __fmul_rn(p, beta));
}

template <typename T>
__global__ void __launch_bounds__(NTHREADS, 2) cg_resident_kernel(Launch L, int iters)
{
    extern __shared__ __align__(16) unsigned char rsm[];
    __shared__ int s_job, s_ok;
    __shared__ Coef<T> C;
    __shared__ Scalars s_sc;
    __shared__ double s_red[2 * 2 * (NTHREADS / 32)], s_val[2 * kResidentBlocks];
    const int tid = threadIdx.x;
    if (tid == 0) {
        s_job = find_job(L, (int64_t)blockIdx.x);
        s_ok = 1;
    }
    __syncthreads();
    const Job &J = L.jobs[s_job];
    constexpr int W = (int)(sizeof(Scalars) / 4);
    if (tid < W)
        reinterpret_cast<uint32_t *>(&s_sc)[tid] = __ldcg(reinterpret_cast<const uint32_t *>(J.sc) + tid);
    load_coef<T>(C, J, tid);
    __syncthreads();
    // Written at the end of a launch only, so every block of the right-hand
    // side sees the same state.
    if (s_sc.state != RUNNING) return;

    const Geo g{J.nx, J.ny, J.nz, J.dir >> 1, (J.dir & 1) ? -1 : 1, J.pitch};
    const Faces<T> F = faces_of<T>(J);
    const int64_t local = (int64_t)blockIdx.x - J.tile_base;
    const int x0 = (int)(local % J.tiles_x) * TX, y0 = (int)((local / J.tiles_x) % J.tiles_y) * TY;
    const int z0 = (int)(local / ((int64_t)J.tiles_x * J.tiles_y)) * J.zc;
    const int zn = min(J.zc, g.nz - z0);
    const int64_t plane = (int64_t)g.P * g.ny, total = plane * g.nz;
    const T *r_in = (const T *)J.r[0];
    T *r_out = (T *)J.r[0], *x_out = (T *)J.x;

    T(*P)[HY][PW] = reinterpret_cast<T(*)[HY][PW]>(rsm);  // plane z0 - 1 + k
    T *R = reinterpret_cast<T *>(rsm + (size_t)(J.zc + 2) * HY * PW * sizeof(T));
    T *Q = R + (size_t)J.zc * TX * TY;
    uint8_t(*K)[HY][kBoxW] = reinterpret_cast<uint8_t(*)[HY][kBoxW]>(Q + (size_t)J.zc * TX * TY);

    // The box of p and codes (0 outside the domain, for good), the own r.
    {
        const T *p_in = (const T *)J.p[(int)(s_sc.iter & 1)];
        for (int e = tid; e < (zn + 2) * HY * kBoxW; e += NTHREADS) {
            const int col = e % kBoxW, row = e / kBoxW % HY, k = e / (kBoxW * HY);
            const int x = x0 - 1 + col, y = y0 - 1 + row, z = z0 - 1 + k;
            T p = T(0);
            uint8_t code = 0;
            if (g.in(x, y, z)) {
                const int64_t i = g.idx(x, y, z);
                if (ft_in(J, i, i, total, OOB_SWEEP_STORE)) {
                    p = __ldcg(p_in + i);
                    code = __ldg(J.code + i);
                }
            }
            P[k][row][col + 1] = p;
            K[k][row][col] = code;
        }
    }
    // A thread's own points: columns gx, gx + 1 of row ly, every plane.
    const int lp = tid % TPR, ly = tid / TPR;
    const int gx = x0 + 2 * lp, gy = y0 + ly;
    const bool v0 = gx < g.nx && gy < g.ny, v1 = gx + 1 < g.nx && gy < g.ny;
    const int64_t i_own = g.idx(gx, gy, z0);
    const int own = ly * TX + 2 * lp;
    auto own_pair = [&](T *a, int k) -> Pair<T> & { return *reinterpret_cast<Pair<T> *>(a + k * TX * TY + own); };
    for (int k = 0; k < zn; k++) {
        const int64_t i = i_own + plane * k;
        Pair<T> r{T(0), T(0)};
        if (v0 && ft_in(J, i, i + 1, total, OOB_SWEEP_STORE)) r = Pair<T>{__ldcg(r_in + i), __ldcg(r_in + i + 1)};
        own_pair(R, k) = r;
    }
    __syncthreads();
    auto inv_at = [&](int k, int c) {  // own point, 1/diagonal
        return inv_of<T, false>(C, g, K[k + 1][ly + 1][2 * lp + 1 + c], Pos{gx + c, gy, z0 + k, 0});
    };

    // p = p beta + r / diag at a point of the box (as OpCG1).
    auto direction = [&](int k, int row, int col, int x, int y, T r, T beta) {
        const T inv = inv_of<T, false>(C, g, K[k][row][col], Pos{x, y, z0 - 1 + k, 0});
        T &p = P[k][row][col + 1];
        p = cg_direction<T>(p, beta, r, inv);
    };

#if FAST_TAU_TEST_HOOKS
    // an index outside an empty array: the check records it, nothing is accessed
    if (s_sc.test_resident == 1 && tid == 0 && local == J.ntiles - 1) (void)ft_in(J, 0, 0, 0, OOB_SWEEP_STORE);
#endif
    ulonglong2 *slots = (ulonglong2 *)J.slots;
    bool ok = true;
    for (int it = 0; it < iters; it++) {
#if FAST_TAU_TEST_HOOKS
        const bool silent = s_sc.test_resident == 2 && s_sc.iter == 2 && local == J.ntiles - 1;
#else
        constexpr bool silent = false;
#endif
        const T beta = (T)s_sc.beta;
        // Step 1.  The residual around the tile first (the other blocks wrote
        // it before the barrier): the planes below and above, one row on
        // either side of every plane, one column on either side.
        T rz[2][2], ry[2] = {T(0), T(0)}, rx = T(0);
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int z = s ? z0 + zn : z0 - 1;
            rz[s][0] = rz[s][1] = T(0);
            if (v0 && (unsigned)z < (unsigned)g.nz) {
                const int64_t i = g.idx(gx, gy, z);
                if (ft_in(J, i, i + 1, total, OOB_SWEEP_STORE)) {
                    rz[s][0] = __ldcg(r_in + i);
                    rz[s][1] = __ldcg(r_in + i + 1);
                }
            }
        }
        auto row_load = [&](int t, T(&r)[2]) {  // 64 tasks a plane: side, column pair
            const int k = t / (2 * TPR), y = (t / TPR) & 1 ? y0 + TY : y0 - 1, x = x0 + 2 * (t % TPR);
            r[0] = r[1] = T(0);
            if (g.in(x, y, z0 + k)) {
                const int64_t i = g.idx(x, y, z0 + k);
                if (ft_in(J, i, i + 1, total, OOB_SWEEP_STORE)) {
                    r[0] = __ldcg(r_in + i);
                    r[1] = __ldcg(r_in + i + 1);
                }
            }
        };
        auto row_apply = [&](int t, const T(&r)[2]) {
            const int k = t / (2 * TPR), side = (t / TPR) & 1, c = 2 * (t % TPR);
            const int y = side ? y0 + TY : y0 - 1, row = side ? HY - 1 : 0;
            if (g.in(x0 + c, y, z0 + k)) direction(k + 1, row, c + 1, x0 + c, y, r[0], beta);
            if (g.in(x0 + c + 1, y, z0 + k)) direction(k + 1, row, c + 2, x0 + c + 1, y, r[1], beta);
        };
        auto col_load = [&](int t) {  // 16 tasks a plane: side, row
            const int k = t / (2 * TY), x = (t / TY) & 1 ? x0 + TX : x0 - 1, y = y0 + t % TY;
            if (!g.in(x, y, z0 + k)) return T(0);
            const int64_t i = g.idx(x, y, z0 + k);
            return ft_in(J, i, i, total, OOB_SWEEP_STORE) ? __ldcg(r_in + i) : T(0);
        };
        auto col_apply = [&](int t, T r) {
            const int k = t / (2 * TY), side = (t / TY) & 1, row = t % TY;
            const int x = side ? x0 + TX : x0 - 1;
            if (g.in(x, y0 + row, z0 + k)) direction(k + 1, row + 1, side ? TX + 1 : 0, x, y0 + row, r, beta);
        };
        if (tid < zn * 2 * TPR) row_load(tid, ry);
        if (tid < zn * 2 * TY) rx = col_load(tid);
        for (int k = 0; k < zn; k++) {
            const Pair<T> r = own_pair(R, k);
            Pair<T> &p = *reinterpret_cast<Pair<T> *>(&P[k + 1][ly + 1][2 * lp + 2]);
            if (v0) p.a = cg_direction<T>(p.a, beta, r.a, inv_at(k, 0));
            if (v1) p.b = cg_direction<T>(p.b, beta, r.b, inv_at(k, 1));
        }
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int k = s ? zn + 1 : 0;
            if ((unsigned)(z0 - 1 + k) < (unsigned)g.nz) {
                if (v0) direction(k, ly + 1, 2 * lp + 1, gx, gy, rz[s][0], beta);
                if (v1) direction(k, ly + 1, 2 * lp + 2, gx + 1, gy, rz[s][1], beta);
            }
        }
        if (tid < zn * 2 * TPR) row_apply(tid, ry);
        if (tid < zn * 2 * TY) col_apply(tid, rx);
        for (int t = tid + NTHREADS; t < zn * 2 * TPR; t += NTHREADS) {
            T r[2];
            row_load(t, r);
            row_apply(t, r);
        }
        for (int t = tid + NTHREADS; t < zn * 2 * TY; t += NTHREADS) col_apply(t, col_load(t));
        __syncthreads();
        // q = A p on the own points, p.q
        Acc<T> pap;
        for (int k = 0; k < zn; k++) {
            const T(*B)[PW] = P[k + 1];
            const int row = ly + 1, c = 2 * lp + 2;
            const Pair<T> me = *reinterpret_cast<const Pair<T> *>(&B[row][c]);
            const Pair<T> up = *reinterpret_cast<const Pair<T> *>(&B[row + 1][c]);
            const Pair<T> dn = *reinterpret_cast<const Pair<T> *>(&B[row - 1][c]);
            const Pair<T> zp = *reinterpret_cast<const Pair<T> *>(&P[k + 2][row][c]);
            const Pair<T> zm = *reinterpret_cast<const Pair<T> *>(&P[k][row][c]);
            Pair<T> q{T(0), T(0)};
            if (v0) {
                const uint32_t code = K[k + 1][row][2 * lp + 1];
                q.a = stencil7<T>(F, code, me.a, me.b, B[row][c - 1], up.a, dn.a, zp.a, zm.a,
                                  diag_of<T, false>(C, g, code, Pos{gx, gy, z0 + k, 0}));
                pap.add_prod(me.a, q.a);
            }
            if (v1) {
                const uint32_t code = K[k + 1][row][2 * lp + 2];
                q.b = stencil7<T>(F, code, me.b, B[row][c + 2], me.a, up.b, dn.b, zp.b, zm.b,
                                  diag_of<T, false>(C, g, code, Pos{gx + 1, gy, z0 + k, 0}));
                pap.add_prod(me.b, q.b);
            }
            own_pair(Q, k) = q;
        }
        T va[1] = {pap.hi()};
        const uint64_t epoch = s_sc.iter + 1;
        double t1[1];
        if (!(ok = exchange<1, T>(va, slots, local, J.ntiles, epoch, t1, s_red, s_val, &s_ok, silent))) break;
        if (tid == 0) OpCG1<T, T>::finish(s_sc, t1);
        __syncthreads();
        // Step 2.
        const T alpha = (T)s_sc.alpha;
        Acc<T> rr, rzd;
        for (int k = 0; k < zn; k++) {
            const int64_t i = i_own + plane * k;
            if (!v0 || !ft_in(J, i, i + 1, total, OOB_SWEEP_STORE)) continue;
            Pair<T> x = load_pair((const T *)x_out, i);
            const Pair<T> p = *reinterpret_cast<const Pair<T> *>(&P[k + 1][ly + 1][2 * lp + 2]);
            const Pair<T> q = own_pair(Q, k);
            Pair<T> r = own_pair(R, k);
            x.a = x.a + alpha * p.a;
            r.a = r.a + (-alpha) * q.a;
            rr.add_prod(r.a, r.a);
            rzd.add_prod(r.a, r.a * inv_at(k, 0));
            if (v1) {
                x.b = x.b + alpha * p.b;
                r.b = r.b + (-alpha) * q.b;
                rr.add_prod(r.b, r.b);
                rzd.add_prod(r.b, r.b * inv_at(k, 1));
            }
            own_pair(R, k) = r;
            store2<T>(x_out, i, x.a, x.b, true, v1);
            store2<T>(r_out, i, r.a, r.b, true, v1);
        }
        T vb[2] = {rr.hi(), rzd.hi()};
        double t2[2];
        if (!(ok = exchange<2, T>(vb, slots + 1, local, J.ntiles, epoch, t2, s_red, s_val, &s_ok, false))) break;
        if (tid == 0) OpCG2<T, T>::finish(s_sc, t2);
        __syncthreads();
        if (s_sc.state != RUNNING) break;
    }
    if (!ok) {
        if (tid == 0) atomicExch(&J.sc->state, (int32_t)FAULT);
        return;
    }
    // For the next launch: p where its first iteration looks for it, and the
    // scalars (by one block; the others have their copies).  The state only
    // replaces RUNNING: a block that gave up may have marked a FAULT.  The
    // bounds checks' record is the blocks' own (ft_in).
    T *p_out = (T *)J.p[(int)(s_sc.iter & 1)];
    for (int k = 0; k < zn && s_sc.state == RUNNING; k++) {
        const int64_t i = i_own + plane * k;
        const Pair<T> p = *reinterpret_cast<const Pair<T> *>(&P[k + 1][ly + 1][2 * lp + 2]);
        if (v0 && ft_in(J, i, i + 1, total, OOB_SWEEP_STORE)) store2<T>(p_out, i, p.a, p.b, true, v1);
    }
    constexpr int kState = (int)(offsetof(Scalars, state) / 4), kOob = (int)(offsetof(Scalars, oob) / 4);
    if (local == 0 && tid < W) {
        if (tid == kState) atomicCAS(&J.sc->state, (int32_t)RUNNING, s_sc.state);
        else if (tid != kOob) reinterpret_cast<uint32_t *>(J.sc)[tid] = reinterpret_cast<const uint32_t *>(&s_sc)[tid];
    }
}

// Blocks of zc planes that an SM holds: two by their registers, and by their
// shared memory (static arrays 7.5 KB in F64, 12.6 KB in F32; 1 KB a block and
// 1 KB an SM are the system's).
template <typename T>
constexpr int resident_fit(int zc)
{
    const size_t block = resident_smem<T>(zc) + (sizeof(T) == 8 ? 8192 : 13312) + 1024, sm = 227 * 1024 + 1024;
    return zc > kResidentDepth ? 0 : block * 2 <= sm ? 2 : block <= sm ? 1 : 0;
}

template <typename T>
cudaError_t configure_resident()
{
    int zc = kResidentDepth;
    while (resident_fit<T>(zc) == 0) zc--;
    return cudaFuncSetAttribute(cg_resident_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)resident_smem<T>(zc));
}

template <typename T>
cudaError_t launch_resident(const Launch &L, int zc, int iters, cudaStream_t st)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)L.nblocks);
    c.blockDim = dim3(NTHREADS);
    c.dynamicSmemBytes = resident_smem<T>(zc);
    c.stream = st;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeCooperative;
    a[0].val.cooperative = 1;
    c.attrs = a;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, cg_resident_kernel<T>, L, iters);
}

}  // namespace FT_TILES
}  // namespace ft
