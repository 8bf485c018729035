// The steps of a pure-precision solve (F64, and the reference's F32 mode)
// that end an iteration, as pointwise passes: the matrix product they need
// (q = A p of CG, t = A z of BiCGSTAB) is stored by the sweep before them
// instead of being evaluated a second time.
//
// What bounds them: in FP64 the sweeps are bound by the FP64 pipe (about two
// multiply-adds a clock on an SM), not by memory, so 16 bytes per voxel of
// extra traffic buy seven FP64 operations, the halo handling and the
// shared-memory planes.  A block takes the same tile and slab as a sweep's
// block, a thread the same two columns, and adds its dot products in the same
// order, so the partial sums and every scalar are those of the sweep.  U
// planes are loaded before the first is used: two (of 1, 2 and 4, F64 CG
// differs by 1 %; one is 29 % slower in F32 CG at 72 M voxels, four 46 %
// slower in F64 BiCGSTAB at 256^3, where their registers spill).
//
// us per iteration with the product evaluated twice -> stored (both with the
// domain-face table's gain): F64 CG 52.2 -> 27.4 at 64^3, 195.9 -> 88.1 at
// 128^3, 1041 -> 562 at 256^3 (step 2 there 203 us, 4.0 TB/s); F64 BiCGSTAB
// 247 -> 133 at 97 x 83 x 110, 2038 -> 1156 at 256^3; F32 CG 206 -> 165 at
// 256^3, 727 -> 665 at 450 x 400 x 400; F32 BiCGSTAB 473 -> 315 at 256^3.
#pragma once
#include "tau_sweep.cuh"

namespace ft {
inline namespace FT_TILES {

template <class Op, int U>
__global__ void __launch_bounds__(NTHREADS) pointwise_kernel(Launch L)
{
    using T = typename Op::T;
    __shared__ int s_job, s_go, s_flag;
    __shared__ Coef<T> C;
    __shared__ double s_red[2 * Op::NV * (NTHREADS / 32)];
    const int tid = threadIdx.x;
    if (tid == 0) s_job = find_job(L, (int64_t)blockIdx.x);
    __syncthreads();
    const Job &J = L.jobs[s_job];
    if (tid == 0) s_go = J.sc->state == RUNNING ? 1 : 0;
    load_coef<T>(C, J, tid);
    const Geo g{J.nx, J.ny, J.nz, J.dir >> 1, (J.dir & 1) ? -1 : 1, J.pitch};
    const int64_t local = (int64_t)blockIdx.x - J.tile_base;
    const int tx_t = (int)(local % J.tiles_x);
    const int ty_t = (int)((local / J.tiles_x) % J.tiles_y);
    const int tz_t = (int)(local / ((int64_t)J.tiles_x * J.tiles_y));
    const int gx = tx_t * TX + 2 * (tid % TPR), gy = ty_t * TY + tid / TPR;
    const int z0 = tz_t * J.zc, z1 = min(z0 + J.zc, g.nz);
    const bool v0 = gx < g.nx && gy < g.ny, v1 = gx + 1 < g.nx && gy < g.ny;
    const int64_t plane = (int64_t)g.P * g.ny;
    const int64_t i_col = (int64_t)gx + (int64_t)g.P * gy;
    Op op;
    op.init(J);
    __syncthreads();
    if (!s_go) return;
    if (v0) {
        for (int z = z0; z < z1; z += U) {
            typename Op::Vals v[U];
            uint32_t code[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t i = i_col + plane * (z + u);
                // a row is padded to 16 elements, so the pair at gx is inside it
                if (z + u < z1 && ft_in(J, i, i + 1, plane * g.nz, OOB_SWEEP_STORE)) {
                    v[u] = op.load(i);
                    code[u] = *reinterpret_cast<const unsigned short *>(J.code + i);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (z + u >= z1) break;
                const int64_t i = i_col + plane * (z + u);
                typename Op::Out a{}, b{};
                const uint32_t c0 = code[u] & 0xffu, c1 = code[u] >> 8;
                a = op.apply(inv_of<T, false>(C, g, c0, Pos{gx, gy, z + u, 0}), v[u], 0);
                if (v1) b = op.apply(inv_of<T, false>(C, g, c1, Pos{gx + 1, gy, z + u, 0}), v[u], 1);
                if (ft_in(J, i, i + 1, plane * g.nz, OOB_SWEEP_STORE)) op.store(i, a, b, v0, v1);
            }
        }
    }
    T v[Op::NV];
    op.partials(v);
    if (!ft_in(J, local * NPART, local * NPART + NPART - 1, J.ntiles * NPART, OOB_PARTIALS)) return;
    block_sum_store<Op::NV, T>(v, J.part + local * NPART, s_red);
    if (arrive_last(J.counter, J.ntiles, &s_flag)) finish_job<Op, Op::NV>(L, J, s_red);
}

// A pair of neighbouring elements (even index: one vector load).
template <typename T>
__device__ __forceinline__ Pair<T> load_pair(const T *p, int64_t i)
{
    return *reinterpret_cast<const Pair<T> *>(p + i);
}

template <typename T>
__device__ __forceinline__ T lane_of(const Pair<T> &v, int lane) { return lane ? v.b : v.a; }

// CG step 2 on the stored q: x += alpha p, r -= alpha q, z = r/diag, dots
// |r|^2 and r.z (the expressions of OpCG2).
template <typename TT>
struct PwCG2 {
    using T = TT;
    static constexpr int NV = 2;
    struct Vals { Pair<T> p, x, r, q; };
    struct Out { T x, r; };
    const T *p, *q;
    T *x, *r;
    T alpha;
    Acc<T> rr, rz;

    __device__ void init(const Job &J)
    {
        const int par = (int)(J.sc->iter & 1);
        p = (const T *)J.p[par ^ 1];
        q = (const T *)J.q;
        x = (T *)J.x;
        r = (T *)J.r[0];
        alpha = (T)J.sc->alpha;
    }
    __device__ Vals load(int64_t i) const
    {
        return Vals{load_pair(p, i), load_pair(x, i), load_pair(r, i), load_pair(q, i)};
    }
    __device__ Out apply(T inv, const Vals &v, int lane)
    {
        const T xn = lane_of(v.x, lane) + alpha * lane_of(v.p, lane);
        const T rn = lane_of(v.r, lane) + (-alpha) * lane_of(v.q, lane);
        rr.add_prod(rn, rn);
        rz.add_prod(rn, rn * inv);
        return Out{xn, rn};
    }
    __device__ void store(int64_t i, const Out &a, const Out &b, bool v0, bool v1)
    {
        store2<T>(x, i, a.x, b.x, v0, v1);
        store2<T>(r, i, a.r, b.r, v0, v1);
    }
    __device__ void partials(T (&v)[NV]) const { v[0] = rr.hi(); v[1] = rz.hi(); }
    __device__ static void finish(Scalars &sc, const double (&t)[NV]) { OpCG2<T, T>::finish(sc, t); }
};

// BiCGSTAB step 3 on the t that step 2 stored (in the v buffer that step 1
// read and the next step 1 writes): s = r - alpha v, z = s/diag,
// x += alpha y + w z (y = p/diag), r = s - w t, dots r0.r and |r|^2;
// divergence, iteration count, convergence, next rho/beta or a restart.
// BICGSTAB.cu:187-212 + the loop head :93-112.
template <typename TT>
struct PwBi3 {
    using T = TT;
    using ST = TT;
    static constexpr int NV = 2;
    struct Vals { Pair<T> r, v, p, x, r0, t; };
    struct Out { T x, r; };
    const T *r, *v, *p, *r0, *t;
    T *x, *rnew;
    T alpha, omega, nalpha, nomega;
    Acc<T> r0r, rr;

    __device__ void init(const Job &J)
    {
        const int par = (int)(J.sc->iter & 1);
        r = (const T *)J.r[par];
        v = (const T *)J.v[par ^ 1];
        t = (const T *)J.v[par];
        p = (const T *)J.p[par ^ 1];
        r0 = (const T *)J.r0;
        x = (T *)J.x;
        rnew = (T *)J.r[par ^ 1];
        alpha = (T)J.sc->alpha;
        omega = (T)J.sc->omega;
        nalpha = -alpha;
        nomega = -omega;
    }
    __device__ Vals load(int64_t i) const
    {
        return Vals{load_pair(r, i), load_pair(v, i), load_pair(p, i), load_pair(x, i), load_pair(r0, i), load_pair(t, i)};
    }
    __device__ Out apply(T inv, const Vals &a, int lane)
    {
        const T s = lane_of(a.r, lane) + nalpha * lane_of(a.v, lane);
        const T z = s * inv, y = lane_of(a.p, lane) * inv;
        const T xn = lane_of(a.x, lane) + (alpha * y + omega * z);   // __ABC_BetaGammaKernel: x += a*y + w*z
        const T rn = s + nomega * lane_of(a.t, lane);                // __aPlusBetaBKernel(s, t, r, -w)
        r0r.add_prod(lane_of(a.r0, lane), rn);
        rr.add_prod(rn, rn);
        return Out{xn, rn};
    }
    __device__ void store(int64_t i, const Out &a, const Out &b, bool v0, bool v1)
    {
        store2<T>(x, i, a.x, b.x, v0, v1);
        store2<T>(rnew, i, a.r, b.r, v0, v1);
    }
    __device__ void partials(T (&v_)[NV]) const { v_[0] = r0r.hi(); v_[1] = rr.hi(); }
    __device__ static void finish(Scalars &sc, const double (&t_)[NV])
    {
        const ST rsq = (ST)t_[1];
        sc.rsq = rsq;
        if (rsq > (ST)sc.div_thresh) {  // BICGSTAB.cu:206-209, before ++i
            sc.state = DIVERGED;
            return;
        }
        sc.iter += 1;  // BICGSTAB.cu:211
        if (!(rsq > (ST)sc.tol2)) { sc.state = CONVERGED; return; }
        if (sc.iter >= sc.max_iter) { sc.state = MAXITER; return; }
        // Loop head of the next iteration (BICGSTAB.cu:95-112).
        const ST rho_old = (ST)sc.rho;
        const ST rho = (ST)t_[0];
        sc.rho_old = rho_old;
        sc.rho = rho;
        const ST mag = rho < ST(0) ? -rho : rho;
        if (mag < (ST)sc.eps2 * (ST)sc.r0_sq) {
            sc.restart = 1;
        } else {
            sc.beta = (double)((rho / rho_old) * ((ST)sc.alpha / (ST)sc.omega));
        }
    }
};

}  // namespace FT_TILES
}  // namespace ft
