// Host-side launchers of the device kernels (one translation unit per
// precision family so the build compiles them in parallel).
#pragma once
#include <cuda_runtime.h>
#include "tau_types.h"

namespace ft {

enum class Step {
    INIT_CG, INIT_BI, CG1, CG2, CG2_Q, BI_RESTART, BI1, BI2, BI3, REPLACE_CG, REPLACE_BI, BI_K1, BI_K2, CG_F,
    REPLACE_CG_FF, REPLACE_BI_FF  // the replacement with a float-float iterate (opt-in)
};

// The solver kernels of a tile W columns wide (64, or 32 for CG alone).
template <int W>
struct Kernels {
    // Pure-precision solves (scalars in the solve precision, as the
    // reference's T).
    static void pure_f64(Step s, const Launch &L, cudaStream_t st);
    static void pure_f32(Step s, const Launch &L, cudaStream_t st);
    // FP32 iterations of a MIXED solve (scalars in double); BI_K1/BI_K2 are
    // the two-sweep BiCGSTAB steps, MIXED only.
    static void mixed_inner(Step s, const Launch &L, cudaStream_t st);
    // Residual replacement of a MIXED solve (a no-op launch unless the solve
    // asked for one): FP64 iterate, or float-float with `ff`.
    static void replace(bool bicg, bool ff, const Launch &L, cudaStream_t st);
    // CG of volumes whose blocks of zc planes all fit on the GPU at once:
    // `iters` iterations in one cooperative launch (tau_resident.cuh), and the
    // blocks of zc planes that an SM holds (at most two, by their registers).
    static cudaError_t resident_f64(const Launch &L, int zc, int iters, cudaStream_t st);
    static cudaError_t resident_f32(const Launch &L, int zc, int iters, cudaStream_t st);
    static int resident_per_sm(bool f32, int zc);
    // Raise the dynamic shared-memory limit of every sweep kernel (once per
    // device).
    static cudaError_t configure_f64();
    static cudaError_t configure_f32();
    static cudaError_t configure_replace();
};
constexpr int kResidentDepth = 24;  // planes per block at most
constexpr int kResidentBlocks = 2 * 152;
constexpr size_t kResidentSlotBytes = 48;  // of a block, in Job::slots, zero before the first launch

void launch_init64(const Launch &L, cudaStream_t st);
// Adds the zero bytes of mask[0..n) (16-byte aligned) to *total.
void launch_count_zero(const uint8_t *mask, uint64_t n, unsigned long long *total, cudaStream_t st);
void launch_code(const Launch &L, cudaStream_t st);
// Fills the domain-face tables (Job::bnd) of the first `count` of jobs[job[0..2]]
// (device table): one job per primary axis.
void launch_bnd(bool f32, const Job *jobs, const int (&job)[3], int count, cudaStream_t st);
// tau flux sum: src 0 = double x, 1 = float x, 2 = the current MIXED iterate
// as float-float pairs, 3 = the current MIXED iterate as doubles.
void launch_tau(int src, const Launch &L, cudaStream_t st);
// n float-float pairs at src -> n doubles at dst (device).
void launch_ff_to_double(const void *src, double *dst, int64_t n, cudaStream_t st);

}  // namespace ft
