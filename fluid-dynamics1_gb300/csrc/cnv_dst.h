// cnv_dst.h -- exact Poisson solve by discrete sine transforms (internal; cnv_dst.cu).
#pragma once

#include <cuda_runtime.h>

#include "cnv_internal.h"

namespace cnv {

constexpr int kMaxFftStages = 16;  // radices of the FFT length (2s grouped into 8s and 4s)

// One stage of the FFT row transform: radix p after sub-transforms of length L.
struct FftStage {
    int p, L, nb, csoff;                  // nb = N / p butterflies; the radix' table at csoff
    int qt, bt;                           // outputs x butterflies per thread of a large-radix stage
    int pad, cmoff;                       // its cosine and sine matrix: row length (0: none), offset of row 0
    int nbt;                              // ceil(nb / bt)
    unsigned magic_L, magic_nb, magic_nbt;  // division by L, nb, nbt as a high multiply
};

// What the transform kernels take from the plan.
struct FftArgs {
    int n, m, len;                        // grid, interior size m = n - 2, FFT length N = m + 1
    int ld;                               // columns of the work fields (N + 1 or more)
    int nstages;
    FftStage st[kMaxFftStages];
    int fields;                           // float2 of shared memory for a row's two buffers
    // tables, one after the other (byte offsets): tw exp(-2 pi i t / N); sc (sin, cos)(pi j / N), j = 0 .. N/2; li, lj the
    // eigenvalue parts of the integer stencil by mode number; cm the cosine and sine matrices of the large radices; cs
    // per stage (cos, sin)(2 pi t / p)
    const char* tables;
    int off_sc, off_li, off_lj, off_cm, off_cs, table_bytes;
    float norm;                           // (2 / N)^2: the four orthonormal transforms
    double norm64;
    long long a2, b2;                     // the stencil a2 (along i) + b2 (along j): (Ly : Lx) squared, in lowest terms
    float* t;                             // (m + 2) x ld transform field
    double* t64;                          // the same of the FP64 form
    float* e0;                            // (m + 2) x ld first solution, zero outside the interior
    long long* psi;                       // (m + 2) x ld solution in fixed point, zero outside the interior
    int* ex;                              // per row of `in`: its largest biased exponent
    unsigned* mx;                         // per row of e0: its largest magnitude (float bits)
    int* ctl;                             // exponent E of the right-hand side, shift S of the fixed point, grid barrier, its ticket
    int cols_b;                           // columns per block of pass B
};

struct DstPlan {
    int n = 0, m = 0;          // grid size and interior size m = n - 2
    double dx2 = 0, dy2 = 0;
    // FFT row transforms with refinement (F.len > 0), else dense FP64 products with S
    FftArgs F{};
    int threads_a = 0, threads_b = 0, smem_a = 0, smem_b = 0;
    int form = 0;              // the passes' form (cnv_dst.cu)
    bool one_launch = false;   // all passes in one cooperative launch, whose waits report to ctrl
    bool fp64 = false;         // in FP64 at once (small grids)
    bool far = false;          // residual modulo 2^128 (very stretched cells)
    Ctrl* ctrl = nullptr;
    long long timeout_ns = 0;
    int stall_block = -1;      // testing only: a block of the one-launch forms that never arrives at their barriers
    int solves = 3;            // FP32 solves, each of the residual the ones before left
    double kappa = 1;          // the equation's operator over the integer stencil
    int rows = 4;              // rows per block of the dense product kernel
    double* S = nullptr;       // m x m orthonormal DST-I matrix (symmetric), dense path only
    double* lam_i = nullptr;   // 4 dy^2 sin^2(pi (a+1) / (2 (m+1))): the eigenvalue part along i (dense path)
    double* lam_j = nullptr;   // 4 dx^2 sin^2(pi (b+1) / (2 (m+1))): along j
    double* t1 = nullptr;      // m x m scratch between the dense passes
    double* t2 = nullptr;
    void* arena = nullptr;     // the FFT path's tables and fields
};

// Lx and Ly are the cavity's extents (dx = Lx / n, dy = Ly / n). ctrl takes the status and the abort flag
// of a solve whose blocks wait for one another (bounded by timeout_ns). stall_block: see DstPlan (-1: none).
int dst_plan_create(int n, int Lx, int Ly, Ctrl* ctrl, long long timeout_ns, int stall_block, DstPlan* plan);
// Re-arm the barrier after a solve that timed out: once before the solves of a call.
cudaError_t dst_reset(const DstPlan& plan, cudaStream_t s);
void dst_plan_destroy(DstPlan* plan);

// out(interior) = M^-1 (scale * in(interior)): in and out are n x n row-major; the edges of
// `in` are not read and the edges of `out` are not written. With scale = c4 and in = w this
// is the converged streamfunction of the reference's solver for f = -w.
cudaError_t dst_solve(const DstPlan& plan, const double* in, double scale, double* out, cudaStream_t s);
// The same solve with the result written into the red/black split layout (the layout the
// velocity pass reads); edge cells are not written.
cudaError_t dst_solve_split(const DstPlan& plan, const double* in, double scale, double* red, double* black,
                            int pitch, cudaStream_t s);

}  // namespace cnv
