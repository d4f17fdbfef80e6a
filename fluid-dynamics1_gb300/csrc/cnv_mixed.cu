// cnv_mixed.cu -- mixed-precision Poisson solve: FP32 red-black SOR sweeps inside FP64 defect
// correction, one persistent cooperative launch per solve.
//
// The equation is the reference's discrete Poisson problem (src/poisson.c:247 at its fixed
// point), written with the scaled right-hand side g = dx^2 dy^2 f that the transport pass
// produces:
//     dy^2 (psi[i+1][j] + psi[i-1][j]) + dx^2 (psi[i][j+1] + psi[i][j-1]) - den psi[i][j] = g[i][j]
// on the interior, psi = 0 on the edge, den = 2 (dx^2 + dy^2). Defect correction:
//     psi = 0 (FP64)
//     loop: R = g - A psi (FP64); stop when ||R||_2 <= rtol ||g||_2
//           solve A e = R approximately with `epochs * kSweepsPerExchange` FP32 red-black SOR
//           sweeps from e = 0
//           psi += e (FP64)
// Only the residual, the norm and the correction accumulation are FP64; every sweep is FP32.
//
// Layout. g, psi, the FP32 correction right-hand side R/den and the FP32 border-exchange copies
// of e all use the red/black split layout of the rest of the library (colour c = (i+j)&1 of cell
// (i, j) at A_c[i*pitch + (j>>1)]), and so does the shared-memory tile: every access in a sweep
// is unit-stride, and warps walk whole rows, so no integer division is needed per cell.
//
// Inner sweeps. Each block owns one tile and keeps e on the tile plus a halo of width
// H = 2*kSweepsPerExchange in shared memory. An "epoch" is kSweepsPerExchange red-black sweeps
// done entirely in shared memory: half-sweep s updates its colour on the tile grown by H - s
// cells on every side (clipped to the interior), so after 2*kSweepsPerExchange half-sweeps the
// tile holds exactly what global red-black SOR would hold. The redundant halo work buys one
// neighbour exchange per epoch instead of one per half-sweep. At an epoch's end every block
// writes its border strips (width H) into a global FP32 copy of e (double-buffered by epoch
// parity) and raises its flag; the next epoch waits for the eight neighbours' flags and loads
// their strips into the halo. Tiles are at least H cells wide and tall, so a halo only ever
// comes from the eight adjacent tiles.
//
// All waits are bounded (timeout + abort flag) and report CNV_TIMEOUT instead of hanging.
#include <algorithm>
#include <cfloat>

#include "cnv_kernels.h"
#include "cnv_stencil.cuh"
#include "cnv_sync.cuh"

namespace cnv {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kSweepsPerExchange = 8;  // k_mixed at 1024^2: 4: 4.05 us per sweep, 8: 3.45, 12: 3.40, 16: 3.47
constexpr int kHalo = 2 * kSweepsPerExchange;

struct MixedSync {
    unsigned int bar_count;     // grid barrier (outer iterations)
    unsigned int pad;
    double partial[2][kMaxSolverBlocks];  // per-block ||R||^2 and ||g||^2
    unsigned int flag[kMaxSolverBlocks];  // last epoch whose border strips a block has written
};

// Grid-wide barrier (counter of arrivals); false if it timed out or another block aborted.
__device__ bool grid_sync(MixedSync* sy, unsigned& epoch, Ctrl* ctl, long long timeout_ns, int* s_ok) {
    __syncthreads();
    ++epoch;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&sy->bar_count, 1u);
        *s_ok = wait_geq(&sy->bar_count, epoch * gridDim.x, ctl, timeout_ns) ? 1 : 0;
        __threadfence();
    }
    __syncthreads();
    return *s_ok != 0;
}

struct MTile {
    int r0, r1, c0, c1;  // owned rows/cols (absolute)
    int nb[8];           // the eight adjacent tiles' blocks, -1 where there is none
};

// First column of tile column x of gx: the interior columns 1 .. n-2 shared out evenly, the inner bounds a multiple of
// `align` columns from the first.
__host__ __device__ __forceinline__ int mtile_col(int n, int gx, int x, int align) {
    const int c = 1 + (int)((long long)(n - 2) * x / gx);
    return x == gx ? c : 1 + (c - 1 + align / 2) / align * align;
}

__device__ __forceinline__ MTile make_mtile(int n, int gx, int gy, int b, int align) {
    MTile t;
    const int ni = n - 2;
    const int tx = b % gx, ty = b / gx;
    t.c0 = mtile_col(n, gx, tx, align);
    t.c1 = mtile_col(n, gx, tx + 1, align);
    t.r0 = 1 + (int)((long long)ni * ty / gy);
    t.r1 = 1 + (int)((long long)ni * (ty + 1) / gy);
    int k = 0;
    for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
            if (!dx && !dy) continue;
            const int x = tx + dx, y = ty + dy;
            t.nb[k++] = (x >= 0 && x < gx && y >= 0 && y < gy) ? y * gx + x : -1;
        }
    return t;
}

// Shared-memory tile in split layout: rows sr0 .. sr0+sh-1, global split columns m0 .. m0+swm-1.
struct SmemTile {
    int sr0, sh, m0, swm;
    float* c[2];
    __device__ __forceinline__ float& at(int col, int i, int m) const { return c[col][(i - sr0) * swm + (m - m0)]; }
};

}  // namespace

size_t mixed_sync_bytes() { return sizeof(MixedSync); }

// Shared-memory bytes the mixed kernel needs for the largest tile of a gx x gy tiling of n:
// e (both colours) on the tile plus halo, and the same again when the correction right-hand side
// is also kept there (rq_in_smem).
size_t mixed_smem_bytes(int n, int gx, int gy, bool rq_in_smem) {
    const int ni = n - 2;
    const int tw = (ni + gx - 1) / gx + 2 * kHalo;
    const int th = (ni + gy - 1) / gy + 2 * kHalo;
    const int swm = tw / 2 + 2;
    return (rq_in_smem ? 4 : 2) * (size_t)th * swm * sizeof(float);
}

namespace {

// The dynamic shared memory of k_mixed. The hot loop addresses it through this array with
// integer offsets, so every access compiles to a shared-memory load or store.
extern __shared__ float mx_smem[];

// One colour c of an FP32 red-black SOR half-sweep on rows [lo_r, hi_r), columns [lo_c, hi_c) of
// the shared-memory tile (split layout: row i of colour k at mx_smem[k_off + (i - sr0) * swm + (m -
// m0)]): e of colour c at sc_off, of the other colour at so_off; the correction right-hand side
// R/den at rq_off in shared memory (RQ_SMEM) or in the global split array rq (pitch P). Kept out
// of line so that it gets its own register allocation: it is the hot loop of the solve.
template <bool RQ_SMEM>
__device__ __noinline__ void mixed_half_sweep(int sc_off, int so_off, int rq_off, const float* __restrict__ rq,
                                              int sr0, int swm, int m0, int lo_r, int hi_r, int lo_c, int hi_c,
                                              int c, int P, float wx, float wy, float beta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = lo_r + warp; i < hi_r; i += kWarps) {
        const int q = (i + c) & 1;
        const int mlo = floor_half(lo_c - q + 1), mhi = floor_half(hi_c - 1 - q);
        const int row = (i - sr0) * swm - m0;
        const float* rqrow = rq + (size_t)i * P;
        // unrolled 4 deep where R/den comes from L2 (the large grids): 2048^2 8.87 vs 9.18 us per
        // sweep; with R/den in shared memory (1024^2) unrolling ran slower (3.50 vs 3.46), and the
        // batch kernel's strip sweep, the same loop, ran its step 24 % slower unrolled
#pragma unroll(RQ_SMEM ? 1 : 4)
        for (int m = mlo + lane; m <= mhi; m += 32) {
            const int k = row + m;
            const float up = mx_smem[so_off + k + swm], dn = mx_smem[so_off + k - swm];
            const float lt = mx_smem[so_off + k - 1 + q], rt = mx_smem[so_off + k + q];
            // R/den: shared-memory copy, or L2 (rewritten every outer iteration)
            const float r = RQ_SMEM ? mx_smem[rq_off + k] : __ldcg(rqrow + m);
            const float me = mx_smem[sc_off + k];
            const float gs = fmaf(wy, up + dn, fmaf(wx, lt + rt, -r));
            mx_smem[sc_off + k] = fmaf(beta, gs - me, me);
        }
    }
}

// FP64 residual R = g - A psi on the block's own cells, its norm's (and in outer iteration 0 |g|'s) partial sums, and
// the FP32 right-hand side R/den of the correction: cell (i, j) of colour c at rq[c][i * pitch + ((j - first) >> 1)].
// WARPS: the block's warps (0: blockDim.x / 32), so that the last sum's loads are issued together.
template <int FIRST, int WARPS>
__device__ __forceinline__ void mixed_residual(const MixedLaunch& L, const MTile& t, MixedSync* sy, int outer,
                                               double (*s_red)[2]) {
    const int P = L.pitch, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = WARPS ? WARPS : blockDim.x >> 5;
    const double dx2 = L.dx2, dy2 = L.dy2, den = L.den;
    double rr = 0.0, gg = 0.0;
    for (int i = t.r0 + warp; i < t.r1; i += warps) {
        for (int c = 0; c < 2; ++c) {
            const int q = (i + c) & 1;  // cell (i, j) of colour c has j = 2m + q
            const int mlo = floor_half(t.c0 - q + 1), mhi = floor_half(t.c1 - 1 - q);
            const double* pc = L.psi[c];
            const double* po = L.psi[c ^ 1];
            for (int m = mlo + lane; m <= mhi; m += 32) {
                const size_t k = (size_t)i * P + m;
                const double g = L.g[c][k];
                const double R = poisson_defect(dy2, dx2, den, __ldcg(po + k + P), __ldcg(po + k - P),
                                                __ldcg(po + k - 1 + q), __ldcg(po + k + q), __ldcg(pc + k), g);
                rr = fma(R, R, rr);
                if (outer == 0) gg = fma(g, g, gg);
                L.rq[c][FIRST ? k - 1 + q : k] = (float)(R * L.rden);
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        rr += __shfl_xor_sync(0xffffffffu, rr, off);
        gg += __shfl_xor_sync(0xffffffffu, gg, off);
    }
    if (lane == 0) {
        s_red[warp][0] = rr;
        s_red[warp][1] = gg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < warps; ++w) {
            a += s_red[w][0];
            b += s_red[w][1];
        }
        sy->partial[0][blockIdx.x] = a;
        if (outer == 0) sy->partial[1][blockIdx.x] = b;
    }
}

// |R| / |g| from every block's partial sums (after a grid barrier); the same in every thread.
__device__ __forceinline__ double mixed_norm(MixedSync* sy, double* s_tot) {
    if (threadIdx.x < 32) {
        double a = 0.0, b = 0.0;
        for (int q = threadIdx.x; q < (int)gridDim.x; q += 32) {
            a += __ldcg(&sy->partial[0][q]);
            b += __ldcg(&sy->partial[1][q]);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, off);
            b += __shfl_xor_sync(0xffffffffu, b, off);
        }
        if (threadIdx.x == 0) {
            s_tot[0] = a;
            s_tot[1] = b;
        }
    }
    __syncthreads();
    const double rnorm = sqrt(s_tot[0]), gnorm = sqrt(s_tot[1]);
    __syncthreads();
    return gnorm > 0 ? rnorm / gnorm : rnorm;
}

// Waits until the eight neighbours have written their strips of `epoch`. False on a timeout or abort.
__device__ __forceinline__ bool mixed_wait(const MixedLaunch& L, const MTile& t, MixedSync* sy, unsigned epoch, int* s_flag) {
    if (threadIdx.x < 8) {
        const int nb = t.nb[threadIdx.x];
        s_flag[threadIdx.x] = nb < 0 ? 1 : (wait_geq(&sy->flag[nb], epoch, L.ctrl, L.timeout_ns) ? 1 : 0);
    }
    __syncthreads();
    bool ok = true;
    for (int q = 0; q < 8; ++q) ok = ok && s_flag[q];
    return ok;
}

// The solve's result into the control block and the step record (one thread of the grid).
__device__ __forceinline__ void mixed_report(const MixedLaunch& L, int outer, int status, double rel, long long sweeps) {
    Ctrl* ctl = L.ctrl;
    ctl->iters = outer;
    ctl->err = rel;
    ctl->status = status;
    ctl->sweeps += sweeps;
    const int step = ctl->step;
    if (step < ctl->max_records) {
        StepRecord& r = ctl->records[step];
        r.iters = outer;
        r.status = status;
        r.err = rel;
        r.cont_max = 0.0;
        r.cont_min = 0.0;
    }
    if (status != CNV_OK) ctl->abort = 1;
}

__global__ void __launch_bounds__(kThreads, 1) k_mixed(MixedLaunch L) {
    Ctrl* ctl = L.ctrl;
    if (ctl->abort) return;
    float* const s_mem = mx_smem;
    __shared__ int s_ok;
    __shared__ int s_flag[8];
    __shared__ double s_red[kWarps][2];
    __shared__ double s_tot[2];
    MixedSync* sy = reinterpret_cast<MixedSync*>(L.sync);
    const int n = L.n, P = L.pitch;
    const MTile t = make_mtile(n, L.gx, L.gy, blockIdx.x, 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    SmemTile S;
    S.sr0 = t.r0 - kHalo;
    S.sh = t.r1 - t.r0 + 2 * kHalo;
    S.m0 = floor_half(t.c0 - kHalo);
    S.swm = floor_half(t.c1 + kHalo - 1) - S.m0 + 1;
    S.c[0] = s_mem;
    S.c[1] = s_mem + S.sh * S.swm;
    const int ssz = 2 * S.sh * S.swm;
    // correction right-hand side tile (both colours) after e, when it fits in shared memory
    float* const srq = L.rq_in_smem ? s_mem + ssz : nullptr;

    const float wx = (float)(L.dx2 / L.den), wy = (float)(L.dy2 / L.den), beta = (float)L.beta;
    unsigned bar = 0, ep = 0;
    int outer = 0, status = CNV_NOT_CONVERGED;
    long long sweeps = 0;
    double rel = 0.0;

    for (outer = 0;; ++outer) {
        mixed_residual<0, kWarps>(L, t, sy, outer, s_red);
        if (!grid_sync(sy, bar, ctl, L.timeout_ns, &s_ok)) { status = CNV_TIMEOUT; break; }
        rel = mixed_norm(sy, s_tot);
        if (!isfinite(rel)) { status = CNV_NONFINITE; break; }
        if (rel <= L.rtol) { status = CNV_OK; break; }
        if (outer >= L.max_outer) break;
        if (srq) {
            // R/den on the tile plus halo (every block wrote its own cells before the barrier)
            for (int r = warp; r < S.sh; r += kWarps) {
                const int i = S.sr0 + r;
                for (int c = 0; c < 2; ++c) {
                    const int q = (i + c) & 1;
                    float* dst = srq + c * (S.sh * S.swm) + r * S.swm;
                    for (int mm = lane; mm < S.swm; mm += 32) {
                        const int j = 2 * (S.m0 + mm) + q;
                        dst[mm] = (i >= 1 && i <= n - 2 && j >= 1 && j <= n - 2)
                                      ? __ldcg(L.rq[c] + (size_t)i * P + S.m0 + mm)
                                      : 0.0f;
                    }
                }
            }
            __syncthreads();
        }

        // ---- FP32 inner solve: e = 0, then `epochs` epochs of kSweepsPerExchange sweeps
        for (int x = threadIdx.x; x < ssz; x += kThreads) s_mem[x] = 0.0f;
        __syncthreads();
        bool ok = true;
        for (int e = 0; e < L.epochs && ok; ++e) {
            ++ep;
            if (e > 0) {
                // neighbours' border strips of the previous epoch -> halo
                ok = mixed_wait(L, t, sy, ep - 1, s_flag);
                if (!ok) break;
                // one flat loop over the tile-plus-halo box: every thread issues its few
                // independent L2 loads at once (a warp walking rows would wait for each in turn)
                const int par = (ep - 1) & 1;
                const int box = S.sh * S.swm;
                for (int x = threadIdx.x; x < box; x += kThreads) {
                    const int r = x / S.swm;
                    const int i = S.sr0 + r;
                    if (i < 1 || i > n - 2) continue;
                    const int m = S.m0 + (x - r * S.swm);
                    const bool own_row = i >= t.r0 && i < t.r1;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int j = 2 * m + ((i + c) & 1);
                        if (j < max(1, t.c0 - kHalo) || j >= min(n - 1, t.c1 + kHalo)) continue;
                        if (own_row && j >= t.c0 && j < t.c1) continue;  // own cell: already current
                        S.at(c, i, m) = __ldcg(L.eg[par][c] + (size_t)i * P + m);
                    }
                }
                __syncthreads();
            }
            for (int s = 1; s <= 2 * kSweepsPerExchange; ++s) {
                const int c = (s - 1) & 1;  // red first
                const int lo_r = max(1, t.r0 - kHalo + s), hi_r = min(n - 1, t.r1 + kHalo - s);
                const int lo_c = max(1, t.c0 - kHalo + s), hi_c = min(n - 1, t.c1 + kHalo - s);
                const int plane = S.sh * S.swm;  // e colour k at k * plane, R/den colour k at (2 + k) * plane
                if (srq)
                    mixed_half_sweep<true>(c * plane, (c ^ 1) * plane, (2 + c) * plane, L.rq[c], S.sr0, S.swm,
                                           S.m0, lo_r, hi_r, lo_c, hi_c, c, P, wx, wy, beta);
                else
                    mixed_half_sweep<false>(c * plane, (c ^ 1) * plane, 0, L.rq[c], S.sr0, S.swm, S.m0, lo_r,
                                            hi_r, lo_c, hi_c, c, P, wx, wy, beta);
                __syncthreads();
            }
            sweeps += kSweepsPerExchange;
            if (e + 1 < L.epochs) {
                // own border strips (width H) -> global copy of this epoch; raise the flag
                const int par = ep & 1;
                const int tw = t.c1 - t.c0, th = t.r1 - t.r0;
                for (int x = threadIdx.x; x < tw * th; x += kThreads) {
                    const int r = x / tw;
                    const int i = t.r0 + r;
                    const int j = t.c0 + (x - r * tw);
                    if (i >= t.r0 + kHalo && i < t.r1 - kHalo && j >= t.c0 + kHalo && j < t.c1 - kHalo) continue;
                    const int c = (i + j) & 1;
                    L.eg[par][c][(size_t)i * P + (j >> 1)] = S.at(c, i, j >> 1);
                }
                __syncthreads();
                if (threadIdx.x == 0 && (int)blockIdx.x != L.stall_block) st_release(&sy->flag[blockIdx.x], ep);
            }
        }
        if (!ok) { status = CNV_TIMEOUT; break; }
        // ---- FP64 correction psi += e on own cells
        for (int i = t.r0 + warp; i < t.r1; i += kWarps) {
            for (int c = 0; c < 2; ++c) {
                const int q = (i + c) & 1;
                const int mlo = floor_half(t.c0 - q + 1), mhi = floor_half(t.c1 - 1 - q);
                double* pc = L.psi[c];
                for (int m = mlo + lane; m <= mhi; m += 32) pc[(size_t)i * P + m] += (double)S.at(c, i, m);
            }
        }
        if (!grid_sync(sy, bar, ctl, L.timeout_ns, &s_ok)) { status = CNV_TIMEOUT; break; }
    }
    if (status == CNV_TIMEOUT) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) mixed_report(L, outer, status, rel, sweeps);
}

// ---------------------------------------------------------------------------------------
// The same solve with e in registers, the default (k_mixed above takes the smallest grids and the largest, where no box fits).
// k_mixed moves seven shared-memory words per cell and half-sweep and spends about 20 instructions on it. Here a thread keeps a
// patch of e (and of R/den, or that in shared memory, private to the thread) for the whole inner solve; a half-sweep takes six
// packed FP32 instructions per two cells, and only patch borders go through shared memory. Microseconds per sweep, k_mixed ->
// this kernel, the exchange of the halo included, the same bits: 64^2 1.99 -> 1.26, 256^2 1.78 -> 0.90, 512^2 2.21 -> 0.82,
// 1024^2 3.45 -> 1.12, 1500^2 5.04 -> 1.89, 2048^2 8.85 -> 2.40. At 1024^2 a half-sweep takes 700 cycles, where its
// operations on the box need 330 of the FP32 pipe, and an exchange 7,000 per 16 of them.
//
// Box. A block works on a box of 8 ntx columns and BH = 2 PH nty rows around its tile with at least kHalo cells (or the wall) on
// every side. Cells outside the box count as 0: at a wall that is the boundary value, elsewhere the error moves in by one cell
// per half-sweep and stays kHalo half-sweeps away from the tile, like the values a shrinking region would leave out. So every
// cell of the box is updated in every half-sweep with no test, and the tile holds what global red-black sweeps give, bit for
// bit. The rows lie inside the interior (1 <= sr0, sr0 + BH <= n - 1). The columns start a multiple of 8 from column 1, as the
// tiles do, so that a thread's cells are 16-byte vectors of the exchanged fields (whose split layout counts from column 1 for
// that), all of them in the tile or none. Where n - 2 is no multiple of 8 the last tiles' boxes hold the right wall: that column
// is kept at 0 by a SOR factor of 0, and what lies beyond it stays 0 by itself.
//
// Patch. Thread (tx, ty) owns 2 PH rows from sr0 + 2 PH ty on and, of each colour, 4 cells of each row: local colour c of row k
// is at columns 8 tx + 2 u + ((k + c) & 1) of the box (PH is even, so the parity of k is the row's); local colours are the
// grid's, or swapped when sr0 is even. Rows k and k + PH form the two halves of a packed pair (f32x2): every neighbour of a pair
// is a pair too, except in the first and last row, which take single adds. A cell's neighbours in its row are the other
// colour's u and u-1 (or u+1); a row of a colour needs one cell from one side, and passes one on. Larger patches pass less
// through shared memory per cell and have more independent work per thread, so few threads with many registers win: cycles per
// sweep at 1024^2 (box 160 x 88) 2467 with 2 x 2 pairs of a colour and 896 threads, 2009 with 2 x 4 and 448, 1407 with 4 x 4
// and 224; us per sweep at 2048^2 (288 x 144) 3.86 with 4 x 8 and 352 threads of 168 registers, 2.47 with 4 x 10 and 252 of 255.
typedef unsigned long long pair_t;  // two floats

__device__ __forceinline__ pair_t pk(float lo, float hi) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo_of(pair_t a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi_of(pair_t a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
    pair_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
    pair_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Halo cells with their epoch: two cells per access, each a 64-bit word with the epoch above the value. A vector access is only
// whole element by element, so the word, not the vector, is what keeps a value and its epoch together; a reader then needs no
// flag, and the writer no fence.
__device__ __forceinline__ ulonglong2 ld_cells(const uint2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_cells(uint2* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ unsigned long long tagged(unsigned value, unsigned epoch) {
    return (unsigned long long)epoch << 32 | value;
}

extern __shared__ ulonglong2 mr_smem[];

// A thread's place in the box.
struct Patch {
    int tx, ty, ntx, nty;
    int up, dn;         // threads above and below (at the box' ends blockDim.x: a vector of zeros)
    bool on;            // a thread of the box with a column inside the walls
    int wall;           // column of the right wall in the patch, 2u + q (or a number it does not have)
};

constexpr int PW = 4;  // cells of a colour per row of a patch

template <int V> struct Int { static constexpr int value = V; };

// Shared memory: the exchanged borders of one colour (or of both, DB): the last row of every patch, the first, each with
// a vector of zeros after them, and a side cell pair per row; then R/den (!RREG). In units of 16 bytes.
template <int PH, bool RREG, bool DB>
struct MrShape {
    static constexpr int kV = PW / 2;  // 16-byte vectors per row of pairs
    static __host__ __device__ constexpr int border(int threads) { return 2 * (threads + 1) + PH / 2 * threads; }
    static __host__ __device__ constexpr int units(int threads) {
        return (DB ? 2 : 1) * border(threads) + (RREG ? 0 : 2 * PH * kV * threads);
    }
};

// The sweeps' weights as pairs, and for each cell of a row on the wall's side of the parity the SOR factor, 0 on the wall: a
// cell there starts at 0 and stays 0 (setting it back after each half-sweep took the wall's blocks 19 % longer, and the others wait
// for them).
template <int WALL>
struct MrWeights {
    pair_t wx, wy, beta, minus, at_wall[WALL ? PW : 1];
};

// The borders of colour C that the other colour's half-sweep reads: first and last row of the patch, and a cell per row.
template <int C, int PH, bool RREG, bool DB>
__device__ __forceinline__ void mr_publish(const pair_t (&E)[2][PH][PW], ulonglong2* out) {
    const int T = blockDim.x, tid = threadIdx.x;
    const pair_t *top = E[C][PH - 1], *bot = E[C][0];
    float4* rows = reinterpret_cast<float4*>(out);
    rows[tid] = make_float4(hi_of(top[0]), hi_of(top[1]), hi_of(top[2]), hi_of(top[3]));          // read by the thread above
    rows[T + 1 + tid] = make_float4(lo_of(bot[0]), lo_of(bot[1]), lo_of(bot[2]), lo_of(bot[3]));  // by the one below
    pair_t* ps = reinterpret_cast<pair_t*>(out + 2 * (T + 1));
#pragma unroll
    for (int k = 0; k < PH; ++k)  // the other colour's row k reads its left (even k + 1 - C) or right neighbour
        ps[k * T + tid] = ((k + 1 - C) & 1) ? E[C][k][0] : E[C][k][PW - 1];
}

// One half-sweep of local colour C; the borders of the other colour are in shared memory and a barrier has passed since. Ends
// with its own borders there and a barrier. WALL 1 (2): the block's box
// holds the right wall, in an even (odd) column 2u (2u + 1) of a patch.
template <int C, int PH, bool RREG, bool DB, int WALL>
__device__ __forceinline__ void mr_half(pair_t (&E)[2][PH][PW], const pair_t (&R)[RREG ? 2 : 1][RREG ? PH : 1][PW],
                                        const Patch& p, const MrWeights<WALL>& W) {
    using S = MrShape<PH, RREG, DB>;
    constexpr int O = 1 - C;
    const int T = blockDim.x, tid = threadIdx.x, B = S::border(T);
    ulonglong2* in = mr_smem + (DB ? O * B : 0);
    ulonglong2* out = mr_smem + (DB ? C * B : 0);
    const ulonglong2* rs = mr_smem + (DB ? 2 : 1) * B + C * PH * S::kV * T;
    if (p.on) {
        const float4 below4 = reinterpret_cast<const float4*>(in)[p.dn], above4 = reinterpret_cast<const float4*>(in)[T + 1 + p.up];
        const float below[PW] = {below4.x, below4.y, below4.z, below4.w}, above[PW] = {above4.x, above4.y, above4.z, above4.w};
        // rows whose cells lie left of the other colour's take the left neighbour's last cell, the others the right one's first
        const bool left = p.tx > 0, right = p.tx < p.ntx - 1;
        const pair_t* ps = reinterpret_cast<const pair_t*>(in + 2 * (T + 1));
        pair_t side[PH];
#pragma unroll
        for (int k = 0; k < PH; ++k) {
            const bool q = (k + C) & 1;
            side[k] = (q ? right : left) ? ps[k * T + tid + (q ? 1 : -1)] : 0ull;
        }
#pragma unroll
        for (int k = 0; k < PH; ++k) {
            const int q = (k + C) & 1;
            pair_t r[PW];
            if constexpr (!RREG) {
#pragma unroll
                for (int v = 0; v < S::kV; ++v) {
                    const ulonglong2 x = rs[(k * S::kV + v) * T + tid];
                    r[2 * v] = x.x;
                    r[2 * v + 1] = x.y;
                }
            }
#pragma unroll
            for (int u = 0; u < PW; ++u) {
                pair_t vert;  // up + down
                if (k == 0) {
                    const pair_t up = E[O][1][u];
                    vert = pk(__fadd_rn(lo_of(up), below[u]), __fadd_rn(hi_of(up), lo_of(E[O][PH - 1][u])));
                } else if (k == PH - 1) {
                    const pair_t dn = E[O][PH - 2][u];
                    vert = pk(__fadd_rn(hi_of(E[O][0][u]), lo_of(dn)), __fadd_rn(above[u], hi_of(dn)));
                } else {
                    vert = add2(E[O][k < PH - 1 ? k + 1 : 0][u], E[O][k ? k - 1 : 0][u]);
                }
                const pair_t lt = q ? E[O][k][u] : u ? E[O][k][u ? u - 1 : 0] : side[k];
                const pair_t rt = !q ? E[O][k][u] : u < PW - 1 ? E[O][k][u < PW - 1 ? u + 1 : 0] : side[k];
                const pair_t me = E[C][k][u];
                // r holds -R/den
                const pair_t gs = fma2(W.wy, vert, fma2(W.wx, add2(lt, rt), RREG ? R[RREG ? C : 0][RREG ? k : 0][u] : r[u]));
                E[C][k][u] = fma2(WALL == q + 1 ? W.at_wall[WALL ? u : 0] : W.beta, fma2(me, W.minus, gs), me);
            }
        }
    }
    if (!DB) __syncthreads();  // every thread has read the other colour's borders
    if (p.on) mr_publish<C, PH, RREG, DB>(E, out);
    __syncthreads();
}

// The sweeps of an epoch; grid colour 0 is local colour `flip`. The borders of the other colour are not published yet. False
// when a wait of the exchange before gave up.
template <int PH, bool RREG, bool DB, int WALL>
__device__ __forceinline__ bool mr_sweeps(pair_t (&E)[2][PH][PW], const pair_t (&R)[RREG ? 2 : 1][RREG ? PH : 1][PW],
                                          const Patch& p, int flip, const int* s_ok, const MrWeights<WALL>& W) {
    using S = MrShape<PH, RREG, DB>;
    if (p.on) {
        if (flip) mr_publish<0, PH, RREG, DB>(E, mr_smem);
        else mr_publish<1, PH, RREG, DB>(E, mr_smem + (DB ? S::border(blockDim.x) : 0));
    }
    __syncthreads();
    if (!*s_ok) return false;
    if (flip) mr_half<1, PH, RREG, DB, WALL>(E, R, p, W);
#pragma unroll 1
    for (int s = 1; s < kSweepsPerExchange; ++s) {
        mr_half<0, PH, RREG, DB, WALL>(E, R, p, W);
        mr_half<1, PH, RREG, DB, WALL>(E, R, p, W);
    }
    mr_half<0, PH, RREG, DB, WALL>(E, R, p, W);
    if (!flip) mr_half<1, PH, RREG, DB, WALL>(E, R, p, W);
    return true;
}

template <int PH, bool RREG, bool DB, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_mixed_reg(MixedLaunch L) {
    using S = MrShape<PH, RREG, DB>;
    Ctrl* ctl = L.ctrl;
    if (ctl->abort) return;
    __shared__ int s_ok;
    __shared__ int s_flag[8];
    __shared__ double s_red[MAXT / 32][2];
    __shared__ double s_tot[2];
    MixedSync* sy = reinterpret_cast<MixedSync*>(L.sync);
    const int n = L.n, P = L.pitch, T = blockDim.x, tid = threadIdx.x;
    const MTile t = make_mtile(n, L.gx, L.gy, blockIdx.x, 2 * PW);
    const int sr0 = max(1, min(t.r0 - kHalo, n - 1 - 2 * PH * L.nty)), j0 = max(1, t.c0 - kHalo);
    Patch p;
    p.ntx = L.ntx;
    p.nty = L.nty;
    p.tx = tid % p.ntx;
    p.ty = tid / p.ntx;
    p.dn = p.ty ? tid - p.ntx : T;
    p.up = p.ty < p.nty - 1 ? tid + p.ntx : T;
    const int jt = j0 + 2 * PW * p.tx, row0 = sr0 + p.ty * 2 * PH;  // the patch's first column, first row
    p.on = p.ty < p.nty && jt <= n - 2;
    p.wall = n - 1 - jt;  // jt is odd: its parity is that of n
    const int flip = (sr0 + 1) & 1;  // grid colour of local colour 0
    const bool wall = j0 + 2 * PW * p.ntx > n - 1;
    const size_t mt = (jt - 1) >> 1;  // the patch's first cell in a row of either colour
    const bool own_col = jt + 2 * PW > t.c0 && jt < t.c1;
    const bool near_col = jt < t.c1 + kHalo;
    // the patch's columns lie within kHalo of the tile's sides
    const bool side_col = jt < t.c0 + kHalo || jt + 2 * PW > t.c1 - kHalo;
    const float wxf = (float)(L.dx2 / L.den), wyf = (float)(L.dy2 / L.den), bf = (float)L.beta;
    const pair_t wx = pk(wxf, wxf), wy = pk(wyf, wyf), beta = pk(bf, bf), minus = pk(-1.f, -1.f);

    // the zeros at the box' ends; and cells beyond the walls are never published: their borders stay 0
    for (int x = tid; x < (DB ? 2 : 1) * S::border(T); x += T) mr_smem[x] = make_ulonglong2(0, 0);
    // no epochs of an earlier solve in the tile's cells (the first grid barrier comes before the first exchange)
    for (int par = 0; RREG && par < 4; ++par)
        for (int i = t.r0 + (tid >> 5); i < t.r1; i += T >> 5)
            for (int m = ((t.c0 - 1) >> 1) + (tid & 31); 2 * m < t.c1 - 1; m += 32)
                L.eg2[((size_t)par * n + i) * P + m] = make_uint2(0, 0);

    unsigned bar = 0, ep = 0;
    int outer = 0, status = CNV_NOT_CONVERGED;
    long long sweeps = 0;
    double rel = 0.0;
    for (outer = 0;; ++outer) {
        mixed_residual<1, 0>(L, t, sy, outer, s_red);
        if (!grid_sync(sy, bar, ctl, L.timeout_ns, &s_ok)) { status = CNV_TIMEOUT; break; }
        rel = mixed_norm(sy, s_tot);
        if (!isfinite(rel)) { status = CNV_NONFINITE; break; }
        if (rel <= L.rtol) { status = CNV_OK; break; }
        if (outer >= L.max_outer) break;

        // ---- FP32 inner solve from e = 0
        pair_t E[2][PH][PW], R[RREG ? 2 : 1][RREG ? PH : 1][PW];
        ulonglong2* rs = mr_smem + (DB ? 2 : 1) * S::border(T);
        if (p.on) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float* src = L.rq[flip ^ c] + (size_t)row0 * P + mt;
#pragma unroll
                for (int k = 0; k < PH; ++k) {
                    const float4 a = __ldcg(reinterpret_cast<const float4*>(src + (size_t)k * P));
                    const float4 b = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(k + PH) * P));
                    const pair_t r[PW] = {pk(-a.x, -b.x), pk(-a.y, -b.y), pk(-a.z, -b.z), pk(-a.w, -b.w)};
                    if (RREG) {
#pragma unroll
                        for (int u = 0; u < PW; ++u) R[RREG ? c : 0][RREG ? k : 0][u] = r[u];
                    } else {
#pragma unroll
                        for (int v = 0; v < S::kV; ++v)
                            rs[((c * PH + k) * S::kV + v) * T + tid] = make_ulonglong2(r[2 * v], r[2 * v + 1]);
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int k = 0; k < PH; ++k)
#pragma unroll
                for (int u = 0; u < PW; ++u) E[c][k][u] = 0;
        bool ok = true;
        for (int e = 0; e < L.epochs; ++e) {
            ++ep;
            if (e > 0 && !RREG) {
                // the neighbours' strips of the epoch before -> the cells outside the tile (what lies further out than
                // kHalo does not matter)
                if (!mixed_wait(L, t, sy, ep - 1, s_flag)) { ok = false; break; }
                if (p.on)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i0 = row0 + h * PH;
                        if (own_col && i0 >= t.r0 && i0 + PH <= t.r1) continue;
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const float* src = L.eg[(ep - 1) & 1][c ^ flip] + (size_t)i0 * P + mt;
                            float4 x[PH];
#pragma unroll
                            for (int k = 0; k < PH; ++k) x[k] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)k * P));
#pragma unroll
                            for (int k = 0; k < PH; ++k) {
                                if (own_col && i0 + k >= t.r0 && i0 + k < t.r1) continue;
                                const float v[PW] = {x[k].x, x[k].y, x[k].z, x[k].w};
#pragma unroll
                                for (int u = 0; u < PW; ++u)
                                    E[c][k][u] = h ? pk(lo_of(E[c][k][u]), v[u]) : pk(v[u], hi_of(E[c][k][u]));
                            }
                        }
                    }
            }
            if (e > 0 && RREG && p.on && near_col) {
                // the same, each cell with its epoch: no flag, no fence
                const uint2* eg = L.eg2 + (size_t)((ep - 1) & 1) * 2 * n * P + (size_t)row0 * P + mt;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i0 = row0 + h * PH;
                    if (own_col && i0 >= t.r0 && i0 + PH <= t.r1) continue;
                    ulonglong2 x[2][PH][2];
                    int polls = 0;
                    long long t0 = 0;
                    for (;;) {
#pragma unroll
                        for (int c = 0; c < 2; ++c)
#pragma unroll
                            for (int k = 0; k < PH; ++k)
#pragma unroll
                                for (int v = 0; v < 2; ++v)
                                    x[c][k][v] = ld_cells(eg + ((size_t)(c ^ flip) * n + h * PH + k) * P + 2 * v);
                        bool there = true;
#pragma unroll
                        for (int k = 0; k < PH; ++k) {
                            const int i = i0 + k;
                            const bool want = i >= t.r0 - kHalo && i < t.r1 + kHalo && !(own_col && i >= t.r0 && i < t.r1);
                            unsigned d = 0;
#pragma unroll
                            for (int v = 0; v < 4; ++v)
                                d |= ((unsigned)(x[v >> 1][k][v & 1].x >> 32) ^ (ep - 1)) |
                                     ((unsigned)(x[v >> 1][k][v & 1].y >> 32) ^ (ep - 1));
                            there = there && !(want && d);
                        }
                        if (there) break;
                        if ((polls & 15) == 15 && ld_volatile_int(&ctl->abort)) { s_ok = 0; break; }
                        if (++polls == 64) t0 = globaltimer_ns();
                        if (polls > 64 && globaltimer_ns() - t0 > L.timeout_ns) {
                            atomicExch(&ctl->status, CNV_TIMEOUT);
                            atomicExch(&ctl->abort, 1);
                            s_ok = 0;
                            break;
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int k = 0; k < PH; ++k) {
                            if (own_col && i0 + k >= t.r0 && i0 + k < t.r1) continue;
                            const unsigned v[PW] = {(unsigned)x[c][k][0].x, (unsigned)x[c][k][0].y, (unsigned)x[c][k][1].x, (unsigned)x[c][k][1].y};
#pragma unroll
                            for (int u = 0; u < PW; ++u) {
                                pair_t& E1 = E[c][k][u];
                                E1 = h ? pk(lo_of(E1), __uint_as_float(v[u])) : pk(__uint_as_float(v[u]), hi_of(E1));
                            }
                        }
                }
            }
            auto sweep = [&](auto w) {
                MrWeights<w.value> W{wx, wy, beta, minus, {}};
#pragma unroll
                for (int u = 0; w.value && u < PW; ++u) W.at_wall[u] = p.wall >> 1 == u ? 0ull : beta;
                return mr_sweeps<PH, RREG, DB, w.value>(E, R, p, flip, &s_ok, W);
            };
            ok = !wall ? sweep(Int<0>{}) : n % 2 == 0 ? sweep(Int<1>{}) : sweep(Int<2>{});
            if (!ok) break;
            sweeps += kSweepsPerExchange;
            if (e + 1 < L.epochs) {
                // own cells near the tile's border -> global copy of this epoch, each with the epoch
                if (p.on && own_col && (int)blockIdx.x != L.stall_block) {
                    uint2* eg = L.eg2 + (size_t)(ep & 1) * 2 * n * P + mt;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int k = 0; k < PH; ++k) {
                            const int i = row0 + k + h * PH;
                            if (i < t.r0 || i >= t.r1 || !(side_col || i < t.r0 + kHalo || i >= t.r1 - kHalo)) continue;
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const pair_t* w = E[c][k];
                                if (!RREG)
                                    *reinterpret_cast<float4*>(L.eg[ep & 1][c ^ flip] + (size_t)i * P + mt) =
                                        h ? make_float4(hi_of(w[0]), hi_of(w[1]), hi_of(w[2]), hi_of(w[3]))
                                          : make_float4(lo_of(w[0]), lo_of(w[1]), lo_of(w[2]), lo_of(w[3]));
                                uint2* d = eg + ((size_t)(c ^ flip) * n + i) * P;
#pragma unroll
                                for (int v = 0; RREG && v < S::kV; ++v) {
                                    const pair_t a = E[c][k][2 * v], b = E[c][k][2 * v + 1];
                                    st_cells(d + 2 * v, tagged((unsigned)(h ? a >> 32 : a), ep), tagged((unsigned)(h ? b >> 32 : b), ep));
                                }
                            }
                        }
                }
                if (!RREG) {
                    __syncthreads();
                    if (threadIdx.x == 0 && (int)blockIdx.x != L.stall_block) st_release(&sy->flag[blockIdx.x], ep);
                }
            }
        }
        if (!ok) { status = CNV_TIMEOUT; break; }
        // ---- FP64 correction psi += e on own cells
        if (p.on && own_col) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < PH; ++k) {
                    const int i = row0 + k + h * PH;
                    if (i < t.r0 || i >= t.r1) continue;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int q = (k + c) & 1;
                        double* d = L.psi[c ^ flip] + (size_t)i * P + mt + q;  // column jt + q + 2 u, jt odd
#pragma unroll
                        for (int u = 0; u < PW; ++u)
                            if (jt + q + 2 * u < n - 1) d[u] += (double)(h ? hi_of(E[c][k][u]) : lo_of(E[c][k][u]));
                    }
                }
        }
        if (!grid_sync(sy, bar, ctl, L.timeout_ns, &s_ok)) { status = CNV_TIMEOUT; break; }
    }
    if (status == CNV_TIMEOUT) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) mixed_report(L, outer, status, rel, sweeps);
}

// The forms of the kernel; the first that fits is taken (mixed_pick).
struct MrForm {
    int ph, threads;
    int (*units)(int);  // shared memory for a number of threads, in units of 16 bytes
    const void* kernel;
};
template <int PH, bool RREG, bool DB, int MAXT>
MrForm mr_form() {
    return MrForm{PH, MAXT, &MrShape<PH, RREG, DB>::units, reinterpret_cast<const void*>(&k_mixed_reg<PH, RREG, DB, MAXT>)};
}
const MrForm kForms[] = {
    mr_form<4, true, true, 256>(),  mr_form<6, false, true, 256>(),  mr_form<8, false, true, 256>(),
    mr_form<10, false, true, 256>(), mr_form<12, false, false, 256>(),
};

}  // namespace

// Form and box of the register kernel for a gx x gy tiling (form -1: none fits).
void mixed_pick(int n, int gx, int gy, size_t smem_max, int* form, int* ntx, int* nty) {
    const int ni = n - 2, h = std::min(ni, (ni + gy - 1) / gy + 2 * kHalo);
    *form = -1;
    int w = 0;  // columns of the widest box
    for (int x = 0; x < gx; ++x) {
        const int c0 = mtile_col(n, gx, x, 2 * PW), c1 = mtile_col(n, gx, x + 1, 2 * PW);
        if (c1 - c0 < kHalo) return;
        w = std::max(w, std::min(c1 + kHalo, n - 1) - (x ? c0 - kHalo : 1));
    }
    const int tx = (w + 2 * PW - 1) / (2 * PW);
    for (int f = 0; f < (int)(sizeof kForms / sizeof kForms[0]); ++f) {
        const MrForm& F = kForms[f];
        const int ty = (h + 2 * F.ph - 1) / (2 * F.ph);
        if (2 * F.ph * ty > ni) continue;  // the box's rows lie inside the interior
        const int threads = (tx * ty + 31) / 32 * 32;
        if (threads > F.threads || (size_t)F.units(threads) * 16 + 2048 > smem_max) continue;
        *form = f;
        *ntx = tx;
        *nty = ty;
        return;
    }
}

cudaError_t launch_mixed(const MixedLaunch& L, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(L.sync, 0, sizeof(MixedSync), s);
    if (e != cudaSuccess) return e;
    size_t smem = mixed_smem_bytes(L.n, L.gx, L.gy, L.rq_in_smem != 0);
    int threads = kThreads;
    const void* kernel = reinterpret_cast<const void*>(&k_mixed);
    if (L.form >= 0) {
        threads = (L.ntx * L.nty + 31) / 32 * 32;
        smem = (size_t)kForms[L.form].units(threads) * 16;
        kernel = kForms[L.form].kernel;
    }
    // one limit for all solves: the attribute belongs to the function, and another thread may launch it between the two calls
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem_max);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.gx * L.gy);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {const_cast<MixedLaunch*>(&L)};
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

int mixed_threads() { return kThreads; }
int mixed_sweeps_per_exchange() { return kSweepsPerExchange; }

}  // namespace cnv
