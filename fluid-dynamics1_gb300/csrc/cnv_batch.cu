// cnv_batch.cu -- many independent cavities (uneven grid size, Re and lid speed) advanced by one
// persistent launch.
//
// Work unit: one cavity for `nsteps` time steps, run by a group of g blocks (g = 1 for most
// cavities). Each step is the reference's loop body (src/main.c:283-395) with the same device
// arithmetic as the single-cavity path (reference rounding for the wall, transport, velocity and
// continuity passes) and the mixed-precision Poisson solve of cnv_mixed.cu: FP32 red-black SOR
// sweeps inside FP64 defect correction to a relative FP64 residual.
//
// One block (g = 1) keeps the FP32 correction in shared memory when the cavity fits (with its
// right-hand side when both fit), in the cavity's global arrays otherwise. A cavity whose
// correction does not fit one block's shared memory is split into g row strips, one per block of
// its group: every pass runs on the block's strip, the FP32 correction of the strip plus a halo
// of 2S rows lives in that block's shared memory, and the blocks meet at group barriers (global
// counters with bounded waits): after the wall pass, after the transport pass, around each
// residual norm, once per S FP32 sweeps to exchange border rows (the halo rows are recomputed, as
// in cnv_mixed.cu, so the iterates equal global red-black sweeps), after the correction update,
// after the velocity pass and after the continuity pass.
//
// Schedule. The host orders the jobs (largest estimated cost first) and places each on the g
// blocks that become free first (longest-processing-time scheduling); every block runs its list
// in start-time order, so members of a group reach their common job in the same global order and
// no wait can close a cycle. The launch is cooperative (all blocks resident), captured in a CUDA
// graph with the per-launch counters reset, and reads the step count from device memory so one
// graph serves every call. The autotuner (cnv_batch_tune) times one step of each candidate
// decomposition (strips only where shared memory needs them, or more, or the strip counts per
// cavity size that minimise the schedule's estimated makespan) and keeps the fastest.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "cnv_kernels.h"
#include "cnv_sor.cuh"
#include "cnv_stencil.cuh"
#include "cnv_sync.cuh"

namespace cnv {

// The passes' band coefficients are multiplied on the integer pipes (the same bits): 192^2, 152 cavities, 5.38 -> 5.22 ms
// per step (the passes themselves are bound by their loads; they change little).
template <>
__device__ __forceinline__ double band_mul<kMulInt>(double c, double x) {
    return mul_rn(c, x);
}

struct CavityDesc {
    int n, pitch;       // grid size; split-layout pitch (doubles/floats per row)
    int spitch;         // split-layout pitch of the shared-memory tile as the plan counts it (floats per row)
    int epitch;         // its pitch in use: a multiple of 4 where the vector sweeps run (vec)
    int vec;
    int smem_mode;      // 0: e and R/den in global memory, 1: e in shared, 2: both in shared
    int inner;          // FP32 sweeps per correction
    int cur;            // current vorticity buffer
    double inv_re, dt, beta, c4, dx2, dy2, den, rden;
    BoundaryValues bc;
    const FdBands* bands;
    double* w[2];
    double* u;
    double* v;
    double* psi_rm;     // row-major psi (output)
    double* psi[2];     // split layout, FP64 iterate
    double* g[2];       // split layout, c4*f
    float* e[2];        // split layout, FP32 correction (global mode); group jobs: border copies, parity 0
    float* ex1[2];      // split layout, FP32 border copies of parity 1 (group jobs)
    float* rq[2];       // split layout, FP32 R/den (global mode and group jobs)
    StepRecord last;    // record of the cavity's last step
    long long sweeps;   // FP32 sweeps done in the last call
    int steps_done;     // steps completed in the last call
    int group;          // blocks that run this cavity (row strips)
};

// Group barrier and reductions of one cavity's group (zeroed before every launch).
constexpr int kMaxGroup = 16;
constexpr size_t kBatchGuardBytes = 4096;  // guard region size (test_guard_cells)
struct GroupSync {
    unsigned int bar;
    unsigned int pad;
    double part[kMaxGroup][2];  // per rank: residual and right-hand-side sums of squares
    double cont[kMaxGroup][2];  // per rank: continuity max and min
};

// One entry of a block's job list: cavity, this block's strip (rank) and the group size.
struct SchedEntry {
    int cav, rank, group, pad;
};

struct BatchLaunch {
    CavityDesc* cav;
    const SchedEntry* sched;  // job lists of all blocks, one after another
    const int* sched_off;     // block b's list: sched[sched_off[b] .. sched_off[b+1])
    GroupSync* gsync;         // one per cavity
    int* abort;               // set when a group wait gives up (CNV_TIMEOUT)
    const int* nsteps;  // steps per cavity for this call (device memory)
    int count;
    int max_outer;
    double rtol;
    int warm;           // start each step's solve from the previous psi (mixed_warm_start)
    int smem_floats;    // dynamic shared memory available to a block (floats)
};

namespace {

constexpr int kMaxBatchThreads = 1024;
// A batch of cavities smaller than this runs k_batch<SMALL>: scalar sweeps, FP64 multiplications in the passes. With a cell a thread
// at most a step is a chain of latencies, which the vector sweeps' set-up and the integer multiplications lengthen (a kernel of its own:
// a second copy of the step in one kernel cost the larger cavities 2 %). us per step, k_batch<false> / k_batch<true>: 8^2 203 / 180, 16^2
// 203 / 188, 22^2 237 / 226, 24^2 236 / 245, 64^2 532 / 750.
constexpr int kSmallN = 24;

// The dynamic shared memory of k_batch; the sweeps address it through this array with integer offsets, so every access
// compiles to a shared-memory load or store.
extern __shared__ __align__(16) float bt_smem[];

// Block-wide sum of a double (deterministic: xor butterfly, then warps in order).
__device__ double block_sum(double x, double* s_red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) s_red[warp] = x;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_red[w];
    __syncthreads();
    return t;
}

__device__ void block_minmax(double& mx, double& mn, double* s_red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double a = __shfl_xor_sync(0xffffffffu, mx, off);
        const double b = __shfl_xor_sync(0xffffffffu, mn, off);
        mx = a > mx ? a : mx;
        mn = b < mn ? b : mn;
    }
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_red[warp] = mx;
        s_red[32 + warp] = mn;
    }
    __syncthreads();
    mx = -DBL_MAX;
    mn = DBL_MAX;
    for (int w = 0; w < nw; ++w) {
        mx = s_red[w] > mx ? s_red[w] : mx;
        mn = s_red[32 + w] < mn ? s_red[32 + w] : mn;
    }
    __syncthreads();
}

// The FP32 sweeps of a cavity (or strip) whose correction is in shared memory. A thread takes 4 neighbouring cells of a colour
// (a 16-byte vector of the split layout) and walks down `run` rows with the other colour's rows above, at and below in
// registers, so a row costs it three vector loads (the other colour's next row, its own cells, R/den), one word from the side
// and one vector store: 17 to 21 bytes of shared memory and about 9 instructions per cell, where a cell per lane took 28 and
// 20. Per sweep, 128^2 on one block: 4.1 -> 1.9 us; 192^2 9.2 -> 4.1; the same bits. (Loading R/den two rows ahead where it
// comes from global memory changed nothing.) Wall cells and the pitch' padding start at 0 and stay 0 with a SOR factor of 0 (b0
// for rows with cells at even columns, b1 for the others).
struct QuadSweep {
    int col, seg, run;      // first cell of the thread's vectors; its run of rows, and its length (even)
    float b0[4], b1[4];
    float wx, wy;
};

// rows: at most this many are swept
__device__ __forceinline__ QuadSweep quad_sweep(int n, int rows, float wx, float wy, float beta) {
    QuadSweep Q;
    const int quads = ((n + 1) / 2 + 3) / 4, segs = blockDim.x / quads;
    Q.seg = threadIdx.x / quads;
    Q.col = 4 * (threadIdx.x - Q.seg * quads);
    Q.run = ((rows + segs - 1) / segs + 1) & ~1;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int j = 2 * (Q.col + u);
        Q.b0[u] = j >= 1 && j <= n - 2 ? beta : 0.0f;
        Q.b1[u] = j + 1 <= n - 2 ? beta : 0.0f;
    }
    Q.wx = wx;
    Q.wy = wy;
    return Q;
}

// A row whose cells of the swept colour lie at columns 2m + ODD; o: the other colour's row, s: its cell beside the vector (left
// for even columns, right for odd ones).
template <int ODD>
__device__ __forceinline__ float4 quad_row(const QuadSweep& Q, float4 up, float4 dn, float4 o, float s, float4 r, float4 me) {
    const float a = o.x + o.y, b = o.y + o.z, c = o.z + o.w, e = ODD ? o.w + s : s + o.x;
    const float h[4] = {ODD ? a : e, ODD ? b : a, ODD ? c : b, ODD ? e : c};
    const float* w = ODD ? Q.b1 : Q.b0;
    float4 v;
    v.x = fmaf(w[0], fmaf(Q.wy, up.x + dn.x, fmaf(Q.wx, h[0], -r.x)) - me.x, me.x);
    v.y = fmaf(w[1], fmaf(Q.wy, up.y + dn.y, fmaf(Q.wx, h[1], -r.y)) - me.y, me.y);
    v.z = fmaf(w[2], fmaf(Q.wy, up.z + dn.z, fmaf(Q.wx, h[2], -r.z)) - me.z, me.z);
    v.w = fmaf(w[3], fmaf(Q.wy, up.w + dn.w, fmaf(Q.wx, h[3], -r.w)) - me.w, me.w);
    return v;
}

// Where R/den is: the block's own global array, one that other blocks write too (read through L2), or shared memory.
enum RhsIn { kRhsOwn, kRhsL2, kRhsShared };

// Half-sweep of colour c on rows [lo, hi): ec, eo, the offsets of row 0 of the two colours in shared memory (pitch ep, rows beside
// [lo, hi) present); R/den's row 0 at rq (pitch rp), or at offset rs0 in shared memory (pitch ep). FIRST: parity of lo + c.
template <int FIRST, int RHS>
__device__ __forceinline__ void quad_half_sweep_p(const QuadSweep& Q, int ec, int eo, const float* rq, int rs0, int ep, int rp,
                                                  int lo, int hi) {
    int i = lo + Q.seg * Q.run;
    const int end = min(hi, i + Q.run);
    if (i >= end) return;
    auto vec = [](int at) { return *reinterpret_cast<const float4*>(bt_smem + at); };
    auto rhs = [&](int row) {
        if (RHS == kRhsShared) return vec(rs0 + row * ep + Q.col);
        const float4* p = reinterpret_cast<const float4*>(rq + (size_t)row * rp + Q.col);
        return RHS == kRhsL2 ? __ldcg(p) : *p;
    };
    const int ls = FIRST ? 4 : -1, rs = FIRST ? -1 : 4;  // the side of the first and of the second row
    const bool left = Q.col > 0, right = Q.col + 4 < ep;
    int o = eo + i * ep + Q.col, c = ec + i * ep + Q.col;
    float4 dn = vec(o - ep), at = vec(o);
    for (; i < end; i += 2, o += 2 * ep, c += 2 * ep) {
        float4 up = vec(o + ep);
        float s = (FIRST ? right : left) ? bt_smem[o + ls] : 0.0f;
        *reinterpret_cast<float4*>(bt_smem + c) = quad_row<FIRST>(Q, up, dn, at, s, rhs(i), vec(c));
        if (i + 1 >= end) break;
        dn = at;
        at = up;
        up = vec(o + 2 * ep);
        s = (FIRST ? left : right) ? bt_smem[o + ep + rs] : 0.0f;
        *reinterpret_cast<float4*>(bt_smem + c + ep) = quad_row<1 - FIRST>(Q, up, dn, at, s, rhs(i + 1), vec(c + ep));
        dn = at;
        at = up;
    }
}

template <int RHS>
__device__ __forceinline__ void quad_half_sweep(const QuadSweep& Q, int ec, int eo, const float* rq, int rs0, int ep, int rp, int lo,
                                                int hi, int c) {
    if ((lo + c) & 1) quad_half_sweep_p<1, RHS>(Q, ec, eo, rq, rs0, ep, rp, lo, hi);
    else quad_half_sweep_p<0, RHS>(Q, ec, eo, rq, rs0, ep, rp, lo, hi);
}

// FP32 red-black SOR half-sweep of colour c over the interior, split layout with row pitch ep
// for e and rp for R/den.
__device__ void batch_half_sweep(float* __restrict__ ec, const float* __restrict__ eo, const float* __restrict__ rq,
                                 int n, int ep, int rp, int c, float wx, float wy, float beta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int i = 1 + warp; i < n - 1; i += nw) {
        const int q = (i + c) & 1;
        const int mlo = floor_half(1 - q + 1), mhi = floor_half(n - 2 - q);
        const int row = i * ep;
        const float* rrow = rq + (size_t)i * rp;
        for (int m = mlo + lane; m <= mhi; m += 32) {
            const float up = eo[row + ep + m], dn = eo[row - ep + m];
            const float lt = eo[row + m - 1 + q], rt = eo[row + m + q];
            const float me = ec[row + m];
            const float gs = fmaf(wy, up + dn, fmaf(wx, lt + rt, -rrow[m]));
            ec[row + m] = fmaf(beta, gs - me, me);
        }
    }
}

// One time step of one cavity by the whole block. Returns the step's status.
template <bool SMALL>
__device__ int batch_step(CavityDesc& C, float* smem, int max_outer, double rtol, bool warm, double* s_red) {
    constexpr int MUL = SMALL ? kMulFp64 : kMulInt;
    const int n = C.n, P = C.pitch;
    const int tid = threadIdx.x, nt = blockDim.x;
    double* w_in = C.w[C.cur];
    double* w_out = C.w[C.cur ^ 1];
    const BoundaryValues bc = C.bc;
    const FdBands* B = C.bands;

    // wall vorticity on the four edges (src/main.c:298-320), in place on w_in
    for (int s = tid; s < 4 * n; s += nt) {
        const int side = s / n, t = s - side * n;
        const int i = side == 0 ? 0 : side == 1 ? n - 1 : t;
        const int j = side == 2 ? 0 : side == 3 ? n - 1 : t;
        auto U = [&](int r, int cc) { return vel_bc(C.u, n, r, cc, bc.u1, bc.u2, bc.u3, bc.u4); };
        auto V = [&](int r, int cc) { return vel_bc(C.v, n, r, cc, bc.v1, bc.v2, bc.v3, bc.v4); };
        w_in[(size_t)i * n + j] = dsub(along_j<MUL>(B->d1x, n, i, j, V), along_i<MUL>(B->d1y, n, i, j, U));
    }
    __syncthreads();
    // transport: derivatives of w and the Euler update (src/fluiddyn.c:98); g = c4 * (-w)
    for (int k = tid; k < n * n; k += nt) {
        const int i = k / n, j = k - (k / n) * n;
        auto W = [&](int r, int cc) { return w_in[(size_t)r * n + cc]; };
        const double wx = along_j<MUL>(B->d1x, n, i, j, W), wy = along_i<MUL>(B->d1y, n, i, j, W);
        const double wxx = along_j<MUL>(B->d2x, n, i, j, W), wyy = along_i<MUL>(B->d2y, n, i, j, W);
        const double ue = vel_bc(C.u, n, i, j, bc.u1, bc.u2, bc.u3, bc.u4);
        const double ve = vel_bc(C.v, n, i, j, bc.v1, bc.v2, bc.v3, bc.v4);
        const double conv = dsub(dmul(-ue, wx), dmul(ve, wy));
        const double wn = dadd(dmul(dadd(conv, dmul(C.inv_re, dadd(wxx, wyy))), C.dt), w_in[k]);
        w_out[k] = wn;
        if (i > 0 && i < n - 1 && j > 0 && j < n - 1)
            C.g[(i + j) & 1][(size_t)i * P + (j >> 1)] = dmul(C.c4, -wn);
    }
    // psi = 0 (zero start; zero Dirichlet edge), or the previous step's psi (warm start)
    if (!warm)
        for (int k = tid; k < 2 * n * P; k += nt) (k < n * P ? C.psi[0] : C.psi[1])[k < n * P ? k : k - n * P] = 0.0;
    __syncthreads();

    // mixed-precision Poisson solve (cnv_mixed.cu's scheme, whole cavity in one block)
    const int sp = C.epitch;
    const int eplane = C.smem_mode >= 1 ? n * sp : 0;
    float* e_s[2] = {smem, smem + eplane};
    float* rq_s[2] = {smem + 2 * eplane, smem + 3 * eplane};
    float* ec[2] = {C.smem_mode >= 1 ? e_s[0] : C.e[0], C.smem_mode >= 1 ? e_s[1] : C.e[1]};
    const int ep = C.smem_mode >= 1 ? sp : P;
    float* rqc[2] = {C.smem_mode == 2 ? rq_s[0] : C.rq[0], C.smem_mode == 2 ? rq_s[1] : C.rq[1]};
    const int rp = C.smem_mode == 2 ? sp : P;
    const float wxf = (float)(C.dx2 / C.den), wyf = (float)(C.dy2 / C.den), betaf = (float)C.beta;
    QuadSweep Q;
    if constexpr (!SMALL) {
        Q = quad_sweep(n, n - 2, wxf, wyf, betaf);
        if (C.vec && C.smem_mode == 2)  // R/den is 0 on the walls and in the padding
            for (int k = tid; k < 2 * eplane; k += nt) rq_s[0][k] = 0.0f;
        __syncthreads();
    }
    double rel = 0.0, gnorm = 0.0;
    int outer = 0, status = CNV_NOT_CONVERGED;
    long long sweeps = 0;
    for (outer = 0;; ++outer) {
        double rr = 0.0, gg = 0.0;
        for (int k = tid; k < n * n; k += nt) {
            const int i = k / n, j = k - (k / n) * n;
            if (i == 0 || i == n - 1 || j == 0 || j == n - 1) continue;
            const int c = (i + j) & 1, q = (i + c) & 1, m = j >> 1;
            const double* pc = C.psi[c];
            const double* po = C.psi[c ^ 1];
            const size_t kk = (size_t)i * P + m;
            const double g = C.g[c][kk];
            const double R = poisson_defect(C.dy2, C.dx2, C.den, po[kk + P], po[kk - P], po[kk - 1 + q], po[kk + q],
                                            pc[kk], g);
            rr = fma(R, R, rr);
            if (outer == 0) gg = fma(g, g, gg);
            rqc[c][(size_t)i * rp + m] = (float)(R * C.rden);
        }
        rr = block_sum(rr, s_red);
        if (outer == 0) gnorm = sqrt(block_sum(gg, s_red));
        rel = gnorm > 0 ? sqrt(rr) / gnorm : sqrt(rr);
        if (!isfinite(rel)) { status = CNV_NONFINITE; break; }
        if (rel <= rtol) { status = CNV_OK; break; }
        if (outer >= max_outer) break;
        // e = 0 on the whole split plane (edges included), then the FP32 sweeps
        for (int k = tid; k < 2 * n * ep; k += nt) (k < n * ep ? ec[0] : ec[1])[k < n * ep ? k : k - n * ep] = 0.0f;
        __syncthreads();
        for (int s = 0; s < 2 * C.inner; ++s) {
            const int c = s & 1;
            if (!SMALL && C.vec && C.smem_mode == 2)
                quad_half_sweep<kRhsShared>(Q, c * eplane, (c ^ 1) * eplane, nullptr, (2 + c) * eplane, ep, 0, 1, n - 1, c);
            else if (!SMALL && C.vec)
                quad_half_sweep<kRhsOwn>(Q, c * eplane, (c ^ 1) * eplane, rqc[c], 0, ep, rp, 1, n - 1, c);
            else batch_half_sweep(ec[c], ec[c ^ 1], rqc[c], n, ep, rp, c, wxf, wyf, betaf);
            __syncthreads();
        }
        sweeps += C.inner;
        // psi += e (FP64)
        for (int k = tid; k < n * n; k += nt) {
            const int i = k / n, j = k - (k / n) * n;
            if (i == 0 || i == n - 1 || j == 0 || j == n - 1) continue;
            const int c = (i + j) & 1;
            C.psi[c][(size_t)i * P + (j >> 1)] += (double)ec[c][(size_t)i * ep + (j >> 1)];
        }
        __syncthreads();
    }

    // velocity u = DY psi, v = -(DX psi) (src/main.c:366-383), row-major psi for output
    auto PS = [&](int y, int x) { return C.psi[(y + x) & 1][(size_t)y * P + (x >> 1)]; };
    for (int k = tid; k < n * n; k += nt) {
        const int i = k / n, j = k - (k / n) * n;
        C.u[k] = along_i<MUL>(B->d1y, n, i, j, PS);
        C.v[k] = -along_j<MUL>(B->d1x, n, i, j, PS);
        C.psi_rm[k] = PS(i, j);
    }
    __syncthreads();
    // continuity DX u + DY v, max and min (src/main.c:387-408)
    double mx = -DBL_MAX, mn = DBL_MAX;
    auto Uf = [&](int r, int cc) { return C.u[(size_t)r * n + cc]; };
    auto Vf = [&](int r, int cc) { return C.v[(size_t)r * n + cc]; };
    for (int k = tid; k < n * n; k += nt) {
        const int i = k / n, j = k - (k / n) * n;
        const double cv = dadd(along_j<MUL>(B->d1x, n, i, j, Uf), along_i<MUL>(B->d1y, n, i, j, Vf));
        mx = cv > mx ? cv : mx;
        mn = cv < mn ? cv : mn;
    }
    block_minmax(mx, mn, s_red);
    if (tid == 0) {
        C.last.iters = outer;
        C.last.status = status;
        C.last.err = rel;
        C.last.cont_max = mx;
        C.last.cont_min = mn;
        C.sweeps += sweeps;
        C.cur ^= 1;
    }
    __syncthreads();
    return status;
}

// ------------------------------------------------------------------------------ group jobs
constexpr int kStripSweeps = 4;                // FP32 sweeps between border exchanges (8: 1 % faster, more smem)
constexpr int kStripHalo = 2 * kStripSweeps;   // halo rows of a strip
static_assert(kSmallN <= 4 * kStripHalo, "k_batch<SMALL> has no strips");

// Barrier of the g blocks of a group (counter gs->bar, target gen). False if the wait gave up
// (2 s; sets *abort = CNV_TIMEOUT) or another block has aborted; the caller leaves the job.
__device__ bool group_barrier(GroupSync* gs, unsigned& gen, int g, int* abort, int* s_ok) {
    __syncthreads();
    gen += g;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&gs->bar, 1u);
        int ok = 1, polls = 0;
        long long t0 = 0;
        while ((int)(ld_acquire(&gs->bar) - gen) < 0) {
            if (*(volatile int*)abort) {
                ok = 0;
                break;
            }
            if (++polls == 64) t0 = globaltimer_ns();
            if (polls > 64 && globaltimer_ns() - t0 > 2000000000LL) {
                atomicExch(abort, CNV_TIMEOUT);
                ok = 0;
                break;
            }
        }
        __threadfence();
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// FP32 red-black SOR half-sweep of colour c on rows [lo_r, hi_r) of a strip tile (rows from sr0,
// split pitch ep, full interior width); R/den from the cavity's global array (pitch P, read
// through L2: other blocks of the group write it). Same arithmetic as batch_half_sweep.
__device__ void strip_half_sweep(float* __restrict__ ec, const float* __restrict__ eo, const float* __restrict__ rq,
                                 int sr0, int ep, int P, int lo_r, int hi_r, int n, int c, float wx, float wy,
                                 float beta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int i = lo_r + warp; i < hi_r; i += nw) {
        const int q = (i + c) & 1;
        const int mlo = floor_half(1 - q + 1), mhi = floor_half(n - 2 - q);
        const int row = (i - sr0) * ep;
        const float* rrow = rq + (size_t)i * P;
        for (int m = mlo + lane; m <= mhi; m += 32) {
            const float up = eo[row + ep + m], dn = eo[row - ep + m];
            const float lt = eo[row + m - 1 + q], rt = eo[row + m + q];
            const float me = ec[row + m];
            const float gs = fmaf(wy, up + dn, fmaf(wx, lt + rt, -__ldcg(rrow + m)));
            ec[row + m] = fmaf(beta, gs - me, me);
        }
    }
}

// One time step of a cavity by block `r` of its group of g (rows [n r / g, n (r+1) / g)). Every
// read of a field that other blocks of the group write goes through L2 (__ldcg). Returns the
// step's status (the same in every block of the group); CNV_TIMEOUT if a group wait gave up.
__device__ int group_step(CavityDesc& C, int cur, int r, int g, float* smem, int max_outer, double rtol, bool warm,
                          double* s_red, GroupSync* gs, unsigned& gen, int* abort, int* s_ok, long long& sweeps,
                          StepRecord& rec) {
    const int n = C.n, P = C.pitch, sp = C.epitch;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int R0 = (int)((long long)n * r / g), R1 = (int)((long long)n * (r + 1) / g);
    const int rows = R1 - R0;
    double* const w_in = C.w[cur];
    double* const w_out = C.w[cur ^ 1];
    const BoundaryValues bc = C.bc;
    const FdBands* B = C.bands;
    auto LD = [](const double* p) { return __ldcg(p); };
    auto U = [&](int y, int x) {
        if (x == 0) return bc.u1;
        if (x == n - 1) return bc.u2;
        if (y == 0) return bc.u3;
        if (y == n - 1) return bc.u4;
        return LD(C.u + (size_t)y * n + x);
    };
    auto V = [&](int y, int x) {
        if (x == 0) return bc.v1;
        if (x == n - 1) return bc.v2;
        if (y == 0) return bc.v3;
        if (y == n - 1) return bc.v4;
        return LD(C.v + (size_t)y * n + x);
    };

    // wall vorticity on the strip's edge cells (src/main.c:298-320), in place on w_in
    {
        const int top = R0 == 0 ? n - 2 : 0, bot = R1 == n ? n - 2 : 0;
        const int total = 2 * rows + top + bot;
        for (int x = tid; x < total; x += nt) {
            int i, j;
            if (x < 2 * rows) {
                i = R0 + (x >> 1);
                j = (x & 1) ? n - 1 : 0;
            } else if (x < 2 * rows + top) {
                i = 0;
                j = 1 + (x - 2 * rows);
            } else {
                i = n - 1;
                j = 1 + (x - 2 * rows - top);
            }
            w_in[(size_t)i * n + j] = dsub(along_j<kMulInt>(B->d1x, n, i, j, V), along_i<kMulInt>(B->d1y, n, i, j, U));
        }
    }
    if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;
    // transport on the strip's rows; g = c4 * (-w); psi = 0 on the strip's rows (zero start)
    {
        auto W = [&](int y, int x) { return LD(w_in + (size_t)y * n + x); };
        for (int x = tid; x < rows * n; x += nt) {
            const int i = R0 + x / n, j = x - (x / n) * n;
            const double wx = along_j<kMulInt>(B->d1x, n, i, j, W), wy = along_i<kMulInt>(B->d1y, n, i, j, W);
            const double wxx = along_j<kMulInt>(B->d2x, n, i, j, W), wyy = along_i<kMulInt>(B->d2y, n, i, j, W);
            const double conv = dsub(dmul(-U(i, j), wx), dmul(V(i, j), wy));
            const size_t k = (size_t)i * n + j;
            const double wn = dadd(dmul(dadd(conv, dmul(C.inv_re, dadd(wxx, wyy))), C.dt), W(i, j));
            w_out[k] = wn;
            if (i > 0 && i < n - 1 && j > 0 && j < n - 1) C.g[(i + j) & 1][(size_t)i * P + (j >> 1)] = dmul(C.c4, -wn);
        }
        if (!warm)
            for (int x = tid; x < 2 * rows * P; x += nt) {
                const int c = x >= rows * P;
                const int y = x - c * rows * P;
                C.psi[c][(size_t)R0 * P + y] = 0.0;
            }
    }
    if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;

    // mixed-precision Poisson solve, the strip's FP32 correction (plus halo rows) in shared memory
    const int ri0 = R0 > 1 ? R0 : 1, ri1 = R1 < n - 1 ? R1 : n - 1;  // own interior rows
    const int sr0 = R0 - kStripHalo > 0 ? R0 - kStripHalo : 0;
    const int sr1 = R1 + kStripHalo < n ? R1 + kStripHalo : n;
    const int plane = (sr1 - sr0) * sp;
    float* const es[2] = {smem, smem + plane};
    const float wxf = (float)(C.dx2 / C.den), wyf = (float)(C.dy2 / C.den), betaf = (float)C.beta;
    double rel = 0.0, gnorm = 0.0;
    int outer = 0, status = CNV_NOT_CONVERGED;
    const int epochs = C.inner / kStripSweeps;
    const QuadSweep Q = quad_sweep(n, rows + 2 * kStripHalo - 2, wxf, wyf, betaf);
    for (outer = 0;; ++outer) {
        double rr = 0.0, gg = 0.0;
        for (int x = tid; x < (ri1 - ri0) * (n - 2); x += nt) {
            const int i = ri0 + x / (n - 2), j = 1 + (x - (x / (n - 2)) * (n - 2));
            const int c = (i + j) & 1, q = (i + c) & 1, m = j >> 1;
            const double* pc = C.psi[c];
            const double* po = C.psi[c ^ 1];
            const size_t kk = (size_t)i * P + m;
            const double gv = C.g[c][kk];
            const double R = poisson_defect(C.dy2, C.dx2, C.den, LD(po + kk + P), LD(po + kk - P), LD(po + kk - 1 + q),
                                            LD(po + kk + q), pc[kk], gv);
            rr = fma(R, R, rr);
            if (outer == 0) gg = fma(gv, gv, gg);
            C.rq[c][kk] = (float)(R * C.rden);
        }
        rr = block_sum(rr, s_red);
        if (outer == 0) gg = block_sum(gg, s_red);
        if (tid == 0) {
            gs->part[r][0] = rr;
            if (outer == 0) gs->part[r][1] = gg;
        }
        if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;
        {
            double a = 0.0, b2 = 0.0;
            for (int k = 0; k < g; ++k) {  // rank order: the same sum in every block
                a += __ldcg(&gs->part[k][0]);
                if (outer == 0) b2 += __ldcg(&gs->part[k][1]);
            }
            if (outer == 0) gnorm = sqrt(b2);
            rel = gnorm > 0 ? sqrt(a) / gnorm : sqrt(a);
        }
        if (!isfinite(rel)) { status = CNV_NONFINITE; break; }
        if (rel <= rtol) { status = CNV_OK; break; }
        if (outer >= max_outer) break;
        for (int x = tid; x < 2 * plane; x += nt) smem[x] = 0.0f;
        __syncthreads();
        for (int e = 0; e < epochs; ++e) {
            for (int h = 1; h <= 2 * kStripSweeps; ++h) {
                const int c = (h - 1) & 1, grow = kStripHalo - h;
                const int lo = R0 - grow > 1 ? R0 - grow : 1;
                const int hi = R1 + grow < n - 1 ? R1 + grow : n - 1;
                if (C.vec)
                    quad_half_sweep<kRhsL2>(Q, c * plane - sr0 * sp, (c ^ 1) * plane - sr0 * sp, C.rq[c], 0, sp, P, lo, hi, c);
                else strip_half_sweep(es[c], es[c ^ 1], C.rq[c], sr0, sp, P, lo, hi, n, c, wxf, wyf, betaf);
                __syncthreads();
            }
            if (e + 1 < epochs) {
                // border rows -> exchange copy of this epoch's parity; halo rows <- neighbours'
                // (split columns m < (n+1)/2 hold every interior cell; both pitches cover them)
                float* const* X = (e & 1) ? C.ex1 : C.e;
                const int mw = (n + 1) / 2;
                for (int x = tid; x < 2 * kStripHalo * mw; x += nt) {
                    const int k = x / mw, m = x - k * mw;
                    const int i = k < kStripHalo ? R0 + k : R1 - 2 * kStripHalo + k;
                    if (i < 1 || i > n - 2 || i < R0 || i >= R1) continue;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int j = 2 * m + ((i + c) & 1);
                        if (j >= 1 && j <= n - 2) X[c][(size_t)i * P + m] = es[c][(i - sr0) * sp + m];
                    }
                }
                if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;
                for (int x = tid; x < 2 * kStripHalo * mw; x += nt) {
                    const int k = x / mw, m = x - k * mw;
                    const int i = k < kStripHalo ? R0 - kStripHalo + k : R1 + (k - kStripHalo);
                    if (i < 1 || i > n - 2 || i < sr0 || i >= sr1) continue;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int j = 2 * m + ((i + c) & 1);
                        if (j >= 1 && j <= n - 2) es[c][(i - sr0) * sp + m] = __ldcg(X[c] + (size_t)i * P + m);
                    }
                }
                __syncthreads();
            }
        }
        sweeps += C.inner;
        // psi += e (FP64) on the strip's own interior cells
        for (int x = tid; x < (ri1 - ri0) * (n - 2); x += nt) {
            const int i = ri0 + x / (n - 2), j = 1 + (x - (x / (n - 2)) * (n - 2));
            const int c = (i + j) & 1;
            C.psi[c][(size_t)i * P + (j >> 1)] += (double)es[c][(i - sr0) * sp + (j >> 1)];
        }
        if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;
    }

    // velocity u = DY psi, v = -(DX psi) on the strip's rows (src/main.c:366-383)
    auto PS = [&](int y, int x) { return LD(C.psi[(y + x) & 1] + (size_t)y * P + (x >> 1)); };
    for (int x = tid; x < rows * n; x += nt) {
        const int i = R0 + x / n, j = x - (x / n) * n;
        const size_t k = (size_t)i * n + j;
        C.u[k] = along_i<kMulInt>(B->d1y, n, i, j, PS);
        C.v[k] = -along_j<kMulInt>(B->d1x, n, i, j, PS);
        C.psi_rm[k] = PS(i, j);
    }
    if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;
    // continuity DX u + DY v on the strip's rows, max and min over the group (src/main.c:387-408)
    double mx = -DBL_MAX, mn = DBL_MAX;
    auto Uf = [&](int y, int x) { return LD(C.u + (size_t)y * n + x); };
    auto Vf = [&](int y, int x) { return LD(C.v + (size_t)y * n + x); };
    for (int x = tid; x < rows * n; x += nt) {
        const int i = R0 + x / n, j = x - (x / n) * n;
        const double cv = dadd(along_j<kMulInt>(B->d1x, n, i, j, Uf), along_i<kMulInt>(B->d1y, n, i, j, Vf));
        mx = cv > mx ? cv : mx;
        mn = cv < mn ? cv : mn;
    }
    block_minmax(mx, mn, s_red);
    if (tid == 0) {
        gs->cont[r][0] = mx;
        gs->cont[r][1] = mn;
    }
    if (!group_barrier(gs, gen, g, abort, s_ok)) return CNV_TIMEOUT;
    mx = -DBL_MAX;
    mn = DBL_MAX;
    for (int k = 0; k < g; ++k) {
        const double a = __ldcg(&gs->cont[k][0]), b2 = __ldcg(&gs->cont[k][1]);
        mx = a > mx ? a : mx;
        mn = b2 < mn ? b2 : mn;
    }
    rec.iters = outer;
    rec.status = status;
    rec.err = rel;
    rec.cont_max = mx;
    rec.cont_min = mn;
    return status;
}

template <bool SMALL>
__global__ void __launch_bounds__(kMaxBatchThreads) k_batch(BatchLaunch L) {
    float* const smem = bt_smem;
    __shared__ double s_red[64];
    __shared__ int s_ok;
    const int nsteps = *L.nsteps;
    for (int e = L.sched_off[blockIdx.x]; e < L.sched_off[blockIdx.x + 1]; ++e) {
        const SchedEntry J = L.sched[e];
        CavityDesc& C = L.cav[J.cav];
        if (SMALL || J.group == 1) {
            if (threadIdx.x == 0) {
                C.sweeps = 0;
                C.steps_done = 0;
            }
            __syncthreads();
            for (int t = 0; t < nsteps; ++t) {
                const int st = batch_step<SMALL>(C, smem, L.max_outer, L.rtol, L.warm != 0, s_red);
                if (threadIdx.x == 0) C.steps_done = t + 1;
                if (st != CNV_OK) break;
            }
            __syncthreads();
            continue;
        }
        // a strip of a cavity shared by J.group blocks; the descriptor's cur, sweeps, record and
        // step count are written once, by rank 0, when the job ends
        GroupSync* gs = L.gsync + J.cav;
        unsigned gen = 0;
        int cur = C.cur;
        long long sweeps = 0;
        int done = 0;
        StepRecord rec{};
        for (int t = 0; t < nsteps; ++t) {
            const int st = group_step(C, cur, J.rank, J.group, smem, L.max_outer, L.rtol, L.warm != 0, s_red, gs, gen,
                                      L.abort, &s_ok, sweeps, rec);
            if (st == CNV_TIMEOUT) {
                rec.status = CNV_TIMEOUT;
                break;
            }
            cur ^= 1;
            done = t + 1;
            if (st != CNV_OK) break;
        }
        __syncthreads();
        if (J.rank == 0 && threadIdx.x == 0) {
            C.cur = cur;
            C.sweeps = sweeps;
            C.steps_done = done;
            C.last = rec;
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace cnv

using namespace cnv;

struct cnv_batch {
    int count = 0;
    int device = 0;
    int sms = 0;
    cudaStream_t stream = nullptr;
    std::vector<cnv_cavity_spec> specs;
    std::vector<CavityDesc> host_desc;
    CavityDesc* desc = nullptr;
    FdBands* bands = nullptr;
    void* arena = nullptr;
    size_t arena_bytes = 0;
    // test_guard_cells: byte offsets into the arena of the guard regions (kBatchGuardBytes of 0xFF
    // before the first buffer and after every buffer) and what each follows
    std::vector<std::pair<size_t, std::string>> guards;
    SchedEntry* sched = nullptr;   // job lists (device)
    int* sched_off = nullptr;      // per block offsets into sched (device)
    GroupSync* gsync = nullptr;    // per cavity (device)
    int* abort = nullptr;          // group-wait failure flag (device)
    int split = 1;                 // strips per cavity beyond what shared memory needs
    int split_min_n = 256;         // ... for cavities of at least this many points per side
    std::vector<std::pair<int, int>> group_by_n;  // (n, group) chosen by the cost model; empty: rule above
    int* nsteps = nullptr;
    int threads = 1024;
    int blocks = 0;
    int smem_bytes = 0;
    int max_outer = 100;
    double rtol = 1e-10;
    int warm = 0;
    cudaGraphExec_t graph = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    double last_ms = 0;
    long long cells = 0;
    double makespan_us = 0;        // the schedule's estimated step time
    std::string err;
};

namespace {

int bfail(int status, const std::string& msg) {
    set_last_error(msg.c_str());
    return status;
}

// CNV_OK, or CNV_CUDA_ERROR naming the first guard region (test_guard_cells) whose bytes changed.
int check_guards(cnv_batch* b) {
    if (b->guards.empty()) return CNV_OK;
    std::vector<unsigned char> h(kBatchGuardBytes);
    for (const auto& g : b->guards) {
        if (cudaMemcpy(h.data(), static_cast<char*>(b->arena) + g.first, kBatchGuardBytes, cudaMemcpyDeviceToHost) !=
            cudaSuccess)
            return bfail(CNV_CUDA_ERROR, "guard check: copy failed");
        for (size_t k = 0; k < kBatchGuardBytes; ++k)
            if (h[k] != 0xFF)
                return bfail(CNV_CUDA_ERROR, "guard bytes " + g.second + " changed (byte " + std::to_string(k) + ")");
    }
    return CNV_OK;
}

#define BCUDA(call)                                                                                   \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) return bfail(CNV_CUDA_ERROR, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

inline unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Row strips a cavity needs so that one strip's FP32 correction (plus halo rows) fits a block's
// shared memory: 1 if the whole cavity's correction fits, else the smallest count that does
// (strips at least 2 halos high). 0 if no decomposition fits.
int min_group(int n, int smem_bytes) {
    const size_t sp = (size_t)(n + 1) / 2 + 1;
    if (2 * (size_t)n * sp * 4 <= (size_t)smem_bytes) return 1;
    for (int t = 2; t <= kMaxGroup && n / t >= 2 * kStripHalo; ++t) {
        const size_t rows = (size_t)(n + t - 1) / t + 2 * kStripHalo;
        if (2 * rows * sp * 4 <= (size_t)smem_bytes) return t;
    }
    return 0;
}

// min_group, then `split` times more (doubling while the strips stay 2 halos high) for cavities
// of at least min_n points. 0 if no decomposition fits.
int group_size(int n, int smem_bytes, int split, int min_n) {
    int g = min_group(n, smem_bytes);
    if (!g) return 0;
    if (n >= min_n)
        while (split > 1 && g * 2 <= kMaxGroup && n / (g * 2) >= 2 * kStripHalo) {
            g *= 2;
            split /= 2;
        }
    return g;
}

// Estimated device time of one step of an n x n cavity on g blocks (microseconds): about 4n FP32
// sweeps over n^2 cells at the measured per-SM rates (3.9 k cells/us with the correction in
// shared memory, 1.5 k from L2), with the halo rows of a strip, plus the FP64 passes; and for a
// group, its barriers: one per 4 FP32 sweeps (the border-row swap) plus about 20 around the
// residual norms and the passes, each about kBarrierUs (the wait for the slowest strip and the
// halo rows' L2 round trip), which the strips cannot share out. The rates are those of the scalar sweeps; the vector sweeps do
// about 9 k cells/us, so the estimates are too high (256 cavities 35.3 ms, measured 18.7; ten of 192^2 3.72 and 2.79).
constexpr double kBarrierUs = 3.5;

double step_cost(int n, int g, int smem_mode) {
    const double cells = (double)n * n;
    const double rate = (g > 1 || smem_mode >= 1) ? 3.9e3 : 1.5e3;
    const double halo = g > 1 ? ((double)n / g + 2 * kStripHalo) / ((double)n / g) : 1.0;
    const double barriers = g > 1 ? kBarrierUs * (n + 20.0) : 0.0;
    return (4.0 * n * cells / rate * halo + 0.061 * cells) / g + barriers;
}

bool small_batch(const cnv_batch* b) {
    return std::all_of(b->host_desc.begin(), b->host_desc.end(), [](const CavityDesc& d) { return d.n < kSmallN; });
}

const void* kernel_of(const cnv_batch* b) {
    return small_batch(b) ? reinterpret_cast<const void*>(&k_batch<true>) : reinterpret_cast<const void*>(&k_batch<false>);
}

int build_graph(cnv_batch* b) {
    if (b->graph) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
    BatchLaunch L{};
    L.cav = b->desc;
    L.sched = b->sched;
    L.sched_off = b->sched_off;
    L.gsync = b->gsync;
    L.abort = b->abort;
    L.nsteps = b->nsteps;
    L.count = b->count;
    L.max_outer = b->max_outer;
    L.rtol = b->rtol;
    L.warm = b->warm;
    L.smem_floats = b->smem_bytes / 4;
    const void* kernel = kernel_of(b);
    BCUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, b->smem_bytes));
    cudaGraph_t g = nullptr;
    BCUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t me = cudaMemsetAsync(b->gsync, 0, sizeof(GroupSync) * b->count, b->stream);
    if (me == cudaSuccess) me = cudaMemsetAsync(b->abort, 0, sizeof(int), b->stream);
    // cooperative: the blocks of a group wait for one another, so all must be resident
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b->blocks);
    cfg.blockDim = dim3(b->threads);
    cfg.dynamicSmemBytes = b->smem_bytes;
    cfg.stream = b->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {&L};
    const cudaError_t le =
        me != cudaSuccess ? me : cudaLaunchKernelExC(&cfg, kernel, args);
    cudaError_t e = cudaStreamEndCapture(b->stream, &g);
    if (le != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return bfail(CNV_CUDA_ERROR, std::string("batch launch: ") + cudaGetErrorString(le));
    }
    if (e != cudaSuccess) return bfail(CNV_CUDA_ERROR, std::string("batch capture: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return bfail(CNV_CUDA_ERROR, std::string("batch instantiate: ") + cudaGetErrorString(e));
    return CNV_OK;
}

// Greedy placement of one step's jobs: cavities largest estimated cost first, each on the
// `group` blocks that become free first. Fills the per-block lists (start-time order) when asked;
// returns the estimated makespan (microseconds).
struct Placed {
    double start;
    int cav, rank, group;
};

double place_jobs(const std::vector<CavityDesc>& desc, int nb, std::vector<std::vector<Placed>>* lists) {
    const int count = (int)desc.size();
    std::vector<int> idx(count);
    std::iota(idx.begin(), idx.end(), 0);
    std::vector<double> cost(count);
    for (int k = 0; k < count; ++k) cost[k] = step_cost(desc[k].n, desc[k].group, desc[k].smem_mode);
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int c) { return cost[a] > cost[c]; });
    std::vector<double> avail(nb, 0.0);
    std::vector<int> blocks(nb);
    for (int k : idx) {
        const int g = desc[k].group;
        std::iota(blocks.begin(), blocks.end(), 0);
        std::partial_sort(blocks.begin(), blocks.begin() + g, blocks.end(), [&](int a, int c) {
            return avail[a] < avail[c] || (avail[a] == avail[c] && a < c);
        });
        double start = 0.0;
        for (int r = 0; r < g; ++r) start = std::max(start, avail[blocks[r]]);
        for (int r = 0; r < g; ++r) {
            if (lists) (*lists)[blocks[r]].push_back(Placed{start, k, r, g});
            avail[blocks[r]] = start + cost[k];
        }
    }
    return *std::max_element(avail.begin(), avail.end());
}

// Job lists of the current decomposition (see place_jobs), on the device; every block's list in
// start-time order, so the blocks of a group reach their common jobs in one global order.
int build_schedule(cnv_batch* b) {
    const int nb = b->blocks;
    for (const auto& d : b->host_desc)
        if (d.group > nb) return bfail(CNV_BAD_ARG, "a cavity needs more blocks than the device runs at once");
    std::vector<std::vector<Placed>> lists(nb);
    b->makespan_us = place_jobs(b->host_desc, nb, &lists);
    std::vector<SchedEntry> flat;
    std::vector<int> off(nb + 1, 0);
    for (int q = 0; q < nb; ++q) {
        // start times are non-decreasing within a list already; keep that order
        off[q] = (int)flat.size();
        for (const Placed& e : lists[q]) flat.push_back(SchedEntry{e.cav, e.rank, e.group, 0});
    }
    off[nb] = (int)flat.size();
    if (b->sched) cudaFree(b->sched);
    if (b->sched_off) cudaFree(b->sched_off);
    b->sched = nullptr;
    b->sched_off = nullptr;
    BCUDA(cudaMalloc(&b->sched, sizeof(SchedEntry) * std::max<size_t>(flat.size(), 1)));
    BCUDA(cudaMalloc(&b->sched_off, sizeof(int) * (nb + 1)));
    if (!flat.empty())
        BCUDA(cudaMemcpy(b->sched, flat.data(), sizeof(SchedEntry) * flat.size(), cudaMemcpyHostToDevice));
    BCUDA(cudaMemcpy(b->sched_off, off.data(), sizeof(int) * (nb + 1), cudaMemcpyHostToDevice));
    return CNV_OK;
}

// The decomposition of every cavity for a shared-memory size: group_size's strips (split times
// more than needed for cavities of at least split_min_n points), or the (n, group) overrides; the
// placement of the FP32 correction (smem_mode) to match.
void assign_groups(std::vector<CavityDesc>& desc, int smem_bytes, int split, int split_min_n,
                   const std::vector<std::pair<int, int>>& group_by_n) {
    for (auto& d : desc) {
        const size_t plane = (size_t)d.n * d.spitch * 4;
        d.smem_mode = 4 * plane <= (size_t)smem_bytes ? 2 : 2 * plane <= (size_t)smem_bytes ? 1 : 0;
        d.group = group_size(d.n, smem_bytes, split, split_min_n);
        for (const auto& ng : group_by_n)
            if (ng.first == d.n && d.group > 0) d.group = ng.second;
        if (d.group == 0) d.group = 1;  // no strip decomposition fits: one block, correction in L2
        if (d.group > 1) d.smem_mode = 1;
    }
}

// Smallest cavity that fits one block and that the cost model may still split: two strips of at
// least two halos each. The model weighs the group barriers, so it leaves small cavities whole
// unless splitting them shortens the schedule.
constexpr int kMinSplitN = 4 * kStripHalo;

// Group sizes chosen by the cost model: each of the three largest distinct cavity sizes that
// needs row strips, or fits one block and has at least kMinSplitN points, gets a group from the
// smallest that fits to three more (strips at least 2 halos high, at most `blocks`), the sizes
// tried jointly (smaller ones keep the smallest group), and the combination with the smallest
// estimated makespan is returned as (n, group) pairs. A size that fits one block is so split when
// that shortens the schedule (a few large cavities on many blocks).
std::vector<std::pair<int, int>> model_groups(const std::vector<CavityDesc>& in, int smem_bytes, int blocks) {
    std::vector<int> sizes;
    for (const auto& d : in)
        if ((min_group(d.n, smem_bytes) >= 2 || (min_group(d.n, smem_bytes) == 1 && d.n >= kMinSplitN)) &&
            std::find(sizes.begin(), sizes.end(), d.n) == sizes.end())
            sizes.push_back(d.n);
    std::sort(sizes.rbegin(), sizes.rend());
    if (sizes.size() > 3) sizes.resize(3);
    std::vector<std::vector<int>> opts;
    for (int n : sizes) {
        std::vector<int> o;
        const int g0 = min_group(n, smem_bytes);
        for (int g = g0; g <= g0 + 3 && g <= kMaxGroup && g <= blocks && n / g >= 2 * kStripHalo; ++g) o.push_back(g);
        if (o.empty()) o.push_back(g0);  // more than the device runs: build_schedule reports it
        opts.push_back(o);
    }
    std::vector<CavityDesc> desc = in;
    std::vector<std::pair<int, int>> trial;
    std::vector<int> pick(sizes.size(), 0), best_pick = pick;
    double best = 1e300;
    for (;;) {
        trial.clear();
        for (size_t q = 0; q < sizes.size(); ++q) trial.emplace_back(sizes[q], opts[q][pick[q]]);
        assign_groups(desc, smem_bytes, 1, 1, trial);
        bool fits = true;
        for (const auto& d : desc) fits = fits && d.group <= blocks;
        const double ms = fits ? place_jobs(desc, blocks, nullptr) : 1e300;
        if (ms < best) {
            best = ms;
            best_pick = pick;
        }
        size_t q = 0;  // next combination
        while (q < sizes.size() && ++pick[q] == (int)opts[q].size()) pick[q++] = 0;
        if (q == sizes.size()) break;
    }
    std::vector<std::pair<int, int>> out;
    for (size_t q = 0; q < sizes.size(); ++q) out.emplace_back(sizes[q], opts[q][best_pick[q]]);
    return out;
}

void model_groups(cnv_batch* b) { b->group_by_n = model_groups(b->host_desc, b->smem_bytes, b->blocks); }

// Launch shape: threads per block and blocks per SM; shared memory as the SM allows; the strip
// decomposition and the job lists for it.
int set_shape(cnv_batch* b, int threads, int per_sm) {
    int dev_smem = 0;
    BCUDA(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, b->device));
    int optin = 0;
    BCUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, b->device));
    b->threads = threads;
    b->smem_bytes = std::min(optin, dev_smem / per_sm - 2048) & ~255;
    int occ = 0;
    const void* kernel = kernel_of(b);
    BCUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, b->smem_bytes));
    BCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, b->smem_bytes));
    if (occ < 1) return bfail(CNV_CUDA_ERROR, "batched kernel does not fit on an SM");
    b->blocks = std::min(occ, per_sm) * b->sms;
    // per-cavity placement of the FP32 correction for this shared-memory size, and row strips
    assign_groups(b->host_desc, b->smem_bytes, b->split, b->split_min_n, b->group_by_n);
    // the vector sweeps where the tile fits with rows of whole vectors (nearly always: the plan counts one column more)
    const bool small = small_batch(b);
    for (auto& d : b->host_desc) {
        const int p4 = ((d.n + 1) / 2 + 3) / 4 * 4;
        const size_t rows = d.group > 1 ? (size_t)(d.n + d.group - 1) / d.group + 2 * kStripHalo : d.n;
        d.vec = !small && d.smem_mode >= 1 && 8 * rows * p4 <= (size_t)b->smem_bytes ? 1 : 0;
        d.epitch = d.vec ? p4 : d.spitch;
        if (d.vec && d.smem_mode == 2 && 16 * rows * p4 > (size_t)b->smem_bytes) d.smem_mode = 1;
    }
    BCUDA(cudaMemcpy(b->desc, b->host_desc.data(), sizeof(CavityDesc) * b->count, cudaMemcpyHostToDevice));
    const int rc = build_schedule(b);
    if (rc != CNV_OK) return rc;
    return build_graph(b);
}

int reset_fields(cnv_batch* b) {
    BCUDA(cudaMemsetAsync(b->arena, 0, b->arena_bytes, b->stream));
    for (const auto& g : b->guards)
        BCUDA(cudaMemsetAsync(static_cast<char*>(b->arena) + g.first, 0xFF, kBatchGuardBytes, b->stream));
    for (auto& d : b->host_desc) d.cur = 0;
    BCUDA(cudaMemcpyAsync(b->desc, b->host_desc.data(), sizeof(CavityDesc) * b->count, cudaMemcpyHostToDevice,
                          b->stream));
    BCUDA(cudaStreamSynchronize(b->stream));
    return CNV_OK;
}

int run(cnv_batch* b, int nsteps) {
    BCUDA(cudaMemcpyAsync(b->nsteps, &nsteps, sizeof(int), cudaMemcpyHostToDevice, b->stream));
    BCUDA(cudaEventRecord(b->ev0, b->stream));
    BCUDA(cudaGraphLaunch(b->graph, b->stream));
    BCUDA(cudaEventRecord(b->ev1, b->stream));
    BCUDA(cudaStreamSynchronize(b->stream));
    float ms = 0;
    cudaEventElapsedTime(&ms, b->ev0, b->ev1);
    b->last_ms = ms;
    return CNV_OK;
}

}  // namespace

extern "C" {

int cnv_batch_specs(int count, unsigned long long seed, cnv_cavity_spec* out) {
    if (count < 0 || (count > 0 && !out)) return bfail(CNV_BAD_ARG, "bad count or null output");
    static const int kSizes[6] = {64, 96, 128, 192, 256, 384};
    for (int k = 0; k < count; ++k) {
        const unsigned long long base = seed + 3ull * (unsigned long long)k * 0x9E3779B97F4A7C15ull;
        const double u1 = (double)(mix64(base) >> 11) * 0x1.0p-53;
        const double u2 = (double)(mix64(base + 0x9E3779B97F4A7C15ull) >> 11) * 0x1.0p-53;
        const double u3 = (double)(mix64(base + 2 * 0x9E3779B97F4A7C15ull) >> 11) * 0x1.0p-53;
        out[k].n = kSizes[std::min(5, (int)(u1 * 6))];
        out[k].Re = 100.0 + 1900.0 * u2;
        out[k].lid = 0.5 + u3;
        out[k].dt = 0.0;
    }
    return CNV_OK;
}

int cnv_batch_plan(int count, const cnv_cavity_spec* specs, int blocks, int smem_bytes, int* groups,
                   double* makespan_us) {
    if (count < 1 || !specs || !groups || blocks < 1 || smem_bytes < 1024)
        return bfail(CNV_BAD_ARG, "bad count, block count or shared-memory size, or null argument");
    std::vector<CavityDesc> desc(count);
    for (int k = 0; k < count; ++k) {
        const int n = specs[k].n;
        if (n < 4 || n > 4096) return bfail(CNV_BAD_ARG, "cavity " + std::to_string(k) + ": n out of range");
        std::memset(&desc[k], 0, sizeof(CavityDesc));
        desc[k].n = n;
        desc[k].spitch = (n + 1) / 2 + 1;
    }
    assign_groups(desc, smem_bytes, 1, 1, model_groups(desc, smem_bytes, blocks));
    for (int k = 0; k < count; ++k) {
        if (desc[k].group > blocks) return bfail(CNV_BAD_ARG, "a cavity needs more blocks than the device runs at once");
        groups[k] = desc[k].group;
    }
    if (makespan_us) *makespan_us = place_jobs(desc, blocks, nullptr);
    return CNV_OK;
}

int cnv_batch_create(const cnv_config* base, int count, const cnv_cavity_spec* specs, cnv_batch** out) {
    if (!base || !specs || !out || count < 1) return bfail(CNV_BAD_ARG, "null argument or empty batch");
    *out = nullptr;
    if (base->test_guard_cells < 0 || base->test_guard_cells > 2)
        return bfail(CNV_BAD_ARG, "test_guard_cells must be 0, 1 or 2");
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, base->device) != cudaSuccess || prop.major != 10 || prop.minor != 3)
        return bfail(CNV_NO_DEVICE, "no sm_103 device");
    BCUDA(cudaSetDevice(base->device));
    for (int k = 0; k < count; ++k) {
        const int n = specs[k].n;
        if (n < (base->order == 6 ? 5 : 4) || n > 4096 || !(specs[k].Re > 0) || !(specs[k].lid == specs[k].lid))
            return bfail(CNV_BAD_ARG, "cavity " + std::to_string(k) + ": bad size, Re or lid speed");
    }
    cnv_batch* b = new cnv_batch();
    b->count = count;
    b->device = base->device;
    b->sms = prop.multiProcessorCount;
    b->specs.assign(specs, specs + count);
    b->max_outer = base->mixed_max_outer > 0 ? base->mixed_max_outer : 100;
    b->rtol = base->mixed_rtol > 0 ? base->mixed_rtol : 1e-10;
    b->warm = base->mixed_warm_start ? 1 : 0;
    auto cleanup = [&](int rc, const std::string& m) {
        cnv_batch_destroy(b);
        return bfail(rc, m);
    };
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&b->ev0) != cudaSuccess || cudaEventCreate(&b->ev1) != cudaSuccess)
        return cleanup(CNV_CUDA_ERROR, "stream/event creation failed");

    // arena: per cavity w[2], u, v, psi_rm (n*n doubles each), psi/g split (2 x n*pitch doubles
    // each), e/rq/ex1 split (2 x n*pitch floats each), each 256-byte aligned; with
    // test_guard_cells a guard region before the first and after every buffer
    const size_t gap = base->test_guard_cells ? kBatchGuardBytes : 0;
    auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
    auto cavity_bytes = [&](int n, int pitch) {
        return 5 * (align((size_t)n * n * 8) + gap) + 4 * (align((size_t)n * pitch * 8) + gap) +
               6 * (align((size_t)n * pitch * 4) + gap);
    };
    std::vector<size_t> offs(count);
    size_t total = gap;
    b->host_desc.resize(count);
    for (int k = 0; k < count; ++k) {
        const int n = specs[k].n;
        const int pitch = ((n + 1) / 2 + 31) / 32 * 32;
        offs[k] = total;
        total += cavity_bytes(n, pitch);
        b->cells += (long long)n * n;
    }
    b->arena_bytes = total;
    if (gap) b->guards.emplace_back(0, "before cavity 0");
    if (cudaMalloc(&b->arena, total) != cudaSuccess) return cleanup(CNV_CUDA_ERROR, "arena allocation failed");
    if (cudaMalloc(&b->desc, sizeof(CavityDesc) * count) != cudaSuccess ||
        cudaMalloc(&b->bands, sizeof(FdBands) * count) != cudaSuccess ||
        cudaMalloc(&b->gsync, sizeof(GroupSync) * count) != cudaSuccess ||
        cudaMalloc(&b->abort, sizeof(int)) != cudaSuccess || cudaMalloc(&b->nsteps, sizeof(int)) != cudaSuccess)
        return cleanup(CNV_CUDA_ERROR, "descriptor allocation failed");

    std::vector<FdBands> hb(count);
    const double pi = 3.14159265359;  // include/poisson.h:8
    for (int k = 0; k < count; ++k) {
        const int n = specs[k].n;
        const int pitch = ((n + 1) / 2 + 31) / 32 * 32;
        CavityDesc& d = b->host_desc[k];
        std::memset(&d, 0, sizeof d);
        d.n = n;
        d.pitch = pitch;
        d.spitch = (n + 1) / 2 + 1;
        const double dx = (double)base->Lx / n, dy = (double)base->Ly / n;
        const double h = dx;
        const double dt = specs[k].dt > 0 ? specs[k].dt
                                          : 0.2 * std::min(h * h * specs[k].Re / 4.0, h / std::fabs(specs[k].lid));
        if (build_fd_bands(n, base->order, dx, dy, &hb[k]) != CNV_OK)
            return cleanup(CNV_BAD_ARG, "finite-difference bands for cavity " + std::to_string(k));
        d.inv_re = 1. / specs[k].Re;
        d.dt = dt;
        const double beta_ref = 0.5 * (2 / (1 + sin(pi / (n + 1))) + 2 / (1 + sin(pi / (n + 1))));
        d.beta = base->sor_omega > 0 ? base->sor_omega : beta_ref;
        d.c4 = dx * dx * dy * dy;
        d.dx2 = dx * dx;
        d.dy2 = dy * dy;
        d.den = 2 * (dx * dx + dy * dy);
        d.rden = 1.0 / d.den;
        d.bc = BoundaryValues{base->u1, base->u2, base->u3, specs[k].lid, base->v1, base->v2, base->v3, base->v4};
        // FP32 sweeps per correction, rounded up to whole epochs exactly as the single-cavity
        // mixed solve does, so that both give the same iterates
        const int want = base->mixed_inner_sweeps > 0 ? base->mixed_inner_sweeps : n;
        const int per_epoch = mixed_sweeps_per_exchange();
        d.inner = std::max(1, (want + per_epoch - 1) / per_epoch) * per_epoch;
        d.bands = b->bands + k;
        size_t cur = offs[k];
        auto take = [&](size_t bytes, const char* name) {
            char* q = static_cast<char*>(b->arena) + cur;
            cur += align(bytes);
            if (gap) b->guards.emplace_back(cur, "after cavity " + std::to_string(k) + "'s " + name);
            cur += gap;
            return q;
        };
        const size_t f64b = (size_t)n * n * 8, sp64 = (size_t)n * pitch * 8, sp32 = (size_t)n * pitch * 4;
        d.w[0] = reinterpret_cast<double*>(take(f64b, "w[0]"));
        d.w[1] = reinterpret_cast<double*>(take(f64b, "w[1]"));
        d.u = reinterpret_cast<double*>(take(f64b, "u"));
        d.v = reinterpret_cast<double*>(take(f64b, "v"));
        d.psi_rm = reinterpret_cast<double*>(take(f64b, "psi"));
        d.psi[0] = reinterpret_cast<double*>(take(sp64, "split psi[0]"));
        d.psi[1] = reinterpret_cast<double*>(take(sp64, "split psi[1]"));
        d.g[0] = reinterpret_cast<double*>(take(sp64, "g[0]"));
        d.g[1] = reinterpret_cast<double*>(take(sp64, "g[1]"));
        d.e[0] = reinterpret_cast<float*>(take(sp32, "e[0]"));
        d.e[1] = reinterpret_cast<float*>(take(sp32, "e[1]"));
        d.rq[0] = reinterpret_cast<float*>(take(sp32, "rq[0]"));
        d.rq[1] = reinterpret_cast<float*>(take(sp32, "rq[1]"));
        d.ex1[0] = reinterpret_cast<float*>(take(sp32, "ex1[0]"));
        d.ex1[1] = reinterpret_cast<float*>(take(sp32, "ex1[1]"));
        d.group = 1;
    }
    if (cudaMemcpy(b->bands, hb.data(), sizeof(FdBands) * count, cudaMemcpyHostToDevice) != cudaSuccess)
        return cleanup(CNV_CUDA_ERROR, "descriptor upload failed");
    // the strip counts the cost model picks (set_shape first gives it the launch shape)
    int rc = reset_fields(b);
    if (rc == CNV_OK) rc = set_shape(b, 1024, 1);
    if (rc == CNV_OK) {
        model_groups(b);
        rc = set_shape(b, 1024, 1);
    }
    if (rc == CNV_OK && base->test_guard_cells == 2) {
        // the checker's own test: one changed byte in the guard after cavity 0's u
        for (const auto& g : b->guards)
            if (g.second == "after cavity 0's u" &&
                cudaMemset(static_cast<char*>(b->arena) + g.first, 0, 1) != cudaSuccess)
                rc = bfail(CNV_CUDA_ERROR, "guard setup failed");
    }
    if (rc != CNV_OK) {
        cnv_batch_destroy(b);
        return rc;
    }
    *out = b;
    return CNV_OK;
}

void cnv_batch_destroy(cnv_batch* b) {
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->graph) cudaGraphExecDestroy(b->graph);
    for (void* p : {(void*)b->arena, (void*)b->desc, (void*)b->bands, (void*)b->sched, (void*)b->sched_off,
                    (void*)b->gsync, (void*)b->abort, (void*)b->nsteps})
        if (p) cudaFree(p);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

int cnv_batch_reset(cnv_batch* b) {
    if (!b) return bfail(CNV_BAD_ARG, "null batch");
    BCUDA(cudaSetDevice(b->device));
    return reset_fields(b);
}

int cnv_batch_tune(cnv_batch* b, int* threads_out, int* blocks_per_sm_out) {
    if (!b) return bfail(CNV_BAD_ARG, "null batch");
    BCUDA(cudaSetDevice(b->device));
    // candidates: row-strip decompositions (strips only where shared memory needs them, or 2x or
    // 4x as many for the largest cavities, or the groups the cost model picks), each timed for
    // one step from the initial state, on one block of 1024 threads per SM (the shared-memory
    // tiles need the whole SM)
    const int cand[][3] = {{1, 256, 0}, {2, 256, 0}, {4, 256, 0}, {2, 192, 0}, {1, 256, 1}};
    double best = 1e300;
    int bs = 1, bm = 256;
    std::vector<std::pair<int, int>> bg;
    for (const auto& c : cand) {
        b->split = c[0];
        b->split_min_n = c[1];
        b->group_by_n.clear();
        int rc = set_shape(b, 1024, 1);
        if (rc != CNV_OK) continue;
        if (c[2]) {
            model_groups(b);
            rc = set_shape(b, 1024, 1);
            if (rc != CNV_OK) continue;
        }
        rc = reset_fields(b);
        if (rc == CNV_OK) rc = run(b, 1);
        if (rc != CNV_OK) return rc;
        if (b->last_ms < best) {
            best = b->last_ms;
            bs = c[0];
            bm = c[1];
            bg = b->group_by_n;
        }
    }
    b->split = bs;
    b->split_min_n = bm;
    b->group_by_n = bg;
    int rc = set_shape(b, 1024, 1);
    if (rc == CNV_OK) rc = reset_fields(b);
    if (threads_out) *threads_out = b->threads;
    if (blocks_per_sm_out) *blocks_per_sm_out = 1;
    return rc;
}

int cnv_batch_split(cnv_batch* b, int factor, int min_n) {
    if (!b || factor < 1 || factor > kMaxGroup || min_n < 1) return bfail(CNV_BAD_ARG, "bad batch or split factor");
    BCUDA(cudaSetDevice(b->device));
    b->split = factor;
    b->split_min_n = min_n;
    b->group_by_n.clear();
    int rc = set_shape(b, 1024, 1);
    if (rc == CNV_OK) rc = reset_fields(b);
    return rc;
}

int cnv_batch_groups(cnv_batch* b, int* groups) {
    if (!b || !groups) return bfail(CNV_BAD_ARG, "null argument");
    for (int k = 0; k < b->count; ++k) groups[k] = b->host_desc[k].group;
    return CNV_OK;
}

int cnv_batch_step(cnv_batch* b, int nsteps, cnv_step_info* last) {
    if (!b || nsteps < 0) return bfail(CNV_BAD_ARG, "bad batch or step count");
    BCUDA(cudaSetDevice(b->device));
    int rc = run(b, nsteps);
    if (rc != CNV_OK) return rc;
    rc = check_guards(b);
    if (rc != CNV_OK) return rc;
    int aborted = 0;
    BCUDA(cudaMemcpy(&aborted, b->abort, sizeof(int), cudaMemcpyDeviceToHost));
    BCUDA(cudaMemcpy(b->host_desc.data(), b->desc, sizeof(CavityDesc) * b->count, cudaMemcpyDeviceToHost));
    if (aborted) return bfail(CNV_TIMEOUT, "a wait between the blocks of a cavity's group gave up");
    int status = CNV_OK;
    for (int k = 0; k < b->count; ++k) {
        const CavityDesc& d = b->host_desc[k];
        if (last) std::memcpy(&last[k], &d.last, sizeof(StepRecord));
        if (status == CNV_OK && (d.last.status != CNV_OK || d.steps_done != nsteps)) status = d.last.status ? d.last.status : CNV_CUDA_ERROR;
    }
    if (status != CNV_OK) return bfail(status, "a cavity's step did not converge");
    return CNV_OK;
}

int cnv_batch_get_fields(cnv_batch* b, int index, double* w, double* u, double* v, double* psi) {
    if (!b || index < 0 || index >= b->count) return bfail(CNV_BAD_ARG, "bad batch or index");
    BCUDA(cudaSetDevice(b->device));
    BCUDA(cudaMemcpy(&b->host_desc[index], b->desc + index, sizeof(CavityDesc), cudaMemcpyDeviceToHost));
    const CavityDesc& d = b->host_desc[index];
    const size_t bytes = (size_t)d.n * d.n * 8;
    if (w) BCUDA(cudaMemcpy(w, d.w[d.cur], bytes, cudaMemcpyDeviceToHost));
    if (u) BCUDA(cudaMemcpy(u, d.u, bytes, cudaMemcpyDeviceToHost));
    if (v) BCUDA(cudaMemcpy(v, d.v, bytes, cudaMemcpyDeviceToHost));
    if (psi) BCUDA(cudaMemcpy(psi, d.psi_rm, bytes, cudaMemcpyDeviceToHost));
    return CNV_OK;
}

int cnv_batch_stats(cnv_batch* b, long long* cells, long long* sweeps, double* ms) {
    if (!b) return bfail(CNV_BAD_ARG, "null batch");
    long long sw = 0;
    for (const auto& d : b->host_desc) sw += d.sweeps;
    if (cells) *cells = b->cells;
    if (sweeps) *sweeps = sw;
    if (ms) *ms = b->last_ms;
    return CNV_OK;
}

}  // extern "C"
