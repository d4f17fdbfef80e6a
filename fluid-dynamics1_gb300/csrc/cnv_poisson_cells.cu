// cnv_poisson_cells.cu -- FP64 red-black SOR / Gauss-Seidel up to 1100^2: a cell of each colour per thread (k_poisson_cells, to
// 515^2; FMA 514^2), or tiles of many cells in shared memory (k_poisson_rows, described there).
//
// The same solve as cnv_poisson.cu (the reference's point update and its stop rule, bit for bit), for grids where a sweep
// is a chain of latencies: 64^2 took 5.9 us per sweep and 256^2 6.2 with shared-memory tiles and a border exchange per four
// sweeps, most of it block barriers, fences, flags and recomputed halo cells (three times the cells at 256^2), where the FP64
// operations take 0.1 and 0.6 us.
//
// Cells. The interior is cut into gx x gy tiles, a block each; a compute thread owns one cell of each colour for the whole
// solve, its right-hand side and value in registers. Every iterate goes to a ring of kHist sweeps in shared memory, from which
// the neighbouring threads read; so a sweep is two updates with a block barrier after each, and nothing else on its path.
//
// Borders. A cell at a tile's edge is written to its neighbour's mailbox as two 64-bit words, each half of the value with the
// number of the sweep: the words arrive whole, so the reader polls them and needs no flag, the writer no fence. A mailbox
// cell needs no second copy: its next value is made from the neighbour's value across the edge, which was made from this one.
//   CLUSTER (16 tiles): the blocks form one thread-block cluster and the mailboxes lie in the readers' shared memory. A hop
//   takes 340 cycles.
//   Otherwise they lie in global memory (L2): 620 cycles within a die, up to 1,240 across.
// A sweep is two hops and two updates long (an FP64 operation: 64 cycles, and 16 to 19 cycles of the SM's pipe per warp).
//
// us per sweep, shared-memory tiles or exchange kernel -> here: folded SOR 64^2 5.60 -> 1.30, 256^2 5.70 -> 2.26, 512^2 8.27 ->
// 4.37; general SOR 97^2 5.76 -> 2.65, 192^2 6.29 -> 2.66, 300^2 7.98 -> 3.26, 500^2 10.4 -> 6.72; FMA 97^2 4.12 -> 1.45, 500^2
// 7.25 -> 3.58. Bound by the hops and the chain of FP64 latencies up to 300^2, by the FP64 pipe above.
//
// Stop test. Norm warps form the block's share of e_k from the ring (exact fixed-point sums, as in cnv_sor.cuh) while the
// compute warps run on, and add it to a global ring whose words count the blocks in their upper bits: no fence, no counter, and
// nothing is cleared (the verdict warps subtract what they read a turn before). A verdict warp in each block polls the words,
// evaluates e_k and lets the compute warps run on: sweep k starts when e_{k - kLag} is known, so every block stops before the
// same sweep, with the iterate of the one that converged still in the shared-memory ring. With a counter, fences and a cleared
// slot per sweep the verdicts limited the pace (3,000 cycles a sweep at 64^2); with all blocks' atomics on one line they slowed the
// mailboxes' traffic; gathered by one block and posted, the verdicts came too late (256^2: 2.87 ms a step, here 2.03).
//
// Every wait is bounded (timeout and abort flag) and records CNV_TIMEOUT; a thread that gives up keeps passing its block's
// barriers until the end of the sweep, where all of them learn of it and leave.
#include <algorithm>
#include <climits>

#include <cooperative_groups.h>

#include "cnv_kernels.h"
#include "cnv_sor.cuh"

namespace cnv {
namespace {

constexpr int kHist = 8;       // sweeps kept in shared memory
constexpr int kLag = 6;        // a sweep starts when the one kLag before it is known not to have converged
static_assert(kHist > kLag, "the iterate that converged is still in the ring");
constexpr int kNormRing = 32;  // sweeps' norms in flight: at least 3 kLag (see check_norms)
// Norm warps, a whole sweep's share each, in turn: at most 6, and a tile that leaves room for fewer than 3 (FMA, whose sweeps are
// shorter: 4) is left to k_poisson_rows, because their pace is then the sweep's. us per sweep with 4 / 3 / 2 of them, k_poisson_rows: general SOR
// 514^2 6.6, 515^2 7.5, 516^2 10.9 against 8.5 .. 8.6; FMA 4.8, 6.6, 10.5 against 5.6.
constexpr int kMinNormWarps = 3, kMinNormWarpsFma = 4, kMaxNormWarps = 6;

// The norm's ring. A slot's words: the chunk sums of e_k for the k of that slot, all turns of the ring added up, over the blocks
// b with b % kParts = part. Above kCountBit each word counts the blocks that added (a turn's sums stay below 2^50: 19 blocks of
// 8,300 cells of 32 bits); above kSideBit word 3, whose cells have 31 bits, counts those that added to the FP64 side sum.
constexpr int kParts = 8, kCountBit = 56, kSideBit = 50;
struct CellsSync {
    unsigned long long word[kNormRing][kParts][4];
    double fsum[kNormRing];
};
static_assert(sizeof(CellsSync) % 16 == 0, "the mailboxes follow");

struct CellsDev {
    PoissonParams p;
    int gx, gy;
    int tc;        // compute threads, a multiple of 32
    int nw;        // norm warps
    int rows, plane;  // tiles of many cells: rows per pass of the threads, doubles of a colour's plane
    int side;      // cells of a mailbox side
    const double* rhs[2];
    double* out[2];
    ulonglong2* mail;  // [block][4][side] (global form)
    Ctrl* ctrl;
    CellsSync* sync;
};

struct CellTile {
    int r0, r1, c0, c1;
};

__host__ __device__ __forceinline__ CellTile cell_tile(int n, int gx, int gy, int b) {
    const int ni = n - 2, tx = b % gx, ty = b / gx;
    return CellTile{1 + (int)((long long)ni * ty / gy), 1 + (int)((long long)ni * (ty + 1) / gy),
                    1 + (int)((long long)ni * tx / gx), 1 + (int)((long long)ni * (tx + 1) / gx)};
}

// Cells of a colour at a W x H tile's edge (W, H >= 2; going round it the colours alternate), and threads for a colour in all.
__host__ __device__ __forceinline__ int edge_cells(int W, int H) { return W + H - 2; }
__host__ __device__ __forceinline__ int colour_threads(int W, int H) { return edge_cells(W, H) + (H - 2) * ((W - 1) / 2); }

// The cell of colour c that thread x owns; false if it has none.
__device__ __forceinline__ bool cell_of(const CellTile& t, int c, int x, int& i, int& j) {
    const int W = t.c1 - t.c0, H = t.r1 - t.r0, ne = edge_cells(W, H);
    if (x < ne) {
        const int p = 2 * x + ((t.r0 + t.c0 + c) & 1);  // place going round: bottom row, right column, top row, left column
        if (p < W) {
            i = t.r0;
            j = t.c0 + p;
        } else if (p < W + H - 1) {
            i = t.r0 + p - W + 1;
            j = t.c1 - 1;
        } else if (p < 2 * W + H - 2) {
            i = t.r1 - 1;
            j = t.c1 - 2 - (p - (W + H - 1));
        } else {
            i = t.r1 - 2 - (p - (2 * W + H - 2));
            j = t.c0;
        }
        return true;
    }
    const int wq = (W - 1) / 2;
    if (wq == 0) return false;
    const int r = (x - ne) / wq;
    i = t.r0 + 1 + r;
    j = t.c0 + 1 + 2 * (x - ne - r * wq) + ((i + t.c0 + 1 + c) & 1);
    return i < t.r1 - 1 && j < t.c1 - 1;
}

// The thread that owns cell (i, j) of the tile.
__device__ __forceinline__ int owner_of(const CellTile& t, int i, int j) {
    const int W = t.c1 - t.c0, H = t.r1 - t.r0;
    int p;
    if (i == t.r0) p = j - t.c0;
    else if (j == t.c1 - 1) p = W - 1 + i - t.r0;
    else if (i == t.r1 - 1) p = W + H - 1 + t.c1 - 2 - j;
    else if (j == t.c0) p = 2 * W + H - 2 + t.r1 - 2 - i;
    else return edge_cells(W, H) + (i - t.r0 - 1) * ((W - 1) / 2) + ((j - t.c0 - 1) >> 1);
    return p >> 1;
}

// A cell's surroundings: the threads of its neighbours (tc: a wall, read as 0), and up to two neighbours in other tiles, with
// the mailbox place read and the one written for each (side -1: none). Directions 0 up (i + 1), 1 down, 2 right, 3 left.
struct Links {
    int nb[4];
    int dir[2], from[2], to[2], block[2];
};

__device__ __forceinline__ void link_cell(const CellTile& t, const CellsDev& L, int me, int i, int j, Links& k) {
    const int n = L.p.n;
    int found = 0;
    k.dir[0] = k.dir[1] = -1;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const int y = i + (d == 0) - (d == 1), x = j + (d == 2) - (d == 3);
        k.nb[d] = L.tc;
        if (y < 1 || y > n - 2 || x < 1 || x > n - 2) continue;
        if (y >= t.r0 && y < t.r1 && x >= t.c0 && x < t.c1) {
            k.nb[d] = owner_of(t, y, x);
            continue;
        }
        const int pos = d < 2 ? j - t.c0 : i - t.r0;  // tiles of a row (column) share their rows (columns)
        const int from = d * L.side + pos, to = (d ^ 1) * L.side + pos, b = me + (d == 0 ? L.gx : d == 1 ? -L.gx : d == 2 ? 1 : -1);
        if (found == 0) {
            k.dir[0] = d;
            k.from[0] = from;
            k.to[0] = to;
            k.block[0] = b;
        } else {
            k.dir[1] = d;
            k.from[1] = from;
            k.to[1] = to;
            k.block[1] = b;
        }
        ++found;
    }
}

__device__ __forceinline__ void cells_barrier(int count) { asm volatile("bar.sync 1, %0;" ::"r"(count) : "memory"); }
template <bool CLUSTER>
__device__ __forceinline__ ulonglong2 mail_read(const ulonglong2* p) {
    ulonglong2 v;
    if (CLUSTER) {
        const unsigned a = (unsigned)__cvta_generic_to_shared(p);
        asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a) : "memory");
    } else {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    }
    return v;
}

template <bool CLUSTER>
__device__ __forceinline__ void mail_write(ulonglong2* p, double x, unsigned tag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x), t = (unsigned long long)tag << 32;
    const unsigned long long lo = t | (b & 0xffffffffull), hi = t | (b >> 32);
    if (CLUSTER)
        asm volatile("st.relaxed.cluster.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
    else
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}

__device__ __forceinline__ bool mail_is(const ulonglong2& v, unsigned tag) {
    return (unsigned)(v.x >> 32) == tag && (unsigned)(v.y >> 32) == tag;
}
__device__ __forceinline__ double mail_value(const ulonglong2& v) {
    return __longlong_as_double((long long)((v.x & 0xffffffffull) | (v.y << 32)));
}

// The values of sweep `tag` from the mailboxes of a whole warp's cells, one (na) or two (nb) a lane, polled together until all are
// there: with a loop per lane the lanes left it apart and stayed apart through the update that follows (192^2: 9,600
// cycles a sweep), and a corner cell's second mailbox polled after the first cost a round trip. False: given up.
template <bool CLUSTER>
__device__ __forceinline__ bool mail_wait(const ulonglong2* a, const ulonglong2* b, bool na, bool nb, unsigned tag, Ctrl* ctl,
                                          long long timeout_ns, double& xa, double& xb) {
    long long t0 = 0;
    for (int polls = 1;; ++polls) {
        ulonglong2 va, vb;
        if (na) va = mail_read<CLUSTER>(a);
        if (nb) vb = mail_read<CLUSTER>(b);
        if (na) {
            na = !mail_is(va, tag);
            xa = mail_value(va);
        }
        if (nb) {
            nb = !mail_is(vb, tag);
            xb = mail_value(vb);
        }
        if (!__any_sync(0xffffffffu, na || nb)) return true;
        if ((polls & 63) == 0) {
            bool late = ld_volatile_int(&ctl->abort) != 0;
            const long long t = globaltimer_ns();
            if (t0 == 0) t0 = t;
            if (t - t0 > timeout_ns) {
                atomicExch(&ctl->status, CNV_TIMEOUT);
                atomicExch(&ctl->abort, 1);
                late = true;
            }
            if (__any_sync(0xffffffffu, late)) return false;
        }
    }
}

// The new value of a cell. INT: the multiplications by constants on the integer pipes, as point_value does; else on the FP64
// pipe, which takes longer where its time is what limits but has the shorter latency. oldw: (1 - beta) old formed ahead on the
// FP64 pipe, not used by the general form with INT (us per sweep with and without it: general 500^2 7.05 / 6.70, folded 512^2
// 4.36 / 4.56). The same bits.
template <Arith A, int KIND, bool FOLD, bool INT>
__device__ __forceinline__ double cell_value(const PoissonParams& p, double up, double dn, double rt, double lt, double g,
                                             double old, double oldw) {
    if (A != Arith::kExact) return point_value<A, KIND, FOLD>(p, up, dn, rt, lt, g, old);
    const double s1 = __dadd_rn(up, dn), s2 = __dadd_rn(rt, lt);
    if (FOLD) {
        const double S = __dadd_rn(s1, s2), t = __dsub_rn(S, g);
        if (!all_big_or_zero(s1, s2, S, t)) return point_value<A, KIND, FOLD>(p, up, dn, rt, lt, g, old);
        return KIND == CNV_POISSON_SOR ? __dadd_rn(INT ? mul_rn_k(p.kb4, t) : __dmul_rn(p.b4, t), oldw) : __dmul_rn(0.25, t);
    }
    const double num = INT ? __dsub_rn(__dadd_rn(mul_rn(p.dy2, s1), mul_rn(p.dx2, s2)), g)
                           : __dsub_rn(__dadd_rn(__dmul_rn(p.dy2, s1), __dmul_rn(p.dx2, s2)), g);
    const double bn = KIND != CNV_POISSON_SOR ? num : INT ? mul_rn(p.beta, num) : __dmul_rn(p.beta, num);
    const double q = p.den_pow2 ? __dmul_rn(bn, p.rden) : div_rn_const(bn, p.dden);
    return KIND == CNV_POISSON_SOR ? __dadd_rn(q, INT ? mul_rn(p.omb, old) : oldw) : q;
}

struct CellsShared {
    volatile unsigned long long gate;  // sweeps whose norm is known; above them the sweep that met the tolerance or whose
                                       // norm was not finite (kNone: none yet)
    volatile int done;                 // sweeps whose iterate is in the ring
    volatile int end;                  // the compute warps have left their loop
    volatile int fail;                 // a wait was given up
    volatile int bad[4];               // the same, by a compute thread in sweep k (k % 4)
    int nonfinite;
    double e;                          // the last norm known
    ulonglong2 seen[kNormRing][kParts][2];  // the words as read a turn before
    unsigned char side[kNormRing];          // the side sum was used
};
constexpr unsigned kNone = 0xffffffffu;

__device__ __forceinline__ int gate_checked(unsigned long long g) { return (int)(unsigned)g; }
__device__ __forceinline__ unsigned gate_conv(unsigned long long g) { return (unsigned)(g >> 32); }

// norm_add for the usual pair, without a branch: the same sign and exponent, 2^-28 <= |x| < 2^46, or nothing between them. False
// (nothing added) for the others.
__device__ __forceinline__ bool norm_add_common(NormAcc& acc, double nw, double old) {
    const unsigned long long a = (unsigned long long)__double_as_longlong(nw), b = (unsigned long long)__double_as_longlong(old);
    const int e = (int)((a >> 52) & 0x7ff);
    const bool ok = e < 1069 && (a == b || (((a ^ b) >> 52) == 0 && e >= 995));
    const long long sd = (long long)(a - b);
    const unsigned long long d = ok ? (unsigned long long)(sd < 0 ? -sd : sd) : 0ull;
    const int s = (e - 995) & 127, w = s >> 5, r = s & 31;  // (any shift will do for d = 0)
    const unsigned d0 = (unsigned)d, d1 = (unsigned)(d >> 32);
    const unsigned x0 = d0 << r, x1 = __funnelshift_l(d0, d1, r), x2 = __funnelshift_l(d1, 0u, r);
    acc.c[0] += w == 0 ? x0 : 0u;
    acc.c[1] += w == 0 ? x1 : (w == 1 ? x0 : 0u);
    acc.c[2] += w == 0 ? x2 : (w == 1 ? x1 : (w == 2 ? x0 : 0u));
    acc.c[3] += w == 1 ? x2 : (w == 2 ? x1 : 0u);
    return ok;
}

// Norm warps: this block's shares of e_1, e_2, ..., from the ring, each warp's every nw-th.
__device__ void add_norms(const CellsDev& L, CellsShared& sh, const double* hist, int warp) {
    const int lane = threadIdx.x & 31, row = L.tc + 1;
    for (int k = 1 + warp; k <= L.p.itmax; k += L.nw) {
        for (;;) {
            if (__all_sync(0xffffffffu, sh.done >= k)) break;
            const bool over = sh.fail || gate_conv(sh.gate) != kNone || (sh.end && sh.done < k);
            if (__any_sync(0xffffffffu, over)) return;
            __nanosleep(40);
        }
        __threadfence_block();
        const double* now = hist + (size_t)(k % kHist) * 2 * row;
        const double* old = hist + (size_t)((k - 1) % kHist) * 2 * row;
        NormAcc acc{{0, 0, 0, 0}};
        double side = 0.0;
        bool used = false;
        for (int x0 = 0; x0 < 2 * row; x0 += 128) {  // the same trips for every lane
            double a[4], b[4];
            unsigned rare = 0;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int x = x0 + 32 * r + lane;
                a[r] = x < 2 * row ? now[x] : 0.0;
                b[r] = x < 2 * row ? old[x] : 0.0;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (!norm_add_common(acc, a[r], b[r])) rare |= 1u << r;
            if (rare) {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if ((rare >> r & 1) && !norm_add(acc, a[r], b[r])) {
                        side += fabs(__dsub_rn(a[r], b[r]));
                        used = true;
                    }
            }
        }
        __syncwarp();
        const int slot = k % kNormRing;
        unsigned long long v = 0;
#pragma unroll
        for (int w = 0; w < 4; ++w) {  // a lane's sum is below 2^38
            const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)acc.c[w] & 0x7ffffu);
            const unsigned hi = __reduce_add_sync(0xffffffffu, (unsigned)(acc.c[w] >> 19));
            if (lane == w) v = ((unsigned long long)hi << 19) + lo;
        }
        if (__any_sync(0xffffffffu, used)) {  // values of 2^46 or more, infinities, NaN
            if (used) atomicAdd(&L.sync->fsum[slot], side);
            __threadfence();
            __syncwarp();
            if (lane == 3) v += 1ull << kSideBit;
        }
        if (lane < 4) atomicAdd(&L.sync->word[slot][blockIdx.x % kParts][lane], v + (1ull << kCountBit));
    }
}

// Verdict warp: the words of two sweeps at once (sixteen lanes a sweep, two words a lane), the complete ones judged in order. A
// block adds its share of e_{j + kNormRing} after it knew e_{j + kNormRing - kLag}, to which every block added after it knew
// e_{j + kNormRing - 2 kLag}, so after it read the slot of e_j. The side sums are cleared where they were used: block 0 clears the
// slot of e_{j - kLag} before it posts e_j (every block added to e_j after it knew e_{j - kLag}).
template <int LAG>
__device__ void check_norms(const CellsDev& L, CellsShared& sh) {
    static_assert(kNormRing >= 3 * LAG, "ring too short");
    const int lane = threadIdx.x & 31, q = lane >> 4, part = (lane >> 1) & 7, h = lane & 1;
    const unsigned blocks = (gridDim.x - part + kParts - 1) / kParts;
    long long t0 = 0;
    int polls = 0;
    for (int j = 1; j <= L.p.itmax;) {
        const int slot = (j + q) % kNormRing;
        ulonglong2 now;
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(now.x), "=l"(now.y)
                     : "l"(&L.sync->word[slot][part][2 * h])
                     : "memory");
        const ulonglong2 was = sh.seen[slot][part][h];
        const unsigned long long gx = now.x - was.x, gy = now.y - was.y;
        const bool whole = (unsigned)(gx >> kCountBit) == blocks && (unsigned)(gy >> kCountBit) == blocks;
        const unsigned lack = ~__ballot_sync(0xffffffffu, whole);
        const int ready = min((lack & 0xffffu) ? 0 : lack ? 1 : 2, L.p.itmax - j + 1);
        if (ready == 0) {
            if ((++polls & 63) == 0) {
                // (block 0 aborts a solve that did not converge when it knows the last norm: then every word is whole)
                bool late = sh.fail || (ld_volatile_int(&L.ctrl->abort) && polls >= 128);
                const long long t = globaltimer_ns();
                if (t0 == 0) t0 = t;
                if (t - t0 > L.p.timeout_ns) {
                    atomicExch(&L.ctrl->status, CNV_TIMEOUT);
                    atomicExch(&L.ctrl->abort, 1);
                    late = true;
                }
                if (__any_sync(0xffffffffu, late)) {
                    if (lane == 0) sh.fail = 1;
                    return;
                }
            }
            continue;
        }
        polls = 0;
        t0 = 0;
        if (q < ready) sh.seen[slot][part][h] = now;
        const unsigned long long low = (1ull << kCountBit) - 1, low3 = (1ull << kSideBit) - 1;
        const bool side = h && (gy & low) > low3;
        const bool any = (__ballot_sync(0xffffffffu, side) >> (16 * q)) & 0xffffu;
        unsigned long long x = gx & low, y = gy & (h ? low3 : low);
#pragma unroll
        for (int off = 2; off < 16; off <<= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, off);
            y += __shfl_xor_sync(0xffffffffu, y, off);
        }
        const unsigned long long x2 = __shfl_xor_sync(0xffffffffu, x, 1), y2 = __shfl_xor_sync(0xffffffffu, y, 1);
        const unsigned long long c[4] = {h ? x2 : x, h ? y2 : y, h ? x : x2, h ? y : y2};
        double e = norm_total(c);
        if (any && q < ready) {
            __threadfence();
            e = __dadd_rn(e, __ldcg(&L.sync->fsum[slot]));
        }
        const bool bad = !isfinite(e);
        const unsigned stops = __ballot_sync(0xffffffffu, q < ready && (bad || e < L.p.tol));
        const int first = (stops & 0xffffu) ? 0 : stops ? 1 : -1, last = first >= 0 ? first : ready - 1;
        if ((lane & 15) == 0 && q <= last) {
            sh.side[slot] = any;
            const int old = (j + q + kNormRing - LAG) % kNormRing;
            if (blockIdx.x == 0 && j + q > LAG && sh.side[old]) {
                L.sync->fsum[old] = 0.0;
                __threadfence();
            }
        }
        __syncwarp();
        if (lane == last * 16) {
            sh.e = e;
            if (bad) sh.nonfinite = 1;
            __threadfence_block();
            const unsigned j1 = (unsigned)(j + last);
            sh.gate = (unsigned long long)(first >= 0 ? j1 : kNone) << 32 | j1;
        }
        __syncwarp();
        if (first >= 0) return;
        j += ready;
    }
}

// Nothing known yet (all threads; a block barrier follows).
__device__ __forceinline__ void cells_clear(CellsShared& sh) {
    for (int x = threadIdx.x; x < kNormRing * kParts * 2; x += blockDim.x) (&sh.seen[0][0][0])[x] = make_ulonglong2(0, 0);
    for (int x = threadIdx.x; x < kNormRing; x += blockDim.x) sh.side[x] = 0;
    if (threadIdx.x == 0) {
        sh.gate = (unsigned long long)kNone << 32;
        sh.done = sh.end = sh.fail = 0;
        for (int r = 0; r < 4; ++r) sh.bad[r] = 0;
        sh.nonfinite = 0;
        sh.e = 0.0;
    }
}

// The solve's result into the control block (one thread).
__device__ __forceinline__ void cells_report(const PoissonParams& p, Ctrl* ctl, const CellsShared& sh) {
    const int met = (int)gate_conv(sh.gate);  // (-1: none)
    const bool conv = met >= 0 && !sh.nonfinite;
    const int status = sh.nonfinite ? CNV_NONFINITE : conv ? CNV_OK : CNV_NOT_CONVERGED;
    const int iters = conv ? met - 1 : p.itmax;
    ctl->iters = iters;
    ctl->err = sh.e;
    ctl->status = status;
    ctl->sweeps += conv ? met : p.itmax;
    const int step = ctl->step;
    if (step < ctl->max_records) {
        StepRecord& r = ctl->records[step];
        r.iters = iters;
        r.status = status;
        r.err = sh.e;
        r.cont_max = 0.0;
        r.cont_min = 0.0;
    }
    __threadfence();
    if (status != CNV_OK) ctl->abort = 1;
}

template <Arith A, int KIND, bool FOLD, bool INT, bool CLUSTER, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_poisson_cells(CellsDev L) {
    extern __shared__ __align__(16) double hist[];  // [kHist][2][tc + 1]; then the mailboxes (CLUSTER)
    __shared__ CellsShared sh;
    Ctrl* ctl = L.ctrl;
    if (ctl->abort) return;  // stable for the whole launch: every block returns, or none
    const PoissonParams& p = L.p;
    const int tid = threadIdx.x, me = blockIdx.x, tc = L.tc, row = tc + 1;
    const CellTile t = cell_tile(p.n, L.gx, L.gy, me);
    ulonglong2* mail = CLUSTER ? reinterpret_cast<ulonglong2*>(hist + 2 * kHist * row) : L.mail + (size_t)me * 4 * L.side;
    // psi = 0 before the first sweep, and in the place that stands for the walls
    for (int x = tid; x < 2 * kHist * row; x += blockDim.x) hist[x] = 0.0;
    if (CLUSTER)
        for (int x = tid; x < 4 * L.side; x += blockDim.x) mail[x] = make_ulonglong2(0, 0);
    cells_clear(sh);
    __syncthreads();
    if (CLUSTER) cooperative_groups::this_cluster().sync();
    if (me == p.stall_block) {  // tests only: a block that does nothing but stay until the others have given up
        if (CLUSTER) cooperative_groups::this_cluster().sync();
        return;
    }

    const int warp = tid >> 5, first_norm = tc >> 5;
    if (warp >= first_norm) {
        if (warp < first_norm + L.nw) add_norms(L, sh, hist, warp - first_norm);
        else check_norms<kLag>(L, sh);
    } else {
        int ci[2], cj[2];
        bool on[2];
        Links ln[2];
        double g[2] = {0.0, 0.0}, own[2] = {0.0, 0.0};
        ulonglong2* to[2][2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            on[c] = cell_of(t, c, tid, ci[c], cj[c]);
            ln[c].dir[0] = ln[c].dir[1] = -1;
            if (!on[c]) {
                // no cell: the warp's lanes stay together, this one on numbers of ordinary size that nobody reads
                g[c] = 1.0;
                for (int d = 0; d < 4; ++d) ln[c].nb[d] = tc;
                ln[c].from[0] = ln[c].from[1] = 0;
                to[c][0] = to[c][1] = nullptr;
                continue;
            }
            link_cell(t, L, me, ci[c], cj[c], ln[c]);
            g[c] = __ldg(L.rhs[c] + (size_t)ci[c] * p.pitch + (cj[c] >> 1));
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (ln[c].dir[r] >= 0)
                    to[c][r] = CLUSTER ? cooperative_groups::this_cluster().map_shared_rank(mail, ln[c].block[r]) + ln[c].to[r]
                                       : L.mail + (size_t)ln[c].block[r] * 4 * L.side + ln[c].to[r];
        }
        const bool edge_warp = __any_sync(0xffffffffu, ln[0].dir[0] >= 0 || ln[1].dir[0] >= 0);
        bool bad = false;
        int k = 1;
        for (; k <= p.itmax; ++k) {
            if (k > 1 && sh.bad[(k - 1) & 3]) {  // (set before the barrier that ended that sweep, next written after two more)
                bad = true;
                break;
            }
            if (k > kLag) {
                unsigned long long gate;
                for (;;) {  // by warp: the mailbox waits below need all lanes of one mind
                    gate = sh.gate;
                    if (__all_sync(0xffffffffu, gate_checked(gate) >= k - kLag)) break;
                    if (__any_sync(0xffffffffu, sh.fail)) {
                        bad = true;
                        break;
                    }
                }
                if (!bad && gate_conv(gate) <= (unsigned)(k - kLag)) break;  // the same sweep in every thread of every block
            }
            double* now = hist + (k % kHist) * 2 * row;
            const double* before = hist + ((k - 1) % kHist) * 2 * row;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double* o = c == 0 ? before + row : now;  // red reads black of the sweep before, black red of this one
                const double oldw = A != Arith::kExact || KIND != CNV_POISSON_SOR || (INT && !FOLD) ? 0.0 : __dmul_rn(p.omb, own[c]);
                double v[4];
#pragma unroll
                for (int d = 0; d < 4; ++d) v[d] = o[ln[c].nb[d]];
                if (edge_warp && (c || k > 1) && !bad) {
                    double xa = 0.0, xb = 0.0;
                    if (!mail_wait<CLUSTER>(mail + ln[c].from[0], mail + ln[c].from[1], ln[c].dir[0] >= 0, ln[c].dir[1] >= 0,
                                            (unsigned)(c ? k : k - 1), ctl, p.timeout_ns, xa, xb))
                        bad = true;
#pragma unroll
                    for (int d = 0; d < 4; ++d) v[d] = ln[c].dir[0] == d ? xa : ln[c].dir[1] == d ? xb : v[d];
                }
                const double nw = cell_value<A, KIND, FOLD, INT>(p, v[0], v[1], v[2], v[3], g[c], own[c], oldw);
                own[c] = nw;
                if (edge_warp) {
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        if (ln[c].dir[r] >= 0) mail_write<CLUSTER>(to[c][r], nw, (unsigned)k);
                }
                if (on[c]) now[c * row + tid] = nw;
                if (c == 1 && bad) sh.bad[k & 3] = 1;
                cells_barrier(tc);
            }
            if (tid == tc - 1) {
                __threadfence_block();
                sh.done = k;
            }
        }
        if (k > p.itmax && p.itmax > 0 && sh.bad[p.itmax & 3]) bad = true;
        if (k > p.itmax && !bad) {
            // out of sweeps: the norms of the last ones
            for (;;) {
                const unsigned long long gate = sh.gate;
                if (gate_checked(gate) >= p.itmax || gate_conv(gate) != kNone || sh.fail) break;
            }
        }
        if (bad) sh.fail = 1;
        sh.end = 1;
        cells_barrier(tc);
        if (!sh.fail) {
            __threadfence_block();
            const int last = gate_conv(sh.gate) != kNone ? (int)gate_conv(sh.gate) : p.itmax;
            const double* ans = hist + (last % kHist) * 2 * row;
#pragma unroll
            for (int c = 0; c < 2; ++c)
                if (on[c]) L.out[c][(size_t)ci[c] * p.pitch + (cj[c] >> 1)] = ans[c * row + tid];
        }
    }
    __syncthreads();
    if (CLUSTER) cooperative_groups::this_cluster().sync();  // no block leaves while another may write to its mailboxes
    if (sh.fail) return;
    if (me == 0 && tid == 0) cells_report(p, ctl, sh);
}

// Tiles of many cells: the same solve with the tile's iterates in shared memory and a column of the tile's cells per thread, for grids
// too large for a cell of each colour per thread.
//
// Planes: a colour's cells of a tile row lie together (cell (il, jl) at il pw + jl / 2), so that the neighbours are at +-pw and
// in two adjacent places. kRowsHist iterates are kept: one is written while the last may still turn out to have converged
// two sweeps back (kRowsLag). The ring of edge cells goes one to a thread, first in each half-sweep (mailboxes as above: a
// value sent then is asked for half a sweep later); the inner cells follow in columns, a thread every R-th row (R even: the
// colours' places in a row stay the same), counted from the last thread, so that the threads left over have edge cells. With the
// edge on warps of its own fewer updated the rest: 1024^2 16.2 us a sweep against 15.0. The right-hand side streams through L1. The norm is added up by the
// updating threads, by warp through shared memory, and handed on by a norm warp.
// Bound by the FP64 pipe: 1024^2, folded: 5 additions of 19 cycles for 216 warps of cells, 10.7 us a sweep. us per sweep, exchange kernel ->
// here: FMA 531^2 7.54 -> 4.99, 700^2 10.2 -> 7.5, 1024^2 15.7 -> 14.1; general SOR 531^2 10.6 -> 8.6, 700^2 15.7 -> 12.5, 1000^2 25.0 ->
// 24.0; folded 1024^2 15.4 -> 15.0. Two cells of a thread at once, their multiplications without branches, ran slower (1024^2 18.3):
// integer pipe 52 % and FP64 pipe 61 % busy, in turns.
constexpr int kRowsHist = 3, kRowsLag = 2;
constexpr int kRowsThreads[2] = {768, 960};  // compute threads at most: with 72 registers each, or with 64

struct RowsShared {
    unsigned long long part[4][kRowsThreads[1] / 32][4];
    volatile int side[4];
};

// Norm warp: the warps' shares of e_k, added up and handed to the global ring.
__device__ void add_row_norms(const CellsDev& L, CellsShared& sh, RowsShared& rs) {
    const int lane = threadIdx.x & 31, warps = L.tc / 32;
    for (int k = 1; k <= L.p.itmax; ++k) {
        for (;;) {
            if (__all_sync(0xffffffffu, sh.done >= k)) break;
            const bool over = sh.fail || gate_conv(sh.gate) != kNone || (sh.end && sh.done < k);
            if (__any_sync(0xffffffffu, over)) return;
            __nanosleep(100);
        }
        __threadfence_block();
        unsigned long long c[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            c[w] = lane < warps ? rs.part[k & 3][lane][w] : 0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) c[w] += __shfl_xor_sync(0xffffffffu, c[w], off);
        }
        unsigned long long v = lane == 0 ? c[0] : lane == 1 ? c[1] : lane == 2 ? c[2] : c[3];
        const bool side = __all_sync(0xffffffffu, rs.side[k & 3] != 0);
        if (side) {
            __threadfence();
            __syncwarp();
            if (lane == 0) rs.side[k & 3] = 0;
            if (lane == 3) v += 1ull << kSideBit;
        }
        if (lane < 4) atomicAdd(&L.sync->word[k % kNormRing][blockIdx.x % kParts][lane], v + (1ull << kCountBit));
    }
}

__device__ __forceinline__ void add_change(NormAcc& acc, double& side, bool& used, double nw, double old) {
    if (!norm_add_common(acc, nw, old) && !norm_add(acc, nw, old)) {
        side += fabs(__dsub_rn(nw, old));
        used = true;
    }
}

template <Arith A, int KIND, bool FOLD, int MAXT>
__global__ void __launch_bounds__(MAXT + 64, 1) k_poisson_rows(CellsDev L) {
    extern __shared__ __align__(16) double hist[];  // [kRowsHist][2][plane]
    __shared__ CellsShared sh;
    __shared__ RowsShared rs;
    Ctrl* ctl = L.ctrl;
    if (ctl->abort) return;  // stable for the whole launch: every block returns, or none
    const PoissonParams& p = L.p;
    const int tid = threadIdx.x, me = blockIdx.x, tc = L.tc, lane = tid & 31, warp = tid >> 5;
    const CellTile t = cell_tile(p.n, L.gx, L.gy, me);
    const int W = t.c1 - t.c0, H = t.r1 - t.r0, pw = (W + 1) / 2, plane = L.plane, nothing = plane - 1;
    ulonglong2* mail = L.mail + (size_t)me * 4 * L.side;
    for (int x = tid; x < 2 * kRowsHist * plane; x += blockDim.x) hist[x] = 0.0;  // psi = 0 and the walls' place
    cells_clear(sh);
    if (tid < 4) rs.side[tid] = 0;
    __syncthreads();
    if (me == p.stall_block) return;  // tests only: a block that does nothing

    if (warp == tc / 32) {
        add_row_norms(L, sh, rs);
    } else if (warp > tc / 32) {
        check_norms<kRowsLag>(L, sh);
    } else {
        // the edge cells: one of each colour for the first threads
        const int ne = edge_cells(W, H);
        const bool edge_warp = warp * 32 < ne;
        int eat[2], enb[2][4], efrom[2][2], edir[2][2], eto[2][2];  // eto: place among all blocks' mailboxes
        double eg[2] = {1.0, 1.0}, eold[2] = {0.0, 0.0};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            eat[c] = nothing;
            edir[c][0] = edir[c][1] = -1;
            efrom[c][0] = efrom[c][1] = eto[c][0] = eto[c][1] = 0;
            for (int d = 0; d < 4; ++d) enb[c][d] = nothing;
            int i, j;
            if (tid < ne && cell_of(t, c, tid, i, j)) {
                Links ln;
                link_cell(t, L, me, i, j, ln);
                eat[c] = (i - t.r0) * pw + ((j - t.c0) >> 1);
                eg[c] = __ldg(L.rhs[c] + (size_t)i * p.pitch + (j >> 1));
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const int y = i + (d == 0) - (d == 1) - t.r0, x = j + (d == 2) - (d == 3) - t.c0;
                    if (y >= 0 && y < H && x >= 0 && x < W) enb[c][d] = y * pw + (x >> 1);
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    edir[c][r] = ln.dir[r];
                    if (ln.dir[r] < 0) continue;
                    efrom[c][r] = ln.from[r];
                    eto[c][r] = ln.block[r] * 4 * L.side + ln.to[r];
                }
            }
        }
        // the inner cells: place q of rows 1 + u, 1 + u + R, ... (counted from the last thread: the first have the edge)
        const int nq = (W - 1) / 2, x = tc - 1 - tid, u = x / max(nq, 1), q = x - u * nq, R = L.rows;
        const int il0 = 1 + u, step = R * pw;
        const bool inner = nq > 0 && u < R;
        const int pa = (t.r0 + il0 + t.c0 + 1) & 1;  // colour 0's cell is at jl = 1 + 2 q + pa, colour 1's at 1 + 2 q + 1 - pa
        const bool fits0 = 1 + 2 * q + pa <= W - 2, fits1 = 2 + 2 * q - pa <= W - 2;
        const size_t gstep = (size_t)R * p.pitch;
        const double* gin[2] = {L.rhs[0] + (size_t)(t.r0 + il0) * p.pitch + ((t.c0 + 1 + 2 * q + pa) >> 1),
                                L.rhs[1] + (size_t)(t.r0 + il0) * p.pitch + ((t.c0 + 2 + 2 * q - pa) >> 1)};
        const int base = il0 * pw + q;

        bool bad = false;
        int k = 1;
        for (; k <= p.itmax; ++k) {
            if (k > 1 && sh.bad[(k - 1) & 3]) {
                bad = true;
                break;
            }
            if (k > kRowsLag) {
                unsigned long long gate;
                for (;;) {
                    gate = sh.gate;
                    if (__all_sync(0xffffffffu, gate_checked(gate) >= k - kRowsLag)) break;
                    if (__any_sync(0xffffffffu, sh.fail)) {
                        bad = true;
                        break;
                    }
                }
                if (!bad && gate_conv(gate) <= (unsigned)(k - kRowsLag)) break;
            }
            double* now = hist + (size_t)(k % kRowsHist) * 2 * plane;
            const double* before = hist + (size_t)((k - 1) % kRowsHist) * 2 * plane;
            NormAcc acc{{0, 0, 0, 0}};
            double side = 0.0;
            bool used = false;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double* o = c == 0 ? before + plane : now;
                double* to = now + c * plane;
                const double* old = before + c * plane;
                if (edge_warp) {
                    double v[4];
#pragma unroll
                    for (int d = 0; d < 4; ++d) v[d] = o[enb[c][d]];
                    if ((c || k > 1) && !bad) {
                        double xa = 0.0, xb = 0.0;
                        if (!mail_wait<false>(mail + efrom[c][0], mail + efrom[c][1], edir[c][0] >= 0, edir[c][1] >= 0,
                                              (unsigned)(c ? k : k - 1), ctl, p.timeout_ns, xa, xb))
                            bad = true;
#pragma unroll
                        for (int d = 0; d < 4; ++d) v[d] = edir[c][0] == d ? xa : edir[c][1] == d ? xb : v[d];
                    }
                    const double nw = point_value<A, KIND, FOLD>(p, v[0], v[1], v[2], v[3], eg[c], eold[c]);
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        if (edir[c][r] >= 0) mail_write<false>(L.mail + eto[c][r], nw, (unsigned)k);
                    if (eat[c] != nothing) {
                        to[eat[c]] = nw;
                        add_change(acc, side, used, nw, eold[c]);
                    }
                    eold[c] = nw;
                }
                if (inner && (c == 0 ? fits0 : fits1)) {
                    const int off = c == 0 ? pa : 1 - pa;
                    const double* g = gin[c];
                    int at = base;
                    for (int il = il0; il <= H - 2; il += R, at += step, g += gstep) {
                        const double was = old[at + off];
                        const double nw = point_value<A, KIND, FOLD>(p, o[at + off + pw], o[at + off - pw], o[at + 1], o[at],
                                                                     __ldg(g), was);
                        to[at + off] = nw;
                        add_change(acc, side, used, nw, was);
                    }
                }
                __syncwarp();
                if (c == 1) {
#pragma unroll
                    for (int w = 0; w < 4; ++w) {  // a lane's sum is below 2^38
                        const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)acc.c[w] & 0x7ffffu);
                        const unsigned hi = __reduce_add_sync(0xffffffffu, (unsigned)(acc.c[w] >> 19));
                        if (lane == w) rs.part[k & 3][warp][w] = ((unsigned long long)hi << 19) + lo;
                    }
                    if (used) {  // values of 2^46 or more, infinities, NaN
                        atomicAdd(&L.sync->fsum[k % kNormRing], side);
                        __threadfence();
                        rs.side[k & 3] = 1;
                    }
                    if (bad) sh.bad[k & 3] = 1;
                }
                cells_barrier(tc);
            }
            if (tid == tc - 1) {
                __threadfence_block();
                sh.done = k;
            }
        }
        if (k > p.itmax && p.itmax > 0 && sh.bad[p.itmax & 3]) bad = true;
        if (k > p.itmax && !bad) {
            for (;;) {
                const unsigned long long gate = sh.gate;
                if (gate_checked(gate) >= p.itmax || gate_conv(gate) != kNone || sh.fail) break;
            }
        }
        if (bad) sh.fail = 1;
        sh.end = 1;
        cells_barrier(tc);
        if (!sh.fail) {
            __threadfence_block();
            const int last = gate_conv(sh.gate) != kNone ? (int)gate_conv(sh.gate) : p.itmax;
            const double* ans = hist + (size_t)(last % kRowsHist) * 2 * plane;
            for (int y = tid; y < W * H; y += tc) {
                const int il = y / W, jl = y - il * W, i = t.r0 + il, j = t.c0 + jl, c = (i + j) & 1;
                L.out[c][(size_t)i * p.pitch + (j >> 1)] = ans[c * plane + il * pw + (jl >> 1)];
            }
        }
    }
    __syncthreads();
    if (sh.fail) return;
    if (me == 0 && tid == 0) cells_report(p, ctl, sh);
}

constexpr int kRowsMax = 1100;               // (1150^2, us per sweep: general SOR 31.9, the exchange kernel 31.2)
constexpr int kClusterSide = 4;              // the cluster's tiles: 4 x 4
constexpr size_t kCellsSmem = 128 * 1024;    // dynamic shared memory that the kernels with a cell per thread may ask for
constexpr size_t kCellsStatic = 14 * 1024;   // static shared memory, at most
static_assert(sizeof(CellsShared) + sizeof(RowsShared) <= kCellsStatic, "shared memory");

template <bool INT, bool CLUSTER, int MAXT>
const void* cells_kernel(Arith a, int kind, bool fold) {
    const bool sor = kind == CNV_POISSON_SOR;
    if (a == Arith::kFma)
        return sor ? (const void*)&k_poisson_cells<Arith::kFma, CNV_POISSON_SOR, false, INT, CLUSTER, MAXT>
                   : (const void*)&k_poisson_cells<Arith::kFma, CNV_POISSON_GS, false, INT, CLUSTER, MAXT>;
    if (fold)
        return sor ? (const void*)&k_poisson_cells<Arith::kExact, CNV_POISSON_SOR, true, INT, CLUSTER, MAXT>
                   : (const void*)&k_poisson_cells<Arith::kExact, CNV_POISSON_GS, true, INT, CLUSTER, MAXT>;
    return sor ? (const void*)&k_poisson_cells<Arith::kExact, CNV_POISSON_SOR, false, INT, CLUSTER, MAXT>
               : (const void*)&k_poisson_cells<Arith::kExact, CNV_POISSON_GS, false, INT, CLUSTER, MAXT>;
}

template <int MAXT>
const void* rows_kernel(Arith a, int kind, bool fold) {
    const bool sor = kind == CNV_POISSON_SOR;
    if (a == Arith::kFma)
        return sor ? (const void*)&k_poisson_rows<Arith::kFma, CNV_POISSON_SOR, false, MAXT>
                   : (const void*)&k_poisson_rows<Arith::kFma, CNV_POISSON_GS, false, MAXT>;
    if (fold)
        return sor ? (const void*)&k_poisson_rows<Arith::kExact, CNV_POISSON_SOR, true, MAXT>
                   : (const void*)&k_poisson_rows<Arith::kExact, CNV_POISSON_GS, true, MAXT>;
    return sor ? (const void*)&k_poisson_rows<Arith::kExact, CNV_POISSON_SOR, false, MAXT>
               : (const void*)&k_poisson_rows<Arith::kExact, CNV_POISSON_GS, false, MAXT>;
}

const void* cells_kernel(const CellsPlan& P, Arith a, int kind, bool fold) {
    if (P.rows) return P.threads <= kRowsThreads[0] + 64 ? rows_kernel<kRowsThreads[0]>(a, kind, fold) : rows_kernel<kRowsThreads[1]>(a, kind, fold);
    // constants multiplied on the integer pipes from about 400^2 (general SOR, us per sweep: 300^2 3.93 against 3.26 on the FP64
    // pipe, 384^2 4.85 / 4.82, 400^2 5.01 / 5.27, 500^2 6.72 / 7.54)
    if (P.cluster) return cells_kernel<false, true, 640>(a, kind, fold);
    return P.threads <= 640 ? cells_kernel<false, false, 640>(a, kind, fold) : cells_kernel<true, false, 1024>(a, kind, fold);
}

size_t cells_smem(const CellsPlan& P) {
    if (P.rows) return sizeof(double) * 2 * kRowsHist * P.plane;
    return sizeof(double) * 2 * kHist * (P.tc + 1) + (P.cluster ? sizeof(ulonglong2) * 4 * P.side : 0);
}

cudaLaunchConfig_t cells_config(const CellsPlan& P, cudaLaunchAttribute* attr, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P.gx * P.gy);
    cfg.blockDim = dim3(P.threads);
    cfg.dynamicSmemBytes = cells_smem(P);
    cfg.stream = s;
    if (P.cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = P.gx * P.gy;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Tiles, threads and mailbox length of a gx x gy cut; false where a tile is a single row or column.
bool cells_cut(int n, int gx, int gy, int min_norm_warps, CellsPlan* P) {
    P->gx = gx;
    P->gy = gy;
    const int ni = n - 2, W = (ni + gx - 1) / gx, H = (ni + gy - 1) / gy;  // of the largest tile
    P->cluster = P->rows = P->plane = 0;
    if (ni / gx < 2 || ni / gy < 2) return false;
    P->side = std::max(W, H);
    P->tc = colour_threads(W, H);
    P->tc = (P->tc + 31) / 32 * 32;
    P->norm_warps = std::max(min_norm_warps, std::min(kMaxNormWarps, 31 - P->tc / 32));
    P->threads = P->tc + 32 * (P->norm_warps + 1);  // and the verdict's warp
    return true;
}

}  // namespace

// The cut for an n x n grid on `sms` SMs (tc 0: the kernel does not take it), its kernel made ready to launch.
CellsPlan cells_plan(int n, int sms, size_t smem_max, Arith a, int kind, bool fold) {
    const CellsPlan none{};
    CellsPlan best{}, q{};
    if (kind != CNV_POISSON_SOR && kind != CNV_POISSON_GS) return none;
    const int cap = std::min(sms, kMaxSolverBlocks), min_norm = a == Arith::kFma ? kMinNormWarpsFma : kMinNormWarps;
    // One cluster up to 90^2 (the exact arithmetic) or 112^2 (FMA, with fewer FP64 operations a cell): its 16 SMs' FP64 pipes
    // take as long there as the hops between all SMs (general SOR: 64^2 1.76 us a sweep against 2.61, 97^2 2.91 against 2.65;
    // FMA: 112^2 1.90 against 1.98).
    if (n <= (a == Arith::kFma ? 112 : 90)) {
        const int g = std::min(kClusterSide, (n - 2) / 2);
        if (g < 1 || !cells_cut(n, g, g, min_norm, &best)) return none;
        best.cluster = 1;
        if (best.threads > 640) return none;
    } else {
        for (int gx = 1; gx <= cap; ++gx)
            for (int gy = cap / gx; gy >= 1 && gy >= cap / gx - 1; --gy)
                if (cells_cut(n, gx, gy, min_norm, &q) && q.threads <= 1024 &&
                    (best.tc == 0 || q.tc < best.tc || (q.tc == best.tc && q.side < best.side)))
                    best = q;
        if (best.tc == 0 && n <= kRowsMax) {
            // tiles of many cells: few cells a tile and a short edge
            int cells = 0;
            const int ni = n - 2;
            for (int gx = 1; gx <= cap; ++gx) {
                const int gy = cap / gx, W = (ni + gx - 1) / gx, H = (ni + gy - 1) / gy;
                if (!cells_cut(n, gx, gy, min_norm, &q) || ni / gx < 3 || ni / gy < 3) continue;
                const int cost = W * H + W + H, nq = (W - 1) / 2, ne = edge_cells(W, H);
                if (best.tc && cost >= cells) continue;
                // fewer threads with more registers unless that costs a turn of the rows; warps of their own for the edge, or inner
                // cells on them too if that saves more than a turn (us per sweep, own / shared: 700^2 13.0 / 14.5, 1024^2 16.3 /
                // 15.0; 768 / 960 threads: 700^2 13.0 / 12.5, 900^2 20.3 / 19.5, 1024^2 15.0 / 15.2)
                int turns = 0, rows = 0;
                for (int threads : kRowsThreads) {
                    if (ne > threads) continue;
                    int m1 = 0, r1 = 0, tc = 0;
                    for (int own = 1; own >= 0; --own) {
                        const int most = (threads - (own ? (ne + 31) / 32 * 32 : 0)) / nq & ~1;
                        if (most < 2) continue;
                        const int m = (H - 2 + most - 1) / most;
                        if (r1 && m + 1 >= m1) continue;
                        m1 = m;
                        r1 = ((H - 2 + m - 1) / m + 1) & ~1;
                        tc = own ? (ne + 31) / 32 * 32 + (nq * r1 + 31) / 32 * 32 : (std::max(nq * r1, ne) + 31) / 32 * 32;
                    }
                    if (r1 == 0 || (rows && m1 >= turns)) continue;
                    turns = m1;
                    rows = r1;
                    q.tc = tc;
                }
                if (rows == 0) continue;
                best = q;
                best.rows = rows;
                best.plane = (W + 1) / 2 * H + 1;
                best.norm_warps = 1;
                best.threads = best.tc + 64;
                cells = cost;
            }
        }
        if (best.tc == 0) return none;
    }
    const size_t smem = cells_smem(best), most = best.rows ? smem_max - kCellsStatic : kCellsSmem;
    if (smem > most || most + kCellsStatic > smem_max) return none;
    const void* k = cells_kernel(best, a, kind, fold);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) return none;
    if (best.cluster) {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return none;
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = cells_config(best, attr, nullptr);
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess || clusters < 1) return none;
    } else {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, best.threads, smem) != cudaSuccess || per_sm < 1) return none;
    }
    return best;
}

size_t cells_sync_bytes(const CellsPlan& P) {
    return sizeof(CellsSync) + (P.cluster ? 0 : sizeof(ulonglong2) * 4 * (size_t)P.side * P.gx * P.gy);
}

cudaError_t launch_poisson_cells(const CellsLaunch& C, cudaStream_t s) {
    const CellsPlan& P = C.plan;
    cudaError_t e = cudaMemsetAsync(C.sync, 0, cells_sync_bytes(P), s);
    if (e != cudaSuccess) return e;
    const void* k = cells_kernel(P, C.p.arith, C.p.kind, C.p.fold != 0);
    CellsDev L{};
    L.p = C.p;
    L.gx = P.gx;
    L.gy = P.gy;
    L.tc = P.tc;
    L.nw = P.norm_warps;
    L.rows = P.rows;
    L.plane = P.plane;
    L.side = P.side;
    for (int c = 0; c < 2; ++c) {
        L.rhs[c] = C.rhs[c];
        L.out[c] = C.out[c];
    }
    L.sync = static_cast<CellsSync*>(C.sync);
    L.mail = reinterpret_cast<ulonglong2*>(L.sync + 1);
    L.ctrl = C.ctrl;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cells_config(P, attr, s);
    void* args[] = {&L};
    return cudaLaunchKernelExC(&cfg, k, args);
}

}  // namespace cnv
