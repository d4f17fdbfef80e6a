// cnv_dst.cu -- exact solve of the reference's discrete Poisson equation by sine transforms.
//
// The equation that every SOR sweep of src/poisson.c:241-272 moves towards is, on the interior
// cells (i, j) = 1 .. n-2 with psi = 0 on the edges,
//
//     den psi(i,j) - dy^2 (psi(i+1,j) + psi(i-1,j)) - dx^2 (psi(i,j+1) + psi(i,j-1)) = c4 w(i,j)
//
// (den = 2 (dx^2 + dy^2), c4 = dx^2 dy^2, f = -w). Its matrix is the Kronecker sum of two
// tridiagonal Toeplitz matrices, diagonalised by the orthonormal DST-I basis
//     S[a][b] = sqrt(2 / (m+1)) sin(pi (a+1)(b+1) / (m+1)),  m = n - 2,  S = S^T = S^-1.
// The answer is what the reference's solver converges to, to rounding, at a fixed cost; the map is
// linear and symmetric, so the adjoint solve is the same call.
//
// FP64 answer from FP32 transforms. A GB300 runs FP64 at about 1/60 of its FP32 rate, and four FP64
// row transforms kept the FP64 pipe 85-91 % busy for the whole solve (0.66 ms at 1000^2, 3.0 ms at
// 2048^2). So the transforms run in FP32 and the FP64 answer comes from correcting the residual,
// which is formed exactly in integers:
//   - With dx = Lx / n, dy = Ly / n and a : b = Ly : Lx in lowest terms the equation is
//     kappa (a^2 Di + b^2 Dj) psi = scale in, where Di = 2 psi - up - down and Dj = 2 psi - left - right: a stencil
//     with integer coefficients.
//   - psi is held as 64-bit fixed point: psi = I 2^(E-1023-S) scale / kappa, with E the largest biased exponent
//     of `in` and S such that the largest |I| is about 2^58. In these units the right-hand side is in * 2^(S-E+1023),
//     an exponent shift of the double, and the residual in * 2^.. - (a^2 Di + b^2 Dj) I is a sum of 64-bit integers and
//     the right-hand side's fraction. The integers are taken modulo 2^64 (2^128 where a or b is above 512), which is exact
//     because the residual itself is small; the fraction is added to them as a float. (A unit is 2^-58 of the largest |psi|, and psi is up to 0.07 n^2 times the
//     right-hand side: without the fraction, cells of one value, all rounded alike, put psi off by 6e-14 at 1000^2, 2e-13 at 2048^2.)
//   - The first FP32 solve starts from `in`, each later one from the residual, and adds to I. A solve leaves about
//     3e-7 of the answer, the next 1e-11 .. 1e-10, the third less than the rounding of psi to FP64 for most right-hand sides
//     (against extended-precision solves, n = 200 .. 4097: noise, a point and smooth ones 6e-17 .. 1e-15, a constant and
//     a disc of one value up to 4e-15, at 4097^2; FP64 sine transforms: 5e-16 .. 1e-13). Where the estimate of the third is
//     above 1e-16 (long transforms, large radices, stretched cells) a fourth is made.
//   - I times scale / kappa is rounded once to FP64, in integer arithmetic.
// The residual is part of the next solve's first pass and the addition of the last one, so a solve is three
// launches: A rows (residual, transform along j), B columns (transform along i, divide by the eigenvalues, transform
// back, in place), C rows (transform back, add). B reads and writes whole columns, a few neighbouring ones per block, so
// no pass writes transposed. 1000^2: 0.66 -> 0.20 ms per solve; 2048^2: 3.0 -> 1.1 ms.
//
// The row transforms. The DST-I F_k = sum_j y_j sin(pi j k / N) of a row y_1 .. y_{N-1} (N = m+1) comes from one complex
// DFT of length N: with d_j = (y_j - y_{N-j}) / 2 and c_j = (y_j + y_{N-j}) / 2,
//     z_j = d_j + c_j sin(pi j / N) + i c_j cos(pi j / N),      Z_l = sum_j z_j exp(-2 pi i j l / N) = F_{2l+1} - i F_{2l},
// because the even outputs depend on the antisymmetric part d alone, the odd ones on the symmetric part c (times
// exp(-i pi j / N)), and each part's DFT is purely imaginary. (The usual half-cost form packs two rows into one DFT and gets the
// odd outputs from a prefix sum, whose FP32 rounding grows with the row: modelled, it needs a fourth solve from n = 300.)
// The DFT is a mixed-radix Stockham transform in shared memory over the factors of N, the large primes first (the first
// stage has no twiddles). Radices 2 .. 10 are done by one thread in registers. A larger prime p takes two steps: the sums and
// differences u_q +- u_{p-q} of every butterfly, then the outputs q and p-q from the (p-1)/2-long cosine and sine sums, which
// are small matrix products (outputs x sums x butterflies) in register tiles of qt outputs x bt butterflies. A block
// carries rows_a rows (cols_b columns) interleaved, so neighbouring lanes share table entries. Grids whose transform does
// not fit shared memory (N above about 9,600 for a prime N) take dense FP64 products with S instead (each folded by the
// mirror symmetry S[b][m-1-c] = (-1)^b S[b][c]); there the eigenvalues are formed as sums of squared sines, because the
// difference den - 2 dy^2 cos - 2 dx^2 cos cancels in the lowest modes.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "cnv_dst.h"
#include "cnv_sync.cuh"

namespace cnv {
namespace {

// Destination of a solve: row-major out (leading dimension n), or, when red is set, the red/black
// split layout of an n x n field (cell (i, j) at (i + j odd ? black : red)[i * pitch + j / 2]).
struct DstDest {
    double* out;
    int ld;
    double* red;
    double* black;
    int pitch;
};

// ------------------------------------------------------------------ FFT in shared memory, in FP32 or FP64 (R)
template <class R> struct Pair;
template <> struct Pair<float> { typedef float2 t; typedef double wide; };
template <> struct Pair<double> { typedef double2 t; typedef long double wide; };
template <class R> using C2 = typename Pair<R>::t;
__device__ __forceinline__ float2 c2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 c2(double x, double y) { return make_double2(x, y); }

template <class V>
__device__ __forceinline__ V cmul(V a, V b) {
    return c2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
template <class V>
__device__ __forceinline__ V cadd(V a, V b) { return c2(a.x + b.x, a.y + b.y); }
template <class V>
__device__ __forceinline__ V csub(V a, V b) { return c2(a.x - b.x, a.y - b.y); }
template <class V>
__device__ __forceinline__ V mul_mi(V a) { return c2(a.y, -a.x); }  // -i a

// e / d for e * d < 2^32, with magic = magic_of(d)
__device__ __forceinline__ int fdiv(int e, unsigned magic) { return magic ? (int)__umulhi((unsigned)e, magic) : e; }

// P = A B with A the smaller factor, for the composite radices (0: P is prime, 2, 4 or 8).
template <int P>
constexpr int kSmallFactor = P == 6 || P == 10 ? 2 : P == 9 ? 3 : 0;

// One P-point DFT in registers; cs[t * STEP] = (cos, sin)(2 pi t / P).
template <int P, int STEP = 1, class R>
__device__ __forceinline__ void dft(C2<R> (&u)[P], const C2<R>* cs) {
    if constexpr (kSmallFactor<P> > 0) {
        // A B points: B-point DFTs of the elements q mod A, twiddles, A-point DFTs
        constexpr int A = kSmallFactor<P>, B = P / A;
        C2<R> v[A][B];
#pragma unroll
        for (int a = 0; a < A; ++a) {
#pragma unroll
            for (int b = 0; b < B; ++b) v[a][b] = u[b * A + a];
            dft<B, STEP * A, R>(v[a], cs);
#pragma unroll
            for (int b = 1; b < B; ++b)
                if (a) {
                    const C2<R> w = cs[a * b * STEP];
                    v[a][b] = cmul(v[a][b], c2(w.x, -w.y));
                }
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            C2<R> x[A];
#pragma unroll
            for (int a = 0; a < A; ++a) x[a] = v[a][b];
            dft<A, STEP * B, R>(x, cs);
#pragma unroll
            for (int a = 0; a < A; ++a) u[b + B * a] = x[a];
        }
    } else if constexpr (P == 2) {
        const C2<R> a = u[0];
        u[0] = cadd(a, u[1]);
        u[1] = csub(a, u[1]);
    } else if constexpr (P == 4) {
        const C2<R> a = cadd(u[0], u[2]), b = csub(u[0], u[2]), c = cadd(u[1], u[3]), d = mul_mi(csub(u[1], u[3]));
        u[0] = cadd(a, c);
        u[1] = cadd(b, d);
        u[2] = csub(a, c);
        u[3] = csub(b, d);
    } else if constexpr (P == 8) {
        C2<R> e[4] = {u[0], u[2], u[4], u[6]}, o[4] = {u[1], u[3], u[5], u[7]};
        dft<4, STEP, R>(e, cs);
        dft<4, STEP, R>(o, cs);
        const R h = R(0.70710678118654752440);
        const C2<R> w[4] = {o[0], c2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x)), mul_mi(o[2]),
                             c2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y))};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            u[k] = cadd(e[k], w[k]);
            u[k + 4] = csub(e[k], w[k]);
        }
    } else {
        constexpr int H = (P - 1) / 2;
        C2<R> A[H], B[H], w[H];
        const C2<R> u0 = u[0];
        C2<R> s = u0;
#pragma unroll
        for (int q = 0; q < H; ++q) {
            A[q] = cadd(u[q + 1], u[P - 1 - q]);
            B[q] = csub(u[q + 1], u[P - 1 - q]);
            w[q] = cs[(q + 1) * STEP];
            s = cadd(s, A[q]);
        }
        u[0] = s;
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            C2<R> C = u0, D = c2(R(0), R(0));
#pragma unroll
            for (int q = 1; q <= H; ++q) {
                const int t = (q * k) % P;  // cos(2 pi t / P) = cos(2 pi (P - t) / P), sin changes sign
                const R c = w[(t <= H ? t : P - t) - 1].x, d = t <= H ? w[t - 1].y : -w[P - t - 1].y;
                C.x = fma(A[q - 1].x, c, C.x);
                C.y = fma(A[q - 1].y, c, C.y);
                D.x = fma(B[q - 1].x, d, D.x);
                D.y = fma(B[q - 1].y, d, D.y);
            }
            u[k] = c2(C.x + D.y, C.y - D.x);
            u[P - k] = c2(C.x - D.y, C.y + D.x);
        }
    }
}

// Where a pass finds its tables.
template <class R>
struct Tables {
    const C2<R> *tw, *sc, *cs;
    const R *li, *lj, *cm;
};

// A stage of radix P, one thread per butterfly: src -> dst.
template <int P, int RP, class R>
__device__ __forceinline__ void small_stage(const FftStage& S, const C2<R>* src, C2<R>* dst, const C2<R>* cs,
                                            const C2<R>* tw) {
    const int nb = S.nb, L = S.L, r2 = nb / L;
    for (int e = threadIdx.x; e < nb * RP; e += blockDim.x) {
        const int pr = e % RP, b = e / RP;
        const int k = fdiv(b, S.magic_L), j1 = b - k * L;
        C2<R> u[P];
#pragma unroll
        for (int q = 0; q < P; ++q) u[q] = src[(b + q * nb) * RP + pr];
        if (L > 1) {
            const int tj = j1 * r2;
#pragma unroll
            for (int q = 1; q < P; ++q) u[q] = cmul(u[q], tw[q * tj]);
        }
        dft<P, 1, R>(u, cs);
        const int ob = k * L * P + j1;
#pragma unroll
        for (int q = 0; q < P; ++q) dst[(ob + L * q) * RP + pr] = u[q];
    }
}

// The output step of a large odd radix: T holds, per butterfly b, u_0 at row 0, the sums u_q + u_{p-q} at rows 1 .. h and
// the differences at rows h+1 .. p-1 (row q of butterfly b at q * nb + b). A thread takes QT outputs of BT butterflies:
// 2 BT shared loads and, for MAT, two vector loads of the cosines and sines of its outputs (the matrix at cm: row q holds
// cos(2 pi q k / p), k = 0 .. pad-1, then the sines) for 4 QT BT multiply-adds. Without MAT (p above kMaxMatrixRadix) the
// table index q k mod p is stepped instead.
template <int N, class R>
struct alignas(N * sizeof(R) < 16 ? N * sizeof(R) : 16) Vec {
    R v[N];
};

template <int QT, int BT, int RP, bool MAT, class R>
__device__ __forceinline__ void large_outputs(const FftStage& S, const C2<R>* T, C2<R>* X, const C2<R>* cs,
                                              const R* cm) {
    const int p = S.p, h = (p - 1) / 2, nb = S.nb, L = S.L, nbt = S.nbt;
    const int nqt = (h + QT) / QT;  // outputs 0 .. h
    for (int e = threadIdx.x; e < nqt * nbt * RP; e += blockDim.x) {
        const int pr = e % RP, x = e / RP;
        const int qi = fdiv(x, S.magic_nbt), bi = x - qi * nbt;
        const C2<R>* tb[BT];
        int q2[QT], t[QT];
#pragma unroll
        for (int i = 0; i < BT; ++i) tb[i] = T + min(bi + i * nbt, nb - 1) * RP + pr;
#pragma unroll
        for (int i = 0; i < QT; ++i) {
            q2[i] = min(qi * QT + i, h);
            t[i] = 0;
        }
        C2<R> C[QT][BT], D[QT][BT];
#pragma unroll
        for (int i = 0; i < QT; ++i)
#pragma unroll
            for (int k = 0; k < BT; ++k) {
                C[i][k] = tb[k][0];
                D[i][k] = c2(R(0), R(0));
            }
        const int row = nb * RP, hrow = h * row, pad = S.pad;
        const R* w = cm + 2 * pad + qi * QT;
#pragma unroll 4
        for (int q = 1; q <= h; ++q) {
            C2<R> A[BT], B[BT];
            Vec<QT, R> wc, ws;
#pragma unroll
            for (int k = 0; k < BT; ++k) {
                tb[k] += row;
                A[k] = tb[k][0];
                B[k] = tb[k][hrow];
            }
            if constexpr (MAT) {
                wc = *reinterpret_cast<const Vec<QT, R>*>(w);
                ws = *reinterpret_cast<const Vec<QT, R>*>(w + pad);
                w += 2 * pad;
            } else {
#pragma unroll
                for (int i = 0; i < QT; ++i) {
                    t[i] += q2[i];
                    t[i] -= t[i] >= p ? p : 0;
                    const C2<R> v = cs[t[i]];
                    wc.v[i] = v.x;
                    ws.v[i] = v.y;
                }
            }
#pragma unroll
            for (int i = 0; i < QT; ++i)
#pragma unroll
                for (int k = 0; k < BT; ++k) {
                    C[i][k].x = fma(A[k].x, wc.v[i], C[i][k].x);
                    C[i][k].y = fma(A[k].y, wc.v[i], C[i][k].y);
                    D[i][k].x = fma(B[k].x, ws.v[i], D[i][k].x);
                    D[i][k].y = fma(B[k].y, ws.v[i], D[i][k].y);
                }
        }
#pragma unroll
        for (int k = 0; k < BT; ++k) {
            const int b = bi + k * nbt;
            if (b >= nb) continue;
            const int kk = fdiv(b, S.magic_L), ob = kk * L * p + (b - kk * L);
#pragma unroll
            for (int i = 0; i < QT; ++i) {
                const int q = qi * QT + i;
                if (q > h) continue;
                X[(ob + L * q) * RP + pr] = c2(C[i][k].x + D[i][k].y, C[i][k].y - D[i][k].x);
                if (q) X[(ob + L * (p - q)) * RP + pr] = c2(C[i][k].x - D[i][k].y, C[i][k].y + D[i][k].x);
            }
        }
    }
}

// DFT of RP interleaved sequences (element j of sequence r at X[j * RP + r]); returns the buffer
// (X or T) with the result. A barrier precedes the first read and follows the last write.
template <int RP, bool WIDE, class R>
__device__ __forceinline__ C2<R>* fft(const FftArgs& F, const Tables<R>& tab, C2<R>* X, C2<R>* T) {
    __syncthreads();
    for (int s = 0; s < F.nstages; ++s) {
        const FftStage& S = F.st[s];
        const C2<R>* cs = tab.cs + S.csoff;
        bool swap = true;
        switch (S.p) {
            case 2: small_stage<2, RP, R>(S, X, T, cs, tab.tw); break;
            case 3: small_stage<3, RP, R>(S, X, T, cs, tab.tw); break;
            case 4: small_stage<4, RP, R>(S, X, T, cs, tab.tw); break;
            case 5: small_stage<5, RP, R>(S, X, T, cs, tab.tw); break;
            case 7: small_stage<7, RP, R>(S, X, T, cs, tab.tw); break;
            case 8: small_stage<8, RP, R>(S, X, T, cs, tab.tw); break;
            case 6: small_stage<6, RP, R>(S, X, T, cs, tab.tw); break;
            case 9: small_stage<9, RP, R>(S, X, T, cs, tab.tw); break;
            case 10: small_stage<10, RP, R>(S, X, T, cs, tab.tw); break;
            default: {
                const int p = S.p, h = (p - 1) / 2, nb = S.nb, L = S.L, r2 = nb / L;
                for (int e = threadIdx.x; e < (h + 1) * nb * RP; e += blockDim.x) {
                    const int pr = e % RP, x = e / RP;
                    const int q = fdiv(x, S.magic_nb), b = x - q * nb;
                    if (q == 0) {
                        T[e] = X[e];
                    } else {
                        C2<R> uq = X[(b + q * nb) * RP + pr], up = X[(b + (p - q) * nb) * RP + pr];
                        if (L > 1) {
                            const int tj = (b - fdiv(b, S.magic_L) * L) * r2;
                            uq = cmul(uq, tab.tw[q * tj]);
                            up = cmul(up, tab.tw[(p - q) * tj]);
                        }
                        T[e] = cadd(uq, up);
                        T[e + h * nb * RP] = csub(uq, up);
                    }
                }
                __syncthreads();
                if (!S.pad) large_outputs<WIDE ? 4 : 2, 2, RP, false, R>(S, T, X, cs, nullptr);
                else if (WIDE && S.qt == 4) large_outputs<4, 2, RP, true, R>(S, T, X, cs, tab.cm + S.cmoff);
                else if (S.qt == 2) large_outputs<2, 2, RP, true, R>(S, T, X, cs, tab.cm + S.cmoff);
                else large_outputs<1, 1, RP, true, R>(S, T, X, cs, tab.cm + S.cmoff);
                swap = false;
            }
        }
        __syncthreads();
        if (swap) {
            C2<R>* q = X;
            X = T;
            T = q;
        }
    }
    return X;
}

// z_j and z_{N-j} from y_j and y_{N-j} (0 <= j <= N/2; y_0 = y_N = 0).
template <int RP, class R>
__device__ __forceinline__ void put_z(const FftArgs& F, const Tables<R>& tab, C2<R>* X, int j, int pr, R y1, R y2) {
    const C2<R> w = tab.sc[j];
    const R d = R(0.5) * (y1 - y2), c = R(0.5) * (y1 + y2);
    X[j * RP + pr] = c2(fma(c, w.x, d), c * w.y);
    if (j && 2 * j != F.len) X[(F.len - j) * RP + pr] = c2(fma(c, w.x, -d), -c * w.y);
}

// Largest of a non-negative int over the block.
__device__ __forceinline__ int block_max(int v, int* s_red) {
    v = __reduce_max_sync(0xffffffffu, v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) s_red[warp] = v;
    __syncthreads();
    return __reduce_max_sync(0xffffffffu, lane < warps ? s_red[lane] : 0);
}

// ------------------------------------------------------------------ fixed point
// Biased exponent of a double, at least 1 (subnormals count as the smallest normal exponent).
__device__ __forceinline__ int biased_exp(double x) { return max(1, (__double2hiint(x) >> 20) & 0x7ff); }

// x * 2^(1023 - E) as a float for |x| < 2^(E - 1022): bits moved, rounded half up; below 2^-126: 0.
__device__ __forceinline__ float scaled_float(double x, int E) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int f = (int)((hi >> 20) & 0x7ff), e = f - E + 127;
    if (f == 0 || e <= 0) return 0.f;  // a subnormal double counts as zero: its psi underflows too
    const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);
    return __uint_as_float((((unsigned)e << 23) | m) + ((lo >> 28) & 1u) | (hi & 0x80000000u));
}

// x * 2^(1023 - E + S), rounded to an integer (half up in magnitude), modulo 2^64; `rest` takes what the rounding left out, between
// -1/2 and 1/2. Without branches: neighbouring cells take either side.
__device__ __forceinline__ unsigned long long scaled_int(double x, int E, int S, float& rest) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int f = (int)((b >> 52) & 0x7ff);
    unsigned long long m = (b & ((1ull << 52) - 1)) | (f ? 1ull << 52 : 0ull);
    const int sh = max(f, 1) - E - 52 + S;
    m >>= min(max(-53 - sh, 0), 63);         // below half a unit: all of it is rest
    const int r = min(max(10 - sh, 1), 63);  // right shift of m << 10
    const unsigned long long q = (m << 10) + (1ull << (r - 1));
    const unsigned long long left = sh < 64 ? m << max(min(sh, 63), 0) : 0ull;
    const unsigned long long v = sh < 10 ? q >> r : left;
    const float below = fmaf((float)(unsigned)((q << (64 - r)) >> 32), 0x1p-32f, -0.5f);  // (0 for sh >= 0)
    rest = (long long)b < 0 ? -below : below;
    return (long long)b < 0 ? 0ull - v : v;
}

// v * k 2^(kexp) rounded to nearest, for the multiplier k in [2^63, 2^64) and results in the
// normal range (others by scaling a normal one).
__device__ __forceinline__ double scaled_double(long long v, unsigned long long k, int kexp, bool neg) {
    unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    if (a == 0) return 0.0;
    const int lz = __clzll((long long)a);
    unsigned long long p = __umul64hi(a << lz, k);  // in [2^62, 2^64)
    int e = kexp + 64 - lz;
    if (!(p >> 63)) {
        p <<= 1;
        --e;
    }
    // p in [2^63, 2^64), value p 2^e: significand of 53 bits
    unsigned long long mant = (p >> 11) + ((p >> 10) & 1ull);  // 2^52 .. 2^53
    const int be = e + 63 + 1023;
    const unsigned long long sign = ((v < 0) != neg) ? 1ull << 63 : 0;
    if (be >= 1 && be < 0x7fe) return __longlong_as_double((long long)(sign | (((unsigned long long)be << 52) + (mant - (1ull << 52)))));
    const double x = __longlong_as_double((long long)(sign | ((1023ull << 52) + (mant - (1ull << 52)))));
    return scalbn(x, be - 1023);
}

// scaled_int modulo 2^128.
__device__ __forceinline__ unsigned __int128 scaled_int128(double x, int E, int S, float& rest) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int f = (int)((b >> 52) & 0x7ff), sh = max(f, 1) - E - 52 + S;
    const unsigned long long low = scaled_int(x, E, S, rest);
    if (sh < 10) return (unsigned __int128)(__int128)(long long)low;
    const unsigned __int128 m = (b & ((1ull << 52) - 1)) | (f ? 1ull << 52 : 0ull);
    const unsigned __int128 v = sh < 128 ? m << sh : 0;
    return (long long)b < 0 ? 0 - v : v;
}

// Conversions between 64-bit integers and floats by 32-bit ones: the instructions on 64-bit types run at the
// FP64 pipe's rate (two per cycle and SM; the residual of e0 with six of them per cell took 27 us at 1000^2, no more than the later residuals since).
__device__ __forceinline__ float float_of(unsigned long long v) {
    const unsigned long long a = (long long)v < 0 ? 0ull - v : v;
    const float x = fmaf((float)(unsigned)(a >> 32), 4294967296.f, (float)(unsigned)a);
    return (long long)v < 0 ? -x : x;
}
__device__ __forceinline__ float float_of(unsigned __int128 v) {
    const bool neg = (long long)(v >> 64) < 0;
    const unsigned __int128 a = neg ? 0 - v : v;
    const unsigned long long hi = (unsigned long long)(a >> 64), lo = (unsigned long long)a;
    const float top = fmaf((float)(unsigned)(hi >> 32), 0x1p32f, (float)(unsigned)hi);
    const float x = fmaf(top, 0x1p64f, fmaf((float)(unsigned)(lo >> 32), 0x1p32f, (float)(unsigned)lo));
    return neg ? -x : x;
}
__device__ __forceinline__ unsigned long long int_of(float v) {  // |v| < 2^50, to nearest
    const int hi = __float2int_rn(v * 0x1p-20f);
    return (unsigned long long)((long long)hi * (1 << 20) + __float2int_rn(fmaf((float)hi, -0x1p20f, v)));
}
// e0 2^S as fixed point (|e0| 2^S < 2^60), rounded half up in magnitude, without branches.
__device__ __forceinline__ unsigned long long fixed_of(float e0, int S) {
    const unsigned b = __float_as_uint(e0);
    const int f = (int)((b >> 23) & 0xff);
    const unsigned long long m = (unsigned long long)(f ? (b & 0x7fffffu) | 0x800000u : 0u) << 37;  // < 2^61
    const int r = min(max(187 - f - S, 1), 63);  // value m 2^-37 2^(f - 150 + S)
    const unsigned long long v = (m + (1ull << (r - 1))) >> r;
    return (int)b < 0 ? 0ull - v : v;
}

// ------------------------------------------------------------------ the passes
constexpr int kMaxMatrixRadix = 131;  // largest radix whose cosine and sine matrix is tabulated (36 KB)
constexpr int kOneLaunchRows = 1300;  // largest m whose solve is one launch
constexpr int kFp64Rows = 304;        // largest m solved in FP64 at once (fp64_radix_ok)
// Largest extent of the cavity, in lowest terms, whose residual is taken modulo 2^64: it is at most about 2^-22 4 (a^2 + b^2) 2^58 =
// 2^57. Above (very stretched cells, or extents like 1000 x 999) modulo 2^128, where every pair of ints has room (modelled to 2^31 with
// exact integers: three solves leave 1e-17 .. 2e-16). us per solve, 64 / 128 bits: 1024^2 229 (511 : 512) / 237 (1000 : 999), 2048^2 1633
// (1 : 512) / 1700 (1 : 513). Dense products took 4,290 and 29,400 there, FP64 transforms in three launches 610 and 4,370.
constexpr int kMaxExtent = 512;
constexpr int kThreads64 = 256;
constexpr int kThreadsMax = 128;  // threads of a row's (column's) block

// Forms of the passes: kSmall keeps every table in shared memory; kWide, where shared memory leaves room for few blocks
// anyway, takes larger register tiles.
enum Form { kSmall, kMid, kWide };
constexpr int blocks_per_sm(int form) { return form == kWide ? 5 : 8; }  // blocks of kThreadsMax the registers allow


struct KScale {  // scale / kappa = +- k 2^kexp
    unsigned long long k;
    int kexp;
    int neg;
};

// What a pass does before the one ahead of it is done: the tables into shared memory at `sm` (ALL of them on small grids, whose
// passes are a chain of latencies; the large radices' otherwise, the rest through the first-level cache). Then it lets the
// next pass start likewise and waits for the one ahead (each pass waits before it touches any field, so the passes stay in
// order one by one).
template <class R, bool ALL>
__device__ __forceinline__ Tables<R> begin_pass(const FftArgs& F, float4* sm) {
    const float4* src = reinterpret_cast<const float4*>(F.tables + (ALL ? 0 : F.off_cm));
    for (int t = threadIdx.x; t < (F.table_bytes - (ALL ? 0 : F.off_cm)) / 16; t += blockDim.x) sm[t] = __ldg(src + t);
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __syncthreads();
    const char* s = reinterpret_cast<const char*>(sm) - (ALL ? 0 : F.off_cm);
    const char* g = ALL ? s : F.tables;
    return Tables<R>{reinterpret_cast<const C2<R>*>(g), reinterpret_cast<const C2<R>*>(g + F.off_sc),
                     reinterpret_cast<const C2<R>*>(s + F.off_cs), reinterpret_cast<const R*>(g + F.off_li),
                     reinterpret_cast<const R*>(g + F.off_lj), reinterpret_cast<const R*>(s + F.off_cm)};
}

enum { kFirst = 0, kSecond = 1, kLater = 2 };  // pass A: from `in`; residual of e0; residual of psi
enum { kToE0 = 0, kAddToE0 = 1, kAdd = 2, kAddLast = 3 };  // pass C: e0 = ; psi = e0 + ; psi += ; answer = psi +

// Cells (i, 2l) and (i, 2l + 1) of the answer (columns 0 and m + 1 are not written).
__device__ __forceinline__ void store_pair(const DstDest& dst, int i, int l, int m, double x0, double x1) {
    const int j = 2 * l;
    if (dst.red) {
        const size_t o = (size_t)i * dst.pitch + l;
        if (l) (i & 1 ? dst.black : dst.red)[o] = x0;
        if (j < m) (i & 1 ? dst.red : dst.black)[o] = x1;
    } else {
        double* o = dst.out + (size_t)i * dst.ld + j;
        if (l) o[0] = x0;
        if (j < m) o[1] = x1;
    }
}

// What other blocks wrote: through L2 when they ran in this launch (ONE), as it comes otherwise.
template <bool ONE, class V>
__device__ __forceinline__ V field(const V* p) {
    return ONE ? __ldcg(p) : *p;
}

// The shift of the fixed point, from the largest |e0|: it becomes about 2^58.
template <bool ONE>
__device__ __forceinline__ int fixed_shift(const FftArgs& F, int* s_red) {
    int top = 0;
    for (int q = threadIdx.x; q < F.m; q += blockDim.x) top = max(top, (int)field<ONE>(F.mx + q));
    top = block_max(top, s_red);
    return top ? min(127, 58 - ((top >> 23) - 127)) : 0;
}

// A: grid row i: the right-hand side or the residual, transformed along j into t. FAR: the residual modulo 2^128 (kMaxExtent).
template <bool WIDE, bool ONE, bool FAR>
__device__ __forceinline__ void pass_a(const FftArgs& F, const Tables<float>& tab, float2* X, int* s_red, int i, int mode, int E,
                                       int S, const double* in) {
    const int N = F.len, ld = F.ld, half = N / 2 + 1, m = F.m;
    const double* row = in + (size_t)i * F.n;
    if (mode == kFirst) {
        int top = 1;
        for (int j = 1 + threadIdx.x; j <= m; j += blockDim.x) top = max(top, biased_exp(row[j]));
        top = block_max(top, s_red);
        if (threadIdx.x == 0) F.ex[i - 1] = top;
        for (int j = threadIdx.x; j < half; j += blockDim.x) {
            float y1 = 0.f, y2 = 0.f;
            if (j && top != 0x7ff) {
                y1 = scaled_float(row[j], top);
                y2 = scaled_float(row[N - j], top);
            }
            put_z<1, float>(F, tab, X, j, 0, y1, y2);
        }
    } else {
        const unsigned long long a2 = (unsigned long long)F.a2, b2 = (unsigned long long)F.b2, ab = 2 * (a2 + b2);
        const bool unit = a2 == 1 && b2 == 1;
        for (int j = threadIdx.x; j < half; j += blockDim.x) {
            float y[2] = {0.f, 0.f};
            if (j) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int jj = q ? N - j : j;
                    const size_t at = (size_t)i * ld + jj;
                    unsigned long long c, v, h;  // centre, up + down, left + right
                    if (mode == kSecond) {
                        const float* p = F.e0 + at;
                        c = fixed_of(field<ONE>(p), S);
                        v = fixed_of(field<ONE>(p + ld), S) + fixed_of(field<ONE>(p - ld), S);
                        h = fixed_of(field<ONE>(p + 1), S) + fixed_of(field<ONE>(p - 1), S);
                    } else {
                        const unsigned long long* p = reinterpret_cast<const unsigned long long*>(F.psi) + at;
                        c = field<ONE>(p);
                        v = field<ONE>(p + ld) + field<ONE>(p - ld);
                        h = field<ONE>(p + 1) + field<ONE>(p - 1);
                    }
                    float rest;
                    if constexpr (FAR) {
                        auto wide = [](unsigned long long x) { return (unsigned __int128)(__int128)(long long)x; };
                        const unsigned __int128 a = a2, b = b2, g = scaled_int128(row[jj], E, S, rest);
                        y[q] = float_of(g - 2 * (a + b) * wide(c) + a * wide(v) + b * wide(h)) + rest;
                    } else {
                        const unsigned long long g = scaled_int(row[jj], E, S, rest);
                        y[q] = float_of(unit ? g - 4 * c + v + h : g - ab * c + a2 * v + b2 * h) + rest;
                    }
                }
            }
            put_z<1, float>(F, tab, X, j, 0, y[0], y[1]);
        }
    }
    const float2* Z = fft<1, WIDE, float>(F, tab, X, X + N);
    const int nl = (m >> 1) + 1;  // l = 0 .. m/2: modes 2l, 2l+1 (mode 0 is not read)
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        const float2 z = Z[l];
        *reinterpret_cast<float2*>(F.t + (size_t)i * ld + 2 * l) = make_float2(-z.y, z.x);
    }
}

// The exponent of the whole right-hand side, from its rows'.
template <bool ONE>
__device__ __forceinline__ int exponent(const FftArgs& F, int* s_red) {
    int top = 1;
    for (int q = threadIdx.x; q < F.m; q += blockDim.x) top = max(top, field<ONE>(F.ex + q));
    return block_max(top, s_red);
}

// B: columns (j-modes) c0 .. c0 + RP - 1 of t (those in 1 .. m count): transform along i, division by the eigenvalues,
// transform back, in place. In the first solve the rows come scaled by their own exponents.
template <int RP, bool WIDE, bool ONE>
__device__ __forceinline__ void pass_b(const FftArgs& F, const Tables<float>& tab, float2* X, int c0, bool first, int E) {
    const int N = F.len, ld = F.ld, half = N / 2 + 1, m = F.m;
    float2* T = X + (size_t)N * RP;
    for (int e = threadIdx.x; e < half * RP; e += blockDim.x) {
        const int pr = e % RP, j = e / RP;
        float y1 = 0.f, y2 = 0.f;
        if (j) {
            y1 = field<ONE>(F.t + (size_t)j * ld + c0 + pr);
            y2 = field<ONE>(F.t + (size_t)(N - j) * ld + c0 + pr);
            if (first) {
                const int d1 = field<ONE>(F.ex + j - 1) - E + 127, d2 = field<ONE>(F.ex + N - j - 1) - E + 127;
                y1 *= d1 > 0 ? __int_as_float(d1 << 23) : 0.f;
                y2 *= d2 > 0 ? __int_as_float(d2 << 23) : 0.f;
            }
        }
        put_z<RP, float>(F, tab, X, j, pr, y1, y2);
    }
    float2* Z = fft<RP, WIDE, float>(F, tab, X, T);
    float2* O = Z == X ? T : X;
    float* Y = reinterpret_cast<float*>(O);  // modes 0 .. N of every column
    const int nl = (m >> 1) + 1;
    for (int e = threadIdx.x; e < nl * RP; e += blockDim.x) {
        const int pr = e % RP, l = e / RP;
        const float2 z = Z[l * RP + pr];
        const float lj = tab.lj[min(c0 + pr, m)];
        const int k = 2 * l;
        Y[k * RP + pr] = l ? __fdividef(-z.y * F.norm, tab.li[k] + lj) : 0.f;
        Y[(k + 1) * RP + pr] = k < m ? __fdividef(z.x * F.norm, tab.li[k + 1] + lj) : 0.f;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < half * RP; e += blockDim.x) {
        const int pr = e % RP, j = e / RP;
        const float y1 = j ? Y[j * RP + pr] : 0.f, y2 = j ? Y[(N - j) * RP + pr] : 0.f;
        put_z<RP, float>(F, tab, Z, j, pr, y1, y2);
    }
    const float2* R = fft<RP, WIDE, float>(F, tab, Z, O);
    for (int e = threadIdx.x; e < nl * RP; e += blockDim.x) {
        const int pr = e % RP, l = e / RP;
        const float2 z = R[l * RP + pr];
        float* d = F.t + (size_t)(2 * l) * ld + c0 + pr;
        if (l) d[0] = -z.y;
        if (2 * l < m) d[ld] = z.x;
    }
}

// C: row i of t transformed back along j and added to the solution.
template <bool WIDE, bool ONE>
__device__ __forceinline__ void pass_c(const FftArgs& F, const Tables<float>& tab, float2* X, int* s_red, int i, int mode, int E,
                                       int S, const KScale& ks, const DstDest& dst) {
    const int N = F.len, ld = F.ld, half = N / 2 + 1, m = F.m;
    const float* r = F.t + (size_t)i * ld;
    for (int j = threadIdx.x; j < half; j += blockDim.x)
        put_z<1, float>(F, tab, X, j, 0, j ? field<ONE>(r + j) : 0.f, j ? field<ONE>(r + N - j) : 0.f);
    const float2* Z = fft<1, WIDE, float>(F, tab, X, X + N);
    const int nl = (m >> 1) + 1;
    float top = 0.f;
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        const int j = 2 * l;
        const float2 z = Z[l];
        const float v0 = l ? -z.y : 0.f, v1 = j < m ? z.x : 0.f;  // columns j, j + 1 (0 and N stay zero)
        const size_t at = (size_t)i * ld + j;
        if (mode == kToE0) {
            *reinterpret_cast<float2*>(F.e0 + at) = make_float2(v0, v1);
            top = fmaxf(top, fmaxf(fabsf(v0), fabsf(v1)));
            continue;
        }
        longlong2 p;  // this row's block wrote these
        if (mode == kAddToE0) {
            const float2 e0 = *reinterpret_cast<const float2*>(F.e0 + at);
            p = make_longlong2((long long)fixed_of(e0.x, S), (long long)fixed_of(e0.y, S));
        } else {
            p = *reinterpret_cast<const longlong2*>(F.psi + at);
        }
        p.x += (long long)int_of(v0);
        p.y += (long long)int_of(v1);
        if (mode != kAddLast) {
            *reinterpret_cast<longlong2*>(F.psi + at) = p;
            continue;
        }
        const int kexp = ks.kexp + E - 1023 - S;
        double x0 = scaled_double(p.x, ks.k, kexp, ks.neg), x1 = scaled_double(p.y, ks.k, kexp, ks.neg);
        if (E == 0x7ff) x0 = x1 = __longlong_as_double(0x7ff8000000000000ll);  // NaN or Inf in the input
        store_pair(dst, i, l, m, x0, x1);
    }
    if (mode == kToE0) {
        const int t = block_max(__float_as_int(top), s_red);
        if (threadIdx.x == 0) F.mx[i - 1] = (unsigned)t;
    }
}

__device__ __forceinline__ int a_mode(int k) { return k == 0 ? kFirst : k == 1 ? kSecond : kLater; }
__device__ __forceinline__ int c_mode(int k, int solves) {
    return k == 0 ? kToE0 : k == solves - 1 ? kAddLast : k == 1 ? kAddToE0 : kAdd;
}

// The passes as launches of their own (kMid and kWide): solve k of `solves`, a row (cols_b columns) per block.
template <int FORM, bool FAR>
__global__ void __launch_bounds__(kThreadsMax, blocks_per_sm(FORM)) k_dst_a(FftArgs F, int k, const double* in) {
    extern __shared__ float2 fsm[];
    __shared__ int s_red[8];
    const Tables<float> tab = begin_pass<float, false>(F, reinterpret_cast<float4*>(fsm + F.fields));
    const int E = k ? F.ctl[0] : 0;
    const int S = k == 0 ? 0 : k == 1 ? fixed_shift<false>(F, s_red) : F.ctl[1];
    if (k == 1 && blockIdx.x == 0 && threadIdx.x == 0) F.ctl[1] = S;
    pass_a<FORM == kWide, false, FAR>(F, tab, fsm, s_red, 1 + blockIdx.x, a_mode(k), E, S, in);
}

template <int RP, int FORM>
__global__ void __launch_bounds__(RP * kThreadsMax, blocks_per_sm(FORM) / RP) k_dst_b(FftArgs F, int k) {
    extern __shared__ float2 fsm[];
    __shared__ int s_red[8];
    const Tables<float> tab = begin_pass<float, false>(F, reinterpret_cast<float4*>(fsm + F.fields * RP));
    const int E = k ? 0 : exponent<false>(F, s_red);
    if (k == 0 && blockIdx.x == 0 && threadIdx.x == 0) F.ctl[0] = E;
    pass_b<RP, FORM == kWide, false>(F, tab, fsm, blockIdx.x * RP, k == 0, E);
}

template <int FORM>
__global__ void __launch_bounds__(kThreadsMax, blocks_per_sm(FORM)) k_dst_c(FftArgs F, int k, int solves, KScale ks, DstDest dst) {
    extern __shared__ float2 fsm[];
    __shared__ int s_red[8];
    const Tables<float> tab = begin_pass<float, false>(F, reinterpret_cast<float4*>(fsm + F.fields));
    pass_c<FORM == kWide, false>(F, tab, fsm, s_red, 1 + blockIdx.x, c_mode(k, solves), F.ctl[0], k ? F.ctl[1] : 0, ks, dst);
}

// Bounded grid barrier between passes: ctl[2] counts arrivals; the last block to leave, by the ticket ctl[3], re-arms it.
struct GridBarrier {
    int* ctl;
    Ctrl* ctrl;
    long long timeout_ns;
    int stall_block;
    unsigned arrivals;
    __device__ __forceinline__ bool wait() {
        __shared__ int s_ok;
        unsigned* count = reinterpret_cast<unsigned*>(ctl + 2);
        __syncthreads();
        arrivals += gridDim.x;
        if (threadIdx.x == 0) {
            __threadfence();
            if ((int)blockIdx.x != stall_block) atomicAdd(count, 1u);
            s_ok = wait_geq(count, arrivals, ctrl, timeout_ns) ? 1 : 0;
        }
        __syncthreads();
        return s_ok != 0;
    }
    __device__ __forceinline__ void leave() {
        if (threadIdx.x == 0 && atomicInc(reinterpret_cast<unsigned*>(ctl + 3), gridDim.x - 1) == gridDim.x - 1)
            atomicExch(reinterpret_cast<unsigned*>(ctl + 2), 0u);
    }
};

// All passes of a solve in one cooperative launch, block b taking row b + 1 and column b + 1, with a grid barrier between passes.
template <int FORM, bool FAR>
__global__ void __launch_bounds__(kThreadsMax, blocks_per_sm(FORM))
    k_dst_all(FftArgs F, int solves, const double* in, KScale ks, DstDest dst, Ctrl* ctrl, long long timeout_ns, int stall_block) {
    extern __shared__ float2 fsm[];
    __shared__ int s_red[8];
    if (ctrl->abort) return;
    const Tables<float> tab = begin_pass<float, FORM == kSmall>(F, reinterpret_cast<float4*>(fsm + F.fields));
    GridBarrier bar{F.ctl, ctrl, timeout_ns, stall_block, 0};
    const int i = 1 + blockIdx.x;
    int E = 0, S = 0;
    for (int k = 0; k < solves; ++k) {
        if (k == 1) S = fixed_shift<true>(F, s_red);
        pass_a<FORM == kWide, true, FAR>(F, tab, fsm, s_red, i, a_mode(k), E, S, in);
        if (!bar.wait()) return;
        if (k == 0) E = exponent<true>(F, s_red);
        pass_b<1, FORM == kWide, true>(F, tab, fsm, i, k == 0, E);
        if (!bar.wait()) return;
        pass_c<FORM == kWide, true>(F, tab, fsm, s_red, i, c_mode(k, solves), E, S, ks, dst);
        if (k + 1 < solves && !bar.wait()) return;
    }
    bar.leave();
}

// The same for small grids, where a solve is a chain of latencies, in FP64 at once: three passes and two barriers (1.6 us
// each) for nine and eight. 130^2: 48 us, where the FP32 form in one launch takes 52 and a launch per pass 70 (three FP64
// passes in launches of their own took 58); at 256^2 a step takes 15 % less than with the FP32 form. It lasts while an SM has
// no more than two rows (kFp64Rows): the FP64 work of a third costs more than the FP32 form's further passes.
__global__ void __launch_bounds__(kThreads64)
    k_dst_fp64(FftArgs F, const double* in, double scale, DstDest dst, Ctrl* ctrl, long long timeout_ns, int stall_block) {
    extern __shared__ double2 dsm[];
    if (ctrl->abort) return;
    const int N = F.len, m = F.m, ld = F.ld, half = N / 2 + 1, nl = (m >> 1) + 1, i = 1 + blockIdx.x;
    double2* X = dsm;
    double2* T = dsm + N;
    const Tables<double> tab = begin_pass<double, true>(F, reinterpret_cast<float4*>(dsm + F.fields));
    GridBarrier bar{F.ctl, ctrl, timeout_ns, stall_block, 0};
    // along j
    const double* row = in + (size_t)i * F.n;
    for (int j = threadIdx.x; j < half; j += blockDim.x)
        put_z<1, double>(F, tab, X, j, 0, j ? scale * row[j] : 0.0, j ? scale * row[N - j] : 0.0);
    double2* Z = fft<1, false, double>(F, tab, X, T);
    double* t = F.t64 + (size_t)i * ld;
    for (int l = threadIdx.x; l < nl; l += blockDim.x) *reinterpret_cast<double2*>(t + 2 * l) = make_double2(-Z[l].y, Z[l].x);
    if (!bar.wait()) return;
    // along i, divided, back along i: column i
    t = F.t64 + i;
    for (int j = threadIdx.x; j < half; j += blockDim.x)
        put_z<1, double>(F, tab, X, j, 0, j ? __ldcg(t + (size_t)j * ld) : 0.0, j ? __ldcg(t + (size_t)(N - j) * ld) : 0.0);
    Z = fft<1, false, double>(F, tab, X, T);
    double2* O = Z == X ? T : X;
    double* Y = reinterpret_cast<double*>(O);
    const double lj = tab.lj[i];
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        const int k = 2 * l;
        Y[k] = l ? -Z[l].y * F.norm64 / (tab.li[k] + lj) : 0.0;
        Y[k + 1] = k < m ? Z[l].x * F.norm64 / (tab.li[k + 1] + lj) : 0.0;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < half; j += blockDim.x)
        put_z<1, double>(F, tab, Z, j, 0, j ? Y[j] : 0.0, j ? Y[N - j] : 0.0);
    Z = fft<1, false, double>(F, tab, Z, O);
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        if (l) t[(size_t)(2 * l) * ld] = -Z[l].y;
        if (2 * l < m) t[(size_t)(2 * l + 1) * ld] = Z[l].x;
    }
    if (!bar.wait()) return;
    // back along j
    t = F.t64 + (size_t)i * ld;
    for (int j = threadIdx.x; j < half; j += blockDim.x)
        put_z<1, double>(F, tab, X, j, 0, j ? __ldcg(t + j) : 0.0, j ? __ldcg(t + N - j) : 0.0);
    Z = fft<1, false, double>(F, tab, X, T);
    for (int l = threadIdx.x; l < nl; l += blockDim.x) store_pair(dst, i, l, m, -Z[l].y, Z[l].x);
    bar.leave();
}

// ------------------------------------------------------- dense fallback: out = X * S
// Destination of a dense product's value for row r, column c: row-major out[(r + off) * ld + c +
// off], out[c * ld + r] when transposed, or the split layout (as DstDest). With lam_r set, the
// value is first divided by lam_r[r] + lam_c[c].
struct DenseDest {
    double* out;
    int ld, off;
    double* red;
    double* black;
    int pitch;
    int transposed;
    const double* lam_r;
    const double* lam_c;
    __device__ __forceinline__ void put(int r, int c, double val) const {
        if (lam_r) val = val / (__ldg(lam_r + r) + __ldg(lam_c + c));
        if (transposed) {
            out[(size_t)c * ld + r] = val;
            return;
        }
        const int i = r + off, j = c + off;
        if (red) ((i + j) & 1 ? black : red)[(size_t)i * pitch + (j >> 1)] = val;
        else out[(size_t)i * ld + j] = val;
    }
};

constexpr int kCols = 64;     // output columns per block (one per thread column)
constexpr int kRowsT = 4;     // thread rows per block
constexpr int kBk = 32;       // reduction chunk (even, so chunk-local parity = global parity)
constexpr int kThreads = kCols * kRowsT;

// X(r, b) = xs * x[(r + xo) * xld + b + xo]. Column c < half gets E + O, column m-1-c gets E - O
// (E, O: the even-b and odd-b halves of the dot product). RR rows per block.
template <int RR>
__global__ void __launch_bounds__(kThreads) k_dst_right(const double* __restrict__ S, int m,
                                                        const double* __restrict__ x, int xld, int xo, double xs,
                                                        DenseDest dst) {
    __shared__ double s_x[RR][kBk + 1];
    __shared__ double s_s[kBk][kCols];
    const int half = (m + 1) / 2;
    const int tx = threadIdx.x % kCols, ty = threadIdx.x / kCols;
    const int r0 = blockIdx.y * RR, c = blockIdx.x * kCols + tx;  // folded column
    constexpr int Q = RR / kRowsT;
    double e[Q], o[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) e[q] = o[q] = 0.0;
    for (int b0 = 0; b0 < m; b0 += kBk) {
        for (int t = threadIdx.x; t < RR * kBk; t += kThreads) {
            const int r = t / kBk, bb = t % kBk;
            const int row = r0 + r, b = b0 + bb;
            s_x[r][bb] = (row < m && b < m) ? xs * x[(size_t)(row + xo) * xld + b + xo] : 0.0;
        }
        for (int t = threadIdx.x; t < kBk * kCols; t += kThreads) {
            const int bb = t / kCols, cc = t % kCols;
            const int b = b0 + bb, col = blockIdx.x * kCols + cc;
            s_s[bb][cc] = (b < m && col < half) ? S[(size_t)b * m + col] : 0.0;  // S symmetric
        }
        __syncthreads();
#pragma unroll 8
        for (int bb = 0; bb < kBk; bb += 2) {
            const double se = s_s[bb][tx], so = s_s[bb + 1][tx];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                e[q] = __fma_rn(s_x[ty + kRowsT * q][bb], se, e[q]);
                o[q] = __fma_rn(s_x[ty + kRowsT * q][bb + 1], so, o[q]);
            }
        }
        __syncthreads();
    }
    if (c >= half) return;
    const int c2 = m - 1 - c;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int r = r0 + ty + kRowsT * q;
        if (r >= m) continue;
        dst.put(r, c, e[q] + o[q]);
        if (c2 != c) dst.put(r, c2, e[q] - o[q]);
    }
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

// One dense transform along j of every row: dst(r, c) = sum_b X(r, b) S[b][c], X(r, b) = xs *
// x[(r + xo) * xld + b + xo].
cudaError_t transform_rows(const DstPlan& P, const double* x, int xld, int xo, double xs, const DenseDest& d,
                           cudaStream_t s) {
    const dim3 grid(ceil_div((P.m + 1) / 2, kCols), ceil_div(P.m, P.rows));
    switch (P.rows) {
        case 16: k_dst_right<16><<<grid, kThreads, 0, s>>>(P.S, P.m, x, xld, xo, xs, d); break;
        case 8: k_dst_right<8><<<grid, kThreads, 0, s>>>(P.S, P.m, x, xld, xo, xs, d); break;
        default: k_dst_right<4><<<grid, kThreads, 0, s>>>(P.S, P.m, x, xld, xo, xs, d); break;
    }
    return cudaGetLastError();
}

// scale / kappa as +- k 2^kexp
KScale multiplier(double scale, double kappa) {
    int ex = 0;
    const long double f = std::frexp(std::fabs((long double)scale / (long double)kappa), &ex);
    KScale ks;
    ks.k = (unsigned long long)std::ldexp(f, 64);  // f in [1/2, 1)
    if (!(ks.k >> 63)) ks.k = 1ull << 63;
    ks.kexp = ex - 64;
    ks.neg = scale < 0 ? 1 : 0;
    return ks;
}

// One pass, whose successor may start before it is done (begin_pass); or, cooperative, all of them.
template <class... Params, class... Args>
cudaError_t launch_pass(void (*k)(Params...), int blocks, int threads, int smem, bool cooperative, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (cooperative) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, Params(args)...);
}

// The kernels of a plan. k_dst_a, k_dst_b and k_dst_c come in the forms that may need more than one launch (plan_fft).
template <bool FAR>
auto kernel_all(int form) { return form == kSmall ? k_dst_all<kSmall, FAR> : form == kMid ? k_dst_all<kMid, FAR> : k_dst_all<kWide, FAR>; }
auto kernel_all(const DstPlan& P) { return P.far ? kernel_all<true>(P.form) : kernel_all<false>(P.form); }
auto kernel_a(const DstPlan& P) {
    return P.form == kMid ? (P.far ? k_dst_a<kMid, true> : k_dst_a<kMid, false>) : P.far ? k_dst_a<kWide, true> : k_dst_a<kWide, false>;
}
auto kernel_b(const DstPlan& P) { return P.F.cols_b == 1 ? k_dst_b<1, kWide> : P.form == kMid ? k_dst_b<2, kMid> : k_dst_b<2, kWide>; }
auto kernel_c(const DstPlan& P) { return P.form == kMid ? k_dst_c<kMid> : k_dst_c<kWide>; }

cudaError_t solve(const DstPlan& P, const double* in, double scale, const DstDest& d, cudaStream_t s) {
    const int m = P.m;
    cudaError_t e;
    if (P.F.len) {
        const FftArgs& F = P.F;
        const KScale ks = multiplier(scale, P.kappa);
        const int blocks_b = ceil_div(m + 1, F.cols_b);  // modes 0 .. m; mode 0 is padding
        if (P.fp64)
            return launch_pass(k_dst_fp64, m, kThreads64, P.smem_a, true, s, F, in, scale, d, P.ctrl, P.timeout_ns, P.stall_block);
        if (P.one_launch) {
            return launch_pass(kernel_all(P), m, P.threads_a, P.smem_a, true, s, F, P.solves, in, ks, d, P.ctrl, P.timeout_ns, P.stall_block);
        }
        for (int k = 0; k < P.solves; ++k) {
            if ((e = launch_pass(kernel_a(P), m, P.threads_a, P.smem_a, false, s, F, k, in)) != cudaSuccess) return e;
            if ((e = launch_pass(kernel_b(P), blocks_b, P.threads_b, P.smem_b, false, s, F, k)) != cudaSuccess) return e;
            if ((e = launch_pass(kernel_c(P), m, P.threads_a, P.smem_a, false, s, F, k, P.solves, ks, d)) != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    const DenseDest t1_tr{P.t1, m, 0, nullptr, nullptr, 0, 1, nullptr, nullptr};
    if ((e = transform_rows(P, in, P.n, 1, scale, t1_tr, s)) != cudaSuccess) return e;  // along j
    const DenseDest t2_div{P.t2, m, 0, nullptr, nullptr, 0, 0, P.lam_j, P.lam_i};  // rows b, columns a
    if ((e = transform_rows(P, P.t1, m, 0, 1.0, t2_div, s)) != cudaSuccess) return e;  // along i, / lambda
    if ((e = transform_rows(P, P.t2, m, 0, 1.0, t1_tr, s)) != cudaSuccess) return e;   // back along a
    const DenseDest last{d.out, d.ld, 1, d.red, d.black, d.pitch, 0, nullptr, nullptr};
    return transform_rows(P, P.t1, m, 0, 1.0, last, s);                                 // back along b
}

// Radices of the FFT: the large prime factors of len, then its small ones grouped into radices one
// thread does in registers (up to 10), largest first. False when there are too many stages.
bool radices(int len, std::vector<int>* out) {
    std::vector<int> small;  // ascending
    out->clear();
    for (int p = 2; len > 1; ++p) {
        if (p * p > len) p = len;
        for (; len % p == 0; len /= p) (p <= 7 ? small : *out).push_back(p);
    }
    while (!small.empty()) {  // the largest left, times the largest others that fit
        int r = small.back();
        small.pop_back();
        for (int k = (int)small.size() - 1; k >= 0; --k)
            if (r * small[k] <= 10) {
                r *= small[k];
                small.erase(small.begin() + k);
            }
        out->push_back(r);
    }
    std::sort(out->rbegin(), out->rend());
    return (int)out->size() <= kMaxFftStages;
}

unsigned magic_of(int d) { return d == 1 ? 0u : 0xffffffffu / (unsigned)d + 1u; }

int gcd(int a, int b) { return b ? gcd(b, a % b) : a; }

// Solves needed so that the last correction leaves less than 1e-16: an FP32 transform of a row is
// off by about 1e-7 (1 + sqrt(p) / 8) of the row's norm for a largest radix p; a solve's error in psi
// is that of its last two transforms, and through the residual (an operator norm of 4.5 over the
// smallest eigenvalue's share N / 20, more where the cells are stretched) it becomes the next one's.
int solves_needed(int len, int radix, double a2, double b2) {
    const double eps = 1e-7 * (1 + std::sqrt((double)radix) / 8);
    const double amp = len / 20.0 * (a2 + b2) / (2 * std::min(a2, b2));
    double high = 2 * eps, low = 0;  // error of psi: all over the spectrum, and in the lowest modes
    int k = 1;
    for (; k < 6 && high + low > 1e-16; ++k) {
        const double r = 4.5 * high + low / (amp * len);  // the residual
        low = eps * r * amp;
        high = 2 * eps * (high + low);
    }
    return std::max(k, 3);
}

// exp(2 pi i t / M), M = 4 len, in W: computed for the first eighth of the circle, exact symmetries for the rest (on an Arm
// host a long double sine takes a microsecond of software).
template <class W>
struct Roots {
    int len;
    std::vector<W> c, s;
    explicit Roots(int len) : len(len), c(len / 2 + 1), s(len / 2 + 1) {
        const W pi = (W)3.141592653589793238462643383279502884L;
        for (int t = 0; t <= len / 2; ++t) {
            c[t] = std::cos(pi * t / (2 * len));
            s[t] = std::sin(pi * t / (2 * len));
        }
    }
    W first(int r, bool sine) const { return 2 * r <= len ? (sine ? s[r] : c[r]) : (sine ? c[len - r] : s[len - r]); }
    W cos(long long t) const {  // t >= 0
        const int q = (int)(t / len % 4), r = (int)(t % len);
        const W v = first(r, q & 1);
        return q == 1 || q == 2 ? -v : v;
    }
    W sin(long long t) const { return cos(t + 3LL * len); }
};

// The FFT path's tables and fields for len = m + 1; false where it does not apply.
template <class R>
bool plan_fft(DstPlan* P, int a, int b, int sms, int smem_max, int* status) {
    const int m = P->m, len = m + 1;
    std::vector<int> rad;
    if (!radices(len, &rad)) return false;
    FftArgs& F = P->F;
    int ncs = 0, ncm = 0;  // entries of the radices' tables and of the large ones' matrices
    for (int p : rad) {
        const int h = (p - 1) / 2;
        ncs += p;
        if (p > 10 && p <= kMaxMatrixRadix) ncm += 2 * h * ((h + 1 + 3) / 4 * 4);
    }
    constexpr bool kF64 = sizeof(R) == 8;
    auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const int own = (int)(align(sizeof(R) * (size_t)std::max(ncm, 1)) + align(2 * sizeof(R) * (size_t)ncs));  // the part every block holds
    const int fields = (len + 1) / 2 * 4;  // two buffers of a row, in pairs, a multiple of 32 bytes
    const size_t row_bytes = 2 * sizeof(R) * (size_t)fields;
    if (row_bytes + own + 512 > (size_t)smem_max) return false;
    F.fields = fields;
    F.n = P->n;
    F.m = m;
    F.ld = (len + 1 + 7) / 8 * 8;
    F.nstages = (int)rad.size();
    F.norm64 = 4.0 / ((double)len * len);
    F.norm = (float)F.norm64;
    F.a2 = (long long)a * a;
    F.b2 = (long long)b * b;
    // columns per block of B: one on small grids (a block per column keeps the SMs busy), two on larger ones (8 bytes
    // of each row)
    F.cols_b = m <= 2 * sms || 2 * (2 * row_bytes + own) > (size_t)smem_max ? 1 : 2;
    P->threads_a = kThreadsMax;
    P->threads_b = F.cols_b * kThreadsMax;
    // every table in shared memory on small grids; the wide form where a row and its tables take more than a sixth of it
    P->form = kF64 || (F.cols_b == 1 && 24 * len + 4 * ncm <= 12288) ? kSmall : row_bytes + own > (size_t)smem_max / 6 ? kWide : kMid;
    // stages; a large radix takes the largest register tile that still leaves every thread one
    for (int s = 0, L = 1, off = 0, cm = 0; s < F.nstages; ++s) {
        FftStage& S = F.st[s];
        S.p = rad[s];
        S.L = L;
        S.nb = len / S.p;
        S.csoff = off;
        const int h = (S.p - 1) / 2;
        S.qt = S.bt = 1;
        if (S.p > 10) {
            const bool mat = S.p <= kMaxMatrixRadix;
            for (int qt : {P->form == kWide ? 4 : 2, 2})
                if (S.qt == 1 && S.nb > 1 && (!mat || ceil_div(h + 1, qt) * ceil_div(S.nb, 2) >= kThreadsMax / 2)) S.qt = qt, S.bt = 2;
            if (mat) {
                S.pad = (h + 1 + 3) / 4 * 4;
                S.cmoff = cm - 2 * S.pad;  // rows q = 1 .. h
                cm += 2 * h * S.pad;
            } else {
                S.qt = P->form == kWide ? 4 : 2, S.bt = 2;
            }
        }
        S.nbt = ceil_div(S.nb, S.bt);
        S.magic_L = magic_of(L);
        S.magic_nb = magic_of(S.nb);
        S.magic_nbt = magic_of(S.nbt);
        L *= S.p;
        off += S.p;
    }
    const Roots<typename Pair<R>::wide> roots(len);  // exp(2 pi i t / 4N), from which every table comes
    std::vector<C2<R>> tw(len), cs(ncs), sc(len / 2 + 1);
    std::vector<R> li(len + 1, R(0)), lj(len + 1, R(0));
    for (int t = 0; t < len; ++t) tw[t] = C2<R>{(R)roots.cos(4 * t), (R)-roots.sin(4 * t)};  // exp(-2 pi i t / N)
    for (int t = 0; t <= len / 2; ++t) sc[t] = C2<R>{(R)roots.sin(2 * t), (R)roots.cos(2 * t)};
    for (int s = 0; s < F.nstages; ++s)
        for (int t = 0; t < rad[s]; ++t)
            cs[F.st[s].csoff + t] = C2<R>{(R)roots.cos(4 * t * (len / rad[s])), (R)roots.sin(4 * t * (len / rad[s]))};
    for (int k = 1; k <= m; ++k) {
        const auto sk = roots.sin(k);
        li[k] = (R)(4 * (kF64 ? P->dy2 : (double)F.a2) * sk * sk);
        lj[k] = (R)(4 * (kF64 ? P->dx2 : (double)F.b2) * sk * sk);
    }
    std::vector<R> cm(std::max(ncm, 1));
    for (int s = 0; s < F.nstages; ++s) {
        const FftStage& S = F.st[s];
        for (int q = 1; S.pad && q <= (S.p - 1) / 2; ++q)
            for (int k = 0; k < S.pad; ++k) {
                R* row = cm.data() + S.cmoff + 2 * q * S.pad + k;
                row[0] = cs[S.csoff + q * k % S.p].x;
                row[S.pad] = cs[S.csoff + q * k % S.p].y;
            }
    }
    // one allocation: tables, then the fields (zeroed: their edges stay zero)
    const size_t field = (size_t)(m + 2) * F.ld;
    const size_t part[] = {tw.size() * sizeof(tw[0]), sc.size() * sizeof(sc[0]), li.size() * sizeof(R), lj.size() * sizeof(R),
                           cm.size() * sizeof(R), cs.size() * sizeof(cs[0]), field * sizeof(R), kF64 ? 0 : field * 4,
                           kF64 ? 0 : field * 8, (size_t)m * 4, (size_t)m * 4, 16};
    constexpr int kParts = 12, kTables = 6;
    size_t total = 0;
    for (size_t x : part) total += align(x);
    *status = CNV_CUDA_ERROR;
    if (cudaMalloc(&P->arena, total) != cudaSuccess || cudaMemset(P->arena, 0, total) != cudaSuccess) return true;
    char* at = static_cast<char*>(P->arena);
    char* ptr[kParts];
    for (int k = 0; k < kParts; ++k) {
        ptr[k] = at;
        at += align(part[k]);
    }
    const void* tables[] = {tw.data(), sc.data(), li.data(), lj.data(), cm.data(), cs.data()};
    std::vector<char> host(ptr[kTables] - ptr[0], 0);
    for (int k = 0; k < kTables; ++k) std::memcpy(host.data() + (ptr[k] - ptr[0]), tables[k], part[k]);
    if (cudaMemcpy(P->arena, host.data(), host.size(), cudaMemcpyHostToDevice) != cudaSuccess) return true;
    F.tables = ptr[0];
    F.off_sc = (int)(ptr[1] - ptr[0]);
    F.off_li = (int)(ptr[2] - ptr[0]);
    F.off_lj = (int)(ptr[3] - ptr[0]);
    F.off_cm = (int)(ptr[4] - ptr[0]);
    F.off_cs = (int)(ptr[5] - ptr[0]);
    F.table_bytes = (int)(ptr[6] - ptr[0]);
    const int held = kF64 || P->form == kSmall ? F.table_bytes : own;
    P->smem_a = (int)row_bytes + held;
    P->smem_b = (int)row_bytes * F.cols_b + held;
    F.t = reinterpret_cast<float*>(ptr[6]);
    F.t64 = reinterpret_cast<double*>(ptr[6]);
    F.e0 = reinterpret_cast<float*>(ptr[7]);
    F.psi = reinterpret_cast<long long*>(ptr[8]);
    F.ex = reinterpret_cast<int*>(ptr[9]);
    F.mx = reinterpret_cast<unsigned*>(ptr[10]);
    F.ctl = reinterpret_cast<int*>(ptr[11]);
    F.len = len;
    P->solves = solves_needed(len, rad[0], (double)F.a2, (double)F.b2);
    P->kappa = 0.5 * (P->dy2 / F.a2 + P->dx2 / F.b2);
    P->far = std::max(a, b) > kMaxExtent;
    P->fp64 = kF64;
    // the same limit for every plan: a function's attribute is shared by all of them
    auto allow = [&](const void* k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max - 512) == cudaSuccess;
    };
    int per_sm = 0;
    const void* all = kF64 ? (const void*)k_dst_fp64 : (const void*)kernel_all(*P);
    if (!allow(all) ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, all, kF64 ? kThreads64 : P->threads_a, P->smem_a) != cudaSuccess)
        return true;
    P->one_launch = m <= per_sm * sms && m <= kOneLaunchRows;
    if (!P->one_launch) {
        // (a device with room for fewer blocks than a GB300; there the small forms always fit)
        if (kF64 || P->form == kSmall || (P->form == kMid && F.cols_b == 1)) return false;
        if (!allow((const void*)kernel_a(*P)) || !allow((const void*)kernel_b(*P)) || !allow((const void*)kernel_c(*P))) return true;
    }
    // copies from pageable memory may still be on their way, and the callers' streams do not wait for the default one
    if (cudaDeviceSynchronize() != cudaSuccess) return true;
    *status = CNV_OK;
    return true;
}

// Whether a transform of length len suits the FP64 form: its work grows with the largest prime factor p, which the FP32 form
// does at FP32 rates. us per step, FP64 / FP32 (and the dense products of before): 135^2 (p = 67) 84.9 / 90.7 (113.7), 159^2 (79)
// 95.5 / 94.6, 98^2 (97) 90.3 / 86.2, 202^2 (67) 109.7 / 103.6, 296^2 (59) 130.2 / 128.8, 200^2 (199) 299 / 149 (182).
bool fp64_radix_ok(int len) {
    int p = 1, rest = len;
    for (int f = 2; f * f <= rest; ++f)
        while (rest % f == 0) {
            rest /= f;
            p = std::max(p, f);
        }
    p = std::max(p, rest);
    return p <= 61 || (p <= 79 && len <= 160);
}

}  // namespace

int dst_plan_create(int n, int Lx, int Ly, Ctrl* ctrl, long long timeout_ns, int stall_block, DstPlan* P) {
    *P = DstPlan{};
    P->ctrl = ctrl;
    P->timeout_ns = timeout_ns;
    P->stall_block = stall_block;
    if (n < 3 || Lx < 1 || Ly < 1) return CNV_BAD_ARG;
    const int m = n - 2;
    const double dx = (double)Lx / n, dy = (double)Ly / n;
    P->n = n;
    P->m = m;
    P->dx2 = dx * dx;
    P->dy2 = dy * dy;
    int dev = 0, smem_max = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess) return CNV_CUDA_ERROR;
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int g = gcd(Lx, Ly);
    int status = CNV_OK;
    const DstPlan bare = *P;
    if (m <= kFp64Rows && fp64_radix_ok(m + 1)) {
        if (plan_fft<double>(P, Ly / g, Lx / g, sms, smem_max, &status)) {
            if (status != CNV_OK) dst_plan_destroy(P);
            return status;
        }
        dst_plan_destroy(P);
        *P = bare;
    }
    if (plan_fft<float>(P, Ly / g, Lx / g, sms, smem_max, &status)) {
        if (status != CNV_OK) dst_plan_destroy(P);
        return status;
    }
    dst_plan_destroy(P);
    *P = bare;
    // dense products with the DST matrix
    const double pi = std::acos(-1.0);
    std::vector<double> S((size_t)m * m);
    const double scale = std::sqrt(2.0 / (m + 1));
    const long long period = 2LL * (m + 1);
    for (int a = 0; a < m; ++a)
        for (int b = 0; b < m; ++b) {
            const long long k = ((long long)(a + 1) * (b + 1)) % period;  // exact argument reduction
            S[(size_t)a * m + b] = scale * std::sin(pi * (double)k / (m + 1));
        }
    // more, smaller blocks when the grid is small, so that every SM gets work
    const int cols = ceil_div((m + 1) / 2, kCols);
    P->rows = (cols * ceil_div(m, 16) >= 2 * sms) ? 16 : (cols * ceil_div(m, 8) >= 2 * sms) ? 8 : 4;
    // eigenvalue parts 4 h^2 sin^2(pi (k+1) / (2 (m+1))), in long double, rounded once
    std::vector<double> li(m), lj(m);
    for (int k = 0; k < m; ++k) {
        const long double sk = std::sin(3.141592653589793238462643383279502884L * (k + 1) / (2.0L * (m + 1)));
        li[k] = (double)(4.0L * (long double)P->dy2 * sk * sk);
        lj[k] = (double)(4.0L * (long double)P->dx2 * sk * sk);
    }
    const size_t mm = (size_t)m * m;
    if (cudaMalloc(&P->S, mm * sizeof(double)) != cudaSuccess ||
        cudaMemcpy(P->S, S.data(), mm * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMalloc(&P->t1, mm * sizeof(double)) != cudaSuccess || cudaMalloc(&P->t2, mm * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&P->lam_i, m * sizeof(double)) != cudaSuccess || cudaMalloc(&P->lam_j, m * sizeof(double)) != cudaSuccess ||
        cudaMemcpy(P->lam_i, li.data(), m * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(P->lam_j, lj.data(), m * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) {
        dst_plan_destroy(P);
        return CNV_CUDA_ERROR;
    }
    return CNV_OK;
}

void dst_plan_destroy(DstPlan* P) {
    cudaFree(P->arena);
    cudaFree(P->S);
    cudaFree(P->t1);
    cudaFree(P->t2);
    cudaFree(P->lam_i);
    cudaFree(P->lam_j);
    *P = DstPlan{};
}

cudaError_t dst_reset(const DstPlan& P, cudaStream_t s) {
    return P.one_launch ? cudaMemsetAsync(P.F.ctl + 2, 0, 8, s) : cudaSuccess;
}

cudaError_t dst_solve(const DstPlan& P, const double* in, double scale, double* out, cudaStream_t s) {
    return solve(P, in, scale, DstDest{out, P.n, nullptr, nullptr, 0}, s);
}

cudaError_t dst_solve_split(const DstPlan& P, const double* in, double scale, double* red, double* black, int pitch,
                            cudaStream_t s) {
    return solve(P, in, scale, DstDest{nullptr, 0, red, black, pitch}, s);
}

}  // namespace cnv
