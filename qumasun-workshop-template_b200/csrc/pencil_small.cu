// The lowest n eigenpairs of a small Hermitian / symmetric definite pencil
// A c = lambda B c (the Rayleigh-Ritz step of the FP64 solvers), one launch of
// one CTA, everything in its shared memory.
//
// Why: a library solve of a 48 x 48 real or 72 x 72 complex pencil is some
// hundred small launches (reduction, tridiagonalisation, divide and conquer,
// back-transformations with one launch per reflector): 0.5 and 1.1 ms, most of a
// solver iteration at 32^3 x 16 bands or 48^3 x 24 complex bands, for less than
// a million operations.  Here it is a chain of ~5 m block barriers, bound by the
// latency of dependent FP64 operations: 0.24 and 0.62 ms.
//
//   1. B = L L^H, right-looking, one barrier per column; the same step applies
//      L^-1 to A from the left (column scales are applied once at the end).
//   2. A <- A L^-H from the right, lower part, one barrier per column.
//   3. Householder tridiagonalisation A = Q T Q^H (LAPACK's ?hetd2 in the lower
//      form): matrix-vector products a warp per row, rank-2 updates.
//   4. The lowest n eigenvalues of T by multisection on Sturm counts, several lanes to an
//      eigenvalue (Givens' bisection; Lo, Philippe & Sameh 1987).
//   5. Their eigenvectors by inverse iteration, a thread to an eigenvalue
//      (tridiagonal LU with partial pivoting; Wilkinson 1965, Peters & Wilkinson),
//      from pseudo-random starts, so that a cluster's vectors are independent.
//   6. Orthonormalised together by Cholesky QR, twice where a cluster's vectors are far
//      from orthogonal (separated ones are orthogonal to rounding already; a cluster's
//      span is kept).
//   7. Q and L^-H applied, a warp to a vector, no barriers; the largest component real
//      and positive.
// The eigenvalues have the absolute accuracy eps |T| of any tridiagonal route.
// info: 0; m + k when the leading minor of order k of B is not positive (the
// library's convention); -1 when step 6 meets dependent vectors: the caller
// then takes the library's solver.
#include "qsb_internal.h"

#include <algorithm>

namespace qsb {
namespace {

constexpr int PS_THREADS = 512;
constexpr int PS_WARPS = PS_THREADS / 32;
constexpr int PS_MAX_ROWS = 4;    // most entries of a vector per lane: m <= 128

template <bool CPLX>
struct Num;
template <>
struct Num<false> {
    using S = double;
};
template <>
struct Num<true> {
    using S = double2;
};
__device__ __forceinline__ double re(double a) { return a; }
__device__ __forceinline__ double re(double2 a) { return a.x; }
__device__ __forceinline__ double im(double) { return 0.0; }
__device__ __forceinline__ double im(double2 a) { return a.y; }
__device__ __forceinline__ double abs2(double a) { return a * a; }
__device__ __forceinline__ double abs2(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double cj(double a) { return a; }
__device__ __forceinline__ double2 cj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 mul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double scl(double a, double s) { return a * s; }
__device__ __forceinline__ double2 scl(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
template <typename S>
__device__ __forceinline__ S mk(double r, double i);
template <>
__device__ __forceinline__ double mk<double>(double r, double) { return r; }
template <>
__device__ __forceinline__ double2 mk<double2>(double r, double i) { return make_double2(r, i); }
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double2 warp_sum(double2 v) { return make_double2(warp_sum(v.x), warp_sum(v.y)); }
__device__ __forceinline__ double bcast(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ double2 bcast(double2 v, int lane) {
    return make_double2(bcast(v.x, lane), bcast(v.y, lane));
}

// M[i, c] -= f(c) for c = c0, c0 + PS_WARPS, ... < c1: the loads of four columns before the
// first use (the compiler cannot move them past the stores to M)
template <typename S, typename F>
__device__ __forceinline__ void columns(S* M, int ld, int i, int c0, int c1, F f) {
    for (int c = c0; c < c1; c += 4 * PS_WARPS) {
        S v[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c + u * PS_WARPS < c1) {
                v[u] = M[i + ld * (c + u * PS_WARPS)];
                g[u] = f(c + u * PS_WARPS);
            }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c + u * PS_WARPS < c1) M[i + ld * (c + u * PS_WARPS)] = sub(v[u], g[u]);
    }
}

// shared memory in doubles: A, then B (later the LU factors, later L^H), then Z and vectors
struct PsLayout {
    int ld, a, b, z, vec, total;
    __host__ __device__ PsLayout(int m, int n, bool cplx) {
        const int c = cplx ? 2 : 1;
        ld = m | 1;                          // odd pitch: rows and columns both free of bank conflicts
        a = 0;
        b = ld * m * c;
        const int bsz = ld * m * c, lu = 5 * m * n;
        z = b + (bsz > lu ? bsz : lu);
        z += z & 1;
        vec = z + m * n + n * n;             // Z [m][n], Gram [n][n]
        vec += vec & 1;
        total = vec + 2 * m /* d, e */ + m /* r */ + 2 * n /* lambda, shifted */ + 3 * 2 * m /* tau, v, p */ + 8;
    }
};

// PS_ROWS: entries of a vector per lane, m <= 32 PS_ROWS
template <bool CPLX, int PS_ROWS>
__global__ void __launch_bounds__(PS_THREADS, 1)
pencil_small_kernel(int m, int n, void* Sa_, void* Sb_, double* __restrict__ W, int* __restrict__ info) {
    using S = typename Num<CPLX>::S;
    extern __shared__ __align__(16) double ps_sm[];
    const PsLayout ly(m, n, CPLX);
    const int ld = ly.ld;
    S* A = reinterpret_cast<S*>(ps_sm + ly.a);
    S* B = reinterpret_cast<S*>(ps_sm + ly.b);
    double* LU = ps_sm + ly.b;
    double* Z = ps_sm + ly.z;
    double* G = Z + m * n;
    double* d = ps_sm + ly.vec;
    double* e = d + m;
    double* r = e + m;
    double* lam = r + m;
    double* lam2 = lam + n;
    S* tau = reinterpret_cast<S*>(ps_sm + ((ly.vec + 3 * m + 2 * n + 1) & ~1));
    S* vv = tau + m;
    S* pp = vv + m;
    __shared__ int fail;
    S* Sa = static_cast<S*>(Sa_);
    S* Sb = static_cast<S*>(Sb_);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;

    for (int j = warp; j < m; j += PS_WARPS)
        for (int i = lane; i < m; i += 32) {
            A[i + ld * j] = Sa[i + (size_t)m * j];
            B[i + ld * j] = Sb[i + (size_t)m * j];
        }
    if (t == 0) fail = 0;
    __syncthreads();

    // 1. B = L L^H (unscaled columns: L_ik = B_ik r_k, r_k = 1 / sqrt(B_kk)), A <- L^-1 A
    for (int k = 0; k < m; ++k) {
        const double bkk = re(B[k + ld * k]);
        if (!(bkk > 0.0) || !isfinite(bkk)) {
            if (t == 0) *info = m + k + 1;
            return;
        }
        const double inv = 1.0 / bkk;
        if (t == 0) r[k] = 1.0 / sqrt(bkk);
        for (int i = k + 1 + lane; i < m; i += 32) {
            const S bik = scl(B[i + ld * k], inv);
            columns<S>(A, ld, i, warp, m, [&](int c) { return mul(bik, A[k + ld * c]); });
            columns<S>(B, ld, i, k + 1 + warp, i + 1, [&](int j) { return mul(bik, cj(B[j + ld * k])); });
        }
        __syncthreads();
    }
    for (int j = warp; j < m; j += PS_WARPS)
        for (int i = lane; i < m; i += 32) A[i + ld * j] = scl(A[i + ld * j], r[i]);
    __syncthreads();
    // 2. A <- A L^-H, lower part
    for (int k = 0; k < m; ++k) {
        const double inv = r[k] * r[k];
        for (int i = k + 1 + lane; i < m; i += 32) {
            const S aik = scl(A[i + ld * k], inv);
            columns<S>(A, ld, i, k + 1 + warp, i + 1, [&](int j) { return mul(aik, cj(B[j + ld * k])); });
        }
        __syncthreads();
    }
    // L^H to Sb (column k: conj L_ki, i <= k), A scaled and mirrored
    for (int k = warp; k < m; k += PS_WARPS)
        for (int i = lane; i < m; i += 32) {
            if (i <= k) Sb[i + (size_t)m * k] = scl(cj(B[k + ld * i]), r[i]);
            if (i >= k) {
                S v = scl(A[i + ld * k], r[k]);
                if (i == k) v = mk<S>(re(v), 0.0);
                A[i + ld * k] = v;
                if (i > k) A[k + ld * i] = cj(v);
            }
        }
    __syncthreads();

    // 3. Q^H A Q = T; column k keeps the reflector v (v_{k+1} = 1)
    const int kend = CPLX ? m - 1 : m - 2;
    for (int k = 0; k < kend; ++k) {
        // every warp for itself: the reflector's scalars
        double s2 = 0.0;
        for (int i = k + 2 + lane; i < m; i += 32) s2 += abs2(A[i + ld * k]);
        s2 = warp_sum(s2);
        const S alpha = A[k + 1 + ld * k];
        S tk = mk<S>(0.0, 0.0), fac = mk<S>(0.0, 0.0);
        double beta = re(alpha);
        const bool flat = s2 == 0.0 && im(alpha) == 0.0;
        if (!flat) {
            beta = -copysign(sqrt(abs2(alpha) + s2), re(alpha));
            tk = mk<S>((beta - re(alpha)) / beta, -im(alpha) / beta);
            const S den = sub(alpha, mk<S>(beta, 0.0));
            fac = scl(cj(den), 1.0 / abs2(den));         // 1 / (alpha - beta)
        }
        if (warp == 0) {
            for (int i = k + 1 + lane; i < m; i += 32)
                vv[i] = i == k + 1 ? mk<S>(1.0, 0.0) : mul(A[i + ld * k], fac);
            if (lane == 0) {
                e[k] = beta;
                tau[k] = tk;
            }
        }
        __syncthreads();
        // p = tau A v: row i is the conjugate of column i
        for (int i0 = k + 1 + warp; i0 < m; i0 += 4 * PS_WARPS) {     // four rows at a time: their sums overlap
            S s[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] = mk<S>(0.0, 0.0);
            for (int j = k + 1 + lane; j < m; j += 32) {
                const S vj = vv[j];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i0 + u * PS_WARPS < m) s[u] = add(s[u], mul(cj(A[j + ld * (i0 + u * PS_WARPS)]), vj));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * PS_WARPS < m) {
                    s[u] = warp_sum(s[u]);
                    if (lane == 0) pp[i0 + u * PS_WARPS] = mul(tk, s[u]);
                }
        }
        if (warp == PS_WARPS - 1)
            for (int i = k + 1 + lane; i < m; i += 32) A[i + ld * k] = vv[i];
        __syncthreads();
        if (!flat) {
            // w = p - tau/2 (p^H v) v;  A -= v w^H + w v^H
            S dot = mk<S>(0.0, 0.0);
            for (int i = k + 1 + lane; i < m; i += 32) dot = add(dot, mul(cj(pp[i]), vv[i]));
            const S al = scl(mul(tk, warp_sum(dot)), -0.5);
            for (int i = k + 1 + lane; i < m; i += 32) {
                const S vi = vv[i], wi = add(pp[i], mul(al, vi));
                columns<S>(A, ld, i, k + 1 + warp, m, [&](int j) {
                    return add(mul(vi, cj(add(pp[j], mul(al, vv[j])))), mul(wi, cj(vv[j])));
                });
            }
        }
        __syncthreads();
    }
    for (int i = t; i < m; i += PS_THREADS) d[i] = re(A[i + ld * i]);
    if (!CPLX && t == 0 && m > 1) e[m - 2] = re(A[m - 1 + ld * (m - 2)]);
    __syncthreads();

    // 4. lowest n eigenvalues: G lanes per eigenvalue, each a Sturm count of one point
    double lo = d[0], hi = d[0], tn = 0.0;
    for (int i = lane; i < m; i += 32) {
        const double off = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < m ? fabs(e[i]) : 0.0);
        lo = fmin(lo, d[i] - off);
        hi = fmax(hi, d[i] + off);
        tn = fmax(tn, fabs(d[i]) + off);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
    }
    if (!isfinite(tn)) {
        if (t == 0) *info = -1;
        return;
    }
    const double eps = 2.220446049250313e-16;
    lo -= 2.0 * eps * tn + 1e-290;
    hi += 2.0 * eps * tn + 1e-290;
    // r2: d_i / |T| and e_{i-1}^2 / |T|^2 interleaved (the reflector scratch is free)
    const double itn = tn > 0.0 ? 1.0 / tn : 1.0;
    double* r2 = reinterpret_cast<double*>(vv);
    for (int i = t; i < m; i += PS_THREADS) {
        r2[2 * i] = d[i] * itn;
        if (i > 0) r2[2 * i - 1] = (e[i - 1] * itn) * (e[i - 1] * itn);
    }
    __syncthreads();
    {
        int lanes = 32, bits = 5;
        while (lanes > 1 && n * lanes > PS_THREADS) {
            lanes >>= 1;
            --bits;
        }
        const int step = PS_THREADS / lanes, l = t & (lanes - 1);
        for (int j0 = 0; j0 < n; j0 += step) {
            const int j = min(j0 + t / lanes, n - 1);      // idle groups repeat the last one
            double a = lo, b = hi;
            for (int pass = 0; pass < 1 + 58 / max(bits, 1); ++pass) {
                const double x = a + (b - a) * ((double)(l + 1) / (double)(lanes + 1));
                // sign changes of the leading minors p_i (one dependent FMA each where the
                // quotient form has a division), scaled by |T|, their size reset every 8
                const double xs = x * itn;
                // (signs and the zero test on the bits: the FP64 pipe's compares are as long as its FMA)
                double p0 = 1.0, p1 = r2[0] - xs;
                if (p1 == 0.0) p1 = -1e-200;
                int neg = (unsigned)__double2hiint(p1) >> 31;
                for (int i0 = 1; i0 < m; i0 += 8) {
                    double a8[8], b8[8];                   // off the chain
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int i = min(i0 + u, m - 1);
                        a8[u] = r2[2 * i] - xs;
                        b8[u] = r2[2 * i - 1];
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if (i0 + u >= m) break;
                        double p2 = fma(a8[u], p1, -(b8[u] * p0));
                        const int h1 = __double2hiint(p1), h2 = __double2hiint(p2);
                        if (((h2 & 0x7fffffff) | __double2loint(p2)) == 0)
                            p2 = __hiloint2double(0x16687e92 | (~h1 & 0x80000000), 0);   // 1e-200, the other sign
                        neg += (unsigned)(__double2hiint(p2) ^ h1) >> 31;
                        p0 = p1;
                        p1 = p2;
                    }
                    const double big = fmax(fabs(p0), fabs(p1));
                    const double f =
                        __longlong_as_double((0x7fdLL << 52) - (__double_as_longlong(big) & (0x7ffLL << 52)));
                    p0 *= f;
                    p1 *= f;
                }
                // first point with more than j eigenvalues below it
                const unsigned hit = __ballot_sync(0xffffffffu, neg > j) >> ((t & 31) & ~(lanes - 1));
                const unsigned mask = lanes == 32 ? 0xffffffffu : (1u << lanes) - 1u;
                const int f = (hit & mask) ? __ffs(hit & mask) - 1 : lanes;
                const double na = a + (b - a) * ((double)f / (double)(lanes + 1));
                const double nb = f == lanes ? b : a + (b - a) * ((double)(f + 1) / (double)(lanes + 1));
                a = na;
                b = nb;
            }
            if (l == 0 && j0 + t / lanes < n) lam[j] = 0.5 * (a + b);
        }
    }
    __syncthreads();
    // shifts of a cluster pushed apart (a few rounding errors of |T|), so that their factors differ
    if (t == 0) {
        double last = -1e300;
        for (int j = 0; j < n; ++j) {
            double x = lam[j];
            if (x - last < 4.0 * eps * tn) x = last + 4.0 * eps * tn;
            lam2[j] = x;
            last = x;
        }
    }
    __syncthreads();
    // 5. inverse iteration: thread j factors T - lambda_j (dl, d, du, du2 and the row swaps, [i][n])
    if (t < n) {
        double *l0 = LU + t, *u0 = l0 + m * n, *u1 = u0 + m * n, *u2 = u1 + m * n, *sw = u2 + m * n;
        const double x = lam2[t], small = eps * tn;
        double di = d[0] - x, ui = m > 1 ? e[0] : 0.0;
        for (int i = 0; i + 1 < m; ++i) {
            const double li = e[i], dn = d[i + 1] - x, un = i + 2 < m ? e[i + 1] : 0.0;
            if (fabs(di) >= fabs(li)) {
                if (fabs(di) < small) di = copysign(small, di);
                const double f = li / di;
                l0[i * n] = f;
                u0[i * n] = 1.0 / di;
                u1[i * n] = ui;
                u2[i * n] = 0.0;
                sw[i * n] = 0.0;
                di = dn - f * ui;
                ui = un;
            } else {
                const double f = di / li;
                l0[i * n] = f;
                u0[i * n] = 1.0 / li;
                u1[i * n] = dn;
                u2[i * n] = un;
                sw[i * n] = 1.0;
                di = ui - f * dn;
                ui = -f * un;
            }
        }
        if (fabs(di) < small) di = copysign(small, di);
        u0[(m - 1) * n] = 1.0 / di;
        double* z = Z + t;
        unsigned seed = 12345u + 7919u * (unsigned)t;
        for (int i = 0; i < m; ++i) {
            seed = seed * 1664525u + 1013904223u;
            z[i * n] = (double)(int)(seed >> 8) * 0x1p-23 - 1.0 + 1e-3;
        }
        for (int it = 0; it < 3; ++it) {
            double y = z[0];
            for (int i = 0; i + 1 < m; ++i) {
                const double yn = z[(i + 1) * n];
                if (sw[i * n] == 0.0) {
                    z[i * n] = y;
                    y = yn - l0[i * n] * y;
                } else {
                    z[i * n] = yn;
                    y = y - l0[i * n] * yn;
                }
            }
            double x1 = y * u0[(m - 1) * n], x2 = 0.0, s2 = x1 * x1;
            z[(m - 1) * n] = x1;
            for (int i = m - 2; i >= 0; --i) {
                const double xi = (z[i * n] - u1[i * n] * x1 - u2[i * n] * x2) * u0[i * n];
                z[i * n] = xi;
                s2 += xi * xi;
                x2 = x1;
                x1 = xi;
            }
            const double sc = 1.0 / sqrt(s2);
            for (int i = 0; i < m; ++i) z[i * n] *= sc;
        }
    }
    __syncthreads();
    // 6. Cholesky QR, twice (row i of Z is Z[i n ..])
    bool again = true;      // a second pass unless the first found them orthogonal to 1e-3
    for (int pass = 0; pass < 2 && again; ++pass) {
        bool skew = false;
        for (int q = t; q < n * n; q += PS_THREADS) {
            const int a = q / n, b = q - a * n;
            if (a < b) continue;
            double s = 0.0;
            for (int i = 0; i < m; ++i) s += Z[i * n + a] * Z[i * n + b];
            G[a * n + b] = s;                              // lower
            skew |= a != b && !(fabs(s) < 1e-3);
        }
        again = __syncthreads_or(skew);
        if (warp == 0) {
            for (int k = 0; k < n; ++k) {
                const double g = G[k * n + k];
                // a unit vector's part outside its predecessors: below 1e-6 they are dependent
                if (!(g > 1e-12)) {
                    if (lane == 0) fail = 1;
                    break;
                }
                const double inv = 1.0 / sqrt(g);
                __syncwarp();
                for (int i = k + lane; i < n; i += 32) G[i * n + k] *= inv;
                __syncwarp();
                for (int i = k + 1 + lane; i < n; i += 32)
                    for (int j = k + 1; j <= i; ++j) G[i * n + j] -= G[i * n + k] * G[j * n + k];
                __syncwarp();
            }
        }
        __syncthreads();
        if (fail) {
            if (t == 0) *info = -1;
            return;
        }
        for (int i = t; i < m; i += PS_THREADS) {          // Z <- Z L^-T, row by row
            double* z = Z + i * n;
            for (int b = 0; b < n; ++b) {
                double s = z[b];
                for (int a = 0; a < b; ++a) s -= z[a] * G[b * n + a];
                z[b] = s / G[b * n + b];
            }
        }
        __syncthreads();
    }
    // L^H back into shared memory
    for (int k = warp; k < m; k += PS_WARPS)
        for (int i = lane; i <= k; i += 32) B[i + ld * k] = Sb[i + (size_t)m * k];
    __syncthreads();
    // 7. c = L^-H Q z, a warp per vector, entries lane + 32 q
    for (int j = warp; j < n; j += PS_WARPS) {
        S x[PS_ROWS];
#pragma unroll
        for (int q = 0; q < PS_ROWS; ++q) x[q] = mk<S>(lane + 32 * q < m ? Z[(lane + 32 * q) * n + j] : 0.0, 0.0);
        for (int k = kend - 1; k >= 0; --k) {
            S a[PS_ROWS], sum = mk<S>(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < PS_ROWS; ++q) {
                const int i = lane + 32 * q;
                a[q] = i > k && i < m ? A[i + ld * k] : mk<S>(0.0, 0.0);
                sum = add(sum, mul(cj(a[q]), x[q]));
            }
            sum = mul(tau[k], warp_sum(sum));
#pragma unroll
            for (int q = 0; q < PS_ROWS; ++q) x[q] = sub(x[q], mul(a[q], sum));
        }
        for (int k = m - 1; k >= 0; --k) {
            S b[PS_ROWS], xk = x[0];
#pragma unroll
            for (int q = 0; q < PS_ROWS; ++q) b[q] = lane + 32 * q < k ? B[lane + 32 * q + ld * k] : mk<S>(0.0, 0.0);
#pragma unroll
            for (int q = 1; q < PS_ROWS; ++q)
                if (k >> 5 == q) xk = x[q];
            xk = scl(bcast(xk, k & 31), r[k]);             // r_k = 1 / L_kk
#pragma unroll
            for (int q = 0; q < PS_ROWS; ++q) {
                if (lane + 32 * q == k) x[q] = xk;
                x[q] = sub(x[q], mul(b[q], xk));
            }
        }
        // the free sign (phase): the largest component positive (real), so that nearly equal
        // pencils give nearly equal vectors whatever the iteration started from
        double big = 0.0;
        S xm = x[0];
#pragma unroll
        for (int q = 0; q < PS_ROWS; ++q)
            if (lane + 32 * q < m && abs2(x[q]) > big) {
                big = abs2(x[q]);
                xm = x[q];
            }
        double top = big;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
        const unsigned owners = __ballot_sync(0xffffffffu, big == top);
        xm = bcast(xm, owners ? __ffs(owners) - 1 : 0);
        const S turn = top > 0.0 ? scl(cj(xm), 1.0 / sqrt(abs2(xm))) : mk<S>(1.0, 0.0);
#pragma unroll
        for (int q = 0; q < PS_ROWS; ++q) {
            const int i = lane + 32 * q;
            if (i < m) Sa[i + (size_t)m * j] = mul(x[q], turn);
        }
    }
    for (int j = t; j < n; j += PS_THREADS) W[j] = lam[j];
    if (t == 0) *info = 0;
}

}  // namespace

// Rows and vectors that fit one CTA's shared memory (m = 3 n: up to 93 real, 78
// complex rows; above that the library's blocked solver)
bool pencil_small_fits(int m, int n, bool cplx) {
    return m >= 2 && m <= 32 * PS_MAX_ROWS && n >= 1 && n <= m &&
           (size_t)PsLayout(m, n, cplx).total * sizeof(double) <= 220 * 1024;
}

qsb_status pencil_small(int m, int n, bool cplx, double* Sa, double* Sb, double* W, int* info, cudaStream_t s) {
    const size_t smem = (size_t)PsLayout(m, n, cplx).total * sizeof(double);
    auto kern = cplx ? (m <= 64 ? pencil_small_kernel<true, 2> : pencil_small_kernel<true, 3>)
                     : (m <= 64 ? pencil_small_kernel<false, 2> : pencil_small_kernel<false, 4>);
    if (cplx && m > 96) return fail(QSB_ERR_INVALID, "pencil_small: too many rows");   // past shared memory as well
    QSB_TRY(allow_shared_memory(kern));
    kern<<<1, PS_THREADS, smem, s>>>(m, n, Sa, Sb, W, info);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

}  // namespace qsb
