// Block LOBPCG eigensolvers on the device.
//
//  qsb_lobpcg_z : LOBPCG::Eigen_z_multi_mpi   (source/lobpcg_z_multi_mpi.h:1732-2852)
//                 complex SoA bands, sqrt(dV) scaling, soft locking of converged
//                 bands (num_fix), P kept across calls, norm-check rollback.
//  qsb_lobpcg_d : EigenLOBPCG_d_multi          (source/lobpcg_d_multi.h:23-545)
//                 real bands, dV-weighted Gram, per-iteration renormalization,
//                 stop at max ||r||^2 < 1e-10 (dV-weighted).
//
// B200 mapping.  All bundles stay in HBM.  Gram blocks are DGEMMs on the
// reference's 2n-real view of the SoA bundle (MakeMatrix_z_blas,
// :300-558) followed by a kernel that assembles the complex block
// (AoSComplexFrom2by2Real, source/matrix_2x2real_to_complex.h:8-28) directly
// into the 2n x 2n / 3n x 3n Hermitian pencil; the pencil is solved on the
// device (cusolverDn ?hegvd, the role of lapack_ZHEGVD_emu / lapack_DSYGVX);
// the rotation X' = X Cx + R Cr + P Cp is the two-DGEMM "conj / rot"
// real-view product of NextVector_z2 (:1515-1598).  Band-wise reductions are
// deterministic two-pass kernels (fixed-order partial sums, no atomics).
// The real FP64 pencil is formed whole, in gram_small.cu (up to 32 bands) or
// gram_i8_f64.cu.  The complex solver recomputes every block on the first and
// every 6th iteration and updates some from the eigenvectors in between
// (NextMatrix_z_blasmp, :2093); the real one recomputes all of them always.
#include "qsb_internal.h"

#include <cublas_v2.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace qsb {
namespace {

constexpr int RED_THREADS = 256;
constexpr int RED_CHUNK = 1 << 16;   // elements per reduction block (mixed precision)

// Elements per reduction block of a context: the FP64 solvers cut a band into up to 32 pieces of
// 4096 or more, so that a few bands of a small grid fill the GPU (16 bands of 32^3: 16 blocks
// of 65536, 14 us a pass, against 128 of 4096, 3 us).  The mixed solver keeps the longer
// ones: its results depend on the order of these sums.
inline int red_chunk_of(size_t L, bool mixed) {
    if (mixed) return RED_CHUNK;
    const size_t piece = ((L + 31) / 32 + 1023) / 1024 * 1024;
    return (int)std::min<size_t>(RED_CHUNK, std::max<size_t>(4096, piece));
}

// partial[s * nch + ch] = sum over chunk ch of segment s of a[i]*b[i]
// (fp64 or fp32 bundles, fp64 sums)
template <typename T>
__global__ void seg_dot_partial(const T* __restrict__ a, const T* __restrict__ b, size_t L, int chunk, int nch,
                                double* __restrict__ partial) {
    const int s = blockIdx.y, ch = blockIdx.x;
    const size_t i0 = (size_t)ch * chunk, i1 = min(L, i0 + chunk);
    const T* A = a + (size_t)s * L;
    const T* B = b + (size_t)s * L;
    double acc = 0.0;
    for (size_t i = i0 + threadIdx.x; i < i1; i += RED_THREADS) acc += (double)A[i] * (double)B[i];
    __shared__ double red[RED_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < RED_THREADS / 32; ++w) t += red[w];
        partial[(size_t)s * nch + ch] = t;
    }
}

// r = ax - eps[s]*x; partial sums of r^2 (if partial != nullptr)
template <typename T>
__global__ void seg_residual_partial(T* __restrict__ r, const T* __restrict__ ax, const T* __restrict__ x,
                                     const double* __restrict__ eps, size_t L, int chunk, int nch,
                                     double* __restrict__ partial) {
    const int s = blockIdx.y, ch = blockIdx.x;
    const size_t i0 = (size_t)ch * chunk, i1 = min(L, i0 + chunk);
    const size_t off = (size_t)s * L;
    const double e = eps[s];
    double acc = 0.0;
    for (size_t i = i0 + threadIdx.x; i < i1; i += RED_THREADS) {
        const T v = (T)((double)ax[off + i] - e * (double)x[off + i]);
        r[off + i] = v;
        acc += (double)v * (double)v;
    }
    if (!partial) return;
    __shared__ double red[RED_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < RED_THREADS / 32; ++w) t += red[w];
        partial[(size_t)s * nch + ch] = t;
    }
}

__global__ void seg_finalize(const double* __restrict__ partial, int nseg, int nch, double scale,
                             double* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    double t = 0.0;
    for (int c = 0; c < nch; ++c) t += partial[(size_t)s * nch + c];
    out[s] = t * scale;
}

// sums as seg_finalize, and their inverse square roots (1 where the sum is not finite: the
// band stays as it is and the host refuses the call by the sum)
__global__ void seg_finalize_rsqrt(const double* __restrict__ partial, int nseg, int nch, double scale,
                                   double* __restrict__ out, double* __restrict__ inv) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    double t = 0.0;
    for (int c = 0; c < nch; ++c) t += partial[(size_t)s * nch + c];
    out[s] = t * scale;
    inv[s] = isfinite(t * scale) ? 1.0 / sqrt(t * scale) : 1.0;
}

// out[s] = in[s] * scale[s] and, with partial, partial sums of out[s] * y[s] in
// seg_dot_partial's order: the copy, the scaling and the inner product of a
// rotated bundle in one pass (three took 9 bytes moved per byte of it, this 3).
template <bool DOT>
__global__ void seg_scale_to(const double* __restrict__ in, double* __restrict__ out, const double* __restrict__ scale,
                             const double* __restrict__ y, size_t L, int chunk, int nch,
                             double* __restrict__ partial) {
    const int s = blockIdx.y, ch = blockIdx.x;
    const size_t i0 = (size_t)ch * chunk, i1 = min(L, i0 + chunk);
    const size_t off = (size_t)s * L;
    const double c = scale[s];
    double acc = 0.0;
#pragma unroll 4
    for (size_t i = i0 + threadIdx.x; i < i1; i += RED_THREADS) {
        const double v = in[off + i] * c;
        out[off + i] = v;
        if (DOT) acc += v * y[off + i];
    }
    if constexpr (DOT) {
        __shared__ double red[RED_THREADS / 32];
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < RED_THREADS / 32; ++w) t += red[w];
            partial[(size_t)s * nch + ch] = t;
        }
    }
}

// x[s] *= scale[s]  (or a single scalar when scale == nullptr)
template <typename T>
__global__ void seg_scale(T* __restrict__ x, size_t L, const double* __restrict__ scale, double scalar) {
    const int s = blockIdx.y;
    const double c = scale ? scale[s] : scalar;
    T* X = x + (size_t)s * L;
    const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    constexpr int V = 16 / sizeof(T);
    size_t done = 0;
    // 16-byte accesses, four in flight per thread: 96^3 x 128 FP32 250 -> 137 us (one element
    // per access read and wrote at 3.6 TB/s)
    if (((uintptr_t)X & 15) == 0) {
        struct alignas(16) Vec { T v[V]; };
        Vec* Xv = reinterpret_cast<Vec*>(X);
        const size_t n = L / V;
        done = n * V;
        auto scaled = [c](Vec q) {
#pragma unroll
            for (int j = 0; j < V; ++j) q.v[j] = (T)((double)q.v[j] * c);
            return q;
        };
        size_t i = t0;
        for (; i + 3 * step < n; i += 4 * step) {
            Vec q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = Xv[i + k * step];
#pragma unroll
            for (int k = 0; k < 4; ++k) Xv[i + k * step] = scaled(q[k]);
        }
        for (; i < n; i += step) Xv[i] = scaled(Xv[i]);
    }
    for (size_t i = done + t0; i < L; i += step) X[i] = (T)((double)X[i] * c);
}

// out[s] = in[s] * scale[s] (or scalar) with a type change (fp64 <-> fp32 bundles)
template <typename Ti, typename To>
__global__ void seg_convert(const Ti* __restrict__ in, To* __restrict__ out, size_t L, const double* __restrict__ scale,
                            double scalar) {
    const int s = blockIdx.y;
    const double c = scale ? scale[s] : scalar;
    const Ti* I = in + (size_t)s * L;
    To* O = out + (size_t)s * L;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < L; i += (size_t)gridDim.x * blockDim.x)
        O[i] = (To)((double)I[i] * c);
}

// small matrices: out[i] = (float)in[i]
__global__ void to_f32(const double* __restrict__ in, float* __restrict__ out, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

// Complex block from the 2n x 2n real Gram T (column-major, ld 2na x ...):
// M[(I0+a) + m (J0+b)] = T[2a,2b] + T[2a+1,2b+1] + i (T[2a,2b+1] - T[2a+1,2b])
// (AoSComplexFrom2by2Real); lower triangle of M gets the conjugate.
// diag: the block is on the diagonal (only a <= b written from T).
__global__ void assemble_complex_block(const double* __restrict__ T, int na, int nb_, int ldt, double2* __restrict__ M,
                                       int m, int I0, int J0, int diag) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (a >= na || b >= nb_) return;
    if (diag && a > b) return;
    const double re = T[(2 * a) + (size_t)ldt * (2 * b)] + T[(2 * a + 1) + (size_t)ldt * (2 * b + 1)];
    const double im = T[(2 * a) + (size_t)ldt * (2 * b + 1)] - T[(2 * a + 1) + (size_t)ldt * (2 * b)];
    const int r = I0 + a, c = J0 + b;
    M[r + (size_t)m * c] = make_double2(re, (diag && a == b) ? 0.0 : im);
    M[c + (size_t)m * r] = make_double2(re, (diag && a == b) ? 0.0 : -im);
}

// Real block: M[(I0+a) + m (J0+b)] = T[a,b] (upper, a<=b on the diagonal) and its mirror.
__global__ void assemble_real_block(const double* __restrict__ T, int na, int nb_, int ldt, double* __restrict__ M,
                                    int m, int I0, int J0, int diag, double scale) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (a >= na || b >= nb_) return;
    if (diag && a > b) return;
    const double v = T[a + (size_t)ldt * b] * scale;
    M[(I0 + a) + (size_t)m * (J0 + b)] = v;
    M[(J0 + b) + (size_t)m * (I0 + a)] = v;
}

// NextVector_z2's coefficient views: for block B (rows B0..B0+na of the m x N
// complex eigenvector matrix C), cnj[2j,k] = Re C, cnj[2j+1,k] = -Im C,
// rot[2j,k] = Im C, rot[2j+1,k] = Re C   (ld 2*na).
__global__ void make_rot_cnj(const double2* __restrict__ C, int m, int B0, int na, int ncol, double* __restrict__ cnj,
                             double* __restrict__ rot) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (j >= na || k >= ncol) return;
    const double2 c = C[(B0 + j) + (size_t)m * k];
    cnj[2 * j + (size_t)2 * na * k] = c.x;
    cnj[2 * j + 1 + (size_t)2 * na * k] = -c.y;
    rot[2 * j + (size_t)2 * na * k] = c.y;
    rot[2 * j + 1 + (size_t)2 * na * k] = c.x;
}

// real eigenvector block copy: out[j + na*k] = C[B0+j + m*k]
__global__ void copy_real_block(const double* __restrict__ C, int m, int B0, int na, int ncol, double* __restrict__ out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (j >= na || k >= ncol) return;
    out[j + (size_t)na * k] = C[(B0 + j) + (size_t)m * k];
}

// VectorOrthogonalization's packed real matrix from the complex X_fix^H X_act
// built with the 2x2 rule, in place on T (2f x 2a, ld 2f).
__global__ void pack_orth(double* __restrict__ T, int nf, int na) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (j >= nf || k >= na) return;
    const int ld = 2 * nf;
    const double re = T[(2 * j) + (size_t)ld * (2 * k)] + T[(2 * j + 1) + (size_t)ld * (2 * k + 1)];
    const double im = -T[(2 * j + 1) + (size_t)ld * (2 * k)] + T[(2 * j) + (size_t)ld * (2 * k + 1)];
    T[(2 * j) + (size_t)ld * (2 * k)] = re;
    T[(2 * j + 1) + (size_t)ld * (2 * k + 1)] = re;
    T[(2 * j) + (size_t)ld * (2 * k + 1)] = im;
    T[(2 * j + 1) + (size_t)ld * (2 * k)] = -im;
}

// One n x n block (I0, J0) of the full Hermitian pencil M (ld m) from the dense
// complex matrix B (ld n): value = B, minus Bs[a,b] E[b] (mode 1) or E[a] Bs[a,b]
// (mode 2).  On a diagonal block only a <= b is read and the diagonal's imaginary
// part is dropped; the mirrored position gets the conjugate.
__global__ void put_pencil_block(const double2* __restrict__ B, const double2* __restrict__ Bs,
                                 const double* __restrict__ E, int mode, int n, double2* __restrict__ M, int m, int I0,
                                 int J0, int diag) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (a >= n || b >= n) return;
    if (diag && a > b) return;
    double2 v = B[a + (size_t)n * b];
    if (mode != 0) {
        const double2 w = Bs[a + (size_t)n * b];
        const double e = mode == 1 ? E[b] : E[a];
        v.x -= w.x * e;
        v.y -= w.y * e;
    }
    if (diag && a == b) v.y = 0.0;
    const int r = I0 + a, c = J0 + b;
    M[r + (size_t)m * c] = v;
    M[c + (size_t)m * r] = make_double2(v.x, -v.y);
}

const char* cublas_name(cublasStatus_t s) {
    switch (s) {
    case CUBLAS_STATUS_SUCCESS: return "CUBLAS_STATUS_SUCCESS";
    case CUBLAS_STATUS_NOT_INITIALIZED: return "CUBLAS_STATUS_NOT_INITIALIZED";
    case CUBLAS_STATUS_ALLOC_FAILED: return "CUBLAS_STATUS_ALLOC_FAILED";
    case CUBLAS_STATUS_INVALID_VALUE: return "CUBLAS_STATUS_INVALID_VALUE";
    case CUBLAS_STATUS_EXECUTION_FAILED: return "CUBLAS_STATUS_EXECUTION_FAILED";
    default: return "cublas error";
    }
}

#define QSB_BLAS_TRY(expr)                                                                              \
    do {                                                                                                \
        cublasStatus_t st_ = (expr);                                                                    \
        if (st_ != CUBLAS_STATUS_SUCCESS) return fail(QSB_ERR_CUDA, std::string(#expr) + ": " + cublas_name(st_)); \
    } while (0)
#define QSB_SOLVER_TRY(expr)                                                                            \
    do {                                                                                                \
        cusolverStatus_t st_ = (expr);                                                                  \
        if (st_ != CUSOLVER_STATUS_SUCCESS)                                                             \
            return fail(QSB_ERR_CUDA, std::string(#expr) + ": cusolver status " + std::to_string((int)st_)); \
    } while (0)

}  // namespace
}  // namespace qsb

using namespace qsb;

struct qsb_eigensolver {
    int64_t N = 0;       // grid points per band
    int nmax = 0;        // bands
    int cplx = 0;
    size_t L = 0;        // doubles per band (N or 2N)
    cublasHandle_t blas = nullptr;
    cusolverDnHandle_t sol = nullptr;
    double *R = nullptr, *AX = nullptr, *AR = nullptr, *AP = nullptr, *TMP = nullptr;
    double* T = nullptr;             // real Gram scratch, up to (2*3n)^2
    double* Sa = nullptr;            // pencil A (complex: m*m double2; real: m*m)
    double* Sb = nullptr;            // pencil B
    double* W = nullptr;             // eigenvalues (m)
    double* rc = nullptr;            // rotation coefficient views, 6 x (2n x n)
    double* vec = nullptr;           // small per-band vectors (eps, norms, scales): 8 x nmax
    double* partial = nullptr;       // reduction partials: nmax x nch
    double* gsmall = nullptr;        // tiles of the small real pencil (gram_small), few bands only
    void* gi8 = nullptr;             // workspace of the large real pencil (gram_f64_i8): TMP, or gi8_own
    void* gi8_own = nullptr;         // where TMP is too small for it (few points)
    size_t gi8_bytes = 0;
    int nch = 0, chunk = 0;          // pieces of a band in the reductions, elements per piece
    void* swork = nullptr;
    int slwork = 0;
    int* info = nullptr;             // [0] of the dense solves, [1] of the pencil's products and its look-over
    // operator
    qsb_ham* ham = nullptr;
    double g[3] = {0, 0, 0};
    qsb_apply_fn op = nullptr;
    void* user = nullptr;
    // statistics of the last call
    int last_iters = 0;
    int last_rollback = 0;
    // mixed precision (QSB_PREC_MIXED): fp32 bundles, split-BF16x3 tensor-core
    // Gram products, fp64 pencil / norms; the fp64 bundles above stay unallocated
    int mixed = 0;
    float *X32 = nullptr, *R32 = nullptr, *P32 = nullptr, *AX32 = nullptr, *AR32 = nullptr, *AP32 = nullptr,
          *TMP32 = nullptr;
    void* su = nullptr;      // bf16 hi/lo split of the basis [X R P] (active bands)
    void* sau = nullptr;     // split of [AX AR AP]
    size_t split_bytes = 0;
    void* gpart = nullptr;   // split-K partial tiles of the Gram products
    size_t gpart_bytes = 0;
    double* T2 = nullptr;    // full-pencil real Gram (up to (2*3n)^2)
    float* rc32 = nullptr;   // fp32 copies of the rotation coefficients / orthogonalization matrix
    double* svq = nullptr;   // overlap-basis pencil solve: W, scratch, reduced matrix (m x m each), lambda, d
    double* rotw = nullptr;  // tensor-core rotations: saved overlap, rotation coefficients, their overlap product, norms
    void* rotc = nullptr;    // int8 slices of the rotation coefficients
    size_t rotc_bytes = 0;
    double drop_tol = 0.0;   // overlap eigenvalues below drop_tol * max are dropped
    int gram_kind = QSB_GRAM_INT8_OZAKI;   // Gram products: BF16x3, BF16x4 or INT8 Ozaki
    int last_chol = 0;       // pencil solves of the last call by Cholesky (?hegvd on the scaled pencil)
    int last_svqb = 0;       // ... and by the overlap-basis fallback
    int last_dropped = 0;    // most directions dropped in one iteration of the last call
    double last_min_kept = 1.0;   // smallest kept overlap eigenvalue / max in the last call
    qsb_apply_f32_fn op32 = nullptr;
    void* user32 = nullptr;
    // steady-state pencil update of the FP64 complex solver (NextMatrix_z): the
    // previous pencil (S0a, S0b, m x m each), the X'/P' blocks it gives (6 x n x n)
    // and two m x n products, complex
    double* nxt = nullptr;
    int pencil_update = 1;   // 1: X/P blocks from the previous pencil between full recomputes; 0: all from the grid
    int last_full = 0;       // pencils of the last call formed from the grid in full ...
    int last_steady = 0;     // ... and with only the R blocks from the grid
};

namespace qsb {
namespace {

qsb_status apply_op(qsb_eigensolver* es, int nb, const double* x, double* ax, cudaStream_t s) {
    if (nb <= 0) return QSB_OK;
    if (es->ham) return qsb_ham_apply(es->ham, QSB_F64, es->cplx, nb, x, ax, es->g[0], es->g[1], es->g[2], s);
    const int st = es->op(es->user, nb, x, ax, (void*)s);
    if (st != 0) return fail((qsb_status)(st > 0 && st <= 6 ? st : QSB_ERR_STATE), "eigensolver: operator callback failed");
    return QSB_OK;
}

qsb_status apply_op32(qsb_eigensolver* es, int nb, const float* x, float* ax, cudaStream_t s) {
    if (nb <= 0) return QSB_OK;
    if (es->ham) return qsb_ham_apply(es->ham, QSB_F32, es->cplx, nb, x, ax, es->g[0], es->g[1], es->g[2], s);
    if (!es->op32)
        return fail(QSB_ERR_STATE, "eigensolver: mixed precision needs the built-in Hamiltonian or an fp32 operator");
    const int st = es->op32(es->user32, nb, x, ax, (void*)s);
    if (st != 0) return fail((qsb_status)(st > 0 && st <= 6 ? st : QSB_ERR_STATE), "eigensolver: operator callback failed");
    return QSB_OK;
}

template <typename Ti, typename To>
qsb_status seg_convert_by(qsb_eigensolver* es, int nseg, const Ti* in, To* out, const double* scale_dev, double scalar,
                          cudaStream_t s) {
    if (nseg <= 0) return QSB_OK;
    const int bx = (int)std::min<size_t>((es->L + 255) / 256, 512);
    seg_convert<Ti, To><<<dim3(bx, nseg), 256, 0, s>>>(in, out, es->L, scale_dev, scalar);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// out[s] = scale * sum(a_s * b_s) over nseg segments of L values (device out)
template <typename T>
qsb_status seg_dot(qsb_eigensolver* es, int nseg, const T* a, const T* b, double scale, double* out, cudaStream_t s) {
    if (nseg <= 0) return QSB_OK;
    const int nch = es->nch;
    seg_dot_partial<<<dim3(nch, nseg), RED_THREADS, 0, s>>>(a, b, es->L, es->chunk, nch, es->partial);
    seg_finalize<<<(nseg + 127) / 128, 128, 0, s>>>(es->partial, nseg, nch, scale, out);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// norms[s] = scale * sum(a_s^2), inv[s] = 1 / sqrt(norms[s]) (device vectors)
qsb_status seg_norms(qsb_eigensolver* es, int nseg, const double* a, double scale, double* norms, double* inv,
                     cudaStream_t s) {
    if (nseg <= 0) return QSB_OK;
    const int nch = es->nch;
    seg_dot_partial<<<dim3(nch, nseg), RED_THREADS, 0, s>>>(a, a, es->L, es->chunk, nch, es->partial);
    seg_finalize_rsqrt<<<(nseg + 127) / 128, 128, 0, s>>>(es->partial, nseg, nch, scale, norms, inv);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// out_s = in_s * f[s]; with y: dot[s] = scale * sum(out_s * y_s)
qsb_status seg_scaled_copy(qsb_eigensolver* es, int nseg, const double* in, double* out, const double* f,
                           const double* y, double scale, double* dot, cudaStream_t s) {
    if (nseg <= 0) return QSB_OK;
    const int nch = es->nch;
    if (y) {
        seg_scale_to<true><<<dim3(nch, nseg), RED_THREADS, 0, s>>>(in, out, f, y, es->L, es->chunk, nch, es->partial);
        seg_finalize<<<(nseg + 127) / 128, 128, 0, s>>>(es->partial, nseg, nch, scale, dot);
    } else {
        seg_scale_to<false><<<dim3(nch, nseg), RED_THREADS, 0, s>>>(in, out, f, nullptr, es->L, es->chunk, nch, nullptr);
    }
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

template <typename T>
qsb_status seg_residual(qsb_eigensolver* es, int nseg, T* r, const T* ax, const T* x, const double* eps,
                        double* norms, double scale, cudaStream_t s) {
    if (nseg <= 0) return QSB_OK;
    const int nch = es->nch;
    seg_residual_partial<<<dim3(nch, nseg), RED_THREADS, 0, s>>>(r, ax, x, eps, es->L, es->chunk, nch,
                                                                 norms ? es->partial : nullptr);
    if (norms) seg_finalize<<<(nseg + 127) / 128, 128, 0, s>>>(es->partial, nseg, nch, scale, norms);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

template <typename T>
qsb_status seg_scale_by(qsb_eigensolver* es, int nseg, T* x, const double* scale_dev, double scalar, cudaStream_t s) {
    if (nseg <= 0) return QSB_OK;
    const int bx = (int)std::min<size_t>((es->L + 255) / 256, std::max(16, 4736 / nseg));
    seg_scale<<<dim3(bx, nseg), 256, 0, s>>>(x, es->L, scale_dev, scalar);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// T (p x q, ld p) = U^T V over N rows: U is N x p, V is N x q (column-major, ld N)
qsb_status gemm_tn(qsb_eigensolver* es, int p, int q, const double* U, const double* V, double* T) {
    const double one = 1.0, zero = 0.0;
    QSB_BLAS_TRY(cublasDgemm(es->blas, CUBLAS_OP_T, CUBLAS_OP_N, p, q, (int)es->N, &one, U, (int)es->N, V, (int)es->N,
                             &zero, T, p));
    return QSB_OK;
}

// OUT (N x q, ldo) = beta*OUT + alpha * U (N x p, ld N) . C (p x q, ld p)
qsb_status gemm_nn(qsb_eigensolver* es, int p, int q, double alpha, const double* U, const double* C, double beta,
                   double* OUT, int ldo) {
    QSB_BLAS_TRY(cublasDgemm(es->blas, CUBLAS_OP_N, CUBLAS_OP_N, (int)es->N, q, p, &alpha, U, (int)es->N, C, p, &beta,
                             OUT, ldo));
    return QSB_OK;
}

// OUT (N x q, ldo) = beta*OUT + alpha * U (N x p, ld N) . C (p x q, ld p), fp32
qsb_status sgemm_nn(qsb_eigensolver* es, int p, int q, float alpha, const float* U, const float* C, float beta,
                    float* OUT, int ldo) {
    QSB_BLAS_TRY(cublasSgemm(es->blas, CUBLAS_OP_N, CUBLAS_OP_N, (int)es->N, q, p, &alpha, U, (int)es->N, C, p, &beta,
                             OUT, ldo));
    return QSB_OK;
}

// Hermitian (complex) or symmetric (real) pencil block (I, J) from bundles U_I, V_J
// of na bands each.  Complex: 2na real planes per bundle.
qsb_status gram_block(qsb_eigensolver* es, const double* U, const double* V, int na, double* M, int m, int I, int J,
                      double scale, cudaStream_t s) {
    if (es->cplx) {
        QSB_TRY(gemm_tn(es, 2 * na, 2 * na, U, V, es->T));
        dim3 grid((na + 127) / 128, na);
        assemble_complex_block<<<grid, 128, 0, s>>>(es->T, na, na, 2 * na, (double2*)M, m, I * na, J * na, I == J);
    } else {
        QSB_TRY(gemm_tn(es, na, na, U, V, es->T));
        dim3 grid((na + 127) / 128, na);
        assemble_real_block<<<grid, 128, 0, s>>>(es->T, na, na, na, M, m, I * na, J * na, I == J, scale);
    }
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// state |= 1: an entry of the pencil (n doubles each) is not finite, 2: a diagonal entry of
// B (every dstep-th) is not positive (B null: a matrix A alone, looked over for 1)
__global__ void pencil_state(const double* __restrict__ A, const double* __restrict__ B, size_t n, size_t dstep,
                             int* __restrict__ state) {
    int bad = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (!isfinite(A[i])) bad |= 1;
        if (!B) continue;
        if (!isfinite(B[i])) bad |= 1;
        if (i % dstep == 0 && !(B[i] > 0.0)) bad |= 2;
    }
    if (bad) atomicOr(state, bad);
}
// the pencil (diag(1, 2, ...), identity) in place of one with a state
__global__ void pencil_replace(double* __restrict__ A, double* __restrict__ B, size_t n, size_t dstep,
                               const int* __restrict__ state) {
    if (*state == 0) return;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        A[i] = i % dstep == 0 ? (double)(i / dstep + 1) : 0.0;
        if (B) B[i] = i % dstep == 0 ? 1.0 : 0.0;
    }
}

// The library's dense solvers may never come back from entries that are not finite (observed:
// from a pencil of zeros, whose reduction divides by zero): such a pencil is refused, one
// with a vanishing column of B is not positive definite.  Both are told by the wait for
// the solve's info (es->info[1]); until then the solve runs on a pencil put in its place.
qsb_status look_over(qsb_eigensolver* es, int m, double* A, double* B, cudaStream_t s) {
    const size_t c2 = es->cplx ? 2 : 1, cnt = (size_t)m * m * c2, dstep = ((size_t)m + 1) * c2;
    const int grid = (int)std::min<size_t>((cnt + 255) / 256, 512);
    QSB_CUDA_TRY(cudaMemsetAsync(es->info + 1, 0, sizeof(int), s));
    pencil_state<<<grid, 256, 0, s>>>(A, B, cnt, dstep, es->info + 1);
    pencil_replace<<<grid, 256, 0, s>>>(A, B, cnt, dstep, es->info + 1);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// generalized eigenproblem Sa c = lambda Sb c (m x m), eigenvalues ascending into
// es->W, eigenvectors into Sa (B-orthonormal).
qsb_status solve_pencil(qsb_eigensolver* es, int m, cudaStream_t s) {
    QSB_TRY(look_over(es, m, es->Sa, es->Sb, s));
    int lwork = 0;
    if (es->cplx) {
        QSB_SOLVER_TRY(cusolverDnZhegvd_bufferSize(es->sol, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                                   CUBLAS_FILL_MODE_UPPER, m, (cuDoubleComplex*)es->Sa, m,
                                                   (cuDoubleComplex*)es->Sb, m, es->W, &lwork));
    } else {
        QSB_SOLVER_TRY(cusolverDnDsygvd_bufferSize(es->sol, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR,
                                                   CUBLAS_FILL_MODE_UPPER, m, es->Sa, m, es->Sb, m, es->W, &lwork));
    }
    const size_t bytes = (size_t)lwork * (es->cplx ? sizeof(cuDoubleComplex) : sizeof(double));
    if ((size_t)es->slwork < bytes) {
        if (es->swork) cudaFree(es->swork);
        es->swork = nullptr;
        es->slwork = 0;
        QSB_CUDA_TRY(cudaMalloc(&es->swork, bytes));
        es->slwork = (int)bytes;
    }
    if (es->cplx) {
        QSB_SOLVER_TRY(cusolverDnZhegvd(es->sol, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, m,
                                        (cuDoubleComplex*)es->Sa, m, (cuDoubleComplex*)es->Sb, m, es->W,
                                        (cuDoubleComplex*)es->swork, lwork, es->info));
    } else {
        QSB_SOLVER_TRY(cusolverDnDsygvd(es->sol, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, m,
                                        es->Sa, m, es->Sb, m, es->W, (double*)es->swork, lwork, es->info));
    }
    int words[2] = {0, 0};
    QSB_CUDA_TRY(cudaMemcpyAsync(words, es->info, sizeof(words), cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    const int info = words[0];
    if (words[1] & 1) return fail(QSB_ERR_NUMERIC, "eigensolver: non-finite pencil");
    if (words[1] & 2)
        return fail(QSB_ERR_SOLVER, "eigensolver: generalized eigenproblem failed (overlap matrix not positive definite)");
    if (info != 0)
        return fail(QSB_ERR_SOLVER, "eigensolver: generalized eigenproblem failed, info = " + std::to_string(info) +
                                        (info > m ? " (overlap matrix not positive definite)" : ""));
    return QSB_OK;
}

// OUT = U*C_u [+ V*C_v] for complex bundles via the cnj / rot real views
// (NextVector_z2).  cu/cv: index of the coefficient block (0:x 1:r 2:p) in es->rc.
qsb_status rotate_complex(qsb_eigensolver* es, int na, double* OUT, const double* U, int cu, double beta,
                          cudaStream_t) {
    const size_t blk = (size_t)2 * na * na;
    const double* cnj = es->rc + (size_t)(2 * cu) * blk;
    const double* rot = es->rc + (size_t)(2 * cu + 1) * blk;
    const int ldo = (int)(2 * es->N);
    QSB_TRY(gemm_nn(es, 2 * na, na, 1.0, U, cnj, beta, OUT, ldo));
    QSB_TRY(gemm_nn(es, 2 * na, na, 1.0, U, rot, beta, OUT + es->N, ldo));
    return QSB_OK;
}

qsb_status rotate_real(qsb_eigensolver* es, int na, double* OUT, const double* U, int cu, double beta, cudaStream_t) {
    const double* C = es->rc + (size_t)cu * na * na;
    return gemm_nn(es, na, na, 1.0, U, C, beta, OUT, (int)es->N);
}

// coefficient blocks of the lowest na eigenvectors (columns of Sa, m rows)
qsb_status make_coefficients(qsb_eigensolver* es, int na, int m, int nblk, cudaStream_t s) {
    dim3 grid((na + 127) / 128, na);
    for (int b = 0; b < nblk; ++b) {
        if (es->cplx) {
            const size_t blk = (size_t)2 * na * na;
            make_rot_cnj<<<grid, 128, 0, s>>>((const double2*)es->Sa, m, b * na, na, na, es->rc + (size_t)(2 * b) * blk,
                                              es->rc + (size_t)(2 * b + 1) * blk);
        } else {
            copy_real_block<<<grid, 128, 0, s>>>(es->Sa, m, b * na, na, na, es->rc + (size_t)b * na * na);
        }
    }
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// The steady-state pencil update of LOBPCG::Eigen_z_multi_mpi (NextMatrix_z,
// source/lobpcg_z_multi_mpi.h:579-794, with DIRECT_S_MATRIX_XR_RP, :58): with
// X' = X Cx + P', P' = R Cr + P Cp and C = [Cx; Cr; Cp] the lowest n generalized
// eigenvectors of the pencil S0 (first n columns of Sa, ld m), the X'/P' blocks of
// the next pencil follow from S0 alone:
//   W = S0[:, n:m] C[n:m],  U = S0[:, 0:n] C[0:n] + W   (= S0 C),
//   X'^H S X' = C^H U,  X'^H S P' = C^H W,  P'^H S P' = C[n:m]^H W[n:m]
// for S = the overlap and for S = the Hamiltonian (small complex GEMMs).
// Layout of es->nxt (complex): S0a, S0b (m x m), then XX, XP, PP, HXX, HXP, HPP
// (n x n), then W, U (m x n).
qsb_status next_pencil_blocks(qsb_eigensolver* es, int n, int m, cudaStream_t s) {
    const int mmax = 3 * es->nmax;
    double2* base = (double2*)es->nxt;
    const double2* S0[2] = {base, base + (size_t)mmax * mmax};      // Hamiltonian, overlap
    double2* blk = base + (size_t)2 * mmax * mmax;
    const size_t nn = (size_t)es->nmax * es->nmax;
    double2* Wk = blk + 6 * nn;
    double2* Uk = Wk + (size_t)mmax * es->nmax;
    const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), zero = make_cuDoubleComplex(0.0, 0.0);
    const cuDoubleComplex* C = (const cuDoubleComplex*)es->Sa;
    for (int h = 0; h < 2; ++h) {
        const cuDoubleComplex* S = (const cuDoubleComplex*)S0[h];
        cuDoubleComplex* XX = (cuDoubleComplex*)(blk + (size_t)(h == 0 ? 3 : 0) * nn);
        cuDoubleComplex* XP = XX + nn;
        cuDoubleComplex* PP = XP + nn;
        QSB_BLAS_TRY(cublasZgemm(es->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, n, m - n, &one, S + (size_t)n * m, m, C + n, m,
                                 &zero, (cuDoubleComplex*)Wk, m));
        QSB_CUDA_TRY(cudaMemcpyAsync(Uk, Wk, sizeof(double2) * (size_t)m * n, cudaMemcpyDeviceToDevice, s));
        QSB_BLAS_TRY(cublasZgemm(es->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, n, n, &one, S, m, C, m, &one,
                                 (cuDoubleComplex*)Uk, m));
        QSB_BLAS_TRY(cublasZgemm(es->blas, CUBLAS_OP_C, CUBLAS_OP_N, n, n, m, &one, C, m, (cuDoubleComplex*)Uk, m, &zero,
                                 XX, n));
        QSB_BLAS_TRY(cublasZgemm(es->blas, CUBLAS_OP_C, CUBLAS_OP_N, n, n, m, &one, C, m, (cuDoubleComplex*)Wk, m, &zero,
                                 XP, n));
        QSB_BLAS_TRY(cublasZgemm(es->blas, CUBLAS_OP_C, CUBLAS_OP_N, n, n, m - n, &one, C + n, m,
                                 (cuDoubleComplex*)Wk + n, m, &zero, PP, n));
    }
    return QSB_OK;
}

// The X/P blocks of the 3n pencil from next_pencil_blocks, and the two overlap
// blocks of R that follow from them with R = AX - X E (E the Ritz values the
// residual was formed with, es->W): X^H R = X^H A X - X^H X E,
// R^H P = X^H A P - E X^H P.
qsb_status put_next_blocks(qsb_eigensolver* es, int n, int m, cudaStream_t s) {
    const int mmax = 3 * es->nmax;
    const size_t nn = (size_t)es->nmax * es->nmax;
    const double2* blk = (const double2*)es->nxt + (size_t)2 * mmax * mmax;
    const double2 *XX = blk, *XP = blk + nn, *PP = blk + 2 * nn;
    const double2 *HXX = blk + 3 * nn, *HXP = blk + 4 * nn, *HPP = blk + 5 * nn;
    double2* Sa = (double2*)es->Sa;
    double2* Sb = (double2*)es->Sb;
    const dim3 g((n + 127) / 128, n);
    put_pencil_block<<<g, 128, 0, s>>>(HXX, nullptr, nullptr, 0, n, Sa, m, 0, 0, 1);
    put_pencil_block<<<g, 128, 0, s>>>(HXP, nullptr, nullptr, 0, n, Sa, m, 0, 2 * n, 0);
    put_pencil_block<<<g, 128, 0, s>>>(HPP, nullptr, nullptr, 0, n, Sa, m, 2 * n, 2 * n, 1);
    put_pencil_block<<<g, 128, 0, s>>>(XX, nullptr, nullptr, 0, n, Sb, m, 0, 0, 1);
    put_pencil_block<<<g, 128, 0, s>>>(XP, nullptr, nullptr, 0, n, Sb, m, 0, 2 * n, 0);
    put_pencil_block<<<g, 128, 0, s>>>(PP, nullptr, nullptr, 0, n, Sb, m, 2 * n, 2 * n, 1);
    put_pencil_block<<<g, 128, 0, s>>>(HXX, XX, es->W, 1, n, Sb, m, 0, n, 0);
    put_pencil_block<<<g, 128, 0, s>>>(HXP, XP, es->W, 2, n, Sb, m, n, 2 * n, 0);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

}  // namespace
}  // namespace qsb

// ---------------------------------------------------------------------------
// Mixed precision (QSB_PREC_MIXED): fp32 bundles, split-BF16x3 tensor-core
// Gram products, fp32 rotations, fp64 pencil / Rayleigh quotients / norms.
// The steps and their order are those of the fp64 solvers above.
// ---------------------------------------------------------------------------
namespace qsb {
namespace {

// Sb = U^H U, Sa = U^H AU over the whole basis (m bands) in two tensor-core
// Gram products (upper tiles; the pencil's lower triangle is the mirror, as
// MakeMatrix_z_blas computes only the upper blocks).  scale: dV for the real solver.
// split copy of an fp32 operand in the solver's Gram form
qsb_status gram_split_operand(qsb_eigensolver* es, const ColumnSet& src, void* dst, cudaStream_t s) {
    if (es->gram_kind == QSB_GRAM_INT8_OZAKI) return ozaki_split(QSB_F32, es->N, src, dst, s);
    return split_bf16(QSB_F32, es->N, src, dst, s);
}
// T (ld ldt) = A^T B from split operands, in the solver's Gram form
qsb_status gram_of_splits(qsb_eigensolver* es, const void* A, int p, const void* B, int q, bool upper, double* T,
                          int ldt, cudaStream_t s) {
    if (es->gram_kind == QSB_GRAM_INT8_OZAKI)
        return gram_ozaki_tc(es->N, A, p, B, q, upper, T, ldt, 1.0, false, es->gpart, es->gpart_bytes, s);
    return gram_split_tc(es->N, A, p, B, q, upper, T, ldt, 1.0, false, es->gpart, es->gpart_bytes, s,
                         es->gram_kind == QSB_GRAM_BF16X4 ? 4 : 3);
}

qsb_status mixed_pencil(qsb_eigensolver* es, const ColumnSet& U, const ColumnSet& AU, int m, double scale,
                        cudaStream_t s) {
    const int p = column_count(U);   // real columns: m (real) or 2m (complex)
    QSB_TRY(gram_split_operand(es, U, es->su, s));
    QSB_TRY(gram_split_operand(es, AU, es->sau, s));
    const dim3 grid((m + 127) / 128, m);
    QSB_TRY(gram_of_splits(es, es->su, p, es->su, p, true, es->T2, p, s));
    if (es->cplx)
        assemble_complex_block<<<grid, 128, 0, s>>>(es->T2, m, m, p, (double2*)es->Sb, m, 0, 0, 1);
    else
        assemble_real_block<<<grid, 128, 0, s>>>(es->T2, m, m, p, es->Sb, m, 0, 0, 1, scale);
    QSB_CUDA_TRY(cudaGetLastError());
    QSB_TRY(gram_of_splits(es, es->su, p, es->sau, p, true, es->T2, p, s));
    if (es->cplx)
        assemble_complex_block<<<grid, 128, 0, s>>>(es->T2, m, m, p, (double2*)es->Sa, m, 0, 0, 1);
    else
        assemble_real_block<<<grid, 128, 0, s>>>(es->T2, m, m, p, es->Sa, m, 0, 0, 1, scale);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// ---- overlap-basis pencil solve (mixed precision) --------------------------
// d_i = 1 / sqrt(B_ii) (0 for a vanishing column)
__global__ void pencil_diag(const double* __restrict__ B, int m, int cplx, double* __restrict__ d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double b = cplx ? B[2 * ((size_t)i + (size_t)m * i)] : B[(size_t)i + (size_t)m * i];
    d[i] = b > 0.0 ? 1.0 / sqrt(b) : 0.0;
}
// A_ij *= d_i d_j, B_ij *= d_i d_j
__global__ void pencil_scale(double* __restrict__ A, double* __restrict__ B, int m, int cplx,
                             const double* __restrict__ d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (i >= m) return;
    const double f = d[i] * d[j];
    const size_t e = (size_t)i + (size_t)m * j;
    if (cplx) {
        A[2 * e] *= f; A[2 * e + 1] *= f;
        B[2 * e] *= f; B[2 * e + 1] *= f;
    } else {
        A[e] *= f;
        B[e] *= f;
    }
}
// Wm[:, j] = V[:, c0 + j] / sqrt(lam[c0 + j])  (m x k)
__global__ void overlap_basis(const double* __restrict__ V, const double* __restrict__ lam, int m, int c0, int k,
                              int cplx, double* __restrict__ Wm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (i >= m || j >= k) return;
    const double f = 1.0 / sqrt(lam[c0 + j]);
    const size_t src = (size_t)i + (size_t)m * (c0 + j), dst = (size_t)i + (size_t)m * j;
    if (cplx) {
        Wm[2 * dst] = V[2 * src] * f;
        Wm[2 * dst + 1] = V[2 * src + 1] * f;
    } else {
        Wm[dst] = V[src] * f;
    }
}
// C_ij = d_i Z_ij  (m x ncol, ld m)
__global__ void rows_scale(const double* __restrict__ Z, const double* __restrict__ d, int m, int ncol, int cplx,
                           double* __restrict__ C) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (i >= m || j >= ncol) return;
    const size_t e = (size_t)i + (size_t)m * j;
    if (cplx) {
        C[2 * e] = Z[2 * e] * d[i];
        C[2 * e + 1] = Z[2 * e + 1] * d[i];
    } else {
        C[e] = Z[e] * d[i];
    }
}

qsb_status ensure_swork(qsb_eigensolver* es, size_t bytes) {
    if ((size_t)es->slwork >= bytes) return QSB_OK;
    if (es->swork) cudaFree(es->swork);
    es->swork = nullptr;
    es->slwork = 0;
    QSB_CUDA_TRY(cudaMalloc(&es->swork, bytes));
    es->slwork = (int)bytes;
    return QSB_OK;
}

// Hermitian / symmetric eigendecomposition in place (ascending eigenvalues in w)
qsb_status dense_evd(qsb_eigensolver* es, int k, double* A, double* w, cudaStream_t s) {
    const int lda = k;
    QSB_TRY(look_over(es, k, A, nullptr, s));
    int lwork = 0;
    if (es->cplx) {
        QSB_SOLVER_TRY(cusolverDnZheevd_bufferSize(es->sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, k,
                                                   (cuDoubleComplex*)A, lda, w, &lwork));
        QSB_TRY(ensure_swork(es, (size_t)lwork * sizeof(cuDoubleComplex)));
        QSB_SOLVER_TRY(cusolverDnZheevd(es->sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, k,
                                        (cuDoubleComplex*)A, lda, w, (cuDoubleComplex*)es->swork, lwork, es->info));
    } else {
        QSB_SOLVER_TRY(cusolverDnDsyevd_bufferSize(es->sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, k, A, lda,
                                                   w, &lwork));
        QSB_TRY(ensure_swork(es, (size_t)lwork * sizeof(double)));
        QSB_SOLVER_TRY(cusolverDnDsyevd(es->sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, k, A, lda, w,
                                        (double*)es->swork, lwork, es->info));
    }
    int words[2] = {0, 0};
    QSB_CUDA_TRY(cudaMemcpyAsync(words, es->info, sizeof(words), cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    const int info = words[0];
    if (words[1] & 1) return fail(QSB_ERR_NUMERIC, "eigensolver: non-finite pencil");
    if (info != 0) return fail(QSB_ERR_SOLVER, "eigensolver: dense eigendecomposition failed, info = " + std::to_string(info));
    return QSB_OK;
}

// OUT (r x c, ld ldo) = op(X) (r x kk) . Y (kk x c); op = conjugate transpose when herm
qsb_status small_gemm(qsb_eigensolver* es, bool herm, int r, int c, int kk, const double* X, int ldx, const double* Y,
                      int ldy, double* OUT, int ldo) {
    const cublasOperation_t opx = herm ? (es->cplx ? CUBLAS_OP_C : CUBLAS_OP_T) : CUBLAS_OP_N;
    if (es->cplx) {
        const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), zero = make_cuDoubleComplex(0.0, 0.0);
        QSB_BLAS_TRY(cublasZgemm(es->blas, opx, CUBLAS_OP_N, r, c, kk, &one, (const cuDoubleComplex*)X, ldx,
                                 (const cuDoubleComplex*)Y, ldy, &zero, (cuDoubleComplex*)OUT, ldo));
    } else {
        const double one = 1.0, zero = 0.0;
        QSB_BLAS_TRY(cublasDgemm(es->blas, opx, CUBLAS_OP_N, r, c, kk, &one, X, ldx, Y, ldy, &zero, OUT, ldo));
    }
    return QSB_OK;
}

// Lowest nout Ritz pairs of the pencil (Sa, Sb) (m x m, full Hermitian) on the
// well-conditioned part of the basis: scale to a unit diagonal, eigendecompose
// the overlap, keep the directions with eigenvalue above drop_tol * max, and
// solve the standard problem there (the overlap-basis "SVQB" form of
// Stathopoulos & Wu, used in LOBPCG by Hetmaniuk & Lehoucq).  Eigenvalues go to
// es->W, B-orthonormal eigenvectors to the first nout columns of Sa (ld m),
// where the cholesky-based solve_pencil leaves them.
qsb_status solve_pencil_overlap_basis(qsb_eigensolver* es, int m, int nout, cudaStream_t s) {
    const int c2 = es->cplx ? 2 : 1;
    const size_t mm = (size_t)m * m * c2;
    double* Wm = es->svq;
    double* tmp = Wm + mm;
    double* Ah = tmp + mm;
    double* lam = Ah + mm;
    double* d = lam + m;
    pencil_diag<<<(m + 127) / 128, 128, 0, s>>>(es->Sb, m, es->cplx, d);
    pencil_scale<<<dim3((m + 127) / 128, m), 128, 0, s>>>(es->Sa, es->Sb, m, es->cplx, d);
    QSB_CUDA_TRY(cudaGetLastError());
    // First the Cholesky route (one eigendecomposition): with an unbiased Gram the
    // scaled overlap stays numerically positive definite in most iterations.
    // The scaled pencil is kept in Wm / tmp for the fallback.
    if (es->gram_kind == QSB_GRAM_INT8_OZAKI) {
        QSB_CUDA_TRY(cudaMemcpyAsync(Wm, es->Sa, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
        QSB_CUDA_TRY(cudaMemcpyAsync(tmp, es->Sb, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
        const std::string saved_error = qsb_last_error();
        const qsb_status st = solve_pencil(es, m, s);
        if (st == QSB_ERR_NUMERIC) return st;
        if (st == QSB_OK) {
            rows_scale<<<dim3((m + 127) / 128, nout), 128, 0, s>>>(es->Sa, d, m, nout, es->cplx, es->Sa);
            QSB_CUDA_TRY(cudaGetLastError());
            ++es->last_chol;
            return QSB_OK;
        }
        set_last_error(saved_error);   // a failed Cholesky here is expected, not an error of the call
        QSB_CUDA_TRY(cudaMemcpyAsync(es->Sa, Wm, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
        QSB_CUDA_TRY(cudaMemcpyAsync(es->Sb, tmp, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
    }
    ++es->last_svqb;
    QSB_TRY(dense_evd(es, m, es->Sb, lam, s));
    std::vector<double> hl(m);
    QSB_CUDA_TRY(cudaMemcpyAsync(hl.data(), lam, sizeof(double) * m, cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    const double lmax = hl[m - 1];
    if (!(lmax > 0.0) || !std::isfinite(lmax)) return fail(QSB_ERR_NUMERIC, "eigensolver: overlap matrix vanishes");
    int c0 = 0;
    while (c0 < m && !(hl[c0] > es->drop_tol * lmax)) ++c0;
    const int k = m - c0;
    es->last_dropped = std::max(es->last_dropped, c0);
    if (c0 < m) es->last_min_kept = std::min(es->last_min_kept, hl[c0] / lmax);
    if (k < nout)
        return fail(QSB_ERR_SOLVER, "eigensolver: search basis rank " + std::to_string(k) + " below the " +
                                        std::to_string(nout) + " bands sought");
    overlap_basis<<<dim3((m + 127) / 128, k), 128, 0, s>>>(es->Sb, lam, m, c0, k, es->cplx, Wm);
    QSB_CUDA_TRY(cudaGetLastError());
    QSB_TRY(small_gemm(es, false, m, k, m, es->Sa, m, Wm, m, tmp, m));   // A Wm
    QSB_TRY(small_gemm(es, true, k, k, m, Wm, m, tmp, m, Ah, k));        // Wm^H A Wm
    QSB_TRY(dense_evd(es, k, Ah, es->W, s));
    QSB_TRY(small_gemm(es, false, m, nout, k, Wm, m, Ah, k, tmp, m));    // Wm Y
    rows_scale<<<dim3((m + 127) / 128, nout), 128, 0, s>>>(tmp, d, m, nout, es->cplx, es->Sa);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// The FP64 solvers' Rayleigh-Ritz step: ZHEGVD / DSYGVD (the reference's
// lapack_ZHEGVD / lapack_DSYGVX route) on the pencil as formed.  If its Cholesky
// finds the overlap not positive definite (a search basis [X R P] that has
// turned numerically dependent, e.g. when a run is continued from states of
// another precision), the same pencil is solved on its well-conditioned part
// by the overlap-basis route instead of failing the call.  The reference prints
// the LAPACK info and carries on with the garbage; here the step stays defined.
qsb_status solve_pencil_fp64(qsb_eigensolver* es, int m, int nout, cudaStream_t s) {
    const size_t mm = (size_t)m * m * (es->cplx ? 2 : 1);
    double* Sa0 = es->svq;
    double* Sb0 = Sa0 + mm;
    QSB_CUDA_TRY(cudaMemcpyAsync(Sa0, es->Sa, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(Sb0, es->Sb, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
    const std::string saved_error = qsb_last_error();
    qsb_status st = QSB_OK;
    bool solved = false;
    if (pencil_small_fits(m, nout, es->cplx != 0)) {
        // one launch for what the library does in some hundred: 48 x 48 real 0.5 -> 0.24 ms,
        // 72 x 72 complex 1.1 -> 0.62 ms
        QSB_TRY(pencil_small(m, nout, es->cplx != 0, es->Sa, es->Sb, es->W, es->info, s));
        int info = 0;
        QSB_CUDA_TRY(cudaMemcpyAsync(&info, es->info, sizeof(int), cudaMemcpyDeviceToHost, s));
        QSB_CUDA_TRY(cudaStreamSynchronize(s));
        solved = info >= 0;
        if (info > 0)
            st = fail(QSB_ERR_SOLVER, "eigensolver: generalized eigenproblem failed, info = " + std::to_string(info) +
                                          " (overlap matrix not positive definite)");
        if (!solved) {
            QSB_CUDA_TRY(cudaMemcpyAsync(es->Sa, Sa0, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
            QSB_CUDA_TRY(cudaMemcpyAsync(es->Sb, Sb0, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
        }
    }
    if (!solved) st = solve_pencil(es, m, s);
    if (st == QSB_OK) {
        ++es->last_chol;
        return QSB_OK;
    }
    if (st != QSB_ERR_SOLVER) return st;
    set_last_error(saved_error);
    QSB_CUDA_TRY(cudaMemcpyAsync(es->Sa, Sa0, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(es->Sb, Sb0, sizeof(double) * mm, cudaMemcpyDeviceToDevice, s));
    return solve_pencil_overlap_basis(es, m, nout, s);
}

// a[i] /= b[i]
__global__ void divide_by(double* __restrict__ a, const double* __restrict__ b, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] /= b[i];
}

// Rotation coefficients of the real solver for one tensor-core product per
// bundle set: [X' | P'] = [X R P] C2 with C2 (m x 2n) = [[Cx, 0], [Cr, Cr], [Cp, Cp]]
// (P' = R Cr + P Cp, X' = X Cx + P'), from the eigenvectors C (m x n, ld m).
__global__ void build_rot_coef_real(const double* __restrict__ C, int m, int n, double* __restrict__ C2) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (k >= m) return;
    C2[(size_t)k + (size_t)m * j] = j < n ? C[(size_t)k + (size_t)m * j]
                                          : (k < n ? 0.0 : C[(size_t)k + (size_t)m * (j - n)]);
}

// Column j of C2 scaled to unit B-norm: norms_j = C2_j^T (B C2)_j (G = B C2),
// C2_j /= sqrt(norms_j) — the per-band renormalisation of x' and p' (dV-weighted,
// B = dV U^T U) done on the coefficients instead of on the bundles.
__global__ void normalize_rot_coef(double* __restrict__ C2, const double* __restrict__ G, int m,
                                   double* __restrict__ norms) {
    const int j = blockIdx.x;
    double acc = 0.0;
    for (int k = threadIdx.x; k < m; k += blockDim.x) acc += C2[(size_t)k + (size_t)m * j] * G[(size_t)k + (size_t)m * j];
    __shared__ double red[256];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    const double nrm = red[0];
    const double f = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    if (threadIdx.x == 0) norms[j] = nrm;
    for (int k = threadIdx.x; k < m; k += blockDim.x) C2[(size_t)k + (size_t)m * j] *= f;
}

// [X' | P'] and [AX' | AP'] of the real mixed solver as two INT8 tensor-core
// rotations of the Gram's slices (es->su, es->sau hold [X R P], [AX AR AP]),
// normalised through the coefficients; written straight into the bundles.
qsb_status rotate_real_ozaki(qsb_eigensolver* es, int m, int n, const double* Bsave, cudaStream_t s) {
    double* C2 = es->rotw + (size_t)m * m;
    double* G = C2 + (size_t)m * 2 * n;
    double* norms = G + (size_t)m * 2 * n;
    build_rot_coef_real<<<dim3((m + 127) / 128, 2 * n), 128, 0, s>>>(es->Sa, m, n, C2);
    QSB_CUDA_TRY(cudaGetLastError());
    const double one = 1.0, zero = 0.0;
    QSB_BLAS_TRY(cublasDgemm(es->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, 2 * n, m, &one, Bsave, m, C2, m, &zero, G, m));
    // only the x' columns: their B-norm is 1 up to rounding, so the coefficient
    // route is exact enough.  p' = R Cr + P Cp can be tiny once a band has
    // converged, and its B-norm from the overlap is then dominated by the Gram
    // products' error: p' is normalised from its measured norm after the rotation.
    normalize_rot_coef<<<n, 256, 0, s>>>(C2, G, m, norms);
    QSB_CUDA_TRY(cudaGetLastError());
    QSB_TRY(ozaki_rotate(es->N, es->su, m, C2, m, 2 * n, column_set(es->X32, n, es->P32, n), es->rotc, es->rotc_bytes,
                         s, n, n));
    QSB_TRY(ozaki_rotate(es->N, es->sau, m, C2, m, 2 * n, column_set(es->AX32, n, es->AP32, n), es->rotc,
                         es->rotc_bytes, s, n, n));
    return QSB_OK;
}

// fp32 copies of the first count rotation coefficients
qsb_status coefficients_f32(qsb_eigensolver* es, size_t count, cudaStream_t s) {
    to_f32<<<(int)std::min<size_t>((count + 255) / 256, 1024), 256, 0, s>>>(es->rc, es->rc32, count);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

qsb_status rotate_real32(qsb_eigensolver* es, int na, float* OUT, const float* U, int cu, float beta) {
    return sgemm_nn(es, na, na, 1.0f, U, es->rc32 + (size_t)cu * na * na, beta, OUT, (int)es->N);
}

qsb_status rotate_complex32(qsb_eigensolver* es, int na, float* OUT, const float* U, int cu, float beta) {
    const size_t blk = (size_t)2 * na * na;
    const int ldo = (int)(2 * es->N);
    QSB_TRY(sgemm_nn(es, 2 * na, na, 1.0f, U, es->rc32 + (size_t)(2 * cu) * blk, beta, OUT, ldo));
    QSB_TRY(sgemm_nn(es, 2 * na, na, 1.0f, U, es->rc32 + (size_t)(2 * cu + 1) * blk, beta, OUT + es->N, ldo));
    return QSB_OK;
}

// B_act -= X_fix (X_fix^H B_act) for complex fp32 bundles (VectorOrthogonalization)
qsb_status orthogonalize32(qsb_eigensolver* es, int nf, int na, const float* Xfix, float* B, cudaStream_t s) {
    QSB_TRY(gram_split_operand(es, column_set(Xfix, 2 * nf), es->su, s));
    QSB_TRY(gram_split_operand(es, column_set(B, 2 * na), es->sau, s));
    QSB_TRY(gram_of_splits(es, es->su, 2 * nf, es->sau, 2 * na, false, es->T2, 2 * nf, s));
    pack_orth<<<dim3((nf + 127) / 128, na), 128, 0, s>>>(es->T2, nf, na);
    QSB_CUDA_TRY(cudaGetLastError());
    const size_t cnt = (size_t)2 * nf * 2 * na;
    to_f32<<<(int)std::min<size_t>((cnt + 255) / 256, 1024), 256, 0, s>>>(es->T2, es->rc32, cnt);
    QSB_CUDA_TRY(cudaGetLastError());
    return sgemm_nn(es, 2 * nf, 2 * na, -1.0f, Xfix, es->rc32, 1.0f, B, (int)es->N);
}

qsb_status copy32(float* dst, const float* src, size_t count, cudaStream_t s) {
    QSB_CUDA_TRY(cudaMemcpyAsync(dst, src, sizeof(float) * count, cudaMemcpyDeviceToDevice, s));
    return QSB_OK;
}

// EigenLOBPCG_d_multi (source/lobpcg_d_multi.h:23-545) on fp32 bundles.
qsb_status lobpcg_d_mixed(qsb_eigensolver* es, double dVol, int n, int iter_max, double* eigen_values, double* X64,
                          double* keep64, int is_first_time, cudaStream_t s) {
    const size_t L = es->L;
    double* eps_d = es->vec;
    double* nrm_d = es->vec + n;
    double* scl_d = es->vec + 2 * n;
    std::vector<double> v(n), scl(n);
    auto host_vec = [&](const double* d, std::vector<double>& h) -> qsb_status {
        QSB_CUDA_TRY(cudaMemcpyAsync(h.data(), d, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
        QSB_CUDA_TRY(cudaStreamSynchronize(s));
        for (int k = 0; k < n; ++k)
            if (!std::isfinite(h[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_d: non-finite value");
        return QSB_OK;
    };
    // x /= sqrt(|x|^2 dV) per band (Normalize, source/vecmath.h:128-134), fp64 sums
    auto inv_norms = [&](const float* B, std::vector<double>& out) -> qsb_status {
        QSB_TRY(seg_dot(es, n, B, B, dVol, nrm_d, s));
        QSB_TRY(host_vec(nrm_d, v));
        for (int k = 0; k < n; ++k) out[k] = 1.0 / std::sqrt(v[k]);
        return QSB_OK;
    };
    auto scale_bands = [&](float* B, const std::vector<double>& f) -> qsb_status {
        QSB_CUDA_TRY(cudaMemcpyAsync(scl_d, f.data(), sizeof(double) * n, cudaMemcpyHostToDevice, s));
        return seg_scale_by(es, n, B, scl_d, 0.0, s);
    };

    QSB_TRY(seg_convert_by(es, n, X64, es->X32, nullptr, 1.0, s));
    QSB_TRY(inv_norms(es->X32, scl));
    QSB_TRY(scale_bands(es->X32, scl));
    QSB_TRY(apply_op32(es, n, es->X32, es->AX32, s));
    if (is_first_time) {
        QSB_CUDA_TRY(cudaMemsetAsync(es->P32, 0, sizeof(float) * L * n, s));
        QSB_CUDA_TRY(cudaMemsetAsync(es->AP32, 0, sizeof(float) * L * n, s));
    } else {
        QSB_TRY(seg_convert_by(es, n, keep64, es->P32, nullptr, 1.0, s));
        QSB_TRY(apply_op32(es, n, es->P32, es->AP32, s));
    }
    QSB_TRY(seg_dot(es, n, es->X32, es->AX32, dVol, eps_d, s));
    QSB_TRY(seg_residual(es, n, es->R32, es->AX32, es->X32, eps_d, (double*)nullptr, 1.0, s));
    QSB_TRY(inv_norms(es->R32, scl));
    QSB_TRY(scale_bands(es->R32, scl));
    std::vector<double> eps(n), sx(n), sp(n);
    QSB_TRY(host_vec(eps_d, eps));
    for (int k = 0; k < n; ++k) eigen_values[k] = eps[k];

    int iter;
    for (iter = 0; iter < iter_max; ++iter) {
        QSB_TRY(apply_op32(es, n, es->R32, es->AR32, s));
        const bool two = is_first_time && iter == 0;
        const int nblk = two ? 2 : 3;
        const int m = nblk * n;
        const ColumnSet U = column_set(es->X32, n, es->R32, n, es->P32, two ? 0 : n);
        const ColumnSet AU = column_set(es->AX32, n, es->AR32, n, es->AP32, two ? 0 : n);
        QSB_TRY(mixed_pencil(es, U, AU, m, dVol, s));
        const bool tc_rot = es->gram_kind == QSB_GRAM_INT8_OZAKI;
        if (tc_rot)   // the overlap B, kept for the coefficient norms
            QSB_CUDA_TRY(cudaMemcpyAsync(es->rotw, es->Sb, sizeof(double) * m * m, cudaMemcpyDeviceToDevice, s));
        QSB_TRY(solve_pencil_overlap_basis(es, m, n, s));
        if (tc_rot) {
            // P' = R Cr (+ P Cp); X' = X Cx + P'; the same on the A-bundles (:226-365),
            // on the tensor cores; x renormalised (:493-505) through the coefficients,
            // p from its measured norm
            QSB_TRY(rotate_real_ozaki(es, m, n, es->rotw, s));
            QSB_TRY(inv_norms(es->P32, sp));
            QSB_TRY(scale_bands(es->P32, sp));
            QSB_TRY(scale_bands(es->AP32, sp));
        } else {
            QSB_TRY(make_coefficients(es, n, m, nblk, s));
            QSB_TRY(coefficients_f32(es, (size_t)nblk * n * n, s));
            // P' = R Cr (+ P Cp); X' = X Cx + P'; the same on the A-bundles (:226-365)
            QSB_TRY(rotate_real32(es, n, es->TMP32, es->R32, 1, 0.0f));
            if (!two) QSB_TRY(rotate_real32(es, n, es->TMP32, es->P32, 2, 1.0f));
            std::swap(es->P32, es->TMP32);
            QSB_TRY(copy32(es->TMP32, es->P32, L * n, s));
            QSB_TRY(rotate_real32(es, n, es->TMP32, es->X32, 0, 1.0f));
            std::swap(es->X32, es->TMP32);
            QSB_TRY(rotate_real32(es, n, es->TMP32, es->AR32, 1, 0.0f));
            if (!two) QSB_TRY(rotate_real32(es, n, es->TMP32, es->AP32, 2, 1.0f));
            std::swap(es->AP32, es->TMP32);
            QSB_TRY(copy32(es->TMP32, es->AP32, L * n, s));
            QSB_TRY(rotate_real32(es, n, es->TMP32, es->AX32, 0, 1.0f));
            std::swap(es->AX32, es->TMP32);
            // renormalize x, p and Ax, Ap (:493-505)
            QSB_TRY(inv_norms(es->X32, sx));
            QSB_TRY(inv_norms(es->P32, sp));
            QSB_TRY(scale_bands(es->X32, sx));
            QSB_TRY(scale_bands(es->AX32, sx));
            QSB_TRY(scale_bands(es->P32, sp));
            QSB_TRY(scale_bands(es->AP32, sp));
        }
        // eps = <x|Ax> dV; r = Ax - eps x; ||r||^2 dV (:507-513).  After the tensor-core
        // rotation |x|^2 dV is 1 only to the coefficient slices' rounding (~1e-6), so
        // eps is taken as the normalised Rayleigh quotient <x|Ax> / <x|x>.
        QSB_TRY(seg_dot(es, n, es->X32, es->AX32, dVol, eps_d, s));
        if (tc_rot) {
            QSB_TRY(seg_dot(es, n, es->X32, es->X32, dVol, nrm_d, s));
            divide_by<<<(n + 127) / 128, 128, 0, s>>>(eps_d, nrm_d, n);
            QSB_CUDA_TRY(cudaGetLastError());
        }
        QSB_TRY(seg_residual(es, n, es->R32, es->AX32, es->X32, eps_d, nrm_d, dVol, s));
        QSB_TRY(host_vec(eps_d, eps));
        QSB_TRY(host_vec(nrm_d, v));
        double rmax = 0.0;
        for (int k = 0; k < n; ++k) {
            eigen_values[k] = eps[k];
            rmax = std::max(rmax, v[k]);
        }
        if (rmax < 1.0e-10 * dVol) { ++iter; break; }   // :525
    }
    es->last_iters = iter;
    QSB_TRY(seg_convert_by(es, n, es->X32, X64, nullptr, 1.0, s));
    QSB_TRY(seg_convert_by(es, n, es->P32, keep64, nullptr, 1.0, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    return QSB_OK;
}

// LOBPCG::Eigen_z_multi_mpi (source/lobpcg_z_multi_mpi.h:1732-2852) on fp32
// bundles.  The fixed (locked) bands of the caller's X are read, never written.
qsb_status lobpcg_z_mixed(qsb_eigensolver* es, double dVol, int n, int iter_max, double* eigen_values, double* X64,
                          double* keep64, int* p_num_fix, double residual_threshold, int scf_step, cudaStream_t s) {
    const size_t L = es->L;
    auto b32 = [&](float* base, int k) { return base + (size_t)k * L; };
    auto b64 = [&](double* base, int k) { return base + (size_t)k * L; };
    double* eps_d = es->vec;
    double* nrm_d = es->vec + n;
    double* scl_d = es->vec + 2 * n;
    std::vector<double> eps(n), nr(n), nx(n), scl(n);

    int num_fix = std::max(0, std::min(*p_num_fix, n));
    int num_active = n - num_fix;
    const int head0 = num_fix;
    // X32 = sqrt(dV) X (:1851), all bands: the fixed ones orthogonalize the active ones
    QSB_TRY(seg_convert_by(es, n, X64, es->X32, nullptr, std::sqrt(dVol), s));
    // the active bands normalised (the reference takes them as passed in, which a
    // normalised input makes the same; FP32 rounding of the conversion aside)
    QSB_TRY(seg_dot(es, num_active, b32(es->X32, head0), b32(es->X32, head0), 1.0, nrm_d + head0, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(nx.data(), nrm_d + head0, sizeof(double) * num_active, cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    for (int k = 0; k < num_active; ++k) {
        if (!(nx[k] > 0.0) || !std::isfinite(nx[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_z: zero or non-finite band");
        scl[k] = 1.0 / std::sqrt(nx[k]);
    }
    QSB_CUDA_TRY(cudaMemcpyAsync(scl_d, scl.data(), sizeof(double) * num_active, cudaMemcpyHostToDevice, s));
    QSB_TRY(seg_scale_by(es, num_active, b32(es->X32, head0), scl_d, 0.0, s));
    QSB_TRY(apply_op32(es, num_active, b32(es->X32, head0), b32(es->AX32, head0), s));
    QSB_TRY(seg_dot(es, num_active, b32(es->X32, head0), b32(es->AX32, head0), 1.0, eps_d + head0, s));
    QSB_TRY(seg_residual(es, num_active, b32(es->R32, head0), b32(es->AX32, head0), b32(es->X32, head0), eps_d + head0,
                         nrm_d + head0, 1.0, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(eps.data() + head0, eps_d + head0, sizeof(double) * num_active, cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(nr.data() + head0, nrm_d + head0, sizeof(double) * num_active, cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    for (int k = head0; k < n; ++k)
        if (!std::isfinite(eps[k]) || !std::isfinite(nr[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_z: non-finite Rayleigh quotient");
    // soft locking (:1962-1986)
    int fix_pos = n;
    const double th2 = residual_threshold * residual_threshold;
    for (int k = head0; k < n; ++k)
        if (th2 < nr[k]) { fix_pos = k; break; }
    const int org_active = num_active;
    num_fix = std::min(fix_pos, n / 2);
    num_active = n - num_fix;
    if (num_active != org_active) *p_num_fix = num_fix;
    if (iter_max < 1) return QSB_OK;
    const int head = num_fix;
    const int N_ = num_active;
    const bool is_first_time = (scf_step == 0);
    float* Xa = b32(es->X32, head);
    float* Ra = b32(es->R32, head);
    float* Pa = b32(es->P32, head);
    float* AXa = b32(es->AX32, head);
    float* ARa = b32(es->AR32, head);
    float* APa = b32(es->AP32, head);
    float* TMP = es->TMP32;
    if (is_first_time) {
        QSB_CUDA_TRY(cudaMemsetAsync(es->P32, 0, sizeof(float) * L * n, s));
        QSB_CUDA_TRY(cudaMemsetAsync(es->AP32, 0, sizeof(float) * L * n, s));
    } else {
        QSB_TRY(seg_convert_by(es, N_, b64(keep64, head), Pa, nullptr, 1.0, s));
        if (num_active != org_active && num_fix > 0) QSB_TRY(orthogonalize32(es, num_fix, N_, es->X32, Pa, s));
        QSB_TRY(apply_op32(es, N_, Pa, APa, s));
    }
    // X64 (active) <- X32 (active) / sqrt(|x'|^2 dV)  (:2792-2803, and the rollback's rescale :2651)
    auto write_back_x = [&]() -> qsb_status {
        for (int k = 0; k < N_; ++k) scl[k] = 1.0 / std::sqrt(nx[k] * dVol);
        QSB_CUDA_TRY(cudaMemcpyAsync(scl_d, scl.data(), sizeof(double) * N_, cudaMemcpyHostToDevice, s));
        return seg_convert_by(es, N_, Xa, b64(X64, head), scl_d, 0.0, s);
    };
    int iter;
    for (iter = 0; iter < iter_max; ++iter) {
        if (num_fix > 0) QSB_TRY(orthogonalize32(es, num_fix, N_, es->X32, Ra, s));   // :2080
        QSB_TRY(apply_op32(es, N_, Ra, ARa, s));                                          // :2084
        const bool use_p = !(is_first_time && iter == 0);
        const int nblk = use_p ? 3 : 2;
        const int m = nblk * N_;
        const ColumnSet U = column_set(Xa, 2 * N_, Ra, 2 * N_, Pa, use_p ? 2 * N_ : 0);
        const ColumnSet AU = column_set(AXa, 2 * N_, ARa, 2 * N_, APa, use_p ? 2 * N_ : 0);
        QSB_TRY(mixed_pencil(es, U, AU, m, 1.0, s));
        QSB_TRY(solve_pencil_overlap_basis(es, m, N_, s));
        QSB_TRY(make_coefficients(es, N_, m, nblk, s));
        QSB_TRY(coefficients_f32(es, (size_t)nblk * 2 * (2 * N_) * N_, s));
        // P' = R Cr + P Cp; X' = X Cx + P'  (NextVector_z2)
        QSB_TRY(rotate_complex32(es, N_, TMP, Ra, 1, 0.0f));
        if (use_p) QSB_TRY(rotate_complex32(es, N_, TMP, Pa, 2, 1.0f));
        QSB_TRY(copy32(Pa, TMP, L * N_, s));
        QSB_TRY(rotate_complex32(es, N_, TMP, Xa, 0, 1.0f));
        QSB_TRY(seg_dot(es, N_, TMP, TMP, 1.0, nrm_d, s));                               // :2570
        QSB_CUDA_TRY(cudaMemcpyAsync(nx.data(), nrm_d, sizeof(double) * N_, cudaMemcpyDeviceToHost, s));
        QSB_CUDA_TRY(cudaStreamSynchronize(s));
        double maxdiff = 0.0;
        for (int k = 0; k < N_; ++k) {
            if (!std::isfinite(nx[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_z: non-finite vector norm");
            maxdiff = std::max(maxdiff, std::fabs(1.0 - nx[k]));
        }
        if (maxdiff > 1.0e-3) {   // rollback (:2611-2666): keep X, P <- R
            es->last_rollback = 1;
            QSB_TRY(copy32(Pa, Ra, L * N_, s));
            // The reference rescales the kept X with the norms of the rejected X'
            // (:2651), harmless when they are 1 +- 1e-3.  Here the rollback can
            // come from coefficients spoilt by an ill-conditioned basis, with
            // norms far from 1: the kept X is normalised with its own norms, or
            // the next call would start from mis-scaled bands.
            QSB_TRY(seg_dot(es, N_, Xa, Xa, 1.0, nrm_d, s));
            QSB_CUDA_TRY(cudaMemcpyAsync(nx.data(), nrm_d, sizeof(double) * N_, cudaMemcpyDeviceToHost, s));
            QSB_CUDA_TRY(cudaStreamSynchronize(s));
            QSB_TRY(write_back_x());
            ++iter;
            break;
        }
        QSB_TRY(copy32(Xa, TMP, L * N_, s));
        // AP' = AR Cr + AP Cp; AX' = AX Cx + AP' (:2718), on the last iteration too:
        // the eigenvalues are the Rayleigh quotients <x'|Ax'> / <x'|x'> summed in
        // fp64, not the pencil's Ritz values, which carry the Gram products'
        // error (with 3 products, no lo*lo term, the overlap diagonal is low by
        // sum(lo^2) ~ 2^-16/3 relative and the Ritz values sit that much high).
        QSB_TRY(rotate_complex32(es, N_, TMP, ARa, 1, 0.0f));
        if (use_p) QSB_TRY(rotate_complex32(es, N_, TMP, APa, 2, 1.0f));
        QSB_TRY(copy32(APa, TMP, L * N_, s));
        QSB_TRY(rotate_complex32(es, N_, TMP, AXa, 0, 1.0f));
        QSB_TRY(copy32(AXa, TMP, L * N_, s));
        QSB_TRY(seg_dot(es, N_, Xa, AXa, 1.0, eps_d, s));
        std::vector<double> w(N_);
        QSB_CUDA_TRY(cudaMemcpyAsync(w.data(), eps_d, sizeof(double) * N_, cudaMemcpyDeviceToHost, s));
        QSB_CUDA_TRY(cudaStreamSynchronize(s));
        for (int k = 0; k < N_; ++k) {
            w[k] /= nx[k];
            if (!std::isfinite(w[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_z: non-finite Rayleigh quotient");
            eps[head + k] = w[k];
        }
        if (iter + 1 < iter_max) {
            QSB_CUDA_TRY(cudaMemcpyAsync(eps_d, w.data(), sizeof(double) * N_, cudaMemcpyHostToDevice, s));
            QSB_TRY(seg_residual(es, N_, Ra, AXa, Xa, eps_d, (double*)nullptr, 1.0, s));   // :2750
        } else {
            QSB_TRY(write_back_x());
        }
    }
    es->last_iters = iter;
    for (int k = head; k < n; ++k) eigen_values[k] = eps[k];
    QSB_TRY(seg_convert_by(es, N_, Pa, b64(keep64, head), nullptr, 1.0, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    return QSB_OK;
}

}  // namespace
}  // namespace qsb

void qsb::eigensolver_shape(const qsb_eigensolver* es, int64_t* N, int* nmax, int* cplx, int* mixed) {
    *N = es->N;
    *nmax = es->nmax;
    *cplx = es->cplx;
    *mixed = es->mixed;
}

extern "C" {

qsb_status qsb_eigensolver_create(qsb_eigensolver** out, int64_t N, int n, int is_complex) {
    return qsb_eigensolver_create_ex(out, N, n, is_complex, QSB_PREC_FP64);
}

qsb_status qsb_eigensolver_create_ex(qsb_eigensolver** out, int64_t N, int n, int is_complex, qsb_precision precision) {
    if (!out) return fail(QSB_ERR_INVALID, "eigensolver_create: null handle pointer");
    *out = nullptr;
    if (N < 1 || n < 1) return fail(QSB_ERR_INVALID, "eigensolver_create: N and n must be >= 1");
    if (precision != QSB_PREC_FP64 && precision != QSB_PREC_MIXED)
        return fail(QSB_ERR_INVALID, "eigensolver_create: unknown precision");
    const int c2 = is_complex ? 2 : 1;
    if (precision == QSB_PREC_MIXED && 3 * n * c2 > 65535)
        return fail(QSB_ERR_INVALID, "eigensolver_create: too many bands for the mixed-precision Gram");
    qsb_eigensolver* es = new qsb_eigensolver();
    es->N = N;
    es->nmax = n;
    es->cplx = is_complex ? 1 : 0;
    es->mixed = precision == QSB_PREC_MIXED ? 1 : 0;
    es->L = (size_t)N * c2;
    auto cleanup = [&](qsb_status st) {
        qsb_eigensolver_destroy(es);
        return st;
    };
    if (cublasCreate(&es->blas) != CUBLAS_STATUS_SUCCESS) return cleanup(fail(QSB_ERR_CUDA, "cublasCreate failed"));
    if (cusolverDnCreate(&es->sol) != CUSOLVER_STATUS_SUCCESS)
        return cleanup(fail(QSB_ERR_CUDA, "cusolverDnCreate failed"));
    if (!es->mixed) {
        const size_t big = es->L * n * sizeof(double);
        double** bigs[5] = {&es->R, &es->AX, &es->AR, &es->AP, &es->TMP};
        for (double** p : bigs)
            if (cudaMalloc((void**)p, big) != cudaSuccess)
                return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: bundle allocation"));
    } else {
        const size_t big = es->L * n * sizeof(float);
        float** bigs[7] = {&es->X32, &es->R32, &es->P32, &es->AX32, &es->AR32, &es->AP32, &es->TMP32};
        for (float** p : bigs)
            if (cudaMalloc((void**)p, big) != cudaSuccess)
                return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: fp32 bundle allocation"));
        // split-BF16x3 Gram entries carry random errors ~ 2^-17 / sqrt(N) of the
        // (unit) diagonal: overlap directions weaker than about that are noise
        es->drop_tol = std::min(1e-5, std::max(1e-8, 1e-5 / std::sqrt((double)N)));
        const int pmax = 3 * n * c2;
        es->split_bytes = std::max(split_bf16_bytes(N, pmax), ozaki_split_bytes(N, pmax));
        es->gpart_bytes = std::max({gram_partial_bytes_bound(pmax, pmax, true), gram_partial_bytes_bound(n, 2 * n, false),
                                    ozaki_partial_bytes_bound(N, pmax, pmax, true),
                                    ozaki_partial_bytes_bound(N, n, 2 * n, false)});
        if (cudaMalloc(&es->su, es->split_bytes) != cudaSuccess || cudaMalloc(&es->sau, es->split_bytes) != cudaSuccess ||
            cudaMalloc(&es->gpart, es->gpart_bytes) != cudaSuccess ||
            cudaMalloc((void**)&es->T2, sizeof(double) * (size_t)pmax * pmax) != cudaSuccess ||
            cudaMalloc((void**)&es->rc32, sizeof(float) * (size_t)6 * 2 * n * n) != cudaSuccess ||
            cudaMalloc((void**)&es->rotw, sizeof(double) * ((size_t)(3 * n) * (3 * n) * c2 +
                                                            (size_t)2 * (3 * n * c2) * (2 * n * c2) + 2 * n * c2)) !=
                cudaSuccess ||
            cudaMalloc(&es->rotc, es->rotc_bytes = ozaki_rot_coef_bytes(3 * n * c2, 2 * n * c2)) != cudaSuccess)
            return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: mixed-precision workspace allocation"));
    }
    // overlap-basis pencil solve (both precisions: the mixed solver's route, the
    // FP64 solvers' fallback); FP64 Gram entries are exact to ~1e-16 of the
    // diagonal, so only directions below 1e-12 of the largest are dropped there
    if (cudaMalloc((void**)&es->svq, sizeof(double) * ((size_t)3 * (3 * n) * (3 * n) * c2 + 2 * (3 * n))) !=
        cudaSuccess)
        return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: pencil workspace allocation"));
    if (!es->mixed) es->drop_tol = 1e-12;
    if (!es->mixed && !is_complex && gram_small_doubles(n) > 0 &&
        cudaMalloc((void**)&es->gsmall, gram_small_doubles(n) * sizeof(double)) != cudaSuccess)
        return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: pencil tile allocation"));
    if (!es->mixed && is_complex) {
        const size_t mx = (size_t)3 * n;
        if (cudaMalloc((void**)&es->nxt, sizeof(double2) * (2 * mx * mx + (size_t)6 * n * n + 2 * mx * n)) !=
            cudaSuccess)
            return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: pencil update allocation"));
    }
    const int m = 3 * n;
    const size_t cm = (size_t)m * m * (is_complex ? 2 : 1);
    const size_t tsz = (size_t)(2 * n) * (2 * n);
    es->chunk = red_chunk_of(es->L, es->mixed != 0);
    es->nch = (int)((es->L + es->chunk - 1) / es->chunk);
    const size_t small = tsz + 2 * cm + m + (size_t)6 * 2 * n * n + 8 * (size_t)n + (size_t)n * es->nch;
    double* base = nullptr;
    if (cudaMalloc((void**)&base, small * sizeof(double)) != cudaSuccess)
        return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: matrix allocation"));
    es->T = base;
    es->Sa = es->T + tsz;
    es->Sb = es->Sa + cm;
    es->W = es->Sb + cm;
    es->rc = es->W + m;
    es->vec = es->rc + (size_t)6 * 2 * n * n;
    es->partial = es->vec + 8 * (size_t)n;
    if (cudaMalloc((void**)&es->info, 2 * sizeof(int)) != cudaSuccess)
        return cleanup(fail(QSB_ERR_NOMEM, "eigensolver: info allocation"));
    if (!es->mixed && !is_complex) {
        // TMP is not in use while a pencil is formed; where it is too small and there is no
        // memory for another one either, the form runs in what TMP holds or (gram_f64_i8_fits)
        // the pencil is formed by the library
        const size_t tmp = es->L * n * sizeof(double), own = gram_f64_i8_own_bytes(N, n, tmp);
        es->gi8 = es->TMP;
        es->gi8_bytes = tmp;
        if (own > 0) {
            if (cudaMalloc(&es->gi8_own, own) == cudaSuccess) {
                es->gi8 = es->gi8_own;
                es->gi8_bytes = own;
            } else {
                cudaGetLastError();
                es->gi8_own = nullptr;
            }
        }
    }
    *out = es;
    return QSB_OK;
}

qsb_status qsb_eigensolver_destroy(qsb_eigensolver* es) {
    if (!es) return QSB_OK;
    double* bigs[5] = {es->R, es->AX, es->AR, es->AP, es->TMP};
    for (double* p : bigs)
        if (p) cudaFree(p);
    float* b32[7] = {es->X32, es->R32, es->P32, es->AX32, es->AR32, es->AP32, es->TMP32};
    for (float* p : b32)
        if (p) cudaFree(p);
    void* mw[11] = {es->su,   es->sau,  es->gpart, es->T2,     es->rc32, es->svq,
                    es->rotw, es->rotc, es->nxt,   es->gsmall, es->gi8_own};
    for (void* p : mw)
        if (p) cudaFree(p);
    if (es->T) cudaFree(es->T);
    if (es->swork) cudaFree(es->swork);
    if (es->info) cudaFree(es->info);
    if (es->blas) cublasDestroy(es->blas);
    if (es->sol) cusolverDnDestroy(es->sol);
    delete es;
    return QSB_OK;
}

qsb_status qsb_eigensolver_set_hamiltonian(qsb_eigensolver* es, qsb_ham* ham, double gx, double gy, double gz) {
    if (!es) return fail(QSB_ERR_INVALID, "set_hamiltonian: null solver");
    if (ham && (int64_t)ham->N != es->N) return fail(QSB_ERR_INVALID, "set_hamiltonian: grid size differs from the solver's N");
    es->ham = ham;
    es->op = nullptr;
    es->user = nullptr;
    es->op32 = nullptr;
    es->user32 = nullptr;
    es->g[0] = gx; es->g[1] = gy; es->g[2] = gz;
    return QSB_OK;
}

qsb_status qsb_eigensolver_set_operator(qsb_eigensolver* es, qsb_apply_fn op, void* user) {
    if (!es || !op) return fail(QSB_ERR_INVALID, "set_operator: null argument");
    es->ham = nullptr;
    es->op = op;
    es->user = user;
    es->op32 = nullptr;
    es->user32 = nullptr;
    return QSB_OK;
}

qsb_status qsb_eigensolver_set_operator_f32(qsb_eigensolver* es, qsb_apply_f32_fn op, void* user) {
    if (!es || !op) return fail(QSB_ERR_INVALID, "set_operator_f32: null argument");
    es->ham = nullptr;
    es->op = nullptr;
    es->user = nullptr;
    es->op32 = op;
    es->user32 = user;
    return QSB_OK;
}

qsb_status qsb_eigensolver_set_drop_tolerance(qsb_eigensolver* es, double tol) {
    if (!es) return fail(QSB_ERR_INVALID, "set_drop_tolerance: null solver");
    if (!(tol > 0.0 && tol < 1.0)) return fail(QSB_ERR_INVALID, "set_drop_tolerance: needs 0 < tol < 1");
    es->drop_tol = tol;
    return QSB_OK;
}

qsb_status qsb_eigensolver_set_gram_kind(qsb_eigensolver* es, qsb_gram_kind kind) {
    if (!es) return fail(QSB_ERR_INVALID, "set_gram_kind: null solver");
    if (kind != QSB_GRAM_BF16X3 && kind != QSB_GRAM_BF16X4 && kind != QSB_GRAM_INT8_OZAKI)
        return fail(QSB_ERR_INVALID, "set_gram_kind: unknown kind");
    es->gram_kind = kind;
    return QSB_OK;
}

qsb_status qsb_eigensolver_set_pencil_update(qsb_eigensolver* es, int mode) {
    if (!es || (mode != 0 && mode != 1)) return fail(QSB_ERR_INVALID, "eigensolver_set_pencil_update: bad arguments");
    es->pencil_update = mode;
    return QSB_OK;
}

qsb_status qsb_eigensolver_pencil_stats(const qsb_eigensolver* es, int* full, int* steady) {
    if (!es || !full || !steady) return fail(QSB_ERR_INVALID, "eigensolver_pencil_stats: bad arguments");
    *full = es->last_full;
    *steady = es->last_steady;
    return QSB_OK;
}

qsb_status qsb_eigensolver_solve_stats(const qsb_eigensolver* es, int* cholesky_solves, int* overlap_basis_solves) {
    if (!es) return fail(QSB_ERR_INVALID, "solve_stats: null solver");
    if (cholesky_solves) *cholesky_solves = es->last_chol;
    if (overlap_basis_solves) *overlap_basis_solves = es->last_svqb;
    return QSB_OK;
}

qsb_status qsb_eigensolver_overlap_stats(const qsb_eigensolver* es, int* max_dropped, double* min_kept_ratio,
                                         double* drop_tolerance) {
    if (!es) return fail(QSB_ERR_INVALID, "overlap_stats: null solver");
    if (max_dropped) *max_dropped = es->last_dropped;
    if (min_kept_ratio) *min_kept_ratio = es->last_min_kept;
    if (drop_tolerance) *drop_tolerance = es->drop_tol;
    return QSB_OK;
}

qsb_status qsb_eigensolver_last_stats(const qsb_eigensolver* es, int* iterations, int* rolled_back) {
    if (!es) return fail(QSB_ERR_INVALID, "last_stats: null solver");
    if (iterations) *iterations = es->last_iters;
    if (rolled_back) *rolled_back = es->last_rollback;
    return QSB_OK;
}

// ---------------------------------------------------------------------------
// LOBPCG::Eigen_z_multi_mpi (source/lobpcg_z_multi_mpi.h:1732-2852), one rank.
// ---------------------------------------------------------------------------
qsb_status qsb_lobpcg_z(qsb_eigensolver* es, double dVol, int n, int iter_max, double* eigen_values, double* X,
                        double* keep, int* p_num_fix, double residual_threshold, int scf_step, void* stream) {
    if (!es || !es->cplx) return fail(QSB_ERR_INVALID, "lobpcg_z: needs a complex eigensolver context");
    if (!es->ham && !(es->mixed ? (void*)es->op32 : (void*)es->op))
        return fail(QSB_ERR_STATE, es->mixed ? "lobpcg_z: no fp32 operator or Hamiltonian set (mixed precision)"
                                             : "lobpcg_z: no operator or Hamiltonian set");
    if (n < 1 || n > es->nmax || !X || !keep || !eigen_values || !p_num_fix || !(dVol > 0))
        return fail(QSB_ERR_INVALID, "lobpcg_z: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    QSB_BLAS_TRY(cublasSetStream(es->blas, s));
    QSB_SOLVER_TRY(cusolverDnSetStream(es->sol, s));
    es->last_iters = 0;
    es->last_rollback = 0;
    es->last_dropped = 0;
    es->last_chol = 0;
    es->last_svqb = 0;
    es->last_min_kept = 1.0;
    es->last_full = 0;
    es->last_steady = 0;
    if (es->mixed)
        return lobpcg_z_mixed(es, dVol, n, iter_max, eigen_values, X, keep, p_num_fix, residual_threshold, scf_step, s);
    const size_t L = es->L;
    auto band = [&](double* base, int b) { return base + (size_t)b * L; };
    double* eps_d = es->vec;             // n
    double* nrm_d = es->vec + n;         // n
    double* scl_d = es->vec + 2 * n;     // n
    std::vector<double> eps(n), nr(n), nx(n), scl(n);

    int num_fix = std::max(0, std::min(*p_num_fix, n));
    int num_active = n - num_fix;
    const int head0 = num_fix;

    // scale X by sqrt(dV) (:1851)
    QSB_TRY(seg_scale_by(es, n, X, nullptr, std::sqrt(dVol), s));
    // AX = A X for the active bands (:1863)
    QSB_TRY(apply_op(es, num_active, band(X, head0), band(es->AX, head0), s));
    // eps_k = <x_k|Ax_k> (:1873), r = Ax - eps x, ||r||^2 (:1895)
    QSB_TRY(seg_dot(es, num_active, band(X, head0), band(es->AX, head0), 1.0, eps_d + head0, s));
    QSB_TRY(seg_residual(es, num_active, band(es->R, head0), band(es->AX, head0), band(X, head0), eps_d + head0,
                         nrm_d + head0, 1.0, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(eps.data() + head0, eps_d + head0, sizeof(double) * num_active, cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaMemcpyAsync(nr.data() + head0, nrm_d + head0, sizeof(double) * num_active, cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    for (int k = head0; k < n; ++k)
        if (!std::isfinite(eps[k]) || !std::isfinite(nr[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_z: non-finite Rayleigh quotient");
    // soft locking (:1962-1986): fix the leading bands whose residual is below threshold
    {
        int fix_pos = n;
        const double th2 = residual_threshold * residual_threshold;
        for (int k = head0; k < n; ++k)
            if (th2 < nr[k]) { fix_pos = k; break; }
        const int org_active = num_active;
        num_fix = std::min(fix_pos, n / 2);
        num_active = n - num_fix;
        if (num_active != org_active) *p_num_fix = num_fix;
        // newly fixed bands keep the eigenvalues passed in (only active ones are written back, :2846-2848)
        if (iter_max < 1) {
            QSB_TRY(seg_scale_by(es, n, X, nullptr, 1.0 / std::sqrt(dVol), s));
            return QSB_OK;
        }
        const int head = num_fix;
        const int N_ = num_active;
        const bool is_first_time = (scf_step == 0);
        if (is_first_time) {
            QSB_CUDA_TRY(cudaMemsetAsync(keep, 0, sizeof(double) * L * n, s));
            QSB_CUDA_TRY(cudaMemsetAsync(es->AP, 0, sizeof(double) * L * n, s));
        } else {
            if (num_active != org_active && num_fix > 0) {
                // VectorOrthogonalization of P against X_fix (:2062, :1637-1723)
                QSB_TRY(gemm_tn(es, 2 * num_fix, 2 * N_, X, band(keep, head), es->T));
                pack_orth<<<dim3((num_fix + 127) / 128, N_), 128, 0, s>>>(es->T, num_fix, N_);
                QSB_TRY(gemm_nn(es, 2 * num_fix, 2 * N_, -1.0, X, es->T, 1.0, band(keep, head), (int)es->N));
            }
            QSB_TRY(apply_op(es, N_, band(keep, head), band(es->AP, head), s));
        }
        // if the active set moved, the residuals of newly active bands are in R already;
        // the Rayleigh quotients of the active bands drive the loop
        int iter;
        bool large_difference = false;
        bool have_next = false;   // X'/P' pencil blocks of this iteration were formed by the update
        for (iter = 0; iter < iter_max; ++iter) {
            // orthogonalize R to X_fix (:2080)
            if (num_fix > 0) {
                QSB_TRY(gemm_tn(es, 2 * num_fix, 2 * N_, X, band(es->R, head), es->T));
                pack_orth<<<dim3((num_fix + 127) / 128, N_), 128, 0, s>>>(es->T, num_fix, N_);
                QSB_TRY(gemm_nn(es, 2 * num_fix, 2 * N_, -1.0, X, es->T, 1.0, band(es->R, head), (int)es->N));
            }
            QSB_TRY(apply_op(es, N_, band(es->R, head), band(es->AR, head), s));   // AR = A R (:2084)
            const bool use_p = !(is_first_time && iter == 0);
            const int nblk = use_p ? 3 : 2;
            const int m = nblk * N_;
            const double* U[3] = {band(X, head), band(es->R, head), band(keep, head)};
            const double* AU[3] = {band(es->AX, head), band(es->AR, head), band(es->AP, head)};
            // Hermitian pencil (MakeMatrix_z_blas, :300-558): upper blocks, lower = conj.
            // Between full recomputes (every S_MAT_REST_LIMIT = 6 iterations, :1808,
            // :2091-2101) only X^H A R, R^H A R, R^H A P and R^H R come from the grid;
            // the X and P blocks are the previous iteration's update (:2782).
            if (have_next && use_p) {
                QSB_TRY(gram_block(es, U[0], AU[1], N_, es->Sa, m, 0, 1, 1.0, s));
                QSB_TRY(gram_block(es, U[1], AU[1], N_, es->Sa, m, 1, 1, 1.0, s));
                QSB_TRY(gram_block(es, U[1], AU[2], N_, es->Sa, m, 1, 2, 1.0, s));
                QSB_TRY(gram_block(es, U[1], U[1], N_, es->Sb, m, 1, 1, 1.0, s));
                QSB_TRY(put_next_blocks(es, N_, m, s));
                ++es->last_steady;
            } else {
                for (int I = 0; I < nblk; ++I)
                    for (int J = I; J < nblk; ++J) {
                        QSB_TRY(gram_block(es, U[I], AU[J], N_, es->Sa, m, I, J, 1.0, s));
                        QSB_TRY(gram_block(es, U[I], U[J], N_, es->Sb, m, I, J, 1.0, s));
                    }
                ++es->last_full;
            }
            have_next = false;
            // the next iteration updates its X/P blocks from this pencil unless it
            // is the last one or a full recompute
            const bool update_next = es->pencil_update && iter + 1 < iter_max && (iter + 1) % 6 != 0;
            if (update_next) {
                const size_t mmax = (size_t)3 * es->nmax;
                QSB_CUDA_TRY(cudaMemcpyAsync(es->nxt, es->Sa, sizeof(double2) * (size_t)m * m, cudaMemcpyDeviceToDevice, s));
                QSB_CUDA_TRY(cudaMemcpyAsync((double2*)es->nxt + mmax * mmax, es->Sb, sizeof(double2) * (size_t)m * m,
                                             cudaMemcpyDeviceToDevice, s));
            }
            QSB_TRY(solve_pencil_fp64(es, m, N_, s));   // ZHEGVD (:2254-2263 / :2492-2511)
            QSB_TRY(make_coefficients(es, N_, m, nblk, s));
            // P' = R Cr + P Cp (into TMP), P = TMP; TMP += X Cx  (NextVector_z2)
            QSB_TRY(rotate_complex(es, N_, es->TMP, U[1], 1, 0.0, s));
            if (use_p) QSB_TRY(rotate_complex(es, N_, es->TMP, U[2], 2, 1.0, s));
            QSB_CUDA_TRY(cudaMemcpyAsync(band(keep, head), es->TMP, sizeof(double) * L * N_, cudaMemcpyDeviceToDevice, s));
            QSB_TRY(rotate_complex(es, N_, es->TMP, U[0], 0, 1.0, s));
            // ||X'||^2 (:2570) and the rollback test (:2611-2666)
            QSB_TRY(seg_dot(es, N_, es->TMP, es->TMP, 1.0, nrm_d, s));
            QSB_CUDA_TRY(cudaMemcpyAsync(nx.data(), nrm_d, sizeof(double) * N_, cudaMemcpyDeviceToHost, s));
            std::vector<double> w(N_);                       // the Ritz values, in the same wait
            QSB_CUDA_TRY(cudaMemcpyAsync(w.data(), es->W, sizeof(double) * N_, cudaMemcpyDeviceToHost, s));
            QSB_CUDA_TRY(cudaStreamSynchronize(s));
            double maxdiff = 0.0;
            for (int k = 0; k < N_; ++k) {
                if (!std::isfinite(nx[k])) return fail(QSB_ERR_NUMERIC, "lobpcg_z: non-finite vector norm");
                maxdiff = std::max(maxdiff, std::fabs(1.0 - nx[k]));
            }
            large_difference = maxdiff > 1.0e-3;   // LIMIT_Z_NORM_X_FOR_RESET_MATRIX (:101)
            if (large_difference) {
                // keep X, P <- R, undo the scaling with the previous norms
                // (the reference rescales the kept X with the norms of the rejected X', :2651)
                es->last_rollback = 1;
                QSB_CUDA_TRY(cudaMemcpyAsync(band(keep, head), band(es->R, head), sizeof(double) * L * N_,
                                             cudaMemcpyDeviceToDevice, s));
                if (num_fix > 0) QSB_TRY(seg_scale_by(es, num_fix, X, nullptr, 1.0 / std::sqrt(dVol), s));
                for (int k = 0; k < N_; ++k) scl[k] = 1.0 / std::sqrt(nx[k] * dVol);
                QSB_CUDA_TRY(cudaMemcpyAsync(scl_d, scl.data(), sizeof(double) * N_, cudaMemcpyHostToDevice, s));
                QSB_TRY(seg_scale_by(es, N_, band(X, head), scl_d, 0.0, s));
                ++iter;
                break;
            }
            QSB_CUDA_TRY(cudaMemcpyAsync(band(X, head), es->TMP, sizeof(double) * L * N_, cudaMemcpyDeviceToDevice, s));
            for (int k = 0; k < N_; ++k) eps[head + k] = w[k];
            const bool final_step = (iter + 1 == iter_max);
            if (!final_step) {
                // AP' = AR Cr + AP Cp; AX' = AX Cx + AP'  (NextVector_z2 on A-bundles, :2718)
                QSB_TRY(rotate_complex(es, N_, es->TMP, AU[1], 1, 0.0, s));
                if (use_p) QSB_TRY(rotate_complex(es, N_, es->TMP, AU[2], 2, 1.0, s));
                QSB_CUDA_TRY(cudaMemcpyAsync(band(es->AP, head), es->TMP, sizeof(double) * L * N_,
                                             cudaMemcpyDeviceToDevice, s));
                QSB_TRY(rotate_complex(es, N_, es->TMP, AU[0], 0, 1.0, s));
                QSB_CUDA_TRY(cudaMemcpyAsync(band(es->AX, head), es->TMP, sizeof(double) * L * N_,
                                             cudaMemcpyDeviceToDevice, s));
                // R = AX - eps X (:2750)
                QSB_CUDA_TRY(cudaMemcpyAsync(eps_d, w.data(), sizeof(double) * N_, cudaMemcpyHostToDevice, s));
                QSB_TRY(seg_residual(es, N_, band(es->R, head), band(es->AX, head), band(X, head), eps_d, nullptr, 1.0, s));
                if (update_next) {
                    // NextMatrix_z (:2782): the next pencil's X'/P' blocks (S0 saved before the solve)
                    QSB_TRY(next_pencil_blocks(es, N_, m, s));
                    have_next = true;
                }
            } else {
                // undo the scaling: fixed bands by 1/sqrt(dV), active by 1/sqrt(|x|^2 dV) (:2792-2803)
                if (num_fix > 0) QSB_TRY(seg_scale_by(es, num_fix, X, nullptr, 1.0 / std::sqrt(dVol), s));
                for (int k = 0; k < N_; ++k) scl[k] = 1.0 / std::sqrt(nx[k] * dVol);
                QSB_CUDA_TRY(cudaMemcpyAsync(scl_d, scl.data(), sizeof(double) * N_, cudaMemcpyHostToDevice, s));
                QSB_TRY(seg_scale_by(es, N_, band(X, head), scl_d, 0.0, s));
            }
        }
        es->last_iters = iter;
        for (int k = head; k < n; ++k) eigen_values[k] = eps[k];
        QSB_CUDA_TRY(cudaStreamSynchronize(s));
    }
    return QSB_OK;
}

// ---------------------------------------------------------------------------
// EigenLOBPCG_d_multi (source/lobpcg_d_multi.h:23-545).
// ---------------------------------------------------------------------------
qsb_status qsb_lobpcg_d(qsb_eigensolver* es, double dVol, int n, int iter_max, double* eigen_values, double* X,
                        double* keep, int is_first_time, void* stream) {
    if (!es || es->cplx) return fail(QSB_ERR_INVALID, "lobpcg_d: needs a real eigensolver context");
    if (!es->ham && !(es->mixed ? (void*)es->op32 : (void*)es->op))
        return fail(QSB_ERR_STATE, es->mixed ? "lobpcg_d: no fp32 operator or Hamiltonian set (mixed precision)"
                                             : "lobpcg_d: no operator or Hamiltonian set");
    if (n < 1 || n > es->nmax || !X || !keep || !eigen_values || !(dVol > 0))
        return fail(QSB_ERR_INVALID, "lobpcg_d: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    QSB_BLAS_TRY(cublasSetStream(es->blas, s));
    QSB_SOLVER_TRY(cusolverDnSetStream(es->sol, s));
    es->last_iters = 0;
    es->last_rollback = 0;
    es->last_dropped = 0;
    es->last_chol = 0;
    es->last_svqb = 0;
    es->last_min_kept = 1.0;
    if (es->mixed) return lobpcg_d_mixed(es, dVol, n, iter_max, eigen_values, X, keep, is_first_time, s);
    const size_t L = es->L;
    double* eps_d = es->vec;
    double* nrm_d = es->vec + n;
    // eps, |r|^2, |x|^2, |p|^2 next to each other (one copy to the host per iteration), then
    // the factors of x and p, and the scale of the initial normalisations
    double* xn_d = es->vec + 2 * n;
    double* pn_d = es->vec + 3 * n;
    double* sx_d = es->vec + 4 * n;
    double* sp_d = es->vec + 5 * n;
    std::vector<double> v(n);

    auto to_host = [&](std::vector<double>& h) -> qsb_status {      // the first h.size() of es->vec
        QSB_CUDA_TRY(cudaMemcpyAsync(h.data(), es->vec, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
        QSB_CUDA_TRY(cudaStreamSynchronize(s));
        return QSB_OK;
    };
    auto normalize = [&](double* B, double* norms) -> qsb_status {
        // Normalize (source/vecmath.h:128-134): x /= sqrt(|x|^2 dV); the norms are looked at
        // in the wait for the Rayleigh quotients below
        QSB_TRY(seg_norms(es, n, B, dVol, norms, sx_d, s));
        return seg_scale_by(es, n, B, sx_d, 0.0, s);
    };

    // initial residual (:63-90)
    QSB_TRY(normalize(X, xn_d));
    QSB_TRY(apply_op(es, n, X, es->AX, s));
    if (is_first_time) {
        QSB_CUDA_TRY(cudaMemsetAsync(keep, 0, sizeof(double) * L * n, s));
        QSB_CUDA_TRY(cudaMemsetAsync(es->AP, 0, sizeof(double) * L * n, s));
    } else {
        QSB_TRY(apply_op(es, n, keep, es->AP, s));
    }
    QSB_TRY(seg_dot(es, n, X, es->AX, dVol, eps_d, s));
    QSB_TRY(seg_residual(es, n, es->R, es->AX, X, eps_d, nullptr, 1.0, s));
    QSB_TRY(normalize(es->R, pn_d));
    std::vector<double> eps(n);
    {
        // an infinite |x|^2 or |r|^2 (its band finite, so the quotients can be) is refused here as
        // any other: the pencil of such a band is NaN
        std::vector<double> first(4 * (size_t)n);       // eps, (not yet written), |x|^2, |r|^2
        QSB_TRY(to_host(first));
        for (int k = 0; k < n; ++k)
            if (!std::isfinite(first[k]) || !std::isfinite(first[2 * n + k]) || !std::isfinite(first[3 * n + k]))
                return fail(QSB_ERR_NUMERIC, "lobpcg_d: non-finite value");
        std::copy(first.begin(), first.begin() + n, eps.begin());
    }
    for (int k = 0; k < n; ++k) eigen_values[k] = eps[k];

    bool gi8 = !es->gsmall && gram_f64_i8_fits(es->N, n, es->gi8_bytes);
    int iter;
    for (iter = 0; iter < iter_max; ++iter) {
        QSB_TRY(apply_op(es, n, es->R, es->AR, s));
        const bool two = is_first_time && iter == 0;
        const int nblk = two ? 2 : 3;
        const int m = nblk * n;
        const double* U[3] = {X, es->R, keep};
        const double* AU[3] = {es->AX, es->AR, es->AP};
        if (es->gsmall) {
            QSB_TRY(gram_small(es->N, n, nblk, U, AU, dVol, es->Sa, es->Sb, es->gsmall, s));
        } else if (gi8) {
            QSB_CUDA_TRY(cudaMemsetAsync(es->info + 1, 0, sizeof(int), s));
            QSB_TRY(gram_f64_i8(es->N, n, nblk, U, AU, dVol, es->Sa, es->Sb, es->gi8, es->gi8_bytes, es->info + 1, s));
            // the products' waits are bounded: a pencil that they did not finish is formed
            // by the library instead, here and for the rest of the call (the device error
            // word says so too).  Looked at before anything is solved: the library's dense
            // solvers may never come back from a pencil of zeros.
            int gave_up = 0;
            QSB_CUDA_TRY(cudaMemcpyAsync(&gave_up, es->info + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
            QSB_CUDA_TRY(cudaStreamSynchronize(s));
            gi8 = gave_up == 0;
        }
        if (!es->gsmall && !gi8) {
            for (int I = 0; I < nblk; ++I)
                for (int J = I; J < nblk; ++J) {
                    QSB_TRY(gram_block(es, U[I], AU[J], n, es->Sa, m, I, J, dVol, s));
                    QSB_TRY(gram_block(es, U[I], U[J], n, es->Sb, m, I, J, dVol, s));
                }
        }
        QSB_TRY(solve_pencil_fp64(es, m, n, s));   // DSYGVX, lowest n (:209, :284)
        QSB_TRY(make_coefficients(es, n, m, nblk, s));
        // P = R Cr (+ P Cp); X = X Cx + P; same for A-bundles (:226-365), each renormalised
        // as it leaves TMP (x, p and with their factors Ax, Ap, :493-505), and eps = <x|Ax> dV
        // (:507) taken in Ax's pass.  The norms stay on the device until the iteration's end.
        QSB_TRY(rotate_real(es, n, es->TMP, es->R, 1, 0.0, s));
        if (!two) QSB_TRY(rotate_real(es, n, es->TMP, keep, 2, 1.0, s));
        QSB_TRY(seg_norms(es, n, es->TMP, dVol, pn_d, sp_d, s));
        QSB_TRY(seg_scaled_copy(es, n, es->TMP, keep, sp_d, nullptr, 0.0, nullptr, s));
        QSB_TRY(rotate_real(es, n, es->TMP, X, 0, 1.0, s));
        QSB_TRY(seg_norms(es, n, es->TMP, dVol, xn_d, sx_d, s));
        QSB_TRY(seg_scaled_copy(es, n, es->TMP, X, sx_d, nullptr, 0.0, nullptr, s));
        QSB_TRY(rotate_real(es, n, es->TMP, es->AR, 1, 0.0, s));
        if (!two) QSB_TRY(rotate_real(es, n, es->TMP, es->AP, 2, 1.0, s));
        QSB_TRY(seg_scaled_copy(es, n, es->TMP, es->AP, sp_d, nullptr, 0.0, nullptr, s));
        QSB_TRY(rotate_real(es, n, es->TMP, es->AX, 0, 1.0, s));
        QSB_TRY(seg_scaled_copy(es, n, es->TMP, es->AX, sx_d, X, dVol, eps_d, s));
        // r = Ax - eps x; ||r||^2 dV (:507-513)
        QSB_TRY(seg_residual(es, n, es->R, es->AX, X, eps_d, nrm_d, dVol, s));
        std::vector<double> all(4 * (size_t)n);      // eps, |r|^2, |x|^2, |p|^2
        QSB_TRY(to_host(all));
        for (double q : all)
            if (!std::isfinite(q)) return fail(QSB_ERR_NUMERIC, "lobpcg_d: non-finite value");
        std::copy(all.begin(), all.begin() + n, eps.begin());
        std::copy(all.begin() + n, all.begin() + 2 * n, v.begin());
        double rmax = 0.0;
        for (int k = 0; k < n; ++k) {
            eigen_values[k] = eps[k];
            rmax = std::max(rmax, v[k]);
        }
        if (rmax < 1.0e-10 * dVol) { ++iter; break; }   // :525
    }
    es->last_iters = iter;
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    return QSB_OK;
}

}  // extern "C"
