// The real Rayleigh-Ritz pencil of few bands in two launches: all upper tiles of
// S = dV U^T U and A = dV U^T (AU), U = [X R P], for up to 96 columns.
//
// Why: block by block this is 12 DGEMMs of n x n x N with their split-K
// reductions and assemblies, 36 launches of 2 to 7 microseconds around products
// that take a few: 0.17 ms per solver iteration at 32^3 x 16 bands, where a pass
// over the six bundles takes 5 us from L2.  Here (21 + 5 us there) one kernel reads
// every bundle once and forms both matrices from shared memory on the FP64 tensor cores
// (mma.m8n8k4), a second one sums the CTAs' tiles in a fixed order and writes the
// pencil with its mirror.
//
// CTA: chunks of GS_KC grid points, [column][point] in shared memory at a pitch of
// GS_KC + 4 (a fragment's 8 columns x 4 points touch every bank once); the 8 x 8
// tiles of both matrices are dealt to the warps, whose sums stay in registers over
// all of the CTA's chunks.
#include "qsb_internal.h"

#include <algorithm>

namespace qsb {
namespace {

constexpr int GS_KC = 64;
constexpr int GS_PITCH = GS_KC + 4;
constexpr int GS_WARPS = 16;
constexpr int GS_MAX_COLS = 96;
constexpr int GS_CTAS = 148;
constexpr int GS_MAXT = 10;      // tiles per warp: 2 * 12 * 13 / 2 tiles over 16 warps

struct GsBundles {
    const double* u[3];
    const double* au[3];
};

__global__ void __launch_bounds__(GS_WARPS * 32, 1)
gram_small_kernel(GsBundles b, int n, int p, int pt, int64_t N, double* __restrict__ partial) {
    extern __shared__ __align__(16) double gs_sm[];      // U columns [8 pt][PITCH], then AU columns
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nt = pt * (pt + 1) / 2, cols = 8 * pt;
    // this warp's tiles: q-th is tile warp + q GS_WARPS of [S tiles, A tiles]
    int ao[GS_MAXT], bo[GS_MAXT];
    double acc[GS_MAXT][2];
#pragma unroll
    for (int q = 0; q < GS_MAXT; ++q) {
        int k = warp + q * GS_WARPS;
        ao[q] = bo[q] = -1;
        acc[q][0] = acc[q][1] = 0.0;
        if (k < 2 * nt) {
            const int a = k >= nt;
            k -= a * nt;
            int tj = 0;
            while (k > tj) k -= ++tj;                    // tiles in column order: (0,0) (0,1) (1,1) ...
            ao[q] = (8 * k + (lane >> 2)) * GS_PITCH + (lane & 3);
            bo[q] = (a * cols + 8 * tj + (lane >> 2)) * GS_PITCH + (lane & 3);
        }
    }
    const int64_t chunks = (N + GS_KC - 1) / GS_KC;
    for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int64_t g0 = c * GS_KC;
        __syncthreads();                                 // the last chunk is no longer read
#pragma unroll 4
        for (int col = warp; col < 2 * cols; col += GS_WARPS) {
            const int k = col < cols ? col : col - cols;
            const double* src = nullptr;
            if (k < p) {
                const int blk = k / n;
                src = (col < cols ? b.u[blk] : b.au[blk]) + (size_t)(k - blk * n) * N;
            }
#pragma unroll
            for (int h = 0; h < GS_KC; h += 32) {
                const int64_t g = g0 + h + lane;
                gs_sm[col * GS_PITCH + h + lane] = src && g < N ? __ldg(src + g) : 0.0;
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < GS_MAXT; ++q) {
            if (ao[q] < 0) continue;
            const double* a = gs_sm + ao[q];
            const double* v = gs_sm + bo[q];
#pragma unroll
            for (int k = 0; k < GS_KC; k += 4)
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                             : "+d"(acc[q][0]), "+d"(acc[q][1])
                             : "d"(a[k]), "d"(v[k]));
        }
    }
#pragma unroll
    for (int q = 0; q < GS_MAXT; ++q) {
        const int k = warp + q * GS_WARPS;
        if (k < 2 * nt)
            *reinterpret_cast<double2*>(partial + ((size_t)blockIdx.x * 2 * nt + k) * 64 + 2 * lane) =
                make_double2(acc[q][0], acc[q][1]);
    }
}

// Sum of the CTAs' tiles (eight lanes to an entry, each its CTAs in order, then the
// lanes pairwise), scaled, to the pencil's upper triangle and its mirror.
__global__ void gram_small_reduce_kernel(const double* __restrict__ partial, int ctas, int m, int pt, double scale,
                                         double* __restrict__ A, double* __restrict__ B) {
    const int nt = pt * (pt + 1) / 2;
    const int id = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, l = threadIdx.x & 7;
    if (id >= 2 * nt * 64) return;                       // whole groups of eight
    double s = 0.0;
#pragma unroll 4
    for (int c = l; c < ctas; c += 8) s += partial[(size_t)c * 2 * nt * 64 + id];
    const unsigned mask = 0xffu << (threadIdx.x & 24);
    s += __shfl_xor_sync(mask, s, 4);
    s += __shfl_xor_sync(mask, s, 2);
    s += __shfl_xor_sync(mask, s, 1);
    if (l != 0) return;
    int k = id >> 6;
    const int e = id & 63;
    double* M = k < nt ? B : A;
    if (k >= nt) k -= nt;
    int tj = 0;
    while (k > tj) k -= ++tj;
    const int r = 8 * k + (e >> 3), c = 8 * tj + (e & 7);
    if (r > c || c >= m) return;
    const double v = s * scale;
    M[r + (size_t)m * c] = v;
    M[c + (size_t)m * r] = v;
}

}  // namespace

// doubles of the partial tiles for up to 3 n columns (0: more than this form takes)
size_t gram_small_doubles(int n) {
    if (3 * n > GS_MAX_COLS) return 0;
    const int pt = (3 * n + 7) / 8;
    return (size_t)GS_CTAS * pt * (pt + 1) * 64;
}

// A = scale U^T AU and B = scale U^T U (both m x m, full), m = nblk * n columns
qsb_status gram_small(int64_t N, int n, int nblk, const double* const* U, const double* const* AU, double scale,
                      double* A, double* B, double* partial, cudaStream_t s) {
    GsBundles b{};
    for (int k = 0; k < nblk; ++k) {
        b.u[k] = U[k];
        b.au[k] = AU[k];
    }
    const int p = nblk * n, pt = (p + 7) / 8, tiles = pt * (pt + 1);
    const int ctas = (int)std::min<int64_t>(GS_CTAS, (N + GS_KC - 1) / GS_KC);
    const int smem = 2 * 8 * pt * GS_PITCH * (int)sizeof(double);
    QSB_TRY(allow_shared_memory(gram_small_kernel));
    gram_small_kernel<<<ctas, GS_WARPS * 32, smem, s>>>(b, n, p, pt, N, partial);
    gram_small_reduce_kernel<<<(tiles * 64 * 8 + 255) / 256, 256, 0, s>>>(partial, ctas, p, pt, scale, A, B);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

}  // namespace qsb
