// The real FP64 Rayleigh-Ritz pencil of many bands on the INT8 tensor cores: all
// upper tiles of S = dV U^T U and A = dV U^T (AU), U = [X R P] gathered columns,
// from products that are exact up to a fixed fraction of the columns' maxima.
//
// Splitting: column c becomes integers x = rint(u 2^e_c), 2^54 <= max |x| < 2^55,
// each written as seven balanced base-256 digits
//   x = sum_i d_i 256^(6-i),  -128 <= d_i <= 127.
//   U^T V = 2^(-e_u - e_v) sum_l 256^(12-l) D_l,  D_l = sum_{i+j=l} d_i^T d'_j
// The 34 products with i + j <= 7 and the product d_4^T d'_4 are summed without
// rounding in INT32 (7 * 2^14 * K < 2^31 for the at most 18688 points of a CTA), a
// level at a time.
//
// Precision: what is kept is relative to a column's largest value, not to each
// element: an element below a quarter of it has fewer bits here than in FP64, with
// an error of at most 2^-55 max|u|.  The products left out are each below 2^-64 of
// max|u| max|v| at a point.  Their signs alternate from point to point, except where
// a column meets itself (or its double) digit on equal digit: sum d_4^2, without which
// <u|u> of a column with one dominant point was low by N 2^-66, 5e-14 at 96^3 and
// 2e-13 at 144^3, is therefore one of the products; the next, sum d_5^2, is below
// N 2^-82.  Errors of entries relative to |u||v| in exact integers at 96^3 and 144^3:
//   one point at 1, the others uniform within 1e-2 to 1e-6, or a Gaussian one
//     grid spacing wide on a tail of 1e-4:        at most 4e-16 (FP64 sums up to 6e-15)
//   the others within 10 % of one value:           at most 3e-15 (9e-15)
//   uniform, waves, wide Gaussians, exponentials: at most 3e-17 (1e-14)
//   one point at 1, all others the same number (signs alternate nowhere):
//                                                 up to 3e-13 (6e-13; 5e-16 where the
//                                                 partner's digits do vary, 5e-14 here)
//
// Why: the FP64 units give 37 TFLOP/s, and a library product of 128 x 128 columns
// over 96^3 points, 29 GFLOP, takes 1.0 ms; a pencil of 384 columns is 12 of them,
// three with a lower triangle that no one needs.  Pencil of 3 n columns, library ->
// here: n = 128, 96^3 12.9 -> 6.8 ms (maxima 0.8, digits 1.7, products 4.3); n = 200,
// 64^3 11.6 -> 4.9; n = 48, 96^3 3.8 -> 3.3 (144 columns are padded to 256); n = 33,
// 32^3 0.25 -> 0.14 ms.  The digits are bound by their 15 bytes moved per element,
// the products by the integer MMA rate and the operands' way from L2 to shared memory (tensor
// pipe 65 % busy in the levels 4 to 7 and 52 % in 0 to 3, operands at 4.3 to 4.6 TB/s;
// 96^3 x 48 bands).
//
// The digits of one chunk of grid points are laid out at a time, as many as the
// workspace holds (the solver's temporary bundle, free while a pencil is formed),
// [digit][column][point]; a chunk takes three launches of CTAs with 128 x 128 output
// tiles, for d_4 d'_4, the levels 4 to 7 and 0 to 3, because no more than four INT32
// accumulators (128 TMEM columns each) fit the 512 columns of an SM.  Pipeline per
// CTA as in gram_i8.cu: warp 0 lane 0 streams 64-point stages of the digit tiles
// with 2-D TMA copies (64-byte swizzle), warp 1 lane 0 issues the MMAs, the four
// warps combine the levels into FP64 partial tiles.  All waits are bounded; a wait
// that runs out sets the device error word and the caller's own word, and the CTA
// drains, frees TMEM and returns.
#include "qsb_internal.h"
#include "tc_common.cuh"

#include <algorithm>
#include <cstdlib>

namespace qsb {
namespace {
using namespace tc;

constexpr int GF_T = 128;                        // output tile
constexpr int GF_K = 64;                         // points per stage (one 64-byte swizzle row)
constexpr int GF_DIGITS = 7;
constexpr int GF_TILE = GF_T * GF_K;             // 8 KB per digit tile
constexpr int GF_THREADS = 128;
constexpr int GF_MAX_STAGES = 18688 / GF_K;      // 7 * 128 * 128 * 18688 < 2^31
constexpr unsigned GF_WAIT_LIMIT = 1u << 22;
constexpr unsigned GF_DRAIN_LIMIT = 1u << 16;
constexpr int GF_PASSES = 3;                     // launches per chunk of points
constexpr int ERR_GEMM_TIMEOUT = 2;
constexpr size_t GF_DIGIT_BYTES = (size_t)1 << 30;   // most digits laid out at a time
constexpr size_t GF_OWN_BYTES = (size_t)192 << 20;   // largest workspace of a solver's own

// One launch: the products of levels LO..HI of the digits FIRST..LAST of both operands
template <int LO, int HI, int FIRST, int LAST>
struct GfPass {
    static_assert(HI - LO < 4, "four accumulators of 128 TMEM columns");
    static constexpr int digits = LAST - FIRST + 1;
    // (more than half of the shared memory: a CTA takes all of the SM's TMEM)
    static constexpr int stages = digits > 4 ? 2 : (digits > 1 ? 3 : 8);
    static constexpr size_t stage_bytes = (size_t)2 * digits * GF_TILE;
    static constexpr size_t smem = stages * stage_bytes + 1024 + 256;
};
using GfLow = GfPass<8, 8, 4, 4>;
using GfMid = GfPass<4, 7, 0, 6>;
using GfTop = GfPass<0, 3, 0, 3>;
static_assert(GfLow::smem <= 232448 && GfMid::smem <= 232448 && GfTop::smem <= 232448,
              "stages must fit the 227 KB of a CTA");

// weight of level l in units of level 0
constexpr double gf_weight(int l) { return l == 0 ? 1.0 : gf_weight(l - 1) / 256.0; }

// kind::i8: signed 8-bit A and B, signed 32-bit D, both K-major, M = N = 128
constexpr uint32_t GF_IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GF_T >> 3) << 17) |
                              ((uint32_t)(GF_T >> 4) << 24);

__device__ __forceinline__ void gf_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(GF_IDESC), "r"(accumulate)
        : "memory");
}

// K-major tile in 64-byte swizzle atoms (8 rows x 64 B, 512 bytes apart)
__device__ __forceinline__ uint64_t sw64_kmajor_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

struct GfBundles {
    const double* base[6];   // up to three bundles of U, then of AU, n columns each
    int n, nblk;
};

__device__ __forceinline__ const double* gf_column(const GfBundles& b, int col, int64_t N) {
    const int k = col / b.n;
    return b.base[k] + (size_t)(col - k * b.n) * N;
}

// maxbits[col] = bits of max_i |u_i,col|: non-negative doubles order like their bits,
// with infinities and NaNs above all others
__global__ void gf_absmax_kernel(GfBundles b, int64_t N, unsigned long long* __restrict__ maxbits) {
    const double* s = gf_column(b, blockIdx.y, N);
    const bool vec = ((uintptr_t)s % 16) == 0;
    unsigned long long m = 0;
    auto take = [&](double x) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
        m = m > u ? m : u;
    };
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    int64_t done = 0;                                // points that went in pairs
    if (vec) {
        done = N / 2 * 2;
#pragma unroll 4
        for (int64_t q = t0; q < N / 2; q += step) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(s) + q);
            take(v.x);
            take(v.y);
        }
    }
#pragma unroll 4
    for (int64_t i = done + t0; i < N; i += step) take(__ldg(s + i));
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_down_sync(0xffffffffu, m, o);
        m = m > u ? m : u;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(&maxbits[blockIdx.y], m);
}

// Scale exponent e of a column: |u| 2^e < 127/128 2^55, the range of seven digits.
// A zero column has none; a column with an infinity or NaN makes its entries NaN
// (gf_reduce_kernel).
__device__ __forceinline__ int gf_exponent(unsigned long long bits) {
    if (bits == 0 || bits >= 0x7ff0000000000000ull) return 0;
    const double m = __longlong_as_double((long long)bits);
    const int E = ilogb(m);
    // mantissas of 127/64 and more (and subnormal maxima) keep one more bit of room
    const bool top = ((bits >> 46) & 63) == 63 || (bits >> 52) == 0;
    return top ? 53 - E : 54 - E;
}

// Digits of the points [g0, g0 + ldk) of every column (zero past N): one
// conversion per element, one addition that biases all digits to bytes, and the
// bytes of four elements transposed to a word per digit.  Bound by the 15 bytes
// moved per element.
__global__ void gf_digit_kernel(GfBundles b, int64_t N, int64_t g0, int64_t ldk,
                                const unsigned long long* __restrict__ maxbits, int8_t* __restrict__ digits,
                                size_t half) {
    const int col = blockIdx.y, p = b.n * b.nblk;
    const double* s = gf_column(b, col, N) + g0;
    const bool vec = ((uintptr_t)s % 16) == 0;
    const int64_t left = N - g0;
    const int e = gf_exponent(maxbits[col]);
    const int na = min(e, 1000);
    const double sa = ldexp(1.0, na), sb = ldexp(1.0, e - na);
    const bool second = col >= p;
    int8_t* out = digits + (second ? half : 0) + (size_t)(second ? col - p : col) * ldk;
    const size_t stride = (size_t)p * ldk;
    const int64_t n4 = ldk / 4;
    const unsigned long long bias = 0x0080808080808080ull;
#pragma unroll 2
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = 4 * q;
        double v[4];
        if (vec && i + 3 < left) {
            const double2 a = __ldg(reinterpret_cast<const double2*>(s + i));
            const double2 c = __ldg(reinterpret_cast<const double2*>(s + i + 2));
            v[0] = a.x; v[1] = a.y; v[2] = c.x; v[3] = c.y;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = i + j < left ? s[i + j] : 0.0;
        }
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned long long x = ((unsigned long long)__double2ll_rn(v[j] * sa * sb) + bias) ^ bias;
            lo[j] = (uint32_t)x;
            hi[j] = (uint32_t)(x >> 32);
        }
        // byte k of the four words -> one word; digit i is byte 6 - i
        uint32_t w[7];
        {
            const uint32_t a01 = __byte_perm(lo[0], lo[1], 0x5140), a23 = __byte_perm(lo[2], lo[3], 0x5140);
            const uint32_t b01 = __byte_perm(lo[0], lo[1], 0x7362), b23 = __byte_perm(lo[2], lo[3], 0x7362);
            w[6] = __byte_perm(a01, a23, 0x5410);
            w[5] = __byte_perm(a01, a23, 0x7632);
            w[4] = __byte_perm(b01, b23, 0x5410);
            w[3] = __byte_perm(b01, b23, 0x7632);
        }
        {
            const uint32_t a01 = __byte_perm(hi[0], hi[1], 0x5140), a23 = __byte_perm(hi[2], hi[3], 0x5140);
            const uint32_t b01 = __byte_perm(hi[0], hi[1], 0x7362), b23 = __byte_perm(hi[2], hi[3], 0x7362);
            w[2] = __byte_perm(a01, a23, 0x5410);
            w[1] = __byte_perm(a01, a23, 0x7632);
            w[0] = __byte_perm(b01, b23, 0x5410);
        }
#pragma unroll
        for (int k = 0; k < 7; ++k) reinterpret_cast<uint32_t*>(out + k * stride)[q] = w[k];
    }
}

// upper tile t, column order
__device__ __forceinline__ void gf_tile_of(int t, int* mt, int* nt) {
    int c = 0;
    while (t > c) t -= ++c;
    *mt = t;
    *nt = c;
}

// CTA: tile blockIdx.x of [S tiles, A tiles], K split blockIdx.y of the chunk.
// partial[((split * tiles + tile) * 128 + row) * 128 + col] = sum over the levels of D_l 256^-l
template <int LO, int HI, int FIRST, int LAST>
__global__ void __launch_bounds__(GF_THREADS, 1)
gram_f64_i8_kernel(const __grid_constant__ CUtensorMap mU, const __grid_constant__ CUtensorMap mV, int p, int ntl,
                   int kstages, int ksplit, double* __restrict__ partial, int* __restrict__ err,
                   int* __restrict__ own_err) {
    using P = GfPass<LO, HI, FIRST, LAST>;
    constexpr int ND = P::digits, NS = P::stages;
    extern __shared__ unsigned char gf_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)gf_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(base + NS * P::stage_bytes);
    uint64_t* empty = full + NS;
    uint64_t* done = empty + NS;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = gridDim.x, split = blockIdx.y;
    const bool second = (int)blockIdx.x >= ntl;
    int mt, nt;
    gf_tile_of(second ? blockIdx.x - ntl : blockIdx.x, &mt, &nt);
    const bool one = !second && mt == nt;           // both operands are the same tiles
    const int per = (kstages + ksplit - 1) / ksplit;
    const int kb0 = min(kstages, split * per), kb1 = min(kstages, kb0 + per);
    const int nk = kb1 - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], 1);
        }
        bar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    int issued = 0;
    auto give_up = [&]() {
        atomicOr(err, ERR_GEMM_TIMEOUT);
        atomicOr(own_err, ERR_GEMM_TIMEOUT);
        atomicExch(abort_flag, 1);
    };
    if (warp == 0 && lane == 0) {
        // ---- TMA producer ----
        const CUtensorMap* mB = second ? &mV : &mU;
        for (int it = 0; it < nk; ++it) {
            const int s = it % NS;
            if (it >= NS && !bar_wait(&empty[s], (uint32_t)(((it / NS) - 1) & 1), GF_WAIT_LIMIT)) {
                give_up();
                break;
            }
            if (*(volatile int*)abort_flag) break;
            unsigned char* st = base + s * P::stage_bytes;
            const int kx = (kb0 + it) * GF_K;
            bar_expect_tx(&full[s], (uint32_t)((one ? 1 : 2) * ND * GF_TILE));
            // rows past the last column of a digit are the next digit's (or past the
            // array: zero); they reach only entries that no one reads
            for (int k = 0; k < ND; ++k) tma_2d(st + k * GF_TILE, &mU, kx, (FIRST + k) * p + mt * GF_T, &full[s]);
            if (!one)
                for (int k = 0; k < ND; ++k)
                    tma_2d(st + (ND + k) * GF_TILE, mB, kx, (FIRST + k) * p + nt * GF_T, &full[s]);
            issued = it + 1;
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer ----
        for (int it = 0; it < nk; ++it) {
            const int s = it % NS;
            if (!bar_wait(&full[s], (uint32_t)((it / NS) & 1), GF_WAIT_LIMIT)) {
                give_up();
                break;
            }
            if (*(volatile int*)abort_flag) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = su32(base + s * P::stage_bytes), b = one ? a : a + ND * GF_TILE;
#pragma unroll
            for (int kk = 0; kk < GF_K / 32; ++kk)
#pragma unroll
                for (int l = LO; l <= HI; ++l) {
                    const int i0 = l - LAST > FIRST ? l - LAST : FIRST;      // digits i and l - i, both loaded
#pragma unroll
                    for (int i = i0; i <= l - FIRST && i <= LAST; ++i)
                        gf_mma(tmem + 128u * (l - LO), sw64_kmajor_desc(a + (i - FIRST) * GF_TILE + kk * 32),
                               sw64_kmajor_desc(b + (l - i - FIRST) * GF_TILE + kk * 32),
                               it > 0 || kk > 0 || i > i0 ? 1u : 0u);
                }
            umma_commit(&empty[s]);
        }
        umma_commit(done);
    }
    __syncwarp();

    // ---- epilogue: warp w owns TMEM lanes (rows) 32w .. 32w+31 ----
    const bool ok = bar_wait(done, 0, GF_WAIT_LIMIT);
    if (!ok) give_up();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    double* prow = partial + (((size_t)split * tiles + blockIdx.x) * GF_T + warp * 32 + lane) * GF_T;
    const bool have = ok && nk > 0;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
#pragma unroll 1
    for (int c0 = 0; c0 < GF_T; c0 += 32) {
        double v[32];
#pragma unroll
        for (int l = HI; l >= LO; --l) {             // smallest level first
            uint32_t r[32];
            tmem_ld32(tmem + lane_base + 128u * (l - LO) + (uint32_t)c0, r);
            const double f = gf_weight(l);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = l == HI ? (double)(int)r[j] * f : fma((double)(int)r[j], f, v[j]);
        }
#pragma unroll
        for (int j = 0; j < 32; j += 2)
            *reinterpret_cast<double2*>(prow + c0 + j) = have ? make_double2(v[j], v[j + 1]) : make_double2(0.0, 0.0);
    }

    // ---- teardown ----
    __syncthreads();
    if (threadIdx.x == 0 && *(volatile int*)abort_flag) {
        for (int it = max(0, issued - NS); it < issued; ++it)
            (void)bar_wait(&full[it % NS], (uint32_t)((it / NS) & 1), GF_DRAIN_LIMIT);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Sums a chunk's partial tiles (all passes, smallest levels first) onto acc [2][p][p]; the
// last chunk writes scale 2^(...) acc to B = S (blockIdx.z = 0) and A, with the mirror.
__global__ void gf_reduce_kernel(const double* __restrict__ partial, int slots, int ntl, int p, bool first, bool last,
                                 const unsigned long long* __restrict__ maxbits, double scale,
                                 double* __restrict__ acc, double* __restrict__ A, double* __restrict__ B) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y, z = blockIdx.z;
    if (n >= p || m > n) return;
    const int mt = m / GF_T, nt = n / GF_T;
    const int t = z * ntl + nt * (nt + 1) / 2 + mt;
    const size_t off = ((size_t)t * GF_T + m % GF_T) * GF_T + n % GF_T;
    const size_t stride = (size_t)2 * ntl * GF_T * GF_T;
    double s = 0.0;
    for (int k = 0; k < slots; ++k) s += partial[off + (size_t)k * stride];
    double* a = acc + ((size_t)z * p + m) * p + n;
    if (!first) s += *a;
    if (!last) {
        *a = s;
        return;
    }
    const unsigned long long bu = maxbits[m], bv = maxbits[z * p + n];
    // the digits d_0 are worth 256^6 = 2^48 each
    double r = ldexp(s, 96 - gf_exponent(bu) - gf_exponent(bv)) * scale;
    if (bu >= 0x7ff0000000000000ull || bv >= 0x7ff0000000000000ull) r = __longlong_as_double(0x7ff8000000000000ll);
    double* M = z ? A : B;
    M[m + (size_t)p * n] = r;
    M[n + (size_t)p * m] = r;
}

// Stands in for a wait that ran out: the words the kernel sets and a pencil of zeros, set by the
// host after the launches where QSB_GRAM_F64_GIVE_UP is in the environment (read once per
// process; no wait on the GPU is involved).
bool forced_give_up() {
    static const bool on = std::getenv("QSB_GRAM_F64_GIVE_UP") != nullptr;
    return on;
}
__global__ void set_words_kernel(int* err, int* own_err) {
    atomicOr(err, ERR_GEMM_TIMEOUT);
    atomicOr(own_err, ERR_GEMM_TIMEOUT);
}

bool make_digit_map(CUtensorMap* map, const void* base, int64_t ldk, int64_t rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)ldk, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ldk};
    const cuuint32_t box[2] = {GF_K, GF_T};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t a1k(size_t b) { return (b + 1023) & ~(size_t)1023; }
int64_t up128(int64_t x) { return (x + 127) / 128 * 128; }

struct GfPlan {
    int ntl, ksplit, chunks;
    int64_t kc;                                  // points per chunk, a multiple of 128
    size_t half, partial, bytes;                 // bytes of U's digits, of the partial tiles, in all (0: no plan)
    double cost;
};

// Points per chunk and K splits within `avail` bytes: whole waves of CTAs as far as
// the workspace and the accumulators' range allow
GfPlan plan_gf(int64_t N, int p, size_t avail) {
    GfPlan g{};
    const int t = (p + GF_T - 1) / GF_T;
    g.ntl = t * (t + 1) / 2;
    const size_t tile = (size_t)GF_T * GF_T * sizeof(double);
    const size_t fixed = a1k((size_t)2 * p * p * sizeof(double)) + a1k((size_t)2 * p * sizeof(unsigned long long));
    for (int k = 1; k <= 148; ++k) {
        const size_t partial = a1k((size_t)GF_PASSES * k * 2 * g.ntl * tile);
        if (avail < partial + fixed + 2048) break;
        const size_t room = std::min(GF_DIGIT_BYTES, avail - partial - fixed - 2048);    // 2048: a1k of both halves
        const int64_t most = (int64_t)(room / (2 * GF_DIGITS * (size_t)p)) / 128 * 128;
        if (most < 128) break;
        const int64_t cap = std::min<int64_t>(most, (int64_t)k * GF_MAX_STAGES * GF_K / 128 * 128);
        const int64_t chunks = (N + cap - 1) / cap, kc = up128((N + chunks - 1) / chunks);
        const int64_t stages = kc / GF_K;
        if (k > stages) break;
        const int64_t per = (stages + k - 1) / k, waves = ((int64_t)2 * g.ntl * k + 147) / 148;
        if (per > GF_MAX_STAGES) continue;
        // stages that the busiest SM works through, with some for each wave's fill and readout
        const double cost = (double)chunks * waves * (per + 16);
        if (g.bytes == 0 || cost < g.cost) {
            g.cost = cost;
            g.ksplit = k;
            g.chunks = (int)chunks;
            g.kc = kc;
            g.half = a1k((size_t)GF_DIGITS * p * kc);
            g.partial = partial;
            g.bytes = 2 * g.half + partial + fixed;
        }
    }
    return g;
}

bool gf_takes(int n) { return n >= GRAM_F64_I8_MIN_BANDS && 6 * (int64_t)n <= 65535; }

}  // namespace

// Whether the pencils of n bands can be formed within ws_bytes
bool gram_f64_i8_fits(int64_t N, int n, size_t ws_bytes) {
    return gf_takes(n) && plan_gf(N, 2 * n, ws_bytes).bytes > 0 && plan_gf(N, 3 * n, ws_bytes).bytes > 0;
}

// Bytes of a workspace of its own that the pencils of up to n bands are to have, 0 where
// `scratch` bytes that are free at that time do about as well or where n is not for this
// form.  Only small bundles want one: the partial tiles of a wave of CTAs take 57 MB,
// whatever the number of points (33 bands of 32^3 in the 9 MB of a bundle would take 12
// times the stages).
size_t gram_f64_i8_own_bytes(int64_t N, int n, size_t scratch) {
    if (!gf_takes(n)) return 0;
    const GfPlan two = plan_gf(N, 2 * n, GF_OWN_BYTES), three = plan_gf(N, 3 * n, GF_OWN_BYTES),
                 have = plan_gf(N, 3 * n, scratch);
    if (have.bytes > 0 && have.cost <= 1.1 * three.cost) return 0;
    return std::max(two.bytes, three.bytes) + 2048;      // plan_gf's reserve: the same plans within these bytes
}

// A = scale U^T AU and B = scale U^T U (both m x m, full), m = nblk * n columns; *gave_up
// (device) becomes non-zero when a bounded wait ran out and A and B are not to be used
qsb_status gram_f64_i8(int64_t N, int n, int nblk, const double* const* U, const double* const* AU, double scale,
                       double* A, double* B, void* ws, size_t ws_bytes, int* gave_up, cudaStream_t s) {
    const int p = n * nblk;
    const GfPlan g = plan_gf(N, p, ws_bytes);
    if (g.bytes == 0) return fail(QSB_ERR_INVALID, "gram_f64_i8: workspace too small");
    GfBundles b{};
    b.n = n;
    b.nblk = nblk;
    for (int k = 0; k < nblk; ++k) {
        b.base[k] = U[k];
        b.base[nblk + k] = AU[k];
    }
    unsigned char* w = (unsigned char*)ws;
    int8_t* digits = (int8_t*)w;
    double* partial = (double*)(w + 2 * g.half);
    double* acc = (double*)(w + 2 * g.half + g.partial);
    unsigned long long* maxbits =
        (unsigned long long*)(w + 2 * g.half + g.partial + a1k((size_t)2 * p * p * sizeof(double)));
    QSB_CUDA_TRY(cudaMemsetAsync(maxbits, 0, (size_t)2 * p * sizeof(unsigned long long), s));
    const int mblocks = (int)std::min<int64_t>((N / 2 + 256) / 256, std::max(1, 4736 / (2 * p)));
    gf_absmax_kernel<<<dim3(mblocks, 2 * p), 256, 0, s>>>(b, N, maxbits);
    QSB_CUDA_TRY(cudaGetLastError());
    auto low = gram_f64_i8_kernel<8, 8, 4, 4>;
    auto mid = gram_f64_i8_kernel<4, 7, 0, 6>;
    auto top = gram_f64_i8_kernel<0, 3, 0, 3>;
    QSB_TRY(allow_shared_memory(low));
    QSB_TRY(allow_shared_memory(mid));
    QSB_TRY(allow_shared_memory(top));
    const int tiles = 2 * g.ntl;
    for (int c = 0; c < g.chunks; ++c) {
        const int64_t g0 = c * g.kc;
        if (g0 >= N) return fail(QSB_ERR_INVALID, "gram_f64_i8: chunk");
        const int64_t ldk = up128(std::min(g.kc, N - g0));
        CUtensorMap mU, mV;
        if (!make_digit_map(&mU, digits, ldk, (int64_t)GF_DIGITS * p) ||
            !make_digit_map(&mV, digits + g.half, ldk, (int64_t)GF_DIGITS * p))
            return fail(QSB_ERR_CUDA, "gram_f64_i8: tensor map encoding failed");
        const int dblocks = (int)std::min<int64_t>((ldk / 4 + 255) / 256, std::max(1, 9472 / (2 * p)));
        gf_digit_kernel<<<dim3(dblocks, 2 * p), 256, 0, s>>>(b, N, g0, ldk, maxbits, digits, g.half);
        QSB_CUDA_TRY(cudaGetLastError());
        const int kstages = (int)(ldk / GF_K);
        const dim3 grid(tiles, g.ksplit);
        const size_t slots = (size_t)g.ksplit * tiles * GF_T * GF_T;       // of one pass
        int* const word = device_error_word();
        low<<<grid, GF_THREADS, GfLow::smem, s>>>(mU, mV, p, g.ntl, kstages, g.ksplit, partial, word, gave_up);
        QSB_CUDA_TRY(cudaGetLastError());
        mid<<<grid, GF_THREADS, GfMid::smem, s>>>(mU, mV, p, g.ntl, kstages, g.ksplit, partial + slots, word,
                                                           gave_up);
        QSB_CUDA_TRY(cudaGetLastError());
        top<<<grid, GF_THREADS, GfTop::smem, s>>>(mU, mV, p, g.ntl, kstages, g.ksplit, partial + 2 * slots,
                                                           word, gave_up);
        QSB_CUDA_TRY(cudaGetLastError());
        gf_reduce_kernel<<<dim3((p + 127) / 128, p, 2), 128, 0, s>>>(partial, GF_PASSES * g.ksplit, g.ntl, p, c == 0,
                                                                   c + 1 == g.chunks, maxbits, scale, acc, A, B);
        QSB_CUDA_TRY(cudaGetLastError());
    }
    if (forced_give_up()) {
        QSB_CUDA_TRY(cudaMemsetAsync(A, 0, sizeof(double) * p * p, s));
        QSB_CUDA_TRY(cudaMemsetAsync(B, 0, sizeof(double) * p * p, s));
        set_words_kernel<<<1, 1, 0, s>>>(device_error_word(), gave_up);
        QSB_CUDA_TRY(cudaGetLastError());
    }
    return QSB_OK;
}

}  // namespace qsb
