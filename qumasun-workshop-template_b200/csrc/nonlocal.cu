// Nonlocal Kleinman-Bylander projector apply for sm_100a.
//
//   Hpsi_c += sum_a sum_w |beta_aw> E_w dV <beta_aw | psi_c>
//
// The order of operations is the reference's ProjectionPP_bundle_1 /
// mInnerNonlocalPsi_v4_bundle (source/PseudoPotNonlocal_SvF2_kpoint.h:3911-4046,
// :4463-4576): gather psi on each atom's points, multiply by exp(+i k.r) (k != 0),
// contract with the projector table (DGEMM_t, times dV), scale by E_w, expand
// (DGEMM_n), multiply by exp(-i k.r), scatter-add.
//
// B200 layout: the projector points are held twice.
//  * atom-major ("gather") order, cut into chunks of one atom's points, for the
//    projection.  Each CTA reduces one chunk for a group of bands in registers
//    and shared memory and writes one partial sum per (chunk, w, column); a
//    second tiny kernel sums the chunks of each atom in a fixed order, so the
//    result is deterministic (no floating-point atomics).
//  * grid-ordered CSR (entries of grid point g are [grid_ptr[g], grid_ptr[g+1]))
//    for the expansion, done as a PULL: each output point sums its own entries.
//    Overlapping spheres (different atoms, or an atom and its own periodic
//    images) therefore need no atomics and no non-overlap grouping
//    (mCreateNonoverlapList, :3410-3487), and the pull can be fused into the H
//    stencil so Hpsi is written once.
#include "qsb_internal.h"
#include "apply_schedule.h"
#include <cmath>
#include <algorithm>
#include <numeric>
#include <cstring>

namespace qsb {

namespace {

constexpr int PROJ_THREADS = 256;
constexpr int CHUNK = 8192;          // points per projection chunk (32 per thread: amortizes the block reduction)
constexpr int APPLY_THREADS = 256;

template <typename T>
void dfree(T*& p) {
    if (p) cudaFree((void*)p);
    p = nullptr;
}

// Device copies of host tables in two allocations, the short ones of each going up in
// one copy, so that a small cell's two dozen tables do not cost as many allocations
// and waits (10.5 -> 10.2 ms for two atoms on 32^3, 12.9 -> 12.2 for three on 45 x 50 x 63).
// Tables of a few KB stay apart from the large ones: the allocator serves what they
// take, and the workspace of the first apply after them, from one small block (in
// one allocation with the rest that workspace cost the first apply 0.5 ms).
class TableUpload {
public:
    template <typename T>
    void add(T*& dst, const T* src, size_t n) {
        dst = nullptr;
        if (n > 0) items_.push_back({&dst, src, n * sizeof(T), 0});
    }
    template <typename T>
    void add(T*& dst, const std::vector<T>& v) {
        add(dst, v.data(), v.size());
    }
    // base: the allocations (also those made before an error), null where nothing is needed
    qsb_status run(void* (&base)[2]) {
        std::stable_sort(items_.begin(), items_.end(), [](const Item& a, const Item& b) { return a.bytes < b.bytes; });
        const auto cut = std::find_if(items_.begin(), items_.end(), [](const Item& it) { return it.bytes > TINY; });
        QSB_TRY(place(items_.begin(), cut, base[0]));
        return place(cut, items_.end(), base[1]);
    }

private:
    static constexpr size_t TINY = (size_t)1 << 16, SHORT = (size_t)1 << 20;
    struct Item {
        void* dst;                 // the pointer to set
        const void* src;
        size_t bytes, off;
    };
    using Iter = std::vector<Item>::iterator;
    static qsb_status place(Iter first, Iter last, void*& base) {
        size_t total = 0, packed = 0;
        for (Iter it = first; it != last; ++it) {
            it->off = total;
            total += (it->bytes + 255) / 256 * 256;
            if (it->bytes <= SHORT) packed = total;
        }
        if (total == 0) return QSB_OK;
        if (cudaMalloc(&base, total) != cudaSuccess) {
            cudaGetLastError();
            base = nullptr;
            return fail(QSB_ERR_NOMEM, "nonlocal tables: cudaMalloc failed");
        }
        std::vector<unsigned char> stage(packed);
        for (Iter it = first; it != last; ++it) {
            void* const at = (unsigned char*)base + it->off;
            if (it->bytes <= SHORT) std::memcpy(stage.data() + it->off, it->src, it->bytes);
            else QSB_CUDA_TRY(cudaMemcpy(at, it->src, it->bytes, cudaMemcpyHostToDevice));
            std::memcpy(it->dst, &at, sizeof(at));      // whatever type of pointer it is
        }
        if (packed > 0) QSB_CUDA_TRY(cudaMemcpy(base, stage.data(), packed, cudaMemcpyHostToDevice));
        return QSB_OK;
    }
    std::vector<Item> items_;
};

inline int fold(int v, int n) {
    int m = v % n;
    return m < 0 ? m + n : m;
}

// ---------------------------------------------------------------------------
// projection: partial[chunk][w][col] = sum_{p in chunk} beta[p][w] * phi_col[idx_p]
// phi = psi (real) or psi*exp(+i k.r) (complex; columns 2b = re, 2b+1 = im)
//
// The gathers' latency is hidden by an asynchronous pipeline: each thread copies
// its own points' psi values, beta rows (and coordinates) S - 1 passes ahead into
// its own slots of a shared ring (cp.async; no thread reads another's slots, so
// no barrier), which takes no registers.  What bounds it then is the traffic
// from L2 (~8.8 TB/s for the whole chip, measured, 1.25x the DRAM rate): the
// beta rows once per CB columns and the sectors at the ends of the sphere's rows.
// 144^3 x 384 FP32 bands, 54 atoms: 4.69 -> 1.93 ms; 96^3 x 128 FP64, 16 atoms
// 0.280 -> 0.286 ms (at that bound before).
// Thread t sums the points t + 256 m in increasing m, then lanes, warps and
// chunks in order, whatever CB and S are: the mixed-precision solver's results
// depend on the order of these sums to the bit.
// ---------------------------------------------------------------------------
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
    static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async sizes");
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

struct ProjTables {
    const void* t[4];    // beta and its gradients, [point][wmax]
    int n;               // how many
};

template <typename T, bool CPLX, int WM, int CB>
struct ProjCfg {
    static constexpr int NCB = CPLX ? 2 * CB : CB;
    // one point of one thread: psi values, beta rows, coordinates
    static constexpr int BYTES = NCB * (int)sizeof(T) + WM * (int)sizeof(T) + (CPLX ? 12 : 0);
    static constexpr int NV = WM * NCB;                      // sums per thread
    static constexpr int MINB = NV <= 32 ? 2 : 1;            // CTAs per SM (128 / 255 registers)
    static constexpr int FIT = (MINB == 2 ? 104 : 200) * 1024 / (BYTES * PROJ_THREADS);
    static constexpr int S = FIT < 2 ? 2 : (FIT > 8 ? 8 : FIT);
    static constexpr int RING = S * BYTES * PROJ_THREADS;
    static constexpr int RED = (PROJ_THREADS / 32) * NV * 8;
    static constexpr int SMEM = RING > RED ? RING : RED;
    static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
};

template <typename T, bool CPLX, int WM, int CB>
__global__ void __launch_bounds__(PROJ_THREADS, (ProjCfg<T, CPLX, WM, CB>::MINB))
nl_proj_kernel(const int* __restrict__ chunk_order, const int* __restrict__ chunk_begin,
               const int* __restrict__ chunk_end, const int* __restrict__ pt_idx, const int* __restrict__ pt_xyz,
               const T* __restrict__ pt_beta, int wmax, const T* __restrict__ psi, size_t N, int nb, double gx_dx,
               double gy_dy, double gz_dz, double* __restrict__ partial, int ncol) {
    using C = ProjCfg<T, CPLX, WM, CB>;
    constexpr int NCB = C::NCB, S = C::S, NV = C::NV;
    extern __shared__ __align__(16) unsigned char proj_sm[];
    // launch order: chunks of all atoms by their position along the grid, so
    // that the CTAs in flight together gather from the same region of psi and
    // the overlapping spheres of neighbouring atoms meet in L2; each CTA writes
    // the partials of its own chunk, so the sums do not depend on the order
    const int chunk = chunk_order[blockIdx.y];
    const int band0 = blockIdx.x * CB;
    const int nbl = min(CB, nb - band0);
    const int p0 = chunk_begin[chunk], p1 = chunk_end[chunk];
    const int passes = (p1 - p0 + PROJ_THREADS - 1) / PROJ_THREADS;
    const int t = threadIdx.x;

    // ring layout, per stage: psi [NCB][256] T, beta (rows of 16 bytes [256] when
    // whole rows can be copied so, else [WM][256] T), coordinates [3][256] int
    constexpr int STAGE = C::BYTES * PROJ_THREADS;
    constexpr int BOFF = NCB * (int)sizeof(T) * PROJ_THREADS;
    constexpr int XOFF = BOFF + WM * (int)sizeof(T) * PROJ_THREADS;
    constexpr bool VROW = (WM * (int)sizeof(T)) % 16 == 0;
    constexpr int VPR = VROW ? WM * (int)sizeof(T) / 16 : 1;     // 16-byte pieces of a row
    const bool vrow = VROW && wmax == WM;
    const uint32_t sm0 = (uint32_t)__cvta_generic_to_shared(proj_sm);
    const T* psi0 = psi + (size_t)(CPLX ? 2 * band0 : band0) * N;

    auto issue = [&](int m, int idx) {      // copies of this thread's point of pass m
        const int p = p0 + t + m * PROJ_THREADS;
        if (p < p1) {
            const uint32_t st = sm0 + (uint32_t)((m % S) * STAGE);
#pragma unroll
            for (int j = 0; j < NCB; ++j)
                if (j < (CPLX ? 2 * nbl : nbl))
                    cp_async<(int)sizeof(T)>(st + (uint32_t)((j * PROJ_THREADS + t) * (int)sizeof(T)),
                                             psi0 + (size_t)j * N + idx);
            const T* row = pt_beta + (size_t)p * wmax;
            if (vrow) {
#pragma unroll
                for (int v = 0; v < VPR; ++v)
                    cp_async<16>(st + (uint32_t)(BOFF + (v * PROJ_THREADS + t) * 16), (const char*)row + v * 16);
            } else {
#pragma unroll
                for (int w = 0; w < WM; ++w)
                    if (w < wmax)
                        cp_async<(int)sizeof(T)>(st + (uint32_t)(BOFF + (w * PROJ_THREADS + t) * (int)sizeof(T)),
                                                 row + w);
            }
            if (CPLX)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    cp_async<4>(st + (uint32_t)(XOFF + (d * PROJ_THREADS + t) * 4), pt_xyz + 3 * (size_t)p + d);
        }
        cp_commit();
    };
    auto index_of = [&](int m) {
        const int p = p0 + t + m * PROJ_THREADS;
        return p < p1 ? __ldg(pt_idx + p) : 0;
    };

    double acc[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[i] = 0.0;
    {
        int idx[S - 1];
#pragma unroll
        for (int m = 0; m < S - 1; ++m) idx[m] = index_of(m);
#pragma unroll
        for (int m = 0; m < S - 1; ++m) issue(m, idx[m]);
    }
    int i0 = index_of(S - 1), i1 = index_of(S);
    for (int m = 0; m < passes; ++m) {
        const int i2 = index_of(m + S + 1);
        issue(m + S - 1, i0);
        i0 = i1;
        i1 = i2;
        cp_wait<S - 1>();
        const int p = p0 + t + m * PROJ_THREADS;
        if (p >= p1) continue;
        const unsigned char* st = proj_sm + (m % S) * STAGE;
        double b[WM];
        if (vrow) {
#pragma unroll
            for (int v = 0; v < VPR; ++v) {
                const int4 r = *reinterpret_cast<const int4*>(st + BOFF + (v * PROJ_THREADS + t) * 16);
                constexpr int E = 16 / (int)sizeof(T);
                T e[E];
                memcpy(e, &r, 16);
#pragma unroll
                for (int n = 0; n < E; ++n)
                    if (v * E + n < WM) b[v * E + n] = (double)e[n];
            }
        } else {
#pragma unroll
            for (int w = 0; w < WM; ++w)
                b[w] = w < wmax ? (double)*reinterpret_cast<const T*>(st + BOFF + (w * PROJ_THREADS + t) *
                                                                                      (int)sizeof(T))
                                : 0.0;
        }
        const T* ps = reinterpret_cast<const T*>(st) + t;
        if (CPLX) {
            const int* xs = reinterpret_cast<const int*>(st + XOFF) + t;
            // mCreateBlochExp (source/PseudoPotNonlocal_SvF2_kpoint.h:3580-3590)
            const double kxx = gx_dx * (double)xs[0];
            const double kyy = gy_dy * (double)xs[PROJ_THREADS];
            const double kzz = gz_dz * (double)xs[2 * PROJ_THREADS];
            double cs = 1.0, sn = 0.0;
            sincos(kxx + kyy + kzz, &sn, &cs);
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                const double pr = (double)ps[(2 * j) * PROJ_THREADS], pi = (double)ps[(2 * j + 1) * PROJ_THREADS];
                const double fr = cs * pr - sn * pi;   // :4514-4515
                const double fi = cs * pi + sn * pr;
#pragma unroll
                for (int w = 0; w < WM; ++w) {
                    acc[w * NCB + 2 * j] += b[w] * fr;
                    acc[w * NCB + 2 * j + 1] += b[w] * fi;
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                const double v = (double)ps[j * PROJ_THREADS];
#pragma unroll
                for (int w = 0; w < WM; ++w) acc[w * NCB + j] += b[w] * v;
            }
        }
    }

    // block reduction, in the ring's memory once every thread has left the loop
    cp_wait<0>();
    __syncthreads();
    double(*red)[NV] = reinterpret_cast<double(*)[NV]>(proj_sm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        double v = acc[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][i] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NV; i += PROJ_THREADS) {
        const int w = i / NCB, jc = i % NCB;
        if (w >= wmax) continue;
        const int col = (CPLX ? 2 * band0 : band0) + jc;
        if (jc >= (CPLX ? 2 * nbl : nbl)) continue;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < PROJ_THREADS / 32; ++q) s += red[q][i];
        partial[((size_t)chunk * wmax + w) * ncol + col] = s;
    }
}

// ---------------------------------------------------------------------------
// The projection as FP64 tensor-core products (mma.m8n8k4; there is no FP64 kind
// of tcgen05): per chunk, D (projector rows x columns) += B^T (rows x points)
// psi (points x columns).
//
// What bounds it is the traffic from L2 (~8.8 TB/s for the whole chip, measured,
// 1.25x the DRAM rate): a thread that keeps its own sums (nl_proj_kernel) holds
// at most 8 columns, so the beta rows cross L2 once per 8 columns, 36 bytes
// beside 64 of psi.  Here the sums of 8 rows x 8 columns take two registers per
// lane and the reduction over points happens inside the MMA, so one read of the
// rows serves NC = 32 columns, or the four tables of the forces (16 rows).
// The FP64 MMA rate is that of the FP64 pipe; half of the 8 rows are idle at four
// real projectors, all are used by a complex bundle (beta cos, beta sin) and by
// the forces.
//
// WARPS warps, each with its own batches of 32 points (warp w takes batches w,
// w + WARPS, ...): the psi values of the next batch are loaded to registers
// (lanes along points, so the gathers coalesce) while this batch is multiplied
// from the warp's shared buffer, whose columns lie 36 elements apart, so that a
// fragment's 4 points x 8 columns touch every bank once.  (cp.async straight to
// shared memory cost 10 to 18 clocks of the load pipe per 8-byte copy.)  Sums over the
// batches of a warp in order, then over the warps in order: deterministic.
// Points past the chunk's end count as zeros.
// ---------------------------------------------------------------------------
constexpr int MMA_P = 36;       // elements between columns (rows) of a 32-point batch

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Shared memory of one warp: a batch of psi [NC][36] T, its beta rows [32][rows] T
// and coordinates [32][3] int, and the A operand [8 MT][36] double
struct MmaLayout {
    int beta_off, xyz_off, a_off, warp_bytes;
    __host__ __device__ MmaLayout(int elem, int NC, int MT, int trows, bool cplx) {
        beta_off = NC * MMA_P * elem;
        xyz_off = beta_off + ((32 * trows * elem + 15) / 16) * 16;
        a_off = xyz_off + (cplx ? 384 : 0);
        warp_bytes = a_off + 8 * MT * MMA_P * 8;
    }
};

// MT: 8-row tiles of the A operand; rows r = table * wmax + w (real), and the
// same again for the sine parts (complex).  NC: columns per CTA.
template <typename T, bool CPLX, int MT, int NC, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, (WARPS <= 8 ? 2 : 1))
nl_proj_mma_kernel(const int* __restrict__ chunk_order, const int* __restrict__ chunk_begin,
                   const int* __restrict__ chunk_end, const int* __restrict__ pt_idx,
                   const int* __restrict__ pt_xyz, const ProjTables tabs, int wmax, const T* __restrict__ psi,
                   size_t N, double gx_dx, double gy_dy, double gz_dz, double* __restrict__ partial,
                   size_t table_stride, int ncol) {
    extern __shared__ __align__(16) unsigned char mma_sm[];
    constexpr int NT = NC / 8;
    constexpr int TB = (int)sizeof(T);
    const int trows = tabs.n * wmax;                     // rows without the complex split
    const MmaLayout ly(TB, NC, MT, trows, CPLX);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* mine = mma_sm + warp * ly.warp_bytes;
    const uint32_t mine_u = (uint32_t)__cvta_generic_to_shared(mine);
    double* A = reinterpret_cast<double*>(mine + ly.a_off);
    const int chunk = chunk_order[blockIdx.y];
    const int col0 = blockIdx.x * NC;
    const int ncl = min(NC, ncol - col0);
    const int p0 = chunk_begin[chunk], p1 = chunk_end[chunk];
    const int batches = (p1 - p0 + 31) / 32;
    const T* psi0 = psi + (size_t)col0 * N;

    for (int i = lane; i < 8 * MT * MMA_P; i += 32) A[i] = 0.0;   // rows past the last stay zero
    auto index_of = [&](int b) {
        const int p = p0 + 32 * b + lane;
        return p < p1 ? __ldg(pt_idx + p) : 0;
    };
    const bool rows16 = (wmax * TB) % 16 == 0;
    T v[NC];                                             // psi of the next batch, this lane's point
    auto load = [&](int b, int idx) {
        const bool live = p0 + 32 * b + lane < p1;
        const T* src = psi0 + idx;
#pragma unroll
        for (int j = 0; j < NC; ++j, src += N) v[j] = live && j < ncl ? __ldg(src) : T(0);
    };
    auto copy_rows = [&](int b) {                        // beta rows and coordinates of batch b
        const int p = p0 + 32 * b + lane;
        const size_t pl = (size_t)(p < p1 ? p : p0);
        for (int k = 0; k < tabs.n; ++k) {
            const char* row = (const char*)((const T*)tabs.t[k] + pl * wmax);
            const uint32_t db = mine_u + (uint32_t)(ly.beta_off + (lane * trows + k * wmax) * TB);
            if (rows16) {
                for (int o = 0; o < wmax * TB; o += 16) cp_async<16>(db + o, row + o);
            } else {
                for (int o = 0; o < wmax * TB; o += TB) cp_async<TB>(db + o, row + o);
            }
        }
        if (CPLX)
#pragma unroll
            for (int d = 0; d < 3; ++d)
                cp_async<4>(mine_u + (uint32_t)(ly.xyz_off + (lane * 3 + d) * 4), pt_xyz + 3 * pl + d);
        cp_commit();
    };

    // one column tile: two sums per entry (even and odd fours of points), half the chain of dependent MMAs
    constexpr int KS = NT == 1 ? 2 : 1;
    double acc[KS][MT][NT][2];
#pragma unroll
    for (int q = 0; q < KS; ++q)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n) acc[q][m][n][0] = acc[q][m][n][1] = 0.0;

    int idx = index_of(warp);
    if (warp < batches) {
        copy_rows(warp);
        load(warp, idx);
    }
    idx = index_of(warp + WARPS);
    for (int b = warp; b < batches; b += WARPS) {
        cp_wait<0>();
        {
            T* ps = reinterpret_cast<T*>(mine) + lane;
#pragma unroll
            for (int j = 0; j < NC; ++j) ps[j * MMA_P] = v[j];
        }
        __syncwarp();
        const unsigned char* sb = mine;
        // A operand: this lane's point
        {
            const T* br = reinterpret_cast<const T*>(sb + ly.beta_off) + lane * trows;
            const bool live = p0 + 32 * b + lane < p1;
            if (CPLX) {
                const int* xs = reinterpret_cast<const int*>(sb + ly.xyz_off) + lane * 3;
                // mCreateBlochExp (source/PseudoPotNonlocal_SvF2_kpoint.h:3580-3590)
                const double kxx = gx_dx * (double)xs[0];
                const double kyy = gy_dy * (double)xs[1];
                const double kzz = gz_dz * (double)xs[2];
                double cs = 1.0, sn = 0.0;
                sincos(kxx + kyy + kzz, &sn, &cs);
                for (int r = 0; r < trows; ++r) {
                    const double v = live ? (double)br[r] : 0.0;
                    A[r * MMA_P + lane] = v * cs;
                    A[(trows + r) * MMA_P + lane] = v * sn;
                }
            } else {
                for (int r = 0; r < trows; ++r) A[r * MMA_P + lane] = live ? (double)br[r] : 0.0;
            }
        }
        __syncwarp();
        if (b + WARPS < batches) {                       // the next batch, in flight during the products
            copy_rows(b + WARPS);
            load(b + WARPS, idx);
        }
        idx = index_of(b + 2 * WARPS);
        const T* ps = reinterpret_cast<const T*>(sb) + (lane >> 2) * MMA_P + (lane & 3);
        const double* as = A + (lane >> 2) * MMA_P + (lane & 3);
        // a batch's sums from zero, one column tile after the other, and then onto the running
        // ones, which so take one rounding per 32 points (with the running sums as the
        // products' accumulators the forces of 96^3 x 128 bands were 2.95e-15 off 64 bits, now
        // 2.65e-15, and 2.58e-15 with the sums per thread; 2 % of the time)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            double part[KS][MT][2];
#pragma unroll
            for (int q = 0; q < KS; ++q)
#pragma unroll
                for (int m = 0; m < MT; ++m) part[q][m][0] = part[q][m][1] = 0.0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double x = (double)ps[n * 8 * MMA_P + 4 * k];
#pragma unroll
                for (int m = 0; m < MT; ++m) mma_f64(part[k % KS][m], as[m * 8 * MMA_P + 4 * k], x);
            }
#pragma unroll
            for (int q = 0; q < KS; ++q)
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    acc[q][m][n][0] += part[q][m][0];
                    acc[q][m][n][1] += part[q][m][1];
                }
        }
        __syncwarp();   // the batch's buffers are free again
    }
#pragma unroll
    for (int q = 1; q < KS; ++q)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) acc[0][m][n][h] += acc[q][m][n][h];

    // sums over the warps, in the buffers' memory once every warp has left the loop
    cp_wait<0>();
    __syncthreads();
    double* red = reinterpret_cast<double*>(mma_sm);     // [warp][8 MT][NC]
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                red[(warp * 8 * MT + m * 8 + (lane >> 2)) * NC + n * 8 + 2 * (lane & 3) + h] = acc[0][m][n][h];
    __syncthreads();
    auto total = [&](int r, int c) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < WARPS; ++q) t += red[(q * 8 * MT + r) * NC + c];
        return t;
    };
    for (int i = threadIdx.x; i < trows * NC; i += WARPS * 32) {
        const int r = i / NC, c = i % NC;
        if (c >= ncl) continue;
        double v = total(r, c);
        // (cos + i sin)(re + i im): re' = cos re - sin im, im' = cos im + sin re (:4514-4515)
        if (CPLX) v = (c & 1) == 0 ? v - total(trows + r, c + 1) : v + total(trows + r, c - 1);
        const int k = r / wmax, w = r - k * wmax;
        partial[k * table_stride + ((size_t)chunk * wmax + w) * ncol + col0 + c] = v;
    }
}

// coef[a][w][col] = dV * (E_w) * sum_{chunks of a} partial
__global__ void nl_finalize_kernel(const int* __restrict__ atom_chunk_begin, const int* __restrict__ atom_chunk_end,
                                   const double* __restrict__ atom_E, const int* __restrict__ atom_width, int wmax,
                                   const double* __restrict__ partial, int ncol, double dV, int inner_only,
                                   double* __restrict__ coef) {
    const int a = blockIdx.x;
    const int c0 = atom_chunk_begin[a], c1 = atom_chunk_end[a];
    const int wa = atom_width[a];
    for (int i = threadIdx.x; i < wmax * ncol; i += blockDim.x) {
        const int w = i / ncol, col = i % ncol;
        double s = 0.0;
        if (w < wa)
            for (int ch = c0; ch < c1; ++ch) s += partial[((size_t)ch * wmax + w) * ncol + col];
        const double e = inner_only ? 1.0 : atom_E[(size_t)a * wmax + w];
        coef[((size_t)a * wmax + w) * ncol + col] = (w < wa) ? (s * dV) * e : 0.0;
    }
}

// ---------------------------------------------------------------------------
// expansion, pull form over covered grid points:
//   hpsi_col[g] += sum_{e on g} sum_w beta_e[w] * coef[atom_e][w][col]
// One thread per covered grid point loops over every band, so the point's
// entries (atom, beta, Bloch phase) are loaded once into registers and the
// band loop streams the read-modify-write of hpsi, coalesced along x.
// Entries are taken MAXE at a time (points covered by more spheres loop).
// ---------------------------------------------------------------------------
template <typename T, bool CPLX, int WM>
__global__ void __launch_bounds__(APPLY_THREADS, 2)
nl_apply_kernel(const int* __restrict__ cov_grid, int n_cov, const int* __restrict__ grid_ptr,
                const int* __restrict__ ent_atom, const int* __restrict__ ent_xyz, const T* __restrict__ ent_beta,
                int wmax, const double* __restrict__ coef, int ncol, T* __restrict__ hpsi, size_t N, int nb,
                double gx_dx, double gy_dy, double gz_dz) {
    // entries held in registers at a time
    constexpr int MAXE = CPLX ? (WM <= 4 ? 2 : 1) : (WM <= 4 ? 4 : (WM <= 9 ? 2 : 1));
    constexpr int BG = CPLX ? 4 : 8;   // bands per group
    constexpr int CG = 8;              // coefficient columns per group: BG real, 2 BG complex
    const int r = blockIdx.x * APPLY_THREADS + threadIdx.x;
    if (r >= n_cov) return;
    const int g = __ldg(cov_grid + r);
    const int e0 = __ldg(grid_ptr + g), e1 = __ldg(grid_ptr + g + 1);
    // coefficient rows are read 8 columns at a time as four 16-byte loads
    const bool vec = (ncol % 2 == 0) && (((uintptr_t)coef) % 16 == 0);
    for (int eb = e0; eb < e1; eb += MAXE) {
        const int ne = min(MAXE, e1 - eb);
        const double* cf[MAXE];
        double b[MAXE][WM];
        double cs[MAXE], sn[MAXE];
#pragma unroll
        for (int q = 0; q < MAXE; ++q) {
            const int e = eb + min(q, ne - 1);
            cf[q] = coef + (size_t)__ldg(ent_atom + e) * wmax * ncol;
#pragma unroll
            for (int w = 0; w < WM; ++w)
                b[q][w] = (q < ne && w < wmax) ? (double)__ldg(ent_beta + (size_t)e * wmax + w) : 0.0;
            cs[q] = 1.0;
            sn[q] = 0.0;
            if (CPLX) {
                const double kxx = gx_dx * (double)__ldg(ent_xyz + 3 * (size_t)e + 0);
                const double kyy = gy_dy * (double)__ldg(ent_xyz + 3 * (size_t)e + 1);
                const double kzz = gz_dz * (double)__ldg(ent_xyz + 3 * (size_t)e + 2);
                sincos(kxx + kyy + kzz, &sn[q], &cs[q]);
            }
        }
        for (int b0 = 0; b0 < nb; b0 += BG) {
            const int c0 = CPLX ? 2 * b0 : b0;
            const bool full = vec && (b0 + BG <= nb);
            // hpsi of the group first: CG independent loads in flight
            T cur[CG];
#pragma unroll
            for (int k = 0; k < CG; ++k) {
                const int col = c0 + k;
                cur[k] = (col < ncol) ? hpsi[(size_t)col * N + g] : T(0);
            }
            double acc[CG];
#pragma unroll
            for (int k = 0; k < CG; ++k) acc[k] = 0.0;
#pragma unroll
            for (int q = 0; q < MAXE; ++q) {
                if (q < ne) {
                    double tq[CG];
#pragma unroll
                    for (int k = 0; k < CG; ++k) tq[k] = 0.0;
#pragma unroll
                    for (int w = 0; w < WM; ++w) {
                        if (w < wmax) {
                            const double* row = cf[q] + (size_t)w * ncol + c0;
                            double c[CG];
                            if (full) {
#pragma unroll
                                for (int k = 0; k < CG; k += 2) {
                                    const double2 v = __ldg(reinterpret_cast<const double2*>(row + k));
                                    c[k] = v.x;
                                    c[k + 1] = v.y;
                                }
                            } else {
#pragma unroll
                                for (int k = 0; k < CG; ++k) c[k] = (c0 + k < ncol) ? __ldg(row + k) : 0.0;
                            }
#pragma unroll
                            for (int k = 0; k < CG; ++k) tq[k] += b[q][w] * c[k];
                        }
                    }
                    if (CPLX) {
                        // exp(-i k.r) (source/PseudoPotNonlocal_SvF2_kpoint.h:4026-4027)
#pragma unroll
                        for (int j = 0; j < BG; ++j) {
                            acc[2 * j] += cs[q] * tq[2 * j] + sn[q] * tq[2 * j + 1];
                            acc[2 * j + 1] += cs[q] * tq[2 * j + 1] - sn[q] * tq[2 * j];
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < CG; ++k) acc[k] += tq[k];
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < CG; ++k) {
                const int col = c0 + k;
                if (col < ncol) hpsi[(size_t)col * N + g] = cur[k] + (T)acc[k];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// expansion, pipelined: the pull of nl_apply_kernel with the coefficient rows of
// the CTA's own atoms (a list made with the tables: the few spheres its 256
// points lie in, not every atom of the cell) staged in shared memory one
// APPLY_CW-column slice ahead, up to MAXE entries of the point held in registers
// for all columns, and hpsi read S - 1 groups of SG columns ahead
// into the thread's own slots of a shared ring (cp.async).
// Read-modify-write of hpsi.  Before, every group's loads were issued and waited
// for in turn and every atom's rows staged by every CTA (2.6 long- and 2.3
// short-scoreboard stalls per issue, DRAM 25 %); now the load pipe is half busy,
// with the coefficients' 16-byte loads above all (2.7 passes each where a warp's
// lanes lie in different spheres), and hpsi moves at 5.0 TB/s (FP64) and 3.2 TB/s
// (FP32) of the 6.4 a plain read-modify-write reaches.
// 144^3 x 384 FP32 bands, 54 atoms: 3.37 -> 2.87 ms; 96^3 x 128 bands, 16 atoms:
// FP32 0.311 -> 0.284, FP64 0.384 -> 0.363 ms.  As FP64 tensor-core products (one
// coefficient load per 4 x 8 of them) it took 3.08 and 0.456 ms: the accumulator's
// layout splits every 256-byte row of hpsi into 64-byte pieces.
// ---------------------------------------------------------------------------
constexpr int APPLY_CW = 32;    // columns per coefficient slice
// Real FP64 bundles load a group's hpsi directly, 16 columns at a time (0.366 against 0.388 ms
// with the ring at 96^3 x 128 bands).
template <typename T, bool CPLX>
struct ApplyCfg {
    static constexpr bool DIRECT = sizeof(T) == 8 && !CPLX;
    static constexpr int SG = DIRECT ? 16 : 8;               // columns per group
    static constexpr int S = DIRECT ? 0 : (sizeof(T) == 8 ? 3 : 5);   // groups in the ring
    static constexpr int RING = S * SG * APPLY_THREADS * (int)sizeof(T);
    using Order = ApplySchedule<S, APPLY_CW / SG>;           // when which copies are committed and waited for
};

// doubles of one atom's rows in a slice: 16 bytes of padding keep two atoms' rows in different banks
__host__ __device__ constexpr int apply_row(int wmax) { return wmax * APPLY_CW + 2; }

// FULL: wmax == WM (no row is padding)
template <typename T, bool CPLX, int WM, bool FULL>
__global__ void __launch_bounds__(APPLY_THREADS, (WM <= 4 ? (CPLX || sizeof(T) == 8 ? 2 : 3) : 1))
nl_apply_ring_kernel(const int* __restrict__ cov_grid, int n_cov, const int* __restrict__ grid_ptr,
                     const int* __restrict__ ent_local, const int* __restrict__ ent_xyz,
                     const T* __restrict__ ent_beta, int wmax_, const int* __restrict__ cta_ptr,
                     const int* __restrict__ cta_atoms, int max_local, const double* __restrict__ coef, int ncol,
                     T* __restrict__ hpsi, size_t N, double gx_dx, double gy_dy, double gz_dz) {
    const int wmax = FULL ? WM : wmax_;
    extern __shared__ __align__(16) unsigned char apply_sm[];   // ring [S][SG][256] T, then 2 coefficient slices
    constexpr int MAXE = WM <= 4 ? 3 : 1;                       // entries kept in registers
    using CF = ApplyCfg<T, CPLX>;
    constexpr int SG = CF::SG, S = CF::S, PROLOGUE = CF::Order::PROLOGUE;
    constexpr int STAGE = SG * APPLY_THREADS * (int)sizeof(T);
    const int arow = apply_row(wmax);
    double* csm = reinterpret_cast<double*>(apply_sm + CF::RING);
    const int t = threadIdx.x;
    const int r = blockIdx.x * APPLY_THREADS + t;
    const bool active = r < n_cov;
    const int a0 = cta_ptr[blockIdx.x], na = cta_ptr[blockIdx.x + 1] - a0;
    const uint32_t sm0 = (uint32_t)__cvta_generic_to_shared(apply_sm);
    const uint32_t cm0 = sm0 + (uint32_t)CF::RING;
    int g = 0, e0 = 0, e1 = 0;
    if (active) {
        g = __ldg(cov_grid + r);
        e0 = __ldg(grid_ptr + g);
        e1 = __ldg(grid_ptr + g + 1);
    }
    T* hp = hpsi + g;
    // group n: columns [n SG, n SG + SG); its first group also brings slice n SG / CW + 1
    auto slice = [&](int sl) {
        const int c0 = sl * APPLY_CW, cw = min(APPLY_CW, ncol - c0);
        const uint32_t dst = cm0 + (uint32_t)((sl & 1) * max_local * arow * 8);
        for (int i = t; i < na * wmax * APPLY_CW; i += APPLY_THREADS) {
            const int k = i % APPLY_CW, aw = i / APPLY_CW, al = aw / wmax, w = aw - al * wmax;
            if (k < cw)
                cp_async<8>(dst + (uint32_t)((al * arow + w * APPLY_CW + k) * 8),
                            coef + ((size_t)__ldg(cta_atoms + a0 + al) * wmax + w) * ncol + c0 + k);
        }
    };
    const int groups = (ncol + SG - 1) / SG;
    auto issue = [&](int n) {
        if (!CF::DIRECT && active && n < groups) {
            const uint32_t dst = sm0 + (uint32_t)((n % (S > 0 ? S : 1)) * STAGE) + (uint32_t)(t * (int)sizeof(T));
            const T* src = hp + (size_t)(n * SG) * N;
            const int kc = min(SG, ncol - n * SG);
#pragma unroll
            for (int k = 0; k < SG; ++k, src += N)
                if (k < kc) cp_async<(int)sizeof(T)>(dst + (uint32_t)(k * APPLY_THREADS * (int)sizeof(T)), src);
        }
    };
    // slice 0 is in the first committed group, with or without a ring
    slice(0);
#pragma unroll
    for (int n = 0; n < PROLOGUE; ++n) {
        issue(n);
        cp_commit();
    }

    const int ne = min(MAXE, e1 - e0);
    double b[MAXE][WM];
    int ao[MAXE];
    double cs[MAXE], sn[MAXE];
    auto load_entry = [&](int e, double* bq, int& aq, double& cq, double& sq) {
        aq = __ldg(ent_local + e) * arow;
#pragma unroll
        for (int w = 0; w < WM; ++w) bq[w] = w < wmax ? (double)__ldg(ent_beta + (size_t)e * wmax + w) : 0.0;
        cq = 1.0;
        sq = 0.0;
        if (CPLX) {
            const double kxx = gx_dx * (double)__ldg(ent_xyz + 3 * (size_t)e + 0);
            const double kyy = gy_dy * (double)__ldg(ent_xyz + 3 * (size_t)e + 1);
            const double kzz = gz_dz * (double)__ldg(ent_xyz + 3 * (size_t)e + 2);
            sincos(kxx + kyy + kzz, &sq, &cq);
        }
    };
#pragma unroll
    for (int q = 0; q < MAXE; ++q) {
        if (q < ne) {
            load_entry(e0 + q, b[q], ao[q], cs[q], sn[q]);
        } else {
#pragma unroll
            for (int w = 0; w < WM; ++w) b[q][w] = 0.0;
            ao[q] = 0;
            cs[q] = 1.0;
            sn[q] = 0.0;
        }
    }
    // adds entry (bq, aq, phase) times the staged slice to acc[SG]
    auto contract = [&](const double* sl, const double* bq, int aq, double cq, double sq, int s0, double* acc) {
        if constexpr (!CPLX) {
            // real: no phase, accumulate in place
#pragma unroll
            for (int w = 0; w < WM; ++w) {
                if (w < wmax) {
                    const double* row = sl + aq + w * APPLY_CW + s0;
#pragma unroll
                    for (int k = 0; k < SG; k += 2) {
                        const double2 v = *reinterpret_cast<const double2*>(row + k);
                        acc[k] += bq[w] * v.x;
                        acc[k + 1] += bq[w] * v.y;
                    }
                }
            }
        } else {
            double tq[SG];
#pragma unroll
            for (int k = 0; k < SG; ++k) tq[k] = 0.0;
#pragma unroll
            for (int w = 0; w < WM; ++w) {
                if (w < wmax) {
                    const double* row = sl + aq + w * APPLY_CW + s0;
#pragma unroll
                    for (int k = 0; k < SG; k += 2) {
                        const double2 v = *reinterpret_cast<const double2*>(row + k);
                        tq[k] += bq[w] * v.x;
                        tq[k + 1] += bq[w] * v.y;
                    }
                }
            }
            // exp(-i k.r) (source/PseudoPotNonlocal_SvF2_kpoint.h:4026-4027)
#pragma unroll
            for (int j = 0; j < SG / 2; ++j) {
                acc[2 * j] += cq * tq[2 * j] + sq * tq[2 * j + 1];
                acc[2 * j + 1] += cq * tq[2 * j + 1] - sq * tq[2 * j];
            }
        }
    };
    for (int n = 0; n < groups; ++n) {
        const int sl = n / (APPLY_CW / SG);
        cp_wait<CF::Order::PENDING>();      // groups up to n have landed (this thread's copies)
        if (n % (APPLY_CW / SG) == 0) {
            __syncthreads();                // slice sl is whole, slice sl - 1 is no longer read
            if ((sl + 1) * APPLY_CW < ncol) slice(sl + 1);
        }
        issue(n + PROLOGUE);
        cp_commit();
        if (!active) continue;
        const int kc = min(SG, ncol - n * SG);
        T* out = hp + (size_t)(n * SG) * N;
        T direct[CF::DIRECT ? SG : 1];
        if constexpr (CF::DIRECT) {
#pragma unroll
            for (int k = 0; k < SG; ++k) direct[k] = k < kc ? out[(size_t)k * N] : T(0);
        }
        const T* cur = reinterpret_cast<const T*>(apply_sm + (n % (S > 0 ? S : 1)) * STAGE) + t;
        const double* cf = csm + (size_t)(sl & 1) * max_local * arow;
        const int s0 = n * SG - sl * APPLY_CW;
        double acc[SG];
#pragma unroll
        for (int k = 0; k < SG; ++k) acc[k] = 0.0;
#pragma unroll
        for (int q = 0; q < MAXE; ++q)
            if (q < ne) contract(cf, b[q], ao[q], cs[q], sn[q], s0, acc);
        // points covered by more than MAXE spheres
        for (int e = e0 + MAXE; e < e1; ++e) {
            double bx[WM], cx, sx;
            int ax;
            load_entry(e, bx, ax, cx, sx);
            contract(cf, bx, ax, cx, sx, s0, acc);
        }
#pragma unroll
        for (int k = 0; k < SG; ++k, out += N)
            if (k < kc) *out = (CF::DIRECT ? direct[CF::DIRECT ? k : 0] : cur[k * APPLY_THREADS]) + (T)acc[k];
    }
    cp_wait<0>();
}

template <typename T, bool CPLX, int WM, int CB>
qsb_status launch_proj(const NLDevice& d, const T* beta, int nb, const void* psi, size_t N, double gx_dx,
                       double gy_dy, double gz_dz, double* partial, int ncol, cudaStream_t s) {
    using C = ProjCfg<T, CPLX, WM, CB>;
    auto kern = nl_proj_kernel<T, CPLX, WM, CB>;
    QSB_TRY(allow_shared_memory(kern));
    const dim3 grid((nb + CB - 1) / CB, d.n_chunks);
    kern<<<grid, PROJ_THREADS, C::SMEM, s>>>(d.chunk_order, d.chunk_begin, d.chunk_end, d.pt_idx, d.pt_xyz, beta,
                                             d.wmax, (const T*)psi, N, nb, gx_dx, gy_dy, gz_dz, partial, ncol);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// One table, sums kept per thread
template <typename T, bool CPLX>
qsb_status launch_proj_w(const NLDevice& d, const T* beta, int nb, const void* psi, size_t N, double gx_dx,
                         double gy_dy, double gz_dz, double* partial, int ncol, cudaStream_t s) {
    // bands per CTA: 8 real / 4 complex share one read of the beta rows (16 at one CTA per SM:
    // 0.41 against 0.29 ms, FP64 96^3 x 128); 2 real where
    // that would leave most SMs without a CTA (few chunks and bands: 18.1 -> 13.1 us for
    // 12 chunk-groups; a complex point's sincos costs more than the idle SMs)
    // (half of them at more than 9 projectors: the sums of one thread must fit its registers)
    constexpr int CB = CPLX ? 4 : 8, CBS = CPLX ? 4 : 2;
    const bool few = (long long)((nb + CB - 1) / CB) * d.n_chunks < 148;
#define QSB_PROJ(WM, CBV) \
    return launch_proj<T, CPLX, WM, CBV>(d, beta, nb, psi, N, gx_dx, gy_dy, gz_dz, partial, ncol, s)
    if (few && CBS != CB) {
        if (d.wmax <= 1) QSB_PROJ(1, CBS);
        if (d.wmax <= 4) QSB_PROJ(4, CBS);
    }
    if (d.wmax <= 1) QSB_PROJ(1, CB);
    if (d.wmax <= 4) QSB_PROJ(4, CB);
    if (d.wmax <= 9) QSB_PROJ(9, CB);
    QSB_PROJ(16, (CB / 2));
#undef QSB_PROJ
}

template <typename T, bool CPLX, int MT, int NC, int WARPS>
qsb_status launch_proj_mma(const NLDevice& d, const ProjTables& tabs, const void* psi, size_t N, double gx_dx,
                           double gy_dy, double gz_dz, double* partial, size_t table_stride, int ncol,
                           cudaStream_t s) {
    auto kern = nl_proj_mma_kernel<T, CPLX, MT, NC, WARPS>;
    const MmaLayout ly((int)sizeof(T), NC, MT, tabs.n * d.wmax, CPLX);
    const int smem = std::max(WARPS * ly.warp_bytes, WARPS * 8 * MT * NC * 8);
    QSB_TRY(allow_shared_memory(kern));
    const dim3 grid((ncol + NC - 1) / NC, d.n_chunks);
    kern<<<grid, WARPS * 32, smem, s>>>(d.chunk_order, d.chunk_begin, d.chunk_end, d.pt_idx, d.pt_xyz, tabs,
                                            d.wmax, (const T*)psi, N, gx_dx, gy_dy, gz_dz, partial, table_stride,
                                            ncol);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

// Tensor-core projection on tabs.n tables, partials of table k at partial + k *
// table_stride; tabs.n * wmax <= 16.
template <typename T, bool CPLX>
qsb_status launch_proj_mma_w(const NLDevice& d, const ProjTables& tabs, const void* psi, size_t N, double gx_dx,
                             double gy_dy, double gz_dz, double* partial, size_t table_stride, int ncol,
                             cudaStream_t s) {
    const int rows = tabs.n * d.wmax * (CPLX ? 2 : 1);
    // 32 columns per CTA, two CTAs per SM (fewer warps, then columns, as the rows take more
    // shared memory).  8 columns where fewer CTAs than SMs would come of it, and there with
    // many warps: the time is then a warp's chain of batches, not bandwidth
    const int wide = rows <= 16 ? 32 : 16;
    const bool few = (long long)((ncol + wide - 1) / wide) * d.n_chunks < 148;
#define QSB_PROJ(MT, NC, WARPS) \
    return launch_proj_mma<T, CPLX, MT, NC, WARPS>(d, tabs, psi, N, gx_dx, gy_dy, gz_dz, partial, table_stride, ncol, s)
    if (rows <= 8) {
        if (few) QSB_PROJ(1, 8, 32);
        QSB_PROJ(1, 32, 8);
    }
    if (rows <= 16) {
        if (few) QSB_PROJ(2, 8, 16);
        QSB_PROJ(2, 32, 6);
    }
    if constexpr (CPLX) {
        if (few) QSB_PROJ(4, 8, 12);
        QSB_PROJ(4, 16, 6);
    }
#undef QSB_PROJ
    return fail(QSB_ERR_INVALID, "nonlocal: more than 16 projector rows");
}

// Per atom (one block): energy = sum over bands and projectors of occ E_w |c|^2;
// force_d = sum 2 occ E_w Re(conj(c) g_d) with c = dV <beta|psi>, g_d = dV <d beta/dd|psi>
// (coefficient arrays [atom][w][col], complex bands as columns 2b, 2b+1).
// Fixed-order block reduction: the result does not depend on timing.
__global__ void nl_energy_force_kernel(const double* __restrict__ c, const double* __restrict__ gx,
                                       const double* __restrict__ gy, const double* __restrict__ gz,
                                       const double* __restrict__ atom_E, const int* __restrict__ atom_width, int wmax,
                                       int nb, int is_complex, const double* __restrict__ occ, double* __restrict__ out) {
    const int a = blockIdx.x;
    const int wa = atom_width[a];
    const int ncol = is_complex ? 2 * nb : nb;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = threadIdx.x; i < wa * nb; i += blockDim.x) {
        const int w = i / nb, b = i % nb;
        const double e = atom_E[(size_t)a * wmax + w] * occ[b];
        const size_t base = ((size_t)a * wmax + w) * ncol;
        const int c0 = is_complex ? 2 * b : b;
        const double cr = c[base + c0], ci = is_complex ? c[base + c0 + 1] : 0.0;
        acc[0] += e * (cr * cr + ci * ci);
        if (gx) {
            acc[1] += 2.0 * e * (cr * gx[base + c0] + (is_complex ? ci * gx[base + c0 + 1] : 0.0));
            acc[2] += 2.0 * e * (cr * gy[base + c0] + (is_complex ? ci * gy[base + c0 + 1] : 0.0));
            acc[3] += 2.0 * e * (cr * gz[base + c0] + (is_complex ? ci * gz[base + c0 + 1] : 0.0));
        }
    }
    __shared__ double red[4][256];
#pragma unroll
    for (int k = 0; k < 4; ++k) red[k][threadIdx.x] = acc[k];
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h)
#pragma unroll
            for (int k = 0; k < 4; ++k) red[k][threadIdx.x] += red[k][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x < 4) out[(size_t)a * 4 + threadIdx.x] = red[threadIdx.x][0];
}

}  // namespace

void nl_free(NLDevice& d) {
    for (void*& p : d.tables) dfree(p);
    d.pt_idx = d.pt_xyz = nullptr;
    d.pt_beta64 = nullptr;
    d.pt_beta32 = nullptr;
    d.atom_width = d.atom_proj_off = nullptr;
    d.atom_E = nullptr;
    d.chunk_atom = d.chunk_order = d.chunk_begin = d.chunk_end = d.atom_chunk_begin = d.atom_chunk_end = nullptr;
    d.grid_ptr = d.cov_grid = d.ent_atom = d.ent_local = d.cta_ptr = d.cta_atoms = d.ent_xyz = nullptr;
    d.ent_beta64 = nullptr;
    d.ent_beta32 = nullptr;
    dfree(d.pt_dbeta64); dfree(d.pt_dbeta32);
    d.n_atoms = 0; d.wmax = 0; d.n_points = 0; d.total_proj = 0; d.n_chunks = 0; d.n_cov = 0; d.max_local = 0;
    d.h_atom_width.clear(); d.h_atom_proj_off.clear(); d.h_npts.clear(); d.h_src.clear();
}

qsb_status nl_upload(NLDevice& d, int nx, int ny, int nz, int n_atoms, const int* npts, const int* widths,
                     const int* coords, const double* beta, const double* energy) {
    nl_free(d);
    if (n_atoms < 0) return fail(QSB_ERR_INVALID, "set_projectors: n_atoms < 0");
    const size_t N = (size_t)nx * ny * nz;
    int64_t total = 0;
    int wmax = 0, total_proj = 0;
    for (int a = 0; a < n_atoms; ++a) {
        if (npts[a] < 0 || widths[a] < 0) return fail(QSB_ERR_INVALID, "set_projectors: negative npts/width");
        if (widths[a] > 16) return fail(QSB_ERR_INVALID, "set_projectors: width > 16 per atom is not supported");
        total += npts[a];
        wmax = std::max(wmax, widths[a]);
        total_proj += widths[a];
    }
    if (total >= (int64_t)1 << 31) return fail(QSB_ERR_INVALID, "set_projectors: more than 2^31 points");
    d.n_atoms = n_atoms;
    d.wmax = wmax;
    d.n_points = total;
    d.total_proj = total_proj;
    d.h_atom_width.assign(widths, widths + n_atoms);
    d.h_npts.assign(npts, npts + n_atoms);
    d.h_atom_proj_off.resize(n_atoms);
    {
        int off = 0;
        for (int a = 0; a < n_atoms; ++a) { d.h_atom_proj_off[a] = off; off += widths[a]; }
    }
    if (total == 0 || wmax == 0) {
        // nothing to apply; keep an empty CSR so the fused stencil can skip it
        d.n_points = 0;
        return QSB_OK;
    }

    // atom-major points, sorted by folded grid index within each atom
    std::vector<int> idx(total), xyz(3 * total), atom_of(total);
    d.h_src.assign(total, 0);
    std::vector<double> b64((size_t)total * wmax, 0.0);
    std::vector<double> E((size_t)n_atoms * wmax, 0.0);
    std::vector<int> chunk_atom, chunk_b, chunk_e, acb(n_atoms), ace(n_atoms);
    {
        int64_t off = 0, boff = 0;
        std::vector<int> order;
        for (int a = 0; a < n_atoms; ++a) {
            const int np = npts[a], w = widths[a];
            for (int k = 0; k < w; ++k) E[(size_t)a * wmax + k] = energy[d.h_atom_proj_off[a] + k];
            order.resize(np);
            std::vector<int> fidx(np);
            for (int i = 0; i < np; ++i) {
                const int* c = coords + 3 * (off + i);
                fidx[i] = fold(c[0], nx) + nx * (fold(c[1], ny) + ny * fold(c[2], nz));
            }
            std::iota(order.begin(), order.end(), 0);
            std::stable_sort(order.begin(), order.end(), [&](int u, int v) { return fidx[u] < fidx[v]; });
            for (int i = 0; i < np; ++i) {
                const int src = order[i];
                const int64_t dst = off + i;
                idx[dst] = fidx[src];
                atom_of[dst] = a;
                d.h_src[dst] = src;
                for (int c = 0; c < 3; ++c) xyz[3 * dst + c] = coords[3 * (off + src) + c];
                for (int k = 0; k < w; ++k) b64[(size_t)dst * wmax + k] = beta[boff + (int64_t)k * np + src];
            }
            acb[a] = (int)chunk_b.size();
            if (w > 0)
                for (int i = 0; i < np; i += CHUNK) {
                    chunk_atom.push_back(a);
                    chunk_b.push_back((int)(off + i));
                    chunk_e.push_back((int)(off + std::min(np, i + CHUNK)));
                }
            ace[a] = (int)chunk_b.size();
            off += np;
            boff += (int64_t)np * w;
        }
    }
    d.n_chunks = (int)chunk_b.size();
    // launch order of the projection: by the grid index of each chunk's middle point
    std::vector<int> corder(d.n_chunks);
    std::iota(corder.begin(), corder.end(), 0);
    {
        std::vector<int> mid(d.n_chunks);
        for (int c = 0; c < d.n_chunks; ++c) mid[c] = idx[(chunk_b[c] + chunk_e[c] - 1) / 2];
        std::stable_sort(corder.begin(), corder.end(), [&](int u, int v) { return mid[u] < mid[v]; });
    }

    // grid-ordered CSR (counting sort by folded index, stable in atom-major order)
    std::vector<int> gptr(N + 1, 0);
    for (int64_t p = 0; p < total; ++p) gptr[idx[p] + 1]++;
    for (size_t g = 0; g < N; ++g) gptr[g + 1] += gptr[g];
    std::vector<int> fillp(gptr.begin(), gptr.end() - 1);
    std::vector<int> e_atom(total), e_xyz(3 * total);
    std::vector<double> e_b64((size_t)total * wmax);
    for (int64_t p = 0; p < total; ++p) {
        const int e = fillp[idx[p]]++;
        e_atom[e] = atom_of[p];
        for (int c = 0; c < 3; ++c) e_xyz[3 * e + c] = xyz[3 * p + c];
        for (int k = 0; k < wmax; ++k) e_b64[(size_t)e * wmax + k] = b64[(size_t)p * wmax + k];
    }
    std::vector<int> cov;
    for (size_t g = 0; g < N; ++g)
        if (gptr[g + 1] > gptr[g]) cov.push_back((int)g);
    d.n_cov = (int)cov.size();

    // atoms of each run of APPLY_THREADS covered points (one CTA of the expansion), ascending,
    // and every entry's place in its run's list
    std::vector<int> cptr(1, 0), catoms, e_local(total);
    d.max_local = 0;
    {
        std::vector<int> seen(n_atoms, -1), place(n_atoms), here;
        for (size_t r0 = 0; r0 < cov.size(); r0 += APPLY_THREADS) {
            const size_t r1 = std::min(cov.size(), r0 + (size_t)APPLY_THREADS);
            here.clear();
            for (size_t r = r0; r < r1; ++r)
                for (int e = gptr[cov[r]]; e < gptr[cov[r] + 1]; ++e)
                    if (seen[e_atom[e]] != (int)r0) {
                        seen[e_atom[e]] = (int)r0;
                        here.push_back(e_atom[e]);
                    }
            std::sort(here.begin(), here.end());
            for (size_t i = 0; i < here.size(); ++i) place[here[i]] = (int)i;
            for (int e = gptr[cov[r0]]; e < gptr[cov[r1 - 1] + 1]; ++e) e_local[e] = place[e_atom[e]];
            catoms.insert(catoms.end(), here.begin(), here.end());
            cptr.push_back((int)catoms.size());
            d.max_local = std::max(d.max_local, (int)here.size());
        }
    }

    std::vector<float> b32(b64.begin(), b64.end()), e_b32(e_b64.begin(), e_b64.end());
    TableUpload up;
    up.add(d.pt_idx, idx);
    up.add(d.pt_xyz, xyz);
    up.add(d.pt_beta64, b64);
    up.add(d.pt_beta32, b32);
    up.add(d.atom_width, widths, (size_t)n_atoms);
    up.add(d.atom_proj_off, d.h_atom_proj_off.data(), (size_t)n_atoms);
    up.add(d.atom_E, E);
    up.add(d.chunk_atom, chunk_atom);
    up.add(d.chunk_order, corder);
    up.add(d.chunk_begin, chunk_b);
    up.add(d.chunk_end, chunk_e);
    up.add(d.atom_chunk_begin, acb);
    up.add(d.atom_chunk_end, ace);
    up.add(d.grid_ptr, gptr);
    up.add(d.cov_grid, cov);
    up.add(d.ent_atom, e_atom);
    up.add(d.ent_local, e_local);
    up.add(d.cta_ptr, cptr);
    up.add(d.cta_atoms, catoms);
    up.add(d.ent_xyz, e_xyz);
    up.add(d.ent_beta64, e_b64);
    up.add(d.ent_beta32, e_b32);
    const qsb_status st = up.run(d.tables);
    if (st != QSB_OK) nl_free(d);           // no projectors rather than half of them
    return st;
}

size_t nl_workspace_bytes(const NLDevice& d, int ncol) {
    if (d.n_points == 0) return 0;
    const size_t part = (size_t)d.n_chunks * d.wmax * ncol * sizeof(double);
    const size_t coef = (size_t)d.n_atoms * d.wmax * ncol * sizeof(double);
    return ((part + 255) / 256) * 256 + ((coef + 255) / 256) * 256;
}

namespace {
// coef_out[k] of table first_table + k (-1: beta, 0..2: the gradient tables), each
// table with its own partials and coefficients in ws (nl_workspace_bytes apart)
qsb_status nl_project_tables(qsb_dtype dt, const NLDevice& d, int first_table, int ntab, int nx, int ny, int nz, int nb,
                             int is_complex, const void* psi, double dV, double gx_dx, double gy_dy, double gz_dz,
                             bool inner_only, void* ws, double** coef_out, cudaStream_t s) {
    const size_t N = (size_t)nx * ny * nz;
    const int ncol = is_complex ? 2 * nb : nb;
    const size_t part = (size_t)d.n_chunks * d.wmax * ncol * sizeof(double);
    const size_t one = nl_workspace_bytes(d, ncol);
    double* partial = (double*)ws;
    ProjTables tabs{};
    for (int k = 0; k < ntab; ++k) {
        coef_out[k] = (double*)((char*)ws + k * one + ((part + 255) / 256) * 256);
        const int table = first_table + k;
        const size_t toff = table < 0 ? 0 : (size_t)table * d.n_points * d.wmax;
        if (dt == QSB_F64) tabs.t[k] = table < 0 ? d.pt_beta64 : d.pt_dbeta64 + toff;
        else tabs.t[k] = table < 0 ? (const void*)d.pt_beta32 : (const void*)(d.pt_dbeta32 + toff);
    }
    if (d.n_points == 0) return QSB_OK;
    if ((nb + 7) / 8 > 65535) return fail(QSB_ERR_INVALID, "nonlocal: too many bands");
    const size_t stride = one / sizeof(double);
    tabs.n = ntab;
    // The tensor-core form where its rows are full: a complex bundle (the phases once per 32
    // columns instead of once per 8: 48^3 x 24 bands, FP64, 45 -> 27 us) and the forces' four
    // tables (0.75 against 1.07 ms at 96^3 x 128); one real table fills half of them and runs
    // faster in the other (0.29 against 0.48 ms).  FP32 applies keep that one's order of sums.
#define QSB_MMA(T, C) launch_proj_mma_w<T, C>(d, tabs, psi, N, gx_dx, gy_dy, gz_dz, partial, stride, ncol, s)
#define QSB_VEC(T, C) launch_proj_w<T, C>(d, (const T*)tabs.t[0], nb, psi, N, gx_dx, gy_dy, gz_dz, partial, ncol, s)
    if (dt == QSB_F64) {
        if (is_complex) QSB_TRY((QSB_MMA(double, true)));
        else if (ntab > 1) QSB_TRY((QSB_MMA(double, false)));
        else QSB_TRY((QSB_VEC(double, false)));
    } else {
        if (ntab > 1) QSB_TRY(is_complex ? (QSB_MMA(float, true)) : (QSB_MMA(float, false)));
        else QSB_TRY(is_complex ? (QSB_VEC(float, true)) : (QSB_VEC(float, false)));
    }
#undef QSB_MMA
#undef QSB_VEC
    for (int k = 0; k < ntab; ++k)
        nl_finalize_kernel<<<d.n_atoms, 256, 0, s>>>(d.atom_chunk_begin, d.atom_chunk_end, d.atom_E, d.atom_width,
                                                     d.wmax, partial + k * stride, ncol, dV, inner_only ? 1 : 0,
                                                     coef_out[k]);
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}
}  // namespace

qsb_status nl_project(qsb_dtype dt, const NLDevice& d, int nx, int ny, int nz, int nb, int is_complex,
                      const void* psi, double dV, double gx_dx, double gy_dy, double gz_dz, bool inner_only, void* ws,
                      double** coef_out, cudaStream_t s) {
    return nl_project_tables(dt, d, -1, 1, nx, ny, nz, nb, is_complex, psi, dV, gx_dx, gy_dy, gz_dz, inner_only, ws,
                             coef_out, s);
}

qsb_status nl_upload_gradients(NLDevice& d, const double* dbeta) {
    if (d.n_points == 0 || d.wmax == 0) return QSB_OK;
    if (!dbeta) return fail(QSB_ERR_INVALID, "set_projector_gradients: null table");
    const size_t per_dir = (size_t)d.n_points * d.wmax;
    std::vector<double> g64(3 * per_dir, 0.0);
    int64_t off = 0, goff = 0;
    for (int a = 0; a < d.n_atoms; ++a) {
        const int np = d.h_npts[a], w = d.h_atom_width[a];
        for (int i = 0; i < np; ++i) {
            const int64_t dst = off + i;
            const int src = d.h_src[dst];
            for (int dir = 0; dir < 3; ++dir)
                for (int k = 0; k < w; ++k)
                    g64[dir * per_dir + (size_t)dst * d.wmax + k] =
                        dbeta[goff + (int64_t)dir * np * w + (int64_t)k * np + src];
        }
        off += np;
        goff += (int64_t)3 * np * w;
    }
    std::vector<float> g32(g64.begin(), g64.end());
    dfree(d.pt_dbeta64);
    dfree(d.pt_dbeta32);
    QSB_CUDA_TRY(cudaMalloc((void**)&d.pt_dbeta64, g64.size() * sizeof(double)));
    QSB_CUDA_TRY(cudaMalloc((void**)&d.pt_dbeta32, g32.size() * sizeof(float)));
    QSB_CUDA_TRY(cudaMemcpy(d.pt_dbeta64, g64.data(), g64.size() * sizeof(double), cudaMemcpyHostToDevice));
    QSB_CUDA_TRY(cudaMemcpy(d.pt_dbeta32, g32.data(), g32.size() * sizeof(float), cudaMemcpyHostToDevice));
    return QSB_OK;
}

size_t nl_energy_force_bytes(const NLDevice& d, int ncol, int nb) {
    const size_t one = nl_workspace_bytes(d, ncol);
    return 4 * one + (((size_t)d.n_atoms * 4 + nb) * sizeof(double) + 256);
}

qsb_status nl_energy_force(qsb_dtype dt, const NLDevice& d, int nx, int ny, int nz, int nb, int is_complex,
                           const void* psi, const double* occ_host, double dV, double gx_dx, double gy_dy,
                           double gz_dz, double* energy, double* forces, void* ws, cudaStream_t s) {
    *energy = 0.0;
    if (d.n_points == 0 || nb == 0) return QSB_OK;
    if (forces && !d.pt_dbeta64) return fail(QSB_ERR_STATE, "nonlocal forces: no projector gradients set");
    const int ncol = is_complex ? 2 * nb : nb;
    const size_t one = nl_workspace_bytes(d, ncol);
    unsigned char* w = (unsigned char*)ws;
    double* coef[4] = {nullptr, nullptr, nullptr, nullptr};
    const int ntab = forces ? 4 : 1;
    // beta and its gradients share one gather of psi up to 4 projectors per atom (16 rows)
    const int at_once = ntab == 4 && d.wmax <= 4 ? 4 : 1;
    for (int t = 0; t < ntab; t += at_once)
        QSB_TRY(nl_project_tables(dt, d, t - 1, at_once, nx, ny, nz, nb, is_complex, psi, dV, gx_dx, gy_dy, gz_dz,
                                  true, w + t * one, &coef[t], s));
    double* out = (double*)(w + 4 * one);
    double* occ = out + (size_t)d.n_atoms * 4;
    QSB_CUDA_TRY(cudaMemcpyAsync(occ, occ_host, sizeof(double) * nb, cudaMemcpyHostToDevice, s));
    nl_energy_force_kernel<<<d.n_atoms, 256, 0, s>>>(coef[0], coef[1], coef[2], coef[3], d.atom_E, d.atom_width,
                                                     d.wmax, nb, is_complex, occ, out);
    QSB_CUDA_TRY(cudaGetLastError());
    std::vector<double> h((size_t)d.n_atoms * 4);
    QSB_CUDA_TRY(cudaMemcpyAsync(h.data(), out, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
    QSB_CUDA_TRY(cudaStreamSynchronize(s));
    double e = 0.0;
    for (int a = 0; a < d.n_atoms; ++a) {
        e += h[(size_t)a * 4];
        if (forces)
            for (int k = 0; k < 3; ++k) forces[3 * a + k] += h[(size_t)a * 4 + 1 + k];
    }
    if (!std::isfinite(e)) return fail(QSB_ERR_NUMERIC, "nonlocal energy: non-finite value");
    *energy = e;
    return QSB_OK;
}

qsb_status nl_apply(qsb_dtype dt, const NLDevice& d, int N, int nb, int is_complex, void* hpsi, const double* coef,
                    double gx_dx, double gy_dy, double gz_dz, cudaStream_t s) {
    if (d.n_points == 0 || d.n_cov == 0) return QSB_OK;
    const int ncol = is_complex ? 2 * nb : nb;
    const dim3 grid((d.n_cov + APPLY_THREADS - 1) / APPLY_THREADS);
    // pipelined form while two slices of the CTA's own atoms fit beside the ring (up to
    // ~60 atoms x 4 projectors meeting in 256 points at two CTAs per SM); else per-point loads
#define QSB_APPLY(T, C, W, B)                                                                                        \
    do {                                                                                                             \
        const size_t smem = (size_t)ApplyCfg<T, C>::RING +                                                                \
                            (size_t)2 * d.max_local * apply_row(d.wmax) * sizeof(double);                            \
        if (smem <= 200 * 1024) {                                                                                    \
            auto kern = d.wmax == W ? nl_apply_ring_kernel<T, C, W, true> : nl_apply_ring_kernel<T, C, W, false>;    \
            QSB_TRY(allow_shared_memory(kern));        \
            kern<<<grid, APPLY_THREADS, smem, s>>>(d.cov_grid, d.n_cov, d.grid_ptr, d.ent_local, d.ent_xyz, B,       \
                                                   d.wmax, d.cta_ptr, d.cta_atoms, d.max_local, coef, ncol,          \
                                                   (T*)hpsi, (size_t)N, gx_dx, gy_dy, gz_dz);                        \
        } else {                                                                                                     \
            nl_apply_kernel<T, C, W><<<grid, APPLY_THREADS, 0, s>>>(d.cov_grid, d.n_cov, d.grid_ptr, d.ent_atom,      \
                                                                    d.ent_xyz, B, d.wmax, coef, ncol, (T*)hpsi,      \
                                                                    (size_t)N, nb, gx_dx, gy_dy, gz_dz);            \
        }                                                                                                            \
    } while (0)
#define QSB_APPLY_W(T, C, B)                      \
    do {                                          \
        if (d.wmax <= 1) QSB_APPLY(T, C, 1, B);   \
        else if (d.wmax <= 4) QSB_APPLY(T, C, 4, B); \
        else if (d.wmax <= 9) QSB_APPLY(T, C, 9, B); \
        else QSB_APPLY(T, C, 16, B);              \
    } while (0)
    if (dt == QSB_F64) {
        if (is_complex) QSB_APPLY_W(double, true, d.ent_beta64);
        else QSB_APPLY_W(double, false, d.ent_beta64);
    } else {
        if (is_complex) QSB_APPLY_W(float, true, d.ent_beta32);
        else QSB_APPLY_W(float, false, d.ent_beta32);
    }
#undef QSB_APPLY_W
#undef QSB_APPLY
    QSB_CUDA_TRY(cudaGetLastError());
    return QSB_OK;
}

}  // namespace qsb
