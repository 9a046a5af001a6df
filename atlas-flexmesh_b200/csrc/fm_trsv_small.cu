// fm_trsv_small.cu — triangular solves of a generic CSR factorization whose
// vector fits one SM's shared memory.
//
// On short rows the solves are chains of dependency levels with little work
// in each (2 x 299 levels of at most 150 rows on a 150 x 150 five-point
// matrix), so their time is the cost of passing values from one level to the
// next.  Through L2, with a warp per row and a release flag each, a level
// cost 3.7 us (2.2 ms per apply there).  Here one CTA keeps the whole vector
// in shared memory and takes a level at a time, one thread per row, with a
// block barrier between levels: 0.19 us per level.
//
// The factors come as one stream per direction in level order, entry m of
// position t at [m * n + t] (rows with fewer entries are padded with zero
// coefficients that read a zero), packed after each factorization; a
// thread's entries of the next level are in flight in registers (113 us per
// apply there; two, three and four levels ahead, with the loop unrolled as
// often, took 125, 126 and 141; 16-byte packed rows 160, a cp.async ring 143;
// a build without any loads in the loop 90).
//
// Used when the vector and the level pointers fit shared memory, no row has
// more than kSmallMaxEntries off-diagonal entries on one side (longer rows
// would leave a thread with a long serial sum) and the levels are not too wide
// (small_tri_pays).  The rest belongs to the warp-per-row solves.
#include <algorithm>
#include <vector>

#include "fm_kernels.hpp"

namespace fm {

namespace {

template <int M>
struct Row {
    double v[M];
    uint32_t c[M];
    double d;
    uint32_t row;
};

// the row at position t (unconditional, so that nothing waits for the loads
// before the row is solved: the caller clamps t)
template <int M, bool Upper>
__device__ __forceinline__ void load_row(const SmallTri& S, uint32_t t, uint32_t n, Row<M>& E) {
    E.row = __ldg(S.row + t);
    if (Upper) E.d = __ldg(S.dinv + t);
#pragma unroll
    for (int m = 0; m < M; ++m) {
        E.c[m] = __ldg(S.col + (size_t)m * n + t);
        E.v[m] = __ldg(S.val + (size_t)m * n + t);
    }
}

template <int M, bool Upper>
__device__ __forceinline__ void solve_row(const Row<M>& E, double* z) {
    double s = z[E.row];
#pragma unroll
    for (int m = 0; m < M; ++m) s -= E.v[m] * z[E.c[m]];
    z[E.row] = Upper ? s * E.d : s;
}

// one direction, in place on z (z[n] = 0 for the padding); lvl[n_levels] and
// lvl[n_levels + 1] = n
template <int M, bool Wide, bool Upper>
__device__ __forceinline__ void sweep(const SmallTri& S, const uint32_t* lvl, uint32_t n,
                                      double* z) {
    Row<M> e;
    load_row<M, Upper>(S, min(lvl[0] + threadIdx.x, n - 1), n, e);
    for (uint32_t l = 0; l < S.n_levels; ++l) {
        const uint32_t b = lvl[l], end = lvl[l + 1];
        if (b + threadIdx.x < end) solve_row<M, Upper>(e, z);
        if (Wide)  // rows of a level beyond the block's width
            for (uint32_t t = b + threadIdx.x + blockDim.x; t < end; t += blockDim.x) {
                Row<M> x;
                load_row<M, Upper>(S, t, n, x);
                solve_row<M, Upper>(x, z);
            }
        load_row<M, Upper>(S, min(end + threadIdx.x, n - 1), n, e);
        __syncthreads();
    }
}

template <int M, int Threads, bool Wide>
__global__ void __launch_bounds__(Threads, 1)
    k_trsv_small(SmallTri L, SmallTri U, uint32_t n, const double* r, double* out,
                 const unsigned* skip) {
    chain_begin();
    if (skipped(skip)) return;
    extern __shared__ __align__(16) unsigned char small_smem[];
    double* z = reinterpret_cast<double*>(small_smem);
    uint32_t* lf = reinterpret_cast<uint32_t*>(z + n + 1);
    uint32_t* lb = lf + L.n_levels + 2;
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) z[i] = ld_prev(r + i);
    if (threadIdx.x == 0) z[n] = 0.0;
    for (uint32_t i = threadIdx.x; i <= L.n_levels + 1; i += blockDim.x)
        lf[i] = i < L.n_levels ? __ldg(L.level + i) : n;
    for (uint32_t i = threadIdx.x; i <= U.n_levels + 1; i += blockDim.x)
        lb[i] = i < U.n_levels ? __ldg(U.level + i) : n;
    __syncthreads();
    sweep<M, Wide, false>(L, lf, n, z);
    sweep<M, Wide, true>(U, lb, n, z);
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) out[i] = z[i];
}

__global__ void k_pack_small(uint32_t n, uint32_t total, const uint32_t* __restrict__ src_f,
                             const uint32_t* __restrict__ src_b,
                             const uint32_t* __restrict__ row_b, const double* __restrict__ lu,
                             const double* __restrict__ diag, double* __restrict__ val_f,
                             double* __restrict__ val_b, double* __restrict__ dinv) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += gridDim.x * blockDim.x) {
        const uint32_t a = src_f[i], b = src_b[i];
        val_f[i] = a != ~0u ? lu[a] : 0.0;
        val_b[i] = b != ~0u ? lu[b] : 0.0;
        if (i < n) dinv[i] = 1.0 / diag[row_b[i]];
    }
}

template <int M, int Threads, bool Wide>
cudaError_t launch_w(const SmallTri& L, const SmallTri& U, uint32_t n, unsigned th, size_t smem,
                     const double* r, double* out, const unsigned* skip, cudaStream_t s) {
    // one limit for every matrix: it is the kernel's, not the call's, and
    // another thread may be between its own call and launch
    const cudaError_t e =
        cudaFuncSetAttribute(k_trsv_small<M, Threads, Wide>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallMaxSmem);
    if (e != cudaSuccess) return e;
    return launch_chained(k_trsv_small<M, Threads, Wide>, 1, th, smem, s, L, U, n, r, out, skip);
}

// threads of the widest block that the registers of a row allow
constexpr unsigned max_threads(uint32_t entries) { return entries <= 2 ? 1024 : 512; }
// no more threads than the widest level has rows (fewer warps, a cheaper
// barrier) or than the copies in and out can use
unsigned threads_for(uint32_t entries, uint32_t n, uint32_t width) {
    return std::min(max_threads(entries),
                    std::max(32u, (std::max(width, n / 64) + 31u) & ~31u));
}

template <int M, int Threads>
cudaError_t launch_t(const SmallTri& L, const SmallTri& U, uint32_t n, uint32_t width,
                     const double* r, double* out, const unsigned* skip, cudaStream_t s) {
    const size_t smem = small_tri_smem(n, L.n_levels, U.n_levels);
    const unsigned th = threads_for(M, n, width);
    return width > th ? launch_w<M, Threads, true>(L, U, n, th, smem, r, out, skip, s)
                      : launch_w<M, Threads, false>(L, U, n, th, smem, r, out, skip, s);
}

}  // namespace

size_t small_tri_smem(uint32_t n, uint32_t nlf, uint32_t nlb) {
    return 8 * ((size_t)n + 1) + 4 * ((size_t)nlf + nlb + 4);
}

// A level costs the warp-per-row solves about 3.9 us whatever its width (148
// SMs take its rows at once), and one CTA half a microsecond for every block's
// width of rows in it.  us per apply on both paths, warp per row / one CTA:
// diagonal of 7,000 rows 17.9 / 15.1, of 14,000 21.9 / 21.6, of 27,000 27.1 /
// 36.0; red-black five-point 90 x 90 25.7 / 21.0, 120 x 120 26.6 / 31.4, 164 x
// 164 27.0 / 53.6; 26,000 rows in four levels 40.8 / 35.2, in three 31.5 / 33.8
// (two entries per side), in eleven 101 / 59 (four), in eight 79 / 76 and in
// six 54 / 75 (eight).
bool small_tri_pays(uint32_t entries, uint32_t n, const std::vector<uint32_t>& fwd_ptr,
                    const std::vector<uint32_t>& bwd_ptr) {
    uint64_t turns = 0, levels = 0;
    uint32_t width = 0;
    for (const auto* p : {&fwd_ptr, &bwd_ptr})
        for (size_t l = 0; l + 1 < p->size(); ++l) width = std::max(width, (*p)[l + 1] - (*p)[l]);
    const uint32_t th = threads_for(entries, n, width);
    for (const auto* p : {&fwd_ptr, &bwd_ptr})
        for (size_t l = 0; l + 1 < p->size(); ++l, ++levels)
            turns += ((*p)[l + 1] - (*p)[l] + th - 1) / th;
    return (entries <= 4 ? 50 : 55) * turns <= 390 * levels + 250;
}

void launch_pack_small(uint32_t n, uint32_t entries, const uint32_t* src_f, const uint32_t* src_b,
                       const uint32_t* row_b, const double* lu, const double* diag, double* val_f,
                       double* val_b, double* dinv, cudaStream_t s) {
    const uint32_t total = entries * n;
    k_pack_small<<<(total + 255) / 256, 256, 0, s>>>(n, total, src_f, src_b, row_b, lu, diag,
                                                     val_f, val_b, dinv);
}

cudaError_t launch_trsv_small(const SmallTri& L, const SmallTri& U, uint32_t n, uint32_t entries,
                              uint32_t width, const double* r, double* out, const unsigned* skip,
                              cudaStream_t s) {
    if (entries <= 2) return launch_t<2, max_threads(2)>(L, U, n, width, r, out, skip, s);
    if (entries <= 4) return launch_t<4, max_threads(4)>(L, U, n, width, r, out, skip, s);
    return launch_t<8, max_threads(8)>(L, U, n, width, r, out, skip, s);
}

}  // namespace fm
