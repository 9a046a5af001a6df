// fm_spmv.cu — y = K x on the node-block solve pattern.
//
// A warp that loads its own node's row pointer, then its entries and
// neighbours, then x, has three dependent latencies per node, and the sums of
// three rows over a warp are a third of its instructions (72 us at 64^3 FP32,
// 57 us at 48^3 FP64; issue slots 60% busy, DRAM 36%).  Here each CTA takes
// tiles of 16 consecutive nodes; a producer thread copies a tile's entries,
// neighbour lists and row pointers, all contiguous, into a shared-memory
// stage with bulk copies (cp.async.bulk) several tiles ahead, and eight warps
// take two nodes each from the stage, one per half-warp.  What is left on a
// warp's path is the gather of x, which hits L1 and L2.  64^3 FP32 72 -> 47.6
// us (210 MB, 0.67 of the copy bandwidth), FP64 117 -> 69 us (390 MB, 0.86);
// 48^3 FP64 57 -> 36 us; at 8^3 the two are equal (9.8 us).
//
// Bulk copies start and end on 16-byte boundaries: the tile is widened to
// them (at most 15 bytes on either side; K and the neighbour lists are
// allocated with that much room at the end).
#include <algorithm>

#include "fm_cluster.cuh"
#include "fm_kernels.hpp"

namespace fm {

namespace {

constexpr int kTile = 16;                  // nodes per tile
constexpr int kTakers = kTile / 2;         // consumer warps, two nodes each
constexpr int kStreamThreads = 32 * (kTakers + 1);  // and a producer warp
constexpr int kRounds = 4;  // columns per lane held in registers: 64 of a row's at most 96
constexpr unsigned kPtrBytes = 4 * (kTile + 4);  // kTile + 1 row pointers, to 16 bytes

__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Wait for the phase with the given parity; false: given up after kWaitCycles
// (the copies are this CTA's own, so neither the context's limit for waits on
// other warps nor an earlier timeout ends it: a CTA must not leave while a
// copy into its shared memory is in flight).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, unsigned parity, unsigned* status) {
    const auto test = [&] {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        return ok != 0u;
    };
    if (test()) return true;
    const long long t0 = clock64();
    while (!test())
        if (clock64() - t0 > kWaitCycles) {
            raise_flag(status, FM_FLAG_TIMEOUT);
            return false;
        }
    return true;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, unsigned bytes,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

// the 16-byte-aligned range that holds elements [b, e) of an array of
// `size`-byte elements: first byte and length
__device__ __forceinline__ void widen(uint64_t b, uint64_t e, unsigned size, uint64_t& first,
                                      unsigned& bytes) {
    first = (b * size) & ~15ull;
    bytes = (unsigned)(((e * size + 15ull) & ~15ull) - first);
}

// A stage: the tile's entries, its neighbour lists (each with 32 bytes of
// room for the widening), and its row pointers.
struct StageLayout {
    uint32_t nbr, ptr, bytes;
};
template <typename T>
StageLayout stage_layout(uint32_t max_deg) {
    StageLayout l;
    l.nbr = (uint32_t)(((size_t)kTile * 9 * max_deg * sizeof(T) + 15) / 16 * 16 + 32);
    l.ptr = l.nbr + (kTile * max_deg * 4 + 15) / 16 * 16 + 32;
    l.bytes = l.ptr + kPtrBytes;
    return l;
}

// Sums of a, b and c over each half-warp, dropping half of the values in each
// of the first two rounds: 5 shuffles instead of 12.  The sums end in lanes
// 0, 4 and 8 of the half.
template <typename T>
__device__ __forceinline__ T half_sum3(T a, T b, T c, int hl) {
    const bool h = hl & 8, q = hl & 4;
    // lanes below 8 keep a and b, the others c
    const T u = (h ? c : a) + __shfl_xor_sync(kFull, h ? a : c, 8);
    const T v = b + __shfl_xor_sync(kFull, b, 8);
    T r = !h && q ? v : u;
    r += __shfl_xor_sync(kFull, !h && !q ? v : u, 4);
    r += __shfl_xor_sync(kFull, r, 2);
    r += __shfl_xor_sync(kFull, r, 1);
    return r;
}

template <typename T, int S>
__global__ void __launch_bounds__(kStreamThreads)
    k_spmv_nodes(uint32_t nn, StageLayout L, const uint32_t* __restrict__ nbr_ptr,
                  const uint32_t* __restrict__ nbr, const T* __restrict__ val,
                  const T* x, T* __restrict__ y, T* partials, unsigned* counter, double* dot,
                  const unsigned* skip, unsigned* status) {
    extern __shared__ __align__(16) unsigned char stream_smem[];
    __shared__ __align__(8) unsigned long long full_s[S], empty_s[S];
    chain_let_next();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int q = 0; q < S; ++q) {
            mbar_init(clu::smem_u32(&full_s[q]), 1);
            mbar_init(clu::smem_u32(&empty_s[q]), kTakers);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    chain_wait();
    if (skipped(skip)) return;
    const uint32_t tiles = (nn + kTile - 1) / kTile;
    const uint32_t smem = clu::smem_u32(stream_smem);
    T dsum = T(0);
    if (w == kTakers) {
        if (lane == 0) {
            uint32_t i = 0;
            for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
                const uint32_t n0 = t * kTile, n1 = min(nn, n0 + kTile);
                const uint32_t b = __ldg(nbr_ptr + n0), e = __ldg(nbr_ptr + n1);
                const uint32_t q = i % S;
                // the stage's previous tile has been taken by all warps
                if (i >= S && !mbar_wait(clu::smem_u32(&empty_s[q]), (i / S - 1) & 1, status))
                    break;
                uint64_t kf, nf;
                unsigned kb, nb;
                widen(9ull * b, 9ull * e, sizeof(T), kf, kb);
                widen(b, e, 4, nf, nb);
                const uint32_t bar = clu::smem_u32(&full_s[q]), dst = smem + q * L.bytes;
                mbar_expect(bar, kb + nb + kPtrBytes);
                bulk_load(dst + L.ptr, nbr_ptr + n0, kPtrBytes, bar);
                if (kb)
                    bulk_load(dst, reinterpret_cast<const unsigned char*>(val) + kf, kb, bar);
                if (nb)
                    bulk_load(dst + L.nbr, reinterpret_cast<const unsigned char*>(nbr) + nf, nb,
                              bar);
            }
            // every copy has landed before this CTA leaves (at once unless a
            // warp gave up)
            for (uint32_t k = i > S ? i - S : 0; k < i; ++k)
                mbar_wait(clu::smem_u32(&full_s[k % S]), (k / S) & 1, status);
        }
    } else {
        const int hl = lane & 15, mine = 2 * w + (lane >> 4);  // node of the tile
        int ck[kRounds], cq[kRounds];  // neighbour and component of the lane's columns
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            ck[r] = (hl + 16 * r) / 3;
            cq[r] = (hl + 16 * r) % 3;
        }
        uint32_t q = 0, phase = 0;
        for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
            if (!__all_sync(kFull, mbar_wait(clu::smem_u32(&full_s[q]), phase, status))) break;
            const unsigned char* st = stream_smem + q * L.bytes;
            const uint32_t* ptr = reinterpret_cast<const uint32_t*>(st + L.ptr);
            const uint32_t n = t * kTile + mine, b = ptr[0], nb0 = ptr[mine];
            const int rl = n < nn ? 3 * (int)(ptr[mine + 1] - nb0) : 0;
            const int most = max(rl, __shfl_xor_sync(kFull, rl, 16));
            // the tile's first entry and neighbour sit where widening put them
            const T* v = reinterpret_cast<const T*>(st + ((9u * sizeof(T) * b) & 15u)) +
                         9 * (nb0 - b) + hl;
            const uint32_t* nl =
                reinterpret_cast<const uint32_t*>(st + L.nbr + ((4u * b) & 15u)) + (nb0 - b);
            T xv[kRounds], s0 = T(0), s1 = T(0), s2 = T(0);
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {  // gathers in flight together
                xv[r] = T(0);
                if (hl + 16 * r < rl) xv[r] = ld_prev(x + (3u * nl[ck[r]] + (unsigned)cq[r]));
            }
#pragma unroll
            for (int r = 0; r < kRounds; ++r)
                if (hl + 16 * r < rl) {
                    s0 += v[16 * r] * xv[r];
                    s1 += v[rl + 16 * r] * xv[r];
                    s2 += v[2 * rl + 16 * r] * xv[r];
                }
            // nodes of more than 21 neighbours
            for (int idx = hl + 16 * kRounds; 16 * kRounds < most && idx < rl; idx += 16) {
                const T xi = ld_prev(x + (3u * nl[idx / 3] + (unsigned)(idx % 3)));
                s0 += v[idx - hl] * xi;
                s1 += v[rl + idx - hl] * xi;
                s2 += v[2 * rl + idx - hl] * xi;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(clu::smem_u32(&empty_s[q]));
            if (++q == S) {
                q = 0;
                phase ^= 1u;
            }
            const T yv = half_sum3(s0, s1, s2, hl);
            if ((hl & 3) == 0 && hl < 12 && n < nn) {  // lanes 0, 4, 8 of the half
                const uint32_t row = 3 * n + (uint32_t)(hl >> 2);
                y[row] = yv;
                if (dot) dsum += yv * ld_prev(x + row);
            }
        }
    }
    __syncwarp();
    if (dot) {
        __shared__ T sbuf[32];
        const T bt = block_sum(dsum, sbuf);
        grid_reduce_finish<T>(bt, partials, counter, [&](T total) { *dot = (double)total; });
    }
}

constexpr size_t kSmStages = 220 * 1024;  // shared memory of an SM for its CTAs' stages

template <typename T, int S>
cudaError_t launch_stages(uint32_t nn, const StageLayout& L, int per_sm, const uint32_t* nbr_ptr,
                          const uint32_t* nbr, const T* val, const T* x, T* y, T* partials,
                          unsigned* counter, double* dot, unsigned* status, cudaStream_t s,
                          const unsigned* skip) {
    const size_t smem = (size_t)S * L.bytes;
    // The limit is the kernel's own, shared by every context and thread on the
    // device: always the same value, so that a thread with a smaller mesh
    // cannot lower it between another thread's call and launch.
    const cudaError_t e = cudaFuncSetAttribute(
        k_spmv_nodes<T, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmStages / S));
    if (e != cudaSuccess) return e;
    const uint32_t tiles = (nn + kTile - 1) / kTile;
    // a fixed grid per mesh: the dot product's summation order is fixed
    const unsigned grid = std::min<unsigned>(tiles, 148u * per_sm);
    return launch_chained(k_spmv_nodes<T, S>, grid, kStreamThreads, smem, s, nn, L, nbr_ptr, nbr,
                          val, x, y, partials, counter, dot, skip, status);
}

}  // namespace

// As many CTAs per SM as each has stages: four of four where an SM's shared
// memory holds 16 stages (FP64 up to 11 neighbours, FP32 up to 21; 64^3 FP32 4 x
// 49.2 KB), else three of three (FP64 up to 20, 64^3 3 x 69.7 KB; FP32 up to the
// limit of 32), else two of two (FP64 up to 32, 2 x 78.1 KB).
template <typename T>
cudaError_t launch_spmv_nodes(uint32_t nn, uint32_t max_deg, const uint32_t* nbr_ptr,
                              const uint32_t* nbr, const T* val, const T* x, T* y, T* partials,
                              unsigned* counter, double* dot, unsigned* status, cudaStream_t s,
                              const unsigned* skip) {
    const StageLayout L = stage_layout<T>(max_deg);
    if (16 * (size_t)L.bytes <= kSmStages)
        return launch_stages<T, 4>(nn, L, 4, nbr_ptr, nbr, val, x, y, partials, counter, dot,
                                   status, s, skip);
    // (in FP32 the largest valence still fits three)
    if (sizeof(T) == 4 || 9 * (size_t)L.bytes <= kSmStages)
        return launch_stages<T, 3>(nn, L, 3, nbr_ptr, nbr, val, x, y, partials, counter, dot,
                                   status, s, skip);
    if constexpr (sizeof(T) == 8)
        return launch_stages<T, 2>(nn, L, 2, nbr_ptr, nbr, val, x, y, partials, counter, dot,
                                   status, s, skip);
    return cudaErrorInvalidValue;  // not reached
}
template cudaError_t launch_spmv_nodes<double>(uint32_t, uint32_t, const uint32_t*, const uint32_t*,
                                               const double*, const double*, double*, double*,
                                               unsigned*, double*, unsigned*, cudaStream_t,
                                               const unsigned*);
template cudaError_t launch_spmv_nodes<float>(uint32_t, uint32_t, const uint32_t*, const uint32_t*,
                                              const float*, const float*, float*, float*,
                                              unsigned*, double*, unsigned*, cudaStream_t,
                                              const unsigned*);

}  // namespace fm
