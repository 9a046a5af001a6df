// fm_kernels.cu — sm_100a kernels of the FlexMesh hot path.
//
// Assembly: an element pass evaluates every tet once (kinematics,
// Neo-Hookean stress, tangent scalars, FP64); in the node pass one warp owns
// one node and writes that node's three CSR rows exactly once (no atomics,
// deterministic), from the 3x3 blocks its lanes form, one tet each.  The
// diagonal block is minus the sum of the off-diagonal blocks (rows of every
// element tangent sum to zero because the shape gradients do).  Without a
// tangent the node pass is a gather of the vertex forces.
//
// Solvers: SpMV over the node-block pattern, and sync-free ILU(0) and
// triangular solves: a persistent grid walks the rows in a topological
// order (dependency levels); each row waits on its dependencies' release
// flags with a bounded spin, so there is no per-level launch or barrier.
#include <algorithm>
#include <cstdio>

#include "fm_kernels.hpp"
#include "fm_sync.cuh"

namespace fm {

// ===========================================================================
// Assembly
// ===========================================================================
// warps per CTA of the node pass: FP64 takes 96 registers, so that 20 warps
// are resident in five CTAs of four (at 80 for 24 it spills: 478 against 420
// us at 64^3), FP32 64 for 32 (four CTAs of eight; 40 warps at 48 registers
// spill: 352 against 311)
template <typename KT>
constexpr int kAsmWarps = sizeof(KT) == 4 ? 8 : 4;
template <typename KT>
constexpr int kAsmCtas = sizeof(KT) == 4 ? 4 : 5;

// The element pass leaves per tet the 12 components of its vertex forces
// vol M dN_a (fvert, FP64: 96 bytes) and, when a tangent is assembled, a
// record in the tangent's type: the shape gradients and the tangent scalars
// vol a, vol b, vol mu.  dN_0 = -dN_1 - dN_2 - dN_3, as tet_kinematics forms
// it, so the FP64 record leaves it out (96 bytes); the FP32 record keeps it
// (64 bytes): summing the rounded gradients would lose precision.
template <typename KT>
struct TanRec;
template <>
struct __align__(16) TanRec<double> {
    static constexpr int kFirst = 1;  // first stored gradient
    double d[9];
    double s[3];
};
template <>
struct __align__(16) TanRec<float> {
    static constexpr int kFirst = 0;
    float d[12];
    float s[3];
    float pad;
};
static_assert(sizeof(TanRec<double>) <= kTanRecBytes && sizeof(TanRec<double>) % 16 == 0, "");
static_assert(sizeof(TanRec<float>) <= kTanRecBytes && sizeof(TanRec<float>) % 16 == 0, "");

// The lanes' records (W 8-byte words each, in registers) to consecutive
// records of global memory, through the warp's stage so that every store
// instruction writes whole 512-byte runs: a lane's own 16-byte stores, one
// record apart from the next lane's, took 128 us of the 64^3 residual's
// element pass against 44 us.  The stage rows are padded to an odd number of
// words, so neither side has bank conflicts.
template <int W>
__device__ __forceinline__ void store_records(double* dst, uint32_t n_rec, const double (&r)[W],
                                              double* stage, int lane) {
    static_assert(W % 2 == 0, "records are whole 16-byte units");
#pragma unroll
    for (int i = 0; i < W; ++i) stage[lane * (W + 1) + i] = r[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < W / 2; ++i) {
        const int t = lane + 32 * i, rec = t / (W / 2), o = 2 * (t % (W / 2));
        if (rec < (int)n_rec) {
            const double* q = stage + rec * (W + 1) + o;
            reinterpret_cast<double2*>(dst)[t] = make_double2(q[0], q[1]);
        }
    }
    __syncwarp();
}

// 8-byte word i of a record held in registers
__device__ __forceinline__ double word_of(const double* r, int i) { return r[i]; }
__device__ __forceinline__ double word_of(const float* r, int i) {
    return __hiloint2double(__float_as_int(r[2 * i + 1]), __float_as_int(r[2 * i]));
}

// Element pass: one thread per tet.  WithK = false (residual only) leaves
// out the tangent records.
template <typename KT, bool WithK>
__global__ void __launch_bounds__(128, 4)
    k_asm_elements(MeshDev m, const double* __restrict__ u, double* __restrict__ fvert,
                   TanRec<KT>* __restrict__ tan, unsigned* __restrict__ status) {
    __shared__ double stage_s[4][32 * 13];
    chain_let_next();  // the node pass: its first lists load while this one ends
    const int lane = threadIdx.x & 31;
    double* stage = stage_s[threadIdx.x >> 5];
    const uint32_t e0 = blockIdx.x * 128u + (threadIdx.x & ~31u);  // the warp's first tet
    if (e0 >= m.n_elems) return;                                   // uniform per warp
    const uint32_t e = e0 + lane, n_rec = min(32u, m.n_elems - e0);
    unsigned flags = 0;
    double f[12];
    KT r[sizeof(TanRec<KT>) / sizeof(KT)];  // the tangent record
#pragma unroll
    for (int i = 0; i < 12; ++i) f[i] = 0.0;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(TanRec<KT>) / sizeof(KT)); ++i) r[i] = KT(0);
    uint4 c = make_uint4(0x80000000u, 0, 0, 0);
    if (e < m.n_elems) c = m.conn[e];
    if (!(c.x & 0x80000000u)) {
        const uint32_t cn[4] = {c.x, c.y, c.z, c.w};
        double x[12], ue[12];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                x[3 * a + d] = __ldg(m.xyz + 3 * (size_t)cn[a] + d);
                ue[3 * a + d] = __ldg(u + 3 * (size_t)cn[a] + d);
            }
        TetKin k;
        if (tet_kinematics(x, ue, k)) {
            double mu, lam;
            material_of(m.mat_mode, m.m0, m.m1, e, m.mu_s, m.lam_s, m.c_mu, m.c_lam, mu, lam);
            const Mandel M = mandel_stress(k.F, k.J, mu, lam);
            double fs = 0.0;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const double* dI = k.d[a];
                f[3 * a + 0] = k.vol * (M.m00 * dI[0] + M.m01 * dI[1] + M.m02 * dI[2]);
                f[3 * a + 1] = k.vol * (M.m01 * dI[0] + M.m11 * dI[1] + M.m12 * dI[2]);
                f[3 * a + 2] = k.vol * (M.m02 * dI[0] + M.m12 * dI[1] + M.m22 * dI[2]);
                fs += f[3 * a] + f[3 * a + 1] + f[3 * a + 2];
            }
            if (!(k.J > 0.0)) flags |= FM_FLAG_INVERTED;
            if (k.J < kJSafe) flags |= FM_FLAG_J_CLAMPED;
            if (!isfinite(fs)) flags |= FM_FLAG_NONFINITE;
            if (WithK) {
                double a, b;
                tangent_ab(mu, lam, k.J, M.lnJ, m.inv_cnu, a, b);
                constexpr int q0 = TanRec<KT>::kFirst;
#pragma unroll
                for (int q = q0; q < 4; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) r[3 * (q - q0) + d] = (KT)k.d[q][d];
                constexpr int s0 = 3 * (4 - q0);
                r[s0] = (KT)(k.vol * a);
                r[s0 + 1] = (KT)(k.vol * b);
                r[s0 + 2] = (KT)(k.vol * mu);
                if (!isfinite(a + b)) flags |= FM_FLAG_NONFINITE;
            }
        }
    }
    store_records<12>(fvert + 12 * (size_t)e0, n_rec, f, stage, lane);
    if (WithK) {
        constexpr int W = (int)(sizeof(TanRec<KT>) / 8);
        double w[W];
#pragma unroll
        for (int i = 0; i < W; ++i) w[i] = word_of(r, i);
        store_records<W>(reinterpret_cast<double*>(tan + e0), n_rec, w, stage, lane);
    }
    if (flags) raise_flag(status, flags);
}

// Sum of the vertex forces of each node's tets, ascending element order: one
// thread per DOF (36 us at 64^3, L2-bound; a warp per node that staged whole
// records took 217).  f (may be null) gets the sums, R (may be null) minus them,
// zero on constrained DOFs.
__global__ void __launch_bounds__(256)
    k_gather_forces(uint32_t n_nodes, const uint32_t* __restrict__ act_ptr,
                    const uint32_t* __restrict__ act_v, const double* fvert,
                    const uint8_t* __restrict__ mask, double* __restrict__ f,
                    double* __restrict__ R) {
    chain_wait();
    const uint32_t row = blockIdx.x * 256u + threadIdx.x;
    if (row >= 3 * n_nodes) return;
    const uint32_t n = row / 3, c = row - 3 * n;
    const uint32_t b = __ldg(act_ptr + n), e = __ldg(act_ptr + n + 1);
    double s = 0.0;
    uint32_t i = b;
    for (; i + 8 <= e; i += 8) {  // eight gathers in flight
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = ld_prev(fvert + 3 * (size_t)__ldg(act_v + i + q) + c);
#pragma unroll
        for (int q = 0; q < 8; ++q) s += v[q];
    }
    for (; i < e; ++i) s += ld_prev(fvert + 3 * (size_t)__ldg(act_v + i) + c);
    if (f) f[row] = s;
    if (R) R[row] = (mask && mask[row]) ? 0.0 : -s;
}

void launch_gather_forces(const MeshDev& m, double* f, double* R, cudaStream_t s) {
    launch_chained(k_gather_forces, (3 * m.n_nodes + 255) / 256, 256, 0, s, m.n_nodes, m.act_ptr,
                   m.act_v, m.fvert, m.mask, f, R);
}

// gradients of a tet's four vertices and its tangent scalars, from a staged
// record
__device__ __forceinline__ void load_tan(const uint4* q, double D[4][3], double s[3]) {
    double w[12];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double2 v = reinterpret_cast<const double2*>(q)[i];
        w[2 * i] = v.x;
        w[2 * i + 1] = v.y;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        D[1][c] = w[c];
        D[2][c] = w[3 + c];
        D[3][c] = w[6 + c];
        D[0][c] = -w[c] - w[3 + c] - w[6 + c];
        s[c] = w[9 + c];
    }
}
__device__ __forceinline__ void load_tan(const uint4* q, float D[4][3], float s[3]) {
    float w[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = reinterpret_cast<const float4*>(q)[i];
        w[4 * i] = v.x;
        w[4 * i + 1] = v.y;
        w[4 * i + 2] = v.z;
        w[4 * i + 3] = v.w;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int a = 0; a < 4; ++a) D[a][c] = w[3 * a + c];
        s[c] = w[12 + c];
    }
}

template <int Bytes>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(Bytes)
                 : "memory");
}

// A warp's shared memory in the node pass: the staged records (a 16-byte
// word more than a record apart: no bank conflicts) give way to the blocks,
// entry (j, p, q) of tet l at (9 (j - 1) + 3 p + q) PL + l, and those to the
// three rows.
template <typename KT, int PL>
struct __align__(16) AsmWarp {
    static constexpr int kWords = (int)(sizeof(TanRec<KT>) / 16);
    union {
        uint4 rec[(PL - 1) * (kWords + 1)];
        KT block[27 * PL];
        KT row[3 * 96];
    };
    double f[96];        // owner's forces: component c of tet l at 3 l + c
    uint16_t pair[96];   // the node's pair offsets
};

// Node pass: one warp owns node n and writes its three CSR rows once (no
// atomics, every sum in a fixed order).
//   1. The warp copies its active tets' records and the owner's forces to
//      shared memory, neighbouring lanes copying neighbouring words.
//   2. Lane l takes the l-th tet: turns its record so that the owner's
//      gradient comes first, forms the 3x3 blocks against the three other
//      vertices and leaves them in shared memory, entry by entry with
//      neighbouring tets in neighbouring words.
//   3. Lane c takes column c of the rows (c = 3k + q) and sums neighbour k's
//      blocks through the pair list, ascending element order, for the three
//      rows at once.
//   4. The diagonal block is minus the sum of the row's other blocks.
// The loop over nodes loads the next node's lists meanwhile.  Bound: the L1
// data pipe (89% busy in FP64: 360 shared-memory wavefronts per node).  Before
// the copies overlapped, a node's three dependent loads were most of its 7 us:
// 572 -> 478 us with the copies in flight together, 420 with the lists ahead
// and no spills (FP64 at 64^3).  One lane per neighbour walking its tets took
// 605.  Whole assembly: 128^3 FP64 5.67 -> 3.97 ms, 33^3 FP32 88 -> 62 us.
template <typename KT, int PL>
__global__ void __launch_bounds__(kAsmWarps<KT> * 32, kAsmCtas<KT>)
    k_assemble(MeshDev m, const TanRec<KT>* __restrict__ tan, KT* __restrict__ K,
               double* __restrict__ f, double* __restrict__ R, int apply_bc) {
    extern __shared__ __align__(16) unsigned char asm_smem[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    AsmWarp<KT, PL>& S = reinterpret_cast<AsmWarp<KT, PL>*>(asm_smem)[wi];
    const uint32_t step = gridDim.x * kAsmWarps<KT>;
    // the node's lists, loaded while the node before is worked on
    struct Node {
        uint32_t nb0, a0, v, nbr, edge;
        int deg, ma;
    } nx;
    auto pointers = [&](uint32_t n) {
        if (n >= m.n_nodes) return;
        nx.nb0 = __ldg(m.nbr_ptr + n);
        nx.deg = (int)(__ldg(m.nbr_ptr + n + 1) - nx.nb0);
        nx.a0 = __ldg(m.act_ptr + n);
        nx.ma = (int)(__ldg(m.act_ptr + n + 1) - nx.a0);
    };
    auto lists = [&](uint32_t n) {
        if (n >= m.n_nodes) return;
        nx.v = lane < nx.ma ? __ldg(m.act_v + nx.a0 + lane) : 0u;
        nx.nbr = lane < nx.deg ? __ldg(m.nbr + nx.nb0 + lane) : 0xffffffffu;
        nx.edge = lane < nx.deg ? __ldg(m.edge + nx.nb0 + lane) : 0u;
    };
    uint32_t n = blockIdx.x * kAsmWarps<KT> + wi;
    pointers(n);
    lists(n);
    chain_wait();  // so far only the mesh's own structure was read
    for (; n < m.n_nodes; n += step) {  // uniform per warp
        const uint32_t nb0 = nx.nb0, a0 = nx.a0, v = nx.v, my_nbr = nx.nbr, my_edge = nx.edge;
        const int deg = nx.deg, ma = nx.ma;
        const bool bc = apply_bc && m.mask;
        uint32_t fixed = 0;  // the neighbour's constrained DOFs, one bit each
        if (bc && lane < deg) {
            const uint8_t* q = m.mask + 3 * (size_t)my_nbr;
            fixed = (q[0] ? 1u : 0u) | (q[1] ? 2u : 0u) | (q[2] ? 4u : 0u);
        }
        // every copy in flight at once (cp.async: no registers, and no copy waits
        // for the one before)
        constexpr int W = AsmWarp<KT, PL>::kWords;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            if (32 * i >= W * ma) break;  // uniform
            const int t = lane + 32 * i, l = t / W, word = t - W * l;
            const uint32_t e = __shfl_sync(kFull, v, l & 31) >> 2;
            if (t < W * ma)
                copy_async<16>(&S.rec[l * (W + 1) + word],
                               reinterpret_cast<const uint4*>(tan + e) + word);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (32 * i >= 3 * ma) break;
            const int t = lane + 32 * i, l = t / 3;
            const uint32_t vl = __shfl_sync(kFull, v, l & 31);
            if (t < 3 * ma) copy_async<8>(&S.f[t], m.fvert + 3 * (size_t)vl + (t - 3 * l));
        }
        uint16_t pr[3] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (lane + 32 * i < 3 * ma) pr[i] = __ldg(m.pair_off + 3 * (size_t)a0 + lane + 32 * i);
#pragma unroll
        for (int i = 0; i < 3; ++i) S.pair[lane + 32 * i] = pr[i];
        pointers(n + step);
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        const int self_k = __ffs(__ballot_sync(kFull, my_nbr == n)) - 1;
        __syncwarp();
        KT D[4][3], sc[3];
        if (lane < ma) load_tan(S.rec + lane * (W + 1), D, sc);
        lists(n + step);
        __syncwarp();  // the records are in registers: their place is the blocks'
        if (lane < ma) {
            // rotate by the owner's local index: D[0] is its gradient
            const bool r1 = v & 1u, r2 = v & 2u;
            KT T[4][3], dI[3], hI[3], aI[3], bI[3], mI[3];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c) T[a][c] = r1 ? D[(a + 1) & 3][c] : D[a][c];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c) D[a][c] = r2 ? T[(a + 2) & 3][c] : T[a][c];
            // K_pq = va dI_p dJ_q (p==q) + vb dI_p dJ_q (p!=q)
            //      + vm (p==q ? sum_{r!=p} dI_r dJ_r : dI_q dJ_p) + (p==q) fI.dJ
            // with the products by dI formed once per tet
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                dI[c] = D[0][c];
                bI[c] = sc[1] * dI[c];
                mI[c] = sc[2] * dI[c];
                aI[c] = sc[0] * dI[c] - mI[c];
                hI[c] = (KT)S.f[3 * lane + c] + mI[c];
            }
#pragma unroll
            for (int j = 1; j < 4; ++j) {
                KT* o = S.block + (j - 1) * 9 * PL + lane;
                const KT* dJ = D[j];
                const KT h = hI[0] * dJ[0] + hI[1] * dJ[1] + hI[2] * dJ[2];
                o[0 * PL] = h + aI[0] * dJ[0];
                o[1 * PL] = bI[0] * dJ[1] + mI[1] * dJ[0];
                o[2 * PL] = bI[0] * dJ[2] + mI[2] * dJ[0];
                o[3 * PL] = bI[1] * dJ[0] + mI[0] * dJ[1];
                o[4 * PL] = h + aI[1] * dJ[1];
                o[5 * PL] = bI[1] * dJ[2] + mI[2] * dJ[1];
                o[6 * PL] = bI[2] * dJ[0] + mI[0] * dJ[2];
                o[7 * PL] = bI[2] * dJ[1] + mI[1] * dJ[2];
                o[8 * PL] = h + aI[2] * dJ[2];
            }
        }
        __syncwarp();
        if (lane < 3 && (f || R)) {
            double s = 0.0;
            for (int l = 0; l < ma; ++l) s += S.f[3 * l + lane];
            const uint32_t row = 3 * n + lane;
            if (f) f[row] = s;
            if (R) R[row] = (m.mask && m.mask[row]) ? 0.0 : -s;
        }
        const int rl = 3 * deg;
        KT acc[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            acc[r][0] = acc[r][1] = acc[r][2] = KT(0);
            if (32 * r < rl) {  // uniform
                const int c = lane + 32 * r, k = c / 3;
                const uint32_t ed = __shfl_sync(kFull, my_edge, k & 31);
                if (c < rl) {
                    const KT* base = S.block + (c - 3 * k) * PL;
                    const uint16_t* pr = S.pair + (ed & 0xffu);
                    for (uint32_t i = ed >> 8; i; --i, ++pr) {
                        const KT* q = base + *pr;
                        acc[r][0] += q[0];
                        acc[r][1] += q[3 * PL];
                        acc[r][2] += q[6 * PL];
                    }
                }
            }
        }
        __syncwarp();  // the blocks are read: their place is the rows'
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int c = lane + 32 * r;
            if (c < rl)
#pragma unroll
                for (int p = 0; p < 3; ++p) S.row[p * rl + c] = acc[r][p];
        }
        __syncwarp();
        // diagonal block: lane (third, p, q) sums entry (p, q) of every third
        // neighbour, then the thirds are added
        {
            const int third = lane / 9, pq = lane - 9 * third, p = pq / 3, q = pq - 3 * p;
            KT s = KT(0);
            if (lane < 27)
                for (int k = third; k < deg; k += 3) s += S.row[p * rl + 3 * k + q];
            const KT s1 = __shfl_sync(kFull, s, pq + 9), s2 = __shfl_sync(kFull, s, (pq + 18) & 31);
            if (lane < 9 && deg) S.row[p * rl + 3 * self_k + q] = -(s + s1 + s2);
        }
        __syncwarp();
        KT* out = K + 9 * (size_t)nb0;
        const uint32_t fixed_row = __shfl_sync(kFull, fixed, self_k & 31);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            if (32 * r < rl) {  // uniform
                const int c = lane + 32 * r, k = c / 3, q = c - 3 * k;
                const uint32_t fc = (__shfl_sync(kFull, fixed, k & 31) >> q) & 1u;
                if (c < rl)
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        KT val = k == self_k ? S.row[p * rl + c] : acc[r][p];
                        if (bc && (fc || ((fixed_row >> p) & 1u)))
                            val = (k == self_k && p == q) ? KT(1) : KT(0);
                        out[p * rl + c] = val;
                    }
            }
        }
        __syncwarp();  // the next node's copies overwrite the rows
    }
}

template <typename KT, int PL>
static void launch_node_pass(const MeshDev& m, KT* K, double* f, double* R, int apply_bc,
                             cudaStream_t s) {
    const unsigned grid = std::min<unsigned>((m.n_nodes + kAsmWarps<KT> - 1) / kAsmWarps<KT>,
                                             148u * kAsmCtas<KT>);
    constexpr size_t smem = kAsmWarps<KT> * sizeof(AsmWarp<KT, PL>);
    static_assert(smem <= 48 * 1024, "what a kernel may use without raising its limit");
    launch_chained(k_assemble<KT, PL>, grid, kAsmWarps<KT> * 32, smem, s, m,
                   static_cast<const TanRec<KT>*>(m.tan_rec), K, f, R, apply_bc);
}

template <typename KT>
static void launch_assemble_t(const MeshDev& m, const double* u, KT* K, double* f, double* R,
                              int apply_bc, unsigned* status, cudaStream_t s) {
    if (m.n_nodes == 0) return;
    const unsigned ge = (m.n_elems + 127) / 128;
    TanRec<KT>* tan = static_cast<TanRec<KT>*>(m.tan_rec);
    if (!K) {
        if (ge) k_asm_elements<KT, false><<<ge, 128, 0, s>>>(m, u, m.fvert, tan, status);
        launch_gather_forces(m, f, R, s);
        return;
    }
    if (ge) k_asm_elements<KT, true><<<ge, 128, 0, s>>>(m, u, m.fvert, tan, status);
    if (m.pair_lane == 21) launch_node_pass<KT, 21>(m, K, f, R, apply_bc, s);
    else launch_node_pass<KT, 33>(m, K, f, R, apply_bc, s);
}
void launch_assemble(const MeshDev& m, const double* u, double* K, double* f, double* R,
                     int apply_bc, unsigned* status, cudaStream_t s) {
    launch_assemble_t<double>(m, u, K, f, R, apply_bc, status, s);
}
void launch_assemble(const MeshDev& m, const double* u, float* K, double* f, double* R,
                     int apply_bc, unsigned* status, cudaStream_t s) {
    launch_assemble_t<float>(m, u, K, f, R, apply_bc, status, s);
}

// Full element tangent/force of one tet into Ke (row-major 12x12), fe.
// Returns false for a degenerate tet (outputs zero).
__device__ __forceinline__ bool element_full(const double x[12], const double ue[12], double mu,
                                             double lam, double inv_cnu, double* Ke, double* fe,
                                             size_t ks, unsigned& flags) {
    TetKin k;
    if (!tet_kinematics(x, ue, k)) {
        for (int q = 0; q < 144; ++q) Ke[q * ks] = 0.0;
        for (int q = 0; q < 12; ++q) fe[q] = 0.0;
        return false;
    }
    const Mandel M = mandel_stress(k.F, k.J, mu, lam);
    double a, b;
    tangent_ab(mu, lam, k.J, M.lnJ, inv_cnu, a, b);
    const double va = k.vol * a, vb = k.vol * b, vm = k.vol * mu;
    double fI[4][3];
    for (int i = 0; i < 4; ++i) {
        const double* d = k.d[i];
        fI[i][0] = k.vol * (M.m00 * d[0] + M.m01 * d[1] + M.m02 * d[2]);
        fI[i][1] = k.vol * (M.m01 * d[0] + M.m11 * d[1] + M.m12 * d[2]);
        fI[i][2] = k.vol * (M.m02 * d[0] + M.m12 * d[1] + M.m22 * d[2]);
        for (int p = 0; p < 3; ++p) fe[3 * i + p] = fI[i][p];
    }
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) {
            double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            tangent_block_acc<double>(k.d[i], k.d[j], fI[i], va, vb, vm, acc);
            for (int p = 0; p < 3; ++p)
                for (int q = 0; q < 3; ++q) Ke[((i * 3 + p) * 12 + j * 3 + q) * ks] = acc[3 * p + q];
        }
    if (!(k.J > 0.0)) flags |= FM_FLAG_INVERTED;
    if (k.J < kJSafe) flags |= FM_FLAG_J_CLAMPED;
    if (!isfinite(fe[0] + fe[4] + fe[8] + a + b)) flags |= FM_FLAG_NONFINITE;
    return true;
}

// Batched elements: one thread per tet, one warp per 32 consecutive tets.
// A tet's 12x12 tangent is formed three rows (36 doubles, 288 bytes) at a
// time and leaves through the warp's stage, neighbouring lanes storing
// neighbouring words (a lane's own stores, 1,152 bytes from the next lane's,
// wrote a quarter of a sector each: 457 us for a call with 200,003 tets, now
// 85, 44 of them the bytes at copy bandwidth).  Stage rows of 37 doubles have no
// bank conflicts on the way in.
constexpr int kElemWarps = 4;

__global__ void __launch_bounds__(kElemWarps * 32)
    k_elements(uint32_t n, const double* __restrict__ x, const double* __restrict__ u,
               const double* __restrict__ E, double nu, double* __restrict__ K,
               double* __restrict__ f, unsigned* status) {
    __shared__ double stage_s[kElemWarps][32 * 37];
    const int lane = threadIdx.x & 31;
    double* stage = stage_s[threadIdx.x >> 5];
    const uint32_t e0 = blockIdx.x * (kElemWarps * 32u) + (threadIdx.x & ~31u);
    if (e0 >= n) return;  // uniform per warp
    const uint32_t n_rec = min(32u, n - e0);
    const uint32_t e = e0 + min((uint32_t)lane, n_rec - 1);  // spare lanes repeat the last tet
    double xe[12], ue[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) {
        xe[q] = x[12 * (size_t)e + q];
        ue[q] = u[12 * (size_t)e + q];
    }
    const double Ee = E[e];
    const double mu = Ee / (2.0 * (1.0 + nu));
    const double lam = Ee * nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    const double one_m = 1.0 - 2.0 * nu;
    const double inv_cnu = 1.0 / (one_m < 0.1 ? 0.1 : one_m);
    unsigned flags = 0;
    TetKin k;
    double fI[12], a = 0.0, b = 0.0;
#pragma unroll
    for (int q = 0; q < 12; ++q) fI[q] = 0.0;
    const bool ok = tet_kinematics(xe, ue, k);  // false: degenerate, outputs zero
    if (ok) {
        const Mandel M = mandel_stress(k.F, k.J, mu, lam);
        tangent_ab(mu, lam, k.J, M.lnJ, inv_cnu, a, b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double* d = k.d[i];
            fI[3 * i + 0] = k.vol * (M.m00 * d[0] + M.m01 * d[1] + M.m02 * d[2]);
            fI[3 * i + 1] = k.vol * (M.m01 * d[0] + M.m11 * d[1] + M.m12 * d[2]);
            fI[3 * i + 2] = k.vol * (M.m02 * d[0] + M.m12 * d[1] + M.m22 * d[2]);
        }
        if (!(k.J > 0.0)) flags |= FM_FLAG_INVERTED;
        if (k.J < kJSafe) flags |= FM_FLAG_J_CLAMPED;
        if (!isfinite(fI[0] + fI[4] + fI[8] + a + b)) flags |= FM_FLAG_NONFINITE;
    }
    const double va = ok ? k.vol * a : 0.0, vb = ok ? k.vol * b : 0.0, vm = ok ? k.vol * mu : 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            if (ok) tangent_block_acc<double>(k.d[i], k.d[j], fI + 3 * i, va, vb, vm, acc);
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int q = 0; q < 3; ++q) stage[lane * 37 + p * 12 + 3 * j + q] = acc[3 * p + q];
        }
        __syncwarp();
        double* o = K + 144 * (size_t)e0 + 36 * i;
#pragma unroll 6
        for (int t = lane; t < 36 * (int)n_rec; t += 32) {
            const int rec = t / 36, w = t - 36 * rec;
            o[144 * (size_t)rec + w] = stage[rec * 37 + w];
        }
        __syncwarp();
    }
#pragma unroll
    for (int q = 0; q < 12; ++q) stage[lane * 13 + q] = fI[q];
    __syncwarp();
#pragma unroll 4
    for (int t = lane; t < 12 * (int)n_rec; t += 32) {
        const int rec = t / 12;
        f[12 * (size_t)e0 + t] = stage[rec * 13 + (t - 12 * rec)];
    }
    if (flags) raise_flag(status, flags);
}

void launch_elements(uint32_t n, const double* x, const double* u, const double* E, double nu,
                     double* K, double* f, unsigned* status, cudaStream_t s) {
    if (!n) return;
    k_elements<<<(n + kElemWarps * 32 - 1) / (kElemWarps * 32), kElemWarps * 32, 0, s>>>(
        n, x, u, E, nu, K, f, status);
}

// Reference-pattern scatter: thread per tet, slot map with -1 for entries
// the reference's defective pattern lacks (last duplicate wins in the map).
__global__ void k_assemble_slotmap(MeshDev m, const double* __restrict__ u,
                                   const int32_t* __restrict__ slot, double* K, double* f,
                                   double* Ke_scratch, unsigned* status) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m.n_elems) return;
    uint4 c = m.conn[e];
    if (c.x & 0x80000000u) return;
    const uint32_t cn[4] = {c.x, c.y, c.z, c.w};
    double x[12], ue[12];
    for (int a = 0; a < 4; ++a)
        for (int d = 0; d < 3; ++d) {
            x[3 * a + d] = m.xyz[3 * (size_t)cn[a] + d];
            ue[3 * a + d] = u[3 * (size_t)cn[a] + d];
        }
    double mu, lam;
    material_of(m.mat_mode, m.m0, m.m1, e, m.mu_s, m.lam_s, m.c_mu, m.c_lam, mu, lam);
    double fe[12];
    unsigned flags = 0;
    double* Ke = Ke_scratch + (size_t)e;  // strided by n_elems
    if (!element_full(x, ue, mu, lam, m.inv_cnu, Ke, fe, m.n_elems, flags)) return;
    if (flags) raise_flag(status, flags);
    for (int q = 0; q < 144; ++q) {
        const int32_t sl = slot[144 * (size_t)e + q];
        if (sl >= 0) atomicAdd(K + sl, Ke[(size_t)q * m.n_elems]);
    }
    for (int a = 0; a < 4; ++a)
        for (int d = 0; d < 3; ++d) atomicAdd(f + 3 * (size_t)cn[a] + d, fe[3 * a + d]);
}

void launch_assemble_slotmap(const MeshDev& m, const double* u, const int32_t* slot, double* K,
                             double* f, double* Ke_scratch, unsigned* status, cudaStream_t s) {
    if (!m.n_elems) return;
    k_assemble_slotmap<<<(m.n_elems + 127) / 128, 128, 0, s>>>(m, u, slot, K, f, Ke_scratch,
                                                               status);
}

// ===========================================================================
// SpMV
// ===========================================================================
constexpr int kSpmvBlocks = 148 * 8;

// G lanes per row (spmv_csr_lanes: a warp per five-entry row leaves 27 of its
// lanes idle)
template <typename T, int G>
__global__ void __launch_bounds__(256)
    k_spmv_csr(uint32_t n, const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
               const T* __restrict__ val, const T* x, T* __restrict__ y, T* partials,
               unsigned* counter, double* dot, const unsigned* skip) {
    chain_begin();
    if (skipped(skip)) return;
    const int lane = threadIdx.x & (G - 1);
    const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const uint32_t ngroups = gridDim.x * blockDim.x / G;
    T dsum = T(0);
    // whole warps step together: the group sum shuffles over the full warp
    const uint32_t steps = (n + ngroups - 1) / ngroups;
    for (uint32_t q = 0; q < steps; ++q) {
        const uint32_t i = group + q * ngroups;
        T s = T(0), xi = T(0);
        if (i < n) {
            if (dot && lane == 0) xi = ld_prev(x + i);
            for (uint32_t k = rp[i] + lane; k < rp[i + 1]; k += G)
                s += __ldg(val + k) * ld_prev(x + ci[k]);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
        if (i < n && lane == 0) {
            y[i] = s;
            dsum += s * xi;
        }
    }
    if (dot) {
        __shared__ T sbuf[32];
        const T bt = block_sum(dsum, sbuf);
        grid_reduce_finish<T>(bt, partials, counter, [&](T total) { *dot = (double)total; });
    }
}

// Lanes per row from the mean length, and more where a long row is what the
// product waits for: G lanes take about 0.156 us per G entries of the longest
// row, and each lane more costs a row 4 ps.  us with 4 / 8 / 32 lanes: a
// 22,500-row five-point matrix 10.5 / 11.1 / 14.2, an arrowhead matrix with a
// row of 500 entries 28.5 / 19.9 / 13.8, 40 of them (20,000 rows) 32.6 / 23.8 /
// 19.7, 400 of them 38.3 / 30.5 / 40.3, 2,000 of 200 26.2 / 27.6 / 61.
static uint32_t spmv_csr_lanes(uint32_t n, uint64_t nnz, uint32_t max_row) {
    const uint64_t mean = n ? nnz / n : 0;
    uint32_t lanes = mean <= 6 ? 4 : mean <= 16 ? 8 : 32;
    if (max_row <= 4 * lanes) return lanes;
    auto cost = [&](uint32_t g) { return (uint64_t)n * g + 39000ull * max_row / g; };
    for (uint32_t g : {8u, 32u})
        if (g > lanes && cost(g) < cost(lanes)) lanes = g;
    return lanes;
}

template <typename T, int G>
static cudaError_t launch_spmv_csr_g(uint32_t n, const uint32_t* rp, const uint32_t* ci,
                                     const T* val, const T* x, T* y, T* partials,
                                     unsigned* counter, double* dot, cudaStream_t s,
                                     const unsigned* skip) {
    const uint32_t per = 256 / G;  // rows per block and step
    const int grid = (int)std::min<uint32_t>(kSpmvBlocks, std::max(1u, (n + per - 1) / per));
    return launch_chained(k_spmv_csr<T, G>, grid, 256, 0, s, n, rp, ci, val, x, y, partials,
                          counter, dot, skip);
}

template <typename T>
cudaError_t launch_spmv_csr(uint32_t n, uint64_t nnz, uint32_t max_row, const uint32_t* rp,
                            const uint32_t* ci, const T* val, const T* x, T* y, T* partials,
                            unsigned* counter, double* dot, cudaStream_t s,
                            const unsigned* skip) {
    switch (spmv_csr_lanes(n, nnz, max_row)) {
        case 4:
            return launch_spmv_csr_g<T, 4>(n, rp, ci, val, x, y, partials, counter, dot, s, skip);
        case 8:
            return launch_spmv_csr_g<T, 8>(n, rp, ci, val, x, y, partials, counter, dot, s, skip);
        default:
            return launch_spmv_csr_g<T, 32>(n, rp, ci, val, x, y, partials, counter, dot, s, skip);
    }
}

// ===========================================================================
// Sync-free ILU(0) and triangular solves (scalar CSR rows, warp per row)
// ===========================================================================
__device__ __forceinline__ int find_sorted(const uint32_t* a, int len, uint32_t key) {
    int lo = 0, hi = len - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const uint32_t v = a[mid];
        if (v == key) return mid;
        if (v < key) lo = mid + 1;
        else hi = mid - 1;
    }
    return -1;
}

constexpr int kSfWarps = 8;  // warps per block of the persistent kernels

// Row i of ILU(0), IKJ form in natural order, which performs the same
// subtractions in the same order as the reference's Doolittle loop
// (FEM/adaptive_fem_engine.hpp:327-466):
//   for each lower column c of row i, ascending:  l = w_c / d_c,
//     w_j -= l U(c,j) for every j > c of row c present in row i,
//     and u_ii -= l U(c,i);
//   u_ii perturbed by +-1e-8 when |u_ii| < 1e-12.
// The diagonal slot keeps a_ii (the reference's U_val does); pivots go to diag.
template <typename T>
__global__ void __launch_bounds__(kSfWarps * 32)
    k_ilu0_csr(CsrDev A, const T* __restrict__ a,
               T* __restrict__ lu, T* __restrict__ diag, unsigned* __restrict__ done,
               unsigned epoch, unsigned* __restrict__ status) {
    extern __shared__ unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const uint32_t stride = (A.max_row + 1) & ~1u;
    uint32_t* cols = reinterpret_cast<uint32_t*>(smem_raw) + wi * stride;
    T* w = reinterpret_cast<T*>(reinterpret_cast<uint32_t*>(smem_raw) + kSfWarps * stride) +
           wi * stride;
    __shared__ T s_uii[kSfWarps];
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t W = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = gw; t < A.n; t += W) {
        const uint32_t i = A.fwd_order[t];
        const uint32_t b = A.rp[i];
        const int len = (int)(A.rp[i + 1] - b);
        const int dp = (int)(A.dpos[i] - b);
        for (int q = lane; q < len; q += 32) {
            cols[q] = A.ci[b + q];
            w[q] = a[b + q];
        }
        __syncwarp();
        const bool has_diag = dp < len && cols[dp] == i;
        bool ok = true;
        for (int q = lane; q < dp; q += 32) ok &= wait_flag(done + cols[q], epoch, status);
        ok = __all_sync(kFull, ok);
        if (lane == 0) s_uii[wi] = has_diag ? w[dp] : T(0);
        __syncwarp();
        if (ok) {
            for (int q = 0; q < dp; ++q) {
                const uint32_t c = cols[q];
                const T l = w[q] / ld_cg(diag + c);
                const uint32_t ue = A.rp[c + 1];
                for (uint32_t mm = A.upos[c] + lane; mm < ue; mm += 32) {
                    const uint32_t j = A.ci[mm];
                    const T uv = ld_cg(lu + mm);
                    if (j == i) {
                        s_uii[wi] -= l * uv;
                    } else {
                        const int p = find_sorted(cols + q + 1, len - q - 1, j);
                        if (p >= 0) w[q + 1 + p] -= l * uv;
                    }
                }
                __syncwarp();
                if (lane == 0) w[q] = l;
                __syncwarp();
            }
        }
        T uii = s_uii[wi];
        for (int q = lane; q < len; q += 32) lu[b + q] = w[q];
        if (lane == 0) {
            if (fabs((double)uii) < kPivotThreshold) {
                uii += (uii >= T(0) ? T(kPivotPerturb) : T(-kPivotPerturb));
                raise_flag(status, FM_FLAG_PIVOT);
            }
            if (!isfinite((double)uii)) raise_flag(status, FM_FLAG_NONFINITE);
            diag[i] = uii;
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) st_release(done + i, epoch);
        __syncwarp();
    }
}

// z_i = r_i - sum_{c<i} L_ic z_c  (unit lower)
template <typename T>
__global__ void __launch_bounds__(kSfWarps * 32)
    k_trsv_lower_csr(CsrDev A, const T* __restrict__ lu, const T* __restrict__ r, T* z,
                     unsigned* __restrict__ done, unsigned epoch, unsigned* __restrict__ status,
                     const unsigned* __restrict__ skip) {
    if (skipped(skip)) return;
    const int lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t W = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = gw; t < A.n; t += W) {
        const uint32_t i = A.fwd_order[t];
        const uint32_t e = A.dpos[i];
        T s = T(0);
        for (uint32_t k = A.rp[i] + lane; k < e; k += 32) {
            const uint32_t c = A.ci[k];
            if (!wait_flag(done + c, epoch, status)) break;
            s += lu[k] * ld_cg(z + c);
        }
        s = warp_sum(s);
        if (lane == 0) {
            z[i] = r[i] - s;
            st_release(done + i, epoch);
        }
    }
}

// y_i = (z_i - sum_{c>i} U_ic y_c) / d_i
template <typename T>
__global__ void __launch_bounds__(kSfWarps * 32)
    k_trsv_upper_csr(CsrDev A, const T* __restrict__ lu,
                     const T* __restrict__ diag, const T* __restrict__ z, T* y,
                     unsigned* __restrict__ done, unsigned epoch, unsigned* __restrict__ status,
                     const unsigned* __restrict__ skip) {
    if (skipped(skip)) return;
    const int lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t W = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = gw; t < A.n; t += W) {
        const uint32_t i = A.bwd_order[t];
        const uint32_t e = A.rp[i + 1];
        T s = T(0);
        for (uint32_t k = A.upos[i] + lane; k < e; k += 32) {
            const uint32_t c = A.ci[k];
            if (!wait_flag(done + c, epoch, status)) break;
            s += lu[k] * ld_cg(y + c);
        }
        s = warp_sum(s);
        if (lane == 0) {
            y[i] = (z[i] - s) / diag[i];
            st_release(done + i, epoch);
        }
    }
}


static size_t ilu_smem_bytes(const CsrDev& A, size_t tsize) {
    const size_t stride = (A.max_row + 1) & ~1u;
    return kSfWarps * stride * (sizeof(uint32_t) + tsize);
}

template <typename T>
void launch_ilu0_csr(const CsrDev& A, const T* a_val, T* lu, T* diag, unsigned* done,
                     unsigned epoch, unsigned* status, int grid, cudaStream_t s) {
    if (!A.n) return;
    k_ilu0_csr<T><<<grid, kSfWarps * 32, ilu_smem_bytes(A, sizeof(T)), s>>>(A, a_val, lu, diag,
                                                                             done, epoch, status);
}
template <typename T>
cudaError_t launch_trsv_lower_csr(const CsrDev& A, const T* lu, const T* r, T* z, unsigned* done,
                                  unsigned epoch, unsigned* status, int grid, cudaStream_t s,
                                  const unsigned* skip) {
    if (!A.n) return cudaSuccess;
    return launch_plain(k_trsv_lower_csr<T>, grid, kSfWarps * 32, 0, s, A, lu, r, z, done, epoch,
                        status, skip);
}
template <typename T>
cudaError_t launch_trsv_upper_csr(const CsrDev& A, const T* lu, const T* diag, const T* z, T* y,
                                  unsigned* done, unsigned epoch, unsigned* status, int grid,
                                  cudaStream_t s, const unsigned* skip) {
    if (!A.n) return cudaSuccess;
    return launch_plain(k_trsv_upper_csr<T>, grid, kSfWarps * 32, 0, s, A, lu, diag, z, y, done,
                        epoch, status, skip);
}

// All blocks of a sync-free kernel must be resident at once (rows wait on
// rows handled by other blocks), so the grid is the occupancy limit times
// the SM count.
template <typename K>
static int resident_grid(K kernel, int device, size_t smem) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSfWarps * 32, smem);
    if (per_sm < 1) per_sm = 1;
    return sms * per_sm;
}
int persistent_grid_ilu0_csr(int device, bool fp32, const CsrDev& A) {
    return fp32 ? resident_grid(k_ilu0_csr<float>, device, ilu_smem_bytes(A, 4))
                : resident_grid(k_ilu0_csr<double>, device, ilu_smem_bytes(A, 8));
}
int persistent_grid_trsv_csr(int device, bool fp32) {
    const int a = fp32 ? resident_grid(k_trsv_lower_csr<float>, device, 0)
                       : resident_grid(k_trsv_lower_csr<double>, device, 0);
    const int b = fp32 ? resident_grid(k_trsv_upper_csr<float>, device, 0)
                       : resident_grid(k_trsv_upper_csr<double>, device, 0);
    return a < b ? a : b;
}

// ===========================================================================
// Vector kernels (PCG and Newton)
// ===========================================================================
constexpr int kVecThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kVecThreads)
    k_dot(uint32_t n, const T* __restrict__ x, const T* __restrict__ y, T* partials,
          unsigned* counter, double* out) {
    T s = T(0);
#pragma unroll 4
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        s += x[i] * y[i];
    __shared__ T sbuf[32];
    const T bt = block_sum(s, sbuf);
    grid_reduce_finish<T>(bt, partials, counter, [&](T total) { *out = (double)total; });
}
template <typename T>
void launch_dot(uint32_t n, const T* x, const T* y, T* partials, unsigned* counter, double* out,
                cudaStream_t s) {
    k_dot<T><<<red_blocks(n), kVecThreads, 0, s>>>(n, x, y, partials, counter, out);
}

// PCG entry: r = b - r (zero_x: r = b, the start vector is zero), rr = r.r,
// the early exit ||r|| < tol 1e-3 as the reference takes it (:1298), and the
// wait sentinel into tmp (null: none) for the solve that follows.
// The grid's elements four at a time: load(q, i) for each of them, then use(q,
// i), in ascending order.  A store may alias a later load as far as the
// compiler can tell, so loads written behind stores wait for them.
template <typename Load, typename Use>
__device__ __forceinline__ void by_four(uint32_t n, Load load, Use use) {
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * step) {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
            if (i0 + q * step < n) load(q, i0 + q * step);
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
            if (i0 + q * step < n) use(q, i0 + q * step);
    }
}

template <typename T>
__global__ void __launch_bounds__(kVecThreads)
    k_pcg_init(uint32_t n, const T* b, T* __restrict__ r, int zero_x, T* __restrict__ tmp,
               double tol, T* partials, unsigned* counter, DevScalars* sc, PcgReport* rep,
               unsigned seq) {
    chain_begin();
    T s = T(0), v[4];
    by_four(
        n,
        [&](uint32_t q, uint32_t i) {
            v[q] = ld_prev(b + i);
            if (!zero_x) v[q] -= r[i];
        },
        [&](uint32_t q, uint32_t i) {
            r[i] = v[q];
            if (tmp) tmp[i] = Sentinel<T>::value();
            s += v[q] * v[q];
        });
    __shared__ T sbuf[32];
    const T bt = block_sum(s, sbuf);
    grid_reduce_finish<T>(bt, partials, counter, [&](T total) {
        sc->rr = (double)total;
        sc->stop = 0u;
        sc->done = sqrt((double)total) < tol * 1e-3 ? 1u : 0u;
        pcg_report(rep, seq, sc);
    });
}
template <typename T>
cudaError_t launch_pcg_init(uint32_t n, const T* b, T* r, bool zero_x, T* tmp, double tol,
                            T* partials, unsigned* counter, DevScalars* sc, PcgReport* rep,
                            unsigned seq, cudaStream_t s) {
    return launch_chained(k_pcg_init<T>, red_blocks(n), kVecThreads, 0, s, n, b, r, zero_x, tmp,
                          tol, partials, counter, sc, rep, seq);
}

// p = z; rz = r.z; bb = b.b.  Two sums share one pass (partials: 2 slots per block)
template <typename T>
__global__ void __launch_bounds__(kVecThreads)
    k_pcg_start(uint32_t n, const T* r, const T* z, const T* b, T* __restrict__ p, T* partials,
                unsigned* counter, DevScalars* sc) {
    chain_begin();
    if (skipped(&sc->done)) return;
    T s1 = T(0), s2 = T(0), zv[4], rv[4], bv[4];
    by_four(
        n,
        [&](uint32_t q, uint32_t i) {
            zv[q] = ld_prev(z + i);
            rv[q] = ld_prev(r + i);
            bv[q] = ld_prev(b + i);
        },
        [&](uint32_t q, uint32_t i) {
            p[i] = zv[q];
            s1 += rv[q] * zv[q];
            s2 += bv[q] * bv[q];
        });
    __shared__ T sbuf[32];
    const T b1 = block_sum(s1, sbuf);
    const T b2 = block_sum(s2, sbuf);
    grid_reduce_finish<T>(b1, partials, counter, [&](T total) {
        sc->rz_new = (double)total;
        sc->rz = (double)total;
    });
    grid_reduce_finish<T>(b2, partials + gridDim.x, counter + 1,
                          [&](T total) { sc->bb = (double)total; });
}
template <typename T>
cudaError_t launch_pcg_start(uint32_t n, const T* r, const T* z, const T* b, T* p, T* partials,
                             unsigned* counter, DevScalars* sc, cudaStream_t s) {
    return launch_chained(k_pcg_start<T>, red_blocks(n), kVecThreads, 0, s, n, r, z, b, p,
                          partials, counter, sc);
}

// alpha = rz/pAp (current rz is rz_new); breakdown |pAp| < 1e-60 stops
// before touching x and r, as the reference breaks out (:1320).  Also writes
// the wait sentinel into tmp (null: none), the intermediate of the
// triangular solves that follow.
template <typename T>
__global__ void __launch_bounds__(kVecThreads)
    k_pcg_update_xr(uint32_t n, const T* p, const T* Ap, T* __restrict__ x, T* __restrict__ r,
                    T* __restrict__ tmp, DevScalars* sc) {
    chain_begin();
    if (skipped(&sc->done)) return;
    const double pAp = sc->pAp;
    if (fabs(pAp) < 1e-60) {
        if (blockIdx.x == 0 && threadIdx.x == 0) sc->stop = 1u;
        return;
    }
    const T alpha = (T)(sc->rz_new / pAp);
    T pv[4], av[4], xv[4], rv[4];
    by_four(
        n,
        [&](uint32_t q, uint32_t i) {
            pv[q] = ld_prev(p + i);
            av[q] = ld_prev(Ap + i);
            xv[q] = x[i];
            rv[q] = r[i];
        },
        [&](uint32_t q, uint32_t i) {
            x[i] = xv[q] + alpha * pv[q];
            r[i] = rv[q] - alpha * av[q];
            if (tmp) tmp[i] = Sentinel<T>::value();
        });
}
template <typename T>
cudaError_t launch_pcg_update_xr(uint32_t n, const T* p, const T* Ap, T* x, T* r, T* tmp,
                                 DevScalars* sc, cudaStream_t s) {
    return launch_chained(k_pcg_update_xr<T>, 2 * red_blocks(n), kVecThreads, 0, s, n, p, Ap, x, r,
                          tmp, sc);
}

// rz <- rz_new (old value kept for beta), rz_new <- r.z, relres, the stop
// tests, and the report.  After a breakdown only the report.
template <typename T>
__global__ void __launch_bounds__(kVecThreads)
    k_pcg_rz(uint32_t n, const T* r, const T* z, double tol, T* partials, unsigned* counter,
             DevScalars* sc, PcgReport* rep, unsigned seq) {
    chain_begin();
    if (skipped(&sc->done)) return;
    if (ld_volatile_u32(&sc->stop)) {
        // the other blocks return here or, once done is set, above
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            sc->done = 1u;
            pcg_report(rep, seq, sc);
        }
        return;
    }
    T s = T(0);
#pragma unroll 4
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        s += ld_prev(r + i) * ld_prev(z + i);
    __shared__ T sbuf[32];
    const T bt = block_sum(s, sbuf);
    grid_reduce_finish<T>(bt, partials, counter, [&](T total) {
        sc->rz = sc->rz_new;
        sc->rz_new = (double)total;
        const double bb = sc->bb > 1e-300 ? sc->bb : 1e-300;
        sc->relres = sqrt((double)total / bb);
        if (sc->relres < tol) sc->done = 1u;
        pcg_report(rep, seq, sc);
    });
}
template <typename T>
cudaError_t launch_pcg_rz(uint32_t n, const T* r, const T* z, double tol, T* partials,
                          unsigned* counter, DevScalars* sc, PcgReport* rep, unsigned seq,
                          cudaStream_t s) {
    return launch_chained(k_pcg_rz<T>, red_blocks(n), kVecThreads, 0, s, n, r, z, tol, partials,
                          counter, sc, rep, seq);
}

template <typename T>
__global__ void __launch_bounds__(kVecThreads)
    k_pcg_update_p(uint32_t n, const T* z, T* __restrict__ p, const DevScalars* sc) {
    chain_begin();
    if (skipped(&sc->done)) return;
    const T beta = (T)(sc->rz_new / sc->rz);
    T zv[4], pv[4];
    by_four(
        n,
        [&](uint32_t q, uint32_t i) {
            zv[q] = ld_prev(z + i);
            pv[q] = p[i];
        },
        [&](uint32_t q, uint32_t i) { p[i] = zv[q] + beta * pv[q]; });
}
template <typename T>
cudaError_t launch_pcg_update_p(uint32_t n, const T* z, T* p, DevScalars* sc, cudaStream_t s) {
    return launch_chained(k_pcg_update_p<T>, 2 * red_blocks(n), kVecThreads, 0, s, n, z, p, sc);
}

__global__ void k_set_bc_values(uint32_t n, const uint8_t* __restrict__ mask,
                                const double* __restrict__ val, double frac, double* u) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        if (mask[i]) u[i] = val ? frac * val[i] : 0.0;
}
void launch_set_bc_values(uint32_t n, const uint8_t* mask, const double* val, double frac,
                          double* u, cudaStream_t s) {
    k_set_bc_values<<<kRedBlocks, kVecThreads, 0, s>>>(n, mask, val, frac, u);
}

void launch_norm2(uint32_t n, const double* R, double* partials, unsigned* counter, double* out,
                  cudaStream_t s) {
    k_dot<double><<<red_blocks(n), kVecThreads, 0, s>>>(n, R, R, partials, counter, out);
}

__global__ void k_to_f32_scaled(uint32_t n, const double* __restrict__ R, double inv_scale,
                                float* __restrict__ b32, float* __restrict__ x32) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        b32[i] = (float)(R[i] * inv_scale);
        if (x32) x32[i] = 0.0f;
    }
}

template <typename T>
__global__ void k_scale(uint32_t n, T* __restrict__ x, T g) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        x[i] *= g;
}
void launch_scale_f32(uint32_t n, float* x, float g, cudaStream_t s) {
    k_scale<float><<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, x, g);
}
void launch_to_f32_scaled(uint32_t n, const double* R, double inv_scale, float* b32, float* x32,
                          cudaStream_t s) {
    k_to_f32_scaled<<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, R, inv_scale, b32, x32);
}

__global__ void k_axpy_u(uint32_t n, const double* __restrict__ du, double* __restrict__ u) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        u[i] += du[i];
}
void launch_axpy_u(uint32_t n, const double* du, double* u, cudaStream_t s) {
    k_axpy_u<<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, du, u);
}
__global__ void k_axpy_u_f32(uint32_t n, const float* __restrict__ du, double scale,
                             double* __restrict__ u) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        u[i] += scale * (double)du[i];
}
void launch_axpy_u_f32(uint32_t n, const float* du, double scale, double* u, cudaStream_t s) {
    k_axpy_u_f32<<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, du, scale, u);
}

__global__ void k_f32_to_f64_scaled(uint32_t n, const float* __restrict__ x, double scale,
                                    double* __restrict__ y) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        y[i] = scale * (double)x[i];
}
void launch_f32_to_f64_scaled(uint32_t n, const float* x, double scale, double* y,
                              cudaStream_t s) {
    k_f32_to_f64_scaled<<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, x, scale, y);
}
// y = u + alpha du
__global__ void k_axpby_trial(uint32_t n, const double* __restrict__ u, double alpha,
                              const double* __restrict__ du, double* __restrict__ y) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        y[i] = u[i] + alpha * du[i];
}
void launch_trial(uint32_t n, const double* u, double alpha, const double* du, double* y,
                  cudaStream_t s) {
    k_axpby_trial<<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, u, alpha, du, y);
}

// One warp, one bounded wait on a flag that nothing sets: the wait gives up
// after the status word's wait limit and raises FM_FLAG_TIMEOUT.
__global__ void __launch_bounds__(32) k_wait_probe(const unsigned* flag, unsigned* status) {
    wait_flags_warp(flag, true, 1u, status, 0u);
}

void launch_wait_probe(const unsigned* flag, unsigned* status, cudaStream_t s) {
    k_wait_probe<<<1, 32, 0, s>>>(flag, status);
}

// Load-step predictor: v = frac*val - u on constrained DOFs (0 elsewhere),
// in FP64 and (optionally) FP32; ||v||^2 through the deterministic reduction.
__global__ void __launch_bounds__(kVecThreads)
    k_bc_increment(uint32_t n, const uint8_t* __restrict__ mask, const double* __restrict__ val,
                   double frac, const double* __restrict__ u, double* __restrict__ v,
                   float* __restrict__ v32, double* partials, unsigned* counter, double* out) {
    double s = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        const double d = mask[i] ? (val ? frac * val[i] : 0.0) - u[i] : 0.0;
        v[i] = d;
        if (v32) v32[i] = (float)d;
        s += d * d;
    }
    __shared__ double sbuf[32];
    const double bt = block_sum(s, sbuf);
    grid_reduce_finish<double>(bt, partials, counter, [&](double total) { *out = total; });
}
void launch_bc_increment(uint32_t n, const uint8_t* mask, const double* val, double frac,
                         const double* u, double* v, float* v32, double* partials,
                         unsigned* counter, double* out, cudaStream_t s) {
    k_bc_increment<<<kRedBlocks, kVecThreads, 0, s>>>(n, mask, val, frac, u, v, v32, partials,
                                                     counter, out);
}

// R = -f - K v on free DOFs, 0 on constrained
template <typename T>
__global__ void k_predictor_rhs(uint32_t n, const uint8_t* __restrict__ mask,
                                const double* __restrict__ f, const T* __restrict__ Kv,
                                double* __restrict__ R) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        R[i] = mask[i] ? 0.0 : -f[i] - (double)Kv[i];
}
template <typename T>
void launch_predictor_rhs(uint32_t n, const uint8_t* mask, const double* f, const T* Kv,
                          double* R, cudaStream_t s) {
    k_predictor_rhs<T><<<kRedBlocks * 2, kVecThreads, 0, s>>>(n, mask, f, Kv, R);
}

// Dirichlet elimination on an assembled node-block K: entries in a
// constrained row or column become 0, constrained diagonals 1.
template <typename T>
__global__ void __launch_bounds__(256)
    k_apply_bc_nodes(uint32_t nn, const uint32_t* __restrict__ nbr_ptr,
                     const uint32_t* __restrict__ nbr, const uint8_t* __restrict__ mask,
                     T* __restrict__ K) {
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t n = warp; n < nn; n += nwarps) {
        const uint32_t nb0 = nbr_ptr[n];
        const int deg = (int)(nbr_ptr[n + 1] - nb0);
        const int rl = 3 * deg;
        T* v = K + 9 * (size_t)nb0;
        for (int idx = lane; idx < 3 * rl; idx += 32) {
            const int p = idx / rl;
            const int rem = idx - p * rl;
            const int k = rem / 3;
            const uint32_t row = 3 * n + p;
            const uint32_t col = 3 * __ldg(nbr + nb0 + k) + (rem - 3 * k);
            if (mask[row] | mask[col]) v[idx] = (row == col) ? T(1) : T(0);
        }
    }
}
template <typename T>
void launch_apply_bc_nodes(uint32_t nn, const uint32_t* nbr_ptr, const uint32_t* nbr,
                           const uint8_t* mask, T* K, cudaStream_t s) {
    k_apply_bc_nodes<T><<<kSpmvBlocks, 256, 0, s>>>(nn, nbr_ptr, nbr, mask, K);
}

// ---- explicit instantiations ------------------------------------------------
template void launch_predictor_rhs<double>(uint32_t, const uint8_t*, const double*,
                                           const double*, double*, cudaStream_t);
template void launch_predictor_rhs<float>(uint32_t, const uint8_t*, const double*, const float*,
                                          double*, cudaStream_t);
template void launch_apply_bc_nodes<double>(uint32_t, const uint32_t*, const uint32_t*,
                                            const uint8_t*, double*, cudaStream_t);
template void launch_apply_bc_nodes<float>(uint32_t, const uint32_t*, const uint32_t*,
                                           const uint8_t*, float*, cudaStream_t);
#define FM_INST(T)                                                                              \
    template cudaError_t launch_spmv_csr<T>(uint32_t, uint64_t, uint32_t, const uint32_t*,      \
                                            const uint32_t*, const T*, const T*, T*, T*,        \
                                            unsigned*, double*, cudaStream_t, const unsigned*); \
    template void launch_ilu0_csr<T>(const CsrDev&, const T*, T*, T*, unsigned*, unsigned,      \
                                     unsigned*, int, cudaStream_t);                             \
    template cudaError_t launch_trsv_lower_csr<T>(const CsrDev&, const T*, const T*, T*,        \
                                                  unsigned*, unsigned, unsigned*, int,          \
                                                  cudaStream_t, const unsigned*);               \
    template cudaError_t launch_trsv_upper_csr<T>(const CsrDev&, const T*, const T*, const T*,  \
                                                  T*, unsigned*, unsigned, unsigned*, int,      \
                                                  cudaStream_t, const unsigned*);               \
    template void launch_dot<T>(uint32_t, const T*, const T*, T*, unsigned*, double*,           \
                                cudaStream_t);                                                  \
    template cudaError_t launch_pcg_init<T>(uint32_t, const T*, T*, bool, T*, double, T*,       \
                                            unsigned*, DevScalars*, PcgReport*, unsigned,       \
                                            cudaStream_t);                                      \
    template cudaError_t launch_pcg_start<T>(uint32_t, const T*, const T*, const T*, T*, T*,    \
                                             unsigned*, DevScalars*, cudaStream_t);             \
    template cudaError_t launch_pcg_update_xr<T>(uint32_t, const T*, const T*, T*, T*, T*,      \
                                                 DevScalars*, cudaStream_t);                    \
    template cudaError_t launch_pcg_rz<T>(uint32_t, const T*, const T*, double, T*, unsigned*,  \
                                          DevScalars*, PcgReport*, unsigned, cudaStream_t);     \
    template cudaError_t launch_pcg_update_p<T>(uint32_t, const T*, T*, DevScalars*,            \
                                                cudaStream_t);
FM_INST(double)
FM_INST(float)
#undef FM_INST

}  // namespace fm
