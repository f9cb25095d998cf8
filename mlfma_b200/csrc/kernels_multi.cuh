// Many right-hand sides in one product: the far-field stages and the near
// field applied to nr vectors at once.  Included once, by kernels.cu.
//
// Layout with the right-hand side innermost, so that every thread of a warp
// reads a different right-hand side of the same element (coalesced), and
// every coefficient (pattern, transfer function, stencil weight, near-field
// entry) is read once per product instead of once per right-hand side:
//   x, y (tree order)     [n][nr]
//   A_l, B_l per level     [box][direction][2 components][nr]
//
// S2M, L2T and the near field are small dense complex products per leaf
// (patterns x right-hand sides), done by one register-tiled complex GEMM
// device routine; M2L works on sibling groups (the children of one parent
// share their candidate source boxes), so each source pattern is read once per
// group rather than once per interaction pair; interpolation and
// anterpolation keep the single-product structure over chunks of right-hand
// sides.
#pragma once

#include "device.cuh"
#include "zmath.cuh"

namespace mlfma {
namespace {

// ------------------------------------------------------------ complex GEMM tile
// One thread block computes a BM x BN tile of
//   Cm[m][n] = sum_k opA(m, k) * B(k, n)
// with opA(m, k) = A[m * sam + k * sak] (conjugated when CONJ_A), B row k at
// B + (bidx ? bidx[k] : k) * ldb (entries n contiguous), output element (m, n)
// at out + m * ldc + n, converted to the output type.  K is walked in chunks of
// BK through shared memory; each of the 128 threads keeps a 4 x TN register
// tile.  TN = 1..4 is the least with BN = 16 TN >= nr, so that a product on few
// right-hand sides does not multiply a 64-wide tile of padding (12,347 dipoles
// x 17, complex-float far field: S2M 158 -> 85, L2T 252 -> 122, near field 277 ->
// 174 us with TN = 2 in place of 4).  Every output's sum runs over k in order, whatever TN.
constexpr int kGemmThreads = 128;
constexpr int kBM = 32, kBK = 8;
constexpr int kLdA = kBM * kBK / kGemmThreads;  // A entries loaded per thread (2)

template <class C> __device__ __forceinline__ C conj_c(C a) { a.y = -a.y; return a; }
template <class C, class S> __device__ __forceinline__ C to_c(S v);
template <> __device__ __forceinline__ double2 to_c<double2, double2>(double2 v) { return v; }
template <> __device__ __forceinline__ float2 to_c<float2, float2>(float2 v) { return v; }
template <> __device__ __forceinline__ float2 to_c<float2, double2>(double2 v) {
    return make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
}
template <> __device__ __forceinline__ double2 to_c<double2, float2>(float2 v) { return make_double2(v.x, v.y); }

template <int TN, class C, class TA, class TB, class TO, bool CONJ_A, bool A_KMAJOR>
__device__ __forceinline__ void cgemm_tile(int M, int N, int K, int m0, int n0, const TA* __restrict__ A,
                                           long long sam, long long sak, const TB* __restrict__ B,
                                           const int* __restrict__ bidx, long long ldb, TO* __restrict__ out,
                                           long long ldc, C (*As)[kBM + 1], C (*Bs)[16 * TN]) {
    constexpr int kBN = 16 * TN, kLdB = kBK * kBN / kGemmThreads;  // B entries loaded per thread
    const int tid = threadIdx.x;
    const int ty = tid >> 4, tx = tid & 15;  // rows 4 ty .. 4 ty + 3, columns tx + 16 j
    C acc[4][TN];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = zero<C>();
    // Registers of the next tile: its global loads are in flight while the
    // current tile is multiplied out of shared memory.
    C ra[kLdA], rb[kLdB];
    auto load = [&](int k0) {
#pragma unroll
        for (int u = 0; u < kLdA; ++u) {  // A tile: BM x BK
            const int idx = tid + u * kGemmThreads;
            int mm, kk;
            if (A_KMAJOR) { mm = idx / kBK; kk = idx % kBK; } else { kk = idx / kBM; mm = idx % kBM; }
            const int m = m0 + mm, k = k0 + kk;
            C v = zero<C>();
            if (m < M && k < K) {
                v = to_c<C, TA>(A[m * sam + k * sak]);
                if (CONJ_A) v = conj_c(v);
            }
            ra[u] = v;
        }
#pragma unroll
        for (int u = 0; u < kLdB; ++u) {  // B tile: BK x BN
            const int idx = tid + u * kGemmThreads;
            const int kk = idx / kBN, nn = idx % kBN;
            const int k = k0 + kk, n = n0 + nn;
            C v = zero<C>();
            if (k < K && n < N) {
                const long long row = bidx ? static_cast<long long>(bidx[k]) : static_cast<long long>(k);
                v = to_c<C, TB>(B[row * ldb + n]);
            }
            rb[u] = v;
        }
    };
    load(0);
    for (int k0 = 0; k0 < K; k0 += kBK) {
#pragma unroll
        for (int u = 0; u < kLdA; ++u) {
            const int idx = tid + u * kGemmThreads;
            if (A_KMAJOR) As[idx % kBK][idx / kBK] = ra[u]; else As[idx / kBM][idx % kBM] = ra[u];
        }
#pragma unroll
        for (int u = 0; u < kLdB; ++u) {
            const int idx = tid + u * kGemmThreads;
            Bs[idx / kBN][idx % kBN] = rb[u];
        }
        __syncthreads();
        if (k0 + kBK < K) load(k0 + kBK);
#pragma unroll
        for (int kk = 0; kk < kBK; ++kk) {
            C a[4], b[TN];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][4 * ty + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = cfma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + 4 * ty + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n < N) out[m * ldc + n] = to_c<TO, C>(acc[i][j]);
        }
    }
}

// ------------------------------------------------------------ S2M (many)
// A_B[e][r] = sum_s R_s[e] x_s[r]  (Leaf::buildMpoleCoeffs, src/fmm/leaf.cpp:212-230,
// for nr vectors).  Work item: (leaf, first row e0 of a BM-row tile).
template <class R, int TN>
__global__ void __launch_bounds__(kGemmThreads)
k_s2m_m(const DevLevelT<R>* __restrict__ lvs, const int2* __restrict__ items, const DevFarLeaf* __restrict__ leaves,
        const typename Cx<R>::T* __restrict__ pat, const double2* __restrict__ x, int nr) {
    using C = typename Cx<R>::T;
    __shared__ C As[kBK][kBM + 1];
    __shared__ C Bs[kBK][16 * TN];
    const int2 it = items[blockIdx.x];
    const DevFarLeaf lf = leaves[it.x];
    const int ne = 2 * lvs[lf.level].ndir;
    C* Am = lvs[lf.level].Am + static_cast<size_t>(lf.box) * ne * nr;
    for (int n0 = 0; n0 < nr; n0 += 16 * TN)
        cgemm_tile<TN, C, C, double2, C, false, false>(ne, nr, lf.nsrc, it.y, n0, pat + lf.pat_off * 2, 1, ne,
                                                   x + static_cast<size_t>(lf.src0) * nr, nullptr, nr, Am, nr,
                                                   As, Bs);
}

// ------------------------------------------------------------ L2T (many)
// y_s[r] = sum_e conj(R_s[e]) b_B[e][r]  (Leaf::evalFarSols, src/fmm/leaf.cpp:257-280).
// Work item: (leaf, first source s0 of a BM-source tile).
template <class R, int TN>
__global__ void __launch_bounds__(kGemmThreads)
k_l2t_m(const DevLevelT<R>* __restrict__ lvs, const int2* __restrict__ items, const DevFarLeaf* __restrict__ leaves,
        const typename Cx<R>::T* __restrict__ pat, double2* __restrict__ yfar, int nr) {
    using C = typename Cx<R>::T;
    __shared__ C As[kBK][kBM + 1];
    __shared__ C Bs[kBK][16 * TN];
    const int2 it = items[blockIdx.x];
    const DevFarLeaf lf = leaves[it.x];
    const int ne = 2 * lvs[lf.level].ndir;
    const C* Bm = lvs[lf.level].Bm + static_cast<size_t>(lf.box) * ne * nr;
    for (int n0 = 0; n0 < nr; n0 += 16 * TN)
        cgemm_tile<TN, C, C, C, double2, true, true>(lf.nsrc, nr, ne, it.y, n0, pat + lf.pat_off * 2, ne, 1, Bm,
                                                 nullptr, nr, yfar + static_cast<size_t>(lf.src0) * nr, nr, As, Bs);
}

// ------------------------------------------------------------ near field (many)
// y_i[r] = sum_j Z_ij x_cols(j)[r] per block row (gather form, both
// orientations stored).  Work item: (row block, first row of a BM-row tile).
template <int TN>
__global__ void __launch_bounds__(kGemmThreads)
k_near_m(const DevNearRow* __restrict__ rows, const int2* __restrict__ items, const double2* __restrict__ Z,
         const int* __restrict__ cols, const double2* __restrict__ x, double2* __restrict__ y, int nr) {
    __shared__ double2 As[kBK][kBM + 1];
    __shared__ double2 Bs[kBK][16 * TN];
    const int2 it = items[blockIdx.x];
    const DevNearRow Rw = rows[it.x];
    for (int n0 = 0; n0 < nr; n0 += 16 * TN)
        cgemm_tile<TN, double2, double2, double2, double2, false, true>(
            Rw.nrow, nr, Rw.ncol, it.y, n0, Z + Rw.off, Rw.ncol, 1, x, cols + Rw.col_off, nr,
            y + static_cast<size_t>(Rw.row0) * nr, nr, As, Bs);
}

// ------------------------------------------------------------ M2L (many)
// b_B = w (2 pi / nph) sum_{S in list 2 of B} T[c_B - c_S] a_S
// (Node::buildMpoleToLocalCoeffs, src/fmm/node.cpp:105-134).  One block per
// (sibling group, run of D directions), D the most that 2 nr threads each leave
// room for (at most kM2LmDirs); thread = (direction, component, rhs).  The
// group's candidate sources are walked once; each loaded pattern value is used
// for every target of the group that has the source in its list 2.
//
// Bound by FP64 (FP32) multiply-adds: the loop is instantiated per number of
// targets, as a group of a surface holds about four of eight (with all eight
// slots multiplied: r = 2 sphere x 64, FP64, 1,500 us, now 1,093 us), and blocks
// of few right-hand sides take several directions (12,347 dipoles x 17, complex
// float: 438 us, now 328 us).  Two columns per thread, sharing a transfer value's
// read, measured 1,062 us there, but 437 us on the 17 and 710 in place of 458 us
// on 5 right-hand sides.
constexpr int kM2LmThreads = 128;  // nr <= 64
constexpr int kM2LmDirs = 4;       // most directions of a block

// The transfer values are pre-gathered per group at setup, already scaled by
// the quadrature weight: t8[group][direction][candidate][target] (zero where
// the candidate is not in the target's list 2), so the inner loop has one
// dependent global load (the candidate's pattern) and reads the transfer
// values from shared memory.
constexpr int kCandChunk = 64;

template <class R>
__global__ void __launch_bounds__(kM2LmThreads)
k_m2l_m(const DevLevelT<R>* __restrict__ lvs, const DevM2LGroup* __restrict__ groups, int ngroups,
        const int* __restrict__ cand_src, const typename Cx<R>::T* __restrict__ t8, int nr, int D, int zero_empty) {
    using C = typename Cx<R>::T;
    constexpr int U = sizeof(R) == 4 ? 8 : 4;  // candidates whose loads are in flight together
    extern __shared__ __align__(16) unsigned char smraw[];
    C* tsm = reinterpret_cast<C*>(smraw);  // [D][kCandChunk][kMaxGroup]
    __shared__ int ssm[kCandChunk];
    const DevM2LGroup g = groups[blockIdx.x % ngroups];
    const DevLevelT<R> lv = lvs[g.level];
    const int per_dir = 2 * nr, ndir = lv.ndir;
    const int d0 = (blockIdx.x / ngroups) * D, dn = min(D, ndir - d0);
    const int ds = threadIdx.x / per_dir;           // direction of the run
    const int cr = threadIdx.x - ds * per_dir;      // component * nr + r
    const bool live = ds < dn;
    const int d = d0 + (live ? ds : 0);
    const C* tg = t8 + g.t8_off + static_cast<long long>(d0) * g.ncand * kMaxGroup;
    auto group = [&](auto nt) {
        constexpr int NT = decltype(nt)::value;
        C acc[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t] = zero<C>();
        for (int c0 = 0; c0 < g.ncand; c0 += kCandChunk) {
            const int nc = min(kCandChunk, g.ncand - c0);
            for (int q = 0; q < dn; ++q)
                for (int i = threadIdx.x; i < nc * kMaxGroup; i += blockDim.x)
                    tsm[q * kCandChunk * kMaxGroup + i] =
                        tg[(static_cast<long long>(q) * g.ncand + c0) * kMaxGroup + i];
            for (int i = threadIdx.x; i < nc; i += blockDim.x) ssm[i] = cand_src[g.cand0 + c0 + i];
            __syncthreads();
            if (live) {
                const C* ts = tsm + ds * kCandChunk * kMaxGroup;
                for (int i = 0; i < nc; i += U) {
                    C a[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        a[u] = (i + u < nc) ? lv.Am[(static_cast<size_t>(ssm[i + u]) * ndir + d) * per_dir + cr] : zero<C>();
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (i + u >= nc) break;
#pragma unroll
                        for (int t = 0; t < NT; ++t) acc[t] = cfma(ts[(i + u) * kMaxGroup + t], a[u], acc[t]);
                    }
                }
            }
            __syncthreads();
        }
        if (!live) return;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            C* out = lv.Bm + (static_cast<size_t>(g.tgt[t]) * ndir + d) * per_dir + cr;
            if ((g.empty_mask >> t) & 1) {
                if (zero_empty) *out = zero<C>();
            } else {
                *out = acc[t];
            }
        }
    };
    switch (g.ntgt) {
        case 1: group(std::integral_constant<int, 1>()); break;
        case 2: group(std::integral_constant<int, 2>()); break;
        case 3: group(std::integral_constant<int, 3>()); break;
        case 4: group(std::integral_constant<int, 4>()); break;
        case 5: group(std::integral_constant<int, 5>()); break;
        case 6: group(std::integral_constant<int, 6>()); break;
        case 7: group(std::integral_constant<int, 7>()); break;
        default: group(std::integral_constant<int, 8>()); break;
    }
}

// ------------------------------------------------------------ M2M (many)
// Interpolation and anterpolation on many right-hand sides work on chunks of
// 16 x RPL right-hand sides: lane = component * 16 + r, and each lane carries
// right-hand sides r, r + 16, ... of the chunk, so the 32 lanes of a warp read
// one pattern entry for the whole chunk and both components, while every
// stencil index, weight and shift is the same for the whole warp and is paid
// once per RPL values; warps stride over grid positions.  (kRc: the chunk of
// the anterpolation kernel, RPL = 2.)
constexpr int kRc = 32;
constexpr int kInterpThreads = 256;
constexpr int kInterpWarps = kInterpThreads / 32;
constexpr size_t kWinSmem = 108 * 1024;  // largest tile of the windowed kernels: two blocks per SM
constexpr int kM2MOut = 16;  // most parent phi columns per warp held in registers

// Parent outgoing patterns = sum over children of Interp[shift(child)]
// (Stem::buildMpoleCoeffs and addInterpCoeffs, src/fmm/stem.cpp:72-184).
// Block = (parent, parent theta row, rhs chunk of 16 m2m_rpl right-hand
// sides).  Children one at a time: theta pass of the child into shared memory
// (one row of child phi columns), then the phi pass accumulated in registers
// over the children.  Complex double carries two right-hand sides per lane;
// complex float one (two measured slower: register pressure).
template <class R> __host__ __device__ constexpr int m2m_rpl() { return sizeof(R) == 4 ? 1 : 2; }
template <class R> __host__ __device__ constexpr bool m2m_rows_fast() { return sizeof(R) == 8; }

template <class R, int W, int OUT>  // OUT: parent phi columns per warp (nph <= OUT * 8)
__global__ void __launch_bounds__(kInterpThreads)
k_m2m_m(const DevLevelT<R>* __restrict__ lvs, DevTransT<R> T, int nr, int rows_fast) {
    using C = typename Cx<R>::T;
    constexpr int RPL = m2m_rpl<R>();
    extern __shared__ unsigned char smraw[];
    C* sm = reinterpret_cast<C*>(smraw);  // [mph][32 lanes][RPL]
    // grid order: rows fastest (the blocks of one parent together, its
    // children read from DRAM about once; the FP64 default) or parents
    // fastest (the complex-float default); the autotuner may change it
    const int jth = rows_fast ? blockIdx.x : blockIdx.y;
    const int par = rows_fast ? blockIdx.z : blockIdx.x;
    const int r0 = (rows_fast ? blockIdx.y : blockIdx.z) * 16 * RPL;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int comp = lane >> 4, r = lane & 15;
    bool live[RPL];
#pragma unroll
    for (int j = 0; j < RPL; ++j) live[j] = r0 + r + 16 * j < nr;
    const int col = comp * nr + r0 + r;  // offset of (component, rhs) inside a direction
    const DevLevelT<R> P = lvs[T.plevel];
    const DevLevelT<R> Cl = lvs[T.plevel + 1];
    const int nph = P.nph, mph = Cl.nph, halfm = Cl.nph / 2;
    const int c0 = T.child_ptr[par], nch = T.child_ptr[par + 1] - c0;
    // Stencils in shared memory: this row's theta taps (sources; the weights
    // come with the shift from fold_up), every column's phi taps.
    __shared__ int th_src[W], th_refl[W];
    __shared__ int ph_src[OUT * kInterpWarps * W];
    __shared__ R ph_cf[OUT * kInterpWarps * W];
    if (threadIdx.x < W) {
        th_src[threadIdx.x] = T.up_th.src[jth * W + threadIdx.x];
        th_refl[threadIdx.x] = T.up_th.refl[jth * W + threadIdx.x];
    }
    for (int i = threadIdx.x; i < nph * W; i += blockDim.x) {
        ph_src[i] = T.up_ph.src[i];
        ph_cf[i] = T.up_ph.coef[i];
    }
    __syncthreads();
    C acc[OUT][RPL];
#pragma unroll
    for (int u = 0; u < OUT; ++u)
#pragma unroll
        for (int j = 0; j < RPL; ++j) acc[u][j] = zero<C>();
    if (nch == 0)  // (a listed parent has a child; kept well defined regardless)
        for (int iph = warp; iph < mph; iph += kInterpWarps)
#pragma unroll
            for (int j = 0; j < RPL; ++j) sm[(iph * 32 + lane) * RPL + j] = zero<C>();
    for (int c = 0; c < nch; ++c) {
        const C* Ac = Cl.Am + static_cast<size_t>(T.child_box[c0 + c]) * Cl.ndir * 2 * nr + col;
        // weights of this row with the child's octant shift folded in: [iph][k]
        const C* fu = T.fold_up + (static_cast<size_t>(T.child_oct[c0 + c]) * P.nth + jth) * mph * W;
        for (int iph = warp; iph < mph; iph += kInterpWarps) {
            const int iref = iph < halfm ? iph + halfm : iph - halfm;
            C v[RPL];
#pragma unroll
            for (int j = 0; j < RPL; ++j) v[j] = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const C* a = Ac + static_cast<size_t>(th_src[k] * mph + (th_refl[k] ? iref : iph)) * 2 * nr;
                const C f = fu[iph * W + k];
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                    if (live[j]) v[j] = cfma(f, a[16 * j], v[j]);
            }
            // the phi pass is the same linear map for every child: sum the
            // children's theta passes first (each entry is this thread's own)
#pragma unroll
            for (int j = 0; j < RPL; ++j) {
                C& o = sm[(iph * 32 + lane) * RPL + j];
                o = c == 0 ? v[j] : cadd(o, v[j]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < OUT; ++u) {
        const int jph = warp + u * kInterpWarps;
        if (jph >= nph) break;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const R cf = ph_cf[jph * W + k];
            const C* v = sm + (ph_src[jph * W + k] * 32 + lane) * RPL;
#pragma unroll
            for (int j = 0; j < RPL; ++j) acc[u][j] = crfma(cf, v[j], acc[u][j]);
        }
    }
    C* Ap = P.Am + (static_cast<size_t>(T.par_box[par]) * P.ndir + static_cast<size_t>(jth) * nph) * 2 * nr + col;
#pragma unroll
    for (int u = 0; u < OUT; ++u) {
        const int jph = warp + u * kInterpWarps;
        if (jph >= nph) break;
#pragma unroll
        for (int j = 0; j < RPL; ++j)
            if (live[j]) Ap[static_cast<size_t>(jph) * 2 * nr + 16 * j] = acc[u][j];
    }
}

// ------------------------------------------------------------ L2L (many)
// child local += Anterp[shift(parent local)] (Stem::getShiftedLocalCoeffs and
// addAnterpCoeffs, src/fmm/stem.cpp:109-244).  Block = ((parent, child) pair,
// l2l_pairs child phi column pairs {j, j + cph/2}, rhs chunk): the transposed
// phi pass for those columns over all parent theta rows into shared memory
// (neighbouring columns share most of their parent taps, which then hit L1),
// then the transposed theta pass, whose pole reflection only moves between
// the two columns of a pair.
// (default: 2 column pairs for complex float; 1 for complex double, whose tile
// would otherwise hold occupancy to two blocks per SM; the autotuner may change
// it)
template <class R> __host__ __device__ constexpr int l2l_pairs() { return sizeof(R) == 4 ? 2 : 1; }

template <class R, int W, int kL2LPairs>
__global__ void __launch_bounds__(kInterpThreads)
k_l2l_m(const DevLevelT<R>* __restrict__ lvs, DevTransT<R> T, const int2* __restrict__ pairs, int nr) {
    using C = typename Cx<R>::T;
    constexpr int NC = 2 * kL2LPairs;  // columns of the block
    extern __shared__ unsigned char smraw[];
    C* sm = reinterpret_cast<C*>(smraw);  // [pth][NC][32 lanes][2], then the theta taps
    const int2 pc = pairs[blockIdx.x];
    const int r0 = blockIdx.z * kRc;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int comp = lane >> 4, r = lane & 15;
    const bool live0 = r0 + r < nr, live1 = r0 + r + 16 < nr;
    const int col = comp * nr + r0 + r;
    const DevLevelT<R> P = lvs[T.plevel];
    const DevLevelT<R> Cl = lvs[T.plevel + 1];
    const int pth = P.nth, pph = P.nph, cth = Cl.nth, cph = Cl.nph, halfc = Cl.nph / 2;
    const int j0 = blockIdx.y * kL2LPairs, npair = min(kL2LPairs, halfc - j0);
    const C* Bp = P.Bm + static_cast<size_t>(T.par_box[pc.x]) * P.ndir * 2 * nr + col;
    // weights with the child's octant shift folded in: [ith][jph][k]
    const C* fd = T.fold_dn + static_cast<size_t>(T.child_oct[pc.y]) * pth * cph * W;
    // column c of the block: pair c % kL2LPairs, side c / kL2LPairs
    __shared__ int ph_src[NC * W];
    // dynamic shared memory: the tile, then cth x W theta taps (weight, source, reflection)
    R* th_cf = reinterpret_cast<R*>(sm + static_cast<size_t>(pth) * NC * 64);
    int* th_src = reinterpret_cast<int*>(th_cf + cth * W);
    int* th_refl = th_src + cth * W;
    for (int i = threadIdx.x; i < NC * W; i += blockDim.x) {
        const int c = i / W, k = i - c * W;
        const int pr = c % kL2LPairs;
        const int jph = j0 + min(pr, npair - 1) + (c / kL2LPairs) * halfc;
        ph_src[i] = T.dn_ph.src[jph * W + k];
    }
    for (int i = threadIdx.x; i < cth * W; i += blockDim.x) {
        th_src[i] = T.dn_th.src[i];
        th_refl[i] = T.dn_th.refl[i];
        th_cf[i] = T.dn_th.coef[i];
    }
    __syncthreads();
    for (int pos = warp; pos < pth * NC; pos += kInterpWarps) {
        const int ith = pos / NC, c = pos - ith * NC;
        const int jph = j0 + min(c % kL2LPairs, npair - 1) + (c / kL2LPairs) * halfc;
        const C* f = fd + (static_cast<size_t>(ith) * cph + jph) * W;
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const C* b = Bp + static_cast<size_t>(ith * pph + ph_src[c * W + k]) * 2 * nr;
            const C fk = f[k];
            if (live0) v0 = cfma(fk, b[0], v0);
            if (live1) v1 = cfma(fk, b[16], v1);
        }
        sm[(pos * 32 + lane) * 2] = v0;
        sm[(pos * 32 + lane) * 2 + 1] = v1;
    }
    __syncthreads();
    C* Bc = Cl.Bm + static_cast<size_t>(T.child_box[pc.y]) * Cl.ndir * 2 * nr + col;
    for (int pos = warp; pos < cth * NC; pos += kInterpWarps) {
        const int jth = pos / NC, c = pos - jth * NC;
        const int pr = c % kL2LPairs, side = c / kL2LPairs;
        if (pr >= npair) continue;
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int q = jth * W + k;
            const int c2 = th_refl[q] ? pr + (1 - side) * kL2LPairs : c;
            const C* v = sm + ((th_src[q] * NC + c2) * 32 + lane) * 2;
            v0 = crfma(th_cf[q], v[0], v0);
            v1 = crfma(th_cf[q], v[1], v1);
        }
        C* o = Bc + static_cast<size_t>(jth * cph + j0 + pr + side * halfc) * 2 * nr;
        if (live0) o[0] = cadd(o[0], v0);
        if (live1) o[16] = cadd(o[16], v1);
    }
}

// ------------------------------------------------------------ windowed interpolation (many)
// k_m2m_m and k_l2l_m read every tap of every output, and a folded weight for it,
// from L2, one dependent on the other.  Here a warp forms the kWinRows (parent
// theta rows) or kWinCols (child phi columns) neighbouring outputs of one
// position together: it walks the union of their taps in order, loads each value
// once, and adds it to the outputs that have that tap (a mask).  Used where the
// unions fit kWinTapsUp / kWinTapsDn (the default six-point interpolation) and the
// tile fits kWinSmem; wider stencils and larger grids keep the per-output
// kernels.  Measured (M2M, L2L): r = 2 sphere x 64, FP64, 605 and 1,250 us before,
// 448 and 915 now; 12,347 dipoles x 17, complex float, L2L 245 -> 149 us.

// Shared memory of the two tiles.
template <class R>
size_t m2m_w_smem(int child_nph) {
    return sizeof(typename Cx<R>::T) * child_nph * kWinRows * 32;
}
template <class R>
size_t l2l_w_smem(int parent_nth, int child_nth, int rpl) {
    return sizeof(typename Cx<R>::T) * parent_nth * 2 * kWinCols * 32 * rpl +
           static_cast<size_t>((child_nth + kWinCols - 1) / kWinCols) * kWinTapsTh * (kWinCols * sizeof(R) + sizeof(int2));
}

// Parent outgoing patterns, complex double (complex float, whose sums keep the
// folded weights' rounding, was slower this way: 161 -> 244 us).  Children
// shifted and summed at every tap of the union first, then one theta pass with
// real weights from shared memory, then the phi pass.  Block = (parent, group of
// kWinRows parent theta rows, chunk of 16 rhs); lane = component * 16 + rhs.
template <int W>
__global__ void __launch_bounds__(kInterpThreads, 2)
k_m2m_w(const DevLevelT<double>* __restrict__ lvs, DevTransT<double> T, int nr, int ng) {
    constexpr int J = kWinRows;
    extern __shared__ __align__(16) unsigned char smraw[];
    double2* sm = reinterpret_cast<double2*>(smraw);  // [mph][J][32 lanes]
    __shared__ int2 taps[kWinTapsUp];                 // source row, reflected (bit 0) and the rows that have it
    __shared__ double2 wt[kWinTapsUp][J / 2];         // weights of the group's rows, sign included
    // row groups fastest: the blocks of one parent together
    const int jg = blockIdx.x % ng, nc = (nr + 15) / 16;
    const int r0 = (blockIdx.x / ng) % nc * 16, par = blockIdx.x / ng / nc;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int comp = lane >> 4, r = lane & 15;
    const bool live = r0 + r < nr;
    const int col = comp * nr + r0 + (live ? r : 0);
    const DevLevelT<double> P = lvs[T.plevel];
    const DevLevelT<double> Cl = lvs[T.plevel + 1];
    const int nph = P.nph, mph = Cl.nph, halfm = Cl.nph / 2;
    const int j0 = jg * J, nj = min(J, P.nth - j0);
    const int c0 = T.child_ptr[par], nch = T.child_ptr[par + 1] - c0;
    if (threadIdx.x < kWinTapsUp) {
        taps[threadIdx.x] = T.win_up[jg * kWinTapsUp + threadIdx.x];
#pragma unroll
        for (int h = 0; h < J / 2; ++h) {
            const double* q = T.win_up_w + (jg * kWinTapsUp + threadIdx.x) * J + 2 * h;
            wt[threadIdx.x][h] = make_double2(q[0], q[1]);
        }
    }
    __syncthreads();
    const int nt = T.win_up_n[jg];
    for (int iph = warp; iph < mph; iph += kInterpWarps) {
        const int iref = iph < halfm ? iph + halfm : iph - halfm;
        double2 v[J];
#pragma unroll
        for (int j = 0; j < J; ++j) v[j] = z0();
        constexpr int U = 5;  // taps taken together
        static_assert(kWinTapsUp % U == 0, "whole runs of taps");
        for (int t0 = 0; t0 < nt; t0 += U) {
            double2 sum[U];
            int at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int2 q = taps[t0 + u];  // (past the union: some direction, in no row)
                at[u] = q.x * mph + (q.y & 1 ? iref : iph);
                sum[u] = z0();
            }
            for (int c = 0; c < nch; ++c) {
                const double2* Ac = Cl.Am + static_cast<size_t>(T.child_box[c0 + c]) * Cl.ndir * 2 * nr + col;
                const double2* sh = Cl.shift_up + static_cast<size_t>(T.child_oct[c0 + c]) * Cl.ndir;
                double2 a[U], f[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    a[u] = Ac[static_cast<size_t>(at[u]) * 2 * nr];
                    f[u] = sh[at[u]];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) sum[u] = cfma(f[u], a[u], sum[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int m = taps[t0 + u].y;
#pragma unroll
                for (int h = 0; h < J / 2; ++h) {
                    const double2 q = wt[t0 + u][h];
                    if (m & 2 << 2 * h) v[2 * h] = crfma(q.x, sum[u], v[2 * h]);
                    if (m & 4 << 2 * h) v[2 * h + 1] = crfma(q.y, sum[u], v[2 * h + 1]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) sm[(iph * J + j) * 32 + lane] = v[j];
    }
    __syncthreads();
    double2* Ap = P.Am + (static_cast<size_t>(T.par_box[par]) * P.ndir + static_cast<size_t>(j0) * nph) * 2 * nr + col;
    for (int jph = warp; jph < nph; jph += kInterpWarps) {
        int src[W];
        double cf[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            src[k] = T.up_ph.src[jph * W + k];
            cf[k] = T.up_ph.coef[jph * W + k];
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (j >= nj) break;
            double2 acc = z0();
#pragma unroll
            for (int k = 0; k < W; ++k) acc = crfma(cf[k], sm[(src[k] * J + j) * 32 + lane], acc);
            if (live) Ap[static_cast<size_t>(j * nph + jph) * 2 * nr] = acc;
        }
    }
}

// Child local patterns (as k_l2l_m).  Block = ((parent, child) pair, group of
// kWinCols child phi columns and their partners half a turn on, chunk of 16 RPL
// rhs); lane = component * 16 + rhs, RPL right-hand sides a lane.  The phi pass
// goes to shared memory; complex double shifts each value as it is loaded and then
// has real weights, from shared memory; complex float reads weights with the
// shift folded in, with the values.  The theta pass takes kWinCols child rows of a
// column together in the same way (it was bound by its shared-memory reads).
template <class R, int RPL>
__global__ void __launch_bounds__(kInterpThreads, 3)
k_l2l_w(const DevLevelT<R>* __restrict__ lvs, DevTransT<R> T, const int2* __restrict__ pairs, int nr) {
    using C = typename Cx<R>::T;
    constexpr int J = kWinCols, NC = 2 * J;
    extern __shared__ __align__(16) unsigned char smraw[];
    C* sm = reinterpret_cast<C*>(smraw);  // [pth][NC][RPL][32 lanes], then the theta weights and taps
    constexpr bool F64 = sizeof(R) == 8;
    __shared__ int2 taps[2][kWinTapsDn];  // parent column, mask of outputs
    __shared__ R wt[2][kWinTapsDn][J];    // complex double: weights of the group's columns
    __shared__ int ntap[2];
    const int2 pc = pairs[blockIdx.x];
    const int g = blockIdx.y, ng = gridDim.y, r0 = blockIdx.z * 16 * RPL;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int comp = lane >> 4, r = lane & 15;
    bool live[RPL];
#pragma unroll
    for (int q = 0; q < RPL; ++q) live[q] = r0 + r + 16 * q < nr;
    const int col = comp * nr + r0 + r;
    const DevLevelT<R> P = lvs[T.plevel];
    const DevLevelT<R> Cl = lvs[T.plevel + 1];
    const int pth = P.nth, pph = P.nph, cth = Cl.nth, cph = Cl.nph, halfc = Cl.nph / 2;
    const int j0 = g * J, nj = min(J, halfc - j0);
    const C* Bp = P.Bm + static_cast<size_t>(T.par_box[pc.x]) * P.ndir * 2 * nr + col;
    // theta pass: groups of kWinCols child rows
    const int ngt = (cth + J - 1) / J;
    R* th_w = reinterpret_cast<R*>(sm + static_cast<size_t>(pth) * NC * 32 * RPL);  // [ngt][kWinTapsTh][J]
    int2* th_tap = reinterpret_cast<int2*>(th_w + ngt * kWinTapsTh * J);            // parent row, reflected and mask
    if (threadIdx.x < 2 * kWinTapsDn) {
        const int side = threadIdx.x / kWinTapsDn, t = threadIdx.x % kWinTapsDn;
        taps[side][t] = T.win_dn[(side * ng + g) * kWinTapsDn + t];
#pragma unroll
        for (int j = 0; j < J; ++j)
            if (F64) wt[side][t][j] = T.win_dn_w[((side * ng + g) * kWinTapsDn + t) * J + j];
    }
    if (threadIdx.x < 2) ntap[threadIdx.x] = T.win_dn_n[threadIdx.x * ng + g];
    for (int i = threadIdx.x; i < ngt * kWinTapsTh; i += blockDim.x) th_tap[i] = T.win_th[i];
    for (int i = threadIdx.x; i < ngt * kWinTapsTh * J; i += blockDim.x) th_w[i] = T.win_th_w[i];
    __syncthreads();
    for (int pos = warp; pos < pth * 2; pos += kInterpWarps) {
        const int ith = pos >> 1, side = pos & 1, nt = ntap[side];
        const C* f = F64 ? P.shift_down + static_cast<size_t>(T.child_oct[pc.y]) * P.ndir + ith * pph
                         : T.fold_dnw + ((static_cast<size_t>(T.child_oct[pc.y]) * pth + ith) * (2 * ng) + side * ng + g) *
                                            (kWinTapsDn * J);
        const C* b = Bp + static_cast<size_t>(ith) * pph * 2 * nr;
        C v[J][RPL];
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int q = 0; q < RPL; ++q) v[j][q] = zero<C>();
        constexpr int U = 4;  // taps loaded together
        static_assert(kWinTapsDn % U == 0, "whole runs of taps");
        for (int t0 = 0; t0 < nt; t0 += U) {
            C a[U][RPL], w[U][F64 ? 1 : J];
            int m[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int2 tp = taps[side][t0 + u];  // (past the union: column 0, in no output)
                m[u] = tp.y;
#pragma unroll
                for (int q = 0; q < RPL; ++q)
                    a[u][q] = live[q] ? b[static_cast<size_t>(tp.x) * 2 * nr + 16 * q] : zero<C>();
                if (F64) {
                    w[u][0] = f[tp.x];
                } else {
#pragma unroll
                    for (int j = 0; j < J; ++j) w[u][F64 ? 0 : j] = f[(t0 + u) * J + j];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (F64) {
#pragma unroll
                    for (int q = 0; q < RPL; ++q) a[u][q] = cmul(w[u][0], a[u][q]);
                }
#pragma unroll
                for (int j = 0; j < J; ++j)
                    if (m[u] >> j & 1) {
#pragma unroll
                        for (int q = 0; q < RPL; ++q)
                            v[j][q] = F64 ? crfma(wt[side][t0 + u][j], a[u][q], v[j][q])
                                          : cfma(w[u][F64 ? 0 : j], a[u][q], v[j][q]);
                    }
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int q = 0; q < RPL; ++q) sm[((ith * NC + side * J + j) * RPL + q) * 32 + lane] = v[j][q];
    }
    __syncthreads();
    C* Bc = Cl.Bm + static_cast<size_t>(T.child_box[pc.y]) * Cl.ndir * 2 * nr + col;
    for (int pos = warp; pos < ngt * NC; pos += kInterpWarps) {
        const int gt = pos / NC, c = pos - gt * NC;
        const int j = c % J, side = c / J, rows = min(J, cth - gt * J);
        if (j >= nj) continue;
        C* o = Bc + static_cast<size_t>(gt * J * cph + j0 + j + side * halfc) * 2 * nr;
        const size_t row = static_cast<size_t>(cph) * 2 * nr;  // from one child row to the next
        C v[J][RPL], old[J][RPL];
#pragma unroll
        for (int i = 0; i < J; ++i)
#pragma unroll
            for (int q = 0; q < RPL; ++q) {
                v[i][q] = zero<C>();
                old[i][q] = i < rows && live[q] ? o[i * row + 16 * q] : zero<C>();
            }
        const int nt = T.win_th_n[gt], partner = j + (1 - side) * J;
#pragma unroll 4
        for (int t = 0; t < nt; ++t) {
            const int2 tp = th_tap[gt * kWinTapsTh + t];
            const R* w = th_w + (gt * kWinTapsTh + t) * J;
            const C* s1 = sm + (tp.x * NC + (tp.y & 1 ? partner : c)) * RPL * 32 + lane;
#pragma unroll
            for (int q = 0; q < RPL; ++q) {
                const C a = s1[q * 32];
#pragma unroll
                for (int i = 0; i < J; ++i)
                    if (tp.y >> (i + 1) & 1) v[i][q] = crfma(w[i], a, v[i][q]);
            }
        }
#pragma unroll
        for (int i = 0; i < J; ++i)
#pragma unroll
            for (int q = 0; q < RPL; ++q)
                if (i < rows && live[q]) o[i * row + 16 * q] = cadd(old[i][q], v[i][q]);
    }
}

// ------------------------------------------------------------ boundary (many)
// xt[t][r] = x[r][perm[t]]: caller layout (one vector after another, caller
// order) to tree order with the right-hand side innermost.
__global__ void k_gather_m(const double2* __restrict__ x, const int* __restrict__ perm, double2* __restrict__ xt,
                           int n, int nr) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<long long>(n) * nr) return;
    const int t = static_cast<int>(i / nr), r = static_cast<int>(i - static_cast<long long>(t) * nr);
    xt[i] = x[static_cast<size_t>(r) * n + perm[t]];
}

// y[r][perm[t]] (+)= ck (yfar[t][r] + ynear[t][r]) + loads[t] xt[t][r] (loads may
// be null); perm == nullptr: tree order, rhs innermost.
__global__ void k_finish_m(const double2* __restrict__ yfar, const double2* __restrict__ ynear,
                           const int* __restrict__ perm, double2* __restrict__ y, int n, int nr, double2 ck,
                           int accumulate, const double2* __restrict__ xt, const double2* __restrict__ loads) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<long long>(n) * nr) return;
    const int t = static_cast<int>(i / nr), r = static_cast<int>(i - static_cast<long long>(t) * nr);
    double2 v = cmul(ck, cadd(yfar[i], ynear[i]));
    if (loads) v = cfma(loads[t], xt[i], v);
    const size_t o = perm ? static_cast<size_t>(r) * n + perm[t] : static_cast<size_t>(i);
    y[o] = accumulate ? cadd(y[o], v) : v;
}

}  // namespace
}  // namespace mlfma
