// Far-field kernels of the MLFMA matvec: aggregation (S2M), interpolation
// (M2M), translation (M2L), anterpolation (L2L) and disaggregation (L2T).
// Templated on the real type R of the far field (double: FP64 path; float:
// mixed path, complex float storage with float accumulation).  Included once,
// by kernels.cu.
//
// Layout: per level, patterns are [box][direction][2 components] complex;
// element e = 2*direction + component runs contiguously, so a box's
// pattern is one contiguous run of 2*ndir values.
#pragma once

#include <type_traits>

#include "device.cuh"
#include "zmath.cuh"
#include "bulk_copy.cuh"

namespace mlfma {
namespace {

// Programmatic dependent launch.  The far-field chain's kernels after the first
// are launched with programmatic stream serialization, so that a kernel's
// blocks are scheduled while its predecessor on the stream is still draining
// its last wave.  Every chain kernel therefore starts with griddepcontrol.wait,
// which returns once the predecessor grid has completed and its writes are
// visible (a no-op for a kernel launched without the attribute): nothing a
// predecessor writes is read, and nothing it reads is overwritten, before it.
// Only then does the kernel let its own successor launch, so at most one
// kernel's blocks wait ahead of the running one.
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ------------------------------------------------------------ S2M
// a_B[e] = sum_n x_n R_n[e]  (Leaf::buildMpoleCoeffs, src/fmm/leaf.cpp:212-230).
// One block per work item (leaf, run of at most kS2MThreads elements), all leaf
// levels in one launch; one thread per element e (direction, component), so
// every pattern row is read once with coalesced loads; eight sources are in
// flight per thread.
//
// HBM-bound.  An item carries all its pointers, so a block's first eight rows
// are requested after one load instead of a chain of three, and while the
// sources are staged; blocks of 192 threads at 64 registers keep five on an SM
// (352 at 74 kept two).  One B200: r = 8 sphere 510 -> 420 us (2.75 GB, 6.55 TB/s,
// the copy rate), complex float 207 -> 130 us (0.69 GB); r = 2 sphere 37 -> 33
// us, complex float 21 -> 14 us.
constexpr int kS2MThreads = 192;
constexpr int kL2TThreads = 128;
constexpr size_t kL2TStageBytes = 72 * 1024;  // largest local pattern k_l2t stages
constexpr int kL2TRows = 2;  // sources per warp
constexpr int kL2TSrcPerBlock = kL2TRows * kL2TThreads / 32;

// CJ: conjugated patterns, a_B[e] = sum_n x_n conj(R_n[e]) -- the transpose of
// L2T, first stage of the transposed product.
template <class R, bool CJ>
__global__ void __launch_bounds__(kS2MThreads, 5)
k_s2m(const DevS2MItem<R>* __restrict__ items, const double2* __restrict__ x) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ unsigned char smraw[];
    C* xs = reinterpret_cast<C*>(smraw);
    const DevS2MItem<R> it = items[blockIdx.x];
    const int ne = it.ne, nsrc = it.nsrc;
    const bool live = static_cast<int>(threadIdx.x) < it.ec;
    const C* r = it.pat + threadIdx.x;
    C v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
        v[u] = live && u < nsrc ? ldg_stream(r + static_cast<size_t>(u) * ne) : zero<C>();
    for (int i = threadIdx.x; i < nsrc; i += blockDim.x) xs[i] = from_d2<C>(x[it.src0 + i]);
    __syncthreads();
    if (!live) return;
    C a[4] = {zero<C>(), zero<C>(), zero<C>(), zero<C>()};
    for (int s = 0;;) {
        if (s + 8 <= nsrc) {
#pragma unroll
            for (int u = 0; u < 8; ++u) a[u & 3] = CJ ? cjfma(v[u], xs[s + u], a[u & 3]) : cfma(xs[s + u], v[u], a[u & 3]);
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (s + u >= nsrc) break;
                a[u & 3] = CJ ? cjfma(v[u], xs[s + u], a[u & 3]) : cfma(xs[s + u], v[u], a[u & 3]);
            }
        }
        s += 8;
        if (s >= nsrc) break;
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = s + u < nsrc ? ldg_stream(r + static_cast<size_t>(s + u) * ne) : zero<C>();
    }
    it.a[it.e0 + threadIdx.x] = cadd(cadd(a[0], a[1]), cadd(a[2], a[3]));
}

// ------------------------------------------------------------ L2T
// y_m = sum_e conj(R_m[e]) b_B[e]  (Leaf::evalFarSols, src/fmm/leaf.cpp:257-280;
// C k is applied when the result is written out).  One block per work item
// (leaf, run of up to eight sources), two sources per warp with eight loads in
// flight for each and lane, issued before the leaf's local pattern is staged in
// shared memory; the sum is widened to complex double on output.
//
// HBM-bound (latency of the short rows: 3-5 KB a source).  Self-contained items
// and the early loads: r = 2 sphere 45 -> 41 us, r = 8 sphere 597 -> 614 us
// (4.5 TB/s); complex float 22 -> 18 us and 246 -> 183 us.  The four sums per
// lane are a solve's: their order decides its last bits (two sums with twelve
// loads in flight took 575 us on the r = 8 sphere).  Blocks of 256
// threads left more warps idle at a leaf's last run of sources (FP64 598 us,
// complex float 200 us on the r = 8 sphere).
// CJ = false: plain patterns, y_m = sum_e R_m[e] b_B[e] -- the transpose of S2M,
// last stage of the transposed product.
template <class R, bool CJ, bool STAGE>  // STAGE: the local pattern in shared memory
__global__ void __launch_bounds__(kL2TThreads, 4)
k_l2t(const DevL2TItem<R>* __restrict__ items, double2* __restrict__ yfar) {
    chain_wait();
    using C = typename Cx<R>::T;
    constexpr int RW = kL2TRows, U = 8;
    extern __shared__ unsigned char smraw[];
    C* bs = reinterpret_cast<C*>(smraw);
    const DevL2TItem<R> it = items[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ne = it.ne;
    C v[RW][U];  // the rows' first runs, in flight while the local pattern is staged
    auto load = [&](int e) {
#pragma unroll
        for (int q = 0; q < RW; ++q) {
            const int row = warp + q * (kL2TThreads / 32);
            const C* r = it.pat + static_cast<size_t>(row) * ne;
#pragma unroll
            for (int u = 0; u < U; ++u)
                v[q][u] = row < it.cnt && e + 32 * u < ne ? ldg_stream(r + e + 32 * u) : zero<C>();
        }
    };
    load(lane);
    if (STAGE) {
        for (int e = threadIdx.x; e < ne; e += blockDim.x) bs[e] = it.b[e];
        __syncthreads();
    }
    const C* b = STAGE ? bs : it.b;
    C a[RW][4];
#pragma unroll
    for (int q = 0; q < RW; ++q)
#pragma unroll
        for (int k = 0; k < 4; ++k) a[q][k] = zero<C>();
    for (int e = lane;;) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (e + 32 * u >= ne) continue;
            const C bv = b[e + 32 * u];
#pragma unroll
            for (int q = 0; q < RW; ++q) a[q][u & 3] = CJ ? cjfma(v[q][u], bv, a[q][u & 3]) : cfma(v[q][u], bv, a[q][u & 3]);
        }
        e += 32 * U;
        if (e - lane >= ne) break;  // (the whole warp: the sums below shuffle)
        load(e);
    }
#pragma unroll
    for (int q = 0; q < RW; ++q) {
        const C acc = warp_sum(cadd(cadd(a[q][0], a[q][1]), cadd(a[q][2], a[q][3])));
        const int row = warp + q * (kL2TThreads / 32);
        if (lane == 0 && row < it.cnt) yfar[it.src0 + row] = to_d2(acc);
    }
}

// Half patterns (the complex-float far field of the mixed operator): patterns
// are kept for the first half of the directions only (d < ndir/2,
// `hpat`: per source, ndir elements (direction, component)).  The direction
// grid is symmetric under k -> -k (Gauss-Legendre theta rows in mirror pairs,
// an even number of phi columns), and for a real basis function
// R(-k) = conj(R(k)) as a vector; theta-hat is the same at -k and phi-hat flips,
// so the antipodal element anti[e] holds sgn(e) conj(R[e]), sgn = +1 for the
// theta component and -1 for the phi component.  S2M and L2T read each stored
// value once and use it for both directions: half the pattern bytes.  The
// closed-form RWG integrals are ill-conditioned enough that the derived
// antipodal values differ from directly computed ones by about 1e-8 relative:
// far below complex-float rounding, but above the 1e-10 agreement the FP64
// operator keeps with the reference, so the FP64 far field stores every
// direction and uses k_s2m / k_l2t.
// hpat from the full patterns: the first ndir elements of every source.
template <class R>
__global__ void k_half_patterns(const DevLevelT<R>* __restrict__ lvs, const DevFarLeaf* __restrict__ leaves,
                                const double2* __restrict__ pat, typename Cx<R>::T* __restrict__ hpat) {
    using C = typename Cx<R>::T;
    const DevFarLeaf lf = leaves[blockIdx.x];
    const int ne = lvs[lf.level].ndir;
    for (int i = threadIdx.x; i < lf.nsrc * ne; i += blockDim.x) {
        const int s = i / ne, e = i - s * ne;
        hpat[lf.pat_off + static_cast<long long>(s) * ne + e] =
            from_d2<C>(pat[(lf.pat_off + static_cast<long long>(s) * ne) * 2 + e]);
    }
}

// ------------------------------------------------------------ S2M, half patterns
// a_B[e] = sum_n x_n R_n[e]  (Leaf::buildMpoleCoeffs, src/fmm/leaf.cpp:212-230).
// One block per work item (leaf, run of at most kS2MThreads elements of the
// first half), all leaf levels in one launch; one thread per element e, which
// also forms the antipodal element a_B[anti[e]] = sgn sum_n x_n conj(R_n[e]);
// every stored pattern row is read once with coalesced loads; eight sources
// are in flight per thread, the first before the sources are staged (as k_s2m).
// CJ: conjugated patterns, a_B[e] = sum_n x_n conj(R_n[e]) -- the transpose of
// L2T, first stage of the transposed product.
template <class R, bool CJ>
__global__ void __launch_bounds__(kS2MThreads)
k_s2m_half(const DevS2MItem<R>* __restrict__ items, const double2* __restrict__ x) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ unsigned char smraw[];
    C* xs = reinterpret_cast<C*>(smraw);
    const DevS2MItem<R> it = items[blockIdx.x];
    const int ne = it.ne, nsrc = it.nsrc;  // ne: stored elements per source
    const bool live = static_cast<int>(threadIdx.x) < it.ec;
    const C* r = it.pat + threadIdx.x;
    C v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
        v[u] = live && u < nsrc ? ldg_stream(r + static_cast<size_t>(u) * ne) : zero<C>();
    const int e = it.e0 + threadIdx.x;
    const int ea = live ? it.anti[e] : 0;
    for (int i = threadIdx.x; i < nsrc; i += blockDim.x) xs[i] = from_d2<C>(x[it.src0 + i]);
    __syncthreads();
    if (!live) return;
    // a: this element, b: sum of x conj(v) (or x v), the antipodal one up to its sign
    C a[4] = {zero<C>(), zero<C>(), zero<C>(), zero<C>()};
    C b[4] = {zero<C>(), zero<C>(), zero<C>(), zero<C>()};
    for (int s = 0;;) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (s + u >= nsrc) break;
            const C xv = xs[s + u];
            a[u & 3] = CJ ? cjfma(v[u], xv, a[u & 3]) : cfma(xv, v[u], a[u & 3]);
            b[u & 3] = CJ ? cfma(xv, v[u], b[u & 3]) : cjfma(v[u], xv, b[u & 3]);
        }
        s += 8;
        if (s >= nsrc) break;
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = s + u < nsrc ? ldg_stream(r + static_cast<size_t>(s + u) * ne) : zero<C>();
    }
    it.a[e] = cadd(cadd(a[0], a[1]), cadd(a[2], a[3]));
    const C q = cadd(cadd(b[0], b[1]), cadd(b[2], b[3]));
    it.a[ea] = (e & 1) ? C{-q.x, -q.y} : q;
}

// ------------------------------------------------------------ L2T, half patterns
// y_m = sum_e conj(R_m[e]) b_B[e] over the stored half:
// y_m = sum_{e < ndir} conj(R_m[e]) b_B[e] + R_m[e] b'_B[e], b'_B[e] =
// sgn(e) b_B[anti[e]].  One block per work item (leaf, run of up to eight
// sources): two sources per warp, eight loads in flight for each and lane,
// issued before the block stages b_B and b'_B in shared memory (as k_l2t).
// CJ = false: plain patterns (the transpose of S2M).
template <class R, bool CJ>
__global__ void __launch_bounds__(kL2TThreads)
k_l2t_half(const DevL2TItem<R>* __restrict__ items, double2* __restrict__ yfar) {
    chain_wait();
    using C = typename Cx<R>::T;
    constexpr int RW = kL2TRows, U = 8;
    extern __shared__ unsigned char smraw[];
    const DevL2TItem<R> it = items[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ne = it.ne;  // stored elements per source
    C v[RW][U];  // the rows' first runs, in flight while the local pattern is staged
    auto load = [&](int e) {
#pragma unroll
        for (int q = 0; q < RW; ++q) {
            const int row = warp + q * (kL2TThreads / 32);
            const C* r = it.pat + static_cast<size_t>(row) * ne;
#pragma unroll
            for (int u = 0; u < U; ++u)
                v[q][u] = row < it.cnt && e + 32 * u < ne ? ldg_stream(r + e + 32 * u) : zero<C>();
        }
    };
    load(lane);
    C* bs = reinterpret_cast<C*>(smraw);
    C* bp = bs + ne;
    for (int e = threadIdx.x; e < ne; e += blockDim.x) {
        const C q = it.b[it.anti[e]];
        bs[e] = it.b[e];
        bp[e] = (e & 1) ? C{-q.x, -q.y} : q;
    }
    __syncthreads();
    C a[RW][4];
#pragma unroll
    for (int q = 0; q < RW; ++q)
#pragma unroll
        for (int k = 0; k < 4; ++k) a[q][k] = zero<C>();
    for (int e = lane;;) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int ee = e + 32 * u;
            if (ee >= ne) continue;
            const C b0 = bs[ee], b1 = bp[ee];
#pragma unroll
            for (int q = 0; q < RW; ++q) {
                C& acc = a[q][u & 3];
                acc = CJ ? cjfma(v[q][u], b0, acc) : cfma(v[q][u], b0, acc);
                acc = CJ ? cfma(v[q][u], b1, acc) : cjfma(v[q][u], b1, acc);
            }
        }
        e += 32 * U;
        if (e - lane >= ne) break;  // (the whole warp: the sums below shuffle)
        load(e);
    }
#pragma unroll
    for (int q = 0; q < RW; ++q) {
        const C acc = warp_sum(cadd(cadd(a[q][0], a[q][1]), cadd(a[q][2], a[q][3])));
        const int row = warp + q * (kL2TThreads / 32);
        if (lane == 0 && row < it.cnt) yfar[it.src0 + row] = to_d2(acc);
    }
}

// ------------------------------------------------------------ M2M
// Parent outgoing pattern = sum over non-empty children of Interp[shift(child)]:
// shift on the child grid, theta pass with pole reflection, periodic phi pass
// (Stem::buildMpoleCoeffs and addInterpCoeffs, src/fmm/stem.cpp:72-184).
// Block = (parent, tile of `rows` parent theta rows).  Phase 1 computes the
// theta pass of every child into shared memory at once (all loads
// independent); phase 2 forms each parent output from the children's rows.
// POST: the transposed L2L -- no shift before the theta pass; each child's
// interpolated pattern is multiplied by the parent-grid shift of its octant
// (shift_down of the parent level) before the sum over children.
template <class R, int W, bool POST>  // taps per row: 2 * interp_order (both passes)
__global__ void __launch_bounds__(128)
k_m2m(const DevLevelT<R>* __restrict__ lvs, DevTransT<R> T, int rows) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ unsigned char smraw[];
    C* sm = reinterpret_cast<C*>(smraw);
    const int par = blockIdx.x;
    const DevLevelT<R> P = lvs[T.plevel];
    const DevLevelT<R> Cl = lvs[T.plevel + 1];
    const int nph = P.nph, mph = Cl.nph, halfm = Cl.nph / 2;
    const int r0 = blockIdx.y * rows;
    const int nrow = min(P.nth, r0 + rows) - r0;
    if (nrow <= 0) return;
    const int c0 = T.child_ptr[par], nch = T.child_ptr[par + 1] - c0;
    const int per_child = nrow * mph;
    for (int it = threadIdx.x; it < nch * per_child; it += blockDim.x) {
        const int c = it / per_child, e = it - c * per_child;
        const int jr = e / mph, iph = e - jr * mph;
        const int jth = r0 + jr;
        const C* Ac = Cl.A + static_cast<size_t>(T.child_box[c0 + c]) * Cl.ndir * 2;
        const C* sh = Cl.shift_up + static_cast<size_t>(T.child_oct[c0 + c]) * Cl.ndir;
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int q = jth * W + k;
            const bool rf = T.up_th.refl[q];
            const int sp = rf ? (iph < halfm ? iph + halfm : iph - halfm) : iph;
            const R cf = T.up_th.coef[q];
            const int d = T.up_th.src[q] * mph + sp;
            if (POST) {
                v0 = crfma(cf, Ac[2 * d], v0);
                v1 = crfma(cf, Ac[2 * d + 1], v1);
            } else {
                const C ph = sh[d];
                v0 = crfma(cf, cmul(ph, Ac[2 * d]), v0);
                v1 = crfma(cf, cmul(ph, Ac[2 * d + 1]), v1);
            }
        }
        sm[2 * it] = v0;
        sm[2 * it + 1] = v1;
    }
    __syncthreads();
    C* Ap = P.A + (static_cast<size_t>(T.par_box[par]) * P.ndir + static_cast<size_t>(r0) * nph) * 2;
    for (int o = threadIdx.x; o < nrow * nph; o += blockDim.x) {
        const int jr = o / nph, jph = o - jr * nph;
        C a0 = zero<C>(), a1 = zero<C>();
        for (int c = 0; c < nch; ++c) {
            const C* row = sm + (static_cast<size_t>(c) * per_child + static_cast<size_t>(jr) * mph) * 2;
            if (POST) {
                C t0 = zero<C>(), t1 = zero<C>();
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const int q = k * nph + jph;  // tap-major
                    const int s = T.up_ph.src_t[q];
                    const R cf = T.up_ph.coef_t[q];
                    t0 = crfma(cf, row[2 * s], t0);
                    t1 = crfma(cf, row[2 * s + 1], t1);
                }
                const C ph = P.shift_down[static_cast<size_t>(T.child_oct[c0 + c]) * P.ndir + (r0 + jr) * nph + jph];
                a0 = cfma(ph, t0, a0);
                a1 = cfma(ph, t1, a1);
            } else {
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    const int q = k * nph + jph;  // tap-major
                    const int s = T.up_ph.src_t[q];
                    const R cf = T.up_ph.coef_t[q];
                    a0 = crfma(cf, row[2 * s], a0);
                    a1 = crfma(cf, row[2 * s + 1], a1);
                }
            }
        }
        Ap[2 * o] = a0;
        Ap[2 * o + 1] = a1;
    }
}

// ------------------------------------------------------------ M2L
// b_B = w_theta (2 pi / nph) sum_{S in list 2} T[c_B - c_S] a_S
// (Node::buildMpoleToLocalCoeffs, src/fmm/node.cpp:105-134).  One block per
// (level, box, direction chunk) item, all levels in one launch; four list
// entries in flight per thread.
// TR: the transposed translation, T(c_S - c_B) in place of T(c_B - c_S): the
// negated offset, id 315 - id in the order of Math::getINodeDistVecs (the
// offset set is symmetric and listed lexicographically).  Lists 2 are
// symmetric, so the same lists serve.
template <class R, bool TR>
__global__ void __launch_bounds__(128)
k_m2l(const DevLevelT<R>* __restrict__ lvs, const int4* __restrict__ items, int zero_empty) {
    chain_wait();
    using C = typename Cx<R>::T;
    const int4 it = items[blockIdx.x];  // level, box, first direction, count
    if (static_cast<int>(threadIdx.x) >= it.w) return;
    const DevLevelT<R> lv = lvs[it.x];
    const int b = it.y, d = it.z + threadIdx.x, ndir = lv.ndir;
    const int p0 = lv.m2l_ptr[b], p1 = lv.m2l_ptr[b + 1];
    C* Bo = lv.B + (static_cast<size_t>(b) * ndir + d) * 2;
    if (p0 == p1) {
        if (zero_empty) { Bo[0] = zero<C>(); Bo[1] = zero<C>(); }
        return;
    }
    C a0 = zero<C>(), a1 = zero<C>(), c0 = zero<C>(), c1 = zero<C>();
    int p = p0;
    for (; p + 4 <= p1; p += 4) {
        int sb[4], ob[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            sb[u] = lv.m2l_src[p + u];
            ob[u] = TR ? 315 - lv.m2l_off[p + u] : lv.m2l_off[p + u];
        }
        C t[4], xa[4], xb[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            t[u] = lv.transl[static_cast<size_t>(ob[u]) * ndir + d];
            const C* As = lv.A + (static_cast<size_t>(sb[u]) * ndir + d) * 2;
            xa[u] = As[0];
            xb[u] = As[1];
        }
        a0 = cfma(t[0], xa[0], a0);
        a1 = cfma(t[0], xb[0], a1);
        c0 = cfma(t[1], xa[1], c0);
        c1 = cfma(t[1], xb[1], c1);
        a0 = cfma(t[2], xa[2], a0);
        a1 = cfma(t[2], xb[2], a1);
        c0 = cfma(t[3], xa[3], c0);
        c1 = cfma(t[3], xb[3], c1);
    }
    for (; p < p1; ++p) {
        const int s0 = lv.m2l_src[p], o0 = TR ? 315 - lv.m2l_off[p] : lv.m2l_off[p];
        const C t0 = lv.transl[static_cast<size_t>(o0) * ndir + d];
        const C* A0 = lv.A + (static_cast<size_t>(s0) * ndir + d) * 2;
        a0 = cfma(t0, A0[0], a0);
        a1 = cfma(t0, A0[1], a1);
    }
    const R w = lv.w[d];
    Bo[0] = cscale(w, cadd(a0, c0));
    Bo[1] = cscale(w, cadd(a1, c1));
}

// The same translation with the box's list 2 (source boxes, offset ids)
// staged in shared memory first, so the inner loop's loads of patterns and
// transfer values depend on nothing but shared memory and U of them are in
// flight at once.  Bound by operand delivery from L1 and L2: complex float loads
// both components of a pattern at once, and blocks have only the warps their
// run of directions fills (r = 8 sphere, complex float, all levels 498 -> 449 us,
// its 16,344-box level 210 -> 178 us).
constexpr int kM2LStage = 256;  // list entries staged per round (list 2 holds at most 189)

template <class R, bool TR>
__global__ void __launch_bounds__(128)
k_m2l_staged(const DevLevelT<R>* __restrict__ lvs, const int4* __restrict__ items, int zero_empty) {
    chain_wait();
    using C = typename Cx<R>::T;
    constexpr int U = sizeof(R) == 4 ? 8 : 6;
    __shared__ int s_src[kM2LStage], s_off[kM2LStage];
    const int4 it = items[blockIdx.x];  // level, box, first direction, count
    const DevLevelT<R> lv = lvs[it.x];
    const int b = it.y, ndir = lv.ndir;
    const bool live = static_cast<int>(threadIdx.x) < it.w;
    const int d = it.z + (live ? threadIdx.x : 0);
    const int p0 = lv.m2l_ptr[b], p1 = lv.m2l_ptr[b + 1];
    C* Bo = lv.B + (static_cast<size_t>(b) * ndir + d) * 2;
    if (p0 == p1) {
        if (zero_empty && live) { Bo[0] = zero<C>(); Bo[1] = zero<C>(); }
        return;
    }
    C a0 = zero<C>(), a1 = zero<C>(), c0 = zero<C>(), c1 = zero<C>();
    for (int base = p0; base < p1; base += kM2LStage) {
        const int cnt = min(kM2LStage, p1 - base);
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            s_src[i] = lv.m2l_src[base + i];
            const int o = lv.m2l_off[base + i];
            s_off[i] = TR ? 315 - o : o;
        }
        __syncthreads();
        if (!live) continue;
        int p = 0;
        for (; p + U <= cnt; p += U) {
            C t[U], xa[U], xb[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                t[u] = lv.transl[static_cast<size_t>(s_off[p + u]) * ndir + d];
                load_pair(lv.A + (static_cast<size_t>(s_src[p + u]) * ndir + d) * 2, xa[u], xb[u]);
            }
#pragma unroll
            for (int u = 0; u < U; u += 2) {
                a0 = cfma(t[u], xa[u], a0);
                a1 = cfma(t[u], xb[u], a1);
                c0 = cfma(t[u + 1], xa[u + 1], c0);
                c1 = cfma(t[u + 1], xb[u + 1], c1);
            }
        }
        for (; p < cnt; ++p) {
            const C t0 = lv.transl[static_cast<size_t>(s_off[p]) * ndir + d];
            C x0, x1;
            load_pair(lv.A + (static_cast<size_t>(s_src[p]) * ndir + d) * 2, x0, x1);
            a0 = cfma(t0, x0, a0);
            a1 = cfma(t0, x1, a1);
        }
    }
    if (!live) return;
    const R w = lv.w[d];
    store_pair(Bo, cscale(w, cadd(a0, c0)), cscale(w, cadd(a1, c1)));
}

// The complex-double translation for up to four boxes of one parent together.
// Siblings share most of their candidate sources (the children of the parent's
// neighbours), so a warp takes one family of siblings and 16 directions (lane =
// (direction, component)), keeps the targets' sums in registers, loads every
// candidate's pattern once for all of them, and reads the transfer values from
// shared memory, where the block holds all 316 offsets of its directions: per
// (pair, direction) one 16-byte shared-memory read and a fraction of a pattern
// load, in place of a transfer value and a whole pattern from L2.  Block = (run
// of directions, every nsplit-th batch of the level's families); each warp has
// its next family's header and the next 32 candidates in flight while it
// computes, and four or eight patterns ahead.
//
// Bound by shared-memory reads (two wavefronts a pair, four a pattern) and
// instruction issue, so a candidate's transfer rows are staged as shared-memory
// offsets (the row past the table where it is not in a target's list 2, about one
// pair in ten) and the loop is instantiated per number of targets: a shared-memory
// read and four multiply-adds per pair.  Those of the row past the table are
// predicated off (at most 1 % of a product, 8,192 dipoles 121.5 -> 122.8 us): a
// pattern that overflowed may come from a neighbour whose near entries are finite.
// One B200, k_m2l_staged -> this: 8,192 dipoles, level 3 (512 boxes, 392
// directions) 77 -> 48 us; r = 8 sphere, level 6 (16,344 boxes, 162 directions)
// 392 -> 220 us, all levels 932 -> 566 us; r = 2 sphere, levels 3 and 4 27/36 ->
// 23/26 us.  In complex float, whose sums keep their order and run in two halves,
// the same form was issue-bound and no faster (r = 2 sphere, levels 2-4 18/19/22 ->
// 20/26/34 us, r = 8 sphere 498 -> 505 us): complex float keeps k_m2l_staged.
constexpr int kM2LOffsets = 316;
constexpr int kM2LDirs = 16;            // directions per block
constexpr int kM2LRow = kM2LDirs * 16;  // bytes of a row of transfer values
constexpr int kM2LMaxWarps = 12;        // two blocks per SM at 80 registers
constexpr int kM2LPerWarp = 32 * (sizeof(int4) + sizeof(int));  // staged candidates
constexpr size_t m2l_group_smem(int warps) {
    return static_cast<size_t>(kM2LOffsets + 1) * kM2LRow + static_cast<size_t>(warps) * kM2LPerWarp;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

template <bool TR>
__global__ void __launch_bounds__(32 * kM2LMaxWarps, 2)
k_m2l_group(const DevLevelT<double>* __restrict__ lvs, int level, const DevM2LFamily* __restrict__ fams, int nfam,
            const int2* __restrict__ cand_off, const int* __restrict__ cand_src, int nchunk, int zero_empty) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char smraw[];
    double2* tsm = reinterpret_cast<double2*>(smraw);  // [316 + 1][kM2LDirs], the last row zero
    const int nwarp = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* cand = smraw + (kM2LOffsets + 1) * kM2LRow;
    int4* soff = reinterpret_cast<int4*>(cand) + warp * 32;
    int* ssrc = reinterpret_cast<int*>(cand + sizeof(int4) * 32 * nwarp) + warp * 32;
    const DevLevelT<double> lv = lvs[level];
    const int ndir = lv.ndir;
    const int chunk = blockIdx.x % nchunk, split = blockIdx.x / nchunk, nsplit = gridDim.x / nchunk;
    const int d0 = chunk * kM2LDirs, dn = min(kM2LDirs, ndir - d0);
    for (int i = threadIdx.x; i < kM2LOffsets * kM2LDirs; i += blockDim.x) {
        const int o = i / kM2LDirs, q = i - o * kM2LDirs;
        if (q < dn) cp_async16(tsm + i, lv.transl + static_cast<size_t>(TR ? kM2LOffsets - 1 - o : o) * ndir + d0 + q);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (threadIdx.x < kM2LDirs) tsm[kM2LOffsets * kM2LDirs + threadIdx.x] = z0();
    const int dl = min(lane >> 1, dn - 1), comp = lane & 1;
    const bool live = (lane >> 1) < dn;
    const int d = d0 + dl;
    const double w = lv.w[d];
    const unsigned char* tl = reinterpret_cast<const unsigned char*>(tsm + dl);
    const double2* Al = lv.A + 2 * static_cast<size_t>(d) + comp;
    const size_t astride = 2 * static_cast<size_t>(ndir);
    // families largest first: neighbouring warps take families of one parent
    // (two at a time), blocks take them in turn
    const int step = nsplit * nwarp, nw2 = nwarp & ~1;
    int f = warp < nw2 ? 2 * ((warp >> 1) * nsplit + split) + (warp & 1) : nw2 * nsplit + split;
    const int* hdr = reinterpret_cast<const int*>(fams);
    constexpr int HW = sizeof(DevM2LFamily) / sizeof(int);
    static_assert(HW == 8 && kM2LFamily == 4, "a family header is one word per lane of a quarter warp");
    int hv = f < nfam ? hdr[static_cast<size_t>(f) * HW + (lane & 7)] : 0;
    int hn = 0;
    int2 co = make_int2(-1, -1);
    int cs = 0;
    auto fetch = [&](int h, int c0) {  // this lane's candidate of the batch at c0
        const int cand0 = __shfl_sync(0xffffffffu, h, 6), n = __shfl_sync(0xffffffffu, h, 7);
        const int c = min(c0 + lane, n - 1);
        co = make_int2(-1, -1);
        cs = 0;
        if (c >= 0) cs = cand_src[cand0 + c];
        if (c0 + lane < n) co = cand_off[cand0 + c];
    };
    auto row = [](int o) { return (o < 0 ? kM2LOffsets : o) * kM2LRow; };
    auto family = [&](auto nt) {  // one family of NT targets
        constexpr int NT = decltype(nt)::value;
        constexpr int U = NT > 2 ? 4 : 8;  // patterns loaded ahead
        double2 acc[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t] = z0();
        const int ncand = __shfl_sync(0xffffffffu, hv, 7);
        for (int c0 = 0; c0 < ncand; c0 += 32) {
            __syncwarp();
            soff[lane] = make_int4(row(static_cast<short>(co.x & 0xffff)), row(co.x >> 16),
                                   row(static_cast<short>(co.y & 0xffff)), row(co.y >> 16));
            ssrc[lane] = cs;
            __syncwarp();
            if (c0 + 32 < ncand) fetch(hv, c0 + 32); else fetch(hn, 0);
            const int nb = min(32, ncand - c0);
            double2 a[U], an[U];
#pragma unroll
            for (int u = 0; u < U; ++u) a[u] = Al[ssrc[u] * astride];
            for (int i = 0; i < nb; i += U) {
#pragma unroll
                for (int u = 0; u < U; ++u) an[u] = Al[ssrc[(i + U + u) & 31] * astride];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int4 o4 = soff[i + u];  // (past the list's end: in no target's list)
                    const int o[4] = {o4.x, o4.y, o4.z, o4.w};
                    double2 tv[NT];
#pragma unroll
                    for (int t = 0; t < NT; ++t) tv[t] = *reinterpret_cast<const double2*>(tl + o[t]);
#pragma unroll
                    for (int t = 0; t < NT; ++t)
                        if (o[t] != kM2LOffsets * kM2LRow) acc[t] = cfma(tv[t], a[u], acc[t]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) a[u] = an[u];
            }
        }
        if (ncand == 0) fetch(hn, 0);
        const int empty = __shfl_sync(0xffffffffu, hv, 5);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int box = __shfl_sync(0xffffffffu, hv, t);
            const bool none = (empty >> t) & 1;
            // (an empty list under the reference's rule: kept from the previous product)
            if (live && (!none || zero_empty))
                lv.B[(static_cast<size_t>(box) * ndir + d) * 2 + comp] = none ? z0() : cscale(w, acc[t]);
        }
    };
    fetch(hv, 0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the transfer values
    for (; f < nfam; f += step) {
        const int fn = f + step;
        hn = fn < nfam ? hdr[static_cast<size_t>(fn) * HW + (lane & 7)] : 0;
        switch (__shfl_sync(0xffffffffu, hv, 4)) {
            case 1: family(std::integral_constant<int, 1>()); break;
            case 2: family(std::integral_constant<int, 2>()); break;
            case 3: family(std::integral_constant<int, 3>()); break;
            default: family(std::integral_constant<int, 4>()); break;
        }
        hv = hn;
    }
}

// ------------------------------------------------------------ L2L
// child local += Anterp[shift(parent local)]: shift on the parent grid, then
// the transposed phi pass, then the transposed theta pass with pole
// reflection (Stem::getShiftedLocalCoeffs and addAnterpCoeffs,
// src/fmm/stem.cpp:109-244).  One block per (parent, child) pair; the
// pair list already omits parents that pass nothing down.
// POST: the transposed M2M -- no shift before the phi pass; the anterpolated
// pattern is multiplied by the child-grid shift of the child's octant
// (shift_up of the child level) as it is added to the child.
template <class R, int W, bool POST>  // both transposed stencils padded to W taps per row
__global__ void __launch_bounds__(256)
k_l2l(const DevLevelT<R>* __restrict__ lvs, DevTransT<R> T, const int2* __restrict__ pairs) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ unsigned char smraw[];
    C* sm = reinterpret_cast<C*>(smraw);
    const int2 pc = pairs[blockIdx.x];  // parent index, child entry
    const DevLevelT<R> P = lvs[T.plevel];
    const DevLevelT<R> Cl = lvs[T.plevel + 1];
    const int pth = P.nth, pph = P.nph, cth = Cl.nth, cph = Cl.nph, halfc = Cl.nph / 2;
    const C* Bp = P.B + static_cast<size_t>(T.par_box[pc.x]) * P.ndir * 2;
    const C* sh = P.shift_down + static_cast<size_t>(T.child_oct[pc.y]) * P.ndir;
    for (int e = threadIdx.x; e < pth * cph; e += blockDim.x) {
        const int ith = e / cph, jph = e - ith * cph;
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int q = k * cph + jph;  // tap-major
            const int d = ith * pph + T.dn_ph.src_t[q];
            const R cf = T.dn_ph.coef_t[q];
            if (POST) {
                v0 = crfma(cf, Bp[2 * d], v0);
                v1 = crfma(cf, Bp[2 * d + 1], v1);
            } else {
                const C ph = sh[d];
                v0 = crfma(cf, cmul(ph, Bp[2 * d]), v0);
                v1 = crfma(cf, cmul(ph, Bp[2 * d + 1]), v1);
            }
        }
        sm[2 * e] = v0;
        sm[2 * e + 1] = v1;
    }
    __syncthreads();
    C* Bc = Cl.B + static_cast<size_t>(T.child_box[pc.y]) * Cl.ndir * 2;
    for (int e = threadIdx.x; e < cth * cph; e += blockDim.x) {
        const int jth = e / cph, jph = e - jth * cph;
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int q = jth * W + k;
            const bool rf = T.dn_th.refl[q];
            const int sp = rf ? (jph < halfc ? jph + halfc : jph - halfc) : jph;
            const R cf = T.dn_th.coef[q];
            const C* row = sm + (static_cast<size_t>(T.dn_th.src[q]) * cph + sp) * 2;
            v0 = crfma(cf, row[0], v0);
            v1 = crfma(cf, row[1], v1);
        }
        if (POST) {
            const C ph = Cl.shift_up[static_cast<size_t>(T.child_oct[pc.y]) * Cl.ndir + e];
            v0 = cmul(ph, v0);
            v1 = cmul(ph, v1);
        }
        Bc[2 * e] = cadd(Bc[2 * e], v0);
        Bc[2 * e + 1] = cadd(Bc[2 * e + 1], v1);
    }
}

// ------------------------------------------------------------ staged interpolation
// M2M with the children shifted and summed on the child grid first:
// U = sum_c shift_up(oct_c) A_c over the child theta rows the block's
// stencils read, then the theta pass (pole reflection as in k_m2m) into V,
// then the phi pass to the parent.  Interpolation is linear and the same for
// every child, so this is k_m2m's sum in another order (one interpolation per
// parent instead of one per child).  Block = (parent, tile of `rows` parent
// theta rows); each child value is read from global memory once per block and
// every stencil tap reads shared memory.
//
// Latency-bound: a block's life is its chain of dependent loads and its
// barriers.  Grid sizes come with the launch, children as pointers, both
// stencils are staged in shared memory while the children's values are on their
// way, and every warp finds the band of child rows by itself.  With level
// descriptors read by each block, shared atomics for the band and the stencils
// from global memory: 181 against 173 us (complex float, sphere of radius 8
// wavelengths, five transitions), 24 against 21.6 us (FP64, radius 2).
template <class R, int W, bool CS>  // taps per row: 2 * interp_order (both passes); CS: column-stationary phi pass
__global__ void __launch_bounds__(256)
k_m2m_sum(DevTransT<R> T, int rows) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int par = blockIdx.x;
    const int nph = T.pph, mph = T.cph, halfm = T.cph / 2;
    const int r0 = blockIdx.y * rows;
    const int nrow = min(T.pth, r0 + rows) - r0;
    if (nrow <= 0) return;  // the whole block
    const int c0 = T.child_ptr[par], nch = T.child_ptr[par + 1] - c0;
    C* Ap = T.par_a[par] + static_cast<size_t>(r0) * nph * 2;
    int lo = T.cth, hi = -1;
    for (int q = threadIdx.x & 31; q < nrow * W; q += 32) {
        const int src = T.up_th.src[r0 * W + q];
        lo = min(lo, src);
        hi = max(hi, src);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    const int nb = hi - lo + 1;
    // component planes (theta, phi), so that neighbouring threads read
    // neighbouring 8- or 16-byte words of shared memory
    const size_t nu = static_cast<size_t>(nb) * mph, nv = static_cast<size_t>(nrow) * mph;
    C* U0 = reinterpret_cast<C*>(smraw);  // [nb * mph], child rows lo..lo+nb-1
    C* U1 = U0 + nu;
    C* V0 = U1 + nu;                      // [nrow * mph]
    C* V1 = V0 + nv;
    R* th_cf = reinterpret_cast<R*>(V1 + nv);          // [nrow * W], then phi [W * nph] (tap-major)
    R* ph_cf = th_cf + nrow * W;
    int* th_src = reinterpret_cast<int*>(ph_cf + W * nph);  // row, reflected in bit 30
    int* ph_src = th_src + nrow * W;
    for (int e = threadIdx.x; e < nb * mph; e += blockDim.x) {
        const int d = lo * mph + e;
        C u0 = zero<C>(), u1 = zero<C>();
#pragma unroll 8
        for (int c = 0; c < nch; ++c) {
            const C ph = T.child_up[c0 + c][d];
            C x0, x1;
            load_pair(T.child_a[c0 + c] + 2 * d, x0, x1);
            u0 = cfma(ph, x0, u0);
            u1 = cfma(ph, x1, u1);
        }
        U0[e] = u0;
        U1[e] = u1;
    }
    for (int q = threadIdx.x; q < nrow * W; q += blockDim.x) {
        th_cf[q] = T.up_th.coef[r0 * W + q];
        th_src[q] = (T.up_th.src[r0 * W + q] - lo) | (T.up_th.refl[r0 * W + q] ? 1 << 30 : 0);
    }
    for (int q = threadIdx.x; q < W * nph; q += blockDim.x) {
        ph_cf[q] = T.up_ph.coef_t[q];
        ph_src[q] = T.up_ph.src_t[q];
    }
    __syncthreads();
    for (int it = threadIdx.x; it < nrow * mph; it += blockDim.x) {
        const int jr = it / mph, iph = it - jr * mph;
        const int iref = iph < halfm ? iph + halfm : iph - halfm;
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int q = th_src[jr * W + k];
            const R cf = th_cf[jr * W + k];
            const int e = (q & ~(1 << 30)) * mph + (q >> 30 ? iref : iph);
            v0 = crfma(cf, U0[e], v0);
            v1 = crfma(cf, U1[e], v1);
        }
        V0[it] = v0;
        V1[it] = v1;
    }
    __syncthreads();
    if (!CS) {  // one output per thread, stencil read per tap (tap-major)
        for (int o = threadIdx.x; o < nrow * nph; o += blockDim.x) {
            const int jr = o / nph, jph = o - jr * nph;
            const C* row0 = V0 + static_cast<size_t>(jr) * mph;
            const C* row1 = V1 + static_cast<size_t>(jr) * mph;
            C a0 = zero<C>(), a1 = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const int q = k * nph + jph;
                const int s = ph_src[q];
                const R cf = ph_cf[q];
                a0 = crfma(cf, row0[s], a0);
                a1 = crfma(cf, row1[s], a1);
            }
            store_pair(Ap + 2 * o, a0, a1);
        }
        return;
    }
    // phi pass, column-stationary: a thread keeps one output column's stencil
    // in registers and walks the tile's rows (every row uses the same stencil)
    const int ng = max(1, static_cast<int>(blockDim.x) / nph);  // row groups
    for (int t = threadIdx.x; t < nph * ng; t += blockDim.x) {
        const int jph = t % nph, g = t / nph;
        int sk[W];
        R ck[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            sk[k] = ph_src[k * nph + jph];
            ck[k] = ph_cf[k * nph + jph];
        }
        for (int jr = g; jr < nrow; jr += ng) {
            const C* row0 = V0 + static_cast<size_t>(jr) * mph;
            const C* row1 = V1 + static_cast<size_t>(jr) * mph;
            C a0 = zero<C>(), a1 = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                a0 = crfma(ck[k], row0[sk[k]], a0);
                a1 = crfma(ck[k], row1[sk[k]], a1);
            }
            const int o = jr * nph + jph;
            store_pair(Ap + 2 * o, a0, a1);
        }
    }
}

// L2L (and, POST, the transposed M2M) with the parent's local pattern, shifted
// to the child's octant, staged in shared memory once per block: the same
// arithmetic in the same order as k_l2l, every phi tap then reading shared
// memory instead of global memory.  One block per (parent, child) pair.
//
// Latency-bound as k_m2m_sum: one load finds a pair's pointers, the stencils are
// staged beside the parent's values, and the child's pattern is requested before
// the last pass.  Without these (level descriptor, pair, box and octant read one
// after the other): 337 against 288 us (complex float, sphere of radius 8
// wavelengths, five transitions), 38 against 31.7 us (FP64, radius 2).
template <class R, int W, bool POST, bool CS>  // both transposed stencils padded to W taps per row
__global__ void __launch_bounds__(256)
k_l2l_st(DevTransT<R> T) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ __align__(16) unsigned char smraw[];
    const DevL2LItem<R> it = T.l2l[blockIdx.x];
    const int pth = T.pth, pph = T.pph, cth = T.cth, cph = T.cph, halfc = T.cph / 2;
    // component planes (theta, phi): neighbouring threads read neighbouring words
    const size_t np = static_cast<size_t>(pth) * pph, nq = static_cast<size_t>(pth) * cph;
    C* SB0 = reinterpret_cast<C*>(smraw);  // [pth * pph]
    C* SB1 = SB0 + np;
    C* S10 = SB1 + np;                     // [pth * cph]
    C* S11 = S10 + nq;
    R* ph_cf = reinterpret_cast<R*>(S11 + nq);              // [W * cph] (tap-major), then theta [cth * W]
    R* th_cf = ph_cf + W * cph;
    int* ph_src = reinterpret_cast<int*>(th_cf + cth * W);
    int* th_src = ph_src + W * cph;                         // row, reflected in bit 30
    for (int d = threadIdx.x; d < pth * pph; d += blockDim.x) {
        C b0, b1;
        load_pair(it.parent + 2 * d, b0, b1);
        if (!POST) {
            const C ph = it.down[d];
            b0 = cmul(ph, b0);
            b1 = cmul(ph, b1);
        }
        SB0[d] = b0;
        SB1[d] = b1;
    }
    for (int q = threadIdx.x; q < W * cph; q += blockDim.x) {
        ph_cf[q] = T.dn_ph.coef_t[q];
        ph_src[q] = T.dn_ph.src_t[q];
    }
    for (int q = threadIdx.x; q < cth * W; q += blockDim.x) {
        th_cf[q] = T.dn_th.coef[q];
        th_src[q] = T.dn_th.src[q] | (T.dn_th.refl[q] ? 1 << 30 : 0);
    }
    __syncthreads();
    if (!CS) {  // one output per thread, stencil read per tap (tap-major)
        for (int e = threadIdx.x; e < pth * cph; e += blockDim.x) {
            const int ith = e / cph, jph = e - ith * cph;
            const C* row0 = SB0 + static_cast<size_t>(ith) * pph;
            const C* row1 = SB1 + static_cast<size_t>(ith) * pph;
            C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const int d = ph_src[k * cph + jph];
                const R cf = ph_cf[k * cph + jph];
                v0 = crfma(cf, row0[d], v0);
                v1 = crfma(cf, row1[d], v1);
            }
            S10[e] = v0;
            S11[e] = v1;
        }
    }
    // phi pass, column-stationary: a thread keeps one child column's stencil in
    // registers and walks the parent's theta rows (the same stencil for each)
    const int ng = CS ? max(1, static_cast<int>(blockDim.x) / cph) : 0;  // row groups
    for (int t = threadIdx.x; t < cph * ng; t += blockDim.x) {
        const int jph = t % cph, g = t / cph;
        int sk[W];
        R ck[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            sk[k] = ph_src[k * cph + jph];
            ck[k] = ph_cf[k * cph + jph];
        }
        for (int ith = g; ith < pth; ith += ng) {
            const C* row0 = SB0 + static_cast<size_t>(ith) * pph;
            const C* row1 = SB1 + static_cast<size_t>(ith) * pph;
            C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                v0 = crfma(ck[k], row0[sk[k]], v0);
                v1 = crfma(ck[k], row1[sk[k]], v1);
            }
            S10[ith * cph + jph] = v0;
            S11[ith * cph + jph] = v1;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < cth * cph; e += blockDim.x) {
        const int jth = e / cph, jph = e - jth * cph;
        const int jref = jph < halfc ? jph + halfc : jph - halfc;
        C c0, c1;  // the child's local pattern, in flight during the taps
        load_pair(it.child + 2 * e, c0, c1);
        C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int q = th_src[jth * W + k];
            const R cf = th_cf[jth * W + k];
            const int at = (q & ~(1 << 30)) * cph + (q >> 30 ? jref : jph);
            v0 = crfma(cf, S10[at], v0);
            v1 = crfma(cf, S11[at], v1);
        }
        if (POST) {
            const C ph = it.up[e];
            v0 = cmul(ph, v0);
            v1 = cmul(ph, v1);
        }
        store_pair(it.child + 2 * e, cadd(c0, v0), cadd(c1, v1));
    }
}

// The staged L2L as a persistent, software-pipelined kernel: each block walks
// the pairs blockIdx.x, blockIdx.x + gridDim.x, ... and, while it computes one
// pair, the next pair's parent pattern, shift and child local pattern arrive by
// asynchronous copies (cp.async, 8 or 16 bytes per copy) into the other half of
// a double buffer; the child's updated local is written with plain stores.
// Same arithmetic in the same order as k_l2l_st<..., false>.
__device__ __forceinline__ void cp_async_elem(void* dst, const void* src, int bytes) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if (bytes == 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

template <class R, int W, bool POST>
__global__ void __launch_bounds__(256)
k_l2l_pipe(const DevLevelT<R>* __restrict__ lvs, DevTransT<R> T, const int2* __restrict__ pairs, int npairs) {
    chain_wait();
    using C = typename Cx<R>::T;
    extern __shared__ __align__(16) unsigned char smraw[];
    const DevLevelT<R> P = lvs[T.plevel];
    const DevLevelT<R> Cl = lvs[T.plevel + 1];
    const int pth = P.nth, pph = P.nph, cth = Cl.nth, cph = Cl.nph, halfc = Cl.nph / 2;
    const int np = pth * pph, nq = pth * cph, nc = cth * cph;
    const int nsh = POST ? nc : np;  // shift values: parent grid (before) or child grid (after, POST)
    // per buffer: raw parent [2 np] (interleaved, as stored), shift [nsh], child [2 nc]
    const size_t per_buf = 2 * static_cast<size_t>(np) + nsh + 2 * static_cast<size_t>(nc);
    C* buf0 = reinterpret_cast<C*>(smraw);
    C* SB0 = buf0 + 2 * per_buf;  // planes [np] x 2, then S1 planes [nq] x 2
    C* SB1 = SB0 + np;
    C* S10 = SB1 + np;
    C* S11 = S10 + nq;
    auto issue = [&](int pi, int b) {
        const int2 pc = pairs[pi];
        C* raw = buf0 + b * per_buf;
        C* shv = raw + 2 * np;
        C* cl = shv + nsh;
        const C* Bp = P.B + static_cast<size_t>(T.par_box[pc.x]) * P.ndir * 2;
        const C* sh = POST ? Cl.shift_up + static_cast<size_t>(T.child_oct[pc.y]) * Cl.ndir
                           : P.shift_down + static_cast<size_t>(T.child_oct[pc.y]) * P.ndir;
        const C* Bc = Cl.B + static_cast<size_t>(T.child_box[pc.y]) * Cl.ndir * 2;
        for (int i = threadIdx.x; i < 2 * np; i += blockDim.x) cp_async_elem(raw + i, Bp + i, sizeof(C));
        for (int i = threadIdx.x; i < nsh; i += blockDim.x) cp_async_elem(shv + i, sh + i, sizeof(C));
        for (int i = threadIdx.x; i < 2 * nc; i += blockDim.x) cp_async_elem(cl + i, Bc + i, sizeof(C));
    };
    int b = 0;
    if (static_cast<int>(blockIdx.x) < npairs) issue(blockIdx.x, 0);
    cp_async_commit();
    for (int pi = blockIdx.x; pi < npairs; pi += gridDim.x, b ^= 1) {
        const int nxt = pi + gridDim.x;
        if (nxt < npairs) issue(nxt, b ^ 1);
        cp_async_commit();  // (possibly empty) group, so that wait_group 1 means "this pair"
        cp_async_wait1();
        __syncthreads();
        const C* raw = buf0 + b * per_buf;
        const C* shv = raw + 2 * np;
        const C* cl = shv + nsh;
        for (int d = threadIdx.x; d < np; d += blockDim.x) {
            C b0 = raw[2 * d], b1 = raw[2 * d + 1];
            if (!POST) {
                const C ph = shv[d];
                b0 = cmul(ph, b0);
                b1 = cmul(ph, b1);
            }
            SB0[d] = b0;
            SB1[d] = b1;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nq; e += blockDim.x) {
            const int ith = e / cph, jph = e - ith * cph;
            const C* row0 = SB0 + static_cast<size_t>(ith) * pph;
            const C* row1 = SB1 + static_cast<size_t>(ith) * pph;
            C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const int q = k * cph + jph;
                const int d = T.dn_ph.src_t[q];
                const R cf = T.dn_ph.coef_t[q];
                v0 = crfma(cf, row0[d], v0);
                v1 = crfma(cf, row1[d], v1);
            }
            S10[e] = v0;
            S11[e] = v1;
        }
        __syncthreads();
        const int2 pc = pairs[pi];
        C* Bc = Cl.B + static_cast<size_t>(T.child_box[pc.y]) * Cl.ndir * 2;
        for (int e = threadIdx.x; e < nc; e += blockDim.x) {
            const int jth = e / cph, jph = e - jth * cph;
            C v0 = zero<C>(), v1 = zero<C>();
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const int q = jth * W + k;
                const bool rf = T.dn_th.refl[q];
                const int sp = rf ? (jph < halfc ? jph + halfc : jph - halfc) : jph;
                const R cf = T.dn_th.coef[q];
                const size_t at = static_cast<size_t>(T.dn_th.src[q]) * cph + sp;
                v0 = crfma(cf, S10[at], v0);
                v1 = crfma(cf, S11[at], v1);
            }
            if (POST) {
                const C ph = shv[e];
                v0 = cmul(ph, v0);
                v1 = cmul(ph, v1);
            }
            Bc[2 * e] = cadd(cl[2 * e], v0);
            Bc[2 * e + 1] = cadd(cl[2 * e + 1], v1);
        }
        __syncthreads();  // buffers and planes free for the next pair
    }
}

inline size_t l2l_pipe_smem(int pth, int pph, int cth, int cph, size_t csize) {
    const size_t np = static_cast<size_t>(pth) * pph, nc = static_cast<size_t>(cth) * cph;
    const size_t per_buf = 2 * np + std::max(np, nc) + 2 * nc;
    return (2 * per_buf + 2 * np + 2 * static_cast<size_t>(pth) * cph) * csize;
}

template <class R>
size_t l2l_st_smem(int parent_nth, int parent_nph, int child_nth, int child_nph, int w) {
    return static_cast<size_t>(parent_nth) * (parent_nph + child_nph) * 2 * sizeof(typename Cx<R>::T) +
           static_cast<size_t>(child_nph + child_nth) * w * (sizeof(R) + sizeof(int));
}

// Complex double -> far-field type (patterns, tables at setup).
template <class C>
__global__ void k_narrow(const double2* __restrict__ src, C* __restrict__ dst, long long n) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = from_d2<C>(src[i]);
}

}  // namespace
}  // namespace mlfma
