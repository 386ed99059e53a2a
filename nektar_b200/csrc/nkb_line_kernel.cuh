// Line kernels: the element operators with one thread per grid line.
//
// A one-dimensional contraction (basis to points, points to basis, the
// collocation derivative and its transpose) is done by a thread that loads one
// whole line of the element into registers, multiplies it by the 1-D table and
// stores the whole result line. The tables are kernel parameters and every
// index into them is a compile-time constant, so the n*n multiply-adds of a
// line cost n loads and n stores of shared memory and no table traffic; a
// thread that computes one output per dot product (the shape-generic kernel)
// loads 2n values for n multiply-adds.
//
// That holds for every stage of a hexahedron, every derivative, and the first
// direction of the collapsed shapes (and a prism's second). Their third
// direction's table depends on (p, q): a thread keeps one column (or row) of it
// in registers, walks the CTA's elements, and takes one shared load per
// multiply-add. A tetrahedron's second direction depends on p, which differs
// between a warp's lanes: its table entries are global loads (L1), one per
// multiply-add.
//
// What bounds the operators: HBM for curved hexahedra in FP64 (Helmholtz at 0.72 of
// the copy rate in long runs under the power cap, 0.82 in short ones, PhysDeriv
// 0.81), instruction issue in FP32 (79 %), the
// L1/shared pipe for prisms and tetrahedra (70 to 81 %).
//
// Directions. A kernel has a register direction (0) and two lane directions
// (1, and 2 fastest). Hexahedra, and PhysDeriv on every shape, take the mesh's
// third direction as 0, so that a warp's lanes follow the arrays' fastest
// direction and physical arrays go between global memory and registers
// without staging. Prisms and tetrahedra with a basis must expand the mesh's
// first direction last (the triangular truncation couples the others), so
// they take it as 0, and the Helmholtz-like ones read geometry packed with
// the third direction fastest (nkb_op::geo_perm).
//
// Straight-sided elements have one Jacobian and one set of derivative
// factors: 16 values per element (geoc), the weights and collapsed-coordinate
// factors being products of 1-D tables, instead of 1 to 10 values per point.
// FP32 operators apply them in FP64 and round the results, or (Helmholtz,
// LinearADR) read factors per point that were formed in FP64 and rounded once:
// formed in FP32 they put results up to 11 % further from the FP64 ones (tet
// LinearADR, 4 modes). Of the two, FP64 arithmetic is the quicker where a point
// takes nine factors (IProductWRTDerivBase, tet 8 modes x 37202: 206 us, factors
// 229; in FP32 235), factors where it takes seven or ten (Helmholtz, prism 7 modes
// x 47831: 204, FP64 219, in FP32 200; tets of 8 modes alone 284, 245 and 221).
//
// The collapsed-vertex and singular-edge terms of BwdTransKernels.hpp:231-403
// and IProductKernels.hpp:355-655 are folded into the first stage: with A_p,
// B_pq the tabulated modes, a prism's singular-edge mode (0, q, 1) has
// A_0 + A_1 = 1 in place of A_0, i.e. its line is added to that of (1, q); a
// tetrahedron's (0, 0, 1) has (A_0 + A_1)(B_00 + B_01), and (0, 1, r) has
// (A_0 + A_1) B_01, i.e. its lines are added to (0, 1), (1, 0) and to one more
// line of p = 1 whose table row is B_01 (kept in the unused slot (1, nm-1)).
//
// Measured on a B200 (us per call, FP64, before -> with the first line kernels; a
// shared-memory layout without conflicts, shared index work and the geometry's
// prefetch came later): prism
// BwdTrans 5 modes x 13718 elements 70.6 -> 21.2; hexahedral IProduct 4 modes at 8
// points x 10648 82 -> 23.6; straight-sided tet IProductWRTDerivBase 5 modes x
// 24576 145.9 -> 55.6; hexahedral PhysDeriv 8 points x 13824 189 -> 163; curved tet
// Helmholtz 7 modes x 10368 152.7 -> 92.9; straight-sided prism Helmholtz 6 modes x
// 11664 106 -> 54.3 (the first four ran on the shape-generic kernel, the last two on
// kernels with a thread per (i, j) column and one dot product per output).
#pragma once

#include "nkb_internal.h"
#include "nkb_op.h"
#include "nkb_tma.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <vector>

namespace nkb
{

enum
{
    LN_BWD  = 0,
    LN_IP   = 1,
    LN_PD   = 2,
    LN_IPD  = 3,
    LN_HELM = 4,
    LN_ADR  = 5
};

constexpr int kGeoc = 16; // values per straight-sided element: J, J (F K F^T)
                          // (00 11 22 01 02 12), df[k*3+j]

template <typename T> struct LineArgs
{
    const T *in, *in1, *in2;
    T *out0, *out1, *out2;
    const T *geo;       // packed [e][c][nt], element stride gstride (curved)
    const double *geoc; // [e][kGeoc] (straight-sided), else NULL
    const T *tB1;  // Tet Modified_B table [(p,q)][j]
    const T *tB2;  // Prism Modified_B [(p,r)][k], Tet Modified_C [(p,q,r)][k]
    const T *tC;   // the table row of every coefficient, [k][coefficient]
    const unsigned *pairs; // Tet (p, q): p | q << 4 | modes << 8 | first << 12
    const unsigned *coefs; // of every coefficient: p | q << 4 | fold << 8
    const int *gmap;
    const double *gsign;
    const int *skip;
    long gstride;
    T lambda;
    int nelmt, nm;
    int epb; // elements per CTA of this launch
    const uint2 *lanes; // each thread's lines along directions 1 and 2 (DEALT kernels):
                        // offset | x << 16 | y << 20 | element << 24
};

// ---- shared-memory layout ------------------------------------------------
// A cube's entry (a, b, c) sits at a*ps + b*k2 + c, elements `cube` apart. Lines
// along a are walked by lanes (b, c) in the arrays' order. Which lane walks which
// line along b (a line per (a, c)) or c (per (a, b)) is free: a table
// (LineLanes) deals them out so that the lanes of one shared-memory phase (16
// in FP64, 32 in FP32) start in different banks. The strides are those for which
// the lines spread most evenly over the banks. A row of 4 or 8 entries may
// instead be rotated by the exclusive-or of c with b, with lanes in line order,
// where that needs fewer wavefronts (e.g. 8 points: none in conflict).
struct LineLayout
{
    int ps, cube;
    bool rotate;
};

// wavefronts of one access by all of a CTA's lanes, lines (x, y) in order:
// entry 0 at e*cube + x*sx + y*sy, entry p of a rotated layout at the address
// that `kind` (0, 1, 2: lines along a, b, c) gives
constexpr int LineOrdered(int kind, int k0, int k1, int k2, int epb, int banks, LineLayout l)
{
    const int n1 = kind == 0 ? k1 : k0, n2 = kind == 2 ? k1 : k2;
    const int len = kind == 0 ? k0 : (kind == 1 ? k1 : k2);
    const int pos = l.rotate ? len : 1; // otherwise every entry as the first
    int total     = 0;
    for (int p = 0; p < pos; ++p)
        for (int t0 = 0; t0 < epb * n1 * n2; t0 += banks)
        {
            int hits[32] = {};
            int worst    = 0;
            for (int t = t0; t < t0 + banks && t < epb * n1 * n2; ++t)
            {
                const int e = t / (n1 * n2), x = t / n2 % n1, y = t % n2;
                const int a = kind == 0 ? p : x, b = kind == 0 ? x : (kind == 1 ? p : y);
                const int c = kind == 2 ? p : y;
                const int at =
                    e * l.cube + a * l.ps + b * k2 + (l.rotate ? (c ^ (b & (k2 - 1))) : c);
                if (++hits[at % banks] > worst)
                    worst = hits[at % banks];
            }
            total += worst;
        }
    return (total + pos - 1) / pos;
}

struct LineCounts
{
    int n[32];
};

// lines of one element per starting bank
constexpr LineCounts LineBanks(int n1, int s1, int n2, int s2, int banks)
{
    LineCounts h = {};
    for (int x = 0; x < n1; ++x)
        for (int y = 0; y < n2; ++y)
            ++h.n[(x * s1 + y * s2) % banks];
    return h;
}

// wavefronts when the CTA's lines are dealt out by bank over `th` lanes
constexpr int LineDealt(const LineCounts &h, int shift, int epb, int banks, int th)
{
    const int phases = th / banks;
    int most = 0, over = 0;
    for (int b = 0; b < banks; ++b)
    {
        int n = 0;
        for (int e = 0; e < epb; ++e)
            n += h.n[(b + (banks - shift) * e) % banks];
        most = n > most ? n : most;
        over += n > phases ? n - phases : 0;
    }
    return (most < phases ? most : phases) + over;
}

// About the accesses of the Helmholtz operator per line and direction. The other
// operators' layouts follow them too: with equal weights, FP64 BwdTrans, IProduct,
// IProductWRTDerivBase and PhysDeriv of 3 to 10 modes took 0.92 to 1.05 of the
// time, within 1 % at 123 of 144 sizes.
constexpr int LineCost(int r, int b, int c, int k0, int k1, int k2)
{
    return 8 * k0 * r + 7 * k1 * b + 6 * k2 * c;
}

constexpr LineLayout LineFind(int k0, int k1, int k2, int epb, int th, int banks, int least,
                              bool deal)
{
    LineLayout best = {};
    int cost        = 1 << 30;
    if (k2 == 4 || k2 == 8)
    {
        const int ps = k1 * k2 + k2;
        best         = {ps, ((k0 * ps > least ? k0 * ps : least) + 7) & ~7, true};
        cost         = LineCost(LineOrdered(0, k0, k1, k2, epb, banks, best),
                                LineOrdered(1, k0, k1, k2, epb, banks, best),
                                LineOrdered(2, k0, k1, k2, epb, banks, best), k0, k1, k2);
    }
    int r[32] = {};
    for (int shift = 0; shift < banks; ++shift)
        r[shift] = LineOrdered(0, k0, k1, k2, epb, banks, {0, shift, false});
    for (int pad = 0; pad < 16; ++pad)
    {
        const int ps  = k1 * k2 + pad;
        const auto hb = LineBanks(k0, ps, k2, 1, banks), hc = LineBanks(k0, ps, k1, k2, banks);
        const int min = k0 * ps > least ? k0 * ps : least;
        for (int add = 0; add < (epb > 1 ? (deal ? banks : 8) : 1); ++add)
        {
            const int shift    = (min + add) % banks;
            const LineLayout l = {ps, min + add, false};
            const int c =
                LineCost(r[shift],
                         deal ? LineDealt(hb, shift, epb, banks, th)
                              : LineOrdered(1, k0, k1, k2, epb, banks, l),
                         deal ? LineDealt(hc, shift, epb, banks, th)
                              : LineOrdered(2, k0, k1, k2, epb, banks, l), k0, k1, k2);
            if (c < cost)
            {
                cost = c;
                best = {ps, min + add, false};
            }
        }
    }
    return best;
}

// one search per set of sizes, whatever the operator
template <int K0, int K1, int K2, int EPB, int TH, int BANKS, int LEAST, bool DEAL>
struct LineLayoutOf
{
    static constexpr LineLayout V = LineFind(K0, K1, K2, EPB, TH, BANKS, LEAST, DEAL);
};

template <int SHAPE, int NM, int NQ, int OP, typename T> struct LineDims
{
    // the modes per direction: NM, or with more points than nm + 1 (over-
    // integration) a run-time count up to NM
    static constexpr bool VAR = NQ != NM + 1;
    static constexpr bool REV = SHAPE == NKB_HEX || OP == LN_PD;
    // the mesh's point counts
    static constexpr int M0 = NQ, M1 = SHAPE == NKB_TET ? NQ - 1 : NQ;
    static constexpr int M2 = SHAPE == NKB_HEX ? NQ : NQ - 1;
    static constexpr int K0 = REV ? M2 : M0, K1 = M1, K2 = REV ? M0 : M2;
    static constexpr int NT = K0 * K1 * K2;
    static constexpr int NP = NM * (NM + 1) / 2;
    static constexpr int NC = SHAPE == NKB_HEX     ? NM * NM * NM
                              : SHAPE == NKB_PRISM ? NM * NP
                                                   : NM * (NM + 1) * (NM + 2) / 6;
    static constexpr int XR = SHAPE == NKB_HEX ? NM | 1 : 1; // coefficient row stride
    static constexpr int XSIZE = SHAPE == NKB_HEX ? NM * NM * XR : NC;
    // straight-sided elements too read a value per point, formed in FP64 and rounded
    // once (nkb_ops.cu allocates no geoc then)
    static constexpr bool PACKED = (OP == LN_HELM || OP == LN_ADR) && sizeof(T) == 4;
    static constexpr int NCUBE = OP == LN_IP ? 1 : (OP == LN_BWD ? 2 : 3);
    // threads: one per line of the direction with the most lines
    static constexpr int LA = K1 * K2, LB = K0 * K2, LC = K0 * K1;
    static constexpr int LMAX = LA > LB ? (LA > LC ? LA : LC) : (LB > LC ? LB : LC);

    // elements per CTA: the fewest idle lanes at 96 to 256 threads
    static constexpr int Epb()
    {
        int best = 1, num = 0, den = 1;
        for (int e = 1; e <= 32; ++e)
        {
            const int th = (e * LMAX + 31) / 32 * 32;
            if (e > 1 && th > 256)
                break;
            if (th < 96 && e < 32 && ((e + 1) * LMAX + 31) / 32 * 32 <= 256)
                continue;
            // e*LMAX/th > num/den, or equal within 2 %: keep the smaller CTA
            if (e * LMAX * den * 50 > num * th * 51)
            {
                best = e;
                num  = e * LMAX;
                den  = th;
            }
        }
        return best;
    }
    static constexpr int EPB = Epb();
    static constexpr int TH  = (EPB * LMAX + 31) / 32 * 32;
    static constexpr int BANKS = 128 / int(sizeof(T));
    // without derivatives only lines of modes are walked in directions 1 and 2:
    // lanes stay in order, so that whole warps are left idle
    static constexpr bool DEAL = OP != LN_BWD && OP != LN_IP;
    static constexpr LineLayout LAY = LineLayoutOf<K0, K1, K2, EPB, TH, BANKS, XSIZE, DEAL>::V;
    static constexpr int PS = LAY.ps, CUBE = LAY.cube;
    static constexpr bool DEALT = DEAL && !LAY.rotate && EPB < 31;
    static_assert(EPB * CUBE < 65536, "line offsets have 16 bits");
    // register budget per thread: the lowest that spills next to nothing (49 of the
    // 630 instantiations spill, 4 to 92 bytes; PhysDeriv's FP64 chain rule and
    // LinearADR's extra rows take more). Warps in flight hide the barriers and the
    // shared-memory latency: at 80 instead of 128 registers the FP64 Helmholtz
    // operator took 87 instead of 118 us (hex, 8 modes x 7140), 103 instead of 143
    // (9 x 5172), 115 instead of 184 (tet, 8 x 10241); FP32 at 48 instead of 64
    // gained 0-25 %
    static constexpr int REGS =
        sizeof(T) == 8 ? (K0 <= (OP == LN_ADR ? 9 : 10) ? 80 : 96)
                       : (OP == LN_PD && SHAPE == NKB_TET ? 56 : (K0 <= 9 ? 48 : 64));
    static constexpr int MINB0 = 65536 / (TH * REGS);
    static constexpr int MINB  = MINB0 < 1 ? 1 : (MINB0 * TH > 2048 ? 2048 / TH : MINB0);
    static constexpr size_t SMEM = size_t(EPB) * NCUBE * CUBE * sizeof(T);

    __device__ static __forceinline__ int Idx(int a, int b, int c)
    {
        return a * PS + b * K2 + (LAY.rotate ? (c ^ (b & (K2 - 1))) : c);
    }
    // position in the mesh's point order (first direction fastest)
    __device__ static __forceinline__ int Natural(int a, int b, int c)
    {
        return REV ? (a * K1 + b) * K2 + c : (c * K1 + b) * K0 + a;
    }
};

// 1-D tables in kernel directions, passed by value
template <int SHAPE, int NM, int NQ, int OP, typename T> struct LineTabs
{
    using L = LineDims<SHAPE, NM, NQ, OP, T>;
    static constexpr bool BASIS = OP != LN_PD, DERIV = OP != LN_BWD && OP != LN_IP;
    T B0[BASIS ? NM * L::K0 : 1];
    T B1[BASIS && SHAPE != NKB_TET ? NM * L::K1 : 1];
    T B2[BASIS && SHAPE == NKB_HEX ? NM * L::K2 : 1];
    // D[m*K + i] = l_m'(z_i)
    T D0[DERIV ? L::K0 * L::K0 : 1], D1[DERIV ? L::K1 * L::K1 : 1], D2[DERIV ? L::K2 * L::K2 : 1];
    // of the mesh's directions: quadrature weights; collapsed coordinates
    // (1+z0)/2, (1+z1)/2, 2/(1-z1), 2/(1-z2)
    // (FP64: an FP32 kernel rounds products of them once, as packed factors are)
    double w0[L::M0], w1[L::M1], w2[L::M2];
    double h0[L::M0], h1[L::M1], g1[L::M1], g2[L::M2];
};

// d/d xi of the standard element from the collapsed-coordinate derivatives at
// one point (in the mesh's directions), and the transpose; g12 = g1 g2
template <int SHAPE, typename T>
__device__ __forceinline__ void LineChain(T h0, T h1, T g2, T g12, T &d0, T &d1, T &d2)
{
    if (SHAPE == NKB_TET)
    {
        d0        = g12 * d0;
        const T a = h0 * d0, b = g2 * d1;
        d2        = fma(h1, b, a) + d2;
        d1        = a + b;
    }
    else if (SHAPE == NKB_PRISM)
    {
        d0 = g2 * d0;
        d2 = fma(h0, d0, d2);
    }
}

template <int SHAPE, typename T>
__device__ __forceinline__ void LineChainT(T h0, T h1, T g2, T g12, T &v0, T &v1, T &v2)
{
    if (SHAPE == NKB_TET)
    {
        v0 = g12 * fma(h0, v1 + v2, v0);
        v1 = g2 * fma(h1, v2, v1);
    }
    else if (SHAPE == NKB_PRISM)
    {
        v0 = g2 * fma(h0, v2, v0);
    }
}

// out[n] = sum_m in[m] tab[m*N + n] (m < M, n < N) and its transpose; VAR:
// only the first `count` m exist
// DOWN: from the last m, so that the small high modes are added before the
// large low ones
template <bool VAR = false, bool DOWN = false, int M, int N, typename T>
__device__ __forceinline__ void LineMul(const T *__restrict__ tab, const T (&in)[M], T (&out)[N],
                                        int count = M)
{
#pragma unroll
    for (int n = 0; n < N; ++n)
        out[n] = DOWN ? T(0) : in[0] * tab[n];
#pragma unroll
    for (int v = DOWN ? 0 : 1; v < M; ++v)
    {
        const int m = DOWN ? M - 1 - v : v;
        if (!VAR || m < count)
        {
#pragma unroll
            for (int n = 0; n < N; ++n)
                out[n] = fma(in[m], tab[m * N + n], out[n]);
        }
    }
}
template <bool VAR = false, int M, int N, typename T>
__device__ __forceinline__ void LineMulT(const T *__restrict__ tab, const T (&in)[N], T (&out)[M],
                                         int count = M)
{
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (!VAR || m < count)
        {
            T s = in[0] * tab[m * N];
#pragma unroll
            for (int n = 1; n < N; ++n)
                s = fma(in[n], tab[m * N + n], s);
            out[m] = s;
        }
}

struct LineOf
{
    int e, at, x, y; // element of the CTA, offset of the line, its two indices
};

template <int SHAPE, int NM, int NQ, int OP, typename T>
__global__ void __launch_bounds__(LineDims<SHAPE, NM, NQ, OP, T>::TH,
                                  LineDims<SHAPE, NM, NQ, OP, T>::MINB)
    k_line(const __grid_constant__ LineArgs<T> a,
           const __grid_constant__ LineTabs<SHAPE, NM, NQ, OP, T> c)
{
    using L = LineDims<SHAPE, NM, NQ, OP, T>;
    constexpr int K0 = L::K0, K1 = L::K1, K2 = L::K2, NT = L::NT;
    constexpr int CUBE = L::CUBE, PS = L::PS;
    constexpr bool VAR = L::VAR;
    constexpr bool HEX = SHAPE == NKB_HEX, TET = SHAPE == NKB_TET;
    constexpr bool HELM = OP == LN_HELM || OP == LN_ADR;
    constexpr bool PACKED = L::PACKED;
    constexpr bool FROM_COEFFS = HELM || OP == LN_BWD, TO_COEFFS = OP != LN_BWD && OP != LN_PD;
    extern __shared__ __align__(128) unsigned char line_raw[];
    T *S0 = reinterpret_cast<T *>(line_raw);
    const int EPB = a.epb, TH = blockDim.x;
    T *S1 = S0 + EPB * CUBE, *S2 = S1 + EPB * CUBE;
    const long e0 = long(blockIdx.x) * EPB;
    const int ne  = int(min(long(EPB), long(a.nelmt) - e0));
    const int tid = threadIdx.x;
    if (ne <= 0 || (a.skip && *a.skip))
        return;
    const bool curved = PACKED || a.geoc == nullptr;
    const int nm      = VAR ? a.nm : NM, nm2 = nm * nm, np = nm * (nm + 1) / 2;
    const int nc      = HEX ? nm2 * nm : (TET ? nm * (nm + 1) * (nm + 2) / 6 : nm * np);
    if ((HELM || OP == LN_IPD || OP == LN_PD) && tid == 0 && curved)
        BulkPrefetchL2(a.geo + e0 * a.gstride, uint32_t(ne * a.gstride * long(sizeof(T))));

    // this thread's line along the register direction
    const int re = tid / L::LA, rl = tid - re * L::LA;
    const int rj = rl / K2, rk = rl - rj * K2;
    const bool ract = re < ne;
    const int rbase = re * CUBE + L::Idx(0, rj, rk);
    const long rgeo = (e0 + re) * a.gstride + rl;

    // its lines along directions 1 (a, c) and 2 (a, b)
    uint2 lanes;
    if constexpr (L::DEALT)
        lanes = __ldg(a.lanes + tid);
    // the thread's line along `dir` if its x < n1 and y < n2
    auto line = [&](int dir, int n1, int n2) -> LineOf {
        int e, at, x, y;
        if constexpr (L::DEALT)
        {
            const unsigned w = dir == 1 ? lanes.x : lanes.y;
            e = w >> 24, at = w & 0xffff, x = w >> 16 & 15, y = w >> 20 & 15;
        }
        else
        {
            const int c2 = dir == 1 ? K2 : K1;
            e = tid / (K0 * c2), x = tid / c2 % K0, y = tid % c2;
            at = e * CUBE + x * PS + (dir == 1 ? (L::LAY.rotate ? 0 : y) : y * K2);
        }
        return {x < n1 && y < n2 ? e : 31, at, x, y};
    };
    // entry j of a line along direction 1, k of one along direction 2
    auto at1 = [&](const LineOf &l, int j) {
        return l.at + j * K2 + (L::LAY.rotate ? (l.y ^ (j & (K2 - 1))) : 0);
    };
    auto at2 = [&](const LineOf &l, int k) {
        return l.at + (L::LAY.rotate ? (k ^ (l.y & (K2 - 1))) : k);
    };

    // the CTA's points in the arrays' order, fn(element, point, i, j, k): a point's
    // indices are worked out once for all elements, or, with few elements, per
    // point so that several are in flight. Unrolled, several points' loads are in
    // flight at once: without it FP64 IProduct took 1.09 to 1.51 times as long
    // (prisms and tets of 3 to 10 modes), IProductWRTDerivBase, whose points take
    // three loads each, 0.95 to 1.13 (prisms) and 0.97 to 1.21 (tets) and BwdTrans,
    // which only stores, 0.93 to 1.04
    auto each_point = [&](auto fn) {
        if constexpr (L::EPB >= 2)
        {
            constexpr int U = OP == LN_IPD ? 2 : (L::EPB < 4 ? L::EPB : 4), UN = L::EPB == 2 ? 2 : 1;
#pragma unroll(UN)
            for (int n = tid; n < NT; n += TH)
            {
                const int i = n % K0, j = n / K0 % K1, k = n / (K0 * K1);
#pragma unroll(U)
                for (int e = 0; e < ne; ++e)
                    fn(e, n, i, j, k);
            }
        }
        else
        {
#pragma unroll 2
            for (int t = tid; t < ne * NT; t += TH)
            {
                const int e = t / NT, n = t - e * NT;
                fn(e, n, n % K0, n / K0 % K1, n / (K0 * K1));
            }
        }
    };

    T u[K0], f[K0];

    // ---------------- coefficients to points -----------------------------
    if constexpr (FROM_COEFFS)
    {
        // Bwd: x in S0, first stage to S1, second to S0; Helmholtz: x in S1,
        // S2, S0
        T *X = OP == LN_BWD ? S0 : S1, *A = OP == LN_BWD ? S1 : S2, *Bc = S0;
        {
            constexpr int PER = (L::NC + L::LMAX - 1) / L::LMAX; // TH >= EPB * LMAX
            const int nall    = ne * nc;
            const T *in0      = a.gmap ? a.in : a.in + e0 * nc;
            int src[PER];
#pragma unroll
            for (int v = 0; v < PER; ++v)
            {
                const int t = tid + v * TH;
                src[v]      = t < nall ? (a.gmap ? a.gmap[e0 * nc + t] : t) : -1;
            }
            T val[PER];
#pragma unroll
            for (int v = 0; v < PER; ++v)
                val[v] = src[v] >= 0 ? in0[src[v]] : T(0);
#pragma unroll
            for (int v = 0; v < PER; ++v)
            {
                const int t = tid + v * TH;
                if (t < nall)
                {
                    const int e = t / nc, m = t - e * nc;
                    T x         = val[v];
                    if (a.gmap && a.gsign)
                        x *= T(a.gsign[e0 * nc + t]);
                    X[e * CUBE + (HEX ? (m / nm) * L::XR + m % nm : m)] = x;
                }
            }
        }
        __syncthreads();
        // third mode direction
        if constexpr (HEX)
        {
            if (tid < ne * nm2)
            {
                const int e = tid / nm2, pq = tid - e * nm2;
                const int p = pq / nm, q = pq - p * nm;
                T x[NM], w[K2];
#pragma unroll
                for (int r = 0; r < NM; ++r)
                    if (!VAR || r < nm)
                        x[r] = X[e * CUBE + pq * L::XR + r];
                LineMul<VAR>(c.B2, x, w, nm);
#pragma unroll
                for (int k = 0; k < K2; ++k)
                    A[e * CUBE + L::Idx(p, q, k)] = w[k];
            }
        }
        else
        {
            // a thread keeps one column of the (p, q)-dependent table and
            // walks the CTA's elements
            const int items = (TET ? np : nm2) * K2;
            const int G     = TH / items > 1 ? TH / items : 1;
            for (int it = tid; it < items * G; it += TH)
            {
                const int g = it / items, item = it - g * items;
                const int pair = item / K2, k = item - pair * K2;
                int p, q, len, row, xo;
                if constexpr (TET)
                {
                    const unsigned w = __ldg(a.pairs + pair);
                    p = w & 15, q = w >> 4 & 15, len = w >> 8 & 15, row = xo = w >> 12;
                }
                else
                {
                    p = pair / nm, q = pair - p * nm, len = nm - p;
                    row = p * nm - p * (p - 1) / 2, xo = nm * row + q * len;
                }
                // the coefficient folded into this line
                const int fold = TET ? (p + q == 1 ? 1 : -1) : (p == 1 ? q * nm + 1 : -1);
                const T ft     = fold >= 0 ? __ldg(a.tB2 + K2 + k) : T(0);
                T tab[NM];
#pragma unroll
                for (int r = 0; r < NM; ++r)
                    tab[r] = r < len ? __ldg(a.tB2 + (row + r) * K2 + k) : T(0);
                for (int e = g; e < ne; e += G)
                {
                    const T *x = X + e * CUBE;
                    T s        = fold >= 0 ? x[fold] * ft : T(0);
#pragma unroll
                    for (int r = 0; r < NM; ++r)
                        if (r < len)
                            s = fma(x[xo + r], tab[r], s);
                    A[e * CUBE + L::Idx(p, q, k)] = s;
                    if (TET && p == 0 && q == 1)
                        A[e * CUBE + L::Idx(1, nm - 1, k)] = s;
                }
            }
        }
        __syncthreads();
        // second mode direction
        if constexpr (TET)
        {
            const int p = tid / (EPB * K2), ek = tid - p * EPB * K2;
            const int e = ek / K2, k = ek - e * K2;
            if (p < nm && e < ne)
            {
                const int len = p == 1 ? nm : nm - p, pr = p * nm - p * (p - 1) / 2;
                T s[K1];
#pragma unroll
                for (int j = 0; j < K1; ++j)
                    s[j] = 0;
#pragma unroll
                for (int q = 0; q < NM; ++q)
                    if (q < len)
                    {
                        const T w   = A[e * CUBE + L::Idx(p, q, k)];
                        const T *tb = a.tB1 + ((q == nm - 1 && p == 1) ? 1 : pr + q) * K1;
#pragma unroll
                        for (int j = 0; j < K1; ++j)
                            s[j] = fma(w, __ldg(tb + j), s[j]);
                    }
#pragma unroll
                for (int j = 0; j < K1; ++j)
                    Bc[e * CUBE + L::Idx(p, j, k)] = s[j];
            }
        }
        else
        {
            if (const LineOf l = line(1, nm, K2); l.e < ne)
            {
                T w[NM], s[K1];
#pragma unroll
                for (int q = 0; q < NM; ++q)
                    if (!VAR || q < nm)
                        w[q] = A[at1(l, q)];
                LineMul<VAR>(c.B1, w, s, nm);
#pragma unroll
                for (int j = 0; j < K1; ++j)
                    Bc[at1(l, j)] = s[j];
            }
        }
        __syncthreads();
        // register direction, in place
        if (ract)
        {
            T w[NM];
#pragma unroll
            for (int p = 0; p < NM; ++p)
                if (!VAR || p < nm)
                    w[p] = Bc[rbase + p * PS];
            LineMul<VAR, !HEX>(c.B0, w, u, nm);
            if (OP == LN_BWD && L::REV)
            {
                T *o = a.out0 + (e0 + re) * NT + rl;
#pragma unroll
                for (int i = 0; i < K0; ++i)
                    o[i * L::LA] = u[i];
            }
            else
            {
#pragma unroll
                for (int i = 0; i < K0; ++i)
                    S0[rbase + i * PS] = u[i];
            }
        }
        if constexpr (OP == LN_BWD)
        {
            if constexpr (!L::REV)
            {
                __syncthreads();
                T *o = a.out0 + e0 * NT;
                each_point([&](int e, int n, int i, int j, int k) {
                    o[e * NT + n] = S0[e * CUBE + L::Idx(i, j, k)];
                });
            }
            return;
        }
    }

    // ---------------- physical input ---------------------------------------
    if constexpr (OP == LN_PD)
    {
        if (ract)
        {
            const T *in = a.in + (e0 + re) * NT + rl;
#pragma unroll
            for (int i = 0; i < K0; ++i)
                u[i] = in[i * L::LA];
#pragma unroll
            for (int i = 0; i < K0; ++i)
                S0[rbase + i * PS] = u[i];
        }
    }
    if constexpr (OP == LN_IP || OP == LN_IPD)
    {
        // values of one point: f = W in, or v = W A^T (in, in1, in2) in the
        // mesh's directions
        auto point = [&](long e, int n, int m0, int m1, int m2, T &v0, T &v1, T &v2) {
            // the packing's order of products
            const double W =
                curved ? 0.0 : a.geoc[e * kGeoc] * c.w0[m0] * c.w1[m1] * c.w2[m2];
            if (OP == LN_IP)
            {
                v0 = a.in[e * NT + n] * (curved ? a.geo[e * a.gstride + n] : T(W));
                return;
            }
            const T f0 = a.in[e * NT + n], f1 = a.in1[e * NT + n], f2 = a.in2[e * NT + n];
            if (curved)
            {
                const T *P = a.geo + e * a.gstride + n;
                v0         = fma(P[2 * NT], f2, fma(P[1 * NT], f1, P[0] * f0));
                v1         = fma(P[5 * NT], f2, fma(P[4 * NT], f1, P[3 * NT] * f0));
                v2         = fma(P[8 * NT], f2, fma(P[7 * NT], f1, P[6 * NT] * f0));
                return;
            }
            // in FP64 for FP32 fields too, so that nothing is rounded but the results
            const double *P = a.geoc + e * kGeoc, d0 = f0, d1 = f1, d2 = f2;
            double x0 = W * fma(P[13], d2, fma(P[10], d1, P[7] * d0));
            double x1 = W * fma(P[14], d2, fma(P[11], d1, P[8] * d0));
            double x2 = W * fma(P[15], d2, fma(P[12], d1, P[9] * d0));
            LineChainT<SHAPE>(c.h0[m0], c.h1[m1], c.g2[m2], c.g1[m1] * c.g2[m2], x0, x1, x2);
            v0 = T(x0), v1 = T(x1), v2 = T(x2);
        };
        if constexpr (L::REV)
        {
            if (ract)
            {
#pragma unroll
                for (int i = 0; i < K0; ++i)
                {
                    T v0, v1, v2;
                    point(e0 + re, i * L::LA + rl, rk, rj, i, v0, v1, v2);
                    if (OP == LN_IP)
                    {
                        f[i] = v0;
                    }
                    else
                    {
                        u[i]               = v2;
                        S1[rbase + i * PS] = v1;
                        S2[rbase + i * PS] = v0;
                    }
                }
            }
        }
        else
        {
            each_point([&](int e, int n, int i, int j, int k) {
                T v0, v1, v2;
                point(e0 + e, n, i, j, k, v0, v1, v2);
                const int s = e * CUBE + L::Idx(i, j, k);
                S0[s]       = v0;
                if (OP == LN_IPD)
                {
                    S1[s] = v1;
                    S2[s] = v2;
                }
            });
            __syncthreads();
            if (ract)
            {
#pragma unroll
                for (int i = 0; i < K0; ++i)
                    (OP == LN_IP ? f[i] : u[i]) = S0[rbase + i * PS];
            }
        }
        if constexpr (OP == LN_IPD)
        {
            if (ract)
                LineMulT(c.D0, u, f);
            if (L::REV)
                __syncthreads();
        }
    }

    if constexpr (HELM || OP == LN_PD)
    {
        // ---------------- gradient -----------------------------------------
        T g0[K0];
        if (ract)
            LineMul(c.D0, u, g0);
        __syncthreads();
        if (const LineOf l = line(1, K0, K2); l.e < ne)
        {
            T v[K1], g[K1];
#pragma unroll
            for (int j = 0; j < K1; ++j)
                v[j] = S0[at1(l, j)];
            LineMul(c.D1, v, g);
#pragma unroll
            for (int j = 0; j < K1; ++j)
                S1[at1(l, j)] = g[j];
        }
        if (const LineOf l = line(2, K0, K1); l.e < ne)
        {
            T v[K2], g[K2];
#pragma unroll
            for (int k = 0; k < K2; ++k)
                v[k] = S0[at2(l, k)];
            LineMul(c.D2, v, g);
#pragma unroll
            for (int k = 0; k < K2; ++k)
                S2[at2(l, k)] = g[k];
        }
        __syncthreads();
        if constexpr (OP == LN_PD)
        {
            if (!ract)
                return;
            const long o = (e0 + re) * NT + rl;
            if (curved)
            {
                const T *A = a.geo + rgeo;
#pragma unroll
                for (int i = 0; i < K0; ++i)
                {
                    const T q0 = S2[rbase + i * PS], q1 = S1[rbase + i * PS], q2 = g0[i];
                    const T *Ai = A + i * L::LA;
                    a.out0[o + i * L::LA] = fma(Ai[6 * NT], q2, fma(Ai[3 * NT], q1, Ai[0] * q0));
                    a.out1[o + i * L::LA] = fma(Ai[7 * NT], q2, fma(Ai[4 * NT], q1, Ai[NT] * q0));
                    a.out2[o + i * L::LA] = fma(Ai[8 * NT], q2, fma(Ai[5 * NT], q1, Ai[2 * NT] * q0));
                }
                return;
            }
            // the chain rule in FP64 for FP32 collapsed elements too: its products
            // would otherwise add to the rounding of the packed factors it replaces
            using C        = typename std::conditional<HEX, T, double>::type;
            const double g = c.g1[rj];
            C F[9];
#pragma unroll
            for (int m = 0; m < 9; ++m)
                F[m] = C(a.geoc[(e0 + re) * kGeoc + 7 + m]);
#pragma unroll
            for (int i = 0; i < K0; ++i)
            {
                C q0 = S2[rbase + i * PS], q1 = S1[rbase + i * PS], q2 = g0[i];
                LineChain<SHAPE>(C(c.h0[rk]), C(c.h1[rj]), C(c.g2[i]), C(g * c.g2[i]), q0, q1, q2);
                a.out0[o + i * L::LA] = T(fma(F[2], q2, fma(F[1], q1, F[0] * q0)));
                a.out1[o + i * L::LA] = T(fma(F[5], q2, fma(F[4], q1, F[3] * q0)));
                a.out2[o + i * L::LA] = T(fma(F[8], q2, fma(F[7], q1, F[6] * q0)));
            }
            return;
        }
        // ---------------- metric ---------------------------------------------
        if (ract)
        {
            const T lam = a.lambda;
            if (curved)
            {
                const T *G = a.geo + rgeo;
                // components in kernel directions (hexahedra: reversed)
                constexpr int C00 = HEX ? 3 : 1, C11 = 2, C22 = HEX ? 1 : 3;
                constexpr int C01 = HEX ? 6 : 4, C02 = 5, C12 = HEX ? 4 : 6;
                constexpr int A0 = HEX ? 9 : 7, A2 = HEX ? 7 : 9;
#pragma unroll
                for (int i = 0; i < K0; ++i)
                {
                    const int s = rbase + i * PS;
                    const T *Gi = G + i * L::LA;
                    const T q0 = g0[i], q1 = S1[s], q2 = S2[s];
                    const T G01 = __ldg(Gi + C01 * NT), G02 = __ldg(Gi + C02 * NT),
                            G12 = __ldg(Gi + C12 * NT);
                    T mass = __ldg(Gi) * u[i];
                    if (OP == LN_ADR)
                        mass = fma(__ldg(Gi + A2 * NT), q2,
                                   fma(__ldg(Gi + 8 * NT), q1, fma(__ldg(Gi + A0 * NT), q0, mass)));
                    f[i]  = lam * mass;
                    S1[s] = fma(G12, q2, fma(__ldg(Gi + C11 * NT), q1, G01 * q0));
                    S2[s] = fma(__ldg(Gi + C22 * NT), q2, fma(G12, q1, G02 * q0));
                    g0[i] = fma(G02, q2, fma(G01, q1, __ldg(Gi + C00 * NT) * q0));
                }
            }
            else if constexpr (!PACKED)
            {
                const double *P = a.geoc + (e0 + re) * kGeoc;
                const T J = P[0], G00 = P[1], G11 = P[2], G22 = P[3], G01 = P[4], G02 = P[5],
                        G12 = P[6];
                const T ww = HEX ? c.w0[rk] * c.w1[rj] : c.w1[rj] * c.w2[rk];
                const T h1 = c.h1[rj], g2 = HEX ? 0.0 : c.g2[rk],
                        g12 = HEX ? 0.0 : c.g1[rj] * c.g2[rk];
                const T *V = OP == LN_ADR ? a.geo + rgeo + 7 * NT : nullptr;
#pragma unroll
                for (int i = 0; i < K0; ++i)
                {
                    const int s = rbase + i * PS;
                    // in the mesh's directions
                    T q0 = HEX ? S2[s] : g0[i], q1 = S1[s], q2 = HEX ? g0[i] : S2[s];
                    const T W = ww * (HEX ? c.w2[HEX ? i : 0] : c.w0[i]);
                    T mass    = W * J * u[i];
                    if (OP == LN_ADR)
                        mass = fma(__ldg(V + 2 * NT + i * L::LA), q2,
                                   fma(__ldg(V + NT + i * L::LA), q1,
                                       fma(__ldg(V + i * L::LA), q0, mass)));
                    f[i] = lam * mass;
                    LineChain<SHAPE>(T(c.h0[HEX ? 0 : i]), h1, g2, g12, q0, q1, q2);
                    T v0 = W * fma(G02, q2, fma(G01, q1, G00 * q0));
                    T v1 = W * fma(G12, q2, fma(G11, q1, G01 * q0));
                    T v2 = W * fma(G22, q2, fma(G12, q1, G02 * q0));
                    LineChainT<SHAPE>(T(c.h0[HEX ? 0 : i]), h1, g2, g12, v0, v1, v2);
                    S1[s] = v1;
                    S2[s] = HEX ? v0 : v2;
                    g0[i] = HEX ? v2 : v0;
                }
            }
            T t[K0];
            LineMulT(c.D0, g0, t);
#pragma unroll
            for (int i = 0; i < K0; ++i)
                f[i] += t[i];
        }
        __syncthreads();
    }

    if constexpr (HELM || OP == LN_IPD)
    {
        // ---------------- transposed gradient, in place ----------------------
        if (const LineOf l = line(1, K0, K2); l.e < ne)
        {
            T v[K1], g[K1];
#pragma unroll
            for (int j = 0; j < K1; ++j)
                v[j] = S1[at1(l, j)];
            LineMulT(c.D1, v, g);
#pragma unroll
            for (int j = 0; j < K1; ++j)
                S1[at1(l, j)] = g[j];
        }
        if (const LineOf l = line(2, K0, K1); l.e < ne)
        {
            T v[K2], g[K2];
#pragma unroll
            for (int k = 0; k < K2; ++k)
                v[k] = S2[at2(l, k)];
            LineMulT(c.D2, v, g);
#pragma unroll
            for (int k = 0; k < K2; ++k)
                S2[at2(l, k)] = g[k];
        }
        __syncthreads();
        if (ract)
        {
#pragma unroll
            for (int i = 0; i < K0; ++i)
                f[i] = (f[i] + S2[rbase + i * PS]) + S1[rbase + i * PS];
        }
    }

    // ---------------- points to coefficients ---------------------------------
    if constexpr (TO_COEFFS && HEX)
    {
        // the lane directions first, in place, the register direction last:
        // its threads then write the coefficients in the arrays' order
        if (ract)
        {
#pragma unroll
            for (int i = 0; i < K0; ++i)
                S0[rbase + i * PS] = f[i];
        }
        __syncthreads();
        if (const LineOf l = line(2, K0, K1); l.e < ne)
        {
            T v[K2], s[NM];
#pragma unroll
            for (int k = 0; k < K2; ++k)
                v[k] = S0[at2(l, k)];
            LineMulT<VAR>(c.B2, v, s, nm);
#pragma unroll
            for (int r = 0; r < NM; ++r)
                if (!VAR || r < nm)
                    S0[at2(l, r)] = s[r];
        }
        __syncthreads();
        if (const LineOf l = line(1, K0, nm); l.e < ne)
        {
            T v[K1], s[NM];
#pragma unroll
            for (int j = 0; j < K1; ++j)
                v[j] = S0[at1(l, j)];
            LineMulT<VAR>(c.B1, v, s, nm);
#pragma unroll
            for (int q = 0; q < NM; ++q)
                if (!VAR || q < nm)
                    S0[at1(l, q)] = s[q];
        }
        __syncthreads();
        {
            if (ract && rj < nm && rk < nm)
            {
                T v[K0], s[NM];
#pragma unroll
                for (int i = 0; i < K0; ++i)
                    v[i] = S0[rbase + i * PS];
                LineMulT<VAR>(c.B0, v, s, nm);
                T *y = a.out0 + (e0 + re) * nc + rj * nm + rk;
#pragma unroll
                for (int p = 0; p < NM; ++p)
                    if (!VAR || p < nm)
                        y[p * nm2] = s[p];
            }
        }
    }
    if constexpr (TO_COEFFS && !HEX)
    {
        if (ract)
        {
            T y[NM];
            LineMulT<VAR>(c.B0, f, y, nm);
#pragma unroll
            for (int p = 0; p < NM; ++p)
                if (!VAR || p < nm)
                    S0[rbase + p * PS] = y[p];
        }
        __syncthreads();
        if constexpr (TET)
        {
            const int p = tid / (EPB * K2), ek = tid - p * EPB * K2;
            const int e = ek / K2, k = ek - e * K2;
            if (p < nm && e < ne)
            {
                const int len = p == 1 ? nm : nm - p, pr = p * nm - p * (p - 1) / 2;
                T v[K1];
#pragma unroll
                for (int j = 0; j < K1; ++j)
                    v[j] = S0[e * CUBE + L::Idx(p, j, k)];
#pragma unroll
                for (int q = 0; q < NM; ++q)
                    if (q < len)
                    {
                        const T *tb = a.tB1 + ((q == nm - 1 && p == 1) ? 1 : pr + q) * K1;
                        T s         = 0;
#pragma unroll
                        for (int j = 0; j < K1; ++j)
                            s = fma(v[j], __ldg(tb + j), s);
                        S0[e * CUBE + L::Idx(p, q, k)] = s;
                    }
            }
        }
        else
        {
            if (const LineOf l = line(1, nm, K2); l.e < ne)
            {
                T v[K1], s[NM];
#pragma unroll
                for (int j = 0; j < K1; ++j)
                    v[j] = S0[at1(l, j)];
                LineMulT<VAR>(c.B1, v, s, nm);
#pragma unroll
                for (int q = 0; q < NM; ++q)
                    if (!VAR || q < nm)
                        S0[at1(l, q)] = s[q];
            }
        }
        __syncthreads();
        T *y = a.out0 + e0 * nc;
        // a thread keeps one coefficient's table row and walks the elements
        const int G = TH / nc > 1 ? TH / nc : 1;
        for (int it = tid; it < nc * G; it += TH)
        {
            const int g = it / nc, m = it - g * nc;
            const unsigned w = __ldg(a.coefs + m);
            const int p = w & 15, q = (w >> 4) & 15, fold = w >> 8;
            T tab[K2];
#pragma unroll
            for (int k = 0; k < K2; ++k)
                tab[k] = __ldg(a.tC + k * nc + m);
            for (int e = g; e < ne; e += G)
            {
                const T *s = S0 + e * CUBE;
                T v[K2];
#pragma unroll
                for (int k = 0; k < K2; ++k)
                    v[k] = s[L::Idx(p, q, k)];
                if (fold)
                {
#pragma unroll
                    for (int k = 0; k < K2; ++k)
                    {
                        if (!TET)
                            v[k] += s[L::Idx(1, q, k)];
                        else if (fold == 2)
                            v[k] += (s[L::Idx(0, 1, k)] + s[L::Idx(1, nm - 1, k)]) +
                                    s[L::Idx(1, 0, k)];
                        else
                            v[k] += s[L::Idx(1, nm - 1, k)];
                    }
                }
                T z = v[0] * tab[0];
#pragma unroll
                for (int k = 1; k < K2; ++k)
                    z = fma(v[k], tab[k], z);
                y[e * nc + m] = z;
            }
        }
    }
}

// ---- host side ---------------------------------------------------------------

// the tables of one operator in the kernel's parameter layout
template <int SHAPE, int NM, int NQ, int OP, typename T>
void LineBuildTabs(const nkb_op *op, std::vector<unsigned char> &blob)
{
    using L   = LineDims<SHAPE, NM, NQ, OP, T>;
    using Tab = LineTabs<SHAPE, NM, NQ, OP, T>;
    static_assert(std::is_trivially_copyable<Tab>::value, "passed by value");
    Tab t;
    std::memset(&t, 0, sizeof(t));
    const int dir[3] = {L::REV ? 2 : 0, 1, L::REV ? 0 : 2}; // mesh direction of kernel direction
    auto put         = [](T *dst, const std::vector<double> &src, size_t n) {
        for (size_t i = 0; i < n; ++i)
            dst[i] = T(src[i]);
    };
    if (Tab::BASIS)
    {
        put(t.B0, op->hB[dir[0]], op->nm * L::K0);
        if (SHAPE != NKB_TET)
            put(t.B1, op->hB[1], op->nm * L::K1);
        if (SHAPE == NKB_HEX)
            put(t.B2, op->hB[dir[2]], op->nm * L::K2);
    }
    if (Tab::DERIV)
    {
        put(t.D0, op->hD[dir[0]], L::K0 * L::K0);
        put(t.D1, op->hD[1], L::K1 * L::K1);
        put(t.D2, op->hD[dir[2]], L::K2 * L::K2);
    }
    for (int i = 0; i < L::M0; ++i)
    {
        t.w0[i] = op->hw[0][i];
        t.h0[i] = 0.5 * (1.0 + op->hz[0][i]);
    }
    for (int i = 0; i < L::M1; ++i)
    {
        t.w1[i] = op->hw[1][i];
        t.h1[i] = 0.5 * (1.0 + op->hz[1][i]);
        t.g1[i] = 2.0 / (1.0 - op->hz[1][i]);
    }
    for (int i = 0; i < L::M2; ++i)
    {
        t.w2[i] = op->hw[2][i];
        t.g2[i] = 2.0 / (1.0 - op->hz[2][i]);
    }
    blob.resize(sizeof(t));
    std::memcpy(blob.data(), &t, sizeof(t));
}

// deals the lines (x, y) of epb elements out to th lanes, at most one per bank to
// the lanes of a phase where the banks allow it (words of LineArgs::lanes)
inline void LineDeal(int epb, int cube, int n1, int s1, int n2, int s2, int banks, int th,
                     bool in_order, std::vector<unsigned> &lanes)
{
    lanes.assign(th, 31u << 24); // element 31: none
    std::vector<std::vector<unsigned>> by_bank(banks);
    for (int e = 0, t = 0; e < epb; ++e)
        for (int x = 0; x < n1; ++x)
            for (int y = 0; y < n2; ++y, ++t)
            {
                const int at     = e * cube + x * s1 + y * s2;
                const unsigned w = unsigned(at | x << 16 | y << 20) | unsigned(e) << 24;
                if (in_order)
                    lanes[t] = w;
                else
                    by_bank[at % banks].push_back(w);
            }
    std::vector<int> spare;
    for (int t0 = 0; t0 < th && !in_order; t0 += banks)
        for (int b = 0; b < banks; ++b)
        {
            if (by_bank[b].empty())
            {
                spare.push_back(t0 + b);
                continue;
            }
            lanes[t0 + b] = by_bank[b].back();
            by_bank[b].pop_back();
        }
    for (auto &rest : by_bank)
        for (unsigned line : rest)
        {
            lanes[spare.back()] = line;
            spare.pop_back();
        }
}

// device tables of an operator, one allocation: the table row of every
// coefficient ([k][coefficient]), then lanes, pairs and coefs of LineArgs
template <int SHAPE, int NM, int NQ, int OP, typename T> int LineBuildAux(nkb_op *op)
{
    using L      = LineDims<SHAPE, NM, NQ, OP, T>;
    const int nm = op->nm;
    std::vector<T> rows;
    std::vector<unsigned> words;
    // dealt out for full CTAs, in order for the smaller ones of small collections
    for (int in_order = 0; in_order < 2 && L::DEALT; ++in_order)
    {
        std::vector<unsigned> l1, l2;
        LineDeal(L::EPB, L::CUBE, L::K0, L::PS, L::K2, 1, L::BANKS, L::TH, in_order, l1);
        LineDeal(L::EPB, L::CUBE, L::K0, L::PS, L::K1, L::K2, L::BANKS, L::TH, in_order, l2);
        for (int t = 0; t < L::TH; ++t)
        {
            words.push_back(l1[t]);
            words.push_back(l2[t]);
        }
    }
    if (SHAPE != NKB_HEX && OP != LN_PD)
    {
        std::vector<unsigned> coefs;
        std::vector<int> row;
        for (int p = 0, first = 0; p < nm; ++p)
            for (int q = 0; q < (SHAPE == NKB_TET ? nm - p : nm); ++q)
            {
                const int len = SHAPE == NKB_TET ? nm - p - q : nm - p;
                if (SHAPE == NKB_TET)
                    words.push_back(unsigned(p | q << 4 | len << 8 | first << 12));
                for (int r = 0; r < len; ++r, ++first)
                {
                    // prism (0, q, 1) and tet (0, 1, r): one more line; tet (0, 0, 1): three
                    const int fold = SHAPE == NKB_TET ? (first == 1 ? 2 : p == 0 && q == 1)
                                                      : p == 0 && r == 1;
                    coefs.push_back(unsigned(p | q << 4 | fold << 8));
                    row.push_back(SHAPE == NKB_TET ? first : p * nm - p * (p - 1) / 2 + r);
                }
            }
        words.insert(words.end(), coefs.begin(), coefs.end());
        for (int k = 0; k < L::K2; ++k)
            for (int m : row)
                rows.push_back(T(op->hB[2][size_t(m) * L::K2 + k]));
    }
    if (rows.size() % 2)
        rows.push_back(T(0));
    const size_t nr = rows.size() * sizeof(T), nw = words.size() * sizeof(unsigned);
    std::vector<unsigned char> image(nr + nw);
    if (nr)
        std::memcpy(image.data(), rows.data(), nr);
    std::memcpy(image.data() + nr, words.data(), nw);
    op->line_words = nr;
    NKB_CUDA_TRY(cudaMalloc(&op->line_aux, image.size()));
    NKB_CUDA_TRY(CopyIn(op->line_aux, image.data(), image.size()));
    return NKB_OK;
}

// one kernel: build its tables (setup) or launch it
template <int SHAPE, int NM, int NQ, int OP, typename T>
int LineOne(nkb_op *setup, const nkb_op *op, const LineArgs<T> *a, cudaStream_t s)
{
    using L   = LineDims<SHAPE, NM, NQ, OP, T>;
    auto kern = k_line<SHAPE, NM, NQ, OP, T>;
    static_assert(L::SMEM <= 227 * 1024, "shared memory");
    if (setup)
    {
        LineBuildTabs<SHAPE, NM, NQ, OP, T>(setup, setup->line_tabs);
        const int rc = LineBuildAux<SHAPE, NM, NQ, OP, T>(setup);
        if (rc)
            return rc;
        NKB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          int(L::SMEM)));
        return NKB_OK;
    }
    // a collection smaller than one wave of full CTAs is spread over all SMs in
    // smaller ones (64 hexahedra of 4 modes: 6.5 us in 64 CTAs, 8.4 in 13)
    const int slots   = op->sms * L::MINB;
    LineArgs<T> run   = *a;
    run.epb           = std::min(L::EPB, (op->nelmt + slots - 1) / slots);
    const unsigned nb = unsigned((op->nelmt + run.epb - 1) / run.epb);
    const unsigned th = unsigned((run.epb * L::LMAX + 31) / 32 * 32);
    const unsigned char *aux = static_cast<const unsigned char *>(op->line_aux);
    const unsigned *words    = reinterpret_cast<const unsigned *>(aux + op->line_words);
    run.tC    = reinterpret_cast<const T *>(aux);
    run.lanes = reinterpret_cast<const uint2 *>(words) + (run.epb == L::EPB ? 0 : L::TH);
    run.pairs = words + (L::DEALT ? 4 * L::TH : 0);
    run.coefs = run.pairs + (SHAPE == NKB_TET ? op->nm * (op->nm + 1) / 2 : 0);
    void *params[2]   = {&run, const_cast<unsigned char *>(op->line_tabs.data())};
    NKB_CUDA_TRY(cudaLaunchKernel((const void *)kern, dim3(nb), dim3(th), params,
                                  size_t(run.epb) * L::NCUBE * L::CUBE * sizeof(T), s));
    return NKB_OK;
}

constexpr int kLineNone = 1; // no line kernel for these sizes (no error set)

template <int OP, int NM, int NQ, typename T>
int LineShapes(nkb_op *setup, const nkb_op *op, const LineArgs<T> *a, cudaStream_t s)
{
    if (op->shape == NKB_HEX)
        return LineOne<NKB_HEX, NM, NQ, OP, T>(setup, op, a, s);
    if (op->shape == NKB_PRISM)
        return LineOne<NKB_PRISM, NM, NQ, OP, T>(setup, op, a, s);
    return LineOne<NKB_TET, NM, NQ, OP, T>(setup, op, a, s);
}

// the kernel of the operator's sizes: 3 to 12 points in the first direction, with
// one more point than modes (compile-time modes; PhysDeriv has none) or more
// (over-integration: run-time modes)
template <int OP, typename T>
int LineSwitch(nkb_op *setup, const nkb_op *op, const LineArgs<T> *a, cudaStream_t s)
{
    const bool std = OP == LN_PD || op->nq[0] == op->nm + 1;
    if (op->nm > op->nq[0] - 1)
        return kLineNone;
    switch (op->nq[0])
    {
#define NKB_LN(N)                                                                                  \
    case N:                                                                                        \
        if constexpr (OP != LN_PD && N > 3)                                                        \
            if (!std)                                                                              \
                return LineShapes<OP, N - 2, N, T>(setup, op, a, s);                               \
        return LineShapes<OP, N - 1, N, T>(setup, op, a, s);
        NKB_LN(3) NKB_LN(4) NKB_LN(5) NKB_LN(6) NKB_LN(7) NKB_LN(8) NKB_LN(9) NKB_LN(10) NKB_LN(11)
        NKB_LN(12)
#undef NKB_LN
        default: return kLineNone;
    }
}

} // namespace nkb
