// Kernel selection for the element operators, and the Hex Helmholtz kernels that
// NKB_HEX_VARIANT requests instead of the line kernels (nkb_line_kernel.cuh):
// k_hex_helm, one thread per (i, j) column of the nq x nq slab with the third
// direction in registers and the packed geometry fetched by one bulk TMA copy per
// CTA that completes on an mbarrier (bounded wait), and the tcgen05 kernel of
// nkb_hex_tc.cuh. The line kernels were faster at every order in FP64 and FP32.
#include "nkb_hex_kernel.cuh"
#include "nkb_op.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

namespace nkb
{

// NKB_KERNEL=generic selects the shape-generic kernels for every operator
// (used to test both implementations against each other).
static bool ForceGeneric()
{
    const char *v = std::getenv("NKB_KERNEL");
    return v && std::strcmp(v, "generic") == 0;
}

static bool SameTable(const std::vector<double> &a, const std::vector<double> &b);

// TF32 high part of an FP32 value (round to nearest, ties away from zero,
// as cvt.rna.tf32.f32)
static float Tf32HiHost(float x)
{
    uint32_t u;
    std::memcpy(&u, &x, 4);
    u = (u + 0x1000u) & 0xFFFFE000u;
    float h;
    std::memcpy(&h, &u, 4);
    return h;
}

// Tables of the tensor-core Hex kernel (nkb_hex_tc.cuh) for an FP32 Hex
// Helmholtz operator with nq = nm + 1: per direction d, with B[p][i] the
// basis at the points (Basis::GetBdata) and dB = D B its derivative
// (Basis.cpp:493-495), the coefficient -> point table (K = mode p, rows
// [B_hi | B_lo | dB_hi | dB_lo] over the points i, each padded to 8) and the
// point -> coefficient table (K = point i, rows over the modes p). Directions
// with equal tables share one copy. Built once per operator, in the order and
// layout the kernel copies into shared memory.
int BuildTcTables(nkb_op *op)
{
    const int nm = op->nm, nq = op->nq[0];
    int v = 0;
    if (!HexVariantRequested(op, &v) || v != 5)
        return NKB_OK;
    auto pad8 = [](int v) { return (v + 7) / 8 * 8; };
    const int KM = pad8(nm), KQ = pad8(nq), NQP = pad8(nq), NMN = pad8(nm);
    const int TBROWS = 4 * NQP, TBTROWS = 4 * NMN;
    const size_t tbn = size_t(TBROWS) * KM, tbtn = size_t(TBTROWS) * KQ;
    std::vector<float> img;
    int uniq[3] = {-1, -1, -1};
    for (int d = 0; d < 3; ++d)
    {
        for (int e = 0; e < d && uniq[d] < 0; ++e)
            if (SameTable(op->hB[d], op->hB[e]) && SameTable(op->hD[d], op->hD[e]))
                uniq[d] = uniq[e];
        if (uniq[d] >= 0)
        {
            op->tc_tb[d]  = op->tc_tb[uniq[d]];
            op->tc_tbt[d] = op->tc_tbt[uniq[d]];
            continue;
        }
        uniq[d] = d;
        // B[p][i] and dB[p][i] = sum_m D[i][m] B[p][m] (host D column-major)
        const std::vector<double> &hB = op->hB[d], &hD = op->hD[d];
        std::vector<double> B(size_t(nm) * nq), dB(size_t(nm) * nq, 0.0);
        for (int p = 0; p < nm; ++p)
            for (int i = 0; i < nq; ++i)
            {
                B[p * nq + i] = hB[size_t(p) * nq + i];
                double s      = 0.0;
                for (int m = 0; m < nq; ++m)
                    s += hD[size_t(m) * nq + i] * hB[size_t(p) * nq + m];
                dB[p * nq + i] = s;
            }
        auto part = [&](int which, int p, int i) -> float {
            const double v = (which < 2 ? B : dB)[p * nq + i];
            const float hi = Tf32HiHost(float(v));
            return (which & 1) ? float(v - double(hi)) : hi;
        };
        const size_t base = img.size();
        img.resize(base + tbn + tbtn, 0.f);
        for (int n = 0; n < TBROWS; ++n)
            for (int k = 0; k < KM; ++k)
            {
                const int which = n / NQP, i = n % NQP, p = k;
                if (i < nq && p < nm)
                    img[base + tc::OffB(n, k, TBROWS) / 4] = part(which, p, i);
            }
        for (int n = 0; n < TBTROWS; ++n)
            for (int k = 0; k < KQ; ++k)
            {
                const int which = n / NMN, p = n % NMN, i = k;
                if (i < nq && p < nm)
                    img[base + tbn + tc::OffB(n, k, TBTROWS) / 4] = part(which, p, i);
            }
        op->tc_tb[d]  = int(base * 4);
        op->tc_tbt[d] = int((base + tbn) * 4);
    }
    img.resize((img.size() + 31) / 32 * 32, 0.f); // 128-byte multiple
    cudaFree(op->tc_tab);
    op->tc_tab = nullptr;
    if (cudaMalloc(&op->tc_tab, img.size() * sizeof(float)) != cudaSuccess)
        return SetError(NKB_ERR_NOMEM, "tensor-core Hex tables");
    NKB_CUDA_TRY(CopyIn(op->tc_tab, img.data(), img.size() * sizeof(float)));
    op->tc_bytes = int(img.size() * sizeof(float));
    return NKB_OK;
}

// kernel template and variants: nkb_hex_kernel.cuh, instantiated per precision
// in nkb_hex_f64.cu and nkb_hex_f32.cu
extern template int HexLaunchT<double>(const nkb_op *, const HexArgs<double> &, bool, cudaStream_t,
                                       int, bool);
extern template int HexLaunchT<float>(const nkb_op *, const HexArgs<float> &, bool, cudaStream_t,
                                      int, bool);

template <typename T> static HexArgs<T> MakeHexArgs(const nkb_op *op)
{
    HexArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.geo     = std::is_same<T, double>::value ? (const T *)op->geo : (const T *)op->geo32;
    a.gstride = op->gstride;
    const void *const *B = std::is_same<T, double>::value ? (const void *const *)op->dB
                                                           : (const void *const *)op->fB;
    const void *const *D = std::is_same<T, double>::value ? (const void *const *)op->dD
                                                           : (const void *const *)op->fD;
    a.B0     = (const T *)B[0];
    a.B1     = (const T *)B[1];
    a.B2     = (const T *)B[2];
    a.D      = (const T *)D[0];
    a.lambda = T(op->lambda);
    a.nelmt  = op->nelmt;
    a.err    = op->d_err;
    return a;
}

static std::mutex g_tune_mu;

// Launch shape of the generic kernel (threads per CTA, elements per CTA),
// timed on the operator's own sizes the same way and cached per (shape,
// operator, precision, nm, element count). The arithmetic of an element does
// not depend on the launch shape, so the choice never changes results.
static std::map<std::tuple<int, int, int, int, int>, std::pair<int, int>> g_gen_cache;

template <typename T> static int AutotuneGeneric(nkb_op *op)
{
    const auto key = std::make_tuple(op->shape, op->optype, op->precision, op->nm, op->nelmt);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_gen_cache.find(key);
        if (it != g_gen_cache.end())
        {
            op->gen_epb     = it->second.first;
            op->gen_threads = it->second.second;
            return NKB_OK;
        }
    }
    if (op->nelmt <= 0)
        return NKB_OK;
    const size_t ebyt = GenericSmemBytes(op, int(sizeof(T)));
    const size_t nmax = size_t(op->nelmt) * size_t(std::max(op->nc, op->nt));
    T *buf            = nullptr;
    if (cudaMalloc(&buf, 4 * nmax * sizeof(T)) != cudaSuccess)
        return SetError(NKB_ERR_NOMEM, "autotune buffers");
    cudaMemsetAsync(buf, 0, 4 * nmax * sizeof(T), op->stream);
    float best_ms = 1e30f;
    int best_e = 0, best_t = 0, rc = NKB_OK;
    const int threads[3] = {64, 128, 256};
    const int epbs[4]    = {1, 2, 4, 8};
    for (int ti = 0; ti < 3 && !rc; ++ti)
        for (int ei = 0; ei < 4 && !rc; ++ei)
        {
            if (ebyt * epbs[ei] > 96 * 1024)
                continue;
            op->gen_threads = threads[ti];
            op->gen_epb     = epbs[ei];
            T *in = buf, *o0 = buf + nmax, *o1 = buf + 2 * nmax, *o2 = buf + 3 * nmax;
            if (op->optype == NKB_IPRODUCT_DERIV)
            {
                // three input fields, one output
                o0 = buf + 3 * nmax;
                o1 = o2 = nullptr;
            }
            if ((rc = LaunchGeneric<T>(op, in, o0, o1, o2, nullptr, nullptr, op->stream)))
                break;
            cudaEventRecord(op->ev0, op->stream);
            for (int it = 0; it < 3 && !rc; ++it)
                rc = LaunchGeneric<T>(op, in, o0, o1, o2, nullptr, nullptr, op->stream);
            cudaEventRecord(op->ev1, op->stream);
            if (rc || cudaEventSynchronize(op->ev1) != cudaSuccess)
                break;
            float ms = 0.f;
            cudaEventElapsedTime(&ms, op->ev0, op->ev1);
            if (ms < best_ms)
            {
                best_ms = ms;
                best_e  = epbs[ei];
                best_t  = threads[ti];
            }
        }
    cudaFree(buf);
    op->gen_epb     = best_e;
    op->gen_threads = best_t;
    if (rc)
        return rc;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_gen_cache[key] = std::make_pair(best_e, best_t);
    return NKB_OK;
}

static bool SameTable(const std::vector<double> &a, const std::vector<double> &b)
{
    return a.size() == b.size() && std::equal(a.begin(), a.end(), b.begin());
}

bool HexVariantRequested(const nkb_op *op, int *v)
{
    const char *env = std::getenv("NKB_HEX_VARIANT");
    const int nm    = op->nm;
    if (!env || op->shape != NKB_HEX || nm < 2 || nm > 11 || op->nq[0] != nm + 1 ||
        (op->optype != NKB_HELMHOLTZ && op->optype != NKB_LINEAR_ADR) ||
        !SameTable(op->hD[0], op->hD[1]) || !SameTable(op->hD[0], op->hD[2]) || ForceGeneric())
        return false;
    *v = std::atoi(env);
    return *v == 0 || (*v == 5 && op->optype == NKB_HELMHOLTZ && op->precision == NKB_FP32 &&
                       nm >= kTcMinNm && nm <= kTcMaxNm);
}

int ChooseKernel(nkb_op *op)
{
    op->variant  = kVariantGeneric;
    if (!op->line_tabs.empty())
        return NKB_OK; // a line kernel (nkb_line.cu): nothing to choose
    const int eb = op->precision == NKB_FP64 ? 8 : 4;
    int v = 0;
    if (HexVariantRequested(op, &v))
    {
        HexArgs<double> ad = MakeHexArgs<double>(op);
        HexArgs<float> af  = MakeHexArgs<float>(op);
        const int rc = op->precision == NKB_FP64
                           ? HexLaunchT<double>(op, ad, false, op->stream, v, true)
                           : HexLaunchT<float>(op, af, false, op->stream, v, true);
        if (rc == NKB_OK)
        {
            op->variant     = kVariantHexHelm;
            op->hex_variant = v;
            return NKB_OK;
        }
        ClearError();
    }
    if (GenericSmemBytes(op, eb) > 200 * 1024)
        return SetError(NKB_ERR_UNSUPPORTED,
                        "nkb_op_create: nm=%d nq=(%d,%d,%d) needs %zu bytes of shared memory per "
                        "element", op->nm, op->nq[0], op->nq[1], op->nq[2], GenericSmemBytes(op, eb));
    const char *tune = std::getenv("NKB_GENERIC_TUNE");
    if (tune && std::strcmp(tune, "0") == 0)
        return NKB_OK;
    return op->precision == NKB_FP64 ? AutotuneGeneric<double>(op) : AutotuneGeneric<float>(op);
}

void FreeKernelData(nkb_op *op)
{
    op->kdata = nullptr;
}

const char *KernelName(const nkb_op *op, bool)
{
    if (op->optype == NKB_DENSE_BLOCK)
        return "k_dense_gemv (per-element dense blocks)";
    if (op->variant != kVariantHexHelm)
        return op->line_tabs.empty() ? "k_generic" : "k_line (one thread per grid line)";
    return op->hex_variant == 5
               ? "k_hex_helm_tc (tcgen05 TF32 high/low tensor cores, FP32 accumulate)"
               : "k_hex_helm (TMA-staged geometry)";
}

template <typename T>
int LaunchOp(const nkb_op *op, const T *in, T *o0, T *o1, T *o2, const int *gmap,
             const double *gsign, cudaStream_t s, const int *skip, const double *lambda)
{
    if (op->nelmt == 0)
        return NKB_OK; // an empty collection: nothing to launch (a zero-CTA grid is invalid)
    if (op->optype == NKB_DENSE_BLOCK)
    {
        if (!std::is_same<T, double>::value)
            return SetError(NKB_ERR_UNSUPPORTED, "dense operators are FP64");
        return LaunchDense(op, reinterpret_cast<const double *>(in), reinterpret_cast<double *>(o0),
                           gmap, gsign, s, skip);
    }
    if (op->variant == kVariantHexHelm)
    {
        HexArgs<T> a = MakeHexArgs<T>(op);
        if (lambda)
            a.lambda = T(*lambda);
        a.in         = in;
        a.out        = o0;
        a.gmap       = gmap;
        a.gsign      = gsign;
        a.skip       = skip;
        return HexLaunchT<T>(op, a, gmap != nullptr, s, op->hex_variant, false);
    }
    return LaunchGeneric<T>(op, in, o0, o1, o2, gmap, gsign, s, skip, lambda);
}

template int LaunchOp<double>(const nkb_op *, const double *, double *, double *, double *,
                              const int *, const double *, cudaStream_t, const int *,
                              const double *);
template int LaunchOp<float>(const nkb_op *, const float *, float *, float *, float *,
                             const int *, const double *, cudaStream_t, const int *,
                             const double *);

} // namespace nkb

extern "C" const char *nkb_op_kernel(const nkb_op *op, int gather)
{
    return op ? nkb::KernelName(op, gather != 0) : "";
}
