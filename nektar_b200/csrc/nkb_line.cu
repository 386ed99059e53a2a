// Set-up and dispatch of the line kernels (nkb_line_kernel.cuh).
#include "nkb_line_kernel.cuh"

#include <cstdlib>
#include <cstring>

namespace nkb
{

#define NKB_LINE_EXTERN(OP)                                                                        \
    extern template int LineSwitch<OP, double>(nkb_op *, const nkb_op *, const LineArgs<double> *, \
                                               cudaStream_t);                                      \
    extern template int LineSwitch<OP, float>(nkb_op *, const nkb_op *, const LineArgs<float> *,   \
                                              cudaStream_t);
NKB_LINE_EXTERN(LN_BWD)
NKB_LINE_EXTERN(LN_IP)
NKB_LINE_EXTERN(LN_PD)
NKB_LINE_EXTERN(LN_IPD)
NKB_LINE_EXTERN(LN_HELM)
NKB_LINE_EXTERN(LN_ADR)
#undef NKB_LINE_EXTERN

template <typename T>
static int LineDispatch(nkb_op *setup, const nkb_op *op, const LineArgs<T> *a, cudaStream_t s)
{
    switch (op->optype)
    {
        case NKB_BWDTRANS: return LineSwitch<LN_BWD, T>(setup, op, a, s);
        case NKB_IPRODUCT: return LineSwitch<LN_IP, T>(setup, op, a, s);
        case NKB_PHYSDERIV: return LineSwitch<LN_PD, T>(setup, op, a, s);
        case NKB_IPRODUCT_DERIV: return LineSwitch<LN_IPD, T>(setup, op, a, s);
        case NKB_LINEAR_ADR: return LineSwitch<LN_ADR, T>(setup, op, a, s);
        default: return LineSwitch<LN_HELM, T>(setup, op, a, s);
    }
}

int LineSetup(nkb_op *op)
{
    const bool helm = op->optype == NKB_HELMHOLTZ || op->optype == NKB_LINEAR_ADR;
    const bool hex  = op->shape == NKB_HEX;
    const char *kernel = std::getenv("NKB_KERNEL");
    if (kernel && std::strcmp(kernel, "generic") == 0)
        return NKB_OK;
    int v = 0;
    if (HexVariantRequested(op, &v))
        return NKB_OK; // one of nkb_hex.cu's kernels, by request
    const int rc = op->precision == NKB_FP64
                       ? LineDispatch<double>(op, op, nullptr, nullptr)
                       : LineDispatch<float>(op, op, nullptr, nullptr);
    if (rc == kLineNone)
        return NKB_OK;
    op->geo_perm = helm && !hex ? 1 : 0;
    return rc;
}

template <typename T>
int LaunchLine(const nkb_op *op, const T *in, const T *in1, const T *in2, T *o0, T *o1, T *o2,
               const int *gmap, const double *gsign, cudaStream_t s, const int *skip, T lambda)
{
    constexpr bool f64 = std::is_same<T, double>::value;
    LineArgs<T> a;
    a.in      = in;
    a.in1     = in1;
    a.in2     = in2;
    a.out0    = o0;
    a.out1    = o1;
    a.out2    = o2;
    a.geo     = f64 ? (const T *)op->geo : (const T *)op->geo32;
    a.geoc    = op->geoc;
    a.tB1     = f64 ? (const T *)op->dB[1] : (const T *)op->fB[1];
    a.tB2     = f64 ? (const T *)op->dB[2] : (const T *)op->fB[2];
    a.gmap    = gmap;
    a.gsign   = gsign;
    a.skip    = skip;
    a.gstride = op->gstride;
    a.lambda  = lambda;
    a.nelmt   = op->nelmt;
    a.nm      = op->nm;
    return LineDispatch<T>(nullptr, op, &a, s);
}

template int LaunchLine<double>(const nkb_op *, const double *, const double *, const double *,
                                double *, double *, double *, const int *, const double *,
                                cudaStream_t, const int *, double);
template int LaunchLine<float>(const nkb_op *, const float *, const float *, const float *, float *,
                               float *, float *, const int *, const double *, cudaStream_t,
                               const int *, float);

} // namespace nkb
